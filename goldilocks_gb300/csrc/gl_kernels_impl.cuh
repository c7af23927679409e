// Instantiates one set of pass-kernel variants.  Included by the gl_kern_*.cu
// translation units so that the sets compile in parallel.
#pragma once
#include "gl_internal.h"

template <int R1, int R2, int R3, int LANES, int NT, bool INV, int MINB = 1, bool GT = false, bool UNI = false>
static void gl_launch_pass3(const gl_pass_args &args, dim3 grid, cudaStream_t stream, bool pdl) {
  constexpr size_t smem =
      UNI ? (size_t)gl_uni_layout<R1, R2, R3, LANES>::WORDS * 8 : gl_p3_smem_bytes<R1, R2, R3, LANES>();
  auto kern = gl_pass3_kernel<R1, R2, R3, LANES, NT, INV, MINB, GT, UNI>;
  static std::atomic<uint64_t> optin{0};
  gl_smem_optin(optin, kern, smem);
  if (!pdl) {
    kern<<<grid, NT, smem, stream>>>(args);
    return;
  }
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, args);
}

#define GL_ENTRY3(R1, R2, R3, LANES, NT, INV)                                                 \
  {R1 * R2 * R3, R1, R2, R3, LANES, INV, gl_p3_smem_bytes<R1, R2, R3, LANES>(), NT,          \
   gl_launch_pass3<R1, R2, R3, LANES, NT, INV>, false,                                        \
   (const void *)gl_pass3_kernel<R1, R2, R3, LANES, NT, INV, 1>}

// MINB CTAs resident per SM (registers capped to fit), so that one CTA's
// loads overlap another's arithmetic.
#define GL_ENTRY3M(R1, R2, R3, LANES, NT, MINB, INV)                                          \
  {R1 * R2 * R3, R1, R2, R3, LANES, INV, gl_p3_smem_bytes<R1, R2, R3, LANES>(), NT,          \
   gl_launch_pass3<R1, R2, R3, LANES, NT, INV, MINB>, false,                                  \
   (const void *)gl_pass3_kernel<R1, R2, R3, LANES, NT, INV, MINB>}

// Two forms of one pass: NT threads for a launch of up to PER_SM tiles per SM
// (two), where a tile's own latency counts, and for more tiles NTM threads with
// MINB CTAs per SM, sized so that the groups of each round fill whole walks of the
// threads (the 1024-thread 16 x 16 x 8 form idles half its threads in two
// rounds of three: barrier stalls 5.4 per issued instruction) and one CTA's
// loads overlap another's arithmetic.  Measured on GB300 (us): 8 transforms of
// 2^20 124.9 -> 112.7 (2048-point rows), LDE 2^20 x 64 5589 -> 5130; one 2^20
// (128 tiles) 23.1 -> 29.1, which is why the first form stays.  PER_SM is per
// shape, from 3, 4, 6 and 9 transforms of 512 x m (2.5, 3.4, 5.1 and 7.6 tiles
// per SM), second form against first: m = 1280 0.84, 0.95, 1.06, 1.18 (four);
// 2040 0.96, 0.96, 1.05, 1.04 (four); 1536 0.90, 1.03, 1.06, 1.15, 1360
// and 2176 alike (three); 1088 1.15 .. 1.21, 1920, 2048, 2720 and 3264 1.03 and
// up throughout (two).  m = 1024 stays at two (three transforms 27.4 us, with
// the first form 28.8).
template <int R1, int R2, int R3, int LANES, int NT, int NTM, int MINB, bool INV, int PER_SM = 2>
static void gl_launch_pass3_by_tiles(const gl_pass_args &args, dim3 grid, cudaStream_t stream, bool pdl) {
  if ((uint64_t)grid.x * grid.y * grid.z > (uint64_t)PER_SM * (unsigned)gl_sm_count())
    gl_launch_pass3<R1, R2, R3, LANES, NTM, INV, MINB>(args, grid, stream, pdl);
  else
    gl_launch_pass3<R1, R2, R3, LANES, NT, INV>(args, grid, stream, pdl);
}

#define GL_ENTRY3T(R1, R2, R3, LANES, NT, NTM, MINB, INV, ...)                                \
  {R1 * R2 * R3, R1, R2, R3, LANES, INV, gl_p3_smem_bytes<R1, R2, R3, LANES>(), NT,          \
   gl_launch_pass3_by_tiles<R1, R2, R3, LANES, NT, NTM, MINB, INV, ##__VA_ARGS__>, false,     \
   (const void *)gl_pass3_kernel<R1, R2, R3, LANES, NT, INV, 1>, false,                       \
   (const void *)gl_pass3_kernel<R1, R2, R3, LANES, NTM, INV, MINB>}

// The uniform form (gl_block3's UNI) where it applies: a pass twiddle from the
// two-level table, and a number of interleaved columns that is a multiple of
// the lanes.
template <int R1, int R2, int R3, int LANES, int NT, int MINB, bool INV>
static void gl_launch_pass3_cols(const gl_pass_args &args, dim3 grid, cudaStream_t stream, bool pdl) {
  const bool uniform = (args.flags & (GL_PF_PASS_TWIDDLE | GL_PF_TW_TABLE)) == GL_PF_PASS_TWIDDLE &&
                       args.tw_lane_div % LANES == 0;
  if (uniform) gl_launch_pass3<R1, R2, R3, LANES, NT, INV, MINB, false, true>(args, grid, stream, pdl);
  else gl_launch_pass3<R1, R2, R3, LANES, NT, INV, MINB>(args, grid, stream, pdl);
}

#define GL_ENTRY3C(R1, R2, R3, LANES, NT, MINB, INV)                                          \
  {R1 * R2 * R3, R1, R2, R3, LANES, INV, gl_p3_smem_bytes<R1, R2, R3, LANES>(), NT,          \
   gl_launch_pass3_cols<R1, R2, R3, LANES, NT, MINB, INV>, false,                             \
   (const void *)gl_pass3_kernel<R1, R2, R3, LANES, NT, INV, MINB>, false,                    \
   (const void *)gl_pass3_kernel<R1, R2, R3, LANES, NT, INV, MINB, false, true>}

// Good-Thomas inner transform (gcd(R2, R3) = 1): for passes without a pass
// twiddle (rows, column batches); MINB as above.
#define GL_ENTRY3G(R1, R2, R3, LANES, NT, MINB, INV)                                          \
  {R1 * R2 * R3, R1, R2, R3, LANES, INV, gl_p3_smem_bytes<R1, R2, R3, LANES>(), NT,          \
   gl_launch_pass3<R1, R2, R3, LANES, NT, INV, MINB, true>, false,                            \
   (const void *)gl_pass3_kernel<R1, R2, R3, LANES, NT, INV, MINB, true>, true}
