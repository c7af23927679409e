// The whole Rader step over the factor 257 in one kernel (m = n / 257 lanes of
// C columns, L = m*C lanes): gather, 256-point transform, product with the
// transformed Rader kernel, inverse transform, x[0] and twiddle, for LN adjacent
// lanes per CTA of 16*LN threads and 272*LN words of shared memory.
//
// Both transforms are 16 x 16, a thread's 16-point group in registers.  The first
// leaves frequency k1 + 16 t at t of the thread of group k1, which is the input
// the second one's first round takes, so the product stays in registers and only
// two exchanges go through shared memory (word (17*k + d)*lanes + lane: a half-warp
// on distinct banks either way).  One read and one write of the data, where the
// step took five kernels and about nine passes over memory.  Bound by the
// integer pipes and, for few tiles, by the four codelets in a row of each thread.
// Whole transforms on GB300 (us, before -> now): 257 x 4096 45.9 -> 38.0, 257 x
// 65536 545 -> 361, 257 x 256 over 64 columns 111 -> 66, one 257 15.1 -> 11.3.
#pragma once
#include "gl_pass.cuh"

struct gl_rader257_args {
  const uint64_t *src;   // 257 rows of L words
  uint64_t *dst;         // word (j2*257 + k1)*C + c for lane l = j2*C + c
  uint64_t L, C;
  const uint32_t *gpow;  // g^p mod 257, p < 256
  const uint32_t *gneg;  // g^-p
  const uint64_t *tw_f;  // omega_256^e (Montgomery form)
  const uint64_t *tw_i;  // omega_256^-e / 256 (Montgomery form)
  const uint64_t *bhat;  // transformed Rader kernel (Montgomery form)
  const uint64_t *tw_lo, *tw_hi;  // omega_n^e (Montgomery form, perhaps scaled)
  // Debug builds: the extents of src and dst in words (0: unchecked), the check word.
  uint64_t dbg_in_words, dbg_out_words;
  uint32_t *dbg_err;
};

template <int LN>
__device__ __forceinline__ void gl_rader257_block(const gl_rader257_args &a, uint64_t bx, uint64_t *sm) {
  const uint32_t c = threadIdx.x % LN, g = threadIdx.x / LN;
  const uint64_t l = bx * LN + c;
  const bool live = l < a.L;
  gl_pdl_launch_dependents();
  gl_pdl_wait();
  constexpr int SM = LN * 272;
  auto load = [&](const uint64_t *p) { return gl_dbg_ok(a, p - a.src, a.dbg_in_words, GL_DBG_IN) ? *p : 0; };
  auto store = [&](uint64_t *p, uint64_t v) {
    if (gl_dbg_ok(a, p - a.dst, a.dbg_out_words, GL_DBG_OUT)) *p = v;
  };
  uint64_t x[16];
  const uint64_t x0 = live ? gl_canon(load(a.src + l)) : 0;
#pragma unroll
  for (int t = 0; t < 16; t++) x[t] = live ? load(a.src + (__ldg(a.gpow + g + 16 * t) * a.L + l)) : 0;
  gl_dft_lazy<16, false>(x);
#pragma unroll
  for (int t = 0; t < 16; t++)
    gl_sm_st(a, sm, (t * 17 + g) * LN + c, SM, t ? gl_mont_mul(x[t], __ldg(a.tw_f + g * t)) : x[t]);
  __syncthreads();
#pragma unroll
  for (int t = 0; t < 16; t++) x[t] = gl_sm_ld(a, sm, (g * 17 + t) * LN + c, SM);
  gl_dft_lazy<16, false>(x);
  // Frequency k = g + 16 t; that of k = 0 is the sum of all inputs but x[0].
  const uint64_t sum = gl_add(x0, gl_canon(x[0]));
#pragma unroll
  for (int t = 0; t < 16; t++) x[t] = gl_mont_mul(x[t], __ldg(a.bhat + g + 16 * t));
  gl_dft_lazy<16, true>(x);
  __syncthreads();
#pragma unroll
  for (int t = 0; t < 16; t++)
    gl_sm_st(a, sm, (t * 17 + g) * LN + c, SM, gl_mont_mul(x[t], __ldg(a.tw_i + g * t)));
  __syncthreads();
#pragma unroll
  for (int t = 0; t < 16; t++) x[t] = gl_sm_ld(a, sm, (g * 17 + t) * LN + c, SM);
  gl_dft_lazy<16, true>(x);
  // Convolution outputs p = g + 16 t.
  const uint64_t j2 = a.C == 1 ? l : l / a.C;
  // One column: a tile's outputs are one contiguous block, written through
  // shared memory so that adjacent threads store adjacent words.
  const bool block = a.C == 1;
  if (block) __syncthreads();  // uniform
  uint64_t *out = a.dst + (l - j2 * a.C) + j2 * 257 * a.C;
#pragma unroll
  for (int t = 0; t < 16; t++) {
    const uint32_t k1 = __ldg(a.gneg + g + 16 * t);
    const uint64_t v = live ? gl_mont_mul(gl_add(x0, gl_canon(x[t])), gl_tw2m(a.tw_lo, a.tw_hi, j2 * k1)) : 0;
    if (block) gl_sm_st(a, sm, c * 257 + k1, SM, v);
    else if (live) store(out + k1 * a.C, v);
  }
  if (g == 0) {
    const uint64_t v = live ? gl_mont_mul(sum, gl_tw2m(a.tw_lo, a.tw_hi, 0)) : 0;
    if (block) gl_sm_st(a, sm, c * 257, SM, v);
    else if (live) store(out, v);
  }
  if (!block) return;
  __syncthreads();
  const uint64_t first = bx * (LN * 257), end = a.L * 257;
  for (int i = threadIdx.x; i < LN * 257; i += LN * 16)
    if (first + i < end) store(a.dst + first + i, gl_sm_ld(a, sm, i, SM));
}
