// Block-DFT pass kernel with up to three register rounds.
//
// Every CTA transforms LANES independent m-point sequences ("lanes"),
// m = R1*R2*R3, held in one shared-memory tile.  Positions are mixed-radix
// digits p = d1*(R2*R3) + d2*R3 + d3; decimation in frequency:
//
//   round 1: DFT_R1 over d1 for each (d2, d3) = jB; then * omega_m^(jB*k1)
//   round 2: DFT_R2 over d2 for each (k1, d3);     then * omega_(R2 R3)^(d3*k2)
//   round 3: DFT_R3 over d3 for each (k1, k2)
//   output frequency k = k1 + R1*k2 + R1*R2*k3.
//
// GT variant (gcd(R2, R3) = 1; passes without a pass twiddle): the inner
// R2*R3-point transform of rounds 2 and 3 is Good-Thomas instead of
// Cooley-Tukey, so it needs no twiddles.  Round 2 gathers its inputs at
// d' = (R3*a + R2*b) mod R2*R3 over a (b fixed) and writes its outputs k2
// back to the same positions; round 3 gathers d' = (R3*k2 + R2*b) mod R2*R3
// over b; the output frequency is k = k1 + R1*k', k' = CRT(k2 mod R2,
// k3 mod R3).  (Adjacent threads take adjacent b in round 2 and adjacent k2
// in round 3, so the gathers stay on distinct banks.)
//
// Each thread holds one radix-R group in registers (R <= 17), so the code per
// round is one straight-line codelet.  Round 1 reads global memory directly
// and the last round writes it; rounds exchange through shared memory
// (XOR-swizzled against bank conflicts).  Strides give the COL / ROW / FULL
// roles of gl_pass.cuh; the same flags apply (pass twiddle, zero padding,
// coset factor, scale).  The codelets take and give any words congruent to
// the values (gl_dft_lazy); a twiddle product reduces them, and what leaves
// without one is reduced on the store.
#pragma once
#include "gl_pass.cuh"

template <int R1, int R2, int R3, int LANES>
struct gl_p3_layout {
  static constexpr int M = R1 * R2 * R3;
  static constexpr int S1 = R2 * R3;
  static constexpr int NR = R2 == 1 ? 1 : (R3 == 1 ? 2 : 3);
  static constexpr int RL = NR == 3 ? R3 : (NR == 2 ? R2 : R1);  // last radix
  static constexpr bool POW2 = (RL & (RL - 1)) == 0 && (M & (M - 1)) == 0;
  static constexpr int SH = RL == 16 ? 4 : RL == 8 ? 3 : RL == 4 ? 2 : RL == 2 ? 1 : 0;
  static constexpr int MSK = POW2 ? (RL < 16 ? RL - 1 : 15) : 0;
  // A half-warp's 16 accesses (64-bit words; 16 words per 128-byte wavefront)
  // cover 16 / LANES positions of each of LANES lanes, so the lanes must fall
  // on distinct word residues mod 16, LSTEP apart: by an XOR of the word
  // index in the power-of-two tiles, by the lane stride in the others (odd
  // for 16 lanes or more).
  static constexpr int LSTEP = 16 / (LANES < 16 ? LANES : 16);
  static constexpr int LS = POW2 ? M : ((M + 15) / 16) * 16 + LSTEP;
  static_assert(!POW2 || NR == 1 || M % 16 == 0, "power-of-two tiles are whole 16-word blocks");
  // Word of position p of lane c.
  static __device__ __forceinline__ uint32_t word(uint32_t c, uint32_t p) {
    return POW2 ? c * LS + (p ^ ((p >> SH) & MSK) ^ ((c * LSTEP) & 15)) : c * LS + p;
  }
  // Word of position pb + tb from base = word(c, pb), where tb is a multiple
  // of the digit a round walks and shares no bit with pb: the swizzle is
  // linear over XOR, so the step is an XOR of the low four bits with a
  // constant and an immediate offset.  (Evaluating word() for every access
  // took three to four instructions each, 16 of the 259 per element of the
  // 4096-point column pass.)
  static __device__ __forceinline__ uint32_t at(uint32_t base, uint32_t tb) {
    const uint32_t w = tb ^ ((tb >> SH) & MSK);
    return POW2 ? (base ^ (w & 15u)) + (w & ~15u) : base + tb;
  }
  // Shared memory after the tile (words), staged before round 1 and
  // published by the barrier that ends it.  Three rounds (the Cooley-Tukey
  // form):
  //   T2    the round-2 twiddles omega_(R2 R3)^(d3*k2) at [k2*R3 + d3];
  // two or three rounds:
  //   STEP  per lane c and last-round output digit t, the pass-twiddle step
  //         omega_n^(col_c * SL * t) (SL: output stride of the last digit),
  //         RL + 1 words per lane so that the lanes fall on distinct banks.
  static constexpr int TILE = NR == 1 ? 0 : LANES * LS;
  static constexpr int T2 = TILE;
  static constexpr int NT2 = NR == 3 ? S1 : 0;
  static constexpr int STEP = T2 + NT2;
  static constexpr int SS = RL + 1;  // per-lane stride: lanes on distinct banks
  static constexpr int NSTEP = NR == 1 ? 0 : LANES * SS;
  static constexpr int WORDS = STEP + NSTEP;
};

// The tables of the uniform form (gl_block3's UNI), words after the tile:
//   T2   omega_(R2 R3)^(d3*k2) * omega_n^(col*R1*k2) at [k2*R3 + d3] (three rounds)
//   PT   the rest of the pass twiddle at [t*R1 + k1]: omega_n^(col*(k1 + SL*t))
//   IG   the input factor's step g^(S1*itw_jmul*t), t < R1
//   IB   the input factor's base g^(j*itw_jmul + col), j < S1
//   T1   the round-1 twiddles times the base: tw_m[g*t] * IB[g] at [t*S1 + g]
template <int R1, int R2, int R3, int LANES>
struct gl_uni_layout : gl_p3_layout<R1, R2, R3, LANES> {
  using B = gl_p3_layout<R1, R2, R3, LANES>;
  static constexpr int NPT = B::NR == 3 ? R1 * B::RL : B::M;
  static constexpr int T2 = B::TILE;
  static constexpr int PT = T2 + (B::NR == 3 ? B::S1 : 0);
  static constexpr int IG = PT + NPT;
  static constexpr int IB = IG + R1;
  static constexpr int T1 = IB + B::S1;
  static constexpr int WORDS = T1 + B::M;
};

template <int R1, int R2, int R3, int LANES>
constexpr size_t gl_p3_smem_bytes() {
  return (size_t)gl_p3_layout<R1, R2, R3, LANES>::WORDS * 8;
}

// Good-Thomas constants of the inner R2 x R3 transform.
constexpr int gl_gcd(int a, int b) { return b == 0 ? a : gl_gcd(b, a % b); }
constexpr int gl_modinv(int a, int m) {  // a^-1 mod m, 0 when there is none
  for (int r = 1; r < m; r++)
    if ((a * r) % m == 1) return r;
  return 0;
}
template <int R2, int R3>
struct gl_gt_consts {
  static constexpr int S = R2 * R3;
  static constexpr int AINV = gl_modinv(R3 % R2, R2);  // a = d' * AINV mod R2
  static constexpr int BINV = gl_modinv(R2 % R3, R3);  // b = d' * BINV mod R3
  static constexpr int E2 = R3 * AINV;                 // 1 mod R2, 0 mod R3
  static constexpr int E3 = R2 * BINV;                 // 0 mod R2, 1 mod R3
};

// A round's groups over the CTA's threads: idx = threadIdx.x + it*NT, without
// a bound check where the groups fill every pass over them.
#define GL_ROUND(idx, COUNT)                                                                       \
  _Pragma("unroll 1") for (uint32_t gl_it = 0, idx = threadIdx.x; gl_it < ((COUNT) + NT - 1) / NT;      \
                           gl_it++, idx += NT)                                                     \
    if ((COUNT) % NT == 0 || idx < (COUNT))

// One CTA's work: tile (bx, by, bz) of the pass described by `a`, with NT
// threads and the dynamic shared memory `sm`.  Called by gl_pass3_kernel
// (tile = blockIdx) and by the persistent batch kernel (tile from its queue).
//
// UNI: a pass with a pass twiddle over interleaved columns whose number is a
// multiple of LANES, so that the lanes of a tile have one column index: the
// pass twiddle and the coset factor are tables of the tile.  Each element then
// takes one product for the pass twiddle (its factor in k2 rides on the round-2
// twiddle) where a base and a step per lane take two, and the coset factor
// g^(j*itw_jmul + col), j = g + S1*t, splits into a step in t on the load and
// a base that rides on the round-1 twiddle, where two table loads, an index
// computation and two products an element took a quarter of the instructions.
template <int R1, int R2, int R3, int LANES, int NT, bool INV, bool GT = false, bool UNI = false>
__device__ __forceinline__ void gl_block3(const gl_pass_args &a, int64_t bx, int64_t by,
                                          int64_t bz, uint64_t *sm) {
  using L = gl_p3_layout<R1, R2, R3, LANES>;
  using U = gl_uni_layout<R1, R2, R3, LANES>;
  using GTC = gl_gt_consts<R2, R3>;
  constexpr int M = L::M;
  constexpr int S1 = R2 * R3;
  constexpr int TILE = LANES * L::LS;
  static_assert(!GT || (L::NR == 3 && gl_gcd(R2, R3) == 1), "Good-Thomas inner transform needs coprime R2, R3");

  // Lanes, groups and positions are 32-bit (a pass has fewer than 2^32 lanes);
  // only addresses are 64-bit.  The lane's column index is a division only
  // for interleaved columns: as a 64-bit division in each thread it cost up
  // to ten instructions per element.
  const uint32_t lane0 = (uint32_t)bx * LANES;
  auto column = [&](uint32_t lane) { return a.tw_lane_div == 1 ? lane : lane / a.tw_lane_div; };
  if (!(a.flags & GL_PF_LATE)) gl_pdl_launch_dependents();

  // Stage the tables (read after the barrier that ends round 1).  They come
  // from constant tables, so they are loaded before the wait below and their
  // latency overlaps the previous pass's tail (under programmatic dependent
  // launch) and this pass's loads.
  constexpr int SL = L::NR == 3 ? R1 * R2 : R1;  // output stride of the last digit
  const bool tw_steps = (a.flags & (GL_PF_PASS_TWIDDLE | GL_PF_TW_TABLE)) == GL_PF_PASS_TWIDDLE;
  if constexpr (L::NR == 3 && !GT && !UNI) {
    for (int i = threadIdx.x; i < S1; i += NT)
      gl_sm_st(a, sm, L::T2 + i, L::WORDS, __ldg(a.tw_r2 + R1 * (i % R3) * (i / R3)));
  }
  if constexpr (L::NR > 1 && !UNI) {
    if (tw_steps) {
      for (uint32_t i = threadIdx.x; i < L::NSTEP; i += NT) {
        const uint32_t c = i / L::SS, t = i % L::SS;
        if (t >= L::RL) continue;
        if (lane0 + c >= a.lanes) continue;  // lanes past the end read no table
        const uint64_t col = column(lane0 + c) + a.tw_col0;
        uint64_t v = gl_tw2m(a.tw_lo, a.tw_hi, col * (uint32_t)(SL * t));
        if (a.tw_unscale) v = gl_mont_mul(v, a.tw_unscale);
        gl_sm_st(a, sm, L::STEP + i, L::WORDS, v);
      }
    }
  }
  // Everything below reads data an earlier kernel of the stream may write,
  // or writes global memory.
  gl_pdl_wait();
  if (a.flags & GL_PF_LATE) gl_pdl_launch_dependents();

  const bool ptr_table = (a.flags & GL_PF_PTR_TABLE) != 0;
  const uint64_t *in = ptr_table ? a.in_ptrs[by] + bz * a.in_bs2 : a.in + by * a.in_bs + bz * a.in_bs2;
  uint64_t *out = ptr_table ? a.out_ptrs[by] + bz * a.out_bs2 : a.out + by * a.out_bs + bz * a.out_bs2;
  const bool scale_all = (a.flags & GL_PF_SCALE_ALL) != 0;
  const bool load_lane_fast = (a.flags & GL_PF_LOAD_LANE_FAST) != 0;
  const bool store_lane_fast = (a.flags & GL_PF_STORE_LANE_FAST) != 0;
  const bool load_cg = (a.flags & GL_PF_LOAD_CG) != 0;  // written earlier in the same launch: read via L2
  // Every lane and index of the tile is there (uniform over the CTA).
  const bool whole = lane0 + LANES <= a.lanes && lane0 + LANES > lane0 && a.in_limit >= (uint32_t)M;

  const bool in_twiddle = (a.flags & GL_PF_IN_TWIDDLE) != 0;
  // The uniform form's tables, staged behind the data loads of round 1.
  [[maybe_unused]] auto stage_uniform = [&]() {
    const uint64_t col = column(lane0) + a.tw_col0;
    if constexpr (L::NR == 3) {
      for (uint32_t i = threadIdx.x; i < S1; i += NT) {
        const uint32_t k2 = i / R3, d3 = i % R3;
        uint64_t v = gl_tw2m(a.tw_lo, a.tw_hi, col * (R1 * k2));
        if (a.tw_unscale) v = gl_mont_mul(v, a.tw_unscale);
        gl_sm_st(a, sm, U::T2 + i, U::WORDS, gl_mont_mul(v, __ldg(a.tw_r2 + R1 * d3 * k2)));
      }
    }
    for (uint32_t i = threadIdx.x; i < U::NPT; i += NT)  // k = k1 + SL*t; two rounds: k = i
      gl_sm_st(a, sm, U::PT + i, U::WORDS, gl_tw2m(a.tw_lo, a.tw_hi, col * (L::NR == 3 ? i % R1 + SL * (i / R1) : i)));
    if (in_twiddle) {
      // Indices at or past in_limit load as zero and lie outside the tables:
      // their factor is any word.
      const uint32_t icol = column(lane0);
      for (uint32_t i = threadIdx.x; i < R1; i += NT)
        gl_sm_st(a, sm, U::IG + i, U::WORDS,
                 S1 * i < a.in_limit ? gl_tw2m(a.itw_lo, a.itw_hi, (uint64_t)(S1 * i) * a.itw_jmul) : 0);
      for (uint32_t i = threadIdx.x; i < S1; i += NT)
        gl_sm_st(a, sm, U::IB + i, U::WORDS,
                 i < a.in_limit ? gl_tw2m(a.itw_lo, a.itw_hi, i * a.itw_jmul + icol) : 0);
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < (uint32_t)M; i += NT) {
        const uint32_t g = i % S1, t = i / S1;
        gl_sm_st(a, sm, U::T1 + i, U::WORDS,
                 gl_mont_mul(__ldg(a.tw_m + g * t), gl_sm_ld(a, sm, U::IB + g, U::WORDS)));
      }
    }
    __syncthreads();
  };

  // ------------------------------------------------------------- round 1
  {
    static_assert(!UNI || (!GT && L::NR > 1 && LANES * (M / R1) == NT), "one round-1 group per thread");
    constexpr uint32_t G = M / R1;  // groups per lane: jB = (d2, d3)
    GL_ROUND(idx, LANES * G) {
      uint32_t c, g;
      if (load_lane_fast) { c = idx % LANES; g = idx / LANES; }
      else { g = idx % G; c = idx / G; }
      const uint32_t lane = lane0 + c;
      const bool live = lane < a.lanes;
      uint64_t x[R1];
      const uint64_t *src = in + (uint64_t)a.in_ls * lane + (uint64_t)a.in_is * g;
      const int64_t step = (int64_t)S1 * a.in_is;
      if (whole && !load_cg) {
#pragma unroll
        for (int t = 0; t < R1; t++) x[t] = gl_ld_in(a, src + t * step, false);
      } else {
#pragma unroll
        for (int t = 0; t < R1; t++) {
          const uint32_t j = g + S1 * t;
          x[t] = (live && j < a.in_limit) ? gl_ld_in(a, src + t * step, load_cg) : 0;
        }
      }
      if constexpr (UNI) {
        stage_uniform();
        if (in_twiddle) {
#pragma unroll
          for (int t = 1; t < R1; t++) x[t] = gl_mont_mul(x[t], gl_sm_ld(a, sm, U::IG + t, U::WORDS));
        }
      } else if (in_twiddle) {
        const uint32_t col = column(lane);
#pragma unroll
        for (int t = 0; t < R1; t++) {
          const uint32_t j = g + S1 * t;
          if (j < a.in_limit) x[t] = gl_mont_mul(x[t], gl_tw2m(a.itw_lo, a.itw_hi, j * a.itw_jmul + col));
        }
      }
      gl_dft_lazy<R1, INV>(x);
      if constexpr (L::NR == 1) {
        // Single round: t is the output index.
        if (scale_all) {
          const uint64_t s = a.tw_m[0];
#pragma unroll
          for (int t = 0; t < R1; t++) x[t] = gl_mont_mul(x[t], s);
        }
        if (live) {
          uint64_t *dst = out + (uint64_t)a.out_ls * lane;
          if (a.flags & GL_PF_PASS_TWIDDLE) {
            const uint64_t col = column(lane);
#pragma unroll
            for (int t = 0; t < R1; t++)
              gl_st_out(a, dst + (int64_t)t * a.out_is, gl_mont_mul(x[t], gl_pass_tw(a, col, t)));
          } else if (a.flags & GL_PF_OUT_MUL) {
            const uint64_t *mb = a.mul + by * a.mul_bs + bz * a.mul_bs2;
#pragma unroll
            for (int t = 0; t < R1; t++) gl_st_out(a, dst + (int64_t)t * a.out_is, gl_out_mul(a, mb, lane, t, x[t]));
          } else {
#pragma unroll
            for (int t = 0; t < R1; t++) gl_st_out(a, dst + (int64_t)t * a.out_is, gl_canon(x[t]));
          }
        }
      } else {
        const uint32_t base = L::word(c, g);
        if (UNI && in_twiddle) {
#pragma unroll
          for (int t = 0; t < R1; t++)
            gl_sm_st(a, sm, L::at(base, S1 * t), TILE, gl_mont_mul(x[t], gl_sm_ld(a, sm, U::T1 + S1 * t + g, U::WORDS)));
          continue;
        }
#pragma unroll
        for (int t = 0; t < R1; t++) {
          uint64_t v = x[t];
          if (t > 0 || scale_all) v = gl_mont_mul(v, __ldg(a.tw_m + g * t));
          gl_sm_st(a, sm, L::at(base, S1 * t), TILE, v);
        }
      }
    }
  }
  if constexpr (L::NR == 1) return;
  __syncthreads();  // uniform: every thread of the CTA reaches it

  // ------------------------------------------------------------- round 2
  if constexpr (L::NR == 3) {
    constexpr uint32_t G = R1 * R3;  // groups (k1, d3)
    GL_ROUND(idx, LANES * G) {
      const uint32_t c = idx % LANES, g = idx / LANES;
      const uint32_t k1 = g / R3, d3 = g % R3;
      uint64_t x[R2];
      if constexpr (GT) {
        // inputs a at (R3*a + R2*b) mod S1, b = d3; outputs k2 = t in their place
        int pos[R2];
#pragma unroll
        for (int t = 0; t < R2; t++) {
          int v = R2 * d3 + R3 * t;
          if (v >= S1) v -= S1;
          pos[t] = L::word(c, k1 * S1 + v);
        }
#pragma unroll
        for (int t = 0; t < R2; t++) x[t] = gl_sm_ld(a, sm, pos[t], TILE);
        gl_dft_lazy<R2, INV>(x);
#pragma unroll
        for (int t = 0; t < R2; t++) gl_sm_st(a, sm, pos[t], TILE, x[t]);
      } else {
        const uint32_t base = L::word(c, k1 * S1 + d3);
        const uint32_t tw = (UNI ? (int)U::T2 : (int)L::T2) + d3;
#pragma unroll
        for (int t = 0; t < R2; t++) x[t] = gl_sm_ld(a, sm, L::at(base, R3 * t), TILE);
        gl_dft_lazy<R2, INV>(x);
#pragma unroll
        for (int t = 0; t < R2; t++) {
          uint64_t v = x[t];
          if (t > 0) v = gl_mont_mul(v, gl_sm_ld(a, sm, tw + R3 * t, UNI ? (int)U::WORDS : (int)L::WORDS));
          gl_sm_st(a, sm, L::at(base, R3 * t), TILE, v);
        }
      }
    }
    __syncthreads();
  }

  // ------------------------------------------------------- last round
  {
    constexpr int RL = L::RL;
    constexpr uint32_t G = M / RL;                 // groups: (k1, k2) or k1
    GL_ROUND(idx, LANES * G) {
      uint32_t c, g;
      if (store_lane_fast) { c = idx % LANES; g = idx / LANES; }
      else { g = idx % G; c = idx / G; }
      // group g enumerates (k1, k2) with k2 fastest for 3 rounds (positions
      // k1*S1 + k2*R3 + t), or k1 for 2 rounds (positions k1*R2 + t).
      const uint32_t k1 = L::NR == 3 ? g / R2 : g, k2 = L::NR == 3 ? g % R2 : 0;
      uint64_t x[RL];
      if constexpr (GT) {
        // inputs b at (R3*k2 + R2*b) mod S1 of block k1
#pragma unroll
        for (int t = 0; t < RL; t++) {
          int v = R3 * k2 + R2 * t;
          if (v >= S1) v -= S1;
          x[t] = gl_sm_ld(a, sm, L::word(c, k1 * S1 + v), TILE);
        }
      } else {
        const uint32_t base = L::word(c, g * RL);
#pragma unroll
        for (int t = 0; t < RL; t++) x[t] = gl_sm_ld(a, sm, L::at(base, t), TILE);
      }
      gl_dft_lazy<RL, INV>(x);
      const uint32_t lane = lane0 + c;
      if (lane >= a.lanes) continue;
      uint64_t *dst = out + (uint64_t)a.out_ls * lane;
      if constexpr (GT) {
        // Rows and column batches only: no pass twiddle in this form.
        // k = k1 + R1 * ((k2 * E2 + t * E3) mod S1)
        const int kbase = (k2 * GTC::E2) % S1;
        dst += (uint64_t)a.out_is * k1;
        const int64_t kstride = (int64_t)R1 * a.out_is;
        const bool mul = (a.flags & GL_PF_OUT_MUL) != 0;
        const uint64_t *mb = mul ? a.mul + by * a.mul_bs + bz * a.mul_bs2 : nullptr;
#pragma unroll
        for (int t = 0; t < RL; t++) {
          int kk = kbase + (t * GTC::E3) % S1;
          if (kk >= S1) kk -= S1;
          const uint64_t v = mul ? gl_out_mul(a, mb, lane, k1 + R1 * kk, x[t]) : gl_canon(x[t]);
          gl_st_out(a, dst + (int64_t)kk * kstride, v);
        }
      } else {
        const uint32_t kbase = k1 + R1 * k2;  // output index of t: kbase + SL*t
        dst += (uint64_t)a.out_is * kbase;
        const int64_t kstep = (int64_t)SL * a.out_is;
        if constexpr (UNI) {
#pragma unroll
          for (int t = 0; t < RL; t++)
            gl_st_out(a, dst + t * kstep, gl_mont_mul(x[t], gl_sm_ld(a, sm, U::PT + R1 * t + k1, U::WORDS)));
        } else if (tw_steps) {
          // tw(col, kbase + SL*t) = tw(col, kbase) * omega_n^(col*SL*t).
          const uint64_t col = column(lane) + a.tw_col0;
          const uint64_t first = gl_tw2m(a.tw_lo, a.tw_hi, col * kbase);
#pragma unroll
          for (int t = 0; t < RL; t++) {
            const uint64_t tw =
                t == 0 ? first : gl_mont_mul(first, gl_sm_ld(a, sm, L::STEP + c * L::SS + t, L::WORDS));
            gl_st_out(a, dst + t * kstep, gl_mont_mul(x[t], tw));
          }
        } else if (a.flags & GL_PF_PASS_TWIDDLE) {
          const uint64_t col = column(lane);
#pragma unroll
          for (int t = 0; t < RL; t++)
            gl_st_out(a, dst + t * kstep, gl_mont_mul(x[t], gl_pass_tw(a, col, (uint64_t)(kbase + SL * t))));
        } else if (a.flags & GL_PF_OUT_MUL) {
          const uint64_t *mb = a.mul + by * a.mul_bs + bz * a.mul_bs2;
#pragma unroll
          for (int t = 0; t < RL; t++)
            gl_st_out(a, dst + t * kstep, gl_out_mul(a, mb, lane, kbase + SL * t, x[t]));
        } else {
#pragma unroll
          for (int t = 0; t < RL; t++) gl_st_out(a, dst + t * kstep, gl_canon(x[t]));
        }
      }
    }
  }
}

template <int R1, int R2, int R3, int LANES, int NT, bool INV, int MINB = 1, bool GT = false, bool UNI = false>
__global__ void __launch_bounds__(NT, MINB) gl_pass3_kernel(const gl_pass_args a) {
  extern __shared__ uint64_t sm[];
  gl_block3<R1, R2, R3, LANES, NT, INV, GT, UNI>(a, blockIdx.x, blockIdx.y, blockIdx.z, sm);
}
