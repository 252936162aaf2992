// Device functions shared by the step kernels (dsm_kernels.cu: one or two
// chains per warp; dsm_lockstep.cu: eight or four chains per warp in lockstep): rate
// quantisation, random words, lifetime samplers, sliding rates, the split of a
// created strand and the correlator's level-0 counters.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

#include "dsm_internal.h"
#include "dsm_math.cuh"

namespace dsm {

#define FULL_MASK 0xffffffffu
#define NEND 5

// Quantisation of a rate component to 64-bit fixed point: llrint(x * sf).
__device__ __forceinline__ unsigned long long quant(float x, float sf) {
  return (unsigned long long)__float2ll_rn(__fmul_rn(x, sf));
}

// The same rounding built from 32-bit operations, for update_pairs.  sm_103a
// runs the 64-bit conversion instruction on its narrow FP64 pipe: about 100
// cycles of latency and as many cycles of pipe occupancy per warp instruction
// (about 31 cycles of latency for this form).  update_pairs converts the
// components of every recomputed pair on the critical path of each event.
// Where one or two conversions stand alone (event classification, dt) the extra
// instructions of this form cost more than they save at full occupancy, and the
// instruction stays; the flow pass, which converts every pair of the chain each
// event, takes this form for two of a pair's four components (each measured on the
// N_K = 200 melt and shear).
//
// f2u64_rn: y in [0, 2^63) (or -0.0), the value llrint(y) takes.  Below 2^23
// adding 2^23 rounds y to an integer (the sum's ulp is 1) and the sum's bit
// pattern minus that of 2^23 is the integer, also across the carry into 2^24;
// from 2^23 up y is an integer and its significand shifted by the exponent is
// it.  NaN, infinity and y >= 2^63 give an unspecified value; update_pairs
// flags those inputs and never uses the result.  Both forms are computed and
// one is selected, so no branch splits the caller.
__device__ __forceinline__ unsigned long long f2u64_rn(float y) {
  const unsigned b = __float_as_uint(y) & 0x7fffffffu;
  const int e = (int)(b >> 23) - 150;
  const unsigned small = __float_as_uint(__fadd_rn(__uint_as_float(b), 8388608.0f)) - 0x4B000000u;
  const unsigned long long big = (unsigned long long)((b & 0x7fffffu) | 0x800000u) << (e & 63);
  return e < 0 ? (unsigned long long)small : big;
}

// Philox words (counter layout shared with the oracle)
__device__ __forceinline__ U4 rng_at(const EnsDev& E, uint32_t purpose, uint64_t ctr, uint32_t hi24,
                                     uint32_t chain) {
  // keyed by the global chain id: a chain's stream does not depend on how the
  // chains are sharded over GPUs
  return philox((uint32_t)ctr, (purpose << 24) | (hi24 & 0xffffffu), chain + E.chain_offset, E.stream, E.seed_lo,
                E.seed_hi);
}

// Lifetime samplers returning rates (gpu_random.cu:143-148, pcd_tau.h:67-82)
__device__ __forceinline__ float rate_f_t(const PcdDev& p, float u) {
  return (u < p.one_minus_g) ? m_pow(__fmaf_rn(u, p.At_, p.Dt_), p.Ct_) : p.tau_d_inv;
}
__device__ __forceinline__ float rate_f_dt(const PcdDev& p, float u) {
  return (u < p.Bdt_) ? m_pow(__fmaf_rn(u, p.Adt_, p.Ddt_), p.Cdt_) : p.tau_d_inv;
}
// p_cd fit constants (common/pcd_tau.h:32-66) evaluated in float for a
// partner of N_K = nk Kuhn steps (GEX background, gpu_random.cu:212-228);
// the oracle restates the same float operations
static __device__ __noinline__ PcdDev pcd_from_nk(float be, float nk) {
  const float z = (nk + be) / (be + 1.0f);
  const float g = 0.667f;
  float alpha, tau0, tau_max, tau_d;
  if (be != 1.0f) {
    const float lb = m_log(be);
    alpha = (0.053f * lb + 0.31f) * m_pow(z, -0.012f * lb - 0.024f);
    tau0 = 0.285f * m_pow(be + 2.0f, 0.515f);
    tau_max = (nk < 2.0f) ? tau0 : 0.025f * m_pow(be + 2.0f, 2.6f) * m_pow(z, 2.83f);
    tau_d = (nk < 2.0f) ? tau0 : 0.036f * m_pow(be + 2.0f, 3.07f) * m_pow(z - 1.0f, 3.02f);
  } else {
    alpha = 0.267096f - 0.375571f * m_exp(-0.0838237f * nk);
    tau0 = 0.460277f + 0.298913f * m_exp(-0.0705314f * nk);
    tau_max = (nk < 4.0f) ? tau0 : 0.0156137f * m_pow(nk, 3.18849f);
    tau_d = (nk < 4.0f) ? tau0 : 0.0740131f * m_pow(nk, 3.18363f);
  }
  const float pa = m_pow(tau_max, alpha), p0 = m_pow(tau0, alpha);
  const float pam1 = m_pow(tau_max, alpha - 1.0f), p0m1 = m_pow(tau0, alpha - 1.0f);
  const float c1 = pa - p0, cm1 = pam1 - p0m1;
  const float rcm1c1 = (c1 == 0.0f) ? (alpha - 1.0f) / alpha / tau0 : cm1 / c1;
  const float At = 1.0f - g;
  const float Adt = At * alpha / (alpha - 1.0f);
  const float Bdt = Adt * rcm1c1;
  const float normdt = Bdt + g / tau_d;
  PcdDev d;
  d.At_ = c1 / At; d.Dt_ = p0; d.Ct_ = -1.0f / alpha;
  d.Adt_ = normdt * c1 / Adt; d.Bdt_ = Bdt / normdt; d.Cdt_ = -1.0f / (alpha - 1.0f); d.Ddt_ = p0m1;
  d.tau_d_inv = 1.0f / tau_d; d.one_minus_g = 1.0f - g; d.normdt = normdt;
  d.pad_[0] = d.pad_[1] = 0.f;
  return d;
}

// Partner law of a new entanglement.  Monodisperse: the ensemble's p_cd.
// Per-chain N_K: p_cd of a partner chain drawn uniformly from the ensemble.
// GEX background: partner mass from the inverse table (linear interpolation
// at u / step), the CD-weighted table for CD-created entanglements.
__device__ __forceinline__ PcdDev partner_pcd(const EnsDev& E, uint32_t w, bool cd_created) {
  if (E.gex) {
    const float* T = cd_created ? E.gex_Md : E.gex_M;
    const int n = cd_created ? E.gex_nd : E.gex_n;
    const float x = __fdiv_rn(u01(w), cd_created ? E.gex_step_d : E.gex_step);
    int i = (int)floorf(x);
    float di = __fsub_rn(x, (float)i);
    if (i > n - 2) { i = n - 2; di = 1.0f; }
    const float mw = __fadd_rn(__fmul_rn(__ldg(&T[i]), __fsub_rn(1.0f, di)), __fmul_rn(__ldg(&T[i + 1]), di));
    return pcd_from_nk(E.beta, __fmul_rn(mw, E.gex_scale));
  }
  if (!E.poly) return E.pcd;
  const uint32_t idx = __umulhi(w, (uint32_t)E.n_chains);
  return E.pcd_by_nk[__ldg(&E.nk_chain[idx])];
}

// Shift components of the pair (strand j, strand j+1), ensemble_kernel.cu:149-179:
// wp moves a Kuhn step from strand j+1 into strand j, wm the reverse.
// a = NT[N1], b = NT[N2].
// SHORT: by m_exp_lt88, *ok cleared when the exponent is out of its range.
template <bool SHORT>
__device__ __forceinline__ float shift_plus(const EnsDev& E, int N1, float q1, int N2, float q2, const float4& a,
                                            const float4& b, bool* ok = nullptr) {
  const bool z1 = (q1 == 0.0f), z2 = (q2 == 0.0f);
  const int i = (z1 ? 4 * N1 + 1 : 2 * N1) + (z2 ? 4 * N2 - 1 : 2 * N2);
  const float t2 = __fmul_rn(q2, b.y);
  const float arg = __fmaf_rn(q1, a.x, -t2);
  const float pw = __fmul_rn(z1 ? 1.0f : a.z, z2 ? 1.0f : b.w);
  if (SHORT) *ok = *ok && arg < kExpMost;
  const float w = __fmul_rn(__fmul_rn(__ldg(&E.FRIC[i]), pw), SHORT ? m_exp_lt88(arg) : m_exp(arg));
  return (N2 > 1) ? w : 0.0f;
}
template <bool SHORT>
__device__ __forceinline__ float shift_minus(const EnsDev& E, int N1, float q1, int N2, float q2, const float4& a,
                                             const float4& b, bool* ok = nullptr) {
  const bool z1 = (q1 == 0.0f), z2 = (q2 == 0.0f);
  const int i = (z1 ? 4 * N1 - 1 : 2 * N1) + (z2 ? 4 * N2 + 1 : 2 * N2);
  const float t1 = __fmul_rn(q1, a.y);
  const float arg = __fmaf_rn(q2, b.x, -t1);
  const float pw = __fmul_rn(z1 ? 1.0f : a.w, z2 ? 1.0f : b.z);
  if (SHORT) *ok = *ok && arg < kExpMost;
  const float w = __fmul_rn(__fmul_rn(__ldg(&E.FRIC[i]), pw), SHORT ? m_exp_lt88(arg) : m_exp(arg));
  return (N1 > 1) ? w : 0.0f;
}

// One of the two shift components, chosen per lane without divergence:
// minus = false gives shift_plus, minus = true shift_minus, with the same
// operations in the same order on selected operands (one exponential per lane).
// *ok: the exponent is below kExpMost (else the result is not used).
__device__ __forceinline__ float shift_comp(const EnsDev& E, bool minus, int N1, float q1, int N2, float q2,
                                            const float4& a, const float4& b, bool* ok) {
  const bool z1 = (q1 == 0.0f), z2 = (q2 == 0.0f);
  const int i = (z1 ? 4 * N1 + (minus ? -1 : 1) : 2 * N1) + (z2 ? 4 * N2 + (minus ? 1 : -1) : 2 * N2);
  const float u = minus ? q2 : q1, ux = minus ? b.x : a.x;
  const float v = minus ? q1 : q2, vy = minus ? a.y : b.y;
  const float arg = __fmaf_rn(u, ux, -__fmul_rn(v, vy));
  const float pw = __fmul_rn(z1 ? 1.0f : (minus ? a.w : a.z), z2 ? 1.0f : (minus ? b.z : b.w));
  *ok = arg < kExpMost;
  const float w = __fmul_rn(__fmul_rn(__ldg(&E.FRIC[i]), pw), m_exp_lt88(arg));
  return ((minus ? N1 : N2) > 1) ? w : 0.0f;
}

// status flags of a component: bit0 NaN, bit1 inf
__device__ __forceinline__ int comp_bad(float x) {
  return (x != x) ? 1 : ((__float_as_uint(x) == 0x7f800000u) ? 2 : 0);
}

struct Corr0 {  // correlator level-0 counters of the resident chain
  int ins, navg;
  long long nins;
  float a0, a1, a2;  // block sum (stress) or first value of the block (MSD)
  float r1x;         // MSD mode: first entanglement in the lab frame
  float r1y, r1z;
  long long k_next, t_next;
};

__host__ __device__ inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// ---- time slices (EnsDev::subs)
// End of slice `sub` of a launch window
__device__ __forceinline__ long long slice_end(const EnsDev& E, int sub) {
  const long long a = E.t_begin_ticks, b = E.t_end_ticks;
  return (sub + 1 >= E.subs || b <= a) ? b : a + (b - a) / E.subs * (sub + 1);
}
// Slices of the chain that are done; what the SM that ran the last one wrote is
// visible after it (by every lane that synchronises with this one)
__device__ __forceinline__ unsigned slices_done(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// (one lane, after the chain's lanes have synchronised on their stores)
__device__ __forceinline__ void slices_set(unsigned* p, unsigned v) {
  __threadfence();
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Position of a CD creation inside a strand of N1 Kuhn steps
// (ensemble_kernel.cu:386: newn = floor(0.5 + pr (N1 - 2) / w) + 1) on the
// quantised values r < w: x = floor((2 r (N1 - 2) + w) / (2 w)), exactly.  An
// FP32 estimate from the leading 24 bits of r and w (32-bit conversions only)
// is corrected with 128-bit integer products, so no FP64 operation is needed
// (sm_103a's FP64 divide costs about 430 cycles).  x stays in [0, N1 - 2]; the
// estimate is within one of it, and each correction loop moves x towards it.
__device__ __forceinline__ int split_pos(unsigned long long r, unsigned long long w, int N1) {
  const unsigned m = (unsigned)max(N1 - 2, 0);
  if (m == 0u || w == 0ull) return 0;
  // numerator 2 r m + w as nh:nl
  unsigned long long nl = r * m, nh = __umul64hi(r, (unsigned long long)m);
  nh = (nh << 1) | (nl >> 63);
  nl <<= 1;
  nl += w;
  nh += (nl < w) ? 1ull : 0ull;
  const unsigned long long d = w << 1;  // w < 2^62
  const int sh = max(0, 40 - __clzll((long long)w));  // w >> sh < 2^24, r >> sh <= w >> sh
  const float ratio = __fdiv_rn((float)(unsigned)(r >> sh), (float)(unsigned)(w >> sh));
  int q = (int)__fmaf_rn(ratio, (float)m, 0.5f);
  q = min(max(q, 0), (int)m);
  // q d as ph:pl; step q down while q d > num, then up while (q + 1) d <= num
  unsigned long long pl = (unsigned long long)q * d, ph = __umul64hi((unsigned long long)q, d);
  while (ph > nh || (ph == nh && pl > nl)) {
    ph -= (pl < d) ? 1ull : 0ull;
    pl -= d;
    --q;
  }
  for (;;) {
    const unsigned long long l2 = pl + d, h2 = ph + ((l2 < pl) ? 1ull : 0ull);
    if (h2 > nh || (h2 == nh && l2 > nl)) break;
    pl = l2;
    ph = h2;
    ++q;
  }
  return q;
}

}  // namespace dsm
