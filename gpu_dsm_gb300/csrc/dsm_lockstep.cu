// Lockstep step kernel for monodisperse equilibrium ensembles (sm_103a).
//
// Most kMC events are slides (N_K = 200: 94 %).  A slide warp runs 8 chains with
// 4 lanes each (4 chains with 8 lanes where slots are long) and does one event of
// all of them per round, every lane on the same instruction, so that one
// instruction stream serves 8 chains: 172 warp instructions per event at
// N_K = 200 without G(t) (198 with it), against 301 of the 16-lane tiles of
// dsm_kernels.cu.  A tile's rare paths (a creation runs 4600 cycles) would hold
// up the whole warp here; so whatever is not a slide -- creations and
// destructions, samples, the end of a window, the next chain, full rate passes --
// is posted to the service warps of the same block, through bits in shared
// memory, and the chain's lanes sit the rounds out until it is done.
//
// What bounds it: the rounds of a slide warp (about 650 dependent instructions)
// and the instruction cache.  An SM fetches up to 32 KB of code at one
// instruction per cycle and the next 96 KB at 2.7 cycles each; the slide loop
// (12 KB), the creations and destructions (10 KB) and the samples just about
// fill it (with G(t) a quarter of the stalls are waits for instructions, 2.1 warps
// per issue; without, 0.7).  Hence one copy
// of the random words, of the full rate pass and of the correlator (which takes
// kCorrBuf samples at a time), rare code kept rolled, and two service warps per
// two slide warps: with three or four, more code is in flight at once and the
// kernel slows down (N_K = 200 with G(t): 2.98e9, 2.89e9, 2.45e9 events/s).
//
// Chains resident per SM: the strand vectors Q are not in shared memory (only
// creations, destructions and samples read them, in the service warps, from L2),
// which leaves 24 bytes per strand: 60 chains per SM at N_K = 200 instead of 32.
// Four lanes per chain against eight at that size: 3.87e9 against 3.17e9 events/s
// without G(t).  4.10e9 now without G(t), 3.15e9 with it (500 tau).
//
// Trajectories, samples and sums are those of dsm_kernels.cu bit for bit.
#include <cstdint>

#include <cuda_runtime.h>

#include "dsm_device.cuh"
#include "dsm_internal.h"
#include "dsm_math.cuh"

namespace dsm {

namespace {

// What a slide warp asks a service warp for
enum : int { RQ_STRUCT = 1, RQ_FULL = 4, RQ_TIME = 8, RQ_STALL = 16, RQ_LOAD = 32 };

// Scalars of a resident chain, handed between its slide lanes and a service warp
struct __align__(16) Hdr {
  unsigned long long tot, etot;  // sum of all rates; of the chain-end rates
  long long T, t_chk;            // chain time; the next time a service warp has to see
  uint64_t step, hash;
  unsigned long long r, wsel;    // RQ_STRUCT: remainder of the pick within the component (jj < 0: within the chain
                                 // ends) and, of a creation, the component's rate (0: a destruction)
  int rq, jj;                    // request; picked pair (-1: chain end) or stall code
  int Z, S, left, fresh;         // strands (0: slot out of work), scale, events until the next look, what is new
                                 // (bit 0 the chain, bit 1 the rates)
  int e, c, stall, cap;
  int zlim;
  float wz1;
  long long t_end, step_lim, lim0;
  int sub, pend;                 // time slice of the resident chain; item that waits for its chain, plus one
};

struct LCorr : Corr0 {
  long long nbuf;  // samples in the chain's buffer
};

// Request and completion bits of a block's slots; per warp, what lock_moved saw last
struct Ctl {
  unsigned req, done, dead, pad_;
  unsigned seen[4];
};

// Shared-memory slot of one chain.  The strand vectors Q stay in HBM (L2), in
// the chain's own conformation entries: strand s is entry id(s), and a creation
// takes the first free entry, so no vector moves while the chain is resident.
struct LSlot {
  unsigned long long* R;  // quantised pair totals
  int4* C;                // per strand {shift +1 rate of the pair, Q^2, CD lifetime rate, N | id << 16} (floats as bits)
  unsigned long long* B;  // prefix of the pair totals at the sub-chunk boundaries
  Hdr* h;
  LCorr* k0;              // correlator level-0 counters
};

constexpr size_t kLockHead = (sizeof(Hdr) + sizeof(LCorr) + 15) / 16 * 16;  // C is read 16 bytes at a time
static_assert(sizeof(Hdr) % 16 == 0 && sizeof(Ctl) == 32, "slot alignment");

__host__ __device__ inline size_t lock_bytes(int slot_cap, int subs, int sb) {
  size_t b = ((size_t)slot_cap + 1) * 16 + kLockHead;
  b += ((size_t)slot_cap + sb) * 8;  // a pick reads up to one sub-chunk past the last pair
  b += ((size_t)subs + 1) * 8;
  return align_up(b, 16);
}

__device__ __forceinline__ LSlot lock_slot(unsigned char* base, int slot_cap, int sb) {
  LSlot s;
  s.h = (Hdr*)base;
  s.k0 = (LCorr*)(base + sizeof(Hdr));
  s.C = (int4*)(base + kLockHead);
  s.R = (unsigned long long*)(s.C + slot_cap + 1);
  s.B = s.R + slot_cap + sb;
  return s;
}

__device__ __forceinline__ int strand_n(int w) { return w & 0xffff; }
__device__ __forceinline__ int strand_id(int w) { return (int)((unsigned)w >> 16); }

template <int G, class T>
__device__ __forceinline__ T gshfl(T v, int src) { return __shfl_sync(FULL_MASK, v, src, G); }
template <class T>
__device__ __forceinline__ T gxor(T v, int d) { return __shfl_xor_sync(FULL_MASK, v, d); }
template <class T>
__device__ __forceinline__ T wshfl(T v, int src) { return __shfl_sync(FULL_MASK, v, src); }
// bits of the chain's G lanes in a ballot
template <int G>
__device__ __forceinline__ unsigned gbits(unsigned b, int lane) { return (b >> (lane & ~(G - 1))) & ((1u << G) - 1u); }

// Random words of an event (one copy of the code for slides and services: the
// event loop's code has to stay in the instruction cache)
__device__ __noinline__ U4 lock_words(const EnsDev& E, uint32_t purpose, uint64_t ctr, int c) {
  return rng_at(E, purpose, ctr, (uint32_t)(ctr >> 32), (uint32_t)c);
}

// Chain-end component q (order and branches of end_comp in dsm_kernels.cu,
// ensemble_kernel.cu:219-260)
__device__ __forceinline__ float lock_end_comp(const float4* NE, bool cd, int q, int Z, const int4* C, float wz1) {
  const bool tail = (q == 0) || (q == 2) || (q == 4);
  const int Ne = strand_n(C[tail ? Z - 1 : 0].w);
  const int Nn = (Z >= 2) ? strand_n(C[tail ? Z - 2 : 1].w) : 1;
  const float4 e1 = __ldg(&NE[Ne]);
  const float4 e2 = __ldg(&NE[Nn]);
  const float cdc = cd ? e1.w : 0.0f;
  const float sdc = (Z == 1) ? wz1 : ((Ne == 1) ? 0.0f : e1.x);
  const float sdd = (Z == 1 || Ne != 1) ? 0.0f : ((Z == 2) ? e2.y : e2.z);
  return (q == 0) ? cdc : ((q <= 2) ? sdc : sdd);
}

__device__ __forceinline__ void lock_pair(const EnsDev& E, const LSlot& sl, int p, float o[4]) {
  const int4 c1 = sl.C[p], c2 = sl.C[p + 1];
  const int N1 = strand_n(c1.w), N2 = strand_n(c2.w);
  const float q1 = __int_as_float(c1.y), q2 = __int_as_float(c2.y);
  const float4 a = __ldg(&E.NT[N1]), b = __ldg(&E.NT[N2]);
  o[0] = E.cd_flag ? __int_as_float(c1.z) : 0.0f;
  o[1] = shift_plus<false>(E, N1, q1, N2, q2, a, b);
  o[2] = shift_minus<false>(E, N1, q1, N2, q2, a, b);
  o[3] = E.cd_flag ? __ldg(&E.NE[N1]).w : 0.0f;
}

// Full rate pass of one chain: every pair and the chain ends quantised at scale
// 2^S; S drops on overflow (full_rates_body of dsm_kernels.cu, equilibrium).
// Returns the scale; *flags_out NaN / inf bits, *etot the chain-end total.
__device__ __noinline__ int lock_full_rates(const EnsDev& E, const LSlot sl, int Z, int S, float wz1,
                                            int* flags_out, unsigned long long* etot) {
  const int lane = threadIdx.x & 31;
  const int np = Z - 1;
  int emax = -200, flags = 0;
  unsigned mx = 0u;
  unsigned long long eq = 0;
  int Snew = S;
  const float ev = lane < NEND ? lock_end_comp(E.NE, E.cd_flag != 0, lane, Z, sl.C, wz1) : 0.0f;
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {  // a second pass when the scale changed
    const float sf = pow2f(Snew);
#pragma unroll 1
    for (int p = lane; p < np; p += 32) {
      float o[4];
      lock_pair(E, sl, p, o);
      unsigned long long tot = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const unsigned b = __float_as_uint(o[q]);
        mx = max(mx, b & 0x7fffffffu);
        if (b == 0x7f800000u) flags |= 2;
        tot += quant(o[q], sf);
      }
      sl.R[p] = tot;
      sl.C[p].x = __float_as_int(o[1]);
    }
    eq = quant(ev, sf);
    if (pass == 1) break;
    if (mx > 0x7f800000u) flags |= 1;
    if (mx >= 0x00800000u) emax = max(emax, (int)(mx >> 23) - 127);
    if (lane < NEND) emax = max(emax, fexp(ev));
    emax = __reduce_max_sync(FULL_MASK, emax);
    flags = __reduce_or_sync(FULL_MASK, flags);
    if (flags != 0 || emax + S <= LIMIT_E) break;
    Snew = LIMIT_E - emax;
  }
  eq += __shfl_xor_sync(FULL_MASK, eq, 4);
  eq += __shfl_xor_sync(FULL_MASK, eq, 2);
  eq += __shfl_xor_sync(FULL_MASK, eq, 1);
  *etot = wshfl(eq, 0);
  __syncwarp();
  *flags_out = flags;
  return Snew;
}

// The buffered samples of a chain into its multi-tau correlator by one warp,
// level by level (corr_samples and corr_push_levels of dsm_kernels.cu: the same
// values into every sum in the same order).  A lane owns a lag and runs over the
// samples, so its sum stays in a register (FP32 compensated at level 0, FP64
// above); the block averages of a level are the samples of the next.
//
// The samples are correlated kCorrBuf at a time because the code of the event
// loop, of the service and of the correlator together do not fit the 32 KB
// instruction cache of an SM: taken at every sample, the lags and level pushes
// evicted the event loop (N_K = 200, p = 64, m = 8: 2.82e9 events/s with 32
// samples at a time, 2.85e9 with 64, 2.85e9 with 128).
template <bool MSD>
__device__ __noinline__ void lock_flush(const EnsDev& E, int c, LCorr* k0) {
  int n = (int)k0->nbuf;
  const int lane = threadIdx.x & 31;
  const int L = E.corr_levels, p = E.corr_p, m = E.corr_m;
  float* const in = E.corr_buf + (size_t)c * (kCorrBuf * 3);
#pragma unroll 1
  for (int k = 0; k < L && n > 0; ++k) {
    const size_t lk = (size_t)c * L + k;
    float* sh = E.corr_shift + lk * p * 3;
    float* av = E.corr_avg + lk * 3;
    int ins, navg;
    long long nins;
    float a0, a1, a2;
    if (k == 0) {
      ins = k0->ins; navg = k0->navg; nins = k0->nins;
      a0 = k0->a0; a1 = k0->a1; a2 = k0->a2;
    } else {
      const int4 cn = E.corr_cnt[lk];
      ins = cn.x; navg = cn.y;
      nins = (long long)(unsigned)cn.w << 32 | (unsigned)cn.z;
      a0 = av[0]; a1 = av[1]; a2 = av[2];
    }
#pragma unroll 1
    for (int j = (k == 0 ? 0 : p / m) + lane; j < p; j += 32) {
      float2 s = make_float2(0.f, 0.f);
      double acc = 0.0;
      if (k == 0) s = E.corr_comp[(size_t)c * p + j];
      else acc = E.corr_acc[lk * p + j];
      const int first = (int)max(0ll, j - nins);
      auto term = [&](int i) {  // sample i times the one j samples before it
        const float w0 = in[3 * i], w1 = in[3 * i + 1], w2 = in[3 * i + 2];
        int q = ins + i - j;
        if (q < 0) q += p;
        const float* x = i >= j ? in + 3 * (i - j) : sh + 3 * q;
        if (MSD) {
          const float d0 = __fsub_rn(w0, x[0]), d1 = __fsub_rn(w1, x[1]), d2 = __fsub_rn(w2, x[2]);
          return __fmaf_rn(d2, d2, __fmaf_rn(d1, d1, __fmul_rn(d0, d0)));
        }
        return __fmaf_rn(w2, x[2], __fmaf_rn(w1, x[1], __fmul_rn(w0, x[0])));
      };
      if (k == 0) {
#pragma unroll 2
        for (int i = first; i < n; ++i) {
          const float y = __fsub_rn(term(i), s.y);
          const float t = __fadd_rn(s.x, y);
          s.y = __fsub_rn(__fsub_rn(t, s.x), y);
          s.x = t;
        }
      } else {
#pragma unroll 1
        for (int i = first; i < n; ++i) acc += (double)term(i);
      }
      if (k == 0) E.corr_comp[(size_t)c * p + j] = s;
      else E.corr_acc[lk * p + j] = acc;
    }
    __syncwarp();
    // the last p samples into the shift register
#pragma unroll 1
    for (int i = max(0, n - p) + lane; i < n; i += 32) {
      const int q = 3 * ((ins + i) % p);
      sh[q] = in[3 * i]; sh[q + 1] = in[3 * i + 1]; sh[q + 2] = in[3 * i + 2];
    }
    // block sums (MSD: the first value of a block) in sample order
    int nout = 0;
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      const float w0 = in[3 * i], w1 = in[3 * i + 1], w2 = in[3 * i + 2];
      if (!MSD) {
        a0 = __fadd_rn(a0, w0); a1 = __fadd_rn(a1, w1); a2 = __fadd_rn(a2, w2);
      } else if (navg == 0) {
        a0 = w0; a1 = w1; a2 = w2;
      }
      if (++navg == m) {
        if (!MSD) {
          const float rm = (float)m;
          a0 = __fdiv_rn(a0, rm); a1 = __fdiv_rn(a1, rm); a2 = __fdiv_rn(a2, rm);
        }
        __syncwarp();  // every lane has read sample i >= nout
        if (lane == 0) { in[3 * nout] = a0; in[3 * nout + 1] = a1; in[3 * nout + 2] = a2; }
        ++nout;
        navg = 0;
        a0 = a1 = a2 = 0.f;
      }
    }
    ins = (ins + n) % p;
    nins += n;
    if (lane == 0) {
      if (k == 0) {
        k0->ins = ins; k0->navg = navg; k0->nins = nins;
        k0->a0 = a0; k0->a1 = a1; k0->a2 = a2;
      } else {
        E.corr_cnt[lk] = make_int4(ins, navg, (int)(unsigned)(nins & 0xffffffffll), (int)(unsigned)(nins >> 32));
        av[0] = a0; av[1] = a1; av[2] = a2;
      }
    }
    __syncwarp();
    n = nout;
  }
  if (threadIdx.x % 32 == 0) k0->nbuf = 0;
  __syncwarp();
}

// Level 0's counters and running average from HBM, and back (one lane)
__device__ __forceinline__ void lock_corr_load(const EnsDev& E, int c, LCorr* k0) {
  const size_t l0 = (size_t)c * E.corr_levels;
  const int4 cn = E.corr_cnt[l0];
  k0->ins = cn.x; k0->navg = cn.y;
  k0->nins = ((long long)(unsigned)cn.w) << 32 | (unsigned)cn.z;
  k0->a0 = E.corr_avg[l0 * 3 + 0]; k0->a1 = E.corr_avg[l0 * 3 + 1]; k0->a2 = E.corr_avg[l0 * 3 + 2];
}
__device__ __forceinline__ void lock_corr_store(const EnsDev& E, int c, const LCorr& k0) {
  const size_t l0 = (size_t)c * E.corr_levels;
  E.corr_cnt[l0] = make_int4(k0.ins, k0.navg, (int)(unsigned)(k0.nins & 0xffffffffll), (int)(unsigned)(k0.nins >> 32));
  E.corr_avg[l0 * 3 + 0] = k0.a0; E.corr_avg[l0 * 3 + 1] = k0.a1; E.corr_avg[l0 * 3 + 2] = k0.a2;
}

// End of a chain's launch: the buffered samples, then the compensated level-0
// sums into the FP64 ones (one warp)
template <bool MSD>
__device__ __forceinline__ void lock_corr_out(const EnsDev& E, int c, LCorr* k0) {
  lock_flush<MSD>(E, c, k0);
  const int p = E.corr_p;
  const size_t l0 = (size_t)c * E.corr_levels;
  const float2* Cacc = E.corr_comp + (size_t)c * p;
#pragma unroll 1
  for (int j = threadIdx.x % 32; j < p; j += 32) {
    const float2 a = Cacc[j];
    E.corr_acc[l0 * p + j] += (double)a.x - (double)a.y;
  }
}

// Centre of mass of the chain (chain_com of dsm_kernels.cu in the arithmetic of
// its 16-lane tile; both half warps compute the same)
__device__ __forceinline__ void lock_com(const EnsDev& E, const LSlot& sl, int Z, int c, float* v) {
  const int l = threadIdx.x & 15;
  const float4* Q = E.QN + (size_t)c * E.cap;
  float cm[3] = {0.f, 0.f, 0.f}, pf[3] = {0.f, 0.f, 0.f};
#pragma unroll 1
  for (int base = 0; base < Z; base += 16) {
    const int s = base + l;
    const bool in = s < Z;
    const int w = in ? sl.C[s].w : 0;
    const float4 q = in ? Q[strand_id(w)] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float n = (float)strand_n(w);
    const float qq[3] = {q.x, q.y, q.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      float ix = qq[d];
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {
        const float u = __shfl_up_sync(FULL_MASK, ix, o, 16);
        if (l >= o) ix = __fadd_rn(ix, u);
      }
      float ex = __shfl_up_sync(FULL_MASK, ix, 1, 16);
      if (l == 0) ex = 0.f;
      cm[d] = __fmaf_rn(__fadd_rn(__fadd_rn(pf[d], ex), __fmul_rn(0.5f, qq[d])), n, cm[d]);
      pf[d] = __fadd_rn(pf[d], __shfl_sync(FULL_MASK, ix, 15, 16));
    }
  }
  const float nk = (float)(E.poly ? __ldg(&E.nk_chain[c]) : E.nk);
  const float r1[3] = {sl.k0->r1x, sl.k0->r1y, sl.k0->r1z};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    float x = cm[d];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) x = __fadd_rn(x, __shfl_xor_sync(FULL_MASK, x, o));
    v[d] = __fadd_rn(__fdiv_rn(x, nk), r1[d]);
  }
}

// One due sample: the shear stresses or the centre of mass (corr_samples of
// dsm_kernels.cu; strand i goes to partial i mod 16) into the chain's sample
// buffer.  Returns the samples now in the buffer.
template <bool MSD>
__device__ __forceinline__ int lock_sample(const EnsDev& E, const LSlot& sl, int Z, int c) {
  const int lane = threadIdx.x & 31;
  LCorr& k0 = *sl.k0;
  float v[3];
  if (MSD) {
    lock_com(E, sl, Z, c, v);
  } else {
    v[0] = v[1] = v[2] = 0.f;
    const float4* Q = E.QN + (size_t)c * E.cap;
#pragma unroll 4
    for (int s = lane & 15; s < Z; s += 16) {
      const int cw = sl.C[s].w;
      const float4 q = Q[strand_id(cw)];
      const float w = __ldg(&E.INV3N[strand_n(cw)]);
      v[0] = __fmaf_rn(-__fmul_rn(q.x, q.y), w, v[0]);
      v[1] = __fmaf_rn(-__fmul_rn(q.y, q.z), w, v[1]);
      v[2] = __fmaf_rn(-__fmul_rn(q.x, q.z), w, v[2]);
    }
    __syncwarp();
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) v[d] = __fadd_rn(v[d], __shfl_xor_sync(FULL_MASK, v[d], o));
  }
  const int n = (int)k0.nbuf;
  __syncwarp();
  if (lane == 0) {
    float* b = E.corr_buf + (size_t)c * (kCorrBuf * 3) + 3 * n;
    b[0] = v[0]; b[1] = v[1]; b[2] = v[2];
    k0.nbuf = n + 1;
    k0.k_next += 1;
    k0.t_next += E.dt_sample_ticks;
  }
  __syncwarp();
  return n + 1;
}

// split_pos of dsm_device.cuh in 64-bit integers: r < w < 2^48 and N1 < 2^14, so
// the numerator 2 r (N1 - 2) + w stays below 2^64.  The FP32 estimate is within
// one of the quotient.
__device__ __forceinline__ int lock_split(unsigned long long r, unsigned long long w, int N1) {
  const unsigned m = (unsigned)max(N1 - 2, 0);
  if (m == 0u || w == 0ull) return 0;
  const unsigned long long num = 2ull * r * m + w, d = w << 1;
  const int sh = max(0, 40 - __clzll((long long)w));  // w >> sh < 2^24, r >> sh <= w >> sh
  const float ratio = __fdiv_rn((float)(unsigned)(r >> sh), (float)(unsigned)(w >> sh));
  int q = min((int)__fmaf_rn(ratio, (float)m, 0.5f), (int)m);
  if ((unsigned long long)q * d > num) --q;
  if ((unsigned long long)(q + 1) * d <= num) ++q;
  return q;
}

// Which chain-end event remainder *rem of the chain-end rates picks
__device__ __noinline__ int lock_end_pick(const EnsDev& E, const LSlot& sl, int Z, float sf, float wz1,
                                          unsigned long long* rem, unsigned long long* wsel) {
  const int lane = threadIdx.x & 31;
  const unsigned long long ev =
      lane < NEND ? quant(lock_end_comp(E.NE, E.cd_flag != 0, lane, Z, sl.C, wz1), sf) : 0ull;
  int q = 0;
  unsigned long long r = *rem, w = wshfl(ev, 0);
#pragma unroll 1
  while (q < NEND - 1 && r >= w) {
    r -= w;
    ++q;
    w = wshfl(ev, q);
  }
  *rem = r;
  *wsel = w;
  return CDC_TAIL + q;
}
static_assert(CDC_TAIL + 1 == SDC_HEAD && CDC_TAIL + 2 == SDC_TAIL && CDC_TAIL + 3 == SDD_HEAD && CDC_TAIL + 4 == SDD_TAIL,
              "chain-end events in pick order");

// A creation or destruction picked by the chain's slide lanes, applied by the
// whole warp: the event of ensemble_kernel.cu:274-501 on whole strands, then
// the rates of the touched pairs.  Returns the event's code; *full: a rate left
// the fixed-point range; *ends: a strand next to a chain end changed.
template <bool MSD>
__device__ __forceinline__ uint32_t lock_struct(const EnsDev& E, const LSlot& sl, int& Z, int S, int cap, int c,
                                                uint64_t step, int j, unsigned long long rem,
                                                unsigned long long wsel, float wz1, bool* full, bool* ends) {
  const int lane = threadIdx.x & 31;
  const bool cd = E.cd_flag != 0;
  const float sf = pow2f(S);
  int evn = wsel != 0ull ? CDC_MID : CDD;
  if (j < 0) evn = lock_end_pick(E, sl, Z, sf, wz1, &rem, &wsel);
  uint32_t code = ((uint32_t)evn << 24) | (uint32_t)(j < 0 ? 0 : j);
  const bool destroy = evn == CDD || evn == SDD_HEAD || evn == SDD_TAIL;
  if (!destroy && Z >= cap) return code | (uint32_t)NULL_FLAG << 24;  // refused at capacity (ensemble_kernel.cu:380,423,451)
  *ends = !(j >= 2 && j + 3 < Z);
  int up0, upn, dir, lo, sa, na, nb = 0;  // strands sa (and sa + 1 of a creation) after the move
  int ia, ib = 0;                         // their entries of Q
  float4* Q = E.QN + (size_t)c * E.cap;
  float4 qa = make_float4(0.f, 0.f, 0.f, 0.f), qb = qa;
  float trate = 0.f;
  if (destroy) {
    const bool tail = evn == SDD_TAIL;
    sa = evn == CDD ? j : tail ? Z - 2 : 0;
    const int wa = sl.C[sa].w, wb = sl.C[sa + 1].w;
    ia = strand_id(wa);
    ib = strand_id(wb);  // freed
    const float4 a = Q[ia], b = Q[ib];
    // CDD merges strands j and j+1 (ensemble_kernel.cu:312-323); an end
    // destruction merges the one-step end strand into its neighbour
    na = (evn == CDD) ? strand_n(wa) + strand_n(wb) : strand_n(tail ? wa : wb) + 1;
    if (evn == CDD && j != 0 && j != Z - 2) {
      const float x = __fadd_rn(a.x, b.x), y = __fadd_rn(a.y, b.y), z = __fadd_rn(a.z, b.z);
      qa = make_float4(x, y, z, m_q2(x, y, z));
    }
    dir = tail ? 0 : -1;
    lo = sa + 1;
    up0 = evn == CDD ? j - 1 : tail ? Z - 3 : 0;
    upn = evn == CDD ? 2 : 1;
    if (MSD && lane == 0 && ((evn == CDD && j == 0) || evn == SDD_HEAD)) {
      // the first entanglement is now the old second one (eq_ensemble_kernel.cu:447-455,645-653)
      LCorr& k0 = *sl.k0;
      k0.r1x = __fadd_rn(k0.r1x, b.x); k0.r1y = __fadd_rn(k0.r1y, b.y); k0.r1z = __fadd_rn(k0.r1z, b.z);
    }
  } else {
    const bool cdc = evn == CDC_MID || evn == CDC_TAIL;
    const int sj = evn == CDC_MID ? j : evn == SDC_HEAD ? 0 : Z - 1;
    const int wj = sl.C[sj].w;
    const int N1 = strand_n(wj);
    ia = strand_id(wj);
    ib = strand_id(sl.C[Z].w);  // the first free entry
    const float4 qo = Q[ia];
    // even lanes the event's own words, odd lanes the creation's
    const U4 w = lock_words(E, (lane & 1) ? P_CREATE : P_EVENT, step, c);
    const uint32_t w2 = wshfl(w.z, 0);
    // lanes 0 and 1 a pair of normal deviates each, lane 2 the lifetime's power
    const uint32_t gx = wshfl(w.x, 1), gy = wshfl(w.y, 1), gz = wshfl(w.z, 1), gw = wshfl(w.w, 1);
    // (one N_K, no GEX background: the ensemble's own partner law)
    const PcdDev pp = E.pcd;
    const float pA = cdc ? pp.Adt_ : pp.At_, pD = cdc ? pp.Ddt_ : pp.Dt_, pC = cdc ? pp.Cdt_ : pp.Ct_;
    const float pB = cdc ? pp.Bdt_ : pp.one_minus_g;
    const float u = u01(w2);
    const float base = __fmaf_rn(u, pA, pD);
    const float lg = m_log(lane == 0 ? u01(gx) : lane == 1 ? u01(gz) : base);
    float sn, cs;
    m_sincos2pi((lane == 0 ? gy : gw) >> 8, &sn, &cs);
    // (other lanes' logarithms may be positive, a slow case of the square root)
    const float rr = __fsqrt_rn(lane < 2 ? __fmul_rn(-2.0f, lg) : 1.0f);
    const float ga = __fmul_rn(rr, cs), gb = __fmul_rn(rr, sn);
    const float pw = wshfl(m_exp(__fmul_rn(pC, lg)), 2);
    const float g0 = wshfl(ga, 0), g1 = wshfl(gb, 0), g2 = wshfl(ga, 1);
    trate = cd ? ((u < pB) ? pw : pp.tau_d_inv) : 0.0f;
    int newn = 0;
    if (cdc) {
      newn = lock_split(rem, wsel, N1) + 1;
      newn = max(1, min(N1 - 1, newn));
    }
    code |= (uint32_t)newn << 8;
    const bool inner = evn == CDC_MID && j > 0;
    const bool head = (evn == CDC_MID && j == 0) || evn == SDC_HEAD;
    const int nn = inner ? newn : head ? (evn == SDC_HEAD ? N1 - 1 : N1 - newn) : (evn == SDC_TAIL ? N1 - 1 : newn);
    const int nd = N1 - nn;
    float sg = __fsqrt_rn(__fdiv_rn(inner ? (float)(newn * (N1 - newn)) : (float)nn, inner ? (float)(3 * N1) : 3.0f));
    if (Z == 1) sg = 0.0f;  // (no pair: an end creation)
    const float x0 = __fmul_rn(g0, sg), y0 = __fmul_rn(g1, sg), z0 = __fmul_rn(g2, sg);
    if (inner) {
      const float ra = __fdiv_rn((float)newn, (float)N1);
      const float x = __fmaf_rn(qo.x, ra, x0), y = __fmaf_rn(qo.y, ra, y0), z = __fmaf_rn(qo.z, ra, z0);
      const float x2 = __fsub_rn(qo.x, x), y2 = __fsub_rn(qo.y, y), z2 = __fsub_rn(qo.z, z);
      sa = j; na = nn; nb = nd;
      qa = make_float4(x, y, z, m_q2(x, y, z));
      qb = make_float4(x2, y2, z2, m_q2(x2, y2, z2));
      dir = 1; lo = j; up0 = j - 1; upn = 3;
    } else {
      const float4 qn = make_float4(x0, y0, z0, m_q2(x0, y0, z0));
      upn = 2;
      if (head) {
        sa = 0; na = nd; nb = nn; qb = qn;
        dir = 1; lo = 0; up0 = 0;
        if (MSD && lane == 0) {  // the new first entanglement (eq_ensemble_kernel.cu:531-539,606-614)
          LCorr& k0 = *sl.k0;
          k0.r1x = __fsub_rn(k0.r1x, x0); k0.r1y = __fsub_rn(k0.r1y, y0); k0.r1z = __fsub_rn(k0.r1z, z0);
        }
      } else {
        sa = Z - 1; na = nn; nb = nd; qa = qn;
        dir = 0; lo = Z; up0 = Z - 2;
      }
    }
  }
  __syncwarp();
  // strands from lo on move one place up or down, 32 per round
  if (dir != 0) {
#pragma unroll 1
    for (int done = 0; done < Z - lo; done += 32) {
      const int s = dir > 0 ? Z - 1 - done - lane : lo + done + lane;
      const bool in = s >= lo && s < Z;
      int4 v = make_int4(0, 0, 0, 0);
      unsigned long long rr = 0;
      if (in) { v = sl.C[s]; rr = sl.R[s]; }
      __syncwarp();
      if (in) { sl.C[s + dir] = v; sl.R[s + dir] = rr; }
    }
    __syncwarp();
  }
  if (lane == 0) {
    // a creation: strand sa keeps entry ia, the new one takes ib; a
    // destruction: strand sa keeps ia, ib is the first free entry now
    sl.C[sa].y = __float_as_int(qa.w);
    sl.C[sa].w = na | ia << 16;
    Q[ia] = qa;
    if (destroy) {
      sl.C[Z - 1].w = ib << 16;
    } else {
      sl.C[sa].z = __float_as_int(trate);
      sl.C[sa + 1].y = __float_as_int(qb.w);
      sl.C[sa + 1].w = nb | ib << 16;
      Q[ib] = qb;
    }
  }
  Z += destroy ? -1 : 1;
  __syncwarp();
  // the touched pairs, four lanes each (update_pairs of dsm_kernels.cu)
  {
    const int k = lane & 3, p = up0 + (lane >> 2);
    const bool act = lane < 4 * upn && p >= 0 && p < Z - 1;
    const int pc = act ? p : 0;
    const int4 c1 = sl.C[pc], c2 = sl.C[pc + 1];
    const int N1 = act ? strand_n(c1.w) : 1, N2 = act ? strand_n(c2.w) : 1;
    bool ok;
    const float w = shift_comp(E, k == 2, N1, __int_as_float(c1.y), N2, __int_as_float(c2.y), __ldg(&E.NT[N1]),
                               __ldg(&E.NT[N2]), &ok);
    const float cde = k == 0 ? __int_as_float(c1.z) : __fmul_rn(E.prefact, (float)(N1 - 1));
    const float y = __fmul_rn((k == 1 || k == 2) ? w : (cd ? cde : 0.0f), sf);
    *full = __any_sync(FULL_MASK, act && !(ok && y < 281474976710656.0f));  // 2^(LIMIT_E+1); NaN too
    const unsigned long long v = f2u64_rn(y);
    unsigned long long tot = v + __shfl_xor_sync(FULL_MASK, v, 1);
    tot += __shfl_xor_sync(FULL_MASK, tot, 2);
    if (act && k == 0) sl.R[p] = tot;
    if (act && k == 1) sl.C[p].x = __float_as_int(w);
  }
  __syncwarp();
  return code;
}

// Every 4096 events of a chain: a sign that the launch moves (lock_moved), and
// whether it is to be aborted
__device__ __noinline__ bool lock_look(const EnsDev* ens, const volatile int* abort_flag) {
  if ((threadIdx.x & 31) == 0) atomicAdd(&ens[0].counters[3], 1ull);
  return abort_flag != nullptr && wshfl(*abort_flag, 0) != 0;
}

// Everything a chain needs before its next slide, by one service warp: the
// requested event, due samples, the way back to HBM and the next chain, rate
// passes, the prefix of the pair totals.  False: the slot's next chain is not back
// from its earlier time slice yet, ask again.
template <int CK, int SUBS, int SB>
__device__ __forceinline__ bool lock_serve(const EnsDev* __restrict__ ens, int n_ens,
                                           const long long* __restrict__ prefix, long long n_items, int subs,
                                           unsigned int* work, int slot_cap, const LSlot& sl, unsigned bit, Ctl* ctl,
                                           const volatile int* abort_flag, int* status, const StepList& lst) {
  constexpr bool CORR = CK != 0, MSD = CK == 2;
  const int lane = threadIdx.x & 31;
  Hdr& h = *sl.h;
  const int rq = h.rq;
  bool live = !(rq & RQ_LOAD);
  bool fresh = false, aborted = false, full = (rq & RQ_FULL) != 0, ends = false;
  int e = h.e, c = h.c, Z = h.Z, S = h.S, stall = (rq & RQ_STALL) ? h.jj : h.stall, cap = h.cap, zlim = h.zlim;
  long long T = h.T, t_end = h.t_end, step_lim = h.step_lim, lim0 = h.lim0;
  uint64_t step = h.step, hash = h.hash;
  unsigned long long etot = h.etot;
  float wz1 = h.wz1;
  if (rq & RQ_STRUCT) {
    bool fl = false, en = false;
    const uint32_t code = lock_struct<MSD>(ens[e], sl, Z, S, cap, c, step, h.jj, h.r, h.wsel, wz1, &fl, &en);
    full = full || fl;
    ends = en;
    hash = (hash ^ (uint64_t)code) * 0x100000001B3ull;
    ++step;
  }
  if (live && (step & 4095) == 0) aborted = lock_look(ens, abort_flag);
#pragma unroll 1
  for (;;) {
    if (live) {
      if (CORR && stall == 0 && !aborted) {
#pragma unroll 1
        while (sl.k0->k_next < ens[e].nsamples && T > sl.k0->t_next)
          if (lock_sample<MSD>(ens[e], sl, Z, c) == kCorrBuf) lock_flush<MSD>(ens[e], c, sl.k0);
      }
      // window, event limit, full slot, stall, abort: the chain goes back to HBM
      if (T >= t_end || (long long)step >= step_lim || Z >= zlim || stall != 0 || aborted) {
        const EnsDev& E = ens[e];
        if (stall == 0 && !aborted && T < t_end && (long long)step >= step_lim && step_lim != lim0) stall = ST_WATCHDOG;
        const bool deferred = cap > slot_cap && Z >= slot_cap && stall == 0 && T < t_end && (long long)step < step_lim;
        const size_t ecap = (size_t)E.cap;
        float4* wq = E.QN + (size_t)c * ecap;
        float* wt = E.tau + (size_t)c * ecap;
        // the vectors into strand order, through the pair totals (no longer needed)
#pragma unroll 2
        for (int s = lane; s < Z; s += 32) {
          const float4 q = wq[strand_id(sl.C[s].w)];
          sl.R[s] = (unsigned long long)__float_as_uint(q.y) << 32 | __float_as_uint(q.x);
          sl.C[s].x = __float_as_int(q.z);
        }
        __syncwarp();
#pragma unroll 2
        for (int s = lane; s < Z; s += 32) {
          const unsigned long long xy = sl.R[s];
          const int4 v = sl.C[s];
          wq[s] = make_float4(__uint_as_float((unsigned)xy), __uint_as_float((unsigned)(xy >> 32)), __int_as_float(v.x),
                              (float)strand_n(v.w));
          wt[s] = (s < Z - 1) ? __int_as_float(v.z) : 0.0f;
        }
        // the chain's last time slice of the launch: else buffered samples and
        // sums stay for the next one
        const bool last = h.sub + 1 >= subs || deferred || aborted;
        if (CORR && last) lock_corr_out<MSD>(E, c, sl.k0);
        if (lane == 0) {
          ChainState* cs = &E.cs[c];
          // the launch's start values are still in HBM: events done, stored scale
          const unsigned long long done = step - cs->step;
          // a rescale at load is kept only if an event followed (as in the oracle)
          if (done > 0) cs->S = S;
          cs->Z = Z; cs->stall = stall; cs->dt_prev = 0.0f;
          cs->T = T; cs->step = step; cs->hash = hash;
          if (CORR) {
            const LCorr& k0 = *sl.k0;
            cs->k_next = k0.k_next;
            lock_corr_store(E, c, k0);
            if (!last) E.slice[c].nbuf = (unsigned)k0.nbuf;
            if (MSD) { cs->r1[0] = k0.r1x; cs->r1[1] = k0.r1y; cs->r1[2] = k0.r1z; }
          }
          atomicAdd(&E.counters[0], done);
          if (aborted) atomicOr(status, 1);
          if (deferred) {
            lst.defer[atomicAdd(lst.n_defer, 1u)] = (int)(prefix[e] + c);
            atomicAdd(&E.counters[2], 1ull);
          } else if (last) {
            atomicAdd(&E.counters[1], 1ull);
          }
        }
        live = false;
        __syncwarp();
        if (subs > 1 && lane == 0) slices_set(&E.slice[c].done, deferred || aborted ? kMoved : (unsigned)h.sub + 1u);
      }
    }
    if (!live) {  // the next chain of the work list
      unsigned int item = 0;
      if (lane == 0) {
        item = h.pend != 0 ? (unsigned)h.pend - 1u : atomicAdd(work, 1u);
        h.pend = 0;
      }
      item = wshfl(item, 0);
      const bool none = (long long)item >= n_items * subs;
      const bool stop = !none && abort_flag != nullptr && wshfl(*abort_flag, 0) != 0;
      if (none || stop) {
        if (lane == 0) {
          if (stop) atomicOr(status, 1);
          h.Z = 0;
          atomicOr(&ctl->dead, bit);
        }
        return true;
      }
      int sub = 0;
      unsigned int idx = item;
      if (subs > 1) {
        sub = (int)(item / (unsigned)n_items);
        idx -= (unsigned)sub * (unsigned)n_items;
      }
      const long long gid = lst.order != nullptr ? (long long)lst.order[idx] : (long long)idx;
      e = 0;
#pragma unroll 1
      while (e + 1 < n_ens && prefix[e + 1] <= gid) ++e;
      const EnsDev& E = ens[e];
      c = (int)(gid - prefix[e]);
      if (sub > 0) {
        // the chain's earlier slice: a slot of this block may be running it, so
        // the request is posted again instead of waiting here
        const unsigned done = wshfl(slices_done(&E.slice[c].done), 0);
        __syncwarp();
        if (done < (unsigned)sub) {
          if (lane == 0) {
            h.pend = (int)item + 1;
            h.rq = RQ_LOAD;
          }
          return false;
        }
        if (done == kMoved) continue;
      }
      const ChainState st = E.cs[c];
      if (st.Z > slot_cap) {  // does not fit at all: hand it to a larger slot
        if (lane == 0) {
          lst.defer[atomicAdd(lst.n_defer, 1u)] = (int)gid;
          atomicAdd(&E.counters[2], 1ull);
          if (subs > 1) slices_set(&E.slice[c].done, kMoved);
        }
        continue;
      }
      cap = E.cap;
      zlim = cap > slot_cap ? slot_cap : 0x7fffffff;
      Z = st.Z; S = st.S; stall = st.stall; T = st.T; step = st.step; hash = st.hash;
      t_end = sub + 1 < subs ? slice_end(E, sub) : E.t_end_ticks;
      lim0 = E.step_limit;
      // (the event cap counts from the start of the launch)
      const long long wd = E.watchdog_events;
      long long first = (long long)step;
      if (subs > 1) {
        if (sub > 0) first = (long long)E.slice[c].step0;
        else if (lane == 0) E.slice[c].step0 = step;
      }
      step_lim = (wd < lim0 - first) ? first + wd : lim0;
      if (lane == 0) h.sub = sub;
      wz1 = __double2float_rn(__ddiv_rn(1.0, __dmul_rn(E.beta_d, (double)st.nk)));
      const size_t ecap = (size_t)cap;
      const float4* gq = E.QN + (size_t)c * ecap;
      const float* gt = E.tau + (size_t)c * ecap;
#pragma unroll 2
      for (int s = lane; s <= slot_cap; s += 32) {
        const bool in = s < Z;
        const float4 q = in ? gq[s] : make_float4(0.f, 0.f, 0.f, 0.f);
        sl.C[s] = make_int4(0, __float_as_int(m_q2(q.x, q.y, q.z)), in ? __float_as_int(gt[s]) : 0, (int)q.w | s << 16);
      }
      // (a pick may read past the last pair: no leftovers there)
#pragma unroll 1
      for (int s = lane; s < slot_cap + SB; s += 32) sl.R[s] = 0ull;
      if (CORR) {
        const int p = E.corr_p;
        float2* Cacc = E.corr_comp + (size_t)c * p;
        if (sub == 0) {
#pragma unroll 1
          for (int j = lane; j < p; j += 32) Cacc[j] = make_float2(0.f, 0.f);
        }
        if (lane == 0) {
          LCorr& k0 = *sl.k0;
          lock_corr_load(E, c, &k0);
          k0.nbuf = sub == 0 ? 0 : E.slice[c].nbuf;
          k0.k_next = st.k_next;
          k0.t_next = st.k_next * E.dt_sample_ticks;
          if (MSD) { k0.r1x = st.r1[0]; k0.r1y = st.r1[1]; k0.r1z = st.r1[2]; }
        }
      }
      __syncwarp();
      live = fresh = full = true;
      aborted = false;
      continue;  // samples due or nothing to do in this launch
    }
    if (ends && !full) {
      const float ev = lane < NEND ? lock_end_comp(ens[e].NE, ens[e].cd_flag != 0, lane, Z, sl.C, wz1) : 0.0f;
      full = __any_sync(FULL_MASK, lane < NEND && fexp(ev) + S > LIMIT_E);
      unsigned long long q = quant(ev, pow2f(S));
      q += __shfl_xor_sync(FULL_MASK, q, 4);
      q += __shfl_xor_sync(FULL_MASK, q, 2);
      q += __shfl_xor_sync(FULL_MASK, q, 1);
      etot = wshfl(q, 0);
    }
    if (full) {
      int fl = 0;
      S = lock_full_rates(ens[e], sl, Z, S, wz1, &fl, &etot);
      if (fl & 3) {
        stall = (fl & 1) ? ST_NAN : ST_INF;
        continue;
      }
    }
    break;
  }
  // prefix of the pair totals at the sub-chunk boundaries (a chain that only
  // gave a sample keeps its own)
  const bool rates = fresh || full || (rq & RQ_STRUCT);
  if (rates) {
    const int np = Z - 1;
    unsigned long long s = 0;
    if (SUBS == 32 || lane < SUBS) {
#pragma unroll 3
      for (int i = 0; i < SB; ++i) {
        const int a = lane * SB + i;
        if (a < np) s += sl.R[a];
      }
    }
#pragma unroll
    for (int o = 1; o < SUBS; o <<= 1) {
      const unsigned long long u = __shfl_up_sync(FULL_MASK, s, o);
      if (lane >= o) s += u;
    }
    if (SUBS == 32 || lane < SUBS) sl.B[lane + 1] = s;
    const unsigned long long ptot = wshfl(s, SUBS - 1);
    if (lane == 0) {
      sl.B[0] = 0;
      h.tot = ptot + etot; h.etot = etot;
      h.Z = Z; h.S = S;
      h.step = step; h.hash = hash;
    }
  }
  if (lane == 0) {
    long long tc = t_end;
    if (CORR && sl.k0->k_next < ens[e].nsamples) tc = min(tc, sl.k0->t_next + 1);
    h.t_chk = tc;
    // the abort flag is looked at when the event counter is a multiple of 4096
    h.left = (int)min(step_lim - (long long)step, (long long)(4096 - (step & 4095)));
    h.fresh = (fresh ? 1 : 0) | (rates ? 2 : 0);
    if (fresh) {
      h.e = e; h.c = c; h.cap = cap; h.zlim = zlim; h.wz1 = wz1; h.stall = stall;
      h.T = T;
      h.t_end = t_end; h.step_lim = step_lim; h.lim0 = lim0;
    }
  }
  return true;
}

// After a launch in time slices: a chain that an abort stopped between two of
// them still has its samples and sums of this launch.  One warp per chain.
template <bool MSD>
__global__ void __launch_bounds__(128) k_slice_flush(const EnsDev* __restrict__ ensp, int n_chains) {
  __shared__ LCorr k0s[4];
  const EnsDev& E = *ensp;
  const int c = blockIdx.x * 4 + threadIdx.x / 32, lane = threadIdx.x % 32;
  if (E.subs <= 1 || c >= n_chains) return;
  const unsigned done = E.slice[c].done;
  if (done == 0 || done >= (unsigned)E.subs) return;
  LCorr* k0 = &k0s[threadIdx.x / 32];
  if (lane == 0) {
    lock_corr_load(E, c, k0);
    k0->nbuf = E.slice[c].nbuf;
  }
  __syncwarp();
  lock_corr_out<MSD>(E, c, k0);
  __syncwarp();
  if (lane == 0) lock_corr_store(E, c, *k0);
}

// Whether the launch has moved since the warp last asked: a chain taken from the
// work list or 4096 more events of one.  A wait that has polled StepList::polls
// times goes on if so (a chain's earlier time slice may run for minutes in another
// block), else gives up (status bit 1).
__device__ __noinline__ bool lock_moved(const EnsDev* ens, const unsigned int* work, unsigned* seen) {
  int moved = 0;
  if ((threadIdx.x & 31) == 0) {
    const unsigned n = *(const volatile unsigned int*)work + (unsigned)*(const volatile unsigned long long*)&ens[0].counters[3];
    moved = n != *seen;
    *seen = n;
  }
  return wshfl(moved, 0) != 0;
}

// A slide warp runs 32 / G chains with G lanes each; the pick has 4 sub-chunks of
// SB pairs per lane.
template <int CK, int G, int SB, int TB, int MB>
__global__ void __launch_bounds__(TB, MB) k_lock(const EnsDev* __restrict__ ens, int n_ens,
                                                  const long long* __restrict__ prefix, long long total,
                                                  unsigned int* work, int slot_cap, int tiles, int slides,
                                                  const volatile int* abort_flag, int* status, StepList lst) {
  constexpr int CPW = 32 / G, SUBS = 4 * G;
  extern __shared__ __align__(16) unsigned char smem[];
  Ctl* const ctl = (Ctl*)smem;
  unsigned char* const slots = smem + sizeof(Ctl);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t sbytes = lock_bytes(slot_cap, SUBS, SB);
  const unsigned all = tiles >= 32 ? 0xffffffffu : (1u << tiles) - 1u;
  {
    // every slot starts with a request for its first chain
#pragma unroll 1
    for (int t = 0; t < tiles; ++t) {
      const LSlot s = lock_slot(slots + (size_t)t * sbytes, slot_cap, SB);
#pragma unroll 1
      for (int i = threadIdx.x; i < slot_cap + SB; i += blockDim.x) s.R[i] = 0ull;
      if (threadIdx.x == 0) {
        s.h->rq = RQ_LOAD;
        s.h->e = 0;
        s.h->pend = 0;
      }
    }
    if (threadIdx.x == 0) { ctl->req = all; ctl->done = 0u; ctl->dead = 0u; }
    if (threadIdx.x < 4) ctl->seen[threadIdx.x] = 0u;
  }
  __syncthreads();

  if (warp >= slides) {
    // ------------------------------------------------ service warp
    const long long n_items = lst.dyn_total != nullptr ? (long long)*lst.dyn_total : total;
    const int subs = lst.dyn_total != nullptr ? 1 : ens[0].subs;  // time slices
    unsigned idle = 0, turn = ~0u;  // polls since this warp last served a request
    for (;;) {
      int b = -1;
      if (lane == 0) {
        const unsigned q = *(volatile unsigned*)&ctl->req;
        if (q != 0u) {
          // in turn: a slot that polls for its chain's earlier time slice must not
          // keep the slot that runs it from being served
          const unsigned next = q & turn;
          b = __ffs(next != 0u ? next : q) - 1;
          turn = b == 31 ? ~0u : ~0u << (b + 1);
          if ((atomicAnd(&ctl->req, ~(1u << b)) >> b & 1u) == 0u) b = -2;  // another warp took it
        } else if (*(volatile unsigned*)&ctl->dead == all) {
          b = -3;
        }
      }
      b = wshfl(b, 0);
      if (b == -3) return;
      if (b >= 0) {
        // what the slide lanes wrote before the request, seen by lane 0, now by all
        __threadfence_block();
        __syncwarp();
        const LSlot sl = lock_slot(slots + (size_t)b * sbytes, slot_cap, SB);
        const bool done = lock_serve<CK, SUBS, SB>(ens, n_ens, prefix, n_items, subs, work, slot_cap, sl, 1u << b, ctl,
                                                   abort_flag, status, lst);
        __syncwarp();
        if (lane == 0) {
          __threadfence_block();
          atomicOr(done ? &ctl->done : &ctl->req, 1u << b);
        }
        if (done) {
          idle = 0;
          continue;
        }
      }
      if (++idle > lst.polls) {
        if (!lock_moved(ens, work, &ctl->seen[warp])) {
          if (lane == 0) atomicOr(status, 2);
          return;
        }
        idle = 0;
      }
      if (b == -1) __nanosleep(100);
      else if (b >= 0) __nanosleep(1000);
    }
  }

  // -------------------------------------------------- slide warp
  const int gl = lane & (G - 1);
  const int slot = warp * CPW + lane / G;
  const bool has = slot < tiles;
  const unsigned bit = has ? 1u << slot : 0u;
  const LSlot sl = lock_slot(slots + (size_t)min(slot, tiles - 1) * sbytes, slot_cap, SB);
  Hdr* const h = sl.h;
  const int j0 = gl * 4 * SB;
  bool run = false, dead = !has;
  int Z = 1, S = 0, left = 0, wi = G, c = 0;
  long long T = 0, t_chk = 0;
  uint64_t step = 0, hash = 0;
  float pfx = 0.f;
  bool cd = false;
  const EnsDev* E = ens;
  const float4 *tNT = ens[0].NT, *tNE = ens[0].NE;
  const float* tFR = ens[0].FRIC;
  uint32_t r0 = 0, r1 = 0;
  unsigned long long A0 = 0, A1 = 0, A2 = 0, A3 = 0, tot = 0, etot = 0;
  unsigned idle = 0;

  for (;;) {
    // chains that a service warp has finished
    // (one lane reads for all: the lanes must act on the same value)
    const unsigned dn = wshfl(*(volatile unsigned*)&ctl->done, 0);
    const bool res = !run && (dn & bit) != 0u;
    if (__any_sync(FULL_MASK, res)) {
      __threadfence_block();
      __syncwarp();  // (as in the service warps)
      if (res) {
        if (gl == 0) atomicAnd(&ctl->done, ~bit);
        const int what = h->fresh;
        if (h->Z == 0) {
          dead = true;
        } else {
          run = true;
          left = h->left;
          t_chk = h->t_chk;
          if (what & 2) {
            Z = h->Z; S = h->S;
            step = h->step; hash = h->hash;
            tot = h->tot; etot = h->etot;
            const unsigned long long* B = sl.B + 4 * gl;
            A0 = B[0]; A1 = B[1]; A2 = B[2]; A3 = B[3];
          }
          if (what & 1) {
            E = ens + h->e;
            c = h->c;
            T = h->T;
            cd = E->cd_flag != 0;
            pfx = cd ? E->prefact : 0.0f;
            tNT = E->NT; tNE = E->NE; tFR = E->FRIC;
            wi = G;
          }
        }
      }
      __syncwarp();
    }
    if (!__any_sync(FULL_MASK, run)) {
      if (__all_sync(FULL_MASK, dead)) return;
      if (++idle > lst.polls) {
        if (!lock_moved(ens, work, &ctl->seen[warp])) {
          if (lane == 0) atomicOr(status, 2);
          return;
        }
        idle = 0;
      }
      __nanosleep(20);
      continue;
    }
    idle = 0;
    // random words of the next G events of every chain
    if (__any_sync(FULL_MASK, run && wi == G)) {
      const uint64_t ctr = step + (uint64_t)gl;
      const U4 q = lock_words(*E, P_EVENT, ctr, c);
      r0 = q.x; r1 = q.y;
      wi = 0;
    }
    // ------------------------------------------------ one event of every running chain
    const uint32_t w0 = gshfl<G>(r0, wi), w1 = gshfl<G>(r1, wi);
    const unsigned long long pr = __umul64hi(tot, ((unsigned long long)w1 << 32) | w0);
    const float sf = pow2f(S);
    // dt = 1 / sum W (ensemble_kernel.cu:262-272)
    const float sumw = __fmul_rn(__ll2float_rn((long long)tot), pow2f(-S));
    const float dt = __fdiv_rn(1.0f, sumw);
    const long long dtt = __float2ll_rn(__fmul_rn(dt, 4294967296.0f));
    // pick (ensemble_kernel.cu:274-501): pr uniform in [0, tot)
    // (the last lane whose pairs begin at or below pr; A0 of the first is 0)
    const int L = __popc(gbits<G>(__ballot_sync(FULL_MASK, pr >= A0), lane)) - 1;
    const bool isp = run && pr < tot - etot;  // else a chain end
    const bool c1 = pr >= A1, c2 = pr >= A2, c3 = pr >= A3;
    int jj = j0 + (c3 ? 3 * SB : c2 ? 2 * SB : c1 ? SB : 0);
    unsigned long long r = pr - (c3 ? A3 : c2 ? A2 : c1 ? A1 : A0);
    {
      const unsigned long long* b = sl.R + (isp && gl == L ? jj : 0);
      unsigned long long s[SB];
#pragma unroll
      for (int i = 0; i < SB; ++i) s[i] = b[i];
      unsigned long long lo = 0;
      int n = 0;
#pragma unroll
      for (int i = 0; i + 1 < SB; ++i) {
        if (i > 0) s[i] += s[i - 1];
        if (r >= s[i]) { n = i + 1; lo = s[i]; }
      }
      jj += n;
      r -= lo;
    }
    jj = gshfl<G>(jj, L);
    r = gshfl<G>(r, L);
    if (!isp) jj = 0;
    // classification: lane k holds pair jj - 1 + k (k = 0, 1, 2) and classifies
    // as if that pair had been picked; lane 1's answer counts
    const int np = Z - 1;
    const int p = jj - 1 + gl;
    bool act = isp && gl < 3 && p >= 0 && p < np;
    const int pc = act ? p : 0;
    const int4 ca = sl.C[pc], cb = sl.C[pc + 1];
    const unsigned long long rold = sl.R[pc];
    const float yt = __fmul_rn(cd ? __int_as_float(ca.z) : 0.0f, sf);
    const unsigned long long vt = f2u64_rn(yt);
    const unsigned long long qc = f2u64_rn(__fmul_rn(__fmul_rn(pfx, (float)(strand_n(ca.w) - 1)), sf));
    const unsigned long long qp = f2u64_rn(__fmul_rn(__int_as_float(ca.x), sf));
    const bool okdt = dt != 0.0f && dt < 2.0e9f;
    int cls = (r >= vt && r < rold - qc) ? ((r - vt < qp) ? 1 : -1) : 0;  // shift +1, shift -1, CD event
    cls = gshfl<G>(cls, 1);
    const int d = (isp && okdt) ? cls : 0;
    const bool slide = d != 0;
    // the touched pairs: both sliding rates of a pair on its lane
    act = act && slide;
    const int W1 = ca.w + (gl == 1 ? d : gl == 2 ? -d : 0), W2 = cb.w + (gl == 0 ? d : gl == 1 ? -d : 0);
    const int N1 = act ? strand_n(W1) : 1;
    const int N2 = act ? strand_n(W2) : 1;
    const float q1 = __int_as_float(ca.y), q2 = __int_as_float(cb.y);
    float wp, wm;
    bool ok;
    {
      const float4 ta = __ldg(&tNT[N1]), tb = __ldg(&tNT[N2]);
      const bool z1 = (q1 == 0.0f), z2 = (q2 == 0.0f);
      const int i = (z1 ? 4 * N1 + 1 : 2 * N1) + (z2 ? 4 * N2 - 1 : 2 * N2);
      const int k = (z1 ? 4 * N1 - 1 : 2 * N1) + (z2 ? 4 * N2 + 1 : 2 * N2);
      const float fp = __ldg(&tFR[i]), fm = __ldg(&tFR[k]);
      const float ep = __fmaf_rn(q1, ta.x, -__fmul_rn(q2, tb.y)), em = __fmaf_rn(q2, tb.x, -__fmul_rn(q1, ta.y));
      const float pp = __fmul_rn(z1 ? 1.0f : ta.z, z2 ? 1.0f : tb.w), pm = __fmul_rn(z1 ? 1.0f : ta.w, z2 ? 1.0f : tb.z);
      ok = ep < kExpMost && em < kExpMost;
      wp = __fmul_rn(__fmul_rn(fp, pp), m_exp_lt88(ep));
      wm = __fmul_rn(__fmul_rn(fm, pm), m_exp_lt88(em));
      wp = N2 > 1 ? wp : 0.0f;
      wm = N1 > 1 ? wm : 0.0f;
    }
    const float yp = __fmul_rn(wp, sf), ym = __fmul_rn(wm, sf);
    const float ye = __fmul_rn(__fmul_rn(pfx, (float)(N1 - 1)), sf);
    constexpr float kMost = 281474976710656.0f;  // 2^(LIMIT_E+1); NaN fails the comparisons too
    // (a sum above the limit of one asks for a full pass that changes nothing)
    const bool bad = act && !(ok && __fadd_rn(__fadd_rn(yp, ym), __fadd_rn(yt, ye)) < kMost);
    const unsigned long long pt = f2u64_rn(yp) + f2u64_rn(ym) + vt + f2u64_rn(ye);
    const unsigned long long dl = act ? pt - rold : 0ull;
    // (shuffles and votes do not order memory: the neighbours' loads of a strand
    // come before its store, and the chain-end loads below after it)
    __syncwarp();
    if (act) {
      sl.R[p] = pt;
      sl.C[p].x = __float_as_int(wp);
      if (gl == 1) { sl.C[p].w = W1; sl.C[p + 1].w = W2; }
    }
    {
      // the prefix sums move by the deltas of pairs jj-1, jj, jj+1
      const unsigned long long e0 = gshfl<G>(dl, 0), e1 = e0 + gshfl<G>(dl, 1), e2 = e1 + gshfl<G>(dl, 2);
      auto patch = [&](unsigned long long& A, int b) {
        A += b > jj + 1 ? e2 : b == jj + 1 ? e1 : b == jj ? e0 : 0ull;
      };
      patch(A0, j0);
      patch(A1, j0 + SB);
      patch(A2, j0 + 2 * SB);
      patch(A3, j0 + 3 * SB);
      tot += e2;
    }
    int rq = gbits<G>(__ballot_sync(FULL_MASK, bad), lane) != 0u ? RQ_FULL : 0;
    // a slide next to a chain end changes the chain-end rates
    const bool near = slide && (jj <= 1 || jj + 1 >= Z - 2);
    if (__any_sync(FULL_MASK, near)) {
      __syncwarp();
      // lane 0 the head, lane 1 the tail (its sliding creation, or with one
      // Kuhn step its sliding destruction), lane 2 the tail's CD creation
      // (ensemble_kernel.cu:219-260; the others of the five rates are zero)
      bool over = false;
      unsigned long long q = 0;
      if (near && gl < 3) {
        const int Ne = strand_n(sl.C[gl == 0 ? 0 : np].w), Nn = strand_n(sl.C[gl == 0 ? 1 : np - 1].w);
        const float4 e1 = __ldg(&tNE[Ne]), e2 = __ldg(&tNE[Nn]);
        const float ev = gl == 2 ? (cd ? e1.w : 0.0f) : Ne != 1 ? e1.x : Z == 2 ? e2.y : e2.z;
        over = fexp(ev) + S > LIMIT_E;
        q = f2u64_rn(__fmul_rn(ev, sf));
      }
      q = gshfl<G>(q, 0) + gshfl<G>(q, 1) + gshfl<G>(q, 2);
      if (gbits<G>(__ballot_sync(FULL_MASK, over), lane) != 0u) rq |= RQ_FULL;
      if (near) {
        tot += q - etot;
        etot = q;
      }
    }
    if (slide) {
      const uint32_t code = ((uint32_t)(d > 0 ? SDP : SDM) << 24) | (uint32_t)jj;
      hash = (hash ^ (uint64_t)code) * 0x100000001B3ull;
      T += dtt;
      ++step;
      ++wi;
      --left;
      if (T >= t_chk || left == 0) rq |= RQ_TIME;
    } else if (run) {
      rq = okdt ? RQ_STRUCT : RQ_STALL;
      if (okdt) {
        T += dtt;
        ++step;  // the next event's; the service warp is given this one's
        ++wi;
      }
    }
    __syncwarp();
    if (__any_sync(FULL_MASK, run && rq != 0)) {
      if (run && rq != 0) {
        run = false;
        if (gl == 1) {  // the lane that classified the picked pair
          h->T = T; h->step = rq == RQ_STRUCT ? step - 1 : step; h->hash = hash; h->etot = etot;
          const bool cdd = r < vt;
          h->r = !isp ? pr - (tot - etot) : cdd ? r : r - (rold - qc);
          h->wsel = (!isp || cdd) ? 0ull : qc;
          h->rq = rq;
          h->jj = okdt ? (isp ? jj : -1) : dt == 0.0f ? ST_DT_ZERO : ST_INF;
          __threadfence_block();
          atomicOr(&ctl->req, bit);
        }
      }
      __syncwarp();
    }
  }
}

}  // namespace

// Lanes per chain and pairs per sub-chunk built for a slot size: the fewest
// pairs that cover it; lanes 0: no lockstep build
struct LockShape {
  int lanes, sb;
};
static LockShape lock_shape(int slot_cap) {
  for (int sb : {3, 5, 9})
    if (slot_cap <= 16 * sb) return {4, sb};
  for (int sb : {8, 12})
    if (slot_cap <= 32 * sb) return {8, sb};
  return {0, 0};
}
int lock_lanes(int slot_cap) { return lock_shape(slot_cap).lanes; }
bool lock_slices(int slot_cap) { return lock_shape(slot_cap).lanes == 8; }
size_t lock_block_bytes(int slot_cap, int tiles) {
  const LockShape f = lock_shape(slot_cap);
  return sizeof(Ctl) + lock_bytes(slot_cap, 4 * f.lanes, f.sb) * tiles;
}

template <int CK, int MB>
static void* lock_pick(const LockShape& f) {
  switch (f.sb) {
    case 3: return (void*)k_lock<CK, 4, 3, 128, MB>;
    case 5: return (void*)k_lock<CK, 4, 5, 128, MB>;
    case 9: return (void*)k_lock<CK, 4, 9, 128, MB>;
    case 8: return (void*)k_lock<CK, 8, 8, 128, MB>;
    case 12: return (void*)k_lock<CK, 8, 12, 128, MB>;
    default: return nullptr;
  }
}
void* lock_kernel(int ck, int slot_cap, bool hi) {
  const LockShape f = lock_shape(slot_cap);
  if (hi) return ck == 0 ? lock_pick<0, 5>(f) : nullptr;
  return ck == 0 ? lock_pick<0, 4>(f) : ck == 2 ? lock_pick<2, 4>(f) : lock_pick<1, 4>(f);
}

cudaError_t launch_slice_flush(const EnsDev* d_ens, int ck, int n_chains, cudaStream_t st) {
  const unsigned blocks = (unsigned)((n_chains + 3) / 4);
  if (ck == 2) k_slice_flush<true><<<blocks, 128, 0, st>>>(d_ens, n_chains);
  else k_slice_flush<false><<<blocks, 128, 0, st>>>(d_ens, n_chains);
  return cudaGetLastError();
}

}  // namespace dsm

