// k_kspace.cu -- random batch Ewald: k-vector sampling, structure factor, and the Ewald energy sum.
//
//   RBEPSAMPLE::Fetch_P_Sample / MH_Algorithm   framework/model/RBEPSample.h:64-177  (host in the
//                                                reference, reseeded mt19937 per draw)
//   ComputePnumberChargeStructureFactorWorklet + ReduceByKey  RunWorklet.cpp:2209-2270,
//                                                framework/run/ExecutionMD.cpp:469-501
//   ComputeEwaldEnergy                           framework/run/ExecutionMD.cpp:405-443
//
// Sampling runs on the device so a step never returns to the host.  Proposal probabilities come from per-system tables of
// P(m) and q(m) built on the host with the reference's formulas, so the chain makes the same
// accept/reject decisions as the CPU oracle on the same stream.
#include "kernels.h"

namespace rbmd {

constexpr int kMaxRbeSlots = 1024;  // proposal slots of a system decided at a time

// Box-Muller proposal of slot t, dimension d (FetchSample_1D, RBEPSample.h:115-145).
__device__ inline double rbe_gauss(const SysDev& s, uint32_t step, uint32_t t, int d) {
  double U1 = 0.5, U2 = 0.5;
  if (s.random_mode != RBMD_RANDOM_TEST) {
    for (uint32_t attempt = 0; attempt < 64; ++attempt) {  // P(U1 < 1e-6)^64 is nil
      uint32_t o[4];
      philox4x32_10(t, (uint32_t)d | (attempt << 2), step, kTagRbeGauss, s.seed_lo, s.seed_hi, o);
      U1 = u01(o[0], o[1]);
      U2 = u01(o[2], o[3]);
      if (!(U1 < 1e-6)) break;
    }
  }
  return s.rbe_sigma[d] * sqrt(-2.0 * log(U1)) * cos(2 * kPi * U2) + 0.0;
}

__device__ inline double rbe_accept(const SysDev& s, uint32_t step, uint32_t t, int d) {
  if (s.random_mode == RBMD_RANDOM_TEST) return 0.5;
  uint32_t o[4];
  philox4x32_10(t, (uint32_t)d, step, kTagRbeAccept, s.seed_lo, s.seed_hi, o);
  return u01(o[0], o[1]);
}

// Probability of moving a chain from m = im to m = iw (MH_Algorithm, RBEPSample.h:64-83), indices into
// the tables of one dimension.
__device__ __forceinline__ double rbe_move(const double* tabP, const double* tabQ, int tw, int im, int iw) {
  double p = 0.0;
  if (iw >= 0 && iw < tw && im >= 0 && im < tw) p = (tabP[iw] / tabP[im]) * (tabQ[im] / tabQ[iw]);
  return fmin(p, 1.0);
}

// One block per system, the proposal slots taken kMaxRbeSlots at a time.  A slot's proposal and uniform
// do not depend on the chain, and the chain's state is almost always the slot before's proposal (the
// proposals follow the target closely, so about one in a hundred is refused), so every slot decides
// in parallel whether it would be accepted from the proposal one slot back and from the one two slots
// back.  Only the refused slots are left to walk in order: a warp per dimension goes from one clear
// bit of the first decision to the next, and evaluates a move itself when three or more slots in a row
// are refused.  The dimensions' chains do not see each other: an all-zero vector is left out of the
// samples but stays the chain's state.  Counting the slots with a non-zero vector gives each
// sample's place.  Walking the chain slot by slot was a serial string of table reads and divisions:
// 91 us for P = 200 and 52 us for P = 100, whatever the system's size.
constexpr int kRbeThreads = 512;
constexpr int kRbeWords = kMaxRbeSlots / 32;
static_assert(kRbeThreads >= 96 && kMaxRbeSlots % 32 == 0, "a warp per dimension, whole words");

__global__ void __launch_bounds__(kRbeThreads) k_rbe_sample(const SysDev* __restrict__ S,
                                                           const int* __restrict__ slots) {
  const SysDev& s = S[slots[blockIdx.x]];
  if (s.coul != RBMD_COUL_RBE) return;
  __shared__ int s_m[3][kMaxRbeSlots];         // proposals
  __shared__ double s_u[3][kMaxRbeSlots];      // acceptance uniforms
  __shared__ short s_src[3][kMaxRbeSlots];     // slot whose proposal the chain holds after each slot, -1: the
                                               // state before the first
  __shared__ unsigned s_acc[2][3][kRbeWords];  // accepted from the proposal one / two slots back
  __shared__ unsigned s_nz[kRbeWords];         // slots after which the vector is not zero
  __shared__ int s_prev[3], s_first, s_used;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const unsigned FULL = 0xffffffffu;
  const uint32_t step = (uint32_t)s.st->step;
  const int P = s.P, mmax = s.rbe_mmax, tw = 2 * mmax + 1;
  // The reference loops until it finds non-zero vectors; bound the slots so that a degenerate
  // distribution (all proposals rounding to 0) ends with an error word instead of spinning.
  const int tmax = 4096 + 64 * P;
  int t0 = 0, done = 0;     // slots and samples before this round
  bool started = false;
  if (tid < 3) s_prev[tid] = tid == 0 ? 1 : 0;
  while (done < P && t0 < tmax) {
    const int ns = min(min(kMaxRbeSlots, P - done + kRbeSlack), tmax - t0);
    const int nw = (ns + 31) >> 5;
    if (tid == 0) s_first = started ? -1 : ns;
    for (int k = tid; k < 3 * ns; k += kRbeThreads) {
      const int d = k / ns, t = k - d * ns;
      s_m[d][t] = (int)round(rbe_gauss(s, step, (uint32_t)(t0 + t), d));
      s_u[d][t] = rbe_accept(s, step, (uint32_t)(t0 + t), d);
    }
    __syncthreads();
    if (!started) {  // the chains start at the first slot with a non-zero vector, taken as it is
      for (int t = tid; t < ns; t += kRbeThreads)
        if ((s_m[0][t] | s_m[1][t] | s_m[2][t]) != 0) atomicMin(&s_first, t);
      __syncthreads();
    }
    const int first = s_first;
    if (first < ns) {
      for (int w = wid; w < 3 * nw; w += kRbeThreads / 32) {
        const int d = w / nw, t = 32 * (w - d * nw) + lane;
        const double *tabP = s.rbe_tab + (size_t)d * tw * 2, *tabQ = tabP + tw;
        bool one = false, two = false;
        if (t < ns) {
          const int iw = s_m[d][t] + mmax;
          const double u = s_u[d][t];
          one = u <= rbe_move(tabP, tabQ, tw, (t > 0 ? s_m[d][t - 1] : s_prev[d]) + mmax, iw);
          if (t > 0) two = u <= rbe_move(tabP, tabQ, tw, (t > 1 ? s_m[d][t - 2] : s_prev[d]) + mmax, iw);
          one |= t <= first;
        }
        const unsigned o = __ballot_sync(FULL, one), q = __ballot_sync(FULL, two);
        if (lane == 0) {
          s_acc[0][d][w - d * nw] = o;
          s_acc[1][d][w - d * nw] = q;
        }
        if (t < ns) s_src[d][t] = (short)t;  // overwritten where the chain stays
      }
      __syncthreads();
      if (wid < 3 && lane == 0) {
        const int d = wid;
        const double *tabP = s.rbe_tab + (size_t)d * tw * 2, *tabQ = tabP + tw;
        for (int t = 0; t < ns;) {
          const unsigned w = s_acc[0][d][t >> 5] | ((1u << (t & 31)) - 1u);
          if (w == FULL) {  // no refusal up to the end of the word
            t = (t | 31) + 1;
            continue;
          }
          t = (t & ~31) + __ffs(~w) - 1;
          if (t >= ns) break;
          const int src = t - 1;  // slot t refused: the chain stays at the proposal of the slot before
          const int im = (src >= 0 ? s_m[d][src] : s_prev[d]) + mmax;
          s_src[d][t] = (short)src;
          for (++t; t < ns; ++t) {
            const bool a = t == src + 2 ? (s_acc[1][d][t >> 5] >> (t & 31)) & 1u
                                        : s_u[d][t] <= rbe_move(tabP, tabQ, tw, im, s_m[d][t] + mmax);
            if (a) break;
            s_src[d][t] = (short)src;
          }
          ++t;  // accepted
        }
      }
      __syncthreads();
      auto state = [&](int d, int t) { return s_src[d][t] >= 0 ? s_m[d][s_src[d][t]] : s_prev[d]; };
      for (int w = wid; w < nw; w += kRbeThreads / 32) {
        const int t = 32 * w + lane;
        const bool nz = t < ns && t >= first && (state(0, t) | state(1, t) | state(2, t)) != 0;
        const unsigned b = __ballot_sync(FULL, nz);
        if (lane == 0) s_nz[w] = b;
      }
      __syncthreads();
      for (int w = wid; w < nw; w += kRbeThreads / 32) {
        int before = 0;  // samples of the words before
        for (int v = lane; v < w; v += 32) before += __popc(s_nz[v]);
        before = done + __reduce_add_sync(FULL, before);
        const int t = 32 * w + lane, l = before + __popc(s_nz[w] & lanemask_lt(lane));
        if ((s_nz[w] >> lane) & 1u && l < P) {
          for (int d = 0; d < 3; ++d) s.km[3 * l + d] = state(d, t);
        }
      }
      if (wid == 0) {
        int all = 0;
        for (int v = lane; v < nw; v += 32) all += __popc(s_nz[v]);
        all = __reduce_add_sync(FULL, all);
        if (lane == 0) s_used = all;
      }
      int last = 0;
      if (tid < 3) last = state(tid, ns - 1);
      __syncthreads();
      if (tid < 3) s_prev[tid] = last;
      done += s_used;
      started = true;
    }
    t0 += ns;
    __syncthreads();
  }
  if (done < P) {  // out of slots: the rest repeats the last vector, and the system is flagged
    for (int k = 3 * done + tid; k < 3 * P; k += kRbeThreads) s.km[k] = s_prev[k % 3];
    if (tid == 0) atomicOr(&s.st->status, kErrRbeSlots);
  }
  __syncthreads();
  // k vectors and force coefficients: k_l = 2 pi m_l / L, coef = -4 pi / (V |k_l|^2)
  for (int l = tid; l < P; l += kRbeThreads) {
    const double kx = 2 * kPi * s.km[3 * l] / s.L[0];
    const double ky = 2 * kPi * s.km[3 * l + 1] / s.L[1];
    const double kz = 2 * kPi * s.km[3 * l + 2] / s.L[2];
    const double k2 = kx * kx + ky * ky + kz * kz;
    s.kv[l] = make_double4(kx, ky, kz, -4 * kPi / (s.volume * k2));
  }
}

// Structure factor over a chunk of a system's atoms per block; the last block of the system sums the
// chunk partials in chunk order (deterministic, FP64).  Bound by the sine / cosine arithmetic (SFU in
// mixed precision, FP64 otherwise) once every SM has blocks, and by how many have before that: the
// block takes the k indices 32 at a time, one per lane, and its eight warps an eighth of the chunk's
// atoms each, so that a small system's few thousand atom-k terms spread over 64-atom blocks and all
// their warps (one k per thread over 256 atoms left 100 of 256 threads, and an SM per 256 atoms, with
// work).  The chunk length depends on the system alone, so its sums do not depend on the batch.
constexpr int kRhoWarps = 8;

template <bool MIXED, bool ENERGY>
__global__ void __launch_bounds__(kRhoWarps * 32) k_rho(const SysDev* __restrict__ S, const int2* __restrict__ work) {
  const int2 wk = work[blockIdx.x];
  const SysDev& s = S[wk.x];
  const int nk = ENERGY ? s.nk_e : (s.coul == RBMD_COUL_RBE ? s.P : s.nk_ewald);
  const double4* kv = ENERGY ? s.kv_e : s.kv;
  constexpr bool kF32 = MIXED && !ENERGY;
  __shared__ double4 s_x[kF32 ? 1 : kRhoChunk];
  __shared__ float4 s_u[kF32 ? kRhoChunk : 1];
  __shared__ double2 s_red[2][kRhoWarps][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int chunk = s.rho_chunk, a0 = wk.y;
  const int na = min(chunk, s.n - a0);
  for (int k = threadIdx.x; k < na; k += blockDim.x) {
    const double4 p = s.x[a0 + k];
    if (kF32)
      s_u[k] = make_float4((float)(p.x / s.L[0]), (float)(p.y / s.L[1]), (float)(p.z / s.L[2]), (float)p.w);
    else
      s_x[k] = p;
  }
  __syncthreads();
  const int per = chunk / kRhoWarps;  // at most 32 atoms per warp
  const int j0 = min(na, wid * per), j1 = min(na, j0 + per);
  const int blk = a0 / chunk;
  // the warps' sums of 32 k indices at l0: warp `who` adds them in warp order and hands them to `put`;
  // two buffers in turn, so one barrier per 32 indices
  auto gather = [&](int buf, int who, double re, double im, auto&& put) {
    s_red[buf][wid][lane] = make_double2(re, im);
    __syncthreads();
    if (wid == who) {
      double tr = 0.0, ti = 0.0;
#pragma unroll
      for (int w = 0; w < kRhoWarps; ++w) {
        const double2 v = s_red[buf][w][lane];
        tr += v.x;
        ti += v.y;
      }
      put(tr, ti);
    }
  };
  double* part = s.rho_part + (size_t)blk * 2 * nk;
  // FP32: the next 32 indices are loaded during the present ones' atoms
  int3 m = make_int3(0, 0, 0);
  auto index = [&](int l) {
    if (kF32 && l < nk) m = make_int3(s.km[3 * l], s.km[3 * l + 1], s.km[3 * l + 2]);
  };
  index(lane);
  for (int l0 = 0, turn = 0; l0 < nk; l0 += 32, ++turn) {
    const int l = l0 + lane;
    double re = 0.0, im = 0.0;
    const float mxr = (float)m.x, myr = (float)m.y, mzr = (float)m.z;
    index(l + 32);
    if (l < nk) {
      if (kF32) {
        // phase in turns m . (r / L), reduced to [-1/2, 1/2] before the FP32 sine and cosine (the
        // SFU approximations, absolute error about 4e-7 on [-pi, pi]); FP32 partial sums over the
        // warp's atoms (at most 32), added in FP64 (the SFU also converts FP32 to FP64); the nearest
        // integer of the phase by the 1.5 * 2^23 addition (round to nearest even, |ph| < 2^22), on
        // the FMA pipe
        float pr = 0.0f, pm = 0.0f;
        for (int j = j0; j < j1; ++j) {
          const float4 u = s_u[j];
          float ph = mxr * u.x + myr * u.y + mzr * u.z;
          ph -= __fsub_rn(__fadd_rn(ph, 12582912.0f), 12582912.0f);
          float sn, cs;
          __sincosf(6.28318531f * ph, &sn, &cs);  // hardware sin / cos: |2 pi ph| <= pi
          pr += u.w * cs;
          pm += u.w * sn;
        }
        re = (double)pr;
        im = (double)pm;
      } else {
        const double4 k = kv[l];
        for (int j = j0; j < j1; ++j) {
          const double4 p = s_x[j];
          const double dot = k.x * p.x + k.y * p.y + k.z * p.z;
          double sn, cs;
          sincos(dot, &sn, &cs);
          re += p.w * cs;
          im += p.w * sn;
        }
      }
    }
    gather(turn & 1, turn % kRhoWarps, re, im, [&](double tr, double ti) {
      if (l < nk) {
        part[2 * l] = tr;
        part[2 * l + 1] = ti;
      }
    });
  }
  if (arrive_last(&s.st->counter[ENERGY ? 4 : 1], (unsigned)s.blocks_rho)) {
    // every warp takes a run of the chunks, lanes 32 k indices
    double* out = ENERGY ? s.rhok_e : s.rhok;
    double esum = 0.0;
    const int seg = (s.blocks_rho + kRhoWarps - 1) / kRhoWarps;
    const int b0 = wid * seg, b1 = min(s.blocks_rho, b0 + seg);
    for (int l0 = 0, turn = 0; l0 < nk; l0 += 32, ++turn) {
      const int l = l0 + lane;
      double re = 0.0, im = 0.0;
      if (l < nk) {
        const double2* p = reinterpret_cast<const double2*>(s.rho_part) + l;
#pragma unroll 4
        for (int b = b0; b < b1; ++b) {
          const double2 v = __ldcg(&p[(size_t)b * nk]);
          re += v.x;
          im += v.y;
        }
      }
      gather(turn & 1, 0, re, im, [&](double tr, double ti) {
        if (l < nk) {
          out[2 * l] = tr;
          out[2 * l + 1] = ti;
          if (ENERGY) esum += kv[l].w * (tr * tr + ti * ti);
        }
      });
    }
    if (ENERGY && wid == 0) {
      esum = warp_sum(esum);
      if (lane == 0) s.st->energy[6] = esum;
    }
  }
}

void launch_rbe_sample(const Batch& b, cudaStream_t st) {
  k_rbe_sample<<<b.nsys, kRbeThreads, 0, st>>>(b.sys, b.d_slots);
  note_launch();
}

void launch_rho(const Batch& b, cudaStream_t st, int ewald) {
  (void)ewald;
  if (b.prec == RBMD_PREC_MIXED && b.coul == RBMD_COUL_RBE)
    k_rho<true, false><<<b.rho.n, kRhoWarps * 32, 0, st>>>(b.sys, b.rho.d);
  else
    k_rho<false, false><<<b.rho.n, kRhoWarps * 32, 0, st>>>(b.sys, b.rho.d);
  note_launch();
}

void launch_ewald_energy(const Batch& b, cudaStream_t st) {
  k_rho<false, true><<<b.rho.n, kRhoWarps * 32, 0, st>>>(b.sys, b.rho.d);
  note_launch();
}

}  // namespace rbmd
