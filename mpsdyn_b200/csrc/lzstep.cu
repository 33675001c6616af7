// One reorthogonalised Lanczos step for a group of independent local
// eigenproblems, in a single cooperative launch (replaces the
// orthogonalisation inside the PRIMME call of Contractor::solveEigs,
// src/core/cpp/Contractor.cpp:3067-3138).
//
// For every instance q, with k = j+1 basis vectors V[:, 0..j] and
// w = (H - sigma) v_j computed by the matvec:
//   projector  w += U (U^H v_j)        (excited states: U holds sqrt(pen) u_t)
//   pass 1     w' = w - beta_{j-1} v_{j-1};  h = V^H w', |w'|^2;  w'' = w' - V h
//   pass 2     only when |w''|^2 < |w'|^2 / 2 (Daniel, Gragg, Kaufman,
//              Stewart 1976): h2 = V^H w''; w''' = w'' - V h2
//   alpha_j = sigma + Re(h_j + h2_j), beta_j = |w|, V[:, j+1] = w / beta_j.
// Without a second pass |w''|^2 = |w'|^2 - |h|^2 (V orthonormal; the test
// bounds the cancellation to a factor 2), so beta_j is known before the
// update and the update writes v_{j+1} directly.
//
// Work split.  An instance owns a set of CTAs and every CTA a range of its
// rows.  A CTA keeps its rows of w' in shared memory from the first read to
// the end of the step.  For the dots a warp owns every eighth basis vector and
// its lanes the rows, sixteen loads in flight per lane whatever k is (more
// rows at a time when there are few vectors), so the sums stay in registers
// over all rows of the CTA and cost one warp reduction per vector, and a CTA
// writes one partial sum per vector.  After one barrier among the instance's
// CTAs each of them adds the partials of the instance in the same fixed order,
// so all hold the same coefficients and reach the same second-pass decision.
// An unflagged step costs that one barrier.  How many rows a CTA takes, and
// whether the basis goes to registers, follows the whole group of a launch: the
// order of an instance's sums, and so its rounding, depends on the instances beside
// it (as the contractions' split of K does), and a chain agrees with the same chain
// alone to the solver's tolerance, not to the last bit.
//
// Small groups (at most 64 rows per CTA with one CTA per SM slot, and k <= 64)
// are bound by latency, not by bytes: a launch, the chain w -> dots -> barrier
// -> sums -> update.  There the basis rows are loaded into registers at once
// at the start, overlapped with the loads of w, and the update reads them
// again from there.
//
// Bound by bytes for large groups (the basis is read twice, 16 B an entry) and
// by latency for small ones.  Measured, with the products' shift following the
// diagonal elements so that second passes are rare: eight chains of N = 32768
// at k = 60 in 95 us (5.5 TB/s of algorithmic bytes, part of them from L2), four
// of N = 18432 in 27 us, one of N = 8192 in 11 us and of N = 800 in 8.5 us; one
// row block of 256 per partial sum, a second pass in nearly every step and a
// barrier of three atomics took 150 us and more, 44, 30 and 25 us.
//
// Barriers are bounded: a CTA that waits longer than 2 s sets the error word
// and returns (the host reports MPSGPU_TIMEOUT and resets the barrier words);
// the kernel has no copies in flight at any barrier.
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"

namespace mpsgpu {

namespace {

constexpr int T = LZ_THREADS;         // threads per CTA
constexpr int NW = T / 32;
constexpr int KMAXS = 256;            // Krylov vectors
constexpr int WCAP = 2048;            // rows of w' kept in shared memory (more stay in w itself)
constexpr int RES_ROWS = 64;          // rows per CTA of the form with the basis in registers
constexpr int RES_K = 64;             // its vectors
constexpr int PHASES = LZ_BAR_WORDS;  // barriers of a step: projector, pass 1, pass 2, its norm
constexpr double DGKS2 = 0.5;

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Bounded barrier over the n co-resident CTAs of one instance: every CTA adds
// one to a word that was zero when the launch began and waits for n.  Returns
// false (and sets *err) when the wait ran out.
__device__ bool group_barrier(unsigned* word, unsigned n, int* err) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    unsigned seen;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(word) : "memory");
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(word) : "memory");
    if (seen < n) {
      const unsigned long long t0 = gtimer();
      do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(word) : "memory");
        if (seen < n && gtimer() - t0 > 2000000000ull) {
          atomicExch(err, 1);
          ok = 0;
          break;
        }
      } while (seen < n);
    }
  }
  __syncthreads();
  return ok != 0;
}

__device__ __forceinline__ void cfma(cplx& s, cplx a, cplx b) {  // s += a b
  s.x = fma(a.x, b.x, fma(-a.y, b.y, s.x));
  s.y = fma(a.x, b.y, fma(a.y, b.x, s.y));
}
__device__ __forceinline__ void ccfma(cplx& s, cplx a, cplx b) {  // s += conj(a) b
  s.x = fma(a.x, b.x, fma(a.y, b.y, s.x));
  s.y = fma(a.x, b.y, fma(-a.y, b.x, s.y));
}

__device__ __forceinline__ double warp_sumd(double s) {
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// Sum of v[0..TV-1] over the 32 lanes by a transposing butterfly: the first
// log2(TV) exchanges halve the values a lane keeps; afterwards the lanes
// [32/TV t', ...) hold the total of vector vector_of_lane<TV>.
template <int TV>
__device__ __forceinline__ cplx warp_sum_v(cplx (&v)[TV]) {
  const int lane = threadIdx.x & 31;
  int mask = 16;
#pragma unroll
  for (int half = TV / 2; half >= 1; half >>= 1, mask >>= 1) {
    const bool up = lane & mask;
#pragma unroll
    for (int i = 0; i < half; i++) {
      const cplx send = up ? v[i] : v[i + half];
      cplx keep = up ? v[i + half] : v[i];
      keep.x += __shfl_xor_sync(0xffffffffu, send.x, mask);
      keep.y += __shfl_xor_sync(0xffffffffu, send.y, mask);
      v[i] = keep;
    }
  }
  cplx r = v[0];
#pragma unroll
  for (int o = 16 / TV; o > 0; o >>= 1) {
    r.x += __shfl_xor_sync(0xffffffffu, r.x, o);
    r.y += __shfl_xor_sync(0xffffffffu, r.y, o);
  }
  return r;
}
// the vector whose total a lane holds (the leading log2(TV) lane bits), and
// whether it is the lane that writes it
template <int TV>
__device__ __forceinline__ int vector_of_lane(int lane) { return lane / (32 / TV); }
template <int TV>
__device__ __forceinline__ bool writes_vector(int lane) { return lane % (32 / TV) == 0; }

// Partial dots of the basis vectors lb + warp + 8 t (t < TV, below k) with x
// over the n rows from r0 of the instance, to part[l ncta + rank].
template <int TV>
__device__ __forceinline__ void dots_block(const cplx* __restrict__ V, long long ldv, int lb, int k, const cplx* x,
                                           int n, int ncta, int rank, cplx* part) {
  constexpr int RL = 16 / TV;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  cplx acc[TV];
#pragma unroll
  for (int t = 0; t < TV; t++) acc[t] = make_double2(0.0, 0.0);
  const int l0 = lb + warp;
  if (l0 >= k) return;  // uniform over the warp
  const cplx* v0 = V + (long long)l0 * ldv;
  for (int c = lane; c < n; c += 32 * RL) {
    cplx v[TV][RL];
#pragma unroll
    for (int t = 0; t < TV; t++)
#pragma unroll
      for (int i = 0; i < RL; i++)
        v[t][i] = (l0 + NW * t < k && c + 32 * i < n) ? __ldcg(v0 + (long long)(NW * t) * ldv + c + 32 * i)
                                                      : make_double2(0.0, 0.0);
#pragma unroll
    for (int i = 0; i < RL; i++) {
      const cplx xi = c + 32 * i < n ? x[c + 32 * i] : make_double2(0.0, 0.0);
#pragma unroll
      for (int t = 0; t < TV; t++) ccfma(acc[t], v[t][i], xi);
    }
  }
  const cplx s = warp_sum_v<TV>(acc);
  const int l = l0 + NW * vector_of_lane<TV>(lane);
  if (writes_vector<TV>(lane) && l < k) part[(long long)l * ncta + rank] = s;
}

__device__ void cta_dots(const cplx* V, long long ldv, int k, const cplx* x, int n, int ncta, int rank, cplx* part) {
  if (k <= NW) dots_block<1>(V, ldv, 0, k, x, n, ncta, rank, part);
  else if (k <= 2 * NW) dots_block<2>(V, ldv, 0, k, x, n, ncta, rank, part);
  else if (k <= 4 * NW) dots_block<4>(V, ldv, 0, k, x, n, ncta, rank, part);
  else
    for (int lb = 0; lb < k; lb += 8 * NW) dots_block<8>(V, ldv, lb, k, x, n, ncta, rank, part);
}

// (V h)[row] for RT rows 256 apart from `row` on, sixteen loads in flight
template <int RT>
__device__ __forceinline__ void vh_rows(const cplx* __restrict__ V, long long ldv, int k, const cplx* hs, int row,
                                        int n, cplx (&s)[RT]) {
  constexpr int LB = 16 / RT;
#pragma unroll
  for (int i = 0; i < RT; i++) s[i] = make_double2(0.0, 0.0);
  for (int l0 = 0; l0 < k; l0 += LB) {
    cplx v[LB][RT];
#pragma unroll
    for (int t = 0; t < LB; t++)
#pragma unroll
      for (int i = 0; i < RT; i++)
        v[t][i] = (l0 + t < k && row + T * i < n) ? __ldcg(V + (long long)(l0 + t) * ldv + row + T * i)
                                                  : make_double2(0.0, 0.0);
#pragma unroll
    for (int t = 0; t < LB; t++) {
      if (l0 + t < k) {
        const cplx h = hs[l0 + t];
#pragma unroll
        for (int i = 0; i < RT; i++) cfma(s[i], v[t][i], h);
      }
    }
  }
}

// x - V h over the CTA's rows, handed row by row to out(row, value); last
// rows first: the dots read them last, so that the rows still in L2 are read
// again before they go (bases of a large group exceed it), and the next step's
// dots begin with the rows this update ends with
template <int RT, class Out>
__device__ __forceinline__ void update_block(const cplx* V, long long ldv, int k, const cplx* hs, const cplx* x, int n,
                                             Out out) {
  for (int row = (n - 1) / (T * RT) * (T * RT) + threadIdx.x; row >= 0; row -= T * RT) {
    cplx s[RT];
    vh_rows<RT>(V, ldv, k, hs, row, n, s);
#pragma unroll
    for (int i = 0; i < RT; i++)
      if (row + T * i < n) out(row + T * i, csub(x[row + T * i], s[i]));
  }
}
template <class Out>
__device__ __forceinline__ void cta_update(const cplx* V, long long ldv, int k, const cplx* hs, const cplx* x, int n,
                                           Out out) {
  if (k <= 4) update_block<4>(V, ldv, k, hs, x, n, out);
  else if (k <= 8) update_block<2>(V, ldv, k, hs, x, n, out);
  else update_block<1>(V, ldv, k, hs, x, n, out);
}

// out[l] = sum over the instance's CTAs of part[l ncta + r], l < k: a warp per
// coefficient, lanes over the CTAs, a fixed order.
__device__ void reduce_coeffs(const cplx* __restrict__ part, int ncta, int k, cplx* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int lb = 0; lb < k; lb += 4 * NW) {
    cplx s[4];
#pragma unroll
    for (int t = 0; t < 4; t++) s[t] = make_double2(0.0, 0.0);
    for (int r = lane; r < ncta; r += 32)
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const int l = lb + warp + NW * t;
        if (l < k) s[t] = cadd(s[t], __ldcg(&part[(long long)l * ncta + r]));
      }
    const cplx v = warp_sum_v<4>(s);
    const int l = lb + warp + NW * vector_of_lane<4>(lane);
    if (writes_vector<4>(lane) && l < k) out[l] = v;
  }
}

// sum over the instance's CTAs of pn (fixed order), by every warp for itself
__device__ __forceinline__ double sum_norms(const double* __restrict__ pn, int ncta) {
  double s = 0.0;
  for (int r = threadIdx.x & 31; r < ncta; r += 32) s += __ldcg(&pn[r]);
  return warp_sumd(s);
}
// sum_l |h_l|^2, by every warp for itself
__device__ __forceinline__ double coeff_norm(const cplx* hs, int k) {
  double s = 0.0;
  for (int l = threadIdx.x & 31; l < k; l += 32) s += cabs2(hs[l]);
  return warp_sumd(s);
}
// sum of one value per thread, to *out (thread 0 writes; redn: NW doubles)
__device__ void block_sum_to(double s, double* redn, double* out) {
  s = warp_sumd(s);
  if ((threadIdx.x & 31) == 0) redn[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < NW; q++) t += redn[q];
    *out = t;
  }
}

struct LzShared {
  cplx hs[KMAXS], hs2[KMAXS];
  cplx ucs[LZ_MAXU];
  double redn[NW];
};

template <bool RES>
__global__ void __launch_bounds__(T, 2) lanczos_step_kernel(const __grid_constant__ LzBatch b) {
  __shared__ LzShared sm;
  __shared__ cplx wsm[RES ? RES_ROWS : WCAP];
  __shared__ cplx usum[RES ? NW : 1][RES ? RES_ROWS : 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (blockIdx.x == 0 && tid < LZ_MAXI * PHASES) b.bar_next[tid] = 0;  // of the stream's next launch
  // the instance this CTA serves (instances own consecutive CTA ranges)
  int q = 0;
  while (q + 1 < b.ninst && b.in[q + 1].cta0 <= (int)blockIdx.x) q++;
  const LzInst& in = b.in[q];
  const int rank = (int)blockIdx.x - in.cta0, ncta = in.ncta, k = in.k;
  unsigned* bar = b.bar + PHASES * q;
  const int r0 = rank * in.rows, n = min(in.rows, in.n - r0);
  const cplx* V = in.V + r0;
  cplx* part = b.part + (long long)in.cta0 * KMAXS;
  cplx* part2 = b.part2 + (long long)in.cta0 * KMAXS;
  double* pn1 = b.pn1 + in.cta0;
  double* pn2 = b.pn2 + in.cta0;
  cplx* x = RES || n <= WCAP ? wsm : in.w + r0;  // this CTA's rows of w', w''

  // basis rows in registers: vectors warp + 8 t, rows lane + 32 i
  constexpr int RV = RES ? RES_K / NW : 1, RR = RES ? RES_ROWS / 32 : 1;
  cplx v[RV][RR];
  if constexpr (RES) {
#pragma unroll
    for (int t = 0; t < RV; t++)
#pragma unroll
      for (int i = 0; i < RR; i++)
        v[t][i] = (warp + NW * t < k && lane + 32 * i < n)
                      ? __ldcg(V + (long long)(warp + NW * t) * in.ldv + lane + 32 * i)
                      : make_double2(0.0, 0.0);
  }
  auto dots = [&](cplx* to) {
    if constexpr (RES) {
      cplx acc[RV];
#pragma unroll
      for (int t = 0; t < RV; t++) acc[t] = make_double2(0.0, 0.0);
#pragma unroll
      for (int i = 0; i < RR; i++) {
        const cplx xi = lane + 32 * i < n ? x[lane + 32 * i] : make_double2(0.0, 0.0);
#pragma unroll
        for (int t = 0; t < RV; t++) ccfma(acc[t], v[t][i], xi);
      }
      const cplx s = warp_sum_v<RV>(acc);
      const int l = warp + NW * vector_of_lane<RV>(lane);
      if (writes_vector<RV>(lane) && l < k) to[(long long)l * ncta + rank] = s;
    } else {
      cta_dots(V, in.ldv, k, x, n, ncta, rank, to);
    }
  };
  // x - V h, handed row by row to out
  auto update = [&](const cplx* hs, auto out) {
    if constexpr (RES) {
#pragma unroll
      for (int i = 0; i < RR; i++) {
        cplx s = make_double2(0.0, 0.0);
#pragma unroll
        for (int t = 0; t < RV; t++)
          if (warp + NW * t < k) cfma(s, v[t][i], hs[warp + NW * t]);
        usum[warp][lane + 32 * i] = s;
      }
      __syncthreads();
      if (tid < n) {
        cplx s = usum[0][tid];
#pragma unroll
        for (int u = 1; u < NW; u++) s = cadd(s, usum[u][tid]);
        out(tid, csub(x[tid], s));
      }
      __syncthreads();  // usum and x are read again in a second pass
    } else {
      cta_update(V, in.ldv, k, hs, x, n, out);
    }
  };

  // ---- projector (excited states): c = U^H v_j ----
  if (in.nu > 0) {
    cta_dots(in.U + r0, in.n, in.nu, in.V + (long long)in.j * in.ldv + r0, n, ncta, rank, part2);
    if (!group_barrier(bar + 0, ncta, b.err)) return;
    reduce_coeffs(part2, ncta, in.nu, sm.ucs);
    __syncthreads();
  }

  // ---- pass 1: w' = w [+ U c] - beta_{j-1} v_{j-1}; partial h = V^H w', |w'|^2 ----
  {
    const double bp = in.j > 0 ? in.sc->beta[in.j - 1] : 0.0;
    const cplx* vp = V + (long long)(in.j > 0 ? in.j - 1 : 0) * in.ldv;
    double s2 = 0.0;
    for (int r = tid; r < n; r += T) {
      cplx a = in.w[r0 + r];
      const cplx p = __ldcg(&vp[r]);
      for (int t = 0; t < in.nu; t++) a = cadd(a, cmul(in.U[r0 + r + (long long)t * in.n], sm.ucs[t]));
      if (in.j > 0) a = csub(a, cscale(p, bp));
      x[r] = a;
      s2 += cabs2(a);
    }
    block_sum_to(s2, sm.redn, &pn1[rank]);  // its barrier also publishes x to the warps
    dots(part);
  }
  if (!group_barrier(bar + 1, ncta, b.err)) return;

  // ---- every CTA of the instance: h, |w'|^2 and the DGKS test (after the
  // first pass |w''|^2 = |w'|^2 - |h|^2, the basis being orthonormal; a second
  // pass when that drops below half of |w'|^2, else beta_j = |w''| at once) ----
  const double nw = sum_norms(pn1, ncta);
  reduce_coeffs(part, ncta, k, sm.hs);
  __syncthreads();
  const double b2 = nw - coeff_norm(sm.hs, k);
  const bool flag = b2 < DGKS2 * nw;
  double beta = sqrt(fmax(b2, 0.0));
  double alpha = in.sigma + sm.hs[in.j].x;
  cplx* vn = in.V + (long long)(in.j + 1) * in.ldv + r0;

  if (!flag) {
    // w'' / beta_j straight into the basis (w'' itself into w when the basis
    // is full: the residual the restart needs)
    const double inv = beta > 0.0 ? 1.0 / beta : 0.0;
    const bool next = in.write_next;
    update(sm.hs, [&](int r, cplx a) {
      if (next) vn[r] = cscale(a, inv);
      else in.w[r0 + r] = a;
    });
  } else {
    // w'' and its second-pass dots
    update(sm.hs, [&](int r, cplx a) { x[r] = a; });
    __syncthreads();
    dots(part2);
    if (!group_barrier(bar + 2, ncta, b.err)) return;
    reduce_coeffs(part2, ncta, k, sm.hs2);
    __syncthreads();
    alpha += sm.hs2[in.j].x;
    // the norm after the second pass is summed explicitly (no cancellation
    // argument holds for it)
    double s2 = 0.0;
    update(sm.hs2, [&](int r, cplx a) {
      x[r] = a;
      s2 += cabs2(a);
    });
    block_sum_to(s2, sm.redn, &pn2[rank]);
    if (!group_barrier(bar + 3, ncta, b.err)) return;
    beta = sqrt(sum_norms(pn2, ncta));
    const double inv = beta > 0.0 ? 1.0 / beta : 0.0;
    for (int r = tid; r < n; r += T) {
      if (in.write_next) vn[r] = cscale(x[r], inv);
      else in.w[r0 + r] = x[r];
    }
  }

  // ---- alpha_j, beta_j ----
  if (rank == 0 && tid == 0) {
    in.sc->alpha[in.j] = alpha;
    in.sc->beta[in.j] = beta;
    in.sc->flag = flag ? 1 : 0;
    if (in.mirror) {  // mapped host memory, read by the host after the launch's event
      in.mirror->alpha[in.j] = alpha;
      in.mirror->beta[in.j] = beta;
    }
  }
}

// ---- normalised combinations: the start vector of a solve and its Ritz vector ----
// out = y / |y| with y = sum_l s_l V[:, l] (k > 0) or y = V[:, 0] (k = 0), of a
// group of instances in one cooperative launch: rows of y stay in shared memory
// across the barrier that closes the norms.  k = 0 replaces a zero or
// non-finite y by the flat vector.
__global__ void __launch_bounds__(T, 2) lanczos_combine_kernel(const __grid_constant__ LzCombineBatch b) {
  __shared__ cplx ysm[WCAP];
  __shared__ double ss[KMAXS], redn[NW];
  const int tid = threadIdx.x;
  if (blockIdx.x == 0 && tid < LZ_MAXI * PHASES) b.bar_next[tid] = 0;
  int q = 0;
  while (q + 1 < b.ninst && b.in[q + 1].cta0 <= (int)blockIdx.x) q++;
  const LzCombine& in = b.in[q];
  const int rank = (int)blockIdx.x - in.cta0, k = in.k;
  const int r0 = rank * in.rows, n = min(in.rows, in.n - r0);
  cplx* y = n <= WCAP ? ysm : in.out + r0;
  for (int l = tid; l < k; l += T) ss[l] = b.s[in.s0 + l];
  __syncthreads();
  double s2 = 0.0;
  for (int r = tid; r < n; r += T) {
    const cplx* v = in.V + r0 + r;
    cplx a = make_double2(0.0, 0.0);
    if (k == 0) a = v[0];
#pragma unroll 8
    for (int l = 0; l < k; l++) {
      const cplx x = __ldcg(v + (long long)l * in.ldv);
      a.x = fma(ss[l], x.x, a.x);
      a.y = fma(ss[l], x.y, a.y);
    }
    y[r] = a;
    s2 += cabs2(a);
  }
  block_sum_to(s2, redn, &b.pn[in.cta0 + rank]);
  if (!group_barrier(b.bar + PHASES * q, in.ncta, b.err)) return;
  const double nrm = sqrt(sum_norms(b.pn + in.cta0, in.ncta)), inv = 1.0 / nrm;
  const bool flat = k == 0 && !(nrm > 0.0 && nrm < __longlong_as_double(0x7ff0000000000000ll));
  const double f = 1.0 / sqrt((double)in.n);
  for (int r = tid; r < n; r += T) in.out[r0 + r] = flat ? make_double2(f, 0.0) : cscale(y[r], inv);
}

std::atomic<unsigned long long> g_lz_setup{0};
int g_lz_sms[64] = {0};

}  // namespace

// Workspace of a launch in complex entries: two arrays of partial dots and two
// of partial norms for at most two CTAs per SM.
static int lz_max_ctas(int sms) { return 2 * sms; }
long long lanczos_step_workspace(int sms) { return 2LL * lz_max_ctas(sms) * KMAXS + lz_max_ctas(sms); }

// One-time set-up of the device's kernels; its SM count.
static int lz_setup() {
  int dev = 0;
  MPSGPU_CUDA(cudaGetDevice(&dev));
  MPSGPU_CHECK(dev < 64, MPSGPU_INVALID, "lanczos step: device number");
  if (device_needs_setup(g_lz_setup)) {
    int nsm = 148;
    MPSGPU_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    for (const void* f : {(const void*)lanczos_step_kernel<false>, (const void*)lanczos_step_kernel<true>,
                          (const void*)lanczos_combine_kernel}) {
      int per = 0;
      MPSGPU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, T, 0));
      MPSGPU_CHECK(per >= 2, MPSGPU_BAD_SHAPE, "lanczos step: kernel does not fit twice on an SM");
    }
    g_lz_sms[dev] = nsm;
    mark_device_done(g_lz_setup);
  }
  return g_lz_sms[dev];
}

void lanczos_combine(const Stream& st, LzCombineBatch& b, cplx* ws, unsigned* bars, int& parity) {
  MPSGPU_CHECK(b.ninst >= 1 && b.ninst <= LZ_MAXI, MPSGPU_BAD_SHAPE, "lanczos combine: group size");
  const int G = lz_max_ctas(lz_setup());
  long long rows = 0;
  for (int q = 0; q < b.ninst; q++) rows += b.in[q].n;
  // a row per thread until every slot has a CTA
  const int per = std::max(T, ceil_div(ceil_div(rows, G - b.ninst), 32) * 32);
  int c0 = 0;
  for (int q = 0; q < b.ninst; q++) {
    LzCombine& in = b.in[q];
    MPSGPU_CHECK(in.n > 0 && in.k >= 0 && in.k <= KMAXS, MPSGPU_BAD_SHAPE, "lanczos combine: sizes");
    in.rows = per;
    in.ncta = ceil_div(in.n, per);
    in.cta0 = c0;
    c0 += in.ncta;
  }
  b.pn = reinterpret_cast<double*>(ws);
  b.bar = bars + parity * LZ_MAXI * PHASES;
  b.bar_next = bars + (parity ^ 1) * LZ_MAXI * PHASES;
  void* args[] = {&b};
  MPSGPU_CUDA(cudaLaunchCooperativeKernel((void*)lanczos_combine_kernel, dim3(c0), dim3(T), args, 0, st.s));
  after_launch(st);
  parity ^= 1;  // a launch that failed has not cleared the other set
}

void lanczos_step(const Stream& st, LzBatch& b, cplx* ws, unsigned* bars, int& parity) {
  MPSGPU_CHECK(b.ninst >= 1 && b.ninst <= LZ_MAXI, MPSGPU_BAD_SHAPE, "lanczos step: group size");
  double wsum = 0.0;
  long long rows = 0;
  int kmax = 0;
  for (int q = 0; q < b.ninst; q++) {
    LzInst& in = b.in[q];
    MPSGPU_CHECK(in.k == in.j + 1 && in.k <= KMAXS && in.n > 0, MPSGPU_BAD_SHAPE, "lanczos step: basis size");
    MPSGPU_CHECK(in.nu <= LZ_MAXU && in.nu <= KMAXS, MPSGPU_BAD_SHAPE, "lanczos step: projector size");
    rows += in.n;
    kmax = std::max(kmax, in.k);
    wsum += (double)in.n * (2.0 * in.k + 6.0 + 2.0 * in.nu);
  }
  const int nsm = lz_setup(), G = lz_max_ctas(nsm);
  // the form with the basis in registers while every CTA slot's share is at
  // most 64 rows
  long long small = 0;
  for (int q = 0; q < b.ninst; q++) small += ceil_div(b.in[q].n, RES_ROWS);
  const bool res = small <= G && kmax <= RES_K;
  int total = 0;
  if (res) {
    for (int q = 0; q < b.ninst; q++) {
      b.in[q].rows = RES_ROWS;
      b.in[q].ncta = ceil_div(b.in[q].n, RES_ROWS);
    }
  } else {
    // CTAs per instance in proportion to its bytes, one per SM until a CTA
    // has 256 rows (more CTAs mean more partial sums for each of them to add),
    // then two; evened out so that every CTA of an instance has equal rows
    const int slots = rows <= 256LL * nsm ? nsm : G;
    for (int q = 0; q < b.ninst; q++) {
      LzInst& in = b.in[q];
      const double w = (double)in.n * (2.0 * in.k + 6.0 + 2.0 * in.nu);
      const int c = std::max(1, std::min(ceil_div(in.n, RES_ROWS), (int)(slots * w / wsum)));
      in.rows = ceil_div(ceil_div(in.n, c), 32) * 32;
      in.ncta = ceil_div(in.n, in.rows);
      total += in.ncta;
    }
    while (total > G) {  // only when many instances took their minimum of one
      int big = 0;
      for (int q = 1; q < b.ninst; q++)
        if (b.in[q].ncta > b.in[big].ncta) big = q;
      LzInst& in = b.in[big];
      MPSGPU_CHECK(in.ncta > 1, MPSGPU_BAD_SHAPE, "lanczos step: more instances than co-resident CTAs");
      total -= in.ncta;
      in.rows = ceil_div(ceil_div(in.n, in.ncta - 1), 32) * 32;
      in.ncta = ceil_div(in.n, in.rows);
      total += in.ncta;
    }
  }
  int c0 = 0;
  for (int q = 0; q < b.ninst; q++) {
    b.in[q].cta0 = c0;
    c0 += b.in[q].ncta;
  }
  b.part = ws;
  b.part2 = b.part + (long long)G * KMAXS;
  b.pn1 = reinterpret_cast<double*>(b.part2 + (long long)G * KMAXS);
  b.pn2 = b.pn1 + G;
  b.bar = bars + parity * LZ_MAXI * PHASES;
  b.bar_next = bars + (parity ^ 1) * LZ_MAXI * PHASES;
  // algorithmic bytes: the basis read twice (projections, update), w read
  // and written three times (three-term step, update, normalisation) and
  // v_{j-1} once; the projector vectors twice
  double bytes = 0.0;
  for (int q = 0; q < b.ninst; q++)
    bytes += 16.0 * (double)b.in[q].n * (2.0 * b.in[q].k + 6.0 + 2.0 * b.in[q].nu);
  ProfScope ps(st, GemmProfiler::LZSTEP, bytes);
  void* args[] = {&b};
  MPSGPU_CUDA(cudaLaunchCooperativeKernel(res ? (void*)lanczos_step_kernel<true> : (void*)lanczos_step_kernel<false>,
                                          dim3(c0), dim3(T), args, 0, st.s));
  after_launch(st);
  parity ^= 1;  // a launch that failed has not cleared the other set
}

}  // namespace mpsgpu
