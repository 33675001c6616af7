// The two contractions of the effective-Hamiltonian product L.W.R.x
// (src/wrapper/multipliers/TensorMultiplier.cpp:61-93, three zgemm calls
// and three full permutes there) and of the environment updates
// (src/core/cpp/Operator.cpp:273-387), as two kernels on the FP64 tensor
// pipe (DMMA, mma.sync m8n8k4 f64):
//
//   heff_gemm1w   T2 = W . (A B): the product C = A B with the rows of a CTA
//                 tile chosen as (x, i0) -> row x + X i0 and the columns as
//                 (i1, y) -> column i1 + n_i1 y, so that every "pixel" (x, y)
//                 of the tile holds all n_i0 n_i1 values the MPO-leg matrix
//                 Wm contracts; the epilogue applies Wm per pixel from shared
//                 memory and writes T2 with arbitrary strides.  The
//                 intermediate A B never reaches global memory.
//   heff_gemm3    C = alpha (A1 B1 [+ A2 B2]) + beta Cin: the K range (two
//                 sources concatenated along K for the Hermitian multiplier)
//                 is split over the CTAs of a thread-block cluster, whose
//                 partial tiles are summed through distributed shared memory
//                 in rank order (deterministic, no second kernel).
//
// Both take a group of independent problems (different shapes) in one
// launch; tiles of all problems are numbered consecutively.  Operands are
// streamed through a three-stage shared-memory ring filled by cp.async
// (16-byte copies, zero-fill beyond the edges); complex entries stay
// interleaved in shared memory and each product is four real DMMAs, two into
// each accumulator (re, im): at two registers a value that leaves room for
// three CTAs per SM (with four accumulators two fit).  Groups of single-tile
// problems (bonds up to 16) keep four independent accumulators (re.re, -im.im,
// re.im, im.re): they are bound by the latency of one tile, and the chain of
// dependent DMMAs (27 cycles each) is half as long.
//
// Bound by the FP64 tensor pipe (a DMMA per 4 cycles and SM, 36.8 TF) once a
// group has tiles for every SM, by latency below.  Around the main loop:
//   - a thread keeps two running addresses per operand and an early-out per
//     slab instead of recomputing rows, columns and edges for every copy
//     (gemm3, eight problems at D = 96: 31.3 us -> 28.9 us);
//   - the leg epilogue is itself a product, pixels x legs, on the DMMA from
//     shared memory with offsets in tables (with it as scalar code eight problems
//     at D = 128, w = 5 took 84 us, now 67 us).
// Measured now: D = 128, w = 5, eight problems 67 and 57 us (20 and 23.5 TF), one
// 20.6 and 14.5 us; D = 64, w = 3, one 10.3 and 8.3 us; D = 400, w = 3, four 446
// and 440 us (28 TF).
#include <cooperative_groups.h>

#include <mutex>

#include "common.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace mpsgpu {

namespace {

constexpr int BK = 16;
constexpr int PADC = 2;      // complex padding of a shared row: conflict-free 16-byte fragment loads
constexpr int STAGES = 3;
// Warp groups splitting the k steps of every slab: two for 32-row tiles
// (twice the warps per SM for the small sweep shapes), one for 64-row
// tiles (whose accumulators already fill the registers); each group is 4
// warps, 2 x 2 over the tile.
template <int BM>
__host__ __device__ constexpr int kgroups() { return BM <= 32 ? 2 : 1; }
template <int BM>
__host__ __device__ constexpr int nthreads() { return 128 * kgroups<BM>(); }
// CTAs per SM that the registers are cut for.  Two for four accumulators: cut for
// three they spilled 150 bytes in launches of few blocks, which are bound by latency
// (both products of a site at D = 16, w = 3, one or sixteen problems: 12.3 -> 10.3 us and
// 14.3 -> 12.3 us; of 192 problems 22.5 -> 23.0 us).
template <int BM, int NS>
__host__ __device__ constexpr int ctas_per_sm() { return BM > 32 || NS == 4 ? 2 : 3; }

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp_async16(unsigned smem, const void* gmem, bool valid) {
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

template <int BM, int BN>
struct Ring {
  cplx A[STAGES][BK][BM + PADC];
  cplx B[STAGES][BK][BN + PADC];
};

template <int BM, int BN>
__host__ __device__ constexpr size_t ring_bytes() {
  return sizeof(Ring<BM, BN>) > (size_t)BM * (BN + PADC) * sizeof(cplx) ? sizeof(Ring<BM, BN>)
                                                                       : (size_t)BM * (BN + PADC) * sizeof(cplx);
}

// Accumulators of a warp tile: [MT][NT][set][half], sets re, im (NS = 2) or
// re.re, -im.im, re.im, im.re (NS = 4)
template <int BM, int BN, int NS>
struct Acc {
  static constexpr int WM = BM / 2, WN = BN / 2, MT = WM / 8, NT = WN / 8;
  double v[MT][NT][NS][2];
};

// The copies a thread makes of every slab: a column of the A slab (one row,
// AE values of k) and BE columns of the B slab at one k.  The addresses step by
// constants from slab to slab; only a slab that K ends in tests k.
template <int BM, int BN>
struct Feed {
  static constexpr int NT_ = nthreads<BM>(), AK = NT_ / BM, BC = NT_ / BK;
  static constexpr int AE = BK / AK, BE = BN / BC;
  const cplx *pa, *pb;          // the thread's first entries of the next slab
  long long ua, ub;             // between its entries
  long long sa;                 // of A per slab (B: BK)
  const cplx *base_a, *base_b;  // any valid address, for copies that read nothing
  unsigned da, db;              // shared addresses in stage 0
  bool oka;
  unsigned okb;                 // per column

  // row: the thread's row of A (offset arow, negative: outside); ncols: columns of the tile inside
  __device__ __forceinline__ void start(Ring<BM, BN>& r, const cplx* A, long long lda, long long arow, const cplx* B,
                                        long long ldb, int ncols) {
    const int tid = threadIdx.x, mt = tid % BM, ka = tid / BM, kb = tid % BK, nt = tid / BK;
    da = (unsigned)__cvta_generic_to_shared(&r.A[0][ka][mt]);
    db = (unsigned)__cvta_generic_to_shared(&r.B[0][kb][nt]);
    oka = arow >= 0;
    okb = 0;
#pragma unroll
    for (int u = 0; u < BE; u++) okb |= (nt + u * BC < ncols ? 1u : 0u) << u;
    source(A, lda, arow, B, ldb);
  }
  __device__ __forceinline__ void source(const cplx* A, long long lda, long long arow, const cplx* B, long long ldb) {
    const int tid = threadIdx.x;
    base_a = A;
    base_b = B;
    ua = AK * lda;
    sa = BK * lda;
    pa = A + (oka ? arow : 0) + (tid / BM) * lda;
    ub = BC * ldb;
    pb = B + tid % BK + (long long)(tid / BK) * ldb;
  }
  __device__ __forceinline__ void skip(int slabs) {
    pa += slabs * sa;
    pb += (long long)slabs * BK;
  }
  // the next slab into a stage; left: values of k it still holds
  __device__ __forceinline__ void issue(int stage, int left) {
    const unsigned a = da + stage * (unsigned)(BK * (BM + PADC) * sizeof(cplx));
    const unsigned b = db + stage * (unsigned)(BK * (BN + PADC) * sizeof(cplx));
    constexpr unsigned astep = AK * (BM + PADC) * sizeof(cplx), bstep = BC * sizeof(cplx);
    if (left >= BK) {
#pragma unroll
      for (int u = 0; u < AE; u++) cp_async16(a + u * astep, oka ? pa + u * ua : base_a, oka);
#pragma unroll
      for (int u = 0; u < BE; u++) {
        const bool ok = (okb >> u) & 1;
        cp_async16(b + u * bstep, ok ? pb + u * ub : base_b, ok);
      }
    } else {
      const int ka = threadIdx.x / BM, kb = threadIdx.x % BK;
#pragma unroll
      for (int u = 0; u < AE; u++) {
        const bool ok = oka && ka + u * AK < left;
        cp_async16(a + u * astep, ok ? pa + u * ua : base_a, ok);
      }
#pragma unroll
      for (int u = 0; u < BE; u++) {
        const bool ok = ((okb >> u) & 1) && kb < left;
        cp_async16(b + u * bstep, ok ? pb + u * ub : base_b, ok);
      }
    }
    pa += sa;
    pb += BK;
  }
};

// Main loop over nslab slabs: issue(stage, slab) copies one.
template <int BM, int BN, int NS, class Issue>
__device__ __forceinline__ void mainloop(Ring<BM, BN>& r, Acc<BM, BN, NS>& acc, int nslab, Issue issue) {
  using AC = Acc<BM, BN, NS>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm0 = (warp & 1) * AC::WM, wn0 = ((warp >> 1) & 1) * AC::WN, kg = warp >> 2;
  const int fr = lane >> 2, fc = lane & 3;
#pragma unroll
  for (int i = 0; i < AC::MT; i++)
#pragma unroll
    for (int j = 0; j < AC::NT; j++)
#pragma unroll
      for (int s = 0; s < NS; s++) acc.v[i][j][s][0] = acc.v[i][j][s][1] = 0.0;
#pragma unroll
  for (int s = 0; s < STAGES - 1; s++) {
    if (s < nslab) issue(s, s);
    cp_async_commit();
  }
  int st = 0, fill = STAGES - 1;  // stages: computed on, filled
  for (int it = 0; it < nslab; it++) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    if (it + STAGES - 1 < nslab) issue(fill, it + STAGES - 1);
    cp_async_commit();
    fill = fill + 1 == STAGES ? 0 : fill + 1;
#pragma unroll
    for (int kk0 = 0; kk0 < BK; kk0 += 4 * kgroups<BM>()) {
      const int kk = kk0 + 4 * kg;  // this group's k step of the slab
      double are[AC::MT], aim[AC::MT], naim[AC::MT], bre[AC::NT], bim[AC::NT];
#pragma unroll
      for (int i = 0; i < AC::MT; i++) {
        const cplx a = r.A[st][kk + fc][wm0 + i * 8 + fr];
        are[i] = a.x;
        aim[i] = a.y;
        naim[i] = -a.y;
      }
#pragma unroll
      for (int j = 0; j < AC::NT; j++) {
        const cplx b = r.B[st][kk + fc][wn0 + j * 8 + fr];
        bre[j] = b.x;
        bim[j] = b.y;
      }
#pragma unroll
      for (int i = 0; i < AC::MT; i++)
#pragma unroll
        for (int j = 0; j < AC::NT; j++) {
          constexpr int II = NS == 4 ? 1 : 0, RI = NS / 2, IR = NS - 1;
          dmma(acc.v[i][j][0][0], acc.v[i][j][0][1], are[i], bre[j]);
          dmma(acc.v[i][j][RI][0], acc.v[i][j][RI][1], are[i], bim[j]);
          dmma(acc.v[i][j][II][0], acc.v[i][j][II][1], naim[i], bim[j]);
          dmma(acc.v[i][j][IR][0], acc.v[i][j][IR][1], aim[i], bre[j]);
        }
    }
    st = st + 1 == STAGES ? 0 : st + 1;
  }
  cp_async_wait<0>();
  __syncthreads();
}

// Accumulators -> shared tile Cs[m][n] (ld BN + PADC): the warp groups'
// partial sums added in group order.  Every thread of the block calls it.
template <int BM, int BN, int NS>
__device__ __forceinline__ void acc_to_smem(const Acc<BM, BN, NS>& acc, cplx* Cs) {
  using AC = Acc<BM, BN, NS>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm0 = (warp & 1) * AC::WM, wn0 = ((warp >> 1) & 1) * AC::WN, kg = warp >> 2;
  const int fr = lane >> 2, fc = lane & 3;
#pragma unroll
  for (int g = 0; g < kgroups<BM>(); g++) {
    if (kg == g) {
#pragma unroll
      for (int i = 0; i < AC::MT; i++)
#pragma unroll
        for (int j = 0; j < AC::NT; j++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int m = wm0 + i * 8 + fr, n = wn0 + j * 8 + 2 * fc + h;
            cplx v;
            if constexpr (NS == 4)
              v = make_double2(acc.v[i][j][0][h] + acc.v[i][j][1][h], acc.v[i][j][2][h] + acc.v[i][j][3][h]);
            else
              v = make_double2(acc.v[i][j][0][h], acc.v[i][j][1][h]);
            cplx& c = Cs[m * (BN + PADC) + n];
            c = g == 0 ? v : cadd(c, v);
          }
    }
    __syncthreads();
  }
}

// Descriptors of a launch (consecutive tile ranges): up to GEMM_MAXP as kernel
// parameters, up to GEMM_MAXX in device memory, with the tile ranges as
// parameters (the search reads constant memory) and the tile's descriptor
// copied to shared memory.
template <class D>
struct Extern {
  int n;
  const D* d;
  int tile_begin[GEMM_MAXX];
};
template <class B>
struct Source;
template <class D, class B>
struct ParamSource {
  using Desc = D;
  struct Slot {};
  static constexpr bool IN_MEMORY = false;
  static __device__ __forceinline__ const D& pick(const B& b, int t, Slot&) {
    int q = 0;
    while (q + 1 < b.n && b.d[q + 1].tile_begin <= t) q++;
    return b.d[q];
  }
};
template <>
struct Source<Gemm1wBatch> : ParamSource<Gemm1wDesc, Gemm1wBatch> {};
template <>
struct Source<Gemm3Batch> : ParamSource<Gemm3Desc, Gemm3Batch> {};
template <class D>
struct Source<Extern<D>> {
  using Desc = D;
  using Slot = D;
  static constexpr bool IN_MEMORY = true;
  static __device__ __forceinline__ const D& pick(const Extern<D>& b, int t, Slot& slot) {
    int lo = 0, hi = b.n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (b.tile_begin[mid] <= t) lo = mid;
      else hi = mid - 1;
    }
    const int* src = reinterpret_cast<const int*>(b.d + lo);
    for (int e = threadIdx.x; e < (int)(sizeof(D) / sizeof(int)); e += blockDim.x)
      reinterpret_cast<int*>(&slot)[e] = src[e];
    __syncthreads();
    return slot;
  }
};

// ---------------------------------------------------------------------------
// heff_gemm1w
// ---------------------------------------------------------------------------
template <int BM, int BN, int NS, class B>
__global__ void __launch_bounds__(nthreads<BM>(), ctas_per_sm<BM, NS>()) heff_gemm1w_kernel(const __grid_constant__ B b) {
  __shared__ typename Source<B>::Slot slot;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NT_ = nthreads<BM>();
  Ring<BM, BN>& ring = *reinterpret_cast<Ring<BM, BN>*>(smem_raw);
  if (Source<B>::IN_MEMORY) await_predecessor();
  const Gemm1wDesc& d = Source<B>::pick(b, blockIdx.x, slot);
  const int local = blockIdx.x - d.tile_begin;
  const int TX = BM / d.n_i0, TY = BN / d.n_i1;
  const int tx = local % d.tiles_x, ty = local / d.tiles_x;
  const int x0 = tx * TX, y0 = ty * TY;
  const int tid = threadIdx.x;
  long long arow;
  {
    const int mt = tid % BM, xl = mt % TX, i0 = mt / TX, x = x0 + xl;
    arow = (i0 < d.n_i0 && x < d.X) ? x + (long long)d.X * i0 : -1;
  }
  Feed<BM, BN> feed;
  feed.start(ring, d.A, d.lda, arow, d.B + (long long)d.n_i1 * y0 * d.ldb, d.ldb, min(TY, d.Y - y0) * d.n_i1);
  Acc<BM, BN, NS> acc;
  if (!Source<B>::IN_MEMORY) await_predecessor();
  mainloop<BM, BN, NS>(ring, acc, (d.K + BK - 1) / BK, [&](int stage, int slab) { feed.issue(stage, d.K - slab * BK); });
  admit_successor();
  cplx* Cs = reinterpret_cast<cplx*>(smem_raw);
  constexpr int LD = BN + PADC;
  constexpr int ROOM = (int)(ring_bytes<BM, BN>() - BM * LD * sizeof(cplx));  // behind the tile
  const int nin = d.n_i0 * d.n_i1, nout = d.n_o0 * d.n_o1, nw = nin * nout, npix = TX * TY;
  // index of leg matrix element e (as stored) in an (i, o) order with o ld apart 1, i apart ld
  auto leg_index = [&](int e, int ld) {
    if (!d.w_ref) return e % nout + ld * (e / nout);
    int r = e;  // W(o0, i0, i1, o1)
    const int o0 = r % d.n_o0; r /= d.n_o0;
    const int i0 = r % d.n_i0; r /= d.n_i0;
    return o0 + d.n_o0 * (r / d.n_i1) + ld * (i0 + d.n_i0 * (r % d.n_i1));
  };
  // per pixel (x, y): out[o0 + n_o0 o1] = sum_{i0, i1} Wm[o, i0 + n_i0 i1] C[(x, i0), (i1, y)]
  const int kp = (nin + 3) & ~3, no8 = (nout + 7) / 8, np8 = (npix + 7) / 8, wld = 8 * no8 + 2;
  if (NS == 2 && kp * wld * (int)sizeof(cplx) + 20 * npix + 8 * nout + 8 * kp <= ROOM) {
    // on the tensor pipe: pixels x legs in times legs in x legs out, 8 x 8 tiles
    // over the warps; offsets of pixels and legs in tables
    cplx* Ws = Cs + BM * LD;
    long long* goff = reinterpret_cast<long long*>(Ws + kp * wld);  // global, -1 outside
    long long* ooff = goff + npix;
    int* poff = reinterpret_cast<int*>(ooff + nout);
    int* ioff = poff + npix;
    for (int e = tid; e < kp * wld; e += NT_) Ws[e] = make_double2(0.0, 0.0);
    for (int pix = tid; pix < npix; pix += NT_) {
      const int xl = pix % TX, yl = pix / TX, x = x0 + xl, y = y0 + yl;
      goff[pix] = (x < d.X && y < d.Y) ? x * d.ox + y * d.oy : -1;
      poff[pix] = xl * LD + d.n_i1 * yl;
    }
    for (int o = tid; o < nout; o += NT_) ooff[o] = (o % d.n_o0) * d.so0 + (o / d.n_o0) * d.so1;
    for (int i = tid; i < kp; i += NT_) ioff[i] = i < nin ? TX * (i % d.n_i0) * LD + i / d.n_i0 : -1;
    __syncthreads();
    for (int e = tid; e < nw; e += NT_) Ws[leg_index(e, wld)] = __ldcg(&d.Wm[e]);
    acc_to_smem<BM, BN, NS>(acc, Cs);  // ends with a barrier
    const int lane = tid & 31, fr = lane >> 2, fc = lane & 3;
    for (int u = tid >> 5; u < np8 * no8; u += NT_ / 32) {
      const int pix = (u % np8) * 8 + fr, o8 = (u / np8) * 8;
      const cplx* cp = Cs + (pix < npix ? poff[pix] : 0);
      double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0};
      for (int i = fc; i < kp; i += 4) {
        const int io = ioff[i];
        const cplx a = io >= 0 ? cp[io] : make_double2(0.0, 0.0), w = Ws[i * wld + o8 + fr];
        dmma(re[0], re[1], a.x, w.x);
        dmma(im[0], im[1], a.x, w.y);
        dmma(re[0], re[1], -a.y, w.y);
        dmma(im[0], im[1], a.y, w.x);
      }
      const long long go = pix < npix ? goff[pix] : -1;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int o = o8 + 2 * fc + h;
        if (go >= 0 && o < nout) d.out[go + ooff[o]] = make_double2(re[h], im[h]);
      }
    }
    return;
  }
  // scalar form (single-tile problems, and legs whose tables do not fit): ng
  // threads per pixel, each every ng-th output, two at a time
  const cplx* Wp = d.Wm;
  if (nw * (int)sizeof(cplx) <= ROOM) {
    cplx* Ws = Cs + BM * LD;
    for (int e = tid; e < nw; e += NT_) Ws[leg_index(e, nout)] = __ldcg(&d.Wm[e]);
    Wp = Ws;
  }
  acc_to_smem<BM, BN, NS>(acc, Cs);
  __syncthreads();
  const int ng = max(1, NT_ / npix);
  for (int p = tid; p < npix * ng; p += NT_) {
    const int pix = p % npix, g = p / npix;
    const int xl = pix % TX, yl = pix / TX;
    const int x = x0 + xl, y = y0 + yl;
    if (x >= d.X || y >= d.Y) continue;
    const cplx* cp = Cs + xl * LD + d.n_i1 * yl;
    cplx* op = d.out + x * d.ox + y * d.oy;
    for (int o = g; o < nout; o += 2 * ng) {
      const int o2 = o + ng < nout ? o + ng : o;
      cplx s = make_double2(0.0, 0.0), s2 = s;
      const cplx* w = Wp;
      for (int i1 = 0; i1 < d.n_i1; i1++) {
        const cplx* c0 = cp + i1;
        for (int i0 = 0; i0 < d.n_i0; i0++, c0 += TX * LD, w += nout) {
          const cplx c = *c0;
          s = cadd(s, cmul(w[o], c));
          s2 = cadd(s2, cmul(w[o2], c));
        }
      }
      op[(o % d.n_o0) * d.so0 + (o / d.n_o0) * d.so1] = s;
      if (o2 != o) op[(o2 % d.n_o0) * d.so0 + (o2 / d.n_o0) * d.so1] = s2;
    }
  }
}

// ---------------------------------------------------------------------------
// heff_gemm3 (cluster split-K)
// ---------------------------------------------------------------------------
template <int BM, int BN, int CS, int NS, class B>
__global__ void __cluster_dims__(CS, 1, 1) __launch_bounds__(nthreads<BM>(), ctas_per_sm<BM, NS>())
    heff_gemm3_kernel(const __grid_constant__ B b) {
  __shared__ typename Source<B>::Slot slot;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NT_ = nthreads<BM>();
  Ring<BM, BN>& ring = *reinterpret_cast<Ring<BM, BN>*>(smem_raw);
  const int tile = blockIdx.x / CS, rank = blockIdx.x % CS;
  if (Source<B>::IN_MEMORY) await_predecessor();
  const Gemm3Desc& d = Source<B>::pick(b, tile, slot);
  const int local = tile - d.tile_begin;
  const int tm = local % d.tiles_m, tn = local / d.tiles_m;
  const int m0 = tm * BM, n0 = tn * BN;
  // slabs of the two sources, dealt to the ranks in equal runs
  const int n1 = (d.K1 + BK - 1) / BK, ns = n1 + (d.K2 + BK - 1) / BK;
  const int chunk = (ns + CS - 1) / CS, s0 = min(ns, rank * chunk), s1 = min(ns, s0 + chunk);
  const int tid = threadIdx.x;
  const int m = m0 + tid % BM;
  const long long arow = m < d.M ? m : -1;
  Feed<BM, BN> feed;
  feed.start(ring, d.A1, d.lda1, arow, d.B1 + (long long)n0 * d.ldb1, d.ldb1, d.N - n0);
  auto second = [&]() { feed.source(d.A2, d.lda2, arow, d.B2 + (long long)n0 * d.ldb2, d.ldb2); };
  if (s0 <= n1) {
    feed.skip(s0);
  } else {
    second();
    feed.skip(s0 - n1);
  }
  Acc<BM, BN, NS> acc;
  if (!Source<B>::IN_MEMORY) await_predecessor();
  mainloop<BM, BN, NS>(ring, acc, s1 - s0, [&](int stage, int slab) {
    const int sl = s0 + slab;
    if (sl == n1) second();
    feed.issue(stage, sl < n1 ? d.K1 - sl * BK : d.K2 - (sl - n1) * BK);
  });
  admit_successor();
  cplx* Cs = reinterpret_cast<cplx*>(smem_raw);
  acc_to_smem<BM, BN, NS>(acc, Cs);
  // rows [r0, r1) of the tile are finished by this rank: the sum over the
  // ranks' partial tiles in rank order, then the epilogue
  constexpr int RPR = BM / CS;
  const int r0 = rank * RPR;
  if (CS > 1) {
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    for (int e = tid; e < RPR * BN; e += NT_) {
      const int mt = r0 + e % RPR, nt = e / RPR;
      const int m = m0 + mt, n = n0 + nt;
      cplx s = make_double2(0.0, 0.0);
#pragma unroll
      for (int rr = 0; rr < CS; rr++) {
        const cplx* peer = cl.map_shared_rank(Cs, rr);
        s = cadd(s, peer[mt * (BN + PADC) + nt]);
      }
      if (m < d.M && n < d.N) {
        cplx out = cmul(d.alpha, s);
        if (d.Cin) out = cadd(out, cmul(d.beta, d.Cin[m + (long long)n * d.ldcin]));
        d.C[m + (long long)n * d.ldc] = out;
      }
    }
    cl.sync();  // peers' shared tiles stay alive until every rank has read them
  } else {
    __syncthreads();
    for (int e = tid; e < BM * BN; e += NT_) {
      const int mt = e % BM, nt = e / BM;
      const int m = m0 + mt, n = n0 + nt;
      if (m < d.M && n < d.N) {
        cplx out = cmul(d.alpha, Cs[mt * (BN + PADC) + nt]);
        if (d.Cin) out = cadd(out, cmul(d.beta, d.Cin[m + (long long)n * d.ldcin]));
        d.C[m + (long long)n * d.ldc] = out;
      }
    }
  }
}

template <class K>
void set_smem(K kernel, size_t bytes) {
  MPSGPU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

template <class B>
void heff_setup1() {
  set_smem(heff_gemm1w_kernel<64, 32, 2, B>, ring_bytes<64, 32>());
  set_smem(heff_gemm1w_kernel<32, 32, 2, B>, ring_bytes<32, 32>());
  set_smem(heff_gemm1w_kernel<32, 32, 4, B>, ring_bytes<32, 32>());
}
template <class B>
void heff_setup3() {
  set_smem(heff_gemm3_kernel<64, 32, 1, 2, B>, ring_bytes<64, 32>());
  set_smem(heff_gemm3_kernel<64, 32, 2, 2, B>, ring_bytes<64, 32>());
  set_smem(heff_gemm3_kernel<64, 32, 4, 2, B>, ring_bytes<64, 32>());
  set_smem(heff_gemm3_kernel<32, 32, 1, 4, B>, ring_bytes<32, 32>());
  set_smem(heff_gemm3_kernel<32, 32, 1, 2, B>, ring_bytes<32, 32>());
  set_smem(heff_gemm3_kernel<32, 32, 2, 2, B>, ring_bytes<32, 32>());
  set_smem(heff_gemm3_kernel<32, 32, 4, 2, B>, ring_bytes<32, 32>());
  set_smem(heff_gemm3_kernel<32, 32, 8, 2, B>, ring_bytes<32, 32>());
}

std::atomic<unsigned long long> g_heff_setup{0};
std::mutex g_heff_mu;

void heff_setup() {
  if (!device_needs_setup(g_heff_setup)) return;
  std::lock_guard<std::mutex> lk(g_heff_mu);
  heff_setup1<Gemm1wBatch>();
  heff_setup1<Extern<Gemm1wDesc>>();
  heff_setup3<Gemm3Batch>();
  heff_setup3<Extern<Gemm3Desc>>();
  mark_device_done(g_heff_setup);
}

int sm_count() {
  static std::atomic<int> n{0};
  int v = n.load();
  if (v == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      v = 148;
    n.store(v);
  }
  return v;
}

template <class B>
void launch1(const Stream& st, const HeffLaunch& l, const B& b) {
  ProfScope ps(st, GemmProfiler::GEMM64, l.work);
  if (l.bm == 64)
    launch_chained(st, heff_gemm1w_kernel<64, 32, 2, B>, l.tiles, nthreads<64>(), ring_bytes<64, 32>(), b);
  else if (l.single)
    launch_chained(st, heff_gemm1w_kernel<32, 32, 4, B>, l.tiles, nthreads<32>(), ring_bytes<32, 32>(), b);
  else
    launch_chained(st, heff_gemm1w_kernel<32, 32, 2, B>, l.tiles, nthreads<32>(), ring_bytes<32, 32>(), b);
}

template <class B>
void launch3(const Stream& st, const HeffLaunch& l, const B& b) {
  ProfScope ps(st, GemmProfiler::GEMM64, l.work);
  const dim3 grid(l.tiles * l.cs);
#define MPSGPU_G3(BMv, CSv, NSv) \
  launch_chained(st, heff_gemm3_kernel<BMv, 32, CSv, NSv, B>, grid, nthreads<BMv>(), ring_bytes<BMv, 32>(), b)
  if (l.bm == 64 && l.cs == 1) {
    MPSGPU_G3(64, 1, 2);
  } else if (l.bm == 64 && l.cs == 2) {
    MPSGPU_G3(64, 2, 2);
  } else if (l.bm == 64) {
    MPSGPU_G3(64, 4, 2);
  } else if (l.single) {
    MPSGPU_G3(32, 1, 4);
  } else if (l.cs == 1) {
    MPSGPU_G3(32, 1, 2);
  } else if (l.cs == 2) {
    MPSGPU_G3(32, 2, 2);
  } else if (l.cs == 4) {
    MPSGPU_G3(32, 4, 2);
  } else {
    MPSGPU_G3(32, 8, 2);
  }
#undef MPSGPU_G3
}

// tile ranges and launch shape of a group of first contractions
void plan1(Gemm1wDesc* d, int n, HeffLaunch& l) {
  // 64 tile rows (half the B traffic of 32) once those tiles fill every SM
  // twice: eight problems at D = 128, w = 5 take 67 us against 72 us and at
  // D = 96 38 us against 39 us.  Below that 32 rows, with twice the tiles and
  // warps: four problems at D = 96 (192 tiles of 64 rows) take 23 us against
  // 27 us, one at D = 256, w = 3 (208) 41 us against 51 us
  long long t64 = 0;
  l.n = n;
  l.single = true;  // every problem one 16 x 16 tile of pixels at most
  for (int q = 0; q < n; q++) {
    l.single = l.single && d[q].X <= 16 && d[q].Y <= 16;
    MPSGPU_CHECK(d[q].n_i0 >= 1 && d[q].n_i0 <= 32 && d[q].n_i1 >= 1 && d[q].n_i1 <= 32 && d[q].X > 0 && d[q].Y > 0 &&
                     d[q].K > 0 &&
                     (!d[q].w_ref || d[q].n_i0 * d[q].n_i1 * d[q].n_o0 * d[q].n_o1 <= GEMM_WREF),
                 MPSGPU_BAD_SHAPE, "gemm1w: leg dimensions");
    t64 += (long long)ceil_div(d[q].X, 64 / d[q].n_i0) * ceil_div(d[q].Y, 32 / d[q].n_i1);
  }
  l.bm = t64 >= 2LL * sm_count() ? 64 : 32;
  l.tiles = 0;
  l.work = 0.0;  // GEMM flops plus the MPO-leg epilogue
  for (int q = 0; q < n; q++) {
    MPSGPU_CHECK(l.bm / d[q].n_i0 >= 1 && 32 / d[q].n_i1 >= 1, MPSGPU_BAD_SHAPE, "gemm1w: MPO legs wider than a tile");
    d[q].tiles_x = ceil_div(d[q].X, l.bm / d[q].n_i0);
    d[q].tiles_y = ceil_div(d[q].Y, 32 / d[q].n_i1);
    d[q].tile_begin = l.tiles;
    l.tiles += d[q].tiles_x * d[q].tiles_y;
    const double nin = (double)d[q].n_i0 * d[q].n_i1, nout = (double)d[q].n_o0 * d[q].n_o1;
    l.work += 8.0 * ((double)d[q].X * d[q].n_i0 * d[q].Y * d[q].n_i1 * d[q].K + (double)d[q].X * d[q].Y * nout * nin);
  }
}

void plan3(Gemm3Desc* d, int n, HeffLaunch& l) {
  const int nsm = sm_count();
  long long t64 = 0, t32 = 0;
  int kmax = 0;
  l.n = n;
  l.single = true;  // every problem at most one tile of a D = 16 site
  for (int q = 0; q < n; q++) {
    l.single = l.single && d[q].M <= 32 && d[q].N <= 16;
    MPSGPU_CHECK(d[q].M > 0 && d[q].N > 0 && d[q].K1 > 0 && d[q].K2 >= 0, MPSGPU_BAD_SHAPE, "gemm3: shape");
    t64 += (long long)ceil_div(d[q].M, 64) * ceil_div(d[q].N, 32);
    t32 += (long long)ceil_div(d[q].M, 32) * ceil_div(d[q].N, 32);
    kmax = std::max(kmax, d[q].K1 + d[q].K2);
  }
  // 64-row tiles (half the B traffic, two CTAs per SM by shared memory) where
  // they fill the GPU twice, by themselves or with the K range split over
  // clusters of 2 or 4, whose CTAs must come to between 3/2 and 7/4 of the
  // SMs (clusters of 4 do not pack the SMs of a GPC to the last one): eight
  // problems at D = 128, w = 5 in 57 us, against 65 us with 32 rows.  Otherwise
  // 32 rows in clusters of 2 up to two CTAs per SM, of 4 and 8 up to one (four
  // problems at D = 96: 144 CTAs in clusters of 2 take 19.6 us, 288 in clusters
  // of 4 23.6 us).  A rank's share is at least two slabs (one problem at D = 64,
  // w = 3, K = 192: clusters of 4 8.3 us, of 2 10.4 us).
  l.bm = 64;
  l.cs = 1;
  if (t64 < 2LL * nsm) {
    const int room = kmax / (2 * BK);  // largest useful cluster
    int c = 1;
    while (c < 4 && 4 * t64 * c * 2 <= 7LL * nsm && c * 2 <= room) c *= 2;
    if (!l.single && 2 * t64 * c >= 3LL * nsm) {
      l.cs = c;
    } else {
      l.bm = 32;
      while (!l.single && l.cs < 8 && t32 * l.cs * 2 <= (l.cs == 1 ? 2LL : 1LL) * nsm && l.cs * 2 <= room) l.cs *= 2;
    }
  }
  l.tiles = 0;
  l.work = 0.0;
  for (int q = 0; q < n; q++) {
    d[q].tiles_m = ceil_div(d[q].M, l.bm);
    d[q].tiles_n = ceil_div(d[q].N, 32);
    d[q].tile_begin = l.tiles;
    l.tiles += d[q].tiles_m * d[q].tiles_n;
    l.work += 8.0 * (double)d[q].M * d[q].N * (d[q].K1 + d[q].K2);
  }
}

template <class D>
Extern<D> external(const HeffLaunch& l, const D* dev) {
  Extern<D> e;
  e.n = l.n;
  e.d = dev;
  std::copy(l.tile_begin, l.tile_begin + l.n, e.tile_begin);
  return e;
}

}  // namespace

void heff_gemm1w(const Stream& st, Gemm1wBatch& b) {
  MPSGPU_CHECK(b.n >= 1 && b.n <= GEMM_MAXP, MPSGPU_BAD_SHAPE, "gemm1w: group size");
  heff_setup();
  HeffLaunch l;
  plan1(b.d, b.n, l);
  launch1(st, l, b);
}
void heff_gemm1w_plan(Gemm1wDesc* d, int n, HeffLaunch& l) {
  MPSGPU_CHECK(n >= 1 && n <= GEMM_MAXX, MPSGPU_BAD_SHAPE, "gemm1w: group size");
  plan1(d, n, l);
  for (int q = 0; q < n; q++) l.tile_begin[q] = d[q].tile_begin;
}
void heff_gemm1w(const Stream& st, const HeffLaunch& l, const Gemm1wDesc* dev) {
  heff_setup();
  launch1(st, l, external(l, dev));
}

void heff_gemm3(const Stream& st, Gemm3Batch& b) {
  MPSGPU_CHECK(b.n >= 1 && b.n <= GEMM_MAXP, MPSGPU_BAD_SHAPE, "gemm3: group size");
  heff_setup();
  HeffLaunch l;
  plan3(b.d, b.n, l);
  launch3(st, l, b);
}
void heff_gemm3_plan(Gemm3Desc* d, int n, HeffLaunch& l) {
  MPSGPU_CHECK(n >= 1 && n <= GEMM_MAXX, MPSGPU_BAD_SHAPE, "gemm3: group size");
  plan3(d, n, l);
  for (int q = 0; q < n; q++) l.tile_begin[q] = d[q].tile_begin;
}
void heff_gemm3(const Stream& st, const HeffLaunch& l, const Gemm3Desc* dev) {
  heff_setup();
  launch3(st, l, external(l, dev));
}

}  // namespace mpsgpu
