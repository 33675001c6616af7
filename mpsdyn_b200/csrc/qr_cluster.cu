// Householder QR of a site in one thread-block cluster (m <= 512, n <= 256),
// with the LAPACK conventions of qr.cu, read from and written to the site
// through strided views (no gather or scatter pass).
//
// Split.  The columns lie in the shared memory of the CTAs of a cluster, TILES
// tiles of 8 each: one while 16 CTAs hold them all (n <= 128), two beyond.  A
// panel is one tile.  Its owner factors it and publishes the reflectors V and the
// block factor T in global memory (L2); after one cluster barrier every tile
// right of it takes the block reflector.  The factorisation is a serial chain of
// n columns, so its bound is the latency of a column and of one block
// application per panel, not the arithmetic; the layout shortens both:
//
//   * Panel: a column per warp, 2 to 16 rows per lane in registers.  A column takes
//     one block barrier: its warp writes it to shared memory, and after the barrier
//     every warp takes x^H a and |x|^2 over its own lanes, the reflector's scalars
//     for itself, and updates its column.  Products with the columns left of the
//     pivot give V^H v, from which a ninth warp builds T one column behind.
//   * Block application: groups of 16 rows, two or four per warp; both products
//     (W = V^H C and C - V (T' W)) run on the FP64 tensor pipe with V copied to
//     shared memory, while Q is formed one panel ahead (up to 256 rows).
//   * Q: H_p leaves the unit columns left of 8 p alone; with two tiles a CTA holds
//     tiles r and 2 S - 1 - r, so that most applications reach one of them.
//
// Measured on the sites of a chain (launch to end): 256 x 128 in 213 us, 128 x 64
// in 80 us, 64 x 32 in 37 us, 256 x 256 in 415 us, 512 x 256 in 776 us.  Slices of
// 16 columns, two to a warp and two barriers a column, took 284, 111, 47, 620 and
// 767 us, a row per thread with sums folded over the lanes 317 us at 256 x 128, the
// global-memory kernels of qr.cu 3560 us at 512 x 256.  At 256 x 128 a warp waits
// 29 cycles at barriers for every instruction that it issues, and the FP64 tensor pipe
// is active 7 % of the time.
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace mpsgpu {

namespace {

constexpr int PB = 8;           // panel and tile width
constexpr int UW = 8;           // warps: a column of a panel each, or groups of 16 rows; one more builds T
constexpr int QT = 32 * (UW + 1);
constexpr int PAIR_ROWS = 32 * UW;        // two groups per warp
constexpr int MAX_ROWS = 2 * PAIR_ROWS;   // 16 rows per lane of a panel column
constexpr int SQT = 256;            // threads of the small form
constexpr int MAX_CTAS = 16;      // of a cluster
constexpr int NB = 16;            // width of the small form
// Strides (complex entries) of the shared arrays: 5 modulo 8 for the tiles and 9
// for the partial sums, so that the eight lanes of a 16-byte access phase fall
// into different banks in the tiles' three access patterns.
constexpr int RED_LD = 9, RED_SZ = 8 * RED_LD;  // a warp's partial W of one tile
constexpr int T_LD = 17, W2_LD = 20;            // small form

struct QcParams {
  int m, n, K, np, S, ld;
  int a_colfast, q_colfast;  // the view's columns are contiguous: lanes run over columns
  const cplx* A;             // m x n through va
  View2 va;
  cplx* Q;                   // m x K through vq (null: not wanted); may be A's buffer
  View2 vq;
  cplx* R;                   // K x n, zero below the diagonal (null: not wanted)
  long long ldr;
  cplx* V;                   // np panels of m x 8 (ld m), unit lower trapezoidal from row 8 p on
  cplx* T;                   // np block factors (8 x 8)
};

// Shared memory besides the tiles.
struct PanelShared {
  cplx x[2][MAX_ROWS];     // pivot columns
  cplx G[PB * PB], taus[PB];
};
struct ApplyShared {
  cplx red[2][UW][RED_SZ];
  cplx W[2][RED_SZ], W2[2][RED_SZ];
};
struct QcShared {
  cplx rt[PB * PB];  // rows of R of the panel's own columns
  cplx Ts[2][RED_SZ];
  union {
    PanelShared p;
    ApplyShared a;
  };
};
// 15 rows beyond the last one are zero in the tiles and in V: groups of 16 need no edge
__host__ __device__ constexpr int qc_ld(int m) { return m + 15 + ((5 - m - 15) & 7); }
// the tiles and V, twice where it is fetched one panel ahead
__host__ __device__ constexpr size_t qc_smem(int m, int tiles) {
  return sizeof(QcShared) + (size_t)(tiles + (m <= PAIR_ROWS ? 2 : 1)) * PB * qc_ld(m) * sizeof(cplx);
}
static_assert(qc_smem(MAX_ROWS, 2) <= 227 * 1024 && qc_smem(PAIR_ROWS, 2) <= 227 * 1024, "cluster QR plan exceeds the block limit");

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

__device__ __forceinline__ long long view_at(const View2& v, int i, int j) {
  const int rd = (int)v.rd, cd = (int)v.cd;
  return (i % rd) * v.r0 + (i / rd) * v.r1 + (j % cd) * v.c0 + (j / cd) * v.c1;
}

__device__ __forceinline__ void cfma(cplx& s, cplx a, cplx b) {  // s += a b
  s.x = fma(a.x, b.x, fma(-a.y, b.y, s.x));
  s.y = fma(a.x, b.y, fma(a.y, b.x, s.y));
}
__device__ __forceinline__ void ccfma(cplx& s, cplx a, cplx b) {  // s += conj(a) b
  s.x = fma(a.x, b.x, fma(a.y, b.y, s.x));
  s.y = fma(a.x, b.y, fma(-a.y, b.x, s.y));
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Sums of d and n over the lanes of a warp, in every lane: the first two exchanges
// halve what a lane carries.
__device__ __forceinline__ void warp_sum3(cplx& d, double& n) {
  const int lane = threadIdx.x & 31;
  const bool h = lane & 16, q = lane & 8;
  double k0 = (h ? n : d.x) + __shfl_xor_sync(0xffffffffu, h ? d.x : n, 16);
  const double y = d.y + __shfl_xor_sync(0xffffffffu, d.y, 16);
  // lanes below 16: d.x and d.y; from 16 on: n (and d.y)
  double v = (q ? y : k0) + __shfl_xor_sync(0xffffffffu, q ? k0 : y, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  d = make_double2(__shfl_sync(0xffffffffu, v, 0), __shfl_sync(0xffffffffu, v, 8));
  n = __shfl_sync(0xffffffffu, v, 16);
}

// Factor panel pn (rows j0.., jb reflectors) of the tile As (ld p.ld); V and T go
// to global memory, rows j0 to j0 + 7 of R to rt.
//
// Reflector of (alpha, x), both divided by a power of two when their squares
// leave the representable range: beta = -sign(Re alpha) |(alpha, x)|, u = alpha -
// beta (no cancellation: beta and Re alpha have opposite signs), v = (1, x / u),
// tau = -u / beta; x = 0 with a real alpha is tau = 0, H = I, as in zlarfg.
template <int RPL>
__device__ __noinline__ void qc_panel(const QcParams& p, const cplx* As, int pn, int j0, int jb, PanelShared& sh,
                                      cplx* rt) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int mp = p.m - j0;
  const cplx zero = make_double2(0.0, 0.0);
  cplx* T = p.T + pn * PB * PB;
  if (warp == UW) {
    // T one column behind: T[0:c, c] = -tau_c T[0:c, 0:c] G[0:c, c], T[c, c] = tau_c
    // (zlarft, forward, columnwise); lane l holds row l
    const int l = lane & 7;
    cplx t[PB];
#pragma unroll
    for (int c = 0; c < PB; c++) {
      t[c] = zero;
      if (c < jb) {
        __syncthreads();
        if (c == 0) continue;
      }
      // column c - 1; the last one of the panel after the closing barrier
      if (c - 1 >= 0 && c - 1 < jb - 1) {
        cplx s = zero;
#pragma unroll
        for (int q = 0; q < c - 1; q++) cfma(s, t[q], sh.G[q + PB * (c - 1)]);
        const cplx tau = sh.taus[c - 1];
        t[c - 1] = l < c - 1 ? cmul(make_double2(-tau.x, -tau.y), s) : l == c - 1 ? tau : zero;
      }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < PB; c++) {
      if (c == jb - 1) {
        cplx s = zero;
#pragma unroll
        for (int q = 0; q < c; q++) cfma(s, t[q], sh.G[q + PB * c]);
        const cplx tau = sh.taus[c];
        t[c] = l < c ? cmul(make_double2(-tau.x, -tau.y), s) : l == c ? tau : zero;
      }
      if (lane < PB) T[l + PB * c] = t[c];
    }
    return;
  }
  cplx a[RPL];  // column warp; rows from mp on are zero
#pragma unroll
  for (int i = 0; i < RPL; i++) {
    const int r = lane + 32 * i;
    a[i] = r < mp ? As[j0 + r + warp * p.ld] : zero;
  }
  // the warp's column of V and of R's rows, once it is final
  auto store = [&]() {
    cplx* V = p.V + (long long)pn * p.m * PB + j0 + (long long)warp * p.m;
#pragma unroll
    for (int i = 0; i < RPL; i++) {
      const int r = lane + 32 * i;
      cplx v = warp < jb ? a[i] : zero;
      if (i == 0 && lane <= warp) v = make_double2(lane == warp && warp < jb ? 1.0 : 0.0, 0.0);
      if (r < mp) V[r] = v;
    }
    if (lane < PB) rt[lane + PB * warp] = (warp >= jb || lane <= warp) ? a[0] : zero;
  };
#pragma unroll 1
  for (int c = 0; c < jb; c++) {
    cplx* xb = sh.x[c & 1];  // the buffer of column c - 2, which every warp has left
    if (warp == c) {
#pragma unroll
      for (int i = 0; i < RPL; i++) xb[lane + 32 * i] = a[i];
    }
    __syncthreads();
    cplx x[RPL];  // the pivot column below the pivot
#pragma unroll
    for (int i = 0; i < RPL; i++) x[i] = xb[lane + 32 * i];
    if (lane <= c) x[0] = zero;
    cplx alpha = xb[c];
    const cplx ac = make_double2(__shfl_sync(0xffffffffu, a[0].x, c), __shfl_sync(0xffffffffu, a[0].y, c));
    cplx d;  // x^H a
    double sig = 1.0, nrm2;
    bool identity = false;
    // a second pass with alpha and x scaled; every warp takes the same branch
#pragma unroll 1
    for (int pass = 0;; pass++) {
      cplx ds[2] = {zero, zero};
      double ns[2] = {0.0, 0.0};
#pragma unroll
      for (int i = 0; i < RPL; i++) {
        ccfma(ds[i & 1], x[i], a[i]);
        ns[i & 1] = fma(x[i].x, x[i].x, fma(x[i].y, x[i].y, ns[i & 1]));
      }
      d = cadd(ds[0], ds[1]);
      double n2 = ns[0] + ns[1];
      warp_sum3(d, n2);
      nrm2 = cabs2(alpha) + n2;
      if (pass || (n2 > 0.0 && nrm2 > 1e-280 && nrm2 < 1e280)) break;
      double mx = 0.0;
#pragma unroll
      for (int i = 0; i < RPL; i++) mx = fmax(mx, fmax(fabs(x[i].x), fabs(x[i].y)));
      for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      identity = mx == 0.0 && alpha.y == 0.0 && nrm2 == nrm2;  // (the maximum passes NaN by)
      if (identity) break;
      // divided by a power of two near the largest component (at least the smallest normal)
      const int top = __double2hiint(fmax(mx, fmax(fabs(alpha.x), fabs(alpha.y)))) & 0x7ff00000;
      sig = __hiloint2double(max(top, 0x00100000), 0);
#pragma unroll
      for (int i = 0; i < RPL; i++) x[i] = make_double2(x[i].x / sig, x[i].y / sig);
      alpha = make_double2(alpha.x / sig, alpha.y / sig);
    }
    if (identity) {
      if (lane == 0 && warp < c) sh.G[warp + PB * c] = zero;
      if (lane == 0 && warp == c) sh.taus[c] = zero;
      if (warp == c - 1) store();
      continue;
    }
    // (rsqrt would save a division, but takes 450 cycles here against 108 for
    // sqrt and 88 for a reciprocal)
    const double beta = -copysign(sqrt(nrm2), alpha.x);  // signed zero as LAPACK
    const cplx u = make_double2(alpha.x - beta, alpha.y);
    const double rb = 1.0 / beta, iu2 = 1.0 / cabs2(u);
    const cplx iu = make_double2(u.x * iu2, -u.y * iu2);
    if (warp > c) {
      // a <- H^H a: the pivot's row gets g / beta, the rows below g / (beta u) x
      // (columns with v^H a = 0 stay as they are, as in zlarf)
      const cplx g = cscale(cadd(ccmul(u, ac), d), rb), f = cmul(g, iu);
      if (g.x != 0.0 || g.y != 0.0) {
#pragma unroll
        for (int i = 0; i < RPL; i++) cfma(a[i], f, x[i]);
        if (lane == c) a[0] = cadd(a[0], g);
      }
    } else if (warp == c) {  // v, and the column's entry of R
      if (lane == 0) sh.taus[c] = make_double2(-u.x / beta, -u.y / beta);
#pragma unroll
      for (int i = 0; i < RPL; i++)
        if (i > 0 || lane > c) a[i] = cmul(x[i], iu);
      if (lane == c) a[0] = make_double2(beta * sig, 0.0);
    } else {
      // V[:, q]^H v_c = conj(V[c, q]) + (V[c+1:, q]^H x) / u
      if (lane == 0) sh.G[warp + PB * c] = cadd(cconj(ac), cmul(iu, cconj(d)));
      if (warp == c - 1) store();  // beside the other warps' updates
    }
  }
  if (warp >= jb - 1) store();
  __syncthreads();
}

// The panel's columns of R, after the panel is published: rows above j0 from the tile.
__device__ __forceinline__ void qc_store_r(const QcParams& p, const cplx* As, int pn, const cplx* rt) {
  const int j0 = pn * PB;
  for (int t = threadIdx.x; t < p.K * PB; t += QT) {
    const int r = t % p.K, q = t / p.K, col = j0 + q;
    if (col < p.n)
      p.R[r + col * p.ldr] = r < j0 ? As[r + q * p.ld] : r < j0 + PB ? rt[r - j0 + PB * q] : make_double2(0.0, 0.0);
  }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
// V (rows j0 on, ld p.ld) and T of panel pn to shared memory
__device__ __forceinline__ void qc_fetch(const QcParams& p, int pn, cplx* Vs, cplx* Ts) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j0 = pn * PB, mp = p.m - j0;
  if (warp < UW) {
    const cplx* V = p.V + ((long long)pn * PB + warp) * p.m + j0;
    for (int r = lane; r < mp; r += 32) cp_async16(&Vs[r + warp * p.ld], &V[r]);
    if (lane < 15) Vs[mp + lane + warp * p.ld] = make_double2(0.0, 0.0);
  } else {
    for (int t = lane; t < PB * PB; t += 32) cp_async16(&Ts[t % PB + t / PB * RED_LD], &p.T[pn * PB * PB + t]);
  }
  asm volatile("cp.async.commit_group;\n" ::);
}
template <int N>
__device__ __forceinline__ void qc_fetched() {  // all but the last N
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
  __syncthreads();
}

// C <- (I - V T' V^H) C for panel pn with V in Vs, T' = T^H (conjT: the
// factorisation's H^H) or T (forming Q), on tiles tile0 .. TILES - 1 of C (ld p.ld);
// GROUPS groups of 16 rows per warp.
template <int GROUPS, int TILES>
__device__ __forceinline__ void qc_apply(const QcParams& p, cplx* C0, const cplx* Vs, const cplx* Ts, int pn,
                                         bool conjT, int tile0, ApplyShared& sh) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ld = p.ld, fr = lane >> 2, fc = lane & 3, j0 = pn * PB, mp = p.m - j0;
  const cplx zero = make_double2(0.0, 0.0);
  cplx* C = C0 + j0;
  double wr[TILES][2], wi[TILES][2];  // W tiles (reflectors, columns)
#pragma unroll
  for (int j = 0; j < TILES; j++) wr[j][0] = wr[j][1] = wi[j][0] = wi[j][1] = 0.0;
  if (warp < UW) {
#pragma unroll
    for (int g = 0; g < GROUPS; g++) {
      const int r0 = 16 * (warp + UW * g);
      if (r0 >= mp) break;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int r = r0 + 4 * k + fc;
        const cplx v = Vs[r + fr * ld];
#pragma unroll
        for (int j = 0; j < TILES; j++) {
          if (j < tile0) continue;
          const cplx c = C[r + (8 * j + fr) * ld];
          dmma(wr[j][0], wr[j][1], v.x, c.x);  // conj(V)^T C
          dmma(wi[j][0], wi[j][1], v.x, c.y);
          dmma(wr[j][0], wr[j][1], v.y, c.y);
          dmma(wi[j][0], wi[j][1], -v.y, c.x);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < TILES; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) sh.red[j][warp][fr + (2 * fc + h) * RED_LD] = make_double2(wr[j][h], wi[j][h]);
  }
  __syncthreads();
  const int nw = min(UW, (mp + 15) / 16);  // warps with rows
  if (tid < 64 * TILES) {
    // one entry (el, eq) of W each; a warp holds whole columns
    const int j = tid >> 6, el = tid & 7, eq = (tid >> 3) & 7;
    if (j >= tile0) {
      cplx s = zero;
#pragma unroll
      for (int w = 0; w < UW; w++)
        if (w < nw) s = cadd(s, sh.red[j][w][el + eq * RED_LD]);
      sh.W[j][el + eq * RED_LD] = s;
      __syncwarp();
      cplx t[2] = {zero, zero};
#pragma unroll
      for (int l = 0; l < PB; l++) {  // T is zero below its diagonal
        if (conjT) ccfma(t[l & 1], Ts[l + el * RED_LD], sh.W[j][l + eq * RED_LD]);
        else cfma(t[l & 1], Ts[el + l * RED_LD], sh.W[j][l + eq * RED_LD]);
      }
      sh.W2[j][el + RED_LD * eq] = cadd(t[0], t[1]);
    }
  }
  __syncthreads();
  if (warp < UW) {
#pragma unroll
    for (int g = 0; g < GROUPS; g++) {
      const int r0 = 16 * (warp + UW * g);
      if (r0 >= mp) break;
      cplx v[2][2];
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const int r = r0 + 8 * i + fr;
          v[i][k] = Vs[r + (4 * k + fc) * ld];
        }
#pragma unroll
      for (int j = 0; j < TILES; j++) {
        if (j < tile0) continue;
        cplx acc[2][2];
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const int r = r0 + 8 * i + fr;
            acc[i][e] = C[r + (8 * j + 2 * fc + e) * ld];
          }
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const cplx w = sh.W2[j][4 * k + fc + fr * RED_LD];
#pragma unroll
          for (int i = 0; i < 2; i++) {
            dmma(acc[i][0].x, acc[i][1].x, -v[i][k].x, w.x);
            dmma(acc[i][0].y, acc[i][1].y, -v[i][k].x, w.y);
            dmma(acc[i][0].x, acc[i][1].x, v[i][k].y, w.y);
            dmma(acc[i][0].y, acc[i][1].y, -v[i][k].y, w.x);
          }
        }
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const int r = r0 + 8 * i + fr;
            C[r + (8 * j + 2 * fc + e) * ld] = acc[i][e];
          }
      }
    }
  }
  __syncthreads();
}

template <int PAIRS, int TILES>
__global__ void __launch_bounds__(QT, 1) qr_cluster_kernel(const __grid_constant__ QcParams p) {
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char qc_raw[];
  QcShared& sh = *reinterpret_cast<QcShared*>(qc_raw);
  cplx* C = reinterpret_cast<cplx*>(qc_raw + sizeof(QcShared));  // the tiles: 8 TILES columns, ld apart
  constexpr int SW = PB * TILES;
  cplx* Vs[2] = {C + SW * p.ld, C + (SW + (PAIRS == 1 ? PB : 0)) * p.ld};
  const int rank = (int)cl.block_rank(), tid = threadIdx.x;
  const int m = p.m, ld = p.ld;
  for (int t = tid; t < m * SW; t += QT) {
    const int r = p.a_colfast ? t / SW : t % m, c = p.a_colfast ? t % SW : t / m;
    const int j = rank * SW + c;
    cplx v = make_double2(0.0, 0.0);
    if (j < p.n) {
      v = p.A[view_at(p.va, r, j)];
      if (p.va.conj) v.y = -v.y;
    }
    C[r + c * ld] = v;
  }
  for (int t = tid; t < 15 * SW; t += QT) C[m + t % 15 + t / 15 * ld] = make_double2(0.0, 0.0);
  __syncthreads();
  for (int pn = 0; pn < p.np; pn++) {
    const int j0 = pn * PB, owner = pn / TILES, th = pn % TILES;
    if (rank == owner) {
      const int jb = min(PB, p.K - j0);
      const cplx* tile = C + th * PB * ld;
      if (m - j0 <= 64) qc_panel<2>(p, tile, pn, j0, jb, sh.p, sh.rt);
      else if (m - j0 <= 128) qc_panel<4>(p, tile, pn, j0, jb, sh.p, sh.rt);
      else if (PAIRS == 1 || m - j0 <= 256) qc_panel<8>(p, tile, pn, j0, jb, sh.p, sh.rt);
      else qc_panel<16>(p, tile, pn, j0, jb, sh.p, sh.rt);
    }
    cl.sync();  // V and T of panel pn published; the first one also ends every read of A
    if (p.R && rank == owner) qc_store_r(p, C + th * PB * ld, pn, sh.rt);
    const int tile0 = rank > owner ? 0 : rank == owner ? th + 1 : TILES;
    if (tile0 < TILES) {
      qc_fetch(p, pn, Vs[0], sh.Ts[0]);
      qc_fetched<0>();
      qc_apply<2 * PAIRS, TILES>(p, C, Vs[0], sh.Ts[0], pn, true, tile0, sh.a);
    }
  }
  if (p.R)  // the columns right of the last panel
    for (int th = 0; th < TILES; th++) {
      if (rank * TILES + th < p.np) continue;
      for (int t = tid; t < p.K * PB; t += QT) {
        const int r = t % p.K, j = (rank * TILES + th) * PB + t / p.K;
        if (j < p.n) p.R[r + j * p.ldr] = C[r + (th * PB + t / p.K) * ld];
      }
    }
  if (!p.Q) return;
  // Q = H_0 H_1 ... applied to unit columns, last panel first
  auto q_tile = [&](int th) { return th == 0 ? rank : 2 * p.S - 1 - rank; };
  __syncthreads();
  for (int t = tid; t < m * SW; t += QT) {
    const int r = t % m, c = t / m;
    C[r + c * ld] = make_double2(r == q_tile(c / PB) * PB + c % PB ? 1.0 : 0.0, 0.0);
  }
  // H_p reaches the tiles from p on; the first tile of a CTA is the left one
  const int last = min(p.np - 1, q_tile(TILES - 1));
  if (PAIRS == 1) qc_fetch(p, last, Vs[last & 1], sh.Ts[last & 1]);
  for (int pn = last; pn >= 0; pn--) {
    if (PAIRS == 1 && pn > 0) {  // one panel ahead
      qc_fetch(p, pn - 1, Vs[(pn - 1) & 1], sh.Ts[(pn - 1) & 1]);
      qc_fetched<1>();
    } else {
      if (PAIRS > 1) qc_fetch(p, pn, Vs[pn & 1], sh.Ts[pn & 1]);
      qc_fetched<0>();
    }
    qc_apply<2 * PAIRS, TILES>(p, C, Vs[pn & 1], sh.Ts[pn & 1], pn, false, q_tile(0) >= pn ? 0 : 1, sh.a);
  }
  for (int t = tid; t < m * SW; t += QT) {
    const int r = p.q_colfast ? t / SW : t % m, c = p.q_colfast ? t % SW : t / m;
    const int j = q_tile(c / PB) * PB + c % PB;
    if (j < p.K) {
      cplx v = C[r + c * ld];
      if (p.vq.conj) v.y = -v.y;
      p.Q[view_at(p.vq, r, j)] = v;
    }
  }
}

// ---- small form ----
struct __align__(16) Reflector {
  cplx iu, tau;      // 1 / u
  double beta;
  double sig;
  int kind;          // REFLECT, or RESCALED (sig != 1), or IDENTITY (tau = 0, H = I)
};
enum { REFLECT = 0, RESCALED = 1, IDENTITY = 2 };

// Sums of d0 and d1 over the lanes of a warp, in every lane: the first two
// exchanges halve what a lane carries (12 shuffles, and 8 to hand the four
// totals round; shuffles issue at one a clock per SM).
__device__ __forceinline__ void warp_sum_pair(cplx& d0, cplx& d1) {
  const int lane = threadIdx.x & 31;
  const bool h = lane & 16, q = lane & 8;
  const cplx s = h ? d0 : d1;
  cplx k = h ? d1 : d0;
  k.x += __shfl_xor_sync(0xffffffffu, s.x, 16);
  k.y += __shfl_xor_sync(0xffffffffu, s.y, 16);
  double v = q ? k.y : k.x;
  v += __shfl_xor_sync(0xffffffffu, q ? k.x : k.y, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  d0 = make_double2(__shfl_sync(0xffffffffu, v, 0), __shfl_sync(0xffffffffu, v, 8));
  d1 = make_double2(__shfl_sync(0xffffffffu, v, 16), __shfl_sync(0xffffffffu, v, 24));
}
// Reflector of (alpha, x), both divided by sig: tau and 1 / u by division, the
// column scaled by the sum of its largest components when squares leave the
// representable range.
__device__ __forceinline__ Reflector qc_reflector_small(cplx& x, cplx alpha, double n2) {
  Reflector h;
  h.sig = 1.0;
  h.kind = REFLECT;
  double x1 = fmax(fabs(x.x), fabs(x.y));
  x1 = warp_sum(x1);
  // scale test: x exactly zero, or every square and product representable
  const bool slow = x1 != 0.0 && (x1 < 1e-140 || x1 > 1e140 || fabs(alpha.x) > 1e140 || fabs(alpha.y) > 1e140);
  if (slow) {
    h.sig = x1;
    h.kind = RESCALED;
    x = make_double2(x.x / x1, x.y / x1);  // (1 / x1 may overflow)
    n2 = warp_sum(cabs2(x));
    alpha = make_double2(alpha.x / x1, alpha.y / x1);
  }
  h.beta = alpha.x;
  h.iu = h.tau = make_double2(0.0, 0.0);
  if (n2 == 0.0 && alpha.y == 0.0) {
    h.kind = IDENTITY;
    return h;
  }
  // |alpha|^2 + |x|^2 directly while it is representable (alpha alone can be
  // tiny when x is exactly zero), else with the largest part factored out
  const double nrm2 = alpha.x * alpha.x + alpha.y * alpha.y + n2;
  const double nrm = (!slow && nrm2 > 1e-280 && nrm2 < 1e280) ? sqrt(nrm2) : hypot3(alpha.x, alpha.y, sqrt(n2));
  h.beta = -copysign(nrm, alpha.x);
  h.tau = make_double2((h.beta - alpha.x) / h.beta, -alpha.y / h.beta);
  h.iu = recip_smith(make_double2(alpha.x - h.beta, alpha.y));
  return h;
}

// One panel of at most 32 rows (sites of bond dimension up to 16, and the ends
// of every chain): one CTA, a row per lane, warp q with columns q and q + 8, the
// scalars by the pivot's warp, Q = E - V (T V^H E) entry by entry from shared
// memory.  Sums, divisions and products are taken one by one in the order of the
// unblocked algorithm, so that the leading digits of 1 - lambda of nearly
// product states do not depend on the size class.
__global__ void __launch_bounds__(SQT) qr_small_kernel(const __grid_constant__ QcParams p) {
  __shared__ cplx C[NB * 33], Ts[NB * T_LD], G[NB * NB], taus[NB], rowc[NB], V[32 * NB], W2[NB * W2_LD];
  __shared__ Reflector reflector;
  const int tid = threadIdx.x, m = p.m, lane = tid & 31, warp = tid >> 5;
  join_stream();
  for (int t = tid; t < m * NB; t += SQT) {
    const int r = p.a_colfast ? t / NB : t % m, c = p.a_colfast ? t % NB : t / m;
    cplx v = make_double2(0.0, 0.0);
    if (c < p.n) {
      v = p.A[view_at(p.va, r, c)];
      if (p.va.conj) v.y = -v.y;
    }
    C[r + c * p.ld] = v;
  }
  for (int t = tid; t < NB * T_LD; t += SQT) Ts[t] = make_double2(0.0, 0.0);
  __syncthreads();
  cplx a[2];  // columns warp and warp + 8, row lane
#pragma unroll
  for (int j = 0; j < 2; j++)
    a[j] = lane < m ? C[lane + (warp + UW * j) * p.ld] : make_double2(0.0, 0.0);
  // one warp: T[0:c, c] = -tau_c T[0:c, 0:c] G[0:c, c], T[c, c] = tau_c (zlarft)
  auto t_column = [&](int c) {
    const int l = lane & 15;
    const cplx tc = taus[c];
    cplx s = make_double2(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < NB; q++)
      if (q >= l && q < c) s = cadd(s, cmul(Ts[l + T_LD * q], G[q + NB * c]));
    if (lane <= c) Ts[l + T_LD * c] = lane < c ? cmul(make_double2(-tc.x, -tc.y), s) : tc;
  };
#pragma unroll 1
  for (int c = 0; c < p.K; c++) {
    cplx* xc = V + (c & 1) * 32;  // the buffer of column c - 2, which every warp has left
    const bool pivot = warp == (c & (UW - 1));
    cplx x;  // the pivot column below the pivot
    if (pivot) {
      x = lane > c ? (c / UW ? a[1] : a[0]) : make_double2(0.0, 0.0);
      xc[lane] = x;
    }
    if (lane == c) {  // row c of the warp's columns, read back by the same warp
      rowc[warp] = a[0];
      rowc[warp + UW] = a[1];
    }
    __syncthreads();
    if (!pivot) x = xc[lane];
    // x^H a_q of the warp's columns (left of the pivot the conjugate of V^H x,
    // for the pivot column itself |x|^2)
    cplx d[2];
    auto dots = [&]() {
#pragma unroll
      for (int j = 0; j < 2; j++)
        d[j] = warp + UW * j == c ? make_double2(cabs2(x), 0.0) : cconj(ccmul(a[j], x));
      warp_sum_pair(d[0], d[1]);
    };
    dots();
    const cplx ac[2] = {rowc[warp], rowc[warp + UW]};
    if (pivot) {
      const Reflector h = qc_reflector_small(x, c / UW ? ac[1] : ac[0], c / UW ? d[1].x : d[0].x);
      if (lane == 0) reflector = h;
    } else if (c > 0 && warp == ((c + UW / 2) & (UW - 1))) {
      t_column(c - 1);  // while the pivot's warp takes the scalars
    }
    __syncthreads();
    const Reflector h = reflector;
    if (h.kind != REFLECT) {  // uniform over the block
      if (h.kind == IDENTITY) {
#pragma unroll
        for (int j = 0; j < 2; j++)
          if (warp + UW * j < c && lane == 0) G[warp + UW * j + NB * c] = make_double2(0.0, 0.0);
        if (tid == 0) taus[c] = make_double2(0.0, 0.0);
        continue;
      }
      // the products again with the rescaled column
      if (pivot) xc[lane] = x;
      __syncthreads();
      x = xc[lane];
      dots();
    }
    const cplx v = lane == c ? make_double2(1.0, 0.0) : lane > c ? cmul(x, h.iu) : make_double2(0.0, 0.0);
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int q = warp + UW * j;
      if (q > c) {
        const cplx s = cmul(cconj(h.tau), cadd(ac[j], ccmul(h.iu, d[j])));
        if (lane >= c) a[j] = csub(a[j], cmul(s, v));
      } else if (q == c) {
        if (lane > c) a[j] = v;
        if (lane == c) a[j] = make_double2(h.beta * h.sig, 0.0);
        if (lane == 0) taus[c] = h.tau;
      } else if (lane == 0) {
        G[q + NB * c] = cadd(cconj(ac[j]), cmul(h.iu, cconj(d[j])));
      }
    }
  }
  __syncthreads();
  if (warp == 0) t_column(p.K - 1);
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const int q = warp + UW * j;
    V[lane + 32 * q] = (lane >= m || q >= p.K || lane < q) ? make_double2(0.0, 0.0)
                                                           : (lane == q ? make_double2(1.0, 0.0) : a[j]);
    if (p.R && q < p.n && lane < p.K) p.R[lane + q * p.ldr] = lane <= q ? a[j] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  if (!p.Q) return;
  {
    const int i = tid & 15, q = tid >> 4;
    cplx s = make_double2(0.0, 0.0);
    for (int l = i; l < p.K; l++) s = cadd(s, cmul(Ts[i + T_LD * l], cconj(V[q + 32 * l])));
    W2[i + W2_LD * q] = s;
  }
  __syncthreads();
  for (int t = tid; t < m * NB; t += SQT) {
    const int r = p.q_colfast ? t / NB : t % m, q = p.q_colfast ? t % NB : t / m;
    if (q >= p.K) continue;
    cplx s = make_double2(0.0, 0.0);
#pragma unroll
    for (int l = 0; l < NB; l++) s = cadd(s, cmul(V[r + 32 * l], W2[l + W2_LD * q]));
    cplx o = csub(make_double2(r == q ? 1.0 : 0.0, 0.0), s);
    if (p.vq.conj) o.y = -o.y;
    p.Q[view_at(p.vq, r, q)] = o;
  }
}

using QcKernel = void (*)(const QcParams);
QcKernel qc_kernel(int m, int tiles) {
  if (tiles == 1) return m <= PAIR_ROWS ? qr_cluster_kernel<1, 1> : qr_cluster_kernel<2, 1>;
  return m <= PAIR_ROWS ? qr_cluster_kernel<1, 2> : qr_cluster_kernel<2, 2>;
}

std::atomic<unsigned long long> g_qc_setup{0};
std::atomic<int> g_qc_ctas[64];  // largest cluster the device can place with the largest plan

void qc_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int S, int m, int tiles, cudaStream_t s) {
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(S);
  cfg.blockDim = dim3(QT);
  cfg.dynamicSmemBytes = qc_smem(m, tiles);
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
}

int qc_max_ctas() {
  int dev = 0;
  MPSGPU_CUDA(cudaGetDevice(&dev));
  if (dev >= 64) return 0;
  if (device_needs_setup(g_qc_setup)) {
    int best = 0;
    for (int tiles : {1, 2})
      for (int m : {PAIR_ROWS, MAX_ROWS}) {
        MPSGPU_CUDA(cudaFuncSetAttribute(qc_kernel(m, tiles), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)qc_smem(m, tiles)));
        // clusters above 8 CTAs are an opt-in
        MPSGPU_CUDA(cudaFuncSetAttribute(qc_kernel(m, tiles), cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
      }
    for (int S : {8, MAX_CTAS}) {
      cudaLaunchConfig_t cfg;
      cudaLaunchAttribute attr[1];
      qc_config(cfg, attr, S, MAX_ROWS, 2, nullptr);
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, qc_kernel(MAX_ROWS, 2), &cfg) == cudaSuccess && clusters > 0)
        best = S;
      (void)cudaGetLastError();
    }
    g_qc_ctas[dev].store(best);
    mark_device_done(g_qc_setup);
  }
  return g_qc_ctas[dev].load();
}

}  // namespace

// Up to 512 rows and 256 columns, while the device can place a cluster of
// ceil(n/16) CTAs (the limits of the shared-memory plan).
bool cluster_qr_fits(int m, int n) {
  return (m <= 32 && n <= NB) || (m <= MAX_ROWS && ceil_div(n, 2 * PB) <= qc_max_ctas());
}

void cluster_qr(const Stream& st, int m, int n, const cplx* A, const View2& va, cplx* Q, const View2& vq, cplx* R,
                long long ldr, Scratch& scratch) {
  QcParams p;
  p.m = m; p.n = n; p.K = std::min(m, n);
  p.np = ceil_div(p.K, PB);
  p.A = A; p.va = va;
  p.Q = Q; p.vq = vq;
  p.R = R; p.ldr = ldr;
  p.a_colfast = va.cd == 1 && va.c1 == 1;
  p.q_colfast = vq.cd == 1 && vq.c1 == 1;
  p.V = p.T = nullptr;
  // factorisation and explicit Q, complex flops (8 per complex MAC)
  ProfScope ps(st, GemmProfiler::QR, qr_flops(m, n));
  if (m <= 32 && n <= NB) {
    p.S = 1;
    p.ld = m | 1;
    launch_chained(st, qr_small_kernel, 1, SQT, 0, p);
    return;
  }
  // one tile per CTA while the cluster holds them all: half the work between two
  // panels of a CTA with two
  const int tiles = ceil_div(n, PB) <= qc_max_ctas() ? 1 : 2;
  p.S = ceil_div(n, PB * tiles);
  p.ld = qc_ld(m);
  p.V = (cplx*)scratch.get(((size_t)p.np * m * PB + (size_t)p.np * PB * PB) * sizeof(cplx));
  p.T = p.V + (size_t)p.np * m * PB;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  qc_config(cfg, attr, p.S, m, tiles, st.s);
  MPSGPU_CUDA(cudaLaunchKernelEx(&cfg, qc_kernel(m, tiles), p));
  after_launch(st);
}

}  // namespace mpsgpu
