// Householder QR of a site in one thread-block cluster (m <= 512, n <= 256),
// with the LAPACK conventions of qr.cu, read from and written to the site
// through strided views (no gather or scatter pass).
//
// Split.  Column slice q (16 columns) lives in the shared memory of CTA q of
// a cluster of ceil(n/16) CTAs; panel q is the first min(16, K - 16 q)
// columns of slice q.  The owner factors its panel and publishes the
// reflectors V and the block factor T in global memory (L2); after one
// cluster barrier every CTA to its right applies the block reflector to its
// slice.  The factorisation is a serial chain of n columns, so its bound is
// the latency of a column (a dot product over the block, the reflector's
// scalars, an update, a barrier) plus one block application per panel, not
// the arithmetic; the layout below shortens both:
//
//   * Panel: warp q holds columns q and q + 8 in registers (RPL rows per
//     lane; two columns share the loads of the pivot column).  The
//     pivot's warp writes its column, unscaled, to shared memory; after a
//     barrier every warp takes x^H a_q over its own lanes (shuffles, no block
//     reduction), the pivot's |x|^2 and then the reflector's scalars; a second
//     barrier, and each warp updates its columns.  Columns left of the pivot
//     give the products V^H v of the block factor in the same pass, and an
//     idle warp builds T one column behind.
//   * Block application: rows are cut into groups of 16, one warp each; both
//     products (W = V^H C and C - V (T' W)) run on the FP64 tensor pipe with
//     V read once per product from L2 straight into fragments, so the only
//     block-wide steps are the sum of the warps' partial W and T' W.
//   * Q: columns are dealt to the CTAs in pairs, cyclically, so that every
//     CTA applies each block reflector to an equal part of the columns it
//     reaches (H_p leaves the unit columns left of 16 p alone).
//
// Measured on the sites of a chain (one QR at a time, launch to end): 256 x 128
// in 265 us, 512 x 256 in 790 us, 64 x 32 in 47 us; a form with the block
// reflectors in distributed shared memory and scalar products took 484-570 us
// at 256 x 128, the global-memory kernels of qr.cu 3560 us at 512 x 256.  Per
// column of a 256-row panel 2300 cycles (two shared-memory passes over the
// pivot column and the FP64 products 1000, the chain of shuffles, square root
// and reciprocals 900), per block application 9-10 thousand (8200 on the FP64
// tensor pipe).
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace mpsgpu {

namespace {

constexpr int NB = 16;               // slice and panel width
constexpr int UW = 8;                // warps: two columns of a panel each, or groups of 16 rows
constexpr int QT = 32 * UW;
constexpr int MAX_ROWS = 512;         // 16 rows per lane of a panel column
constexpr int MAX_SLICES = 16;
// Strides (complex entries) of the shared arrays; odd, or 4 modulo 8, so that
// the eight lanes of a 16-byte access phase fall into different banks.
constexpr int RED_LD = 17, RED_SZ = 272;  // a warp's partial W: column stride, array stride
constexpr int T_LD = 17, W2_LD = 20;

struct QcParams {
  int m, n, K, npa, np, S, ld;
  int a_colfast, q_colfast;  // the view's columns are contiguous: lanes run over columns
  const cplx* A;             // m x n through va
  View2 va;
  cplx* Q;                   // m x K through vq (null: not wanted); may be A's buffer
  View2 vq;
  cplx* R;                   // K x n, zero below the diagonal (null: not wanted)
  long long ldr;
  cplx* V;                   // np panels of m x 16 (ld m), unit lower trapezoidal
  cplx* T;                   // np block factors (16 x 16)
};

__host__ __device__ constexpr size_t qc_smem_elems(int ld) {
  return (size_t)NB * ld + (size_t)UW * RED_SZ + NB * T_LD + NB * W2_LD + 2 * NB * NB + 2 * NB;
}
__host__ constexpr int qc_ld(int m) { return m | 1; }
static_assert(qc_smem_elems(qc_ld(MAX_ROWS)) * sizeof(cplx) <= 227 * 1024, "cluster QR plan exceeds the block limit");
static_assert(QT == NB * NB, "one thread per entry of a block factor");
static_assert(2 * MAX_ROWS <= UW * RED_SZ, "the pivot columns share the partial sums' space");

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
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Reflector of (alpha, x), both divided by sig: beta = -sign(Re alpha)
// |(alpha, x)|, u = alpha - beta (no cancellation: beta and Re alpha have
// opposite signs), v = (1, x / u), tau = -u / beta.
struct __align__(16) Reflector {
  cplx u, iu;        // u, 1 / u
  double beta, rb;   // beta, 1 / beta
  double sig;
  cplx tau;          // (small form)
  int kind;          // REFLECT, or RESCALED (sig != 1), or IDENTITY (tau = 0, H = I)
};
enum { REFLECT = 0, RESCALED = 1, IDENTITY = 2 };

// x = 0, or squares outside the representable range: the rows of x divided in
// place by a power of two near the largest component first, as zlarfg rescales.
template <int RPL>
__device__ __noinline__ void qc_rescale(cplx (&x)[RPL], cplx& alpha, Reflector& h, double& n2) {
  double mx = 0.0;
#pragma unroll
  for (int i = 0; i < RPL; i++) mx = fmax(mx, fmax(fabs(x[i].x), fabs(x[i].y)));
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  h.kind = mx == 0.0 && alpha.y == 0.0 ? IDENTITY : RESCALED;
  if (h.kind == IDENTITY) return;
  const int top = __double2hiint(fmax(mx, fmax(fabs(alpha.x), fabs(alpha.y)))) & 0x7ff00000;
  const double big = __hiloint2double(max(top, 0x00100000), 0);  // its power of two (at least the smallest normal)
  h.sig = big;
  n2 = 0.0;
#pragma unroll
  for (int i = 0; i < RPL; i++) {
    x[i] = make_double2(x[i].x / big, x[i].y / big);
    n2 += cabs2(x[i]);
  }
  n2 = warp_sum(n2);
  alpha = make_double2(alpha.x / big, alpha.y / big);
}

// The reflector of a column by the warp that holds it: x its rows below the
// pivot (zero elsewhere), n2 the sum of their squares, alpha the pivot.
template <int RPL>
__device__ __forceinline__ Reflector qc_reflector(cplx (&x)[RPL], cplx alpha, double n2) {
  Reflector h;
  h.sig = 1.0;
  h.kind = REFLECT;
  double nrm2 = cabs2(alpha) + n2;
  if (!(n2 > 0.0 && nrm2 > 1e-280 && nrm2 < 1e280)) {
    cplx xs[RPL];  // a copy: the address of x would move it out of registers
#pragma unroll
    for (int i = 0; i < RPL; i++) xs[i] = x[i];
    qc_rescale<RPL>(xs, alpha, h, n2);
#pragma unroll
    for (int i = 0; i < RPL; i++) x[i] = xs[i];
    nrm2 = cabs2(alpha) + n2;
  }
  // (rsqrt would save a division, but takes 450 cycles here against 108 for
  // sqrt and 88 for a reciprocal)
  const double nrm = sqrt(nrm2);
  h.beta = -copysign(nrm, alpha.x);  // signed zero as LAPACK
  h.u = make_double2(alpha.x - h.beta, alpha.y);
  const double q = 1.0 / cabs2(h.u);
  h.rb = 1.0 / h.beta;
  h.iu = make_double2(h.u.x * q, -h.u.y * q);
  return h;
}

// The same for the small form (see qc_small_q): tau and 1 / u by division, the
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
  h.u = h.iu = h.tau = make_double2(0.0, 0.0);
  h.rb = 0.0;
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

// Factor panel pn (rows j0.., jb reflectors) of the slice As (this CTA's, ld
// p.ld); V, T and the panel's columns of R go to global memory.
template <int RPL, bool SMALL>
__device__ void qc_panel(const QcParams& p, const cplx* As, int pn, int j0, int jb, cplx* xb, cplx* Ts, cplx* G,
                         cplx* taus, cplx* rowc, Reflector* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int mp = p.m - j0;
  for (int t = threadIdx.x; t < NB * T_LD; t += QT) Ts[t] = make_double2(0.0, 0.0);
  __syncthreads();  // also: the last block application stored the slice by rows
  cplx a[2][RPL];   // columns warp and warp + 8; rows from mp on are zero
#pragma unroll
  for (int j = 0; j < 2; j++)
#pragma unroll
    for (int i = 0; i < RPL; i++) {
      const int r = lane + 32 * i;
      a[j][i] = r < mp ? As[j0 + r + (warp + UW * j) * p.ld] : make_double2(0.0, 0.0);
    }
  // one warp: T[0:c, c] = -tau_c T[0:c, 0:c] G[0:c, c], T[c, c] = tau_c (zlarft,
  // forward, columnwise); lanes l and l + 16 take the even and odd terms of row l
  auto t_column = [&](int c) {
    const int l = lane & 15, h = lane >> 4;
    const cplx tc = taus[c];
    if constexpr (SMALL) {
      cplx s = make_double2(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < NB; q++)
        if (q >= l && q < c) s = cadd(s, cmul(Ts[l + T_LD * q], G[q + NB * c]));
      if (lane <= c) Ts[l + T_LD * c] = lane < c ? cmul(make_double2(-tc.x, -tc.y), s) : tc;
      return;
    }
    cplx s0 = make_double2(0.0, 0.0), s1 = s0;
#pragma unroll
    for (int q = 0; q < NB; q += 4) {
      if (q + h < c) cfma(s0, Ts[l + T_LD * (q + h)], G[q + h + NB * c]);
      if (q + 2 + h < c) cfma(s1, Ts[l + T_LD * (q + 2 + h)], G[q + 2 + h + NB * c]);
    }
    cplx s = cadd(s0, s1);
    s.x += __shfl_xor_sync(0xffffffffu, s.x, 16);
    s.y += __shfl_xor_sync(0xffffffffu, s.y, 16);
    if (lane <= c) Ts[l + T_LD * c] = lane < c ? cmul(make_double2(-tc.x, -tc.y), s) : tc;
  };
#pragma unroll 1
  for (int c = 0; c < jb; c++) {
    cplx* xc = xb + (c & 1) * MAX_ROWS;  // the buffer of column c - 2, which every warp has left
    const bool pivot = warp == (c & (UW - 1));
    const int pj = c / UW;
    cplx x[RPL];  // the pivot column below the pivot
    if (pivot) {
#pragma unroll
      for (int i = 0; i < RPL; i++) {
        x[i] = (i > 0 || lane > c) ? (pj ? a[1][i] : a[0][i]) : make_double2(0.0, 0.0);
        xc[lane + 32 * i] = x[i];
      }
    }
    if (lane == c) {  // row c of the warp's columns, read back by the same warp
      rowc[warp] = a[0][0];
      rowc[warp + UW] = a[1][0];
    }
    __syncthreads();
    if (!pivot) {
#pragma unroll
      for (int i = 0; i < RPL; i++) x[i] = xc[lane + 32 * i];
    }
    // x^H a_q of the warp's columns (left of the pivot the conjugate of V^H x,
    // for the pivot column itself |x|^2)
    cplx d[2];
    auto dots = [&]() {
#pragma unroll
      for (int j = 0; j < 2; j++) {
        d[j] = make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < RPL; i++) {
          if constexpr (SMALL)
            d[j] = warp + UW * j == c ? make_double2(cabs2(x[i]), 0.0) : cconj(ccmul(a[j][i], x[i]));
          else ccfma(d[j], x[i], a[j][i]);
        }
      }
      warp_sum_pair(d[0], d[1]);
    };
    dots();
    const cplx ac[2] = {rowc[warp], rowc[warp + UW]};
    if (pivot) {
      const cplx alpha = pj ? ac[1] : ac[0];
      const double n2 = pj ? d[1].x : d[0].x;
      Reflector h;
      if constexpr (SMALL) h = qc_reflector_small(x[0], alpha, n2);
      else h = qc_reflector<RPL>(x, alpha, n2);
      if (lane == 0) *sh = h;
    } else if (c > 0 && warp == ((c + UW / 2) & (UW - 1))) {
      t_column(c - 1);  // while the pivot's warp takes the scalars
    }
    __syncthreads();
    const Reflector h = *sh;
    if (h.kind != REFLECT) {  // uniform over the block
      if (h.kind == IDENTITY) {
#pragma unroll
        for (int j = 0; j < 2; j++)
          if (warp + UW * j < c && lane == 0) G[warp + UW * j + NB * c] = make_double2(0.0, 0.0);
        if (threadIdx.x == 0) taus[c] = make_double2(0.0, 0.0);
        continue;
      }
      // the products again with the rescaled column
      if (pivot) {
#pragma unroll
        for (int i = 0; i < RPL; i++) xc[lane + 32 * i] = x[i];
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < RPL; i++) x[i] = xc[lane + 32 * i];
      dots();
    }
    if constexpr (SMALL) {
      const cplx v = lane == c ? make_double2(1.0, 0.0) : lane > c ? cmul(x[0], h.iu) : make_double2(0.0, 0.0);
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int q = warp + UW * j;
        if (q > c) {
          const cplx s = cmul(cconj(h.tau), cadd(ac[j], ccmul(h.iu, d[j])));
          if (lane >= c) a[j][0] = csub(a[j][0], cmul(s, v));
        } else if (q == c) {
          if (lane > c) a[j][0] = v;
          if (lane == c) a[j][0] = make_double2(h.beta * h.sig, 0.0);
          if (lane == 0) taus[c] = h.tau;
        } else if (lane == 0) {
          G[q + NB * c] = cadd(cconj(ac[j]), cmul(h.iu, cconj(d[j])));
        }
      }
    } else {
      // columns right of the pivot: a_q <- H^H a_q, row c gets g / beta, the rows
      // below g / (beta u) x (columns with v^H a_q = 0 stay as they are, as in zlarf)
      cplx g[2], f[2];
      bool upd[2];
#pragma unroll
      for (int j = 0; j < 2; j++) {
        g[j] = cscale(cadd(ccmul(h.u, ac[j]), d[j]), h.rb);
        f[j] = cmul(g[j], h.iu);
        upd[j] = warp + UW * j > c && (g[j].x != 0.0 || g[j].y != 0.0);
      }
      if (upd[0] && upd[1]) {
#pragma unroll
        for (int i = 0; i < RPL; i++) {
          cfma(a[0][i], f[0], x[i]);
          cfma(a[1][i], f[1], x[i]);
        }
      } else if (upd[1]) {
#pragma unroll
        for (int i = 0; i < RPL; i++) cfma(a[1][i], f[1], x[i]);
      } else if (upd[0]) {
#pragma unroll
        for (int i = 0; i < RPL; i++) cfma(a[0][i], f[0], x[i]);
      }
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int q = warp + UW * j;
        if (upd[j] && lane == c) a[j][0] = cadd(a[j][0], g[j]);
        // V[:, q]^H v_c = conj(V[c, q]) + (V[c+1:, q]^H x) / u
        if (q < c && lane == 0) G[q + NB * c] = cadd(cconj(ac[j]), cmul(h.iu, cconj(d[j])));
        if (q == c) {  // v_c, and the column's entry of R
#pragma unroll
          for (int i = 0; i < RPL; i++)
            if (i > 0 || lane > c) a[j][i] = cmul(x[i], h.iu);
          if (lane == c) a[j][0] = make_double2(h.beta * h.sig, 0.0);
          if (lane == 0) taus[c] = make_double2(-h.u.x / h.beta, -h.u.y / h.beta);
        }
      }
    }
  }
  __syncthreads();
  if constexpr (SMALL) {
    // V to xb (32 rows) and T to Ts, both in shared memory
    if (warp == 0) t_column(jb - 1);
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int q = warp + UW * j;
      xb[lane + 32 * q] = (lane >= mp || q >= jb || lane < q) ? make_double2(0.0, 0.0)
                                                              : (lane == q ? make_double2(1.0, 0.0) : a[j][0]);
      if (p.R && q < p.n && lane < p.K) p.R[lane + q * p.ldr] = lane <= q ? a[j][0] : make_double2(0.0, 0.0);
    }
    __syncthreads();
  } else {
    cplx* Vg = p.V + (long long)pn * p.m * NB;
    if (warp == 0) {
      t_column(jb - 1);
      __syncwarp();
      cplx* Tg = p.T + pn * NB * NB;
      for (int t = lane; t < NB * NB; t += 32) Tg[t] = Ts[(t % NB) + (t / NB) * T_LD];
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int q = warp + UW * j, col = pn * NB + q;
#pragma unroll
      for (int i = 0; i < RPL; i++) {
        const int r = lane + 32 * i;
        if (r >= mp) continue;
        Vg[j0 + r + (long long)q * p.m] =
            (q >= jb || r < q) ? make_double2(0.0, 0.0) : (r == q ? make_double2(1.0, 0.0) : a[j][i]);
        if (p.R && col < p.n && j0 + r < p.K)
          p.R[j0 + r + col * p.ldr] = (q >= jb || r <= q) ? a[j][i] : make_double2(0.0, 0.0);
      }
      if (p.R && col < p.n)
        for (int r = lane; r < j0; r += 32) p.R[r + col * p.ldr] = As[r + q * p.ld];
    }
  }
}

// C <- (I - V T' V^H) C for panel pn, T' = T^H (conjT: the factorisation's
// H^H) or T (forming Q), on the columns 8 tile0 .. 15 of the slice C (ld).
// Row groups of 16 are numbered from row 0, so a warp owns the same rows in
// every call and no barrier separates two calls.
__device__ void qc_apply(const QcParams& p, cplx* C, int pn, bool conjT, int tile0, cplx* red, cplx* Ts, cplx* W,
                         cplx* W2) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m = p.m, ld = p.ld, fr = lane >> 2, fc = lane & 3;
  const cplx* V = p.V + (long long)pn * m * NB;
  Ts[(tid % NB) + (tid / NB) * T_LD] = __ldcg(&p.T[pn * NB * NB + tid]);
  const int ngrp = (m + NB - 1) / NB;
  const int g0 = warp + (pn > warp ? (pn - warp + UW - 1) / UW * UW : 0);  // the warp's first group from row 16 pn on
  cplx vu[2][4];  // fragments of V for the update (rows x reflectors) of group g0
  double wr[2][2][2], wi[2][2][2];  // W tile (reflectors, columns)
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 2; j++) wr[i][j][0] = wr[i][j][1] = wi[i][j][0] = wi[i][j][1] = 0.0;
  for (int g = g0; g < ngrp; g += UW) {
    cplx v[4][2];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int r = g * NB + 4 * k + fc;
#pragma unroll
      for (int i = 0; i < 2; i++)
        v[k][i] = r < m ? __ldcg(&V[r + (long long)(8 * i + fr) * m]) : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int r = g * NB + 4 * k + fc;
#pragma unroll
      for (int j = 0; j < 2; j++) {
        if (j < tile0) continue;
        const cplx c = r < m ? C[r + (8 * j + fr) * ld] : make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < 2; i++) {  // conj(V)^T C
          dmma(wr[i][j][0], wr[i][j][1], v[k][i].x, c.x);
          dmma(wi[i][j][0], wi[i][j][1], v[k][i].x, c.y);
          dmma(wr[i][j][0], wr[i][j][1], v[k][i].y, c.y);
          dmma(wi[i][j][0], wi[i][j][1], -v[k][i].y, c.x);
        }
      }
    }
  }
  // in flight while the partial sums are added
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int r = g0 * NB + 8 * i + fr;
      vu[i][k] = r < m ? __ldcg(&V[r + (long long)(4 * k + fc) * m]) : make_double2(0.0, 0.0);
    }
  cplx* mine = red + warp * RED_SZ;
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int h = 0; h < 2; h++)
        if (j >= tile0) mine[8 * i + fr + (8 * j + 2 * fc + h) * RED_LD] = make_double2(wr[i][j][h], wi[i][j][h]);
  __syncthreads();
  const int el = tid & 15, eq = tid >> 4;  // one entry (el, eq) of W each
  const bool live = eq >= 8 * tile0;       // uniform over a warp
  if (live) {
    cplx s = make_double2(0.0, 0.0);
#pragma unroll
    for (int w = 0; w < UW; w++) s = cadd(s, red[w * RED_SZ + el + eq * RED_LD]);
    W[tid] = s;
  }
  __syncthreads();
  if (live) {
    cplx s[4];
#pragma unroll
    for (int l = 0; l < 4; l++) s[l] = make_double2(0.0, 0.0);
#pragma unroll
    for (int l = 0; l < NB; l++) {  // T is zero below its diagonal
      if (conjT) ccfma(s[l & 3], Ts[l + el * T_LD], W[l + NB * eq]);
      else cfma(s[l & 3], Ts[el + l * T_LD], W[l + NB * eq]);
    }
    W2[el + W2_LD * eq] = cadd(cadd(s[0], s[1]), cadd(s[2], s[3]));
  }
  __syncthreads();
  for (int g = g0; g < ngrp; g += UW) {
    if (g != g0) {
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int r = g * NB + 8 * i + fr;
          vu[i][k] = r < m ? __ldcg(&V[r + (long long)(4 * k + fc) * m]) : make_double2(0.0, 0.0);
        }
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
      if (j < tile0) continue;
      cplx acc[2][2];
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int r = g * NB + 8 * i + fr;
          acc[i][h] = r < m ? C[r + (8 * j + 2 * fc + h) * ld] : make_double2(0.0, 0.0);
        }
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const cplx w = W2[4 * k + fc + (8 * j + fr) * W2_LD];
#pragma unroll
        for (int i = 0; i < 2; i++) {
          dmma(acc[i][0].x, acc[i][1].x, -vu[i][k].x, w.x);
          dmma(acc[i][0].y, acc[i][1].y, -vu[i][k].x, w.y);
          dmma(acc[i][0].x, acc[i][1].x, vu[i][k].y, w.y);
          dmma(acc[i][0].y, acc[i][1].y, -vu[i][k].y, w.x);
        }
      }
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int r = g * NB + 8 * i + fr;
          if (r < m) C[r + (8 * j + 2 * fc + h) * ld] = acc[i][h];
        }
    }
  }
}

// Global column of local column j of CTA `rank` when Q is formed: pairs of
// columns dealt cyclically.
__device__ __forceinline__ int q_column(int j, int S, int rank) { return 2 * ((j >> 1) * S + rank) + (j & 1); }

template <int RPL>
__global__ void __launch_bounds__(QT, 1) qr_cluster_kernel(const __grid_constant__ QcParams p) {
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char qc_smem[];
  __shared__ Reflector reflector;
  const int rank = (int)cl.block_rank(), tid = threadIdx.x;
  const int m = p.m, ld = p.ld;
  cplx* C = reinterpret_cast<cplx*>(qc_smem);  // the slice: 16 columns, ld apart
  cplx* red = C + NB * ld;                     // partial W of the warps; the pivot columns of a panel
  cplx* Ts = red + UW * RED_SZ;
  cplx* W2 = Ts + NB * T_LD;
  cplx* W = W2 + NB * W2_LD;
  cplx* G = W + NB * NB;
  cplx* taus = G + NB * NB;
  for (int t = tid; t < m * NB; t += QT) {
    const int r = p.a_colfast ? t / NB : t % m, c = p.a_colfast ? t % NB : t / m;
    const int j = rank * NB + c;
    cplx v = make_double2(0.0, 0.0);
    if (j < p.n) {
      v = p.A[view_at(p.va, r, j)];
      if (p.va.conj) v.y = -v.y;
    }
    C[r + c * ld] = v;
  }
  __syncthreads();
  for (int pn = 0; pn < p.np; pn++) {
    const int j0 = pn * NB;
    if (rank == pn) qc_panel<RPL, false>(p, C, pn, j0, min(NB, p.K - j0), red, Ts, G, taus, taus + NB, &reflector);
    cl.sync();  // V and T of panel pn published; the first one also ends every read of A
    if (rank > pn) qc_apply(p, C, pn, true, 0, red, Ts, W, W2);
  }
  if (p.R && rank >= p.np) {
    __syncthreads();
    for (int t = tid; t < p.K * NB; t += QT) {
      const int r = t % p.K, j = rank * NB + t / p.K;
      if (j < p.n) p.R[r + j * p.ldr] = C[r + (t / p.K) * ld];
    }
  }
  if (!p.Q) return;
  // Q = H_0 H_1 ... applied to unit columns, last panel first
  __syncthreads();
  for (int t = tid; t < m * NB; t += QT) {
    const int r = t % m, c = t / m;
    C[r + c * ld] = make_double2(r == q_column(c, p.S, rank) ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  for (int pn = p.np - 1; pn >= 0; pn--) {
    // H_pn reaches the columns from 16 pn on
    const int tile0 = q_column(7, p.S, rank) >= pn * NB ? 0 : 1;
    if (q_column(15, p.S, rank) >= pn * NB) qc_apply(p, C, pn, false, tile0, red, Ts, W, W2);
  }
  __syncthreads();
  for (int t = tid; t < m * NB; t += QT) {
    const int r = p.q_colfast ? t / NB : t % m, c = p.q_colfast ? t % NB : t / m;
    const int j = q_column(c, p.S, rank);
    if (j < p.K) {
      cplx v = C[r + c * ld];
      if (p.vq.conj) v.y = -v.y;
      p.Q[view_at(p.vq, r, j)] = v;
    }
  }
}

// One panel of at most 32 rows (sites of bond dimension up to 16, and the ends
// of every chain): one CTA, a row per lane, Q = E - V (T V^H E) entry by entry
// from shared memory (a block application costs 3 us at this size, its two L2
// round trips among them).  Sums, divisions and products are taken one by one
// in the order of the unblocked algorithm, so that the leading digits of
// 1 - lambda of nearly product states do not depend on the size class.
__global__ void __launch_bounds__(QT) qr_small_kernel(const __grid_constant__ QcParams p) {
  __shared__ cplx C[NB * 33], Ts[NB * T_LD], G[NB * NB], taus[2 * NB], V[2 * MAX_ROWS], W2[NB * W2_LD];
  __shared__ Reflector reflector;
  const int tid = threadIdx.x, m = p.m;
  join_stream();
  for (int t = tid; t < m * NB; t += QT) {
    const int r = p.a_colfast ? t / NB : t % m, c = p.a_colfast ? t % NB : t / m;
    cplx v = make_double2(0.0, 0.0);
    if (c < p.n) {
      v = p.A[view_at(p.va, r, c)];
      if (p.va.conj) v.y = -v.y;
    }
    C[r + c * p.ld] = v;
  }
  qc_panel<1, true>(p, C, 0, 0, p.K, V, Ts, G, taus, taus + NB, &reflector);
  if (!p.Q) return;
  {
    const int i = tid & 15, q = tid >> 4;
    cplx s = make_double2(0.0, 0.0);
    for (int l = i; l < p.K; l++) s = cadd(s, cmul(Ts[i + T_LD * l], cconj(V[q + 32 * l])));
    W2[i + W2_LD * q] = s;
  }
  __syncthreads();
  for (int t = tid; t < m * NB; t += QT) {
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
// rows per lane of the panel: the smallest that holds m rows
QcKernel qc_kernel(int m) {
  return m <= 64 ? qr_cluster_kernel<2> : m <= 128 ? qr_cluster_kernel<4> : m <= 256 ? qr_cluster_kernel<8>
                                                                                    : qr_cluster_kernel<16>;
}

std::atomic<unsigned long long> g_qc_setup{0};
std::atomic<int> g_qc_slices[64];  // largest cluster the device can place with the largest plan

void qc_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int S, int m, cudaStream_t s) {
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(S);
  cfg.blockDim = dim3(QT);
  cfg.dynamicSmemBytes = qc_smem_elems(qc_ld(m)) * sizeof(cplx);
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
}

int qc_max_slices() {
  int dev = 0;
  MPSGPU_CUDA(cudaGetDevice(&dev));
  if (dev >= 64) return 0;
  if (device_needs_setup(g_qc_setup)) {
    int best = 0;
    for (int m : {64, 128, 256, 512}) {
      MPSGPU_CUDA(cudaFuncSetAttribute(qc_kernel(m), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(qc_smem_elems(qc_ld(m)) * sizeof(cplx))));
      // clusters above 8 CTAs are an opt-in
      MPSGPU_CUDA(cudaFuncSetAttribute(qc_kernel(m), cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    }
    for (int S : {8, MAX_SLICES}) {
      cudaLaunchConfig_t cfg;
      cudaLaunchAttribute attr[1];
      qc_config(cfg, attr, S, MAX_ROWS, nullptr);
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, qc_kernel(MAX_ROWS), &cfg) == cudaSuccess && clusters > 0) best = S;
      (void)cudaGetLastError();
    }
    g_qc_slices[dev].store(best);
    mark_device_done(g_qc_setup);
  }
  return g_qc_slices[dev].load();
}

}  // namespace

// Up to 512 rows and 256 columns, while the device can place a cluster of
// ceil(n/16) CTAs (the limits of the shared-memory plan).
bool cluster_qr_fits(int m, int n) {
  return (m <= 32 && n <= NB) || (m <= MAX_ROWS && ceil_div(n, NB) <= qc_max_slices());
}

void cluster_qr(const Stream& st, int m, int n, const cplx* A, const View2& va, cplx* Q, const View2& vq, cplx* R,
                long long ldr, Scratch& scratch) {
  QcParams p;
  p.m = m; p.n = n; p.K = std::min(m, n);
  p.npa = ceil_div(n, NB);
  p.np = ceil_div(p.K, NB);
  p.S = p.npa;
  p.ld = qc_ld(m);
  p.A = A; p.va = va;
  p.Q = Q; p.vq = vq;
  p.R = R; p.ldr = ldr;
  p.a_colfast = va.cd == 1 && va.c1 == 1;
  p.q_colfast = vq.cd == 1 && vq.c1 == 1;
  // factorisation and explicit Q, complex flops (8 per complex MAC)
  ProfScope ps(st, GemmProfiler::QR, qr_flops(m, n));
  if (m <= 32 && n <= NB) {
    launch_chained(st, qr_small_kernel, 1, QT, 0, p);
    return;
  }
  p.V = (cplx*)scratch.get(((size_t)p.np * m * NB + (size_t)p.np * NB * NB) * sizeof(cplx));
  p.T = p.V + (size_t)p.np * m * NB;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  qc_config(cfg, attr, p.S, m, st.s);
  MPSGPU_CUDA(cudaLaunchKernelEx(&cfg, qc_kernel(m), p));
  after_launch(st);
}

}  // namespace mpsgpu
