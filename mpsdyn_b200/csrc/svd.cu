// Singular values of a small complex matrix by one-sided Jacobi (Hestenes
// 1958; the complex form of Demmel & Veselic 1992): the columns of A are
// rotated pairwise until every pair is orthogonal to working precision;
// the singular values are then the column norms.
//
// Work split (block Jacobi): the columns form blocks of 8, a CTA works on two
// blocks at a time in shared memory, one warp per pair of columns, and a
// round-robin over the blocks brings every two together once a sweep; the CTAs
// exchange blocks through global memory (L2) with one barrier per round, of a
// thread-block cluster up to 256 columns and of the grid beyond.  A rotation is
// a serial chain of a warp reduction and four square roots and reciprocals, so a
// sweep is bound by the latency of its n - 1 steps; eight warps per SM keep the
// FP64 issue rate of the redundant scalars (one warp instruction per two
// cycles) out of that chain.  A matrix of at most 16 columns stays in one CTA.
// Measured: 128 x 128 values in 1.85 ms, 256 x 256 in 3.9 ms, 64 x 64 with
// vectors in 0.82 ms (13 sweeps); one CTA of 32 warps on the matrix in L2 took
// 10.2, 64.9 and 1.45-2.0 ms.
//
// Used for the Schmidt values / entanglement entropy of a bond
// (Contractor::getSchmidtValues / getEntropy, Contractor.cpp:2045-2076 and
// :2243-2270: there the eigenvalues of the reduced density matrix; here the
// squares of the singular values of the bond matrix, which are the same
// numbers and carry full relative accuracy for the small ones, as long as the
// products of two columns stay above 1e-162), and for the cut SVDs of MPO
// application and two-site sweeps.
#include <cooperative_groups.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace mpsgpu {

namespace {

// Matrices of 64 to 256 columns whose columns fall off over 60 to 140 orders without
// being sorted take 40 to 66 sweeps here; ordinary ones 10, after a quench 2 to 11.
constexpr int MAX_SWEEPS = 100;
constexpr int MAX_COLS = 1024;
constexpr int NBJ = 8;               // columns of a block; pairs (warps) of a CTA
constexpr int JT = 32 * NBJ;
constexpr double JTOL = 1e-15;       // |a_p^H a_q| <= JTOL |a_p| |a_q|: orthogonal
enum { JSYNC_NONE = 0, JSYNC_CLUSTER = 1, JSYNC_GRID = 2 };

__device__ __forceinline__ double warp_sumd(double s) {
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

__device__ __forceinline__ cplx warp_sum(cplx v) {
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}

// The sums of (a, b) and c over the lanes of a warp, in every lane: the first
// two exchanges halve what a lane carries.
__device__ __forceinline__ void warp_sum4(double& a, double& b, cplx& c) {
  const int lane = threadIdx.x & 31;
  const bool h = lane & 16, q = lane & 8;
  double kx = h ? c.x : a, ky = h ? c.y : b;
  kx += __shfl_xor_sync(0xffffffffu, h ? a : c.x, 16);
  ky += __shfl_xor_sync(0xffffffffu, h ? b : c.y, 16);
  double v = q ? ky : kx;
  v += __shfl_xor_sync(0xffffffffu, q ? kx : ky, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  a = __shfl_sync(0xffffffffu, v, 0);
  b = __shfl_sync(0xffffffffu, v, 8);
  c = make_double2(__shfl_sync(0xffffffffu, v, 16), __shfl_sync(0xffffffffu, v, 24));
}

// (x, y) <- rotation of the columns ap, aq of `rows` rows by one warp:
// x' = cs x - sn (y ph), y' = sn x + cs (y ph)
__device__ __forceinline__ void rotate_phase(cplx* ap, cplx* aq, int rows, double cs, double sn, cplx ph) {
  for (int r = threadIdx.x & 31; r < rows; r += 32) {
    const cplx x = ap[r];
    const cplx y = cmul(aq[r], ph);
    ap[r] = make_double2(cs * x.x - sn * y.x, cs * x.y - sn * y.y);
    aq[r] = make_double2(sn * x.x + cs * y.x, sn * x.y + cs * y.y);
  }
}
// x' = cs x - s y, y' = conj(s) x + cs y (the same without the phase on y')
__device__ __forceinline__ void rotate_plain(cplx* ap, cplx* aq, int rows, double cs, cplx s) {
#pragma unroll 4
  for (int r = threadIdx.x & 31; r < rows; r += 32) {
    const cplx x = ap[r], y = aq[r];
    ap[r] = make_double2(fma(cs, x.x, fma(-s.x, y.x, s.y * y.y)), fma(cs, x.y, -fma(s.x, y.y, s.y * y.x)));
    aq[r] = make_double2(fma(cs, y.x, fma(s.x, x.x, s.y * x.y)), fma(cs, y.y, fma(s.x, x.y, -(s.y * x.x))));
  }
}

// One warp orthogonalises the columns ap, aq (m rows) and applies the rotation
// to vp, vq (mv rows); true when it rotated.
template <bool SMALL>
__device__ __forceinline__ bool jacobi_pair(cplx* ap, cplx* aq, int m, cplx* vp, cplx* vq, int mv) {
  const int lane = threadIdx.x & 31;
  double al = 0.0, be = 0.0;
  cplx ga = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int r = lane; r < m; r += 32) {
    const cplx x = ap[r], y = aq[r];
    al += cabs2(x);
    be += cabs2(y);
    ga = cadd(ga, ccmul(x, y));
  }
  if constexpr (SMALL) {
    al = warp_sumd(al);
    be = warp_sumd(be);
    ga = warp_sum(ga);
  } else {
    warp_sum4(al, be, ga);
    // in the range where the squares below are representable
    if (al > 1e-140 && be > 1e-140 && al < 1e140 && be < 1e140) {
      const double g2 = cabs2(ga);
      if (!(g2 > JTOL * JTOL * al * be)) return false;
      // tan 2 theta = 2 |gamma| / (beta - alpha): cs^2 = (1 + |beta - alpha| / h) / 2,
      // sn = |gamma| / (h cs) with h^2 = (beta - alpha)^2 + 4 |gamma|^2
      const double dl = be - al, r = 1.0 / sqrt(fma(dl, dl, 4.0 * g2));
      const double cs = sqrt(fma(0.5 * fabs(dl), r, 0.5)), f = copysign(r / cs, dl);
      const cplx s = make_double2(f * ga.x, -f * ga.y);
      rotate_plain(ap, aq, m, cs, s);
      rotate_plain(vp, vq, mv, cs, s);
      return true;
    }
  }
  const double ab = al * be;
  const double g2 = cabs2(ga);
  double g = sqrt(g2);
  if (g2 < 2.3e-308) {
    // below the normal range from the product times 2^200: the root of the square
    // itself, and with it the modulus of the phase below, is off by up to 40 %, and
    // the column it multiplies may be a large one (a second value of 1.7e-6 beside
    // columns of 1e-150 came out 20 % off).  Where the square vanishes the pair is
    // left alone: values below 1e-81, which no one asks for beside larger ones, would
    // take up to 30 sweeps more.
    if (!(g2 > 0.0)) return false;
    g = sqrt(cabs2(cscale(ga, 0x1p200))) * 0x1p-200;
  }
  // (ab underflows for two columns of 1e-80, each square does not)
  if (!(g > JTOL * (ab > 1e-280 ? sqrt(ab) : sqrt(al) * sqrt(be)))) return false;
  // rotate (a_p, a_q conj(phase)) so that the pair becomes orthogonal
  const double zeta = (be - al) / (2.0 * g);
  const double t = (zeta >= 0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
  // no rotation (zeta^2 overflows: the smaller column is below 1e-154 of the
  // larger, as what is left of parallel columns gets after some sweeps); counted
  // as one it kept the sweeps from ending
  if (t == 0.0) return false;
  const double cs = 1.0 / sqrt(1.0 + t * t), sn = cs * t;
  const cplx ph = make_double2(ga.x / g, -ga.y / g);  // conj(gamma)/|gamma|
  rotate_phase(ap, aq, m, cs, sn, ph);
  rotate_phase(vp, vq, mv, cs, sn, ph);
  return true;
}

// Slot k of a round-robin (circle) ordering of n items (even) in step `step`:
// slot k pairs with slot n - 1 - k; slot 0 holds item 0.
__device__ __forceinline__ int circle_item(int k, int step, int n) {
  return k == 0 ? 0 : ((k - 1 - step) % (n - 1) + (n - 1)) % (n - 1) + 1;
}

// A: m x n (n even; n a multiple of 16 with more than one CTA), column-major,
// ld m, rotated in place.  V (n x n, ld n, identity on entry) accumulates the
// rotations when non-null, so that A_in V = A_out.  out: n column norms;
// status[0] = sweeps used (MAX_SWEEPS + 1 if not converged), with more than one
// CTA status[1 + s] zero on entry (rotations left in sweep s).  gridDim.x = n / 16 CTAs (at least 1).
// SMALL (one CTA): sums, tests and rotations in the order and form of the
// unblocked algorithm.
template <bool SMALL, int SYNC>
__global__ void __launch_bounds__(JT) jacobi_sv_kernel(int m, int n, cplx* A, cplx* V, double* out, int* status) {
  extern __shared__ __align__(16) unsigned char jsm[];
  __shared__ int rotated;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int mv = V ? n : 0, ncol = min(n, 2 * NBJ), nblk = n / NBJ, cta = blockIdx.x;
  cplx* As = reinterpret_cast<cplx*>(jsm);
  cplx* Vs = As + (size_t)ncol * m;
  auto everyone = [&]() {
    if constexpr (SYNC == JSYNC_CLUSTER) cg::this_cluster().sync();
    else if constexpr (SYNC == JSYNC_GRID) cg::this_grid().sync();
    else __syncthreads();
  };
  // columns of the CTA's two blocks between global and shared memory
  auto columns = [&](int b0, int b1, bool load) {
    for (int c = warp; c < ncol; c += NBJ) {
      const long long col = SYNC == JSYNC_NONE ? c : (c < NBJ ? b0 : b1) * NBJ + (c & (NBJ - 1));
      cplx* ga = A + col * m;
      cplx* gv = V + (V ? col * n : 0);
      if (load) {
#pragma unroll 4
        for (int r = lane; r < m; r += 32) As[(size_t)c * m + r] = __ldcg(&ga[r]);
#pragma unroll 4
        for (int r = lane; r < mv; r += 32) Vs[(size_t)c * mv + r] = __ldcg(&gv[r]);
      } else {
#pragma unroll 4
        for (int r = lane; r < m; r += 32) ga[r] = As[(size_t)c * m + r];
#pragma unroll 4
        for (int r = lane; r < mv; r += 32) gv[r] = Vs[(size_t)c * mv + r];
      }
    }
  };
  auto pair = [&](int p, int q) {
    return jacobi_pair<SMALL>(As + (size_t)p * m, As + (size_t)q * m, m, Vs + (size_t)p * mv, Vs + (size_t)q * mv, mv);
  };
  if (SYNC == JSYNC_NONE) columns(0, 0, true);
  const int rounds = SYNC == JSYNC_NONE ? 1 : nblk - 1;
  int sweep = 0;
  bool any = false;
  for (; sweep < MAX_SWEEPS; sweep++) {
    for (int rd = 0; rd < rounds; rd++) {
      int b0 = 0, b1 = 0;
      if (SYNC != JSYNC_NONE) {
        b0 = circle_item(cta, rd, nblk);
        b1 = circle_item(nblk - 1 - cta, rd, nblk);
        columns(b0, b1, true);
      }
      if (tid == 0) rotated = 0;
      __syncthreads();
      if (rd == 0) {  // every pair of the two blocks, within them too
        for (int step = 0; step < ncol - 1; step++) {
          if (warp < ncol / 2 && pair(circle_item(warp, step, ncol), circle_item(ncol - 1 - warp, step, ncol)) &&
              lane == 0)
            rotated = 1;
          __syncthreads();
        }
      } else {  // the pairs across
        for (int step = 0; step < NBJ; step++) {
          if (pair(warp, NBJ + ((warp + step) & (NBJ - 1))) && lane == 0) rotated = 1;
          __syncthreads();
        }
      }
      any = rotated;  // written before the last barrier
      if (SYNC != JSYNC_NONE && any) {
        columns(b0, b1, false);
        if (tid == 0) atomicOr(&status[1 + sweep], 1);
      }
      everyone();
    }
    if (SYNC == JSYNC_NONE ? !any : __ldcg(&status[1 + sweep]) == 0) break;
  }
  if (SYNC == JSYNC_NONE) {
    columns(0, 0, false);
    __syncthreads();
  }
  // column norms with the largest magnitude factored out, so that singular
  // values below 1e-154 (squares below the FP64 normal range) keep their
  // relative accuracy
  for (int col = cta * NBJ + warp; col < n; col += gridDim.x * NBJ) {
    const cplx* a = A + (long long)col * m;
    double mx = 0.0;
    for (int r = lane; r < m; r += 32) {
      const cplx x = __ldcg(&a[r]);
      mx = fmax(mx, fmax(fabs(x.x), fabs(x.y)));
    }
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    double s = 0.0;
    if (mx > 0.0) {
      const double inv = 1.0 / mx;
      for (int r = lane; r < m; r += 32) {
        const cplx x = __ldcg(&a[r]);
        const double u = x.x * inv, v = x.y * inv;
        s += u * u + v * v;
      }
    }
    s = warp_sumd(s);
    if (lane == 0) out[col] = mx * sqrt(s);
  }
  if (cta == 0 && tid == 0) status[0] = sweep < MAX_SWEEPS ? sweep + 1 : MAX_SWEEPS + 1;
}

// The same for columns too long for two blocks in shared memory: one CTA of
// 1024 threads on the matrix in global memory, one warp per pair of a
// round-robin over the columns.
constexpr int JLT = 1024;
__global__ void __launch_bounds__(JLT) jacobi_long_kernel(int m, int n, cplx* A, cplx* V, double* out, int* status) {
  __shared__ int rotated;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = JLT / 32;
  const int mv = V ? n : 0;
  int sweep = 0;
  for (; sweep < MAX_SWEEPS; sweep++) {
    if (threadIdx.x == 0) rotated = 0;
    __syncthreads();
    for (int step = 0; step < n - 1; step++) {
      for (int pr = warp; pr < n / 2; pr += nw) {
        const long long p = circle_item(pr, step, n), q = circle_item(n - 1 - pr, step, n);
        if (jacobi_pair<true>(A + p * m, A + q * m, m, V + p * mv, V + q * mv, mv) && lane == 0) rotated = 1;
      }
      __syncthreads();
    }
    const bool more = rotated;
    __syncthreads();
    if (!more) break;
  }
  for (int col = warp; col < n; col += nw) {
    const cplx* a = A + (long long)col * m;
    double mx = 0.0;
    for (int r = lane; r < m; r += 32) mx = fmax(mx, fmax(fabs(a[r].x), fabs(a[r].y)));
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    double s = 0.0;
    if (mx > 0.0) {
      const double inv = 1.0 / mx;
      for (int r = lane; r < m; r += 32) {
        const double u = a[r].x * inv, v = a[r].y * inv;
        s += u * u + v * v;
      }
    }
    s = warp_sumd(s);
    if (lane == 0) out[col] = mx * sqrt(s);
  }
  if (threadIdx.x == 0) status[0] = sweep < MAX_SWEEPS ? sweep + 1 : MAX_SWEEPS + 1;
}

constexpr size_t JSMEM = 224 * 1024;
size_t jacobi_smem(int rows, int colsp, bool vectors) {
  return (size_t)std::min(colsp, 2 * NBJ) * (rows + (vectors ? colsp : 0)) * sizeof(cplx);
}
// Columns of the padded matrix: even for one CTA, whole pairs of blocks for more.
int jacobi_cols(int cols) { return cols <= 2 * NBJ ? cols + (cols & 1) : ceil_div(cols, 2 * NBJ) * 2 * NBJ; }
constexpr size_t JSTATUS = (MAX_SWEEPS + 2) * sizeof(int);

std::atomic<unsigned long long> g_jac_setup{0};
std::atomic<int> g_jac_cluster[64];  // largest cluster placed with the largest plan

void jacobi_launch(const Stream& st, int rows, int colsp, cplx* W, cplx* V, double* d_sig, int* d_status) {
  const size_t smem = jacobi_smem(rows, colsp, V != nullptr);
  const int ctas = std::max(1, colsp / (2 * NBJ));
  int dev = 0;
  MPSGPU_CUDA(cudaGetDevice(&dev));
  MPSGPU_CHECK(dev < 64, MPSGPU_INVALID, "svd: device number");
  auto small = jacobi_sv_kernel<true, JSYNC_NONE>;
  auto one = jacobi_sv_kernel<false, JSYNC_CLUSTER>;
  auto grid = jacobi_sv_kernel<false, JSYNC_GRID>;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  auto config = [&](int c, size_t bytes) {
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(JT);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st.s;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
  };
  if (device_needs_setup(g_jac_setup)) {
    MPSGPU_CUDA(cudaFuncSetAttribute(small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)JSMEM));
    MPSGPU_CUDA(cudaFuncSetAttribute(one, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)JSMEM));
    MPSGPU_CUDA(cudaFuncSetAttribute(grid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)JSMEM));
    MPSGPU_CUDA(cudaFuncSetAttribute(one, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    int best = 0;
    for (int c : {8, 16}) {
      config(c, JSMEM);
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, one, &cfg) == cudaSuccess && clusters > 0) best = c;
      (void)cudaGetLastError();
    }
    g_jac_cluster[dev].store(best);
    mark_device_done(g_jac_setup);
  }
  const bool longc = smem > JSMEM, one_cta = longc || colsp <= 2 * NBJ;
  // (one CTA keeps its flag in shared memory)
  if (!one_cta) MPSGPU_CUDA(cudaMemsetAsync(d_status, 0, JSTATUS, st.s));
  if (longc) {
    jacobi_long_kernel<<<1, JLT, 0, st.s>>>(rows, colsp, W, V, d_sig, d_status);
  } else if (colsp <= 2 * NBJ) {
    small<<<1, JT, smem, st.s>>>(rows, colsp, W, V, d_sig, d_status);
  } else if (ctas <= g_jac_cluster[dev].load()) {
    config(ctas, smem);
    MPSGPU_CUDA(cudaLaunchKernelEx(&cfg, one, rows, colsp, W, V, d_sig, d_status));
  } else {
    void* args[] = {&rows, &colsp, &W, &V, &d_sig, &d_status};
    MPSGPU_CUDA(cudaLaunchCooperativeKernel((void*)grid, dim3(ctas), dim3(JT), args, smem, st.s));
  }
  after_launch(st);
}

}  // namespace

// Singular values (descending) of the m x n matrix at A (device, ld m);
// A is not modified.  Host-synchronous (returns the values on the host).
std::vector<double> singular_values(const Stream& st, int m, int n, const cplx* A, long long lda,
                                    Scratch& scratch, bool by_rows) {
  MPSGPU_CHECK(m > 0 && n > 0, MPSGPU_BAD_SHAPE, "singular_values: empty matrix");
  // work on the orientation with at most as many columns as rows
  const bool tr = n > m || (by_rows && n == m);
  const int rows = tr ? n : m;
  int cols = tr ? m : n;
  const int colsp = jacobi_cols(cols);  // zero columns added
  MPSGPU_CHECK(cols + (cols & 1) <= MAX_COLS && rows <= 8192, MPSGPU_BAD_SHAPE, "singular_values: matrix too large");
  char* ws = (char*)scratch.get((size_t)rows * colsp * sizeof(cplx) + colsp * sizeof(double) + JSTATUS + 64);
  cplx* W = (cplx*)ws;
  double* d_out = (double*)(ws + (size_t)rows * colsp * sizeof(cplx));
  int* d_status = (int*)(d_out + colsp);
  View2 v;
  if (!tr) { v.rd = 1; v.r0 = 0; v.r1 = 1; v.cd = 1; v.c0 = 0; v.c1 = lda; }
  else { v.rd = 1; v.r0 = 0; v.r1 = lda; v.cd = 1; v.c0 = 0; v.c1 = 1; v.conj = true; }
  if (colsp > cols) zfill(st, (long long)rows * (colsp - cols), make_double2(0.0, 0.0), W + (size_t)rows * cols);
  gather2(st, rows, cols, A, v, W);
  jacobi_launch(st, rows, colsp, W, nullptr, d_out, d_status);
  std::vector<double> sv(colsp);
  int status = 0;
  MPSGPU_CUDA(cudaMemcpyAsync(sv.data(), d_out, colsp * sizeof(double), cudaMemcpyDeviceToHost, st.s));
  MPSGPU_CUDA(cudaMemcpyAsync(&status, d_status, sizeof(int), cudaMemcpyDeviceToHost, st.s));
  MPSGPU_CUDA(cudaStreamSynchronize(st.s));
  MPSGPU_CHECK(status <= MAX_SWEEPS, MPSGPU_NOT_CONVERGED, "singular_values: Jacobi did not converge");
  std::sort(sv.begin(), sv.end(), std::greater<double>());
  sv.resize(std::min(m, n));
  return sv;
}

namespace {

// Kept singular triplets in descending order (idx[j] = Jacobi column of the
// j-th largest value).  Not transposed (m >= n, W = A V): U[:, j] =
// W[:, idx_j] / s_j, SVh[j, :] = s_j V[:, idx_j]^H.  Transposed (W = A^H V'):
// A = V' S U'^H, so U[:, j] = V'[:, idx_j] and SVh[j, :] = W[:, idx_j]^H.
// left_s moves diag(s) to the left factor: U diag(s) and V^H.
__global__ void svd_finish_kernel(int m, int n, int rows, int cols, bool tr, const cplx* __restrict__ W,
                                  const cplx* __restrict__ V, const int* __restrict__ idx,
                                  const double* __restrict__ sig, int keep, bool left_s, cplx* __restrict__ U,
                                  cplx* __restrict__ SVh) {
  const long long totU = (long long)m * keep, totS = (long long)keep * n;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < totU + totS;
       t += (long long)gridDim.x * blockDim.x) {
    if (t < totU) {
      const int i = (int)(t % m), j = (int)(t / m);
      const int c = idx[j];
      cplx u = tr ? V[i + (long long)c * cols] : cscale(W[i + (long long)c * rows], 1.0 / sig[c]);
      if (left_s) u = cscale(u, sig[c]);
      U[t] = u;
    } else {
      const long long q = t - totU;
      const int j = (int)(q % keep), k = (int)(q / keep);
      const int c = idx[j];
      cplx x = tr ? W[k + (long long)c * rows] : cscale(V[k + (long long)c * cols], sig[c]);
      if (left_s) x = cscale(x, 1.0 / sig[c]);
      SVh[j + (long long)k * keep] = make_double2(x.x, -x.y);
    }
  }
}

__global__ void identity_kernel(int n, cplx* __restrict__ V) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)n * n;
       t += (long long)gridDim.x * blockDim.x)
    V[t] = make_double2((t % n) == (t / n) ? 1.0 : 0.0, 0.0);
}

}  // namespace

// Thin SVD with the cut of wrapper::svd(A, tol = 0, Xi = cut) (svd.cpp:23-118):
// keep = min(cut, min(m, n)) (cut <= 0: all), then only the values > 0 among
// those.  A (m x n, ld m) is not modified.  Writes U (m x keep, ld m) and
// diag(s) V^H (keep x n, ld keep) -- or, with left_s, U diag(s) and V^H;
// sv gets all min(m, n) values descending.
int svd_cut(const Stream& st, int m, int n, const cplx* A, long long lda, int cut, cplx* U, cplx* SVh,
            std::vector<double>& sv, Scratch& scratch, bool left_s) {
  MPSGPU_CHECK(m > 0 && n > 0, MPSGPU_BAD_SHAPE, "svd: empty matrix");
  const bool tr = n > m;
  const int rows = tr ? n : m;
  const int cols = tr ? m : n;
  const int colsp = jacobi_cols(cols);
  MPSGPU_CHECK(cols + (cols & 1) <= MAX_COLS && rows <= 8192, MPSGPU_BAD_SHAPE, "svd: matrix too large");
  const size_t wbytes = (size_t)rows * colsp * sizeof(cplx), vbytes = (size_t)colsp * colsp * sizeof(cplx);
  char* ws = (char*)scratch.get(wbytes + vbytes + colsp * (sizeof(double) + sizeof(int)) + JSTATUS + 256);
  cplx* W = (cplx*)ws;
  cplx* V = (cplx*)(ws + wbytes);
  double* d_sig = (double*)(ws + wbytes + vbytes);
  int* d_idx = (int*)(d_sig + colsp);
  int* d_status = d_idx + colsp;
  View2 v;
  if (!tr) { v.rd = 1; v.r0 = 0; v.r1 = 1; v.cd = 1; v.c0 = 0; v.c1 = lda; }
  else { v.rd = 1; v.r0 = 0; v.r1 = lda; v.cd = 1; v.c0 = 0; v.c1 = 1; v.conj = true; }
  if (colsp > cols) zfill(st, (long long)rows * (colsp - cols), make_double2(0.0, 0.0), W + (size_t)rows * cols);
  gather2(st, rows, cols, A, v, W);
  identity_kernel<<<std::min(ceil_div((long long)colsp * colsp, 256), 1184), 256, 0, st.s>>>(colsp, V);
  after_launch(st);
  jacobi_launch(st, rows, colsp, W, V, d_sig, d_status);
  std::vector<double> all(colsp);
  int status = 0;
  MPSGPU_CUDA(cudaMemcpyAsync(all.data(), d_sig, colsp * sizeof(double), cudaMemcpyDeviceToHost, st.s));
  MPSGPU_CUDA(cudaMemcpyAsync(&status, d_status, sizeof(int), cudaMemcpyDeviceToHost, st.s));
  MPSGPU_CUDA(cudaStreamSynchronize(st.s));
  MPSGPU_CHECK(status <= MAX_SWEEPS, MPSGPU_NOT_CONVERGED, "svd: Jacobi did not converge");
  // descending order over the real columns (the padding column is not a value)
  std::vector<int> idx(cols);
  for (int j = 0; j < cols; j++) idx[j] = j;
  std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return all[a] > all[b]; });
  sv.resize(cols);
  for (int j = 0; j < cols; j++) sv[j] = all[idx[j]];
  int keep = cut > 0 ? std::min(cut, cols) : cols;
  int pos = 0;
  while (pos < keep && sv[pos] > 0.0) pos++;
  keep = pos;
  MPSGPU_CHECK(keep > 0, MPSGPU_BAD_SHAPE, "svd: no singular value above 0");
  MPSGPU_CUDA(cudaMemcpyAsync(d_idx, idx.data(), keep * sizeof(int), cudaMemcpyHostToDevice, st.s));
  const long long tot = (long long)m * keep + (long long)keep * n;
  svd_finish_kernel<<<std::min(ceil_div(tot, 256), 1184), 256, 0, st.s>>>(m, n, rows, colsp, tr, W, V, d_idx,
                                                                           d_sig, keep, left_s, U, SVh);
  after_launch(st);
  // idx is a host vector: wait for its copy before it goes out of scope
  MPSGPU_CUDA(cudaStreamSynchronize(st.s));
  return keep;
}

}  // namespace mpsgpu
