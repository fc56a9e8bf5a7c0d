// fp64_form.cu -- the lambda_t contraction of the FP64 form as a matrix
// product on the FP64 tensor cores (mma.m8n8k4).
//
// With mu_kq = alpha_k + beta_q and centred delta_t, a_k, b_q (as in
// mixed_gemm.cu, here all in FP64)
//   exp(-(l_t - mu_kq)^2 / 2s^2) = F(t,k) G(t,q) H(k,q),
// so S_i(k,q) = H sum_t F(t,k) [u_t K_i(t,q) G(t,q)] needs one exponential
// per (t,k), (t,q) and (k,q) instead of one per (k,q,t): 131 thousand in
// place of 8.4 million a point at 4x nodes, and 34 M multiply-adds that run
// at the part's 37 TFLOP/s.  The factors' exponents carry their rounding errors
// (fp64_factors.cuh), and L0 = A0 + B0 exactly, so that the identity holds to
// the last places of a factor: a cell is within 1.3e-15 of the exact
// sum, the direct sum, which rounds mu, within 9e-15 (s from 0.06 to 0.24).
// FP64's exponent range holds the factors wherever the point passes the prep
// kernel's bounds (kF64MaxExp, kF64MaxRoom), the others keep the direct sum
// (direct_main_kernel).  48 points at 4x nodes: 178 us a call, 1841 us with
// the direct sum.
//
// The points of a call are taken in rounds that fit the workspace (F, G and Y
// of a round stay in L2); f64_factor_kernel writes them, f64_gemm_kernel
// contracts lambda_t and z_t and writes the mass weights W_ij(k).
#include "common.cuh"
#include "engine_internal.h"
#include "fp64_factors.cuh"
#include "host_common.h"
#include "mor_norm.cuh"

namespace y3b {

namespace {

constexpr int kFactorThreads = 256;

// Workspace of one point: F [n_tp][n_mp] | G [n_tp][n_z] | Y [n_m][n_z].
struct F64Ws {
  int n_mp, n_tp;
  size_t g, y;
};

__host__ __device__ inline F64Ws
f64_ws(int n_m, int n_z, int n_t)
{
  F64Ws w;
  w.n_mp = (n_m + kF64Rows - 1) / kF64Rows * kF64Rows;
  w.n_tp = (n_t + kF64Chunk - 1) / kF64Chunk * kF64Chunk;
  w.g = (size_t)w.n_tp * w.n_mp;
  w.y = w.g + (size_t)w.n_tp * n_z;
  return w;
}

// F, G and Y(k, q) = n(M_k, z_q) H(k, q) / (sqrt(2 pi) s D_kq); F and G only on
// the windows' lam_t stages (zero past the last node and row).  Bound by the
// FP64 units: an exponential and some thirty operations for its exponent an
// element, so that what depends on the column alone is formed once a column.
__global__ void __launch_bounds__(kFactorThreads)
f64_factor_kernel(F64Launch L)
{
  const int p = L.p0 + blockIdx.y;
  const PointDev pt = L.pts[p];
  if (!grid_in_mask(L.grid_mask, pt.grid)) return;
  const GridDev* __restrict__ Gp = L.grids + pt.grid;
  const double* __restrict__ s64 = L.s64 + (size_t)p * Gp->s64_stride;
  const double* hdr = s64 + Gp->o_f64;
  if (hdr[0] == 0.0) return;  // direct sum, or left unprepared
  const int n_m = Gp->n_m, n_z = Gp->n_z, n_t = Gp->n_t;
  const F64Ws w = f64_ws(n_m, n_z, n_t);
  double* ws = L.ws + (size_t)blockIdx.y * L.ws_stride;
  const double A0 = hdr[1], B0 = hdr[2], L0 = A0 + B0, inv_s = 1.0 / pt.sigma;
  const Dd c = f64_half_inv_var(pt.sigma);
  const double* alpha = s64 + Gp->o_alpha;
  const double* beta = s64 + Gp->o_beta;
  const int* win = reinterpret_cast<const int*>(hdr + 4);
  const int step = gridDim.x * kFactorThreads, i0 = blockIdx.x * kFactorThreads + threadIdx.x;
  int h_lo = w.n_tp, h_hi = 0;  // hull of the tiles' windows
  for (int m = 0; m < w.n_mp / kF64Rows; ++m) {
    h_lo = min(h_lo, (win[m] & 0xFFFF) * kF64Chunk);
    h_hi = max(h_hi, (win[m] >> 16) * kF64Chunk);
  }
  // A thread keeps its column (k of F, q of G and Y) and takes rows apart by
  // the rows that the threads cover at once.
  int P = min(step, w.n_mp), R = step / P, r0 = i0 / P;
  for (int k = i0 - r0 * P; r0 < R && k < w.n_mp; k += P) {
    const int v = win[k / kF64Rows], t_end = (v >> 16) * kF64Chunk;
    const bool in = k < n_m;
    const Dd a = dd_diff(alpha[in ? k : 0], A0);
    for (int t = (v & 0xFFFF) * kF64Chunk + r0; t < t_end; t += R)
      ws[(size_t)t * w.n_mp + k] =
        in && t < n_t ? f64_F(dd_diff(Gp->xl[t], L0), a, c) : 0.0;
  }
  P = min(step, n_z);
  R = step / P;
  r0 = i0 / P;
  for (int q = i0 - r0 * P; r0 < R && q < n_z; q += P) {
    const Dd b = dd_diff(beta[q], B0);
    for (int t = h_lo + r0; t < h_hi; t += R)
      ws[w.g + (size_t)t * n_z + q] = t < n_t ? f64_G(dd_diff(Gp->xl[t], L0), b, c) : 0.0;
  }
  const double* dn = L.tables + (size_t)(L.slot ? L.slot[p] : p) * L.lay.stride + L.lay.off[2];
  const double norm0 = inv_s / kSqrt2Pi;
  for (int q = i0 - r0 * P; r0 < R && q < n_z; q += P) {
    const Dd b = dd_diff(beta[q], B0);
    const double u = s64[Gp->o_qu + q];
    const double* row = dn + (size_t)s64[Gp->o_qy + q] * L.lay.n_hm;
    for (int k = r0; k < n_m; k += R) {
      const double t = s64[Gp->o_kt + k];
      const double* d0 = row + (int)s64[Gp->o_kx + k];
      const double* d1 = d0 + L.lay.n_hm;
      const double n = ((1.0 - t) * (1.0 - u) * d0[0] + t * (1.0 - u) * d0[1] +
                        (1.0 - t) * u * d1[0] + t * u * d1[1]) *
                       s64[Gp->o_kf + k] * norm0;
      const double mu = alpha[k] + beta[q];
      const double lo = (Gp->ll_lo - mu) * inv_s, hi = (Gp->ll_hi - mu) * inv_s;
      const bool in = lo <= 0.0 && hi >= 0.0;
      double y = n * f64_H(dd_diff(alpha[k], A0), b, c, in ? 0.0 : ln_mor_norm(lo, hi));
      if (in && !(lo < -8.5 && hi > 8.5)) y /= mor_norm_slow(lo, hi);
      ws[w.y + (size_t)k * n_z + q] = y;
    }
  }
}

__device__ __forceinline__ void
dmma(double* c, double a, double b)
{
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// One block per (64-row lnM tile, richness bin, point): for 32 z_t nodes at a
// time S = sum_t F B over the tile's lam_t window (each of four warps 16 rows
// x 32 columns), then W_ij(k) += sum_q C_j(q) Y(k, q) S(k, q).  Chunks of 16
// lam_t nodes are double-buffered: F by 16-byte async copies, B = G u K_i
// formed in registers a chunk ahead.  Leading dimensions of 4 modulo 16
// doubles keep the fragment loads free of bank conflicts.  Bound by the FP64
// units: 30 KB of shared memory and 128 registers leave four blocks an SM.
constexpr int kCols = 32, kLdF = kF64Rows + 4, kLdB = kCols + 4, kLdS = kCols + 1;

__global__ void __launch_bounds__(128, 4)
f64_gemm_kernel(F64Launch L)
{
  const int p = L.p0 + blockIdx.z, i = blockIdx.y, m0 = blockIdx.x * kF64Rows;
  const PointDev pt = L.pts[p];
  if (!grid_in_mask(L.grid_mask, pt.grid)) return;
  const GridDev* __restrict__ Gp = L.grids + pt.grid;
  const int n_m = Gp->n_m, n_z = Gp->n_z, n_t = Gp->n_t, nJ = Gp->nJ;
  if (i >= Gp->nI || m0 >= n_m) return;
  const double* __restrict__ s64 = L.s64 + (size_t)p * Gp->s64_stride;
  const double* hdr = s64 + Gp->o_f64;
  if (hdr[0] == 0.0) return;
  const F64Ws w = f64_ws(n_m, n_z, n_t);
  const double* ws = L.ws + (size_t)blockIdx.z * L.ws_stride;
  // The tile's window, cut to the nodes where the bin's kernel matters.
  const int win = reinterpret_cast<const int*>(hdr + 4)[blockIdx.x];
  const int t_lo = max((win & 0xFFFF) * kF64Chunk, Gp->k64_lo[i] / kF64Chunk * kF64Chunk);
  const int t_hi = min((win >> 16) * kF64Chunk, w.n_tp);
  const int t_end = min(t_hi, (Gp->k64_hi[i] / kF64Chunk + 1) * kF64Chunk);
  __shared__ __align__(16) double Fs[2][kF64Chunk * kLdF];
  __shared__ __align__(16) double Bs[2][kF64Chunk * kLdB];
  __shared__ double cn[kMaxZBins * kCols], cg[kMaxZBins * kCols];
  double* Ss = Fs[0];  // [64][kLdS] after a column group's last chunk
  static_assert(kF64Rows * kLdS <= 2 * kF64Chunk * kLdF, "S tile fits the F buffers");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int fr = lane >> 2, fk = lane & 3;  // fragment row / column, k
  const double* __restrict__ F = ws + m0;
  const double* __restrict__ UK = Gp->UK64 + (size_t)i * n_t * n_z;
  // Epilogue: thread pair (row, half of the columns).
  const int row = tid >> 1, half = tid & 1;
  double wN[kMaxZBins], wG[kMaxZBins];
#pragma unroll
  for (int j = 0; j < kMaxZBins; ++j) wN[j] = wG[j] = 0.0;

  for (int q0 = 0; q0 < n_z; q0 += kCols) {
    const int nc = min(kCols, n_z - q0);  // 16 or 32
    double acc[2][4][2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
    auto load_F = [&](int t0, int buf) {  // 16 x 64 doubles, 16 bytes a copy
#pragma unroll
      for (int u = 0; u < kF64Chunk * kF64Rows / 2 / 128; ++u) {
        const int e = tid + 128 * u, t = e / (kF64Rows / 2), r = (e % (kF64Rows / 2)) * 2;
        const uint32_t dst =
          static_cast<uint32_t>(__cvta_generic_to_shared(&Fs[buf][t * kLdF + r]));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                     "l"(F + (size_t)(t0 + t) * w.n_mp + r)
                     : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double bv[kF64Chunk * kCols / 128];
    auto load_B = [&](int t0) {
#pragma unroll
      for (int u = 0; u < kF64Chunk * kCols / 128; ++u) {
        const int e = tid + 128 * u, t = t0 + e / kCols, q = e % kCols;
        const size_t at = (size_t)t * n_z + q0 + q;
        bv[u] = t < n_t && q < nc ? __ldg(ws + w.g + at) * __ldg(UK + at) : 0.0;
      }
    };
    auto store_B = [&](int buf) {
#pragma unroll
      for (int u = 0; u < kF64Chunk * kCols / 128; ++u) {
        const int e = tid + 128 * u;
        Bs[buf][(e / kCols) * kLdB + e % kCols] = bv[u];
      }
    };
    for (int u = tid; u < nJ * kCols; u += 128) {
      const int j = u / kCols, q = u % kCols;
      const double kj = q < nc ? Gp->Kj[j * n_z + q0 + q] : 0.0;
      cn[u] = q < nc ? s64[Gp->o_cz + q0 + q] * kj : 0.0;
      cg[u] = q < nc ? s64[Gp->o_czs + q0 + q] * kj : 0.0;
    }
    int buf = 0;
    if (t_lo < t_end) {
      load_F(t_lo, 0);
      load_B(t_lo);
      store_B(0);
    }
    for (int t0 = t_lo; t0 < t_end; t0 += kF64Chunk, buf ^= 1) {
      const bool more = t0 + kF64Chunk < t_end;
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();  // this chunk has landed, and the other buffer is free
      if (more) {
        load_F(t0 + kF64Chunk, buf ^ 1);
        load_B(t0 + kF64Chunk);
      }
#pragma unroll
      for (int k4 = 0; k4 < kF64Chunk; k4 += 4) {
        double a[2], b[4];
#pragma unroll
        for (int x = 0; x < 2; ++x)
          a[x] = Fs[buf][(k4 + fk) * kLdF + warp * 16 + x * 8 + fr];
#pragma unroll
        for (int y = 0; y < 4; ++y) b[y] = Bs[buf][(k4 + fk) * kLdB + y * 8 + fr];
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y) dmma(acc[x][y], a[x], b[y]);
      }
      if (more) store_B(buf ^ 1);
    }
    __syncthreads();  // the F buffers become the S tile
    // Y(k, q) S(k, q) of the fragments (row fr, columns 2 fk, 2 fk + 1).
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int r = warp * 16 + x * 8 + fr;
      const double* Y = ws + w.y + (size_t)min(m0 + r, n_m - 1) * n_z + q0;
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const int q = y * 8 + 2 * fk;
        if (q >= nc) continue;
        const double2 yv = *reinterpret_cast<const double2*>(Y + q);
        Ss[r * kLdS + q] = yv.x * acc[x][y][0];
        Ss[r * kLdS + q + 1] = yv.y * acc[x][y][1];
      }
    }
    __syncthreads();
    const int hc = nc / 2;
    for (int q = half * hc; q < (half + 1) * hc; ++q) {
      const double v = Ss[row * kLdS + q];
#pragma unroll
      for (int j = 0; j < kMaxZBins; ++j) {
        if (j >= nJ) break;
        wN[j] += cn[j * kCols + q] * v;
        if (L.shear) wG[j] += cg[j * kCols + q] * v;
      }
    }
    __syncthreads();  // S and the weights are read; the next group reuses them
  }
#pragma unroll
  for (int j = 0; j < kMaxZBins; ++j) {
    if (j >= nJ) break;
    const double a = wN[j] + __shfl_xor_sync(0xffffffffu, wN[j], 1);
    const double b = wG[j] + __shfl_xor_sync(0xffffffffu, wG[j], 1);
    if (half == 0 && m0 + row < n_m) {
      const size_t o = ((size_t)p * Gp->nB + i + Gp->nI * j) * L.w_stride + m0 + row;
      L.W[o] = a;
      if (L.shear) L.Wg[o] = b;
    }
  }
}

}  // namespace

size_t
f64_ws_doubles(int n_m, int n_z, int n_t)
{
  const F64Ws w = f64_ws(n_m, n_z, n_t);
  return (w.y + (size_t)n_m * n_z + 1) & ~size_t(1);
}

int
launch_f64(const F64Launch& L0, int n, int round, int row_tiles, int nI, cudaStream_t s)
{
  F64Launch L = L0;
  for (int p0 = 0; p0 < n; p0 += round) {
    const int m = n - p0 < round ? n - p0 : round;
    L.p0 = p0;
    // Enough blocks to fill the device with few points, ~20 elements a thread
    // with many.
    const int chunks = (int)((L.ws_stride + 20 * kFactorThreads - 1) / (20 * kFactorThreads));
    const int few = (4 * L.n_ctas + m - 1) / m, most = (int)(L.ws_stride / kFactorThreads + 1);
    f64_factor_kernel<<<dim3(min(max(chunks, few), most), m), kFactorThreads, 0, s>>>(L);
    count_launch();
    Y3B_CUDA(cudaGetLastError());
    f64_gemm_kernel<<<dim3(row_tiles, nI, m), 128, 0, s>>>(L);
    count_launch();
    Y3B_CUDA(cudaGetLastError());
  }
  return Y3B_OK;
}

}  // namespace y3b
