// mis_quad.cu -- the miscentred DeltaSigma of (R, R_mis) pairs at many scale
// radii: one quadrature geometry per pair, shared by its scale radii.
#include <algorithm>
#include <cmath>
#include <vector>

#include "mis_quad.cuh"

namespace y3b {

namespace {

constexpr int kPairThreads = 256;
constexpr int kPairX = 8;  // scale radii of one block

// Node n of the offset integral in units of R_mis, and its weight
// ws s exp(-s) / pi: two GL panels split at the ring crossing s = sk, or one.
__device__ __forceinline__ void
offset_node(const MisQuad& Q, double sk, int n, double* s, double* c)
{
  double ws;
  if (!(sk < Q.s_max && Q.n_s >= 2)) {
    *s = 0.5 * Q.s_max * (1.0 + Q.t0[n]);
    ws = 0.5 * Q.s_max * Q.w0[n];
  } else if (n < Q.n1) {
    *s = 0.5 * sk * (1.0 + Q.t1[n]);
    ws = 0.5 * sk * Q.w1[n];
  } else {
    *s = 0.5 * (sk + Q.s_max) + 0.5 * (Q.s_max - sk) * Q.t2[n - Q.n1];
    ws = 0.5 * (Q.s_max - sk) * Q.w2[n - Q.n1];
  }
  *c = ws * *s * exp(-*s) / kPi;
}

// The block's sum with the closed-form profile, for nodes outside the
// polynomials' range; out of line: the rare path.
__device__ __noinline__ double
pair_closed(const MisQuad& Q, double R, double rmis, double q)
{
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double acc = 0.0;
  for (int n = warp; n < Q.n_s; n += kPairThreads / 32) {
    double s, c;
    offset_node(Q, R / rmis, n, &s, &c);
    const double r = rmis * s;
    for (int t = lane; t < Q.n_theta; t += 32) {
      const double ct = Q.cth[t], D2 = R * R + r * r - 2.0 * R * r * ct, a = R - r * ct;
      acc += c * Q.wth[t] * (2.0 * a * a / D2 - 1.0) * NfwUnit<double>::dsigma(sqrt(D2 * q));
    }
  }
  return acc;
}

// One block per (pair, eight scale radii): a warp takes one offset ring after
// another, its lanes the ring angles.  A node's geometry (distance squared,
// weight times cos 2 phi) is formed once and used for the eight scale radii,
// which only scale the distance; the profile is the polynomial of
// nfw_table.cuh.  64 x 128 nodes, 60 pairs x 96 masses (47 M profile values):
// 168 us, bound by the polynomials' table reads (L1); at three blocks an SM
// the accumulators spill (214 us).
__global__ void __launch_bounds__(kPairThreads, 2)
mis_pairs_kernel(MisQuad Q, const double* __restrict__ nfw, MisPairs a)
{
  __shared__ double q_s[kPairX], amp_s[kPairX], red[kPairThreads / 32][kPairX];
  constexpr int nw = kPairThreads / 32;
  const int p = blockIdx.y, k0 = blockIdx.x * kPairX, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const double R = a.lnM ? a.R[p] : 1.0, rmis = a.rmis[p];
  if (tid < kPairX) {
    const int k = min(k0 + tid, a.nx - 1);
    if (a.lnM) {
      const double rs = nfw_rs(a.lnM[k], a.conc, a.rho);
      q_s[tid] = 1.0 / (rs * rs);
      amp_s[tid] = nfw_norm(a.lnM[k], a.conc, a.rho) * a.amp;
    } else {
      const double x = exp(a.u0 + k * a.du);
      q_s[tid] = x * x;
      amp_s[tid] = 1.0;
    }
  }
  __syncthreads();
  double q[kPairX], acc[kPairX];
#pragma unroll
  for (int u = 0; u < kPairX; ++u) {
    q[u] = q_s[u];
    acc[u] = 0.0;
  }
  bool outside = false;
  for (int n0 = warp; n0 < Q.n_s; n0 += 32 * nw) {  // 32 rings: a lane forms each one's node
    double s_l = 0.0, c_l = 0.0;
    if (n0 + nw * lane < Q.n_s) offset_node(Q, R / rmis, n0 + nw * lane, &s_l, &c_l);
    for (int m = 0; m < 32 && n0 + nw * m < Q.n_s; ++m) {
      const double r = rmis * __shfl_sync(0xffffffffu, s_l, m);
      const double cn = __shfl_sync(0xffffffffu, c_l, m);
      const double s2 = R * R + r * r, c2 = 2.0 * R * r;
      for (int t = lane; t < Q.n_theta; t += 32) {
        const double c = Q.cth[t], av = R - r * c, D2 = s2 - c2 * c;
        const double A = cn * Q.wth[t] * (2.0 * av * av / D2 - 1.0);
#pragma unroll
        for (int u = 0; u < kPairX; ++u) acc[u] += A * nfw_dsigma_w(nfw, D2 * q[u], outside);
      }
    }
  }
  if (__syncthreads_or(outside)) {
#pragma unroll 1
    for (int u = 0; u < kPairX; ++u) {
      const double v = pair_closed(Q, R, rmis, q_s[u]);
#pragma unroll
      for (int w = 0; w < kPairX; ++w) acc[w] = w == u ? v : acc[w];
    }
  }
  // Eight sums over the lanes by halving exchanges, then the warps in order.
#pragma unroll
  for (int h = kPairX / 2; h >= 1; h >>= 1) {
    const bool up = (lane & (4 * h)) != 0;
#pragma unroll
    for (int u = 0; u < h; ++u) {
      const double send = up ? acc[u] : acc[u + h];
      acc[u] = (up ? acc[u + h] : acc[u]) + __shfl_xor_sync(0xffffffffu, send, 4 * h);
    }
  }
  acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 2);
  acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
  if ((lane & 3) == 0) red[warp][lane >> 2] = acc[0];
  __syncthreads();
  if (tid < kPairX && k0 + tid < a.nx) {
    double v = 0.0;
    for (int w = 0; w < nw; ++w) v += red[w][tid];
    a.out[(size_t)p * a.nx + k0 + tid] = amp_s[tid] * v;
  }
}

__global__ void
cos_kernel(const double* x, int n, double* out)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = cos(x[i]);
}

}  // namespace

// Node positions on [lo, hi], then the barycentric interpolation matrix
// [node][mass].
std::vector<double>
cheb_rows(int N, double lo, double hi, const std::vector<double>& x)
{
  const size_t nx = x.size();
  const long double mid = 0.5L * ((long double)lo + hi), half = 0.5L * ((long double)hi - lo);
  std::vector<double> v(N + N * nx);
  std::vector<long double> wt(N), c(N);
  for (int j = 0; j < N; ++j) {
    const long double a = (2 * j + 1) * 3.14159265358979323846264338327950288L / (2 * N);
    v[j] = (double)(mid + half * std::cos(a));
    wt[j] = (j & 1 ? -1.0L : 1.0L) * std::sin(a);
  }
  for (size_t k = 0; k < nx; ++k) {
    long double sum = 0.0L;
    int hit = -1;
    for (int j = 0; j < N; ++j) {
      const long double d = (long double)x[k] - v[j];
      if (d == 0.0L) hit = j;
      c[j] = hit >= 0 ? 0.0L : wt[j] / d;
      sum += c[j];
    }
    for (int j = 0; j < N; ++j)
      v[N + j * nx + k] = hit >= 0 ? (j == hit ? 1.0 : 0.0) : (double)(c[j] / sum);
  }
  return v;
}

int
cos_device(const double* x, int n, double* out, cudaStream_t s)
{
  cos_kernel<<<(n + 127) / 128, 128, 0, s>>>(x, n, out);
  count_launch();
  return cuda_status(cudaGetLastError(), "cos_kernel");
}

int
launch_mis_pairs(const MisQuad& q, const double* nfw, const MisPairs& a, cudaStream_t s)
{
  for (int p0 = 0; p0 < a.n_pairs; p0 += 65535) {  // grid.y limit
    MisPairs b = a;
    b.n_pairs = std::min(65535, a.n_pairs - p0);
    b.R = a.R ? a.R + p0 : nullptr;
    b.rmis = a.rmis + p0;
    b.out = a.out + (size_t)p0 * a.nx;
    mis_pairs_kernel<<<dim3((a.nx + kPairX - 1) / kPairX, b.n_pairs), kPairThreads, 0, s>>>(
      q, nfw, b);
    count_launch();
    Y3B_TRY(cuda_status(cudaGetLastError(), "mis_pairs_kernel"));
  }
  return Y3B_OK;
}

}  // namespace y3b
