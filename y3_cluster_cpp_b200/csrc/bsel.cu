// bsel.cu -- the selection-bias operators P1, I1, J of P_operator
// (src/models/p_operator_t.hh:76-718, CosmoSIS module b_sel_marg, outputs
// b_sel_marg_P1 / _I1 / _J) on the GPU, batched over samples.
//
// Per sample the reference tabulates, on a linear reference grid z_r
// (p_operator_t.hh:124-219):
//   chi(z_r) h, dV/dz(z_r), sigma_z(z_r), n(M, z_r), b(M, z_r), and
//   p(lt | M, z_r) = exp(-lam + (lt + mi - 1) ln lam - lgamma(lt + mi)),
//   lam = l_sat + mi, mi = (l_sat sigma_lambda)^2,
//   l_sat = ((M - Mmin) / (M1 - Mmin))^alpha ((1 + z) / (1 + z_pivot))^epsilon,
// on each richness bin's own lambda_true GL nodes (0, lob_centre];
// then per grid point (z_obs bin, richness bin) (p_operator_t.hh:222-477):
//   a line-of-sight grid (GL on the exclusion ring around z_obs, log-GL in
//   comoving distance in front of and behind it), the tables interpolated
//   linearly in z onto it, the mass sums
//     W_P1[lt, z] = c_z lt w_lt sum_M w_M n p,  W_I = the same with n b,
//     c_z = (1 - u^2)_{|u| < 1} dV/dz w_z,  u = (z - z_obs) / sigma_z(z),
//   a theta grid on [min_z theta_excl(z), 2 theta_lob] split at theta_lob,
//   and
//     P1 = sum_th g_th sum_z sum_lt f_A W_P1,
//     I1 = sum_th g_th s(th) sum_z xi sum_lt f_A W_I,
//     J  = sum_th g_th (1 - s(th)) sum_z xi sum_lt f_A W_I,
//   over theta > theta_excl(z), with g_th = w_th 2 pi sin th, s the sigmoid
//   of the richness aperture, f_A the two-disk overlap fraction and xi the
//   nonlinear correlation function at z_obs and the 3-D separation.
//
// Device layout: one packed FP64 block per sample (scalars and tables) and
// four kernels a batch:
//   bsel_grid_kernel    one small block per (grid point, sample): line-of-sight
//                       and theta grids, and the reference z nodes they read;
//   bsel_sample_kernel  one block per (reference z node, sample): the MOR
//                       contracted over mass, as the moments below, where read;
//   bsel_point_kernel   one 512-thread block per (grid point, sample, group of
//                       theta nodes): the (theta, z, lambda_true) sums;
//   bsel_sum_kernel     the theta sums.
// With n, b and p linear in z between reference nodes i and i + 1 (weights
// g0 = 1 - f, g1 = f), the mass sums are polynomials in f whose coefficients
// do not depend on the grid point:
//   sum_M w n p   = g0 (g0 M0[i] + g1 M1[i]) + g1 (g0 M2[i+1] + g1 M0[i+1]),
//   sum_M w n b p = g0 (g0^2 M3[i] + g0 g1 M4[i] + g1^2 M5[i])
//                 + g1 (g0^2 M7[i+1] + g0 g1 M6[i+1] + g1^2 M3[i+1]),
// with the moments of node j over (lambda_true) sum_M w (.) p_j of
//   M0 n_j, M1 n_{j+1}, M2 n_{j-1}, M3 n_j b_j, M4 n_j b_{j+1} + n_{j+1} b_j,
//   M5 n_{j+1} b_{j+1}, M6 n_{j-1} b_j + n_j b_{j-1}, M7 n_{j-1} b_{j-1}:
// eight values replace the 24 of the mass nodes, and the point kernel reads
// ten instead of 48 per (z, lambda_true).  Every sum has a fixed order.
// This file is compiled without FMA contraction: the reference's separation
// sqrt(chi_z^2 + chi_o^2 - 2 chi_z chi_o cos theta) loses ten digits, and its
// roundings are kept (the loops that bound the kernels call fma()).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "bsel_math.cuh"
#include "common.cuh"
#include "host_common.h"
#include "zkernel_table.h"

namespace y3b {
namespace {

// Richness-bin centres for the edges [20, 30, 45, 60, 200] (p_op_detail::lob_center).
__host__ __device__ inline double
lob_centre(int b)
{
  return b == 0 ? 25.0 : (b == 1 ? 37.5 : (b == 2 ? 52.5 : 130.0));
}
constexpr int kPointThreads = 512, kPointWarps = kPointThreads / 32;
constexpr int kGridThreads = 96;
constexpr int kSampleThreads = 256;
constexpr int kScal = 16;  // scalars at the head of a sample block
constexpr int kMoments = 8;
constexpr int kGpScal = 4;  // scalars at the head of a grid point's grids

// Shapes, offsets and constant tables shared by the kernels of one call.
struct BselDims {
  int n_lt, n_zring, n_zouter, n_lnm, n_th, n_zr, n_gp, nz_max;
  double zr_lo, inv_dz_ref;
  // per-sample block: scal[16] | ln(m_h (Om - Onu)) | hmf z | dn/dlnM | dist z | d_a |
  // d_c | halo lnM | halo z | bias | xi r | xi z | xi
  int n_hm, n_hz, nd, n_hl, n_bz, n_xr, n_xz;
  long o_mh, o_hz, o_dn, o_dz, o_da, o_dc, o_bl, o_bz, o_bi, o_xr, o_xz, o_xi, blk;
  // per-sample moments [4][n_zr][kMoments][n_lt], bits of the reference
  // nodes read per bin [4][need_words], and per (grid point, sample) grids:
  // kGpScal scalars (theta_lob, chi_o, number of z nodes, fully excluded) |
  // bracket, f, chi, c_z, theta_excl, (1 + z) / chi [nz_max each] | theta,
  // g_theta, s(theta), cos theta [n_th each]
  long mom_bin, mom;
  int need_words;
  long g_z, g_th, grid;
  // constants (device): lnM nodes / weights, lambda_true nodes / weights /
  // R_lambda / 1 / (pi R_lambda^2) per bin [4][n_lt], reference z grid, photo-z width table,
  // grid points
  const double *lnm_x, *lnm_w, *lt_x, *lt_w, *rl, *ia, *zr, *zk_z, *zk_s;
  const double *gl_out, *gl_ring, *gl_th, *gl_th1, *gl_th2;  // nodes | weights on [-1, 1]
  const double *gp_zob, *gp_zfg, *gp_zbg;
  const int* gp_bin;
};

__device__ __forceinline__ double
chi_at(const BselDims& D, const double* B, double z)  // chi_.clamp(z) h0
{
  return interp1d_clamp(B + D.o_dz, B + D.o_dc, D.nd, z) * B[4];
}

// Lower bracket of z on the reference grid: i = min(trunc(u), n - 2) with
// u = (z - z_r0) / dz, the reference's size_t conversion
// (p_operator_t.hh:263-270); a u at or below -1 wraps to n - 2 there.
__device__ __forceinline__ int
ref_bracket(const BselDims& D, double z, double* f)
{
  const double u = (z - D.zr_lo) * D.inv_dz_ref;
  const long long t = (long long)u;
  const int i = t < 0 ? D.n_zr - 2 : (int)min(t, (long long)(D.n_zr - 2));
  *f = u - i;
  return i;
}

// z with chi(z) = target: the reference's 40-step bisection of [0.001, 2]
// (p_operator_t.hh:621-632); the table cells of the bracket's ends bound the
// search of each step.
__device__ __forceinline__ double
invert_chi(const BselDims& D, const double* B, double target)
{
  const double* zs = B + D.o_dz;
  const double* dc = B + D.o_dc;
  const double z0 = zs[0], z1 = zs[D.nd - 1], h0 = B[4];
  double lo = 0.001, hi = 2.0;
  int c_lo = 0, c_hi = D.nd - 1;
  for (int it = 0; it < 40; ++it) {
    const double mid = 0.5 * (lo + hi), x = fmin(fmax(mid, z0), z1);
    int a = c_lo, b = c_hi;
    while (b > a + 1) {
      const int m = (a + b) >> 1;
      if (zs[m] > x) b = m; else a = m;
    }
    const double dx = zs[a + 1] - zs[a];
    const double chi = (dx > 0.0 ? dc[a] + (x - zs[a]) / dx * (dc[a + 1] - dc[a]) : 0.0) * h0;
    if (chi < target) {
      lo = mid;
      c_lo = a;
    } else {
      hi = mid;
      c_hi = a + 1;
    }
  }
  return 0.5 * (lo + hi);
}

// One block per (grid point, sample): P_operator::evaluate's grids
// (p_operator_t.hh:222-430).  Latency-bound (interpolations, bisections), so
// small blocks, many to an SM.
__global__ void __launch_bounds__(kGridThreads, 8)
bsel_grid_kernel(BselDims D, const double* __restrict__ blocks, double* __restrict__ grids,
                 unsigned* __restrict__ need)
{
  const int g = blockIdx.x, s = blockIdx.y, tid = threadIdx.x;
  const double* B = blocks + (size_t)s * D.blk;
  double* G = grids + ((size_t)s * D.n_gp + g) * D.grid;
  double* Z = G + D.g_z;
  double* T = G + D.g_th;
  const int NZ = D.nz_max, NT = D.n_th, NO = D.n_zouter, NR = D.n_zring, bin = D.gp_bin[g];
  __shared__ double cq[5], sc[16], red[kGridThreads / 32];
  const double ddz = 1.0e-3, zob = D.gp_zob[g];
  if (tid < 5) {  // the five chi(z) this point needs, one lookup per thread
    const double zq[5] = {zob, D.gp_zfg[g], D.gp_zbg[g], zob + ddz, zob - ddz};
    cq[tid] = chi_at(D, B, zq[tid]);
  }
  __syncthreads();
  const double chi_o = cq[0];
  if (tid == 0) {  // build_z_grid_ (p_operator_t.hh:503-583)
    const double Rlob = pow(lob_centre(bin) / 100.0, 0.2);  // p_op_detail::R_lambda
    const double R_excl = Rlob * (1.0 + zob);
    const double dchi_dz = (cq[3] - cq[4]) / (2.0 * ddz);
    const double dz_excl = R_excl / dchi_dz;
    sc[0] = R_excl / chi_o;  // theta_lob
    sc[1] = R_excl;
    sc[2] = fmax(zob - dz_excl, D.gp_zfg[g]);
    sc[3] = fmin(zob + dz_excl, D.gp_zbg[g]);
    sc[4] = chi_o - cq[1];
    sc[5] = cq[2] - chi_o;
    sc[6] = log(R_excl);
    sc[7] = R_excl < sc[4] ? log(sc[4]) : 0.0;
    sc[8] = R_excl < sc[5] ? log(sc[5]) : 0.0;
  }
  __syncthreads();
  const double theta_lob = sc[0], R_excl = sc[1];
  const int n_fg = R_excl < sc[4] ? NO : 0, n_ring = sc[3] > sc[2] ? NR : 0;
  const int n_bg = R_excl < sc[5] ? NO : 0, Nz = n_fg + n_ring + n_bg;
  unsigned* nd = need + ((size_t)s * 4 + bin) * D.need_words;
  double tmin = 2.0 * theta_lob;
  for (int iz = tid; iz < Nz; iz += kGridThreads) {
    // front wing (farthest first), ring, back wing
    double z, wz;
    if (iz >= n_fg && iz < n_fg + n_ring) {
      const double hl = 0.5 * (sc[3] - sc[2]);
      z = 0.5 * (sc[2] + sc[3]) + hl * D.gl_ring[iz - n_fg];
      wz = hl * D.gl_ring[NR + iz - n_fg];
    } else {
      const bool fg = iz < n_fg;
      const int k = fg ? n_fg - 1 - iz : iz - n_fg - n_ring;
      const double b = fg ? sc[7] : sc[8], hl = 0.5 * (b - sc[6]);
      const double dis = exp(0.5 * (sc[6] + b) + hl * D.gl_out[k]);
      z = invert_chi(D, B, fg ? chi_o - dis : chi_o + dis);
      wz = hl * D.gl_out[NO + k] * dis /
           ((chi_at(D, B, z + ddz) - chi_at(D, B, z - ddz)) / (2.0 * ddz));
    }
    // the reference z tables at the bracket's nodes, linear in z
    double f;
    const int i = ref_bracket(D, z, &f);
    const double z0 = D.zr[i], z1 = D.zr[i + 1];
    double v0 = 0.0, v1 = 0.0;
    dv_do_dz(B + D.o_dz, B + D.o_da, D.nd, B[0], B[2], B[3], B[4], z0, &v0);
    dv_do_dz(B + D.o_dz, B + D.o_da, D.nd, B[0], B[2], B[3], B[4], z1, &v1);
    const double c0 = chi_at(D, B, z0), c1 = chi_at(D, B, z1), cz = c0 + f * (c1 - c0);
    const double s0 = interp1d_clamp(D.zk_z, D.zk_s, kZKernelNodes, z0);
    const double s1 = interp1d_clamp(D.zk_z, D.zk_s, kZKernelNodes, z1);
    const double u = (z - zob) / (s0 + f * (s1 - s0));
    const double wzv = fabs(u) < 1.0 ? 1.0 - u * u : 0.0;
    double ce = (cz * cz + chi_o * chi_o - R_excl * R_excl) / (2.0 * cz * chi_o);
    ce = ce < -1.0 ? -1.0 : (1.0 < ce ? 1.0 : ce);
    const double th = ce >= 1.0 - 1e-12 ? 1e-6 : acos(ce);
    Z[iz] = i;
    Z[NZ + iz] = f;
    Z[2 * NZ + iz] = cz;
    Z[3 * NZ + iz] = wzv == 0.0 ? 0.0 : wzv * (v0 + f * (v1 - v0)) * wz;
    // no theta passes a node outside the photo-z support
    Z[4 * NZ + iz] = wzv == 0.0 ? 1e300 : th;
    Z[5 * NZ + iz] = (1.0 + z) / cz;
    if (th < tmin) tmin = th;
    if (wzv != 0.0) {
      atomicOr(nd + (i >> 5), 1u << (i & 31));
      atomicOr(nd + ((i + 1) >> 5), 1u << ((i + 1) & 31));
    }
  }
  for (int off = 16; off > 0; off >>= 1)
    tmin = fmin(tmin, __shfl_xor_sync(0xffffffffu, tmin, off));
  if ((tid & 31) == 0) red[tid >> 5] = tmin;
  __syncthreads();
  // theta range and split (p_operator_t.hh:352-395)
  double th_lo = red[0];
  for (int w = 1; w < kGridThreads / 32; ++w) th_lo = fmin(th_lo, red[w]);
  const double th_hi = 2.0 * theta_lob;
  const int N1 = NT / 2, N2 = NT - N1;
  const double th_mid = th_lo > theta_lob ? th_lo : (th_hi < theta_lob ? th_hi : theta_lob);
  const bool split = !(N1 == 0 || th_mid <= th_lo || N2 == 0 || th_mid >= th_hi);
  if (tid == 0) {
    G[0] = theta_lob;
    G[1] = chi_o;
    G[2] = Nz;
    G[3] = th_lo >= th_hi ? 1.0 : 0.0;  // fully excluded: the integrand is zero
  }
  for (int it = tid; it < NT; it += kGridThreads) {
    const bool first = it < N1;
    const double a = split && !first ? th_mid : th_lo, b = split && first ? th_mid : th_hi;
    const double* q = split ? (first ? D.gl_th1 : D.gl_th2 - N1) : D.gl_th;
    const int nq = split ? (first ? N1 : N2) : NT;
    const double hl = 0.5 * (b - a), th = 0.5 * (a + b) + hl * q[it];
    T[it] = th;
    T[NT + it] = hl * q[nq + it] * 2.0 * kPi * sin(th);
    T[2 * NT + it] = 1.0 / (1.0 + exp(-(2.5 / theta_lob) * (th - 0.5 * theta_lob)));
    T[3 * NT + it] = cos(th);
  }
}

// Per (reference z node, sample): the moments of the shifted-Poisson MOR
// (P_operator::set_sample, p_operator_t.hh:150-219) of every richness bin
// whose grid points read the node.  The masses' factors stand in shared
// memory, kMassTile at a time (128 bytes a mass, below 48 KB for any count).
constexpr int kMassTile = 320;

__global__ void __launch_bounds__(kSampleThreads, 4)
bsel_sample_kernel(BselDims D, const double* __restrict__ blocks,
                   const unsigned* __restrict__ need, double* __restrict__ mom)
{
  extern __shared__ double ssm[];  // n, b [3][tile] | mi, lam [tile] | weights [tile][8]
  const int iz = blockIdx.x, s = blockIdx.y, tid = threadIdx.x;
  const int NM = D.n_lnm, NL = D.n_lt, NT = min(NM, kMassTile);
  unsigned used = 0;
  for (int bb = 0; bb < 4; ++bb)
    used |= ((need[((size_t)s * 4 + bb) * D.need_words + (iz >> 5)] >> (iz & 31)) & 1u) << bb;
  if (!used) return;
  const double* B = blocks + (size_t)s * D.blk;
  double* n_s = ssm;
  double* b_s = n_s + 3 * NT;
  double* mi_s = b_s + 3 * NT;
  double* lam_s = mi_s + NT;
  double* wt = lam_s + NT;
  const double z = D.zr[iz];
  const double Mmin = B[7], dM1 = B[8], alpha = B[9], sig_l = B[11];
  auto factors = [&](int m0, int nm_t) {  // of masses m0 .. m0 + nm_t - 1
    for (int k = tid; k < 7 * nm_t; k += kSampleThreads) {
      const int what = k / nm_t, iM = k - what * nm_t;
      const double x = D.lnm_x[m0 + iM];
      if (what < 6) {  // n and b at the nodes iz - 1, iz, iz + 1
        const double zn = D.zr[min(max(iz + what % 3 - 1, 0), D.n_zr - 1)];
        if (what < 3)
          n_s[what * NT + iM] =
            interp2d_clamp(B + D.o_mh, D.n_hm, B + D.o_hz, D.n_hz, B + D.o_dn, x, zn) *
            (B[5] * (x * kLog10e - kHmfPivot) + B[6]);
        else
          b_s[(what - 3) * NT + iM] =
            interp2d_clamp(B + D.o_bl, D.n_hl, B + D.o_bz, D.n_bz, B + D.o_bi, x, zn);
      } else {
        const double dM = fmax(exp(x) - Mmin, 0.0);
        const double l_sat = (dM > 0.0 && dM1 > 0.0)
                               ? pow(dM / dM1, alpha) * pow((1.0 + z) / (1.0 + B[12]), B[10])
                               : 0.0;
        const double mi = (l_sat * sig_l) * (l_sat * sig_l);
        mi_s[iM] = mi;
        lam_s[iM] = fmax(l_sat + mi, 1.0e-300);
      }
    }
    __syncthreads();
    for (int iM = tid; iM < nm_t; iM += kSampleThreads) {
      const double w = D.lnm_w[m0 + iM];
      const double nm = w * n_s[iM], n0 = w * n_s[NT + iM], np = w * n_s[2 * NT + iM];
      const double bm = b_s[iM], b0 = b_s[NT + iM], bp = b_s[2 * NT + iM];
      double* v = wt + kMoments * iM;
      v[0] = n0;
      v[1] = np;
      v[2] = nm;
      v[3] = n0 * b0;
      v[4] = n0 * bp + np * b0;
      v[5] = np * bp;
      v[6] = nm * b0 + n0 * bm;
      v[7] = nm * bm;
    }
    __syncthreads();
  };
  if (NM <= kMassTile) factors(0, NM);
  for (int k0 = 0; k0 < 4 * NL; k0 += kSampleThreads) {
    const int k = k0 + tid, bb = k / NL, il = k - bb * NL;
    const bool on = k < 4 * NL && ((used >> bb) & 1u);
    const double lt = on ? D.lt_x[k] : 0.0;
    double acc[kMoments];
#pragma unroll
    for (int m = 0; m < kMoments; ++m) acc[m] = 0.0;
    for (int m0 = 0; m0 < NM; m0 += kMassTile) {
      const int nm_t = min(kMassTile, NM - m0);
      if (NM > kMassTile) {
        __syncthreads();  // the last tile has been read
        factors(m0, nm_t);
      }
      if (!on) continue;
#pragma unroll 2
      for (int iM = 0; iM < nm_t; ++iM) {
        const double p = shifted_poisson(lt + mi_s[iM], lam_s[iM]);
#pragma unroll
        for (int m = 0; m < kMoments; ++m) acc[m] = fma(wt[kMoments * iM + m], p, acc[m]);
      }
    }
    if (!on) continue;
    double* dst = mom + (size_t)s * D.mom + bb * D.mom_bin + (size_t)iz * kMoments * NL + il;
#pragma unroll
    for (int m = 0; m < kMoments; ++m) dst[(size_t)m * NL] = acc[m];
  }
}

// Shared-memory doubles of bsel_point_kernel<LT> for the shapes in D (all
// theta nodes in one block).
inline long
point_smem_doubles(const BselDims& D, bool lt)
{
  const long NZ = D.nz_max, NT = D.n_th;
  return 2L * D.n_lt * NZ + (lt ? 2L * D.n_lt : 0L) + 3 * NZ + (NZ & 1) + NT * NZ +
         (NT * NZ + 7) / 8 + 2 * (NT + kPointWarps);
}

// One block per (grid point, sample, group of theta nodes): the mass sums
// W_P1, W_I from the moments (p_operator_t.hh:433-455), then
// sum_z sum_lt f_A W over theta > theta_excl(z) for each theta node
// (p_operator_t.hh:457-505) -> part[..][theta] = (P, xi I).  The block's
// (theta, z, lambda_true) terms are dealt to its warps in equal runs, z
// fastest, so that a warp's lanes share the overlap's branch; a run's sums are
// written per theta and added in the order of the warps.  Bound by the FP64
// units (the overlap's two angles and square root).
// LT: the lambda_true tables in shared memory too; where they do not fit
// beside the mass sums (hundreds of nodes) they are read from global memory.
template <bool LT>
__global__ void __launch_bounds__(kPointThreads, 2)
bsel_point_kernel(BselDims D, const double* __restrict__ blocks,
                  const double* __restrict__ grids, const double* __restrict__ mom,
                  double2* __restrict__ part)
{
  extern __shared__ __align__(16) double sm[];
  const int g = blockIdx.x, s = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double* B = blocks + (size_t)s * D.blk;
  const double* G = grids + ((size_t)s * D.n_gp + g) * D.grid;
  const double* Z = G + D.g_z;
  const double* T = G + D.g_th;
  const int NZ = D.nz_max, NL = D.n_lt, NT = D.n_th, bin = D.gp_bin[g];
  const int t0 = (int)((long)NT * blockIdx.z / gridDim.z);
  const int t1 = (int)((long)NT * (blockIdx.z + 1) / gridDim.z), nt = t1 - t0;
  double2* out = part + ((size_t)s * D.n_gp + g) * NT;
  if (G[3] != 0.0) {
    for (int it = t0 + tid; it < t1; it += kPointThreads) out[it] = make_double2(0.0, 0.0);
    return;
  }
  const double theta_lob = G[0], chi_o = G[1];
  const int Nz = (int)G[2], n_pair = Nz * NL;
  double* WP = sm;                    // [NL][Nz]
  double* WI = WP + (size_t)NL * NZ;
  double* lt_s = WI + (size_t)NL * NZ;
  const double* rl = LT ? lt_s : D.rl + bin * NL;       // [NL] R_lambda(lambda_true)
  const double* ia = LT ? lt_s + NL : D.ia + bin * NL;  // [NL] 1 / (pi R_lambda^2)
  double* thx = lt_s + (LT ? 2 * NL : 0);               // [Nz]
  double* ic1 = thx + NZ;             // [Nz] (1 + z) / chi
  double* c2 = ic1 + NZ;              // [Nz] its inverse square
  double2* red = reinterpret_cast<double2*>(c2 + NZ + (NZ & 1));
  double* xi = reinterpret_cast<double*>(red + nt + kPointWarps);  // [nt][Nz]
  uint8_t* on = reinterpret_cast<uint8_t*>(xi + (size_t)nt * NZ);  // [nt][Nz]
  for (int il = tid; LT && il < NL; il += kPointThreads) {
    lt_s[il] = D.rl[bin * NL + il];
    lt_s[NL + il] = D.ia[bin * NL + il];
  }
  for (int iz = tid; iz < Nz; iz += kPointThreads) {
    const double c = Z[5 * NZ + iz];
    thx[iz] = Z[4 * NZ + iz];
    ic1[iz] = c;
    c2[iz] = 1.0 / (c * c);
  }
  {
    const double* ltx = D.lt_x + bin * NL;
    const double* ltw = D.lt_w + bin * NL;
    const double* m = mom + (size_t)s * D.mom + bin * D.mom_bin;
    for (int k = tid; k < n_pair; k += kPointThreads) {
      const int iz = k / NL, il = k - iz * NL;
      const double cz = Z[3 * NZ + iz];
      double aP = 0.0, aI = 0.0;
      if (Z[4 * NZ + iz] < 1e299) {
        const double g1 = Z[NZ + iz], g0 = 1.0 - g1;
        const double* a = m + (size_t)(int)Z[iz] * kMoments * NL + il;  // node i
        const double* b = a + kMoments * NL;                            // node i + 1
        aP = g0 * (g0 * a[0] + g1 * a[NL]) + g1 * (g0 * b[2 * NL] + g1 * b[0]);
        aI = g0 * (g0 * g0 * a[3 * NL] + g0 * g1 * a[4 * NL] + g1 * g1 * a[5 * NL]) +
             g1 * (g0 * g0 * b[7 * NL] + g0 * g1 * b[6 * NL] + g1 * g1 * b[3 * NL]);
      }
      const double w = cz * (ltx[il] * ltw[il]);
      WP[il * Nz + iz] = w * aP;
      WI[il * Nz + iz] = w * aI;
    }
  }
  {  // xi_NL at z_obs and the separation (xi_lookup_, p_operator_t.hh:636-647)
    const double* xz = B + D.o_xz;
    const double* xr = B + D.o_xr;
    const double uz = (D.gp_zob[g] - xz[0]) * (1.0 / (xz[1] - xz[0]));
    int j = (int)floor(uz);
    j = j < 0 ? 0 : (j > D.n_xz - 2 ? D.n_xz - 2 : j);
    const double fz = uz - j, r_lo = xr[0], r_hi = xr[D.n_xr - 1];
    const double ln0 = log(r_lo), inv = 1.0 / log(xr[1] / r_lo);
    const double* x0 = B + D.o_xi + (size_t)j * D.n_xr;
    const double* x1 = x0 + D.n_xr;
    for (int k = tid; k < nt * Nz; k += kPointThreads) {
      const int it = k / Nz, iz = k - it * Nz;
      const bool in = T[t0 + it] > Z[4 * NZ + iz];
      on[k] = in;
      double v = 0.0;
      if (in) {
        const double cz = Z[2 * NZ + iz];
        const double dchi =
          sqrt(fmax(cz * cz + chi_o * chi_o - 2.0 * cz * chi_o * T[3 * NT + t0 + it], 0.0));
        const double r = dchi < r_lo ? r_lo : (r_hi < dchi ? r_hi : dchi);
        const double u = (log(r) - ln0) * inv;
        int ir = (int)floor(u);
        ir = ir < 0 ? 0 : (ir > D.n_xr - 2 ? D.n_xr - 2 : ir);
        const double a = x0[ir] + fz * (x1[ir] - x0[ir]);
        const double b = x0[ir + 1] + fz * (x1[ir + 1] - x0[ir + 1]);
        v = a + (u - ir) * (b - a);
      }
      xi[k] = v;
    }
  }
  __syncthreads();
  // Units of 32 (z, lambda_true) pairs; warp w takes [w U / 16, (w + 1) U / 16).
  const int u_th = (n_pair + 31) / 32;
  const long U = (long)nt * u_th;
  const long ua = U * warp / kPointWarps, ub = U * (warp + 1) / kPointWarps;
  for (long u = ua; u < ub;) {
    const int it = (int)(u / u_th);
    const long ue = min(ub, (long)(it + 1) * u_th);
    const double th = T[t0 + it];
    const double* xt = xi + (size_t)it * Nz;
    const uint8_t* ot = on + (size_t)it * Nz;
    int e = (int)(u - (long)it * u_th) * 32 + lane, il = e / Nz, iz = e - il * Nz;
    const double full = kPi * theta_lob * theta_lob;
    double sP = 0.0, sI = 0.0;
    for (; u < ue; ++u) {
      if (e < n_pair && ot[iz]) {
        const double l = rl[il] * ic1[iz];
        double fA = 0.0;
        const double inv = ia[il] * c2[iz];  // 1 / (pi l^2)
        if (th <= fabs(theta_lob - l))
          fA = l <= theta_lob ? 1.0 : full * inv;
        else if (!(th > theta_lob + l))
          fA = lens_area(th, theta_lob, l) * inv;
        sP = fma(fA, WP[e], sP);
        sI = fma(fA * WI[e], xt[iz], sI);
      }
      e += 32;
      iz += 32;
      while (iz >= Nz) {
        iz -= Nz;
        ++il;
      }
    }
    for (int off = 16; off > 0; off >>= 1) {
      sP += __shfl_xor_sync(0xffffffffu, sP, off);
      sI += __shfl_xor_sync(0xffffffffu, sI, off);
    }
    // The (theta, warp) pairs of the runs climb a staircase: theta + warp is
    // a place of its own.
    if (lane == 0) red[it + warp] = make_double2(sP, sI);
  }
  __syncthreads();
  for (int it = tid; it < nt; it += kPointThreads) {
    double a = 0.0, b = 0.0;
    for (int w = 0; w < kPointWarps; ++w) {
      const long lo = max(U * w / kPointWarps, (long)it * u_th);
      const long hi = min(U * (w + 1) / kPointWarps, (long)(it + 1) * u_th);
      if (lo < hi) {
        a += red[it + w].x;
        b += red[it + w].y;
      }
    }
    out[t0 + it] = make_double2(a, b);
  }
}

// P1, I1 and J of every (grid point, sample): theta in order.
__global__ void __launch_bounds__(128)
bsel_sum_kernel(BselDims D, const double* __restrict__ grids, const double2* __restrict__ part,
                int n, double* __restrict__ out)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const double* T = grids + (size_t)k * D.grid + D.g_th;
  const double2* P = part + (size_t)k * D.n_th;
  double a = 0.0, b = 0.0, c = 0.0;
  if (grids[(size_t)k * D.grid + 3] == 0.0)
    for (int it = 0; it < D.n_th; ++it) {
      const double w = T[D.n_th + it], sg = T[2 * D.n_th + it];
      a += w * P[it].x;
      b += w * (P[it].y * sg);
      c += w * (P[it].y * (1.0 - sg));
    }
  out[3 * (size_t)k] = a;
  out[3 * (size_t)k + 1] = b;
  out[3 * (size_t)k + 2] = c;
}

}  // namespace
}  // namespace y3b

namespace y3b {
// A chunk is packed, copied and evaluated in up to kPieces pieces of at least
// kPieceSamples samples: the host packs a piece while the device works on the
// one before.
constexpr int kPieces = 8, kPieceSamples = 24;
}  // namespace y3b

struct y3b_bsel {
  y3b_bsel_config cfg;
  std::vector<double> gp_zlo, gp_zhi, gp_zob, gp_zfg, gp_zbg;
  std::vector<int> gp_bin;
  std::vector<double> lnm_x, lnm_w, lt_x, lt_w, rl, ia, zr;  // lt_x, lt_w, rl, ia: [4][n_lt]
  int n_sm = 1;
  int max_samples = 64;
  y3b::DevBuf<double> d_const, d_blocks, d_work, d_out;
  y3b::DevBuf<int> d_int;  // grid-point bins
  double* h_stage = nullptr;  // pinned: sample blocks
  size_t h_stage_cap = 0;
  double* h_out = nullptr;  // pinned: results
  size_t h_out_cap = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev[2 * y3b::kPieces] = {};  // around the kernels of a chunk's pieces
  double last_kernel_ms = 0.0;
  ~y3b_bsel()
  {
    for (cudaEvent_t e : ev)
      if (e) cudaEventDestroy(e);
    if (h_stage) cudaFreeHost(h_stage);
    if (h_out) cudaFreeHost(h_out);
    if (stream) cudaStreamDestroy(stream);
  }
};

namespace y3b {
namespace {

double
h_sigma_z(double z)  // Interp1D(z_kernel_z, z_kernel_sigma).clamp(z)
{
  z = std::min(std::max(z, kZKernelZ[0]), kZKernelZ[kZKernelNodes - 1]);
  int lo = 0, hi = kZKernelNodes - 1;
  while (hi > lo + 1) {
    const int m = (lo + hi) / 2;
    if (kZKernelZ[m] > z)
      hi = m;
    else
      lo = m;
  }
  const double dx = kZKernelZ[lo + 1] - kZKernelZ[lo];
  return kZKernelSigma[lo] + (z - kZKernelZ[lo]) / dx * (kZKernelSigma[lo + 1] - kZKernelSigma[lo]);
}

// Photo-z support of a z_obs: z_fg + sigma_z(z_fg) = z_obs and
// z_bg - sigma_z(z_bg) = z_obs by bisection (bisect_photoz_fg_ / _bg_,
// p_operator_t.hh:590-618).
double
bisect_fg(double zob)
{
  double lo = 0.01, hi = zob;
  if (lo + h_sigma_z(lo) - zob > 0.0) return lo;
  for (int it = 0; it < 50; ++it) {
    const double mid = 0.5 * (lo + hi);
    const double f = mid + h_sigma_z(mid) - zob;
    if (f < 0.0)
      lo = mid;
    else
      hi = mid;
  }
  return 0.5 * (lo + hi);
}

double
bisect_bg(double zob)
{
  double lo = zob, hi = 1.5;
  if (hi - h_sigma_z(hi) - zob < 0.0) return hi;
  for (int it = 0; it < 50; ++it) {
    const double mid = 0.5 * (lo + hi);
    const double f = mid - h_sigma_z(mid) - zob;
    if (f < 0.0)
      lo = mid;
    else
      hi = mid;
  }
  return 0.5 * (lo + hi);
}

// Shapes and offsets of one call's sample blocks and work areas.
void
layout(const y3b_bsel* h, const y3b_bsel_sample& s0, BselDims& D)
{
  const y3b_bsel_config& c = h->cfg;
  D.n_lt = c.n_lt;
  D.n_zring = c.n_zring;
  D.n_zouter = c.n_zouter;
  D.n_lnm = c.n_lnm;
  D.n_th = c.n_theta;
  D.n_zr = c.n_zt_ref;
  D.n_gp = c.n_gp;
  D.nz_max = c.n_zring + 2 * c.n_zouter;
  D.zr_lo = c.zt_ref_low;
  D.inv_dz_ref = 1.0 / ((c.zt_ref_high - c.zt_ref_low) / (c.n_zt_ref - 1));
  D.n_hm = s0.t.n_hm;
  D.n_hz = s0.t.n_hz;
  D.nd = s0.t.n_dist;
  D.n_hl = s0.n_hl;
  D.n_bz = s0.n_hz;
  D.n_xr = s0.n_xr;
  D.n_xz = s0.n_xz;
  long o = kScal;
  D.o_mh = o, o += D.n_hm;
  D.o_hz = o, o += D.n_hz;
  D.o_dn = o, o += (long)D.n_hm * D.n_hz;
  D.o_dz = o, o += D.nd;
  D.o_da = o, o += D.nd;
  D.o_dc = o, o += D.nd;
  D.o_bl = o, o += D.n_hl;
  D.o_bz = o, o += D.n_bz;
  D.o_bi = o, o += (long)D.n_hl * D.n_bz;
  D.o_xr = o, o += D.n_xr;
  D.o_xz = o, o += D.n_xz;
  D.o_xi = o, o += (long)D.n_xr * D.n_xz;
  D.blk = (o + 1) & ~1L;
  D.mom_bin = (long)D.n_zr * kMoments * D.n_lt;
  D.mom = 4 * D.mom_bin;
  D.need_words = (D.n_zr + 31) / 32;
  D.g_z = kGpScal;
  D.g_th = D.g_z + 6L * D.nz_max;
  D.grid = D.g_th + 4L * D.n_th;
}

}  // namespace
}  // namespace y3b

extern "C" int
y3b_bsel_create(const y3b_bsel_config* cfg, y3b_bsel** out)
{
  using namespace y3b;
  clear_error();
  if (!cfg || !out || cfg->n_gp < 1 || !cfg->zo_low || !cfg->zo_high || !cfg->lambda_bin ||
      cfg->n_lt < 1 || cfg->n_zring < 1 || cfg->n_zouter < 1 || cfg->n_lnm < 1 ||
      cfg->n_theta < 1 || cfg->n_zt_ref < 2 || !(cfg->zt_ref_high > cfg->zt_ref_low) ||
      !(cfg->lnm_high > cfg->lnm_low) || cfg->max_samples < 0 ||
      cfg->max_samples > 65535) {
    set_error("y3b_bsel_create: invalid configuration (grid points, node counts >= 1, "
              "n_zt_ref >= 2, ordered bounds, max_samples <= 65535)");
    return Y3B_ERR_INVALID;
  }
  *out = nullptr;
  Y3B_TRY(require_device());
  y3b_bsel* h = new (std::nothrow) y3b_bsel();
  if (!h) return Y3B_ERR_NOMEM;
  h->cfg = *cfg;
  if (cfg->max_samples > 0) h->max_samples = cfg->max_samples;
  const int ngp = cfg->n_gp;
  for (int i = 0; i < ngp; ++i) {
    const int b = cfg->lambda_bin[i];
    if (b < 0 || b > 3) {
      set_error("y3b_bsel_create: lambda_bin %d outside the four richness bins", b);
      delete h;
      return Y3B_ERR_INVALID;
    }
    const double zob = 0.5 * (cfg->zo_low[i] + cfg->zo_high[i]);
    h->gp_zlo.push_back(cfg->zo_low[i]);
    h->gp_zhi.push_back(cfg->zo_high[i]);
    h->gp_zob.push_back(zob);
    h->gp_bin.push_back(b);
    h->gp_zfg.push_back(bisect_fg(zob));
    h->gp_zbg.push_back(bisect_bg(zob));
  }
  h->cfg.zo_low = h->gp_zlo.data();
  h->cfg.zo_high = h->gp_zhi.data();
  h->cfg.lambda_bin = h->gp_bin.data();
  gl_nodes_host(cfg->lnm_low, cfg->lnm_high, cfg->n_lnm, h->lnm_x, h->lnm_w);
  std::vector<double> x, w;
  for (int b = 0; b < 4; ++b) {
    gl_nodes_host(1.0e-6, lob_centre(b), cfg->n_lt, x, w);
    for (int il = 0; il < cfg->n_lt; ++il) {
      h->lt_x.push_back(x[il]);
      h->lt_w.push_back(w[il]);
      const double r = std::pow(x[il] / 100.0, 0.2);
      h->rl.push_back(r);
      h->ia.push_back(1.0 / (kPi * r * r));
    }
  }
  const double dz_ref = (cfg->zt_ref_high - cfg->zt_ref_low) / (cfg->n_zt_ref - 1);
  for (int i = 0; i < cfg->n_zt_ref; ++i) h->zr.push_back(cfg->zt_ref_low + i * dz_ref);
  // Constant tables in one device buffer.
  std::vector<double> cst;
  auto put = [&](const double* p, size_t n) { cst.insert(cst.end(), p, p + n); };
  put(h->lnm_x.data(), h->lnm_x.size());
  put(h->lnm_w.data(), h->lnm_w.size());
  put(h->lt_x.data(), h->lt_x.size());
  put(h->lt_w.data(), h->lt_w.size());
  put(h->rl.data(), h->rl.size());
  put(h->ia.data(), h->ia.size());
  put(h->zr.data(), h->zr.size());
  put(kZKernelZ, kZKernelNodes);
  put(kZKernelSigma, kZKernelNodes);
  put(h->gp_zob.data(), ngp);
  put(h->gp_zfg.data(), ngp);
  put(h->gp_zbg.data(), ngp);
  for (int n : {cfg->n_zouter, cfg->n_zring, cfg->n_theta, cfg->n_theta / 2,
                cfg->n_theta - cfg->n_theta / 2}) {
    gl_nodes_host(-1.0, 1.0, n, x, w);
    put(x.data(), n);
    put(w.data(), n);
  }
  int dev = 0;
  cudaGetDevice(&dev);
  int rc = cuda_status(cudaDeviceGetAttribute(&h->n_sm, cudaDevAttrMultiProcessorCount, dev),
                       "cudaDeviceGetAttribute");
  if (!rc) rc = allow_max_smem(bsel_point_kernel<true>);
  if (!rc) rc = allow_max_smem(bsel_point_kernel<false>);
  if (!rc) rc = cuda_status(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking),
                       "cudaStreamCreate");
  const std::vector<int>& ints = h->gp_bin;
  for (int i = 0; i < 2 * kPieces && !rc; ++i)
    rc = cuda_status(cudaEventCreate(&h->ev[i]), "cudaEventCreate");
  if (!rc) rc = h->d_const.upload(cst.data(), cst.size(), h->stream);
  if (!rc) rc = h->d_int.upload(ints.data(), ints.size(), h->stream);
  if (!rc) rc = cuda_status(cudaStreamSynchronize(h->stream), "cudaStreamSynchronize");
  if (rc) {
    delete h;
    return rc;
  }
  *out = h;
  return Y3B_OK;
}

extern "C" int
y3b_bsel_kernel_ms(const y3b_bsel* h, double* ms)
{
  y3b::clear_error();
  if (!h || !ms) {
    y3b::set_error("y3b_bsel_kernel_ms: invalid arguments");
    return Y3B_ERR_INVALID;
  }
  *ms = h->last_kernel_ms;
  return Y3B_OK;
}

extern "C" void
y3b_bsel_destroy(y3b_bsel* h)
{
  delete h;
}

extern "C" int
y3b_bsel_eval(y3b_bsel* h, int n_samples, const y3b_bsel_sample* S, double* out)
{
  using namespace y3b;
  clear_error();
  if (!h || n_samples < 0 || (n_samples && (!S || !out))) {
    set_error("y3b_bsel_eval: invalid arguments");
    return Y3B_ERR_INVALID;
  }
  if (n_samples == 0) return Y3B_OK;
  const y3b_bsel_config& c = h->cfg;
  const y3b_bsel_sample& s0 = S[0];
  for (int k = 0; k < n_samples; ++k) {
    const y3b_bsel_sample& s = S[k];
    const y3b_tables& t = s.t;
    if (!t.hmf_m_h || !t.hmf_z || !t.dndlnmh || !t.dist_z || !t.dist_da || !s.dist_dc ||
        !s.halo_lnM || !s.halo_z || !s.bias || !s.xi_r || !s.xi_z || !s.xi_nl || t.n_hm < 2 ||
        t.n_hz < 2 || t.n_dist < 2 || s.n_hl < 2 || s.n_hz < 2 || s.n_xr < 2 || s.n_xz < 2) {
      set_error("y3b_bsel_eval: sample %d is incomplete (tables of at least two nodes each)", k);
      return Y3B_ERR_INVALID;
    }
    if (t.n_hm != s0.t.n_hm || t.n_hz != s0.t.n_hz || t.n_dist != s0.t.n_dist ||
        s.n_hl != s0.n_hl || s.n_hz != s0.n_hz || s.n_xr != s0.n_xr || s.n_xz != s0.n_xz) {
      set_error("y3b_bsel_eval: sample %d has table shapes different from sample 0", k);
      return Y3B_ERR_INVALID;
    }
    if (!(c.zt_ref_low >= t.dist_z[0] && c.zt_ref_high <= t.dist_z[t.n_dist - 1] &&
          h->zr.back() <= t.dist_z[t.n_dist - 1])) {
      set_error("argument out of range in Interp1D (sample %d: the reference z grid "
                "[%g, %g] leaves distances/z)", k, c.zt_ref_low, c.zt_ref_high);
      return Y3B_ERR_DOMAIN;
    }
  }
  BselDims D;
  layout(h, s0, D);
  size_t smem = (size_t)point_smem_doubles(D, true) * sizeof(double);
  const bool lt_smem = smem <= 227 * 1024;
  if (!lt_smem) smem = (size_t)point_smem_doubles(D, false) * sizeof(double);
  if (smem > 227 * 1024) {
    set_error("y3b_bsel_eval: node counts need %zu bytes of shared memory per grid point "
              "(at most 227 KB)", smem);
    return Y3B_ERR_INVALID;
  }
  const double* cd = h->d_const.get();
  const int NL = c.n_lt, ngp = c.n_gp;
  D.lnm_x = cd;
  D.lnm_w = D.lnm_x + c.n_lnm;
  D.lt_x = D.lnm_w + c.n_lnm;
  D.lt_w = D.lt_x + 4 * NL;
  D.rl = D.lt_w + 4 * NL;
  D.ia = D.rl + 4 * NL;
  D.zr = D.ia + 4 * NL;
  D.zk_z = D.zr + c.n_zt_ref;
  D.zk_s = D.zk_z + kZKernelNodes;
  D.gp_zob = D.zk_s + kZKernelNodes;
  D.gp_zfg = D.gp_zob + ngp;
  D.gp_zbg = D.gp_zfg + ngp;
  D.gl_out = D.gp_zbg + ngp;
  D.gl_ring = D.gl_out + 2 * c.n_zouter;
  D.gl_th = D.gl_ring + 2 * c.n_zring;
  D.gl_th1 = D.gl_th + 2 * c.n_theta;
  D.gl_th2 = D.gl_th1 + 2 * (c.n_theta / 2);
  D.gp_bin = h->d_int.get();
  const int chunk = std::min(n_samples, h->max_samples);
  // Pinned staging for the sample blocks and the results.
  const size_t stage = (size_t)chunk * D.blk, outn = (size_t)chunk * ngp * 3;
  if (h->h_stage_cap < stage) {
    if (h->h_stage) cudaFreeHost(h->h_stage);
    h->h_stage = nullptr;
    h->h_stage_cap = 0;
    Y3B_CUDA(cudaHostAlloc((void**)&h->h_stage, stage * sizeof(double), cudaHostAllocDefault));
    h->h_stage_cap = stage;
  }
  if (h->h_out_cap < outn) {
    if (h->h_out) cudaFreeHost(h->h_out);
    h->h_out = nullptr;
    h->h_out_cap = 0;
    Y3B_CUDA(cudaHostAlloc((void**)&h->h_out, outn * sizeof(double), cudaHostAllocDefault));
    h->h_out_cap = outn;
  }
  Y3B_TRY(h->d_blocks.alloc(stage));
  // One work block: theta sums | grids | moments | bits of the reference z
  // nodes read.
  const size_t n_part = 2 * (size_t)chunk * ngp * c.n_theta;
  const size_t n_grids = (size_t)chunk * ngp * D.grid, n_mom = (size_t)chunk * D.mom;
  const size_t needs = (size_t)chunk * 4 * D.need_words;
  Y3B_TRY(h->d_work.alloc(n_part + n_grids + n_mom + (needs + 1) / 2));
  double* const w_part = h->d_work.get();
  double* const w_grids = w_part + n_part;
  double* const w_mom = w_grids + n_grids;
  unsigned* const w_need = reinterpret_cast<unsigned*>(w_mom + n_mom);
  Y3B_TRY(h->d_out.alloc(outn));
  cudaStream_t st = h->stream;
  h->last_kernel_ms = 0.0;
  for (int k0 = 0; k0 < n_samples; k0 += chunk) {
    const int n_chunk = std::min(chunk, n_samples - k0);
    const int pieces = std::max(1, std::min(kPieces, n_chunk / kPieceSamples));
    // The previous chunk's copies out of the staging buffers are done.
    Y3B_CUDA(cudaStreamSynchronize(st));
    Y3B_CUDA(cudaMemsetAsync(w_need, 0, needs * sizeof(unsigned), st));
    for (int pc = 0; pc < pieces; ++pc) {
      const int ka = (int)((long)n_chunk * pc / pieces);
      const int nk = (int)((long)n_chunk * (pc + 1) / pieces) - ka;
      for (int k = 0; k < nk; ++k) {
        const y3b_bsel_sample& s = S[k0 + ka + k];
        double* b = h->h_stage + (size_t)(ka + k) * D.blk;
        const double Mmin = std::pow(10.0, s.hod[0]), M1 = std::pow(10.0, s.hod[1]);
        const double sc[kScal] = {s.cosmo.om, s.cosmo.onu, s.cosmo.ol, s.cosmo.ok, s.cosmo.h0,
                                  s.cosmo.hmf_s, s.cosmo.hmf_q, Mmin, M1 - Mmin, s.hod[2],
                                  s.hod[3], s.hod[4], s.hod[5], 0.0, 0.0, 0.0};
        std::memcpy(b, sc, sizeof sc);
        for (int i = 0; i < D.n_hm; ++i)  // HMF_t's log mass axis (hmf_t.hh:16-25)
          b[D.o_mh + i] = std::log(s.t.hmf_m_h[i] * (s.cosmo.om - s.cosmo.onu));
        std::memcpy(b + D.o_hz, s.t.hmf_z, sizeof(double) * D.n_hz);
        std::memcpy(b + D.o_dn, s.t.dndlnmh, sizeof(double) * D.n_hz * D.n_hm);
        std::memcpy(b + D.o_dz, s.t.dist_z, sizeof(double) * D.nd);
        std::memcpy(b + D.o_da, s.t.dist_da, sizeof(double) * D.nd);
        std::memcpy(b + D.o_dc, s.dist_dc, sizeof(double) * D.nd);
        std::memcpy(b + D.o_bl, s.halo_lnM, sizeof(double) * D.n_hl);
        std::memcpy(b + D.o_bz, s.halo_z, sizeof(double) * D.n_bz);
        std::memcpy(b + D.o_bi, s.bias, sizeof(double) * D.n_hl * D.n_bz);
        std::memcpy(b + D.o_xr, s.xi_r, sizeof(double) * D.n_xr);
        std::memcpy(b + D.o_xz, s.xi_z, sizeof(double) * D.n_xz);
        std::memcpy(b + D.o_xi, s.xi_nl, sizeof(double) * D.n_xr * D.n_xz);
      }
      double* blocks = h->d_blocks.get() + (size_t)ka * D.blk;
      double* grids = w_grids + (size_t)ka * ngp * D.grid;
      double* mom = w_mom + (size_t)ka * D.mom;
      unsigned* need = w_need + (size_t)ka * 4 * D.need_words;
      double2* part = reinterpret_cast<double2*>(w_part) + (size_t)ka * ngp * c.n_theta;
      double* o = h->d_out.get() + (size_t)ka * ngp * 3;
      Y3B_CUDA(cudaMemcpyAsync(blocks, h->h_stage + (size_t)ka * D.blk,
                               sizeof(double) * nk * D.blk, cudaMemcpyHostToDevice, st));
      Y3B_CUDA(cudaEventRecord(h->ev[2 * pc], st));
      bsel_grid_kernel<<<dim3(ngp, nk), kGridThreads, 0, st>>>(D, blocks, grids, need);
      count_launch();
      Y3B_CUDA(cudaGetLastError());
      bsel_sample_kernel<<<dim3(D.n_zr, nk), kSampleThreads,
                           (8 + kMoments) * sizeof(double) * std::min(c.n_lnm, kMassTile), st>>>(
        D, blocks, need, mom);
      count_launch();
      Y3B_CUDA(cudaGetLastError());
      // Few (grid point, sample) pairs: several blocks each, by theta.
      const int split = std::max(1, std::min(c.n_theta, 2 * h->n_sm / std::max(1, ngp * nk)));
      auto point = lt_smem ? bsel_point_kernel<true> : bsel_point_kernel<false>;
      point<<<dim3(ngp, nk, split), kPointThreads, smem, st>>>(D, blocks, grids, mom, part);
      count_launch();
      Y3B_CUDA(cudaGetLastError());
      bsel_sum_kernel<<<(ngp * nk + 127) / 128, 128, 0, st>>>(D, grids, part, ngp * nk, o);
      count_launch();
      Y3B_CUDA(cudaGetLastError());
      Y3B_CUDA(cudaEventRecord(h->ev[2 * pc + 1], st));
    }
    Y3B_CUDA(cudaMemcpyAsync(h->h_out, h->d_out.get(), sizeof(double) * n_chunk * ngp * 3,
                             cudaMemcpyDeviceToHost, st));
    Y3B_CUDA(cudaStreamSynchronize(st));
    for (int pc = 0; pc < pieces; ++pc) {
      float ms = 0.f;
      Y3B_CUDA(cudaEventElapsedTime(&ms, h->ev[2 * pc], h->ev[2 * pc + 1]));
      h->last_kernel_ms += ms;
    }
    std::memcpy(out + (size_t)k0 * ngp * 3, h->h_out, sizeof(double) * n_chunk * ngp * 3);
  }
  return Y3B_OK;
}
