// prj_shear.cu -- the frozen-physics projection-shear observable
// <DeltaSigma_prj>(R | lambda bin, z_obs) of ShearPrjFrozenPhysics
// (src/models/sigma_prj_frozen_t.hh:34-512) on the GPU.
//
// Per sample and per (richness bin, z_obs) slice the reference builds, once:
//   * a log-GL theta grid split at the slice's breakpoints (inner cut, the
//     line-of-sight exclusion angle, theta_R = R / D_A for every radius,
//     theta_lambda, 2 theta_lambda, theta_max; sigma_prj_t.hh:95-180),
//   * a line-of-sight z grid: GL on the exclusion ring around z_obs and
//     log-GL in comoving distance in front of and behind it
//     (sigma_prj_frozen_t.hh:380-455),
// then accumulates, in FP64,
//   wrnd(M)    = sum_z c_z n(M, z) w_M,                   (random channel)
//   Psi(theta) = sum_z c_z a_b(z) xi_NL(dchi(z, theta), z_obs)   over theta > theta_excl(z),
//   a_b(z)     = sum_M w_M r_s(M) n(M, z) b(M, z) / sum_M w_M r_s(M) n(M, z_obs) b(M, z_obs),
//   c_z        = dV/dz Omega(z) w_z (1 - u^2)_{|u| < 1},  u = (z - z_obs) / sigma_z(z),
// and per grid point (slice, R)
//   rnd = sum_theta g_theta sum_M wrnd(M) DSigma_mis(R | theta D_A, M),
//   cl  = sum_theta g_theta b_sel(theta) Psi(theta) sum_M w_M n(M, z_obs) b(M, z_obs) DSigma_mis,
// g_theta = w_theta 2 pi sin theta, b_sel a sigmoid between the
// b_sel_marginalised asymptotes; the shear is the same times
// Sigma_crit^-1(z_obs).  DSigma_mis is NFW_DSIGMA_MIS with the single
// (fixed-offset) kernel: the reference's table when loaded, else its direct
// quadrature.
//
// A call copies the sample's tables in one transfer and runs four kernels:
// prj_slice_kernel (one block per slice: both grids, the line-of-sight sums),
// prj_psi_kernel (one warp per theta node), prj_profile_kernel (one warp per
// (grid point, theta node): the profile of every mass or Chebyshev node,
// contracted with the slice's mass weights) and prj_sum_kernel (one block per
// grid point: the theta sums).  Every sum has a fixed order.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "common.cuh"
#include "host_common.h"
#include "mis_quad.cuh"
#include "nfw_table.cuh"
#include "zkernel_table.h"

namespace y3b {
namespace {

constexpr double kPiP = 3.14159265358979323846;
constexpr double kConc = 4.0;  // NFW_DSIGMA_MIS(4, RHOC, SINGLE), sigma_prj_frozen_t.hh:71

// Gauss-Legendre nodes on [a, b] (p_operator_cuhre_t.hh:66-95).
void
h_gl(double a, double b, int n, std::vector<double>& x, std::vector<double>& w)
{
  gl_nodes_host(a, b, n, x, w);
}

// ---- device side ----------------------------------------------------------
// Shapes, offsets and constants of one call.  The sample block holds, in
// order, 8 scalars (Omega_M, Omega_nu, Omega_L, Omega_k, h0, hmf_s, hmf_q,
// n(sci) > 1) and the tables; a slice's scratch its grids and sums.
struct PrjDims {
  int n_lnm, n_seg, n_zring, n_zouter, ngp, nsl, nR_max, nt_max, nz;  // n_seg: nodes a segment
  double zt_low, zt_high, R_max;
  int omega_z;
  int n_hm, n_hz, nd, n_sci, n_bl, n_bz, n_xr, n_xz, n_blob, n_bzob;
  long o_mh, o_hz, o_dn, o_dz, o_da, o_dc, o_sz, o_sv, o_bl, o_bz, o_bi, o_xr, o_xz, o_xi, o_bzob,
    o_bs, o_blg;
  long s_mh, s_xi, s_bd, s_th, s_geom, s_bsel, s_wcl_th, s_z, s_zc, s_chi, s_thex, s_ab, s_wz,
    s_wrnd, s_wcl, s_pr, s_pc, s_scal, scratch;
  int n_prof;            // masses of the profile: n_lnm, or the Chebyshev nodes
  // constants of the handle (device)
  const double *lnm_x, *lnm_w, *anchor;        // [n_lnm]; anchor = w r_s
  const double *gl_seg, *gl_ring, *gl_out;     // nodes | weights on [-1, 1]
  const double *zk_z, *zk_s;                   // photo-z width
  const double *sl_lob, *sl_zob, *radii;       // per slice; radii ascending, slice by slice
  const double* gp_R;
  const double* cheb;    // [n_prof][n_lnm] projection of mass weights on the nodes, or null
  const int *sl_lb, *r0, *gp_slice;            // r0 [nsl + 1]
};

// The single-kernel miscentring table (nfw_dsigma_mis.hh:62-72).
struct PrjTable {
  int n_lx, n_lxm;
  const double *lx, *lxm, *ltab;
};

// The fixed-offset profile without a table: the 256-node GL rule over the
// ring angle, and the 32, 64 and 128-node rules that give the same ring
// average to FP64 rounding where the ring keeps clear of the offset centre.
// At ring angle t the integrand has its nearest singularity (d = 0) at
// t = i ln(x_mis / x), so an m-node rule on [0, pi] converges as
// rho_E^-2m with rho_E = a + sqrt(a^2 - 1), a = exp(asinh(|ln(x_mis / x)| / pi)):
// 1e-18 from the |ln| below on.  In 24-node theta grids over two decades
// the rules average about 50 nodes a ring.
constexpr int kRuleN0 = 32, kRuleN1 = 64, kRuleN2 = 128, kRuleN3 = 256;
constexpr int kRuleTot = kRuleN0 + kRuleN1 + kRuleN2 + kRuleN3;
constexpr double kRuleLn0 = 0.609, kRuleLn1 = 0.1587, kRuleLn2 = 0.0401;

// The profile of a ring is analytic in ln r_s = lnM / 3 + const, |Im| < pi
// (it sums the NFW DeltaSigma at distances proportional to 1 / r_s), and
// enters only through sums over the masses with the slice's weights.  Where
// it saves a group of masses (more than 20 of them, on at most six e-folds)
// the profile is taken at 20 Chebyshev nodes of lnM and the weights are
// projected on the nodes instead.  It is the profile per unit mass that is
// interpolated, which spans the range within two decades: the interpolant
// converges as rho^-n (rho = h + sqrt(h^2 + 1), h = 6 pi / range, 6.4 at six
// e-folds) from a constant of some tens, the branch points of the ring's many
// distances.  At six e-folds, over radii from 0.05 to 30 and R_mis from
// R / 100 to 100 R, the error of a mass is at most 5.6e-15 of its ring's sum
// of |terms| (1.6e-11 with 16 nodes, 1e-15 the sum's own rounding).
// 24 masses, 120 grid points: 97 -> 82 us (16 nodes: 67).
constexpr int kProfNodes = 20;
constexpr double kProfRange = 6.0;

struct PrjQuad {
  const double* rule;    // cos(t) [kRuleTot] | weights [kRuleTot] of the GL nodes on [0, pi]
  const double* mass;    // 1 / r_s^2 [n_prof] | profile amplitude without Omega_M [n_prof]
                         // (Chebyshev nodes: times exp(-(lnM - mid)))
  const double* nfw;     // DeltaSigma polynomials
};

// NFW_DSIGMA_MIS(R, R_mis, lnM), single kernel (nfw_dsigma_mis.hh:95-114),
// from its table: r_s from rho_c, amplitude 2 r_s delta_c rho_c Omega_M
// 1e-12 [h Msun/pc^2].
__device__ double
dsigma_single_table(const PrjTable& T, double R, double Rmis, double lnM)
{
  const double rs = nfw_rs(lnM, kConc, kRhoCrit);
  const double unit = exp(
    interp2d_clamp(T.lx, T.n_lx, T.lxm, T.n_lxm, T.ltab, log(R / rs), log(Rmis / rs)));
  return nfw_norm(lnM, kConc, kRhoCrit) * unit;
}

// Per slice: the theta and z grids and the sums over the line of sight.
// One block; the node counts are a few dozen to a few hundred, so the block
// is bound by the latency of its phases (interpolations, the 40-step chi(z)
// bisections), which run one node a thread.  24 masses, 60 z nodes, 12 slices:
// 64 -> 41 us with bisections that narrow their table search with the interval,
// the table cells of a mass and of a z node found once, and the scalar set-up on
// three warps.
constexpr int kSliceThreads = 512;

__global__ void __launch_bounds__(kSliceThreads)
prj_slice_kernel(PrjDims D, const double* __restrict__ B, double* __restrict__ scratch,
                 int* __restrict__ nt_out, int* status)
{
  const int sl = blockIdx.x, tid = threadIdx.x, nt_thr = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = nt_thr >> 5;
  double* S = scratch + (size_t)sl * D.scratch;
  const double om = B[0], h0 = B[4];
  const double* dz = B + D.o_dz;
  const double zob = D.sl_zob[sl];
  __shared__ double sc[16], chis[5];
  __shared__ int n_bd_s;
  auto chi = [&](double z) { return interp1d_clamp(dz, B + D.o_dc, D.nd, z) * h0; };
  constexpr double dz1 = 1.0e-3;
  if (tid < 5) {
    const double zq[5] = {zob, D.zt_low, D.zt_high, zob + dz1, zob - dz1};
    chis[tid] = chi(zq[tid]);
  }
  // HMF mass axis ln(m_h (Omega_M - Omega_nu)) and xi_NL(r, z_obs)
  for (int i = tid; i < D.n_hm; i += nt_thr) S[D.s_mh + i] = log(B[D.o_mh + i] * (om - B[1]));
  {
    const double* xz = B + D.o_xz;
    const double y = fmin(fmax(zob, xz[0]), xz[D.n_xz - 1]);
    const int j = bsearch_cell(xz, D.n_xz, y);
    const double u = (y - xz[j]) / (xz[j + 1] - xz[j]);
    const double* r0 = B + D.o_xi + (size_t)j * D.n_xr;
    const double* r1 = r0 + D.n_xr;
    for (int i = tid; i < D.n_xr; i += nt_thr) S[D.s_xi + i] = (1.0 - u) * r0[i] + u * r1[i];
  }
  __syncthreads();
  // Three chains of scalar work, a warp's first thread each.
  const double D_A = chis[0] / (1.0 + zob);
  if (tid == 0) {
    const double chi_o = chis[0];
    const double Rl = pow(D.sl_lob[sl] / 100.0, 0.2), R_excl = Rl * (1.0 + zob);
    // theta breakpoints (sp_detail::build_theta_grid, sigma_prj_t.hh:95-180):
    // the radii ascend, so the sorted list is a merge of theta_R with the
    // five others; those outside (0, theta_max] are left out and neighbours
    // closer than 1e-6 kept once.
    const int ra = D.r0[sl], nR = D.r0[sl + 1] - ra;
    const double th_lam = Rl * (1.0 + zob) / chi_o, th_ex = R_excl / chi_o;
    int top = nR - 1;
    while (top > 0 && isnan(D.radii[ra + top])) --top;
    const double t_min = D.radii[ra] / D_A, t_max = D.radii[ra + top] / D_A;
    const double th_max = fmax(D.R_max / D_A, 3.0 * t_max);
    const double lower = fmax(1.0e-8, 0.1 * fmin(th_ex, fmin(t_min, th_lam)));
    double sp[5] = {lower, th_ex, th_lam, 2.0 * th_lam, th_max};
    for (int a = 1; a < 5; ++a)
      for (int b = a; b > 0 && sp[b] < sp[b - 1]; --b) {
        const double v = sp[b];
        sp[b] = sp[b - 1];
        sp[b - 1] = v;
      }
    double* bd = S + D.s_bd;
    int n = 0;
    double back = 0.0, last = 0.0;  // last kept, last of the sorted list
    auto put = [&](double x) {
      if (n == 0 || x > back * (1.0 + 1.0e-6)) {
        bd[n++] = x;
        back = x;
      }
      last = x;
    };
    int is = 0, ir = 0;
    while (is < 5 || ir < nR) {
      const double tr = ir < nR ? D.radii[ra + ir] / D_A : 0.0;
      double x;
      if (ir >= nR || (is < 5 && sp[is] <= tr)) {
        x = sp[is++];
      } else {
        x = tr;
        ++ir;
      }
      if (!(isfinite(x) && x > 0.0 && x <= th_max)) continue;
      if (n == 0 && x > lower) put(lower);
      put(x);
    }
    if (n == 0) put(lower);
    if (last < th_max) put(th_max);
    n_bd_s = n;
  } else if (tid == 32) {
    const double Rl = pow(D.sl_lob[sl] / 100.0, 0.2), th_lam = Rl * (1.0 + zob) / chis[0];
    // b_sel asymptotes linear in z_obs (sigma_prj_frozen_t.hh:200-217)
    const double* bz = B + D.o_bzob;
    const int nzb = D.n_bzob, nlb = D.n_blob, lb = D.sl_lb[sl];
    int j = 0;
    while (j + 1 < nzb && bz[j + 1] < zob) ++j;
    const int j0 = j + 1 < nzb ? j : max(nzb - 2, 0), j1 = j + 1 < nzb ? j + 1 : nzb - 1;
    const double za = bz[j0], zb = bz[j1];
    const double f = zb > za ? fmin(fmax((zob - za) / (zb - za), 0.0), 1.0) : 0.0;
    const double* bs = B + D.o_bs;
    const double* bl = B + D.o_blg;
    sc[0] = (1.0 - f) * bs[j0 * nlb + lb] + f * bs[j1 * nlb + lb];
    sc[1] = (1.0 - f) * bl[j0 * nlb + lb] + f * bl[j1 * nlb + lb];
    sc[2] = 2.5 / th_lam;
    sc[3] = 0.5 * th_lam;
  } else if (tid == 64) {
    const double chi_o = chis[0];
    const double R_excl = pow(D.sl_lob[sl] / 100.0, 0.2) * (1.0 + zob);
    // line-of-sight ranges (sigma_prj_frozen_t.hh:380-455)
    const double dchi_dz = (chis[3] - chis[4]) / (2.0 * dz1);
    const double dz_ex = R_excl / dchi_dz;
    sc[4] = fmax(zob - dz_ex, D.zt_low);
    sc[5] = fmin(zob + dz_ex, D.zt_high);
    sc[6] = R_excl;
    sc[7] = chi_o - chis[1];
    sc[8] = chis[2] - chi_o;
    S[D.s_scal] = chi_o;
    S[D.s_scal + 1] = D_A;
    S[D.s_scal + 2] =
      B[7] != 0.0 ? interp1d_clamp(B + D.o_sz, B + D.o_sv, D.n_sci, zob) : 0.0;
  }
  __syncthreads();
  const double chi_o = chis[0], R_excl = sc[6];
  const int n_th = (n_bd_s - 1) * D.n_seg;
  const int n_f = R_excl < sc[7] ? D.n_zouter : 0, n_r = sc[5] > sc[4] ? D.n_zring : 0;
  const int n_b = R_excl < sc[8] ? D.n_zouter : 0, nz = n_f + n_r + n_b;
  for (int i = tid; i < D.nz + n_th; i += nt_thr) {
    if (i >= D.nz) {  // theta node
      const int t = i - D.nz, s = t / D.n_seg, q = t - s * D.n_seg;
      const double a = log(S[D.s_bd + s]), b = log(S[D.s_bd + s + 1]), hl = 0.5 * (b - a);
      const double th = exp(0.5 * (a + b) + hl * D.gl_seg[q]);
      S[D.s_th + t] = th;
      S[D.s_geom + t] = hl * D.gl_seg[D.n_seg + q] * th * 2.0 * kPiP * sin(th);
      S[D.s_bsel + t] = sc[0] + (sc[1] - sc[0]) * (1.0 / (1.0 + exp(-sc[2] * (th - sc[3]))));
      continue;
    }
    // z node: front wing (farthest first), ring, back wing
    double z, wz;
    if (i >= nz) {
      S[D.s_zc + i] = 0.0;
      continue;
    }
    if (i >= n_f && i < n_f + n_r) {
      const int q = i - n_f;
      const double hl = 0.5 * (sc[5] - sc[4]);
      z = 0.5 * (sc[4] + sc[5]) + hl * D.gl_ring[q];
      wz = hl * D.gl_ring[D.n_zring + q];
    } else {
      const bool fg = i < n_f;
      const int q = fg ? n_f - 1 - i : i - n_f - n_r;
      const double a = log(R_excl), b = log(fg ? sc[7] : sc[8]), hl = 0.5 * (b - a);
      const double dis = exp(0.5 * (a + b) + hl * D.gl_out[q]);
      const double target = fg ? chi_o - dis : chi_o + dis;
      // sigma_prj_frozen_t.hh:458-468; the cells of the two ends bracket the
      // one of the midpoint, so its search shrinks with the interval.
      double lo = 0.001, hi = 2.0;
      int c_lo = 0, c_hi = D.nd - 1;
      for (int it = 0; it < 40; ++it) {
        const double mid = 0.5 * (lo + hi), x = fmin(fmax(mid, dz[0]), dz[D.nd - 1]);
        int a = c_lo, b = c_hi;
        while (b > a + 1) {
          const int m = (a + b) >> 1;
          if (dz[m] > x)
            b = m;
          else
            a = m;
        }
        if (interp1d_cell(dz, B + D.o_dc, a, x) * h0 < target) {
          lo = mid;
          c_lo = a;
        } else {
          hi = mid;
          c_hi = a + 1;
        }
      }
      z = 0.5 * (lo + hi);
      wz = hl * D.gl_out[D.n_zouter + q] * dis / ((chi(z + dz1) - chi(z - dz1)) / (2.0 * dz1));
    }
    const double chz = chi(z);
    double dv;
    if (!dv_do_dz(dz, B + D.o_da, D.nd, om, B[2], B[3], h0, z, &dv)) {
      set_err(status, kDevDomain);
      dv = 0.0;
    }
    const double up = (z - zob) / interp1d_clamp(D.zk_z, D.zk_s, kZKernelNodes, z);
    const double wph = fabs(up) < 1.0 ? 1.0 - up * up : 0.0;
    S[D.s_z + i] = z;
    S[D.s_zc + i] = dv * (D.omega_z ? omega_z_des(z) : 1.0) * wz * wph;
    S[D.s_chi + i] = chz;
    // sp_detail::theta_excl_at_z (sigma_prj_t.hh:185-194)
    const double ce =
      (chz * chz + chi_o * chi_o - R_excl * R_excl) / (2.0 * chz * chi_o + 1.0e-30);
    S[D.s_thex + i] = ce >= 1.0 - 1.0e-12 ? 0.0 : acos(fmax(ce, -1.0));
  }
  if (tid == 0) nt_out[sl] = n_th;
  __syncthreads();
  // n and b at every z node of non-zero weight and, in the last item, at
  // z_obs: one warp a node, lanes over the masses.  A lane keeps the mass
  // cells of both tables over its warp's nodes, whose z cells the lanes find
  // side by side, one node each.
  const double *hz = B + D.o_hz, *bl = B + D.o_bl, *bz = B + D.o_bz;
  for (int i0 = warp; i0 <= D.nz; i0 += 32 * nw) {
    const int il = i0 + nw * lane;  // this lane's node
    double c_l = 0.0, z_l = zob, uh_l, ub_l;
    if (il == D.nz) {
      c_l = 1.0;
    } else if (il < D.nz) {
      c_l = S[D.s_zc + il];
      if (c_l != 0.0) z_l = S[D.s_z + il];
    }
    const int jh_l = clamp_cell(hz, D.n_hz, z_l, &uh_l), jb_l = clamp_cell(bz, D.n_bz, z_l, &ub_l);
    for (int k0 = 0; k0 < D.n_lnm; k0 += 32) {
      const int k = k0 + lane;
      const bool in = k < D.n_lnm;
      const double x = D.lnm_x[in ? k : 0], w = D.lnm_w[in ? k : 0];
      const double an = in ? D.anchor[k] : 0.0, f = B[5] * (x * kLog10e - kHmfPivot) + B[6];
      double th, tb;
      const int xh = clamp_cell(S + D.s_mh, D.n_hm, x, &th), xb = clamp_cell(bl, D.n_bl, x, &tb);
      for (int m = 0; m < 32 && i0 + nw * m <= D.nz; ++m) {
        const int i = i0 + nw * m, jh = __shfl_sync(0xffffffffu, jh_l, m);
        const int jb = __shfl_sync(0xffffffffu, jb_l, m);
        const double c = __shfl_sync(0xffffffffu, c_l, m), uh = __shfl_sync(0xffffffffu, uh_l, m);
        const double ub = __shfl_sync(0xffffffffu, ub_l, m);
        const bool anchor = i == D.nz;
        double num = 0.0;
        if (c == 0.0) {  // the reference skips these nodes entirely
          if (in) S[D.s_wz + (size_t)i * D.n_lnm + k] = 0.0;
        } else {
          const double n = bilinear_at(B + D.o_dn, D.n_hm, xh, jh, th, uh) * f;
          const double b = bilinear_at(B + D.o_bi, D.n_bl, xb, jb, tb, ub);
          num = an * n * b;
          if (in && anchor)
            S[D.s_wcl + k] = w * n * b;
          else if (in)
            S[D.s_wz + (size_t)i * D.n_lnm + k] = c * n * w;
        }
        for (int off = 16; off > 0; off >>= 1) num += __shfl_xor_sync(0xffffffffu, num, off);
        if (lane == 0) {  // the mass chunks in order
          double* to = anchor ? &sc[9] : &S[D.s_ab + i];
          *to = (k0 ? *to : 0.0) + num;
        }
      }
    }
    if (lane == 0 && i0 <= D.nz && (D.nz - i0) % nw == 0 && (D.nz - i0) / nw < 32)
      sc[9] += 1.0e-300;
  }
  __syncthreads();
  for (int i = tid; i < D.nz; i += nt_thr) {
    const double c = S[D.s_zc + i];
    S[D.s_ab + i] = c != 0.0 ? c * (S[D.s_ab + i] / sc[9]) : 0.0;
  }
  for (int k = tid; k < D.n_lnm; k += nt_thr) {
    double acc = 0.0;
    for (int i = 0; i < D.nz; ++i) acc += S[D.s_wz + (size_t)i * D.n_lnm + k];
    S[D.s_wrnd + k] = acc;
  }
  if (!D.cheb) return;
  __syncthreads();
  for (int i = warp; i < 2 * D.n_prof; i += nw) {  // both channels' weights on the nodes
    const double* v = S + (i < D.n_prof ? D.s_wrnd : D.s_wcl);
    const double* row = D.cheb + (size_t)(i < D.n_prof ? i : i - D.n_prof) * D.n_lnm;
    double acc = 0.0;
    for (int k = lane; k < D.n_lnm; k += 32) acc += row[k] * v[k];
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0) S[(i < D.n_prof ? D.s_pr : D.s_pc - D.n_prof) + i] = acc;
  }
}

// The clustered channel's weight g_theta b_sel Psi of every theta node: one
// warp a node, lanes over the z nodes.
__global__ void __launch_bounds__(256)
prj_psi_kernel(PrjDims D, const double* __restrict__ B, double* __restrict__ scratch,
               const int* __restrict__ nt)
{
  const int sl = blockIdx.y, lane = threadIdx.x & 31;
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= nt[sl]) return;
  double* S = scratch + (size_t)sl * D.scratch;
  const double th = S[D.s_th + t], ct = cos(th), co = S[D.s_scal];
  const double* xr = B + D.o_xr;
  const double* row = S + D.s_xi;
  double acc = 0.0;
  for (int u = lane; u < D.nz; u += 32) {
    if (S[D.s_zc + u] == 0.0 || th <= S[D.s_thex + u]) continue;
    const double cz = S[D.s_chi + u];
    const double dchi = sqrt(fmax(cz * cz + co * co - 2.0 * cz * co * ct, 0.0));
    const double r = fmin(fmax(dchi, xr[0]), xr[D.n_xr - 1]);
    const int i = bsearch_cell(xr, D.n_xr, r);
    const double f = (r - xr[i]) / (xr[i + 1] - xr[i]);
    acc += S[D.s_ab + u] * ((1.0 - f) * row[i] + f * row[i + 1]);
  }
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (lane == 0) S[D.s_wcl_th + t] = S[D.s_geom + t] * S[D.s_bsel + t] * acc;
}

// The mass contractions sum_M wrnd(M) DSigma_mis and sum_M w_M n b DSigma_mis
// of every (grid point, theta node): P[g][t] = (rnd, cl).  From the table,
// one warp a node, lanes over the masses.
__global__ void __launch_bounds__(256)
prj_profile_table_kernel(PrjDims D, PrjTable T, const double* __restrict__ scratch,
                         const int* __restrict__ nt, double2* __restrict__ P)
{
  const int g = blockIdx.y, sl = D.gp_slice[g], lane = threadIdx.x & 31;
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= nt[sl]) return;
  const double* S = scratch + (size_t)sl * D.scratch;
  const double R = D.gp_R[g], Rm = S[D.s_th + t] * S[D.s_scal + 1];
  double ar = 0.0, ac = 0.0;
  for (int k = lane; k < D.n_lnm; k += 32) {
    const double v = dsigma_single_table(T, R, Rm, D.lnm_x[k]);
    ar += S[D.s_wrnd + k] * v;
    ac += S[D.s_wcl + k] * v;
  }
  for (int off = 16; off > 0; off >>= 1) {
    ar += __shfl_xor_sync(0xffffffffu, ar, off);
    ac += __shfl_xor_sync(0xffffffffu, ac, off);
  }
  if (lane == 0) P[(size_t)g * D.nt_max + t] = make_double2(ar, ac);
}

// The ring averages with the closed-form profile, for rings that leave the
// polynomials' range; out of line: the rare path.
__device__ __noinline__ double2
ring_masses_closed(const PrjQuad& Q, const double* __restrict__ rule, int n, double R, double Rm,
                   int n_lnm, const double* __restrict__ w, const double* __restrict__ wc, int lane)
{
  double ar = 0.0, ac = 0.0;
  for (int k = 0; k < n_lnm; ++k) {
    const double q = Q.mass[k];
    double acc = 0.0;
    for (int t = lane; t < n; t += 32) {
      const double ct = rule[t], D2 = R * R + Rm * Rm - 2.0 * R * Rm * ct, a = R - Rm * ct;
      acc += rule[kRuleTot + t] * (2.0 * a * a / D2 - 1.0) / kPiP *
             NfwUnit<double>::dsigma(sqrt(D2 * q));
    }
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    ar += w[k] * Q.mass[n_lnm + k] * acc;
    ac += wc[k] * Q.mass[n_lnm + k] * acc;
  }
  return make_double2(ar, ac);
}

// One warp's ring average of NJ nodes a lane, for all masses, contracted with
// the mass weights w and wc: the mean
// tangential shear on the circle of radius R around the offset centre,
// (1/pi) int dt DSigma(d / r_s) (2 a^2 / d^2 - 1), d^2 = R^2 + Rm^2 -
// 2 R Rm cos t, a = R - Rm cos t.  The geometry is shared by the masses,
// which only scale d; eight masses (four at the end, where they suffice)
// accumulate side by side and are summed over the lanes by halving exchanges
// (nine 64-bit shuffles for eight sums).
template <int NJ>
__device__ __forceinline__ double2
ring_masses(const PrjQuad& Q, const double* __restrict__ rule, double R, double Rm, int n_lnm,
            const double* __restrict__ w, const double* __restrict__ wc, int lane)
{
  double D2[NJ], A[NJ], ar = 0.0, ac = 0.0;
  bool outside = false;
  const double s2 = R * R + Rm * Rm, c2 = 2.0 * R * Rm;
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const double ct = rule[lane + 32 * j], a = R - Rm * ct;
    D2[j] = s2 - c2 * ct;
    A[j] = rule[kRuleTot + lane + 32 * j] * (2.0 * a * a / D2[j] - 1.0) / kPiP;
  }
  auto group = [&](auto masses, int k0) {
    constexpr int U = decltype(masses)::value, S = 32 / U;  // a sum ends on S lanes
    double acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double q = __ldg(Q.mass + min(k0 + u, n_lnm - 1));
      acc[u] = 0.0;
#pragma unroll
      for (int j = 0; j < NJ; ++j) acc[u] += A[j] * nfw_dsigma_w(Q.nfw, D2[j] * q, outside);
    }
#pragma unroll
    for (int h = U / 2; h >= 1; h >>= 1) {
      const bool up = (lane & (S * h)) != 0;
#pragma unroll
      for (int u = 0; u < h; ++u) {
        const double send = up ? acc[u] : acc[u + h];
        acc[u] = (up ? acc[u + h] : acc[u]) + __shfl_xor_sync(0xffffffffu, send, S * h);
      }
    }
#pragma unroll
    for (int off = S / 2; off >= 1; off >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], off);
    const int k = k0 + lane / S;
    if (lane % S == 0 && k < n_lnm) {
      const double v = Q.mass[n_lnm + k] * acc[0];
      ar += w[k] * v;
      ac += wc[k] * v;
    }
  };
  int k0 = 0;
  for (; k0 + 4 < n_lnm; k0 += 8) group(std::integral_constant<int, 8>{}, k0);
  if (k0 < n_lnm) group(std::integral_constant<int, 4>{}, k0);
  if (__any_sync(0xffffffffu, outside))
    return ring_masses_closed(Q, rule, 32 * NJ, R, Rm, n_lnm, w, wc, lane);
  for (int off = 16; off >= 4; off >>= 1) {
    ar += __shfl_xor_sync(0xffffffffu, ar, off);
    ac += __shfl_xor_sync(0xffffffffu, ac, off);
  }
  return make_double2(ar, ac);
}

// The same contractions by quadrature, one warp per (grid point, theta
// node): the lanes take the ring's nodes, so the profile's table reads of a
// warp fall on few, neighbouring segments.  12 slices x 10 radii x ~130
// theta x 20 nodes (24 masses): 82 us, bound by those reads (L1); 98 us with
// a profile at every mass.
__global__ void __launch_bounds__(256, 3)
prj_profile_kernel(PrjDims D, PrjQuad Q, const double* __restrict__ scratch,
                   const int* __restrict__ nt, double2* __restrict__ P)
{
  const int g = blockIdx.y, sl = D.gp_slice[g], lane = threadIdx.x & 31;
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= nt[sl]) return;
  const double* S = scratch + (size_t)sl * D.scratch;
  const double R = D.gp_R[g], Rm = S[D.s_th + t] * S[D.s_scal + 1], lr = fabs(log(Rm / R));
  const double *w = S + D.s_pr, *wc = S + D.s_pc;
  double2 v;
  if (lr >= kRuleLn0)
    v = ring_masses<1>(Q, Q.rule, R, Rm, D.n_prof, w, wc, lane);
  else if (lr >= kRuleLn1)
    v = ring_masses<2>(Q, Q.rule + kRuleN0, R, Rm, D.n_prof, w, wc, lane);
  else if (lr >= kRuleLn2)
    v = ring_masses<4>(Q, Q.rule + kRuleN0 + kRuleN1, R, Rm, D.n_prof, w, wc, lane);
  else
    v = ring_masses<8>(Q, Q.rule + kRuleN0 + kRuleN1 + kRuleN2, R, Rm, D.n_prof, w, wc, lane);
  if (lane == 0) P[(size_t)g * D.nt_max + t] = v;
}

// The theta sums of one grid point; block 0 also copies the status word
// behind the results.
__global__ void __launch_bounds__(128)
prj_sum_kernel(PrjDims D, const double* __restrict__ B, const double* __restrict__ scratch,
               const int* __restrict__ nt, const double2* __restrict__ P,
               const int* __restrict__ status, double* __restrict__ out)
{
  __shared__ double red[128];
  const int g = blockIdx.x, sl = D.gp_slice[g];
  const double* S = scratch + (size_t)sl * D.scratch;
  const double2* Pg = P + (size_t)g * D.nt_max;
  double rnd = 0.0, cl = 0.0;
  for (int t = threadIdx.x; t < nt[sl]; t += blockDim.x) {
    const double2 v = Pg[t];
    rnd += S[D.s_geom + t] * v.x;
    cl += S[D.s_wcl_th + t] * v.y;
  }
  rnd = block_sum<128>(rnd, red) * B[0];  // the amplitude's Omega_M
  cl = block_sum<128>(cl, red) * B[0];
  if (threadIdx.x == 0) {
    const double tot = rnd + cl, s = S[D.s_scal + 2];
    double* o = out + (size_t)g * 9;
    o[0] = tot;
    o[1] = rnd;
    o[2] = cl;
    o[3] = o[6] = tot * s;
    o[4] = o[7] = rnd * s;
    o[5] = o[8] = cl * s;
    if (g == 0) *reinterpret_cast<int*>(out + (size_t)D.ngp * 9) = *status;
  }
}

}  // namespace

// Device and pinned buffers of the handle, grown on demand.
struct PrjBufs {
  DevBuf<double> d_const, d_quad, d_tab, d_blk, d_scratch, d_P, d_out;
  DevBuf<int> d_int, d_nt;
  double* h_stage = nullptr;
  size_t stage_cap = 0;
  ~PrjBufs()
  {
    if (h_stage) cudaFreeHost(h_stage);
  }
  int stage(size_t n)  // pinned doubles
  {
    if (n <= stage_cap) return Y3B_OK;
    if (h_stage) cudaFreeHost(h_stage);
    h_stage = nullptr;
    stage_cap = 0;
    Y3B_CUDA(cudaHostAlloc((void**)&h_stage, n * sizeof(double), cudaHostAllocDefault));
    stage_cap = n;
    return Y3B_OK;
  }
};

}  // namespace y3b

struct y3b_prj {
  y3b_prj_config cfg;
  std::vector<double> lob;                   // richness-bin centres
  std::vector<int> gp_lb;                    // per grid point
  std::vector<double> gp_zob, gp_R;
  std::vector<int> gp_slice;
  std::vector<int> sl_lb;                    // per slice (first-appearance order)
  std::vector<double> sl_zob;
  std::vector<std::vector<double>> sl_Rs;    // distinct radii, first-appearance order
  std::vector<double> lnm_x, lnm_w;
  int tab_lx = 0, tab_lxm = 0;               // shape of the miscentring table in bufs.d_tab
  y3b::PrjBufs bufs;
  cudaStream_t stream = nullptr;
  ~y3b_prj()
  {
    if (stream) cudaStreamDestroy(stream);
  }
};

namespace y3b {
namespace {

// cos(t) [kRuleTot] | weights [kRuleTot] of the ring rules, formed once per
// process.
const std::vector<double>&
ring_rules()
{
  static const std::vector<double> rules = [] {
    std::vector<double> q, w, th, wth;
    for (int m : {kRuleN0, kRuleN1, kRuleN2, kRuleN3}) {
      h_gl(0.0, kPiP, m, th, wth);
      for (double t : th) q.push_back(std::cos(t));
      w.insert(w.end(), wth.begin(), wth.end());
    }
    q.insert(q.end(), w.begin(), w.end());
    return q;
  }();
  return rules;
}

bool
prof_nodes(const y3b_prj_config& c)
{
  return c.n_lnm > kProfNodes && c.lnm_high > c.lnm_low && c.lnm_high - c.lnm_low <= kProfRange;
}

// The quadrature's constants on the device, once per handle: DeltaSigma
// polynomials | ring rules | 1 / r_s^2 and the amplitude 2 r_s delta_c rho_c
// 1e-12 of the mass nodes.
int
upload_quad(y3b_prj* h)
{
  std::vector<double> x = h->lnm_x, tilt(x.size(), 1.0);
  if (prof_nodes(h->cfg)) {
    x = cheb_rows(kProfNodes, h->cfg.lnm_low, h->cfg.lnm_high, {});
    tilt.clear();
    for (double v : x) tilt.push_back(std::exp(0.5 * (h->cfg.lnm_low + h->cfg.lnm_high) - v));
  }
  const int n = (int)x.size();
  const double* nfw = nfw_table_host();
  std::vector<double> q(nfw, nfw + kNfwSegs * kNfwCoef);
  q.insert(q.end(), ring_rules().begin(), ring_rules().end());
  const double delta_c =
    (200.0 * kConc * kConc * kConc / 3.0) / (std::log(1.0 + kConc) - kConc / (1.0 + kConc));
  std::vector<double> rs(n);
  for (int i = 0; i < n; ++i) {
    rs[i] = std::cbrt(3.0 * std::exp(x[i]) / (800.0 * kPiP * kRhoCrit)) / kConc;
    q.push_back(1.0 / (rs[i] * rs[i]));
  }
  for (int i = 0; i < n; ++i) q.push_back(2.0 * rs[i] * delta_c * kRhoCrit * 1e-12 * tilt[i]);
  y3b::DevBuf<double>& d = h->bufs.d_quad;
  Y3B_TRY(d.upload(q.data(), q.size(), h->stream));
  const int rc = cuda_status(cudaStreamSynchronize(h->stream), "upload of the ring rules");
  if (rc) d.reset();
  return rc;
}

// The handle's constants: mass nodes, weights and anchors w r_s (NFW_DSIGMA_MIS::
// r_s, nfw_dsigma_mis.hh:82-88), unit GL rules, the photo-z width table, the
// slices' centres and ascending radii, the grid points.
int
upload_const(y3b_prj* h)
{
  const y3b_prj_config& c = h->cfg;
  std::vector<double> q, x, w;
  auto put = [&](const std::vector<double>& v) { q.insert(q.end(), v.begin(), v.end()); };
  put(h->lnm_x);
  put(h->lnm_w);
  for (int i = 0; i < c.n_lnm; ++i)
    q.push_back(h->lnm_w[i] *
                (std::cbrt(3.0 * std::exp(h->lnm_x[i]) / (800.0 * kPiP * kRhoCrit)) / kConc));
  for (int n : {c.n_per_seg, c.n_zring, c.n_zouter}) {
    h_gl(-1.0, 1.0, n, x, w);
    put(x);
    put(w);
  }
  q.insert(q.end(), kZKernelZ, kZKernelZ + kZKernelNodes);
  q.insert(q.end(), kZKernelSigma, kZKernelSigma + kZKernelNodes);
  for (int lb : h->sl_lb) q.push_back(h->lob[lb]);
  put(h->sl_zob);
  std::vector<int> ints(h->sl_lb);
  int off = 0;
  for (const auto& Rs : h->sl_Rs) {
    std::vector<double> s(Rs);
    std::sort(s.begin(), s.end(),  // a NaN last: it never becomes a breakpoint
              [](double a, double b) { return std::isnan(b) ? !std::isnan(a) : a < b; });
    put(s);
    ints.push_back(off);
    off += (int)s.size();
  }
  ints.push_back(off);
  put(h->gp_R);
  if (prof_nodes(c)) {
    const std::vector<double> v = cheb_rows(kProfNodes, c.lnm_low, c.lnm_high, h->lnm_x);
    for (int j = 0; j < kProfNodes; ++j)
      for (int k = 0; k < c.n_lnm; ++k)
        q.push_back(v[kProfNodes + (size_t)j * c.n_lnm + k] *
                    std::exp(h->lnm_x[k] - 0.5 * (c.lnm_low + c.lnm_high)));
  }
  ints.insert(ints.end(), h->gp_slice.begin(), h->gp_slice.end());
  Y3B_TRY(h->bufs.d_const.upload(q.data(), q.size(), h->stream));
  Y3B_TRY(h->bufs.d_int.upload(ints.data(), ints.size(), h->stream));
  return cuda_status(cudaStreamSynchronize(h->stream), "upload of the handle's constants");
}

// Shapes and offsets of one call.
PrjDims
layout(const y3b_prj* h, const y3b_prj_sample& S)
{
  const y3b_prj_config& c = h->cfg;
  PrjDims D{};
  D.n_lnm = c.n_lnm;
  D.n_seg = c.n_per_seg;
  D.n_zring = c.n_zring;
  D.n_zouter = c.n_zouter;
  D.ngp = c.n_gp;
  D.nsl = (int)h->sl_lb.size();
  size_t n_radii = 0;
  for (const auto& Rs : h->sl_Rs) {
    D.nR_max = std::max(D.nR_max, (int)Rs.size());
    n_radii += Rs.size();
  }
  D.nt_max = (D.nR_max + 6) * c.n_per_seg;  // five more breakpoints, and the two ends
  D.nz = c.n_zring + 2 * c.n_zouter;
  D.zt_low = c.zt_low;
  D.zt_high = c.zt_high;
  D.R_max = c.R_max_cMpch;
  D.omega_z = c.include_omega_z;
  D.n_hm = S.t.n_hm;
  D.n_hz = S.t.n_hz;
  D.nd = S.t.n_dist;
  D.n_sci = S.t.n_sci;
  D.n_bl = S.n_hl;
  D.n_bz = S.n_hz;
  D.n_xr = S.n_xr;
  D.n_xz = S.n_xz;
  D.n_blob = S.n_blob;
  D.n_bzob = S.n_bzob;
  long o = 8;
  auto blk = [&](long& at, long n) { at = o, o += n; };
  blk(D.o_mh, D.n_hm);
  blk(D.o_hz, D.n_hz);
  blk(D.o_dn, (long)D.n_hz * D.n_hm);
  blk(D.o_dz, D.nd);
  blk(D.o_da, D.nd);
  blk(D.o_dc, D.nd);
  blk(D.o_sz, std::max(D.n_sci, 0));
  blk(D.o_sv, std::max(D.n_sci, 0));
  blk(D.o_bl, D.n_bl);
  blk(D.o_bz, D.n_bz);
  blk(D.o_bi, (long)D.n_bl * D.n_bz);
  blk(D.o_xr, D.n_xr);
  blk(D.o_xz, D.n_xz);
  blk(D.o_xi, (long)D.n_xr * D.n_xz);
  blk(D.o_bzob, D.n_bzob);
  blk(D.o_bs, (long)D.n_bzob * D.n_blob);
  blk(D.o_blg, (long)D.n_bzob * D.n_blob);
  o = 0;
  blk(D.s_mh, D.n_hm);
  blk(D.s_xi, D.n_xr);
  blk(D.s_bd, D.nR_max + 7);
  blk(D.s_th, D.nt_max);
  blk(D.s_geom, D.nt_max);
  blk(D.s_bsel, D.nt_max);
  blk(D.s_wcl_th, D.nt_max);
  for (long* at : {&D.s_z, &D.s_zc, &D.s_chi, &D.s_thex, &D.s_ab}) blk(*at, D.nz);
  blk(D.s_wz, (long)D.nz * D.n_lnm);
  blk(D.s_wrnd, D.n_lnm);
  blk(D.s_wcl, D.n_lnm);
  D.n_prof = prof_nodes(c) ? kProfNodes : c.n_lnm;
  D.s_pr = D.s_wrnd;
  D.s_pc = D.s_wcl;
  if (prof_nodes(c)) {
    blk(D.s_pr, D.n_prof);
    blk(D.s_pc, D.n_prof);
  }
  blk(D.s_scal, 4);
  D.scratch = o;
  const double* q = h->bufs.d_const.get();
  auto take = [&](size_t n) {
    const double* at = q;
    q += n;
    return at;
  };
  D.lnm_x = take(c.n_lnm);
  D.lnm_w = take(c.n_lnm);
  D.anchor = take(c.n_lnm);
  D.gl_seg = take(2 * (size_t)c.n_per_seg);
  D.gl_ring = take(2 * (size_t)c.n_zring);
  D.gl_out = take(2 * (size_t)c.n_zouter);
  D.zk_z = take(kZKernelNodes);
  D.zk_s = take(kZKernelNodes);
  D.sl_lob = take(D.nsl);
  D.sl_zob = take(D.nsl);
  D.radii = take(n_radii);
  D.gp_R = take(c.n_gp);
  D.cheb = prof_nodes(c) ? take((size_t)kProfNodes * c.n_lnm) : nullptr;
  D.sl_lb = h->bufs.d_int.get();
  D.r0 = D.sl_lb + D.nsl;
  D.gp_slice = D.r0 + D.nsl + 1;
  return D;
}

}  // namespace
}  // namespace y3b

extern "C" int
y3b_prj_create(const y3b_prj_config* cfg, y3b_prj** out)
{
  using namespace y3b;
  clear_error();
  if (!cfg || !out || cfg->n_gp < 1 || cfg->n_gp > 65535 || !cfg->lambda_bin || !cfg->zo_low ||
      !cfg->zo_high ||
      !cfg->radii || cfg->n_lnm < 1 || cfg->n_per_seg < 1 || cfg->n_zring < 1 ||
      cfg->n_zouter < 1 || !(cfg->zt_high > cfg->zt_low) || !(cfg->lnm_high > cfg->lnm_low)) {
    set_error("y3b_prj_create: invalid configuration (1..65535 grid points, node counts >= 1, "
              "ordered bounds)");
    return Y3B_ERR_INVALID;
  }
  *out = nullptr;
  Y3B_TRY(require_device());
  y3b_prj* h = new (std::nothrow) y3b_prj();
  if (!h) return Y3B_ERR_NOMEM;
  h->cfg = *cfg;
  if (cfg->lob_centers && cfg->n_lob > 0)
    h->lob.assign(cfg->lob_centers, cfg->lob_centers + cfg->n_lob);
  else
    h->lob = {25.0, 37.5, 52.5, 130.0};  // sp_detail::default_lob_centers
  for (int i = 0; i < cfg->n_gp; ++i) {
    const int lb = cfg->lambda_bin[i];
    if (lb < 0 || lb >= (int)h->lob.size()) {
      set_error("y3b_prj_create: lambda_bin %d outside lob_centers", lb);
      delete h;
      return Y3B_ERR_INVALID;
    }
    const double zob = 0.5 * (cfg->zo_low[i] + cfg->zo_high[i]), R = cfg->radii[i];
    int found = -1;  // the slice registry of sigma_prj_frozen_t.hh:81-107
    for (size_t k = 0; k < h->sl_lb.size(); ++k)
      if (h->sl_lb[k] == lb && std::abs(h->sl_zob[k] - zob) < 1e-12) {
        found = (int)k;
        break;
      }
    if (found < 0) {
      h->sl_lb.push_back(lb);
      h->sl_zob.push_back(zob);
      h->sl_Rs.emplace_back();
      found = (int)h->sl_lb.size() - 1;
    }
    auto& Rs = h->sl_Rs[found];
    bool have = false;
    for (double x : Rs) have |= std::abs(x - R) < 1e-12;
    if (!have) Rs.push_back(R);
    h->gp_lb.push_back(lb);
    h->gp_zob.push_back(zob);
    h->gp_R.push_back(R);
    h->gp_slice.push_back(found);
  }
  h_gl(cfg->lnm_low, cfg->lnm_high, cfg->n_lnm, h->lnm_x, h->lnm_w);
  int rc = cuda_status(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking),
                       "cudaStreamCreate");
  if (!rc) rc = upload_const(h);
  if (rc) {
    delete h;
    return rc;
  }
  *out = h;
  return Y3B_OK;
}

extern "C" void
y3b_prj_destroy(y3b_prj* h)
{
  delete h;
}

extern "C" int
y3b_prj_set_mis_table(y3b_prj* h, int n_lx, const double* logx, int n_lxm,
                      const double* logxmis, const double* log_tab)
{
  using namespace y3b;
  clear_error();
  if (!h) return Y3B_ERR_INVALID;
  if (n_lx == 0) {
    h->tab_lx = h->tab_lxm = 0;
    return Y3B_OK;
  }
  if (n_lx < 2 || n_lxm < 2 || !logx || !logxmis || !log_tab) {
    set_error("y3b_prj_set_mis_table: need at least 2 x 2 nodes and three arrays");
    return Y3B_ERR_INVALID;
  }
  for (size_t i = 0; i < (size_t)n_lx * n_lxm; ++i)
    if (!std::isfinite(log_tab[i])) {
      set_error("y3b_prj_set_mis_table: non-finite table entry");
      return Y3B_ERR_DOMAIN;
    }
  h->tab_lx = h->tab_lxm = 0;
  std::vector<double> tab(logx, logx + n_lx);
  tab.insert(tab.end(), logxmis, logxmis + n_lxm);
  tab.insert(tab.end(), log_tab, log_tab + (size_t)n_lx * n_lxm);
  Y3B_TRY(h->bufs.d_tab.upload(tab.data(), tab.size(), h->stream));
  Y3B_CUDA(cudaStreamSynchronize(h->stream));
  h->tab_lx = n_lx;
  h->tab_lxm = n_lxm;
  return Y3B_OK;
}

extern "C" int
y3b_prj_eval(y3b_prj* h, const y3b_prj_sample* S, double* out)
{
  using namespace y3b;
  clear_error();
  if (!h || !S || !out || !S->dist_dc || S->t.n_dist < 2 || S->t.n_hm < 2 ||
      S->t.n_hz < 2 || S->n_hl < 2 || S->n_hz < 2 || S->n_xr < 2 || S->n_xz < 2 ||
      S->n_blob < 1 || S->n_bzob < 1 || !S->bsel_lob || !S->bsel_zob || !S->b_small ||
      !S->b_large) {
    set_error("y3b_prj_eval: incomplete sample (tables of at least two nodes each)");
    return Y3B_ERR_INVALID;
  }
  const y3b_tables& t = S->t;
  for (int lb : h->sl_lb)
    if (lb >= S->n_blob) {
      set_error("y3b_prj_eval: b_sel_marginalised has %d richness bins, bin %d requested",
                S->n_blob, lb);
      return Y3B_ERR_INVALID;
    }
  const PrjDims D = layout(h, *S);
  cudaStream_t s = h->stream;
  PrjBufs& B = h->bufs;  // kept by the handle: no allocation after the first call
  const bool table = h->tab_lx > 0;
  if (!table && !B.d_quad.get()) Y3B_TRY(upload_quad(h));
  // The sample's block, with the status word (zero) behind it.
  const size_t blk = (size_t)D.o_blg + (size_t)D.n_bzob * D.n_blob, n_out = (size_t)D.ngp * 9 + 1;
  Y3B_TRY(B.stage(blk + 1 + n_out));
  Y3B_TRY(B.d_blk.alloc(blk + 1));
  Y3B_TRY(B.d_scratch.alloc((size_t)D.nsl * D.scratch));
  Y3B_TRY(B.d_nt.alloc(D.nsl));
  Y3B_TRY(B.d_P.alloc(2 * (size_t)D.ngp * D.nt_max));
  Y3B_TRY(B.d_out.alloc(n_out));
  double* b = B.h_stage;
  const double sc[8] = {S->cosmo.om, S->cosmo.onu, S->cosmo.ol, S->cosmo.ok, S->cosmo.h0,
                        S->cosmo.hmf_s, S->cosmo.hmf_q, t.n_sci > 1 ? 1.0 : 0.0};
  std::memcpy(b, sc, sizeof sc);
  auto put = [&](long at, const double* v, size_t n) {
    if (n) std::memcpy(b + at, v, n * sizeof(double));
  };
  put(D.o_mh, t.hmf_m_h, D.n_hm);
  put(D.o_hz, t.hmf_z, D.n_hz);
  put(D.o_dn, t.dndlnmh, (size_t)D.n_hz * D.n_hm);
  put(D.o_dz, t.dist_z, D.nd);
  put(D.o_da, t.dist_da, D.nd);
  put(D.o_dc, S->dist_dc, D.nd);
  if (t.n_sci > 1) {
    put(D.o_sz, t.sci_z, D.n_sci);
    put(D.o_sv, t.sci_val, D.n_sci);
  }
  put(D.o_bl, S->halo_lnM, D.n_bl);
  put(D.o_bz, S->halo_z, D.n_bz);
  put(D.o_bi, S->bias, (size_t)D.n_bl * D.n_bz);
  put(D.o_xr, S->xi_r, D.n_xr);
  put(D.o_xz, S->xi_z, D.n_xz);
  put(D.o_xi, S->xi_nl, (size_t)D.n_xr * D.n_xz);
  put(D.o_bzob, S->bsel_zob, D.n_bzob);
  put(D.o_bs, S->b_small, (size_t)D.n_bzob * D.n_blob);
  put(D.o_blg, S->b_large, (size_t)D.n_bzob * D.n_blob);
  b[blk] = 0.0;
  Y3B_CUDA(
    cudaMemcpyAsync(B.d_blk.get(), b, (blk + 1) * sizeof(double), cudaMemcpyHostToDevice, s));
  int* status = reinterpret_cast<int*>(B.d_blk.get() + blk);
  double2* P = reinterpret_cast<double2*>(B.d_P.get());
  const dim3 per_theta((D.nt_max + 7) / 8, D.nsl), per_gp((D.nt_max + 7) / 8, D.ngp);
  prj_slice_kernel<<<D.nsl, kSliceThreads, 0, s>>>(D, B.d_blk.get(), B.d_scratch.get(),
                                                   B.d_nt.get(), status);
  count_launch();
  Y3B_CUDA(cudaGetLastError());
  prj_psi_kernel<<<per_theta, 256, 0, s>>>(D, B.d_blk.get(), B.d_scratch.get(), B.d_nt.get());
  count_launch();
  Y3B_CUDA(cudaGetLastError());
  if (table) {
    const double* tb = B.d_tab.get();
    const PrjTable T{h->tab_lx, h->tab_lxm, tb, tb + h->tab_lx, tb + h->tab_lx + h->tab_lxm};
    prj_profile_table_kernel<<<per_gp, 256, 0, s>>>(D, T, B.d_scratch.get(), B.d_nt.get(), P);
  } else {
    const double* qd = B.d_quad.get();
    const PrjQuad Q{qd + kNfwSegs * kNfwCoef, qd + kNfwSegs * kNfwCoef + 2 * kRuleTot, qd};
    prj_profile_kernel<<<per_gp, 256, 0, s>>>(D, Q, B.d_scratch.get(), B.d_nt.get(), P);
  }
  count_launch();
  Y3B_CUDA(cudaGetLastError());
  prj_sum_kernel<<<D.ngp, 128, 0, s>>>(D, B.d_blk.get(), B.d_scratch.get(), B.d_nt.get(), P,
                                       status, B.d_out.get());
  count_launch();
  Y3B_CUDA(cudaGetLastError());
  double* ho = B.h_stage + blk + 1;
  Y3B_CUDA(cudaMemcpyAsync(ho, B.d_out.get(), n_out * sizeof(double), cudaMemcpyDeviceToHost, s));
  Y3B_CUDA(cudaStreamSynchronize(s));
  int st;
  std::memcpy(&st, ho + n_out - 1, sizeof st);
  if (st == kDevDomain) {
    set_error("argument out of range in Interp1D (a line-of-sight z node outside distances/z)");
    return Y3B_ERR_DOMAIN;
  }
  if (st != kDevOk) return device_status_rc(st);
  std::memcpy(out, ho, (n_out - 1) * sizeof(double));
  return Y3B_OK;
}
