// ref_modules.cu -- reference-compatible FP64 kernels behind the CosmoSIS
// module boundary:
//   * y3b_sel_function   sel_function.py:555-615 (S_stack producer)
//   * y3b_selgl_*        SelGLCore / NumCountsSelGL / Shear1hMisSelGL,
//                        src/models/n_operator_sel_gl_t.hh:75-361
//   * y3b_sigma_crit_inv average_sigma_crit_inv.py:40-58
//   * y3b_nfw_mis        NFW_DSIGMA_MIS / NFW_SIGMA_MIS operator()
// All arithmetic is FP64 so the module outputs track the reference chain to
// <= 1e-8 relative.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include <cuda.h>

#include "common.cuh"
#include "host_common.h"
#include "mis_quad.cuh"

namespace y3b {

// ---------------------------------------------------------------------------
// GL nodes on [a,b]: one thread per node pair.
__global__ void
gl_nodes_kernel(double a, double b, int n, double* xs, double* ws)
{
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < (n + 1) / 2) gl_node_pair(a, b, n, i, xs, ws);
}

int
gl_nodes_device(double a, double b, int n, double* xs, double* ws, cudaStream_t s)
{
  int pairs = (n + 1) / 2;
  gl_nodes_kernel<<<(pairs + 127) / 128, 128, 0, s>>>(a, b, n, xs, ws);
  count_launch();
  return cuda_status(cudaGetLastError(), "gl_nodes_kernel");
}

// ---------------------------------------------------------------------------
// sel_function: one warp per (lnM, z) cell; lanes stride over the N_q GL
// lambda_t nodes of the cell's bracket (sel_function.py:516-547), evaluate the
// MOR density, the EMG CDF at the unique edges (195-226) and accumulate
// W_k (CDF[hi] - CDF[lo]) P per distinct edge pair; a fixed xor-tree warp
// reduction makes the sum order independent of scheduling.
constexpr int kMaxEdges = 32;
constexpr int kMaxPairs = 32;

struct SelFuncArgs {
  int n_lnm, n_z, n_q, n_bins, n_edges, n_pairs;
  double lnm_low, lnm_high, zt_low, zt_high;
  int mor_kind;
  double mor[8];
  int n_plob;
  const double* plob_z;
  const double* plob_coef;
  const double* edges;       // [n_edges]
  const int* pair_lo;        // [n_pairs] edge index
  const int* pair_hi;
  const int* bin_pair;       // [n_bins] -> pair
  const double* zob_min;     // [n_bins]
  const double* zob_max;
  const double* sigma_z;
  const double* gl_t;        // [n_q] on [-1,1]
  const double* gl_w;
  double* lnm_out;
  double* z_out;
  double* S_out;             // [n_bins][n_z][n_lnm]
};

__device__ __forceinline__ double
hod_mu_sat(double M, double z, const double* hod)
{
  double Mmin = pow(10.0, hod[0]), M1 = pow(10.0, hod[1]);
  double dM1 = M1 - Mmin;
  if (dM1 <= 0.0) return 0.0;
  double dM = fmax(M - Mmin, 0.0);
  double base = dM > 0.0 ? dM / dM1 : 0.0;
  if (!(base > 0.0)) return 0.0;
  return pow(base, hod[2]) * pow((1.0 + z) / (1.0 + hod[5]), hod[3]);
}

// P_HOD(ltr | M, z): sel_function.py:295-343.
__device__ __forceinline__ double
hod_density(double ltr, double M, double ms, double lcentral, const double* hod)
{
  double delta = (hod[4] * ms) * (hod[4] * ms);
  double nu = ms + delta;
  double density;
  if (ms <= 1e-8) {
    double t = (ltr - lcentral) / 1.0e-3;
    density = exp(-0.5 * t * t) / (kSqrt2Pi * 1.0e-3);
  } else {
    double x = ltr - lcentral + delta;
    density = x > 0.0 ? exp(-nu + (x - 1.0) * log(fmax(nu, 1e-300)) - lgamma(x)) : 0.0;
  }
  if (ltr < 0.0 || ltr < lcentral) density = 0.0;
  return density;
}

// CHAIN: the distinct richness bins are consecutive edges, pair p = edges
// (p, p + 1), at most kChainEdges edges (the wall grids of the configs): the
// CDF differences and sums then stay in registers; other layouts index
// per-thread arrays in local memory.
constexpr int kChainEdges = 9;

template <bool CHAIN>
__global__ void __launch_bounds__(128, 6)
sel_function_kernel(SelFuncArgs a)
{
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int n_cells = a.n_lnm * a.n_z;
  if (warp >= n_cells) return;
  const int m = warp / a.n_z;  // lnM index
  const int j = warp % a.n_z;  // z index
  const double lnM = a.n_lnm > 1 ? a.lnm_low + (a.lnm_high - a.lnm_low) * m / (a.n_lnm - 1)
                                 : a.lnm_low;
  const double z = a.n_z > 1 ? a.zt_low + (a.zt_high - a.zt_low) * j / (a.n_z - 1) : a.zt_low;
  const double M = exp(lnM);
  if (lane == 0) {
    if (j == 0) a.lnm_out[m] = lnM;
    if (m == 0) a.z_out[j] = z;
  }
  // Bracket (per cell).
  double lo, hi, mu_ln = 0.0, D = 1.0, ms = 0.0, lcentral = 0.0;
  if (a.mor_kind == Y3B_MOR_HOD) {
    ms = hod_mu_sat(M, z, a.mor);
    lcentral = (M >= pow(10.0, a.mor[0])) ? 1.0 : 0.0;
    double mu_eff = lcentral + ms;
    double sig_eff = sqrt(fmax(ms + (a.mor[4] * ms) * (a.mor[4] * ms), 0.0));
    lo = fmax(0.0, mu_eff - 6.0 * sig_eff);
    hi = mu_eff + 6.0 * sig_eff;
  } else {
    mu_ln = a.mor[0] + a.mor[1] * (lnM - log(a.mor[4])) + a.mor[2] * log1p(z);
    lo = fmax(a.mor[5], exp(mu_ln - 6.0 * a.mor[3]));
    hi = fmin(a.mor[6], exp(mu_ln + 6.0 * a.mor[3]));
    D = phi_diff((log(a.mor[5]) - mu_ln) / a.mor[3], (log(a.mor[6]) - mu_ln) / a.mor[3]);
  }
  const bool degenerate = !(hi > lo);
  const double half = 0.5 * (hi - lo), mid = 0.5 * (hi + lo);
  // The eight EMG coefficients depend on z alone: one lane each.
  const double cl =
    interp1d_clamp(a.plob_z, a.plob_coef + (lane & 7) * a.n_plob, a.n_plob, z);
  double c[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) c[k] = __shfl_sync(0xffffffffu, cl, k);

  double acc[CHAIN ? kChainEdges - 1 : kMaxPairs];
#pragma unroll
  for (int p = 0; p < (CHAIN ? kChainEdges - 1 : kMaxPairs); ++p) acc[p] = 0.0;
  for (int t = lane; t < a.n_q && !degenerate; t += 32) {
    double ltr = mid + half * a.gl_t[t];
    double W = half * a.gl_w[t];
    double P;
    if (a.mor_kind == Y3B_MOR_HOD) {
      P = hod_density(ltr, M, ms, lcentral, a.mor);
    } else {
      double d = (log(ltr) - mu_ln) / a.mor[3];
      P = exp(-0.5 * d * d) / (kSqrt2Pi * a.mor[3] * ltr * D);
    }
    double mu, sg, tau, fp;
    plob_from_coef(c, ltr, &mu, &sg, &tau, &fp);
    if constexpr (CHAIN) {
      const double WP = W * P;
      double prev = cdf_lob(a.edges[0], mu, sg, tau, fp);
#pragma unroll
      for (int e = 1; e < kChainEdges; ++e) {
        if (e < a.n_edges) {
          const double v = cdf_lob(a.edges[e], mu, sg, tau, fp);
          acc[e - 1] += WP * (v - prev);
          prev = v;
        }
      }
    } else {
      double cdf[kMaxEdges];
      for (int e = 0; e < a.n_edges; ++e) cdf[e] = cdf_lob(a.edges[e], mu, sg, tau, fp);
      for (int p = 0; p < a.n_pairs; ++p)
        acc[p] += W * (cdf[a.pair_hi[p]] - cdf[a.pair_lo[p]]) * P;
    }
  }
#pragma unroll
  for (int p = 0; p < (CHAIN ? kChainEdges - 1 : kMaxPairs); ++p) {
    if (p >= a.n_pairs) break;
    double v = acc[p];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    acc[p] = v;
  }
  // One bin a lane.
  for (int k = lane; k < a.n_bins; k += 32) {
    double Si = 0.0;
#pragma unroll
    for (int p = 0; p < (CHAIN ? kChainEdges - 1 : kMaxPairs); ++p)
      if (p < a.n_pairs && p == a.bin_pair[k]) Si = acc[p];
    if (degenerate) Si = 0.0;
    const double Kj = phi_cdf((a.zob_max[k] - z) / a.sigma_z[k]) -
                      phi_cdf((a.zob_min[k] - z) / a.sigma_z[k]);
    a.S_out[((size_t)k * a.n_z + j) * a.n_lnm + m] = Si * Kj;
  }
}

// Chained bins (see above)?
static bool
chained(const std::vector<int>& lo, const std::vector<int>& hi, size_t n_edges)
{
  if (n_edges > (size_t)kChainEdges || lo.size() + 1 != n_edges) return false;
  for (size_t p = 0; p < lo.size(); ++p)
    if (lo[p] != (int)p || hi[p] != (int)p + 1) return false;
  return true;
}

static int
launch_sel_function(const SelFuncArgs& a, bool chain, cudaStream_t s)
{
  const long long warps = (long long)a.n_lnm * a.n_z;
  const int blocks = (int)((warps * 32 + 127) / 128);
  if (chain)
    sel_function_kernel<true><<<blocks, 128, 0, s>>>(a);
  else
    sel_function_kernel<false><<<blocks, 128, 0, s>>>(a);
  count_launch();
  return cuda_status(cudaGetLastError(), "sel_function_kernel");
}

}  // namespace y3b

namespace y3b {

constexpr int kNoAllocMaxQ = 1024;      // N_q
constexpr int kNoAllocMaxBins = 256;    // bins
constexpr int kNoAllocMaxPlob = 256;    // projection-table z nodes
constexpr size_t kNoAllocScratchDoubles =
  2 * kNoAllocMaxQ + kMaxEdges + 3 * kNoAllocMaxBins + 9 * kNoAllocMaxPlob +
  (2 * kMaxPairs + kNoAllocMaxBins);    // last term holds the int tables
static __device__ __align__(256) double g_selfunc_scratch[kNoAllocScratchDoubles];

// Device workspace of y3b_sel_function (inputs, GL rule, results): 2 MiB hold
// a 12-bin table of 192 x 64 cells and more.  Allocating and freeing 1.2 MB a
// call took 0.6 ms, at times tens of ms; one call at a time uses the array
// (g_selfunc_mu), an overlapping or larger one allocates its own.
constexpr size_t kSelFuncWork = 262144;  // doubles
static __device__ __align__(256) double g_selfunc_work[kSelFuncWork];
static std::mutex g_selfunc_mu;

// Device address of g_selfunc_scratch, looked up once per device context
// (host code may not use the symbol itself: it names a host-side stand-in).
// The address belongs to the context the module image was loaded into: a
// caller that resets the device gets a new context, in which the array lives
// elsewhere, so the cache is keyed by the context's unique id and the lookup
// is repeated for a new one.
static std::mutex g_scratch_mu;
static void* g_scratch_addr[128];
static void* g_work_addr[128];
static unsigned long long g_scratch_ctx[128];

// Unique id of the calling thread's current context (0 if it cannot be
// read, in which case the address is looked up on every call).  The driver
// entry points are fetched through the runtime: the library links no
// driver-API import.
static unsigned long long
current_context_id()
{
  using GetCurrentFn = CUresult (*)(CUcontext*);
  using GetIdFn = CUresult (*)(CUcontext, unsigned long long*);
  static GetCurrentFn get_current = nullptr;
  static GetIdFn get_id = nullptr;
  static bool resolved = false;
  if (!resolved) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<GetCurrentFn>(f);
    f = nullptr;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<GetIdFn>(f);
    resolved = true;
  }
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || !ctx ||
      get_id(ctx, &id) != CUDA_SUCCESS)
    return 0;
  return id;
}

static int
scratch_address(double** out, double** work = nullptr)
{
  int dev = 0;
  Y3B_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 128) {
    set_error("y3b_sel_function_noalloc: device index %d out of range", dev);
    return Y3B_ERR_INVALID;
  }
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  const unsigned long long ctx = current_context_id();
  if (!g_scratch_addr[dev] || ctx == 0 || ctx != g_scratch_ctx[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_selfunc_scratch);
    if (e != cudaSuccess || !p) {
      set_error("cudaGetSymbolAddress(g_selfunc_scratch): %s", cudaGetErrorString(e));
      return Y3B_ERR_CUDA;
    }
    void* w = nullptr;
    Y3B_CUDA(cudaGetSymbolAddress(&w, g_selfunc_work));
    g_work_addr[dev] = w;
    g_scratch_addr[dev] = p;
    // The lookup made the device's context current if it was not yet.
    g_scratch_ctx[dev] = ctx ? ctx : current_context_id();
  }
  *out = static_cast<double*>(g_scratch_addr[dev]);
  if (work) *work = static_cast<double*>(g_work_addr[dev]);
  return Y3B_OK;
}

}  // namespace y3b

using namespace y3b;

extern "C" int
y3b_sel_function(const y3b_selfunc_config* cfg, const y3b_mor* mor,
                 const y3b_plob* plob, double* lnm_out, double* z_out, double* S_out)
{
  clear_error();
  if (!cfg || !mor || !plob || !lnm_out || !z_out || !S_out) {
    set_error("y3b_sel_function: null argument");
    return Y3B_ERR_INVALID;
  }
  if (cfg->n_bins <= 0 || cfg->n_lnm <= 0 || cfg->n_z <= 0 || cfg->n_q <= 0 ||
      plob->n < 1 || (mor->kind != Y3B_MOR_HOD && mor->kind != Y3B_MOR_LOGNORMAL)) {
    set_error("y3b_sel_function: invalid sizes or MOR kind");
    return Y3B_ERR_INVALID;
  }
  Y3B_TRY(require_device());
  const int nb = cfg->n_bins;
  // Unique sorted edges and per-bin edge pairs (np.unique + searchsorted,
  // sel_function.py:550-552, 592-599).
  std::vector<double> edges;
  for (int k = 0; k < nb; ++k) {
    edges.push_back(cfg->lam_min[k]);
    edges.push_back(cfg->lam_max[k]);
  }
  std::sort(edges.begin(), edges.end());
  edges.erase(std::unique(edges.begin(), edges.end()), edges.end());
  if ((int)edges.size() > kMaxEdges) {
    set_error("y3b_sel_function: more than %d unique richness edges", kMaxEdges);
    return Y3B_ERR_UNSUPPORTED;
  }
  std::vector<int> plo, phi_, bin_pair(nb);
  for (int k = 0; k < nb; ++k) {
    int lo = int(std::lower_bound(edges.begin(), edges.end(), cfg->lam_min[k]) - edges.begin());
    int hi = int(std::lower_bound(edges.begin(), edges.end(), cfg->lam_max[k]) - edges.begin());
    int p = 0;
    for (; p < (int)plo.size(); ++p)
      if (plo[p] == lo && phi_[p] == hi) break;
    if (p == (int)plo.size()) {
      plo.push_back(lo);
      phi_.push_back(hi);
    }
    bin_pair[k] = p;
  }
  if ((int)plo.size() > kMaxPairs) {
    set_error("y3b_sel_function: more than %d distinct richness bins", kMaxPairs);
    return Y3B_ERR_UNSUPPORTED;
  }
  cudaStream_t s = 0;
  // The inputs (copied at once) | GL rule | lnM | z | S.
  const size_t ne = edges.size(), np = plob->n, nS = (size_t)nb * cfg->n_z * cfg->n_lnm;
  std::vector<double> in(edges);
  in.insert(in.end(), cfg->zob_min, cfg->zob_min + nb);
  in.insert(in.end(), cfg->zob_max, cfg->zob_max + nb);
  in.insert(in.end(), cfg->sigma_z, cfg->sigma_z + nb);
  in.insert(in.end(), plob->z, plob->z + np);
  in.insert(in.end(), plob->coef, plob->coef + 8 * np);
  std::vector<int> ints(plo);
  ints.insert(ints.end(), phi_.begin(), phi_.end());
  ints.insert(ints.end(), bin_pair.begin(), bin_pair.end());
  const size_t n_in = in.size();
  in.resize(n_in + (ints.size() + 1) / 2);
  std::memcpy(in.data() + n_in, ints.data(), ints.size() * sizeof(int));
  const size_t need = in.size() + 2 * (size_t)cfg->n_q + cfg->n_lnm + cfg->n_z + nS;
  std::unique_lock<std::mutex> lock(g_selfunc_mu, std::defer_lock);
  DevBuf<double> own;
  double *dev = nullptr, *unused = nullptr;
  if (need <= kSelFuncWork && lock.try_lock()) {
    Y3B_TRY(scratch_address(&unused, &dev));
  } else {
    Y3B_TRY(own.alloc(need));
    dev = own.get();
  }
  Y3B_CUDA(cudaMemcpyAsync(dev, in.data(), in.size() * sizeof(double), cudaMemcpyHostToDevice, s));
  double* d_glt = dev + in.size();
  double* d_glw = d_glt + cfg->n_q;
  double* d_lnm = d_glw + cfg->n_q;
  double* d_z = d_lnm + cfg->n_lnm;
  double* d_S = d_z + cfg->n_z;
  Y3B_TRY(gl_nodes_device(-1.0, 1.0, cfg->n_q, d_glt, d_glw, s));

  SelFuncArgs a;
  a.n_lnm = cfg->n_lnm;
  a.n_z = cfg->n_z;
  a.n_q = cfg->n_q;
  a.n_bins = nb;
  a.n_edges = (int)edges.size();
  a.n_pairs = (int)plo.size();
  a.lnm_low = cfg->lnm_low;
  a.lnm_high = cfg->lnm_high;
  a.zt_low = cfg->zt_low;
  a.zt_high = cfg->zt_high;
  a.mor_kind = mor->kind;
  for (int i = 0; i < 8; ++i) a.mor[i] = mor->p[i];
  a.n_plob = plob->n;
  a.edges = dev;
  a.zob_min = a.edges + ne;
  a.zob_max = a.zob_min + nb;
  a.sigma_z = a.zob_max + nb;
  a.plob_z = a.sigma_z + nb;
  a.plob_coef = a.plob_z + np;
  a.pair_lo = reinterpret_cast<const int*>(dev + n_in);
  a.pair_hi = a.pair_lo + plo.size();
  a.bin_pair = a.pair_hi + phi_.size();
  a.gl_t = d_glt;
  a.gl_w = d_glw;
  a.lnm_out = d_lnm;
  a.z_out = d_z;
  a.S_out = d_S;
  Y3B_TRY(launch_sel_function(a, chained(plo, phi_, edges.size()), s));
  Y3B_CUDA(cudaMemcpyAsync(lnm_out, d_lnm, cfg->n_lnm * sizeof(double), cudaMemcpyDeviceToHost, s));
  Y3B_CUDA(cudaMemcpyAsync(z_out, d_z, cfg->n_z * sizeof(double), cudaMemcpyDeviceToHost, s));
  Y3B_CUDA(cudaMemcpyAsync(S_out, d_S, nS * sizeof(double), cudaMemcpyDeviceToHost, s));
  Y3B_CUDA(cudaStreamSynchronize(s));
  return Y3B_OK;
}

// ===========================================================================
// SelGLCore
namespace y3b {

struct SelGLTablesDev {
  int n_hm, n_hz, n_dist, n_sci;
  const double* hax;       // ln(m_h (om - onu)) [n_hm]
  const double* hz;        // [n_hz]
  const double* dn;        // [n_hz][n_hm]
  const double* dz;
  const double* da;
  const double* sz;
  const double* sv;
};

// One CTA per bin b: W_b[k] = sum_q zfac[q] hmf(k, q) sel_b(k, q)
// (n_operator_sel_gl_t.hh:115-124), one warp per lnM node with the lanes over
// q, then the plain lnM moments n0, n1, m2 with fixed-order tree sums
// (129-141).  Everything that depends on q alone (z factor, HMF and selection
// z cells) is formed once, one q a thread; a thread that summed a node's 64 q
// by itself, both bilinear searches per term, took 190 us at 96 x 64.  A
// selection cell of -1 marks a z outside its box (sel_function_t.hh:228-242).
constexpr int kBuildThreads = 1024;

__host__ __device__ inline size_t
build_smem_bytes(int n_z)
{
  return ((size_t)3 * n_z + kBuildThreads) * sizeof(double) + (size_t)2 * n_z * sizeof(int);
}

__global__ void __launch_bounds__(kBuildThreads)
selgl_build_kernel(int n_lnm, int n_z, const double* lnm_x, const double* lnm_w,
                   const double* z_x, const double* z_w, double lnm_lo, double lnm_hi,
                   y3b_cosmo c, SelGLTablesDev t, int include_sci, int n_sel_lnm,
                   const double* sel_lnm, int n_sel_z, const double* sel_z,
                   const double* S_stack, double* W, double* norm, double* lnm_eff,
                   double* mu2, int* status)
{
  extern __shared__ double sh[];
  double* zfac = sh;             // [n_z]
  double* hu = zfac + n_z;       // [n_z] weight in the HMF z cell
  double* su = hu + n_z;         // [n_z] weight in the selection z cell
  double* red = su + n_z;        // [blockDim.x]
  int* hy = reinterpret_cast<int*>(red + kBuildThreads);  // [n_z] HMF z cell
  int* sy = hy + n_z;                                     // [n_z] selection z cell, or -1
  const int b = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double slo = sel_lnm[0], shi = sel_lnm[n_sel_lnm - 1];
  const double zlo = sel_z[0], zhi = sel_z[n_sel_z - 1];
  for (int q = threadIdx.x; q < n_z; q += blockDim.x) {
    double z = z_x[q], dv;
    if (!dv_do_dz(t.dz, t.da, t.n_dist, c.om, c.ol, c.ok, c.h0, z, &dv)) {
      set_err(status, kDevDomain);
      dv = 0.0;
    }
    double sci = (include_sci && t.n_sci > 0) ? interp1d_clamp(t.sz, t.sv, t.n_sci, z) : 1.0;
    zfac[q] = z_w[q] * dv * omega_z_des(z) * sci;
    const double zh = fmin(fmax(z, t.hz[0]), t.hz[t.n_hz - 1]);
    const int yh = bsearch_cell(t.hz, t.n_hz, zh);
    hy[q] = yh;
    hu[q] = (zh - t.hz[yh]) / (t.hz[yh + 1] - t.hz[yh]);
    const int ys = z < zlo || z > zhi ? -1 : bsearch_cell(sel_z, n_sel_z, z);
    sy[q] = ys;
    su[q] = ys < 0 ? 0.0 : (z - sel_z[ys]) / (sel_z[ys + 1] - sel_z[ys]);
  }
  __syncthreads();
  const double* plane = S_stack + (size_t)b * n_sel_z * n_sel_lnm;
  for (int k = warp; k < n_lnm; k += kBuildThreads / 32) {
    const double lnM = lnm_x[k];
    const double xh = fmin(fmax(lnM, t.hax[0]), t.hax[t.n_hm - 1]);
    const int ih = bsearch_cell(t.hax, t.n_hm, xh);
    const double th = (xh - t.hax[ih]) / (t.hax[ih + 1] - t.hax[ih]);
    const double hs = c.hmf_s * (lnM * kLog10e - kHmfPivot) + c.hmf_q;
    const bool in = !(lnM < slo || lnM > shi);
    const double xs = fmin(fmax(lnM, slo), shi);
    const int is = bsearch_cell(sel_lnm, n_sel_lnm, xs);
    const double ts = (xs - sel_lnm[is]) / (sel_lnm[is + 1] - sel_lnm[is]);
    double acc = 0.0;
    for (int q = lane; q < n_z; q += 32) {
      const double u = hu[q];
      const double* h0 = t.dn + (size_t)hy[q] * t.n_hm + ih;
      const double* h1 = h0 + t.n_hm;
      const double h = ((1.0 - th) * (1.0 - u) * h0[0] + th * (1.0 - u) * h0[1] +
                        (1.0 - th) * u * h1[0] + th * u * h1[1]) *
                       hs;
      double s = 0.0;
      if (in && sy[q] >= 0) {
        const double v = su[q];
        const double* s0 = plane + (size_t)sy[q] * n_sel_lnm + is;
        const double* s1 = s0 + n_sel_lnm;
        s = (1.0 - ts) * (1.0 - v) * s0[0] + ts * (1.0 - v) * s0[1] + (1.0 - ts) * v * s1[0] +
            ts * v * s1[1];
      }
      acc += zfac[q] * h * s;
    }
    acc = warp_sum(acc);
    if (lane == 0) W[(size_t)b * n_lnm + k] = acc;
  }
  __syncthreads();
  double n0 = 0.0, n1 = 0.0;
  for (int k = threadIdx.x; k < n_lnm; k += blockDim.x) {
    const double w = lnm_w[k] * W[(size_t)b * n_lnm + k];
    n0 += w;
    n1 += w * lnm_x[k];
  }
  n0 = block_sum<1024>(n0, red);
  n1 = block_sum<1024>(n1, red);
  double eff = (n0 != 0.0) ? n1 / n0 : 0.5 * (lnm_lo + lnm_hi);
  double m2 = 0.0;
  for (int k = threadIdx.x; k < n_lnm; k += blockDim.x) {
    double d = lnm_x[k] - eff;
    m2 += lnm_w[k] * W[(size_t)b * n_lnm + k] * d * d;
  }
  m2 = block_sum<1024>(m2, red);
  if (threadIdx.x == 0) {
    norm[b] = n0;
    lnm_eff[b] = eff;
    mu2[b] = (n0 != 0.0) ? m2 / n0 : 0.0;
  }
}

// The miscentred-profile table NFW_DSIGMA_MIS reads: log of the unit profile
// on ln x (fastest) and ln x_mis axes (nfw_dsigma_mis.hh:62-72,95-114).
struct MisTable {
  int n_lx, n_lxm;
  const double* logx;
  const double* logxmis;
  const double* log_tab;  // [n_lxm][n_lx]
};

// phi(b, R, lnM) = (1 - f) dSigma_nfw.clamp(R, lnM) + f NFW_DSIGMA_MIS(R,
// r_mis_b, lnM) for a list of (rmis, R, lnM) triples; one warp per triple
// (n_operator_sel_gl_t.hh:343-349).  The module builds NFW_DSIGMA_MIS with
// rho_c and sets rho_mult = Omega_M (n_operator_sel_gl_t.hh:248,264), so r_s
// comes from rho_c and the amplitude 2 r_s delta_c rho_c rho_mult carries
// Omega_M.  The profile is the reference's table (clamped bilinear at
// (ln x, ln x_mis)) when one is loaded, otherwise the direct quadrature that
// generates such a table.
__global__ void __launch_bounds__(128)
phi_list_kernel(int n, const double* rmis, const double* R, const double* lnM,
                double f_mis, double conc, double rhoc, double rho_mult, int n_r,
                const double* r_sigma, int n_ml, const double* lnM_tab, const double* dsig,
                MisQuad q, MisTable tab, double* out)
{
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= n) return;
  const double rs = nfw_rs(lnM[w], conc, rhoc);
  double mis;
  if (tab.log_tab) {
    mis = exp(interp2d_clamp(tab.logx, tab.n_lx, tab.logxmis, tab.n_lxm, tab.log_tab,
                             log(R[w] / rs), log(rmis[w] / rs)));
  } else {
    mis = mis_partial<double>(q, R[w] / rs, rmis[w] / rs, true, lane);
    mis = warp_sum(mis);
  }
  if (lane == 0) {
    double cen = interp2d_clamp(r_sigma, n_r, lnM_tab, n_ml, dsig, R[w], lnM[w]);
    out[w] = (1.0 - f_mis) * cen + f_mis * (nfw_norm(lnM[w], conc, rhoc) * rho_mult) * mis;
  }
}

// NFW_DSIGMA_MIS / NFW_SIGMA_MIS at arbitrary points, one warp per point.
__global__ void __launch_bounds__(128)
nfw_mis_kernel(int which, int n, const double* r, const double* rmis, const double* lnM,
               double conc, double rho, MisQuad q, double* out)
{
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= n) return;
  const double rs = nfw_rs(lnM[w], conc, rho);
  double v = which == 2
               ? dsigma_single_partial(q.th, q.wth, q.n_theta, r[w] / rs, rmis[w] / rs, lane, 32) /
                   kPi
               : mis_partial<double>(q, r[w] / rs, rmis[w] / rs, which == 0, lane);
  v = warp_sum(v);
  if (lane == 0) out[w] = nfw_norm(lnM[w], conc, rho) * v;
}

constexpr int kChebNodes = 24;  // lnM nodes of the miscentred profile (struct y3b_selgl)

// The same with the miscentred profile of the query's (R, R_mis) pair given
// (launch_mis_pairs, amplitude and Omega_M included): sum_k w_k W_b[k]
// [(1 - f) dSigma_nfw.clamp(R, lnM_k) + f mis_pair[k]], one block per query,
// a thread per mass (a warp per query takes 19 us with the interpolation).
// With interp ([kChebNodes][n_lnm]) mis_pair holds the kChebNodes node values
// and mis_pair[k] = sum_j interp[j][k] mis_pair_j.
__global__ void __launch_bounds__(128)
shear_pairs_kernel(int n_lnm, const int* bin, const int* pair, const double* R,
                   const double* lnm_x, const double* lnm_w, const double* W, double f_mis,
                   int n_r, const double* r_sigma, int n_ml, const double* lnM_tab,
                   const double* dsig, const double* mis, int n_mis, const double* interp,
                   double* out)
{
  __shared__ double red[4];
  const int w = blockIdx.x, lane = threadIdx.x & 31;
  const double* Wb = W + (size_t)bin[w] * n_lnm;
  const double* m = mis + (size_t)pair[w] * n_mis;
  double acc = 0.0;
  for (int k = threadIdx.x; k < n_lnm; k += blockDim.x) {
    const double cen = interp2d_clamp(r_sigma, n_r, lnM_tab, n_ml, dsig, R[w], lnm_x[k]);
    double mk = 0.0;
    if (interp) {
      double part[4] = {};
#pragma unroll
      for (int j = 0; j < kChebNodes; ++j) part[j & 3] += interp[(size_t)j * n_lnm + k] * m[j];
      mk = (part[0] + part[1]) + (part[2] + part[3]);
    } else {
      mk = m[k];
    }
    acc += lnm_w[k] * Wb[k] * ((1.0 - f_mis) * cen + f_mis * mk);
  }
  acc = warp_sum(acc);
  if (lane == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) out[w] = (red[0] + red[1]) + (red[2] + red[3]);
}

// sum_k w_k W_b[k] phi[k] for each query (exact method); one warp per query.
__global__ void
shear_contract_kernel(int n, int n_lnm, const int* bin, const double* lnm_w,
                      const double* W, const double* phi, double* out)
{
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= n) return;
  const double* Wb = W + (size_t)bin[w] * n_lnm;
  const double* ph = phi + (size_t)w * n_lnm;
  double acc = 0.0;
  for (int k = lane; k < n_lnm; k += 32) acc += lnm_w[k] * Wb[k] * ph[k];
  acc = warp_sum(acc);
  if (lane == 0) out[w] = acc;
}

}  // namespace y3b

namespace y3b {

// The miscentred profile of a pair is analytic in ln r_s = lnM / 3 + const:
// its quadrature sums the NFW DeltaSigma at distances proportional to 1 / r_s,
// whose only singularities in ln x lie at x <= 0, at |Im| >= pi.  On an lnM
// interval of width D the Chebyshev interpolant of n nodes therefore
// converges as rho^-n, rho = h + sqrt(h^2 + 1) with h = 6 pi / D: 5.7 for the
// default range (6.8), 4.4 at D = 9.  Interpolated is the profile over
// sqrt(M), which changes least (the profile grows as M^1/3 far inside r_s and
// as M far outside): at D = 9, radii from 0.1 to 30 and R_mis from 0.05 to 1,
// 24 nodes are within 1.7e-15 of the profile at every mass (the profile itself
// 2e-13, its rounding at the largest masses beside the smallest).  Wider ranges
// and grids with no more than 32 masses (where the nodes save less than a
// block of eight in four) take the quadrature at every mass.
// 60 pairs x 96 masses: quadrature 168 -> 69 us (one block an SM; four radii a
// block: 64), sum over masses 10 us with either.
constexpr int kChebMinMasses = 32;
constexpr double kChebMaxRange = 9.0;

}  // namespace y3b

struct y3b_selgl {
  y3b_selgl_config cfg;
  cudaStream_t stream = nullptr;
  y3b::DevBuf<double> lnm_x, lnm_w, z_x, z_w;
  y3b::DevBuf<double> W, mom;   // mom: norm | lnm_eff | mu2 [n_bins each] | status word
  y3b::DevBuf<double> tab, S;   // the sample's tables in one block; S_stack
  y3b::MisQuadCache quad;
  y3b::DevBuf<double> sh_in, sh_mis, sh_out;   // shear_by_pairs
  y3b::DevBuf<double> cheb;  // lnM nodes [kChebNodes] | interpolation [kChebNodes][n_lnm]
  y3b::DevBuf<int> sh_int;
  y3b::DevBuf<double> tab_lx, tab_lxm, tab_v;  // miscentred-profile table (optional)
  int tab_nlx = 0, tab_nlxm = 0;
  std::vector<double> h_norm, h_eff, h_mu2, h_lnm_x, h_lnm_w, h_tab;
  int n_bins = 0;
  bool built = false;
  double omega_m = 0.0;
};

extern "C" int
y3b_selgl_create(const y3b_selgl_config* cfg, y3b_selgl** out)
{
  clear_error();
  if (!cfg || !out) {
    set_error("y3b_selgl_create: null argument");
    return Y3B_ERR_INVALID;
  }
  *out = nullptr;
  if (cfg->n_lnm < 1 || cfg->n_z < 1 || cfg->n_lnm > 4096 || cfg->n_z > 4096 ||
      !(cfg->lnm_high > cfg->lnm_low) || !(cfg->zt_high > cfg->zt_low)) {
    set_error("y3b_selgl_create: invalid grid (n_lnm, n_z in [1, 4096], ordered bounds)");
    return Y3B_ERR_INVALID;
  }
  Y3B_TRY(require_device());
  y3b_selgl* h = new (std::nothrow) y3b_selgl();
  if (!h) {
    set_error("y3b_selgl_create: out of host memory");
    return Y3B_ERR_NOMEM;
  }
  h->cfg = *cfg;
  int rc = y3b::cuda_status(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking),
                            "cudaStreamCreate");
  if (rc == Y3B_OK) rc = h->lnm_x.alloc(cfg->n_lnm);
  if (rc == Y3B_OK) rc = h->lnm_w.alloc(cfg->n_lnm);
  if (rc == Y3B_OK) rc = h->z_x.alloc(cfg->n_z);
  if (rc == Y3B_OK) rc = h->z_w.alloc(cfg->n_z);
  if (rc == Y3B_OK)
    rc = y3b::gl_nodes_device(cfg->lnm_low, cfg->lnm_high, cfg->n_lnm, h->lnm_x.get(),
                              h->lnm_w.get(), h->stream);
  if (rc == Y3B_OK)
    rc = y3b::gl_nodes_device(cfg->zt_low, cfg->zt_high, cfg->n_z, h->z_x.get(), h->z_w.get(),
                              h->stream);
  if (rc == Y3B_OK) {
    h->h_lnm_x.resize(cfg->n_lnm);
    h->h_lnm_w.resize(cfg->n_lnm);
    rc = y3b::cuda_status(cudaMemcpyAsync(h->h_lnm_x.data(), h->lnm_x.get(),
                                          cfg->n_lnm * sizeof(double), cudaMemcpyDeviceToHost,
                                          h->stream),
                          "copy lnm_x");
  }
  if (rc == Y3B_OK)
    rc = y3b::cuda_status(cudaMemcpyAsync(h->h_lnm_w.data(), h->lnm_w.get(),
                                          cfg->n_lnm * sizeof(double), cudaMemcpyDeviceToHost,
                                          h->stream),
                          "copy lnm_w");
  if (rc == Y3B_OK) rc = y3b::cuda_status(cudaStreamSynchronize(h->stream), "sync");
  if (rc == Y3B_OK && cfg->n_lnm > y3b::kChebMinMasses &&
      cfg->lnm_high - cfg->lnm_low <= y3b::kChebMaxRange) {
    std::vector<double> v =
      y3b::cheb_rows(y3b::kChebNodes, cfg->lnm_low, cfg->lnm_high, h->h_lnm_x);
    for (int j = 0; j < y3b::kChebNodes; ++j)  // over sqrt(M) at the nodes, times it at the masses
      for (int k = 0; k < cfg->n_lnm; ++k)
        v[y3b::kChebNodes + (size_t)j * cfg->n_lnm + k] *= std::exp(0.5 * (h->h_lnm_x[k] - v[j]));
    rc = h->cheb.upload(v.data(), v.size(), h->stream);
    if (rc == Y3B_OK) rc = y3b::cuda_status(cudaStreamSynchronize(h->stream), "sync");
  }
  if (rc != Y3B_OK) {
    y3b_selgl_destroy(h);
    return rc;
  }
  *out = h;
  return Y3B_OK;
}

extern "C" void
y3b_selgl_destroy(y3b_selgl* h)
{
  if (!h) return;
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
}

extern "C" int
y3b_selgl_n_bins(const y3b_selgl* h)
{
  return h ? h->n_bins : 0;
}

extern "C" int
y3b_selgl_build(y3b_selgl* h, const y3b_cosmo* c, const y3b_tables* t,
                const y3b_selection* sel, int include_sci)
{
  using namespace y3b;
  clear_error();
  if (!h || !c || !t || !sel || !sel->S_stack || !sel->lnm || !sel->z) {
    set_error("y3b_selgl_build: null argument");
    return Y3B_ERR_INVALID;
  }
  if (t->n_hm < 2 || t->n_hz < 2 || t->n_dist < 2 || sel->n_bins < 1 || sel->n_lnm < 2 ||
      sel->n_z < 2 || (include_sci && t->n_sci < 2)) {
    set_error("y3b_selgl_build: tables need >= 2 nodes per axis and >= 1 bin");
    return Y3B_ERR_INVALID;
  }
  if (!(c->om - c->onu > 0.0)) {
    set_error("y3b_selgl_build: omega_M - omega_nu must be positive");
    return Y3B_ERR_INVALID;
  }
  cudaStream_t s = h->stream;
  const int nb = sel->n_bins, n_sci = include_sci ? t->n_sci : 0;
  Y3B_TRY(h->W.alloc((size_t)nb * h->cfg.n_lnm));
  Y3B_TRY(h->mom.alloc(3 * (size_t)nb + 1));
  // One block: HMF mass axis ln(m_h (Omega_M - Omega_nu)) (hmf_t.hh:15-25) |
  // z | dn/dlnM | distances | Sigma_crit^-1 | selection axes.
  std::vector<double>& v = h->h_tab;
  v.clear();
  auto put = [&](const double* p, size_t n) {
    const size_t at = v.size();
    if (n) v.insert(v.end(), p, p + n);
    return at;
  };
  const size_t o_ax = put(t->hmf_m_h, t->n_hm), o_hz = put(t->hmf_z, t->n_hz);
  for (int i = 0; i < t->n_hm; ++i) v[o_ax + i] = std::log(v[o_ax + i] * (c->om - c->onu));
  const size_t o_dn = put(t->dndlnmh, (size_t)t->n_hz * t->n_hm);
  const size_t o_dz = put(t->dist_z, t->n_dist), o_da = put(t->dist_da, t->n_dist);
  const size_t o_sz = put(t->sci_z, n_sci), o_sv = put(t->sci_val, n_sci);
  const size_t o_sl = put(sel->lnm, sel->n_lnm), o_sel_z = put(sel->z, sel->n_z);
  Y3B_TRY(h->tab.upload(v.data(), v.size(), s));
  Y3B_TRY(h->S.upload(sel->S_stack, (size_t)nb * sel->n_z * sel->n_lnm, s));
  double* mom = h->mom.get();
  int* status = reinterpret_cast<int*>(mom + 3 * (size_t)nb);
  Y3B_CUDA(cudaMemsetAsync(status, 0, sizeof(double), s));
  const double* d = h->tab.get();
  SelGLTablesDev td{t->n_hm, t->n_hz, t->n_dist, n_sci, d + o_ax, d + o_hz, d + o_dn, d + o_dz,
                    d + o_da, include_sci ? d + o_sz : nullptr,
                    include_sci ? d + o_sv : nullptr};
  const size_t shm = build_smem_bytes(h->cfg.n_z);
  if (shm > 48 * 1024) Y3B_TRY(allow_max_smem(selgl_build_kernel));
  selgl_build_kernel<<<nb, kBuildThreads, shm, s>>>(
    h->cfg.n_lnm, h->cfg.n_z, h->lnm_x.get(), h->lnm_w.get(), h->z_x.get(), h->z_w.get(),
    h->cfg.lnm_low, h->cfg.lnm_high, *c, td, include_sci, sel->n_lnm, d + o_sl, sel->n_z,
    d + o_sel_z, h->S.get(), h->W.get(), mom, mom + nb, mom + 2 * (size_t)nb, status);
  count_launch();
  Y3B_CUDA(cudaGetLastError());
  std::vector<double> hm(3 * (size_t)nb + 1);
  Y3B_CUDA(cudaMemcpyAsync(hm.data(), mom, hm.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
  Y3B_CUDA(cudaStreamSynchronize(s));
  h->h_norm.assign(hm.begin(), hm.begin() + nb);
  h->h_eff.assign(hm.begin() + nb, hm.begin() + 2 * (size_t)nb);
  h->h_mu2.assign(hm.begin() + 2 * (size_t)nb, hm.end() - 1);
  int code;
  std::memcpy(&code, &hm.back(), sizeof code);
  const int st = device_status_rc(code);
  h->n_bins = nb;
  h->omega_m = c->om;
  h->built = (st == Y3B_OK);
  if (st == Y3B_ERR_DOMAIN)
    set_error("y3b_selgl_build: a GL z node lies outside distances/z (argument out of range in Interp1D)");
  return st;
}

extern "C" int
y3b_selgl_counts(y3b_selgl* h, int n, const int* bin_index, double* vals)
{
  y3b::clear_error();
  if (!h || (n > 0 && (!bin_index || !vals))) {
    y3b::set_error("y3b_selgl_counts: null argument");
    return Y3B_ERR_INVALID;
  }
  if (!h->built) {
    y3b::set_error("y3b_selgl_counts: no sample built");
    return Y3B_ERR_INVALID;
  }
  for (int i = 0; i < n; ++i) {
    int b = bin_index[i];
    if (b < 0 || b >= h->n_bins) {
      y3b::set_error("NumCountsSelGL: bin_index outside sel_function/S_stack range");
      return Y3B_ERR_INVALID;
    }
    vals[i] = h->h_norm[b];
  }
  return Y3B_OK;
}

extern "C" int
y3b_selgl_weights(y3b_selgl* h, double* W, double* norm, double* lnm_eff, double* mu2,
                  double* lnm_x, double* lnm_w)
{
  y3b::clear_error();
  if (!h || !h->built) {
    y3b::set_error("y3b_selgl_weights: no sample built");
    return Y3B_ERR_INVALID;
  }
  const int nb = h->n_bins, nl = h->cfg.n_lnm;
  if (W)
    Y3B_CUDA(cudaMemcpy(W, h->W.get(), (size_t)nb * nl * sizeof(double), cudaMemcpyDeviceToHost));
  if (norm) std::memcpy(norm, h->h_norm.data(), nb * sizeof(double));
  if (lnm_eff) std::memcpy(lnm_eff, h->h_eff.data(), nb * sizeof(double));
  if (mu2) std::memcpy(mu2, h->h_mu2.data(), nb * sizeof(double));
  if (lnm_x) std::memcpy(lnm_x, h->h_lnm_x.data(), nl * sizeof(double));
  if (lnm_w) std::memcpy(lnm_w, h->h_lnm_w.data(), nl * sizeof(double));
  return Y3B_OK;
}

// NFW_DSIGMA_MIS's profile table (nfw_dsigma_mis.hh:62-72): kept on the
// device for the handle's shear evaluations; n_lx = 0 drops it.
extern "C" int
y3b_selgl_set_mis_table(y3b_selgl* h, int n_lx, const double* logx, int n_lxm,
                        const double* logxmis, const double* log_tab)
{
  using namespace y3b;
  clear_error();
  if (!h) {
    set_error("y3b_selgl_set_mis_table: null handle");
    return Y3B_ERR_INVALID;
  }
  if (n_lx == 0) {
    h->tab_nlx = h->tab_nlxm = 0;
    return Y3B_OK;
  }
  if (n_lx < 2 || n_lxm < 2 || !logx || !logxmis || !log_tab) {
    set_error("y3b_selgl_set_mis_table: need at least 2 x 2 nodes and three arrays");
    return Y3B_ERR_INVALID;
  }
  for (int i = 1; i < n_lx; ++i)
    if (!(logx[i] > logx[i - 1])) {
      set_error("y3b_selgl_set_mis_table: ln x axis not increasing");
      return Y3B_ERR_INVALID;
    }
  for (int j = 1; j < n_lxm; ++j)
    if (!(logxmis[j] > logxmis[j - 1])) {
      set_error("y3b_selgl_set_mis_table: ln x_mis axis not increasing");
      return Y3B_ERR_INVALID;
    }
  const size_t nv = (size_t)n_lx * n_lxm;
  for (size_t i = 0; i < nv; ++i)
    if (!std::isfinite(log_tab[i])) {
      set_error("y3b_selgl_set_mis_table: non-finite table entry");
      return Y3B_ERR_DOMAIN;
    }
  h->tab_nlx = h->tab_nlxm = 0;
  Y3B_TRY(h->tab_lx.upload(logx, n_lx, h->stream));
  Y3B_TRY(h->tab_lxm.upload(logxmis, n_lxm, h->stream));
  Y3B_TRY(h->tab_v.upload(log_tab, nv, h->stream));
  Y3B_CUDA(cudaStreamSynchronize(h->stream));
  h->tab_nlx = n_lx;
  h->tab_nlxm = n_lxm;
  return Y3B_OK;
}

namespace y3b {

// Exact method, profile by quadrature: the queries share few distinct
// (R_mis, R) pairs (the z_obs bins of a richness bin have the same ones), and
// a pair's quadrature geometry serves all masses.  12 bins x 15 radii x 96
// masses: one warp per (query, mass) with the closed-form profile took
// 6.2 ms.
static int
shear_by_pairs(y3b_selgl* h, const y3b_shear_table* st, int n, const int* bin_index,
               const double* r, double* vals)
{
  cudaStream_t s = h->stream;
  Y3B_TRY(h->quad.ensure_nfw(s));
  std::map<std::pair<int, uint64_t>, int> seen;  // (richness centre, bits of R) -> pair
  std::vector<double> buf, rmis;
  std::vector<int> ints(bin_index, bin_index + n);
  for (int i = 0; i < n; ++i) {
    uint64_t bits;
    std::memcpy(&bits, r + i, sizeof bits);
    const int c = bin_index[i] % st->n_lob;
    const auto it = seen.emplace(std::make_pair(c, bits), (int)buf.size());
    if (it.second) {
      buf.push_back(r[i]);
      rmis.push_back(st->tau_mis * std::pow(st->lob_centers[c] / 100.0, 0.2));
    }
    ints.push_back(it.first->second);
  }
  const int np = (int)buf.size(), nl = h->cfg.n_lnm;
  const double* cheb = h->cheb.get();  // null: the quadrature at every mass
  const int n_mis = cheb ? kChebNodes : nl;
  buf.insert(buf.end(), rmis.begin(), rmis.end());
  buf.insert(buf.end(), r, r + n);
  buf.insert(buf.end(), st->r_sigma, st->r_sigma + st->n_r);
  buf.insert(buf.end(), st->lnM, st->lnM + st->n_lnm);
  buf.insert(buf.end(), st->dsigma, st->dsigma + (size_t)st->n_r * st->n_lnm);
  Y3B_TRY(h->sh_in.upload(buf.data(), buf.size(), s));
  Y3B_TRY(h->sh_int.upload(ints.data(), ints.size(), s));
  Y3B_TRY(h->sh_mis.alloc((size_t)np * n_mis));
  Y3B_TRY(h->sh_out.alloc(n));
  const double* R = h->sh_in.get();
  const double* d_r = R + 2 * (size_t)np;
  const double* d_rs = d_r + n;
  const MisPairs a{np,       n_mis,      R,   R + np, cheb ? cheb : h->lnm_x.get(), st->conc,
                   kRhoCrit, h->omega_m, 0.0, 0.0,    h->sh_mis.get()};
  Y3B_TRY(launch_mis_pairs(h->quad.view(), h->quad.nfw.get(), a, s));
  shear_pairs_kernel<<<n, 128, 0, s>>>(
    nl, h->sh_int.get(), h->sh_int.get() + n, d_r, h->lnm_x.get(), h->lnm_w.get(), h->W.get(),
    st->f_mis, st->n_r, d_rs, st->n_lnm, d_rs + st->n_r, d_rs + st->n_r + st->n_lnm,
    h->sh_mis.get(), n_mis, cheb ? cheb + kChebNodes : nullptr, h->sh_out.get());
  count_launch();
  Y3B_CUDA(cudaGetLastError());
  Y3B_CUDA(cudaMemcpyAsync(vals, h->sh_out.get(), n * sizeof(double), cudaMemcpyDeviceToHost, s));
  Y3B_CUDA(cudaStreamSynchronize(s));
  return Y3B_OK;
}

}  // namespace y3b

// Shear1hMisSelGL::evaluate (n_operator_sel_gl_t.hh:293-319): exact =
// sum_k w_k W_b[k] phi(b, R, lnM_k); idea2 = norm_b [phi + mu2/2 d2phi] at
// lnm_eff with a 3-point stencil.
extern "C" int
y3b_selgl_shear(y3b_selgl* h, const y3b_shear_table* st, int n, const int* bin_index,
                const double* r, double* vals)
{
  using namespace y3b;
  clear_error();
  if (!h || !st || (n > 0 && (!bin_index || !r || !vals))) {
    set_error("y3b_selgl_shear: null argument");
    return Y3B_ERR_INVALID;
  }
  if (!h->built) {
    set_error("y3b_selgl_shear: no sample built");
    return Y3B_ERR_INVALID;
  }
  if (st->n_lob < 1 || st->n_r < 2 || st->n_lnm < 2 || !st->r_sigma || !st->lnM || !st->dsigma) {
    set_error("Shear1hMisSelGL: lob_centers is empty or haloModel table missing");
    return Y3B_ERR_INVALID;
  }
  for (int i = 0; i < n; ++i)
    if (bin_index[i] < 0 || bin_index[i] >= h->n_bins) {
      set_error("Shear1hMisSelGL: bin_index outside sel_function/S_stack range");
      return Y3B_ERR_INVALID;
    }
  if (n == 0) return Y3B_OK;
  cudaStream_t s = h->stream;
  if (!h->tab_nlx) Y3B_TRY(h->quad.ensure(st->n_theta, st->n_s, st->s_max, s));
  MisTable tab{h->tab_nlx, h->tab_nlxm, h->tab_lx.get(), h->tab_lxm.get(),
               h->tab_nlx ? h->tab_v.get() : nullptr};
  const int nl = h->cfg.n_lnm;
  if (!st->use_idea2 && !h->tab_nlx) return shear_by_pairs(h, st, n, bin_index, r, vals);
  // Triples (rmis, R, lnM) of phi evaluations.
  std::vector<double> trm, tR, tM;
  if (!st->use_idea2) {
    trm.reserve((size_t)n * nl);
    for (int i = 0; i < n; ++i) {
      double rmis = st->tau_mis * std::pow(st->lob_centers[bin_index[i] % st->n_lob] / 100.0, 0.2);
      for (int k = 0; k < nl; ++k) {
        trm.push_back(rmis);
        tR.push_back(r[i]);
        tM.push_back(h->h_lnm_x[k]);
      }
    }
  } else {
    for (int i = 0; i < n; ++i) {
      int b = bin_index[i];
      double rmis = st->tau_mis * std::pow(st->lob_centers[b % st->n_lob] / 100.0, 0.2);
      double y0 = h->h_eff[b];
      for (double dy : {0.0, st->stencil_h, -st->stencil_h}) {
        trm.push_back(rmis);
        tR.push_back(r[i]);
        tM.push_back(y0 + dy);
      }
    }
  }
  const int nt = (int)trm.size();
  DevBuf<double> d_rm, d_R, d_M, d_phi, d_rs, d_lt, d_ds, d_out;
  DevBuf<int> d_bin;
  Y3B_TRY(d_rm.upload(trm.data(), nt, s));
  Y3B_TRY(d_R.upload(tR.data(), nt, s));
  Y3B_TRY(d_M.upload(tM.data(), nt, s));
  Y3B_TRY(d_phi.alloc(nt));
  Y3B_TRY(d_rs.upload(st->r_sigma, st->n_r, s));
  Y3B_TRY(d_lt.upload(st->lnM, st->n_lnm, s));
  Y3B_TRY(d_ds.upload(st->dsigma, (size_t)st->n_r * st->n_lnm, s));
  phi_list_kernel<<<(nt * 32 + 127) / 128, 128, 0, s>>>(
    nt, d_rm.get(), d_R.get(), d_M.get(), st->f_mis, st->conc, kRhoCrit, h->omega_m, st->n_r,
    d_rs.get(), st->n_lnm, d_lt.get(), d_ds.get(), h->tab_nlx ? MisQuad{} : h->quad.view(), tab,
    d_phi.get());
  count_launch();
  Y3B_CUDA(cudaGetLastError());
  if (!st->use_idea2) {
    Y3B_TRY(d_bin.upload(bin_index, n, s));
    Y3B_TRY(d_out.alloc(n));
    shear_contract_kernel<<<(n * 32 + 127) / 128, 128, 0, s>>>(
      n, nl, d_bin.get(), h->lnm_w.get(), h->W.get(), d_phi.get(), d_out.get());
    count_launch();
    Y3B_CUDA(cudaGetLastError());
    Y3B_CUDA(cudaMemcpyAsync(vals, d_out.get(), n * sizeof(double), cudaMemcpyDeviceToHost, s));
    Y3B_CUDA(cudaStreamSynchronize(s));
  } else {
    std::vector<double> phi(nt);
    Y3B_CUDA(cudaMemcpyAsync(phi.data(), d_phi.get(), nt * sizeof(double),
                             cudaMemcpyDeviceToHost, s));
    Y3B_CUDA(cudaStreamSynchronize(s));
    for (int i = 0; i < n; ++i) {
      int b = bin_index[i];
      double c0 = phi[3 * i], p = phi[3 * i + 1], m = phi[3 * i + 2];
      double hh = st->stencil_h;
      double d2 = (p - 2.0 * c0 + m) / (hh * hh);
      vals[i] = h->h_norm[b] * (c0 + 0.5 * h->h_mu2[b] * d2);
    }
  }
  return Y3B_OK;
}

// ===========================================================================
namespace y3b {

// <Sigma_crit^-1>(z_l): one CTA per lens redshift, threads over sources,
// trapezoid by a fixed-order tree (average_sigma_crit_inv.py:53-58).
__global__ void __launch_bounds__(256)
sigma_crit_inv_kernel(const double* zl, int n_zs, const double* zs, const double* pz,
                      double delta_z, double h0, int nd, const double* dz, const double* da,
                      double* out, int* status)
{
  __shared__ double red[256];
  const double G = 4.51710305e-48, cl = 9.71561189e-15;
  const double kk = 4.0 * kPi * G / cl / cl;
  const int j = blockIdx.x;
  double dl;
  if (!interp1d(dz, da, nd, zl[j], &dl)) {
    set_err(status, kDevDomain);
    dl = 0.0;
  }
  auto f = [&](int i) -> double {
    double ds, p;
    if (!interp1d(dz, da, nd, zs[i], &ds) || !interp1d(zs, pz, n_zs, zs[i] + delta_z, &p)) {
      set_err(status, kDevDomain);
      return 0.0;
    }
    double dls = ds - (1.0 + zl[j]) / (1.0 + zs[i]) * dl;
    double v = ds > 0.0 ? p * kk * dl * dls / ds : 0.0;
    return v > 0.0 ? v : 0.0;
  };
  double acc = 0.0;
  for (int i = threadIdx.x; i + 1 < n_zs; i += blockDim.x)
    acc += 0.5 * (f(i) + f(i + 1)) * (zs[i + 1] - zs[i]);
  acc = block_sum<256>(acc, red);
  if (threadIdx.x == 0) out[j] = acc * h0;
}

}  // namespace y3b

extern "C" int
y3b_sigma_crit_inv(int n_zl, const double* zl, int n_zs, const double* zs, const double* pz,
                   double delta_z, double h0, int n_dist, const double* dist_z,
                   const double* dist_da, double* out)
{
  using namespace y3b;
  clear_error();
  if (n_zl < 1 || n_zs < 2 || n_dist < 2 || !zl || !zs || !pz || !dist_z || !dist_da || !out) {
    set_error("y3b_sigma_crit_inv: invalid arguments");
    return Y3B_ERR_INVALID;
  }
  Y3B_TRY(require_device());
  cudaStream_t s = 0;
  DevBuf<double> a, b, c, d, e, o;
  DevBuf<int> st;
  Y3B_TRY(a.upload(zl, n_zl, s));
  Y3B_TRY(b.upload(zs, n_zs, s));
  Y3B_TRY(c.upload(pz, n_zs, s));
  Y3B_TRY(d.upload(dist_z, n_dist, s));
  Y3B_TRY(e.upload(dist_da, n_dist, s));
  Y3B_TRY(o.alloc(n_zl));
  Y3B_TRY(st.alloc(1));
  Y3B_CUDA(cudaMemsetAsync(st.get(), 0, sizeof(int), s));
  sigma_crit_inv_kernel<<<n_zl, 256, 0, s>>>(a.get(), n_zs, b.get(), c.get(), delta_z, h0,
                                             n_dist, d.get(), e.get(), o.get(), st.get());
  count_launch();
  Y3B_CUDA(cudaGetLastError());
  Y3B_CUDA(cudaMemcpyAsync(out, o.get(), n_zl * sizeof(double), cudaMemcpyDeviceToHost, s));
  int rc = read_device_status(st.get(), s);
  if (rc == Y3B_ERR_DOMAIN) set_error("y3b_sigma_crit_inv: redshift outside distances or n(z) table");
  return rc;
}

extern "C" int
y3b_nfw_mis(int which, int n, const double* r, const double* rmis, const double* lnM,
            double conc, double rho, int n_theta, int n_s, double s_max, double* out)
{
  using namespace y3b;
  clear_error();
  if (n < 0 || (n > 0 && (!r || !rmis || !lnM || !out)) || which < 0 || which > 2 ||
      !(conc > 0.0) || !(rho > 0.0)) {
    set_error("y3b_nfw_mis: invalid arguments");
    return Y3B_ERR_INVALID;
  }
  if (n == 0) return Y3B_OK;
  Y3B_TRY(require_device());
  cudaStream_t s = 0;
  MisQuadCache quad;
  Y3B_TRY(quad.ensure(n_theta, n_s, s_max, s));
  DevBuf<double> a, b, c, o;
  Y3B_TRY(a.upload(r, n, s));
  Y3B_TRY(b.upload(rmis, n, s));
  Y3B_TRY(c.upload(lnM, n, s));
  Y3B_TRY(o.alloc(n));
  nfw_mis_kernel<<<(n * 32 + 127) / 128, 128, 0, s>>>(which, n, a.get(), b.get(), c.get(), conc,
                                                     rho, quad.view(), o.get());
  count_launch();
  Y3B_CUDA(cudaGetLastError());
  Y3B_CUDA(cudaMemcpyAsync(out, o.get(), n * sizeof(double), cudaMemcpyDeviceToHost, s));
  Y3B_CUDA(cudaStreamSynchronize(s));
  return Y3B_OK;
}

// ===========================================================================
// y3b_sel_function_noalloc: the S_stack producer for callers that cannot
// allocate device memory.  Everything the kernel needs besides the caller's
// output buffers (Gauss-Legendre nodes, the unique richness edges and their
// bin pairing, the per-bin photo-z edges and widths, the projection table)
// lives in one file-scope __device__ array of fixed size that every call
// shares.
extern "C" int
y3b_sel_function_noalloc(const y3b_selfunc_config* cfg, const y3b_mor* mor,
                         const y3b_plob* plob, double* lnm_dev, double* z_dev, double* S_dev,
                         void* stream)
{
  using namespace y3b;
  clear_error();
  if (!cfg || !mor || !plob || !lnm_dev || !z_dev || !S_dev || !plob->z || !plob->coef ||
      !cfg->lam_min || !cfg->lam_max || !cfg->zob_min || !cfg->zob_max || !cfg->sigma_z) {
    set_error("y3b_sel_function_noalloc: null argument");
    return Y3B_ERR_INVALID;
  }
  if (cfg->n_bins <= 0 || cfg->n_lnm <= 0 || cfg->n_z <= 0 || cfg->n_q <= 0 || plob->n < 1 ||
      (mor->kind != Y3B_MOR_HOD && mor->kind != Y3B_MOR_LOGNORMAL)) {
    set_error("y3b_sel_function_noalloc: invalid sizes or MOR kind");
    return Y3B_ERR_INVALID;
  }
  if (cfg->n_q > kNoAllocMaxQ || cfg->n_bins > kNoAllocMaxBins || plob->n > kNoAllocMaxPlob) {
    set_error("y3b_sel_function_noalloc: sizes exceed the fixed scratch (N_q <= %d, "
              "n_bins <= %d, projection-table nodes <= %d); use y3b_sel_function",
              kNoAllocMaxQ, kNoAllocMaxBins, kNoAllocMaxPlob);
    return Y3B_ERR_INVALID;
  }
  Y3B_TRY(require_device());
  const int nb = cfg->n_bins;
  std::vector<double> edges;
  for (int k = 0; k < nb; ++k) {
    edges.push_back(cfg->lam_min[k]);
    edges.push_back(cfg->lam_max[k]);
  }
  std::sort(edges.begin(), edges.end());
  edges.erase(std::unique(edges.begin(), edges.end()), edges.end());
  if ((int)edges.size() > kMaxEdges) {
    set_error("y3b_sel_function_noalloc: more than %d unique richness edges", kMaxEdges);
    return Y3B_ERR_UNSUPPORTED;
  }
  std::vector<int> ints;  // pair_lo | pair_hi | bin_pair
  std::vector<int> plo, phi_, bin_pair(nb);
  for (int k = 0; k < nb; ++k) {
    int lo = int(std::lower_bound(edges.begin(), edges.end(), cfg->lam_min[k]) - edges.begin());
    int hi = int(std::lower_bound(edges.begin(), edges.end(), cfg->lam_max[k]) - edges.begin());
    int p = 0;
    for (; p < (int)plo.size(); ++p)
      if (plo[p] == lo && phi_[p] == hi) break;
    if (p == (int)plo.size()) {
      plo.push_back(lo);
      phi_.push_back(hi);
    }
    bin_pair[k] = p;
  }
  if ((int)plo.size() > kMaxPairs) {
    set_error("y3b_sel_function_noalloc: more than %d distinct richness bins", kMaxPairs);
    return Y3B_ERR_UNSUPPORTED;
  }
  double* scratch = nullptr;
  Y3B_TRY(scratch_address(&scratch));
  // Scratch layout (doubles, then ints).
  const int nq = cfg->n_q, np = plob->n;
  double* d_glt = scratch;
  double* d_glw = d_glt + nq;
  double* d_edges = d_glw + nq;
  double* d_zmin = d_edges + edges.size();
  double* d_zmax = d_zmin + nb;
  double* d_sz = d_zmax + nb;
  double* d_pz = d_sz + nb;
  double* d_pc = d_pz + np;
  int* d_ints = reinterpret_cast<int*>(d_pc + 8 * (size_t)np);
  int* d_plo = d_ints;
  int* d_phi = d_plo + plo.size();
  int* d_bp = d_phi + phi_.size();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  auto put = [&](void* dst, const void* src, size_t bytes) {
    return cuda_status(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s),
                       "y3b_sel_function_noalloc: copy to scratch");
  };
  Y3B_TRY(put(d_edges, edges.data(), edges.size() * sizeof(double)));
  Y3B_TRY(put(d_zmin, cfg->zob_min, nb * sizeof(double)));
  Y3B_TRY(put(d_zmax, cfg->zob_max, nb * sizeof(double)));
  Y3B_TRY(put(d_sz, cfg->sigma_z, nb * sizeof(double)));
  Y3B_TRY(put(d_pz, plob->z, np * sizeof(double)));
  Y3B_TRY(put(d_pc, plob->coef, 8 * (size_t)np * sizeof(double)));
  Y3B_TRY(put(d_plo, plo.data(), plo.size() * sizeof(int)));
  Y3B_TRY(put(d_phi, phi_.data(), phi_.size() * sizeof(int)));
  Y3B_TRY(put(d_bp, bin_pair.data(), nb * sizeof(int)));
  Y3B_TRY(gl_nodes_device(-1.0, 1.0, nq, d_glt, d_glw, s));

  SelFuncArgs a;
  a.n_lnm = cfg->n_lnm;
  a.n_z = cfg->n_z;
  a.n_q = nq;
  a.n_bins = nb;
  a.n_edges = (int)edges.size();
  a.n_pairs = (int)plo.size();
  a.lnm_low = cfg->lnm_low;
  a.lnm_high = cfg->lnm_high;
  a.zt_low = cfg->zt_low;
  a.zt_high = cfg->zt_high;
  a.mor_kind = mor->kind;
  for (int i = 0; i < 8; ++i) a.mor[i] = mor->p[i];
  a.n_plob = np;
  a.plob_z = d_pz;
  a.plob_coef = d_pc;
  a.edges = d_edges;
  a.pair_lo = d_plo;
  a.pair_hi = d_phi;
  a.bin_pair = d_bp;
  a.zob_min = d_zmin;
  a.zob_max = d_zmax;
  a.sigma_z = d_sz;
  a.gl_t = d_glt;
  a.gl_w = d_glw;
  a.lnm_out = lnm_dev;
  a.z_out = z_dev;
  a.S_out = S_dev;
  return launch_sel_function(a, chained(plo, phi_, edges.size()), s);
}
