"""The entry points of perf/cases.py at the edges of their kernels' tiles and
rules, against that file's 64-bit restatements.  FP64 outputs: 1e-9 of each
output's scale (the restatements resolve the chi(z) bisections to 2^-40, the
largest difference); mixed-form outputs: 1e-4, the engine's stated bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compare(case, tol, seed=3):
    import torch

    from perf import cases

    state = cases.prepare(case, seed)
    got = cases.run(state)
    torch.cuda.synchronize()
    got = got if isinstance(got, list) else [got]
    want = cases.exact(case, seed)
    want = want if isinstance(want, list) else [want]
    assert len(got) == len(want)
    for g, w in zip(got, want):
        g = np.asarray(g.cpu() if hasattr(g, "cpu") else g)
        w = np.asarray(w.cpu() if hasattr(w, "cpu") else w)
        assert g.shape == w.shape and np.all(np.isfinite(g))
        np.testing.assert_allclose(g, w, rtol=0, atol=tol * np.max(np.abs(w)))


# Masses are summed in groups of eight; one radius leaves the widest theta
# segments (short ring rules), ten the narrowest (long ones near the radii).
@pytest.mark.parametrize("n_lnm,radii,n_per_seg", [(1, 1, 3), (7, 2, 9), (8, 3, 8), (9, 10, 17),
                                                   (33, 4, 5)])
def test_projection_shear_by_quadrature(gpu, n_lnm, radii, n_per_seg):
    _compare(dict(kind="prj", radii=radii, n_lnm=n_lnm, n_per_seg=n_per_seg, n_zring=7,
                  n_zouter=9), 1e-9)


# 33 masses: a partial last group of eight; the distinct (R_mis, R) pairs are
# shared by the z_obs bins; radii from 0.1 to 30 cover both quadrature forms.
@pytest.mark.parametrize("mor,n_lnm,radii", [("hod", 2, 1), ("lognormal", 33, 4), ("hod", 96, 15)])
def test_module_chain(gpu, mor, n_lnm, radii):
    _compare(dict(kind="module", mor=mor, tab_m=40, tab_z=24, n_q=17, n_lnm=n_lnm, n_z=19,
                  radii=radii), 1e-9)


# The FP64 form: lnM tiles of 64 rows, groups of 32 z_t columns and stages of
# 16 lam_t nodes, whole and with remainders; more points than one workspace
# round (128); both table ends of the radii, and no shear.
@pytest.mark.parametrize("n,n_m,n_z,n_t,radii", [(1, 33, 16, 40, 15), (3, 64, 32, 64, 1),
                                                 (5, 65, 48, 97, 2), (2, 130, 16, 33, 0),
                                                 (3, 256, 128, 256, 0), (1, 2, 16, 2, 0),
                                                 (150, 40, 16, 48, 0)])
def test_fp64_engine(gpu, n, n_m, n_z, n_t, radii):
    _compare(dict(kind="engine", api="device", precision="fp64", n=n, radii=radii, hmf_fp32=False,
                  loglike=False, mixed_density=False, n_m=n_m, n_z=n_z, n_t=n_t, n_o=32, n_zo=9),
             1e-11)


def test_fp64_shear_outside_the_profile_table(gpu):
    """Omega_m = 60 lies beyond the profile table (0.01 to 1, widened by 1.5
    in x): such a point takes the direct quadrature, next to others that do
    not.  With Sigma_crit^-1 = 1 the shear is the weighted sum of
    y3b_nfw_mis profiles over the mass weights; both sides sum ~33 FP64 terms
    of profiles good to ~1e-14."""
    from perf import cases
    from y3_cluster_cpp_b200 import engine as E
    from y3_cluster_cpp_b200 import synthetic

    pts = [synthetic.fiducial(1) for _ in range(3)]
    for p in pts:
        p.tables["sci_val"] = np.ones_like(p.tables["sci_val"])
    pts[1].om = 60.0
    g = synthetic.grid(1, n_m=33, n_z=16, n_t=40, n_o=16, n_zo=8)
    so = synthetic.shear_opts(n_theta=16, n_s=32, n_R=4)
    t = pts[0].tables
    eng = E.Engine([g], len(t["hmf_m_h"]), len(t["hmf_z"]), len(t["dist_z"]),
                   synthetic.plob_baseline(), max_points=3, n_sci=len(t["sci_z"]), shear=so)
    out = eng.eval(pts, E.FP64, grid_of=lambda p: 0, weights=True)
    lnM, wm = (v.cpu().numpy() for v in cases._gl(g["lnm_lo"], g["lnm_hi"], 33))
    conc = so["c0"] * (np.exp(lnM) / so["c_pivot"]) ** so["c_slope"]
    for p in range(3):
        want = np.zeros((12, 4))
        for k in range(33):
            rho = cases.RHO_CRIT * pts[p].om
            cen = E.nfw_mis("dsigma_single", so["R"], 1e-9, lnM[k], conc[k], rho, 16, 32, 20.0)
            for i in range(4):
                rmis = so["tau_mis"] * (so["lob_centers"][i] / 100) ** 0.2
                mis = E.nfw_mis("dsigma", so["R"], rmis, lnM[k], conc[k], rho, 16, 32, 20.0)
                phi = (1 - so["f_mis"]) * cen + so["f_mis"] * mis
                for b in range(i, 12, 4):
                    want[b] += wm[k] * out["W"][p, b, k] * phi
        np.testing.assert_allclose(out["shear"][p], want, rtol=1e-11)
    eng.close()


# Few samples split a grid point's theta nodes over blocks, many do not; one
# and two theta nodes (no split at theta_lob), node counts that leave partial
# warps of (z, lambda_true) pairs and odd z grids.
@pytest.mark.parametrize("n,n_lt,n_zring,n_zouter,n_lnm,n_theta,n_zt_ref", [
    (1, 60, 20, 30, 24, 10, 80), (3, 7, 5, 3, 9, 2, 40), (40, 31, 9, 15, 13, 5, 33),
    (2, 1, 20, 30, 24, 3, 64)])
def test_selection_bias(gpu, n, n_lt, n_zring, n_zouter, n_lnm, n_theta, n_zt_ref):
    _compare(dict(kind="bsel", n=n, n_lt=n_lt, n_zring=n_zring, n_zouter=n_zouter, n_lnm=n_lnm,
                  n_theta=n_theta, n_zt_ref=n_zt_ref), 1e-10)


# The mixed form's stacked shear: 12 bins take whole passes of 4 x 3; one
# point, several per warp, node sets of different sizes in one call.
@pytest.mark.parametrize("n,radii,mixed", [(1, 1, False), (45, 15, False), (40, 4, True)])
def test_mixed_shear(gpu, n, radii, mixed):
    _compare(dict(kind="engine", api="device", precision="mixed", n=n, radii=radii, hmf_fp32=False,
                  loglike=radii == 15, mixed_density=mixed, n_m=70, n_z=32, n_t=64, n_o=32,
                  n_zo=9), 1e-4)


@pytest.mark.parametrize("nI,nJ", [(1, 1), (3, 2), (5, 4), (8, 3)])
def test_mixed_shear_bin_layouts(gpu, nI, nJ):
    """Bin counts that leave partial passes of richness and z_obs bins, against
    the engine's FP64 form (the mixed form's bound, 1e-4)."""
    from y3_cluster_cpp_b200 import engine as E
    from y3_cluster_cpp_b200 import synthetic

    g = synthetic.grid(1, n_m=40, n_z=16, n_t=64, n_o=16, n_zo=8,
                       lam_edges=np.geomspace(20.0, 200.0, nI + 1),
                       zob_edges=np.linspace(0.2, 0.65, nJ + 1))
    so = synthetic.shear_opts(n_theta=16, n_s=32, n_R=3)
    so["lob_centers"] = np.geomspace(25.0, 130.0, nI)
    pts = synthetic.walkers(5, seed=4, densities=(1,))
    t = pts[0].tables
    eng = E.Engine([g], len(t["hmf_m_h"]), len(t["hmf_z"]), len(t["dist_z"]),
                   synthetic.plob_baseline(), max_points=5, n_sci=len(t["sci_z"]), shear=so)
    a = eng.eval(pts, E.MIXED, grid_of=lambda p: 0)
    b = eng.eval(pts, E.FP64, grid_of=lambda p: 0)
    for k in ("counts", "shear"):
        assert a[k].shape == b[k].shape and np.all(np.isfinite(a[k]))
        np.testing.assert_allclose(a[k], b[k], rtol=1e-4)
    eng.close()


# The mixed form's lnM tiles: one group of 32 rows, two, four, and a second
# tile with a remainder; z rows that leave warps of the factor kernel short or
# without work; FP32 and FP64 HMF tables.
@pytest.mark.parametrize("n_m,n_z,n_t,hmf_fp32", [(20, 16, 32, False), (32, 16, 64, True),
                                                  (33, 48, 40, False), (64, 32, 64, True),
                                                  (65, 80, 96, False), (128, 16, 33, True),
                                                  (129, 112, 64, False), (161, 128, 160, True),
                                                  (193, 32, 256, False)])
def test_mixed_row_groups(gpu, n_m, n_z, n_t, hmf_fp32):
    _compare(dict(kind="engine", api="device", precision="mixed", n=3, radii=0, hmf_fp32=hmf_fp32,
                  loglike=False, mixed_density=False, n_m=n_m, n_z=n_z, n_t=n_t, n_o=32, n_zo=9),
             1e-4)


# The miscentred profile at 24 Chebyshev nodes in lnM (grids above 32 masses on
# at most nine e-folds) and at every mass on the rule's other side, against the
# closed-form profile's quadrature at every mass, which cancels to about 1e-12
# of itself near r_s: 1e-10.
@pytest.mark.parametrize("n_lnm,lo,hi", [(33, 29.9336, 36.73), (96, 27.9, 36.9), (200, 31.0, 31.5),
                                         (96, 27.8, 36.9), (32, 29.9336, 36.73)])
def test_miscentred_profile_nodes(gpu, n_lnm, lo, hi):
    from perf import cases
    from y3_cluster_cpp_b200 import engine as E

    s = cases._module_inputs(dict(mor="lognormal", tab_m=40, tab_z=24, n_q=17, radii=4), 3)
    sel = E.sel_function(s["cfg"], s["kind"], s["mor"], *s["plob"])
    h = E.SelGL(n_lnm=n_lnm, n_z=19, lnm_low=lo, lnm_high=hi).build(s["cz"], s["tab"], sel)
    w = h.weights()
    got = h.shear(s["bins"], s["r"], s["halo"], f_mis=1.0)
    rmis = 0.17 * (np.array((25.0, 37.5, 52.5, 130.0))[s["bins"] % 4] / 100.0) ** 0.2
    prof = E.nfw_mis("dsigma", s["r"][:, None], rmis[:, None], w["lnm_x"], 4.0, cases.RHO_CRIT)
    want = s["om"] * np.sum(w["lnm_w"] * w["W"][s["bins"]] * prof, axis=1)
    np.testing.assert_allclose(got, want, rtol=1e-10, atol=1e-10 * np.max(np.abs(want)))


# The profile at 16 Chebyshev nodes in lnM starts at 17 masses.  By the rule's
# bound its error is 1e-13 of the profile; 1e-9 is the restatement's.
@pytest.mark.parametrize("n_lnm,radii", [(16, 3), (17, 3), (24, 10), (40, 2)])
def test_projection_shear_profile_nodes(gpu, n_lnm, radii):
    _compare(dict(kind="prj", radii=radii, n_lnm=n_lnm, n_per_seg=6, n_zring=8, n_zouter=8), 1e-9)


@pytest.mark.parametrize("hmf_fp32", [False, True])
def test_points_given_up_by_their_tables(gpu, hmf_fp32):
    """A non-finite table entry of a point whose scratch holds another grid's
    values (the engine ran the larger grid before, in every form it has) gives
    the domain error, and the next call gives what a fresh engine gives."""
    from y3_cluster_cpp_b200 import _capi, synthetic
    from y3_cluster_cpp_b200 import engine as E

    grids = [synthetic.grid(4), synthetic.grid(1, n_m=33, n_z=16, n_t=40, n_o=16, n_zo=8)]
    so = synthetic.shear_opts(n_theta=16, n_s=32, n_R=3)
    pts = synthetic.walkers(3, seed=8, densities=(1,))
    t = pts[0].tables
    precs = (E.MIXED,) if hmf_fp32 else (E.MIXED, E.FP64)

    def engine():
        return E.Engine(grids, len(t["hmf_m_h"]), len(t["hmf_z"]), len(t["dist_z"]),
                        synthetic.plob_baseline(), max_points=3, n_sci=len(t["sci_z"]), shear=so,
                        hmf_fp32=hmf_fp32)

    eng, fresh = engine(), engine()
    want = {p: fresh.eval(pts, p, grid_of=lambda _: 1) for p in precs}
    for where in ("dndlnmh", "dist_da", "hmf_z"):
        for p in precs:
            eng.eval(pts, p, grid_of=lambda _: 0)
        bad = synthetic.walkers(3, seed=8, densities=(1,))
        bad[1].tables[where] = np.array(bad[1].tables[where], copy=True)
        bad[1].tables[where].flat[3] = np.nan
        for p in precs:
            with pytest.raises(_capi.Y3BError) as err:
                eng.eval(bad, p, grid_of=lambda _: 1)
            assert err.value.status == _capi.ERR_DOMAIN
            got = eng.eval(pts, p, grid_of=lambda _: 1)
            for k in ("counts", "shear"):
                np.testing.assert_array_equal(got[k], want[p][k])
    eng.close()
    fresh.close()


def test_fp64_bins_far_from_every_mass(gpu):
    """Mass-richness relations that leave richness bins many sigma above every
    mass, with a P(lambda_o | lambda_t) without projection tail: small positive
    counts, not zero, down to the bins that no factor holds.  An exponent of
    up to 600 is rounded to 1e-13 of itself on both sides, mu (in 1 / sigma per
    sigma) to 3e-13: 1e-11."""
    import oracle
    from y3_cluster_cpp_b200 import engine as E
    from y3_cluster_cpp_b200 import synthetic

    pz, pc = synthetic.plob_baseline()
    pc = np.array(pc).reshape(8, -1)
    pc[7] = 0.0
    g = synthetic.grid(1, n_m=64, n_z=16, n_t=256, n_o=32, n_zo=8)
    pts = []
    for sigma in (0.05, 0.1, 0.2):
        for A in (-0.5, 0.5, 1.5, 2.5, 3.2):
            p = synthetic.fiducial(1)
            p.A, p.sigma = A, sigma
            pts.append(p)
    t = pts[0].tables
    eng = E.Engine([g], len(t["hmf_m_h"]), len(t["hmf_z"]), len(t["dist_z"]), (pz, pc.ravel()),
                   max_points=len(pts))
    got = eng.eval(pts, E.FP64, grid_of=lambda _: 0)["counts"]
    want = np.array([oracle.direct_eval(g, pz, pc.ravel(), p.mor, oracle.cosmo(p.om, p.h0),
                                        p.tables)[0] for p in pts])
    assert np.all(want > 0) and want.min() < 1e-200
    np.testing.assert_allclose(got, want, rtol=1e-11)
    eng.close()


@pytest.mark.parametrize("n_lnm", [21, 24, 40])
@pytest.mark.parametrize("peak", [30.5, 33.1, 35.5])
def test_projection_profile_nodes_against_every_mass(gpu, n_lnm, peak):
    """The profile at Chebyshev nodes of lnM (six e-folds, the widest range of
    the rule) against the profile at every mass (the next double above it),
    with an HMF of one narrow peak, so that few masses carry the sums and the
    interpolation's error is not averaged.  The mass nodes of the two differ by
    1e-16 of themselves; interpolation and the ring sums' rounding leave 1e-14
    of a profile: 5e-14 of the largest output of each channel."""
    from perf import cases
    from y3_cluster_cpp_b200 import engine as E

    om, t, p, grid = cases._prj_inputs(dict(radii=6), 5)
    lnm = np.log(t["hmf_m_h"] * om)
    t = dict(t, dndlnmh=t["dndlnmh"] * (np.abs(lnm - peak) < 0.15))
    kw = dict(n_lnm=n_lnm, n_per_seg=6, n_zring=8, n_zouter=8, lnm_low=30.0)
    cz = E.cosmo(om, cases.H0)
    nodes = E.PrjShear(grid, lnm_high=36.0, **kw).eval(cz, t, p)
    every = E.PrjShear(grid, lnm_high=np.nextafter(36.0, 40.0), **kw).eval(cz, t, p)
    for c in range(3):
        np.testing.assert_allclose(nodes[:, c], every[:, c], rtol=0,
                                   atol=5e-14 * np.max(np.abs(every[:, c])))


@pytest.mark.parametrize("peak", [28.2, 30.0, 36.5])
@pytest.mark.parametrize("n_lnm", [33, 96])
def test_miscentred_profile_nodes_against_every_mass(gpu, n_lnm, peak):
    """The module's profile at Chebyshev nodes of lnM (nine e-folds, the widest
    range of the rule) against the profile at every mass (the next double above
    it), with a selection of one narrow mass peak.  Per unit number count: the
    mass nodes of the two differ by their rounding, which the selection's ramps
    turn into 4e-14 of the mass weights, alike for every radius.  The sums of
    the two sides are rounded alike; 2e-14 of each value is ten times the
    interpolation."""
    from perf import cases
    from y3_cluster_cpp_b200 import engine as E

    s = cases._module_inputs(dict(mor="lognormal", tab_m=40, tab_z=24, n_q=17, radii=6), 3)
    lnm, z = np.linspace(28.0, 37.0, 181), np.linspace(0.05, 0.8, 9)
    S = np.tile((np.abs(lnm - peak) < 0.2).astype(float), (12, 9, 1))
    got = []
    for hi in (37.0, np.nextafter(37.0, 40.0)):
        h = E.SelGL(n_lnm=n_lnm, n_z=19, lnm_low=28.0, lnm_high=hi).build(s["cz"], s["tab"],
                                                                          (lnm, z, S))
        got.append(h.shear(s["bins"], s["r"], s["halo"], f_mis=1.0) /
                   h.weights()["norm"][s["bins"]])
    assert np.all(got[1] != 0)
    np.testing.assert_allclose(got[0], got[1], rtol=2e-14)


def test_engines_of_different_bin_counts_side_by_side(gpu):
    """An engine made later, with smaller tiles and tables, takes no shared
    memory away from the launches of an earlier one."""
    from y3_cluster_cpp_b200 import engine as E
    from y3_cluster_cpp_b200 import synthetic

    pts = synthetic.walkers(3, seed=4, densities=(1,))
    t = pts[0].tables

    def engine(nI, n_z):
        g = synthetic.grid(1, n_m=40, n_z=n_z, n_t=64, n_o=16, n_zo=8,
                           lam_edges=np.geomspace(20.0, 200.0, nI + 1))
        so = synthetic.shear_opts(n_theta=16, n_s=32, n_R=3)
        so["lob_centers"] = np.geomspace(25.0, 130.0, nI)
        return E.Engine([g], len(t["hmf_m_h"]), len(t["hmf_z"]), len(t["dist_z"]),
                        synthetic.plob_baseline(), max_points=3, n_sci=len(t["sci_z"]), shear=so)

    first = engine(8, 128)
    want = first.eval(pts, E.MIXED, grid_of=lambda p: 0)
    second = engine(1, 16)
    second.eval(pts, E.MIXED, grid_of=lambda p: 0)
    for prec in (E.MIXED, E.FP64):
        got = first.eval(pts, prec, grid_of=lambda p: 0)
        for k in ("counts", "shear"):
            np.testing.assert_allclose(got[k], want[k], rtol=0 if prec == E.MIXED else 1e-4)
    first.close()
    second.close()


# The masses' factors stand in shared memory 320 at a time: whole tiles, a
# remainder, several tiles, and more (bin, lambda_true) pairs than threads.
@pytest.mark.parametrize("n_lnm,n_lt", [(320, 5), (321, 5), (400, 70), (1900, 3)])
def test_selection_bias_many_masses(gpu, n_lnm, n_lt):
    _compare(dict(kind="bsel", n=2, n_lt=n_lt, n_zring=4, n_zouter=3, n_lnm=n_lnm, n_theta=3,
                  n_zt_ref=12), 1e-10)


# lambda_true tables that do not fit in shared memory beside the mass sums.
@pytest.mark.parametrize("n_lt,n_zring,n_zouter", [(4500, 1, 1), (2600, 3, 1)])
def test_selection_bias_many_richness_nodes(gpu, n_lt, n_zring, n_zouter):
    _compare(dict(kind="bsel", n=1, n_lt=n_lt, n_zring=n_zring, n_zouter=n_zouter, n_lnm=5,
                  n_theta=2, n_zt_ref=12), 1e-10)


def test_selection_bias_pieces_of_a_batch(gpu):
    """A batch is evaluated in pieces of a chunk: two unequal pieces, chunks of
    several pieces with a short last chunk, then smaller and larger batches on
    the same handles (reused work blocks).  With one theta node a grid point's
    terms are dealt to the warps alike in every batch: bit for bit the samples
    one at a time."""
    from perf import cases
    from y3_cluster_cpp_b200 import engine as E

    nodes = dict(n_lt=5, n_zring=4, n_zouter=3, n_lnm=6, n_theta=1, n_zt_ref=12)
    state = cases.prepare(dict(kind="bsel", n=130, **nodes), 7)
    samples, whole = state["samples"], state["h"]
    want = np.concatenate([whole.eval([s]) for s in samples])
    grid = dict(zo_low=np.repeat(cases.ZOB_EDGES[:3], 4), zo_high=np.repeat(cases.ZOB_EDGES[1:], 4),
                lambda_bin=np.tile(np.arange(4), 3))
    chunked = E.BselMarg(grid, *cases.LNM, max_samples=60, **nodes)
    for h in (whole, chunked):
        for a, b in ((0, 53), (0, 130), (53, 60), (3, 128), (129, 130)):
            np.testing.assert_array_equal(h.eval(samples[a:b]), want[a:b])
    chunked.close()


@pytest.mark.parametrize("c_slope,R_lo,R_hi,rtol", [(-0.1, 0.1, 30.0, 1e-14),
                                                    (-0.1, 0.1, 1e6, 2e-14),
                                                    (-1.5, 10.0, 1e8, 2e-13)])
def test_fp64_shear_profile_interpolation(gpu, c_slope, R_lo, R_hi, rtol):
    """The centred profile (f_mis = 0) of the FP64 form over the radii's usual
    range, over one that makes the table three times as coarse as that, and
    past the spacing that is interpolated, against 40-digit values summed with
    the engine's own mass weights (Sigma_crit^-1 = 1).  The closed form (at x
    above 0.1, where it keeps its digits) and the sum of 33 positive terms leave
    about 5e-15; the last case's concentrations near 0.03 cost its normalisation
    two digits more."""
    import mpmath as mp

    from perf import cases
    from y3_cluster_cpp_b200 import engine as E
    from y3_cluster_cpp_b200 import synthetic

    p = synthetic.fiducial(1)
    p.tables["sci_val"] = np.ones_like(p.tables["sci_val"])
    g = synthetic.grid(1, n_m=33, n_z=16, n_t=40, n_o=16, n_zo=8)
    so = synthetic.shear_opts(n_theta=16, n_s=32, n_R=7)
    so.update(R=np.geomspace(R_lo, R_hi, 7), c_slope=c_slope, f_mis=0.0)
    t = p.tables
    eng = E.Engine([g], len(t["hmf_m_h"]), len(t["hmf_z"]), len(t["dist_z"]),
                   synthetic.plob_baseline(), max_points=1, n_sci=len(t["sci_z"]), shear=so)
    out = eng.eval([p], E.FP64, grid_of=lambda _: 0, weights=True)
    eng.close()
    lnM, wm = (v.cpu().numpy() for v in cases._gl(g["lnm_lo"], g["lnm_hi"], 33))

    def profile(R, x):
        M = mp.exp(mp.mpf(x))
        c = so["c0"] * (M / so["c_pivot"]) ** mp.mpf(c_slope)
        rho = mp.mpf(cases.RHO_CRIT) * mp.mpf(p.om)
        rs = mp.cbrt(3 * M / (800 * mp.pi * rho)) / c
        delta = mp.mpf(200) / 3 * c ** 3 / (mp.log(1 + c) - c / (1 + c))
        q = mp.mpf(R) / rs
        v = 1 - q * q
        y = mp.sqrt(abs(v))
        gq = mp.atan(y) / y if q > 1 else mp.log((1 + y) / q) / y
        return 2 * rs * delta * rho * mp.mpf("1e-12") * (2 * (gq + mp.log(q / 2)) / q ** 2
                                                         - (gq - 1) / v)

    with mp.workdps(40):
        prof = [[profile(R, x) for x in lnM] for R in so["R"]]
        want = np.array([[float(sum(mp.mpf(w) * mp.mpf(k) * f for w, k, f in
                                    zip(out["W"][0, b], wm, row))) for row in prof]
                         for b in range(12)])
    np.testing.assert_allclose(out["shear"][0], want, rtol=rtol)


@pytest.mark.parametrize("seed", range(4))
def test_fp64_product_against_direct_sum(gpu, seed):
    """The FP64 form's matrix product, where its bounds admit a point, against
    the direct sum (an engine whose memory budget leaves the product no
    workspace), over node counts, bin layouts, scatters from 0.03 to 0.6 and
    mass-richness relations that leave bins out of reach: the direct sum's
    rounding of mu leaves 1e-14 of a cell, 2e-14 of a count."""
    import re

    from y3_cluster_cpp_b200 import _capi, prj_params, synthetic
    from y3_cluster_cpp_b200 import engine as E

    r = np.random.default_rng(seed)
    g = synthetic.grid(1, n_m=int(r.integers(2, 200)), n_z=16 * int(r.integers(1, 5)),
                       n_t=int(r.integers(20, 260)), n_o=16, n_zo=8,
                       lam_edges=np.geomspace(10, 200, int(r.integers(2, 7))),
                       zob_edges=np.linspace(0.2, 0.65, int(r.integers(2, 6))))
    plob = synthetic.plob_baseline() if seed % 2 else prj_params.default_table()
    pts = [synthetic.fiducial(1) for _ in range(10)]
    for p in pts:
        p.sigma = float(np.exp(r.uniform(np.log(0.03), np.log(0.6))))
        p.A, p.B, p.C = r.uniform(-1, 5), r.uniform(0.3, 1.5), r.uniform(-1, 1.5)
    t = pts[0].tables

    def engine(budget):
        return E.Engine([g], len(t["hmf_m_h"]), len(t["hmf_z"]), len(t["dist_z"]), plob,
                        max_points=10, n_sci=len(t["sci_z"]), hbm_budget=budget)

    with pytest.raises(_capi.Y3BError) as err:
        engine(1)
    direct = engine(int(re.search(r"(\d+) bytes for", str(err.value)).group(1)))
    product = engine(0)
    want = direct.eval(pts, E.FP64, grid_of=lambda _: 0)["counts"]
    got = product.eval(pts, E.FP64, grid_of=lambda _: 0)["counts"]
    assert np.all(want > 0)
    np.testing.assert_allclose(got, want, rtol=2e-14)
    direct.close()
    product.close()


@pytest.mark.parametrize("edges", [(20, 30, 45, 60, 200), (5, 10, 15, 20, 25, 30, 40, 60, 100),
                                   (5, 10, 15, 20, 25, 30, 40, 60, 100, 200)])
def test_selection_bins_in_and_out_of_order(gpu, edges):
    """Bins that follow one another (at most nine edges) take their CDF
    differences from registers, others from arrays: the same table, by a few
    roundings of its largest value, from the bins in reverse."""
    from perf import cases
    from y3_cluster_cpp_b200 import engine as E

    s = cases._module_inputs(dict(mor="hod", tab_m=20, tab_z=9, n_q=17, radii=2), 3)
    e = np.array(edges, dtype=float)
    bins = dict(lam_min=e[:-1], lam_max=e[1:], zob_min=np.full(len(e) - 1, 0.2),
                zob_max=np.full(len(e) - 1, 0.35), sigma_z=np.full(len(e) - 1, 0.01))
    a = E.sel_function(dict(s["cfg"], **bins), s["kind"], s["mor"], *s["plob"])[2]
    b = E.sel_function(dict(s["cfg"], **{k: v[::-1].copy() for k, v in bins.items()}), s["kind"],
                       s["mor"], *s["plob"])[2]
    np.testing.assert_allclose(a[::-1], b, rtol=0, atol=1e-15 * a.max())
