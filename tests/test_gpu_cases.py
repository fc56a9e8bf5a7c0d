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
