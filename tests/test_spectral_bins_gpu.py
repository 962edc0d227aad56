"""Sums over an odd or even number of spectral bins: rays that no radiation
gets through (infinite path integrals), and path integrals near the largest
float."""
import numpy as np
import pytest

import oracle as O
from tests.cases import proj_case, spectrum
from virtualcbct_b200 import Projector

pytestmark = pytest.mark.gpu


def _case(bins, H, **kw):
    g, tabs, vol, _ = proj_case("random", seed=4, H=H, **kw)
    mu, pdf = spectrum()
    b = (len(pdf) - bins) // 2  # the first bins hardly pass this phantom
    mu, pdf = mu[:, b:b + bins], pdf[b:b + bins]
    p = Projector(g, *tabs)
    p.set_spectrum(mu, pdf, 1000.0)
    return g, tabs, vol.astype(np.float32), mu, pdf, p


@pytest.mark.parametrize("H", [16, 96])  # rays on their own; shared columns and scatter
@pytest.mark.parametrize("bins", [1, 89, 90])
def test_rays_through_an_infinite_voxel_are_dark_and_scatter_nothing(cuda, bins, H):
    import torch
    g, tabs, vol, mu, pdf, p = _case(bins, H)
    y, x = 37, 30  # in every slice: 16 rows leave slices out
    one = np.zeros_like(vol)
    one[:, 2, y, x] = 1.0
    p.load_volume_f32(one)
    through = p.path_integrals().cpu().numpy()[..., 2] > 0.0
    assert through.any() and not through.all()
    p.load_volume_f32(vol)
    clear = p.forward().cpu().numpy()
    bad = vol.copy()
    bad[:, 2, y, x] = np.inf
    p.load_volume_f32(bad)
    out, L = p.forward_state()
    got = out.cpu().numpy()
    assert (got[through] == 0.0).all()
    assert np.array_equal(got[~through], clear[~through])
    # such a ray's derivative is 0 in every bin: the gradient is that of the others
    resid = np.random.default_rng(1).normal(size=(g.V, g.H, g.W)).astype(np.float32)
    ref = O.mbfpa_adjoint(g, tabs, vol, mu, pdf, 1000.0, np.where(through, 0.0, resid))
    go = torch.from_numpy(resid).cuda()
    for grad in (p.adjoint_state(L, go), p.adjoint(go)):
        d = grad.cpu().numpy().astype(np.float64) - ref
        assert np.linalg.norm(d) <= 1e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("xfactor", [1000.0, 40.0, 15.0])  # all sums above the floor; most; few
def test_a_heavy_spectrum_keeps_its_weakest_sums(cuda, xfactor):
    """Which sums are done again follows the spectrum's own weight, here 2^30."""
    g, tabs, vol, mu, pdf, p = _case(90, 64)
    p.load_volume_f32(vol)
    pdf = pdf * np.float32(2.0 ** 30)
    p.set_spectrum(mu, pdf, xfactor)
    got = p.forward().cpu().numpy().astype(np.float64) / 2.0 ** 30
    ref = O.mbfpa_forward(g, tabs, None, mu, pdf, xfactor, volf=vol, exact=True, want=("d",))["d"] / 2.0 ** 30
    ok = ref > 1e-36
    # a float exponent T is off by a few of its last places: the path
    # integrals (1e-7 each), the products and the scaling
    T = 1.0 - np.log(ref[ok])
    assert ok.any() and (np.abs(got[ok] - ref[ok]) <= (16 * T + 40) * 2.0 ** -24 * ref[ok]).all()


@pytest.mark.parametrize("bins", [89, 90])
def test_finite_path_integrals_near_the_largest_float(cuda, bins):
    """An element without attenuation whose path integrals are finite, but not
    once they are scaled to base 2, changes nothing."""
    g, tabs, vol, mu, pdf, p = _case(bins, 96, N=16, s=3.0)
    mu = mu.copy()
    mu[2] = 0.0
    p.set_spectrum(mu, pdf, 1000.0)
    vol[:, 2] = 0.0
    p.load_volume_f32(vol)
    want = p.forward().cpu().numpy()
    vol[:, 2, 7, 8] = 8.4e37  # 3.0 to 3.2 cm of a ray that crosses the whole voxel
    p.load_volume_f32(vol)
    L = p.path_integrals().cpu().numpy()[..., 2]
    assert np.isfinite(L).all() and L.max() > 2.36e38
    # the same sums by two exponentials, each within 2 places of float at
    # exponents of at most a few, and their 90-term sums
    assert np.abs(p.forward().cpu().numpy() / want - 1.0).max() <= 2e-6
