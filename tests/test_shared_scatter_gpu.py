"""The adjoint's scatter by shared columns: element counts (the kernels of six
and of eight elements, a last group of one or two), strips of volume rows, and
shapes on either side of its line; against the FP64 gradient, with path
integrals kept and re-marched."""
import numpy as np
import pytest

import oracle as O
from tests.cases import proj_case, spectrum
from tests.test_march_rule_gpu import _shares
from tests.test_materials_gpu import _case, _mu
from virtualcbct_b200 import Projector

pytestmark = pytest.mark.gpu


def _scatters(g):
    """scatter_shares_columns of the library."""
    half = g.piso * g.dpn / 2.0
    rays, planes = g.step * g.H / (2.0 * half), 32.0 * g.s / g.sad / g.step * half
    inside = planes * min(1.0, g.Z * g.step / 2.0 / half) ** 1.25
    small = g.N * g.N * g.Z < 2e6
    least = max(1.4, 1.7 + 0.9 * (inside - 0.8) if small else 1.4 + 0.75 * (inside - 1.2))
    slices = 32.0 / rays * (1.0 + g.N * g.s / 2.0 / g.sad) + planes + 1.0
    whole = abs(1.0 / g.s - round(1.0 / g.s)) < 1e-6
    return rays >= least and planes <= 2.5 and (not small or slices <= 32.8 or inside <= (0.9 if whole else 1.6))


def _gradients_match(g, tabs, volf, mu, pdf, seed):
    import torch
    resid = np.random.default_rng(seed).normal(size=(g.V, g.H, g.W)).astype(np.float32)
    resid[:, ::5] = 0.0  # rays that do not scatter
    p = Projector(g, *tabs)
    p.set_spectrum(mu, pdf, 1000.0)
    p.load_volume_f32(volf)
    _, L = p.forward_state()
    go = torch.from_numpy(resid).cuda()
    ref = O.mbfpa_adjoint(g, tabs, volf, mu, pdf, 1000.0, resid)
    for got in (p.adjoint_state(L, go), p.adjoint(go)):
        d = got.cpu().numpy().astype(np.float64) - ref
        assert np.linalg.norm(d) <= 1e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("nmat", [1, 2, 4, 5, 7, 8])
def test_element_counts(cuda, nmat):
    g, tabs, vol = _case(nmat, seed=nmat, s=0.1, H=96)
    assert _scatters(g) and _shares(g)
    _gradients_match(g, tabs, vol.astype(np.float32), *_mu(nmat), seed=nmat)


@pytest.mark.parametrize("strips", [2, 3, 5])
@pytest.mark.parametrize("nmat", [6, 8])
def test_row_strips(cuda, monkeypatch, strips, nmat):
    monkeypatch.setenv("VCBCT_ADJ_STRIPS", str(strips))
    g, tabs, vol = _case(nmat, seed=strips, s=0.1, H=96, z_reg=0.0)
    assert _scatters(g)
    _gradients_match(g, tabs, vol.astype(np.float32), *_mu(nmat), seed=strips)


@pytest.mark.parametrize("shares,shape", [
    (True, dict(N=64, s=0.2, Z=6, step=0.5, dpn=1200.0, H=117, W=8, V=2)),    # two planes, most rays leave the slab
    (False, dict(N=64, s=0.2, Z=32, step=0.5, dpn=1200.0, H=117, W=8, V=2)),  # the same slices, more of them
    (True, dict(N=64, s=0.2, Z=32, step=0.5, dpn=1200.0, H=195, W=8, V=2)),   # and more rays to each
    (True, dict(N=210, s=0.1, Z=50, step=0.25, dpn=1200.0, H=234, W=6, V=2)),  # a larger volume
])
def test_both_sides_of_the_line(cuda, shares, shape):
    g, tabs, vol, _ = proj_case("random", seed=9, **shape)
    assert _scatters(g) == shares
    _gradients_match(g, tabs, vol.astype(np.float32), *spectrum(), seed=1)
