"""The projection on either side of the lines where rays stop being walked and
share columns: many z planes along a ray, more slices in a warp than the
column table holds, few planes in a small volume; against the FP64 oracle."""
import numpy as np
import pytest

import oracle as O
from tests.cases import proj_case, spectrum
from virtualcbct_b200 import Projector

pytestmark = pytest.mark.gpu

RTOL = 1e-5  # the projections' parity bar, relative per detector pixel


def _shares(g):
    """march_shares_columns of the library."""
    half = g.piso * g.dpn / 2.0
    rays, per_batch = g.step * g.H / (2.0 * half), 32.0 * g.s / g.sad / g.step
    planes, in_slab = per_batch * half, min(1.0, g.Z * g.step / 2.0 / half)
    inside = planes * in_slab ** 1.25
    slices = 32.0 / rays * (1.0 + g.N * g.s / 2.0 / g.sad) + planes + 1.0
    whole, small = abs(1.0 / g.s - round(1.0 / g.s)) < 1e-6, g.N * g.N * g.Z < 2e6
    if not whole:
        least = min(2.2, 1.15 + 1.5 * (inside - 2.0))
    else:
        least = 1.15 + 1.35 * (inside - 1.3) if small else min(2.6, 1.15 + 2.5 * (inside - 1.5))
    return rays >= max(1.15, least) and (not small or slices <= 32.8 or inside <= (0.9 if whole else 1.6))


@pytest.mark.parametrize("shares,shape", [
    (True, dict(N=64, s=0.2, Z=80, step=0.25, dpn=1600.0, H=666, W=6, V=2)),    # up to six planes per batch of steps
    (False, dict(N=64, s=0.2, Z=80, step=0.25, dpn=1600.0, H=416, W=6, V=2)),   # the same, fewer rays to a slice
    (True, dict(N=64, s=0.23, Z=80, step=0.25, dpn=1600.0, H=480, W=6, V=2)),   # 1 / s not an integer
    (True, dict(N=210, s=0.13, Z=50, step=0.5, dpn=1600.0, H=122, W=6, V=2)),   # batches with more than 32 slices walk
    (True, dict(N=96, s=0.26, Z=14, step=0.5, dpn=800.0, H=60, W=10, V=3)),     # a small volume of few planes
    (False, dict(N=96, s=0.26, Z=44, step=0.5, dpn=800.0, H=60, W=10, V=3)),    # and of more
])
def test_both_sides_of_the_lines_match_fp64_oracle(cuda, shares, shape):
    g, tabs, vol, _ = proj_case("random", seed=3, **shape)
    assert _shares(g) == shares
    mu, pdf = spectrum()
    p = Projector(g, *tabs)
    p.set_spectrum(mu, pdf, 1000.0)
    p.load_volume(vol)
    got = p.forward().cpu().numpy()
    p.load_volume_f32(vol.astype(np.float32))
    assert np.array_equal(p.forward().cpu().numpy(), got)  # both forms, bit for bit
    ref = O.mbfpa_forward(g, tabs, vol, mu, pdf, 1000.0, exact=True, want=("d",))["d"]
    rel = np.abs(got.astype(np.float64) - ref) / ref
    assert rel.max() <= RTOL, f"max rel err {rel.max():.3e} at {np.unravel_index(rel.argmax(), rel.shape)}"
