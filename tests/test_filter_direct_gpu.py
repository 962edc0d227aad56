"""The direct FP32 ramp filter at the widths and row counts where its column
passes, stages and blocks change, against the FP64 filter."""
import numpy as np
import pytest

import oracle as O
from virtualcbct_b200 import Fdk, FdkGeometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,H,W", [(2, 2, 2), (3, 7, 31), (2, 33, 33), (5, 64, 64), (3, 45, 193), (3, 50, 225), (2, 66, 257),
                                   (2, 31, 400), (4, 40, 521), (40, 250, 65), (150, 129, 97), (2, 9, 1030)])
def test_direct_filter_matches_fp64(cuda, V, H, W):
    rng = np.random.default_rng(W)
    proj = rng.uniform(0.02, 1.0, size=(V, H, W)).astype(np.float32)
    geom = FdkGeometry(W=W, H=H, V=V, N=8, Z=2, zstart=-1, step=0.5, scale=0.4)
    ang, xs, ys = np.deg2rad(np.arange(V) * 360.0 / V), np.full(V, 2.0), np.zeros(V)
    got = Fdk(geom, ang, xs, ys).filter(proj)
    ref = O.filter_sinogram(proj, xs, ys, O.fdk_consts(geom.piso), mode=1)
    # one float rounding per fused multiply-add of a W-term chain, and a few
    # for the logarithm, the coefficient and the cosine factor (at most 1):
    # bounded by the terms' magnitudes
    consts = O.fdk_consts(geom.piso)
    h = np.abs(O.const_map(W, consts)) + abs(O.filter_coeff(W, consts)) * np.eye(W)
    bound = (W + 10) * 2.0 ** -24 * (np.abs(np.log(proj.astype(np.float64))) @ h.T)
    assert (np.abs(got - ref) <= bound).all()


@pytest.mark.parametrize("V,H,W", [(40, 250, 200), (48, 200, 256), (40, 250, 193)])
def test_staged_rows_serve_every_column_pass(cuda, V, H, W):
    """Two column passes a block over rows that stay in shared memory (193 to 256
    columns, more row blocks than SMs): each row filtered as in a stack that
    gives every pass a block of its own."""
    import torch
    assert V * H > 64 * 148
    proj = torch.rand((V, H, W), generator=torch.Generator().manual_seed(W)).mul_(0.98).add_(0.02).cuda()
    ang, xs, ys = np.deg2rad(np.arange(V) * 360.0 / V), np.full(V, 2.0), np.zeros(V)
    geom = dict(H=H, W=W, N=8, Z=2, zstart=-1, step=0.5, scale=0.4)
    got = Fdk(FdkGeometry(V=V, **geom), ang, xs, ys).filter(proj)
    few = Fdk(FdkGeometry(V=8, **geom), ang[:8], xs[:8], ys[:8])
    for v in range(0, V, 8):
        assert torch.equal(got[v:v + 8], few.filter(proj[v:v + 8].contiguous()))
    ref = O.filter_sinogram(proj[:2].cpu().numpy(), xs[:2], ys[:2], O.fdk_consts(few.geom.piso), mode=1)
    consts = O.fdk_consts(few.geom.piso)
    h = np.abs(O.const_map(W, consts)) + abs(O.filter_coeff(W, consts)) * np.eye(W)
    bound = (W + 10) * 2.0 ** -24 * (np.abs(np.log(proj[:2].cpu().numpy().astype(np.float64))) @ h.T)
    assert (np.abs(got[:2].cpu().numpy() - ref) <= bound).all()
