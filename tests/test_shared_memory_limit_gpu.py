"""A kernel's limit of dynamic shared memory is one for all callers: launches
of different sizes, prepared or issued in turn or by several threads, must not
lower it under each other."""
import sys
import threading

import numpy as np
import pytest

from tests.cases import proj_case, spectrum
from virtualcbct_b200 import FILTER_BF16X3, FILTER_DIRECT_F32, Batch, Fdk, FdkGeometry, Projector

pytestmark = pytest.mark.gpu


def _projector(bins, **kw):
    g, tabs, vol, _ = proj_case("random", H=96, **kw)
    mu, pdf = spectrum("spectrum_kramers120_111.csv")
    p = Projector(g, *tabs)
    p.set_spectrum(mu[:, :bins], pdf[:bins], 1000.0)
    p.load_volume(vol)
    return p


@pytest.mark.parametrize("strategy", [Batch.PERSISTENT, Batch.FLAT])
def test_batches_of_other_bin_counts_in_turn(cuda, strategy):
    """The limit a batch was built with survives a batch of fewer bins."""
    batches = []
    for bins in (111, 73):
        p = _projector(bins)
        b = Batch()
        b.add(p)
        b.configure(strategy, 8)
        b.forward(use_graph=False)
        batches.append((p, b))
    for p, b in batches:
        assert np.array_equal(b.forward(use_graph=False)[0].cpu().numpy(), p.forward().cpu().numpy())


def _together(calls, times):
    errors = []

    def work(call):
        try:
            for _ in range(times):
                call()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    assert not errors, errors


@pytest.mark.parametrize("method", [FILTER_DIRECT_F32, FILTER_BF16X3])
def test_threads_filter_detectors_of_other_widths(cuda, method):
    import torch
    calls = []
    for W in (100, 400) * 3:
        f = Fdk(FdkGeometry(W=W, H=8, V=2, N=8, Z=2, zstart=-1, step=0.5, scale=0.4), np.deg2rad([0.0, 180.0]), np.zeros(2),
                np.zeros(2))
        proj, out = torch.full((2, 8, W), 0.5, device=cuda), torch.empty((2, 8, W), device=cuda)
        calls.append(lambda f=f, proj=proj, out=out: f.filter(proj, out, method=method))
    _together(calls, 3000)
    torch.cuda.synchronize()


def test_threads_project_with_other_bin_counts(cuda):
    import torch
    calls = []
    for bins in (111, 73) * 3:
        p = _projector(bins, V=25)  # enough blocks for eight columns each
        out = torch.empty((p.geom.V, p.geom.H, p.geom.W), device=cuda)
        calls.append(lambda p=p, out=out: p.forward(out))
    _together(calls, 1000)
    torch.cuda.synchronize()
