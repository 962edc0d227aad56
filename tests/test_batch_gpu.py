"""Batched projection: uneven phantoms in one persistent launch, in one flat
launch or as per-item launches on graph branches (and their CUDA-graph
replay) give exactly the per-phantom results, and each strategy's output of
every item agrees with the FP64 oracle; more items than one launch's
parameter block holds take several launches."""
import numpy as np
import pytest

import oracle as O
from tests.cases import proj_case, spectrum
from virtualcbct_b200 import Batch, Projector

pytestmark = pytest.mark.gpu


RTOL = 1e-5  # projections: relative, per detector pixel


def _projector(cuda, kind, seed, keep=False, **kw):
    import torch
    g, tabs, vol, _ = proj_case(kind, seed=seed, **kw)
    mu, pdf = spectrum()
    p = Projector(g, *tabs)
    p.set_spectrum(mu, pdf, 1000.0)
    p.load_volume(torch.from_numpy(vol.view(np.int16)).to(cuda))
    if keep:
        p.case = (g, tabs, vol, mu, pdf)
    return p


def test_every_strategy_matches_the_fp64_oracle(cuda):
    import torch
    ps = [_projector(cuda, "ellipsoid", 5, keep=True, N=48, Z=12, V=3, W=40, H=36),
          _projector(cuda, "random", 6, keep=True, N=40, Z=20, V=2, W=33, H=41, xshift=0.4),
          _projector(cuda, "water", 0, keep=True, N=56, Z=10, V=4, W=24, H=24)]
    refs = []
    for p in ps:
        g, tabs, vol, mu, pdf = p.case
        refs.append(O.mbfpa_forward(g, tabs, vol, mu, pdf, 1000.0, exact=False, want=("d",))["d"])
    b = Batch()
    outs = [b.add(p) for p in ps]
    for strategy in (Batch.PERSISTENT, 1, Batch.FLAT):
        b.configure(strategy, 4)
        for o in outs:
            o.fill_(float("nan"))
        b.forward(use_graph=True)
        torch.cuda.synchronize()
        for o, ref in zip(outs, refs):
            got = o.cpu().numpy().astype(np.float64)
            assert np.isfinite(got).all()
            assert np.max(np.abs(got - ref) / ref) <= RTOL, strategy


def test_more_items_than_one_launch_holds(cuda):
    """45 items: the single-launch strategies split them into launches of at
    most 40 (the parameter block's capacity)."""
    import torch
    ps = [_projector(cuda, "random", 100 + i, N=16, Z=4 + i % 5, V=1 + i % 3, W=8 + i % 4, H=6) for i in range(45)]
    plain = [p.forward().cpu().numpy() for p in ps]
    b = Batch()
    outs = [b.add(p) for p in ps]
    for strategy in (Batch.PERSISTENT, Batch.FLAT):
        b.configure(strategy, 2)
        for o in outs:
            o.fill_(float("nan"))
        b.forward(use_graph=True)
        torch.cuda.synchronize()
        for o, ref in zip(outs, plain):
            assert np.array_equal(o.cpu().numpy(), ref), strategy


def test_batched_equals_plain_launches(cuda):
    import torch
    ps = [_projector(cuda, "ellipsoid", 1, N=64, Z=20, V=5),
          _projector(cuda, "random", 2, N=48, Z=9, V=2, W=36, H=70),
          _projector(cuda, "water", 0, N=80, Z=33, V=7, W=52, H=44),
          _projector(cuda, "random", 3, N=32, Z=64, s=0.3, step=0.02, V=2, W=24, H=40, dpn=900.0)]
    plain = [p.forward().cpu().numpy() for p in ps]
    b = Batch()
    outs = [b.add(p) for p in ps]
    for strategy, cpb in ((0, 4), (1, 4), (2, 4), (0, 2), (1, 8), (2, 8), (2, 2)):
        b.configure(strategy, cpb)
        for use_graph in (False, True, True):
            for o in outs:
                o.fill_(float("nan"))
            b.forward(use_graph=use_graph)
            torch.cuda.synchronize()
            for o, ref in zip(outs, plain):
                assert np.array_equal(o.cpu().numpy(), ref), (strategy, cpb, use_graph)
    c = b.autotune()
    assert c % 100 in (2, 4, 8) and c // 100 in (0, 1, 2)
    b.forward(use_graph=True)
    torch.cuda.synchronize()
    for o, ref in zip(outs, plain):
        got = o.cpu().numpy()
        assert np.max(np.abs(got - ref) / ref) <= 1e-6


def test_projector_autotune_keeps_results(cuda):
    p = _projector(cuda, "ellipsoid", 4)
    ref = p.forward().cpu().numpy()
    c = p.autotune()
    assert c in (2, 4, 8)
    assert np.max(np.abs(p.forward().cpu().numpy() - ref) / ref) <= 1e-6


@pytest.mark.parametrize("strategy", [Batch.PERSISTENT, Batch.PER_ITEM, Batch.FLAT])
def test_items_of_every_kind(cuda, strategy):
    """Walked and by shared columns (H), uint16 and float volumes in turn, 46
    items (more than a launch holds of one kind); then with every volume's type
    the other way round, by the launches already prepared."""
    import torch
    ps, b = [], Batch()
    for i in range(46):
        g, tabs, vol, _ = proj_case("random", seed=200 + i, N=16 + i % 3, Z=4 + i % 5, V=1 + i % 2, W=8 + i % 4,
                                    H=96 if i % 23 == 1 else 6)
        mu, pdf = spectrum()
        p = Projector(g, *tabs)
        p.set_spectrum(mu, pdf, 1000.0)
        ps.append((p, vol))
    for turn in (0, 1):
        plain = []
        for i, (p, vol) in enumerate(ps):
            (p.load_volume if (i % 7 != 0) != bool(turn) else lambda v: p.load_volume_f32(v.astype(np.float32)))(vol)
            plain.append(p.forward().cpu().numpy())
        if turn == 0:
            outs = [b.add(p) for p, _ in ps]
            b.configure(strategy, 2)
        for use_graph in (True, False):
            for o in outs:
                o.fill_(float("nan"))
            b.forward(use_graph=use_graph)
            torch.cuda.synchronize()
            for o, ref in zip(outs, plain):
                assert np.array_equal(o.cpu().numpy(), ref), (turn, use_graph)


def test_more_tiles_than_a_grid_holds(cuda):
    """Two items of 1.09e9 one-row tiles: 2.2e9 blocks are more than one launch
    takes (2^31 - 1)."""
    import torch
    ps = []
    for i in range(2):
        g, tabs, vol, _ = proj_case("random", seed=i, N=8, Z=2, V=33000, W=33000, H=1,
                                    angles=np.arange(33000) * (360.0 / 33000))
        mu, pdf = spectrum()
        p = Projector(g, *tabs)
        p.set_spectrum(mu[:, 40:41], pdf[40:41], 1000.0)
        p.load_volume(vol)
        ps.append(p)
    b = Batch()
    outs = [b.add(p) for p in ps]
    b.configure(Batch.FLAT, 1)
    b.forward(use_graph=False)
    for p, o in zip(ps, outs):
        assert torch.equal(o, p.forward())


def test_tuned_choices_are_kept_apart_by_kernel(cuda, monkeypatch, tmp_path):
    """Projectors and batches of equal sizes, walked or by shared columns, of
    uint16 or float volumes: none takes a choice that was timed for another."""
    file = tmp_path / "tuned"
    monkeypatch.setenv("VCBCT_TUNE_CACHE", str(file))
    seen = 0
    for step in (0.2, 0.6):
        for f32 in (False, True):
            g, tabs, vol, _ = proj_case("random", seed=1, N=31, Z=7, V=3, W=21, H=45, step=step)
            mu, pdf = spectrum()
            p = Projector(g, *tabs)
            p.set_spectrum(mu, pdf, 1000.0)
            p.load_volume_f32(vol.astype(np.float32)) if f32 else p.load_volume(vol)
            b = Batch()
            b.add(p)
            for again in (0, 1):
                p.autotune()
                b.autotune()
                assert len(file.read_text().splitlines()) == seen + 2
            seen += 2
