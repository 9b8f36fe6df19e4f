"""The guiding network's tcgen05 inference kernel (tensor-memory
accumulators, shared-memory descriptors) against the warp-level mma.sync
kernel: the same BF16 products summed in FP32, so the outputs agree to FP32
summation-order differences (and the rare activation that then rounds to the
neighbouring BF16 value)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 128, 129, 5000, 100000])
def test_tcgen05_matches_mma_sync(native, ctx, n):
    rng = np.random.default_rng(n)
    tc = native.Guide(ctx, seed=4, center=(0.0, 0.0, 0.0), half_extent=10.0, infer_kernel=0)
    ms = native.Guide(ctx, seed=4, center=(0.0, 0.0, 0.0), half_extent=10.0, infer_kernel=1)
    p = tc.params()
    p[-48:] = rng.normal(0, 0.3, 48)   # nonzero output biases
    tc.set_params(p)
    ms.set_params(p)
    pos = torch.from_numpy(rng.uniform(-10, 10, (n, 3)).astype(np.float32)).cuda()
    d = rng.normal(size=(n, 3))
    nrm = torch.from_numpy((d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)).cuda()
    y_tc = torch.full((n, 40), float("nan"), dtype=torch.float32, device="cuda")
    y_ms = torch.full((n, 40), float("nan"), dtype=torch.float32, device="cuda")
    tc.infer(pos, nrm, n, y_tc)
    ms.infer(pos, nrm, n, y_ms)
    torch.cuda.synchronize()
    ctx.check()
    a, b = y_tc.cpu().numpy(), y_ms.cpu().numpy()
    assert np.all(np.isfinite(a))
    err = np.abs(a - b)
    scale = np.abs(b).max() + 1e-6
    assert np.median(err) <= 1e-6 * scale + 1e-7 and err.max() <= 2e-2 * scale, (np.median(err), err.max(), scale)


@pytest.mark.parametrize("n", [300, 50000])
def test_tcgen05_training_matches_mma_sync(native, ctx, n):
    """Gradients of the tcgen05 training kernel against the mma.sync one on the
    same batch (50,000 rows: more 128-row tiles than resident CTAs)."""
    rng = np.random.default_rng(n + 1)
    tc = native.Guide(ctx, seed=5, center=(0.0, 0.0, 0.0), half_extent=10.0, infer_kernel=0)
    ms = native.Guide(ctx, seed=5, center=(0.0, 0.0, 0.0), half_extent=10.0, infer_kernel=1)
    p = tc.params()
    p[-48:] = rng.normal(0, 0.3, 48)
    tc.set_params(p)
    ms.set_params(p)

    def unit(k):
        d = rng.normal(size=(k, 3))
        return torch.from_numpy((d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)).cuda()

    pos = torch.from_numpy(rng.uniform(-10, 10, (n, 3)).astype(np.float32)).cuda()
    nrm, sdir = unit(n), unit(n)
    w = torch.from_numpy(rng.lognormal(0.0, 1.0, n).astype(np.float32)).cuda()
    l_tc, g_tc = tc.gradients(pos, nrm, sdir, w, n)
    l_ms, g_ms = ms.gradients(pos, nrm, sdir, w, n)
    ctx.check()
    assert np.all(np.isfinite(g_tc))
    assert abs(l_tc - l_ms) <= 1e-4 * abs(l_ms)
    a, b = g_tc.astype(np.float64), g_ms.astype(np.float64)
    rel = np.linalg.norm(a - b) / np.linalg.norm(b)
    assert rel <= 1e-2, rel


def test_tcgen05_rows_do_not_depend_on_the_launch(native, ctx):
    """Row counts around the tiles (128 rows), the blocks (one per SM) and the
    groups of a block (six): every row has the bits it has in the largest
    launch, whichever tile, group and pass carries it, and no other row is
    written; the largest launch agrees with the mma.sync kernel."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    big = 2 * 6 * 128 * sms + 130
    rng = np.random.default_rng(11)
    tc = native.Guide(ctx, seed=6, half_extent=10.0, infer_kernel=0)
    ms = native.Guide(ctx, seed=6, half_extent=10.0, infer_kernel=1)
    pos = torch.from_numpy(rng.uniform(-11, 11, (big, 3)).astype(np.float32)).cuda()
    d = rng.normal(size=(big, 3))
    nrm = torch.from_numpy((d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)).cuda()

    def run(g, n):
        y = torch.full((big, 40), float("nan"), dtype=torch.float32, device="cuda")
        g.infer(pos, nrm, n, y)
        return y

    want = run(tc, big)
    assert bool(torch.isfinite(want).all())
    for n in (1, 127, 128, 129, 128 * sms, 128 * sms + 1, 6 * 128 * sms, 6 * 128 * sms + 1, big - 1):
        y = run(tc, n)
        assert torch.equal(y[:n], want[:n]), n
        assert bool(torch.isnan(y[n:]).all()), n
    ctx.check()
    err = (want - run(ms, big)).abs()
    scale = float(want.abs().max()) + 1e-6
    assert float(err.median()) <= 1e-6 * scale + 1e-7 and float(err.max()) <= 2e-2 * scale


@pytest.mark.parametrize("n", [1, 127, 129, 19456, 19457])
def test_tcgen05_training_at_tile_edges(native, ctx, n):
    """Row counts around one tile and around one tile per SM: the gradients
    agree with the mma.sync kernels (the bounds of the test above), and two runs
    have the same bits."""
    rng = np.random.default_rng(n + 7)
    tc = native.Guide(ctx, seed=8, half_extent=10.0, infer_kernel=0)
    ms = native.Guide(ctx, seed=8, half_extent=10.0, infer_kernel=1)
    p = tc.params()
    p[-48:] = rng.normal(0, 0.3, 48)
    tc.set_params(p)
    ms.set_params(p)

    def unit(k):
        d = rng.normal(size=(k, 3))
        return torch.from_numpy((d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)).cuda()

    pos = torch.from_numpy(rng.uniform(-10, 10, (n, 3)).astype(np.float32)).cuda()
    nrm, sdir = unit(n), unit(n)
    w = torch.from_numpy(rng.lognormal(0.0, 1.0, n).astype(np.float32)).cuda()
    l_tc, g_tc = tc.gradients(pos, nrm, sdir, w, n)
    l_2, g_2 = tc.gradients(pos, nrm, sdir, w, n)
    l_ms, g_ms = ms.gradients(pos, nrm, sdir, w, n)
    ctx.check()
    assert l_tc == l_2 and np.array_equal(g_tc, g_2)
    assert abs(l_tc - l_ms) <= 1e-4 * abs(l_ms)
    a, b = g_tc.astype(np.float64), g_ms.astype(np.float64)
    assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b)
    # the step uses the same sums: one Adam step from the same parameters agrees
    tc.train_step(pos, nrm, sdir, w, n)
    assert tc.last_loss() == l_tc


@pytest.mark.parametrize("n", [5, 300])
def test_rows_of_non_finite_directions_stay_finite(native, ctx, n):
    """The ReLU takes a NaN to 0, in both kernels: a row whose direction is not
    finite gives the outputs of a network whose hidden layers are 0 (here the
    output biases, as the hidden ones are 0), and leaves its neighbours alone."""
    rng = np.random.default_rng(n)
    pos = torch.from_numpy(rng.uniform(-10, 10, (n, 3)).astype(np.float32)).cuda()
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    bad = np.arange(0, n, 4)
    odd = d.copy()
    odd[bad, rng.integers(0, 3, len(bad))] = np.nan
    out = {}
    for kernel in (0, 1):
        g = native.Guide(ctx, seed=9, half_extent=10.0, infer_kernel=kernel)
        p = g.params()
        bias = rng.normal(0, 0.3, 48).astype(np.float32) if kernel == 0 else bias
        p[-48:] = bias
        g.set_params(p)
        for name, rows in (("good", d), ("odd", odd)):
            y = torch.full((n, 40), float("nan"), dtype=torch.float32, device="cuda")
            g.infer(pos, torch.from_numpy(rows).cuda(), n, y)
            out[kernel, name] = y.cpu().numpy()
    ctx.check()
    keep = np.setdiff1d(np.arange(n), bad)
    for kernel in (0, 1):
        assert np.array_equal(out[kernel, "odd"][bad], np.broadcast_to(bias[:40], (len(bad), 40)))
        assert np.array_equal(out[kernel, "odd"][keep], out[kernel, "good"][keep])


@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
def test_non_finite_rows_over_many_tiles(native, ctx, value):
    """Tiles that hold a row of a non-finite direction are carried through twice,
    in any group and pass of a block: both kernels give finite outputs for such
    rows and agree; every other row has the bits it has without them."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 6 * 128 * sms + 7 * 128 + 50
    rng = np.random.default_rng(12)
    pos = torch.from_numpy(rng.uniform(-10, 10, (n, 3)).astype(np.float32)).cuda()
    d = rng.normal(size=(n, 3))
    d = torch.from_numpy((d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)).cuda()
    bad = torch.from_numpy(np.unique(rng.integers(0, n, 200))).cuda()
    odd = d.clone()
    odd[bad, 1] = value
    out = []
    for kernel in (0, 1):
        g = native.Guide(ctx, seed=10, half_extent=10.0, infer_kernel=kernel)
        y, z = (torch.full((n, 40), float("nan"), dtype=torch.float32, device="cuda") for _ in range(2))
        g.infer(pos, d, n, y)
        g.infer(pos, odd, n, z)
        keep = torch.ones(n, dtype=torch.bool, device="cuda")
        keep[bad] = False
        assert bool(torch.isfinite(z).all()) and torch.equal(y[keep], z[keep])
        out.append(z[bad])
    ctx.check()
    scale = float(out[1].abs().max()) + 1e-6
    assert float((out[0] - out[1]).abs().max()) <= 2e-2 * scale
