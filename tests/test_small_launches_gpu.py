"""Launches with few rays or paths: teams of lanes per ray (public traversal)
and whole paths per kernel (renderer), at the sizes where the kernels change.
Every result is bit for bit that of the large launches and of the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from devilray_gb300 import scenes

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _team_limit():
    return 432 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("tris", [7, 20000])
def test_few_rays_equal_many(native, ctx, oracle, mode, tris):
    half = scenes.density_half(tris)
    soup, _, _ = scenes.incoherent_soup(tris, seed=3, half=half)
    scene = native.Scene(ctx, soup)
    limit = _team_limit()
    rays = scenes.incoherent_rays(limit + 4096, seed=4, half=half)
    rays[1::5, 3] = np.random.default_rng(5).uniform(0, half, len(rays[1::5])).astype(np.float32)  # segments
    rays[7::97, 4:7] = 0.0      # no direction: a miss
    rays[11::97, 5] = np.inf    # not finite: a miss
    dev = torch.from_numpy(rays).cuda()

    def closest(n):
        out = torch.full((n, 2), -7, dtype=torch.int32, device="cuda")
        scene.trace_closest(dev, n, out, mode)
        return out

    def occluded(n):
        out = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
        scene.trace_any(dev, n, out, mode)
        return out

    hits, occ = closest(len(rays)), occluded(len(rays))
    assert int((hits[:, 1] >= 0).sum()) > 0 and 0 < int(occ.sum()) < len(rays)
    for n in (1, 2, 31, 33, 1021, 4864, 4865, 19456, 19457, 40000, limit, limit + 1):
        assert torch.equal(closest(n), hits[:n]) and torch.equal(occluded(n), occ[:n]), n
    ctx.check()
    if mode == 0:
        n = 3000
        t, prim = oracle.BBH(soup).trace_canonical(rays[:n], slack=scene.info().slack)
        h = hits[:n].cpu().numpy()
        ok = np.isfinite(rays[:n, 4:7]).all(1) & (rays[:n, 4:7] != 0).any(1)
        assert np.array_equal(h[ok, 0], t.view(np.int32)[ok]) and np.array_equal(h[ok, 1], prim[ok])
        assert (h[~ok, 1] == -1).all()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("kind,w,h,depth", [("box", 405, 384, 10), ("lights", 405, 384, 16), ("lights", 97, 61, 5),
                                            ("box", 33, 1, 1)])
def test_whole_paths_equal_waves(native, ctx, oracle, mode, kind, w, h, depth):
    """One sample per wave (a wave of up to 1,024 paths per SM runs whole paths
    in one kernel; 405 x 384 is the last such size on 152 SMs) against all
    samples in one wave (per-bounce kernels, then the tail), and against a
    third split whose waves cross the limit; both against the oracle."""
    if kind == "box":
        spec, cam = scenes.box_room(2), scenes.camera(w, h)
    else:
        spec = scenes.many_light(20000, 1000, seed=5, half=scenes.density_half(20000))
        half = scenes.density_half(20000)
        cam = scenes.outside_camera(w, h, distance=2.0 * half, half=half)
    scene = native.Scene.from_spec(ctx, spec)
    n, spp = w * h, 5
    images = []
    for wave_paths in (n, 2 * n, spp * n):
        acc = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
        casts = torch.zeros(n, dtype=torch.int32, device="cuda")
        scene.render(cam, acc, casts, spp=spp, max_depth=depth, seed=2, wave_paths=wave_paths, tri_mode=mode)
        stats = scene.render_stats()
        assert stats.path_rays == int(casts.sum())
        images.append((acc, casts, stats.shadow_rays))
    ctx.check()
    for acc, casts, shadows in images[1:]:
        assert torch.equal(acc.view(torch.int32), images[0][0].view(torch.int32)) and torch.equal(casts, images[0][1])
        assert shadows == images[0][2]
    if mode == 0:
        pix = np.unique(np.linspace(0, n - 1, 400).astype(np.int64))
        oacc, ocasts, _ = oracle.RenderScene(spec).render(cam, spp, max_depth=depth, seed=2, pixels=pix)
        acc = images[0][0].cpu().numpy()
        assert np.array_equal(acc[pix].view(np.uint32), oacc[pix].view(np.uint32))
        assert np.array_equal(images[0][1].cpu().numpy()[pix], ocasts[pix].astype(np.int64))


@pytest.mark.parametrize("streams", [1, 2])
def test_captured_waves_equal_a_plain_render(native, ctx, streams):
    """Waves above the whole-path limit as one captured schedule: with one
    stream their kernels are launched before their predecessors end, with more
    they are not. Two replays against one plain render of twice the samples."""
    scene = native.Scene.from_spec(ctx, scenes.box_room(2))
    cam, depth, n = scenes.camera(405, 384), 7, 405 * 384
    images = []
    for replays in (2, 0):
        acc = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
        casts = torch.zeros(n, dtype=torch.int32, device="cuda")
        if replays:
            job = native.make_job(scene, cam, acc, casts, spp=4, max_depth=depth, seed=6)
            batch = native.Batch(ctx, [job], wave_paths=2 * n, streams=streams, use_graph=True)
            for _ in range(replays):
                batch.render()
            torch.cuda.synchronize()
            assert batch.info().num_waves == 2
            batch.close()
        else:
            scene.render(cam, acc, casts, spp=8, max_depth=depth, seed=6)
            torch.cuda.synchronize()
        images.append((acc, casts))
    assert torch.equal(images[0][0].view(torch.int32), images[1][0].view(torch.int32))
    assert torch.equal(images[0][1], images[1][1])
