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


def test_grazing_rays_in_a_large_launch(native, ctx, oracle):
    """Rays through vertices and edges, in a launch above the team limit: the
    persistent closest-hit and any-hit kernels, both triangle tests."""
    from test_trace_gpu import grazing_rays
    half = scenes.density_half(6000)
    soup, _, _ = scenes.incoherent_soup(6000, seed=41, half=half)
    rays = grazing_rays(soup, _team_limit() + 1, seed=42)
    scene = native.Scene(ctx, soup)
    dev = torch.from_numpy(rays).cuda()
    for mode in (0, 1):
        hits = torch.empty((len(rays), 2), dtype=torch.int32, device="cuda")
        occ = torch.empty(len(rays), dtype=torch.uint8, device="cuda")
        scene.trace_closest(dev, len(rays), hits, mode)
        scene.trace_any(dev, len(rays), occ, mode)
        h = hits.cpu().numpy()
        tb, pb = oracle.trace_brute(soup, rays, tri_mode=mode)
        assert (pb >= 0).mean() > 0.5
        assert np.array_equal(h[:, 0], tb.view(np.int32)) and np.array_equal(h[:, 1], pb)
        assert np.array_equal(occ.cpu().numpy().astype(bool), pb >= 0)
    ctx.check()


def test_stack_cap_reports_overflow_in_large_launches(native):
    """The overflow exits of the persistent kernels (the small launches take the
    team kernels): closest hit, any hit and the renderer's per-bounce traversal
    report it, and are exact again with the full stack."""
    lib = native.load()
    c = native.Context(0)
    half = scenes.density_half(65536)
    soup, _, _ = scenes.incoherent_soup(65536, seed=5, half=half)
    n = _team_limit() + 1
    dev = torch.from_numpy(scenes.incoherent_rays(n, seed=6, half=half)).cuda()
    scene = native.Scene(c, soup)
    rscene = native.Scene.from_spec(c, scenes.many_light(6 * 1280, 40, seed=3, half=6.0))
    w, h = 512, -(-1024 * torch.cuda.get_device_properties(0).multi_processor_count // 512) + 1
    cam = scenes.outside_camera(w, h, distance=20.0, half=6.0)

    def closest():
        out = torch.zeros((n, 2), dtype=torch.int32, device="cuda")
        scene.trace_closest(dev, n, out)
        return out

    def occluded():
        out = torch.zeros(n, dtype=torch.uint8, device="cuda")
        scene.trace_any(dev, n, out)
        return out

    def image():
        acc = torch.zeros((w * h, 4), dtype=torch.float32, device="cuda")
        rscene.render(cam, acc, spp=1, max_depth=6)
        return acc.view(torch.int32)

    want = [f() for f in (closest, occluded, image)]
    c.check()
    for f in (closest, occluded, image):
        native.check(lib.dr_debug_stack_limit(c.handle, 1))
        f()
        torch.cuda.synchronize()
        assert lib.dr_context_check(c.handle) == 6  # DR_ERR_STACK_OVERFLOW
        native.check(lib.dr_debug_stack_limit(c.handle, 0))
    assert all(torch.equal(f(), w0) for f, w0 in zip((closest, occluded, image), want))
    c.check()


@pytest.mark.parametrize("streams,chunk,stack", [(1, 64, 4), (2, 128, 16), (3, 0, 4), (1, 0, 16), (2, 96, 8)])
def test_large_batch_waves_of_several_scenes(native, ctx, streams, chunk, stack):
    """Waves above the whole-path limit that mix the images of three scenes, with
    every shared-stack depth and fetch size of the per-bounce traversal: each
    image equals the one rendered alone."""
    specs = [scenes.box_room(2), scenes.many_light(6 * 1280, 40, seed=3, half=6.0), scenes.box_room(1)]
    scs = [native.Scene.from_spec(ctx, s) for s in specs]
    jobs, outs, alone = [], [], []
    for k, (si, w, h, spp, depth) in enumerate([(0, 300, 200, 3, 6), (1, 257, 190, 2, 9), (2, 320, 240, 2, 4), (1, 129, 65, 5, 12)]):
        cam = scenes.outside_camera(w, h, distance=20.0, half=6.0) if si == 1 else scenes.camera(w, h)
        acc, ref = (torch.zeros((w * h, 4), dtype=torch.float32, device="cuda") for _ in range(2))
        casts, rcasts = (torch.zeros(w * h, dtype=torch.int32, device="cuda") for _ in range(2))
        jobs.append(native.make_job(scs[si], cam, acc, casts, spp=spp, max_depth=depth, seed=k))
        scs[si].render(cam, ref, rcasts, spp=spp, max_depth=depth, seed=k)
        outs.append((acc, casts))
        alone.append((ref, rcasts))
    native.render_batch(ctx, jobs, wave_paths=200000, streams=streams, chunk=chunk, stack=stack)
    torch.cuda.synchronize()
    ctx.check()
    for (a, c), (ra, rc) in zip(outs, alone):
        assert torch.equal(a.view(torch.int32), ra.view(torch.int32)) and torch.equal(c, rc)
