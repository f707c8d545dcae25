"""The differentiable passes as waves against the one-thread passes: a budget
large enough for waves equals the weighted sum of its parts, each small enough
for one thread per sample (same samples, same random numbers; the sums are
accumulated in another order)."""
import ctypes

import numpy as np
import pytest

from lightmetrica_b200 import create_renderer, create_scene, native as N, scenes
from lightmetrica_b200.diff import light_emission, triangle_albedo

pytestmark = pytest.mark.gpu

SIDE = 160              # an image whose larger budgets run as waves:
WAVE_MIN = 1 << 20      # from this many samples on (pt: twice as many)
PART = 1 << 17


def _closed_box():
    """Mirrors and diffuse faces all around: no path leaves."""
    prims = scenes.cornell_box(SIDE, SIDE, variant="mixed")
    prims.environment_light = None
    prims.add(scenes.Primitive(mesh=scenes._mesh([scenes._quad((0, 0, 1.0), (1, 0, 1.0), (1, 1, 1.0), (0, 1, 1.0), (0, 0, -1))]),
                               bsdf=scenes.PerfectMirrorBSDF((0.9, 0.9, 0.9))))
    prims.camera.eye = (0.5, 0.5, 0.9)
    # Small triangles: of the 2^20 x 45 vertices each then gets about 10^4 gradient terms. (With 10^6 on each of 50, a
    # single-precision sum in progress loses the terms below its half ulp, a share of 10^6 x 6e-8 of them.)
    for p in prims.primitives:
        p.mesh = scenes.subdivide(p.mesh, 3)
    return prims


def _pass(scene, params, diff, torch, albedo, emission, dL, backward):
    st = N.RenderStats()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if not backward:
        img = torch.zeros(dL.numel(), device="cuda")
        N.check(N.lib().lmgpu_adjoint_forward(scene.handle, ctypes.byref(params), ctypes.byref(diff), img.data_ptr(), stream,
                                              ctypes.byref(st)))
        scene.status(stream.value)
        return (img.double().cpu().numpy(),)
    da, de = torch.zeros_like(albedo), torch.zeros_like(emission)
    N.check(N.lib().lmgpu_adjoint_backward(scene.handle, ctypes.byref(params), ctypes.byref(diff), dL.data_ptr(), da.data_ptr(),
                                           de.data_ptr(), stream, ctypes.byref(st)))
    scene.status(stream.value)
    return da.double().cpu().numpy(), de.double().cpu().numpy()


@pytest.mark.parametrize("technique,box,max_pv,rr,n", [
    ("pt.mis", "mixed", 9, 3, WAVE_MIN), ("pt.direct", "classic", 2, 1, WAVE_MIN + 1), ("pt", "mixed", 9, -1, 2 * WAVE_MIN + 77),
    ("pt.mis", "closed", 45, -1, WAVE_MIN),          # beyond the vertices a wave records: tails
    ("pt", "closed", -1, 8, 2 * WAVE_MIN),           # unbounded depth: tails
    ("pt.direct", "closed", 33, -1, WAVE_MIN + 5)])  # exactly the recorded vertices
def test_waves_equal_the_sum_of_one_thread_passes(cuda, technique, box, max_pv, rr, n):
    import torch
    prims = _closed_box() if box == "closed" else scenes.cornell_box(SIDE, SIDE, variant=box)
    scene = create_scene("bvh")
    scene.load(prims)
    scene.configure({})
    scene.build()
    r = create_renderer(technique)
    r.configure({"rr_depth": rr, "max_path_vertices": max_pv, "sampler": {"rng_seed": 5}})
    albedo = torch.from_numpy(triangle_albedo(prims) * np.float32(0.9)).cuda()
    emission = torch.from_numpy(light_emission(prims)).cuda()
    dL = 1.0 + 0.5 * torch.rand((SIDE, SIDE, 3), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    diff = N.DiffParams(albedo.data_ptr(), emission.data_ptr())
    for backward in (False, True):
        whole = _pass(scene, r.params(n), diff, torch, albedo, emission, dL, backward)
        parts = [np.zeros_like(x) for x in whole]
        for off in range(0, n, PART):
            m = min(PART, n - off)
            for acc, x in zip(parts, _pass(scene, r.params(m, sample_offset=off), diff, torch, albedo, emission, dL, backward)):
                acc += x * (m / n)                   # a pass scales by W*H / its own samples
        for got, want in zip(whole, parts):
            # Single-precision sums of up to n terms in two orders: rounding of sqrt(n) ulps of the largest partial sums.
            assert np.linalg.norm(got - want) <= 4 * np.sqrt(n) * 6e-8 * np.linalg.norm(want) + 1e-12
            assert np.linalg.norm(want) > 0 or max_pv == 2   # (one bounce: light seen directly, no albedo on any prefix)
    scene.close()


@pytest.mark.parametrize("technique,max_pv,n,levels", [("pt.mis", 9, 160 * 160 * 41, 5), ("pt", 4, 1 << 21, 2), ("pt.direct", 6, 777, 2)])
def test_a_captured_pass_equals_the_direct_one(cuda, technique, max_pv, n, levels):
    """Under capture every budget runs one thread per sample, over the binary render tree."""
    import torch
    prims = scenes.cornell_refined(levels, 160, 160)
    scene = create_scene("bvh")
    scene.load(prims)
    scene.configure({})
    scene.build()
    r = create_renderer(technique)
    r.configure({"rr_depth": 3, "max_path_vertices": max_pv, "sampler": {"rng_seed": 6}})
    albedo = torch.from_numpy(triangle_albedo(prims) * np.float32(0.8)).cuda()
    emission = torch.from_numpy(light_emission(prims)).cuda()
    dL = 1.0 + 0.5 * torch.rand((160, 160, 3), generator=torch.Generator(device="cuda").manual_seed(2), device="cuda")
    diff, params = N.DiffParams(albedo.data_ptr(), emission.data_ptr()), r.params(n)
    direct = _pass(scene, params, diff, torch, albedo, emission, dL, False) + \
        _pass(scene, params, diff, torch, albedo, emission, dL, True)
    img, da, de = torch.zeros(dL.numel(), device="cuda"), torch.zeros_like(albedo), torch.zeros_like(emission)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        N.check(N.lib().lmgpu_adjoint_forward(scene.handle, ctypes.byref(params), ctypes.byref(diff), img.data_ptr(), s, None))
        N.check(N.lib().lmgpu_adjoint_backward(scene.handle, ctypes.byref(params), ctypes.byref(diff), dL.data_ptr(), da.data_ptr(),
                                               de.data_ptr(), s, None))
    graph.replay()
    torch.cuda.synchronize()
    scene.status(torch.cuda.current_stream().cuda_stream)
    for got, want in zip((img, da, de), direct):
        got = got.double().cpu().numpy()
        # Sums of single-precision terms in two orders: n of them on a few hundred triangles, about 2^8 on each of 36,864.
        # (Both walks answer rays within rounding of a shared edge alike: by the wide walk's own order, 1.4e-4 apart.)
        assert np.linalg.norm(got - want) <= (4 * np.sqrt(n if levels == 2 else 256) * 6e-8 + 2e-5) * np.linalg.norm(want)
        assert np.linalg.norm(want) > 0
    del graph
    scene.close()


def _idle(torch):
    """Gives back what this library and torch keep idle; the device's free bytes."""
    torch.cuda.synchronize()
    N.check(N.lib().lmgpu_render_release())
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_the_waves_workspace_is_bounded_and_gives_way(cuda):
    """What idle passes keep stays below 4 GiB; on a nearly full device a pass runs without it, and a render gets it."""
    import torch
    prims = scenes.cornell_refined(2, SIDE, SIDE)
    scene = create_scene("bvh")
    scene.load(prims)
    scene.configure({})
    scene.build()
    albedo, emission = torch.from_numpy(triangle_albedo(prims)).cuda(), torch.from_numpy(light_emission(prims)).cuda()
    dL = torch.ones((SIDE, SIDE, 3), device="cuda")
    diff = N.DiffParams(albedo.data_ptr(), emission.data_ptr())
    r = create_renderer("pt.mis")

    def gradients(n, max_pv):
        r.configure({"rr_depth": 3, "max_path_vertices": max_pv, "sampler": {"rng_seed": 7}})
        return _pass(scene, r.params(n), diff, torch, albedo, emission, dL, True)

    def render(n):
        r.configure({"rr_depth": 3, "max_path_vertices": 9, "sampler": {"rng_seed": 7}})
        film, st = torch.zeros(SIDE * SIDE * 3, device="cuda"), N.RenderStats()
        rc = N.lib().lmgpu_render_device(scene.handle, ctypes.byref(r.params(n, wave_paths=n)), ctypes.c_void_p(film.data_ptr()),
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.byref(st))
        torch.cuda.synchronize()
        return rc

    gradients(1 << 18, 9)                            # (kernels loaded, their local memory reserved)
    render(1 << 18)
    free = _idle(torch)
    gradients(1 << 23, 33)                           # 732 bytes a path
    torch.cuda.synchronize()
    kept = free - torch.cuda.mem_get_info()[0]
    assert (1 << 30) < kept <= (1 << 32) + (1 << 28)

    n = 1 << 21                                      # waves of 2^20 paths would take 365 MB
    want = gradients(n, 9)
    free = _idle(torch)
    room = 300 << 20
    full = torch.empty(free - room, dtype=torch.uint8, device="cuda")
    got = gradients(n, 9)
    for a, b in zip(got, want):                      # (bounds as in the captured passes above)
        assert np.linalg.norm(a - b) <= (4 * np.sqrt(n) * 6e-8 + 1e-4) * np.linalg.norm(b)
    del full
    _idle(torch)

    gradients(n, 9)                                  # its workspace (730 MB) is idle now
    torch.cuda.empty_cache()
    full = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
    assert render(n) == N.OK                         # 453 MB
    del full
    _idle(torch)
    scene.close()
