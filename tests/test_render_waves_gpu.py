"""The waves of the renderers where they can go wrong: the order in which paths take
samples (ragged films, parts of a sample plane), bounces traced together with the
shadow rays before them (deep and many waves), few rays spread over the GPU, and
ties between coincident triangles."""
import ctypes

import numpy as np
import pytest

from lightmetrica_b200 import create_renderer, create_scene, native as N, scenes
from lightmetrica_b200.batch import SceneBatch
from lightmetrica_b200.scene import soup_primitives
from lightmetrica_b200.workloads import random_rays, random_soup, rays_soa

pytestmark = pytest.mark.gpu


def _built(prims):
    s = create_scene("bvh")
    s.load(prims)
    s.configure({})
    s.build()
    return s


def _render(scene, renderer, n, torch, offset=0, wave_paths=0, fp64=True):
    cam = scene.main_camera()
    film = torch.zeros(cam.film.width * cam.film.height * 3, dtype=torch.float64 if fp64 else torch.float32, device="cuda")
    p = renderer.params(n, sample_offset=offset, film_fp64=fp64, wave_paths=wave_paths)
    st = N.RenderStats()
    N.check(N.lib().lmgpu_render_device(scene.handle, ctypes.byref(p), ctypes.c_void_p(film.data_ptr()),
                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.byref(st)))
    return film.cpu().numpy(), st


def _renderer(tech, max_pv, rr, sampling="stratified"):
    r = create_renderer(tech)
    r.configure({"rr_depth": rr, "max_path_vertices": max_pv, "sampler": {"rng_seed": 3, "sampling": sampling}})
    return r


# A path's radiance is the same in every order; a double film sums it with relative errors of 2^-53 an addition.
SUMS = dict(rtol=1e-11, atol=1e-13)


@pytest.mark.parametrize("w,h,n,split", [(1, 1, 5, 2), (3, 2, 6, 1), (7, 5, 100, 33), (8, 4, 64, 32), (9, 7, 63 * 3 + 11, 70),
                                         (33, 13, 429 * 8, 429 * 3), (64, 36, 2304 * 33, 2304 * 32 + 1)])
@pytest.mark.parametrize("tech", ["pt", "pt.mis"])
def test_any_split_renders_the_same_samples(cuda, tech, w, h, n, split):
    import torch
    s = _built(scenes.cornell_box(w, h, variant="mixed"))
    r = _renderer(tech, 6, 3)
    whole, _ = _render(s, r, n, torch)
    parts = _render(s, r, split, torch)[0] + _render(s, r, n - split, torch, offset=split)[0]
    assert whole.any()
    np.testing.assert_allclose(whole, parts, **SUMS)
    single, _ = _render(s, r, n, torch, fp64=False)
    np.testing.assert_allclose(single, whole, rtol=n * 6e-8, atol=1e-6)   # n additions of 2^-24 relative error each
    s.close()


@pytest.mark.parametrize("tech,max_pv,rr,sampling", [("pt.mis", -1, 1, "stratified"), ("pt.direct", 14, 30, "uniform"),
                                                     ("pt", -1, 4, "uniform"), ("pt.mis", 2, 1, "stratified"),
                                                     ("pt.mis", 1, 1, "stratified"), ("pt.direct", 10, 5, "stratified")])
def test_waves_of_any_size_and_the_batch_count_and_render_alike(cuda, tech, max_pv, rr, sampling):
    import torch
    s = _built(scenes.cornell_box(31, 17, variant="mixed"))
    r = _renderer(tech, max_pv, rr, sampling)
    n = 31 * 17 * 9 + 4
    film, st = _render(s, r, n, torch)
    for wave in (n, 1000, 257):
        other, so = _render(s, r, n, torch, wave_paths=wave)
        np.testing.assert_allclose(other, film, **SUMS)
        assert (so.rays_traced, so.shadow_rays, so.paths, so.max_bounces_run) == \
               (st.rays_traced, st.shadow_rays, st.paths, st.max_bounces_run)
        assert so.waves == -(-n // wave)
    if max_pv == 1:
        assert st.rays_traced == 0 and not film.any()
        return
    b = SceneBatch([s])
    for mode in ("waves", "overlap", "stream"):
        b.configure(mode=mode, wave_paths=1024)
        out = b.render([r], [n])[0].reshape(-1)
        np.testing.assert_allclose(out, film * (31 * 17 / n), rtol=n * 6e-8, atol=1e-6)
        assert b.last_stats["rays_traced"] == st.rays_traced and b.last_stats["shadow_rays"] == st.shadow_rays
    b.close()
    s.close()


@pytest.mark.parametrize("n", [1, 2, 31, 127, 593, 4735, 4737, 9473, 151552, 151553])
def test_few_rays_answer_as_among_many(cuda, n):
    """Around one ray and 32 rays for each of 148 x 8 x 4 resident warps."""
    import torch
    pos, faces = random_soup(5003, seed=11, sigma=0.1)
    s = _built(soup_primitives(pos, faces))
    soa = {k: torch.from_numpy(v).to(cuda) for k, v in rays_soa(random_rays(400009, seed=12)).items()}
    stream = torch.cuda.current_stream().cuda_stream

    def ask(m):
        out = {"tri_id": torch.zeros(m, dtype=torch.int32, device=cuda), **{k: torch.zeros(m, device=cuda) for k in "tuv"}}
        occ = torch.zeros(m, dtype=torch.uint8, device=cuda)
        rays = {k: v.data_ptr() for k, v in soa.items()}
        s.intersect_device(rays, {k: v.data_ptr() for k, v in out.items()}, m, stream)
        s.occluded_device(rays, occ.data_ptr(), m, stream)
        s.status(stream)
        return [out[k] for k in ("tri_id", "t", "u", "v")] + [occ]
    for few, many in zip(ask(n), ask(400009)):
        assert torch.equal(few, many[:n])
    s.close()


def _layered_grids(width, height):
    """Four emitting grids some units of rounding apart, far from the origin: a leaf box may be entered after its own
    triangle's t, and before or after the t of a triangle of another layer."""
    prims = scenes.Primitives()
    at, ulp = np.float32(300.0), np.float32(2.0 ** -15)
    for layer, (n, radiance) in enumerate([(20, 1.0), (24, 2.0), (31, 4.0), (37, 8.0)]):
        lin = np.linspace(-1, 1, n + 1).astype(np.float32)
        x, y = np.meshgrid(lin, lin, indexing="ij")
        pos = np.stack([x, y, np.zeros_like(x)], -1).reshape(-1, 3).astype(np.float32) + at
        pos[:, 2] += np.float32(layer) * ulp
        i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
        a = (i * (n + 1) + j).reshape(-1)
        faces = np.concatenate([np.stack([a, a + n + 1, a + n + 2], 1), np.stack([a, a + n + 2, a + 1], 1)]).astype(np.uint32)
        normals = np.tile(np.array([0, 0, 1], np.float32), (pos.shape[0], 1))
        prims.add(scenes.Primitive(mesh=scenes.TriangleMesh(pos, faces, normals), bsdf=scenes.DiffuseBSDF((0, 0, 0)),
                                   light=scenes.AreaLight((radiance,) * 3)))
    film = scenes.HDRBitmapFilm(width, height)
    prims.camera = scenes.PerspectiveCamera(film=film, eye=(340.3, 280.8, 1100.0), center=(300, 300, 300), up=(0, 1, 0), fovy=0.14)
    return prims


def test_a_rays_hit_does_not_depend_on_the_rays_beside_it(cuda):
    """Waves of one size against another: other rays share a ray's warp, so its triangles are tested in another order.
    Radiances are powers of two, whose sums are exact."""
    import torch
    s = _built(_layered_grids(96, 64))
    r = _renderer("pt", 2, -1)
    n = 96 * 64 * 8
    film, _ = _render(s, r, n, torch)
    assert len(np.unique(film)) > 4
    for wave in (61, 997, 4736, 20000):
        np.testing.assert_array_equal(_render(s, r, n, torch, wave_paths=wave)[0], film)
    s.close()
