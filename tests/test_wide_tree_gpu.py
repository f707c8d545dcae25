"""The 8-wide walk where it can go wrong: rays whose answer it cannot certify and
hands back to the reference's own walk (exact ties, far origins, zero and
subnormal direction components), and trees of unusual shape. Closest hits and
visibility are compared bit for bit with the oracle's restatement of the
reference's walk."""
import numpy as np
import pytest

import oracle
from lightmetrica_b200.scene import create_scene, soup_primitives
from lightmetrica_b200.workloads import FLT_MAX, random_rays, random_soup, rays_soa

pytestmark = pytest.mark.gpu


def _grid(n):
    """Axis-aligned quads in the plane z = 0: shared edges and vertices, flat boxes."""
    lin = np.linspace(-1, 1, n + 1).astype(np.float32)
    x, y = np.meshgrid(lin, lin, indexing="ij")
    pos = np.stack([x, y, np.zeros_like(x)], -1).reshape(-1, 3).astype(np.float32)
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    a = (i * (n + 1) + j).reshape(-1)
    faces = np.concatenate([np.stack([a, a + n + 1, a + n + 2], 1), np.stack([a, a + n + 2, a + 1], 1)])
    return pos, faces.astype(np.uint32)


def _scene(kind):
    if kind == "soup":
        return random_soup(3000, seed=3, sigma=0.08)
    if kind == "doubled":                            # every hit is a tie
        pos, faces = random_soup(1500, seed=4, sigma=0.1)
        return np.concatenate([pos, pos]), np.concatenate([faces, faces + np.uint32(pos.shape[0])])
    if kind == "coincident":                         # one leaf of many triangles: equal centroids
        pos, faces = random_soup(1, seed=5, sigma=0.5)
        return np.tile(pos, (300, 1)), np.arange(900, dtype=np.uint32).reshape(-1, 3)
    if kind == "grid":
        return _grid(24)
    if kind == "slivers":
        pos, faces = random_soup(2000, seed=6, sigma=0.05)
        p = pos.reshape(-1, 3, 3).copy()
        p[:, 2] = p[:, 0] + (p[:, 1] - p[:, 0]) * np.float32(0.5) + (p[:, 2] - p[:, 0]) * np.float32(1e-5)
        return p.reshape(-1, 3), faces
    if kind == "offset":
        pos, faces = random_soup(2000, seed=7, sigma=0.05)
        return pos + np.float32(300.0), faces
    if kind == "tiny_scale":
        pos, faces = random_soup(500, seed=8, sigma=0.1)
        return pos * np.float32(1e-22), faces
    return random_soup(int(kind), seed=9, sigma=0.4)  # a number: that many triangles


def _rays(pos, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = pos.min(0), pos.max(0)
    mid, half = (lo + hi) / 2, float(np.max(hi - lo)) / 2 + 1e-30
    rays = random_rays(n, seed=seed, extent=1.0)
    rays[:, 0:3] = mid + rays[:, 0:3] * np.float32(2 * half)
    k = np.arange(n)
    axis = k % 7 == 0                                # axis-aligned: two zero components
    d = np.zeros((int(axis.sum()), 3), np.float32)
    d[np.arange(d.shape[0]), rng.integers(0, 3, d.shape[0])] = rng.choice([-1.0, 1.0], d.shape[0])
    rays[axis, 3:6] = d
    onto = k % 7 == 1                                # through vertices of the scene
    t = pos[rng.integers(0, pos.shape[0], int(onto.sum()))]
    v = t - rays[onto, 0:3]
    rays[onto, 3:6] = v / np.linalg.norm(v.astype(np.float64), axis=1, keepdims=True)
    far = k % 7 == 2                                 # beyond the boxes' origin bound, aimed back
    o = mid + rng.normal(size=(int(far.sum()), 3)).astype(np.float32) * np.float32(200 * (half + float(np.abs(mid).max())))
    v = mid - o
    rays[far, 0:3] = o
    rays[far, 3:6] = v / np.linalg.norm(v.astype(np.float64), axis=1, keepdims=True)
    one_zero = k % 7 == 3
    rays[one_zero, 3 + seed % 3] = 0.0
    sub = k % 49 == 4                                # 1/d overflows
    rays[sub, 3] = 1e-41
    rays[:, 7] = np.where(k % 5 == 0, half * 1.5, FLT_MAX)
    rays[k % 11 == 0, 6] = half * 0.25
    return rays.astype(np.float32)


@pytest.mark.parametrize("n", [1, 33, 20011])
@pytest.mark.parametrize("kind", ["soup", "doubled", "coincident", "grid", "slivers", "offset", "tiny_scale", "1", "8", "9", "70"])
def test_hits_and_visibility_equal_the_reference_walk(cuda, kind, n):
    import torch
    pos, faces = _scene(kind)
    rays = _rays(pos, n, seed=21 + n % 3)
    s = create_scene("qbvh" if n == 33 else "bvh")
    s.load(soup_primitives(pos, faces))
    s.configure({})
    s.build()
    want = oracle.OracleScene(pos, faces, "bvh").intersect(rays)
    got = s.intersect_host(rays)
    np.testing.assert_array_equal(got["tri_id"], want["tri_id"])
    hit = want["tri_id"] >= 0
    for k in ("t", "u", "v"):
        np.testing.assert_array_equal(got[k][hit], want[k][hit])
    soa = {k: torch.from_numpy(v).to(cuda) for k, v in rays_soa(rays).items()}
    occ = torch.zeros(n, dtype=torch.uint8, device=cuda)
    stream = torch.cuda.current_stream().cuda_stream
    s.occluded_device({k: v.data_ptr() for k, v in soa.items()}, occ.data_ptr(), n, stream)
    s.status(stream)
    np.testing.assert_array_equal(occ.cpu().numpy().astype(bool), hit)
    s.close()


def _equal_to_the_reference_walk(cuda, pos, faces, rays, impl="bvh"):
    import torch
    n = rays.shape[0]
    s = create_scene(impl)
    s.load(soup_primitives(pos, faces))
    s.configure({})
    s.build()
    want = oracle.OracleScene(pos, faces, "bvh").intersect(rays)
    got = s.intersect_host(rays)
    np.testing.assert_array_equal(got["tri_id"], want["tri_id"])
    hit = want["tri_id"] >= 0
    for k in ("t", "u", "v"):
        np.testing.assert_array_equal(got[k][hit], want[k][hit])
    soa = {k: torch.from_numpy(v).to(cuda) for k, v in rays_soa(rays).items()}
    occ = torch.zeros(n, dtype=torch.uint8, device=cuda)
    stream = torch.cuda.current_stream().cuda_stream
    s.occluded_device({k: v.data_ptr() for k, v in soa.items()}, occ.data_ptr(), n, stream)
    s.status(stream)
    np.testing.assert_array_equal(occ.cpu().numpy().astype(bool), hit)
    s.close()
    return hit


@pytest.mark.parametrize("zeros", [1, 2])
@pytest.mark.parametrize("kind", ["soup", "grid", "offset", "9"])
def test_negated_zero_directions_hit_as_the_reference(cuda, kind, zeros):
    """Direction components of either zero, alone and in pairs, from inside the boxes and from outside."""
    pos, faces = _scene(kind)
    n = 4001
    rng = np.random.default_rng(31)
    rays = _rays(pos, n, seed=30)
    k = np.arange(n)
    first = k % 3
    d = rng.normal(size=(n, 3)).astype(np.float32)
    for z in range(zeros):
        d[k, (first + z) % 3] = np.copysign(np.float32(0), rng.choice([-1.0, 1.0], n).astype(np.float32))
    rays[:, 3:6] = d / np.linalg.norm(d.astype(np.float64), axis=1, keepdims=True).astype(np.float32)
    centre = pos.reshape(-1, 3)[faces].mean(1)[rng.integers(0, faces.shape[0], n)]
    aim = k % 2 == 0                                 # towards a triangle from beside it: many hits
    rays[aim, 0:3] = (centre - rays[:, 3:6] * rng.uniform(0.01, 0.5, (n, 1)).astype(np.float32))[aim]
    zero = rays[:, 3:6] == 0
    assert (np.signbit(rays[:, 3:6]) & zero).any() and (~np.signbit(rays[:, 3:6]) & zero).any()
    hit = _equal_to_the_reference_walk(cuda, pos, faces, rays, "qbvh" if zeros == 2 else "bvh")
    assert hit[np.signbit(rays[:, 3]) & zero[:, 0]].any()


def test_a_negated_axis_hits(cuda):
    pos = np.array([[-1, -1, -1], [1, -1, -1], [0, 1, -1]], np.float32)
    rays = np.array([[0.01, 0.02, 0, -0.0, 0, -1, 0, FLT_MAX], [0.01, 0.02, 0, -0.0, -0.0, -1, 0, FLT_MAX],
                     [0.01, 0.02, -2, -0.0, -0.0, 1, 0, FLT_MAX]], np.float32)
    assert _equal_to_the_reference_walk(cuda, pos, np.array([[0, 1, 2]], np.uint32), rays).all()


@pytest.mark.parametrize("scale", [1e-6, 1e-10, 1e-13, 1e-15, 1e-18, 1e-20, 1e-25, 1e-37, 1e9, 1e15, 1e25, 1e37])
@pytest.mark.parametrize("kind", ["soup", "grid"])
def test_directions_of_any_length_hit_as_the_reference(cuda, kind, scale):
    """Unnormalised directions, with no, one and two zero components or ones far below the others; ray intervals that do
    and do not begin or end on the way."""
    pos, faces = _scene(kind)
    n = 3001
    rng = np.random.default_rng(41)
    rays = _rays(pos, n, seed=40)
    k = np.arange(n)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d[k % 5 == 1, 0] = 0.0
    d[k % 5 == 2, 1:] = 0.0
    d[k % 5 == 3, 2] *= np.float32(1e-9)
    d[k % 5 == 4, 0] *= np.float32(1e-20)
    d /= np.linalg.norm(d.astype(np.float64), axis=1, keepdims=True).astype(np.float32)
    centre = pos[faces].mean(1)[rng.integers(0, faces.shape[0], n)]
    aim = k % 2 == 0                                 # grazing the far side of the boxes, too: offsets of 1 down to 1e-5
    away = (10.0 ** rng.uniform(-5, 0, (n, 1))).astype(np.float32)
    rays[aim, 0:3] = (centre - d * away)[aim]
    with np.errstate(under="ignore", over="ignore"):
        rays[:, 3:6] = d * np.float32(scale)
        rays[:, 6] = np.where(k % 3 == 0, np.float32(0.3 / scale if scale > 1e-38 else 0), 0)
        rays[:, 7] = np.where(k % 4 == 0, np.minimum(2.0 / scale, FLT_MAX), FLT_MAX).astype(np.float32)
    hit = _equal_to_the_reference_walk(cuda, pos, faces, rays)
    assert hit.any() or scale < 1e-30


def test_very_short_axis_directions_hit(cuda):
    """The exit of a zero axis against an entry 1e15 and more away (in units of the direction's length)."""
    pos = np.array([[-1, -1, -100], [1, -1, -100], [0, 1, -100]], np.float32)
    rays = np.array([[0.49, -0.99, 0, 0, 0, -s, 0, FLT_MAX] for s in (1e-12, 1e-15, 1e-18, 1e-20, 1e-30)], np.float32)
    assert _equal_to_the_reference_walk(cuda, pos, np.array([[0, 1, 2]], np.uint32), rays).all()
