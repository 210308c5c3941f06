"""Ray queries against brute force at the sizes where the hierarchy's build and
the traversal change form: one triangle (the root is a leaf), a few, the
build's cluster size (16) and its double, one more or less than a warp; meshes
in one plane, of equal triangles, with degenerate ones. The watertight test is
individually rounded and ties go to the smaller triangle, so the results are
those of the oracle bit for bit."""
import numpy as np
import pytest
import torch

from oracle import tr_oracle as O
from tensorray_b200 import api, scenes

pytestmark = pytest.mark.gpu


def _scene(P, F):
    spec = scenes.SceneSpec()
    spec.bsdfs = [scenes.BsdfSpec(scenes.DIFFUSE, (0.5, 0.5, 0.5))]
    spec.meshes.append(scenes.MeshSpec(P.astype(np.float32), F.astype(np.int32), bsdf=0))
    spec.cameras = [scenes.CameraSpec((0.0, 0.0, 4.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 8, 8, 45.0)]
    return api.Scene(spec)


def _mesh(kind, n, rng):
    c = rng.uniform(-1, 1, (n, 1, 3))
    P = c + 0.4 * rng.normal(size=(n, 3, 3))
    if kind == "plane":
        P[:, :, 1] = -1.0
    elif kind == "same":
        P[:] = P[:1]
    elif kind == "degenerate":
        P[::2, 2] = P[::2, 1]
    elif kind == "graded":  # a gradient of sizes, as at a sphere's pole
        P = c * np.geomspace(1e-4, 1, n)[:, None, None] + 0.4 * np.geomspace(1e-4, 1, n)[:, None, None] * (P - c)
    return P.reshape(-1, 3), np.arange(3 * n).reshape(n, 3)


def _rays(n, rng):
    org = rng.uniform(-2, 2, (n, 3))
    d = rng.normal(size=(n, 3))
    d[::7] = np.eye(3)[rng.integers(0, 3, len(d[::7]))] * rng.choice([-1.0, 1.0], (len(d[::7]), 1))  # along an axis
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    tmin, tmax = np.full(n, 1e-2), np.full(n, 1e32)
    tmin[::5], tmax[::5] = -3.0, 0.5     # an interval that starts behind the origin
    f = lambda x: torch.as_tensor(np.ascontiguousarray(x, np.float32))
    return f(org), f(d), f(tmin), f(tmax)


@pytest.mark.parametrize("kind,n", [("soup", 1), ("soup", 2), ("soup", 3), ("soup", 5), ("soup", 16), ("soup", 17),
                                    ("soup", 31), ("soup", 32), ("soup", 33), ("soup", 129), ("soup", 2000),
                                    ("plane", 40), ("same", 40), ("degenerate", 40), ("graded", 300)])
def test_queries_match_brute_force(built_lib, kind, n):
    rng = np.random.default_rng(n)
    P, F = _mesh(kind, n, rng)
    scene = _scene(P, F)
    pos = torch.as_tensor(P.astype(np.float32)).reshape(n, 3, 3)
    for refit in (False, True):
        scene.configure(refit=refit)
        for count in (1, 31, 700):
            org, d, tmin, tmax = _rays(count, rng)
            ref = O.intersect_brute(pos[:, 0], pos[:, 1], pos[:, 2], org, d, tmin, tmax)
            got = [x.cpu() for x in scene.intersect(*(x.cuda() for x in (org, d, tmin, tmax)))]
            assert torch.equal(got[0].long(), ref[0])
            hit = ref[0] >= 0
            for a, b in zip(got[1:], ref[1:]):
                assert torch.equal(a[hit], b[hit])
            vis = scene.occluded(*(x.cuda() for x in (org, d, tmin, tmax))).cpu()
            assert torch.equal(vis, (~hit).int())


def test_rays_without_a_direction_hit_nothing(built_lib):
    rng = np.random.default_rng(0)
    scene = _scene(*_mesh("soup", 200, rng))
    scene.configure()
    org, d, tmin, tmax = _rays(64, rng)
    d[::3] = 0.0
    d[1::3, 1] = float("nan")
    org[2::3, 0] = float("nan")
    args = [x.cuda() for x in (org, d, tmin, tmax)]
    assert bool((scene.intersect(*args)[0] == -1).all())
    assert bool((scene.occluded(*args) == 1).all())


def test_queries_of_every_size_agree(built_lib):
    """A batch's size decides between the two traversals (one ray per thread from
    1/8 of the GPU's lanes to 3/2 of them, or 5/2 in a large tree): the same rays
    give the same results in any batch, at both sides of each limit."""
    lanes = torch.cuda.get_device_properties(0).multi_processor_count * 8 * 128
    gen = torch.Generator(device="cuda").manual_seed(5)
    for spec, high in ((scenes.config1_scene(8, 8), lanes * 3 // 2), (scenes.config2_scene(8, 8, tris=40_000), lanes * 5 // 2)):
        scene = api.Scene(spec)
        scene.configure()
        n = high + 1
        org = torch.randn(n, 3, generator=gen, device="cuda") * 2
        d = torch.randn(n, 3, generator=gen, device="cuda") - 0.5 * org
        d /= d.norm(dim=1, keepdim=True)
        rays = (org, d, torch.full((n,), 1e-2, device="cuda"), torch.full((n,), 1e32, device="cuda"))
        small = lanes // 8 - 1
        parts = [[x[i:i + small].contiguous() for x in rays] for i in range(0, n, small)]
        ref = [torch.cat(x) for x in zip(*(scene.intersect(*p) for p in parts))]
        vis = torch.cat([scene.occluded(*p) for p in parts])
        assert 0.1 < float((ref[0] >= 0).float().mean()) < 0.9
        for k in (lanes // 8 - 1, lanes // 8, high - 1, high, high + 1):
            part = [x[:k].contiguous() for x in rays]
            for a, b in zip(scene.intersect(*part), ref):
                assert torch.equal(a, b[:k])
            assert torch.equal(scene.occluded(*part), vis[:k])


@pytest.mark.parametrize("kind,n", [("nested", 100), ("nested", 512), ("nested", 3000), ("equal", 3000)])
def test_trees_of_nested_boxes_have_a_bounded_height(built_lib, kind, n):
    """Triangles around one centre, from which a ray meets the boxes of all of
    them at once: merged nearest first they made one chain (95 levels for 512, 127
    for 2,048), above the traversal's 72 stack entries, and triangles were missed.
    (The sizes of 100 stay a chain.) Equal boxes tie and chain likewise."""
    rng = np.random.default_rng(n)
    tri = np.array([[1.0, -0.5, -0.5], [-0.5, 1.0, -0.5], [-0.5, -0.5, 1.0]])
    size = np.geomspace(1, 8, n) if kind == "nested" else np.ones(n)
    P = (size[:, None, None] * tri).reshape(-1, 3)
    F = np.arange(3 * n).reshape(n, 3)
    scene = _scene(P, F)
    pos = torch.as_tensor(P.astype(np.float32)).reshape(n, 3, 3)
    org = 0.02 * rng.normal(size=(600, 3))
    d = rng.normal(size=(600, 3))
    d[::2] = -tri[0] + 0.2 * d[::2]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    f = lambda x: torch.as_tensor(np.ascontiguousarray(x, np.float32))
    rays = f(org), f(d), torch.full((600,), 1e-4), torch.full((600,), 20.0)
    ref = O.intersect_brute(pos[:, 0], pos[:, 1], pos[:, 2], *rays)
    hit = ref[0] >= 0
    assert int(hit.sum()) > 100
    for refit in (False, True):
        scene.configure(refit=refit)
        for k in (7, 600):
            part = [x[:k] for x in rays]
            got = [x.cpu() for x in scene.intersect(*(x.cuda() for x in part))]
            assert torch.equal(got[0].long(), ref[0][:k])
            for a, b in zip(got[1:], ref[1:]):
                assert torch.equal(a[hit[:k]], b[:k][hit[:k]])
            assert torch.equal(scene.occluded(*(x.cuda() for x in part)).cpu(), (~hit[:k]).int())


def test_positions_without_a_finite_box_are_refused(built_lib):
    """No tree over triangles whose common box's area overflows, or that have no
    number in some coordinate; single ones of either kind are left alone, and the
    scene works again with other positions."""
    rng = np.random.default_rng(1)
    P, F = _mesh("soup", 50, rng)
    scene = _scene(P, F)
    scene.configure()
    good = scene._raw_positions.clone()
    rays = [x.cuda() for x in _rays(200, rng)]
    ref = [x.clone() for x in scene.intersect(*rays)]
    for value, part in ((3e19, slice(0, 1)), (float("nan"), slice(None)), (float("inf"), slice(7, 8))):
        bad = good.clone()
        bad[part, :2] = value
        scene.set_vertex_positions(bad)
        with pytest.raises(RuntimeError, match="finite"):
            scene.configure()
        scene.set_vertex_positions(good)
        scene.configure()
        for a, b in zip(scene.intersect(*rays), ref):
            assert torch.equal(a, b)
    far = good.clone()
    far[0] = 1e18
    few = good.clone()
    few[:3] = float("nan")   # one triangle
    for ok in (far, few):
        scene.set_vertex_positions(ok)
        scene.configure()
    one = _scene(P[:3] * 1e25, F[:1])
    one.configure()
