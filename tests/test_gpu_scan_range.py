"""Rays at the ends of what a scan accepts (directions of any length, no direction, NaN, intervals that open
behind the origin): the bounding-ball test ahead of the tree drops none that the leaves would hit."""
import numpy as np
import pytest

from opticks_b200 import foundry as F
from opticks_b200 import scenes
from oracle import oracle as O

pytestmark = pytest.mark.gpu

R = 250.0


def _scan(trees, rays, t_min=0.0, polish=0):
    import torch
    from opticks_b200 import engine as E
    fd = F.Foundry()
    prims = [fd.add_prim(t, 0) for t in trees]
    fd.add_inst(np.eye(4), fd.add_solid("s", prims))
    _, lib, _, _ = scenes.sphere_in_box(1)
    A = fd.arrays()
    eng = E.Engine(A, lib.arrays(), E.default_config(max_photon=64))
    d = torch.from_numpy(np.ascontiguousarray(rays, dtype=np.float32)).cuda()
    out = torch.empty((rays.shape[1], 4), device="cuda")
    got = []
    for p in prims:
        eng.scan_device(p, d, rays.shape[1], out, t_min, polish)
        torch.cuda.synchronize()
        got.append(out.cpu().numpy())
    eng.close()
    return A, prims, got


@pytest.mark.parametrize("length", [1e-14, 1e-6, 1.0, 1e9, 6.64e16])
def test_hits_do_not_depend_on_the_direction_s_length(cuda, length):
    """origins at 1.14 radii, lines at 0.72 to 0.92 of the radius: every ray hits the sphere.  At 6.64e16 the
    squared direction times the squared distance exceeds FP32, the leaf's own products do not."""
    rng = np.random.default_rng(3)
    n = 4097
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    v = np.cross(u, rng.normal(size=(n, 3)))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    cos = np.sqrt(rng.uniform(0.35, 0.6, n))[:, None]
    o = np.sqrt(1.3) * R * u
    d = -cos * u + np.sqrt(1.0 - cos * cos) * v
    rays = np.concatenate([o, d * length], 1).T.astype(np.float32)
    _, _, (got, tree) = _scan([F.sphere(R), F.op("union", F.sphere(R), F.sphere(0.5 * R))], rays)
    o, d = rays[:3].T.astype(np.float64), rays[3:].T.astype(np.float64)
    a, b, c = (d * d).sum(1), (o * d).sum(1), (o * o).sum(1) - R * R
    near = (-b - np.sqrt(b * b - a * c)) / a
    assert np.all(got[:, 3] > 0.0) and np.all(tree[:, 3] > 0.0)
    # FP32 root c / q of operands a few ulp off, c within 4 ulp of |o|^2 = 1.3 R^2
    np.testing.assert_allclose(got[:, 3], near, rtol=1e-5)
    np.testing.assert_allclose(tree[:, 3], near, rtol=1e-5)


def test_rays_without_a_direction_or_a_number_miss(cuda):
    rays = scenes.scan_rays(2000, seed=4, half=400.0)
    base = rays.copy()
    rays[3:, 3::7] = 0.0
    rays[0, 5::11] = np.nan
    rays[4, 6::13] = np.nan
    bad = (rays[3:] == 0.0).all(0) | np.isnan(rays).any(0)
    trees = [F.sphere(R), F.op("difference", F.sphere(R), F.sphere(150.0))]
    _, _, got = _scan(trees, rays)
    _, _, ref = _scan(trees, base)
    for g, r in zip(got, ref):
        assert not g[bad].any()
        np.testing.assert_array_equal(g[~bad].view(np.uint32), r[~bad].view(np.uint32))
        assert (g[:, 3] > 0).any()


def test_intervals_that_open_behind_the_origin(cuda):
    rays = scenes.scan_rays(20_001, seed=8, half=600.0)
    trees = [F.sphere(R), F.cylinder(200.0, -150.0, 150.0), F.zsphere(R, -50.0, 190.0)]
    A, prims, got = _scan(trees, rays, t_min=-300.0)
    for p, g in zip(prims, got):
        root = int(A["prim"].view(np.int32).reshape(-1, 16)[p, 1])
        ref, _ = O.csg_scan(A["node"], A["itra"], root, rays, -300.0)
        hg, hr = g[:, 3] != 0, ref[:, 3] != 0
        assert (g[:, 3] < 0).sum() > 100
        assert np.mean(hg != hr) <= 1e-3                     # fast-math against IEEE at the silhouette
        both = hg & hr
        assert np.mean(np.abs(g[both, 3] - ref[both, 3]) <= 0.1) >= 0.99


@pytest.mark.parametrize("n", [30_001, 300_001])              # one thread per ray; the stream of rays
def test_trace_of_rays_that_are_no_numbers(cuda, n):
    """a NaN ray neither holds up nor changes the others"""
    from opticks_b200 import engine as E
    fd, lib, icdf = scenes.detector()
    phys = lib.arrays()
    phys["icdf"] = icdf
    eng = E.Engine(fd.arrays(), phys, E.default_config(max_photon=64))
    rays = scenes.scan_rays(n, seed=2, half=11000.0)
    base = rays.copy()
    rays[1, 4::9] = np.nan
    rays[3:, 7::31] = np.nan
    ok = ~np.isnan(rays).any(0)
    a, _ = eng.trace(rays, 0.05)
    b, _ = eng.trace(base, 0.05)
    eng.close()
    np.testing.assert_array_equal(a[ok].view(np.uint32), b[ok].view(np.uint32))
