"""Rules that pick a kernel or a variant by size, geometry or key range, at the edges where they turn:
spread and starting-kernel calls, the one-launch hit copy, the closest-hit kernels with and without
the general evaluator, the scan's bounding ball, the event jump tables and the merge's key table."""
import numpy as np
import pytest

from opticks_b200 import foundry as F
from opticks_b200 import scenes
from oracle import merge as M
from oracle import oracle as O
from tests.test_merge import SD, random_records

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def _rays(n, seed, half=1500.0):
    return scenes.scan_rays(n, seed=seed, half=half)


def _props():
    _, lib, _, _ = scenes.sphere_in_box(1)
    return lib.arrays()


# ---------------------------------------------------------------- call sizes
@pytest.fixture(scope="module")
def forms(cuda):
    from opticks_b200 import engine as E
    fd, lib, icdf = scenes.detector()
    phys = lib.arrays()
    phys["icdf"] = icdf
    eng = [E.Engine(fd.arrays(), phys, E.default_config(max_photon=600_000, num_sensor=scenes.NUM_PMT, kernel_mode=m)) for m in (1, 2)]
    yield eng, lib
    for e in eng:
        e.close()


@pytest.mark.parametrize("n", [1, 31, 33, 1000, 16383, 16384, 57_001, 262_144, 262_145, 524_288])
def test_call_sizes_equal_the_one_kernel_loop(forms, n):
    (one, wave), lib = forms
    gs = scenes.detector_gensteps(1, n, seed=n, lib=lib)
    a, b = one.simulate(gs, 6, sensor_hits=True), wave.simulate(gs, 6, sensor_hits=True)
    assert a["status"] == 0 and b["status"] == 0
    for k in ("photon", "seq", "hit", "sensor_hits"):
        np.testing.assert_array_equal(a[k].view(np.uint32), b[k].view(np.uint32))
    sel = (_bits(b["photon"]).reshape(-1, 4, 4)[:, 3, 3] & SD) == SD
    np.testing.assert_array_equal(_bits(b["hit"]), _bits(b["photon"][sel]))
    assert b["num_hit"] == int(sel.sum())


# ---------------------------------------------------------------- event jumps
@pytest.mark.parametrize("event", [1, 15, 16, 4095, 65536, 0x10203040, 2**31 - 1])
def test_event_streams_are_the_skipahead_streams(cuda, event):
    """the first uniform of a torch photon is its zenith: cos(theta) = 1 - 2 u, u from cuRAND's own skipahead"""
    from opticks_b200 import engine as E
    fd, lib, _, _ = scenes.sphere_in_box(1)
    n = 300
    gs = scenes.torch_genstep(n)[None]
    for mode in (0, 1, 2):
        eng = E.Engine(fd.arrays(), lib.arrays(), E.default_config(max_photon=n, max_bounce=0, kernel_mode=mode))
        z = eng.simulate(gs, event)["photon"][:, 1, 2]
        u = eng.rng_sequence(event, 0, n, 1)[:, 0]
        eng.close()
        np.testing.assert_allclose(z, 1.0 - 2.0 * u, atol=2.0 ** -22)      # one FP32 rounding each of 2u, 1 - 2u


# ---------------------------------------------------------------- closest hit
def _bodies():
    cap = F.op("union", F.zsphere(254.0, 0.0, 190.0), F.cylinder(50.0, -200.0, 0.0))
    lens = F.op("intersection", F.translate(F.sphere(300.0), 0.0, 0.0, 200.0), F.translate(F.sphere(300.0), 0.0, 0.0, -200.0))
    cup = F.op("difference", F.cylinder(200.0, -150.0, 150.0), F.translate(F.zsphere(180.0, -180.0, 100.0), 0.0, 0.0, 120.0))
    shell = F.op("difference", F.sphere(250.0), F.sphere(150.0))
    return [cap, lens, cup, shell, F.sphere(180.0), F.translate(F.zsphere(220.0, -100.0, 150.0), 20.0, -30.0, 10.0), F.cylinder(90.0, -250.0, 120.0)]


def _scene(extra=None):
    fd = F.Foundry()
    world = fd.add_prim(F.sphere(4000.0), 0)
    inner = fd.add_prim(F.box3(7000.0, 7000.0, 7000.0), 0)
    fd.add_inst(np.eye(4), fd.add_solid("world", [world, inner]))
    rng = np.random.default_rng(5)
    for i, b in enumerate(_bodies() + ([extra] if extra is not None else [])):
        s = fd.add_solid(f"s{i}", [fd.add_prim(b, 1)])
        for _ in range(6):
            p = rng.uniform(-1300.0, 1300.0, 3)
            fd.add_inst(F.look_at_z(p, rng.normal(size=3)), s, sensor_identifier=i, sensor_index=i)
    return fd


@pytest.mark.parametrize("n", [1, 33, 5000, 100_001])
def test_trace_variants_agree(cuda, n):
    """the variant without the general evaluator against the one a cone in the scene asks for, and both
    against the FP64 distance to the prim they name"""
    from opticks_b200 import engine as E
    rays = _rays(n, seed=n)
    plain, general = _scene(), _scene(F.cone(120.0, -100.0, 60.0, 100.0))
    out = []
    for fd in (plain, general):
        eng = E.Engine(fd.arrays(), _props(), E.default_config(max_photon=64))
        prd, st = eng.trace(rays, 0.05)
        eng.close()
        assert st == 0
        out.append(prd)
    prim = _bits(out[1]).reshape(n, 2, 4)[:, 1, 3] >> 16
    cone = prim == len(_bodies()) + 2
    np.testing.assert_array_equal(_bits(out[0][~cone]), _bits(out[1][~cone]))
    for fd, prd in zip((plain, general), out):
        w = _bits(prd).reshape(n, 2, 4)
        t64 = O.trace_t64(fd.arrays(), rays, (w[:, 1, 2] >> 16).astype(np.int32), (w[:, 1, 3] >> 16).astype(np.int32), 0.05)
        # FP32 roots of bodies of a few hundred mm from a few m: millimetres at grazing, far less elsewhere
        assert np.mean(np.abs(prd[:, 0, 3] - t64) <= 0.2) >= 0.99


# ---------------------------------------------------------------- scan
@pytest.mark.parametrize("n", [1, 31, 33, 7105, 60_001])
@pytest.mark.parametrize("t_min", [0.0, 300.0])
def test_scan_sizes_against_the_oracle(cuda, n, t_min):
    from opticks_b200 import engine as E
    fd = F.Foundry()
    comp = F.sphere(200.0)
    comp.complement = True
    roots = _bodies() + [comp, F.op("intersection", F.sphere(250.0), comp), F.op("difference", F.box3(300.0, 200.0, 500.0), F.translate(F.sphere(150.0), 0.0, 0.0, 200.0))]
    prims = [fd.add_prim(b, 0) for b in roots]
    fd.add_inst(np.eye(4), fd.add_solid("scan", prims))
    A = fd.arrays()
    eng = E.Engine(A, _props(), E.default_config(max_photon=64))
    rays = _rays(n, seed=n + 1, half=700.0)
    for p in prims:
        got = eng.scan(p, rays, t_min)
        root = int(A["prim"].view(np.int32).reshape(-1, 16)[p, 1])
        ref, _ = O.csg_scan(A["node"], A["itra"], root, rays, t_min)
        hg, hr = got[:, 3] > 0, ref[:, 3] > 0
        assert np.mean(hg != hr) <= 1e-3, p                  # fast-math against IEEE at the silhouette
        both = hg & hr
        if both.sum() > 100:
            assert np.mean(np.abs(got[both, 3] - ref[both, 3]) <= 0.1) >= 0.99, p
    eng.close()


@pytest.mark.parametrize("far", [1e3, 1e4, 1e5])
def test_scan_ball_keeps_far_rays(cuda, far):
    """rays from far away through the inner nine tenths of a sphere: none may be dropped"""
    from opticks_b200 import engine as E
    fd = F.Foundry()
    p = fd.add_prim(F.translate(F.sphere(250.0), 40.0, -20.0, 10.0), 0)
    fd.add_inst(np.eye(4), fd.add_solid("s", [p]))
    eng = E.Engine(fd.arrays(), _props(), E.default_config(max_photon=64))
    rng = np.random.default_rng(int(far))
    n = 20_000
    o = rng.normal(size=(n, 3))
    o *= far / np.linalg.norm(o, axis=1, keepdims=True)
    aim = rng.normal(size=(n, 3))
    aim *= 225.0 * rng.random((n, 1)) / np.linalg.norm(aim, axis=1, keepdims=True)
    d = aim + (40.0, -20.0, 10.0) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    got = eng.scan(p, np.concatenate([o, d], 1).T.astype(np.float32))
    away = eng.scan(p, np.concatenate([o, -d], 1).T.astype(np.float32))
    eng.close()
    assert np.all(got[:, 3] > 0) and not np.any(away[:, 3] > 0)


# ---------------------------------------------------------------- merge
@pytest.mark.parametrize("lite", [0, 1])
@pytest.mark.parametrize("tmax,num_id,tw", [(40.0, 60, 1.0),          # a few thousand cells: the table
                                            (1.0e5, 10, 0.0625),      # 15.9M cells: just in the table
                                            (1.0e5, 11, 0.0625),      # 17.5M: the sort
                                            (1.0e9, 60000, 1.0)])     # 32-bit buckets: the sort
@pytest.mark.parametrize("n", [1, 2049, 30_001])
def test_merge_ranges(forms, lite, tmax, num_id, tw, n):
    eng = forms[0][0]
    rec = random_records(n, lite, np.random.default_rng(n + num_id), num_id=num_id, tmax=tmax, tq=tmax / 200.0)
    for mask in (0xFFFFFFFF, SD, 0):
        got, ref = eng.merge_hits(rec, mask, tw), M.merge(rec, mask, tw)
        assert got.shape == ref.shape
        np.testing.assert_array_equal(_bits(got), _bits(ref))
