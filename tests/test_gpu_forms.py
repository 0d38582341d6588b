"""The loop forms (kernel_mode 0: one thread per photon, 1: persistent threads, 2: wavefront) give the same
photons, seq and hits bit for bit, in geometries of each kind of closest-hit search."""
import numpy as np
import pytest

from opticks_b200 import foundry as F
from opticks_b200 import scenes

pytestmark = pytest.mark.gpu


def _detector(n):
    fd, lib, icdf = scenes.detector()
    phys = lib.arrays()
    phys["icdf"] = icdf
    return fd, phys, scenes.detector_gensteps(1, n, seed=n, lib=lib)


def _zoo(n):
    fd, lib, _, _ = scenes.leaf_zoo_detector(1)
    return fd, lib.arrays(), scenes.torch_genstep(n, wavelength=440.0, radius=0.0)[None]


def filled(world, extra=(), each=20):
    """bodies throughout the volume, its centre too, so that no ball is free of the hierarchy"""
    fd = F.Foundry()
    fd.add_inst(np.eye(4), fd.add_solid("world", [fd.add_prim(world, 0)]))
    cap = F.op("union", F.zsphere(254.0, 0.0, 190.0), F.cylinder(50.0, -200.0, 0.0))
    shell = F.op("difference", F.sphere(250.0), F.sphere(150.0))
    rng = np.random.default_rng(5)
    for i, b in enumerate([cap, shell, F.sphere(180.0), F.cylinder(90.0, -250.0, 120.0), *extra]):
        s = fd.add_solid(f"s{i}", [fd.add_prim(b, 1)])
        for k in range(each):
            at = rng.uniform(-1800.0, 1800.0, 3) if (i or k) else np.array([30.0, 20.0, 10.0])
            fd.add_inst(F.look_at_z(at, rng.normal(size=3)), s, sensor_identifier=i, sensor_index=i)
    return fd


def _filled(world, extra=()):
    def make(n):
        _, lib, _, _ = scenes.leaf_zoo_detector(1)
        return filled(world, extra), lib.arrays(), scenes.torch_genstep(n, wavelength=440.0, radius=0.0, pos=(500.0, 300.0, 200.0))[None]
    return make


CONE = F.cone(120.0, -100.0, 60.0, 100.0)
SCENES = {
    "detector": _detector,                                                     # plain globals, a ball free of the hierarchy
    "zoo": _zoo,                                                               # further leaves
    "sphere world": _filled(F.sphere(4000.0)),                                 # plain global, no ball
    "cylinder world": _filled(F.cylinder(4000.0, -4000.0, 4000.0)),            # a global leaf without a parameter row
    "with cones": _filled(F.sphere(4000.0), (CONE,)),                          # the general evaluator in the hierarchy
}


def simulate(E, scene, n, event, **kw):
    fd, phys, gs = scene(n)
    eng = E.Engine(fd.arrays(), phys, E.default_config(max_photon=n, **kw))
    r = eng.simulate(gs, event)
    r["stats"] = eng.last_call_stats()
    eng.close()
    return r


def assert_same(a, b):
    assert a["status"] == 0 and b["status"] == 0
    for k in ("photon", "seq", "hit"):
        np.testing.assert_array_equal(a[k].view(np.uint32), b[k].view(np.uint32))


@pytest.mark.parametrize("name", SCENES)
def test_one_thread_per_photon_equals_the_persistent_loop(cuda, name):
    from opticks_b200 import engine as E
    a, b = (simulate(E, SCENES[name], 200_000, 3, kernel_mode=m) for m in (0, 1))
    assert_same(a, b)


# ---------------------------------------------------------------- closest hits
@pytest.mark.parametrize("polish", [0, 1])
@pytest.mark.parametrize("name", ["detector", "zoo", "sphere world", "with cones"])
def test_trace_in_pieces(cuda, name, polish):
    """queries up to and beyond the lanes of one resident grid (148 SMs of 3 or 4 blocks of 128: one thread per ray
    and the stream of rays) against queries of a few thousand"""
    from opticks_b200 import engine as E
    fd, phys, _ = SCENES[name](1)
    eng = E.Engine(fd.arrays(), phys, E.default_config(max_photon=64, root_polish=polish))
    n = 262_145
    rays = scenes.scan_rays(n, seed=5, half=11000.0 if name == "detector" else 1400.0)
    piece = 20_011
    ref = np.concatenate([eng.trace(np.ascontiguousarray(rays[:, a:a + piece]), 0.05)[0] for a in range(0, n, piece)])
    for m in (1, 31, 2369, 56_832, 56_833, 75_776, 75_777, n):
        got, st = eng.trace(np.ascontiguousarray(rays[:, :m]), 0.05)
        assert st == 0
        np.testing.assert_array_equal(got.view(np.uint32), ref[:m].view(np.uint32))
    eng.close()


# ---------------------------------------------------------------- root polish
@pytest.mark.parametrize("name,n", [("detector", 16_383), ("detector", 16_384), ("detector", 524_288), ("zoo", 50_000),
                                    ("sphere world", 300_000), ("cylinder world", 50_000), ("with cones", 300_000)])
def test_polished_forms_agree(cuda, name, n):
    """root_polish: the starting kernel's own sphere, the tail kernel, the rounds and the one-kernel loops"""
    from opticks_b200 import engine as E
    ref = simulate(E, SCENES[name], n, 3, kernel_mode=1, root_polish=1)
    for mode in (0, 2):
        assert_same(simulate(E, SCENES[name], n, 3, kernel_mode=mode, root_polish=1), ref)


# ---------------------------------------------------------------- fixed rounds
@pytest.mark.parametrize("name", ["sphere world", "cylinder world", "with cones"])
@pytest.mark.parametrize("rounds", [2, 3])
@pytest.mark.parametrize("polish", [0, 1])
def test_fixed_rounds_equal_the_persistent_loop(cuda, name, rounds, polish):
    """more photons than the small-call rule takes, and no ball or a global leaf without a parameter row: rounds of
    a closest-hit and a physics kernel, then the tail kernel"""
    from opticks_b200 import engine as E
    n = 262_145
    ref = simulate(E, SCENES[name], n, 2, kernel_mode=1, root_polish=polish)
    got = simulate(E, SCENES[name], n, 2, kernel_mode=2, root_polish=polish, wave_rounds=rounds)
    assert got["stats"]["wave_rounds"] == rounds          # the schedule this test is about
    assert_same(got, ref)


@pytest.mark.parametrize("name", ["sphere world", "with cones"])
def test_captured_fixed_rounds(cuda, name):
    """the same in a batched call, captured as a graph and replayed"""
    from opticks_b200 import engine as E
    torch = cuda
    fd, phys, _ = SCENES[name](1)
    counts = [100_000, 1, 70_000, 110_000]
    gs = np.concatenate([scenes.torch_genstep(c, wavelength=440.0, radius=0.0, pos=(500.0, 300.0, 200.0))[None] for c in counts])
    N = sum(counts)
    g, ev = torch.from_numpy(gs).cuda(), torch.arange(3, 3 + len(counts), dtype=torch.int32, device="cuda")
    outs = []
    for mode, calls in ((1, 1), (2, 3)):
        eng = E.Engine(fd.arrays(), phys, E.default_config(max_photon=max(counts), kernel_mode=mode, wave_rounds=2, use_graph=1))
        ph = torch.empty((N, 4, 4), dtype=torch.float32, device="cuda")
        sq = torch.empty((N, 2, 2), dtype=torch.int64, device="cuda")
        for _ in range(calls):
            ph.fill_(0.0)
            sq.fill_(0)
            _, st = eng.simulate_batched_device(g, ev, N, photon=ph, seq=sq, stream=torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            assert st == 0
        stats = eng.last_call_stats()
        eng.close()
        outs.append((ph.clone(), sq.clone()))
    assert stats["graph"] == 1
    assert torch.equal(outs[0][0].view(torch.int32), outs[1][0].view(torch.int32)) and torch.equal(outs[0][1], outs[1][1])
