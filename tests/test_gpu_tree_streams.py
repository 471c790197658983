"""A tree built or copied out on one stream and read from another, with the copies
held back behind a bounded spin: the host's reads and the consumers on other
streams see the finished arrays, and the builder's buffers are not handed on before
the copies out of them are done.  The reference is the host build."""

from __future__ import annotations

import copy
import pickle

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from jaccpot_b200 import engine, tree, workloads  # noqa: E402

FIELDS = ("permutation", "inverse_permutation", "node_ranges", "left_child", "right_child", "parent", "node_level",
          "leaf_of_particle", "far_offsets", "far_sources", "near_offsets", "near_leaves", "centers_f64", "radii_f64",
          "m2l_targets")
SPIN = 200_000_000  # clock cycles, about a tenth of a second


def _poison(nbytes):
    """Leaves freed memory that holds no old copy of the arrays for the next buffer."""
    torch.full((nbytes,), 0x55, dtype=torch.uint8, device="cuda")


def _same(host, dev):
    for f in FIELDS:
        assert np.array_equal(getattr(host, f), getattr(dev, f)), f


@pytest.fixture
def particles():
    return workloads.GENERATORS["plummer"](20_000, 9)


def test_host_reads_wait_for_the_copies(particles):
    pos, mass = particles
    host = tree.build_topology(pos, mass, leaf_size=16, theta=0.6)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        _poison(1 << 26)
        with tree.DeviceTree(pos, mass, leaf_size=16, theta=0.6) as dtree:
            torch.cuda._sleep(SPIN)
            topo = dtree.topology()
    _same(host, topo)


def test_moved_geometry_waits_too(particles):
    pos, mass = particles
    host = tree.build_topology(pos, mass, leaf_size=16, theta=0.6)
    topo = tree.build_topology(pos, mass, leaf_size=16, theta=0.6, device="cuda")
    c = torch.from_numpy(host.centers_f64 + 1.0).cuda()
    r = torch.from_numpy(host.radii_f64 * 2.0).cuda()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        _poison(1 << 22)
        torch.cuda._sleep(SPIN)
        moved = topo.with_geometry(c.clone(), r.clone())
    assert np.array_equal(moved.centers_f64, host.centers_f64 + 1.0)
    assert np.array_equal(moved.radii_f64, host.radii_f64 * 2.0)
    assert np.array_equal(moved.far_sources, host.far_sources) and np.array_equal(topo.radii_f64, host.radii_f64)


def test_buffers_outlive_copies_on_another_stream(particles):
    pos, mass = particles
    host = tree.build_topology(pos, mass, leaf_size=16, theta=0.6)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        dtree = tree.DeviceTree(pos, mass, leaf_size=16, theta=0.6)
    with torch.cuda.stream(b):
        torch.cuda._sleep(SPIN)
        topo = dtree.topology()
    dtree.free()
    with torch.cuda.stream(a):  # takes what the first tree gave back
        other = tree.DeviceTree(pos[::-1].copy() * 3.0, mass, leaf_size=16, theta=0.5)
    _same(host, topo)
    other.free()


def test_a_pass_on_another_stream_waits(particles):
    pos, mass = particles
    p, m = torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda()
    ref = engine.Pass(engine.DeviceTopology(tree.build_topology(pos, mass, leaf_size=16, theta=0.6), "cuda"), 4)
    ref.load_particles(p, m)
    want = ref.run().clone()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        with tree.DeviceTree(p, m, leaf_size=16, theta=0.6) as dtree:
            torch.cuda._sleep(SPIN)
            topo = dtree.topology()
    ps = engine.Pass(engine.DeviceTopology(topo, "cuda"), 4)
    del topo
    ps.load_particles(p, m)
    assert torch.equal(ps.run(), want)


@pytest.mark.parametrize("gears", [False, True])
@pytest.mark.parametrize("again", [lambda t: pickle.loads(pickle.dumps(t)), copy.deepcopy, copy.copy])
def test_saved_and_copied_topologies_are_host_arrays(particles, again, gears):
    pos, mass = particles
    with tree.DeviceTree(pos, mass, leaf_size=16, theta=0.6) as dtree:
        if gears:
            nn = dtree.info.num_nodes
            dtree.adaptive_walk(torch.ones((nn, 4), device="cuda"), torch.ones(nn, device="cuda"), G=1.0, eps=1e-2,
                                gear_orders=(1, 3))
        topo = dtree.topology()
    back = again(topo)
    assert type(back) is tree.Topology
    assert all(v is None or isinstance(v, (int, float, tuple, np.ndarray)) for v in vars(back).values())
    assert (back.theta, back.leaf_size, back.gear_orders) == (topo.theta, topo.leaf_size, topo.gear_orders)
    assert (back.far_gears is None) == (not gears) and (not gears or np.array_equal(back.far_gears, topo.far_gears))
    _same(back, topo)
