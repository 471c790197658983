"""The device walk when its first guess of the lists' or the frontier's room is
too small (it runs again with more) and the split of ranges deeper than one
batch of queued levels: the same arrays as the host build."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from jaccpot_b200 import tree, workloads  # noqa: E402
from oracle import adaptive_walk as aw  # noqa: E402

FIELDS = ("permutation", "inverse_permutation", "node_ranges", "left_child", "right_child", "parent", "node_level",
          "level_offsets", "leaf_of_particle", "far_offsets", "far_sources", "near_offsets", "near_leaves", "centers_f64",
          "radii_f64", "m2l_targets")


def _same(pos, mass, leaf, theta):
    a = tree.build_topology(pos, mass, leaf_size=leaf, theta=theta)
    b = tree.build_topology(pos, mass, leaf_size=leaf, theta=theta, device="cuda")
    assert (a.num_nodes, a.num_internal, a.num_levels, a.max_leaf_occupancy, a.num_far_pairs, a.num_near_pairs) == (
        b.num_nodes, b.num_internal, b.num_levels, b.max_leaf_occupancy, b.num_far_pairs, b.num_near_pairs)
    for f in FIELDS:
        assert np.array_equal(getattr(a, f), getattr(b, f)), f
    return a


@pytest.mark.parametrize("n,leaf,theta,grows", [(3000, 1, 0.02, "far"), (3000, 3, 0.02, "near"), (1200, 1, 0.2, "")])
def test_lists_longer_than_the_first_room(n, leaf, theta, grows):
    pos, mass = workloads.plummer(n, 5)
    t = _same(pos, mass, leaf, theta)
    if grows == "far":  # single particles have no extent: every pair is far
        assert t.num_far_pairs > max(1 << 16, 256 * t.num_nodes)
    if grows == "near":
        assert t.num_near_pairs > max(1 << 16, 256 * t.num_leaves)


@pytest.mark.parametrize("copies,leaf", [(2, 1), (300, 2), (513, 64), (5000, 1)])  # 6 to 16 levels
def test_ranges_of_equal_codes_split_to_the_end(copies, leaf):
    rng = np.random.default_rng(1)
    pos = np.concatenate([np.repeat(rng.uniform(-1, 1, (3, 3)), copies, axis=0), rng.uniform(-1, 1, (50, 3)) * 1e-9])
    _same(pos, np.ones(pos.shape[0]), leaf, 0.5)


def _widest_frontier(t, theta):
    """Node pairs in the widest step of the theta walk over t (breadth first)."""
    ni, left, right = t.num_internal, t.left_child.astype(np.int64), t.right_child.astype(np.int64)
    A = B = np.zeros(1, np.int64)
    widest = 0
    while A.size:
        widest = max(widest, A.size)
        own = A == B
        st = A[own][A[own] < ni]
        a, b = A[~own], B[~own]
        d2 = ((t.centers_f64[a] - t.centers_f64[b]) ** 2).sum(1)
        r = t.radii_f64[a] + t.radii_f64[b]
        far = (d2 > 0) & (r * r <= theta * theta * d2)
        open_ = ~far & ~((a >= ni) & (b >= ni))
        a, b = a[open_], b[open_]
        sa = (a < ni) & ((b >= ni) | (t.radii_f64[a] >= t.radii_f64[b]))
        x, y, u, v = a[sa], b[sa], a[~sa], b[~sa]
        A = np.concatenate([left[st], right[st], left[st], left[x], right[x], u, u])
        B = np.concatenate([left[st], right[st], right[st], y, y, left[v], right[v]])
    return widest


@pytest.mark.parametrize("kind,n,leaf,theta", [("uniform", 16384, 16, 0.2), ("uniform", 6000, 4, 0.2),
                                               ("uniform", 8001, 16, 0.1), ("plummer", 3000, 1, 0.02)])
def test_frontier_wider_than_the_first_room(kind, n, leaf, theta):
    pos, mass = workloads.GENERATORS[kind](n, 5)
    t = _same(pos, mass, leaf, theta)
    assert _widest_frontier(t, theta) > max(1 << 16, 64 * t.num_nodes)


def test_directed_frontier_wider_than_the_first_room():
    pos, mass = workloads.GENERATORS["uniform"](6000, 5)
    with tree.DeviceTree(pos, mass, leaf_size=4, theta=0.6, device="cuda") as dtree:
        t0 = dtree.topology()
        nn, top = t0.num_nodes, 3
        power = torch.rand((nn, top + 1), device="cuda", dtype=torch.float64)
        fs = torch.rand(nn, device="cuda") + 0.5
        args = dict(G=1.0, eps=1e2, theta_max=0.2)
        dtree.adaptive_walk(power, fs, gear_orders=(1, top), **args)
        t = dtree.topology()
    want = aw.adaptive_walk(t0.left_child, t0.right_child, t0.centers_f64, t0.radii_f64, t0.num_internal,
                            power.cpu().numpy(), fs.cpu().numpy(), orders=(1, top), **args)
    # the directed walk visits every pair of the theta walk's both ways, and more
    assert _widest_frontier(t0, args["theta_max"]) > max(1 << 16, 64 * nn)
    for g, w in zip((t.far_offsets, t.far_sources, t.far_gears, t.near_offsets, t.near_leaves), want):
        assert np.array_equal(np.asarray(g), np.asarray(w))
