"""The device walk when its first guess of the lists' room is too small (it is
counted to its end and run again) and the split of ranges deeper than one
batch of queued levels: the same arrays as the host build."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from jaccpot_b200 import tree, workloads  # noqa: E402

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
