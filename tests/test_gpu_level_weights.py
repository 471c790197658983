"""Block-step weights of the far pairs (jb_far_level_weights): the weight of the
finer of the two nodes' rungs, a node's rung being its particles' finest,
against numpy, with rungs outside the table and a tree of one leaf."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from jaccpot_b200 import engine, tree, workloads  # noqa: E402


@pytest.mark.parametrize("kind,n,leaf,levels", [("uniform", 5, 8, 3), ("uniform", 700, 1, 1), ("plummer", 9000, 33, 4),
                                                ("clustered", 30_000, 16, 32)])
def test_weights_equal_numpy(kind, n, leaf, levels):
    pos, mass = workloads.GENERATORS[kind](n, 2)
    topo = tree.build_topology(pos, mass, leaf_size=leaf, theta=0.7, device="cuda")
    ps = engine.Pass(engine.DeviceTopology(topo, "cuda"), 3)
    rng = np.random.default_rng(5)
    rung = rng.integers(-2, levels + 2, n).astype(np.int32)
    lw = rng.normal(size=levels).astype(np.float32)
    for _ in range(2):  # the scratch is left ready for the next call
        got = ps.far_level_weights(torch.from_numpy(rung).cuda(), torch.from_numpy(lw).cuda()).cpu().numpy()
    node = np.array([max(-1, rung[a:b + 1].max()) for a, b in topo.node_ranges])
    want = lw[np.clip(np.maximum(node[topo.far_pair_targets()], node[topo.far_sources]), 0, levels - 1)]
    assert got.shape == (topo.num_far_pairs,) and np.array_equal(got, want)


def test_rungs_and_weights_of_any_type_and_layout():
    n = 5000
    pos, mass = workloads.GENERATORS["plummer"](n, 2)
    topo = tree.build_topology(pos, mass, leaf_size=16, theta=0.7, device="cuda")
    ps = engine.Pass(engine.DeviceTopology(topo, "cuda"), 3)
    ps.load_particles(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda())
    rung = torch.from_numpy(np.random.default_rng(5).integers(0, 4, n).astype(np.int32)).cuda()
    lw = torch.tensor([1.0, 0.5, 0.25, 0.125], device="cuda")
    want_w, want = ps.far_level_weights(rung, lw).clone(), ps.run_weighted(rung, lw).clone()
    odd = (torch.stack([rung, rung - 7], dim=1)[:, 0].long(), torch.stack([lw, lw + 1], dim=1).double()[:, 0])
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for r, w in (odd, (odd[0].cpu(), odd[1].cpu())):
        assert torch.equal(ps.far_level_weights(r, w), want_w)
        assert torch.equal(ps.run_weighted(r, w), want)
        got = ps.far_level_weights(r, w, side)
        side.synchronize()
        assert torch.equal(got, want_w)
    for call in (ps.far_level_weights, ps.run_weighted, ps.evaluate_weighted):
        with pytest.raises(ValueError, match="one rung per particle"):
            call(rung[:-1], lw)
