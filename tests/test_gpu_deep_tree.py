"""A caller's own tree, deeper than any the builders make: a chain of one particle
to a leaf.  The schedules of the sweeps refuse it or hold everything, the forward
pass goes level by level (all pairs near, so it is a direct sum: p99 within the 1e-5
of every FP32 parity test), the adjoint says what it is built for."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from jaccpot_b200 import _lib, engine, tree, workloads  # noqa: E402


def _chain(leaves, far):
    ni, nn = leaves - 1, 2 * leaves - 1
    i = np.arange(ni)
    parent = np.empty(nn, np.int32)
    parent[0], parent[1:ni] = -1, i[:-1]
    parent[ni:] = np.minimum(np.arange(leaves), ni - 1)
    ranges = np.concatenate([np.stack([i, np.full(ni, leaves - 1)], 1), np.repeat(np.arange(leaves)[:, None], 2, 1)])
    counts = np.zeros(nn, np.int64)
    if far:  # every internal node below the root has the leaf beside it
        counts[1:ni] = 1
    near = np.array([k for j in range(leaves) for k in range(leaves) if k != j], np.int32)
    return tree.Topology(
        num_particles=leaves, num_nodes=nn, num_internal=ni, num_leaves=leaves, num_levels=ni, max_leaf_occupancy=1,
        leaf_size=1, theta=0.5, permutation=np.arange(leaves), inverse_permutation=np.arange(leaves),
        node_ranges=ranges.astype(np.int32), left_child=(ni + i).astype(np.int32),
        right_child=np.concatenate([i[1:], [nn - 1]]).astype(np.int32), parent=parent,
        node_level=np.concatenate([i, np.minimum(np.arange(leaves) + 1, ni)]).astype(np.int32),
        level_offsets=np.arange(ni + 1, dtype=np.int32), leaf_of_particle=np.arange(leaves, dtype=np.int32),
        far_offsets=np.concatenate([[0], np.cumsum(counts)]),
        far_sources=(ni + i[1:] - 1).astype(np.int32) if far else np.zeros(0, np.int32),
        near_offsets=np.arange(leaves + 1, dtype=np.int64) * (leaves - 1), near_leaves=near,
        centers_f64=np.zeros((nn, 3)), radii_f64=np.zeros(nn),
        m2l_targets=np.nonzero(counts)[0].astype(np.int32))


@pytest.mark.parametrize("leaves", [150, 209, 210, 300, 600])
def test_chain(leaves):
    topo = _chain(leaves, far=False)
    dt = engine.DeviceTopology(topo, "cuda")
    dt.validate()
    deep = topo.num_levels > _lib.JB_M2M_HOPS_MAX_LEVELS
    ps = engine.Pass(dt, 3, G=1.0, eps2=1e-4)
    assert ps.m2m_hops == (not deep)
    if leaves == 600:
        with pytest.raises(_lib.JBError):
            dt.m2m_hops()
    pos, mass = workloads.plummer(leaves, 2)
    ps.load_particles(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda())
    got = ps.run()[:, :3].double().cpu().numpy()
    x = pos.astype(np.float64)
    d = x[None] - x[:, None]
    want = ((mass.astype(np.float64) / ((d ** 2).sum(-1) + 1e-4) ** 1.5)[..., None] * d).sum(1)
    assert np.percentile(workloads.relative_errors(got, want), 99) <= 1e-5
    w, gx, gm = (torch.ones(leaves, c, device="cuda") for c in (3, 3, 1))
    if deep:
        with pytest.raises(ValueError, match="levels"):
            ps.vjp(w, gx, gm)
    else:
        ps.vjp(w, gx, gm)


@pytest.mark.parametrize("leaves", [120, 256, 300, 700])
def test_leaf_ancestor_schedule_of_a_chain_holds_every_leaf(leaves):
    topo = _chain(leaves, far=True)
    dt = engine.DeviceTopology(topo, "cuda")
    units, anc = (a.cpu().numpy() for a in engine.l2l_leaf_schedule_device(dt, (0, leaves)))
    want_units, want_anc = engine.l2l_leaf_schedule(topo, (0, leaves))
    rows = lambda u, a: {int(x[0]): tuple(a[x[1]:x[2]]) for x in u}
    assert len(units) == len(want_units) and rows(units, anc) == rows(want_units, want_anc)
    assert dt.l2l_first_level == 1
