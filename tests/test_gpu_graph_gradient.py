"""A captured step and gradients on one state: a replay rewrites the pass's
particles and coefficients without the host, and whatever reads them afterwards
must see the replay's, not an earlier gradient's.  The reference is a pass of its
own on the same topology, which runs the same kernels: equal bits."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from jaccpot_b200 import FastMultipoleMethod, engine, tree, workloads  # noqa: E402


def _particles(kind, n):
    pos, mass = (torch.from_numpy(a).cuda() for a in workloads.GENERATORS[kind](n, 3))
    return pos, mass, pos + 1e-2 * torch.randn(n, 3, device="cuda", generator=torch.Generator("cuda").manual_seed(1))


@pytest.mark.parametrize("kind,n,p", [("clustered", 20_000, 4), ("plummer", 3_001, 9)])
def test_evaluation_after_a_gradient_and_a_replay(kind, n, p):
    pos, mass, moved = _particles(kind, n)
    kw = dict(theta=0.6, softening=1e-3)
    f_g = FastMultipoleMethod(**kw, advanced={"cuda_graph": True})
    f_e = FastMultipoleMethod(**kw)
    st = f_g.prepare_state(pos, mass, leaf_size=32, max_order=p)
    want = f_e.prepare_state(pos, mass, leaf_size=32, max_order=p)
    f_g.differentiable_accelerations(st, pos, mass)  # captures
    x = pos.clone().requires_grad_()
    f_g.differentiable_accelerations(st, x, mass).square().sum().backward()
    acc = f_g.differentiable_accelerations(st, moved, mass)  # replays
    assert torch.equal(acc, f_e.differentiable_accelerations(want, moved, mass))
    targets = torch.arange(0, n, 7, device="cuda")
    assert torch.equal(f_g.evaluate_prepared_state(st, as_numpy=False), acc)
    assert torch.equal(f_g.evaluate_prepared_state(st, target_indices=targets),
                       f_e.evaluate_prepared_state(want, target_indices=targets))
    # and the next gradient is the moved particles'
    g = []
    for f, s in ((f_g, st), (f_e, want)):
        x = moved.clone().requires_grad_()
        f.differentiable_accelerations(s, x, mass).square().sum().backward()
        g.append(x.grad)
    assert torch.equal(*g)


def test_vjp_after_a_replay_does_not_reuse_an_earlier_pass():
    pos, mass, moved = _particles("plummer", 20_000)
    n = pos.shape[0]
    topo = tree.build_topology(pos, mass, leaf_size=16, theta=0.6, device="cuda")
    w = torch.randn(n, 3, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    ps, ref = (engine.Pass(engine.DeviceTopology(topo, "cuda"), 5, G=1.0, eps2=1e-6) for _ in range(2))
    buf, acc = pos.clone(), torch.empty_like(pos)
    graph = ps.capture(buf, mass, acc)
    out = [torch.empty(n, c, device="cuda") for c in (3, 1, 3, 1)]
    ps.vjp(w, out[0], out[1])  # at `pos`
    buf.copy_(moved)
    graph.replay()
    ps.vjp(w, out[0], out[1], recompute=False)
    ref.load_particles(moved, mass)
    ref.vjp(w, out[2], out[3])
    assert torch.equal(out[0], out[2]) and torch.equal(out[1], out[3])


def test_gradient_leaves_complete_locals_for_later_evaluations():
    pos, mass, moved = _particles("uniform", 10_000)
    topo = tree.build_topology(pos, mass, leaf_size=16, theta=0.6, device="cuda")
    ps, ref = (engine.Pass(engine.DeviceTopology(topo, "cuda"), 6, G=1.0, eps2=1e-6) for _ in range(2))
    rows = torch.empty((topo.num_leaves, ps.ws.stride), device="cuda")
    for q, own in ((ps, rows), (ref, None)):
        q.load_particles(moved, mass)
        q.run(own_rows=own)
    assert torch.equal(ps.ws.locals, ref.ws.locals) and not torch.equal(rows, ps.ws.locals[topo.num_internal:])
    assert torch.equal(ps.evaluate().clone(), ref.evaluate())
    out = [torch.empty(10_000, c, device="cuda") for c in (3, 1, 3, 1)]
    w = torch.randn(10_000, 3, device="cuda")
    ps.vjp(w, out[0], out[1], recompute=False, own_rows=rows)
    ref.vjp(w, out[2], out[3])
    assert torch.equal(out[0], out[2]) and torch.equal(out[1], out[3])
    with pytest.raises(ValueError, match="own_rows"):
        ps.downward(own_rows=rows[1:])
    with pytest.raises(ValueError, match="level-by-level"):
        ps.downward(own_rows=rows, cascade=True)
