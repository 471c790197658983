"""Target subsets against the whole evaluation: leaves from one particle to
the largest, neighbour lists around the 32 leaves a warp looks up at once,
target counts around the kernels' blocks, repeated targets.

Tolerance: both sides sum the same terms in FP32, each through fewer than 200
roundings of partial sums that are at most S_i = sum_j m_j / r_ij^2 (the far
field's terms are smaller), so |difference| <= 2 * 200 * 2^-24 * S_i."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from jaccpot_b200 import FastMultipoleMethod, workloads  # noqa: E402

EPS = 1e-2
TOL = 2 * 200 * 2.0 ** -24


@pytest.mark.parametrize("kind,n,leaf,p,nt", [
    ("uniform", 1, 16, 2, 1), ("uniform", 33, 64, 4, 33), ("uniform", 700, 1, 3, 129), ("plummer", 2500, 16, 10, 2500),
    ("plummer", 3000, 64, 6, 127), ("clustered", 2777, 33, 8, 8), ("plummer", 3000, 5, 1, 128)])
def test_subset_equals_the_whole_evaluation(kind, n, leaf, p, nt):
    pos, mass = workloads.GENERATORS[kind](n, 11)
    fmm = FastMultipoleMethod(theta=0.6, softening=EPS)
    st = fmm.prepare_state(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda(), leaf_size=leaf, max_order=p)
    acc, pot = (t.double() for t in fmm.evaluate_prepared_state(st, return_potential=True, as_numpy=False))
    x, m = torch.from_numpy(pos).cuda().double(), torch.from_numpy(mass).cuda().double()
    r2 = torch.cdist(x, x) ** 2 + EPS ** 2
    r2.fill_diagonal_(np.inf)
    size, psize = (m / r2).sum(1), (m / r2.sqrt()).sum(1)
    rng = np.random.default_rng(3)
    tg = torch.from_numpy(rng.integers(0, n, nt)).cuda()  # with repeats
    sub, spot = fmm.evaluate_prepared_state(st, target_indices=tg, return_potential=True)
    assert sub.shape == (nt, 3) and spot.shape == (nt,)
    assert bool(((sub.double() - acc[tg]).abs().amax(1) <= TOL * size[tg]).all())
    assert bool(((spot.double() - pot[tg]).abs() <= TOL * psize[tg]).all())


@pytest.mark.parametrize("bad", [-1, 500, 1 << 40])
def test_out_of_range_is_refused_and_the_next_call_works(bad):
    pos, mass = workloads.uniform_cube(500, 2)
    fmm = FastMultipoleMethod(softening=EPS)
    st = fmm.prepare_state(pos, mass, leaf_size=16, max_order=4)
    tg = torch.arange(300, device="cuda")
    want = fmm.evaluate_prepared_state(st, target_indices=tg)
    with pytest.raises(IndexError):
        fmm.evaluate_prepared_state(st, target_indices=torch.cat([tg, torch.tensor([bad], device="cuda")]))
    assert torch.equal(fmm.evaluate_prepared_state(st, target_indices=tg), want)
