"""Restriction and prolongation of levels above the one-kernel cycle: cell
counts around the four cells of a thread, its two rows and two planes, and
the 128 cells of a warp; axes that are halved on every level and axes that
are not (whose levels take the residual and the restriction as two
launches); batches that hold both.  Each solve must reach the exact discrete
solution of its manufactured right-hand side to 1e-9 at rtol 1e-12; where
every axis is halved, in no more cycles than a tenfold reduction per cycle
with one restart's slack allows: rows left out of a transfer would not.
"""
import numpy as np
import pytest
import torch

from feicar_b200 import fg, synth

pytestmark = pytest.mark.gpu


def _problem(cells, seed, prec, mgrids=None):
    h = 1.0 / min(cells)
    grid = synth.Grid(*[synth.uniform_nodes(n, 0, n * h) for n in cells])
    kw = dict(mgrids=mgrids) if mgrids else {}
    c = fg.Case(grid, fg.default_config(precision=prec, rtol=1e-12, max_cycles=60, **kw))
    z = np.zeros(grid.shape, np.int8, order="F")
    none = np.zeros((0, 3), np.int32)
    rows = dict(ijk=none, cell=none, coefN=np.zeros((0, 8)), probe=np.zeros(0), ip=np.zeros((0, 3)))
    c.set_geometry(z, z, z, rows, rows)
    c.mg_prepare()
    rng = np.random.default_rng(seed)
    phi = synth.fortran_zeros(grid)
    phi[1:grid.nx, 1:grid.ny, 1:grid.nz] = synth.box_smooth(rng.standard_normal(cells), 2)
    synth.neumann_fill(grid, phi)
    return c, grid, synth.laplacian(grid, phi), phi


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a.transpose(2, 1, 0))).cuda()


def _error(grid, t, phi):
    I = (slice(1, grid.nx), slice(1, grid.ny), slice(1, grid.nz))
    a, b = t.cpu().numpy().transpose(2, 1, 0)[I], phi[I]
    a, b = a - a.mean(), b - b.mean()
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("prec", [fg.FG_PREC_MIXED, fg.FG_PREC_FP64])
@pytest.mark.parametrize("mgrids", [None, (0, 0, 1), (0, 2, 0)])
@pytest.mark.parametrize("cells", [(64, 64, 64), (129, 34, 17), (130, 33, 18), (131, 35, 19), (258, 17, 20),
                                   (37, 41, 43)])
def test_transfers(cells, mgrids, prec):
    c, grid, rhs, phi = _problem(cells, 8, prec, mgrids)
    d_f, d_p = _dev(rhs), _dev(np.zeros_like(phi))
    torch.cuda.synchronize()
    st = c.solve_poisson_device(d_p.data_ptr(), d_f.data_ptr())
    assert st["relres"] <= 1e-12 and _error(grid, d_p, phi) <= 1e-9
    if mgrids is None:
        assert st["cycles"] <= 12 + 8
    c.close()


def test_batch_of_both_transfers():
    probs = [_problem((66, 34, 30), 9, fg.FG_PREC_MIXED), _problem((40, 41, 42), 10, fg.FG_PREC_MIXED, (0, 0, 1)),
             _problem((129, 35, 18), 11, fg.FG_PREC_MIXED)]
    bt = fg.Batch(fg.default_config(precision=fg.FG_PREC_MIXED, rtol=1e-12, max_cycles=60))
    for c, *_ in probs:
        bt.add(c)
    fs, ps = [_dev(q[2]) for q in probs], [_dev(np.zeros_like(q[3])) for q in probs]
    torch.cuda.synchronize()
    bt.solve_device([p.data_ptr() for p in ps], [f.data_ptr() for f in fs])
    for (c, grid, rhs, phi), p in zip(probs, ps):
        assert _error(grid, p, phi) <= 1e-9
    bt.close()
    for c, *_ in probs:
        c.close()
