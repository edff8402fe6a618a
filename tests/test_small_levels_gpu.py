"""Solves whose hierarchy runs through the one-block cycle of the small
levels at its edges: lines of 1 to 16 lanes and ragged remainders, levels
just inside and outside its shared memory, axes that stop coarsening before
the others, Dirichlet faces on its levels, one and several smoothing steps,
batches of problems whose hierarchies end on different levels.  Each solve
must reach the exact discrete solution of its manufactured right-hand side
to 1e-9 at rtol 1e-12, in no more cycles than a tenfold reduction per cycle
(with one restart's slack) allows: a smoother that skipped lines would not.
"""
import numpy as np
import pytest
import torch

from feicar_b200 import fg, synth

pytestmark = pytest.mark.gpu


def _problem(cells, outlet, seed, prec, nu=(2, 2)):
    h = 1.0 / min(cells)
    grid = synth.Grid(*[synth.uniform_nodes(n, 0, n * h) for n in cells])
    pbc = [fg.FG_PBC_NEUMANN] * 6
    if outlet:
        pbc[1] = fg.FG_PBC_DIRICHLET
        pbc[2] = fg.FG_PBC_DIRICHLET
    c = fg.Case(grid, fg.default_config(precision=prec, rtol=1e-12, max_cycles=60, pbc=pbc, nu1=nu[0], nu2=nu[1]))
    z = np.zeros(grid.shape, np.int8, order="F")
    none = np.zeros((0, 3), np.int32)
    rows = dict(ijk=none, cell=none, coefN=np.zeros((0, 8)), probe=np.zeros(0), ip=np.zeros((0, 3)))
    c.set_geometry(z, z, z, rows, rows)
    c.mg_prepare()
    rng = np.random.default_rng(seed)
    nx, ny, nz = grid.nx, grid.ny, grid.nz
    phi = synth.fortran_zeros(grid)
    phi[1:nx, 1:ny, 1:nz] = synth.box_smooth(rng.standard_normal((nx - 1, ny - 1, nz - 1)), 2)
    synth.neumann_fill(grid, phi)
    if outlet:  # p = 0 on the far x and the near y face
        phi[nx] = -phi[nx - 1]
        phi[:, 0] = -phi[:, 1]
    return c, grid, synth.laplacian(grid, phi), phi


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a.transpose(2, 1, 0))).cuda()


def _error(grid, t, phi, outlet):
    p = t.cpu().numpy().transpose(2, 1, 0)
    I = (slice(1, grid.nx), slice(1, grid.ny), slice(1, grid.nz))
    a, b = p[I], phi[I]
    if not outlet:
        a, b = a - a.mean(), b - b.mean()
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("prec", [fg.FG_PREC_MIXED, fg.FG_PREC_FP64])
@pytest.mark.parametrize("outlet", [False, True])
@pytest.mark.parametrize("cells", [(8, 8, 8), (9, 13, 10), (34, 17, 21), (32, 32, 32), (47, 45, 43), (56, 50, 61),
                                   (130, 18, 20), (16, 18, 200), (264, 16, 12)])
def test_small_levels(cells, outlet, prec):
    c, grid, rhs, phi = _problem(cells, outlet, 5, prec)
    d_f, d_p = _dev(rhs), _dev(np.zeros_like(phi))
    torch.cuda.synchronize()
    st = c.solve_poisson_device(d_p.data_ptr(), d_f.data_ptr())
    assert st["relres"] <= 1e-12 and _error(grid, d_p, phi, outlet) <= 1e-9
    assert st["cycles"] <= 12 + 8
    c.close()


@pytest.mark.parametrize("nu", [(1, 1), (2, 1), (3, 3)])
def test_smoothing_steps(nu):
    c, grid, rhs, phi = _problem((36, 30, 27), False, 6, fg.FG_PREC_MIXED, nu)
    d_f, d_p = _dev(rhs), _dev(np.zeros_like(phi))
    torch.cuda.synchronize()
    st = c.solve_poisson_device(d_p.data_ptr(), d_f.data_ptr())
    assert st["relres"] <= 1e-12 and _error(grid, d_p, phi, False) <= 1e-9
    c.close()


@pytest.mark.parametrize("prec", [fg.FG_PREC_MIXED, fg.FG_PREC_FP64])
def test_batch_of_uneven_hierarchies(prec):
    probs = [_problem(n, False, 7 + i, prec) for i, n in enumerate([(8, 8, 8), (20, 24, 18), (40, 40, 40), (66, 34, 30)])]
    bt = fg.Batch(fg.default_config(precision=prec, rtol=1e-12, max_cycles=60))
    for c, *_ in probs:
        bt.add(c)
    fs, ps = [_dev(q[2]) for q in probs], [_dev(np.zeros_like(q[3])) for q in probs]
    torch.cuda.synchronize()
    st = bt.solve_device([p.data_ptr() for p in ps], [f.data_ptr() for f in fs])
    assert st["cycles"] <= 12 + 8
    for (c, grid, rhs, phi), p in zip(probs, ps):
        assert _error(grid, p, phi, False) <= 1e-9
    bt.close()
    for c, *_ in probs:
        c.close()
