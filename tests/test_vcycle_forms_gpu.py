"""One V-cycle in each of the forms its levels can take, against the others:
levels in one kernel on a cluster of blocks, on one block (batches of more
than 16 problems) and as one launch per stage (line families chosen by
hand); residual and restriction as one launch and as two (a batch with a
problem one of whose axes is not halved).  A solve hides a wrong row or a
skipped line behind its outer iteration; the field after one cycle does not.

All forms do the same arithmetic up to the order of a few additions, so they
differ by rounding, carried by a cycle whose largest gain is the coarse
inverse's, below (n / 2)^2 for lines of n <= 258 cells: 2e4 x 1e-16 (FP64) and
2e4 x 6e-8 (FP32) of the field at worst, and a few hundred times less in
practice, as rounding has no smooth part to speak of.  Tolerances: 1e-11 and
1e-3 of the largest value; a row left out changes its cells by a tenth and
more of it.
"""
import numpy as np
import pytest
import torch

from feicar_b200 import fg, synth

pytestmark = pytest.mark.gpu

TOL = {fg.FG_PREC_FP64: 1e-11, fg.FG_PREC_MIXED: 1e-3}
LAUNCHES = {"x": 1, "y": 2, "z": 2}


def _config(prec, outlet=False, **kw):
    pbc = [fg.FG_PBC_NEUMANN] * 6
    if outlet:
        pbc[1] = fg.FG_PBC_DIRICHLET
        pbc[2] = fg.FG_PBC_DIRICHLET
    return fg.default_config(precision=prec, outer=fg.FG_OUTER_RICHARDSON, rtol=1e-30, max_cycles=1, pbc=pbc, **kw)


def _case(cells, prec, body=None, outlet=False, seed=0, **kw):
    """A case with its fields: right-hand side and start value on the device."""
    h = 1.0 / min(cells)
    grid = synth.Grid(*[synth.uniform_nodes(n, 0, n * h) for n in cells])
    c = fg.Case(grid, _config(prec, outlet, **kw))
    if body:
        at = tuple(f * n * h for f, n in zip((0.45, 0.55, 0.5), cells))
        c.add_body(synth.sphere_body(at, body, 3))
        c.set_iblank_body_fast()
        c.gcm_set_internal_boundary()
        assert c.nGhost > 0
    else:
        z = np.zeros(grid.shape, np.int8, order="F")
        none = np.zeros((0, 3), np.int32)
        rows = dict(ijk=none, cell=none, coefN=np.zeros((0, 8)), probe=np.zeros(0), ip=np.zeros((0, 3)))
        c.set_geometry(z, z, z, rows, rows)
    c.mg_prepare()
    rng = np.random.default_rng(seed)
    f, p = (torch.from_numpy(rng.standard_normal(grid.shape[::-1])).cuda() for _ in range(2))
    torch.cuda.synchronize()
    return c, f, p


def _cycle(c, f, p0):
    p = p0.clone()
    torch.cuda.synchronize()
    st = c.solve_poisson_device(p.data_ptr(), f.data_ptr(), allow_not_converged=True)
    assert st["cycles"] == 1
    return p


def _batch_cycle(prec, probs):
    bt = fg.Batch(_config(prec))
    for c, *_ in probs:
        bt.add(c)
    ps = [p.clone() for _, _, p in probs]
    torch.cuda.synchronize()
    bt.solve_device([p.data_ptr() for p in ps], [f.data_ptr() for _, f, _ in probs], allow_not_converged=True)
    bt.close()
    return ps


def _same(a, b, prec):
    assert torch.isfinite(a).all() and torch.isfinite(b).all()
    assert float((a - b).abs().max() / b.abs().max()) <= TOL[prec]


@pytest.mark.parametrize("prec", [fg.FG_PREC_FP64, fg.FG_PREC_MIXED])
@pytest.mark.parametrize("body,outlet", [(None, False), (0.5, False), (0.5, True)])
@pytest.mark.parametrize("cells", [(8, 8, 8), (9, 13, 10), (34, 17, 21), (32, 32, 32), (21, 128, 12), (47, 45, 43),
                                   (16, 18, 200)])
def test_cluster_and_launches(cells, body, outlet, prec):
    c, f, p0 = _case(cells, prec, body, outlet)
    one = _cycle(c, f, p0)
    fg.case_set_tuning(c, LAUNCHES)
    _same(one, _cycle(c, f, p0), prec)
    c.close()


@pytest.mark.parametrize("prec", [fg.FG_PREC_FP64, fg.FG_PREC_MIXED])
@pytest.mark.parametrize("cells", [(63, 150, 16), (64, 150, 16), (64, 150, 17), (130, 2, 150), (200, 16, 140),
                                   (65, 5, 200)])
def test_families_of_short_lines(cells, prec):
    """The default families of y/z lines around 16 rows and x lines around 64
    cells against one family for all."""
    c, f, p0 = _case(cells, prec)
    one = _cycle(c, f, p0)
    for fams in (LAUNCHES, {"x": 1, "y": 1, "z": 1}):
        fg.case_set_tuning(c, fams)
        _same(one, _cycle(c, f, p0), prec)
    c.close()


@pytest.mark.parametrize("nu", [(1, 1), (1, 0), (3, 2)])
def test_smoothing_steps(nu):
    c, f, p0 = _case((33, 20, 27), fg.FG_PREC_FP64, 0.5, nu1=nu[0], nu2=nu[1])
    one = _cycle(c, f, p0)
    fg.case_set_tuning(c, LAUNCHES)
    _same(one, _cycle(c, f, p0), fg.FG_PREC_FP64)
    c.close()


def test_many_rows_at_level_0():
    """More ghost rows than two per thread of the cluster: their values go
    through memory, and the launches take them in two passes."""
    cells, prec = (32, 30, 31), fg.FG_PREC_FP64
    grid = synth.Grid(*[synth.uniform_nodes(n, 0, 0.1 * n) for n in cells])
    c = fg.Case(grid, _config(prec))
    rng = np.random.default_rng(4)
    z = np.zeros(grid.shape, np.int8, order="F")
    gh = z.copy(order="F")
    I = tuple(slice(1, n + 1) for n in cells)
    gh[I] = rng.random(cells) < 0.65
    ijk = np.argwhere(gh).astype(np.int32)
    assert len(ijk) > 2 * 8192
    w = rng.random((len(ijk), 8))
    rows = dict(ijk=ijk, cell=np.minimum(ijk, np.array(cells) - 1), coefN=0.8 * w / w.sum(axis=1, keepdims=True),
                probe=np.zeros(len(ijk)), ip=np.zeros((len(ijk), 3)))
    none = dict(ijk=ijk[:0], cell=ijk[:0], coefN=w[:0], probe=np.zeros(0), ip=np.zeros((0, 3)))
    c.set_geometry(z, gh, z, rows, none)
    c.mg_prepare()
    f, p0 = (torch.from_numpy(rng.standard_normal(grid.shape[::-1])).cuda() for _ in range(2))
    one = _cycle(c, f, p0)
    fg.case_set_tuning(c, LAUNCHES)
    _same(one, _cycle(c, f, p0), prec)
    c.close()


@pytest.mark.parametrize("prec", [fg.FG_PREC_FP64, fg.FG_PREC_MIXED])
def test_one_block_per_problem(prec):
    sizes = [(8, 8, 8), (12, 9, 10), (20, 24, 18), (33, 17, 21), (40, 40, 40), (48, 30, 52), (66, 34, 30)]
    probs = [_case(sizes[q % len(sizes)], prec, 0.5 if q % 3 else None, seed=q) for q in range(18)]
    together = _batch_cycle(prec, probs)
    for (c, f, p0), p in zip(probs, together):
        _same(p, _batch_cycle(prec, [(c, f, p0)])[0], prec)
        c.close()


@pytest.mark.parametrize("prec", [fg.FG_PREC_FP64, fg.FG_PREC_MIXED])
@pytest.mark.parametrize("cells", [(64, 64, 64), (129, 34, 17), (130, 33, 18), (131, 35, 19), (258, 17, 20)])
def test_one_and_two_pass_restriction(cells, prec):
    both = [_case(cells, prec, 0.5, seed=1), _case((66, 70, 40), prec, 0.5, seed=2)]
    other = _case((40, 41, 42), prec, mgrids=(0, 0, 1), seed=3)  # its z axis is not halved
    fused, two = _batch_cycle(prec, both), _batch_cycle(prec, both + [other])
    for (c, f, p0), a, b in zip(both, fused, two):
        alone = _batch_cycle(prec, [(c, f, p0)])[0]
        _same(a, alone, prec)
        _same(b, alone, prec)
        c.close()
    other[0].close()


def test_large_levels_beside_a_large_coarsest_system():
    """One problem's levels and another's coarsest system fit a block's shared
    memory each with its own problem's other part, not with one another's.
    The batch's solve reaches the exact discrete solutions of manufactured
    right-hand sides to 1e-9 at rtol 1e-12."""
    bt = fg.Batch(fg.default_config(precision=fg.FG_PREC_FP64, rtol=1e-12, max_cycles=60))
    probs = []
    for q in range(17):
        cells, kw = ((36, 44, 46), {}) if q < 16 else ((30, 30, 32), dict(mgrids=(2, 2, 2)))  # coarsest 15 x 15 x 16
        h = 1.0 / min(cells)
        grid = synth.Grid(*[synth.uniform_nodes(n, 0, n * h) for n in cells])
        c = fg.Case(grid, fg.default_config(precision=fg.FG_PREC_FP64, rtol=1e-12, max_cycles=60, **kw))
        z = np.zeros(grid.shape, np.int8, order="F")
        none = np.zeros((0, 3), np.int32)
        rows = dict(ijk=none, cell=none, coefN=np.zeros((0, 8)), probe=np.zeros(0), ip=np.zeros((0, 3)))
        c.set_geometry(z, z, z, rows, rows)
        c.mg_prepare()
        bt.add(c)
        phi = synth.fortran_zeros(grid)
        phi[1:grid.nx, 1:grid.ny, 1:grid.nz] = synth.box_smooth(np.random.default_rng(q).standard_normal(cells), 2)
        synth.neumann_fill(grid, phi)
        f = torch.from_numpy(np.ascontiguousarray(synth.laplacian(grid, phi).transpose(2, 1, 0))).cuda()
        probs.append((c, grid, phi, f, torch.zeros_like(f)))
    torch.cuda.synchronize()
    st = bt.solve_device([q[4].data_ptr() for q in probs], [q[3].data_ptr() for q in probs])
    assert st["relres"] <= 1e-12
    bt.close()
    for c, grid, phi, f, p in probs:
        I = (slice(1, grid.nx), slice(1, grid.ny), slice(1, grid.nz))
        a, b = p.cpu().numpy().transpose(2, 1, 0)[I], phi[I]
        a, b = a - a.mean(), b - b.mean()
        assert np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(b)
        c.close()
