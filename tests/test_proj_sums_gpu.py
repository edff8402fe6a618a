"""rhs_poisson and the mass correction where their sums change place: partials
summed by the caller's thread (up to 1024 of them) and by a reduction of one
and of several blocks, thin grids whose faces differ in size.  Against the
oracle: the divergence to 1e-12 and the faces to 1e-13 of the largest value
(the device contracts multiply-adds), the sums to 1e-11; the boundary layers
of a divergence full of other values come back zero."""
import numpy as np
import pytest
import torch

from feicar_b200 import fg, synth
import oracle as O

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a.transpose(*range(a.ndim)[::-1]))).cuda()


def _host(t):
    return t.cpu().numpy().transpose(*range(t.ndim)[::-1])


def _close(got, want, tol):
    return float(np.abs(got - want).max()) <= tol * max(1e-300, float(np.abs(want).max()))


@pytest.mark.parametrize("cells", [(2, 2, 2), (5, 90, 4), (64, 64, 64), (64, 68, 64), (70, 6, 300)])
@pytest.mark.parametrize("vzg", [[0] * 6, [0, 1, 0, 0, 0, 0], [1] * 6])
def test_divergence_and_mass(cells, vzg):
    grid = synth.small_grid(*cells, tuple(0.125 * n for n in cells))
    oc = O.OracleCase(grid)
    c = fg.Case(grid, fg.default_config())
    z = np.zeros(grid.shape, np.int8, order="F")
    none = np.zeros((0, 3), np.int32)
    rows = dict(ijk=none, cell=none, coefN=np.zeros((0, 8)), probe=np.zeros(0), ip=np.zeros((0, 3)))
    c.set_geometry(z, z, z, rows, rows)
    c.mg_prepare()
    rng = np.random.default_rng(5)
    sh, dt = grid.shape, 0.02
    f = [np.asfortranarray(rng.standard_normal(sh)) for _ in range(3)]
    bc = [np.asfortranarray(rng.standard_normal(q)) for q in ((2, sh[1], sh[2]), (sh[0], 2, sh[2]), (sh[0], sh[1], 2))]
    P = lambda ts: [t.data_ptr() for t in ts]
    d_f, d_bc = [_dev(a) for a in f], [_dev(a) for a in bc]
    m_f, m_bc = [t.clone() for t in d_f], [t.clone() for t in d_bc]
    d_div = torch.full_like(d_f[0], 7.0)
    div, so, ro = oc.rhs_poisson(*f, *bc, vzg, dt)
    sd, rd = fg.rhs_poisson_device(c, *P(d_f), *P(d_bc), vzg, dt, d_div.data_ptr())
    assert _close(_host(d_div), div, 1e-12)
    assert abs(sd - so) <= 1e-11 * max(1.0, abs(so)) and abs(rd - ro) <= 1e-12 * ro
    if any(vzg):
        fg.enforce_global_mass_consv_device(c, *P(m_f), *P(m_bc), vzg)
    for a, t, q in zip(f + bc, d_f + d_bc, m_f + m_bc):
        assert _close(_host(t), a, 1e-13) and _close(_host(q), a, 1e-13)
    c.close()
