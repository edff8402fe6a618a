"""The projection steps at the sizes where their kernels change form: grids
smaller and larger than a block of columns, remainders in each direction,
one and several planes per thread, correction faces that share cells, against
the oracle's restatement.  The stencils to 1e-13 of the largest value (the
device contracts multiply-adds), the sums to 1e-11; update_pressure bit for
bit."""
import numpy as np
import pytest
import torch

from feicar_b200 import fg, synth
import oracle as O

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(np.asfortranarray(a).transpose(*range(a.ndim)[::-1]))).cuda()


def _host(t):
    return t.cpu().numpy().transpose(*range(t.ndim)[::-1])


def _close(got, want, tol):
    return float(np.abs(got - want).max()) <= tol * max(1e-300, float(np.abs(want).max()))


@pytest.mark.parametrize("cells", [(24, 16, 16), (65, 17, 18), (63, 33, 20), (130, 19, 67)])
@pytest.mark.parametrize("vzg", [[0] * 6, [0, 1, 0, 0, 0, 0], [1, 1, 1, 0, 0, 1], [1] * 6])
def test_projection_shapes(cells, vzg):
    grid = synth.small_grid(*cells, tuple(0.125 * n for n in cells), stretch=1.2)
    body = synth.sphere_body(tuple(0.0625 * n + 0.01 for n in cells), 0.9, 3)
    oc = O.OracleCase(grid)
    oc.add_body(body)
    oc.set_iblank()
    oc.gcm(2.0, 2.0)
    c = fg.Case(grid, fg.default_config())
    c.add_body(body)
    c.set_iblank_body_fast()
    c.gcm_set_internal_boundary()
    c.mg_prepare()
    rng = np.random.default_rng(5)
    sh = grid.shape
    u, v, w, pp = (np.asfortranarray(rng.standard_normal(sh)) for _ in range(4))
    bc = [np.asfortranarray(rng.standard_normal((2, sh[1], sh[2]))), np.asfortranarray(rng.standard_normal((sh[0], 2, sh[2]))),
          np.asfortranarray(rng.standard_normal((sh[0], sh[1], 2)))]
    dt = 0.02
    P = lambda ts: [t.data_ptr() for t in ts]
    d_vel, d_bc, d_pp = [_dev(a) for a in (u, v, w)], [_dev(a) for a in bc], _dev(pp)
    d_f = [torch.zeros_like(d_pp) for _ in range(3)]
    d_div = torch.full_like(d_pp, 7.0)
    fo = oc.face_vel(u, v, w, *bc)
    fg.face_vel_device(c, *P(d_vel), *P(d_bc), *P(d_f))
    for a, t in zip(fo, d_f):
        assert _close(_host(t), a, 1e-13)
    div, so, ro = oc.rhs_poisson(*fo, *bc, vzg, dt)
    sd, rd = fg.rhs_poisson_device(c, *P(d_f), *P(d_bc), vzg, dt, d_div.data_ptr())
    assert _close(_host(d_div), div, 1e-12)
    for a, t in zip(list(fo) + bc, d_f + d_bc):
        assert _close(_host(t), a, 1e-13)
    assert abs(sd - so) <= 1e-11 * max(1.0, abs(so)) and abs(rd - ro) <= 1e-12 * ro
    uo, vo, wo = (a.copy(order="F") for a in (u, v, w))
    go = oc.correct_vel(pp, dt, uo, vo, wo)
    d_g = [torch.zeros_like(d_pp) for _ in range(3)]
    fg.correct_vel_device(c, d_pp.data_ptr(), dt, *P(d_vel), *P(d_g))
    for a, t in zip([uo, vo, wo, *go], d_vel + d_g):
        assert _close(_host(t), a, 1e-13)
    po = pp.copy(order="F")
    p_o = oc.update_pressure(po)
    for d_p in (torch.full_like(d_pp, 3.0), None):
        q = _dev(pp)
        fg.update_pressure_device(c, q.data_ptr(), d_p.data_ptr() if d_p is not None else None)
        assert np.array_equal(_host(q), po)
        assert d_p is None or np.array_equal(_host(d_p), p_o)
    c.close()
