"""The velocity correction and the pressure update where a thread walks
several planes: one, two and three planes left over from the four it loads
ahead, columns of four and of eight planes; velocities alone, gradients
alone and both.  Against the oracle: the correction to 1e-13 of the largest
value (the device contracts multiply-adds), the update bit for bit."""
import numpy as np
import pytest
import torch

from feicar_b200 import fg, synth
import oracle as O

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a.transpose(2, 1, 0))).cuda()


def _host(t):
    return t.cpu().numpy().transpose(2, 1, 0)


@pytest.mark.parametrize("cells", [(129, 100, 65), (131, 101, 66), (129, 103, 67), (257, 131, 23)])
def test_planes(cells):
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
    rng = np.random.default_rng(9)
    vel = [np.asfortranarray(rng.standard_normal(grid.shape)) for _ in range(3)]
    pp = np.asfortranarray(rng.standard_normal(grid.shape))
    want = [a.copy(order="F") for a in vel]
    grad = oc.correct_vel(pp, 0.02, *want)
    d_pp = _dev(pp)
    for with_vel, with_grad in ((True, True), (True, False), (False, True)):
        dv, dg = [_dev(a) for a in vel], [torch.zeros_like(d_pp) for _ in range(3)]
        fg.correct_vel_device(c, d_pp.data_ptr(), 0.02, *[t.data_ptr() if with_vel else None for t in dv],
                              *[t.data_ptr() if with_grad else None for t in dg])
        pairs = list(zip(want if with_vel else vel, dv))
        pairs += list(zip(grad if with_grad else [np.zeros(grid.shape)] * 3, dg))
        for a, t in pairs:
            assert np.abs(_host(t) - a).max() <= 1e-13 * np.abs(a).max()
    po = pp.copy(order="F")
    p_o = oc.update_pressure(po)
    for d_p in (torch.full_like(d_pp, 3.0), None):
        q = _dev(pp)
        fg.update_pressure_device(c, q.data_ptr(), d_p.data_ptr() if d_p is not None else None)
        assert np.array_equal(_host(q), po)
        assert d_p is None or np.array_equal(_host(d_p), p_o)
    c.close()
