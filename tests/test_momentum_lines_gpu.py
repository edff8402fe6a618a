"""The momentum line sweeps at the sizes where their kernels change form,
bit for bit: lines of 1, 2 and 4 rows per thread and longer ones, the
shortest lines, columns along either transverse direction, more columns
than blocks fit on the device at once, and the three components of a
momentum iteration swept together against one by one."""
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


def _open_case(grid):
    """A case without a body: every cell fluid."""
    c = fg.Case(grid, fg.default_config())
    z = np.zeros(grid.shape, np.int8, order="F")
    none = np.zeros((0, 3), np.int32)
    rows = dict(ijk=none, cell=none, coefN=np.zeros((0, 8)), probe=np.zeros(0), ip=np.zeros((0, 3)))
    c.set_geometry(z, z, z, rows, rows)
    c.mg_prepare()
    return c


@pytest.mark.parametrize("cells", [(2, 2, 2), (9, 2, 5), (33, 7, 18), (18, 31, 8), (511, 4, 5), (512, 5, 4),
                                   (1030, 4, 3), (3, 520, 4), (4, 3, 1100), (2060, 3, 3), (4, 4, 3300)])
@pytest.mark.parametrize("cn", [1, 0])
def test_itsolv_ad_line_lengths(cells, cn):
    grid = synth.small_grid(*cells, tuple(0.1 * n for n in cells))
    oc = O.OracleCase(grid)
    c = _open_case(grid)
    dt, reinv = 0.02, 0.01
    ad = oc.set_solve_ad(dt, reinv)
    half_dt = 0.5 * dt if cn else 0.0
    rng = np.random.default_rng(11)
    fu, fv, fw, r, var = (np.asfortranarray(rng.standard_normal(grid.shape)) for _ in range(5))
    d = [_dev(a) for a in (var, r, fu, fv, fw)]
    ptr = [t.data_ptr() for t in d]
    prm = fg.AdParams(dt=dt, reinv=reinv, omega_ad=1.2, crank_nicolson=cn)
    for it in range(2):
        oc.itsolv_ad(ad, var, r, fu, fv, fw, half_dt, 1.2)
        fg.itsolv_ad_device(c, *ptr, prm)
        assert np.array_equal(_host(d[0]), var), it
        assert fg.calc_residual_ad_device(c, *ptr, prm) == oc.calc_residual_ad(ad, var, r, fu, fv, fw, half_dt)
    c.close()


def test_solve_ad_components_together_and_one_by_one():
    grid = synth.small_grid(40, 22, 18, (4.0, 2.2, 1.8))
    c = fg.Case(grid, fg.default_config())
    c.add_body(synth.sphere_body((1.3, 1.1, 0.9), 0.7, 3))
    c.set_iblank_body_fast()
    c.gcm_set_internal_boundary()
    c.mg_prepare()
    rng = np.random.default_rng(3)
    NX, NY, NZ = grid.shape
    vel0 = [_dev(0.1 * rng.standard_normal(grid.shape)) for _ in range(3)]
    vel0[0] += 1.0
    rhs = [v.clone() for v in vel0]
    bc0 = [torch.zeros(sh, dtype=torch.float64, device="cuda")
           for sh in [(NZ, NY, 2)] * 3 + [(NZ, 2, NX)] * 3 + [(2, NY, NX)] * 3]
    vb = fg.VelocityBC()
    for f, ty in enumerate((1, 2, 4, 4, 4, 4)):
        vb.type[f] = ty
    vb.val[0][0] = 1.0
    prm = fg.AdParams(dt=0.02, reinv=0.01, omega_ad=1.0, crank_nicolson=1)
    ubi = [torch.zeros(max(1, 3 * n), dtype=torch.float64, device="cuda") for n in (c.nGhost, c.nDead)]
    ug, ud = (t.data_ptr() for t in ubi)
    P = lambda ts: [t.data_ptr() for t in ts]

    def state():
        vel, bc = [t.clone() for t in vel0], [t.clone() for t in bc0]
        faces = [torch.zeros_like(vel0[0]) for _ in range(3)]
        fg.set_outer_velocity_bc_device(c, *P(vel), P(bc), vb)
        fg.set_outer_ghost_velocity_device(c, *P(vel), P(bc))
        fg.face_vel_device(c, *P(vel), *P([bc[0], bc[4], bc[8]]), *P(faces))
        torch.cuda.synchronize()
        return vel, bc, faces

    va, ba, fa = state()
    it, res, loc = fg.solve_ad_device(c, *P(va), *P(rhs), *P(fa), P(ba), ug, ud, prm, vb, itermax_ad=2, restol_ad=0.0)
    assert it == 2
    v1, b1, f1 = state()
    for _ in range(2):
        for a in range(3):
            fg.itsolv_ad_device(c, *P([v1[a], rhs[a], *f1]), prm)
        fg.ghostcell_velocity_device(c, *P(v1), ug, ud)
        fg.face_vel_device(c, *P(v1), *P([b1[0], b1[4], b1[8]]), *P(f1))
        fg.enforce_global_mass_consv_device(c, *P(f1), *P([b1[0], b1[4], b1[8]]), [0, 1, 0, 0, 0, 0])
        fg.set_outer_velocity_bc_device(c, *P(v1), P(b1), vb)
        fg.set_outer_ghost_velocity_device(c, *P(v1), P(b1))
        each = [fg.calc_residual_ad_device(c, *P([v1[a], rhs[a], *f1]), prm) for a in range(3)]
    for x, y in zip(va + ba + fa, v1 + b1 + f1):
        assert torch.equal(x, y)
    best = max(range(3), key=lambda a: each[a][0])
    assert (res, loc) == each[best]
    c.close()
