"""The momentum sweeps where their scratch cannot be had, and their three
components together on lines of 2 and 4 rows per thread and on longer ones:
bit for bit the component-by-component and the unconstrained result."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from feicar_b200 import fg, synth

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(np.asfortranarray(a).transpose(*range(a.ndim)[::-1]))).cuda()


def _open_case(cells):
    """A case without a body: every cell fluid."""
    grid = synth.small_grid(*cells, tuple(0.1 * n for n in cells))
    c = fg.Case(grid, fg.default_config())
    z = np.zeros(grid.shape, np.int8, order="F")
    none = np.zeros((0, 3), np.int32)
    rows = dict(ijk=none, cell=none, coefN=np.zeros((0, 8)), probe=np.zeros(0), ip=np.zeros((0, 3)))
    c.set_geometry(z, z, z, rows, rows)
    c.mg_prepare()
    return c, grid


def without_scratch():
    """Run in a process of its own: nothing of the library's block cache."""
    c, grid = _open_case((200, 300, 250))  # three fields of pivots: 366 MB
    rng = np.random.default_rng(1)
    var, r, fu, fv, fw = (_dev(rng.standard_normal(grid.shape)) for _ in range(5))
    prm = fg.AdParams(dt=0.02, reinv=0.01, omega_ad=1.1, crank_nicolson=1)
    # one small pass first, so that the kernels are loaded
    s, sgrid = _open_case((4, 4, 2060))
    t = [_dev(rng.standard_normal(sgrid.shape)) for _ in range(5)]
    torch.cuda.synchronize()
    fg.itsolv_ad_device(s, *[x.data_ptr() for x in t], prm)
    s.close()
    got = var.clone()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - (200 << 20), dtype=torch.uint8, device="cuda")
    n0 = fg.launch_count()
    fg.itsolv_ad_device(c, got.data_ptr(), *[x.data_ptr() for x in (r, fu, fv, fw)], prm)
    slow = fg.launch_count() - n0
    del held
    torch.cuda.empty_cache()
    n0 = fg.launch_count()
    fg.itsolv_ad_device(c, var.data_ptr(), *[x.data_ptr() for x in (r, fu, fv, fw)], prm)
    assert fg.launch_count() - n0 == 2 and slow > 1000  # a launch per anti-diagonal
    assert torch.equal(got, var)
    print("same")


def test_without_scratch():
    here = os.path.dirname(os.path.abspath(__file__))
    code = f"import sys; sys.path.insert(0, {here!r}); import conftest, test_momentum_scratch_gpu as t; t.without_scratch()"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("cells", [(600, 9, 10), (9, 600, 10), (1100, 9, 8), (8, 9, 1100), (8, 2060, 9)])
def test_three_components_on_long_lines(cells):
    grid = synth.small_grid(*cells, tuple(0.1 * n for n in cells))
    c = fg.Case(grid, fg.default_config())
    c.add_body(synth.sphere_body(tuple(0.05 * n for n in cells), 0.45, 3))
    c.set_iblank_body_fast()
    c.gcm_set_internal_boundary()
    c.mg_prepare()
    assert c.nGhost > 0
    rng = np.random.default_rng(2)
    NX, NY, NZ = grid.shape
    va, rhs, fa = ([_dev(rng.standard_normal(grid.shape)) for _ in range(3)] for _ in range(3))
    ba = [torch.zeros(sh, dtype=torch.float64, device="cuda")
          for sh in [(NZ, NY, 2)] * 3 + [(NZ, 2, NX)] * 3 + [(2, NY, NX)] * 3]
    v1, f1, b1 = ([t.clone() for t in ts] for ts in (va, fa, ba))
    vb = fg.VelocityBC()
    for f, ty in enumerate((1, 2, 4, 4, 4, 4)):
        vb.type[f] = ty
    prm = fg.AdParams(dt=0.02, reinv=0.01, omega_ad=1.0, crank_nicolson=1)
    ubi = [torch.zeros(max(1, 3 * n), dtype=torch.float64, device="cuda") for n in (c.nGhost, c.nDead)]
    ug, ud = (t.data_ptr() for t in ubi)
    P = lambda ts: [t.data_ptr() for t in ts]
    it, res, loc = fg.solve_ad_device(c, *P(va), *P(rhs), *P(fa), P(ba), ug, ud, prm, vb, itermax_ad=1, restol_ad=0.0)
    assert it == 1
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
    assert (res, loc) == each[max(range(3), key=lambda a: each[a][0])]
    c.close()
