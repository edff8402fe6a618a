"""Several host threads, each with a handle of its own, whose kernels take
very different amounts of shared memory: no call may fail, and each thread's
results are those of the same calls made alone.  The launch limit of a
kernel's shared memory is state of the device, so a small problem's thread
must not lower it under a large one's; one test sends every kernel from the
host, one has graphs captured and patched again as a body moves, one sweeps
momentum lines of two lengths that share a kernel.
"""
import threading

import numpy as np
import pytest
import torch

from feicar_b200 import fg, synth

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a).transpose(2, 1, 0))).cuda()


def _host(t):
    return t.cpu().numpy().transpose(2, 1, 0)


SMALL = 5  # threads with a small problem beside the one with a large problem


def _together(large, small):
    """Runs large() on a thread, small() over and over on theirs meanwhile."""
    gate, over, failed = threading.Barrier(1 + len(small)), threading.Event(), []

    def body(job, again):
        try:
            gate.wait()
            while True:
                job()
                if not again or over.is_set():
                    break
        except Exception as e:  # noqa: BLE001
            failed.append(e)
        finally:
            if not again:
                over.set()

    ts = [threading.Thread(target=body, args=(j, a)) for j, a in [(large, False)] + [(q, True) for q in small]]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failed, failed


def _open_case(cells, prec=fg.FG_PREC_FP64):
    h = 1.0 / min(cells)
    grid = synth.Grid(*[synth.uniform_nodes(n, 0, n * h) for n in cells])
    c = fg.Case(grid, fg.default_config(precision=prec, rtol=1e-12, max_cycles=60))
    z = np.zeros(grid.shape, np.int8, order="F")
    none = np.zeros((0, 3), np.int32)
    rows = dict(ijk=none, cell=none, coefN=np.zeros((0, 8)), probe=np.zeros(0), ip=np.zeros((0, 3)))
    c.set_geometry(z, z, z, rows, rows)
    c.mg_prepare()
    return c, grid


def _smooth_rhs(grid, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = grid.nx, grid.ny, grid.nz
    phi = synth.fortran_zeros(grid)
    phi[1:nx, 1:ny, 1:nz] = synth.box_smooth(rng.standard_normal((nx - 1, ny - 1, nz - 1)), 2)
    synth.neumann_fill(grid, phi)
    return synth.laplacian(grid, phi)


# (24, 25, 25) FP64: 12 x 13 x 13 cells below it, the largest level one block
# keeps in shared memory, some 55 KB of it; 8^3 takes about 10
def test_solves_sent_from_the_host():
    work = []
    for q, cells in enumerate([(24, 25, 25)] + [(8, 8, 8)] * SMALL):
        c, grid = _open_case(cells)
        f, p = _dev(_smooth_rhs(grid, q)), torch.zeros(grid.shape[::-1], dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        c.profile(True)  # launch classes timed: every kernel from the host
        c.solve_poisson_device(p.data_ptr(), f.data_ptr())
        assert c.solve_mode() == 0
        work.append((c, f, p, p.clone()))

    def job(c, f, p, alone, times):
        def run():
            for _ in range(times):
                p.zero_()
                torch.cuda.current_stream().synchronize()
                c.solve_poisson_device(p.data_ptr(), f.data_ptr())
        return run

    _together(job(*work[0], 200), [job(*w, 1) for w in work[1:]])
    for c, f, p, alone in work:
        # both solve to 1e-12 of the right-hand side: 1e-9 allows the
        # solution a thousand times that
        assert float((p - alone).abs().max() / alone.abs().max()) <= 1e-9
        c.close()


def test_moving_bodies_in_graphs():
    def make(cells, radius, steps):
        h = 0.1
        grid = synth.Grid(*[synth.uniform_nodes(n, 0, n * h) for n in cells])
        c = fg.Case(grid, fg.default_config(precision=fg.FG_PREC_FP64, rtol=1e-10, max_cycles=4))
        body = synth.sphere_body(tuple(0.5 * n * h for n in cells), radius, 3)
        c.add_body(body)
        verts = np.array(body.verts, dtype=np.float64)
        f, p = _dev(_smooth_rhs(grid, 3)), torch.zeros(grid.shape[::-1], dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        out = []

        def run():
            out.clear()
            for step in range(steps):
                moved = verts.copy()
                moved[:, 0] += 0.03 * (step % 8)
                c.update_body(0, moved)
                c.set_iblank_body_fast()
                c.gcm_set_internal_boundary()
                c.mg_prepare()
                p.zero_()
                torch.cuda.current_stream().synchronize()
                # (the right-hand side is not a body's: no convergence asked for)
                c.solve_poisson_device(p.data_ptr(), f.data_ptr(), allow_not_converged=True)
                assert c.solve_mode() == 1
                out.append((c.nGhost, c.nDead))
        return c, run, out

    large = make((24, 25, 25), 0.6, 64)
    small = [make((10, 10, 10), 0.25, 1) for _ in range(SMALL)]
    alone = []
    for c, run, out in [large] + small:
        run()
        alone.append(list(out))
    _together(large[1], [q[1] for q in small])
    for (c, run, out), a in zip([large] + small, alone):
        assert out == a
        c.close()


def test_momentum_lines_of_two_lengths():
    work = []
    for q, n in enumerate([2040] + [1240] * SMALL):  # 4 rows per thread, 80 and 50 KB
        c, grid = _open_case((n, 3, 3))
        rng = np.random.default_rng(q)
        d = [_dev(rng.standard_normal(grid.shape)) for _ in range(5)]
        torch.cuda.synchronize()
        prm = fg.AdParams(dt=0.02, reinv=0.01, omega_ad=1.0, crank_nicolson=1)
        v0 = d[0].clone()
        fg.itsolv_ad_device(c, *[t.data_ptr() for t in d], prm)
        work.append((c, d, prm, v0, d[0].clone()))

    def job(c, d, prm, v0, alone, times):
        def run():
            for _ in range(times):
                d[0].copy_(v0)
                torch.cuda.current_stream().synchronize()
                fg.itsolv_ad_device(c, *[t.data_ptr() for t in d], prm)
        return run

    _together(job(*work[0], 600), [job(*w, 1) for w in work[1:]])
    for c, d, prm, v0, alone in work:
        assert torch.equal(d[0], alone)
        c.close()
