"""The stage kernel's warp teams and the many-steps launch at the edges of their layout.

A team steps 256/NZ modes at once; a CTA holds one to three teams; the sums over CTAs run in
groups of 16.  The mode counts below give one mode, a ragged block, one CTA more than a group,
two teams per CTA and several blocks per team.  Tolerance against the oracle: the 1e-10 bar of
the step (relative L2 of the state).  One launch of n steps and n launches of one step run the
same kernel on the same sums, so their states agree bit for bit.
"""
import ctypes
import threading
import time

import numpy as np
import pytest

from gpu_util import rel, require_gpu
from oracle import oracle as O
from ql_dns_b200 import _capi
from ql_dns_b200.batch import QLBatch
from ql_dns_b200.initial import initial_state
from ql_dns_b200.params import QLParams
from ql_dns_b200.solver import QLSolver

pytestmark = pytest.mark.gpu

# (nx, ny, NZ): (nx - 1) * ny / 2 modes
EDGES = [(2, 2, 128), (4, 2, 128), (12, 6, 128), (36, 18, 128), (32, 40, 128), (2, 2, 16), (36, 2, 16), (34, 32, 16),
         (18, 2, 256), (20, 34, 256), (10, 8, 32), (36, 34, 64)]


@pytest.mark.parametrize("integ", [0, 1])
@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("nx,ny,NZ", EDGES)
def test_layout_edges(nx, ny, NZ, model, integ):
    require_gpu()
    p = QLParams(model=model, integrator=integ, nx=nx, ny=ny, NZ=NZ, dt=0.02, B0z=0.02 if model else 0.0)
    lin, mf, kx0 = initial_state(p, 3, sigma=0.2, B0=0.05, mean_u=0.02 if model else 0.0)
    n = 3
    with QLSolver(p) as s:
        s.set_state(0.0, lin, mf, kx0)
        rec = s.step(n, diag_every=1)
        t, lo, mo, ko = s.get_state()
        s.set_state(0.0, lin, mf, kx0)
        for _ in range(n):
            s.step(1)
        t1, l1, m1, k1 = s.get_state()
    assert t == t1 and np.array_equal(lo, l1) and np.array_equal(mo, m1) and np.array_equal(ko, k1)
    t2, lo2, mo2, ko2, d2 = O.run(p, 0.0, lin, mf, kx0, n, diag_every=1)
    assert t == t2 and np.array_equal(ko, ko2)
    assert rel(mo, mo2) < 1e-10
    assert rel(lo, lo2) < 1e-10 if np.linalg.norm(lo2) else not lo.any()
    scale = np.abs(d2[1:, 1:13]).max(0)
    assert np.all(np.abs(rec[:, 1:13] - d2[1:, 1:13]) <= 1e-10 * scale)


@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("warps", [1, 3, 5, 8, 9, 14, 15, 16])
def test_work_item_widths(warps, model):
    """Work items of every kind of team: less than one, one wider than its tasks, several, idle warps."""
    require_gpu()
    p = QLParams(model=model, nx=6, ny=6, NZ=16, dt=0.02, B0z=0.02 if model else 0.0)
    lin, mf, kx0 = initial_state(p, 3, sigma=0.2, B0=0.05, mean_u=0.02 if model else 0.0)
    with QLBatch([p]) as b:
        b.set_mapping(warps, [1])
        b.set_state(0, 0.0, lin, mf, kx0)
        b.step(3)
        t, lo, mo, ko = b.get_state(0)
    t2, lo2, mo2, ko2, _ = O.run(p, 0.0, lin, mf, kx0, 3)
    assert t == t2 and np.array_equal(ko, ko2)
    assert rel(mo, mo2) < 1e-10 and rel(lo, lo2) < 1e-10


@pytest.mark.parametrize("integ", [0, 1])
@pytest.mark.parametrize("model", [0, 1])
@pytest.mark.parametrize("nx,ny,NZ", [(2, 2, 128), (32, 40, 128), (18, 2, 256), (36, 34, 64), (8, 8, 16)])
def test_forced_layout_edges(nx, ny, NZ, model, integ):
    """Noise and the CFL time step inside the launch; a record every second step."""
    require_gpu()
    p = QLParams(model=model, integrator=integ, nx=nx, ny=ny, NZ=NZ, dt=0.02, B0z=0.02 if model else 0.0)
    lin, mf, kx0 = initial_state(p, 3, sigma=0.02, B0=0.2, mean_u=0.05 if model else 0.0)
    n, cfl, noise = 6, (0.3, 0.05), (0.02, 0.5, 50.0, 7)
    with QLSolver(p) as s:
        s.set_noise(*noise)
        s.set_cfl(*cfl)
        s.set_state(0.0, lin, mf, kx0)
        rec = s.step(n, diag_every=2)
        t, lo, mo, ko = s.get_state()
        dtm = s.mean_time_step()
        s.set_state(0.0, lin, mf, kx0)
        for _ in range(n):
            s.step(1)
        t1, l1, m1, k1 = s.get_state()
        assert dtm == s.mean_time_step()
    assert t == t1 and np.array_equal(lo, l1) and np.array_equal(mo, m1) and np.array_equal(ko, k1)
    t2, lo2, mo2, ko2, d2, dtm2 = O.run_forced(p, 0.0, lin, mf, kx0, n, diag_every=2, cfl=cfl[0], dt_max=cfl[1],
                                              f_noise=noise[0], k_lo=noise[1], k_hi=noise[2], seed=noise[3])
    assert abs(t - t2) <= 1e-13 * t2 and abs(dtm - dtm2) <= 1e-13 * dtm2 and np.array_equal(ko, ko2)
    assert rel(mo, mo2) < 1e-10
    assert rel(lo, lo2) < 1e-10 if np.linalg.norm(lo2) else not lo.any()
    assert rec.shape[0] == 3
    scale = np.abs(d2[1:, 1:13]).max(0)
    assert np.all(np.abs(rec[:, 1:13] - d2[1:, 1:13]) <= 1e-10 * scale)


def test_forced_across_launches():
    """260 steps are two launches: noise counter, time step and its mean carry over."""
    require_gpu()
    p = QLParams(nx=8, ny=8, NZ=16, dt=0.02)
    st = initial_state(p, 3, sigma=0.02, B0=0.2)
    out = []
    for parts in ((260,), (100, 160)):
        with QLSolver(p) as s:
            s.set_noise(0.02, 0.5, 50.0, 7)
            s.set_cfl(0.3, 0.05)
            s.set_state(0.0, *st)
            for n in parts:
                rec = s.step(n, diag_every=20)
            out.append(s.get_state() + (s.mean_time_step(), rec[-1]))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("model", [0, 1])
def test_status_keeps_the_bits_of_every_cta(model):
    """The first reducer drops records (4) while the others see a non-finite field (1), in the same launch."""
    require_gpu()
    p = QLParams(model=model, nx=8, ny=8, NZ=16, dt=0.02)
    lin, mf, kx0 = initial_state(p, 3, sigma=0.02, B0=0.2)
    mf[1, 1] = np.nan
    out, n = np.zeros((2, 15)), ctypes.c_int()
    with QLSolver(p) as s:
        s.set_state(0.0, lin, mf, kx0)
        assert s.L.qlgpu_step(s.h, 6, 1, _capi.dptr(out), 2, ctypes.byref(n)) == 4
        assert n.value == 2 and s.status() == 5


def run_state(s, st, n, forced):
    s.set_noise(0.02 if forced else 0.0, 0.5, 50.0, 7)
    s.set_cfl(0.3 if forced else 0.0, 0.05 if forced else 0.0)
    s.set_state(0.0, *st)
    rec = s.step(n, diag_every=2)
    return s.get_state() + (rec,)


@pytest.mark.parametrize("forced", [False, True])
@pytest.mark.parametrize("model,nx,ny,NZ,launch", [(0, 8, 8, 16, 1), (0, 8, 8, 16, 2), (0, 32, 40, 128, 1), (1, 36, 34, 64, 1)])
def test_wait_bound_reports_timeout(model, nx, ny, NZ, launch, forced):
    """A count that never comes: the bounded waits end the launch (and those after it) with a status, and
    the handle is as good as new once a state is set."""
    require_gpu()
    p = QLParams(model=model, nx=nx, ny=ny, NZ=NZ, dt=0.02, B0z=0.02 if model else 0.0)
    st = initial_state(p, 3, sigma=0.02, B0=0.2, mean_u=0.05 if model else 0.0)
    n = 6 if launch == 1 else 260  # 256 steps a launch
    with QLSolver(p) as s:
        good = run_state(s, st, n, forced)
    with QLSolver(p) as s:
        s.set_wait(0.2)
        s.debug_drop_arrival(launch)
        with pytest.raises(_capi.QLGPUError) as ei:
            run_state(s, st, n, forced)
        assert ei.value.code == 4 and "gave up" in str(ei.value)
        assert s.status() & 8
        for a, b in zip(run_state(s, st, n, forced), good):
            assert np.array_equal(a, b)
        assert s.status() == 0


# eighteen steps, a checkpoint every five: four forward launches, then three recomputes
@pytest.mark.parametrize("launch", [1, 4, 5, 7])
def test_adjoint_wait_bound_reports_timeout(launch):
    require_gpu()
    p = QLParams(nx=8, ny=8, NZ=32, dt=0.02)
    st = initial_state(p, 3, sigma=0.2)
    with QLSolver(p) as s:
        good = s.adjoint_maxwell(0.0, *st, 18, 5)
    with QLSolver(p) as s:
        s.set_wait(0.2)
        s.debug_drop_arrival(launch)
        with pytest.raises(_capi.QLGPUError) as ei:
            s.adjoint_maxwell(0.0, *st, 18, 5)
        assert ei.value.code == 4 and "gave up" in str(ei.value)
        for a, b in zip(s.adjoint_maxwell(0.0, *st, 18, 5), good):
            assert np.array_equal(a, b)


def test_wait_bound_does_not_run_before_the_launch_does():
    """Another stream's launch holds most SMs for far longer than the bound: the step waits its turn."""
    require_gpu()
    p = QLParams(nx=64, ny=64, NZ=128, dt=0.005)
    st = initial_state(p, 1)
    q = QLParams(nx=8, ny=8, NZ=128, dt=1e-4)
    with QLSolver(p) as s, QLBatch([q] * 100) as b:
        good = run_state(s, st, 4, False)
        b.set_mapping(15, [1] * 100)  # a CTA, and so an SM, for each case
        for c in range(100):
            b.set_state(c, 0.0, *initial_state(q, 1))
        steps = int(1500.0 / (b.step_timed(100) / 100))  # 1.5 s
        s.set_wait(0.1)
        s.set_state(0.0, *st)
        th = threading.Thread(target=b.step, args=(steps,))
        th.start()
        time.sleep(0.3)
        t0 = time.time()
        rec = s.step(4, diag_every=2)
        assert time.time() - t0 > 0.2, "the step was not held up"
        th.join()
        for a, c in zip(s.get_state() + (rec,), good):
            assert np.array_equal(a, c)


@pytest.mark.parametrize("nx,ny,NZ", [(32, 32, 64), (64, 64, 16), (48, 48, 32)])
def test_handles_on_threads_share_the_gpu(nx, ny, NZ):
    """Launches of handles whose teams have an SM each leave room for a second one, and threads that step
    their own handles at the same time get what one alone gets."""
    require_gpu()
    p = QLParams(nx=nx, ny=ny, NZ=NZ, dt=0.005)
    st = initial_state(p, 3)
    ss = [QLSolver(p) for _ in range(4)]
    try:
        assert ss[0].kernel_attrs()["ctas_per_sm"] >= 2
        good = run_state(ss[0], st, 40, False)
        for s in ss:
            s.set_state(0.0, *st)
        th = [threading.Thread(target=s.step, args=(40,)) for s in ss]
        for t in th:
            t.start()
        for t in th:
            t.join()
        for s in ss:
            for a, b in zip(s.get_state(), good):
                assert np.array_equal(a, b)
    finally:
        for s in ss:
            s.close()
