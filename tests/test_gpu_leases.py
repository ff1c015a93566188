"""Kernels whose blocks wait on one another share a GPU by lease: a resident
pressure solve takes every SM and is refused beside a large extrapolation (the
streaming kernels solve instead); a large extrapolation waits for a resident
solve; an extrapolation that is one thread block cluster needs no lease.
"""
import threading
import time

import numpy as np
import pytest
import torch

import hfgrid
import oracle
import scenes

pytestmark = pytest.mark.gpu
UNKNOWN = np.finfo(np.float32).max
DT = 1 / 60
NONE, SHARED, EXCLUSIVE = 0, 1, 2


@pytest.fixture
def lease(cuda):
    yield hfgrid.hold_lease
    hfgrid.hold_lease(NONE)


def _system(res, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    nx, ny, nz = res
    mk = torch.zeros((nz, ny, nx), dtype=torch.uint8, device="cuda")
    mk[:, : max(1, int(0.7 * ny)), : max(1, int(0.9 * nx))] = 1
    for kind in (2, 0):
        mk[torch.rand(mk.shape, generator=g, device="cuda") < 0.01] = kind
    v = [torch.randn(s, generator=g, device="cuda") for s in hfgrid.face_shapes(res)]
    return mk, v, [torch.zeros_like(t) for t in v]


def _project(res, system, precond, iters):
    mk, v, sv = system
    v = [t.clone() for t in v]
    p = torch.empty(mk.shape, device="cuda")
    st = hfgrid.op_project(res, (1 / 64, 1 / 60, 1 / 70), DT, mk, v, sv, precond=precond, tol_mode=1, tol=1e-30,
                           max_iter=iters, p_out=p)
    # the longest solves reach 1e-30 before their cap, and after the 512 iterations of one launch
    assert st["iterations"] == iters or 520 < st["iterations"] < iters
    return [p] + v, st


# More tile columns times planes than a cluster takes: shares of a few planes
# (x, r and A p in registers) and of more than 16 (x and r streamed, A p formed
# twice).  Both forms do the same FP32 operations on every cell; their FP64 dot
# products are summed in another order, and a scalar of the recurrence, once
# rounded to FP32, differs only if its rounding is decided by a last bit of
# FP64: at odds of the order of 2**-26 a scalar, not in these systems.  The longest take
# more than one launch of the resident form.
@pytest.mark.parametrize("res,iters", [((128, 96, 100), 1), ((128, 96, 100), 20), ((128, 96, 100), 200),
                                       ((300, 40, 60), 1300), ((200, 160, 150), 1), ((200, 160, 150), 200),
                                       ((200, 160, 150), 1300)])
@pytest.mark.parametrize("precond", [hfgrid.PRECOND_IDENTITY, hfgrid.PRECOND_JACOBI])
def test_refused_solve_gives_the_same_bits(lease, res, iters, precond):
    system = _system(res, 3)
    resident, st = _project(res, system, precond, iters)
    lease(SHARED)
    pair, st2 = _project(res, system, precond, iters)
    assert st["iterations"] == st2["iterations"]
    assert st["residual"] == pytest.approx(st2["residual"], rel=1e-12)
    for a, b in zip(resident, pair):
        assert torch.equal(a, b)


def test_refused_solve_takes_the_streaming_kernels(lease):
    """The launches of a step tell the forms apart."""
    sc = scenes.Scene(res=(100, 96, 90), seed=3)
    steps = []
    for kind in (NONE, SHARED, EXCLUSIVE, NONE):
        g = scenes.gpu_solver(sc, precond=1, tol_mode=1, tol=1e-6, max_iter=60)
        lease(kind)  # the extrapolation of this grid is a cluster: no lease of its own
        before = g.launch_count
        g.update()
        steps.append((g.launch_count - before, g.stats()["cg_iterations"]))
    assert steps[0] == steps[3] and steps[1] == steps[2]
    assert steps[0][1] == steps[1][1] >= 20
    assert steps[1][0] - steps[0][0] >= 2 * steps[0][1] - 2


def _extrapolation(res):
    rng = np.random.default_rng(2)
    v = [rng.standard_normal(s).astype(np.float32) for s in oracle.face_shapes(res)]
    for a in v:
        a[rng.random(a.shape) < 0.99] = UNKNOWN
    return v


@pytest.mark.parametrize("res,waits", [((60, 50, 40), False), ((99, 99, 99), False), ((105, 101, 102), True)])
def test_extrapolation_waits_only_as_a_grid(lease, res, waits):
    v = _extrapolation(res)
    vd = [torch.from_numpy(a).cuda() for a in v]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    done = threading.Event()

    def work():
        hfgrid.op_extrapolate_fc(res, vd, 1000, stream=stream.cuda_stream)
        done.set()

    lease(EXCLUSIVE)
    t = threading.Thread(target=work)
    t.start()
    assert done.wait(2.0 if waits else 20.0) == (not waits)
    lease(NONE)
    t.join(20.0)
    assert done.is_set()
    for a, b in zip(vd, oracle.extrapolate_fc(res, v, 1000)):
        assert np.array_equal(a.cpu().numpy(), b)


def test_shared_leases_do_not_exclude_one_another(lease):
    lease(SHARED)
    res = (105, 101, 102)
    v = _extrapolation(res)
    vd = [torch.from_numpy(a).cuda() for a in v]
    t0 = time.perf_counter()
    hfgrid.op_extrapolate_fc(res, vd, 1000)
    assert time.perf_counter() - t0 < 20
    for a, b in zip(vd, oracle.extrapolate_fc(res, v, 1000)):
        assert np.array_equal(a.cpu().numpy(), b)


def test_large_jacobi_scenes_side_by_side(cuda):
    """Two served scenes whose solves and extrapolations both want the GPU:
    each ends where it ends alone (P2G's atomics: FP32 rounding)."""
    reqs = [hfgrid.scene_desc((112, 108, 104), steps=4, spheres=[(0.5, 0.15, 0.5, 0.12)], seed=5 + i,
                              keep_particles=True, precond=hfgrid.PRECOND_JACOBI, tol_mode=hfgrid.TOL_RELATIVE,
                              tol=1e-6, max_iter=200) for i in range(2)]
    ends = []
    for slots in (1, 2):
        srv = hfgrid.Server(slots=slots, budget_bytes=8 << 30)
        ids = [srv.submit(d) for d in reqs]
        srv.drain()
        for i in ids:
            inf = srv.wait(i)
            assert inf["status"] == 2 and inf["steps_done"] == 4
            ends.append((inf["last"]["substeps"], srv.particles(i, inf["particles"])))
        srv.close()
    for (n0, a), (n1, b) in zip(ends[:2], ends[2:]):
        assert n0 == n1
        # single particles that decide a marker move their surroundings more
        assert (np.abs(a - b).max(1) > 1e-4).mean() < 1e-3


@pytest.mark.parametrize("precond", [hfgrid.PRECOND_IDENTITY, hfgrid.PRECOND_JACOBI])
def test_long_solve_of_a_cluster(cuda, precond):
    """A channel of 1300 fluid cells needs more iterations than one launch of
    the cluster form makes (512).  The FP64 iterate is solved by the streaming
    kernels with the same r, p and scalars, so the iterations and the residual
    are the same and the pressures differ by the rounding of x: at most one
    2**-24 of the largest partial sum an iteration."""
    out = []
    for fp64 in (0, 1):
        sc = scenes.Scene(res=(1500, 6, 5), seed=3, fluid_max=(0.9, 1.0, 1.0))
        g = scenes.gpu_solver(sc, precond=precond, tol_mode=1, tol=1e-12, max_iter=1100, pressure_fp64=fp64)
        rng = np.random.default_rng(1)
        g.set_velocity_field(*[rng.standard_normal(s).astype(np.float32) for s in hfgrid.face_shapes(sc.res)])
        g.solve_pressure()
        out.append((g.stats(), g.pressure().astype(np.float64)))
    (s0, p0), (s1, p1) = out
    assert s0["cg_iterations"] == s1["cg_iterations"] > 520
    assert s0["cg_residual"] == pytest.approx(s1["cg_residual"], rel=1e-9)
    assert np.abs(p0 - p1).max() <= s0["cg_iterations"] * 2.0 ** -24 * np.abs(p1).max()


def test_idle_scenes_leave_their_share_to_an_extrapolation(cuda):
    """31 scenes that are not extrapolating: a call takes twice the fair 32nd of
    the GPU.  A layer is bound by the latency of a block's chain, so a sixteenth
    costs some twice the time of the whole GPU here, and a 32nd four times."""
    res = (160, 160, 160)
    shapes = hfgrid.face_shapes(res)
    v0 = [torch.full(s, float(UNKNOWN), device=cuda) for s in shapes]
    for a in v0:
        a[:, :96, :64] = 1.0

    def best():
        t = []
        for _ in range(7):
            v = [a.clone() for a in v0]
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            hfgrid.op_extrapolate_fc(res, v, 1000)
            t.append(time.perf_counter() - t0)
        return min(t)

    alone = best()
    idle = [hfgrid.Solver(1 / 60, (4, 4, 4)) for _ in range(31)]
    assert best() < 3 * alone
    for s in idle:
        s.close()
