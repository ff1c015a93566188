"""The stages' kernels at the sizes where their launch shapes turn: tile and warp
edges, one-cell axes, scan chunks, ragged multigrid levels, values that are not
finite.
"""
import ctypes
import ctypes.util
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


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def host(t):
    torch.cuda.synchronize()
    return t.cpu().numpy()


# --- distance fields: integers, so exact ------------------------------------
def _steps(seed, closed):
    """6-neighbour steps from `seed` through the cells that are not `closed`."""
    d = np.full(seed.shape, -1, np.int64)
    d[seed] = 0
    front, k = seed.copy(), 0
    while front.any():
        k += 1
        grow = np.zeros_like(front)
        for ax in range(3):
            for s in (1, -1):
                moved = np.roll(front, s, ax)
                edge = [slice(None)] * 3
                edge[ax] = 0 if s == 1 else -1
                moved[tuple(edge)] = False
                grow |= moved
        front = grow & ~closed & (d < 0)
        d[front] = k
    return d


def _serpentine(res):
    """Walls with a gap at alternating ends: every corridor is one more turn."""
    nx, ny, nz = res
    closed = np.zeros((nz, ny, nx), bool)
    for i, y in enumerate(range(1, ny - 1, 2)):
        closed[:, y, :] = True
        closed[:, y, -1 if i % 2 else 0] = False
    return closed


@pytest.mark.parametrize("res,kind", [((1, 1, 1), "random"), ((7, 1, 1), "random"), ((33, 5, 2), "random"),
                                      ((31, 17, 40), "random"), ((64, 33, 9), "random"), ((5, 121, 2), "serpentine"),
                                      ((40, 9, 3), "serpentine")])
@pytest.mark.parametrize("distance", [1, 5, 1000])
def test_side_distance_fields(cuda, res, kind, distance):
    rng = np.random.default_rng(sum(res))
    shape = res[::-1]
    if kind == "random":
        density = rng.choice(np.array([0, 0.2, 1], np.float32), shape, p=(0.47, 0.06, 0.47))
        solid = np.where(rng.random(shape) < 0.2, -1.0, 1.0).astype(np.float32)
    else:  # one seed at the start of a long corridor; more turns than rounds between two host reads
        closed = _serpentine(res)
        density = np.zeros(shape, np.float32)
        density[:, 0, 0] = 0.2
        solid = np.where(closed, -1.0, 1.0).astype(np.float32)
    for outside in (True, False):
        seed = (density == np.float32(0.2)) & (solid >= 0)
        closed = (solid < 0) | ((density == (1 if outside else 0)) & ~seed)
        d = _steps(seed, closed & ~seed)
        s = 0.5 - 0.2 if outside else 0.2 - 0.5
        sweeps = 1
        while sweeps < distance and np.float32(sweeps + s - 1) == np.float32((sweeps - 1) + s):
            sweeps += 1
        ref = np.full(shape, UNKNOWN, np.float32)
        near = (d >= 0) & (d < sweeps)
        ref[near] = np.maximum((d[near] + s).astype(np.float32), 0)
        ref[closed] = 0
        out = torch.empty(shape, device=cuda)
        f = hfgrid.op_build_fluid_outside_sdf if outside else hfgrid.op_build_fluid_inside_sdf
        f(res, dev(density), dev(solid), out, distance)
        assert np.array_equal(host(out), ref)


def _porous(res, closed, seed):
    """A seed plane below cells of which a share is closed: walks that wind."""
    rng = np.random.default_rng(seed)
    shape = res[::-1]
    density = np.ones(shape, np.float32)
    density[:, 0, :] = 0.2
    solid = np.where(rng.random(shape) < closed, -1.0, 1.0).astype(np.float32)
    return density, solid


@pytest.mark.parametrize("res,closed", [((31, 9, 7), 0.3), ((32, 40, 8), 0.3), ((33, 41, 17), 0.6), ((70, 90, 60), 0.45),
                                        ((100, 64, 65), 0.2), ((3, 200, 2), 0.1)])
@pytest.mark.parametrize("distance", [1, 2, 4, 5, 12, 1000])
def test_side_distance_fields_among_scattered_solids(cuda, res, closed, distance):
    density, solid = _porous(res, closed, 1)
    wall = solid < 0
    seed = (density == np.float32(0.2)) & ~wall
    d = _steps(seed, wall)
    sweeps = 1
    while sweeps < distance and np.float32(sweeps - 0.3 - 1) == np.float32(sweeps - 1 - 0.3):
        sweeps += 1
    ref = np.where((d >= 0) & (d < sweeps), np.maximum((d - 0.3).astype(np.float32), 0), UNKNOWN).astype(np.float32)
    ref[wall] = 0
    out = torch.empty(res[::-1], device=cuda)
    hfgrid.op_build_fluid_inside_sdf(res, dev(density), dev(solid), out, distance)
    got = host(out)
    assert np.array_equal(got == UNKNOWN, ref == UNKNOWN)
    assert np.allclose(got, ref, rtol=1e-6)  # the value's rounding; the steps are whole


def test_side_distance_field_time_among_scattered_solids(cuda):
    """Each round of line passes settles one straight piece of a walk; among
    scattered solids a walk has dozens, and no call may cost dozens of rounds."""
    def best(closed, distance):
        density, solid = (dev(a) for a in _porous((128, 128, 128), closed, 1))
        out = torch.empty_like(density)
        t = []
        for _ in range(5):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            hfgrid.op_build_fluid_inside_sdf((128, 128, 128), density, solid, out, distance)
            t.append(time.perf_counter() - t0)
        return min(t)

    open_, winding = best(0.0, 1000), best(0.3, 30)
    assert winding < 15 * open_, (open_, winding)


@pytest.mark.parametrize("res", [(1, 1, 1), (2, 1, 1), (33, 31, 5), (64, 3, 70), (17, 130, 4)])
@pytest.mark.parametrize("layers", [1, 4, 1000])
def test_fluid_distance_field(cuda, res, layers):
    rng = np.random.default_rng(res[0] + layers)
    dom = np.where(rng.random(res[::-1]) < 0.02, -500.0, 500.0).astype(np.float32)
    ins = dom < 0
    mixed = np.zeros_like(ins)
    for ax in range(3):
        for s in (1, -1):
            i = np.clip(np.arange(ins.shape[ax]) + s, 0, ins.shape[ax] - 1)
            mixed |= np.take(ins, i, ax) != ins
    d = np.where(ins, _steps(mixed & ins, ~ins), _steps(mixed & ~ins, ins))
    ok = (d == 0) | ((d > 0) & (d < layers))
    ref = np.where(ins, np.where(d == 0, 0.5 - 0.2, -(d - (0.5 - 0.2))), d + (1.5 - 0.2)).astype(np.float32)
    ref[~ok] = np.where(ins, -UNKNOWN, UNKNOWN)[~ok]
    out = torch.empty(res[::-1], device=cuda)
    hfgrid.op_build_fluid_sdf(res, dev(dom), out, layers)
    assert np.array_equal(host(out), ref)


# --- extrapolation: means in a fixed order, so exact --------------------------
@pytest.mark.parametrize("res", [(1, 1, 1), (31, 2, 3), (33, 17, 1), (40, 129, 3), (257, 9, 5),
                                 (90, 80, 60), (101, 100, 102)])
def test_extrapolation_shapes(cuda, res):
    """Both forms of the layer pass (one cluster up to 3 M faces, a grid above)."""
    rng = np.random.default_rng(res[1])
    v = [rng.standard_normal(s).astype(np.float32) for s in oracle.face_shapes(res)]
    for a in v:
        a[rng.random(a.shape) < (0.97 if a.size < 10000 else 0.9999)] = UNKNOWN
        a.flat[0] = 1.0
    for layers in (2, 7, 1000) if res[0] < 90 else (1000,):
        vd = [dev(a) for a in v]
        hfgrid.op_extrapolate_fc(res, vd, layers)
        for x, y in zip(vd, oracle.extrapolate_fc(res, v, layers)):
            assert np.array_equal(host(x), y)


# --- transfers ------------------------------------------------------------------
@pytest.mark.parametrize("alg", [hfgrid.LINEAR, hfgrid.QUADRATIC, hfgrid.CUBIC])
@pytest.mark.parametrize("res", [(1, 1, 1), (2, 3, 1), (8, 5, 6), (13, 4, 7)])
def test_p2g_rows_of_both_alignments(cuda, alg, res):
    """Rows that start on and off 16 bytes, and rows shorter than the stencil,
    face by face against the FP64 oracle.  A coordinate of at most 15 cells is off
    by a few 2**-24 of that, 4e-6 cells, so is each weight, and the FP32 sums add
    less than 1e-5 of theirs; values, at most 5, weigh as much more."""
    rng = np.random.default_rng(alg)
    h = (0.1, 0.12, 0.09)
    n = 400
    pos = ((rng.random((n, 3)) * 1.2 - 0.1) * np.array(res) * np.array(h)).astype(np.float32)
    vel = rng.standard_normal((n, 3)).astype(np.float32)
    out = [torch.empty(s, device=cuda) for s in oracle.face_shapes(res)]
    wgt = [torch.empty(s, device=cuda) for s in oracle.face_shapes(res)]
    hfgrid.op_p2g_fc(res, (0, 0, 0), h, dev(pos), dev(vel), alg, out, wgt)
    ref, refw = oracle.p2g_fc(res, (0, 0, 0), h, pos, vel, alg, dbl=1)
    assert np.abs(vel).max() < 5
    for v, w, rv, rw in zip(out, wgt, ref, refw):
        c = min(n, 64 * n / w.numel())  # about as many particles reach a face, at most
        v, w, rv, rw = (a.astype(np.float64) for a in (host(v), host(w), rv, rw))
        assert (np.abs(w - rw) <= 4e-6 * c + 1e-5 * rw).all()
        assert (np.abs(v * w - rv * rw) <= 5 * (4e-6 * c + 2e-5 * rw)).all()
    # weights: the sum over all faces of a component is one per particle
    for w in wgt:
        assert abs(float(w.double().sum()) / n - 1) < 1e-5
    num = [torch.empty(s, device=cuda) for s in oracle.face_shapes(res)]
    hfgrid.op_p2g_fc(res, (0, 0, 0), h, dev(pos), dev(np.ones_like(vel)), alg, num)
    for v, w in zip(num, wgt):  # a constant comes back where anything arrived
        assert torch.allclose(v[w > 1e-6], torch.ones_like(v[w > 1e-6]), rtol=1e-5)


def test_p2g_value_not_finite_reaches_its_whole_stencil(cuda):
    """0 times infinity is not 0: the taps of weight 0 turn NaN as well."""
    res, h = (12, 11, 10), (0.1, 0.1, 0.1)
    pos = np.array([[0.53, 0.52, 0.47]], np.float32)
    vel = np.full((1, 3), np.inf, np.float32)
    out = [torch.empty(s, device=cuda) for s in oracle.face_shapes(res)]
    hfgrid.op_p2g_fc(res, (0, 0, 0), h, dev(pos), dev(vel), hfgrid.QUADRATIC, out)
    for o in out:
        assert int((~torch.isfinite(o)).sum()) == 64


@pytest.mark.parametrize("special", [np.inf, -np.inf, 3e38, np.nan])
def test_linear_samples_next_to_values_not_finite(cuda, special):
    """LINEAR G2P and semi-Lagrangian advection weigh the eight corners: between
    equal infinities that is the infinity, between large values of both signs it
    is finite, next to a NaN or between opposite infinities it is NaN."""
    rng = np.random.default_rng(6)
    res, h = (9, 8, 7), (0.1, 0.1, 0.1)
    v = [rng.standard_normal(s).astype(np.float32) for s in oracle.face_shapes(res)]
    for a in v:
        a[:, :, :3] = special
        a[:, :, 3] = special if np.isinf(special) else -special
        a[:2, :, 6:] = -special
    cell = ((rng.random((500, 3)) * 0.8 + 0.1) + rng.integers(1, 5, (500, 3))) + 0.5  # weights off 0 and 1 ...
    cell[:, 0] = rng.integers(1, 8, 500) + 0.1 + 0.3 * rng.random(500)  # ... on both grids
    cell[:, 1:] = np.floor(cell[:, 1:]) + 0.1 + 0.3 * rng.random((500, 2))
    pos = (cell * 0.1).astype(np.float32)

    def weigh(f, u):
        f = f.astype(np.float64)
        i = [np.floor(t).astype(int) for t in u]
        w = [t - b for t, b in zip(u, i)]
        acc = np.zeros(len(u[0]))
        for c in range(8):
            d = [c & 1, c >> 1 & 1, c >> 2]
            j = [np.clip(i[k] + d[k], 0, f.shape[2 - k] - 1) for k in range(3)]
            acc += np.prod([w[k] if d[k] else 1 - w[k] for k in range(3)], 0) * f[j[2], j[1], j[0]]
        return acc

    def same(got, ref):
        assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(np.isinf(got), np.isinf(ref))
        ok = ~np.isnan(ref)
        assert np.array_equal(np.sign(got[ok]), np.sign(ref[ok]))
        ok = np.isfinite(ref)
        np.testing.assert_allclose(got[ok], ref[ok], rtol=1e-4, atol=1e-5 * max(1, np.abs(ref[ok]).max()))

    with np.errstate(all="ignore"):
        u = pos.astype(np.float64) / 0.1
        refs = [weigh(v[a], [u[:, k] - (0.0 if k == a else 0.5) for k in range(3)]) for a in range(3)]
        out = torch.empty(pos.shape, device=cuda)
        hfgrid.op_g2p_fc(res, (0, 0, 0), h, [dev(a) for a in v], dev(pos), hfgrid.LINEAR, out)
        for a in range(3):
            same(host(out)[:, a], refs[a])
        # a uniform flow that moves every sample by (0.3, 0.2, 0.25) cells
        shift, dt = np.array((0.3, 0.2, 0.25)), 0.5
        flow = [np.full(s, -0.1 * shift[a] / dt, np.float32) for a, s in enumerate(oracle.face_shapes(res))]
        f = v[0][:, :, :9].copy()
        fout = torch.empty(res[::-1], device=cuda)
        hfgrid.op_sl_advect_cc(res, (0, 0, 0), h, dev(f), [dev(a) for a in flow], dt, 0, fout)
        z, y, x = np.meshgrid(*[np.arange(n) for n in res[::-1]], indexing="ij")
        ref = weigh(f, [t.reshape(-1) + shift[k] for k, t in enumerate((x, y, z))])
        same(host(fout).reshape(-1), ref)


@pytest.mark.parametrize("alg", [hfgrid.LINEAR, hfgrid.QUADRATIC, hfgrid.CUBIC])
def test_carried_scalars_match_the_operators(cuda, alg):
    """One step's colour and domain against the transfers of the operators."""
    sc = scenes.Scene(res=(20, 17, 13), seed=2)
    s = scenes.gpu_solver(sc, advect_scalars=True, kind=hfgrid.ADV_PIC)
    s.set_advection(hfgrid.ADV_PIC, hfgrid.RK3, alg, 1.0, 0.05)
    s.seed_particles(4, 2)
    rng = np.random.default_rng(1)
    col = [rng.random(sc.res[::-1]).astype(np.float32) for _ in range(3)]
    s.set_color_field(*col)
    dom0 = s.fluid_domain_field()
    p0, _ = s.particles()
    s.update()
    p1, _ = s.particles()
    got = list(s.color_field()) + [s.fluid_domain_field()]
    args = (sc.res, sc.origin, sc.spacing)
    for f, g in zip(col + [dom0], got):
        val = torch.empty(len(p0), device=cuda)
        hfgrid.op_g2p_cc(*args, dev(f), dev(p0), alg, val)
        ref = torch.empty(sc.res[::-1], device=cuda)
        hfgrid.op_p2g_cc(*args, dev(p1), val, alg, ref)
        # the order of the atomics: at most some 500 addends of one sign pattern
        np.testing.assert_allclose(g, host(ref), rtol=2e-4, atol=1e-5 * np.abs(f).max())


# --- multigrid --------------------------------------------------------------------
@pytest.mark.parametrize("res", [(15, 9, 11), (32, 16, 16), (33, 40, 18), (48, 25, 50), (64, 64, 30)])
@pytest.mark.parametrize("half", [0, 1])
def test_multigrid_level_splits(cuda, res, half):
    """Ragged grids of two to five levels: the pressure of a converged multigrid
    solve is the Jacobi solve's (both to 1e-6 of the right-hand side; the
    system's smallest eigenvalue scales the difference up by < 100)."""
    sc = scenes.Scene(res=res, seed=1, fluid_max=(0.7, 0.7, 1.0))
    out = []
    for opt in (dict(precond=2, mg_half=half), dict(precond=1)):
        s = scenes.gpu_solver(sc, tol=1e-6, max_iter=4000, **opt)
        s.update(2)
        assert s.stats()["cg_converged"]
        out.append((s.pressure().astype(np.float64), s.stats()["cg_iterations"]))
    (pm, im), (pj, ij) = out
    assert np.linalg.norm(pm - pj) < 2e-4 * np.linalg.norm(pj)
    assert im <= ij


# --- particle advection ------------------------------------------------------------
@pytest.mark.parametrize("res", [(1, 1, 1), (2, 1, 3), (9, 8, 7)])
@pytest.mark.parametrize("rk", [0, 1, 2])
def test_substep_samples_at_and_beyond_the_grid(cuda, res, rk):
    """Particles on cell centres, faces, edges of the grid and beyond it, one
    step against the FP64 formula (a substep's rounding is a few 2**-24 of the
    position: 1e-5 cells)."""
    rng = np.random.default_rng(rk)
    h = np.array((0.1, 0.12, 0.09))
    o = np.array((0.25, -0.5, 1.0))
    grid = np.stack(np.meshgrid(*[np.arange(-2, 2 * n + 3) / 2 for n in res], indexing="ij"), -1).reshape(-1, 3)
    pos = (o + np.concatenate([grid, rng.random((200, 3)) * (np.array(res) + 2) - 1]) * h).astype(np.float32)
    v = [rng.standard_normal(s).astype(np.float32) for s in oracle.face_shapes(res)]
    dt = float(0.2 * h.min() / max(np.abs(a).max() for a in v))  # one substep

    def sample(p):
        out = np.empty_like(p)
        for a in range(3):
            f = v[a].astype(np.float64)
            acc = np.zeros(len(p))
            u = [(p[:, k] - o[k]) / h[k] - (0.0 if k == a else 0.5) for k in range(3)]
            i = [np.floor(t).astype(int) for t in u]
            w = [t - b for t, b in zip(u, i)]
            for dz in (0, 1):
                for dy in (0, 1):
                    for dx in (0, 1):
                        idx = [np.clip(i[k] + d, 0, f.shape[2 - k] - 1) for k, d in enumerate((dx, dy, dz))]
                        acc += (np.where(dx, w[0], 1 - w[0]) * np.where(dy, w[1], 1 - w[1]) *
                                np.where(dz, w[2], 1 - w[2])) * f[idx[2], idx[1], idx[0]]
            out[:, a] = acc
        return out

    p = pos.astype(np.float64)
    w0 = sample(p)
    if rk == 0:
        ref = p + dt * w0
    elif rk == 1:
        ref = p + dt * sample(p + 0.5 * dt * w0)
    else:
        w1 = sample(p + 0.5 * dt * w0)
        ref = p + dt * (2 * w0 + 3 * w1 + 4 * sample(p + 0.75 * dt * w1)) / 9
    ref = np.clip(ref, o, o + np.array(res) * h)
    pd = dev(pos)
    n = hfgrid.op_advect_particles(res, o, h, [dev(a) for a in v], pd, dt, 1.0, rk, clamp_mode=0)
    assert n == 1
    assert np.abs(host(pd) - ref).max() < 1e-5 * h.max() + 4 * 2.0 ** -24 * np.abs(ref).max()

def test_substep_sample_is_its_formula_to_the_bit(cuda):
    """A floor and a weight per coordinate, then lerps of the corners along x, y
    and z, every operation rounded to FP32 once: one Euler substep against that
    formula, bit for bit.  (The substeps' positions feed the next step's
    markers, so a weight off in its last bit is another trajectory.)  One
    coordinate of each particle is small, so that its displacement's last bits
    are not rounded away with the position's."""
    fmaf = ctypes.CDLL(ctypes.util.find_library("m")).fmaf
    fmaf.restype, fmaf.argtypes = ctypes.c_float, [ctypes.c_float] * 3
    fma = np.vectorize(lambda a, b, c: np.float32(fmaf(a, b, c)), otypes=[np.float32])
    f32 = np.float32
    rng = np.random.default_rng(4)
    res, o, h, dt = (21, 18, 33), np.array((0.3, 0.0, -0.7), f32), np.array((0.11, 0.25, 0.07), f32), f32(0.05)
    ext = (np.array(res) * h.astype(np.float64))
    v = [(0.1 * ext[a] / dt * (1 + rng.random(s))).astype(f32) for a, s in enumerate(oracle.face_shapes(res))]
    pos = 0.75 * rng.random((1500, 3)) * ext
    pos[np.arange(1500), np.arange(1500) % 3] *= 0.02
    pos[:30] += rng.choice((-1, 1), (30, 3)) * 0.2 * ext  # beyond the grid: the box clamp makes some of them equal
    pos = (o + pos).astype(f32)
    inv = f32(1) / h
    off = -(o * inv)
    ref = np.empty_like(pos)
    for a in range(3):
        i, w = [], []
        for k in range(3):
            n = res[k] + (k == a)
            t = fma(pos[:, k], inv[k], off[k] if k == a else off[k] - f32(0.5))
            t = np.minimum(np.maximum(t, f32(-1)), np.nextafter(f32(n), f32(0)))
            j = np.floor(t)
            w.append(t - j)
            j = j.astype(int)
            i.append((np.clip(j, 0, n - 1), np.clip(j + 1, 0, n - 1)))

        def lerp(w, p, q):
            return fma(w, q - p, p)
        at = {(z, y, x): v[a][i[2][z], i[1][y], i[0][x]] for z in (0, 1) for y in (0, 1) for x in (0, 1)}
        row = {(z, y): lerp(w[0], at[z, y, 0], at[z, y, 1]) for z in (0, 1) for y in (0, 1)}
        val = lerp(w[2], lerp(w[1], row[0, 0], row[0, 1]), lerp(w[1], row[1, 0], row[1, 1]))
        top = o[a] + f32(res[a]) * h[a]
        ref[:, a] = np.maximum(o[a], np.minimum(fma(dt, val, pos[:, a]), top))
    pd = dev(pos)
    n = hfgrid.op_advect_particles(res, o, h, [dev(x) for x in v], pd, float(dt), 1e4, 0, clamp_mode=0)
    assert n == 1
    got = host(pd)
    inside = (ref > o) & (ref < o + np.array(res) * h * f32(0.999))  # the box bound itself rounds as an FMA may
    assert inside.mean() > 0.9
    assert np.array_equal(got[inside], ref[inside])


# --- operator scratch -----------------------------------------------------------------
def test_operators_on_several_threads_and_streams(cuda):
    """The operators' scratch pool: the same results from four threads on
    streams of their own, and at most its bound (512 MiB, and the driver's
    granularity) stays with it afterwards."""
    rng = np.random.default_rng(0)
    res, h = (40, 36, 30), (1 / 40, 1 / 36, 1 / 30)
    pos = dev(rng.random((20000, 3)).astype(np.float32))
    vel = dev(rng.standard_normal((20000, 3)).astype(np.float32))
    shapes = oracle.face_shapes(res)

    def work(stream, outs):
        with torch.cuda.stream(stream):
            for _ in range(20):
                hfgrid.op_p2g_fc(res, (0, 0, 0), h, pos, vel, hfgrid.LINEAR, outs)

    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    runs = [(torch.cuda.Stream(), [torch.empty(s, device=cuda) for s in shapes]) for _ in range(4)]
    threads = [threading.Thread(target=work, args=r) for r in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for _, outs in runs[1:]:
        for a, b in zip(outs, runs[0][1]):
            assert torch.allclose(a, b, rtol=1e-4, atol=1e-4)
    big = (256, 256, 200)
    v = [torch.zeros(s, device=cuda) for s in oracle.face_shapes(big)]
    p = torch.rand((1000, 3), device=cuda)
    hfgrid.op_advect_particles(big, (0, 0, 0), (1 / 256, 1 / 256, 1 / 200), v, p, 1 / 60)  # 0.9 GB of tables
    del v
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] < (512 + 256) << 20


def _keep_scratch(cuda):
    """An operator call whose scratch (0.45 GB of tables) the pool keeps."""
    res = (200, 200, 176)
    v = [torch.zeros(s, device=cuda) for s in oracle.face_shapes(res)]
    p = torch.rand((1000, 3), device=cuda)
    hfgrid.op_advect_particles(res, (0, 0, 0), tuple(1 / n for n in res), v, p, 1 / 60)
    del v, p
    torch.cuda.empty_cache()
    torch.cuda.synchronize()


def test_release_scratch_gives_the_pool_back(cuda):
    hfgrid.release_scratch()
    _keep_scratch(cuda)
    free0 = torch.cuda.mem_get_info()[0]
    hfgrid.release_scratch()
    assert torch.cuda.mem_get_info()[0] - free0 > 300 << 20
    _keep_scratch(cuda)  # the next call takes it anew


def test_kept_scratch_does_not_refuse_a_scene(cuda):
    """A scene that fits the free memory and what the pool keeps, but not the
    free memory alone: its allocations get the pool's."""
    res = (200, 200, 176)
    h = tuple(1 / n for n in res)
    hfgrid.release_scratch()
    hfgrid.Solver(1 / 60, res, (0, 0, 0), h)  # what the constructor leaves behind the first time
    _keep_scratch(cuda)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    hfgrid.release_scratch()
    kept = torch.cuda.mem_get_info()[0] - free0
    s = hfgrid.Solver(1 / 60, res, (0, 0, 0), h)
    need = free0 + kept - torch.cuda.mem_get_info()[0]
    del s
    assert kept > 300 << 20 and need > kept
    _keep_scratch(cuda)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - need + kept // 2, dtype=torch.uint8, device=cuda)
    s = hfgrid.Solver(1 / 60, res, (0, 0, 0), h)
    s.synchronize()
    del s, hold
    torch.cuda.empty_cache()
