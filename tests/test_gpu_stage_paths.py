"""The stages' kernels at the sizes where their launch shapes turn: tile and warp
edges, one-cell axes, scan chunks, ragged multigrid levels, values that are not
finite.
"""

import numpy as np
import pytest
import torch

import hfgrid

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
