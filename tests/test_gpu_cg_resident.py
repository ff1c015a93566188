"""The pressure CG's two forms against the same CG in plain PyTorch FP64.

`op_project` solves a system whose fluid fits the GPU's shared memory in one
resident launch (shares of up to 16 planes keep x and r in registers, larger
ones stream them) and any other with the streaming kernel pair.  Stopped after
K iterations every form has to hold the K-th CG iterate: the FP32 recurrences
differ from FP64 by the rounding of x, r and p, amplified by the
orthogonality the CG loses, which at K = 20 stays far below 1e-4 (2**-24 * K
* 50 = 6e-5) relative to the iterate.
"""
import numpy as np
import pytest
import torch

import hfgrid

pytestmark = pytest.mark.gpu
K = 20
DT = 1 / 60


def _markers(res, fill, seed):
    nx, ny, nz = res
    g = torch.Generator().manual_seed(seed)
    mk = torch.zeros((nz, ny, nx), dtype=torch.uint8)
    mk[:, : max(1, int(ny * fill)), :] = 1
    mk[:, :, nx - nx // 8:] = 0
    mk[torch.rand(mk.shape, generator=g) < 0.02] = 2
    mk[torch.rand(mk.shape, generator=g) < 0.02] = 0
    return mk.cuda()


def _cg64(mk, b, h, precond):
    fl, so = mk == 1, mk == 2
    diag = torch.zeros(mk.shape, dtype=torch.float64, device="cuda")
    scale = [DT / (s * s) for s in h]
    for d, s in ((2, scale[0]), (1, scale[1]), (0, scale[2])):
        n = mk.shape[d]
        if n > 1:
            open_ = (~so).double()
            diag.narrow(d, 1, n - 1).add_(s * open_.narrow(d, 0, n - 1))
            diag.narrow(d, 0, n - 1).add_(s * open_.narrow(d, 1, n - 1))
    inv = torch.where(fl & (diag > 0), 1 / diag.clamp_min(1e-300), 0.0) if precond else fl.double()

    def apply(x):
        y = diag * x
        for d, s in ((2, scale[0]), (1, scale[1]), (0, scale[2])):
            n = mk.shape[d]
            if n > 1:
                y.narrow(d, 1, n - 1).sub_(s * x.narrow(d, 0, n - 1))
                y.narrow(d, 0, n - 1).sub_(s * x.narrow(d, 1, n - 1))
        return y * fl

    x, r = torch.zeros_like(diag), b.double() * fl
    z = r * inv
    p, rz = z.clone(), (r * z).sum()
    for _ in range(K):
        q = apply(p)
        a = rz / (p * q).sum()
        x += a * p
        r -= a * q
        z = r * inv
        rz, old = (r * z).sum(), rz
        p = z + (rz / old) * p
    return x


# tile edges (32 x 16 columns), one plane, shares of several short columns,
# shares beyond the register form (more than 148 * 16 planes), and a system
# that does not fit (the streaming pair)
@pytest.mark.parametrize("res,fill", [
    ((31, 15, 9), 1.0), ((32, 16, 8), 1.0), ((33, 17, 40), 1.0), ((5, 3, 2), 1.0), ((70, 50, 1), 1.0),
    ((97, 100, 3), 0.9), ((64, 33, 130), 0.5), ((160, 150, 170), 0.5), ((200, 190, 200), 1.0),
])
@pytest.mark.parametrize("precond", [0, 1])
def test_cg_iterate_vs_fp64(cuda, res, fill, precond):
    h = (1 / 64, 1 / 60, 1 / 70)
    mk = _markers(res, fill, 3)
    g = torch.Generator(device="cuda").manual_seed(5)
    v = [torch.randn(s, generator=g, device="cuda") for s in hfgrid.face_shapes(res)]
    sv = [torch.zeros_like(t) for t in v]
    b = torch.empty(mk.shape, device="cuda")
    hfgrid.op_build_rhs(res, h, v, sv, mk, b)
    p = torch.empty(mk.shape, device="cuda")
    st = hfgrid.op_project(res, h, DT, mk, v, sv, precond=precond, tol_mode=1, tol=1e-30, max_iter=K, p_out=p)
    ref = _cg64(mk, b, [float(np.float32(s)) for s in h], precond)
    assert st["iterations"] == K or st["converged"]
    if not torch.isfinite(ref).all():  # fewer cells than iterations: the FP64 CG has run out of directions
        assert res == (5, 3, 2)
        return
    err = float((p.double() - ref).norm() / ref.norm())
    assert err < 1e-4, err
    assert bool((p[mk != 1] == 0).all())


@pytest.mark.parametrize("res", [(5, 3, 2), (40, 20, 12), (128, 96, 100), (200, 160, 150)])
@pytest.mark.parametrize("precond", [0, 1])
def test_cells_off_the_fluid_stay_zero_when_a_solve_breaks_down(cuda, res, precond):
    """Past an exact solution (a tolerance of 0 asks for more iterations) the CG's
    scalars are 0 / 0: no number comes out at the fluid's cells, but air and
    solid keep pressure 0.  One fluid cell in each quad of four, each a system
    of its own that one iteration solves; 600 iterations are two launches."""
    nx, ny, nz = res
    mk = torch.zeros((nz, ny, nx), dtype=torch.uint8, device=cuda)
    mk[::2, ::2, 1::4] = 1
    v = [torch.zeros(s, device=cuda) for s in hfgrid.face_shapes(res)]
    v[0][::2, ::2, 1::4] = 1.0  # the same inflow into every fluid cell, from its left face
    v[0][:, :, 0] = 0.0
    sv = [torch.zeros_like(t) for t in v]
    for iters in (1, 3, 600):
        p = torch.full(mk.shape, 7.0, device=cuda)
        w = [t.clone() for t in v]
        st = hfgrid.op_project(res, (1 / 8, 1 / 8, 1 / 8), DT, mk, w, sv, precond=precond, tol_mode=1, tol=0.0,
                               max_iter=iters, p_out=p)
        assert st["iterations"] == iters
        assert bool((p[mk == 0] == 0).all())
        if iters == 600:
            assert bool(torch.isnan(p[mk == 1]).any())
