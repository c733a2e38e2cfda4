"""cada3's blending band in the stage kernels that have the limiter compiled in
(3-D and 2.5-D MHD HLLD): their face loop leaves a face near the band to a
recomputation.

The density's increments along one axis are 3d, d, -3d, -d, with d a power of two
(exact differences), so both slopes of every face have d0^2 + d1^2 = 10 d^2, and
cada3_radius puts 10 d^2 / (radius dx)^2 at 1: the middle of the 2e-14 wide band,
where the slope is the mean of the asymptotic and the limited form.  One rounding
there moves the mean by 2^-53 / 2e-14 = 0.6 % of their difference; up to eight of
them (squares, sum, reciprocal, product) are allowed, 5 %.
"""
import numpy as np
import pytest

from tests import _problems as P

pytestmark = pytest.mark.gpu

N = 32
D = 2.0 ** -8


def _blocks(ndim, axis):
    step = np.cumsum(np.tile([3.0, 1.0, -3.0, -1.0], N // 4)) * D
    prim = np.zeros((9, N if ndim == 3 else 1, N, N))
    shape = [1, 1, 1]
    shape[2 - axis] = N
    prim[0] = 1.0 + step.reshape(shape)
    for c, v in enumerate((0.5, 0.25, 0.125)):
        prim[1 + c] = v
        prim[5 + c] = 0.5 * v
    prim[4] = 1.0
    return P.to_blocks(P.prim_to_cons(prim, "mhd", 3, 5.0 / 3.0), ndim)


def _radius(shift):
    return float(np.sqrt(10.0)) * D * N * (1.0 + shift)


def _oracle(O, ndim, blocks, shift, dt):
    c = O.make_cfg(physics="mhd", ndim=ndim, ndir=3, flux_scheme="hlld", limiter="cada3", divb="glm",
                   cada3_radius=_radius(shift))
    g = O.Grid(c, [N] * ndim, [0.0] * ndim, [1.0] * ndim, ["periodic"] * (2 * ndim))
    for ib in range(g.nblocks):
        g.set_block(ib, blocks[ib])
    g.getbc()
    L = O.lib()
    L.orc_grid_copy_reg(g.h, 1, 0)
    L.orc_grid_advect1(g.h, 1, 0, dt, 1.0, 1.0, 0)
    return P.interior(np.array([g.get_block(ib) for ib in range(g.nblocks)]), ndim)


@pytest.mark.parametrize("ndim,axis", [(3, 0), (3, 1), (3, 2), (2, 0), (2, 1)])
def test_faces_in_the_blending_band(oracle_lib, ndim, axis):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from amrvac_b200 import Context, make_cfg
    dt = 5e-3
    blocks = _blocks(ndim, axis)
    got = {}
    for shift in (-1e-9, 0.0, 1e-9):
        with Context(make_cfg(physics="mhd", ndim=ndim, ndir=3, flux_scheme="hlld", limiter="cada3", typedivbfix="glm",
                              cada3_radius=_radius(shift))) as c:
            c.set_uniform_grid([N] * ndim, [0.0] * ndim, [1.0] * ndim)
            c.upload(blocks)
            c.set_cmax_global(1.0)
            assert c.advect1("ps", "ps1", 1.0, dt) == 0
            got[shift] = P.interior(c.download("ps1"), ndim)[:, 0]
    ref = {s: _oracle(oracle_lib, ndim, blocks, s, dt)[:, 0] for s in got}
    width = np.abs(ref[1e-9] - ref[-1e-9]).max()  # asymptotic against limited
    assert width > 1e-6
    for s in (-1e-9, 1e-9):
        assert np.abs(got[s] - ref[s]).max() <= 1e-12
    assert np.abs(got[0.0] - ref[0.0]).max() <= 0.05 * width
    # it is the blend: neither of the two forms
    assert np.abs(ref[0.0] - ref[1e-9]).max() > 0.2 * width and np.abs(ref[0.0] - ref[-1e-9]).max() > 0.2 * width
