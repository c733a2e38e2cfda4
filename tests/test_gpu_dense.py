"""The builds of the FP64 2-D hydrodynamics stage kernel (a thread per face up
to 148 tiles at block edge 16, two CTAs per SM up to 296 tiles, four above) on
both sides of those lines, at block edges 16 and 32 (four tiles per block), and
at 8, 10 and 12 (lines at 1184, 592 and 444 tiles: eight, four and three CTAs
per SM), against the oracle: one full step, cell by cell
(tests/_parity.py; bar 1e-12), with the persistent distribution and with one
tile per CTA.
"""
import numpy as np
import pytest

from tests import _problems as P
from tests._parity import percell_err

pytestmark = pytest.mark.gpu

RTOL = 1e-12


@pytest.mark.parametrize("bn,nb", [(16, (1, 1)), (16, (37, 4)), (16, (1, 149)), (16, (17, 17)), (16, (37, 8)), (16, (11, 27)), (32, (2, 37)), (32, (5, 15)),
                                   (8, (34, 34)), (8, (35, 34)), (10, (37, 16)), (10, (37, 17)), (12, (37, 12)), (12, (37, 13))])
@pytest.mark.parametrize("kw", [dict(flux_scheme="hllc", limiter="vanleer"), dict(flux_scheme="hll", limiter="minmod"),
                                dict(flux_scheme="tvdlf", limiter="koren", time_stepper="twostep")])
def test_every_build_matches_oracle(oracle_lib, bn, nb, kw):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from amrvac_b200 import Context, make_cfg
    O = oracle_lib
    nx, ny = bn * nb[0], bn * nb[1]
    ocfg = O.make_cfg(physics="hd", ndim=2, gamma=1.4, block_nx=bn, **kw)
    y, x = np.meshgrid((np.arange(ny) + 0.5) / ny, (np.arange(nx) + 0.5) / nx, indexing="ij")
    prim = np.zeros((4, 1, ny, nx))
    prim[0, 0] = 1.0 + 0.3 * np.sin(2 * np.pi * (x + 2 * y))
    prim[1, 0] = 0.4 * np.cos(2 * np.pi * (2 * x - y))
    prim[2, 0] = 0.3 * np.sin(2 * np.pi * (x - 3 * y))
    prim[3, 0] = 1.0 + 0.2 * np.cos(2 * np.pi * (3 * x + y))
    blocks = P.to_blocks(P.prim_to_cons(prim, "hd", 2, 1.4), 2, bn=bn)
    og = O.Grid(ocfg, [nx, ny], [0.0] * 2, [1.0, 1.3], ["periodic"] * 4)
    for ib in range(og.nblocks):
        og.set_block(ib, blocks[ib])
    og.getbc()
    dt, cg = og.getdt()
    og.advance(dt, cg)
    ref = P.interior(np.array([og.get_block(ib) for ib in range(og.nblocks)]), 2)
    ctx = Context(make_cfg(physics="hd", ndim=2, gamma=1.4, block_nx=bn, **kw))
    ctx.set_uniform_grid([nx, ny], [0.0] * 2, [1.0, 1.3])
    for z in (0, bn):
        ctx.set_zchunk(z)
        ctx.upload(blocks)
        ctx.set_time(0.0, 1.0e99, 0.0)
        ctx.step()
        assert percell_err(P.interior(ctx.download(), 2), ref) <= RTOL, z
    assert ctx.status() == 0
