"""Mixed 3-D MHD HLLD + vanleer + GLM (the FP32 star states from the primitive
face states, and their FP64 repair) against the FP64 form: a smooth state and a
strong blast with a nearly unmagnetised, nearly pressureless ambient, on a
uniform grid and on one with level jumps.

Bar: an FP32 face value is off by a few 2^-24 of the largest term of its flux,
which the state takes in as dt/dx times that, once a stage.  Per variable the
difference is bounded by STEPS * 3 stages * 6 faces * 8 * 2^-24 = 1.7e-4 of the
variable's scale (its maximum over the grid, for momenta and field that of the
whole vector); measured 1e-7 (smooth) and 3e-6 (blast).
"""
import numpy as np
import pytest

from tests import _amr as A
from tests import _problems as P

pytestmark = pytest.mark.gpu

STEPS = 20
BAR = STEPS * 3 * 6 * 8 * 2.0 ** -24


def _cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _field(strong):
    def f(X, Y, Z):
        out = np.zeros((9,) + X.shape)
        r = np.sqrt((X - 0.5) ** 2 + (Y - 0.5) ** 2 + (Z - 0.5) ** 2)
        if strong:  # p ratio 1e5; the field vanishes on planes of cells
            out[0] = np.where(r < 0.2, 1.0, 0.1)
            out[4] = np.where(r < 0.2, 10.0, 1.0e-4)
            out[5] = 0.1 * np.where(X < 0.5, 1.0, 0.0)
        else:
            out[0] = 1.0 + 0.3 * np.sin(2 * np.pi * (X + Y)) * np.cos(2 * np.pi * Z)
            for c in range(3):
                out[1 + c] = 0.3 * np.cos(2 * np.pi * (X + (c + 1) * Y - Z))
                out[5 + c] = 0.4 + 0.2 * np.sin(2 * np.pi * ((X, Y, Z)[(c + 1) % 3]))
            out[4] = 1.0 + 0.2 * np.sin(2 * np.pi * (Z - X))
        return out
    return f


def _run(precision, strong, jumps):
    from amrvac_b200 import Context, make_cfg
    with Context(make_cfg(physics="mhd", ndim=3, ndir=3, flux_scheme="hlld", limiter="vanleer", typedivbfix="glm",
                          courantpar=0.4, precision=precision)) as c:
        if jumps:
            leaves = A.build_leaves(3, [4] * 3, 2, lambda x, lv: np.linalg.norm(x - 0.5) < 0.3)
            c.set_amr_grid(leaves, [4] * 3, [0.0] * 3, [1.0] * 3)
        else:
            leaves = [(2, i, j, k) for k in range(2) for j in range(2) for i in range(2)]
            c.set_uniform_grid([32] * 3, [0.0] * 3, [1.0] * 3)
        nb = [4] * 3 if jumps else [1] * 3
        c.upload(A.fill_blocks(leaves, 3, nb, _field(strong), "mhd", 3, 5.0 / 3.0))
        c.set_time(0.0, 1.0e99, 0.0)
        c.run(STEPS)
        assert c.status() == 0
        return P.interior(c.download(), 3), c.get_time()[1]


@pytest.mark.parametrize("jumps", [False, True])
@pytest.mark.parametrize("strong", [False, True])
def test_mixed_vanleer_against_fp64(strong, jumps):
    _cuda()
    (ref, cg), (got, _) = _run("fp64", strong, jumps), _run("mixed", strong, jumps)
    assert np.isfinite(got).all()
    for v in (slice(0, 1), slice(1, 4), slice(4, 5), slice(5, 8), slice(8, 9)):
        scale = np.abs(ref[:, v]).max() if v.start < 8 else cg * np.abs(ref[:, 5:8]).max()
        err = np.abs(got[:, v] - ref[:, v]).max() / scale
        assert err <= BAR, (v, err)
    if not jumps:  # FP64 accumulation conserves mass
        assert abs(got[:, 0].sum() - ref[:, 0].sum()) <= 1e-12 * ref[:, 0].sum()
