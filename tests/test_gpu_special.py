"""Operands that are not numbers: how far a NaN cell, and one of negative
pressure, reaches in one stage.  The
limiters that ignore a NaN difference (minmod) reach one cell, those that carry
it two; the compiled-in limiters as the run-time ones and as the oracle.
"""
import numpy as np
import pytest

from tests import _problems as P

pytestmark = pytest.mark.gpu

N = 32
DT = 1e-3


def _blocks(physics, ndim, value):
    ndir = 3 if physics == "mhd" else ndim
    kw = dict(glm=True) if physics == "mhd" else {}
    prim = np.array(P.random_smooth(physics, ndim, ndir, N, **kw))
    b = P.to_blocks(P.prim_to_cons(prim, physics, ndir, 1.4 if physics == "hd" else 5.0 / 3.0), ndim)
    b[0, ndir + 1, 2 + 8 if ndim == 3 else 0, 2 + 7, 2 + 7] = value  # the energy of one cell
    return b


def _bad(physics, ndim, value, precision="fp64", **kw):
    """Cells that one stage leaves non-finite."""
    from amrvac_b200 import Context, make_cfg
    if physics == "mhd":
        kw.update(ndir=3, typedivbfix="glm")
    with Context(make_cfg(physics=physics, ndim=ndim, gamma=1.4 if physics == "hd" else 5.0 / 3.0, precision=precision,
                          **kw)) as c:
        c.set_uniform_grid([N] * ndim, [0.0] * ndim, [1.0] * ndim)
        c.upload(_blocks(physics, ndim, value))
        c.set_cmax_global(1.0)
        c.advect1("ps", "ps1", 1.0, DT)
        return ~np.isfinite(P.interior(c.download("ps1"), ndim)).all(axis=1)


def _bad_oracle(O, physics, ndim, value, **kw):
    if physics == "mhd":
        kw.update(ndir=3, divb="glm")
    g = O.Grid(O.make_cfg(physics=physics, ndim=ndim, gamma=1.4 if physics == "hd" else 5.0 / 3.0, **kw), [N] * ndim,
               [0.0] * ndim, [1.0] * ndim, ["periodic"] * (2 * ndim))
    for ib, w in enumerate(_blocks(physics, ndim, value)):
        g.set_block(ib, w)
    g.getbc()
    L = O.lib()
    L.orc_grid_copy_reg(g.h, 1, 0)
    L.orc_grid_advect1(g.h, 1, 0, DT, 1.0, 1.0, 0)
    out = P.interior(np.array([g.get_block(ib) for ib in range(g.nblocks)]), ndim)
    return ~np.isfinite(out).all(axis=1)


def _cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("physics,ndim,fs,limiter", [
    ("hd", 2, "hll", "minmod"), ("hd", 2, "tvdlf", "minmod"), ("hd", 2, "hllc", "vanleer"), ("hd", 2, "hll", "cada3"),
    ("hd", 2, "hll", "koren"), ("hd", 3, "hllc", "vanleer"), ("hd", 3, "hll", "minmod"), ("mhd", 3, "hll", "minmod")])
def test_nan_reaches_as_far_as_in_the_oracle(oracle_lib, physics, ndim, fs, limiter):
    _cuda()
    kw = dict(flux_scheme=fs, limiter=limiter)
    assert np.array_equal(_bad(physics, ndim, np.nan, **kw), _bad_oracle(oracle_lib, physics, ndim, np.nan, **kw))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ndim", [2, 3])
def test_nan_in_hlld(ndim, precision):
    """HLLD, whose flux takes a NaN speed to one side: cada3 and vanleer carry
    a NaN difference alike, minmod ignores it."""
    _cuda()
    kw = dict(precision=precision, flux_scheme="hlld")
    bad = {lim: _bad("mhd", ndim, np.nan, limiter=lim, **kw) for lim in ("cada3", "vanleer", "minmod")}
    assert np.array_equal(bad["cada3"], bad["vanleer"])
    assert bad["minmod"].sum() < bad["vanleer"].sum()


@pytest.mark.parametrize("physics,ndim,fs,limiter", [
    ("hd", 2, "hllc", "vanleer"), ("hd", 2, "hll", "minmod"), ("hd", 2, "tvdlf", "minmod"), ("hd", 3, "hllc", "vanleer")])
def test_negative_pressure_is_not_passed_over(oracle_lib, physics, ndim, fs, limiter):
    """The signal speeds' root of a negative number is NaN, as in the oracle;
    an infinity of either sign would choose one side's flux."""
    _cuda()
    kw = dict(flux_scheme=fs, limiter=limiter)
    bad = _bad_oracle(oracle_lib, physics, ndim, -5.0, **kw)
    assert bad.any()
    assert np.array_equal(_bad(physics, ndim, -5.0, **kw), bad)
