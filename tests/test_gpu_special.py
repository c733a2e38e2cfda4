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


def _block_hd2(value=None):
    """A 64^2 state, the energy of cell (20, 20) set to value."""
    prim = np.array(P.random_smooth("hd", 2, 2, 64))
    cons = P.prim_to_cons(prim, "hd", 2, 1.4)
    if value is not None:
        cons[3, 0, 20, 20] = value
    return cons


@pytest.mark.parametrize("value", [np.inf, np.nan, 0.0, 1e-310])
@pytest.mark.parametrize("fs,limiter", [("hll", "minmod"), ("hllc", "vanleer")])
def test_adjoint_beside_a_special_operand(fs, limiter, value):
    """One adjoint step: cells that the state's special cell (infinite, NaN, no
    energy, subnormal) does not reach get the gradient they get without it, bit
    for bit; a value that is not a number is not passed over."""
    _cuda()
    import torch
    from amrvac_b200.adjoint import blocks_to_domain, domain_to_blocks, solve
    lam = torch.from_numpy(np.random.default_rng(3).standard_normal((4, 64, 64))).cuda()
    grad = []
    for v in (None, value):
        u = domain_to_blocks(torch.from_numpy(_block_hd2(v)[:, 0]).cuda()).requires_grad_(True)
        g = torch.tensor(1.4, dtype=torch.float64, device="cuda", requires_grad=True)
        un = solve(u, g, np.array([1e-3]), (64, 64), (0.0, 0.0), (1.0, 1.0), limiter=limiter, flux_scheme=fs)
        d = blocks_to_domain(un, 64, 64)
        w = lam.clone()
        w[:, 12:29, 12:29] = 0.0  # the loss does not see what the cell reaches forward
        d = torch.where(w == 0.0, torch.zeros_like(d), d)
        (d * w).sum().backward()
        grad.append(blocks_to_domain(u.grad, 64, 64).cpu().numpy())
    far = np.ones((64, 64), bool)
    far[4:37, 4:37] = False  # six cells a step forward, as many back
    assert np.array_equal(grad[0][:, far], grad[1][:, far])
    assert np.isfinite(grad[0]).all()


@pytest.mark.parametrize("value", [np.nan, 0.0, 1e-310])
def test_ensemble_beside_a_special_operand(value):
    """FP64 ensembles repeat a face that met a special operand with the guarded
    forms, as the single-grid kernel does: the same bits, and the instances
    beside it do not notice."""
    _cuda()
    from amrvac_b200 import Context, Ensemble, Instance, make_cfg
    kw = dict(physics="hd", ndim=2, gamma=1.4, typeboundary=["cont"] * 4, typeboundspeed="cmaxleftright")
    states = [P.to_blocks(_block_hd2(v), 2) for v in (None, value, None)]
    inst = [Instance(2, (64, 64), flux_scheme="hllc", limiter="vanleer", time_max=1.0) for _ in states]
    ens = Ensemble(make_cfg(**kw), inst)
    for i, w in enumerate(states):
        ens.upload(i, w)
    ens.step()
    out = [P.interior(ens.download(i), 2) for i in range(3)]
    ens.close()
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[2])
    with Context(make_cfg(flux_scheme="hllc", limiter="vanleer", **kw)) as c:
        c.set_uniform_grid([64, 64], [0.0] * 2, [1.0] * 2)
        c.upload(states[1])
        c.set_time(0.0, 1.0, 0.0)
        c.step()
        ref = P.interior(c.download(), 2)
    assert np.array_equal(np.isfinite(out[1]), np.isfinite(ref))
    m = np.isfinite(ref)
    assert np.abs(out[1][m] - ref[m]).max() <= 1e-12 * np.abs(ref[m]).max()
