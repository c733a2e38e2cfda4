"""Which build of the stage kernels a context launches and with how many CTAs, on
a runtime without a GPU (tests/fake_cudart.cpp): from the launches it logs
("launch <CTAs> x <threads>")."""
import pytest

from tests._fakecuda import Fake

HD2 = dict(physics="hd", ndim=2, gamma=1.4)


@pytest.fixture
def fake():
    return Fake()


def _launches(fake, n, **kw):
    """(CTAs, threads) of a step's kernels after getdt's."""
    h = fake.create(**HD2, **kw)
    assert fake.grid(h, list(n)) == 0, fake.error()
    fake.clear()
    assert fake.L.amrvac_gpu_step(h) == 0, fake.error()
    out = [(int(l.split()[1]), int(l.split()[3])) for l in fake.log() if l.startswith("launch")]
    assert fake.L.amrvac_gpu_destroy(h) == 0
    return out[1:]


@pytest.mark.parametrize("bn,threads,per_sm", [(8, 64, 8), (10, 128, 4), (12, 160, 3), (16, 256, 2)])
def test_predictor_fills_the_device(fake, bn, threads, per_sm):
    """MUSCL-Hancock predictor: one wave of its own CTAs, not of another block
    edge's; per_sm of them are what its registers are capped for."""
    kw = dict(flux_scheme="tvdlf", limiter="koren", time_stepper="twostep", block_nx=bn)
    (ctas, t), _ = _launches(fake, (128 * bn, 64 * bn), **kw)
    assert t == threads and ctas >= 148 * per_sm


@pytest.mark.parametrize("sms", [20, 148])
def test_builds_follow_the_devices_size(fake, sms):
    """A thread per face (576) up to a tile per SM."""
    kw = dict(flux_scheme="hllc", limiter="vanleer")
    fake.L.fake_sms(sms)
    assert {t for _, t in _launches(fake, (16 * sms, 16), **kw)} == {576}
    assert {t for _, t in _launches(fake, (16 * sms + 16, 16), **kw)} == {256}


@pytest.mark.parametrize("tiles", [1, 148, 149, 296, 297])
def test_stage_variant_reports_what_runs(fake, tiles):
    import ctypes
    h = fake.create(**HD2, flux_scheme="hllc", limiter="vanleer")
    assert fake.grid(h, [16 * tiles, 16]) == 0
    fake.clear()
    assert fake.L.amrvac_gpu_step(h) == 0
    ran = {int(l.split()[3]) for l in fake.log()[1:] if l.startswith("launch")}
    v = [ctypes.c_int() for _ in range(5)]
    assert fake.L.amrvac_gpu_stage_variant(h, *[ctypes.byref(x) for x in v]) == 0
    assert ran == {v[2].value}
    assert v[3].value == (1 if tiles <= 148 else 2 if tiles <= 296 else 4)
    assert fake.L.amrvac_gpu_destroy(h) == 0
