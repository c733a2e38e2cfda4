"""Where a context's memory comes from and goes, on a runtime without a GPU
(tests/fake_cudart.cpp): the waits before registers are given back, full
devices, failing calls."""
import pytest

from tests._fakecuda import Fake

HD2 = dict(physics="hd", ndim=2, gamma=1.4, flux_scheme="hllc", limiter="vanleer")


@pytest.fixture
def fake():
    return Fake()


def _first(log, *names):
    return next((i for i, l in enumerate(log) if l.split()[0] in names), len(log))


def test_registers_are_given_back_behind_a_wait_for_the_device(fake):
    """Work queued on other streams may still read a register (register_ptr):
    the whole device is waited for, also when it is full, before a register is
    freed, and a failed wait is reported."""
    h = fake.create(**HD2)
    assert fake.grid(h, [64, 64]) == 0
    fake.clear()
    fake.fail("cudaMalloc")  # a full device: the growth below fails further on
    fake.grid(h, [128, 128])
    log = fake.log()
    wait = log.index("cudaDeviceSynchronize 0 = 0")
    assert wait < _first(log, "cudaFree", "cudaFreeAsync", "cudaMalloc", "cudaMallocFromPoolAsync"), log
    fake.L.fake_reset()
    assert fake.grid(h, [128, 128]) == 0
    fake.clear()
    assert fake.L.amrvac_gpu_destroy(h) == 0
    log = fake.log()
    assert log.index("cudaDeviceSynchronize 0 = 0") < _first(log, "cudaFree", "cudaFreeAsync"), log


def test_a_failed_wait_is_reported(fake):
    h = fake.create(**HD2)
    assert fake.grid(h, [64, 64]) == 0
    fake.clear()
    fake.fail("cudaDeviceSynchronize", err=700)
    assert fake.grid(h, [128, 128]) < 0
    assert _first(fake.log(), "cudaFree", "cudaFreeAsync") == len(fake.log())  # nothing was given back
    fake.fail("cudaDeviceSynchronize", err=700)
    assert fake.L.amrvac_gpu_destroy(h) < 0


def test_context_closed_from_another_device(fake):
    """Its own device is waited for, and the caller's stays current."""
    h = fake.create(**HD2)
    assert fake.grid(h, [64, 64]) == 0
    fake.L.cudaSetDevice(1)
    fake.clear()
    assert fake.L.amrvac_gpu_destroy(h) == 0
    assert "cudaDeviceSynchronize 0 = 0" in fake.log()
    assert [l for l in fake.log() if l.startswith("cudaSetDevice")][-1].split()[1] == "1"


def test_a_failed_allocation_is_reported_once(fake):
    """The runtime's last error goes with the call that reports it: a later
    kernel launch does not report it again."""
    import ctypes
    import numpy as np
    h = fake.create(**HD2)
    assert fake.grid(h, [64, 64]) == 0
    w = np.zeros((16, 4, 1, 20, 20))
    fake.fail("cudaMalloc")
    assert fake.L.amrvac_gpu_upload(h, 0, 0, 16, w.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) < 0
    assert "out of memory" in fake.error()
    assert fake.L.amrvac_gpu_step_dt(h, 1e-3) == 0, fake.error()
