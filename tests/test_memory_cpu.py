"""Where a context's memory comes from and goes, on a runtime without a GPU
(tests/fake_cudart.cpp): the waits before registers are given back, full
devices, failing calls."""
import pytest

from tests._fakecuda import Fake

HD2 = dict(physics="hd", ndim=2, gamma=1.4, flux_scheme="hllc", limiter="vanleer")


@pytest.fixture
def fake():
    return Fake()


WAIT = "cudaFree 256 = 0"  # wait_device's allocation: cudaFree waits for all streams of the device


def _first(log, *names):
    """Index of the first call of one of the names on memory, the wait's apart."""
    return next((i for i, l in enumerate(log) if l.split()[0] in names and l.split()[1] not in ("0", "256")), len(log))


def test_registers_are_given_back_behind_a_wait_for_the_device(fake):
    """Work queued on other streams may still read a register (register_ptr):
    the whole device is waited for, also when it is full, before a register is
    freed or used again."""
    h = fake.create(**HD2)
    assert fake.grid(h, [64, 64]) == 0
    for n in (128, 256, 512):
        fake.clear()
        fake.fail("cudaMalloc", times=2)  # a full device: the growth fails further on
        assert fake.grid(h, [n, n]) < 0
        log = fake.log()
        assert log.index(WAIT) < _first(log, "cudaFree", "cudaMalloc"), log
        fake.L.fake_reset()
        assert fake.grid(h, [n, n]) == 0
    fake.clear()
    assert fake.L.amrvac_gpu_destroy(h) == 0
    log = fake.log()
    assert log.index(WAIT) < _first(log, "cudaFree"), log


def test_a_failed_wait_is_reported(fake):
    h = fake.create(**HD2)
    assert fake.grid(h, [64, 64]) == 0
    reg = next(l.split()[1] for l in fake.log() if l.startswith("cudaMalloc") and int(l.split()[1]) > 100000)
    for fn, err in (("cudaFree", 700), ("cudaMalloc", 2)):  # the wait itself, and nothing to wait with
        fake.clear()
        fake.fail(fn, times=9, err=err)
        assert fake.grid(h, [128, 128]) < 0
        assert f"cudaFree {reg} = 0" not in fake.log()  # nothing was given back
        fake.L.fake_reset()
    fake.fail("cudaFree", err=700)
    assert fake.L.amrvac_gpu_destroy(h) < 0
    assert f"cudaFree {reg} = 0" not in fake.log()


def test_the_wait_is_valid_while_another_thread_captures(fake):
    """cudaDeviceSynchronize is an invalid call while any stream of the device
    is being captured."""
    h = fake.create(**HD2)
    assert fake.grid(h, [64, 64]) == 0 and fake.grid(h, [512, 512]) == 0
    assert fake.L.amrvac_gpu_destroy(h) == 0
    assert not [l for l in fake.log() if l.startswith("cudaDeviceSynchronize")]


def test_context_closed_from_another_device(fake):
    """What it allocates to wait is its own device's, and the caller's stays
    current."""
    h = fake.create(**HD2)
    assert fake.grid(h, [64, 64]) == 0
    fake.L.cudaSetDevice(1)
    fake.clear()
    assert fake.L.amrvac_gpu_destroy(h) == 0
    devs = [l.split()[1] for l in fake.log() if l.startswith("cudaSetDevice")]
    assert devs == ["0", "1"] and WAIT in fake.log()


def test_a_failed_allocation_is_reported_once(fake):
    """The runtime's last error goes with the call that reports it: a later
    kernel launch does not report it again."""
    import ctypes
    import numpy as np
    h = fake.create(**HD2)
    assert fake.grid(h, [64, 64]) == 0
    w = np.zeros((16, 4, 1, 20, 20))
    fake.fail("cudaMalloc", times=2)
    assert fake.L.amrvac_gpu_upload(h, 0, 0, 16, w.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) < 0
    assert "out of memory" in fake.error()
    assert fake.L.amrvac_gpu_step_dt(h, 1e-3) == 0, fake.error()


KEEP = 256 << 20  # devmem.cuh REGISTER_KEEP


def test_grown_registers_fit_where_the_old_ones_were(fake):
    """set_blocks on a device that holds the new registers only once the old
    ones are gone."""
    h = fake.create(**HD2)
    assert fake.grid(h, [1600, 1600]) == 0  # 3 x 102 MB
    fake.L.fake_capacity(fake.L.fake_used() + (260 << 20))
    assert fake.grid(h, [2048, 2048]) == 0, fake.error()  # 3 x 168 MB
    assert fake.L.amrvac_gpu_destroy(h) == 0


def test_closed_context_keeps_no_more_than_the_bound(fake):
    """Without any wait of the caller's after the close."""
    for n in (2048, 1024, 512, 2048, 4096):  # one register: 168, 42, 10, 168, 671 MB
        h = fake.create(**HD2)
        assert fake.grid(h, [n, n]) == 0
        used = fake.L.fake_used()
        assert fake.L.amrvac_gpu_destroy(h) == 0
        assert fake.L.fake_used() <= min(KEEP, used)


def test_registers_are_used_again(fake):
    h = fake.create(**HD2)
    assert fake.grid(h, [512, 512]) == 0
    assert fake.L.amrvac_gpu_destroy(h) == 0
    h = fake.create(**HD2)
    fake.clear()
    assert fake.grid(h, [512, 512]) == 0
    assert not [l for l in fake.log() if l.startswith("cudaMalloc") and int(l.split()[1]) > 1 << 20]
    # a much smaller grid does not sit on a large register
    small = fake.create(**HD2)
    assert fake.L.amrvac_gpu_destroy(h) == 0
    fake.clear()
    assert fake.grid(small, [256, 256]) == 0
    assert [l for l in fake.log() if l.startswith("cudaMalloc") and int(l.split()[1]) > 1 << 20]
    assert fake.L.amrvac_gpu_destroy(small) == 0


def test_kept_registers_make_room_for_other_memory(fake):
    """A device that is full but for what the library keeps unused: staging
    buffers, small per-block arrays and ensembles still fit."""
    import ctypes
    import numpy as np
    from amrvac_b200 import _lib, make_cfg
    dp = ctypes.POINTER(ctypes.c_double)

    def keep():
        h = fake.create(**HD2)
        assert fake.grid(h, [1024, 1024]) == 0
        assert fake.L.amrvac_gpu_destroy(h) == 0

    h = fake.create(**HD2)
    assert fake.grid(h, [64, 64]) == 0
    keep()
    fake.L.fake_capacity(fake.L.fake_used())
    w = np.zeros((16, 4, 1, 20, 20))
    assert fake.L.amrvac_gpu_upload(h, 0, 0, 16, w.ctypes.data_as(dp)) == 0, fake.error()
    fake.L.fake_capacity(1 << 40)
    keep()
    fake.L.fake_capacity(fake.L.fake_used())
    inst = (_lib.AmrvacEnsInstance * 1)()
    inst[0].ndim, inst[0].time_max = 2, 1.0
    for d in range(2):
        inst[0].domain_nx[d], inst[0].xprobmax[d] = 64, 1.0
    inst[0].flux_scheme, inst[0].limiter = _lib.FS["hllc"], _lib.LIMITER["vanleer"]
    cfg = make_cfg(physics="hd", ndim=2, gamma=1.4, typeboundary=["cont"] * 4)
    e = ctypes.c_void_p()
    assert fake.L.amrvac_ens_create(ctypes.byref(cfg), 1, inst, ctypes.byref(e)) == 0, fake.error()
    assert fake.L.amrvac_ens_destroy(e) == 0
    assert fake.L.amrvac_gpu_destroy(h) == 0


def test_registers_lost_with_their_device_context_are_not_used_again(fake):
    """cudaDeviceReset between two contexts takes the kept registers away."""
    h = fake.create(**HD2)
    assert fake.grid(h, [512, 512]) == 0
    assert fake.L.amrvac_gpu_destroy(h) == 0
    fake.L.fake_device_reset()
    h = fake.create(**HD2)
    fake.clear()
    assert fake.grid(h, [512, 512]) == 0
    assert len([l for l in fake.log() if l.startswith("cudaMalloc") and int(l.split()[1]) > 1 << 20]) == 3
    fake.clear()
    fake.L.fake_device_reset()
    fake.L.amrvac_gpu_destroy(h)
    # nothing of that size is freed or kept: the addresses may be others' now
    assert not [l for l in fake.log() if l.startswith("cudaFree ") and l.endswith("= 0") and int(l.split()[1]) > 1 << 20]
    h = fake.create(**HD2)
    fake.clear()
    assert fake.grid(h, [512, 512]) == 0
    assert len([l for l in fake.log() if l.startswith("cudaMalloc") and int(l.split()[1]) > 1 << 20]) == 3
    assert fake.L.amrvac_gpu_destroy(h) == 0


def _getdt(fake, h):
    import ctypes
    dt, cm = ctypes.c_double(), ctypes.c_double()
    return fake.L.amrvac_gpu_getdt(h, 0, ctypes.byref(dt), ctypes.byref(cm))


@pytest.mark.parametrize("fn", ["cudaHostAlloc", "cudaHostGetDevicePointer"])
def test_getdt_never_runs_without_its_result_words(fake, fn):
    """They are made with the context, which is refused where they cannot be;
    getdt itself allocates nothing."""
    import ctypes
    from amrvac_b200 import make_cfg
    fake.L.fake_device_reset()  # no page is there yet
    h = ctypes.c_void_p()
    fake.fail(fn)
    cfg = make_cfg(**HD2)
    assert fake.L.amrvac_gpu_create(ctypes.byref(cfg), ctypes.byref(h)) < 0
    fake.L.fake_reset()
    h = fake.create(**HD2)
    assert fake.grid(h, [64, 64]) == 0
    fake.clear()
    fake.fail(fn)
    assert _getdt(fake, h) >= 0 and _getdt(fake, h) >= 0
    assert {l.split()[0] for l in fake.log()} == {"launch", "cudaStreamSynchronize"}
    assert fake.L.amrvac_gpu_destroy(h) == 0


def test_result_words_share_pages(fake):
    """One page for 256 contexts, kept; each context has words of its own."""
    fake.L.fake_device_reset()
    hs = [fake.create(**HD2) for _ in range(257)]
    for h in hs:
        assert fake.L.amrvac_gpu_destroy(h) == 0
    h = fake.create(**HD2)
    assert len([l for l in fake.log() if l.startswith("cudaHostAlloc")]) == 2
    assert not [l for l in fake.log() if l.startswith("cudaFreeHost")]
    assert fake.L.amrvac_gpu_destroy(h) == 0


@pytest.mark.parametrize("after", range(7))
def test_a_failed_growth_leaves_no_blocks(fake, after):
    """Whichever allocation fails, a step is refused instead of launched on
    registers or tables that are not there."""
    fake.L.fake_device_reset()  # no kept registers
    h = fake.create(**HD2)
    assert fake.grid(h, [64, 64]) == 0
    fake.fail("cudaMalloc", after=after, times=99)
    assert fake.grid(h, [128, 128]) < 0
    fake.L.fake_reset()
    assert fake.L.amrvac_gpu_step(h) < 0 and "no blocks set" in fake.error()
    assert not [l for l in fake.log() if l.startswith("launch")]
    assert fake.grid(h, [128, 128]) == 0 and fake.L.amrvac_gpu_step(h) == 0
    assert fake.L.amrvac_gpu_destroy(h) == 0
