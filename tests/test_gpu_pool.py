"""The contexts' registers, some of which are kept for the next context: contexts
made, stepped and closed by several threads at once give the bits a context
alone gives, and closing large ones gives their memory back down to the bound.
"""
import threading

import numpy as np
import pytest

from tests import _problems as P

pytestmark = pytest.mark.gpu

KEEP = 256 << 20  # devmem.cuh REGISTER_KEEP


def _run(n, out, key, reps):
    from amrvac_b200 import Context, make_cfg
    prim, geo = P.kh_2d(n=n, seed=5)
    blocks = P.to_blocks(P.prim_to_cons(prim, "hd", 2, 1.4), 2)
    for _ in range(reps):
        with Context(make_cfg(physics="hd", ndim=2, gamma=1.4, flux_scheme="hllc", limiter="vanleer")) as ctx:
            ctx.set_uniform_grid(geo["domain_nx"], geo["xprobmin"], geo["xprobmax"])
            ctx.upload(blocks)
            ctx.set_time(0.0, 1.0e99, 0.0)
            ctx.run(4)
            out.setdefault(key, []).append(ctx.download())


def test_threads_share_the_pool():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sizes = (64, 160, 64, 160)
    alone, got = {}, {}
    for n in set(sizes):
        _run(n, alone, n, 1)
    th = [threading.Thread(target=_run, args=(n, got, (i, n), 3)) for i, n in enumerate(sizes)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert len(got) == len(sizes)
    for (_, n), runs in got.items():
        assert len(runs) == 3
        for r in runs:
            assert np.array_equal(r, alone[n][0])


def test_closed_contexts_give_memory_back():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from amrvac_b200 import Context, make_cfg
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    # 1024^2 HD: 32 MB per register, 42 MB with its headroom, three registers,
    # twelve contexts: 1.5 GB, of which the library may hold KEEP already (what
    # earlier contexts left), so at least 1.2 GB > 2 KEEP are new
    ctxs = []
    for _ in range(12):
        c = Context(make_cfg(physics="hd", ndim=2, gamma=1.4, flux_scheme="hllc", limiter="vanleer"))
        c.set_uniform_grid([1024, 1024], [0.0] * 2, [1.0] * 2)
        ctxs.append(c)
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    assert used > 2 * KEEP
    for c in ctxs:
        c.close()
    torch.cuda.synchronize()
    kept = before - torch.cuda.mem_get_info()[0]
    # the bound, and the driver's granularity of a few blocks of 32 MB
    assert kept <= KEEP + (128 << 20), (used, kept)


def test_memory_is_back_when_close_returns():
    """No wait of the caller's after the close."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from amrvac_b200 import Context, make_cfg
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    c = Context(make_cfg(physics="hd", ndim=2, gamma=1.4, flux_scheme="hllc", limiter="vanleer"))
    c.set_uniform_grid([4096, 4096], [0.0] * 2, [1.0] * 2)  # three registers of 671 MB
    c.run(1)
    c.close()
    assert before - torch.cuda.mem_get_info()[0] <= KEEP + (128 << 20)


def test_close_waits_for_other_streams():
    """A stream of the caller's may still read a register (register_ptr)."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from amrvac_b200 import Context, make_cfg
    c = Context(make_cfg(physics="hd", ndim=2, gamma=1.4, flux_scheme="hllc", limiter="vanleer"))
    c.set_uniform_grid([64, 64], [0.0] * 2, [1.0] * 2)
    for act in (lambda: c.set_uniform_grid([128, 128], [0.0] * 2, [1.0] * 2), c.close):
        s, done = torch.cuda.Stream(), torch.cuda.Event()
        with torch.cuda.stream(s):
            torch.cuda._sleep(100_000_000)  # about 50 ms
            done.record()
        assert not done.query()
        act()
        assert done.query()
