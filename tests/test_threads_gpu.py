"""Contexts on different host threads share the kernels, not their launch state."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMOOTH = dict(gradient_smooth=1, main_range=1, x_range=1, y_range=1, z_range=1)


def test_two_contexts_on_two_threads(built_lib, monkeypatch):
    """Two threads, each with its own context and stream, launch the same kernels with
    different shared memory sizes (element type, row alignment, gradient ranges):
    every call succeeds and gives what it gives alone."""
    import torch
    from rfba_gb300 import srrf
    monkeypatch.setenv("RFBA_GRAPH", "0")  # a replayed graph launches with the size it was captured with
    rng = np.random.default_rng(8)
    big = dict(SMOOTH, x_range=3, y_range=3, z_range=3, main_range=3)
    jobs = [(dict(mag=2, method=1, **SMOOTH), (2, 8, 8, 9), np.uint16),
            (dict(mag=2, method=1, **big), (2, 8, 8, 8), np.float32)]
    calls, errors = 400, []
    start = threading.Barrier(len(jobs))

    def work(kw, shape, dtype):
        try:
            x = rng_x[dtype].astype(dtype)
            cfg = srrf.Config.make(**kw)
            ctx, stream = srrf.Context(0), torch.cuda.Stream()
            with torch.cuda.stream(stream):
                xd = torch.from_numpy(x.view(np.int16) if dtype == np.uint16 else x).cuda()
                xf = torch.from_numpy(x.astype(np.float32)).cuda()
                g = torch.ones(tuple(s * 2 for s in shape[1:]), device="cuda")
                first = ctx.forward(cfg, xd).clone()
                start.wait()
                for i in range(calls):
                    m = ctx.forward(cfg, xd)
                    if i % 8 == 0:
                        ctx.backward(cfg, xf, None, g)
                stream.synchronize()
                assert torch.equal(torch.nan_to_num(m, nan=-7.0), torch.nan_to_num(first, nan=-7.0))
            ctx.close()
        except Exception as e:  # noqa: BLE001 - handed to the main thread
            errors.append(repr(e))
            start.abort()

    rng_x = {d: rng.integers(90, 700, s) for _, s, d in jobs}
    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
