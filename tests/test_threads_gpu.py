"""Two host threads, each with its context and stream, run calls of different sizes through
the same kernels: neither's launch configuration disturbs the other's."""
import ctypes as C
import threading

import pytest
import torch

from openholo_gb300 import Context, _lib

pytestmark = pytest.mark.gpu


def conv(ctx, st, h, w, cin, cout):
    x = torch.ones((1, h, w, cin), dtype=torch.bfloat16, device="cuda")
    wt = torch.ones((cout, 9 * cin), dtype=torch.bfloat16, device="cuda")
    out = torch.empty((1, h, w, cout), dtype=torch.bfloat16, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    return lambda: _lib.call("oh_conv2d_bf16", ctx.handle, 9, 1, 1, h, w, cin, cout, p(x), cin, p(wt), None, 0, None, 0,
                             p(out), cout, C.c_void_p(st.cuda_stream)), out, 9 * cin


def ssb(ctx, st, n, m):
    u = torch.ones((m, n), dtype=torch.complex64, device="cuda")
    out = torch.empty((m, n), device="cuda")
    return lambda: _lib.call("oh_encode", ctx.handle, 0, 5, n, m, C.c_void_p(u.data_ptr()), C.c_void_p(out.data_ptr()),
                             C.c_void_p(st.cuda_stream)), None, None


@pytest.mark.parametrize("make,a,b", [(conv, (16, 256, 32, 256), (64, 256, 64, 32)), (ssb, (16384, 2), (256, 2))])
def test_two_threads(lib_built, make, a, b):
    errors = []

    def work(sizes):
        ctx, st = Context(0), torch.cuda.Stream()
        try:
            with torch.cuda.stream(st):
                run, out, inner = make(ctx, st, *sizes)
                for _ in range(20000):
                    run()
                st.synchronize()
                if out is not None and out.shape[1] > 2:      # all ones: 9 cin inside the image
                    assert float(out[0, 1, 1, 0]) == inner
        except Exception as e:      # noqa: BLE001 (reported by the main thread)
            errors.append(e)
        finally:
            st.synchronize()
            ctx.close()

    ts = [threading.Thread(target=work, args=(s,)) for s in (a, b)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
