"""
Host threads with problems of different sizes on one device: a call's settings of a kernel (its shared-memory limit is one
value per function and device) must not reach another thread's launch.
"""
from __future__ import annotations

import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _eigh(N, ctx, dev):
    from fasterlmm_gb300 import _lib
    from fasterlmm_gb300.core import _ptr, _stream
    A = torch.randn(N, N, device=dev)
    A = A + A.T
    U = torch.empty_like(A)
    ev = torch.empty(N, device=dev)
    nbytes = _lib.query_bytes("flmm_eigh_batched_f32_workspace_bytes", ctx, N, 1)
    work = torch.empty(nbytes, dtype=torch.uint8, device=dev)
    return lambda: _lib.call("flmm_eigh_batched_f32", ctx, _ptr(U.copy_(A)), N, 1, _ptr(ev), _ptr(work), nbytes,
                             _stream(dev)), (A, U, ev, work)


def _prep_variants(N, ctx, dev):
    from fasterlmm_gb300 import _lib
    from fasterlmm_gb300.core import _ptr, _stream
    k, M = 8, 4
    z = lambda *s, dtype=torch.float32: torch.zeros(*s, dtype=dtype, device=dev)
    ld, ld2 = (k + N + 7) // 8 * 8, (k + 8) // 8 * 8
    t = [z(M, k), z(M, N, dtype=torch.float64), z(M, N), z(M, ld, dtype=torch.float16), z(M, ld, dtype=torch.float16), z(M),
         z(M, ld2, dtype=torch.float16), z(M, ld2, dtype=torch.float16), z(M)]
    us, zt, ct, b1h, b1l, s1, b2h, b2l, s2 = map(_ptr, t)
    return lambda: _lib.call("flmm_lr_prep_variants", us, k, zt, N, ct, N, M, k, N, None, 0, 0, b1h, b1l, ld, s1, b2h, b2l,
                             ld2, s2, _stream(dev)), t


def _gls_fit(N, ctx, dev):
    from fasterlmm_gb300 import _lib
    from fasterlmm_gb300.core import _ptr, _stream
    rn = lambda *s: torch.randn(*s, dtype=torch.float64, device=dev)
    s, X, Y, ld = rn(N).abs(), rn(1, N), rn(1, N), rn(1)
    idx = torch.empty(1, dtype=torch.int32, device=dev)
    nbytes = _lib.query_bytes("flmm_fit_delta_gls_workspace_bytes", N, 1, 1, 4)
    work = torch.empty(nbytes, dtype=torch.uint8, device=dev)
    return lambda: _lib.call("flmm_fit_delta_gls_f64", _ptr(s), N, _ptr(X), N, 1, _ptr(Y), N, 1, 4, -1.0, 1.0, 1, 0, _ptr(ld),
                             _ptr(idx), _ptr(work), nbytes, _stream(dev)), (s, X, Y, ld, idx, work)


@pytest.mark.parametrize("make,sizes,calls", [(_eigh, (64, 1000), 400), (_eigh, (1320, 1600), 60),
                                              (_prep_variants, (11_000, 50_000), 2000), (_gls_fit, (3200, 9000), 1000)])
def test_two_sizes_at_once(make, sizes, calls):
    from fasterlmm_gb300 import _lib, build
    build()
    dev = torch.device("cuda", torch.cuda.current_device())
    ctx = _lib.context(dev.index)
    jobs = [make(N, ctx, dev) for N in sizes]
    torch.cuda.synchronize()
    errors = []
    start = threading.Barrier(len(jobs))

    def work(job):
        torch.cuda.set_device(dev)
        with torch.cuda.stream(torch.cuda.Stream()):
            start.wait()
            for k in range(calls):
                try:
                    job()
                except _lib.FlmmError as e:
                    errors.append(str(e))
                    return
                if k % 64 == 63:
                    torch.cuda.current_stream().synchronize()
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(j[0],)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
