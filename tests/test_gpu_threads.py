"""
Host threads with problems of different sizes on one device: a call's settings of a kernel (its shared-memory limit is one
value per function and device) must not reach another thread's launch.

The context's worker handles, streams and events serve one caller at a time, whichever entry point takes them.
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


def _perm_orders(N, ctx, dev):
    from fasterlmm_gb300 import _lib
    from fasterlmm_gb300.core import _ptr, _stream
    cols, out = torch.zeros(1, dtype=torch.int64, device=dev), torch.empty(N, dtype=torch.int32, device=dev)
    return lambda: _lib.call("flmm_perm_orders", _ptr(cols), 1, 1, 1, N, _ptr(out), _stream(dev)), (cols, out)


def _perm_threshold(n, ctx, dev):
    from fasterlmm_gb300 import _lib
    from fasterlmm_gb300.core import _ptr, _stream
    F, out = torch.rand(n, dtype=torch.float64, device=dev), torch.empty(1, dtype=torch.float64, device=dev)
    return lambda: _lib.call("flmm_perm_threshold_p", _ptr(F), 1, n, 100, 0.05, _ptr(out), _stream(dev)), (F, out)


@pytest.mark.parametrize("make,sizes,calls", [(_eigh, (64, 1000), 400), (_eigh, (1320, 1600), 60),
                                              (_prep_variants, (11_000, 50_000), 2000), (_gls_fit, (3200, 9000), 1000),
                                              (_perm_orders, (5000, 16_384), 1000),
                                              (_perm_threshold, (7000, 16_384), 1000)])
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


def test_worker_handles_shared_by_threads():
    """flmm_eigh_many, flmm_eigh_batched on the workers and on one of their handles, from three host threads on one context:
    every decomposition has the bits that it has alone."""
    from fasterlmm_gb300 import _lib, build, core
    build()
    dev = torch.device("cuda", torch.cuda.current_device())
    ctx = _lib.context(dev.index)
    g = torch.Generator(device=dev).manual_seed(1)
    src = [torch.randn(5, n, n, generator=g, device=dev, dtype=torch.float64) for n in (150, 180, 200)]
    src = [x + x.mT for x in src]

    def many(A):
        n, N = A.shape[0], A.shape[1]
        ev = torch.empty(n, N, dtype=torch.float64, device=dev)
        sizes = (_lib.C.c_int * n)(*[N] * n)
        nbytes = _lib.query_bytes("flmm_eigh_many_workspace_bytes", ctx, sizes, n)
        work = torch.empty(nbytes, dtype=torch.uint8, device=dev)
        at = lambda t: (_lib.C.c_void_p * n)(*(x.data_ptr() for x in t))
        _lib.call("flmm_eigh_many", ctx, at(A), sizes, n, at(ev), core._ptr(work), nbytes, core._stream(dev))
        return ev

    def batched(mode, slot):
        def run(A):
            ev = torch.empty(A.shape[0], A.shape[1], dtype=torch.float64, device=dev)
            nbytes = _lib.query_bytes("flmm_eigh_batched_workspace_bytes", ctx, A.shape[1], A.shape[0], mode)
            work = torch.empty(nbytes, dtype=torch.uint8, device=dev)
            _lib.call("flmm_eigh_batched", ctx, core._ptr(A), A.shape[1], A.shape[0], core._ptr(ev), mode, slot,
                      core._ptr(work), nbytes, core._stream(dev))
            return ev
        return run

    calls = [many, batched(2, -1), batched(1, 2)]
    alone = []
    for call, x in zip(calls, src):
        A = x.clone()
        alone.append((call(A), A))
    torch.cuda.synchronize()
    wrong, errors = [], []
    start = threading.Barrier(len(calls))

    def work(k):
        torch.cuda.set_device(dev)
        stream = torch.cuda.Stream()
        try:
            with torch.cuda.stream(stream):
                start.wait()
                for _ in range(20):
                    A = src[k].clone()
                    ev = calls[k](A)
                    stream.synchronize()
                    if not (torch.equal(ev, alone[k][0]) and torch.equal(A, alone[k][1])):
                        wrong.append(k)
        except Exception as e:  # (a thread's failure would otherwise pass unseen)
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and not wrong
