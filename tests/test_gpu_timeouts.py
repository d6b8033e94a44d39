"""Bounded waits that run out, part by part: the call ends within a few seconds
with TFHE_GPU_TIMEOUT, and the same context then works.  The waits run out
because a stream is not fed (a flag of the self-test), not by a fault."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _timeout_then(run, check):
    t0 = time.perf_counter()
    st = run()
    assert st == 3, st
    assert time.perf_counter() - t0 < 30
    check()


# one tile with few stages a CTA, both halves of a tile, whole coefficient range in a CTA
@pytest.mark.parametrize("count", [1, 200, 8000])
def test_key_switch_timeout(pkg, torch_cuda, count):
    torch = torch_cuda
    P = pkg.default_params()
    e = pkg.Engine(P)
    try:
        ks = np.random.default_rng(3).integers(-2 ** 31, 2 ** 31, P.ks_words()).astype(np.int32)
        e.upload_keyswitch_key(ks)
        x = torch.randint(-2 ** 31, 2 ** 31, (count, 1025), device="cuda", dtype=torch.int32)
        out = torch.empty((2, count, P.n + 1), device="cuda", dtype=torch.int32)
        sp = torch.cuda.current_stream().cuda_stream
        e.lweKeySwitch(out[0], x, count, stream=sp)
        torch.cuda.synchronize()

        def check():
            e.synchronize()
            e.lweKeySwitch(out[1], x, count, stream=sp)
            torch.cuda.synchronize()
            e.synchronize()
            assert torch.equal(out[0], out[1])

        _timeout_then(lambda: e.selftest_timeout_in("key_switch", count), check)
    finally:
        e.close()


# one-per-CTA split-FP32 kernel: by its own shape, by batch size, in two waves and in the pair kernel's order
@pytest.mark.parametrize("params,shape,count", [("default", 14, 2), ("default", 0, 77), ("stress", 15, 304),
                                                ("default", 0, 230)])
def test_one_per_cta_rotation_timeout(pkg, torch_cuda, params, shape, count):
    torch = torch_cuda
    e = pkg.Engine(pkg.default_params() if params == "default" else pkg.stress_params())
    try:
        e.gate_keyset([9], forms=("split_fp32",), want_bk=False)
        x = torch.randint(-2 ** 31, 2 ** 31, (count, e.params.n + 1), device="cuda", dtype=torch.int32)
        out = torch.empty((2, count, 1025), device="cuda", dtype=torch.int32)
        sp = torch.cuda.current_stream().cuda_stream
        e.set_groups_per_cta("split_fp32", shape)

        def bootstrap(k):
            e.tfhe_bootstrap_woKS_FFT(out[k], x, 1 << 29, count, "split_fp32", stream=sp)
            torch.cuda.synchronize()
            e.synchronize()

        def check():
            bootstrap(1)
            assert torch.equal(out[0], out[1])

        bootstrap(0)
        _timeout_then(lambda: e.selftest_timeout("split_fp32", count), check)
    finally:
        e.close()


# one group; one a group in every SM; the second of two items a group
@pytest.mark.parametrize("params,count", [("default", 1), ("stress", 608), ("default", 1000)])
def test_product_timeout(pkg, torch_cuda, params, count):
    torch = torch_cuda
    e = pkg.Engine(pkg.default_params() if params == "default" else pkg.stress_params())
    try:
        e.gate_keyset([9], forms=("split_fp32",), want_bk=False)
        sp = torch.cuda.current_stream().cuda_stream
        tgsw = torch.randint(-2 ** 31, 2 ** 31, (count, e.params.tgsw_words()), device="cuda", dtype=torch.int32)
        keys = torch.empty(count, e.tgsw_fft_bytes("split_fp32"), device="cuda", dtype=torch.uint8)
        e.tgsw_to_fft(tgsw, keys, count, "split_fp32", stream=sp)
        acc = torch.randint(-2 ** 31, 2 ** 31, (count, 2048), device="cuda", dtype=torch.int32)
        out = [acc.clone(), acc.clone()]

        def product(k):
            e.tGswFFTExternMulToTLwe(out[k], keys, count, "split_fp32", stream=sp)
            torch.cuda.synchronize()
            e.synchronize()

        def check():
            product(1)
            assert torch.equal(out[0], out[1])

        product(0)
        _timeout_then(lambda: e.selftest_timeout_in("product", count), check)
    finally:
        e.close()


# FP64 over two SMs and over eight
@pytest.mark.parametrize("params,shape,count", [("default", 16, 2), ("stress", 0, 60), ("default", 0, 1),
                                                ("stress", 0, 30)])
def test_cluster_timeout(pkg, torch_cuda, params, shape, count):
    torch, form = torch_cuda, "fp64"
    e = pkg.Engine(pkg.default_params() if params == "default" else pkg.stress_params())
    try:
        e.gate_keyset([9], forms=(form,), want_bk=False)
        x = torch.randint(-2 ** 31, 2 ** 31, (count, e.params.n + 1), device="cuda", dtype=torch.int32)
        out = torch.empty((2, count, 1025), device="cuda", dtype=torch.int32)
        e.set_groups_per_cta(form, shape)

        def bootstrap(k):
            e.tfhe_bootstrap_woKS_FFT(out[k], x, 1 << 29, count, form, stream=torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            e.synchronize()

        def check():
            bootstrap(1)
            assert torch.equal(out[0], out[1])

        bootstrap(0)
        _timeout_then(lambda: e.selftest_timeout_in("cluster_fp64", count), check)
    finally:
        e.close()
