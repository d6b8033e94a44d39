"""Times of calls whose launch rule or work depends on the batch: not slower
than the shapes and batches they are held against.  Each limit lies between
the times with and without the rule."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _median_us(torch, call, calls=1, reps=9):
    stream = torch.cuda.current_stream()
    times = []
    for i in range(reps + 2):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(calls):
            call()
        e1.record(stream)
        torch.cuda.synchronize()
        if i >= 2:
            times.append(e0.elapsed_time(e1) * 1000 / calls)
    return float(np.median(times))


def _engine(pkg, name):
    e = pkg.Engine(pkg.default_params() if name == "default" else pkg.stress_params())
    e.gate_keyset([9], forms=("split_fp32",), want_bk=False)
    return e


def _uniform(torch, *shape):
    return torch.randint(-2 ** 31, 2 ** 31, shape, device="cuda", dtype=torch.int32)


def _bootstrap_us(torch, e, shape, x):
    out = torch.empty((x.shape[0], 1025), dtype=torch.int32, device="cuda")
    sp = torch.cuda.current_stream().cuda_stream
    e.set_groups_per_cta("split_fp32", shape)
    try:
        return _median_us(torch, lambda: e.tfhe_bootstrap_woKS_FFT(out, x, 1 << 29, x.shape[0], "split_fp32",
                                                                   stream=sp))
    finally:
        e.set_groups_per_cta("split_fp32", 0)


def test_two_per_sm_with_two_levels_is_not_slower_than_the_pair_kernel(pkg, torch_cuda):
    """l = 2, up to two ciphertexts per SM: two waves of one per CTA take 5 % longer."""
    torch = torch_cuda
    e = _engine(pkg, "stress")
    try:
        x = _uniform(torch, 300, e.params.n + 1)
        assert _bootstrap_us(torch, e, 0, x) < 1.025 * _bootstrap_us(torch, e, 12, x)
    finally:
        e.close()


# one ciphertext per CTA; a ring whose rows still pass
@pytest.mark.parametrize("count,share", [(152, 0.2), (912, 0.5)])
def test_noiseless_constants_cost_no_steps(pkg, torch_cuda, count, share):
    """Samples with no mask (bootsCONSTANT) rotate by nothing: no step is taken
    and no product or transform is made for them."""
    torch = torch_cuda
    e = _engine(pkg, "default")
    try:
        x = _uniform(torch, count, e.params.n + 1)
        zero = torch.zeros_like(x)
        assert _bootstrap_us(torch, e, 0, zero) < share * _bootstrap_us(torch, e, 0, x)
    finally:
        e.close()


def test_rotation_by_nothing_reads_no_key(pkg, torch_cuda):
    """MuxRotate items with rotation 0 are copies of 8 KB: their 96 KB of key
    rows stay where they are."""
    torch = torch_cuda
    e = pkg.Engine(pkg.default_params())
    try:
        count, sp = 3000, torch.cuda.current_stream().cuda_stream
        keys = torch.empty(count, e.tgsw_fft_bytes("split_fp32"), device="cuda", dtype=torch.uint8)
        e.tgsw_to_fft(_uniform(torch, count, e.params.tgsw_words()), keys, count, "split_fp32", stream=sp)
        acc = _uniform(torch, count, 2048)
        out = torch.empty_like(acc)

        def us(a):
            return _median_us(torch, lambda: e.tfhe_MuxRotate_FFT(out, acc, keys, a, count, "split_fp32", stream=sp),
                              calls=20)

        a = torch.randint(1, 2048, (count,), device="cuda", dtype=torch.int32)
        assert us(torch.zeros_like(a)) < 0.4 * us(a)
        e.tfhe_MuxRotate_FFT(out, acc, keys, torch.zeros_like(a), count, "split_fp32", stream=sp)
        torch.cuda.synchronize()
        assert torch.equal(out, acc)
    finally:
        e.close()
