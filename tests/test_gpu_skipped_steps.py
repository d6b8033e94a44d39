"""MuxRotate batches with items that do not rotate, in any place of a group's
sequence, and blind rotations with steps that a ciphertext does not take (a_i = 0): alone,
in runs across the 32 steps that a warp looks at together, first and last, all
of them; in one or both ciphertexts of a lane pair.  Bit for bit the L2-direct
kernel's accumulators."""
import pytest

pytestmark = pytest.mark.gpu


def _rotations(torch, e, shape, acc, bara):
    acc = acc.clone()
    e.set_groups_per_cta("split_fp32", shape)
    try:
        e.tfhe_blindRotate_FFT(acc, bara, acc.shape[0], "split_fp32", stream=torch.cuda.current_stream().cuda_stream)
        e.synchronize()
        torch.cuda.synchronize()
    finally:
        e.set_groups_per_cta("split_fp32", 0)
    return acc


@pytest.mark.parametrize("params", ["default", "stress"])
@pytest.mark.parametrize("shape,like", [(14, 4), (16, 4), (9, 4), (10, 4), (0, 4)])
def test_steps_not_taken(pkg, torch_cuda, params, shape, like):
    torch = torch_cuda
    e = pkg.Engine(pkg.default_params() if params == "default" else pkg.stress_params())
    try:
        e.gate_keyset([9], forms=("split_fp32",), want_bk=False)
        n, count = e.params.n, 19
        acc = torch.randint(-2 ** 31, 2 ** 31, (count, 2048), device="cuda", dtype=torch.int32)
        bara = torch.randint(1, 2048, (count, n), device="cuda", dtype=torch.int32)
        bara[1] = 0
        bara[2, :40] = 0
        bara[3, 31:33] = 0
        bara[4, -33:] = 0
        bara[5, :-1] = 0
        bara[6:10, 64:128] = 0  # pairs and single ciphertexts of a pair
        bara[10:13, ::3] = 0
        bara[14, 1:] = 0
        bara[15] = 0
        bara[16:, 7] = 0
        assert torch.equal(_rotations(torch, e, shape, acc, bara), _rotations(torch, e, like, acc, bara))
    finally:
        e.close()


# fewer items than SMs; more than one a group of 64 threads
@pytest.mark.parametrize("params,count", [("default", 9), ("default", 1900), ("stress", 1301)])
def test_items_that_do_not_rotate(pkg, torch_cuda, params, count):
    torch = torch_cuda
    e = pkg.Engine(pkg.default_params() if params == "default" else pkg.stress_params())
    try:
        sp = torch.cuda.current_stream().cuda_stream
        keys = torch.empty(count, e.tgsw_fft_bytes("split_fp32"), device="cuda", dtype=torch.uint8)
        tgsw = torch.randint(-2 ** 31, 2 ** 31, (count, e.params.tgsw_words()), device="cuda", dtype=torch.int32)
        e.tgsw_to_fft(tgsw, keys, count, "split_fp32", stream=sp)
        acc = torch.randint(-2 ** 31, 2 ** 31, (count, 2048), device="cuda", dtype=torch.int32)
        a = torch.randint(1, 2048, (count,), device="cuda", dtype=torch.int32)
        full, part = torch.empty_like(acc), acc.clone()
        e.tfhe_MuxRotate_FFT(full, acc, keys, a, count, "split_fp32", stream=sp)
        still = torch.rand(count, device="cuda") < 0.5
        still[:2], still[-1] = True, True
        e.tfhe_MuxRotate_FFT(part, part, keys, torch.where(still, torch.zeros_like(a), a), count, "split_fp32",
                             stream=sp)
        torch.cuda.synchronize()
        e.synchronize()
        assert torch.equal(part, torch.where(still[:, None], acc, full))
    finally:
        e.close()
