"""FP64 ciphertexts do not depend on the batch: the kernels that the automatic
shape picks by count give, for the default set, the L2-direct kernel's words."""
import pytest

pytestmark = pytest.mark.gpu


# two SMs a ciphertext | one per CTA in two waves | the 3-per-CTA kernel
@pytest.mark.parametrize("count", [49, 76, 153, 305])
def test_fp64_words_do_not_depend_on_the_batch(pkg, torch_cuda, count):
    torch = torch_cuda
    e = pkg.Engine(pkg.default_params())
    try:
        e.gate_keyset([9], forms=("fp64",), want_bk=False)
        x = torch.randint(-2 ** 31, 2 ** 31, (count, e.params.n + 1), device="cuda", dtype=torch.int32)
        out = torch.empty((2, count, 1025), dtype=torch.int32, device="cuda")
        sp = torch.cuda.current_stream().cuda_stream
        for k, shape in enumerate((0, 3)):
            e.set_groups_per_cta("fp64", shape)
            e.tfhe_bootstrap_woKS_FFT(out[k], x, 1 << 29, count, "fp64", stream=sp)
            torch.cuda.synchronize()
        e.synchronize()
        assert torch.equal(out[0], out[1])
    finally:
        e.close()
