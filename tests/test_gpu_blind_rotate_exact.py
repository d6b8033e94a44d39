"""The blind-rotation kernels that the automatic shapes pick by batch size,
held bit for bit to the kernels that stay selectable, at the edges of their
ranges.  Inputs are uniform Torus32 words (every rotation amount occurs, 0
among them); equality is exact, so there is no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(pkg, name):
    e = pkg.Engine(pkg.default_params() if name == "default" else pkg.stress_params())
    e.gate_keyset([9], want_bk=False)
    return e


@pytest.fixture(scope="module")
def engines(pkg, torch_cuda):
    made = {}

    def get(name):
        if name not in made:
            made[name] = _engine(pkg, name)
        return made[name]

    yield get
    for e in made.values():
        e.close()


def _bootstraps(torch, e, form, shape, x):
    """Extracted samples of x without key switch under a launch shape."""
    out = torch.empty((x.shape[0], 1025), dtype=torch.int32, device="cuda")
    e.set_groups_per_cta(form, shape)
    try:
        e.tfhe_bootstrap_woKS_FFT(out, x, 1 << 29, x.shape[0], form, stream=torch.cuda.current_stream().cuda_stream)
        e.synchronize()
        torch.cuda.synchronize()
    finally:
        e.set_groups_per_cta(form, 0)
    return out.cpu().numpy()


def _rotations(torch, e, form, shape, acc, bara):
    acc = acc.clone()
    e.set_groups_per_cta(form, shape)
    try:
        e.tfhe_blindRotate_FFT(acc, bara, acc.shape[0], form, stream=torch.cuda.current_stream().cuda_stream)
        e.synchronize()
        torch.cuda.synchronize()
    finally:
        e.set_groups_per_cta(form, 0)
    return acc.cpu().numpy()


def _uniform(torch, seed, *shape):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randint(-2 ** 31, 2 ** 31, shape, generator=g, device="cuda", dtype=torch.int32)


# FP64: 48 | 49 .. 76 | 77 .. 304 | 305 .. 456 | 457 is a whole wave and a remainder
@pytest.mark.parametrize("params,count", [("default", 1), ("stress", 16), ("default", 48), ("stress", 49), ("default", 77), ("stress", 76), ("stress", 153), ("stress", 305),
                                          ("stress", 457), ("stress", 533)])
def test_fp64_automatic_shape_matches_l2_direct(engines, torch_cuda, params, count):
    torch = torch_cuda
    e = engines(params)
    x = _uniform(torch, count, count, e.params.n + 1)
    got = _bootstraps(torch, e, "fp64", 0, x)
    assert (got == _bootstraps(torch, e, "fp64", 3, x)).all()


@pytest.mark.parametrize("count", [5, 80])
def test_fp64_blind_rotate_from_accumulators(engines, torch_cuda, count):
    torch = torch_cuda
    e = engines("stress")
    acc = _uniform(torch, 3, count, 2048)
    bara = _uniform(torch, 4, count, e.params.n) & 2047
    bara[:, 5] = 0
    bara[1] = 0
    assert (_rotations(torch, e, "fp64", 0, acc, bara) == _rotations(torch, e, "fp64", 3, acc, bara)).all()


# split-FP32, one per CTA: a few | one per SM and one more (a second wave)
@pytest.mark.parametrize("params,count", [("default", 3), ("stress", 153)])
def test_spread_kernel_matches_l2_direct(engines, torch_cuda, params, count):
    torch = torch_cuda
    e = engines(params)
    x = _uniform(torch, count, count, e.params.n + 1)
    x[0, 7] = 0
    assert (_bootstraps(torch, e, "split_fp32", 14, x) == _bootstraps(torch, e, "split_fp32", 4, x)).all()
    acc = _uniform(torch, 3, count, 2048)
    bara = _uniform(torch, 4, count, e.params.n) & 2047
    bara[:, 5] = 0
    bara[0] = 0
    assert (_rotations(torch, e, "split_fp32", 14, acc, bara) == _rotations(torch, e, "split_fp32", 4, acc, bara)).all()


# split-FP32 in lane pairs, 6 and (l = 2) 4 per SM: one, an odd number in the last set, a whole wave and one more
@pytest.mark.parametrize("params,shape,count", [("default", 10, 1), ("stress", 10, 911), ("default", 10, 913),
                                                ("stress", 9, 3), ("stress", 9, 609)])
def test_lane_pair_ring_matches_l2_direct(engines, torch_cuda, params, shape, count):
    torch = torch_cuda
    e = engines(params)
    x = _uniform(torch, count, count, e.params.n + 1)
    x[0, 7] = 0  # one of a pair stands still
    assert (_bootstraps(torch, e, "split_fp32", shape, x) == _bootstraps(torch, e, "split_fp32", 4, x)).all()
    if count < 10:
        acc = _uniform(torch, 3, count, 2048)
        bara = _uniform(torch, 4, count, e.params.n) & 2047
        bara[:, 5] = 0
        assert (_rotations(torch, e, "split_fp32", shape, acc, bara)
                == _rotations(torch, e, "split_fp32", 4, acc, bara)).all()


# shape 9 as 3 per CTA up to 3 per SM: a part of a CTA, the last count of it, one more
@pytest.mark.parametrize("params,shape,count", [("default", 9, 2), ("default", 0, 305), ("stress", 0, 456), ("stress", 9, 457),
                                                ("default", 0, 912 + 457)])
def test_three_per_sm_ring_matches_l2_direct(engines, torch_cuda, params, shape, count):
    torch = torch_cuda
    e = engines(params)
    x = _uniform(torch, count, count, e.params.n + 1)
    x[0, 7] = 0
    assert (_bootstraps(torch, e, "split_fp32", shape, x) == _bootstraps(torch, e, "split_fp32", 4, x)).all()
    if count < 10:
        acc = _uniform(torch, 3, count, 2048)
        bara = _uniform(torch, 4, count, e.params.n) & 2047
        bara[:, 5] = 0
        assert (_rotations(torch, e, "split_fp32", shape, acc, bara)
                == _rotations(torch, e, "split_fp32", 4, acc, bara)).all()


# shape 0 over 1 to 2 per SM keeps the pair kernel's summation order (shape 12)
# whatever runs it; shape 15, and shape 0 elsewhere, the order of the rows
# (shape 4): edges of 1, 1.5, 2, 4, 4.5 and 5 per SM, and after a full wave
@pytest.mark.parametrize("params,shape,count,like", [
    ("stress", 0, 152, 4), ("stress", 0, 153, 12), ("default", 0, 228, 12), ("stress", 0, 229, 12),
    ("default", 0, 304, 12), ("stress", 15, 153, 4), ("default", 15, 229, 4), ("stress", 0, 305, 4),
    ("stress", 0, 609, 4), ("default", 0, 685, 4), ("stress", 0, 760, 4), ("stress", 0, 761, 4),
    ("stress", 15, 912 + 160, 4), ("stress", 0, 912 + 650, 4)])
def test_split_automatic_shape_keeps_its_summation_order(engines, torch_cuda, params, shape, count, like):
    torch = torch_cuda
    e = engines(params)
    x = _uniform(torch, count, count, e.params.n + 1)
    x[0, 9] = 0
    assert (_bootstraps(torch, e, "split_fp32", shape, x) == _bootstraps(torch, e, "split_fp32", like, x)).all()


def _cur(torch):
    return torch.cuda.current_stream().cuda_stream


def _fft_keys(torch, e, form, count, seed):
    tgsw = _uniform(torch, seed, count, e.params.tgsw_words())
    out = torch.empty(count, e.tgsw_fft_bytes(form), device="cuda", dtype=torch.uint8)
    e.tgsw_to_fft(tgsw, out, count, form, stream=_cur(torch))
    return out


# one item | a few SMs | one more than the SMs | one more than a round of four per SM
@pytest.mark.parametrize("params,form,count", [("default", "split_fp32", 1), ("stress", "split_fp32", 5),
                                               ("default", "split_fp32", 153), ("stress", "split_fp32", 609),
                                               ("default", "fp64", 153), ("stress", "fp64", 457)])
def test_products_do_not_depend_on_the_batch(engines, torch_cuda, params, form, count):
    """Item k of a batch of products equals the same item alone, and MuxRotate
    equals the product of (X^a - 1) acc plus acc (integer identities)."""
    torch = torch_cuda
    e = engines(params)
    gsw = _fft_keys(torch, e, form, count, count)
    acc = _uniform(torch, count + 1, count, 2048)
    a = _uniform(torch, count + 2, count) & 2047
    a[count // 2] = 0
    got = acc.clone()
    e.tGswFFTExternMulToTLwe(got, gsw, count, form, stream=_cur(torch))
    for k in sorted({0, count // 3, count - 1}):
        one = acc[k:k + 1].clone()
        e.tGswFFTExternMulToTLwe(one, gsw[k:k + 1], 1, form, stream=_cur(torch))
        assert torch.equal(one[0], got[k]), k
    mux = torch.empty_like(acc)
    e.tfhe_MuxRotate_FFT(mux, acc, gsw, a, count, form, stream=_cur(torch))
    diff = torch.empty_like(acc)
    e.tLweMulByXaiMinusOne(diff, a, acc, count, stream=_cur(torch))
    e.tGswFFTExternMulToTLwe(diff, gsw, count, form, stream=_cur(torch))
    assert torch.equal(mux, diff + acc)
    # in place, one TGSW for all
    e.tfhe_MuxRotate_FFT(mux, acc, gsw, a, count, form, per_item=False, stream=_cur(torch))
    acc2 = acc.clone()
    e.tfhe_MuxRotate_FFT(acc2, acc2, gsw, a, count, form, per_item=False, stream=_cur(torch))
    assert torch.equal(mux, acc2)
    e.synchronize()


@pytest.mark.parametrize("params", ["default", "stress"])
def test_steps_of_the_blind_rotation_are_the_products(engines, torch_cuda, params):
    """n MuxRotate calls, one key sample each, give the blind rotation's
    accumulators bit for bit (split-FP32, key rows summed in order)."""
    torch = torch_cuda
    e = engines(params)
    n, count = e.params.n, 7
    lwe, tlwe, ks, bk = e.gate_keyset([9])
    d_bk = torch.from_numpy(bk.reshape(n, -1)).cuda()
    keys = torch.empty(n, e.tgsw_fft_bytes("split_fp32"), device="cuda", dtype=torch.uint8)
    e.tgsw_to_fft(d_bk, keys, n, "split_fp32", stream=_cur(torch))
    acc = _uniform(torch, 21, count, 2048)
    bara = _uniform(torch, 22, count, n) & 2047
    want = _rotations(torch, e, "split_fp32", 4, acc, bara)
    for i in range(n):
        e.tfhe_MuxRotate_FFT(acc, acc, keys[i], bara[:, i].contiguous(), count, "split_fp32", per_item=False,
                             stream=_cur(torch))
    e.synchronize()
    torch.cuda.synchronize()
    assert (acc.cpu().numpy() == want).all()
