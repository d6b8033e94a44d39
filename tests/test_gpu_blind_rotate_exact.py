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


# FP64: 76 | 77 .. 304 | 305 .. 456 | 457 is a whole wave and a remainder
@pytest.mark.parametrize("params,count", [("default", 77), ("stress", 76), ("stress", 153), ("stress", 305),
                                          ("stress", 457), ("stress", 533)])
def test_fp64_automatic_shape_matches_l2_direct(engines, torch_cuda, params, count):
    torch = torch_cuda
    e = engines(params)
    x = _uniform(torch, count, count, e.params.n + 1)
    got = _bootstraps(torch, e, "fp64", 0, x)
    assert (got == _bootstraps(torch, e, "fp64", 3, x)).all()


@pytest.mark.parametrize("count", [80])
def test_fp64_blind_rotate_from_accumulators(engines, torch_cuda, count):
    torch = torch_cuda
    e = engines("stress")
    acc = _uniform(torch, 3, count, 2048)
    bara = _uniform(torch, 4, count, e.params.n) & 2047
    bara[:, 5] = 0
    bara[1] = 0
    assert (_rotations(torch, e, "fp64", 0, acc, bara) == _rotations(torch, e, "fp64", 3, acc, bara)).all()
