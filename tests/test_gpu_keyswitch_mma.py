"""The key switch against its definition, word for word: the tensor-core
kernel (t = 8) at the edges of its tiles (128 and 256 ciphertexts, 80 output
words, the split of the coefficients) and on tables whose 11-bit pieces are at
their extremes, where the sums reach 2^23; the gather kernel for t = 4, 12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(pkg, n, t):
    P = pkg.default_params()
    P.n, P.ks_t = n, t
    return P


def _reference(P, ks, x):
    """lweKeySwitch of one sample (lwe-keyswitch-functions.cpp:114-129)."""
    n_in = P.k * P.N
    a = (x[:n_in].astype(np.int64) & 0xffffffff) + (1 << (32 - (1 + 2 * P.ks_t)))
    table = ks.reshape(n_in, P.ks_t, 4, P.n + 1)
    out = np.zeros(P.n + 1, np.int64)
    out[P.n] = x[n_in]
    for j in range(P.ks_t):
        d = (a >> (30 - 2 * j)) & 3
        rows = table[np.arange(n_in), j, d].astype(np.int64)
        out -= (rows * (d != 0)[:, None]).sum(0)
    return ((out + 2 ** 31) % 2 ** 32 - 2 ** 31).astype(np.int32)


def _run(pkg, torch, P, ks, x):
    e = pkg.Engine(P)
    try:
        e.upload_keyswitch_key(np.zeros_like(ks))
        e.upload_keyswitch_key(ks)  # a later key takes the earlier one's place
        d_in = torch.from_numpy(x).cuda()
        out = torch.full((len(x), P.n + 1), 77, dtype=torch.int32, device="cuda")
        st = torch.cuda.current_stream().cuda_stream
        torch.cuda.synchronize()
        e.lweKeySwitch(out, d_in, len(x), stream=st)
        torch.cuda.synchronize()
        e.synchronize()
        return out.cpu().numpy()
    finally:
        e.close()


@pytest.mark.parametrize("n,t,count", [(630, 8, 1), (630, 8, 129), (500, 8, 257), (79, 8, 128), (80, 8, 256),
                                       (1, 8, 3), (630, 8, 2500), (500, 4, 9), (630, 12, 17)])
def test_key_switch_matches_its_definition(pkg, torch_cuda, n, t, count):
    P = _params(pkg, n, t)
    rng = np.random.default_rng(n * 100 + t)
    ks = rng.integers(-2 ** 31, 2 ** 31, P.ks_words()).astype(np.int32)
    x = rng.integers(-2 ** 31, 2 ** 31, (count, P.k * P.N + 1)).astype(np.int32)
    got = _run(pkg, torch_cuda, P, ks, x)
    for c in sorted({0, count // 2, min(127, count - 1), min(128, count - 1), count - 1}):
        assert (got[c] == _reference(P, ks, x[c])).all(), c


# every piece at its least; the low two at their greatest; the low one alone
@pytest.mark.parametrize("value", [-1024 - 1024 * 2 ** 11 - 512 * 2 ** 22, 1023 + 1023 * 2 ** 11 + 511 * 2 ** 22, 1024])
def test_key_switch_at_the_pieces_extremes(pkg, torch_cuda, value):
    """All 8,192 digits non-zero and every table word the same."""
    P = _params(pkg, 630, 8)
    v = (value + 2 ** 31) % 2 ** 32 - 2 ** 31
    ks = np.full(P.ks_words(), v, np.int32)
    x = np.full((5, P.k * P.N + 1), 0x55550000, np.int32)  # every digit 1
    x[1, :-1] = np.int32(-0x55560000)                      # every digit 2
    x[2, :-1] = np.int32(-0x8001)                          # every digit 3
    x[3, 100] = 0
    x[4, :-1] = 0
    got = _run(pkg, torch_cuda, P, ks, x)
    for c in range(len(x)):
        assert (got[c] == _reference(P, ks, x[c])).all(), c
