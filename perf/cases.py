"""The measured cases: gate bootstrapping through the public entry points.

Each case is one call (or, for the server, one burst of requests) as a user's
program makes it.  Ciphertexts are encryptions under the uploaded key, fresh
for each seed; the keys stay, as a server keeps its clients' cloud key.

Kinds:
  gates    a batch of independent gates, mixed NAND/AND/XOR/OR
  mux      bootsMUX, two bootstraps and one key switch each
  lut      programmable bootstrap with an 8-entry table
  extprod  external products, one TGSW per TLWE
  serve    encrypted circuits of several clients through the gate server

Every output is whole: the Torus32 ciphertexts themselves.  They are int32
and depend on each rounding of the transforms, so there is no 64-bit value to
compare them with (`exact` gives None): they are held to equality.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if _ROOT not in sys.path:
    sys.path.insert(0, _ROOT)

import __graft_entry__  # noqa: E402

pkg = __graft_entry__.load_package()
import tfhe_gb300.circuits as circuits  # noqa: E402

_MIXED = ("NAND", "AND", "XOR", "OR")
_PARAMS = {"default": pkg.default_params, "stress": pkg.stress_params}
_engines = {}  # parameter set -> (engine, LWE key): made once, as a user's program does
_streams = []


def listed():
    return [
        # one gate on host buffers: the drop-in bootsNAND of a program that evaluates its circuit gate by gate
        {"name": "host_gate_1", "kind": "gates", "count": 1, "form": "split_fp32", "params": "default", "host": True},
        # one 16-bit word: the test bench's server evaluates a gate on every bit of a word
        {"name": "word_16", "kind": "gates", "count": 16, "form": "split_fp32", "params": "default", "host": False},
        # a few clients' words under one select each: 128 bootstraps, one per SM or less
        {"name": "mux_64", "kind": "mux", "count": 64, "form": "split_fp32", "params": "default"},
        # a ragged layer of a middling circuit, one to two gates per SM
        {"name": "layer_263", "kind": "gates", "count": 263, "form": "split_fp32", "params": "default", "host": False},
        # a wider one, three to four gates per SM
        {"name": "layer_517", "kind": "gates", "count": 517, "form": "split_fp32", "params": "default", "host": False},
        # lookup tables over a batch of small integers
        {"name": "lut_700", "kind": "lut", "count": 700, "form": "split_fp32", "params": "default"},
        # the benchmark's circuit layer, the largest layer the server admits in one batch
        {"name": "layer_4096", "kind": "gates", "count": 4096, "form": "split_fp32", "params": "default", "host": False},
        # the alternative parameter set (n = 500, l = 2, Bgbit = 10)
        {"name": "stress_1100", "kind": "gates", "count": 1100, "form": "split_fp32", "params": "stress", "host": False},
        # the plain FP64 form: a single gate, and a layer
        {"name": "fp64_gate_1", "kind": "gates", "count": 1, "form": "fp64", "params": "default", "host": False},
        {"name": "fp64_layer_300", "kind": "gates", "count": 300, "form": "fp64", "params": "default", "host": False},
        # the external-product benchmark
        {"name": "extprod_1024", "kind": "extprod", "count": 1024, "form": "split_fp32", "params": "default"},
        # a burst of circuits (32-bit adders, 16-bit comparators, 8-bit multiplexers) through the gate server
        {"name": "serve_24", "kind": "serve", "count": 24, "form": "split_fp32", "params": "default"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gates", "gates", "gates", "gates", "stress", "mux", "lut", "fp64", "extprod", "serve"])
    if kind == "gates":
        count = _log_int(rng, 1, 4096)
        return {"kind": "gates", "count": count, "form": "split_fp32", "params": "default", "host": rng.random() < 0.25}
    if kind == "stress":
        return {"kind": "gates", "count": _log_int(rng, 1, 4096), "form": "split_fp32", "params": "stress", "host": False}
    if kind == "mux":
        return {"kind": "mux", "count": _log_int(rng, 1, 1500), "form": "split_fp32", "params": "default"}
    if kind == "lut":
        return {"kind": "lut", "count": _log_int(rng, 1, 3000), "form": "split_fp32", "params": "default"}
    if kind == "fp64":
        return {"kind": "gates", "count": _log_int(rng, 1, 456), "form": "fp64", "params": rng.choice(["default", "stress"]),
                "host": False}
    if kind == "extprod":
        return {"kind": "extprod", "count": _log_int(rng, 1, 3000), "form": rng.choice(["split_fp32", "split_fp32", "fp64"]),
                "params": rng.choice(["default", "stress"])}
    return {"kind": "serve", "count": rng.randint(1, 40), "form": "split_fp32", "params": "default"}


def _engine(name):
    if name not in _engines:
        eng = pkg.Engine(_PARAMS[name](), device=0)
        lwe, _, _, _ = eng.gate_keyset([0], want_bk=False)
        _engines[name] = (eng, lwe)
    return _engines[name]


def _stream():
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def _encrypt(P, lwe, mu, gen):
    """LWE samples of the Torus32 messages mu: uniform mask, body <mask, key> + mu + noise."""
    dev = mu.device
    n = P.n
    out = torch.randint(-2 ** 31, 2 ** 31, (mu.numel(), n + 1), generator=gen, device=dev, dtype=torch.int64)
    noise = torch.randn(mu.numel(), generator=gen, device=dev, dtype=torch.float64) * (P.lwe_alpha * 2.0 ** 32)
    key = torch.from_numpy(np.asarray(lwe, np.int64)).to(dev)
    body = (out[:, :n] * key).sum(1) + mu.reshape(-1).to(torch.int64) + noise.round().to(torch.int64)
    out[:, n] = (body + 2 ** 31) % 2 ** 32 - 2 ** 31
    return out.to(torch.int32).contiguous()


def _bits(count, gen, dev):
    return torch.randint(0, 2, (count,), generator=gen, device=dev, dtype=torch.int64)


def _encrypt_bits(P, lwe, bits, gen):
    return _encrypt(P, lwe, (2 * bits - 1) * 2 ** 29, gen)  # +-1/8


def _prepare_serve(case, seed, P, lwe, eng, gen, dev):
    rng = np.random.default_rng(seed)
    make = [lambda: circuits.ripple_carry_adder(32), lambda: circuits.comparator(16), lambda: circuits.multiplexer(8)]
    requests = []
    for i in range(case["count"]):
        gates, nin, outs = make[i % 3]()
        x = _encrypt_bits(P, lwe, _bits(nin, gen, dev), gen).cpu().numpy()
        requests.append((gates, nin, x, np.array(outs, np.int32)))
    order = rng.permutation(len(requests))
    return {"server": pkg.Server(eng, pool_slots=65536, max_batch=4096, form=case["form"]),
            "requests": [requests[i] for i in order]}


def prepare(case, seed):
    eng, lwe = _engine(case["params"])
    P = eng.params
    dev = torch.device("cuda:0")
    st = _stream()
    with torch.cuda.stream(st):
        gen = torch.Generator(device=dev)
        gen.manual_seed(seed)
        s = {"kind": case["kind"], "eng": eng, "count": case["count"], "form": case["form"], "stream": st.cuda_stream}
        count = case["count"]
        if case["kind"] == "gates":
            a, b = (_encrypt_bits(P, lwe, _bits(count, gen, dev), gen) for _ in range(2))
            kinds = torch.tensor([pkg.GATES[g] for g in _MIXED], device=dev, dtype=torch.int32)
            gates = kinds[torch.randint(0, len(_MIXED), (count,), generator=gen, device=dev)].contiguous()
            s["host"] = case["host"]
            if case["host"]:
                s["args"] = [t.cpu().numpy() for t in (a, b, gates)]
            else:
                s["args"] = [a, b, gates]
                s["out"] = torch.empty_like(a)
        elif case["kind"] == "mux":
            s["args"] = [_encrypt_bits(P, lwe, _bits(count, gen, dev), gen) for _ in range(3)]
            s["out"] = torch.empty_like(s["args"][0])
        elif case["kind"] == "lut":
            # messages 0..7 at the centres of 8 slots of the half turn; table f(m) = 5m + 3 mod 8
            m = torch.randint(0, 8, (count,), generator=gen, device=dev, dtype=torch.int64)
            s["x"] = _encrypt(P, lwe, (2 * m + 1) * 2 ** 27, gen)
            table = np.array([((2 * ((5 * i + 3) % 8) + 1) << 27) for i in range(8)], np.int64).astype(np.int32)
            s["tv"] = torch.from_numpy(pkg.test_vector(P.N, table)).to(dev)
            s["out"] = torch.empty_like(s["x"])
        elif case["kind"] == "extprod":
            # masks and bodies of TGSW and TLWE samples are uniform to whoever lacks the key
            tgsw = torch.randint(-2 ** 31, 2 ** 31, (count, P.tgsw_words()), generator=gen, device=dev, dtype=torch.int32)
            s["gsw"] = torch.empty(count * eng.tgsw_fft_bytes(case["form"]), device=dev, dtype=torch.uint8)
            eng.tgsw_to_fft(tgsw, s["gsw"], count, case["form"], stream=st.cuda_stream)
            s["acc"] = torch.randint(-2 ** 31, 2 ** 31, (count, 2 * P.N), generator=gen, device=dev, dtype=torch.int32)
        else:
            s.update(_prepare_serve(case, seed, P, lwe, eng, gen, dev))
    st.synchronize()
    return s


def run(s):
    eng, count, form, stream = s["eng"], s["count"], s["form"], s["stream"]
    if s["kind"] == "gates":
        a, b, gates = s["args"]
        if s["host"]:
            return eng.bootsGates_host(a, b, gates=gates, form=form)
        eng.bootsGates(gates, s["out"], a, b, count, form, stream=stream)
        return s["out"]
    if s["kind"] == "mux":
        eng.bootsMUX(s["out"], *s["args"], count, form, stream=stream)
        return s["out"]
    if s["kind"] == "lut":
        eng.bootstrap_tv(s["out"], s["x"], s["tv"], count, form, stream=stream)
        return s["out"]
    if s["kind"] == "extprod":
        eng.tGswFFTExternMulToTLwe(s["acc"], s["gsw"], count, form, stream=stream)  # in place
        return s["acc"]
    srv = s["server"]
    ids = [srv.submit(*r) for r in s["requests"]]
    got = {}
    while len(got) < len(ids):
        srv.step()
        for i in ids:
            if i not in got:
                r = srv.poll(i)
                if r is not None:
                    got[i] = r[0]
    return np.concatenate([got[i] for i in ids])


def work(case):
    P = _PARAMS[case["params"]]()
    count = case["count"]
    # transforms: 512 points, 5 N log2 N operations each, of 2l digit polynomials and 2 results a step, the
    # twist (6 a point) and the products (2 x 2l x 8 a point)
    step = (2 * P.l + 2) * (5 * 512 * 9 + 6 * 512) + 2 * 2 * P.l * 512 * 8
    step_key = 2 * P.l * 2 * 512 * 16
    lwe = 4 * (P.n + 1)
    if case["kind"] == "extprod":
        return {"bytes": count * (step_key + 2 * 2 * P.N * 4), "flops": count * step}
    boots = switches = count
    io = {"gates": 3, "mux": 4, "lut": 2, "serve": 0}[case["kind"]] * count * lwe
    if case["kind"] == "mux":
        boots = 2 * count
    if case["kind"] == "lut":
        io += 4 * P.N
    if case["kind"] == "serve":
        made = [circuits.ripple_carry_adder(32), circuits.comparator(16), circuits.multiplexer(8)]
        per = [made[i % 3] for i in range(count)]
        boots = sum(circuits.bootstraps(g) for g, _, _ in per)
        switches = sum(int((g[:, 0] <= circuits.MUX).sum()) for g, _, _ in per)
        io = sum(nin + len(outs) for _, nin, outs in per) * lwe
    # each key-switch level takes one of three table rows, or none, per ciphertext
    rows = P.N * P.ks_t * 3
    touched = rows * (1.0 - 0.75 ** switches)
    adds = switches * P.N * P.ks_t * 0.75 * (P.n + 1)
    return {"bytes": P.n * step_key + touched * lwe + io, "flops": boots * P.n * step + adds}


def exact(case, seed):
    # Every output is a Torus32 ciphertext, a whole number that is compared as such.  A blind rotation has no
    # 64-bit value of its own: a digit that falls on the other side of a boundary brings in another key row.
    return None
