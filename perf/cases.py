"""The prover's measured workloads: multi-exponentiations, transforms and whole proofs.

Each case is one call, or one batch, of the public Python API over the range of sizes that a
Groth16 prover meets: single MSMs from a few hundred terms to 2^20, transforms from 2^10 to
2^22 points, proofs from 2^10 to 2^20 constraints.  All outputs are integers mod a 254-bit
prime, so every comparison is exact.

Inputs are drawn on the GPU from the seed.  Scalars and field elements are uniform below the
modulus; with ``bits`` that share of the scalars is 0 or 1, as most wires of a real circuit
(boolean gadgets: hashes, range checks) are.  Curve points are k G with seeded k.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

from cusnarks_b200 import Context, synth
from cusnarks_b200.groth import Prover, SyntheticCircuit, setup_pk

Q, R = synth.Q, synth.R
MONT = 1 << 256


# ------------------------------------------------------------------------- cases ----
def listed() -> list:
    return [
        # a short multi-exponentiation from host arrays (verification-key sums, small statements):
        # latency of the launch sequence and of its dependent chains
        {"name": "msm_g1_host_1000", "kind": "msm", "ec2": False, "n": 1000, "bits": 0.0, "host": True},
        # one G1 multi-exponentiation with bases that come with the call
        {"name": "msm_g1_2e20", "kind": "msm", "ec2": False, "n": 1 << 20, "bits": 0.0, "host": False},
        # the same over G2, at a size that fills the GPU only in part
        {"name": "msm_g2_40001", "kind": "msm", "ec2": True, "n": 40001, "bits": 0.0, "host": False},
        # a witness (half of it bits) over a proving key's resident tables, ragged size
        {"name": "msm_g1_fixed_100003_bits", "kind": "fixed", "ec2": False, "n": 100003, "bits": 0.5},
        # many instances of uneven size in one captured pass
        {"name": "msm_g1_batch_24", "kind": "batch", "ec2": False, "count": 24, "log_lo": 10, "log_hi": 16,
         "sizes_seed": 5},
        # transforms: launch-bound, and larger than the L2
        {"name": "ntt_2e12", "kind": "ntt", "log_n": 12, "direction": 1, "fmat": 1},
        {"name": "intt_2e22", "kind": "ntt", "log_n": 22, "direction": -1, "fmat": 0},
        # polynomial-H step: the prover's variant, and the coset quotient
        {"name": "hstep_2e18", "kind": "hstep", "log_m": 18, "coset": False},
        {"name": "hstep_coset_2e15", "kind": "hstep", "log_m": 15, "coset": True},
        # one proof of a small statement, witness and proof in host memory: latency
        {"name": "prove_2e12_host", "kind": "prove", "log_m": 12, "n_public": 1, "n_inputs": 64, "bits": 0.0, "k": 1,
         "host": True},
        # what the server runs for queued requests with one small key
        {"name": "prove_2e13_batch8", "kind": "prove", "log_m": 13, "n_public": 3, "n_inputs": 101, "bits": 0.5, "k": 8,
         "host": False},
        # the headline statement: 2^20 constraints, witness resident on the device
        {"name": "prove_2e20", "kind": "prove", "log_m": 20, "n_public": 1, "n_inputs": 64, "bits": 0.0, "k": 1,
         "host": False},
    ]


def _log_uniform(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["msm", "msm", "msm", "fixed", "batch", "ntt", "hstep", "prove", "prove"])
    bits = rng.choice([0.0, 0.0, 0.3, 0.6, 0.9])
    if kind == "msm":
        ec2 = rng.random() < 0.4
        n = _log_uniform(rng, 300, 1 << (17 if ec2 else 20))
        return {"kind": kind, "ec2": ec2, "n": n, "bits": bits, "host": n < 20000 and rng.random() < 0.5}
    if kind == "fixed":
        ec2 = rng.random() < 0.4
        return {"kind": kind, "ec2": ec2, "n": _log_uniform(rng, 300, 1 << (17 if ec2 else 20)), "bits": bits}
    if kind == "batch":
        ec2 = rng.random() < 0.3
        lo = rng.randint(8, 11)
        return {"kind": kind, "ec2": ec2, "count": rng.randint(2, 32), "log_lo": lo,
                "log_hi": rng.randint(lo + 1, 13 if ec2 else 16), "sizes_seed": rng.randint(1, 10 ** 6)}
    if kind == "ntt":
        return {"kind": kind, "log_n": rng.randint(10, 22), "direction": rng.choice([1, -1]), "fmat": rng.choice([0, 1])}
    if kind == "hstep":
        return {"kind": kind, "log_m": rng.randint(10, 20), "coset": rng.random() < 0.5}
    k = rng.choice([1, 1, rng.randint(2, 16)])
    return {"kind": kind, "log_m": rng.randint(10, 18 if k == 1 else 13), "n_public": rng.randint(1, 8),
            "n_inputs": rng.randint(16, 300), "bits": bits, "k": k, "host": k == 1 and rng.random() < 0.5}


# ------------------------------------------------------------------------ inputs ----
@functools.lru_cache(maxsize=1)
def _ctx() -> Context:
    return Context(0)


def _gen(seed: int, stream: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + stream) & 0x7FFFFFFFFFFFFFFF)
    return g


def _field(g: torch.Generator, n: int, bits: float = 0.0) -> torch.Tensor:
    """(n, 8) limbs below the moduli (whose top limb is 0x30644e72), that share of them 0 or 1."""
    x = torch.randint(-(1 << 31), 1 << 31, (n, 8), device="cuda", dtype=torch.int64, generator=g).to(torch.int32)
    x[:, 7] = torch.randint(0, 0x30644E72, (n,), device="cuda", dtype=torch.int64, generator=g).to(torch.int32)
    if bits > 0:
        small = torch.rand(n, device="cuda", generator=g) < bits
        bit = torch.randint(0, 2, (n,), device="cuda", dtype=torch.int32, generator=g)
        x[small] = 0
        x[:, 0] = torch.where(small, bit, x[:, 0])
    return x


def _dev(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()


def _host(t: torch.Tensor) -> np.ndarray:
    return t.cpu().numpy().view(np.uint32)


def _points(g: torch.Generator, n: int, ec2: bool) -> torch.Tensor:
    k = _field(g, n)
    base = _dev(synth.g2_generator() if ec2 else synth.g1_generator())
    out = torch.empty((n, 32 if ec2 else 16), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    _ctx().scmul_device(k.data_ptr(), base.data_ptr(), n, out.data_ptr(), ec2=ec2, point_stride_words=0)
    _ctx().sync()
    return out


@functools.lru_cache(maxsize=1)
def _prover(log_m: int, n_public: int, n_inputs: int) -> Prover:
    """A resident proving key: a program keeps it for all witnesses of its statement."""
    circ = SyntheticCircuit(_ctx(), log_m, seed=100, n_public=n_public, n_inputs=n_inputs)
    return Prover(_ctx(), setup_pk(_ctx(), circ, seed=101))


def _batch_sizes(case: dict) -> list:
    rng = random.Random(case["sizes_seed"])
    return [_log_uniform(rng, 1 << case["log_lo"], 1 << case["log_hi"]) for _ in range(case["count"])]


def prepare(case: dict, seed: int) -> dict:
    kind, ec2 = case["kind"], bool(case.get("ec2"))
    pw = 32 if ec2 else 16
    st = {"case": case}
    if kind in ("msm", "fixed"):
        n = case["n"]
        scalars, points = _field(_gen(seed, 1), n, case["bits"]), _points(_gen(seed, 2), n, ec2)
        if case.get("host"):
            st["scalars"], st["points"] = _host(scalars), _host(points)
        else:
            st["scalars"], st["points"] = scalars, points
            st["out"] = torch.zeros(pw, dtype=torch.int32, device="cuda")
        if kind == "fixed":
            st["window"] = c = Context.msm_fixed_window(n, ec2)
            table = torch.empty(Context.msm_fixed_table_points(n, c) * pw, dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            _ctx().msm_fixed_table_device(points.data_ptr(), n, c, table.data_ptr(), ec2=ec2)
            _ctx().sync()
            st["table"] = table
    elif kind == "batch":
        sizes = _batch_sizes(case)
        st["scalars"] = [_field(_gen(seed, 10 + 2 * i), n) for i, n in enumerate(sizes)]
        st["points"] = [_points(_gen(seed, 11 + 2 * i), n, ec2) for i, n in enumerate(sizes)]
        st["out"] = torch.zeros((len(sizes), pw), dtype=torch.int32, device="cuda")
        jobs = [(s.data_ptr(), p.data_ptr(), n, o.data_ptr())
                for s, p, n, o in zip(st["scalars"], st["points"], sizes, st["out"])]
        st["plan"] = _ctx().msm_batch(jobs, ec2)
    elif kind == "ntt":
        st["x"] = _field(_gen(seed, 1), 1 << case["log_n"])
        st["out"] = torch.empty_like(st["x"])
    elif kind == "hstep":
        m = 1 << case["log_m"]
        st["abc"] = [_field(_gen(seed, 1 + i), m) for i in range(3)]
        st["out"] = torch.empty((m if case["coset"] else 2 * m, 8), dtype=torch.int32, device="cuda")
    else:
        st["prover"] = p = _prover(case["log_m"], case["n_public"], case["n_inputs"])
        ws = []
        for i in range(case["k"]):
            w = _field(_gen(seed, 20 + i), p.n_vars, case["bits"])
            w[0] = 0
            w[0, 0] = 1  # the constant wire
            ws.append(_host(w) if case["host"] else w)
        st["w"] = ws
        st["rs"], st["ss"] = _host(_field(_gen(seed, 3), case["k"])), _host(_field(_gen(seed, 4), case["k"]))
        if not case["host"]:
            st["out"] = torch.zeros((case["k"], 64), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()  # the library works on its own streams
    return st


# --------------------------------------------------------------------------- run ----
def run(st: dict):
    case, ctx = st["case"], _ctx()
    kind, ec2 = case["kind"], bool(case.get("ec2"))
    if kind == "msm" and case["host"]:
        return ctx.msm(st["scalars"], st["points"], ec2=ec2)
    if kind == "msm":
        ctx.msm_device(st["scalars"].data_ptr(), st["points"].data_ptr(), case["n"], st["out"].data_ptr(), ec2=ec2)
    elif kind == "fixed":
        ctx.msm_fixed_device(st["scalars"].data_ptr(), st["table"].data_ptr(), case["n"], st["window"],
                             st["out"].data_ptr(), ec2=ec2)
    elif kind == "batch":
        st["plan"].run()
    elif kind == "ntt":
        ctx.ntt_device(st["x"].data_ptr(), st["out"].data_ptr(), case["log_n"], case["direction"], case["fmat"])
    elif kind == "hstep":
        a, b, c = (t.data_ptr() for t in st["abc"])
        ctx.hstep_device(int(case["coset"]), a, b, c, case["log_m"], st["out"].data_ptr())
    elif case["host"]:
        return st["prover"].prove(st["w"][0], st["rs"][0], st["ss"][0])
    elif case["k"] == 1:
        st["prover"].prove_device(st["w"][0].data_ptr(), st["rs"][0], st["ss"][0], st["out"].data_ptr())
    else:
        st["prover"].prove_batch_device([w.data_ptr() for w in st["w"]], st["rs"], st["ss"],
                                        [o.data_ptr() for o in st["out"]])
    return st["out"]


def tolerance(case: dict):
    return "exact"


# -------------------------------------------------------------------------- work ----
PRODUCT = 2 * 136  # operations of a 256-bit Montgomery product: 136 32x32-bit multiply-adds


def _msm_products(n: int, ec2: bool, fixed: bool) -> float:
    """Base-field products of the bucket method at its best window."""
    best = math.inf
    for c in range(4, 23):
        w = 254 // c + 1
        best = min(best, w * 10.0 * n + (1 if fixed else w) * 14.0 * 2 ** c + (0 if fixed else 9 * 254))
    return best * (3 if ec2 else 1)


def _ntt_products(log_n: int) -> float:
    return 0.5 * log_n * 2 ** log_n


def work(case: dict) -> dict:
    kind, ec2 = case["kind"], bool(case.get("ec2"))
    point = 128 if ec2 else 64
    if kind in ("msm", "fixed"):
        n = case["n"]
        return {"bytes": n * (32.0 + point), "flops": PRODUCT * _msm_products(n, ec2, kind == "fixed")}
    if kind == "batch":
        sizes = _batch_sizes(case)
        return {"bytes": sum(sizes) * (32.0 + point), "flops": PRODUCT * sum(_msm_products(n, ec2, False) for n in sizes)}
    if kind == "ntt":
        return {"bytes": 64.0 * 2 ** case["log_n"], "flops": PRODUCT * _ntt_products(case["log_n"])}
    log_m = case["log_m"]
    m = 2 ** log_m
    h = 4 * _ntt_products(log_m) + _ntt_products(log_m + 1) + 3 * m
    if kind == "hstep":
        if case["coset"]:
            return {"bytes": 128.0 * m, "flops": PRODUCT * (7 * _ntt_products(log_m) + 5 * m)}
        return {"bytes": 128.0 * m, "flops": PRODUCT * h}
    msms = 4 * _msm_products(m, False, True) + _msm_products(m, True, True)
    # witness, key points (four G1 arrays, one G2) and the matrices' entries (3 a row)
    return {"bytes": 32.0 * m * case["k"] + m * (4 * 64.0 + 128.0 + 6 * 36.0),
            "flops": PRODUCT * case["k"] * (msms + h + 6 * m)}


# ------------------------------------------------------------------------- exact ----
def _ints(t) -> list:
    rows = t if isinstance(t, np.ndarray) else _host(t)
    return [int.from_bytes(x.tobytes(), "little") for x in rows.reshape(-1, 8)]


def _limbs(values) -> np.ndarray:
    return np.frombuffer(b"".join(v.to_bytes(32, "little") for v in values), dtype=np.uint32)


class _Fq2:
    __slots__ = ("a", "b")

    def __init__(self, a, b=0):
        self.a, self.b = a % Q, b % Q

    def __add__(self, o):
        return _Fq2(self.a + o.a, self.b + o.b)

    def __sub__(self, o):
        return _Fq2(self.a - o.a, self.b - o.b)

    def __mul__(self, o):
        return _Fq2(self.a * o.a - self.b * o.b, self.a * o.b + self.b * o.a)

    def __bool__(self):
        return bool(self.a or self.b)

    def inverse(self):
        d = pow(self.a * self.a + self.b * self.b, -1, Q)
        return _Fq2(self.a * d, -self.b * d)


def _jac_double(p):
    x, y, z = p
    a, b = x * x, y * y
    c = b * b
    d = (x + b) * (x + b) - a - c
    d, e = d + d, a + a + a
    x3 = e * e - d - d
    c = c + c + c + c
    return x3, e * (d - x3) - c - c, (y + y) * z


def _jac_add(p, q):
    if p is None or q is None:
        return q if p is None else p
    (x1, y1, z1), (x2, y2, z2) = p, q
    zz1, zz2 = z1 * z1, z2 * z2
    u1, u2, s1, s2 = x1 * zz2, x2 * zz1, y1 * z2 * zz2, y2 * z1 * zz1
    h, r = u2 - u1, s2 - s1
    if not h:
        return None if r else _jac_double(p)
    hh = h * h
    hhh, v = h * hh, u1 * hh
    x3 = r * r - hhh - v - v
    return x3, r * (v - x3) - s1 * hhh, z1 * z2 * h


def _exact_msm(scalars, points, ec2: bool) -> np.ndarray:
    """sum k_i P_i by buckets of 8-bit digits, Python integers throughout."""
    words, unmont, ks = _ints(points), pow(MONT, -1, Q), _ints(scalars)
    words = [w * unmont % Q for w in words]
    if ec2:
        pts = [(_Fq2(*words[i:i + 2]), _Fq2(*words[i + 2:i + 4]), _Fq2(1)) for i in range(0, len(words), 4)]
    else:
        pts = [(_Fq2(words[i]), _Fq2(words[i + 1]), _Fq2(1)) for i in range(0, len(words), 2)]
    total = None
    for shift in range(248, -8, -8):
        if total is not None:
            for _ in range(8):
                total = _jac_double(total)
        buckets = [None] * 256
        for k, p in zip(ks, pts):
            d = (k % R) >> shift & 255
            if d:
                buckets[d] = _jac_add(buckets[d], p)
        run_, acc = None, None
        for b in reversed(buckets[1:]):
            run_ = _jac_add(run_, b)
            acc = _jac_add(acc, run_)
        total = _jac_add(total, acc)
    x, y, z = total
    zi = z.inverse()
    x, y = x * zi * zi, y * zi * zi * zi
    vals = [x.a, x.b, y.a, y.b] if ec2 else [x.a, y.a]
    return _limbs([v * MONT % Q for v in vals]).view(np.int32)


def _root(log_n: int) -> int:
    return pow(5, (R - 1) >> log_n, R)


def _exact_ntt(x: list, root: int) -> list:
    if len(x) == 1:
        return x
    even, odd = _exact_ntt(x[::2], root * root % R), _exact_ntt(x[1::2], root * root % R)
    w, lo, hi = 1, [], []
    for a, b in zip(even, odd):
        t = w * b % R
        lo.append((a + t) % R)
        hi.append((a - t) % R)
        w = w * root % R
    return lo + hi


def _exact_intt(x: list, log_n: int) -> list:
    s = pow(len(x), -1, R)
    return [v * s % R for v in _exact_ntt(x, pow(_root(log_n), -1, R))]


def exact(case: dict, seed: int):
    kind, ec2 = case["kind"], bool(case.get("ec2"))
    if kind in ("msm", "fixed"):
        if case["n"] > (2000 if ec2 else 5000):
            return None  # minutes in Python integers
        st = prepare(case, seed)
        v = _exact_msm(st["scalars"], st["points"], ec2)
        return v.view(np.uint32) if case.get("host") else v
    if kind == "ntt" and case["log_n"] <= 18:
        L, unmont = case["log_n"], pow(MONT, -1, R)
        x = [v * unmont % R for v in _ints(prepare(case, seed)["x"])]
        y = _exact_ntt(x, _root(L)) if case["direction"] > 0 else _exact_intt(x, L)
        mont = case["direction"] > 0 or case["fmat"]
        return _limbs([v * MONT % R if mont else v for v in y]).view(np.int32).reshape(-1, 8)
    if kind == "hstep" and case["log_m"] <= 15:
        L, unmont = case["log_m"], pow(MONT, -1, R)
        a, b, c = ([v * unmont % R for v in _ints(t)] for t in prepare(case, seed)["abc"])
        pa, pb, pc = (_exact_intt(v, L) for v in (a, b, c))
        if not case["coset"]:  # coefficients of A(x) B(x)
            pad, w = [0] * len(a), _root(L + 1)
            y = _exact_intt([u * v % R for u, v in zip(_exact_ntt(pa + pad, w), _exact_ntt(pb + pad, w))], L + 1)
        else:  # (A B - C) / (x^m - 1) on 5 <w>
            g = [pow(5, i, R) for i in range(len(a))]
            ea, eb, ec = (_exact_ntt([u * v % R for u, v in zip(p, g)], _root(L)) for p in (pa, pb, pc))
            z, gi = pow(pow(5, len(a), R) - 1, -1, R), pow(5, -1, R)
            y = _exact_intt([(u * v - w) * z % R for u, v, w in zip(ea, eb, ec)], L)
            y = [v * pow(gi, i, R) % R for i, v in enumerate(y)]
        return _limbs(y).view(np.int32).reshape(-1, 8)
    return None  # batches and whole proofs: minutes in Python integers
