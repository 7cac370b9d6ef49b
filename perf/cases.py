"""Workloads of the ring-arithmetic hot path, each through the public Python API.

A case is a dict of plain values. `kind` names the call, the other keys its
sizes; `prepare` makes the seeded inputs and the plan or prepared matrices a
prover keeps, `run` is one pass, `work` the bytes and operations it cannot do
without, `exact` the same results from plain torch arithmetic.

Words are uint32 Montgomery words (value * 2^32 mod q) in int32 tensors.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from lattica_b200 import poly_mul_ntt, twisted_ntt_plan
from lattica_b200.batch import UnevenCommitBatch, sample_uneven_instances
from lattica_b200.commit import PreparedMatrix
from lattica_b200.labrador import (CommitKey, JLMatrix, OuterCommitKey, amortize_witness,
                                   compute_garbage_g, compute_garbage_h, garbage_count,
                                   prover_round_dev, sample_uniform_polys)
from lattica_b200.ntt import RingPlan

Q64 = 4294966657      # largest prime < 2^32 with q = 1 mod 128
Q256 = 4294962689     # largest prime < 2^32 with q = 1 mod 512
Q_RING = 4294967291   # 2^32 - 5, the reference's LaBRADOR modulus: no NTT

JL_ROWS = 256
BASE, LIMBS = 256, 4  # gadget base 2^8, 4 limbs cover a 32-bit word


def listed():
    return [
        # The plain Ajtai commitment: A 8 x 64, a batch of 64 ternary witnesses. The
        # smallest call a prover makes; launches and latency are all it costs.
        {"name": "commit_small", "kind": "commit", "rows": 8, "cols": 64, "batch": 64},
        # Batched ring products INTT(NTT(a) * b), b prepared: the headline throughput
        # workload, 3 GiB through HBM.
        {"name": "products_d64", "kind": "product", "d": 64, "polys": 1 << 22},
        # The same chain in the larger ring, d = 256.
        {"name": "products_d256", "kind": "product", "d": 256, "polys": 1 << 20},
        # A ring product with neither side prepared (forward of both, inverse of the
        # product), then one batch each way on its own: an odd number of polys.
        {"name": "ring_mul_d64", "kind": "ring_mul", "d": 64, "polys": 100003},
        # The Gram matrix of a smaller prover step whose length is no multiple of
        # anything: what a request stream of mixed sizes sends.
        {"name": "gram_ragged", "kind": "gram", "r": 30, "n": 1021},
        # One LaBRADOR prover round: inner commitments, Gram matrix, JL projection and
        # both decompositions, r = 64 vectors of n = 2048 polys, kappa = 16.
        {"name": "round", "kind": "round", "r": 64, "n": 2048, "kappa": 16, "ntt": True},
        # The round over q = 2^32 - 5, where R_q has no NTT.
        {"name": "round_no_ntt", "kind": "round", "r": 64, "n": 2048, "kappa": 16,
         "ntt": False},
        # The aggregation side of that round: the 256 conjugated JL evaluations.
        {"name": "jl_evals", "kind": "jl_evals", "r": 64, "n": 2048},
        # The end of the level: garbage h from the aggregated phis, amortized witness.
        {"name": "level_close", "kind": "close", "r": 64, "n": 2048},
        # The level's outer commitments u1 = B t + C g and u2 = D h.
        {"name": "outer_commit", "kind": "outer", "r": 64, "kappa": 16},
        # 4096 commitments of uneven length (log-uniform in [64, 8192]) and rank 8, 16
        # or 32, the largest batch a server collects.
        {"name": "uneven_batch", "kind": "batch", "instances": 4096, "n_hi": 8192},
        # The round's commitment key (A, B, C, D) expanded from its 32-byte seed.
        {"name": "key_from_seed", "kind": "key", "polys": 364544},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["commit", "product", "ring_mul", "gram", "round", "jl_evals", "close",
                       "outer", "batch", "key"])
    r, n = rng.randint(6, 64), _log_int(rng, 100, 2048)
    if kind == "commit":
        return {"kind": kind, "rows": rng.choice([8, 12, 16, 32]), "cols": _log_int(rng, 24, 2048),
                "batch": _log_int(rng, 5, 64)}
    if kind == "product":
        d = rng.choice([64, 256])
        return {"kind": kind, "d": d, "polys": _log_int(rng, 1000, (1 << 28) // d)}
    if kind == "ring_mul":
        d = rng.choice([64, 256])
        return {"kind": kind, "d": d, "polys": _log_int(rng, 200, (1 << 26) // d)}
    if kind == "round":
        return {"kind": kind, "r": r, "n": n, "kappa": rng.randint(4, 16),
                "ntt": rng.random() < 0.6}
    if kind == "outer":
        return {"kind": kind, "r": r, "kappa": rng.randint(4, 16)}
    if kind == "batch":
        return {"kind": kind, "instances": _log_int(rng, 40, 4096),
                "n_hi": _log_int(rng, 500, 8192)}
    if kind == "key":
        return {"kind": kind, "polys": _log_int(rng, 500, 364544)}
    return {"kind": kind, "r": r, "n": n}  # gram, jl_evals, close


# ---- inputs ------------------------------------------------------------------


def _device():
    return torch.device("cuda:0" if torch.cuda.is_available() else "cpu")


def _rng(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _uniform(g, q, shape):
    """Uniform canonical words."""
    return torch.randint(0, q, shape, dtype=torch.int64, device=_device(),
                         generator=g).to(torch.int32)


def _short(g, q, shape, bound):
    """Coefficients uniform in [-bound, bound] as Montgomery words."""
    v = torch.randint(-bound, bound + 1, shape, dtype=torch.int64, device=_device(), generator=g)
    return (((v % q) * ((1 << 32) % q)) % q).to(torch.int32)


def _seed_bytes(seed):
    return np.random.default_rng(int(seed)).bytes(32)


def _modulus(case):
    if case["kind"] == "round" and not case["ntt"]:
        return Q_RING
    return Q256 if case.get("d") == 256 else Q64


def _inputs(case, seed):
    """The tensors of one case, from the seed alone."""
    kind, q, g = case["kind"], _modulus(case), _rng(seed)
    if kind == "commit":
        return {"A": _uniform(g, q, (case["rows"], case["cols"], 64)),
                "s": _short(g, q, (case["batch"], case["cols"], 64), 1)}
    if kind in ("product", "ring_mul"):
        shape = (case["polys"], case["d"])
        return {"a": _uniform(g, q, shape), "b": _uniform(g, q, shape)}
    if kind in ("gram", "jl_evals", "close", "round"):
        r, n = case["r"], case["n"]
        x = {"s": _short(g, q, (r, n, 64), 1 << 11)}
        if kind == "close":
            x["phi"] = _uniform(g, q, (r, n, 64))
            x["c"] = _short(g, q, (r, 64), 2)
        if kind == "round":
            x["A"] = _uniform(g, q, (case["kappa"], n, 64))
        return x
    if kind == "outer":
        kappa, t_len = case["kappa"], case["r"] * case["kappa"] * LIMBS
        g_len = garbage_count(case["r"]) * LIMBS
        mats = {k: _uniform(g, q, (kappa, cols, 64))
                for k, cols in (("B", t_len), ("C", g_len), ("D", g_len))}
        limbs = {k: _short(g, q, (cols, 64), BASE // 2)
                 for k, cols in (("t", t_len), ("g", g_len), ("h", g_len))}
        return {**mats, **limbs}
    if kind == "batch":
        ranks = (8, 16, 32)
        # the batch's shape belongs to the case, its words to the seed
        items, s_polys, t_polys = sample_uneven_instances(case["instances"], 11, 64,
                                                          case["n_hi"], ranks)
        return {"items": items, "t_polys": t_polys,
                "mats": [_uniform(g, q, (m, case["n_hi"], 64)) for m in ranks],
                "s": _short(g, q, (s_polys, 64), 1)}
    return {}


def prepare(case, seed):
    kind, q = case["kind"], _modulus(case)
    st = {"kind": kind, **_inputs(case, seed)}
    if kind == "round" and not case["ntt"]:
        plan = RingPlan(q, 64)
    else:
        plan = twisted_ntt_plan(q, case.get("d", 64))
    st["plan"] = plan
    if kind == "commit":
        st["key"] = PreparedMatrix(plan, st["A"], case["rows"], case["cols"])
    elif kind == "round":
        st["key"] = CommitKey(plan, st["A"], case["kappa"], case["n"])
        st["seed"] = _seed_bytes(seed)
    elif kind == "jl_evals":
        st["jl"] = JLMatrix.from_seed(JL_ROWS, case["n"] * 64, _seed_bytes(seed))
        st["s"] = st["s"].reshape(case["r"], case["n"] * 64)
        st["r"] = case["r"]
    elif kind == "outer":
        st["key"] = OuterCommitKey(plan, st["B"], st["C"], st["D"], case["kappa"], case["kappa"],
                                   st["t"].shape[0], st["g"].shape[0], st["h"].shape[0])
    elif kind == "batch":
        st["mats"] = [PreparedMatrix(plan, m, m.shape[0], m.shape[1]) for m in st["mats"]]
        st["batch"] = UnevenCommitBatch(plan, st["mats"], st["items"])
        st["t"] = torch.empty((st["t_polys"], 64), dtype=torch.int32, device=_device())
    elif kind == "key":
        st["seed"], st["polys"] = _seed_bytes(seed), case["polys"]
    return st


def run(st):
    kind, plan = st["kind"], st["plan"]
    if kind == "commit":
        return st["key"].mul_vec(st["s"])
    if kind == "product":
        return plan.ntt_mul_inverse(st["a"], st["b"])
    if kind == "ring_mul":
        prod = poly_mul_ntt(st["a"], st["b"], plan.q)
        evals, coeffs = st["a"].clone(), st["b"].clone()
        plan.forward_in_place(evals)
        plan.inverse_in_place(coeffs)
        return {"prod": prod, "evals": evals, "coeffs": coeffs}
    if kind == "gram":
        return compute_garbage_g(plan, st["s"])
    if kind == "round":
        out = prover_round_dev(st["key"], st["s"], BASE, LIMBS, BASE, LIMBS, st["seed"], JL_ROWS)
        return {"t_limbs": out.t_limbs, "g": out.g, "g_limbs": out.g_limbs, "p": out.p}
    if kind == "jl_evals":
        return st["jl"].conjugated_evals(plan, st["s"], st["r"], 64)
    if kind == "close":
        return {"h": compute_garbage_h(plan, st["s"], st["phi"]),
                "z": amortize_witness(plan, st["s"], st["c"])}
    if kind == "outer":
        return {"u1": st["key"].outer_commit_u1_slice(st["t"], st["g"]),
                "u2": st["key"].outer_commit_u2_slice(st["h"])}
    if kind == "batch":
        return st["batch"].commit_dev(st["s"], st["t"])
    return sample_uniform_polys(plan, st["seed"], st["polys"], device=_device())


# ---- what a pass cannot do without ---------------------------------------------


def work(case):
    """Bytes: every input read once, every output written once. Operations: two
    per multiply-add of a d log d transform and of the dense products over
    evaluations; the JL entries' additions (and their keystream, about 1000
    integer operations per 64-byte block); the sampler's keystream."""
    kind, d = case["kind"], case.get("d", 64)
    poly = 4 * d
    ntt = 2.0 * d * math.log2(d)
    block = 1000.0
    if kind == "commit":
        m, n, b = case["rows"], case["cols"], case["batch"]
        return {"bytes": poly * (m * n + b * n + b * m),
                "flops": ntt * b * (m + n) + 2.0 * d * b * m * n}
    if kind == "product":
        return {"bytes": 3.0 * poly * case["polys"], "flops": (2 * ntt + 2 * d) * case["polys"]}
    if kind == "ring_mul":
        return {"bytes": 7.0 * poly * case["polys"], "flops": (5 * ntt + 2 * d) * case["polys"]}
    if kind == "key":
        return {"bytes": poly * case["polys"], "flops": block * case["polys"] * d / 8}
    if kind == "outer":
        kappa, t = case["kappa"], case["r"] * case["kappa"] * LIMBS
        cols = t + 2 * garbage_count(case["r"]) * LIMBS
        return {"bytes": poly * (kappa * cols + cols + 2 * kappa),
                "flops": ntt * cols + 2.0 * d * kappa * cols}
    if kind == "batch":
        mean_n = (case["n_hi"] - 64) / math.log(case["n_hi"] / 64)
        k, m = case["instances"], 56 / 3
        return {"bytes": poly * (k * (mean_n + m) + 56 * case["n_hi"]),
                "flops": k * (ntt * (mean_n + m) + 2.0 * d * mean_n * m)}
    r, n, pairs = case["r"], case["n"], garbage_count(case["r"])
    if kind == "gram":
        return {"bytes": poly * (r * n + pairs), "flops": ntt * (r * n + pairs) + 2.0 * d * pairs * n}
    if kind == "close":
        return {"bytes": poly * (2 * r * n + r + pairs + n),
                "flops": ntt * (2 * r * n + pairs + n) + 2.0 * d * (r * r + r) * n}
    cols = r * n * d
    if kind == "jl_evals":
        return {"bytes": 4 * cols + 4 * JL_ROWS * d, "flops": cols * (block + JL_ROWS * d)}
    m = case["kappa"]
    return {"bytes": poly * (r * n + m * n + LIMBS * m * r + (1 + LIMBS) * pairs) + 4 * JL_ROWS,
            "flops": ntt * (r * n + r * m + pairs) + 2.0 * d * (m * r + pairs) * n
            + cols * (block + JL_ROWS)}


# ---- the same results from plain arithmetic ------------------------------------


def _mulmod(a, b, q):
    """a * b mod q for 0 <= a, b < 2^32 in int64."""
    return ((a * (b >> 16) % q) * 65536 + a * (b & 0xFFFF)) % q


def _matmul_mod(x, y, q):
    """x @ y mod q for words below 2^32: four float64 products of 16-bit halves,
    each sum below 2^53 (up to 2^21 terms)."""
    xs = (x & 0xFFFF).double(), (x >> 16).double()
    ys = (y & 0xFFFF).double(), (y >> 16).double()
    part = lambda i, j: (xs[i] @ ys[j]).to(torch.int64) % q
    hi, mid, lo = part(1, 1), (part(0, 1) + part(1, 0)) % q, part(0, 0)
    return (((hi * 65536 + mid) % q) * 65536 + lo) % q


def _wide(x):
    return x.to(torch.int64) & 0xFFFFFFFF


def _narrow(x):
    return x.to(torch.int32)


def _psi(q, d):
    """The primitive 2d-th root g^((q-1)/2d), g the smallest generator mod q."""
    m, primes, f = q - 1, [], 2
    while f * f <= m:
        if m % f == 0:
            primes.append(f)
            while m % f == 0:
                m //= f
        f += 1
    primes += [m] if m > 1 else []
    g = 2
    while any(pow(g, (q - 1) // p, q) == 1 for p in primes):
        g += 1
    return pow(g, (q - 1) // (2 * d), q)


def _transforms(q, d):
    """(forward, inverse) matrices, to be multiplied from the right: slot j of the
    forward is sum_k x_k psi^((2j+1) k)."""
    psi = _psi(q, d)
    powers = torch.tensor([pow(psi, e, q) for e in range(2 * d)], device=_device())
    j, k = torch.meshgrid(torch.arange(d), torch.arange(d), indexing="ij")
    e = ((2 * j + 1) * k).to(_device())
    inv = _mulmod(powers[(-e) % (2 * d)], torch.tensor(pow(d, -1, q), device=_device()), q)
    return powers[e % (2 * d)].T.contiguous(), inv


def _ring_sums(x, y, q):
    """sum_k x[m, k] * y[n, k] in Z_q[X]/(X^d + 1) as Montgomery words: (M, N, d)
    from (M, K, d) and (N, K, d), the schoolbook rule as one matrix product."""
    (m, k, d), n = x.shape, y.shape[0]
    u, c = torch.meshgrid(torch.arange(d), torch.arange(d), indexing="ij")
    at, wraps = ((c - u) % d).to(x.device), (c < u).to(x.device)
    out = torch.zeros((m, n * d), dtype=torch.int64, device=x.device)
    step = max(1, (1 << 26) // (n * d * d))
    for k0 in range(0, k, step):
        yk = y[:, k0:k0 + step][:, :, at]                     # (N, k, u, c)
        yk = torch.where(wraps, (q - yk) % q, yk).permute(1, 2, 0, 3).reshape(-1, n * d)
        out = (out + _matmul_mod(x[:, k0:k0 + step].reshape(m, -1), yk, q)) % q
    r_inv = torch.tensor(pow(1 << 32, -1, q), device=x.device)
    return _mulmod(out, r_inv, q).reshape(m, n, d)


def _balanced(polys, q):
    """Centered base-2^8 limbs of (P, d) words, as words (P * limbs, d)."""
    v = _mulmod(polys, torch.tensor(pow(1 << 32, -1, q), device=polys.device), q)
    v = torch.where(v > q // 2, v - q, v)
    out = []
    for _ in range(LIMBS):
        limb = torch.fmod(v, BASE)
        limb = torch.where(limb > BASE // 2, limb - BASE, limb)
        limb = torch.where(limb < -(BASE // 2), limb + BASE, limb)
        out.append((limb % q) * ((1 << 32) % q) % q)
        v = torch.div(v - limb, BASE, rounding_mode="trunc")
    return torch.stack(out, 1).reshape(-1, polys.shape[1])


def _by_rows(fn, *xs):
    """fn over blocks of 2^17 rows (bounds the 64-bit temporaries)."""
    rows = range(0, xs[0].shape[0], 1 << 17)
    return torch.cat([_narrow(fn(*(_wide(x[i:i + (1 << 17)]) for x in xs))) for i in rows])


def exact(case, seed):
    kind, q = case["kind"], _modulus(case)
    if kind in ("jl_evals", "batch", "key"):  # keystreams, and 4096 separate products
        return None
    x = _inputs(case, seed)
    if kind in ("product", "ring_mul"):
        fwd, inv = _transforms(q, case["d"])
        r_inv = torch.tensor(pow(1 << 32, -1, q), device=_device())
        mont = lambda a, b: _mulmod(_mulmod(a, b, q), r_inv, q)
        ntt, intt = lambda a: _matmul_mod(a, fwd, q), lambda a: _matmul_mod(a, inv, q)
        if kind == "product":
            return _by_rows(lambda a, b: intt(mont(ntt(a), b)), x["a"], x["b"])
        return {"prod": _by_rows(lambda a, b: intt(mont(ntt(a), ntt(b))), x["a"], x["b"]),
                "evals": _by_rows(ntt, x["a"]), "coeffs": _by_rows(intt, x["b"])}
    x = {k: _wide(v) for k, v in x.items()}
    if kind == "commit":
        return _narrow(_ring_sums(x["s"], x["A"], q))
    if kind == "outer":
        dot = lambda mat, v: _ring_sums(x[v][None], x[mat], q)[0]
        return {"u1": _narrow((dot("B", "t") + dot("C", "g")) % q), "u2": _narrow(dot("D", "h"))}
    i, j = torch.triu_indices(case["r"], case["r"], device=_device())
    if kind == "close":
        cross = _ring_sums(x["phi"], x["s"], q)
        half = torch.tensor((q + 1) // 2, device=_device())
        z = _ring_sums(x["s"].transpose(0, 1), x["c"][None], q)[:, 0]
        return {"h": _narrow(_mulmod((cross[i, j] + cross[j, i]) % q, half, q)), "z": _narrow(z)}
    gram = _ring_sums(x["s"], x["s"], q)[i, j]
    if kind == "gram":
        return _narrow(gram)
    t = _ring_sums(x["s"], x["A"], q).reshape(-1, 64)
    return {"t_limbs": _narrow(_balanced(t, q)), "g": _narrow(gram),
            "g_limbs": _narrow(_balanced(gram, q)), "p": None}
