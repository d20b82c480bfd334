"""The work that a user of this framework has it do, as cases with sizes.

Each case is one call (or, for PLONK and Groth16, the call sequence of one prover step)
through the public Python binding: inputs on the device in Montgomery form where a prover
keeps them there, in page-locked host memory where the call takes host buffers. Every
output is exact: canonical point coordinates as bytes, field elements as four 64-bit limbs.
"""

import math

import numpy as np
import torch

from pyzkp_gb300 import _native as N
from pyzkp_gb300 import groth16 as G
from pyzkp_gb300.plugin import fixed_base_window

R = 21888242871839275222246405745257275088548364400416034343698204186575808495617
Q = 21888242871839275222246405745257275088696311157297823662689037894645226208583
MAC = 136  # 32-bit multiply-adds of one 8-limb Montgomery product


# ------------------------------------------------------------------------------------ cases
def listed():
    return [
        # the queries of a small circuit, canonical witness values straight from a frontend
        {"name": "msm_777_witness", "kind": "msm", "n": 777, "scalars": "witness", "mont": False},
        # the size the reference itself runs on the CPU (its benchmark's 4096-point MSM)
        {"name": "msm_4096", "kind": "msm", "n": 4096, "scalars": "uniform", "mont": True},
        # a witness commitment of a mid-sized circuit, size not a power of two
        {"name": "msm_100003_witness", "kind": "msm", "n": 100003, "scalars": "witness", "mont": True},
        # the headline: a polynomial commitment of 2^20 coefficients, bases resident
        {"name": "msm_2e20", "kind": "msm", "n": 1 << 20, "scalars": "uniform", "mont": True},
        # one MSM whose points and scalars arrive in host memory with the call
        {"name": "msm_host_300000", "kind": "msm_host", "n": 300000, "scalars": "uniform", "mont": False},
        # a proving key's query (n - 1 points) with its fixed-base rows
        {"name": "msm_fixed_65535", "kind": "msm_fixed", "n": 65535, "scalars": "uniform", "mont": True},
        # many commitments of mixed lengths in one call (KZG batch commit, several proofs)
        {"name": "msm_batch_64", "kind": "msm_batch", "count": 64, "lo": 10.0, "hi": 20.0, "mont": True},
        # Groth16's b-query over G2
        {"name": "msm_g2_65536", "kind": "msm_g2", "n": 65536, "scalars": "uniform", "mont": True},
        # the smallest transforms: a circuit of a few thousand rows, coefficients -> evaluations
        {"name": "ntt_2e12", "kind": "ntt", "log_n": 12, "mode": 0, "in_len": 4096},
        # the largest of the sweeps, the way back from a coset (the quotient's coefficients)
        {"name": "ntt_2e22_coset_inverse", "kind": "ntt", "log_n": 22, "mode": 3, "in_len": 1 << 22},
        # a Groth16 prover's batch: eight witnesses of one circuit
        {"name": "groth16_8x20000", "kind": "groth16", "m": 20000, "count": 8},
        # the PLONK quotient step: 15 coset NTTs n -> 4n, quotient, batch inverse, coset iNTT
        {"name": "plonk_quotient_2e17", "kind": "plonk", "log_n": 17},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(2.0 ** rng.uniform(lo, hi)))


def draw(rng):
    kind = rng.choice(["msm", "msm", "msm", "msm_host", "msm_fixed", "msm_batch", "msm_g2", "ntt", "ntt", "ntt",
                       "groth16", "plonk"])
    if kind in ("msm", "msm_host", "msm_fixed", "msm_g2"):
        hi = {"msm": 21.0, "msm_host": 20.0, "msm_fixed": 20.0, "msm_g2": 19.0}[kind]
        n = _log_uniform(rng, 8.0, hi)
        return {"kind": kind, "n": n, "scalars": rng.choice(["uniform", "witness"]),
                "mont": False if kind == "msm_host" else rng.random() < 0.7}
    if kind == "msm_batch":
        lo = rng.uniform(8.0, 14.0)
        return {"kind": kind, "count": rng.randint(2, 64), "lo": lo, "hi": rng.uniform(lo, 19.5),
                "mont": rng.random() < 0.7}
    if kind == "ntt":
        log_n = rng.randint(8, 22)
        n = 1 << log_n
        mode = rng.randint(0, 3)
        # a forward transform may get fewer coefficients than the domain has points
        in_len = rng.choice([n, n // 4, n - rng.randint(1, n // 8)]) if mode in (0, 2) else n
        return {"kind": kind, "log_n": log_n, "mode": mode, "in_len": in_len}
    if kind == "groth16":
        return {"kind": kind, "m": _log_uniform(rng, 8.0, 16.0), "count": rng.randint(1, 8)}
    return {"kind": kind, "log_n": rng.randint(8, 18)}


# ----------------------------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _words(g, *shape):
    return torch.randint(-(1 << 63), (1 << 63) - 1, shape, generator=g, device="cuda", dtype=torch.int64)


def _uniform(g, n):
    """n field elements (canonical, below r) as int64[n, 4] little-endian limbs."""
    v = _words(g, n, 4)
    v[:, 3] = torch.randint(0, R >> 192, (n,), generator=g, device="cuda", dtype=torch.int64)
    return v


def _witness(g, n):
    """Witness-like: 10% in {0, 1}, 60% below 2^64, the rest uniform."""
    v = _uniform(g, n)
    kind = torch.rand(n, generator=g, device="cuda")
    small, bit = kind < 0.70, kind < 0.10
    v[small, 1:] = 0
    v[bit, 0] = torch.randint(0, 2, (n,), generator=g, device="cuda", dtype=torch.int64)[bit]
    return v


def _scalars(g, n, how):
    return _witness(g, n) if how == "witness" else _uniform(g, n)


def _dlogs(seed, n):
    """Discrete logarithms of the bases P_i = [k_i] G (not zero)."""
    k = _uniform(_generator(seed * 2 + 1), n)
    k[:, 0] |= 1
    return k


def _view(ctx, t):
    return N.DeviceArray(ctx, t.numel() * t.element_size(), ptr=t.data_ptr(), owned=False)


def _to_mont(ctx, t):
    d = _view(ctx, t)
    ctx.fr_to_mont(d, d, t.shape[0])
    return d


def _g1_points(ctx, seed, n):
    k = _dlogs(seed, n)
    xy = torch.empty((n, 8), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    ctx.g1_fixed_base_mul(G.G1_GEN, _view(ctx, k), n, _view(ctx, xy))
    ctx.sync()
    return xy


def _batch_sizes(case):
    c = case["count"]
    return [int(round(2.0 ** (case["lo"] + (case["hi"] - case["lo"]) * (i + 0.5) / c))) for i in range(c)]


def prepare(case, seed):
    ctx = N.default_context()
    kind, s = case["kind"], {"ctx": ctx, "case": case}
    g = _generator(seed * 2)
    if kind in ("msm", "msm_fixed", "msm_g2"):
        n = case["n"]
        sc = _scalars(g, n, case["scalars"])
        if kind == "msm_g2":
            k = _dlogs(seed, n)
            xy = torch.empty((n, 16), dtype=torch.int64, device="cuda")
            torch.cuda.synchronize()
            ctx.g2_fixed_base_mul(G.G2_GEN, _view(ctx, k), n, _view(ctx, xy))
            ctx.sync()
            s["bases"] = ctx.bases_g2_from_device(_view(ctx, xy), n)
        else:
            s["bases"] = ctx.bases_from_device(_view(ctx, _g1_points(ctx, seed, n)), n)
        if kind == "msm_fixed":
            ctx.bases_precompute(s["bases"], fixed_base_window(n))
        torch.cuda.synchronize()
        s["held"], s["scalars"] = sc, _to_mont(ctx, sc) if case["mont"] else _view(ctx, sc)
    elif kind == "msm_host":
        n = case["n"]
        s["xy"] = N.pinned_copy(_g1_points(ctx, seed, n).cpu().numpy().view(np.uint64))
        s["scalars"] = N.pinned_copy(_scalars(g, n, case["scalars"]).cpu().numpy().view(np.uint64))
    elif kind == "msm_batch":
        s["sizes"] = _batch_sizes(case)
        most = max(s["sizes"])
        s["bases"] = ctx.bases_from_device(_view(ctx, _g1_points(ctx, seed, most)), most)
        s["held"] = _uniform(g, sum(s["sizes"]))
        torch.cuda.synchronize()
        flat = _to_mont(ctx, s["held"]) if case["mont"] else _view(ctx, s["held"])
        at = np.cumsum([0] + s["sizes"][:-1])
        s["scalars"] = [N.DeviceArray(ctx, 32 * m, ptr=flat.ptr + 32 * int(o), owned=False)
                        for o, m in zip(at, s["sizes"])]
    elif kind == "ntt":
        n = 1 << case["log_n"]
        s["held"] = _uniform(g, case["in_len"])
        s["out"] = torch.empty((n, 4), dtype=torch.int64, device="cuda")
        s["in_view"], s["out_view"] = _view(ctx, s["held"]), _view(ctx, s["out"])
        s["omega"] = G.omega_for_size(n)
    elif kind == "groth16":
        m, count = case["m"], case["count"]
        s["prover"] = G.Prover(ctx)
        s["key"] = G.setup(ctx, G.diagonal_r1cs(m), G.Trapdoors.seeded(seed))
        rnd = np.random.default_rng(seed)
        s["requests"] = [
            G.Request(s["key"], G.pin_witness(G.diagonal_witness(ctx, m, seed * 16 + j)[0]),
                      int.from_bytes(rnd.bytes(31), "little"), int.from_bytes(rnd.bytes(31), "little"))
            for j in range(count)]
    elif kind == "plonk":
        n = 1 << case["log_n"]
        m, shift = 4 * n, 7 + seed % 1000
        s["held"] = [_uniform(g, n) for _ in range(15)]
        s["ext"] = [torch.empty((m, 4), dtype=torch.int64, device="cuda") for _ in range(15)]
        s["num"], s["zh"], s["inv"], s["t"] = (torch.empty((m, 4), dtype=torch.int64, device="cuda")
                                              for _ in range(4))
        om_n, s["omega"], s["shift"] = G.omega_for_size(n), G.omega_for_size(m), shift
        s["shift_n"] = pow(shift, n, R)
        rnd = np.random.default_rng(seed)
        s["challenges"] = [int.from_bytes(rnd.bytes(31), "little") for _ in range(5)]
        s["ext_views"] = [_view(ctx, t) for t in s["ext"]]
        s["views"] = {k: _view(ctx, s[k]) for k in ("num", "zh", "inv", "t")}
        # z is evaluated at the shifted point too (polynomial 13)
        s["jobs"] = [(N.NTT_COSET_EVALS_FROM_COEFFS, s["ext_views"][j], _view(ctx, s["held"][j]), n,
                      case["log_n"] + 2, s["omega"], shift * om_n % R if j == 13 else shift) for j in range(15)]
    else:
        raise ValueError("unknown kind %r" % kind)
    torch.cuda.synchronize()
    ctx.sync()
    return s


# --------------------------------------------------------------------------------- one pass
def _point(p, coords):
    """A point's canonical coordinates as bytes; infinity as zeros."""
    if p is None:
        return np.zeros(32 * coords, dtype=np.uint8)
    flat = [c for v in p for c in (v if isinstance(v, tuple) else (v,))]
    return np.frombuffer(b"".join(c.to_bytes(32, "little") for c in flat), dtype=np.uint8)


def run(s):
    ctx, case = s["ctx"], s["case"]
    kind = case["kind"]
    if kind in ("msm", "msm_fixed"):
        return _point(ctx.msm_g1(s["bases"], s["scalars"], case["n"], scalars_mont=case["mont"]), 2)
    if kind == "msm_g2":
        return _point(ctx.msm_g2(s["bases"], s["scalars"], case["n"], scalars_mont=case["mont"]), 4)
    if kind == "msm_host":
        return _point(ctx.msm_g1_host(s["xy"], s["scalars"], case["n"], scalars_mont=False), 2)
    if kind == "msm_batch":
        pts = ctx.msm_g1_batch(s["bases"], s["scalars"], s["sizes"], scalars_mont=case["mont"])
        return np.stack([_point(p, 2) for p in pts])
    if kind == "ntt":
        ctx.ntt(case["mode"], s["out_view"], s["in_view"], case["in_len"], case["log_n"], s["omega"],
                G.COSET_SHIFT if case["mode"] >= 2 else 1)
        return s["out"]
    if kind == "groth16":
        proofs = s["prover"].prove_batch(s["requests"])
        return np.stack([np.concatenate([_point(p.a, 2), _point(p.b, 4), _point(p.c, 2)]) for p in proofs])
    v, n = s["views"], 1 << case["log_n"]
    m = 4 * n
    ctx.ntt_batch(s["jobs"])
    ctx.plonk_quotient_evals(s["ext_views"], m, n, s["omega"], s["shift"], s["shift_n"], *s["challenges"], v["num"],
                             v["zh"])
    ctx.fr_batch_inv(v["inv"], v["zh"], m)
    ctx.fr_mul(v["t"], v["num"], v["inv"], m)
    ctx.ntt(N.NTT_COSET_COEFFS_FROM_EVALS, v["t"], v["t"], m, case["log_n"] + 2, s["omega"], s["shift"])
    return {"evals": s["ext"], "num": s["num"], "t": s["t"]}


# ------------------------------------------------------------------------------------- work
def _msm_ops(n, g2=False):
    """Operations (2 per multiply-add) of n 254-bit scalars: 254 / log2(n) additions a point
    (Pippenger's bound), 10 products an addition, three base-field products each over G2."""
    return n * 254.0 / max(1.0, math.log2(max(2, n))) * 10 * MAC * 2 * (3 if g2 else 1)


def _ntt_ops(log_n):
    return (1 << log_n) / 2 * log_n * MAC * 2


def work(case):
    kind = case["kind"]
    if kind in ("msm", "msm_host", "msm_fixed"):
        return {"bytes": case["n"] * 96 + 64, "flops": _msm_ops(case["n"])}
    if kind == "msm_g2":
        return {"bytes": case["n"] * 160 + 128, "flops": _msm_ops(case["n"], True)}
    if kind == "msm_batch":
        sizes = _batch_sizes(case)
        return {"bytes": 32 * sum(sizes) + 64 * max(sizes) + 64 * len(sizes), "flops": sum(map(_msm_ops, sizes))}
    if kind == "ntt":
        return {"bytes": 32 * ((1 << case["log_n"]) + case["in_len"]), "flops": _ntt_ops(case["log_n"])}
    if kind == "groth16":
        m, c = case["m"], case["count"]
        lg = (m - 1).bit_length()
        g1 = _msm_ops(m) * 2 + _msm_ops(3 * m) + _msm_ops((1 << lg) - 1)  # a, b, l and h queries
        return {"bytes": c * 96 * m + 64 * (6 * m) + 128 * m, "flops": c * (g1 + _msm_ops(m, True) + 7 * _ntt_ops(lg))}
    n = 1 << case["log_n"]
    ops = 16 * _ntt_ops(case["log_n"] + 2) + 4 * n * (23 + 4) * MAC * 2
    return {"bytes": 32 * n * (15 + 4 * (15 + 2)), "flops": ops}


# ------------------------------------------------------------------------------------ exact
def _ints(t):
    b = t.cpu().numpy().tobytes()
    return [int.from_bytes(b[i:i + 32], "little") for i in range(0, len(b), 32)]


def _g1_add(p, q):
    if p is None or q is None:
        return q if p is None else p
    if p[0] == q[0]:
        if (p[1] + q[1]) % Q == 0:
            return None
        lam = 3 * p[0] * p[0] * pow(2 * p[1], -1, Q)
    else:
        lam = (q[1] - p[1]) * pow(q[0] - p[0], -1, Q)
    x = (lam * lam - p[0] - q[0]) % Q
    return x, (lam * (p[0] - x) - p[1]) % Q


def _g1_mul(k):
    acc, p = None, (1, 2)
    while k:
        if k & 1:
            acc = _g1_add(acc, p)
        p, k = _g1_add(p, p), k >> 1
    return acc


def _transform(x, omega):
    """Values of the polynomial x at the powers of omega, by the definition's even / odd halves."""
    n = len(x)
    if n == 1:
        return x
    even, odd = _transform(x[0::2], omega * omega % R), _transform(x[1::2], omega * omega % R)
    w, lo, hi = 1, [], []
    for a, b in zip(even, odd):
        b = b * w % R
        lo.append((a + b) % R)
        hi.append((a - b) % R)
        w = w * omega % R
    return lo + hi


def exact(case, seed):
    """[sum k_i s_i] G for a G1 MSM over P_i = [k_i] G; small transforms in Python integers
    (a transform is linear, so it may take the Montgomery forms as they are)."""
    g = _generator(seed * 2)
    if case["kind"] in ("msm", "msm_host", "msm_fixed") and case["n"] <= 1 << 21:
        n = case["n"]
        total = sum(a * b for a, b in zip(_ints(_scalars(g, n, case["scalars"])), _ints(_dlogs(seed, n)))) % R
        return _point(_g1_mul(total), 2)
    if case["kind"] == "ntt" and case["log_n"] <= 14:
        n, mode = 1 << case["log_n"], case["mode"]
        x = _ints(_uniform(g, case["in_len"]))
        x += [0] * (n - len(x))
        omega = pow(19103219067921713944291392827692070036145651957329286315305642004821462161904,
                    (1 << 28) // n, R)
        shift = 5 if mode >= 2 else 1
        if mode in (0, 2):
            y = _transform([v * pow(shift, i, R) % R for i, v in enumerate(x)], omega)
        else:
            k, back = pow(n, -1, R), pow(shift, -1, R)
            y = [v * k * pow(back, i, R) % R for i, v in enumerate(_transform(x, pow(omega, -1, R)))]
        return torch.from_numpy(np.frombuffer(b"".join(v.to_bytes(32, "little") for v in y), dtype=np.int64)
                                .reshape(n, 4).copy())
    return None
