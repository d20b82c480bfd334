"""MSMs whose partial sums meet in the special cases of the point addition inside the
reduction trees (a point held by four lanes): equal points (doubling), opposite points
(infinity) and infinity on either side, at sizes around the trees' edges. Bases are
multiples +-1, +-2 of one point (or infinity), so the exact answer is [sum k_i s_i] G."""

import numpy as np
import pytest

from oracle import oracle as O
from pyzkp_gb300 import _native as N
from pyzkp_gb300 import groth16 as G
from pyzkp_gb300 import synth

pytestmark = pytest.mark.gpu
R = synth.FR_MODULUS


@pytest.fixture(scope="module")
def ctx():
    return N.default_context()


def _case(pattern: str, n: int, seed: int):
    """(discrete logs k_i of the bases, scalars s_i) as Python ints."""
    rng = np.random.default_rng(seed)
    if pattern == "equal":
        k = [1] * n
    elif pattern == "opposite":
        k = [1 if i % 2 == 0 else R - 1 for i in range(n)]
    else:  # mixed: a few multiples, and infinity
        k = [[1, R - 1, 2, R - 2, 0][int(v)] for v in rng.integers(0, 5, n)]
    small = rng.integers(1, 4, n)
    wide = synth.limbs_to_ints(synth.fr_uniform(seed, n))
    s = [int(a) if i % 3 else b for i, (a, b) in enumerate(zip(small, wide))]
    if pattern == "opposite":
        s = [s[i - i % 2] for i in range(n)]  # pairs cancel
    return k, s


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 777, 4097, 20000])
@pytest.mark.parametrize("pattern", ["equal", "opposite", "mixed"])
def test_g1_special_cases(ctx, pattern, n):
    k, s = _case(pattern, n, 1000 + n)
    dk = ctx.to_device(synth.ints_to_limbs(k))
    xy = ctx.alloc(n * 64)
    ctx.g1_fixed_base_mul((1, 2), dk, n, xy)
    bases = ctx.bases_from_device(xy, n)
    d = ctx.to_device(synth.ints_to_limbs(s))
    want = N.host_g1_mul((1, 2), sum(a * b for a, b in zip(k, s)) % R)
    for c in (0, 4, 8, 13):
        assert ctx.msm_g1(bases, d, n, scalars_mont=False, window_bits=c) == want
    assert ctx.msm_g1_batch(bases, [d, d], [n, max(1, n // 2)], scalars_mont=False)[0] == want


@pytest.mark.parametrize("n", [1, 33, 777, 5000])
@pytest.mark.parametrize("pattern", ["equal", "opposite", "mixed"])
def test_g2_special_cases(ctx, pattern, n):
    k, s = _case(pattern, n, 2000 + n)
    dk = ctx.to_device(synth.ints_to_limbs(k))
    xy = ctx.alloc(n * 128)
    ctx.g2_fixed_base_mul(G.G2_GEN, dk, n, xy)
    bases = ctx.bases_g2_from_device(xy, n)
    d = ctx.to_device(synth.ints_to_limbs(s))
    want = N.host_g2_mul(G.G2_GEN, sum(a * b for a, b in zip(k, s)) % R)
    for c in (0, 6, 12):
        assert ctx.msm_g2(bases, d, n, scalars_mont=False, window_bits=c) == want


@pytest.mark.parametrize("n", [100, 3000])
def test_fixed_base_special_cases(ctx, n):
    k, s = _case("mixed", n, 3000 + n)
    dk = ctx.to_device(synth.ints_to_limbs(k))
    xy = ctx.alloc(n * 64)
    ctx.g1_fixed_base_mul((1, 2), dk, n, xy)
    d = ctx.to_device(synth.ints_to_limbs(s))
    want = N.host_g1_mul((1, 2), sum(a * b for a, b in zip(k, s)) % R)
    for c in (8, 13, 17):
        bases = ctx.bases_from_device(xy, n)
        ctx.bases_precompute(bases, c)
        assert ctx.msm_g1(bases, d, n, scalars_mont=False) == want


def test_oracle_agrees(ctx):
    """The known-answer rule above against the oracle's Pippenger on one mixed case."""
    n = 65
    k, s = _case("mixed", n, 5)
    pts = O.g1_fixed_base_mul(O.G1_GENERATOR, synth.ints_to_limbs(k))
    exp = O.affine_to_ints(O.msm_pippenger(pts, synth.ints_to_limbs(s), O.msm_window_rule(n)))
    assert exp == N.host_g1_mul((1, 2), sum(a * b for a, b in zip(k, s)) % R)
