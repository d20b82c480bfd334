"""Fr values whose bits are not below r: the vector operations take them as their residues."""

import numpy as np
import pytest

from oracle import oracle as O
from pyzkp_gb300 import _native as N
from pyzkp_gb300 import groth16 as G
from pyzkp_gb300 import synth

pytestmark = pytest.mark.gpu
R = synth.FR_MODULUS
RINV = pow(1 << 256, -1, R)


@pytest.fixture(scope="module")
def ctx():
    return N.default_context()


def _raw_up(ctx, raw):
    assert all(0 <= v < 1 << 256 for v in raw)
    return ctx.to_device(np.array([[(v >> (64 * j)) & (2**64 - 1) for j in range(4)] for v in raw], dtype=np.uint64))


def _down(ctx, d, n):
    t = ctx.alloc(n * 32)
    ctx.fr_from_mont(t, d, n)
    return synth.limbs_to_ints(t.download().view("<u8").reshape(n, 4))


@pytest.mark.parametrize("n", [1, 33, 512, 700])
def test_batch_inverse(ctx, n):
    """Multiples of r are zeros and touch no neighbour."""
    raw = synth.limbs_to_ints(synth.fr_uniform(900 + n, n))
    for i in range(0, n, 3):
        raw[i] = R * ((i // 3 + 1) % 6) if i % 2 == 0 else raw[i] + R * (i % 5)
    out = ctx.alloc(n * 32)
    ctx.fr_batch_inv(out, _raw_up(ctx, raw), n)
    assert _down(ctx, out, n) == [pow(v * RINV, -1, R) if v % R else 0 for v in raw]


def _unreduced(n, seed):
    """Residues in the top 2r of the 256 bits, with multiples of r among them."""
    raw = synth.limbs_to_ints(synth.fr_uniform(seed, n))
    return [(v if i % 7 else 0) + R * ((2**256 - 1 - v) // R - i % 2) for i, v in enumerate(raw)]


@pytest.mark.parametrize("n", [1, 257, 4096])
def test_vector_products(ctx, n):
    a, b, s = _unreduced(n, 1), _unreduced(n, 2), 12345678901234567890
    da, db, out = _raw_up(ctx, a), _raw_up(ctx, b), ctx.alloc(n * 32)
    ctx.fr_mul(out, da, db, n)
    assert _down(ctx, out, n) == [x * y * RINV * RINV % R for x, y in zip(a, b)]
    ctx.fr_scale(out, da, s, n)
    assert _down(ctx, out, n) == [x * RINV * s % R for x in a]


@pytest.mark.parametrize("log_n", [3, 8, 10, 13, 18])
def test_coset_ntt(ctx, log_n):
    n, shift = 1 << log_n, 5
    om = O.omega_for_size(n)
    raw = _unreduced(n, 30 + log_n)
    out = ctx.alloc(n * 32)
    ctx.ntt(N.NTT_COSET_EVALS_FROM_COEFFS, out, _raw_up(ctx, raw), n, log_n, om, shift)
    want = O.ntt_op(N.NTT_COSET_EVALS_FROM_COEFFS, synth.ints_to_limbs([v * RINV % R for v in raw]), n, om, shift)
    assert _down(ctx, out, n) == synth.limbs_to_ints(want)


def test_quotient(ctx):
    """Inputs below 4r, which the sums of the quotient kernel still hold."""
    log_m = 9
    m, n = 1 << log_m, 1 << (log_m - 2)
    om, shift = G.omega_for_size(m), 11
    shift_n = pow(shift, n, R)
    par = [synth.limbs_to_ints(synth.fr_uniform(70 + j, 1))[0] for j in range(5)]
    vecs = [synth.limbs_to_ints(synth.fr_uniform(80 + j, m)) for j in range(15)]
    num, zh = ctx.alloc(m * 32), ctx.alloc(m * 32)
    got = []
    for k in (0, 3):
        ins = [_raw_up(ctx, [v + R * (k if j in (0, 1, 2, 3, 5, 6, 7, 8) else 0) for v in vec])
               for j, vec in enumerate(vecs)]
        ctx.plonk_quotient_evals(ins, m, n, om, shift, shift_n, *par, num, zh)
        got.append((_down(ctx, num, m), _down(ctx, zh, m)))
    assert got[0] == got[1]
