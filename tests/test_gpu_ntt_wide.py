"""The wide form of the NTT passes (radix-8 steps in registers, taken by launches of at least
2^18 elements) against the narrow form and the oracle: every radix's remainder by 3, tiles of
one and of many columns, every mode, in one batch and alone."""

import numpy as np
import pytest

from oracle import oracle as O
from pyzkp_gb300 import _native as N
from pyzkp_gb300 import groth16 as G
from pyzkp_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return N.Context(0)


def _data(ctx, n, seed):
    d = ctx.to_device(synth.fr_uniform(seed, n))
    ctx.fr_to_mont(d, d, n)
    return d


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_batch_matches_single_transforms(ctx, mode):
    """2^0 .. 2^17 in one batch of more than 2^18 elements (wide) against one call each (narrow)."""
    logs = list(range(18)) + [17]
    ins = [_data(ctx, 1 << lg, 100 * mode + lg) for lg in logs]
    outs = [ctx.alloc(32 << lg) for lg in logs]
    shift = 5 if mode >= 2 else 1
    lens = [(1 << lg) - (lg > 3 and mode in (0, 2)) for lg in logs]  # forward: one coefficient short
    ctx.ntt_batch([(mode, o, d, m, lg, G.omega_for_size(1 << lg), shift)
                   for o, d, m, lg in zip(outs, ins, lens, logs)])
    for o, d, m, lg in zip(outs, ins, lens, logs):
        want = ctx.alloc(32 << lg)
        ctx.ntt(mode, want, d, m, lg, G.omega_for_size(1 << lg), shift)
        assert (o.download() == want.download()).all(), lg


@pytest.mark.parametrize("split", [(9, 9), (7, 11), (11, 7), (8, 10), (6, 6, 6), (1, 11, 6), (2, 5, 11)])
def test_splits_match_oracle(ctx, split):
    """A 2^18 transform (wide) through passes of every radix's remainder, coset and inverse coset."""
    lg, n = 18, 1 << 18
    om = G.omega_for_size(n)
    v = synth.fr_uniform(77, n)
    d = ctx.to_device(v)
    ctx.fr_to_mont(d, d, n)
    out = ctx.alloc(n * 32)
    ctx.tune_set_ntt_split(lg, split)
    try:
        for mode in (2, 3):
            ctx.ntt(mode, out, d, n, lg, om, 5)
            ctx.fr_from_mont(out, out, n)
            got = out.download().view("<u8").reshape(n, 4)
            assert (got == _expected(mode, v, n, om)).all(), mode
    finally:
        ctx.tune_set_ntt_split(lg, [])


_cache = {}


def _expected(mode, v, n, om):
    if mode not in _cache:
        _cache[mode] = O.ntt_op(mode, v, n, om, 5)
    return _cache[mode]


@pytest.mark.parametrize("log_n", [8, 9, 10, 11, 12])
def test_small_sizes_match_oracle(ctx, log_n):
    """2^9 .. 2^11 alone take two passes; in and out of place, every mode."""
    n = 1 << log_n
    om = G.omega_for_size(n)
    v = synth.fr_uniform(log_n, n)
    for mode in range(4):
        want = O.ntt_op(mode, v, n, om, 5 if mode >= 2 else 1)
        d, out = ctx.to_device(v), ctx.alloc(n * 32)
        ctx.fr_to_mont(d, d, n)
        ctx.ntt(mode, out, d, n, log_n, om, 5 if mode >= 2 else 1)
        ctx.ntt(mode, d, d, n, log_n, om, 5 if mode >= 2 else 1)
        for o in (out, d):
            ctx.fr_from_mont(o, o, n)
            assert (o.download().view("<u8").reshape(n, 4) == want).all(), mode


@pytest.mark.parametrize("log_n", [18, 19, 20])
def test_extreme_values(ctx, log_n):
    """All values r - 1 and alternating r - 1, 0: sums and differences at the ends of their range."""
    n = 1 << log_n
    om = G.omega_for_size(n)
    for vals in ([synth.FR_MODULUS - 1, synth.FR_MODULUS - 1], [synth.FR_MODULUS - 1, 0]):
        v = np.tile(synth.ints_to_limbs(vals), (n // 2, 1))
        d = ctx.to_device(v)
        ctx.fr_to_mont(d, d, n)
        ctx.ntt(2, d, d, n, log_n, om, 5)
        ctx.ntt(3, d, d, n, log_n, om, 5)
        ctx.fr_from_mont(d, d, n)
        assert (d.download().view("<u8").reshape(n, 4) == v).all()
