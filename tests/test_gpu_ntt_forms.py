"""The two forms of the NTT passes on one (omega, shift, mode), each used first and after the other."""

import numpy as np
import pytest

from oracle import oracle as O
from pyzkp_gb300 import _native as N
from pyzkp_gb300 import groth16 as G
from pyzkp_gb300 import synth

pytestmark = pytest.mark.gpu


def _data(ctx, n, seed):
    d = ctx.to_device(synth.fr_uniform(seed, n))
    ctx.fr_to_mont(d, d, n)
    return d


@pytest.mark.parametrize("mode", [2, 3])
@pytest.mark.parametrize("wide_first", [False, True])
@pytest.mark.parametrize("log_n", [17, 8])
def test_both_forms_of_one_plan(mode, wide_first, log_n):
    """A transform alone (narrow) and in a batch of 2^18 elements (wide), either one first."""
    ctx = N.Context(0)
    n, om = 1 << log_n, G.omega_for_size(1 << log_n)
    v = synth.fr_uniform(7, n)
    want = O.ntt_op(mode, v, n, om, 5)
    d = ctx.to_device(v)
    ctx.fr_to_mont(d, d, n)
    outs = [ctx.alloc(n * 32) for _ in range(1 << (18 - log_n))]
    for wide in (wide_first, not wide_first, wide_first):
        if wide:
            ctx.ntt_batch([(mode, o, d, n, log_n, om, 5) for o in outs])
        else:
            ctx.ntt(mode, outs[0], d, n, log_n, om, 5)
        for o in (outs[0], outs[-1]) if wide else outs[:1]:
            got = ctx.alloc(n * 32)
            ctx.fr_from_mont(got, o, n)
            assert (got.download().view("<u8").reshape(n, 4) == want).all()
    ctx.close()
