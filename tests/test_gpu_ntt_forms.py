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


@pytest.mark.parametrize("shape", [{8: 1024}, {7: 2048}, {3: 4096, 7: 2048}, {6: 4096, 10: 1, 8: 2}, {6: 4096, 10: 256},
                                   {5: 8200, 17: 2}])
def test_batches_of_small_transforms(shape):
    """Batches of 2^18 elements and more around the share of small ones at which the form changes."""
    ctx = N.default_context()
    jobs, ins, outs = [], {}, {}
    for lg, count in shape.items():
        n = 1 << lg
        ins[lg], outs[lg] = _data(ctx, n * count, lg), ctx.alloc(n * count * 32)
        for i in range(count):
            jobs.append((2, N.DeviceArray(ctx, 32 * n, ptr=outs[lg].ptr + 32 * n * i, owned=False),
                         N.DeviceArray(ctx, 32 * n, ptr=ins[lg].ptr + 32 * n * i, owned=False), n, lg,
                         G.omega_for_size(n), 5))
    ctx.ntt_batch(jobs)
    for lg, count in shape.items():
        n = 1 << lg
        host = ctx.alloc(n * count * 32)
        ctx.fr_from_mont(host, ins[lg], n * count)
        src = host.download().view("<u8").reshape(count, n, 4)
        ctx.fr_from_mont(host, outs[lg], n * count)
        got = host.download().view("<u8").reshape(count, n, 4)
        for i in sorted({0, 1 % count, count // 2, count - 1}):
            assert (got[i] == O.ntt_op(2, np.ascontiguousarray(src[i]), n, G.omega_for_size(n), 5)).all(), (lg, i)
