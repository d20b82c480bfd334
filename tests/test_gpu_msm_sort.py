"""The bucket sort's forms (a CTA per set, tiles with a one-CTA or a device scan, fixed-base sets)
at the sizes where one gives way to the next, against [sum k_i s_i] G."""

import numpy as np
import pytest

from pyzkp_gb300 import _native as N
from pyzkp_gb300 import synth

pytestmark = pytest.mark.gpu
R = synth.FR_MODULUS


@pytest.fixture(scope="module")
def pool():
    """Bases [k_i] G with the k_i, and scalars of three kinds, for up to 40000 points."""
    ctx, n = N.default_context(), 40000
    k = synth.base_dlogs(91, n)
    xy = ctx.alloc(n * 64)
    ctx.g1_fixed_base_mul((1, 2), ctx.to_device(k), n, xy)
    kinds = {"uniform": synth.fr_uniform(92, n), "witness": synth.fr_witness_like(93, n),
             "zeros": np.where(np.arange(n)[:, None] % 97 == 0, synth.fr_uniform(94, n), np.uint64(0))}
    return ctx, xy, synth.limbs_to_ints(k), {m: (v, synth.limbs_to_ints(v)) for m, v in kinds.items()}


def _want(k, s, n):
    return N.host_g1_mul((1, 2), sum(a * b for a, b in zip(k[:n], s[:n])) % R)


@pytest.mark.parametrize("kind", ["uniform", "witness", "zeros"])
@pytest.mark.parametrize("n", [1, 2, 512, 513, 4096, 16383, 16384, 16385, 40000])
def test_single_sizes(pool, kind, n):
    ctx, xy, k, scalars = pool
    bases = ctx.bases_from_device(xy, n)
    limbs, ints = scalars[kind]
    d, want = ctx.to_device(limbs[:n]), _want(k, ints, n)
    for c in (0, 4, 9, 13, 16):
        assert ctx.msm_g1(bases, d, n, scalars_mont=False, window_bits=c) == want, c


@pytest.mark.parametrize("sizes", [[16384, 1, 16384, 9000], [16385, 300, 16384], [5] * 70])
def test_batches(pool, sizes):
    ctx, xy, k, scalars = pool
    bases = ctx.bases_from_device(xy, max(sizes))
    limbs, ints = scalars["witness"]
    d = ctx.to_device(limbs)
    got = ctx.msm_g1_batch(bases, [d] * len(sizes), sizes, scalars_mont=False, window_bits=11)
    assert got == [_want(k, ints, m) for m in sizes]


@pytest.mark.parametrize("n,c", [(60, 8), (2000, 11), (2520, 13), (5000, 12)])
def test_fixed_base(pool, n, c):
    ctx, xy, k, scalars = pool
    bases = ctx.bases_from_device(xy, n)
    ctx.bases_precompute(bases, c)
    for limbs, ints in scalars.values():
        assert ctx.msm_g1(bases, ctx.to_device(limbs[:n]), n, scalars_mont=False) == _want(k, ints, n)
