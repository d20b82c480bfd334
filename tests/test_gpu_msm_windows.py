"""Single G1 and G2 MSMs on both sides of every line of the window table, against [sum k_i s_i] G."""

import pytest

from pyzkp_gb300 import _native as N
from pyzkp_gb300 import groth16 as G
from pyzkp_gb300 import synth

pytestmark = pytest.mark.gpu
R = synth.FR_MODULUS
LINES = [575, 1100, 2300, 16384, 196608, 260000, 287000, 298000]


def _answers(seed, sizes):
    """Exponents, scalars and the sums of their products at each size."""
    n = max(sizes)
    k, s = synth.base_dlogs(seed, n), synth.fr_witness_like(seed + 1, n)
    sums, acc, at = {}, 0, 0
    ki, si = synth.limbs_to_ints(k), synth.limbs_to_ints(s)
    for m in sorted(sizes):
        acc += sum(a * b for a, b in zip(ki[at:m], si[at:m]))
        sums[m], at = acc % R, m
    return k, s, sums


def test_g1():
    ctx = N.default_context()
    sizes = [n + d for n in LINES for d in (0, 1)]
    k, s, sums = _answers(31, sizes)
    n = max(sizes)
    xy = ctx.alloc(n * 64)
    ctx.g1_fixed_base_mul((1, 2), ctx.to_device(k), n, xy)
    bases, d = ctx.bases_from_device(xy, n), ctx.to_device(s)
    for m in sizes:
        assert ctx.msm_g1(bases, d, m, scalars_mont=False) == N.host_g1_mul((1, 2), sums[m]), m
    got = ctx.msm_g1_batch(bases, [d] * len(sizes), sizes, scalars_mont=False)
    assert got == [N.host_g1_mul((1, 2), sums[m]) for m in sizes]


def test_g2():
    ctx = N.default_context()
    sizes = [n + d for n in LINES[:5] for d in (0, 1)]
    k, s, sums = _answers(33, sizes)
    n = max(sizes)
    xy = ctx.alloc(n * 128)
    ctx.g2_fixed_base_mul(G.G2_GEN, ctx.to_device(k), n, xy)
    bases, d = ctx.bases_g2_from_device(xy, n), ctx.to_device(s)
    for m in sizes:
        assert ctx.msm_g2(bases, d, m, scalars_mont=False) == N.host_g2_mul(G.G2_GEN, sums[m]), m
