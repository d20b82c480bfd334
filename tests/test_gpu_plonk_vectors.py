"""BATCH_INV at the edges of its warps (zeros, ones, values near r, powers of two, in place) and the
PLONK quotient at every number of points a thread takes, sampled against the oracle's formula."""

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


def _up(ctx, v):
    d = ctx.to_device(v)
    ctx.fr_to_mont(d, d, v.shape[0])
    return d


def _down(ctx, d, n):
    t = ctx.alloc(n * 32)
    ctx.fr_from_mont(t, d, n)
    return synth.limbs_to_ints(t.download().view("<u8").reshape(n, 4))


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 511, 512, 513, 1500])
@pytest.mark.parametrize("kind", ["random", "zeros", "edges"])
def test_batch_inverse(ctx, n, kind):
    vals = synth.limbs_to_ints(synth.fr_uniform(n, n))
    if kind == "zeros":
        vals = [0 if i % 3 == 0 else v for i, v in enumerate(vals)]
    elif kind == "edges":
        edges = [1, 2, R - 1, R - 2, (R + 1) // 2, 1 << 253, 0, 3, 1 << 128, (1 << 32) - 1]
        vals = [edges[i % len(edges)] for i in range(n)]
    d = _up(ctx, synth.ints_to_limbs(vals))
    want = [pow(v, -1, R) if v else 0 for v in vals]
    out = ctx.alloc(n * 32)
    ctx.fr_batch_inv(out, d, n)
    assert _down(ctx, out, n) == want
    ctx.fr_batch_inv(d, d, n)
    assert _down(ctx, d, n) == want


@pytest.mark.parametrize("v", [1 << e for e in range(0, 254, 23)] + [R - (1 << e) for e in range(1, 253, 31)])
def test_single_inverse(ctx, v):
    d = _up(ctx, synth.ints_to_limbs([v]))
    ctx.fr_batch_inv(d, d, 1)
    assert _down(ctx, d, 1) == [pow(v, -1, R)]


@pytest.mark.parametrize("log_m", [9, 16, 18, 19, 20])
def test_quotient_samples(ctx, log_m):
    m, n = 1 << log_m, 1 << (log_m - 2)
    om, shift = G.omega_for_size(m), 11
    par = [synth.limbs_to_ints(synth.fr_uniform(70 + j, 1))[0] for j in range(5)]
    ins = [_up(ctx, synth.fr_uniform(80 + j, m)) for j in range(15)]
    num, zh = ctx.alloc(m * 32), ctx.alloc(m * 32)
    shift_n = pow(shift, n, R)
    ctx.plonk_quotient_evals(ins, m, n, om, shift, shift_n, *par, num, zh)
    idx = np.array(sorted({0, 1, 31, 32, 63, 64, 511, m // 2, m - 1}
                          | {int(x) for x in np.random.default_rng(log_m).integers(0, m, 40)}), dtype=np.uint32)
    didx = ctx.to_device(idx)
    got = []
    for src in ins + [num, zh]:
        g = ctx.alloc(idx.size * 32)
        ctx.fr_gather(g, src, didx, idx.size)
        got.append(_down(ctx, g, idx.size))
    u = pow(om, n, R)
    for t, i in enumerate(idx):
        x = shift * pow(om, int(i), R) % R
        want, _ = O.plonk_t_quotient_evals([[g[t]] for g in got[:15]], n, om, x, shift_n, *par)
        assert got[15][t] == want[0] and got[16][t] == (shift_n * pow(u, int(i), R) - 1) % R
