"""Fr values whose bits are not below r: the vector operations take them as their residues."""

import numpy as np
import pytest

from pyzkp_gb300 import _native as N
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
