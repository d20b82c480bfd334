"""Small MSMs from several threads at once, each with its own context: one call's early-woken
host helpers (they wait for its device work) must neither block nor serve another call wrongly."""

import threading

import pytest

from pyzkp_gb300 import _native as N
from pyzkp_gb300 import synth

pytestmark = pytest.mark.gpu
R = synth.FR_MODULUS


@pytest.mark.parametrize("threads", [2, 6])
def test_concurrent_small_msms(threads):
    sizes = [1, 40, 777, 3000]
    errors = []

    def work(i):
        try:
            ctx = N.Context(0)
            n = sizes[-1]
            k = synth.base_dlogs(50 + i, n)
            xy = ctx.alloc(n * 64)
            ctx.g1_fixed_base_mul((1, 2), ctx.to_device(k), n, xy)
            bases = ctx.bases_from_device(xy, n)
            s = synth.fr_witness_like(60 + i, n)
            d = ctx.to_device(s)
            ki, si = synth.limbs_to_ints(k), synth.limbs_to_ints(s)
            want = {m: N.host_g1_mul((1, 2), sum(a * b for a, b in zip(ki[:m], si[:m])) % R) for m in sizes}
            for _ in range(20):
                for m in sizes:
                    assert ctx.msm_g1(bases, d, m, scalars_mont=False) == want[m]
                got = ctx.msm_g1_batch(bases, [d] * 4, sizes, scalars_mont=False)
                assert got == [want[m] for m in sizes]
        except BaseException as e:  # noqa: BLE001 -- reported by the main thread
            errors.append(repr(e))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join(timeout=120)
    assert not any(t.is_alive() for t in ts) and not errors, errors
