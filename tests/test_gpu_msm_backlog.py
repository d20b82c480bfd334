"""Single MSMs behind work that their stream already holds (longer than woken helpers wait awake), while
another context combines batches: the same points as without the backlog."""

import threading

import pytest

from pyzkp_gb300 import _native as N
from pyzkp_gb300 import groth16 as G
from pyzkp_gb300 import synth

pytestmark = pytest.mark.gpu


def _bases(ctx, n, seed):
    xy = ctx.alloc(n * 64)
    ctx.g1_fixed_base_mul((1, 2), ctx.to_device(synth.base_dlogs(seed, n)), n, xy)
    return ctx.bases_from_device(xy, n)


def test_small_msm_behind_a_backlog():
    n, log_n = 2000, 21
    errors = []
    stop = threading.Event()

    def batches():
        try:
            ctx = N.Context(0)
            bases, d = _bases(ctx, n, 3), ctx.to_device(synth.fr_uniform(4, n))
            sizes = [n - 7 * i for i in range(24)]
            want = [ctx.msm_g1(bases, d, m, scalars_mont=False) for m in sizes]
            while not stop.is_set():
                assert ctx.msm_g1_batch(bases, [d] * len(sizes), sizes, scalars_mont=False) == want
        except BaseException as e:  # noqa: BLE001 -- reported by the main thread
            errors.append(repr(e))

    other = threading.Thread(target=batches)
    other.start()
    try:
        ctx = N.Context(0)
        bases, d = _bases(ctx, n, 1), ctx.to_device(synth.fr_witness_like(2, n))
        want = ctx.msm_g1(bases, d, n, scalars_mont=False)
        v = ctx.alloc(32 << log_n)
        ctx.memset(v)
        om = G.omega_for_size(1 << log_n)
        for queued in (0, 1, 10, 30):
            for _ in range(queued):
                ctx.ntt(N.NTT_EVALS_FROM_COEFFS, v, v, 1 << log_n, log_n, om)
            assert ctx.msm_g1(bases, d, n, scalars_mont=False) == want
    finally:
        stop.set()
        other.join(timeout=120)
    assert not other.is_alive() and not errors, errors
