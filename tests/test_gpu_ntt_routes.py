"""Which kernels a transform launches, where a rule sends it the one or the other way."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


def field(cols, n, seed):
    return np.random.default_rng(seed).integers(0, O.P, size=(cols, n), dtype=np.uint64)


def launches(sgpu, call):
    """Kernel launches of a call by name."""
    sgpu.profile_enable(True)
    try:
        sgpu.profile_reset()
        call()
        return {name: n for name, (n, _) in sgpu.profile_read().items()}
    finally:
        sgpu.profile_enable(False)


@pytest.mark.parametrize("log_n", [13, 14, 15, 16, 19])
def test_autotuned_split_restores(sgpu, ctx, log_n):
    """What ntt_autotune returned, set again, is the choice that it made, the default among them."""
    x = field(3, 1 << log_n, log_n)

    def run():
        with sgpu.Context(0) as c:  # (a new one builds its tables, so the launches show them too)
            return launches(sgpu, lambda: c.ntt(x, log_n, False))

    try:
        best = ctx.ntt_autotune(3, log_n)
        tuned = run()
        sgpu.ntt_set_split(log_n, False, 0)
        sgpu.ntt_set_split(log_n, False, best)
        assert run() == tuned
    finally:
        sgpu.ntt_set_split(log_n, False, 0)
