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


@pytest.mark.parametrize("log_n", [11, 15, 16, 18])
def test_pinned_splits_leave_the_lde_alone(sgpu, log_n):
    """An LDE of 2^11 .. 2^20 rows has no four-step split, so none that is pinned slows it down."""
    x = field(2, 1 << log_n, log_n)
    want = O.lde(x, 8, 7)

    def run():
        with sgpu.Context(0) as c:
            got = []
            n = launches(sgpu, lambda: got.append(c.lde(x, 8, 7)))
            assert np.array_equal(got[0], want)
            return n

    free = run()
    pins = [(n, p, l1) for n, p in ((log_n, False), (log_n + 3, True)) if n >= 13
            for l1 in (max(1, n - 12), min(12, n - 1))]
    for n, p, l1 in pins:
        try:
            sgpu.ntt_set_split(n, p, l1)
            assert run() == free, (n, p, l1)
        finally:
            sgpu.ntt_set_split(n, p, 0)


@pytest.mark.parametrize("log_n", [13, 15, 17])
def test_pinned_padded_splits(sgpu, ctx, log_n):
    """The quotient's zero-padded transform (merge) under every split that may be pinned for it."""
    n_trace = (1 << log_n) // 32
    lde = field(4, 1 << log_n, log_n)
    coeffs = [3, 5, 7]
    run = lambda: ctx.merge(sgpu.AIR_HASH_ROLLUP, lde, n_trace, 32, coeffs)
    want = O.merge(sgpu.AIR_HASH_ROLLUP, lde, n_trace, 32, coeffs)
    for l1 in range(max(1, log_n - 12), min(12, log_n - 1) + 1):
        try:
            sgpu.ntt_set_split(log_n, True, l1)
            assert np.array_equal(run(), want), l1
        finally:
            sgpu.ntt_set_split(log_n, True, 0)


@pytest.mark.parametrize("log_n,most", [(1, 32768), (4, 32768), (5, 16384)])
def test_tiny_transforms_up_to_their_line(sgpu, ctx, log_n, most):
    """A thread a column as far as it is the faster one; the results on both sides of the line."""
    for cols, name in ((most, "ntt_radix"), (most + 1, "ntt_pass")):
        x = field(cols, 1 << log_n, cols)
        got = []
        assert launches(sgpu, lambda: got.append(ctx.ntt(x, log_n, True))) == {name: 1}
        for c in (0, cols // 2, cols - 1):
            assert np.array_equal(got[0][c], O.ntt(x[c], True)), c
