"""Tables of the tensor-core NTT passes (ntt_tc.cu): lane tables of a four-step transform's
first pass, tables that no longer fit their cache, and contexts that build the same ones at
the same time."""
import hashlib

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


def field(cols, n, seed):
    return np.random.default_rng(seed).integers(0, O.P, size=(cols, n), dtype=np.uint64)


def lane_units(log_m, log_e, lanes, cols):
    """Units of 8 columns that the pass (2^log_m points a lane onto 2^(log_m + log_e)) has, and
    how many it takes for lane tables: two waves of CTAs."""
    lr = 5 if log_m == 10 else 4
    tile = 4 if log_m == 10 else 8
    return lanes // tile * (1 << (log_e + log_m - 2 * lr)) * (cols // 8), 2 * 148 * (2 if log_m == 8 else 1)


# first passes of 2^8, 2^9 and 2^10 points, ragged last column ranges among them
@pytest.mark.parametrize("cols,log_n,inverse", [(153, 16, True), (160, 16, False), (41, 17, True), (43, 17, False),
                                                (40, 18, True), (26, 20, False)])
def test_lane_tables(ctx, cols, log_n, inverse):
    units, least = lane_units(log_n - log_n // 2, 0, 1 << (log_n // 2), cols)
    assert units >= least
    x = field(cols, 1 << log_n, cols)
    got = ctx.ntt(x, log_n, inverse)
    for c in sorted({0, 7, 8, cols // 2, cols - 1}):
        assert np.array_equal(got[c], O.ntt(x[c], inverse)), c


@pytest.mark.parametrize("w,log_n,blowup,shift", [(9, 16, 32, 7), (17, 16, 16, 1), (24, 17, 8, 1), (11, 17, 16, 7),
                                                  (9, 18, 16, 7), (16, 19, 4, 1), (9, 20, 8, 7)])
def test_lane_tables_of_an_lde(ctx, w, log_n, blowup, shift):
    units, least = lane_units(log_n // 2, blowup.bit_length() - 1, 1 << (log_n - log_n // 2), w)
    assert units >= least
    x = field(w, 1 << log_n, w)
    pick = sorted({0, w // 2, w - 1})
    assert np.array_equal(ctx.lde(x, blowup, shift)[pick], O.lde(np.ascontiguousarray(x[pick]), blowup, shift))


def test_full_cache(sgpu):
    """The cache holds 64 MiB: 2^10 rows onto 2^19 points take 36 MiB, 2^8 onto 2^19 as much
    again (built for the call alone), 2^9 onto 2^19 more than the whole cache (no tables)."""
    cases = [(10, 512), (8, 2048), (9, 1024)]
    xs = {c: field(2, 1 << c[0], c[0]) for c in cases}
    want = {c: O.lde(xs[c], c[1]) for c in cases}
    with sgpu.Context(0) as c:
        for _ in range(3):
            for case in cases:
                assert np.array_equal(c.lde(xs[case], case[1], 1), want[case]), case


def test_same_tables_at_once(sgpu, ctx):
    """Workers share their parent's tables: on a new one all of them build them at once."""
    jobs = [(sgpu.JOB_SHA256, bytes([i]) * 64, hashlib.sha3_256(bytes([i])).digest()) for i in range(12)]
    want = [ctx.prove_sha256(m, pi)[0] for _, m, pi in jobs]
    for _ in range(4):
        with sgpu.Context(0) as c:
            assert [p for p, _ in c.prove_batch(jobs, n_streams=12)] == want
