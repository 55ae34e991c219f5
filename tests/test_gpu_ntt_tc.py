"""The tensor-core NTT passes (ntt_tc.cu) against the oracle, bit-exact, at the sizes
where their tiling can go wrong: one lane, a tile's lanes and one more, more tiles than a
CTA keeps in flight, more than one chunk, both passes of a four-step transform, zero
padding, and element values whose bytes make the digit sums extreme."""
import numpy as np
import pytest
import torch

import oracle_lib as O

pytestmark = pytest.mark.gpu
P = O.P


def field(rng, cols, n, kind="random"):
    if kind == "random":
        return rng.integers(0, P, size=(cols, n), dtype=np.uint64)
    # values of all-ones bytes (high word), the largest element, zero and one
    return rng.choice(np.array([0, 1, P - 1, 0xFFFFFFFEFFFFFFFF, 0xFFFFFFFF], dtype=np.uint64), size=(cols, n))


# one pass: 2^8 and 2^9 have 8 lanes a tile, 2^10 has 4
@pytest.mark.parametrize("log_n", [8, 9, 10])
@pytest.mark.parametrize("cols", [1, 4, 5, 8, 9, 37])
@pytest.mark.parametrize("inverse", [False, True])
def test_one_pass(ctx, log_n, cols, inverse):
    rng = np.random.default_rng(cols * 100 + log_n)
    for kind in ("random", "extreme"):
        x = field(rng, cols, 1 << log_n, kind)
        got = ctx.ntt(x, log_n, inverse)
        for c in (0, cols // 2, cols - 1):
            assert np.array_equal(got[c], O.ntt(x[c], inverse)), (kind, c)


# output over the input, with more tiles than the GPU holds at a time (a 2^9-point column
# leaves its tile in two chunks, so the second would read what the first wrote)
@pytest.mark.parametrize("log_n", [8, 9, 10])
@pytest.mark.parametrize("inverse", [False, True])
def test_in_place(ctx, log_n, inverse):
    x = field(np.random.default_rng(log_n), 6001, 1 << log_n)
    d = torch.from_numpy(x.view(np.int64)).cuda()
    torch.cuda.synchronize()
    ctx.ntt(d, log_n, inverse, d)
    torch.cuda.synchronize()
    got = d.cpu().numpy().view(np.uint64)
    assert np.array_equal(got, ctx.ntt(x, log_n, inverse))
    for c in (0, 3000, 6000):
        assert np.array_equal(got[c], O.ntt(x[c], inverse)), c


# 2 .. 32 points, a thread a column: a warp's columns and one more, and both sides of the line
# above which the shared-memory pass takes them; in place too
@pytest.mark.parametrize("log_n", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("cols", [1, 6, 33, 32768, 32769])
@pytest.mark.parametrize("inverse", [False, True])
def test_tiny(ctx, log_n, cols, inverse):
    x = field(np.random.default_rng(log_n + cols), cols, 1 << log_n, "extreme" if cols == 33 else "random")
    got = ctx.ntt(x, log_n, inverse)
    for c in {0, cols // 2, cols - 1}:
        assert np.array_equal(got[c], O.ntt(x[c], inverse)), c
    d = torch.from_numpy(x.view(np.int64)).cuda()
    torch.cuda.synchronize()
    ctx.ntt(d, log_n, inverse, d)
    torch.cuda.synchronize()
    assert np.array_equal(d.cpu().numpy().view(np.uint64), got)


# 2^11 .. 2^15 points: interleaved transforms and a radix stage (columns that share a
# thread's powers in the stage's loop and a last ragged turn, one column, in place)
@pytest.mark.parametrize("log_n,cols", [(11, 1), (11, 1200), (12, 1), (12, 301), (13, 2), (13, 160), (14, 1), (14, 75), (15, 3),
                                        (15, 40)])
@pytest.mark.parametrize("inverse", [False, True])
def test_radix_stage(ctx, log_n, cols, inverse):
    x = field(np.random.default_rng(log_n + cols), cols, 1 << log_n, "extreme" if cols == 1 else "random")
    got = ctx.ntt(x, log_n, inverse)
    for c in (0, cols // 2, cols - 1):
        assert np.array_equal(got[c], O.ntt(x[c], inverse)), c
    d = torch.from_numpy(x.view(np.int64)).cuda()
    torch.cuda.synchronize()
    ctx.ntt(d, log_n, inverse, d)
    torch.cuda.synchronize()
    assert np.array_equal(d.cpu().numpy().view(np.uint64), got)


# LDE of fewer than 2^8 rows as zero-padded cosets, and of 2^11 .. 2^15 rows in interleaved
# parts joined by a radix stage
@pytest.mark.parametrize("w,log_n,blowup,shift", [
    (3, 3, 256, 7), (1, 4, 128, 1), (9, 5, 64, 5), (2, 6, 32, 1), (17, 6, 64, 7), (5, 7, 16, 1), (33, 7, 32, 7), (1, 7, 256, 3),
    (1, 11, 2, 7), (301, 11, 8, 1), (7, 11, 32, 3), (2, 12, 2, 1), (75, 12, 32, 7), (1, 13, 4, 7), (3, 13, 32, 1), (2, 14, 2, 5),
    (5, 14, 16, 1), (1, 15, 2, 1), (3, 15, 32, 7),
])
def test_lde_radix_and_short(ctx, w, log_n, blowup, shift):
    tr = field(np.random.default_rng(w + 10 * log_n), w, 1 << log_n, "extreme" if w == 2 else "random")
    pick = [0, w // 2, w - 1]
    assert np.array_equal(ctx.lde(tr, blowup, shift)[pick], O.lde(np.ascontiguousarray(tr[pick]), blowup, shift))


# two passes: both on the tensor cores (2^16 .. 2^20), or the first one only
@pytest.mark.parametrize("log_n,cols", [(13, 3), (14, 1), (15, 2), (16, 1), (16, 5), (17, 2), (18, 1), (19, 3), (20, 1),
                                        (21, 1), (22, 1)])
def test_two_passes(ctx, log_n, cols):
    rng = np.random.default_rng(log_n)
    x = field(rng, cols, 1 << log_n, "extreme" if log_n % 2 else "random")
    for inverse in (False, True):
        got = ctx.ntt(x, log_n, inverse)
        for c in range(cols):
            assert np.array_equal(got[c], O.ntt(x[c], inverse)), (inverse, c)


# LDE: coset evaluation in one pass (traces of 2^8 .. 2^10 rows), and padded two-pass
# transforms (2^11 .. 2^16 rows), with and without a coset shift
@pytest.mark.parametrize("w,log_n,blowup,shift", [
    (1, 8, 2, 1), (9, 8, 4, 7), (17, 8, 32, 1), (8, 9, 2, 3), (3, 9, 16, 1), (5, 10, 2, 7), (1, 10, 4, 1), (33, 10, 32, 5),
    (2, 11, 4, 7), (3, 12, 32, 1), (1, 13, 2, 1), (2, 14, 8, 7), (1, 15, 16, 1), (2, 16, 4, 7), (1, 17, 8, 1), (1, 8, 1024, 7),
])
def test_lde(ctx, w, log_n, blowup, shift):
    rng = np.random.default_rng(w + 10 * log_n)
    tr = field(rng, w, 1 << log_n)
    assert np.array_equal(ctx.lde(tr, blowup, shift), O.lde(tr, blowup, shift))


# enough columns for the first pass's lane tables (whole waves of units of 8 columns and
# more, a ragged last range), and the LDE with its coefficients in blocks
@pytest.mark.parametrize("cols,log_n", [(50, 16), (37, 17), (33, 18), (24, 20)])
def test_many_columns(ctx, cols, log_n):
    rng = np.random.default_rng(cols)
    x = field(rng, cols, 1 << log_n)
    got = ctx.ntt(x, log_n, True)
    for c in range(0, cols, 5):
        assert np.array_equal(got[c], O.ntt(x[c], True)), c


@pytest.mark.parametrize("w,log_n,blowup,shift", [(20, 16, 8, 7), (9, 17, 4, 1), (35, 18, 2, 3), (3, 19, 4, 7), (2, 20, 8, 7)])
def test_lde_blocked_coefficients(ctx, w, log_n, blowup, shift):
    rng = np.random.default_rng(w)
    tr = field(rng, w, 1 << log_n)
    got, pick = ctx.lde(tr, blowup, shift), [0, w // 2, w - 1]
    assert np.array_equal(got[pick], O.lde(np.ascontiguousarray(tr[pick]), blowup, shift))


def test_repeated_calls_and_tables(ctx):
    """A shape's tables are built once and shared by later calls, another shift in between."""
    rng = np.random.default_rng(5)
    tr = field(rng, 12, 256)
    want = {s: O.lde(tr, 8, s) for s in (1, 7, 11)}
    for s in (1, 7, 1, 11, 1, 7):
        assert np.array_equal(ctx.lde(tr, 8, s), want[s]), s
