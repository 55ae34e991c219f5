"""Merkle levels at the widths where their kernels change (a thread a node, a warp a node,
the last levels in one CTA), with full and padded last parents, against the oracle."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


# parents of the first level: 1, 16, 17 (one CTA or a warp each), 1024, 1025 (a warp or a
# thread each); arities with one to five permutations a node, one that is no power of two
@pytest.mark.parametrize("arity", [2, 3, 8, 16])
@pytest.mark.parametrize("parents,cut", [(1, 0), (16, 0), (16, 1), (17, 0), (17, 1), (1024, 0), (1024, 1), (1025, 1)])
def test_level_widths(ctx, arity, parents, cut):
    n = arity * parents - cut
    cols = np.random.default_rng(n).integers(0, O.P, size=(2, n), dtype=np.uint64)
    rows = np.ascontiguousarray(cols.T)
    arities = [arity] * 12
    assert ctx.merkle_commit(cols, arities, 7) == O.merkle_root(rows, arities, 7)
