"""What a context does after a call that failed on the way, with the failure raised on the
host (SG_OPT_FAULT): no kernel is made to fault, trap or wait."""
import random

import numpy as np
import pytest
import torch

import oracle_p256 as E

pytestmark = pytest.mark.gpu


def test_staging_after_a_failed_stir_proof(sgpu):
    """A STIR proof that fails while its first layer (2^24 leaves, some milliseconds) is in the
    making: its results must not land in the staging that the next call's witness lies in."""
    rng = random.Random(1)
    a, b = [rng.randrange(2) for _ in range(8)], [rng.randrange(2) for _ in range(8)]
    _, q = E.keypair(0x1357)
    want, _ = E.trace(E.G, a, q, b)
    n0 = 1 << 24
    f0 = torch.arange(n0, device="cuda", dtype=torch.int64)
    torch.cuda.synchronize()
    with sgpu.Context(0) as c:
        params = sgpu.build_params(n0, b"\1" * 32)
        for _ in range(3):
            c.set_option(sgpu.OPT_FAULT, sgpu.FAULT_STIR)
            with pytest.raises(sgpu.StarkGpuError) as ei:
                c.deep_fri_prove(f0, n0, params)
            assert ei.value.code == sgpu.SG_ENOMEM
            assert np.array_equal(c.p256_chain_trace(E.G, a, q, b), want)
        # the context goes on proving
        small = f0[:4096].contiguous()
        p = sgpu.build_params(4096, b"\2" * 32)
        assert sgpu.deep_fri_verify(p, c.deep_fri_prove(small, 4096, p))
