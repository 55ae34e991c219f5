"""What a context does after a call that failed on the way, with the failure raised on the
host (SG_OPT_FAULT): no kernel is made to fault, trap or wait."""
import random

import numpy as np
import pytest
import torch

import oracle_lib as O
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


def test_a_wait_that_ran_out_is_the_context_s_own(sgpu):
    """A kernel whose bounded wait ran out sets its context's word (here set from the host): that
    context's next call reports it, no other context's does, nor that context's later ones."""
    x = np.random.default_rng(1).integers(0, O.P, size=(3, 1 << 10), dtype=np.uint64)
    want = np.stack([O.ntt(c) for c in x])
    msg, pi = b"one record", b"\1" * 32
    p = sgpu.build_params(4096, pi)
    f0 = np.arange(4096, dtype=np.uint64)
    with sgpu.Context(0) as c, sgpu.Context(0) as other:
        proof, digest = other.prove_sha256(msg, pi)
        stir = other.deep_fri_prove(f0, 4096, p)
        calls = [
            (lambda: c.ntt(x, 10, False).tolist(), want.tolist()),
            (lambda: c.prove_sha256(msg, pi), (proof, digest)),
            (lambda: c.deep_fri_prove(f0, 4096, p), stir),
            (lambda: c.deep_fri_prove_group(np.stack([f0, f0]), [p, p]), [stir, stir]),
        ]
        for call, result in calls:
            c.set_option(sgpu.OPT_FAULT, sgpu.FAULT_WAIT)
            assert np.array_equal(other.ntt(x, 10, False), want)
            # a server's workers are contexts of their own
            assert c.prove_batch([(sgpu.JOB_SHA256, msg, pi)], n_streams=2)[0][0] == proof
            with pytest.raises(sgpu.StarkGpuError) as ei:
                call()
            assert ei.value.code == sgpu.SG_ECUDA and "wait" in str(ei.value)
            assert call() == result


# LDEs that run as one tensor-core pass (rows of 2^8 .. 2^10, or fewer onto 2^11 points), with
# fewer and with more cosets than a lane-per-coset pass has lanes; in interleaved parts (2^11
# .. 2^15 rows); in blocks (2^16 rows)
@pytest.mark.parametrize("log_n,blowup", [(3, 256), (5, 64), (7, 16), (7, 32), (8, 2), (8, 4), (8, 64), (9, 2),
                                          (9, 8), (9, 32), (10, 2), (10, 4), (10, 8), (10, 32), (11, 2), (11, 32), (13, 4),
                                          (15, 2), (16, 8)])
@pytest.mark.parametrize("shift", [1, 7])
def test_lde_without_room_for_tables(sgpu, log_n, blowup, shift):
    x = np.random.default_rng(log_n).integers(0, O.P, size=(3, 1 << log_n), dtype=np.uint64)
    with sgpu.Context(0) as c:
        c.set_option(sgpu.OPT_FAULT, sgpu.FAULT_TABLES)
        assert np.array_equal(c.lde(x, blowup, shift), O.lde(x, blowup, shift))


@pytest.mark.parametrize("log_n", [8, 9, 10, 11, 12, 13, 15, 16, 17, 20, 21, 22])
def test_ntt_without_room_for_tables(sgpu, log_n):
    x = np.random.default_rng(log_n).integers(0, O.P, size=(2, 1 << log_n), dtype=np.uint64)
    with sgpu.Context(0) as c:
        c.set_option(sgpu.OPT_FAULT, sgpu.FAULT_TABLES)
        for inverse in (False, True):
            assert np.array_equal(c.ntt(x, log_n, inverse), np.stack([O.ntt(col, inverse) for col in x]))


def test_proofs_without_room_for_tables(sgpu):
    rng = random.Random(2)
    a, b = [rng.randrange(2) for _ in range(256)], [rng.randrange(2) for _ in range(256)]
    _, q = E.keypair(0x1357)
    pi = b"\3" * 32
    with sgpu.Context(0) as c, sgpu.Context(0) as free:
        c.set_option(sgpu.OPT_FAULT, sgpu.FAULT_TABLES)
        c.set_option(sgpu.OPT_WIDE_MERGE, sgpu.WIDE_MERGE_COSETS)
        assert c.prove_sha256(b"x" * 64, pi) == free.prove_sha256(b"x" * 64, pi)
        assert c.prove_sha512(b"x" * 300, pi) == free.prove_sha512(b"x" * 300, pi)
        assert c.prove_p256_chains(E.G, a, q, b, pi) == free.prove_p256_chains(E.G, a, q, b, pi)
