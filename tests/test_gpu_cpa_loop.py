"""The tcgen05 IND-CPA kernel runs one CTA per instance until the GPU is full
and then hands further instances to the resident CTAs (cluster launch
control).  Batches at the edges of that: one, the CTAs of a full GPU less and
plus one, and a ragged count that gives every CTA several instances.  All
outputs are bytes and must equal the oracle's."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 4


@pytest.mark.parametrize("set_id", range(6))
@pytest.mark.parametrize("n", [1, 152 * 4 + 1, 152 * 8 - 1, 4001])
def test_kem_matches_oracle(kem, oracle, set_id, n):
    T, ctx = kem
    kc = T.splitmix_bytes(7100 + 10 * set_id + n, n * 96).reshape(n, 96)
    ec = T.splitmix_bytes(7200 + 10 * set_id + n, n * 32).reshape(n, 32)
    opk, osk = oracle.kem_keypair_batch(set_id, kc, THREADS)
    pk, sk = ctx.kem_keypair(set_id, kc)
    assert np.array_equal(pk, opk) and np.array_equal(sk, osk)
    oct_, oss = oracle.kem_enc_batch(set_id, opk, ec, THREADS)
    ct, ss = ctx.kem_enc(set_id, pk, ec)
    assert np.array_equal(ct, oct_) and np.array_equal(ss, oss)
    bad = ct.copy()
    bad[::5, (3 * n) % bad.shape[1]] ^= 0x12  # every fifth ciphertext tampered, the last byte range too
    bad[-1, -1] ^= 0x80
    want, _ = oracle.kem_dec_batch(set_id, bad, osk, THREADS)
    assert np.array_equal(ctx.kem_dec(set_id, bad, sk), want)


@pytest.mark.parametrize("l", [2, 3, 4])
@pytest.mark.parametrize("transpose", [False, True])
def test_matvec_matches_oracle(kem, oracle, l, transpose):
    T, ctx = kem
    n = 152 * 8 + 5
    rng = np.random.default_rng(77 + l)
    A = rng.integers(0, 1 << 13, (n, l, l, 256), dtype=np.uint16)
    s = rng.integers(-7, 8, (n, l, 256), dtype=np.int8)
    A[0] = 8191
    s[0] = 7
    A[1] = 4096
    s[1] = -7
    assert np.array_equal(ctx.matvec(A, s, 13, transpose), oracle.matvec(A, s, 13, transpose, THREADS))
