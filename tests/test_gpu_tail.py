"""Small batches end inside the IND-CPA kernel (K or H(pk) by a warp of each
instance's CTA): one instance, both sides of one and two instances per SM, all
sets, against the oracle, on every entry point that takes that way."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 4


@pytest.mark.parametrize("set_id", range(6))
@pytest.mark.parametrize("n", [1, 2, 152, 153, 304, 305])
def test_small_batches_match_oracle(kem, oracle, set_id, n):
    import torch
    T, ctx = kem
    z = T.sizes(set_id)
    kc = T.splitmix_bytes(9700 + 10 * set_id + n, n * 96).reshape(n, 96)
    ec = T.splitmix_bytes(9800 + 10 * set_id + n, n * 32).reshape(n, 32)
    opk, osk = oracle.kem_keypair_batch(set_id, kc, THREADS)
    pk, sk = ctx.kem_keypair(set_id, kc)
    assert np.array_equal(pk, opk) and np.array_equal(sk, osk)
    oct_, oss = oracle.kem_enc_batch(set_id, opk, ec, THREADS)
    ct, ss = ctx.kem_enc(set_id, pk, ec)
    assert np.array_equal(ct, oct_) and np.array_equal(ss, oss)
    bad = oct_.copy()
    bad[::2, (7 * n) % bad.shape[1]] ^= 0x10
    want, fail = oracle.kem_dec_batch(set_id, bad, osk, THREADS)
    assert fail[0] and (n == 1 or not fail[1])
    assert np.array_equal(ctx.kem_dec(set_id, bad, sk), want)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    a = torch.empty((n, T.genmatrix_bytes(set_id)), dtype=torch.uint8, device="cuda")
    out, out2, ct2 = (torch.zeros((n, w), dtype=torch.uint8, device="cuda") for w in (32, 32, z.ct_bytes))
    dpk, dsk, dbad = dev(pk), dev(sk), dev(bad)
    ctx.genmatrix_ptr(set_id, n, a, dpk)
    ctx.kem_dec_a_ptr(set_id, n, out, dbad, dsk, a)
    ctx.kem_enc_a_ptr(set_id, n, ct2, out2, dpk, dev(ec), a)
    ctx.sync_status()
    assert np.array_equal(out.cpu().numpy(), want)
    assert np.array_equal(ct2.cpu().numpy(), oct_) and np.array_equal(out2.cpu().numpy(), oss)
    # one key
    ct1, ss1 = oracle.kem_enc_batch(set_id, np.repeat(opk[:1], n, axis=0), ec, THREADS)
    ct1[-1, -1] ^= 0x80
    want1, _ = oracle.kem_dec_batch(set_id, ct1, np.repeat(osk[:1], n, axis=0), THREADS)
    assert np.array_equal(ctx.kem_dec_onekey(set_id, ct1, sk[0]), want1)
