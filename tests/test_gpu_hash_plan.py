"""How a Keccak launch's sponges are spread (plan_sponges): one warp, two
threads or one thread per sponge by count, whole rounds of 32 sponges per SM
sub-partition with the remainder in a finer form, and two launches side by side
just above one round; below it the shorter of two roles partly in two threads a
sponge.  Batches at both sides of every line, against the oracle."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 4
PARTS = 4 * 152  # sub-partitions


@pytest.mark.parametrize("n", [9800, 14001, 15000, 16384, 11 * PARTS // 8, 11 * PARTS // 8 + 1, 11 * PARTS // 4 + 1, 16 * PARTS, 16 * PARTS + 1,
                               32 * PARTS - 1, 32 * PARTS, 32 * PARTS + 9 * PARTS // 8 + 1, 32 * PARTS + 9 * PARTS // 4 + 1,
                               48 * PARTS - 1, 48 * PARTS, 64 * PARTS + 3])
def test_kem_matches_oracle(kem, oracle, n):
    T, ctx = kem
    set_id = T.SABER if n % 2 else T.LIGHTSABLE
    kc = T.splitmix_bytes(8100 + n, n * 96).reshape(n, 96)
    ec = T.splitmix_bytes(8200 + n, n * 32).reshape(n, 32)
    opk, osk = oracle.kem_keypair_batch(set_id, kc, THREADS)
    pk, sk = ctx.kem_keypair(set_id, kc)
    assert np.array_equal(pk, opk) and np.array_equal(sk, osk)
    oct_, oss = oracle.kem_enc_batch(set_id, opk, ec, THREADS)
    ct, ss = ctx.kem_enc(set_id, pk, ec)
    assert np.array_equal(ct, oct_) and np.array_equal(ss, oss)
    ct[::3, 5] ^= 0x41
    want, _ = oracle.kem_dec_batch(set_id, ct, osk, THREADS)
    import torch
    dev = [torch.from_numpy(x).cuda() for x in (ct, sk)]
    out = torch.empty((n, 32), dtype=torch.uint8, device="cuda")
    ctx.kem_dec_ptr(set_id, n, out, *dev)  # device buffers: the front split over two streams where the plan says so
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)
    assert np.array_equal(ctx.kem_dec(set_id, ct, sk), want)


@pytest.mark.parametrize("n", [PARTS, PARTS + 1, 3 * PARTS // 2, 3 * PARTS // 2 + 1, 11 * PARTS // 4 + 1])
def test_cached_decapsulation_matches_oracle(kem, oracle, n):
    """H(c) and G beside others, with GenMatrix and as launches of their own: both
    sides of the lines where they leave the warp form."""
    import torch
    T, ctx = kem
    set_id = T.FIRESABER if n % 2 else T.SABER
    opk, osk = oracle.kem_keypair_batch(set_id, T.splitmix_bytes(8300 + n, n * 96).reshape(n, 96), THREADS)
    ct, _ = oracle.kem_enc_batch(set_id, opk, T.splitmix_bytes(8400 + n, n * 32).reshape(n, 32), THREADS)
    ct[::3, 5] ^= 0x41
    want, _ = oracle.kem_dec_batch(set_id, ct, osk, THREADS)
    dpk, dsk, dct = (torch.from_numpy(x).cuda() for x in (opk, osk, ct))
    a = torch.empty((n, T.genmatrix_bytes(set_id)), dtype=torch.uint8, device="cuda")
    out = torch.empty((n, 32), dtype=torch.uint8, device="cuda")
    ctx.genmatrix_ptr(set_id, n, a, dpk)
    ctx.kem_dec_a_ptr(set_id, n, out, dct, dsk, a)
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)
    ctx.kem_dec_ptr(set_id, n, out, dct, dsk)
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)
