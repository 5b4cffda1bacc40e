"""A capped Keccak front strides over its plan's blocks: sizes below a round of
sponges, with a rest in each finer form above one, and of several rounds, against
the oracle."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 4
PARTS = 4 * 152


@pytest.mark.parametrize("cap", [1, 8, 64])
@pytest.mark.parametrize("set_id,n", [(0, 12001), (3, 48 * PARTS), (0, 64 * PARTS + 700), (4, 64 * PARTS + 9000)])
def test_capped_front_matches_oracle(kem, oracle, set_id, n, cap):
    import torch
    T, _ = kem
    pk, sk = oracle.kem_keypair_batch(set_id, T.splitmix_bytes(9900, n * 96).reshape(n, 96), THREADS)
    ct, _ = oracle.kem_enc_batch(set_id, pk, T.splitmix_bytes(9901, n * 32).reshape(n, 32), THREADS)
    ct[::3, 7] ^= 0x20
    want, _ = oracle.kem_dec_batch(set_id, ct, sk, THREADS)
    dct, dsk = torch.from_numpy(ct).cuda(), torch.from_numpy(sk).cuda()
    out = torch.zeros((n, 32), dtype=torch.uint8, device="cuda")
    ctx = T.Context(0)
    ctx.set_dev_chunk(0)
    ctx.set_front_cap(cap)
    ctx.kem_dec_ptr(set_id, n, out, dct, dsk)
    ctx.sync_status()
    ctx.close()
    assert np.array_equal(out.cpu().numpy(), want)
