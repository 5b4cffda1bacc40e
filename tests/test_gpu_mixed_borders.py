"""Mixed-set passes whose Keccak stages run two threads a sponge, with groups
that end in the middle of a warp (16 sponges): neighbours in a warp then have
sponges of different lengths.  Totals on both sides of the form lines (2.75, 16
and 32 sponges per SM sub-partition, and a rest above one round), against the
oracle."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 4
PARTS = 4 * 152
# groups of a few odd sizes, so that nearly every warp of them holds several sets
SMALL = [(0, 5), (1, 3), (2, 7), (3, 1), (4, 9), (5, 11), (1, 13), (0, 2), (5, 17), (3, 21), (2, 1), (4, 6)]


@pytest.mark.parametrize("total", [11 * PARTS // 4 - 1, 11 * PARTS // 4 + 2, 16 * PARTS - 1, 16 * PARTS + 1,
                                   32 * PARTS + 9 * PARTS // 4 + 3])
def test_groups_end_inside_a_warp(kem, oracle, total):
    import torch
    T, ctx = kem
    rest = total - sum(n for _, n in SMALL)
    big = [(0, rest // 3 + 5), (4, rest // 3 - 1), (1, rest - 2 * (rest // 3) - 4)]
    groups, want = [], []
    for i, (set_id, n) in enumerate(SMALL + big):
        kc = T.splitmix_bytes(9700 + 2 * i, n * 96).reshape(n, 96)
        ec = T.splitmix_bytes(9701 + 2 * i, n * 32).reshape(n, 32)
        pk, sk = oracle.kem_keypair_batch(set_id, kc, THREADS)
        ct, _ = oracle.kem_enc_batch(set_id, pk, ec, THREADS)
        ct[::3, 9] ^= 0x08
        want.append(oracle.kem_dec_batch(set_id, ct, sk, THREADS)[0])
        groups.append((set_id, torch.zeros((n, 32), dtype=torch.uint8, device="cuda"),
                       torch.from_numpy(ct).cuda(), torch.from_numpy(sk).cuda()))
    assert sum(n for _, n in SMALL + big) == total
    ctx.kem_dec_mixed(groups)
    ctx.sync_status()
    for (set_id, out, _, _), w in zip(groups, want):
        assert np.array_equal(out.cpu().numpy(), w), set_id
