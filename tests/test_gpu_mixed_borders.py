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


def _pass_and_batches(T, ctx, groups, seed):
    """A mixed pass over (set, count) groups, made on the GPU, and each group as a batch."""
    import torch
    made, ref = [], T.Context(0)
    for i, (set_id, n) in enumerate(groups):
        z = T.sizes(set_id)
        new = lambda w: torch.zeros((n, w), dtype=torch.uint8, device="cuda")
        pk, sk, ct, ss, out, want = (new(w) for w in (z.pk_bytes, z.sk_bytes, z.ct_bytes, 32, 32, 32))
        ref.kem_keypair_ptr(set_id, n, pk, sk, torch.from_numpy(T.splitmix_bytes(seed + 2 * i, n * 96)).cuda())
        ref.kem_enc_ptr(set_id, n, ct, ss, pk, torch.from_numpy(T.splitmix_bytes(seed + 2 * i + 1, n * 32)).cuda())
        ct[::3, 9] ^= 0x08
        ref.kem_dec_ptr(set_id, n, want, ct, sk)
        ref.sync_status()
        made.append((set_id, out, ct, sk, want))
    torch.cuda.synchronize()
    ctx.kem_dec_mixed([m[:4] for m in made])
    ctx.sync_status()
    for set_id, out, _, _, want in made:
        assert torch.equal(out, want), set_id
    ref.close()


@pytest.mark.parametrize("total", [32 * PARTS + 5000, 48 * PARTS + 3, 2 * 32 * PARTS + 9001, 4 * 32 * PARTS + 777])
def test_large_passes_match_batches(kem, total):
    """A split front, a round and a rest, and two chains of each."""
    T, ctx = kem
    rest = total - sum(n for _, n in SMALL)
    big = [(s, rest // 6 + (3, -1, 5, -7, 2, 0)[s]) for s in range(5)]
    big.append((5, rest - sum(n for _, n in big)))
    _pass_and_batches(T, ctx, SMALL + big, 12000)


@pytest.mark.parametrize("warp,pair", [(1 << 40, 0), (0, 1 << 40), (0, 0), (500, 3000)])
def test_passes_under_the_callers_limits(kem, warp, pair):
    T, _ = kem
    ctx = T.Context(0)
    ctx.set_warp_hash(warp)
    ctx.set_pair_hash(pair)
    for big in ([], [(1, 701), (4, 1203), (0, 998)]):
        _pass_and_batches(T, ctx, SMALL + big, 12100)
    ctx.close()
