"""Launch counts and stage statistics where a Keccak front is two launches side by
side (128 to 192 instances per SM): one kernel and one launch of the stage more
than just below."""
import pytest

pytestmark = pytest.mark.gpu

BELOW, SPLIT = 128 * 152 - 1, 128 * 152 + 500


def test_split_fronts_count_both_launches(kem):
    import torch
    T, _ = kem
    S = T.LIGHTSABLE
    z = T.sizes(S)
    new = lambda n, w: torch.zeros((n, w), dtype=torch.uint8, device="cuda")
    pk, sk, ct, ss, out = (new(SPLIT, w) for w in (z.pk_bytes, z.sk_bytes, z.ct_bytes, 32, 32))
    kc, ec = (torch.from_numpy(T.splitmix_bytes(w, SPLIT * w).reshape(SPLIT, w)).cuda() for w in (96, 32))
    calls = {
        "shake_jobs": (3, lambda c, n: c.kem_keypair_ptr(S, n, pk, sk, kc)),
        "enc_front": (3, lambda c, n: c.kem_enc_ptr(S, n, ct, ss, pk, ec)),
        "dec_front": (5, lambda c, n: c.kem_dec_ptr(S, n, out, ct, sk)),
        "mix_front": (5, lambda c, n: c.kem_dec_mixed([(S, out[:n], ct[:n], sk[:n])])),
    }
    for n, more in ((BELOW, 0), (SPLIT, 1)):
        for stage, (kernels, call) in calls.items():
            ctx = T.Context(0)
            before = ctx.launches
            ctx.set_timing(True)
            call(ctx, n)
            assert ctx.launches - before == kernels + more, (stage, n)
            assert ctx.stage_stats()[stage][0] == 1 + more, (stage, n)
            ctx.sync_status()
            ctx.close()
