"""The kernels of a pass, and of passes behind each other on a stream, start
before the one in front has left the GPU (programmatic dependent launch) and wait
for its results.  Passes back to back whose inputs are overwritten in place
between them, with no synchronisation, as launches and replayed as a graph,
against the oracle."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 4
PASSES = 4


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("set_id,n", [(0, 1), (1, 17), (2, 300), (4, 3001), (1, 6200)])
def test_passes_back_to_back(kem, oracle, set_id, n, captured):
    import torch
    T, ctx = kem
    z = T.sizes(set_id)
    kc = T.splitmix_bytes(9300 + n, PASSES * n * 96).reshape(PASSES, n, 96)
    ec = T.splitmix_bytes(9400 + n, PASSES * n * 32).reshape(PASSES, n, 32)
    src_k, src_e = torch.from_numpy(kc).cuda(), torch.from_numpy(ec).cuda()
    new = lambda *shape: torch.zeros(shape, dtype=torch.uint8, device="cuda")
    k, e, pk, sk, ct = new(n, 96), new(n, 32), new(n, z.pk_bytes), new(n, z.sk_bytes), new(n, z.ct_bytes)
    ss, ss2, ss3 = new(n, 32), new(n, 32), new(n, 32)
    out = {name: new(PASSES, *t.shape) for name, t in (("pk", pk), ("sk", sk), ("ct", ct), ("ss", ss), ("ss2", ss2),
                                                       ("ss3", ss3))}

    def run():
        st = torch.cuda.current_stream().cuda_stream
        for i in range(PASSES):
            k.copy_(src_k[i])
            e.copy_(src_e[i])
            ctx.kem_keypair_ptr(set_id, n, pk, sk, k, stream=st)
            ctx.kem_enc_ptr(set_id, n, ct, ss, pk, e, stream=st)
            ctx.kem_dec_ptr(set_id, n, ss2, ct, sk, stream=st)
            ct[::3, 2] ^= 0x21
            ctx.kem_dec_onekey_ptr(set_id, n, ss3, ct, sk, stream=st)
            for name, t in (("pk", pk), ("sk", sk), ("ct", ct), ("ss", ss), ("ss2", ss2), ("ss3", ss3)):
                out[name][i].copy_(t)

    run()
    if captured:
        torch.cuda.synchronize()
        for t in out.values():
            t.zero_()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            run()
        g.replay()
        g.replay()
    ctx.sync_status()
    torch.cuda.synchronize()
    for i in range(PASSES):
        opk, osk = oracle.kem_keypair_batch(set_id, kc[i], THREADS)
        oct_, oss = oracle.kem_enc_batch(set_id, opk, ec[i], THREADS)
        got = {name: t[i].cpu().numpy() for name, t in out.items()}
        assert np.array_equal(got["pk"], opk) and np.array_equal(got["sk"], osk)
        bad = oct_.copy()
        bad[::3, 2] ^= 0x21
        assert np.array_equal(got["ct"], bad)
        assert np.array_equal(got["ss"], oss) and np.array_equal(got["ss2"], oss)
        want, _ = oracle.kem_dec_batch(set_id, bad, np.repeat(osk[:1], n, axis=0), THREADS)
        assert np.array_equal(got["ss3"], want)
