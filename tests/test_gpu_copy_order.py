"""Decapsulation in chunks with copies ahead of the kernels, queued behind work
that still runs on the caller's stream: an earlier pass of the same context
(same workspace), and the kernels that write the inputs (device buffers that
are not 16-byte aligned are copied like host buffers).  No synchronisation in
between; both passes against the oracle."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 4
N = 3000


@pytest.mark.parametrize("onekey", [False, True])
@pytest.mark.parametrize("where", ["pinned", "unaligned"])
def test_copies_follow_the_callers_stream(kem, oracle, onekey, where):
    import torch
    T, _ = kem
    S = T.LIGHTSABER
    pk, sk = oracle.kem_keypair_batch(S, T.splitmix_bytes(9800, N * 96).reshape(N, 96), THREADS)
    if onekey:
        pk, sk = np.repeat(pk[:1], N, axis=0), np.repeat(sk[:1], N, axis=0)
    ct, _ = oracle.kem_enc_batch(S, pk, T.splitmix_bytes(9801, N * 32).reshape(N, 32), THREADS)
    ct[::3, 4] ^= 0x02
    want, _ = oracle.kem_dec_batch(S, ct, sk, THREADS)
    reps = 40  # an earlier pass long enough to be running while the next call is enqueued
    big_ct = torch.from_numpy(ct).cuda().repeat(reps, 1)
    big_sk = torch.from_numpy(sk).cuda().repeat(reps, 1)
    key = torch.from_numpy(sk[0].copy()).cuda()
    big_out = torch.zeros((reps * N, 32), dtype=torch.uint8, device="cuda")
    src = [torch.from_numpy(x).cuda() for x in (ct, sk)]
    if where == "pinned":
        ins = [torch.from_numpy(x).pin_memory() for x in (ct, sk)]
    else:
        ins = [torch.zeros(x.size + 8, dtype=torch.uint8, device="cuda")[8:].view(x.shape) for x in (ct, sk)]
    out = torch.zeros((N, 32), dtype=torch.uint8, device="cuda")
    ctx = T.Context(0)
    ctx.set_host_chunk(1024)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        for _ in range(2):
            if onekey:
                ctx.kem_dec_onekey_ptr(S, reps * N, big_out, big_ct, key, stream=st.cuda_stream)
            else:
                ctx.kem_dec_ptr(S, reps * N, big_out, big_ct, big_sk, stream=st.cuda_stream)
        if where == "unaligned":
            for d, x in zip(ins, src):
                d.copy_(x)
        if onekey:
            ctx.kem_dec_onekey_ptr(S, N, out, ins[0], key, stream=st.cuda_stream)
        else:
            ctx.kem_dec_ptr(S, N, out, ins[0], ins[1], stream=st.cuda_stream)
    st.synchronize()
    ctx.sync_status()
    ctx.close()
    assert np.array_equal(out.cpu().numpy(), want)
    assert np.array_equal(big_out.cpu().numpy(), np.tile(want, (reps, 1)))
