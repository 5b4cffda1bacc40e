"""Key generation and encapsulation of a batch whose Keccak front is
two launches side by side, captured into a graph: they use the caller's stream
alone, so that another call of the context runs on other streams before the
capture has ended."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 20011  # (128 to 192 instances per SM)
OTHER = 33000  # chunks over the context's lanes


def test_other_calls_during_a_capture(kem, oracle):
    import os

    import torch
    T, _ = kem
    S = T.LIGHTSABLE
    z = T.sizes(S)
    threads = os.cpu_count() or 4
    new = lambda n, w: torch.zeros((n, w), dtype=torch.uint8, device="cuda")
    kc, ec = (T.splitmix_bytes(seed, N * w).reshape(N, w) for seed, w in ((9950, 96), (9951, 32)))
    dkc, dec_ = (torch.from_numpy(x).cuda() for x in (kc, ec))
    pk, sk, ct, ss = new(N, z.pk_bytes), new(N, z.sk_bytes), new(N, z.ct_bytes), new(N, 32)
    ctx = T.Context(0)
    opk, osk, oct_, oss = new(OTHER, z.pk_bytes), new(OTHER, z.sk_bytes), new(OTHER, z.ct_bytes), new(OTHER, 32)
    ctx.kem_keypair_ptr(S, OTHER, opk, osk, torch.from_numpy(T.splitmix_bytes(9953, OTHER * 96)).cuda())
    ctx.kem_enc_ptr(S, OTHER, oct_, oss, opk, torch.from_numpy(T.splitmix_bytes(9954, OTHER * 32)).cuda())
    out = torch.zeros_like(oss)
    ctx.kem_dec_ptr(S, OTHER, out, oct_, osk)  # (the workspace has its size now)
    ctx.sync_status()
    torch.cuda.synchronize()
    out.zero_()
    torch.cuda.synchronize()
    st, st2 = torch.cuda.Stream(), torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
        ctx.kem_keypair_ptr(S, N, pk, sk, dkc, stream=st.cuda_stream)
        ctx.kem_enc_ptr(S, N, ct, ss, pk, dec_, stream=st.cuda_stream)
        ctx.kem_dec_ptr(S, OTHER, out, oct_, osk, stream=st2.cuda_stream)
    st2.synchronize()
    assert torch.equal(out, oss)
    g.replay()
    torch.cuda.synchronize()
    ctx.sync_status()
    ctx.close()
    wpk, wsk = oracle.kem_keypair_batch(S, kc, threads)
    wct, wss = oracle.kem_enc_batch(S, wpk, ec, threads)
    for got, want in ((pk, wpk), (sk, wsk), (ct, wct), (ss, wss)):
        assert np.array_equal(got.cpu().numpy(), want)


def test_captured_decapsulation_and_mixed_plan(kem):
    """Decapsulation and a mixed plan of such a batch keep their two launches in a graph."""
    import torch
    T, _ = kem
    S = T.LIGHTSABER
    z = T.sizes(S)
    new = lambda w: torch.zeros((N, w), dtype=torch.uint8, device="cuda")
    pk, sk, ct, ss, out, mix = (new(w) for w in (z.pk_bytes, z.sk_bytes, z.ct_bytes, 32, 32, 32))
    ctx = T.Context(0)
    ctx.kem_keypair_ptr(S, N, pk, sk, torch.from_numpy(T.splitmix_bytes(9955, N * 96)).cuda())
    ctx.kem_enc_ptr(S, N, ct, ss, pk, torch.from_numpy(T.splitmix_bytes(9956, N * 32)).cuda())
    ctx.kem_dec_ptr(S, N, out, ct, sk)
    ctx.sync_status()
    out.zero_()
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        ctx.kem_dec_ptr(S, N, out, ct, sk, stream=st.cuda_stream)
    plan = T.MixedPlan(ctx, [(S, mix[:N // 2], ct[:N // 2], sk[:N // 2]), (S, mix[N // 2:], ct[N // 2:], sk[N // 2:])])
    for _ in range(2):
        g.replay()
        plan.launch()
    ctx.sync_status()
    torch.cuda.synchronize()
    assert torch.equal(out, ss) and torch.equal(mix, ss)
    plan.close()
    ctx.close()
