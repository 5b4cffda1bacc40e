"""Two host threads, a context and a stream each, with batches whose Keccak
launches ask for different amounts of shared memory (the limit belongs to the
kernel, not to the launch): every call succeeds and gives the same bytes as
alone."""
import threading

import pytest

pytestmark = pytest.mark.gpu

CALLS = 150


def _make(T, ctx, n, seed):
    import torch
    z = T.sizes(T.LIGHTSABLE)
    new = lambda w: torch.empty((n, w), dtype=torch.uint8, device="cuda")
    kc = torch.from_numpy(T.splitmix_bytes(seed, n * 96).reshape(n, 96)).cuda()
    ec = torch.from_numpy(T.splitmix_bytes(seed + 1, n * 32).reshape(n, 32)).cuda()
    pk, sk, ct, ss = new(z.pk_bytes), new(z.sk_bytes), new(z.ct_bytes), new(32)
    ctx.kem_keypair_ptr(T.LIGHTSABLE, n, pk, sk, kc)
    ctx.kem_enc_ptr(T.LIGHTSABLE, n, ct, ss, pk, ec)
    torch.cuda.synchronize()
    return pk, ec, ct, ss, sk


def test_two_contexts_at_once(kem):
    import torch
    T, _ = kem
    sizes = (16384, 39000)  # one block of the first role per SM, and three of a single role's
    ctxs = [T.Context(0) for _ in sizes]
    made = [_make(T, c, n, 9600 + 10 * i) for i, (c, n) in enumerate(zip(ctxs, sizes))]
    errors, start = [], threading.Barrier(len(sizes))

    def work(c, n, m):
        pk, ec, ct, ss, sk = m
        st = torch.cuda.Stream()
        ct2, ss2, ss3 = torch.empty_like(ct), torch.empty_like(ss), torch.empty_like(ss)
        torch.cuda.synchronize()
        start.wait()
        try:
            for _ in range(CALLS):
                c.kem_enc_ptr(T.LIGHTSABLE, n, ct2, ss2, pk, ec, stream=st.cuda_stream)
                c.kem_dec_ptr(T.LIGHTSABLE, n, ss3, ct, sk, stream=st.cuda_stream)
            st.synchronize()
            c.sync_status()
            assert torch.equal(ct2, ct) and torch.equal(ss2, ss) and torch.equal(ss3, ss)
        except Exception as e:  # reported by the test's own thread
            errors.append((n, repr(e)))

    ts = [threading.Thread(target=work, args=(c, n, m)) for c, n, m in zip(ctxs, sizes, made)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    for c in ctxs:
        c.close()
    assert not errors
