"""Two host threads, a context and a stream each, with batches whose Keccak
launches ask for different amounts of shared memory (the limit belongs to the
kernel, not to the launch): every call succeeds and gives the same bytes as
alone."""
import threading

import pytest

pytestmark = pytest.mark.gpu

CALLS = 150


def _make(T, ctx, set_id, n, seed):
    import torch
    z = T.sizes(set_id)
    new = lambda w: torch.empty((n, w), dtype=torch.uint8, device="cuda")
    kc = torch.from_numpy(T.splitmix_bytes(seed, n * 96).reshape(n, 96)).cuda()
    ec = torch.from_numpy(T.splitmix_bytes(seed + 1, n * 32).reshape(n, 32)).cuda()
    pk, sk, ct, ss = new(z.pk_bytes), new(z.sk_bytes), new(z.ct_bytes), new(32)
    ctx.kem_keypair_ptr(set_id, n, pk, sk, kc)
    ctx.kem_enc_ptr(set_id, n, ct, ss, pk, ec)
    torch.cuda.synchronize()
    return pk, ec, ct, ss, sk


def _both_at_once(T, jobs, form):
    """Encapsulates and decapsulates each (set, n) of jobs on a thread of its own."""
    import torch
    ctxs = [T.Context(0) for _ in jobs]
    made = [_make(T, c, s, n, 9600 + 10 * i) for i, (c, (s, n)) in enumerate(zip(ctxs, jobs))]
    errors, start = [], threading.Barrier(len(jobs))

    def work(c, job, m):
        set_id, n = job
        pk, ec, ct, ss, sk = m
        st = torch.cuda.Stream()
        ct2, ss2, ss3 = torch.empty_like(ct), torch.empty_like(ss), torch.empty_like(ss)
        torch.cuda.synchronize()
        start.wait()
        try:
            for _ in range(CALLS):
                c.kem_enc_ptr(set_id, n, ct2, ss2, pk, ec, form, stream=st.cuda_stream)
                c.kem_dec_ptr(set_id, n, ss3, ct, sk, form, stream=st.cuda_stream)
            st.synchronize()
            c.sync_status()
            assert torch.equal(ct2, ct) and torch.equal(ss2, ss) and torch.equal(ss3, ss)
        except Exception as e:  # reported by the test's own thread
            errors.append((job, repr(e)))

    ts = [threading.Thread(target=work, args=a) for a in zip(ctxs, jobs, made)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    for c in ctxs:
        c.close()
    assert not errors


def test_two_contexts_at_once(kem):
    T, _ = kem
    # one block of the first role per SM, and three of a single role's
    _both_at_once(T, [(T.LIGHTSABLE, 16384), (T.LIGHTSABLE, 39000)], T.FORM_AUTO)


@pytest.mark.parametrize("form", ["FORM_CUDA_CORE", "FORM_INT8_TC", "FORM_FP8_TC", "FORM_DP2A", "FORM_TOOM_COOK"])
def test_two_sets_of_one_kernel(kem, form):
    """Saber and Sable have one kernel per form and step, with different layouts."""
    T, _ = kem
    _both_at_once(T, [(T.SABER, 600), (T.SABLE, 601)], getattr(T, form))


def test_two_sets_of_the_persistent_kernel(kem):
    T, _ = kem
    jobs = [(T.LIGHTSABER, 600), (T.FIRESABLE, 601)]
    try:
        for step in range(5):
            for s, _n in jobs:
                T.tune_set(step, s, 1)
        _both_at_once(T, jobs, T.FORM_FP8_TCGEN05)
    finally:
        T.tune_clear()
