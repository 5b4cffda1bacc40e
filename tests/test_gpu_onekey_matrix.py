"""One-key decapsulation whose re-encryption is one matrix product (6144
ciphertexts and more), and whose decryption is (8192; 16384 for l = 4): both
sides of those lines, blocks of 128 ciphertexts with a remainder, runs of output
polynomials that start inside a block, one to four blocks an SM, against the
oracle, from device and from host buffers; and the secrets that the decryption
accepts."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 4


@pytest.mark.parametrize("set_id,n", [(1, 6143), (1, 6144), (1, 6145), (0, 6271), (2, 6272), (3, 6273), (4, 6144 + 64),
                                      (5, 6144 + 65), (1, 152 * 128), (2, 152 * 128 + 1), (3, 152 * 64 - 1),
                                      (0, 24577), (5, 20011), (0, 8191), (0, 8192), (3, 8193), (2, 16383), (2, 16384),
                                      (5, 16385), (4, 152 * 256 + 1), (1, 152 * 384 + 5)])
def test_onekey_matches_oracle(kem, oracle, set_id, n):
    import torch
    T, ctx = kem
    pk, sk = oracle.kem_keypair_batch(set_id, T.splitmix_bytes(9100 + n, 96).reshape(1, 96), 1)
    ec = T.splitmix_bytes(9200 + n, n * 32).reshape(n, 32)
    ct, ss = oracle.kem_enc_batch(set_id, np.repeat(pk, n, axis=0), ec, THREADS)
    # one bit off, anywhere: each output polynomial, the first and the last bit
    rows = np.arange(2, n, 5)
    ct[rows, (rows * 37) % ct.shape[1]] ^= (1 << (rows % 8)).astype(np.uint8)
    ct[0, 0] ^= 1
    ct[-1, -1] ^= 0x80
    want, fail = oracle.kem_dec_batch(set_id, ct, np.repeat(sk, n, axis=0), THREADS)
    assert fail[0] and fail[-1] and fail[rows].all() and not fail[1]
    out = torch.empty((n, 32), dtype=torch.uint8, device="cuda")
    ctx.kem_dec_onekey_ptr(set_id, n, out, torch.from_numpy(ct).cuda(), torch.from_numpy(sk[0]).cuda())
    ctx.sync_status()
    assert np.array_equal(out.cpu().numpy(), want)
    assert np.array_equal(ctx.kem_dec_onekey(set_id, ct, sk[0]), want)


@pytest.mark.parametrize("set_id,l", [(0, 2), (1, 3), (2, 4)])
def test_onekey_secret_range(kem, oracle, set_id, l):
    """-7 .. 7, as the per-instance decryption."""
    T, ctx = kem
    n = 16400
    pk, sk = oracle.kem_keypair_batch(set_id, T.splitmix_bytes(9600, 96).reshape(1, 96), 1)
    ct, _ = oracle.kem_enc_batch(set_id, np.repeat(pk, 16, axis=0), T.splitmix_bytes(9601, 512).reshape(16, 32), 1)
    ct = np.tile(ct, (n // 16, 1))
    rng = np.random.RandomState(5)
    s = rng.randint(-7, 8, 256 * l)
    s[::3] = 7
    s[1::3] = -7

    def pack(v):
        return np.packbits((((v[:, None] & 0x1FFF) >> np.arange(13)) & 1).astype(np.uint8).reshape(-1), bitorder="little")

    sk[0, :416 * l] = pack(s)
    want, _ = oracle.kem_dec_batch(set_id, ct[:16], np.repeat(sk, 16, axis=0), THREADS)
    assert np.array_equal(ctx.kem_dec_onekey(set_id, ct, sk[0]), np.tile(want, (n // 16, 1)))
    for i, bad in enumerate((8, -8, 4095, -4096, 128)):
        t = s.copy()
        t[(97 * i + 3) % (256 * l)] = bad
        sk[0, :416 * l] = pack(t)
        with pytest.raises(T.TmvpError) as e:
            ctx.kem_dec_onekey(set_id, ct, sk[0])
        assert e.value.code == T.EINVAL
