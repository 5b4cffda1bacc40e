"""Secret coefficients that the tcgen05 form accepts: -7 .. 7, at every position
of a packed word and next to each other; everything else is refused, for the
13-bit fields of a secret key and for matvec's bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pack13(v):
    bits = ((v[:, None] & 0x1FFF) >> np.arange(13)) & 1
    return np.packbits(bits.astype(np.uint8).reshape(-1), bitorder="little")


@pytest.mark.parametrize("set_id,l", [(0, 2), (1, 3), (2, 4)])
def test_decryption_keys(kem, oracle, set_id, l):
    T, ctx = kem
    n = 8
    pk, sk = ctx.kem_keypair(set_id, T.splitmix_bytes(9500, n * 96).reshape(n, 96))
    ct, _ = ctx.kem_enc(set_id, pk, T.splitmix_bytes(9501, n * 32).reshape(n, 32))
    rng = np.random.RandomState(17 + set_id)
    # accepted: all of -7 .. 7, the neighbours -1, 7 and 7, -7 in every phase of the packing
    for r in range(n):
        s = rng.randint(-7, 8, 256 * l)
        if r % 2:
            s[r // 2::4] = -1
            s[r // 2 + 1::4] = 7
            s[r // 2 + 2::4] = -7
        sk[r, :416 * l] = _pack13(s)
    want, _ = oracle.kem_dec_batch(set_id, ct, sk, 4)
    assert np.array_equal(ctx.kem_dec(set_id, ct, sk, form=T.FORM_FP8_TCGEN05), want)
    good = sk.copy()
    for i, bad in enumerate((8, -8, 9, -9, 127, 128, -128, 256, 4095, -4096, 16, -16)):
        s = rng.randint(-7, 8, 256 * l)
        s[(37 * i + 5) % (256 * l)] = bad
        sk = good.copy()
        sk[i % n, :416 * l] = _pack13(s)
        with pytest.raises(T.TmvpError) as e:
            ctx.kem_dec(set_id, ct, sk, form=T.FORM_FP8_TCGEN05)
        assert e.value.code == T.EINVAL


@pytest.mark.parametrize("l", [2, 3, 4])
def test_matvec_bytes(kem, oracle, l):
    T, ctx = kem
    n = 9
    rng = np.random.RandomState(23 + l)
    A = rng.randint(0, 8192, (n, l, l, 256)).astype(np.uint16)
    s = rng.randint(-7, 8, (n, l, 256)).astype(np.int8)
    s[:, :, ::3] = -7
    s[:, :, 1::3] = 7
    assert np.array_equal(ctx.matvec(A, s, form=T.FORM_FP8_TCGEN05), oracle.matvec(A, s, eq=13, nthreads=4))
    for i, bad in enumerate((8, -8, 9, -9, 16, -16, 120, 127, -128)):
        t = s.copy()
        t[i % n, i % l, (41 * i + 3) % 256] = bad
        with pytest.raises(T.TmvpError) as e:
            ctx.matvec(A, t, form=T.FORM_FP8_TCGEN05)
        assert e.value.code == T.EINVAL
