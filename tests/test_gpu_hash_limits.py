"""The caller's limits on the forms of a sponge: setting one to the value it has
changes nothing, and the initial values bring the library's own choice back (seen
by the launches of a small batch, whose last stage then needs none)."""
import pytest

pytestmark = pytest.mark.gpu


def test_initial_limits_are_the_librarys_choice(kem):
    import numpy as np
    T, _ = kem
    ctx = T.Context(0)
    pk, sk = ctx.kem_keypair(T.SABER, T.splitmix_bytes(1, 96).reshape(1, 96))
    ct, ss = ctx.kem_enc(T.SABER, pk, T.splitmix_bytes(2, 32).reshape(1, 32))

    def launches():
        before = ctx.launches
        assert np.array_equal(ctx.kem_dec(T.SABER, ct, sk), ss)
        return ctx.launches - before

    own = launches()
    ctx.set_warp_hash(1024)
    ctx.set_pair_hash(32768)
    assert launches() == own
    ctx.set_warp_hash(0)
    ctx.set_pair_hash(0)
    assert launches() == own + 1
    ctx.set_warp_hash(1024)
    assert launches() == own + 1
    ctx.set_pair_hash(32768)
    assert launches() == own
    ctx.close()
