"""The planner of the Keccak launches (plan_sponges, host code) by itself: no GPU."""
import ctypes

import pytest

SMS = 152
THREAD, WARP, PAIR = 0, 1, 2
PER_BLOCK = {THREAD: 128, WARP: 4, PAIR: 64}
# GenMatrix and H(c) permutations of the six sets, in the library's order
SETS = {"lightsaber": (10, 6), "saber": (23, 9), "firesaber": (40, 11), "lightsable": (9, 5), "sable": (19, 8),
        "firesable": (34, 11)}


class Cfg(ctypes.Structure):
    _fields_ = [("sms", ctypes.c_int), ("limits", ctypes.c_bool), ("warp_max", ctypes.c_size_t),
                ("pair_max", ctypes.c_size_t), ("cap", ctypes.c_int), ("beside", ctypes.c_bool),
                ("even", ctypes.c_bool), ("one", ctypes.c_bool)]


class Seg(ctypes.Structure):
    _fields_ = [("role", ctypes.c_int), ("form", ctypes.c_int), ("block0", ctypes.c_uint), ("first", ctypes.c_uint),
                ("count", ctypes.c_uint)]


class Plan(ctypes.Structure):
    _fields_ = [("nseg", ctypes.c_int), ("blocks", ctypes.c_uint), ("threads", ctypes.c_uint), ("smem", ctypes.c_uint),
                ("seg", Seg * 8)]


class Role(ctypes.Structure):
    _fields_ = [("n", ctypes.c_size_t), ("perms", ctypes.c_int), ("id", ctypes.c_int),
                ("brief", ctypes.c_bool)]


@pytest.fixture(scope="module")
def plan():
    import tmvpkem
    tmvpkem.build.build()
    lib = ctypes.CDLL(tmvpkem.LIB_PATH)
    fn = lib._ZN4tmvp12plan_spongesERKNS_7HashCfgEPKNS_10SpongeRoleEiRA2_NS_10SpongePlanE
    fn.restype = None

    def call(perms, n, **cfg):
        brief = cfg.pop("brief", False)
        c = Cfg(sms=SMS, warp_max=cfg.pop("warp_max", 1024), pair_max=cfg.pop("pair_max", 32768), **cfg)
        roles = (Role * len(perms))(*[Role(n, p, i, brief) for i, p in enumerate(perms)])
        out = (Plan * 2)()
        fn(ctypes.byref(c), roles, len(perms), out)
        return out

    return call


@pytest.mark.parametrize("name", SETS)
@pytest.mark.parametrize("n", [9729, 16384, 29184, 32768, 65536])
def test_a_capped_front_holds_no_shared_memory(plan, name, n):
    """The cap is there to leave room for decryption CTAs: the plan that a capped
    front strides over is one launch and asks for no shared memory."""
    main, second = plan(SETS[name], n, beside=True, cap=4)
    assert main.seg[0].form == THREAD and main.blocks > 0
    assert main.smem == 0 and second.blocks == 0


@pytest.mark.parametrize("perms,brief,times", [((9,), False, (1, 1)), ((40,), False, (1, 1)), ((23, 9), False, (2, 2)),
                                               ((6,), True, (4, 2)), ((1,), True, (4, 2))])
def test_the_callers_limits_count_each_sponge_once(plan, perms, brief, times):
    """... but those of G, the final key and the key-generation tail four times
    against the warp limit and twice against the pair limit, whatever their length."""
    for form, limit, k in ((WARP, 1024, times[0]), (PAIR, 32768, times[1])):
        at, above = limit // k, limit // k + 1
        cfg = dict(limits=True, pair_max=32768 if form == PAIR else 0)
        assert plan(perms, at, brief=brief, **cfg)[0].seg[0].form == form
        assert plan(perms, above, brief=brief, **cfg)[0].seg[0].form == THREAD
