"""The planner of the Keccak launches (plan_sponges, host code) by itself: no GPU."""
import ctypes

import pytest

SMS = 152
THREAD, WARP, PAIR = 0, 1, 2
PER_BLOCK = {THREAD: 128, WARP: 4, PAIR: 64}
W = 4 * SMS  # sub-partitions
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


# permutations of every two-role stage: decapsulation front, encapsulation front, key generation
GS, HPK = (4, 5, 5, 1, 2, 2), (5, 8, 10, 5, 7, 10)
STAGES = ([(gm, h) for gm, h in SETS.values()] +
          [(gm, 2 + hp + gs) for (gm, _), gs, hp in zip(SETS.values(), GS, HPK)] +
          [(gm + 1, gs) for (gm, _), gs in zip(SETS.values(), GS)])
LINES = [W, 3 * W // 2, 2 * W, 9 * W // 4, 11 * W // 4, 11 * W // 8, 9 * W // 8, 16 * W, 24 * W, 32 * W, 48 * W]
COUNTS = sorted({1, 2, 31, 33} | {n + d for n in LINES for d in (-1, 0, 1)} |
                {r * 32 * W + d for r in (1, 2, 3, 5, 6) for d in (-1, 0, 1, 700, 16 * W + 1, 20 * W, 17 * W)} |
                {9800, 12500, 14001, 16384, 20011, 65536, 1 << 20})


@pytest.mark.parametrize("perms", sorted(set(STAGES)) + [(1,), (3,), (10,), (40,)])
@pytest.mark.parametrize("cfg", [{}, {"beside": True}, {"beside": True, "even": True}, {"beside": True, "cap": 3},
                                 {"one": True}, {"limits": True, "warp_max": 0}, {"limits": True, "pair_max": 0}])
def test_a_plan_takes_every_sponge_once(plan, perms, cfg):
    for n in COUNTS:
        both = plan(perms, n, **cfg)
        split = len(perms) == 2 and not cfg.get("limits") and not cfg.get("one") and 128 * SMS <= n < 192 * SMS
        assert (both[1].blocks > 0) == split
        taken = [[] for _ in perms]
        for p in both:
            blocks = 0
            for s in p.seg[:p.nseg]:
                assert s.block0 == blocks and s.count > 0
                blocks += -(-s.count // PER_BLOCK[s.form])
                taken[s.role].append((s.first, s.first + s.count))
            assert p.blocks == blocks and p.smem <= 117000 and p.nseg <= 8
        for t in taken:
            t.sort()
            assert t[0][0] == 0 and t[-1][1] == n
            assert all(a[1] == b[0] for a, b in zip(t, t[1:]))


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


@pytest.mark.parametrize("perms", [9, 23, 40])
@pytest.mark.parametrize("rounds,most", [(1, W - 1), (2, 2 * W), (3, 9 * W // 4)])
def test_the_rest_of_one_role_leaves_the_warp_form_early(plan, perms, rounds, most):
    """Beside one or two rounds more sponges than that take longer in the warp
    form than in pairs, and longer than no plan at all."""
    for rest, form in ((most, WARP), (most + 1, PAIR)):
        p = plan((perms,), rounds * 32 * W + rest)[0]
        assert [s.form for s in p.seg[:p.nseg]] == [THREAD, form]
