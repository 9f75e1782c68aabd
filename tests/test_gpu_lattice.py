"""GPU backward induction on the reference's lattice (binom_vanilla_eur /
binom_vanilla_amer) against the oracle's restatement, which is pinned bit for
bit to the reference's own outputs: the prices must be identical."""
import pytest

pytestmark = pytest.mark.gpu

CASES = [(100, 100, .05, .2, 1.0), (100, 110, .02, .75, 1.0), (100, 90, .03, .4, .5),
         (50, 60, .08, .3, 2.0)]


@pytest.mark.parametrize("american", [False, True])
@pytest.mark.parametrize("pf", [1, -1])
@pytest.mark.parametrize("N", [1, 2, 7, 100, 1000, 2047, 2048, 2049, 2177, 5000, 20000])
def test_lattice_bit_exact(orc, ctx, N, pf, american):
    import parcompfin_gb300 as pcf
    fn = pcf.binom_vanilla_amer if american else pcf.binom_vanilla_eur
    ref = orc.ref_binom_vanilla_amer if american else orc.ref_binom_vanilla_eur
    for S0, E, r, sig, T in CASES[:1 if N > 5000 else 4]:
        got = fn(S0, E, r, sig, T, N, pf, ctx=ctx)
        want = ref(S0, E, r, sig, T, N, float(pf))
        assert got == want, (S0, E, r, sig, T, N, pf, american, got, want)


def test_lattice_converges_and_orders(orc, ctx):
    import parcompfin_gb300 as pcf
    bs = orc.orc_bs_price(100, 100, .05, .3, 1.0, -1)
    eur = pcf.binom_vanilla_eur(100, 100, .05, .3, 1.0, 100000, "put", ctx=ctx)
    amer = pcf.binom_vanilla_amer(100, 100, .05, .3, 1.0, 100000, "put", ctx=ctx)
    assert abs(eur - bs) < 1e-3
    assert amer > eur + 0.4  # early-exercise premium of the put
    # the American call on a non-dividend stock is the European call
    c_am = pcf.binom_vanilla_amer(100, 100, .05, .3, 1.0, 20000, "call", ctx=ctx)
    c_eu = pcf.binom_vanilla_eur(100, 100, .05, .3, 1.0, 20000, "call", ctx=ctx)
    assert abs(c_am - c_eu) < 1e-12 * c_eu


def test_lattice_rejects_bad_input(ctx):
    import parcompfin_gb300 as pcf
    with pytest.raises(ValueError):
        pcf.binom_vanilla_eur(100, 100, .05, .3, 1.0, 0, "put", ctx=ctx)
    with pytest.raises(ValueError):
        pcf.binom_vanilla_amer(100, 100, .05, .3, 1.0, 3_000_000, "put", ctx=ctx)


@pytest.mark.parametrize("american", [False, True])
@pytest.mark.parametrize("N", [8, 9, 23, 24, 25, 31, 33, 191, 192, 193, 3647, 3648])
def test_lattice_strip_edges_bit_exact(orc, ctx, N, american):
    """Around the strips' edges: 8 levels between exchanges, 24 columns a warp,
    24 columns a block up to 152 blocks, then 48. Both are the same FP64
    operations in the same order, so the prices are equal."""
    import parcompfin_gb300 as pcf
    fn = pcf.binom_vanilla_amer if american else pcf.binom_vanilla_eur
    ref = orc.ref_binom_vanilla_amer if american else orc.ref_binom_vanilla_eur
    for pf in (1, -1):
        for args in CASES[:2 if N < 1000 else 1]:
            assert fn(*args, N, pf, ctx=ctx) == ref(*args, N, float(pf)), (args, N, pf, american)


@pytest.mark.parametrize("N", [7296, 10944, 14592])
def test_lattice_strip_widths_bit_exact(orc, ctx, N):
    """The first N of 72 and 96 columns a block, and of two blocks an SM."""
    import parcompfin_gb300 as pcf
    for american in (True, False):
        fn = pcf.binom_vanilla_amer if american else pcf.binom_vanilla_eur
        ref = orc.ref_binom_vanilla_amer if american else orc.ref_binom_vanilla_eur
        assert fn(100, 110, .02, .75, 1.0, N, -1, ctx=ctx) == ref(100, 110, .02, .75, 1.0, N, -1.0)


@pytest.mark.parametrize("american", [False, True])
@pytest.mark.parametrize("args", [
    (100, 1e300, .05, .2, 1.0, 300, 1),    # no terminal payoff: the price is 0
    (1e-280, 2e-280, .05, .2, 1.0, 60, 1),  # a price below 2^-700
    (100, 100, .05, .2, 1.0, 1, -1),
    (100, 100, 1.5, .2, 1.0, 1, -1),       # R = e^1.5: beyond the fast division's range
    (100, 100, -.2, .3, 2.0, 50, -1),      # R < 1
    (100, 120, .9, .05, 1.0, 2, -1),       # p > 1: negative weights
])
def test_lattice_division_range_bit_exact(orc, ctx, args, american):
    """Prices and parameters outside the three-operation division's range take
    the IEEE division: the reference's value in every case."""
    import parcompfin_gb300 as pcf
    fn = pcf.binom_vanilla_amer if american else pcf.binom_vanilla_eur
    ref = orc.ref_binom_vanilla_amer if american else orc.ref_binom_vanilla_eur
    assert fn(*args, ctx=ctx) == ref(*args[:6], float(args[6]))


def _same(a, b):
    return a == b or (a != a and b != b)


# Lattices whose powers or values leave the FP64 range. (S0, E, r, sigma, T, N):
OUT_OF_RANGE = {
    "inf-times-0": (100, 100, .03, 20.0, 4.0, 1000),     # S0 u^i = inf and d^(N-i) = 0: NaN nodes
    "inf": (100, 100, .03, 18.0, 1.0, 1500),             # S0 u^N = inf alone
    "growing": (100, 1e200, -260.0, 25.3, 1.0, 400),     # R = 0.52: E R^-N overflows
    "zero-d": (100, 100, .03, 30.0, 1.0, 20),            # d rounds to 0
    "zero-d-inf": (100, 100, .03, 60.0, 1.0, 40),
}


@pytest.mark.parametrize("american", [False, True])
@pytest.mark.parametrize("pf", [1, -1])
@pytest.mark.parametrize("name", OUT_OF_RANGE)
def test_lattice_out_of_range_nodes(orc, ctx, name, pf, american):
    """Infinite and not-a-number nodes go where the reference's operations take
    them: the same price, infinite or not a number included."""
    import parcompfin_gb300 as pcf
    fn = pcf.binom_vanilla_amer if american else pcf.binom_vanilla_eur
    ref = orc.ref_binom_vanilla_amer if american else orc.ref_binom_vanilla_eur
    args = OUT_OF_RANGE[name]
    got, want = fn(*args, pf, ctx=ctx), ref(*args, float(pf))
    assert _same(got, want), (name, pf, american, got, want)


WAITS = {2: "right neighbour's nodes", 3: "ring's reader", 4: "courier's words"}


@pytest.mark.parametrize("american", [True, False])
@pytest.mark.parametrize("N", [1200, 4000, 9000, 20000])  # 24, 48, 72 and 96 columns a strip
@pytest.mark.parametrize("withhold", WAITS)
def test_lattice_starved_waits_give_up_then_recover(orc, ctx, withhold, N, american):
    """Each bounded wait between the strips is made to run out: a strip that
    stops publishing, a reader that stops reporting, a courier that stops
    handing on. The call returns PCF_ETIMEOUT and names the wait, with and
    without the warp that computes exercise values; the next call on the same
    context gives the reference's price."""
    import parcompfin_gb300 as pcf
    from parcompfin_gb300._lib import PCF_ETIMEOUT, PcfError
    fn = pcf.binom_vanilla_amer if american else pcf.binom_vanilla_eur
    ref = orc.ref_binom_vanilla_amer if american else orc.ref_binom_vanilla_eur
    args = CASES[0]
    ctx.set_test_lattice(withhold, 2000)
    try:
        with pytest.raises(PcfError, match=WAITS[withhold]) as e:
            fn(*args, N, -1, ctx=ctx)
        assert e.value.status == PCF_ETIMEOUT
    finally:
        ctx.set_test_lattice(0)
    assert fn(*args, N, -1, ctx=ctx) == ref(*args, N, -1.0)


@pytest.mark.parametrize("american", [True, False])
@pytest.mark.parametrize("args", [(100, 110, .02, .75, 1.0, -1), (50, 60, .08, .3, 2.0, 1),
                                  (1e-280, 2e-280, .05, .2, 1.0, -1)])  # last: IEEE division
@pytest.mark.parametrize("above", [1, 127, 128, 129, 256, 257])
def test_lattice_blocked_levels_bit_exact(orc, ctx, above, args, american):
    """The levels above the strips, 128 a grid step, and the hand-over: one
    level, partial and whole steps, an odd and an even number of them (the two
    level arrays alternate), above 800 and 2500 levels of strips."""
    import parcompfin_gb300 as pcf
    fn = pcf.binom_vanilla_amer if american else pcf.binom_vanilla_eur
    ref = orc.ref_binom_vanilla_amer if american else orc.ref_binom_vanilla_eur
    try:
        for top in (800, 2500):
            ctx.set_test_strip_level(top)
            N = top + above
            before = ctx.launches
            got = fn(*args[:5], N, args[5], ctx=ctx)
            assert ctx.launches - before in (2, 4)  # blocked and strips, once or twice
            assert got == ref(*args[:5], N, float(args[5])), (N, top, args, american)
    finally:
        ctx.set_test_strip_level(0)


def test_lattice_blocked_barrier_gives_up_then_recovers(orc, ctx):
    """The grid barrier of the levels above the strips, waiting for a block
    more than there are, gives up; the next call is the reference's price."""
    import parcompfin_gb300 as pcf
    from parcompfin_gb300._lib import PCF_ETIMEOUT, PcfError
    args = (*CASES[0], 2757, -1)
    try:
        ctx.set_test_strip_level(2500)
        ctx.set_test_barrier(1, 2000)
        with pytest.raises(PcfError, match="grid barrier") as e:
            pcf.binom_vanilla_amer(*args, ctx=ctx)
        assert e.value.status == PCF_ETIMEOUT
        ctx.set_test_barrier(0)
        assert pcf.binom_vanilla_amer(*args, ctx=ctx) == orc.ref_binom_vanilla_amer(
            *args[:6], float(args[6]))
    finally:
        ctx.set_test_barrier(0)
        ctx.set_test_strip_level(0)


@pytest.mark.parametrize("american", [True, False])
def test_lattice_under_a_memory_limit(orc, pcf_lib, american):
    """The strips' rings (8 KB a strip) are scratch that the levels above them
    do without: a limit that leaves no room for them is no refusal, and the
    price is the same."""
    import parcompfin_gb300 as pcf
    fn = pcf.binom_vanilla_amer if american else pcf.binom_vanilla_eur
    ref = orc.ref_binom_vanilla_amer if american else orc.ref_binom_vanilla_eur
    for N in (3300, 20_000):
        with pcf.Context(0) as c:
            c.set_memory_limit(1 << 20)
            for args in CASES[:2]:
                assert fn(*args, N, -1, ctx=c) == ref(*args, N, -1.0), (N, args, american)
            if N < 10_000:  # the IEEE division
                args = (1e-280, 2e-280, .05, .2, 1.0, N)
                assert fn(*args, -1, ctx=c) == ref(*args, -1.0)
            with pytest.raises(pcf.PcfError, match="budget"):
                fn(*CASES[0], 40_000, -1, ctx=c)
