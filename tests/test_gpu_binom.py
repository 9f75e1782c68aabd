"""GPU parity of the closed binomial sum (the reference's binom_embar).

Bars:
  * mode "reference" against the reference's own FP64 result
    (tests/golden/ref_outputs.json, produced by the reference's code) and the
    oracle restatement: 1e-10 relative (the stated bar; the kernel reproduces
    the reference's comb() rounding, so the observed gap is ~1e-14);
  * mode "accurate" against exact 50-digit sums (tests/golden/binom_exact.json):
    1e-12 relative.
"""
import ctypes as C
import json
import math
import os
import random

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
REF_TOL = 1e-10
EXACT_TOL = 1e-12


def _golden(name):
    with open(os.path.join(HERE, "golden", name)) as f:
        return json.load(f)


def rel(a, b):
    return abs(a - b) / max(abs(b), 1e-300)


@pytest.mark.parametrize("case", [c for c in _golden("ref_outputs.json")["cases"]
                                  if c["fn"] == "binom_embar"],
                         ids=lambda c: f"N{c['N']}-E{int(c['E'])}-pf{int(c['payoff_fun'])}")
def test_reference_mode_matches_reference_outputs(ctx, case):
    from parcompfin_gb300 import binom_embar
    v = binom_embar(case["S0"], case["E"], case["r"], case["sigma"], case["T"], case["N"],
                    case["payoff_fun"], ctx=ctx)
    ref = float.fromhex(case["value"])
    assert rel(v, ref) < REF_TOL, (v, ref, rel(v, ref))


def test_reference_mode_random_contracts_vs_oracle(orc, ctx):
    """Contracts drawn like the 1024-contract book (K, r, sigma, T, call/put)
    at N the O(N^2) oracle finishes quickly; one batched launch."""
    from parcompfin_gb300 import binom_embar_batch
    rng = random.Random(7)
    cs = []
    for _ in range(24):
        cs.append((100.0, rng.uniform(80, 120), rng.uniform(.01, .06), rng.uniform(.1, .5),
                   rng.uniform(.25, 2.0), rng.randint(1, 3000), rng.choice([1, -1])))
    got = binom_embar_batch(cs, ctx=ctx)
    worst = 0.0
    for c, v in zip(cs, got):
        ref = orc.ref_binom_embar(*c[:6], float(c[6]))
        worst = max(worst, rel(v, ref))
        assert rel(v, ref) < REF_TOL, (c, v, ref)
    print("worst relative gap", worst)


@pytest.mark.parametrize("N", [199_999, 200_000])
def test_reference_mode_large_n_vs_windowed_oracle(orc, ctx, N):
    """At the largest binomial-book N the full O(N^2) oracle is too slow; the
    oracle's windowed restatement runs the same exact comb() chain for every
    pair index near N/2 (where all of the weight is)."""
    from parcompfin_gb300 import binom_embar
    S0, E, r, sig, T = 100.0, 105.0, .03, .3, 1.5
    w = int(9 * math.sqrt(N)) + 400
    for pf in (1, -1):
        v = binom_embar(S0, E, r, sig, T, N, pf, ctx=ctx)
        part = orc.ref_binom_embar_window(S0, E, r, sig, T, N, float(pf), N // 2 - w, N)
        ref = math.exp(-r * T) * part
        assert rel(v, ref) < REF_TOL, (pf, v, ref)


def test_binomial_book_stratified_sample_vs_reference(orc, ctx):
    """The binomial book (1024 contracts from seed 7, N uneven in
    1e3..2e5) priced in one launch, as the benchmark runs it; a stratified
    sample of 32 contracts, one from each N-stratum of 32, against the
    reference's sum at 1e-10. The oracle restates comb()'s exact sequential
    chain for every pair index within 9 sqrt(N) + 400 of the binomial
    weights' centres (N p and N p u / R, and their mirrors), which holds all
    of the weight; the full O(N^2) sum would take ~25 CPU-hours for the book.
    The sample's oracle sums run in parallel threads (ctypes releases the
    interpreter lock)."""
    from concurrent.futures import ThreadPoolExecutor

    import parcompfin_gb300 as pcf
    from parcompfin_gb300 import workloads
    book = workloads.binom_book()
    got = pcf.binom_embar_batch(book, ctx=ctx)
    order = sorted(range(len(book)), key=lambda i: book[i][5])
    sample = order[16::32]
    assert len(sample) == 32 and book[sample[0]][5] < 10_000 and book[sample[-1]][5] > 190_000

    def ref(i):
        S0, E, r, sig, T, N, pf = book[i]
        lat = (C.c_double * 5)()
        orc.ref_lattice(r, sig, T, N, lat)
        p, u, R = lat[2], lat[0], lat[4]
        centre = min(N * p, N * (1 - p), N * p * u / R, N * (1 - p * u / R))
        lo = max(0, int(centre - 9 * math.sqrt(N) - 400))
        return math.exp(-r * T) * orc.ref_binom_embar_window(S0, E, r, sig, T, N, float(pf), lo, N)

    with ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
        refs = list(ex.map(ref, sample))
    worst = 0.0
    for i, v in zip(sample, refs):
        worst = max(worst, rel(got[i], v))
        assert rel(got[i], v) < REF_TOL, (book[i], got[i], v)
    print("binomial book sample: worst relative gap", worst)


def test_reference_50000_survey_value(ctx):
    from parcompfin_gb300 import binom_embar
    v = binom_embar(100, 100, .05, .2, 1, 50000, 1, ctx=ctx)
    assert rel(v, 10.450553297126545) < REF_TOL


@pytest.mark.parametrize("case", _golden("binom_exact.json")["cases"],
                         ids=lambda c: f"N{c['contract'][5]}")
def test_accurate_mode_matches_exact_sum(ctx, case):
    from parcompfin_gb300 import binom_embar
    c = case["contract"]
    v = binom_embar(*c, mode="accurate", ctx=ctx)
    assert rel(v, case["exact"]) < EXACT_TOL, (v, case["exact"])
    vr = binom_embar(*c, mode="reference", ctx=ctx)
    assert rel(vr, case["reference"]) < REF_TOL


def test_accurate_mode_converges_to_black_scholes(orc, ctx):
    from parcompfin_gb300 import binom_embar
    bs = orc.orc_bs_price(100, 100, .05, .2, 1.0, 1)
    v = binom_embar(100, 100, .05, .2, 1.0, 200_000, 1, mode="accurate", ctx=ctx)
    assert abs(v - bs) < 1e-4


def test_batch_equals_single(ctx):
    from parcompfin_gb300 import binom_embar, binom_embar_batch
    cs = [(100.0, 95.0, .02, .25, 1.0, 1234, 1), (100.0, 101.0, .04, .35, .75, 5001, -1),
          (100.0, 110.0, .02, .75, 1.0, 1000, 1)]
    b = binom_embar_batch(cs, ctx=ctx)
    for c, v in zip(cs, b):
        assert v == binom_embar(*c, ctx=ctx)


def test_edge_cases(orc, ctx):
    from parcompfin_gb300 import binom_embar
    for N in (1, 2, 3, 4):
        for pf in (1, -1):
            v = binom_embar(100, 100, .05, .2, 1, N, pf, ctx=ctx)
            ref = orc.ref_binom_embar(100, 100, .05, .2, 1, N, float(pf))
            assert rel(v, ref) < REF_TOL
    with pytest.raises(ValueError):
        binom_embar(100, 100, .05, .2, 1, 0, 1, ctx=ctx)
    with pytest.raises(ValueError):
        binom_embar(100, 100, .05, .2, 1, 2_000_000, 1, ctx=ctx)
    with pytest.raises(ValueError, match="Unknown payoff"):
        binom_embar(100, 100, .05, .2, 1, 100, "straddle", ctx=ctx)


def test_reference_mode_small_and_edge_n_vs_oracle(orc, ctx):
    """Every N up to 70 (the accumulator's low binades, whose ties are dense)
    and N around multiples of the 256-term blocks and the 32 serial steps of
    the accumulator's walk, one batch. A term is the reference's up to the
    rounding of its two powers and its exponential (2^-57 against one ulp) and
    all terms are positive, so 1e-13 leaves a factor of 100."""
    from parcompfin_gb300 import binom_embar_batch
    rng = random.Random(3)
    cs = [(100.0, rng.uniform(80, 120), rng.uniform(.01, .06), rng.uniform(.1, .5),
           rng.uniform(.25, 2.0), N, pf)
          for N in list(range(1, 71)) + [255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2049]
          for pf in (1, -1)]
    for c, v in zip(cs, binom_embar_batch(cs, ctx=ctx)):
        ref = orc.ref_binom_embar(*c[:6], float(c[6]))
        assert abs(v - ref) <= 1e-13 * abs(ref) + 1e-300, (c, v, ref)


def test_reference_mode_wide_powers_vs_oracle(orc, ctx):
    """A contract whose powers span almost the whole FP64 range takes the FP64
    pow and exp; one just below the switch the fixed-point ones. Both agree
    with the reference's sum, alone and in one batch."""
    from parcompfin_gb300 import binom_embar, binom_embar_batch
    N, T = 2000, 4.0
    cs = []
    for span in (690.0 - 20.0, 702.0):  # log u times N
        sig = (span / N) * math.sqrt(N / T)
        for _ in range(20):  # log u depends on the drift too: settle it
            lat = (C.c_double * 5)()
            orc.ref_lattice(.03, sig, T, N, lat)
            sig *= (span / N) / math.log(lat[0])
        for pf in (1, -1):
            cs.append((1.0, 2.0, .03, sig, T, N, pf))
    got = binom_embar_batch(cs, ctx=ctx)
    for c, v in zip(cs, got):
        ref = orc.ref_binom_embar(*c[:6], float(c[6]))
        assert rel(v, ref) < REF_TOL, (c, v, ref)
        assert binom_embar(*c, ctx=ctx) == v


def _exact_binom(orc, S0, E, r, sig, T, N, pf):
    """The sum over the lattice's FP64 u, d, p in 60-digit decimals: weights
    and share prices by their ratios from k = 0."""
    from decimal import Decimal, getcontext
    getcontext().prec = 60
    getcontext().Emin, getcontext().Emax = -10**8, 10**8
    lat = (C.c_double * 5)()
    orc.ref_lattice(r, sig, T, N, lat)
    u, d, p = (Decimal(lat[k]) for k in range(3))
    q = 1 - p
    w, S, odds, step = q ** N, Decimal(S0) * d ** N, p / q, u / d
    total = Decimal(0)
    for k in range(N + 1):
        pay = pf * (S - Decimal(E))
        if pay > 0:
            total += w * pay
        w = w * (N - k) / (k + 1) * odds
        S *= step
    return math.exp(-r * T) * float(total)


@pytest.mark.parametrize("N", [1, 2, 15, 16, 17, 35, 36, 81, 100, 501, 502, 1001, 30_000, 200_000])
def test_accurate_mode_matches_exact_decimals(orc, ctx, N):
    """Around the boundaries of the weights' series, at p away from 1/2 too."""
    from parcompfin_gb300 import binom_embar
    for r, sig, T, pf in ((.03, .3, 1.5, 1), (.25, .2, 2.0, -1)):
        if N >= 30_000 and pf < 0:
            continue
        ref = _exact_binom(orc, 100.0, 105.0, r, sig, T, N, pf)
        v = binom_embar(100.0, 105.0, r, sig, T, N, pf, mode="accurate", ctx=ctx)
        assert abs(v - ref) <= EXACT_TOL * abs(ref), (N, r, v, ref)


def test_first_tables_beside_a_busy_default_stream(ctx):
    """A context's first sum uploads its tables on the context's own stream and
    waits for them, whatever the default stream has queued; so do larger
    tables and the tables after a release."""
    torch = pytest.importorskip("torch")
    from parcompfin_gb300 import Context, binom_embar
    args = (100.0, 105.0, .03, .3, 1.5)
    want = {N: binom_embar(*args, N, -1, ctx=ctx) for N in (1000, 50_000)}
    with Context(0) as c:
        for _ in range(2):
            for N in (1000, 50_000):
                torch.cuda._sleep(100_000_000)  # about 50 ms on the default stream
                assert binom_embar(*args, N, -1, ctx=c) == want[N]
                torch.cuda.synchronize()
            c.release()


@pytest.mark.parametrize("r,sig,T,N", [(.06, .02, 2.0, 2001), (.1, .02, 5.0, 20_001),
                                       (.1, .005, 10.0, 50_001), (.05, .01, 1.0, 30_000)])
@pytest.mark.parametrize("sign", [1, -1])
def test_accurate_mode_away_from_even_odds(orc, ctx, r, sig, T, N, sign):
    """Drifts of 3 to 20 volatilities, p above and below 1/2: of a pair's two weights
    either may be the one that matters, also for a payoff that only the smaller
    one has (strikes at the forward and three deviations to both sides).
    Bound: N p and N q are rounded, which moves a weight's logarithm by
    |k - N p| 2^-53 each; within four deviations, |k - N p| <= 2 sqrt(N). Eight
    more units for the logarithm's other terms, the powers and the sum."""
    from parcompfin_gb300 import binom_embar_batch
    r *= sign
    forward = 100.0 * math.exp(r * T)
    cs = [(100.0, forward * math.exp(k * sig * math.sqrt(T)), r, sig, T, N, pf)
          for k in (-3, 0, 3) for pf in (1, -1)]
    for c, v in zip(cs, binom_embar_batch(cs, mode="accurate", ctx=ctx)):
        ref = _exact_binom(orc, *c)
        assert abs(v - ref) <= (8 + 2 * math.sqrt(N)) * 2**-52 * ref, (c, v, ref, rel(v, ref))


@pytest.mark.parametrize("mode", ["reference", "accurate"])
def test_batch_under_a_memory_limit(ctx, mode):
    """A batch whose scratch exceeds the context's limit is priced in parts,
    with the prices of the whole batch."""
    from parcompfin_gb300 import Context, binom_embar_batch
    rng = random.Random(11)
    cs = [(100.0, rng.uniform(80, 120), rng.uniform(.01, .06), rng.uniform(.1, .5),
           rng.uniform(.25, 2.0), rng.randint(1, 300), rng.choice([1, -1])) for _ in range(5001)]
    want = binom_embar_batch(cs, mode=mode, ctx=ctx)
    with Context(0) as c:
        c.set_memory_limit(1 << 20)
        assert binom_embar_batch(cs, mode=mode, ctx=c) == want
