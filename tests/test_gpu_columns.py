"""The FP64 column passes (limiter flags, explicit update, implicit sweep, dry
levels with diagnostics) at the sizes where their blocks, patches, level chunks
and stages can go wrong, bit for bit against the oracle: grids one column short
of, at and beyond the 32 x 4 blocks and 8 x 4 patches, chunks of up to 4 levels
on small grids and of up to 56 on large ones, level counts around the stages'
eight, row pitches with and without TMA boxes, closed and folded boundaries."""
import numpy as np
import pytest

import pyoracle

CASES = [
    # nx, ny, km, cyclic, tripole, hypsometry
    (8, 8, 3, 1, 1, 0),
    (28, 9, 4, 1, 1, 1),
    (30, 28, 8, 1, 1, 1),
    (29, 12, 9, 0, 0, 1),
    (33, 13, 17, 1, 0, 1),
    (61, 31, 33, 0, 0, 1),
    (64, 40, 65, 1, 1, 1),
]


def compare(lt, syn, f, steps, diagnostics):
    dom = lt.TracerDomain(syn.nx, syn.ny, syn.km, syn.params, precision=lt.PREC_FP64, diagnostics=diagnostics,
                          ew_cyclic=bool(syn.cfg.ew_cyclic), tripole=bool(syn.cfg.tripole))
    o = pyoracle.Oracle(syn.nx, syn.ny, syn.km, syn.params, ew_cyclic=syn.cfg.ew_cyclic, tripole=syn.cfg.tripole)
    o.load(f)
    o.sum_order(1)
    for n in lt.INPUT_FIELDS:
        dom.set(n, f[n])
    dom.step(steps)
    dom.sync()
    o.step(steps)
    for n in ("AT", "ATB", "WS", "NET") + (("AX", "AY", "AZ", "DZ", "PENETRATE", "TEND", "DT_DIFF") if diagnostics else ()):
        g, r = dom.get(n), o.get(n)
        assert g.tobytes() == r.tobytes(), (n, float(np.nanmax(np.abs(g - r))), int((g != r).sum()))
    dom.close()


@pytest.mark.gpu
@pytest.mark.parametrize("diagnostics", [False, True])
@pytest.mark.parametrize("nx,ny,km,cyclic,tripole,hyp", CASES)
def test_column_passes_bitexact(lt, nx, ny, km, cyclic, tripole, hyp, diagnostics):
    syn = lt.Synth(nx, ny, km, seed=17 + nx, forced=1, ew_cyclic=cyclic, tripole=tripole, hypsometry=hyp,
                   cap_north=0 if tripole else 2, cap_south=2)
    f = syn.all_fields()
    compare(lt, syn, f, 3, diagnostics)


def large(lt, nx, ny, km, cyclic, tripole, hyp):
    return lt.Synth(nx, ny, km, seed=3 + km, forced=1, ew_cyclic=cyclic, tripole=tripole, hypsometry=hyp,
                    cap_north=0 if tripole else 2, cap_south=2)


# Grids whose continuity marches (74 tiles and more), with and without TMA row
# pitches; the larger ones run the Laplacian in a launch of its own and long
# chunks of levels, whose slots and barriers are used again and again: 28 levels
# a block at 720 x 460 x 55, 20 at 721 x 461 x 40, 56 at 1180 x 508 x 56.
LARGE = [
    (260, 90, 8, 1, 1, 1),
    (261, 93, 17, 0, 0, 0),
    (720, 460, 55, 1, 1, 0),
    (721, 461, 40, 0, 0, 1),
]


@pytest.mark.gpu
@pytest.mark.parametrize("diagnostics", [False, True])
@pytest.mark.parametrize("nx,ny,km,cyclic,tripole,hyp", LARGE)
def test_large_grids_bitexact(lt, nx, ny, km, cyclic, tripole, hyp, diagnostics):
    syn = large(lt, nx, ny, km, cyclic, tripole, hyp)
    compare(lt, syn, syn.all_fields(), 2 if nx < 300 else 1, diagnostics)


@pytest.mark.gpu
@pytest.mark.parametrize("diagnostics", [False, True])
def test_more_rows_than_a_grid_dimension_of_blocks(lt, diagnostics):
    """262204 rows are 65551 blocks of four: more than a launch's y dimension
    takes.  The step and the convective adjustment after it."""
    syn = large(lt, 8, 262200, 3, 0, 0, 1)
    f = syn.all_fields()
    compare(lt, syn, f, 1, diagnostics)
    if diagnostics:
        dom = lt.TracerDomain(syn.nx, syn.ny, syn.km, syn.params, ew_cyclic=False, tripole=False)
        o = pyoracle.Oracle(syn.nx, syn.ny, syn.km, syn.params, ew_cyclic=0, tripole=0)
        f["AT"] = f["AT"] + np.random.default_rng(1).normal(0.0, 2.0, size=f["AT"].shape) * np.array([1.0, 1e-4])[:, None, None, None]
        o.load(f)
        for n in lt.INPUT_FIELDS:
            dom.set(n, f[n])
        dom.convadj()
        o.convadj()
        dom.sync()
        assert (dom.get("AT") != f["AT"]).any()
        for n in ("AT", "ATB", "DT_CONV"):
            assert dom.get(n).tobytes() == o.get(n).tobytes(), n


@pytest.mark.gpu
def test_longest_chunk_bitexact(lt):
    syn = large(lt, 1180, 508, 56, 1, 1, 1)
    compare(lt, syn, syn.all_fields(), 1, False)


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,km,cyclic,tripole", [(260, 90, 37, 1, 1), (261, 93, 16, 0, 0), (322, 61, 3, 1, 0)])
def test_dry_levels_with_diagnostics_bitexact(lt, nx, ny, km, cyclic, tripole):
    """The diagnostics of dry cells, zeros of either sign that depend on every
    input there: velocities down to a level of each U point's own, above or
    below the bottom, zeros of both signs beneath; a quarter of the grid and the
    land in it without any flow."""
    syn = large(lt, nx, ny, km, cyclic, tripole, 1)
    f = syn.all_fields()
    rng = np.random.default_rng(km)
    jmt, imt = f["KMT"].shape
    depth = rng.integers(0, km + 1, size=(jmt, imt))
    depth[:, : imt // 4] = 0
    depth[jmt // 2 :, imt // 2 :] = np.minimum(depth, 1)[jmt // 2 :, imt // 2 :]
    flow = np.arange(km)[:, None, None] < depth
    for n in ("UTF", "VTF", "UTL", "VTL"):
        v = rng.normal(0.0, 0.1, size=f[n].shape)
        f[n] = np.where(flow, v, np.copysign(0.0, v))
    compare(lt, syn, f, 2, True)


@pytest.mark.gpu
def test_batch_members_with_diagnostics(lt):
    """Members with diagnostics, one whose continuity marches (and so leaves its
    dry levels to the last launch's blocks) and one whose does not, in a batch's
    graph: as stepped alone."""
    sizes = [(260, 90, 17), (61, 33, 9)]
    kw = dict(tripole=0, ew_cyclic=0, cap_north=2, cap_south=2, forced=1)
    alone, both = ([lt.Synth(*s, seed=k, **kw).domain(precision=lt.PREC_FP64, diagnostics=True)
                    for k, s in enumerate(sizes)] for _ in range(2))
    b = lt.Batch(both)
    b.step(3)
    b.sync()
    for x, y in zip(alone, both):
        x.step(3)
        x.sync()
        for n in ("AT", "ATB", "NET", "AX", "AY", "AZ", "DZ", "PENETRATE", "TEND", "DT_DIFF"):
            assert x.get(n).tobytes() == y.get(n).tobytes(), n
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,km,cyclic,tripole", [(40, 30, 9, 1, 1), (261, 93, 9, 0, 0)])
def test_diagnostics_of_denormal_values_bitexact(lt, nx, ny, km, cyclic, tripole):
    """Values and velocities whose products are below the smallest normal
    number, where a factor of two before a rounding is not one after it, and
    values beyond the limiter's masks of 1e10."""
    syn = large(lt, nx, ny, km, cyclic, tripole, 1)
    f = syn.all_fields()
    rng = np.random.default_rng(1)
    values = np.array([0.0, -0.0, 5e-324, 1e-310, -1e-310, -1e-300, 1e-200, 1e-122, 2e10, -2e10, 1e30])
    for n, share, v in (("AT", 0.5, values), ("ATB", 0.3, values), ("UTF", 0.2, values[:8]), ("VTF", 0.2, values[:8])):
        f[n] = np.where(rng.random(f[n].shape) < share, rng.choice(v, size=f[n].shape), f[n])
    dom = lt.TracerDomain(nx, ny, km, syn.params, diagnostics=True, ew_cyclic=bool(cyclic), tripole=bool(tripole))
    o = pyoracle.Oracle(nx, ny, km, syn.params, ew_cyclic=cyclic, tripole=tripole)
    o.load(f)
    o.sum_order(1)
    for n in lt.INPUT_FIELDS:
        dom.set(n, f[n])
    dom.step(1)
    dom.sync()
    o.step(1)
    for n in ("WS", "NET", "AX", "AY", "AZ", "DZ", "PENETRATE"):
        assert dom.get(n).tobytes() == o.get(n).tobytes(), n
    # a dry cell's -0 is kept, where the reference's masked terms make it +0
    np.testing.assert_array_equal(dom.get("AT"), o.get("AT"))
    dom.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,km", [(8, 8, 3), (36, 40, 55), (130, 90, 7), (300, 130, 12)])
def test_chained_launches_keep_order(lt, nx, ny, km, precision):
    """Steps launched without a pause, of two domains in turn on their own
    streams and of grids on both sides of the chained launches' line, equal
    steps with the host waiting after each."""
    syn = lt.Synth(nx, ny, km, seed=5, forced=1)
    f = syn.all_fields()
    doms = []
    for _ in range(3):
        d = lt.TracerDomain(nx, ny, km, syn.params, precision=lt.PREC_FP64 if precision == "fp64" else lt.PREC_MIXED)
        for n in lt.INPUT_FIELDS:
            d.set(n, f[n])
        doms.append(d)
    for _ in range(6):
        doms[0].step(1)
        doms[0].sync()
    for _ in range(3):
        doms[1].step(2)
        doms[2].step(2)
    for n in ("AT", "ATB", "NET"):
        r = doms[0].get(n)
        for d in doms[1:]:
            assert d.get(n).tobytes() == r.tobytes(), n


def test_quotient_by_reciprocal_is_correctly_rounded():
    """The face divisions' two-step form (a*y, then q - y*(h*q - a) twice, y the
    rounded reciprocal) equals IEEE division for dividends and divisors of the
    admitted range, zeros of both signs included: exact rational arithmetic
    stands in for the fused operations."""
    from fractions import Fraction

    def fma(a, b, c):
        v = Fraction(a) * Fraction(b) + Fraction(c)
        if v == 0:   # the sign of an exact zero: that of the sum of signed zeros, else plus
            p = a * b if a == 0 or b == 0 else 0.0
            return p + c if p == 0 and c == 0 else 0.0
        return v.numerator / v.denominator

    def divide(a, h):
        y = 1.0 / h
        q = a * y
        q = fma(-fma(h, q, -a), y, q)
        return fma(-fma(h, q, -a), y, q)

    rng = np.random.default_rng(3)
    n = 20000
    a = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-120, 120, n) * rng.choice([-1.0, 1.0], n)
    h = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-60, 60, n)
    # hard cases: mantissas at either end, quotients next to a rounding boundary
    a[:2000] = np.nextafter(2.0 ** rng.integers(-20, 20, 2000).astype(float), 0.0)
    h[1000:3000] = np.nextafter(2.0 ** rng.integers(-20, 20, 2000).astype(float), np.inf)
    a[3000:6000] = h[3000:6000] * np.nextafter(a[3000:6000], np.inf)
    a[6000], a[6001] = 0.0, -0.0
    for x, d in zip(a.tolist(), h.tolist()):
        got, want = divide(x, d), x / d
        assert got == want and np.signbit(got) == np.signbit(want), (x, d, got, want)
