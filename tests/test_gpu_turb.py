"""GPU parity of the Canuto turbulence closure (lt_turb) against the CPU
oracle, which is itself pinned bit for bit to the reference's turb_cu
(test_turb_pin).  The kernel keeps the reference's operation order
(-fmad=false), but log, atan, sin, cos and acosh are CUDA's rather than the
host C library's, so the diffusivities agree to a stated relative tolerance
of 1e-12 (a few units in the last place, carried through the table
interpolation); the parts that use none of those functions (tidal mixing,
mixed-layer depth, tidal diagnostics) agree bit for bit."""
import numpy as np
import pytest
from turb_case import DFRICMX, NCC, case, tables

import pyoracle

pytestmark = pytest.mark.gpu

RTOL = 1e-12
EXACT = ["AK_TIDE", "AMLD", "RICHARDSON", "FZTIDAL", "WP3_TIDAL"]
CLOSE = ["AKT", "AKMT"]


@pytest.fixture(scope="module")
def tab(lt):
    t = lt.TurbTab(tables(lt))
    yield t
    t.close()


def gpu_run(lt, syn, f, tab, precision):
    dom = lt.TracerDomain(syn.nx, syn.ny, syn.km, syn.params, precision=precision,
                          ew_cyclic=bool(syn.cfg.ew_cyclic), tripole=bool(syn.cfg.tripole))
    for n in lt.INPUT_FIELDS + lt.TURB_FIELDS:
        dom.set(n, f[n])
    dom.turb(tab, ncc=NCC, dfricmx=DFRICMX)
    dom.sync()
    return dom


def oracle_run(lt, syn, f):
    o = pyoracle.Oracle(syn.nx, syn.ny, syn.km, syn.params, ew_cyclic=syn.cfg.ew_cyclic, tripole=syn.cfg.tripole)
    o.load(f)
    o.turb(lt.turb_tables_struct(tables(lt)), NCC, DFRICMX)
    return o


def compare(dom, o):
    for n in EXACT:
        g, r = dom.get(n), o.get(n)
        assert np.array_equal(g.view(np.uint64), r.view(np.uint64)), n
    for n in CLOSE:
        g, r = dom.get(n), o.get(n)
        np.testing.assert_allclose(g, r, rtol=RTOL, atol=0, err_msg=n)
        same = np.mean(g == r)
        print("%s: %.4f of the values bit-identical" % (n, same))


@pytest.mark.parametrize("seed,forced", [(3, 1), (8, 0), (21, 1)])
def test_turb_matches_oracle_reference_size(lt, tab, seed, forced):
    syn, f = case(lt, seed, forced)
    compare(gpu_run(lt, syn, f, tab, lt.PREC_FP64), oracle_run(lt, syn, f))


def test_turb_mixed_domain_rounds_akt_once(lt, tab):
    syn, f = case(lt, 3, 1)
    dom = gpu_run(lt, syn, f, tab, lt.PREC_MIXED)
    o = oracle_run(lt, syn, f)
    g = dom.get("AKT")                    # f32 storage read back as f64
    r = o.get("AKT").astype(np.float32).astype(np.float64)
    np.testing.assert_allclose(g, r, rtol=1.2e-7, atol=0)
    for n in EXACT:
        assert np.array_equal(dom.get(n), o.get(n)), n


def test_turb_then_tracer_step(lt, tab):
    """The closure feeding the tracer step, as readyc_ feeds tracer_: AKT from
    lt_turb, then one FP64 step, against the oracle doing the same."""
    syn, f = case(lt, 21, 1)
    dom = gpu_run(lt, syn, f, tab, lt.PREC_FP64)
    dom.step(1)
    dom.sync()
    o = oracle_run(lt, syn, f)
    o.sum_order(1)
    o.step(1)
    for n in ("AT", "ATB"):
        np.testing.assert_allclose(dom.get(n), o.get(n), rtol=1e-12, atol=1e-15, err_msg=n)


def test_turb_one_degree_tripole(lt, tab):
    syn, f = case(lt, 13, 1, nx=360, ny=218, km=30, dz_top=10.0, dz_bot=250.0)
    compare(gpu_run(lt, syn, f, tab, lt.PREC_FP64), oracle_run(lt, syn, f))


def with_ri(f, rng, rit, rid):
    """The case with Ri and Ri_d replaced at every interface by draws from the
    given values."""
    g = dict(f)
    g["RIT"] = r = rng.choice(rit, size=f["RIT"].shape)
    g["RICDTTMS"] = d = rid(r)
    # not at the critical angles, tan = -1/2 and -2, where the background is a
    # step and an arctangent's last bit decides
    with np.errstate(all="ignore"):
        tan = (r - d) / (r + d)
    d[(np.abs(tan + 0.5) < 1e-6) | (np.abs(tan + 2.0) < 1e-6)] *= 0.9
    return g


def test_turb_ri_beyond_the_squares_range(lt, tab):
    """Ri and Ri_d whose squares underflow or overflow, zeros and denormals
    among them: the background's angle keeps its components' ratio."""
    syn, f = case(lt, 3, 1)
    rng = np.random.default_rng(5)
    tiny = np.array([5e-324, 1e-310, 1e-300, 1e-200, 1e-162, 1e-154, 1e-140, 1e-120, 0.0])
    huge = np.array([1e140, 1e152, 1e155, 1e200, 1e300])
    for values in (tiny, huge, np.concatenate([-tiny, tiny, [0.1, 0.2]]), np.concatenate([-huge, huge, [0.1, 0.2]])):
        g = with_ri(f, rng, values, lambda r: r * rng.choice([-1.2, -1.0, -0.4, 0.0, 0.4, 1.0, 1.2], size=r.shape))
        dom = gpu_run(lt, syn, g, tab, lt.PREC_FP64)
        assert np.isfinite(dom.get("AKT")).all() and np.isfinite(dom.get("AKMT")).all()
        compare(dom, oracle_run(lt, syn, g))


@pytest.mark.parametrize("part", ["linear", "geometric_rid", "geometric_ri", "ends"])
def test_turb_ri_on_table_entries(lt, tab, part):
    """Ri and Ri_d that meet table entries, lie one rounding off them, on both
    sides of the linear part's last entry, at the ends and beyond them.  Where
    an entry of the geometric part is met, the side is left to a logarithm's
    rounding, so the other of the two stays off the entries there (the
    realizable limit is a step)."""
    import turb_synth
    t = tables(lt)
    rib, mt, mt0 = t["rib"], turb_synth.MT, turb_synth.MT0
    syn, f = case(lt, 8, 1)
    rng = np.random.default_rng(9)
    i = np.arange(-mt, mt + 1)
    lin, geo = rib[np.abs(i) < mt0], rib[np.abs(i) > mt0]
    near = np.concatenate([lin, np.nextafter(lin, -np.inf), np.nextafter(lin, np.inf)])
    near = np.concatenate([near, lin[np.abs(lin) < 0.5], lin[np.abs(lin) < 0.5]])   # about the realizable limit
    free = lambda r: rng.uniform(-3.0, 3.0, size=r.shape)
    if part == "linear":
        g = with_ri(f, rng, near, lambda r: rng.choice(near, size=r.shape))
    elif part == "geometric_rid":
        off = rng.uniform(-1.0, 1.0, 4000)
        off = off[np.abs(np.abs(off) - 0.2) > 0.12]          # clear of the realizable limits, 0.1 .. 0.3
        g = with_ri(f, rng, off, lambda r: rng.choice(geo, size=r.shape))
    elif part == "geometric_ri":
        g = with_ri(f, rng, geo, free)
    else:
        ends = [rib[0], rib[-1], np.nextafter(rib[-1], 0.0), np.nextafter(rib[-1], np.inf), 3.0 * rib[-1],
                rib[mt + mt0], np.nextafter(rib[mt + mt0], 0.0), np.nextafter(rib[mt + mt0], np.inf), 0.0, -0.0]
        ends = np.array(ends + [-e for e in ends])
        g = with_ri(f, rng, ends, lambda r: rng.choice(np.concatenate([ends, [0.3, -0.3]]), size=r.shape))
    compare(gpu_run(lt, syn, g, tab, lt.PREC_FP64), oracle_run(lt, syn, g))


def test_turb_ri_nan(lt, tab):
    """Some Ri not a number, beside an Ri_d within the table and beyond either
    end of it: as in the reference, the level takes the largest diffusivity."""
    syn, f = case(lt, 8, 1)
    rng = np.random.default_rng(2)
    g = dict(f)
    g["RIT"] = np.where(rng.random(f["RIT"].shape) < 0.1, np.nan, f["RIT"])
    beyond = 3.0 * tables(lt)["rib"][-1]
    at = np.isnan(g["RIT"])
    g["RICDTTMS"] = np.where(at, rng.choice([beyond, -beyond, 0.3, -2.0], size=at.shape), f["RICDTTMS"])
    compare(gpu_run(lt, syn, g, tab, lt.PREC_FP64), oracle_run(lt, syn, g))


@pytest.mark.parametrize("name,value", [("ssb", 1e-150), ("smb", np.inf), ("slq2b", 1e-101)])
def test_turb_tables_that_are_divided(lt, name, value):
    """A table entry beyond the quick quotient's range (the tables' far corner,
    which no level reaches): every quotient is a division, with the same
    results."""
    t = {k: v.copy() if isinstance(v, np.ndarray) else v for k, v in tables(lt).items()}
    t[name].flat[-1] = value
    syn, f = case(lt, 21, 1)
    odd = lt.TurbTab(t)
    dom = gpu_run(lt, syn, f, odd, lt.PREC_FP64)
    plain = lt.TurbTab(tables(lt))
    same = gpu_run(lt, syn, f, plain, lt.PREC_FP64)
    for n in EXACT + CLOSE:
        assert dom.get(n).tobytes() == same.get(n).tobytes(), n
    compare(dom, oracle_run(lt, syn, f))
    odd.close()
    plain.close()
