"""Convective adjustment, the SSS-norm sum and the batch's continuity at the
sizes where their loops can go wrong."""
import numpy as np
import pytest

import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,km", [(8, 8, 3), (33, 12, 5), (31, 29, 8), (40, 24, 55), (16, 16, 128)])
def test_convadj_bitexact(lt, nx, ny, km):
    """Columns from stable to overturned from top to bottom, one to km levels
    deep, with a previous state and a tendency to add to: bit for bit."""
    syn = lt.Synth(nx, ny, km, seed=5 + km, hypsometry=1, tripole=0, ew_cyclic=0, cap_north=2, cap_south=2)
    f = syn.all_fields()
    rng = np.random.default_rng(km)
    at = f["AT"].copy()
    jmt, imt = at.shape[2:]
    kind = rng.integers(0, 4, size=(jmt, imt))
    noise = rng.normal(0.0, 1.0, size=at.shape)
    at[0] += np.where(kind == 1, 0.5, np.where(kind == 2, 6.0, 0.0)) * noise[0]
    at[1] += 1e-3 * np.where(kind == 2, 1.0, 0.1) * noise[1]
    cold = np.linspace(-2.0, 20.0, km)[:, None, None]
    at[0] = np.where(kind == 3, cold, at[0])          # overturned columns
    f["AT"] = at
    f["KMT"] = np.where(f["KMT"] > 0, rng.integers(1, km + 1, size=f["KMT"].shape), 0).astype(np.int32)
    dom = lt.TracerDomain(nx, ny, km, syn.params, ew_cyclic=False, tripole=False)
    o = pyoracle.Oracle(nx, ny, km, syn.params, ew_cyclic=0, tripole=0)
    o.load(f)
    for n in lt.INPUT_FIELDS:
        dom.set(n, f[n])
    for _ in range(2):
        dom.convadj()
        o.convadj()
    dom.sync()
    assert (dom.get("AT") != at).any()
    for n in ("AT", "ATB", "DT_CONV", "TEND"):
        g, r = dom.get(n), o.get(n)
        assert g.tobytes() == r.tobytes(), (n, int((g != r).sum()))


def tree_sum(x):
    """The fixed tree: blocks of 2048 terms, halves added, until one is left."""
    x = np.asarray(x, dtype=np.float64)
    while True:
        nb = max(1, -(-len(x) // 2048))
        s = np.zeros(nb * 2048)
        s[:len(x)] = x
        s = s.reshape(nb, 2048)
        h = 1024
        while h:
            s = s[:, :h] + s[:, h:2 * h]
            h //= 2
        x = s[:, 0]
        if nb == 1:
            return x[0]


@pytest.mark.parametrize("nx,ny", [(32, 64), (33, 63), (2100, 2001)])
def test_sss_norm_tree(lt, nx, ny):
    """fw_norm2 is the fixed tree's sum over one block, two blocks and enough
    blocks for a third level, twice in a row (the finishing block clears its
    counter)."""
    syn = lt.Synth(nx, ny, 3, seed=2, forced=1, tripole=0, ew_cyclic=0, cap_north=2, cap_south=2)
    dom = syn.domain(precision=lt.PREC_FP64)
    for _ in range(2):
        dom.step(1)
        dom.sync()
        net, tarea, kmt = dom.get("NET")[1], dom.get("TAREA"), dom.get("KMT")
        terms = (tarea * net * (kmt > 0))[2:-2, 2:-2].reshape(-1)
        assert dom.fw_norm2() == -tree_sum(terms) / syn.params.area_t


@pytest.mark.parametrize("tile_y", [4, 8])
def test_batch_continuity_aligned_and_not(lt, tile_y):
    """Members with and without TMA row pitches in one batch: the vertical
    velocity and state of each equal those of the member stepped alone."""
    sizes = [(64, 40, 20), (61, 33, 9), (130, 66, 30)]
    kw = dict(tripole=0, ew_cyclic=0, cap_north=2, cap_south=2, forced=1, hypsometry=1)
    alone = [lt.Synth(*s, seed=k, **kw).domain(precision=lt.PREC_MIXED) for k, s in enumerate(sizes)]
    both = [lt.Synth(*s, seed=k, **kw).domain(precision=lt.PREC_MIXED) for k, s in enumerate(sizes)]
    b = lt.Batch(both)
    b.set_config(column_ctas_per_sm=2, continuity_tile_y=tile_y, use_graph=0)
    b.step(3)
    b.sync()
    for x, y in zip(alone, both):
        x.step(3)
        x.sync()
        for n in ("WS", "AT", "UTF_OUT"):
            assert x.get(n).tobytes() == y.get(n).tobytes(), n


def test_batch_of_more_rows_than_a_grid_dimension(lt):
    """262204 rows are more blocks of four than a launch's y dimension takes:
    the batch's continuity takes taller tiles there, with the same results."""
    kw = dict(tripole=0, ew_cyclic=0, cap_north=2, cap_south=2, forced=1, hypsometry=1)
    got = []
    for tile_y in (4, 16):
        dom = lt.Synth(8, 262200, 3, seed=4, **kw).domain(precision=lt.PREC_MIXED)
        b = lt.Batch([dom])
        b.set_config(continuity_tile_y=tile_y)
        b.step(1)
        b.sync()
        got.append([dom.get(n).tobytes() for n in ("WS", "AT")])
        b.close()
        dom.close()
    assert got[0] == got[1]
