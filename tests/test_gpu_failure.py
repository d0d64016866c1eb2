"""Failure detection on the device without a fault.

The TMA-fed column kernels bound every wait for their level data.  Setting
the bound to zero polls makes every wait give up at once: each CTA records
the timeout, drains the boxes it already issued and returns.  The host must
see LT_E_TIMEOUT at the next synchronising call, and the context must stay
usable: a fresh domain then steps exactly like an untouched twin.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_wait_timeout_is_reported_and_context_survives(lt, precision):
    prec = lt.PREC_MIXED if precision == "mixed" else lt.PREC_FP64
    syn = lt.Synth(64, 40, 20)
    bad = syn.domain(precision=prec)
    bad.set_wait_limit(0)
    bad.step(1)
    with pytest.raises(lt.LtError) as err:
        bad.sync()
    assert err.value.code == lt.LT_E_TIMEOUT
    # reported once: the next synchronising call is clean
    bad.sync()

    a = syn.domain(precision=prec)
    b = syn.domain(precision=prec)
    a.step(2)
    b.step(2)
    a.sync()
    b.sync()
    np.testing.assert_array_equal(a.get("AT"), b.get("AT"))
    assert a.check_numeric() == 0

    # the domain that timed out steps normally again once the bound is restored
    bad.set_wait_limit(1 << 24)
    bad.step(1)
    bad.sync()


def test_wait_timeout_in_the_continuity_march(lt):
    """The same on a grid whose mixed continuity is the march fed by boxes (74
    tiles and more; smaller grids form it level by level, without a wait)."""
    syn = lt.Synth(260, 90, 8)
    bad = syn.domain(precision=lt.PREC_MIXED)
    bad.set_wait_limit(0)
    bad.step(1)
    with pytest.raises(lt.LtError) as err:
        bad.sync()
    assert err.value.code == lt.LT_E_TIMEOUT
    bad.sync()
    twins = [syn.domain(precision=lt.PREC_MIXED) for _ in range(2)]
    for d in twins:
        d.step(2)
        d.sync()
    assert twins[0].get("AT").tobytes() == twins[1].get("AT").tobytes()
    assert twins[0].check_numeric() == 0


def test_wait_timeout_in_a_batch(lt):
    """Members whose waits run out in the batch's continuity and column kernel:
    reported at the batch's synchronisation, once; the batch steps on when the
    bound is restored."""
    sizes = [(64, 40, 20), (96, 48, 12)]
    doms = [lt.Synth(*s).domain(precision=lt.PREC_MIXED) for s in sizes]
    for d in doms:
        d.set_wait_limit(0)
    b = lt.Batch(doms)
    b.step(1)
    with pytest.raises(lt.LtError) as err:
        b.sync()
    assert err.value.code == lt.LT_E_TIMEOUT
    b.sync()
    for d in doms:
        d.set_wait_limit(1 << 24)
    b.set_config()   # takes the members' parameters
    b.step(1)
    b.sync()
    b.close()
