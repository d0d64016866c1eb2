"""The phases that lt_phase_ms reports hold the launches they are named for."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("diagnostics", [False, True])
def test_surface_phase_holds_the_surface_kernel(lt, diagnostics):
    """A wide, flat grid, whose surface kernel moves 130 bytes of each of three
    million columns: at 8 TB/s no less than 49 us of a step, far above what two
    adjacent events are apart.  The phases together are the step."""
    nx, ny, steps = 2000, 1500, 4
    syn = lt.Synth(nx, ny, 3, seed=1, forced=1)
    dom = syn.domain(precision=lt.PREC_FP64, diagnostics=diagnostics)
    dom.step(2)
    dom.sync()
    dom.profile(True)
    dom.step(steps)
    dom.sync()
    n, ph = dom.phase_ms()
    dom.profile(False)
    assert n == steps
    assert ph["surface"] / n > 0.04, ph
    if diagnostics:   # two levels' ghost cells in a launch of their own
        assert ph["net_halo"] > 0.0
    assert abs(sum(ph.values()) - dom.last_step_ms()) < 0.1 * dom.last_step_ms()


def test_host_steps_book_the_wait_with_the_surface(lt):
    """Steps with and without forcing copies in one profile: each under its own
    launch order, the continuity (here most of the step's bytes beside the
    columns) at a like time in both."""
    syn = lt.Synth(720, 460, 30, seed=1, forced=1)
    dom = syn.domain(precision=lt.PREC_FP64)
    host = {k: syn.field(k) for k in ("SWV", "NSWV", "SST", "SSS", "FRESH", "SEAICE")}

    def phases(step):
        step()
        dom.sync()
        dom.profile(True)
        for _ in range(3):
            step()
        dom.sync()
        n, ph = dom.phase_ms()
        dom.profile(False)
        return {k: v / n for k, v in ph.items()}

    plain, hosted = phases(lambda: dom.step(1)), phases(lambda: dom.step_host(host))
    for name in ("continuity", "tracer"):
        assert 0.5 * plain[name] < hosted[name] < 2.0 * plain[name], (name, plain, hosted)
