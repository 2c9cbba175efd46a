"""Errors inside a span of several steps.  dt falls from 7.3e-3 to 4.2e-3 in
the fixture's second step; with an abort threshold between them the second step
reports EDT.  A solve that gave up in the first step (the failure-detection
hook: a barrier arrival that never comes, each wait bounded) is reported before
it, and its mark and its barrier count reach no later solve: the next step from
a good state matches the reference."""
import pytest

from conftest import load_golden, rel_l2, slab_setup

from beta1_b200 import mhd, solver

pytestmark = pytest.mark.gpu

STATE = ["U_H", "B_xi", "B_eta", "B_zeta"]


@pytest.mark.parametrize("stalled,error", [(True, "EKRYLOV"), (False, "EDT")])
@pytest.mark.parametrize("steps", [2, 4])
def test_span_with_a_small_dt_after_a_solve(stalled, error, steps, monkeypatch):
    keep = solver.make_params

    def params(*a, **k):
        p = keep(*a, **k)
        p.dt_abort = 6e-3
        return p

    monkeypatch.setattr(solver, "make_params", params)
    g = load_golden("slab_6x5x6_t2x2_r11_steps.npz")
    assert float(g["s2/dt"]) < 6e-3 < float(g["s1/dt"])
    spec, st = slab_setup(g)
    s = solver.Solver(spec, topology="tiled")
    try:
        for _ in range(2):  # an error leaves nothing behind for the next one either
            s.ctx.set_time(0.0, 0.0, 0)
            s.load_state(st)
            if stalled:
                s.ctx.test_stall_barrier(4096)
            with pytest.raises(mhd.MHDError, match=error):
                s.step(steps)
            s.ctx.set_time(0.0, 0.0, 0)
            s.load_state(st)
            dt, _ = s.step(1)
            assert abs(dt - float(g["s1/dt"])) <= 1e-10 * float(g["s1/dt"])
            for b in range(len(spec.blocks)):
                for f in STATE:
                    assert rel_l2(s.field(f, b), g["s1/b%d/%s" % (b, f)]) <= 1e-10, (b, f)
            assert s.ctx.resistive_stats()["reason"] in (2, 3)
    finally:
        s.ctx.close()
