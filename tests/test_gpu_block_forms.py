"""Forms that only many blocks, or many boxes, take: a single run of more
blocks than one launch holds, the implicit resistive solve with more blocks
than it keeps in shared memory, a block with more zeroed Hall boxes than fit
there.  Each gives the bits of the form the reference's fixtures cover."""
import numpy as np
import pytest

from conftest import load_golden, slab_setup

from beta1_b200 import case, mhd, solver

pytestmark = pytest.mark.gpu

FIELDS = ("U_H", "B_xi", "B_eta", "B_zeta", "PV_H", "B_cell", "J_cell", "E_xi", "Eface_eta", "RHS_H", "RHS_B_zeta")


@pytest.mark.parametrize("integrator", [mhd.INTEGRATOR_EULER, mhd.INTEGRATOR_SSPRK2])
@pytest.mark.parametrize("precision", [mhd.PREC_FP64, mhd.PREC_MIXED])
def test_run_of_72_blocks(integrator, precision):
    """alone (a grid row per block, two launches per kernel) and beside another
    run (flattened launches, whose split over launches the batches of copies of
    the reference's fixture cover)"""
    spec = case.slab_case(9, (4, 5), (9, 8))
    other = case.slab_case(7, (4, 33), (1, 1))
    st, st2 = case.inflow_state(spec, seed=3), case.inflow_state(other, seed=4)
    s = solver.Solver(spec, topology="tiled", precision=precision, geometry_on="device")
    bt = solver.Batch([(other, "tiled"), (spec, "tiled")], precision=precision, geometry_on="device")
    try:
        for c in (s.ctx, bt.ctx):
            c.set_integrator(integrator)
        s.load_state(st)
        bt.load_states([st2, st])
        dt, _ = s.step(2)
        bt.step(2)
        assert bt.ctx.run_time(1)[0] == dt
        for b in (0, 1, 62, 63, 64, 65, 71):
            for f in FIELDS:
                assert np.array_equal(bt.field(1, f, b), s.field(f, b)), (b, f)
    finally:
        s.ctx.close()
        bt.ctx.close()


@pytest.mark.parametrize("extra", [20, 21, 66])
def test_resistive_solve_beside_unused_blocks(extra, monkeypatch):
    """blocks without geometry, tables or unknowns beside the fixture's four:
    24 in all fit in shared memory, 25 and more are read from global memory, 70
    take two launches per kernel"""
    spec, st = slab_setup(load_golden("slab_6x5x6_t2x2_r11_steps.npz"))
    keep = mhd.Context.__init__
    out = []
    for more in (0, extra):
        monkeypatch.setattr(mhd.Context, "__init__",
                            lambda self, n, *a, **k: keep(self, list(n) + [(2, 2, 2)] * more, *a, **k))
        s = solver.Solver(spec, topology="tiled")
        try:
            assert len(s.ctx.ncells) == len(spec.blocks) + more
            s.load_state(st)
            s.step(2)
            assert s.ctx.resistive_stats()["reason"] in (2, 3)
            out.append({(f, b): s.field(f, b) for f in FIELDS + ("Eres_xi", "Eres_eta", "Eres_zeta")
                        for b in range(len(spec.blocks))})
        finally:
            s.ctx.close()
    for k, a in out[0].items():
        assert np.array_equal(a, out[1][k]), k


@pytest.mark.parametrize("copies", [2, 9])
def test_many_zeroed_hall_boxes(copies, monkeypatch):
    """every box of the Solid_Surface given several times (3 per block: 6 fit in
    shared memory, 27 do not), among boxes that hold no edge"""
    spec = case.slab_case(24, (5, 6), (2, 2))
    st = case.inflow_state(spec, seed=20261205)
    keep = mhd.Context.set_hall
    out = []
    for n in (1, copies):
        monkeypatch.setattr(mhd.Context, "set_hall", lambda self, c, rows: keep(
            self, c, np.concatenate([np.asarray(rows, dtype=np.int32).reshape(-1, 8)] * n +
                                    [np.array([[b, 1, 3, 3, 3, 3, 3, 3] for b in range(4)], dtype=np.int32)])))
        s = solver.Solver(spec, topology="tiled")
        try:
            s.load_state(st)
            s.install_hall_implicit("tiled", rtol=1e-10, maxit=20, ksp_rtol=1e-6, ksp_maxit=200)
            s.step(2)
            out.append({(f, b): s.field(f, b) for f in ("U_H", "B_xi", "B_zeta", "Ehall_xi", "Ehall_eta", "Ehall_zeta")
                        for b in range(len(spec.blocks))})
        finally:
            s.ctx.close()
    assert np.any(out[0][("Ehall_eta", 0)] != 0.0)
    for k, a in out[0].items():
        assert np.array_equal(a, out[1][k]), k
