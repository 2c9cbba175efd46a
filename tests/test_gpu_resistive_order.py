"""The persistent resistive solve over many CTAs, repeated: every element a
product reads from another CTA is complete, so the same state gives the same
bits each time, in the short lists and with the copies as lists of their own."""
import numpy as np
import pytest

from beta1_b200 import case, mhd, solver

pytestmark = pytest.mark.gpu

FIELDS = ("U_H", "B_xi", "B_eta", "B_zeta", "Eres_xi", "Eres_eta", "Eres_zeta", "dB_xi", "dB_eta", "dB_zeta")


@pytest.mark.parametrize("chained", [False, True])
def test_repeated_solves_give_the_same_bits(chained, monkeypatch):
    sc = case.ref_scales()
    spec = case.slab_case(40, (24, 22), (2, 2), is_Lunar_resistance=1, use_implicit_lunar_resistance=1,
                          eta_max_lunar=1e-3 * case.MU0 * sc["U"] * sc["L_ref"], implicit_resistive_ksp_rtol=1e-12)
    st = case.inflow_state(spec, seed=20261205)
    keep = mhd.Context.set_sync_map

    def record(ctx, name, dst, src):
        if chained and name == "Eres1form":  # a point onto itself: the copies run as lists of their own
            own = np.setdiff1d(src, dst)[:1]
            dst, src = np.concatenate([dst, own]), np.concatenate([src, own])
        return keep(ctx, name, dst, src)

    monkeypatch.setattr(mhd.Context, "set_sync_map", record)
    s = solver.Solver(spec, topology="tiled", geometry_on="device")
    try:
        first = None
        for _ in range(12):
            s.ctx.set_time(0.0, 0.0, 0)
            s.load_state(st)
            s.step(2)
            stats = s.ctx.resistive_stats()
            assert stats["reason"] in (2, 3) and stats["its"] > 3, stats
            out = {(f, b): s.field(f, b) for f in FIELDS for b in range(len(spec.blocks))}
            first = first or out
            for k, a in out.items():
                assert np.array_equal(a, first[k]), k
        assert len(s.resistive_dofs[0]) > 4 * 256  # several CTAs
    finally:
        s.ctx.close()
