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


def test_fixed_values_that_another_group_overwrites(monkeypatch):
    """a fixed value of Sync("dB") next to an unknown's edge, and a copy of
    Sync("Eres1form") onto the same point: every product writes the fixed value
    after the copy, so the copy changes nothing (but the point itself at the end:
    the solution's own Sync("Eres1form"), after the last product, writes it)"""
    sc = case.ref_scales()
    spec = case.slab_case(16, (7, 6), (2, 2), is_Lunar_resistance=1, use_implicit_lunar_resistance=1,
                          eta_max_lunar=1e-3 * case.MU0 * sc["U"] * sc["L_ref"], implicit_resistive_ksp_rtol=1e-12)
    st = case.inflow_state(spec, seed=20261205)
    maps = {}
    keep = mhd.Context.set_sync_map

    def record(ctx, name, dst, src):
        maps[name] = (np.asarray(dst), np.asarray(src))
        return keep(ctx, name, dst, src)

    monkeypatch.setattr(mhd.Context, "set_sync_map", record)
    out = []
    for extra in (False, True):
        s = solver.Solver(spec, topology="tiled", geometry_on="device")
        try:
            # an unknown zeta edge on the block's face j = n_j reads dB_xi one layer past it
            b, _, i, j, k = next(r for r in s.resistive_dofs[0].tolist() if r[1] == 3 and r[3] == 7)
            at = s.ctx.lib.mhd_point_id(s.ctx.h, b"dB_xi", b, i, j, k, 0)
            edge = s.ctx.lib.mhd_point_id(s.ctx.h, b"Eres_zeta", b, i, j, k, 0)
            dst, src = maps["dB"]
            assert at in dst and at not in src
            keep(s.ctx, "dB", dst[dst != at], src[dst != at])
            s.ctx.set_sync_consts("dB", np.array([at]), np.array([1e-6]))
            if extra:
                dst, src = maps["Eres1form"]
                keep(s.ctx, "Eres1form", np.concatenate([dst, [at]]), np.concatenate([src, [edge]]))
            s.load_state(st)
            s.step(2)
            assert s.ctx.resistive_stats()["its"] > 2
            out.append({(f, q): s.field(f, q) for f in FIELDS for q in range(len(spec.blocks))})
            out[-1][("dB_xi", b)][4 + i, 4 + j, 4 + k] = 0.0
        finally:
            s.ctx.close()
    for key, a in out[0].items():
        assert np.array_equal(a, out[1][key]), key
