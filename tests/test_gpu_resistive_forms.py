"""Which form the operator of the implicit resistive solve takes, and that
short and long lists give the same bits on ragged blocks and over several
restart cycles (a cycle after the first writes no static point)."""
import numpy as np
import pytest

from beta1_b200 import case, mhd, solver

pytestmark = pytest.mark.gpu

FIELDS = ("U_H", "B_xi", "B_eta", "B_zeta") + tuple(q + x for q in ("Eres_", "dB_", "dJ_") for x in ("xi", "eta", "zeta"))


@pytest.mark.parametrize("restart", [2, 30])
@pytest.mark.parametrize("n,tiles", [((7, 9), (3, 2)), ((16, 15), (1, 1))])
def test_forms(n, tiles, restart, monkeypatch):
    sc = case.ref_scales()
    spec = case.slab_case(41, n, tiles, is_Lunar_resistance=1, use_implicit_lunar_resistance=1,
                          eta_max_lunar=1e-3 * case.MU0 * sc["U"] * sc["L_ref"], implicit_resistive_ksp_rtol=1e-10)
    st = case.inflow_state(spec, seed=20261205)
    keep, res = mhd.Context.set_sync_map, mhd.Context.set_resistive
    monkeypatch.setattr(mhd.Context, "set_resistive", lambda self, *a: res(self, *a[:-1], restart))
    out, forms = [], []
    for form in ("short", "foreign", "chained"):
        def tables(ctx, name, dst, src, form=form):
            dst, src = np.asarray(dst), np.asarray(src)
            if form == "foreign" and name == "dB":  # a copy into a field outside the group's own
                at = np.array([ctx.lib.mhd_point_id(ctx.h, b"divB", 0, 0, 1, 1, 0)])
                dst, src = np.concatenate([dst, at]), np.concatenate([src, src[:1]])
            if form == "chained" and name == "Eres1form":  # a point onto itself
                own = np.setdiff1d(src, dst)[:1]
                dst, src = np.concatenate([dst, own]), np.concatenate([src, own])
            return keep(ctx, name, dst, src)

        monkeypatch.setattr(mhd.Context, "set_sync_map", tables)
        s = solver.Solver(spec, topology="tiled", geometry_on="device")
        try:
            forms.append(s.ctx.resistive_lists())
            s.load_state(st)
            s.step(3)
            stats = s.ctx.resistive_stats()
            assert stats["reason"] in (2, 3) and stats["its"] > 2, stats
            out.append({(f, b): s.field(f, b) for f in FIELDS for b in range(len(spec.blocks))})
        finally:
            s.ctx.close()
    short, foreign, chained = forms
    assert all(0 < dyn < total for total, dyn in short.values()), short
    assert foreign["region"] == (-1, -1), foreign
    assert all(foreign[q][0] == foreign[q][1] > 0 for q in ("Eres", "dB")), foreign
    assert chained["Eres"] == (-1, -1) and chained["region"] == (-1, -1), chained
    for o in out[1:]:
        for k, a in out[0].items():
            assert np.array_equal(a, o[k]), k
