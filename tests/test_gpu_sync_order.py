"""Sync tables that reach fields of other groups run in the reference's order:
Sync("Ucell") goes beside the B_cell pass only where its table keeps to U_H.
With a copy of face B values in the table of "Ucell", or of U_H in that of
"Bface", the step's graph gives what the same step gives launch by launch on
one stream (profile_step), bit for bit."""
import numpy as np
import pytest

from beta1_b200 import case, mhd, solver

pytestmark = pytest.mark.gpu

FIELDS = ("U_H", "B_xi", "B_eta", "B_zeta", "B_cell", "Bind_cell", "J_xi", "J_eta", "J_zeta", "J_cell", "PV_H")


@pytest.mark.parametrize("grid", ["slab", "shell"])
@pytest.mark.parametrize("group", [None, "Ucell", "Bface"])
def test_tables_that_reach_other_fields(grid, group, monkeypatch):
    if grid == "slab":
        spec, topo = case.slab_case(40, (17, 16), (2, 1)), "tiled"
    else:
        spec, topo = case.shell_case(40, 16, 18), "shell"
    st = case.inflow_state(spec, seed=20261205)
    keep = mhd.Context.set_sync_map

    def extra(ctx, name, dst, src):
        if name == group:
            # a layer of values of the other field, from the layer above it
            f, m = ("B_xi", 0) if group == "Ucell" else ("U_H", 1)
            pid = [[ctx.lib.mhd_point_id(ctx.h, f.encode(), 0, i, j, k, m) for j in range(2, 14) for k in range(2, 14)]
                   for i in (7, 8)]
            dst = np.concatenate([dst, np.array(pid[0], dst.dtype)])
            src = np.concatenate([src, np.array(pid[1], src.dtype)])
        return keep(ctx, name, dst, src)

    monkeypatch.setattr(mhd.Context, "set_sync_map", extra)
    out = []
    for eager in (False, True):
        s = solver.Solver(spec, topology=topo, geometry_on="device")
        try:
            s.load_state(st)
            for _ in range(3):
                s.ctx.profile_step() if eager else s.step(1)
            out.append({(f, b): s.field(f, b) for f in FIELDS for b in range(len(spec.blocks))})
        finally:
            s.ctx.close()
    for k, a in out[0].items():
        assert np.array_equal(a, out[1][k]), k
    if group == "Ucell":
        g = 4
        a = out[0][("B_xi", 0)][g:, g:, g:, 0]
        assert np.array_equal(a[7, 2:14, 2:14], a[8, 2:14, 2:14])
