"""The hot kernels' launch forms: batches past the blocks of one launch (65
runs and more: two launches per kernel), grids past the small argument form
(9 blocks and more), a batch of several runs against each run alone, the
components of Eface the face kernel leaves alone, the resistive operator's
lists, the weights' order in memory and restarts of the Hall solve.  Every form
but the last runs the same arithmetic per point, so the fields agree bit for
bit."""
import numpy as np
import pytest

from conftest import load_golden, periodic_setup, rel_l2, slab_setup

from beta1_b200 import case, mhd, solver

pytestmark = pytest.mark.gpu

FIELDS = ("U_H", "B_xi", "B_eta", "B_zeta", "PV_H", "J_cell", "E_xi", "Eface_eta", "RHS_H", "RHS_B_zeta")


@pytest.mark.parametrize("nruns", [2, 9, 64, 65, 70])
def test_batch_sizes(nruns):
    """copies of the periodic fixture, one run each: the reference's step"""
    g = load_golden("periodic_8x6x5_steps.npz")
    spec, st = periodic_setup(g)
    host = solver.host_setup(spec, "periodic", "device")
    bt = solver.Batch([(spec, "periodic")] * nruns, host=iter([host] * nruns))
    try:
        bt.load_states([st] * nruns)
        bt.step(1)
        for r in sorted({0, 1, nruns // 2, nruns - 1}):
            for f in FIELDS:
                assert np.array_equal(bt.field(r, f), g["s1/" + f]), (r, f)
    finally:
        bt.ctx.close()


def test_twelve_blocks_alone_and_in_a_batch():
    """a 12-block slab (one launch of the large argument form) and the same
    run beside another of other extents in a batch (flattened launches)"""
    spec = case.slab_case(11, (5, 7), (3, 4))
    other = case.slab_case(9, (4, 33), (1, 2))
    st, st2 = case.inflow_state(spec, seed=3), case.inflow_state(other, seed=4)
    s = solver.Solver(spec, topology="tiled", geometry_on="device")
    bt = solver.Batch([(other, "tiled"), (spec, "tiled")], geometry_on="device")
    try:
        s.load_state(st)
        bt.load_states([st2, st])
        s.step(3)
        bt.step(3)
        for b in range(12):
            for f in FIELDS:
                assert np.array_equal(bt.field(1, f, b), s.field(f, b)), (b, f)
    finally:
        s.ctx.close()
        bt.ctx.close()


def test_uploaded_eface():
    """the zero components of an uploaded Eface are zero after a step"""
    g = load_golden("periodic_8x6x5_steps.npz")
    spec, st = periodic_setup(g)
    s = solver.Solver(spec)
    try:
        s.load_state(st)
        for f in ("Eface_xi", "Eface_eta", "Eface_zeta"):
            s.ctx.upload(f, 0, np.full_like(s.field(f), 3.0))
            assert np.all(s.field(f) == 3.0)
        s.step(1)
        n = spec.blocks[0].ncell
        for d, f in enumerate(("Eface_xi", "Eface_eta", "Eface_zeta")):
            inner = tuple(slice(4, 4 + n[a] + (a == d)) for a in range(3))
            assert np.array_equal(s.field(f)[inner], g["s1/" + f][inner]), f
    finally:
        s.ctx.close()


@pytest.mark.parametrize("group", ["dB", "Eres1form"])
def test_resistive_operator_forms(group, monkeypatch):
    """one more copy, without effect on the compared fields, takes the implicit
    solve off its short lists: into divB (a field outside the group's own, so
    every product writes every point), or of a point onto itself (a chain, so
    the copies run as lists of their own).  It is given after the solve is set
    up, which rebuilds the operator.  Same operations per point: the same bits."""
    g = load_golden("slab_6x5x6_t2x2_r11_steps.npz")
    spec, st = slab_setup(g)
    maps, out = {}, []
    keep = mhd.Context.set_sync_map

    def record(ctx, name, dst, src):
        maps[name] = (np.asarray(dst), np.asarray(src))
        return keep(ctx, name, dst, src)

    monkeypatch.setattr(mhd.Context, "set_sync_map", record)
    for extra in (False, True):
        s = solver.Solver(spec, topology="tiled")
        try:
            if extra:
                dst, src = maps[group]
                i, j = np.setdiff1d(src, dst)[:1], np.setdiff1d(src, dst)[:1]
                if group == "dB":
                    i = np.array([s.ctx.lib.mhd_point_id(s.ctx.h, b"divB", int(src[0]) >> 40 & 0xFFFF, 0, 1, 1, 0)])
                    j = src[:1]
                keep(s.ctx, group, np.concatenate([dst, i]).astype(dst.dtype),
                     np.concatenate([src, j]).astype(src.dtype))
            s.load_state(st)
            s.step(3)
            out.append({(f, b): s.field(f, b) for f in FIELDS + tuple(
                q + x for q in ("Eres_", "dB_", "dJ_") for x in ("xi", "eta", "zeta"))
                        for b in range(len(spec.blocks))})
        finally:
            s.ctx.close()
    for k, a in out[0].items():
        assert np.array_equal(a, out[1][k]), k


@pytest.mark.parametrize("n", [(3, 4, 5), (2, 5, 33)])
def test_weights_keep_their_points(n):
    """the least-squares weights, stored in tiles of inner cells: every value
    of an uploaded field, ghosts included, comes back from its own point"""
    s = solver.Solver(case.periodic_box_case(n))
    try:
        for f in ("Bcell_from_Bface_w", "Jcell_from_Jedge_w"):
            a = np.random.Generator(np.random.PCG64(5)).standard_normal(s.field(f).shape)
            s.ctx.upload(f, 0, a)
            assert np.array_equal(s.field(f), a), f
    finally:
        s.ctx.close()


def test_hall_restart_cycles():
    """linear solves held past a restart (30 basis vectors) by an unreachable
    tolerance take the norms of dx and r that a first cycle leaves out: the
    Newton steps reach the root that unrestarted solves reach.  Both stop at
    1e-12 of the first residual, as the comparison with the reference's solve,
    whose bound is 1e-10 relative L2."""
    spec = case.slab_case(24, (5, 6), (2, 2))
    st = case.inflow_state(spec, seed=20261205)
    out, stats = [], []
    for ksp in (dict(ksp_rtol=1e-10, ksp_maxit=2000), dict(ksp_rtol=1e-300, ksp_maxit=65)):
        s = solver.Solver(spec, topology="tiled")
        try:
            s.load_state(st)
            s.install_hall_implicit("tiled", rtol=1e-12, atol=1e-30, maxit=200, **ksp)
            s.step(1)
            stats.append(s.ctx.hall_stats())
            out.append({(f, b): s.field(f, b) for f in ("Ehall_xi", "Ehall_eta", "B_xi", "B_zeta", "U_H")
                        for b in range(len(spec.blocks))})
        finally:
            s.ctx.close()
    assert stats[1]["reason"] in (2, 3) and stats[1]["linear_its"] > 30 * stats[1]["its"], stats
    for k, a in out[0].items():
        assert rel_l2(out[1][k], a) <= 1e-10, (k, stats)
