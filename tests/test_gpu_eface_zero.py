"""The components of Eface that the face kernel leaves alone (component a of
the faces of axis a) are zero after a step whatever wrote them before it: a
table that has been replaced, another group's Sync, or the step's own table in
the step before."""
import numpy as np
import pytest

from conftest import load_golden, periodic_setup

from beta1_b200 import case, solver

pytestmark = pytest.mark.gpu

EF = ("Eface_xi", "Eface_eta", "Eface_zeta")
AT = (3, 2, 2)


def _solver():
    g = load_golden("periodic_8x6x5_steps.npz")
    spec, st = periodic_setup(g)
    s = solver.Solver(spec)
    s.load_state(st)
    ids = {f: [s.ctx.lib.mhd_point_id(s.ctx.h, f.encode(), 0, *AT, m) for m in range(3)] for f in EF}
    ids["U_H"] = [s.ctx.lib.mhd_point_id(s.ctx.h, b"U_H", 0, *AT, 0)]
    return g, s, ids


def _check(s, g):
    """the reference's Eface of the first step on every inner face"""
    n = s.spec.blocks[0].ncell
    for d, f in enumerate(EF):
        inner = tuple(slice(4, 4 + n[a] + (a == d)) for a in range(3))
        assert np.array_equal(s.field(f)[inner], g["s1/" + f][inner]), f


def _i64(*v):
    return np.array(v, dtype=np.int64)


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_a_replaced_table_leaves_nothing(axis):
    g, s, ids = _solver()
    try:
        st = periodic_setup(g)[1]
        s.ctx.set_sync_consts("Eface", _i64(ids[EF[axis]][axis]), np.array([3.0]))
        s.step(1)
        assert s.field(EF[axis])[tuple(4 + x for x in AT)][axis] == 3.0
        s.ctx.set_sync_consts("Eface", _i64(), np.array([]))
        s.ctx.set_time(0.0, 0.0, 0)
        s.load_state(st)
        s.step(1)
        _check(s, g)
    finally:
        s.ctx.close()


def test_another_groups_sync_leaves_nothing():
    g, s, ids = _solver()
    try:
        s.ctx.set_sync_map("other", _i64(ids[EF[1]][1]), _i64(ids["U_H"][0]))
        s.ctx.sync("other")
        at = tuple(4 + x for x in AT)
        assert s.field(EF[1])[at][1] == s.field("U_H")[at][0]
        s.step(1)
        _check(s, g)
    finally:
        s.ctx.close()


def test_a_table_reads_the_zero_of_its_own_step():
    """a <- b and b <- c in one table, b a zero component: every step a takes
    b's zero, not what the step before left in b"""
    g, s, ids = _solver()
    try:
        maps = [ids["Eface_zeta"][2], ids["Eface_xi"][0], ids["Eface_eta"][0]]  # a, b, c
        s.ctx.set_sync_map("Eface", _i64(maps[0], maps[1]), _i64(maps[1], maps[2]))
        at = tuple(4 + x for x in AT)
        for _ in range(2):
            s.step(2)
            assert s.field("Eface_zeta")[at][2] == 0.0
            assert s.field("Eface_xi")[at][0] == s.field("Eface_eta")[at][0] != 0.0
    finally:
        s.ctx.close()


@pytest.mark.parametrize("kind", ["box", "slab", "shell"])
def test_the_grid_families_need_no_extra_pass(kind):
    spec, topo, state = {
        "box": (case.periodic_box_case((8, 6, 5)), "periodic", case.initial_state),
        "slab": (case.slab_case(12, (7, 6), (2, 2)), "tiled", case.inflow_state),
        "shell": (case.shell_case(12, 8, 10), "shell", case.inflow_state)}[kind]
    s = solver.Solver(spec, topology=topo)
    try:
        s.load_state(state(spec, seed=1))
        assert [k for k, _ in s.ctx.profile_step()].count("k_eface") == 1
    finally:
        s.ctx.close()
