"""Tables that copy the temperature of PV_H (its fifth component, which a step
leaves to read-out): through mhd_sync after steps, and in a Sync of the step
itself, the copy takes the present state's temperature."""
import numpy as np
import pytest

from beta1_b200 import case, mhd, solver

pytestmark = pytest.mark.gpu

SPOTS = [(2, 3, 1), (5, 0, 4), (7, 5, 2)]


def _ids(s, name, m):
    return np.array([s.ctx.lib.mhd_point_id(s.ctx.h, name.encode(), 0, *p, m) for p in SPOTS], dtype=np.int64)


def _at(a, m):
    return np.array([a[tuple(4 + x for x in p)][m] for p in SPOTS])


@pytest.mark.parametrize("precision", [mhd.PREC_FP64, mhd.PREC_MIXED])
@pytest.mark.parametrize("group", ["other", "Uplus"])
def test_copies_of_the_temperature(precision, group):
    spec = case.periodic_box_case((8, 6, 5))
    st = case.initial_state(spec, seed=11)
    keep = {}
    set_map = mhd.Context.set_sync_map

    def record(ctx, name, dst, src):
        keep[name] = (np.asarray(dst), np.asarray(src))
        return set_map(ctx, name, dst, src)

    mhd.Context.set_sync_map = record
    try:
        s = solver.Solver(spec, precision=precision)
    finally:
        mhd.Context.set_sync_map = set_map
    try:
        s.load_state(st)
        dst, src = keep.get(group, (np.zeros(0, np.int64), np.zeros(0, np.int64)))
        # into the ghost-free diagnostic field, whose values nothing else writes
        s.ctx.set_sync_map(group, np.concatenate([dst, _ids(s, "divB", 0)]), np.concatenate([src, _ids(s, "PV_H", 4)]))
        for steps in (0, 3, 2):  # the derived fields of a new state, then steps
            if steps:
                s.step(steps)
            else:
                s.ctx.update_derived()
            if group == "other":
                s.ctx.sync(group)
            inf = s.ctx.field_info("divB")
            div = s.ctx.download("divB")
            got = np.array([div[tuple(x - l for x, l in zip(p, inf["lo"]))][0] for p in SPOTS])
            T = _at(s.field("PV_H"), 4)
            assert np.all(T > 0.0) and np.array_equal(got, T), (steps, got, T)
    finally:
        s.ctx.close()


def test_no_extra_pass_without_such_a_table():
    s = solver.Solver(case.periodic_box_case((8, 6, 5)))
    try:
        s.load_state(case.initial_state(s.spec, seed=11))
        assert [k for k, _ in s.ctx.profile_step()].count("k_pv_uplus_dt") == 1
    finally:
        s.ctx.close()
