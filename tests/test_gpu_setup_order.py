"""What a set-up call hands to the device is there before the next launch, and
what it clears is cleared before the next upload."""
import numpy as np
import pytest

from conftest import load_golden, slab_setup

from beta1_b200 import case, solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 700, 9000])
def test_a_tables_values_reach_the_sync_that_follows(n):
    s = solver.Solver(case.periodic_box_case((24, 23, 21)))
    try:
        inf = s.ctx.field_info("E_xi")
        ext = [h - l for l, h in zip(inf["lo"], inf["hi"])]
        ids = s.ctx.point_base("E_xi", 0) + np.arange(n, dtype=np.int64)
        for q in range(20):
            val = np.arange(n) + 1000.0 * q
            s.ctx.set_sync_consts("other", ids, val)
            s.ctx.sync("other")
            assert np.array_equal(s.field("E_xi").reshape(-1)[:n], val), q
        assert int(np.prod(ext)) > n
    finally:
        s.ctx.close()


def test_an_upload_after_the_resistive_set_up_stays():
    spec, _ = slab_setup(load_golden("slab_6x5x6_t2x2_r11_steps.npz"))
    s = solver.Solver(spec, topology="tiled")
    try:
        rng = np.random.Generator(np.random.PCG64(7))
        for _ in range(5):
            a = {f: rng.standard_normal(s.ctx.download(f).shape) for f in ("Eres_zeta", "dB_xi", "RHS_Bres_zeta")}
            s.install_resistive("tiled")
            for f, x in a.items():
                s.ctx.upload(f, 0, x)
            for f, x in a.items():
                assert np.array_equal(s.ctx.download(f), x), f
            assert s.ctx.resistive_stats() == dict(its=0, rnorm=0.0, bnorm=0.0, reason=0)
    finally:
        s.ctx.close()


def test_a_set_time_counts_for_the_step_that_follows():
    spec = case.periodic_box_case((8, 6, 5))
    st = case.initial_state(spec, seed=2)
    s = solver.Solver(spec)
    try:
        s.load_state(st)
        s.step(1)
        for q in range(20):
            s.ctx.set_time(0.0, 100.0 * q, q)
            dt, t = s.step(1)
            assert t == 100.0 * q + dt and s.ctx.get_time() == (dt, t, q + 1)
    finally:
        s.ctx.close()
