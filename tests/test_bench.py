"""What bench.py reports of the library's launches: the profile's scopes."""
import os
import sys

import pytest

from conftest import ROOT

sys.path.insert(0, ROOT)
import bench  # noqa: E402


@pytest.mark.gpu
def test_dominant_kernel_of_a_real_profile():
    """On the headline's grid the predictor takes longest of the kernels of a
    step that does not reinitialise, so its scope has to hold that kernel
    alone; the kernel that prepares its near rows and the one that begins the
    band sweeps have their own, so that they are counted."""
    from icls_gpu import Solver
    wl = bench.make_workload("multi_drop_256_4")
    ls, u, v, w = bench.initial_state(wl)
    s = Solver(wl.cfg)
    s.setup(ls, u, v, w)
    s.step(1, 0)
    s.profile(True)
    s.profile_reset()
    for istep in range(2, 5):
        s.step(istep, 0)
    table = s.profile_table()
    assert s.launch_count() == sum(e["launches"] for e in table.values())
    s.profile(False)
    for name in ("ab2", "ab2_near", "band_begin"):
        assert table[name]["launches"] == table[name]["timed"] == 3, name
    assert bench.dominant_scope(table)[0] == "ab2"
    s.close()


@pytest.mark.gpu
def test_y_walls_are_scopes_of_their_own():
    """With walls in y: the wall rows of the predicted and the corrected
    velocities and of the pressure, and the probe for NaN, each step."""
    from icls_gpu import Solver, init_drops, make_config
    from icls_gpu.config import BCY_WALLS
    cfg = make_config(itot=32, jtot=32, ktot=32, bc_y=BCY_WALLS, timestep=1e-4)
    s = Solver(cfg)
    s.setup(init_drops(cfg, [(0.5, 0.5, 0.5)], [0.2]))
    s.profile(True)
    s.profile_reset()
    s.step(1, 0)
    table = s.profile_table()
    s.profile(False)
    assert table["ywalls"]["launches"] == 3
    for name in ("ab2", "bounduvw", "nan_probe"):
        assert table[name]["launches"] == table[name]["timed"] == 1, name
    s.close()


def test_predictor_bytes_follow_the_pressures_it_reads():
    """Far from the drops the predictor reads the two pressures only where the
    carrier is the heavier phase (1/rho1 - 1/min(rho1, rho2) is zero
    otherwise): 12 values per cell, or 14."""
    from icls_gpu import make_config
    n = 8 * 8 * 8
    for rho2, values in ((10.0, 12), (1.0, 12), (0.1, 14)):
        cfg = make_config(itot=8, jtot=8, ktot=8, rho1=1.0, rho2=rho2)
        assert bench.alg_bytes_per_launch("ab2", cfg, {}) == 8 * values * n
        assert bench.alg_bytes_per_launch("ab2", cfg, {}, True) == 4 * values * n


def test_captured_traffic_stands_for_its_own_workload():
    for workload, kernel, _ in bench.TRAFFIC:
        assert bench.make_workload(workload).name == workload and kernel in bench.ALG_VALUES
