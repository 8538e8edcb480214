"""Batched and compacted launches against the one-drop or whole-array ones.

Each test runs the same steps through two routes that evaluate the same
expressions per cell, so the fields have to be the same bits.
"""
import numpy as np
import pytest

from icls_gpu import FP32, FP64, HOUC5, Solver, init_drops, initial_velocity, make_config

pytestmark = pytest.mark.gpu


def run_steps(cfg, ls, steps, shear=0.5, **env):
    """the solver after `steps` steps, created under the given environment"""
    mp = pytest.MonkeyPatch()
    for k, v in env.items():
        mp.setenv(k, v)
    s = Solver(cfg)
    mp.undo()
    s.setup(ls, *initial_velocity(cfg, shear))
    for istep in range(1, steps + 1):
        s.step(istep, 0)
    return s


@pytest.mark.parametrize("gain_one", [0, 1])
@pytest.mark.parametrize("precision", [FP64, FP32])
def test_corrections_of_all_drops_equal_one_at_a_time(precision, gain_one):
    """Drops a few cells apart (their sweep regions overlap), one across the
    periodic seam and one near a wall, corrected in the same launches or one
    drop at a time (ICLS_GROUP=1)."""
    cfg = make_config(itot=64, jtot=48, ktot=50, lmax=4, ly=0.75, lz=50 / 64, timestep=1e-4, rho2=10.0, miu2=10.0,
                      Re=100.0, We=0.5, v_wall_lower=-0.5, v_wall_upper=0.5, ls_adv_space=HOUC5, inflate_step=2,
                      reinit_step=2, mass_threshold=1e-13, mass_gain_one=gain_one, precision=precision)
    ls = init_drops(cfg, [(0.3, 0.3, 0.4), (0.62, 0.3, 0.42), (0.02, 0.6, 0.36), (0.5, 0.6, 0.14)],
                    [0.12, 0.13, 0.11, 0.09], all_images=True)
    one = run_steps(cfg, ls, 4, ICLS_GROUP="1")
    all_ = run_steps(cfg, ls, 4)
    assert one.scalars()["last_inflated"] == all_.scalars()["last_inflated"] == 4
    for l in range(1, 5):
        assert np.array_equal(one.download("lvset", l), all_.download("lvset", l)), l
    for name in ("u", "v", "w", "pnew", "jiemian", "curv", "normal_m"):
        assert np.array_equal(one.download(name), all_.download(name)), name
    assert np.array_equal(one.volumes()[0], all_.volumes()[0])
    assert one.scalars()["maxchk_glb"] == all_.scalars()["maxchk_glb"]
