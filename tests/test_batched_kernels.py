"""Batched and compacted launches against the one-drop or whole-array ones.

Each test runs the same steps through two routes that evaluate the same
expressions per cell, so the fields have to be the same bits.
"""
import numpy as np
import pytest

from icls_gpu import FP32, FP64, HOUC5, WENO5, Solver, init_drops, initial_velocity, make_config

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


@pytest.mark.parametrize("n,precision", [((64, 48, 50), FP64), ((48, 32, 41), FP32), ((32, 64, 33), FP64)])
def test_segment_maps_equal_whole_sweeps(n, precision):
    """Materials and jumps rebuilt near the drops only, against a context
    whose fields are re-uploaded (unchanged) before every step, so that it
    knows nothing of where they differ from their far values; and against the
    materials' whole sweep (ICLS_MATERIALS=rows1).  Moving drops, one across
    the seam and one near a wall; segments that are not full (48), one per
    row (32), odd row counts."""
    nx, ny, nz = n
    h = 1.0 / 64
    cfg = make_config(itot=nx, jtot=ny, ktot=nz, lmax=2, lx=nx * h, ly=ny * h, lz=nz * h, timestep=1e-3, rho2=10.0,
                      miu2=10.0, Re=100.0, We=0.5, v_wall_lower=-2.0, v_wall_upper=2.0, reinit_step=3,
                      precision=precision)
    ls = init_drops(cfg, [(0.01, 0.2, 0.25), (0.28, 0.3, 0.16)], [0.1, 0.09], all_images=True)
    plain, told, rows = (run_steps(cfg, ls, 0, **env) for env in ({}, {}, {"ICLS_MATERIALS": "rows1"}))
    for istep in range(1, 7):
        for name in ("jiemian", "p_x", "p_xold", "p_jump"):
            told.upload(name, told.download(name))
        for s in (plain, told, rows):
            s.step(istep, 0)
        for name in ("jiemian", "miu", "rho", "rho_u", "rho_v", "rho_w", "p_x", "p_y", "p_z", "p_xold", "p_yold",
                     "p_zold", "p_jump", "u", "v", "w", "pnew", "ucc"):
            a = plain.download(name)
            assert np.array_equal(a, told.download(name)), (istep, name)
            assert np.array_equal(a, rows.download(name)), (istep, name)
    # a field written by the caller is rebuilt whole
    plain.upload("miu", 3.0 + plain.download("miu"))
    plain.upload("p_x", 3.0 + plain.download("p_x"))
    plain.upload("p_xold", 3.0 + plain.download("p_xold"))
    plain.update_materials()
    plain.gfm4p()
    rows.gfm4p()
    for name in ("miu", "p_x", "p_jump"):
        assert np.array_equal(plain.download(name), rows.download(name)), name


@pytest.mark.parametrize("precision", [FP64, FP32])
@pytest.mark.parametrize("grid,scheme,drops", [((64, 48, 50), HOUC5, 3), ((96, 48, 40), WENO5, 3),
                                               ((96, 48, 40), HOUC5, 3), ((32, 32, 32), HOUC5, 66)])
def test_band_list_equals_columns(grid, scheme, drops, precision):
    """The advection stages over the tube's list of band cells against the
    column sweeps (ICLS_ADV=column): a drop across the seam, one whose region
    holds the wall and ghost rows, spacings where a/3 + 2a/3 is and is not a,
    reinitialisation and corrections in between, and more drops than one
    batch holds."""
    nx, ny, nz = grid
    h = 1.0 / max(nx, ny)
    cfg = make_config(itot=nx, jtot=ny, ktot=nz, lmax=drops, lx=nx * h, ly=ny * h, lz=nz * h, timestep=1e-3,
                      rho2=10.0, miu2=10.0, Re=100.0, We=0.5, v_wall_lower=-1.0, v_wall_upper=1.0,
                      ls_adv_space=scheme, reinit_step=2, inflate_step=3, mass_threshold=1e-9, mass_gain_one=1,
                      precision=precision)
    at = [((0.02, 0.4, 0.55), 11.0), ((0.5, 0.3, 0.2), 7.0), ((0.6, 0.75, 0.6), 8.0)]
    at = [at[l % 3] for l in range(drops)]
    ls = init_drops(cfg, [(x * cfg.lx, y * cfg.ly, z * cfg.lz) for (x, y, z), _ in at],
                    [r * h * (nx / 64 if drops > 3 else 1.0) for _, r in at], all_images=True)
    lists = run_steps(cfg, ls, 5)
    cols = run_steps(cfg, ls, 5, ICLS_ADV="column")
    for l in list(range(1, min(drops, 3) + 1)) + [drops]:
        assert np.array_equal(lists.download("lvset", l), cols.download("lvset", l)), l
        assert lists.band_count(l) == cols.band_count(l)
    for name in ("u", "v", "w", "pnew", "jiemian", "curv"):
        assert np.array_equal(lists.download(name), cols.download(name)), name
    assert np.array_equal(lists.volumes()[0], cols.volumes()[0])


@pytest.mark.parametrize("precision", [FP64, FP32])
def test_short_chunks_equal_long_ones(precision):
    """A batch of twelve drops has chunks of eight rows, a drop alone
    (ICLS_GROUP=1) chunks of two, longer at the walls that the upper and lower
    drops' regions reach; every step reinitialises."""
    h = 1.0 / 64
    cfg = make_config(itot=96, jtot=96, ktot=45, lmax=12, lx=96 * h, ly=96 * h, lz=45 * h, timestep=1e-3, rho2=10.0,
                      miu2=10.0, Re=100.0, We=0.5, v_wall_lower=-0.5, v_wall_upper=0.5, reinit_step=1,
                      reinit_iter_max=2, precision=precision)
    pos = [(12 + 24 * (l % 4), 16 + 32 * (l // 4), (10, 22, 34)[l % 3]) for l in range(12)]
    ls = init_drops(cfg, [tuple(h * x for x in q) for q in pos], [8 * h] * 12, all_images=True)
    one = run_steps(cfg, ls, 3, ICLS_GROUP="1")
    all_ = run_steps(cfg, ls, 3)
    for l in range(1, 13):
        assert np.array_equal(one.download("lvset", l), all_.download("lvset", l)), l
    for name in ("u", "v", "w", "pnew", "jiemian", "miu", "rho_u", "p_x", "p_y", "p_z", "p_jump"):
        assert np.array_equal(one.download(name), all_.download(name)), name
    assert np.array_equal(one.volumes()[0], all_.volumes()[0])


@pytest.mark.parametrize("n,precision", [((64, 48, 50), FP64), ((48, 32, 41), FP32), ((64, 32, 6), FP64)])
def test_separate_projection_calls_equal_whole_sweeps(n, precision):
    """correc reads the jumps near the drops only, against a context told (by
    an upload of the same values) that it knows nothing of them; row counts
    that the rows per thread do and do not divide."""
    nx, ny, nz = n
    h = 1.0 / 64
    cfg = make_config(itot=nx, jtot=ny, ktot=nz, lx=nx * h, ly=ny * h, lz=nz * h, timestep=1e-3, rho2=10.0, miu2=10.0,
                      Re=100.0, We=0.5, v_wall_lower=-0.5, v_wall_upper=0.5, precision=precision)
    ls = init_drops(cfg, [(0.02, 0.3, 0.5 * nz * h)], [0.1], all_images=True)
    near, told = run_steps(cfg, ls, 2), run_steps(cfg, ls, 2)
    told.upload("p_x", told.download("p_x"))
    for s in (near, told):
        s.fillps()
        s.add_pjump()
        s.correc()
    for name in ("p", "u", "v", "w"):
        assert np.array_equal(near.download(name), told.download(name)), name
    assert np.any(near.download("p_x"))


@pytest.mark.parametrize("precision", [FP64, FP32])
@pytest.mark.parametrize("rho1,rho2,miu1,iFr", [(1.5, 0.3, 0.7, 0.0), (0.75, 2.5, 1.3, 0.98), (2.0, 1.0, 1.0, 0.98)])
def test_far_rows_of_the_predictor_equal_general_ones(rho1, rho2, miu1, iFr, precision):
    """The predictor's far rows against a context told (by an upload of the
    same values) that it knows nothing of the fields: a carrier that is the
    heavier phase, so that far rows read the pressures, densities that are and
    are not powers of two, buoyancy along all three axes.  FP64: the same
    bits.  FP32, whose rows may contract and divide differently: du/dt is u
    plus a step dt R of some hundredths of it, so a few ulps of R are below an
    ulp of u, and the last sums round to within four."""
    cfg = make_config(itot=64, jtot=48, ktot=50, ly=0.75, lz=50 / 64, timestep=1e-3, rho1=rho1, rho2=rho2, miu1=miu1,
                      miu2=0.4, Re=100.0, We=0.5, iFr=iFr, g_unit=(0.3, -0.2, -1.0), v_wall_lower=-0.5,
                      v_wall_upper=0.5, precision=precision)
    ls = init_drops(cfg, [(0.15, 0.15, 0.4)], [0.1], all_images=True)
    far, told = run_steps(cfg, ls, 2), run_steps(cfg, ls, 2)
    told.upload("p_x", told.download("p_x"))
    for s in (far, told):
        s.ab2()
    for name in ("dudt", "dvdt", "dwdt", "duold", "dvold", "dwold"):
        a, b = far.download(name), told.download(name)
        if precision == FP64:
            assert np.array_equal(a, b), name
        elif name.endswith("dt"):
            assert np.max(np.abs(a - b)) <= 4 * 2.0 ** -23 * np.max(np.abs(b)), name


@pytest.mark.parametrize("precision", [FP64, FP32])
def test_far_rows_read_a_pressure_that_is_not_finite(precision):
    """Far rows skip the pressures where their factor is zero; an infinite one
    far from the drop still reaches the cells whose gradient reads it."""
    cfg = make_config(itot=64, jtot=48, ktot=50, ly=0.75, lz=50 / 64, timestep=1e-3, rho2=10.0, miu2=10.0, Re=100.0,
                      We=0.5, v_wall_lower=-0.5, v_wall_upper=0.5, precision=precision)
    ls = init_drops(cfg, [(0.15, 0.15, 0.4)], [0.1], all_images=True)
    far, told = run_steps(cfg, ls, 2), run_steps(cfg, ls, 2)
    for s in (far, told):
        p = s.download("p")
        p[56, 40, 9] = np.inf
        s.upload("p", p)
        s.pressure_update(3, 0)
    told.upload("p_x", told.download("p_x"))
    for s in (far, told):
        s.ab2()
    for name in ("dudt", "dvdt", "dwdt"):
        a, b = far.download(name), told.download(name)
        assert np.array_equal(np.isnan(a), np.isnan(b)) and np.isnan(b).any(), name
        if precision == FP64:
            assert np.array_equal(a, b, equal_nan=True), name
