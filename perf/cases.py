"""The work that a user of this framework has it do, as cases that can be timed and compared.

Six kinds of case, each through the public entry points of ``icls_gpu``:

  step        whole main-loop iterations (``Solver.step``): a static drop, a
              rising bubble, seeded drops in shear or in turbulence
  momentum    the AB2 predictor (``Solver.ab2``)
  projection  fillps, p + p_jump, solver2d, boundp, correc, bounduvw, the
              pressure update and the cell-centre velocities, called one by
              one as the Fortran driver calls them
  levelset    ``Solver.ls_main``: tube, RK3 advection, (reinitialisation,)
              materials, for all drops
  interface   ``Solver.gfm4p``: curvature and the ghost-fluid pressure jumps
  mlp_grad    forward and backward pass of the curvature network over a batch

A case names its grid (nx, ny, nz; the spacing is 1 / max(nx, ny) along every
axis), the number of drops, the form ("fp64" or "fp32") and what its kind
takes besides.  Grid lengths are those the solver accepts: 48, 96, 192, 384 and
powers of two along x (and y, when periodic), any length along z (and along y
between walls).

The solver's fields stay on the GPU.  ``run`` queues the calls and returns
handles of the solver's own fields (``Fields``), which are downloaded when they
are read, as a tensor on the GPU would be.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "icls-release_b200"))

from icls_gpu import (BCY_PERIODIC, BCY_WALLS, CURV_MLP, CURV_STENCIL, FP32, FP64, HOUC5, WENO5,  # noqa: E402
                      Solver, make_config)
from icls_gpu.binding import Mlp  # noqa: E402

RHO2, MIU2 = 10.0, 10.0  # drops ten times as dense and as viscous as the carrier (rho1 = miu1 = 1)
DT = 1e-5


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest run in use: the static drop at 64^3, WENO5, two reinitialisation iterations a step;
        # one step is about thirty short launches
        dict(name="step_static_64", kind="step", flow="static", nx=64, ny=64, nz=64, drops=1, form="fp64", steps=1),
        # the rising bubble at its stated size, reinitialised and volume-corrected every step
        dict(name="step_bubble_128x128x256", kind="step", flow="bubble", nx=128, ny=128, nz=256, drops=1, form="fp64",
             steps=1),
        # the headline box: 256^3 with 48 seeded drops in shear, plain FP64, one output interval (20 steps with one
        # reinitialisation and one divergence check)
        dict(name="step_drops_256_fp64", kind="step", flow="shear", nx=256, ny=256, nz=256, drops=48, form="fp64",
             steps=20),
        # the same box in the FP32 form with the learned curvature, in a turbulent flow
        dict(name="step_drops_256_learned", kind="step", flow="turbulent", nx=256, ny=256, nz=256, drops=48,
             form="fp32", learned=True, steps=20),
        # the predictor alone, as the driver calls it: the largest FP64 box, and a wide FP32 box whose z extent
        # is no multiple of anything
        dict(name="momentum_256_fp64", kind="momentum", nx=256, ny=256, nz=256, form="fp64"),
        dict(name="momentum_384x192x150_fp32", kind="momentum", nx=384, ny=192, nz=150, form="fp32"),
        # the projection, call by call: periodic at the largest FP64 box, and a channel between y walls of odd
        # extents in the FP32 form (cosine transform by the direct product)
        dict(name="projection_256_fp64", kind="projection", nx=256, ny=256, nz=256, form="fp64", walls_y=False),
        dict(name="projection_walls_128x90x75", kind="projection", nx=128, ny=90, nz=75, form="fp32", walls_y=True),
        # the level-set step: 48 drops, HOUC5, FP32 (an ordinary step), and WENO5 with reinitialisation on a ragged
        # FP64 box with a spacing that is no power of two
        dict(name="levelset_256_fp32", kind="levelset", nx=256, ny=256, nz=256, drops=48, form="fp32", scheme="houc5",
             reinit=False),
        dict(name="levelset_96x192x100_reinit", kind="levelset", nx=96, ny=192, nz=100, drops=10, form="fp64",
             scheme="weno5", reinit=True),
        # curvature and pressure jumps of 24 drops in FP64
        dict(name="interface_256_fp64", kind="interface", nx=256, ny=256, nz=256, drops=24, form="fp64"),
        # one training batch of the curvature network, forward and backward
        dict(name="mlp_grad_8192", kind="mlp_grad", n=8192),
    ]


def draw(rng):
    lengths = [32, 48, 64, 96, 128, 192, 256]

    def between(a, b):  # a whole number, spread over its logarithm
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["step", "step", "momentum", "projection", "levelset", "levelset", "interface", "mlp_grad"])
    if kind == "mlp_grad":
        return dict(kind=kind, n=2 ** rng.randint(9, 16))
    small = kind in ("step", "levelset", "interface")
    while True:
        nx, ny = rng.choice(lengths[1 if small else 0:]), rng.choice(lengths[1 if small else 0:])
        nz = between(52 if small else 24, 280)
        if 1 / 4 <= nx / ny <= 4 and 40000 <= nx * ny * nz <= 15_000_000:
            break
    form = rng.choice(["fp64", "fp32"])
    case = dict(kind=kind, nx=nx, ny=ny, nz=nz, form=form)
    # at most one drop to 40 cells cubed, so that seeded drops find room
    most = max(1, min(48, nx * ny * nz // 64000))
    if kind == "step":
        learned = form == "fp32" and rng.random() < 0.5
        case.update(flow=rng.choice(["shear", "turbulent"]), drops=between(1, most), steps=rng.choice([1, 3, 20]),
                    learned=learned)
        h = spacing(case)
        while learned and case["nz"] * h / case["nz"] != h:  # the network wants the same spacing to the last bit
            case["nz"] += 1
    elif kind == "projection":
        case.update(walls_y=rng.random() < 0.4)
        if case["walls_y"]:
            case["ny"] = between(24, 256)
    elif kind == "levelset":
        case.update(drops=between(1, most), scheme=rng.choice(["houc5", "weno5"]), reinit=rng.random() < 0.4)
    elif kind == "interface":
        case.update(drops=between(1, most))
    return case


# --------------------------------------------------------------- seeded inputs
# Fields are [k, j, i] tensors in FP64 on the GPU; the solver's arrays are their transposes.
def generator(seed, what):
    return torch.Generator("cuda").manual_seed((int(seed) * 64 + what) % (1 << 62))


def smooth(case, seed, what, count=6, most=5):
    """a sum of low modes over the cell centres, periodic in x and y, of unit size"""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = np.random.default_rng([int(seed), what])
    f = torch.zeros(nz, ny, nx, dtype=torch.float64, device="cuda")
    x, y, z = (2 * math.pi * (torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) / n for n in (nx, ny, nz))
    for _ in range(count):
        kx, ky, kz = (int(v) for v in r.integers(0, most, 3))
        a, b, c = r.uniform(0, 2 * math.pi, 3)
        f += (torch.sin(kz * z + c) + 0.2)[:, None, None] * (torch.sin(ky * y + b) + 0.1)[None, :, None] * \
            (torch.sin(kx * x + a) + 0.1)[None, None, :]
    return f / math.sqrt(count)


def noise(case, seed, what):
    return torch.randn(case["nz"], case["ny"], case["nx"], dtype=torch.float64, device="cuda",
                       generator=generator(seed, what))


def rounded(case, f):
    """inputs that the form holds exactly, so that every computation starts from the same values"""
    return f.float().double() if case["form"] == "fp32" else f


def spacing(case):
    return 1.0 / max(case["nx"], case["ny"])


def placed(case, seed):
    """seeded drops (centre and radius in cells): radii 7.7 to 15 cells, smaller on small grids, at least 4 cells
    apart and clear of the z walls; positions are spread by rejection"""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = np.random.default_rng([int(seed), 7])
    big = min(15.0, 0.25 * min(nx, ny, nz))
    drops = []
    for tries in range(200000):
        if len(drops) == case["drops"]:
            break
        rad = r.uniform(0.55 * big, big) * (1.0 if tries < 2000 else 0.7)
        edge = rad + 8.0
        c = np.array([r.uniform(0, nx), r.uniform(0, ny), r.uniform(edge, nz - edge)])
        far = True
        for c2, r2 in drops:
            d = c - c2
            d[0] -= nx * round(d[0] / nx)
            d[1] -= ny * round(d[1] / ny)
            far = far and float(np.linalg.norm(d)) >= rad + r2 + 4.0
        if far:
            drops.append((c, rad))
    if len(drops) < case["drops"]:
        raise RuntimeError("no room for the drops")
    return drops


def drop_field(case, drop, halo=0):
    """a drop's level set (a signed distance with a ripple of a twentieth of a cell, capped at 12 cells) over
    the cells -halo+1 .. n+halo"""
    h = spacing(case)
    (cx, cy, cz), rad = drop

    def away(n, c, period):
        d = torch.arange(1 - halo, n + halo + 1, dtype=torch.float64, device="cuda") - 0.5 - c
        return d - period * torch.round(d / period) if period else d

    x, y, z = away(case["nx"], cx, case["nx"]), away(case["ny"], cy, case["ny"]), away(case["nz"], cz, 0)
    f = (x * x)[None, None, :] + (y * y)[None, :, None]
    f = torch.sqrt(f + (z * z)[:, None, None]) - rad
    f += 0.05 * torch.sin(0.5 * x)[None, None, :] * torch.cos(0.4 * y)[None, :, None] * torch.sin(0.45 * z)[:, None, None]
    return rounded(case, torch.clamp(f, max=12.0) * h)


def solenoidal(case, seed, rms=0.2, count=10, most=6):
    """u, v, w as the discrete curl of a seeded potential on the cell edges, which vanishes at the z walls"""
    nx, ny, nz, h = case["nx"], case["ny"], case["nz"], spacing(case)
    r = np.random.default_rng([int(seed), 11])

    def axis(n, shift, k, ph):
        p = (torch.arange(1, n + 1, dtype=torch.float64, device="cuda") + shift) / n
        return torch.sin(2 * math.pi * k * p + ph)

    def wall(shift, m):
        p = (torch.arange(0 if shift == 0 else 1, nz + 1, dtype=torch.float64, device="cuda") + shift) / nz
        return torch.sin(math.pi * m * p)

    def potential(sx, sy, sz):
        a = 0
        for _ in range(count):
            kx, ky, m = (int(v) for v in r.integers(1, most, 3))
            p, q, s = r.uniform(0, 2 * math.pi, 3)
            amp = math.cos(s) / (kx * kx + ky * ky + 0.25 * m * m)
            a = a + amp * wall(sz, m)[:, None, None] * axis(ny, sy, ky, q)[None, :, None] * axis(nx, sx, kx, p)[None, None, :]
        return a

    ax, ay, az = potential(-0.5, 0, 0), potential(0, -0.5, 0), potential(0, 0, -0.5)
    u = (az - az.roll(1, 1)) - (ay[1:] - ay[:-1])
    v = (ax[1:] - ax[:-1]) - (az - az.roll(1, 2))
    w = (ay - ay.roll(1, 2))[1:] - (ax - ax.roll(1, 1))[1:]
    scale = rms / math.sqrt(float((u * u).mean() + (v * v).mean() + (w * w).mean()) / 3.0) if h else 0.0
    return [scale * f for f in (u, v, w)]


def halo(f, kind, walls_y=False):
    """one layer of halo cells around an interior field: periodic x and y, and at the z walls a copy ("p"), the
    reflection of a tangential velocity ("t") or a wall-normal one ("w", zero at the top face)"""
    g = torch.cat([f[..., -1:], f, f[..., :1]], dim=2)
    g = torch.cat([g[:, -1:], g, g[:, :1]], dim=1)
    if kind == "p":
        return torch.cat([g[:1], g, g[-1:]])
    if kind == "t":
        return torch.cat([-g[:1], g, -g[-1:]])
    return torch.cat([torch.zeros_like(g[:1]), g, g[-2:-1]])


def materials(case, seed):
    """a smeared indicator (1 in the carrier, 0 in the dense phase) as drops give it, the viscosity and the three
    face densities"""
    j = torch.clamp(0.5 + 3.0 * (smooth(case, seed, 21) + 0.5), 0.0, 1.0)
    rho = j + RHO2 * (1 - j)
    ru, rv = 0.5 * (rho + rho.roll(-1, 2)), 0.5 * (rho + rho.roll(-1, 1))
    rw = 0.5 * (rho + torch.cat([rho[1:], rho[-1:]]))
    return [rounded(case, f) for f in (j, j + MIU2 * (1 - j), ru, rv, rw)]


def jump(case, seed, what, j, size):
    """a face jump: nonzero at the interface only"""
    return rounded(case, size * noise(case, seed, what) * ((j > 0) & (j < 1)))


def momentum_fields(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    F = {}
    for q, n in enumerate("uvw"):
        f = 0.3 * smooth(case, seed, 1 + q) + 0.003 * noise(case, seed, 1 + q)
        if n == "w":
            f[-1] = 0.0
        F[n] = halo(rounded(case, f), "w" if n == "w" else "t")
    j, miu, F["rho_u"], F["rho_v"], F["rho_w"] = materials(case, seed)
    F["miu"] = halo(miu, "p")
    for q, n in enumerate(("duold", "dvold", "dwold")):
        F[n] = rounded(case, smooth(case, seed, 31 + q) + 0.1 * noise(case, seed, 31 + q))
    p = 5.0 * smooth(case, seed, 41) + 10.0 * (1 - j)
    F["pnew"] = halo(rounded(case, p), "p")
    F["pold"] = halo(rounded(case, p + 0.01 * smooth(case, seed, 42)), "p")
    for q, n in enumerate(("p_x", "p_y", "p_z")):
        a = jump(case, seed, 51 + q, j, 10.0)
        F[n], F[n + "old"] = halo(a, "p"), halo(rounded(case, 0.99 * a), "p")
    return F


def projection_fields(case, seed):
    F = {}
    walls = case["walls_y"]
    for q, n in enumerate(("dudt", "dvdt", "dwdt")):
        f = 0.3 * smooth(case, seed, 1 + q) + 0.003 * noise(case, seed, 1 + q)
        if n == "dwdt":
            f[-1] = 0.0
        if n == "dvdt" and walls:
            f[:, -1] = 0.0
        f = halo(rounded(case, f), "w" if n == "dwdt" else "t")
        if n == "dvdt" and walls:
            f[:, 0] = 0.0
            f[:, -1] = 0.0
        F[n] = f
    j = torch.clamp(0.5 + 3.0 * (smooth(case, seed, 21) + 0.5), 0.0, 1.0)
    for q, n in enumerate(("p_x", "p_y", "p_z")):
        f = jump(case, seed, 51 + q, j, 10.0)
        if n == "p_y" and walls:
            f[:, -1] = 0.0
        F[n] = halo(f, "p")
    f = 1e4 * noise(case, seed, 61) * ((j > 0) & (j < 1))
    F["p_jump"] = halo(f - f.mean(), "p")
    F["pnew"] = halo(rounded(case, 5.0 * smooth(case, seed, 41)), "p")
    return F


def cell_velocity(case, seed):
    return {n: rounded(case, 0.3 * smooth(case, seed, 71 + q)) for q, n in enumerate(("ucc", "vcc", "wcc"))}


def network(seed, out=0.05):
    """parameters of the curvature network, of a trained network's size (corrections of about a thousandth)"""
    r = np.random.default_rng([int(seed), 13])
    w1 = np.zeros((128, 32))
    w1[:, :27] = r.uniform(-1, 1, (128, 27)) / math.sqrt(27)
    parts = [w1, 0.02 * r.standard_normal(128), r.uniform(-1, 1, (128, 128)) / math.sqrt(128),
             0.02 * r.standard_normal(128), r.uniform(-1, 1, (64, 128)) / math.sqrt(128),
             0.02 * r.standard_normal(64), out * r.uniform(-1, 1, 64) / 8, np.zeros(1)]
    return np.concatenate([p.ravel() for p in parts]).astype(np.float32)


def samples(case, seed):
    """inputs of the network as the level sets give them: small second differences and a unit gradient"""
    g = generator(seed, 81)
    x = torch.zeros(case["n"], 32, device="cuda")
    x[:, :27] = 0.05 * torch.randn(case["n"], 27, device="cuda", generator=g)
    d = torch.randn(case["n"], 3, device="cuda", generator=g)
    x[:, 27:30] = d / d.norm(dim=1, keepdim=True)
    return x, 0.02 * torch.randn(case["n"], device="cuda", generator=g)


# ---------------------------------------------------------------- the solver
class Fields(dict):
    """The solver's fields by name, each downloaded when it is read: a [k, j, i] array over the interior cells,
    in the type that the solver holds it in."""

    FP64 = ("p", "p_jump")

    def __init__(self, solver, names):
        super().__init__((n, None) for n in names)
        self.solver = solver

    def __getitem__(self, name):
        s = self.solver
        if name == "volumes":
            v = s.volumes()[0]
        elif name.startswith("lvset_"):
            v = s.interior("lvset", int(name[6:])).T
        else:
            v = s.interior(name).T
        narrow = s.cfg.precision == FP32 and name not in self.FP64
        return np.ascontiguousarray(v, dtype=np.float32 if narrow else np.float64)


def upload(solver, name, f, l=1):
    solver.upload(name, f.cpu().numpy().T, l)


def upload_drops(solver, case, drops):
    n = [case["nz"] + 6, case["ny"] + 6, case["nx"] + 6]
    pinned = torch.empty(n, dtype=torch.float64, pin_memory=True)
    for l, d in enumerate(drops):
        pinned.copy_(drop_field(case, d, halo=3))
        solver.upload_ptr("lvset", pinned.data_ptr(), l + 1)


def config(case, **more):
    h = spacing(case)
    kw = dict(itot=case["nx"], jtot=case["ny"], ktot=case["nz"], lmax=case.get("drops", 1),
              lx=case["nx"] * h, ly=case["ny"] * h, lz=case["nz"] * h, timestep=DT,
              rho1=1.0, rho2=RHO2, miu1=1.0, miu2=MIU2, Re=10.0, We=2.0,
              precision=FP32 if case["form"] == "fp32" else FP64, bc_y=BCY_PERIODIC)
    kw.update(more)
    return make_config(**kw)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp_grad":
        net = Mlp(1)
        net.set_params(network(seed, out=1.0))
        x, label = samples(case, seed)
        torch.cuda.synchronize()
        return dict(case=case, net=net, x=x, label=label)
    if kind == "step":
        return prepare_step(case, seed)
    if kind in ("momentum", "projection"):
        walls = case.get("walls_y", False)
        solver = Solver(config(case, bc_y=BCY_WALLS if walls else BCY_PERIODIC, mass_correction=0))
        upload_drops(solver, case, [((0.5 * case["nx"], 0.5 * case["ny"], 0.5 * case["nz"]),
                                     0.2 * min(case["nx"], case["ny"], case["nz"]))])
        solver.init_program()
        fields = momentum_fields(case, seed) if kind == "momentum" else projection_fields(case, seed)
        for name, f in fields.items():
            upload(solver, name, f)
        return dict(case=case, solver=solver, count=0)
    # levelset, interface
    scheme = WENO5 if case.get("scheme") == "weno5" else HOUC5
    solver = Solver(config(case, ls_adv_space=scheme, mass_correction=0, reinit_step=1 if case.get("reinit") else 20))
    upload_drops(solver, case, placed(case, seed))
    solver.init_program()
    if kind == "levelset":
        for name, f in cell_velocity(case, seed).items():
            upload(solver, name, f)
    return dict(case=case, solver=solver, count=0)


def prepare_step(case, seed):
    flow, h = case["flow"], spacing(case)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = np.random.default_rng([int(seed), 3])
    # the volume correction that stays stable over a long run: gain one, 1e-7
    more = dict(mass_gain_one=1, mass_threshold=1e-7)
    if flow == "static":
        more.update(timestep=1e-4, Re=100.0, We=0.1, ls_adv_space=WENO5, reinit_step=1, reinit_iter_max=2)
        drops = [((0.5 * nx + r.uniform(-1, 1), 0.5 * ny + r.uniform(-1, 1), 0.5 * nz + r.uniform(-1, 1)), 0.25 * nx)]
    elif flow == "bubble":
        more.update(timestep=4e-5, rho2=0.1, miu2=0.1, Re=100.0, We=1000.0 / 24.5, iFr=0.98,
                    g_unit=(0.0, 0.0, -1.0), ls_adv_space=HOUC5, reinit_step=1, inflate_step=1)
        drops = [((0.5 * nx + r.uniform(-1, 1), 0.5 * ny + r.uniform(-1, 1), 0.25 * nz + r.uniform(-1, 1)), 0.125 * nx)]
    else:
        drops = placed(case, seed)
        if flow == "shear":
            more.update(v_wall_lower=-0.5, v_wall_upper=0.5)
        else:
            more.update(We=5.0)
    learned = case.get("learned", False)
    more.update(curvature_model=CURV_MLP if learned else CURV_STENCIL)
    solver = Solver(config(case, **more))
    if flow == "shear":
        z = (torch.arange(0, nz + 2, dtype=torch.float64, device="cuda") - 0.5) / nz
        upload(solver, "v", (0.5 * (2.0 * z - 1.0))[:, None, None].expand(nz + 2, ny + 2, nx + 2).contiguous())
    elif flow == "turbulent":
        for name, f in zip("uvw", solenoidal(case, seed)):
            upload(solver, name, halo(f, "w" if name == "w" else "t"))
    upload_drops(solver, case, drops)
    solver.init_program()
    state = dict(case=case, solver=solver, count=0)
    if learned:
        state["net"] = Mlp(1)
        state["net"].set_params(network(seed))
        state["net"].attach(solver)
    return state


def level_sets(case):
    """the drops' level sets, up to twelve of them (the indicator jiemian is made of all)"""
    return ["lvset_%d" % (l + 1) for l in range(min(case["drops"], 12))]


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "mlp_grad":
        grad, loss = state["net"].grad(state["x"].data_ptr(), state["label"].data_ptr(), case["n"], 2.0 / case["n"])
        return dict(grad=grad, loss=np.float32(loss))
    s = state["solver"]
    if kind == "step":
        for _ in range(case["steps"]):
            state["count"] += 1
            s.step(state["count"])
        return Fields(s, ["u", "v", "w", "pnew", "pold", "p_x", "p_y", "p_z", "jiemian"] + level_sets(case))
    state["count"] += 1
    if kind == "momentum":
        s.ab2()
        return Fields(s, ["dudt", "dvdt", "dwdt", "duold", "dvold", "dwold"])
    if kind == "projection":
        s.fillps()
        s.add_pjump()
        s.solver2d()
        s.boundp()
        s.correc()
        s.bounduvw()
        s.pressure_update(1)
        s.average_vel_at_center()
        return Fields(s, ["p", "u", "v", "w", "pnew", "pold", "ucc", "vcc", "wcc"])
    if kind == "levelset":
        s.ls_main(state["count"])
        return Fields(s, ["jiemian", "miu", "rho", "rho_u", "rho_v", "rho_w"] + level_sets(case))
    s.gfm4p()
    return Fields(s, ["p_x", "p_y", "p_z", "p_jump"])


# ------------------------------------------------------------------- the work
def band_cells(case):
    """cells within 6 spacings of the drops' surfaces, and within 2"""
    big = min(15.0, 0.25 * min(case["nx"], case["ny"], case["nz"]))
    if case.get("flow") in ("static", "bubble"):
        r = (0.25 if case["flow"] == "static" else 0.125) * case["nx"]
    else:
        r = 0.78 * big
    band = [4 / 3 * math.pi * ((r + w) ** 3 - max(0.0, r - w) ** 3) * case.get("drops", 1) for w in (6.0, 2.0)]
    return band


def work(case):
    """Bytes of one pass with every input read once and every output written once, in the form's types (the
    pressure solve and the Laplacian of the jumps are FP64 in both forms)."""
    kind = case["kind"]
    if kind == "mlp_grad":
        macs = 64 * 128 + 128 * 128 + 128 * 64 + 64
        return {"bytes": case["n"] * 33 * 4 + 2 * 29057 * 4, "flops": 3 * 2 * macs * case["n"]}
    n = case["nx"] * case["ny"] * case["nz"]
    t = 4 if case["form"] == "fp32" else 8
    if kind == "momentum":  # u v w miu, 3 densities, 3 histories, 2 pressures, 6 jumps in; 3 velocities, 3 histories out
        return {"bytes": 24 * t * n, "flops": 330 * n}
    fft = 5 * n * (math.log2(case["nx"]) + math.log2(case["ny"])) + 10 * n
    if kind == "projection":  # dudt.., jumps, pnew in; u.., ucc.., pnew, pold out; p_jump in, p out
        return {"bytes": (3 + 3 + 1 + 3 + 3 + 2) * t * n + 2 * 8 * n, "flops": fft + 40 * n}
    band, shell = band_cells(case)
    advect = band * (2 * t + 3 * t)  # a level set in and out, three velocities
    mats = 6 * t * n
    if kind == "levelset":
        return {"bytes": advect + mats, "flops": 3 * 60 * band + 20 * n}
    face = shell * t + (3 * t + 8) * n  # level sets in, the three face jumps and their Laplacian out
    if kind == "interface":
        return {"bytes": face, "flops": 600 * shell}
    # step: the predictor, the solve with its right-hand side, the correction with the cell-centre velocities, the
    # pressure update, and the level-set work
    step = 24 * t * n + (3 * t + 2 * 8) * n + (6 * t + 6 * t + 8) * n + (3 * t + 8) * n + advect + mats + face
    return {"bytes": case["steps"] * step, "flops": case["steps"] * (330 * n + fft + 60 * n + 800 * shell + 180 * band)}


# --------------------------------------------- the same in plain torch, 64 bits
def at(f, di, dj, dk):
    """a field with halo at the interior cells shifted by (di, dj, dk)"""
    nz, ny, nx = (v - 2 for v in f.shape)
    return f[1 + dk:1 + dk + nz, 1 + dj:1 + dj + ny, 1 + di:1 + di + nx]


def exact_momentum(case, seed):
    F, h = momentum_fields(case, seed), spacing(case)
    visc, dt, off = 1.0 / 10.0, DT, {"u": (1, 0, 0), "v": (0, 1, 0), "w": (0, 0, 1)}
    out = {}

    def vel(n, s, a=None):  # velocity n at the shift s (+ a)
        s = s if a is None else tuple(x + y for x, y in zip(s, a))
        return at(F[n], *s)

    def neg(a):
        return tuple(-x for x in a)

    zero = (0, 0, 0)
    for n in "uvw":
        e, conv, diff = off[n], 0, 0
        for m in "uvw":
            d = off[m]
            # momentum flux of component n through the faces of its cell along m, and the viscous flux
            up = 0.25 * (vel(n, zero) + vel(n, d)) * (vel(m, zero) + vel(m, e))
            dn = 0.25 * (vel(n, zero) + vel(n, neg(d))) * (vel(m, neg(d)) + vel(m, neg(d), e))
            conv = conv - (up - dn) / h
            if m == n:
                mp, mm = at(F["miu"], *e), at(F["miu"], 0, 0, 0)
            else:
                def corner(s):
                    return 0.25 * sum(at(F["miu"], *(x * a + y * b for x, y in zip(e, s)))
                                      for a in (0, 1) for b in (0, 1))
                mp, mm = corner(d), corner(neg(d))
            sp = (vel(n, d) - vel(n, zero)) + (vel(m, e) - vel(m, zero))
            sm = (vel(n, zero) - vel(n, neg(d))) + (vel(m, neg(d), e) - vel(m, neg(d)))
            diff = diff + (mp * sp - mm * sm) / (h * h)
        rf = F["rho_" + n]
        R = conv + visc * diff / rf
        ph = 2 * F["pnew"] - F["pold"]
        ax = "xyz"["uvw".index(n)]
        pj = at(2 * F["p_" + ax] - F["p_%sold" % ax], 0, 0, 0)
        new = vel(n, zero) + dt * (1.5 * R - 0.5 * F["d%sold" % n])
        new = new - dt * (1 / rf - 1.0) / h * ((at(ph, *e) - pj) - at(ph, 0, 0, 0))
        if n == "w":
            new[-1] = 0.0
        out["d%sdt" % n], out["d%sold" % n] = new, R
    return out


def cosines(n):
    """orthonormal cosine modes of a line between walls, and their eigenvalues for unit spacing"""
    k = torch.arange(n, dtype=torch.float64, device="cuda")
    c = torch.cos(math.pi * k[:, None] * (k[None, :] + 0.5) / n) * math.sqrt(2.0 / n)
    c[0] /= math.sqrt(2.0)
    return c, -4 * torch.sin(math.pi * k / (2 * n)) ** 2


def exact_projection(case, seed):
    F, h, walls = projection_fields(case, seed), spacing(case), case["walls_y"]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    du, dv, dw = F["dudt"], F["dvdt"], F["dwdt"]
    c = (0, 0, 0)
    div = (at(du, *c) - at(du, -1, 0, 0)) + (at(dv, *c) - at(dv, 0, -1, 0)) + (at(dw, *c) - at(dw, 0, 0, -1))
    rhs = div / (h * DT) + at(F["p_jump"], *c)

    def ring(n):
        return -4 * torch.sin(math.pi * torch.arange(n, dtype=torch.float64, device="cuda") / n) ** 2

    C, ez = cosines(nz)
    f = torch.einsum("ak,kji->aji", C, rhs)
    f = torch.fft.fft(f, dim=2)
    if walls:
        D, ey = cosines(ny)
        f = torch.einsum("bj,aji->abi", D.to(f.dtype), f)
    else:
        f, ey = torch.fft.fft(f, dim=1), ring(ny)
    lam = ez[:, None, None] + ey[None, :, None] + ring(nx)[None, None, :]
    lam[0, 0, 0] = 1.0
    f = f * (h * h) / lam
    f[0, 0, 0] = 0.0
    f = torch.einsum("bj,abi->aji", D.to(f.dtype), f) if walls else torch.fft.ifft(f, dim=1)
    p = torch.einsum("ak,aji->kji", C, torch.fft.ifft(f, dim=2).real)
    # the mean mode, whose last value the elimination sets to zero: along z, or along y between walls
    line = rhs.mean(dim=(0, 2)) if walls else rhs.mean(dim=(1, 2))
    own = p.mean(dim=(0, 2)) if walls else p.mean(dim=(1, 2))
    grad = torch.cumsum(line, 0)[:-1] * h * h
    mode = -torch.cat([torch.flip(torch.cumsum(torch.flip(grad, [0]), 0), [0]), torch.zeros_like(grad[:1])])
    shift = mode - own
    p = p + (shift[None, :, None] if walls else shift[:, None, None])
    full = halo(p, "p")
    if walls:
        full[:, 0], full[:, -1] = full[:, 1], full[:, -2]
    out = dict(p=p)
    for n, d, g, e in (("u", du, F["p_x"], (1, 0, 0)), ("v", dv, F["p_y"], (0, 1, 0)), ("w", dw, F["p_z"], (0, 0, 1))):
        f = at(d, *c) - DT / h * ((at(full, *e) - p) - at(g, *c))
        if n == "w":
            f[-1] = 0.0
        if n == "v" and walls:
            f[:, -1] = 0.0
        b = halo(f, "w" if n == "w" else "t")
        if n == "v" and walls:
            b[:, 0] = 0.0
        out[n] = f
        out[n + "cc"] = 0.5 * (f + at(b, *(-x for x in e)))
    norm = full[1].sum() / (nx * ny)
    out["pnew"] = p - norm
    out["pold"] = at(F["pnew"], *c) - norm
    return out


def houc5(f, v, axis, h):
    s = lambda d: f.roll(-d, axis)  # noqa: E731
    pos = (-2 * s(-3) + 15 * s(-2) - 60 * s(-1) + 20 * f + 30 * s(1) - 3 * s(2)) / 60
    neg = (2 * s(3) - 15 * s(2) + 60 * s(1) - 20 * f - 30 * s(-1) + 3 * s(-2)) / 60
    return torch.where(v >= 0, pos, neg) / h


def weno5(v1, v2, v3, v4, v5):
    s1 = 13 / 12 * (v1 - 2 * v2 + v3) ** 2 + 0.25 * (v1 - 4 * v2 + 3 * v3) ** 2
    s2 = 13 / 12 * (v2 - 2 * v3 + v4) ** 2 + 0.25 * (v2 - v4) ** 2
    s3 = 13 / 12 * (v3 - 2 * v4 + v5) ** 2 + 0.25 * (3 * v3 - 4 * v4 + v5) ** 2
    a1, a2, a3 = 0.1 / (1e-6 + s1) ** 2, 0.6 / (1e-6 + s2) ** 2, 0.3 / (1e-6 + s3) ** 2
    return (a1 * (v1 / 3 - 7 / 6 * v2 + 11 / 6 * v3) + a2 * (-v2 / 6 + 5 / 6 * v3 + v4 / 3) +
            a3 * (v3 / 3 + 5 / 6 * v4 - v5 / 6)) / (a1 + a2 + a3)


def one_sided(f, axis, h):
    """the WENO5 derivatives from the left and from the right"""
    d = [(f.roll(-q, axis) - f.roll(1 - q, axis)) / h for q in range(-2, 4)]
    return weno5(*d[:5]), weno5(d[5], d[4], d[3], d[2], d[1])


def advected(case, f0, vel, h):
    """one step of the drop's level set: clip to six spacings, band, RK3 transport"""
    nb = 6 * h
    f0 = torch.clamp(f0, -nb, nb)
    inside = f0.abs() != nb
    band = inside.clone()
    for axis in range(3):
        for d in (-2, -1, 1, 2):
            band |= inside.roll(d, axis)

    def rhs(f):
        g = 0
        for v, axis in zip(vel, (2, 1, 0)):
            if case.get("scheme") == "weno5":
                l, r = one_sided(f, axis, h)
                g = g - v * torch.where(v >= 0, l, r)
            else:
                g = g - v * houc5(f, v, axis, h)
        return g * band

    a = f0 + DT * rhs(f0)
    b = 0.75 * f0 + 0.25 * (a + DT * rhs(a))
    return f0 / 3 + 2 / 3 * (b + DT * rhs(b))


def reinitialised(f0, h):
    nb, dtau = 6 * h, 0.5 * h
    sgn = torch.where(f0 < -h, -1.0, torch.where(f0 > h, 1.0, f0 / torch.sqrt(f0 * f0 + h * h)))

    def rhs(f):
        g = 0
        for axis in range(3):
            l, r = one_sided(f, axis, h)
            d = torch.where((r * sgn < 0) & ((l + r) * sgn < 0), r,
                            torch.where((l * sgn > 0) & ((l + r) * sgn > 0), l, 0.5 * (l + r)))
            g = g + d * d
        return torch.where(f.abs() < nb + h, sgn * (1 - torch.sqrt(g)), torch.zeros_like(g))

    a = f0 + dtau * rhs(f0)
    b = 0.75 * f0 + 0.25 * (a + dtau * rhs(a))
    return f0 / 3 + 2 / 3 * (b + dtau * rhs(b))


def exact_levelset(case, seed):
    h = spacing(case)
    vel = [cell_velocity(case, seed)[n] for n in ("ucc", "vcc", "wcc")]
    jie = torch.ones(case["nz"], case["ny"], case["nx"], dtype=torch.float64, device="cuda")
    out = {}
    for l, drop in enumerate(placed(case, seed)):
        f = advected(case, drop_field(case, drop), vel, h)
        if case["reinit"]:
            f = reinitialised(f, h)
        if l < 12:
            out["lvset_%d" % (l + 1)] = f
        e = 1.5 * h
        g = torch.clamp(f, -e, e)
        H = 0.5 + 0.5 * g / e + 0.5 / math.pi * torch.sin(math.pi * g / e)
        jie = torch.minimum(jie, torch.where(f < -e, 0.0, torch.where(f < e, H, 1.0)))
    out["jiemian"] = jie
    out["miu"] = jie + MIU2 * (1 - jie)
    out["rho"] = rho = jie + RHO2 * (1 - jie)
    out["rho_u"], out["rho_v"] = 0.5 * (rho + rho.roll(-1, 2)), 0.5 * (rho + rho.roll(-1, 1))
    out["rho_w"] = 0.5 * (rho + torch.cat([rho[1:], rho[-1:]]))
    return out


def exact_interface(case, seed):
    h, nondi = spacing(case), 0.5
    offs = [(di, dj, dk) for dk in (-1, 0, 1) for dj in (-1, 0, 1) for di in (-1, 0, 1)]
    A = np.array([[1, x, y, z, x * x / 2, y * y / 2, z * z / 2, x * y, x * z, y * z] for x, y, z in
                  (tuple(h * v for v in o) for o in offs)])
    P = np.linalg.pinv(A)
    zero = lambda: torch.zeros(case["nz"], case["ny"], case["nx"], dtype=torch.float64, device="cuda")  # noqa: E731
    out = {n: zero() for n in ("p_x", "p_y", "p_z", "p_jump")}

    def near(f, o):
        return f.roll((-o[2], -o[1], -o[0]), (0, 1, 2))

    for drop in placed(case, seed):
        f = drop_field(case, drop)
        x = [0] * 10
        for q, o in enumerate(offs):
            g = near(f, o)
            for r in range(1, 10):
                x[r] = x[r] + P[r, q] * g
        n2 = x[1] ** 2 + x[2] ** 2 + x[3] ** 2
        m = torch.sqrt(n2)
        cv = -((x[4] + x[5] + x[6]) / m - (x[1] ** 2 * x[4] + x[2] ** 2 * x[5] + x[3] ** 2 * x[6]) / m ** 3 -
               2 * (x[1] * x[2] * x[7] + x[1] * x[3] * x[8] + x[2] * x[3] * x[9]) / m ** 3)
        cv = torch.clamp(torch.where(m < 0.9, torch.zeros_like(cv), cv), -1 / h, 1 / h)
        cv = torch.where((f.abs() <= 5 * h) & (cv.abs() >= 1e-9), cv, torch.zeros_like(cv))
        re = sum(P[0, q] * near(cv, o) for q, o in enumerate(offs))
        cv = torch.where(f.abs() < 2 * h, re, torch.zeros_like(re))
        shell, lap = f.abs() <= 2 * h, zero()
        for name, e in (("p_x", (1, 0, 0)), ("p_y", (0, 1, 0)), ("p_z", (0, 0, 1))):
            for side in (-1, 1):
                o = tuple(side * v for v in e)
                fn, cn = near(f, o), near(cv, o)
                cut = (f * fn < 0) & (cv * cn > 0) & shell
                k = (fn * cv - f * cn) / torch.where(cut, fn - f, torch.ones_like(f))
                j = torch.where(cut, -nondi * k * torch.sign(f), torch.zeros_like(k))
                lap += j / (h * h)
                if side == 1:
                    out[name] += j
        out["p_jump"] += lap
    return out


def exact_mlp_grad(case, seed):
    x, label = samples(case, seed)
    theta = torch.tensor(network(seed, out=1.0), dtype=torch.float64, device="cuda", requires_grad=True)
    cut = torch.split(theta, [128 * 32, 128, 128 * 128, 128, 64 * 128, 64, 64, 1])
    a = torch.nn.functional.silu(x.double() @ cut[0].view(128, 32).T + cut[1])
    a = torch.nn.functional.silu(a @ cut[2].view(128, 128).T + cut[3])
    a = torch.nn.functional.silu(a @ cut[4].view(64, 128).T + cut[5])
    d = a @ cut[6] + cut[7] - label.double()
    sq = (d * d).sum()
    grad, = torch.autograd.grad(0.5 * (2.0 / case["n"]) * sq, theta)
    return dict(grad=grad, loss=sq.detach())


def exact(case, seed):
    """What run() returns for these inputs, in 64 bits.  None for whole steps, whose twenty iterations over
    48 drops take too long this way."""
    by = dict(momentum=exact_momentum, projection=exact_projection, levelset=exact_levelset,
              interface=exact_interface, mlp_grad=exact_mlp_grad)
    if case["kind"] not in by:
        return None
    return {n: v.cpu().numpy() for n, v in by[case["kind"]](case, seed).items()}
