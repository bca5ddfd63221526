"""The work that a user of this framework has it do, as cases to time and to compare.

A case is a dict of plain values; ``kind`` says which part of the framework it
goes through:

* ``lattice``: one two-phase lattice, ``Lattice.step(n)`` (the loop body of the
  reference's scripts, ``n`` iterations), in each storage type, from the size of
  a unit test to the 4096 x 2048 lattice of the benchmark;
* ``ensemble``: many lattices of mixed sizes advanced together (``Ensemble.step``);
* ``frames``: the surrogate's training data, ``jump`` batched iterations and
  then one frame of every member (``generate_trajectories``' inner loop);
* ``loop``: the reference's own loop body, one call per function, on the
  drop-in ``Compute`` object in FP64;
* ``train``: one training step of the surrogate (loss, gradients, AdamW);
* ``predict``: one jump of the surrogate.

``exact`` restates the lattice iteration and the network in plain torch in
64 bits.
"""
import copy
import functools
import math

import numpy as np
import torch

from fingering_dynamics_gb300 import fingering, fingering_periodic
from fingering_dynamics_gb300 import geometry as geo
from fingering_dynamics_gb300.bounce_back import Bounce_back
from fingering_dynamics_gb300.create_block import Createblock
from fingering_dynamics_gb300.ensemble import Ensemble, ensemble_specs
from fingering_dynamics_gb300.lattice import Lattice
from fingering_dynamics_gb300.params import from_relaxation_times, periodic_reference_params, walls_reference_params
from fingering_dynamics_gb300.surrogate import UNet, member_frame

SIZES_W, SIZES_H = (256, 512, 1024, 2048), (128, 256, 512)  # the ensemble's members
WIDTHS = (32, 64, 128, 256)                                 # the surrogate's channel counts
BYTES_PER_CELL = {"f64": 144, "f32": 72, "f16": 38, "bf16": 38}
FLOPS_PER_CELL = 420                                        # one iteration of a fluid cell, divisions counted once
ON_CHIP_BYTES = 100e6                                       # a state below this stays in L2 from one iteration to the next


def listed():
    return [
        # the smallest call: a unit-test or calibration lattice, where launches and latency count
        lattice("small_f32_64x128", "f32", "periodic", 64, 128, 50),
        # the reference's own periodic script, size and defaults (FP64, 400 x 400)
        lattice("reference_f64_400x400", "f64", "periodic", 400, 400, 25),
        # the reference's walled script (380 x 380: a width that is not a multiple of 8) in FP32
        lattice("reference_f32_380x380", "f32", "walls", 380, 380, 50),
        # an exact-parity run of a large porous medium
        lattice("porous_f64_1024x2048", "f64", "walls", 1024, 2048, 10),
        # a ragged size in the other 16-bit type
        lattice("ragged_bf16_1021x1500", "bf16", "walls", 1021, 1500, 50),
        # the benchmark's lattice in the two storage types that production runs use
        lattice("bench_f32_2048x4096", "f32", "walls", 2048, 4096, 50),
        lattice("bench_f16_2048x4096", "f16", "walls", 2048, 4096, 50),
        # a parameter study: members of mixed sizes and parameters in one batch
        {"name": "ensemble_f32_24", "kind": "ensemble", "dtype": "f32", "members": 24, "steps": 50, "layout": 2024},
        # training data for the surrogate: 200 iterations, then a frame of every member
        {"name": "frames_f32_8", "kind": "frames", "dtype": "f32", "members": 8, "H": 256, "W": 512, "jump": 200,
         "layout": 1},
        # the reference's driver code, unchanged, on the drop-in modules
        {"name": "loop_f64_400x400", "kind": "loop", "variant": "periodic", "H": 400, "W": 400, "layout": 2024},
        # the surrogate: a training step at the training batch size, one jump of a single lattice (the rollout);
        # conv="tma" is the choice that makes a training run reproducible, "auto" is the default
        {"name": "train_b32_256x512", "kind": "train", "conv": "tma", "batch": 32, "H": 256, "W": 512},
        {"name": "predict_b1_256x512", "kind": "predict", "conv": "auto", "batch": 1, "H": 256, "W": 512},
    ]


def lattice(name, dtype, variant, H, W, steps):
    c = {"kind": "lattice", "dtype": dtype, "variant": variant, "H": H, "W": W, "steps": steps, "layout": 2024}
    return c if name is None else {"name": name, **c}


def draw(rng):
    kind = rng.choice(("lattice",) * 6 + ("ensemble", "frames", "loop", "train", "predict", "predict"))
    if kind == "lattice":
        dtype = rng.choice(("f64", "f32", "f32", "f16", "bf16"))
        variant = rng.choice(("walls", "walls", "periodic"))
        step = rng.choice((4, 8, 8))                                # widths that are multiples of 4, of 8
        H, W = log_int(rng, 48, 2048, 1), log_int(rng, 64, 4096, step)
        if variant == "periodic":
            H += H % 2                                              # the Gaussian inlet needs an even height
        if dtype == "f64":
            W = min(W, 2 * 1024 * 1024 // H // 4 * 4)
        cells = H * W
        steps = max(4, min(50, int((4e8 if dtype != "f64" else 2e7) / cells)))
        return lattice(None, dtype, variant, H, W, steps)
    if kind == "ensemble":
        return {"kind": kind, "dtype": rng.choice(("f32", "f32", "f16", "bf16")), "members": log_int(rng, 4, 24, 1),
                "steps": rng.randrange(20, 51), "layout": rng.randrange(1 << 20)}
    if kind == "frames":
        return {"kind": kind, "dtype": rng.choice(("f32", "f16")), "members": log_int(rng, 1, 16, 1),
                "H": rng.randrange(8, 17) * 16, "W": rng.randrange(16, 65) * 8, "jump": rng.randrange(20, 101),
                "layout": rng.randrange(1 << 20)}
    if kind == "loop":
        H = log_int(rng, 64, 400, 2)
        return {"kind": kind, "variant": rng.choice(("periodic", "walls")), "H": H, "W": log_int(rng, 80, 400, 4),
                "layout": rng.randrange(1 << 20)}
    wide = rng.random() < 0.6                                       # widths that are multiples of 128, or of 8 only
    H = rng.randrange(8, 33) * 8
    W = rng.randrange(1, 5) * 128 if wide else rng.randrange(8, 65) * 8
    return {"kind": kind, "conv": "tma" if kind == "train" else rng.choice(("auto", "tma")),
            "batch": log_int(rng, 1, 16 if kind == "train" else 32, 1), "H": H, "W": W}


def log_int(rng, lo, hi, step):
    """A multiple of `step` in [lo, hi], uniform over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=32)
def medium(variant, H, W, layout):
    """(parameters, geometry) of one lattice; the medium belongs to the case, its state to the seed."""
    if variant == "periodic":
        prm = periodic_reference_params().with_size(H, W)           # fingering_periodic.py's constants
        prm.M = 4.0
        r = max(2, min(10, H // 10))
        _, circles = geo.random_blocks(H, W, 0.85, max(2, r // 2), r, layout, kinds=("circle",), x_margin=8)
        return prm, geo.build_geometry(H, W, circles=circles)
    if H * W >= 1 << 20:                                            # the benchmark's workload
        prm = from_relaxation_times(H, W, tau_inv=0.6, tau_def=1.0, sigma=5e-4, contact_angle_deg=120.0, u_in=0.01)
        porosity, rmin, rmax = 0.7, 6, 14
    else:                                                           # fingering.py's constants
        prm = walls_reference_params().with_size(H, W)
        prm.M, prm.u0 = 3.0, 0.006
        prm.inlet_ux = np.full(H, prm.u0)
        porosity, rmax = 0.78, max(3, min(14, H // 12))
        rmin = min(6, rmax)
    rects, circles = geo.random_blocks(H, W, porosity, rmin, rmax, layout, x_margin=min(32, W // 8))
    return prm, geo.build_geometry(H, W, rects=rects, circles=circles, walls=True)


@functools.lru_cache(maxsize=8)
def members(kind, count, H, W, layout):
    sizes = dict(sizes_h=(H,), sizes_w=(W,)) if kind == "frames" else dict(sizes_h=SIZES_H, sizes_w=SIZES_W)
    return [s.build() for s in ensemble_specs(count, layout, u_in=(0.003, 0.006), **sizes)]


def start(prm, g, seed):
    """The order parameter and density that a run starts from: invading fluid up to a wavy front, density near 1."""
    rng = np.random.default_rng(seed)
    y = np.arange(prm.H)[:, None] * (2 * math.pi / prm.H)
    front = 8 + prm.W * 0.02 + sum(rng.uniform(0.3, 1.5) * np.sin(k * y + rng.uniform(0, 6.28)) for k in (1, 2, 3, 5))
    psi = np.tanh((front - np.arange(prm.W)[None, :]) / 2.0)
    psi[:, :prm.slab] = 1.0
    psi[g.solid] = prm.psi_wall
    return psi, 1.0 + 1e-3 * rng.standard_normal((prm.H, 1)) * np.ones((1, prm.W))


def loop_setup(c, seed):
    """The reference's module, the globals its user sets (the inlet speed and the wettability differ from run to
    run), and the obstacles."""
    H, W = c["H"], c["W"]
    mod = fingering if c["variant"] == "walls" else fingering_periodic
    prm = (walls_reference_params if c["variant"] == "walls" else periodic_reference_params)().with_size(H, W)
    rng = np.random.default_rng(seed)
    values = dict(H=H, W=W, M=4.0, u0=prm.u0 if c["variant"] == "periodic" else 0.006, tau=prm.tau, Eta_n=prm.eta_n,
                  a=prm.a, kappa=prm.kappa, gamma=prm.gamma, psi_wall=float(rng.uniform(-0.7, -0.3)))
    values["u0"] = float(values["u0"] * rng.uniform(0.5, 1.0))
    r = max(3, H // 20)
    rects, circles = geo.random_blocks(H, W, 0.9, 2, r, c["layout"], x_margin=10,
                                       kinds=("circle",) if c["variant"] == "periodic" else ("square",))
    return mod, values, rects, circles


def weights(seed, device="cpu"):
    """A network some steps into its training: He-initialised layers, a small output layer."""
    rng = np.random.default_rng(seed)
    c1, c2, c3, c4 = WIDTHS
    shapes = {"enc1a": (16, c1), "enc1b": (c1, c1), "enc2a": (c1, c2), "enc2b": (c2, c2), "enc3a": (c2, c3),
              "enc3b": (c3, c3), "enc4a": (c3, c4), "enc4b": (c4, c4), "dec3a": (c4 + c3, c3), "dec3b": (c3, c3),
              "dec2a": (c3 + c2, c2), "dec2b": (c2, c2), "dec1a": (c2 + c1, c1), "dec1b": (c1, c1), "out": (c1, 16)}
    p = {}
    for name, (ci, co) in shapes.items():
        std = math.sqrt(2.0 / (9 * ci)) * (0.05 if name == "out" else 1.0)
        p[name + ".w"] = rng.standard_normal((co, 3, 3, ci), dtype=np.float32) * np.float32(std)
        p[name + ".b"] = rng.standard_normal(co, dtype=np.float32) * np.float32(0.02)
    return p


def pair(c, seed):
    """A batch of frames and of the frames one jump later: (psi, u_x, u_y, solid) and twelve zero channels."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    N, H, W = c["batch"], c["H"], c["W"]

    def smooth(ch):
        low = torch.randn((N, ch, H // 8, W // 8), generator=g, device="cuda")
        return torch.nn.functional.interpolate(low, size=(H, W), mode="bilinear", align_corners=False)

    solid = (smooth(1) > 0.6).float()
    x = torch.cat([torch.tanh(4 * smooth(1)), 0.5 * smooth(2) * (1 - solid), solid], dim=1)
    xn = x.clone()
    xn[:, :3] += 0.2 * smooth(3) * (1 - solid)
    out = []
    for v in (x, xn):
        fr = torch.zeros((N, H, W, 16), dtype=torch.bfloat16, device="cuda")
        fr[..., :4] = v.permute(0, 2, 3, 1).to(torch.bfloat16)
        out.append(fr)
    return out


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "lattice":
        prm, g = medium(c["variant"], c["H"], c["W"], c["layout"])
        psi0, rho0 = start(prm, g, seed)
        return c, Lattice(prm, g, dtype=c["dtype"], psi0=psi0, rho0=rho0, seed=seed)
    if kind in ("ensemble", "frames"):
        made = members(kind, c["members"], c.get("H", 0), c.get("W", 0), c["layout"])
        ens = Ensemble([(p, g, start(p, g, seed + k)[0]) for k, (p, g) in enumerate(made)], dtype=c["dtype"])
        if kind == "ensemble":
            return c, ens
        return c, ens, torch.empty((c["members"], c["H"], c["W"], 4), dtype=torch.bfloat16, device="cuda")
    if kind == "loop":
        mod, values, rects, circles = loop_setup(c, seed)
        for k, v in values.items():
            setattr(mod, k, v)
        cb = Createblock(c["H"], c["W"])
        lists, corners = None, []
        if circles:
            blocks, *lists = cb.setCirleblock(circles)
        else:
            blocks, corners = cb.setblock(rects)
        mask = blocks != 1
        np.random.seed(seed)
        return c, mod, values, mod.Compute(mask), mask, Bounce_back(c["H"], c["W"]), lists, corners
    net = UNet(WIDTHS, params=weights(seed), conv=c["conv"])
    return (c, net, *pair(c, seed))


def run(state):
    kind = state[0]["kind"]
    if kind == "lattice":
        c, lat = state
        lat.step(c["steps"])
        return {"f": lat.f, "g": lat.g, "psi": lat.psi, "ux": lat.ux, "uy": lat.uy, "rho": lat.rho}
    if kind == "ensemble":
        c, ens = state
        ens.step(c["steps"])
        return [planes(lat) for lat in ens.lattices]
    if kind == "frames":
        c, ens, out = state
        ens.step(c["jump"])
        for m, lat in enumerate(ens.lattices):
            out[m] = member_frame(lat)[..., :4]
        return {"frames": out, "state": [planes(lat) for lat in ens.lattices]}
    if kind == "loop":
        return loop_body(*state[1:])
    c, net, x, xn = state
    if kind == "train":
        loss = net.loss_grad(x, xn)
        net.adamw(lr=1e-4)
        return {"loss": loss, "w": dict(net.gw), "b": dict(net.gb)}
    return net.predict(x)


def planes(lat):
    """A member's state: its packed planes in their type (a member's cells fill whole 256-byte units, so there is
    no padding between them)."""
    buf = lat.current_buffer()
    if lat.dtype == "f32":
        return buf.view(torch.float32)
    t = torch.float16 if lat.dtype == "f16" else torch.bfloat16
    P = lat.H * lat.W
    return {"f": buf[:18 * P].view(t), "g0": buf[18 * P:22 * P].view(torch.float32), "g": buf[22 * P:].view(t)}


def loop_body(mod, values, cm, mask, bb, lists, corners):
    """One iteration as the reference's scripts write it (fingering_periodic.py:454-479, fingering.py:558-585)."""
    mod.u0 = values["u0"]
    for j in range(9):
        cm.F[j] = cm.getLarge_F(j)
        cm.feq[j] = cm.getfeq(j)
        cm.geq[j] = cm.getgeq(j)
        cm.f[j][mask] = cm.getF(j)
        cm.g[j][mask] = cm.getG(j)
    f_behind, g_behind = copy.deepcopy(cm.f), copy.deepcopy(cm.g)
    mod.stream(cm.f, cm.g)
    if lists is not None:
        bb.halfway_bounceback_circle(*lists, f_behind, g_behind, cm.f, cm.g)
    if corners:
        bb.halfway_bounceback_rec(corners, f_behind, g_behind, cm.f, cm.g)
    if mod is fingering:
        mod.bottom_top_wall(f_behind[:, 1:-1], g_behind[:, 1:-1], cm.f[:, 1:-1], cm.g[:, 1:-1])
    cm.zou_he_boundary_inlet()
    cm.zou_he_boundary_outlet()
    cm.rho = cm.getRho()
    cm.udpatePsi()
    cm.nabla_psix = cm.getNabla_psix()
    cm.nabla_psiy = cm.getNabla_psiy()
    cm.nabla_psi2 = cm.getNabla_psi2()
    cm.mu = cm.getMu()
    cm.ux = cm.getUx()
    cm.uy = cm.getUy()
    cm.p = cm.getP()
    cm.mix_tau = cm.getMix_tau()
    return {"f": cm.f, "g": cm.g, "psi": cm.psi, "F": cm.F, "feq": cm.feq, "geq": cm.geq, "rho": cm.rho, "ux": cm.ux,
            "uy": cm.uy, "p": cm.p, "mu": cm.mu, "mix_tau": cm.mix_tau}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    c, kind = case, case["kind"]
    if kind in ("lattice", "ensemble", "frames", "loop"):
        if kind == "lattice":
            cells, steps, per = c["H"] * c["W"], c["steps"], BYTES_PER_CELL[c["dtype"]]
            extra = cells * 24 * (8 if c["dtype"] == "f64" else 4)  # the state and the fields in the reference's layout
        elif kind == "ensemble":
            cells = sum(p.H * p.W for p, _ in members(kind, c["members"], 0, 0, c["layout"]))
            steps, per, extra = c["steps"], BYTES_PER_CELL[c["dtype"]], 0
        elif kind == "frames":
            cells, steps, per = c["members"] * c["H"] * c["W"], c["jump"], BYTES_PER_CELL[c["dtype"]]
            extra = cells * (per + 8)
        else:
            cells, steps, per, extra = c["H"] * c["W"], 1, 144, c["H"] * c["W"] * 8 * 33
        passes = steps if 2 * cells * per > ON_CHIP_BYTES else 1
        return {"bytes": 2.0 * cells * per * passes + extra, "flops": float(FLOPS_PER_CELL) * cells * steps}
    c1, c2, c3, c4 = WIDTHS
    P = c["batch"] * c["H"] * c["W"]
    layers = [(16, c1, 1), (c1, c1, 1), (c1, c2, 4), (c2, c2, 4), (c2, c3, 16), (c3, c3, 16), (c3, c4, 64), (c4, c4, 64),
              (c4 + c3, c3, 16), (c3, c3, 16), (c3 + c2, c2, 4), (c2, c2, 4), (c2 + c1, c1, 1), (c1, c1, 1), (c1, 16, 1)]
    params = sum(9 * ci * co + co for ci, co, _ in layers)
    flops = sum(18.0 * ci * co * P / d for ci, co, d in layers)
    acts = sum(co * P / d for _, co, d in layers)
    if kind == "predict":
        return {"bytes": 2.0 * 32 * P + 2.0 * params, "flops": flops}
    # forward, data gradient (not of the first layer), weight gradient; each layer's output kept for the backward
    first = 18.0 * 16 * c1 * P
    return {"bytes": 2.0 * 2 * acts + 2.0 * 32 * P + 30.0 * params, "flops": 3 * flops - first}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
EX = (0, 1, 0, -1, 0, 1, -1, -1, 1)
EY = (0, 0, 1, 0, -1, 1, 1, -1, -1)
OPP = (0, 3, 4, 1, 2, 7, 8, 5, 6)
WGT = (4 / 9, 1 / 9, 1 / 9, 1 / 9, 1 / 9, 1 / 36, 1 / 36, 1 / 36, 1 / 36)


class Exact:
    """One lattice of the two-phase model in 64 bits (the reference's loop body)."""

    def __init__(self, prm, word, psi0, rho0):
        dev = torch.device("cuda")
        w = torch.from_numpy(np.ascontiguousarray(word).astype(np.int32)).to(dev)
        self.p, self.walls = prm, prm.variant == "walls"
        self.solid = (w & 256) != 0
        self.fluid = ~self.solid
        self.link = [None] + [((w >> (i - 1)) & 1) != 0 for i in range(1, 9)]
        self.uin = torch.from_numpy(np.asarray(prm.inlet_ux, np.float64)).to(dev)
        self.psi = torch.from_numpy(np.ascontiguousarray(psi0)).to(dev).double()
        self.psi[self.solid] = prm.psi_wall
        self.rho = torch.from_numpy(np.ascontiguousarray(rho0)).to(dev).double()
        self.ux, self.uy = torch.zeros_like(self.psi), torch.zeros_like(self.psi)
        self.stencil()
        mu = self.mu_of()
        self.mu = mu if prm.init_mu else torch.zeros_like(mu)
        if prm.init_uy:
            self.uy = self.mu * self.gy / 2 / self.rho
        self.tau_of()
        self.P = self.rho / 3  # the pressure is taken before mu is
        zero = torch.zeros_like(self.psi)
        both = [self.equilibrium(i) for i in range(9)]
        self.f = torch.stack([torch.where(self.fluid, a, zero) for a, _ in both])
        self.g = torch.stack([torch.where(self.fluid, b, zero) for _, b in both])

    def stencil(self):
        t = torch.nn.functional.pad(self.psi[None, None], (1, 1, 1, 1))[0, 0]
        t[1:-1, 0], t[1:-1, -1] = 1.0, -1.0
        if self.walls:
            t[0], t[-1] = self.p.psi_wall, self.p.psi_wall
        else:
            t[0], t[-1] = t[-2].clone(), t[1].clone()
        C, E, W, N, S = t[1:-1, 1:-1], t[1:-1, 2:], t[1:-1, :-2], t[2:, 1:-1], t[:-2, 1:-1]
        NE, NW, SE, SW = t[2:, 2:], t[2:, :-2], t[:-2, 2:], t[:-2, :-2]
        self.gx = (4 * (E - W) + NE - NW - SW + SE) / 12
        self.gy = (4 * (N - S) + NE + NW - SW - SE) / 12
        self.lap = (-20 * C + 4 * (N + E + W + S) + NE + NW + SW + SE) / 6

    def mu_of(self):
        return self.p.a * self.psi * (1 - self.psi ** 2) - self.p.kappa * self.lap

    def tau_of(self):
        v1, v2 = self.p.eta_n / self.rho, self.p.eta_n * self.p.M / self.rho
        self.tau = 3 * (2 * v1 * v2 / (v1 * (1 - self.psi) + v2 * (1 + self.psi))) + 0.5

    def equilibrium(self, i):
        eu = EX[i] * self.ux + EY[i] * self.uy
        q = 3 * eu + 4.5 * eu * eu - 1.5 * (self.ux ** 2 + self.uy ** 2)
        if i == 0:
            k = 3 * (1 - WGT[0])
            A, B = (self.rho - k * self.P) / WGT[0], (self.psi - k * self.p.gamma * self.mu) / WGT[0]
        else:
            A, B = 3 * self.P, 3 * self.p.gamma * self.mu
        return WGT[i] * (A + self.rho * q), WGT[i] * (B + self.psi * q)

    def force(self, i):
        eu = EX[i] * self.ux + EY[i] * self.uy
        ax, ay = 3 * (EX[i] - self.ux) + 9 * EX[i] * eu, 3 * (EY[i] - self.uy) + 9 * EY[i] * eu
        return self.mu * WGT[i] * (1 - 1 / (2 * self.tau)) * (ax * self.gx + ay * self.gy)

    def collide(self):
        for i in range(9):
            feq, geq = self.equilibrium(i)
            f, g = self.f[i], self.g[i]
            self.f[i] = torch.where(self.fluid, f - (f - feq) / self.tau + self.force(i), f)
            self.g[i] = torch.where(self.fluid, g - (g - geq) / self.p.tau, g)

    def finish(self):
        for name in ("f", "g"):
            b = getattr(self, name)
            n = torch.stack([torch.roll(b[i], (EY[i], EX[i]), (0, 1)) for i in range(9)])
            for i in range(1, 9):
                n[i] = torch.where(self.link[i], b[OPP[i]], n[i])
            setattr(self, name, n)
        self.inlet()
        self.outlet()
        self.rho = torch.where(self.fluid, self.f.sum(0), self.rho)
        self.psi = torch.where(self.fluid, self.g.sum(0), self.psi)
        self.stencil()
        self.mu = self.mu_of()
        jx, jy = sum(EX[i] * self.f[i] for i in range(9)), sum(EY[i] * self.f[i] for i in range(9))
        self.ux, self.uy = (jx + self.mu * self.gx / 2) / self.rho, (jy + self.mu * self.gy / 2) / self.rho
        self.P = self.rho / 3 + self.psi * self.mu
        self.tau_of()

    def inlet(self):
        f, g, u = self.f[:, :, 0], self.g[:, :, 0], self.uin
        px, py, m = self.gx[:, 0], self.gy[:, 0], self.mu_of()[:, 0]
        rho = (f[0] + f[2] + f[4] + 2 * (f[3] + f[6] + f[7]) - px * m / 2) / (1 - u)
        psi = 1 - (g[0] + g[2] + g[3] + g[4] + g[6] + g[7])
        f0, g0 = f.clone(), g.clone()
        f[1] = f[3] + 2 / 3 * u * rho - px * m / 6
        f[5] = f[7] - 0.5 * (f[2] - f[4]) + u * rho / 6 - px * m / 6 - py * m / 4
        f[8] = f[6] + 0.5 * (f[2] - f[4]) + u * rho / 6 - px * m / 6 + py * m / 4
        g[1], g[5], g[8] = psi * 2 / 3, psi / 6, psi / 6
        if self.walls:
            # (y, row of rho_inlet, copies to <- from, the two unknown diagonals)
            for y, n, copies, ab in ((0, 1, ((1, 3), (2, 4), (5, 7)), (6, 8)), (-1, -2, ((1, 3), (4, 2), (8, 6)), (5, 7))):
                for v, v0, total in ((f, f0, rho[n]), (g, g0, 1.0)):
                    v[:, y] = v0[:, y]
                    for to, of in copies:
                        v[to, y] = v[of, y]
                    known = sum(v[i, y] for i in range(9) if i not in ab)
                    v[ab[0], y] = 0.5 * (total - known)
                    v[ab[1], y] = v[ab[0], y]

    def outlet(self):
        f, g, u = self.f[:, :, -1], self.g[:, :, -1], self.uin
        px, py, m = self.gx[:, -1], self.gy[:, -1], self.mu_of()[:, -1]
        rho = (f[0] + f[2] + f[4] + 2 * (f[1] + f[5] + f[8]) + px * m / 2) / (1 + u)
        psi = -1 - (g[0] + g[1] + g[2] + g[4] + g[5] + g[8])
        f[3] = f[1] - self.p.outlet_coef * u * rho + px * m / 6
        f[6] = f[8] - 0.5 * (f[2] - f[4]) - u * rho / 6 + py * m / 4 + px * m / 6
        f[7] = f[5] + 0.5 * (f[2] - f[4]) - u * rho / 6 - py * m / 4 + px * m / 6
        g[3], g[6], g[7] = psi * 2 / 3, psi / 6, psi / 6
        if self.walls:
            for v in (f, g):
                v[2, 0] = v[4, 0]
                v[4, -1] = v[2, -1]

    def step(self, n):
        for _ in range(n):
            self.collide()
            self.finish()

    def at(self, name):
        """A field on fluid cells, 0 on solid ones (rho: 1)."""
        return torch.where(self.fluid, getattr(self, name), torch.zeros_like(self.psi))


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "lattice":
        prm, g = medium(c["variant"], c["H"], c["W"], c["layout"])
        e = Exact(prm, g.mask_word, *start(prm, g, seed))
        e.step(c["steps"])
        return {"f": e.f, "g": e.g, "psi": e.psi, "ux": e.at("ux"), "uy": e.at("uy"), "rho": None}
    if kind in ("ensemble", "frames"):
        frames, state = [], []
        for k, (prm, g) in enumerate(members(kind, c["members"], c.get("H", 0), c.get("W", 0), c["layout"])):
            e = Exact(prm, g.mask_word, start(prm, g, seed + k)[0], np.ones((prm.H, prm.W)))
            e.step(c["steps"] if kind == "ensemble" else c["jump"])
            # the fused state holds the populations after the collision, f as its deviation from the weights
            e.collide()
            f = torch.cat([(e.f[i] - WGT[i]).reshape(-1) for i in range(9)])
            g0, gi = e.g[0].reshape(-1), e.g[1:].reshape(-1)
            state.append(torch.cat([f, g0, gi]) if c["dtype"] == "f32" else {"f": f, "g0": g0, "g": gi})
            if kind == "frames":  # the fields of the next iteration
                e.finish()
                frames.append(torch.stack([e.psi, e.at("ux") / 0.01, e.at("uy") / 0.01, e.solid.double()], dim=-1))
        return state if kind == "ensemble" else {"frames": torch.stack(frames), "state": state}
    if kind == "loop":
        return exact_loop(c, seed)
    return exact_net(c, seed)


def exact_loop(c, seed):
    mod, values, rects, circles = loop_setup(c, seed)
    walls = c["variant"] == "walls"
    H, W = c["H"], c["W"]
    prm = (walls_reference_params if walls else periodic_reference_params)().with_size(H, W)
    prm.M, prm.psi_wall = values["M"], values["psi_wall"]
    prm.inlet_ux = np.full(H, values["u0"]) if walls else prm.inlet_ux * (values["u0"] / prm.u0)
    g = geo.build_geometry(H, W, rects=rects, circles=circles, walls=walls)
    psi0, rho0 = np.full((H, W), -1.0), np.ones((H, W))
    psi0[:, :5] = 1.0
    if walls:
        np.random.seed(seed)
        np.random.randint(0, 1, size=(H, W))
        rho0 = rho0 - np.random.rand(H, W) * 0.001
    e = Exact(prm, g.mask_word, psi0, rho0)
    m = e.fluid
    F = torch.stack([e.force(i)[m] for i in range(9)])
    both = [e.equilibrium(i) for i in range(9)]
    feq, geq = torch.stack([a[m] for a, _ in both]), torch.stack([b[m] for _, b in both])
    e.step(1)
    return {"f": e.f, "g": e.g, "psi": e.psi, "F": F, "feq": feq, "geq": geq, "rho": e.rho[m], "ux": e.ux[m],
            "uy": e.uy[m], "p": e.P[m], "mu": e.mu[m], "mix_tau": e.tau[m]}


def exact_net(c, seed):
    if c["kind"] == "train" and c["batch"] * c["H"] * c["W"] > 32 * 256 * 512:
        return None
    p = weights(seed)
    par = {}
    for k, v in p.items():
        t = torch.from_numpy(v).cuda()
        t = t.to(torch.bfloat16).double() if k.endswith(".w") else t.double()  # the weights the network multiplies by
        par[k] = t.requires_grad_(c["kind"] == "train")
    x, xn = pair(c, seed)

    def net(v):
        def conv(a, name, act=True):
            N, Ci, H, W = a.shape
            w = par[name + ".w"]
            # one product per tap: (pixels, Ci) x (Ci, Co)
            ap = torch.nn.functional.pad(a.permute(0, 2, 3, 1), (0, 0, 1, 1, 1, 1))
            z = par[name + ".b"].expand(N * H * W, -1)
            for ky in range(3):
                for kx in range(3):
                    z = z + ap[:, ky:ky + H, kx:kx + W].reshape(-1, Ci) @ w[:, ky, kx].t()
            z = z.reshape(N, H, W, -1).permute(0, 3, 1, 2)
            return torch.nn.functional.gelu(z, approximate="tanh") if act else z

        pool = lambda a: torch.nn.functional.avg_pool2d(a, 2)  # noqa: E731
        up = lambda a: torch.nn.functional.interpolate(a, scale_factor=2, mode="nearest")  # noqa: E731
        e1 = conv(conv(v, "enc1a"), "enc1b")
        e2 = conv(conv(pool(e1), "enc2a"), "enc2b")
        e3 = conv(conv(pool(e2), "enc3a"), "enc3b")
        e4 = conv(conv(pool(e3), "enc4a"), "enc4b")
        d3 = conv(conv(torch.cat([up(e4), e3], 1), "dec3a"), "dec3b")
        d2 = conv(conv(torch.cat([up(d3), e2], 1), "dec2a"), "dec2b")
        d1 = conv(conv(torch.cat([up(d2), e1], 1), "dec1a"), "dec1b")
        return conv(d1, "out", act=False)

    count = (x[..., 3] == 0).sum().double()
    total, outs = 0.0, []
    for n in range(c["batch"]):  # a frame at a time
        v = x[n:n + 1].double().permute(0, 3, 1, 2)
        pred = v[:, :3] + net(v)[:, :3]
        if c["kind"] == "predict":
            outs.append(torch.cat([pred, v[:, 3:]], 1).permute(0, 2, 3, 1))
            continue
        d = (pred - xn[n:n + 1].double().permute(0, 3, 1, 2)[:, :3]) * (v[:, 3:4] == 0)
        loss = (d * d).sum() / (3 * count)
        loss.backward()
        total = total + loss.detach()
    if c["kind"] == "predict":
        return torch.cat(outs)
    return {"loss": total, "w": {k[:-2]: par[k].grad for k in par if k.endswith(".w")},
            "b": {k[:-2]: par[k].grad for k in par if k.endswith(".b")}}
