"""The timed cases of this framework: what its users have it do, through its public entry points.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program has in hand before the call
    run(state)           one pass
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    the outputs in 64-bit arithmetic, by plain torch

Kinds of case:
    steps       a stats interval of a solve: n coupled steps, the convergence stats and the fields (Lattice)
    batch       many designs in one persistent solve (Batch)
    solve       run_simulation from host arrays to host arrays, lattice creation included
    operators   one step through the unfused operators of fluid_engine3d / thermal_engine3d
    reduce      scalar outputs and field stats of given fields (device_scalars, field_stats)
    conv        one inference convolution of the surrogate (conv_forward)
    conv_train  one training convolution, forward and backward (conv3d)
    predict     the surrogate's warm-start fields of one design (predict)
    train       the surrogate's loss and gradients on a mini-batch
"""
import functools

import numpy as np
import torch
import torch.nn.functional as F

from xadvcool_b200 import designs, fluid_engine3d, metrics, simulation, surrogate, thermal_engine3d
from xadvcool_b200.batch import Batch
from xadvcool_b200.lattice import Lattice

DEV = "cuda"
TAU, PR, K_RATIO, POWER, T_IN, RHO_OUT = 0.55, 7.0, 628.0, 0.1, 25.0, 1.0
ELEM = {"fp32": (4, 4), "fp16": (2, 2), "bf16": (2, 2), "fp32_t16": (4, 2)}  # fluid, thermal bytes per population


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the parity plate: the smallest solve, a stats interval of 100 launches on a part of the chip
        dict(name="plate64_steps", kind="steps", family="plate", nx=64, ny=32, nz=16, steps=100, precision="fp32"),
        # the benchmark design: a gyroid cold plate in the default storage
        dict(name="gyroid148_steps", kind="steps", family="gyroid", nx=148, ny=128, nz=32, steps=100,
             precision="fp32"),
        # the same design in 16-bit population storage
        dict(name="gyroid148_steps_fp16", kind="steps", family="gyroid", nx=148, ny=128, nz=32, steps=100,
             precision="fp16"),
        # a fine-grid plate of odd sizes, far larger than the L2 cache; its row length has no kernel of its own
        dict(name="ragged301_steps", kind="steps", family="straight", nx=301, ny=203, nz=61, steps=100,
             precision="fp32"),
        # a design sweep: small uneven designs, none of which fills the GPU alone
        dict(name="batch16_small", kind="batch", designs=16, nx=48, ny=24, nz=12, steps=200, precision="fp32"),
        # the drop-in call of a design study, stopped after 1500 steps: host arrays in, host arrays out
        dict(name="gyroid148_solve", kind="solve", family="gyroid", nx=148, ny=128, nz=32, steps=1500,
             precision="fp32"),
        # a caller's own time loop on the unfused operators
        dict(name="operators148", kind="operators", family="gyroid", nx=148, ny=128, nz=32),
        # scalars and stats of a small design's fields: a latency-bound call
        dict(name="plate64_reduce", kind="reduce", family="plate", nx=64, ny=32, nz=16),
        # the surrogate's full-resolution convolution at inference
        dict(name="conv16_infer", kind="conv", N=1, D=32, H=128, W=152, Ci=16, Co=16, ksize=3, act=0, fp32=False),
        # a decoder convolution in training
        dict(name="conv96_32_train", kind="conv_train", N=4, D=16, H=64, W=76, Ci=96, Co=32, ksize=3),
        # a warm start of the benchmark design: host mask to device fields
        dict(name="gyroid148_predict", kind="predict", family="gyroid", nx=148, ny=128, nz=32),
        # a training step's gradients at the study's mini-batch
        dict(name="surrogate_train4", kind="train", N=4, D=32, H=128, W=152),
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def _draw_shape(rng, most):
    while True:
        nx, ny, nz = _log_int(rng, 30, 320), _log_int(rng, 12, 220), rng.randint(9, 64)
        if 6000 <= nx * ny * nz <= most:
            return nx, ny, nz


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "batch", "solve", "operators", "reduce", "conv", "conv",
                       "conv_train", "conv_train"])
    family = rng.choice(list(designs.FAMILIES))
    precision = rng.choice(["fp32", "fp32", "fp16", "bf16", "fp32_t16"])
    if kind == "steps":
        nx, ny, nz = _draw_shape(rng, 3_700_000)
        return dict(kind=kind, family=family, nx=nx, ny=ny, nz=nz, steps=rng.randint(10, 100), precision=precision)
    if kind == "batch":
        while True:
            n, nx, ny, nz = rng.randint(2, 20), _log_int(rng, 30, 128), _log_int(rng, 12, 64), rng.randint(9, 32)
            if n * nx * ny * nz <= 1_000_000:
                break
        return dict(kind=kind, designs=n, nx=nx, ny=ny, nz=nz, steps=rng.choice([100, 150, 200]),
                    precision=precision)
    if kind == "solve":
        nx, ny, nz = _draw_shape(rng, 800_000)
        return dict(kind=kind, family=family, nx=nx, ny=ny, nz=nz, steps=rng.randint(200, 1500), precision=precision)
    if kind in ("operators", "reduce"):
        nx, ny, nz = _draw_shape(rng, 1_200_000)
        return dict(kind=kind, family=family, nx=nx, ny=ny, nz=nz)
    Ci, Co = 16 * rng.choice([1, 1, 2, 3, 4, 6, 8, 12, 16]), 16 * rng.choice([1, 1, 2, 3, 4, 8, 16])
    ksize = rng.choice([3, 3, 3, 1])
    while True:
        N, D, H, W = rng.randint(1, 4), _log_int(rng, 4, 32), _log_int(rng, 8, 128), _log_int(rng, 9, 160)
        if N * D * H * W * (27 if ksize == 3 else 1) * Ci * Co <= 4.5e10:
            break
    c = dict(kind=kind, N=N, D=D, H=H, W=W, Ci=Ci, Co=Co, ksize=ksize)
    if kind == "conv":
        c.update(act=rng.choice([0, 1]), fp32=rng.choice([False, True]))
    return c


# ------------------------------------------------------------------------------------------------ inputs
def _design(family, nx, ny, nz, seed):
    """(mask, heat source, inlet speed) of a seeded cold plate; wide enough plates have the 10-cell buffers."""
    rng = np.random.default_rng(seed)
    buf = 10 if nx >= 60 else 3
    core = nx - 2 * buf
    hot = designs.draw_hotspots(rng, core, ny)
    u_in = float(rng.uniform(0.015, 0.03))
    if family == "plate":
        return (designs.straight_fin_plate(nx, ny, nz),
                designs.floor_heat_source((nx, ny, nz), designs.hotspot_map(hot, core, ny), buf), u_in)
    spec = {"family": family, "shape": (nx, ny, nz), "buf": buf, "margin": 0, "hot": hot, "seed": seed, "u_in": u_in}
    if family == "straight":
        n = max(1, min(int(rng.integers(4, 13)), (ny - 2) // 4))
        spec.update(n=n, width=max(2, (ny - 2) // (2 * n)))
    elif family == "pin_fin":
        radius = int(rng.integers(2, 6))
        spec.update(radius=radius, pitch=int(rng.integers(max(8, 2 * radius + 2), 17)))
    else:
        spec.update(L=int(rng.integers(12, 25)), t=float(rng.uniform(-0.3, 0.3)))
    mask, heat = designs.build_from_spec(spec)
    return mask, heat, u_in


def _sizes(case, k):
    """The k-th design's size in a batch: uneven, at most 1.5 times the case's each way."""
    f = (1.0, 0.75, 1.5, 1.2)[k % 4]
    return max(24, int(case["nx"] * f)), max(9, int(case["ny"] * (1.0, 1.3)[k % 2])), max(8, case["nz"] - k % 3)


def _batch_designs(case, seed):
    out = []
    for k in range(case["designs"]):
        fam = designs.FAMILIES[k % len(designs.FAMILIES)]
        m, h, u = _design(fam, *_sizes(case, k), 1000 * seed + k)
        out.append(dict(mask=m, heat_source=h, tau_fluid=TAU, heat_power=POWER, t_inlet=T_IN, u_inlet_val=u))
    return out


def _fields(case, seed):
    """Fields of a flow in the case's design (reference layout, on the GPU): near-rest density, a streamwise
    profile with a small swirl, a heated floor."""
    mask, heat, u_in = _design(case["family"], case["nx"], case["ny"], case["nz"], seed)
    g = torch.Generator(DEV).manual_seed(seed)
    m = torch.from_numpy(mask).to(DEV)
    solid = m == 1

    def noise():
        return torch.randn(m.shape, generator=g, device=DEV)

    rho = 1.0 + 0.01 * noise()
    u = torch.stack([u_in + 0.005 * noise(), 0.003 * noise(), 0.003 * noise()], dim=-1)
    T = T_IN + 3.0 * noise().abs()
    rho[solid] = 1.0
    u[solid] = 0.0
    return m, torch.from_numpy(heat).to(DEV), u_in, rho, u.contiguous(), T


def _conv_inputs(case, seed):
    """A convolution's operands: activations as a GELU leaves them, He-scaled weights."""
    g = torch.Generator(DEV).manual_seed(seed)
    N, D, H, W, Ci, Co = (case[k] for k in ("N", "D", "H", "W", "Ci", "Co"))
    taps = 27 if case["ksize"] == 3 else 1
    x = F.gelu(torch.randn((N, D, H, W, Ci), generator=g, device=DEV)).to(torch.bfloat16)
    w = torch.randn((taps, Co, Ci), generator=g, device=DEV) * (2.0 / (taps * Ci)) ** 0.5
    b = 0.1 * torch.randn((Co,), generator=g, device=DEV)
    dy = 0.01 * torch.randn((N, D, H, W, Co), generator=g, device=DEV).to(torch.bfloat16)
    return x, w, b, dy


def _train_inputs(case, seed):
    """Features of gyroid plates and normalised targets, as the training loop hands them to the network."""
    g = torch.Generator(DEV).manual_seed(seed)
    N, D, H, W = (case[k] for k in ("N", "D", "H", "W"))
    x = torch.zeros((N, D, H, W, 16), dtype=torch.bfloat16, device=DEV)
    for k in range(N):
        m, h, u_in = _design("gyroid", 148, H, D, 100 * seed + k)
        x[k] = surrogate.features(m, h, u_in, DEV)[0]
    y = torch.randn((N, D // 4, H // 4, W // 4, surrogate.OUT_FIELDS), generator=g, device=DEV)
    y = F.interpolate(y.permute(0, 4, 1, 2, 3), size=(D, H, W), mode="trilinear").permute(0, 2, 3, 4, 1).contiguous()
    return x, y


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("steps", "solve", "predict"):
        m, h, u_in = _design(case["family"], case["nx"], case["ny"], case["nz"], seed)
        if kind == "steps":
            lat = Lattice(m, tau_fluid=TAU, heat_power=POWER, t_inlet=T_IN, u_inlet_val=u_in, heat_source=h, Pr=PR,
                          k_ratio=K_RATIO, rho_outlet=RHO_OUT, precision=case["precision"])
            return dict(case=case, lat=lat)
        if kind == "solve":
            return dict(case=case, mask=m, heat=h, u_in=u_in)
        return dict(case=case, mask=m, heat=h, u_in=u_in, model=surrogate.load_pretrained())
    if kind == "batch":
        return dict(case=case, batch=Batch(_batch_designs(case, seed), precision=case["precision"]))
    if kind in ("operators", "reduce"):
        m, h, u_in, rho, u, T = _fields(case, seed)
        s = dict(case=case, mask=m, u_in=u_in, rho=rho, u=u, T=T)
        if kind == "operators":
            s["heat"] = (h / h.max()).contiguous()
            s["inlet"] = torch.tensor([u_in], dtype=torch.float32, device=DEV)
            f = [torch.empty((19,) + tuple(m.shape), device=DEV) for _ in range(4)]
            s["f"], s["f_post"], s["g"], s["g_post"] = f
            fluid_engine3d.compute_equilibrium_kernel(rho, u, s["f"])
            thermal_engine3d.compute_thermal_equilibrium_kernel(rho, u, T, s["g"], m)
        return s
    if kind in ("conv", "conv_train"):
        x, w, b, dy = _conv_inputs(case, seed)
        if kind == "conv":
            return dict(case=case, x=x, w=w.to(torch.bfloat16), b=b)
        return dict(case=case, x=x.requires_grad_(), w=w.requires_grad_(), b=b.requires_grad_(), dy=dy)
    x, y = _train_inputs(case, seed)
    return dict(case=case, x=x, y=y, model=surrogate.load_pretrained())


# ------------------------------------------------------------------------------------------------ passes
def _run_steps(s):
    lat = s["lat"]
    lat.step(s["case"]["steps"])
    stats = lat.stats()
    rho, u, T = lat.fields()
    return dict(stats=stats, rho=rho, u=u, T=T)


def _run_batch(s):
    b, steps = s["batch"], s["case"]["steps"]
    for i in range(len(b)):
        b.lattice(i).init_fields()
    res = b.run(max_steps=steps, stats_every=100, tol_ke=0.0, tol_T=0.0)
    return dict(steps=[r["steps"] for r in res], fields=[b.lattice(i).fields() for i in range(len(b))])


def _run_solve(s):
    c = s["case"]
    r = simulation.run_simulation(s["mask"], max_steps=c["steps"], tau_fluid=TAU, heat_power=POWER, t_inlet=T_IN,
                                  u_inlet_val=s["u_in"], tol_ke=0.0, tol_T=0.0, silent=True, heat_source=s["heat"],
                                  Pr=PR, k_ratio=K_RATIO, precision=c["precision"])
    return {k: r[k] for k in ("rho", "u", "T", "steps")}


def _run_operators(s):
    c, m = s["case"], s["mask"]
    n = (c["nx"], c["ny"], c["nz"])
    tau_f, tau_s = simulation.derived_taus(TAU, PR, K_RATIO)
    fe, te = fluid_engine3d, thermal_engine3d
    fe.fused_equilibrium_collision_kernel(s["f"], s["rho"], s["u"], s["f_post"], m, TAU)
    fe.streaming_kernel(s["f_post"], s["f"], m, s["inlet"], RHO_OUT, *n)
    fe.compute_macroscopic_kernel(s["f"], s["rho"], s["u"])
    te.fused_thermal_equilibrium_collision_kernel(s["g"], s["u"], s["T"], s["g_post"], m, tau_f, tau_s, s["heat"],
                                                  POWER)
    te.thermal_streaming_kernel(s["g_post"], s["g"], m, T_IN, *n)
    te.compute_thermal_macroscopic_kernel(s["g"], s["T"])
    return {k: s[k] for k in ("f", "g", "rho", "u", "T")}


def _run_reduce(s):
    sc = metrics.device_scalars(s["rho"], s["u"], s["T"], s["mask"], tau_fluid=TAU, Pr=PR, u_inlet_val=s["u_in"],
                                t_inlet=T_IN, buf=_buf(s["case"]))
    return dict(scalars=sc, stats=fluid_engine3d.field_stats(s["rho"], s["u"], s["T"], s["mask"]))


def _run_conv(s):
    c = s["case"]
    return surrogate.conv_forward(s["x"], s["w"], s["b"], c["ksize"], act=c["act"], out_fp32=c["fp32"])


def _run_conv_train(s):
    y = surrogate.conv3d(s["x"], s["w"], s["b"], s["case"]["ksize"])
    dx, dw, db = torch.autograd.grad(y, (s["x"], s["w"], s["b"]), s["dy"])
    return dict(y=y, dx=dx, dw=dw, db=db)


def _run_predict(s):
    return dict(zip(("rho", "u", "T"), surrogate.predict(s["model"], s["mask"], s["heat"], s["u_in"], POWER)))


def _run_train(s):
    model = s["model"]
    for p in model.parameters():
        p.grad = None
    loss = F.mse_loss(model.forward(s["x"])[..., :surrogate.OUT_FIELDS], s["y"])
    loss.backward()
    return dict(loss=loss.detach(), grads={k: p.grad for k, p in model.params.items()})


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


# ------------------------------------------------------------------------------------------------ work
def _buf(case):
    return 10 if case["nx"] >= 60 else 3


@functools.lru_cache(maxsize=64)
def _nonsolid(family, nx, ny, nz):
    return int((_design(family, nx, ny, nz, 0)[0] != 1).sum())


def _step_work(family, nx, ny, nz, steps, precision):
    """Populations of the cells read and written once a step (a solid cell has no fluid populations to move), the
    two collisions' operations, and the five field values of a cell written once."""
    n, nf = nx * ny * nz, _nonsolid(family, nx, ny, nz)
    pe, qe = ELEM[precision]
    return (steps * 2 * 19 * (qe * n + pe * nf) + 20 * n, steps * (19 * 11 * n + 19 * 14 * nf))


def _net_work(V, train):
    """The surrogate's convolutions at batch x volume V: activations once in and once out, weights aside."""
    ch = [(16, 16, 1), (16, 16, 1), (16, 32, 8), (32, 32, 8), (32, 64, 64), (64, 64, 64), (64, 128, 512),
          (128, 128, 512), (192, 64, 64), (64, 64, 64), (96, 32, 8), (32, 32, 8), (48, 16, 1), (16, 16, 1)]
    k = 3 if train else 1
    return (k * sum(2 * (a + b) * V // r for a, b, r in ch), k * sum(54 * a * b * V // r for a, b, r in ch))


def work(case):
    kind = case["kind"]
    if kind in ("steps", "solve"):
        b, f = _step_work(case["family"], case["nx"], case["ny"], case["nz"], case["steps"], case["precision"])
    elif kind == "batch":
        b = f = 0
        for k in range(case["designs"]):
            wb, wf = _step_work(designs.FAMILIES[k % len(designs.FAMILIES)], *_sizes(case, k), case["steps"],
                                case["precision"])
            b, f = b + wb, f + wf
    elif kind in ("operators", "reduce"):
        n, nf = case["nx"] * case["ny"] * case["nz"], _nonsolid(case["family"], case["nx"], case["ny"], case["nz"])
        if kind == "reduce":  # rho, u, T and the label, for each of the two calls
            b, f = 2 * 24 * n, 30 * n
        else:  # each operator reads its populations once and writes them once; a solid cell is not streamed
            b, f = 76 * (9 * n + 2 * nf) + 76 * n, 19 * (11 * n + 14 * nf)
    elif kind in ("conv", "conv_train"):
        V, Ci, Co = case["N"] * case["D"] * case["H"] * case["W"], case["Ci"], case["Co"]
        taps = 27 if case["ksize"] == 3 else 1
        if kind == "conv":
            b, f = V * (2 * Ci + (4 if case["fp32"] else 2) * Co) + 2 * taps * Ci * Co, 2 * taps * Ci * Co * V
        else:
            b, f = V * (4 * Ci + 4 * Co) + 8 * taps * Ci * Co, 6 * taps * Ci * Co * V
    elif kind == "predict":
        b, f = _net_work(case["nz"] * case["ny"] * 152, False)
    else:
        b, f = _net_work(case["N"] * case["D"] * case["H"] * case["W"], True)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------------------------ 64 bits
E = np.array([[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1], [1, 1, 0], [-1, -1, 0],
              [1, -1, 0], [-1, 1, 0], [1, 0, 1], [-1, 0, -1], [1, 0, -1], [-1, 0, 1], [0, 1, 1], [0, -1, -1],
              [0, 1, -1], [0, -1, 1]])
OPP = [0, 2, 1, 4, 3, 6, 5, 8, 7, 10, 9, 12, 11, 14, 13, 16, 15, 18, 17]
WT = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12


class _Lbm64:
    """The coupled D3Q19 step in float64 (reference layout)."""

    def __init__(self, mask, heat, u_in, power):
        self.m = m = torch.as_tensor(mask).to(DEV)
        self.solid, self.inlet, self.outlet = m == 1, m == 2, m == 3
        h = torch.as_tensor(heat).to(DEV).double()
        self.q = h / h.max() * power
        self.u_in = float(np.float32(u_in))
        tf = 0.5 + (TAU - 0.5) / PR
        ts = 0.5 + K_RATIO * (tf - 0.5)
        self.om_t = torch.where(self.solid, 1.0 / ts, 1.0 / tf)
        self.e = torch.from_numpy(E).to(DEV).double()
        pad = F.pad(m, (1, 1, 1, 1, 1, 1), value=1)
        self.bb = [self._pull(pad, i) == 1 for i in range(19)]
        self.rows = {}
        for d, n in enumerate(m.shape):  # cells whose source along d would lie before the first / after the last
            at = torch.arange(n, device=DEV).view([n if k == d else 1 for k in range(3)])
            self.rows[d, 1], self.rows[d, -1] = (at == 0).expand(m.shape), (at == n - 1).expand(m.shape)

    def _pull(self, p, i):
        nx, ny, nz = self.m.shape
        x, y, z = (1 - int(v) for v in E[i])
        return p[x:x + nx, y:y + ny, z:z + nz]

    def eq(self, s, u):
        usq = 1.5 * (u * u).sum(-1)
        out = []
        for i in range(19):
            eu = (u * self.e[i]).sum(-1)
            out.append(WT[i] * s * (1 + 3 * eu + 4.5 * eu * eu - usq))
        return torch.stack(out)

    def fluid(self, f, rho, u):
        """collide, stream, moments -> f, rho, u"""
        post = f - (f - self.eq(rho, u)) / TAU
        post = torch.where(self.solid, f, post)
        new = []
        for i in range(19):
            src = self._pull(F.pad(post[i], (1, 1, 1, 1, 1, 1)), i)
            new.append(torch.where(self.bb[i], post[OPP[i]], src))
        new = torch.stack(new)
        k = post[:, self.inlet]
        if k.numel():
            rn = (k[[0, 3, 4, 5, 6, 15, 16, 17, 18]].sum(0) + 2 * k[[2, 8, 10, 12, 14]].sum(0)) / (1 - self.u_in)
            v = k.clone()
            v[1] = k[2] + 2 / 3 * rn * self.u_in
            for i, j in ((7, 10), (9, 8), (11, 14), (13, 12)):
                v[i] = k[j] + rn * self.u_in / 6
            new[:, self.inlet] = v
        west = torch.cat([post[:, :1], post[:, :-1]], 1)[:, self.outlet]
        if west.numel():
            tot = west.sum(0)
            new[:, self.outlet] = torch.where(tot > 1e-6, west * RHO_OUT / tot, west)
        f = torch.where(self.solid, f, new)
        rho = f.sum(0)
        u = torch.einsum("ixyz,id->xyzd", f, self.e) / rho[..., None]
        return f, rho, u

    def thermal(self, g, u, T):
        u = torch.where(self.solid[..., None], 0.0, u)
        src = (1 - 0.5 * self.om_t) * self.q
        post = g - self.om_t * (g - self.eq(T, u))
        post = post + torch.tensor(WT, device=DEV, dtype=torch.float64).view(19, 1, 1, 1) * src
        west = torch.cat([post[:, :1], post[:, :-1]], 1)
        new = []
        for i in range(19):
            v = self._pull(F.pad(post[i], (1, 1, 1, 1, 1, 1)), i)
            for d in (1, 2):
                if E[i][d]:
                    v = torch.where(self.rows[d, int(E[i][d])], post[OPP[i]], v)
            if E[i][0] == 1:
                v = torch.where(self.rows[0, 1], WT[i] * T_IN, v)
            elif E[i][0] == -1:
                v = torch.where(self.rows[0, -1], post[i], v)
            v = torch.where(self.inlet, WT[i] * T_IN, v)
            new.append(torch.where(self.outlet, west[i], v))
        g = torch.stack(new)
        return g, g.sum(0)

    def cold(self, steps):
        rho = torch.ones(self.m.shape, device=DEV, dtype=torch.float64)
        u = torch.zeros(tuple(self.m.shape) + (3,), device=DEV, dtype=torch.float64)
        T = torch.full_like(rho, T_IN)
        f, g = self.eq(rho, u), self.eq(T, u)
        for _ in range(steps):
            f, rho, u = self.fluid(f, rho, u)
            g, T = self.thermal(g, u, T)
        return dict(rho=rho, u=u, T=T)


def _stats64(m, rho, u, T):
    solid, out = m == 1, m == 3
    sq = (u * u).sum(-1)
    mag, fl = sq.sqrt(), ~solid
    n, plane = m.numel(), m.shape[1] * m.shape[2]
    v = [mag[fl].max(), mag[fl].sum(), sq.sum(), fl.sum(), rho[fl].sum(), rho[1].sum(), rho[-2].sum(),
         u[..., 0][out].sum(), plane, plane, out.sum(), T.max(), T.sum(), n, (u[..., 0] * T)[out].sum(), out.sum(), 0]
    return np.array([float(x) for x in v])


def _scalars64(m, rho, u, T, u_in, buf):
    """The scalar outputs of given fields (a 128 x 128 heated core behind `buf` inlet cells)."""
    nx, ny, nz = m.shape
    solid, ux = m == 1, u[..., 0]
    fluid = ~solid

    def mean(v, k):
        return float(v[k].mean()) if bool(k.any()) else 1.0

    r1, r2 = mean(rho[1], fluid[1]), mean(rho[-2], fluid[-2])
    out = (m == 3) & (torch.arange(nx, device=DEV) == nx - 1).view(-1, 1, 1)
    q_vol, q_out = float(ux[out].sum()), float((ux * T)[out].sum())
    dp = (r1 - r2) / 3
    floor = T[buf:min(buf + 128, nx), :min(128, ny), 0]
    q_abs = max(abs(q_out - T_IN * q_vol), 1e-12)
    t_out = q_out / q_vol if abs(q_vol) > 1e-12 else T_IN
    box = (slice(buf, nx - buf), slice(1, ny - 1), slice(4, nz - 2))
    bf, bs = fluid[box], solid[box]
    v_fluid = int(bf.sum())
    wet = sum(int((bs.narrow(d, 1, bs.shape[d] - 1) != bs.narrow(d, 0, bs.shape[d] - 1)).sum()) for d in range(3))
    tf = float(T[box][bf].mean()) if v_fluid else T_IN
    dh = 4.0 * v_fluid / wet if wet else float(ny)
    dt = float(floor.mean()) - tf
    h = q_abs / (wet * abs(dt)) if abs(dt) > 1e-6 and wet else 0.0
    k_f = (TAU - 0.5) / PR / 3
    pump, r_avg = abs(dp * q_vol), (r1 + r2) / 2
    core = solid[buf:nx - buf]
    return dict(delta_P=dp, R_th=(float(floor.max()) - T_IN) / q_abs, Nu=h * dh / k_f,
                f_friction=abs(dp) * dh / (2 * (nx - 2 * buf) * r_avg * u_in * u_in), P_pump=pump,
                COP=q_abs / pump if pump > 1e-12 else 0.0, Q_vol=q_vol, T_max_surface=float(floor.max()),
                T_avg_surface=float(floor.mean()), delta_T_max=float(floor.max() - floor.min()),
                sigma_T=float(floor.std(unbiased=False)), fluid_temp_rise=t_out - T_IN,
                pressure_drop=float(rho[1].mean() - rho[-2].mean()) / 3, max_velocity=float((u * u).sum(-1).max().sqrt()),
                max_temperature=float(T.max()), mean_temperature=float(T.mean()), Dh=dh, V_fluid=float(v_fluid),
                A_wetted=float(wet), porosity=1.0 - float(core.sum()) / core.numel(), Q_absorbed=q_abs, dT_conv=dt,
                rho_avg=r_avg)


def _conv64(x, w, b, ksize):
    """x [N,D,H,W,Ci], w [taps,Co,Ci] -> [N,D,H,W,Co], one tap after another (float64)."""
    if ksize == 1:
        return x @ w[0].T + b
    N, D, H, W, _ = x.shape
    p = F.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    y = torch.zeros((N, D, H, W, w.shape[1]), device=x.device, dtype=x.dtype) + b
    for t in range(27):
        z, r, c = t // 9, t // 3 % 3, t % 3
        y = y + p[:, z:z + D, r:r + H, c:c + W] @ w[t].T
    return y


def _net64(model, x):
    """The surrogate's network in float64."""
    p = {k: v.detach().double() for k, v in model.params.items()}

    def unit(x, n):
        y = _conv64(x, p[n + ".w"], p[n + ".b"], 3)
        N, C = y.shape[0], y.shape[-1]
        G = model.groups(C)
        h = y.reshape(N, -1, G, C // G)
        h = (h - h.mean(dim=(1, 3), keepdim=True)) / (h.var(dim=(1, 3), unbiased=False, keepdim=True) + 1e-5).sqrt()
        return F.gelu(h.reshape(y.shape) * p[n + ".g"] + p[n + ".s"])

    def pool(x):
        N, D, H, W, C = x.shape
        return x.view(N, D // 2, 2, H // 2, 2, W // 2, 2, C).mean(dim=(2, 4, 6))

    def up(x):
        return x.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)

    def block(x, n):
        return unit(unit(x, n + "a"), n + "b")

    e0 = block(x.double(), "e0")
    e1 = block(pool(e0), "e1")
    e2 = block(pool(e1), "e2")
    d2 = block(torch.cat([up(block(pool(e2), "b3")), e2], -1), "d2")
    d1 = block(torch.cat([up(d2), e1], -1), "d1")
    d0 = block(torch.cat([up(d1), e0], -1), "d0")
    return _conv64(d0, p["head.w"], p["head.b"], 1)


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind in ("steps", "solve"):
            m, h, u_in = _design(case["family"], case["nx"], case["ny"], case["nz"], seed)
            if kind == "solve" and m.size * case["steps"] > 1.2e9:
                return None  # more than 20 seconds
            r = _Lbm64(m, h, u_in, POWER).cold(case["steps"])
            if kind == "steps":
                r["stats"] = _stats64(torch.from_numpy(m).to(DEV), r["rho"], r["u"], r["T"])
            else:
                r["steps"] = None
            return r
        if kind == "batch":
            out = []
            for d in _batch_designs(case, seed):
                r = _Lbm64(d["mask"], d["heat_source"], d["u_inlet_val"], POWER).cold(case["steps"])
                out.append((r["rho"], r["u"], r["T"]))
            return dict(steps=[None] * len(out), fields=out)
        if kind in ("operators", "reduce"):
            m, h, u_in, rho, u, T = _fields(case, seed)
            rho, u, T = rho.double(), u.double(), T.double()
            if kind == "reduce":
                return dict(scalars=_scalars64(m, rho, u, T, u_in, _buf(case)), stats=_stats64(m, rho, u, T))
            b = _Lbm64(m, h, u_in, POWER)
            f, r, v = b.fluid(b.eq(rho, u), rho, u)
            g, t = b.thermal(b.eq(T, torch.where(b.solid[..., None], 0.0, u)), v, T)
            return dict(f=f, g=g, rho=r, u=v, T=t)
        if kind in ("conv", "conv_train"):
            x, w, b, dy = _conv_inputs(case, seed)
            w = w.to(torch.bfloat16).double()
            x, b, dy = x.double(), b.double(), dy.double()
            y = _conv64(x, w, b, case["ksize"])
            if kind == "conv":
                return F.gelu(y) if case["act"] else y
            dx = _conv64(dy, w.flip(0).transpose(1, 2), 0.0, case["ksize"])
            D, H, W = (case[k] for k in ("D", "H", "W"))
            p, dw = F.pad(x, (0, 0, 1, 1, 1, 1, 1, 1)), torch.empty_like(w)
            d2 = dy.reshape(-1, case["Co"])
            for t in range(w.shape[0]):
                z, r, c = (t // 9, t // 3 % 3, t % 3) if w.shape[0] == 27 else (1, 1, 1)
                dw[t] = d2.T @ p[:, z:z + D, r:r + H, c:c + W].reshape(-1, case["Ci"])
            return dict(y=y, dx=dx, dw=dw, db=d2.sum(0))
        if kind == "predict":
            m, h, u_in = _design(case["family"], case["nx"], case["ny"], case["nz"], seed)
            model = surrogate.load_pretrained()
            mean, std = (t.double() for t in model.norm)
            md = torch.from_numpy(m).to(DEV)
            p = _net64(model, surrogate.features(m, h, u_in, DEV))[..., :surrogate.OUT_FIELDS] * std + mean
            p = p[0, :, :, :case["nx"]].permute(2, 1, 0, 3)
            solid, inlet = md == 1, md == 2
            return dict(rho=torch.where(solid | inlet, 1.0, 1.0 + p[..., 3] * u_in),
                        u=torch.where((solid | inlet)[..., None], 0.0, p[..., 0:3] * u_in),
                        T=torch.where(inlet, T_IN, T_IN + p[..., 4] * POWER))
        return None  # the network's gradients in 64 bits take longer than 20 seconds
