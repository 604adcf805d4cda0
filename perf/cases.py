"""Workloads of the B200 lattice-Boltzmann library, as programs run them.

Each case is one call pattern of a user's program: a driver run (`run_*`), a
few steps of a fused kernel on a grid that the program keeps, a batched
cavity sweep, a cut-link step around a body, or the gradient of the
warm-start network.  `prepare` makes what the program holds before the call,
`run` is the call, `exact` restates it in FP64 torch.  Sizes follow the
reference's defaults (128 x 32 Rayleigh-Benard, N = 128 cavities), the
repository's benchmark (256^3 Taylor-Green, 4096^2 D2Q9, 512^2 natural
convection, cavities of N = 64..512, a sphere in a box, batch 16 at 256^2)
and ragged sizes between them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from __graft_entry__ import load_package

F64 = torch.float64
DTYPE = {"f64": torch.float64, "f32": torch.float32, "f32dev": torch.float32,
         "f16dev": torch.float16, "bf16dev": torch.bfloat16, "f16sr": torch.float16,
         "bf16sr": torch.bfloat16}
L2_BYTES = 126e6


def listed():
    return [
        # The quick-start: a lid-driven cavity on the reference's default
        # 128^2 grid, stepped by its driver in double precision.  Small
        # launches; latency counts.
        dict(name="cavity2d_128_f64", kind="cavity2d", Nx=128, Ny=128, steps=2000, storage="f64",
             lid="zou_he"),
        # The 3D cavity driver in single precision, an ordinary grid.
        dict(name="cavity3d_96_f32", kind="cavity3d", Nx=96, Ny=96, Nz=96, steps=400,
             storage="f32"),
        # Rayleigh-Benard convection, the thermal driver of the reference's
        # 4:1 box at twice its default size.
        dict(name="rayleigh_benard_256x64_f64", kind="rayleigh", Nx=256, Ny=64, steps=2000,
             storage="f64", orientation="vertical"),
        # The 3D heated cube, flow and thermal populations on D3Q19.
        dict(name="natconv3d_48_f64", kind="natconv3d", N=48, steps=800, storage="f64"),
        # De Vahl Davis natural convection at 512^2 in single precision.
        dict(name="natconv2d_512_f32", kind="natconv2d", N=512, steps=1000, storage="f32", Rc=1.0),
        # The benchmark's Taylor-Green box in FP32 deviations (largest grid),
        # moments at the last step.
        dict(name="trt3d_256_f32dev", kind="trt3d", Nx=256, Ny=256, Nz=256, steps=4,
             storage="f32dev", periodic=7, solid=False, moments=True),
        # The same box at half the memory.
        dict(name="trt3d_256_f16dev", kind="trt3d", Nx=256, Ny=256, Nz=256, steps=4,
             storage="f16dev", periodic=7, solid=False, moments=False),
        # A ragged walled duct with obstacles, reference arithmetic, moments.
        dict(name="trt3d_97x130x65_f64", kind="trt3d", Nx=97, Ny=130, Nz=65, steps=10,
             storage="f64", periodic=1, solid=True, moments=True),
        # A large D2Q9 step as the reference issues it (moments every step).
        dict(name="trt2d_4096_f32", kind="trt2d", op="trt", Nx=4096, Ny=4096, steps=4,
             storage="f32", solid=False),
        # A sensitivity sweep of cavities in FP16 deviations, one launch.
        dict(name="sweep_48_f16", kind="sweep", cases=48, N_lo=64, N_hi=512, N_step=32, steps=1000,
             storage="f16"),
        # Flow around a rotating sphere with interpolated walls.
        dict(name="libb_192_f32", kind="libb", Nx=192, Ny=192, Nz=192, R=0.16, steps=4,
             storage="f32", periodic=7),
        # One backward pass of the warm-start network at its training batch.
        dict(name="network_grad_b16_256", kind="network", mode="grad", batch=16, size=256, base=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cavity2d", "cavity3d", "rayleigh", "natconv3d", "natconv2d", "trt3d",
                       "trt3d", "trt2d", "sweep", "libb", "network"])
    plain = rng.choice(["f64", "f32"])
    if kind == "cavity2d":
        Nx, Ny = _log(rng, 24, 512), _log(rng, 24, 512)
        return dict(kind=kind, Nx=Nx, Ny=Ny, steps=_log(rng, 200, 2000), storage=plain,
                    lid=rng.choice(["zou_he", "moving_wall"]))
    if kind == "cavity3d":
        Nx, Ny, Nz = (_log(rng, 12, 128) for _ in range(3))
        return dict(kind=kind, Nx=Nx, Ny=Ny, Nz=Nz, steps=_log(rng, 50, 400), storage=plain)
    if kind == "rayleigh":
        return dict(kind=kind, Nx=_log(rng, 32, 1024), Ny=_log(rng, 32, 256),
                    steps=_log(rng, 400, 2000), storage=plain,
                    orientation=rng.choice(["vertical", "horizontal"]))
    if kind == "natconv3d":
        N = _log(rng, 12, 128)
        return dict(kind=kind, N=N, steps=_log(rng, 200, 800) if N <= 64 else 200, storage=plain)
    if kind == "natconv2d":
        return dict(kind=kind, N=_log(rng, 24, 768), steps=_log(rng, 100, 1000), storage=plain,
                    Rc=rng.choice([1.0, 2.0]))
    if kind == "trt3d":
        Nx, Ny, Nz = (_log(rng, 16, 256) for _ in range(3))
        if rng.random() < 0.5:
            Nx = max(16, Nx // 16 * 16)
        return dict(kind=kind, Nx=Nx, Ny=Ny, Nz=Nz, steps=rng.choice([2, 4]),
                    storage=rng.choice(["f64", "f32", "f32dev", "f16dev", "bf16dev", "f16sr"]),
                    periodic=rng.randrange(8), solid=rng.random() < 0.4,
                    moments=rng.random() < 0.5)
    if kind == "trt2d":
        return dict(kind=kind, op=rng.choice(["trt", "bgk"]), Nx=_log(rng, 64, 4096),
                    Ny=_log(rng, 64, 4096), steps=rng.choice([2, 4]), storage=plain,
                    solid=rng.random() < 0.4)
    if kind == "sweep":
        lo = rng.choice([33, 64, 96])
        return dict(kind=kind, cases=rng.randrange(4, 49), N_lo=lo,
                    N_hi=lo + _log(rng, 32, 400), N_step=rng.choice([17, 32, 64]),
                    steps=100 * rng.randrange(2, 9),
                    storage=rng.choice(["f16", "f16", "f16sr", "bf16", "f32"]))
    if kind == "libb":
        Nx, Ny, Nz = (_log(rng, 32, 192) for _ in range(3))
        if rng.random() < 0.5:
            Nx = max(32, Nx // 32 * 32)
        return dict(kind=kind, Nx=Nx, Ny=Ny, Nz=Nz, R=rng.uniform(0.12, 0.3), steps=4,
                    storage=rng.choice(["f64", "f32", "f32dev", "f16dev"]),
                    periodic=rng.choice([0, 1, 7]))
    size = rng.choice([64, 128, 256])
    return dict(kind=kind, mode=rng.choice(["grad", "infer"]), batch=rng.randrange(1, 17),
                size=size, base=rng.choice([16, 32]))


# ------------------------------------------------------------------ lattices

C9 = [(0, 0), (1, 0), (0, 1), (-1, 0), (0, -1), (1, 1), (-1, 1), (-1, -1), (1, -1)]
W9 = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
C19 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1),
       (1, 1, 0), (-1, 1, 0), (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1),
       (-1, 0, -1), (0, 1, 1), (0, -1, 1), (0, 1, -1), (0, -1, -1)]
W19 = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
OPP9 = [C9.index((-a, -b)) for a, b in C9]
OPP19 = [C19.index((-a, -b, -c)) for a, b, c in C19]


def _lat(f):
    return (C9, W9, OPP9) if f.shape[0] == 9 else (C19, W19, OPP19)


def _pull(f, per):
    """Pull streaming with half-way bounce-back where an axis is not periodic."""
    C, _, opp = _lat(f)
    nd = f.dim() - 1
    out = torch.empty_like(f)
    for q, c in enumerate(C):
        ax = [a for a in range(len(c)) if c[a]]
        out[q] = torch.roll(f[q], [c[a] for a in ax], [nd - 1 - a for a in ax]) if ax else f[q]
        for a in ax:
            if not per[a]:
                e = 0 if c[a] > 0 else -1
                out[q].select(nd - 1 - a, e).copy_(f[opp[q]].select(nd - 1 - a, e))
    return out


def _dot(c, v):
    s = None
    for ca, va in zip(c, v):
        if ca:
            t = va if ca > 0 else -va
            s = t if s is None else s + t
    return s if s is not None else torch.zeros_like(v[0])


def _moments(f, force=None):
    """(rho, [u]) with the half-force correction where a force is given."""
    C, _, _ = _lat(f)
    rho = f.sum(0)
    u = []
    for a in range(f.dim() - 1):
        j = sum((f[q] if c[a] > 0 else -f[q]) for q, c in enumerate(C) if c[a])
        if force is not None and force[a] is not None:
            j = j + force[a] / 2
        u.append(j / rho)
    return rho, u


def _feq(q, f_like, rho, u, usq):
    C, W, _ = f_like
    cu = _dot(C[q], u)
    return W[q] * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * usq)


def _bgk(f, om, solid=None):
    lat = _lat(f)
    rho, u = _moments(f)
    usq = sum(a * a for a in u)
    return torch.stack([f[q] - om * (f[q] - _feq(q, lat, rho, u, usq)) for q in range(f.shape[0])])


def _trt(f, sp, sm):
    lat = _lat(f)
    opp = lat[2]
    rho, u = _moments(f)
    usq = sum(a * a for a in u)
    a, b = (sp + sm) / 2, (sp - sm) / 2
    ne = [f[q] - _feq(q, lat, rho, u, usq) for q in range(f.shape[0])]
    out = torch.empty_like(f)
    for q in range(f.shape[0]):
        out[q] = f[q] - (sp * ne[q] if q == 0 else a * ne[q] + b * ne[opp[q]])
    return out, rho, u


def _guo(f, om, force):
    """BGK with the Guo source of a body force (None: no component)."""
    lat = _lat(f)
    C, W, _ = lat
    rho, u = _moments(f, force)
    usq = sum(a * a for a in u)
    out = torch.empty_like(f)
    F = [x if x is not None else torch.zeros_like(rho) for x in force]
    uF = sum(a * b for a, b in zip(u, F))
    for q in range(f.shape[0]):
        cF, cu = _dot(C[q], F), _dot(C[q], u)
        S = W[q] * (3 * (cF - uF) + 9 * cu * cF)
        out[q] = f[q] - om * (f[q] - _feq(q, lat, rho, u, usq)) + (1 - om / 2) * S
    return out


def _thermal(g, u, om):
    C, W, _ = _lat(g)
    T = g.sum(0)
    return torch.stack([g[q] - om * (g[q] - W[q] * T * (1 + 3 * _dot(C[q], u)))
                        for q in range(g.shape[0])])


def _abb(g, axis, high, T_wall):
    """Half-way anti-bounce-back of one fixed-temperature face, in place."""
    C, W, _ = _lat(g)
    d = g.dim() - 2 - axis
    for q, c in enumerate(C):
        if c[axis] == (-1 if high else 1):
            s = g[q].select(d, -1 if high else 0)
            s.copy_(-s + 2 * W[q] * T_wall)


def _trt_rates(nu, Lam):
    return 1 / (3 * nu + 0.5), 1 / (Lam / (3 * nu) + 0.5)


# -------------------------------------------------------------------- inputs

def _rng(seed):
    return np.random.default_rng([17, seed])


def _numbers(case, seed):
    """Physical parameters of a run, drawn from the seed."""
    r = _rng(seed)
    n = dict(nu=float(r.uniform(0.05, 0.12)), u=float(r.uniform(0.05, 0.1)),
             Pr=float(r.uniform(0.7, 1.0)), T_hot=float(r.uniform(0.9, 1.1)))
    # thermal runs: Rayleigh numbers that grow with the box, from the onset of
    # convection in a 32-node layer to 1e6 at 512^2, so that the buoyancy per
    # node stays in the range the scheme is used in
    if case["kind"] == "natconv2d":
        n["Ra"] = float(r.uniform(0.003, 0.0075)) * case["N"] ** 3
    elif case["kind"] == "natconv3d":
        n["Ra"] = float(r.uniform(1.0, 3.0)) * case["N"] ** 2
    elif case["kind"] == "rayleigh":
        H = case["Ny"] if case["orientation"] == "vertical" else case["Nx"]
        n["Ra"] = float(r.uniform(2.0, 4.0)) * H ** 2
    return n


def _flow(shape, Q, seed):
    """Populations of a developed flow in FP64 on the GPU: equilibrium of a
    few random smooth modes plus a small non-equilibrium part."""
    r = _rng(seed)
    nd = len(shape)
    W = W9 if Q == 9 else W19
    C = C9 if Q == 9 else C19
    x = [torch.arange(shape[nd - 1 - a], dtype=F64, device="cuda").view(
        [-1 if d == nd - 1 - a else 1 for d in range(nd)]) * (2 * math.pi / shape[nd - 1 - a])
        for a in range(nd)]

    def mode(amp):
        s = 0
        for _ in range(2):
            p = 1.0
            for a in range(nd):
                p = p * torch.sin(int(r.integers(1, 4)) * x[a] + float(r.uniform(0, 6.28)))
            s = s + amp * float(r.uniform(0.5, 1.0)) * p
        return s

    u = [mode(0.03) for _ in range(nd)]
    rho = 1 + mode(0.005)
    usq = sum(a * a for a in u)
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7 + 1)
    f = torch.empty((Q,) + tuple(shape), dtype=F64, device="cuda")
    for q in range(Q):
        f[q] = _feq(q, (C, W, None), rho, u, usq)
        f[q] += (1e-3 * W[q]) * torch.randn(tuple(shape), dtype=torch.float32, device="cuda",
                                            generator=gen)
    return f


def _stored(case, f):
    """Populations in the case's storage (f, or f - w rounded once)."""
    s = case["storage"]
    if s not in ("f64", "f32"):
        for q, w in enumerate(W9 if f.shape[0] == 9 else W19):
            f[q] -= w
    return f.to(DTYPE[s])


def _loaded(case, st):
    f = st.to(F64).clone()
    if case["storage"] not in ("f64", "f32"):
        for q, w in enumerate(W9 if f.shape[0] == 9 else W19):
            f[q] += w
    return f


def _unloaded(case, f):
    if case["storage"] in ("f64", "f32"):
        return f
    f = f.clone()
    for q, w in enumerate(W9 if f.shape[0] == 9 else W19):
        f[q] -= w
    return f


def _solid(shape, seed):
    """A few box obstacles (about 5 % of the nodes)."""
    r = _rng(seed + 5)
    m = torch.zeros(shape, dtype=torch.bool, device="cuda")
    for _ in range(6):
        sl = []
        for n in shape:
            w = max(1, int(n * r.uniform(0.12, 0.3)))
            a = int(r.integers(0, max(1, n - w + 1)))
            sl.append(slice(a, a + w))
        m[tuple(sl)] = True
    return m


def _sweep_table(case, seed):
    r = _rng(seed)
    Ns = np.arange(case["N_lo"], case["N_hi"] + 1, case["N_step"])
    N = _rng(0).choice(Ns, size=case["cases"]).astype(np.int32)  # sizes belong to the case
    Re = np.exp(r.uniform(np.log(100.0), np.log(np.minimum(1000.0, 9.0 * N))))
    u = np.full(case["cases"], 0.1)
    return N, u * N / Re, u


def _sphere(case, seed):
    """Cut fractions, solid mask and wall velocity of a rotating sphere."""
    Nx, Ny, Nz = case["Nx"], case["Ny"], case["Nz"]
    r = _rng(seed + 3)
    ctr = [(n - 1) / 2 + float(r.uniform(-0.4, 0.4)) for n in (Nx, Ny, Nz)]
    R2 = (case["R"] * min(Nx, Ny, Nz)) ** 2
    Om = [float(v) for v in r.uniform(-2e-3, 2e-3, 3)]
    dt = F64 if case["storage"] == "f64" else torch.float32
    shape = (Nz, Ny, Nx)
    ax = [torch.arange(n, dtype=F64, device="cuda").view(v) - c
          for n, v, c in zip((Nx, Ny, Nz), ((1, 1, -1), (1, -1, 1), (-1, 1, 1)), ctr)]
    d2 = ax[0] ** 2 + ax[1] ** 2 + ax[2] ** 2
    solid = d2 <= R2
    qw = torch.zeros((19,) + shape, dtype=dt, device="cuda")
    uw = [torch.zeros((19,) + shape, dtype=dt, device="cuda") for _ in range(3)]
    for q in range(1, 19):
        c = C19[q]
        end = sum((a + ci) ** 2 for a, ci in zip(ax, c))
        k, j, i = torch.nonzero(~solid & (end <= R2), as_tuple=True)
        p = [ax[0][0, 0, i], ax[1][0, j, 0], ax[2][k, 0, 0]]
        A = float(sum(ci * ci for ci in c))
        B = sum(a * ci for a, ci in zip(p, c))
        t = (-B - torch.sqrt(B * B - A * (sum(a * a for a in p) - R2))) / A
        t = t.clamp(1e-3, 1.0)
        w = [a + t * ci for a, ci in zip(p, c)]
        qw[q, k, j, i] = t.to(dt)
        for n, v in enumerate((Om[1] * w[2] - Om[2] * w[1], Om[2] * w[0] - Om[0] * w[2],
                               Om[0] * w[1] - Om[1] * w[0])):
            uw[n][q, k, j, i] = v.to(dt)
    return qw, solid, uw


# The warm-start network: a 4-level encoder-decoder of 3x3 convolutions (zero
# padding, ReLU but for the head), 2x2 mean pooling, nearest upsampling and
# skip concatenation [upsampled, skip]; weights [cout][3][3][cin] then biases.
def _net_layers(base):
    b = base
    return [(8, b), (b, b), (b, 2 * b), (2 * b, 2 * b), (2 * b, 4 * b), (4 * b, 4 * b),
            (4 * b, 8 * b), (8 * b, 8 * b), (12 * b, 4 * b), (4 * b, 4 * b), (6 * b, 2 * b),
            (2 * b, 2 * b), (3 * b, b), (b, b), (b, 16)]


SCALE, OFFSET = (30.0, 10.0, 10.0), (1.0, 0.0, 0.0)


def _net_inputs(case, seed):
    """Parameters (He-normal, small biases), inputs and target fields."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 13 + 5)
    parts = []
    for cin, cout in _net_layers(case["base"]):
        w = torch.randn(cout * 9 * cin, device="cuda", generator=g) * math.sqrt(2 / (9 * cin))
        parts += [w, 0.05 * torch.randn(cout, device="cuda", generator=g)]
    p = torch.cat(parts).bfloat16().float()
    n, S = case["batch"], case["size"]
    re = torch.exp(torch.rand(n, device="cuda", generator=g) * math.log(32.0)) * 100.0
    h = torch.arange(S, device="cuda").view(1, S, 1)
    w = torch.arange(S, device="cuda").view(1, 1, S)
    x = torch.zeros((n, S, S, 8), device="cuda")
    x[..., 0] = ((w == 0) | (w == S - 1) | (h == 0)).float()
    x[..., 1] = (h == S - 1).float()
    x[..., 2] = (torch.log(re / 100.0) / math.log(32.0)).view(n, 1, 1)
    x[..., 3] = S / 512.0
    x[..., 4] = 2.0 * (w + 0.5) / S - 1.0
    x[..., 5] = 2.0 * (h + 0.5) / S - 1.0
    a = torch.rand((n, 3, 4), device="cuda", generator=g)
    px = (w / S * 6.28).view(1, 1, 1, S)
    py = (h / S * 6.28).view(1, 1, S, 1)
    t = 0.08 * (a[:, :, 0, None, None] * torch.sin(px + 6.28 * a[:, :, 1, None, None]) *
                torch.sin(py + 6.28 * a[:, :, 2, None, None]))
    t[:, 0] = 1.0 + 0.1 * t[:, 0]
    return p, x.bfloat16().contiguous(), t.contiguous()


# ------------------------------------------------------------------- prepare

def prepare(case, seed):
    kb = load_package()
    s = dict(kb=kb, case=case, n=_numbers(case, seed))
    k = case["kind"]
    if k in ("trt3d", "trt2d", "libb"):
        shape = (case["Ny"], case["Nx"]) if k == "trt2d" else (case["Nz"], case["Ny"], case["Nx"])
        s["f0"] = _stored(case, _flow(shape, 9 if k == "trt2d" else 19, seed))
        s["a"], s["b"] = torch.empty_like(s["f0"]), torch.empty_like(s["f0"])
        fd = F64 if case["storage"] == "f64" else torch.float32
        s["m"] = [torch.zeros(shape, dtype=fd, device="cuda") for _ in range(1 + len(shape))]
        s["solid"] = _solid(shape, seed) if case.get("solid") else None
        if k == "libb":
            qw, solid, uw = _sphere(case, seed)
            s["links"] = kb.libb.CutLinks(solid, qw, *uw)
    elif k == "sweep":
        N, nu, u = _sweep_table(case, seed)
        s["batch"] = kb.CavityBatch(N, nu, u, case["storage"])
    elif k == "network":
        p, x, t = _net_inputs(case, seed)
        net = kb.surrogate.Surrogate(max_batch=case["batch"], H=case["size"], W=case["size"],
                                     base_channels=case["base"], seed=0, scale=SCALE,
                                     offset=OFFSET)
        net.set_params(p)
        s.update(net=net, x=x, t=t)
    torch.cuda.synchronize()
    return s


# ----------------------------------------------------------------------- run

def run(s):
    kb, c, n = s["kb"], s["case"], s["n"]
    k = c["kind"]
    if k == "cavity2d":
        cfg = kb.LBMConfig.d2q9(c["Nx"], c["Ny"], n["nu"], n["u"], c["steps"])
        r = kb.run_cavity_2d(cfg, T=DTYPE[c["storage"]], lid=c["lid"])
        return dict(rho=r["rho"], ux=r["ux"], uy=r["uy"], f=r["state"]["f_in"])
    if k == "cavity3d":
        cfg = kb.LBMConfig.d3q19(c["Nx"], c["Ny"], c["Nz"], n["nu"], n["u"], c["steps"])
        r = kb.run_cavity_3d(cfg, T=DTYPE[c["storage"]])
        return {x: r[x] for x in ("rho", "ux", "uy", "uz")}
    if k == "rayleigh":
        r = kb.run_rayleigh_benard_2d(c["Nx"], c["Ny"], n["Ra"], n["Pr"], n["T_hot"], 0.0,
                                      c["steps"], orientation=c["orientation"],
                                      FT=DTYPE[c["storage"]])
        return {x: r[x] for x in ("rho", "ux", "uy", "Temp", "f", "g")}
    if k == "natconv3d":
        r = kb.run_natural_convection_3d(c["N"], n["Ra"], n["Pr"], n["T_hot"], 0.0, c["steps"],
                                         FT=DTYPE[c["storage"]])
        return {x: r[x] for x in ("rho", "ux", "uy", "uz", "Temp", "f", "g")}
    if k == "natconv2d":
        r = kb.run_natural_convection_2d(c["N"], n["Ra"], n["Pr"], c["Rc"], n["T_hot"], 0.0,
                                         c["steps"], FT=DTYPE[c["storage"]])
        return {x: r[x] for x in ("rho", "ux", "uy", "Temp")}
    if k == "sweep":
        b = s["batch"]
        b.reset()
        b.run(max_steps=c["steps"], check_every=100, tol=1e-9)
        out = [b.case(i) for i in range(c["cases"])]
        return dict(ux=np.concatenate([o["ux"].ravel() for o in out]),
                    uy=np.concatenate([o["uy"].ravel() for o in out]),
                    steps=np.array([o["steps"] for o in out]))
    if k == "network":
        if c["mode"] == "infer":
            return s["net"].infer(s["x"])
        loss = s["net"].loss_backward(s["x"], s["t"])
        return dict(loss=loss, grads=s["net"].grads())
    # a few steps of a fused kernel between two buffers of the program
    src, dst, m = s["f0"], s["a"], s["m"]
    dev = c["storage"] not in ("f64", "f32")
    sr = c["storage"].endswith("sr")
    none = [None] * len(m)
    per = c.get("periodic", 0)
    for i in range(c["steps"]):
        last = i == c["steps"] - 1
        if k == "trt2d":
            if c["op"] == "trt":
                kb.fused_trt_step_(dst, src, *m, s["solid"], c["Nx"], c["Ny"], n["nu"])
            else:
                kb.fused_bgk_step_(dst, src, *m, s["solid"], c["Nx"], c["Ny"],
                                   1 / (3 * n["nu"] + 0.5))
        elif k == "libb":
            kb.fused_trt_libb_links_step_3d_(dst, src, *(m if last else none), s["links"], n["nu"],
                                             periodic=per, deviation=dev)
        else:
            kb.fused_trt_step_3d_(dst, src, *(m if last and c["moments"] else none), s["solid"],
                                  c["Nx"], c["Ny"], c["Nz"], n["nu"], 0.25, periodic=per,
                                  deviation=dev, stochastic_rounding=sr)
        src, dst = dst, (s["b"] if dst is s["a"] else s["a"])
    return dict(f=src, moments=m if (k != "trt3d" or c["moments"]) else [])


# ---------------------------------------------------------------------- work

def work(case):
    k = case["kind"]
    b = torch.empty((), dtype=DTYPE.get(case.get("storage"), torch.float16)).element_size()
    if k == "network":
        n, S, tot, px = case["batch"], case["size"], 0.0, []
        lev = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0, 0]
        par = 0
        for (ci, co), l in zip(_net_layers(case["base"]), lev):
            tot += 2.0 * 9 * ci * co * n * (S >> l) ** 2
            par += co * (9 * ci + 1)
        # gradient: forward, data gradient (not of the input layer), weight gradient
        first = 2.0 * 9 * 8 * case["base"] * n * S * S
        fl = tot if case["mode"] == "infer" else 3 * tot - first
        by = n * S * S * (16 + 12) + par * (2 if case["mode"] == "infer" else 6)
        return {"bytes": by, "flops": fl}
    if k == "sweep":
        b = {"f32": 4}.get(case["storage"], 2)
        Ns = np.arange(case["N_lo"], case["N_hi"] + 1, case["N_step"]).astype(float)
        nodes = float(np.mean(Ns ** 2)) * case["cases"]
        state, out, fl = nodes * 9 * b, nodes * 8, 90
    elif k in ("trt2d",):
        nodes = case["Nx"] * case["Ny"]
        fl = 110
        return {"bytes": nodes * case["steps"] * (21 * b + (1 if case["solid"] else 0)),
                "flops": nodes * case["steps"] * fl}
    elif k in ("trt3d", "libb"):
        nodes = case["Nx"] * case["Ny"] * case["Nz"]
        mom = (8 if case["storage"] == "f64" else 4) * 4 if case.get("moments", True) else 0
        mask = 1 if case.get("solid") or k == "libb" else 0
        return {"bytes": nodes * (case["steps"] * (38 * b + mask) + mom),
                "flops": nodes * case["steps"] * 260}
    elif k == "cavity2d":
        nodes = case["Nx"] * case["Ny"]
        state, out, fl = nodes * 9 * b, nodes * 3 * b, 110
    elif k == "cavity3d":
        nodes = case["Nx"] * case["Ny"] * case["Nz"]
        state, out, fl = nodes * 19 * b, nodes * 4 * b, 260
    elif k == "rayleigh":
        nodes = case["Nx"] * case["Ny"]
        state, out, fl = nodes * 18 * b, nodes * 4 * b, 330
    elif k == "natconv2d":
        nodes = case["N"] ** 2
        state, out, fl = nodes * 18 * b, nodes * 4 * b, 330
    else:
        nodes = case["N"] ** 3
        state, out, fl = nodes * 38 * b, nodes * 5 * b, 850
    # a run whose populations fit the L2 cache needs HBM for its first and
    # last state only; a larger one reads and writes them every step
    n = case["steps"] if state > L2_BYTES else 1
    return {"bytes": 2 * state * n + out, "flops": nodes * case["steps"] * fl}


# ----------------------------------------------------------------- tolerance

def tolerance(case):
    """About four times the difference from the same run with FP64 sums (or
    between two runs that round stochastically), per storage."""
    k = case["kind"]
    if k == "network":
        if case["mode"] == "infer":
            return {"rel": 1.5e-3}
        # BF16 activations of 15 layers; fewer pixels average less of it out
        return {"rel": 3e-3 if case["batch"] * case["size"] ** 2 >= 500000 else 2e-2}
    st = case["storage"]
    if k == "sweep":
        return {"rel": {"f32": 4e-5, "f16sr": 2e-3, "f16": 2e-2}.get(st, 8e-2)}
    thermal = k in ("rayleigh", "natconv3d", "natconv2d")
    if st == "f64":
        return {"rel": 1e-9 if thermal else 1e-11}
    if st == "f32":
        # whole populations: every step rounds O(w) values once, and a driver
        # run collects those roundings in velocities far below 1
        return {"rel": 5e-2 if thermal else {"cavity2d": 1e-4, "cavity3d": 1e-3}.get(k, 1e-5)}
    return {"rel": {"f32dev": 1e-6, "f16dev": 1e-3, "f16sr": 2e-3}.get(st, 8e-3)}


# --------------------------------------------------------------------- exact

def exact(case, seed):
    k, n = case["kind"], _numbers(case, seed)
    with torch.no_grad():
        return {"cavity2d": _exact_cavity2d, "cavity3d": _exact_cavity3d,
                "rayleigh": _exact_rayleigh, "natconv3d": _exact_natconv3d,
                "natconv2d": _exact_natconv2d, "sweep": _exact_sweep, "network": _exact_network,
                "trt2d": _exact_trt, "trt3d": _exact_trt, "libb": _exact_trt}[k](case, n, seed)


def _rest(shape, Q):
    w = torch.tensor(W9 if Q == 9 else W19, dtype=F64, device="cuda")
    return w.view([-1] + [1] * len(shape)).expand((Q,) + tuple(shape)).contiguous()


def _exact_cavity2d(c, n, seed):
    f = _rest((c["Ny"], c["Nx"]), 9)
    om, u = 1 / (3 * n["nu"] + 0.5), n["u"]
    for _ in range(c["steps"]):
        p = _pull(f, (0, 0))
        if c["lid"] == "zou_he":
            t = p[:, -1, :].clone()
            rw = t[0] + t[1] + t[3] + 2 * (t[2] + t[5] + t[6])
            p[4, -1] = t[2]
            p[8, -1] = t[6] - 0.5 * (t[1] - t[3]) + 0.5 * rw * u
            p[7, -1] = t[5] + 0.5 * (t[1] - t[3]) - 0.5 * rw * u
        else:
            p[4, -1] = f[2, -1]
            p[7, -1] = f[5, -1] - u / 6
            p[8, -1] = f[6, -1] + u / 6
            mom = _moments(p)
        f = _bgk(p, om)
    rho, uu = _moments(f) if c["lid"] == "zou_he" else mom
    return dict(rho=rho, ux=uu[0], uy=uu[1], f=f)


def _exact_cavity3d(c, n, seed):
    f = _rest((c["Nz"], c["Ny"], c["Nx"]), 19)
    om, u = 1 / (3 * n["nu"] + 0.5), n["u"]
    for _ in range(c["steps"]):
        p = _pull(f, (0, 0, 0))
        t = p[:, -1].clone()
        rw = t[0] + t[1] + t[2] + t[3] + t[4] + t[7] + t[8] + t[9] + t[10] + 2 * (
            t[5] + t[11] + t[12] + t[15] + t[16])
        t1 = (t[1] - t[2]) + (t[7] - t[8] + t[9] - t[10])
        t2 = (t[3] - t[4]) + (t[7] + t[8] - t[9] - t[10])
        p[6, -1] = t[5]
        p[13, -1] = t[12] - 0.5 * t1 + 0.5 * rw * u
        p[14, -1] = t[11] + 0.5 * t1 - 0.5 * rw * u
        p[17, -1] = t[16] - 0.5 * t2
        p[18, -1] = t[15] + 0.5 * t2
        f = _bgk(p, om)
    rho, uu = _moments(f)
    return dict(rho=rho, ux=uu[0], uy=uu[1], uz=uu[2])


def _exact_rayleigh(c, n, seed):
    Nx, Ny = c["Nx"], c["Ny"]
    nu = 0.05
    al = nu / n["Pr"]
    Th = n["T_hot"]
    vert = c["orientation"] == "vertical"
    beta = n["Ra"] * nu * al / (Th * (Ny if vert else Nx) ** 3)
    i = torch.arange(1, Nx + 1, dtype=F64, device="cuda")[None, :]
    j = torch.arange(1, Ny + 1, dtype=F64, device="cuda")[:, None]
    if vert:
        T0 = Th - Th * (j - 0.5) / Ny + 0.01 * Th * torch.sin(2 * math.pi * i / Nx) * \
            torch.sin(math.pi * j / Ny)
    else:
        T0 = (Th - Th * (i - 0.5) / Nx).expand(Ny, Nx)
    f = _rest((Ny, Nx), 9)
    g = torch.stack([w * T0 for w in W9])
    wf, wT, Tr = 1 / (3 * nu + 0.5), 1 / (3 * al + 0.5), Th / 2
    per = (1, 0) if vert else (0, 0)
    for _ in range(c["steps"]):
        f, g = _pull(f, per), _pull(g, per)
        _abb(g, 1 if vert else 0, False, Th)
        _abb(g, 1 if vert else 0, True, 0.0)
        T = g.sum(0)
        _, u = _moments(f)
        g = _thermal(g, u, wT)
        f = _guo(f, wf, [None, beta * (T - Tr)])
    rho, u = _moments(f)
    return dict(rho=rho, ux=u[0], uy=u[1], Temp=g.sum(0), f=f, g=g)


def _exact_natconv3d(c, n, seed):
    N = c["N"]
    nu = 0.05
    al = nu / n["Pr"]
    Th = n["T_hot"]
    beta = n["Ra"] * nu * al / (Th * float(N) ** 3)
    i = torch.arange(1, N + 1, dtype=F64, device="cuda")
    T0 = (Th - Th * (i - 0.5) / N).expand(N, N, N)
    f = _rest((N, N, N), 19)
    g = torch.stack([w * T0 for w in W19])
    wf, wT, Tr = 1 / (3 * nu + 0.5), 1 / (3 * al + 0.5), Th / 2
    for _ in range(c["steps"]):
        f, g = _pull(f, (0, 0, 0)), _pull(g, (0, 0, 0))
        _abb(g, 0, False, Th)
        _abb(g, 0, True, 0.0)
        T = g.sum(0)
        _, u = _moments(f)
        g = _thermal(g, u, wT)
        f = _guo(f, wf, [None, beta * (T - Tr), None])
    rho, u = _moments(f)
    return dict(rho=rho, ux=u[0], uy=u[1], uz=u[2], Temp=g.sum(0), f=f, g=g)


def _exact_natconv2d(c, n, seed):
    N = c["N"]
    nu = 0.05
    al = nu / n["Pr"]
    Th = n["T_hot"]
    beta = n["Ra"] * nu * al / (Th * float(N) ** 3)
    i = torch.arange(1, N + 1, dtype=F64, device="cuda")[None, :]
    j = torch.arange(1, N + 1, dtype=F64, device="cuda")[:, None]
    T0 = Th - Th * (i - 0.5) / N + 0.01 * Th * torch.sin(2 * math.pi * i / N) * \
        torch.sin(math.pi * j / N)
    f = _rest((N, N), 9)
    g = torch.stack([w * T0 for w in W9])
    wf, wT, Tr = 1 / (3 * nu + 0.5), 1 / (3 * al + 0.5), Th / 2
    for _ in range(c["steps"]):
        f, g = _pull(f, (0, 0)), _pull(g, (0, 0))
        _abb(g, 0, False, Th)
        _abb(g, 0, True, 0.0)
        T = g.sum(0)
        F = [None, beta * (T - Tr)]
        _, u = _moments(f, F)
        g = _thermal(g, u, wT)
        w = wf if c["Rc"] == 1.0 else 1 / (3 * nu * torch.exp(-math.log(c["Rc"]) * T) + 0.5)
        f = _guo(f, w, F)
    rho, u = _moments(f)
    return dict(rho=rho, ux=u[0], uy=u[1], Temp=g.sum(0))


def _exact_trt(c, n, seed):
    k = c["kind"]
    shape = (c["Ny"], c["Nx"]) if k == "trt2d" else (c["Nz"], c["Ny"], c["Nx"])
    f = _loaded(c, _stored(c, _flow(shape, 9 if k == "trt2d" else 19, seed)))
    C, W, opp = _lat(f)
    sol = _solid(shape, seed) if c.get("solid") else None
    if k == "libb":
        qw, sol, uw = _sphere(c, seed)
        cut = []
        order = [1, 2, 3, 4, 5, 6, 7, 10, 8, 9, 11, 14, 12, 13, 15, 18, 16, 17]
        for q in order:
            at = torch.nonzero(qw[q] > 0, as_tuple=True)
            t = qw[q][at].to(F64)
            d = -6 * W[q] * sum(ci * uw[a][q][at].to(F64) for a, ci in enumerate(C[q]) if ci)
            cut.append((q, at, t, d))
    Lam = 0.25 if k == "trt3d" else 3 / 16
    sp, sm = _trt_rates(n["nu"], Lam)
    if k == "trt2d" and c["op"] == "bgk":
        sm = sp
    per = c.get("periodic", 0)
    per = [(per >> a) & 1 for a in range(len(shape))]
    for _ in range(c["steps"]):
        p = _pull(f, per)
        if k == "libb":
            for q, at, t, d in cut:
                here, back, bar = f[q][at], p[q][at], f[opp[q]][at]
                inv = 1 / (2 * t)
                p[opp[q]][at] = torch.where(t <= 0.5, 2 * t * here + (1 - 2 * t) * back + d,
                                            inv * here + (1 - inv) * bar + d * inv)
        new, rho, u = _trt(p, sp, sm)
        if sol is not None:
            for q in range(f.shape[0]):
                # D2Q9 solid nodes reflect, D3Q19 solid nodes rest
                new[q] = torch.where(sol, p[opp[q]] if k == "trt2d" else
                                     torch.full_like(rho, W[q]), new[q])
            rho = torch.where(sol, torch.ones_like(rho), rho)
            u = [torch.where(sol, torch.zeros_like(rho), a) for a in u]
        f = new
    mom = [rho] + u if (k != "trt3d" or c["moments"]) else []
    return dict(f=_unloaded(c, f), moments=mom)


def _exact_sweep(c, n, seed):
    N, nu, u = _sweep_table(c, seed)
    if len(set(N.tolist())) * c["steps"] > 15000:  # about 20 s
        return None
    ux, uy = [None] * len(N), [None] * len(N)
    for size in sorted(set(N.tolist())):
        ids = [i for i in range(len(N)) if N[i] == size]
        s_nu = torch.tensor([1 / (3 * nu[i] + 0.5) for i in ids], dtype=F64, device="cuda")
        s_nu, ul = s_nu.view(-1, 1, 1), float(u[ids[0]])
        f = _rest((len(ids), size, size), 9)
        for _ in range(c["steps"]):
            d = _pull(f, (0, 0))  # the case axis does not stream
            t = d[:, :, -1].clone()
            rw = t[0] + t[1] + t[3] + 2 * (t[2] + t[5] + t[6])
            d[4, :, -1] = t[2]
            d[8, :, -1] = t[6] - 0.5 * (t[1] - t[3]) + 0.5 * rw * ul
            d[7, :, -1] = t[5] + 0.5 * (t[1] - t[3]) - 0.5 * rw * ul
            rho = d.sum(0)
            da, dg = d[1] + d[2] + d[3] + d[4], d[5] + d[6] + d[7] + d[8]
            x2, y2 = d[5] - d[6] - d[7] + d[8], d[5] + d[6] - d[7] - d[8]
            jx, jy = d[1] - d[3] + x2, d[2] - d[4] + y2
            vx, vy = jx / rho, jy / rho
            r3 = 3 * rho * (vx * vx + vy * vy)
            e = -4 * d[0] - da + 2 * dg
            ep = 4 * d[0] - 2 * da + dg
            e = e - 1.4 * (e + 2 * rho - r3)
            ep = ep - 1.4 * (ep - rho + r3)
            qx, qy = -2 * (d[1] - d[3]) + x2, -2 * (d[2] - d[4]) + y2
            qx, qy = qx - 1.2 * (qx + jx), qy - 1.2 * (qy + jy)
            pd, po = d[1] - d[2] + d[3] - d[4], d[5] - d[6] + d[7] - d[8]
            pd = (pd - s_nu * (pd - rho * (vx * vx - vy * vy))) / 4
            po = (po - s_nu * (po - rho * vx * vy)) / 4
            A, D = rho / 9 - e / 36 - ep / 18, rho / 9 + e / 18 + ep / 36
            ax, ay = (jx - qx) / 6, (jy - qy) / 6
            bx, by = jx / 6 + qx / 12, jy / 6 + qy / 12
            f = torch.stack([(rho - e + ep) / 9, A + ax + pd, A + ay - pd, A - ax + pd,
                             A - ay - pd, D + bx + by + po, D - bx + by - po, D - bx - by + po,
                             D + bx - by - po])
        for k, i in enumerate(ids):
            ux[i], uy[i] = vx[k].cpu().numpy().ravel(), vy[k].cpu().numpy().ravel()
    return dict(ux=np.concatenate(ux), uy=np.concatenate(uy), steps=np.full(len(N), c["steps"]))


def _exact_network(c, n, seed):
    from torch.nn.functional import avg_pool2d, conv2d, interpolate
    p, x, t = _net_inputs(c, seed)
    p = p.to(F64)
    grad = c["mode"] == "grad"
    L, off = [], 0
    for ci, co in _net_layers(c["base"]):
        w = p[off:off + co * 9 * ci].view(co, 3, 3, ci).permute(0, 3, 1, 2).contiguous()
        off += co * 9 * ci
        L.append([w.requires_grad_(grad), p[off:off + co].clone().requires_grad_(grad)])
        off += co
    with torch.set_grad_enabled(grad):
        def conv(i, a, relu=True):
            y = conv2d(a, L[i][0], L[i][1], padding=1)
            return y.relu() if relu else y

        def up(a, skip):
            return torch.cat([interpolate(a, scale_factor=2, mode="nearest"), skip], 1)

        a = x.to(F64).permute(0, 3, 1, 2).contiguous()
        e1 = conv(1, conv(0, a))
        e2 = conv(3, conv(2, avg_pool2d(e1, 2)))
        e3 = conv(5, conv(4, avg_pool2d(e2, 2)))
        y = conv(7, conv(6, avg_pool2d(e3, 2)))
        y = conv(9, conv(8, up(y, e3)))
        y = conv(11, conv(10, up(y, e2)))
        y = conv(13, conv(12, up(y, e1)))
        y = conv(14, y, relu=False)[:, :3]
        sc = torch.tensor(SCALE, dtype=F64, device="cuda").view(1, 3, 1, 1)
        of = torch.tensor(OFFSET, dtype=F64, device="cuda").view(1, 3, 1, 1)
        if not grad:
            return y / sc + of
        loss = ((y - (t.to(F64) - of) * sc) ** 2).mean()
        loss.backward()
    g = torch.cat([torch.cat([w.grad.permute(0, 2, 3, 1).reshape(-1), b.grad]) for w, b in L])
    return dict(loss=loss.detach().view(1), grads=g)
