"""Performance cases: the work a user of coral_b200 has the library do, through
its public entry points, over the sizes and options it is used at.

Kinds of case
  march        the time loop of a driver that steps with march_forward and reads
               the state back (for analysis or a checkpoint) every few steps
  loop         the same through run(): the library's own CFL-controlled loop with
               timeseries objects, one small readback per step
  change_dt    a change of dt and back, each with its refactorisation, as the CFL
               rule causes it in a run whose flow speeds up and slows down
  ensemble     many independent runs advanced together
  transform    the device-to-device inverse transform
  infer, train the learned subgrid closure: inference on a coarse grid, and one
               gradient evaluation of its training

A case names a recipe, a grid (NX, NY Fourier x NZ Chebyshev modes; the physical
grid is 3/2 of it each way) and, for steps, dt and the number of steps per pass.
"""
import ctypes
import math
import os

import numpy as np
import torch

from coral_b200 import CONFIG_DIR, _lib
from coral_b200.closure import Closure
from coral_b200.ensemble import Ensemble, seeded_members
from coral_b200.solver import PlaneLayer

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GOLDEN = os.path.join(ROOT, "tests", "golden")

# recipe: equations file, box length, number of coupled kxky variables, full and
# quadratic variables, kinds of the coupled variables (u velocity, t temperature,
# s and f the velocity's potentials, 0 slaved), the flow's typical velocity,
# command-line switches
RECIPES = {
    "rbc_1e5": (os.path.join(CONFIG_DIR, "rbc_noslip_ra1e5.equations"), 2 * math.pi, 6, 4, 9, "uuu0t0", 30.0,
                None),
    "rbc_1e8": (os.path.join(CONFIG_DIR, "rbc_noslip_ra1e8.equations"), 2 * math.pi, 6, 4, 9, "uuu0t0", 300.0,
                None),
    "rrbc": (os.path.join(CONFIG_DIR, "rrbc_stressfree_ek1e-4_ra5e7.equations"), 2.916396276132465, 6, 4, 9, "uuu0t0",
             100.0, None),
    "penalised": (os.path.join(CONFIG_DIR, "rbc_penalised_ra1e8.equations"), 2 * math.pi, 6, 5, 12, "uuu0t0",
                  100.0, None),
    "smagorinsky": (os.path.join(CONFIG_DIR, "rbc_smagorinsky_ra1e8.equations"), 2 * math.pi, 6, 9, 13, "uuu0t0",
                    100.0, "--withHorizontalSmagorinsky --smagorinsky-prefactor 0.1"),
    # the published rotating-convection benchmark in its two forms
    "bench02_vp": (os.path.join(GOLDEN, "benchmark02", "coral.equations.velocityPressure"), 2.0, 6, 4, 9, "uuu0t0",
                   30.0, None),
    "bench02_tp": (os.path.join(GOLDEN, "benchmark02", "coral.equations.toroidalPoloidal"), 2.0, 3, 4, 9, "sft", 30.0,
                   None),
}
# volume averages of the kinetic-energy terms, horizontal averages of one level
TIMESERIES = (">>Volume_average :: uu <<\n>>Volume_average :: vv <<\n>>Volume_average :: ww <<\n"
              ">>Horizontal_avg :: tFull ;; Position= 1 <<\n>>EOF<<\n")


def listed():
    def step(name, kind, recipe, nx, ny, nz, dt, steps, scheme="ARS_222"):
        return dict(name=name, kind=kind, recipe=recipe, NX=nx, NY=ny, NZ=nz, dt=dt, steps=steps, scheme=scheme)

    return [
        # the smallest run: moderate convection, latency and launches count
        step("rbc_64x64x48", "march", "rbc_1e5", 64, 64, 48, 2e-5, 10),
        # the four-stage scheme on a small grid
        step("rbc_96x96x64_ars443", "march", "rbc_1e5", 96, 96, 64, 2e-5, 6, "ARS_443"),
        # unequal sides, lengths without a compiled FFT plan
        step("rbc_108x64x72", "march", "rbc_1e5", 108, 64, 72, 2e-5, 8),
        # a fine vertical grid on a moderate horizontal one
        step("rbc_128x128x192", "march", "rbc_1e8", 128, 128, 192, 2e-7, 8),
        # production: rotating stress-free convection in the CFL loop with timeseries
        step("rrbc_192x192x96_loop", "loop", "rrbc", 192, 192, 96, 5e-7, 10),
        # the headline configuration, the largest run
        step("rbc_384x384x192", "march", "rbc_1e8", 384, 384, 192, 1e-6, 8),
        # a recipe whose operators are dense in z (potentials, z derivatives)
        step("bench02_tp_96x96x48_loop", "loop", "bench02_tp", 96, 96, 48, 1e-5, 10),
        # the CFL rule's refactorisations
        step("change_dt_128x128x96", "change_dt", "rbc_1e8", 128, 128, 96, 2e-7, 1),
        # a parameter study: 16 independent runs on mixed small grids
        dict(name="ensemble_16", kind="ensemble", members=16, draw_seed=3, dt=1e-5, steps=4),
        # one scalar to physical space, device to device
        dict(name="transform_128x128x96", kind="transform", NX=128, NY=128, NZ=96),
        # the closure on the coarse grid of a 64 x 64 x 48 run; one training batch
        dict(name="closure_infer_64x64x48", kind="infer", NX=64, NY=64, NZ=48),
        dict(name="closure_train_8192", kind="train", NX=64, NY=64, NZ=48, snapshots=4, points=8192),
    ]


# mode counts whose 3/2 multiples are 2^a 3^b, as the grids must be
_SIDES = [16, 24, 32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 216, 256, 288, 324, 384]


def _side(rng, lo, hi):
    """a mode count in [lo, hi], spread over the logarithm"""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min((s for s in _SIDES if lo <= s <= hi), key=lambda s: abs(math.log(s / v)))


def draw(rng):
    kind = rng.choice(["march", "march", "march", "loop", "loop", "change_dt", "ensemble", "transform", "infer",
                       "train"])
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(2, 16), draw_seed=rng.randint(0, 10 ** 6), dt=1e-5,
                    steps=rng.randint(2, 4))
    if kind == "transform":
        return dict(kind=kind, NX=_side(rng, 16, 128), NY=_side(rng, 16, 128), NZ=_side(rng, 16, 96))
    if kind == "infer":
        return dict(kind=kind, NX=_side(rng, 16, 96), NY=_side(rng, 16, 96), NZ=_side(rng, 16, 72))
    if kind == "train":
        return dict(kind=kind, NX=_side(rng, 24, 72), NY=_side(rng, 24, 72), NZ=_side(rng, 16, 48),
                    snapshots=rng.randint(1, 6), points=int(math.exp(rng.uniform(math.log(500), math.log(20000)))))
    recipe = rng.choice(["rbc_1e5", "rbc_1e5", "rbc_1e8", "rbc_1e8", "rrbc", "penalised", "smagorinsky", "bench02_vp",
                         "bench02_tp"])
    fine = recipe in ("rbc_1e8", "rrbc", "penalised", "smagorinsky")  # strongly driven: short steps
    while True:
        nx, ny, nz = _side(rng, 24, 288), _side(rng, 24, 288), _side(rng, 24, 192)
        if nx * ny * nz <= (3 << 20):
            break
    return dict(kind=kind, recipe=recipe, NX=nx, NY=ny, NZ=nz, dt=2e-7 if fine else 5e-6,
                steps=1 if kind == "change_dt" else rng.randint(3, 10),
                scheme=rng.choice(["ARS_222", "ARS_222", "ARS_443"] + ([] if fine else ["ARS_111"])))


# ---- inputs ---------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _parameters(case):
    L = RECIPES[case["recipe"]][1]
    return ("0\n%d\n%d\n%d\n0\n%r\n%r\n1.d0\n0.5d0\n0\n%r\n0.3d0\n0.5d0\n'%s'\n0\n.True.\n0\n1.d9\n"
            % (case["NX"], case["NY"], case["NZ"], L, L, case["dt"], case["scheme"]))


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def _starting_state(pl, kinds, U, g):
    """A developed-flow-like state for every coupled system: random phases under
    a spectrum that decays in kx, ky and the Chebyshev degree, Hermitian on the
    kx = 0 line, nothing in the dealiased modes.  U: root mean square of a
    velocity component, about.  Returns the page-locked read-back buffers."""
    dev = "cuda"
    NX, NYAA, NXH = pl.NX, pl.NYAA, pl.NXH
    NY = 2 * NYAA // 3
    iy = torch.arange(NYAA, device=dev)
    ky = torch.where(iy <= NYAA // 2, iy, iy - NYAA).double()
    kx = torch.arange(NXH, device=dev).double()
    kcx, kcy, nc = NX / 12.0, NY / 12.0, pl.NZ / 8.0
    horizontal = torch.exp(-kx / kcx)[:, None] * torch.exp(-ky.abs() / kcy)[None, :]
    horizontal[:, ky.abs() >= NY // 2] = 0.0
    horizontal[0, 0] = 0.0
    unit = 1.0 / math.sqrt(2.0 * max(kcx * kcy * nc / 4.0, 1.0))
    amplitude = {"u": U, "0": 0.0, "t": 0.01, "s": 0.3 * U / max(kcx, kcy), "f": 0.03 * U / max(kcx, kcy) ** 2}
    out = {}
    for s in range(pl.n_kxky):
        T = pl.T[s]
        a = torch.zeros(T, device=dev, dtype=torch.float64)
        for v in range(pl.query(300 + s)):
            pos = torch.from_numpy(pl.var_positions(s, v).astype(np.int64)).to(dev)
            a[pos] = amplitude[kinds[v]] * torch.exp(-torch.arange(len(pos), device=dev).double() / nc)
        f = torch.randn((NXH, NYAA, T), dtype=torch.complex128, device=dev, generator=g)
        f *= unit * horizontal[:, :, None]
        f *= a
        mirror = (-iy) % NYAA
        f[0] = 0.5 * (f[0] + f[0, mirror].conj())
        buf = _pinned((NXH, NYAA, T), torch.complex128)
        buf.copy_(f)
        del f
        pl.set_field(s, buf.numpy())
        out["field%d" % s] = buf
    for s in range(pl.n_zero):
        n = torch.arange(pl.Tz[s], device=dev).double()
        z = 0.01 * torch.randn(pl.Tz[s], dtype=torch.float64, device=dev, generator=g) * torch.exp(-n / nc)
        pl.set_mean_field(s, z.cpu().numpy())
    return out


def prepare(case, seed):
    g, kind = _generator(seed), case["kind"]
    if kind in ("march", "loop", "change_dt"):
        path, _, _, _, _, kinds, U, args = RECIPES[case["recipe"]]
        with open(path) as f:
            equations = f.read()
        pl = PlaneLayer(equations, _parameters(case), args=args)
        if kind == "loop":
            pl.set_timeseries(TIMESERIES)
        # long runs remove the invisible anti-Hermitian part of the kx = 0 line
        pl.set_hermitian_kx0(True)
        out = _starting_state(pl, kinds, U, g)
        pl.factorize_operators(case["dt"])
        return dict(kind=kind, pl=pl, out=out, dt=case["dt"], steps=case["steps"])
    if kind == "ensemble":
        spec = seeded_members(case["members"], seed=case["draw_seed"], dt=case["dt"])
        ens = Ensemble([s[0] for s in spec], [s[1] for s in spec])
        outs = [_starting_state(m, "uuu0t0", 30.0, g) for m in ens.members]
        return dict(kind=kind, ens=ens, out=outs, dt=case["dt"], steps=case["steps"])
    if kind == "transform":
        NX, NY, NZ = case["NX"], case["NY"], case["NZ"]
        return dict(kind=kind, n=(NX, NY, NZ), spec=_spectrum(case, seed),
                    phys=torch.empty((3 * NY // 2, 3 * NX // 2, 3 * NZ // 2), dtype=torch.float64, device="cuda"))
    grid = (3 * case["NY"] // 2, 3 * case["NX"] // 2, 3 * case["NZ"] // 2)
    net, weights, scales = _network(seed)
    if kind == "infer":
        return dict(kind=kind, net=net, fields=_fields(grid, g),
                    tau=torch.empty((9,) + grid, dtype=torch.float64, device="cuda"))
    inputs, targets, points = _batch(case, grid, g)
    return dict(kind=kind, net=net, inputs=inputs, targets=targets, points=points)


def _spectrum(case, seed):
    NX, NY, NZ = case["NX"], case["NY"], case["NZ"]
    NYAA = 3 * NY // 2
    iy = torch.arange(NYAA, device="cuda")
    ky = torch.where(iy <= NYAA // 2, iy, iy - NYAA).abs().double()
    s = torch.randn((NX // 2, NYAA, NZ), dtype=torch.complex128, device="cuda", generator=_generator(seed))
    s *= torch.exp(-12.0 * torch.arange(NX // 2, device="cuda") / NX)[:, None, None]
    s *= (torch.exp(-12.0 * ky / NY) * (ky < NY // 2))[None, :, None]
    s *= torch.exp(-8.0 * torch.arange(NZ, device="cuda") / NZ)
    return s


# ---- the closure network's inputs: weights as after training, fields of order one ------
_LAYERS = ((64, 135), (64, 64), (64, 64), (9, 64))


def _network(seed):
    """the network with its parameters and scales set; the parameters as (W, b)
    pairs in float32 and the scales, for exact()"""
    r = np.random.default_rng(seed)
    flat, layers = [], []
    for o, i in _LAYERS:
        W = (r.uniform(-1, 1, (o, i)) * math.sqrt(6.0 / (o + i))).astype(np.float32)
        b = (0.05 * r.standard_normal(o)).astype(np.float32)
        layers.append((W, b))
        flat += [W.ravel(), b]
    ins = [float(np.float32(v)) for v in r.uniform(0.5, 1.5, 4)]
    outs = [float(np.float32(v)) for v in r.uniform(0.5, 2.0, 9)]
    net = Closure(seed=1)
    net.set_scales(ins, outs)
    net.set_params(np.concatenate(flat))
    return net, layers, (ins, outs)


def _fields(grid, g):
    return torch.randn((4,) + grid, dtype=torch.float64, device="cuda", generator=g)


def _batch(case, grid, g):
    n = case["snapshots"]
    inputs = torch.randn((n, 4) + grid, dtype=torch.float32, device="cuda", generator=g)
    targets = torch.randn((n, 9) + grid, dtype=torch.float32, device="cuda", generator=g)
    points = torch.randint(0, n * math.prod(grid), (case["points"],), device="cuda", generator=g)
    return inputs, targets, points


# ---- one pass -------------------------------------------------------------------------
def _read(pl, out):
    got = {}
    for s in range(pl.n_kxky):
        pl.get_field(s, out=out["field%d" % s].numpy())
        got["field%d" % s] = out["field%d" % s]
    for s in range(pl.n_zero):
        got["mean%d" % s] = pl.get_mean_field(s)
    return got


def run(state):
    kind = state["kind"]
    if kind == "march":
        state["pl"].march_forward(state["dt"], state["steps"])
        return _read(state["pl"], state["out"])
    if kind == "loop":
        pl = state["pl"]
        pl.run(state["steps"])
        return dict(_read(pl, state["out"]), timeseries=pl.timeseries())
    if kind == "change_dt":
        pl, dt, n = state["pl"], state["dt"], state["steps"]
        pl.march_forward(0.6 * dt, n)
        pl.march_forward(dt, n)
        return _read(pl, state["out"])
    if kind == "ensemble":
        state["ens"].march_forward(state["dt"], state["steps"])
        state["ens"].synchronize()
        return [_read(m, o) for m, o in zip(state["ens"].members, state["out"])]
    if kind == "transform":
        D = ctypes.POINTER(ctypes.c_double)
        NX, NY, NZ = state["n"]
        rc = _lib.load().coral_spec_to_phys_noalloc(
            NX, NY, NZ, ctypes.cast(state["spec"].data_ptr(), D), ctypes.cast(state["phys"].data_ptr(), D),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError("coral_spec_to_phys_noalloc: %d" % rc)
        return state["phys"]
    net = state["net"]
    if kind == "infer":
        net.infer(state["fields"], state["tau"], stream=torch.cuda.current_stream().cuda_stream)
        # the network computes in FP32 and tau holds its values widened: as what they are
        return state["tau"].float()
    net.zero_gradient()
    loss = net.train(state["inputs"], state["targets"], state["points"], apply=False)
    return dict(loss=torch.tensor(loss, dtype=torch.float32), gradient=net.gradient())


# ---- the work a pass cannot do without ------------------------------------------------
def _step_work(nx, ny, nz, nvars, nfull, nquad, stages, steps):
    """per stage: the state read and written once, and the 3-D transforms of the
    full and quadratic variables (2.5 N log2 N operations each)"""
    state = 16.0 * (nx / 2) * (1.5 * ny) * nz * nvars
    n = 1.5 ** 3 * nx * ny * nz
    return 2 * state * stages * steps, 2.5 * n * math.log2(n) * (nfull + nquad) * stages * steps


def work(case):
    kind = case["kind"]
    if kind in ("march", "loop", "change_dt"):
        _, _, nv, nf, nq, _, _, _ = RECIPES[case["recipe"]]
        stages = int(case["scheme"][-1])  # implicit stages: ARS_111 1, ARS_222 2, ARS_443 3 (+ the last update)
        stages = {1: 1, 2: 2, 3: 4}[stages]
        b, f = _step_work(case["NX"], case["NY"], case["NZ"], nv, nf, nq, stages,
                          case["steps"] * (2 if kind == "change_dt" else 1))
        return dict(bytes=b, flops=f)
    if kind == "ensemble":
        b = f = 0.0
        for _, _, grid, _, _ in seeded_members(case["members"], seed=case["draw_seed"], dt=case["dt"]):
            x = _step_work(*grid, 6, 4, 9, 2, case["steps"])
            b, f = b + x[0], f + x[1]
        return dict(bytes=b, flops=f)
    n = 1.5 ** 3 * case["NX"] * case["NY"] * case["NZ"]
    if kind == "transform":
        return dict(bytes=16.0 * case["NX"] / 2 * 1.5 * case["NY"] * case["NZ"] + 8 * n, flops=2.5 * n * math.log2(n))
    params = sum(o * i + o for o, i in _LAYERS)
    if kind == "infer":
        return dict(bytes=(4 + 9) * 8 * n, flops=2.0 * params * n)
    return dict(bytes=case["points"] * 4.0 * (27 * 4 + 9), flops=6.0 * params * case["points"])


# ---- what a pass returns, in 64 bits by plain torch -----------------------------------
def _stencil(fields, points, in_scale):
    """(npoints, 135) inputs of the network: channel c of 5, tap (dy, dx, dz);
    periodic in x and y, zero beyond the walls"""
    _, NYA, NXA, NZA = fields.shape
    z, x, y = points % NZA, (points // NZA) % NXA, points // (NZA * NXA)
    zeta = torch.cos(math.pi * (2 * torch.arange(1, NZA + 1, device="cuda").double() - 1) / (2 * NZA))
    cols = [[] for _ in range(5)]
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            for dz in (-1, 0, 1):
                zz = z + dz
                inside = (zz >= 0) & (zz < NZA)
                zc = zz.clamp(0, NZA - 1)
                yy, xx = (y + dy) % NYA, (x + dx) % NXA
                for c in range(4):
                    cols[c].append(fields[c, yy, xx, zc] * in_scale[c] * inside)
                cols[4].append(zeta[zc] * inside)
    return torch.stack([t for c in cols for t in c], dim=1)


def _layers64(layers):
    """weights as the network uses them (rounded to bfloat16), biases in float32, both widened"""
    return [(torch.from_numpy(W).cuda().bfloat16().double(), torch.from_numpy(b).cuda().double()) for W, b in layers]


def _forward(layers, X):
    acts = [X]
    for k, (W, b) in enumerate(layers):
        a = acts[-1] @ W.T + b
        acts.append(torch.tanh(a) if k < 3 else a)
    return acts


def exact(case, seed):
    kind = case["kind"]
    if kind == "transform":
        spec = _spectrum(case, seed)
        NXAA, NZ, NZAA = 3 * case["NX"] // 2, case["NZ"], 3 * case["NZ"] // 2
        f = torch.fft.ifft(spec, dim=1, norm="forward")          # y, e^{+i ky y}
        f = torch.fft.irfft(f, n=NXAA, dim=0, norm="forward")    # x
        k = torch.arange(NZAA, dtype=torch.int64, device="cuda")
        n = torch.arange(NZ, dtype=torch.int64, device="cuda")
        angle = (n[:, None] * (2 * k[None, :] + 1)) % (4 * NZAA)  # cos(pi n (k + 1/2) / NZAA), reduced exactly
        return (f @ torch.cos(angle.double() * (math.pi / (2 * NZAA)))).permute(1, 0, 2).contiguous()
    if kind not in ("infer", "train"):
        return None  # whole time steps: no 64-bit restatement but the library's own
    g = _generator(seed)
    grid = (3 * case["NY"] // 2, 3 * case["NX"] // 2, 3 * case["NZ"] // 2)
    _, layers, (ins, outs) = _network(seed)
    layers, outs = _layers64(layers), torch.tensor(outs, dtype=torch.float64, device="cuda")
    if kind == "infer":
        fields, tau = _fields(grid, g), []
        for points in torch.arange(math.prod(grid), device="cuda").split(1 << 17):
            tau.append(_forward(layers, _stencil(fields, points, ins))[-1] * outs)
        return torch.cat(tau).T.reshape((9,) + grid).contiguous()
    inputs, targets, points = _batch(case, grid, g)
    n = math.prod(grid)
    fields = inputs.double().transpose(0, 1).reshape(4, -1)
    snap, lin = points // n, points % n
    X = torch.empty((len(points), 135), dtype=torch.float64, device="cuda")
    want = torch.empty((len(points), 9), dtype=torch.float64, device="cuda")
    for s in range(case["snapshots"]):
        at = snap == s
        X[at] = _stencil(inputs[s].double(), lin[at], ins)
        want[at] = targets[s].reshape(9, -1)[:, lin[at]].T.double() / outs
    acts = _forward(layers, X)
    d = acts[-1] - want
    delta, grads = 2.0 * d / len(points), []
    for k in (3, 2, 1, 0):
        W, _ = layers[k]
        grads.insert(0, torch.cat([(delta.T @ acts[k]).reshape(-1), delta.sum(0)]))
        if k:
            delta = (delta @ W) * (1.0 - acts[k] ** 2)
    return dict(loss=(d * d).sum() / len(points), gradient=torch.cat(grads))
