"""Cases that stand for the work users have this library do.

A case is one pass through public entry points: a number of time steps of a
lattice (context API), of an ensemble or through the reference's drop-in entry
points, or a stretch of closure-network training.  Step counts are those
between two looks at the flow (a program steps, reads the moments, steps on).

Outputs of the context API are the moment fields the call leaves on the device
(lb_device_fields); the populations stay inside the handle and every later
pass on the same state reads them all.  The drop-in cases return the
populations, moments, plot buffer and cursor value, the ensemble its moments
in host memory, training the parameters and the loss log.

exact() restates each path in 64 bits with plain torch.
"""
import ctypes
import importlib.util
import math
import os
import random  # noqa: F401  (draw takes a random.Random)
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "lattibol_0.3.31f_gb300")


def _package():
    name = "lattibol_gb300"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            name, os.path.join(PACKAGE, "__init__.py"), submodule_search_locations=[PACKAGE])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


# Node updates of the largest pass (256^3 nodes for 16 steps, or the headline
# channel for 64).
MOST = 256 ** 3 * 16


def listed():
    return [
        # The lid-driven cavity at its usual size: everything in L2, 20 passes
        # make the 10 000-step run.
        dict(name="cavity2d_256", kind="flow2d", nx=256, ny=256, tau=0.6, lid=0.1, force=0.0,
             steps=500),
        # A 2-D flow past obstacles at the size of the oscillator sample case,
        # between two displays.
        dict(name="flow2d_1568x1024", kind="flow2d", nx=1568, ny=1024, tau=0.7, lid=0.0,
             force=1e-6, steps=100),
        # A handful of steps on a small odd lattice: launches and latency.
        dict(name="flow3d_small", kind="flow3d", nx=45, ny=23, nz=17, tau=0.6, lid=0.05,
             force=1e-5, storage="f32", steps=7),
        # The headline: channel past a sphere, FP32 populations.
        dict(name="channel3d_f32", kind="flow3d", nx=256, ny=128, nz=128, tau=0.55, lid=0.0,
             force=1e-6, storage="f32", steps=64),
        # The same in 16-bit deviation storage.
        dict(name="channel3d_f16", kind="flow3d", nx=256, ny=128, nz=128, tau=0.55, lid=0.0,
             force=1e-6, storage="f16", steps=64),
        # Shan-Chen phase separation, periodic, FP32 and 16-bit storage.
        dict(name="spinodal_f32", kind="spinodal", nx=256, ny=256, nz=256, G=-5.0, storage="f32",
             steps=16),
        dict(name="spinodal_f16", kind="spinodal", nx=256, ny=256, nz=256, G=-5.0, storage="f16",
             steps=16),
        # Independent droplets of many sizes advanced together.
        dict(name="ensemble_64", kind="ensemble", domains=64, side_min=64, side_max=512,
             side_of=32, steps=64),
        # The learned closure on the coarse Taylor-Green grid.
        dict(name="closure_128", kind="closure", nx=128, ny=128, nz=128, steps=32),
        # Training of its network.
        dict(name="train_16384", kind="train", samples=1 << 18, batch=16384, steps=200),
        # The reference's own 3-D host loop (streaming, collision into the plot
        # buffer, cursor value), run inside the library.
        dict(name="dropin3d_fused", kind="dropin3d", nx=256, ny=128, nz=128, tau=0.8, mode="fused",
             steps=32),
        # The reference's 2-D host loop on a multiphase sample case (porous
        # medium), entry point by entry point, in the default drop-in mode.
        dict(name="dropin2d_multiphase", kind="dropin2d", nx=704, ny=440, mode="standalone",
             steps=50),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape3(rng, lo, hi, most):
    while True:
        s = [_log(rng, lo, hi) for _ in range(3)]
        if s[0] * s[1] * s[2] <= most:
            return s


def _steps(rng, nodes, lo, hi):
    return max(1, min(_log(rng, lo, hi), MOST // nodes))


def draw(rng):
    kind = rng.choice(["flow2d", "flow2d", "flow3d", "flow3d", "flow3d", "spinodal", "spinodal",
                       "ensemble", "closure", "train", "dropin3d", "dropin2d"])
    if kind == "flow2d":
        nx, ny = _log(rng, 48, 2048), _log(rng, 48, 2048)
        return dict(kind=kind, nx=nx, ny=ny, tau=round(rng.uniform(0.56, 1.0), 3),
                    lid=rng.choice([0.0, 0.05, 0.1]), force=rng.choice([0.0, 1e-6, 1e-5]),
                    steps=_steps(rng, nx * ny, 20, 500))
    if kind == "flow3d":
        nx, ny, nz = _shape3(rng, 12, 320, 1 << 23)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, tau=round(rng.uniform(0.55, 1.0), 3),
                    lid=rng.choice([0.0, 0.05]), force=rng.choice([0.0, 1e-6, 1e-5]),
                    storage=rng.choice(["f32", "f16", "bf16"]),
                    steps=_steps(rng, nx * ny * nz, 4, 100))
    if kind == "spinodal":
        nx, ny, nz = _shape3(rng, 32, 288, 1 << 24)
        if rng.random() < 0.67:  # most such runs are on round sizes
            nx, ny, nz = 32 * max(1, nx // 32), 8 * max(1, ny // 8), 4 * max(1, nz // 4)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, G=round(rng.uniform(-5.4, -4.7), 3),
                    storage=rng.choice(["f32", "f16", "bf16"]),
                    steps=_steps(rng, nx * ny * nz, 2, 40))
    if kind == "ensemble":
        lo = rng.choice([32, 64, 96])
        return dict(kind=kind, domains=_log(rng, 4, 96), side_min=lo,
                    side_max=lo * rng.randint(2, 4), side_of=rng.choice([32, 32, 16, 1]),
                    steps=_log(rng, 16, 80))
    if kind == "closure":
        nx, ny, nz = _shape3(rng, 24, 160, 1 << 21)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=_log(rng, 4, 32))
    if kind == "train":
        batch = rng.choice([2048, 4096, 10000, 16384])
        return dict(kind=kind, samples=batch * rng.randint(1, 16) + rng.randint(0, 127),
                    batch=batch, steps=_log(rng, 20, 200))
    if kind == "dropin3d":
        nx, ny, nz = _shape3(rng, 16, 256, 1 << 22)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, tau=0.8,
                    mode=rng.choice(["fused", "standalone"]),
                    steps=max(1, _steps(rng, nx * ny * nz, 2, 40) // 2))
    nx, ny = _log(rng, 96, 1024), _log(rng, 96, 768)
    return dict(kind="dropin2d", nx=nx, ny=ny, mode=rng.choice(["standalone", "fused"]),
                steps=_log(rng, 5, 60))


# ------------------------------------------------------------------- inputs

def _modes(rng, shape, n=3):
    """A smooth periodic field of unit size: a few Fourier modes of random
    phase.  shape is (nx, ny[, nz]); x runs fastest."""
    out = np.zeros(shape[::-1])
    for _ in range(n):
        f = np.ones(shape[::-1])
        for a, m in enumerate(shape):
            k, ph = rng.integers(1, 4), rng.uniform(0, 2 * np.pi)
            v = np.sin(2 * np.pi * k * (np.arange(m) + 0.5) / m + ph)
            f = f * v.reshape([-1 if len(shape) - 1 - d == a else 1 for d in range(len(shape))])
        out += rng.uniform(0.5, 1.0) * f
    return (out / n).astype(np.float32).reshape(-1)


def _flow_inputs(case, seed):
    """Density, velocities and wall flags of a flow in full swing: a channel
    walled in y (and z), periodic in x, past a disc or sphere; with a lid the 2-D
    box is a closed cavity under a moving wall, the 3-D channel's top wall moves."""
    rng = np.random.default_rng(seed)
    shape = (case["nx"], case["ny"]) + ((case["nz"],) if "nz" in case else ())
    rho = (1 + 0.01 * _modes(rng, shape)).astype(np.float32)
    u = [0.04 * _modes(rng, shape) for _ in shape]
    solid = np.zeros(shape[::-1], np.uint8)
    ax = np.meshgrid(*[np.arange(m) for m in shape[::-1]], indexing="ij")
    r = max(2, min(shape) // 8)
    centre = [m // 2 for m in shape[::-1]]
    centre[-1] = min(shape[0] // 4 + int(rng.integers(0, 3)), shape[0] - 1)
    if len(shape) == 3 or not case["lid"]:
        solid[sum((a - c) ** 2 for a, c in zip(ax, centre)) <= r * r] = 1
    if len(shape) == 2:
        if case["lid"]:
            solid[:, 0] = solid[:, -1] = 1
        solid[-1, :] = 1
        solid[0, :] = 3 if case["lid"] else 1
    else:
        solid[:, 0, :] = solid[:, -1, :] = 1
        solid[0, :, :] = 1
        solid[-1, :, :] = 3 if case["lid"] else 1
    return rho, u, solid.reshape(-1)


def _spinodal_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n = case["nx"] * case["ny"] * case["nz"]
    return (0.693 * (1 + rng.uniform(-0.01, 0.01, n))).astype(np.float32)


def _closure_inputs(case, seed):
    rng = np.random.default_rng(seed)
    shape = (case["nx"], case["ny"], case["nz"])
    u = [0.05 * _modes(rng, shape) for _ in shape]
    rho = (1 + 0.004 * _modes(rng, shape)).astype(np.float32)
    p = _mlp_params(rng)
    nu0 = np.float32(0.05 * (shape[0] / (2 * np.pi)) / 1600.0)
    return rho, u, p, nu0, np.float32(0.05 * 2 * np.pi / shape[0]), np.float32(200.0)


H, IN = 64, 19


def _mlp_params(rng):
    """Weights of the 19 -> 64 -> 64 -> 1 network: W1, b1, W2, b2, w3, b3."""
    return np.concatenate([
        rng.uniform(-1, 1, H * IN) * math.sqrt(6 / IN), rng.uniform(-0.1, 0.1, H),
        rng.uniform(-1, 1, H * H) * math.sqrt(6 / H), rng.uniform(-0.1, 0.1, H),
        rng.uniform(-1, 1, H) * math.sqrt(3 / H), [0.1]]).astype(np.float32)


def _train_inputs(case, seed):
    """Rows as the closure sees them (stress features and |S| of order one) and
    an eddy viscosity that depends on them."""
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((case["samples"], IN), dtype=np.float32)
    z = (2 * np.abs(x[:, 18]) + np.maximum(x[:, 3], 0) - 0.5 * x[:, 6] ** 2).astype(np.float32)
    return x, z, _mlp_params(rng)


def _ensemble_inputs(case, seed):
    """Droplets at densities near the coexistence pair of a mid-range G."""
    rng = np.random.default_rng(seed)
    # the domain sizes belong to the case: another seed is other droplets
    size_rng = np.random.default_rng(case["domains"] * 7919 + case["side_max"])
    sides = np.arange(case["side_min"], case["side_max"] + 1, case["side_of"])
    nx = size_rng.choice(sides, case["domains"]).astype(np.int32)
    ny = nx.copy()
    G = rng.uniform(-5.2, -4.8, case["domains"]).astype(np.float32)
    rhos = []
    for n in nx:
        y, x = np.mgrid[0:n, 0:n]
        c = rng.uniform(0.3, 0.7, 2) * n
        r = np.hypot(x - c[0], y - c[1])
        rhos.append((1.05 - 0.87 * np.tanh((r - rng.uniform(0.15, 0.25) * n) / 2.0))
                    .astype(np.float32).reshape(-1))
    return nx, ny, G, np.concatenate(rhos)


def _solid_bound(solid, q):
    """The reference's rule: a solid node whose neighbours are all solid, never in the x faces."""
    sb = solid.copy()
    for k in range(q):
        d = C3[k] if q == 19 else (C2[k][0], -C2[k][1])
        sb &= np.roll(solid, [-v for v in reversed(d)], tuple(range(solid.ndim)))
    sb[..., 0] = sb[..., -1] = 0
    return sb


def _dropin3d_inputs(case, seed):
    rng = np.random.default_rng(seed)
    shape = (case["nx"], case["ny"], case["nz"])
    z, y, x = np.meshgrid(*[np.arange(m) for m in shape[::-1]], indexing="ij")
    r = max(2, min(shape) // 8)
    s = ((z == 0) | (z == shape[2] - 1) | (y == 0) | (y == shape[1] - 1)
         | ((x - shape[0] // 4) ** 2 + (y - shape[1] // 2) ** 2 + (z - shape[2] // 2) ** 2
            <= r * r)).astype(np.uint8)
    rho = 1 + 0.002 * _modes(rng, shape)
    u = [0.01 * _modes(rng, shape) for _ in shape]
    return s, _solid_bound(s, 19), _feq(torch.from_numpy(rho).double(),
                                        [torch.from_numpy(v).double() for v in u], C3,
                                        WT3).float().numpy()


def _dropin2d_inputs(case, seed):
    """A droplet of the multiphase samples' fluid (psi = 4 exp(-200 / rho), G =
    -120) among round grains."""
    rng = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    y, x = np.mgrid[0:ny, 0:nx]
    s = np.zeros((ny, nx), np.uint8)
    s[0, :] = s[-1, :] = 1
    for _ in range(12):
        cx, cy = rng.uniform(0.15, 0.85) * nx, rng.uniform(0.1, 0.9) * ny
        s[np.hypot(x - cx, y - cy) <= rng.uniform(0.02, 0.06) * min(nx, ny)] = 1
    r = np.hypot(x - nx / 2, y - ny / 2)
    rho = (305.0 - 219.0 * np.tanh((r - 0.2 * min(nx, ny)) / 3.0)).astype(np.float32)
    rho = np.where(s.astype(bool), np.float32(86.0), rho).astype(np.float32).reshape(-1)
    zero = torch.zeros(nx * ny, dtype=torch.float64)
    f = _feq(torch.from_numpy(rho).double(), [zero, zero], C2, WT2).float().numpy()
    return s, _solid_bound(s, 9), f


# ------------------------------------------------------------------ prepare

class _Field:
    """A float32 device buffer of the library, for torch; keeps its owner alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f4",
                                         "data": (int(ptr), False), "version": 2}


def _tensor(owner, ptr, *shape):
    return torch.as_tensor(_Field(owner, ptr, shape), device="cuda")


def _device_fields(pkg, lat):
    p = [ctypes.c_void_p() for _ in range(4)]
    lat._check(pkg.lib().lb_device_fields(lat.h, *[ctypes.byref(v) for v in p]), "device fields")
    return {n: _tensor(lat, v.value, lat.N)
            for n, v in zip(("rho", "ux", "uy", "uz"), p) if v.value}


def _storage(pkg, case):
    return {"f32": pkg.abi.LB_STORE_F32, "f16": pkg.abi.LB_STORE_F16,
            "bf16": pkg.abi.LB_STORE_BF16}[case["storage"]]


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True)


def prepare(case, seed):
    pkg = _package()
    kind = case["kind"]
    st = {"case": case, "pkg": pkg}
    if kind in ("flow2d", "flow3d"):
        rho, u, flags = _flow_inputs(case, seed)
        q = 9 if kind == "flow2d" else 19
        lat = pkg.Lattice(q, case["nx"], case["ny"], case.get("nz", 1),
                          tau_inv=np.float32(1 / case["tau"]),
                          force=(np.float32(case["force"]), 0, 0), wall_u=(case["lid"], 0, 0),
                          storage=_storage(pkg, case) if q == 19 else pkg.abi.LB_STORE_F32)
        lat.set_flags(flags)
        lat.init_equilibrium(rho, *u)
        st.update(lat=lat, out=_device_fields(pkg, lat))
    elif kind == "spinodal":
        lat = pkg.Lattice(19, case["nx"], case["ny"], case["nz"], tau_inv=np.float32(1.0),
                          G=case["G"], storage=_storage(pkg, case), rho_ref=0.693)
        lat.set_flags(np.zeros(lat.N, np.uint8))
        lat.init_equilibrium(_spinodal_inputs(case, seed))
        st.update(lat=lat, out=_device_fields(pkg, lat))
    elif kind == "closure":
        rho, u, p, nu0, s_ref, z_max = _closure_inputs(case, seed)
        lat = pkg.Lattice(19, case["nx"], case["ny"], case["nz"],
                          tau_inv=np.float32(1 / (0.5 + 3 * nu0)))
        lat.set_flags(np.zeros(lat.N, np.uint8))
        lat.init_equilibrium(rho, *u)
        net = pkg.closure.Mlp(seed=1)
        net.set_params(p)
        lat._check(pkg.lib().lb_closure_enable(lat.h, net.h, nu0, s_ref, z_max, None), "closure")
        lat.net = net  # the network outlives its use
        st.update(lat=lat, out=_device_fields(pkg, lat))
    elif kind == "train":
        x, z, p = _train_inputs(case, seed)
        net = pkg.closure.Mlp(seed=1)
        net.set_params(p)
        dx, dz = pkg.closure.DeviceArray(x.size), pkg.closure.DeviceArray(z.size)
        dx.upload(x)
        dz.upload(z)
        st.update(net=net, dx=dx, dz=dz)
    elif kind == "ensemble":
        nx, ny, G, rho = _ensemble_inputs(case, seed)
        ens = pkg.Ensemble(nx, ny, G)
        ens.init_equilibrium(rho)
        st.update(ens=ens, out=[_pinned(ens.NT) for _ in range(3)])
    elif kind == "dropin3d":
        s, sb, f = _dropin3d_inputs(case, seed)
        d = pkg.DeviceData(19, case["nx"], case["ny"], case["nz"])
        d.set_solid(s.reshape(-1), sb.reshape(-1))
        d.upload(f)
        prm = pkg.abi.lb_run_params_d3q19()
        prm.w0, prm.w1, prm.w7 = (float(w) for w in pkg.W3)
        prm.tau_inv, prm.ux_in, prm.rho_out = np.float32(1 / case["tau"]), 0.01, 1.0
        prm.cursor[0], prm.cursor[1], prm.cursor[2] = _cursor(case)
        st.update(data=d, prm=prm, value=_pinned(4))
    elif kind == "dropin2d":
        s, sb, f = _dropin2d_inputs(case, seed)
        inp = pkg.Input()
        inp.setSolids(s)
        p = inp.p
        p.device_count, p.max_dim, p.update_steps = 1, 1, case["steps"]
        p.ux, p.rho, p.G, p.G_ads = 0.0, 86.0, -120.0, -187.0
        inp.setViscosity(1.0 / 6.0)
        sim = pkg.SimulationD2Q9(inp)
        d = sim.data
        d.upload(f)
        d.set_solid(s.reshape(-1), sb.reshape(-1))
        for n in sim.MOMENTS:
            d.h2d(getattr(d.s, n), np.zeros(d.N, np.float32))
        st.update(sim=sim, data=d)
    return st


def _cursor(case):
    return case["nx"] // 2, case["ny"] // 3, case["nz"] // 2


def _dropin_outputs(st, names):
    d = st["data"]
    out = {"f%d" % k: _tensor(st, getattr(d.s, n), d.N) for k, n in enumerate(d.s.POP)}
    out.update({n: _tensor(st, getattr(d.s, n), d.N) for n in names})
    out["plot"] = _tensor(st, d.plot, d.N, 4)
    out["cursor"] = _tensor(st, d.s.valueCur, 4)
    return out


def run(st):
    case, pkg = st["case"], st["pkg"]
    L, kind = pkg.lib(), case["kind"]
    if "lat" in st:
        st["lat"].step(case["steps"])
        return st["out"]
    if kind == "train":
        log = st["net"].train_device(st["dx"], st["dz"], case["samples"], case["steps"],
                                     case["batch"], np.float32(1e-3), seed=11)
        return {"params": st["net"].params(), "loss": log}
    if kind == "ensemble":
        ens = st["ens"]
        ens.step(case["steps"])
        ens._check(L.lb_ensemble_get_moments(ens.h, *[ctypes.c_void_p(t.data_ptr())
                                                      for t in st["out"]]), "moments")
        return st["out"]
    d = st["data"]
    L.lb_abi_set_mode(pkg.abi.LB_ABI_FUSED if case["mode"] == "fused"
                      else pkg.abi.LB_ABI_STANDALONE)
    if kind == "dropin3d":
        rc = L.lb_run_lbm_d3q19(d.ptr(), ctypes.c_void_p(d.plot), ctypes.byref(st["prm"]),
                                case["steps"], ctypes.c_void_p(st["value"].data_ptr()))
        if rc != pkg.abi.LB_OK:
            raise pkg.LBError(L.lb_abi_last_error().decode())
        return _dropin_outputs(st, ("rho", "ux", "uy", "uz"))
    st["sim"].runLBM(case["steps"])
    return _dropin_outputs(st, ("rho", "ux", "uy"))


# --------------------------------------------------------------------- work

# floating-point operations of one node update (moments, force, relaxation)
FLOPS = {"flow2d": 110, "flow3d": 220, "spinodal": 300, "closure": 520 + 2 * (IN * H + H * H + H),
         "ensemble": 170, "dropin3d": 330, "dropin2d": 240}


def work(case):
    """Each state and field read and written once per pass, the node updates of
    every step."""
    kind = case["kind"]
    if kind == "train":
        rows = min(case["batch"], case["samples"]) * case["steps"]
        # forward, input gradient of layer 2, and the weight gradients
        return {"bytes": 4 * (IN + 1) * rows, "flops": rows * (3 * 2 * (IN * H + H * H + H))}
    if kind == "ensemble":
        nx, ny, _, _ = _ensemble_inputs(dict(case), 0)
        n = int(np.sum(nx.astype(np.int64) * ny))
        per = 2 * 9 * 4 + 3 * 4
    else:
        n = case["nx"] * case["ny"] * case.get("nz", 1)
        q = 9 if kind.endswith("2d") else 19
        size = 2 if case.get("storage", "f32") != "f32" else 4
        per = 2 * q * size + (3 if q == 9 else 4) * 4  # populations in and out, moments
        if kind.startswith("dropin"):
            per += 2 + 16  # solid arrays, plot buffer
        elif kind.startswith("flow"):
            per += 1  # cell flags
    return {"bytes": per * n, "flops": FLOPS[kind] * n * case["steps"]}


# -------------------------------------------------------------------- exact

C3 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0),
      (1, -1, 0), (1, 0, 1), (1, 0, -1), (-1, 1, 0), (-1, -1, 0), (-1, 0, 1), (-1, 0, -1),
      (0, 1, 1), (0, 1, -1), (0, -1, 1), (0, -1, -1)]
C2 = [(0, 0), (1, 0), (0, 1), (-1, 0), (0, -1), (1, 1), (-1, 1), (-1, -1), (1, -1)]
WT3 = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
WT2 = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4


def _opp(c):
    return [c.index(tuple(-v for v in k)) for k in c]


def _feq(rho, u, c, w):
    usq = sum(v * v for v in u)
    out = []
    for k, wk in zip(c, w):
        cu = sum(a * v for a, v in zip(k, u) if a)
        if isinstance(cu, int):
            cu = torch.zeros_like(rho)
        out.append(wk * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * usq))
    return torch.stack(out)


class _Box:
    """Shifts on a periodic lattice stored x fastest (2-D rows run down: +y is
    the row above)."""

    def __init__(self, *shape):
        self.shape, self.dims = shape, shape[::-1]

    def at(self, a, c):
        """a(x + c) at every x."""
        d = c if len(self.shape) == 3 else (c[0], -c[1])
        if not any(d):
            return a
        return torch.roll(a.reshape(self.dims), [-v for v in reversed(d)],
                          tuple(range(len(d)))).reshape(-1)


def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda").double()


def _sum_c(f, c, axis):
    return sum(k[axis] * f[i] for i, k in enumerate(c) if k[axis])


def _native(box, c, w, f, steps, tau_inv, force=None, flags=None, lid=0.0, G=0.0, closure=None):
    """Pull, half-way bounce-back, moments, force and Shan-Chen velocity shifts, BGK."""
    opp, dim = _opp(c), len(c[0])
    wall = None if flags is None else (flags & 1).bool()
    moving = None if flags is None else (flags & 2).bool()
    up = None if wall is None else [box.at(wall, tuple(-v for v in k)) for k in c]
    up_m = None if wall is None else [box.at(moving, tuple(-v for v in k)) for k in c]
    for _ in range(steps):
        g = torch.empty_like(f)
        for k, ck in enumerate(c):
            v = box.at(f[k], tuple(-v for v in ck))
            if wall is not None and k:
                back = f[opp[k]] - up_m[k] * (6 * w[k] * c[opp[k]][0] * lid)
                v = torch.where(up[k], back, v)
            g[k] = v
        rho = g.sum(0)
        u = [_sum_c(g, c, a) / rho for a in range(dim)]
        e = list(u)
        if closure is not None:
            tau_inv = closure(g, rho, u)
        if force:
            e[0] = e[0] + force / (rho * tau_inv)
        if G:
            psi = 1 - torch.exp(-rho)
            ps = [box.at(psi, k) for k in c]
            for a in range(dim):
                e[a] = e[a] - G * psi * sum(w[i] * k[a] * ps[i] for i, k in enumerate(c) if k[a]) \
                    / (rho * tau_inv)
        f_new = g + tau_inv * (_feq(rho, e, c, w) - g)
        if wall is not None:
            f_new = torch.where(wall, f, f_new)
            rho = torch.where(wall, torch.zeros_like(rho), rho)
            u = [torch.where(wall, torch.zeros_like(v), v) for v in u]
        f = f_new
    return dict(zip(("rho", "ux", "uy", "uz"), [rho] + u))


def _network(p, x):
    o = np.cumsum([0, H * IN, H, H * H, H, H, 1])
    w1, b1, w2, b2, w3, b3 = (p[a:b] for a, b in zip(o, o[1:]))
    h = torch.relu(x @ w1.reshape(H, IN).T + b1)
    return torch.relu(h @ w2.reshape(H, H).T + b2) @ w3 + b3


POWERS = [(1, 0, 0), (0, 1, 0), (0, 0, 1), (2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1),
          (0, 1, 1), (1, 2, 0), (1, 0, 2), (2, 1, 0), (0, 1, 2), (2, 0, 1), (0, 2, 1), (2, 2, 0),
          (2, 0, 2), (0, 2, 2)]


def _closure(p, nu0, s_ref, z_max):
    nu0, s_ref, z_max = float(nu0), float(s_ref), float(z_max)
    tau0 = 0.5 + 3 * nu0

    def tau_inv(g, rho, u):
        neq = g - _feq(rho, u, C3, WT3)
        scale = 1 / (rho / 3 * tau0 * s_ref)
        m = []
        for pw in POWERS:
            co = [math.prod(v ** q for v, q in zip(k, pw)) for k in C3]
            m.append(sum(a * neq[i] for i, a in enumerate(co) if a) * scale)
        s = [-0.5 * v for v in m[3:9]]
        m.append(torch.sqrt(2 * (s[0] ** 2 + s[1] ** 2 + s[2] ** 2
                                 + 2 * (s[3] ** 2 + s[4] ** 2 + s[5] ** 2))))
        x = torch.stack(m, 1)
        y = torch.cat([_network(p, r) for r in x.split(1 << 18)])
        return 1 / (0.5 + 3 * (nu0 + nu0 * y.clamp(0, z_max)))
    return tau_inv


def _train(case, x, z, p):
    n, batch = case["samples"], min(case["batch"], case["samples"])
    p = p.clone().requires_grad_(True)
    m1, m2 = torch.zeros_like(p), torch.zeros_like(p)
    mask = (1 << 64) - 1
    s = (11 * 2862933555777941757 + 3037000493) & mask  # the window starts: a 64-bit LCG
    log = []
    lr = float(np.float32(1e-3))
    for t in range(1, case["steps"] + 1):
        s = (s * 6364136223846793005 + 1442695040888963407) & mask
        a = (s >> 17) % (n - batch + 1)
        loss = ((_network(p, x[a:a + batch]) - z[a:a + batch]) ** 2).mean()
        grad, = torch.autograd.grad(loss, p)
        with torch.no_grad():
            m1 = 0.9 * m1 + 0.1 * grad
            m2 = 0.999 * m2 + 0.001 * grad * grad
            p -= lr * (m1 / (1 - 0.9 ** t)) / (torch.sqrt(m2 / (1 - 0.999 ** t)) + 1e-8)
        log.append(loss.detach())
    return {"params": p.detach(), "loss": torch.stack(log)}


def _zou_he_3d(g, west, east, ux_in, rho_out):
    """The reference's velocity inlet and pressure outlet on the x faces."""
    def ty():
        return g[3] + g[15] + g[16] - g[4] - g[17] - g[18]

    def tz():
        return g[5] + g[11] + g[15] - g[6] - g[16] - g[18]

    def put(at, k, v):
        g[k] = torch.where(at, v, g[k])

    flat = g[0] + g[3] + g[4] + g[5] + g[6] + g[15] + g[16] + g[17] + g[18]
    ru = (flat + 2 * (g[2] + g[11] + g[12] + g[13] + g[14])) / (1 - ux_in) * ux_in
    a, b = ty(), tz()
    for k, v in ((1, g[2] + ru / 3), (8, g[11] + ru / 6 + a / 2), (7, g[12] + ru / 6 - a / 2),
                 (9, g[14] + ru / 6 - b / 2), (10, g[13] + ru / 6 + b / 2)):
        put(west, k, v)
    ru = rho_out * (-1 + (flat + 2 * (g[1] + g[7] + g[8] + g[9] + g[10])) / rho_out)
    a = ty()
    for k, v in ((2, g[1] - ru / 3), (11, g[8] - ru / 6 - a / 2), (12, g[7] - ru / 6 + a / 2)):
        put(east, k, v)
    b = tz()  # with the f11 just set, as the reference does
    put(east, 14, g[9] - ru / 6 + b / 2)
    put(east, 13, g[10] - ru / 6 - b / 2)


def _zou_he_2d(g, west, east, ux_in, rho_out):
    def put(at, k, v):
        g[k] = torch.where(at, v, g[k])

    flat = g[0] + g[2] + g[4]
    ru = (flat + 2 * (g[3] + g[7] + g[6])) / (1 - ux_in) * ux_in
    d = 0.5 * (g[2] - g[4])
    put(west, 1, g[3] + ru * 2 / 3)
    put(west, 5, g[7] + ru / 6 - d)
    put(west, 8, g[6] + ru / 6 + d)
    ru = rho_out * (-1 + (flat + 2 * (g[1] + g[5] + g[8])) / rho_out)
    put(east, 3, g[1] - ru * 2 / 3)
    put(east, 7, g[5] - ru / 6 + d)
    put(east, 6, g[8] - ru / 6 - d)


def _reference(box, c, w, f, solid, sb, steps, tau_inv, ux_in, rho_out, cursor, G=0.0, G_ads=0.0):
    """The reference's step: swap streaming with full-way bounce-back stored in
    the solid nodes, Zou-He x faces, BGK; with G < 0 its Shan-Chen pass."""
    opp = _opp(c)
    x = torch.arange(f.shape[1], device=f.device) % box.shape[0]
    west, east = (x == 0) & ~solid, (x == box.shape[0] - 1) & ~solid
    # a pair of slots belongs to the node that streams it
    own = {k for k in (1, 3, 5, 7, 8, 9, 10, 15, 16)} if len(c) == 19 else {1, 2, 5, 6}
    zero = torch.zeros_like(f[0])
    for _ in range(steps):
        g, back = torch.empty_like(f), torch.empty_like(f)
        for k, ck in enumerate(c):
            g[k] = box.at(f[k], tuple(-v for v in ck))
            kept = torch.zeros_like(sb) if k == 0 else sb if k in own else box.at(sb, ck)
            back[k] = torch.where(kept, f[k], box.at(f[opp[k]], ck))
        (_zou_he_3d if len(c) == 19 else _zou_he_2d)(g, west, east, ux_in, rho_out)
        rho = g.sum(0)
        u = [_sum_c(g, c, a) / rho for a in range(len(c[0]))]
        e = list(u)
        if G:
            psi = torch.where(solid, zero, 4 * torch.exp(-200 / rho))
            sd = solid.double()
            for a in range(len(e)):
                e[a] = e[a] - psi * sum(
                    w[i] * k[a] * (G * box.at(psi, k) + G_ads * box.at(sd, k))
                    for i, k in enumerate(c) if k[a]) / (tau_inv * rho)
        f = torch.where(solid, back, g + tau_inv * (_feq(rho, e, c, w) - g))
        rho = torch.where(solid, zero, rho)
        u = [torch.where(solid, zero, v) for v in u]
    uz = u[2] if len(u) == 3 else zero
    plot = torch.stack([u[0], u[1], uz, rho], 1)
    at = 0
    for v, m in zip(reversed(cursor), reversed(box.shape)):
        at = at * m + v
    out = {"f%d" % k: f[k] for k in range(len(c))}
    out.update(dict(zip(("rho", "ux", "uy", "uz"), [rho] + u)))
    out.update(plot=plot, cursor=plot[at])
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("flow2d", "flow3d"):
        rho, u, flags = _flow_inputs(case, seed)
        c, w = (C2, WT2) if kind == "flow2d" else (C3, WT3)
        box = _Box(case["nx"], case["ny"], *([case["nz"]] if kind == "flow3d" else []))
        f = _feq(_gpu(rho), [_gpu(v) for v in u], c, w)
        return _native(box, c, w, f, case["steps"], float(np.float32(1 / case["tau"])),
                       force=float(np.float32(case["force"])),
                       flags=torch.from_numpy(flags).to("cuda"), lid=float(np.float32(case["lid"])))
    if kind == "spinodal":
        rho = _gpu(_spinodal_inputs(case, seed))
        zero = torch.zeros_like(rho)
        return _native(_Box(case["nx"], case["ny"], case["nz"]), C3, WT3,
                       _feq(rho, [zero] * 3, C3, WT3), case["steps"], 1.0,
                       G=float(np.float32(case["G"])))
    if kind == "closure":
        rho, u, p, nu0, s_ref, z_max = _closure_inputs(case, seed)
        f = _feq(_gpu(rho), [_gpu(v) for v in u], C3, WT3)
        return _native(_Box(case["nx"], case["ny"], case["nz"]), C3, WT3, f, case["steps"], None,
                       closure=_closure(_gpu(p), nu0, s_ref, z_max))
    if kind == "train":
        x, z, p = _train_inputs(case, seed)
        return _train(case, _gpu(x), _gpu(z), _gpu(p))
    if kind == "ensemble":
        nx, ny, G, rho = _ensemble_inputs(case, seed)
        parts, at = [], 0
        for m, n, g in zip(nx.tolist(), ny.tolist(), G.tolist()):
            r = _gpu(rho[at:at + m * n])
            at += m * n
            zero = torch.zeros_like(r)
            parts.append(_native(_Box(m, n), C2, WT2, _feq(r, [zero] * 2, C2, WT2),
                                 case["steps"], 1.0, G=g))
        return [torch.cat([d[k] for d in parts]).cpu() for k in ("rho", "ux", "uy")]
    if kind == "dropin3d":
        s, sb, f = _dropin3d_inputs(case, seed)
        return _reference(_Box(case["nx"], case["ny"], case["nz"]), C3, WT3, _gpu(f),
                          _gpu(s).bool().reshape(-1), _gpu(sb).bool().reshape(-1), case["steps"],
                          float(np.float32(1 / case["tau"])), float(np.float32(0.01)), 1.0,
                          _cursor(case))
    s, sb, f = _dropin2d_inputs(case, seed)
    return _reference(_Box(case["nx"], case["ny"]), C2, WT2, _gpu(f), _gpu(s).bool().reshape(-1),
                      _gpu(sb).bool().reshape(-1), case["steps"],
                      float(np.float32(1.0 / (3.0 * float(np.float32(1 / 6)) + 0.5))), 0.0, 86.0,
                      (case["nx"] // 2, case["ny"] // 2), G=-120.0, G_ads=-187.0)
