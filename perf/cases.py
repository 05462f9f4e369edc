"""The work that users of the framework have it do, as measurable cases.

A run of the solver is: a context or an ensemble is created and given a velocity
field, it is advanced by the steps between two snapshots, and the snapshot is
brought to the host (the last step of the interval is `step_host` with an output
array, which is page-locked as the API asks for its fast path). FP32 contexts hand
their snapshots on in single precision, the precision they hold.

Kinds of a case (`kind`):
  run       advance one context by `steps` and bring the snapshot back
  host      one step through host arrays in and out (RK4Step's contract)
  ensemble  a device-side run of several contexts, every member's state back
  output    what is written at a save: the measurables and the real-space fields
  closure   the learned subgrid closure: gradients of one sample, and one inference
"""
import importlib
import math
import os

import numpy as np
import torch

ns3d = importlib.import_module("3d_navier_stokes_gb300")
SHAPES = os.path.join(os.path.dirname(os.path.abspath(ns3d.__file__)), "tuning", "gb300.txt")


def _run(name, N, precision, integrator, steps, **kw):
    c = {"name": name, "kind": "run", "N": N, "precision": precision, "integrator": integrator, "steps": steps,
         "visc_pow": 1, "forcing": "", "cfl": 0.0}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest grid in use: a teaching or debugging run of the reference's own
        # RK4Step in its own precision, where launches and latency count
        _run("f64 rk4cn 32", 32, "fp64", "rk4cn", 100),
        # adaptive Dormand-Prince at a size with a factor 3, in the reference's precision
        _run("f64 dp5cn 96", 96, "fp64", "dp5cn", 6),
        # forced, CFL-controlled turbulence in double precision, an ordinary size
        _run("f64 ifrk4 forced 128", 128, "fp64", "ifrk4", 10, forcing="SHELL", cfl=0.5),
        # the reference's RK4Step in its own precision at a production size
        _run("f64 rk4cn 256", 256, "fp64", "rk4cn", 6),
        # RK4Step's host-array contract (u_hat in, u_hat out), a 3 x 2^k size
        {"name": "f64 host step 192", "kind": "host", "N": 192, "precision": "fp64", "integrator": "rk4cn",
         "visc_pow": 1, "forcing": "", "cfl": 0.0},
        # small FP32 run: parameter sweeps and tests
        _run("f32 ifrk4 64", 64, "fp32", "ifrk4", 100),
        # fifth order with hyperviscosity, a 3 x 2^k size that no tuning entry covers
        _run("f32 rk5cn 192 hyper", 192, "fp32", "rk5cn", 10, visc_pow=2),
        # forced turbulence at the DNS size of the closure's training data
        _run("f32 ifrk4 forced 256", 256, "fp32", "ifrk4", 20, forcing="SHELL", cfl=0.5),
        # the headline workload: forced 512^3 turbulence, CFL 0.5
        _run("f32 ifrk4 forced 512", 512, "fp32", "ifrk4", 10, forcing="SHELL", cfl=0.5),
        # a mixed-size ensemble, the whole run in one device-side loop
        {"name": "ensemble f32 48-96", "kind": "ensemble", "sizes": "48 64 96", "each": 8, "precision": "fp32",
         "integrator": "ifrk4", "steps": 100},
        # a save: totals and spectra, and the real-space velocity and vorticity
        {"name": "output f64 128", "kind": "output", "N": 128, "precision": "fp64"},
        # the closure's training direction and its inference on the grid it is used at
        {"name": "closure 64", "kind": "closure", "N": 64},
    ]


# relative cost of one step (the work of one evaluation of the nonlinear term, FP64
# arithmetic weighted), used to keep drawn cases within the listed ones
def _step_cost(N, precision, integrator):
    evals = {"ifrk4": 4, "rk4cn": 4, "rk5cn": 6, "dp5cn": 7}[integrator]
    return evals * N ** 3 * math.log2(N) * (16 if precision == "fp64" else 1)


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["host", "host", "ensemble", "output", "closure"])
    if kind == "closure":
        return {"kind": kind, "N": rng.choice([16, 32, 64]), "sample": rng.randrange(1 << 20)}
    if kind == "ensemble":
        sizes = rng.choice(["32 48", "48 64", "64 96", "48 96", "32 64 96", "48 64 96"])
        return {"kind": kind, "sizes": sizes, "each": rng.randint(2, 8), "precision": "fp32",
                "integrator": rng.choice(["ifrk4", "rk4cn"]), "steps": round(math.exp(rng.uniform(math.log(10), math.log(100))))}
    precision = rng.choice(["fp64", "fp32"])
    if kind == "output":
        return {"kind": kind, "N": rng.choice([32, 48, 64, 96, 128]), "precision": precision,
                "sample": rng.randrange(1 << 20)}
    if precision == "fp64":
        N = rng.choice([24, 32, 48, 64, 96, 128, 192, 256])
    else:
        N = rng.choice([32, 48, 64, 96, 128, 192, 256, 384, 512])
    integrator = rng.choice(["ifrk4", "rk4cn", "rk5cn"] + (["dp5cn"] if kind == "run" and precision == "fp64" else []))
    fixed = integrator == "dp5cn"
    c = {"kind": kind, "N": N, "precision": precision, "integrator": integrator,
         "visc_pow": rng.choice([1, 1, 2]), "forcing": rng.choice(["", "SHELL"]),
         "cfl": 0.0 if fixed else rng.choice([0.0, 0.4, 0.5, 0.6])}
    if kind == "run":
        most = _step_cost(256, "fp64", "rk4cn") * 6 if precision == "fp64" else _step_cost(512, "fp32", "ifrk4") * 10
        top = max(1, min(100 if not fixed else 8, int(most / _step_cost(N, precision, integrator))))
        c["steps"] = max(1, round(math.exp(rng.uniform(math.log(max(1, top / 4)), math.log(top)))))
    else:
        c["sample"] = rng.randrange(1 << 20)
    return c


# ---------------------------------------------------------------- inputs
def _grid(N, dev):
    k = torch.fft.fftfreq(N, 1.0 / N, device=dev, dtype=torch.float64)
    return k[:, None, None], k[None, :, None], torch.arange(N // 2 + 1, device=dev, dtype=torch.float64)


def _k2(N, dev):
    kx, ky, kz = _grid(N, dev)
    return kx * kx + ky * ky + kz * kz


def _mask(N, dev):
    return _k2(N, dev) <= float((N // 3) ** 2)


def _project(f, N):
    """Leray projection of f[..., 3, N, N, N/2+1], dealiased, zero mean."""
    kx, ky, kz = _grid(N, f.device)
    k2 = _k2(N, f.device)
    keep = (k2 <= float((N // 3) ** 2)) & (k2 > 0)
    d = (f[..., 0, :, :, :] * kx + f[..., 1, :, :, :] * ky + f[..., 2, :, :, :] * kz) / k2.clamp(min=1.0)
    out = torch.stack([f[..., 0, :, :, :] - d * kx, f[..., 1, :, :, :] - d * ky, f[..., 2, :, :, :] - d * kz], dim=-4)
    return out * keep


def _velocity(N, seed):
    """A turbulent solenoidal velocity with a developed spectrum, E(k) = k^4 (k0^2 + k^2)^(-17/6)
    rolled off at the dealiasing radius, and half its mean square 1; unnormalised transform [3, N, N, N/2+1]."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + N)
    f = torch.empty(3, N, N, N // 2 + 1, dtype=torch.complex128, device="cuda")
    for c in range(3):
        f[c] = torch.fft.rfftn(torch.randn(N, N, N, dtype=torch.float64, device="cuda", generator=g))
    k2 = _k2(N, "cuda")
    k = k2.sqrt()
    f *= torch.sqrt(k2 * (4.0 + k2) ** (-17.0 / 6.0) * torch.exp(-4.0 * k / (N // 3)))
    f = _project(f, N)
    w = torch.full((N // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
    w[0] = 1.0
    e = 0.5 * sum(((f[c].real ** 2 + f[c].imag ** 2) * w).sum() for c in range(3)) / float(N) ** 6
    return f * (1.0 / e.sqrt())


def _options(case, N):
    """Viscosity and step of a resolved run on this grid."""
    nu = 0.5 / N
    if case.get("visc_pow", 1) == 2:
        nu /= (N / 3.0) ** 2
    dt = 0.05 / N if case["integrator"] != "dp5cn" else 0.02 / N
    kw = {"nu": nu, "dt": dt, "integrator": case["integrator"], "precision": case["precision"],
          "visc_pow": case.get("visc_pow", 1), "cfl": case.get("cfl", 0.0)}
    if case.get("forcing"):
        kw["forcing"] = case["forcing"]
    return kw


def _to_host(f):
    """Page-locked host array in the reference layout [N][N][N/2+1][3]."""
    host = torch.empty(tuple(f.shape[1:]) + (3,), dtype=torch.complex128, pin_memory=True)
    host.copy_(f.permute(1, 2, 3, 0).contiguous())
    return host


def _closure_inputs(case, seed):
    D = case["N"]
    u = torch.fft.irfftn(_velocity(D, seed + case.get("sample", 0)), s=(D, D, D), dim=(1, 2, 3))
    tau = torch.stack([u[a] * u[b] for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]) * 0.05
    return u.float().cpu().numpy(), tau.float().cpu().numpy()


def prepare(case, seed):
    ns3d.tuning_load(SHAPES)   # the shapes that ship with the package
    if case["kind"] == "closure":
        les = ns3d.LES(case["N"], capacity=0, seed=seed)   # its own initial weights
        les.set_scales(0.8, 0.05)
        u, tau = _closure_inputs(case, seed)
        return {"kind": "closure", "les": les, "u": u, "tau": tau}
    if case["kind"] == "ensemble":
        members = []
        for N in map(int, case["sizes"].split()):
            for i in range(case["each"]):
                kw = _options(case, N)
                kw["nu"] *= 1.0 + 0.1 * i
                members.append(dict(kw, N=N))
        ens = ns3d.Ensemble(members)
        for i, m in enumerate(members):
            ens.set_state(i, _to_host(_velocity(m["N"], seed * 64 + i)).numpy())
        torch.cuda.synchronize()
        return {"kind": "ensemble", "ens": ens, "count": len(members), "steps": case["steps"]}
    N = case["N"]
    if case["kind"] == "output":
        case = dict(case, integrator="ifrk4")
    s = ns3d.Solver(N, **_options(case, N))
    host = _to_host(_velocity(N, seed + case.get("sample", 0)))
    st = {"kind": case["kind"], "solver": s, "single": case["precision"] == "fp32", "steps": case.get("steps", 1)}
    if case["kind"] == "host":
        st["in"] = host.numpy()
        st["out"] = torch.empty_like(host, pin_memory=True)
        if case.get("forcing"):
            s.set_state(st["in"])   # the forcing holds this field's energy
    else:
        s.set_state(host.numpy())
        torch.cuda.synchronize()
        st["out"] = host            # read already; now it receives the snapshots
    return st


def run(st):
    if st["kind"] == "closure":
        loss, grads = st["les"].gradients(st["u"], st["tau"])
        return {"loss": loss, "grads": grads, "tau": st["les"].infer(st["u"])}
    if st["kind"] == "ensemble":
        st["ens"].run(st["steps"])
        return [torch.from_numpy(st["ens"].get_state(i)).to(torch.complex64) for i in range(st["count"])]
    s = st["solver"]
    if st["kind"] == "output":
        totals, ek, ok = s.ComputeSystemMeasurables()
        u, w = s.real_space()
        fields = {"totals": np.array([totals[k] for k in sorted(totals)]), "ek": ek, "ok": ok, "u": u, "w": w}
        return {k: torch.from_numpy(v).to(torch.float32) for k, v in fields.items()} if st["single"] else fields
    if st["kind"] == "host":
        s.step_host(st["in"], st["out"].numpy())
    else:
        if st["steps"] > 1:
            s.RK4Step(st["steps"] - 1)
        s.step_host(None, st["out"].numpy())
    if st["single"]:
        return st["out"].to("cuda", non_blocking=True).to(torch.complex64)
    return st["out"].numpy()


# ------------------------------------------------------------------ work
def _sphere(N):
    """Modes inside the dealiasing sphere with kz >= 0."""
    return 2.0 / 3.0 * math.pi * (N // 3) ** 3 + math.pi * (N // 3) ** 2 / 2 + 1


def _evaluations(integrator):
    return {"ifrk4": 4, "rk4cn": 4, "rk5cn": 6, "dp5cn": 7}[integrator]


def _eval_flops(N):
    return 9 * 2.5 * N ** 3 * 3 * math.log2(N)   # six inverse and three forward real transforms


def work(case):
    if case["kind"] == "closure":
        p = case["N"] ** 3
        layers = 2 * 27 * (3 * 32 + 32 * 32 + 32 * 32 + 32 * 6) * p
        # forward, weight gradients, and input gradients of all but the first layer; then an inference
        return {"bytes": 4.0 * p * (3 + 6 + 3 + 6) + 8.0 * 62000, "flops": 3 * layers - 2.0 * 27 * 3 * 32 * p + layers}
    if case["kind"] == "ensemble":
        b = f = 0.0
        for N in map(int, case["sizes"].split()):
            n = _evaluations(case["integrator"]) * case["steps"]
            b += case["each"] * (n * 2 * 3 * 8 * _sphere(N) + 48.0 * N * N * (N // 2 + 1))
            f += case["each"] * n * _eval_flops(N)
        return {"bytes": b, "flops": f}
    N = case["N"]
    w = 16 if case["precision"] == "fp64" else 8
    if case["kind"] == "output":
        return {"bytes": 3.0 * w * _sphere(N) + 2 * 24.0 * N * N * (N + 2), "flops": 6 * 2.5 * N ** 3 * 3 * math.log2(N)}
    # each evaluation reads the three fields' modes and writes them; the snapshot crosses the link once
    # (its modes inside the sphere, and the rest of the host array is written as zeros)
    n = _evaluations(case["integrator"]) * case.get("steps", 1)
    bytes_ = n * 2 * 3 * w * _sphere(N) + 48.0 * N * N * (N // 2 + 1)
    if case["kind"] == "host":
        bytes_ += 48.0 * _sphere(N)
    return {"bytes": bytes_, "flops": n * _eval_flops(N)}


# ----------------------------------------------------------------- exact
_A = [[1 / 5],
      [3 / 40, 9 / 40],
      [44 / 45, -56 / 15, 32 / 9],
      [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
      [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
      [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
_B = [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84, 0]
_BS = [5179 / 57600, 0, 7571 / 16695, 393 / 640, -92097 / 339200, 187 / 2100, 1 / 40]


def _real(f, N):
    return torch.stack([torch.fft.irfftn(f[c], s=(N, N, N)) for c in range(3)])


def _curl(f, N):
    kx, ky, kz = _grid(N, f.device)
    return torch.stack([1j * (ky * f[2] - kz * f[1]), 1j * (kz * f[0] - kx * f[2]), 1j * (kx * f[1] - ky * f[0])])


def _nonlinear(f, N):
    """(P[FFT(u x w)] dealiased, max(|u| + |v| + |w|))"""
    u, w = _real(f, N), _real(_curl(f, N), N)
    prod = torch.stack([torch.fft.rfftn(u[1] * w[2] - u[2] * w[1]), torch.fft.rfftn(u[2] * w[0] - u[0] * w[2]),
                        torch.fft.rfftn(u[0] * w[1] - u[1] * w[0])])
    return _project(prod, N), float(u.abs().sum(0).max())


def _shell(f, N, kf):
    k2 = _k2(N, f.device)
    m = ((k2 > 0) & (k2 <= kf * (kf + 1))).to(torch.float64)
    w = torch.full((N // 2 + 1,), 2.0, dtype=torch.float64, device=f.device)
    w[0] = 1.0
    return float((m * w * (f.real ** 2 + f.imag ** 2).sum(0)).sum()), m


def _advance(f, N, kw, steps):
    """`steps` steps of the integrator in 64 bits from the transform f[3, N, N, N/2+1]."""
    visc = kw["nu"] * _k2(N, f.device) ** kw["visc_pow"]
    h, kind = kw["dt"], kw["integrator"]
    target = _shell(f, N, 2)[0] if kw.get("forcing") else None
    done = 0
    while done < steps:
        k1, um = _nonlinear(f, N)
        if kw["cfl"] > 0:
            h = kw["cfl"] * 2 * math.pi / N / um
        took = True
        if kind == "ifrk4":
            eh, ef = torch.exp(-0.5 * h * visc), torch.exp(-h * visc)
            k2 = _nonlinear((f + k1 * (h / 2)) * eh, N)[0]
            k3 = _nonlinear(f * eh + k2 * (h / 2), N)[0]
            k4 = _nonlinear(f * ef + k3 * (h * eh), N)[0]
            f = (f + k1 * (h / 6)) * ef + (k2 + k3) * (h / 3 * eh) + k4 * (h / 6)
        else:
            a, b = (2 - h * visc) / (2 + h * visc), 2 * h / (2 + h * visc)
            if kind == "rk4cn":
                k2 = _nonlinear(f + k1 * (h / 2), N)[0]
                k3 = _nonlinear(f + k2 * (h / 2), N)[0]
                k4 = _nonlinear(f + k3 * h, N)[0]
                f = a * f + b * (k1 / 6 + k2 / 3 + k3 / 3 + k4 / 6)
            else:
                ks = [k1]
                for row in _A[:5 if kind == "rk5cn" else 6]:
                    ks.append(_nonlinear(f + h * sum(c * k for c, k in zip(row, ks) if c), N)[0])
                new = a * f + b * sum(c * k for c, k in zip(_B, ks) if c)
                if kind == "dp5cn":
                    diff = b * sum((c - d) * k for c, d, k in zip(_B, _BS, ks) if c != d)
                    den = 1e-7 + torch.maximum(f.abs(), new.abs()) * 1e-7
                    q = ((diff.abs() / den) ** 2 * _mask(N, f.device)).sum((1, 2, 3)) / (N * N * (N // 2 + 1))
                    err = float(q.max().sqrt())
                    took = err <= 1.0
                    h *= min(1.5, max(0.01, 0.8 * err ** -0.2))
                if took:
                    f = new
        if not took:
            continue
        done += 1
        if target is not None:
            e, m = _shell(f, N, 2)
            f = f * (1 + m * (math.sqrt(target / e) - 1))
    return f


def _layout(f):
    return f.permute(1, 2, 3, 0).contiguous()


def exact(case, seed):
    if case["kind"] == "closure":
        return None   # the network's weights are the library's own initialisation
    if case["kind"] == "ensemble":
        out, i = [], 0
        for N in map(int, case["sizes"].split()):
            for j in range(case["each"]):
                kw = _options(case, N)
                kw["nu"] *= 1.0 + 0.1 * j
                # 64-bit runs of all members take long: the first of each size
                out.append(_layout(_advance(_velocity(N, seed * 64 + i), N, kw, case["steps"])) if j == 0 else None)
                i += 1
        return out
    N = case["N"]
    f = _velocity(N, seed + case.get("sample", 0))
    if case["kind"] != "output":
        return _layout(_advance(f, N, _options(case, N), case.get("steps", 1)))
    nu = 0.5 / N
    k2 = _k2(N, f.device)
    w = torch.full((N // 2 + 1,), 2.0, dtype=torch.float64, device=f.device)
    w[0] = 1.0
    norm = 8 * math.pi ** 3 * 0.5 / float(N) ** 6
    curl = _curl(f, N)
    e = w * (f.real ** 2 + f.imag ** 2).sum(0) * norm
    o = w * (curl.real ** 2 + curl.imag ** 2).sum(0) * norm
    palin = w * k2 * (curl.real ** 2 + curl.imag ** 2).sum(0) * norm
    heli = w * (f.real * curl.real + f.imag * curl.imag).sum(0) * norm
    ns = int(math.sqrt(3.0 * (N / 2.0) ** 2)) + 1
    bins = torch.floor(k2.sqrt() + 0.5).long().expand_as(e).reshape(-1)
    spec = [torch.zeros(ns, dtype=torch.float64, device=f.device).index_add_(0, bins.clamp(max=ns - 1), q.reshape(-1)) for q in (e, o)]
    tot = {"energy": e.sum(), "enstrophy": o.sum(), "palinstrophy": palin.sum(), "helicity": heli.sum(), "dissipation": None}
    real = []
    for g in (f, curl):
        r = torch.zeros(N, N, N + 2, 3, dtype=torch.float64, device=f.device)
        r[:, :, :N] = _real(g, N).permute(1, 2, 3, 0)
        real.append(r)
    tot["dissipation"] = 2 * nu * tot["enstrophy"]
    return {"totals": torch.stack([tot[k] for k in sorted(tot)]), "ek": spec[0], "ok": spec[1], "u": real[0], "w": real[1]}
