"""The work that users of this solver have it do, as measurable cases.

A case is a dict of plain values; ``prepare`` builds what a program holds
before the call (potentials, a context, output buffers, loss weights), ``run``
makes one pass through the public entry points, ``exact`` restates the result
in 64-bit torch where that is affordable.  Potentials have the distributions of
``epseon_backend_gb300.synth`` (Morse, shifted Lennard-Jones 12-6, Morse with
Gaussian bumps on a natural spline of 1024 knots).

``do`` names the entry points:

* ``count``    -- ``epscu_count_levels_static``: bound-level counts of one
  device-resident potential on a ladder of trial energies (no allocation).
* ``host``     -- ``Context.solve`` on host arrays: energies, node counts,
  status, wavefunctions when ``psi``; otherwise the wavefunctions stay on the
  device and ``Context.adjoint`` returns the gradient of a least-squares loss.
* ``task``     -- the device/task interface of the reference
  (``EpseonComputeContext`` to ``TaskHandleFloat32``) in spectroscopic units.
* ``plain``    -- ``Context.solve`` with the plain FP64 method, wavefunctions out.
* ``device``   -- ``DeviceBatch.solve`` on resident tensors, with wavefunctions
  when ``psi``, and ``DeviceBatch.adjoint`` when ``adjoint`` (from the kept
  wavefunctions, or recomputing them when there are none).
* ``fit``      -- ``autograd.tabulate`` and ``autograd.levels``, forward and
  backward: a parameter fit's step.
* ``tabulate`` -- ``autograd.tabulate`` alone, forward and backward.

err_est, the solver's estimate of its own last correction (a rounding
residual), is written by the solves but is not among the outputs.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from epseon_backend_gb300 import autograd, capi, synth

CAP = 512  # level slots per potential
KNOTS = 1024
# levels a potential: WKB counts averaged over the parameter ranges
LEVELS = {"long": 280.0, "morse": 53.0, "bumps": 53.0, "mixed": 46.0}


def listed():
    return [
        # the smallest call: how many levels lie below each energy, for one
        # curve inside another program's loop
        {"name": "count_one", "do": "count", "n": 10007, "n_trial": 1024},
        # one curve at a time from numpy, levels and wavefunctions back (an
        # interactive session, a potential read from a paper)
        {"name": "single_host", "do": "host", "batch": 1, "n_min": 4096, "n_max": 4096, "n_trial": 1024,
         "kind": "morse", "psi": True},
        # the reference's own interface: a list of Morse curves as one task
        {"name": "task_24", "do": "task", "batch": 24, "n_min": 6000, "step": 0.5, "top": 120},
        # the FP64 method, used to check the fast one
        {"name": "plain_6", "do": "plain", "batch": 6, "n_min": 3001, "n_max": 3001, "n_trial": 1500,
         "kind": "morse", "psi": True},
        # tabulating a parametrised family and pulling a gradient back to its
        # parameters
        {"name": "tabulate_2048", "do": "tabulate", "batch": 2048, "n_min": 2048, "n_max": 65536, "kind": "mixed"},
        # a few dozen curves resident on the device, solve and gradient in a loop
        {"name": "morse_64", "do": "device", "batch": 64, "n_min": 16384, "n_max": 16384, "n_trial": 8192,
         "kind": "morse", "psi": True, "adjoint": True},
        # the same without room for wavefunctions: the gradient recomputes them
        {"name": "recompute_48", "do": "device", "batch": 48, "n_min": 4096, "n_max": 32768, "n_trial": 4096,
         "kind": "mixed", "psi": False, "adjoint": True},
        # screening many curves for their level energies only
        {"name": "screen_512", "do": "device", "batch": 512, "n_min": 2048, "n_max": 65536, "n_trial": 8192,
         "kind": "mixed", "psi": False, "adjoint": False},
        # a batch from host memory with its gradient back to host memory
        {"name": "host_256", "do": "host", "batch": 256, "n_min": 2048, "n_max": 65536, "n_trial": 8192,
         "kind": "mixed", "psi": False},
        # fitting Morse + bump parameters to measured levels
        {"name": "fit_256", "do": "fit", "batch": 256, "n_min": 32768, "n_max": 32768, "n_trial": 8192,
         "kind": "bumps"},
        # the largest batch: uneven grids of every kind, wavefunctions, gradient
        {"name": "mixed_2048", "do": "device", "batch": 2048, "n_min": 2048, "n_max": 65536, "n_trial": 8192,
         "kind": "mixed", "psi": True, "adjoint": True},
        # one heavy pair on a very fine grid
        {"name": "long_1m", "do": "device", "batch": 1, "n_min": 1 << 20, "n_max": 1 << 20, "n_trial": 65536,
         "kind": "long", "psi": True, "adjoint": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["count", "host", "task", "plain", "tabulate", "device", "device", "fit", "long"])
    if do == "count":
        return {"do": do, "n": _log(rng, 2048, 65536), "n_trial": _log(rng, 64, 8192)}
    if do == "task":
        return {"do": do, "batch": _log(rng, 1, 128), "n_min": _log(rng, 2048, 16384),
                "step": round(math.exp(rng.uniform(math.log(0.2), math.log(4.0))), 3), "top": rng.randint(10, 200)}
    if do == "plain":
        n = _log(rng, 1024, 3001)
        return {"do": do, "batch": _log(rng, 1, 48), "n_min": n, "n_max": n, "n_trial": _log(rng, 128, 4096),
                "kind": "morse", "psi": rng.random() < 0.5}
    if do == "long":
        n = _log(rng, 65537, 1 << 20)
        return {"do": "device", "batch": 1, "n_min": n, "n_max": n, "n_trial": _log(rng, 8192, 65536), "kind": "long",
                "psi": True, "adjoint": rng.random() < 0.7}
    n_min = _log(rng, 2048, 32768)
    n_max = min(65536, _log(rng, n_min, 16 * n_min))
    if do == "tabulate":
        return {"do": do, "batch": _log(rng, 1, 2048), "n_min": n_min, "n_max": n_max,
                "kind": rng.choice(["mixed", "morse", "bumps"])}
    if do == "fit":
        return {"do": do, "batch": _log(rng, 1, 320), "n_min": n_min, "n_max": n_max, "n_trial": _log(rng, 512, 8192),
                "kind": rng.choice(["bumps", "mixed"])}
    case = {"do": do, "batch": _log(rng, 1, 768), "n_min": n_min, "n_max": n_max, "n_trial": _log(rng, 512, 8192),
            "kind": rng.choice(["mixed", "mixed", "morse"]), "psi": rng.random() < 0.6}
    if do == "host":
        case["psi"] = case["psi"] and case["batch"] * n_max <= 65536  # (wavefunctions copied out: small batches)
    else:
        case["adjoint"] = rng.random() < 0.6
    return case


# ------------------------------------------------------------------- inputs


def _batch(case, seed):
    """Parameters and grids of the case's potentials (no values yet).  The grid
    lengths are the case's; the potentials on them are the seed's."""
    B, n0, n1, kind = case["batch"], case["n_min"], case["n_max"], case["kind"]
    n_trial = case.get("n_trial", 8192)
    if kind == "long":
        b = synth.morse_long(N=n0, n_trial=n_trial)
        b.morse[0] *= 1.0 + 0.05 * np.random.default_rng(seed).uniform(-1.0, 1.0, 3)
        b.De[0] = b.morse[0, 0]
        b.e_cap = synth.CAP_FRACTION * b.De
        return b
    if kind == "mixed":
        b = synth.mixed_batch(B=B, n_trial=n_trial, seed=seed, n_min=n0, n_max=n1)
    else:
        make = synth.bump_adjoint if kind == "bumps" else synth.morse_batch
        b = make(B=B, N=n0, n_trial=n_trial, seed=seed)
    lengths = np.random.default_rng([B, n0, n1]).uniform(math.log(n0), math.log(n1), B)
    b.N[:] = np.rint(np.exp(lengths)).astype(np.int32)
    return b


def _psi_room(case, b):
    """Doubles set aside for the batch's wavefunctions: the expected number of
    levels (as in ``work``) with room for the spread of a small batch."""
    most = 400.0  # levels of the heaviest, widest well of the ranges
    per = min(most, LEVELS[case["kind"]] * (1.0 + 6.0 / math.sqrt(len(b))))
    return int((most if case["kind"] == "long" else per) * float(b.N.astype(np.float64).sum()))


def _spline_map(K, hk, dev):
    """M = S y: second derivatives of the natural cubic spline on K knots."""
    A = 4.0 * torch.eye(K - 2, dtype=torch.float64, device=dev)
    A += torch.diag(torch.ones(K - 3, dtype=torch.float64, device=dev), 1)
    A += torch.diag(torch.ones(K - 3, dtype=torch.float64, device=dev), -1)

    def apply(y):
        rhs = 6.0 * (y[..., 2:] - 2.0 * y[..., 1:-1] + y[..., :-2]) / (hk * hk)
        x = torch.linalg.solve(A, rhs.transpose(-1, -2)).transpose(-1, -2)
        return torch.nn.functional.pad(x, (1, 1))

    return apply


def _values(b, P, dev):
    """The potentials' values, concatenated, from parameter rows P [n, 12] in
    plain 64-bit torch (differentiable in P)."""
    N = torch.as_tensor(b.N.astype(np.int64), device=dev)
    n = N.numel()
    r0 = torch.as_tensor(b.r_min, device=dev)
    r1 = torch.as_tensor(b.r_max, device=dev)
    h = (r1 - r0) / (N - 1)
    p = torch.repeat_interleave(torch.arange(n, device=dev), N)
    first = torch.cumsum(N, 0) - N
    i = torch.arange(p.numel(), device=dev) - first[p]
    r = r0[p] + i * h[p]
    kind = torch.as_tensor(b.kind.astype(np.int64), device=dev)
    V = torch.zeros_like(r)
    kp = kind[p]
    m = (kp == synth.KIND_MORSE).nonzero()[:, 0]
    if m.numel():
        q = p[m]
        V = V.index_put((m,), P[q, 0] * (1.0 - torch.exp(-P[q, 1] * (r[m] - P[q, 2]))) ** 2)
    m = (kp == synth.KIND_LJ).nonzero()[:, 0]
    if m.numel():
        q = p[m]
        s6 = (P[q, 1] / r[m]) ** 6
        V = V.index_put((m,), 4.0 * P[q, 0] * (s6 * s6 - s6) + P[q, 0])
    sp = (kind == synth.KIND_SPLINE).nonzero()[:, 0]
    if sp.numel():
        S = P[sp]
        hk = ((r1 - r0) / (KNOTS - 1))[sp][:, None]
        rk = r0[sp][:, None] + torch.arange(KNOTS, device=dev) * hk
        y = S[:, 0:1] * (1.0 - torch.exp(-S[:, 1:2] * (rk - S[:, 2:3]))) ** 2
        for j in (3, 6, 9):
            used = S[:, j:j + 1] != 0.0
            w = torch.where(used, S[:, j + 1:j + 2], torch.ones_like(hk))
            y = y + S[:, j:j + 1] * torch.exp(-((rk - S[:, j + 2:j + 3]) ** 2) / (2.0 * w * w))
        M = _spline_map(KNOTS, hk, dev)(y)
        row = torch.full((n,), -1, device=dev)
        row[sp] = torch.arange(sp.numel(), device=dev)
        m = (kp == synth.KIND_SPLINE).nonzero()[:, 0]
        q = row[p[m]]
        hq = hk[q, 0]
        t = (r[m] - r0[p[m]]) / hq
        j = t.floor().long().clamp(0, KNOTS - 2)
        u = t - j
        w = 1.0 - u
        V = V.index_put((m,), w * y[q, j] + u * y[q, j + 1]
                        + hq * hq / 6.0 * ((w ** 3 - w) * M[q, j] + (u ** 3 - u) * M[q, j + 1]))
    return V


def _params(b, dev):
    return torch.as_tensor(capi.batch_params(b), device=dev)


def _weights(b, seed, cap=CAP):
    """Loss weights and target levels of a least-squares fit."""
    rng = np.random.Generator(np.random.PCG64([seed, 11]))
    w = rng.uniform(0.5, 1.0, (len(b), cap))
    t = np.sort(rng.uniform(0.0, 1.0, (len(b), cap)), axis=1) * b.De[:, None]
    return w, t


def _layout(b, V):
    N = np.asarray(b.N, np.int32)
    off = np.zeros(N.size, np.int64)
    off[1:] = np.cumsum(N[:-1].astype(np.int64))
    return capi.Concatenated(V, off, N)


def prepare(case, seed):
    do = case["do"]
    s = {"do": do, "case": case}
    if do == "task":
        return _prepare_task(s, case, seed)
    if do == "count":
        b = _batch({**case, "batch": 3, "n_min": case["n"], "n_max": case["n"], "kind": "mixed"}, seed)
        b = b.subset([seed % 3])
        s["b"] = b
        s["V"] = _values(b, _params(b, "cuda"), "cuda")
        s["counts"] = torch.zeros(case["n_trial"], dtype=torch.int32, device="cuda")
        s["lib"] = capi.load()
        return s
    b = _batch(case, seed)
    s["b"] = b
    P = _params(b, "cuda")
    if do in ("fit", "tabulate"):
        s["P"] = P.requires_grad_(True)
        s["kind"] = b.kind
        s["grids"] = autograd.Grids(b.N, b.r_min, b.r_max, b.mu, b.e_cap, case.get("n_trial", 1024), CAP)
        s["solver"] = autograd.Solver(0)
        if do == "fit":
            w, t = _weights(b, seed)
            s["w"], s["t"] = torch.as_tensor(w, device="cuda"), torch.as_tensor(t, device="cuda")
        else:
            g = torch.Generator(device="cuda").manual_seed(seed)
            s["gV"] = torch.randn(s["grids"].total, dtype=torch.float64, device="cuda", generator=g)
        return s
    with torch.no_grad():
        V = _values(b, P, "cuda")
    if do in ("host", "plain"):
        keep = torch.empty(V.numel(), dtype=torch.float64, pin_memory=True)
        keep.copy_(V)
        s["keep"] = keep
        s["Vs"] = _layout(b, keep.numpy())
        s["ctx"] = capi.Context(0)
        s["w"], s["t"] = _weights(b, seed)
        return s
    s["ctx"] = capi.Context(0)
    host = _layout(b, np.empty(V.numel()))
    s["db"] = capi.DeviceBatch(s["ctx"], host, b.r_min, b.r_max, b.mu, b.e_cap, b.n_trial, CAP, want_psi=case["psi"],
                               psi_capacity=_psi_room(case, b))
    s["db"].V.copy_(V)
    s["gE"] = torch.as_tensor(_weights(b, seed)[0], device="cuda")
    return s


def _prepare_task(s, case, seed):
    import epseon_backend_gb300.device.cuda as dev

    rng = np.random.default_rng(seed)
    ctx = dev.EpseonComputeContext.create()
    info = next(iter(ctx.get_physical_device_info()))
    s["iface"] = ctx.get_device_interface(info.device_properties.device_id)
    s["configurator"] = (
        s["iface"].get_task_configurator("float32")
        .set_hardware_config(potential_buffer_size=case["n_min"], group_size=512, allocation_block_size=1 << 26)
        .set_morse_potential([
            dev.MorsePotentialConfig(dissociation_energy=float(rng.uniform(3000.0, 6000.0)),
                                     equilibrium_bond_distance=float(rng.uniform(2.5, 4.0)),
                                     well_width=float(rng.uniform(0.8, 1.5)), min_r=1.0, max_r=20.0,
                                     point_count=case["n_min"]) for _ in range(case["batch"])])
        .set_vibwa_algorithm(mass_atom_0=87.62, mass_atom_1=87.62, integration_step=case["step"],
                             min_distance_to_asymptote=0.1, min_level=0, max_level=case["top"]))
    return s


# --------------------------------------------------------------------- runs


def run(s):
    do, case = s["do"], s["case"]
    if do == "task":
        handle = s["iface"].submit_task(s["configurator"])
        handle.wait()
        r = handle.get_results()
        shape = (case["batch"], case["top"] + 1)
        energies, nodes = np.full(shape, np.nan), np.full(shape, -1, np.int32)
        for p, (e, v) in enumerate(zip(r["energies"], r["nodes"])):
            energies[p, :e.size], nodes[p, :v.size] = e, v
        return {"energies": energies, "nodes": nodes, "n_total": np.asarray(r["n_total"])}
    b = s.get("b")
    if do == "count":
        V, counts = s["V"], s["counts"]
        capi._check(s["lib"].epscu_count_levels_static(
            C.cast(C.c_void_p(V.data_ptr()), capi._dp), int(b.N[0]), float(b.r_min[0]), float(b.r_max[0]),
            float(b.mu[0]), float(b.e_cap[0]), int(b.n_trial), C.cast(C.c_void_p(counts.data_ptr()), capi._ip),
            C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return counts
    if do == "tabulate":
        s["P"].grad = None
        V = autograd.tabulate(s["P"], s["kind"], s["grids"], KNOTS, s["solver"])
        V.backward(s["gV"])
        return {"V": V.detach(), "gP": s["P"].grad}
    if do == "fit":
        s["P"].grad = None
        V = autograd.tabulate(s["P"], s["kind"], s["grids"], KNOTS, s["solver"])
        E, mask = autograd.levels(V, s["grids"], s["solver"])
        loss = (s["w"] * torch.where(mask, E - s["t"], torch.zeros_like(E)) ** 2).sum()
        loss.backward()
        return {"E": E.detach(), "mask": mask, "loss": loss.detach(), "gP": s["P"].grad}
    if do in ("host", "plain"):
        sol = s["ctx"].solve(s["Vs"], b.r_min, b.r_max, b.mu, b.e_cap, b.n_trial,
                             method=capi.METHOD_PLAIN_FP64 if do == "plain" else capi.METHOD_FAST_FP32C,
                             level_capacity=CAP, want_psi=case["psi"], psi_capacity=_psi_room(case, b),
                             keep_psi=not case["psi"] and do == "host")
        out = {"energy": sol.energy, "nodes": sol.nodes, "status": sol.status, "n_total": sol.n_total}
        if case["psi"]:
            out["psi"] = sol.psi
        elif do == "host":
            inside = np.arange(CAP)[None, :] < sol.n_out[:, None]
            gE = np.where(inside, 2.0 * s["w"] * (np.where(inside, sol.energy, 0.0) - s["t"]), 0.0)
            out["gV"] = s["ctx"].adjoint(gE, int(s["Vs"][0].size))
        return out
    db = s["db"]
    db.solve()
    out = {"energy": db.energy, "nodes": db.nodes, "status": db.status, "n_total": db.n_total}
    if case["psi"]:
        out["psi"] = db.psi
    if case["adjoint"]:
        out["gV"] = db.adjoint(s["gE"], recompute=not case["psi"])
    return out


# --------------------------------------------------------------------- work


def _mean_log(lo, hi):
    return float(lo) if hi <= lo else (hi - lo) / math.log(hi / lo)


def work(case):
    """Bytes: every input value read once and every output written once.
    Flops: one march of the three-term recurrence (9 flops a point) over the
    grid for each level (the expected number of levels of the case's
    potentials); for counts on a ladder of energies, which are monotone, the
    marches of one bisection of the ladder."""
    do = case["do"]
    if do == "count":
        return {"bytes": 8.0 * case["n"] + 4.0 * case["n_trial"], "flops": 9.0 * case["n"] * math.log2(case["n_trial"])}
    B, N = case["batch"], _mean_log(case["n_min"], case.get("n_max", case["n_min"]))
    if do == "tabulate":  # V and its gradient; an exponential or a spline piece a point, twice
        return {"bytes": 16.0 * B * N + 200.0 * B, "flops": 30.0 * B * N}
    if do == "task":
        levels = B * min(case["top"] + 1, 70.0)
        return {"bytes": 100.0 * B + 24.0 * levels, "flops": 10.0 * B * N + 9.0 * N * levels}
    levels = LEVELS[case["kind"]] * B
    moved = 8.0 * B * N + 24.0 * levels
    flops = 9.0 * N * levels
    if do == "fit":
        return {"bytes": 200.0 * B + 24.0 * levels, "flops": flops + 6.0 * N * levels + 60.0 * B * N}
    if case["psi"]:
        moved += 8.0 * N * levels
    if case.get("adjoint") or (do == "host" and not case["psi"]):
        moved += 8.0 * B * N + 8.0 * levels
        flops += 3.0 * N * levels
    return {"bytes": moved, "flops": flops}


# -------------------------------------------------------------------- exact


def _dense(V, h, mu, e_cap):
    """Levels below e_cap and wavefunctions of the discrete problem by dense
    symmetric diagonalisation: H = diag(V) - B^-1 D2 / (2 mu h^2) on the points
    kept by the E-independent cut-offs, B = tridiag(1, 10, 1)/12, D2 =
    tridiag(1, -2, 1), both diagonal in the sine basis."""
    N = V.numel()
    a = mu * h * h / 6.0
    inside = (a * (V - V.min()) <= 0.5).nonzero()[:, 0]
    i0, i1 = max(1, int(inside[0])), min(N - 2, int(inside[-1]))
    n = i1 - i0 + 1
    k = torch.arange(1, n + 1, dtype=torch.float64, device=V.device)
    S = torch.sin(torch.outer(k, k) % (2 * (n + 1)) * (math.pi / (n + 1))) * math.sqrt(2.0 / (n + 1))
    d = 4.0 * torch.sin(0.5 * math.pi * k / (n + 1)) ** 2
    H = (S * (d / (1.0 - d / 12.0) / (2.0 * mu * h * h))) @ S
    H += torch.diag(V[i0:i1 + 1])
    E, X = torch.linalg.eigh(0.5 * (H + H.T))
    E = E[E < e_cap]
    psi = torch.zeros((E.numel(), N), dtype=torch.float64, device=V.device)
    psi[:, i0:i1 + 1] = X[:, :E.numel()].T / math.sqrt(h)
    # positive next to the inner wall
    big = psi.abs() > 1e-6 * psi.abs().amax(1, keepdim=True)
    at = big.to(torch.int8).argmax(1, keepdim=True)
    return E, psi * torch.sign(psi.gather(1, at))


def exact(case, seed):
    do = case["do"]
    if do in ("count", "task"):
        return None  # whole numbers; spectroscopic units (the solve is the host case's)
    if do == "tabulate":
        b = _batch(case, seed)
        P = _params(b, "cuda").requires_grad_(True)
        V = _values(b, P, "cuda")
        g = torch.Generator(device="cuda").manual_seed(seed)
        V.backward(torch.randn(V.numel(), dtype=torch.float64, device="cuda", generator=g))
        return {"V": V.detach(), "gP": P.grad}
    b = _batch(case, seed)
    if do == "fit" or float(np.sum(b.N.astype(np.float64) ** 3)) > 3e11:
        return None  # a dense diagonalisation would take too long
    V = _values(b, _params(b, "cuda"), "cuda")
    off = np.concatenate([[0], np.cumsum(b.N.astype(np.int64))])
    energy = torch.full((len(b), CAP), math.nan, dtype=torch.float64, device="cuda")
    w, t = _weights(b, seed)
    rows, grads = [], []
    for p in range(len(b)):
        h = (b.r_max[p] - b.r_min[p]) / (b.N[p] - 1)
        E, psi = _dense(V[off[p]:off[p + 1]], h, b.mu[p], b.e_cap[p])
        n = min(CAP, E.numel())
        energy[p, :n] = E[:n]
        rows.append(psi[:n].reshape(-1))
        gE = torch.as_tensor(w[p, :n], device="cuda")
        if do == "host":
            gE = 2.0 * gE * (E[:n] - torch.as_tensor(t[p, :n], device="cuda"))
        grads.append((gE[:, None] * psi[:n] ** 2).sum(0) * h)
    out = {"energy": energy, "nodes": None, "status": None, "n_total": None}
    if case["psi"]:
        psi = torch.cat(rows)
        out["psi"] = torch.nn.functional.pad(psi, (0, _psi_room(case, b) - psi.numel()))
    elif do == "host":
        out["gV"] = torch.cat(grads)
    if case.get("adjoint"):
        out["gV"] = torch.cat(grads)
    return out
