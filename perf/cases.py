"""Performance cases of the explicit r-z step, through the public entry points.

listed()  the cases; draw(rng)  one more of the same ranges; prepare(case,
seed)  inputs on the GPU (page-locked host arrays for the host-array steps)
and the solver that a program keeps; run(state)  one pass; work(case)  the
bytes and operations of one pass; exact(case, seed)  the same outputs in 64
bits by plain torch.

Kinds of case:
  solver  a resident ast_solver: the state set from device arrays (a coupled
          or restarted run), n steps, the state and the clock read back;
  raw     the kernel-level drop-in: ast_step_raw + ast_funk_time on the
          caller's own device arrays, ping-pong, as the reference's loop
          launches Kernel_TVD and funk_time;
  add2    the same loop with the first-order drop-in ast_add2_raw;
  batch   many independent problems advanced together, autotuned once;
  host    steps from page-locked host arrays to page-locked host arrays;
  train   the start-value network trained on recorded faces.
"""
import os

import numpy as np
import torch

from asteriy_2d_gb300 import abi as A
from asteriy_2d_gb300 import problems, solver

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FLUX = {"hll": A.FLUX_HLL, "hllc": A.FLUX_HLLC, "godunov": A.FLUX_GODUNOV}
GAMMA = 5.0 / 3.0


# ---------------------------------------------------------------- the cases
def listed():
    def solve(name, setup, N, M, flux, prec, steps, learned=False):
        return {"name": name, "kind": "solver", "setup": setup, "N": N, "M": M, "flux": flux, "prec": prec,
                "steps": steps, "learned": learned}

    return [
        # a first look at a tiny grid (the size of the smoke test): launches and latency
        solve("blast 64x32 f64 hll", "blast", 64, 32, "hll", 64, 10),
        # the small plain problem, from its initial discontinuity on: every step waits for the one before
        solve("blast 256x128 f64 hll", "blast", 256, 128, "hll", 64, 100),
        # the wind against a noisy counterflow in FP64, its production size; no cell is undisturbed
        solve("wind 2048x1024 f64 hllc", "wind", 2048, 1024, "hllc", 64, 16),
        # the plain exact-Godunov solver with the reference's iteration, an odd size
        solve("blast 1021x509 f64 godunov", "grown", 1021, 509, "godunov", 64, 8),
        # the step kernel's drop-in on the reference's own grid and boundary set-up
        {"name": "raw 32000x400 f64 hllc", "kind": "raw", "N": 32000, "M": 400, "steps": 4},
        # the first-order drop-in on that grid
        {"name": "add2 32000x400 f64", "kind": "add2", "N": 32000, "M": 400, "steps": 2},
        # the FP32 form at its production size, the blast grown to a third of the radius
        solve("blast 4096x2048 f32 hll", "grown", 4096, 2048, "hll", 32, 32),
        # the headline: exact Godunov in FP32 with the learned start value
        solve("blast 4096x2048 f32 learned", "grown", 4096, 2048, "godunov", 32, 32, True),
        # FP32 HLLC where every face is disturbed, an odd size
        solve("wind 1537x771 f32 hllc", "wind", 1537, 771, "hllc", 32, 20),
        # 64 uneven problems (blasts and winds, HLLC and exact Godunov) advanced together
        {"name": "batch 64 f32", "kind": "batch", "count": 64, "set": 64, "steps": 16},
        # a program that keeps its state in host memory: every step copies it in and out
        {"name": "host 2048x1024 f64 hll", "kind": "host", "N": 2048, "M": 1024, "flux": "hll", "prec": 64, "steps": 4},
        # training the start-value network on recorded faces
        {"name": "train 131072", "kind": "train", "samples": 131072, "batch": 16384, "epochs": 2},
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi]; odd ones among them."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["solver", "solver", "solver", "solver", "raw", "add2", "batch", "host", "train"])
    if kind == "solver":
        prec = rng.choice([32, 64])
        flux = rng.choice(["hll", "hllc", "godunov"])
        N = _size(rng, 64, 4096 if prec == 32 else 2048)
        M = max(32, int(N * rng.uniform(0.4, 0.5)))
        return {"kind": kind, "setup": rng.choice(["blast", "grown", "wind"]), "N": N, "M": M, "flux": flux,
                "prec": prec, "steps": _size(rng, 4, 32 if prec == 32 else 16),
                "learned": flux == "godunov" and prec == 32 and rng.random() < 0.5}
    if kind in ("raw", "add2"):
        return {"kind": kind, "N": _size(rng, 96, 32000), "M": _size(rng, 12, 400), "steps": rng.randint(1, 2)}
    if kind == "batch":
        return {"kind": kind, "count": _size(rng, 2, 64), "set": rng.randint(1, 1 << 20), "steps": _size(rng, 4, 16)}
    if kind == "host":
        N = _size(rng, 256, 2048)
        return {"kind": kind, "N": N, "M": N // 2, "flux": rng.choice(["hll", "hllc"]), "prec": rng.choice([32, 64]),
                "steps": rng.randint(1, 4)}
    batch = 256 * _size(rng, 4, 64)
    return {"kind": "train", "samples": batch * rng.randint(2, 8) + rng.randint(0, batch - 1), "batch": batch,
            "epochs": rng.randint(1, 2)}


# ---------------------------------------------------------------- configurations and inputs
def _config(case):
    """The runtime configuration of a solver, host, raw or add2 case."""
    if case["kind"] in ("raw", "add2"):
        # the reference's domain and boundary rules: inflow (1, 7), (1, 0) at n = 0, outflow, reflecting r sides,
        # the high-order region and the body force (4 rho in Kernel_TVD, 2.5 rho in add2)
        c = A.default_config()
        c.N, c.M = case["N"], case["M"]
        c.flux, c.geom = A.FLUX_HLLC, A.GEOM_PLANAR
        c.recon = A.RECON_MINMOD if case["kind"] == "raw" else A.RECON_NONE
        c.region_select, c.region_lo, c.region_hi = 1, 10.000001, 40.000001
        A.set_bc(c, A.Z_LO, A.BC_FIXED, 1.0, 7.0, 1.0, 0.0)
        A.set_bc(c, A.Z_HI, A.BC_OUTFLOW)
        A.set_bc(c, A.R_LO, A.BC_REFLECT)
        A.set_bc(c, A.R_HI, A.BC_REFLECT)
        c.body_force, c.body_lo, c.body_hi, c.body_rsplit = 1, 20.000001, 30.000001, 0.5
        c.body_amp = 4.0 if case["kind"] == "raw" else 2.5
        return c
    make = problems.wind_config if case.get("setup") == "wind" else problems.blast_config
    c = make(case["N"], case["M"], flux=FLUX[case["flux"]], precision=A.PREC_FP32 if case["prec"] == 32 else A.PREC_FP64)
    if case["prec"] == 32 and case["flux"] == "godunov":
        c.riemann_tol = 1e-8
        c.guess = A.GUESS_MLP if case.get("learned") else A.GUESS_PVRS
    return c


def _grid(c):
    dx = (c.x_max - c.x_min) / (c.N - 1)
    dy = c.y_max / c.M
    x = c.x_min + dx * torch.arange(c.N, dtype=torch.float64, device="cuda")
    y = 0.5 * dy + dy * torch.arange(c.M, dtype=torch.float64, device="cuda")
    return x[None, :], y[:, None], dx, dy


def _waves(c, g, count, amp, shape):
    """A sum of `count` smooth random waves of amplitude about `amp` on the grid."""
    x, y, _, _ = _grid(c)
    out = torch.zeros(shape, dtype=torch.float64, device="cuda")
    for _ in range(count):
        k = (torch.rand(4, generator=g, device="cuda", dtype=torch.float64) * 2 - 1).tolist()
        lx, ly = 40.0 * k[0] / (c.x_max - c.x_min), 20.0 * k[1] / c.y_max
        out += amp * k[2] * torch.sin(lx * x + ly * y + 6.28 * k[3])
    return out


def _state(c, setup, seed):
    """(s, u) of a set-up as the reference's arrays (K, 2) in FP64, and a first time step."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    shape = (c.M, c.N)
    x, y, dx, dy = _grid(c)
    one = torch.ones(shape, dtype=torch.float64, device="cuda")
    draws = torch.rand(4, generator=g, device="cuda", dtype=torch.float64).tolist()
    if setup == "channel":
        # the inflow state with smooth waves everywhere and grid-scale noise downstream
        noise = torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) - 0.5
        far = (x > 0.5 * c.x_max).double()
        rho = 1.0 + _waves(c, g, 4, 0.08, shape) + 0.02 * noise * far
        p = 7.0 * (1.0 + _waves(c, g, 4, 0.05, shape))
        vz = 1.0 + _waves(c, g, 4, 0.3, shape)
        vr = _waves(c, g, 4, 0.2, shape) * torch.sin(3.14159 * y / c.y_max)
    elif setup == "blast":
        # the initial discontinuity: gas at rest, high pressure inside a sphere
        inside = x * x + y * y < (0.2 + 0.01 * draws[0]) ** 2
        rho = one.clone()
        p = torch.where(inside, (8.0 + 4.0 * draws[1]) * one, 0.1 * one)
        vz, vr = 0 * one, 0 * one
    elif setup == "grown":
        # the blast some time later: a strong shell around hot gas in motion, the ambient gas still at rest
        R = torch.sqrt(x * x + y * y)
        Rs = 0.31 + 0.02 * draws[0]
        q = R / Rs
        ripple = 1.0 + _waves(c, g, 6, 0.01, shape)
        inside = q < 1.0
        rho = torch.where(inside, (0.08 + 2.9 * q ** 8) * ripple, one)
        p = torch.where(inside, (0.45 + 0.45 * q ** 8) * ripple, 0.1 * one)
        v = torch.where(inside, 0.8 * q * ripple, 0 * one) / torch.clamp(R, min=1e-12)
        vz, vr = v * x, v * y
    else:
        # wind: the radial wind blown out to R = 0.2, against the counterflow with 1% density noise
        R = torch.clamp(torch.sqrt(x * x + y * y), min=0.5 * dx)
        inside = R < 0.19 + 0.02 * draws[0]
        e = 0.05 / R
        noise = 1.0 + 0.01 * (2.0 * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) - 1.0)
        vin = c.bc[A.Z_HI].vz
        rho = torch.where(inside, e * e, noise)
        p = torch.where(inside, 1.0 / c.gamma * e ** (2.0 * c.gamma), one / c.gamma)
        vz = torch.where(inside, 10.0 * x / R, vin * one)
        vr = torch.where(inside, 10.0 * y / R, 0 * one)
    speed = float((torch.sqrt(vz * vz + vr * vr) + torch.sqrt(c.gamma * p / rho)).max())
    s = torch.stack([rho.reshape(-1), p.reshape(-1)], 1).contiguous()
    u = torch.stack([vz.reshape(-1), vr.reshape(-1)], 1).contiguous()
    return s, u, 0.9 * c.cfl * min(dx, dy) / speed


def _problems(case):
    return solver.problem_set(case["set"], case["count"], A.PREC_FP32)


def _params():
    return np.load(os.path.join(ROOT, "asteriy_2d_gb300", "data", "guess_blast.npy"))


def _faces(n, seed):
    """n recorded faces: features and log(p*/p_L) of random two-shock and shock-rarefaction faces."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    t = torch.rand(5, n, generator=g, device="cuda", dtype=torch.float64)
    rL, pL = torch.ones_like(t[0]), torch.exp(6 * t[0] - 3)
    cL = torch.sqrt(GAMMA * pL)
    pR, rR = pL * torch.exp(4 * t[1] - 2), torch.exp(2 * t[2] - 1)
    uL, uR = torch.zeros_like(cL), -cL * (0.3 + 2.0 * t[3])
    p, _ = _pstar(GAMMA, rL, pL, uL, rR, pR, uR)
    rec = torch.zeros(n, A.AST_RECORD_FLOATS, dtype=torch.float64, device="cuda")
    cR = torch.sqrt(GAMMA * pR / rR)
    for k, v in enumerate((rR / rL, pR / pL, (uR - uL) / cL, cR / cL, torch.full_like(pL, GAMMA), torch.log(pL),
                           torch.log(p / pL))):
        rec[:, k] = v
    return rec.float().cpu().numpy()


# ---------------------------------------------------------------- prepare and run
def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "train":
        st["samples"] = _faces(case["samples"], seed)
        st["params"] = solver.mlp_init(st["samples"], 7)
        return st
    if kind == "batch":
        probs = _problems(case)
        st["cfgs"] = [p.cfg.copy() for p in probs]
        st["B"] = solver.Batch(st["cfgs"])
        st["in"], cells = [], 0
        for i, p in enumerate(probs):
            s, u, dt = _state(p.cfg, "grown" if p.setup == A.SETUP_BLAST else "wind", seed * 4099 + i)
            st["B"].set_state_device(i, s.data_ptr(), u.data_ptr())
            st["B"].set_clock(i, dt)
            st["in"].append((s, u))
            cells += s.shape[0]
        torch.cuda.synchronize()
        st["B"].autotune(2)
        st["s"] = torch.empty(cells, 2, dtype=torch.float64, device="cuda")
        st["u"] = torch.empty_like(st["s"])
        return st
    c = st["cfg"] = _config(case)
    s, u, dt = _state(c, "channel" if kind in ("raw", "add2") else case.get("setup", "grown"), seed)
    if kind in ("raw", "add2"):
        st["in"] = (s, u)
        st["work"] = [(torch.empty_like(s), torch.empty_like(u)) for _ in range(2)]
        # T, T_do, TT, and the step counter, as the reference's program allocates them
        st["clock0"] = torch.tensor([1e7, dt, 0.25], dtype=torch.float64, device="cuda")
        st["clock"] = st["clock0"].clone()
        st["i"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        return st
    st["S"] = solver.Solver(c)
    if case.get("learned"):
        st["S"].set_mlp(_params())
    st["S"].set_clock(dt)
    if kind == "host":
        st["a"] = tuple(t.cpu().pin_memory() for t in (s, u))
        st["b"] = tuple(torch.empty_like(t).pin_memory() for t in st["a"])
        st["in"] = tuple(t.clone() for t in st["a"])
        return st
    st["in"] = (s, u)
    st["out"] = (torch.empty_like(s), torch.empty_like(u))
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "solver":
        S, (s, u), (so, uo) = st["S"], st["in"], st["out"]
        S.set_state_device(s.data_ptr(), u.data_ptr())
        S.step(case["steps"], sync=False)
        S.get_state_device(so.data_ptr(), uo.data_ptr())
        # the program looks at the time to know whether it is done
        T_do, TT, step = S.clock()
        return {"s": so, "u": uo, "T_do": T_do, "TT": TT, "step": step}
    if kind in ("raw", "add2"):
        fn = solver.step_raw if kind == "raw" else solver.add2_raw
        clock = st["clock"]
        clock.copy_(st["clock0"])
        T, T_do, TT = (clock.data_ptr() + 8 * k for k in range(3))
        src = st["in"]
        for k in range(case["steps"]):
            dst = st["work"][k & 1]
            fn(src[0].data_ptr(), src[1].data_ptr(), dst[0].data_ptr(), dst[1].data_ptr(), T, T_do, TT, st["cfg"])
            solver.funk_time(T, T_do, TT, st["i"].data_ptr())
            src = dst
        return {"s": src[0], "u": src[1], "clock": clock}
    if kind == "batch":
        B = st["B"]
        for i, (s, u) in enumerate(st["in"]):
            B.set_state_device(i, s.data_ptr(), u.data_ptr())
        B.step(case["steps"], sync=False)
        at = 0
        for i, (s, u) in enumerate(st["in"]):
            B.get_state_device(i, st["s"].data_ptr() + 16 * at, st["u"].data_ptr() + 16 * at)
            at += s.shape[0]
        return {"s": st["s"], "u": st["u"]}
    if kind == "host":
        # a chain of host-array steps between the program's two pairs of arrays; the next pass goes on from there
        (sa, ua), (sb, ub) = st["a"], st["b"]
        st["S"].step_host_n(case["steps"], sa.data_ptr(), ua.data_ptr(), sb.data_ptr(), ub.data_ptr())
        if case["steps"] % 2:
            st["a"], st["b"] = st["b"], st["a"]
        return {"s": st["a"][0], "u": st["a"][1]}
    params, losses = solver.mlp_train(st["samples"], st["params"], epochs=case["epochs"], batch=case["batch"])
    return {"params": params, "losses": losses}


# ---------------------------------------------------------------- bytes and operations
# operations a cell and step cannot do without: two faces (reconstruction 4 x 8 each; the flux), the update
_FLOPS = {"hll": 2 * (32 + 75) + 50, "hllc": 2 * (32 + 80) + 50, "godunov": 2 * (32 + 60) + 50}


def work(case):
    kind = case["kind"]
    if kind == "train":
        n = case["samples"] // case["batch"] * case["batch"] * case["epochs"]
        # 1313 weights: a multiply-add each forward, two each backward; every record read once an epoch
        return {"bytes": n * 4 * A.AST_RECORD_FLOATS, "flops": n * 6 * 1313}
    if kind == "batch":
        cells = sum(p.cfg.N * p.cfg.M for p in _problems(case))
        return {"bytes": cells * (32 * case["steps"] + 2 * (32 + 16)), "flops": cells * case["steps"] * _FLOPS["hllc"]}
    cells = case["N"] * case["M"]
    steps = case["steps"]
    if kind in ("raw", "add2"):
        # the state read and written by every step: the next dt is a maximum over the whole grid
        per = _FLOPS["hllc"] if kind == "raw" else 4 * 80 + 50
        return {"bytes": cells * 64 * steps, "flops": cells * steps * per}
    elem = case["prec"] // 8
    flops = cells * steps * _FLOPS[case["flux"]]
    if kind == "host":
        return {"bytes": cells * 64 * steps, "flops": flops}
    # a state in and out in FP64, and a read and a write of the state by every step
    return {"bytes": cells * (8 * elem * steps + 2 * (32 + 4 * elem)), "flops": flops}


# ---------------------------------------------------------------- the same outputs in 64 bits, by plain torch
def _minmod(a, b):
    return torch.where(a * b > 0, torch.where(a.abs() < b.abs(), a, b), torch.zeros_like(a))


def _hll(ga, L, R, hllc):
    """HLL (or HLLC with a contact wave) of (rho, p, un, ut) states with the bounds min u - max c, max u + max c."""
    (rL, pL, uL, tL), (rR, pR, uR, tR) = L, R
    c = torch.maximum(torch.sqrt(ga * pL / rL), torch.sqrt(ga * pR / rR))
    SL, SR = torch.minimum(uL, uR) - c, torch.maximum(uL, uR) + c
    eL = pL / (ga - 1) + 0.5 * rL * (uL * uL + tL * tL)
    eR = pR / (ga - 1) + 0.5 * rR * (uR * uR + tR * tR)
    UL, UR = (rL, rL * uL, rL * tL, eL), (rR, rR * uR, rR * tR, eR)
    FL = (rL * uL, rL * uL * uL + pL, rL * uL * tL, (eL + pL) * uL)
    FR = (rR * uR, rR * uR * uR + pR, rR * uR * tR, (eR + pR) * uR)
    if hllc:
        aL, aR = rL * (SL - uL), rR * (SR - uR)
        SM = (aR * uR - aL * uL - pR + pL) / (aR - aL)
        ps = 0.5 * (pR + aR * (SM - uR) + pL + aL * (SM - uL))

        def star(r, p, u, t, e, S, a, U, F):
            rs = a / (S - SM)
            es = ((S - u) * e + ps * SM - p * u) / (S - SM)
            return [f + S * (q - w) for f, q, w in zip(F, (rs, rs * SM, rs * t, es), U)]

        left = star(rL, pL, uL, tL, eL, SL, aL, UL, FL)
        right = star(rR, pR, uR, tR, eR, SR, aR, UR, FR)
        mid = [torch.where(SM >= 0, a, b) for a, b in zip(left, right)]
    else:
        mid = [(SR * f - SL * h + SL * SR * (b - a)) / (SR - SL) for f, h, a, b in zip(FL, FR, UL, UR)]
    F = [torch.where(SL >= 0, f, torch.where(SR <= 0, h, m)) for f, h, m in zip(FL, FR, mid)]
    return F, torch.maximum(SL.abs(), SR.abs())


def _branch(ga, p, pK, rK, cK):
    """The pressure function of one side and its derivative: a shock for p > pK, else a rarefaction."""
    q = torch.sqrt((ga + 1) / (2 * ga) * p / pK + (ga - 1) / (2 * ga))
    fs = (p - pK) / (rK * cK * q)
    ds = ((ga + 1) * p / pK + 3 * ga - 1) / (4 * ga * rK * cK * q ** 3)
    x = (p / pK) ** ((ga - 1) / (2 * ga))
    fr, dr = 2 / (ga - 1) * cK * (x - 1), x * pK / (p * rK * cK)
    return torch.where(p > pK, fs, fr), torch.where(p > pK, ds, dr)


def _pstar(ga, rL, pL, uL, rR, pR, uR):
    """The pressure and velocity of the contact. The pressure function is concave: Newton rises from below."""
    cL, cR = torch.sqrt(ga * pL / rL), torch.sqrt(ga * pR / rR)
    z = (ga - 1) / (2 * ga)
    both = torch.clamp(cL + cR - 0.5 * (ga - 1) * (uR - uL), min=1e-300)
    p = (both / (cL * pL ** -z + cR * pR ** -z)) ** (1 / z)      # two rarefactions: exact where p* < pL, pR
    p = torch.where(p > torch.minimum(pL, pR), torch.minimum(pL, pR), p)
    for _ in range(40):
        fL, dL = _branch(ga, p, pL, rL, cL)
        fR, dR = _branch(ga, p, pR, rR, cR)
        p = torch.clamp(p - (fL + fR + uR - uL) / (dL + dR), min=1e-300)
    fL, _ = _branch(ga, p, pL, rL, cL)
    fR, _ = _branch(ga, p, pR, rR, cR)
    return p, 0.5 * (uL + uR) + 0.5 * (fR - fL)


def _godunov(ga, L, R):
    (rL, pL, uL, tL), (rR, pR, uR, tR) = L, R
    cL, cR = torch.sqrt(ga * pL / rL), torch.sqrt(ga * pR / rR)
    p, us = _pstar(ga, rL, pL, uL, rR, pR, uR)

    def side(r, pk, u, c, sgn):
        """Density, pressure and velocity at rest between the contact and side K (sgn -1: the left), its wave speeds."""
        shock = p > pk
        w = torch.sqrt((ga + 1) / (2 * ga) * p / pk + (ga - 1) / (2 * ga))
        head = u + sgn * c * torch.where(shock, w, torch.ones_like(w))
        cs = c * (p / pk) ** ((ga - 1) / (2 * ga))
        tail = torch.where(shock, head, us + sgn * cs)
        k = (ga - 1) / (ga + 1)
        rs = torch.where(shock, r * (p / pk + k) / (k * p / pk + 1), r * (p / pk) ** (1 / ga))
        # inside the fan at rest the velocity is the sound speed
        cf = torch.clamp(2 / (ga + 1) * c - sgn * k * u, min=1e-300)
        rf, pf, uf = r * (cf / c) ** (2 / (ga - 1)), pk * (cf / c) ** (2 * ga / (ga - 1)), -sgn * cf
        out, mid = sgn * head <= 0, sgn * tail >= 0
        pick = lambda a, b, f: torch.where(out, a, torch.where(mid, b, f))  # noqa: E731
        return pick(r, rs, rf), pick(pk, p, pf), pick(u, us, uf), torch.maximum(head.abs(), tail.abs())

    l, r = side(rL, pL, uL, cL, -1.0), side(rR, pR, uR, cR, 1.0)
    left = us >= 0
    rho, pp, un = (torch.where(left, a, b) for a, b in zip(l[:3], r[:3]))
    ut = torch.where(left, tL, tR)
    e = pp / (ga - 1) + 0.5 * rho * (un * un + ut * ut)
    return [rho * un, rho * un * un + pp, rho * un * ut, un * (e + pp)], torch.clamp(torch.maximum(l[3], r[3]), min=1e-7)


def _ghosts(c, q):
    """The state (4, M, N) with two ghost layers on each side."""
    P = torch.nn.functional.pad(q[None], (2, 2, 2, 2), mode="replicate")[0].clone()
    flip = {0: 2, 1: 3}
    for side, (axis, low) in enumerate([(2, True), (2, False), (1, True), (1, False)]):
        b = c.bc[side]
        n = P.shape[axis]
        for j in range(2):
            at = 1 - j if low else n - 2 + j
            if b.kind == A.BC_FIXED:
                v = torch.tensor([b.rho, b.p, b.vz, b.vr], dtype=P.dtype, device=P.device)[:, None]
                P.select(axis, at).copy_(v.expand(4, P.shape[3 - axis]))
            elif b.kind == A.BC_REFLECT:
                m = P.select(axis, 2 + j if low else n - 3 - j).clone()
                m[flip[2 - axis]] *= -1
                P.select(axis, at).copy_(m)
    return P


def _faces_of(c, P, axis):
    """Left and right states of the faces along an axis of the padded state, first order and reconstructed."""
    if axis == 2:
        P = P[:, 2:-2, :]
        cut = lambda a, b: P[:, :, a:P.shape[2] + b]  # noqa: E731
    else:
        P = P[:, :, 2:-2]
        cut = lambda a, b: P[:, a:P.shape[1] + b, :]  # noqa: E731
    a, l, r, b = cut(0, -3), cut(1, -2), cut(2, -1), cut(3, 0)
    if c.recon != A.RECON_MINMOD:
        return (l, r), (l, r)
    L, R = l + 0.5 * _minmod(l - a, r - l), r - 0.5 * _minmod(r - l, b - r)
    for k in (0, 1):
        L[k], R[k] = torch.where(L[k] <= 0, l[k], L[k]), torch.where(R[k] <= 0, r[k], R[k])
    return (l, r), (L, R)


def _exact_step(c, q, dt, TT=None):
    """One step of the scheme in FP64: (state, next dt). TT: the time of the first-order drop-in, whose two cells of
    a z face may use different fluxes."""
    ga = c.gamma
    x, y, dx, dy = _grid(c)
    P = _ghosts(c, q)
    if TT is not None and TT < 3.0:
        P[0, 2:-2, :2] *= torch.where(y < 0.5, 1.0 + 0.01 * np.sin(2 * np.pi * TT), 1.0)
    flux, speed, other = [], [], None
    for axis in (2, 1):
        low, high = _faces_of(c, P, axis)
        turn = (lambda v: v) if axis == 2 else (lambda v: (v[0], v[1], v[3], v[2]))
        if c.flux == A.FLUX_GODUNOV:
            F, S = _godunov(ga, turn(high[0]), turn(high[1]))
        else:
            F, S = _hll(ga, turn(high[0]), turn(high[1]), c.flux == A.FLUX_HLLC)
        if c.region_select:
            G, V = _hll(ga, turn(low[0]), turn(low[1]), False)
            # the face's position as the lower cell sees it
            xf = torch.cat([x[:, :1] - dx, x], 1) + 0.5 * dx if axis == 2 else x
            inside = (xf > c.region_lo) & (xf < c.region_hi)
            if TT is not None and axis == 2:
                other = [torch.where(inside, g, f) for f, g in zip(F, G)]
            F = [torch.where(inside, f, g) for f, g in zip(F, G)]
            S = torch.maximum(S, V) if TT is not None and axis == 2 else torch.where(inside, S, V)
        flux.append(torch.stack([F[0], F[2], F[1], F[3]] if axis == 1 else F))
        speed.append(S)
    keep = torch.zeros_like(q[0], dtype=torch.bool)
    if c.fixed_region:
        keep = (x - c.fixed_zc) ** 2 / c.fixed_az ** 2 + y ** 2 / c.fixed_ar ** 2 < 1
    live = ~keep
    zl = torch.nn.functional.pad(live, (1, 1)) if c.fixed_region else torch.ones_like(speed[0])[:, :1].bool()
    rl = torch.nn.functional.pad(live, (0, 0, 1, 1)) if c.fixed_region else None
    if c.fixed_region:
        sz, sr = speed[0][zl[:, 1:] | zl[:, :-1]].max(), speed[1][rl[1:] | rl[:-1]].max()
    else:
        sz, sr = speed[0].max(), speed[1].max()
    left = flux[0] if other is None else torch.stack(other)
    div = (flux[0][:, :, 1:] - left[:, :, :-1]) / dx + (flux[1][:, 1:] - flux[1][:, :-1]) / dy
    rho, p, vz, vr = q
    E = p / (ga - 1) + 0.5 * rho * (vz * vz + vr * vr)
    U = torch.stack([rho, rho * vz, rho * vr, E]) - dt * div
    if c.geom == A.GEOM_AXISYM:
        U = U - dt / y * vr * torch.stack([rho, rho * vz, rho * vr, E + p])
    if c.body_force:
        on = ((x > c.body_lo) & (x < c.body_hi)).double()
        Q = on * torch.where(y >= c.body_rsplit, -c.body_amp, c.body_amp) * rho
        U[2] += dt * Q
        U[3] += dt * Q * vr
    r2 = torch.where(U[0] <= 0, rho, U[0])
    p2 = (ga - 1) * (U[3] - 0.5 * (U[1] ** 2 + U[2] ** 2) / r2)
    new = torch.stack([r2, torch.where(p2 <= 0, c.p_floor, p2), U[1] / r2, U[2] / r2])
    return torch.where(keep, q, new), c.cfl * min(dx / float(sz), dy / float(sr))


def _exact_run(c, s, u, dt, steps, TT=0.0, add2=False):
    q = torch.cat([s.t(), u.t()]).reshape(4, c.M, c.N).contiguous()
    for _ in range(steps):
        q, dt = _exact_step(c, q, dt, TT if add2 else None)
        TT += dt
    q = q.reshape(4, -1)
    return q[:2].t().contiguous(), q[2:].t().contiguous(), dt, TT


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return None     # the order of the samples is the library's own
    if kind == "batch":
        got = []
        for i, p in enumerate(_problems(case)):
            s, u, dt = _state(p.cfg, "grown" if p.setup == A.SETUP_BLAST else "wind", seed * 4099 + i)
            got.append(_exact_run(p.cfg, s, u, dt, case["steps"]))
        return {"s": torch.cat([g[0] for g in got]), "u": torch.cat([g[1] for g in got])}
    c = _config(case)
    s, u, dt = _state(c, "channel" if kind in ("raw", "add2") else case.get("setup", "grown"), seed)
    s, u, dt, TT = _exact_run(c, s, u, dt, case["steps"], 0.25 if kind in ("raw", "add2") else 0.0, kind == "add2")
    if kind == "host":
        return {"s": s, "u": u}
    if kind == "solver":
        return {"s": s, "u": u, "T_do": dt, "TT": TT, "step": case["steps"]}
    return {"s": s, "u": u, "clock": torch.tensor([1e7, dt, TT], dtype=torch.float64)}
