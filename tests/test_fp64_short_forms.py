"""The FP64 kernels' short forms (integer comparisons, third-order reciprocals
and roots, the exact solver's replayed bisection) against the oracle, one step
from random states: inside their range, outside it (the reference's formulas
take over) and across its edges, supersonic and nearly equal sides, several
gammas (1/gm whole or not) and tolerances.

Bars.  One step changes a conserved value by sums of at most 16 products, each
off by a few 2^-53 of the largest; the pressure subtracts the kinetic energy,
here at most 50 times it: 1e-12 of the largest value.  The exact solver's p* may
move by its tolerance where a stopping test falls the other way: 1e-9 at the
reference's tolerance, 1e-11 at 1e-13."""
import numpy as np
import pytest

import pyoracle as O
from asteriy_2d_gb300 import abi as A
from asteriy_2d_gb300 import problems, solver

pytestmark = pytest.mark.gpu


def states(N, M, rho, p, mach, seed):
    """Random cells around (rho, p): a third with strong jumps, a third with
    weak ones, a third nearly or exactly equal."""
    rng = np.random.default_rng(seed)
    K = N * M
    amp = np.repeat([1.0, 1e-3, 1e-12], -(-K // 3))[:K]
    c = np.sqrt(p / rho)
    s = np.stack([rho * np.exp(amp * rng.uniform(-0.7, 0.7, K)), p * np.exp(amp * rng.uniform(-1, 1, K))], 1)
    u = np.stack([c * (mach + 2 * amp * rng.uniform(-1, 1, K)), c * amp * rng.uniform(-1, 1, K)], 1)
    s[-5:], u[-5:] = s[-5], u[-5]
    return s, u, c


def one_step(cfg, s, u, dt):
    with solver.Solver(cfg) as S:
        S.set_state(s, u)
        S.set_clock(dt)
        S.step(1)
        gs, gu = S.get_state()
        tdo = S.clock()[0]
    os_, ou, otdo, _, _, _ = O.run(cfg, s, u, 1, T_do=dt)
    e = [np.max(np.abs(g - o)) / np.max(np.abs(o)) for g, o in ((gs[:, 0], os_[:, 0]), (gs[:, 1], os_[:, 1]), (gu, ou))]
    return max(e), abs(tdo - otdo) / otdo


# rho, p: the middle, the edges of the exact solver's range (2^+-40) and of
# the other fluxes' (2^+-150), and far outside
SCALES = [(1.0, 1.0), (2.0 ** 40, 2.0 ** -40), (2.0 ** -150, 2.0 ** -149), (2.0 ** 150, 2.0 ** 60), (1e70, 1e-60)]


@pytest.mark.parametrize("flux", [A.FLUX_HLL, A.FLUX_HLLC, A.FLUX_GODUNOV])
@pytest.mark.parametrize("scale", range(len(SCALES)))
@pytest.mark.parametrize("mach", [0.0, 0.9, 3.0])
def test_one_step_matches_oracle(flux, scale, mach):
    rho, p = SCALES[scale]
    cfg = problems.blast_config(37, 19, flux=flux)
    cfg.p_floor = 1e-300
    cfg.riemann_tol = 1e-9 * np.sqrt(p / rho)
    s, u, c = states(37, 19, rho, p, mach, 5)
    dt = 0.1 * (2.0 / 36) / ((mach + 4) * c)
    err, terr = one_step(cfg, s, u, dt)
    assert err <= (1e-9 if flux == A.FLUX_GODUNOV else 1e-12), err
    assert terr <= 1e-9


@pytest.mark.parametrize("gamma", [5.0 / 3.0, 1.4, 4.0 / 3.0, 1.3, 3.0])
@pytest.mark.parametrize("tol,bar", [(1e-9, 1e-9), (1e-13, 1e-11), (1e-4, 1e-9), (1e-7, 1e-9)])
@pytest.mark.parametrize("geom", [A.GEOM_AXISYM, A.GEOM_PLANAR])
def test_exact_solver_gammas_and_tolerances(gamma, tol, bar, geom):
    cfg = problems.blast_config(65, 33, flux=A.FLUX_GODUNOV)
    cfg.gamma, cfg.riemann_tol, cfg.geom = gamma, tol, geom
    s, u, c = states(65, 33, 1.0, 1.0, 0.4, 9)
    err, terr = one_step(cfg, s, u, 0.004)
    assert err <= bar, err
    assert terr <= max(bar, 1e-9)


def numpy_add2(cfg, s, u, dt, TT, method):
    """add2 as the reference evaluates it, each cell its own four faces, in numpy."""
    N, M, ga = cfg.N, cfg.M, cfg.gamma
    q = np.stack([s[:, 0], s[:, 1], u[:, 0], u[:, 1]]).reshape(4, M, N)
    dx, dy = (cfg.x_max - cfg.x_min) / (N - 1), cfg.y_max / M
    x, y = cfg.x_min + np.arange(N) * dx, cfg.y_max / (2 * M) + np.arange(M) * dy

    def faces(L, R):
        c = np.maximum(np.sqrt(ga * L[1] / L[0]), np.sqrt(ga * R[1] / R[0]))
        SL, SR = np.minimum(L[2], R[2]) - c, np.maximum(L[2], R[2]) + c
        U, F = [], []
        for r, p, un, ut in (L, R):
            e = p / (ga - 1) + 0.5 * r * (un * un + ut * ut)
            U.append(np.stack([r, r * un, r * ut, e]))
            F.append(np.stack([r * un, r * un * un + p, r * un * ut, (e + p) * un]))
        hll = (SR * F[0] - SL * F[1] + SL * SR * (U[1] - U[0])) / (SR - SL)
        aL, aR = L[0] * (SL - L[2]), R[0] * (SR - R[2])
        SM = (aR * R[2] - aL * L[2] - R[1] + L[1]) / (aR - aL)
        ps = 0.5 * (R[1] + aR * (SM - R[2]) + L[1] + aL * (SM - L[2]))
        star = []
        for (r, p, un, ut), a, S, V, G in ((L, aL, SL, U[0], F[0]), (R, aR, SR, U[1], F[1])):
            rs = a / (S - SM)
            es = ((S - un) * V[3] + ps * SM - p * un) / (S - SM)
            star.append(G + S * (np.stack([rs, rs * SM, rs * ut, es]) - V))
        hllc = np.where(SM >= 0, star[0], star[1])
        pick = lambda m: np.where(SL >= 0, F[0], np.where(SR <= 0, F[1], m))  # noqa: E731
        return pick(hll), pick(hllc), np.maximum(np.abs(SL), np.abs(SR))

    b = cfg.bc[A.Z_LO]
    left = np.empty((4, M, 1))
    left[:, :, 0] = np.array([b.rho, b.p, b.vz, b.vr])[:, None]
    if method and TT < 3.0:
        left[0, y < 0.5, 0] *= 1.0 + 0.01 * np.sin(2 * np.pi * TT)
    z = np.concatenate([left, q, q[:, :, -1:]], 2)
    A_, B_, Sz = faces(z[:, :, :-1], z[:, :, 1:])
    inside = lambda v: (v > cfg.region_lo) & (v < cfg.region_hi)  # noqa: E731
    # the face's position as its lower cell sees it, and as its upper one does
    right = np.where(inside(np.concatenate([[x[0] - dx], x]) + 0.5 * dx), B_, A_)
    lft = np.where(inside(np.concatenate([x, [x[-1] + dx]]) - 0.5 * dx), A_, B_)
    flip = np.array([1.0, 1.0, 1.0, -1.0])[:, None, None]
    r = np.concatenate([q[:, :1] * flip, q, q[:, -1:] * flip], 1)[[0, 1, 3, 2]]
    A_, B_, Sr = faces(r[:, :-1], r[:, 1:])
    Fr = np.where(inside(x), B_, A_)[[0, 2, 1, 3]]
    U = np.stack([q[0], q[0] * q[2], q[0] * q[3], q[1] / (ga - 1) + 0.5 * q[0] * (q[2] ** 2 + q[3] ** 2)])
    U = U - dt * ((right[:, :, 1:] - lft[:, :, :-1]) / dx + (Fr[:, 1:] - Fr[:, :-1]) / dy)
    Q = np.where((x > cfg.body_lo) & (x < cfg.body_hi), 1.0, 0.0) * np.where(y >= cfg.body_rsplit, -1.0, 1.0)[:, None]
    Q = Q * cfg.body_amp * q[0]
    U[2] += dt * Q
    U[3] += dt * Q * q[3]
    new = np.stack([U[0], (ga - 1) * (U[3] - 0.5 * (U[1] ** 2 + U[2] ** 2) / U[0]), U[1] / U[0], U[2] / U[0]])
    return new.reshape(4, -1), cfg.cfl * min(dx / Sz.max(), dy / Sr.max())


# the smallest grid, and below, at and just past the tile (32x16)
@pytest.mark.parametrize("N,M", [(4, 4), (31, 17), (32, 16), (33, 15), (65, 33), (97, 4)])
def test_add2_tiles(N, M):
    import torch
    import golden_configs as G
    cfg = G.add2_config(N, M)
    cfg.region_lo, cfg.region_hi, cfg.body_lo, cfg.body_hi = 20.0, 60.0, 30.0, 50.0
    s, u = G.random_state(N * M, np.random.default_rng(3))
    u *= 3.0        # supersonic faces among them
    dt, TT = 1e-4, 0.3
    dev = torch.device("cuda:0")
    a = [torch.tensor(v, device=dev) for v in (s, u)]
    b = [torch.zeros_like(v) for v in a]
    clock = torch.tensor([1e7, dt, TT], dtype=torch.float64, device=dev)
    T = [clock.data_ptr() + 8 * k for k in range(3)]
    solver.add2_raw(a[0].data_ptr(), a[1].data_ptr(), b[0].data_ptr(), b[1].data_ptr(), *T, cfg, method=1)
    torch.cuda.synchronize()
    want, T_new = numpy_add2(cfg, s, u, dt, TT, 1)
    got = np.concatenate([b[0].cpu().numpy().T, b[1].cpu().numpy().T])
    err = np.max(np.abs(got - want), axis=1) / np.max(np.abs(want), axis=1)
    assert np.all(err <= 1e-12), err
    assert abs(float(clock[0]) - T_new) <= 1e-12 * T_new
