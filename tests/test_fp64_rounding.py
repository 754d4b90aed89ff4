"""The rounding errors of the FP64 step: one first-order step against the same
formulas in long double (64 or 113 bits), beside the same formulas in plain FP64.

Bar.  The last roundings of an output are, in plain FP64, the conserved sum's and
the division's by rho; the kernels multiply by 1/rho, one rounding more of the
same size: sqrt(3/2) = 1.22 times the plain rms error at most.  A sum rounded
twice at its own size is above it."""
import numpy as np
import pytest

from asteriy_2d_gb300 import abi as A
from asteriy_2d_gb300 import problems, solver

pytestmark = pytest.mark.gpu


def fluxes(L, R, ga, T):
    """HLL and HLLC of the states L and R (rho, p, un, ut), evaluated in T."""
    c = np.maximum(np.sqrt(ga * L[1] / L[0]), np.sqrt(ga * R[1] / R[0]))
    SL, SR = np.minimum(L[2], R[2]) - c, np.maximum(L[2], R[2]) + c
    U, F = [], []
    for r, p, un, ut in (L, R):
        e = p / (ga - T(1)) + T(0.5) * r * (un * un + ut * ut)
        U.append(np.stack([r, r * un, r * ut, e]))
        F.append(np.stack([r * un, r * un * un + p, r * un * ut, (e + p) * un]))
    hll = (SR * F[0] - SL * F[1] + SL * SR * (U[1] - U[0])) / (SR - SL)
    aL, aR = L[0] * (SL - L[2]), R[0] * (SR - R[2])
    SM = (aR * R[2] - aL * L[2] - R[1] + L[1]) / (aR - aL)
    ps = T(0.5) * (R[1] + aR * (SM - R[2]) + L[1] + aL * (SM - L[2]))
    star = []
    for (r, p, un, ut), a, S, V, G in ((L, aL, SL, U[0], F[0]), (R, aR, SR, U[1], F[1])):
        rs = a / (S - SM)
        es = ((S - un) * V[3] + ps * SM - p * un) / (S - SM)
        star.append(G + S * (np.stack([rs, rs * SM, rs * ut, es]) - V))
    upwind = lambda m: np.where(SL >= 0, F[0], np.where(SR <= 0, F[1], m))  # noqa: E731
    return upwind(hll), upwind(np.where(SM >= 0, star[0], star[1]))


def step_in(T, cfg, s, u, dt):
    """(rho, p, vz, vr) after one first-order step with outflow on every side."""
    N, M, ga = cfg.N, cfg.M, T(cfg.gamma)
    q = np.stack([s[:, 0], s[:, 1], u[:, 0], u[:, 1]]).astype(T).reshape(4, M, N)
    dx, dy, dt = T((cfg.x_max - cfg.x_min) / (N - 1)), T(cfg.y_max / M), T(dt)
    which = 0 if cfg.flux == A.FLUX_HLL else 1
    z = np.concatenate([q[:, :, :1], q, q[:, :, -1:]], 2)
    r = np.concatenate([q[:, :1], q, q[:, -1:]], 1)[[0, 1, 3, 2]]
    Fz = fluxes(z[:, :, :-1], z[:, :, 1:], ga, T)[which]
    Fr = fluxes(r[:, :-1], r[:, 1:], ga, T)[which][[0, 2, 1, 3]]
    rho, p, vz, vr = q
    E = p / (ga - T(1)) + T(0.5) * rho * (vz * vz + vr * vr)
    U = np.stack([rho, rho * vz, rho * vr, E])
    U = U - (dt / dx * (Fz[:, :, 1:] - Fz[:, :, :-1]) + dt / dy * (Fr[:, 1:] - Fr[:, :-1]))
    if cfg.geom == A.GEOM_AXISYM:
        y = (T(cfg.y_max / (2.0 * M)) + np.arange(M) * dy)[:, None]
        U = U - dt / y * np.stack([rho * vr, rho * vr * vz, rho * vr * vr, vr * (E + p)])
    out = np.stack([U[0], (ga - T(1)) * (U[3] - T(0.5) * (U[1] ** 2 + U[2] ** 2) / U[0]), U[1] / U[0], U[2] / U[0]])
    return out.reshape(4, -1)


@pytest.mark.parametrize("flux", [A.FLUX_HLL, A.FLUX_HLLC])
@pytest.mark.parametrize("geom", [A.GEOM_PLANAR, A.GEOM_AXISYM])
@pytest.mark.parametrize("mach", [0.0, 1.0, 3.0])
@pytest.mark.parametrize("N,M", [(257, 129), (633, 250)])    # 16x16 tiles; the persistent kernel, ragged
def test_error_is_that_of_plain_fp64(flux, geom, mach, N, M):
    if np.finfo(np.longdouble).nmant <= 52:
        pytest.skip("long double is no longer than double")
    cfg = problems.blast_config(N, M, flux=flux)
    cfg.recon, cfg.geom = A.RECON_NONE, geom
    for side in range(4):
        A.set_bc(cfg, side, A.BC_OUTFLOW)
    rng = np.random.default_rng(5)
    s = np.exp(rng.uniform(-0.3, 0.3, (N * M, 2)))
    u = mach + rng.uniform(-0.3, 0.3, (N * M, 2))
    dt = 0.3 * min(2.0 / (N - 1), 1.0 / M) / (2 * mach + 3)
    with solver.Solver(cfg) as S:
        S.set_state(s, u)
        S.set_clock(dt)
        S.step(1)
        gpu = np.concatenate(S.get_state(), 1).T
    exact, plain = step_in(np.longdouble, cfg, s, u, dt), step_in(np.float64, cfg, s, u, dt)
    for k in range(4):
        rms = [float(np.sqrt(np.mean((v[k] - exact[k]) ** 2))) for v in (gpu, plain)]
        assert rms[0] <= 1.22 * rms[1], (k, rms[0] / rms[1])
