"""The FP64 exact solver's wave patterns on single faces: the pattern decides
the formulas, so faces are placed on both sides of its thresholds, at pressure
ratios up to 1e12, in both orders of the sides and both orientations, and one
step is compared with the oracle.

Each test face is the middle one of four cells (A A B B) in a row of such
groups, first order, so a cell next to it changes by this face's flux alone
(its other neighbour equals it)."""
import numpy as np
import pytest

import pyoracle as O
from asteriy_2d_gb300 import abi as A
from asteriy_2d_gb300 import problems, solver

pytestmark = pytest.mark.gpu


def line(faces, along_z):
    """The groups of `faces` ((rho, p, un) of the lower and of the upper side)
    along z or r, four cells wide across: a configuration and its state."""
    n = 4 * len(faces)
    cfg = problems.blast_config(n if along_z else 4, 4 if along_z else n, flux=A.FLUX_GODUNOV)
    cfg.recon, cfg.geom = A.RECON_NONE, A.GEOM_PLANAR
    cfg.x_min, cfg.x_max, cfg.y_max = 0.0, float(cfg.N - 1), float(cfg.M)   # dx = dy = 1
    cfg.p_floor = 1e-300
    for side in range(4):
        A.set_bc(cfg, side, A.BC_OUTFLOW)
    q = np.repeat(np.array(faces, dtype=np.float64).reshape(-1, 3), 2, axis=0)
    k = np.arange(cfg.N * cfg.M)
    q = q[k % cfg.N if along_z else k // cfg.N]
    s, u = q[:, :2].copy(), np.zeros((len(k), 2))
    u[:, 0 if along_z else 1] = q[:, 2]
    return cfg, s, u


def step(cfg, s, u, dt):
    cfg.collect_stats = 1
    with solver.Solver(cfg) as S:
        S.set_state(s, u)
        S.set_clock(dt)
        S.step(1)
        return (*S.get_state(), S.clock()[0], S.stats())


def worst(cfg, s, u, dt):
    """The largest difference from the oracle's step, each cell by its own
    scales: rho, p + rho u^2, |u| + c."""
    gs, gu, tdo, _ = step(cfg, s, u, dt)
    os_, ou, otdo, _, _, _ = O.run(cfg, s, u, 1, T_do=dt)
    q = np.sum(ou * ou, 1)
    e = max(np.max(np.abs(gs[:, 0] - os_[:, 0]) / os_[:, 0]),
            np.max(np.abs(gs[:, 1] - os_[:, 1]) / (os_[:, 1] + os_[:, 0] * q)),
            np.max(np.abs(gu - ou) / (np.sqrt(q) + np.sqrt(cfg.gamma * os_[:, 1] / os_[:, 0]))[:, None]))
    return e, abs(tdo - otdo) / otdo


def threshold_faces(ga, cII):
    """Faces at a fraction f beside the threshold between two rarefactions (f <
    0) and shock and rarefaction, in the frame in which the sampled state is
    the one between the low-pressure side's wave and the contact."""
    g1, g2 = ga - 1.0, ga + 1.0
    gm = g1 / (2 * ga)
    out = []
    for ratio in (1e2, 1e4, 1e6, 1e7, 1e8, 1e9, 1e10, 1e12):
        for dens in (1.0, 30.0):
            rI, rII = dens, 1.0
            pII = cII * cII * rII / ga
            pI = pII / ratio
            cI = np.sqrt(ga * pI / rI)
            Urz = -2 * cII / g1 * (1 - ratio ** -gm)
            for f in (-3e-2, -3e-3, -3e-4, 3e-4, 7e-4, 1e-3, 3e-3, 6e-3, 1e-2, 1.5e-2, 2.5e-2, 5e-2):
                U = Urz * (1 - f)

                def res(p):    # rises with p
                    fI = (p - pI) / np.sqrt(rI * (0.5 * g2 * p + 0.5 * g1 * pI)) if p > pI else \
                        2 * cI / g1 * ((p / pI) ** gm - 1)
                    return fI + 2 * cII / g1 * ((p / pII) ** gm - 1) - U

                lo, hi = 1e-6 * pI, pII
                for _ in range(200):
                    p = np.sqrt(lo * hi)
                    lo, hi = (lo, p) if res(p) > 0 else (p, hi)
                a = np.sqrt(rI * (0.5 * g2 * p + 0.5 * g1 * pI))
                if p > pI:
                    u, edge = -(p - pI) / a, -a / rI
                else:
                    u = -2 * cI / g1 * ((p / pI) ** gm - 1)
                    edge = u - cI * (p / pI) ** gm
                w = 0.5 * (u + edge)            # (enI = 0 so far)
                I, II = (rI, pI, -w), (rII, pII, -U - w)
                out.append((I, II))
                out.append(((rII, pII, U + w), (rI, pI, w)))
    return out


# p* is found to the tolerance in velocity, 1e-9 cII: relative to p_I that is
# 1e-3 at most (c_I >= 1e-6 cII), and the low-pressure cell changes by at most
# 1e-7 of itself here (dt c_I/dx): 1e-10.  A face in the wrong pattern is
# off by tenths of the change of the cells, 1e-9 and more.
@pytest.mark.parametrize("gamma", [5.0 / 3.0, 1.4, 4.0 / 3.0])
@pytest.mark.parametrize("along_z", [True, False])
def test_patterns_at_large_pressure_ratios(gamma, along_z):
    cII = 10.0
    cfg, s, u = line(threshold_faces(gamma, cII), along_z)
    cfg.gamma, cfg.riemann_tol = gamma, 1e-9 * cII
    err, terr = worst(cfg, s, u, 0.1 / (np.max(np.abs(u)) + cII))
    assert err <= 1e-10, err
    assert terr <= 1e-9, terr


# two shocks with p* up to 1e48 times the lower pressure, both sides inside the
# short solver's range: its FP32 derivative does not reach that far.  p* is
# found to the rounding of the residual, some 1e-15; the cells change by tenths
@pytest.mark.parametrize("low,high", [((1e12, 1e-12, 1e9), (1e12, 1e12, -1e9)),
                                      ((1e6, 1e-12, 1e12), (1e6, 1e10, -1e12)),
                                      ((1.0, 1e-10, 1e8), (1.0, 1.0, 0.0))])
@pytest.mark.parametrize("along_z", [True, False])
def test_two_shocks_far_above_both_pressures(low, high, along_z):
    cfg, s, u = line([(low, high)], along_z)
    err, terr = worst(cfg, s, u, 0.05 / np.max(np.abs(u)))
    assert err <= 1e-12, err
    assert terr <= 1e-12, terr


# faces with equal pressures and equal normal velocities (contacts) take the
# closed form: nothing iterates, and the gas stays as it is but for the
# density's advection (the oracle's step to a few roundings)
@pytest.mark.parametrize("recon", [A.RECON_NONE, A.RECON_MINMOD])
@pytest.mark.parametrize("p", [0.1, 1.0 / 3.0, 1.0, 7.3])
@pytest.mark.parametrize("v", [0.0, 0.3])
def test_contacts_take_the_closed_form(recon, p, v):
    cfg = problems.blast_config(37, 21, flux=A.FLUX_GODUNOV)
    cfg.recon, cfg.geom = recon, A.GEOM_PLANAR
    for side in range(4):
        A.set_bc(cfg, side, A.BC_OUTFLOW)
    K = cfg.N * cfg.M
    s = np.stack([np.exp(np.random.default_rng(1).uniform(-1.0, 1.0, K)), np.full(K, p)], 1)
    u = np.stack([np.full(K, v), np.full(K, -v)], 1)
    stats = step(cfg, s, u, 1e-4)[3]
    assert stats["bisect_calls"] == stats["newton_calls"] == 0, stats
    err, terr = worst(cfg, s, u, 1e-4)
    assert err <= 1e-13, err
    assert terr <= 1e-13, terr


# gas at rest beside its mirror image at the axis (v_r = +0 and -0 on the two
# sides of that face) stays at rest, exactly, and takes the identical-state path
@pytest.mark.parametrize("recon", [A.RECON_NONE, A.RECON_MINMOD])
@pytest.mark.parametrize("p", [0.1, 1.0, 7.3, 10.0])
def test_gas_at_rest_at_a_reflecting_axis_stays_at_rest(recon, p):
    cfg = problems.blast_config(37, 21, flux=A.FLUX_GODUNOV)
    cfg.recon = recon
    K = cfg.N * cfg.M
    s, u = np.stack([np.ones(K), np.full(K, p)], 1), np.zeros((K, 2))
    gs, gu, _, stats = step(cfg, s, u, 1e-3)
    assert np.all(gu == 0.0), np.max(np.abs(gu))
    assert len(np.unique(gs[:, 0])) == len(np.unique(gs[:, 1])) == 1
    assert stats["bisect_calls"] == stats["newton_calls"] == 0, stats


def random_faces(ga, n, span, rspan, rng):
    """Faces of every pattern: pressure ratios to 10^span, densities over
    10^(2 rspan), Udf inside the patterns, beside their thresholds, far above
    them and zero, in moving frames, scaled to speeds of 10."""
    g1, g2 = ga - 1.0, ga + 1.0
    out = []
    while len(out) < n:
        pI = 10.0 ** -rng.uniform(0.0, span) if rng.random() < 0.8 else 1.0
        rI, rII = 10.0 ** rng.uniform(-rspan, rspan), 10.0 ** rng.uniform(-rspan, rspan)
        cI, cII = np.sqrt(ga * pI / rI), np.sqrt(ga / rII)
        Uud = (1.0 - pI) / np.sqrt(rI * (g2 + g1 * pI) / 2)
        Urz, Uvk = -2 * cII / g1 * (1 - pI ** (g1 / (2 * ga))), -2 * (cI + cII) / g1
        near = (cI + cII) * 10.0 ** rng.uniform(-8, -1) * rng.choice([-1, 1])
        U = [rng.uniform(Uvk, Urz), rng.uniform(Urz, Uud), Uud + 10.0 ** rng.uniform(-3, 3) * (cI + cII), Urz + near,
             Uud + near, 0.0][rng.integers(6)]
        base = (cI + cII) * rng.choice([0.0, 1e-3, 0.1, 1.0, 3.0]) * rng.uniform(-1, 1)
        k = 10.0 / max(cI, cII, abs(U), abs(base))
        if pI * k * k < 2e-12 or k * k > 5e11:
            continue            # outside the short solver's range
        I, II = (rI, pI * k * k, base * k), (rII, k * k, (base - U) * k)
        out.append((I, II) if rng.random() < 0.5 else ((II[0], II[1], -II[2]), (I[0], I[1], -I[2])))
    return out


# each cell's change against the oracle's.  A stopping test on the edge moves p*
# by the tolerance, 1e-9 of the largest speed, which is 1e-3 of the slowest
# sound speed: 1e-2 of the change.  (Cells that change by less than 1e-8 of
# themselves are compared to 1e-10 of themselves.)
@pytest.mark.parametrize("gamma", [5.0 / 3.0, 1.4, 4.0 / 3.0, 1.3, 3.0, 1.1])
@pytest.mark.parametrize("span,rspan", [(2, 1), (8, 2), (12, 5)])
def test_random_faces_of_every_pattern(gamma, span, rspan):
    cfg, s, u = line(random_faces(gamma, 1000, span, rspan, np.random.default_rng(11)), True)
    cfg.gamma, cfg.riemann_tol = gamma, 1e-8
    dt = 0.02 / 60
    gs, gu, tdo, _ = step(cfg, s, u, dt)
    os_, ou, otdo, _, _, _ = O.run(cfg, s, u, 1, T_do=dt)
    q = np.sum(ou * ou, 1)
    k = np.arange(cfg.N)
    mid = (k % 4 == 1) | (k % 4 == 2)           # the two cells of a test face, in the first row
    c = np.sqrt(gamma * s[:, 1] / s[:, 0])
    for got, want, old, scale in ((gs[:, 0], os_[:, 0], s[:, 0], s[:, 0]),
                                  (gs[:, 1], os_[:, 1], s[:, 1], os_[:, 1] + os_[:, 0] * q),
                                  (gu[:, 0], ou[:, 0], u[:, 0], np.abs(u[:, 0]) + c)):
        err = np.abs(got - want) / np.maximum(np.abs(want - old), 1e-8 * scale)
        assert np.max(err[: cfg.N][mid]) <= 1e-2, np.max(err[: cfg.N][mid])
    assert abs(tdo - otdo) <= 1e-9 * otdo
