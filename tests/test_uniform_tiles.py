"""Tiles whose staged cells are all one state skip the faces (and, in the
persistent kernel, an update whose result the output tile already holds).
region_select over the whole domain gives every face the same flux but takes
the full path, so the two runs have to agree bit for bit: blasts at rest and
in moving gas (v_r too), a source, negative zeros, ragged tiles, every flux,
both precisions, the per-tile and the persistent kernels, the batch.

The FP32 exact solver (plain start value, its queue split by pattern) against
the FP64 one: the update's sixteen
products round to 2^-24 each and the pressure subtracts the kinetic energy
(here at most four times it), p* is found to 1e-6, its flux moves a cell by at
most half a wave crossing: 2e-5 of the largest value after one step."""
import numpy as np
import pytest

from asteriy_2d_gb300 import abi as A
from asteriy_2d_gb300 import problems, solver

pytestmark = pytest.mark.gpu


def pair(cfg):
    full = cfg.copy()
    full.region_select, full.region_lo, full.region_hi = 1, -1e6, 1e6
    return cfg, full


def state(cfg, vz, vr):
    s, u = solver.fill_blast(cfg)
    u = np.zeros_like(u)
    u[:, 0], u[:, 1] = vz, vr
    return s, u


def run(cfg, s, u, n):
    with solver.Solver(cfg) as S:
        S.set_state(s, u)
        S.step(n)
        return (*S.get_state(), S.clock())


def same(a, b):
    return np.array_equal(a[0], b[0], equal_nan=True) and np.array_equal(a[1], b[1], equal_nan=True) and a[2] == b[2]


# several persistent tiles per CTA (1500x700: more than 24 of 64x16 per SM and
# ragged), a few tiles, less than one
@pytest.mark.parametrize("N,M,steps", [(1500, 700, 12), (200, 90, 25), (20, 9, 5)])
@pytest.mark.parametrize("precision", [A.PREC_FP32, A.PREC_FP64])
@pytest.mark.parametrize("flux", [A.FLUX_HLL, A.FLUX_HLLC, A.FLUX_GODUNOV, A.FLUX_HLLC_A])
@pytest.mark.parametrize("vz,vr", [(0.0, 0.0), (-0.0, -0.0), (0.7, 0.0), (-0.3, 0.2)])
def test_uniform_tiles_match_the_full_path(N, M, steps, precision, flux, vz, vr):
    out = []
    for cfg in pair(problems.blast_config(N, M, flux=flux, precision=precision)):
        out.append(run(cfg, *state(cfg, vz, vr), steps))
    assert same(*out)


@pytest.mark.parametrize("persistent", [0, 1])
@pytest.mark.parametrize("change", ["planar", "body_force", "tiny", "scale"])
def test_uniform_tiles_options_match_the_full_path(persistent, change):
    cfg = problems.blast_config(420, 210, flux=A.FLUX_HLL, precision=A.PREC_FP32)
    cfg.persistent = persistent
    if change == "planar":
        cfg.geom = A.GEOM_PLANAR
    if change == "body_force":
        cfg.body_force, cfg.body_lo, cfg.body_hi, cfg.body_rsplit, cfg.body_amp = 1, -0.4, 0.3, 0.3, 1e-3
    out = []
    for c in pair(cfg):
        s, u = state(c, 0.25, 0.0)
        if change == "tiny":       # below the pressure floor: the update is not one state
            s[:, 1] *= 1e-9
        if change == "scale":      # kinetic energy far above the internal: FP64 pressure recovery
            u[:, 0] = 60.0
        out.append(run(c, s, u, 10))
    assert same(*out)


@pytest.mark.parametrize("precision", [A.PREC_FP32, A.PREC_FP64])
@pytest.mark.parametrize("flux", [A.FLUX_HLL, A.FLUX_GODUNOV])
def test_batch_uniform_tiles_match_the_full_path(precision, flux):
    cfgs = [problems.blast_config(2 * m, m, flux=flux, precision=precision) for m in (48, 61, 96, 130)]
    out = []
    for full in (0, 1):
        with solver.Batch([pair(c)[full] for c in cfgs]) as B:
            for i, c in enumerate(cfgs):
                B.set_state(i, *state(c, 0.1 * i, 0.0))
            B.step(15)
            out.append([(*B.get_state(i), B.clock(i)) for i in range(len(cfgs))])
    assert all(same(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("gamma", [5.0 / 3.0, 1.4, 1.3, 3.0])
@pytest.mark.parametrize("N,M,persistent", [(16, 16, 0), (65, 33, 0), (130, 70, 1)])
def test_fp32_exact_solver_matches_fp64(gamma, N, M, persistent):
    rng = np.random.default_rng(4)
    s = np.exp(rng.uniform(-0.5, 0.5, (N * M, 2)))
    u = rng.uniform(-1.0, 1.0, (N * M, 2))
    s[: N * M // 2] = 1.0 + 1e-3 * (s[: N * M // 2] - 1.0)     # weak waves
    out = []
    for precision in (A.PREC_FP32, A.PREC_FP64):
        cfg = problems.blast_config(N, M, flux=A.FLUX_GODUNOV, precision=precision)
        cfg.gamma, cfg.persistent = gamma, persistent if precision == A.PREC_FP32 else 1
        with solver.Solver(cfg) as S:
            S.set_state(s, u)
            S.set_clock(0.05 * 2.0 / (N - 1))
            S.step(1)
            out.append(np.concatenate(S.get_state(), 1))
    for k in range(4):
        assert np.max(np.abs(out[0][:, k] - out[1][:, k])) <= 2e-5 * np.max(np.abs(out[1][:, k]))
