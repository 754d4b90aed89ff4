"""Uniform tiles against the full path (region_select over the whole domain,
which gives every face the same flux and skips nothing), where
test_uniform_tiles.py does not look: boundary kinds whose ghost cells continue
the uniform state and ones that do not, the counters, the learned start value, a
batch of several fluxes in one launch, and the bands of the host-array step.
State, clock and counters have to be the same, bit for bit."""
import os

import numpy as np
import pytest

from asteriy_2d_gb300 import abi as A
from asteriy_2d_gb300 import problems, solver

pytestmark = pytest.mark.gpu
PARAMS = os.path.join(os.path.dirname(solver.__file__), "data", "guess_blast.npy")


def both(cfg):
    full = cfg.copy()
    full.region_select, full.region_lo, full.region_hi = 1, -1e6, 1e6
    for c in (cfg, full):
        c.collect_stats = 1
    return cfg, full


def moving(cfg, vz=0.3, vr=-0.2):
    s, u = solver.fill_blast(cfg)
    u[:, 0], u[:, 1] = vz, vr
    return s, u


def compare(cfg, s, u, steps, params=None):
    out = []
    for c in both(cfg):
        with solver.Solver(c) as S:
            if params is not None:
                S.set_mlp(params)
            S.set_state(s, u)
            S.step(steps)
            out.append((*S.get_state(), S.clock(), S.stats()))
    a, b = out
    assert np.array_equal(a[0], b[0], equal_nan=True) and np.array_equal(a[1], b[1], equal_nan=True)
    assert a[2:] == b[2:], (a[2:], b[2:])


KINDS = [(A.BC_REFLECT,) * 4, (A.BC_OUTFLOW,) * 4, (A.BC_FIXED, A.BC_OUTFLOW, A.BC_REFLECT, A.BC_SUCTION),
         (A.BC_NONREFLECT, A.BC_FIXED, A.BC_REFLECT, A.BC_OUTFLOW), (A.BC_SUCTION, A.BC_NONREFLECT) * 2]


@pytest.mark.parametrize("kinds", KINDS)
@pytest.mark.parametrize("precision,persistent", [(A.PREC_FP32, 1), (A.PREC_FP32, 0), (A.PREC_FP64, 1)])
@pytest.mark.parametrize("flux", [A.FLUX_HLL, A.FLUX_HLLC, A.FLUX_GODUNOV])
@pytest.mark.parametrize("N,M", [(160, 96), (1500, 700)])
def test_boundary_kinds(kinds, precision, persistent, flux, N, M):
    cfg = problems.blast_config(N, M, flux=flux, precision=precision)
    cfg.persistent = persistent
    for side, kind in enumerate(kinds):
        if kind == A.BC_FIXED:
            A.set_bc(cfg, side, kind, 1.0, 0.1, 0.3, -0.2)      # the gas's own state: uniform ghost cells
        elif kind == A.BC_SUCTION:
            A.set_bc(cfg, side, kind, 0.0, 0.0, 0.02, -0.01)
        else:
            A.set_bc(cfg, side, kind)
    compare(cfg, *moving(cfg), 12)


@pytest.mark.parametrize("precision", [A.PREC_FP32, A.PREC_FP64])
@pytest.mark.parametrize("N,M", [(257, 129), (1500, 700)])
def test_learned_start(precision, N, M):
    cfg = problems.blast_config(N, M, flux=A.FLUX_GODUNOV, precision=precision)
    cfg.guess, cfg.riemann_tol, cfg.riemann_newton = A.GUESS_MLP, 1e-8, 1
    compare(cfg, *moving(cfg, 0.0, 0.0), 20, np.load(PARAMS))


# (one launch for several fluxes takes FP32 problems)
@pytest.mark.parametrize("precision,mixed", [(A.PREC_FP32, 0), (A.PREC_FP32, 1), (A.PREC_FP64, 0)])
def test_batch_of_several_fluxes(precision, mixed):
    cfgs = [problems.blast_config(2 * m, m, flux=f, precision=precision)
            for m in (48, 61, 96) for f in (A.FLUX_HLL, A.FLUX_HLLC, A.FLUX_GODUNOV, A.FLUX_HLLC_A)]
    out = []
    for full in (0, 1):
        with solver.Batch([both(c)[full] for c in cfgs]) as B:
            for i, c in enumerate(cfgs):
                B.set_state(i, *moving(c, 0.1 * i, 0.0))
            B.set_mixed(mixed)
            B.step(15)
            out.append([(*B.get_state(i), B.clock(i), B.stats(i)) for i in range(len(cfgs))])
    for a, b in zip(*out):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2:] == b[2:]


@pytest.mark.parametrize("precision", [A.PREC_FP32, A.PREC_FP64])
@pytest.mark.parametrize("flux", [A.FLUX_HLL, A.FLUX_GODUNOV])
def test_host_array_bands(precision, flux):
    torch = pytest.importorskip("torch")
    cfg = problems.blast_config(1500, 700, flux=flux, precision=precision)
    s, u = moving(cfg, 0.25, 0.0)
    out = []
    for c in both(cfg):
        a = [torch.zeros(s.shape, dtype=torch.float64, pin_memory=True) for _ in range(4)]
        a[0].numpy()[:], a[1].numpy()[:] = s, u
        with solver.Solver(c) as S:
            S.step_host_n(3, *(t.data_ptr() for t in a))
            S.synchronize()
            out.append([t.numpy().copy() for t in a] + [S.clock(), S.stats()])
    assert all(np.array_equal(x, y) for x, y in zip(out[0][:4], out[1][:4]))
    assert out[0][4:] == out[1][4:], (out[0][4:], out[1][4:])
