"""The FP64 exact solver on the persistent tile kernel (grids of at least eight
32x16 tiles per SM): the same bits and counters as one CTA per tile, through
ast_step and the banded host-array step, with the learned start value and with
the recorder, on a ragged grid just past that line."""
import os

import numpy as np
import pytest

from asteriy_2d_gb300 import abi as A
from asteriy_2d_gb300 import problems, solver

pytestmark = pytest.mark.gpu
PARAMS = os.path.join(os.path.dirname(solver.__file__), "data", "guess_blast.npy")


def config(persistent):
    # 41 x 31 = 1271 tiles, the last column and row of them cut
    cfg = problems.blast_config(1291, 487, flux=A.FLUX_GODUNOV)
    cfg.persistent, cfg.collect_stats = persistent, 1
    s, u = solver.fill_blast(cfg, radius=0.3)
    u[:, 0] = np.linspace(-0.3, 0.4, len(u))      # disturbed everywhere
    u[: len(u) // 2] = 0.1                        # and uniform tiles
    return cfg, s, u


@pytest.mark.parametrize("newton", [0, 1])
@pytest.mark.parametrize("learned", [0, 1])
def test_persistent_equals_per_tile(newton, learned):
    out = []
    for persistent in (1, 0):
        cfg, s, u = config(persistent)
        cfg.riemann_newton, cfg.guess = newton, A.GUESS_MLP if learned else A.GUESS_PVRS
        with solver.Solver(cfg) as S:
            if learned:
                S.set_mlp(np.load(PARAMS))
            S.set_state(s, u)
            S.step(12)
            out.append((S.get_state(), S.clock(), S.stats()))
    (a, ca, sa), (b, cb, sb) = out
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and ca == cb
    assert sa == sb, (sa, sb)
    assert sa["bisect_calls"] + sa["newton_calls"] > 0


def test_banded_host_steps_equal_resident_steps():
    torch = pytest.importorskip("torch")
    cfg, s, u = config(1)
    with solver.Solver(cfg) as S:
        S.set_state(s, u)
        S.step(4)
        want, clock, stats = S.get_state(), S.clock(), S.stats()
    a = [torch.zeros(s.shape, dtype=torch.float64, pin_memory=True) for _ in range(4)]
    a[0].numpy()[:], a[1].numpy()[:] = s, u
    with solver.Solver(cfg) as S:
        S.step_host_n(4, *(t.data_ptr() for t in a))
        S.synchronize()
        assert S.clock() == clock and S.stats() == stats
    # an even number of steps ends in the first pair of arrays
    got = [(a[0].numpy(), a[1].numpy()), (a[2].numpy(), a[3].numpy())]
    assert any(np.array_equal(x, want[0]) and np.array_equal(y, want[1]) for x, y in got)


def test_recorder_records_the_same_faces():
    out = []
    for persistent in (1, 0):
        cfg, s, u = config(persistent)
        with solver.Solver(cfg) as S:
            S.set_state(s, u)
            S.record_start(1 << 20, 1, 0.05)
            S.step(2)
            rec, offered = S.record_stop()
        rec = rec[np.lexsort(rec.view(np.int32).reshape(rec.shape)[:, [8, 7]].T)]
        out.append((rec.tobytes(), offered, len(rec)))
    assert out[0] == out[1] and out[0][2] > 100
