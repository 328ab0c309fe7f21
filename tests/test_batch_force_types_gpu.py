"""Batched ions of different force types in one call (GPU): charged targets
with LJ only, with Coulomb, and with the induced dipole too.  The kernels of a
batch are those of its richest ion, and every ion must still come out as in a
run of its own.  FP64, the shorter half of trajectories aimed at the target;
rounding (1e-16 a step) stays far below 1e-7 there."""
import numpy as np
import pytest

from helpers import engine_for
from test_warp_roles_gpu import _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gas,types", [("N2", (2, 4, 6)), ("N2", (6, 2, 5)), ("CO2", (6, 4, 2)), ("He", (4, 2, 3))])
def test_batch_of_mixed_force_types_matches_separate_runs(oracle, gas, types):
    from massccs_b200 import engine as E
    n = 160
    systems = [_system(oracle, 300 + 50 * k, gas, ft, net=3.0) for k, ft in enumerate(types)]
    rnds = []
    for s in systems:
        rnd = s.predraw(n)
        rnd[0] *= 0.4
        rnds.append(rnd)
    engs = [engine_for(s, precision=1, park_steps=16, lanes_per_traj=32, resume_block=64) for s in systems]
    sep = [e.run(r) for e, r in zip(engs, rnds)]
    bat, st = E.run_batch(engs, rnds)
    assert st["parked"] == 3 * n
    for ft, a, b in zip(types, sep, bat):
        short = a["steps"] <= np.median(a["steps"])
        close = (a["status"] == b["status"]) & (np.abs(a["one_minus_cos"] - b["one_minus_cos"]) <= 1e-7)
        assert close[short].mean() >= 0.97, (ft, close[short].mean())
    for e in engs:
        e.close()
