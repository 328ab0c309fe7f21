"""The warp pass's roles and candidate blocks at the sizes where they can go
wrong, and the ways work is spread, which must change no result.

The warp pass splits a force evaluation into independent sums (one warp each),
walks the candidates in blocks of four per lane, keeps small targets in
registers or packed, and runs usual steps and free flights in loops of their
own; the lane pass spreads few trajectories over all warps.
"""
import numpy as np
import pytest

import os

from helpers import engine_for, input_dict, workdir, write_input

pytestmark = pytest.mark.gpu


def _system(oracle, natoms, gas, ft, net=1.0):
    """A globule of natoms atoms at protein density, net charge +1 e."""
    from massccs_b200 import synth
    d = workdir(files=())
    rng = np.random.default_rng(natoms)
    sym, xyz, q = synth.globule_atoms(natoms, 1.3 * natoms ** (1 / 3) * (5 / 3) ** 0.5, net, rng)
    synth.write_xyz(os.path.join(d, "target.xyz"), sym, xyz, q)
    return oracle.OracleSystem(write_input(d, input_dict("target.xyz", gas, ft)))


# atoms per virtual thread (64): below one, exactly one, one more, two (the
# register-held limit), one more (lists), a whole block of four, one more
SIZES = [5, 63, 64, 65, 128, 129, 256, 257]


@pytest.mark.parametrize("natoms", SIZES)
@pytest.mark.parametrize("gas,ft", [("He", 4), ("He", 2), ("N2", 6), ("N2", 4), ("N2", 2), ("CO2", 6)])
def test_fp64_warp_pass_matches_oracle_at_block_edges(oracle, natoms, gas, ft):
    """Nearly every step in the warp pass (parked after 16).  The bars are those
    of the FP64 trajectory tests on charged globules: the shares that agree
    with the oracle (chaotic orbits differ between any two builds)."""
    n = 120
    s = _system(oracle, natoms, gas, ft)
    rnd = s.predraw(n)
    ref = s.run(rnd)
    out = engine_for(s, precision=1, park_steps=16, lanes_per_traj=32).run(rnd)
    assert out["stats"]["parked"] > n // 4
    same = out["status"] == ref["status"]
    close = same & (np.abs(out["one_minus_cos"] - ref["one_minus_cos"]) <= 1e-7)
    assert close.mean() >= {"He": 0.97, "N2": 0.90, "CO2": 0.85}[gas], close.mean()


@pytest.mark.parametrize("natoms", [5, 64, 65, 128, 129, 257, 513])
@pytest.mark.parametrize("gas,ft", [("He", 4), ("N2", 6), ("CO2", 6), ("N2", 5)])
def test_fp32_splits_of_a_run_change_no_result(oracle, natoms, gas, ft):
    """One run of n trajectories against the same ones in runs of their own
    (other trajectories per warp, other CTAs, other tries at once): every
    trajectory's arithmetic is the same, so its results are, bit for bit."""
    n = 192
    s = _system(oracle, natoms, gas, ft)
    rnd = s.predraw(n)
    eng = engine_for(s, precision=0, park_steps=64, lanes_per_traj=32)
    whole = eng.run(rnd)
    seq = engine_for(s, precision=0, park_steps=64, lanes_per_traj=32, spec_tries=-1)
    parts = []
    for lo, hi in ((0, 1), (1, 34), (34, 127), (127, n)):
        parts.append(seq.run(np.ascontiguousarray(rnd[:, lo:hi])))
    for key in ("status", "one_minus_cos", "steps", "visits"):
        assert np.array_equal(whole[key], np.concatenate([p[key] for p in parts])), key


@pytest.mark.parametrize("gas,ft", [("He", 4), ("N2", 6)])
def test_wide_run_equals_narrow_run(oracle, gas, ft):
    """Enough trajectories to fill every warp of the lane pass, and the first
    of them alone: other lanes, other trajectories per warp, same results."""
    s = _system(oracle, 300, gas, ft)
    rnd = s.predraw(20000)
    eng = engine_for(s, precision=0, lanes_per_traj=32)
    wide = eng.run(rnd)
    narrow = eng.run(np.ascontiguousarray(rnd[:, :500]))
    for key in ("status", "one_minus_cos", "steps", "visits"):
        assert np.array_equal(wide[key][:500], narrow[key]), key
