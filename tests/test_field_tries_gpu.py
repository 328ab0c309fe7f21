"""The learned field's warp pass with tries run at once (GPU): a try past the
one that decides a trajectory is skipped or stopped, which must change no
result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gas", ["N2", "He"])
def test_field_tries_at_once_equal_tries_in_sequence(tmp_path, gas):
    from massccs_b200 import host, synth
    n = 2000
    S = host.System(synth.globule(str(tmp_path), 1231, 4, gas=gas, ft=6 if gas == "N2" else 4, nprobe=n, niter=1))
    rnd = S.predraw(n)
    out = {}
    weights = None
    for tries in (0, -1):  # the default, and never at once
        eng = S.engine(precision=0, lanes_per_traj=32, park_steps=512, spec_tries=tries)
        if weights is None:  # little training: many failed energy tests, so many tries
            eng.field_train(samples=200000, iterations=200)
            weights = eng.field_get_weights()
        else:
            eng.field_setup()
            eng.field_set_weights(*weights)
        eng.field_enable(True)
        out[tries] = eng.run(rnd)
        eng.close()
    at_once, sequence = out[0], out[-1]
    assert at_once["stats"]["speculated"] > 0 and sequence["stats"]["speculated"] == 0
    for key in ("status", "one_minus_cos", "steps", "visits"):
        assert np.array_equal(at_once[key], sequence[key]), key
    for key in ("nfree", "nscatter", "nlost", "ncapped", "steps", "visits"):
        assert at_once["stats"][key] == sequence["stats"][key], key
