"""Contexts of one GPU used from several host threads at once (GPU): one
thread per context, targets that ask the same kernels for different amounts
of shared memory.  No call may be refused, and every result is that of the
context running alone, bit for bit."""
import threading

import numpy as np
import pytest

from helpers import engine_for
from test_warp_roles_gpu import _system

pytestmark = pytest.mark.gpu


def test_threads_with_targets_of_different_list_sizes(oracle):
    # N2 lists of 1231 and 2000 candidates, packed: 42 and 57 KB a CTA; short
    # runs, so that the threads' launches meet often
    jobs = []
    for natoms in (1231, 2000):
        s = _system(oracle, natoms, "N2", 6, net=4.0)
        rnd = s.predraw(4)
        for _ in range(4):
            eng = engine_for(s, precision=0, lanes_per_traj=32)
            jobs.append((eng, rnd, eng.run(rnd)))
    bad = []

    def work(eng, rnd, alone):
        for k in range(400):
            try:
                out = eng.run(rnd)
            except Exception as e:  # a refused launch
                bad.append((k, str(e)))
                continue
            if not all(np.array_equal(out[key], alone[key]) for key in ("status", "one_minus_cos", "steps", "visits")):
                bad.append((k, "results differ"))

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, (len(bad), bad[:3])
