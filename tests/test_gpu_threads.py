"""Two host threads, each stepping a run of its own: the runs share the kernels'
attributes, so neither launch may depend on the other's size.  Results equal those
of the same steps one run after the other."""
import threading

import numpy as np
import pytest

from eprem_gb300 import EpremRun, abi, workloads as W

from helpers import primed_state

pytestmark = pytest.mark.gpu

STEPS = 150


def _steps(run, errors):
    try:
        for _ in range(STEPS):
            run.update_energetic_particles(0.0)
        run.read_stats()
    except Exception as e:  # noqa: BLE001 (handed to the test's thread)
        errors.append(e)


@pytest.mark.parametrize("precision,alg,sizes", [
    (abi.EPREM_FP64, 1, [(140, 20, 8), (500, 6, 8)]), (abi.EPREM_FP64, 3, [(40, 6, 8), (60, 16, 8)]),
    (abi.EPREM_FP32, 1, [(100, 20, 20), (1000, 6, 20)])])
def test_runs_of_two_sizes_side_by_side(precision, alg, sizes, oracle_lib):
    results = []
    for together in (False, True):
        runs = []
        for nodes, energies, mu in sizes:
            w = W.custom(1, 1, nodes, energies, mu, e_max=1.0, num_ep_steps=6,
                         adiabatic_focus_alg=alg, adiabatic_change_alg=alg)
            d, g, f, fields = primed_state(w, oracle_lib, precision)
            run = EpremRun(d, w.params, g)
            run.upload_f(f)
            run.upload_nodes(fields)
            run.synchronize()
            runs.append(run)
        errors = []
        threads = [threading.Thread(target=_steps, args=(r, errors)) for r in runs]
        for t in threads:
            t.start()
            if not together:
                t.join()
        for t in threads:
            t.join()
        assert not errors, errors
        results.append([r.download_f() for r in runs])
        for r in runs:
            r.close()
    for a, b in zip(*results):
        np.testing.assert_array_equal(a, b)
