"""An ensemble step comes after everything its runs have queued on their own
streams: the runs are not waited for on the host in between."""
import numpy as np
import pytest

from eprem_gb300 import Ensemble, EpremRun, abi, workloads as W

from helpers import primed_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chains", [-1, 0, 2])
def test_step_follows_the_runs_queued_work(chains, oracle_lib):
    ws = [W.custom(2, 2, 300, 12, 12, num_ep_steps=10) for _ in range(4)]
    _, g, f, nodes = primed_state(ws[0], oracle_lib)
    results = []
    for wait in (True, False):
        runs = [EpremRun(w.dims(abi.EPREM_FP32), w.params, g) for w in ws]
        ens = Ensemble(runs)
        ens.set_chains(chains)
        for call in range(2):  # the first one makes the graph
            for r in runs:
                r.upload_f(f)
                r.upload_nodes(nodes)
                r.synchronize()
            ens.set_time([0.0] * 4)
            for r in runs:
                r.update_energetic_particles(0.0)
                if wait:
                    r.synchronize()
            ens.step()
            ens.synchronize()
        results.append([r.download_f() for r in runs])
        ens.close()
        for r in runs:
            r.close()
    for a, b in zip(*results):
        np.testing.assert_array_equal(a, b)
