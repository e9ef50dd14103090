"""An ensemble's autotuner keeps runs of one size apart that differ in what their
kernels need: with and without the seed boundary."""
import pytest

from eprem_gb300 import EpremRun, Ensemble, abi, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [(1, 0), (0, 1)])
@pytest.mark.parametrize("mu", [40, 24])
def test_ensemble_of_runs_with_and_without_the_boundary(order, mu):
    runs = []
    for boundary in order:
        w = W.custom(4, 4, 1000, 8, mu, num_ep_steps=2, use_ep_boundary=boundary)
        g = W.build_grids(w)
        run = EpremRun(w.dims(abi.EPREM_FP32), w.params, g)
        run.upload_nodes(W.initial_nodes(w))
        run.update_mhd(0.0)
        run.init_seed_population(1, 0.01)
        runs.append(run)
    alone = []
    for run in runs:  # what each run's own tuner may choose
        run.autotune()
        alone.append(run.stream_kernel.startswith("k_stream2m"))
        run.set_stream_variant(0)
    ens = Ensemble(runs)
    ens.autotune()
    for boundary, run in zip(order, runs):
        if not boundary:
            assert not run.stream_kernel.startswith("k_stream2m")
    assert [r.stream_kernel.startswith("k_stream2m") for r in runs] == alone
    ens.step()
    ens.synchronize()
    ens.close()
    for run in runs:
        run.close()
