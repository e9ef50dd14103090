"""A cell that is not a number, of either sign bit, is an error at the node phase
(FP64) and stays what it is in f."""
import numpy as np
import pytest

from eprem_gb300 import EpremGpuError, EpremRun, abi, workloads as W

from helpers import primed_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("focus,change", [(1, 0), (0, 1), (1, 1)])
def test_cell_stays(sign, focus, change, oracle_lib):
    w = W.custom(1, 1, 40, 6, 8, num_ep_steps=1, use_parallel_diffusion=0,
                 use_adiabatic_focus=focus, use_adiabatic_change=change, check_seed_population=0)
    d, g, f, nodes = primed_state(w, oracle_lib)
    cells = f.reshape(w.num_streams, w.num_nodes, 6, 8)
    cells[2, 20, 3, 4] = np.copysign(np.nan, sign)
    run = EpremRun(d, w.params, g)
    run.upload_f(f)
    run.upload_nodes(nodes)
    run.update_energetic_particles(0.0)
    with pytest.raises(EpremGpuError) as ei:
        run.read_stats()
    assert ei.value.code == abi.EPREM_GPU_ERR_NAN
    assert "node 20" in str(ei.value), str(ei.value)
    out = run.download_f().reshape(cells.shape)
    run.close()
    assert np.isnan(out[2, 20, 3, 4])
    assert np.isnan(out).sum() == np.isnan(out[2, 20]).sum()
