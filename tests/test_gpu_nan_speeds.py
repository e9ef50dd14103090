"""A face speed that is not a number (from a mu grid with a hole) is an error at the
focusing, as in the reference's upwind flux, in both forms."""
import numpy as np
import pytest

from eprem_gb300 import EpremGpuError, EpremRun, abi, workloads as W

from helpers import primed_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.EPREM_FP64, abi.EPREM_FP32])
@pytest.mark.parametrize("mu", [8, 10, 13])
def test_face_speed(precision, mu, oracle_lib):
    w = W.custom(1, 1, 40, 6, mu, num_ep_steps=1, use_parallel_diffusion=0,
                 use_adiabatic_change=0)
    d, g, f, nodes = primed_state(w, oracle_lib, precision)
    g["mugrid"] = g["mugrid"].copy()
    g["mugrid"][2] = np.nan
    run = EpremRun(d, w.params, g)
    run.upload_f(f)
    run.upload_nodes(nodes)
    run.update_energetic_particles(0.0)
    with pytest.raises(EpremGpuError) as ei:
        run.read_stats()
    assert ei.value.code == abi.EPREM_GPU_ERR_NAN
    assert "Adiabatic Focusing" in str(ei.value), str(ei.value)
    run.close()
