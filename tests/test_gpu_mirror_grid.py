"""The mirrored streaming kernels are refused on mu grids whose cells do not mirror,
however they are asked for."""
import numpy as np
import pytest

from eprem_gb300 import EpremGpuError, EpremRun, abi, workloads as W

from helpers import oracle_update, primed_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mu", [20, 40])
@pytest.mark.parametrize("kind", [6, 7])
def test_mirrored_kinds_need_a_mirrored_grid(kind, mu, oracle_lib):
    w = W.custom(1, 1, 80, 3, mu, num_ep_steps=2, use_adiabatic_focus=0, use_adiabatic_change=0)
    d, g, f, nodes = primed_state(w, oracle_lib)
    shifted = dict(g, mugrid=g["mugrid"] + 0.01)
    w.params.stream_variant = kind
    run = EpremRun(w.dims(abi.EPREM_FP32), w.params, g)  # its own grid: taken
    assert run.stream_kernel.startswith("k_stream2m")
    run.close()
    with pytest.raises(EpremGpuError):
        EpremRun(w.dims(abi.EPREM_FP32), w.params, shifted)
    w.params.stream_variant = 0
    f_ref, _, _ = oracle_update(oracle_lib, w, shifted, f, nodes)
    run = EpremRun(w.dims(abi.EPREM_FP32), w.params, shifted)
    with pytest.raises(EpremGpuError):
        run.set_stream_variant(kind)
    run.upload_f(f)
    run.upload_nodes(nodes)
    run.autotune()
    assert not run.stream_kernel.startswith("k_stream2m")
    run.update_energetic_particles(0.0)
    run.read_stats()
    out = run.download_f()
    run.close()
    assert np.max(np.abs(out - f_ref) / f_ref) <= 1e-3
