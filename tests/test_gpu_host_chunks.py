"""The host-buffer update of runs with enough slabs to go through in chunks:
six of them here, the first and last of three streams.  Bit-identical to the
whole run's update, in place and out of place, contiguous and with the reference's
ghost shell before each stream; statistics and the stream of an error are the
run's."""
import numpy as np
import pytest

from eprem_gb300 import EpremGpuError, EpremRun, abi, workloads as W

from helpers import primed_state

pytestmark = pytest.mark.gpu

PRECISIONS = [abi.EPREM_FP64, abi.EPREM_FP32]


def _workload():
    return W.custom(4, 4, 20, 64, 6, num_ep_steps=2)


def _chunks(run, update):
    """Chunks of a host update, by the launches of one device-resident update."""
    n0 = run.kernel_launches
    run.update_energetic_particles(0.0)
    one = run.kernel_launches - n0
    n0 = run.kernel_launches
    update()
    fp32 = run.dims.precision == abi.EPREM_FP32
    return (run.kernel_launches - n0) / (one + (2 if fp32 else 0))  # two conversions a chunk


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("ghost", [False, True])
def test_chunked_update_equals_whole_run_update(precision, in_place, ghost, oracle_lib):
    w = _workload()
    d, g, f, nodes = primed_state(w, oracle_lib, precision)
    whole = EpremRun(d, w.params, g)
    whole.upload_f(f)
    whole.upload_nodes(nodes)
    whole.update_energetic_particles(0.0)
    st_w = whole.read_stats()
    f_w = whole.download_f()
    whole.close()
    S, per = d.num_streams, d.num_nodes * d.num_energies * d.num_mu
    gap = d.num_energies * d.num_mu if ghost else 0
    pitch = per + gap
    src = np.full(S * pitch, -7.0)
    src.reshape(S, pitch)[:, gap:] = f.reshape(S, per)
    dst = src if in_place else np.full_like(src, -7.0)
    run = EpremRun(d, w.params, g)
    run.upload_f(f)
    run.upload_nodes(nodes)

    def update():
        run.read_stats()  # what the update before counted
        run.update_energetic_particles_host(src[gap:], dst[gap:], 0.0,
                                            stream_pitch=pitch if ghost else 0)

    assert _chunks(run, update) == 6
    st = run.read_stats()
    run.close()
    np.testing.assert_array_equal(dst.reshape(S, pitch)[:, gap:].reshape(-1), f_w)
    assert np.all(dst.reshape(S, pitch)[:, :gap] == -7.0)
    assert st.as_dict() == st_w.as_dict()
    if not in_place:
        np.testing.assert_array_equal(src.reshape(S, pitch)[:, gap:], f.reshape(S, per))


@pytest.mark.parametrize("s_bad", [1, 40, 94])
def test_an_error_names_the_runs_stream(s_bad, oracle_lib):
    w = _workload()
    d, g, f, nodes = primed_state(w, oracle_lib)
    f.reshape(d.num_streams, 20, 64, 6)[s_bad, 15, 3, 2] = np.nan
    run = EpremRun(d, w.params, g)
    run.upload_nodes(nodes)
    with pytest.raises(EpremGpuError) as ei:
        run.update_energetic_particles_host(f, np.empty_like(f), 0.0)
    assert ei.value.code == abi.EPREM_GPU_ERR_NAN
    assert f"stream {s_bad}," in str(ei.value), str(ei.value)
    run.close()


def test_runs_of_few_slabs_go_in_one_piece(oracle_lib):
    """The long chunks hold 1,216 slabs or more on average: 90 streams of 27 energies
    between the two short chunks are 1,215 for each of two."""
    for rows, cols, energies, chunks in ((1, 5, 8, 1), (4, 4, 27, 1), (4, 4, 28, 4)):
        w = W.custom(rows, cols, 8, energies, 4, num_ep_steps=1)
        d, g, f, nodes = primed_state(w, oracle_lib)
        run = EpremRun(d, w.params, g)
        run.upload_f(f)
        run.upload_nodes(nodes)
        assert _chunks(run, lambda: run.update_energetic_particles_host(f, f, 0.0)) == chunks
        run.close()
