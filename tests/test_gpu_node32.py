"""FP32 focusing and change in one pass over whole nodes (node32.cuh): the edges
of the row buckets, each access width (mu counts of a bucket, even, odd) with
CTAs that start at every alignment, the smallest and largest energies, a ragged
last CTA, and either operator alone.  Held to the form's 1e-3 of the FP64 oracle
on every cell that is not within float's floor of its row's top; sub-cycle
counts equal."""
import numpy as np
import pytest

from eprem_gb300 import EpremRun, abi, workloads as W

from helpers import oracle_update, primed_state

pytestmark = pytest.mark.gpu


def _check(w, oracle_lib, tweak=None):
    d, g, f, nodes = primed_state(w, oracle_lib)
    if tweak:
        tweak(f.reshape(w.num_streams, w.num_nodes, w.num_energies, w.num_mu))
    f_ref, _, stats = oracle_update(oracle_lib, w, g, f, nodes)
    run = EpremRun(w.dims(abi.EPREM_FP32), w.params, g)
    run.upload_f(f)
    run.upload_nodes(nodes)
    run.update_energetic_particles(0.0)
    st = run.read_stats()
    out = run.download_f()
    run.close()
    rows = f_ref.reshape(-1, w.num_mu)
    seen = (rows > 1e-60 * rows.max(1, keepdims=True)).reshape(-1)
    assert np.max(np.abs(out - f_ref)[seen] / f_ref[seen]) <= 1e-3
    assert st.focus_cell_subcycles == stats[0].focus_cell_subcycles
    assert st.change_cell_subcycles == stats[0].change_cell_subcycles


@pytest.mark.parametrize("mu", [2, 3, 7, 8, 9, 12, 15, 16, 17, 20, 21, 24, 25, 28, 32, 33, 40, 41,
                                48, 50, 56, 57, 63, 64])
def test_mu_counts(mu, oracle_lib):
    _check(W.custom(1, 1, 43, 7, mu, num_ep_steps=2, use_parallel_diffusion=0), oracle_lib)


@pytest.mark.parametrize("energies,mu", [(2, 33), (3, 22), (5, 9), (26, 33), (64, 40), (64, 64),
                                         (63, 7)])
def test_energy_counts(energies, mu, oracle_lib):
    _check(W.custom(1, 1, 31, energies, mu, num_ep_steps=2, use_parallel_diffusion=0), oracle_lib)


@pytest.mark.parametrize("switch", ["use_adiabatic_focus", "use_adiabatic_change"])
def test_either_operator_alone(switch, oracle_lib):
    for mu in (10, 20, 33):
        _check(W.custom(1, 1, 40, 9, mu, num_ep_steps=2, **{switch: 0}), oracle_lib)


def test_rows_with_a_far_tail(oracle_lib):
    """Cells down to 1e-50 of their row's top leave the fast logarithm and
    exponential; they come back within the form's bound."""
    def tweak(f):
        f *= 10.0 ** -np.linspace(0.0, 50.0, f.shape[-1])
    _check(W.custom(1, 1, 40, 6, 40, num_ep_steps=1, use_parallel_diffusion=0,
                    check_seed_population=0, use_adiabatic_focus=0), oracle_lib, tweak)


def test_cooling_and_its_damping(oracle_lib):
    _check(W.custom(1, 2, 60, 12, 14, num_ep_steps=3, damp_cooling=0.5), oracle_lib)


@pytest.mark.parametrize("nodes,mu", [(5, 33), (7, 22), (7, 20)])
def test_parts_of_a_run_that_begin_anywhere_in_f(nodes, mu, oracle_lib):
    """The host-memory update takes f's streams in parts: a part of odd streams
    of nodes x 27 x mu cells begins at any of float's alignments.  Bit-identical
    to the whole run's update."""
    w = W.custom(4, 4, nodes, 27, mu, num_ep_steps=1)
    _, g, f, values = primed_state(w, oracle_lib)
    out = []
    for host in (False, True):
        run = EpremRun(w.dims(abi.EPREM_FP32), w.params, g)
        run.upload_nodes(values)
        if host:
            got = np.empty_like(f)
            run.update_energetic_particles_host(f, got, 0.0)
        else:
            run.upload_f(f)
            run.update_energetic_particles(0.0)
            got = run.download_f()
        run.close()
        out.append(got)
    np.testing.assert_array_equal(out[0], out[1])
