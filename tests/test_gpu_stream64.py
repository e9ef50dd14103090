"""FP64 streaming in three operations per cell (stream64.cu): list lengths at
the edges of warps, CTAs and clusters, mu counts at the edges of its bins,
mu grids that do not mirror, and streams long enough to fall back to the four-operation
kernel, each within the plain form's 1e-12 of the oracle on every cell."""
import numpy as np
import pytest

from eprem_gb300 import EpremRun, abi, runtime, workloads as W

from helpers import oracle_update, primed_state, rel_err

pytestmark = pytest.mark.gpu

F_RTOL = 1e-12


def _check(w, oracle_lib, g=None):
    d, g0, f, nodes = primed_state(w, oracle_lib)
    g = g or g0
    f_ref, _, stats = oracle_update(oracle_lib, w, g, f, nodes)
    run = EpremRun(d, w.params, g)
    run.upload_f(f)
    run.upload_nodes(nodes)
    run.update_energetic_particles(0.0)
    st = run.read_stats()
    out = run.download_f()
    kernel = run.stream_kernel
    run.close()
    assert rel_err(out, f_ref) <= F_RTOL
    assert st.stream_cell_subcycles == stats[0].stream_cell_subcycles
    return kernel


def _streaming(nodes, mu, **kw):
    return W.custom(1, 1, nodes, 3, mu, num_ep_steps=1, use_adiabatic_focus=0,
                    use_adiabatic_change=0, **kw)


@pytest.mark.parametrize("nodes", [4, 32, 33, 64, 255, 257, 513, 1025])
def test_list_lengths(nodes, oracle_lib):
    assert _check(_streaming(nodes, 40), oracle_lib).startswith("k_stream64")


@pytest.mark.parametrize("mu", [2, 3, 6, 7, 9, 13, 20, 21, 25, 29, 33, 48, 49, 64])
def test_mu_bins(mu, oracle_lib):
    assert _check(_streaming(70, mu), oracle_lib).startswith("k_stream64")


@pytest.mark.parametrize("seed_check,boundary", [(0, 0), (1, 0), (0, 1)])
def test_switches(seed_check, boundary, oracle_lib):
    _check(_streaming(100, 10, check_seed_population=seed_check, use_ep_boundary=boundary),
           oracle_lib)


@pytest.mark.parametrize("nodes,mu", [(512, 6), (512, 12), (512, 20), (512, 32), (512, 39),
                                      (384, 47), (256, 63), (257, 64)])
def test_widest_block_of_a_bin(nodes, mu, oracle_lib):
    assert _check(_streaming(nodes, mu), oracle_lib).startswith("k_stream64")


@pytest.mark.parametrize("rows,nodes,energies,mu,kernel", [
    (4, 40, 8, 6, "k_stream64<6>"), (4, 33, 14, 21, "k_stream64<24>"),
    (4, 64, 14, 40, "k_stream64<40>"), (1, 128, 3, 7, "k_stream64_short<8>"),
    (1, 128, 3, 64, "k_stream64_short<64>"), (1, 129, 3, 7, "k_stream64<8>")])
def test_short_streams_few_and_many(rows, nodes, energies, mu, kernel, oracle_lib):
    w = W.custom(rows, rows, nodes, energies, mu, e_max=1.0, num_ep_steps=1,
                 use_adiabatic_focus=0, use_adiabatic_change=0)
    assert _check(w, oracle_lib).startswith(kernel)


@pytest.mark.parametrize("m0", [0, 2, 7, 10])
def test_mu_grid_that_does_not_mirror(m0, oracle_lib):
    w = _streaming(60, 10)
    g = W.build_grids(w)
    g["mugrid"] = (np.arange(10) - m0 + 0.5) / 11.0
    assert _check(w, oracle_lib, g).startswith("k_stream<")


def test_thinned_stream(oracle_lib):
    w = _streaming(90, 8)
    w.cluster_inner = 9
    _check(w, oracle_lib)


def test_strong_scattering(oracle_lib):
    """exp(-dt/tau) from below the last place of the coefficients to near 1."""
    _check(_streaming(60, 8, lamo=1e-4), oracle_lib)


@pytest.mark.parametrize("nodes,mu,kernel", [(4096, 8, "k_stream64<8>"), (4097, 8, "k_stream<8>"),
                                             (3072, 48, "k_stream64<48>"),
                                             (2049, 64, "k_stream<64>")])
def test_longest_streams(nodes, mu, kernel, oracle_lib):
    w = W.custom(1, 1, nodes, 2, mu, e_max=0.2, num_ep_steps=1, use_adiabatic_focus=0,
                 use_adiabatic_change=0)
    assert _check(w, oracle_lib).startswith(kernel)


def test_plan_holds_every_stream_that_it_held():
    for mu, most in ((8, 8192), (16, 6144), (24, 4096), (40, 4096), (48, 3072), (64, 3072)):
        for n in (3, 100, 1000, most):
            p = runtime.plan_stream(n, mu, mu // 2, abi.EPREM_FP64)
            assert p["slots"] >= n and p["cluster"] <= 8
