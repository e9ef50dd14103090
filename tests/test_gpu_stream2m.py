"""FP32 streaming in mirror order (stream2m.cuh): every mu count's layout (pairs,
halves of odd length, the cell at mu = 0), every width (list nodes per thread),
list lengths at the edges of threads, warps, CTAs and clusters, thinned streams.
The widths hold the same arithmetic per node, so they agree bit for bit; the
scalar kernel (variant 3) agrees to 1e-4, the FP64 oracle to the form's 1e-3."""
import numpy as np
import pytest

from eprem_gb300 import EpremRun, abi, runtime, workloads as W

from helpers import oracle_update, primed_state

pytestmark = pytest.mark.gpu


def _workload(nodes, mu, **kw):
    return W.custom(1, 1, nodes, 3, mu, num_ep_steps=2, use_adiabatic_focus=0,
                    use_adiabatic_change=0, **kw)


def _stream(w, g, f, nodes, variant):
    w.params.stream_variant = variant
    try:
        run = EpremRun(w.dims(abi.EPREM_FP32), w.params, g)
    except RuntimeError:
        return None, ""
    finally:
        w.params.stream_variant = 0
    run.upload_f(f)
    run.upload_nodes(nodes)
    run.update_energetic_particles(0.0)
    run.read_stats()
    out, kernel = run.download_f(), run.stream_kernel
    run.close()
    return out, kernel


def _check(w, oracle_lib, widths=True):
    d, g, f, nodes = primed_state(w, oracle_lib)
    f_ref, _, _ = oracle_update(oracle_lib, w, g, f, nodes)
    auto, kernel = _stream(w, g, f, nodes, 0)
    assert kernel.startswith("k_stream2m"), kernel
    assert np.max(np.abs(auto - f_ref) / f_ref) <= 1e-3
    scalar, _ = _stream(w, g, f, nodes, 3)
    assert np.max(np.abs(auto - scalar) / scalar) <= 1e-4
    seen = {kernel}
    for shape in range(1, 12) if widths else ():
        out, kernel = _stream(w, g, f, nodes, 4 + 8 * shape)
        if kernel.startswith("k_stream2m"):
            seen.add(kernel)
            np.testing.assert_array_equal(out, auto)
    return seen


@pytest.mark.parametrize("mu", list(range(4, 65)))
def test_mu_counts_and_widths(mu, oracle_lib):
    seen = _check(_workload(131, mu), oracle_lib)
    assert mu > 55 or len(seen) >= 2


@pytest.mark.parametrize("nodes", [3, 4, 31, 32, 33, 63, 64, 65, 127, 129, 255, 257])
def test_list_lengths(nodes, oracle_lib):
    _check(_workload(nodes, 10), oracle_lib)


@pytest.mark.parametrize("nodes,mu", [(1023, 40), (1300, 33), (1025, 30), (2400, 10), (769, 48),
                                      (515, 63)])
def test_clusters(nodes, mu, oracle_lib):
    """More than 256 threads' nodes: clusters, their last CTA partly empty."""
    seen = _check(_workload(nodes, mu), oracle_lib)
    assert any("cluster 1" not in k for k in seen)


@pytest.mark.parametrize("thin", [5, 40])
def test_thinned_streams(thin, oracle_lib):
    """Shorter lists than the CTA was made for: idle threads, idle CTAs."""
    for nodes, mu in ((200, 23), (1300, 40)):
        w = _workload(nodes, mu, dsh_min=5e-3 if thin == 40 else 5e-5)
        w.cluster_inner = thin
        _check(w, oracle_lib, widths=False)


def test_without_the_seed_check(oracle_lib):
    _check(_workload(90, 22, check_seed_population=0), oracle_lib)


def test_other_mu_grids_keep_the_general_kernels(oracle_lib):
    """A mu grid that is not symmetric has no mirror cells."""
    w = _workload(80, 10)
    d, g, f, nodes = primed_state(w, oracle_lib)
    g["mugrid"] = g["mugrid"] + 0.01
    f_ref, _, _ = oracle_update(oracle_lib, w, g, f, nodes)
    out, kernel = _stream(w, g, f, nodes, 0)
    assert kernel.startswith("k_stream2_pairs")
    assert np.max(np.abs(out - f_ref) / f_ref) <= 1e-3


def test_every_length_that_a_plan_held_it_still_holds():
    for mu, most in ((8, 8192), (20, 8192), (24, 8192), (32, 8192), (40, 8192), (48, 6144),
                     (64, 4096)):
        for n in (3, 500, 1500, most):
            p = runtime.plan_stream(n, mu, mu // 2, abi.EPREM_FP32)
            assert p["slots"] >= n and p["cluster"] <= 8
