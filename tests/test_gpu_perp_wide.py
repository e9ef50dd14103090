"""Shell diffusion and drift of runs whose (node, energy) slices are too large for
shared memory: one pass per operator from one f buffer into a second one, which the
runs whose slices fit do without.  FP64 within the plain form's 1e-12 of the oracle,
FP32 flux within 1e-3."""
import numpy as np
import pytest
import torch

from eprem_gb300 import EpremRun, abi, workloads as W

from helpers import rel_err
from test_gpu_drift import gpu_drift_run, primed, random_news

pytestmark = pytest.mark.gpu

KP = 0.05


def _reference(w, oracle_lib, calls, shell, drift):
    d, g, nodes, curl, f = primed(oracle_lib, w)
    news = random_news(d.num_streams, seed=11)
    gs, keep = W.grids_struct(g)
    f_ref, n_ref = f.copy(), nodes.copy()
    for _ in range(calls):
        if drift:
            rc, _, err = oracle_lib.update_energetic_particles_perp(
                d, w.params, gs, f_ref, n_ref, news, KP if shell else None, W.drift_params(w, g),
                curl, nthreads=8)
        else:
            rc, _, err = oracle_lib.update_energetic_particles(d, w.params, gs, f_ref, n_ref,
                                                               nthreads=8, news=news,
                                                               kperxkpar=KP)
        assert rc == 0, err
    return d, g, gs, news, f, nodes, f_ref


def _run(w, precision, g, news, nodes, shell, drift):
    if drift:
        return gpu_drift_run(w, precision, g, news, KP if shell else None, 0)
    run = EpremRun(w.dims(precision), w.params, g)
    run.set_shell_diffusion(news, KP)
    run.upload_nodes(nodes)
    return run


@pytest.mark.parametrize("sub_steps", [1, 2])
@pytest.mark.parametrize("shell,drift", [(1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("mu", [40, 39])
def test_wide_slices(mu, shell, drift, sub_steps, oracle_lib):
    w = W.custom(10, 10, 4, 2, mu, num_ep_steps=sub_steps)
    d, g, gs, news, f, nodes, f_ref = _reference(w, oracle_lib, 2, shell, drift)
    run = _run(w, abi.EPREM_FP64, g, news, nodes, shell, drift)
    run.upload_f(f)
    for _ in range(2):
        run.update_energetic_particles(0.0)
    run.read_stats()
    out = run.download_f()
    run.close()
    assert rel_err(out, f_ref) <= 1e-12
    j_ref = oracle_lib.omni_flux(d, gs, f_ref)
    run = _run(w, abi.EPREM_FP32, g, news, nodes, shell, drift)
    run.upload_f(f)
    for _ in range(2):
        run.update_energetic_particles(0.0)
    run.read_stats()
    j = run.omni_flux()
    run.close()
    mask = j_ref > 1e-30 * j_ref.max()
    assert float(np.max(np.abs(j[mask] - j_ref[mask]) / j_ref[mask])) <= 1e-3


@pytest.mark.parametrize("precision", [abi.EPREM_FP64, abi.EPREM_FP32])
def test_second_f_only_where_slices_do_not_fit(precision):
    """What switching shell diffusion and drift on takes of the device's memory: per
    (stream, node, energy) nine fractions, and f itself only for wide slices."""
    for rows, cols, nodes, energies, wide in ((4, 4, 1000, 10, False), (10, 10, 100, 10, True)):
        w = W.custom(rows, cols, nodes, energies, 40)
        g = W.build_grids(w)
        run = EpremRun(w.dims(precision), w.params, g)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        news = random_news(w.num_streams, seed=3)
        run.set_shell_diffusion(news, KP)
        run.set_drift(news, W.drift_params(w, g))
        run.synchronize()
        taken = before - torch.cuda.mem_get_info()[0]
        run.close()
        rest = 9 * 8 * w.cells // w.num_mu + 3 * 8 * w.num_streams * nodes + (16 << 20)
        f_bytes = w.cells * (8 if precision == abi.EPREM_FP64 else 4)
        assert (taken > f_bytes) if wide else (taken <= rest), (taken, rest, f_bytes)
        assert wide or rest < f_bytes
