"""FP32 change of rows that rise or fall by more powers of two in one sub-step than
float's exponential and scalings hold: a strong shock over spectra whose energies
lie up to 2^370 apart.  Held to the form's 1e-3 of the FP64 oracle on every cell that
is not within float's floor of its row's top or of the exponents' limit."""
import numpy as np
import pytest

from eprem_gb300 import EpremRun, abi, workloads as W

from helpers import oracle_update, primed_state

pytestmark = pytest.mark.gpu


def _shock(energies, mu, **kw):
    w = W.testsuite_like("cone", 1, 1, 60)
    w.num_energies, w.num_mu, w.e_max = energies, mu, 1000.0
    p = w.params
    p.num_ep_steps = 1
    p.ideal_shock_init_time = 0.0
    p.ideal_shock_jump = 4.0
    p.use_parallel_diffusion = p.use_adiabatic_focus = 0
    for k, v in kw.items():
        setattr(p, k, v)
    return w


def _update(w, g, f, nodes):
    run = EpremRun(w.dims(abi.EPREM_FP32), w.params, g)
    try:
        run.upload_f(f)
        run.upload_nodes(nodes)
        run.update_energetic_particles(0.0)
        run.read_stats()
        return run.download_f()
    finally:
        run.close()


def _check(w, g, f, nodes, oracle_lib):
    """Powers of two by which the rows' tops rose (largest) and fell."""
    f_ref, _, _ = oracle_update(oracle_lib, w, g, f, nodes)
    rows = f_ref.reshape(-1, w.num_mu)
    top = rows.max(1, keepdims=True)
    out = _update(w, g, f, nodes)
    seen = ((rows > 1e-50 * top) & (rows > 1e-290)).reshape(-1)
    assert np.all(np.isfinite(out))
    assert np.max(np.abs(out - f_ref)[seen] / f_ref[seen]) <= 1e-3
    rise = np.log2(top / f.reshape(-1, w.num_mu).max(1, keepdims=True))
    return rise.max(), rise.min()


@pytest.mark.parametrize("energies,mu", [(6, 8), (12, 33), (12, 20), (20, 8)])
def test_seed_spectrum(energies, mu, oracle_lib):
    w = _shock(energies, mu)
    _, g, f, nodes = primed_state(w, oracle_lib)
    rise, _ = _check(w, g, f, nodes, oracle_lib)
    assert rise > 128


@pytest.mark.parametrize("energies,mu,decades", [(5, 20, -65.0), (6, 33, -45.0), (4, 2, 90.0),
                                                 (5, 4, 60.0), (4, 8, 90.0), (4, 64, 60.0)])
def test_power_laws(energies, mu, decades, oracle_lib):
    """f changes by so many decades from energy to energy."""
    w = _shock(energies, mu, check_seed_population=0)
    _, g, f, nodes = primed_state(w, oracle_lib)
    e = np.arange(energies) if decades < 0 else np.arange(energies) - energies + 1
    f.reshape(-1, energies, mu)[...] = (10.0 ** (decades * e))[:, None]
    rise, fall = _check(w, g, f, nodes, oracle_lib)
    assert rise > 128 or fall < -35
