"""FP64 focusing and change (node64.cu): the smallest and largest rows and
columns, counts that leave lanes idle, a ragged last CTA, Euler and third-order
operators, and either operator alone, within 1e-12 of the oracle; sub-cycle
counts, whose speeds are prefiltered in float, exactly equal."""
import numpy as np
import pytest

from eprem_gb300 import EpremRun, abi, workloads as W

from helpers import oracle_update, primed_state, rel_err

pytestmark = pytest.mark.gpu

F_RTOL = 1e-12


def _check(w, oracle_lib, tweak=None):
    d, g, f, nodes = primed_state(w, oracle_lib)
    if tweak:
        tweak(nodes)
    f_ref, _, stats = oracle_update(oracle_lib, w, g, f, nodes, calls=2)
    run = EpremRun(d, w.params, g)
    run.upload_f(f)
    run.upload_nodes(nodes)
    got = []
    for _ in range(2):
        run.update_energetic_particles(0.0)
        got.append(run.read_stats())
    out = run.download_f()
    run.close()
    assert rel_err(out, f_ref) <= F_RTOL
    for a, b in zip(got, stats):
        assert a.max_subcycles_focusing == b.max_subcycles_focusing
        assert a.max_subcycles_change == b.max_subcycles_change
        assert a.focus_cell_subcycles == b.focus_cell_subcycles
        assert a.change_cell_subcycles == b.change_cell_subcycles


@pytest.mark.parametrize("alg", [1, 2])
@pytest.mark.parametrize("energies,mu", [(2, 2), (2, 64), (64, 2), (3, 5), (17, 33), (50, 40),
                                         (64, 64)])
def test_sizes(energies, mu, alg, oracle_lib):
    _check(W.custom(1, 1, 37, energies, mu, num_ep_steps=2, adiabatic_focus_alg=alg,
                    adiabatic_change_alg=alg), oracle_lib)


@pytest.mark.parametrize("focus,change", [(1, 2), (2, 1)])
def test_mixed_operators(focus, change, oracle_lib):
    _check(W.custom(1, 2, 50, 12, 9, num_ep_steps=2, adiabatic_focus_alg=focus,
                    adiabatic_change_alg=change, damp_cooling=0.4), oracle_lib)


@pytest.mark.parametrize("scale", [1e-40, 1e-27, 40.0])
def test_rates_outside_and_inside_the_float_prefilter(scale, oracle_lib):
    """Nodes whose rates are far below the float prefilter's range take the
    exact expressions everywhere; larger ones take many sub-cycles."""
    def tweak(nodes):
        for fld in ("DLNB", "DLNN", "DUPAR"):
            nodes[abi.NODE[fld], 5:40] *= scale
        if scale < 1.0:
            nodes[abi.NODE["BMAG"], 5:40] = 1.0  # no focusing by dlnB/ds either
    _check(W.custom(1, 1, 60, 8, 10, num_ep_steps=2), oracle_lib, tweak)


def test_logarithm_and_exponential(oracle_lib):
    """Nodes whose rates are zero take no sub-cycle, so the change writes back
    exp(ln f): ln to half a unit in its last place (7e-17 below 1) and exp to 0.7
    of one, with room for a tenth of each, over the whole range of f."""
    w = W.custom(1, 1, 40, 8, 12, num_ep_steps=1, use_parallel_diffusion=0,
                 use_adiabatic_focus=0, check_seed_population=0)
    d, g, f, nodes = primed_state(w, oracle_lib)
    for fld in ("DLNB", "DLNN", "DUPAR"):
        nodes[abi.NODE[fld]] = 0.0
    rng = np.random.default_rng(3)
    f = np.exp(rng.uniform(-700.0, 700.0, f.size))
    f[::7] = np.exp(rng.uniform(-2.0, 2.0, f[::7].size))
    f[0::1001] = np.finfo(np.float64).tiny
    run = EpremRun(d, w.params, g)
    run.upload_f(f)
    run.upload_nodes(nodes)
    run.update_energetic_particles(0.0)
    assert run.read_stats().max_subcycles_change == 0
    out = run.download_f()
    run.close()
    eps = 2.0 ** -53
    bound = 1.1 * (np.maximum(np.spacing(np.abs(np.log(f))) / 2.0, 7e-17) + 1.4 * eps) + eps
    assert np.all(np.abs(out - f) <= bound * f)
