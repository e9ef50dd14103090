"""FP64 streaming where a node drains by many decades within one launch: weak
scattering, over ten thousand sub-cycles and a pulse far above the seed that leaves
the stream.  The isotropisation term is carried over the sub-cycles and must not
keep the last place of what it was while the pulse stood there.  Held to the plain
form's 1e-12 of the same recurrence with the mean summed in every sub-cycle, cell
by cell in numpy (the reference's iso + (f - iso) em rounds f to the last place of
iso, 1e-7 of f here)."""
import numpy as np
import pytest

from eprem_gb300 import EpremRun, abi, workloads as W

from helpers import primed_state

pytestmark = pytest.mark.gpu

F_RTOL = 1e-12


def _slab(w, g, f, nodes, s, e):
    """One (stream, energy) slab's streaming of one sub-step; nothing is thinned."""
    p, N, M = w.params, w.num_nodes, w.num_mu
    xyz = np.array([nodes[abi.NODE[k]].reshape(-1, N)[s] for k in ("RX", "RY", "RZ")]) * p.r_scale
    seg = np.sqrt(((xyz[:, 1:] - xyz[:, :-1]) ** 2).sum(0))
    ds = np.concatenate([seg[:1], 0.5 * (seg[1:] + seg[:-1]), seg[-1:]])
    dt = p.t_del / p.num_ep_steps
    nst = int(np.floor(dt / (0.4 * seg.min() * g["vgrid_i"][e]) + 1.0))
    dtp = dt / nst
    tau = g["vgrid_i"][e] * (g["rigidity"][e] * p.lamo)  # no dependence on r
    em = np.exp(-dtp / tau)
    assert dtp < tau
    c = (1.0 / ds)[:, None] * (g["vgrid"][e] * dtp * np.abs(g["mugrid"]))
    m0 = M // 2
    cl, cr = c[:-1, :m0], c[1:, m0:]
    h = f.reshape(-1, N, w.num_energies, M)[s, :, e].copy()
    seed = h[:3].copy()
    z = np.empty_like(h)
    for _ in range(nst):
        h[:3] = seed
        z[:-1, :m0] = h[:-1, :m0] + cl * (h[1:, :m0] - h[:-1, :m0])
        z[-1, :m0] = h[-1, :m0]
        z[1:, m0:] = h[1:, m0:] + cr * (h[:-1, m0:] - h[1:, m0:])
        z[0, m0:] = h[0, m0:]
        h = em * z + ((1.0 - em) * (z.sum(1) / M))[:, None]
    return h, nst


# (exp(-dt/tau) lies a tenth of its last place or more from a rounding boundary in
# every stream and energy here, so that its two libraries agree on it)
@pytest.mark.parametrize("nodes,mu,lamo,t_del,kernel", [
    (60, 6, 1e7, 120.0, "k_stream64_short"), (128, 40, 1e6, 120.0, "k_stream64_short"),
    (200, 20, 3e6, 40.0, "k_stream64<"), (600, 40, 3e5, 15.0, "k_stream64<")])
def test_node_that_drains(nodes, mu, lamo, t_del, kernel, oracle_lib):
    w = W.custom(1, 1, nodes, 2, mu, r_min=1.0, r_max=2.0, num_ep_steps=1, lamo=lamo,
                 t_del=t_del, use_adiabatic_focus=0, use_adiabatic_change=0, use_ep_boundary=0)
    d, g, f, fields = primed_state(w, oracle_lib)
    w.params.use_ep_boundary = 1
    cells = f.reshape(w.num_streams, nodes, 2, mu)
    # the boundary's seeds are those of the moved nodes: taken from the first pass
    # of a run that only checks the seed population
    w.params.use_parallel_diffusion = 0
    run = EpremRun(d, w.params, g)
    run.upload_f(np.zeros_like(f))
    run.upload_nodes(fields)
    run.update_energetic_particles(0.0)
    run.read_stats()
    seeds = run.download_f().reshape(cells.shape)
    run.close()
    w.params.use_parallel_diffusion = 1
    cells[...] = np.maximum(cells, seeds)
    cells[:, :3] = seeds[:, :3]
    cells[:, nodes // 3:nodes // 2] *= 1e15
    run = EpremRun(d, w.params, g)
    assert run.stream_kernel.startswith(kernel)
    run.upload_f(f)
    run.upload_nodes(fields)
    run.update_energetic_particles(0.0)
    assert run.read_stats().max_substeps_stream > 10000
    out = run.download_f().reshape(cells.shape)
    run.close()
    for s, e in ((4, 1), (5, 1)):  # the polar faces' streams, the most sub-cycles
        ref, nst = _slab(w, g, f, fields, s, e)
        assert nst > 10000
        assert np.max(cells[s, :, e].sum(1) / ref.sum(1)) > 1e6
        assert np.max(np.abs(out[s, :, e] - ref) / ref) <= F_RTOL
