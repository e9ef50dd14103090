"""FP32 streaming in mirror order of lists that fill their CTA, warp or cluster to the
last slot, and of lists that thinning leaves at such a length in a larger one: every
width bit for bit, the oracle and the scalar kernel within the form's bounds."""
import numpy as np
import pytest

from helpers import primed_state
from test_gpu_stream2m import _check, _stream, _workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes,mu", [(1024, 36), (512, 64), (768, 48), (512, 63), (768, 47),
                                      (1536, 24), (32, 64), (64, 56), (128, 37), (320, 33),
                                      (1280, 28), (512, 4)])
def test_full_ctas_and_warps(nodes, mu, oracle_lib):
    _check(_workload(nodes, mu), oracle_lib)


@pytest.mark.parametrize("nodes,mu", [(1536, 36), (1152, 48), (768, 64)])
def test_full_clusters(nodes, mu, oracle_lib):
    seen = _check(_workload(nodes, mu), oracle_lib)
    assert any("cluster 1" not in k for k in seen)


def test_longest_full_cluster(oracle_lib):
    """4,096 nodes take 17,140 sub-cycles, after which the form itself, in either
    kernel, is 1.06e-3 from the oracle at the outer nodes: the kernels alone."""
    w = _workload(4096, 39)
    _, g, f, nodes = primed_state(w, oracle_lib)
    auto, kernel = _stream(w, g, f, nodes, 0)
    assert kernel == "k_stream2m<39,128,4> cluster 8"
    scalar, _ = _stream(w, g, f, nodes, 3)
    assert np.max(np.abs(auto - scalar) / scalar) <= 1e-4


@pytest.mark.parametrize("nodes,mu,thin", [(1024 + 39, 36, 40), (512 + 39, 64, 40),
                                           (1536 + 39, 38, 40), (96 + 4, 33, 5)])
def test_thinned_to_a_full_length(nodes, mu, thin, oracle_lib):
    """The nodes packed at the inner end become one list node."""
    w = _workload(nodes, mu, dsh_min=5e-3 if thin == 40 else 5e-5)
    w.cluster_inner = thin
    _check(w, oracle_lib, widths=False)
