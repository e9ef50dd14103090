"""FP32 streaming plans of lists that fill their CTA: every slot of the widest thread
counts, none is kept free (no GPU: the planner alone).  20 and 40 mu cells, whose
shapes have numbers of their own, keep theirs."""
import pytest

from eprem_gb300 import abi, runtime

# mu count, list nodes per thread of the widest thread
WIDEST = [(4, 16), (8, 10), (12, 8), (16, 8), (24, 6), (28, 5), (33, 5), (36, 4), (44, 3),
          (48, 3), (52, 3), (56, 2), (63, 2), (64, 2)]


@pytest.mark.parametrize("mu,npt", WIDEST)
def test_one_cta_holds_what_its_threads_hold(mu, npt):
    full = runtime.plan_stream(256 * npt, mu, mu // 2, abi.EPREM_FP32)
    assert (full["threads"], full["npt"], full["cluster"]) == (256, npt, 1)
    over = runtime.plan_stream(256 * npt + 1, mu, mu // 2, abi.EPREM_FP32)
    assert over["cluster"] > 1


@pytest.mark.parametrize("mu,npt", WIDEST)
@pytest.mark.parametrize("ctas", [3, 5, 8])
def test_clusters_hold_what_their_threads_hold(mu, npt, ctas):
    nodes = ctas * 128 * npt
    if nodes > (8192 if mu <= 40 else 6144 if mu <= 48 else 4096):
        pytest.skip("longer than a run of this mu count may be")
    p = runtime.plan_stream(nodes, mu, mu // 2, abi.EPREM_FP32)
    assert p["threads"] * p["npt"] * p["cluster"] >= nodes
    if (p["threads"], p["npt"]) == (128, npt):
        assert p["cluster"] == ctas
