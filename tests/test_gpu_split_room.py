"""Forms that need room of their own (near-field lists dealt to several blocks, direct sums split over the sources, sorted
treecode queries, split M2L and M2M tiles): without that room the plain forms run, to the same results up to the
order of the sums."""
import numpy as np
import pytest

from bachelors_b200 import Plan

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
def test_results_without_room(monkeypatch, precision, tol):
    rng = np.random.default_rng(5)
    n, m = 20000, 2003
    xyz, w, J, tgt = rng.uniform(-1, 1, (n, 3)), rng.uniform(0.5, 1, n), rng.normal(size=(n, 3)), rng.uniform(-1.2, 1.2, (m, 3))
    pts = rng.uniform(-2, 2, (40000, 3))

    def everything():
        plan = Plan(order=7, leaf_capacity=700, precision=precision)
        plan.set_sources(xyz, w, J)
        plan.set_targets(tgt)
        out = [plan.direct(1.0, 1)[0], plan.direct_fp64(tgt[:9])]
        out += plan.solve(1.0, 3)
        out += plan.treecode(pts, 1.0, 3)
        plan.graph_capture(1)
        out.append(plan.graph_launch(1.0)[0])
        out = [np.array(v, np.float64) for v in out]
        plan.close()
        return out

    split = everything()
    monkeypatch.setenv("FMM_SPLIT_SUMS", "0")
    for a, b in zip(split, everything()):
        assert rel(a, b) < tol
