"""Plans made, used and dropped by several threads at once: kernels launched with different sizes of shared memory, device
blocks and pinned words from what the process shares."""
import threading

import numpy as np
import pytest

from bachelors_b200 import Plan, geometry as G

pytestmark = pytest.mark.gpu


def small_problem(k):
    xyz, w, J = G.torus(12 + k, 8, 4, 2.0, 0.5)
    return xyz, w, J, G.uniform_points(100 + 31 * k, -3, 3, k)


def solve(k, plans=None):
    xyz, w, J, tgt = small_problem(k)
    plan = Plan(order=4 + 3 * (k % 4), leaf_capacity=10, precision="fp64" if k % 2 else "fp32")
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    out = [plan.solve(1.0, 1)[0], plan.direct(1.0, 1)[0], plan.treecode(tgt, 1.0, 1 + k % 3)[(1 + k % 3) // 2]]
    out = [np.array(v) for v in out]
    if plans is None:
        plan.close()
    else:
        plans.append(plan)
    return out


def test_plans_of_several_threads():
    """Eight threads make, use and drop plans of sizes of their own at once: every result is that of a single thread."""
    want = [solve(k) for k in range(8)]
    wrong = []

    def work(k):
        try:
            for r in range(12):
                kept = []
                for a, b in zip(solve((k + r) % 8, kept), want[(k + r) % 8]):
                    if not np.array_equal(a, b):
                        wrong.append((k, r))
                solve(k)
                kept[0].close()
        except Exception as e:   # (raised in the thread, reported by the test)
            wrong.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
