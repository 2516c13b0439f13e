"""The pool of small device blocks: what it keeps of dropped plans, and what it gives back."""
import pytest

from bachelors_b200 import Plan, geometry as G

pytestmark = pytest.mark.gpu
KEEP, MB = 128 << 20, 1 << 20   # the pool's limit on freed blocks


def test_freed_blocks_are_kept_and_given_back(monkeypatch):
    """With more than the limit in use, a dropped plan's blocks are still kept for the next one; with nothing in use, at
    most the limit is."""
    import torch
    monkeypatch.setenv("FMM_SPLIT_SUMS", "0")   # (no large block for split sums: a plan is mostly small blocks)
    free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[1]
    xyz, w, J = G.torus(64, 24, 12, 2.0, 0.5)
    tgt = G.uniform_points(18000, -3, 3, 3)

    def make():
        plan = Plan(order=6, leaf_capacity=40, precision="fp32")
        plan.set_sources(xyz, w, J)
        plan.set_targets(tgt)
        plan.solve(1.0, 1)
        return plan

    make().close()
    empty = free()
    plans = [make()]
    while len(plans) < 100 and empty - free() < 3 * KEEP:
        plans.append(make())
    full = free()
    assert empty - full >= 2 * KEEP, "the plans are too small for this test"
    each = (empty - full) / len(plans)
    plans.pop().close()
    assert free() - full <= each / 2      # what came back: its few large blocks
    plans.append(make())
    assert free() >= full - 4 * MB        # the next plan took the blocks kept
    for p in plans:
        p.close()
    assert free() >= empty - KEEP - 64 * MB
