"""perf/cases.py without a GPU: every drawn case can be made and costed."""
import importlib.util
import os
import random

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _cases():
    spec = importlib.util.spec_from_file_location("cases", os.path.join(ROOT, "perf", "cases.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def test_draws_of_every_seed():
    """A batch whose angles were drawn for a smaller grid (fewer than 90) too
    (seed 48 among others)."""
    cases = _cases()
    most = max(cases._cost(c) for c in cases.listed())
    for seed in range(2000):
        c = cases.draw(random.Random(seed))
        w = cases.work(c)
        assert w["bytes"] > 0 and w["flops"] > 0 and cases._cost(c) <= most, (seed, c)
        for q in cases._problems(c) if c["kind"] == "batch" else [c]:
            assert 45 <= q["P"] <= 1500 and q["C"] >= 64 and q["S"] >= 1, (seed, q)
