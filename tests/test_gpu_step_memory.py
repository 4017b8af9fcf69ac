"""The time-step selection's device memory follows the level budget, not the
contacts: the CCD's records only feed each pair's new step, and are consumed in
parts of about half the budget, a body pair's too."""
import numpy as np
import pytest

import delta2_gb300 as D
from tests.clusters import separate

pytestmark = pytest.mark.gpu


def test_select_steps_memory_is_bounded_by_the_level_budget(gpu_required):
    import torch

    from delta2_gb300 import build as B
    B.build()
    s = D.make_scene(5, nx=3, ny=2, nz=3, spacing=1.15, speed_sigma=3.0, seed=8)
    s.last_dt[:] = 0.05
    pairs = D.broad_phase(s)
    clusters = separate(pairs, s.is_static, s.n_bodies)
    flat = np.array([p for _, inter in clusters for p in inter], dtype=np.int32).reshape(-1, 2)
    grouped = [(parts, len(inter)) for parts, inter in clusters]

    def select(budget):
        ctx = D.Context(0)
        try:
            ctx.set_level_budget(budget)
            ctx.set_scene(s.copy())
            ctx.sync()
            before = torch.cuda.mem_get_info()[0]
            steps, counters = ctx.select_time_steps(flat, grouped, s.opt_dt)
            ctx.sync()
            return steps, counters, before - torch.cuda.mem_get_info()[0]
        finally:
            ctx.close()

    ctx = D.Context(0)
    try:
        ctx.set_scene(s.copy())
        n_records = len(ctx.compare_trees_full_continuous(flat, np.full(len(flat), 0.05), capacity=1 << 23)[0])
    finally:
        ctx.close()
    budget = 16 << 20
    whole, whole_counters, whole_bytes = select(0)
    steps, counters, used = select(budget)
    print(f"{n_records} records ({112 * n_records >> 20} MB); device bytes of the call: {whole_bytes >> 20} MB, "
          f"with a budget of {budget >> 20} MB {used >> 20} MB")
    assert np.array_equal(steps.view(np.uint64), whole.view(np.uint64))
    assert np.any(steps < s.opt_dt)  # contacts cut some step
    assert counters[:3].tolist() == whole_counters[:3].tolist()
    # the records and their sorted copy alone would take more than what the call
    # may use: a few budgets' worth of level, range and record buffers
    assert 2 * 112 * n_records > 8 * budget
    assert used < 8 * budget
