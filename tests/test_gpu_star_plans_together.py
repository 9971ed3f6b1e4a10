"""Star plans of different shared-memory sizes alive at the same time: made and
run in every order, direct and through a graph, against the oracle."""
import numpy as np
import pytest
import torch

from proteus_gb300 import star

pytestmark = pytest.mark.gpu


def make(ctx, rows, rng):
    cols = [np.ascontiguousarray(rng.integers(0, s, rows).astype(np.int8)) for s in (25, 5)]
    dim = star.Dim("d", rows, cols, ["a", "b"], [0, 0], [24, 4])
    n = 20_001
    data = star.StarData([dim], [rng.integers(1, rows + 1, n).astype(np.int32)],
                         rng.integers(1, 51, n).astype(np.int32), rng.integers(1, 1000, n).astype(np.int32))
    return data, star.StarPlan(ctx, data)


# rows: staged masks (300, 4000), codes (5000, 60,000), masks in L2 only (70,000)
@pytest.mark.parametrize("sizes", [(60_000, 300), (4000, 300), (300, 60_000), (60_000, 5000, 70_000), (70_000, 60_000)])
@pytest.mark.parametrize("use_graph", [False, True])
def test_plans_together(ctx, oracle, sizes, use_graph):
    rng = np.random.default_rng(sum(sizes))
    plans = [make(ctx, rows, rng) for rows in sizes]
    q = star.Query(join_mask=1)
    q.pred_attr[0], q.pred_lo[0], q.pred_hi[0] = 0, 3, 20
    q.group_dim, q.group_attr = [0, 0], [0, 1]
    for order in (range(len(plans)), reversed(range(len(plans)))):
        for i in order:
            data, plan = plans[i]
            got = star.StarPlan.results(plan.run([q], use_graph=use_graph), 1)[0]
            ctx.sync()
            exp = oracle.star_query(data, q)
            assert len(got[0]) == len(exp[0]) and all((x == y).all() for x, y in zip(got, exp))
    torch.cuda.synchronize()
    for _, plan in plans:
        plan.close()
