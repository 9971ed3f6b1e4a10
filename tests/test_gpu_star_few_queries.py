"""Star batches without filters, of one to 64 queries: the additions of a batch
of few queries go to copies of its groups.  Against the oracle, and what few
groups cost against many."""
import numpy as np
import pytest
import torch

from proteus_gb300 import star

pytestmark = pytest.mark.gpu


def query(gd, ga):
    return star.Query(join_mask=15, group_dim=list(gd), group_attr=list(ga))


@pytest.mark.parametrize("nq", [1, 2, 3, 4, 5, 16, 21, 22, 32, 33, 63, 64])
@pytest.mark.parametrize("use_graph", [False, True])
def test_unfiltered(ctx, oracle, nq, use_graph):
    data = star.gen_star(2, n_fact=700_003, dim_rows=(9000, 2557, 700, 5000))
    plan = star.StarPlan(ctx, data)
    kinds = [query((0, 1), (1, 1)), query((0, 2), (0, 0)), query((3, 1), (0, 0)), query((2, 2), (1, 0))]
    exp = [oracle.star_query(data, q) for q in kinds]
    batch = [kinds[q % 4] for q in range(nq)]
    for _ in range(2):
        out = plan.run(batch, use_graph=use_graph)
        ctx.sync()
        for q, got in enumerate(star.StarPlan.results(out, nq)):
            assert all(len(x) == len(y) and (x == y).all() for x, y in zip(got, exp[q % 4]))
    plan.close()


def test_few_groups(ctx):
    """35 groups against 625: 4.5 times the time when all CTAs added to the same ones, 1.7 times with copies."""
    data = star.gen_star(3, n_fact=1 << 22, dim_rows=(1 << 17, 2557, 9000, 5000))
    plan = star.StarPlan(ctx, data)
    out = plan.new_output(1)

    def best(q):
        t = float("inf")
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            plan.run([q], out=out)
            b.record()
            torch.cuda.synchronize()
            t = min(t, a.elapsed_time(b))
        return t

    assert best(query((0, 1), (1, 1))) < 3 * best(query((0, 2), (0, 0)))
    plan.close()
