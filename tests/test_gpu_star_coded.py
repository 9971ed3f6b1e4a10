"""Star batches over a dimension coded by its attribute classes: classes at the
limit, rows outside the declared domains, two candidates, ragged and unaligned
fact columns, batches in which every row matches and batches in which few do,
against the oracle."""
import numpy as np
import pytest
import torch

from proteus_gb300 import star

pytestmark = pytest.mark.gpu


def dim(name, n, spans, rng, stray=0):
    cols, lo, hi = [], [], []
    for a, span in enumerate(spans):
        c = rng.integers(0, span, n).astype(np.int8 if span < 100 else np.int32) + (3 if a else 0)
        cols.append(np.ascontiguousarray(c))
        lo.append(3 if a else 0)
        hi.append(span - 1 + (3 if a else 0))
    if stray:  # values of the last attribute outside what is declared: it is no group key here
        cols[-1] = cols[-1].astype(np.int32)
        cols[-1][::stray] += 1000
    return star.Dim(name, n, cols, ["a%d" % a for a in range(len(spans))], lo, hi)


def query(dims, join, preds, group):
    q = star.Query(join_mask=sum(1 << d for d in join))
    for d, (a, lo, hi) in preds.items():
        q.pred_attr[d], q.pred_lo[d], q.pred_hi[d] = a, lo, hi
    for k, (d, a) in enumerate(group):
        q.group_dim[k], q.group_attr[k] = d, a
    return q


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("n_fact,shift,stray", [(1, 0, 0), (4099, 1, 0), (200_003, 0, 7), (700_001, 3, 1)])
@pytest.mark.parametrize("spans,rows", [((25, 5), 65536), ((5, 3, 17), 5000), ((16, 16), 9000)])
def test_coded(ctx, oracle, n_fact, shift, stray, spans, rows, use_graph):
    rng = np.random.default_rng(n_fact + rows)
    dims = [dim("big", 70_000, (20, 7), rng), dim("coded", rows, spans, rng, stray), dim("small", 300, (9, 4), rng),
            dim("other", 6000, (12, 2), rng)]
    fk = [rng.integers(0, d.n + d.n // 8 + 2, n_fact + shift).astype(np.int32) for d in dims]  # some keys match nothing
    qty = rng.integers(1, 51, n_fact + shift).astype(np.int32)
    price = rng.integers(-(1 << 31), 1 << 31, n_fact + shift).astype(np.int32)
    data = star.StarData(dims, [c[shift:] for c in fk], qty[shift:], price[shift:])
    up = lambda c: torch.from_numpy(c).cuda()[shift:]  # noqa: E731
    plan = star.StarPlan(ctx, data, fact_tensors=([up(c) for c in fk], up(qty), up(price)))
    last = len(spans) - 1
    queries = [
        query(dims, (0, 1, 2, 3), {}, ((0, 0), (2, 0))),  # every row with all keys present
        query(dims, (1,), {1: (0, 0, 2)}, ((1, 0), (1, 0))),
        query(dims, (1, 3), {1: (last, 4, 2000), 3: (0, 1, 3)}, ((3, 0), (3, 1))),
        query(dims, (0, 1), {0: (0, 4, 4), 1: (last, 1003, 1004)}, ((0, 1), (0, 0))),
        query(dims, (2,), {}, ((2, 0), (2, 1))),
    ]
    for _ in range(2):
        for nq in (len(queries), 1, 64):
            batch = (queries * 13)[:nq]
            out = plan.run(batch, use_graph=use_graph)
            ctx.sync()
            for q, got in zip(batch[:len(queries)], star.StarPlan.results(out, nq)):
                exp = oracle.star_query(data, q)
                assert len(got[0]) == len(exp[0]) and all((x == y).all() for x, y in zip(got, exp))
    plan.close()


def test_without_room_for_the_codes(ctx, oracle):
    """A plan that the pool has room for without the codes is made without them."""
    rng = np.random.default_rng(8)
    dims = [dim("big", 70_000, (20, 7), rng), dim("coded", 65_536, (25, 5), rng)]
    fk = [rng.integers(0, d.n, 50_001).astype(np.int32) for d in dims]
    qty, price = rng.integers(1, 51, 50_001).astype(np.int32), rng.integers(-1000, 1000, 50_001).astype(np.int32)
    data = star.StarData(dims, fk, qty, price)
    cols = ([torch.from_numpy(c).cuda() for c in fk], torch.from_numpy(qty).cuda(), torch.from_numpy(price).cuda())
    ctx.sync()
    before = ctx.pool_stats()["in_use"]
    plan = star.StarPlan(ctx, data, fact_tensors=cols)
    ctx.sync()
    need = ctx.pool_stats()["in_use"] - before
    plan.close()
    ctx.sync()
    ctx.set_pool_limit(ctx.pool_stats()["in_use"] + need - 40_000)
    try:
        plan = star.StarPlan(ctx, data, fact_tensors=cols)
        assert ctx.pool_stats()["in_use"] - before <= need - 40_000
    finally:
        ctx.set_pool_limit(0)
    q = query(dims, (0, 1), {1: (0, 0, 12)}, ((1, 0), (0, 1)))
    got = star.StarPlan.results(plan.run([q]), 1)[0]
    exp = oracle.star_query(data, q)
    assert len(got[0]) == len(exp[0]) and all((x == y).all() for x, y in zip(got, exp))
    plan.close()
