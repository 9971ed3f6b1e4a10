"""Partitioning on 9 bits and more into the input's own columns, crossed columns
and columns that overlap it in part, against the oracle's clusters."""
import numpy as np
import pytest
import torch

from gpu_util import host
from proteus_gb300 import abi
from proteus_gb300.engine import _cur_stream

pytestmark = pytest.mark.gpu


# where keys, payload, output keys and output payload start, in columns of n
@pytest.mark.parametrize("at", [(0, 1, 0, 1), (0, 1, 1, 0), (0, 1, 0, 2), (0, 1, 2, 0), (0, 1, 2, 1), (0, 1, 0.5, 2)])
@pytest.mark.parametrize("n,bits", [(1000, 9), (400_000, 11), (3_000_001, 12), (400_000, 13)])
def test_in_place(ctx, oracle, n, bits, at):
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(-(1 << 31), 1 << 31, n).astype(np.int32)
    pay = rng.integers(-(1 << 31), 1 << 31, n).astype(np.int32)
    if at == (0, 1, 0.5, 2):  # the output starts inside the keys and ends inside the payload's place: no payload
        pay = None
    room = torch.zeros(4 * n + 8, dtype=torch.int32, device="cuda")
    cols = [room[int(a * n):int(a * n) + n] for a in at]
    cols[0].copy_(torch.from_numpy(keys))
    if pay is not None:
        cols[1].copy_(torch.from_numpy(pay))
    off = torch.empty((1 << bits) + 1, dtype=torch.int64, device="cuda")
    ctx.check(ctx.lib.gbj_partition(ctx.handle, cols[0].data_ptr(), cols[1].data_ptr() if pay is not None else None, n,
                                    abi.DIGIT_HASH, 0, bits, cols[2].data_ptr(), cols[3].data_ptr(), off.data_ptr(),
                                    _cur_stream()))
    ctx.sync()
    ek, ep, eoff = oracle.radix_cluster(keys, pay, 0, bits, True)
    assert (host(off).astype(np.uint64) == eoff).all()
    part = np.repeat(np.arange(1 << bits), np.diff(eoff.astype(np.int64)))
    out = []
    for k, p in ((host(cols[2]), host(cols[3])), (ek, ep)):  # tuples keep no order inside a partition
        order = np.lexsort((p, k, part))
        out.append((k[order], p[order]))
    assert (out[0][0] == out[1][0]).all() and (out[0][1] == out[1][1]).all()
