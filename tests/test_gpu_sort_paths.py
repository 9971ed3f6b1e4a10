"""ORDER BY at the sizes where the sort changes its path or its last tile is
ragged, with keys that share digits (skipped passes), all equal keys, one to
four columns and the key at either end: the order of a stable host sort."""
import numpy as np
import pytest

from gpu_util import dev, host

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 1023, 1024, 1025, 4097, 8191, 8192, 8193, 8192 + 2048, 100_001, (1 << 20) - 1, 1 << 20,
         (1 << 20) + 6145]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("keys", ["any", "equal", "low", "high", "ends"])
def test_paths(ctx, n, keys):
    rng = np.random.default_rng(n)
    i32 = np.iinfo(np.int32)
    key = {
        "any": lambda: rng.integers(i32.min, i32.max, n, dtype=np.int64, endpoint=True),
        "equal": lambda: np.full(n, -7),
        "low": lambda: rng.integers(0, 200, n),  # three digits are the same for all
        "high": lambda: rng.integers(-100, 100, n) << 24,
        "ends": lambda: rng.choice([i32.min, i32.max, 0, -1], n),
    }[keys]().astype(np.int32)
    n_cols = 1 + n % 4
    cols = [rng.integers(-1000, 1000, n).astype(np.int32) for _ in range(n_cols)]
    at = n % n_cols
    cols[at] = key
    for desc in (False, True):
        out = ctx.sort_by_key([dev(c) for c in cols], at, descending=desc)
        ctx.sync()
        order = np.argsort(-key.astype(np.int64) if desc else key, kind="stable")
        for o, c in zip(out, cols):
            assert (host(o) == c[order]).all()
