"""Radix tiles and triangle tiles at the sizes where their rules change, against stable sorts and the oracle.

Sorts of up to 131072 keys are cut into tiles of 1024 keys, larger ones into 4096;
launches of up to 32 triangles an SM take their triangles in tiles of 8, larger
ones in tiles of 64.  Look-backs read several tiles at once, so the tile counts
here lie around multiples of four and of 32.
"""
import numpy as np
import pytest

import oracle
from tests import parity
from tests.test_zz_no_alloc import _bind, _noalloc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 4 * 1024 + 1, 33 * 1024 - 1, 131071, 131072, 131073, 5 * 4096 * 8 + 1])
@pytest.mark.parametrize("key_range", [3, 70000])
def test_sort_equals_a_stable_sort(cuda_ok, fdzb, n, key_range):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, key_range, n).astype(np.uint32)
    vals = np.arange(n, dtype=np.uint32)
    k, v, _ = _noalloc(_bind(fdzb.load()), keys, vals, key_range)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k, keys[order]) and np.array_equal(v, vals[order])


@pytest.mark.parametrize("per_sm,more", [(0, 1), (0, 9), (0, 257), (32, 0), (32, 1)])
@pytest.mark.parametrize("order", [0, 1])
def test_pairs_equal_the_oracle(cuda_ok, fdzb, scenes, per_sm, more, order):
    import torch
    T = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    s = scenes.make_scene(160, 90, T, n=8, bins=8, seed=5, sigma=0.1)
    orc = oracle.frame(s)
    ctx, t = fdzb.context_for_scene(s, masks=True, debug=True, tri_order=order)
    ctx.launch()
    out, st, ex = parity.collect(ctx, t, s, tri_order=order)
    errs = parity.compare(s, gpu=(out, st, ex), orc=orc)
    ctx.close()
    assert not errs, errs
