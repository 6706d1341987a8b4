"""The one-pass expansion level (k_ks_expand) and the sliced absorb against the
oracle where they can go wrong: the last level that fits a tile of 1024
positions, the first that does not, one tile per polynomial and several, item
counts around the slices, and more items than one REDC takes."""
import ctypes

import numpy as np
import pytest

from conftest import Q59, Q60

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,q,levels,log_b,items,count", [
    (10, Q60, 10, 15, 1000, 2), (11, Q59, 11, 30, 2048, 1), (11, Q60, 4, 8, 9, 3),
    (12, Q59, 5, 20, 7, 2), (12, Q60, 3, 59, 1, 5)])
def test_expand_and_absorb(sg, oracle, log_n, q, levels, log_b, items, count):
    lib, n = sg.lib(), 1 << log_n
    p, ctx = oracle.Prime(q, log_n), sg.Context(log_n, [q])
    dim = p.gadget_size(log_b)
    mats = [[oracle.uniform_limbs(70 + 2 * j + c, [q], n, dim) for c in (0, 1)]
            for j in range(levels)]
    keys = [sg.Key(ctx, [log_b], (n >> j) + 1, *mats[j]) for j in range(levels)]
    arr = (ctypes.c_void_p * levels)(*[k.h for k in keys])
    cts = oracle.uniform_limbs(5, [q], n, 2 * count).reshape(count, 2, n)
    db = oracle.uniform_limbs(6, [q], n, items).reshape(items, n)
    full = [p.oblivious_expand(levels, log_b, np.stack(mats).reshape(levels, 2, dim, n), cts[i])
            for i in range(count)]
    d, ddb = sg.DeviceBuffer.from_array(cts), sg.DeviceBuffer.from_array(db)
    out, big = sg.DeviceBuffer(cts.nbytes), sg.DeviceBuffer(cts.nbytes << levels)
    sg.check(lib.shg_oblivious_expand(ctx.h, arr, levels, big.ptr, d.ptr, count, None))
    assert np.array_equal(big.download((count, 1 << levels, 2, n)), np.stack(full))
    sg.check(lib.shg_pir_expand_absorb(ctx.h, arr, levels, ddb.ptr, items, out.ptr, d.ptr, count,
                                       None))
    want = np.stack([p.absorb_sum(f[:items], db) for f in full])
    assert np.array_equal(out.download((count, 2, n)), want)
