"""The device bytes of a context on dense data stay within hpc_ctx_footprint, its edges' lists and records,
and hpc_ctx_footprint_wide, which is nearly all used."""
import ctypes as C

import numpy as np
import pytest

import heterogpc as hg


def _footprints(p, n, precision, max_level):
    o = hg.Opts()
    hg.lib().hpc_opts_default(C.byref(o))
    o.precision, o.max_level = precision, max_level
    out = []
    for call in (lambda b: hg.lib().hpc_ctx_footprint(p, n, C.byref(o), b),
                 lambda b: hg.lib().hpc_ctx_footprint_wide(p, C.byref(o), b)):
        b = C.c_int64(-1)
        assert call(C.byref(b)) == 0
        out.append(b.value)
    return out


def test_which_contexts_may_take_more():
    def wide(p, precision, level):
        return _footprints(p, 100, precision, level)[1]

    assert wide(46340, hg.PREC_FP64, 4) == wide(9000, hg.PREC_MIXED, 0) == wide(100, hg.PREC_MIXED_TC, 4) == 0
    snapshot = 9000 * 282 * 4
    assert wide(9000, hg.PREC_MIXED_TC, 1) == snapshot
    assert wide(9000, hg.PREC_MIXED, 1) == snapshot + 144 * 2 ** 20
    for level in (2, -1):
        assert wide(9000, hg.PREC_MIXED_TC, level) > snapshot + 304 * 4 * (2 ** 20 + 33 * 9000)
    assert wide(46340, hg.PREC_MIXED_TC, 2) > 304 * 4 * 65 * 46340
    o, b = hg.Opts(), C.c_int64(0)
    hg.lib().hpc_opts_default(C.byref(o))
    assert hg.lib().hpc_ctx_footprint_wide(1, C.byref(o), C.byref(b)) == 1  # HPC_ERR_INVALID_ARG


def _pool_used():
    hg.lib()
    rt = C.CDLL("libcudart.so.13")  # the one that the library has loaded
    pool, used = C.c_void_p(), C.c_uint64(0)
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 7, C.byref(used)) == 0  # cudaMemPoolAttrUsedMemCurrent
    return used.value


@pytest.mark.gpu
@pytest.mark.parametrize("p,max_level", [(1600, 1), (1600, 2), (3001, 2)])
def test_bytes_of_a_dense_context(p, max_level):
    n = 100
    sk0 = hg.SkeletonCalculator(50, n)
    sk0.close()  # the library's stream and pool are up
    before = _pool_used()
    sk = hg.SkeletonCalculator(p, n, alpha=0.0033, max_level=max_level)
    sk.add_correlation_matrix(0.5 * np.ones((p, p)) + 0.5 * np.eye(p))
    for _ in range(2):
        sk.reset()
        sk.run()
    used = _pool_used() - before
    sk.close()
    base, wide = _footprints(p, n, hg.PREC_MIXED, max_level)
    edges = p * (p - 1) // 2
    assert used <= base + wide + edges * (8 + 4 * (6 + 2)) + 2 ** 20  # ids, records; small tables
    assert used >= 0.9 * wide
