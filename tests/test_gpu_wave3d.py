"""The 3D recursion on the GPU vs the oracle at the edges of its units (8 planes, 32 rows) and of its
8-step windows (short rows, rows whose first and last inner window lie next to each other), with raw
points scattered through the field."""
import numpy as np
import pytest

import cpsz_b200
from tests._util import assert_bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 31, 2), (2, 32, 7), (7, 33, 8), (8, 32, 9), (9, 31, 45), (8, 33, 46), (8, 32, 47),
                                   (16, 32, 53), (17, 65, 40), (3, 97, 23), (24, 64, 61), (25, 33, 130)])
@pytest.mark.parametrize("raw", [False, True])
def test_recursion_edges(ctx, oracle, shape, raw):
    rng = np.random.default_rng(int(np.prod(shape)) + raw)
    x = np.linspace(0, 3, shape[2], dtype=np.float32) + np.arange(shape[1], dtype=np.float32)[:, None] / 7
    fields = [(np.sin(x * f + 0.3 * np.arange(shape[0])[:, None, None]) + 1.5).astype(np.float32) for f in (1.0, 1.7, 2.3)]
    if raw:
        for a in fields:
            a *= np.where(rng.random(shape) < 0.05, 2.0 ** rng.integers(-30, 30, shape), 1.0).astype(np.float32)
            a[rng.random(shape) < 0.03] = 0.0
    blob = cpsz_b200.sz_compress_cp_preserve_3d_offline_log(*fields, max_pwr_eb=0.05, ctx=ctx)
    expect = oracle.compress_3d(*fields, 0.05)
    assert blob == expect
    got = cpsz_b200.sz_decompress_cp_preserve_3d_online_log(blob, *shape, ctx=ctx)
    for a, b in zip(got, oracle.decompress_3d(expect, *shape)):
        assert_bits_equal(a, b)


@pytest.mark.parametrize("shape", [(2, 33, 1), (2, 64, 2), (9, 97, 1), (16, 160, 3), (2, 1000, 1)])
def test_first_column_above_a_unit(ctx, oracle, shape):
    """A unit's second plane predicts its first column from the row above the
    unit in its first step, before the compute warps' first barrier: thin
    fields of many units, many times over, always the oracle's bytes."""
    rng = np.random.default_rng(shape[1])
    fields = [(rng.standard_normal(shape) * 0.1 + 2.0 ** c).astype(np.float32) for c in (0, 3, -4)]
    expect = oracle.compress_3d(*fields, 0.1)
    out = oracle.decompress_3d(expect, *shape)
    for _ in range(20):
        blob = cpsz_b200.sz_compress_cp_preserve_3d_offline_log(*fields, max_pwr_eb=0.1, ctx=ctx)
        assert blob == expect
        for a, b in zip(cpsz_b200.sz_decompress_cp_preserve_3d_online_log(blob, *shape, ctx=ctx), out):
            assert_bits_equal(a, b)
