"""Raster codes to 12x12 block order and back on the GPU vs the oracle at the edges of its strips (384
columns, 12 rows) and at every alignment of a row, with many unpredictable points and with none."""
import numpy as np
import pytest

import cpsz_b200
from cpsz_b200 import workloads as W
from tests._util import assert_bits_equal, assert_blob_equal_2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("noisy", [False, True])
@pytest.mark.parametrize("r1", [11, 12, 25])
@pytest.mark.parametrize("r2", [383, 384, 385, 386, 388, 391, 395, 396, 397, 768, 773, 780, 1154])
def test_strip_edges(ctx, oracle, r1, r2, noisy):
    if noisy:
        rng = np.random.default_rng(r1 * 2003 + r2)
        U, V = (rng.uniform(0.5, 1.5, (r1, r2)) * 10.0 ** rng.integers(-3, 4, (r1, r2)) for _ in range(2))
        U, V = U.astype(np.float32), V.astype(np.float32)
        eb = 1e-4
    else:
        U, V = W.cfg0_like(r1 * 17 + r2, r1, r2)
        eb = 0.1
    blob = cpsz_b200.sz_compress_cp_preserve_2d_offline(U, V, max_pwr_eb=eb, ctx=ctx)
    expect = oracle.compress_2d(U, V, eb)
    assert_blob_equal_2d(blob, expect)
    du, dv = cpsz_b200.sz_decompress_cp_preserve_2d_offline(blob, r1, r2, ctx=ctx)
    ou, ov = oracle.decompress_2d(expect, r1, r2)
    assert_bits_equal(du, ou)
    assert_bits_equal(dv, ov)
