"""The 2D recurrence on the GPU vs the oracle at the sizes where its schedule can go wrong: the edges
of an 8-column block, of a 32-column window, of a 32-row warp and of a 128-row group, alone and beside
the bound kernel.  Codes, reconstructions, blob bytes and decoded fields are compared exactly."""
import numpy as np
import pytest

import cpsz_b200
from cpsz_b200 import workloads as W
from tests._util import assert_bits_equal, assert_blob_equal_2d

pytestmark = pytest.mark.gpu


def fields(kind, r1, r2):
    rng = np.random.default_rng(r1 * 1009 + r2)
    if kind == "smooth":
        return W.cfg0_like(r1 * 31 + r2, r1, r2)
    if kind == "noise":
        # neighbours that differ by far more than the bound: quantization codes up to the
        # capacity, and points beyond it
        return tuple((rng.uniform(0.5, 1.5, (r1, r2)) * 10.0 ** rng.integers(-3, 4, (r1, r2))).astype(np.float32)
                     for _ in range(2))
    # whole rows of +-0 (precision 0) between values of both signs and very unlike sizes
    out = []
    for _ in range(2):
        a = (rng.standard_normal((r1, r2)) * 2.0 ** rng.integers(-12, 13, (r1, r2))).astype(np.float32)
        a[rng.random(r1) < 0.3] = -0.0
        a[rng.random((r1, r2)) < 0.1] = 0.0
        out.append(a)
    return tuple(out)


@pytest.mark.parametrize("kind,eb", [("smooth", 0.05), ("noise", 0.05), ("noise", 2e-5), ("signs", 0.2)])
@pytest.mark.parametrize("r1,r2", [(31, 7), (32, 8), (33, 9), (2, 40), (127, 31), (128, 32), (129, 33), (161, 1),
                                   (257, 63), (300, 65), (385, 130), (513, 258)])
def test_recurrence_edges(ctx, oracle, r1, r2, kind, eb):
    U, V = fields(kind, r1, r2)
    blob = cpsz_b200.sz_compress_cp_preserve_2d_offline(U, V, max_pwr_eb=eb, ctx=ctx)
    expect = oracle.compress_2d(U, V, eb)
    assert_blob_equal_2d(blob, expect)
    du, dv = cpsz_b200.sz_decompress_cp_preserve_2d_offline(blob, r1, r2, ctx=ctx)
    ou, ov = oracle.decompress_2d(expect, r1, r2)
    assert_bits_equal(du, ou)
    assert_bits_equal(dv, ov)
    st = cpsz_b200.compress_2d_stages(U, V, eb, ctx=ctx)
    ids, eu, ev = oracle.quantize_eb_2d(U, V, oracle.eb_2d(U, V, eb))
    assert np.array_equal(st["ids"], ids)
    for data, prec, key, rkey in ((U, eu, "codes_u", "recon_u"), (V, ev, "codes_v", "recon_v")):
        codes, _, rec = oracle.lorenzo_2d(data, prec.reshape(data.shape))
        assert np.array_equal(st[key], codes)
        assert_bits_equal(st[rkey], rec)
