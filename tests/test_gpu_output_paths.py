"""Where a device blob is built and how its streams are packed: in the caller's
buffer at any alignment when it has room for the blob and 8 bytes more, else in
the workspace; the id stream beside the wavefront (fields of 2^19 points and
more) or all streams together; batches blob behind blob in the caller's
buffer.  Every path gives the oracle's bytes and leaves the bytes around them
alone."""
import numpy as np
import pytest

import cpsz_b200
from cpsz_b200 import workloads as W
from tests._util import assert_blob_equal_2d

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

GUARD = 64


def into_device(call, cap, offset):
    """call(out) into a device buffer of `cap` bytes at a byte offset, with guarded surroundings."""
    whole = torch.full((GUARD + offset + cap + GUARD,), 0xA5, dtype=torch.uint8, device="cuda")
    n = call(whole[GUARD + offset: GUARD + offset + cap])
    host = whole.cpu().numpy()
    assert (host[: GUARD + offset] == 0xA5).all() and (host[GUARD + offset + cap:] == 0xA5).all()
    return host[GUARD + offset:][:n].tobytes()


@pytest.mark.parametrize("r1,r2", [(1, 1), (37, 41), (723, 725), (724, 725)])  # 2^19 lies between the last two
def test_2d_device_output(ctx, oracle, r1, r2):
    U, V = W.cfg0_like(31, r1, r2)
    dU, dV = torch.from_numpy(U).cuda(), torch.from_numpy(V).cuda()
    want = oracle.compress_2d(U, V, 0.05)
    for cap in (len(want), len(want) + 7, len(want) + 8, 2 * len(want) + (32 << 20)):
        for offset in (0, 1, 3):
            got = into_device(lambda out: cpsz_b200.compress_2d_into(dU, dV, r1, r2, 0.05, out, ctx=ctx), cap, offset)
            assert_blob_equal_2d(got, want)
    with pytest.raises(cpsz_b200.CpszError):
        into_device(lambda out: cpsz_b200.compress_2d_into(dU, dV, r1, r2, 0.05, out, ctx=ctx), len(want) - 1, 0)


@pytest.mark.parametrize("shape", [(5, 6, 7), (40, 33, 50)])
def test_3d_device_output(ctx, oracle, shape):
    F = W.field_3d(32, *shape, 6, 8.0)
    dev = [torch.from_numpy(a).cuda() for a in F]
    want = oracle.compress_3d(*F, 0.05)
    for cap in (len(want), len(want) + 7, len(want) + 8, len(want) + (1 << 20)):
        for offset in (0, 2, 3):
            got = into_device(lambda out: cpsz_b200.compress_3d_into(*dev, *shape, 0.05, out, ctx=ctx), cap, offset)
            assert got == want
    with pytest.raises(cpsz_b200.CpszError):
        into_device(lambda out: cpsz_b200.compress_3d_into(*dev, *shape, 0.05, out, ctx=ctx), len(want) - 1, 0)


def test_batch_device_output(ctx, oracle):
    """35 fields (two passes) into exact, nearly exact and roomy buffers, and
    the same from host fields into host memory."""
    rng = np.random.default_rng(33)
    shapes = [(int(a), int(b)) for a, b in zip(rng.integers(1, 300, 35), rng.integers(1, 300, 35))]
    shapes[3], shapes[20] = (1, 1), (700, 801)
    fields = [W.cfg0_like(100 + k, *s) for k, s in enumerate(shapes)]
    ebs = rng.choice([0.01, 0.05, 0.1], 35)
    dev = [(torch.from_numpy(U).cuda(), torch.from_numpy(V).cuda()) for U, V in fields]
    want = [oracle.compress_2d(U, V, e) for (U, V), e in zip(fields, ebs)]
    total = sum(map(len, want))
    for cap in (total, total + 8, total + (1 << 20)):
        for offset in (0, 3):
            offs = []

            def call(out):
                offs[:] = [int(x) for x in cpsz_b200.compress_2d_batch(dev, ebs, out=out, ctx=ctx)]
                return offs[-1]

            got = into_device(call, cap, offset)
            assert offs[-1] == total
            for k in range(35):
                assert_blob_equal_2d(got[offs[k]:offs[k + 1]], want[k])
    for g, w in zip(cpsz_b200.compress_2d_batch(fields, ebs, ctx=ctx), want):
        assert_blob_equal_2d(g, w)


def test_codes_of_every_kind(ctx, oracle):
    """Code histograms with very many and very few occurring symbols."""
    rng = np.random.default_rng(34)
    for U, V in ((rng.standard_normal((300, 301)), rng.standard_normal((300, 301)) * 100),
                 (np.ones((90, 70)), np.full((90, 70), 2.0)),
                 (np.cumsum(rng.standard_normal((400, 500)), 1), np.cumsum(rng.standard_normal((400, 500)), 0))):
        U, V = U.astype(np.float32), V.astype(np.float32)
        for eb in (1e-4, 0.1):
            assert_blob_equal_2d(cpsz_b200.sz_compress_cp_preserve_2d_offline(U, V, max_pwr_eb=eb, ctx=ctx),
                                 oracle.compress_2d(U, V, eb))
