"""The GPU lossless stage writes standard Zstandard frames: the system libzstd
(the decoder behind the reference's sz_lossless_decompress) reads every frame
back to the input bytes, from host and device buffers, for empty, one-byte,
constant (RLE), incompressible and real compressor blobs."""
import os
import shutil
import struct
import subprocess

import numpy as np
import pytest

import cpsz_b200
from cpsz_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _roundtrip(data: bytes, ctx):
    frame = cpsz_b200.lossless_compress_gpu(data, ctx=ctx)
    assert cpsz_b200.sz_lossless_decompress(frame, len(data)) == data
    return frame


def test_small_and_degenerate_inputs(ctx):
    rng = np.random.default_rng(0)
    for data in (b"", b"\x07", bytes(100000), bytes(32768 * 3), rng.integers(0, 256, 200001, np.uint8).tobytes(),
                 (b"abcd" * 50000)[:199999]):
        frame = _roundtrip(data, ctx)
        assert len(frame) <= cpsz_b200.lib().cpsz_b200_lossless_bound(len(data))


def test_compressor_blobs_shrink(ctx, reference):
    U, V = W.cfg0_like(21, 1500, 1700)
    for eb in (0.1, 0.01):
        blob = cpsz_b200.sz_compress_cp_preserve_2d_offline(U, V, max_pwr_eb=eb, ctx=ctx)
        frame = _roundtrip(blob, ctx)
        assert len(frame) < 0.9 * len(blob)
        # the reference's own lossless decoder reads it
        assert reference.zstd_decompress(frame, len(blob)) == blob


def test_device_buffers(ctx):
    torch = pytest.importorskip("torch")
    U, V = W.cfg0_like(22, 900, 800)
    blob = cpsz_b200.sz_compress_cp_preserve_2d_offline(U, V, max_pwr_eb=0.1, ctx=ctx)
    d_in = torch.from_numpy(np.frombuffer(blob, np.uint8).copy()).cuda()
    d_out = torch.zeros(cpsz_b200.lib().cpsz_b200_lossless_bound(len(blob)), dtype=torch.uint8, device="cuda")
    n = cpsz_b200.lossless_compress_gpu(d_in, out=d_out, ctx=ctx)
    frame = d_out[:n].cpu().numpy().tobytes()
    assert frame == cpsz_b200.lossless_compress_gpu(blob, ctx=ctx)
    assert cpsz_b200.sz_lossless_decompress(frame, len(blob)) == blob
    small = torch.zeros(16, dtype=torch.uint8, device="cuda")
    with pytest.raises(cpsz_b200.CpszError):
        cpsz_b200.lossless_compress_gpu(d_in, out=small, ctx=ctx)


@pytest.mark.parametrize("n", [1, 2, 7, 8191, 8192, 8193, 8192 * 8 - 1, 8192 * 8 + 5, 8192 * 9])
@pytest.mark.parametrize("kind", ["text", "sparse", "long", "mixed"])
def test_block_edges(ctx, n, kind):
    """Blocks of every sequence count and literal header: a few matches and
    many (batches of 32 sequences, one- and two-byte counts), literal runs over
    31 and 4095 bytes, matches that reach a block's end."""
    rng = np.random.default_rng(n)
    if kind == "text":  # short matches everywhere
        a = rng.integers(0, 4, n).astype(np.uint8)
    elif kind == "sparse":  # mostly literals, a repeated run now and then
        a = rng.integers(0, 256, n).astype(np.uint8)
        for at in range(0, n - 600, 1500):
            a[at + 300:at + 500] = a[at:at + 200]
    elif kind == "long":  # matches of thousands of bytes
        a = np.resize(rng.integers(0, 256, 97), n).astype(np.uint8)
    else:
        a = rng.integers(0, 256, n).astype(np.uint8)
        a[: n // 2] = rng.integers(0, 3, n // 2)
        a[-20:] = 5
    frame = _roundtrip(a.tobytes(), ctx)
    assert len(frame) <= cpsz_b200.lib().cpsz_b200_lossless_bound(n)


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_frames_equal_the_format_header_s_coder(ctx, tmp_path):
    """Every frame byte for byte: tests/zstd_frame_check.cpp reads the blocks'
    sequences back and writes them again with the host coder of
    cpsz_b200/csrc/zstd_format.h."""
    rng = np.random.default_rng(9)
    U, V = W.cfg0_like(24, 700, 900)
    inputs = [b"", b"\x07", bytes(20000), rng.integers(0, 256, 30001, np.uint8).tobytes(),
              cpsz_b200.sz_compress_cp_preserve_2d_offline(U, V, max_pwr_eb=0.1, ctx=ctx),
              cpsz_b200.sz_compress_cp_preserve_2d_offline(U, V, max_pwr_eb=0.01, ctx=ctx)]
    for n in (5, 33, 100, 8191, 8192, 8193, 70001):
        for alphabet, run in ((2, 1), (4, 1), (256, 3), (16, 40), (256, 4096)):
            a = np.repeat(rng.integers(0, alphabet, n // run + 1), run)[:n].astype(np.uint8)
            if n > 600:  # a distant repeat, so that every offset code occurs
                a[-300:] = a[:300]
            inputs.append(a.tobytes())
    path = tmp_path / "frames"
    with open(path, "wb") as f:
        for data in inputs:
            frame = _roundtrip(data, ctx)
            f.write(struct.pack("<QQ", len(data), len(frame)) + data + frame)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    exe = str(tmp_path / "zframe")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(root, "cpsz_b200", "csrc"), "-o", exe,
                    os.path.join(root, "tests", "zstd_frame_check.cpp")], check=True)
    r = subprocess.run([exe, str(path)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "ALL OK" in r.stdout, r.stdout + r.stderr
    assert int(r.stdout.split(" compressed")[0].split()[-1]) > 100
