"""The GPU Huffman decoder against the oracle, on 2D blobs with made-up streams.

Any code and id sequence is a valid blob, so the streams aim at the decoder's
own edges: codes longer than one and both look-up tables, trees of every index
width, streams that end at, before and after a subsequence's or a tile's end,
and fixed-length codes that never synchronise (the settling rounds)."""
import os
import re
import struct

import numpy as np
import pytest

import cpsz_b200
from tests._util import assert_bits_equal

pytestmark = pytest.mark.gpu

SUB_BITS, SCAN_TILE, WRITE_TILE = 512, 240, 256  # the decoder's subsequence and its tiles


def blob_2d(oracle, ids, codes, r1, r2, rng):
    """A 2D offline blob of the given streams (unpredictable values made up)."""
    nblocks = ((r1 - 1) // 12 + 1) * ((r2 - 1) // 12 + 1)
    sec = oracle.huffman_encode(2048, ids.astype(np.int32))
    fields = []
    for c in codes:
        un = rng.standard_normal(int((c == 0).sum())).astype(np.float32)
        fields.append(struct.pack("<iBi8xQQ", 12, 0, 32768, 0, un.size) + un.tobytes() +
                      bytes((nblocks - 1) // 8 + 1) + oracle.huffman_encode(131072, c.astype(np.int32)))
    head = struct.pack("<idQQQ", 4, 2.0 ** -52, len(sec), *map(len, fields))
    return head + sec + fields[0] + fields[1]


def fibonacci(rng, n, symbols):
    """n symbols with Fibonacci-like shares: code lengths 1, 2, 3, ... symbols."""
    f = [1, 1]
    while len(f) < symbols:
        f.append(f[-1] + f[-2])
    s = np.repeat(32768 + np.arange(symbols), np.array(f[::-1]))
    s = np.concatenate([s, np.full(n - s.size, 32768)])
    rng.shuffle(s)
    return s


def streams(kind, n, rng):
    if kind == "fixed3":       # eight equal shares: 3-bit codes never synchronise
        return 32764 + rng.permutation(np.arange(n) % 8)
    if kind == "fixed16":      # every symbol: 16-bit codes and 32-bit tree indices
        return rng.permutation(np.arange(n) % 65535 + 1)
    if kind == "two":          # one bit each
        return 32768 + (rng.random(n) < 0.5)
    if kind == "one":
        return np.full(n, 32768)
    if kind == "deep":         # codes over 20 bits: beyond both tables
        return fibonacci(rng, n, 29)
    if kind == "wide":         # many distinct symbols, most codes over 12 bits, and unpredictable points
        c = (32768 + np.round(rng.standard_normal(n) * 3000)).clip(1, 65535)
        return np.where(rng.random(n) < 0.01, 0, c)
    return (32768 + np.round(rng.standard_cauchy(n) * 2)).clip(0, 65535)


def ids_of(kind, n, rng):
    if kind == "one":
        return np.full(n, 21)
    if kind == "fixed3":
        return 20 + rng.permutation(np.arange(n) % 8)
    return np.where(rng.random(n) < 0.6, 22, rng.integers(0, 30, n))


@pytest.mark.parametrize("kind,r1,r2", [
    ("cauchy", 1, 1), ("one", 1, 1), ("cauchy", 1, 7), ("cauchy", 13, 1), ("two", 25, 13), ("one", 40, 60),
    # one-bit codes: exactly one subsequence, one symbol more, one scan / write tile, and around them
    ("two", 1, SUB_BITS), ("two", 1, SUB_BITS + 1), ("two", SCAN_TILE, SUB_BITS), ("two", WRITE_TILE, SUB_BITS),
    ("two", WRITE_TILE, SUB_BITS + 1), ("two", 2 * SCAN_TILE + 1, SUB_BITS - 1),
    ("fixed3", 300, 501), ("fixed16", 300, 500), ("deep", 1100, 1300), ("wide", 401, 999), ("cauchy", 800, 1201),
])
def test_gpu_decoder_matches_oracle(ctx, oracle, kind, r1, r2):
    rng = np.random.default_rng(r1 * 4099 + r2)
    n = r1 * r2
    codes = [streams(kind, n, rng), streams(kind, n, rng)]
    blob = blob_2d(oracle, ids_of(kind, 2 * n, rng), codes, r1, r2, rng)
    du, dv = cpsz_b200.sz_decompress_cp_preserve_2d_offline(blob, r1, r2, ctx=ctx)
    ou, ov = oracle.decompress_2d(blob, r1, r2)
    assert_bits_equal(du, ou)
    assert_bits_equal(dv, ov)


def test_gpu_decoder_streams_sent_one_by_one(ctx, oracle):
    """A blob above 4 MiB goes up and is decoded stream by stream, here with a
    code stream that needs the settling rounds."""
    rng = np.random.default_rng(5)
    r1, r2 = 1000, 3001
    codes = [streams("wide", r1 * r2, rng), streams("fixed3", r1 * r2, rng)]
    blob = blob_2d(oracle, ids_of("cauchy", 2 * r1 * r2, rng), codes, r1, r2, rng)
    assert len(blob) > 4 << 20
    du, dv = cpsz_b200.sz_decompress_cp_preserve_2d_offline(blob, r1, r2, ctx=ctx)
    ou, ov = oracle.decompress_2d(blob, r1, r2)
    assert_bits_equal(du, ou)
    assert_bits_equal(dv, ov)


def test_gpu_decoder_refuses_short_streams(ctx, oracle):
    """Streams that hold fewer symbols than the field has points, and a tree
    that is not one."""
    rng = np.random.default_rng(6)
    r1, r2 = 60, 70
    codes = [streams("wide", r1 * r2, rng), streams("wide", r1 * r2, rng)]
    ids = ids_of("cauchy", 2 * r1 * r2, rng)
    short = [codes[0], codes[1][: r1 * r2 // 2]]
    with pytest.raises(cpsz_b200.CpszError):
        cpsz_b200.sz_decompress_cp_preserve_2d_offline(blob_2d(oracle, ids, short, r1, r2, rng), r1, r2, ctx=ctx)
    blob = bytearray(blob_2d(oracle, ids, codes, r1, r2, rng))
    blob[36 + 13] = 0  # the id tree's root is its own left child
    with pytest.raises(cpsz_b200.CpszError):
        cpsz_b200.sz_decompress_cp_preserve_2d_offline(bytes(blob), r1, r2, ctx=ctx)


def shared_node_section(oracle, states, sym, rng, chain=12):
    """The Huffman section of `sym` with `chain` nodes put before its tree,
    each the next one's parent twice over, and a made-up `chain`-bit prefix
    before every code: a node array that is no tree, of which every
    `chain`-bit pattern leads to one inner node."""
    sec = oracle.huffman_encode(states, sym.astype(np.int32))
    nc, size = struct.unpack_from("<QI", sec)
    wdt = lambda k: np.uint8 if k <= 256 else np.uint16 if k <= 65536 else np.uint32  # noqa: E731
    w, at = np.dtype(wdt(nc)).itemsize, 13
    left, right = (np.frombuffer(sec, wdt(nc), nc, at + k * w * nc).astype(np.int64) for k in (0, 1))
    symbols = np.frombuffer(sec, "<u4", nc, at + 2 * w * nc)
    leaf = np.frombuffer(sec, np.uint8, nc, at + (2 * w + 4) * nc)
    code, length = {}, {}
    todo = [(0, 0, 0)]
    while todo:
        node, c, n = todo.pop()
        if leaf[node]:
            code[int(symbols[node])], length[int(symbols[node])] = c, n
        else:
            todo += [(left[node], 2 * c, n + 1), (right[node], 2 * c + 1, n + 1)]
    step = np.arange(1, chain + 1)
    shift = lambda a: np.concatenate([step, np.where(leaf != 0, 0, a + chain)]).astype(wdt(nc + chain))  # noqa: E731
    tree = b"".join([shift(left).tobytes(), shift(right).tobytes(),
                     np.concatenate([np.zeros(chain, "<u4"), symbols]).astype("<u4").tobytes(),
                     bytes(chain) + leaf.tobytes()])
    prefix = rng.integers(0, 1 << chain, sym.size)
    bits = "".join(f"{p:0{chain}b}{code[s]:0{length[s]}b}" for p, s in zip(prefix.tolist(), sym.tolist()))
    data = int(bits.ljust(-(-len(bits) // 8) * 8, "0"), 2).to_bytes(-(-len(bits) // 8), "big")
    return struct.pack("<QI", nc + chain, 1 + len(tree)) + sec[12:13] + tree + struct.pack("<Q", len(data)) + data


@pytest.mark.parametrize("kind,chain", [("two", 12), ("fixed3", 12), ("cauchy", 13), ("wide", 12), ("two", 21)])
def test_gpu_decoder_node_arrays_that_are_no_tree(ctx, oracle, kind, chain):
    """Nodes shared by several parents: 4096 patterns of 12 bits that no code
    ends in, where the second-level tables have room for half the nodes (8 of
    them in the smallest case).  The codes past the room are walked, and the
    symbols are those of the plain tree."""
    rng = np.random.default_rng(chain)
    r1, r2 = 90, 130
    n = r1 * r2
    codes = [np.asarray(streams(kind, n, rng)), np.asarray(streams("wide", n, rng))]
    ids = ids_of("cauchy", 2 * n, rng)
    blob = blob_2d(oracle, ids, codes, r1, r2, rng)
    eb_size, u_size = struct.unpack_from("<QQ", blob, 12)
    v = blob[36 + eb_size + u_size:]
    n_unpred = struct.unpack_from("<Q", blob, 36 + eb_size + 25)[0]
    head = 33 + 4 * n_unpred + ((r1 - 1) // 12 * ((r2 - 1) // 12 + 1) + (r2 - 1) // 12) // 8 + 1
    u = blob[36 + eb_size:36 + eb_size + head] + shared_node_section(oracle, 131072, codes[0], rng, chain)
    sec = shared_node_section(oracle, 2048, ids, rng, chain)
    made = blob[:12] + struct.pack("<QQQ", len(sec), len(u), len(v)) + sec + u + v
    ou, ov = oracle.decompress_2d(blob, r1, r2)
    du, dv = cpsz_b200.sz_decompress_cp_preserve_2d_offline(made, r1, r2, ctx=ctx)
    assert_bits_equal(du, ou)
    assert_bits_equal(dv, ov)


def upload_whole():
    """The library's limit for blobs that go up in one piece (bytes)."""
    src = os.path.join(os.path.dirname(cpsz_b200.__file__), "csrc", "transfer.h")
    m = re.search(r"UPLOAD_WHOLE = \(size_t\)(\d+) << (\d+)", open(src).read())
    return int(m.group(1)) << int(m.group(2))


@pytest.mark.parametrize("r1,r2", [(400, 903), (1700, 3001)])
@pytest.mark.parametrize("which", ["ids", "u", "all"])
@pytest.mark.parametrize("device", [False, True])
def test_gpu_decoder_settles_streams_sent_whole_or_one_by_one(ctx, oracle, r1, r2, which, device):
    """Streams that never synchronise in a blob that goes up whole and in one
    above the limit, whose streams go up and are decoded one by one; into host
    arrays and into device memory (what is queued behind the first attempt
    must leave both to the second)."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(r1)
    n = r1 * r2
    kinds = {"ids": ("wide", "wide"), "u": ("fixed3", "wide"), "all": ("fixed3", "fixed16")}[which]
    codes = [np.asarray(streams(k, n, rng)) for k in kinds]
    blob = blob_2d(oracle, ids_of("cauchy" if which == "u" else "fixed3", 2 * n, rng), codes, r1, r2, rng)
    assert (len(blob) > upload_whole()) == (r1 > 1000)
    if device:
        out = [torch.full((r1, r2), 7.0, device="cuda") for _ in range(2)]
    else:
        out = [np.full((r1, r2), 7.0, np.float32) for _ in range(2)]
    cpsz_b200.sz_decompress_cp_preserve_2d_offline(blob, r1, r2, *out, ctx=ctx)
    # (the made-up values grow past the largest float: inf - inf is a NaN, which
    # x86 and the GPU encode differently)
    for a, b in zip(out, oracle.decompress_2d(blob, r1, r2)):
        assert_bits_equal(a.cpu().numpy() if device else a, b, nan_equal=True)


@pytest.mark.parametrize("shape", [(20, 33, 47), (100, 160, 110)])
@pytest.mark.parametrize("kind", ["fixed3", "wide"])
@pytest.mark.parametrize("device", [False, True])
def test_gpu_3d_decoder_settles_streams_sent_whole_or_one_by_one(ctx, oracle, shape, kind, device):
    """The same for volumes: made-up id and code streams, most points raw."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(shape[0])
    n = int(np.prod(shape))
    ids = rng.permutation(np.arange(n) % 8) + 5 if kind == "fixed3" else rng.integers(5, 12, n)
    ids = np.where(rng.random(n) < 0.65, np.where(rng.random(n) < 0.5, 0, 24), ids)
    npred = int(((ids != 0) & (ids != 24)).sum())
    codes = np.asarray(streams(kind, 3 * npred, rng)).clip(1, 65535)
    raw = np.exp2(rng.uniform(-3, 3, 3 * (n - npred))).astype(np.float32) * rng.choice([-1, 1], 3 * (n - npred))
    signs = rng.integers(0, 256, 3 * ((n - 1) // 8 + 1), np.uint8).tobytes()
    blob = struct.pack("<ii", 2, 32768) + signs + struct.pack("<Q", raw.size) + raw.astype(np.float32).tobytes() + \
        struct.pack("<Q", n) + oracle.huffman_encode(512, ids.astype(np.int32)) + struct.pack("<Q", codes.size) + \
        oracle.huffman_encode(131072, codes.astype(np.int32))
    assert (len(blob) > upload_whole()) == (n > 1 << 20)
    if device:
        out = [torch.full(shape, 7.0, device="cuda") for _ in range(3)]
    else:
        out = [np.full(shape, 7.0, np.float32) for _ in range(3)]
    cpsz_b200.sz_decompress_cp_preserve_3d_online_log(blob, *shape, *out, ctx=ctx)
    for a, b in zip(out, oracle.decompress_3d(blob, *shape)):
        assert_bits_equal(a.cpu().numpy() if device else a, b)
