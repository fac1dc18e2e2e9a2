"""Blocks whose inverse zfp wraps around 64 bits. The coder writes none from finite samples (they
are quantised three bits below the word's sign, and the transform averages), but a stream may hold
them: half of the coefficients the lowest 64-bit integer, the rest small. The streams of one
subband of an encoded field are replaced by such blocks, and the lane-per-block decode must give
what the general single-kernel decode (idx2g_decode_noalloc) gives, bit for bit."""
import os
import struct

import numpy as np
import pytest

from idx2_files import parse_data_file, varbytes
from test_zz_no_alloc import _noalloc

MASK = np.uint64(0xAAAAAAAAAAAAAAAA)
# coefficient j of a 3D block is the sample x + 4 y + 16 z (the reference's Core/Zfp.h:419 Perm3)
ORDER = [
    0, 1, 4, 16, 20, 17, 5, 2, 8, 32, 21, 6, 18, 24, 9, 33, 36, 3, 12, 48, 22, 25,
    37, 40, 34, 10, 7, 19, 28, 13, 49, 52, 41, 38, 26, 23, 29, 53, 11, 35, 44, 14, 50, 56,
    42, 27, 39, 45, 30, 54, 57, 60, 51, 15, 43, 46, 58, 61, 55, 31, 62, 59, 47, 63]
SUBBAND = 7  # 16^3 samples: 64 whole blocks


def _varbyte(v):
    out = bytearray()
    while True:
        out.append((v & 0x7F) | (0x80 if v >> 7 else 0))
        v >>= 7
        if not v:
            return bytes(out)


def _plane_bits(bits, n):
    """One plane of 64 coefficients by group tests, n of them significant before it: the stream's
    bits and the significant ones after it (the reference's Core/Zfp.h:990, read the other way)."""
    out = list(bits[:n])
    while n < 64:
        rest = bits[n:]
        out.append(int(any(rest)))
        if not any(rest):
            break
        run = list(rest).index(1)
        out += [0] * run
        n += run + 1
        if n < 64:
            out.append(1)
    return out, n


def _pack(bits):
    return np.packbits(np.array(bits, dtype=np.uint8), bitorder="little").tobytes()


def _blocks(rng, planes):
    """Planes (top first, a list of 64 bits each) of a block whose coefficients are the lowest integer
    or small: the top plane set at random, nothing down to the 26th, the others at random."""
    p = rng.random()
    top = (rng.random(64) < p).astype(int).tolist()
    low = [(rng.random(64) < rng.random()).astype(int).tolist() for _ in range(max(0, planes - 26))]
    return ([top] + [[0] * 64] * 25 + low)[:planes]


def _ilift(a, axis):
    x, y, z, w = np.moveaxis(a, axis, 0)
    y = y + (w >> 1)
    w = w - (y >> 1)
    y = y + w
    w = (w << 1) - y
    z = z + x
    x = (x << 1) - z
    y = y + z
    z = (z << 1) - y
    w = w + x
    x = (x << 1) - w
    return np.moveaxis(np.stack([x, y, z, w]), 0, axis)


def _inverse(q):
    a = q.reshape(4, 4, 4)
    for axis in (0, 1, 2):
        a = _ilift(a, axis)
    return a.reshape(-1)


def _coefficients(planes, first, count):
    u = np.zeros(64, dtype=np.uint64)
    for k in range(first, min(first + count, len(planes))):
        u |= np.array(planes[k], dtype=np.uint64) << np.uint64(63 - k)
    q = np.zeros(64, dtype=np.int64)
    q[ORDER] = ((u ^ MASK) - MASK).view(np.int64)
    return q


def _replace_streams(path, exps_bytes, bias, rng):
    """The data of every (brick, channel) of the subband replaced, the file's tables with them. Returns
    the blocks written."""
    data = open(path, "rb").read()
    p = parse_data_file(data)
    addrs = np.frombuffer(p["chunk_addrs"], dtype=np.uint64)
    key = (addrs & np.uint64(0xFFF)).astype(int)
    sub = ((addrs >> np.uint64(12)) & np.uint64(0x3F)).astype(int)
    kmin = key[sub == SUBBAND].min()
    raw = p["exp_chunks"][[int(a >> 12) & 0x3F for a in np.frombuffer(p["exp_addrs"], np.uint64)].index(SUBBAND)]
    emax = np.frombuffer(raw, dtype="<u2" if exps_bytes == 2 else "u1").astype(int)[:64] - bias
    top = emax + 63 + 1024
    blocks = [_blocks(rng, max(0, int(t - kmin + 1))) for t in top]
    stream, seen = {}, [0] * 64
    for k in range(int(top.max()), kmin - 1, -1):
        bits = []
        for b in range(64):
            if top[b] >= k:
                more, seen[b] = _plane_bits(blocks[b][top[b] - k], seen[b])
                bits += more
        stream[k] = _pack(bits)
    body, sizes, at = b"", b"", 0
    for i, n in enumerate(p["chunk_sizes"]):
        chunk = data[at:at + n]
        at += n
        if sub[i] == SUBBAND:
            # a chunk of the 8 like bricks: their number, the first, a bit per further one, sizes, data
            assert chunk[0] == 8 and chunk[1] == 0 and chunk[2] == 0x7F, chunk[:4]
            s = stream[int(key[i])]
            chunk = chunk[:3] + 8 * _varbyte(len(s)) + 8 * s
        body += chunk
        sizes += _varbyte(len(chunk))
    exps_total = struct.unpack("<i", data[-4:])[0]
    exps = data[len(data) - exps_total:]
    tail = data[:len(data) - exps_total]
    nz = struct.unpack("<i", tail[-8:-4])[0]
    z = tail[len(tail) - 8 - nz:]
    with open(path, "wb") as f:
        f.write(body + sizes + struct.pack("<i", len(sizes)) + z + exps)
    assert varbytes(sizes) == parse_data_file(open(path, "rb").read())["chunk_sizes"]
    return [b for b in blocks if b]


def _like_bricks(dtype):
    rng = np.random.default_rng(4)
    return np.ascontiguousarray(np.tile(rng.standard_normal((32, 32, 32)), (2, 2, 2)).astype(dtype))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [("float64", 1e-6), ("float64", 1e-8), ("float64", 1e-9), ("float32", 1e-7)])
def test_wrapping_blocks_match_wavefront(idx2g, tmp_path, dtype, tol):
    import torch
    idx2g.encode(_like_bricks(dtype), out_dir=str(tmp_path), name="w", field_name="f", num_levels=1, tolerance=tol)
    path = str(tmp_path / "w" / "f" / "L00.bin")
    blocks = _replace_streams(path, 2 if dtype == "float64" else 1, 1023 if dtype == "float64" else 127,
                              np.random.default_rng(7))
    assert 27 <= max(len(b) for b in blocks) <= 44
    # (the two parts' transforms, added, are not the whole's where it wraps: what the test is about)
    apart = [_inverse(_coefficients(b, 0, 26)) + _inverse(_coefficients(b, 26, 64)) for b in blocks]
    assert any((a != _inverse(_coefficients(b, 0, 64))).any() for a, b in zip(apart, blocks))
    ds = idx2g.Dataset(str(tmp_path / "w" / "f.idx2"))
    ours, want = (torch.empty((64, 64, 64), dtype=getattr(torch, dtype), device="cuda") for _ in range(2))
    ds.decode(out=ours)
    assert _noalloc(idx2g, ds, {"ds": (0, 0, 0), "tol": 0.0}, want) == 0
    torch.cuda.synchronize()
    assert ours.cpu().numpy().tobytes() == want.cpu().numpy().tobytes()
    ds.close()
