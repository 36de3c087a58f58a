"""HDF5 bitshuffle + LZ4 chunks on the GPU (qssb_decode_bslz4_u16,
qssb_encode_bslz4_u16 / qssb_pack_bslz4): round trips over full, tail and
leftover blocks; chunks written by the oracle and by the reference's own
writer kernels decode bit for bit, ours decode with the oracle's and the
reference's readers; malformed chunks are reported per chunk without a
fault; decoded counts reconstruct exactly as the originals."""
from __future__ import annotations

import ctypes
import struct

import numpy as np
import pytest
import torch

from oracle import bslz4_oracle as bo
from oracle.ref_cuda import build_bslz4
from quantem.gpu_b200 import SSB, _lib, ops
from quantem.gpu_b200.decode import decode_bslz4, encode_bslz4, from_chunks
from quantem.gpu_b200.synthetic import CONFIGS, generate

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _frames(n, shape, seed=0, dense=False):
    rng = np.random.default_rng(seed)
    f = rng.poisson(0.4, (n, *shape)).astype(np.uint16)
    if dense:
        f = rng.integers(0, 65536, (n, *shape), dtype=np.uint16)
    else:
        hot = rng.random((n, *shape)) < 0.002
        f[hot] = rng.integers(1000, 65536, int(hot.sum()), dtype=np.uint16)
    return f


@pytest.mark.parametrize("shape", [(128, 128), (96, 96), (192, 192), (3, 5), (41, 40), (64, 63)])
@pytest.mark.parametrize("dense", [False, True])
def test_round_trip_and_oracle_interchange(shape, dense):
    frames = _frames(6, shape, seed=shape[0] + shape[1], dense=dense)
    t = torch.as_tensor(frames, device=DEV)
    packed, offsets = encode_bslz4(t)
    np.testing.assert_array_equal(decode_bslz4(packed, offsets, shape).cpu().numpy(), frames)
    # our chunks through the oracle's reader
    host = packed.cpu().numpy().tobytes()
    offs = list(offsets.cpu().numpy()) + [len(host)]
    for i in range(len(frames)):
        np.testing.assert_array_equal(bo.decode_chunk(host[offs[i]:offs[i + 1]]).reshape(shape), frames[i])
    # the oracle's chunks through our reader
    chunks = [bo.encode_chunk(f) for f in frames[:3]]
    np.testing.assert_array_equal(from_chunks(chunks, shape, DEV).cpu().numpy(), frames[:3])


@pytest.mark.skipif(not build_bslz4.available(), reason="reference bitshuffle-LZ4 cubin not built")
@pytest.mark.parametrize("shape", [(128, 128), (192, 192)])
def test_reference_writer_and_reader_interchange(shape):
    from oracle.ref_cuda.bslz4 import ReferenceBslz4

    ref = ReferenceBslz4(DEV)
    frames = _frames(33, shape, seed=7)
    t = torch.as_tensor(frames, device=DEV)
    packed, offsets = ref.encode(t)
    np.testing.assert_array_equal(decode_bslz4(packed, offsets, shape).cpu().numpy(), frames)
    ours, our_offsets = encode_bslz4(t)
    np.testing.assert_array_equal(ref.decode(ours, our_offsets, shape).cpu().numpy(), frames)


def _corrupt(chunk: bytes, kind: str) -> bytes:
    if kind == "header":
        return struct.pack(">QI", 12345, 8192) + chunk[12:]
    if kind == "block_size":
        return chunk[:12] + struct.pack(">I", 0x7fffffff) + chunk[16:]
    if kind == "truncated":
        return chunk[: len(chunk) // 2]
    if kind == "lz4":  # first block replaced by literals 'abc' + a match at offset 9
        bad = bytes([0x35]) + b"abc" + struct.pack("<H", 9) + bytes([0x50]) + b"xyz12"
        (csz,) = struct.unpack(">I", chunk[12:16])
        return chunk[:12] + struct.pack(">I", len(bad)) + bad + chunk[16 + csz:]
    raise ValueError(kind)


@pytest.mark.parametrize("kind,code", [("header", 1), ("block_size", 2), ("truncated", 2), ("lz4", 3)])
def test_malformed_chunks_are_reported(kind, code):
    frames = _frames(3, (96, 96), seed=1)
    chunks = [bo.encode_chunk(f) for f in frames]
    chunks[1] = _corrupt(chunks[1], kind)
    offsets = np.zeros(3, np.int64)
    np.cumsum([len(c) for c in chunks[:-1]], out=offsets[1:])
    data = torch.as_tensor(np.frombuffer(b"".join(chunks), np.uint8).copy(), device=DEV)
    offs = torch.as_tensor(offsets, device=DEV)
    with pytest.raises(ValueError, match="chunk 1"):
        decode_bslz4(data, offs, (96, 96))
    out = decode_bslz4(data, offs, (96, 96), check=False).cpu().numpy()
    np.testing.assert_array_equal(out[0], frames[0])
    np.testing.assert_array_equal(out[2], frames[2])
    # the same call again: the context is intact
    assert torch.cuda.synchronize() is None


def test_decoded_acquisition_reconstructs_identically():
    spec = CONFIGS["plain_128x128_det128"]
    counts = generate(spec, DEV).counts
    packed, offsets = encode_bslz4(counts.reshape(-1, 128, 128))
    decoded = decode_bslz4(packed, offsets, (128, 128)).reshape(counts.shape)
    assert torch.equal(decoded.view(torch.int16), counts.view(torch.int16))
    assert packed.numel() < counts.numel() * 2 // 3  # sparse counts compress
    kw = dict(voltage_kV=spec.voltage_kV, semiangle_mrad=spec.semiangle_mrad,
              scan_sampling_A=spec.scan_step_A, det_sampling=spec.det_sampling_mrad)
    a = SSB.from_array(counts, **kw).reconstruct({"C10": 0.0, "C12": 0.0, "phi12": 0.0})
    b = SSB.from_array(decoded, **kw).reconstruct({"C10": 0.0, "C12": 0.0, "phi12": 0.0})
    assert torch.equal(a.object_wave, b.object_wave)


def test_ssb_from_chunks_matches_from_array():
    spec = CONFIGS["plain_32x32_det64"]
    counts = generate(spec, DEV).counts  # [32, 32, 64, 64] -> padded to 128^2 scans by the session
    kw = dict(voltage_kV=spec.voltage_kV, semiangle_mrad=spec.semiangle_mrad,
              scan_sampling_A=spec.scan_step_A, det_sampling=spec.det_sampling_mrad)
    packed, offsets = encode_bslz4(counts.reshape(-1, 64, 64))
    host = packed.cpu().numpy().tobytes()
    offs = list(offsets.cpu().numpy()) + [len(host)]
    chunks = [host[offs[i]:offs[i + 1]] for i in range(len(offs) - 1)]
    ab = {"C10": 50.0, "C12": 20.0, "phi12": 0.3}
    want = SSB.from_array(counts, **kw).reconstruct(ab).object_wave
    a = SSB.from_chunks(chunks, frame_shape=(64, 64), scan_shape=(32, 32), **kw).reconstruct(ab)
    b = SSB.from_chunks(packed.cpu().pin_memory(), chunk_offsets=offsets.cpu(), frame_shape=(64, 64),
                        scan_shape=(32, 32), **kw).reconstruct(ab)
    assert torch.equal(a.object_wave, want) and torch.equal(b.object_wave, want)


def _serial_lz4(src: bytes) -> bytes:
    """The encoder's search one position at a time: the last position of each
    12-bit hash, entered at every position looked at."""
    n, out, anchor, ip, table = len(src), bytearray(), 0, 0, {}

    def length(x):
        return b"\xff" * (x // 255) + bytes([x % 255])

    def literals(end, extra):
        lit = end - anchor
        out.append(min(lit, 15) << 4 | extra)
        if lit >= 15:
            out.extend(length(lit - 15))
        out.extend(src[anchor:end])

    while ip < n - 12:
        h = (int.from_bytes(src[ip:ip + 4], "little") * 2654435761 & 0xFFFFFFFF) >> 20
        cand, table[h] = table.get(h), ip
        if cand is None or src[cand:cand + 4] != src[ip:ip + 4]:
            ip += 1
            continue
        m = 4
        while ip + m < n - 5 and src[cand + m] == src[ip + m]:
            m += 1
        literals(ip, min(m - 4, 15))
        out.extend((ip - cand).to_bytes(2, "little"))
        if m - 4 >= 15:
            out.extend(length(m - 19))
        ip += m
        anchor = ip
    literals(n, 0)
    return bytes(out)


@pytest.mark.parametrize("shape", [(1, 8), (1, 23), (64, 64), (64, 65), (67, 62), (128, 96)])
@pytest.mark.parametrize("kind", ["zeros", "dense", "counts", "period", "collide"])
def test_encoder_writes_the_serial_search_bytes(shape, kind):
    """Blocks of 8 elements up to several blocks with a remainder; runs longer
    than a step, no match at all, matches of every distance, one hash shared by
    lanes of a step."""
    rng = np.random.default_rng(shape[0] * 131 + shape[1])
    n = shape[0] * shape[1]
    frames = np.zeros((3, *shape), np.uint16)
    if kind == "dense":
        frames = rng.integers(0, 65536, frames.shape, dtype=np.uint16)
    elif kind == "counts":
        frames = _frames(3, shape, seed=n)
    elif kind == "period":
        frames[:] = np.resize(np.repeat(rng.integers(0, 65536, 7, dtype=np.uint16), 11), frames.shape)
    elif kind == "collide":
        frames[:] = np.where(rng.random(frames.shape) < 0.03, 1, 0)
    packed, offsets = encode_bslz4(torch.as_tensor(frames, device=DEV))
    want = []
    for f in frames.reshape(3, n):
        chunk = struct.pack(">QI", 2 * n, 8192)
        for e0 in range(0, n // 8 * 8, 4096):
            comp = _serial_lz4(bo.bitshuffle(f[e0:min(e0 + 4096, n // 8 * 8)]))
            chunk += struct.pack(">I", len(comp)) + comp
        want.append(chunk + f[n // 8 * 8:].tobytes())
    assert offsets.cpu().tolist() == [0, len(want[0]), len(want[0]) + len(want[1])]
    assert packed.cpu().numpy().tobytes() == b"".join(want)
    np.testing.assert_array_equal(decode_bslz4(packed, offsets, shape).cpu().numpy(), frames)


@pytest.mark.parametrize("elements", [1, 7, 8, 4104, 12291])
@pytest.mark.parametrize("shift", [0, 1, 2, 3, 4, 16])
def test_pack_takes_scratch_and_output_at_any_address(elements, shift):
    """The C entries with scratch (and, the other way round, packed bytes)
    ``shift`` bytes into a buffer, down to chunks of raw elements alone."""
    frames = _frames(3, (elements, 1), seed=elements)
    t = torch.as_tensor(frames, device=DEV)
    want, want_offsets = bo.pack([bo.encode_chunk(f) for f in frames])
    nbytes = ctypes.c_size_t(0)
    _lib.check(_lib.load().qssb_encode_bslz4_scratch_bytes(3, 2 * elements, ctypes.byref(nbytes)))
    scratch = torch.empty(nbytes.value + 64, dtype=torch.uint8, device=DEV)[shift:]
    sizes = torch.empty(3, dtype=torch.int64, device=DEV)
    ops._call("qssb_encode_bslz4_u16", DEV, ops._ptr(t), 3, 2 * elements, ops._ptr(scratch),
              ops._ptr(sizes), ops._stream(t))
    offsets = torch.cumsum(sizes, 0) - sizes
    packed = torch.zeros(int(sizes.sum()) + 32, dtype=torch.uint8, device=DEV)[16 - shift:]
    ops._call("qssb_pack_bslz4", DEV, ops._ptr(scratch), ops._ptr(t), 3, 2 * elements,
              ops._ptr(offsets), ops._ptr(packed), ops._stream(t))
    host, offs = packed.cpu().numpy(), offsets.cpu().tolist()
    end = offs[1:] + [int(sizes.sum())]
    assert not host[end[-1]:].any()
    for f, a, b in zip(frames, offs, end):
        np.testing.assert_array_equal(bo.decode_chunk(host[a:b].tobytes()).reshape(f.shape), f)
    if elements < 8:  # raw elements only: the same bytes from any encoder
        assert offs == want_offsets.tolist()
        np.testing.assert_array_equal(host[:end[-1]], want)


def _many():
    """More chunks than the decoder gives four warps each."""
    return 13 * torch.cuda.get_device_properties(DEV).multi_processor_count + 1


def _decode_raw(chunks, elements, n):
    """(frames, statuses) of the first n of the chunks, repeated in turn."""
    picked = [chunks[i % len(chunks)] for i in range(n)]
    data, offsets = bo.pack(picked)
    comp, offs = torch.as_tensor(data, device=DEV), torch.as_tensor(offsets, device=DEV)
    out = torch.full((n, elements), 0x5a5a, dtype=torch.uint16, device=DEV)
    status = torch.full((n,), -1, dtype=torch.int32, device=DEV)
    ops._call("qssb_decode_bslz4_u16", DEV, ops._ptr(comp), comp.numel(), ops._ptr(offs), n,
              2 * elements, ops._ptr(out), ops._ptr(status), ops._stream(out))
    return out.cpu().numpy(), status.cpu().numpy()


def _sequence(lit: bytes, off=None, ml=4) -> bytes:
    """One LZ4 sequence (the last of a block without an offset)."""
    def ext(x):
        return b"\xff" * ((x - 15) // 255) + bytes([(x - 15) % 255]) if x >= 15 else b""

    head = bytes([min(len(lit), 15) << 4 | (0 if off is None else min(ml - 4, 15))])
    body = head + ext(len(lit)) + lit
    return body if off is None else body + struct.pack("<H", off) + ext(ml - 4)


OFFSETS = (1, 2, 3, 5, 31, 32, 33, 100, 127, 128, 129, 255, 511, 512, 513, 700)
LENGTHS = (4, 18, 19, 32, 33, 127, 131, 260, 515, 700, 6000)


def _blocks(rng):
    """LZ4 blocks of 8192 bytes with every offset and match length above at
    every output alignment, between literal runs of every token form, so that
    tokens fall anywhere in the 32 bytes that the decoder parses at once."""
    wanted = [(o, m, a) for o in OFFSETS for m in LENGTHS for a in range(4)]
    rng.shuffle(wanted)
    blocks, src, op = [], b"", 0
    for off, ml, align in wanted:
        for _ in range(2):
            lit = max(off - op, 0) + int(rng.choice([0, 0, 1, 3, 14, 15, 16, 40]))
            lit += (align - op - lit) % 4
            if op + lit + ml <= 8192:
                break
            blocks.append(src + _sequence(rng.bytes(8192 - op)))
            src, op = b"", 0
        src += _sequence(rng.bytes(lit), off, ml)
        op += lit + ml
    return blocks + [src + _sequence(rng.bytes(8192 - op))]


def _tail(rng, nbytes):
    """A block of a few bytes: literals, a short match where it fits, the rest."""
    if nbytes < 24:
        return _sequence(rng.bytes(nbytes))
    return _sequence(rng.bytes(5), 3, 9) + _sequence(rng.bytes(nbytes - 14))


def _chunk(blocks, raw=b"", total=None):
    body = b"".join(struct.pack(">I", len(b)) + b for b in blocks)
    return struct.pack(">QI", total, 8192) + body + raw


@pytest.mark.parametrize("elements", [4160, 4104, 4127])  # 32-byte, 16-byte and 2-byte stores
@pytest.mark.parametrize("many", [False, True])  # four warps a chunk, one
def test_matches_of_every_offset_length_and_alignment(elements, many):
    rng = np.random.default_rng(elements)
    chunks = [_chunk([b, _tail(rng, 2 * (elements // 8 * 8 - 4096))], rng.bytes(2 * (elements % 8)),
                     2 * elements) for b in _blocks(rng)]
    assert len(chunks) > 40
    want = np.stack([bo.decode_chunk(c) for c in chunks])
    n = _many() if many else len(chunks)
    got, status = _decode_raw(chunks, elements, n)
    assert not status.any()
    np.testing.assert_array_equal(got, want[np.arange(n) % len(chunks)])


@pytest.mark.parametrize("elements", [8, 15, 23])
def test_chunks_of_one_short_block(elements):
    rng = np.random.default_rng(elements)
    chunks = [_chunk([_tail(rng, 2 * (elements // 8 * 8))], rng.bytes(2 * (elements % 8)),
                     2 * elements) for _ in range(33)]
    want = np.stack([bo.decode_chunk(c) for c in chunks])
    got, status = _decode_raw(chunks, elements, 33)
    assert not status.any()
    np.testing.assert_array_equal(got, want)


RUN = _sequence(b"ab", 1, 8170)  # 8172 bytes of output
MALFORMED = {
    "no bytes": b"",
    "literal length cut off": b"\xf0\xff\xff",
    "match length cut off": b"\x1fa\x01\x00\xff",
    "literals cut off": b"\xe0abc",
    "offset cut off": _sequence(b"abcd", 2, 9) + b"\x10a\x01",
    "offset 0": _sequence(b"abc", 0, 9) + _sequence(b"x" * 8180),
    "offset 0 of a long match": _sequence(b"abc", 0, 99) + _sequence(b"x" * 8090),
    "offset before the output": _sequence(b"abc", 4, 9) + _sequence(b"x" * 8180),
    "offset before the output, long": _sequence(b"abc", 9, 99) + _sequence(b"x" * 8090),
    "match past the output": RUN + _sequence(b"12345678", 2, 13) + _sequence(b"x"),
    "long match past the output": _sequence(b"ab", 1, 9000) + _sequence(b"x"),
    "literals past the output": _sequence(b"x" * 8193),
    "literals past the output, short": RUN + _sequence(b"x" * 14, 1, 9) + _sequence(b"x"),
    "ends with a match": RUN + _sequence(b"12345678", 2, 12),
    "ends with a long match": _sequence(b"ab", 1, 8190),
    "ends with the parsed window": b"".join(_sequence(b"a", 1, 4) for _ in range(8)),
    "too short": RUN + _sequence(b"x" * 19),
    "goes on when full": RUN + _sequence(b"x" * 8, 1, 12) + _sequence(b"", 1, 4) + _sequence(b""),
}


@pytest.mark.parametrize("many", [False, True])
def test_malformed_blocks_in_both_kernels(many):
    """Between well-formed chunks: status 3, the bad block zero, the rest kept."""
    rng = np.random.default_rng(8)
    good = _blocks(rng)
    kinds = list(MALFORMED)
    for k in kinds:
        with pytest.raises(ValueError):
            bo.lz4_decompress(MALFORMED[k], 8192)
    tail = _tail(rng, 128)
    rest = bo.bitunshuffle(bo.lz4_decompress(tail, 128), 64, np.uint16)
    chunks, want = [], []
    for i, k in enumerate(kinds):
        for block in (MALFORMED[k], good[i]):
            chunks.append(_chunk([block, tail], total=2 * 4160))
            head = (np.zeros(4096, np.uint16) if block is MALFORMED[k]
                    else bo.bitunshuffle(bo.lz4_decompress(block, 8192), 4096, np.uint16))
            want.append(np.concatenate([head, rest]))
    # the chain and the header: the whole chunk is zero
    for bad, code in ((chunks[1][:-1], 2), (_corrupt(chunks[1], "header"), 1), (b"\x00" * 11, 1)):
        chunks.append(bad)
        want.append(np.zeros(4160, np.uint16))
    codes = np.array([3, 0] * len(kinds) + [2, 1, 1])
    n = _many() if many else len(chunks)
    got, status = _decode_raw(chunks, 4160, n)
    at = np.arange(n) % len(chunks)
    assert [int(s) for s in status] == codes[at].tolist()
    np.testing.assert_array_equal(got, np.stack(want)[at])
