"""Block-wise unpacking of zstd frames against ZSTD_decompress, on the CPU: frames that libzstd writes
of stored, run and compressed blocks in all orders, the headers it can give them, and damaged ones.
What is unpacked equals ZSTD_decompress's content; what ZSTD_decompress refuses is not unpacked."""
import ctypes as C

import numpy as np
import pytest

import asz_b200.api as api

Z = C.CDLL("libzstd.so.1")
for f in ("ZSTD_compress2", "ZSTD_decompress", "ZSTD_compressBound", "ZSTD_CCtx_setParameter"):
    getattr(Z, f).restype = C.c_size_t
Z.ZSTD_createCCtx.restype = C.c_void_p
LEVEL, WINDOW_LOG, CONTENT_SIZE, CHECKSUM = 100, 101, 200, 201


def _compress(data, **params):
    z = C.c_void_p(Z.ZSTD_createCCtx())
    for name, value in params.items():
        assert not Z.ZSTD_isError(Z.ZSTD_CCtx_setParameter(z, {"level": LEVEL, "window": WINDOW_LOG, "size": CONTENT_SIZE,
                                                               "checksum": CHECKSUM}[name], value))
    out = C.create_string_buffer(Z.ZSTD_compressBound(C.c_size_t(len(data))))
    n = Z.ZSTD_compress2(z, out, C.c_size_t(len(out)), data, C.c_size_t(len(data)))
    Z.ZSTD_freeCCtx(z)
    return out.raw[:n]


def _library(frame, raw):
    out = C.create_string_buffer(max(raw, 1))
    n = Z.ZSTD_decompress(out, C.c_size_t(raw), frame, C.c_size_t(len(frame)))
    return out.raw[:raw] if n == raw else None


def _ours(frame, raw):
    L = api.lib()
    L.asz_check_unframe.restype = C.c_int64
    L.asz_check_unframe.argtypes = [C.c_char_p, C.c_uint64, C.c_void_p, C.c_uint64]
    out = np.full(raw + 64, 0xA5, np.uint8)
    rc = L.asz_check_unframe(frame, len(frame), out.ctypes.data, raw)
    assert rc in (0, 1) and (out[raw:] == 0xA5).all()
    return out[:raw].tobytes() if rc else None


def _content(rng, kinds, block):
    parts = []
    for k in kinds:
        if k == "r":
            parts.append(rng.integers(0, 256, block, dtype=np.uint8))
        elif k == "z":
            parts.append(np.full(block, rng.integers(0, 256), np.uint8))
        elif k == "h":  # Huffman-compressible, no matches to speak of
            parts.append(rng.integers(0, 16, block, dtype=np.uint8) ** 2)
        elif k == "t":
            parts.append(np.tile(rng.integers(0, 256, 97, dtype=np.uint8), block // 97 + 1)[:block])
        else:  # matches that reach back over stored blocks
            old = np.concatenate(parts) if parts else rng.integers(0, 256, block, dtype=np.uint8)
            at = rng.integers(0, max(1, len(old) - 3000), 64)
            parts.append(np.concatenate([np.concatenate([old[a : a + 1500], rng.integers(0, 256, 40, dtype=np.uint8)])
                                         for a in at])[:block])
    return np.concatenate(parts).tobytes()


@pytest.mark.parametrize("kinds", ["r", "rrrrrr", "z", "zzrz", "h", "rhrh", "hhrrtt", "rmrm", "trmhz" * 4, "rrrrm" * 6])
@pytest.mark.parametrize("block", [131072, 131071, 50001, 7])
def test_equal_to_the_library(kinds, block):
    rng = np.random.default_rng(len(kinds) * block)
    data = _content(rng, kinds, block)
    for params in ({"level": 3}, {"level": 1}, {"level": 19}, {"level": 3, "window": 10}, {"level": 3, "window": 17}):
        frame = _compress(data, **params)
        assert _library(frame, len(data)) == data
        assert _ours(frame, len(data)) == data
    for params in ({"level": 3, "checksum": 1}, {"level": 3, "size": 0}):
        assert _ours(_compress(data, **params), len(data)) is None


def test_hand_made_frames():
    """Blocks that libzstd does not write: empty ones, short ones, runs of one byte value in the middle."""
    rng = np.random.default_rng(4)

    def block(kind, body, n, last):
        return (last | kind << 1 | n << 3).to_bytes(3, "little") + body

    stored = [rng.integers(0, 256, n, dtype=np.uint8).tobytes() for n in (5, 0, 131072, 1)]
    body = b"".join(block(0, s, len(s), 0) for s in stored) + block(1, b"\x07", 131072, 0) + block(1, b"\x09", 0, 0)
    body += block(0, b"", 0, 1)
    data = b"".join(stored) + b"\x07" * 131072
    frame = (0xFD2FB528).to_bytes(4, "little") + b"\xa0" + len(data).to_bytes(4, "little") + body
    assert _library(frame, len(data)) == data and _ours(frame, len(data)) == data
    assert _ours(frame + b"x", len(data)) is None and _ours(frame + frame, 2 * len(data)) is None
    assert _ours(frame, len(data) + 1) is None and _ours(frame, len(data) - 1) is None
    for n in list(range(0, 40)) + [len(frame) - 1]:
        assert _ours(frame[:n], len(data)) is None
    for head in (b"\xa1", b"\xa4", b"\xa8", b"\x20", b"\x00"):
        assert _ours(frame[:4] + head + frame[5:], len(data)) is None
    long = (0xFD2FB528).to_bytes(4, "little") + b"\xa0" + (131073).to_bytes(4, "little") + block(1, b"\x01", 131073, 1)
    assert _ours(long, 131073) is None  # left to the library, which takes runs above the format's block size


def test_damaged_frames():
    """A frame with a byte changed or cut short: refused, or the content that ZSTD_decompress finds too."""
    rng = np.random.default_rng(9)
    data = _content(rng, "hrmtzrhm", 20000)
    frame = _compress(data, level=3)
    for trial in range(600):
        bad = bytearray(frame)
        for _ in range(rng.integers(1, 4)):
            bad[rng.integers(4, len(bad))] = rng.integers(0, 256)
        bad = bytes(bad[: rng.integers(1, len(bad))] if trial % 5 == 0 else bad)
        got = _ours(bad, len(data))
        assert got is None or got == _library(bad, len(data))
