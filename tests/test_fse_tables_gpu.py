"""Class blocks whose table an encoder elsewhere made larger than the ones written here (2^12 and 2^13 cells), with and
without low-probability symbols, and the scratch that decoding blocks takes."""
import ctypes
import struct

import numpy as np
import pytest

from test_entropy_rules import rules  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


def _records(rules, cls, log, low):  # noqa: F811
    """fse_enc records of a class stream: 64 Ki blocks, FSE with tables of 2^log cells."""
    out = b""
    for b in range(0, cls.size, 65536):
        src = np.ascontiguousarray(cls[b:b + 65536])
        if (src == src[0]).all():
            out += bytes([2, src[0]])
            continue
        dst = np.zeros(2 * src.size + 4096, np.uint8)
        n = rules.rules_fse_block(src.ctypes.data_as(ctypes.c_void_p), ctypes.c_ulonglong(src.size), log, low,
                                  dst.ctypes.data_as(ctypes.c_void_p), ctypes.c_ulonglong(dst.size))
        assert n > 0
        assert (dst[0] & 15) + 5 == log
        out += b"\x01" + struct.pack("<I", n) + dst[:n].tobytes()
    return out


def _payload(rules, q, log, low):  # noqa: F811
    """A method 0 payload of nonzero codes (no runs of zeros)."""
    v = np.where(q >= 0, 2 * q, -2 * q - 1).astype(np.int64) + 1
    k = np.floor(np.log2(v)).astype(np.uint8)
    bits = ((v[:, None] >> np.arange(16, -1, -1)) & 1).astype(np.uint8)
    man = np.packbits(bits[np.arange(16, -1, -1)[None, :] < k[:, None]]).tobytes()
    runs = _records(rules, np.zeros(q.size, np.uint8), log, low)
    vals = _records(rules, k, log, low)
    return bytes(5) + struct.pack("<6Q", q.size, q.size, len(runs), len(vals), 0, len(man)) + runs + vals + man


@pytest.mark.parametrize("low", [0, 1])
@pytest.mark.parametrize("log", [5, 11, 12, 13])
@pytest.mark.parametrize("n", [300, 301, 65536, 65536 + 4099, 3 * 65536 + 7])
def test_blocks_with_tables_of_any_size(cuda, rules, n, log, low):  # noqa: F811
    import torch
    from falcons_b200 import device as D
    rng = np.random.default_rng(n + log)
    # classes 1 to 15, the last ones rare (a cell of their own)
    q = np.exp2(rng.exponential(3.0, n).clip(0, 14.9)).astype(np.int64) * rng.choice([-1, 1], n)
    p = torch.frombuffer(bytearray(_payload(rules, q, log, low)), dtype=torch.uint8).to(cuda)
    back = D.decode_codes(p, n)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(back.cpu().numpy(), q.astype(np.int16))


def test_scratch_of_blocks(cuda):
    """No block reserves a table of the largest size (32 KiB), which no encoder here writes."""
    import torch
    from cuda.bindings import driver, runtime as rt
    from falcons_b200 import device as D
    n = 1 << 22
    rng = np.random.default_rng(3)
    q = torch.from_numpy((rng.integers(128, 32000, n) * rng.choice([-1, 1], n)).astype(np.int16)).to(cuda)
    torch.cuda.synchronize()
    enc = D.encode_codes(q)
    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    attr = rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh
    zero = driver.cuuint64_t(0)
    assert rt.cudaMemPoolSetAttribute(pool, attr, zero)[0] == 0
    back = D.decode_codes(enc, n)
    torch.cuda.synchronize()
    err, high = rt.cudaMemPoolGetAttribute(pool, attr)
    assert torch.equal(back, q)
    # all codes are escapes: values 2 B, classes 1 B and a sign bit a code, and a slab of 1 MiB for everything else on
    # each of the two streams; half a MiB for rounding (64 tables of 32 KiB would be 2 MiB more)
    assert int(high) <= 3 * n + n // 8 + (5 << 19), int(high)
