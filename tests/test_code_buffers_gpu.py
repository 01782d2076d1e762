"""Codes decoded into any place of a caller's buffer: the decoder's 16-byte stores must not need it aligned."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GUARD = 64


def _decode_into(buf, at, payload, n):
    """falcons_decode_codes into buf[at : at + n] (int16 elements)."""
    import torch
    from falcons_b200 import _lib
    ctx = _lib.default_context(0)
    _lib.check(_lib.lib().falcons_decode_codes(ctx.ptr, ctypes.c_void_p(payload.data_ptr()),
                                               ctypes.c_size_t(payload.numel()), ctypes.c_size_t(n),
                                               ctypes.c_void_p(buf.data_ptr() + 2 * at),
                                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "decode_codes")


def _codes(kind, n):
    rng = np.random.default_rng(n)
    if kind == "calm":        # method 1, no escapes
        q = rng.integers(-9, 10, n)
    elif kind == "escapes":   # method 1, escapes filled in afterwards
        q = np.round(rng.laplace(0, 90, n))
    elif kind == "delta":     # differences are coded
        q = np.cumsum(rng.choice([0, 0, 0, 1, -1, 300], n)) % 20000 - 10000
    else:                     # method 0
        q = np.where(rng.random(n) < 0.05, rng.integers(-300, 300, n), 0)
    return q.astype(np.int16)


@pytest.mark.parametrize("n", [76800, 76800 + 16 * 5 + 3, 262144 + 257])
@pytest.mark.parametrize("kind", ["calm", "escapes", "delta", "sparse"])
@pytest.mark.parametrize("offset", [0, 1, 3, 4, 7, 8])
def test_decode_into_a_slice(cuda, kind, n, offset):
    import torch
    from falcons_b200 import device as D
    q = torch.from_numpy(_codes(kind, n)).to(cuda)
    buf = torch.full((n + 2 * GUARD,), 12345, dtype=torch.int16, device=cuda)
    assert buf.data_ptr() % 16 == 0
    torch.cuda.synchronize()
    payload = D.encode_codes(q)
    _decode_into(buf, GUARD + offset, payload, n)
    torch.cuda.synchronize()
    assert payload.cpu().numpy()[0] & 0x7F == (0 if kind == "sparse" else 1)
    assert torch.equal(buf[GUARD + offset:GUARD + offset + n], q)
    assert bool((buf[:GUARD + offset] == 12345).all()) and bool((buf[GUARD + offset + n:] == 12345).all())
