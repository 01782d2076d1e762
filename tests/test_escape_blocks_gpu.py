"""Escape values at the edges of their class blocks, parts and units, with and without decode checkpoints.

A field of one row of anchors apart is hard to steer to an escape count, so the counts go through the code
coder (no checkpoints: a block is one part); the checkpointed form goes through a field whose codes are
mostly escapes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("escapes", [1, 2, 3, 4, 7, 8, 9, 1023, 1025, 1027, 65535, 65536, 65537, 66561])
def test_blocks_of_escapes_round_trip(cuda, escapes):
    import torch
    from falcons_b200 import device as D
    rng = np.random.default_rng(escapes)
    n = 76800 + escapes
    q = rng.integers(-20, 21, n)
    at = rng.choice(n, escapes, replace=False)
    q[at] = np.exp2(rng.uniform(7.01, 14.9, escapes)).astype(np.int64) * rng.choice([-1, 1], escapes)
    q = torch.from_numpy(q.astype(np.int16)).to(cuda)
    torch.cuda.synchronize()
    back = D.decode_codes(D.encode_codes(q), n)
    torch.cuda.synchronize()
    assert torch.equal(back, q)


@pytest.mark.parametrize("shape", [(44, 45, 46), (61, 59, 57), (300, 301)])
def test_checkpointed_blocks_of_a_field(cuda, shape):
    import torch
    from falcons_b200 import api
    from falcons_b200 import device as D
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        g = torch.Generator(device=cuda)
        g.manual_seed(5)
        x = torch.randn(shape, generator=g, device=cuda, dtype=torch.float64)
        conf = api.Config(*shape, errorBoundMode="ABS", absErrorBound=1e-4, cmprAlgo="INTERP")
        stream, _ = D.compress(x.clone(), conf)
        y, _ = D.decompress(stream, torch.float64)
        z, _ = api.decompress(stream.cpu().numpy(), np.float64)
    s.synchronize()
    assert float((y.view(shape) - x).abs().max()) <= 1e-4
    assert np.array_equal(y.cpu().numpy(), z.reshape(-1))


@pytest.mark.parametrize("n,gap", [(5000, 3), (76801, 40), (1 << 20, 1024), (3000001, 2999999), (4096 * 40, 4096)])
def test_runs_and_values_round_trip(cuda, n, gap):
    """Method 0: runs of zeros of any length (mantissas up to 21 bits) beside short values."""
    import torch
    from falcons_b200 import device as D
    rng = np.random.default_rng(n)
    q = np.zeros(n, np.int16)
    at = np.arange(gap - 1, n, gap) if gap != 3 else np.arange(0, n, 3)[::5]
    q[at] = rng.integers(1, 30000, at.size) * rng.choice([-1, 1], at.size)
    q = torch.from_numpy(q).to(cuda)
    torch.cuda.synchronize()
    enc = D.encode_codes(q)
    back = D.decode_codes(enc, n)
    torch.cuda.synchronize()
    assert enc.cpu().numpy()[0] & 0x7F == 0
    assert torch.equal(back, q)
