"""Class blocks that are coded alone on an SM: rows of all states where their symbols are few, step rows where not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _runs(lengths, rng):
    """Codes whose runs of zeros between nonzero codes have these lengths (method 0: classes of run and value)."""
    at = np.cumsum(np.asarray(lengths) + 1) - 1
    q = np.zeros(int(at[-1]) + 1, np.int16)
    q[at] = rng.integers(1, 100, at.size) * rng.choice([-1, 1], at.size)
    return q


# a run of 2^c - 1 zeros has class c: 24 classes are the most whose rows fit (2^11 states), 25 one more, each once
# between short runs that fill the block; small tables, one symbol beside another, the smallest blocks
@pytest.mark.parametrize("classes,n", [(24, 65536), (25, 65536), (25, 300), (2, 65536), (2, 3), (3, 4), (12, 2 * 65536 + 3)])
def test_classes_of_runs(cuda, classes, n):
    import torch
    from falcons_b200 import device as D
    rng = np.random.default_rng(n + classes)
    once = (1 << np.arange(min(classes, n)).astype(np.int64)) - 1
    rest = (1 << rng.integers(0, min(classes, 4), n - once.size)) - 1
    q = _runs(rng.permutation(np.concatenate([once, rest])), rng)
    t = torch.from_numpy(q).to(cuda)
    torch.cuda.synchronize()
    enc = D.encode_codes(t)
    back = D.decode_codes(enc, q.size)
    torch.cuda.synchronize()
    assert torch.equal(back, t)
    if classes > 20:
        assert enc.cpu().numpy()[0] & 0x7F == 0


# blocks beside the chain encoder of a few codes, which they outlast: an SM each
@pytest.mark.parametrize("escapes", [40000, 65536, 65537, 150000])
def test_blocks_beside_few_codes(cuda, escapes):
    import torch
    from falcons_b200 import api
    from falcons_b200 import device as D
    rng = np.random.default_rng(escapes)
    n = 300000
    q = rng.integers(-20, 21, n)
    at = rng.choice(n, escapes, replace=False)
    q[at] = np.exp2(rng.uniform(7.01, 14.9, escapes)).astype(np.int64) * rng.choice([-1, 1], escapes)
    q = torch.from_numpy(q.astype(np.int16)).to(cuda)
    torch.cuda.synchronize()
    back = D.decode_codes(D.encode_codes(q), n)
    torch.cuda.synchronize()
    assert torch.equal(back, q)
    # through a field, whose stream carries the blocks' checkpoints
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        x = torch.from_numpy(rng.normal(0, 1, (3, escapes // 3))).to(cuda)
        conf = api.Config(3, escapes // 3, errorBoundMode="ABS", absErrorBound=1e-4, cmprAlgo="INTERP")
        stream, _ = D.compress(x.clone(), conf)
        y, _ = D.decompress(stream, torch.float64)
    s.synchronize()
    assert float((y.view(x.shape) - x).abs().max()) <= 1e-4
