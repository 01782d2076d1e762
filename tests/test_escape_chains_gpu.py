"""The class block encoder's chains at the edges of its batches, units and rows.

A block's two chains are staged 512 positions at a time and packed 16 positions a lane; a wrong state or a
bit out of place anywhere shows as other escape values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _round_trip(cuda, q):
    import torch
    from falcons_b200 import device as D
    q = torch.from_numpy(q.astype(np.int16)).to(cuda)
    torch.cuda.synchronize()
    back = D.decode_codes(D.encode_codes(q), q.numel())
    torch.cuda.synchronize()
    assert torch.equal(back, q)


def _escapes(kind, m, rng):
    if kind == "even":            # all classes alike: rows of several bit counts
        v = np.exp2(rng.uniform(7.01, 14.9, m))
    elif kind == "two":           # two classes of half a table: one bit a step
        v = np.where(rng.random(m) < 0.5, 200, 300)
    else:                         # one class and a few others: a long row of no bits beside rows of one cell
        v = np.where(rng.random(m) < 0.995, 200, np.exp2(rng.uniform(8, 14.9, m)))
    return v.astype(np.int64) * rng.choice([-1, 1], m)


@pytest.mark.parametrize("kind", ["even", "two", "skewed"])
@pytest.mark.parametrize("escapes", [18, 19, 513, 514, 515, 530, 531, 1026, 65536 - 14, 2 * 65536 + 514])
def test_chains_at_batch_and_unit_edges(cuda, kind, escapes):
    rng = np.random.default_rng(escapes)
    n = 76800 + escapes
    q = rng.integers(-20, 21, n)
    q[rng.choice(n, escapes, replace=False)] = _escapes(kind, escapes, rng)
    _round_trip(cuda, q)


def test_blocks_side_by_side(cuda):
    """More blocks than SMs (eight to a CTA), the last CTA not full, the last block short."""
    rng = np.random.default_rng(7)
    m = 171 * 65536 + 1000
    q = rng.integers(-20, 21, m + m // 8)
    q[rng.choice(q.size, m, replace=False)] = _escapes("even", m, rng)
    _round_trip(cuda, q)
