"""The order-1 tANS tables at the edges of what a context's counts can be, through whole round trips.

The encoder's and the decoder's tables are built apart (the decoder's from the stream's counts), so a
round trip that returns the codes has the same spread, ranks and transforms on both sides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _codes(kind, n):
    rng = np.random.default_rng(n)
    if kind == "one symbol":          # a context with one symbol: all 8192 cells
        return np.full(n, 7)
    if kind == "all symbols":         # every symbol in the widest contexts, a cell or more each
        return rng.integers(-127, 128, n)
    if kind == "rare symbols":        # many symbols at the one-cell floor beside a dominant one
        return np.where(rng.random(n) < 0.002, rng.integers(-127, 128, n), 3)
    if kind == "escapes":             # the escape symbol dominates
        return np.where(rng.random(n) < 0.95, rng.integers(128, 30000, n), rng.integers(-3, 4, n))
    return rng.choice([-1, 1], n)     # two symbols of half a table each


@pytest.mark.parametrize("kind", ["one symbol", "all symbols", "rare symbols", "escapes", "two symbols"])
@pytest.mark.parametrize("n", [76800, 76807])
def test_tables_round_trip(cuda, kind, n):
    import torch
    from falcons_b200 import device as D
    q = torch.from_numpy(_codes(kind, n).astype(np.int16)).to(cuda)
    torch.cuda.synchronize()
    enc = D.encode_codes(q)
    back = D.decode_codes(enc, n)
    torch.cuda.synchronize()
    assert enc.cpu().numpy()[0] & 0x7F == 1, "method 1 is the one with these tables"
    assert torch.equal(back, q)
