"""The chain decoder's edges: tables of every symbol, contexts outside shared memory, escapes filled in at the
edges of the fill's vectors and tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _round_trip(q, cuda):
    import torch
    from falcons_b200 import device as D
    q = torch.from_numpy(q.astype(np.int16)).to(cuda)
    torch.cuda.synchronize()
    enc = D.encode_codes(q)
    back = D.decode_codes(enc, q.numel())
    torch.cuda.synchronize()
    assert enc.cpu().numpy()[0] & 0x7F == 1, "method 1"
    assert torch.equal(back, q)


@pytest.mark.parametrize("where", ["first", "last", "vector ends", "tile ends", "runs", "all"])
@pytest.mark.parametrize("n", [76800, 76800 + 255, 76800 + 257, 131072 + 7])
def test_escapes_are_filled_in(cuda, where, n):
    rng = np.random.default_rng(n)
    q = rng.integers(-9, 10, n)
    at = {"first": [0], "last": [n - 1], "vector ends": [i for i in range(7, n, 8 * 31)],
          "tile ends": [i + d for i in range(256, n - 1, 256) for d in (-1, 0)],
          "runs": [i for i in range(n) if (i // 300) % 7 == 0], "all": range(n)}[where]
    at = np.asarray(list(at))
    q[at] = rng.integers(128, 32767, at.size) * rng.choice([-1, 1], at.size)
    q[at[0]] = -32768
    _round_trip(q, cuda)


@pytest.mark.parametrize("kind", ["wide tables", "all contexts", "rare contexts"])
def test_tables_and_contexts(cuda, kind):
    rng = np.random.default_rng(7)
    n = 200003
    if kind == "wide tables":      # 255 symbols beside a dominant one: the most chunks that a table can have
        q = np.where(rng.random(n) < 0.1, rng.integers(-127, 128, n), 100)
    elif kind == "all contexts":   # every context about as often
        q = rng.choice([0, 1, -1, 2, -2, 3, -3, 4, -4, 6, -6, 9, -9, 20, -20, 90, -90], n)
    else:                          # a stretch that lives in contexts that are rare over the whole
        q = np.where(rng.random(n) < 0.5, 0, rng.integers(-2, 3, n))
        q[-3000:] = rng.choice([9, -9, 6, -6, 4, -4], 3000)
    _round_trip(q, cuda)
