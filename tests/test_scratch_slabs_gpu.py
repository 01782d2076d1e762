"""Scratch cut from slabs: blocks around the size that gets an allocation of its own, and calls side by side.

Two blocks that overlap, or scratch of one call that another one's stream reuses too early, show as other codes."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def _codes(n, seed, device):
    import torch
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    q = torch.randn(n, generator=g, device=device) * 30
    q[:: 97] *= 60  # some escapes
    return q.round().clamp(-32000, 32000).to(torch.int16)


# codes of two bytes a block of 256 KB holds, less the slack behind them, and one block more
@pytest.mark.parametrize("n", [131072 - 168, 131072 - 40, 131072 - 39, 131072 - 8, 131072, 131073, 524288 - 33])
def test_blocks_around_the_slab_limit(cuda, n):
    import torch
    from falcons_b200 import device as D
    q = _codes(n, n, cuda)
    torch.cuda.synchronize()
    back = D.decode_codes(D.encode_codes(q), n)
    torch.cuda.synchronize()
    assert torch.equal(back, q)


def test_calls_side_by_side(cuda):
    import torch
    from falcons_b200 import device as D
    from falcons_b200 import _lib
    sizes = [80000, 131072, 262144, 90001]
    qs = [_codes(n, i, cuda) for i, n in enumerate(sizes)]
    torch.cuda.synchronize()
    same = [0] * len(qs)

    def work(i):
        s = torch.cuda.Stream()
        ctx = _lib.Context(0)
        with torch.cuda.stream(s):
            for _ in range(6):
                back = D.decode_codes(D.encode_codes(qs[i], ctx=ctx, stream=s), sizes[i], ctx=ctx, stream=s)
                s.synchronize()
                same[i] += int(torch.equal(back, qs[i]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(qs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert same == [6] * len(qs)
