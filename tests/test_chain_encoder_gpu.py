"""The parallel chain encoder where its parts' states meet late or never.

The payload carries no checkpoints, so the decoder that reads it back walks every chain from its end to
its start: one wrong state anywhere shows as other codes behind it."""
import pytest

pytestmark = pytest.mark.gpu


def _codes(kind, n, device):
    import torch
    g = torch.Generator(device=device)
    g.manual_seed(n)
    normal = torch.randn(n, generator=g, device=device)
    if kind == "many bits":        # every part meets its kept states
        return (normal * 40).round()
    if kind == "few bits":         # most parts do not: the exact states come from the super parts' maps
        return (normal * 0.7).round()
    if kind == "mixed":            # some do not, several in a row: rounds
        scale = 10.0 ** (torch.rand(n // 3000 + 1, generator=g, device=device) * 3.5 - 1)
        return (normal * scale.repeat_interleave(3000)[:n]).round()
    if kind == "sign only":        # two symbols of half a table each: one bit a code
        return (normal > 0).float()
    return torch.full((n,), 7.0, device=device)  # certain codes merge no states: walked through


@pytest.mark.parametrize("kind", ["many bits", "few bits", "mixed", "sign only", "one symbol"])
@pytest.mark.parametrize("n", [76800, 76801, 16 * 256 * 20 + 1, 16 * 4096 * 8 - 7, 3000000])
def test_chains_decode_from_the_stream_alone(cuda, kind, n):
    import torch
    from falcons_b200 import device as D
    q = _codes(kind, n, cuda).clamp(-32768, 32767).to(torch.int16)
    torch.cuda.synchronize()
    enc = D.encode_codes(q)
    back = D.decode_codes(enc, n)
    torch.cuda.synchronize()
    assert torch.equal(back, q)


def test_super_parts_of_one_warp(cuda):
    """Enough super parts that a single warp takes each, in several segments."""
    import torch
    from falcons_b200 import device as D
    n = 40 * 1000 * 1000 + 3
    q = _codes("few bits", n, cuda).to(torch.int16)
    torch.cuda.synchronize()
    back = D.decode_codes(D.encode_codes(q), n)
    torch.cuda.synchronize()
    assert torch.equal(back, q)
