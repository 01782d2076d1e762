"""Key counts of the chain coder at the smallest sizes it is used for (76800 codes) and at the edges of slices.

Below that size the codes take method 0, so the method is checked: the chains here have 4800 codes and more."""
import pytest

pytestmark = pytest.mark.gpu

# chains that start at every offset within a vector, the last chain short, slices of 4 Ki and 16 Ki codes and one code
# more or less; whole vectors only; one segment and two
SIZES = [76800, 76801, 76800 + 16 * 7 + 9, 16 * 4802 - 13, 16 * 8192 - 1, 16 * 8192 + 1, 16 * 16385, 16 * 32768 + 17,
         (1 << 24) + 1]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("offset", [0, 1, 5])  # codes on and off 16 bytes
def test_counts_of_short_chains(cuda, n, offset):
    import torch
    from falcons_b200 import device as D
    g = torch.Generator(device=cuda)
    g.manual_seed(n)
    pick = torch.rand(n + offset, generator=g, device=cuda)
    calm = torch.randint(-2, 3, (n + offset,), generator=g, device=cuda)
    wild = torch.randint(-300, 301, (n + offset,), generator=g, device=cuda)
    q = torch.where(pick < 0.9, calm, wild)
    # the clamps of the lookup table and the type's ends, first and last codes of chains among them
    edge = torch.tensor([-129, -128, -127, 127, 128, 129, -32768, 32767], device=cuda)
    at = torch.cat([torch.arange(0, n, max(1, n // 16), device=cuda), torch.arange(n - 8, n, device=cuda)]) + offset
    q[at] = edge[torch.arange(at.numel(), device=cuda) % 8]
    q = q.to(torch.int16)[offset:]
    torch.cuda.synchronize()
    enc = D.encode_codes(q)
    back = D.decode_codes(enc, n)
    torch.cuda.synchronize()
    assert enc.cpu().numpy()[0] & 0x7F == 1
    assert torch.equal(back, q)
