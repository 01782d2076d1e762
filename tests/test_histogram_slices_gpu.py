"""Key counts of the chain coder at the edges of its chains, slices and vectors.

The tables are built from these counts and the encoder codes the keys written beside them, so a code
counted or keyed as another one shows as a stream that does not decode to its codes."""
import pytest

pytestmark = pytest.mark.gpu

# one code a chain; less than a vector; chain starts at every offset within a vector; a slice more;
# two segments, the last one short
SIZES = [1, 15, 16, 17, 127, 76800 + 16 * 3 + 5, 16 * 16384 - 1, 16 * 16384 + 9, 16 * 3 * 16384 + 16 * 5 + 2,
         (1 << 24) + 4099]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("offset", [0, 1])  # 1: codes not on 16 bytes, read one at a time
def test_counts_at_slice_edges(cuda, n, offset):
    import torch
    from falcons_b200 import device as D
    g = torch.Generator(device=cuda)
    g.manual_seed(n)
    # every symbol, both clamps of the lookup table (-128 and 128) and the extremes of the type
    wild = torch.randint(-300, 301, (n + offset,), generator=g, device=cuda)
    calm = torch.randint(-2, 3, (n + offset,), generator=g, device=cuda)
    pick = torch.rand(n + offset, generator=g, device=cuda)
    q = torch.where(pick < 0.9, calm, wild)
    q = torch.where(pick > 0.9995, torch.full_like(q, 32767), q)
    q = torch.where((pick < 0.9995) & (pick > 0.999), torch.full_like(q, -32768), q)
    q = q.to(torch.int16)[offset:]
    torch.cuda.synchronize()
    back = D.decode_codes(D.encode_codes(q), n)
    torch.cuda.synchronize()
    assert torch.equal(back, q)
