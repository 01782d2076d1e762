"""Decompress stages only the points of coarser levels: what the output buffer held before must not matter."""
import pytest

pytestmark = pytest.mark.gpu


# fields at the edges of the 64 x 64 tiles: last rows, columns and planes odd and even, one tile and several,
# rows on and off 16 bytes, two dimensions
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("shape", [(33, 64, 64), (32, 65, 68), (35, 63, 130), (34, 129, 127), (5, 66, 132), (3, 70, 72),
                                   (200, 260), (131, 193)])
def test_old_contents_do_not_matter(cuda, shape, dtype):
    import torch
    from falcons_b200 import api
    from falcons_b200 import device as D
    dt = getattr(torch, dtype)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        g = torch.Generator(device=cuda)
        g.manual_seed(3)
        x = torch.randn(shape, generator=g, device=cuda, dtype=dt).cumsum(-1)
        conf = api.Config(*shape, errorBoundMode="ABS", absErrorBound=1e-2, cmprAlgo="INTERP")
        stream, _ = D.compress(x.clone(), conf)
        outs = []
        for old in (0.0, float("nan"), float("inf")):
            # the allocator hands the freed block of this size to the output
            junk = torch.full(shape, old, device=cuda, dtype=dt).reshape(-1)
            del junk
            outs.append(D.decompress(stream, dt)[0].clone())
    s.synchronize()
    assert float((outs[0].view(shape) - x).abs().max()) <= 1e-2 * (1 + 1e-6)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
