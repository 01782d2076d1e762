"""What a caller's output tensor holds before a decompress must not matter: NaN, infinities, the type's largest value."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("offset", [0, 1])  # rows on and off 16 bytes
@pytest.mark.parametrize("shape", [(33, 64, 64), (35, 63, 130), (34, 129, 127), (5, 66, 132), (200, 260), (131, 193), (70, 70, 70)])
def test_given_output(cuda, shape, offset, dtype):
    import torch
    from falcons_b200 import api
    from falcons_b200 import device as D
    dt = getattr(torch, dtype)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        g = torch.Generator(device=cuda)
        g.manual_seed(4)
        x = torch.randn(shape, generator=g, device=cuda, dtype=dt).cumsum(-1)
        conf = api.Config(*shape, errorBoundMode="ABS", absErrorBound=1e-2, cmprAlgo="INTERP")
        stream, _ = D.compress(x.clone(), conf)
        outs = []
        for old in (0.0, float("nan"), float("-inf"), torch.finfo(dt).max):
            buf = torch.full((x.numel() + 8,), old, device=cuda, dtype=dt)
            out = buf[offset:offset + x.numel()]
            D.decompress(stream, dt, out=out)
            outs.append(out.clone())
            rest = torch.cat([buf[:offset], buf[offset + x.numel():]])
            assert torch.equal(rest.nan_to_num(7.0), torch.full_like(rest, old).nan_to_num(7.0))
    s.synchronize()
    assert float((outs[0].view(shape) - x).abs().max()) <= 1e-2 * (1 + 1e-6)
    assert all(torch.equal(outs[0], o) for o in outs[1:])
