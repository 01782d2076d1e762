"""The chain encoder's ways to settle its parts' states: rounds of any number, and maps where a forecast from the first
rounds says that rounds would take longer."""
import re

import pytest

pytestmark = pytest.mark.gpu


def _codes(kind, n, device):
    import torch
    g = torch.Generator(device=device)
    g.manual_seed(n)
    if kind == "laplace":       # of few bits a code: about half of the parts do not meet
        u = torch.rand(n, generator=g, device=device) - 0.5
        q = -0.6 * u.sign() * torch.log1p(-2 * u.abs().clamp(max=0.49999))
    else:                       # stretches of few bits between others, 80 parts long or 20
        i = torch.arange(n, device=device)
        calm = (i // 40960) % 8 == 0 if kind == "long stretches" else (i // 20000) % 4 == 0
        q = torch.randn(n, generator=g, device=device) * torch.where(calm, 0.45, 3.0)
    return q.round().clamp(-32000, 32000).to(torch.int16)


# (codes, least and most rounds, whether the maps code the call)
@pytest.mark.parametrize("kind,n,rounds,maps", [("laplace", 40_000_000, (17, 25), False), ("long stretches", 4_000_000, (8, 16), True),
                                               ("short stretches", 40_000_000, (8, 12), True)])
def test_settling_rounds(cuda, monkeypatch, capfd, kind, n, rounds, maps):
    import torch
    from falcons_b200 import device as D
    q = _codes(kind, n, cuda)
    torch.cuda.synchronize()
    D.encode_codes(q)
    monkeypatch.setenv("FALCONS_TRACE", "1")
    capfd.readouterr()
    enc = D.encode_codes(q)
    torch.cuda.synchronize()
    m = re.search(r"re-run, (\d+) rounds, (\d+) of (\d+) parts not met, (\d+) chains unsettled", capfd.readouterr().err)
    monkeypatch.delenv("FALCONS_TRACE")
    took, unmet, parts, unsettled = (int(v) for v in m.groups())
    assert unmet <= parts // 2 and rounds[0] <= took <= rounds[1] and (unsettled > 0) == maps, m.group(0)
    back = D.decode_codes(enc, n)
    torch.cuda.synchronize()
    assert torch.equal(back, q)
