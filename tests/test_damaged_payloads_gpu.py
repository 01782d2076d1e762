"""Damaged payloads: a chain or part that gives up leaves its codes unwritten, the call says so and the next works."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _payload(cuda, n):
    import torch
    from falcons_b200 import device as D
    rng = np.random.default_rng(n)
    q = torch.from_numpy(np.round(rng.laplace(0, 90, n)).clip(-32767, 32767).astype(np.int16)).to(cuda)
    torch.cuda.synchronize()
    enc = D.encode_codes(q)
    torch.cuda.synchronize()
    return q, enc.cpu().numpy()


def _chains(p):
    """Method 1 payload of one segment: offsets of the chains' end bytes."""
    assert p[0] & 0x7F == 1 and int(p[5:13].view(np.uint64)[0]) == 1
    k = int(p[21:29].view(np.uint64)[0])
    blen = p[29:29 + 8 * k].view(np.uint64).astype(np.int64)
    return 29 + 16 * k + 15 * 256 * 2 + np.cumsum(blen) - 1


@pytest.mark.parametrize("bad", [[0], [15], [3, 4], list(range(16))])
def test_a_chain_without_its_end_mark_is_refused(cuda, bad):
    import torch
    from falcons_b200 import device as D
    n = 76800 + 41
    q, enc = _payload(cuda, n)
    ends = _chains(enc)
    assert ends.size == 16 and (enc[ends] != 0).all()
    d = enc.copy()
    d[ends[bad]] = 0
    with pytest.raises(ValueError):
        D.decode_codes(torch.from_numpy(d).to(cuda), n)
    back = D.decode_codes(torch.from_numpy(enc).to(cuda), n)
    torch.cuda.synchronize()
    assert torch.equal(back, q)


@pytest.mark.parametrize("field,value", [(8, 0xFFFF), (10, 0xFFFF), (0, 0xFFFF), (4, 0xFFFF)])
def test_a_checkpoint_out_of_range_is_not_used(cuda, field, value):
    """State, context, bit position or escape count of every seventh chain checkpoint out of range: those parts give
    up and the stream is decoded again from its ends."""
    import torch
    from falcons_b200 import api
    from falcons_b200 import device as D
    shape = (48, 64, 80)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        g = torch.Generator(device=cuda)
        g.manual_seed(1)
        x = torch.randn(shape, generator=g, device=cuda).cumsum(-1)
        conf = api.Config(*shape, errorBoundMode="ABS", absErrorBound=1e-2, cmprAlgo="INTERP")
        stream, _ = D.compress(x.clone(), conf)
        want, _ = D.decompress(stream, torch.float32)
        s.synchronize()
        b = stream.cpu().numpy().copy()
        tag = b.tobytes().rfind(b"FB2C")
        assert tag > 0
        n_o1 = int(b[tag + 16:tag + 24].copy().view(np.uint64)[0])
        assert n_o1 > 14
        for i in range(0, n_o1, 7):
            at = tag + 32 + 12 * i + field
            b[at:at + 2] = np.frombuffer(value.to_bytes(2, "little"), np.uint8)
            if field in (0, 4):
                b[at + 2:at + 4] = 0xFF
        got, _ = D.decompress(torch.from_numpy(b).to(cuda), torch.float32)
        s.synchronize()
    assert torch.equal(got, want)


@pytest.mark.parametrize("spread", ["some", "none in the first", "none counted"])
def test_escape_counts_of_the_header_only_place_the_values(cuda, spread):
    """A chain's escape count says where its values start, no more: with equal values the counts of neighbours may
    differ from what the chains hold, and the payload decodes as it is."""
    import torch
    from falcons_b200 import device as D
    n = 76800 + 41
    rng = np.random.default_rng(5)
    q = rng.integers(-20, 21, n)
    at = rng.choice(n, 3000, replace=False)
    if spread == "none in the first":
        at = at[at > n // 2]
    q[at] = 777
    q = torch.from_numpy(q.astype(np.int16)).to(cuda)
    torch.cuda.synchronize()
    enc = D.encode_codes(q).cpu().numpy()
    k = int(enc[21:29].view(np.uint64)[0])
    nvk = enc[29 + 8 * k:29 + 16 * k].view(np.uint64)
    assert k == 16 and int(nvk.sum()) == at.size and nvk[8] > 2 and (nvk[0] == 0) == (spread == "none in the first")
    d = enc.copy()
    counts = d[29 + 8 * k:29 + 16 * k].view(np.uint64)
    moved = counts[8] if spread == "none counted" else 2
    counts[8] -= moved
    counts[15] += moved - 1
    counts[0] += 1
    back = D.decode_codes(torch.from_numpy(d).to(cuda), n)
    torch.cuda.synchronize()
    assert torch.equal(back, q)
    counts[0] += 1  # more values than the payload holds
    with pytest.raises(ValueError):
        D.decode_codes(torch.from_numpy(d).to(cuda), n)
