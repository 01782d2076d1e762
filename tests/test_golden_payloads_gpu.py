"""Code payloads that the reference's encoder wrote (tests/golden/rlefse_*.npz), decoded on the GPU without its build:
methods 0 and 1, deltas, counts and blocks of its own making, at any place in memory."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


@pytest.mark.parametrize("offset", [0, 1, 3, 8])
@pytest.mark.parametrize("name,first", [("sparse", 0), ("dense", 1), ("delta", 129)])
def test_payload_of_the_reference(cuda, name, first, offset):
    import torch
    from falcons_b200 import device as D
    g = np.load(os.path.join(GOLDEN, f"rlefse_{name}.npz"))
    p = g["payload"]
    assert p[0] == first
    buf = torch.zeros(p.size + 16, dtype=torch.uint8, device=cuda)
    buf[offset:offset + p.size] = torch.from_numpy(p.copy()).to(cuda)
    back = D.decode_codes(buf[offset:offset + p.size], g["codes"].size)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(back.cpu().numpy(), g["codes"])
