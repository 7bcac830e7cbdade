"""Device memory of a standalone tree handle: it is built from the caller's packed primitives and keeps no
copy of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_handle_keeps_no_primitives(xrt):
    torch = pytest.importorskip("torch")
    from xrtailor_gb300 import Lbvh
    n = 1 << 20
    p = np.random.default_rng(1).uniform(-1, 1, (n, 9)).astype(np.float32)
    d = torch.from_numpy(p).cuda()
    g = Lbvh()
    g.build_device(d.data_ptr(), 1)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    g.build_device(d.data_ptr(), n)
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    # leaf boxes 32, nodes 96, keys and sort 24, slots and prefixes 9, escapes 8 bytes a primitive;
    # two arrays of three float4 vertices would be 96 more
    assert used < (169 + 48) * n, used / n
