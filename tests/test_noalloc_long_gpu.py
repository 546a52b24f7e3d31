"""fdtd_interior_step_noalloc on boxes far longer along one axis than the others, up to
its limit of 2^20 box cells, against the same expressions in numpy (the same order, so
bit for bit), with p_next apart from the others (one launch) and over p_curr (two)."""
import ctypes as C

import numpy as np
import pytest

from acoustics_b200._lib import load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(140002, 3, 3), (131073, 3, 3), ((1 << 20) + 2, 3, 3), (3, (1 << 20) + 2, 3),
                                  (3, 3, (1 << 20) + 2), (70001, 4, 9)])
@pytest.mark.parametrize("over", [False, True])
def test_long_boxes_equal_numpy(fdtd_lib, dims, over):
    import torch
    rng = np.random.default_rng(5)
    p, q = rng.normal(size=dims), rng.normal(size=dims)
    c2k2, scale = 0.0021, 37.5
    out = p if over else rng.normal(size=dims)
    want = out.copy()
    B = (slice(1, -1),) * 3
    lap = np.zeros_like(p[B])
    for d in range(3):
        up, dn = [slice(1, -1)] * 3, [slice(1, -1)] * 3
        up[d], dn[d] = slice(2, None), slice(0, -2)
        lap = lap + (p[tuple(up)] + p[tuple(dn)] - 2.0 * p[B])
    want[B] = 2.0 * p[B] - q[B] + (lap * scale) * c2k2
    dp, dq = torch.tensor(p, device="cuda"), torch.tensor(q, device="cuda")
    do = dp if over else torch.tensor(out, device="cuda")
    i3 = C.c_int32 * 3
    st = load().fdtd_interior_step_noalloc(dp.data_ptr(), dq.data_ptr(), do.data_ptr(), i3(*dims), i3(1, 1, 1),
                                           i3(*(n - 1 for n in dims)), c2k2, scale,
                                           torch.cuda.current_stream().cuda_stream)
    assert st == 0
    torch.cuda.synchronize()
    assert np.array_equal(do.cpu().numpy(), want)
