"""fdtd_interior_step_noalloc against the same expressions in numpy (the same
order, so bit for bit): boxes of one cell, one row and one plane, odd sizes,
every remainder of the planes a thread takes, boxes at the domain edge and far
from it, p_next apart from the others, over p_prev, and over p_curr."""
import ctypes as C

import numpy as np
import pytest

from acoustics_b200._lib import load

pytestmark = pytest.mark.gpu

SHAPES = [((3, 3, 3), (1, 1, 1), (2, 2, 2)), ((5, 4, 70), (1, 1, 1), (4, 3, 69)), ((70, 5, 4), (1, 1, 1), (69, 4, 3)),
          ((4, 300, 5), (1, 1, 1), (3, 299, 4)), ((33, 34, 35), (2, 3, 5), (31, 30, 34)),
          ((64, 48, 40), (1, 1, 1), (63, 47, 39)), ((103, 101, 104), (1, 1, 1), (102, 100, 103))]


@pytest.mark.parametrize("dims,lo,hi", SHAPES)
@pytest.mark.parametrize("where", ["apart", "over p_prev", "over p_curr"])
def test_step_equals_numpy(fdtd_lib, dims, lo, hi, where):
    import torch
    rng = np.random.default_rng(3)
    p, q = rng.normal(size=dims), rng.normal(size=dims)
    c2k2, scale = 0.0021, 37.5
    out = {"apart": rng.normal(size=dims), "over p_prev": q, "over p_curr": p}[where]
    want = out.copy()
    B = tuple(slice(a, b) for a, b in zip(lo, hi))

    def at(d, s):
        return p[tuple(slice(a + s * (e == d), b + s * (e == d)) for e, (a, b) in enumerate(zip(lo, hi)))]

    lap = np.zeros_like(p[B])
    for d in range(3):
        lap = lap + (at(d, 1) + at(d, -1) - 2.0 * p[B])
    want[B] = 2.0 * p[B] - q[B] + (lap * scale) * c2k2
    dp, dq = torch.tensor(p, device="cuda"), torch.tensor(q, device="cuda")
    do = {"apart": torch.tensor(out, device="cuda"), "over p_prev": dq, "over p_curr": dp}[where]
    i3 = C.c_int32 * 3
    st = load().fdtd_interior_step_noalloc(dp.data_ptr(), dq.data_ptr(), do.data_ptr(), i3(*dims), i3(*lo), i3(*hi), c2k2,
                                           scale, torch.cuda.current_stream().cuda_stream)
    assert st == 0
    torch.cuda.synchronize()
    assert np.array_equal(do.cpu().numpy(), want)
