"""GPU: the encoder's levels reach pageable, part-touched and pinned host
memory and device memory alike, whatever the destination's alignment (large
pageable copies are staged in slots by several threads)."""
import ctypes as C

import numpy as np
import pytest

from test_encode_gpu import OPT_DBF, OPT_DQ, OPT_FULL, _desc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,n", [(64, 64, 1), (1408, 992, 1), (1440, 992, 1), (1920, 1088, 1), (1312, 736, 5)])
def test_levels_reach_every_kind_of_destination(ctx, pkg, w, h, n):
    import torch

    rng = np.random.default_rng(w + n)
    pics = np.array([_desc(pkg, w, h, 10, 30, 5, OPT_FULL | OPT_DBF | OPT_DQ, 1) for _ in range(n)])
    yy, xx = np.mgrid[0:h, 0:w]
    base = (yy * 3 + xx * 2) % 1024
    srcs = [tuple((base[::s, ::s] + rng.integers(0, 64, base[::s, ::s].shape)).clip(0, 1023).astype(np.uint16)
                  for s in (1, 2, 2)) for _ in range(n)]
    cus, levels = ctx.encode_batch(pics, srcs)  # fresh pageable memory
    assert levels.any()
    nl = len(levels)
    arr = (pkg._PlaneIn * (3 * n))()
    for i, planes in enumerate(srcs):
        for c, a in enumerate(planes):
            arr[i * 3 + c] = pkg._PlaneIn(a.ctypes.data, a.strides[0] // 2, 0)
    host = np.full(nl + 64, 77, np.int16)
    pinned = torch.full((nl + 64,), 77, dtype=torch.int16, pin_memory=True)
    dev = torch.full((nl + 64,), 77, dtype=torch.int16, device="cuda")
    torch.cuda.synchronize()
    for buf, addr in ((host, host.ctypes.data), (pinned, pinned.data_ptr()), (dev, dev.data_ptr())):
        cu2 = np.zeros_like(cus)
        st = ctx._L.vvcg_encode_batch(ctx._h, pics.ctypes.data_as(C.c_void_p), n, arr,
                                      cu2.ctypes.data_as(C.c_void_p), len(cu2), C.c_void_p(addr + 2), nl)
        assert st == pkg.OK
        torch.cuda.synchronize()
        got = buf if isinstance(buf, np.ndarray) else buf.cpu().numpy()
        assert (got[1:nl + 1] == levels).all() and got[0] == 77 and (got[nl + 1:] == 77).all()
        assert cu2.tobytes() == cus.tobytes()
