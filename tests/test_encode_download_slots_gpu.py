"""GPU: the encoder's levels in fresh and in part-touched pageable memory, just
below and above the 16 MB from which the copies of a context's second and later
calls are staged in pinned slots of 1 MB, the first call's being a plain one."""
import ctypes as C

import numpy as np
import pytest

from test_encode_gpu import OPT_DBF, OPT_DQ, OPT_FULL, _desc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,n", [(2048, 2720, 1), (2080, 2720, 1), (1312, 736, 6), (1920, 1088, 3)])
def test_levels_of_first_and_later_calls(pkg, w, h, n):
    rng = np.random.default_rng(w + n)
    pics = np.array([_desc(pkg, w, h, 10, 30, 5, OPT_FULL | OPT_DBF | OPT_DQ, 1) for _ in range(n)])
    yy, xx = np.mgrid[0:h, 0:w]
    base = (yy * 3 + xx * 2) % 1024
    srcs = [tuple((base[::s, ::s] + rng.integers(0, 64, base[::s, ::s].shape)).clip(0, 1023).astype(np.uint16)
                  for s in (1, 2, 2)) for _ in range(n)]
    arr = (pkg._PlaneIn * (3 * n))()
    for i, planes in enumerate(srcs):
        for c, a in enumerate(planes):
            arr[i * 3 + c] = pkg._PlaneIn(a.ctypes.data, a.strides[0] // 2, 0)
    with pkg.Context(0) as ctx:
        cus, levels = ctx.encode_batch(pics, srcs)
        assert levels.any() and levels.nbytes == 3 * w * h * n
        for _ in range(2):
            cu2, lv2 = ctx.encode_batch(pics, srcs)
            assert cu2.tobytes() == cus.tobytes() and (lv2 == levels).all()
        host = np.full(len(levels) + 64, 77, np.int16)
        st = ctx._L.vvcg_encode_batch(ctx._h, pics.ctypes.data_as(C.c_void_p), n, arr,
                                      cu2.ctypes.data_as(C.c_void_p), len(cu2), C.c_void_p(host.ctypes.data + 2),
                                      len(levels))
        assert st == pkg.OK and (host[1:len(levels) + 1] == levels).all()
        assert host[0] == 77 and (host[len(levels) + 1:] == 77).all()
