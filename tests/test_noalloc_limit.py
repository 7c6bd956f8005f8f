"""The no-allocation floodfill takes the grids whose workspace, as
cubvh_floodfill_workspace_size gives it, fits into 32 MiB, and no others."""

import ctypes

import pytest
import torch

from cubvh_b200 import _lib


@pytest.mark.parametrize("W", [180, 192, 193, 224])
def test_limit_is_the_workspace(W):
    L = _lib.lib()
    taken = []
    for n in range(150, 260):
        nb = ctypes.c_size_t()
        assert L.cubvh_floodfill_workspace_size(1, n, W, n, ctypes.byref(nb)) == 0
        # the check of a NULL workspace looks at the limit first; what follows needs a GPU
        rc = L.cubvh_floodfill_check(None, 1, n, W, n, None)
        refused = rc != 0 and b"bytes of scratch" in L.cubvh_last_error()
        assert refused == (nb.value > 32 << 20), (n, nb.value)
        taken.append(not refused)
    assert taken[0] and not taken[-1]


@pytest.mark.gpu
def test_largest_grid():
    L, dev = _lib.lib(), torch.device("cuda:0")
    nb = ctypes.c_size_t()

    def size(n):
        assert L.cubvh_floodfill_workspace_size(1, n, 192, n, ctypes.byref(nb)) == 0
        return nb.value

    n = max(k for k in range(150, 260) if size(k) <= 32 << 20)
    shape = (1, n, 192, n)
    g = torch.rand(shape, generator=torch.Generator(device=dev).manual_seed(n), device=dev) < 0.4
    out = [torch.empty(shape, dtype=torch.int32, device=dev) for _ in range(2)]
    stream = torch.cuda.current_stream(dev).cuda_stream
    ws = torch.empty(size(n), dtype=torch.uint8, device=dev)
    fn = L.cubvh_floodfill_noalloc
    fn.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 4 + [ctypes.c_void_p] * 2
    fn.restype = ctypes.c_int
    assert fn(g.data_ptr(), *shape, out[0].data_ptr(), stream) == 0, L.cubvh_last_error()
    assert L.cubvh_floodfill_check(None, *shape, stream) == 0, L.cubvh_last_error()
    assert L.cubvh_floodfill(g.data_ptr(), *shape, out[1].data_ptr(), ws.data_ptr(), nb.value, stream) == 0
    assert torch.equal(*out)
