"""Device memory of a surrogate network whose layers are too large to split.

Its weight-gradient GEMMs have more tiles than the GPU has SMs, so each writes its
gradient in one piece and none needs room for partial products: the network holds
its parameters, gradient and two moments (FP32), two BF16 copies of the weights, its
batch buffers and no layer's weights besides.  Allocations are rounded up to 2 MiB
each: 50 of them are 100 MiB, below one such layer's 144 MiB of weights."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_unsplit_layers_reserve_no_partial_products(lcb):
    width, hidden, n_in, n_out, batch = 6144, 3, 8, 256, 8
    L = lcb._capi.load()
    h = C.c_void_p()
    # the library's code and context are loaded by a small network first
    lcb._capi.check_mlp(L.lcb_mlp_create(0, n_in, 8, 1, 8, 8, 1, C.byref(h)))
    L.lcb_mlp_destroy(h)
    torch.cuda.synchronize()
    free0, _ = torch.cuda.mem_get_info()
    lcb._capi.check_mlp(L.lcb_mlp_create(0, n_in, width, hidden, n_out, batch, 1, C.byref(h)))
    torch.cuda.synchronize()
    free1, _ = torch.cuda.mem_get_info()
    L.lcb_mlp_destroy(h)
    weights = n_in * width + (hidden - 1) * width * width + width * n_out
    params = weights + hidden * width + n_out
    assert free0 - free1 <= 4 * 4 * params + 2 * 2 * weights + 100 * 2 ** 20
