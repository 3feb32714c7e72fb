"""The small tiles' tensor-core products, which two SMs share, against exact host products: bytes over their full
range, fp16 and e4m3 operands whose sums are all representable."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["s8", "u8", "f16", "e4m3", "f16 heads"])
def test_products_of_a_pair(what):
    from brokefish_b200 import _native
    from brokefish_b200.nn.pack import sw128_image
    rng = np.random.default_rng(len(what))
    rows, n = 128, 128 if what == "f16 heads" else 256
    if what in ("s8", "u8"):
        a = rng.integers(0 if what == "u8" else -128, 256 if what == "u8" else 128, size=(rows, 256))
        w = rng.integers(-128, 128, size=(n, 256))
        for r in (0, 63, 64, 127):                       # the largest sums there are, on the edges of both halves
            a[r, :], w[r, :] = (255 if what == "u8" else -128), -128
        a_bytes, w_bytes = a.astype(np.uint8 if what == "u8" else np.int8).view(np.uint8), w.astype(np.int8).view(np.uint8)
    else:
        a, w = rng.integers(-2, 3, size=(rows, 256)), rng.integers(-2, 3, size=(n, 256))
        if what == "e4m3":
            a_bytes, w_bytes = (torch.from_numpy(m.astype(np.float32)).to(torch.float8_e4m3fn).view(torch.uint8).numpy()
                                for m in (a, w))
        else:
            a_bytes, w_bytes = a.astype(np.float16).view(np.uint8), w.astype(np.float16).view(np.uint8)
    image = np.concatenate([sw128_image(np.ascontiguousarray(w_bytes[:, s:s + 128])) for s in range(0, w_bytes.shape[1], 128)])
    cu = lambda m: torch.from_numpy(np.ascontiguousarray(m)).cuda()
    d_a, d_w, d_out = cu(a_bytes), cu(image), torch.zeros(rows, n, dtype=torch.int32, device="cuda")
    mode = 15 + ["s8", "u8", "f16", "e4m3", "f16 heads"].index(what)
    _native.check(_native.lib().bf_selftest_umma(0, mode, *(ctypes.c_void_p(t.data_ptr()) for t in (d_a, d_w, d_out))),
                  "bf_selftest_umma")
    got = d_out.cpu().numpy()
    if what == "e4m3":
        got = got.view(np.float32)
    elif what.startswith("f16"):
        got = np.ascontiguousarray(got.view(np.float16)[:, ::2])
    assert np.array_equal(got.astype(np.int64), a.astype(np.int64) @ w.astype(np.int64).T)
