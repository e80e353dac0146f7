"""The tensor-core weight gradient beside the image's ends: an infinite
activation reaches the taps that pair it with a pixel of the image and no
others (tiles of 4 rows x 32 pixels, the rest of them zero-filled)."""
import ctypes as C
import os
import re

import pytest

torch = pytest.importorskip("torch")


def P(t):
    return C.c_void_p(t.data_ptr())


def _law(x, dy):
    """[k, 3, 3, c] in FP64: sums over the pairs inside the image only."""
    n, h, w, c = x.shape
    out = torch.zeros(dy.shape[3], 3, 3, c, dtype=torch.float64)
    for r in range(3):
        for s in range(3):
            i0, i1, j0, j1 = max(0, 1 - r), min(h, h + 1 - r), max(0, 1 - s), min(w, w + 1 - s)
            d = dy[:, i0:i1, j0:j1].reshape(-1, dy.shape[3]).double()
            v = x[:, i0 + r - 1:i1 + r - 1, j0 + s - 1:j1 + s - 1].reshape(-1, c).double()
            out[:, r, s] = (d[:, :, None] * v[:, None, :]).sum(0)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["last column", "last row", "corner"])
@pytest.mark.parametrize("h,w", [(4, 32), (5, 33), (6, 63), (7, 40), (3, 31), (2, 1), (1, 18), (8, 47)])
@pytest.mark.parametrize("c,k", [(8, 32), (40, 64)])
def test_infinite_activations_stay_in_their_taps(c, k, h, w, where):
    from pic_b200 import unet
    lib = unet.load()
    g = torch.Generator().manual_seed(100 * h + w)
    x = torch.randn(2, h, w, c, generator=g).bfloat16()
    dy = (torch.rand(2, h, w, k, generator=g) + 0.5).bfloat16()  # one sign: no inf - inf
    if where == "last column":
        x[:, :, w - 1, 3] = float("inf")
    elif where == "last row":
        x[:, h - 1, :, 5] = float("inf")
    else:
        x[1, h - 1, w - 1, :] = float("inf")
    dw = torch.zeros(k, 3, 3, c, dtype=torch.float32, device="cuda")
    xd, dyd = x.cuda(), dy.cuda()
    assert lib.unet_wgrad(2, h, w, c, k, P(xd), P(dyd), P(dw), None) == 0
    torch.cuda.synchronize()
    got, want = dw.double().cpu(), _law(x, dy)
    finite = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), finite)
    assert torch.equal(got[~finite], want[~finite])
    # FP32 sums of up to 750 exact products
    assert (got[finite] - want[finite]).abs().max() <= 1e-5 * max(1.0, float(want[finite].abs().max())) if finite.any() else True


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(1, 1), (1, 2), (2, 1), (9, 1), (1, 3), (2, 2)])
def test_narrow_images_match_fp64(h, w):
    """On both sides of what the CUDA cores keep: images one pixel wide, or of two."""
    from pic_b200 import unet
    lib = unet.load()
    g = torch.Generator().manual_seed(10 * h + w)
    n, c, k = 37, 16, 40
    x = torch.randn(n, h, w, c, generator=g).bfloat16()
    dy = torch.randn(n, h, w, k, generator=g).bfloat16()
    dw = torch.zeros(k, 3, 3, c, dtype=torch.float32, device="cuda")
    xd, dyd = x.cuda(), dy.cuda()
    assert lib.unet_wgrad(n, h, w, c, k, P(xd), P(dyd), P(dw), None) == 0
    torch.cuda.synchronize()
    got, want = dw.double().cpu(), _law(x, dy)
    assert (got - want).norm() <= 1e-5 * want.norm()  # FP32 sums of up to 333 exact products


@pytest.mark.gpu
def test_images_of_one_pixel_take_no_tile_each():
    """100,000 images of one pixel."""
    from pic_b200 import unet
    lib = unet.load()
    best = {}
    for n, h, w in ((100000, 1, 1),):
        x = torch.randn(n, h, w, 32, device="cuda").bfloat16()
        dy = torch.randn(n, h, w, 32, device="cuda").bfloat16()
        dw = torch.zeros(32, 3, 3, 32, device="cuda")
        best[h] = 1e9
        for _ in range(20):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda.synchronize()
            e[0].record()
            assert lib.unet_wgrad(n, h, w, 32, 32, P(x), P(dy), P(dw), None) == 0
            e[1].record()
            torch.cuda.synchronize()
            best[h] = min(best[h], e[0].elapsed_time(e[1]))
    # 273 us, against 671 with a tile each
    assert best[1] <= 0.45


def test_tile_counter_does_not_wrap():
    """Up to 2^31 - 1 tiles go to the kernel, and its CTAs step past the last one
    by up to their number: counted in 32 bits without a sign (34 GB operands:
    read from the source)."""
    from pic_b200 import unet
    src = open(os.path.join(os.path.dirname(unet.__file__), "csrc", "unet_ops.cu")).read()
    body = src[src.index(") k_wgrad_mma("):src.index("int run_wgrad_mma(")]
    loop = re.search(r"for \((\w+) (\w+) = blockIdx\.y; \2 < tiles; \2 \+= gridDim\.y", body)
    assert loop and loop.group(1) == "unsigned"
    assert re.search(r"const unsigned next = %s \+ gridDim\.y;" % loop.group(2), body)
    assert re.search(r"const unsigned tiles = ", body)
    assert "np < ((int64_t)1 << 31)" in src[src.index("int unet_wgrad("):]
