"""The operators of the stage interface at sizes where their kernels change: padding of the tiled scales, and the row counts
at which the router logits go from one kernel to another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _u16(t):
    import torch

    return t.view(torch.int16).cpu().numpy().view(np.uint16)


@pytest.mark.parametrize("rows,scale_columns", [(1, 1), (3, 7), (128, 4), (129, 10), (300, 64)])
def test_swizzled_scales_are_padded_with_zeros(cuda, pkg, rows, scale_columns):
    """cuda/nvfp4_ops.cu:869-890, byte for byte, also into a buffer that starts off a word boundary."""
    torch = cuda
    linear = torch.randint(0, 256, (rows, scale_columns), dtype=torch.uint8, device="cuda")
    n = pkg.nvfp4_swizzled_scale_bytes(rows, scale_columns)
    blocks = (scale_columns + 3) // 4
    want = np.zeros(n, np.uint8)
    r, c = np.meshgrid(np.arange(rows), np.arange(scale_columns), indexing="ij")
    at = ((r >> 7) * blocks + (c >> 2)) * 512 + (r & 31) * 16 + ((r >> 5) & 3) * 4 + (c & 3)
    want[at] = linear.cpu().numpy()
    for offset in (0, 1):
        out = torch.full((n + offset,), 0xAA, dtype=torch.uint8, device="cuda")[offset:]
        pkg.nvfp4_swizzle_scales(linear, out, rows, scale_columns)
        assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("batch", [2, 3, 4, 5, 7, 8, 9, 16, 17, 64, 255])
@pytest.mark.parametrize("experts,columns", [(256, 2560), (7, 256), (256, 384)])
def test_router_logits_keep_their_order_of_sums(cuda, pkg, orc, batch, experts, columns):
    """Bit for bit: a lane's chain over columns l, l + 32, ... and the shuffle tree (cuda/nvfp4_ops.cu:178-207)."""
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(batch)
    x = torch.empty((batch, columns), device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)
    w = torch.empty((experts, columns), device="cuda").normal_(0, 0.02, generator=g).to(torch.bfloat16)
    out = torch.full((batch, experts), float("nan"), dtype=torch.float32, device="cuda")
    pkg.bf16_gemm_f32(x, w, out, batch)
    want = orc.router_logits(_u16(x), _u16(w), gemv_order=False)
    assert np.array_equal(out.cpu().numpy(), want)
