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


@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 4128, 5119, 5120, 5121, 8192])
def test_permutation_either_side_of_the_one_block_form(cuda, pkg, n):
    """A stable sort by expert id, whole numbers: sizes around whole steps of its warps and around its largest, 5,120."""
    torch = cuda
    ids = np.random.default_rng(n).integers(0, 256, size=n).astype(np.int32)
    ids[: n // 3] = 77                                               # more of one expert than a warp's share holds
    order, position = (torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    counts, offsets = (torch.full((k,), -1, dtype=torch.int32, device="cuda") for k in (256, 257))
    pkg.moe_permute_static(torch.from_numpy(ids).cuda(), order, position, counts, offsets)
    want = np.argsort(ids, kind="stable")
    assert np.array_equal(order.cpu().numpy(), want)
    assert np.array_equal(position.cpu().numpy()[want], np.arange(n))
    assert np.array_equal(counts.cpu().numpy(), np.bincount(ids, minlength=256))
    assert np.array_equal(offsets.cpu().numpy(), np.concatenate([[0], np.cumsum(np.bincount(ids, minlength=256))]))
    assert pkg.moe_permute_static_status() == 0
