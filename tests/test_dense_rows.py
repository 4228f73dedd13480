"""The dense MLP of a few rows (its own pair of kernels) against the CPU oracle.

Row counts sit on both sides of the column count of the MMA (16), of the hand-over to the grouped kernels (after 9, 10 or 18
rows at these shapes) and of the hand-over to the large-batch ones (32);
shapes cover a K extent of the down product that its parts do not divide, fewer K blocks than parts, one part per tile
(hidden 4096 has 32 tiles for 148 SMs: 4 parts) and the model's own MLP.  Both products accumulate in FP32 over FP4
operands, so a result differs from the oracle's only where another order of the sums moves a SwiGLU value to the
neighbouring FP4 value: the 1e-2 of the block's parity bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(256, 512), (512, 1536), (2560, 1024), (4096, 512), (2560, 9216)]


def _u16(t):
    import torch

    return t.view(torch.int16).cpu().numpy().view(np.uint16)


def _dense_bank(torch, pkg, hidden, inter, generator):
    """A bank of one MLP with random weights, and per matrix the packed values, linear scales and alpha on the host."""
    entries, packed_np, scales_np, alphas = [], [], [], []
    for rows, cols in ((inter, hidden), (inter, hidden), (hidden, inter)):
        w = torch.empty((rows, cols), dtype=torch.float32, device="cuda").normal_(0, 0.02, generator=generator).to(torch.bfloat16)
        packed = torch.empty((rows, cols // 2), dtype=torch.uint8, device="cuda")
        linear = torch.empty((rows, cols // 16), dtype=torch.uint8, device="cuda")
        alpha = torch.empty(1, dtype=torch.float32, device="cuda")
        pkg.nvfp4_pack_weight(w, packed, linear, alpha)
        swizzled = torch.empty(pkg.nvfp4_swizzled_scale_bytes(rows, cols // 16), dtype=torch.uint8, device="cuda")
        pkg.nvfp4_swizzle_scales(linear, swizzled, rows, cols // 16)
        entries.append((packed, swizzled, alpha))
        packed_np.append(packed.cpu().numpy().reshape(-1))
        scales_np.append(linear.cpu().numpy().reshape(-1))
        alphas.append(float(alpha))
    bank = pkg.ExpertBank(entries, first_expert=0, local_experts=0, hidden=hidden, intermediate=inter)
    return bank, np.stack(packed_np), np.stack(scales_np), np.array(alphas, np.float32)


@pytest.mark.parametrize("hidden,inter", SHAPES)
def test_dense_few_rows_against_the_oracle(cuda, pkg, orc, hidden, inter):
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(hidden + inter)
    bank, packed, scales, alphas = _dense_bank(torch, pkg, hidden, inter, g)
    # the oracle is row by row, so one call at the largest size has every row's result
    most = 33 if inter < 9216 else 19
    x = torch.empty((most, hidden), dtype=torch.float32, device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)
    want = orc.bf16_to_f32(orc.dense_forward(_u16(x), packed, scales, alphas, hidden, inter))
    plan = pkg.MoePlan(max_rows=most, hidden=hidden, intermediate=inter)
    for rows in (1, 2, 9, 10, 11, 15, 16, 17, 18, 19, 20, 21, 31, 32, 33):
        if rows > most:
            continue
        out = torch.full((rows, hidden), float("nan"), dtype=torch.bfloat16, device="cuda")
        pkg.run_dense_rows(plan, bank, x[:rows].contiguous(), out, rows)
        first = out.clone()
        pkg.run_dense_rows(plan, bank, x[:rows].contiguous(), out, rows)
        torch.cuda.synchronize()
        assert plan.status() == 0
        assert torch.equal(first.view(torch.int16), out.view(torch.int16))      # the parts are added in a fixed order
        got = orc.bf16_to_f32(_u16(out))
        assert np.linalg.norm(got - want[:rows]) <= 1e-2 * np.linalg.norm(want[:rows]), rows
    plan.close()
    bank.close()


@pytest.mark.parametrize("hidden,inter", [(512, 1536), (768, 2048), (2560, 9216)])
def test_dense_large_batch_equals_its_rows_sent_a_few_at_a_time(cuda, pkg, hidden, inter):
    """The large-batch kernel cuts the items of its last round into pieces of 128 or 64 weight rows; 33 to 1,300 rows reach
    every width at one shape or another.  Both sides accumulate the same FP4 products in FP32, in another order, which at
    most moves a few SwiGLU values of a row to the neighbouring FP4 value.  One such value changes the row's results by
    about 1 / sqrt(intermediate) of their size, 0.026 at 1,536; the bound on a row's groups of 64 columns leaves room for four
    of them and is below what one wrong column in a group makes, sqrt(2 / 64) = 0.18."""
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(inter)
    bank = _dense_bank(torch, pkg, hidden, inter, g)[0]
    most = 1300
    x = torch.empty((most, hidden), device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)
    plan = pkg.MoePlan(max_rows=most, hidden=hidden, intermediate=inter)
    want = torch.empty_like(x)
    for r in range(0, most, 20):
        n = min(20, most - r)
        pkg.run_dense_rows(plan, bank, x[r:r + n], want[r:r + n], n)
    for rows in (21, 33, 64, 128, 129, 400, 640, 1300):
        out = torch.full((rows, hidden), float("nan"), dtype=torch.bfloat16, device="cuda")
        pkg.run_dense_rows(plan, bank, x[:rows], out, rows)
        torch.cuda.synchronize()
        assert plan.status() == 0
        got, ref = out.double(), want[:rows].double()
        assert float((got - ref).norm()) <= 1e-2 * float(ref.norm()), rows
        worst = (got - ref).view(rows, -1, 64).norm(dim=2) / ref.view(rows, -1, 64).norm(dim=2)
        assert float(worst.max()) <= 0.1, rows
    plan.close()
    bank.close()
