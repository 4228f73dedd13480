"""Sizes at which the large-batch gate/up kernel and the packed top-8 can go wrong.

The large-batch kernel works on 128-row token tiles of an expert; the fused decode kernel (up to 16 rows) computes the
same numbers with the weights on the other side of the MMA.  Products are exact in FP32 accumulation over the same
K order on both, so the rows of a large batch must equal the same rows sent through the decode kernel bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same_rows(torch, pkg, layer, bias, rows, probe):
    from p92moe_b200 import synth

    x = synth.make_activations(77, rows, rows)
    out = torch.full_like(x, float("nan"))
    plan = pkg.MoePlan(max_rows=rows)
    block = pkg.MoeBlock(layer.bank, layer.router_weight, bias, plan)
    block.run_moe_rows(x, out, rows)
    torch.cuda.synchronize()
    assert plan.status() == 0
    picked = x[probe].contiguous()
    small = torch.empty_like(picked)
    block.run_moe_rows(picked, small, len(probe))
    torch.cuda.synchronize()
    assert plan.status() == 0
    assert torch.equal(out[probe].view(torch.int16), small.view(torch.int16))
    assert torch.isfinite(out.float()).all()
    plan.close()


@pytest.mark.parametrize("rows", [33, 63, 64, 65, 127, 128, 129, 160, 255, 257, 1025])
def test_rows_of_a_large_batch_equal_the_decode_kernel(cuda, pkg, layer0, rows):
    torch = cuda
    # first, around the middle, and last rows; two or more of them, so the decode call uses the batched logits order
    probe = sorted({0, 1, rows // 3, rows // 2, rows - 2, rows - 1})
    _same_rows(torch, pkg, layer0, layer0.bias, rows, probe)
    # every token on the same eight experts: tiles of exactly `rows` rows, all other experts empty
    bias = layer0.bias.clone()
    bias[[0, 7, 31, 64, 128, 200, 254, 255]] += 4.0
    _same_rows(torch, pkg, layer0, bias, rows, probe)


@pytest.mark.parametrize("step", [2.0 ** -24, 2.0 ** -22, 2.0 ** -17, 2.0 ** -15])
def test_top8_orders_scores_that_are_equal_or_nearly_equal(cuda, pkg, step):
    """Zero logits make every sigmoid exactly 0.5, so the corrected scores are 0.5 + bias rounded once and the expected
    order is known: higher score first, equal scores by lower id.  The steps lie on both sides of what the selection's
    24-bit keys can tell apart (2^-16 for scores in [0.5, 1))."""
    torch = cuda
    rows = 64
    rng = np.random.default_rng(5)
    logits = torch.zeros((rows, 256), dtype=torch.float32, device="cuda")
    for trial in range(4):
        bias = (rng.integers(0, 40, size=256) * step).astype(np.float32)
        score = (np.float32(0.5) + bias).astype(np.float32)
        want = np.lexsort((np.arange(256), -score))[:8]
        ids = torch.empty((rows, 8), dtype=torch.int32, device="cuda")
        weights = torch.empty((rows, 8), dtype=torch.float32, device="cuda")
        pkg.router_top8_rows(logits, torch.from_numpy(bias).cuda(), ids, weights, rows)
        assert np.array_equal(ids.cpu().numpy(), np.tile(want, (rows, 1)).astype(np.int32))
        assert np.array_equal(weights.cpu().numpy(), np.full((rows, 8), 0.3125, np.float32))    # 0.5 * 2.5 / 4, exact


def test_decode_rows_equal_the_large_batch_at_both_gate_up_tiles(cuda, pkg, layer0):
    """The fused decode kernel takes half gate/up tiles up to three rows and whole ones above, in a build for 8 and one for 16
    rows: the first rows of a 64-row batch, sent alone, must come out with the batch's bits."""
    torch = cuda
    from p92moe_b200 import synth

    x = synth.make_activations(78, 0, 64)
    want = torch.empty_like(x)
    plan = pkg.MoePlan(max_rows=64)
    plan.set_path(plan.PATH_AUTO)
    block = pkg.MoeBlock(layer0.bank, layer0.router_weight, layer0.bias, plan)
    block.run_moe_rows(x, want, 64)
    for rows in (2, 3, 4, 5, 8, 9, 15, 16):
        for first in (0, 64 - rows):
            out = torch.full((rows, x.shape[1]), float("nan"), dtype=torch.bfloat16, device="cuda")
            block.run_moe_rows(x[first:first + rows], out, rows)
            torch.cuda.synchronize()
            assert plan.status() == 0 and plan.last_launches == 1
            assert torch.equal(out.view(torch.int16), want[first:first + rows].view(torch.int16)), rows
    plan.close()
