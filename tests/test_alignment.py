"""Rows that start off the boundary their kernel's loads need: refused on the host, or served where the kernel has a form
for them - never a fault."""
import pytest

pytestmark = pytest.mark.gpu

HIDDEN = 2560


def _off(torch, shape, dtype, elements=1):
    """A contiguous tensor whose first element lies `elements` behind an allocation's start."""
    n = 1
    for s in shape:
        n *= s
    return torch.zeros(n + elements, dtype=dtype, device="cuda")[elements:].view(shape)


def _refused(pkg, call, *args):
    with pytest.raises(pkg.P92Error) as err:
        call(*args)
    assert err.value.code == 1                                    # cudaErrorInvalidValue


def test_operators_refuse_rows_they_cannot_load(cuda, pkg):
    torch = cuda
    bf16, u8 = torch.bfloat16, torch.uint8
    x, w = torch.zeros((4, HIDDEN), dtype=bf16, device="cuda"), torch.zeros((256, HIDDEN), dtype=bf16, device="cuda")
    for rows in (2, 8, 9, 300):
        xs = torch.zeros((rows, HIDDEN), dtype=bf16, device="cuda")
        out = torch.zeros((rows, 256), dtype=torch.float32, device="cuda")
        _refused(pkg, pkg.bf16_gemm_f32, _off(torch, (rows, HIDDEN), bf16), w, out, rows)
        _refused(pkg, pkg.bf16_gemm_f32, xs, _off(torch, (256, HIDDEN), bf16), out, rows)
    packed, scales = torch.zeros((4, HIDDEN // 2), dtype=u8, device="cuda"), torch.zeros((4, HIDDEN // 16), dtype=u8, device="cuda")
    _refused(pkg, pkg.nvfp4_quantize, _off(torch, (4, HIDDEN), bf16), packed, scales, 4 * HIDDEN)
    _refused(pkg, pkg.nvfp4_quantize, x, _off(torch, (4, HIDDEN // 2), u8), scales, 4 * HIDDEN)
    alpha = torch.zeros(1, dtype=torch.float32, device="cuda")
    _refused(pkg, pkg.nvfp4_pack_weight, _off(torch, (4, HIDDEN), bf16), packed, scales, alpha)
    # one row of the single-token order is read element by element
    one = torch.full((1, 256), float("nan"), dtype=torch.float32, device="cuda")
    pkg.bf16_gemv_f32(_off(torch, (1, HIDDEN), bf16), w, one)
    assert bool((one == 0).all())


@pytest.mark.parametrize("rows", [1, 4, 13, 17, 33, 300])
def test_block_refuses_rows_it_cannot_load(cuda, pkg, layer0, rows):
    torch = cuda
    bf16 = torch.bfloat16
    plan = pkg.MoePlan(max_rows=rows)
    plan.set_path(plan.PATH_AUTO)
    block = pkg.MoeBlock(layer0.bank, layer0.router_weight, layer0.bias, plan)
    x, out = torch.zeros((rows, HIDDEN), dtype=bf16, device="cuda"), torch.zeros((rows, HIDDEN), dtype=bf16, device="cuda")
    _refused(pkg, block.run_moe_rows, _off(torch, (rows, HIDDEN), bf16), out, rows)
    _refused(pkg, block.run_moe_rows, x, _off(torch, (rows, HIDDEN), bf16), rows)
    router = _off(torch, (256, HIDDEN), bf16)
    _refused(pkg, pkg.MoeBlock(layer0.bank, router, layer0.bias, plan).run_moe_rows, x, out, rows)
    ids = torch.arange(8, dtype=torch.int32, device="cuda").expand(rows, 8).contiguous()
    gate, up = (torch.zeros((rows * 8, 1024), dtype=bf16, device="cuda") for _ in range(2))
    _refused(pkg, block.project_expert_gate_up, ids, _off(torch, (rows, HIDDEN), bf16), gate, up, rows)
    _refused(pkg, block.project_expert_down, ids, _off(torch, (rows * 8, 1024), bf16), torch.zeros((rows * 8, HIDDEN), dtype=bf16, device="cuda"), rows)
    # the block is as before after the refusals
    block.run_moe_rows(x, out, rows)
    assert plan.status() == 0 and not bool(out.any())
    plan.close()


@pytest.mark.parametrize("rows", [1, 4, 18, 19, 33, 300])
def test_dense_mlp_writes_rows_at_any_element(cuda, pkg, rows):
    torch = cuda
    from p92moe_b200 import synth

    raw = synth.make_raw_layer_batched(9, 0, experts=0, intermediate=9216)
    bank = pkg.ExpertBank(raw.entries(), 0, 0, HIDDEN, 9216)
    plan = pkg.MoePlan(rows, HIDDEN, 9216)
    x = synth.make_activations(9, rows, rows)
    want = torch.empty_like(x)
    pkg.run_dense_rows(plan, bank, x, want, rows)
    got = _off(torch, (rows, HIDDEN), torch.bfloat16)
    pkg.run_dense_rows(plan, bank, x, got, rows)
    assert plan.status() == 0
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    _refused(pkg, pkg.run_dense_rows, plan, bank, _off(torch, (rows, HIDDEN), torch.bfloat16), want, rows)
    plan.close()
    bank.close()


def test_bank_refuses_matrices_it_cannot_load(cuda, pkg):
    torch = cuda
    from p92moe_b200 import synth

    entries = list(synth.make_raw_layer_batched(9, 0, experts=0, hidden=512, intermediate=512).entries())
    weight, scales, alpha = entries[1]
    entries[1] = (_off(torch, tuple(weight.shape), torch.uint8), scales, alpha)
    with pytest.raises(pkg.P92Error) as err:
        pkg.ExpertBank(entries, 0, 0, 512, 512)
    assert err.value.code == 1
