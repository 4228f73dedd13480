"""Routing that a model does not produce but a caller's arrays can hold: one expert several times in a token.

An expert then has more rows than the batch has tokens, so a small batch needs several of its 16- or 32-row token tiles for
one expert.  Every (row, slot) result depends on its row and its expert alone: the same rows in a batch of 64, which runs
in 64-row tiles, must give the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HIDDEN, INTER = 2560, 1024


def _patterns(torch, rows, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    one = torch.full((rows, 8), 7, dtype=torch.int32, device="cuda")
    two = one.clone()
    two[:, 3:] = 200
    few = torch.randint(0, 3, (rows, 8), generator=g, device="cuda").to(torch.int32)
    return {"one": one, "two": two, "few": few}


def _at_64_rows(torch, ids, rows):
    """The rows' ids followed by rows on other experts."""
    rest = torch.arange(8, 16, dtype=torch.int32, device="cuda").expand(64 - rows, 8)
    return torch.cat([ids, rest]).contiguous()


def _quantised(torch, pkg, x):
    n, width = x.shape
    packed = torch.empty((n, width // 2), dtype=torch.uint8, device="cuda")
    linear = torch.empty((n, width // 16), dtype=torch.uint8, device="cuda")
    pkg.nvfp4_quantize(x, packed, linear, n * width)
    tiled = torch.empty(pkg.nvfp4_swizzled_scale_bytes(n, width // 16), dtype=torch.uint8, device="cuda")
    pkg.nvfp4_swizzle_scales(linear, tiled, n, width // 16)
    return packed, tiled


def _table(torch, raw):
    table = np.array([[w.data_ptr(), s.data_ptr(), a.data_ptr()] for w, s, a in raw.entries()], dtype=np.uint64)
    return torch.from_numpy(table.view(np.int64)).cuda()


def _same_bits(torch, got, want):
    return torch.equal(got.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("pattern", ["one", "two", "few"])
@pytest.mark.parametrize("rows", [1, 2, 3, 5, 16, 17, 32])
def test_products_of_an_expert_that_a_token_names_several_times(cuda, pkg, layer0, rows, pattern):
    torch = cuda
    from p92moe_b200 import synth

    ids = _patterns(torch, rows, rows)[pattern]
    table = _table(torch, layer0.raw)
    x = synth.make_activations(81, rows, 64)
    h = torch.empty((64 * 8, INTER), device="cuda").normal_(0, 1, generator=torch.Generator(device="cuda").manual_seed(5)).to(torch.bfloat16)
    results = {}
    for n, these in ((rows, ids), (64, _at_64_rows(torch, ids, rows))):
        plan = pkg.MoePlan(max_rows=n)
        block = pkg.MoeBlock(layer0.bank, layer0.router_weight, layer0.bias, plan)
        out = [torch.full((n * 8, width), float("nan"), dtype=torch.bfloat16, device="cuda") for width in (INTER, INTER, HIDDEN) * 2]
        block.project_expert_gate_up(these, x[:n], out[0], out[1], n)
        block.project_expert_down(these, h[:n * 8], out[2], n)
        assert plan.status() == 0
        gate_up, down = pkg.GroupedPlan(n * 16, INTER, HIDDEN), pkg.GroupedPlan(n * 8, HIDDEN, INTER)
        gate_up.grouped_rows(*_quantised(torch, pkg, x[:n]), table, these, out[3], out[4], 0, n, False)
        down.grouped_rows(*_quantised(torch, pkg, h[:n * 8]), table, these, out[5], None, 2, n, True)
        assert gate_up.status() == 0 and down.status() == 0
        results[n] = out
        for p in (plan, gate_up, down):
            p.close()
    for got, want in zip(results[rows], results[64]):
        assert torch.isfinite(got.float()).all()
        assert _same_bits(torch, got, want[:rows * 8])
    for bank, in_place in zip(results[rows][:3], results[rows][3:]):
        assert _same_bits(torch, bank, in_place)


@pytest.mark.parametrize("rows", [4, 17, 32])
def test_rows_without_an_expert_are_counted_as_expert_0(cuda, pkg, layer0, rows):
    """Ids out of range are clamped and reported; a batch of nothing but padding rows is eight such ids a row."""
    torch = cuda
    from p92moe_b200 import synth

    x = synth.make_activations(82, rows, rows)
    plan = pkg.MoePlan(max_rows=rows)
    block = pkg.MoeBlock(layer0.bank, layer0.router_weight, layer0.bias, plan)
    outs = []
    for value in (0, -1):
        ids = torch.full((rows, 8), value, dtype=torch.int32, device="cuda")
        out = [torch.full((rows * 8, INTER), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
        block.project_expert_gate_up(ids, x, out[0], out[1], rows)
        assert plan.status() == (0 if value == 0 else 1)
        outs.append(out)
    for got, want in zip(outs[1], outs[0]):
        assert torch.isfinite(want.float()).all() and _same_bits(torch, got, want)
    plan.close()


@pytest.mark.parametrize("rows", [1, 2, 7, 16, 17, 33, 63, 64, 65])
def test_fronts_of_the_operators_on_a_callers_ids(cuda, pkg, layer0, rows):
    """Up to 64 rows one kernel counts, ranks and places, above two do; ids repeat within a token and leave the range.  Operators
    on the bank and on weights in place go through different forms of it and give the same bits, and so do a batch's rows
    and the same rows at the head of one of 72."""
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(rows)
    ids = torch.randint(-2, 258, (72, 8), generator=g, device="cuda").to(torch.int32)
    ids[::3, 4:] = 9                                              # an expert with more rows than the batch
    x = torch.empty((72, HIDDEN), device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)
    h = torch.empty((72 * 8, INTER), device="cuda").normal_(0, 1, generator=g).to(torch.bfloat16)
    table = _table(torch, layer0.raw)
    results = []
    for n in (rows, 72):
        plan = pkg.MoePlan(max_rows=n)
        block = pkg.MoeBlock(layer0.bank, layer0.router_weight, layer0.bias, plan)
        out = [torch.full((n * 8, width), float("nan"), dtype=torch.bfloat16, device="cuda") for width in (INTER, INTER, HIDDEN) * 2]
        these = ids[:n].contiguous()
        block.project_expert_gate_up(these, x[:n], out[0], out[1], n)
        block.project_expert_down(these, h[:n * 8], out[2], n)
        gate_up, down = pkg.GroupedPlan(n * 16, INTER, HIDDEN), pkg.GroupedPlan(n * 8, HIDDEN, INTER)
        gate_up.grouped_rows(*_quantised(torch, pkg, x[:n]), table, these, out[3], out[4], 0, n, False)
        down.grouped_rows(*_quantised(torch, pkg, h[:n * 8]), table, these, out[5], None, 2, n, True)
        bad = int(((these < 0) | (these > 255)).any())
        assert plan.status() == bad and gate_up.status() == bad and down.status() == bad
        results.append(out)
        for p in (plan, gate_up, down):
            p.close()
    for k in range(6):
        assert torch.isfinite(results[0][k].float()).all()
        assert _same_bits(torch, results[0][k], results[1][k][:rows * 8])
        assert _same_bits(torch, results[0][k], results[0][k % 3])
