"""Lists and places of the block's own routing, and batches in which a few experts have most of the tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [9, 31, 32, 33, 255, 511, 512, 513, 1024, 1025, 1030, 2049, 8192, 8193])
@pytest.mark.parametrize("popular", [0, 2])
def test_places_of_the_routed_rows(cuda, pkg, layer0, rows, popular):
    """The ranks come from chunks of 32 tokens, the sums over the chunks from every block, through spans of 512 tokens, up to 8,192
    rows and from a kernel of their own above; up to 1,024 rows a block has one token.  Either side of these sizes the
    permutation is the stable sort of the ids, bit for bit, and an expert's rows lie one behind the other from a multiple of
    128 on, the shared expert's last."""
    torch = cuda
    from p92moe_b200 import synth

    bias = layer0.bias.clone()
    bias[[3, 255][:popular]] += 4.0
    plan = pkg.MoePlan(max_rows=rows)
    plan.set_path(plan.PATH_TENSOR_CORE)
    x = synth.make_activations(91, rows, rows)
    pkg.MoeBlock(layer0.bank, layer0.router_weight, bias, plan).run_moe_rows(x, torch.empty_like(x), rows)
    views = {k: v.cpu().numpy() for k, v in plan.views(rows).items() if v is not None and v.dtype == torch.int32}
    assert plan.status() == 0
    plan.close()
    ids = views["expert_ids"].reshape(-1)
    want = np.argsort(ids, kind="stable")
    counts = np.bincount(ids, minlength=256)
    offsets = np.concatenate([[0], np.cumsum(counts)])
    assert np.array_equal(views["order"], want)
    assert np.array_equal(views["position"][want], np.arange(rows * 8))
    assert np.array_equal(views["counts"], counts)
    assert np.array_equal(views["offsets"], offsets)
    base = np.concatenate([[0], np.cumsum((counts + 127) // 128 * 128)])
    rank = views["position"] - offsets[ids]
    assert np.array_equal(views["mixed_index"][: rows * 8], base[ids] + rank)
    assert np.array_equal(views["mixed_index"][rows * 8:], base[256] + np.arange(rows))


@pytest.mark.parametrize("rows", [1024, 1025, 1153, 8193])
@pytest.mark.parametrize("popular", [[], [3, 255]])
def test_scales_stored_by_row(cuda, pkg, layer0, rows, popular):
    """Above 1,024 rows the token scales reach the gate/up product as 16 bytes per row and K block and are turned round there.
    The rows equal the same rows sent through the decode kernel, which has a layout of its own, bit for bit; the popular experts
    have several tiles, the others one with a ragged end."""
    torch = cuda
    from p92moe_b200 import synth

    bias = layer0.bias.clone()
    bias[popular] += 4.0
    x = synth.make_activations(92, rows, rows)
    out = torch.full_like(x, float("nan"))
    plan = pkg.MoePlan(max_rows=rows)
    block = pkg.MoeBlock(layer0.bank, layer0.router_weight, bias, plan)
    block.run_moe_rows(x, out, rows)
    assert plan.status() == 0 and torch.isfinite(out.float()).all()
    for first in (0, 120, rows - 16):
        small = torch.empty_like(x[:16])
        block.run_moe_rows(x[first:first + 16].contiguous(), small, 16)
        assert plan.status() == 0
        assert torch.equal(out[first:first + 16].view(torch.int16), small.view(torch.int16))
    plan.close()


@pytest.mark.parametrize("hidden,inter", [(256, 512), (512, 1024), (768, 512), (1024, 2048), (2816, 512), (4096, 1024)])
@pytest.mark.parametrize("rows", [33, 1025, 2305, 8200])
def test_block_at_other_shapes(cuda, pkg, orc, hidden, inter, rows):
    """Places, token scales and products at hidden sizes with one K block to sixteen and K extents of the down product with one
    chunk, two or four (the last beyond the form with the token rows in shared memory): the lists are the stable sort's,
    and the rows equal the same rows in batches of eight, which take other kernels throughout, bit for bit.  The first rows
    are held to the CPU oracle."""
    torch = cuda
    from p92moe_b200 import synth
    from conftest import u16

    raw = synth.make_raw_layer_batched(13, 0, hidden=hidden, intermediate=inter)
    bank = pkg.ExpertBank(raw.entries(), hidden=hidden, intermediate=inter)
    router, bias = synth.make_router(13, 0, hidden=hidden)
    bias[[3, 255]] += 4.0
    x = synth.make_activations(93, rows, rows, hidden=hidden)
    out = torch.full_like(x, float("nan"))
    plan = pkg.MoePlan(rows, hidden, inter)
    block = pkg.MoeBlock(bank, router, bias, plan)
    block.run_moe_rows(x, out, rows)
    assert plan.status() == 0
    views = {k: v.cpu().numpy() for k, v in plan.views(rows).items() if v is not None and v.dtype == torch.int32}
    ids = views["expert_ids"].reshape(-1)
    counts = np.bincount(ids, minlength=256)
    base = np.concatenate([[0], np.cumsum((counts + 127) // 128 * 128)])
    rank = np.empty(rows * 8, dtype=np.int64)
    rank[np.argsort(ids, kind="stable")] = np.concatenate([np.arange(c) for c in counts])
    assert np.array_equal(views["order"], np.argsort(ids, kind="stable"))
    assert np.array_equal(views["mixed_index"][: rows * 8], base[ids] + rank)
    assert np.array_equal(views["mixed_index"][rows * 8:], base[256] + np.arange(rows))
    for first in (0, 16, rows // 2, rows - 8):
        small = torch.empty_like(x[:8])
        block.run_moe_rows(x[first:first + 8].contiguous(), small, 8)
        assert plan.status() == 0
        assert torch.equal(out[first:first + 8].view(torch.int16), small.view(torch.int16))
    if rows == 33:
        want = orc.moe_forward(u16(x[:4]), u16(router), bias.cpu().numpy(), raw.packed.cpu().numpy(), raw.scales_linear.cpu().numpy(),
                               raw.alpha.cpu().numpy(), hidden, inter)
        got, want = out[:4].float().cpu().numpy(), orc.bf16_to_f32(want)
        assert np.linalg.norm(got - want) <= 1e-2 * np.linalg.norm(want)
    plan.close()
    bank.close()


def test_batch_of_more_rows_than_a_grid_has_in_y(cuda, pkg):
    """65,536 rows, with and without the norm behind the block: the bits of its two halves.  And the combine operator at as many."""
    torch = cuda
    from p92moe_b200 import synth

    hidden, inter, rows = 256, 512, 65536
    bank = pkg.ExpertBank(synth.make_raw_layer_batched(14, 0, hidden=hidden, intermediate=inter).entries(), hidden=hidden,
                          intermediate=inter)
    router, bias = synth.make_router(14, 0, hidden=hidden)
    x = synth.make_activations(94, 0, rows, hidden=hidden)
    weight = synth.make_activations(94, 1, 1, hidden=hidden).view(-1)
    plan = pkg.MoePlan(rows, hidden, inter)
    block = pkg.MoeBlock(bank, router, bias, plan)
    half = rows // 2
    for post in (None, weight):
        out, want = torch.full_like(x, float("nan")), torch.empty_like(x)
        block.run_moe_rows_normed(x, None, post, out, rows, 1e-5)
        for first in (0, half):
            block.run_moe_rows_normed(x[first:first + half], None, post, want[first:first + half], half, 1e-5)
        assert plan.status() == 0
        assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    plan.close()
    bank.close()
    g = torch.Generator(device="cuda").manual_seed(15)
    expert_rows = torch.empty((rows, 8, 24), device="cuda").normal_(generator=g).to(torch.bfloat16)
    weights = torch.empty((rows, 8), device="cuda").uniform_(generator=g)
    out, want = (torch.empty((rows, 24), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    pkg.expert_combine_rows(expert_rows, weights, out, rows, 8, 24)
    for first in (0, half):
        pkg.expert_combine_rows(expert_rows[first:], weights[first:], want[first:], half, 8, 24)
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))
