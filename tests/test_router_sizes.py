"""The tensor-core router with exact repair, at the sizes where its kernels change, against the operators that keep the
reference's order of sums throughout (bf16_gemm_f32 and router_top8_rows, themselves held to the CPU oracle bit for bit)."""
import pytest

pytestmark = pytest.mark.gpu

# K in eight slices and a block per token up to 256 rows, a warp per token above; eight slices up to 512, then fewer
# (three from 1,153, two from 1,537) and none above 2,304 rows; tiles of 64 experts, of 128 from 4,737 and of 256 from 9,473
# rows on (148 SMs).  Ends of these ranges, and odd sizes inside them.
SIZES = [9, 17, 255, 256, 257, 300, 512, 513, 1025, 1152, 1153, 1200, 1536, 1537, 2304, 2305, 4736, 4737, 7001, 9000, 9472, 9473]


def _check(torch, pkg, block, rows, x, bias):
    plan, router = block.plan, block.router_weight
    logits = torch.empty((rows, 256), dtype=torch.float32, device="cuda")
    ids = torch.empty((rows, 8), dtype=torch.int32, device="cuda")
    weights = torch.empty((rows, 8), dtype=torch.float32, device="cuda")
    pkg.bf16_gemm_f32(x, router, logits, rows)
    pkg.router_top8_rows(logits, bias, ids, weights, rows)
    block.run_moe_rows(x, torch.empty_like(x), rows)
    views = plan.views(rows)
    assert plan.status() == 0
    assert torch.equal(views["expert_ids"], ids)
    assert torch.equal(views["expert_weights"], weights)
    picked = ids.long()
    assert torch.equal(torch.gather(views["logits"], 1, picked), torch.gather(logits, 1, picked))
    # the others may deviate by 2^-14 |x| |w| without a wrong choice; they stay 8 times inside that
    bound = 2.0 ** -14 * x.double().norm(dim=1, keepdim=True) * router.double().norm(dim=1)
    assert bool(((views["logits"].double() - logits.double()).abs() <= 0.125 * bound).all())


@pytest.mark.parametrize("rows", SIZES)
def test_router_of_the_block_equals_the_exact_operators(cuda, pkg, layer0, rows):
    torch = cuda
    from p92moe_b200 import synth

    plan = pkg.MoePlan(max_rows=rows)
    plan.set_path(plan.PATH_TENSOR_CORE)
    x = synth.make_activations(4500, rows, rows)
    for bias in (layer0.bias, torch.zeros_like(layer0.bias)):             # without a bias the scores lie closer together
        _check(torch, pkg, pkg.MoeBlock(layer0.bank, layer0.router_weight, bias, plan), rows, x, bias)
    plan.close()


def test_router_at_other_hidden_sizes(cuda, pkg):
    """Hidden sizes other than 2,560 take the form that reads token row and router rows in place; its shared memory
    grows with the size, so a larger plan behind a smaller one in the same process needs a higher limit."""
    torch = cuda
    from p92moe_b200 import synth

    for hidden, inter in ((256, 512), (512, 512), (1024, 512), (4096, 512)):
        bank = pkg.ExpertBank(synth.make_raw_layer_batched(11, 0, hidden=hidden, intermediate=inter).entries(), hidden=hidden,
                              intermediate=inter)
        router, bias = synth.make_router(11, 0, hidden=hidden)
        for rows in (9, 100, 257, 1200, 2305):
            plan = pkg.MoePlan(rows, hidden, inter)
            x = synth.make_activations(11, rows, rows, hidden=hidden)
            _check(torch, pkg, pkg.MoeBlock(bank, router, bias, plan), rows, x, bias)
            plan.close()
        bank.close()


@pytest.mark.parametrize("rows", [9, 17, 64, 257, 300, 2305])
@pytest.mark.parametrize("what", ["nan row", "infinite row", "six experts left", "nan bias", "infinite bias"])
def test_router_of_the_block_with_scores_that_are_no_numbers(cuda, pkg, layer0, rows, what):
    """Whatever a token holds, it names eight different experts, the ones that the exact operators name; and the other tokens
    of the batch are not touched by it."""
    torch = cuda
    from p92moe_b200 import synth

    x = synth.make_activations(4600, rows, rows)
    bias = layer0.bias.clone()
    odd = torch.zeros(rows, dtype=torch.bool, device="cuda")
    if what == "nan row":
        odd[::3] = True
        x[odd, 11] = float("nan")
    elif what == "infinite row":
        odd[1::3] = True
        x[odd, 11] = float("inf")
    elif what == "six experts left":
        bias[:250] = -float("inf")
    elif what == "nan bias":
        bias[[0, 5, 31, 40]] = float("nan")
    else:
        bias[77] = float("inf")
    plan = pkg.MoePlan(max_rows=rows)
    plan.set_path(plan.PATH_TENSOR_CORE)
    logits = torch.empty((rows, 256), dtype=torch.float32, device="cuda")
    ids = torch.empty((rows, 8), dtype=torch.int32, device="cuda")
    weights = torch.empty((rows, 8), dtype=torch.float32, device="cuda")
    pkg.bf16_gemm_f32(x, layer0.router_weight, logits, rows)
    pkg.router_top8_rows(logits, bias, ids, weights, rows)
    out = torch.zeros_like(x)
    block = pkg.MoeBlock(layer0.bank, layer0.router_weight, bias, plan)
    block.run_moe_rows(x, out, rows)
    views = plan.views(rows)
    assert plan.status() == 0
    assert torch.equal(views["expert_ids"], ids)
    ordered = ids.sort(dim=1).values
    assert int(ordered.min()) >= 0 and int(ordered.max()) <= 255 and bool((ordered[:, 1:] > ordered[:, :-1]).all())
    assert torch.equal(views["expert_weights"].nan_to_num(nan=-1.0), weights.nan_to_num(nan=-1.0))
    if bool(odd.any()):
        clean = torch.where(odd[:, None], torch.zeros_like(x), x)
        want = torch.zeros_like(x)
        block.run_moe_rows(clean, want, rows)
        assert torch.equal(out[~odd].view(torch.int16), want[~odd].view(torch.int16))
    plan.close()


def _uneven_case(torch, hidden, rows, seed):
    """Token rows whose columns are equal in pairs and router rows whose columns of a pair are opposite, the pairs anywhere: every
    logit is zero but for the rounding of its sums, which grows with the norm of the router row.  Experts 0 - 3 are taken by their bias, eight experts of norms
    far apart and eight of norm zero contend for the other four places, and each pair of sums in another order may rank
    them differently."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    half = torch.empty((256, hidden // 2), device="cuda").normal_(generator=g)
    scale = torch.zeros((256, 1), device="cuda")
    scale[100:108, 0] = 2.0 ** torch.arange(5, 13, device="cuda")
    router = (torch.cat([half, -half], 1) * scale).to(torch.bfloat16)
    bias = torch.full((256,), -1.0, device="cuda")
    bias[0:4] = 1.0
    bias[50:58] = 0.0
    bias[100:108] = 0.0
    x = torch.empty((rows, hidden // 2), device="cuda").normal_(generator=g).to(torch.bfloat16)
    columns = torch.randperm(hidden, generator=g, device="cuda")
    return router[:, columns].contiguous(), bias, torch.cat([x, x], 1)[:, columns].contiguous()


@pytest.mark.parametrize("hidden,rows", [(2560, 9), (2560, 100), (2560, 300), (2560, 4097), (1024, 100), (1024, 300)])
def test_router_rows_of_very_different_norms(cuda, pkg, layer0, hidden, rows):
    """How far an approximate logit may lie from the exact one depends on the norm of its own router row: an expert may only be
    left out for being behind the eight best by its own bound and theirs together."""
    torch = cuda
    from p92moe_b200 import synth

    router, bias, x = _uneven_case(torch, hidden, rows, 70 + rows)
    inter = 1024 if hidden == 2560 else 512
    bank = layer0.bank if hidden == 2560 else pkg.ExpertBank(
        synth.make_raw_layer_batched(11, 0, hidden=hidden, intermediate=inter).entries(), hidden=hidden, intermediate=inter)
    plan = pkg.MoePlan(rows, hidden, inter)
    plan.set_path(plan.PATH_TENSOR_CORE)
    _check(torch, pkg, pkg.MoeBlock(bank, router, bias, plan), rows, x, bias)
    plan.close()


@pytest.mark.parametrize("rows", [9, 300, 1000])
@pytest.mark.parametrize("whose", ["token", "expert"])
def test_router_with_a_norm_beyond_float(cuda, pkg, layer0, rows, whose):
    """Squares that overflow leave a bound of infinity, or of no number where the other norm is zero, and then nothing is known of
    that logit's deviation: the token is ranked by its exact scores all the same."""
    torch = cuda
    router, bias, x = _uneven_case(torch, 2560, rows, 90 + rows)
    if whose == "token":
        x[::2] *= 2.0 ** 66                        # most router rows are zero
    else:
        router[60] = torch.where(router[107] > 0, 1e30, -1e30)
        bias[60] = 0.5
        x[::2] = 0.0
    plan = pkg.MoePlan(rows)
    plan.set_path(plan.PATH_TENSOR_CORE)
    _check(torch, pkg, pkg.MoeBlock(layer0.bank, router, bias, plan), rows, x, bias)
    plan.close()


@pytest.mark.parametrize("above", [0, 1])
def test_router_either_side_of_a_block_per_token(cuda, pkg, layer0, above):
    """Up to four tokens per SM the repair has a block of four warps per token, above a warp."""
    torch = cuda
    from p92moe_b200 import synth

    rows = 4 * torch.cuda.get_device_properties(0).multi_processor_count + above
    plan = pkg.MoePlan(max_rows=rows)
    plan.set_path(plan.PATH_TENSOR_CORE)
    x = synth.make_activations(4700, rows, rows)
    for bias in (layer0.bias, torch.zeros_like(layer0.bias)):
        _check(torch, pkg, pkg.MoeBlock(layer0.bank, layer0.router_weight, bias, plan), rows, x, bias)
    plan.close()
