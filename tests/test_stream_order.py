"""A block may follow, on its stream and without a synchronisation, the kernel that produces its parameters.

The operators let the next kernel of the stream start before they have written their results, so a kernel that reads what the
caller owns - token rows, router rows, bias, norm weights - before it has waited for its predecessor sees old values."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "openpangu-2.0-flash-cuda-rocm_b200", "csrc")
REPEATS = 40


@pytest.mark.parametrize("source,kernel", [("decode_mega.cu", "moe_decode_kernel"), ("decode_ep.cu", "moe_decode_ep_kernel")])
def test_nothing_of_the_caller_is_read_before_the_wait(source, kernel):
    text = open(os.path.join(CSRC, source)).read()
    text = re.sub(r"//[^\n]*", "", text)
    body = text[re.search(r"__global__[^;{]*\b" + kernel + r"\(", text).end():]
    before = body[:body.index("pdl_wait();")]
    statements = [s for s in before.split(";") if "prefetch_l2(" not in s]          # a request to the L2 reads nothing
    used = [s.strip() for s in statements if re.search(r"\bp\.(x|router_w|bias|pre_norm_w|post_norm_w)\b", s)]
    assert used == []


def _parameter_sets(torch, layer):
    """Two routers, biases and norm weights that an operator makes from what lies in `start`, each far from the other."""
    g = torch.Generator(device="cuda").manual_seed(3)
    steps = [torch.empty_like(layer.router_weight, dtype=torch.float32).normal_(0, 0.02, generator=g).to(torch.bfloat16)
             for _ in range(2)]
    vectors = [torch.empty((1, 128), device="cuda").normal_(0, 0.1, generator=g).to(torch.bfloat16) for _ in range(2)]
    matrix = torch.empty((256, 128), device="cuda").normal_(0, 0.1, generator=g).to(torch.bfloat16)
    norm_steps = [torch.empty(2560, device="cuda").normal_(0, 0.5, generator=g).to(torch.bfloat16) for _ in range(2)]
    return steps, vectors, matrix, norm_steps


def _compare(torch, produce_and_run, shape):
    """produce_and_run(k, out) with parameter set k: results without any synchronisation against synchronised ones."""
    want = []
    for k in range(2):
        out = torch.zeros(shape, dtype=torch.bfloat16, device="cuda")
        produce_and_run(k, out, torch.cuda.synchronize)
        torch.cuda.synchronize()
        want.append(out)
    assert not torch.equal(want[0], want[1])
    outs = [torch.zeros(shape, dtype=torch.bfloat16, device="cuda") for _ in range(2 * REPEATS)]
    torch.cuda.synchronize()
    for i, out in enumerate(outs):
        produce_and_run(i & 1, out, lambda: None)
    torch.cuda.synchronize()
    for i, out in enumerate(outs):
        assert torch.equal(out.view(torch.int16), want[i & 1].view(torch.int16)), i


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["router", "bias", "pre", "post"])
@pytest.mark.parametrize("rows", [1, 4, 13, 33])
def test_block_behind_the_operator_that_makes_its_parameters(cuda, pkg, layer0, rows, what):
    torch = cuda
    from p92moe_b200 import synth

    steps, vectors, matrix, norm_steps = _parameter_sets(torch, layer0)
    x = synth.make_activations(91, rows, rows)
    plan = pkg.MoePlan(max_rows=rows)
    router, bias = layer0.router_weight.clone(), layer0.bias.clone()
    norm = torch.ones(2560, dtype=torch.bfloat16, device="cuda")
    block = pkg.MoeBlock(layer0.bank, router, bias, plan)

    def produce_and_run(k, out, synchronise):
        if what == "router":
            router.copy_(layer0.router_weight)
            pkg.add_inplace(router, steps[k], router.numel())
        elif what == "bias":
            pkg.bf16_gemv_f32(vectors[k], matrix, bias)
        else:
            norm.fill_(1.0)
            pkg.add_inplace(norm, norm_steps[k], norm.numel())
        synchronise()
        if what in ("pre", "post"):
            block.run_moe_rows_normed(x, norm if what == "pre" else None, norm if what == "post" else None, out, rows)
        else:
            block.run_moe_rows(x, out, rows)

    _compare(torch, produce_and_run, x.shape)
    assert plan.status() == 0
    plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["router", "bias"])
def test_expert_parallel_kernel_behind_the_operator_that_makes_its_parameters(cuda, pkg, layer0, what):
    """One GPU that owns all experts: the kernel's exchange goes through its own window."""
    torch = cuda
    from p92moe_b200 import ep, synth

    steps, vectors, matrix, _ = _parameter_sets(torch, layer0)
    x = synth.make_activations(92, 0, 4)
    plan = pkg.MoePlan(max_rows=32)
    router, bias = layer0.router_weight.clone(), layer0.bias.clone()
    window = ep.EpWindow(0, 1, 8)

    def produce_and_run(k, out, synchronise):
        if what == "router":
            router.copy_(layer0.router_weight)
            pkg.add_inplace(router, steps[k], router.numel())
        else:
            pkg.bf16_gemv_f32(vectors[k], matrix, bias)
        synchronise()
        ep.forward_fused(window, plan, layer0.bank, router, bias, x, out, 4)

    try:
        _compare(torch, produce_and_run, x.shape)
        assert plan.status() == 0
    finally:
        window.close()
        plan.close()
