"""The work that users of this package have it do, as cases to time.

Every case goes through the package's public entry points as an engine calls them, one call per layer and step:

  block   the MoE block of a few layers: `MoeBlock.run_moe_rows`, `run_moe_rows_normed` (the RMSNorms either side of
          the block folded in) or `run_moe_rows_host_async` + `MoePlan.host_flush` (token rows in pinned host memory);
  dense   the dense SwiGLU MLP of the model's first two layers: `run_dense_rows`;
  stages  the routed experts operator by operator, the way an executor that keeps its own call sequence does it: router
          logits, top-8, quantise, tile the scales, grouped gate/up product, SwiGLU, quantise, tile, grouped down
          product, combine - on weights left in place (`GroupedPlan.grouped_rows`) or on a bank
          (`MoeBlock.project_expert_gate_up` / `project_expert_down`).

Sizes are the model's: hidden 2560, 256 routed experts of 1024 and one shared expert, top-8, dense MLP 9216.  Layers are
independent weight sets, so a step's weights are not left in the L2 cache by the step before; every layer has token rows
of its own, because attention sits between two MoE blocks.  Weights and inputs are synthetic, with the distributions
of `synth.py`.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package of the tree in the working folder (its directory name is not an identifier)."""
    if "p92moe_b200" not in sys.modules:
        here = next(p for p in (os.getcwd(), ROOT) if os.path.isdir(os.path.join(p, "openpangu-2.0-flash-cuda-rocm_b200")))
        folder = os.path.join(here, "openpangu-2.0-flash-cuda-rocm_b200")
        spec = importlib.util.spec_from_file_location("p92moe_b200", os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        module = importlib.util.module_from_spec(spec)
        sys.modules["p92moe_b200"] = module
        spec.loader.exec_module(module)
    return sys.modules["p92moe_b200"]


pkg = _package()
from p92moe_b200 import synth  # noqa: E402

HIDDEN, INTER, EXPERTS, TOP = pkg.HIDDEN, pkg.INTERMEDIATE, pkg.EXPERTS, pkg.TOP_K
DENSE_INTER = 9216
EXPERT_BYTES = 3 * INTER * HIDDEN * 9 // 16          # E2M1 values and one E4M3 scale per 16 of them
ROUTER_BYTES = EXPERTS * HIDDEN * 2 + EXPERTS * 4
PLAN_ROWS = 64                                       # the engine's prefill block; larger batches get a plan of their size


def _block(name, rows, layers, norms="none", host=False, bias="normal", alpha=0.0):
    return {"name": name, "kind": "block", "rows": rows, "layers": layers, "norms": norms, "host": host, "bias": bias,
            "alpha": alpha}


def listed():
    return [
        # plain decoding of one sequence, eight layers of a step: the smallest call, all latency and weight streaming
        _block("decode_t1", 1, 8),
        # the verify step of speculative decoding (one token and three drafts), the engine's usual decode call
        _block("decode_t4", 4, 8),
        # the same for a host-resident caller: token rows travel to and from pinned memory at every layer
        _block("decode_t4_host", 4, 8, host=True),
        # a few sequences decoded together, with the two norms of the call site folded in
        _block("batch_t13_normed", 13, 4, norms="both"),
        # one block of the engine's prefill loop
        _block("block_t64", 64, 4),
        # batched serving: 128 sequences x 4 positions, some experts much more popular than others
        _block("serve_t512_zipf", 512, 2, bias="zipf", alpha=1.0),
        # a whole prompt at once, ragged, with both norms
        _block("prompt_t3807_normed", 3807, 1, norms="both"),
        # a prefill chunk with skewed routing
        _block("prefill_t4096_zipf", 4096, 1, bias="zipf", alpha=1.2),
        # the largest prefill chunk, even routing
        _block("prefill_t16384", 16384, 1, bias="zero"),
        # the two dense layers of the model, verify step and prompt
        {"name": "dense_t4", "kind": "dense", "rows": 4, "layers": 2},
        {"name": "dense_t3807", "kind": "dense", "rows": 3807, "layers": 2},
        # an executor that keeps its own sequence of operator calls, on weights left in place, at the verify step
        {"name": "stages_t4", "kind": "stages", "rows": 4, "layers": 4, "in_place": True},
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "serve", "serve", "prefill", "prefill", "dense", "stages"])
    if kind == "dense":
        return {"kind": "dense", "rows": _log_uniform(rng, 1, 4096), "layers": 2}
    if kind == "stages":
        return {"kind": "stages", "rows": _log_uniform(rng, 1, 64), "layers": rng.randint(2, 4),
                "in_place": rng.random() < 0.5}
    if kind == "decode":
        rows, layers = rng.randint(1, 16), rng.randint(4, 8)
    elif kind == "serve":
        rows, layers = _log_uniform(rng, 17, 1024), rng.randint(1, 3)
    else:
        rows, layers = _log_uniform(rng, 1025, 16384), 1
    host = kind == "decode" and rng.random() < 0.25
    norms = "none" if host else rng.choice(["none", "none", "both", "pre", "post"])
    bias = rng.choice(["normal", "zero"] if kind == "decode" else ["normal", "zero", "zipf"])
    case = _block("", rows, layers, norms, host, bias, round(rng.uniform(1.0, 1.2), 2) if bias == "zipf" else 0.0)
    del case["name"]
    return case


def _router(case, seed, layer):
    """Router weight and correction bias of one layer."""
    router, bias = synth.make_router(seed, layer, bias_std=0.0 if case.get("bias") == "zero" else 0.01)
    if case.get("bias") == "zipf":
        bias, _ = synth.fit_zipf_bias(router, case["alpha"], seed + layer, sample_rows=4096)
    return router, bias.contiguous()


def _bank(seed, layer):
    return pkg.ExpertBank(synth.make_raw_layer_batched(seed, layer).entries())


def _norm_weight(seed, layer):
    g = torch.Generator(device="cuda").manual_seed(seed * 131 + layer)
    return torch.empty(HIDDEN, device="cuda").normal_(1.0, 0.1, generator=g).to(torch.bfloat16)


def prepare(case, seed):
    rows, layers = case["rows"], case["layers"]
    state = {"case": case, "rows": rows}
    if case["kind"] == "dense":
        state["x"] = [synth.make_activations(seed, l, rows) for l in range(layers)]
        state["out"] = [torch.empty_like(x) for x in state["x"]]
        # one matrix triple of an MLP is drawn and quantised like an expert's of that width
        raws = [synth.make_raw_layer_batched(seed, l, experts=0, intermediate=DENSE_INTER) for l in range(layers)]
        state["banks"] = [pkg.ExpertBank(r.entries(), 0, 0, HIDDEN, DENSE_INTER) for r in raws]
        state["plan"] = pkg.MoePlan(max(PLAN_ROWS, rows), HIDDEN, DENSE_INTER)
        return state
    state["x"] = [synth.make_activations(seed, l, rows) for l in range(layers)]
    if case["kind"] == "stages":
        return _prepare_stages(state, seed)
    state["plan"] = pkg.MoePlan(max(PLAN_ROWS, rows))
    state["blocks"] = [pkg.MoeBlock(_bank(seed, l), *_router(case, seed, l), state["plan"]) for l in range(layers)]
    if case["norms"] != "none":
        state["pre"] = [_norm_weight(seed, l) if case["norms"] in ("both", "pre") else None for l in range(layers)]
        state["post"] = [_norm_weight(seed + 1, l) if case["norms"] in ("both", "post") else None for l in range(layers)]
    if case["host"]:
        state["x"] = [x.cpu().pin_memory() for x in state["x"]]
        state["out"] = [torch.empty_like(x).pin_memory() for x in state["x"]]
    else:
        state["out"] = [torch.empty_like(x) for x in state["x"]]
    return state


def _prepare_stages(state, seed):
    case, rows, layers = state["case"], state["rows"], state["case"]["layers"]

    def new(n, dtype):
        return torch.empty(n, dtype=dtype, device="cuda")

    # scratch that an executor reserves once and uses for every layer
    state["scratch"] = {
        "logits": new((rows, EXPERTS), torch.float32), "ids": new((rows, TOP), torch.int32),
        "weights": new((rows, TOP), torch.float32),
        "xq": new((rows, HIDDEN // 2), torch.uint8), "xs": new((rows, HIDDEN // 16), torch.uint8),
        "xt": new(pkg.nvfp4_swizzled_scale_bytes(rows, HIDDEN // 16), torch.uint8),
        "gate": new((rows * TOP, INTER), torch.bfloat16), "up": new((rows * TOP, INTER), torch.bfloat16),
        "hq": new((rows * TOP, INTER // 2), torch.uint8), "hs": new((rows * TOP, INTER // 16), torch.uint8),
        "ht": new(pkg.nvfp4_swizzled_scale_bytes(rows * TOP, INTER // 16), torch.uint8),
        "down": new((rows * TOP, HIDDEN), torch.bfloat16),
    }
    state["router"], state["bias"] = zip(*[_router(case, seed, l) for l in range(layers)])
    state["out"] = [torch.empty_like(x) for x in state["x"]]
    if case["in_place"]:
        state["raw"] = [synth.make_raw_layer_batched(seed, l) for l in range(layers)]
        state["table"] = []
        for raw in state["raw"]:
            table = np.array([[w.data_ptr(), s.data_ptr(), a.data_ptr()] for w, s, a in raw.entries()], dtype=np.uint64)
            state["table"].append(torch.from_numpy(table.view(np.int64)).cuda())
        state["gate_up_plan"] = pkg.GroupedPlan(rows * 2 * TOP, INTER, HIDDEN)
        state["down_plan"] = pkg.GroupedPlan(rows * TOP, HIDDEN, INTER)
    else:
        state["plan"] = pkg.MoePlan(max(PLAN_ROWS, rows))
        state["blocks"] = [pkg.MoeBlock(_bank(seed, l), state["router"][l], state["bias"][l], state["plan"])
                           for l in range(layers)]
    return state


def _run_stages(state):
    rows, s = state["rows"], state["scratch"]
    for l, (x, out) in enumerate(zip(state["x"], state["out"])):
        if rows == 1:
            pkg.bf16_gemv_f32(x, state["router"][l], s["logits"])
        else:
            pkg.bf16_gemm_f32(x, state["router"][l], s["logits"], rows)
        pkg.router_top8_rows(s["logits"], state["bias"][l], s["ids"], s["weights"], rows)
        if state["case"]["in_place"]:
            pkg.nvfp4_quantize(x, s["xq"], s["xs"], rows * HIDDEN)
            pkg.nvfp4_swizzle_scales(s["xs"], s["xt"], rows, HIDDEN // 16)
            state["gate_up_plan"].grouped_rows(s["xq"], s["xt"], state["table"][l], s["ids"], s["gate"], s["up"], 0, rows, False)
            pkg.swiglu(s["gate"], s["up"], s["gate"], rows * TOP * INTER)
            pkg.nvfp4_quantize(s["gate"], s["hq"], s["hs"], rows * TOP * INTER)
            pkg.nvfp4_swizzle_scales(s["hs"], s["ht"], rows * TOP, INTER // 16)
            state["down_plan"].grouped_rows(s["hq"], s["ht"], state["table"][l], s["ids"], s["down"], None, 2, rows, True)
        else:
            state["blocks"][l].project_expert_gate_up(s["ids"], x, s["gate"], s["up"], rows)
            pkg.swiglu(s["gate"], s["up"], s["gate"], rows * TOP * INTER)
            state["blocks"][l].project_expert_down(s["ids"], s["gate"], s["down"], rows)
        pkg.expert_combine_rows(s["down"], s["weights"], out, rows, TOP, HIDDEN)
    return state["out"]


def run(state):
    case, rows = state["case"], state["rows"]
    if case["kind"] == "stages":
        return _run_stages(state)
    if case["kind"] == "dense":
        for bank, x, out in zip(state["banks"], state["x"], state["out"]):
            pkg.run_dense_rows(state["plan"], bank, x, out, rows)
    elif case["host"]:
        for block, x, out in zip(state["blocks"], state["x"], state["out"]):
            block.run_moe_rows_host_async(x, out, rows)
        state["plan"].host_flush()
    elif case["norms"] != "none":
        for block, x, out, pre, post in zip(state["blocks"], state["x"], state["out"], state["pre"], state["post"]):
            block.run_moe_rows_normed(x, pre, post, out, rows)
    else:
        for block, x, out in zip(state["blocks"], state["x"], state["out"]):
            block.run_moe_rows(x, out, rows)
    return state["out"]


def _distinct(case):
    """Routed experts that a batch is expected to hit: an expert with share s of the assignments gets a given token with
    probability 8 s."""
    if case.get("bias") == "zipf":
        share = synth.zipf_target(case["alpha"], 0).double().numpy()
    else:
        share = np.full(EXPERTS, 1.0 / EXPERTS)
    return float((1.0 - (1.0 - np.minimum(1.0, TOP * share)) ** case["rows"]).sum())


def work(case):
    rows, layers = case["rows"], case["layers"]
    token_bytes = rows * HIDDEN * 2 * 2
    if case["kind"] == "dense":
        return {"bytes": layers * (3 * DENSE_INTER * HIDDEN * 9 / 16 + token_bytes),
                "flops": layers * 2.0 * 3 * DENSE_INTER * HIDDEN * rows}
    shared = 0 if case["kind"] == "stages" else 1
    norm_bytes = 2 * HIDDEN * {"none": 0, "both": 2}.get(case.get("norms", "none"), 1)
    return {"bytes": layers * ((_distinct(case) + shared) * EXPERT_BYTES + ROUTER_BYTES + token_bytes + norm_bytes),
            "flops": layers * 2.0 * rows * (3 * INTER * HIDDEN * (TOP + shared) + EXPERTS * HIDDEN)}


def tolerance(case):
    # BF16 outputs of two chained FP4 products: a different FP32 summation order moves some SwiGLU values to the
    # neighbouring FP4 value, which is the 1e-2 that the block's parity with the reference is held to
    return {"rel": 1e-2}
