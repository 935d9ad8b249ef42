"""The layer calls by which this library's speed is judged: one MoE expert layer, from bf16 activations and the router's
choice to the bf16 output, through the public entry points, at the shard shapes and batch sizes that serving meets.

Shapes are those of configs/ and bench.py: the DeepSeek-V3 TP8 shard ("tp8"), the Qwen3-Next TP2 shard ("qwen3") and the
unsharded DeepSeek-V3 layer ("full").  Three ways of calling are in use:

  graph   fused_experts_impl captured once into a CUDA graph, a decode step replays it (how engines run decode batches)
  layer   fused_experts_impl called eagerly (prefill, and decode without graphs)
  steps   the call-site sequence spelled out: quantise, block schedule, zeroed output, the operator
"""
import math
import os

import torch

import alpha_moe_ops
from alpha_moe_b200.layer import fused_experts_impl
from alpha_moe_b200.prologue import moe_align_block_size, per_token_group_quant_fp8
from alpha_moe_b200.utils import get_best_config, interleave_tensor

# experts (the last one shared and always chosen where `shared`), hidden size, intermediate size on this GPU, experts per
# token (counting the shared one), routed scaling factor, knob table (the unsharded layer has none of its own: it takes
# the one of the same hidden size)
SHAPES = {
    "tp8": dict(e=257, k=7168, i=256, top_k=9, scaling=2.5, shared=True, table="moe_b200_E257_I256_K7168.json"),
    "qwen3": dict(e=512, k=2048, i=256, top_k=10, scaling=1.0, shared=False, table="moe_b200_E512_I256_K2048.json"),
    "full": dict(e=257, k=7168, i=2048, top_k=9, scaling=2.5, shared=True, table="moe_b200_E257_I256_K7168.json"),
}
CONFIGS = os.path.join(os.getcwd(), "configs")
MAX_TOKENS = {"tp8": 8192, "qwen3": 8192, "full": 4096}
GRAPH_MAX_TOKENS = 256      # engines capture decode batches up to about this size


def listed():
    return [
        # one user: latency and launches are all there is; eagerly, and as decode runs it
        {"name": "tp8_m1_layer", "shape": "tp8", "tokens": 1, "call": "layer", "routing": "logits"},
        {"name": "tp8_m1_graph", "shape": "tp8", "tokens": 1, "call": "graph", "routing": "logits"},
        # one user with speculative tokens, or a handful of users
        {"name": "tp8_m5_graph", "shape": "tp8", "tokens": 5, "call": "graph", "routing": "logits"},
        {"name": "qwen3_m3_graph", "shape": "qwen3", "tokens": 3, "call": "graph", "routing": "logits"},
        # decode batches: every token brings new experts, the weight stream decides
        {"name": "tp8_m24_graph", "shape": "tp8", "tokens": 24, "call": "graph", "routing": "logits"},
        {"name": "qwen3_m96_graph", "shape": "qwen3", "tokens": 96, "call": "graph", "routing": "logits"},
        {"name": "tp8_m203_graph", "shape": "tp8", "tokens": 203, "call": "graph", "routing": "logits"},
        # a ragged rest of a chunked prefill
        {"name": "tp8_m777_layer", "shape": "tp8", "tokens": 777, "call": "layer", "routing": "logits"},
        # prefill chunks: bench.py's headline batch, the small shape, the skewed batch of bench.py, the unsharded layer
        {"name": "tp8_m4096_steps", "shape": "tp8", "tokens": 4096, "call": "steps", "routing": "logits"},
        {"name": "qwen3_m4096_layer", "shape": "qwen3", "tokens": 4096, "call": "layer", "routing": "logits"},
        {"name": "tp8_m8192_zipf_layer", "shape": "tp8", "tokens": 8192, "call": "layer", "routing": "zipf"},
        {"name": "full_m4096_layer", "shape": "full", "tokens": 4096, "call": "layer", "routing": "logits"},
    ]


def draw(rng):
    shape = rng.choices(["tp8", "qwen3", "full"], weights=[5, 3, 2])[0]
    tokens = round(math.exp(rng.uniform(0.0, math.log(MAX_TOKENS[shape]))))
    if tokens <= GRAPH_MAX_TOKENS:
        call = rng.choices(["graph", "layer", "steps"], weights=[6, 1, 1])[0]
    else:
        call = rng.choices(["layer", "steps"], weights=[2, 1])[0]
    routing = rng.choices(["logits", "zipf"], weights=[3, 1])[0]
    return {"shape": shape, "tokens": tokens, "call": call, "routing": routing}


def _block_quant(rows, cols, experts, gen):
    """fp8 weights [experts, rows, cols] with 128 x 128 block scales, from N(0, 0.02) values."""
    v = torch.randn(experts, rows // 128, 128, cols // 128, 128, generator=gen, device="cuda").mul_(0.02)
    s = v.abs().amax(dim=(2, 4)).div_(448.0)
    q = v.div_(s[:, :, None, :, None]).clamp_(-448.0, 448.0).to(torch.float8_e4m3fn)
    return q.view(experts, rows, cols), s


def _weights(sh, gen):
    """w [E, 2I, K] in the operator's gate/up interleave, its scales, w2 [E, K, I], its scales."""
    e, k, i = sh["e"], sh["k"], sh["i"]
    w = torch.empty(e, 2 * i, k, dtype=torch.float8_e4m3fn, device="cuda")
    w2 = torch.empty(e, k, i, dtype=torch.float8_e4m3fn, device="cuda")
    ws, w2s = [], []
    step = max(1, (1 << 28) // (2 * i * k))
    for lo in range(0, e, step):
        n = min(step, e - lo)
        q, s = _block_quant(2 * i, k, n, gen)
        w[lo:lo + n] = interleave_tensor(q.view(torch.uint8), 8).view(torch.float8_e4m3fn)
        ws.append(interleave_tensor(s, 1))
        q, s = _block_quant(k, i, n, gen)
        w2[lo:lo + n] = q
        w2s.append(s)
    return w, torch.cat(ws), w2, torch.cat(w2s).contiguous()


def _zipf_law(sh):
    """bench.py's skewed routing: Zipf(1.2) over all but 16 of the routed experts."""
    n = (sh["e"] - 1 if sh["shared"] else sh["e"]) - 16
    p = 1.0 / torch.arange(1, n + 1, dtype=torch.float64) ** 1.2
    return (p / p.sum()).float()


def _route(sh, tokens, routing, gen):
    """topk_ids int32 and topk_weights f32, [tokens, top_k]."""
    routed = sh["e"] - 1 if sh["shared"] else sh["e"]
    k = sh["top_k"] - 1 if sh["shared"] else sh["top_k"]
    if routing == "zipf":
        ids = torch.multinomial(_zipf_law(sh).cuda().expand(tokens, -1), k, replacement=False, generator=gen)
        wts = torch.softmax(torch.randn(tokens, k, generator=gen, device="cuda"), -1)
    else:
        vals, ids = torch.topk(torch.randn(tokens, routed, generator=gen, device="cuda"), k, dim=-1)
        wts = torch.softmax(vals, -1)
    ids = ids.to(torch.int32)
    if sh["shared"]:
        ids = torch.cat([ids, torch.full((tokens, 1), sh["e"] - 1, dtype=torch.int32, device="cuda")], 1)
        wts = torch.cat([wts, torch.ones(tokens, 1, device="cuda")], 1)
    return ids.contiguous(), wts.contiguous()


def prepare(case, seed):
    sh = SHAPES[case["shape"]]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    st = {"sh": sh, "call": case["call"], "table": os.path.join(CONFIGS, sh["table"]), "weights": _weights(sh, gen)}
    st["ids"], st["wts"] = _route(sh, case["tokens"], case["routing"], gen)
    st["x"] = torch.randn(case["tokens"], sh["k"], generator=gen, device="cuda").to(torch.bfloat16)
    st["hidden"] = torch.empty_like(st["x"])
    if case["call"] == "graph":
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _layer(st)
        torch.cuda.current_stream().wait_stream(side)
        st["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st["graph"]):
            _layer(st)
    return st


def _layer(st):
    """The layer works in place: its activations are the copy of the residual stream that the layer before it would leave."""
    w, ws, w2, w2s = st["weights"]
    st["hidden"].copy_(st["x"])
    return fused_experts_impl(st["hidden"], w, ws, w2, w2s, st["wts"], st["ids"], st["sh"]["scaling"], config=st["table"])


def _steps(st):
    w, ws, w2, w2s = st["weights"]
    sh, x = st["sh"], st["x"]
    conf = get_best_config(st["table"], x.shape[0])
    xq, xs = per_token_group_quant_fp8(x)
    sid, eid, npp = moe_align_block_size(st["ids"], conf["block_m"], sh["e"])
    return alpha_moe_ops.fused_moe_w8a8_up_down(xq, xs, w, ws, w2, w2s, sid, eid, npp, st["wts"], torch.zeros_like(x),
                                                sh["top_k"], conf["block_m"], conf["block_n"], conf["warp_n"],
                                                conf["stages"], sh["scaling"])


def run(state):
    if state["call"] == "graph":
        state["graph"].replay()
        return state["hidden"]
    return _layer(state) if state["call"] == "layer" else _steps(state)


def _active_experts(case):
    """Experts that a batch is expected to reach."""
    sh, m = SHAPES[case["shape"]], case["tokens"]
    k = sh["top_k"] - 1 if sh["shared"] else sh["top_k"]
    if case["routing"] == "zipf":
        # k draws without replacement hit expert j with probability 1 - exp(-c p_j), c such that k are hit on average
        p = _zipf_law(sh).double()
        lo, hi = 0.0, 1e6
        for _ in range(60):
            c = 0.5 * (lo + hi)
            lo, hi = (c, hi) if float((1 - torch.exp(-c * p)).sum()) < k else (lo, c)
        routed = float((1 - torch.exp(-c * m * p)).sum())
    else:
        n = sh["e"] - 1 if sh["shared"] else sh["e"]
        routed = n * (1.0 - (1.0 - k / n) ** m)
    return routed + (1 if sh["shared"] else 0)


def work(case):
    """fp8 weights and fp32 block scales of the experts reached, bf16 activations in, routing, bf16 output."""
    sh, m = SHAPES[case["shape"]], case["tokens"]
    k, i = sh["k"], sh["i"]
    expert = 3 * i * k + 4 * 3 * (i // 128) * (k // 128)
    return {"bytes": _active_experts(case) * expert + 4.0 * m * k + 8.0 * m * sh["top_k"],
            "flops": 6.0 * m * sh["top_k"] * i * k}


def tolerance(case):
    # bf16 output, summed over the experts in any order by bf16 additions.  Measured over these shapes: two orders of the
    # sums differ by 0.004-0.0075 (largest value 0.07), each by 0.003-0.006 from the same chain in 64 bits.
    return {"rel": 0.02, "max": 0.25}
