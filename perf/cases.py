"""Workloads of the fused MoE layer, as users of this framework run them: sizes, inputs, one pass, the work a pass cannot
do without, and how far two correct implementations may differ.

Every case is one layer of the DeepSeek-V3 shape (hidden 7168, intermediate 2048, 256 experts, top-8) seen from one GPU.
Plain values of a case:

  entry    which public entry point a pass goes through
             "kernel"  fused_moe_b200.kernel.kernel on e4m3 activations
             "bf16"    quantize_activations on bf16 activations, then kernel
             "topk"    kernel_from_topk with float32 sums: a shard whose tokens were routed elsewhere
             "ep"      the expert-parallel shard's forward (peer transport, half rows), one rank owning every expert
  tokens   batch size T
  experts  local experts E (the weights on this GPU), `offset` = global id of the first
  skew     per-expert logit offsets ~N(0, 1.5) on top of the N(0, 1) logits: a few hot experts take most of the tokens
  router   which router is in use: seeds the expert bias and the skew offsets, which belong to the model, not the batch
"""
import torch

from fused_moe_b200 import ep
from fused_moe_b200 import kernel as moe

H = 7168
I = 2048
EXPERTS = 256
GROUPS = 8
TOP_GROUPS = 4
TOP_K = 8
SCALE = 2.5
W13_BYTES = 2 * I * H
W2_BYTES = H * I
SCALE_BYTES = 4 * (2 * I // 128 * (H // 128) + H // 128 * (I // 128))


def _case(name, entry, tokens, experts, offset=0, skew=False, router=0):
    return {"name": name, "entry": entry, "tokens": tokens, "experts": experts, "offset": offset, "skew": skew,
            "router": router}


def listed():
    return [
        # one sequence being decoded: about one (token, local expert) pair, latency and launches count
        _case("decode_1", "kernel", 1, 32),
        # a handful of sequences
        _case("decode_7", "kernel", 7, 32),
        # a small decode batch, most experts see one token or none
        _case("decode_20", "kernel", 20, 32),
        # a decode batch that touches nearly every local expert: bound by reading the weights once
        _case("decode_80", "kernel", 80, 32),
        # the same regime with the whole model's experts on one GPU
        _case("decode_64_all_experts", "kernel", 64, 256),
        # a large decode batch or a short prompt: some ten rows per expert
        _case("batch_333", "kernel", 333, 32, offset=96),
        # a prompt whose activations arrive in bf16 and are quantised first
        _case("prompt_901_bf16", "bf16", 901, 32),
        # a shard of a larger deployment: routing ran elsewhere, un-rounded sums travel on
        _case("shard_1500_topk", "topk", 1500, 64, offset=64),
        # the expert-parallel step: rank, exchange, pack, layer over received records, combine
        _case("ep_2048", "ep", 2048, 256),
        # prefill with hot experts
        _case("prefill_4096_skew", "kernel", 4096, 32, skew=True, router=1),
        # a long ragged prefill with hot experts
        _case("prefill_14107_skew", "kernel", 14107, 32, skew=True, router=2),
        # long prefill through all 256 experts on one GPU: the largest
        _case("prefill_16384_all_experts", "kernel", 16384, 256),
    ]


def draw(rng):
    """A case of the same ranges: decode to prefill batches (1 .. 16384, log-uniform), a shard of 8 .. 256 experts
    anywhere in the model, either kind of router.  The expert-parallel step owns all experts and moves every token
    twice, so it is drawn up to half the largest batch."""
    entry = rng.choice(["kernel", "kernel", "kernel", "bf16", "topk", "ep"])
    tokens = int(round(2.0 ** rng.uniform(0.0, 13.0 if entry == "ep" else 14.0)))
    experts = EXPERTS if entry == "ep" else rng.choice([8, 32, 32, 64, 128, 256])
    return {"entry": entry, "tokens": tokens, "experts": experts, "offset": rng.randint(0, EXPERTS - experts),
            "skew": rng.random() < 0.5, "router": rng.randint(0, 999)}


def _router(case):
    """Expert bias and logit offsets of the case's router (CPU, so that work() sees the same ones)."""
    g = torch.Generator().manual_seed(1000003 + case["router"])
    bias = (0.1 * torch.randn(EXPERTS, generator=g)).bfloat16()
    offsets = 1.5 * torch.randn(EXPERTS, generator=g)
    return bias, offsets if case["skew"] else torch.zeros(EXPERTS)


def _local_load(case, logits, bias):
    """(token, local expert) pairs of a batch and local experts with at least one token: group-limited top-8."""
    score = torch.sigmoid(logits) + bias.float()
    by_group = score.view(-1, GROUPS, EXPERTS // GROUPS)
    keep = by_group.topk(2, dim=2).values.sum(dim=2).topk(TOP_GROUPS, dim=1).indices
    mask = torch.zeros(by_group.shape[:2], device=logits.device).scatter_(1, keep, 1.0)
    masked = torch.where(mask.unsqueeze(2) > 0, by_group, torch.full_like(by_group, -1.0)).view(-1, EXPERTS)
    count = torch.bincount(masked.topk(TOP_K, dim=1).indices.flatten(), minlength=EXPERTS)
    local = count[case["offset"]:case["offset"] + case["experts"]]
    return int(local.sum()), int((local > 0).sum())


def _draw_logits(case, gen, bias, offsets):
    """Router logits of a batch in which at least one token has a local expert (a shard is not handed a batch that has
    nothing for it): one draw but for the very smallest batches."""
    while True:
        logits = torch.randn((case["tokens"], EXPERTS), generator=gen, device=gen.device) + offsets
        load = _local_load(case, logits, bias)
        if load[0] > 0:
            return logits, load


def _quantize_rows(x):
    """[T, 7168] -> e4m3 rows and the [56, T] scales, one per token per 128 columns."""
    blocks = x.view(x.shape[0], H // 128, 128)
    s = (blocks.abs().amax(dim=2) / 448.0).clamp_min(1e-12)
    q = (blocks / s.unsqueeze(2)).to(torch.float8_e4m3fn).view(x.shape[0], H)
    return q, s.t().contiguous()


def _weights(gen, experts, rows, cols):
    """N(0, 0.02) expert matrices as e4m3 with one float32 scale per 128 x 128 block."""
    q = torch.empty((experts, rows, cols), dtype=torch.float8_e4m3fn, device="cuda")
    s = torch.empty((experts, rows // 128, cols // 128), dtype=torch.float32, device="cuda")
    for e in range(experts):
        w = (0.02 * torch.randn((rows, cols), generator=gen, device="cuda")).view(rows // 128, 128, cols // 128, 128)
        s[e] = w.abs().amax(dim=(1, 3)) / 448.0
        q[e] = (w / s[e][:, None, :, None]).to(torch.float8_e4m3fn).view(rows, cols)
    return q, s


def _inputs(case, seed):
    """Layer weights, router logits and bias, bf16 activations."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    tokens, experts = case["tokens"], case["experts"]
    w13, w13_scale = _weights(gen, experts, 2 * I, H)
    w2, w2_scale = _weights(gen, experts, H, I)
    bias, offsets = _router(case)
    bias = bias.cuda()
    logits, _ = _draw_logits(case, gen, bias, offsets.cuda())
    x = torch.randn((tokens, H), generator=gen, device="cuda").bfloat16()
    weights = {"gemm1_weights": w13, "gemm1_weights_scale": w13_scale, "gemm2_weights": w2,
               "gemm2_weights_scale": w2_scale}
    return weights, logits, bias, x


def prepare(case, seed):
    tokens, entry = case["tokens"], case["entry"]
    weights, logits, bias, x = _inputs(case, seed)
    state = {"entry": entry, "weights": weights, "offset": case["offset"], "logits": logits, "bias": bias}
    if entry == "bf16":
        state["x"] = x
    else:
        state["hidden"], state["hidden_scale"] = _quantize_rows(x.float())
    if entry == "topk":
        state["topk"], state["topk_weights"] = moe.route(logits, bias, SCALE)
    if entry == "ep":
        state["shard"] = ep.make_cuda_shard(weights, rank=0, world=1, transport="peer", max_tokens_per_rank=tokens,
                                            partial_rows="half")
    return state


def run(state):
    entry = state["entry"]
    if entry == "ep":
        return state["shard"].forward(state["logits"], state["bias"], state["hidden"], state["hidden_scale"], SCALE)
    if entry == "topk":
        return moe.kernel_from_topk(state["topk"], state["topk_weights"], state["hidden"], state["hidden_scale"],
                                    local_expert_offset=state["offset"], out_dtype=torch.float32, **state["weights"])
    if entry == "bf16":
        hidden, hidden_scale = moe.quantize_activations(state["x"])
        out = moe.kernel(state["logits"], state["bias"], hidden, hidden_scale, local_expert_offset=state["offset"],
                         routed_scaling_factor=SCALE, **state["weights"])
        return {"hidden": hidden, "hidden_scale": hidden_scale, "out": out}
    return moe.kernel(state["logits"], state["bias"], state["hidden"], state["hidden_scale"],
                      local_expert_offset=state["offset"], routed_scaling_factor=SCALE, **state["weights"])


def _route64(logits, bias):
    """Group-limited top-8 in 64 bits: expert ids and weights."""
    s = torch.sigmoid(logits.double())
    by_group = (s + bias.double()).view(-1, GROUPS, EXPERTS // GROUPS)
    keep = by_group.topk(2, dim=2).values.sum(dim=2).topk(TOP_GROUPS, dim=1).indices
    mask = torch.zeros(by_group.shape[:2], device=logits.device).scatter_(1, keep, 1.0)
    idx = torch.where(mask.unsqueeze(2) > 0, by_group, -1.0).view(-1, EXPERTS).topk(TOP_K, dim=1).indices
    w = s.gather(1, idx)
    return idx, w / (w.sum(dim=1, keepdim=True) + 1e-20) * SCALE


def _dequant64(q, scale):
    rows, cols = q.shape
    return (q.double().view(rows // 128, 128, cols // 128, 128) * scale.double()[:, None, :, None]).view(rows, cols)


def exact(case, seed):
    """The layer in 64 bits on the same e4m3 values and scales."""
    weights, logits, bias, x = _inputs(case, seed)
    hidden, hidden_scale = _quantize_rows(x.double() if case["entry"] == "bf16" else x.float())
    idx, w = _route64(logits, bias)
    scale_rows = hidden_scale.t().double()
    out = torch.zeros((case["tokens"], H), dtype=torch.float64, device="cuda")
    for e in range(case["experts"]):
        token, k = (idx == case["offset"] + e).nonzero(as_tuple=True)
        if token.numel() == 0:
            continue
        w13 = _dequant64(weights["gemm1_weights"][e], weights["gemm1_weights_scale"][e])
        w2 = _dequant64(weights["gemm2_weights"][e], weights["gemm2_weights_scale"][e])
        for part in torch.arange(token.numel(), device="cuda").split(2048):
            t = token[part]
            a = (hidden[t].double().view(-1, H // 128, 128) * scale_rows[t].unsqueeze(2)).view(-1, H)
            up, gate = (a @ w13.t()).split(I, dim=1)
            y = (gate * torch.sigmoid(gate) * up) @ w2.t()
            out.index_add_(0, t, y * w[t, k[part]].unsqueeze(1))
    if case["entry"] == "bf16":
        return {"hidden": None, "hidden_scale": hidden_scale, "out": out}
    return out


def work(case):
    """For one batch of the case's router.  Bytes: the weights and scales of every local expert that has a token, the
    activations and router inputs, the output.  Operations: both products of every (token, local expert) pair.  Nothing in between the two products, no
    second term of the intermediate and no padding is counted."""
    tokens, entry = case["tokens"], case["entry"]
    bias, offsets = _router(case)
    _, (pairs, active) = _draw_logits(case, torch.Generator().manual_seed(7), bias, offsets)
    per_token = H + H // 128 * 4                       # e4m3 row and its scales
    if entry == "bf16":
        per_token = 2 * H + H + H // 128 * 4           # bf16 row in, e4m3 row and scales out
    per_token += TOP_K * 8 if entry == "topk" else EXPERTS * 4
    per_token += 4 * H if entry == "topk" else 2 * H
    return {"bytes": active * (W13_BYTES + W2_BYTES + SCALE_BYTES) + tokens * per_token,
            "flops": 2 * pairs * (W13_BYTES + W2_BYTES)}


def tolerance(case):
    """About four times the error of the layer against the same layer in float64 (same routing, scales and e4m3 values)
    at 1 .. 14107 tokens: bf16 results 1.73e-3 .. 1.79e-3 in the 2-norm, of which 1.66e-3 is the rounding to bf16, and at
    most 1.1e-2 on one value; float32 sums 5.7e-4 and 4.3e-3."""
    if case["entry"] == "topk":
        return {"rel": 2.3e-3, "max": 1.7e-2}
    return {"rel": 7e-3, "max": 4.4e-2}
