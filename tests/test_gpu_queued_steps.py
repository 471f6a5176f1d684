"""GPU: calls of different sizes queued without a host wait between them.  The kernels of a call are resident while those of
the call before still run and share its buffers, so anything read ahead of the dependency wait (a row count, a selection word,
an offset) would be the other call's.  Every output must be the bytes that the same call gives alone."""
import pytest
import torch

from test_gpu_parity import _world1_weights, gpu_inputs, moe  # noqa: F401  (fixture and helpers)

pytestmark = pytest.mark.gpu

ARGS = ("routing_logits", "routing_bias", "hidden_states", "hidden_states_scale", "routed_scaling_factor")


def _queued(step, batches, rounds):
    """`step(batch, out)` queues one call.  Returns nothing; asserts that queued calls give what single ones give."""
    want = []
    for b in batches:
        out = torch.empty((b["routing_logits"].shape[0], 7168), dtype=torch.bfloat16, device="cuda")
        step(b, out)
        torch.cuda.synchronize()
        want.append(out)
    outs = [[torch.full_like(w, 3.0) for w in want] for _ in range(rounds)]
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)   # ~50 ms, in which the host queues calls: they then run back to back
    for r in range(rounds):
        for b, o in zip(batches, outs[r]):
            step(b, o)
    torch.cuda.synchronize()
    for r in range(rounds):
        for i, (o, w) in enumerate(zip(outs[r], want)):
            assert torch.equal(o, w), f"round {r}, call {i}: {int((o != w).any(dim=1).sum())} of {w.shape[0]} rows differ"


@pytest.mark.parametrize("rows", ["float", "half"])
def test_expert_parallel_steps_of_changing_size(moe, rows):  # noqa: F811
    from fused_moe_b200 import ep, synth
    inp = gpu_inputs(300, 32, 4, 64, True)
    shard = ep.make_cuda_shard(_world1_weights(inp), rank=0, world=1, transport="peer", max_tokens_per_rank=512,
                               partial_rows=rows)
    batches = [synth.make_inputs(T, 32, seed=seed, local_expert_offset=64, skew=True, device="cuda", weights=inp)
               for T, seed in ((412, 12), (206, 13), (130, 14), (511, 15), (33, 16))]
    _queued(lambda b, o: shard.forward(*[b[k] for k in ARGS], o), batches, 20)
    moe.check_status()
    shard.check_status()


def test_expert_parallel_host_memory_runs_repeated(moe):  # noqa: F811
    """Host-memory calls of one, two and three runs back to back: the runs' sizes change from step to step."""
    from fused_moe_b200 import ep, synth
    inp = gpu_inputs(300, 32, 4, 64, True)
    shard = ep.make_cuda_shard(_world1_weights(inp), rank=0, world=1, transport="peer", max_tokens_per_rank=512)
    cur = synth.make_inputs(412, 32, seed=12, local_expert_offset=64, skew=True, device="cuda", weights=inp)
    want = shard.forward(*[cur[k] for k in ARGS]).cpu()
    host = {k: cur[k].cpu().pin_memory() for k in ("routing_logits", "hidden_states", "hidden_states_scale")}
    outs = [torch.empty((412, 7168), dtype=torch.bfloat16).pin_memory() for _ in range(4)]
    for rep in range(50):
        evs = [torch.cuda.Event() for _ in outs]
        for o, ev, slices in zip(outs, evs, (1, 2, 1, 3)):
            o.fill_(3.0)
            shard.forward_host(host["routing_logits"], cur["routing_bias"], host["hidden_states"],
                               host["hidden_states_scale"], cur["routed_scaling_factor"], o, slices=slices, ready_event=ev)
        for i, (o, ev) in enumerate(zip(outs, evs)):
            ev.synchronize()
            assert torch.equal(o, want), f"repetition {rep}, call {i}"
    shard.check_status()


def test_layer_calls_of_changing_size(moe):  # noqa: F811
    """Decode, token-minor, tile and scan paths in turn on one workspace."""
    from fused_moe_b200 import synth
    inp = gpu_inputs(300, 32, 4, 64, True)
    batches = [synth.make_inputs(T, 32, seed=20 + i, local_expert_offset=64, skew=bool(i & 1), device="cuda", weights=inp)
               for i, T in enumerate((333, 7, 40, 1500, 20, 1, 113, 80))]
    _queued(lambda b, o: moe.kernel(**b, output=o), batches, 10)
    moe.check_status()
