"""GPU: the single-launch prologue stage (b200moe_prologue_small) leaves what route, sort and gather leave, byte for byte, in
every array that a later stage reads."""
import ctypes as C

import pytest
import torch

from test_gpu_parity import gpu_inputs, moe  # noqa: F401  (fixture and helper)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E_local,skew", [(1, 32, False), (9, 32, True), (32, 256, False)])
def test_prologue_equals_separate_stages(moe, T, E_local, skew):  # noqa: F811
    from fused_moe_b200 import _lib
    from fused_moe_b200.kernel import _problem
    lib = _lib.load()
    inp = gpu_inputs(T, E_local, 61, 0, skew)
    out = moe.kernel(**inp)
    ws = moe.last_workspace()
    stream = torch.cuda.current_stream().cuda_stream
    p = _problem(T, E_local, 0, float(inp["routed_scaling_factor"]), inp["routing_logits"], inp["routing_bias"],
                 inp["hidden_states"], inp["hidden_states_scale"], inp["gemm1_weights"], inp["gemm1_weights_scale"],
                 inp["gemm2_weights"], inp["gemm2_weights_scale"], out)
    R = ws.struct.R_max

    arrays = (("topk_idx", T * 8), ("topk_w", T * 8), ("chunk_bits", E_local), ("counts", E_local),
              ("block_offsets", E_local + 1), ("total_blocks", 1), ("scatter_map", T * 8), ("sorted_token_ids", R),
              ("sorted_weights", R), ("a_scale_sorted", 56 * R), ("a_sorted", R * 7168 // 4))

    def run(stages):
        for name, n in arrays:   # whatever a stage does not write is told from what it does
            ws.view(name, torch.int32, (n,)).fill_(0x22222222)
        for stage in stages:
            _lib.check(getattr(lib, "b200moe_" + stage)(C.byref(p), C.byref(ws.struct), stream), stage)
        torch.cuda.synchronize()
        return {name: ws.view(name, torch.int32, (n,)).clone() for name, n in arrays}

    one, three = run(("prologue_small",)), run(("route", "sort", "gather"))
    for name in one:
        assert torch.equal(one[name], three[name]), name
    for name in ("topk_idx", "topk_w", "chunk_bits", "counts", "block_offsets", "total_blocks", "scatter_map"):
        assert not (one[name] == 0x22222222).any(), name   # written in full
