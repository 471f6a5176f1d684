"""GPU: the decode path (at most eight tokens) where its work split changes: one expert for all tokens, more pairs than one
staging pass of the second kernel holds, every token on experts of its own, no local expert for some tokens; against the CPU
oracle, the stage entry points against the whole call, the range and the precision of its sums against 64 bits."""
import ctypes as C

import pytest
import torch

from conftest import assert_close
from test_gpu_parity import KEYS, gpu_inputs, moe, run_and_check  # noqa: F401  (fixture and helpers)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E_local,seed,offset,skew", [
    (8, 256, 31, 0, False),    # 64 pairs: three staging passes, a list cut between two of them
    (8, 256, 32, 0, True),     # 64 pairs on few experts: lists of several tokens
    (5, 256, 33, 0, True),     # 40 pairs
    (3, 256, 34, 0, False),    # exactly 24 pairs: one full staging pass
    (8, 32, 35, 32, True),     # hot experts
    (7, 5, 36, 201, True),     # fewer experts than tokens, tokens without a local expert
    (8, 1, 37, 77, True),      # one expert
    (2, 128, 38, 128, False),
])
def test_decode_matches_oracle(moe, oracle, T, E_local, seed, offset, skew):  # noqa: F811
    out, ref, _ = run_and_check(moe, oracle, T, E_local, seed, offset, skew)
    empty = (torch.as_tensor(ref["out_bf16"]).float() == 0).all(dim=1)
    assert not out.cpu()[empty].any()


@pytest.mark.parametrize("T,E_local,skew", [(1, 32, False), (8, 256, True), (6, 32, True)])
def test_decode_stages_equal_the_call(moe, T, E_local, skew):  # noqa: F811
    """route, gemv1, gemv2 launched one by one give the bytes of the whole call (which routes inside gemv1), into bf16 and
    into float32, also where the destination is aligned to its element only."""
    from fused_moe_b200 import _lib
    from fused_moe_b200.kernel import _problem
    lib = _lib.load()
    inp = gpu_inputs(T, E_local, 41, 0, skew)
    whole = moe.kernel(**inp)
    ws = moe.last_workspace()
    stream = torch.cuda.current_stream().cuda_stream
    flat16 = torch.full((T * 7168 + 1,), 3.0, dtype=torch.bfloat16, device="cuda")
    flat32 = torch.full((T * 7168 + 1,), 3.0, dtype=torch.float32, device="cuda")
    for out in (flat16[:-1], flat16[1:], flat32[:-1], flat32[1:]):
        p = _problem(T, E_local, 0, float(inp["routed_scaling_factor"]), inp["routing_logits"], inp["routing_bias"],
                     inp["hidden_states"], inp["hidden_states_scale"], inp["gemm1_weights"], inp["gemm1_weights_scale"],
                     inp["gemm2_weights"], inp["gemm2_weights_scale"], out)
        for stage in ("route", "gemv1", "gemv2"):
            _lib.check(getattr(lib, "b200moe_" + stage)(C.byref(p), C.byref(ws.struct), stream), stage)
        torch.cuda.synchronize()
        assert torch.equal(out.view(T, 7168).to(torch.bfloat16), whole)
        flat, spare = (flat16 if out.dtype == torch.bfloat16 else flat32), (0 if out.storage_offset() else -1)
        assert flat[spare] == 3.0   # the element beside the destination
        flat.fill_(3.0)


@pytest.mark.parametrize("T,E_local,seed,offset,skew", [(5, 32, 14, 0, True), (1, 256, 15, 0, False), (8, 16, 14, 32, True)])
def test_sorted_path_of_small_batches(moe, oracle, T, E_local, seed, offset, skew):  # noqa: F811
    """At most eight tokens whose routing ran elsewhere: route, sort, gather and the token-minor GEMMs, which a routed call of
    that size does not reach."""
    inp = gpu_inputs(T, E_local, seed, offset, skew)
    idx, w = moe.route(inp["routing_logits"], inp["routing_bias"], inp["routed_scaling_factor"])
    out = moe.kernel_from_topk(idx, w, inp["hidden_states"], inp["hidden_states_scale"], inp["gemm1_weights"],
                               inp["gemm1_weights_scale"], inp["gemm2_weights"], inp["gemm2_weights_scale"], offset)
    moe.check_status()
    ref = oracle.kernel(*[inp[k] for k in KEYS])
    assert_close(out.float().cpu(), ref["out_bf16"].float(), what=f"T={T} E={E_local}")


def layer64(inp, E_local, offset=0):
    """The layer in 64 bits on the same e4m3 values, scales and routing, [T, 7168]."""
    from fused_moe_b200.kernel import route
    idx, w = route(inp["routing_logits"], inp["routing_bias"], inp["routed_scaling_factor"])

    def dequant(q, s):
        r, c = q.shape
        return (q.double().view(r // 128, 128, c // 128, 128) * s.double()[:, None, :, None]).view(r, c)

    x = inp["hidden_states"].double().view(-1, 56, 128) * inp["hidden_states_scale"].t().double().unsqueeze(2)
    x = x.view(-1, 7168)
    out = torch.zeros_like(x)
    for e in range(E_local):
        token, k = (idx == offset + e).nonzero(as_tuple=True)
        if token.numel():
            up, gate = (x[token] @ dequant(inp["gemm1_weights"][e], inp["gemm1_weights_scale"][e]).t()).split(2048, dim=1)
            y = (gate * torch.sigmoid(gate) * up) @ dequant(inp["gemm2_weights"][e], inp["gemm2_weights_scale"][e]).t()
            out.index_add_(0, token, y * w[token, k].double().unsqueeze(1))
    return out


@pytest.mark.parametrize("T,E_local,skew,factor", [(8, 32, False, 3e-20), (8, 256, True, 3e-20), (2, 32, True, 1e-20)])
def test_decode_keeps_small_rows(moe, T, E_local, skew, factor):  # noqa: F811
    """Activation scales so small that the intermediate (quadratic in them) lies near the smallest normal float32, where the
    reciprocal of a row's maximum overflows; W2 scales bring the result back into range."""
    inp = dict(gpu_inputs(T, E_local, 44, 0, skew))
    inp["hidden_states_scale"] = inp["hidden_states_scale"] * factor
    inp["gemm2_weights_scale"] = inp["gemm2_weights_scale"] * 1e36
    out = moe.kernel(**inp)
    ref = layer64(inp, E_local)
    assert torch.isfinite(out).all()
    # bf16 rounding 1.7e-3 and the float32 intermediate's own step near 1e-39 (2^-149 / 1e-40: 1.4e-5)
    assert (out.double() - ref).norm() <= 3e-3 * ref.norm()
    inp["gemm2_weights_scale"] = gpu_inputs(T, E_local, 44, 0, skew)["gemm2_weights_scale"]
    assert torch.isfinite(moe.kernel(**inp)).all()


@pytest.mark.parametrize("T,E_local,skew", [(1, 128, False), (7, 32, False), (8, 32, True), (8, 256, True), (4, 1, False)])
@pytest.mark.parametrize("wide", [1.0, 1e6])
def test_decode_sums_keep_32_bits(moe, T, E_local, skew, wide):  # noqa: F811
    """The un-rounded sums against 64 bits.  The one rounding below 32 bits is the intermediate's to float16, whose relative
    error has a root mean square of 2.1e-4 over a binade and no weight in which to add up: so much is left of it in the
    2-norm of the result.  Also where one 128-column block of the intermediate is `wide` times larger than the others and
    its W2 scale as much smaller."""
    from fused_moe_b200 import _lib
    from fused_moe_b200.kernel import _problem, route
    inp = dict(gpu_inputs(T, E_local, 43, 0, skew))
    if E_local == 1:   # every token on the one expert
        inp["routing_logits"] = inp["routing_logits"].clone()
        inp["routing_logits"][:, 0] += 20.0
        assert (route(inp["routing_logits"], inp["routing_bias"], 2.5)[0] == 0).any(dim=1).all()
    for name, at, f in (("gemm1_weights_scale", (slice(None), 5), wide), ("gemm2_weights_scale", (slice(None), slice(None), 5), 1 / wide)):
        inp[name] = inp[name].clone()
        inp[name][at] *= f
    moe.kernel(**inp)
    ws = moe.last_workspace()
    out = torch.full((T, 7168), 3.0, device="cuda")
    p = _problem(T, E_local, 0, float(inp["routed_scaling_factor"]), inp["routing_logits"], inp["routing_bias"],
                 inp["hidden_states"], inp["hidden_states_scale"], inp["gemm1_weights"], inp["gemm1_weights_scale"],
                 inp["gemm2_weights"], inp["gemm2_weights_scale"], out)
    _lib.check(_lib.load().b200moe_forward(C.byref(p), C.byref(ws.struct), torch.cuda.current_stream().cuda_stream), "forward")
    ref = layer64(inp, E_local)
    err = ((out.double() - ref).norm() / ref.norm()).item()
    print(f"T={T} E={E_local} skew={skew} wide={wide:g}: {err:.3g}")
    assert err <= 2.6e-4
