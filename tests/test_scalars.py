"""The two scalar arguments as 0-d tensors: every call uses the value that the tensor holds at that call."""
import pytest
import torch

from test_gpu_parity import KEYS, gpu_inputs, moe  # noqa: F401  (fixture and helper)


@pytest.mark.parametrize("dtype,cast,values", [(torch.int32, int, (0, 32, 64, 96)), (torch.int64, int, (224, 0, 31)),
                                               (torch.float32, float, (2.5, 1.0, 0.5)), (torch.float64, float, (2.5, 3.0))])
def test_cpu_scalar_is_read_on_every_call(dtype, cast, values):
    from fused_moe_b200.kernel import _host_scalar
    # temporaries: the allocator gives the next one the address of the last
    assert [_host_scalar(torch.tensor(v, dtype=dtype), cast) for v in values] == list(values)
    t = torch.zeros((), dtype=dtype)
    for v in values:
        t.fill_(v)
        assert _host_scalar(t, cast) == v
        assert _host_scalar(v, cast) == v


@pytest.mark.gpu
@pytest.mark.parametrize("device", ["cpu", "cuda"])
def test_scalar_tensors_follow_their_value(moe, device):  # noqa: F811
    inp = gpu_inputs(7, 32, 0, 0, False)
    values = ((0, 2.5), (32, 1.0), (96, 2.0), (0, 0.5))
    want = [moe.kernel(*[dict(inp, local_expert_offset=o, routed_scaling_factor=s)[k] for k in KEYS]).clone()
            for o, s in values]
    assert not torch.equal(want[0], want[1]) and not torch.equal(want[0], want[3])
    kept_o = torch.zeros((), dtype=torch.int32, device=device)
    kept_s = torch.zeros((), dtype=torch.float32, device=device)
    for (o, s), ref in zip(values, want):
        fresh = dict(inp, local_expert_offset=torch.tensor(o, dtype=torch.int32, device=device),
                     routed_scaling_factor=torch.tensor(s, dtype=torch.float32, device=device))
        assert torch.equal(moe.kernel(*[fresh[k] for k in KEYS]), ref)
        del fresh
        kept_o.fill_(o)
        kept_s.fill_(s)
        kept = dict(inp, local_expert_offset=kept_o, routed_scaling_factor=kept_s)
        assert torch.equal(moe.kernel(*[kept[k] for k in KEYS]), ref)


@pytest.mark.gpu
def test_device_scalar_under_capture(moe):  # noqa: F811
    """A captured call takes the value of a device scalar that an earlier call read; one that was written since, or never
    read, is refused, and the capture goes on."""
    inp = gpu_inputs(7, 32, 0, 0, False)
    want = moe.kernel(**inp).clone()
    seen = torch.tensor(2.5, device="cuda")
    written = torch.tensor(2.5, device="cuda")
    unseen = torch.tensor(2.5, device="cuda")
    out = torch.zeros((7, 7168), dtype=torch.bfloat16, device="cuda")

    def call(scale):
        return moe.kernel(*[dict(inp, routed_scaling_factor=scale)[k] for k in KEYS], out)

    call(seen)
    call(written)
    written.fill_(1.0)
    torch.cuda.synchronize()
    out.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for scale in (written, unseen):
            with pytest.raises(RuntimeError, match="capture"):
                call(scale)
        call(seen)
    graph.replay()
    torch.cuda.synchronize()
    moe.check_status()
    assert torch.equal(out, want)
