"""GPU: the 128-row-tile path where a CTA's next tile lies beyond experts without rows, in the next n-tile of the same
expert, or in another 128-row block of it; against the CPU oracle (metadata bit-exact, output within the layer's bound)."""
import pytest
import torch

from test_gpu_parity import gpu_inputs, moe, run_and_check  # noqa: F401  (fixture and helpers)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E_local,seed,offset,skew", [
    (130, 256, 51, 0, True),     # few hot experts, most of the others empty
    (150, 256, 52, 0, False),    # nearly every expert has a few rows: thousands of tiles
    (700, 3, 53, 8, True),       # fewer tiles than SMs, experts with several 128-row blocks
    (120, 1, 54, 130, False),    # one expert
])
def test_tile_path_matches_oracle(moe, oracle, T, E_local, seed, offset, skew):  # noqa: F811
    out, ref, _ = run_and_check(moe, oracle, T, E_local, seed, offset, skew)
    empty = (torch.as_tensor(ref["out_bf16"]).float() == 0).all(dim=1)
    assert not out.cpu()[empty].any()


def test_row_counts_at_warp_edges(moe):  # noqa: F811
    """Experts with one row, with 32 rows (a promotion warp's) or one more, 128 (a tile's) or one more.  The same batch cut
    into two runs of 80 tokens goes through the token-minor GEMMs instead.  Both add the same float32 products, in another
    association in tiles that several CTAs share (2e-7 relative), which can move an intermediate by one step of its second
    e4m3 term (2^-8 of its value) in one of 2048 terms of a sum, and the tile path's rows are rounded to float16 (2^-12)
    before the eight of a token are added: 1e-3 of the largest sum bounds them."""
    counts = [1, 32, 33, 64, 97, 128, 129, 160]
    T, E = 160, len(counts)
    inp = gpu_inputs(T, E, 71, 8, False)
    t = torch.arange(T, device="cuda")
    idx = torch.stack([torch.where(t < c, 8 + e, 255) for e, c in enumerate(counts)], dim=1).int()
    w = torch.rand((T, 8), generator=torch.Generator(device="cuda").manual_seed(72), device="cuda") + 0.1
    rest = [inp[k] for k in ("gemm1_weights", "gemm1_weights_scale", "gemm2_weights", "gemm2_weights_scale")]

    def layer(a, b):
        return moe.kernel_from_topk(idx[a:b].contiguous(), w[a:b].contiguous(), inp["hidden_states"][a:b].contiguous(),
                                    inp["hidden_states_scale"][:, a:b].contiguous(), *rest, 8,
                                    out_dtype=torch.float32)
    whole = layer(0, T).clone()
    moe.check_status()
    parts = torch.cat([layer(0, 80).clone(), layer(80, T).clone()])
    moe.check_status()
    assert torch.isfinite(whole).all()
    assert float((whole - parts).abs().max()) <= 1e-3 * float(parts.abs().max())
