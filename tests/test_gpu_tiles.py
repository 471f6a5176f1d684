"""GPU: the 128-row-tile path where a CTA's next tile lies beyond experts without rows, in the next n-tile of the same
expert, or in another 128-row block of it; against the CPU oracle (metadata bit-exact, output within the layer's bound)."""
import pytest
import torch

from test_gpu_parity import moe, run_and_check  # noqa: F401  (fixture and helper)

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
