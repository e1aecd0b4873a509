"""GPU: the kernels of a prefill block and the batched routing of a decode step at the edges of their tiles."""
import pytest
import torch

from tests.helpers import orc, rel_err
from tests.scenarios import randomize_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Dh,H,Hkv,W,Me,Ms,norm", [(64, 4, 2, 50, 9, 5, "full"), (64, 3, 1, 64, 32, 32, "identity"),
                                                   (128, 2, 1, 40, 8, 16, "full"), (128, 8, 1, 100, 70, 22, "identity")])
@pytest.mark.parametrize("block,L", [(1, 3), (63, 130), (64, 192), (65, 131), (128, 320), (200, 333)])
def test_prefill_attention_at_tile_edges(Dh, H, Hkv, W, Me, Ms, norm, block, L):
    """64-row query tiles and 64-key tiles, their remainders, prefix tiles without a visible slot (fresh states: the first
    block reads none, later ones skip the banks that are still empty) against the shape-generic kernel (bf16; P and the two
    streams are rounded to bf16 at different places: a few 2^-9 of the result)."""
    from coda_gqa_l_b200 import CoDAGQALandmarkPerf2, _deep_copy_state
    torch.manual_seed(3)
    mod = CoDAGQALandmarkPerf2(embed_dim=H * Dh, num_heads=H, num_kv_heads=Hkv, window=W, num_landmarks_exact=Me,
                               num_landmarks_summary=Ms, head_norm_mode=norm).eval()
    randomize_weights(mod, 3)
    mod = mod.to(torch.bfloat16).cuda()
    x = orc.mixture_inputs(3, L, H * Dh, centroids=16, sigma=0.3, seed=5, dtype=torch.bfloat16).cuda()
    sa = mod.init_state(batch_size=3, device="cuda", dtype=torch.bfloat16)
    sb = _deep_copy_state(sa)
    ya, sa = mod.prefill_chunked(x, sa, block_size=block)
    assert mod.device_status() == 0
    mod.use_tuned_kernels = False
    yb, sb = mod.prefill_chunked(x, sb, block_size=block)
    assert torch.equal(sa.k_buf, sb.k_buf) and torch.equal(sa.allowed, sb.allowed)
    assert rel_err(ya, yb) < 8e-3
