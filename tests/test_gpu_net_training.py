"""The two-kernel training pass and the weight gradients' runs: batches at the
edges of units, CTAs and runs, targets off the 32-byte grid, against the CPU
oracle (float64 with the GPU's BF16 roundings)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 148


@pytest.mark.parametrize("B,ctas,shift", [
    (128, 0, 0),                   # one unit; one slot of the one CTA
    (256, 1, 0),                   # both slots
    (384, 1, 4),                   # a slot reused; targets off the 32-byte grid
    (640, 2, 0),                   # CTAs with 3 and 2 units
    (64 * 8 * 3 + 128, 0, 4),      # runs that end inside a layer
    (SMS * 128, 0, 0),             # one unit per CTA
    (SMS * 128 + 128, 0, 0),       # one CTA with two
    (64 * 8 * SMS // 2 + 128, 0, 0),   # runs longer than the least
])
def test_gradients_at_the_edges(B, ctas, shift):
    import torch
    from crysplight_b200.surrogate import MLP
    from oracle import mlp_oracle
    from oracle.mlp_oracle import SHAPES
    rng = np.random.default_rng(B)
    x = rng.uniform(-1, 1, size=(B, 3)).astype(np.float32)
    t = (np.sin(2 * x[:, :1]) * np.cos(x[:, 1:2]) + 0.3 * x[:, 2:3]
         + 0.1 * rng.standard_normal((B, 192))).astype(np.float32)
    buf = torch.empty(B * 192 + 8, device="cuda")
    tt = buf[shift:shift + B * 192].view(B, 192)
    tt.copy_(torch.from_numpy(t))
    m = MLP(0, max_batch=B, seed=8)
    m.set_max_ctas(ctas)
    p = m.get_params().astype(np.float64)
    torch.cuda.synchronize()
    loss, g = m.gradient(torch.from_numpy(x).cuda(), tt)
    m.close()
    rloss, rg = mlp_oracle.gradient(p, x, t)
    assert loss == pytest.approx(rloss, rel=1e-3)
    o = 0
    for name, shp in SHAPES:
        n = int(np.prod(shp))
        a, b = g[o:o + n].astype(np.float64), rg[o:o + n]
        rel = float(np.linalg.norm(a - b) / (np.linalg.norm(b) + 1e-30))
        # the bound of the gradients' existing tests: the oracle rounds where the GPU does
        assert rel < 2e-3, (name, rel)
        o += n
