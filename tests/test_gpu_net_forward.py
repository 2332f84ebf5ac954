"""The one-kernel network evaluation: rows at the edges of its 128-row units,
ensembles, few CTAs walking many units, outputs that TMA cannot store, against
the CPU oracle (float64 with the GPU's BF16 roundings) and against each other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nets():
    from crysplight_b200.surrogate import MLP
    m = [MLP(0, max_batch=128, seed=k) for k in range(9)]
    yield m
    for n in m:
        n.close()


def _x(n, seed=1):
    import torch
    rng = np.random.default_rng(seed)
    return torch.from_numpy(rng.uniform(-1, 1, (n, 3)).astype(np.float32)).cuda()


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 257, 4097])
def test_rows_match_the_oracle(nets, n):
    from oracle import mlp_oracle
    x = _x(n)
    out = nets[0].forward(x).cpu().numpy()
    ref, _ = mlp_oracle.forward(nets[0].get_params().astype(np.float64), x.cpu().numpy())
    # the tolerance of the layer-wise kernels' forward test
    assert np.abs(out - ref).max() < 2e-3 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("members,n,ctas", [(1, 5000, 1), (2, 129, 3), (5, 1000, 0), (5, 40_001, 0), (8, 700, 5),
                                            (9, 300, 2)])
def test_ensemble_equals_its_members(nets, members, n, ctas):
    import torch
    from crysplight_b200.surrogate import forward_ensemble, sync_networks
    x = _x(n, 2)
    torch.cuda.synchronize()
    ref = [m.forward(x) for m in nets[:members]]
    out = torch.full((members, n, 192), float("nan"), device="cuda")
    nets[0].set_max_ctas(ctas)
    try:
        forward_ensemble(nets[:members], x, out, 1)
        sync_networks(nets, 1)
    finally:
        nets[0].set_max_ctas(0)
    for k in range(members):
        assert torch.equal(out[k], ref[k]), k


def test_output_off_the_16_byte_grid(nets):
    import torch
    x = _x(1000, 3)
    buf = torch.zeros(1000 * 192 + 8, device="cuda")
    torch.cuda.synchronize()
    ref = nets[1].forward(x)
    nets[1].forward_into(x, buf[1:1 + 1000 * 192].view(1000, 192))
    assert torch.equal(buf[1:1 + 1000 * 192].view(1000, 192), ref)
    assert float(buf[0]) == 0 and float(buf[-7:].abs().max()) == 0
