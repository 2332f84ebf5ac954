"""A refused call of the networks says why, in the message of that call."""
import ctypes as C

import pytest

from crysplight_b200 import _lib
from crysplight_b200.surrogate import MLP

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nets():
    made = [MLP(0, max_batch=128, seed=k) for k in range(2)]
    yield made
    for n in made:
        n.close()


def test_a_refused_ensemble_says_why(nets):
    import torch
    lib = _lib.load()
    x = torch.zeros((128, 3), device="cuda")
    out = torch.empty((2, 128, 192), device="cuda")
    both = (C.c_void_p * 2)(nets[0].h, nets[1].h)
    missing = (C.c_void_p * 2)(nets[0].h, None)

    def call(a, d_x, n):
        rc = lib.cl_mlp_forward_ensemble(a, 2, C.c_void_p(d_x), C.c_void_p(out.data_ptr()), n, C.c_void_p(1))
        return rc, lib.cl_mlp_last_error(nets[0].h).decode()
    assert call(both, None, 128) == (_lib.CL_ERR_ARG, "null input or output")
    rc, msg = call(missing, x.data_ptr(), 128)
    assert rc == _lib.CL_ERR_ARG and "network 1" in msg
    rc, msg = call(both, x.data_ptr(), -1)
    assert rc == _lib.CL_ERR_ARG and "rows" in msg
    # a call that succeeds leaves no message of an earlier one
    assert call(both, x.data_ptr(), 128) == (_lib.CL_OK, "")
    assert lib.cl_mlp_sync(nets[0].h, C.c_void_p(1)) == _lib.CL_OK


def test_misaligned_targets_are_refused_by_name(nets):
    import torch
    x = torch.rand((256, 3), device="cuda")
    flat = torch.randn(256 * 192 + 1, device="cuda")
    torch.cuda.synchronize()
    t = flat[1:].view(256, 192)                  # 4 bytes past a boundary
    nets[0].set_data(x, t)
    with pytest.raises(_lib.CudaTransportError, match="16-byte boundary"):
        nets[0].train(1, batch=128)
    with pytest.raises(_lib.CudaTransportError, match="16-byte boundary"):
        nets[0].gradient(x[:128], t[:128])
    nets[0].set_data(x, flat[:-1].view(256, 192))
    assert nets[0].train(1, batch=128) > 0.0
