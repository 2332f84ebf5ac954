"""The ensemble reduction for any number of members (batches of five, the last one
shorter), against NumPy in Float64."""
import ctypes as C

import numpy as np
import pytest

from crysplight_b200 import _lib
from crysplight_b200.params import Box, Readout, SipmGrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 2, 4, 5, 6, 9, 10, 11])
def test_any_number_of_members(K):
    import torch
    rng = np.random.default_rng(K)
    n = 203
    raw = (rng.standard_normal((K, n, 192)) * 0.3).astype(np.float32)
    y_mean = np.concatenate([np.full(64, -5.5), np.full(64, 3.0), np.full(64, -0.5)]).astype(np.float32)
    y_std = np.concatenate([np.full(64, 0.8), np.full(64, 1.0), np.full(64, 0.2)]).astype(np.float32)
    xyz = (rng.uniform(0.0, 1.0, (n, 3)) * [48, 48, 22.4]).astype(np.float32)
    dev = [torch.from_numpy(v).cuda() for v in (raw, y_mean, y_std, xyz)]
    out = [torch.empty((n, 64), device="cuda") for _ in range(3)] + [
        torch.empty(n, device="cuda"), torch.empty(n, dtype=torch.uint8, device="cuda")]
    P = [C.c_void_p(t.data_ptr()) for t in dev + out]
    rc = _lib.load().cl_surrogate_combine_direct(P[0], K, n, P[1], P[2], P[3], None, C.byref(Box((48.0, 48.0, 22.4))),
                                                 C.byref(Readout(SipmGrid(6.0, 8, 8))), 0.4, 0.1, 1.0, *P[4:], None)
    assert rc == _lib.CL_OK
    torch.cuda.synchronize()
    p, tm, ts, sp, fl = (t.cpu().numpy() for t in out)
    y = raw.astype(np.float64) * y_std + y_mean
    pk = np.exp(y[:, :, :64])
    spread = pk.std(0).sum(1) / pk.mean(0).sum(1)
    assert np.allclose(p, np.float32(0.4) * pk.mean(0), rtol=1e-6)
    assert np.allclose(tm, y[:, :, 64:128].mean(0), rtol=1e-6, atol=1e-6)
    assert np.allclose(ts, np.exp(y[:, :, 128:].mean(0)), rtol=1e-6)
    # the variance of one member is the rounding of its square (2^-53 of it): its root, 1e-8
    assert np.allclose(sp, spread, rtol=1e-5, atol=2e-8)
    assert np.array_equal(fl & 1, (spread > 0.1).astype(np.uint8))
