"""The first-pass term on pixel grids that end before the face does: the last
column and row reach the face edge (a detection beyond them is the last pixel's,
src/transport.jl:96-108), so light that lands there is theirs."""
import numpy as np
import pytest

from crysplight_b200.params import Box, OpticalParams, Readout, SipmGrid
from oracle import first_pass as FP
from test_gpu_first_pass import _direct_gpu

pytestmark = pytest.mark.gpu
L = (48.0, 48.0, 22.4)
OP = OpticalParams(2.15, 1.45, 20000.0, 2222.0, 0.985, True, True, 0.0227, 1.0)


@pytest.mark.parametrize("nx,ny,pitch", [
    (8, 8, 6.0), (8, 8, 5.0), (8, 8, 1.0), (8, 8, 9.0), (64, 1, 0.75), (1, 64, 0.75), (32, 2, 1.5), (2, 32, 1.5),
    (16, 4, 3.0), (4, 16, 3.0), (64, 1, 48.0), (1, 64, 0.1)])
def test_pixels_reach_the_face_edge(nx, ny, pitch):
    rng = np.random.default_rng(3)
    xyz = rng.uniform(0, 1, (1200, 3)) * L
    xyz[:, 2] = L[2] * (1.0 - rng.uniform(0.0005, 0.9, 1200))
    # the corners, and sites whose light lands beyond the last edge alone
    xyz[:5] = [[24.0, 24.0, 22.3], [0.0, 0.0, 20.0], [48.0, 48.0, 20.0], [47.0, 47.0, 22.39], [24.0, 24.0, 22.4]]
    xyz = xyz.astype(np.float32)
    got = _direct_gpu(xyz, Box(L), OP, Readout(SipmGrid(pitch, nx, ny)))
    # the box and the pitch as the kernel sees them (Float32)
    want = FP.direct(xyz.astype(np.float64), [float(v) for v in np.float32(L)], float(OP.n_crystal),
                     float(OP.n_coupling), float(OP.abs_len_mm), float(OP.rayleigh_mm), float(np.float32(pitch)), nx, ny)
    err = np.abs(got - want)
    assert np.all(err <= 2e-4 * want + 2e-6), (float(err.max()), int(err.argmax()))
    assert got[4].sum() == 0.0
