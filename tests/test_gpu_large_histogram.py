"""A histogram of more than 2^31 counts (device buffers, 9 GB): detections land in the
bin that their time gives, at a 64-bit offset."""
import numpy as np
import pytest

from crysplight_b200.params import Readout, SipmGrid, TimeBinning
from cases import BOX_CSI, CENTRE_CSI, OP_CSI_TEFLON

pytestmark = pytest.mark.gpu


def test_counts_beyond_2_31(engine, oracle):
    import torch
    grid, nbins = SipmGrid(1.5, 32, 32), (1 << 21) + (1 << 17)       # 1,024 cells x 2,228,225 bins
    total = 1024 * (nbins + 1)
    assert total > 1 << 31
    free, _ = torch.cuda.mem_get_info()
    if free < 4 * total + (2 << 30):
        pytest.skip("not enough device memory")
    t0s = np.array([5.0, (1 << 21) - 3.0, (1 << 21) + 100_000.0], np.float32)
    kw = dict(n_photons=30_000, seed=8, tau_ns=0.0)
    pos = np.repeat(np.array([CENTRE_CSI], np.float32), 3, 0)
    _, rec = oracle.run_photons_ka(BOX_CSI, OP_CSI_TEFLON, grid, TimeBinning(1.0, 1), positions=pos, t0s=t0s,
                                   return_records=True, **kw)
    det = rec.status == 1
    slot = (rec.idx[det].astype(np.int64) - 1) + 1024 * np.minimum(rec.t[det].astype(np.int64), nbins)
    assert slot.max() > 1 << 31
    src = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (pos[:, 0], pos[:, 1], pos[:, 2], t0s)]
    counts = torch.empty(total, dtype=torch.int32, device="cuda")
    first = torch.empty(1024, dtype=torch.float32, device="cuda")
    ctr = torch.empty(9, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    engine.run_photons_device(BOX_CSI, OP_CSI_TEFLON, Readout(grid), TimeBinning(1.0, nbins), px=src[0].data_ptr(),
                              py=src[1].data_ptr(), pz=src[2].data_ptr(), pt=src[3].data_ptr(), npos=3,
                              counts=counts.data_ptr(), first_ns=first.data_ptr(), counters=ctr.data_ptr(),
                              **kw)
    engine.sync()
    at, want = np.unique(slot, return_counts=True)
    got = counts[torch.from_numpy(at).cuda()].cpu().numpy()
    assert np.array_equal(got, want)
    step = 1 << 28
    assert sum(int(counts[i:i + step].sum()) for i in range(0, total, step)) == det.sum() == int(ctr[0])
