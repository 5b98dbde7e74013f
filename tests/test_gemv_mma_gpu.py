"""The tensor-core matvec (batches of 3 to 8) where its tiled copies are ragged: matrices that end inside a group of 16
rows, columns that end inside a 128-byte piece, a chunk or a part of K, the second matrix of a stack.  Against the f64
oracle; the sums are f32 over at most 272 runs, worst case 272 * 2^-24 = 1.6e-5 of the summed magnitudes, for sums of
random sign well below 1e-5 of the result's norm."""
import numpy as np
import pytest
import torch

from oracle import frink_oracle as fo
from tests.helpers import rel_l2, synth_acts, synth_weights

pytestmark = pytest.mark.gpu
COLS = {fo.Q8_0: (32, 288, 2080, 8192), fo.MXFP4: (32, 480, 2880, 8192), fo.Q6_K: (256, 768, 2048, 8192), fo.Q4_K: (256, 768, 2048, 8192),
        fo.Q5_K: (256, 768, 2048, 8192)}


@pytest.mark.parametrize("kind", list(COLS))
@pytest.mark.parametrize("ci", range(4))
@pytest.mark.parametrize("rows,batch", [(33, 2), (1, 3), (15, 8), (17, 5), (1000, 7), (5000, 8)])
def test_ragged_tiles(kind, ci, rows, batch):
    from frink_b200 import device
    cols = COLS[kind][ci]
    raws = [fo.encode(kind, synth_weights(rows, cols, 61 + m + rows)) for m in range(2)]
    x = synth_acts(batch, cols, 62 + rows)
    w = device.Weights(np.concatenate(raws), kind, rows, cols, n_mats=2)
    xq = fo.q8_1_round(x)
    for m in range(2):
        out = torch.full((batch + 1, rows), float("nan"), device="cuda")
        device.gemv(w, torch.from_numpy(x).cuda(), mat=m, out=out[:batch])
        torch.cuda.synchronize()
        assert device.device_error() == 0
        assert torch.isnan(out[batch]).all()
        assert rel_l2(out[:batch].cpu().numpy(), fo.matmul_f64(kind, raws[m], rows, cols, xq)) <= 1e-5, m


@pytest.mark.parametrize("kind,cols,batch", [(fo.Q4_K, 35072, 3), (fo.Q4_K, 19456, 7), (fo.Q5_K, 19200, 7), (fo.Q8_0, 23232, 5), (fo.Q6_K, 16384, 6),
                                             (fo.MXFP4, 23232, 5), (fo.MXFP4, 17440, 7)])
def test_widest_rows_that_fit(kind, cols, batch):
    """A single stage beside the activations fills shared memory to its last kilobyte."""
    from frink_b200 import device
    rows = 40
    raw, x = fo.encode(kind, synth_weights(rows, cols, 71)), synth_acts(batch, cols, 72)
    y = device.gemv(device.Weights(raw, kind, rows, cols), torch.from_numpy(x).cuda())
    torch.cuda.synchronize()
    assert device.device_error() == 0
    # at most 1096 runs summed in f32: worst case 6.6e-5 of the summed magnitudes, random signs well below 1e-5
    assert rel_l2(y.cpu().numpy(), fo.matmul_f64(kind, raw, rows, cols, fo.q8_1_round(x))) <= 1e-5
