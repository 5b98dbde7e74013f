"""The plain Q4_K matvec of one row around the width that its blocks load in one pass (4096 values of x): one pass, a full
one, one with a short second or third.  Against the f64 oracle; the sums are f32 over at most 336 runs, worst case
2e-5 of the summed magnitudes, for sums of random sign well below 1e-5 of the result's norm."""
import pytest
import torch

from oracle import frink_oracle as fo
from tests.helpers import rel_l2, synth_acts, synth_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 301])
@pytest.mark.parametrize("cols", [256, 3840, 4096, 4352, 8192, 8448, 10752])
def test_passes_over_x(rows, cols):
    from frink_b200 import device
    raw, x = fo.encode(fo.Q4_K, synth_weights(rows, cols, 97)), synth_acts(1, cols, 98)
    w, xd = device.Weights(raw, fo.Q4_K, rows, cols), torch.from_numpy(x).cuda()
    y = device.gemv(w, xd)
    assert rel_l2(y.cpu().numpy(), fo.matmul_f64(fo.Q4_K, raw, rows, cols, fo.q8_1_round(x))) <= 1e-5
    assert torch.equal(y, device.gemv(w, xd)) and device.device_error() == 0
