"""What the q8_1 GEMM's entry points take as x: any 4-byte aligned view, and NaN and infinity, which have to
reach the output; and what the fixed block of fk_gemm_static holds."""
import numpy as np
import pytest
import torch

from oracle import frink_oracle as fo
from tests.helpers import synth_acts, synth_weights

pytestmark = pytest.mark.gpu
KINDS = [fo.Q8_0, fo.Q4_K, fo.Q6_K, fo.MXFP4]


def _off(x, n):
    """A copy of x that starts n floats behind a 16-byte boundary."""
    v = torch.empty(x.numel() + n, device="cuda")[n:].view(x.shape)
    assert v.data_ptr() % 16 == 4 * n
    return v.copy_(x)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("off", [1, 2, 3])
def test_x_off_a_16_byte_boundary(kind, off):
    """The same values at another address: the same bits out."""
    from frink_b200 import device
    rows, cols, m, n_exp = 130, 768, 19, 3
    w = device.Weights(fo.encode(kind, synth_weights(n_exp * rows, cols, 91)), kind, rows, cols, n_mats=n_exp)
    x = torch.from_numpy(synth_acts(m, cols, 92)).cuda()
    ids = torch.from_numpy(np.arange(2 * m, dtype=np.int32).reshape(m, 2) % n_exp).cuda()
    group, gather, _ = device.moe_permute(ids, n_exp)
    for f in (lambda v: device.gemm(w, v, mat=1), lambda v: device.gemm_static(w, v, mat=1),
              lambda v: device.gemm_grouped(w, group, gather, v, 2 * m)):
        assert torch.equal(f(_off(x, off)), f(x))
    assert device.device_error() == 0


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_nan_and_infinity_reach_the_output(kind, bad):
    """A run's scale is the largest magnitude's: NaN or infinite, and so is every output of that token.  Infinity times the
    codes of the run's finite values, 0, is NaN.  The other tokens keep their bits."""
    from frink_b200 import device
    rows, cols, m, n_exp = 130, 768, 19, 3
    w = device.Weights(fo.encode(kind, synth_weights(n_exp * rows, cols, 93)), kind, rows, cols, n_mats=n_exp)
    clean = torch.from_numpy(synth_acts(m, cols, 94)).cuda()
    ids = torch.from_numpy(np.arange(2 * m, dtype=np.int32).reshape(m, 2) % n_exp).cuda()
    group, gather, _ = device.moe_permute(ids, n_exp)
    hit = torch.zeros(m, dtype=torch.bool, device="cuda")
    x = clean.clone()
    for t, c in ((0, 0), (7, 33), (18, 767), (18, 2)):      # each place in a lane's four values
        x[t, c] = bad
        hit[t] = True
    for f, mask in ((lambda v: device.gemm(w, v, mat=2), hit), (lambda v: device.gemm_static(w, v, mat=2), hit),
                    (lambda v: device.gemm_grouped(w, group, gather, v, 2 * m), hit[gather.long()])):
        got, want = f(x), f(clean)
        assert torch.isnan(got[mask]).all()
        assert torch.equal(got[~mask], want[~mask])
    assert device.device_error() == 0


@pytest.mark.parametrize("m,cols,fits", [(9600, 512, True), (9601, 512, False), (512, 9824, True), (513, 9824, False), (128, 39296, True), (128, 39328, False)])
def test_what_the_fixed_block_holds(m, cols, fits):
    """m padded to 128: m * cols bytes of codes, two scales of 4 bytes a run of 32 (each plane rounded to 1 KB) and two
    words a row, in 6 MiB."""
    from frink_b200 import _lib, device
    w = device.Weights(fo.encode(fo.Q8_0, synth_weights(8, cols, 95)), fo.Q8_0, 8, cols)
    x, y = torch.from_numpy(synth_acts(m, cols, 96)).cuda(), torch.zeros((m, 8), device="cuda")
    if fits:
        assert torch.equal(device.gemm_static(w, x, out=y), device.gemm(w, x))
    else:
        with pytest.raises(_lib.Invalid):
            device.gemm_static(w, x, out=y)
        torch.cuda.synchronize()
        assert not y.any()
    assert device.device_error() == 0
