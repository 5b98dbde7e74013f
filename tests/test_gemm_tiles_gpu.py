"""The GEMM's tile plan: token tiles of 128, 64 and 32 columns and 1 to 8 CTAs along K, at the sizes where a tile or a
part of K is ragged, against the f64 oracle.  The sums are f32 over at most 256 runs (x 2 halves for Q6_K), so the
relative error is below runs * 2^-24 = 1.5e-5 of the summed magnitudes even if every rounding went one way, and well
below 1e-5 of the result's norm for sums of random sign."""
import numpy as np
import pytest
import torch

from oracle import frink_oracle as fo
from tests.helpers import rel_l2, synth_acts, synth_weights

pytestmark = pytest.mark.gpu
KINDS = [fo.Q8_0, fo.Q4_K, fo.Q6_K, fo.MXFP4]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rows,cols,m", [
    (1, 512, 9),            # one weight row, two to four stages over the parts
    (130, 1280, 31), (130, 1280, 33),     # ten stages over eight parts; a 32-token tile short of one, over by one
    (640, 8192, 16),        # the deepest split
    (2100, 768, 65), (3100, 512, 129),    # wide matrices: no split, ragged 64- and 128-token tiles
    (1030, 2048, 300)])
def test_tiles_and_parts_of_k(kind, rows, cols, m):
    from frink_b200 import device
    raw = fo.encode(kind, synth_weights(rows, cols, 31 + rows))
    x = synth_acts(m, cols, 32 + m)
    w = device.Weights(raw, kind, rows, cols)
    out = torch.full((m + 1, rows), float("nan"), device="cuda")
    device.gemm(w, torch.from_numpy(x).cuda(), out=out[:m])
    torch.cuda.synchronize()
    assert device.device_error() == 0
    assert torch.isnan(out[m]).all(), "a padding row was written"
    want = fo.matmul_f64(kind, raw, rows, cols, fo.q8_1_round(x))
    assert rel_l2(out[:m].cpu().numpy(), want) <= 1e-5
    again = device.gemm(w, torch.from_numpy(x).cuda())
    assert torch.equal(again, out[:m]), "the parts of K are summed in a fixed order"
    assert torch.equal(device.gemm_static(w, torch.from_numpy(x).cuda()), again)


@pytest.mark.parametrize("kind", KINDS)
def test_integers_of_split_tiles(kind):
    from frink_b200 import device
    rows, cols, m = 70, 2304 if kind in (fo.Q4_K, fo.Q6_K) else 2336, 40
    raw = fo.encode(kind, synth_weights(rows, cols, 41))
    x = synth_acts(m, cols, 42)
    w = device.Weights(raw, kind, rows, cols)
    _, isums = device.gemm_isums(w, torch.from_numpy(x).cuda())
    got = isums.cpu().numpy()
    assert device.device_error() == 0
    for t in range(m):
        assert np.array_equal(got[t], fo.matrix_isums(kind, raw, rows, cols, fo.quantize_q8_1(x[t]))), f"token {t}"


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n_exp,rows,cols,batch,k", [(64, 96, 512, 12, 4), (4, 300, 1280, 150, 2), (3, 1100, 512, 260, 3)])
def test_grouped_tiles(kind, n_exp, rows, cols, batch, k):
    from frink_b200 import device
    rng = np.random.default_rng(51)
    raws = [fo.encode(kind, synth_weights(rows, cols, 600 + e)) for e in range(n_exp)]
    w = device.Weights(np.concatenate(raws), kind, rows, cols, n_mats=n_exp)
    x = synth_acts(batch, cols, 52)
    ids = np.stack([rng.choice(n_exp, k, replace=False) for _ in range(batch)]).astype(np.int32)
    off, gather, _ = device.moe_permute(torch.from_numpy(ids).cuda(), n_exp)
    got = device.gemm_grouped(w, off, gather, torch.from_numpy(x).cuda(), batch * k).cpu().numpy()
    assert device.device_error() == 0
    off_h, gather_h = off.cpu().numpy(), gather.cpu().numpy()
    xq = fo.q8_1_round(x)
    for e in range(n_exp):
        lo, hi = off_h[e], off_h[e + 1]
        if hi > lo:
            assert rel_l2(got[lo:hi], fo.matmul_f64(kind, raws[e], rows, cols, xq[gather_h[lo:hi]])) <= 1e-5, e
