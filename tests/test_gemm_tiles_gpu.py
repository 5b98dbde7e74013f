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
    (1, 512, 9),            # one weight row, one CTA
    (130, 1280, 31), (130, 1280, 33),     # ten stages over eight parts; a 32-token tile short of one, over by one
    (640, 8192, 16),        # the deepest split
    (2100, 768, 65), (3100, 512, 129),    # wide matrices: no split, ragged 32-token tiles (Q6_K, 129 tokens: 64)
    (1030, 2048, 300)])     # 128-token tiles in two (Q6_K) or four parts
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


# ---- every tile and split, whatever the plan would pick ----
def _cols(kind, split):
    """Nine stages and more in every part (the ring of four wraps twice, the slots of the unpack warps rotate through), parts
    of unequal length, and the last stage ragged where the kind allows it."""
    return 1280 * split + (0 if kind in (fo.Q4_K, fo.Q6_K) else 32)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("tile", [32, 64, 128])
@pytest.mark.parametrize("split", [1, 2, 4, 8])
def test_given_plan(kind, tile, split):
    """Results and raw integers of a given plan on ragged rows and tokens.  At most 322 runs summed in f32 (x 2 halves for Q6_K):
    worst case 3.8e-5 of the summed magnitudes, for sums of random sign well below 1e-5 of the result's norm."""
    from frink_b200 import device
    rows, cols, m = 150, _cols(kind, split), tile + 13
    raw, x = fo.encode(kind, synth_weights(rows, cols, 101)), synth_acts(m, cols, 102)
    w, xd = device.Weights(raw, kind, rows, cols), torch.from_numpy(x).cuda()
    got = device.gemm_tiled(w, xd, tile, split)
    assert rel_l2(got.cpu().numpy(), fo.matmul_f64(kind, raw, rows, cols, fo.q8_1_round(x))) <= 1e-5
    with_ints, isums = device.gemm_tiled(w, xd, tile, split, isums=True)
    assert torch.equal(with_ints, got) and device.device_error() == 0
    for t in (0, 1, tile - 1, tile, m - 1):
        assert np.array_equal(isums[t].cpu().numpy(), fo.matrix_isums(kind, raw, rows, cols, fo.quantize_q8_1(x[t]))), f"token {t}"
    # the order of the sums follows the split alone: not the tile, nor how many tokens are in the call
    assert torch.equal(device.gemm_tiled(w, xd[:9], 32, split), got[:9])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("tile,split", [(32, 1), (64, 1), (128, 1), (32, 4), (64, 2), (128, 2)])
def test_given_plan_grouped(kind, tile, split):
    """Experts with no row, one row, one over a tile; columns as above."""
    from frink_b200 import device
    rows, cols, sizes = 150, _cols(kind, split), [0, 1, tile + 1, 0, 7, tile]
    pairs = sum(sizes)
    raws = [fo.encode(kind, synth_weights(rows, cols, 110 + e)) for e in range(len(sizes))]
    w = device.Weights(np.concatenate(raws), kind, rows, cols, n_mats=len(sizes))
    x = synth_acts(40, cols, 103)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    gather = np.random.default_rng(104).integers(0, 40, pairs).astype(np.int32)
    xd, offd, gd = torch.from_numpy(x).cuda(), torch.from_numpy(off).cuda(), torch.from_numpy(gather).cuda()
    got = device.gemm_tiled(w, xd, tile, split, group_off=offd, gather=gd, pairs=pairs).cpu().numpy()
    assert device.device_error() == 0
    xq = fo.q8_1_round(x)
    for e in range(len(sizes)):
        lo, hi = off[e], off[e + 1]
        if hi > lo:
            assert rel_l2(got[lo:hi], fo.matmul_f64(kind, raws[e], rows, cols, xq[gather[lo:hi]])) <= 1e-5, e


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rows,cols,m", [(8192, 512, 512), (1030, 2048, 300), (640, 2048, 16), (2100, 768, 65)])
def test_the_call_runs_its_plan(kind, rows, cols, m):
    from frink_b200 import _lib, device
    w = device.Weights(fo.encode(kind, synth_weights(rows, cols, 105)), kind, rows, cols)
    x = torch.from_numpy(synth_acts(m, cols, 106)).cuda()
    tile, split = device.gemm_plan(w, m)
    assert tile in (32, 64, 128) and split in (1, 2, 4, 8) and split * 128 <= cols
    want = device.gemm_tiled(w, x, tile, split)
    assert torch.equal(device.gemm(w, x), want) and torch.equal(device.gemm_static(w, x), want)
    for bad in ((48, 1), (32, 3), (32, 16), (32, 0)):
        with pytest.raises(_lib.Invalid):
            device.gemm_tiled(w, x, *bad)
    assert device.device_error() == 0


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rows,cols,m", [(300, 1280, 33), (2100, 768, 65), (1030, 2048, 300)])
def test_captured_and_replayed(kind, rows, cols, m):
    """Two launches per call, the second under the first; in a graph, with new inputs between replays."""
    from frink_b200 import device
    w = device.Weights(fo.encode(kind, synth_weights(2 * rows, cols, 107)), kind, rows, cols, n_mats=2)
    xs = [torch.from_numpy(synth_acts(m, cols, 108 + i)).cuda() for i in range(3)]
    off = torch.tensor([0, m // 3, m], dtype=torch.int32, device="cuda")
    calls = [lambda v, y: device.gemm(w, v, mat=1, out=y), lambda v, y: device.gemm_static(w, v, mat=1, out=y),
             lambda v, y: device.gemm_grouped(w, off, None, v, m, out=y)]
    for call in calls:
        want = [call(v, None).clone() for v in xs]
        x, y = xs[0].clone(), torch.empty((2, m, rows), device="cuda")
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            call(x, y[0])
            call(x, y[1])        # the second call's quantizer writes the block that the first call's GEMM reads
        for v, ref in zip(xs[1:] + xs[:1], want[1:] + want[:1]):
            x.copy_(v)
            y.fill_(float("nan"))
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(y[0], ref) and torch.equal(y[1], ref)
    assert device.device_error() == 0
