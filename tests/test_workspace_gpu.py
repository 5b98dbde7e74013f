"""Which calls use the context's one workspace: include/frink_b200.h names the GEMM, the batch 3..8 matvec, the split
attention and the integer hook, and lets two streams run anything else together."""
import ctypes as C

import pytest
import torch

from oracle import frink_oracle as fo
from tests.helpers import synth_acts, synth_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [fo.Q4_K, fo.Q5_K, fo.Q6_K, fo.Q8_0, fo.MXFP4])
def test_batch_of_two_is_one_launch_and_keeps_its_results_beside_a_gemm(kind):
    """One launch: no activation image in the workspace in front of it.  Its results beside a GEMM on another stream (whose
    int8 plane starts where an image would) are those it has alone, bit for bit."""
    from frink_b200 import device
    rows, cols = 1000, 2048
    w = device.Weights(fo.encode(kind, synth_weights(rows, cols, 81)), kind, rows, cols)
    big = device.Weights(fo.encode(fo.Q4_K, synth_weights(2048, cols, 82)), fo.Q4_K, 2048, cols)
    x, xb = torch.from_numpy(synth_acts(2, cols, 83)).cuda(), torch.from_numpy(synth_acts(512, cols, 84)).cuda()
    want, want_big = device.gemv(w, x), device.gemm(big, xb)
    torch.cuda.synchronize()
    device.counters(reset=True)
    device.gemv(w, x)
    assert device.counters()["launches"] == 1
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    got, got_big = [], []
    for _ in range(40):
        with torch.cuda.stream(one):
            got_big.append(device.gemm(big, xb))
        with torch.cuda.stream(two):
            got += [device.gemv(w, x) for _ in range(4)]
    torch.cuda.synchronize()
    assert all(torch.equal(y, want) for y in got) and all(torch.equal(y, want_big) for y in got_big)
    assert device.device_error() == 0


@pytest.mark.parametrize("cols,batch,launches", [(768, 1, 1), (768, 2, 1), (768, 3, 2), (3072, 8, 2), (18432, 8, 1)])
def test_q5k_takes_one_kernel_whether_or_not_there_is_a_workspace(cols, batch, launches):
    """A context's first call, under capture (where no workspace can be allocated), takes the kernels that any other call of
    the shape takes, and gives the same bits.  One launch: fk_gemv_q5k.cu; 8 x 18432 columns do not fit the other form.
    Sums of at most 576 runs in f32: worst case 3.5e-5 of the summed magnitudes, random signs well below 1e-5."""
    from frink_b200 import _lib, device
    from tests.helpers import rel_l2
    lib, rows = _lib.lib(), 40
    raw, x = fo.encode(fo.Q5_K, synth_weights(rows, cols, 85)), synth_acts(batch, cols, 86)
    xd, y = torch.from_numpy(x).cuda(), torch.zeros((batch, rows), device="cuda")
    want = device.gemv(device.Weights(raw, fo.Q5_K, rows, cols), xd)
    ctx, w, n = C.c_void_p(), C.c_void_p(), C.c_uint64()
    _lib.check(lib.fk_init(torch.cuda.current_device(), C.byref(ctx)))
    try:
        _lib.check(lib.fk_register_weights(ctx, raw.ctypes.data_as(C.c_void_p), raw.size, fo.Q5_K, 1, rows, cols, C.byref(w)))
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            _lib.check(lib.fk_gemv(ctx, device._stream(), w, 0, device._ptr(xd), batch, device._ptr(y)))
        _lib.check(lib.fk_counters(ctx, None, None, C.byref(n), 0))
        for _ in range(2):
            y.zero_()
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, want)
        assert n.value == launches
        del g
        _lib.check(lib.fk_release_weights(ctx, w))
    finally:
        lib.fk_destroy(ctx)
    assert rel_l2(want.cpu().numpy(), fo.matmul_f64(fo.Q5_K, raw, rows, cols, fo.q8_1_round(x))) <= 1e-5
    assert device.device_error() == 0
