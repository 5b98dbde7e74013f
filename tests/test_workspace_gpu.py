"""Which calls use the context's one workspace: include/frink_b200.h names the GEMM, the batch 3..8 matvec, the split
attention and the integer hook, and lets two streams run anything else together."""
import numpy as np
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
