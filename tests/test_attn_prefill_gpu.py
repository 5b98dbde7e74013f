"""Prompt attention at each of its block heights (8, 16 or 32 query rows a block: whichever first gives two blocks per SM),
with ragged last blocks and tiles, against a float64 restatement.  The sums are f32 over at most 460 keys and the softmax
uses the same exponentials in f32: 2e-6 is the bound of the attention tests beside this one."""
import numpy as np
import pytest
import torch

from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_q,n_heads,n_kv,hd,p0", [(16, 8, 8, 128, 0), (77, 8, 2, 64, 3), (75, 64, 8, 64, 31), (150, 32, 8, 128, 0),
                                                    (301, 32, 4, 128, 0), (333, 64, 8, 64, 127), (20, 3, 1, 4, 33)])
@pytest.mark.parametrize("window", [0, 30])
def test_block_heights(n_q, n_heads, n_kv, hd, p0, window):
    from frink_b200 import device
    from tests import cpu_ops
    rng = np.random.default_rng(41 + n_q)
    rnd = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32))
    q, kc, vc = rnd(n_q, n_heads * hd), rnd(p0 + n_q, n_kv * hd), rnd(p0 + n_q, n_kv * hd)
    pos = torch.tensor([p0], dtype=torch.int32)
    want = cpu_ops.attention(q, kc, vc, n_heads, n_kv, hd, pos, window=window).numpy()
    out = device.attention(q.cuda(), kc.cuda(), vc.cuda(), n_heads, n_kv, hd, pos.cuda(), window=window)
    assert rel_l2(out.cpu().numpy(), want) <= 2e-6
    assert device.device_error() == 0


@pytest.mark.parametrize("n_q,n_heads,n_kv", [(16, 8, 8), (75, 64, 8), (150, 32, 8), (333, 64, 8)])
def test_block_heights_with_sinks(n_q, n_heads, n_kv):
    """gpt-oss's logit per head in the denominator, under its window and without one."""
    from frink_b200 import device
    from tests import cpu_ops
    rng, hd, p0 = np.random.default_rng(42 + n_q), 64, 5
    rnd = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32))
    q, kc, vc, sinks = rnd(n_q, n_heads * hd), rnd(p0 + n_q, n_kv * hd), rnd(p0 + n_q, n_kv * hd), rnd(n_heads)
    pos = torch.tensor([p0], dtype=torch.int32)
    for window in (0, 128):
        want = cpu_ops.attention(q, kc, vc, n_heads, n_kv, hd, pos, window=window, sinks=sinks).numpy()
        out = device.attention(q.cuda(), kc.cuda(), vc.cuda(), n_heads, n_kv, hd, pos.cuda(), window=window, sinks=sinks.cuda())
        assert rel_l2(out.cpu().numpy(), want) <= 2e-6
    assert device.device_error() == 0
