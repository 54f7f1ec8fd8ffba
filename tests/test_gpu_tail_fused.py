"""GPU test of the one-kernel tail network: its TOD equals the layer-by-layer
path's outputs bit for bit at the edges of its 128-sample tiles, with fewer and
more tiles than resident CTAs, and over widths, depths and output counts."""

import numpy as np
import pytest
import torch

from tod_generation_mapbased_beam_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("F,H,D,O,B", [
    (64, 128, 1, 1, 1), (64, 128, 2, 3, 127), (128, 128, 3, 4, 129), (256, 128, 2, 2, 50_001),
    (64, 256, 2, 4, 128), (192, 256, 3, 2, 255), (256, 256, 4, 3, 37_889), (256, 256, 1, 1, 76_033),
    (320, 256, 2, 3, 300),  # more frequencies than the fused operand holds: layer by layer
])
def test_fused_tail_equals_layers_bit_for_bit(F, H, D, O, B, dtype):
    from tod_generation_mapbased_beam_b200 import tailnet

    lib = _native.lib()
    net = tailnet.TailNet(F, H, D, O, sigma=(2.0, 1.0), seed=3)
    rng = np.random.default_rng(B)
    th, ph, ps = (torch.from_numpy(a).to(dtype).cuda() for a in (
        np.arccos(rng.uniform(-1, 1, B)), rng.uniform(-9, 9, B), rng.uniform(-9, 9, B)))
    net.scale, net.shift = np.ones(O), np.zeros(O)
    y = net.forward(net.inputs(th, ph, ps))[:B].double()
    tod = torch.zeros((O + 1, B), dtype=torch.float64, device="cuda")
    n0 = lib.todgpu_mlp_tcgen05_launches()
    net.accumulate(th, ph, ps, tod, rows=tuple(range(O, 0, -1)))
    assert lib.todgpu_mlp_tcgen05_launches() == n0 + D
    assert lib.todgpu_mlp_wait_timeouts() == 0
    assert torch.equal(tod[1:].flip(0), y.T)
    assert not tod[0].any()
