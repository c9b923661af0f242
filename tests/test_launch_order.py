"""Launches behind one another on one stream: a kernel's set-up runs under the tail of the kernel in front of it, so its
CTAs start while others are still leaving."""
import numpy as np
import pytest
import torch

from oracle import formats


@pytest.mark.gpu
def test_layers_behind_one_another(stream):
    """Two hundred layers queued without a wait: kernels of CTA pairs start on SMs that the kernel in front leaves one by
    one. Every wait ends, and the last pass gives the bytes of the first."""
    from x17ai_b200.block import BlockConfig, BlockForward
    rng = np.random.default_rng(8)
    m, dm, h, d, f = 4096, 1024, 16, 64, 4096
    codes = lambda *s: torch.from_numpy(formats.quantize_fixedi8(rng.standard_normal(s))).cuda()
    w = [codes(*s) for s in ((h * d, dm), (2 * h * d, dm), (2 * dm, h * d), (2 * f, dm), (2 * dm, f))]
    x = torch.randn(m, dm, device="cuda").clamp_(0.05, 4.0).to(torch.float8_e4m3fn).view(torch.uint8)
    sk, sv, temp = codes(h, d), codes(h, d), torch.rand(h, device="cuda") + 0.5
    torch.cuda.synchronize()
    blk = BlockForward(stream, BlockConfig(dm, h, d, f, 512), *w, sk, sv, temp, fused_qkv=True)
    out = blk.forward_layer(x)
    stream.synchronize()
    first = {k: v.clone() for k, v in out.items()}
    torch.cuda.synchronize()
    for _ in range(200):
        out = blk.forward_layer(x)
    stream.synchronize()
    assert all(torch.equal(out[k], first[k]) for k in first)
