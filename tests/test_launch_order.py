"""Launches behind one another on one stream: a kernel's set-up runs under the tail of the kernel in front of it, so its
inputs are written during its lifetime."""
from pathlib import Path

import numpy as np
import pytest
import torch

from oracle import formats

CSRC = Path(__file__).resolve().parent.parent / "x17ai_b200" / "csrc"


def test_no_read_only_loads():
    """ld.global.nc (and __ldg, which issues it) may be moved above the wait for the kernel in front and need not see its
    writes."""
    for path in sorted(CSRC.rglob("*.cu*")):
        code = "\n".join(line.split("//")[0] for line in path.read_text().splitlines())
        assert "__ldg" not in code and "ld.global.nc" not in code, path.name


@pytest.mark.gpu
def test_norm_reads_the_gemm_in_front(stream):
    """Gated-residual GEMM -> RMSNorm over the same two buffers, inputs changing from pass to pass, nothing waited for in
    between: every pass gives the bytes of the pass that is waited for."""
    from x17ai_b200 import kernels as K
    rng = np.random.default_rng(3)
    m, d, n = 640, 1024, 40
    codes = lambda *s: torch.from_numpy(formats.quantize_fixedi8(rng.standard_normal(s))).cuda()
    a, w, res = [codes(m, d) for _ in range(3)], codes(2 * d, d), codes(m, d)
    kern = K.GemmKernel(K.attn_y_fwd_config(d, d))
    y = torch.zeros((m, d), dtype=torch.uint8, device="cuda")
    outs = torch.zeros((n, m, d), dtype=torch.int8, device="cuda")
    want = torch.zeros((3, m, d), dtype=torch.int8, device="cuda")
    torch.cuda.synchronize()
    for i in range(3):
        kern.launch(stream, a[i], w, y, residual=res)
        stream.synchronize()
        K.rms_norm(stream, K.RMS_E4M3_FIXED, y, want[i])
        stream.synchronize()
    for i in range(n):
        kern.launch(stream, a[i % 3], w, y, residual=res)
        K.rms_norm(stream, K.RMS_E4M3_FIXED, y, outs[i])
    stream.synchronize()
    assert all(torch.equal(outs[i], want[i % 3]) for i in range(n))


@pytest.mark.gpu
@pytest.mark.parametrize("splits", [1, 4])
def test_decode_reads_what_torch_wrote_in_front(splits):
    """Cache rows, query and temperature written by torch on the same stream right in front of the decode."""
    from x17ai_b200 import device, kernels as K
    rng = np.random.default_rng(4)
    b, h, d, t, n = 4, 4, 128, 700, 30
    codes = lambda *s: torch.from_numpy(formats.quantize_fixedi8(rng.standard_normal(s))).cuda()
    src = [(codes(b, t, 2 * h * d), codes(b, h * d), torch.rand(h, device="cuda") + 0.5) for _ in range(3)]
    sk, sv = codes(h, d), codes(h, d)
    kern = K.AttnKernel(K.AttnKernelConfig(h, d, h * d, 2 * h * d, h * d))
    cache, q, temp = (torch.zeros_like(x) for x in src[0])
    outs = torch.zeros((n, b, h * d), dtype=torch.int8, device="cuda")
    want = torch.zeros((3, b, h * d), dtype=torch.int8, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        st = device.TorchStream()
        for i in range(3):
            kern.decode(st, src[i][1], src[i][0], t, sk, sv, src[i][2], want[i], n_splits=splits)
            side.synchronize()
        for i in range(n):
            for dst, x in zip((cache, q, temp), src[i % 3]):
                dst.copy_(x)
            kern.decode(st, q, cache, t, sk, sv, temp, outs[i], n_splits=splits)
    side.synchronize()
    assert st.read_status() == [0, 0, 0, 0]
    assert all(torch.equal(outs[i], want[i % 3]) for i in range(n))


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
