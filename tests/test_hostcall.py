"""The native launch path (csrc/hostcall.cpp): on arguments whose attributes cannot be read the launchers raise, as their Python
checks do, and the process goes on; without it they launch through those checks."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent

_CALLS = """
import torch
from x17ai_b200 import kernels as K

class Unreadable(torch.Tensor):
    @staticmethod
    def __new__(cls, dtype, *shape):
        return torch.Tensor._make_wrapper_subclass(cls, shape, dtype=dtype, device="cuda", dispatch_sizes_strides_policy="sizes")
    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        raise RuntimeError("unreadable")

class Stream:
    handle = 1 << 40    # never reached

t = lambda dtype, *shape: Unreadable(dtype, *shape)
i8, f32, bf16 = torch.int8, torch.float32, torch.bfloat16
q, kv, s, temp, out = t(i8, 16, 128), t(i8, 16, 256), t(i8, 2, 64), t(f32, 2), t(i8, 16, 128)
attn = K.AttnKernel(K.AttnKernelConfig(2, 64, 128, 256, 128))
gemm = K.GemmKernel(K.GemmConfig(K.DTYPE_INT8, K.DTYPE_INT8, K.DTYPE_INT8, K.EPI_SCALE, 128, 128))
st, sc = Stream(), t(f32, 2, 16)
calls = dict(
    attn=lambda: attn.launch(st, q, kv, s, s, temp, out),
    attn_pv_fp8=lambda: attn.launch_pv_fp8(st, q, kv, s, t(torch.uint8, 2, 64), temp, temp, t(bf16, 16, 128)),
    attn_scaled=lambda: attn.launch_scaled(st, q, sc, kv, sc, sc, s, s, temp, t(bf16, 16, 128)),
    decode=lambda: attn.decode(st, q, t(i8, 16, 32, 256), 20, s, s, temp, out),
    gemm=lambda: gemm.launch(st, q, t(i8, 128, 128), out),
    qkvg=lambda: K.qkvg_fwd_i8(st, q, t(i8, 768, 128), 4, 64, t(i8, 16, 256), t(i8, 16, 512), t(f32, 16, 4)),
    rms_norm=lambda: K.rms_norm(st, K.RMS_BF16_FIXED, t(bf16, 16, 128), out),
)
for name, call in calls.items():
    try:
        call()
    except RuntimeError as e:
        print("raised", name, flush=True)
"""


def test_unreadable_tensors_raise():
    r = subprocess.run([sys.executable, "-c", _CALLS], cwd=ROOT, capture_output=True, text=True, timeout=120)
    names = ["attn", "attn_pv_fp8", "attn_scaled", "decode", "gemm", "qkvg", "rms_norm"]
    assert r.returncode == 0 and r.stdout.split("\n")[:-1] == [f"raised {n}" for n in names], (r.returncode, r.stdout, r.stderr[-500:])


@pytest.mark.gpu
def test_sparse_tensors_raise(stream):
    from x17ai_b200 import kernels as K
    x = torch.ones((4, 512), dtype=torch.uint8).to_sparse_csr().cuda()
    with pytest.raises(RuntimeError):
        K.rms_norm(stream, K.RMS_E4M3_FIXED, x, torch.zeros((4, 512), dtype=torch.int8, device="cuda"))


@pytest.fixture(params=["missing", "another torch"])
def no_native_path(request, monkeypatch):
    import types
    import x17ai_b200
    from x17ai_b200 import _lib
    mod = types.SimpleNamespace(built_for="torch 0.1;") if request.param == "another torch" else None
    monkeypatch.setattr(_lib, "_hostcall", None)
    monkeypatch.setitem(sys.modules, "x17ai_b200._hostcall", mod)
    monkeypatch.delattr(x17ai_b200, "_hostcall", raising=False)
    if mod is not None:
        monkeypatch.setattr(x17ai_b200, "_hostcall", mod, raising=False)


def test_kernels_without_the_native_path(no_native_path):
    from x17ai_b200 import X17Error, kernels as K
    with pytest.warns(RuntimeWarning, match="native launch path"):
        kern = K.GemmKernel(K.attn_q_fwd_config(128, 128))
    t = torch.zeros((16, 64), dtype=torch.int8)
    with pytest.raises(X17Error, match="64 columns, but should have 128"):
        kern.launch(type("Stream", (), {"handle": 1})(), t, t, t)


@pytest.mark.gpu
def test_launches_without_the_native_path(stream, no_native_path):
    from x17ai_b200 import kernels as K
    x = torch.randn(16, 512, device="cuda").to(torch.bfloat16)
    outs = [torch.zeros((16, 512), dtype=torch.int8, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    with pytest.warns(RuntimeWarning, match="native launch path"):
        K.rms_norm(stream, K.RMS_BF16_FIXED, x, outs[0])
    K.rms_norm(stream, K.RMS_BF16_FIXED, x, outs[1])
    stream.synchronize()
    assert outs[0].any() and torch.equal(*outs)


@pytest.mark.gpu
def test_a_replaced_config_is_the_one_that_launches(stream):
    from x17ai_b200 import X17Error, kernels as K
    x, w = (torch.randint(-9, 9, s, dtype=torch.int8, device="cuda") for s in ((16, 128), (256, 128)))
    outs = [torch.zeros((16, 256), dtype=torch.int8, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    kern = K.GemmKernel(K.attn_q_fwd_config(128, 128))
    kern.config = K.attn_q_fwd_config(128, 256)
    kern.launch(stream, x, w, outs[0])
    K.GemmKernel(K.attn_q_fwd_config(128, 256)).launch(stream, x, w, outs[1])
    stream.synchronize()
    assert outs[0].any() and torch.equal(*outs)
    with pytest.raises(X17Error, match="256 rows, but should have 128"):
        kern.config = K.attn_q_fwd_config(128, 128)
        kern.launch(stream, x, w, outs[0])
