"""The native launch path (csrc/hostcall.cpp) on arguments whose attributes cannot be read: the launchers raise, as their Python
checks do, and the process goes on."""
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
