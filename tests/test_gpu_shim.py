"""The 21 functions of the reference's driver shim (cpp/cuda_shim.cpp:189-988) exercised the way the
Rust host uses them (src/main.rs:37-385): context and stream, stream-ordered alloc/free, upload and
download, a kernel object loaded from cache/kernels/<name>/kernel.cubin + meta.json, its attributes,
a launch with an array of argument pointers, and the event timer."""
import ctypes

import numpy as np
import pytest

from oracle import formats, rms_norm as o_rms

pytestmark = pytest.mark.gpu


def test_kernel_object_through_the_generic_shim(stream):
    from x17ai_b200 import device, kernel_objects
    rows, dim = 100, 4096
    rng = np.random.default_rng(5)
    x = np.ascontiguousarray(formats.f32_to_e4m3(rng.standard_normal((rows, dim)).astype(np.float32)))
    out = np.zeros((rows, dim), dtype=np.int8)
    assert stream.capability[0] == 10

    d_in, d_out = stream.alloc(x.nbytes), stream.alloc(out.nbytes)
    stream.upload(x.ctypes.data, d_in, 0, x.nbytes)
    kern = kernel_objects.CubinKernel(stream, kernel_objects.build_rms_norm(dim))
    assert kern.attrs.binary_version == 100 and kern.attrs.num_regs > 0 and kern.attrs.local_size_bytes == 0
    timer = device.CudaTimer(stream)
    timer.start()
    grid = ((rows + kernel_objects.ROWS_PER_BLOCK - 1) // kernel_objects.ROWS_PER_BLOCK, 1, 1)
    kern.launch(stream, grid, (kern.meta["THREADS_PER_BLOCK"], 1, 1), kern.meta["SMEM_BYTES"],
                ctypes.c_void_p(d_in), ctypes.c_uint64(rows), ctypes.c_void_p(d_out))
    timer.stop()
    stream.download(d_out, out.ctypes.data, 0, out.nbytes)
    stream.synchronize()
    assert 0.0 < timer.elapsed_seconds() < 1.0
    timer.destroy()
    stream.free(d_in)
    stream.free(d_out)
    kern.unload()
    d = np.abs(out.astype(np.int32) - o_rms.rms_norm_e4m3_i8(x).astype(np.int32))
    assert d.max() <= 1 and (d > 0).mean() <= 2e-3


def test_shim_error_paths(stream, lib):
    from x17ai_b200 import X17Error, _lib
    with pytest.raises(X17Error, match="cuModuleLoad"):
        _lib.unwrap(lib.x17ai_cuda_load_module(stream.ctx, b"/nonexistent/kernel.cubin"))
    with pytest.raises(X17Error, match="device ID out of range"):
        _lib.unwrap(lib.x17ai_cuda_open_context(4096))
    from x17ai_b200 import kernel_objects
    kern = kernel_objects.CubinKernel(stream, kernel_objects.build_rms_norm(512))
    with pytest.raises(X17Error, match="grid dimensions are out of range"):
        kern.launch(stream, (0, 1, 1), (256, 1, 1), 0, ctypes.c_void_p(0), ctypes.c_uint64(0), ctypes.c_void_p(0))
    with pytest.raises(X17Error, match="cuModuleGetFunction"):
        _lib.unwrap(lib.x17ai_cuda_get_kernel(kern.module, b"no_such_kernel", 0))
    kern.unload()


_TWO_CONTEXTS = """
import ctypes
import numpy as np
from x17ai_b200 import _lib, device

lib, cu = _lib.load(), ctypes.CDLL("libcuda.so.1")
H, S, D, M = 4, 256, 128, 300
rng = np.random.default_rng(0)
codes = lambda *s: rng.integers(-20, 20, s, dtype=np.int8)
q, kv, sk, temp, w = codes(S, H * D), codes(S, 2 * H * D), codes(H, D), np.ones(H, np.float32), codes(512, H * D)
attn = _lib.AttnConfig(H, D, H * D, 2 * H * D, H * D)
gemm = _lib.GemmConfig(0x31, 0x31, 0x51, 0, H * D, 512, 1.0, 1.0, 0.0, 0)

def launches(h):
    bufs = []
    def up(a):
        bufs.append(_lib.unwrap(lib.x17ai_cuda_alloc(h, a.nbytes)))
        _lib.check(lib.x17ai_cuda_upload_data(h, a.ctypes.data, bufs[-1], 0, a.nbytes))
        return bufs[-1]
    outs = [np.zeros((S, H * D), np.int8), np.zeros((S, 512), np.int32), np.zeros((1, H * D), np.int8)]
    d = [up(a) for a in (q, kv, sk, temp, w)] + [up(o) for o in outs]
    _lib.check(lib.x17ai_b200_attn_fwd_i8(h, ctypes.byref(attn), 1, S, d[0], d[1], d[2], d[2], d[3], d[5], None, 0))
    _lib.check(lib.x17ai_b200_gemm_fwd(h, ctypes.byref(gemm), d[0], S, d[4], 512, d[6], None, None))
    _lib.check(lib.x17ai_b200_attn_decode_i8_noalloc(h, ctypes.byref(attn), 1, d[0], d[1], S, S, None, d[2], d[2], d[3], d[7], None, 0, 65))
    for o, p in zip(outs, d[5:]):
        _lib.check(lib.x17ai_cuda_download_data(h, p, o.ctypes.data, 0, o.nbytes))
    _lib.check(lib.x17ai_cuda_synchronize(h))
    status = (ctypes.c_uint32 * 4)()
    _lib.check(lib.x17ai_b200_read_status(h, status))
    assert list(status) == [0, 0, 0, 0]
    for b in bufs:
        _lib.check(lib.x17ai_cuda_free(h, b))
    return outs

first = device.CudaStream(0)
want = launches(first.handle)
assert want[1].any() and np.array_equal(want[1], q.astype(np.int32) @ w.astype(np.int32).T)
ctx, st = ctypes.c_void_p(), ctypes.c_void_p()
assert cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, 0) == 0
assert cu.cuStreamCreate(ctypes.byref(st), 1) == 0
assert cu.cuCtxPopCurrent_v2(ctypes.byref(ctypes.c_void_p())) == 0
for handle in (st.value, first.handle, st.value):
    assert all(np.array_equal(a, b) for a, b in zip(launches(handle), want))
first.close()
again = device.CudaStream(0)
assert all(np.array_equal(a, b) for a, b in zip(launches(again.handle), want))
print("same")
"""


def test_two_contexts_on_one_device():
    """A second context on the device, launches in turn from both, and the primary context opened a second time: shared
    memory limits, status words and the built-in decode scratch belong to a context. In a process without torch's CUDA."""
    import subprocess
    import sys
    from pathlib import Path
    r = subprocess.run([sys.executable, "-c", _TWO_CONTEXTS], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "same", (r.returncode, r.stdout, r.stderr[-800:])
