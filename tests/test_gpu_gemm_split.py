"""The GEMM forms for few rows (K split over a cluster) against the oracle: row counts around the edges of A's box and of the
tiles, K that does not divide evenly over the cluster, N of half a tile, and every epilogue family."""
import numpy as np
import pytest
import torch

from oracle import formats, gemm as o_gemm

pytestmark = pytest.mark.gpu


def _i8(rng, shape):
    return formats.quantize_fixedi8(rng.standard_normal(shape))


def _cuda(*arrays):
    r = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]
    torch.cuda.synchronize()   # the launches run on another stream
    return r


# (m, k, n): one row; A's box of 8; just above it; the last row count of the weights-major form and the first after it; a
# whole tile; a second row tile of one row; K of one, three and 36 blocks; N of half a 256-column tile; many tiles
@pytest.mark.parametrize("m,k,n", [(1, 128, 256), (8, 384, 128), (9, 4608, 256), (33, 1024, 384), (48, 4096, 512), (49, 1024, 384),
                                   (127, 2048, 512), (128, 4096, 7168), (129, 4224, 256), (16, 2816, 7040), (3, 1024, 37888),
                                   (64, 1024, 37888)])
def test_split_accumulators_exact(stream, m, k, n):
    from x17ai_b200 import kernels as K
    rng = np.random.default_rng(m + k + n)
    a = rng.integers(-127, 128, (m, k), dtype=np.int8)
    b = rng.integers(-127, 128, (n, k), dtype=np.int8)
    ta, tb = _cuda(a, b)
    c = torch.zeros((m, n), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    K.GemmKernel(K.GemmConfig(K.DTYPE_INT8, K.DTYPE_INT8, K.DTYPE_I32_RAW, K.EPI_SCALE, k, n)).launch(stream, ta, tb, c)
    stream.synchronize()
    assert np.array_equal(c.cpu().numpy(), o_gemm.gemm_i32(a, b))


@pytest.mark.parametrize("m", [1, 17, 48, 100])
@pytest.mark.parametrize("d,heads,gate", [(128, 2, 128), (64, 4, 0), (32, 8, 256)])
def test_split_fused_projection(stream, m, d, heads, gate):
    """Per-head L2 norm whose columns are spread over the cluster, beside plain segments."""
    from x17ai_b200 import kernels as K
    rng = np.random.default_rng(m + d)
    k, hd = 2176, heads * d
    x, wq, wkv, wg = _i8(rng, (m, k)), _i8(rng, (hd, k)), _i8(rng, (2 * hd, k)), _i8(rng, (gate, k))
    tx, tw = _cuda(x, np.concatenate((wq, wkv, wg)))
    q = torch.zeros((m, hd), dtype=torch.int8, device="cuda")
    kv = torch.zeros((m, 2 * hd), dtype=torch.int8, device="cuda")
    rr = torch.zeros((m, heads), dtype=torch.float32, device="cuda")
    g = torch.zeros((m, gate), dtype=torch.int8, device="cuda") if gate else None
    torch.cuda.synchronize()
    K.qkvg_fwd_i8(stream, tx, tw, heads, d, q, kv, rr, g)
    stream.synchronize()
    assert np.array_equal(q.cpu().numpy(), o_gemm.attn_q_fwd(x, wq))
    ref_kv, ref_rr = o_gemm.attn_kv_fwd(x, wkv, d)
    dd = np.abs(kv.cpu().numpy().astype(np.int32) - ref_kv.astype(np.int32))
    # rsqrt.approx and a f32 sum of d squares: one code on a rounding tie
    assert dd.max() <= 1 and (dd > 0).mean() <= 2e-4
    assert np.max(np.abs(rr.cpu().numpy() - ref_rr) / ref_rr) < 1e-6
    if gate:
        assert np.array_equal(g.cpu().numpy(), o_gemm.attn_q_fwd(x, wg))


@pytest.mark.parametrize("m,f", [(1, 512), (33, 1024), (128, 1408)])
def test_split_ffn_pair(stream, m, f):
    """GeGLU and gated-residual epilogues, int8 and split e4m3 weights; bytes as in the other forms up to ties."""
    from x17ai_b200 import kernels as K
    rng = np.random.default_rng(m + f)
    dm = 512
    x, wf, wy = _i8(rng, (m, dm)), _i8(rng, (2 * f, dm)), _i8(rng, (2 * dm, f))
    tx, twf, twy = _cuda(x, wf, wy)
    sp = K.split_i8_weights(stream, twy)
    tf = torch.zeros((m, f), dtype=torch.uint8, device="cuda")
    ty = torch.zeros((m, dm), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    K.GemmKernel(K.ffn_f_fwd_config(dm, f)).launch(stream, tx, twf, tf)
    K.GemmKernel(K.ffn_y_fwd_f8_config(f, dm)).launch(stream, tf, sp, ty, residual=tx)
    stream.synchronize()
    got_f = tf.cpu().numpy()
    # a handful of bytes may sit on a rounding tie whatever the row count
    assert (got_f != o_gemm.ffn_f_fwd(x, wf)).sum() <= max(3, 2e-3 * got_f.size)
    got_y = ty.cpu().numpy()
    assert (got_y != o_gemm.ffn_y_fwd_f8(got_f, wy, x)).sum() <= max(3, 2e-3 * got_y.size)
