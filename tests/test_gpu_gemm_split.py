"""The GEMM forms for few rows (K split over a cluster) against the oracle: row counts around the edges of A's box and of the
tiles, K that does not divide evenly over the cluster, N of half a tile; and the default dispatch with every epilogue, against
the one-CTA form on both sides of the dispatch's lines and against the oracle."""
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


# ---- every epilogue in the default dispatch ----------------------------------------------------------

KINDS = ("scale", "raw", "kv32", "kv64", "kv128", "geglu", "resid_e4m3", "resid_i8", "f8_raw", "f8_resid", "e4m3_geglu", "e4m3_resid")


def _gemm_case(K, kind, m, n, k, g):
    """(config, a, b, c, rrms, residual) on the GPU."""
    i8 = lambda *s: torch.randn(*s, generator=g, device="cuda").mul_(8.0).round_().clamp_(-127, 127).to(torch.int8)
    def f8(*s):   # without subnormal codes, which the reference's e4m3 (the f8 kinds' activations) reads differently
        x = torch.randn(*s, generator=g, device="cuda")
        return torch.where(x.abs() < 2.0 ** -6, 0.0, x).to(torch.float8_e4m3fn).view(torch.uint8)
    new = lambda dtype, *s: torch.zeros(s, dtype=dtype, device="cuda")
    half, d = n // 2, int(kind[2:]) if kind.startswith("kv") else 0
    cfg, c = {
        "scale": lambda: (K.attn_q_fwd_config(k, n), new(torch.int8, m, n)),
        "raw": lambda: (K.GemmConfig(K.DTYPE_INT8, K.DTYPE_INT8, K.DTYPE_I32_RAW, K.EPI_SCALE, k, n), new(torch.int32, m, n)),
        "geglu": lambda: (K.ffn_f_fwd_config(k, half), new(torch.uint8, m, half)),
        "resid_e4m3": lambda: (K.attn_y_fwd_config(k, half), new(torch.uint8, m, half)),
        "resid_i8": lambda: (K.ffn_y_fwd_i8_config(k, half), new(torch.int8, m, half)),
        "f8_raw": lambda: (K.GemmConfig(K.DTYPE_E4M3, K.DTYPE_INT8, K.DTYPE_I32_RAW, K.EPI_SCALE, k, n), new(torch.int32, m, n)),
        "f8_resid": lambda: (K.ffn_y_fwd_f8_config(k, half), new(torch.uint8, m, half)),
        "e4m3_geglu": lambda: (K.ffn_f_fwd_e4m3_config(k, half, 1.0, k ** -0.5), new(torch.uint8, m, half)),
        "e4m3_resid": lambda: (K.ffn_y_fwd_e4m3_config(k, half, k ** -0.5), new(torch.uint8, m, half)),
    }.get(kind, lambda: (K.attn_kv_fwd_config(k, n, d), new(torch.int8, m, n)))()
    a = f8(m, k) if "f8" in kind or kind.startswith("e4m3") else i8(m, k)
    b = f8(n, k) if kind.startswith("e4m3") else i8(n, k)
    return cfg, a, b, c, new(torch.float32, m, n // (2 * d)) if d else None, i8(m, half) if "resid" in kind else None


def _launch_case(K, stream, cfg, a, b, c, rrms, residual):
    torch.cuda.synchronize()
    if cfg.a_dtype == K.DTYPE_E4M3 and cfg.b_dtype == K.DTYPE_INT8:
        b = K.split_i8_weights(stream, b)
    K.GemmKernel(cfg).launch(stream, a, b, c, rrms=rrms, residual=residual)
    stream.synchronize()
    return c.clone(), None if rrms is None else rrms.clone()


def _same_as(kind, got, want, k):
    """int8 x int8: the same bytes in every form. e4m3: f32 sums in another order, bytes on a rounding tie may differ."""
    (c, rr), (cw, rw) = got, want
    if kind == "f8_raw":
        x, y = c.view(torch.float32).double(), cw.view(torch.float32).double()
        assert (x - y).abs().max() <= 1e-5 * k ** 0.5 * y.abs().max()
    elif kind.startswith(("f8", "e4m3")):
        assert (c != cw).sum() <= max(3, 2e-3 * c.numel())
    else:
        assert torch.equal(c, cw) and (rr is None or torch.equal(rr, rw))


# row counts on both sides of every line of the dispatch; K on both sides of them; one tile, a few, more than half the chip
@pytest.mark.parametrize("m", [1, 32, 33, 48, 49, 64, 65, 112, 128, 129, 257])
@pytest.mark.parametrize("kind", KINDS)
def test_default_dispatch_equals_one_cta(stream, kind, m):
    from x17ai_b200 import kernels as K
    g = torch.Generator(device="cuda").manual_seed(m)
    for n, k in ((256, 256), (768, 1024), (2048, 1024), (2048, 2048), (8192, 1024), (512, 4224), (256, 8320), (20480, 512)):
        case = _gemm_case(K, kind, m, n, k, g)
        got = _launch_case(K, stream, *case)
        K.set_gemm_tiling(K.GEMM_ONE_CTA)
        try:
            want = _launch_case(K, stream, *case)
        finally:
            K.set_gemm_tiling()
        _same_as(kind, got, want, k)


@pytest.mark.parametrize("m", [33, 49, 128, 200])
@pytest.mark.parametrize("d,heads,gate,k", [(128, 2, 128, 4224), (128, 8, 0, 2048), (64, 8, 256, 4096), (32, 64, 0, 1024)])
def test_default_dispatch_equals_one_cta_qkvg(stream, d, heads, gate, k, m):
    from x17ai_b200 import kernels as K
    rng = np.random.default_rng(m + d)
    hd = heads * d
    tx, tw = _cuda(_i8(rng, (m, k)), _i8(rng, (3 * hd + gate, k)))
    outs = []
    for tiling in (K.GEMM_AUTO, K.GEMM_ONE_CTA):
        q, kv = torch.zeros((m, hd), dtype=torch.int8, device="cuda"), torch.zeros((m, 2 * hd), dtype=torch.int8, device="cuda")
        rr = torch.zeros((m, heads), dtype=torch.float32, device="cuda")
        g = torch.zeros((m, gate), dtype=torch.int8, device="cuda") if gate else None
        torch.cuda.synchronize()
        K.set_gemm_tiling(tiling)
        try:
            K.qkvg_fwd_i8(stream, tx, tw, heads, d, q, kv, rr, g)
            stream.synchronize()
        finally:
            K.set_gemm_tiling()
        outs.append([t for t in (q, kv, rr, g) if t is not None])
    assert all(torch.equal(a, b) for a, b in zip(*outs))


# against the oracle: the weights-major form (33, 48 rows), the split form up to a tile and beyond it; K of 33 blocks
@pytest.mark.parametrize("m", [1, 33, 48, 49, 128, 130])
@pytest.mark.parametrize("kind", ["scale", "kv32", "kv64", "resid_e4m3", "resid_i8", "geglu", "f8_resid", "e4m3_geglu", "e4m3_resid"])
def test_default_dispatch_vs_oracle(stream, kind, m):
    from x17ai_b200 import kernels as K
    n, k = 384, 4224
    case = _gemm_case(K, kind, m, n, k, torch.Generator(device="cuda").manual_seed(m + 7))
    c, rr = _launch_case(K, stream, *case)
    _, a, b, _, _, res = [x.cpu().numpy() if isinstance(x, torch.Tensor) else x for x in case]
    got = c.cpu().numpy()
    if kind == "scale":
        assert np.array_equal(got, o_gemm.attn_q_fwd(a, b))
    elif kind.startswith("kv"):
        ref, ref_rr = o_gemm.attn_kv_fwd(a, b, int(kind[2:]))
        dd = np.abs(got.astype(np.int32) - ref.astype(np.int32))
        assert dd.max() <= 1 and (dd > 0).mean() <= 2e-4    # rsqrt.approx: one code on a rounding tie
        assert np.max(np.abs(rr.cpu().numpy() - ref_rr) / ref_rr) < 1e-6
    else:
        ref = {"resid_e4m3": lambda: o_gemm.attn_y_fwd(a, b, res), "resid_i8": lambda: o_gemm.ffn_y_fwd_i8(a, b, res),
               "geglu": lambda: o_gemm.ffn_f_fwd(a, b), "f8_resid": lambda: o_gemm.ffn_y_fwd_f8(a, b, res),
               "e4m3_geglu": lambda: o_gemm.ffn_f_fwd_e4m3(a, 1.0, b, k ** -0.5),
               "e4m3_resid": lambda: o_gemm.ffn_y_fwd_e4m3(a, b, k ** -0.5, res)}[kind]()
        # approximate tanh, exp2 and log2 against libm, f32 sums against 64 bits: bytes on rounding ties
        assert (got != ref).sum() <= max(3, 2e-3 * got.size)
