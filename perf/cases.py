"""Performance cases of the quantised block-forward path, driven through the package's public entry points.

A case is a dict of plain values; its `kind` names the calls that one pass makes:

  attn          AttnKernel.launch                 int8 sliding-window attention, FixedI8 in and out, L
  attn_scaled   AttnKernel.launch_scaled          the same with per-token-per-head scales, bf16 out
  attn_pv_fp8   AttnKernel.launch_pv_fp8          the same with e4m3 probabilities and values, bf16 out
  decode        AttnKernel.decode                 one new token per sequence against an int8 KV cache
  ffn           rms_norm (bf16), GemmKernel x 2   normalise, GeGLU projection, gated-residual projection
  ffn_e4m3      GemmKernel x 2                    the FFN pair with e4m3 weights and activations
  decode_layer  rms_norm, qkvg_fwd_i8, decode, GemmKernel, rms_norm, GemmKernel x 2: one layer of a decode step
  layer         BlockForward.forward_layer        one layer over a prompt, RMSNorm before each sub-block
  block         BlockForward.forward              the six launches of the reference's harness

Sizes are those of the repository's benchmark and fixtures, or lie between them.
"""
import math

import torch

from x17ai_b200 import device, kernels as K
from x17ai_b200.block import BlockConfig, BlockForward

_STREAM = None


def _stream():
    """The program's one stream, opened at first use."""
    global _STREAM
    if _STREAM is None:
        _STREAM = device.CudaStream(0)
    return _STREAM


def listed():
    return [
        # the smallest call: the benchmark's CPU-runnable attention case, bound by the launch
        dict(name="attn_small", kind="attn", batch=1, heads=4, seq=256, head_dim=64, window=64),
        # prefill of a batch of long prompts, the benchmark's headline shape
        dict(name="attn_prefill", kind="attn", batch=8, heads=32, seq=8192, head_dim=128, window=1024),
        # the same work in the benchmark's input format: one scale per token and head, bf16 output
        dict(name="attn_scaled_prefill", kind="attn_scaled", batch=8, heads=32, seq=8192, head_dim=128, window=1024),
        # one prompt of an odd length through the fp8 P.V form
        dict(name="attn_pv_fp8_prompt", kind="attn_pv_fp8", batch=1, heads=32, seq=7001, head_dim=128, window=1024),
        # a single user's decode step: few keys, one sequence
        dict(name="decode_one_user", kind="decode", batch=1, heads=32, head_dim=128, capacity=4096, kv_len=1500, window=0,
             ragged=False),
        # continuous batching: 48 sequences at different lengths, windowed attention
        dict(name="decode_ragged_batch", kind="decode", batch=48, heads=32, head_dim=128, capacity=4096, kv_len=4096,
             window=1024, ragged=True),
        # the benchmark's decode shape: a full batch against 8.6 GB of cache
        dict(name="decode_full_batch", kind="decode", batch=256, heads=32, head_dim=128, capacity=4096, kv_len=4096, window=0,
             ragged=False),
        # the FFN of a decode-to-prefill mix at the benchmark's size, from the bf16 hidden state
        dict(name="ffn_16k_tokens", kind="ffn", tokens=16384, model_dim=4096, ffn=14336),
        # the FFN with e4m3 weights and activations on a ragged batch of prompts
        dict(name="ffn_e4m3_ragged", kind="ffn_e4m3", tokens=3001, model_dim=4096, ffn=14336),
        # one layer of a serving step: 16 sequences, one new token each
        dict(name="decode_layer_16", kind="decode_layer", batch=16, model_dim=4096, heads=32, head_dim=128, ffn=14336,
             capacity=2048, kv_len=1800, window=0),
        # one layer over one long prompt, fused projection
        dict(name="layer_prefill", kind="layer", tokens=8192, model_dim=4096, heads=32, head_dim=128, ffn=14336, window=1024),
        # the reference harness's own default configuration: narrow heads, unbounded causal attention
        dict(name="block_default", kind="block", tokens=16384, model_dim=2048, heads=64, head_dim=32, ffn=2048, window=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# (model_dim, heads, head_dim, ffn): the benchmark's, the reference harness's default, and one between the fixtures and these
_MODELS = ((4096, 32, 128, 14336), (2048, 64, 32, 2048), (1024, 16, 64, 4096))


def _pairs(seq, window):
    """Visible (query, key) pairs of one head, the sink included."""
    w = seq if window == 0 else min(window, seq)
    return w * (w - 1) // 2 + (seq - w) * w + seq


def draw(rng):
    kind = rng.choice(("attn", "attn", "attn_scaled", "attn_pv_fp8", "decode", "decode", "ffn", "ffn_e4m3", "decode_layer", "layer",
                       "block"))
    if kind.startswith("attn"):
        heads, head_dim = rng.choice((4, 8, 16, 32, 64)), rng.choice((32, 64, 128, 128))
        seq = _log(rng, 64, 16384)
        window = rng.choice((0, 16 * rng.randint(4, 64), 1024, 4096))
        batch = _log(rng, 1, 8)
        # no more score elements than 2/3 of the benchmark's shape, which every form gets through in less than the largest pass
        most = 1.3e9
        while batch > 1 and batch * heads * _pairs(seq, window) > most:
            batch -= 1
        while heads > 4 and batch * heads * _pairs(seq, window) > most:
            heads //= 2
        return dict(kind=kind, batch=batch, heads=heads, seq=seq, head_dim=head_dim, window=window)
    if kind == "decode":
        capacity = _log(rng, 128, 4096)
        return dict(kind=kind, batch=_log(rng, 1, 256), heads=rng.choice((8, 16, 32)), head_dim=rng.choice((64, 128, 128)),
                    capacity=capacity, kv_len=capacity - rng.randint(0, capacity // 4), window=rng.choice((0, 0, 512, 1024)),
                    ragged=rng.random() < 0.4)
    model_dim, heads, head_dim, ffn = rng.choice(_MODELS)
    if kind in ("ffn", "ffn_e4m3"):
        return dict(kind=kind, tokens=_log(rng, 1, 12000), model_dim=model_dim, ffn=ffn)
    if kind == "decode_layer":
        capacity = _log(rng, 256, 4096)
        return dict(kind=kind, batch=_log(rng, 1, 128), model_dim=model_dim, heads=heads, head_dim=head_dim, ffn=ffn,
                    capacity=capacity, kv_len=capacity - rng.randint(0, capacity // 4), window=rng.choice((0, 1024)))
    return dict(kind=kind, tokens=_log(rng, 32, 7000), model_dim=model_dim, heads=heads, head_dim=head_dim, ffn=ffn,
                window=rng.choice((0, 512, 1024)))


# ---- inputs ------------------------------------------------------------------------------------------

def _codes(g, *shape, std=1.0):
    """N(0, std) values as FixedI8 codes."""
    x = torch.randn(*shape, generator=g, device="cuda")
    return x.mul_(8.0 * std).round_().clamp_(-127, 127).to(torch.int8)


def _unit_heads(x):
    """Heads scaled to unit mean square over their last dimension, as the K projection leaves them."""
    return x.div_(x.square().mean(-1, keepdim=True).sqrt_())


def _kv(g, rows, heads, d):
    """One sequence's K | V rows: K of unit mean square per head, V a little wider."""
    x = torch.randn(rows, heads, 2, d, generator=g, device="cuda")
    _unit_heads(x[:, :, 0])
    x[:, :, 1] *= 1.3
    return x.mul_(8.0).round_().clamp_(-127, 127).to(torch.int8).view(rows, heads * 2 * d)


def _sinks(g, heads, d):
    k = _unit_heads(torch.randn(heads, d, generator=g, device="cuda")).mul_(8.0).round_().clamp_(-127, 127).to(torch.int8)
    return k, _codes(g, heads, d, std=1.3), (0.5 + torch.rand(heads, generator=g, device="cuda")).float()


def _e4m3(g, *shape, std=1.0):
    return torch.randn(*shape, generator=g, device="cuda").mul_(std).to(torch.float8_e4m3fn)


def _hidden(g, rows, cols):
    """A hidden state as the residual epilogue leaves it: e4m3 without subnormal codes."""
    x = torch.randn(rows, cols, generator=g, device="cuda")
    x[x.abs() < 2.0 ** -6] = 0.0
    return x.to(torch.float8_e4m3fn).view(torch.uint8)


def _new(dtype, *shape):
    return torch.zeros(shape, dtype=dtype, device="cuda")


def _attn_kernel(c):
    hd = c["heads"] * c["head_dim"]
    return K.AttnKernel(K.AttnKernelConfig(c["heads"], c["head_dim"], hd, 2 * hd, hd))


def _prepare_attn(c, g):
    b, h, s, d = c["batch"], c["heads"], c["seq"], c["head_dim"]
    st = dict(kern=_attn_kernel(c), l=_new(torch.float32, b, h, s))
    st["sink_k"], st["sink_v"], st["temp"] = _sinks(g, h, d)
    if c["kind"] == "attn_scaled":
        # values quantised per token and head: scale = absmax / 127
        q, kv = _new(torch.int8, b, s, h * d), _new(torch.int8, b, s, h * 2 * d)
        scales = [_new(torch.float32, b, h, s) for _ in range(3)]
        for i in range(b):
            x = torch.randn(s, h, 3, d, generator=g, device="cuda")
            sc = x.abs().amax(-1).div_(127.0)
            x = x.div_(sc.unsqueeze(-1)).round_().to(torch.int8)
            q[i] = x[:, :, 0].reshape(s, h * d)
            kv[i] = x[:, :, 1:].reshape(s, h * 2 * d)
            for j in range(3):
                scales[j][i] = sc[:, :, j].t()
        st.update(q=q, kv=kv, q_scale=scales[0], k_scale=scales[1], v_scale=scales[2], out=_new(torch.bfloat16, b, s, h * d))
        return st
    st["q"] = _new(torch.int8, b, s, h * d)
    st["kv"] = _new(torch.int8, b, s, h * 2 * d)
    for i in range(b):
        st["q"][i] = _codes(g, s, h * d)
        st["kv"][i] = _kv(g, s, h, d)
        if c["kind"] == "attn_pv_fp8":
            st["kv"][i].view(s, h, 2, d)[:, :, 1] = _e4m3(g, s, h, d).view(torch.int8)
    if c["kind"] == "attn_pv_fp8":
        st.update(sink_v=_e4m3(g, h, d), v_scale=(0.5 + torch.rand(h, generator=g, device="cuda")).float(),
                  out=_new(torch.bfloat16, b, s, h * d))
    else:
        st["out"] = _new(torch.int8, b, s, h * d)
    return st


def _cache(c, g):
    b, h, d, t = c["batch"], c["heads"], c["head_dim"], c["capacity"]
    kv = torch.empty((b, t, h * 2 * d), dtype=torch.int8, device="cuda")
    for i in range(b):
        kv[i] = _kv(g, t, h, d)
    return kv


def _prepare_decode(c, g):
    b, h, d = c["batch"], c["heads"], c["head_dim"]
    st = dict(kern=_attn_kernel(c), cache=_cache(c, g), q=_codes(g, b, h * d), out=_new(torch.int8, b, h * d),
              l=_new(torch.float32, b, h), kv_lens=None)
    st["sink_k"], st["sink_v"], st["temp"] = _sinks(g, h, d)
    if c["ragged"]:
        st["kv_lens"] = _lens(c).cuda()
    return st


def _lens(c):
    """Sequence lengths of a continuous batch: spread evenly up to kv_len (the same for every seed, so the work is too)."""
    b = c["batch"]
    return torch.tensor([max(1, c["kv_len"] * (1 + (7 * i + 3) % b) // b) for i in range(b)], dtype=torch.int32)


def _prepare_ffn(c, g):
    m, dm, f = c["tokens"], c["model_dim"], c["ffn"]
    st = dict(f=_new(torch.uint8, m, f), y=_new(torch.uint8, m, dm))
    if c["kind"] == "ffn_e4m3":
        # weights N(0, 0.02) and activations N(0, 1), one scale per tensor
        w_scale = 0.02 / 8.0
        st.update(x=_e4m3(g, m, dm), w_f=_e4m3(g, 2 * f, dm, std=8.0), w_y=_e4m3(g, 2 * dm, f, std=8.0), res=_codes(g, m, dm),
                  k_f=K.GemmKernel(K.ffn_f_fwd_e4m3_config(dm, f, 1.0, w_scale)),
                  k_y=K.GemmKernel(K.ffn_y_fwd_e4m3_config(f, dm, w_scale)))
        return st
    st.update(h=torch.randn(m, dm, generator=g, device="cuda").to(torch.bfloat16), x=_new(torch.int8, m, dm),
              w_f=_codes(g, 2 * f, dm), k_f=K.GemmKernel(K.ffn_f_fwd_config(dm, f)), k_y=K.GemmKernel(K.ffn_y_fwd_f8_config(f, dm)))
    w_y = _codes(g, 2 * dm, f)
    torch.cuda.synchronize()
    st["w_y"] = K.split_i8_weights(_stream(), w_y)
    _stream().synchronize()
    return st


def _prepare_decode_layer(c, g):
    b, dm, h, d, f = c["batch"], c["model_dim"], c["heads"], c["head_dim"], c["ffn"]
    hd = h * d
    st = dict(kern=_attn_kernel(c), cache=_cache(c, g), h=_hidden(g, b, dm), kv_len=c["kv_len"], window=c["window"], heads=h, head_dim=d,
              w_qkv=_codes(g, 3 * hd, dm), w_o=_codes(g, 2 * dm, hd), w_f=_codes(g, 2 * f, dm),
              k_o=K.GemmKernel(K.attn_y_fwd_config(hd, dm)), k_f=K.GemmKernel(K.ffn_f_fwd_config(dm, f)),
              k_y=K.GemmKernel(K.ffn_y_fwd_f8_config(f, dm)),
              x_attn=_new(torch.int8, b, dm), q=_new(torch.int8, b, hd), kv=_new(torch.int8, b, 2 * hd), rrms=_new(torch.float32, b, h),
              attn=_new(torch.int8, b, hd), y=_new(torch.uint8, b, dm), x_ffn=_new(torch.int8, b, dm), f=_new(torch.uint8, b, f),
              out=_new(torch.uint8, b, dm))
    st["sink_k"], st["sink_v"], st["temp"] = _sinks(g, h, d)
    w_y = _codes(g, 2 * dm, f)
    torch.cuda.synchronize()
    st["w_y"] = K.split_i8_weights(_stream(), w_y)
    _stream().synchronize()
    return st


def _prepare_block(c, g):
    dm, h, d, f = c["model_dim"], c["heads"], c["head_dim"], c["ffn"]
    hd = h * d
    w = [_codes(g, *s) for s in ((hd, dm), (2 * hd, dm), (2 * dm, hd), (2 * f, dm), (2 * dm, f))]
    sinks = _sinks(g, h, d)
    x = _hidden(g, c["tokens"], dm) if c["kind"] == "layer" else _codes(g, c["tokens"], dm)
    torch.cuda.synchronize()
    blk = BlockForward(_stream(), BlockConfig(dm, h, d, f, c["window"]), *w, *sinks, fused_qkv=c["kind"] == "layer")
    return dict(blk=blk, x=x)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind.startswith("attn"):
        st = _prepare_attn(case, g)
    elif kind == "decode":
        st = _prepare_decode(case, g)
    elif kind.startswith("ffn"):
        st = _prepare_ffn(case, g)
    elif kind == "decode_layer":
        st = _prepare_decode_layer(case, g)
    else:
        st = _prepare_block(case, g)
    st["case"], st["stream"] = dict(case), _stream()
    torch.cuda.synchronize()   # torch made the inputs on its own stream
    return st


# ---- one pass ----------------------------------------------------------------------------------------

def run(st):
    c, s = st["case"], st["stream"]
    kind = c["kind"]
    if kind == "attn":
        st["kern"].launch(s, st["q"], st["kv"], st["sink_k"], st["sink_v"], st["temp"], st["out"], st["l"], c["window"])
        return {"out": st["out"], "l": st["l"]}
    if kind == "attn_scaled":
        st["kern"].launch_scaled(s, st["q"], st["q_scale"], st["kv"], st["k_scale"], st["v_scale"], st["sink_k"], st["sink_v"],
                                 st["temp"], st["out"], st["l"], c["window"])
        return {"out": st["out"], "l": st["l"]}
    if kind == "attn_pv_fp8":
        st["kern"].launch_pv_fp8(s, st["q"], st["kv"], st["sink_k"], st["sink_v"], st["temp"], st["v_scale"], st["out"], st["l"],
                                 c["window"])
        return {"out": st["out"], "l": st["l"]}
    if kind == "decode":
        st["kern"].decode(s, st["q"], st["cache"], c["kv_len"], st["sink_k"], st["sink_v"], st["temp"], st["out"], st["l"],
                          c["window"], kv_lens=st["kv_lens"])
        return {"out": st["out"], "l": st["l"]}
    if kind == "ffn":
        K.rms_norm(s, K.RMS_BF16_FIXED, st["h"], st["x"])
        st["k_f"].launch(s, st["x"], st["w_f"], st["f"])
        st["k_y"].launch(s, st["f"], st["w_y"], st["y"], residual=st["x"])
        return {"x": st["x"], "f": st["f"], "y": st["y"]}
    if kind == "ffn_e4m3":
        st["k_f"].launch(s, st["x"], st["w_f"], st["f"])
        st["k_y"].launch(s, st["f"], st["w_y"], st["y"], residual=st["res"])
        return {"f": st["f"], "y": st["y"]}
    if kind == "decode_layer":
        K.rms_norm(s, K.RMS_E4M3_FIXED, st["h"], st["x_attn"])
        K.qkvg_fwd_i8(s, st["x_attn"], st["w_qkv"], st["heads"], st["head_dim"], st["q"], st["kv"], st["rrms"])
        st["kern"].decode(s, st["q"], st["cache"], st["kv_len"], st["sink_k"], st["sink_v"], st["temp"], st["attn"], None, st["window"])
        st["k_o"].launch(s, st["attn"], st["w_o"], st["y"], residual=st["x_attn"])
        K.rms_norm(s, K.RMS_E4M3_FIXED, st["y"], st["x_ffn"])
        st["k_f"].launch(s, st["x_ffn"], st["w_f"], st["f"])
        st["k_y"].launch(s, st["f"], st["w_y"], st["out"], residual=st["x_ffn"])
        return {k: st[k] for k in ("x_attn", "q", "kv", "rrms", "attn", "y", "x_ffn", "f", "out")}
    if kind == "layer":
        return st["blk"].forward_layer(st["x"])
    return st["blk"].forward(st["x"])


# ---- what a pass cannot do without ---------------------------------------------------------------------

def _attn_work(batch, heads, seq, d, window, out_bytes=1, scales=False):
    flops = 4.0 * batch * heads * d * _pairs(seq, window)
    return batch * seq * heads * (d * (3 + out_bytes) + 4 + (12 if scales else 0)), flops


def _decode_work(batch, heads, d, kv_lens, window):
    keys = sum(n if window == 0 else min(n, window) for n in kv_lens)
    return keys * heads * 2 * d + 2 * batch * heads * d, 4.0 * d * heads * (keys + batch)


def _gemm_work(m, k, n, a_extra=0):
    """A, B and a C of n / 2 bytes per row (every pair of raw columns gives one byte)."""
    return m * k + n * k + m * n // 2 + a_extra, 2.0 * m * k * n


def work(case):
    c, kind = case, case["kind"]
    parts = []
    if kind.startswith("attn"):
        parts.append(_attn_work(c["batch"], c["heads"], c["seq"], c["head_dim"], c["window"], 1 if kind == "attn" else 2,
                                kind == "attn_scaled"))
    elif kind == "decode":
        lens = _lens(c).tolist() if c["ragged"] else [c["kv_len"]] * c["batch"]
        parts.append(_decode_work(c["batch"], c["heads"], c["head_dim"], lens, c["window"]))
    elif kind in ("ffn", "ffn_e4m3"):
        m, dm, f = c["tokens"], c["model_dim"], c["ffn"]
        # the intermediate tensors are outputs of entry points and inputs of the next
        parts += [_gemm_work(m, dm, 2 * f), _gemm_work(m, f, 2 * dm, m * dm)]
        if kind == "ffn":
            parts.append((3 * m * dm, 0.0))
    else:
        m = c["batch"] if kind == "decode_layer" else c["tokens"]
        dm, h, d, f = c["model_dim"], c["heads"], c["head_dim"], c["ffn"]
        hd = h * d
        parts += [(m * dm + 3 * hd * dm + 3 * m * hd + 4 * m * h, 2.0 * m * dm * 3 * hd), _gemm_work(m, hd, 2 * dm, m * dm),
                  _gemm_work(m, dm, 2 * f), _gemm_work(m, f, 2 * dm, m * dm)]
        if kind != "block":
            parts += [(2 * m * dm, 0.0)] * 2
        if kind == "decode_layer":
            parts.append(_decode_work(m, h, d, [c["kv_len"]] * m, c["window"]))
        else:
            parts.append(_attn_work(1, h, m, d, c["window"]))
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


def tolerance(case):
    """int8 codes and e4m3 bytes may differ where a value lies on a rounding tie; f32 side outputs (L, 1/rms) are sums of
    32-bit values through approximate exponentials and logarithms; bf16 outputs carry eight bits."""
    if case["kind"] in ("attn_scaled", "attn_pv_fp8"):
        return {"rel": 1e-2, "max": 5e-2}
    return {"rel": 1e-5, "max": 1e-3, "differ": 5e-3}
