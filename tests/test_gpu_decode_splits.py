"""Split-KV decode at the edges of its forms: partials merged in a cluster's shared memory (up to 8 CTAs, then several
splits per CTA), and through scratch memory above 64 splits; splits without keys; step counts of 0, 1 and more."""
import numpy as np
import pytest
import torch

from conftest import code_hist
from oracle import attn as o_attn
from test_gpu_decode import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,kv_len,W,splits", [(128, 700, 0, 2), (64, 1024, 0, 8), (128, 1024, 0, 9), (32, 2048, 0, 16),
                                               (128, 2048, 0, 17), (64, 2048, 1024, 40), (128, 2048, 0, 64), (128, 2048, 0, 65),
                                               (128, 100, 0, 16), (128, 1, 0, 3), (128, 2048, 0, 0)])
def test_decode_split_forms(stream, D, kv_len, W, splits):
    from x17ai_b200 import kernels as K
    B, H, T = 2, 3, 2048
    rng = np.random.default_rng(D + kv_len + splits)
    q, kv, sk, sv, temp = _case(rng, B, H, D, T)
    kern = K.AttnKernel(K.AttnKernelConfig(H, D, H * D, 2 * H * D, H * D))
    dev = [torch.from_numpy(a).cuda() for a in (q, kv, sk, sv, temp)]
    ref_out, ref_l = o_attn.attn_decode_i8(q, kv, kv_len, sk, sv, temp, W, H, D, kv_tile=1 << 20)
    for no_alloc in (False, True):
        out = torch.zeros((B, H * D), dtype=torch.int8, device="cuda")
        l = torch.zeros((B, H), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        kern.decode(stream, dev[0], dev[1], kv_len, dev[2], dev[3], dev[4], out, l, window_size=W, n_splits=splits, no_alloc=no_alloc)
        stream.synchronize()
        hist = code_hist(out.cpu().numpy(), ref_out)
        # P is rounded against running maxima here, against the final one in the oracle: at most one code apart
        assert hist[2:].sum() == 0 and hist[1] / ref_out.size <= 0.08, hist
        assert np.max(np.abs(l.cpu().numpy() - ref_l)) <= 1e-3


# one and two steps of keys (nothing loaded ahead), one key more (loaded ahead), in one split and over a cluster
@pytest.mark.parametrize("D,kv_len,splits", [(128, 128, 1), (128, 257, 1), (128, 258, 1), (64, 513, 1), (64, 514, 1), (32, 1025, 1),
                                             (32, 1026, 1), (128, 2048, 7), (128, 2048, 8), (64, 1538, 2), (128, 2048, 11), (64, 2048, 70)])
def test_decode_steps(stream, D, kv_len, splits):
    test_decode_split_forms(stream, D, kv_len, 0, splits)


@pytest.mark.parametrize("D,splits", [(32, 2), (64, 8), (128, 3), (128, 8), (128, 40)])
def test_decode_splits_without_keys(stream, D, splits):
    """A ragged batch of lengths 0 to 33: most splits have no key at all and their CTAs reach the merge before the first
    CTA of the cluster has read its keys. Launched repeatedly, behind one another: every launch gives the same bytes."""
    from x17ai_b200 import kernels as K
    B, H, T = 12, 5, 64
    rng = np.random.default_rng(D + splits)
    q, kv, sk, sv, temp = _case(rng, B, H, D, T)
    lens = np.array([0, 1, 2, 15, 16, 17, 0, 31, 32, 33, 1, 5], dtype=np.int32)
    kern = K.AttnKernel(K.AttnKernelConfig(H, D, H * D, 2 * H * D, H * D))
    dev = [torch.from_numpy(a).cuda() for a in (q, kv, sk, sv, temp, lens)]
    outs = torch.zeros((50, B, H * D), dtype=torch.int8, device="cuda")
    ls = torch.zeros((50, B, H), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    for i in range(50):
        kern.decode(stream, dev[0], dev[1], T, dev[2], dev[3], dev[4], outs[i], ls[i], kv_lens=dev[5], n_splits=splits)
    stream.synchronize()
    assert (outs == outs[0]).all() and (ls == ls[0]).all()
    for b in range(B):
        ref_out, ref_l = o_attn.attn_decode_i8(q[b:b + 1], kv[b:b + 1], int(lens[b]), sk, sv, temp, 0, H, D, kv_tile=1 << 20)
        hist = code_hist(outs[0, b:b + 1].cpu().numpy(), ref_out)
        assert hist[2:].sum() == 0, (b, hist)   # P is rounded against running maxima here: at most one code apart
        assert np.max(np.abs(ls[0, b].cpu().numpy() - ref_l[0])) <= 1e-3
