"""Per-token-per-head scaled attention at the edges of its score fragments: sequences that end inside a column pair, a
fragment or a tile, scale vectors that start on an odd element, narrow windows, a negative temperature."""
import numpy as np
import pytest

from oracle import attn as o_attn
from test_gpu_attn import _launch, _launch_scaled, _scaled_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,D,S,W,sign", [
    (1, 1, 64, 1, 0, 1), (2, 3, 32, 129, 16, 1), (1, 2, 128, 333, 0, 1), (2, 1, 64, 255, 64, -1), (1, 2, 128, 386, 128, -1),
    (1, 1, 32, 97, 32, -1), (2, 2, 128, 640, 272, 1),
])
def test_scaled_fragments(stream, B, H, D, S, W, sign):
    rng = np.random.default_rng(S + W)
    (qs, ks, vs), sk, sv, temp = _scaled_case(rng, B, S, H, D)
    temp = temp * np.float32(sign)
    got, l = _launch_scaled(stream, qs, ks, vs, sk, sv, temp, H, D, W)
    for b in range(B):
        ref, ref_l = o_attn.attn_fwd_i8_scaled(qs[0][b], qs[1][b], ks[0][b], ks[1][b], vs[0][b], vs[1][b], sk, sv, temp, W)
        rms = np.sqrt(np.mean(ref ** 2))
        # u8 probabilities may differ by one step on a rounding tie (1e-2 of the RMS), plus one bf16 ulp
        assert np.max(np.abs(got[b] - ref)) <= 1e-2 * rms + 2.0 ** -8 * np.abs(ref).max()
        assert np.max(np.abs(l[b] - ref_l)) <= 1e-3


def test_scales_of_unseen_keys_do_not_matter(stream):
    """Rows whose window ends in front of a key are unchanged by an infinite scale of that key's value."""
    rng = np.random.default_rng(9)
    B, H, D, S, W = 1, 1, 64, 300, 64
    (qs, ks, vs), sk, sv, temp = _scaled_case(rng, B, S, H, D)
    want, _ = _launch_scaled(stream, qs, ks, vs, sk, sv, temp, H, D, W)
    vinf = (vs[0], vs[1].copy())
    vinf[1][:, :, 40] = np.inf
    got, _ = _launch_scaled(stream, qs, ks, vinf, sk, sv, temp, H, D, W)
    seen = np.zeros(S, dtype=bool)
    seen[41:41 + W] = True
    assert np.array_equal(got[:, ~seen], want[:, ~seen])


def test_large_scores_give_the_fixedi8_probabilities(stream):
    """With every scale 1/8 and a score maximum of 2^12 to 2^15 (long q and k that differ in a few entries: the ulp of the
    maximum is a visible part of a probability step) P is that of the FixedI8 kernel. Values are one-hot per key, with one
    more dimension that sums P: the ratio of two bf16 outputs is P / sum(P) to twice the bf16 rounding of 2^-8."""
    rng = np.random.default_rng(5)
    B, H, D, S = 1, 8, 128, 64
    q = np.full((B, S, H, D), 127, dtype=np.int8)
    k = np.full((B, S, H, D), 127, dtype=np.int8)
    q[..., :8] = rng.integers(1, 5, (B, S, H, 8))
    k[..., :8] -= rng.integers(0, 30, (B, S, H, 8)).astype(np.int8)
    v = np.zeros((B, S, H, D), dtype=np.int8)
    v[:, np.arange(S), :, np.arange(S)] = 127
    v[..., 127] = 127
    sk = np.zeros((H, D), dtype=np.int8)
    temp = np.linspace(0.5, 1.9, H).astype(np.float32)
    kv = np.concatenate((k, v), axis=-1).reshape(B, S, 2 * H * D)
    _, l, _, p, _ = _launch(stream, q.reshape(B, S, H * D), kv, sk, sk, temp, H, D, 0, debug=True)
    assert 2.0 ** 12 < l[:, :, 32:].min() and l.max() < 2.0 ** 15
    eighth = np.full((B, H, S), 0.125, dtype=np.float32)
    got, _ = _launch_scaled(stream, (q, eighth), (k, eighth), (v, eighth), sk, sk, temp, H, D, 0)
    for h in range(H):
        for i in range(1, S):
            want = p[h, i, :i] / p[h, i, :i].sum(dtype=np.float64)
            ratio = got[0, i, h, :i] / got[0, i, h, 127].astype(np.float64)
            assert np.all(np.abs(ratio - want) <= (2.0 ** -7 + 2.0 ** -14) * want), (h, i)
