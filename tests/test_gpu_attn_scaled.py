"""Per-token-per-head scaled attention at the edges of its score fragments: sequences that end inside a column pair, a
fragment or a tile, scale vectors that start on an odd element, narrow windows, a negative temperature."""
import numpy as np
import pytest

from oracle import attn as o_attn
from test_gpu_attn import _launch_scaled, _scaled_case

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
