"""Edge tiles of the int8 attention: a row's visible columns begin and end at every place inside a 32-column chunk; and
the bytes of its probabilities where the scores are too large for 255 * 2^x to stay a byte by itself."""
import numpy as np
import pytest

from oracle import attn as o_attn
from test_gpu_attn import ALL, _inputs, _launch

pytestmark = pytest.mark.gpu


# windows of every multiple of 16 up to a tile and one beyond: the visible columns begin and end at every bit of a word
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("W", [16, 48, 112, 128, 144, 0])
def test_visible_columns(stream, D, W):
    rng = np.random.default_rng(D + W)
    B, H, S = 1, 1, 297
    q, kv, sk, sv, temp = _inputs(rng, B, S, H, D)
    out, l = _launch(stream, q, kv, sk, sv, temp, H, D, W)
    ref, ref_l = o_attn.attn_fwd_i8(q[0], kv[0], sk, sv, temp, W, H, D, kv_tile=ALL)
    d = np.abs(out[0].astype(np.int32) - ref.astype(np.int32))
    # ex2.approx against libm: one code on a rounding tie, as in the other parity tests
    assert d.max() <= 1 and (d > 0).mean() < 5e-3
    assert np.max(np.abs(l[0] - ref_l)) < 1e-3


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("schedule", [0, 1])
def test_probabilities_of_huge_scores(stream, schedule, sign):
    """Score maxima of 2^16 to 2^18 (long q and k that differ in a few entries, temperatures of 4 to 16): half an ulp of the
    maximum is up to 0.4 % of the largest probability and more."""
    from x17ai_b200 import kernels as K
    rng = np.random.default_rng(11)
    B, H, D, S = 1, 32, 128, 64
    q = np.full((B, S, H, D), 127, dtype=np.int8)
    kv = np.zeros((B, S, H, 2, D), dtype=np.int8)
    kv[..., 0, :] = 127 * sign
    q[..., :8] = 1
    kv[..., 0, :8] -= sign * rng.integers(0, 30, (B, S, H, 8)).astype(np.int8)
    kv[..., 1, :] = rng.integers(-127, 128, (B, S, H, D))
    sk = np.zeros((H, D), dtype=np.int8)
    temp = sign * np.linspace(5.5, 16.0, H).astype(np.float32)
    K.set_attn_schedule(schedule)
    try:
        _, l, acc, p, _ = _launch(stream, q.reshape(B, S, H * D), kv.reshape(B, S, -1), sk, sk, temp, H, D, 0, debug=True)
    finally:
        K.set_attn_schedule()
    rt = o_attn.row_temperature(S, D, 0).astype(np.float64)
    for h in range(H):
        for i in range(32, S):
            x = acc[h, i, :i] * rt[i] * temp[h]
            m = x.max()
            assert 2.0 ** 16 < m < 2.0 ** 18
            # x - max to an ulp of the maximum (rounded up or to nearest), P to half a step, ex2.approx
            ulp = 2.0 ** (np.floor(np.log2(m)) - 23)
            want = 255.0 * np.exp2(x - m)
            # the row's temperature itself is known to a few f32 roundings, relative to differences of the scores
            assert np.all(np.abs(p[h, i, :i] - want) <= 255.0 * (2.0 ** ulp - 1) + want * (m - x) * 2.0 ** -21 + 0.51), (h, i)
