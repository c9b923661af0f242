"""Edge tiles of the int8 attention: a row's visible columns begin and end at every place inside a 32-column chunk."""
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
