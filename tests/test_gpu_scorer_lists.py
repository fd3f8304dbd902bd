"""The log-sum-exp behind the block scores: a score that ties to fp32 rounding goes the way its arithmetic decides, so the
arithmetic is part of what the compressed scorer's lists are.  Restated here step by step: in tiles of 128 pooled keys that
all 32 rows of a warp see whole, 3 of every 8 pairs of exponentials come from a cubic (relative error 7.5e-5), the rest from 2^x."""
import numpy as np
import pytest
import torch

from helpers import make_qkv

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nsa():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import nsa_from_scratch_b200 as pkg
    return pkg


def _exp2(x, cubic):
    f32 = lambda v: v.astype(np.float32).astype(np.float64)
    n = np.rint(x)
    f = x - n
    q = np.full_like(f, np.float32(0.0551716685295105), dtype=np.float64)
    for c in (0.2426111251115799, 0.6932609677314758, 0.9999280571937561):
        q = f32(q * f + np.float64(np.float32(c)))
    with np.errstate(under="ignore"):
        return np.where(cubic, q * np.exp2(n), f32(np.exp2(x)))


def _lse(S, vis, scale, mixed):
    """S [rows, keys] raw scores, vis [rows, keys]: rows in warps of 32, keys in tiles of 128."""
    with np.errstate(invalid="ignore"):                  # rows that have seen no key yet
        return _lse_rows(S, vis, scale, mixed)


def _lse_rows(S, vis, scale, mixed):
    sl2 = np.float64(np.float32(scale) * np.float32(1.4426950408889634))
    out = np.full(S.shape[0], -np.inf)
    for r0 in range(0, S.shape[0], 32):
        s, v = S[r0:r0 + 32], vis[r0:r0 + 32]
        m, l = np.full(len(s), -np.inf), np.zeros(len(s))
        for j0 in range(0, S.shape[1], 128):
            st, vt = s[:, j0:j0 + 128], v[:, j0:j0 + 128]
            if not vt.any():
                continue
            full = len(s) == 32 and st.shape[1] % 64 == 0 and vt.all()      # a last tile of one whole 64-key chunk counts
            mx = np.where(vt, st, -np.inf).max(1).astype(np.float32) * np.float32(sl2)
            if (mx > m + 8).any():
                mn = np.maximum(m, mx)
                l *= np.where(np.isfinite(mn), np.exp2(np.where(np.isfinite(m), m - mn, -np.inf)), 1.0)
                m = mn
            x = (st * sl2 - np.where(np.isfinite(m), m, 0.0)[:, None]).astype(np.float32).astype(np.float64)
            cubic = mixed and full
            cols = (np.arange(st.shape[1]) // 2) % 8 < 3
            l += np.where(vt, _exp2(x, cols[None, :] & cubic), 0.0).sum(1)
        with np.errstate(divide="ignore"):
            out[r0:r0 + 32] = np.where(l > 0, m * np.log(2.0) + np.log(l), -np.inf)
    return out


# whole tiles, a last tile of one whole chunk (causal=False: 64 pooled keys of 192), ragged ends
@pytest.mark.parametrize("D,T,causal", [(64, 4111, True), (128, 4111, True), (128, 3088, False)])
def test_lse_behind_the_scores(nsa, D, T, causal):
    from nsa_from_scratch_b200 import ops
    H = 4
    Q, K, _, _ = make_qkv(3, 1, H, 1, T, T, D)
    Kc = ops.pool_mean(K.cuda(), 32, 16)
    kw = dict(branches=1, causal=causal, scale=D ** -0.5, Kc=Kc, Vc=Kc, cmp_block=32, cmp_stride=16, cmp_offset=0)
    _, lse = ops.attention_fwd(Q.cuda(), K.cuda(), K.cuda(), fused=True, fused_lse=True, **kw)
    n = Kc.shape[2]
    pos, end = np.arange(T), np.arange(n) * 16 + 31
    vis = end[None, :] <= pos[:, None] if causal else np.ones((T, n), bool)
    kc = Kc[0, 0].float().cpu().double().numpy()
    worst = 0.0
    for h in range(H):
        S = (Q[0, h].double().numpy() @ kc.T).astype(np.float32).astype(np.float64)
        want, plain = _lse(S, vis, D ** -0.5, True), _lse(S, vis, D ** -0.5, False)
        got = lse[0, h].double().cpu().numpy()
        fin = np.isfinite(want)
        assert np.array_equal(np.isfinite(got), fin)
        got, want, plain = got[fin], want[fin], plain[fin]
        # fp32: scores of up to 8 (ulp 5e-7) from another order of sums, 2^x within 2 ulp, a sum of hundreds of terms
        assert np.abs(got - want).max() <= 4e-6, np.abs(got - want).max()
        worst = max(worst, np.abs(got - plain).max())
    assert worst > 8e-6                                  # the plain exponential's is told apart
