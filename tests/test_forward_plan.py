"""What a forward call keeps between calls: argument structs by shape and geometry, none of a call's own values."""
import pytest
import torch

from nsa_from_scratch_b200 import _lib as L
from nsa_from_scratch_b200 import ops

GEOMETRY = dict(causal=True, cmp_block=32, cmp_stride=16, bm=64, bn=64, window=512, top_k=16, force_first=1, force_local=2, per_group=True,
                idx_shape=None, gate_dtype=None, gate_act=L.GATE_SIGMOID, engine=L.ENGINE_AUTO, token_major=False)
SHAPES = torch.Size((1, 8, 256, 128)), torch.Size((1, 2, 256, 128)), torch.float8_e4m3fn


def _plan(scale, q, k, v):
    return ops.forward_plan(*SHAPES, scale=scale, q_scale=q, k_scale=k, v_scale=v, **GEOMETRY)


def test_a_scale_kept_in_a_tensor_is_read_on_every_call():
    s = torch.tensor(0.25)
    first = _plan(0.125, s, s, s)[0]
    s.fill_(0.5)
    a = _plan(0.125, s, s, s)[0]
    assert (a.q_scale, a.k_scale, a.v_scale) == (0.5, 0.5, 0.5) and first.q_scale == 0.25


def test_new_scales_share_a_plan_and_their_signs_do_not():
    base = _plan(0.125, 1.0, 1.0, 1.0)
    n = len(ops._forward_plans)
    for i in range(1, 300):
        a = _plan(0.125 + i, 1.0 + i, 2.0 + i, 3.0 + i)
        assert (a[0].scale, a[0].q_scale, a[0].k_scale, a[0].v_scale) == (0.125 + i, 1.0 + i, 2.0 + i, 3.0 + i) and a[1:] == base[1:]
    assert len(ops._forward_plans) == n
    # scales that are not positive keep fp8 K and V for the generic kernel: no room for their 16-bit copies
    assert _plan(0.125, 1.0, 0.0, 1.0)[1] < base[1]
    assert _plan(0.125, 1.0, 1e-60, 1.0)[1] < base[1]       # 0 as a 32-bit float
    assert len(ops._forward_plans) == n + 1


@pytest.mark.gpu
def test_fp8_forward_with_an_updated_scale_tensor():
    import nsa_from_scratch_b200 as nsa
    g = torch.Generator(device="cuda").manual_seed(2)
    q, k, v = (torch.randn((1, h, 256, 128), generator=g, device="cuda").to(torch.float8_e4m3fn) for h in (4, 1, 1))
    cfg = nsa.NSAConfig(block_size_c=32, stride_c=16, top_k=3, window_size=64, select_per_group=True)
    s = torch.tensor(0.5, device="cuda")
    for value in (0.5, 2.0):
        s.fill_(value)
        assert torch.equal(nsa.nsa_forward_fp8(q, k, v, s, s, s, cfg), nsa.nsa_forward_fp8(q, k, v, value, value, value, cfg))


def test_given_lists_need_no_top_k():
    plan = ops.forward_plan(*SHAPES, scale=0.125, q_scale=1.0, k_scale=1.0, v_scale=1.0,
                            **{**GEOMETRY, "top_k": None, "idx_shape": torch.Size((1, 2, 4, 3))})
    assert (plan[0].has_idx, plan[0].Hi, plan[0].top_k) == (1, 2, 3)


@pytest.mark.gpu
def test_decoding_takes_a_window_of_another_number_type():
    import nsa_from_scratch_b200 as nsa
    g = torch.Generator(device="cuda").manual_seed(6)
    q, k, v = (torch.randn((1, h, t, 64), generator=g, device="cuda").bfloat16() for h, t in ((4, 1), (2, 300), (2, 300)))
    outs = []
    for window in (100, 100.0):
        cache = nsa.KVCache(1, 2, 64, 320, nsa.NSAConfig(top_k=2, window_size=window))
        cache.append(k, v)
        outs.append(nsa.nsa_decode(q, cache))
    assert torch.equal(*outs)
