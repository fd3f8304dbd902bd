"""The forward as one library call: its window means at the edges of their load batches, and the whole call against
the same steps taken one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nsa():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import nsa_from_scratch_b200 as m
    return m


@pytest.mark.parametrize("block,stride", [(1, 1), (15, 15), (16, 16), (17, 17), (33, 11), (64, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_window_means_are_row_order_sums(nsa, block, stride, dtype):
    """fp32 sum in row order, one exact division, one rounding: bit-equal to the same steps in torch."""
    from nsa_from_scratch_b200 import ops
    T, D = 131, 64
    x = torch.randn(2, 3, T, D, generator=torch.Generator().manual_seed(block)).to(dtype)
    n = ops.n_pooled(T, block, stride)
    want = torch.zeros(2, 3, n, D)
    for s in range(block):
        rows = torch.arange(n) * stride + s
        want += torch.where((rows < T)[:, None], x[:, :, rows.clamp(max=T - 1)].float(), torch.zeros(()))
    got = ops.pool_mean(x.cuda(), block, stride).cpu()
    assert torch.equal(got, (want / block).to(dtype))


@pytest.mark.parametrize("H,Hkv,T,Tq,D,group", [(4, 4, 64, 64, 64, False), (8, 2, 257, 257, 128, True), (4, 1, 300, 65, 64, True), (2, 2, 33, 33, 64, False)])
def test_one_call_equals_the_steps(nsa, H, Hkv, T, Tq, D, group):
    from nsa_from_scratch_b200 import _lib as L, ops
    g = torch.Generator().manual_seed(3)
    Q, K, V = (torch.randn(1, h, t, D, generator=g).to(torch.bfloat16).cuda() for h, t in ((H, Tq), (Hkv, T), (Hkv, T)))
    gates = torch.randn(1, H, Tq, 3, generator=g).cuda()
    cfg = nsa.NSAConfig(block_size_c=32, stride_c=16, top_k=3, window_size=70, force_first=1, force_local=1, select_per_group=group)
    idx = nsa._resolve_block_indices(Q, K, block_size_m=64, block_size_n=64, top_k=3, causal=True, scale=D ** -0.5, force_first=1,
                                     force_local=1, shared_per_group=group)
    want, _ = ops.attention_fwd(Q, K, V, branches=7, fused=True, causal=True, scale=D ** -0.5, Kc=ops.pool_mean(K, 32, 16),
                                Vc=ops.pool_mean(V, 32, 16), cmp_block=32, cmp_stride=16, cmp_offset=T - Tq, idx=idx, window=70,
                                gates=gates, gate_act=L.GATE_SIGMOID)
    assert torch.equal(nsa.nsa_forward(Q, K, V, cfg, gate_logits=gates), want)
    assert torch.equal(nsa.nsa_forward(Q, K, V, cfg, gate_logits=gates, block_indices=idx), want)


def test_window_means_of_more_results_than_a_launch_counts(nsa):
    """2^31 results of 8 columns and some more, in pieces of whole heads: every head marked, the ends of each piece compared."""
    from nsa_from_scratch_b200 import ops
    T, D, heads = 65536, 128, 2049
    if torch.cuda.mem_get_info()[0] < 60e9:
        pytest.skip("needs 52 GB of device memory")
    x = torch.zeros((1, heads, T, D), dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)
    x.view(torch.uint8)[0, :, 0, 0] = torch.arange(heads, device="cuda").remainder(100).to(torch.uint8)     # finite bit patterns
    x.view(torch.uint8)[0, :, T - 1, D - 1] = 0x38                                                          # 1.0
    got = ops.pool_mean(x, 1, 1)
    assert torch.equal(got[0, :, 0, 0], x[0, :, 0, 0].float().bfloat16())
    assert bool((got[0, :, T - 1, D - 1] == 1.0).all())
    assert int((got[0, 2040:] != 0).sum()) == int((x[0, 2040:].view(torch.uint8) != 0).sum())
    del x, got
    torch.cuda.empty_cache()


@pytest.mark.parametrize("H,Hkv,D,group", [(4, 4, 64, False), (4, 1, 128, True), (2, 1, 32, True)])
@pytest.mark.parametrize("Tk,Tq", [(1, 1), (15, 7), (31, 31)])
def test_sequences_shorter_than_one_pooling_window(nsa, H, Hkv, D, group, Tk, Tq):
    """No pooled token: the compressed branch gives nothing, the others their own; against the oracle (2e-2, 16-bit outputs)."""
    from helpers import make_qkv, max_abs
    from oracle import nsa_oracle as O
    Q, K, V, g = make_qkv(5, 2, H, Hkv, Tq, Tk, D)
    gates = torch.randn(2, H, Tq, 3, generator=g)
    cfg = nsa.NSAConfig(block_size_c=32, stride_c=16, top_k=2, window_size=8, select_per_group=group)
    idx = O.select_blocks(Q, K, top_k=2, group_shared=group)
    gv = torch.sigmoid(gates)
    ref = gv[..., 1:2] * O.selected_attention(Q, K, V, block_indices=idx)[0] + gv[..., 2:3] * O.sliding_attention(Q, K, V, window_size=8)[0]
    out = nsa.nsa_forward(Q.cuda(), K.cuda(), V.cuda(), cfg, gate_logits=gates.cuda())
    assert max_abs(out, ref) <= 2e-2


@pytest.mark.parametrize("bm,bn,k", [(64, 32, 3), (128, 128, 2), (64, 64, 70)])
def test_fp8_beyond_the_tcgen05_kernels_shapes(nsa, bm, bn, k):
    """The generic kernel converts as it loads: bit-equal to the same call on the dequantised tensors."""
    g = torch.Generator().manual_seed(7)
    T = 70 * 64 + 5 if k == 70 else 300
    q8, k8, v8 = (torch.randn(1, h, T, 64, generator=g).to(torch.float8_e4m3fn).cuda() for h in (2, 1, 1))
    cfg = nsa.NSAConfig(block_size_c=32, stride_c=16, block_size_m=bm, block_size_n=bn, top_k=k, window_size=65, select_per_group=True)
    s = 0.37
    want = nsa.nsa_forward(*((x.float() * s).bfloat16() for x in (q8, k8, v8)), cfg)
    assert torch.equal(nsa.nsa_forward_fp8(q8, k8, v8, s, s, s, cfg), want)
