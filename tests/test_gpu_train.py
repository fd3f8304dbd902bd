"""The whole forward's backward (streaming kernels over all branches) against autograd through the fp32 oracle.
Tolerance: max-abs <= 2e-2 * max(1, max|reference|), as for the other 16-bit gradients: an entry is a sum over
hundreds of rows whose operands and result are rounded to 8 (bf16) or 11 bits."""
import pytest
import torch

from helpers import make_qkv, max_abs
from oracle import nsa_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nsa():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import nsa_from_scratch_b200 as pkg
    return pkg


# B, H, Hkv, Tq, Tk, D, top_k, window, (cmp block, stride), one list per KV head, dtype, causal, gates, gate dtype
CASES = [
    (1, 2, 2, 256, 256, 64, 3, 64, (64, 64), False, torch.bfloat16, True, "sigmoid", torch.bfloat16),   # a KV head per head
    (2, 3, 1, 200, 200, 64, 3, 100, (32, 16), True, torch.bfloat16, True, "softmax", torch.float32),    # odd heads, ragged
    (1, 4, 2, 130, 333, 128, 4, 65, (32, 16), True, torch.float16, True, "sigmoid", torch.float32),     # Tq < Tk
    (1, 4, 1, 192, 192, 128, 5, 70, (32, 16), False, torch.bfloat16, True, "sigmoid", torch.bfloat16),  # lists per head
    (1, 2, 1, 192, 256, 64, 2, 50, (32, 16), True, torch.bfloat16, False, "sigmoid", torch.bfloat16),   # not causal
    (1, 1, 1, 65, 65, 64, 16, 512, (64, 64), False, torch.float16, True, "softmax", torch.float16),     # one row in the last block
    (1, 16, 1, 640, 640, 64, 4, 128, (32, 16), True, torch.bfloat16, True, "sigmoid", None),            # several segments, no gates
]


@pytest.mark.parametrize("case", CASES)
def test_gradients_vs_oracle(nsa, case):
    from nsa_from_scratch_b200 import ops
    B, H, Hkv, Tq, Tk, D, k, W, (bc, st), group, dt, causal, act, gdt = case
    Q, K, V, g = make_qkv(31, B, H, Hkv, Tq, Tk, D, dtype=dt)
    gates = torch.randn(B, H, Tq, 3, generator=g).to(gdt) if gdt is not None else None
    dO = torch.randn(B, H, Tq, D, generator=g).to(dt)
    ff, fl = (1, 1) if group else (0, 0)
    cfg = nsa.NSAConfig(block_size_c=bc, stride_c=None if st == bc else st, top_k=k, window_size=W, causal=causal, gate_activation=act,
                        select_per_group=group, force_first=ff, force_local=fl)
    idx = O.select_blocks(Q, K, top_k=k, causal=causal, force_first=ff, force_local=fl, group_shared=group)
    leaves = [t.float().clone().requires_grad_(True) for t in (Q, K, V)]
    logits = (torch.zeros(B, H, Tq, 3) if gates is None else gates.float()).clone().requires_grad_(True)
    oc = O.compressed_attention(*leaves, block_size_c=bc, stride_c=None if st == bc else st, causal=causal)[0]
    os_ = O.selected_attention(*leaves, block_indices=idx, causal=causal)[0]
    ow = O.sliding_attention(*leaves, window_size=W, causal=causal)[0]
    gv = torch.sigmoid(logits) if act == "sigmoid" else torch.softmax(logits, -1)
    ref_out = gv[..., 0:1] * oc + gv[..., 1:2] * os_ + gv[..., 2:3] * ow
    ref = torch.autograd.grad(ref_out, [*leaves, logits], dO.float())
    dev = [t.cuda().requires_grad_(True) for t in (Q, K, V)] + ([] if gates is None else [gates.cuda().requires_grad_(True)])
    out = nsa.nsa_forward(*dev[:3], cfg, gate_logits=None if gates is None else dev[3])
    assert out.dtype == dt and max_abs(out.detach(), ref_out.detach()) <= 2e-2
    got = torch.autograd.grad(out, dev, dO.cuda())
    ops.device_status()
    for name, a, r in zip(("dQ", "dK", "dV", "dgates"), got, ref):
        assert a.shape == r.shape
        err, mag = max_abs(a, r), float(r.abs().max())
        assert err <= 2e-2 * max(1.0, mag), (name, err, mag)
    again = torch.autograd.grad(nsa.nsa_forward(*dev[:3], cfg, gate_logits=None if gates is None else dev[3]), dev, dO.cuda())
    assert torch.equal(again[0], got[0])                 # dQ is formed in a fixed order


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("logit", [0.0, -4.0, -8.0])
def test_fp16_small_gates_keep_their_bits(nsa, D, logit):
    """gate * P in fp16: at 4096 keys and logits of -8 it lies far below the smallest normal number, and scaling dO does not
    change it.  Relative error of the gradients against 64 bits: an operand rounded to 11 bits is off by 2^-12 / sqrt(3) on
    average, 1.4e-4, two to four of them come together; bound 5e-4."""
    T, H, W = 4096, 2, 256
    Q, K, V, g = make_qkv(17, 1, H, 1, T, T, D, dtype=torch.float16)
    gates = (logit + 0.3 * torch.randn(1, H, T, 3, generator=g)).cuda()
    dO = (torch.randn(1, H, T, D, generator=g).half() * (1.0 if logit == 0.0 else 1024.0)).cuda()
    cfg = nsa.NSAConfig(block_size_c=32, stride_c=16, top_k=8, window_size=W, select_per_group=True)
    leaves = [t.cuda().requires_grad_(True) for t in (Q, K, V)]
    idx = nsa._resolve_block_indices(*leaves[:2], block_size_m=64, block_size_n=64, top_k=8, causal=True, scale=D ** -0.5, shared_per_group=True)
    got = torch.autograd.grad(nsa.nsa_forward(*leaves, cfg, gate_logits=gates, block_indices=idx), leaves, dO)
    q, k, v = (t.detach().double().requires_grad_(True) for t in leaves)
    pos, n = torch.arange(T, device="cuda"), (T - 32) // 16 + 1
    at = pos[None] - 16 * torch.arange(n, device="cuda")[:, None]
    pool = ((at >= 0) & (at < 32)).double() / 32
    def pooled(x):                                        # the kernels read pooled rows rounded to 16 bits
        y = pool @ x[0, 0]
        return y + (y.detach().half().double() - y.detach())
    past = pos[None] <= pos[:, None]
    listed = torch.zeros(T // 64, T // 64, dtype=torch.bool, device="cuda").scatter_(1, idx[0, 0].long(), True)
    masks = (16 * torch.arange(n, device="cuda")[None] + 31 <= pos[:, None], past & listed.repeat_interleave(64, 0).repeat_interleave(64, 1),
             past & (pos[None] > pos[:, None] - W))
    keys = ((pooled(k), pooled(v)), (k[0, 0], v[0, 0]), (k[0, 0], v[0, 0]))
    total = 0.0
    for h in range(H):
        for c in range(3):
            s = (q[0, h] @ keys[c][0].T * D ** -0.5).masked_fill(~masks[c], -1e30)
            p = torch.softmax(s, -1).masked_fill(~masks[c], 0.0)
            total = total + (torch.sigmoid(gates[0, h, :, c:c + 1].double()) * (p @ keys[c][1]) * dO[0, h].double()).sum()
    for name, a, r in zip(("dQ", "dK", "dV"), got, torch.autograd.grad(total, (q, k, v))):
        err = float((a.double() - r).norm() / r.norm())
        assert err <= 5e-4, (name, err)


@pytest.mark.parametrize("D", [64, 128])
def test_a_window_beyond_the_sequence(nsa, D):
    """2**31 - 1 for "no window": the gradients of a window that just covers the sequence.  dQ repeats bit for bit; dK and dV are
    fp32 sums in another order, rounded to 8 bits: 1e-3 of the norm (a bf16 ulp of 4e-3 here and there)."""
    Q, K, V, g = make_qkv(23, 1, 4, 2, 300, 333, D)
    dO = torch.randn(1, 4, 300, D, generator=g).bfloat16().cuda()
    grads = []
    for window in (333, 2**31 - 1):
        cfg = nsa.NSAConfig(block_size_c=32, stride_c=16, top_k=2, window_size=window, select_per_group=True)
        leaves = [t.cuda().requires_grad_(True) for t in (Q, K, V)]
        grads.append(torch.autograd.grad(nsa.nsa_forward(*leaves, cfg), leaves, dO))
    assert torch.equal(grads[0][0], grads[1][0])
    for a, b in zip(*(x[1:] for x in grads)):
        assert float((a.float() - b.float()).norm() / a.float().norm()) <= 1e-3


def test_refused_gate_logits_and_lists(nsa):
    """What the kernels cannot read is refused before anything is launched."""
    Q, K, V, g = make_qkv(29, 1, 2, 1, 128, 128, 64)
    q, k, v = (t.cuda().requires_grad_(True) for t in (Q, K, V))
    gates = torch.randn(1, 2, 128, 3, generator=g)
    idx = torch.zeros(1, 1, 2, 1, dtype=torch.int32)
    cfg = nsa.NSAConfig(top_k=2, window_size=64)
    for kw in (dict(gate_logits=gates), dict(gate_logits=gates.bfloat16()), dict(block_indices=idx)):
        with pytest.raises(RuntimeError, match="CUDA tensors"):
            nsa.nsa_forward(q, k, v, cfg, **kw)
        with torch.no_grad(), pytest.raises(RuntimeError, match="CUDA tensors"):
            nsa.nsa_forward(q, k, v, cfg, **kw)
    with pytest.raises(TypeError):
        nsa.nsa_forward(q, k, v, cfg, gate_logits=gates.half().cuda())
    with pytest.raises(ValueError):
        nsa.nsa_forward(q, k, v, cfg, gate_logits=gates[:, :, :64].cuda())


def test_the_status_word_reaches_the_host(nsa):
    from nsa_from_scratch_b200 import _lib as L, ops
    lib = L.load()
    ops.device_status()
    assert lib.nsa_debug_set_device_status(3, 5) == 0
    with pytest.raises(RuntimeError, match="barrier 304"):
        ops.device_status()
    ops.device_status()                                    # the report clears it


def test_strict_layout_is_about_the_callers_tensors(nsa):
    """out.sum() sends back an expanded gradient and a transpose a strided one: no copy that a caller could avoid."""
    from nsa_from_scratch_b200 import ops
    Q, K, V, g = make_qkv(37, 1, 2, 1, 128, 128, 64)
    cfg = nsa.NSAConfig(top_k=2, window_size=64)
    leaves = [t.cuda().requires_grad_(True) for t in (Q, K, V)]
    dO = torch.randn(1, 128, 2, 64, generator=g).bfloat16().cuda()
    ops.set_strict_layout(True)
    try:
        one = torch.autograd.grad(nsa.nsa_forward(*leaves, cfg).sum(), leaves)[0]
        swapped = torch.autograd.grad(nsa.nsa_forward(*leaves, cfg).transpose(1, 2), leaves, dO)[0]
    finally:
        ops.set_strict_layout(False)
    assert torch.equal(one, torch.autograd.grad(nsa.nsa_forward(*leaves, cfg), leaves, torch.ones_like(leaves[0]))[0])
    assert torch.equal(swapped, torch.autograd.grad(nsa.nsa_forward(*leaves, cfg), leaves, dO.transpose(1, 2).contiguous())[0])
