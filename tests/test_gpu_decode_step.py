"""The decoding step as one call (nsa_decode without nsplit): every arrangement of a block's warps (row tiles by key
groups), lists per head and per KV head, lengths around the chunk and window edges, and the device-resident length.
Against the oracle with the tolerance of the other 16-bit outputs (2e-2), and that the path is the one that runs."""
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


# B, H, Hkv, Tq, length, D, top_k, window, (cmp block, stride), one list per KV head, dtype, forced (first, local)
CASES = [
    (1, 4, 4, 1, 1, 64, 4, 64, (64, 64), False, torch.bfloat16, (0, 0)),        # a single position
    (2, 4, 4, 4, 129, 64, 4, 64, (64, 64), False, torch.float16, (0, 0)),       # a KV head per head, four tokens
    (1, 8, 2, 1, 700, 128, 3, 130, (32, 16), True, torch.bfloat16, (1, 2)),     # 4 rows
    (3, 16, 1, 1, 1025, 64, 16, 512, (32, 16), True, torch.bfloat16, (1, 2)),   # 16 rows: the last of a one-tile block
    (1, 16, 1, 2, 640, 128, 8, 256, (32, 16), True, torch.float16, (1, 2)),     # 32 rows: two tiles, two key groups
    (1, 12, 1, 3, 333, 64, 8, 100, (32, 16), True, torch.bfloat16, (1, 1)),     # 36 rows: four tiles, the last two part empty
    (2, 16, 1, 4, 1500, 128, 16, 512, (32, 16), True, torch.bfloat16, (1, 2)),  # 64 rows
    (1, 16, 1, 4, 900, 64, 5, 200, (32, 16), False, torch.bfloat16, (0, 1)),    # 64 rows, lists per head
    (1, 8, 2, 64, 900, 64, 4, 200, (32, 16), False, torch.bfloat16, (0, 0)),    # too many rows: the general path
]


@pytest.mark.parametrize("case", CASES)
def test_step_vs_oracle(nsa, case):
    from nsa_from_scratch_b200 import decode, ops
    B, H, Hkv, Tq, n, D, k, W, (bc, st), group, dt, (ff, fl) = case
    Q, K, V, g = make_qkv(7, B, H, Hkv, Tq, n, D, dtype=dt)
    gates = torch.randn(B, H, Tq, 3, generator=g)
    cfg = nsa.NSAConfig(block_size_c=bc, stride_c=None if st == bc else st, top_k=k, window_size=W, force_first=ff, force_local=fl,
                        select_per_group=group)
    cache = nsa.KVCache(B, Hkv, D, n + 70, cfg, dtype=dt)
    if n > Tq:
        cache.append(K[:, :, :n - Tq].cuda(), V[:, :, :n - Tq].cuda())
    cache.append(K[:, :, n - Tq:].cuda(), V[:, :, n - Tq:].cuda())
    q, gl = Q.cuda(), gates.cuda()
    out = nsa.nsa_decode(q, cache, gate_logits=gl)
    kw = dict(block_size_c=bc, stride_c=None if st == bc else st, top_k=k, window_size=W, force_first=ff, force_local=fl, group_shared=group)
    idx = O.select_blocks(Q.float(), K.float(), top_k=k, force_first=ff, force_local=fl, group_shared=group)
    ref = O.nsa_forward(Q.float(), K.float(), V.float(), gate_logits=gates, block_indices=idx, **kw)
    assert max_abs(out, ref) <= 2e-2, max_abs(out, ref)
    if H // Hkv * Tq <= 64:
        assert torch.equal(out, decode._step(q, cache, gl, D ** -0.5))
        filled = torch.full((1,), n, dtype=torch.int32, device="cuda")
        cache.length = n + 70                            # the grid of a full cache, the length read on the device
        assert max_abs(decode._step(q, cache, gl, D ** -0.5, filled), ref) <= 2e-2
    else:
        assert decode._step(q, cache, gl, D ** -0.5) is None
    ops.device_status()


def test_graphed_steps_follow_the_cache(nsa):
    B, H, Hkv, D, T0, steps = 1, 8, 2, 128, 120, 20
    Q, K, V, g = make_qkv(9, B, H, Hkv, T0 + steps, T0 + steps, D)
    cfg = nsa.NSAConfig(block_size_c=32, stride_c=16, top_k=3, window_size=80, force_first=1, force_local=1, select_per_group=True)
    ca, cb = nsa.KVCache(B, Hkv, D, 256, cfg), nsa.KVCache(B, Hkv, D, 256, cfg)
    Qc, Kc, Vc = Q.cuda(), K.cuda(), V.cuda()
    ca.append(Kc[:, :, :T0], Vc[:, :, :T0])
    cb.append(Kc[:, :, :T0], Vc[:, :, :T0])
    dec = nsa.GraphedDecoder(ca, H, gates=False)
    for t in range(T0, T0 + steps):
        dec.q.copy_(Qc[:, :, t:t + 1]); dec.k.copy_(Kc[:, :, t:t + 1]); dec.v.copy_(Vc[:, :, t:t + 1])
        out = dec.step()
        cb.append(Kc[:, :, t:t + 1], Vc[:, :, t:t + 1])
        assert max_abs(out, nsa.nsa_decode(Qc[:, :, t:t + 1], cb, nsplit=1)) <= 1e-2


def test_a_device_count_past_the_allocation_reads_as_a_full_cache(nsa):
    from nsa_from_scratch_b200 import decode
    B, H, Hkv, D, n = 2, 8, 2, 64, 640
    Q, K, V, _ = make_qkv(3, B, H, Hkv, 1, n, D)
    cfg = nsa.NSAConfig(block_size_c=32, stride_c=16, top_k=3, window_size=80, force_first=1, force_local=1, select_per_group=True)
    cache = nsa.KVCache(B, Hkv, D, n, cfg)
    cache.append(K.cuda(), V.cuda())
    want = nsa.nsa_decode(Q.cuda(), cache)
    for count in (n, n + 1, n + 64, 2**31 - 1):
        dyn = torch.full((1,), count, dtype=torch.int32, device="cuda")
        assert max_abs(decode._step(Q.cuda(), cache, None, D ** -0.5, dyn), want) <= 1e-3, count


# B, H, Hkv, Tq, length, allocation, D, top_k, one list per KV head, dtype: what the sizes reach is named per case
LONG = [
    (8, 32, 4, 1, 8200, 8300, 128, 16, False, torch.bfloat16),   # three 64-key chunks and several listed blocks to a task
    (8, 64, 4, 1, 8200, 8300, 128, 16, True, torch.float16),     # the same, lists per KV head
    (1, 4, 1, 1, 20000, 20100, 64, 16, True, torch.bfloat16),    # 8 candidates to a lane, three scoring tasks to a list
    (1, 4, 1, 2, 70000, 70100, 64, 16, False, torch.bfloat16),   # 16 to a lane
    (1, 2, 1, 1, 140000, 140100, 64, 64, True, torch.bfloat16),  # candidates in shared memory
    (2, 4, 1, 1, 1500, 140100, 64, 16, True, torch.bfloat16),    # a grid for 140100 positions, 1500 filled
]


@pytest.mark.parametrize("case", LONG)
def test_long_caches_vs_oracle(nsa, case):
    """Against the oracle over the lists of the selection kernel (64 queries that share the step's query block mean).  Outputs
    are averages of up to thousands of rows, about 0.05 in size: 1e-2 of the norm, four times what 8-bit (bf16)
    probabilities and results give."""
    from nsa_from_scratch_b200 import decode
    B, H, Hkv, Tq, n, room, D, k, group, dt = case
    Q, K, V, g = make_qkv(11, B, H, Hkv, Tq, n, D, dtype=dt)
    gates = torch.randn(B, H, Tq, 3, generator=g)
    cfg = nsa.NSAConfig(block_size_c=32, stride_c=16, top_k=k, window_size=512, force_first=1, force_local=2, select_per_group=group)
    cache = nsa.KVCache(B, Hkv, D, room, cfg, dtype=dt)
    cache.append(K.cuda(), V.cuda())
    idx = nsa._resolve_block_indices(Q.cuda(), K.cuda(), block_size_m=64, block_size_n=64, top_k=k, causal=True, scale=D ** -0.5, force_first=1,
                                     force_local=2, shared_per_group=group).cpu()
    ref = O.nsa_forward(Q.float(), K.float(), V.float(), gate_logits=gates, block_indices=idx, block_size_c=32, stride_c=16, top_k=k,
                        window_size=512, force_first=1, force_local=2, group_shared=group)
    filled = torch.full((1,), n, dtype=torch.int32, device="cuda")
    for out in (nsa.nsa_decode(Q.cuda(), cache, gate_logits=gates.cuda()), decode._step(Q.cuda(), cache, gates.cuda(), D ** -0.5, filled)):
        err = float((out.float().cpu() - ref).norm() / ref.norm())
        assert err <= 1e-2, err


@pytest.mark.parametrize("n", [1000, 20000, 70000, 140000])
def test_tied_scores_take_the_lowest_blocks(nsa, n):
    """All keys zero: every block scores 0 in all four warps' quarters.  V of a block is its index mod 64, so the selected branch's
    average names the blocks that were taken: 0 to 5 and the forced two at the end."""
    D, k = 64, 8
    nk = (n + 63) // 64
    K = torch.zeros(1, 1, n, D)
    V = (torch.arange(n) // 64 % 64).float()[None, None, :, None].expand(1, 1, n, D)
    Q = torch.randn(1, 2, 1, D, generator=torch.Generator().manual_seed(1)).bfloat16()
    cfg = nsa.NSAConfig(block_size_c=32, stride_c=16, top_k=k, window_size=64, force_first=1, force_local=2, select_per_group=True)
    cache = nsa.KVCache(1, 1, D, n + 64, cfg)
    cache.append(K.bfloat16().cuda(), V.bfloat16().cuda())
    gates = torch.tensor([-50.0, 50.0, -50.0]).expand(1, 2, 1, 3).contiguous().cuda()      # the selected branch alone
    out = nsa.nsa_decode(Q.cuda(), cache, gate_logits=gates).float().cpu()
    blocks = [0, 1, 2, 3, 4, 5, nk - 2, nk - 1]
    rows = torch.cat([torch.arange(c * 64, min(c * 64 + 64, n)) for c in blocks])
    want = float((rows // 64 % 64).float().mean())
    assert float((out - want).abs().max()) <= want * 2**-7, (float(out.mean()), want)       # one bf16 rounding of P's sum, one of the result
