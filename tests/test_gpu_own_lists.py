"""One block list per query head at D=64 on tcgen05: row groups that walk lists of their own, of different lengths, with
entries that do not count and entries that count twice."""
import pytest
import torch

from helpers import check_out_lse, make_qkv, max_abs
from oracle import nsa_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nsa():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import nsa_from_scratch_b200 as m
    from nsa_from_scratch_b200 import ops
    yield m
    ops.device_status()


def _lists(B, H, nq, nk, k, seed):
    """Random lists, unsorted: -1, blocks of the future, a repeated block, and rows that list nothing."""
    g = torch.Generator().manual_seed(seed)
    idx = torch.randint(0, nk, (B, H, nq, k), generator=g, dtype=torch.int32)
    idx[torch.rand(idx.shape, generator=g) < 0.2] = -1
    if k > 1:
        idx[:, 0, :, 1] = idx[:, 0, :, 0]
    idx[:, :, nq // 2] = -1
    return idx


# (heads, KV heads): four query blocks of a head, two heads with two blocks, four heads with one block to a work item
@pytest.mark.parametrize("H,Hkv", [(3, 3), (4, 2), (8, 2)])
@pytest.mark.parametrize("Tq,Tk,k,window", [(64, 64, 1, 64), (257, 257, 5, 70), (300, 655, 16, 512), (130, 5000, 64, 33)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_forward_and_selected_branch(nsa, H, Hkv, Tq, Tk, k, window, dtype):
    Q, K, V, g = make_qkv(5, 1, H, Hkv, Tq, Tk, 64, dtype)
    gates = torch.randn(1, H, Tq, 3, generator=g)
    idx = _lists(1, H, (Tq + 63) // 64, (Tk + 63) // 64, k, seed=k)
    cfg = nsa.NSAConfig(block_size_c=32, stride_c=16, top_k=k, window_size=window)
    q, kk, v, i = Q.cuda(), K.cuda(), V.cuda(), idx.cuda()
    ref_s, ref_lse = O.selected_attention(Q, K, V, idx)
    out_s, lse = nsa.selected_attention(q, kk, v, top_k=k, block_indices=i)
    check_out_lse(out_s, lse, ref_s, ref_lse, 2e-2)        # the 16-bit bound of the other kernels' tests
    out = nsa.nsa_forward(q, kk, v, cfg, gate_logits=gates.cuda(), block_indices=i)
    ref = O.nsa_forward(Q, K, V, block_size_c=32, stride_c=16, top_k=k, window_size=window, gate_logits=gates, block_indices=idx)
    assert max_abs(out, ref) <= 2e-2, max_abs(out, ref)


@pytest.mark.parametrize("H,Hkv", [(3, 3), (4, 2), (8, 2)])
@pytest.mark.parametrize("block", [0, 5])                  # 0 also stands in for the entries of a list that has ended
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_rows_take_nothing_from_blocks_they_do_not_list(nsa, H, Hkv, block, bad):
    T = 1024
    Q, K, V, _ = make_qkv(8, 1, H, Hkv, T, T, 64)
    g = torch.Generator().manual_seed(4)
    idx = torch.randint(0, 15, (1, H, 16, 4), generator=g, dtype=torch.int32)
    idx += (idx >= block).int()                             # every block but `block`
    idx[torch.rand(idx.shape, generator=g) < 0.3] = -1
    idx[:, :, 11] = -1
    idx[:, 1, 9, 2] = block                                 # one list names it
    poisoned = V.clone()
    poisoned[:, :, block * 64 + 7] = bad
    out, lse = (x.cpu() for x in nsa.selected_attention(Q.cuda(), K.cuda(), V.cuda(), top_k=4, block_indices=idx.cuda(), causal=False))
    got, glse = (x.cpu() for x in nsa.selected_attention(Q.cuda(), K.cuda(), poisoned.cuda(), top_k=4, block_indices=idx.cuda(), causal=False))
    rows = torch.ones(1, H, T, dtype=torch.bool)
    rows[:, 1, 9 * 64:10 * 64] = False
    assert torch.equal(glse, lse) and torch.equal(got[rows], out[rows])
    assert not torch.isfinite(got[~rows]).any()
