"""The decoding step's entry: which calls it takes and which it leaves to the general path, decided from the sizes alone."""
import ctypes as C

from nsa_from_scratch_b200 import _lib as L


def _args(**kw):
    a = L.DecodeArgs(B=1, H=8, Hkv=2, Tq=1, len=900, D=128, max_len=1024, nc_alloc=63, nk_alloc=16, cmp_block=32, cmp_stride=16, bm=64, bn=64,
                     top_k=16, window=512, force_first=1, force_local=2, per_group=1, gate_act=L.GATE_SIGMOID, dtype=L.BF16, gate_dtype=0, scale=0.1)
    for k, v in kw.items():
        setattr(a, k, v)
    return a


def _ws(**kw):
    return L.load().nsa_decode_ws_bytes(C.byref(_args(**kw)))


def test_negative_forced_counts_are_left_to_the_path_that_refuses_them():
    assert _ws() > 0
    assert _ws(force_first=-1) == 0 and _ws(force_local=-1) == 0


def test_block_means_that_do_not_cover_the_cache_are_an_error():
    count = C.c_int32(0)
    dev = C.addressof(count)                                 # not read: sizes decide
    assert _ws(nk_alloc=15) > 0 and _ws(nk_alloc=14) == -1   # 900 positions: 15 blocks
    assert _ws(dyn_len=dev) > 0 and _ws(nk_alloc=15, dyn_len=dev) == -1
    assert b"do not cover" in L.load().nsa_last_error()
    a = _args(nk_alloc=14, Q=1, K=1, V=1, Kc=1, Vc=1, Kb=1, out=1, ws=256, ws_bytes=1 << 40)
    assert L.load().nsa_decode(C.byref(a), None) == -1
