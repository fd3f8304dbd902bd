// The whole NSA forward behind one call: window means of Q, K and V (one launch), block selection, and the fused
// three-branch attention launch, in a workspace the caller provides.  A short forward is bound by the host and by
// the gaps between its launches: issued from here the step costs three launches (six before: one per pooled tensor)
// and one library call, and the small kernels follow each other through programmatic dependent launch.
// The training forward keeps what the backward needs (the branch outputs and their log-sum-exps, the block lists, the
// pooled keys and values); the backward is one call too (attn_bwd_stream.cu).
#include "common.cuh"

namespace nsa {

int pool_mean_multi(const PoolJob*, int, int, int, cudaStream_t);
int select_blocks(const void*, const void*, int32_t*, int, int, int, int, int, int, int, int, int, int, int, float, int,
                  int, int, int, const int32_t*, cudaStream_t);
bool attention_fwd_tc5_supports(const nsa_fwd_args&);
int fp8_dequantize(const void*, void*, long long, int, float, cudaStream_t);
int combine(const void*, const void*, const void*, const void*, void*, long long, int, int, int, int, int, cudaStream_t);
long long backward_ws_bytes(const nsa_forward_args&);
int backward_stream(const nsa_forward_args&, const void*, const void*, const float*, const int32_t*, const void*, const void*, void*, void*, void*,
                    void*, cudaStream_t);

static bool fp8(int dt) { return dt == NSA_FP8_E4M3 || dt == NSA_FP8_E5M2; }

struct ForwardPlan {
  int Nc, nq, nk, k_sel, Hi;
  bool select, dequant, dequant_q;
  size_t o_qb, o_kb, o_kc, o_vc, o_idx, o_k16, o_v16, o_q16, total;
};

static int forward_plan(const nsa_forward_args& f, ForwardPlan& pl) {
  NSA_REQUIRE(f.B > 0 && f.H > 0 && f.Hkv > 0 && f.H % f.Hkv == 0, NSA_ERR_ARG, "forward: B=%d H=%d Hkv=%d (H must be a multiple of Hkv)",
              f.B, f.H, f.Hkv);
  NSA_REQUIRE(f.Tq > 0 && f.Tk > 0 && f.D > 0 && f.D % 8 == 0, NSA_ERR_ARG, "forward: Tq=%d Tk=%d D=%d", f.Tq, f.Tk, f.D);
  NSA_REQUIRE(f.cmp_block > 0 && f.cmp_stride > 0 && f.cmp_stride <= f.cmp_block, NSA_ERR_ARG, "forward: compression block %d stride %d",
              f.cmp_block, f.cmp_stride);
  NSA_REQUIRE(f.bm > 0 && f.bn > 0 && f.top_k > 0, NSA_ERR_ARG, "forward: bm=%d bn=%d top_k=%d", f.bm, f.bn, f.top_k);
  pl.Nc = f.cmp_stride == f.cmp_block ? (f.Tk + f.cmp_block - 1) / f.cmp_block
                                      : (f.Tk >= f.cmp_block ? (f.Tk - f.cmp_block) / f.cmp_stride + 1 : 0);
  pl.nq = (f.Tq + f.bm - 1) / f.bm;
  pl.nk = (f.Tk + f.bn - 1) / f.bn;
  pl.select = f.has_idx == 0;
  pl.Hi = pl.select ? (f.per_group ? f.Hkv : f.H) : f.Hi;
  pl.k_sel = pl.select ? (f.top_k < pl.nk ? f.top_k : pl.nk) : f.top_k;
  // fp8 storage: K and V, whose tiles every attending query block uses again, are dequantised once in front of the
  // tcgen05 kernel, which takes them as bf16 beside an fp8 Q; the generic kernel converts as it loads
  nsa_fwd_args a = {};
  a.q_dtype = f.q_dtype; a.kv_dtype = NSA_BF16;
  a.D = f.D; a.scale = f.scale; a.q_scale = f.q_scale; a.k_scale = f.k_scale; a.v_scale = f.v_scale;
  a.bm = f.bm; a.bn = f.bn; a.top_k = pl.k_sel; a.Nc = pl.Nc;
  a.branches = NSA_BRANCH_COMPRESSED | NSA_BRANCH_SELECTED | NSA_BRANCH_SLIDING;
  pl.dequant = fp8(f.q_dtype) && f.engine != NSA_ENGINE_GENERIC && attention_fwd_tc5_supports(a);
  // one list per query head at D = 64: Q as well, for the kernel whose row groups walk their own lists (16-bit storage)
  pl.dequant_q = pl.dequant && f.D == 64 && pl.Hi == f.H && f.engine == NSA_ENGINE_AUTO;
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  const size_t row = (size_t)f.D * 2, kv = (size_t)f.B * f.Hkv;
  size_t o = 0;
  pl.o_qb = o; if (pl.select) o = up(o + (size_t)f.B * f.H * pl.nq * row);
  pl.o_kb = o; if (pl.select) o = up(o + kv * pl.nk * row);
  pl.o_kc = o; o = up(o + kv * pl.Nc * row);
  pl.o_vc = o; o = up(o + kv * pl.Nc * row);
  pl.o_idx = o; if (pl.select) o = up(o + (size_t)f.B * pl.Hi * pl.nq * pl.k_sel * 4);
  pl.o_k16 = o; if (pl.dequant) o = up(o + kv * f.Tk * row);
  pl.o_v16 = o; if (pl.dequant) o = up(o + kv * f.Tk * row);
  pl.o_q16 = o; if (pl.dequant_q) o = up(o + (size_t)f.B * f.H * f.Tq * row);
  pl.total = o < 256 ? 256 : o;
  return NSA_OK;
}

// Everything of the attention launch but the branches and what is written.
static nsa_fwd_args attention_args(const nsa_forward_args& f, const ForwardPlan& pl, const void* K, const void* V, const void* Kc, const void* Vc,
                                   const int32_t* idx) {
  nsa_fwd_args a = {};
  a.Q = f.Q; a.K = K; a.V = V; a.Kc = Kc; a.Vc = Vc; a.idx = idx;
  a.B = f.B; a.H = f.H; a.Hkv = f.Hkv; a.Hi = pl.Hi; a.Tq = f.Tq; a.Tk = f.Tk; a.D = f.D; a.offset = f.Tk - f.Tq;
  a.Nc = pl.Nc; a.cmp_block = f.cmp_block; a.cmp_stride = f.cmp_stride;
  a.cmp_offset = (f.cmp_stride == f.cmp_block ? pl.Nc * f.cmp_block : f.Tk) - f.Tq;
  a.nq = pl.nq; a.top_k = pl.k_sel; a.bm = f.bm; a.bn = f.bn; a.sel_key_limit = pl.nk * f.bn;
  a.window = f.window; a.causal = f.causal;
  a.gate_act = f.gate_act; a.q_dtype = f.q_dtype; a.kv_dtype = pl.dequant ? NSA_BF16 : f.q_dtype;
  a.scale = f.scale; a.q_scale = f.q_scale; a.k_scale = f.k_scale; a.v_scale = f.v_scale;
  a.engine = f.engine; a.io_layout = f.io_layout;
  return a;
}

}  // namespace nsa

using namespace nsa;

extern "C" {

int64_t nsa_forward_ws_bytes(const nsa_forward_args* f) {
  NSA_REQUIRE(f, NSA_ERR_ARG, "forward: NULL argument block");
  ForwardPlan pl;
  const int rc = forward_plan(*f, pl);
  return rc != NSA_OK ? rc : (int64_t)pl.total;
}

int nsa_forward(const nsa_forward_args* fa, nsa_stream_t stream) {
  NSA_REQUIRE(fa, NSA_ERR_ARG, "forward: NULL argument block");
  const nsa_forward_args& f = *fa;
  ForwardPlan pl;
  int rc = forward_plan(f, pl);
  if (rc != NSA_OK) return rc;
  NSA_REQUIRE(f.Q && f.K && f.V && f.out && (pl.select || f.idx), NSA_ERR_ARG, "forward: NULL pointer");
  NSA_REQUIRE(f.ws && f.ws_bytes >= (int64_t)pl.total && (reinterpret_cast<uintptr_t>(f.ws) & 255) == 0, NSA_ERR_ARG,
              "forward: needs %lld bytes of workspace (256-byte aligned), %lld given", (long long)pl.total, (long long)f.ws_bytes);
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* ws = reinterpret_cast<unsigned char*>(f.ws);
  const int BH = f.B * f.H, BKV = f.B * f.Hkv;
  PoolJob jobs[4];
  int n = 0;
  if (pl.select) {
    jobs[n++] = {f.Q, ws + pl.o_qb, f.Tq, f.bm, f.bm, pl.nq, BH, f.q_scale, 0u};
    jobs[n++] = {f.K, ws + pl.o_kb, f.Tk, f.bn, f.bn, pl.nk, BKV, f.k_scale, 0u};
  }
  jobs[n++] = {f.K, ws + pl.o_kc, f.Tk, f.cmp_block, f.cmp_stride, pl.Nc, BKV, f.k_scale, 0u};
  jobs[n++] = {f.V, ws + pl.o_vc, f.Tk, f.cmp_block, f.cmp_stride, pl.Nc, BKV, f.v_scale, 0u};
  if ((rc = pool_mean_multi(jobs, n, f.D, f.q_dtype, st)) != NSA_OK) return rc;
  const int cdt = fp8(f.q_dtype) ? NSA_BF16 : f.q_dtype;
  const int32_t* idx = f.idx;
  if (pl.select) {
    int32_t* out = reinterpret_cast<int32_t*>(ws + pl.o_idx);
    // the causal legality offset of the selection uses the lengths padded to the block sizes
    if ((rc = select_blocks(ws + pl.o_qb, ws + pl.o_kb, out, f.B, f.H, f.Hkv, pl.nq, pl.nk, f.D, f.top_k, f.bm, f.bn,
                            pl.nk * f.bn - pl.nq * f.bm, f.causal, f.scale, f.force_first, f.force_local, f.per_group, cdt, nullptr, st)) != NSA_OK)
      return rc;
    idx = out;
  }
  const void *K = f.K, *V = f.V;
  if (pl.dequant) {
    const long long n_kv = (long long)BKV * f.Tk * f.D;
    if ((rc = fp8_dequantize(K, ws + pl.o_k16, n_kv, f.q_dtype, f.k_scale, st)) != NSA_OK) return rc;
    if ((rc = fp8_dequantize(V, ws + pl.o_v16, n_kv, f.q_dtype, f.v_scale, st)) != NSA_OK) return rc;
    K = ws + pl.o_k16;
    V = ws + pl.o_v16;
  }
  nsa_fwd_args a = attention_args(f, pl, K, V, ws + pl.o_kc, ws + pl.o_vc, idx);
  if (pl.dequant_q) {
    if ((rc = fp8_dequantize(f.Q, ws + pl.o_q16, (long long)BH * f.Tq * f.D, f.q_dtype, f.q_scale, st)) != NSA_OK) return rc;
    a.Q = ws + pl.o_q16;
    a.q_dtype = NSA_BF16;
    a.q_scale = a.k_scale = a.v_scale = 1.f;
  }
  a.out = f.out; a.gates = f.gates; a.gate_dtype = f.gate_dtype;
  a.branches = NSA_BRANCH_COMPRESSED | NSA_BRANCH_SELECTED | NSA_BRANCH_SLIDING;
  a.fused = 1;
  return nsa_attention_fwd(&a, stream);
}

int64_t nsa_backward_ws_bytes(const nsa_forward_args* f) {
  NSA_REQUIRE(f, NSA_ERR_ARG, "backward: NULL argument block");
  return backward_ws_bytes(*f);
}

int nsa_forward_train(const nsa_forward_args* fa, void* branch_out, float* branch_lse, int32_t* idx, void* Kc, void* Vc, nsa_stream_t stream) {
  NSA_REQUIRE(fa, NSA_ERR_ARG, "forward (training): NULL argument block");
  const nsa_forward_args& f = *fa;
  ForwardPlan pl;
  int rc = forward_plan(f, pl);
  if (rc != NSA_OK) return rc;
  NSA_REQUIRE(f.Q && f.K && f.V && f.out && branch_out && branch_lse && Kc && Vc && (pl.select ? idx != nullptr : f.idx != nullptr), NSA_ERR_ARG,
              "forward (training): NULL pointer");
  NSA_REQUIRE(!fp8(f.q_dtype) && f.io_layout == 0, NSA_ERR_UNSUPPORTED, "forward (training): 16-bit storage in the default layout only");
  NSA_REQUIRE(!pl.select || (f.ws && f.ws_bytes >= (int64_t)pl.total), NSA_ERR_ARG, "forward (training): needs %lld bytes of workspace, %lld given",
              (long long)pl.total, (long long)f.ws_bytes);
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* ws = reinterpret_cast<unsigned char*>(f.ws);
  const int BH = f.B * f.H, BKV = f.B * f.Hkv;
  PoolJob jobs[4];
  int n = 0;
  if (pl.select) {
    jobs[n++] = {f.Q, ws + pl.o_qb, f.Tq, f.bm, f.bm, pl.nq, BH, 1.f, 0u};
    jobs[n++] = {f.K, ws + pl.o_kb, f.Tk, f.bn, f.bn, pl.nk, BKV, 1.f, 0u};
  }
  jobs[n++] = {f.K, Kc, f.Tk, f.cmp_block, f.cmp_stride, pl.Nc, BKV, 1.f, 0u};
  jobs[n++] = {f.V, Vc, f.Tk, f.cmp_block, f.cmp_stride, pl.Nc, BKV, 1.f, 0u};
  if ((rc = pool_mean_multi(jobs, n, f.D, f.q_dtype, st)) != NSA_OK) return rc;
  if (pl.select && (rc = select_blocks(ws + pl.o_qb, ws + pl.o_kb, idx, f.B, f.H, f.Hkv, pl.nq, pl.nk, f.D, f.top_k, f.bm, f.bn,
                                       pl.nk * f.bn - pl.nq * f.bm, f.causal, f.scale, f.force_first, f.force_local, f.per_group, f.q_dtype,
                                       nullptr, st)) != NSA_OK)
    return rc;
  const size_t rows = (size_t)BH * f.Tq, bytes = rows * f.D * 2;
  unsigned char* bo = reinterpret_cast<unsigned char*>(branch_out);
  for (int br = 0; br < 3; ++br) {
    nsa_fwd_args a = attention_args(f, pl, f.K, f.V, Kc, Vc, pl.select ? idx : f.idx);
    a.out = bo + br * bytes; a.lse = branch_lse + br * rows;
    a.branches = 1 << br;
    if ((rc = nsa_attention_fwd(&a, stream)) != NSA_OK) return rc;
  }
  return combine(bo, bo + bytes, bo + 2 * bytes, f.gates, f.out, (long long)rows, f.D, f.gate_act, f.q_dtype, f.gates ? f.gate_dtype : f.q_dtype,
                 f.q_dtype, st);
}

int nsa_backward(const nsa_forward_args* f, const void* dO, const void* branch_out, const float* branch_lse, const int32_t* idx, const void* Kc,
                 const void* Vc, void* dQ, void* dK, void* dV, void* dgates, nsa_stream_t stream) {
  NSA_REQUIRE(f, NSA_ERR_ARG, "backward: NULL argument block");
  NSA_REQUIRE(f->Q && f->K && f->V && dO && branch_out && branch_lse && idx && Kc && Vc && dQ && dK && dV, NSA_ERR_ARG, "backward: NULL pointer");
  return backward_stream(*f, dO, branch_out, branch_lse, idx, Kc, Vc, dQ, dK, dV, dgates, (cudaStream_t)stream);
}

}  // extern "C"
