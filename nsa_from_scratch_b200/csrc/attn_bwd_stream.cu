// Backward of the whole three-branch attention on tcgen05, D in {64,128}, 64-token blocks.  Two streaming kernels:
//
//   query pass (MODE 1): dQ of all three branches.  A thread block owns 128 query rows (two row groups of 64: two heads
//   that share a KV head, or two query blocks of one head) and streams every 64-key chunk they see -- pooled keys, listed
//   blocks, window -- through a TMA ring:
//       S = Q K^T   dP = dO V^T   dS = P (dP - d) scale (softmax warps)   dQ += dS K
//   dQ accumulates in TMEM across the branches and is written once, in 16 bits.
//
//   key pass (MODE 0): dK, dV of the pooled tokens and of the window.  A thread block owns 128 keys and streams (query
//   block, head) tiles of 64 rows.  The product is formed transposed (keys on the TMEM lanes), so P^T and dS^T are
//   A operands in TMEM where the softmax threads leave them, over the S^T and dP^T they were computed from:
//       S^T = K Q^T   dP^T = V dO^T   dV += P^T dO   dK += dS^T Q
//   Segments of a long query range add their sums to fp32 buffers with reductions in L2.
//
// The gates enter through the log-sum-exp: the gradient of branch i's output is g_i dO, so with P' = g_i P = exp(S - lse +
// ln g_i) both dV = P'^T dO and dS = P' (dP - d_i) hold with the ungated dO and d_i = dO . O_i.  Nothing of size
// [rows, D] is written between the gated combine's gradient and these kernels.  In fp16 a small gate would leave P' few
// bits: there lse2 gives 2^14 P', and dS and the dV sums take the factor back (kGatedPExp).
//
// What bounds a step (128 x 64 pairs): 512 clocks of exp2 on the special-function unit, about 350 of issue slots, 384 to
// 640 of MMAs; a step's own chain (MMA, TMEM load, exp2, TMEM store, MMA) is about 1700.  NBUF steps are therefore in flight,
// each with its own S/dP columns and its own group of four softmax warps, one warp per scheduler and group.
// Every wait is bounded as in the other tcgen05 kernels.
// Measured at B=2, T=32768, 12 heads over one KV head, D=64, 32/16 pooling, 16 listed blocks, window 512: query pass 1.10 ms
// for 2.0e9 pairs, key pass 0.83 ms for 1.2e9; the branch-by-branch backward it replaces took 1.27 ms (listed blocks) +
// 3.76 ms (mma.sync with fp32 atomics, pooled and window) + 2.6 ms of element-wise passes around them.
#include "common.cuh"
#include "tc5_ptx.cuh"

#include <cudaTypedefs.h>
#include <type_traits>

namespace nsa {

using namespace tc5;

int make_map(CUtensorMap* m, const void* ptr, long long slabs, long long rows, int D, int dtype);   // attn_fwd_tc5.cu

__device__ int g_bst_status;   // 0 ok; otherwise (1 + id of the barrier a wait gave up on)

constexpr int BST_MAX_SEL = 64;                 // listed blocks per query block
constexpr int BST_THREADS = 448;                // TMA producer, MMA issuer, 12 softmax warps
constexpr int BST_NST_MAX = 8;

// S/dP buffers in TMEM: three, except where two accumulators of 128 columns leave room for two
__host__ __device__ constexpr int bst_nbuf(int D, int mode) { return mode == 0 && D == 128 ? 2 : 3; }
__host__ __device__ constexpr int bst_stages(int D) { return D == 64 ? 8 : 4; }

struct BstParams {
  CUtensorMap tmQ, tmdO, tmK, tmV, tmKc, tmVc;
  int B, H, Hkv, Hi, Tq, Tqp, Tk, Nc, nq, nk, top_k, G;
  int offset, cmp_offset, cmp_block, cmp_stride, sel_limit, window, causal;
  float scale, scale_log2;
  const float* lse2;       // [3][B*H][Tqp]: log2-sum-exp minus log2 of the branch's gate (fp16: minus kGatedPExp)
  const float* dls;        // [3][B*H][Tqp]: (dO . O_branch) * scale (fp16: * kGatedPInv)
  const int32_t* idx;
  void* dQ;
  float *dK, *dV, *dKc, *dVc;   // [B*Hkv][Tk | Nc][D], added to
  int two_qb;              // query pass: the two row groups are query blocks 2t, 2t+1 of one head (1) or two heads of one block (0)
  int n_pairs;             // query pass: tiles per (batch, KV head) and query block (two_qb == 0)
  int kt_cmp, seg_cmp, kt_sld, seg_sld, L;   // key pass: key tiles and most segments per tile; steps per segment
};

enum { BS_RES = 0, BS_STFULL = 1, BS_STEMPTY = BS_STFULL + BST_NST_MAX, BS_SFULL = BS_STEMPTY + BST_NST_MAX, BS_PFULL = BS_SFULL + 3,
       BS_ACC = BS_PFULL + 3, BS_QTMEM = BS_ACC + 1, BS_COUNT = BS_QTMEM + 1 };

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void red_add4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

template <int D, int FMT, int MODE>
__global__ void __launch_bounds__(BST_THREADS, 1) nsa_bwd_stream_kernel(const __grid_constant__ BstParams p) {
  using T = typename std::conditional<FMT == 1, __nv_bfloat16, __half>::type;
  constexpr int DH = D / 64;                    // 64-element (128-byte) halves of a row
  constexpr int T128 = DH * 128 * 128;          // bytes of a 128-row tile (halves 16384 bytes apart)
  constexpr int T64 = DH * 64 * 128;            // bytes of a 64-row tile (halves 8192 bytes apart)
  constexpr int RES_BYTES = 2 * T128;           // resident: Q,dO (query pass) or K,V (key pass)
  constexpr int ST_BYTES = 2 * T64;             // a ring stage: K,V or Q,dO
  constexpr int NST = bst_stages(D);
  constexpr int NBUF = bst_nbuf(D, MODE);
  // TMEM columns: NBUF x (S 64, dP 64), then the accumulators, then (query pass, D = 64) Q and dO as A operands
  constexpr int C_ACC = NBUF * 128;
  constexpr bool RES_TMEM = MODE == 1 && D == 64;
  constexpr int C_Q = 448, C_DO = 480;

  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sRes = smem_u32(smem), sSt = sRes + RES_BYTES;
  float* vec = reinterpret_cast<float*>(smem + RES_BYTES + NST * ST_BYTES);      // key pass: [NST][2][64] lse2, dls of the stage's rows
  __shared__ __align__(8) uint64_t bars[BS_COUNT];
  __shared__ int ent_blk[2 * BST_MAX_SEL], sel_list[2 * BST_MAX_SEL];
  __shared__ unsigned char ent_p[2 * BST_MAX_SEL], sel_mask[2 * BST_MAX_SEL];
  __shared__ int sel_n;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto bar = [&](int id) { return smem_u32(&bars[id]); };

  // ---- work item ------------------------------------------------------------------------------
  int owner = 0;                                         // b * Hkv + hk
  int g_head[2] = {0, 0}, g_qb[2] = {0, 0};              // query pass: head within the group and query block of the row groups
  bool g_ok[2] = {false, false};
  int br_k = 0, k0 = 0, qb_hi = 0, e0 = 0, n_steps = 0;  // key pass: branch, first key, last query block, first step, steps
  const int NL = p.B * p.Hkv;
  if constexpr (MODE == 1) {
    if (p.two_qb) {
      const int t = (p.nq + 1) / 2 - 1 - (int)(blockIdx.x / (unsigned)(NL * p.G));      // long rows first
      const int rem = (int)(blockIdx.x % (unsigned)(NL * p.G));
      owner = rem / p.G;
      g_head[0] = g_head[1] = rem % p.G;
      g_qb[0] = 2 * t; g_qb[1] = 2 * t + 1;
      g_ok[0] = true; g_ok[1] = g_qb[1] < p.nq;
    } else {
      const int per = NL * p.n_pairs;
      const int qb = p.nq - 1 - (int)(blockIdx.x / (unsigned)per);
      const int rem = (int)(blockIdx.x % (unsigned)per);
      owner = rem / p.n_pairs;
      g_head[0] = 2 * (rem % p.n_pairs); g_head[1] = g_head[0] + 1;
      g_qb[0] = g_qb[1] = qb;
      g_ok[0] = true; g_ok[1] = g_head[1] < p.G;
    }
  } else {
    // blocks that run together share query rows (the key tile varies fastest), segments start at the last query block
    unsigned x = blockIdx.x;
    const unsigned n_cmp = (unsigned)(NL * p.kt_cmp * p.seg_cmp);
    br_k = x < n_cmp ? 0 : 2;
    if (br_k) x -= n_cmp;
    const int nkt = br_k ? p.kt_sld : p.kt_cmp;
    const int kt = (int)(x % (unsigned)nkt);
    owner = (int)(x / (unsigned)nkt) % NL;
    const int seg = (int)(x / (unsigned)(nkt * NL));
    k0 = kt * 128;
    const int k1 = min(k0 + 127, (br_k ? p.Tk : p.Nc) - 1);
    int i_lo = 0, i_hi = p.Tq - 1;                       // query rows that see one of the keys
    if (br_k == 0) {
      if (p.causal) i_lo = max(0, k0 * p.cmp_stride + p.cmp_block - 1 - p.cmp_offset);
    } else {
      i_lo = max(0, k0 - p.offset - (p.causal ? 0 : p.window));
      i_hi = min(i_hi, k1 - p.offset + (p.causal ? p.window - 1 : p.window));
    }
    if (i_lo > i_hi) return;
    qb_hi = i_hi / 64;
    const int total = (qb_hi - i_lo / 64 + 1) * p.G;
    e0 = seg * p.L;
    n_steps = min(p.L, total - e0);
    if (n_steps <= 0) return;
  }
  const int b = owner / p.Hkv, hk = owner % p.Hkv;

  if (tid == 0) {
    abort_flag = 0;
    for (int i = 0; i < BS_COUNT; ++i)
      mbar_init(bar(i), (i >= BS_PFULL && i < BS_PFULL + 3) ? 128 : (i == BS_QTMEM ? 256 : 1));
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(smem_u32(&tmem_base_s), 512); tmem_relinquish(); }
  if (MODE == 1 && warp == 2) {
    // The listed key blocks of the two row groups, merged: a block both list is staged once with both mask bits; a block
    // listed p times by one group is visited p times.
    const int hA = p.Hi == p.H ? hk * p.G + g_head[0] : hk, hB = p.Hi == p.H ? hk * p.G + g_head[1] : hk;
    const bool shared = hA == hB && g_qb[0] == g_qb[1];
    const int n_ent = (shared ? 1 : 2) * p.top_k;
    for (int i = lane; i < n_ent; i += 32) {
      const int g = i / p.top_k;
      int blk = -1;
      if (g_ok[g]) {
        const int per_b = p.Hi;
        blk = p.idx[(((size_t)b * per_b + (g ? hB : hA)) * p.nq + g_qb[g]) * p.top_k + i % p.top_k];
        const int last_pos = min(g_qb[g] * 64 + 64, p.Tq) - 1 + p.offset;
        if (blk < 0 || blk >= p.nk || (p.causal && (long long)blk * 64 > last_pos)) blk = -1;
      }
      ent_blk[i] = blk;
    }
    __syncwarp();
    if (!shared) {
      for (int i = lane; i < n_ent; i += 32) {            // how many earlier entries of the same group name the same block
        int pc = 0;
        for (int j = i / p.top_k * p.top_k; j < i; ++j) pc += ent_blk[j] == ent_blk[i];
        ent_p[i] = (unsigned char)pc;
      }
      __syncwarp();
    }
    int n = 0;
    for (int i0 = 0; i0 < n_ent; i0 += 32) {
      const int i = i0 + lane;
      bool lead = i < n_ent && ent_blk[i] >= 0;
      unsigned msk = shared ? 3u : (i < p.top_k ? 1u : 2u);
      if (lead && !shared) {
        const int other = i < p.top_k ? p.top_k : 0;
        for (int j = other; j < other + p.top_k; ++j)
          if (ent_blk[j] == ent_blk[i] && ent_p[j] == ent_p[i]) { msk = 3u; lead = i < p.top_k; }
      }
      const unsigned bal = __ballot_sync(0xffffffffu, lead);
      if (lead) {
        const int pos = n + __popc(bal & ((1u << lane) - 1));
        sel_list[pos] = ent_blk[i];
        sel_mask[pos] = (unsigned char)msk;
      }
      n += __popc(bal);
    }
    if (lane == 0) sel_n = n;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;

  // what query row i sees in a branch: keys lo..hi
  auto bounds = [&](int br, int i, int& lo, int& hi) {
    lo = 0;
    if (br == 0) {
      hi = p.Nc - 1;
      if (p.causal) {
        const int num = i + p.cmp_offset - (p.cmp_block - 1);
        hi = num < 0 ? -1 : min(hi, num / p.cmp_stride);
      }
    } else if (br == 1) {
      hi = p.causal ? min(i + p.offset, p.sel_limit - 1) : p.sel_limit - 1;
    } else {
      const int pos = i + p.offset;
      lo = max(0, p.causal ? pos - p.window + 1 : pos - p.window);
      hi = min(p.Tk - 1, p.causal ? pos : pos + p.window);
    }
  };
  // query pass: chunks of the three branches in sequence
  int n_ch[3] = {0, 0, 0}, sld_c0 = 0;
  if constexpr (MODE == 1) {
    const int q_first = g_qb[0] * 64, q_last = min((g_ok[1] ? g_qb[1] : g_qb[0]) * 64 + 64, p.Tq) - 1;
    int lo_f, hi_f, lo_l, hi_l;
    bounds(0, q_last, lo_l, hi_l);
    n_ch[0] = hi_l < 0 ? 0 : hi_l / 64 + 1;
    n_ch[1] = sel_n;
    bounds(2, q_first, lo_f, hi_f);
    bounds(2, q_last, lo_l, hi_l);
    if (hi_l >= lo_f) { sld_c0 = lo_f / 64; n_ch[2] = hi_l / 64 - sld_c0 + 1; }
    n_steps = n_ch[0] + n_ch[1] + n_ch[2];
  }
  auto chunk = [&](int st, int& br, int& j0, int& mask) {
    mask = 3;
    if (st < n_ch[0]) { br = 0; j0 = st * 64; }
    else if (st < n_ch[0] + n_ch[1]) { br = 1; j0 = sel_list[st - n_ch[0]] * 64; mask = sel_mask[st - n_ch[0]]; }
    else { br = 2; j0 = (sld_c0 + st - n_ch[0] - n_ch[1]) * 64; }
  };
  // key pass: step -> (head, query block), from the last query block down, all heads of the group per block
  auto q_tile = [&](int st, int& hl, int& qb) { const int e = e0 + st; qb = qb_hi - e / p.G; hl = e % p.G; };
  const int oob_row = (p.Tq + 63) / 64 * 64;             // a box that starts here lies outside the tensor: zeros

  int fail_id = 0, last_st = -1;

  if (warp == 0) {
    // =============================== TMA producer ===============================
    const bool leader = elect_one();
    if (leader) {
      tma_prefetch_desc(&p.tmQ); tma_prefetch_desc(&p.tmdO); tma_prefetch_desc(&p.tmK); tma_prefetch_desc(&p.tmV);
      tma_prefetch_desc(&p.tmKc); tma_prefetch_desc(&p.tmVc);
      mbar_expect_tx(bar(BS_RES), RES_BYTES);
      for (int g = 0; g < 2; ++g)
        for (int dh = 0; dh < DH; ++dh) {
          const uint32_t d0 = sRes + dh * 16384 + g * 8192;
          if constexpr (MODE == 1) {
            const int slab = g_ok[g] ? b * p.H + hk * p.G + g_head[g] : 0, row = g_ok[g] ? g_qb[g] * 64 : oob_row;
            tma_load_3d(d0, &p.tmQ, bar(BS_RES), dh * 64, row, slab);
            tma_load_3d(d0 + T128, &p.tmdO, bar(BS_RES), dh * 64, row, slab);
          } else {
            tma_load_3d(d0, br_k ? &p.tmK : &p.tmKc, bar(BS_RES), dh * 64, k0 + g * 64, owner);
            tma_load_3d(d0 + T128, br_k ? &p.tmV : &p.tmVc, bar(BS_RES), dh * 64, k0 + g * 64, owner);
          }
        }
    }
    __syncwarp();
    for (int st = 0; st < n_steps; ++st) {
      const int s = st % NST;
      if (!__all_sync(0xffffffffu, mbar_wait(bar(BS_STEMPTY + s), ((st / NST) & 1) ^ 1, &abort_flag))) { fail_id = BS_STEMPTY + s + 1; break; }
      const uint32_t dst = sSt + s * ST_BYTES;
      if constexpr (MODE == 1) {
        int br, j0, mask;
        chunk(st, br, j0, mask);
        if (leader) {
          mbar_expect_tx(bar(BS_STFULL + s), ST_BYTES);
          for (int dh = 0; dh < DH; ++dh) {
            tma_load_3d(dst + dh * 8192, br ? &p.tmK : &p.tmKc, bar(BS_STFULL + s), dh * 64, j0, owner);
            tma_load_3d(dst + T64 + dh * 8192, br ? &p.tmV : &p.tmVc, bar(BS_STFULL + s), dh * 64, j0, owner);
          }
        }
      } else {
        int hl, qb;
        q_tile(st, hl, qb);
        if (leader) {
          const int bh = b * p.H + hk * p.G + hl;
          const size_t vi = ((size_t)br_k * p.B * p.H + bh) * p.Tqp + qb * 64;
          mbar_expect_tx(bar(BS_STFULL + s), ST_BYTES + 512);
          for (int dh = 0; dh < DH; ++dh) {
            tma_load_3d(dst + dh * 8192, &p.tmQ, bar(BS_STFULL + s), dh * 64, qb * 64, bh);
            tma_load_3d(dst + T64 + dh * 8192, &p.tmdO, bar(BS_STFULL + s), dh * 64, qb * 64, bh);
          }
          bulk_g2s(smem_u32(vec + s * 128), p.lse2 + vi, 256, bar(BS_STFULL + s));
          bulk_g2s(smem_u32(vec + s * 128 + 64), p.dls + vi, 256, bar(BS_STFULL + s));
        }
      }
      last_st = st;
      __syncwarp();
    }
  } else if (warp == 1) {
    // =============================== MMA issuer ===============================
    const bool leader = elect_one();
    constexpr uint32_t IDESC_S = idesc_f16(FMT, 128, 64, 0, 0);      // [128 x 64] = A (K-major) B^T (K-major)
    constexpr uint32_t IDESC_ACC = idesc_f16(FMT, 128, D, 0, 1);     // [128 x D] += A (TMEM) B (MN-major)
    bool ok = __all_sync(0xffffffffu, mbar_wait(bar(BS_RES), 0, &abort_flag));
    if (!ok) fail_id = BS_RES + 1;
    if constexpr (RES_TMEM) {
      if (ok) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar(BS_QTMEM), 0, &abort_flag));
        if (!ok) fail_id = BS_QTMEM + 1;
        tc_fence_after();
      }
    }
    auto offA = [](int ks) { return (uint32_t)(((ks >> 2) * 16384 + (ks & 3) * 32) >> 4); };
    auto offB = [](int ks) { return (uint32_t)(((ks >> 2) * 8192 + (ks & 3) * 32) >> 4); };
    const uint64_t aS = smem_desc_sw128(sRes, 16, 1024), aP = smem_desc_sw128(sRes + T128, 16, 1024);
    auto issue_sdp = [&](int st, int s, int sb) {
      tc_fence_after();
      if (leader) {
        const uint32_t st_base = sSt + s * ST_BYTES;
        const uint64_t bS = smem_desc_sw128(st_base, 16, 1024), bP = smem_desc_sw128(st_base + T64, 16, 1024);
        const uint32_t tS = tmem + sb * 128, tdP = tS + 64;
        if constexpr (RES_TMEM) {
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) mma_ts(tS, tmem + C_Q + ks * 8, bS + offB(ks), IDESC_S, ks == 0 ? 0u : 1u);
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) mma_ts(tdP, tmem + C_DO + ks * 8, bP + offB(ks), IDESC_S, ks == 0 ? 0u : 1u);
        } else {
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) mma_ss(tS, aS + offA(ks), bS + offB(ks), IDESC_S, ks == 0 ? 0u : 1u);
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) mma_ss(tdP, aP + offA(ks), bP + offB(ks), IDESC_S, ks == 0 ? 0u : 1u);
        }
        tc_commit(bar(BS_SFULL + sb));
      }
      __syncwarp();
    };
    auto issue_acc = [&](int st, int s, int sb) {
      tc_fence_after();
      if (leader) {
        const uint32_t st_base = sSt + s * ST_BYTES;
        const uint32_t tS = tmem + sb * 128, tdP = tS + 64;
        const uint64_t b0 = smem_desc_sw128(st_base, 8192, 1024), b1 = smem_desc_sw128(st_base + T64, 8192, 1024);
        if constexpr (MODE == 1) {
          // dQ += dS K: dS lies over S
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) mma_ts(tmem + C_ACC, tS + ks * 8, b0 + ks * 128, IDESC_ACC, (st > 0 || ks > 0) ? 1u : 0u);
        } else {
          // dV += P^T dO, dK += dS^T Q: P^T lies over S^T, dS^T over dP^T
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) mma_ts(tmem + C_ACC, tS + ks * 8, b1 + ks * 128, IDESC_ACC, (st > 0 || ks > 0) ? 1u : 0u);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) mma_ts(tmem + C_ACC + D, tdP + ks * 8, b0 + ks * 128, IDESC_ACC, (st > 0 || ks > 0) ? 1u : 0u);
        }
        tc_commit(bar(BS_STEMPTY + s));
      }
      __syncwarp();
    };
    // Whatever is ready is issued.  S/dP of step ns overwrites the buffer that the accumulate of step ns - NBUF reads: that
    // one was issued before it, and the tensor pipe executes in order of issue.
    int ns = 0, na = 0, s_ns = 0, s_na = 0, b_ns = 0, b_na = 0, ph_ns = 0, ph_na = 0;
    long long idle = 0;
    while (na < n_steps && ok) {
      bool did = false;
      if (ns < n_steps && ns - na < NBUF) {
        if (__all_sync(0xffffffffu, mbar_test_wait(bar(BS_STFULL + s_ns), ph_ns))) {
          issue_sdp(ns, s_ns, b_ns);
          ++ns; did = true;
          if (++s_ns == NST) { s_ns = 0; ph_ns ^= 1; }
          if (++b_ns == NBUF) b_ns = 0;
        }
      }
      if (na < ns) {
        if (__all_sync(0xffffffffu, mbar_test_wait(bar(BS_PFULL + b_na), ph_na))) {
          issue_acc(na, s_na, b_na);
          ++na; did = true;
          if (++s_na == NST) s_na = 0;
          if (++b_na == NBUF) { b_na = 0; ph_na ^= 1; }
        }
      }
      if (did) { idle = 0; continue; }
      ++idle;
      __nanosleep(20);
      if (idle > 65536) {
        if (abort_flag || idle > (1 << 23)) { abort_flag = 1; fail_id = (na < ns ? BS_PFULL + b_na : BS_STFULL + s_ns) + 1; ok = false; break; }
        __nanosleep(100);
      }
    }
    if (ok && n_steps > 0) {
      if (leader) tc_commit(bar(BS_ACC));
      __syncwarp();
    }
  } else {
    // =============================== softmax / epilogue ===============================
    const int grp = (warp - 2) >> 2;                       // handles the steps st = grp mod NBUF (with two buffers the third group idles)
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;                     // row of the 128-row tile == TMEM lane
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const uint32_t tS = tmem + lane_addr + grp * 128, tdP = tS + 64;
    const float sc = FMT == 1 ? p.scale : p.scale * kGatedPInv, sl2 = p.scale_log2;
    const int g2 = r >> 6;
    bool ok = true;

    // query pass: this row's constants, switched at the branch ends.  key pass: the query rows that see this lane's key.
    int qi = 0, lo = 0, hi = -1, cur_br = -1, i_min = 0, i_max = -1;
    float lse2 = 0.f, dls = 0.f;
    bool row_ok = false;
    const float *lse_row = nullptr, *dls_row = nullptr;
    if constexpr (MODE == 1) {
      qi = g_qb[g2] * 64 + (r & 63);
      row_ok = g_ok[g2] && qi < p.Tq;
      const size_t ri = row_ok ? ((size_t)b * p.H + hk * p.G + g_head[g2]) * p.Tqp + qi : 0;
      lse_row = p.lse2 + ri;
      dls_row = p.dls + ri;
    } else {
      const int j = k0 + r;
      i_max = p.Tq - 1;
      if (br_k == 0) {
        if (p.causal) i_min = max(0, j * p.cmp_stride + p.cmp_block - 1 - p.cmp_offset);
        if (j >= p.Nc) i_max = -1;
      } else {
        i_min = j - p.offset - (p.causal ? 0 : p.window);
        i_max = min(i_max, j - p.offset + (p.causal ? p.window - 1 : p.window));
        if (j >= p.Tk) i_max = -1;
      }
    }
    if constexpr (RES_TMEM) {
      // Q (group 0) and dO (group 1) from their swizzled tiles into TMEM: A operands that no MMA reads from shared memory again
      if (grp < 2) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar(BS_RES), 0, &abort_flag));
        if (!ok) fail_id = BS_RES + 1;
        if (ok) {
          const unsigned char* src = smem + grp * T128 + r * 128;
          uint32_t w[32];
#pragma unroll
          for (int c4 = 0; c4 < 8; ++c4) {
            const uint4 v = *reinterpret_cast<const uint4*>(src + ((c4 ^ (r & 7)) << 4));
            w[4 * c4] = v.x; w[4 * c4 + 1] = v.y; w[4 * c4 + 2] = v.z; w[4 * c4 + 3] = v.w;
          }
          tmem_st32(tmem + lane_addr + (grp == 0 ? C_Q : C_DO), w);
          tc_wait_st();
          tc_fence_before();
          mbar_arrive(bar(BS_QTMEM));
        }
      }
    }

    int ph = 0, s = grp % NST, ph_s = 0;
#pragma unroll 1
    for (int st = grp; st < n_steps && grp < NBUF && ok; st += NBUF) {
      // columns vlo..vhi of the chunk count for this row (query pass: keys; key pass: query rows)
      int vlo, vhi;
      if constexpr (MODE == 1) {
        int br, j0, mask;
        chunk(st, br, j0, mask);
        if (br != cur_br) {
          cur_br = br;
          bounds(br, qi, lo, hi);
          if (!row_ok) hi = -1;
          const size_t bo = (size_t)br * p.B * p.H * p.Tqp;
          lse2 = lse_row[bo];
          dls = dls_row[bo];
        }
        vlo = lo - j0;
        vhi = ((mask >> g2) & 1) ? (br == 1 ? min(hi, j0 + 63) : hi) - j0 : -1;
      } else {
        int hl, qb;
        q_tile(st, hl, qb);
        vlo = i_min - qb * 64;
        vhi = i_max - qb * 64;
        ok = __all_sync(0xffffffffu, mbar_wait(bar(BS_STFULL + s), ph_s, &abort_flag));      // lse2 / dls of the stage
        if (!ok) { fail_id = BS_STFULL + s + 1; break; }
      }
      ok = __all_sync(0xffffffffu, mbar_wait(bar(BS_SFULL + grp), ph, &abort_flag));
      if (!ok) { fail_id = BS_SFULL + grp + 1; break; }
      tc_fence_after();
      const float* vl = vec + s * 128;
      auto sweep = [&](auto masked) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t sv[32], dv[32], pk[16], dk[16];
          tmem_ld32(tS + h * 32, sv);
          tmem_ld32(tdP + h * 32, dv);
          tc_wait_ld();
#pragma unroll
          for (int i4 = 0; i4 < 8; ++i4) {
            float4 l4, d4;
            if constexpr (MODE == 0) {
              l4 = *reinterpret_cast<const float4*>(vl + h * 32 + i4 * 4);
              d4 = *reinterpret_cast<const float4*>(vl + 64 + h * 32 + i4 * 4);
            } else {
              l4 = make_float4(lse2, lse2, lse2, lse2);
              d4 = make_float4(dls, dls, dls, dls);
            }
            const float ls[4] = {l4.x, l4.y, l4.z, l4.w}, ds[4] = {d4.x, d4.y, d4.z, d4.w};
            float pv[4], dd[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int c = h * 32 + i4 * 4 + e;
              float x = ex2(fmaf(__uint_as_float(sv[i4 * 4 + e]), sl2, -ls[e]));
              if constexpr (decltype(masked)::value)
                if (c < vlo || c > vhi) x = 0.f;
              pv[e] = x;
              dd[e] = x * fmaf(__uint_as_float(dv[i4 * 4 + e]), sc, -ds[e]);
            }
            if constexpr (MODE == 0) { pk[i4 * 2] = Elem<T>::pack(pv[0], pv[1]); pk[i4 * 2 + 1] = Elem<T>::pack(pv[2], pv[3]); }
            dk[i4 * 2] = Elem<T>::pack(dd[0], dd[1]);
            dk[i4 * 2 + 1] = Elem<T>::pack(dd[2], dd[3]);
          }
          if constexpr (MODE == 0) { tmem_st16(tS + h * 16, pk); tmem_st16(tdP + h * 16, dk); }
          else tmem_st16(tS + h * 16, dk);
        }
      };
      if (__all_sync(0xffffffffu, vlo <= 0 && vhi >= 63)) sweep(std::false_type{});
      else if (__any_sync(0xffffffffu, vlo <= vhi && vlo < 64 && vhi >= 0)) sweep(std::true_type{});
      else {
        uint32_t z[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) z[i] = 0u;
        tmem_st32(tS, z);
        if constexpr (MODE == 0) tmem_st32(tdP, z);
      }
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(bar(BS_PFULL + grp));
      ph ^= 1;
      s += NBUF;
      if (s >= NST) { s -= NST; ph_s ^= 1; }
    }

    // ---- epilogue: the accumulators are complete once the last MMA has landed ----
    if (ok && n_steps > 0) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar(BS_ACC), 0, &abort_flag));
      if (!ok) fail_id = BS_ACC + 1;
      tc_fence_after();
    }
    if (ok) {
      constexpr int NCH = (MODE == 1 ? D : 2 * D) / 32;    // 32-column pieces of a lane's accumulators, dealt to the three groups
#pragma unroll 1
      for (int c = grp; c < NCH; c += 3) {
        uint32_t v[32];
        if (MODE == 0 || n_steps > 0) {
          tmem_ld32(tmem + lane_addr + C_ACC + c * 32, v);
          tc_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0u;
        }
        if constexpr (MODE == 1) {
          if (row_ok) {
            T* dst = reinterpret_cast<T*>(p.dQ) + (((size_t)b * p.H + hk * p.G + g_head[g2]) * p.Tq + qi) * D + c * 32;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint32_t w[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) w[e] = Elem<T>::pack(__uint_as_float(v[8 * q + 2 * e]), __uint_as_float(v[8 * q + 2 * e + 1]));
              reinterpret_cast<uint4*>(dst)[q] = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        } else {
          const int j = k0 + r, rows = br_k ? p.Tk : p.Nc;
          const bool isk = c >= D / 32;
          const float fac = (FMT == 0 && !isk) ? kGatedPInv : 1.f;
          float* base = br_k ? (isk ? p.dK : p.dV) : (isk ? p.dKc : p.dVc);
          if (j < rows) {
            float* dst = base + ((size_t)owner * rows + j) * D + (c % (D / 32)) * 32;
#pragma unroll
            for (int q = 0; q < 8; ++q)
              red_add4(dst + q * 4, __uint_as_float(v[4 * q]) * fac, __uint_as_float(v[4 * q + 1]) * fac, __uint_as_float(v[4 * q + 2]) * fac,
                       __uint_as_float(v[4 * q + 3]) * fac);
          }
        }
      }
    }
  }

  // ---- teardown (every path reaches it) ----
  if (fail_id != 0) atomicCAS(&g_bst_status, 0, fail_id);
  tc_fence_before();
  __syncthreads();
  if (abort_flag && warp == 0 && lane == 0) {
    // let copies already in flight land (bounded) before the block's shared memory is handed back
    for (int i = 0; i < 20000 && !mbar_try_wait(bar(BS_RES), 0); ++i) __nanosleep(100);
    for (int k = 0; k < NST && last_st - k >= 0; ++k) {
      const int st = last_st - k;
      for (int i = 0; i < 20000 && !mbar_try_wait(bar(BS_STFULL + st % NST), (st / NST) & 1); ++i) __nanosleep(100);
    }
  }
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// ---------------------------------------------------------------- gates
// Gradient of the gated combine, one pass over dO and the three branch outputs: d_i = dO . O_i per row, the gate logits'
// gradients, and what the streaming kernels need of a row -- log2-sum-exp less log2 of the gate, d_i * scale -- in rows
// padded to 64 (zeros past Tq), for the selected branch also in natural units without padding (nsa_bwd_tc5_kernel).
// D/8 lanes per row, 16 bytes each; HBM-bound: four reads of [rows, D] and nothing of that size written.
template <typename T, int D>
__global__ void __launch_bounds__(256) bwd_gates_kernel(const T* __restrict__ dO, const T* __restrict__ O, const float* __restrict__ lse,
                                                        const void* __restrict__ gates, int gate_dtype, int gate_act, void* __restrict__ dgates,
                                                        float* __restrict__ lse2, float* __restrict__ dls, float* __restrict__ sel_lse,
                                                        float* __restrict__ sel_d, long long BH, int Tq, int Tqp, float scale) {
  constexpr int LPR = D / 8;
  constexpr bool F16 = std::is_same<T, __half>::value;
  constexpr float PX = F16 ? kGatedPExp : 0.f, PI = F16 ? kGatedPInv : 1.f;
  grid_dep_wait();
  const int sub = threadIdx.x % LPR;
  const long long rows_p = BH * Tqp, rows = BH * Tq;
  const long long step = (long long)gridDim.x * (256 / LPR);
  for (long long pr0 = (long long)blockIdx.x * (256 / LPR); pr0 < rows_p; pr0 += step) {      // uniform over the block: shuffles stay converged
    const long long pr = pr0 + threadIdx.x / LPR;
    const long long bh = pr / Tqp;
    const int t = (int)(pr % Tqp);
    const bool in = pr < rows_p && t < Tq;
    const long long row = in ? bh * Tq + t : 0;
    const size_t at = (size_t)row * D + sub * 8;
    const uint4 g4 = *reinterpret_cast<const uint4*>(dO + at);
    uint4 o4[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) o4[c] = *reinterpret_cast<const uint4*>(O + (size_t)c * rows * D + at);
    float l[3], x[3] = {0.f, 0.f, 0.f}, d[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) l[c] = lse[(size_t)c * rows + row];
    if (gates != nullptr) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
        x[c] = gate_dtype == NSA_FP32 ? reinterpret_cast<const float*>(gates)[row * 3 + c]
             : gate_dtype == NSA_FP16 ? __half2float(reinterpret_cast<const __half*>(gates)[row * 3 + c])
                                      : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(gates)[row * 3 + c]);
    }
    const uint32_t gw[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const uint32_t ow[4] = {o4[c].x, o4[c].y, o4[c].z, o4[c].w};
      float acc = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 a = Elem<T>::unpack(gw[e]), o = Elem<T>::unpack(ow[e]);
        acc = fmaf(a.x, o.x, acc);
        acc = fmaf(a.y, o.y, acc);
      }
#pragma unroll
      for (int off = LPR / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
      d[c] = acc;
    }
    if (sub != 0 || pr >= rows_p) continue;
    float g[3], lg[3], dx[3];                              // gate, its natural logarithm, gradient of its logit
    if (gate_act == NSA_GATE_SOFTMAX) {
      const float mx = fmaxf(x[0], fmaxf(x[1], x[2]));
      float e[3], sum = 0.f, dot = 0.f;
#pragma unroll
      for (int c = 0; c < 3; ++c) { e[c] = expf(x[c] - mx); sum += e[c]; }
      const float ls = logf(sum);
#pragma unroll
      for (int c = 0; c < 3; ++c) { g[c] = e[c] / sum; lg[c] = x[c] - mx - ls; dot += g[c] * d[c]; }
#pragma unroll
      for (int c = 0; c < 3; ++c) dx[c] = g[c] * (d[c] - dot);
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        g[c] = 1.f / (1.f + expf(-x[c]));
        lg[c] = fminf(x[c], 0.f) - log1pf(expf(-fabsf(x[c])));
        dx[c] = d[c] * g[c] * (1.f - g[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const bool has = in && l[c] > -INFINITY;             // a row without a key in the branch takes no part: its P is masked
      lse2[(size_t)c * rows_p + pr] = has ? (l[c] - lg[c]) * kLog2e - PX : 0.f;
      dls[(size_t)c * rows_p + pr] = has ? d[c] * (scale * PI) : 0.f;
      if (in && dgates != nullptr) {
        if (gate_dtype == NSA_FP32) reinterpret_cast<float*>(dgates)[row * 3 + c] = dx[c];
        else if (gate_dtype == NSA_FP16) reinterpret_cast<__half*>(dgates)[row * 3 + c] = __float2half_rn(dx[c]);
        else reinterpret_cast<__nv_bfloat16*>(dgates)[row * 3 + c] = __float2bfloat16_rn(dx[c]);
      }
    }
    if (in) {
      sel_lse[row] = l[1] > -INFINITY ? l[1] - lg[1] : -INFINITY;
      sel_d[row] = d[1];
    }
  }
}

// ---------------------------------------------------------------- dK, dV in 16 bits
// dX[j] = sum of the raw-key gradients and of (1/block) times those of the windows that cover row j, rounded once.
// 8 columns per thread; K and V in one launch.
template <typename T>
__global__ void __launch_bounds__(256) bwd_keys_kernel(const float* __restrict__ raw, const float* __restrict__ pooled, T* __restrict__ dK,
                                                       T* __restrict__ dV, long long owners, int Tk, int Nc, int D, int block, int stride) {
  grid_dep_wait();
  const int CH = D / 8;
  const long long per = owners * Tk * CH, i0 = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i0 >= 2 * per) return;
  const bool isv = i0 >= per;
  const long long i = isv ? i0 - per : i0;
  const int ch = (int)(i % CH);
  const long long rj = i / CH;
  const int j = (int)(rj % Tk);
  const long long owner = rj / Tk;
  const float4* rp = reinterpret_cast<const float4*>(raw + (isv ? owners * Tk * D : 0) + rj * D) + ch * 2;
  float4 a = rp[0], c = rp[1];
  const int c_hi = min(j / stride, Nc - 1);
  const int c_lo = j - (block - 1) <= 0 ? 0 : (j - (block - 1) + stride - 1) / stride;
  const float4* pp = reinterpret_cast<const float4*>(pooled + (isv ? owners * Nc * D : 0) + owner * Nc * D) + ch * 2;
  float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
  for (int w = c_lo; w <= c_hi; ++w) {
    const float4 v0 = pp[(size_t)w * (D / 4)], v1 = pp[(size_t)w * (D / 4) + 1];
    s0.x += v0.x; s0.y += v0.y; s0.z += v0.z; s0.w += v0.w;
    s1.x += v1.x; s1.y += v1.y; s1.z += v1.z; s1.w += v1.w;
  }
  const float inv = 1.f / (float)block;
  const uint4 o = make_uint4(Elem<T>::pack(fmaf(s0.x, inv, a.x), fmaf(s0.y, inv, a.y)), Elem<T>::pack(fmaf(s0.z, inv, a.z), fmaf(s0.w, inv, a.w)),
                             Elem<T>::pack(fmaf(s1.x, inv, c.x), fmaf(s1.y, inv, c.y)), Elem<T>::pack(fmaf(s1.z, inv, c.z), fmaf(s1.w, inv, c.w)));
  *reinterpret_cast<uint4*>((isv ? dV : dK) + rj * D + ch * 8) = o;
}

// ---------------------------------------------------------------- host side
bool attention_bwd_tc5_supports(const nsa_bwd_args&);
long long attention_bwd_tc5_scratch_bytes(const nsa_bwd_args&);
int attention_bwd_tc5(const nsa_bwd_args&, void*, long long, bool, cudaStream_t);

struct BstPlan {
  int Nc, nq, nk, Tqp, Hi, k_sel;
  size_t o_lse2, o_dls, o_slse, o_sd, o_raw, o_pooled, o_scratch, total;
  size_t acc_bytes;
  long long scratch_bytes;
  nsa_bwd_args sel;
};

static bool bst_plan(const nsa_forward_args& f, BstPlan& pl) {
  if (!(f.q_dtype == NSA_BF16 || f.q_dtype == NSA_FP16) || !(f.D == 64 || f.D == 128) || f.bm != 64 || f.bn != 64) return false;
  if (!(f.B > 0 && f.H > 0 && f.Hkv > 0 && f.H % f.Hkv == 0 && f.Tq > 0 && f.Tk > 0 && f.top_k > 0 && f.scale > 0.f)) return false;
  if (!(f.cmp_block > 0 && f.cmp_stride > 0 && f.cmp_stride <= f.cmp_block && f.window >= 1)) return false;
  pl.Nc = f.cmp_stride == f.cmp_block ? (f.Tk + f.cmp_block - 1) / f.cmp_block
                                      : (f.Tk >= f.cmp_block ? (f.Tk - f.cmp_block) / f.cmp_stride + 1 : 0);
  if (pl.Nc < 1) return false;
  pl.nq = (f.Tq + 63) / 64;
  pl.nk = (f.Tk + 63) / 64;
  pl.Tqp = pl.nq * 64;
  pl.Hi = f.has_idx ? f.Hi : (f.per_group ? f.Hkv : f.H);
  pl.k_sel = f.has_idx ? f.top_k : (f.top_k < pl.nk ? f.top_k : pl.nk);
  if (pl.k_sel > BST_MAX_SEL) return false;
  nsa_bwd_args& s = pl.sel;
  s = {};
  s.B = f.B; s.H = f.H; s.Hkv = f.Hkv; s.Hi = pl.Hi; s.Tq = f.Tq; s.Tk = f.Tk; s.D = f.D;
  s.nq = pl.nq; s.top_k = pl.k_sel; s.bm = 64; s.bn = 64; s.sel_key_limit = pl.nk * 64;
  s.offset = f.Tk - f.Tq; s.causal = f.causal; s.dtype = s.dq_dtype = f.q_dtype; s.scale = f.scale; s.branch = NSA_BRANCH_SELECTED;
  if (!attention_bwd_tc5_supports(s)) return false;
  pl.scratch_bytes = attention_bwd_tc5_scratch_bytes(s);
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  const size_t rows_p = (size_t)f.B * f.H * pl.Tqp, rows = (size_t)f.B * f.H * f.Tq, own = (size_t)f.B * f.Hkv;
  size_t o = 0;
  pl.o_lse2 = o; o = up(o + rows_p * 3 * 4);
  pl.o_dls = o; o = up(o + rows_p * 3 * 4);
  pl.o_slse = o; o = up(o + rows * 4);
  pl.o_sd = o; o = up(o + rows * 4);
  pl.o_raw = o; o = up(o + own * f.Tk * f.D * 8);
  pl.o_pooled = o; o = up(o + own * pl.Nc * f.D * 8);
  pl.acc_bytes = o - pl.o_raw;
  pl.o_scratch = o; o = up(o + (size_t)pl.scratch_bytes);
  pl.total = o;
  return true;
}

long long backward_ws_bytes(const nsa_forward_args& f) {
  BstPlan pl;
  return bst_plan(f, pl) ? (long long)pl.total : 0;
}

template <typename T, int D, int FMT>
static int bst_launch(const nsa_forward_args& f, const BstPlan& pl, BstParams& p, const void* dO, const void* branch_out, const float* branch_lse,
                      void* dK, void* dV, void* dgates, cudaStream_t st) {
  unsigned char* ws = reinterpret_cast<unsigned char*>(f.ws);
  float* raw = reinterpret_cast<float*>(ws + pl.o_raw);
  float* pooled = reinterpret_cast<float*>(ws + pl.o_pooled);
  const size_t own = (size_t)f.B * f.Hkv;
  int dev = 0, sms = 148;
  NSA_CUDA_OK(cudaGetDevice(&dev));
  NSA_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  NSA_CUDA_OK(cudaMemsetAsync(raw, 0, pl.acc_bytes, st));
  const long long BH = (long long)f.B * f.H;
  const long long want = (BH * pl.Tqp + 256 / (D / 8) - 1) / (256 / (D / 8));
  const unsigned ggrid = (unsigned)(want < (long long)sms * 8 ? want : (long long)sms * 8);
  int rc = launch_pdl("bwd_gates", bwd_gates_kernel<T, D>, dim3(ggrid), 256, 0, st, (const T*)dO, (const T*)branch_out, branch_lse, f.gates,
                      f.gate_dtype, f.gate_act, dgates, const_cast<float*>(p.lse2), const_cast<float*>(p.dls),
                      reinterpret_cast<float*>(ws + pl.o_slse), reinterpret_cast<float*>(ws + pl.o_sd), BH, f.Tq, pl.Tqp, f.scale);
  if (rc != NSA_OK) return rc;

  constexpr size_t DHh = D / 64;
  constexpr size_t smem = 2 * DHh * 128 * 128 + (size_t)bst_stages(D) * (2 * DHh * 64 * 128 + 512) + 1024;
  auto fq = nsa_bwd_stream_kernel<D, FMT, 1>;
  auto fk = nsa_bwd_stream_kernel<D, FMT, 0>;
  NSA_CUDA_OK(cudaFuncSetAttribute(fq, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  NSA_CUDA_OK(cudaFuncSetAttribute(fk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const long long NL = (long long)own;
  // query pass: two heads of a block share every tile where they exist and list the same blocks; otherwise two query
  // blocks of one head share the pooled and window tiles at least
  p.two_qb = (p.G == 1 || pl.Hi == f.H) ? 1 : 0;
  p.n_pairs = (p.G + 1) / 2;
  const long long gq = p.two_qb ? (long long)((p.nq + 1) / 2) * NL * p.G : (long long)p.nq * NL * p.n_pairs;
  NSA_REQUIRE(gq < 2147483647LL, NSA_ERR_ARG, "backward: %lld query tiles do not fit a grid", gq);
  fq<<<(unsigned)gq, BST_THREADS, smem, st>>>(p);
  if ((rc = launch_status("backward (query pass)")) != NSA_OK) return rc;

  // key pass: segments of at most L steps, about eight blocks per SM over the launch
  p.kt_cmp = (pl.Nc + 127) / 128;
  p.kt_sld = (f.Tk + 127) / 128;
  const long long most_cmp = (long long)pl.nq * p.G;                     // steps of a pooled key tile that every query sees
  const long long most_sld = (long long)((128 + (f.causal ? 1 : 2) * (long long)p.window) / 64 + 2) * p.G;
  const long long total = NL * (p.kt_cmp * most_cmp / 2 + p.kt_sld * (most_sld < most_cmp ? most_sld : most_cmp));
  long long L = total / ((long long)sms * 8);
  p.L = (int)(L < 32 ? 32 : (L > 256 ? 256 : L));
  p.seg_cmp = (int)((most_cmp + p.L - 1) / p.L);
  p.seg_sld = (int)(((most_sld < most_cmp ? most_sld : most_cmp) + p.L - 1) / p.L);
  const long long gk = NL * ((long long)p.kt_cmp * p.seg_cmp + (long long)p.kt_sld * p.seg_sld);
  NSA_REQUIRE(gk < 2147483647LL, NSA_ERR_ARG, "backward: %lld key segments do not fit a grid", gk);
  fk<<<(unsigned)gk, BST_THREADS, smem, st>>>(p);
  if ((rc = launch_status("backward (key pass)")) != NSA_OK) return rc;

  // dK, dV of the listed blocks: the key-major pass over the inverted lists
  nsa_bwd_args s = pl.sel;
  s.Q = f.Q; s.K = f.K; s.V = f.V; s.dO = dO; s.idx = p.idx; s.dQ = p.dQ; s.dK_f = p.dK; s.dV_f = p.dV;
  s.lse = reinterpret_cast<const float*>(ws + pl.o_slse); s.delta = reinterpret_cast<const float*>(ws + pl.o_sd);
  if ((rc = attention_bwd_tc5(s, ws + pl.o_scratch, pl.scratch_bytes, true, st)) != NSA_OK) return rc;

  const long long nkeys = 2 * NL * f.Tk * (D / 8);
  return launch_pdl("bwd_keys", bwd_keys_kernel<T>, dim3((unsigned)((nkeys + 255) / 256)), 256, 0, st, (const float*)raw, (const float*)pooled,
                    (T*)dK, (T*)dV, NL, f.Tk, pl.Nc, D, f.cmp_block, f.cmp_stride);
}

// Gradients of the forward described by `f` (its workspace pointers mean this call's workspace).
int backward_stream(const nsa_forward_args& f, const void* dO, const void* branch_out, const float* branch_lse, const int32_t* idx,
                    const void* Kc, const void* Vc, void* dQ, void* dK, void* dV, void* dgates, cudaStream_t st) {
  BstPlan pl;
  NSA_REQUIRE(bst_plan(f, pl), NSA_ERR_UNSUPPORTED, "backward: needs D in {64,128}, 16-bit storage, 64-token blocks and at most %d listed blocks", BST_MAX_SEL);
  NSA_REQUIRE(f.ws && f.ws_bytes >= (int64_t)pl.total && (reinterpret_cast<uintptr_t>(f.ws) & 255) == 0, NSA_ERR_ARG,
              "backward: needs %lld bytes of workspace (256-byte aligned), %lld given", (long long)pl.total, (long long)f.ws_bytes);
  unsigned char* ws = reinterpret_cast<unsigned char*>(f.ws);
  const size_t own = (size_t)f.B * f.Hkv;
  BstParams p;
  p.B = f.B; p.H = f.H; p.Hkv = f.Hkv; p.Hi = pl.Hi; p.Tq = f.Tq; p.Tqp = pl.Tqp; p.Tk = f.Tk; p.Nc = pl.Nc; p.nq = pl.nq; p.nk = pl.nk;
  p.top_k = pl.k_sel; p.G = f.H / f.Hkv;
  p.offset = f.Tk - f.Tq;
  p.cmp_offset = (f.cmp_stride == f.cmp_block ? pl.Nc * f.cmp_block : f.Tk) - f.Tq;
  p.cmp_block = f.cmp_block; p.cmp_stride = f.cmp_stride; p.sel_limit = pl.nk * 64; p.causal = f.causal;
  // a window beyond the sequence ("no window", up to INT_MAX) hides no key: cut to it, so that positions plus window stay in range
  const int reach = f.Tq > f.Tk ? f.Tq : f.Tk;
  p.window = f.window < reach ? f.window : reach;
  p.scale = f.scale; p.scale_log2 = f.scale * kLog2e;
  p.lse2 = reinterpret_cast<float*>(ws + pl.o_lse2);
  p.dls = reinterpret_cast<float*>(ws + pl.o_dls);
  p.idx = idx; p.dQ = dQ;
  p.dK = reinterpret_cast<float*>(ws + pl.o_raw); p.dV = p.dK + own * f.Tk * f.D;
  p.dKc = reinterpret_cast<float*>(ws + pl.o_pooled); p.dVc = p.dKc + own * pl.Nc * f.D;
  int rc;
  if ((rc = make_map(&p.tmQ, f.Q, (long long)f.B * f.H, f.Tq, f.D, f.q_dtype)) != NSA_OK) return rc;
  if ((rc = make_map(&p.tmdO, dO, (long long)f.B * f.H, f.Tq, f.D, f.q_dtype)) != NSA_OK) return rc;
  if ((rc = make_map(&p.tmK, f.K, (long long)own, f.Tk, f.D, f.q_dtype)) != NSA_OK) return rc;
  if ((rc = make_map(&p.tmV, f.V, (long long)own, f.Tk, f.D, f.q_dtype)) != NSA_OK) return rc;
  if ((rc = make_map(&p.tmKc, Kc, (long long)own, pl.Nc, f.D, f.q_dtype)) != NSA_OK) return rc;
  if ((rc = make_map(&p.tmVc, Vc, (long long)own, pl.Nc, f.D, f.q_dtype)) != NSA_OK) return rc;
  if (f.q_dtype == NSA_BF16) {
    if (f.D == 64) return bst_launch<__nv_bfloat16, 64, 1>(f, pl, p, dO, branch_out, branch_lse, dK, dV, dgates, st);
    return bst_launch<__nv_bfloat16, 128, 1>(f, pl, p, dO, branch_out, branch_lse, dK, dV, dgates, st);
  }
  if (f.D == 64) return bst_launch<__half, 64, 0>(f, pl, p, dO, branch_out, branch_lse, dK, dV, dgates, st);
  return bst_launch<__half, 128, 0>(f, pl, p, dO, branch_out, branch_lse, dK, dV, dgates, st);
}

// Returns and clears the status word of these kernels (the stream has been synchronised by the caller).
int bst_take_status(int* status) {
  int v = 0, zero = 0;
  NSA_CUDA_OK(cudaMemcpyFromSymbol(&v, g_bst_status, sizeof(int)));
  if (v != 0) NSA_CUDA_OK(cudaMemcpyToSymbol(g_bst_status, &zero, sizeof(int)));
  *status = v;
  return NSA_OK;
}

int bst_set_status(int v) {
  NSA_CUDA_OK(cudaMemcpyToSymbol(g_bst_status, &v, sizeof(int)));
  return NSA_OK;
}

}  // namespace nsa
