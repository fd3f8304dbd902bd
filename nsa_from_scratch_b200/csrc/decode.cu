// One decoding step against a KV cache: a handful of query rows (Tq <= 64 positions of the last query block, G heads per
// KV head, G*Tq <= 64 rows) over a long key range.  The step is latency, not work: 13 MB and 0.2 GFLOP at 65536 cached
// positions, 64 heads over 4, D=128.  One cooperative launch behind the append, two blocks per SM, three phases with a
// grid-wide barrier between them:
//
//   A  tasks of two kinds that need nothing from each other: attention over the pooled keys and the window, a few 64-key
//      chunks per task, and the scores of the selection (one thread per key block).
//   B  attention over the listed blocks; every task first picks the list from the scores (4 warps take the best k of a
//      quarter each, one warp merges), which is cheaper than another barrier.
//   C  the partial (O, m, l) of all tasks per row, the gates, one rounding.
//
// As three launches (chained by programmatic dependent launch) the host was the bound: a launch costs it 3 to 5 us.
// Measured, append and step: B=1, 65536 cached 89 -> 31 us (means, selection, split tcgen05 launch and merge before); B=8,
// 8200 cached 95 -> 36 us.  The kernel takes 23 to 26 us, the host 30.
// A tile has 16 rows, so the products run on mma.sync m16n8k16 (a tcgen05 tile would hold 128 rows for one to four that
// exist); the four warps of a block share a chunk by keys (16 rows), by row tiles (64 rows) or both.
#include "common.cuh"

#include <cooperative_groups.h>

namespace nsa {

constexpr int DC_CHUNK = 64;
constexpr int DC_THREADS = 128;
constexpr int DC_MAX_K = 64;          // listed blocks
constexpr int DC_MAX_NK = 8192;       // key blocks whose scores phase B can hold

struct DecodeParams {
  const void *Q, *K, *V, *Kc, *Vc, *Kb, *gates;
  void* out;
  int gate_dtype, gate_act;
  float* scores;          // [lists][nk_alloc]
  float* part;            // [B*H*Tq][slots][D + 4]: unnormalised O, m (log2 units), l
  const int32_t* dyn_len;
  int B, H, Hkv, G, Tq, len, max_len, nc_alloc, nk_alloc;
  int cmp_block, cmp_stride, top_k, window, ff, fl, per_group;
  int n_cmp, n_sld, n_sel, slots;     // blocks per (batch, KV head) for the pooled keys / window, per list for the listed blocks
  int n_score;                        // scoring blocks per list
  float scale, scale_log2;
};

__device__ __forceinline__ uint32_t dc_key(float v) {      // order-preserving; 0 is below every score
  const uint32_t u = __float_as_uint(v + 0.f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// The k best of s[0..n) (key descending, ties to the lowest index) by one warp.  A lane owns elements lane, lane+32, ... and
// knows its best; a round takes the warp's best (two redux) and its owner looks again.  Up to 32*E elements live in
// registers, where looking again is E selects; more are consumed in shared memory.
template <int E>
__device__ __forceinline__ int dc_warp_topk_regs(const uint32_t* s, int n, int k, int base, uint32_t* out_key, int* out_idx, int lane) {
  uint32_t key[E];
#pragma unroll
  for (int e = 0; e < E; ++e) key[e] = e * 32 + lane < n ? s[e * 32 + lane] : 0u;
  int got = 0;
  for (; got < k; ++got) {
    uint32_t bk = key[0];
    int be = 0;
#pragma unroll
    for (int e = 1; e < E; ++e)
      if (key[e] > bk) { bk = key[e]; be = e; }
    const uint32_t top = __reduce_max_sync(0xffffffffu, bk);
    if (top == 0u) break;
    const int bi = be * 32 + lane;
    const int at = (int)__reduce_min_sync(0xffffffffu, bk == top ? (uint32_t)bi : 0x7fffffffu);
    if (lane == 0) { out_key[got] = top; out_idx[got] = base + at; }
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (e * 32 + lane == at) key[e] = 0u;
  }
  __syncwarp();
  return got;
}

__device__ __forceinline__ int dc_warp_topk(uint32_t* s, int n, int k, int base, uint32_t* out_key, int* out_idx, int lane) {
  if (n <= 64) return dc_warp_topk_regs<2>(s, n, k, base, out_key, out_idx, lane);
  if (n <= 256) return dc_warp_topk_regs<8>(s, n, k, base, out_key, out_idx, lane);
  if (n <= 512) return dc_warp_topk_regs<16>(s, n, k, base, out_key, out_idx, lane);
  uint32_t bk;
  int bi;
  auto best_of = [&]() {
    bk = 0u; bi = 0x7fffffff;
    for (int c = lane; c < n; c += 32)
      if (s[c] > bk) { bk = s[c]; bi = c; }
  };
  best_of();
  int got = 0;
  for (; got < k; ++got) {
    const uint32_t top = __reduce_max_sync(0xffffffffu, bk);
    if (top == 0u) break;
    const int at = (int)__reduce_min_sync(0xffffffffu, bk == top ? (uint32_t)bi : 0x7fffffffu);
    if (lane == 0) { out_key[got] = top; out_idx[got] = base + at; }
    if (bi == at && bk == top) { s[at] = 0u; best_of(); }
    __syncwarp();
  }
  return got;
}

// Attention of one (batch, KV head or head) over the chunks [c0, c1) of one branch; MT row tiles of 16.
// Chunk c covers keys key0(c) .. key0(c)+63; row r sees lo(r) <= key <= hi(r).
template <typename T, int D, int MT, typename Key0, typename Bounds>
__device__ void dc_attend(unsigned char* smem, const DecodeParams& p, const T* Kg, const T* Vg, int key_rows, int b, int h0, int n_rows, int c0,
                          int c1, int slot, Key0 key0, Bounds bounds) {
  constexpr int KW = 16 * MT;                     // keys of a chunk per warp
  constexpr int NT = KW / 8;
  constexpr int KS = D / 16;
  constexpr int CH = D / 8;
  constexpr int TILE = DC_CHUNK * D * 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mt = warp % MT, kg = warp / MT;       // row tile, key group (4 / MT of them)
  const int g8 = lane >> 2, t4 = lane & 3, mi = lane >> 3, r8 = lane & 7;
  const T* Qg = reinterpret_cast<const T*>(p.Q);
  auto stage = [&](int c) {
    const int j0 = key0(c);
    const uint32_t ks = smem_u32(smem + (c & 1) * 2 * TILE), vs = ks + TILE;
    for (int i = threadIdx.x; i < DC_CHUNK * CH; i += DC_THREADS) {
      const int r = i / CH, w = i % CH, j = j0 + r;
      const bool in = j < key_rows;
      const size_t o = (size_t)(in ? j : 0) * D + w * 8;
      cp_async16(ks + tile_off<D>(r, w), Kg + o, in ? 16 : 0);
      cp_async16(vs + tile_off<D>(r, w), Vg + o, in ? 16 : 0);
    }
    cp_async_commit();
  };
  if (c0 < c1) stage(c0);
  // Q fragments straight from global memory: row tile mt, rows g8 and g8+8
  uint32_t qf[KS][4];
  int lo[2], hi[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int r = mt * 16 + g8 + e * 8;
    const bool in = r < n_rows;
    const T* q = Qg + (((size_t)b * p.H + h0 + (in ? r / p.Tq : 0)) * p.Tq + (in ? r % p.Tq : 0)) * D;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      qf[ks][e] = in ? *reinterpret_cast<const uint32_t*>(q + ks * 16 + t4 * 2) : 0u;
      qf[ks][2 + e] = in ? *reinterpret_cast<const uint32_t*>(q + ks * 16 + 8 + t4 * 2) : 0u;
    }
    lo[e] = 0; hi[e] = -1;
    if (in) bounds(r % p.Tq, lo[e], hi[e]);
  }
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  float o[2 * KS][4];
#pragma unroll
  for (int d = 0; d < 2 * KS; ++d) { o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f; }
#pragma unroll 1
  for (int c = c0; c < c1; ++c) {
    if (c + 1 < c1) { stage(c + 1); cp_async_wait<1>(); }
    else cp_async_wait<0>();
    __syncthreads();
    const int j0 = key0(c);
    const uint32_t ks_ = smem_u32(smem + (c & 1) * 2 * TILE), vs_ = ks_ + TILE;
    float s[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) { s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f; }
#pragma unroll
    for (int ks = 0; ks < KS; ++ks)
#pragma unroll
      for (int np = 0; np < NT / 2; ++np) {
        uint32_t b0, b1, b2, b3;
        ldsm_x4(b0, b1, b2, b3, ks_ + tile_off<D>(kg * KW + np * 16 + (mi >> 1) * 8 + r8, ks * 2 + (mi & 1)));
        mma16816<T>(s[2 * np], qf[ks], b0, b1);
        mma16816<T>(s[2 * np + 1], qf[ks], b2, b3);
      }
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = j0 + kg * KW + n * 8 + t4 * 2 + (e & 1), r = e >> 1;
        const float v = (j < lo[r] || j > hi[r]) ? -INFINITY : s[n][e] * p.scale_log2;
        s[n][e] = v;
        mx[r] = fmaxf(mx[r], v);
      }
    float alpha[2], ref[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
      const float mn = fmaxf(m[r], mx[r]);
      ref[r] = mn == -INFINITY ? 0.f : mn;
      alpha[r] = ex2(m[r] - ref[r]);
      m[r] = mn;
      l[r] *= alpha[r];
    }
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float pv = ex2(s[n][e] - ref[e >> 1]);
        s[n][e] = pv;
        l[e >> 1] += pv;
      }
#pragma unroll
    for (int d = 0; d < 2 * KS; ++d) { o[d][0] *= alpha[0]; o[d][1] *= alpha[0]; o[d][2] *= alpha[1]; o[d][3] *= alpha[1]; }
#pragma unroll
    for (int kj = 0; kj < NT / 2; ++kj) {
      uint32_t pa[4];
      pa[0] = Elem<T>::pack(s[2 * kj][0], s[2 * kj][1]);
      pa[1] = Elem<T>::pack(s[2 * kj][2], s[2 * kj][3]);
      pa[2] = Elem<T>::pack(s[2 * kj + 1][0], s[2 * kj + 1][1]);
      pa[3] = Elem<T>::pack(s[2 * kj + 1][2], s[2 * kj + 1][3]);
#pragma unroll
      for (int dp = 0; dp < KS; ++dp) {
        uint32_t b0, b1, b2, b3;
        ldsm_x4_t(b0, b1, b2, b3, vs_ + tile_off<D>(kg * KW + kj * 16 + (mi & 1) * 8 + r8, dp * 2 + (mi >> 1)));
        mma16816<T>(o[2 * dp], pa, b0, b1);
        mma16816<T>(o[2 * dp + 1], pa, b2, b3);
      }
    }
    __syncthreads();                              // the stage is refilled two chunks on
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
    l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
  }
  auto part_row = [&](int r) {
    return p.part + ((((size_t)b * p.H + h0 + r / p.Tq) * p.Tq + r % p.Tq) * p.slots + slot) * (D + 4);
  };
  if constexpr (MT == 4) {                        // a warp holds its rows' whole chunks
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = mt * 16 + g8 + e * 8;
      if (r < n_rows) {
        float* dst = part_row(r);
#pragma unroll
        for (int d = 0; d < 2 * KS; ++d) *reinterpret_cast<float2*>(dst + d * 8 + t4 * 2) = make_float2(o[d][2 * e], o[d][2 * e + 1]);
        if (t4 == 0) { dst[D] = m[e]; dst[D + 1] = l[e]; }
      }
    }
  } else {
    // the key groups of a row tile merge through shared memory
    constexpr int PITCH = D + 4, NKG = 4 / MT;
    float* red = reinterpret_cast<float*>(smem);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float* dst = red + (warp * 16 + g8 + e * 8) * PITCH;
#pragma unroll
      for (int d = 0; d < 2 * KS; ++d) *reinterpret_cast<float2*>(dst + d * 8 + t4 * 2) = make_float2(o[d][2 * e], o[d][2 * e + 1]);
      if (t4 == 0) { dst[D] = m[e]; dst[D + 1] = l[e]; }
    }
    __syncthreads();
    constexpr int C4 = D / 4;
    for (int i = threadIdx.x; i < MT * 16 * C4; i += DC_THREADS) {
      const int r = i / C4, c4 = i % C4;
      if (r >= n_rows) continue;
      const float* src = red + ((r / 16) * 16 + r % 16) * PITCH;      // key group 0 of the row tile; the others MT warps on
      float mm = -INFINITY;
#pragma unroll
      for (int g = 0; g < NKG; ++g) mm = fmaxf(mm, src[g * MT * 16 * PITCH + D]);
      float ll = 0.f;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      if (mm > -INFINITY) {
#pragma unroll
        for (int g = 0; g < NKG; ++g) {
          const float* sg = src + g * MT * 16 * PITCH;
          const float w = ex2(sg[D] - mm);
          const float4 v = *reinterpret_cast<const float4*>(sg + c4 * 4);
          ll = fmaf(sg[D + 1], w, ll);
          acc.x = fmaf(v.x, w, acc.x); acc.y = fmaf(v.y, w, acc.y); acc.z = fmaf(v.z, w, acc.z); acc.w = fmaf(v.w, w, acc.w);
        }
      }
      float* dst = part_row(r);
      *reinterpret_cast<float4*>(dst + c4 * 4) = acc;
      if (c4 == 0) { dst[D] = mm; dst[D + 1] = ll; }
    }
  }
}

// A count on the device is the caller's to keep: one past the allocation reads as a full cache, never outside of it.
__device__ __forceinline__ int dc_len(const DecodeParams& p) { return p.dyn_len != nullptr ? min(*p.dyn_len, p.max_len) : p.len; }

// Tasks of phase A: [B*Hkv][n_cmp + n_sld] attention, then [lists][n_score] scoring.
template <typename T, int D, int MT>
__device__ __forceinline__ void decode_task_a(unsigned char* smem, const DecodeParams& p, int len, int task) {
  const int per = p.n_cmp + p.n_sld, n_att = p.B * p.Hkv * per;
  if (task < n_att) {
    const int unit = task / per, s = task % per;
    const int b = unit / p.Hkv, hk = unit % p.Hkv;
    const int n_rows = p.G * p.Tq, h0 = hk * p.G;
    const int offset = len - p.Tq;
    if (s < p.n_cmp) {
      const int cmp_off = (p.cmp_stride == p.cmp_block ? (len + p.cmp_block - 1) / p.cmp_block * p.cmp_block : len) - p.Tq;
      auto bounds = [&](int t, int& lo, int& hi) {
        const int num = t + cmp_off - (p.cmp_block - 1);
        lo = 0;
        hi = num < 0 ? -1 : num / p.cmp_stride;
      };
      int lo, hi;
      bounds(p.Tq - 1, lo, hi);
      const int chunks = hi < 0 ? 0 : min(hi, p.nc_alloc - 1) / DC_CHUNK + 1;
      const size_t slab = (size_t)unit * p.nc_alloc * D;
      dc_attend<T, D, MT>(smem, p, reinterpret_cast<const T*>(p.Kc) + slab, reinterpret_cast<const T*>(p.Vc) + slab, p.nc_alloc, b, h0, n_rows,
                          (int)((long long)chunks * s / p.n_cmp), (int)((long long)chunks * (s + 1) / p.n_cmp), s,
                          [](int c) { return c * DC_CHUNK; }, bounds);
    } else {
      const int s2 = s - p.n_cmp;
      const int first = max(0, offset - p.window + 1) / DC_CHUNK, last = (len - 1) / DC_CHUNK;
      const int chunks = last - first + 1;
      const size_t slab = (size_t)unit * p.max_len * D;
      dc_attend<T, D, MT>(smem, p, reinterpret_cast<const T*>(p.K) + slab, reinterpret_cast<const T*>(p.V) + slab, len, b, h0, n_rows,
                          (int)((long long)chunks * s2 / p.n_sld), (int)((long long)chunks * (s2 + 1) / p.n_sld), s,
                          [first](int c) { return (first + c) * DC_CHUNK; },
                          [&](int t, int& lo, int& hi) { hi = t + offset; lo = max(0, hi - p.window + 1); });
    }
    return;
  }
  // ---- scores of one list: fp32 sum, in head order, of the heads' query-block means (means rounded to 16 bits as the
  // pooling kernel rounds them), fma chain over D in index order, scale last: select_blocks_kernel's arithmetic ----
  const int si = task - n_att;
  const int list = si / p.n_score, part = si % p.n_score;
  const int Hi = p.per_group ? p.Hkv : p.H, GS = p.per_group ? p.G : 1;
  const int b = list / Hi, hi_ = list % Hi;
  const int hk = p.per_group ? hi_ : hi_ / p.G, h0 = p.per_group ? hi_ * p.G : hi_;
  float* qs = reinterpret_cast<float*>(smem);
  const T* Qg = reinterpret_cast<const T*>(p.Q);
  if (threadIdx.x < D / 2) {
    const int d = threadIdx.x * 2;
    float a0 = 0.f, a1 = 0.f;
    for (int g0 = 0; g0 < GS; g0 += 8) {
      uint32_t w[8];
#pragma unroll
      for (int e = 0; e < 8; ++e)
        w[e] = g0 + e < GS ? *reinterpret_cast<const uint32_t*>(Qg + (((size_t)b * p.H + h0 + g0 + e) * p.Tq) * D + d) : 0u;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if (g0 + e >= GS) break;
        float2 f = Elem<T>::unpack(w[e]);
        f.x += 0.f; f.y += 0.f;
        for (int t = 1; t < p.Tq; ++t) {
          const float2 x = Elem<T>::unpack(*reinterpret_cast<const uint32_t*>(Qg + (((size_t)b * p.H + h0 + g0 + e) * p.Tq + t) * D + d));
          f.x += x.x; f.y += x.y;
        }
        const float2 mean = Elem<T>::unpack(Elem<T>::pack(__fdiv_rn(f.x, 64.f), __fdiv_rn(f.y, 64.f)));
        a0 = g0 + e == 0 ? mean.x : __fadd_rn(a0, mean.x);
        a1 = g0 + e == 0 ? mean.y : __fadd_rn(a1, mean.y);
      }
    }
    qs[d] = a0;
    qs[d + 1] = a1;
  }
  __syncthreads();
  const int nk = (len + 63) / 64;
  for (int c = part * DC_THREADS + threadIdx.x; c < nk; c += p.n_score * DC_THREADS) {
    const uint4* kr = reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.Kb) + (((size_t)b * p.Hkv + hk) * p.nk_alloc + c) * D);
    float acc = 0.f;
#pragma unroll
    for (int w8 = 0; w8 < D / 64; ++w8) {
      uint4 raw[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) raw[e] = kr[w8 * 8 + e];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const uint32_t w[4] = {raw[e].x, raw[e].y, raw[e].z, raw[e].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 f = Elem<T>::unpack(w[k]);
          const int d = w8 * 64 + e * 8 + k * 2;
          acc = __fmaf_rn(qs[d], f.x, acc);
          acc = __fmaf_rn(qs[d + 1], f.y, acc);
        }
      }
    }
    float v = acc * p.scale;
    if (c < p.ff || c > nk - 1 - p.fl) v = INFINITY;
    p.scores[(size_t)list * p.nk_alloc + c] = v;
  }
}

// Tasks of phase B: [lists][n_sel].
template <typename T, int D, int MT>
__device__ __forceinline__ void decode_task_b(unsigned char* smem, const DecodeParams& p, int len, int task) {
  __shared__ uint32_t cand_key[4 * DC_MAX_K], best_key[DC_MAX_K];
  __shared__ int cand_idx[4 * DC_MAX_K], best_idx[DC_MAX_K];
  __shared__ int n_cand[4], n_best;
  const int nk = (len + 63) / 64;
  const int list = task / p.n_sel, s = task % p.n_sel;
  const int Hi = p.per_group ? p.Hkv : p.H;
  const int b = list / Hi, hi_ = list % Hi;
  const int hk = p.per_group ? hi_ : hi_ / p.G, h0 = p.per_group ? hi_ * p.G : hi_;
  const int n_rows = (p.per_group ? p.G : 1) * p.Tq;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // each warp takes the best of its quarter of the key blocks, warp 0 the best of the four quarters' bests
  uint32_t* keys = reinterpret_cast<uint32_t*>(smem);
  for (int c = threadIdx.x; c < nk; c += DC_THREADS) keys[c] = dc_key(__ldcg(p.scores + (size_t)list * p.nk_alloc + c));
  __syncthreads();
  const int q0 = (int)((long long)nk * warp / 4), q1 = (int)((long long)nk * (warp + 1) / 4);
  const int got = dc_warp_topk(keys + q0, q1 - q0, p.top_k, q0, cand_key + warp * DC_MAX_K, cand_idx + warp * DC_MAX_K, lane);
  if (lane == 0) n_cand[warp] = got;
  __syncthreads();
  if (warp == 0) {
    // the quarters are in index order, so a candidate's place in the concatenation orders ties as its index does
    uint32_t* ck = keys;
    int* ci = reinterpret_cast<int*>(keys + 4 * DC_MAX_K);
    int n = 0;
    for (int w = 0; w < 4; ++w) {
      for (int i = lane; i < n_cand[w]; i += 32) { ck[n + i] = cand_key[w * DC_MAX_K + i]; ci[n + i] = cand_idx[w * DC_MAX_K + i]; }
      n += n_cand[w];
    }
    __syncwarp();
    const int k = dc_warp_topk(ck, n, p.top_k, 0, best_key, best_idx, lane);
    for (int i = lane; i < k; i += 32) best_idx[i] = ci[best_idx[i]];
    if (lane == 0) n_best = k;
  }
  __syncthreads();
  const size_t slab = ((size_t)b * p.Hkv + hk) * p.max_len * D;
  const int offset = len - p.Tq;
  dc_attend<T, D, MT>(smem, p, reinterpret_cast<const T*>(p.K) + slab, reinterpret_cast<const T*>(p.V) + slab, len, b, h0, n_rows,
                      (int)((long long)n_best * s / p.n_sel), (int)((long long)n_best * (s + 1) / p.n_sel), p.n_cmp + p.n_sld + s,
                      [&](int c) { return best_idx[c] * DC_CHUNK; },
                      [&](int t, int& lo, int& hi) { lo = 0; hi = t + offset; });
}

// out[row] = sum over branches of gate * (sum over slots of 2^(m - M) O) / (sum of 2^(m - M) l).  A block takes a row: three
// warps turn the slots' (m, l) into coefficients, then the block's warps share the slots.
constexpr int DC_MAX_SLOTS = 320;
template <typename T, int D>
__device__ __forceinline__ void decode_merge_row(const DecodeParams& p, long long row) {
  constexpr int LPS = D / 4;                               // lanes that share a slot's row
  constexpr int SPW = DC_THREADS / LPS;                           // slots in flight
  __shared__ float coef[DC_MAX_SLOTS];
  __shared__ float4 red[SPW][LPS];
  const void* gates = p.gates;
  const int gate_dtype = p.gate_dtype, gate_act = p.gate_act, slots = p.slots, n_cmp = p.n_cmp, n_sld = p.n_sld;
  T* out = reinterpret_cast<T*>(p.out);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* pr = p.part + (size_t)row * slots * (D + 4);
  if (warp < 3) {
    const int br = warp;                                   // order of the slots: pooled keys, window, listed blocks
    const int s0 = br == 0 ? 0 : (br == 2 ? n_cmp : n_cmp + n_sld), s1 = br == 0 ? n_cmp : (br == 2 ? n_cmp + n_sld : slots);
    float x[3] = {0.f, 0.f, 0.f}, gate;
    if (gates != nullptr) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
        x[c] = gate_dtype == NSA_FP32 ? reinterpret_cast<const float*>(gates)[row * 3 + c]
             : gate_dtype == NSA_FP16 ? __half2float(reinterpret_cast<const __half*>(gates)[row * 3 + c])
                                      : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(gates)[row * 3 + c]);
    }
    if (gate_act == NSA_GATE_SOFTMAX) {
      const float mx = fmaxf(x[0], fmaxf(x[1], x[2]));
      const float e0 = __expf(x[0] - mx), e1 = __expf(x[1] - mx), e2 = __expf(x[2] - mx);
      gate = (br == 0 ? e0 : br == 1 ? e1 : e2) / (e0 + e1 + e2);
    } else {
      gate = 1.f / (1.f + __expf(-(br == 0 ? x[0] : br == 1 ? x[1] : x[2])));
    }
    float mm = -INFINITY;
    for (int s = s0 + lane; s < s1; s += 32) mm = fmaxf(mm, __ldcg(pr + (size_t)s * (D + 4) + D));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, off));
    float ll = 0.f;
    for (int s = s0 + lane; s < s1; s += 32) {
      const float2 ml = __ldcg(reinterpret_cast<const float2*>(pr + (size_t)s * (D + 4) + D));
      const float w = ml.x == -INFINITY ? 0.f : ex2(ml.x - mm);
      coef[s] = w;
      ll = fmaf(ml.y, w, ll);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ll += __shfl_xor_sync(0xffffffffu, ll, off);
    const float f = ll > 0.f ? gate / ll : 0.f;
    for (int s = s0 + lane; s < s1; s += 32) coef[s] *= f;
  }
  __syncthreads();
  const int sub = threadIdx.x / LPS, c4 = threadIdx.x % LPS;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int s = sub; s < slots; s += SPW) {
    const float4 v = __ldcg(reinterpret_cast<const float4*>(pr + (size_t)s * (D + 4) + c4 * 4));
    const float w = coef[s];
    acc.x = fmaf(v.x, w, acc.x); acc.y = fmaf(v.y, w, acc.y); acc.z = fmaf(v.z, w, acc.z); acc.w = fmaf(v.w, w, acc.w);
  }
  red[sub][c4] = acc;
  __syncthreads();
  if (threadIdx.x < LPS) {
    float4 o = red[0][threadIdx.x];
#pragma unroll
    for (int k = 1; k < SPW; ++k) {
      const float4 v = red[k][threadIdx.x];
      o.x += v.x; o.y += v.y; o.z += v.z; o.w += v.w;
    }
    *reinterpret_cast<uint2*>(out + (size_t)row * D + threadIdx.x * 4) = make_uint2(Elem<T>::pack(o.x, o.y), Elem<T>::pack(o.z, o.w));
  }
}

template <typename T, int D, int MTA, int MTB>
__global__ void __launch_bounds__(DC_THREADS, 2) decode_step_kernel(const __grid_constant__ DecodeParams p) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int len = dc_len(p);
  const int lists = p.B * (p.per_group ? p.Hkv : p.H);
  const int na = p.B * p.Hkv * (p.n_cmp + p.n_sld) + lists * p.n_score, nb = lists * p.n_sel;
  for (int t = blockIdx.x; t < na; t += gridDim.x) {
    decode_task_a<T, D, MTA>(smem, p, len, t);
    __syncthreads();
  }
  cooperative_groups::this_grid().sync();
  for (int t = blockIdx.x; t < nb; t += gridDim.x) {
    decode_task_b<T, D, MTB>(smem, p, len, t);
    __syncthreads();
  }
  cooperative_groups::this_grid().sync();
  const long long rows = (long long)p.B * p.H * p.Tq;
  for (long long r = blockIdx.x; r < rows; r += gridDim.x) {
    decode_merge_row<T, D>(p, r);
    __syncthreads();
  }
}

// ---------------------------------------------------------------- host side
struct DecodePlan {
  DecodeParams p;
  int grid;
  size_t o_part, total;
};

// Returns false for steps this path does not take: more than 64 rows per KV head, other block sizes or head dims.
static bool decode_plan(const nsa_decode_args& a, DecodePlan& pl) {
  if (!(a.dtype == NSA_BF16 || a.dtype == NSA_FP16) || !(a.D == 64 || a.D == 128) || a.bm != 64 || a.bn != 64) return false;
  if (!(a.B > 0 && a.H > 0 && a.Hkv > 0 && a.H % a.Hkv == 0 && a.Tq > 0 && a.Tq <= 64 && a.max_len >= a.Tq && a.top_k > 0 && a.top_k <= DC_MAX_K)) return false;
  if (!(a.cmp_block > 0 && a.cmp_stride > 0 && a.cmp_stride <= a.cmp_block && a.window > 0 && a.scale > 0.f)) return false;
  if (a.nc_alloc < 1 || a.nk_alloc < 1 || a.nk_alloc > DC_MAX_NK) return false;
  if (a.force_first < 0 || a.force_local < 0) return false;        // the general path refuses them
  DecodeParams& p = pl.p;
  p = {};
  p.G = a.H / a.Hkv;
  if (p.G * a.Tq > 64) return false;
  p.B = a.B; p.H = a.H; p.Hkv = a.Hkv; p.Tq = a.Tq; p.max_len = a.max_len; p.nc_alloc = a.nc_alloc; p.nk_alloc = a.nk_alloc;
  p.cmp_block = a.cmp_block; p.cmp_stride = a.cmp_stride; p.top_k = a.top_k; p.window = a.window;
  p.ff = a.force_first; p.fl = a.force_local; p.per_group = a.per_group;
  p.scale = a.scale; p.scale_log2 = a.scale * kLog2e;
  // a length that lives on the device: the grid is sized for a full cache
  p.len = a.dyn_len ? a.max_len : a.len;
  if (p.len < a.Tq || p.len > a.max_len) return false;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int units = a.B * a.Hkv, lists = a.B * (a.per_group ? a.Hkv : a.H);
  auto cdiv = [](int x, int y) { return (x + y - 1) / y; };
  pl.grid = 2 * sms;
  // as few chunks per task as let phase A be one task per block, so that it is one or two loads deep
  const int nk = cdiv(p.len, 64);
  p.n_score = cdiv(nk, DC_THREADS);
  const int ch_cmp = cdiv(cdiv(p.len, a.cmp_stride), DC_CHUNK), ch_sld = (a.window < p.len ? a.window : p.len) / DC_CHUNK + 2;
  int want = (pl.grid - lists * p.n_score) / units;
  if (want < 2) want = 2;
  int cpb = cdiv(ch_cmp + ch_sld, want);
  while (cdiv(ch_cmp, cpb) + cdiv(ch_sld, cpb) > want && cpb < ch_cmp + ch_sld) ++cpb;
  if (cdiv(ch_cmp, cpb) > 192) cpb = cdiv(ch_cmp, 192);            // slots per row are bounded
  p.n_cmp = cdiv(ch_cmp, cpb);
  p.n_sld = cdiv(ch_sld, cpb);
  if (p.n_sld > 64) p.n_sld = 64;
  const int k = a.top_k < a.nk_alloc ? a.top_k : a.nk_alloc;
  const int want_l = pl.grid / lists < 1 ? 1 : pl.grid / lists;
  p.n_sel = cdiv(k, cdiv(k, want_l));
  p.slots = p.n_cmp + p.n_sld + p.n_sel;
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  pl.o_part = up((size_t)lists * a.nk_alloc * 4);
  pl.total = up(pl.o_part + (size_t)a.B * a.H * a.Tq * p.slots * (a.D + 4) * 4);
  return true;
}

template <typename T, int D, int MTA, int MTB>
static int decode_launch(const DecodePlan& pl, cudaStream_t st) {
  const DecodeParams& p = pl.p;
  constexpr int STAGES = 4 * DC_CHUNK * D * 2;                     // two stages of K and V
  constexpr int RED = 4 * 16 * (D + 4) * 4;
  int smem = STAGES > RED ? STAGES : RED;
  if (smem < p.nk_alloc * 4) smem = p.nk_alloc * 4;                // <= 32 KB: two blocks always fit an SM
  auto fn = decode_step_kernel<T, D, MTA, MTB>;
  NSA_CUDA_OK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)pl.grid);
  cfg.blockDim = dim3(DC_THREADS);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  NSA_CUDA_OK(cudaLaunchKernelEx(&cfg, fn, p));
  return NSA_OK;
}

template <typename T, int D>
static int decode_rows(const DecodePlan& pl, cudaStream_t st) {
  const int ra = pl.p.G * pl.p.Tq, rb = pl.p.per_group ? ra : pl.p.Tq;        // rows of a tile in phase A, in phase B
  const int ma = ra <= 16 ? 1 : (ra <= 32 ? 2 : 4), mb = rb <= 16 ? 1 : (rb <= 32 ? 2 : 4);
  if (ma == 1) return decode_launch<T, D, 1, 1>(pl, st);
  if (ma == 2) return mb == 1 ? decode_launch<T, D, 2, 1>(pl, st) : decode_launch<T, D, 2, 2>(pl, st);
  if (mb == 1) return decode_launch<T, D, 4, 1>(pl, st);
  return mb == 2 ? decode_launch<T, D, 4, 2>(pl, st) : decode_launch<T, D, 4, 4>(pl, st);
}

}  // namespace nsa

using namespace nsa;

extern "C" {

// Key blocks of the filled length (of a full cache where the length lives on the device) against the block means' allocation:
// scores, candidates and means are indexed by key block.
static bool decode_blocks_fit(const nsa_decode_args& a) { return ((long long)(a.dyn_len ? a.max_len : a.len) + 63) / 64 <= a.nk_alloc; }

int64_t nsa_decode_ws_bytes(const nsa_decode_args* a) {
  NSA_REQUIRE(a, NSA_ERR_ARG, "decode: NULL argument block");
  DecodePlan pl;
  if (!decode_plan(*a, pl)) return 0;
  NSA_REQUIRE(decode_blocks_fit(*a), NSA_ERR_ARG, "decode: %d block means do not cover the cache", a->nk_alloc);
  return (int64_t)pl.total;
}

int nsa_decode(const nsa_decode_args* a, nsa_stream_t stream) {
  NSA_REQUIRE(a, NSA_ERR_ARG, "decode: NULL argument block");
  NSA_REQUIRE(a->Q && a->K && a->V && a->Kc && a->Vc && a->Kb && a->out && a->ws, NSA_ERR_ARG, "decode: NULL pointer");
  NSA_REQUIRE(!a->gates || a->gate_dtype == NSA_FP32 || a->gate_dtype == NSA_BF16 || a->gate_dtype == NSA_FP16, NSA_ERR_UNSUPPORTED,
              "decode: gate dtype %d", a->gate_dtype);
  DecodePlan pl;
  NSA_REQUIRE(decode_plan(*a, pl), NSA_ERR_UNSUPPORTED, "decode: needs D in {64,128}, 64-token blocks, at most 64 listed blocks and 64 query rows per KV head");
  NSA_REQUIRE(decode_blocks_fit(*a), NSA_ERR_ARG, "decode: %d block means do not cover the cache", a->nk_alloc);
  NSA_REQUIRE(a->ws_bytes >= (int64_t)pl.total && (reinterpret_cast<uintptr_t>(a->ws) & 255) == 0, NSA_ERR_ARG,
              "decode: needs %lld bytes of workspace (256-byte aligned), %lld given", (long long)pl.total, (long long)a->ws_bytes);
  DecodeParams& p = pl.p;
  p.Q = a->Q; p.K = a->K; p.V = a->V; p.Kc = a->Kc; p.Vc = a->Vc; p.Kb = a->Kb; p.dyn_len = a->dyn_len;
  p.gates = a->gates; p.gate_dtype = a->gate_dtype; p.gate_act = a->gate_act; p.out = a->out;
  p.scores = reinterpret_cast<float*>(a->ws);
  p.part = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(a->ws) + pl.o_part);
  cudaStream_t st = (cudaStream_t)stream;
  if (a->dtype == NSA_BF16) return a->D == 64 ? decode_rows<__nv_bfloat16, 64>(pl, st) : decode_rows<__nv_bfloat16, 128>(pl, st);
  return a->D == 64 ? decode_rows<__half, 64>(pl, st) : decode_rows<__half, 128>(pl, st);
}

}  // extern "C"
