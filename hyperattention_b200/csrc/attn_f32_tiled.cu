// fp32 attention on the CUDA cores, forward and backward, head dims 64 and 128: the float32 configuration of every pattern (sorted
// windows, smooth windows in both gradient enumerations, sampled rows with or without weights, exact attention).
//
// Products of 64 x 64 tiles in shared memory, micro-tiles in registers.  A tile is stored as its rows are (cp.async, no transposition)
// with a pitch of D + 4 floats; a thread's micro-tile rows are interleaved (tm + 8 i, tn + 16 j), so that the 16-byte reads of
// a warp fall into distinct banks: per 4 steps of the contraction a thread of the forward reads 8 + 4 vectors for 128 FMAs, 16
// shared-memory cycles against 32 of the FMA pipe.  64-key tiles also make every window boundary a tile boundary (windows
// start at multiples of 64).
// Every product is summed in short chains (32 columns, or a tile of 64 keys or queries, by themselves, then added as a whole), which keeps the
// errors below those of one warp per query / key with lane-wise dot products (32-bit sums over all keys in one chain were 15 to
// 35% above: o 5.2e-7 instead of 4.5e-7 at 4 heads x 4096 x 64, now 2.4e-7).  The extra additions cost 3% of a training step, 7% of a causal one.
// 4 heads x 4096 x 64, block 256, sample 256: step 326 us (one warp per query / key: 7780 us), about a third of the FMA pipe's rate: 256
// CTAs of four warps on 148 SMs leave each scheduler one or two warps to hide shared memory behind, and a half-empty last wave.
#include "attn_index.cuh"

#include <type_traits>

namespace ha {

namespace f32 {
constexpr int BT = 64;               // tile edge
constexpr int LDP = BT + 4;          // pitch of the score tiles

__device__ __forceinline__ float4 lds4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void red4(float* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ float at(const float4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// 64 rows of W floats by row index into a tile of pitch W + 4; rows < 0 are zero-filled.  Called by all THREADS threads.
template <int W, int THREADS>
__device__ __forceinline__ void load_tile(float* tile, const float* __restrict__ base, int64_t sn, const int* rows) {
  constexpr int CPR = W / 4, RPP = THREADS / CPR;      // chunks per row, rows per pass
  const int c = threadIdx.x % CPR, r0 = threadIdx.x / CPR;
#pragma unroll
  for (int i = 0; i < BT / RPP; ++i) {
    const int r = r0 + i * RPP, row = rows[r];
    cp_async16(smem_u32(tile + r * (W + 4) + c * 4), base + (int64_t)(row < 0 ? 0 : row) * sn + c * 4, row < 0 ? 0u : 16u);
  }
}
}  // namespace f32

// ---------------------------------------------------------------------------------------------------
// forward: one CTA of 128 threads per 64 queries
// ---------------------------------------------------------------------------------------------------
template <int D, int DV>
__global__ void __launch_bounds__(128) attn_f32_fwd_kernel(const ha_attn_params p, int n_qt) {
  using namespace f32;
  extern __shared__ __align__(16) float sm[];
  float* sQ = sm;
  float* sK = sQ + BT * (D + 4);
  float* sV = sK + BT * (D + 4);
  float* sP = sV + BT * (DV + 4);
  __shared__ int s_qrow[BT], s_krow[2][BT];
  __shared__ int s_bail;
  if (cta_sees_failure(p.status, &s_bail)) return;   // a failed index check or an earlier timeout: touch nothing
  const int tid = threadIdx.x, tm = tid >> 4, tn = tid & 15;
  const bool hyper = p.mode == HA_MODE_HYPER, causal = p.flags & HA_FLAG_CAUSAL;
  const int seg = blockIdx.x / n_qt;
  int qt = blockIdx.x - seg * n_qt;
  if (causal) qt = n_qt - 1 - qt;                    // long ones first
  const SegInfo si = seg_info(p, seg);
  const long long kseg = kseg_of(p, seg);
  const bool weighted = hyper && p.sample_logw != nullptr;
  const int q128 = qt / 2;                           // the 128-row query tile that windows and weights are defined on
  Window w{0, 0};
  int n_blk = 0, n_keys;
  if (hyper) {
    w = block_window(q128, (p.block_size + TILE - 1) / TILE, p.m_k, p.flags & HA_FLAG_SMOOTH);
    n_blk = w.count;
    n_keys = n_blk + p.sample_size;
  } else {
    n_keys = causal ? min((qt + 1) * BT, p.m_k) : p.m_k;
  }
  const int n_tiles = (n_keys + BT - 1) / BT;
  auto key_row = [&](int j, int r) -> int {
    const int at = j * BT + r;
    if (at >= n_keys) return -1;
    if (!hyper) return at;
    if (at < n_blk) {
      int pos = w.first + at;
      if (pos >= p.m_k) pos -= p.m_k;
      return p.k_idx[kseg * p.m_k + pos];
    }
    return p.sample_idx ? p.sample_idx[kseg * p.sample_size + at - n_blk] : at - n_blk;
  };
  if (tid < BT) {
    const int pos = qt * BT + tid;
    s_qrow[tid] = pos >= p.m_q ? -1 : hyper ? p.q_idx[(long long)seg * p.m_q + pos] : pos;
    s_krow[0][tid] = key_row(0, tid);
    s_krow[1][tid] = key_row(1, tid);
  }
  __syncthreads();
  const float* qb = (const float*)p.q + si.b * p.q_sb + si.h * p.q_sh + si.q_row0 * p.q_sn;
  const float* kb = (const float*)p.k + si.b * p.k_sb + si.hk * p.k_sh + si.k_row0 * p.k_sn;
  const float* vb = (const float*)p.v + si.b * p.v_sb + si.hk * p.v_sh + si.k_row0 * p.v_sn;
  load_tile<D, 128>(sQ, qb, p.q_sn, s_qrow);
  load_tile<D, 128>(sK, kb, p.k_sn, s_krow[0]);
  cp_async_commit();
  load_tile<DV, 128>(sV, vb, p.v_sn, s_krow[0]);
  cp_async_commit();

  constexpr int NC = DV / 64;
  float4 o[8][NC];
  float m[8], l[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) o[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll 1
  for (int j = 0; j < n_tiles; ++j) {
    cp_async_wait<1>();
    __syncthreads();
    float s[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) s[i][c] = 0.f;
    // 32 columns are summed by themselves and added as a whole: a chain of 32 + D / 32 roundings instead of D
#pragma unroll 1
    for (int k0 = 0; k0 < D; k0 += 32) {
      float t[8][4];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) t[i][c] = 0.f;
#pragma unroll 2
      for (int k = k0; k < k0 + 32; k += 4) {
        float4 b[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) b[c] = lds4(sK + (tn + 16 * c) * (D + 4) + k);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 a = lds4(sQ + (tm + 8 * i) * (D + 4) + k);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            t[i][c] = fmaf(a.x, b[c].x, t[i][c]);
            t[i][c] = fmaf(a.y, b[c].y, t[i][c]);
            t[i][c] = fmaf(a.z, b[c].z, t[i][c]);
            t[i][c] = fmaf(a.w, b[c].w, t[i][c]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) s[i][c] += t[i][c];
    }
    __syncthreads();                       // K is read: its place takes the next tile
    if (j + 1 < n_tiles) load_tile<D, 128>(sK, kb, p.k_sn, s_krow[(j + 1) & 1]);
    cp_async_commit();
    // ---- softmax: a row is spread over 16 lanes ----
    uint32_t drop = 0;                     // bit c: column tn + 16 c of the tile is a dropped sample
    float bias = 0.f;
    if (weighted && j * BT >= n_blk) {
      const long long qtile = (long long)seg * (p.m_q / TILE) + q128;
      bias = p.sample_logw[qtile];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int slot = j * BT - n_blk + tn + 16 * c;
        drop |= ((p.sample_mask[qtile * (p.sample_size / 32) + (slot >> 5)] >> (slot & 31)) & 1u) << c;
      }
    }
    const bool edge = (j + 1) * BT > n_keys || (causal && j == qt) || weighted;
    float alphas[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float mx = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        s[i][c] = s[i][c] * p.scale + bias;
        if (edge) {
          const int key = j * BT + tn + 16 * c;
          if (key >= n_keys || (causal && key > qt * BT + tm + 8 * i) || ((drop >> c) & 1u)) s[i][c] = -INFINITY;
        }
        mx = fmaxf(mx, s[i][c]);
      }
#pragma unroll
      for (int off = 8; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      const float mnew = fmaxf(m[i], mx), use = mnew == -INFINITY ? 0.f : mnew;
      const float alpha = expf(m[i] - use);          // -inf -> 0
      float sum = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        s[i][c] = expf(s[i][c] - use);
        sum += s[i][c];
        sP[(tm + 8 * i) * LDP + tn + 16 * c] = s[i][c];
      }
#pragma unroll
      for (int off = 8; off >= 1; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
      l[i] = l[i] * alpha + sum;
      m[i] = mnew;
      alphas[i] = alpha;
    }
    cp_async_wait<1>();
    __syncthreads();
    // a tile's product is summed by itself and added as a whole: the chain of roundings is 64 + tiles long instead of a row's keys
    float4 t[8][NC];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < NC; ++c) t[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
    for (int k = 0; k < BT; k += 4) {
      float4 a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = lds4(sP + (tm + 8 * i) * LDP + k);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const float4 b = lds4(sV + (k + kk) * (DV + 4) + tn * 4 + 64 * c);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float x = at(a[i], kk);
            t[i][c].x = fmaf(x, b.x, t[i][c].x);
            t[i][c].y = fmaf(x, b.y, t[i][c].y);
            t[i][c].z = fmaf(x, b.z, t[i][c].z);
            t[i][c].w = fmaf(x, b.w, t[i][c].w);
          }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        o[i][c].x = fmaf(o[i][c].x, alphas[i], t[i][c].x);
        o[i][c].y = fmaf(o[i][c].y, alphas[i], t[i][c].y);
        o[i][c].z = fmaf(o[i][c].z, alphas[i], t[i][c].z);
        o[i][c].w = fmaf(o[i][c].w, alphas[i], t[i][c].w);
      }
    __syncthreads();
    if (j + 1 < n_tiles) load_tile<DV, 128>(sV, vb, p.v_sn, s_krow[(j + 1) & 1]);
    cp_async_commit();
    if (tid < BT && j + 2 < n_tiles) s_krow[j & 1][tid] = key_row(j + 2, tid);
  }
  cp_async_wait<0>();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int qrow = s_qrow[tm + 8 * i];
    if (qrow < 0) continue;
    const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
    const float own = l[i] > 0.f ? m[i] + logf(l[i]) : -INFINITY;
    const long long orow = si.q_row0 + qrow, lse_at = ((long long)(si.b * p.H + si.h)) * p.n + orow;
    float lse = own, w1 = 0.f, w2 = 1.f;
    if (p.flags & HA_FLAG_MERGE) {
      const float l1 = p.lse[lse_at];
      if (p.flags & HA_FLAG_MERGE_EXACT) {
        const float mm = fmaxf(l1, own);
        const float e1 = expf(l1 - mm), e2 = expf(own - mm);
        w1 = e1 / (e1 + e2);
        w2 = e2 / (e1 + e2);
        lse = mm + logf(e1 + e2);
      } else {
        w1 = 1.f / (1.f + expf(own - l1));
        w2 = 1.f - w1;
        lse = l1 - logf(w1 + 1.1920929e-07f);
      }
    }
    const int64_t o_at = si.b * p.o_sb + si.h * p.o_sh + orow * p.o_sn;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      float4 v = make_float4(o[i][c].x * inv, o[i][c].y * inv, o[i][c].z * inv, o[i][c].w * inv);
      if (p.part_o) *reinterpret_cast<float4*>((float*)p.part_o + o_at + tn * 4 + 64 * c) = v;
      float4* out = reinterpret_cast<float4*>((float*)p.o + o_at + tn * 4 + 64 * c);
      if (p.flags & HA_FLAG_MERGE) {
        const float4 old = *out;
        v = make_float4(w1 * old.x + w2 * v.x, w1 * old.y + w2 * v.y, w1 * old.z + w2 * v.z, w1 * old.w + w2 * v.w);
      }
      *out = v;
    }
    __syncwarp(0xffffu << (tid & 16));     // (merge) every lane of the row has read the old lse
    if (tn == 0) {
      if (p.part_o && p.part_lse) p.part_lse[lse_at] = own;
      p.lse[lse_at] = lse;
    }
  }
}

// ---------------------------------------------------------------------------------------------------
// backward: one CTA of 256 threads per item = 64 keys x a chunk of the query tiles (64 rows each) that meet them.  dK and dV stay in
// registers over the chunk; dQ rows, and dK / dV at the end, are added to the fp32 accumulators.
// ---------------------------------------------------------------------------------------------------
struct F32BwdPlan {
  int blk_tiles, blk_chunks;       // key tiles per segment (sorted, or all keys of exact attention); chunks of query tiles of each
  int smp_tiles, smp_chunks;       // sampled key tiles per segment; chunks
  int chunk;                       // query tiles per chunk
  int per_seg;                     // items per segment
};

template <int D, int DV>
__global__ void __launch_bounds__(256, D + DV <= 128 ? 2 : 1) attn_f32_bwd_kernel(const ha_attn_params p, const F32BwdPlan pl) {
  using namespace f32;
  extern __shared__ __align__(16) float sm[];
  float* sK = sm;
  float* sV = sK + BT * (D + 4);
  float* sQ = sV + BT * (DV + 4);
  float* sG = sQ + BT * (D + 4);
  float* sP = sG + BT * (DV + 4);
  float* sS = sP + BT * LDP;
  __shared__ int s_krow[BT], s_qrow[BT];
  __shared__ float s_lse[BT], s_delta[BT];
  __shared__ int s_bail;
  if (cta_sees_failure(p.status, &s_bail)) return;   // a failed index check or an earlier timeout: touch nothing
  const int tid = threadIdx.x, tm = tid >> 4, tn = tid & 15;
  const bool hyper = p.mode == HA_MODE_HYPER, causal = p.flags & HA_FLAG_CAUSAL;
  const int bs = (p.block_size + TILE - 1) / TILE;
  const int seg = blockIdx.x / pl.per_seg;
  int item = blockIdx.x - seg * pl.per_seg;
  const SegInfo si = seg_info(p, seg);
  const long long kseg = kseg_of(p, seg);
  const bool sampled = item >= pl.blk_tiles * pl.blk_chunks;
  if (sampled) item -= pl.blk_tiles * pl.blk_chunks;
  const int chunks = sampled ? pl.smp_chunks : pl.blk_chunks;
  const int kt = item / chunks, chunk = item - kt * chunks;
  const int kk = kt * BT;                  // first sorted position / sample slot / key row of the tile
  // The query tiles: `count` tiles of 64; first tile position a.  kind 0: sorted positions a + 64 j (mod m_q); 1: rows a + 64 j;
  // 2: exact transpose of the smooth forward: 128-row query tiles counted down from a, those whose window holds the key tile.
  int kind, a, count;
  if (!hyper) {
    kind = 1;
    a = causal ? kk : 0;
    count = (p.m_q - a + BT - 1) / BT;
  } else if (sampled) {
    kind = p.sample_logw ? 0 : 1;
    a = 0;
    count = p.m_q / BT;
  } else {
    const bool smooth = p.flags & HA_FLAG_SMOOTH;
    if (!smooth || (p.flags & HA_FLAG_BWD_REF_SMOOTH)) {
      const Window w = block_window(kk / TILE, bs, p.m_q, smooth);
      kind = 0;
      a = w.first;
      count = w.count / BT;
    } else {
      const int T_ = p.m_q / TILE;
      kind = 2;
      a = ((kk + (TILE / 2) * (bs - 1)) / TILE) % T_;
      count = 2 * min(bs, T_);             // with fewer tiles than a window spans, every tile pairs with the key once
    }
  }
  const int j0 = chunk * pl.chunk, j1 = min(count, j0 + pl.chunk);
  if (j0 >= j1) return;
  auto q_pos = [&](int j) -> int {         // first sorted position / row of tile j (-1: the tile does not meet these keys)
    if (kind == 1) return a + j * BT;
    int pos;
    if (kind == 0) {
      pos = a + j * BT;
      return pos >= p.m_q ? pos - p.m_q : pos;
    }
    int t = a - (j >> 1);
    if (t < 0) t += p.m_q / TILE;
    const Window w = block_window(t, bs, p.m_k, true);
    int off = kk - w.first;
    if (off < 0) off += p.m_k;
    return off >= w.count ? -1 : t * TILE + (j & 1) * BT;
  };
  const float* qb = (const float*)p.q + si.b * p.q_sb + si.h * p.q_sh + si.q_row0 * p.q_sn;
  const float* gb = (const float*)p.d_o + si.b * p.do_sb + si.h * p.do_sh + si.q_row0 * p.do_sn;
  const float* kb = (const float*)p.k + si.b * p.k_sb + si.hk * p.k_sh + si.k_row0 * p.k_sn;
  const float* vb = (const float*)p.v + si.b * p.v_sb + si.hk * p.v_sh + si.k_row0 * p.v_sn;
  const long long head0 = ((long long)(si.b * p.H + si.h)) * p.n + si.q_row0;
  const float* lse = p.lse + head0;
  const float* delta = p.delta + head0;
  if (tid < BT) {
    const int at = kk + tid;
    int row;
    if (!hyper) row = at < p.m_k ? at : -1;
    else if (sampled) row = p.sample_idx ? p.sample_idx[kseg * p.sample_size + at] : at;
    else row = p.k_idx[kseg * p.m_k + at];
    s_krow[tid] = row;
  }
  __syncthreads();
  load_tile<D, 256>(sK, kb, p.k_sn, s_krow);
  load_tile<DV, 256>(sV, vb, p.v_sn, s_krow);
  cp_async_commit();

  constexpr int NK = D / 64, NV = DV / 64;
  float4 dk[4][NK], dv[4][NV];             // keys tm * 4 + i, columns tn * 4 + 64 c
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int c = 0; c < NK; ++c) dk[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < NV; ++c) dv[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll 1
  for (int j = j0; j < j1; ++j) {
    const int pos0 = q_pos(j);
    if (pos0 < 0) continue;                // uniform over the CTA
    if (tid < BT) {
      const int pos = pos0 + tid;
      const int row = pos >= p.m_q ? -1 : kind == 1 ? pos : p.q_idx[(long long)seg * p.m_q + pos];
      s_qrow[tid] = row;
      s_lse[tid] = row < 0 ? INFINITY : lse[row];     // no such query: P = 0
      s_delta[tid] = row < 0 ? 0.f : delta[row];
    }
    __syncthreads();
    load_tile<D, 256>(sQ, qb, p.q_sn, s_qrow);
    load_tile<DV, 256>(sG, gb, p.do_sn, s_qrow);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    // ---- scores and their gradients: queries tm + 16 i, keys tn + 16 c ----
    float s[4][4], dp[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) s[i][c] = dp[i][c] = 0.f;
    // 32 columns are summed by themselves, as in the forward
    auto product = [&](float (&acc)[4][4], const float* A, const float* B, int W) {
#pragma unroll 1
      for (int k0 = 0; k0 < W; k0 += 32) {
        float t[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) t[i][c] = 0.f;
#pragma unroll 2
        for (int k = k0; k < k0 + 32; k += 4) {
          float4 b[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) b[c] = lds4(B + (tn + 16 * c) * (W + 4) + k);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 x = lds4(A + (tm + 16 * i) * (W + 4) + k);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              t[i][c] = fmaf(x.x, b[c].x, t[i][c]);
              t[i][c] = fmaf(x.y, b[c].y, t[i][c]);
              t[i][c] = fmaf(x.z, b[c].z, t[i][c]);
              t[i][c] = fmaf(x.w, b[c].w, t[i][c]);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[i][c] += t[i][c];
      }
    };
    product(s, sQ, sK, D);
    product(dp, sG, sV, DV);
    float bias = 0.f;
    uint32_t drop = 0;
    if (sampled && p.sample_logw) {
      const long long qtile = (long long)seg * (p.m_q / TILE) + pos0 / TILE;
      bias = p.sample_logw[qtile];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int slot = kk + tn + 16 * c;
        drop |= ((p.sample_mask[qtile * (p.sample_size / 32) + (slot >> 5)] >> (slot & 31)) & 1u) << c;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int qr = tm + 16 * i;
      const float ls = s_lse[qr], de = s_delta[qr];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int kc = tn + 16 * c;
        float pr = expf(s[i][c] * p.scale + bias - ls);
        if (((drop >> c) & 1u) || (!hyper && (kk + kc >= p.m_k || (causal && kk + kc > pos0 + qr)))) pr = 0.f;
        sP[qr * LDP + kc] = pr;
        sS[qr * LDP + kc] = pr * (dp[i][c] - de) * p.scale;
      }
    }
    __syncthreads();
    // ---- dV += P^T dO, dK += dS^T Q: a tile's product is summed by itself, as in the forward ----
    auto fold = [&](auto& acc, const float* weights, const float* rows, auto chunks) {
      constexpr int N = decltype(chunks)::value;
      float4 t[4][N];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < N; ++c) t[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int q = 0; q < BT; ++q) {
        const float4 x = lds4(weights + q * LDP + tm * 4);
#pragma unroll
        for (int c = 0; c < N; ++c) {
          const float4 b = lds4(rows + q * (64 * N + 4) + tn * 4 + 64 * c);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float f = at(x, i);
            t[i][c].x = fmaf(f, b.x, t[i][c].x);
            t[i][c].y = fmaf(f, b.y, t[i][c].y);
            t[i][c].z = fmaf(f, b.z, t[i][c].z);
            t[i][c].w = fmaf(f, b.w, t[i][c].w);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < N; ++c) { acc[i][c].x += t[i][c].x; acc[i][c].y += t[i][c].y; acc[i][c].z += t[i][c].z; acc[i][c].w += t[i][c].w; }
    };
    fold(dv, sP, sG, std::integral_constant<int, NV>{});
    fold(dk, sS, sQ, std::integral_constant<int, NK>{});
    // ---- dQ rows tm + 16 i += dS K ----
    {
      float4 dq[4][NK];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < NK; ++c) dq[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
      for (int k = 0; k < BT; k += 4) {
        float4 x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = lds4(sS + (tm + 16 * i) * LDP + k);
#pragma unroll
        for (int kq = 0; kq < 4; ++kq)
#pragma unroll
          for (int c = 0; c < NK; ++c) {
            const float4 b = lds4(sK + (k + kq) * (D + 4) + tn * 4 + 64 * c);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float f = at(x[i], kq);
              dq[i][c].x = fmaf(f, b.x, dq[i][c].x);
              dq[i][c].y = fmaf(f, b.y, dq[i][c].y);
              dq[i][c].z = fmaf(f, b.z, dq[i][c].z);
              dq[i][c].w = fmaf(f, b.w, dq[i][c].w);
            }
          }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = s_qrow[tm + 16 * i];
        if (row < 0) continue;
#pragma unroll
        for (int c = 0; c < NK; ++c) red4(p.dq_acc + (head0 + row) * D + tn * 4 + 64 * c, dq[i][c]);
      }
    }
    __syncthreads();                       // the tiles take the next queries
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = s_krow[tm * 4 + i];
    if (row < 0) continue;
    const long long r = si.khead0 + si.k_row0 + row;
#pragma unroll
    for (int c = 0; c < NK; ++c) red4(p.dk_acc + r * D + tn * 4 + 64 * c, dk[i][c]);
#pragma unroll
    for (int c = 0; c < NV; ++c) red4(p.dv_acc + r * DV + tn * 4 + 64 * c, dv[i][c]);
  }
  cp_async_wait<0>();
}

template <int D, int DV>
static int launch_f32_fwd(const ha_attn_params& p, cudaStream_t st) {
  const long long segs = (long long)p.B * p.H * p.segs_per_head;
  const int n_qt = (p.m_q + f32::BT - 1) / f32::BT;
  if (segs * n_qt == 0) return HA_OK;
  if (segs * n_qt > 0x7fffffffLL) return HA_ERR_TOO_LARGE;
  constexpr int SMEM = (2 * f32::BT * (D + 4) + f32::BT * (DV + 4) + f32::BT * f32::LDP) * 4;
  HA_SMEM_ATTR_ONCE((attn_f32_fwd_kernel<D, DV>), SMEM, "ha_attn_fwd smem attribute");
  attn_f32_fwd_kernel<D, DV><<<(unsigned)(segs * n_qt), 128, SMEM, st>>>(p, n_qt);
  HA_LAUNCHED("ha_attn_fwd (fp32 tiles)");
  return HA_OK;
}

template <int D, int DV>
static int launch_f32_bwd(const ha_attn_params& p, cudaStream_t st) {
  using f32::BT;
  const long long segs = (long long)p.B * p.H * p.segs_per_head;
  if (segs == 0 || p.m_q == 0 || p.m_k == 0) return HA_OK;
  F32BwdPlan pl{};
  const int n_qt = (p.m_q + BT - 1) / BT;
  int window;                                   // query tiles a block key tile meets at most
  if (p.mode == HA_MODE_HYPER) {
    const int bs = (p.block_size + TILE - 1) / TILE;
    window = 2 * bs < n_qt ? 2 * bs : n_qt;
    pl.smp_tiles = p.sample_size / BT;
  } else {
    window = n_qt;
  }
  pl.blk_tiles = (p.m_k + BT - 1) / BT;
  // Chunks of 16 query tiles, shorter ones (down to 4: an item's K / V loads and its dK / dV additions cost about a pair) where the
  // items would not fill the GPU several times over.
  long long items = 0;
  for (pl.chunk = 16; pl.chunk >= 4; pl.chunk >>= 1) {
    pl.blk_chunks = (window + pl.chunk - 1) / pl.chunk;
    pl.smp_chunks = (n_qt + pl.chunk - 1) / pl.chunk;
    pl.per_seg = pl.blk_tiles * pl.blk_chunks + pl.smp_tiles * pl.smp_chunks;
    items = segs * pl.per_seg;
    if (items >= 148LL * 8 || pl.chunk == 4) break;
  }
  if (items > 0x7fffffffLL) return HA_ERR_TOO_LARGE;
  constexpr int SMEM = (2 * BT * (D + 4) + 2 * BT * (DV + 4) + 2 * BT * f32::LDP) * 4;
  HA_SMEM_ATTR_ONCE((attn_f32_bwd_kernel<D, DV>), SMEM, "ha_attn_bwd smem attribute");
  attn_f32_bwd_kernel<D, DV><<<(unsigned)items, 256, SMEM, st>>>(p, pl);
  HA_LAUNCHED("ha_attn_bwd (fp32 tiles)");
  return HA_OK;
}

bool f32_tiled_supported(const ha_attn_params& p, bool backward) {
  if (p.dtype != HA_FP32 || !((p.d == 64 || p.d == 128) && (p.dv == 64 || p.dv == 128))) return false;
  auto ok = [](const void* ptr, int64_t sb, int64_t sh, int64_t sn) { return ((uintptr_t)ptr % 16 == 0) && sb % 4 == 0 && sh % 4 == 0 && sn % 4 == 0; };
  if (!ok(p.q, p.q_sb, p.q_sh, p.q_sn) || !ok(p.k, p.k_sb, p.k_sh, p.k_sn) || !ok(p.v, p.v_sb, p.v_sh, p.v_sn) || !ok(p.o, p.o_sb, p.o_sh, p.o_sn)) return false;
  if ((uintptr_t)p.part_o % 16 != 0) return false;
  if (!backward) return true;
  return ok(p.d_o, p.do_sb, p.do_sh, p.do_sn) && p.dq_acc && p.dk_acc && p.dv_acc && (uintptr_t)p.dq_acc % 16 == 0 && (uintptr_t)p.dk_acc % 16 == 0 &&
         (uintptr_t)p.dv_acc % 16 == 0;
}

int f32_tiled_fwd(const ha_attn_params& p, cudaStream_t st) {
  if (p.d == 64) return p.dv == 64 ? launch_f32_fwd<64, 64>(p, st) : launch_f32_fwd<64, 128>(p, st);
  return p.dv == 64 ? launch_f32_fwd<128, 64>(p, st) : launch_f32_fwd<128, 128>(p, st);
}
int f32_tiled_bwd(const ha_attn_params& p, cudaStream_t st) {
  if (p.d == 64) return p.dv == 64 ? launch_f32_bwd<64, 64>(p, st) : launch_f32_bwd<64, 128>(p, st);
  return p.dv == 64 ? launch_f32_bwd<128, 64>(p, st) : launch_f32_bwd<128, 128>(p, st);
}

}  // namespace ha
