// Persistent, warp-specialised backward on tcgen05 tensor cores + TMEM, head dims 128, bf16 / fp16: the sorted block windows + sampled
// rows (any block size; smooth windows enumerated per key tile; weighted sampling) and exact attention.  Replaces
// _bwd_permuted_block_diagonal_kernel and _bwd_sampled_col_kernel (src/hyper_attn_triton.py:399-506, :517-665) and the backward of
// src/flash_attn_triton.py:651-792.
//
// At this head dim dQ, dK and dV of a tile take 128 TMEM columns each, and the scores need the rest.  So key tiles are the outer
// loop: dK and dV of one key tile stay in TMEM over the query rows it meets, and dQ, which every key tile adds to, leaves after each
// step as fp32 additions.  An item is a key tile with all its query tiles (exact attention), or a pair of query tiles with the
// key tiles they meet (hyper pattern: the additions to a dQ row then follow one another closely and stay in L2).
//
// A step (unit) is 128 keys x 64 queries.  Scores are computed TRANSPOSED, lanes = keys:  S^T = K Q^T,  dP^T = V dO^T.  P^T goes back
// to TMEM over S^T and feeds  dV += P^T dO  as the A operand; dS^T goes to shared memory only ([key][query] rows), the A operand of
// dK += dS^T Q  and the B operand of  dQ^T = K^T dS^T,  which takes the columns that dP^T has left.  Units alternate
// between two TMEM stages, so that the elementwise phase of one runs underneath the tensor work of the other.
// dQ^T has lanes = head dim: the 32 lanes of a warp add 128 contiguous bytes of a query row, wherever the row lies, straight from
// registers.
//
// Roles (640 threads): two elementwise groups (128 threads each, one per stage), a drain group (128), five MMA warps (one product each,
// one elected lane issuing from warp-uniform code), three loader warps: Q with lse and delta (ring of three units; also works out the
// items), dO (ring of three), V and K tiles.
// TMEM columns: stage s at 128 s: S^T (then P^T) in [0, 64), dP^T (then dQ^T) in [64, 128); dV 256, dK 384.
// What bounds it: dQ's additions, 64 KB a pair of 128 x 128 tiles.  Scattered, they hold the load/store unit, and with it the loaders (32 heads x
// 32768, hyper: 1.06 ms, 4600 cycles a pair-half; the kernel that walked query tiles per key tile with dQ, P and dS through shared
// memory took 1.68 ms).  Consecutive rows, staged and added by the copy engine, are bound by L2 (8 heads x 32768, exact causal: 5.87 ms,
// 57% of the tensor rate; added from registers 6.27 ms).
// Hand-offs are mbarriers with bounded waits; a wait that gives up raises the CTA's abort flag, every role leaves its loop at its
// next wait, and the status words are set at the end.
#include "attn_items.cuh"

#include <type_traits>

namespace ha {

namespace bkt {
constexpr int D = 128, UQ = 64;                                // head dim, query rows of a unit
constexpr int TILE_B = TILE * 128;                             // one slab: 128 rows x 64 elements
constexpr int SLAB_U = UQ * 128;                               // one slab of a unit's operand: 64 rows x 64 elements
constexpr int NU = 3;                                          // units in flight
constexpr int OFF_K = 0;
constexpr int OFF_V = OFF_K + 2 * TILE_B;
constexpr int OFF_Q = OFF_V + 2 * TILE_B;                      // unit slots: Q
constexpr int OFF_DO = OFF_Q + NU * 2 * SLAB_U;                // ... dO
constexpr int OFF_DS = OFF_DO + NU * 2 * SLAB_U;               // dS^T of the two stages: 128 key rows x 64 queries
constexpr int OFF_ST = OFF_DS + 2 * TILE_B;                    // staging of the drain group, 2 x 16 KB (below)
constexpr int OFF_LD = OFF_ST + 2 * TILE_B;                      // per unit slot: -lse log2e [64], -delta scale [64] (fp32)
constexpr int SMEM_USED = OFF_LD + NU * 512;                   // from the first 1 KB boundary after the static variables
constexpr int THREADS = 640;
constexpr int W_DRAIN = 8, W_MMA = 12, W_Q = 17, W_DO = 18;    // first warp of each role (K and V: 19)
constexpr int COL_DV = 256, COL_DK = 384;
constexpr int ND = 4, CONSUMERS = 19;                          // descriptor ring; warps that read every descriptor (all but the writer)
// barrier slots (index + stage / unit slot) and their arrivals per phase
enum {
  B_K_FULL = 0,       // 32: every lane of the loader, through its copies
  B_K_EMPTY = 1,      // 2: the S^T and dQ warps
  B_V_FULL = 2,       // 32
  B_V_EMPTY = 3,      // 1: the dP^T warp
  B_Q_FULL = 4,       // NU x 64: the loader's lanes through their copies, and for the lse / delta they wrote
  B_Q_EMPTY = 7,      // NU x 2: the S^T and dK warps
  B_DO_FULL = 10,     // NU x 32
  B_DO_EMPTY = 13,    // NU x 2: the dP^T and dV warps
  B_S_READY = 16,     // 2 x 2: S^T and dP^T of a stage are in TMEM
  B_P_READY = 18,     // 2 x 128: its elementwise group has written P^T and dS^T
  B_S_FREE = 20,      // 2 x 1: dV of the stage's unit completed: S^T may be overwritten
  B_DS_FREE = 22,     // 2 x 1: dK of the stage's unit completed (dQ's reading is over before the stage's next scores exist)
  B_DQ_FULL = 24,     // 2 x 1: dQ^T of the stage's unit is in TMEM
  B_DQ_FREE = 26,     // 2 x 128: ... drained: dP^T may be overwritten
  B_ACC_FULL = 28,    // 2 x 1: dV / dK of a key tile complete
  B_ACC_FREE = 30,    // 2 x 128: ... drained
  B_ST_FULL = 32,     // 2 x 128: every drain thread has written its column of the staged rows
  B_ST_IDLE = 34,     // 128: every drain thread is done with a key tile's staging
  B_ST_FREE = 35,     // 2 x 1: the copy engine has read the staged rows
  B_D_FULL = 37,      // ND x 1
  B_D_EMPTY = 37 + ND,
  N_BARS = 37 + 2 * ND
};
__device__ __forceinline__ int bar_count(int i) {
  if (i >= B_D_EMPTY) return CONSUMERS;
  if (i >= B_D_FULL || i == B_V_EMPTY) return 1;
  if (i == B_K_FULL || i == B_V_FULL || (i >= B_DO_FULL && i < B_DO_EMPTY)) return 32;
  if (i >= B_Q_FULL && i < B_Q_EMPTY) return 64;
  if (i < B_P_READY) return 2;                       // K_EMPTY, Q_EMPTY, DO_EMPTY, S_READY
  if (i < B_S_FREE || (i >= B_DQ_FREE && i < B_ACC_FULL) || (i >= B_ACC_FREE && i < B_ST_FREE)) return 128;
  return 1;
}
}  // namespace bkt

enum { KT_HYPER = 0, KT_FLASH = 1, KT_ANY = 2 };               // the plain hyper pattern, exact attention, the hyper pattern in any form
struct KtMaps { CUtensorMap tile[4]; };                        // tiles of q, k, v, dO

// Entries [e0, e1) of the list of key tiles, each with the query tiles [y0, y1) it meets.
struct KtItem : AttnItem {
  int e0, e1, y0, y1;
};
__device__ __forceinline__ KtItem kt_item(const ha_attn_params& p, const AttnPlan& pl, int item, bool flash, bool by_keys) {
  KtItem it;
  if (!flash) {
    static_cast<AttnItem&>(it) = attn_item(p, pl, item, false, by_keys);
    it.e0 = 0; it.e1 = it.n_list;
    it.y0 = 0; it.y1 = 2;
    return it;
  }
  // Key tile kt of its segment; causal items shrink with kt
  const bool causal = p.flags & HA_FLAG_CAUSAL;
  int kt;
  if (causal) {
    kt = causal_place(pl, item, it.seg);
  } else {
    it.seg = pl.by_pairs(item);
    kt = item - it.seg * pl.pairs;
  }
  it.qt0 = 0; it.has1 = 1; it.q_pos0 = 0; it.first = 0; it.lo1 = 0;
  it.hi0 = it.hi1 = it.n_win = it.n_list = kt + 1;
  it.e0 = kt; it.e1 = kt + 1;
  it.y0 = causal ? kt : 0; it.y1 = (p.m_q + TILE - 1) / TILE;
  const int bh = pl.by_segs(it.seg), part = it.seg - bh * p.segs_per_head, group = p.kv_group > 1 ? p.kv_group : 1;
  it.b = pl.by_heads(bh);
  it.h = bh - it.b * p.H;
  it.hk = pl.by_group(it.h);
  it.q_row0 = part * p.span + p.q_off;
  it.k_row0 = part * p.span + p.k_off;
  it.kseg = group > 1 ? (it.b * pl.by_group(p.H) + it.hk) * p.segs_per_head + part : it.seg;
  return it;
}

// `bytes` of fp32 in shared memory -> added to global memory; the four below concern the calling thread's copies
__device__ __forceinline__ void bulk_add_f32(float* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void red_add_f32(float* addr, float v) { asm volatile("red.global.add.f32 [%0], %1;" ::"l"(addr), "f"(v) : "memory"); }
// the 64 rows of a unit's operand, gathered by one warp: rows[q] = source row of unit row 32 q + lane (-1: zero fill)
__device__ __forceinline__ void warp_gather_unit(uint32_t dst, const uint16_t* __restrict__ base, int64_t row_stride, int r0, int r1, int lane) {
  const int chunk = lane & 7;
#pragma unroll 1
  for (int q = 0; q < 2; ++q) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int rl = 4 * i + (lane >> 3), row = q * 32 + rl;
      const int src_row = __shfl_sync(0xffffffffu, r0, rl);
      const uint32_t at = dst + row * 128 + ((chunk ^ (row & 7)) << 4);
      const uint16_t* src = base + (int64_t)(src_row < 0 ? 0 : src_row) * row_stride + chunk * 8;
      cp_async16(at, src, src_row >= 0 ? 16u : 0u);
      cp_async16(at + bkt::SLAB_U, src + 64, src_row >= 0 ? 16u : 0u);
    }
    r0 = r1;
  }
}

template <typename T, int KIND>
__global__ void __launch_bounds__(bkt::THREADS, 1) attn_tc_bwd_kt_kernel(const ha_attn_params p, const AttnPlan pl, const __grid_constant__ KtMaps maps) {
  chain_begin();
  using namespace bkt;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t s_base = smem_u32(smem);
  __shared__ __align__(16) KtItem s_item[ND];
  __shared__ uint64_t bars[N_BARS];
  __shared__ uint32_t tmem_slot;
  __shared__ uint32_t s_issued[3];        // units of Q, units of dO, operands of key tiles (V, then K) that the loaders have asked for
  __shared__ int s_abort;
  __shared__ int s_bail;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  constexpr bool flash = KIND == KT_FLASH;
  constexpr bool ANY = KIND == KT_ANY;

  if (cta_sees_failure(p.status, &s_bail)) return;   // an earlier CTA gave up: drain quickly (uniform over the CTA)
  {
    // Should the dynamic window start somewhere else than assumed, do nothing rather than run over its end.
    uint32_t dyn;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
    if ((uint32_t)(smem - smem_raw) + (uint32_t)SMEM_USED > dyn) {      // uniform over the grid
      if (tid == 0) report_status(p.status, p.status_host, HA_DEV_BAD_LAUNCH);
      return;
    }
  }
  const uint32_t bar0 = smem_u32(bars);
  auto bar = [&](int i) -> uint32_t { return bar0 + 8 * i; };
  if (tid == 0) {
    for (int i = 0; i < N_BARS; ++i) mbar_init(bar(i), bar_count(i));
    s_abort = 0;
    mbar_fence_init();
  }
  if (warp == W_MMA) tmem_alloc(smem_u32(&tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  // A wait that gives up (or finds the abort flag up) ends the role's loop; the status word is set once, at the end.  Called by whole
  // warps; one answer for the warp.
  auto wait = [&](int b, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_wait_or_abort(bar(b), parity, &s_abort)); };
  uint32_t n_item = 0;       // descriptors this warp has taken
  // the next item's descriptor; false: no more items (or a wait gave up)
  auto next_item = [&](KtItem& it) -> bool {
    const int slot = n_item % ND;
    if (!wait(B_D_FULL + slot, (n_item / ND) & 1)) return false;
    it = s_item[slot];
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_D_EMPTY + slot));
    ++n_item;
    return it.n_list != 0;
  };
  auto active = [&](const KtItem& it, int y, int e) -> bool { return flash || it.active(y, e); };
  constexpr float LOG2E = 1.4426950408889634f;

  // Register budget: 640 threads x 96 at launch = 61440 = 256 x 128 (elementwise) + 128 x 96 (drain) + 256 x 64 (the rest).
  if (warp < W_DRAIN) {
    // =====================================================================================================
    // elementwise groups: P^T = exp2(S^T scale log2e - lse log2e), dS^T = P^T (dP^T - delta) scale
    // =====================================================================================================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 128;");
    const int g = warp >> 2;
    const uint32_t tS = tmem + 128 * g + ((uint32_t)((warp & 3) * 32) << 16), tDP = tS + 64;
    const uint64_t sc2 = pack_f2(p.scale * LOG2E, p.scale * LOG2E), scl = pack_f2(p.scale, p.scale);
    const bool causal = flash && (p.flags & HA_FLAG_CAUSAL);
    uint32_t pair = 0, slot = g, lap = 0;       // units of this group so far; unit slot and its lap round the ring
    const uint32_t ds_rows = s_base + OFF_DS + g * TILE_B + (32 * (warp & 3) + (lane & 7)) * 128;
    bool ok = true;
    HA_T_DECL(8)
    KtItem it;
    while (ok && next_item(it)) {
#pragma unroll 1
      for (int e = it.e0; e < it.e1 && ok; ++e) {
#pragma unroll 1
        for (int y = it.y0; y < it.y1; ++y) {
          if (!active(it, y, e)) continue;
          HA_T_MARK(0)
          if (!(ok = wait(B_S_READY + g, pair & 1))) break;
          HA_T_MARK(1)
          if (!(ok = wait(B_Q_FULL + slot, lap & 1))) break;                              // (long complete: for lse / delta to be seen)
          if (pair >= 1 && !(ok = wait(B_DS_FREE + g, (pair - 1) & 1))) break;
          HA_T_MARK(2)
          tc_fence_after();
          const float* ld = reinterpret_cast<const float*>(smem + OFF_LD + slot * 512);      // lse; delta 64 floats on
          float bias2 = 0.f;
          const bool weighted = ANY && p.sample_logw && e >= it.n_win;
          const uint32_t* drop = nullptr;
          if (weighted) {
            int pos = it.q_pos0 + y * TILE + UQ * g;
            if (pos >= p.m_q) pos -= p.m_q;
            const long long qtile = (long long)it.seg * (p.m_q / TILE) + pos / TILE;
            bias2 = p.sample_logw[qtile] * LOG2E;
            drop = p.sample_mask + qtile * (p.sample_size / 32) + (e - it.n_win) * (TILE / 32) + (warp & 3);
          }
          const bool diag = causal && e == y, masked = KIND != KT_HYPER && (weighted || diag || (flash && (e + 1) * TILE > p.m_k));
          const uint64_t bias = pack_f2(bias2, bias2);
          // Fragments of 16 keys x 8 queries, two keys and two neighbouring queries a thread, 16 keys x 32 queries at a time: the thread
          // needs the lse and delta of 8 queries, where with a key a thread it needed those of all of them, as broadcast reads (steps: decoder 2 x 16 x
          // 8192 1388 -> 1355 us, 8 x 32 x 2047 exact causal 1532 -> 1488, 32 x 32768 hyper 1868 -> 1827).
#pragma unroll 1
          for (int c = 0; c < 2; ++c) {
            const uint32_t ds_to = ds_rows + (((4 * c + (lane >> 3)) ^ (lane & 7)) << 4);
            uint64_t L[4], Dl[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              L[j] = *reinterpret_cast<const uint64_t*>(ld + 32 * c + 8 * j + 2 * (lane & 3));
              Dl[j] = *reinterpret_cast<const uint64_t*>(ld + UQ + 32 * c + 8 * j + 2 * (lane & 3));
              if (ANY) L[j] = fadd2(L[j], bias);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint32_t rs[16], rp[16], pk[8], dk[8];
              tmem_ld_16x256(tS + 32 * c + (h << 20), rs);
              tmem_ld_16x256(tDP + 32 * c + (h << 20), rp);
              tmem_ld_fence16(rs);
              tmem_ld_fence16(rp);
              // queries [0, hidden) of these 32 do not count for a key row
              int hidden[2] = {0, 0};
              if (masked) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                  const int row = 32 * (warp & 3) + 16 * h + 8 * k + (lane >> 2);
                  if (flash) {
                    if (diag) hidden[k] = row - UQ * g - 32 * c;               // queries before the key
                    if (e * TILE + row >= p.m_k) hidden[k] = 32;               // past the last key
                  } else if ((*drop >> (row & 31)) & 1u) {
                    hidden[k] = 32;
                  }
                }
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                  const int i = 4 * j + 2 * k, at = 8 * j + 2 * (lane & 3);
                  float p0, p1, d0, d1;
                  unpack_f2(ffma2(pack_u2(rs[i], rs[i + 1]), sc2, L[j]), p0, p1);
                  p0 = fast_exp2(p0); p1 = fast_exp2(p1);
                  if (masked) {
                    if (at < hidden[k]) p0 = 0.f;
                    if (at + 1 < hidden[k]) p1 = 0.f;
                  }
                  // ds = p * (dp - delta) * scale
                  unpack_f2(fmul2(pack_f2(p0, p1), ffma2(pack_u2(rp[i], rp[i + 1]), scl, Dl[j])), d0, d1);
                  pk[2 * j + k] = pack2<T>(p0, p1);
                  dk[2 * j + k] = pack2<T>(d0, d1);
                }
              }
              tmem_st_16x128(tS + 32 * c + (h << 20), pk);      // P^T (16 packed columns) over columns this warp has consumed
#pragma unroll
              for (int k = 0; k < 2; ++k) store_matrix_x4(ds_to + (16 * h + 8 * k) * 128, dk[k], dk[2 + k], dk[4 + k], dk[6 + k]);
            }
          }
          HA_T_MARK(3)
          tmem_st_wait();
          fence_async_smem();       // the dS rows are read by the tensor core (async proxy)
          tc_fence_before();
          mbar_arrive(bar(B_P_READY + g));
          ++pair;
          slot += 2;                // the group takes every other unit
          if (slot >= NU) { slot -= NU; ++lap; }
          HA_T_MARK(4)
        }
      }
    }
    HA_T_DUMP(8, (int)blockIdx.x * 8, tid == 0)
  } else if (warp < W_MMA) {
    // =====================================================================================================
    // drain group: dQ^T of every unit, dV and dK of every key tile -> global memory
    // =====================================================================================================
    const int row = tid & 127, rot = row & 7;
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
    uint8_t* my_row = smem + OFF_ST + row * 128;
    const uint8_t* warp_rows = smem + OFF_ST + (row & ~31) * 128;
    const bool kv_init = p.flags & HA_FLAG_BWD_KV_INIT;
    uint32_t unit = 0, n_kt = 0;                            // units / key tiles drained so far
    bool staged = false, last_freed = false;                // a key tile's staging has not been seen idle; (issuer) the last half's rows are known to be read
    bool ok = true;
    HA_T_DECL(8)
    KtItem it;
    while (ok && next_item(it)) {
      const int Hk = p.kv_group > 1 ? pl.by_group(p.H) : p.H;
      float* dq_base = p.dq_acc + ((long long)(it.b * p.H + it.h) * p.n + it.q_row0) * D + (flash ? 0 : row);      // (scattered rows: this lane's element)
#pragma unroll 1
      for (int e = it.e0; e < it.e1 && ok; ++e) {
#pragma unroll 1
        for (int y = it.y0; y < it.y1 && ok; ++y) {
          if (!active(it, y, e)) continue;
#pragma unroll 1
          for (int s = 0; s < 2; ++s, ++unit) {
            int q0 = 0, q1 = 0;                             // query rows lane and 32 + lane of the unit
            if (!flash) {
              int pos0 = it.q_pos0 + y * TILE + UQ * s + lane, pos1 = pos0 + 32;
              if (pos0 >= p.m_q) pos0 -= p.m_q;
              if (pos1 >= p.m_q) pos1 -= p.m_q;
              q0 = p.q_idx[(long long)it.seg * p.m_q + pos0];
              q1 = p.q_idx[(long long)it.seg * p.m_q + pos1];
            }
            HA_T_MARK(0)
            if (!(ok = wait(B_DQ_FULL + s, (unit >> 1) & 1))) break;
            HA_T_MARK(1)
            tc_fence_after();
            uint32_t r[2][32];
            tmem_ld32(tmem + 128 * s + 64 + lane_sel, r[0]);
            tmem_ld32(tmem + 128 * s + 96 + lane_sel, r[1]);
            tmem_ld_fence(r[0]);
            tmem_ld_fence(r[1]);
            tc_fence_before();
            mbar_arrive(bar(B_DQ_FREE + s));          // (the additions do not hold the stage up)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              if (flash) {
                // 32 consecutive rows: staged as they lie in memory, added by the copy engine
                const int pos0 = it.q_pos0 + y * TILE + UQ * s + 32 * hf, valid = min(p.m_q - pos0, 32);
                uint8_t* to = smem + OFF_ST + hf * TILE_B + row * 4;
                if (hf == 0 && staged && !(ok = wait(B_ST_IDLE, (n_kt - 1) & 1))) break;
                staged = false;
                if (unit >= 1 && !(ok = wait(B_ST_FREE + hf, (unit - 1) & 1))) break;
#pragma unroll
                for (int i = 0; i < 32; ++i) *reinterpret_cast<uint32_t*>(to + i * (D * 4)) = r[hf][i];
                fence_async_smem();
                mbar_arrive(bar(B_ST_FULL + hf));
                if (warp == W_DRAIN) {
                  if (!(ok = wait(B_ST_FULL + hf, unit & 1))) break;
                  if (lane == 0) {
                    if (valid > 0) bulk_add_f32(dq_base + (long long)pos0 * D, s_base + OFF_ST + hf * TILE_B, valid * (D * 4));
                    bulk_commit();
                    if (unit + hf > 0) {
                      bulk_wait_read<1>();          // the half before has been read
                      if (!last_freed) mbar_arrive(bar(B_ST_FREE + (hf ^ 1)));
                    }
                    last_freed = false;
                  }
                  __syncwarp();
                }
              } else {
                // the row numbers eight at a time: one by one, each addition would wait for a shuffle
#pragma unroll
                for (int i = 0; i < 32; i += 8) {
                  int to[8];
#pragma unroll
                  for (int j = 0; j < 8; ++j) to[j] = __shfl_sync(0xffffffffu, hf ? q1 : q0, i + j);
#pragma unroll
                  for (int j = 0; j < 8; ++j) red_add_f32(dq_base + (long long)to[j] * D, __uint_as_float(r[hf][i + j]));
                }
              }
            }
            if (!ok) break;
            HA_T_MARK(2)
          }
        }
        if (!ok) break;
        // dV, dK of the key tile: 128 rows x 128 bytes staged at a time, a warp's 32 rows in 4 KB of its own
        if (flash) {
          if (warp == W_DRAIN) {
            if (lane == 0) {
              bulk_wait_read<0>();
              mbar_arrive(bar(B_ST_FREE + 1));
              last_freed = true;
            }
            __syncwarp();
          }
          // (both halves of the last unit: the first was seen free when the second was issued)
          if (!(ok = wait(B_ST_FREE, (unit - 1) & 1)) || !(ok = wait(B_ST_FREE + 1, (unit - 1) & 1))) break;
        }
        int local = item_key_row(p, it, e, row, flash);
        if (local >= 0) local += it.k_row0;
        const bool sampled = !flash && e >= it.n_win;
        const bool typed = p.dk_out && !sampled;
        const bool slots = p.dk_out && sampled;             // rows of the slot buffers
        const long long rows0 = slots ? (long long)it.kseg * p.sample_size + (e - it.n_win) * TILE : (long long)(it.b * Hk + it.hk) * p.n;
        if (slots) local = row;
        int to[8];                                          // the rows this lane writes a sixteenth or an eighth of (-1: none)
#pragma unroll
        for (int j = 0; j < 8; ++j) to[j] = __shfl_sync(0xffffffffu, local, 4 * j + (lane >> 3));
#pragma unroll 1
        for (int is_k = 0; is_k < 2; ++is_k) {
          T* to_typed = (T*)(is_k ? p.dk_out : p.dv_out);
          float* acc = p.dk_out ? (is_k ? p.dk_sacc : p.dv_sacc) : (is_k ? p.dk_acc : p.dv_acc);
          HA_T_MARK(0)
          if (!(ok = wait(B_ACC_FULL + is_k, n_kt & 1))) break;
          HA_T_MARK(3)
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t r[32];
            tmem_ld32(tmem + (is_k ? COL_DK : COL_DV) + c * 32 + lane_sel, r);
            tmem_ld_fence(r);
            if (c == 3) {
              tc_fence_before();
              mbar_arrive(bar(B_ACC_FREE + is_k));
            }
            if (typed) {
              // two chunks fill the 128 bytes of a staged row
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                uint32_t w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) w[j] = pack2<T>(__uint_as_float(r[8 * i + 2 * j]), __uint_as_float(r[8 * i + 2 * j + 1]));
                *reinterpret_cast<uint4*>(my_row + ((((c & 1) * 4 + i) ^ rot) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
              }
              if (!(c & 1)) continue;
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(my_row + ((i ^ rot) << 4)) = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
            }
            // eight lanes cover the 128 contiguous bytes of a row
            __syncwarp();
            const int w = lane & 7;
            float4 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int rl = 4 * j + (lane >> 3);
              v[j] = *reinterpret_cast<const float4*>(warp_rows + rl * 128 + ((w ^ (rl & 7)) << 4));
            }
            if (typed) {
              T* out = to_typed + rows0 * D + (c >> 1) * 64 + w * 8;
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (to[j] >= 0) *reinterpret_cast<float4*>(out + (long long)to[j] * D) = v[j];
            } else {
              float* out = acc + rows0 * D + c * 32 + w * 4;
              if (kv_init) {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                  if (to[j] >= 0) *reinterpret_cast<float4*>(out + (long long)to[j] * D) = v[j];
              } else {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                  if (to[j] >= 0) red_add_v4(out + (long long)to[j] * D, v[j]);
              }
            }
            __syncwarp();
          }
          HA_T_MARK(4)
        }
        if (flash) {
          mbar_arrive(bar(B_ST_IDLE));
          staged = true;
        }
        ++n_kt;
      }
    }
    bulk_wait_all();       // nothing of this thread is in flight when the CTA retires
    HA_T_DUMP(8, (int)blockIdx.x * 8 + 2, row == 0)
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    if (warp < W_Q) {
      // ===================================================================================================
      // MMA issue, one warp per product.  Each walks the units in order and waits (bounded) for what its next instructions need.  The
      // "empty" barriers of the operands collect one commit from every warp that reads them.
      // ===================================================================================================
      constexpr int AB = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
      const int role = warp - W_MMA;            // 0: S^T, 1: dP^T, 2: dV, 3: dK, 4: dQ^T
      uint32_t unit = 0, kt = 0, slot = 0, lap = 0;
      bool ok = true;
      HA_T_DECL(8)
      KtItem it;
      while (ok && next_item(it)) {
#pragma unroll 1
        for (int e = it.e0; e < it.e1 && ok; ++e, ++kt) {
          HA_T_MARK(0)
          if (role < 2) {
            if (!(ok = wait(role ? B_V_FULL : B_K_FULL, kt & 1))) break;
            fence_async_smem();     // (tiles that came by cp.async)
          }
          HA_T_MARK(1)
          bool fresh = true;                    // nothing accumulated yet for this key tile
#pragma unroll 1
          for (int y = it.y0; y < it.y1 && ok; ++y) {
            if (!active(it, y, e)) continue;
            const bool tile_done = flash ? y + 1 == it.y1 : (y == 1 || !it.active(1, e));
#pragma unroll 1
            for (int s = 0; s < 2; ++s) {
              const uint32_t sQ = s_base + OFF_Q + slot * 2 * SLAB_U, sDO = s_base + OFF_DO + slot * 2 * SLAB_U, sDS = s_base + OFF_DS + s * TILE_B;
              const uint32_t par = (unit >> 1) & 1;
              HA_T_MARK(0)
              if (role < 2) {
                // S^T = K Q^T / dP^T = V dO^T: M = 128 keys, N = 64 query rows, both operands K-major
                if (!(ok = wait((role ? B_DO_FULL : B_Q_FULL) + slot, lap & 1))) break;
                fence_async_smem();
                HA_T_MARK(2)
                // P^T of the stage's last unit has been read / its dQ^T drained
                if (unit >= 2 && !(ok = wait((role ? B_DQ_FREE : B_S_FREE) + s, par ^ 1))) break;
                HA_T_MARK(3)
                tc_fence_after();
                const uint32_t idesc = mma_idesc(TILE, UQ, AB, 0, 0);
                const uint64_t dA = smem_desc(s_base + (role ? OFF_V : OFF_K), 16, 1024), dB = smem_desc(role ? sDO : sQ, 16, 1024);
                if (elect_one()) {
#pragma unroll
                  for (int kk = 0; kk < 8; ++kk)
                    mma_ss(tmem + 128 * s + role * 64, dA + (kk >> 2) * (TILE_B >> 4) + (kk & 3) * (32 >> 4), dB + (kk >> 2) * (SLAB_U >> 4) + (kk & 3) * (32 >> 4),
                           idesc, kk > 0);
                  mma_commit(bar(B_S_READY + s));
                  mma_commit(bar((role ? B_DO_EMPTY : B_Q_EMPTY) + slot));
                }
              } else {
                if (!(ok = wait(B_P_READY + s, par))) break;
                if (role < 4 && fresh && kt >= 1 && !(ok = wait(B_ACC_FREE + role - 2, (kt - 1) & 1))) break;    // the accumulator restarts with the key tile
                HA_T_MARK(3)
                fence_async_smem();
                tc_fence_after();
                if (role == 2) {
                  // dV += P^T dO: A in TMEM, B rows as MN-major
                  const uint32_t idesc = mma_idesc(TILE, D, AB, 0, 1);
                  const uint64_t dB = smem_desc(sDO, SLAB_U, 1024);
                  if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) mma_ts(tmem + COL_DV, tmem + 128 * s + (kk >> 1) * 32 + (kk & 1) * 8, dB + kk * (2048 >> 4), idesc, !fresh | (kk > 0));
                    mma_commit(bar(B_S_FREE + s));
                    mma_commit(bar(B_DO_EMPTY + slot));
                    if (s == 1 && tile_done) mma_commit(bar(B_ACC_FULL));
                  }
                } else if (role == 3) {
                  // dK += dS^T Q: A = dS^T rows (K-major), B rows as MN-major
                  const uint32_t idesc = mma_idesc(TILE, D, AB, 0, 1);
                  const uint64_t dA = smem_desc(sDS, 16, 1024), dB = smem_desc(sQ, SLAB_U, 1024);
                  if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) mma_ss(tmem + COL_DK, dA + kk * (32 >> 4), dB + kk * (2048 >> 4), idesc, !fresh | (kk > 0));
                    mma_commit(bar(B_DS_FREE + s));
                    mma_commit(bar(B_Q_EMPTY + slot));
                    if (s == 1 && tile_done) mma_commit(bar(B_ACC_FULL + 1));
                  }
                } else {
                  // dQ^T = K^T dS^T over the 128 keys: both operands have a key per row (MN-major)
                  const uint32_t idesc = mma_idesc(D, UQ, AB, 1, 1);
                  const uint64_t dA = smem_desc(s_base + OFF_K, TILE_B, 1024), dB = smem_desc(sDS, TILE_B, 1024);
                  if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk) mma_ss(tmem + 128 * s + 64, dA + kk * (2048 >> 4), dB + kk * (2048 >> 4), idesc, kk > 0);
                    mma_commit(bar(B_DQ_FULL + s));
                  }
                }
                fresh = false;
              }
              __syncwarp();
              HA_T_MARK(4)
              ++unit;
              if (++slot == NU) { slot = 0; ++lap; }
            }
          }
          if (ok && (role == 0 || role == 1 || role == 4) && elect_one()) mma_commit(bar(role == 1 ? B_V_EMPTY : B_K_EMPTY));      // this warp's last read of the tile
          __syncwarp();
        }
      }
      HA_T_DUMP(8, (int)blockIdx.x * 8 + (role == 0 ? 4 : role == 1 ? 1 : role == 2 ? 5 : 6), lane == 0 && role != 3)
    } else if (warp <= W_DO) {
      // ===================================================================================================
      // loaders of the query side, unit by unit: Q with lse and delta (warp 17, which is also the scheduler), dO (warp 18)
      // ===================================================================================================
      const bool is_q = warp == W_Q;
      const bool by_keys = ANY && (p.flags & HA_FLAG_SMOOTH);
      const bool boxed = flash && pl.tiles;
      int published = 0;
      auto take = [&](KtItem& it) -> bool {        // the next item's descriptor; n_list = 0 past the last one
        if (!is_q) return next_item(it);
#pragma unroll 1
        for (; published <= (int)n_item + 2; ++published) {
          const uint32_t at = published % ND;
          it.n_list = 0;
          const int item = item_of_turn<KIND == KT_FLASH>(pl, published, blockIdx.x, gridDim.x);
          if (item < pl.n_items) it = kt_item(p, pl, item, flash, by_keys);
          if (published >= ND && !wait(B_D_EMPTY + at, (published / ND - 1) & 1)) return false;
          if (lane == 0) {
            s_item[at] = it;
            mbar_arrive(bar(B_D_FULL + at));
          }
          __syncwarp();
        }
        it = s_item[n_item % ND];
        ++n_item;
        return it.n_list != 0;
      };
      KtItem it;
      int e = 0, y = 0;
      bool more = take(it);
      // (every list starts with a key tile that its first query tile meets)
      if (more) { e = it.e0; y = it.y0; }
      auto advance = [&]() {
        do {
          if (++y < it.y1) continue;
          y = it.y0;
          if (++e < it.e1) continue;
          more = take(it);
          if (more) { e = it.e0; y = it.y0; }
          return;
        } while (!active(it, y, e));
      };
      // row numbers of the query tile's two units (-1: none)
      auto row_numbers = [&](int (&rows)[4]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          int pos = it.q_pos0 + y * TILE + 32 * q + lane;
          if (flash) {
            rows[q] = pos < p.m_q ? pos : -1;
          } else {
            if (pos >= p.m_q) pos -= p.m_q;
            rows[q] = p.q_idx[(long long)it.seg * p.m_q + pos];
          }
        }
      };
      auto lse_delta = [&](const int (&rows)[4], float (&l)[4], float (&dl)[4]) {
        const long long at = ((long long)(it.b * p.H + it.h)) * p.n + it.q_row0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          l[q] = rows[q] >= 0 ? p.lse[at + rows[q]] : INFINITY;      // no such query: P = 0
          dl[q] = rows[q] >= 0 ? p.delta[at + rows[q]] : 0.f;
        }
      };
      const uint16_t* tensor = (const uint16_t*)(is_q ? p.q : p.d_o);
      const int64_t sb = is_q ? p.q_sb : p.do_sb, sh = is_q ? p.q_sh : p.do_sh, sn = is_q ? p.q_sn : p.do_sn;
      const int b_full = is_q ? B_Q_FULL : B_DO_FULL, b_empty = is_q ? B_Q_EMPTY : B_DO_EMPTY;
      const uint32_t ring = s_base + (is_q ? OFF_Q : OFF_DO);
      uint32_t n = 0, slot = 0, lap = 0;
      int rows[4] = {0, 0, 0, 0}, ahead[4] = {0, 0, 0, 0};
      float l[4], dl[4], l_ahead[4], dl_ahead[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) l[q] = dl[q] = l_ahead[q] = dl_ahead[q] = 0.f;
      if (more) {
        row_numbers(rows);
        if (is_q) lse_delta(rows, l, dl);
      }
      bool ok = true;
      HA_T_DECL(8)
      while (more && ok) {
        HA_T_MARK(2)
        const int b = it.b, h = it.h, q_row0 = it.q_row0, box_row = q_row0 + it.q_pos0 + y * TILE;
        const uint16_t* base = tensor + b * sb + h * sh + (int64_t)q_row0 * sn;
        // The next query tile's row numbers travel while this one's first unit waits for its slot, what they index while the second does.
        advance();
        if (more) row_numbers(ahead);
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          HA_T_MARK(0)
          if (ok && n >= NU) ok = wait(b_empty + slot, (lap - 1) & 1);
          if (!ok) break;
          HA_T_MARK(1)
          const uint32_t full = bar(b_full + slot), dst = ring + slot * 2 * SLAB_U;
          if (boxed) {
            const int ur = __shfl_sync(0xffffffffu, box_row + UQ * s, 0), uh = __shfl_sync(0xffffffffu, h, 0), ub = __shfl_sync(0xffffffffu, b, 0);
            if (elect_one()) {
              mbar_add_tx(full, 2 * SLAB_U);
              tma_tile(dst, &maps.tile[is_q ? 0 : 3], 0, ur, uh, ub, full);
              tma_tile(dst + SLAB_U, &maps.tile[is_q ? 0 : 3], 64, ur, uh, ub, full);
            }
            __syncwarp();
            mbar_arrive(full);
          } else {
            warp_gather_unit(dst, base, sn, rows[2 * s], rows[2 * s + 1], lane);
            push_copies(full);
          }
          if (is_q) {
            float* at = reinterpret_cast<float*>(smem + OFF_LD + slot * 512);
            at[lane] = -LOG2E * l[2 * s];
            at[32 + lane] = -LOG2E * l[2 * s + 1];
            at[UQ + lane] = -p.scale * dl[2 * s];
            at[UQ + 32 + lane] = -p.scale * dl[2 * s + 1];
            mbar_arrive(full);
            if (s == 0 && more) lse_delta(ahead, l_ahead, dl_ahead);
          }
          ++n;
          if (++slot == NU) { slot = 0; ++lap; }
        }
        if (!flash && more && e == it.e0) {          // rows met for the first time: into L2
          const uint16_t* nb = tensor + it.b * sb + it.h * sh + (int64_t)it.q_row0 * sn;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            prefetch_l2(nb + (int64_t)ahead[q] * sn);
            prefetch_l2(nb + (int64_t)ahead[q] * sn + 64);
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) { rows[q] = ahead[q]; l[q] = l_ahead[q]; dl[q] = dl_ahead[q]; }
      }
      HA_T_DUMP(8, (int)blockIdx.x * 8 + 7, lane == 0 && is_q)
      if (lane == 0) s_issued[warp - W_Q] = n;
      cp_async_commit();
      cp_async_wait<0>();
    } else {
      // ===================================================================================================
      // loader of the key side: V and K tiles
      // ===================================================================================================
      auto is_boxed = [&](const KtItem& it, int e) -> bool { return pl.tiles && (flash || (e >= it.n_win && !p.sample_idx)); };
      auto row_numbers = [&](const KtItem& it, int e, int (&rows)[4]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) rows[q] = item_key_row(p, it, e, 32 * q + lane, flash);
      };
      KtItem it;
      bool more = next_item(it);
      int e = more ? it.e0 : 0, rows[4] = {0, 0, 0, 0};
      uint32_t n = 0, issued = 0;      // tiles / operands of tiles (V, then K) so far
      HA_T_DECL(8)
      if (more) row_numbers(it, e, rows);
      while (more) {
        const bool boxed = is_boxed(it, e);
        const int b = it.b, hd = it.hk, row0 = it.k_row0, tile0 = row0 + (flash ? e : e - it.n_win) * TILE;
        if (++e == it.e1) { more = next_item(it); e = more ? it.e0 : 0; }
        int ahead[4] = {0, 0, 0, 0};
        if (more) row_numbers(it, e, ahead);
        bool ok = true;
        const bool fetch = !flash && more && e < it.n_win;      // the next tile's rows into L2
#pragma unroll 1
        for (int is_k = 0; is_k < 2; ++is_k) {
          HA_T_MARK(0)
          if (n >= 1 && !(ok = wait(is_k ? B_K_EMPTY : B_V_EMPTY, (n - 1) & 1))) break;
          HA_T_MARK(1)
          const uint32_t full = bar(is_k ? B_K_FULL : B_V_FULL), dst = s_base + (is_k ? OFF_K : OFF_V);
          if (boxed) {
            const int ur = __shfl_sync(0xffffffffu, tile0, 0), uh = __shfl_sync(0xffffffffu, hd, 0), ub = __shfl_sync(0xffffffffu, b, 0);
            if (elect_one()) {
              mbar_add_tx(full, 2 * TILE_B);
              tma_tile(dst, &maps.tile[is_k ? 1 : 2], 0, ur, uh, ub, full);
              tma_tile(dst + TILE_B, &maps.tile[is_k ? 1 : 2], 64, ur, uh, ub, full);
            }
            __syncwarp();
            mbar_arrive(full);
          } else {
            int r[4] = {rows[0], rows[1], rows[2], rows[3]};
            const int64_t sn = is_k ? p.k_sn : p.v_sn;
            const uint16_t* base = is_k ? (const uint16_t*)p.k + b * p.k_sb + hd * p.k_sh : (const uint16_t*)p.v + b * p.v_sb + hd * p.v_sh;
            warp_gather_tile(dst, base + (int64_t)row0 * sn, sn, 2, r, lane);
            push_copies(full);
          }
          ++issued;
          if (fetch) {
            const int64_t sn = is_k ? p.k_sn : p.v_sn;
            const uint16_t* nb = (is_k ? (const uint16_t*)p.k + it.b * p.k_sb + it.hk * p.k_sh : (const uint16_t*)p.v + it.b * p.v_sb + it.hk * p.v_sh) + (int64_t)it.k_row0 * sn;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              prefetch_l2(nb + (int64_t)ahead[q] * sn);
              prefetch_l2(nb + (int64_t)ahead[q] * sn + 64);
            }
          }
        }
        if (!ok) break;
        ++n;
#pragma unroll
        for (int q = 0; q < 4; ++q) rows[q] = ahead[q];
        HA_T_MARK(2)
      }
      HA_T_DUMP(8, (int)blockIdx.x * 8 + 3, lane == 0)
      if (lane == 0) s_issued[warp - W_Q] = issued;
      cp_async_commit();
      cp_async_wait<0>();
    }
  }
  // every role is done (or has given up); TMEM goes back
  tc_fence_before();
  __syncthreads();
  if (s_abort) {      // (nobody writes it any more)
    // What is still under way is waited for, with a limit, before TMEM goes and the CTA retires: the last tile of every slot a loader fills, each
    // MMA warp's products, stores to TMEM.  (The drain group's copies out are through.)  A CTA that gets through its items
    // has waited for all of it on the way.
    const uint32_t bar_end = smem_u32(s_item);      // (the descriptors have been used up: their place takes the MMA warps' barriers)
    if (tid < 5) mbar_init(bar_end + 8 * tid, 1);
    mbar_fence_init();
    __syncthreads();
    if (warp > W_DO) {
      const uint32_t n = s_issued[2];
      if (n >= 1) mbar_wait(bar(B_V_FULL), ((n + 1) / 2 - 1) & 1);
      if (n >= 2) mbar_wait(bar(B_K_FULL), (n / 2 - 1) & 1);
    } else if (warp >= W_Q) {
      const uint32_t n = s_issued[warp - W_Q];
      for (uint32_t back = 1; back <= NU && n >= back; ++back) mbar_wait(bar((warp == W_Q ? B_Q_FULL : B_DO_FULL) + (n - back) % NU), ((n - back) / NU) & 1);
    } else if (warp >= W_MMA) {
      mma_settle(bar_end + 8 * (warp - W_MMA));
    } else {
      tmem_st_wait();
    }
    __syncthreads();
    if (tid == 0) report_timeout(p.status, p.status_host);
  }
  if (warp == W_MMA) tmem_dealloc(tmem, 512);
}

bool tc_bwd_supported(const ha_attn_params& p);

bool kt_bwd_supported(const ha_attn_params& p) {
  if (!tc_bwd_supported(p) || p.d != 128 || p.dv != 128 || (p.flags & HA_FLAG_NO_WS)) return false;
  const int bs = (p.block_size + TILE - 1) / TILE;
  const bool hyper = p.mode == HA_MODE_HYPER;
  if (hyper && (p.flags & HA_FLAG_SMOOTH) && p.m_k % (bs * TILE) != 0) return false;
  if (p.dq_out || !p.dq_acc) return false;
  if (p.flags & HA_FLAG_BWD_KV_INIT) {          // an item holds a key tile's whole sum, unless heads share it
    if (hyper || p.kv_group > 1 || p.dk_out) return false;
  }
  if (p.dk_out)                                 // typed rows: one item holds the whole block part of its key rows
    return hyper && !(p.flags & HA_FLAG_SMOOTH) && bs == 2 && p.m_k % (2 * TILE) == 0 && p.kv_group <= 1 && p.dv_out &&
           (p.sample_size == 0 || (p.dk_sacc && p.dv_sacc));
  return p.dk_acc && p.dv_acc;
}

template <typename T, int KIND>
static int launch_kt_bwd(const ha_attn_params& p, cudaStream_t st) {
  AttnPlan pl;
  if (!plan_items(pl, p)) return HA_ERR_TOO_LARGE;
  const bool flash = p.mode == HA_MODE_FLASH;
  if (flash) {                                  // items are key tiles
    const int n_qt = (p.m_q + TILE - 1) / TILE, n_kt = (p.m_k + TILE - 1) / TILE;
    pl.pairs = n_qt == 0 ? 0 : (p.flags & HA_FLAG_CAUSAL) && n_qt < n_kt ? n_qt : n_kt;
    const long long items = (long long)p.B * p.H * p.segs_per_head * pl.pairs;
    if (items > 0x7fffffffLL) return HA_ERR_TOO_LARGE;
    pl.n_items = (int)items;
    pl.by_pairs = FastDiv(pl.pairs > 0 ? pl.pairs : 1);
  }
  if (pl.n_items == 0 || p.m_k == 0) return HA_OK;
  KtMaps maps;
  const int Hk = p.kv_group > 1 ? p.H / p.kv_group : p.H;
  const long long n_q = p.segs_per_head > 1 ? (long long)p.segs_per_head * p.span : p.q_off + p.m_q;
  const long long n_k = p.segs_per_head > 1 ? (long long)p.segs_per_head * p.span : p.k_off + p.m_k;
  const bool boxed_samples = p.sample_size > 0 && !p.sample_idx;
  pl.rows = 0;
  pl.tiles = (flash || boxed_samples) && boxes_end_with_segments(p) && encode_tile_map(&maps.tile[1], p.dtype, p.k, 128, n_k, Hk, p.B, p.k_sn, p.k_sh, p.k_sb, TILE) &&
             encode_tile_map(&maps.tile[2], p.dtype, p.v, 128, n_k, Hk, p.B, p.v_sn, p.v_sh, p.v_sb, TILE) &&
             (!flash || (encode_tile_map(&maps.tile[0], p.dtype, p.q, 128, n_q, p.H, p.B, p.q_sn, p.q_sh, p.q_sb, bkt::UQ) &&
                         encode_tile_map(&maps.tile[3], p.dtype, p.d_o, 128, n_q, p.H, p.B, p.do_sn, p.do_sh, p.do_sb, bkt::UQ)));
  int dyn_bytes;
  HA_WINDOW_BYTES(dyn_bytes, (attn_tc_bwd_kt_kernel<T, KIND>), bkt::SMEM_USED, "ha_attn_bwd kernel attributes");
  HA_SMEM_ATTR_ONCE((attn_tc_bwd_kt_kernel<T, KIND>), dyn_bytes, "ha_attn_bwd smem attribute");
  const int sms = sm_count(), grid = pl.n_items < sms ? pl.n_items : sms;
  plan_order(pl, p, grid, 4);
  launch_chained((attn_tc_bwd_kt_kernel<T, KIND>), grid, bkt::THREADS, dyn_bytes, st, p, pl, maps);
  HA_LAUNCHED("ha_attn_bwd (tcgen05, by key tiles)");
  return HA_OK;
}

int kt_attn_bwd(const ha_attn_params& p, cudaStream_t st) {
  const bool any = p.mode == HA_MODE_HYPER && ((p.flags & HA_FLAG_SMOOTH) || (p.sample_logw && p.sample_size > 0));
#define HA_BKT(TT) (any ? launch_kt_bwd<TT, KT_ANY>(p, st) : p.mode == HA_MODE_FLASH ? launch_kt_bwd<TT, KT_FLASH>(p, st) : launch_kt_bwd<TT, KT_HYPER>(p, st))
  return p.dtype == HA_BF16 ? HA_BKT(__nv_bfloat16) : HA_BKT(__half);
#undef HA_BKT
}

}  // namespace ha

HA_T_SETTER(ha_debug_set_timing_buffer_bwd_kt)
