// Persistent, warp-specialised backward on tcgen05 tensor cores + TMEM, head dims 64, bf16 / fp16: the sorted block windows + sampled
// rows (any block size; smooth windows enumerated per key tile as the reference's backward does; weighted sampling) and exact
// attention.  Replaces _bwd_permuted_block_diagonal_kernel and _bwd_sampled_col_kernel (src/hyper_attn_triton.py:399-506,
// :517-665) and the backward of src/flash_attn_triton.py:651-792.
//
// One CTA per SM walks work items; an item is a pair of query tiles of one segment and the list of key tiles they meet
// (AttnItem).  dQ of a query tile is summed over the list in TMEM and leaves once; dK / dV of a key tile are summed over the
// item's two query tiles and leave after them: complete where no other item meets the key tile (block size 256 on plain
// windows: typed rows), as an fp32 addition elsewhere.
//
// Scores are computed TRANSPOSED, lanes = keys:  S^T = K Q^T,  dP^T = V dO^T.  Then P^T and dS^T, rounded to the input
// dtype, are written back to TMEM in place and feed  dV += P^T dO  and  dK += dS^T Q  as TMEM A operands; only dS also
// goes to shared memory ([key][query] rows, an MN-major A operand) for  dQ += dS K.  A (key tile, query tile) pair is two halves of
// 64 query columns on two TMEM stages, so that the elementwise phase of one half runs underneath the tensor work of the other.
//
// Roles (768 threads):
//   * elementwise groups g = 0, 1 (128 threads each): queries 32 g .. 32 g + 31 of every half.  Both work on one half while the tensor core
//     works for the other; with a half each they met in their waits (32 x 131072: half of a group's time waiting for scores, then a
//     third).  A warp's 32 keys x 32 queries come as MMA fragments (16 x 8, two keys and two queries a thread).
//   * two drain groups (128 threads each, thread = TMEM lane): finished accumulators -> global memory, dV and dQ of query tile 0 by one, dK and
//     dQ of query tile 1 by the other.  A key tile's accumulators are wanted again right away, and with one group dK waited until
//     dV had left.  Rows that lie scattered are transposed through a staging tile and leave coalesced (typed rows, fp32
//     reductions); tiles of contiguous rows leave as TMA additions of 32 x 128 floats.
//   * five MMA warps, one product each (S^T, dP^T, dV, dK of every half, dQ of every pair), one elected lane issuing from
//     warp-uniform code.
//   * three loader warps: (Q, dO, lse, delta) of the item's query tiles, K tiles (ring of two), V tiles (ring of two); the first also
//     works out the items and publishes their descriptors.
// The roles' loops are rolled and small on purpose: the kernel this one replaced, most of it tcgen05.mma from divergent lanes, spent
// its time on instruction fetch and issue.
// What bounds it: the chain S^T -> elementwise -> dV / dK -> S^T of a stage, 3800 cycles a pair of 128 x 128, of which the tensor core is busy 1620
// (shared memory, which feeds it 6 KB an instruction of 48 cycles, about 2500).  With one piece taken out at a time (128 x 1920 rows exact causal,
// backward 278 us): no elementwise phase 218, nothing written out 238, a quarter of the MMAs 265, none of the three 108.  Measured and not
// kept: P^T handed over before dP^T is awaited, with dK out of shared memory (442 -> 459 us the step), one arrival a warp instead of a thread (no
// difference), test_wait instead of try_wait (8% slower), Q, dO and (K, V) as the loaders' shares (no difference; smooth windows 3% slower).
// TMEM columns: stage s at 128 s: S^T in [0, 64), dP^T in [64, 128); P^T / dS^T packed over the first halves of a group's 32 columns.  dV 256, dK 320, dQ of
// query tile 0 / 1 at 384 / 448.
// Hand-offs are mbarriers with bounded waits; a wait that gives up raises the CTA's abort flag, every role leaves its loop at its
// next wait, and the status words are set at the end.
#include "attn_items.cuh"

#include <type_traits>

namespace ha {

namespace bws {
constexpr int D = 64;
constexpr int TILE_B = TILE * 64 * 2;                          // one 128 x 64 tile of 2-byte elements
constexpr int OFF_K = 0;                                       // K ring (2)
constexpr int OFF_V = OFF_K + 2 * TILE_B;                      // V ring (2)
constexpr int OFF_QD = OFF_V + 2 * TILE_B;                     // query tile y of the item: Q, then dO
constexpr int OFF_DS = OFF_QD + 2 * 2 * TILE_B;                // two buffers (pairs alternate) of two slabs (halves)
constexpr int OFF_LD = OFF_DS + 2 * 2 * TILE_B;                // per query tile: lse[128], delta[128] (fp32)
constexpr int OFF_ST = OFF_LD + 2 * 1024;                      // a staging tile for each drain group: 128 rows x 128 bytes
constexpr int SMEM_USED = OFF_ST + 2 * TILE * 128;             // from the first 1 KB boundary after the static variables: all a CTA has
constexpr int THREADS = 768;
constexpr int W_DRAIN = 8, W_MMA = 16, W_QD = 21, W_K = 22;    // first warp of each role (V: 23)
constexpr int COL_DV = 256, COL_DK = 320, COL_DQ = 384;
constexpr int ND = 4, CONSUMERS = 23;                          // descriptor ring; warps that read every descriptor (all but the writer)
// barrier slots (index + stage / buffer / query tile) and their arrivals per phase
enum {
  B_K_FULL = 0,       // 2 x 32: every lane of the loader, through its copies
  B_K_EMPTY = 2,      // 2 x 2: the S^T and dQ warps
  B_V_FULL = 4,       // 2 x 32
  B_V_EMPTY = 6,      // 2 x 1: the dP^T warp
  B_QD_FULL = 8,      // 2 x 64: the loader's lanes through their copies, and for what they stored themselves
  B_QD_EMPTY = 10,    // 2 x 4: the S^T, dP^T, dV and dK warps
  B_S_READY = 12,     // 2 x 2: S^T and dP^T of a half are in TMEM
  B_P_READY = 14,     // 2 x 256: both elementwise groups have written P^T / dS^T of the half
  B_SF_S = 16,        // 2 x 1: dV of the stage's half completed: its S^T columns may be overwritten
  B_SF_P = 18,        // 2 x 1: dK ...: its dP^T columns
  B_DS_FULL = 20,     // 2 x 256: both halves' dS slabs of a pair are in the buffer
  B_DS_FREE = 22,     // 2 x 1: dQ of the pair has read them
  B_DQ_FULL = 24,     // 2 x 1: dQ of a query tile complete
  B_DQ_FREE = 26,     // 2 x 128: ... drained
  B_LDT = 28,         // (2 query tiles x 2 groups) x 128: an elementwise group has scaled the lse / delta of its own columns
  B_ACC_FULL = 32,    // 2 x 1: dV / dK of a key tile complete
  B_ACC_FREE = 34,    // 2 x 128: ... drained
  B_ST_FULL = 36,     // 2 x 128: every thread of a drain group has written its row of the staging tile
  B_ST_FREE = 38,     // 2 x 1: the copy engine has read it
  B_D_FULL = 40,      // ND x 1
  B_D_EMPTY = 40 + ND,
  N_BARS = 40 + 2 * ND
};
__device__ __forceinline__ int bar_count(int i) {
  if (i >= B_D_EMPTY) return CONSUMERS;
  if (i >= B_D_FULL) return 1;
  switch (i >> 1) {
    case B_K_FULL >> 1: case B_V_FULL >> 1: return 32;
    case B_QD_FULL >> 1: return 64;
    case B_K_EMPTY >> 1: case B_S_READY >> 1: return 2;
    case B_QD_EMPTY >> 1: return 4;
    case B_DQ_FREE >> 1: case B_LDT >> 1: case (B_LDT >> 1) + 1: case B_ACC_FREE >> 1: case B_ST_FULL >> 1: return 128;
    case B_P_READY >> 1: case B_DS_FULL >> 1: return 256;
    default: return 1;
  }
}
}  // namespace bws

struct BwdMaps { CUtensorMap tile[4], rows[2], acc[3]; };      // tiles of q, k, v, dO; rows of q, k; accumulators of dq, dv, dk
struct BwdOut {
  int bulk;           // accumulators that take TMA additions: 1 = dq, 2 = dk and dv
  int store_dq;       // fp32 dq rows are stored, not added
};
enum { BWD_HYPER = 0, BWD_FLASH = 1, BWD_ANY = 2 };            // the plain hyper pattern, exact attention, the hyper pattern with smooth windows or weights

__device__ __forceinline__ void bws_bulk_add_f32(float* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bws_bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// all but N of this thread's bulk copies have read their source / everything has completed
template <int N> __device__ __forceinline__ void bws_bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bws_bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
template <typename T, int KIND>
__global__ void __launch_bounds__(bws::THREADS, 1) attn_tc_bwd_ws_kernel(const ha_attn_params p, const AttnPlan pl, const BwdOut out,
                                                                         const __grid_constant__ BwdMaps maps) {
  chain_begin();
  using namespace bws;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t s_base = smem_u32(smem);
  __shared__ __align__(16) AttnItem s_item[ND];
  __shared__ uint64_t bars[N_BARS];
  __shared__ uint32_t tmem_slot;
  __shared__ uint32_t s_issued[4];        // query tiles 0 and 1, K tiles, V tiles that the loaders have asked for
  __shared__ int s_abort;
  __shared__ int s_bail;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  constexpr bool flash = KIND == BWD_FLASH;
  constexpr bool ANY = KIND == BWD_ANY;

  if (cta_sees_failure(p.status, &s_bail)) return;   // an earlier CTA gave up: drain quickly (uniform over the CTA)
  {
    // The layout fills the CTA's shared memory to the last byte.  Should the window start somewhere else than assumed, do nothing
    // rather than run over it.
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
  auto next_item = [&](AttnItem& it) -> bool {
    const int slot = n_item % ND;
    if (!wait(B_D_FULL + slot, (n_item / ND) & 1)) return false;
    it = s_item[slot];
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_D_EMPTY + slot));
    ++n_item;
    return it.n_list != 0;
  };
  constexpr float LOG2E = 1.4426950408889634f;

  // Register budget: 768 threads x 80 at launch = 61440 = 256 x 104 (elementwise) + 256 x 72 (drain) + 256 x 64 (the rest).
  if (warp < W_DRAIN) {
    // =====================================================================================================
    // elementwise groups: P^T = exp2(S^T scale log2e - lse log2e), dS^T = P^T (dP^T - delta) scale
    // =====================================================================================================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    const int g = warp >> 2, row = tid & 127;
    const uint32_t tG = tmem + 32 * g + ((uint32_t)((warp & 3) * 32) << 16);      // this group's columns of stage 0's S^T (dP^T: 64 further on)
    const uint64_t sc2 = pack_f2(p.scale * LOG2E, p.scale * LOG2E), scl = pack_f2(p.scale, p.scale);
    const bool causal = flash && (p.flags & HA_FLAG_CAUSAL);
    uint32_t pair = 0, n_y0 = 0, n_y1 = 0;      // pairs so far; items that had query tile 0 / 1
    bool ok = true;
    HA_T_DECL(8)
    AttnItem it;
    while (ok && next_item(it)) {
#pragma unroll 1
      for (int e = 0; e < it.n_list && ok; ++e) {
#pragma unroll 1
        for (int y = 0; y < 2 && ok; ++y) {
          if (!it.active(y, e)) continue;
          float* ld = reinterpret_cast<float*>(smem + OFF_LD + y * 1024) + 32 * g;      // lse of this group's columns; delta 128 floats on
#pragma unroll 1
          for (int s = 0; s < 2; ++s, ld += 64) {
            HA_T_MARK(0)
            if (!(ok = wait(B_S_READY + s, pair & 1))) break;
            HA_T_MARK(1)
            if (s == 0) {
              if (e == it.first_entry(y)) {
                // lse / delta of the query tile have landed: the group scales those of its columns once for all pairs of the item
                const uint32_t par = (y ? n_y1 : n_y0) & 1;
                if (!(ok = wait(B_QD_FULL + y, par))) break;
                ld[(row >> 6) * TILE + ((row >> 5) & 1) * 64 + (row & 31)] *= row < 64 ? -LOG2E : -p.scale;
                mbar_arrive(bar(B_LDT + 2 * y + g));
                if (!(ok = wait(B_LDT + 2 * y + g, par))) break;
              }
              if (pair >= 2 && !(ok = wait(B_DS_FREE + (pair & 1), ((pair >> 1) - 1) & 1))) break;   // dQ of pair - 2 has read the buffer
            }
            HA_T_MARK(2)
            tc_fence_after();
            float bias2 = 0.f;
            const bool weighted = ANY && !flash && p.sample_logw && e >= it.n_win;
            const uint32_t* drop = nullptr;
            if (weighted) {
              int pos = it.q_pos0 + y * TILE + 64 * s;
              if (pos >= p.m_q) pos -= p.m_q;
              const long long qtile = (long long)it.seg * (p.m_q / TILE) + pos / TILE;
              bias2 = p.sample_logw[qtile] * LOG2E;
              drop = p.sample_mask + qtile * (p.sample_size / 32) + (e - it.n_win) * (TILE / 32) + (warp & 3);
            }
            const bool diag = causal && e == it.qt0 + y, masked = KIND != BWD_HYPER && (weighted || diag || (flash && (e + 1) * TILE > p.m_k));
            const uint64_t bias = pack_f2(bias2, bias2);
            const uint32_t tS = tG + 128 * s, tDP = tS + 64;
            uint8_t* ds_rows = smem + OFF_DS + (pair & 1) * 2 * TILE_B + s * TILE_B + (32 * (warp & 3) + (lane & 7)) * 128;
            // Two keys and two neighbouring queries a fragment and thread: it needs the lse and delta of 8 queries.  With a key a thread it needed
            // those of all 32, and the broadcast reads, four cycles of the shared memory each, held up the tensor core's operands: exact causal 128 x 1920
            // rows 458 -> 442 us (step), 16 x 12287 934 -> 894, smooth 32 x 16384 642 -> 621, 32 x 131072 3398 -> 3256.
            const uint32_t ds_to = smem_u32(ds_rows) + (((4 * g + (lane >> 3)) ^ (lane & 7)) << 4);
            uint64_t L[4], Dl[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              L[j] = *reinterpret_cast<const uint64_t*>(ld + 8 * j + 2 * (lane & 3));
              Dl[j] = *reinterpret_cast<const uint64_t*>(ld + TILE + 8 * j + 2 * (lane & 3));
              if (ANY) L[j] = fadd2(L[j], bias);
            }
#pragma unroll 2
            for (int h = 0; h < 2; ++h) {
              uint32_t rs[16], rp[16], pk[8], dk[8];
              tmem_ld_16x256(tS + (h << 20), rs);
              tmem_ld_16x256(tDP + (h << 20), rp);
              tmem_ld_fence16(rs);
              tmem_ld_fence16(rp);
              // queries [0, hidden) of the group's do not count for a key row
              int hidden[2] = {0, 0};
              if (masked) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                  const int row = 32 * (warp & 3) + 16 * h + 8 * k + (lane >> 2);
                  if (flash) {
                    if (diag) hidden[k] = row - 64 * s - 32 * g;               // queries before the key
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
              // P^T / dS^T (16 packed columns) over columns this warp has consumed
              tmem_st_16x128(tS + (h << 20), pk);
              tmem_st_16x128(tDP + (h << 20), dk);
#pragma unroll
              for (int k = 0; k < 2; ++k) store_matrix_x4(ds_to + (16 * h + 8 * k) * 128, dk[k], dk[2 + k], dk[4 + k], dk[6 + k]);
            }
            HA_T_MARK(3)
            tmem_st_wait();
            fence_async_smem();       // the dS rows are read by the tensor core (async proxy)
            tc_fence_before();
            mbar_arrive(bar(B_P_READY + s));
            // The dQ warp follows the dS buffers, not the TMEM stages: it may run up to two pairs behind this thread, and a parity wait
            // must never fall two phases behind its barrier; the buffer's own barrier cannot run ahead of it.
            if (s == 1) mbar_arrive(bar(B_DS_FULL + (pair & 1)));
            HA_T_MARK(4)
          }
          ++pair;
        }
      }
      ++n_y0;
      n_y1 += it.has1;
    }
    HA_T_DUMP(8, (int)blockIdx.x * 8 + g, row == 0)
  } else if (warp < W_MMA) {
    // =====================================================================================================
    // drain groups: finished accumulators -> global memory
    // =====================================================================================================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    const int row = tid & 127, rot = row & 7, grp = (warp - W_DRAIN) >> 2;
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_stage = OFF_ST + grp * (TILE * 128);   // scattered rows: the warp's own 4 KB
    uint8_t* my_row = smem + s_stage + row * 128;
    const uint8_t* warp_rows = smem + s_stage + (row & ~31) * 128;
    uint32_t n_kt = 0, n_y = 0;                             // key tiles / query tiles drained so far
    uint32_t ops = 0;                                       // tile additions issued
    bool reading = false;                                   // the last of them may still be reading the staging tile
    bool ok = true;
    HA_T_DECL(8)
    AttnItem it;
    while (ok && next_item(it)) {
      const int Hk = p.kv_group > 1 ? pl.by_group(p.H) : p.H;
#pragma unroll 1
      for (int e = 0; e < it.n_list && ok; ++e) {
        // dV (dK) of the key tile, then dQ of query tile 0 (1) if the tile was its last
#pragma unroll 1
        for (int is_q = 0; is_q < 2; ++is_q) {
          if (is_q && ((grp && !it.has1) || e != it.last_entry(grp))) continue;
          HA_T_MARK(0)
          // where this lane's row goes, and how
          enum { TYPED, ROWS_ADD, ROWS_STORE, TILE_ADD, TILE_STORE, SLOTS };
          int mode, local, full, free_bar, map, tile_row;
          uint32_t par, taddr;
          T* typed;
          float* acc;
          const bool sampled = !flash && e >= it.n_win;
          if (is_q) {
            int pos = it.q_pos0 + grp * TILE + row;
            if (pos >= p.m_q && !flash) pos -= p.m_q;
            local = flash ? (pos < p.m_q ? pos : -1) : p.q_idx[(long long)it.seg * p.m_q + pos];
            if (local >= 0) local += it.q_row0;
            map = 0;
            tile_row = it.q_row0 + it.q_pos0 + grp * TILE;
            typed = (T*)p.dq_out;
            acc = p.dq_acc;
            mode = p.dq_out ? TYPED : flash && (out.bulk & 1) ? (out.store_dq ? TILE_STORE : TILE_ADD) : out.store_dq ? ROWS_STORE : ROWS_ADD;
            full = B_DQ_FULL + grp;
            free_bar = B_DQ_FREE + grp;
            par = n_y & 1;
            taddr = COL_DQ + 64 * grp;
          } else {
            local = item_key_row(p, it, e, row, flash);
            if (local >= 0) local += it.k_row0;
            map = 1 + grp;                                        // (accumulator maps: dq, dv, dk)
            tile_row = it.k_row0 + (flash ? e : e - it.n_win) * TILE;
            typed = (T*)(grp ? p.dk_out : p.dv_out);
            acc = grp ? p.dk_acc : p.dv_acc;
            if (p.dk_out) {
              mode = sampled ? SLOTS : TYPED;
              if (sampled) acc = (grp ? p.dk_sacc : p.dv_sacc) + ((long long)it.kseg * p.sample_size + (e - it.n_win) * TILE) * D;
            } else {
              mode = (out.bulk & 2) && (flash || (sampled && !p.sample_idx)) ? TILE_ADD : ROWS_ADD;
            }
            full = B_ACC_FULL + grp;
            free_bar = B_ACC_FREE + grp;
            par = n_kt & 1;
            taddr = grp ? COL_DK : COL_DV;
          }
          const int head = is_q ? it.b * p.H + it.h : it.b * Hk + it.hk;
          const bool by_tile = mode >= TILE_ADD;
          HA_T_MARK(1)
          if (!(ok = wait(full, par))) break;
          HA_T_MARK(2)
          tc_fence_after();
#pragma unroll 1
          for (int hf = 0; hf < 2; ++hf) {
            uint32_t r[32];
            tmem_ld32(tmem + taddr + hf * 32 + lane_sel, r);
            tmem_ld_fence(r);
            if (hf == 1) {
              tc_fence_before();
              mbar_arrive(bar(free_bar));
            }
            if (reading) {
              if (row == 0) {
                bws_bulk_wait_read<0>();
                mbar_arrive(bar(B_ST_FREE + grp));
              }
              __syncwarp();
              if (!(ok = wait(B_ST_FREE + grp, (ops - 1) & 1))) break;
              reading = false;
            }
            if (mode == TYPED) {
              // both halves of a row fill its 128 bytes
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                uint32_t w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) w[j] = pack2<T>(__uint_as_float(r[8 * i + 2 * j]), __uint_as_float(r[8 * i + 2 * j + 1]));
                *reinterpret_cast<uint4*>(my_row + (((hf * 4 + i) ^ rot) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
              }
              if (hf == 0) continue;
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(my_row + ((i ^ rot) << 4)) = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
            }
            if (by_tile) {
              fence_async_smem();
              mbar_arrive(bar(B_ST_FULL + grp));
              if (warp == W_DRAIN + 4 * grp) {
                if (!(ok = wait(B_ST_FULL + grp, ops & 1))) break;
                if (lane == 0) {
                  const uint32_t src = s_base + s_stage;
                  if (mode == SLOTS) bws_bulk_add_f32(acc + hf * (TILE * 32), src, TILE * 128);
                  else if (mode == TILE_ADD) tma_add_tile(&maps.acc[map], hf * 32, tile_row, head, src);
                  else tma_store_tile(&maps.acc[map], hf * 32, tile_row, head, src);
                  bws_bulk_commit();
                }
                __syncwarp();
              }
              reading = true;
              ++ops;
            } else {
              // eight lanes cover the 128 contiguous bytes of a row
              __syncwarp();
              const int c = lane & 7;
              if (KIND != BWD_FLASH && mode == ROWS_ADD) {
                // all reads, then all additions: a branch a row made smooth windows (32 heads x 16384) 7% slower.  Typed rows measured the
                // other way round (2.22 against 2.28 ms at 32 x 131072), and exact attention, whose tiles rarely leave this way, is
                // faster without this branch (4.46 against 4.50 ms, leaves of 32 x 131072).
                float4 v[8];
                int to[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const int rl = 4 * j + (lane >> 3);
                  v[j] = *reinterpret_cast<const float4*>(warp_rows + rl * 128 + ((c ^ (rl & 7)) << 4));
                  to[j] = __shfl_sync(0xffffffffu, local, rl);
                }
                float* dst_rows = acc + (long long)head * p.n * D + hf * 32 + c * 4;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                  if (to[j] >= 0) red_add_v4(dst_rows + (long long)to[j] * D, v[j]);
              } else {
                const long long row0 = (long long)head * p.n;
#pragma unroll 2
                for (int j = 0; j < 8; ++j) {
                  const int rl = 4 * j + (lane >> 3);
                  const float4 v = *reinterpret_cast<const float4*>(warp_rows + rl * 128 + ((c ^ (rl & 7)) << 4));
                  const int to = __shfl_sync(0xffffffffu, local, rl);
                  if (to >= 0) {
                    if (mode == TYPED) *reinterpret_cast<float4*>(typed + (row0 + to) * D + c * 8) = v;
                    else if (mode == ROWS_ADD) red_add_v4(acc + (row0 + to) * D + hf * 32 + c * 4, v);
                    else *reinterpret_cast<float4*>(acc + (row0 + to) * D + hf * 32 + c * 4) = v;
                  }
                }
              }
              __syncwarp();
            }
          }
          if (!ok) break;
          HA_T_MARK(3)
          if (is_q) ++n_y;
          else ++n_kt;
        }
      }
    }
    bws_bulk_wait_all();       // nothing of this thread is in flight when the CTA retires
    HA_T_DUMP(8, (int)blockIdx.x * 8 + 2, row == 0 && grp == 0)
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    if (warp < W_QD) {
      // ===================================================================================================
      // MMA issue, one warp per product.  Each walks the pairs of the items in order and waits (bounded) for what its next
      // instructions need.  The "empty" barriers of the operand tiles collect one commit from every warp that reads them.
      // ===================================================================================================
      constexpr int AB = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
      const int role = warp - W_MMA;            // 0: S^T, 1: dP^T, 2: dV, 3: dK, 4: dQ
      uint32_t pair = 0, kt = 0;                // pairs / key tiles so far
      uint32_t n_y0 = 0, n_y1 = 0;              // items that had query tile 0 / 1
      bool ok = true;
      HA_T_DECL(8)
      AttnItem it;
      while (ok && next_item(it)) {
        const int first0 = it.first_entry(0), first1 = it.first_entry(1), last0 = it.last_entry(0), last1 = it.last_entry(1);
#pragma unroll 1
        for (int e = 0; e < it.n_list && ok; ++e, ++kt) {
          HA_T_MARK(0)
          if (role < 2 && !(ok = wait((role ? B_V_FULL : B_K_FULL) + (kt & 1), (kt >> 1) & 1))) break;
          if (role < 2) fence_async_smem();     // (tiles that came by cp.async)
          HA_T_MARK(1)
          bool fresh = true;                    // nothing accumulated yet for this key tile
#pragma unroll 1
          for (int y = 0; y < 2; ++y) {
            if (!it.active(y, e)) continue;
            const bool last = e == (y ? last1 : last0), y_first = e == (y ? first1 : first0);
            const uint32_t n_y = y ? n_y1 : n_y0, sQD = s_base + OFF_QD + y * 2 * TILE_B;
            if (role < 2) {
              // S^T = K Q^T / dP^T = V dO^T of both halves: M = 128 keys, N = 64 query rows, both operands K-major
              if (y_first) {
                if (!(ok = wait(B_QD_FULL + y, n_y & 1))) break;
                fence_async_smem();
              }
              const uint32_t idesc = mma_idesc(TILE, 64, AB, 0, 0);
              const uint64_t dA = smem_desc(s_base + (role ? OFF_V : OFF_K) + (kt & 1) * TILE_B, 16, 1024), dB = smem_desc(sQD + role * TILE_B, 16, 1024);
#pragma unroll
              for (int s = 0; s < 2; ++s) {
                // the product that read P^T (dS^T) out of these columns has completed
                if (pair >= 1 && !(ok = wait((role ? B_SF_P : B_SF_S) + s, (pair - 1) & 1))) break;
                HA_T_MARK(2)
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                  for (int kk = 0; kk < 4; ++kk)
                    mma_ss(tmem + 128 * s + role * 64, dA + kk * (32 >> 4), dB + s * (TILE_B / 2 >> 4) + kk * (32 >> 4), idesc, kk > 0);
                  mma_commit(bar(B_S_READY + s));
                  if (s == 1 && last) mma_commit(bar(B_QD_EMPTY + y));
                }
                __syncwarp();
                HA_T_MARK(3)
              }
              if (!ok) break;
            } else if (role < 4) {
              // dV += P^T dO / dK += dS^T Q of both halves: A in TMEM, B rows as MN-major
              const uint32_t idesc = mma_idesc(TILE, 64, AB, 0, 1);
              const int is_k = role - 2;
              const uint64_t dB = smem_desc(sQD + (is_k ? 0 : TILE_B), TILE * 128, 1024);
              const bool tile_done = y == 1 || !it.active(1, e);
#pragma unroll
              for (int s = 0; s < 2; ++s) {
                if (!(ok = wait(B_P_READY + s, pair & 1))) break;
                if (s == 0 && y_first) fence_async_smem();
                if (s == 0 && fresh && kt >= 1 && !(ok = wait(B_ACC_FREE + is_k, (kt - 1) & 1))) break;    // the accumulator restarts with the key tile
                HA_T_MARK(2)
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                  for (int kk = 0; kk < 4; ++kk)
                    mma_ts(tmem + (is_k ? COL_DK : COL_DV), tmem + 128 * s + is_k * 64 + (kk >> 1) * 32 + (kk & 1) * 8, dB + s * (TILE_B / 2 >> 4) + kk * (2048 >> 4), idesc,
                           !fresh | (s + kk > 0));
                  mma_commit(bar((is_k ? B_SF_P : B_SF_S) + s));
                  if (s == 1 && tile_done) mma_commit(bar(B_ACC_FULL + is_k));
                  if (s == 1 && last) mma_commit(bar(B_QD_EMPTY + y));
                }
                __syncwarp();
                HA_T_MARK(3)
              }
              if (!ok) break;
            } else {
              // dQ_y += dS K over the pair's 128 keys: A = dS ([key][query] rows: MN-major), B = K rows as MN-major
              const uint32_t idesc = mma_idesc(TILE, 64, AB, 1, 1);
              if (!(ok = wait(B_DS_FULL + (pair & 1), (pair >> 1) & 1))) break;
              fence_async_smem();
              if (y_first && n_y >= 1 && !(ok = wait(B_DQ_FREE + y, (n_y - 1) & 1))) break;      // dQ restarts with the item
              HA_T_MARK(2)
              tc_fence_after();
              const uint64_t dA = smem_desc(s_base + OFF_DS + (pair & 1) * 2 * TILE_B, TILE_B, 1024), dB = smem_desc(s_base + OFF_K + (kt & 1) * TILE_B, TILE_B, 1024);
              if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) mma_ss(tmem + COL_DQ + y * D, dA + kk * (2048 >> 4), dB + kk * (2048 >> 4), idesc, !y_first | (kk > 0));
                mma_commit(bar(B_DS_FREE + (pair & 1)));
                if (last) mma_commit(bar(B_DQ_FULL + y));
              }
              __syncwarp();
              HA_T_MARK(3)
            }
            fresh = false;
            ++pair;
          }
          if (ok && (role == 0 || role == 1 || role == 4) && elect_one())
            mma_commit(bar((role == 1 ? B_V_EMPTY : B_K_EMPTY) + (kt & 1)));       // this warp's last read of the tile
          __syncwarp();
          HA_T_MARK(4)
        }
        ++n_y0;
        n_y1 += it.has1;
      }
      HA_T_DUMP(8, (int)blockIdx.x * 8 + (role == 0 ? 4 : role == 2 ? 5 : 6), lane == 0 && !(role & 1))
    } else if (warp == W_QD) {
      // ===================================================================================================
      // scheduler, loader of the query side: per query tile Q, dO, lse, delta
      // ===================================================================================================
      const bool by_keys = ANY && (p.flags & HA_FLAG_SMOOTH);
      const bool boxed = flash && pl.tiles, gathered = !boxed && (pl.rows & 1);
      int published = 0;
      auto take = [&](AttnItem& it) -> bool {        // the next item's descriptor; n_list = 0 past the last one
#pragma unroll 1
        for (; published <= (int)n_item + 2; ++published) {
          const uint32_t slot = published % ND;
          it.n_list = 0;
          const int item = item_of_turn<KIND == BWD_FLASH>(pl, published, blockIdx.x, gridDim.x);
          if (item < pl.n_items) it = attn_item(p, pl, item, flash, by_keys);
          if (published >= ND && !wait(B_D_EMPTY + slot, (published / ND - 1) & 1)) return false;
          if (lane == 0) {
            s_item[slot] = it;
            mbar_arrive(bar(B_D_FULL + slot));
          }
          __syncwarp();
        }
        it = s_item[n_item % ND];
        ++n_item;
        return it.n_list != 0;
      };
      auto row_numbers = [&](const AttnItem& it, int y, int (&rows)[4]) {
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
      uint32_t n_y0 = 0, n_y1 = 0;
      bool ok = true;
      HA_T_DECL(8)
      AttnItem it;
      int rows[4];
      bool more = take(it);
      if (more) row_numbers(it, 0, rows);
      int y = 0;
      while (more && ok) {
        const AttnItem me = it;
        const int my = y;
        // the next tile's row numbers travel during the wait
        int ahead[4] = {0, 0, 0, 0};
        if (y == 0 && it.has1) y = 1;
        else { y = 0; more = take(it); }
        if (more) row_numbers(it, y, ahead);
        const uint32_t n_y = my ? n_y1 : n_y0;
        HA_T_MARK(0)
        if (n_y >= 1 && !(ok = wait(B_QD_EMPTY + my, (n_y - 1) & 1))) break;
        HA_T_MARK(1)
        const uint32_t full = bar(B_QD_FULL + my), dst = s_base + OFF_QD + my * 2 * TILE_B;
        const uint16_t* gbase = (const uint16_t*)p.d_o + me.b * p.do_sb + me.h * p.do_sh + (int64_t)me.q_row0 * p.do_sn;
        if (boxed) {
          const int ur = __shfl_sync(0xffffffffu, me.q_row0 + me.q_pos0 + my * TILE, 0), uh = __shfl_sync(0xffffffffu, me.h, 0), ub = __shfl_sync(0xffffffffu, me.b, 0);
          if (elect_one()) {
            mbar_add_tx(full, 2 * TILE_B);
            tma_tile(dst, &maps.tile[0], 0, ur, uh, ub, full);
            tma_tile(dst + TILE_B, &maps.tile[3], 0, ur, uh, ub, full);
          }
          __syncwarp();
        } else {
          if (gathered) {
            // lane l takes rows 4 l .. 4 l + 3, whose numbers are with lanes 4 (l & 7) + q, word l / 8
            const int step = pl.row_sn[0], base = me.b * pl.row_sb[0] + me.h * pl.row_sh[0] + me.q_row0 * step;
            int r4[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int from = 4 * (lane & 7) + q;
              const int a = __shfl_sync(0xffffffffu, rows[0], from), b = __shfl_sync(0xffffffffu, rows[1], from), c = __shfl_sync(0xffffffffu, rows[2], from),
                        d = __shfl_sync(0xffffffffu, rows[3], from);
              r4[q] = base + (lane < 8 ? a : lane < 16 ? b : lane < 24 ? c : d) * step;
            }
            mbar_add_tx(full, 512);
            tma_gather4(dst + lane * 512, &maps.rows[0], 0, r4[0], r4[1], r4[2], r4[3], full);
          }
#pragma unroll 1
          for (int x = gathered ? 1 : 0; x < 2; ++x) {
            int r[4] = {rows[0], rows[1], rows[2], rows[3]};
            warp_gather_tile(dst + x * TILE_B, x ? gbase : (const uint16_t*)p.q + me.b * p.q_sb + me.h * p.q_sh + (int64_t)me.q_row0 * p.q_sn, x ? p.do_sn : p.q_sn, 1, r, lane);
          }
        }
        {
          const long long at = ((long long)(me.b * p.H + me.h)) * p.n + me.q_row0;
          float* ld = reinterpret_cast<float*>(smem + OFF_LD + my * 1024);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int r = q * 32 + lane;
            if (rows[q] >= 0) {
              cp_async4(smem_u32(ld + r), p.lse + at + rows[q]);
              cp_async4(smem_u32(ld + TILE + r), p.delta + at + rows[q]);
            } else {           // no such query: P = 0
              ld[r] = INFINITY;
              ld[TILE + r] = 0.f;
            }
          }
        }
        push_copies(full);
        mbar_arrive(full);       // (the copies' arrivals publish the copies only, not the values of absent rows stored above)
        // the next tile's dO rows into L2 (Q's copies do not mind the latency)
        if (!flash && more) {
          const uint16_t* nb = (const uint16_t*)p.d_o + it.b * p.do_sb + it.h * p.do_sh + (int64_t)it.q_row0 * p.do_sn;
#pragma unroll
          for (int q = 0; q < 4; ++q) prefetch_l2(nb + (int64_t)ahead[q] * p.do_sn);
        }
        if (my) ++n_y1;
        else ++n_y0;
#pragma unroll
        for (int q = 0; q < 4; ++q) rows[q] = ahead[q];
        HA_T_MARK(2)
      }
      HA_T_DUMP(8, (int)blockIdx.x * 8 + 7, lane == 0)
      if (lane == 0) { s_issued[0] = n_y0; s_issued[1] = n_y1; }
      cp_async_commit();
      cp_async_wait<0>();
    } else {
      // ===================================================================================================
      // loaders of the key side: K tiles (warp W_K), V tiles (the warp after it)
      // ===================================================================================================
      const bool is_v = warp != W_K;
      const uint16_t* tensor = (const uint16_t*)(is_v ? p.v : p.k);
      const int64_t sb = is_v ? p.v_sb : p.k_sb, sh = is_v ? p.v_sh : p.k_sh, sn = is_v ? p.v_sn : p.k_sn;
      const bool by_rows = !is_v && (pl.rows & 2);
      auto is_boxed = [&](const AttnItem& it, int e) -> bool { return pl.tiles && (flash || (e >= it.n_win && !p.sample_idx)); };
      auto row_numbers = [&](const AttnItem& it, int e, int (&rows)[4]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) rows[q] = item_key_row(p, it, e, by_rows ? 4 * lane + q : 32 * q + lane, flash);
      };
      HA_T_DECL(8)
      AttnItem it;
      bool more = next_item(it);
      int e = 0, rows[4] = {0, 0, 0, 0};
      uint32_t n = 0;
      if (more && !is_boxed(it, 0)) row_numbers(it, 0, rows);
      while (more) {
        const bool boxed = is_boxed(it, e);
        const int b = it.b, hd = it.hk, row0 = it.k_row0, tile0 = row0 + (flash ? e : e - it.n_win) * TILE;
        if (++e == it.n_list) { e = 0; more = next_item(it); }
        int ahead[4] = {0, 0, 0, 0};
        if (more && !is_boxed(it, e)) row_numbers(it, e, ahead);
        const uint32_t slot = n & 1, dst = s_base + (is_v ? OFF_V : OFF_K) + slot * TILE_B, full = bar((is_v ? B_V_FULL : B_K_FULL) + slot);
        HA_T_MARK(0)
        if (n >= 2 && !wait((is_v ? B_V_EMPTY : B_K_EMPTY) + slot, ((n >> 1) - 1) & 1)) break;
        HA_T_MARK(1)
        if (boxed) {
          const int ur = __shfl_sync(0xffffffffu, tile0, 0), uh = __shfl_sync(0xffffffffu, hd, 0), ub = __shfl_sync(0xffffffffu, b, 0);
          if (elect_one()) {
            mbar_add_tx(full, TILE_B);
            tma_tile(dst, &maps.tile[is_v ? 2 : 1], 0, ur, uh, ub, full);
          }
          __syncwarp();
          mbar_arrive(full);
        } else if (by_rows) {
          const int step = pl.row_sn[1], base = b * pl.row_sb[1] + hd * pl.row_sh[1] + row0 * step;
          mbar_expect_tx(full, 512);       // this lane's four rows
          tma_gather4(dst + lane * 512, &maps.rows[1], 0, base + rows[0] * step, base + rows[1] * step, base + rows[2] * step, base + rows[3] * step, full);
        } else {
          warp_gather_tile(dst, tensor + b * sb + hd * sh + (int64_t)row0 * sn, sn, 1, rows, lane);
          push_copies(full);
          if (!flash && more && !is_boxed(it, e) && e < it.n_win) {
            const uint16_t* nb = tensor + it.b * sb + it.hk * sh + (int64_t)it.k_row0 * sn;
#pragma unroll
            for (int q = 0; q < 4; ++q) prefetch_l2(nb + (int64_t)ahead[q] * sn);
          }
        }
        ++n;
#pragma unroll
        for (int q = 0; q < 4; ++q) rows[q] = ahead[q];
        HA_T_MARK(2)
      }
      HA_T_DUMP(8, (int)blockIdx.x * 8 + 3, lane == 0 && !is_v)
      if (lane == 0) s_issued[2 + is_v] = n;
      cp_async_commit();
      cp_async_wait<0>();
    }
  }
  // every role is done (or has given up); TMEM goes back
  tc_fence_before();
  __syncthreads();
  if (s_abort) {      // (nobody writes it any more)
    // What is still under way is waited for, with a limit, before TMEM goes and the CTA retires: the last tile of every slot a loader fills, each
    // MMA warp's products, stores to TMEM.  (The drain groups' copies out are through.)  A CTA that gets through its items
    // has waited for all of it on the way.
    const uint32_t bar_end = smem_u32(s_item);      // (the descriptors have been used up: their place takes the MMA warps' barriers)
    if (tid < 5) mbar_init(bar_end + 8 * tid, 1);
    mbar_fence_init();
    __syncthreads();
    if (warp == W_QD) {
      for (int y = 0; y < 2; ++y)
        if (s_issued[y] > 0) mbar_wait(bar(B_QD_FULL + y), (s_issued[y] - 1) & 1);
    } else if (warp > W_QD) {
      const uint32_t n = s_issued[warp - W_QD + 1];
      for (uint32_t back = 1; back <= 2 && n >= back; ++back) mbar_wait(bar((warp == W_K ? B_K_FULL : B_V_FULL) + ((n - back) & 1)), ((n - back) >> 1) & 1);
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

// Does one item hold the whole block part of its key rows (plain windows over whole blocks of two tiles)?
static bool owns_key_rows(const ha_attn_params& p) {
  return p.mode == HA_MODE_HYPER && !(p.flags & HA_FLAG_SMOOTH) && (p.block_size + TILE - 1) / TILE == 2 && p.m_k % (2 * TILE) == 0;
}
static bool ws_bwd_shape(const ha_attn_params& p) {
  if (!tc_bwd_supported(p) || p.d != 64 || p.dv != 64) return false;
  if (p.flags & (HA_FLAG_NO_WS | HA_FLAG_BWD_KV_INIT)) return false;      // (key rows are added to by several items)
  const int bs = (p.block_size + TILE - 1) / TILE;
  return !(p.mode == HA_MODE_HYPER && (p.flags & HA_FLAG_SMOOTH) && p.m_k % (bs * TILE) != 0);
}
// Every gradient row may be written once, in the tensors' dtype.
bool ws_bwd_direct_ok(const ha_attn_params& p) { return ws_bwd_shape(p) && owns_key_rows(p); }
bool ws_bwd_supported(const ha_attn_params& p) {
  if (!ws_bwd_shape(p) || (!p.dq_out && !p.dq_acc)) return false;
  if (p.dk_out) return owns_key_rows(p) && p.dv_out && (p.sample_size == 0 || (p.dk_sacc && p.dv_sacc));
  return p.dk_acc && p.dv_acc;
}

template <typename T, int KIND>
static int launch_ws_bwd(const ha_attn_params& p, bool store_dq, cudaStream_t st) {
  AttnPlan pl;
  if (!plan_items(pl, p)) return HA_ERR_TOO_LARGE;
  if (pl.n_items == 0 || p.m_k == 0) return HA_OK;
  BwdMaps maps;
  BwdOut out;
  const int Hk = p.kv_group > 1 ? p.H / p.kv_group : p.H;
  const long long n_q = p.segs_per_head > 1 ? (long long)p.segs_per_head * p.span : p.q_off + p.m_q;
  const long long n_k = p.segs_per_head > 1 ? (long long)p.segs_per_head * p.span : p.k_off + p.m_k;
  const bool flash = p.mode == HA_MODE_FLASH, boxed_samples = p.sample_size > 0 && !p.sample_idx;
  pl.tiles = (flash || boxed_samples) && boxes_end_with_segments(p) && encode_tile_map(&maps.tile[1], p.dtype, p.k, 64, n_k, Hk, p.B, p.k_sn, p.k_sh, p.k_sb, TILE) &&
             encode_tile_map(&maps.tile[2], p.dtype, p.v, 64, n_k, Hk, p.B, p.v_sn, p.v_sh, p.v_sb, TILE) &&
             (!flash || (encode_tile_map(&maps.tile[0], p.dtype, p.q, 64, n_q, p.H, p.B, p.q_sn, p.q_sh, p.q_sb, TILE) &&
                         encode_tile_map(&maps.tile[3], p.dtype, p.d_o, 64, n_q, p.H, p.B, p.do_sn, p.do_sh, p.do_sb, TILE)));
  plan_row_maps(pl, p, maps.rows, n_q, n_k);
  out.bulk = 0;
  if (flash && !p.dq_out && (!store_dq || p.m_q % TILE == 0) && encode_acc_map(&maps.acc[0], p.dq_acc, 64, p.n, (long long)p.B * p.H)) out.bulk |= 1;
  if (!p.dk_out && (flash || boxed_samples) && encode_acc_map(&maps.acc[1], p.dv_acc, 64, p.n, (long long)p.B * Hk) &&
      encode_acc_map(&maps.acc[2], p.dk_acc, 64, p.n, (long long)p.B * Hk))
    out.bulk |= 2;
  out.store_dq = store_dq;
  int dyn_bytes;
  HA_WINDOW_BYTES(dyn_bytes, (attn_tc_bwd_ws_kernel<T, KIND>), bws::SMEM_USED, "ha_attn_bwd kernel attributes");
  HA_SMEM_ATTR_ONCE((attn_tc_bwd_ws_kernel<T, KIND>), dyn_bytes, "ha_attn_bwd smem attribute");
  const int sms = sm_count(), grid = pl.n_items < sms ? pl.n_items : sms;
  plan_order(pl, p, grid, 4);
  launch_chained((attn_tc_bwd_ws_kernel<T, KIND>), grid, bws::THREADS, dyn_bytes, st, p, pl, out, maps);
  HA_LAUNCHED("ha_attn_bwd (tcgen05, warp-specialised)");
  return HA_OK;
}

// store_dq: dq_acc holds garbage; every query row of every segment is stored (nothing else may add to it in this launch: an item
// holds a query row's whole sum).
int ws_attn_bwd(const ha_attn_params& p, bool store_dq, cudaStream_t st) {
  const bool any = p.mode == HA_MODE_HYPER && ((p.flags & HA_FLAG_SMOOTH) || (p.sample_logw && p.sample_size > 0));
#define HA_BWS(TT) \
  (any ? launch_ws_bwd<TT, BWD_ANY>(p, store_dq, st)                                                    \
       : p.mode == HA_MODE_FLASH ? launch_ws_bwd<TT, BWD_FLASH>(p, store_dq, st) : launch_ws_bwd<TT, BWD_HYPER>(p, store_dq, st))
  return p.dtype == HA_BF16 ? HA_BWS(__nv_bfloat16) : HA_BWS(__half);
#undef HA_BWS
}

}  // namespace ha

HA_T_SETTER(ha_debug_set_timing_buffer_bwd_ws)
