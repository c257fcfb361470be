// Varlen causal / sliding-window flash attention forward for head_dim 64, bf16, on tcgen05.
//
// Persistent CTAs (two per SM) walk a heaviest-first list of (128-row query tile, query head) items. Roles:
//   warps 0..7  softmax: two threads per query row (64 key columns each); read S from TMEM, online
//               softmax in fp32, write P (bf16) back to TMEM, rescale the O accumulator when the max moves
//   warp 8      TMA producer: Q per item, K and V tiles through two-stage rings (runs ahead into the next item)
//   warp 9      issues tcgen05.mma:  S = Q K^T (smem x smem)  and  O += P V (TMEM x smem)
// TMEM columns: S [0,128) fp32, P [128,192) packed bf16, O [192,256) fp32. Two CTAs fit per SM, so
// one CTA's softmax overlaps the other's tensor-core work.
//
// The next tile's scores are formed as soon as this tile's are in registers (half of them stay there from the maximum
// pass), under its exponentials. Formed only after P was written they were waited for by every tile: 4096-token packs
// 53.3 -> 50.5 us, 16384 tokens with a window of 1024 227 -> 218; one long document is bound by the exponentials either
// way (1316 us, 735 of them at the special-function rate, 1068 without them).
//
// SPLIT (cached prefill and other padded batches, which keep 32-bit probabilities): P leaves the softmax as three bf16
// numbers, its rounding, the rounding of what that left out, and the rest: 8 + 8 + 8 bits hold an fp32 number exactly,
// and O += P V runs once for each. The two lower parts overwrite score columns that the same thread has read, so their
// products are issued before the next tile's scores and the high one after them: the tensor pipe stays ahead of the
// softmax, which is the bound. On sums that cancel, two parts (16 bits) were 10 to 20 times as far from 64 bits as the
// explicit fp32 form; three are nearer than it inside one key tile, and 2e-7 of the sum of magnitudes off over 3001
// keys (2e-8 the explicit form), where the tensor pipe's own fp32 sums are what is left. On ordinary values both forms'
// errors are the output's bf16 rounding and agree to 1e-6. The third part costs two prompts of 3001 tokens 0.55 of 10.0
// ms. The rows of a padded batch are documents of one length, and their tiles are loaded through maps with the row as a
// dimension of its own: what lies past a row's end reads as zero. Read on into the next row, its values would meet
// probabilities of zero, and a NaN or infinity among them (0 x inf) would enter the sums of this row.
//
// Documents never attend across their boundary: a tile's key range is clipped to its own document
// and (with a window) to the last `window` positions. Sinks enter as sink_lse[h] = logsumexp of the
// head's sink logits: the stored lse is logaddexp(lse, sink_lse) and the output is scaled to match.
// Replaces src/kohakuwullm/kernels/attention/flash_attn_fwd.py:35-154 and the vendor FA2 call at
// src/kohakuwullm/models/components/attention.py:170-188 of the reference.
#include "common.cuh"
#include "mx_quant.cuh"

namespace kwu {

constexpr int FA_BM = 128;   // query rows per CTA
constexpr int FA_BN = 128;   // keys per tile
constexpr int FA_D = 64;
constexpr int FA_THREADS = 320;  // 8 softmax warps + TMA warp + MMA warp
constexpr int FA_TILE_BYTES = 128 * 64 * 2;  // 16 KB
constexpr int FA_SMEM = 5 * FA_TILE_BYTES + 1024 + 3072 + 1024;  // tiles + barriers + row-max exchange + alignment slack
constexpr float FA_NEG = -1.0e30f;
template <bool V> struct FwdBoolC { static constexpr bool value = V; };
template <int V> struct IntC { static constexpr int value = V; };

struct FlashFwdParams {
  __nv_bfloat16* out;   // (T, Hq, 64)
  float* lse;           // (Hq, T)
  const int4* plan;     // (q0, doc_start, doc_end, valid)
  int n_tiles;
  int T, Hq, Hkv, window;
  int row_len;            // SPLIT: tokens of one row of the padded batch; every document is one row
  const float* sink_lse;  // (Hq) or null
  float scale_log2;       // softmax scale * log2(e)
  int* status;
  // optional MXFP8 copy of `out` seen as a (T, Hq * 64) matrix: e4m3 bytes + UE8M0 scale chunks (the layout of
  // mxfp8.cu), for an MXFP8 output projection. Each epilogue thread holds exactly one 32-element block.
  uint8_t* q8;
  uint8_t* sf;
};

// Tile lists for packed batches: for every document, ceil(len/tile) entries (q0, doc_start, doc_end, valid),
// written twice: plan[0, max_tiles) sorted by the number of keys a QUERY tile sees (descending: the order
// of the forward and dQ kernels), plan[max_tiles, 2*max_tiles) sorted by the number of queries that see a
// KEY tile (descending: the dK / dV kernel). Unused entries sort last. One block; a rank sort, since the
// list has at most a few hundred entries.
__global__ void attn_plan_kernel(const int* __restrict__ cu, int ndocs, int tile, int4* __restrict__ plan,
                                 int max_tiles) {
  extern __shared__ int4 s_plan[];                                   // max_tiles entries in token order
  int* s_off = reinterpret_cast<int*>(s_plan + max_tiles);           // ndocs + 1
  for (int d = threadIdx.x; d < ndocs; d += blockDim.x) {
    const int len = cu[d + 1] - cu[d];
    s_off[d + 1] = (len + tile - 1) / tile;
  }
  if (threadIdx.x == 0) s_off[0] = 0;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int d = 0; d < ndocs; ++d) s_off[d + 1] += s_off[d];
  __syncthreads();
  const int used = s_off[ndocs];
  for (int d = threadIdx.x; d < ndocs; d += blockDim.x) {
    const int s = cu[d], e = cu[d + 1];
    int idx = s_off[d];
    for (int q0 = s; q0 < e && idx < max_tiles; q0 += tile, ++idx) s_plan[idx] = make_int4(q0, s, e, 1);
  }
  for (int i = used + threadIdx.x; i < max_tiles; i += blockDim.x) s_plan[i] = make_int4(0, 0, 0, 0);
  __syncthreads();
  for (int i = threadIdx.x; i < max_tiles; i += blockDim.x) {
    const int4 me = s_plan[i];
    const int cq = me.w ? min(me.x + tile, me.z) - me.y : -1;   // keys visible to the tile's last query row
    const int ck = me.w ? me.z - me.x : -1;                     // queries that can see the tile's first key
    int rq = 0, rk = 0;
    for (int j = 0; j < max_tiles; ++j) {
      const int4 o = s_plan[j];
      const int oq = o.w ? min(o.x + tile, o.z) - o.y : -1;
      const int ok = o.w ? o.z - o.x : -1;
      rq += (oq > cq) || (oq == cq && j < i);
      rk += (ok > ck) || (ok == ck && j < i);
    }
    plan[rq] = me;
    plan[max_tiles + rk] = me;
  }
}

// Work item = (query tile, query head). A CTA walks items blockIdx.x, blockIdx.x + gridDim.x, ... of the
// heaviest-first list, so TMEM allocation, barrier set-up and the tensor-map fetch are paid once per CTA,
// and the producer warp is already loading the next item's Q and K while the softmax warps finish the
// current one. Barrier phases run on counters that continue across items.
struct FwdItem {
  int q0, ds, de, h, hk, lo, n_kv, q_hi;
};

__device__ __forceinline__ bool fwd_decode(const FlashFwdParams& p, int item, FwdItem& it) {
  const int4 job = p.plan[item / p.Hq];   // the list is sorted: query tiles that see the most keys first
  if (!job.w) return false;
  it.q0 = job.x; it.ds = job.y; it.de = job.z;
  it.h = item % p.Hq;
  it.hk = it.h / (p.Hq / p.Hkv);
  it.q_hi = min(min(it.q0 + FA_BM, it.de), p.T);  // one past the last valid query row; a longer plan stores nothing past T
  it.lo = it.ds;
  if (p.window > 0) it.lo = max(it.ds, it.q0 - p.window + 1);
  it.n_kv = (it.q_hi - it.lo + FA_BN - 1) / FA_BN;
  return it.n_kv > 0;
}

template <bool SPLIT>
__global__ void __launch_bounds__(FA_THREADS, 2)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const FlashFwdParams p) {
  pdl_sync();   // nothing of the previous kernel is read above this line
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = smem + FA_TILE_BYTES;       // 2 stages
  uint8_t* sV = smem + 3 * FA_TILE_BYTES;   // 2 stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 5 * FA_TILE_BYTES);
  uint64_t* q_full = bars + 0;
  uint64_t* k_full = bars + 1;   // [2]
  uint64_t* k_empty = bars + 3;  // [2]
  uint64_t* v_full = bars + 5;   // [2]
  uint64_t* v_empty = bars + 7;  // [2]
  uint64_t* s_full = bars + 9;
  uint64_t* p_full = bars + 10;
  uint64_t* o_done = bars + 11;
  uint64_t* q_empty = bars + 12;  // the item's last S product has read Q
  uint64_t* o_free = bars + 13;   // the softmax warps have read the item's O accumulator
  uint64_t* s_free = bars + 14;   // the scores of a tile are in registers (not SPLIT, which keeps P's lower parts there)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* s_rowmax = reinterpret_cast<float*>(smem + 5 * FA_TILE_BYTES + 1024);  // 2 x 256 max + 256 sums

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_items = p.n_tiles * p.Hq;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(p_full, 8);
    mbar_init(o_done, 1);
    mbar_init(q_empty, 1);
    mbar_init(o_free, 8);
    mbar_init(s_free, 8);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tP = tmem_base + 128, tO = tmem_base + 192;

  if (warp == 8) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tmQ);
      tma_prefetch_desc(&tmK);
      tma_prefetch_desc(&tmV);
      int g = 0, ic = 0;   // K/V tiles and items issued so far by this CTA
      bool ok = true;
      auto load = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int col, int token, const FwdItem& it) {
        if constexpr (SPLIT) tma_load_3d(dst, tm, bar, col, token - it.ds, it.ds / p.row_len);
        else tma_load_2d(dst, tm, bar, col, token);
      };
      for (int rnd = 0; rnd * static_cast<int>(gridDim.x) < n_items && ok; ++rnd) {
        const int item = snake_item(rnd);
        if (item >= n_items) continue;
        FwdItem it;
        if (!fwd_decode(p, item, it)) continue;
        if (!mbar_wait(q_empty, (ic & 1) ^ 1, abort_flag, p.status, KWU_ERR_TIMEOUT_EMPTY)) break;
        ++ic;
        mbar_expect_tx(q_full, FA_TILE_BYTES);
        load(sQ, &tmQ, q_full, it.h * FA_D, it.q0, it);
        for (int j = 0; j < it.n_kv; ++j, ++g) {
          const int s = g & 1;
          const uint32_t ph = (g >> 1) & 1;
          const int kv0 = it.lo + j * FA_BN;
          if (!mbar_wait(&k_empty[s], ph ^ 1, abort_flag, p.status, KWU_ERR_TIMEOUT_EMPTY)) { ok = false; break; }
          mbar_expect_tx(&k_full[s], FA_TILE_BYTES);
          load(sK + s * FA_TILE_BYTES, &tmK, &k_full[s], it.hk * FA_D, kv0, it);
          if (!mbar_wait(&v_empty[s], ph ^ 1, abort_flag, p.status, KWU_ERR_TIMEOUT_EMPTY)) { ok = false; break; }
          mbar_expect_tx(&v_full[s], FA_TILE_BYTES);
          load(sV + s * FA_TILE_BYTES, &tmV, &v_full[s], it.hk * FA_D, kv0, it);
        }
      }
    }
  } else if (warp == 9) {
    // ---------------------------------------------------------------- MMA issuer
    // The whole warp walks the loop, so that descriptors and counters stay warp-uniform (a single-lane
    // branch keeps them in per-thread registers and pays a transfer into the uniform registers for every
    // operand of every tcgen05.mma, on the critical path between two softmax tiles); one elected lane issues.
    const bool leader = elect_one();
    const uint32_t idesc_s = make_idesc_f16(128, 128, 1, 0, 0);
    const uint32_t idesc_o = make_idesc_f16(128, 64, 1, 0, 1);
    const uint64_t dQ0 = make_smem_desc(smem_u32(sQ), 16, 1024, SWZ_128B);
    int g = 0, ic = 0;
    bool ok = true;
    auto issue_s = [&](int gj, bool last_of_item) {
      const int s = gj & 1;
      const uint64_t dK = make_smem_desc(smem_u32(sK + s * FA_TILE_BYTES), 16, 1024, SWZ_128B);
      if (leader) {
#pragma unroll
        for (int k = 0; k < FA_D / 16; ++k) mma_f16_ss(tS, dQ0 + 2 * k, dK + 2 * k, idesc_s, k > 0 ? 1u : 0u);
        tc_commit(s_full);
        tc_commit(&k_empty[s]);
        if (last_of_item) tc_commit(q_empty);
      }
      __syncwarp();
    };
    auto wait_all = [&](uint64_t* bar, uint32_t parity, int code) {
      return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, p.status, code));
    };
    for (int rnd = 0; rnd * static_cast<int>(gridDim.x) < n_items && ok; ++rnd) {
      const int item = snake_item(rnd);
      if (item >= n_items) continue;
      FwdItem it;
      if (!fwd_decode(p, item, it)) continue;
      const int n_kv = it.n_kv;
      ok = wait_all(q_full, ic & 1, KWU_ERR_TIMEOUT_FULL);
      if (ok) ok = wait_all(&k_full[g & 1], (g >> 1) & 1, KWU_ERR_TIMEOUT_FULL);
      if (!ok) break;
      tc_fence_after();
      // S of the previous item has been read (its last p_full was waited for below) and P is rewritten
      // by the softmax warps only after they have waited for the previous item's last o_done
      issue_s(g, n_kv == 1);
      for (int j = 0; j < n_kv && ok; ++j) {
        const int gj = g + j;
        const int s = gj & 1;
        const uint32_t ph = (gj >> 1) & 1;
        if (j + 1 < n_kv) {
          ok = wait_all(&k_full[(gj + 1) & 1], ((gj + 1) >> 1) & 1, KWU_ERR_TIMEOUT_FULL);
          if (!ok) break;
        }
        if (!SPLIT) {
          // the next scores are formed under this tile's exponentials, as soon as its own have left TMEM
          ok = wait_all(s_free, gj & 1, KWU_ERR_TIMEOUT_MISC);
          if (!ok) break;
          tc_fence_after();
          if (j + 1 < n_kv) issue_s(gj + 1, j + 2 == n_kv);
        }
        // P_j written (and S_j fully read) by the softmax warps
        ok = wait_all(p_full, gj & 1, KWU_ERR_TIMEOUT_MISC);
        if (!ok) break;
        tc_fence_after();
        const uint64_t dV = make_smem_desc(smem_u32(sV + s * FA_TILE_BYTES), 8192, 1024, SWZ_128B);
        uint32_t acc = j > 0 ? 1u : 0u;
        ok = wait_all(&v_full[s], ph, KWU_ERR_TIMEOUT_FULL);
        if (!ok) break;
        if (j == 0) {
          // the first product of an item overwrites O: the previous item's epilogue must have read it
          ok = wait_all(o_free, (ic & 1) ^ 1, KWU_ERR_TIMEOUT_ACC_EMPTY);
          if (!ok) break;
        }
        tc_fence_after();
        if (SPLIT) {
          // keys 32 i .. 32 i + 31: middle parts at score columns 32 i .. 32 i + 15, low parts at the 16 after them
          if (leader) {
#pragma unroll
            for (int part = 1; part >= 0; --part)
#pragma unroll
              for (int k = 0; k < FA_BN / 16; ++k)
                mma_f16_ts(tO, tS + (k >> 1) * 32 + part * 16 + (k & 1) * 8, dV + 128 * k, idesc_o, k > 0 || part == 0 ? 1u : acc);
          }
          __syncwarp();
          acc = 1u;
          if (j + 1 < n_kv) issue_s(gj + 1, j + 2 == n_kv);   // in order behind the product that reads these columns
        }
        if (leader) {
          mma_f16_ts(tO, tP, dV, idesc_o, acc);
#pragma unroll
          for (int k = 1; k < FA_BN / 16; ++k) mma_f16_ts(tO, tP + k * 8, dV + 128 * k, idesc_o, 1u);
          tc_commit(o_done);
          tc_commit(&v_empty[s]);
        }
        __syncwarp();
      }
      g += n_kv;
      ++ic;
    }
  } else {
    // ---------------------------------------------------------------- softmax (warps 0..7)
    // Two threads per query row: warp w and warp w+4 share TMEM lane quarter w%4; the first takes key
    // columns [0,64) of the tile, the second [64,128). They exchange only the row maximum (through
    // shared memory, once per tile); each keeps its own partial row sum until the epilogue.
    const int quarter = warp & 3, half = warp >> 2;
    const int row = quarter * 32 + lane;     // query row inside the tile == TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t col_base = half * 64;
    // the two warps that share a row meet on a named barrier of their own
    auto pair_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(quarter + 1) : "memory"); };
    int g = 0;
    bool ok = true;
    for (int rnd = 0; rnd * static_cast<int>(gridDim.x) < n_items; ++rnd) {
      const int item = snake_item(rnd);
      if (item >= n_items) continue;
      FwdItem it;
      if (!fwd_decode(p, item, it)) continue;
      const int q0 = it.q0, n_kv = it.n_kv, h = it.h;
      const int qi = q0 + row;
      float m = FA_NEG, l = 0.f;
      for (int j = 0; j < n_kv; ++j) {
        const int gj = g + j;
        const int kv0 = it.lo + j * FA_BN;
        // after a time-out the loops keep running (so every warp still meets the named barrier below)
        // but do no work; the waits return at once because the abort flag is set
        if (ok) {
          ok = mbar_wait(s_full, gj & 1, abort_flag, p.status, KWU_ERR_TIMEOUT_ACC_FULL);
          ok = __all_sync(0xffffffffu, ok);
        }
        tc_fence_after();
        const bool need_mask = (kv0 + FA_BN - 1 > q0) || (p.window > 0 && (q0 + FA_BM - 1 - kv0) >= p.window);
        // key columns this row may see inside the tile: [c_lo, c_hi]
        const int c_hi = qi - kv0;
        const int c_lo = (p.window > 0) ? (qi - p.window + 1 - kv0) : -1;
        // pass 1: maximum of the raw scores of this thread's 64 columns (the positive scale commutes with max)
        float mx4[4] = {FA_NEG, FA_NEG, FA_NEG, FA_NEG};
        auto max32 = [&](const uint32_t (&r)[32], int base) {
          if (need_mask) {
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              const int col = base + e;
              const float sv = (col <= c_hi && col >= c_lo) ? __uint_as_float(r[e]) : FA_NEG;
              mx4[e & 3] = fmaxf(mx4[e & 3], sv);
            }
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) mx4[e & 3] = fmaxf(mx4[e & 3], __uint_as_float(r[e]));
          }
        };
        uint32_t kept[32];   // the second half's scores stay in registers for pass 2
        if (ok) {
          {
            uint32_t r[32];
            tmem_ld_x32(tS + lane_addr + col_base, r);
            tmem_ld_wait();
            max32(r, col_base);
          }
          tmem_ld_x32(tS + lane_addr + col_base + 32, kept);
          tmem_ld_wait();
          max32(kept, col_base + 32);
        }
        float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        // exchange with the thread that owns the other half of the row (buffers alternate per tile)
        float* xbuf = s_rowmax + (gj & 1) * 256;
        xbuf[half * 128 + row] = mx;
        pair_sync();
        mx = fmaxf(fmaxf(mx, xbuf[(half ^ 1) * 128 + row]), m);
        if (!ok) continue;
        const float neg_ms = __fmul_rn(-mx, p.scale_log2);
        // SPLIT: from the rounded products that the exponents are taken against, so that keys of different tiles keep their
        // ratio to the last bits
        const float alpha = fast_exp2(SPLIT ? neg_ms + __fmul_rn(m, p.scale_log2) : (m - mx) * p.scale_log2);
        m = mx;
        // the previous P V product must be complete before P is overwritten and O is touched; for the
        // first tile of an item that product belongs to the previous item and was waited for in its epilogue
        if (j > 0) {
          ok = mbar_wait(o_done, (gj - 1) & 1, abort_flag, p.status, KWU_ERR_TIMEOUT_ACC_EMPTY);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) continue;
          tc_fence_after();
          if (__any_sync(0xffffffffu, alpha != 1.f)) {
            // this thread rescales its half of the row's 64 output columns
            uint32_t o[32];
            tmem_ld_x32(tO + lane_addr + half * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
            tmem_st_x32(tO + lane_addr + half * 32, o);
          }
        }
        // pass 2: probabilities p = 2^(s*c - m*c), packed to bf16 and stored 32 columns at a time
        float sum4[4] = {0.f, 0.f, 0.f, 0.f};
        // the mask is needed only on diagonal / window-edge tiles (the same for the whole CTA): two copies
        // of the loop, so that the common one carries no compares or selects
        auto pass2 = [&](auto masked) {
          constexpr bool MASK = decltype(masked)::value;
          const uint64_t sl2 = pack_f32x2(p.scale_log2, p.scale_log2), nm2 = pack_f32x2(neg_ms, neg_ms);
          uint64_t acc2[2] = {pack_f32x2(0.f, 0.f), pack_f32x2(0.f, 0.f)};
          // the 32 scores of half c of the thread's columns
          auto exp32 = [&](uint32_t (&r)[32], auto half_c) {
            constexpr int c = decltype(half_c)::value;
            auto exp2of = [&](int e, float& p0, float& p1) {
              unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), sl2, nm2), p0, p1);
              p0 = fast_exp2(p0);
              p1 = fast_exp2(p1);
              if constexpr (MASK) {
                const int col = col_base + c * 32 + e;
                p0 = (col <= c_hi && col >= c_lo) ? p0 : 0.f;
                p1 = (col + 1 <= c_hi && col + 1 >= c_lo) ? p1 : 0.f;
              }
              acc2[(e >> 1) & 1] = add_f32x2(acc2[(e >> 1) & 1], pack_f32x2(p0, p1));
            };
            if constexpr (SPLIT) {
              // 16 scores at a time: their 24 packed words leave before the next 16 are worked on (registers)
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                uint32_t hi[8], mid[8], low[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  float p0, p1;
                  exp2of(16 * q + 2 * i, p0, p1);
                  hi[i] = pack_bf16(p0, p1);
                  float2 f = unpack_bf16(hi[i]);
                  p0 -= f.x;
                  p1 -= f.y;
                  mid[i] = pack_bf16(p0, p1);
                  f = unpack_bf16(mid[i]);
                  low[i] = pack_bf16(p0 - f.x, p1 - f.y);
                }
                tmem_st_x8(tP + lane_addr + half * 32 + c * 16 + q * 8, hi);
                tmem_st_x8(tS + lane_addr + col_base + c * 32 + q * 8, mid);
                tmem_st_x8(tS + lane_addr + col_base + c * 32 + 16 + q * 8, low);
              }
            } else {
              uint32_t pk[16];
#pragma unroll
              for (int e = 0; e < 32; e += 2) {
                float p0, p1;
                exp2of(e, p0, p1);
                pk[e / 2] = pack_bf16(p0, p1);
              }
              tmem_st_x16(tP + lane_addr + half * 32 + c * 16, pk);
            }
          };
          {
            uint32_t r[32];
            tmem_ld_x32(tS + lane_addr + col_base, r);
            tmem_ld_wait();
            if constexpr (!SPLIT) {
              tc_fence_before();
              mbar_arrive_warp(s_free);
            }
            exp32(r, IntC<0>{});
          }
          if constexpr (SPLIT) {   // the parts take registers: read again (each half's parts stay in its own columns)
            uint32_t r[32];
            tmem_ld_x32(tS + lane_addr + col_base + 32, r);
            tmem_ld_wait();
            exp32(r, IntC<1>{});
          } else {
            exp32(kept, IntC<1>{});
          }
          unpack_f32x2(acc2[0], sum4[0], sum4[1]);
          unpack_f32x2(acc2[1], sum4[2], sum4[3]);
        };
        if (need_mask) pass2(FwdBoolC<true>{}); else pass2(FwdBoolC<false>{});
        l = l * alpha + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive_warp(p_full);
      }
      // ---------------------------------------------------------------- epilogue of the item
      if (ok) {
        ok = mbar_wait(o_done, (g + n_kv - 1) & 1, abort_flag, p.status, KWU_ERR_TIMEOUT_ACC_FULL);
        ok = __all_sync(0xffffffffu, ok);
      }
      // total row sum = own partial + the partner's (both are relative to the same final maximum)
      float* lbuf = s_rowmax + 512;
      lbuf[half * 128 + row] = l;
      pair_sync();
      l += lbuf[(half ^ 1) * 128 + row];
      if (ok) {
        tc_fence_after();
        uint32_t o[32];
        tmem_ld_x32(tO + lane_addr + half * 32, o);
        tmem_ld_wait();
        tc_fence_before();
        mbar_arrive_warp(o_free);   // the next item's first product may overwrite O now
        float lse = (m * p.scale_log2 + log2f(l)) * 0.6931471805599453f;  // natural log
        float inv = 1.f / l;
        if (p.sink_lse) {
          const float sl = p.sink_lse[h];
          const float tot = fmaxf(lse, sl) + log1pf(__expf(-fabsf(lse - sl)));
          inv *= __expf(lse - tot);
          lse = tot;
        }
        if (SPLIT && !(l > 0.f && l < INFINITY)) {
          // a row whose scores hold a NaN or an infinity, or are all -inf, has no probabilities: its output is zero
          inv = 0.f;
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = 0u;
        }
        if (qi < it.q_hi) {
          uint4* dst = reinterpret_cast<uint4*>(p.out + (static_cast<size_t>(qi) * p.Hq + h) * FA_D + half * 32);
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            uint4 w;
            w.x = pack_bf16(__uint_as_float(o[8 * v + 0]) * inv, __uint_as_float(o[8 * v + 1]) * inv);
            w.y = pack_bf16(__uint_as_float(o[8 * v + 2]) * inv, __uint_as_float(o[8 * v + 3]) * inv);
            w.z = pack_bf16(__uint_as_float(o[8 * v + 4]) * inv, __uint_as_float(o[8 * v + 5]) * inv);
            w.w = pack_bf16(__uint_as_float(o[8 * v + 6]) * inv, __uint_as_float(o[8 * v + 7]) * inv);
            dst[v] = w;
            // keep the rounded values (what a quantise pass over the stored tensor would read)
            o[8 * v + 0] = w.x << 16; o[8 * v + 1] = w.x & 0xffff0000u;
            o[8 * v + 2] = w.y << 16; o[8 * v + 3] = w.y & 0xffff0000u;
            o[8 * v + 4] = w.z << 16; o[8 * v + 5] = w.z & 0xffff0000u;
            o[8 * v + 6] = w.w << 16; o[8 * v + 7] = w.w & 0xffff0000u;
          }
          if (p.q8) {
            float amax = 0.f;
#pragma unroll
            for (int e = 0; e < 32; ++e) amax = fmaxf(amax, fabsf(__uint_as_float(o[e])));
            const uint32_t e8 = ue8m0_from_amax(amax);
            const float qs = inv_scale_from_ue8m0(e8);
            uint32_t b[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(
                  make_float2(__uint_as_float(o[4 * j]) * qs, __uint_as_float(o[4 * j + 1]) * qs), __NV_SATFINITE, __NV_E4M3);
              const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(
                  make_float2(__uint_as_float(o[4 * j + 2]) * qs, __uint_as_float(o[4 * j + 3]) * qs), __NV_SATFINITE, __NV_E4M3);
              b[j] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
            }
            const int ncols = p.Hq * FA_D;
            uint4* qd = reinterpret_cast<uint4*>(p.q8 + static_cast<size_t>(qi) * ncols + h * FA_D + half * 32);
            qd[0] = make_uint4(b[0], b[1], b[2], b[3]);
            qd[1] = make_uint4(b[4], b[5], b[6], b[7]);
            p.sf[sf_offset(qi, h * 2 + half, ncols >> 7)] = static_cast<uint8_t>(e8);
          }
          if (half == 0) p.lse[static_cast<size_t>(h) * p.T + qi] = lse;
        }
      }
      g += n_kv;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag)
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

}  // namespace kwu

using namespace kwu;

KWU_API int kwu_attn_plan(const int* cu_seqlens, int ndocs, int tile, void* plan, int max_tiles,
                          void* stream) {
  if (ndocs <= 0 || max_tiles <= 0) return 0;
  const size_t smem = static_cast<size_t>(max_tiles) * sizeof(int4) + (ndocs + 1) * sizeof(int);
  if (smem > 96 * 1024) {
    set_last_error("attn_plan: too many tiles / documents (%d / %d)", max_tiles, ndocs);
    return 7;
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  static PerDeviceOnce attr;
  if (smem > 48 * 1024 && attr.pending()) {
    cudaFuncSetAttribute(attn_plan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    attr.mark();
  }
  attn_plan_kernel<<<1, 256, smem, st>>>(cu_seqlens, ndocs, tile, reinterpret_cast<int4*>(plan), max_tiles); kwu::count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_last_error("attn_plan launch: %s", cudaGetErrorString(e)); return 11; }
  return 0;
}

template <bool SPLIT>
static int flash_fwd_impl(const void* q, int q_ld, const void* k, int k_ld, const void* v, int v_ld,
                          void* out, float* lse, const void* plan, int n_tiles, int T, int Hq, int Hkv,
                          int window, const float* sink_lse, float scale, void* q8, void* sf, void* stream,
                          int* status, int row_len = 0) {
  if (T <= 0 || n_tiles <= 0) return 0;
  if (q8 && (T % 128 || (Hq * FA_D) % 128 || !sf)) {
    set_last_error("flash_fwd: the fp8 copy needs tokens and Hq * 64 in multiples of 128");
    return 7;
  }
  if (Hq % Hkv) { set_last_error("flash_fwd: Hq must be a multiple of Hkv"); return 7; }
  CUtensorMap tmQ, tmK, tmV;
  int rc;
  auto encode = [&](CUtensorMap* tm, const void* base, int heads, int ld) {
    const uint64_t cols = static_cast<uint64_t>(heads) * FA_D;
    if (SPLIT)
      return encode_tmap_3d(tm, base, ELEM_BF16, T / row_len, row_len, cols, static_cast<uint64_t>(row_len) * ld, ld, FA_BM, FA_D,
                            CU_TENSOR_MAP_SWIZZLE_128B);
    return encode_tmap_2d(tm, base, ELEM_BF16, T, cols, ld, FA_BM, FA_D, CU_TENSOR_MAP_SWIZZLE_128B);
  };
  static_assert(FA_BM == FA_BN, "query and key tiles have one box");
  if ((rc = encode(&tmQ, q, Hq, q_ld))) return rc;
  if ((rc = encode(&tmK, k, Hkv, k_ld))) return rc;
  if ((rc = encode(&tmV, v, Hkv, v_ld))) return rc;
  static PerDeviceOnce attr;
  if (attr.pending()) {
    cudaError_t e = cudaFuncSetAttribute(flash_fwd_kernel<SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, FA_SMEM);
    if (e != cudaSuccess) { set_last_error("flash_fwd attr: %s", cudaGetErrorString(e)); return 10; }
    attr.mark();
  }
  FlashFwdParams p;
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.lse = lse;
  p.plan = reinterpret_cast<const int4*>(plan);
  p.n_tiles = n_tiles;
  p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.window = window;
  p.row_len = row_len;
  p.sink_lse = sink_lse;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  p.q8 = reinterpret_cast<uint8_t*>(q8);
  p.sf = reinterpret_cast<uint8_t*>(sf);
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  long long items = static_cast<long long>(n_tiles) * Hq;
  int grid = static_cast<int>(items < 2LL * sms ? items : 2LL * sms);   // two resident CTAs per SM, each walks the item list
  launch_k(flash_fwd_kernel<SPLIT>, dim3(grid), dim3(FA_THREADS), FA_SMEM, reinterpret_cast<cudaStream_t>(stream), tmQ, tmK, tmV, p); kwu::count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_last_error("flash_fwd launch: %s", cudaGetErrorString(e)); return 11; }
  return 0;
}

KWU_API int kwu_flash_fwd(const void* q, int q_ld, const void* k, int k_ld, const void* v, int v_ld,
                          void* out, float* lse, const void* plan, int n_tiles, int T, int Hq, int Hkv,
                          int window, const float* sink_lse, float scale, void* stream, int* status) {
  return flash_fwd_impl<false>(q, q_ld, k, k_ld, v, v_ld, out, lse, plan, n_tiles, T, Hq, Hkv, window, sink_lse, scale,
                        nullptr, nullptr, stream, status);
}

// As kwu_flash_fwd, and also writes the MXFP8 copy of `out` viewed as (T, Hq * 64): q8 (T, Hq * 64) e4m3 bytes and
// sf, kwu_mxfp8_sf_bytes(T, Hq * 64) bytes of scale chunks. T must be a multiple of 128 (every row of every
// scale chunk is then written: each token belongs to exactly one query tile).
KWU_API int kwu_flash_fwd_mx(const void* q, int q_ld, const void* k, int k_ld, const void* v, int v_ld,
                             void* out, float* lse, const void* plan, int n_tiles, int T, int Hq, int Hkv,
                             int window, const float* sink_lse, float scale, void* q8, void* sf, void* stream,
                             int* status) {
  return flash_fwd_impl<false>(q, q_ld, k, k_ld, v, v_ld, out, lse, plan, n_tiles, T, Hq, Hkv, window, sink_lse, scale,
                        q8, sf, stream, status);
}

// As kwu_flash_fwd over `rows` rows of `row_len` tokens each (the documents of the plan), with probabilities carried in 24
// bits (SPLIT above): for padded batches, whose callers would otherwise form attention in 32 bits.
KWU_API int kwu_flash_fwd_split(const void* q, int q_ld, const void* k, int k_ld, const void* v, int v_ld,
                                void* out, float* lse, const void* plan, int n_tiles, int rows, int row_len, int Hq, int Hkv,
                                int window, const float* sink_lse, float scale, void* stream, int* status) {
  if (rows <= 0 || row_len <= 0) return 0;
  if (static_cast<long long>(rows) * row_len > 0x7fffffffLL) { set_last_error("flash_fwd_split: too many tokens"); return 7; }
  return flash_fwd_impl<true>(q, q_ld, k, k_ld, v, v_ld, out, lse, plan, n_tiles, rows * row_len, Hq, Hkv, window, sink_lse,
                              scale, nullptr, nullptr, stream, status, row_len);
}
