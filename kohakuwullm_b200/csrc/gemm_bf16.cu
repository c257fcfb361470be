// Persistent, warp-specialised bf16 GEMM on the 5th-generation tensor cores.
//
//   C[M,N] (+)= A * B      fp32 accumulation in TMEM, bf16 or fp32 output
//
// Operand storage (each operand independently):
//   A "K-major":  A stored [M,K] row-major.      A "MN-major": A stored [K,M] row-major.
//   B "K-major":  B stored [N,K] row-major.      B "MN-major": B stored [K,N] row-major.
// so y = x W^T, dx = dy W and dW = dy^T x all run without a transpose pass.
//
// Structure of one CTA (192 threads, one CTA per SM, static round-robin tile schedule):
//   warp 0      TMA producer: cp.async.bulk.tensor tiles into a 128B-swizzled smem ring
//   warp 1      allocates TMEM; one lane issues tcgen05.mma and tcgen05.commit
//   warps 2..5  epilogue: tcgen05.ld the finished accumulator, convert, stage in smem, TMA store / reduce
// Two TMEM accumulators let the epilogue of tile i overlap the main loop of tile i+1.
//
// CG = 2: a cluster of two CTAs works on one 256 x BN tile (`cta_group::2`). Each CTA holds its 128 rows of A and HALF
// of B's BN rows in its shared memory and accumulates its own 128 x BN half; the even CTA issues the products for both.
// Per 64-deep k-block an SM then fetches 16 KB + BN * 64 B instead of 16 KB + BN * 128 B, so the L2 and the
// shared-memory port carry a third less at BN = 256, and a tile of the pair needs half as many loads of A.
//
// The output leaves through shared memory and TMA (whole 128-byte row segments) instead of one 16-byte store per lane
// and row: the scattered stores, not the tensor pipe, bounded the short contractions (4096 x 7168 x 1280: 67 us with
// them; the same main loop with the cross-entropy epilogue, which stores nothing, ran at 1.6 PFLOP/s). fp32 C += is a
// TMA reduction for the same reason. Before / after (one CTA with per-lane stores, stream-K for C +=), B200, us:
//   4096 x 7168 x 1280  67.4 / 54.6    16384 x 1536 x 4096  246 / 145    16384 x 1536 x 8192 (B MN)  420 / 286
//   C +=, both MN: 7168 x 1280 x 4096  74.6 / 56.2    8192 x 1536 x 16384  468 / 301    65536 x 1280 x 4096  647 / 490
// What bounds it now: 8192^3 runs at 1.53 PFLOP/s with 12 TB/s of operands from the L2 (the pair's 256 x 256 tile is
// the largest that TMEM can double-buffer); products of one to three rounds lose their last, partly empty round and
// about 4 us of launch, fill and drain.
// Takes the role of the cuBLAS calls behind nn.Linear in the reference
// (src/kohakuwullm/models/components/attention.py:77-89, mlp.py:15-126).
#include "common.cuh"

#include <cstdio>
#include <mutex>
#include <unordered_map>

namespace kwu {

constexpr int GEMM_BM = 128;  // rows of one CTA
constexpr int GEMM_BK = 64;   // 64 bf16 = one 128-byte swizzle row
constexpr int GEMM_THREADS = 192;

// How the accumulator leaves the kernel (EPI_STORE)
constexpr int OUT_TMA_BF16 = 0;   // bf16, TMA store
constexpr int OUT_TMA_F32 = 1;    // fp32, TMA store
constexpr int OUT_TMA_ADD = 2;    // fp32, TMA reduction (C +=)
constexpr int OUT_DIRECT = 3;     // per-lane stores: scattered rows, bf16 C +=, pitches TMA cannot address

struct GemmParams {
  int M, N, K;
  int ldc;
  int bn;           // width of a tile
  int out_fp32;     // 0: bf16 output, 1: fp32 output
  int accumulate;   // 1: C += A*B
  int out_mode;     // OUT_*
  int out_cols;     // bf16 TMA stores: columns of one store box (64, or 32 when bn is not a multiple of 64)
  float alpha;      // scale applied to the product
  // descriptor constants, computed on the host
  uint32_t a_lbo, a_sbo, a_kadv;
  uint32_t b_lbo, b_sbo, b_kadv;
  uint32_t idesc;
  uint32_t stage_bytes;   // one ring stage of one CTA: its A rows and its share of B
  int b_chunks;           // MN-major B: 64-column boxes of one CTA's share
  int stages;
  int tiles_m, tiles_n;   // tile grid (a tile is 128 * CG rows)
  int* status;
  // split tail (fp32 C += only): tiles [0, full_tiles) are whole work items; each of the `tail_tiles` after them, which
  // would leave the last round of the persistent grid partly empty, is cut into `splits` ranges of the contraction for
  // CTAs (pairs) that would idle, all adding into C. 0 tail tiles: every tile is a whole item.
  int full_tiles, tail_tiles, splits;
  // even ranges (single CTAs, fp32 C += only): the (tile, k-block) units, tiles row by row, are cut into this many equal
  // contiguous ranges, one per CTA; every tile is the sum of the pieces of the ranges that meet in it. 0: off.
  int ranges;
  // grouped (mixture-of-experts) modes
  //   1: rows grouped by expert: row tile t reads group_tiles[t] = (m0, expert, valid); the expert picks
  //      a block of `group_b_rows` rows of B (K-major: output rows; MN-major: contraction rows)
  //   2: contraction grouped by expert (weight gradients): C[e] (+)= A[rows_e]^T B[rows_e] with
  //      rows_e = [group_offsets[e], group_offsets[e+1]); C advances by c_group_rows rows per expert
  //   3: a batch of products of one size: matrix i owns rows [i, i + 1) * c_group_rows of A and C (whole tiles) and a
  //      block of `group_b_rows` rows of B
  int group_mode;
  const int4* group_tiles;
  const int* group_offsets;
  int group_b_rows;
  int num_groups;
  int c_group_rows;
  float diag;       // added on the diagonal of every matrix (mode 3): C = alpha * A B + diag * I
  // scatter epilogue (bf16 EPI_STORE only): output row r goes to the byte address row_ptrs[r] (0: row is
  // dropped) instead of C + r*ldc. The addresses may be peer-mapped memory of another GPU: the expert-
  // parallel combine / gradient return is then done by the GEMM's own epilogue stores, tile by tile.
  const long long* row_ptrs;
  // fused cross-entropy epilogues (EPI_LSE / EPI_DLOGITS)
  const int* labels;     // (M) target column per row, negative = ignored row
  float2* partial;       // EPI_LSE: (tiles_n, M) running (max, sum-exp) per row and column tile
  float* target_logit;   // EPI_LSE: (M) logit of the target column
  const float* lse;      // EPI_DLOGITS: (M) log-sum-exp of the full row
  const float* coef_p;   // EPI_DLOGITS: (M) factor on the probabilities
  const float* coef_y;   // EPI_DLOGITS: (M) factor on the one-hot target
};

constexpr int EPI_STORE = 0;    // C (+)= alpha * acc
constexpr int EPI_LSE = 1;      // no C: per-row (max, sum-exp) partials and the target logit
constexpr int EPI_DLOGITS = 2;  // C = coef_p * exp(acc - lse) - coef_y * onehot   (bf16)

constexpr int GEMM_A_BYTES = GEMM_BM * GEMM_BK * 2;
constexpr int GEMM_MAX_STAGES = 8;
constexpr int GEMM_BAR_BYTES = 1024;
// per epilogue warp two 4 KB patches (32 rows x 128 bytes) that TMA stores read
constexpr int GEMM_OUT_BYTES = 4 * 2 * 4096;
constexpr int GEMM_SMEM_MAX = 227 * 1024;

struct TileInfo {
  int m0, n0;        // output tile origin
  int b_row_off;     // added to B's row coordinate (expert selection)
  int k_begin, nkb;  // contraction range in elements / 64-blocks
  int c_row_off;     // added to the output row (expert selection)
};

constexpr int GEMM_RASTER_ROWS = 2048;

// Same decoding in every role of the CTA. Returns false for tiles that carry no work.
template <int CG>
__device__ __forceinline__ bool decode_tile(const GemmParams& p, int tile, int num_kb, TileInfo& t) {
  constexpr int TM = GEMM_BM * CG;
  t.b_row_off = 0; t.k_begin = 0; t.nkb = num_kb; t.c_row_off = 0;
  if (p.group_mode == 2) {
    const int per = p.tiles_m * p.tiles_n;
    const int e = tile / per, r = tile % per;
    t.m0 = (r / p.tiles_n) * TM;
    t.n0 = (r % p.tiles_n) * p.bn;
    t.k_begin = p.group_offsets[e];
    t.nkb = (p.group_offsets[e + 1] - t.k_begin) / GEMM_BK;
    t.c_row_off = e * p.c_group_rows;
    return t.nkb > 0;
  }
  if (p.group_mode == 3) {
    const int mt = p.c_group_rows / TM, per = mt * p.tiles_n;
    const int i = tile / per, r = tile - i * per;
    t.m0 = i * p.c_group_rows + (r % mt) * TM;
    t.n0 = (r / mt) * p.bn;
    t.b_row_off = i * p.group_b_rows;
    return true;
  }
  if (p.group_mode == 1) {
    const int tm = tile / p.tiles_n;
    t.n0 = (tile % p.tiles_n) * p.bn;
    const int4 g = p.group_tiles[tm];
    t.m0 = g.x;
    t.b_row_off = g.y * p.group_b_rows;
    return g.z != 0;
  }
  // Raster order: panels of GEMM_RASTER_ROWS rows, rows fastest inside a panel. The tiles that run at the
  // same time then share a few B tiles and one A panel, which stays in L2; with columns fastest every wave
  // of a wide product (a 65536-row vocabulary matrix) streams a different stretch of B from HBM for every
  // row tile, 32 times the matrix in total.
  constexpr int RASTER = GEMM_RASTER_ROWS / TM;
  const int span = RASTER * p.tiles_n;
  const int panel = tile / span, within = tile - panel * span;
  const int gm = min(RASTER, p.tiles_m - panel * RASTER);
  t.m0 = (panel * RASTER + within % gm) * TM;
  t.n0 = (within / gm) * p.bn;
  return true;
}

// Work item number `i` of this CTA (pair). 0: none left; 1: `t` holds work; 2: nothing to do for this index, go on.
template <int CG>
__device__ __forceinline__ int next_work(const GemmParams& p, int i, int num_tiles, int num_kb, TileInfo& t) {
  if (CG == 1 && p.ranges > 0) {
    const long long units = static_cast<long long>(num_tiles) * num_kb;
    const long long u0 = units * blockIdx.x / p.ranges, u1 = units * (blockIdx.x + 1) / p.ranges;
    // the piece that begins its tile first, then the one that ends its tile: with about one tile per range every CTA then
    // walks the contraction from 0 to K at the same time as the others, and the slabs of A and B that they share stay in
    // the L2 (tile by tile the ranges are spread over the whole contraction)
    const long long first = u0 / num_kb, pieces = u1 > u0 ? (u1 - 1) / num_kb - first + 1 : 0;
    if (i >= pieces) return 0;
    const long long tile = i == 0 ? first + pieces - 1 : first + i - 1;
    const long long start = max(u0, tile * num_kb), end = min(u1, (tile + 1) * num_kb);
    t.b_row_off = 0; t.c_row_off = 0;
    t.m0 = static_cast<int>(tile / p.tiles_n) * GEMM_BM;
    t.n0 = static_cast<int>(tile % p.tiles_n) * p.bn;
    t.k_begin = static_cast<int>(start - tile * num_kb) * GEMM_BK;
    t.nkb = static_cast<int>(end - start);
    return 1;
  }
  const int item = static_cast<int>(blockIdx.x) / CG + i * (static_cast<int>(gridDim.x) / CG);
  if (p.tail_tiles > 0 && item >= p.full_tiles) {
    const int piece = item - p.full_tiles;
    if (piece >= p.tail_tiles * p.splits) return 0;
    decode_tile<CG>(p, p.full_tiles + piece % p.tail_tiles, num_kb, t);
    const int s = piece / p.tail_tiles;
    const int kb0 = num_kb * s / p.splits, kb1 = num_kb * (s + 1) / p.splits;
    t.k_begin = kb0 * GEMM_BK;
    t.nkb = kb1 - kb0;
    return 1;
  }
  if (item >= num_tiles) return 0;
  return decode_tile<CG>(p, item, num_kb, t) ? 1 : 2;
}

template <int CG, bool A_MN, bool B_MN, int EPI>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmC, void* __restrict__ Cbase, const GemmParams p) {
  constexpr uint32_t TMEM_COLS = 512;

  extern __shared__ uint8_t smem_raw[];
  // both CTAs of a pair see the same offset: dynamic shared memory starts at one address in every CTA
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* out_area = smem;
  uint8_t* ring = smem + GEMM_OUT_BYTES;
  uint8_t* bar_area = ring + p.stages * p.stage_bytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(bar_area);
  uint64_t* empty_bar = full_bar + GEMM_MAX_STAGES;
  uint64_t* acc_full = empty_bar + GEMM_MAX_STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int cta = CG == 2 ? static_cast<int>(cluster_ctarank()) : 0;
  const int num_tiles = p.tiles_m * p.tiles_n * (p.group_mode == 2 ? p.num_groups : 1);
  const int num_kb = (p.K + GEMM_BK - 1) / GEMM_BK;
  const int BN = p.bn;
  const int stages = p.stages;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], 4 * CG);   // one arrival per epilogue warp of the pair
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 0 && elect_one()) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    if (EPI != EPI_LSE && p.out_mode != OUT_DIRECT) tma_prefetch_desc(&tmC);
  }
  if (warp == 1) {
    tmem_alloc_cg<CG>(tmem_slot, TMEM_COLS);
    tmem_relinquish_cg<CG>();
  }
  tc_fence_before();
  __syncwarp();
  if (CG == 2) cluster_sync(); else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_sync();   // set-up above overlapped the previous kernel's tail; operands are read from here on

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    // warp-uniform loop, one elected lane issues (coordinates, addresses and the tensor-map pointers stay
    // in uniform registers). With CG = 2 every load of the pair is counted on the even CTA's barrier, whose CTA
    // issues the products.
    const bool leader = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int wi = 0; ok; ++wi) {
      TileInfo ti;
      const int got = next_work<CG>(p, wi, num_tiles, num_kb, ti);
      if (got == 0) break;
      if (got == 2) continue;
      const int m0 = ti.m0 + cta * GEMM_BM, n0 = ti.n0 + cta * (BN / CG);
      for (int kb = 0; kb < ti.nkb; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, KWU_ERR_TIMEOUT_EMPTY));
        if (!ok) break;
        uint8_t* sa = ring + stage * p.stage_bytes;
        uint8_t* sb = sa + GEMM_A_BYTES;
        const int k0 = ti.k_begin + kb * GEMM_BK;
        if (leader) {
          if (cta == 0) mbar_expect_tx(&full_bar[stage], p.stage_bytes * CG);
          const uint32_t bar = CG == 2 ? mapa_shared(smem_u32(&full_bar[stage]), 0) : smem_u32(&full_bar[stage]);
          if (!A_MN) {
            tma_load_2d_cg<CG>(sa, &tmA, bar, k0, m0);
          } else {
#pragma unroll
            for (int c = 0; c < GEMM_BM / 64; ++c) tma_load_2d_cg<CG>(sa + c * 8192, &tmA, bar, m0 + c * 64, k0);
          }
          if (!B_MN) {
            tma_load_2d_cg<CG>(sb, &tmB, bar, k0, n0 + ti.b_row_off);
          } else {
            for (int c = 0; c < p.b_chunks; ++c)
              tma_load_2d_cg<CG>(sb + c * 8192, &tmB, bar, n0 + c * 64, k0 + ti.b_row_off);
          }
        }
        __syncwarp();
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (even CTA of a pair)
    // The whole warp walks the loop so that stage addresses, descriptors and counters stay warp-uniform
    // (a single-lane branch keeps them in per-thread registers and pays a move into the uniform registers
    // for every operand of every tcgen05.mma); one elected lane issues.
    if (cta == 0) {
      const bool leader = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      // the descriptors of one k-block differ only in the address field: +(bytes >> 4) per 16-wide K step
      const uint32_t a_step = static_cast<uint32_t>(p.a_kadv) >> 4, b_step = static_cast<uint32_t>(p.b_kadv) >> 4;
      for (int wi = 0; ok; ++wi) {
        TileInfo ti;
        const int got = next_work<CG>(p, wi, num_tiles, num_kb, ti);
        if (got == 0) break;
        if (got == 2) continue;
        const int as = it & 1;
        const uint32_t aphase = (it >> 1) & 1;
        ++it;
        ok = __all_sync(0xffffffffu, mbar_wait_cluster<CG>(&acc_empty[as], aphase ^ 1, abort_flag, p.status, KWU_ERR_TIMEOUT_ACC_EMPTY));
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + as * 256;
        for (int kb = 0; kb < ti.nkb; ++kb) {
          ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase, abort_flag, p.status, KWU_ERR_TIMEOUT_FULL));
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = smem_u32(ring + stage * p.stage_bytes);
          const uint64_t ad = make_smem_desc(sa, p.a_lbo, p.a_sbo, SWZ_128B);
          const uint64_t bd = make_smem_desc(sa + GEMM_A_BYTES, p.b_lbo, p.b_sbo, SWZ_128B);
          const uint32_t acc0 = kb > 0 ? 1u : 0u;
          if (leader) {
            mma_f16_ss_cg<CG>(d_tmem, ad, bd, p.idesc, acc0);
#pragma unroll
            for (int k = 1; k < GEMM_BK / 16; ++k) mma_f16_ss_cg<CG>(d_tmem, ad + k * a_step, bd + k * b_step, p.idesc, 1u);
            tc_commit_cg<CG>(&empty_bar[stage]);
          }
          __syncwarp();
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok && leader) tc_commit_cg<CG>(&acc_full[as]);
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5)
    const int quarter = warp & 3;  // TMEM lane quarter this warp may read
    uint8_t* patch = out_area + (warp - 2) * 8192;
    int it = 0, ob = 0;            // tiles done; output patch in use
    bool ok = true;
    for (int wi = 0; ok; ++wi) {
      TileInfo ti;
      const int got = next_work<CG>(p, wi, num_tiles, num_kb, ti);
      if (got == 0) break;
      if (got == 2) continue;
      const int as = it & 1;
      const uint32_t aphase = (it >> 1) & 1;
      ++it;
      const int m0 = ti.m0 + cta * GEMM_BM, n0 = ti.n0;
      ok = mbar_wait(&acc_full[as], aphase, abort_flag, p.status, KWU_ERR_TIMEOUT_ACC_FULL);
      ok = __all_sync(0xffffffffu, ok);  // the TMEM loads below are warp-collective
      if (!ok) break;
      tc_fence_after();
      const int row0 = m0 + quarter * 32;      // first output row of this warp
      const int row = row0 + lane;
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + as * 256;
      // per-row state of the cross-entropy epilogues
      float run_max = -INFINITY, run_sum = 0.f, tgt = 0.f;
      bool tgt_here = false;
      int label = -1;
      float row_lse = 0.f, row_cp = 0.f, row_cy = 0.f;
      if (EPI != EPI_STORE && row < p.M) {
        label = p.labels ? p.labels[row] : -1;
        if (EPI == EPI_DLOGITS) {
          row_lse = p.lse[row];
          row_cp = p.coef_p[row];
          row_cy = p.coef_y[row];
        }
      }
      const int ncols = min(BN, p.N - n0);     // columns of this tile that exist
      const bool tma_rows = row0 < p.M;        // a warp whose rows all lie below the matrix stores nothing
#pragma unroll 1
      for (int c = 0; c * 32 < ncols; ++c) {
        uint32_t r[32];
        tmem_ld_x32(t_row + c * 32, r);
        tmem_ld_wait();
        const int col0 = n0 + c * 32;
        if (EPI == EPI_LSE) {
          if (row < p.M) {
            // the column bound and the label only matter in one chunk of a row each: handled outside the
            // per-element loops, which are a scale, a maximum, and one fused multiply-add + exp2 per logit
            if (col0 + 32 > p.N) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + j >= p.N) r[j] = __float_as_uint(-INFINITY);
            }
            if (label >= col0 && label < col0 + 32) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + j == label) { tgt = __uint_as_float(r[j]) * p.alpha; tgt_here = true; }
            }
            float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int j = 0; j < 32; ++j) m4[j & 3] = fmaxf(m4[j & 3], __uint_as_float(r[j]));
            // alpha > 0 commutes with the maximum
            const float cmax = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * p.alpha;
            const float nm = fmaxf(run_max, cmax);
            const float a2 = p.alpha * 1.4426950408889634f, nb = -nm * 1.4426950408889634f;
            const uint64_t a2p = pack_f32x2(a2, a2), nbp = pack_f32x2(nb, nb);
            uint64_t acc2[2] = {pack_f32x2(0.f, 0.f), pack_f32x2(0.f, 0.f)};
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              float e0, e1;
              unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])), a2p, nbp), e0, e1);
              acc2[(j >> 1) & 1] = add_f32x2(acc2[(j >> 1) & 1], pack_f32x2(fast_exp2(e0), fast_exp2(e1)));
            }
            float c0, c1, c2, c3;
            unpack_f32x2(acc2[0], c0, c1);
            unpack_f32x2(acc2[1], c2, c3);
            run_sum = run_sum * fast_exp2((run_max - nm) * 1.4426950408889634f) + ((c0 + c1) + (c2 + c3));
            run_max = nm;
          }
        } else {
          float f[32];
          if (EPI == EPI_DLOGITS) {
            // g = coef_p * exp2(acc * alpha * log2e - lse * log2e); the one-hot term is applied afterwards, in
            // the one chunk of the row that holds the label
            const float a2 = p.alpha * 1.4426950408889634f, nb = -row_lse * 1.4426950408889634f;
            const uint64_t a2p = pack_f32x2(a2, a2), nbp = pack_f32x2(nb, nb), cpp = pack_f32x2(row_cp, row_cp);
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              float e0, e1;
              unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])), a2p, nbp), e0, e1);
              unpack_f32x2(mul_f32x2(pack_f32x2(fast_exp2(e0), fast_exp2(e1)), cpp), f[j], f[j + 1]);
            }
            if (label >= col0 && label < col0 + 32) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + j == label) f[j] -= row_cy;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(r[j]) * p.alpha;
            if (p.diag != 0.f) {
              const int d = row % p.c_group_rows - col0;
              if (__any_sync(0xffffffffu, d >= 0 && d < 32)) {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (j == d) f[j] += p.diag;
              }
            }
          }
          if (p.out_mode == OUT_TMA_BF16) {
            // 64-column boxes: 128-byte rows, 16-byte units XORed with the row (the TMA's 128-byte swizzle);
            // 32-column boxes: 64-byte rows, units XORed with row / 2 (its 64-byte swizzle). Conflict-free both ways.
            const bool wide = p.out_cols == 64;
            const bool first = !wide || (c & 1) == 0;      // first half of a box: the patch must be free again
            if (first) {
              if (lane == 0) tma_store_wait_read<1>();
              __syncwarp();
            }
            uint8_t* dst = patch + ob * 4096 + lane * (wide ? 128 : 64);
            const int unit0 = wide ? (c & 1) * 4 : 0, key = wide ? (lane & 7) : ((lane >> 1) & 3);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4 v;
              v.x = pack_bf16(f[8 * j + 0], f[8 * j + 1]);
              v.y = pack_bf16(f[8 * j + 2], f[8 * j + 3]);
              v.z = pack_bf16(f[8 * j + 4], f[8 * j + 5]);
              v.w = pack_bf16(f[8 * j + 6], f[8 * j + 7]);
              *reinterpret_cast<uint4*>(dst + (((unit0 + j) ^ key) << 4)) = v;
            }
            if (!wide || (c & 1) || (c + 1) * 32 >= ncols) {   // box complete (a last half box is cut at N by the TMA)
              fence_async_proxy();
              __syncwarp();
              if (lane == 0 && tma_rows) {
                tma_store_2d(&tmC, patch + ob * 4096, wide ? n0 + (c & ~1) * 32 : col0, row0 + ti.c_row_off);
                tma_store_commit();
              }
              ob ^= 1;
            }
          } else if (p.out_mode == OUT_TMA_F32 || p.out_mode == OUT_TMA_ADD) {
            if (lane == 0) tma_store_wait_read<1>();
            __syncwarp();
            uint8_t* dst = patch + ob * 4096 + lane * 128;
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<float4*>(dst + ((j ^ (lane & 7)) << 4)) = make_float4(f[4 * j], f[4 * j + 1], f[4 * j + 2], f[4 * j + 3]);
            fence_async_proxy();
            __syncwarp();
            if (lane == 0 && tma_rows) {
              if (p.out_mode == OUT_TMA_ADD)
                tma_reduce_add_2d(&tmC, patch + ob * 4096, col0, row0 + ti.c_row_off);
              else
                tma_store_2d(&tmC, patch + ob * 4096, col0, row0 + ti.c_row_off);
              tma_store_commit();
            }
            ob ^= 1;
          } else if (row < p.M) {
            const int valid = min(32, p.N - col0);
            const size_t at = static_cast<size_t>(row + ti.c_row_off) * p.ldc + col0;
            if (p.out_fp32) {
              float* dst = reinterpret_cast<float*>(Cbase) + at;
              // several CTAs may add into one element (split tail)
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (j < valid) {
                  if (p.accumulate) atomicAdd(dst + j, f[j]); else dst[j] = f[j];
                }
            } else {
              __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(Cbase) + at;
              bool vec = valid == 32 && (p.ldc & 7) == 0 && (reinterpret_cast<uintptr_t>(Cbase) & 15) == 0;
              bool drop = false;
              if (p.row_ptrs) {
                const long long base = p.row_ptrs[row];
                drop = base == 0;
                dst = reinterpret_cast<__nv_bfloat16*>(base) + col0;
                vec = valid == 32 && (base & 15) == 0;
              }
              if (!drop && vec) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  float* g = f + 8 * j;
                  uint4* d4 = reinterpret_cast<uint4*>(dst) + j;
                  if (p.accumulate) {
                    const uint4 o = *d4;
                    const float2 o0 = unpack_bf16(o.x), o1 = unpack_bf16(o.y), o2 = unpack_bf16(o.z), o3 = unpack_bf16(o.w);
                    g[0] += o0.x; g[1] += o0.y; g[2] += o1.x; g[3] += o1.y;
                    g[4] += o2.x; g[5] += o2.y; g[6] += o3.x; g[7] += o3.y;
                  }
                  uint4 v;
                  v.x = pack_bf16(g[0], g[1]);
                  v.y = pack_bf16(g[2], g[3]);
                  v.z = pack_bf16(g[4], g[5]);
                  v.w = pack_bf16(g[6], g[7]);
                  *d4 = v;
                }
              } else if (!drop) {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (j < valid) dst[j] = __float2bfloat16(p.accumulate ? f[j] + __bfloat162float(dst[j]) : f[j]);
              }
            }
          }
        }
      }
      if (EPI == EPI_LSE && row < p.M) {
        p.partial[static_cast<size_t>(n0 / BN) * p.M + row] = make_float2(run_max, run_sum);
        if (tgt_here) p.target_logit[row] = tgt;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2) mbar_arrive_cluster(mapa_shared(smem_u32(&acc_empty[as]), 0));
        else mbar_arrive(&acc_empty[as]);
      }
    }
    if (lane == 0) tma_store_wait_read<0>();   // the patches are read before this CTA's shared memory goes away
  }

  // ---------------------------------------------------------------- tear-down
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // give copies that are still in flight time to land before the CTA's smem goes away
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  if (CG == 2) cluster_sync();   // the pair leaves together: its barriers and TMEM are used from both sides
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_cg<CG>(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------ products of a few rows
// C[m, n] = alpha * sum_k A[m, k] B[n, k] for M <= 16, both K-major: the step of a decode. It is a stream of B through the
// chip once; a 128-row tile spends its time on the serial k-blocks of a few CTAs instead. Mean of the products of a decode
// step, tile / this, us: 17 layers of 768 wide and the 65536-wide head, one row 8.8 / 4.1; 22 layers of 1280, eight rows
// 12.4 / 6.1. The head alone (2 x 65536 x 1280) takes 37.6 us, 4.5 TB/s.
// A CTA owns 16 rows of B, its eight warps a slice of the contraction each. B's rows are the M side of
// mma.m16n8k16 and A's rows (up to 8 per product) the N side. A lane loads 16 bytes of rows g and g + 8 of B and of row g
// of A at the same eight k's; the products take them as four pairs, so the order of k inside a 32-wide step is permuted
// alike on both sides. Up to four steps of loads are in flight per lane. The eight partial sums meet in shared memory in
// a fixed order.
constexpr int FEW_WARPS = 8, FEW_UNROLL = 4;

__device__ __forceinline__ void mma_m16n8k16_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                  uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int HALVES>   // 8 rows of A each
__global__ void __launch_bounds__(FEW_WARPS * 32)
gemm_few_rows_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ B, void* __restrict__ C, int M,
                     int N, int K, int lda, int ldb, int ldc, int out_fp32, float alpha) {
  pdl_sync();   // nothing of the previous kernel is read above this line
  __shared__ float s_part[FEW_WARPS][HALVES * 8][17];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * 16;
  const int steps = (K + 31) / 32;
  const int s_begin = steps * warp / FEW_WARPS, s_end = steps * (warp + 1) / FEW_WARPS;
  const __nv_bfloat16* b0 = B + static_cast<size_t>(n0 + g) * ldb + 8 * t;
  const __nv_bfloat16* b1 = b0 + static_cast<size_t>(8) * ldb;
  const bool n_lo = n0 + g < N, n_hi = n0 + g + 8 < N;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  float acc[HALVES][4];
#pragma unroll
  for (int h = 0; h < HALVES; ++h)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[h][i] = 0.f;
  for (int s = s_begin; s < s_end; s += FEW_UNROLL) {
    uint4 w0[FEW_UNROLL], w1[FEW_UNROLL], x[FEW_UNROLL][HALVES];
#pragma unroll
    for (int u = 0; u < FEW_UNROLL; ++u) {
      const int k = (s + u) * 32;
      const bool in = s + u < s_end && k + 8 * t < K;     // K is a multiple of 8
      w0[u] = in && n_lo ? __ldg(reinterpret_cast<const uint4*>(b0 + k)) : zero;
      w1[u] = in && n_hi ? __ldg(reinterpret_cast<const uint4*>(b1 + k)) : zero;
#pragma unroll
      for (int h = 0; h < HALVES; ++h) {
        const int m = 8 * h + g;
        x[u][h] = in && m < M ? __ldg(reinterpret_cast<const uint4*>(A + static_cast<size_t>(m) * lda + k + 8 * t)) : zero;
      }
    }
#pragma unroll
    for (int u = 0; u < FEW_UNROLL; ++u)
#pragma unroll
      for (int h = 0; h < HALVES; ++h) {
        mma_m16n8k16_bf16(acc[h], w0[u].x, w1[u].x, w0[u].y, w1[u].y, x[u][h].x, x[u][h].y);
        mma_m16n8k16_bf16(acc[h], w0[u].z, w1[u].z, w0[u].w, w1[u].w, x[u][h].z, x[u][h].w);
      }
  }
  // acc: rows g, g + 8 of B by rows 2 t, 2 t + 1 of A
#pragma unroll
  for (int h = 0; h < HALVES; ++h) {
    s_part[warp][8 * h + 2 * t][g] = acc[h][0];
    s_part[warp][8 * h + 2 * t + 1][g] = acc[h][1];
    s_part[warp][8 * h + 2 * t][g + 8] = acc[h][2];
    s_part[warp][8 * h + 2 * t + 1][g + 8] = acc[h][3];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < HALVES * 128; i += FEW_WARPS * 32) {
    const int m = i >> 4, n = i & 15;
    if (m >= M || n0 + n >= N) continue;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < FEW_WARPS; ++w) v += s_part[w][m][n];
    v *= alpha;
    const size_t at = static_cast<size_t>(m) * ldc + n0 + n;
    if (out_fp32) reinterpret_cast<float*>(C)[at] = v;
    else reinterpret_cast<__nv_bfloat16*>(C)[at] = __float2bfloat16(v);
  }
}

// ------------------------------------------------------------------ host launcher
static int num_sms() {
  static int n = 0;
  if (!n) {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    n = v > 0 ? v : 148;
  }
  return n;
}

struct GroupArgs {
  int mode = 0;
  const int4* tiles = nullptr;
  const int* offsets = nullptr;
  int b_rows = 0;
  int num_groups = 1;
  int c_rows = 0;
  int row_tiles = 0;  // mode 1: number of entries in `tiles`
  float diag = 0.f;   // mode 3
  const long long* row_ptrs = nullptr;
};

struct EpiArgs {
  const int* labels = nullptr;
  float2* partial = nullptr;
  float* target_logit = nullptr;
  const float* lse = nullptr;
  const float* coef_p = nullptr;
  const float* coef_y = nullptr;
};

template <int CG, bool A_MN, bool B_MN, int EPI>
static int launch_gemm(int BN, const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb,
                       int ldc, int out_fp32, int accumulate, float alpha, int max_ctas,
                       cudaStream_t stream, int* status, const EpiArgs& ea = EpiArgs(),
                       const GroupArgs& ga = GroupArgs(), int b_total_rows = 0, int splits = 1, bool even_ranges = false) {
  CUtensorMap tmA, tmB, tmC;
  int rc;
  if (!A_MN)
    rc = encode_tmap_2d(&tmA, A, ELEM_BF16, M, K, lda, GEMM_BM, GEMM_BK, CU_TENSOR_MAP_SWIZZLE_128B);
  else
    rc = encode_tmap_2d(&tmA, A, ELEM_BF16, K, M, lda, GEMM_BK, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  // with expert groups B is the stack of all experts' matrices: b_total_rows rows in storage order
  if (!B_MN)
    rc = encode_tmap_2d(&tmB, B, ELEM_BF16, b_total_rows ? b_total_rows : N, K, ldb, BN / CG, GEMM_BK, CU_TENSOR_MAP_SWIZZLE_128B);
  else
    rc = encode_tmap_2d(&tmB, B, ELEM_BF16, b_total_rows ? b_total_rows : K, N, ldb, GEMM_BK, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;

  GemmParams p;
  p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.bn = BN;
  p.out_fp32 = out_fp32; p.accumulate = accumulate; p.alpha = alpha;
  // K-major, 128B swizzle: rows are 128 B, 8-row groups 1024 B apart, K advances 32 B per MMA.
  // MN-major, 128B swizzle: 64-element chunks along MN are whole 8 KB boxes, 8-row K groups are
  // 1024 B apart, K advances 16 rows = 2048 B per MMA.
  p.a_lbo = A_MN ? 8192 : 16; p.a_sbo = 1024; p.a_kadv = A_MN ? 2048 : 32;
  p.b_lbo = B_MN ? 8192 : 16; p.b_sbo = 1024; p.b_kadv = B_MN ? 2048 : 32;
  p.idesc = make_idesc_f16(GEMM_BM * CG, BN, 1, A_MN ? 1 : 0, B_MN ? 1 : 0);
  p.b_chunks = (BN / CG + 63) / 64;
  p.stage_bytes = GEMM_A_BYTES + (B_MN ? p.b_chunks * 64 : BN / CG) * GEMM_BK * 2;
  p.stages = (GEMM_SMEM_MAX - 1024 - GEMM_BAR_BYTES - GEMM_OUT_BYTES) / static_cast<int>(p.stage_bytes);
  if (p.stages > GEMM_MAX_STAGES) p.stages = GEMM_MAX_STAGES;
  p.tiles_m = ga.mode == 1 ? ga.row_tiles : (M + GEMM_BM * CG - 1) / (GEMM_BM * CG);
  p.tiles_n = (N + BN - 1) / BN;
  p.status = status;
  p.group_mode = ga.mode; p.group_tiles = ga.tiles; p.group_offsets = ga.offsets;
  p.group_b_rows = ga.b_rows; p.num_groups = ga.num_groups; p.c_group_rows = ga.c_rows; p.diag = ga.diag;
  p.row_ptrs = (EPI == EPI_STORE && !out_fp32) ? ga.row_ptrs : nullptr;
  p.labels = ea.labels; p.partial = ea.partial; p.target_logit = ea.target_logit;
  p.lse = ea.lse; p.coef_p = ea.coef_p; p.coef_y = ea.coef_y;

  // TMA addresses the output when its base and pitch are 16-byte multiples; rows of one expert's gradient must fill
  // whole tiles, or the store box would reach into the next expert's rows
  const bool can_tma = EPI != EPI_LSE && (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (ldc * (out_fp32 ? 4 : 2)) % 16 == 0 &&
                       !p.row_ptrs && (ga.mode != 2 || M % (GEMM_BM * CG) == 0);
  p.out_mode = OUT_DIRECT;
  p.out_cols = (BN % 64) ? 32 : 64;
  if (can_tma && (out_fp32 || !accumulate))
    p.out_mode = out_fp32 ? (accumulate ? OUT_TMA_ADD : OUT_TMA_F32) : OUT_TMA_BF16;
  if (p.out_mode != OUT_DIRECT) {
    const uint64_t c_rows = ga.mode == 2 ? static_cast<uint64_t>(ga.num_groups) * ga.c_rows : M;
    if (out_fp32)
      rc = encode_tmap_2d(&tmC, C, ELEM_F32, c_rows, N, ldc, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B);
    else
      rc = encode_tmap_2d(&tmC, C, ELEM_BF16, c_rows, N, ldc, 32, p.out_cols,
                          p.out_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc) return rc;
  } else {
    tmC = tmA;   // not read
  }

  auto kern = gemm_bf16_kernel<CG, A_MN, B_MN, EPI>;
  static PerDeviceOnce attr_set;
  if (attr_set.pending()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM_MAX);
    if (e != cudaSuccess) {
      set_last_error("cudaFuncSetAttribute: %s", cudaGetErrorString(e));
      return 10;
    }
    attr_set.mark();
  }
  long tiles = static_cast<long>(p.tiles_m) * p.tiles_n * (ga.mode == 2 ? ga.num_groups : 1);
  int units = num_sms();
  if (max_ctas > 0 && max_ctas < units) units = max_ctas;
  units = units / CG > 0 ? units / CG : 1;
  p.full_tiles = static_cast<int>(tiles);
  p.tail_tiles = 0;
  p.splits = 1;
  if (splits > 1 && ga.mode == 0 && out_fp32 && accumulate && EPI == EPI_STORE) {
    p.full_tiles = static_cast<int>(tiles - tiles % units);
    p.tail_tiles = static_cast<int>(tiles % units);
    p.splits = splits;
  }
  const long items = p.full_tiles + static_cast<long>(p.tail_tiles) * p.splits;
  p.ranges = 0;
  if (CG == 1 && even_ranges && ga.mode == 0 && out_fp32 && accumulate && EPI == EPI_STORE) {
    const long long all = tiles * static_cast<long long>((K + GEMM_BK - 1) / GEMM_BK);
    p.ranges = units = static_cast<int>(all < units ? all : units);
  } else if (items < units) {
    units = static_cast<int>(items);
  }
  const size_t smem = 1024 + GEMM_BAR_BYTES + GEMM_OUT_BYTES + static_cast<size_t>(p.stages) * p.stage_bytes;
  launch_cluster(kern, dim3(units * CG), dim3(GEMM_THREADS), CG, smem, stream, tmA, tmB, tmC, C, p); kwu::count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_error("gemm launch: %s", cudaGetErrorString(e));
    return 11;
  }
  return 0;
}

struct TilePick {
  int cg, bn, splits;
};

// Tile (one CTA or a pair, width) and split of the tail round with the least predicted time. Measured on one B200
// (8192^3, 4096 x 7168 x 1280, 16384 x 1536 x 8192 and 2560 x 1536 x 16384, operands rotating through four buffers): a
// 64-deep k-block takes a pair 0.070 us + 1.25 ns per column with B K-major, 0.25 us + 0.47 ns with B MN-major (its
// boxes are 64 columns of each CTA whatever the width), and a single CTA 0.19 us + 0.9 ns; every round of the
// persistent grid takes another 0.55 us (accumulator hand-over, pipeline refill). The rounds decide
// between widths: 4096 x 1280 is two rounds of 160 columns or two of 256. fp32 C += may cut the tiles of its last,
// partly empty round along the contraction (no cut below 4 k-blocks).
static TilePick pick_tile(int M, int N, int K, bool b_mn, bool can_split, int tiles_m128 = 0, int max_cg = 2, int max_ctas = 0) {
  int sms = num_sms();
  if (max_ctas > 0 && max_ctas < sms) sms = max_ctas;
  const int nkb = (K + GEMM_BK - 1) / GEMM_BK;
  TilePick best{1, 128, 1};
  double best_cost = 1e30;
  for (int cg = 1; cg <= max_cg; ++cg) {
    if (cg == 2 && (M <= GEMM_BM || sms < 2)) continue;
    const long tm = tiles_m128 ? tiles_m128 : (M + GEMM_BM * cg - 1) / (GEMM_BM * cg);
    const int units = sms / cg;
    for (int bn = cg == 1 ? 64 : 128; bn <= 256; bn += 32) {
      const long tiles = tm * ((N + bn - 1) / bn);
      const double per_kb = cg == 1 ? 0.19 + 0.0009 * bn : (b_mn ? 0.25 + 0.00047 * bn : 0.070 + 0.00125 * bn);
      const long full = tiles / units, tail = tiles % units;
      double cost = full * (nkb * per_kb + 0.55);
      int splits = 1;
      if (tail > 0) {
        if (can_split) {
          splits = static_cast<int>(units / tail);
          if (splits > nkb / 4) splits = nkb / 4;
          if (splits < 1) splits = 1;
        }
        cost += (nkb + splits - 1) / splits * per_kb + 0.55;
      }
      if (cost < best_cost - 1e-9) { best_cost = cost; best = {cg, bn, splits}; }
    }
  }
  return best;
}

}  // namespace kwu

// C[M,N] (+)= alpha * op(A) op(B). a_mn / b_mn select the storage described at the top of the file.
// lda/ldb/ldc are row pitches in elements of the STORED matrices. bn: 0 = choose, 64..256 = a tile of one CTA that
// wide (multiples of 32), 1000 + width = a tile of a CTA pair.
KWU_API int kwu_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb,
                          int ldc, int a_mn, int b_mn, int out_fp32, int accumulate, float alpha,
                          int bn, int max_ctas, void* stream, int* status) {
  using namespace kwu;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // up to 16 rows against a K-major B are a stream of B, which needs no tensor maps; 16-byte loads want aligned rows
  if (bn == 0 && max_ctas == 0 && M <= 16 && !a_mn && !b_mn && !accumulate && K % 8 == 0 && lda % 8 == 0 && ldb % 8 == 0 &&
      ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15) == 0) {
    auto kern = M <= 8 ? gemm_few_rows_kernel<1> : gemm_few_rows_kernel<2>;
    launch_k(kern, dim3((N + 15) / 16), dim3(FEW_WARPS * 32), 0, st, (const __nv_bfloat16*)A, (const __nv_bfloat16*)B, C, M, N, K,
             lda, ldb, ldc, out_fp32, alpha); kwu::count_launch();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { set_last_error("gemm_few_rows launch: %s", cudaGetErrorString(e)); return 11; }
    return 0;
  }
  TilePick pick{bn > 1000 ? 2 : 1, bn > 1000 ? bn - 1000 : bn, 1};
  // The pieces of a cut tile meet in C in the order in which they finish, so a cut costs the fixed order of the sum. Below
  // K = 1024 no tile is cut: it would save at most a few microseconds, and callers rest on the order there (the gate logits
  // of routed layers up to 1023 wide, head plus remainder of the gate matrix: near ties between experts would fall
  // differently from run to run).
  if (bn == 0) pick = pick_tile(M, N, K, b_mn != 0, out_fp32 && accumulate && K >= 1024, 0, 2, max_ctas);
  // dx += dy W with a long contraction is the loss head's input gradient, 65536 deep, on which every layer's gradient
  // rests: rounded to bf16 and re-quantised to e4m3 below, one bit of its sums becomes several percent of noise in the
  // gradients of the first layers. So its sums stay cut the way they always were, into one even range of 128 x 256 tiles'
  // k-blocks per SM: 4096 x 1280 x 65536 in 489 us (683 with the ranges walked tile by
  // tile and per-lane additions, 437 on pairs).
  const bool even = bn == 0 && out_fp32 && accumulate && !a_mn && b_mn && K >= 1024 &&
                    (static_cast<long>((M + GEMM_BM - 1) / GEMM_BM) * ((N + 255) / 256)) % num_sms() != 0;
  if (even) pick = {1, 256, 1};
  if (pick.bn < 64 || pick.bn > 256 || pick.bn % 32) {
    set_last_error("kwu_gemm_bf16: tile width %d", pick.bn);
    return 20;
  }
#define KWU_GEMM_CASE(cgv, amn, bmn)                                                              \
  if (pick.cg == cgv && a_mn == amn && b_mn == bmn)                                               \
    return launch_gemm<cgv, amn != 0, bmn != 0, EPI_STORE>(pick.bn, A, B, C, M, N, K, lda, ldb, ldc, out_fp32,        \
                                                accumulate, alpha, max_ctas, st, status, EpiArgs(), \
                                                GroupArgs(), 0, pick.splits, even);
  KWU_GEMM_CASE(1, 0, 0) KWU_GEMM_CASE(1, 0, 1) KWU_GEMM_CASE(1, 1, 0) KWU_GEMM_CASE(1, 1, 1)
  KWU_GEMM_CASE(2, 0, 0) KWU_GEMM_CASE(2, 0, 1) KWU_GEMM_CASE(2, 1, 0) KWU_GEMM_CASE(2, 1, 1)
#undef KWU_GEMM_CASE
  set_last_error("kwu_gemm_bf16: unsupported variant");
  return 20;
}

// ------------------------------------------------------------------ fused linear cross-entropy
// Forward: logits = alpha * h W^T are never written. Every (row, 256-column tile) leaves one
// (max, sum-exp) pair in partial[tile, row]; the target logit of each row is captured on the way.
// kwu_ce_combine then folds the partials into lse[row].
KWU_API int kwu_ce_tiles_n(int V) { return (V + 255) / 256; }

KWU_API int kwu_gemm_lse(const void* H, const void* W, int T, int V, int D, int ldh, int ldw,
                         const int* labels, void* partial, float* target_logit, float alpha,
                         void* stream, int* status) {
  using namespace kwu;
  if (T <= 0) return 0;
  EpiArgs ea;
  ea.labels = labels;
  ea.partial = reinterpret_cast<float2*>(partial);
  ea.target_logit = target_logit;
  // the partial table has one column per 256 logits, so the width is fixed
  if (T > GEMM_BM)
    return launch_gemm<2, false, false, EPI_LSE>(256, H, W, nullptr, T, V, D, ldh, ldw, 0, 0, 0, alpha, 0,
                                                 reinterpret_cast<cudaStream_t>(stream), status, ea);
  return launch_gemm<1, false, false, EPI_LSE>(256, H, W, nullptr, T, V, D, ldh, ldw, 0, 0, 0, alpha, 0,
                                               reinterpret_cast<cudaStream_t>(stream), status, ea);
}

// Backward recompute: dlogits[row, col] = coef_p[row] * exp(logit - lse[row]) - coef_y[row] * onehot,
// written as bf16 with row pitch ldd.
KWU_API int kwu_gemm_dlogits(const void* H, const void* W, void* dlogits, int T, int V, int D, int ldh,
                             int ldw, int ldd, const int* labels, const float* lse,
                             const float* coef_p, const float* coef_y, float alpha, void* stream,
                             int* status) {
  using namespace kwu;
  if (T <= 0) return 0;
  EpiArgs ea;
  ea.labels = labels;
  ea.lse = lse;
  ea.coef_p = coef_p;
  ea.coef_y = coef_y;
  if (T > GEMM_BM)
    return launch_gemm<2, false, false, EPI_DLOGITS>(256, H, W, dlogits, T, V, D, ldh, ldw, ldd, 0, 0, alpha,
                                                     0, reinterpret_cast<cudaStream_t>(stream), status, ea);
  return launch_gemm<1, false, false, EPI_DLOGITS>(256, H, W, dlogits, T, V, D, ldh, ldw, ldd, 0, 0, alpha,
                                                   0, reinterpret_cast<cudaStream_t>(stream), status, ea);
}

namespace kwu {
// One thread folds a row's partials in order of the tiles (every gradient of the step rests on the last bit of this sum
// through bf16 and e4m3 roundings, so its order stays). A block is one warp, so that 4096 rows reach 128 SMs, and a batch
// of partials is fetched ahead of its use: 128 rows a block and one load behind the other took 40 us at 8190 rows and 256
// tiles, 13 like this (6 with the tiles folded in slices).
constexpr int CE_ROWS = 32, CE_AHEAD = 32;
__global__ void __launch_bounds__(CE_ROWS) ce_combine_kernel(const float2* __restrict__ partial, int tiles_n, int M,
                                                             float* __restrict__ lse) {
  const int row = blockIdx.x * CE_ROWS + threadIdx.x;
  if (row >= M) return;
  float m = -INFINITY, s = 0.f;
  auto fold = [&](const float2& v) {
    const float nm = fmaxf(m, v.x);
    s = s * __expf(m - nm) + v.y * __expf(v.x - nm);
    m = nm;
  };
  const float2* at = partial + row;
  const int whole = tiles_n / CE_AHEAD * CE_AHEAD;
  float2 next[CE_AHEAD];
  if (whole) {
#pragma unroll
    for (int i = 0; i < CE_AHEAD; ++i) next[i] = at[static_cast<size_t>(i) * M];
  }
  for (int t0 = 0; t0 < whole; t0 += CE_AHEAD) {
    float2 now[CE_AHEAD];
#pragma unroll
    for (int i = 0; i < CE_AHEAD; ++i) now[i] = next[i];
    if (t0 + CE_AHEAD < whole) {
#pragma unroll
      for (int i = 0; i < CE_AHEAD; ++i) next[i] = at[static_cast<size_t>(t0 + CE_AHEAD + i) * M];
    }
#pragma unroll
    for (int i = 0; i < CE_AHEAD; ++i) fold(now[i]);
  }
  for (int t = whole; t < tiles_n; ++t) fold(at[static_cast<size_t>(t) * M]);
  lse[row] = m + __logf(s);
}
}  // namespace kwu

KWU_API int kwu_ce_combine(const void* partial, int tiles_n, int M, float* lse, void* stream) {
  if (M <= 0) return 0;
  kwu::ce_combine_kernel<<<(M + kwu::CE_ROWS - 1) / kwu::CE_ROWS, kwu::CE_ROWS, 0,
                           reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const float2*>(partial), tiles_n, M, lse); kwu::count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { kwu::set_last_error("ce_combine launch: %s", cudaGetErrorString(e)); return 11; }
  return 0;
}


// ------------------------------------------------------------------ grouped (mixture-of-experts) GEMMs
// Rows grouped by expert (forward and dgrad):  C[rows of tile] = A[rows of tile] * op(B[expert]).
//   A (M_pad, K) K-major. b_mn = 0: B is (E*N, K), expert e owns rows [e*N, (e+1)*N)  -> y = x W_e^T
//                         b_mn = 1: B is (E*Kc, N) with Kc = K,  expert e owns rows [e*K, (e+1)*K) -> dx = dy W_e
//   tiles: (row_tiles, 4) int32 entries (m0, expert, valid, unused) built by kwu_moe_plan.
//   row_ptrs (optional, bf16 output only): per output row the byte address it is stored at (0 = skip the row);
//   C is then not written.
KWU_API int kwu_gemm_bf16_grouped_rows(const void* A, const void* B, void* C, int M_pad, int N, int K, int lda,
                                       int ldb, int ldc, int b_mn, int num_experts, const void* tiles,
                                       int row_tiles, int out_fp32, const long long* row_ptrs, void* stream,
                                       int* status) {
  using namespace kwu;
  if (M_pad <= 0 || row_tiles <= 0) return 0;
  GroupArgs ga;
  ga.mode = 1;
  ga.row_ptrs = row_ptrs;
  ga.tiles = reinterpret_cast<const int4*>(tiles);
  ga.row_tiles = row_tiles;
  ga.b_rows = b_mn ? K : N;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int total_rows = num_experts * ga.b_rows;
  // tiles stay inside one expert's 128-aligned rows, so a single CTA each
  const int bn = pick_tile(M_pad, N, K, b_mn != 0, false, row_tiles, 1).bn;
  if (b_mn)
    return launch_gemm<1, false, true, EPI_STORE>(bn, A, B, C, M_pad, N, K, lda, ldb, ldc, out_fp32, 0, 1.f, 0, st, status,
                                         EpiArgs(), ga, total_rows);
  return launch_gemm<1, false, false, EPI_STORE>(bn, A, B, C, M_pad, N, K, lda, ldb, ldc, out_fp32, 0, 1.f, 0, st, status,
                                        EpiArgs(), ga, total_rows);
}

// A batch of products of one size: C[i] = alpha * A[i] op(B[i]) + diag * I, all bf16 and contiguous. A[i] (M, K) with M a
// multiple of 128; B[i] is (N, K) with b_mn = 0 (product with its transpose) or (K, N) with b_mn = 1. Pairs of CTAs where
// M is a multiple of 256, so that a pair's rows stay inside one matrix.
KWU_API int kwu_gemm_bf16_batched(const void* A, const void* B, void* C, int batch, int M, int N, int K, int b_mn, float alpha,
                                  float diag, void* stream, int* status) {
  using namespace kwu;
  if (batch <= 0 || M <= 0 || N <= 0 || K <= 0) return 0;
  if (M % GEMM_BM) { set_last_error("gemm_bf16_batched: M must be a multiple of 128 (got %d)", M); return 7; }
  if (static_cast<long long>(batch) * M > 0x7fffffffLL || static_cast<long long>(batch) * (b_mn ? K : N) > 0x7fffffffLL) {
    set_last_error("gemm_bf16_batched: too many rows");
    return 7;
  }
  GroupArgs ga;
  ga.mode = 3;
  ga.b_rows = b_mn ? K : N;
  ga.c_rows = M;
  ga.diag = diag;
  const int rows = batch * M, b_rows = batch * ga.b_rows, ldb = b_mn ? N : K;
  const TilePick pick = pick_tile(rows, N, K, b_mn != 0, false, 0, M % (2 * GEMM_BM) == 0 ? 2 : 1);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
#define KWU_BATCHED(cgv, bmn)                                                                                      \
  if (pick.cg == cgv && (b_mn != 0) == bmn)                                                                        \
    return launch_gemm<cgv, false, bmn, EPI_STORE>(pick.bn, A, B, C, rows, N, K, K, ldb, N, 0, 0, alpha, 0, st, status, \
                                                   EpiArgs(), ga, b_rows)
  KWU_BATCHED(1, false); KWU_BATCHED(1, true); KWU_BATCHED(2, false); KWU_BATCHED(2, true);
#undef KWU_BATCHED
  return 20;
}

// Contraction grouped by expert (weight gradients): dW[e] (N_out, K_out) (+)= dY[rows_e]^T X[rows_e].
//   dY (M_pad, N_out) and X (M_pad, K_out) row-major; offsets: (E+1) padded row offsets (multiples of 128).
KWU_API int kwu_gemm_bf16_grouped_wgrad(const void* dY, const void* X, void* dW, int M_pad, int N_out, int K_out,
                                        int lddy, int ldx, int num_experts, const int* offsets, int out_fp32,
                                        int accumulate, void* stream, int* status) {
  using namespace kwu;
  if (M_pad <= 0 || num_experts <= 0) return 0;
  GroupArgs ga;
  ga.mode = 2;
  ga.offsets = offsets;
  ga.num_groups = num_experts;
  ga.c_rows = N_out;
  // a pair's 256 rows must not reach into the next expert's gradient
  const int cgs = N_out % (2 * GEMM_BM) == 0 ? 2 : 1;
  const int rows = (N_out + GEMM_BM - 1) / GEMM_BM * GEMM_BM * num_experts;
  const TilePick pick = pick_tile(rows, K_out, M_pad / num_experts + GEMM_BK, true, false, 0, cgs);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (pick.cg == 2)
    return launch_gemm<2, true, true, EPI_STORE>(pick.bn, dY, X, dW, N_out, K_out, M_pad, lddy, ldx, K_out, out_fp32,
                                                 accumulate, 1.f, 0, st, status, EpiArgs(), ga, 0);
  return launch_gemm<1, true, true, EPI_STORE>(pick.bn, dY, X, dW, N_out, K_out, M_pad, lddy, ldx, K_out, out_fp32,
                                               accumulate, 1.f, 0, st, status, EpiArgs(), ga, 0);
}
