// MXFP8: e4m3 values with one UE8M0 (power-of-two) scale per 32 elements along the contraction axis.
//
//   kwu_mxfp8_quantize     (M,K) bf16 -> (M,K) e4m3 + scales, blocks along K (rows stay rows)
//   kwu_mxfp8_quantize_t   (R,C) bf16 -> (C,R) e4m3 + scales, blocks along R: the transposed copy a
//                          dgrad needs (dx = dy W contracts over the rows of W)
//   kwu_gemm_mxfp8         C[M,N] (+)= A[M,K] B[N,K]^T with tcgen05.mma.kind::mxf8f6f4.block_scale
//
// Scale layout: the one the tensor core consumes from TMEM. For every 128-row x 128-column tile of
// the matrix there is one 512-byte chunk; inside it the scale of row r, 32-block j sits at byte
// (r % 32) * 16 + (r / 32) * 4 + j. Chunks are ordered [row_tile][k_chunk]. A chunk is moved
// global -> shared by one bulk copy and shared -> TMEM by one tcgen05.cp.32x128b.warpx4.
// Exponent rule: exp = max(ceil(log2(amax / 448)), -127) (round UP so nothing saturates), amax
// clamped at 1e-30, stored as exp + 127; values are divided by 2^exp and rounded to e4m3 (satfinite).
// Rows beyond M inside the last 128-row tile get the neutral scale byte 127 so that padded rows can
// never inject a NaN scale. Reference: src/kohakuwullm/kernels/mxfp8/quantize.py:39-215 and the
// cuBLASLt path behind src/kohakuwullm/kernels/mxfp8/linear.py:49-126.
#include "common.cuh"
#include "mx_quant.cuh"

namespace kwu {

// ------------------------------------------------------------------------------------ quantise
// One thread = 8 consecutive elements; 4 threads = one 32-block; a warp covers 256 columns of a row.
__global__ void __launch_bounds__(256)
mxfp8_quantize_kernel(const __nv_bfloat16* __restrict__ x, int ldx, uint8_t* __restrict__ q, int ldq,
                      uint8_t* __restrict__ sf, int M, int K, int M_pad, int sf_bn) {
  pdl_sync();   // nothing of the previous kernel is read above this line
  const int lane = threadIdx.x & 31;
  const int n_kchunks = K >> 7;
  const int segs = (K + 255) >> 8;  // 256-column segments per row
  const long total = static_cast<long>(M_pad) * segs;
  const int wpb = blockDim.x >> 5;
  for (long w = static_cast<long>(blockIdx.x) * wpb + (threadIdx.x >> 5); w < total;
       w += static_cast<long>(gridDim.x) * wpb) {
    const int row = static_cast<int>(w / segs);
    const int col = static_cast<int>(w % segs) * 256 + lane * 8;
    const bool in_col = col < K;
    float f[8];
    if (row < M && in_col) {
      const uint4 a = *reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * ldx + col);
      float2 t;
      t = unpack_bf16(a.x); f[0] = t.x; f[1] = t.y;
      t = unpack_bf16(a.y); f[2] = t.x; f[3] = t.y;
      t = unpack_bf16(a.z); f[4] = t.x; f[5] = t.y;
      t = unpack_bf16(a.w); f[6] = t.x; f[7] = t.y;
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = 0.f;
    }
    float amax = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(f[e]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const uint32_t e8 = (row < M) ? ue8m0_from_amax(amax) : 127u;
    if (in_col) {
      if (row < M) {
        const float inv = inv_scale_from_ue8m0(e8);
        uint32_t lo = 0, hi = 0;
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          const __nv_fp8x2_storage_t a2 = __nv_cvt_float2_to_fp8x2(make_float2(f[e] * inv, f[e + 1] * inv), __NV_SATFINITE, __NV_E4M3);
          const __nv_fp8x2_storage_t b2 = __nv_cvt_float2_to_fp8x2(make_float2(f[e + 4] * inv, f[e + 5] * inv), __NV_SATFINITE, __NV_E4M3);
          lo |= static_cast<uint32_t>(a2) << (8 * e);
          hi |= static_cast<uint32_t>(b2) << (8 * e);
        }
        *reinterpret_cast<uint2*>(q + static_cast<size_t>(row) * ldq + col) = make_uint2(lo, hi);
      }
      // tile-local layout (sf_bn > 128): only real rows are written, the buffer's padding keeps its neutral fill
      if ((lane & 3) == 0 && (sf_bn <= 128 || row < M))
        sf[sf_offset_any(row, col >> 5, n_kchunks, sf_bn)] = static_cast<uint8_t>(e8);
    }
  }
}

// Transposed quantise: input (R, C) row-major, output qT (C, R) with blocks of 32 along R.
// A block handles a 32 (rows) x 64 COLS (columns) input tile; thread t owns the COLS columns from COLS t. With two, a warp
// reads whole 128-byte lines in half as many loads; rows that are not 4-byte aligned pairs take one. us, one / two columns:
// 1280 x 3584 (mean of a layer's matrices) 9.0 / 6.2, 64 experts of 768 x 1024 20.4 / 12.2.
template <int COLS>
__global__ void __launch_bounds__(64)
mxfp8_quantize_t_kernel(const __nv_bfloat16* __restrict__ x, int ldx, uint8_t* __restrict__ qT, int ldq,
                        uint8_t* __restrict__ sf, int R, int C, int C_pad, long long x_batch, long long q_batch,
                        long long sf_batch, int sf_bn) {
  pdl_sync();   // nothing of the previous kernel is read above this line
  // blockIdx.z: independent matrices (the experts of a stacked weight) at fixed strides
  x += static_cast<size_t>(blockIdx.z) * x_batch;
  qT += static_cast<size_t>(blockIdx.z) * q_batch;
  sf += static_cast<size_t>(blockIdx.z) * sf_batch;
  const int r0 = blockIdx.y * 32;
  const int c0 = (blockIdx.x * 64 + threadIdx.x) * COLS;
  if (c0 >= C_pad) return;
  const int n_kchunks = (R + 127) >> 7;  // contraction axis of the output is R
  uint32_t raw[32];                      // one bf16 in the low half, or the pair of two columns
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int r = r0 + i;
    raw[i] = 0u;
    if (r < R && c0 < C) {               // with two columns C is even: a pair is inside or outside
      const __nv_bfloat16* at = x + static_cast<size_t>(r) * ldx + c0;
      raw[i] = COLS == 2 ? *reinterpret_cast<const uint32_t*>(at) : *reinterpret_cast<const uint16_t*>(at);
    }
  }
#pragma unroll
  for (int k = 0; k < COLS; ++k) {
    const int c = c0 + k;
    auto value = [&](int i) { return __uint_as_float(k == 0 ? raw[i] << 16 : raw[i] & 0xffff0000u); };
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) amax = fmaxf(amax, fabsf(value(i)));
    const uint32_t e8 = (c < C) ? ue8m0_from_amax(amax) : 127u;
    if (r0 < R && (sf_bn <= 128 || c < C)) sf[sf_offset_any(c, r0 >> 5, n_kchunks, sf_bn)] = static_cast<uint8_t>(e8);
    if (c < C) {
      const float inv = inv_scale_from_ue8m0(e8);
      uint32_t w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const __nv_fp8x2_storage_t a2 = __nv_cvt_float2_to_fp8x2(make_float2(value(4 * j) * inv, value(4 * j + 1) * inv), __NV_SATFINITE, __NV_E4M3);
        const __nv_fp8x2_storage_t b2 = __nv_cvt_float2_to_fp8x2(make_float2(value(4 * j + 2) * inv, value(4 * j + 3) * inv), __NV_SATFINITE, __NV_E4M3);
        w[j] = static_cast<uint32_t>(a2) | (static_cast<uint32_t>(b2) << 16);
      }
      uint4* dst = reinterpret_cast<uint4*>(qT + static_cast<size_t>(c) * ldq + r0);
      if (r0 + 32 <= R) {
        dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
        dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
      } else {
        uint8_t* d8 = qT + static_cast<size_t>(c) * ldq + r0;
        for (int i = 0; i < 32 && r0 + i < R; ++i) d8[i] = static_cast<uint8_t>(w[i >> 2] >> (8 * (i & 3)));
      }
    }
  }
}

static void launch_quantize_t(const void* x, int ldx, void* qT, int ldq, void* sf, int R, int C, int C_pad, int batch,
                              long long x_batch, long long q_batch, long long sf_batch, int sf_bn, cudaStream_t st) {
  const bool pairs = C % 2 == 0 && ldx % 2 == 0 && x_batch % 2 == 0 && (reinterpret_cast<uintptr_t>(x) & 3) == 0;
  const int cols = pairs ? 128 : 64;
  launch_k(pairs ? mxfp8_quantize_t_kernel<2> : mxfp8_quantize_t_kernel<1>, dim3((C_pad + cols - 1) / cols, R / 32, batch), dim3(64), 0, st,
           (const __nv_bfloat16*)x, ldx, (uint8_t*)qT, ldq, (uint8_t*)sf, R, C, C_pad, x_batch, q_batch, sf_batch, sf_bn);
  kwu::count_launch();
}

// ------------------------------------------------------------------------------------ GEMM
// CG = 2: a cluster of two CTAs works on one 256 x BN tile (`cta_group::2`), each with its 128 rows of A, half of B's
// rows and its own copy of the scales (a product reads the scales of all BN columns from the TMEM of both SMs). The
// even CTA issues copies and products for both. See gemm_bf16.cu for the roles of the warps and the output path (through
// shared memory and TMA instead of a store per lane and row).
// Per 128-deep k-block an SM fetches 16 KB + BN * 64 B instead of 16 KB + BN * 128 B; what bounds the kernel is that
// traffic (a k-block of a 256 x 224 tile takes 0.29 us) and, below K of about 2000, the output and the last, partly
// empty round. One CTA with per-lane stores / this, best width each, B200, us:
//   4096 x 7168 x 1280  41.1 / 34.9    4096 x 1280 x 7168  37.4 / 34.0    4096 x 3584 x 1280  25.8 / 21.6
//   4096 x 1280 x 3584  23.4 / 20.9    4928 x 1536 x 4096  31.1 / 25.5    8192 x 3072 x 1024  35.4 / 29.8
constexpr int MX_BM = 128;
constexpr int MX_BK = 128;  // 128 e4m3 = one 128-byte swizzle row = four K=32 MMAs = one scale chunk
constexpr int MX_THREADS = 192;
constexpr int MX_MAX_STAGES = 8;
constexpr int MX_A_BYTES = MX_BM * MX_BK;
constexpr int MX_SF_AREA = 2048;            // per stage: the A chunk and up to two B chunks (512 bytes each)
constexpr int MX_OUT_BYTES = 4 * 2 * 4096;  // per epilogue warp two patches that TMA stores read
constexpr int MX_SMEM_MAX = 227 * 1024;

// How the accumulator leaves the kernel
constexpr int MX_OUT_BF16 = 0;    // bf16, TMA store
constexpr int MX_OUT_F32 = 1;     // fp32, TMA store
constexpr int MX_OUT_ADD = 2;     // fp32, TMA reduction (C +=)
constexpr int MX_OUT_DIRECT = 3;  // per-lane stores: scattered rows, bf16 C +=, widths or pitches TMA cannot address

struct MxGemmParams {
  int M, N, K;
  int ldc;
  int bn;
  int out_fp32, accumulate;
  int out_mode, out_cols;   // MX_OUT_*; columns of one bf16 store box (64, or 32 when bn is not a multiple of 64)
  float alpha;
  int stages, stage_bytes;
  int tiles_m, tiles_n;     // tile grid (a tile is 128 * CG rows)
  int sfb_chunks;           // 512-byte chunks of B scales per tile and k-block: 1 (plain, bn = 128) or 2 (tile-local)
  // grouped mode (rows of A grouped by expert): tile table entries (m0, expert, valid, 0); B holds the
  // experts' matrices stacked along its rows, `group_n` rows each (a multiple of 128)
  const int4* group_tiles;
  int group_n;
  const long long* row_ptrs;  // bf16 output: row r is stored at this byte address (0: dropped) instead of C + r*ldc
  int* status;
};

// Tile -> (A row offset, B row offset, output column offset); false: nothing to do for this entry.
template <int CG>
__device__ __forceinline__ bool mx_decode_tile(const MxGemmParams& p, int tile, int& m0, int& n0, int& b_row0) {
  const int tm = tile / p.tiles_n, tn = tile % p.tiles_n;
  n0 = tn * p.bn;
  if (p.group_tiles) {
    const int4 t = p.group_tiles[tm];
    if (!t.z) return false;
    m0 = t.x;
    b_row0 = t.y * p.group_n + n0;
  } else {
    m0 = tm * MX_BM * CG;
    b_row0 = n0;
  }
  return true;
}

template <int CG>
__global__ void __launch_bounds__(MX_THREADS, 1)
gemm_mxfp8_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                  const __grid_constant__ CUtensorMap tmSA, const __grid_constant__ CUtensorMap tmSB,
                  const __grid_constant__ CUtensorMap tmC, void* __restrict__ Cout, const MxGemmParams p) {
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t ACC_COLS = 240;         // distance of the two accumulators (bn <= 240)
  constexpr uint32_t SFA_COL = 2 * ACC_COLS;
  constexpr uint32_t SFB_COL = SFA_COL + 4;  // up to 8 columns

  extern __shared__ uint8_t smem_raw[];
  // both CTAs of a pair see the same offset: dynamic shared memory starts at one address in every CTA
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* out_area = smem;
  uint8_t* ring = smem + MX_OUT_BYTES;
  uint8_t* bar_area = ring + p.stages * p.stage_bytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(bar_area);
  uint64_t* empty_bar = full_bar + MX_MAX_STAGES;
  uint64_t* acc_full = empty_bar + MX_MAX_STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int cta = CG == 2 ? static_cast<int>(cluster_ctarank()) : 0;
  const int unit = static_cast<int>(blockIdx.x) / CG, units = static_cast<int>(gridDim.x) / CG;
  const int num_tiles = p.tiles_m * p.tiles_n;
  const int num_kb = p.K / MX_BK;
  const int BN = p.bn;
  const int stages = p.stages;
  const int b_bytes = BN / CG * MX_BK;       // this CTA's share of B (a multiple of 1024: whole swizzle groups)

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
    tma_prefetch_desc(&tmSA);
    tma_prefetch_desc(&tmSB);
    if (p.out_mode != MX_OUT_DIRECT) tma_prefetch_desc(&tmC);
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
    // warp-uniform loop, one elected lane issues (see the MMA warp below). With CG = 2 every load of the pair is
    // counted on the even CTA's barrier, whose CTA issues the products.
    const bool leader = elect_one();
    const uint32_t tx = (MX_A_BYTES + b_bytes + 512 + 512 * p.sfb_chunks) * CG;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = unit; tile < num_tiles && ok; tile += units) {
      int m0, n0, b_row0;
      if (!mx_decode_tile<CG>(p, tile, m0, n0, b_row0)) continue;
      m0 += cta * MX_BM;
      const int b_row = b_row0 + cta * (BN / CG);
      // scale chunks, one row of the scale maps each: [row tile][k-block], or [tile][k-block][2] in the tile-local layout
      const int sa_row = m0 / MX_BM * num_kb;
      const int sb_row = p.sfb_chunks == 2 ? n0 / BN * num_kb * 2 : b_row0 / 128 * num_kb;
      for (int kb = 0; kb < num_kb; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, KWU_ERR_TIMEOUT_EMPTY));
        if (!ok) break;
        uint8_t* sa = ring + stage * p.stage_bytes;
        uint8_t* ssf = sa + MX_A_BYTES + b_bytes;
        if (leader) {
          if (cta == 0) mbar_expect_tx(&full_bar[stage], tx);
          const uint32_t bar = CG == 2 ? mapa_shared(smem_u32(&full_bar[stage]), 0) : smem_u32(&full_bar[stage]);
          tma_load_2d_cg<CG>(sa, &tmA, bar, kb * MX_BK, m0);
          tma_load_2d_cg<CG>(sa + MX_A_BYTES, &tmB, bar, kb * MX_BK, b_row);
          tma_load_2d_cg<CG>(ssf, &tmSA, bar, 0, sa_row + kb);
          tma_load_2d_cg<CG>(ssf + 512, &tmSB, bar, 0, sb_row + kb * p.sfb_chunks);
        }
        __syncwarp();
        if (++stage == stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    // The whole warp walks the loop so that stage addresses, descriptors and counters stay warp-uniform (under
    // a single-lane branch every operand of every tcgen05 instruction is first moved from a per-thread to a
    // uniform register, and with 128-wide tiles the issue of 2-3 scale copies + 4 MMAs per k-block then takes
    // longer than their execution); one elected lane of the even CTA issues.
    if (cta == 0) {
      const bool leader = elect_one();
      const uint32_t idesc = make_idesc_mxf8(MX_BM * CG, BN, 0, 0);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      for (int tile = unit; tile < num_tiles && ok; tile += units) {
        int m0, n0, b_row0;
        if (!mx_decode_tile<CG>(p, tile, m0, n0, b_row0)) continue;
        const int as = it & 1;
        const uint32_t aphase = (it >> 1) & 1;
        ++it;
        ok = __all_sync(0xffffffffu, mbar_wait_cluster<CG>(&acc_empty[as], aphase ^ 1, abort_flag, p.status, KWU_ERR_TIMEOUT_ACC_EMPTY));
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + as * ACC_COLS;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase, abort_flag, p.status, KWU_ERR_TIMEOUT_FULL));
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = smem_u32(ring + stage * p.stage_bytes);
          const uint64_t ad = make_smem_desc(sa, 16, 1024, SWZ_128B);
          const uint64_t bd = make_smem_desc(sa + MX_A_BYTES, 16, 1024, SWZ_128B);
          const uint64_t sfd = make_smem_desc(sa + MX_A_BYTES + b_bytes, 16, 128, SWZ_NONE);
          const uint32_t acc0 = kb > 0 ? 1u : 0u;
          if (leader) {
            // scale chunks: shared -> TMEM (32 rows x 16 B each, 8-row groups 128 B apart, no swizzle);
            // 512 bytes further in shared memory is +32 in the descriptor's address field
            tc_cp_32x128b_warpx4_cg<CG>(tmem_base + SFA_COL, sfd);
            tc_cp_32x128b_warpx4_cg<CG>(tmem_base + SFB_COL, sfd + 32);
            if (p.sfb_chunks == 2) tc_cp_32x128b_warpx4_cg<CG>(tmem_base + SFB_COL + 4, sfd + 64);
            // 32 fp8 elements along K per instruction: +32 bytes = +2 in the address field, next byte of the scale words
            mma_mxf8_ss_cg<CG>(d_tmem, ad, bd, idesc, tmem_base + SFA_COL, tmem_base + SFB_COL, acc0);
#pragma unroll
            for (uint32_t k = 1; k < MX_BK / 32; ++k)
              mma_mxf8_ss_cg<CG>(d_tmem, ad + 2 * k, bd + 2 * k, idesc | (k << 4) | (k << 29), tmem_base + SFA_COL,
                                 tmem_base + SFB_COL, 1u);
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
    const int quarter = warp & 3;
    uint8_t* patch = out_area + (warp - 2) * 8192;
    int it = 0, ob = 0;            // tiles done; output patch in use
    bool ok = true;
    for (int tile = unit; tile < num_tiles && ok; tile += units) {
      int m0, n0, b_row0;
      if (!mx_decode_tile<CG>(p, tile, m0, n0, b_row0)) continue;
      m0 += cta * MX_BM;
      const int as = it & 1;
      const uint32_t aphase = (it >> 1) & 1;
      ++it;
      ok = mbar_wait(&acc_full[as], aphase, abort_flag, p.status, KWU_ERR_TIMEOUT_ACC_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int row0 = m0 + quarter * 32;
      const int row = row0 + lane;
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + as * ACC_COLS;
      const int ncols = min(BN, p.N - n0);     // columns of this tile that exist
      const bool tma_rows = row0 < p.M;        // a warp whose rows all lie below the matrix stores nothing
#pragma unroll 1
      for (int c = 0; c * 32 < ncols; ++c) {
        uint32_t r[32];
        // a tile width that is an odd multiple of 16 ends in a 16-column chunk
        const int width = (BN % 32 != 0 && c == BN / 32) ? 16 : 32;
        if (width == 32) {
          tmem_ld_x32(t_row + c * 32, r);
        } else {
          tmem_ld_x16(t_row + c * 32, r);
#pragma unroll
          for (int j = 16; j < 32; ++j) r[j] = 0u;
        }
        tmem_ld_wait();
        const int col0 = n0 + c * 32;
        if (p.out_mode == MX_OUT_BF16) {
          // 64-column boxes: 128-byte rows, 16-byte units XORed with the row (the TMA's 128-byte swizzle);
          // 32-column boxes: 64-byte rows, units XORed with row / 2 (its 64-byte swizzle)
          const bool wide = p.out_cols == 64;
          if (!wide || (c & 1) == 0) {      // first half of a box: the patch must be free again
            if (lane == 0) tma_store_wait_read<1>();
            __syncwarp();
          }
          uint8_t* dst = patch + ob * 4096 + lane * (wide ? 128 : 64);
          const int unit0 = wide ? (c & 1) * 4 : 0, key = wide ? (lane & 7) : ((lane >> 1) & 3);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[8 * j + e]) * p.alpha;
            *reinterpret_cast<uint4*>(dst + (((unit0 + j) ^ key) << 4)) =
                make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
          }
          if (!wide || (c & 1) || (c + 1) * 32 >= ncols) {   // box complete (a last half box is cut at N by the TMA)
            fence_async_proxy();
            __syncwarp();
            if (lane == 0 && tma_rows) {
              tma_store_2d(&tmC, patch + ob * 4096, wide ? n0 + (c & ~1) * 32 : col0, row0);
              tma_store_commit();
            }
            ob ^= 1;
          }
          continue;
        }
        if (p.out_mode == MX_OUT_F32 || p.out_mode == MX_OUT_ADD) {
          if (lane == 0) tma_store_wait_read<1>();
          __syncwarp();
          uint8_t* dst = patch + ob * 4096 + lane * 128;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<float4*>(dst + ((j ^ (lane & 7)) << 4)) =
                make_float4(__uint_as_float(r[4 * j]) * p.alpha, __uint_as_float(r[4 * j + 1]) * p.alpha,
                            __uint_as_float(r[4 * j + 2]) * p.alpha, __uint_as_float(r[4 * j + 3]) * p.alpha);
          fence_async_proxy();
          __syncwarp();
          if (lane == 0 && tma_rows) {
            if (p.out_mode == MX_OUT_ADD) tma_reduce_add_2d(&tmC, patch + ob * 4096, col0, row0);
            else tma_store_2d(&tmC, patch + ob * 4096, col0, row0);
            tma_store_commit();
          }
          ob ^= 1;
          continue;
        }
        const int col_end = min(col0 + width, p.N);   // columns past the tile or the matrix are not stored
        if (row < p.M && col0 < col_end) {
          const bool full = (col_end - col0 == 32);
          if (p.out_fp32) {
            float* dst = reinterpret_cast<float*>(Cout) + static_cast<size_t>(row) * p.ldc + col0;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              if (full || col0 + j < col_end) {
                float v = __uint_as_float(r[j]) * p.alpha;
                if (p.accumulate) v += dst[j];
                dst[j] = v;
              }
            }
          } else {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(Cout) + static_cast<size_t>(row) * p.ldc + col0;
            if (p.row_ptrs) {
              const long long base = p.row_ptrs[row];
              if (!base) continue;
              dst = reinterpret_cast<__nv_bfloat16*>(base) + col0;
            }
            const int nvec = (col_end - col0) >> 3;   // whole 8-column vectors (N and the tile edges are multiples of 8)
            if ((col_end - col0) % 8 == 0) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                if (j < nvec) {
                  float f[8];
#pragma unroll
                  for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[8 * j + e]) * p.alpha;
                  uint4* d4 = reinterpret_cast<uint4*>(dst) + j;
                  if (p.accumulate) {
                    const uint4 o = *d4;
                    const float2 o0 = unpack_bf16(o.x), o1 = unpack_bf16(o.y), o2 = unpack_bf16(o.z), o3 = unpack_bf16(o.w);
                    f[0] += o0.x; f[1] += o0.y; f[2] += o1.x; f[3] += o1.y;
                    f[4] += o2.x; f[5] += o2.y; f[6] += o3.x; f[7] += o3.y;
                  }
                  *d4 = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
                }
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                if (col0 + j < col_end) {
                  float v = __uint_as_float(r[j]) * p.alpha;
                  if (p.accumulate) v += __bfloat162float(dst[j]);
                  dst[j] = __float2bfloat16(v);
                }
              }
            }
          }
        }
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

  tc_fence_before();
  __syncthreads();
  if (*abort_flag)
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  if (CG == 2) cluster_sync();   // the pair leaves together: its barriers and TMEM are used from both sides
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_cg<CG>(tmem_base, TMEM_COLS);
  }
}

template <int CG>
static int launch_mx(int BN, const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                     const uint8_t* sfa, const uint8_t* sfb, int out_fp32, int accumulate, float alpha,
                     cudaStream_t stream, int* status, const int4* group_tiles = nullptr, int n_group_tiles = 0,
                     int n_groups = 1, const long long* row_ptrs = nullptr) {
  CUtensorMap tmA, tmB, tmSA, tmSB, tmC;
  int rc;
  const long long b_rows = static_cast<long long>(N) * n_groups;
  const int num_kb = K / MX_BK;
  const int tiled = BN > 128 ? 1 : 0;
  if ((rc = encode_tmap_2d(&tmA, A, ELEM_U8, M, K, lda, MX_BM, MX_BK, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  if ((rc = encode_tmap_2d(&tmB, B, ELEM_U8, b_rows, K, ldb, BN / CG, MX_BK, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
  // scale buffers as rows of one 512-byte chunk (128 words); rows past the end read as zero and meet zero operands
  const long long sa_rows = static_cast<long long>((M + 127) / 128) * num_kb;
  const long long sb_rows = (tiled ? static_cast<long long>((N + BN - 1) / BN) * 2 : (b_rows + 127) / 128) * num_kb;
  if ((rc = encode_tmap_2d(&tmSA, sfa, ELEM_F32, sa_rows, 128, 128, 1, 128, CU_TENSOR_MAP_SWIZZLE_NONE))) return rc;
  if ((rc = encode_tmap_2d(&tmSB, sfb, ELEM_F32, sb_rows, 128, 128, tiled ? 2 : 1, 128, CU_TENSOR_MAP_SWIZZLE_NONE))) return rc;
  MxGemmParams p;
  p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.bn = BN; p.out_fp32 = out_fp32; p.accumulate = accumulate; p.alpha = alpha;
  p.sfb_chunks = tiled ? 2 : 1;
  p.stage_bytes = MX_A_BYTES + BN / CG * MX_BK + MX_SF_AREA;
  p.stages = (MX_SMEM_MAX - 2048 - MX_OUT_BYTES) / p.stage_bytes;
  if (p.stages > MX_MAX_STAGES) p.stages = MX_MAX_STAGES;
  p.tiles_m = group_tiles ? n_group_tiles : (M + MX_BM * CG - 1) / (MX_BM * CG);
  p.tiles_n = (N + BN - 1) / BN;
  p.group_tiles = group_tiles;
  p.group_n = N;
  p.row_ptrs = out_fp32 ? nullptr : row_ptrs;
  p.status = status;
  // TMA addresses the output when its base and pitch are 16-byte multiples; its boxes are 32 or 64 columns wide
  const bool can_tma = (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (static_cast<long long>(ldc) * (out_fp32 ? 4 : 2)) % 16 == 0 &&
                       !p.row_ptrs && BN % 32 == 0;
  p.out_mode = MX_OUT_DIRECT;
  p.out_cols = (BN % 64) ? 32 : 64;
  if (can_tma && (out_fp32 || !accumulate))
    p.out_mode = out_fp32 ? (accumulate ? MX_OUT_ADD : MX_OUT_F32) : MX_OUT_BF16;
  if (p.out_mode != MX_OUT_DIRECT) {
    if (out_fp32)
      rc = encode_tmap_2d(&tmC, C, ELEM_F32, M, N, ldc, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B);
    else
      rc = encode_tmap_2d(&tmC, C, ELEM_BF16, M, N, ldc, 32, p.out_cols,
                          p.out_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc) return rc;
  } else {
    tmC = tmA;   // not read
  }
  auto kern = gemm_mxfp8_kernel<CG>;
  static PerDeviceOnce attr_set;
  if (attr_set.pending()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MX_SMEM_MAX);
    if (e != cudaSuccess) { set_last_error("gemm_mxfp8 attr: %s", cudaGetErrorString(e)); return 10; }
    attr_set.mark();
  }
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int units = sms / CG;
  if (static_cast<long long>(p.tiles_m) * p.tiles_n < units) units = p.tiles_m * p.tiles_n;
  const size_t smem = 2048 + MX_OUT_BYTES + static_cast<size_t>(p.stages) * p.stage_bytes;
  launch_cluster(kern, dim3(units * CG), dim3(MX_THREADS), CG, smem, stream, tmA, tmB, tmSA, tmSB, tmC, C, p); kwu::count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_last_error("gemm_mxfp8 launch: %s", cudaGetErrorString(e)); return 11; }
  return 0;
}

// Tile width. 128 works with the plain scale layout (a tile always starts on a chunk boundary). Wider tiles
// (multiples of 16 up to 240: two accumulators plus the scale columns must fit in 512 TMEM columns) need the B
// operand's scales in the tile-local layout, which only an operand quantised for that width has (weights).
// Why wider: the bytes fetched per output column fall with the width, and it can be chosen so that the tile count
// fills whole rounds of the SM pairs (4096 x 1280: 160 tiles of 128 = 2.2 rounds of 74, 128 tiles of 160 = 1.7).
// Odd multiples of 16 have no pair form (halves of 16-row groups) and stay with one CTA, per-lane stores.
// A variant that kept the plain layout and offset the scale address by (first row % 128) / 32 TMEM columns
// faulted ("misaligned address") at width 160, where that offset is odd; width 192 (offsets 0 and 2) ran
// correctly, so odd column offsets of the scale address are the cause, and no path here uses an offset.
static bool bn_supported(int bn) { return bn == 128 || (bn > 128 && bn <= 240 && bn % 16 == 0); }

}  // namespace kwu

using namespace kwu;

// Bytes of the scale buffer of a (rows, K) operand.
KWU_API long long kwu_mxfp8_sf_bytes(int rows, int K) {
  return static_cast<long long>((rows + 127) / 128) * (K / 128) * 512;
}

KWU_API int kwu_mxfp8_quantize(const void* x, int ldx, void* q, int ldq, void* sf, int M, int K, void* stream) {
  if (K % 128) { set_last_error("mxfp8_quantize: K must be a multiple of 128 (got %d)", K); return 7; }
  if (M <= 0) return 0;
  const int M_pad = (M + 127) / 128 * 128;
  long warps = static_cast<long>(M_pad) * ((K + 255) / 256);
  long grid = (warps + 7) / 8;
  if (grid > 148 * 16) grid = 148 * 16;
  launch_k(mxfp8_quantize_kernel, dim3(static_cast<int>(grid)), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream), 
      (const __nv_bfloat16*)x, ldx, (uint8_t*)q, ldq, (uint8_t*)sf, M, K, M_pad, 0); kwu::count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_last_error("mxfp8_quantize launch: %s", cudaGetErrorString(e)); return 11; }
  return 0;
}

// x (R, C) -> qT (C, R) quantised along R; sf has kwu_mxfp8_sf_bytes(C, R) bytes. R % 128 == 0.
KWU_API int kwu_mxfp8_quantize_t(const void* x, int ldx, void* qT, int ldq, void* sf, int R, int C, void* stream) {
  if (R % 128) { set_last_error("mxfp8_quantize_t: R must be a multiple of 128 (got %d)", R); return 7; }
  if (C <= 0) return 0;
  const int C_pad = (C + 127) / 128 * 128;
  launch_quantize_t(x, ldx, qT, ldq, sf, R, C, C_pad, 1, 0, 0, 0, 0, reinterpret_cast<cudaStream_t>(stream));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_last_error("mxfp8_quantize_t launch: %s", cudaGetErrorString(e)); return 11; }
  return 0;
}

// Weight forms: as kwu_mxfp8_quantize / kwu_mxfp8_quantize_t, with the scales in the tile-local layout for GEMM
// tiles `sf_bn` rows wide (sf_bn <= 128: plain layout). The scale buffer has kwu_mxfp8_sf_bytes_tiled bytes and
// must be pre-filled with the neutral byte 127: only the scales of real rows are written.
KWU_API long long kwu_mxfp8_sf_bytes_tiled(int rows, int K, int sf_bn) {
  if (sf_bn <= 128) return kwu_mxfp8_sf_bytes(rows, K);
  return static_cast<long long>((rows + sf_bn - 1) / sf_bn) * (K / 128) * 1024;
}

KWU_API int kwu_mxfp8_quantize_w(const void* x, int ldx, void* q, int ldq, void* sf, int M, int K, int sf_bn,
                                 void* stream) {
  if (K % 128) { set_last_error("mxfp8_quantize_w: K must be a multiple of 128 (got %d)", K); return 7; }
  if (!bn_supported(sf_bn)) { set_last_error("mxfp8_quantize_w: unsupported tile width %d", sf_bn); return 7; }
  if (M <= 0) return 0;
  const int M_pad = (M + 127) / 128 * 128;
  long warps = static_cast<long>(M_pad) * ((K + 255) / 256);
  long grid = (warps + 7) / 8;
  if (grid > 148 * 16) grid = 148 * 16;
  launch_k(mxfp8_quantize_kernel, dim3(static_cast<int>(grid)), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream), 
      (const __nv_bfloat16*)x, ldx, (uint8_t*)q, ldq, (uint8_t*)sf, M, K, M_pad, sf_bn); kwu::count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_last_error("mxfp8_quantize_w launch: %s", cudaGetErrorString(e)); return 11; }
  return 0;
}

KWU_API int kwu_mxfp8_quantize_t_w(const void* x, int ldx, void* qT, int ldq, void* sf, int R, int C, int sf_bn,
                                   void* stream) {
  if (R % 128) { set_last_error("mxfp8_quantize_t_w: R must be a multiple of 128 (got %d)", R); return 7; }
  if (!bn_supported(sf_bn)) { set_last_error("mxfp8_quantize_t_w: unsupported tile width %d", sf_bn); return 7; }
  if (C <= 0) return 0;
  const int C_pad = (C + 127) / 128 * 128;
  launch_quantize_t(x, ldx, qT, ldq, sf, R, C, C_pad, 1, 0, 0, 0, sf_bn, reinterpret_cast<cudaStream_t>(stream));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_last_error("mxfp8_quantize_t_w launch: %s", cudaGetErrorString(e)); return 11; }
  return 0;
}

// `batch` matrices x[b] (R, C) at stride R*ldx -> qT[b] (C, R) at stride C*ldq, scale buffers at stride
// kwu_mxfp8_sf_bytes(C, R). C must be a multiple of 128 so that the stacked outputs stay chunk-aligned.
KWU_API int kwu_mxfp8_quantize_t_batched(const void* x, int ldx, void* qT, int ldq, void* sf, int R, int C, int batch,
                                         void* stream) {
  if (R % 128 || C % 128) { set_last_error("mxfp8_quantize_t_batched: R and C must be multiples of 128"); return 7; }
  if (batch <= 0) return 0;
  launch_quantize_t(x, ldx, qT, ldq, sf, R, C, C, batch, static_cast<long long>(R) * ldx, static_cast<long long>(C) * ldq,
                    kwu_mxfp8_sf_bytes(C, R), 0, reinterpret_cast<cudaStream_t>(stream));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_last_error("mxfp8_quantize_t_batched launch: %s", cudaGetErrorString(e)); return 11; }
  return 0;
}

// Grouped form: rows of A are grouped by expert in 128-row-aligned ranges described by `tiles`
// ((m0, expert, valid, 0) per 128-row tile); B stacks the experts' (N, K) matrices along its rows.
// out[rows of expert e] = A[rows] B[e]^T. N must be a multiple of 128.
// row_ptrs (optional): per output row the byte address it is stored at (0 = skip); C is then not written.
KWU_API int kwu_gemm_mxfp8_grouped(const void* A, const void* sfa, const void* B, const void* sfb, void* C,
                                   int M, int N, int K, int lda, int ldb, int ldc, int n_experts,
                                   const void* tiles, int n_tiles, const long long* row_ptrs, void* stream,
                                   int* status) {
  if (M <= 0 || N <= 0 || n_tiles <= 0) return 0;
  if (K % 128 || N % 128) { set_last_error("gemm_mxfp8_grouped: K and N must be multiples of 128 (got %d, %d)", K, N); return 7; }
  return launch_mx<1>(128, A, B, C, M, N, K, lda, ldb, ldc, (const uint8_t*)sfa, (const uint8_t*)sfb, 0, 0, 1.f,
                        reinterpret_cast<cudaStream_t>(stream), status, reinterpret_cast<const int4*>(tiles),
                        n_tiles, n_experts, row_ptrs);
}

KWU_API int kwu_gemm_mxfp8(const void* A, const void* sfa, const void* B, const void* sfb, void* C, int M,
                           int N, int K, int lda, int ldb, int ldc, int out_fp32, int accumulate,
                           float alpha, int bn, void* stream, int* status) {
  if (M <= 0 || N <= 0) return 0;
  if (K % 128) { set_last_error("gemm_mxfp8: K must be a multiple of 128 (got %d)", K); return 7; }
  if (bn <= 0) bn = 128;
  if (!bn_supported(bn)) { set_last_error("gemm_mxfp8: tile width %d is not 128 or a multiple of 16 in (128, 240]", bn); return 7; }
  // Pairs of CTAs from two row tiles on (a pair's other half would multiply nothing), at widths that are multiples of 32:
  // 4096 x 1280 x 3584 at 160 columns takes 20.9 us on pairs, 23.4 on single CTAs
  if (M > MX_BM && bn % 32 == 0)
    return launch_mx<2>(bn, A, B, C, M, N, K, lda, ldb, ldc, (const uint8_t*)sfa, (const uint8_t*)sfb, out_fp32, accumulate,
                        alpha, reinterpret_cast<cudaStream_t>(stream), status);
  return launch_mx<1>(bn, A, B, C, M, N, K, lda, ldb, ldc, (const uint8_t*)sfa, (const uint8_t*)sfb, out_fp32, accumulate,
                      alpha, reinterpret_cast<cudaStream_t>(stream), status);
}

// ------------------------------------------------------------------------------------ attention operands
// Per-head MXFP8 quantisation of q / k for attention (head_dim 64 = two 32-blocks per (token, head) row):
//   mxfp8_column_mean   mu[h, d] = mean over the T tokens of the pack of x[t, h, d]  (key smoothing: scores
//                       change by q . mu, a constant along the key axis, which softmax ignores)
//   mxfp8_quant_heads   x[t, h, :] (- mu[h, :]) -> e4m3 bytes + two UE8M0 scale bytes per row, and the
//                       dequantised bf16 copy (e4m3 x 2^e is exact in bf16) that the attention kernels read.
// Reference: src/kohakuwullm/kernels/mxfp8/attention_quant.py:17-78.
namespace kwu {

__global__ void __launch_bounds__(256)
mxfp8_column_mean_kernel(const __nv_bfloat16* __restrict__ x, long long ld_t, int T, int H, float* __restrict__ mu) {
  // block = one head; thread = (channel d = tid % 64, token lane = tid / 64)
  __shared__ float s_part[4][64];
  const int h = blockIdx.x, d = threadIdx.x & 63, tl = threadIdx.x >> 6;
  float acc = 0.f;
  for (int t = tl; t < T; t += 4) acc += __bfloat162float(x[static_cast<size_t>(t) * ld_t + h * 64 + d]);
  s_part[tl][d] = acc;
  __syncthreads();
  if (tl == 0) mu[h * 64 + d] = (s_part[0][d] + s_part[1][d] + s_part[2][d] + s_part[3][d]) / static_cast<float>(T);
}

// One lane = 8 channels; 8 lanes = one (token, head) row; a warp covers 4 rows.
__global__ void __launch_bounds__(256)
mxfp8_quant_heads_kernel(const __nv_bfloat16* __restrict__ x, long long ld_t, const float* __restrict__ mu,
                         uint8_t* __restrict__ q8, uint8_t* __restrict__ sf, __nv_bfloat16* __restrict__ deq,
                         long long rows, int H) {
  const int lane = threadIdx.x & 31;
  const long long wid = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  for (long long r0 = wid * 4; r0 < rows; r0 += nwarps * 4) {
    const long long row = r0 + (lane >> 3);
    const int c = (lane & 7) * 8;
    const bool in = row < rows;
    const long long t = in ? row / H : 0;
    const int h = in ? static_cast<int>(row % H) : 0;
    float f[8];
    if (in) {
      const uint4 a = *reinterpret_cast<const uint4*>(x + static_cast<size_t>(t) * ld_t + h * 64 + c);
      unpack8(a, f);
      if (mu) {
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] -= mu[h * 64 + c + e];
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = 0.f;
    }
    float amax = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(f[e]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    if (!in) continue;
    const uint32_t e8 = ue8m0_from_amax(amax);
    const float inv = inv_scale_from_ue8m0(e8);
    const float scale = __uint_as_float(e8 << 23);  // 2^(e8 - 127); e8 >= 1 here because amax >= 1e-30
    uint32_t lo = 0, hi = 0;
    float d[8];
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      const __nv_fp8x2_storage_t p2 = __nv_cvt_float2_to_fp8x2(make_float2(f[e] * inv, f[e + 1] * inv), __NV_SATFINITE, __NV_E4M3);
      const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2(p2, __NV_E4M3);
      const float2 back = __half22float2(*reinterpret_cast<const __half2*>(&hr));
      d[e] = back.x * scale;
      d[e + 1] = back.y * scale;
      if (e < 4) lo |= static_cast<uint32_t>(p2) << (8 * e);
      else hi |= static_cast<uint32_t>(p2) << (8 * (e - 4));
    }
    if (q8) *reinterpret_cast<uint2*>(q8 + static_cast<size_t>(row) * 64 + c) = make_uint2(lo, hi);
    if (sf && (lane & 3) == 0) sf[static_cast<size_t>(row) * 2 + (c >> 5)] = static_cast<uint8_t>(e8);
    *reinterpret_cast<uint4*>(deq + static_cast<size_t>(row) * 64 + c) =
        make_uint4(pack_bf16(d[0], d[1]), pack_bf16(d[2], d[3]), pack_bf16(d[4], d[5]), pack_bf16(d[6], d[7]));
  }
}

}  // namespace kwu

// x: (T, H, 64) bf16 view with token pitch ld_t elements (heads contiguous). mu: (H, 64) fp32 out.
KWU_API int kwu_mxfp8_column_mean(const void* x, long long ld_t, int T, int H, float* mu, void* stream) {
  if (T <= 0 || H <= 0) return 0;
  mxfp8_column_mean_kernel<<<H, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>((const __nv_bfloat16*)x, ld_t, T, H, mu); kwu::count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_last_error("mxfp8_column_mean launch: %s", cudaGetErrorString(e)); return 11; }
  return 0;
}

// q8 (T,H,64) bytes and sf (T,H,2) bytes are optional; deq (T,H,64) bf16 contiguous is always written.
KWU_API int kwu_mxfp8_quant_heads(const void* x, long long ld_t, const float* mu, void* q8, void* sf, void* deq, int T,
                                  int H, void* stream) {
  if (T <= 0 || H <= 0) return 0;
  const long long rows = static_cast<long long>(T) * H;
  long long grid = (rows + 31) / 32;
  if (grid > 148 * 16) grid = 148 * 16;
  mxfp8_quant_heads_kernel<<<static_cast<int>(grid), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      (const __nv_bfloat16*)x, ld_t, mu, (uint8_t*)q8, (uint8_t*)sf, (__nv_bfloat16*)deq, rows, H); kwu::count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_last_error("mxfp8_quant_heads launch: %s", cudaGetErrorString(e)); return 11; }
  return 0;
}
