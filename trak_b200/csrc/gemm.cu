// Tensor-core GEMM for the after-kernel scoring:  C[M x N] (+)= alpha * s[m] * A[M x K] . B[N x K]^T
//
// Used for the three products of the reference's BasicScoreComputer
// (trak/score_computers.py:145-189):  X^T X  (A = B = X^T, symmetric mode),
// X . inv  (inv is symmetric, so it is its own transpose) and  features . targets^T.
//
// fp32 inputs are not rounded to one tensor-core format.  A packing pass scales every operand
// row by the power of two that brings its largest magnitude into [2^14, 2^15) and splits the
// scaled value into fp16 hi + fp16 lo (hi = rn(x), lo = rn(x - hi): 22 to 23 mantissa bits for
// every element within 2^-18 of its row's maximum, an absolute floor of 2^-40 of that maximum
// below), the kernels accumulate  hi*hi + hi*lo + lo*hi  in fp32 -- three MMAs per k-step at the
// 16-bit rate, the dropped lo*lo term is under 2^-22 -- and the epilogue multiplies the two
// inverse scales back in (powers of two: exact).  The row maxima and the planes come out of one
// read of the operand where a row fits in a block's registers (pack_rows_f32_kernel).
// What is left is the tensor core's own accumulation, which truncates instead of rounding: every MMA whose addends reach below the accumulator's
// last place pulls the sum towards zero, and a K-long contraction is a chain of 3K/16 such steps.
//  * X . inv and features . targets^T (gemm_nt_kernel) keep one accumulation over all of K:
//    about 1e-5 relative at K = 3000 ... 8192 (one TF32 pass would give 5e-4).  With bf16
//    instead of fp16 planes (16 mantissa bits) these two products cost 2.5 times the error in
//    the scores of an ill-conditioned problem and were 5 % faster.
//  * X^T X and W^T W (gemm_nt_chunked_kernel) feed or form an inverse, which multiplies a
//    relative error of the Gram by its condition number (measured: condition number 1000 turned
//    the 1e-5 into 2e-3 in the scores where plain fp32 arithmetic gives 3e-5).  There the tensor
//    core accumulates only 64 k at a time and the chunks are summed with rounded fp32 adds:
//    within 2x of cuBLAS fp32 at n = 5000 and closer to the exact Gram than cuBLAS fp32 at
//    n = 65,536 (5e-7 against 8e-6).
// fp16 and bf16 inputs are exact in one plane and take one MMA per k-step, unscaled.
//
// The packing pass also tiles the operands the way the pipeline consumes them:
// [128-row block][32-wide k block][plane][128 rows][32 k], so every TMA box is one
// contiguous 8 KB run, and it can transpose (for X^T X the operand is X^T).
//
// Kernel: one CTA per 256 x 256 tile of C, or per 128 x 128 tile (two CTAs per SM), with the
// contraction split over several CTAs, where the large tile leaves SMs idle (plan_gemm).
// Warp 0 issues TMA (64-byte swizzle boxes, never multicast), warp 1 issues tcgen05.mma (both
// operands from shared memory; M = 128, N = 256, two accumulators fill the 512 TMEM columns of
// the large tile), the warps from the fifth on run the epilogue (tcgen05.ld, scale, optional accumulate, optional mirrored store for the
// symmetric product).  Every mbarrier wait is bounded.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "gemm.h"
#include "host_util.h"
#include "ptx.cuh"

namespace tb {

constexpr uint32_t GK = 32;                 // k per pipeline stage (one 64-byte swizzle row)
constexpr uint32_t GTILE_BYTES = 128 * GK * 2;  // one [128 x 32] 16-bit tile: 8 KB

struct GemmParams {
    float* C;
    const float* row_scale;  // nullable, length M
    const uint32_t* amax_a;  // fp32 inputs: bit pattern of max |.| of every packed row of A (else null)
    const uint32_t* amax_b;  // the same for B
    uint32_t* status;
    int64_t ldc;
    uint32_t M, N;
    uint32_t kblocks;        // K / 32 (padded)
    uint32_t kb_per_split;   // k blocks of one slice of the grid's z dimension (kblocks when there is one slice);
                             // the chunked kernel divides what `range` leaves of each tile instead
    uint64_t split_stride;   // floats between the partial products of two slices
    uint32_t stages;
    uint32_t idesc;
    float alpha;
    int accumulate;
    int symmetric;           // A and B are the same packed operand; only tiles on/above the
                             // diagonal are computed and every result is stored twice
    int range;               // KRange, chunked kernel only
    int mirror;              // symmetric: whether this launch stores the second copy (not for partial products)
};

// Power-of-two scale of a packed fp32 operand row whose largest magnitude has the bit pattern
// `amax_bits`: the biased exponent E is clamped to [16, 254] so that both 2^(141 - E) (brings
// the maximum into [2^14, 2^15), inside fp16's range) and its inverse are normal numbers.
__device__ __forceinline__ uint32_t scale_exponent(uint32_t amax_bits) {
    const uint32_t e = amax_bits >> 23;
    return e < 16u ? 16u : (e > 254u ? 254u : e);
}
__device__ __forceinline__ float row_scale_up(uint32_t amax_bits) {
    return __uint_as_float((268u - scale_exponent(amax_bits)) << 23);
}
__device__ __forceinline__ float row_scale_down(uint32_t amax_bits) {
    return __uint_as_float((scale_exponent(amax_bits) - 14u) << 23);
}

__device__ __forceinline__ void gemm_fail(uint32_t* status, volatile uint32_t* abort_flag, uint32_t code,
                                          uint32_t detail) {
    *abort_flag = 1u;
    if (record_status(status, code)) {
        status[1] = blockIdx.x + gridDim.x * blockIdx.y;
        status[2] = detail;
    }
}


// Epilogue store of one warp's 32 x COLS block of results, which sits in the warp's shared-memory
// slab as slab[row][column] (row length COLS + 4 floats: 16-byte accesses along a row and of the same column piece by
// a row per lane are both conflict-free).  Whole blocks of aligned rows leave 16 bytes per lane: the epilogue, which no
// other work of the SM covers, is bound by its shared-memory and store instructions, and a quarter of them took a
// 50,000 x 2048 x 2048 product from 922 to 854 us (fp32) and from 433 to 356 us (fp16).  C[m_first + row, n0 + column] is written as rows of COLS consecutive floats
// (a lane holding one row in registers would touch 32 rows per store instruction).  When
// accumulating, the loads of a group are all issued before its first store: a load behind a store
// to a possibly aliasing address would wait for it.  Symmetric products store only n >= m that way
// and write the same bits to C[n, m] for n > m (for a fixed column the lanes run along m: coalesced).
__host__ __device__ constexpr uint32_t slab_ld(uint32_t cols) { return cols + 4u; }
template <uint32_t COLS>
__device__ __forceinline__ void store_block_from_slab(const GemmParams& p, float* C, const float* slab, uint32_t m_first,
                                                      uint32_t n0, uint32_t lane) {
    constexpr uint32_t LD = slab_ld(COLS), CH = COLS / 32u;
    const bool sym = p.symmetric != 0;
    const bool vec = (p.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 15u) == 0 && n0 + COLS <= p.N &&
                     (!sym || n0 >= m_first + 31u);
    if (vec) {
        constexpr uint32_t LANES = COLS / 4u, ROWS = 32u / LANES;  // lanes of a row, rows of an access
        const uint32_t row = lane / LANES, col = lane % LANES * 4u;
#pragma unroll 1
        for (uint32_t r0 = 0; r0 < 32u && m_first + r0 < p.M; r0 += 8u * ROWS) {
            float4 v[8];
#pragma unroll
            for (uint32_t u = 0; u < 8; ++u) {
                const uint32_t mr = m_first + r0 + u * ROWS + row;
                v[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (p.accumulate && mr < p.M) v[u] = *reinterpret_cast<const float4*>(C + (int64_t)mr * p.ldc + n0 + col);
            }
#pragma unroll
            for (uint32_t u = 0; u < 8; ++u) {
                const uint32_t mr = m_first + r0 + u * ROWS + row;
                const float4 w = *reinterpret_cast<const float4*>(slab + (r0 + u * ROWS + row) * LD + col);
                if (mr < p.M)
                    *reinterpret_cast<float4*>(C + (int64_t)mr * p.ldc + n0 + col) =
                        make_float4(v[u].x + w.x, v[u].y + w.y, v[u].z + w.z, v[u].w + w.w);
            }
        }
    }
#pragma unroll 1
    for (uint32_t r0 = 0; !vec && r0 < 32u && m_first + r0 < p.M; r0 += 4u) {
        float v[4][CH];
        bool on[4][CH];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
#pragma unroll
            for (uint32_t ch = 0; ch < CH; ++ch) {
                const uint32_t mr = m_first + r0 + u, n = n0 + ch * 32u + lane;
                on[u][ch] = mr < p.M && n < p.N && (!sym || n >= mr);
                v[u][ch] = (p.accumulate && on[u][ch]) ? C[(int64_t)mr * p.ldc + n] : 0.0f;
            }
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
#pragma unroll
            for (uint32_t ch = 0; ch < CH; ++ch)
                if (on[u][ch])
                    C[(int64_t)(m_first + r0 + u) * p.ldc + n0 + ch * 32u + lane] =
                        v[u][ch] + slab[(r0 + u) * LD + ch * 32u + lane];
    }
    const uint32_t m = m_first + lane;
    if (sym && p.mirror && m < p.N) {
#pragma unroll 1
        for (uint32_t i0 = 0; i0 < COLS; i0 += 16u) {
            float old[16];
#pragma unroll
            for (uint32_t u = 0; u < 16; ++u) {
                const bool on = n0 + i0 + u < p.M && n0 + i0 + u > m;
                old[u] = (p.accumulate && on) ? C[(int64_t)(n0 + i0 + u) * p.ldc + m] : 0.0f;
            }
            float w[16];
#pragma unroll
            for (uint32_t u = 0; u < 16; u += 4) {
                const float4 x = *reinterpret_cast<const float4*>(slab + lane * LD + i0 + u);
                w[u] = x.x; w[u + 1] = x.y; w[u + 2] = x.z; w[u + 3] = x.w;
            }
#pragma unroll
            for (uint32_t u = 0; u < 16; ++u)
                if (n0 + i0 + u < p.M && n0 + i0 + u > m) C[(int64_t)(n0 + i0 + u) * p.ldc + m] = w[u] + old[u];
        }
    }
}

// A CTA owns a tile of T x 128 rows by T x 128 columns; T = 1 is for products of few tiles (launch_gemm).
template <int NPL, int T>
__global__ void __launch_bounds__(384, 3 - T)
gemm_nt_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               const GemmParams p) {
    constexpr uint32_t MAXS = 8;
    constexpr uint32_t A_BYTES = T * NPL * GTILE_BYTES;  // row blocks x planes
    constexpr uint32_t STAGE_BYTES = 2 * A_BYTES;
    constexpr uint32_t TILE = 128u * T, TMEM_COLS = 128u * T * T;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bar_full[MAXS];
    __shared__ uint64_t bar_empty[MAXS];
    __shared__ uint64_t bar_acc;
    __shared__ uint32_t tmem_slot;
    __shared__ uint32_t abort_word;
    __shared__ float col_factor[TILE];  // inverse scale of every column of this tile (1 when unscaled)
    volatile uint32_t* abort_flag = &abort_word;

    // Tile order: CTAs are numbered so that the ~148 that run together cover a block of about
    // 12 x 12 tiles (12 row panels of A and 12 of B share L2) instead of a few rows of all columns.
    constexpr uint32_t GROUP_M = 12;
    const uint32_t tiles_n = gridDim.x, tiles_m = gridDim.y;
    const uint32_t id = blockIdx.y * tiles_n + blockIdx.x;
    const uint32_t width = GROUP_M * tiles_n;
    const uint32_t first_m = (id / width) * GROUP_M;
    const uint32_t gsize = min(tiles_m - first_m, GROUP_M);
    const uint32_t tile_m = first_m + (id % width) % gsize, tile_n = (id % width) / gsize;
    if (p.symmetric && tile_n < tile_m) return;  // whole CTA leaves before any barrier or TMEM use
    const uint32_t kb_first = blockIdx.z * p.kb_per_split, kb_end = min(p.kblocks, kb_first + p.kb_per_split);

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t S = p.stages;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < S; ++s) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        mbar_init(smem_u32(&bar_acc), 1);
        abort_word = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_slot), TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;
    after_earlier_launch();

    if (warp == 0 && lane == 0) {
        // ------------------------------- TMA producer -------------------------------
        prefetch_tmap(&map_a);
        prefetch_tmap(&map_b);
        uint32_t slot = 0, ph = 0;
        for (uint32_t kb = kb_first; kb < kb_end; ++kb) {
            if (!mbar_wait(smem_u32(&bar_empty[slot]), ph ^ 1u, abort_flag)) {
                gemm_fail(p.status, abort_flag, ST_TIMEOUT_EMPTY, kb);
                break;
            }
            const uint32_t bar = smem_u32(&bar_full[slot]);
            const uint32_t sa = smem_base + slot * STAGE_BYTES, sb = sa + A_BYTES;
            mbar_expect_tx(bar, STAGE_BYTES);
            // packed row index of (row block rb, k block kb, plane pl): ((rb*kblocks + kb)*NPL + pl)*128
#pragma unroll
            for (uint32_t h = 0; h < T; ++h) {
                const uint32_t rb_a = tile_m * T + h, rb_b = tile_n * T + h;
#pragma unroll
                for (uint32_t pl = 0; pl < (uint32_t)NPL; ++pl) {
                    // A: [block h][plane]; B: [plane][block h] so that 256 rows of one plane are adjacent
                    tma_load_2d(sa + (h * NPL + pl) * GTILE_BYTES, &map_a, 0,
                                (int)(((rb_a * p.kblocks + kb) * NPL + pl) * 128u), bar);
                    tma_load_2d(sb + (pl * T + h) * GTILE_BYTES, &map_b, 0,
                                (int)(((rb_b * p.kblocks + kb) * NPL + pl) * 128u), bar);
                }
            }
            if (++slot == S) {
                slot = 0;
                ph ^= 1u;
            }
        }
    } else if (warp == 1) {
        // -------------------------------- MMA issuer --------------------------------
        // whole warp in the loop, one elected lane issues (descriptors stay in uniform registers)
        const bool leader = elect_one();
        uint32_t slot = 0, ph = 0;
        bool ok = true;
        for (uint32_t kb = kb_first; kb < kb_end; ++kb) {
            const bool got = mbar_wait(smem_u32(&bar_full[slot]), ph, abort_flag);
            if (!__all_sync(0xffffffffu, got)) {
                if (leader) gemm_fail(p.status, abort_flag, ST_TIMEOUT_FULL_B, kb);
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t sa = smem_base + slot * STAGE_BYTES, sb = sa + A_BYTES;
            const uint64_t b_hi = smem_desc_k_sw64(sb), b_lo = smem_desc_k_sw64(sb + T * GTILE_BYTES);
#pragma unroll
            for (uint32_t mb = 0; mb < T; ++mb) {
                const uint32_t d = tmem_base + mb * TILE;
                const uint64_t a_hi = smem_desc_k_sw64(sa + (mb * NPL) * GTILE_BYTES);
                const uint64_t a_lo = smem_desc_k_sw64(sa + (mb * NPL + (NPL - 1)) * GTILE_BYTES);
                if (leader) {
#pragma unroll
                    for (uint32_t kk = 0; kk < 2; ++kk) {
                        const uint32_t acc = (kb > kb_first || kk > 0) ? 1u : 0u;
                        umma_f16_ss(d, a_hi + 2u * kk, b_hi + 2u * kk, p.idesc, acc);
                        if (NPL == 2) {
                            umma_f16_ss(d, a_hi + 2u * kk, b_lo + 2u * kk, p.idesc, 1u);
                            umma_f16_ss(d, a_lo + 2u * kk, b_hi + 2u * kk, p.idesc, 1u);
                        }
                    }
                }
            }
            if (leader) tc_commit(smem_u32(&bar_empty[slot]));
            if (++slot == S) {
                slot = 0;
                ph ^= 1u;
            }
        }
        if (ok && leader) tc_commit(smem_u32(&bar_acc));
    } else if (warp >= 4) {
        // --------------------------------- epilogue ---------------------------------
        const uint32_t q = warp & 3u, chalf = (warp - 4u) >> 2;  // TMEM lane quarter, column half
        {
            const uint32_t t = threadIdx.x - 128u, n = tile_n * TILE + t;
            if (t < TILE) col_factor[t] = (p.amax_b && n < p.N) ? row_scale_down(p.amax_b[n]) : 1.0f;
            asm volatile("bar.sync 1, 256;" ::: "memory");  // the eight epilogue warps only
        }
        bool got = mbar_wait(smem_u32(&bar_acc), 0u, abort_flag);
        got = __all_sync(0xffffffffu, got);
        if (!got) {
            if (lane == 0) gemm_fail(p.status, abort_flag, ST_TIMEOUT_ACC, warp);
        } else {
            tc_fence_after();
            const uint32_t lane_base = (q * 32u) << 16;
            // The pipeline buffers are idle by now (the commit behind bar_acc covered every MMA and
            // every load has been consumed): each warp turns its 32 x 128 blocks around in its own slab.
            constexpr uint32_t COLS = 64u * T, LD = slab_ld(COLS);  // columns of one epilogue warp
            float* slab = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw))) +
                          (size_t)(warp - 4u) * (32u * LD);
            float* C = p.C + blockIdx.z * p.split_stride;
#pragma unroll 1
            for (uint32_t mb = 0; mb < T; ++mb) {
                const uint32_t m_first = tile_m * TILE + mb * 128u + q * 32u, m = m_first + lane;
                const float rs = p.alpha * ((p.row_scale && m < p.M) ? p.row_scale[m] : 1.0f);
                const float fa = (p.amax_a && m < p.M) ? row_scale_down(p.amax_a[m]) : 1.0f;
#pragma unroll 1
                for (uint32_t cb = 0; cb < COLS / 16u; cb += 2) {
                    const uint32_t c0 = chalf * COLS + cb * 16u;
                    uint32_t r0[16], r1[16];
                    tmem_ld_x16(tmem_base + lane_base + mb * TILE + c0, r0);
                    tmem_ld_x16(tmem_base + lane_base + mb * TILE + c0 + 16u, r1);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; j += 4) {
                        float lo[4], hi[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            lo[e] = ((__uint_as_float(r0[j + e]) * fa) * col_factor[c0 + j + e]) * rs;
                            hi[e] = ((__uint_as_float(r1[j + e]) * fa) * col_factor[c0 + 16u + j + e]) * rs;
                        }
                        float* to = slab + lane * LD + cb * 16u + j;
                        *reinterpret_cast<float4*>(to) = make_float4(lo[0], lo[1], lo[2], lo[3]);
                        *reinterpret_cast<float4*>(to + 16) = make_float4(hi[0], hi[1], hi[2], hi[3]);
                    }
                }
                __syncwarp();
                store_block_from_slab<COLS>(p, C, slab, m_first, tile_n * TILE + chalf * COLS, lane);
                __syncwarp();  // the slab is rewritten for the second row block
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) __nanosleep(200000);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// ---- chunked accumulation: the variant for products whose error gets amplified ---------------
// The tensor core adds into its fp32 accumulator by truncation, not rounding: every MMA whose
// addends reach below the accumulator's last place pulls the sum towards zero by up to one unit
// in the last place, and a K-long contraction is a chain of 3K/16 such steps (measured: 1e-5
// relative at K = 3000, 2e-3 in the scores once a Gram with condition number 1000 is inverted,
// where plain fp32 arithmetic gives 3e-5).  Here the chain is cut every 64 k: one CTA owns a
// 128 x 256 tile, TMEM holds two accumulator sets, the MMA warp fills one set with a 64-wide
// chunk -- per 32-k slot the hi*lo and lo*hi terms, then the two hi*hi MMAs, after which the
// slot goes back to the producer -- while the eight epilogue warps read the other set and add it,
// with ordinary rounded fp32 adds, to running sums they keep in registers (128 per thread).
// (Issuing all small terms of a chunk before its large ones halves the truncation that is left,
// a mean error of -2.3e-7 instead of -3.0e-7 on a Gram diagonal, but holds both slots until the
// chunk's end, and with only four slots the loads then arrive late: 12.6 against 11.5 ms.)
// TN = 128 halves the columns of a tile, for products of so few tiles that SMs are left idle (plan_gemm): each entry of the
// result comes of the same operations in the same order.
template <uint32_t TN>
struct Chunked {
    static constexpr uint32_t BLOCKS = TN / 128u;                            // row blocks of B
    static constexpr uint32_t SLOTS = TN == 256u ? 4u : 6u;
    static constexpr uint32_t SLOT_BYTES = (2u + 2u * BLOCKS) * GTILE_BYTES;  // A: hi, lo; B: [plane][row block]  (per 32 k)
};

template <uint32_t TN>
__global__ void __launch_bounds__(384, 1)
gemm_nt_chunked_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                       const GemmParams p) {
    constexpr uint32_t BLOCKS = Chunked<TN>::BLOCKS, SLOTS = Chunked<TN>::SLOTS, SLOT_BYTES = Chunked<TN>::SLOT_BYTES;
    constexpr uint32_t COLS = TN / 2u;  // of an epilogue warp
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t bar_full[SLOTS];
    __shared__ uint64_t bar_empty[SLOTS];
    __shared__ uint64_t bar_acc_full[2];
    __shared__ uint64_t bar_acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ uint32_t abort_word;
    __shared__ float col_factor[TN];
    volatile uint32_t* abort_flag = &abort_word;

    // same L2-friendly numbering as gemm_nt_kernel, with 128-row tiles
    constexpr uint32_t GROUP_M = 16;
    const uint32_t tiles_n = gridDim.x, tiles_m = gridDim.y;
    const uint32_t id = blockIdx.y * tiles_n + blockIdx.x;
    const uint32_t width = GROUP_M * tiles_n;
    const uint32_t first_m = (id / width) * GROUP_M;
    const uint32_t gsize = min(tiles_m - first_m, GROUP_M);
    uint32_t tile_m = first_m + (id % width) % gsize;
    const uint32_t tile_n = (id % width) / gsize;
    if (p.range == K_TO_ROW) tile_m = tiles_m - 1u - tile_m;  // the longest contractions first
    // symmetric: a tile is needed when it holds some entry with n >= m
    if (p.symmetric && tile_n < tile_m / BLOCKS) return;

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    // The k blocks of this tile, less those where an operand is zero (a triangular factor: a third of W^T W and half of
    // a merge is left), and of them this slice's.  Starts are multiples of 128 and slices even: whole chunks.
    uint32_t kb_lo = 0, kb_hi = p.kblocks;
    if (p.range == K_FROM_ROW) kb_lo = min(p.kblocks, max(tile_m * 4u, p.symmetric ? tile_n * (4u * BLOCKS) : 0u));
    if (p.range == K_TO_ROW) kb_hi = min(p.kblocks, tile_m * 4u + 4u);
    if (p.range == K_TO_COL) kb_hi = min(p.kblocks, (tile_n + 1u) * (4u * BLOCKS));
    const uint32_t slice = ((kb_hi - kb_lo + gridDim.z - 1u) / gridDim.z + 1u) & ~1u;
    const uint32_t kb_first = min(kb_hi, kb_lo + blockIdx.z * slice), kb_end = min(kb_hi, kb_first + slice);
    const uint32_t nchunks = (kb_end - kb_first + 1u) >> 1;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < SLOTS; ++s) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        for (uint32_t s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&bar_acc_full[s]), 1);
            mbar_init(smem_u32(&bar_acc_empty[s]), 8);  // one arrival per epilogue warp
        }
        abort_word = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_slot), 2u * TN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;
    after_earlier_launch();

    // Registers follow the work: the warpgroup of the two single-thread roles gives most of its
    // allocation back (168 -> 56 per thread), the two epilogue warpgroups take it (168 -> 224:
    // 128 running sums + 64 values in flight).  Each role's code sits wholly inside its branch,
    // which is what lets the compiler allocate past the launch bound there.
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == 0 && lane == 0) {
            // ------------------------------- TMA producer -------------------------------
            prefetch_tmap(&map_a);
            prefetch_tmap(&map_b);
            uint32_t slot = 0, ph = 0;
            for (uint32_t kb = kb_first; kb < kb_end; ++kb) {
                if (!mbar_wait(smem_u32(&bar_empty[slot]), ph ^ 1u, abort_flag)) {
                    gemm_fail(p.status, abort_flag, ST_TIMEOUT_EMPTY, kb);
                    break;
                }
                const uint32_t bar = smem_u32(&bar_full[slot]);
                const uint32_t sa = smem_base + slot * SLOT_BYTES, sb = sa + 2u * GTILE_BYTES;
                mbar_expect_tx(bar, SLOT_BYTES);
#pragma unroll
                for (uint32_t pl = 0; pl < 2; ++pl) {
                    tma_load_2d(sa + pl * GTILE_BYTES, &map_a, 0, (int)(((tile_m * p.kblocks + kb) * 2u + pl) * 128u), bar);
#pragma unroll
                    for (uint32_t h = 0; h < BLOCKS; ++h)
                        tma_load_2d(sb + (pl * BLOCKS + h) * GTILE_BYTES, &map_b, 0,
                                    (int)((((tile_n * BLOCKS + h) * p.kblocks + kb) * 2u + pl) * 128u), bar);
                }
                if (++slot == SLOTS) {
                    slot = 0;
                    ph ^= 1u;
                }
            }
        } else if (warp == 1) {
            // -------------------------------- MMA issuer --------------------------------
            // The whole warp runs the loop and one elected lane issues: with warp-uniform control flow the
            // descriptors and addresses stay in uniform registers, which the MMA and commit instructions
            // take directly (computed under a one-lane branch each would be moved there first).
            const bool leader = elect_one();
            uint32_t slot = 0, ph = 0;  // a chunk takes slots (slot, slot + 1); slot stays even, so no wrap inside one
            bool ok = true;
            for (uint32_t c = 0; c < nchunks && ok; ++c) {
                const uint32_t set = c & 1u, use = c >> 1;
                bool got = mbar_wait(smem_u32(&bar_acc_empty[set]), (use & 1u) ^ 1u, abort_flag);
                if (!__all_sync(0xffffffffu, got)) {
                    if (leader) gemm_fail(p.status, abort_flag, ST_TIMEOUT_ACC, 0x10000u + c);
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem_base + set * TN;
                const uint32_t nkb = min(2u, kb_end - kb_first - 2u * c);
                // per 32-k slot: its small terms first, then its large ones, and the slot is released
                for (uint32_t j = 0; j < nkb; ++j) {
                    got = mbar_wait(smem_u32(&bar_full[slot + j]), ph, abort_flag);
                    if (!__all_sync(0xffffffffu, got)) {
                        if (leader) gemm_fail(p.status, abort_flag, ST_TIMEOUT_FULL_B, 2u * c + j);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = smem_base + (slot + j) * SLOT_BYTES, sb = sa + 2u * GTILE_BYTES;
                    const uint64_t a_hi = smem_desc_k_sw64(sa), a_lo = smem_desc_k_sw64(sa + GTILE_BYTES);
                    const uint64_t b_hi = smem_desc_k_sw64(sb), b_lo = smem_desc_k_sw64(sb + BLOCKS * GTILE_BYTES);
                    if (leader) {
#pragma unroll
                        for (uint32_t kk = 0; kk < 2; ++kk) {
                            umma_f16_ss(d, a_hi + 2u * kk, b_lo + 2u * kk, p.idesc, (j > 0 || kk > 0) ? 1u : 0u);
                            umma_f16_ss(d, a_lo + 2u * kk, b_hi + 2u * kk, p.idesc, 1u);
                        }
#pragma unroll
                        for (uint32_t kk = 0; kk < 2; ++kk) umma_f16_ss(d, a_hi + 2u * kk, b_hi + 2u * kk, p.idesc, 1u);
                        tc_commit(smem_u32(&bar_empty[slot + j]));
                    }
                }
                if (!ok) break;
                if (leader) tc_commit(smem_u32(&bar_acc_full[set]));
                slot += nkb;
                if (slot >= SLOTS) {
                    slot = 0;
                    ph ^= 1u;
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
        // ---------------------- running sums, then the epilogue ----------------------
        const uint32_t q = warp & 3u, chalf = (warp - 4u) >> 2;  // TMEM lane quarter, column half
        {
            const uint32_t t = threadIdx.x - 128u, n = tile_n * TN + t;
            if (t < TN) col_factor[t] = (p.amax_b && n < p.N) ? row_scale_down(p.amax_b[n]) : 1.0f;
            asm volatile("bar.sync 1, 256;" ::: "memory");  // the eight epilogue warps only
        }
        const uint32_t lane_base = (q * 32u) << 16;
        float sum[COLS];
#pragma unroll
        for (int i = 0; i < (int)COLS; ++i) sum[i] = 0.0f;
        bool ok = true;
#pragma unroll 1
        for (uint32_t c = 0; c < nchunks; ++c) {
            const uint32_t set = c & 1u, use = c >> 1;
            bool got = mbar_wait(smem_u32(&bar_acc_full[set]), use & 1u, abort_flag);
            got = __all_sync(0xffffffffu, got);
            if (!got) {
                if (lane == 0) gemm_fail(p.status, abort_flag, ST_TIMEOUT_ACC, c);
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t t0 = tmem_base + lane_base + set * TN + chalf * COLS;
#pragma unroll
            for (uint32_t cb = 0; cb < COLS / 16u; cb += 4) {  // four loads in flight per wait
                uint32_t r[4][16];
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) tmem_ld_x16(t0 + (cb + u) * 16u, r[u]);
                tmem_wait_ld();
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u)
#pragma unroll
                    for (int j = 0; j < 16; ++j) sum[(cb + u) * 16 + j] += __uint_as_float(r[u][j]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_acc_empty[set]));
        }
        if (ok) {
            const uint32_t m = tile_m * 128u + q * 32u + lane;
            const uint32_t n0 = tile_n * TN + chalf * COLS;
            const float rs = p.alpha * ((p.row_scale && m < p.M) ? p.row_scale[m] : 1.0f);
            const float fa = (p.amax_a && m < p.M) ? row_scale_down(p.amax_a[m]) : 1.0f;
#pragma unroll
            for (int i = 0; i < (int)COLS; ++i) sum[i] = ((sum[i] * fa) * col_factor[chalf * COLS + i]) * rs;
            // The pipeline buffers are idle by now (the last commit covered every MMA and every load
            // has been consumed), so each warp turns its 32 x 128 block around in its own slab of them.
            float* slab = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw))) +
                          (size_t)(warp - 4u) * (32u * slab_ld(COLS));
#pragma unroll
            for (int i = 0; i < (int)COLS; i += 4)
                *reinterpret_cast<float4*>(slab + lane * slab_ld(COLS) + i) =
                    make_float4(sum[i], sum[i + 1], sum[i + 2], sum[i + 3]);
            __syncwarp();
            store_block_from_slab<COLS>(p, p.C + blockIdx.z * p.split_stride, slab, tile_m * 128u + q * 32u, n0, lane);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) __nanosleep(200000);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 2u * TN);
    }
}

// ---- fp32 operands whose rows are source rows: row maxima and packing in one pass ---------------
// packed[((rb*kblocks + kb)*2 + pl)*128 + r][kk] as below; amax[R] = bit pattern of max_k |operand[R][k]|
// (non-negative floats order like their bits).  W warps share a row and keep it in registers (32 floats a lane,
// W * 1024 k) between the maximum and the packing, so the source is read once -- two kernels, the second reading it
// again, moved 12 bytes per element instead of 8.  Longer rows are walked twice in steps of that length.
// One launch packs both operands of a product: rows beyond the first operand's belong to the second.
struct PackRows {
    const float* src;
    uint16_t* packed;
    uint32_t* amax;
    uint64_t rows, K, ld;
    uint32_t rowblocks, kblocks;
};
template <int W, int THREADS = 256>
__global__ void __launch_bounds__(THREADS) pack_rows_f32_kernel(const PackRows a, const PackRows b) {
    after_earlier_launch();
    constexpr uint32_t ROWS = THREADS / 32 / W;  // of a CTA
    __shared__ uint32_t row_max[THREADS / 32];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, part = warp % W;
    constexpr uint32_t SPAN = W * 1024u;
    const uint64_t rows_a = (uint64_t)a.rowblocks * 128u, total = rows_a + (uint64_t)b.rowblocks * 128u;
    for (uint64_t row0 = (uint64_t)blockIdx.x * ROWS; row0 < total; row0 += (uint64_t)gridDim.x * ROWS) {
        const uint64_t i = row0 + warp / W;  // ROWS divides 128: a CTA's rows belong to one operand
        const bool first = i < rows_a;
        const PackRows& o = first ? a : b;
        const uint64_t R = first ? i : i - rows_a, span_k = (uint64_t)o.kblocks * 32u;
        const float* src = o.src + R * o.ld;
        const bool live = R < o.rows, vec = (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
        float x[4][8];
        auto load = [&](uint64_t base) {
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint64_t k = base + (part * 4u + j) * 256u + lane * 8u;
                if (live && vec && k + 8u <= o.K) {
                    const float4 lo = __ldg(reinterpret_cast<const float4*>(src + k));
                    const float4 hi = __ldg(reinterpret_cast<const float4*>(src + k) + 1);
                    x[j][0] = lo.x; x[j][1] = lo.y; x[j][2] = lo.z; x[j][3] = lo.w;
                    x[j][4] = hi.x; x[j][5] = hi.y; x[j][6] = hi.z; x[j][7] = hi.w;
                } else {
#pragma unroll
                    for (uint32_t e = 0; e < 8; ++e) x[j][e] = (live && k + e < o.K) ? __ldg(src + k + e) : 0.0f;
                }
            }
        };
        uint32_t m = 0;
        for (uint64_t base = 0; base < o.K; base += SPAN) {
            load(base);
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
#pragma unroll
                for (uint32_t e = 0; e < 8; ++e) m = max(m, __float_as_uint(x[j][e]) & 0x7fffffffu);
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
        if (W > 1) {
            if (lane == 0) row_max[warp] = m;
            __syncthreads();
#pragma unroll
            for (uint32_t w = 0; w < W; ++w) m = max(m, row_max[warp / W * W + w]);
            __syncthreads();
        }
        if (live && part == 0 && lane == 0) o.amax[R] = m;
        const float up = row_scale_up(m);
        uint16_t* out = o.packed + ((R >> 7) * o.kblocks * 256u + (R & 127u)) * 32u;
        for (uint64_t base = 0; base < span_k; base += SPAN) {
            if (o.K > SPAN) load(base);
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint64_t k = base + (part * 4u + j) * 256u + lane * 8u;
                if (k >= span_k) continue;
                uint32_t hi[4], lo[4];
#pragma unroll
                for (uint32_t e = 0; e < 4; ++e) {
                    const float u = x[j][2 * e] * up, v = x[j][2 * e + 1] * up;  // exact: a power of two, below 2^15
                    const __half2 h = __floats2half2_rn(u, v);
                    const __half2 l = __floats2half2_rn(u - __low2float(h), v - __high2float(h));  // exact differences
                    hi[e] = *reinterpret_cast<const uint32_t*>(&h);
                    lo[e] = *reinterpret_cast<const uint32_t*>(&l);
                }
                uint16_t* dst = out + (k >> 5) * (256u * 32u) + (k & 31u);
                *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(dst + 128u * 32u) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
        }
    }
}

// ---- transposed fp32 operands -------------------------------------------------------------------
// Operand rows are source columns (the operand is the transpose): threads along the columns,
// blockIdx.y walks chunks of source rows; amax must be zero before the launch.
__global__ void amax_cols_kernel(const float* __restrict__ src, uint32_t* __restrict__ amax, uint64_t rows,
                                 uint64_t K, uint64_t ld, uint64_t chunk) {
    after_earlier_launch();
    const uint64_t R = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (R >= rows) return;
    const uint64_t k0 = (uint64_t)blockIdx.y * chunk, k1 = min(K, k0 + chunk);
    const uint32_t* col = reinterpret_cast<const uint32_t*>(src) + R;
    uint32_t m = 0;
#pragma unroll 8
    for (uint64_t k = k0; k < k1; ++k) m = max(m, col[k * ld] & 0x7fffffffu);
    atomicMax(&amax[R], m);
}

// The same and the packing in one launch for up to J * 256 source rows: a CTA keeps 16 source columns in registers, 8
// consecutive k at a time per thread, finds their maxima and writes both planes.  Bound by latency: a memset, the maxima
// and the packing were three launches of 1 to 8 us with gaps as long (Gram of 2048 x 2048: 70 -> 60 us in all,
// 2000 x 8192: 430 -> 408).  Longer columns do not fit and go through the two kernels, which stream them.
template <int J>
__global__ void __launch_bounds__(512) pack_cols_f32_kernel(const float* __restrict__ src, uint16_t* __restrict__ packed,
                                                            uint32_t* __restrict__ amax, uint64_t rows, uint64_t K,
                                                            uint64_t ld, uint32_t kblocks) {
    after_earlier_launch();
    __shared__ uint32_t warp_max[16][16];
    const uint32_t c = threadIdx.x & 15u, group = threadIdx.x >> 4, warp = threadIdx.x >> 5;
    const uint64_t R = (uint64_t)blockIdx.x * 16u + c, span_k = (uint64_t)kblocks * 32u;
    const bool live = R < rows;
    float x[J][8];
    uint32_t m = 0;
#pragma unroll
    for (int j = 0; j < J; ++j)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint64_t k = (uint32_t)(j * 256 + e) + group * 8u;
            x[j][e] = (live && k < K) ? __ldg(src + k * ld + R) : 0.0f;
        }
#pragma unroll
    for (int j = 0; j < J; ++j)
#pragma unroll
        for (int e = 0; e < 8; ++e) m = max(m, __float_as_uint(x[j][e]) & 0x7fffffffu);
    m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
    if ((threadIdx.x & 16u) == 0) warp_max[warp][c] = m;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 16; ++w) m = max(m, warp_max[w][c]);
    if (live && group == 0) amax[R] = m;
    const float up = row_scale_up(m);
    uint16_t* out = packed + ((R >> 7) * kblocks * 256u + (R & 127u)) * 32u;
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const uint32_t k = (uint32_t)j * 256u + group * 8u;
        if (k >= span_k) continue;
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float u = x[j][2 * e] * up, v = x[j][2 * e + 1] * up;
            const __half2 h = __floats2half2_rn(u, v);
            const __half2 l = __floats2half2_rn(u - __low2float(h), v - __high2float(h));
            hi[e] = *reinterpret_cast<const uint32_t*>(&h);
            lo[e] = *reinterpret_cast<const uint32_t*>(&l);
        }
        uint16_t* dst = out + (k >> 5) * (256u * 32u) + (k & 31u);
        *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(dst + 128u * 32u) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
}

// ---- packing ---------------------------------------------------------------------------
// packed[((rb*kblocks + kb)*planes + pl)*128 + r][kk]  (16-bit), r < 128, kk < 32:
//   operand row  R = rb*128 + r,  k = kb*32 + kk;
//   value = src[R*ld + k]  (TRANS = false)  or  src[k*ld + R]  (TRANS = true: the operand is the
//   transpose of the row-major source), zero outside [rows x K].
// 16-bit types, copied as they are.
template <bool TRANS, int THREADS = 256>
__global__ void __launch_bounds__(THREADS) pack_kernel(const uint16_t* __restrict__ src, uint16_t* __restrict__ packed, uint64_t rows,
                            uint64_t K, uint64_t ld, uint32_t rowblocks, uint32_t kblocks) {
    after_earlier_launch();
    // one thread = 8 consecutive k of one operand row (a 16-byte store)
    const uint64_t total = (uint64_t)rowblocks * kblocks * 128u * 4u;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t r, oct;
        uint64_t rest;
        if (TRANS) {  // lanes run along operand rows = consecutive source columns
            r = (uint32_t)(i & 127u);
            oct = (uint32_t)((i >> 7) & 3u);
        } else {      // lanes run along k = consecutive source columns
            oct = (uint32_t)(i & 3u);
            r = (uint32_t)((i >> 2) & 127u);
        }
        rest = i >> 9;
        // consecutive CTAs take neighbouring pieces of the same source rows: along k when the operand
        // rows are source rows, along the operand rows when they are source columns
        uint32_t kb;
        uint64_t rb;
        if (rest <= 0xffffffffull) {  // 32-bit divisions whenever the piece number fits (it nearly always does)
            const uint32_t r32 = (uint32_t)rest, d = TRANS ? rowblocks : kblocks, q = r32 / d, m = r32 - q * d;
            kb = TRANS ? q : m;
            rb = TRANS ? m : q;
        } else {
            kb = TRANS ? (uint32_t)(rest / rowblocks) : (uint32_t)(rest % kblocks);
            rb = TRANS ? rest % rowblocks : rest / kblocks;
        }
        const uint64_t R = rb * 128u + r, k0 = (uint64_t)kb * 32u + oct * 8u;
        uint4 o;
        const uint16_t* from = src + R * ld + k0;
        if (!TRANS && R < rows && k0 + 8u <= K && (reinterpret_cast<uintptr_t>(from) & 15u) == 0) {
            o = __ldg(reinterpret_cast<const uint4*>(from));
        } else {
            uint16_t v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)
                v[e] = (R < rows && k0 + e < K) ? (TRANS ? src[(k0 + e) * ld + R] : from[e]) : (uint16_t)0;
            o.x = v[0] | ((uint32_t)v[1] << 16);
            o.y = v[2] | ((uint32_t)v[3] << 16);
            o.z = v[4] | ((uint32_t)v[5] << 16);
            o.w = v[6] | ((uint32_t)v[7] << 16);
        }
        *reinterpret_cast<uint4*>(packed + (((rb * kblocks + kb) * 128u + r) * 32u + oct * 8u)) = o;
    }
}

// The transposed fp32 case through shared memory: one CTA step = one [128 operand rows x 32 k]
// tile, i.e. 32 source rows x 128 source columns.  Reads are 512-byte runs of source rows, and
// after the transpose in shared memory each plane of the tile leaves as one contiguous 8 KB run
// (the generic kernel's transposed stores are 16-byte pieces 64 bytes apart).
__global__ void __launch_bounds__(256) pack_trans_f32_kernel(const float* __restrict__ src, uint16_t* __restrict__ packed,
                                                             const uint32_t* __restrict__ amax, uint64_t rows, uint64_t K,
                                                             uint64_t ld, uint32_t rowblocks, uint32_t kblocks) {
    after_earlier_launch();
    constexpr int LDS = 34;  // padded row of a plane tile, in 16-bit elements (17 words: conflict-free)
    __shared__ __align__(16) uint16_t tile[2][128][LDS];
    const uint32_t c = threadIdx.x & 127u, half = threadIdx.x >> 7;
    const uint64_t ntiles = (uint64_t)rowblocks * kblocks;
    for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const uint64_t rb = t % rowblocks, kb = t / rowblocks;  // neighbouring CTAs: neighbouring runs of the same source rows
        const uint64_t R = rb * 128u + c;
        const float up = R < rows ? row_scale_up(amax[R]) : 1.0f;
#pragma unroll 4
        for (uint32_t pass = 0; pass < 16; ++pass) {
            const uint32_t kk = pass * 2u + half;
            const uint64_t k = kb * 32u + kk;
            float x = 0.0f;
            if (R < rows && k < K) x = src[k * ld + R];
            const float xs = x * up;
            const __half h = __float2half_rn(xs);
            const __half l = __float2half_rn(xs - __half2float(h));
            tile[0][c][kk] = __half_as_ushort(h);
            tile[1][c][kk] = __half_as_ushort(l);
        }
        __syncthreads();
        uint16_t* dst = packed + (rb * kblocks + kb) * 2u * 128u * 32u;
#pragma unroll
        for (uint32_t it = 0; it < 4; ++it) {
            const uint32_t q = it * 256u + threadIdx.x;       // 16-byte piece: plane, row, eighth
            const uint32_t pl = q >> 9, r = (q >> 2) & 127u, oct = q & 3u;
            const uint32_t* w = reinterpret_cast<const uint32_t*>(&tile[pl][r][oct * 8u]);
            uint4 o;
            o.x = w[0];
            o.y = w[1];
            o.z = w[2];
            o.w = w[3];
            *reinterpret_cast<uint4*>(dst + (size_t)q * 8u) = o;
        }
        __syncthreads();
    }
}

// ---- sum of the partial products of a split contraction ------------------------------------------
// C (+)= ((sum_z partial[z]) * scale_a[m] * scale_b[n]) * alpha * row_scale[m], slices added in their order.  One CTA
// per 32 x 32 block; symmetric products hold (and write) the blocks on or above the diagonal and turn each around in
// shared memory for its second copy.
__global__ void __launch_bounds__(256) reduce_splits_kernel(const float* __restrict__ partial, uint32_t splits,
                                                            const GemmParams p) {
    after_earlier_launch();
    __shared__ float turn[32][33];
    const uint32_t bm = blockIdx.y, bn = blockIdx.x, tx = threadIdx.x & 31u, ty = threadIdx.x >> 5;
    if (p.symmetric && bn < bm) return;
    const uint32_t n = bn * 32u + tx;
    float v[4];
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
        const uint32_t m = bm * 32u + ty + 8u * u;
        v[u] = 0.0f;
        if (m >= p.M || n >= p.N || (p.symmetric && n < m)) continue;
        const float* src = partial + (uint64_t)m * p.N + n;
        float sum = src[0];
        for (uint32_t z = 1; z < splits; ++z) sum += src[z * p.split_stride];
        const float rs = p.alpha * (p.row_scale ? p.row_scale[m] : 1.0f);
        const float fa = p.amax_a ? row_scale_down(p.amax_a[m]) : 1.0f;
        const float fb = p.amax_b ? row_scale_down(p.amax_b[n]) : 1.0f;
        v[u] = ((sum * fa) * fb) * rs;
        float* dst = p.C + (int64_t)m * p.ldc + n;
        *dst = p.accumulate ? *dst + v[u] : v[u];
    }
    if (!p.symmetric) return;
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) turn[ty + 8u * u][tx] = v[u];
    __syncthreads();
    const uint32_t m2 = bm * 32u + tx;
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
        const uint32_t n2 = bn * 32u + ty + 8u * u;
        if (n2 >= p.N || m2 >= n2) continue;  // strictly below the diagonal of C
        float* dst = p.C + (int64_t)n2 * p.ldc + m2;
        const float w = turn[tx][ty + 8u * u];
        *dst = p.accumulate ? *dst + w : w;
    }
}

// ---- host side -----------------------------------------------------------------------------
Packed packed_geometry(int dtype, int64_t rows, int64_t K) {
    Packed g;
    g.scaled = dtype == TB_F32;
    g.rowblocks = (uint32_t)((rows + 127) / 128);
    g.kblocks = (uint32_t)((K + 31) / 32);
    g.npl = dtype == TB_F32 ? 2u : 1u;
    g.data_bytes = align_up((size_t)g.rowblocks * g.kblocks * g.npl * GTILE_BYTES, 1024);
    // scaled operands carry the row maxima behind the tiles
    g.bytes = g.data_bytes + (g.scaled ? align_up((size_t)g.rowblocks * 128u * sizeof(uint32_t), 1024) : 0);
    return g;
}

static PackRows pack_rows_args(const void* src, uint64_t rows, uint64_t K, uint64_t ld, uint16_t* packed, const Packed& g) {
    return PackRows{static_cast<const float*>(src), packed, packed_amax(packed, g), rows, K, ld, g.rowblocks, g.kblocks};
}

// Whether the packing of so many operand elements is launched while the product before it on the stream still runs.  That
// gains 2 us, but the CTAs of a large one then fill the SMs unevenly, around those of the product: 37,000 x 100 x 2048 in
// a row took 110 us a product in fp16 and 174 in fp32 instead of 97 and 159, 20,000 x 100 x 2048 66 and 103 instead of 61
// and 97; the two meet at about 20 million elements (fp16 25,000 x 100 x 512 21.8 early and 23.2, 10,000 x 100 x 2048 38.0
// and 37.5; fp32 40,000 x 100 x 512 66.5 and 67.7, 60,000 x 100 x 512 81.6 and 80.7).
static bool pack_early(uint64_t elements) { return elements < 25'000'000u; }

// A packing that runs beside an inverse (tb_gemm_nt_pack_beside) leaves it half of the SMs: CTAs of 1024 threads, one to every
// second SM.  Spread over all of them it keeps the inverse's cooperative launch and its products,
// which want whole SMs, waiting until it has ended.  get_x_xtx_inv of 50,000 x 2048 fp32 1671 -> 1638 us, 65,000 x 1024
// 720 -> 704, 80,000 x 512 367 -> 356.
constexpr int BESIDE_THREADS = 1024;
static uint32_t beside_blocks(uint64_t blocks_of_256, int sm_count) {
    return (uint32_t)std::min<uint64_t>((blocks_of_256 + 3) / 4, std::max(1, sm_count / 2));
}

// One or two fp32 operands (b.rowblocks = 0: one) whose rows are source rows.
static int launch_pack_rows(const PackRows& a, const PackRows& b, int sm_count, cudaStream_t stream, bool beside = false) {
    const uint64_t K = a.K > b.K ? a.K : b.K, rows = ((uint64_t)a.rowblocks + b.rowblocks) * 128u;
    // warps per row: enough to hold it in registers, but not so many that most of their lanes idle
    const int w = K <= 1024u ? 1 : K <= 2048u ? 2 : K <= 4096u ? 4 : 8;
    if (beside) {
        auto kern = w == 1   ? pack_rows_f32_kernel<1, BESIDE_THREADS>
                    : w == 2 ? pack_rows_f32_kernel<2, BESIDE_THREADS>
                    : w == 4 ? pack_rows_f32_kernel<4, BESIDE_THREADS>
                             : pack_rows_f32_kernel<8, BESIDE_THREADS>;
        return launch_after(kern, beside_blocks((rows * w + 7) / 8, sm_count), BESIDE_THREADS, 0, stream, false, a, b);
    }
    uint64_t blocks = (rows * w + 7) / 8;
    const uint64_t cap = (uint64_t)sm_count * 32;
    if (blocks > cap) blocks = cap;
    const uint32_t nb = (uint32_t)blocks;
    const bool early = pack_early(a.rows * a.K + b.rows * b.K);
    if (w == 1) return launch_after(pack_rows_f32_kernel<1>, nb, 256, 0, stream, early, a, b);
    if (w == 2) return launch_after(pack_rows_f32_kernel<2>, nb, 256, 0, stream, early, a, b);
    if (w == 4) return launch_after(pack_rows_f32_kernel<4>, nb, 256, 0, stream, early, a, b);
    return launch_after(pack_rows_f32_kernel<8>, nb, 256, 0, stream, early, a, b);
}

int launch_pack_pair(const float* a, uint64_t rows_a, uint64_t K_a, uint64_t ld_a, uint16_t* packed_a, const Packed& ga,
                     const float* b, uint64_t rows_b, uint64_t K_b, uint64_t ld_b, uint16_t* packed_b, const Packed& gb,
                     int sm_count, cudaStream_t stream) {
    return launch_pack_rows(pack_rows_args(a, rows_a, K_a, ld_a, packed_a, ga),
                            pack_rows_args(b, rows_b, K_b, ld_b, packed_b, gb), sm_count, stream);
}

Packed packed_tail(const uint16_t** packed, const Packed& g, uint32_t skip) {
    const size_t skipped = (size_t)skip * g.kblocks * g.npl * GTILE_BYTES;
    Packed t = g;
    t.rowblocks -= skip;
    t.data_bytes = g.data_bytes - skipped + (size_t)skip * 128u * sizeof(uint32_t);  // the row maxima stay where they are
    t.bytes = g.bytes - skipped;
    *packed += skipped / sizeof(uint16_t);
    return t;
}

int launch_pack(const void* src, int dtype, bool trans, uint64_t rows, uint64_t K, uint64_t ld,
                uint16_t* packed, const Packed& g, int sm_count, cudaStream_t stream, bool beside) {
    if (dtype == TB_F32 && !trans)
        return launch_pack_rows(pack_rows_args(src, rows, K, ld, packed, g), PackRows{}, sm_count, stream, beside);
    if (dtype == TB_F32) {
        const float* s = static_cast<const float*>(src);
        uint32_t* amax = packed_amax(packed, g);
        if (K <= 2048u) {
            const uint32_t nb = g.rowblocks * 8u;
            auto kern = K <= 512u ? pack_cols_f32_kernel<2> : K <= 1024u ? pack_cols_f32_kernel<4> : pack_cols_f32_kernel<8>;
            return launch_after(kern, nb, 512, 0, stream, true, s, packed, amax, rows, K, ld, g.kblocks);
        }
        TB_CUDA(cudaMemsetAsync(amax, 0, (size_t)g.rowblocks * 128u * sizeof(uint32_t), stream));
        const uint32_t bx = (uint32_t)((rows + 255) / 256);
        uint64_t by = ((uint64_t)sm_count * 16 + bx - 1) / bx;  // about 16 CTAs per SM in all
        if (by > (K + 15) / 16) by = (K + 15) / 16;
        if (by > 65535) by = 65535;
        const uint64_t chunk = (K + by - 1) / by;
        amax_cols_kernel<<<dim3(bx, (uint32_t)((K + chunk - 1) / chunk)), 256, 0, stream>>>(s, amax, rows, K, ld, chunk);
        TB_CUDA(cudaGetLastError());
        uint64_t tb = (uint64_t)g.rowblocks * g.kblocks;
        if (tb > (uint64_t)sm_count * 16) tb = (uint64_t)sm_count * 16;
        return launch_after(pack_trans_f32_kernel, (uint32_t)tb, 256, 0, stream, true, s, packed, amax, rows, K, ld, g.rowblocks,
                            g.kblocks);
    } else {
        const uint64_t total = (uint64_t)g.rowblocks * g.kblocks * 512u;
        uint64_t blocks = (total + 255) / 256;
        const uint64_t cap = (uint64_t)sm_count * 32;
        if (blocks > cap) blocks = cap;
        const uint32_t nb = (uint32_t)blocks;
        const uint16_t* s = static_cast<const uint16_t*>(src);
        if (beside && !trans)
            return launch_after(pack_kernel<false, BESIDE_THREADS>, beside_blocks((total + 255) / 256, sm_count), BESIDE_THREADS, 0,
                                stream, false, s, packed, rows, K, ld, g.rowblocks, g.kblocks);
        return launch_after(trans ? pack_kernel<true> : pack_kernel<false>, nb, 256, 0, stream, trans || pack_early(rows * K), s,
                            packed, rows, K, ld, g.rowblocks, g.kblocks);
    }
}

// element format of the planes: fp16 for fp16 inputs and for scaled fp32 operands, else bf16
static bool planes_are_fp16(const Packed& g, int dtype) { return dtype == TB_F16 || g.scaled; }

static int packed_tmap(CUtensorMap* map, const uint16_t* packed, const Packed& g, int dtype) {
    const uint64_t dims[2] = {GK, (uint64_t)g.rowblocks * g.kblocks * g.npl * 128u};
    const uint64_t strides[1] = {GK * 2u};
    const uint32_t box[2] = {GK, 128};
    return encode_tmap(map, planes_are_fp16(g, dtype) ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                       2, packed, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B);
}

constexpr uint32_t B200_SMS = 148;

// Tile and number of slices of the contraction.  A 256 x 256 (chunked: 128 x 256) tile per CTA leaves most of the 148 SMs
// idle when the product is small: the Gram of 2048 columns is 36 such tiles however many rows it sums over.  The
// choice minimises an estimate in microseconds: per wave of CTAs a fixed part (launch, first loads, epilogue) plus the
// tensor-core time of its k blocks; slicing adds the kernel that sums the slices, which is bound by memory.
// The 128 x 128 tile, two CTAs to an SM, reads twice the operand bytes per flop, so it is the better one where the
// large tile would compute padding (any number of rows by up to 128 columns) or leave SMs idle, and a contraction is too
// short to slice; at equal fill it is 10 to 30 % slower.  Both tiles measured over 128 to 1,000,000 rows x 64 to 2048
// columns x 512 to 8192, in us, small and large: fp32 1000 x 512 x 512 19 and 32, 20,000 x 300 x 2048 106 and 151,
// 200,000 x 128 x 2048 370 and 517, 200,000 x 512 x 512 341 and 298, 50,000 x 2048 x 2048 1113 and 931; fp16
// 50,000 x 2048 x 512 214 and 171, 1000 x 1024 x 8192 83 and 48 (sliced).  Over those 284 products the choice is 0.3 % (mean)
// and 15 % (worst) slower than the better of the two; with one wave length for both tiles it was 3 % and 72 %.
// The chunked kernel's 128-column tile takes nearly as long per k block as the 256-column one -- with both operands from shared
// memory an MMA of 128 x 128 reads as many bytes a cycle as that gives -- but starts and ends 3 us sooner and makes twice the
// CTAs, so it is for products of one wave: inverse of 512 138 -> 134 us, 700 244 -> 226, 1024 301 -> 287, 2048 633 -> 589, 4096
// 1412 -> 1340; Gram of 1000 x 512 48.8 -> 46.8, 2000 x 256 60.0 -> 56.4, 400 x 400 42.4 -> 37.2.  Taken for three waves it cost
// 25 % (9000 x 3000 352 -> 440 us).
// The sizes alone decide, so that the workspace query, which names no device, agrees: every B200 has 148 SMs.  A product
// that leaves out the k blocks where a triangular factor is zero (KRange) is planned like a whole one.
GemmPlan plan_gemm(uint32_t npl, bool chunked, bool symmetric, int64_t M, int64_t N, uint32_t kblocks) {
    constexpr double SMS = B200_SMS, SUM_FIXED = 7.0, SUM_BYTES_PER_US = 3.0e6;
    constexpr uint32_t MAX_SPLITS = 64;
    constexpr size_t MAX_PARTIAL = 256u << 20;
    constexpr double MAX_GRID_Y = 65535.0;  // tile rows of a launch, 32-row blocks of the sum
    const double tm = (double)((M + 127) / 128), tn2 = (double)((N + 255) / 256), tm2 = (double)((M + 255) / 256);
    GemmPlan best{2, 1, kblocks, 0};
    double best_t = 1e300;
    if (!chunked && tm <= MAX_GRID_Y) {
        // rounds of two CTAs on every SM; what is left over after the last whole one has the SMs to itself, or nearly
        const double tn = (double)((N + 127) / 128), tiles = symmetric ? tm * (tm + 1) / 2 : tm * tn;
        const double rounds = (double)(uint64_t)(tiles / (2 * SMS)), rest = tiles - rounds * 2 * SMS;
        const double pair = npl == 2 ? 2.0 + 0.68 * kblocks : 4.0 + 0.26 * kblocks;
        const double single = 4.0 + (npl == 2 ? 0.5 : 0.18) * kblocks;
        best_t = rounds * pair + (rest > SMS ? pair : rest > 0 ? single : 0.0);
        best.tile = 1;
    }
    for (int tile = chunked ? 1 : 2; tile <= 2; ++tile) {
        const double tiles = tile == 1 ? (symmetric ? tm * (tm + 1) / 2 : tm * (double)((N + 127) / 128))
                             : chunked ? (symmetric ? tm2 * (tm2 + 1) : tm * tn2) : symmetric ? tm2 * (tm2 + 1) / 2 : tm2 * tn2;
        const double per_kb = tile == 1 ? 0.43 : chunked ? 0.48 : npl == 2 ? 0.9 : 0.3, fixed = tile == 1 ? 5.0 : 8.0;
        for (uint32_t s = 1; s <= MAX_SPLITS && s <= kblocks; ++s) {
            const uint32_t per = ((kblocks + s - 1) / s + 1u) & ~1u;  // whole 64-wide chunks
            const uint32_t used = (kblocks + per - 1) / per;
            const size_t bytes = used > 1 ? (size_t)used * M * N * sizeof(float) : 0;
            if (used != s || bytes > MAX_PARTIAL || (s > 1 && M > 32 * MAX_GRID_Y)) continue;
            const double waves = (double)(uint64_t)((tiles * s + SMS - 1) / SMS);
            double t = waves * (fixed + per * per_kb);
            if (s > 1) t += SUM_FIXED + ((double)s * (symmetric ? 0.5 : 1.0) + 1.0) * M * N * 4.0 / SUM_BYTES_PER_US;
            if (t < best_t) {
                best_t = t;
                best = GemmPlan{tile, s, s > 1 ? per : kblocks, align_up(bytes, 1024)};
            }
        }
    }
    return best;
}

template <int NPL, int T>
static int launch_gemm_nt(int device, const CUtensorMap& map_a, const CUtensorMap& map_b, GemmParams& p, uint32_t splits,
                          bool early, cudaStream_t stream) {
    constexpr uint32_t stage_bytes = 2u * T * NPL * GTILE_BYTES;
    const dim3 grid((p.N + 128u * T - 1) / (128u * T), (p.M + 128u * T - 1) / (128u * T), splits);
    // Two CTAs of the small tile share an SM.  Launched while the packing still runs they would do so on the first SMs that
    // become free, also where there is one for every SM and the others stay idle: such a grid takes all of the shared memory
    // (fp32 2000 x 1000 x 1024 29.9 -> 21.9 us, 128 x 8192 x 2048 65.8 -> 47.7, 10,000 x 100 x 2048 71.6 -> 52.4; fp16
    // 18,900 x 100 x 2048 61.9 -> 52.4).
    const bool pairs = T == 1 && !(early && (uint64_t)grid.x * grid.y <= (uint64_t)B200_SMS);
    p.stages = ((pairs ? 100u : 200u) * 1024u) / stage_bytes;
    if (p.stages > 8) p.stages = 8;
    const size_t smem = (size_t)p.stages * stage_bytes + 1024u;
    p.idesc = (p.idesc & 1u) ? idesc_f16(1u, 128u * T) : idesc_f16(0u, 128u * T);
    auto kern = gemm_nt_kernel<NPL, T>;
    if (const int e = set_smem_limit((const void*)kern, device)) return e;
    return launch_after(kern, grid, 384, smem, stream, early, map_a, map_b, p);
}

// C[M x N] (+)= alpha * row_scale[m] * Apacked . Bpacked^T
int launch_gemm(int device, cudaStream_t stream, const uint16_t* pa, const Packed& ga,
                const uint16_t* pb, const Packed& gb, int dtype, int64_t M, int64_t N, float* C,
                int64_t ldc, const float* row_scale, float alpha, int accumulate, int symmetric,
                int chunked, float* partial, KRange range, bool early) {
    CUtensorMap map_a, map_b;
    int rc = packed_tmap(&map_a, pa, ga, dtype);
    if (rc != TB_OK) return rc;
    rc = packed_tmap(&map_b, pb, gb, dtype);
    if (rc != TB_OK) return rc;
    if (ga.scaled != gb.scaled || (chunked && !ga.scaled)) return TB_ERR_BAD_ARG;
    const GemmPlan pl = plan_gemm(ga.npl, chunked != 0, symmetric != 0, M, N, ga.kblocks);
    GemmParams p;
    p.C = C;
    p.row_scale = row_scale;
    p.amax_a = ga.scaled ? packed_amax(pa, ga) : nullptr;
    p.amax_b = gb.scaled ? packed_amax(pb, gb) : nullptr;
    p.status = status_ptr(device);
    p.ldc = ldc;
    p.M = (uint32_t)M;
    p.N = (uint32_t)N;
    p.kblocks = ga.kblocks;
    p.kb_per_split = pl.kb_per_split;
    p.split_stride = (uint64_t)M * N;
    p.idesc = planes_are_fp16(ga, dtype) ? 0u : 1u;  // the element format; the shape is filled in below
    p.alpha = alpha;
    p.accumulate = accumulate;
    p.symmetric = symmetric;
    p.range = range;
    p.mirror = 1;
    const GemmParams whole = p;
    if (pl.splits > 1) {  // raw partial sums; the scales and the destination are the last kernel's
        p.C = partial;
        p.ldc = N;
        p.row_scale = nullptr;
        p.amax_a = p.amax_b = nullptr;
        p.alpha = 1.0f;
        p.accumulate = 0;
        p.mirror = 0;
    } else {
        p.split_stride = 0;
    }
    if (chunked) {
        const uint32_t cols = 128u * (uint32_t)pl.tile;
        p.idesc = idesc_f16(p.idesc, cols);
        auto kern = pl.tile == 2 ? gemm_nt_chunked_kernel<256> : gemm_nt_chunked_kernel<128>;
        const size_t smem = (pl.tile == 2 ? (size_t)Chunked<256>::SLOTS * Chunked<256>::SLOT_BYTES
                                          : (size_t)Chunked<128>::SLOTS * Chunked<128>::SLOT_BYTES) + 1024u;
        const dim3 grid((uint32_t)((N + cols - 1) / cols), (uint32_t)((M + 127) / 128), pl.splits);
        if (const int e = set_smem_limit((const void*)kern, device)) return e;
        rc = launch_after(kern, grid, 384, smem, stream, early, map_a, map_b, p);
        if (rc != TB_OK) return rc;
    } else if (pl.tile == 2) {
        rc = ga.npl == 2 ? launch_gemm_nt<2, 2>(device, map_a, map_b, p, pl.splits, early, stream)
                         : launch_gemm_nt<1, 2>(device, map_a, map_b, p, pl.splits, early, stream);
        if (rc != TB_OK) return rc;
    } else {
        rc = ga.npl == 2 ? launch_gemm_nt<2, 1>(device, map_a, map_b, p, 1, early, stream) : launch_gemm_nt<1, 1>(device, map_a, map_b, p, 1, early, stream);
        if (rc != TB_OK) return rc;
    }
    if (pl.splits > 1) {
        const dim3 grid((uint32_t)((N + 31) / 32), (uint32_t)((M + 31) / 32), 1);
        return launch_after(reduce_splits_kernel, grid, 256, 0, stream, early, partial, pl.splits, whole);
    }
    return TB_OK;
}

}  // namespace tb

extern "C" {

size_t tb_gemm_nt_workspace_bytes(int dtype, int64_t M, int64_t N, int64_t K) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    const tb::Packed a = tb::packed_geometry(dtype, M, K), b = tb::packed_geometry(dtype, N, K);
    return a.bytes + b.bytes + tb::plan_gemm(a.npl, false, false, M, N, a.kblocks).partial_bytes + 1024;
}

// The parts of tb_gemm_nt: A packed at the workspace's start, B packed behind it and the product.
static int gemm_nt_parts(int device, void* stream_, const void* A, int64_t lda, const void* B, int64_t ldb, int dtype,
                         int64_t M, int64_t N, int64_t K, float* C, int64_t ldc, const float* row_scale, float alpha,
                         int accumulate, void* ws, size_t ws_bytes, bool beside = false) {
    using namespace tb;
    if (dtype != TB_F16 && dtype != TB_BF16 && dtype != TB_F32) return TB_ERR_BAD_DTYPE;
    if (M <= 0 || N <= 0 || K <= 0 || lda < K || ldb < K || ldc < N || M > 0x7fffffff || N > 0x7fffffff)
        return TB_ERR_BAD_SHAPE;
    if (!A && !B) return TB_ERR_BAD_ARG;
    if (!ws || ((uintptr_t)ws & 255u) != 0 || ws_bytes < tb_gemm_nt_workspace_bytes(dtype, M, N, K))
        return TB_ERR_WORKSPACE;
    int sm_count = 0;
    int rc = select_device(device, &sm_count);
    if (rc != TB_OK) return rc;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    const Packed ga = packed_geometry(dtype, M, K), gb = packed_geometry(dtype, N, K);
    if ((uint64_t)ga.rowblocks * ga.kblocks * ga.npl * 128u > 0x7fffffffull ||
        (uint64_t)gb.rowblocks * gb.kblocks * gb.npl * 128u > 0x7fffffffull)
        return TB_ERR_UNSUPPORTED;
    uint16_t* pa = static_cast<uint16_t*>(ws);
    uint16_t* pb = reinterpret_cast<uint16_t*>(static_cast<uint8_t*>(ws) + ga.bytes);
    float* partial = reinterpret_cast<float*>(static_cast<uint8_t*>(ws) + ga.bytes + gb.bytes);
    if (A && B && dtype == TB_F32) {
        rc = launch_pack_rows(pack_rows_args(A, M, K, lda, pa, ga), pack_rows_args(B, N, K, ldb, pb, gb), sm_count, stream);
        if (rc != TB_OK) return rc;
    } else {
        if (A && (rc = launch_pack(A, dtype, false, M, K, lda, pa, ga, sm_count, stream, beside)) != TB_OK) return rc;
        if (B && (rc = launch_pack(B, dtype, false, N, K, ldb, pb, gb, sm_count, stream)) != TB_OK) return rc;
    }
    if (!B) return TB_OK;
    return launch_gemm(device, stream, pa, ga, pb, gb, dtype, M, N, C, ldc, row_scale, alpha, accumulate, 0, 0, partial);
}

int tb_gemm_nt(int device, void* stream, const void* A, int64_t lda, const void* B, int64_t ldb, int dtype, int64_t M,
               int64_t N, int64_t K, float* C, int64_t ldc, const float* row_scale, float alpha, int accumulate, void* ws,
               size_t ws_bytes) {
    const bool all = A && B && C;  // none of them: a bad type or shape is still reported before a missing matrix
    return gemm_nt_parts(device, stream, all ? A : nullptr, lda, all ? B : nullptr, ldb, dtype, M, N, K, C, ldc, row_scale,
                         alpha, accumulate, ws, ws_bytes);
}

int tb_gemm_nt_pack(int device, void* stream, const void* A, int64_t lda, int dtype, int64_t M, int64_t N, int64_t K,
                    void* ws, size_t ws_bytes) {
    return gemm_nt_parts(device, stream, A, lda, nullptr, K, dtype, M, N, K, nullptr, N, nullptr, 1.0f, 0, ws, ws_bytes);
}

int tb_gemm_nt_pack_beside(int device, void* stream, const void* A, int64_t lda, int dtype, int64_t M, int64_t N, int64_t K,
                           void* ws, size_t ws_bytes) {
    return gemm_nt_parts(device, stream, A, lda, nullptr, K, dtype, M, N, K, nullptr, N, nullptr, 1.0f, 0, ws, ws_bytes, true);
}

int tb_gemm_nt_packed(int device, void* stream, const void* B, int64_t ldb, int dtype, int64_t M, int64_t N, int64_t K,
                      float* C, int64_t ldc, const float* row_scale, float alpha, int accumulate, void* ws, size_t ws_bytes) {
    return gemm_nt_parts(device, stream, nullptr, K, C ? B : nullptr, ldb, dtype, M, N, K, C, ldc, row_scale, alpha,
                         accumulate, ws, ws_bytes);
}

size_t tb_gram_workspace_bytes(int dtype, int64_t n, int64_t k) {
    if (n <= 0 || k <= 0) return 0;
    const tb::Packed g = tb::packed_geometry(dtype, k, n);
    return g.bytes + tb::plan_gemm(g.npl, dtype == TB_F32, true, k, k, g.kblocks).partial_bytes + 1024;
}

int tb_gram(int device, void* stream_, const void* X, int dtype, int64_t n, int64_t k, int64_t ld, float* G,
            int64_t ldg, int accumulate, void* ws, size_t ws_bytes) {
    using namespace tb;
    if (dtype != TB_F16 && dtype != TB_BF16 && dtype != TB_F32) return TB_ERR_BAD_DTYPE;
    if (n <= 0 || k <= 0 || ld < k || ldg < k || k > 0x7fffffff) return TB_ERR_BAD_SHAPE;
    if (!X || !G) return TB_ERR_BAD_ARG;
    if (!ws || ((uintptr_t)ws & 255u) != 0 || ws_bytes < tb_gram_workspace_bytes(dtype, n, k))
        return TB_ERR_WORKSPACE;
    int sm_count = 0;
    int rc = select_device(device, &sm_count);
    if (rc != TB_OK) return rc;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    // the operand is X^T: k operand rows, contraction over the n rows of X
    const Packed g = packed_geometry(dtype, k, n);
    if ((uint64_t)g.rowblocks * g.kblocks * g.npl * 128u > 0x7fffffffull) return TB_ERR_UNSUPPORTED;
    uint16_t* px = static_cast<uint16_t*>(ws);
    rc = launch_pack(X, dtype, true, k, n, ld, px, g, sm_count, stream);
    if (rc != TB_OK) return rc;
    // the Gram feeds an inverse, which amplifies its error by the condition number: chunked accumulation
    return launch_gemm(device, stream, px, g, px, g, dtype, k, k, G, ldg, nullptr, 1.0f, accumulate, 1,
                       dtype == TB_F32 ? 1 : 0, reinterpret_cast<float*>(static_cast<uint8_t*>(ws) + g.bytes));
}

}  // extern "C"
