// Rademacher projection of small batches on the integer tensor cores.
//
// A small batch costs what its matrix costs to generate, and with a 16-bit operand most of that is not
// XORWOW (7 instructions a draw) but turning 16 signs into 8 words of +-1.  Here the operand is made of bytes and the
// draw's own bits are its values: one AND with 0x01010101 << i leaves four matrix entries as 0 or 2^i, and
//     sum_f (+-1) q_f  =  2 sum_{f: bit set} q_f  -  sum_f q_f
// makes a sign projection of it.  The gradients are integers too: a row is scaled by the power of two that brings its
// largest magnitude below 2^28, rounded to q, and kept as four planes of signed base-256 digits, of which `kind::i8` adds up
// every product exactly in 32 bits.  sum_f q_f comes from the staging.  Only the result of a CTA is rounded, once, to fp32.
//
//   * Exactness.  An fp16 (bf16) value has 11 (8) significant bits, so q is exact for every element within 2^-17 (2^-20) of
//     its row's largest.  Below that an element is off by at most half a step, 2^-28 of the largest: nothing on a row of like
//     elements, ten times the error of the 16-bit kernel on one that a single element outweighs.  So the steps of a row are never
//     coarser than its norm allows (row_exponent): rounding takes at most 2^-24 of its largest element and 2^-22 of the norm of
//     the others.  The few elements that such steps put out of the planes' range are staged as zeros and listed by tile, and the
//     CTAs that find one run the tile's streams once more (7 of the 17 instructions) and add them in 64 bits.
//     Error against 64 bits over the row's norm, 16-bit kernel / steps by the largest element alone / this: 592,003 features
//     beside one of 1 in bf16, N(0, 2^-8) 2.9e-7 / 7.6e-8 / 7.6e-8, N(0, 2^-16) 1.7e-5 / 4.4e-7 / 1.2e-7, uniform in 2^-30..2^-29
//     1.7e-7 / 1.5e-6 / 1.3e-7, all of 2^-28 3.6e-7 / 3.8e-6 / 1.1e-7; 6,000,001 features, N(0, 2^-16) 9.0e-5 / 1.2e-6 / 8.6e-8,
//     uniform 3.2e-7 / 3.9e-6 / 9.4e-8; N(0, 1) without the one 3.2e-6 / 7.4e-8 / 7.4e-8.
//     us a call, the same three, one such element to a row: 16 x 1,000,003 bf16 -> 4096 371 / 238 / 241, 32 rows 400 / 351 / 365,
//     17 x 330,003 -> 1536 79 / 64 / 72; without any, 16 x 2,796,202 fp16 -> 4096 1014 / 617 / 616, 32 x 2,796,202 1168 / 957 / 956,
//     16 x 40,001 -> 8192 58 / 49 / 48, 32 x 1,048,576 fp32 -> 2048 240 / 236 / 231.
//   * 2^i differs from word to word (bit 2j + h of a draw's byte: feature pair j, column parity h; two of the four j after
//     a shift by four).  The column's factor 2^h is undone at the end, the features' 2^(2 (j & 1)) in the staging: even j are
//     staged four times as large.
//   * What bounds it.  Up to 16 rows the integer pipe, 82 % busy with 11 instructions per 16 x 32 entries (4 of the 7 of a draw,
//     5 to spread it, 2 of hand-shakes; 35 instructions in all with a 16-bit operand, now 17): without its MMAs the kernel takes
//     95 % of its time.  us a call, 16-bit operand -> this: 2,796,202 fp16 features -> 4096 1014 -> 616, 1,000,003 -> 8192
//     726 -> 425, 10,000,001 bf16 -> 8192 6970 -> 3989; one row of 1,000,003 -> 2048 196 -> 116.
//     From 17 to 32 rows the accumulators leave room for one CTA per SM, of four groups, and the MMAs bound it (tensor pipe
//     75 % busy at 24 rows, 85 at 32, with 7 TB/s from the L2; without generating it takes as long): 17 rows x 1,000,003 bf16
//     -> 8192 757 -> 537, 24 rows fp16 -> 2048 213 -> 175, 32 rows x 2,796,202 -> 4096 1168 -> 956.
//   * The groups' slots change hands together, and so do their boxes: one warp issues the MMAs beside busy generators, and a
//     hand-over costs it some 300 cycles whatever it covers.  With barriers of each group's own 16 rows took 2 % longer (659
//     us for 647), and four groups of 32-feature slots to a CTA 1023 us; with common ones 693, so two of 64 they stay.
//     Measured and dropped: one slot a group (773 against 692 us), the next slots' barriers polled between MMAs (789), shifts
//     as multiplications (no change; by the upper half of a product 3 % slower), the hand-over of a slot behind the next one's
//     first chunk (no change), a loop over pairs of slots with fixed addresses (no change).
//   * A row with an infinity or a NaN (seen by absmax_kernel) is staged as the signs of its infinities; the CTA compares
//     their signed sum with their number and writes what the sum of the row would be, +-inf or NaN.
//
// Included by project.cu after the generator definitions.
#pragma once

namespace tb {

constexpr uint32_t BITS_K = 64;               // features per operand slot (a stage)
constexpr uint32_t BITS_BOX_K = 128;          // features per box of the staged gradients (128 bytes a row)
constexpr uint32_t BITS_PLANES = 4;           // base-256 digits of a staged gradient
constexpr uint32_t BITS_MAX_ROWS = 32;        // rows per launch
constexpr uint32_t BITS_MAX_CHAIN = 32768;    // stages of a CTA: |digit| <= 128, A <= 8, so 2^31 / 1024 features
// The two shapes: up to 16 rows two groups to a CTA and two CTAs to an SM, up to 32 rows four groups and one; and the stages of
// gradients that arrive and are released together, of which a group has room for two.
__host__ __device__ constexpr uint32_t bits_groups(uint32_t rows) { return rows <= 16u ? 2u : 4u; }
__host__ __device__ constexpr uint32_t bits_batch(uint32_t rows) { return rows <= 16u ? 4u : 2u; }
constexpr uint32_t BITS_MAX_SLICES = 256;     // of a row in absmax_kernel
constexpr uint32_t BITS_RUNS = 4;             // runs of 512 features that a warp of stage_bits_kernel takes at most
constexpr float BITS_RANGE = 268435456.0f;     // 2^28: a rounded gradient stays below
constexpr int BITS_INF = 0x7ffffffe, BITS_NAN = 0x7fffffff;   // BitsParams::row_exp of a row that holds one

// An element that is too large for the planes, in the list of its place in a tile (which of 16 features): 2^e times it.
struct __align__(16) Outlier {
    uint32_t next;              // 1 + the index of the next of the list, 0: the last
    uint32_t row, feature;      // of the 16
    float q;
};

struct BitsParams {
    float* partials;            // [bundles][B][N]
    uint32_t* status;
    const long long* sums;      // [tiles][rows] sum of the rounded gradients q
    const uint32_t* infs;       // [tiles][rows] infinities among them (rows of BITS_INF only)
    const int* row_exp;         // [rows] 4 q is 2^row_exp times the gradient; or BITS_INF, BITS_NAN
    const uint32_t* last_out;   // [tiles] 1 + the last 16 features that have outliers, 0: none
    const uint32_t* heads;      // [tiles][4 nst] 1 + the first of them, 0: none
    const Outlier* outliers;
    uint32_t N, seed;
    uint32_t B, rows;           // rows in this launch, and rounded up to 8
    uint32_t nst;               // pipeline stages per feature tile, even
    uint32_t tiles, tiles_per_bundle;
    uint32_t idesc;
};

// The two streams' signs of 16 features: bit 2j + h of byte b is feature 2j + (b & 1) + 8 (b >> 1) of the 16, column h of the pair.
__device__ __forceinline__ uint32_t gen_bits(Xw& st0, Xw& st1) {
    const uint32_t d0 = xw_next(st0), d1 = xw_next(st1);
    return __byte_perm(d0, d1, 0x5140u);
}
// 16 features of a pair of columns: byte b of word j is feature 2j + (b & 1) + 8 (b >> 1) of the 16, as the staging has them.
__device__ __forceinline__ void gen_bits_pair(Xw& st0, Xw& st1, uint32_t* even, uint32_t* odd) {
    const uint32_t c = gen_bits(st0, st1), c4 = c >> 4;
    even[0] = c & 0x01010101u;
    odd[0] = c & 0x02020202u;
    even[1] = c & 0x04040404u;
    odd[1] = c & 0x08080808u;
    even[2] = c4 & 0x01010101u;
    odd[2] = c4 & 0x02020202u;
    even[3] = c4 & 0x04040404u;
    odd[3] = c4 & 0x08080808u;
}

// v 2^-e for any e: in two steps, each a power of two that fp32 has
__device__ __forceinline__ float scale_by(float v, int e) {
    const int a = e / 2, b = e - a;
    return v * __int_as_float((127 + a) << 23) * __int_as_float((127 + b) << 23);
}

// Signed sums of the elements that the planes do not hold, of the tiles `tile`, `tile` + `step`, ... before `end`: those are
// generated once more, up to the last such element.  `seed` is that of the thread's first stream in tile 0, `sums` its pair of
// columns of row 0.  Not expanded where it is called, and without a pointer to the parameters: the loops in front of it keep
// their registers.
__device__ __noinline__ void add_outliers(const uint32_t* last_out, const uint32_t* heads, const Outlier* outliers, uint32_t nst,
                                          long long* sums, uint32_t seed, uint32_t tile, uint32_t end, uint32_t step) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t t = tile; t < end; t += step) {
        const uint32_t last = last_out[t];
        if (last == 0u) continue;
        Xw st0, st1;
        xw_seed(st0, seed + 359124577u * t);
        xw_seed(st1, seed + 658105236u * 16u + 359124577u * t);
        for (uint32_t k0 = 0; k0 < last; k0 += 32u) {
            const uint32_t k1 = min(32u, last - k0);
            const uint32_t first = lane < k1 ? heads[(size_t)t * nst * 4u + k0 + lane] : 0u;
            for (uint32_t k = 0; k < k1; ++k) {
                const uint32_t c = gen_bits(st0, st1);
                for (uint32_t r = __shfl_sync(0xffffffffu, first, k); r != 0u;) {
                    const Outlier o = outliers[r - 1u];
                    const long long q = (long long)o.q;
                    const uint32_t at = 8u * ((o.feature & 1u) | (o.feature >> 3 << 1)) + 2u * ((o.feature & 7u) >> 1);
                    unsigned long long* const sum = reinterpret_cast<unsigned long long*>(sums + o.row * 256u);
                    atomicAdd(sum, (unsigned long long)(c >> at & 1u ? q : -q));
                    atomicAdd(sum + 1, (unsigned long long)(c >> at & 2u ? q : -q));
                    r = o.next;
                }
            }
        }
    }
}

// One CTA: 256 output columns (two accumulators) x up to ROWS rows x a bundle of feature tiles.  Roles and rings are those of
// project_kernel with two accumulators; what differs is the operand, the digit planes beside one another in the N dimension
// (rows x 4), the common hand-shakes, and that the accumulators are read once, at the end.
template <uint32_t ROWS>
__global__ void __launch_bounds__((4 * bits_groups(ROWS) + 2) * 32, ROWS <= 16 ? 2 : 1)
project_bits_kernel(const __grid_constant__ CUtensorMap tmap, const BitsParams p) {
    constexpr int NG = bits_groups(ROWS);
    constexpr uint32_t BATCH = bits_batch(ROWS);
    constexpr uint32_t GW = 4u, TMEM_COLS = ROWS <= 16u ? 256u : 512u, SA = 2u;
    constexpr uint32_t A_COL0 = 2u * BITS_PLANES * ROWS;            // accumulators, then the generated-operand ring
    constexpr uint32_t SLOT = 2u * BITS_K / 4u;                     // tensor-memory columns of a slot
    static_assert(A_COL0 + NG * SA * SLOT <= TMEM_COLS, "too many generator groups for the TMEM ring");
    extern __shared__ uint8_t smem_raw[];
    // a slot of every group, and the boxes of every group, are handed over together
    __shared__ alignas(16) uint64_t bar_full_a[SA];
    __shared__ alignas(16) uint64_t bar_empty_a[SA];
    __shared__ uint64_t bar_full_b[2];
    __shared__ uint64_t bar_empty_b[2];
    __shared__ uint64_t bar_acc;
    __shared__ uint64_t bar_extra[2];  // between the generators
    __shared__ uint32_t tmem_slot;
    __shared__ uint32_t abort_word;
    volatile uint32_t* abort_flag = &abort_word;

    cudaTriggerProgrammaticLaunchCompletion();
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t brows = BITS_PLANES * p.rows;   // N of the MMAs
    const uint32_t box_bytes = brows * BITS_BOX_K;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t tile0 = blockIdx.y * p.tiles_per_bundle;
    const uint32_t ntile = min(p.tiles_per_bundle, p.tiles - tile0);

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < 2u; ++s) {
            mbar_init(smem_u32(&bar_full_a[s]), GW * NG);
            mbar_init(smem_u32(&bar_empty_a[s]), 1);
            mbar_init(smem_u32(&bar_full_b[s]), 1);
            mbar_init(smem_u32(&bar_empty_b[s]), 1);
        }
        mbar_init(smem_u32(&bar_acc), 1);
        for (uint32_t s = 0; s < 2u; ++s) mbar_init(smem_u32(&bar_extra[s]), GW * NG);
        abort_word = 0;
        fence_mbar_init();
    }
    if (warp == GW * NG + 1) {
        tmem_alloc(smem_u32(&tmem_slot), TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;

    if (warp < GW * NG) {
        // ------------------------- generators, then epilogue -------------------------
        const uint32_t g = warp / GW, q = warp & 3u;
        const uint32_t pair = q * 32u + lane;
        const uint32_t stream_col = blockIdx.x * 256u + 2u * (pair & ~15u) + (pair & 15u);
        const uint32_t lane_base = (q * 32u) << 16;
        const uint32_t a_base = tmem_base + lane_base + A_COL0 + g * (SA * SLOT);
        const uint32_t full = smem_u32(&bar_full_a[0]), empty = smem_u32(&bar_empty_a[0]);
        bool ok = true;
        uint32_t n = 0;  // slots this group has filled
        for (uint32_t ti = g; ti < ntile && ok; ti += NG) {
            Xw st0, st1;
            xw_seed(st0, p.seed + 658105236u * stream_col + 359124577u * (tile0 + ti));
            xw_seed(st1, p.seed + 658105236u * (stream_col + 16u) + 359124577u * (tile0 + ti));
#pragma unroll 2
            for (uint32_t s = 0; s < p.nst; ++s, ++n) {
                const uint32_t slot = n & 1u, parity = (~n >> 1) & 1u;
                // asked for before the generation and looked at behind it: the answer takes its time
                const bool free = mbar_test_wait(empty + slot * 8u, parity);
                uint32_t even[16], odd[16];
#pragma unroll
                for (int c = 0; c < 4; ++c) gen_bits_pair(st0, st1, even + 4 * c, odd + 4 * c);
                if (!__all_sync(0xffffffffu, free) && !mbar_wait_warp(empty + slot * 8u, parity, abort_flag)) {
                    if (lane == 0) fail(p.status, abort_flag, ST_TIMEOUT_EMPTY, (g << 16) | s);
                    ok = false;
                    break;
                }
                tc_fence_after();
                tmem_st_x16(a_base + slot * SLOT, even);
                tmem_st_x16(a_base + slot * SLOT + SLOT / 2u, odd);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(full + slot * 8u);
            }
        }
        // the rounds that the first groups still walk a tile in: the slots change hands without this one
        for (const uint32_t all = ((ntile + NG - 1u) / NG) * p.nst; ok && n < all; ++n) {
            const uint32_t slot = n & 1u;
            ok = mbar_wait_warp(empty + slot * 8u, (~n >> 1) & 1u, abort_flag);
            if (!ok && lane == 0) fail(p.status, abort_flag, ST_TIMEOUT_EMPTY, 0x4000u | (g << 16));
            if (ok && lane == 0) mbar_arrive(full + slot * 8u);
        }
        bool outside = false;  // some tile has elements that the planes do not hold; the same for every warp
        if (ok) {
            cudaGridDependencySynchronize();  // the staging's lists, sums and scales
            for (uint32_t t = lane; t < ntile; t += 32u) outside |= p.last_out[tile0 + t] != 0u;
            outside = __any_sync(0xffffffffu, outside);
        }
        // ---- the exact integer result of this CTA, as fp32 ----
        if (ok && !mbar_wait_warp(smem_u32(&bar_acc), 0u, abort_flag)) {
            if (lane == 0) fail(p.status, abort_flag, ST_TIMEOUT_ACC, g);
            ok = false;
        }
        if (ok) {
            tc_fence_after();
            const uint32_t tmem_acc = tmem_base + lane_base;
            const uint32_t n_out = blockIdx.x * 256u + 2u * pair;
            // What the planes do not hold: those tiles are generated once more, up to the last such element, and the signed
            // sums kept in the boxes' place
            long long(*const extra)[256] = reinterpret_cast<long long(*)[256]>(smem_raw + (smem_base - smem_u32(smem_raw)));
            if (outside) {
                auto meet = [&](int which) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&bar_extra[which]));
                    if (ok && !mbar_wait_warp(smem_u32(&bar_extra[which]), 0u, abort_flag)) {
                        if (lane == 0) fail(p.status, abort_flag, ST_TIMEOUT_ACC, 0x4000u | g);
                        ok = false;
                    }
                };
                for (uint32_t i = threadIdx.x; i < p.rows * 256u; i += GW * NG * 32u) extra[0][i] = 0;
                meet(0);
                if (ok)
                    add_outliers(p.last_out, p.heads, p.outliers, p.nst, extra[0] + 2u * pair, p.seed + 658105236u * stream_col, tile0 + g,
                                 tile0 + ntile, NG);
                meet(1);
            }
            float* dst = p.partials + (size_t)blockIdx.y * p.B * p.N + n_out;
            // twice: with these additions in it the one loop takes 0.3 us longer (16 x 40,001 -> 8192, where eight CTAs follow
            // one another, 53.3 -> 51.3 us)
            auto finish = [&](auto more) {
                for (uint32_t b4 = 4u * g; b4 < p.B && ok; b4 += 4u * NG) {
                    // sums of four rows over the bundle's tiles: eight tiles at a time, row `lane & 3`.  (Fetched before the last
                    // products are there 17 rows x 70,001 -> 8192 take 77 us for 80, but 32 x 11,173,962 -> 4096 3820 for 3740:
                    // the generators' loop is allotted other registers.)
                    const uint32_t row = b4 + (lane & 3u);
                    long long sum = 0;
                    uint32_t ninf = 0;
                    const int exps = p.row_exp[row];
                    for (uint32_t t = lane >> 2; t < ntile; t += 8u) {
                        sum += p.sums[(tile0 + t) * p.rows + row];
                        ninf += p.infs[(tile0 + t) * p.rows + row];
                    }
#pragma unroll
                    for (int o = 4; o < 32; o <<= 1) {
                        sum += __shfl_xor_sync(0xffffffffu, sum, o);
                        ninf += __shfl_xor_sync(0xffffffffu, ninf, o);
                    }
                    uint32_t d[2][BITS_PLANES][4];
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int pl = 0; pl < (int)BITS_PLANES; ++pl)
                            tmem_ld_x4(tmem_acc + h * brows + pl * p.rows + b4, d[h][pl]);
                    tmem_wait_ld();
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) {
                        const uint32_t b = b4 + j;
                        const long long total = __shfl_sync(0xffffffffu, sum, j);
                        const uint32_t infs = __shfl_sync(0xffffffffu, ninf, j);
                        const int e = __shfl_sync(0xffffffffu, exps, j);
                        if (b >= p.B) break;
                        float2 v;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            long long s = 0;  // 4 2^h times the sum of q over the set bits
#pragma unroll
                            for (int pl = (int)BITS_PLANES - 1; pl >= 0; --pl) s = s * 256 + (int)d[h][pl][j];
                            s = (h == 0 ? 2 * s : s) - 4 * total;
                            if constexpr (decltype(more)::value) s += 4 * extra[b][2u * pair + h];
                            float r;
                            if (e < BITS_INF)
                                r = scale_by(__ll2float_rn(s), -e);
                            else if (e == BITS_INF)
                                r = infs == 0u ? 0.0f : s == (long long)infs * 4 ? INFINITY : s == -(long long)infs * 4 ? -INFINITY : NAN;
                            else
                                r = NAN;
                            (h == 0 ? v.x : v.y) = r;
                        }
                        __stcg(reinterpret_cast<float2*>(dst + (size_t)b * p.N), v);
                    }
                }
            };
            if (outside)
                finish(std::true_type{});
            else
                finish(std::false_type{});
        }
    } else {
        // stages of every group (cnt[] does not increase with g)
        uint32_t cnt[NG];
#pragma unroll
        for (int g = 0; g < NG; ++g) cnt[g] = ntile > (uint32_t)g ? ((ntile - g + NG - 1) / NG) * p.nst : 0u;
        const uint32_t maxcnt = cnt[0];
        if (warp == GW * NG) {
            // ------------------------------ TMA producer (one lane) ------------------------------
            if (lane == 0) {
                prefetch_tmap(&tmap);
                cudaGridDependencySynchronize();  // the staged gradients; the generators need nothing and have begun
                bool ok = true;
                const uint32_t boxes = p.nst / 2u;   // per tile
                uint32_t tile[NG], s[NG];
#pragma unroll
                for (int g = 0; g < NG; ++g) {
                    tile[g] = tile0 + g;
                    s[g] = 0;
                }
                for (uint32_t it = 0, n = 0; it < maxcnt && ok; it += BATCH, ++n) {
                    const uint32_t slot = n & 1u, parity = (~n >> 1) & 1u;
                    if (!mbar_wait(smem_u32(&bar_empty_b[slot]), parity, abort_flag)) {
                        fail(p.status, abort_flag, ST_TIMEOUT_EMPTY, 0x8000u | it);
                        ok = false;
                        break;
                    }
                    uint32_t loads = 0;
#pragma unroll
                    for (int g = 0; g < NG; ++g) loads += it < cnt[g] ? min(BATCH, cnt[g] - it) / 2u : 0u;
                    const uint32_t bar = smem_u32(&bar_full_b[slot]);
                    mbar_expect_tx(bar, loads * box_bytes);
#pragma unroll
                    for (int g = 0; g < NG; ++g) {
                        for (uint32_t j = 0; j < BATCH / 2u && it + 2u * j < cnt[g]; ++j) {
                            tma_load_2d(smem_base + ((g * 2u + slot) * (BATCH / 2u) + j) * box_bytes, &tmap, 0,
                                        (int)((tile[g] * boxes + s[g]) * brows), bar);
                            if (++s[g] == boxes) {
                                s[g] = 0;
                                tile[g] += NG;
                            }
                        }
                    }
                }
            }
        } else {
            // ------------------------------- MMA issuer -------------------------------
            // Whole warp in the loop, one elected lane issues (operands stay in uniform registers).  The warp shares its
            // scheduler with busy generators, so what counts is its instructions a slot: rings and parities are unrolled.
            const bool leader = elect_one();
            bool ok = true;
            uint32_t started = 0;
            for (uint32_t it = 0, n = 0; it < maxcnt && ok; it += BATCH, ++n) {
                const uint32_t bslot = n & 1u, bparity = (n >> 1) & 1u;
                if (!mbar_wait_warp(smem_u32(&bar_full_b[bslot]), bparity, abort_flag)) {
                    if (leader) fail(p.status, abort_flag, ST_TIMEOUT_FULL_B, it);
                    ok = false;
                    break;
                }
#pragma unroll
                for (uint32_t j = 0; j < BATCH; ++j) {
                    if (it + j >= maxcnt || !ok) continue;
                    if (!mbar_wait_warp(smem_u32(&bar_full_a[j & 1u]), ((it + j) >> 1) & 1u, abort_flag)) {
                        if (leader) fail(p.status, abort_flag, ST_TIMEOUT_FULL_A, it);
                        ok = false;
                        continue;
                    }
                    tc_fence_after();
                    if (leader) {
#pragma unroll
                        for (int g = 0; g < NG; ++g) {
                            if (it + j >= cnt[g]) continue;
                            const uint32_t a_addr = tmem_base + A_COL0 + (g * SA + (j & 1u)) * SLOT;
                            const uint64_t b_desc =
                                smem_desc_k_sw128(smem_base + ((g * 2u + bslot) * (BATCH / 2u) + j / 2u) * box_bytes) + 4u * (j & 1u);
                            const uint32_t acc = started | (uint32_t)(g > 0);
                            umma_i8_ts(tmem_base, a_addr, b_desc, p.idesc, acc);
                            umma_i8_ts(tmem_base + brows, a_addr + SLOT / 2u, b_desc, p.idesc, acc);
                            // 32 features further: 8 TMEM columns, 32 bytes inside the swizzle row
                            umma_i8_ts(tmem_base, a_addr + 8u, b_desc + 2u, p.idesc, 1u);
                            umma_i8_ts(tmem_base + brows, a_addr + SLOT / 2u + 8u, b_desc + 2u, p.idesc, 1u);
                        }
                        tc_commit(smem_u32(&bar_empty_a[j & 1u]));
                        if (j + 1 == BATCH) tc_commit(smem_u32(&bar_empty_b[bslot]));
                    }
                    started = 1u;
                }
            }
            if (ok && leader) tc_commit(smem_u32(&bar_acc));
        }
    }

    // ---------------------------------- teardown ----------------------------------
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) __nanosleep(200000);  // let copies and MMAs already in flight land
    if (warp == GW * NG + 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// ---- staging of the integer gradients ------------------------------------------------------------------------------
enum class Elem { F32, F16, BF16 };
template <Elem E>
using elem_t = typename std::conditional<E == Elem::F32, float, uint16_t>::type;

// Largest magnitude and sum of squares of a slice of row blockIdx.x.  The former as the bits of the element type
// (monotonic, infinity above every number and NaN above infinity); of the latter three for bf16, whose squares fp32 does not
// hold: of the elements, and of 2^-90 and 2^90 times them.  Also clears what the staging adds to.  The ends of a parameter go
// element by element.  Bound by memory: 16 x 2,796,202 fp16 (89 MB) in 20 us.
template <Elem E>
struct RowStats {
    static constexpr uint32_t SUMS = E == Elem::BF16 ? 3u : 1u;
    uint32_t max_bits;
    float sums[SUMS];
    __device__ __forceinline__ void square(float x) {
        sums[0] = fmaf(x, x, sums[0]);
        if constexpr (SUMS == 3u) {
            const float low = x * 0x1p-90f, high = x * 0x1p90f;
            sums[1] = fmaf(low, low, sums[1]);
            sums[2] = fmaf(high, high, sums[2]);
        }
    }
    __device__ __forceinline__ void add_one(uint32_t bits) {
        max_bits = E == Elem::F32 ? max(max_bits, bits & 0x7fffffffu) : __vmaxu2(max_bits, bits & 0x7fffu);
        square(E == Elem::F32 ? __uint_as_float(bits) : E == Elem::F16 ? __half2float(__ushort_as_half((unsigned short)bits))
                                                                       : __uint_as_float(bits << 16));
    }
    __device__ __forceinline__ void add(uint32_t w) {  // 32 bits of elements
        if constexpr (E == Elem::F32) {
            add_one(w);
        } else {
            max_bits = __vmaxu2(max_bits, w & 0x7fff7fffu);
            if constexpr (E == Elem::F16) {
                const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w));
                square(v.x);
                square(v.y);
            } else {
                square(__uint_as_float(w << 16));
                square(__uint_as_float(w & 0xffff0000u));
            }
        }
    }
    __device__ __forceinline__ void add(const uint4& v) {
        add(v.x);
        add(v.y);
        add(v.z);
        add(v.w);
    }
};
template <Elem E>
__device__ __forceinline__ void add_run(RowStats<E>& st, const elem_t<E>* src, uint64_t n) {
    constexpr uint32_t V = 16u / sizeof(elem_t<E>);
    auto one = [&](uint64_t i) {
        st.add_one(E == Elem::F32 ? reinterpret_cast<const uint32_t*>(src)[i] : reinterpret_cast<const uint16_t*>(src)[i]);
    };
    const uint64_t head = min(n, (uint64_t)(((16u - (uint32_t)(reinterpret_cast<uintptr_t>(src) & 15u)) & 15u) / sizeof(elem_t<E>)));
    const uint64_t vecs = (n - head) / V, tail = head + vecs * V;
    if (threadIdx.x < head) one(threadIdx.x);
    const uint4* vec = reinterpret_cast<const uint4*>(src + head);
    uint64_t i = threadIdx.x;
    for (; i + 3u * 256u < vecs; i += 4u * 256u) {
        uint4 v[4];
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) v[j] = __ldg(vec + i + j * 256u);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) st.add(v[j]);
    }
    for (; i < vecs; i += 256u) st.add(__ldg(vec + i));
    if (tail + threadIdx.x < n) one(tail + threadIdx.x);
}

template <Elem E, bool SEG>
__global__ void __launch_bounds__(256)
absmax_kernel(const elem_t<E>* __restrict__ g, const SegDev* __restrict__ segs, uint32_t nsegs, uint64_t row0,
              uint32_t* __restrict__ maxima, float* __restrict__ squares, uint4* __restrict__ clear, uint32_t clear_n, uint64_t F,
              uint64_t ld, uint64_t slice) {
    after_earlier_launch();
    constexpr uint32_t SUMS = RowStats<E>::SUMS;
    __shared__ RowStats<E> part[8];
    const uint32_t row = blockIdx.x, part_of_row = gridDim.y - 1u - blockIdx.y;
    const uint32_t id = (blockIdx.y * gridDim.x + blockIdx.x) * 256u + threadIdx.x;
    for (uint32_t i = id; i < clear_n; i += gridDim.x * gridDim.y * 256u) clear[i] = make_uint4(0u, 0u, 0u, 0u);
    const uint64_t f0 = part_of_row * slice, f1 = min(F, f0 + slice);
    RowStats<E> st = {};
    if (SEG) {
        uint32_t lo = 0, hi = nsegs;  // last parameter whose start is <= f0
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (segs[mid].start <= f0)
                lo = mid;
            else
                hi = mid;
        }
        for (uint64_t f = f0; f < f1; ++lo) {
            const SegDev s = segs[lo];
            const uint64_t end = min(f1, s.start + s.numel);
            add_run(st, static_cast<const elem_t<E>*>(s.ptr) + (row0 + row) * s.stride + (f - s.start), end - f);
            f = end;
        }
    } else {
        add_run(st, g + (uint64_t)row * ld + f0, f1 - f0);
    }
    if (E != Elem::F32) st.max_bits = max(st.max_bits & 0xffffu, st.max_bits >> 16);
    st.max_bits = __reduce_max_sync(0xffffffffu, st.max_bits);
#pragma unroll
    for (uint32_t j = 0; j < SUMS; ++j)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) st.sums[j] += __shfl_xor_sync(0xffffffffu, st.sums[j], o);
    if ((threadIdx.x & 31u) == 0) part[threadIdx.x >> 5] = st;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 1; w < 8; ++w) {
            st.max_bits = max(st.max_bits, part[w].max_bits);
#pragma unroll
            for (uint32_t j = 0; j < SUMS; ++j) st.sums[j] += part[w].sums[j];
        }
        const uint32_t at = row * gridDim.y + part_of_row;
        maxima[at] = st.max_bits;
#pragma unroll
        for (uint32_t j = 0; j < SUMS; ++j) squares[at * SUMS + j] = st.sums[j];
    }
}

// The value the projection takes an element for: fp32 is rounded to fp16 as in stage_kernel.
template <Elem E>
__device__ __forceinline__ float staged_value(uint32_t bits) {
    if (E == Elem::F32) return __half2float(__float2half_rn(__uint_as_float(bits)));
    if (E == Elem::F16) return __half2float(__ushort_as_half((unsigned short)bits));
    return __uint_as_float(bits << 16);
}

// Scale of a row: the exponent e for which 2^e times every element is below 2^28, or what to do with a row that is not
// finite.  Where that leaves steps so coarse that rounding could take more from the row than 2^-24 of its largest element and
// 2^-22 of the norm of the rest, the exponent is the least that does not, and the elements that 2^e takes out of range go
// beside the planes (`outside`): F / 4096 + 1 of them at most, since more would make that norm, and with it the steps, larger.
// A number that comes as fp16 is a multiple of 2^-24: finer steps than that are never needed.  The last bits of the sums depend on
// how a row is cut into parameters and aligned; a row whose bound they move across a power of two gets the next exponent.
template <Elem E>
__device__ __forceinline__ int row_exponent(uint32_t max_bits, const float (&sums)[RowStats<E>::SUMS], float half_sqrt_f, bool& outside) {
    const float m = staged_value<E>(max_bits);
    outside = false;
    if (m != m) return BITS_NAN;
    if (m == INFINITY) return BITS_INF;
    if (m == 0.0f) return 0;
    int e, by_norm;
    frexpf(m, &e);  // m < 2^e
    const int by_max = 28 - e;
    float square = sums[0], scaled = m;
    int up = 0;     // `square` is of 2^up times the elements, and so is `scaled`
    if constexpr (E == Elem::BF16) {
        if (e > 40) {
            square = sums[1];
            up = -90;
        } else if (e < -40) {
            square = sums[2];
            up = 90;
        }
        scaled = ldexpf(m, up);
    }
    const float rest = sqrtf(fmaxf(square - scaled * scaled, 0.0f));
    by_norm = (int)(__float_as_uint(half_sqrt_f / (scaled * 0x1p-24f + rest * 0x1p-22f)) >> 23) - 126 + up;  // 2^by_norm above it
    if (E != Elem::BF16) by_norm = min(by_norm, 24);
    outside = by_norm > by_max;
    return max(by_norm, by_max);
}

struct OutlierLists {
    uint32_t *count, *last, *heads;  // records in use; BitsParams::last_out, heads
    Outlier* outliers;
    uint32_t most;
};

// stage_kernel for project_bits_kernel: staged[tile][128 features][plane][row].  A warp takes runs of 512 features of one
// row, a lane 16 consecutive features, of which it makes the 16 bytes of every plane (gen_bits_pair says in which order).
// Two bytes read (fp16) and four written an element at 4.8 TB/s, and 24 instructions an element, which take half of the issue
// slots: with 32 warps to an SM it is the loads' latency that bounds it.  16 x 2,796,202 fp16 in 55 us, 32 x 1,048,576 fp32 in 47.
// A CTA takes the scale of its rows once, and up to four runs of 512 features of a tile's even share (16 x 592,003 fp16 13 us;
// 18 with eight runs to a CTA and the scale looked up for each).
template <Elem E, bool SEG>
__global__ void __launch_bounds__(256, !SEG && E == Elem::BF16 ? 5 : 4)
stage_bits_kernel(const elem_t<E>* __restrict__ g, const SegDev* __restrict__ segs, uint32_t nsegs, uint64_t row0,
                  uint8_t* __restrict__ staged, const uint32_t* __restrict__ maxima, const float* __restrict__ squares,
                  uint32_t slices, long long* __restrict__ sums, uint32_t* __restrict__ infs, int* __restrict__ row_exp,
                  const OutlierLists lists, float half_sqrt_f, uint32_t B, uint32_t rows, uint64_t F, uint64_t ld,
                  uint32_t fts, uint32_t nst, uint32_t tiles, uint32_t each) {
    using In = elem_t<E>;
    cudaTriggerProgrammaticLaunchCompletion();  // see launch_after
    constexpr uint32_t RUN = 512u, V = 16u / sizeof(In), LOADS = 16u / V;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t runs = (nst * BITS_K + RUN - 1u) / RUN, blocks = (runs + each - 1u) / each;
    // a CTA stays with eight rows, of which it looks up the scale once
    const uint32_t b_hi_n = rows / 8u, b = blockIdx.x % b_hi_n * 8u + warp;
    const uint64_t total = (uint64_t)tiles * blocks;
    cudaGridDependencySynchronize();  // the maxima, and the cleared sums
    RowStats<E> st = {};
    if (b < B) {
#pragma unroll
        for (uint32_t k = 0; k < BITS_MAX_SLICES / 32u; ++k) {  // all fetched at once
            const uint32_t s = k * 32u + lane;
            if (s >= slices) continue;
            st.max_bits = max(st.max_bits, maxima[b * slices + s]);
#pragma unroll
            for (uint32_t j = 0; j < RowStats<E>::SUMS; ++j) st.sums[j] += squares[(b * slices + s) * RowStats<E>::SUMS + j];
        }
    }
#pragma unroll
    for (uint32_t j = 0; j < RowStats<E>::SUMS; ++j)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) st.sums[j] += __shfl_xor_sync(0xffffffffu, st.sums[j], o);
    bool outside;  // some elements of the row may be too large
    const int e = row_exponent<E>(__reduce_max_sync(0xffffffffu, st.max_bits), st.sums, half_sqrt_f, outside);
    // 2^e in two factors (bf16 reaches beyond one)
    const int e1 = e >= BITS_INF ? 0 : E == Elem::BF16 ? e / 2 : e, e2 = e < BITS_INF ? e - e1 : 0;
    const float f1 = __int_as_float((127 + e1) << 23), f2 = __int_as_float((127 + e2) << 23);
    for (uint64_t i = blockIdx.x / b_hi_n; i < total; i += gridDim.x / b_hi_n) {
        const uint32_t tile = (uint32_t)(i / blocks), run0 = (uint32_t)(i - (uint64_t)tile * blocks) * each;
        if (tile == 0 && run0 == 0 && lane == 0) row_exp[b] = e < BITS_INF ? e + 2 : e;
        uint8_t* const out_tile = staged + (uint64_t)tile * nst * (BITS_PLANES * rows * BITS_K);
        long long sum = 0;
        uint32_t ninf = 0;
        uint32_t seg = 0;
        uint64_t s_start = 0, s_end = SEG ? 0 : F;
        const In* s_row = SEG ? nullptr : g + (uint64_t)b * ld;
        for (uint32_t run = run0; run < min(run0 + each, runs); ++run) {
            const uint32_t t0 = run * RUN, t = t0 + lane * 16u;
            const uint64_t f0 = (uint64_t)tile * fts + t0;
            const bool live = b < B && f0 < F && t0 < fts;
            if (SEG && live && f0 >= s_end) {
                uint32_t lo = 0, hi = nsegs;  // last parameter whose start is <= f0
                while (hi - lo > 1u) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (segs[mid].start <= f0)
                        lo = mid;
                    else
                        hi = mid;
                }
                seg = lo;
                s_start = segs[seg].start;
                s_end = s_start + segs[seg].numel;
                s_row = static_cast<const In*>(segs[seg].ptr) + (row0 + b) * segs[seg].stride;
            }
            const uint64_t at = f0 - s_start, left = s_end - f0;
            const In* src = s_row + at;
            const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 15u);
            uint32_t x[16];  // bits of this lane's elements
            if (live && RUN <= left && (off == 0u || (at >= V && RUN + V <= left))) {
                // whole run inside one contiguous source, aligned vectors around it included; a tile may end in it
                if (t >= nst * BITS_K) continue;
                const uint4* vec = reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(src) - off) + LOADS * lane;
                uint4 c[LOADS + 1];
#pragma unroll
                for (uint32_t j = 0; j < LOADS; ++j) c[j] = __ldg(vec + j);
                if (off) {
                    c[LOADS] = __ldg(vec + LOADS);
#pragma unroll
                    for (uint32_t j = 0; j < LOADS; ++j) c[j] = shift_words(c[j], c[j + 1], off);
                }
#pragma unroll
                for (uint32_t j = 0; j < LOADS; ++j) {
                    const uint32_t w[4] = {c[j].x, c[j].y, c[j].z, c[j].w};
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k) {
                        if constexpr (sizeof(In) == 4) {
                            x[j * 4u + k] = w[k];
                        } else {
                            x[j * 8u + 2u * k] = w[k] & 0xffffu;
                            x[j * 8u + 2u * k + 1u] = w[k] >> 16;
                        }
                    }
                }
                if (t0 + RUN > fts) {
#pragma unroll
                    for (uint32_t k = 0; k < 16; ++k) x[k] = t + k < fts ? x[k] : 0u;
                }
            } else {
                if (t >= nst * BITS_K) continue;
                uint32_t si = seg;
                uint64_t e_start = s_start, e_end = s_end;
                const In* e_row = s_row;
#pragma unroll
                for (uint32_t k = 0; k < 16; ++k) {
                    const uint64_t f = f0 + lane * 16u + k;
                    x[k] = 0;
                    if (b < B && t + k < fts && f < F) {
                        while (SEG && f >= e_end) {
                            ++si;
                            e_start = e_end;
                            e_end += segs[si].numel;
                            e_row = static_cast<const In*>(segs[si].ptr) + (row0 + b) * segs[si].stride;
                        }
                        if constexpr (sizeof(In) == 4)
                            x[k] = __float_as_uint(e_row[f - e_start]);
                        else
                            x[k] = e_row[f - e_start];
                    }
                }
            }
            if (outside) {  // the planes hold zeros for what goes to the lists
                auto scaled = [&](uint32_t bits) { return staged_value<E>(bits) * f1 * f2; };
                uint32_t taken = 0;
#pragma unroll
                for (uint32_t k = 0; k < 16; ++k) taken |= (uint32_t)(fabsf(scaled(x[k])) >= BITS_RANGE) << k;
                for (uint32_t left = taken; left != 0u; left &= left - 1u) {
                    const uint32_t one = left & (0u - left);
                    uint32_t bits = 0;
#pragma unroll
                    for (uint32_t k = 0; k < 16; ++k) bits |= one == 1u << k ? x[k] : 0u;
                    const uint32_t r = atomicAdd(lists.count, 1u);
                    if (r >= lists.most) break;  // never (row_exponent)
                    uint32_t* const head = lists.heads + (size_t)tile * nst * 4u + t / 16u;
                    lists.outliers[r] = {atomicExch(head, r + 1u), b, (uint32_t)__ffs((int)one) - 1u, scaled(bits)};
                    atomicMax(lists.last + tile, t / 16u + 1u);
                }
#pragma unroll
                for (uint32_t k = 0; k < 16; ++k) x[k] = taken >> k & 1u ? 0u : x[k];
            }
            // digits of 2^e x, features of even j four times as large (they meet A's 1 and 2, the others its 4 and 8)
            int q[16];
            if (e < BITS_INF) {
#pragma unroll
                for (uint32_t k = 0; k < 16; ++k) {
                    const float v = staged_value<E>(x[k]);
                    q[k] = __float2int_rn(E == Elem::BF16 ? v * f1 * f2 : v * f1);
                }
            } else {
#pragma unroll
                for (uint32_t k = 0; k < 16; ++k) {
                    const float v = staged_value<E>(x[k]);
                    q[k] = v == INFINITY ? 1 : v == -INFINITY ? -1 : 0;
                    ninf += q[k] != 0;
                }
            }
            uint32_t d[16];
            int part[2] = {0, 0};  // eight values of less than 2^28 each
#pragma unroll
            for (uint32_t k = 0; k < 16; ++k) {
                const bool four = ((k >> 1) & 1u) == 0u;
                part[k >> 3] += q[k];
                d[k] = (uint32_t)(four ? 4 * q[k] : q[k]) + 0x00808080u ^ 0x00808080u;  // bytes: balanced base-256 digits
            }
            sum += (long long)part[0] + part[1];
            uint8_t* const dst = out_tile + ((size_t)(t / BITS_BOX_K) * (BITS_PLANES * rows) + b) * BITS_BOX_K + (t % BITS_BOX_K);
            uint32_t o[BITS_PLANES][4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint32_t a0 = d[2u * j], a1 = d[2u * j + 1u], a2 = d[2u * j + 8u], a3 = d[2u * j + 9u];
                const uint32_t l01 = __byte_perm(a0, a1, 0x5140u), h01 = __byte_perm(a0, a1, 0x7362u);
                const uint32_t l23 = __byte_perm(a2, a3, 0x5140u), h23 = __byte_perm(a2, a3, 0x7362u);
                o[0][j] = __byte_perm(l01, l23, 0x5410u);
                o[1][j] = __byte_perm(l01, l23, 0x7632u);
                o[2][j] = __byte_perm(h01, h23, 0x5410u);
                o[3][j] = __byte_perm(h01, h23, 0x7632u);
            }
#pragma unroll
            for (uint32_t pl = 0; pl < BITS_PLANES; ++pl)
                *reinterpret_cast<uint4*>(dst + (size_t)pl * rows * BITS_BOX_K) = make_uint4(o[pl][0], o[pl][1], o[pl][2], o[pl][3]);
        }
        // one addition per warp to the tile's sum: integers, so their order does not matter
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0 && sum != 0)
            atomicAdd(reinterpret_cast<unsigned long long*>(sums + (size_t)tile * rows + b), (unsigned long long)sum);
        if (e == BITS_INF) {
            ninf = __reduce_add_sync(0xffffffffu, ninf);
            if (lane == 0 && ninf != 0) atomicAdd(infs + (size_t)tile * rows + b, ninf);
        }
    }
}

}  // namespace tb
