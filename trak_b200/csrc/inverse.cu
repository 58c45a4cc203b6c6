// Regularised SPD inverse for the after-kernel:  A <- inv(A + lambda*I), optionally divided by
// the mean absolute entry (the reference's rescale, trak/score_computers.py:160-168).
//
// The reference calls torch.linalg.inv (LU).  A + lambda*I is symmetric positive definite, so this
// goes through Cholesky A = L L^T and W = L^-1, all in fp32, over 512-wide block columns:
//   1. the diagonal block is factored and inverted at once, in eight 64-wide steps of one cooperative
//      launch (block_kernel): one step finishes 64 rows of the block's W and updates everything below
//      them; the CTA that updates the next 64 x 64 diagonal tile factors and inverts it on the spot;
//   2. below it L21 = A21 W11^T, and to its right A22 -= L21 L21^T: tensor-core GEMMs (gemm.cu, chunked
//      accumulation), so the long chain of small steps never touches more than 512 x 512;
//   3. the inverted blocks are merged bottom-up, W21 = -W22 (L21 W11) for block sizes 512, 1024, ...,
//      with the same GEMMs;
//   4. A^-1 = W^T W (symmetric mode, chunked accumulation);
//   5. mean |entry| with a fixed-order two-pass reduction, then the rescale.
// A non-positive pivot is recorded in the device status word (ST_NOT_SPD).
#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

#include "gemm.h"
#include "host_util.h"
#include "ptx.cuh"

namespace tb {

constexpr int NB = 64;      // tile of the steps inside a block column
constexpr int OUTER = 512;  // block column
constexpr int TS = 68;      // padded row length of a shared-memory tile (floats)
typedef float Tile[NB][TS];

// The 256 threads of a CTA share the products of 64 x 64 tiles: a thread of the k group g = tid / 64 accumulates
// four 4 x 4 pieces, 32 rows and 32 columns apart, over a quarter of k, and ends with the piece (ty, tx) of the result.
__device__ __forceinline__ int piece_row(int tid) { return 8 * (tid >> 7) + ((tid & 63) >> 3); }
__device__ __forceinline__ int piece_col(int tid) { return 8 * ((tid >> 6) & 1) + (tid & 7); }
constexpr int EXCHANGE_FLOATS = 4 * 3 * 16 * 64;  // what a product's k groups hand to one another

// acc[4][4] = sum_t At[t][ty*4 + i] * Bt[t][tx*4 + j]   (both tiles stored t-major; 256 threads)
// Shared memory bounds it: a 16-byte load takes the SM four cycles whatever its lanes share.  With one piece a thread
// and all of k that is 1024 loads a product and 4450 cycles; four pieces over a quarter of k each and the exchange of three
// quarters of the partial sums are 704 and 4000, with the next loads issued before a step's multiplications.
__device__ __forceinline__ void tile_mma(const float (*At)[TS], const float (*Bt)[TS], float* exchange, float (&acc)[4][4]) {
    const int tid = threadIdx.x, g = tid >> 6, u = tid & 63, r0 = (u >> 3) * 4, c0 = (u & 7) * 4;
    uint64_t s2[8][4] = {};
    float4 a0, a1, a0n, a1n;
    ulonglong2 b0, b1, b0n, b1n;
    auto load = [&](int t) {
        a0n = *reinterpret_cast<const float4*>(&At[t][r0]);
        a1n = *reinterpret_cast<const float4*>(&At[t][r0 + 32]);
        b0n = *reinterpret_cast<const ulonglong2*>(&Bt[t][c0]);
        b1n = *reinterpret_cast<const ulonglong2*>(&Bt[t][c0 + 32]);
    };
    load(g * 16);
#pragma unroll
    for (int t = 0; t < 16; ++t) {
        a0 = a0n; a1 = a1n; b0 = b0n; b1 = b1n;
        if (t < 15) load(g * 16 + t + 1);
        const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        const uint64_t bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint64_t a = pack_f32x2(av[i], av[i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) s2[i][j] = fma_f32x2(a, bv[j], s2[i][j]);
        }
    }
    float s[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) unpack_f32x2(s2[i][j], s[i][2 * j], s[i][2 * j + 1]);
    // group g keeps its threads' piece in the rows 32 (g >> 1) .. and the columns 32 (g & 1) ..
    float4* ex = reinterpret_cast<float4*>(exchange);
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        if (d == g) continue;
        float4* to = ex + ((d * 3 + (g - (g > d))) * 4) * 64 + u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float* row = &s[4 * (d >> 1) + i][4 * (d & 1)];
            to[i * 64] = make_float4(row[0], row[1], row[2], row[3]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int d = 0; d < 4; ++d)
        if (d == g) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = s[4 * (d >> 1) + i][4 * (d & 1) + j];
        }
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const float4* from = ex + ((g * 3 + e) * 4) * 64 + u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 v = from[i * 64];
            acc[i][0] += v.x; acc[i][1] += v.y; acc[i][2] += v.z; acc[i][3] += v.w;
        }
    }
    __syncthreads();  // the next product writes there again
}

__device__ __forceinline__ void put_piece(Tile& T, int ty, int tx, const float (&acc)[4][4]) {
#pragma unroll
    for (int a = 0; a < 4; ++a)
        *reinterpret_cast<float4*>(&T[ty * 4 + a][tx * 4]) = make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
}

// Rows and columns [0, rows) x [0, cols) of a 64 x 64 tile at src, zero outside, in the registers of N threads (this one is
// number `id`); four consecutive elements of a row each where the rows are 16-byte aligned.  Past the L1: other CTAs write
// the tiles between a CTA's reads.
template <int N>
struct TileRegs {
    float v[4096 / (4 * N)][4];
    static __device__ __forceinline__ void place(int id, int it, int& i, int& t) {  // eight rows x 16 columns a warp
        const int e = it * N + id, warp = e >> 5, lane = e & 31;
        i = (warp >> 2) * 8 + (lane & 7);
        t = (warp & 3) * 16 + (lane >> 3) * 4;
    }
    __device__ __forceinline__ void fetch(int id, const float* src, int64_t ld, int rows, int cols) {
        const bool vec = (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
#pragma unroll
        for (int it = 0; it < 4096 / (4 * N); ++it) {
            int i, t;
            place(id, it, i, t);
            if (vec && i < rows && t + 4 <= cols) {
                const float4 x = __ldcg(reinterpret_cast<const float4*>(src + (int64_t)i * ld + t));
                v[it][0] = x.x; v[it][1] = x.y; v[it][2] = x.z; v[it][3] = x.w;
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) v[it][u] = (i < rows && t + u < cols) ? __ldcg(src + (int64_t)i * ld + t + u) : 0.0f;
            }
        }
    }
    // dst[t][i] (TRANS; the stores meet two to a bank) or dst[i][t]
    template <bool TRANS>
    __device__ __forceinline__ void put(int id, Tile& dst) const {
#pragma unroll
        for (int it = 0; it < 4096 / (4 * N); ++it) {
            int i, t;
            place(id, it, i, t);
            if (TRANS) {
#pragma unroll
                for (int u = 0; u < 4; ++u) dst[t + u][i] = v[it][u];
            } else {
                *reinterpret_cast<float4*>(&dst[i][t]) = make_float4(v[it][0], v[it][1], v[it][2], v[it][3]);
            }
        }
    }
};

// A += lambda I, and zero for the counters that the block columns' CTAs meet at.
__global__ void prepare_kernel(float* A, int64_t lda, int k, float lambda, uint32_t* counters, int n) {
    after_earlier_launch();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < k && lambda != 0.0f) A[(int64_t)i * lda + i] += lambda;
    if (i < n) counters[i] = 0;
}

// Factors the jb x jb diagonal tile S = L L^T (lower triangle used) and inverts L in the same sweep (forward
// elimination of [L | I]); writes inv(L) (lower, zero above, zero-padded to 64 x 64) to dinv and, t-major, to Dt.
// CHOL_THREADS threads: 136 hold the lower triangle's 4 x 4 pieces in registers, warp 0 is the pivot warp.  The tile is
// walked eight columns at a time.  The thread of piece (ty, tx) holds it of S until the step of its columns and of
// W = inv(L) from then on (it is zero until its column has been reached, final from the step of its rows on), so that a
// step is one small product and one rank-eight update whichever it is.  With Ld Ld^T the diagonal block of step q and
//     P[d][i] = S[i, 8q + d] below the block, the identity in it, W[8q + d, i] left of it,
//   1. the pivot warp has factored the block and published Ld^-1;
//   2. O = Ld^-1 P: below the block the columns of L, in it and left of it the block's rows of W, final;
//   3. the threads below update their pieces, x[i, j] -= sum_c O[c][i] O[c][j], and publish P of the next step.
// The pivot warp is a step ahead of the others: what it needs of step q for the next diagonal block are eight rows of O,
// which it computes itself from P, and that block as it was before the step.  Then it factors it,
// every lane for itself in registers (a lane then solves for one column of the inverse): a chain of eight reciprocal
// square roots, 50 cycles each.  So a step takes as long as the pivot warp's part or the others', not as both.
// With four columns a step, a factor published instead of its inverse and substitutions by the threads of its pieces, a
// tile took 12,500 cycles (with 8 x 4 pieces in three warps 12,400: half of it is stores and loads of shared memory, of which
// a warp gets one of 16 bytes every 14 cycles).  Every warp runs through straight code that no other warp of its scheduler
// runs, so each piece of it is there once: with the hand-overs, the factorisation and the products of CTA 0 and of the others
// expanded where they are used, the one-tile launch spent most of its time waiting for instructions (668 misses of the
// instruction cache; 215 with one copy of each, and 15.3 -> 14.0 us with the pivot warp ahead).
// Rows and columns beyond jb are an identity block.  `buf` is CHOL_FLOATS floats of shared memory outside S.
constexpr int CW = 8;                                             // columns of a step
constexpr int CHOL_FLOATS = 3 * CW * NB + 6 * CW * CW;
static_assert(CHOL_FLOATS <= NB * TS, "a tile's worth of shared memory holds chol_block's buffers");
constexpr int CHOL_THREADS = 192;  // warps 0 (pivot), 1, 2, 3, 5 and 6
// 1 / sqrt(d) for a normal d; a subnormal one counts as not positive (the inverse would overflow)
__device__ __forceinline__ float rsqrt_newton(float d) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return fmaf(r, fmaf(-(0.5f * d) * r, r, 0.5f), r);
}
// Column `col` of inv(chol(z)) (rows of z, lower part used) in y; false when a pivot is not positive.
__device__ __forceinline__ bool invert_block(float (&z)[CW][CW], int col, float (&y)[CW]) {
    bool ok = true;
#pragma unroll
    for (int j = 0; j < CW; ++j) {
        ok = ok && z[j][j] >= 1.17549435e-38f;
        const float r = rsqrt_newton(z[j][j]);
#pragma unroll
        for (int i = j + 1; i < CW; ++i) z[i][j] *= r;
#pragma unroll
        for (int l = j + 1; l < CW; ++l)
#pragma unroll
            for (int i = l; i < CW; ++i) z[i][l] = fmaf(-z[i][j], z[l][j], z[i][l]);
        float t = j == col ? 1.0f : 0.0f;
#pragma unroll
        for (int k = 0; k < j; ++k) t = fmaf(-z[j][k], y[k], t);
        y[j] = t * r;
    }
    return ok;
}
__device__ void chol_block(const Tile& S, int jb, float* dinv, Tile& Dt, uint32_t* status, float* buf) {
    // Barriers: 1 between the threads of the pieces; 2 and 3 (even and odd steps) hand them the step's Ld^-1, 4 and 5 hand
    // the pivot warp the step's P.  Either side waits for the other's last hand-over before its next but one, so two of
    // each, and two of the buffers behind them, are enough.
    auto sync = [] { asm volatile("barrier.cta.sync 1, %0;" ::"n"(CHOL_THREADS - 32) : "memory"); };
    auto take = [](int bar) { asm volatile("barrier.cta.sync %0, %1;" ::"r"(bar), "n"(CHOL_THREADS) : "memory"); };
    auto give = [](int bar) { asm volatile("barrier.cta.arrive %0, %1;" ::"r"(bar), "n"(CHOL_THREADS) : "memory"); };
    const int tid = threadIdx.x, lane = tid & 31;
    typedef float Panel[CW][NB];
    typedef float Block[CW][CW];
    Panel* const Ps = reinterpret_cast<Panel*>(buf);                         // P of even and odd steps
    Panel& O = *reinterpret_cast<Panel*>(buf + 2 * CW * NB);
    Block* const invs = reinterpret_cast<Block*>(buf + 3 * CW * NB);         // Ld^-1 of even and odd steps
    Block* const before = invs + 2;                                          // diagonal blocks as they were a step earlier
    Block &now = before[2], &rows_of_o = before[3];                          // the pivot warp's own
    const int warp = tid >> 5;
    const bool pivot = warp == 0;
    // piece (ty, tx) of the grid's threads, row by row: the first rows' warp, done early, shares a scheduler
    const int n = (warp == 5 ? 0 : warp == 6 ? 4 : warp) * 32 + lane;
    const int ty = (int)((sqrtf(8.0f * n + 1.0f) - 1.0f) * 0.5f), tx = n - ty * (ty + 1) / 2;
    const bool owner = !pivot && n < 136;
    const int panel = warp == 5 ? lane : warp >= 1 && warp <= 3 ? warp * 32 + lane : -1;  // of the 128 threads that compute O
    const int steps = (jb + CW - 1) / CW;
    auto entry = [&](int i, int j) { return i < jb && j < jb ? S[i][j] : i == j ? 1.0f : 0.0f; };
    float x[4][4];
    if (owner) {
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            if (ty * 4 + 4 <= jb) {  // (what is above the diagonal of a diagonal piece is never used)
                const float4 v = *reinterpret_cast<const float4*>(&S[ty * 4 + a][tx * 4]);
                x[a][0] = v.x; x[a][1] = v.y; x[a][2] = v.z; x[a][3] = v.w;
            } else {
#pragma unroll
                for (int b = 0; b < 4; ++b) x[a][b] = entry(ty * 4 + a, tx * 4 + b);
            }
        }
    }
    // P of step q, and the diagonal block of step q + 1 for the pivot warp
    auto publish = [&](int q) {
        const int r = ty - 2 * q, c = tx - 2 * q;  // piece row and column relative to the step's block
        Panel& P = Ps[q & 1];
        if (c >= 0 && c < 2 && r >= 2) {
#pragma unroll
            for (int b = 0; b < 4; ++b)
                *reinterpret_cast<float4*>(&P[c * 4 + b][ty * 4]) = make_float4(x[0][b], x[1][b], x[2][b], x[3][b]);
        }
        if (r >= 0 && r < 2) {
#pragma unroll
            for (int a = 0; a < 4; ++a)
                *reinterpret_cast<float4*>(&P[r * 4 + a][tx * 4]) =
                    c < 0 ? make_float4(x[a][0], x[a][1], x[a][2], x[a][3])
                          : make_float4(r == c && a == 0, r == c && a == 1, r == c && a == 2, r == c && a == 3);
            if (r == 0 && c == 0) {  // nobody's piece right of it
#pragma unroll
                for (int a = 0; a < 4; ++a) *reinterpret_cast<float4*>(&P[a][tx * 4 + 4]) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        if (r >= 2 && r < 4 && c >= 2) {
            Block& d = before[(q + 1) & 1];
#pragma unroll
            for (int a = 0; a < 4; ++a)
                *reinterpret_cast<float4*>(&d[(r - 2) * 4 + a][(c - 2) * 4]) = make_float4(x[a][0], x[a][1], x[a][2], x[a][3]);
        }
    };
    bool ok = true;
    if (pivot) {
        float z[CW][CW], y[CW];
        // factors z and publishes the inverse, one column per lane
        auto factor = [&](int q) {
            ok = invert_block(z, lane & (CW - 1), y) && ok;
            if (lane < CW) {
#pragma unroll
                for (int r = 0; r < CW; ++r) invs[q & 1][r][lane] = r >= lane ? y[r] : 0.0f;
            }
            __syncwarp();
            give(2 + (q & 1));
        };
        for (int q = -1; q + 1 < steps; ++q) {
            const int r = lane >> 2, c = (lane & 3) * 2, at = (q + 1) * CW;
            float2 v = make_float2(c <= r ? entry(r, c) : 0.0f, c < r ? entry(r, c + 1) : 0.0f);
            if (q >= 0) {
                float w[CW];
#pragma unroll
                for (int d = 0; d < CW; d += 4) {
                    const float4 t = *reinterpret_cast<const float4*>(&invs[q & 1][r][d]);
                    w[d] = t.x; w[d + 1] = t.y; w[d + 2] = t.z; w[d + 3] = t.w;
                }
                take(4 + (q & 1));
                float2 o = make_float2(0.0f, 0.0f), m[CW];
                float l[CW];
                v = *reinterpret_cast<const float2*>(&before[(q + 1) & 1][r][c]);
#pragma unroll
                for (int d = 0; d < CW; ++d) {
                    const float2 p = *reinterpret_cast<const float2*>(&Ps[q & 1][d][at + c]);
                    o.x = fmaf(w[d], p.x, o.x);
                    o.y = fmaf(w[d], p.y, o.y);
                }
                *reinterpret_cast<float2*>(&rows_of_o[r][c]) = o;
                __syncwarp();
#pragma unroll
                for (int k = 0; k < CW; ++k) {
                    l[k] = rows_of_o[k][r];
                    m[k] = *reinterpret_cast<const float2*>(&rows_of_o[k][c]);
                }
#pragma unroll
                for (int k = 0; k < CW; ++k) {
                    v.x = fmaf(-l[k], m[k].x, v.x);
                    v.y = fmaf(-l[k], m[k].y, v.y);
                }
            }
            *reinterpret_cast<float2*>(&now[r][c]) = v;
            __syncwarp();
#pragma unroll
            for (int i = 0; i < CW; ++i)
#pragma unroll
                for (int j = 0; j < CW; j += 4) {
                    if (j > i) continue;
                    const float4 t = *reinterpret_cast<const float4*>(&now[i][j]);
                    z[i][j] = t.x; z[i][j + 1] = t.y; z[i][j + 2] = t.z; z[i][j + 3] = t.w;
                }
            factor(q + 1);
        }
    } else {
        for (int q = 0; q < steps; ++q) {
            if (owner) publish(q);
            if (q + 1 < steps) give(4 + (q & 1));
            take(2 + (q & 1));
            if (panel >= 0) {  // four entries of O each
                const Block& inv = invs[q & 1];
                const Panel& P = Ps[q & 1];
                const int at = panel & 63, c = (panel >> 6) * 4;
                float o[4] = {}, v[4][CW];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    *reinterpret_cast<float4*>(&v[k][0]) = *reinterpret_cast<const float4*>(&inv[c + k][0]);
                    *reinterpret_cast<float4*>(&v[k][4]) = *reinterpret_cast<const float4*>(&inv[c + k][4]);
                }
#pragma unroll
                for (int d = 0; d < CW; ++d) {
                    const float p = P[d][at];
#pragma unroll
                    for (int k = 0; k < 4; ++k) o[k] = fmaf(v[k][d], p, o[k]);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) O[c + k][at] = o[k];
            }
            sync();
            if (owner) {
                const int r = ty - 2 * q, c = tx - 2 * q;
                if (r >= 0 && r < 2) {  // the step's rows of W
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        const float4 w = *reinterpret_cast<const float4*>(&O[r * 4 + a][tx * 4]);
                        x[a][0] = w.x; x[a][1] = w.y; x[a][2] = w.z; x[a][3] = w.w;
                    }
                } else if (r >= 2) {
                    if (c >= 0 && c < 2) {  // from S, which has become L, to W
#pragma unroll
                        for (int a = 0; a < 4; ++a)
#pragma unroll
                            for (int b = 0; b < 4; ++b) x[a][b] = 0.0f;
                    }
#pragma unroll
                    for (int k = 0; k < CW; ++k) {
                        const float4 l = *reinterpret_cast<const float4*>(&O[k][ty * 4]);
                        const float4 o = *reinterpret_cast<const float4*>(&O[k][tx * 4]);
                        const float lv[4] = {l.x, l.y, l.z, l.w}, ov[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                        for (int a = 0; a < 4; ++a)
#pragma unroll
                            for (int b = 0; b < 4; ++b) x[a][b] = fmaf(-lv[a], ov[b], x[a][b]);
                    }
                }
            }
        }
    }
    if (owner) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int i = ty * 4 + a;
#pragma unroll
            for (int b = 0; b < 4; ++b) x[a][b] = (i < jb && tx * 4 + b <= i) ? x[a][b] : 0.0f;
            *reinterpret_cast<float4*>(dinv + i * NB + tx * 4) = make_float4(x[a][0], x[a][1], x[a][2], x[a][3]);
            if (tx < ty) {  // the piece across the diagonal
                *reinterpret_cast<float4*>(dinv + (tx * 4 + a) * NB + ty * 4) = zero;
                *reinterpret_cast<float4*>(&Dt[i][tx * 4]) = zero;
            }
        }
#pragma unroll
        for (int b = 0; b < 4; ++b)
            *reinterpret_cast<float4*>(&Dt[tx * 4 + b][ty * 4]) = make_float4(x[0][b], x[1][b], x[2][b], x[3][b]);
    }
    if (!ok) record_status(status, (uint32_t)ST_NOT_SPD);
}

// Counters of a block column: `factored` tiles of the diagonal (CTA 0), and steps x CTAs finished by the others.
struct BlockCounters {
    uint32_t factored, finished;
};
// Waits until *counter has reached `target`; one thread.  Bounded.
__device__ bool reached(const uint32_t* counter, uint32_t target, uint32_t* status) {
    const uint64_t t0 = globaltimer_ns();
    for (uint32_t n = 1;; ++n) {
        uint32_t seen;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
        if (seen >= target) return true;
        if ((n & 255u) == 0 && globaltimer_ns() - t0 > WAIT_LIMIT_NS) {
            if (record_status(status, (uint32_t)ST_TIMEOUT_ACC)) status[1] = blockIdx.x;
            return false;
        }
    }
}

// Step j of a block column's diagonal block (kb x kb, kb <= 512), in tiles of 64.  Before the step, rows i >= j hold
// R[i, c] for c < j (what is left of the identity's elimination, W's future rows) and S[i, l] for l >= j (what is
// left of A), and D = inv(chol(S[j, j])) is known.  The step makes row j of W final,
//     W[j, c] = D R[j, c],   W[j, j] = D,
// and with P_i = S[i, j] D^T (the rows of L) updates every row i > j:
//     S[i, l] -= P_i P_l^T (j < l <= i),   R[i, c] -= P_i W[j, c] (c < j),   R[i, j] = -P_i D.
// One CTA per tile, each computing the P and W tiles it needs itself (three 64^3 products instead of another meeting point
// and a trip through memory).  Rows i > j go from X to Y (tiles are read by many CTAs, so they are not updated in place);
// W's rows go to `block`, the matrix itself, with zeros right of the diagonal.  What a tile needs of X is fetched before D is
// waited for (*factored > j), where a CTA spends a quarter of a step.  False when the wait ran out.
__device__ bool block_tile(float* smem, const float* X, int64_t ldx, float* Y, float* block, int64_t lda, int kb, int j, int i,
                           int c, const float* D, const uint32_t* factored, uint32_t* status, uint32_t* have_d) {
    Tile& Dt = *reinterpret_cast<Tile*>(smem);                // Dt[t][c] = D[c][t]
    Tile& T0 = *reinterpret_cast<Tile*>(smem + NB * TS);
    Tile& T1 = *reinterpret_cast<Tile*>(smem + 2 * NB * TS);
    Tile& T2 = *reinterpret_cast<Tile*>(smem + 3 * NB * TS);
    float* const exchange = smem + 4 * NB * TS;
    const int tid = threadIdx.x, ty = piece_row(tid), tx = piece_col(tid);
    const int rows = min(NB, kb - i * NB), jw = min(NB, kb - j * NB), cols = min(NB, kb - c * NB);
    float acc[4][4];
    TileRegs<256> d, t1, t2;
    auto wait_for_d = [&] {
        if (tid == 0) *have_d = reached(factored, (uint32_t)j + 1u, status);
        __syncthreads();
        return *have_d != 0u;
    };
    if (i == j) {  // row j of W
        if (c < j) {
            t1.fetch(tid, X + (int64_t)j * NB * ldx + c * NB, ldx, rows, NB);
            t1.put<false>(tid, T0);
        }
        if (!wait_for_d()) return false;
        if (c < j) {
            d.fetch(tid, D, NB, NB, NB);
            d.put<true>(tid, Dt);
            __syncthreads();
            tile_mma(Dt, T0, exchange, acc);
        }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int r = ty * 4 + a, q = tx * 4 + b;
                if (r < rows && q < cols)
                    block[(int64_t)(j * NB + r) * lda + c * NB + q] = c < j ? acc[a][b] : c == j ? __ldcg(D + r * NB + q) : 0.0f;
            }
        return true;
    }
    t1.fetch(tid, X + (int64_t)i * NB * ldx + j * NB, ldx, rows, jw);
    if (c > j && c != i)
        t2.fetch(tid, X + (int64_t)c * NB * ldx + j * NB, ldx, cols, jw);
    else if (c < j)
        t2.fetch(tid, X + (int64_t)j * NB * ldx + c * NB, ldx, jw, NB);
    // this CTA's own tile, in flight during the products
    float own[4][4];
    const float* mine = X + (int64_t)(i * NB + ty * 4) * ldx + c * NB + tx * 4;
    const bool vec = (ldx & 3) == 0 && (reinterpret_cast<uintptr_t>(X) & 15u) == 0 && tx * 4 + 4 <= cols;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const bool live = c != j && ty * 4 + a < rows;
        if (vec && live) {
            *reinterpret_cast<float4*>(own[a]) = __ldcg(reinterpret_cast<const float4*>(mine + a * ldx));
        } else {
#pragma unroll
            for (int b = 0; b < 4; ++b) own[a][b] = (live && tx * 4 + b < cols) ? __ldcg(mine + a * ldx + b) : 0.0f;
        }
    }
    t1.put<true>(tid, T1);
    if (c > j && c != i)
        t2.put<true>(tid, T2);
    else if (c < j)
        t2.put<false>(tid, T2);
    if (!wait_for_d()) return false;
    d.fetch(tid, D, NB, NB, NB);
    d.put<true>(tid, Dt);
    if (c == j) d.put<false>(tid, T2);
    __syncthreads();
    // P_i^T = D S[i, j]^T, i.e. P_i t-major, into T0; the other operand, P_c^T or W[j, c], into T1 (the product before is done
    // with it); then the product of the two
    const int last = c != i && c != j ? 2 : 1;
#pragma unroll 1
    for (int product = 0;; ++product) {
        tile_mma(product == last ? T0 : Dt,
                 product == 0 ? T1 : product < last ? T2 : c == i ? T0 : c == j ? T2 : T1, exchange, acc);
        if (product == last) break;
        put_piece(product == 0 ? T0 : T1, ty, tx, acc);
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
        *reinterpret_cast<float4*>(Y + (int64_t)(i * NB + ty * 4 + a) * OUTER + c * NB + tx * 4) =
            make_float4(own[a][0] - acc[a][0], own[a][1] - acc[a][1], own[a][2] - acc[a][2], own[a][3] - acc[a][3]);
    return true;
}

// What this CTA's threads have written, then the counter.  All threads; the next use of what they read needs no further
// barrier.
__device__ __forceinline__ void announce(uint32_t* counter) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(counter, 1u);
    }
}

// Factors and inverts a diagonal block (kb x kb).  CTA 0 walks down the diagonal: it factors a tile, updates the next one
// with it from what the two warps left over have fetched meanwhile (the column's tile beside it and the tile itself, as the others
// left them a step earlier) and goes on, without waiting for anyone unless the others fall behind.  They wait for a tile's
// inverse, share the step's tiles and wait for one another.  A cooperative launch of about as many CTAs as the largest step
// has tiles.  With one meeting point of all CTAs per step, CTA 0's tiles fetched behind it and the slower products and
// factorisation of before, the 512-wide block took 126 us; 97 after that, 89.3 with what a tile needs of the step before
// fetched while its inverse is waited for, and 86.8 with one copy of the products' code and chol_block as it is.
constexpr int STEP_THREADS = 256;
constexpr size_t STEP_SMEM = (5 * NB * TS + EXCHANGE_FLOATS + CHOL_FLOATS) * sizeof(float);
__global__ void __launch_bounds__(STEP_THREADS, 1) block_kernel(float* block, int64_t lda, int kb, float* blocks, float* dinv,
                                                                BlockCounters* counters, uint32_t* status) {
    extern __shared__ __align__(16) float smem[];
    __shared__ uint32_t proceed, have_d;
    const int nt = (kb + NB - 1) / NB, tid = threadIdx.x;
    const uint32_t others = gridDim.x - 1;
    auto source = [&](int j) { return j == 0 ? block : blocks + (size_t)((j - 1) & 1) * OUTER * OUTER; };
    auto source_ld = [&](int j) { return j == 0 ? lda : (int64_t)OUTER; };
    if (blockIdx.x == 0) {
        Tile& Dt = *reinterpret_cast<Tile*>(smem);
        Tile& T0 = *reinterpret_cast<Tile*>(smem + NB * TS);
        Tile& T1 = *reinterpret_cast<Tile*>(smem + 2 * NB * TS);
        Tile& S = *reinterpret_cast<Tile*>(smem + 3 * NB * TS);
        Tile& next = *reinterpret_cast<Tile*>(smem + 4 * NB * TS);
        float* const exchange = smem + 5 * NB * TS;
        float* const buf = exchange + EXCHANGE_FLOATS;
        const int warp = tid >> 5, ty = piece_row(tid), tx = piece_col(tid);
        TileRegs<256> first;
        first.fetch(tid, block, lda, min(NB, kb), min(NB, kb));
        first.put<false>(tid, S);
        if (tid == 0) proceed = 1;
        for (int j = 0;; ++j) {
            __syncthreads();
            // the tiles (j + 1, j) and (j + 1, j + 1) of step j, beside the factorisation
            const int rows = min(NB, kb - (j + 1) * NB);
            if (warp != 4 && warp != 7) {
                chol_block(S, min(NB, kb - j * NB), dinv + (size_t)j * NB * NB, Dt, status, buf);
            } else if (j + 1 < nt) {
                const int lane = tid & 31, id = (warp == 7 ? 32 : 0) + lane;
                bool ok = lane != 0 || reached(&counters->finished, (uint32_t)j * others, status);
                ok = __all_sync(0xffffffffu, ok);
                __syncwarp();  // a vote orders no memory: this hands lane 0's acquire on to the lanes that read behind it
                const float* at = source(j) + (int64_t)(j + 1) * NB * source_ld(j) + j * NB;
                if (ok) {
                    TileRegs<64> t, u;
                    t.fetch(id, at, source_ld(j), rows, NB);
                    u.fetch(id, at + NB, source_ld(j), rows, rows);
                    t.put<true>(id, T1);
                    u.put<false>(id, next);
                } else if (lane == 0) {
                    proceed = 0;
                }
            }
            announce(&counters->factored);
            if (j + 1 == nt || !*const_cast<volatile uint32_t*>(&proceed)) return;
            float acc[4][4];
#pragma unroll 1
            for (int product = 0; product < 2; ++product) {  // P^T, then what it takes off
                tile_mma(product ? T0 : Dt, product ? T0 : T1, exchange, acc);
                if (product == 0) put_piece(T0, ty, tx, acc);
                __syncthreads();
            }
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const float4 v = *reinterpret_cast<const float4*>(&next[ty * 4 + a][tx * 4]);
                *reinterpret_cast<float4*>(&S[ty * 4 + a][tx * 4]) =
                    make_float4(v.x - acc[a][0], v.y - acc[a][1], v.z - acc[a][2], v.w - acc[a][3]);
            }
        }
    }
    for (int j = 0; j < nt; ++j) {
        if (tid == 0) proceed = reached(&counters->finished, (uint32_t)j * others, status);
        __syncthreads();
        if (!proceed) return;
        float* Y = blocks + (size_t)(j & 1) * OUTER * OUTER;
        const float* D = dinv + (size_t)j * NB * NB;
        int tiles = nt;  // row j of W, and the tiles (i, c), c <= i, of the rows below
        for (int i = j + 1; i < nt; ++i) tiles += i + 1;
        for (int t = (int)blockIdx.x - 1; t < tiles; t += (int)others) {
            int i = j, c = t;
            if (t >= nt) {
                c = t - nt;
                for (i = j + 1; c > i; ++i) c -= i + 1;
                if (i == j + 1 && c == j + 1) continue;  // CTA 0's
            }
            if (!block_tile(smem, source(j), source_ld(j), Y, block, lda, kb, j, i, c, D, &counters->factored, status, &have_d))
                return;
            __syncthreads();
        }
        announce(&counters->finished);
    }
}

// The three whole-matrix passes below walk rows per CTA and columns per thread (no index division), four
// columns at a time where the rows are 16-byte aligned.
__device__ __forceinline__ bool rows_are_vec4(const float* A, int64_t lda, int k) {
    return (k & 3) == 0 && (lda & 3) == 0 && (reinterpret_cast<uintptr_t>(A) & 15u) == 0;
}

constexpr int RED_BLOCKS = 1024;
__global__ void __launch_bounds__(256) abs_partial_kernel(const float* A, int64_t lda, int k, double* partial) {
    after_earlier_launch();
    __shared__ double sh[256];
    double s = 0.0;
    const bool vec = rows_are_vec4(A, lda, k);
    for (int i = blockIdx.x; i < k; i += RED_BLOCKS) {   // fixed assignment of entries to threads: same sum every run
        const float* row = A + (int64_t)i * lda;
        if (vec) {
            for (int j4 = threadIdx.x; j4 < (k >> 2); j4 += 256) {
                const float4 v = *reinterpret_cast<const float4*>(row + 4 * j4);
                s += (double)fabsf(v.x) + (double)fabsf(v.y) + (double)fabsf(v.z) + (double)fabsf(v.w);
            }
        } else {
            for (int j = threadIdx.x; j < k; j += 256) s += (double)fabsf(row[j]);
        }
    }
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}
// The mean of |entry| from the partial sums, the same in every CTA (256 threads).
__device__ float mean_abs(const double* partial, int k) {
    __shared__ double sh[256];
    double s = 0.0;
    for (int e = threadIdx.x; e < RED_BLOCKS; e += 256) s += partial[e];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    return (float)(sh[0] / ((double)k * (double)k));
}
__global__ void __launch_bounds__(256) abs_final_kernel(const double* partial, int k, float* mean_out) {
    after_earlier_launch();
    const float mean = mean_abs(partial, k);
    if (threadIdx.x == 0) *mean_out = mean;
}
// Every CTA sums the 8 KB of partial sums itself (about 1 us) instead of waiting for a launch that does.
__global__ void __launch_bounds__(256) scale_by_inverse_kernel(float* A, int64_t lda, int k, const double* partial,
                                                               float* mean_out) {
    after_earlier_launch();
    const float mean = mean_abs(partial, k), inv = 1.0f / mean;
    if (mean_out && blockIdx.x == 0 && threadIdx.x == 0) *mean_out = mean;
    const bool vec = rows_are_vec4(A, lda, k);
    for (int i = blockIdx.x; i < k; i += gridDim.x) {
        float* row = A + (int64_t)i * lda;
        if (vec) {
            for (int j4 = threadIdx.x; j4 < (k >> 2); j4 += blockDim.x) {
                float4 v = *reinterpret_cast<float4*>(row + 4 * j4);
                v.x *= inv; v.y *= inv; v.z *= inv; v.w *= inv;
                *reinterpret_cast<float4*>(row + 4 * j4) = v;
            }
        } else {
            for (int j = threadIdx.x; j < k; j += blockDim.x) row[j] *= inv;
        }
    }
}

// C[m x n] = alpha * A[m x kk] . B[n x kk]^T (+ C) with chunked accumulation, operands packed first: the bytes of the
// packed operands (0 rows: B is A, symmetric) and of the partial products behind them.
struct Product {
    Packed a, b;
    size_t partial;
    size_t bytes() const { return a.bytes + b.bytes + partial; }
};
static Product product(int64_t m, int64_t n, int64_t kk, bool symmetric) {
    Product p;
    p.a = packed_geometry(TB_F32, m, kk);
    p.b = symmetric ? Packed{} : packed_geometry(TB_F32, n, kk);
    p.partial = plan_gemm(2, true, symmetric, m, n, p.a.kblocks).partial_bytes;
    return p;
}

struct InvLayout {
    size_t dinv, blocks, partial, counters, chain, rest, left, merge, total;
    // the merges' first products: one per level is waiting for its second at a time
    size_t left_at(int64_t s) const {
        size_t at = left;
        for (int64_t t = OUTER; t < s; t *= 2) at += (size_t)t * t * sizeof(float);
        return at;
    }
};
static InvLayout inv_layout(int64_t k) {
    InvLayout l;
    size_t off = 0;
    l.dinv = off;
    off += (OUTER / NB) * NB * NB * sizeof(float);
    l.blocks = off;  // the two copies of a diagonal block that its steps alternate between
    off += 2u * OUTER * OUTER * sizeof(float);
    l.partial = off;
    off += align_up(RED_BLOCKS * sizeof(double), 256);
    l.counters = off;
    off += align_up((size_t)((k + OUTER - 1) / OUTER) * sizeof(BlockCounters), 256);
    // what the block columns, the rest of their updates and the merges use at the same time
    size_t chain = 0, rest = 0, merge = product(k, k, k, true).bytes();  // W^T W
    for (int64_t o = 0; o + OUTER < k; o += OUTER) {
        const int64_t r = k - o - OUTER, d = std::min<int64_t>(OUTER, r);
        chain = std::max(chain, product(r, OUTER, OUTER, false).bytes());
        chain = std::max(chain, product(r, OUTER, OUTER, true).a.bytes + product(d, d, OUTER, true).partial);
        if (r > d) rest = std::max(rest, std::max(product(r - d, d, OUTER, false).partial, product(r - d, r - d, OUTER, true).partial));
    }
    for (int64_t s = OUTER; s < k; s *= 2)
        for (int64_t b0 = 0; b0 + s < k; b0 += 2 * s) {
            const int64_t s2 = std::min<int64_t>(s, k - b0 - s);
            merge = std::max(merge, std::max(product(s, s2, s, false).bytes(), product(s2, s, s2, false).bytes()));
        }
    l.chain = off = align_up(off, 1024);
    l.rest = off = align_up(off + chain, 1024);
    l.left = off = align_up(off + rest, 1024);
    int64_t levels = OUTER;
    while (levels < k) levels *= 2;
    l.merge = off = l.left_at(levels);
    l.total = off + merge + 1024;
    return l;
}

// Two streams beside the caller's: `chain` (high priority) factors the block columns one after the other, `rest` applies
// the part of their updates that the next column does not wait for.  A call borrows a set and gives it back when
// everything is queued and the caller's stream waits for it (a later borrower at most waits for that work too); at most
// MAX_KEPT idle sets are kept per device.
struct SideStreams {
    cudaStream_t chain = nullptr, rest = nullptr;
    cudaEvent_t forked = nullptr, block = nullptr, packed = nullptr, updated = nullptr;
    int make() {
        int least = 0, greatest = 0;
        TB_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
        TB_CUDA(cudaStreamCreateWithPriority(&chain, cudaStreamNonBlocking, greatest));
        TB_CUDA(cudaStreamCreateWithPriority(&rest, cudaStreamNonBlocking, least));
        for (cudaEvent_t* e : {&forked, &block, &packed, &updated})
            TB_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
        return TB_OK;
    }
    void destroy() {
        for (cudaEvent_t e : {forked, block, packed, updated})
            if (e) cudaEventDestroy(e);
        if (rest) cudaStreamDestroy(rest);
        if (chain) cudaStreamDestroy(chain);
    }
};
constexpr size_t MAX_KEPT = 4;
static std::mutex g_side_mu;
static std::map<int, std::vector<SideStreams>> g_side;

class BorrowedStreams {
   public:
    int take(int device) {
        device_ = device;
        {
            std::lock_guard<std::mutex> lk(g_side_mu);
            std::vector<SideStreams>& idle = g_side[device];
            if (!idle.empty()) {
                s = idle.back();
                idle.pop_back();
                return TB_OK;
            }
        }
        return s.make();
    }
    ~BorrowedStreams() {
        if (!s.updated) {  // not taken, or not made completely
            s.destroy();
            return;
        }
        if (!joined) {  // the call gave up half way: the workspace is the caller's again
            cudaStreamSynchronize(s.chain);
            cudaStreamSynchronize(s.rest);
        }
        std::lock_guard<std::mutex> lk(g_side_mu);
        std::vector<SideStreams>& idle = g_side[device_];
        if (idle.size() < MAX_KEPT) idle.push_back(s);
        else s.destroy();
    }
    SideStreams s;
    bool joined = false;  // everything on them is waited for by the caller's stream

   private:
    int device_ = 0;
};

}  // namespace tb

extern "C" {

size_t tb_spd_inverse_workspace_bytes(int64_t k) {
    if (k <= 0) return 0;
    return tb::inv_layout(k).total;
}

int tb_spd_inverse(int device, void* stream_, float* A, int64_t k, int64_t lda, float lambda,
                   int rescale_by_mean_abs, float* mean_abs_out, void* ws, size_t ws_bytes) {
    using namespace tb;
    if (k <= 0 || lda < k || k > 0x3fffffff) return TB_ERR_BAD_SHAPE;
    if (!A) return TB_ERR_BAD_ARG;
    if (!ws || ((uintptr_t)ws & 255u) != 0 || ws_bytes < tb_spd_inverse_workspace_bytes(k)) return TB_ERR_WORKSPACE;
    int sm_count = 0;
    int rc = select_device(device, &sm_count);
    if (rc != TB_OK) return rc;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    const InvLayout l = inv_layout(k);
    uint8_t* base = static_cast<uint8_t*>(ws);
    float* dinv = reinterpret_cast<float*>(base + l.dinv);
    float* blocks = reinterpret_cast<float*>(base + l.blocks);
    double* partial = reinterpret_cast<double*>(base + l.partial);
    const int K = (int)k;

    // The block columns, the rest of their updates and the merges run on three streams where there is more than one
    // column.  A capture stays on the caller's stream: borrowed streams must not be part of a graph under construction.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    TB_CUDA(cudaStreamIsCapturing(stream, &capture));
    BorrowedStreams side;
    const bool apart = k > OUTER && capture == cudaStreamCaptureStatusNone;
    if (apart && (rc = side.take(device)) != TB_OK) return rc;
    const cudaStream_t chain = apart ? side.s.chain : stream, rest = apart ? side.s.rest : stream;
    auto record = [&](cudaEvent_t event, cudaStream_t on) -> int {
        if (apart) TB_CUDA(cudaEventRecord(event, on));
        return TB_OK;
    };
    auto wait = [&](cudaStream_t on, cudaEvent_t event) -> int {
        if (apart) TB_CUDA(cudaStreamWaitEvent(on, event, 0));
        return TB_OK;
    };

    // operands of one product at `at`, then the product itself
    auto multiply = [&](cudaStream_t on, const Product& pr, uint8_t* at, const float* a, int64_t ld_a, bool trans_a,
                        const float* b, int64_t ld_b, int64_t m, int64_t n, int64_t kk, float* c, int64_t ld_c,
                        float alpha, KRange range) -> int {
        const bool symmetric = b == nullptr;
        uint16_t* pa = reinterpret_cast<uint16_t*>(at);
        uint16_t* pb = symmetric ? pa : reinterpret_cast<uint16_t*>(at + pr.a.bytes);
        int r;
        if (!symmetric && !trans_a) {
            r = launch_pack_pair(a, m, kk, ld_a, pa, pr.a, b, n, kk, ld_b, pb, pr.b, sm_count, on);
            if (r != TB_OK) return r;
        } else {
            r = launch_pack(a, TB_F32, trans_a, (uint64_t)m, (uint64_t)kk, (uint64_t)ld_a, pa, pr.a, sm_count, on);
            if (r != TB_OK) return r;
            if (!symmetric) r = launch_pack(b, TB_F32, false, (uint64_t)n, (uint64_t)kk, (uint64_t)ld_b, pb, pr.b, sm_count, on);
            if (r != TB_OK) return r;
        }
        return launch_gemm(device, on, pa, pr.a, pb, symmetric ? pr.a : pr.b, TB_F32, m, n, c, ld_c, nullptr, alpha, 0,
                           symmetric ? 1 : 0, 1, reinterpret_cast<float*>(at + pr.a.bytes + pr.b.bytes), range);
    };

    // W21 = -W22 (L21 W11), written over L21, in two products: the first as soon as W11 is there, in transposed form
    // (T[s x s2] = W11^T . L21^T), the second when W22 is.  Then zeros in L's place above the diagonal.
    auto merge_left = [&](int64_t b0, int64_t s, int64_t s2) -> int {
        const float *W11 = A + b0 * lda + b0, *L21 = A + (b0 + s) * lda + b0;
        return multiply(stream, product(s, s2, s, false), base + l.merge, W11, lda, true, L21, lda, s, s2, s,
                        reinterpret_cast<float*>(base + l.left_at(s)), s2, 1.0f, K_FROM_ROW);
    };
    auto merge = [&](int64_t b0, int64_t s, int64_t s2) -> int {
        float *L21 = A + (b0 + s) * lda + b0, *W22 = A + (b0 + s) * lda + b0 + s;
        const int r = multiply(stream, product(s2, s, s2, false), base + l.merge, W22, lda, false,
                               reinterpret_cast<float*>(base + l.left_at(s)), s2, s2, s, s2, L21, lda, -1.0f, K_TO_ROW);
        if (r != TB_OK) return r;
        TB_CUDA(cudaMemset2DAsync(A + b0 * lda + b0 + s, (size_t)lda * sizeof(float), 0, (size_t)s2 * sizeof(float), (size_t)s,
                                  stream));
        return TB_OK;
    };

    BlockCounters* counters = reinterpret_cast<BlockCounters*>(base + l.counters);
    prepare_kernel<<<(K + 255) / 256, 256, 0, stream>>>(A, lda, K, lambda, reinterpret_cast<uint32_t*>(counters),
                                                        2 * ((K + OUTER - 1) / OUTER));
    if ((rc = record(side.s.forked, stream)) != TB_OK || (rc = wait(chain, side.s.forked)) != TB_OK) return rc;

    if (const int e = set_smem_limit((const void*)block_kernel, device)) return e;
    uint8_t* const chain_at = base + l.chain;
    for (int64_t o = 0; o < k; o += OUTER) {
        // 1. The diagonal block becomes its W.
        const int kb = (int)std::min<int64_t>(OUTER, k - o), nt = (kb + NB - 1) / NB;
        float* block = A + o * lda + o;
        int tiles = nt;  // of the first step, the largest
        for (int i = 1; i < nt; ++i) tiles += i + 1;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeCooperative;
        attr.val.cooperative = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)std::min(tiles + 1, sm_count));
        cfg.blockDim = dim3(STEP_THREADS);
        cfg.dynamicSmemBytes = STEP_SMEM;
        cfg.stream = chain;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        TB_CUDA(cudaLaunchKernelEx(&cfg, block_kernel, block, lda, kb, blocks, dinv, counters + o / OUTER,
                                   status_ptr(device)));
        if ((rc = record(side.s.block, chain)) != TB_OK || (rc = wait(stream, side.s.block)) != TB_OK) return rc;

        // 2. Below it L21; of what is right of both, first the next diagonal block, then the rest beside the chain.
        const int64_t r = k - o - kb, d = std::min<int64_t>(OUTER, r);
        if (r > 0) {
            float* A21 = A + (o + kb) * lda + o;
            float* A22 = A + (o + kb) * lda + o + kb;
            if (o > 0 && (rc = wait(chain, side.s.updated)) != TB_OK) return rc;
            rc = multiply(chain, product(r, kb, kb, false), chain_at, A21, lda, false, block, lda, r, kb, kb, A21, lda, 1.0f,
                          K_TO_COL);
            if (rc != TB_OK) return rc;
            const Packed g = packed_geometry(TB_F32, r, kb);
            const uint16_t *L = reinterpret_cast<uint16_t*>(chain_at), *tail = L;
            rc = launch_pack(A21, TB_F32, false, r, kb, lda, const_cast<uint16_t*>(L), g, sm_count, chain);
            if (rc != TB_OK) return rc;
            if ((rc = record(side.s.packed, chain)) != TB_OK || (rc = wait(rest, side.s.packed)) != TB_OK) return rc;
            rc = launch_gemm(device, chain, L, g, L, g, TB_F32, d, d, A22, lda, nullptr, -1.0f, 1, 1, 1,
                             reinterpret_cast<float*>(chain_at + g.bytes));
            if (rc != TB_OK) return rc;
            if (r > d) {
                const Packed gt = packed_tail(&tail, g, OUTER / 128);
                float* partial_sums = reinterpret_cast<float*>(base + l.rest);
                rc = launch_gemm(device, rest, tail, gt, L, g, TB_F32, r - d, d, A22 + d * lda, lda, nullptr, -1.0f, 1, 0, 1,
                                 partial_sums, K_ALL, false);
                if (rc != TB_OK) return rc;
                rc = launch_gemm(device, rest, tail, gt, tail, gt, TB_F32, r - d, r - d, A22 + d * lda + d, lda, nullptr,
                                 -1.0f, 1, 1, 1, partial_sums, K_ALL, false);
                if (rc != TB_OK) return rc;
                if ((rc = record(side.s.updated, rest)) != TB_OK) return rc;
            }
        }

        // 3. The inverted blocks so far that complete a pair, and the pairs of pairs; then the first product of the
        // pair whose left half is now complete.
        const int64_t done = o + kb;
        int64_t s = OUTER;
        for (; s < done; s *= 2) {
            if (done < k && done % (2 * s) != 0) break;
            const int64_t b0 = (done - 1) / (2 * s) * (2 * s);
            if (b0 + s < done && (rc = merge(b0, s, done - b0 - s)) != TB_OK) return rc;
        }
        if (done < k) {  // s is now the largest level that divides `done`
            if ((rc = wait(stream, side.s.packed)) != TB_OK) return rc;
            if ((rc = merge_left(done - s, s, std::min<int64_t>(s, k - done))) != TB_OK) return rc;
        }
    }
    TB_CUDA(cudaGetLastError());
    side.joined = true;  // the last block waited for the last update, the caller's stream for the last block

    // A^-1 = W^T W (full symmetric result written over A; the operand is packed first)
    rc = multiply(stream, product(k, k, k, true), base + l.merge, A, lda, true, nullptr, 0, k, k, k, A, lda, 1.0f, K_FROM_ROW);
    if (rc != TB_OK) return rc;

    // mean |entry| and the reference's rescale
    if (rescale_by_mean_abs || mean_abs_out) {
        rc = launch_after(abs_partial_kernel, RED_BLOCKS, 256, 0, stream, true, A, lda, K, partial);
        if (rc != TB_OK) return rc;
        rc = rescale_by_mean_abs ? launch_after(scale_by_inverse_kernel, std::min(K, sm_count * 8), 256, 0, stream, true, A, lda,
                                                K, partial, mean_abs_out)
                                 : launch_after(abs_final_kernel, 1, 256, 0, stream, true, partial, K, mean_abs_out);
        if (rc != TB_OK) return rc;
    }
    return TB_OK;
}

}  // extern "C"
