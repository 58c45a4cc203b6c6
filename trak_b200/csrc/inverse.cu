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

// acc[4][4] += sum_t At[t][ty*4 + i] * Bt[t][tx*4 + j]   (both tiles stored t-major)
__device__ __forceinline__ void tile_mma(const float (*At)[TS], const float (*Bt)[TS], int ty, int tx,
                                         float (&acc)[4][4]) {
#pragma unroll 8
    for (int t = 0; t < NB; ++t) {
        const float4 a = *reinterpret_cast<const float4*>(&At[t][ty * 4]);
        const float4 b = *reinterpret_cast<const float4*>(&Bt[t][tx * 4]);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
}

// dst[t][i] = src[i*ld + t] (transposed) or dst[i][t] = src[i*ld + t], zero outside rows x cols.  The first 256 threads; four
// consecutive elements of a row each where the rows are 16-byte aligned.  A warp covers eight rows x 16 columns, so
// the transposed stores meet two to a bank.
template <bool TRANS>
__device__ __forceinline__ void load_tile(Tile& dst, const float* src, int64_t ld, int rows, int cols) {
    if (threadIdx.x >= 256u) return;
    const bool vec = (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
#pragma unroll
    for (int it = 0; it < 4; ++it) {
        const int e = it * 256 + (int)threadIdx.x, warp = e >> 5, lane = e & 31;
        const int i = (warp >> 2) * 8 + (lane & 7), t = (warp & 3) * 16 + (lane >> 3) * 4;
        float v[4];
        if (vec && i < rows && t + 4 <= cols) {
            const float4 x = *reinterpret_cast<const float4*>(src + (int64_t)i * ld + t);
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = (i < rows && t + u < cols) ? src[(int64_t)i * ld + t + u] : 0.0f;
        }
        if (TRANS) {
#pragma unroll
            for (int u = 0; u < 4; ++u) dst[t + u][i] = v[u];
        } else {
            *reinterpret_cast<float4*>(&dst[i][t]) = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
}

// A += lambda I, and zero for the counters that the block columns' CTAs meet at.
__global__ void prepare_kernel(float* A, int64_t lda, int k, float lambda, uint32_t* counters, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < k && lambda != 0.0f) A[(int64_t)i * lda + i] += lambda;
    if (i < n) counters[i] = 0;
}

// Factors the jb x jb diagonal tile S = L L^T (lower triangle used) and inverts L in the same sweep (forward
// elimination of [L | I]); writes inv(L) (lower, zero above, zero-padded to 64 x 64) to dinv.  STEP_THREADS threads:
// 256 as a 16 x 16 grid of 4 x 4 pieces in registers, and one more warp, the pivot warp, whose lane l keeps the
// diagonal piece (l, l).  The tile is walked four columns at a time, piece column q in step q.  Thread (ty, tx) holds
// a piece of S until step tx and a piece of W = inv(L) from then on (it is zero, or the identity, until its column has
// been reached), so a step is one rank-four update whichever it is:
//   1. the pivot warp has factored the diagonal piece q, D = Ld Ld^T, and published Ld;
//   2. the threads of piece column q turn their pieces into rows of L (B Ld^-T), those of piece row q apply Ld^-1 to
//      their four rows of W, which makes them final; both publish, one vector per column respectively row of q;
//   3. the threads below update their pieces, S -= L_q L_q^T and W -= L_q W_q.
// Beside 2 and 3 the pivot warp applies L_{q-1} to the diagonal pieces, computes the one piece of L_q that the next
// one needs from what its owner published, updates it and factors it: the chain of four reciprocal square roots is
// off the other warps' path.  (With S and W pieces updated one after the other in every thread, and the next piece
// factored after its update by the grid's own diagonal thread, a tile took 9 us.)
// Rows and columns beyond jb are an identity block.  `buf` is CHOL_FLOATS floats of shared memory outside S.
constexpr int CHOL_FLOATS = 64 + 3 * 256;
static_assert(CHOL_FLOATS <= NB * TS, "a tile's worth of shared memory holds chol_block's buffers");
constexpr int STEP_THREADS = 288;
struct __align__(16) Chol4 {
    float l10, l20, l30, l21, l31, l32;  // strictly lower part of Ld
    float r0, r1, r2, r3;                // reciprocals of its diagonal
    float ok, pad;
};
// 1 / sqrt(d) for a normal d; a subnormal one counts as not positive (the inverse would overflow)
__device__ __forceinline__ float rsqrt_newton(float d) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return fmaf(r, fmaf(-(0.5f * d) * r, r, 0.5f), r);
}
__device__ __forceinline__ Chol4 chol4(const float (&D)[4][4]) {  // lower part used
    Chol4 c;
    float p = D[0][0];
    bool ok = p >= 1.17549435e-38f;
    c.r0 = rsqrt_newton(p);
    c.l10 = D[1][0] * c.r0;
    c.l20 = D[2][0] * c.r0;
    c.l30 = D[3][0] * c.r0;
    p = fmaf(-c.l10, c.l10, D[1][1]);
    ok = ok && p >= 1.17549435e-38f;
    c.r1 = rsqrt_newton(p);
    c.l21 = fmaf(-c.l20, c.l10, D[2][1]) * c.r1;
    c.l31 = fmaf(-c.l30, c.l10, D[3][1]) * c.r1;
    p = fmaf(-c.l21, c.l21, fmaf(-c.l20, c.l20, D[2][2]));
    ok = ok && p >= 1.17549435e-38f;
    c.r2 = rsqrt_newton(p);
    c.l32 = fmaf(-c.l31, c.l21, fmaf(-c.l30, c.l20, D[3][2])) * c.r2;
    p = fmaf(-c.l32, c.l32, fmaf(-c.l31, c.l31, fmaf(-c.l30, c.l30, D[3][3])));
    ok = ok && p >= 1.17549435e-38f;
    c.r3 = rsqrt_newton(p);
    c.ok = ok ? 1.0f : 0.0f;
    c.pad = 0.0f;
    return c;
}
// x <- Ld^-1 x for one column of four values (forward substitution)
__device__ __forceinline__ void solve4(const Chol4& c, float& x0, float& x1, float& x2, float& x3) {
    x0 = x0 * c.r0;
    x1 = fmaf(-c.l10, x0, x1) * c.r1;
    x2 = fmaf(-c.l21, x1, fmaf(-c.l20, x0, x2)) * c.r2;
    x3 = fmaf(-c.l32, x2, fmaf(-c.l31, x1, fmaf(-c.l30, x0, x3))) * c.r3;
}
__device__ __forceinline__ float4 row4(const float (&m)[4][4], int a) { return make_float4(m[a][0], m[a][1], m[a][2], m[a][3]); }
__device__ __forceinline__ Chol4 load_factor(const Chol4* factor) {
    const float4* f = reinterpret_cast<const float4*>(factor);
    const float4 f0 = f[0], f1 = f[1], f2 = f[2];
    return Chol4{f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w, f2.x, f2.y, f2.z, 0.0f};
}
__device__ void chol_block(const Tile& S, int jb, float* dinv, uint32_t* status, float* buf) {
    const int tid = threadIdx.x;
    Chol4* factor = reinterpret_cast<Chol4*>(buf);                         // [2]: of pieces q and q + 1
    float4* raw = reinterpret_cast<float4*>(buf + 32);                     // [2][4]: piece (q + 1, q) of S before step q
    float (*colbufs)[NB] = reinterpret_cast<float(*)[NB]>(buf + 64);       // [2][4][64]: columns of L_q and L_{q-1}
    float (*rowbuf)[NB] = reinterpret_cast<float(*)[NB]>(buf + 64 + 512);  // [4][64]: rows of W_q
    static_assert(sizeof(Chol4) <= 16 * sizeof(float), "two factors fit in front of raw");
    const bool pivot = tid >= 256;
    // the pivot warp's lane l stands at (l, l); lanes 16 to 31 repeat lane 15 and publish nothing
    const int ty = pivot ? min(tid - 256, 15) : tid >> 4, tx = pivot ? ty : tid & 15;
    float x[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int i = ty * 4 + a, j = tx * 4 + b;
            const float unit = i == j ? 1.0f : 0.0f;
            // the grid's diagonal threads have no piece of S to keep (the pivot warp has): they start with W's identity
            x[a][b] = (i < jb && j < jb && j <= i && (pivot || tx != ty)) ? S[i][j] : unit;
        }
    const int steps = (jb + 3) >> 2;
    bool bad = false;
    if (tid == 256) {
        const Chol4 c = chol4(x);
        bad = c.ok == 0.0f;
        factor[0] = c;
    }
    if (!pivot && ty == 1 && tx == 0) {
#pragma unroll
        for (int a = 0; a < 4; ++a) raw[a] = row4(x, a);
    }
    // x -= L[ty] . O[tx] with four columns of L and of O
    auto update = [&](const float (*lcol)[NB], const float (*ocol)[NB]) {
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
            const float4 l = *reinterpret_cast<const float4*>(&lcol[cc][ty * 4]);
            const float4 o = *reinterpret_cast<const float4*>(&ocol[cc][tx * 4]);
            const float lv[4] = {l.x, l.y, l.z, l.w}, ov[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) x[a][b] = fmaf(-lv[a], ov[b], x[a][b]);
        }
    };
    for (int q = 0; q < steps; ++q) {
        __syncthreads();
        float (*colbuf)[NB] = colbufs + 4 * (q & 1);
        if (pivot) {
            if (q + 1 < steps) {  // every lane computes lane q + 1's part; that lane keeps it
                const Chol4 c = load_factor(factor + (q & 1));
                const float (*before)[NB] = colbufs + 4 * ((q & 1) ^ 1);
                float l[4][4], z[4][4];
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    const float4 v = raw[4 * (q & 1) + a];
                    l[a][0] = v.x; l[a][1] = v.y; l[a][2] = v.z; l[a][3] = v.w;
                    solve4(c, l[a][0], l[a][1], l[a][2], l[a][3]);
                }
                if (q > 0) update(before, before);
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int b = 0; b <= a; ++b)
                        z[a][b] = fmaf(-l[a][3], l[b][3], fmaf(-l[a][2], l[b][2], fmaf(-l[a][1], l[b][1],
                                       fmaf(-l[a][0], l[b][0], x[a][b]))));
                const Chol4 n = chol4(z);
                if (tid - 256 == q + 1) {
                    bad = bad || n.ok == 0.0f;
                    factor[(q + 1) & 1] = n;
                }
            }
            continue;
        }
        if ((tx == q && ty > q) || (ty == q && tx <= q)) {
            // rows of L: B Ld^-T, i.e. Ld^-1 applied along each row of the piece; rows of W: along each column
            const Chol4 c = load_factor(factor + (q & 1));
            const bool of_l = ty > q;
            float y[4][4];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) y[a][b] = of_l ? x[a][b] : x[b][a];
#pragma unroll
            for (int a = 0; a < 4; ++a) solve4(c, y[a][0], y[a][1], y[a][2], y[a][3]);
            float (*dst)[NB] = of_l ? colbuf : rowbuf;
            const int at = of_l ? ty * 4 : tx * 4;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                *reinterpret_cast<float4*>(&dst[b][at]) = make_float4(y[0][b], y[1][b], y[2][b], y[3][b]);
#pragma unroll
                for (int a = 0; a < 4; ++a) x[b][a] = of_l ? 0.0f : y[a][b];  // a piece of W (zero so far) from here on
            }
        }
        asm volatile("barrier.cta.sync 1, 256;" ::: "memory");  // the grid only
        if (ty > q && tx < ty) {
            update(colbuf, tx > q ? colbuf : rowbuf);
            if (ty == q + 2 && tx == q + 1) {
#pragma unroll
                for (int a = 0; a < 4; ++a) raw[4 * ((q + 1) & 1) + a] = row4(x, a);
            }
        }
    }
    if (!pivot) {
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int i = ty * 4 + a;
            float w[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) w[b] = (i < jb && tx * 4 + b <= i) ? x[a][b] : 0.0f;
            *reinterpret_cast<float4*>(dinv + i * NB + tx * 4) = make_float4(w[0], w[1], w[2], w[3]);
        }
    }
    if (bad) atomicCAS(status, 0u, (uint32_t)ST_NOT_SPD);
}

// Step j of a block column's diagonal block (kb x kb, kb <= 512), in tiles of 64.  Before the step, rows i >= j hold
// R[i, c] for c < j (what is left of the identity's elimination, W's future rows) and S[i, l] for l >= j (what is
// left of A), and D = inv(chol(S[j, j])) is known.  The step makes row j of W final,
//     W[j, c] = D R[j, c],   W[j, j] = D,
// and with P_i = S[i, j] D^T (the rows of L) updates every row i > j:
//     S[i, l] -= P_i P_l^T (j < l <= i),   R[i, c] -= P_i W[j, c] (c < j),   R[i, j] = -P_i D.
// One CTA per tile, each computing the P and W tiles it needs itself (three 64^3 products, 1.1 us each on one SM,
// instead of another meeting point and a trip through memory).  Rows i > j go from X to Y (tiles are read by many
// CTAs, so they are not updated in place); W's rows go to `block`, the matrix itself, with zeros right of the diagonal.
__device__ void block_tile(float* step_smem, const float* X, int64_t ldx, float* Y, int64_t ldy, float* block,
                           int64_t lda, int kb, int j, int i, int c, const float* D, float* D_next, uint32_t* status) {
    Tile& Dt = *reinterpret_cast<Tile*>(step_smem);                // Dt[t][c] = D[c][t]
    Tile& T0 = *reinterpret_cast<Tile*>(step_smem + NB * TS);
    Tile& T1 = *reinterpret_cast<Tile*>(step_smem + 2 * NB * TS);
    Tile& T2 = *reinterpret_cast<Tile*>(step_smem + 3 * NB * TS);
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const bool grid16 = tid < 256;  // the ninth warp is the factorisation's pivot warp
    const int rows = min(NB, kb - i * NB), jw = min(NB, kb - j * NB), cols = min(NB, kb - c * NB);
    float acc[4][4] = {};
    if (i == j) {  // row j of W
        if (c < j) {
            load_tile<true>(Dt, D, NB, NB, NB);
            load_tile<false>(T0, X + (int64_t)j * NB * ldx + c * NB, ldx, rows, NB);
            __syncthreads();
            if (grid16) tile_mma(Dt, T0, ty, tx, acc);
        }
        if (!grid16) return;
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int r = ty * 4 + a, q = tx * 4 + b;
                if (r < rows && q < cols)
                    block[(int64_t)(j * NB + r) * lda + c * NB + q] = c < j ? acc[a][b] : c == j ? D[r * NB + q] : 0.0f;
            }
        return;
    }
    // P_i, t-major, into T0
    load_tile<true>(Dt, D, NB, NB, NB);
    load_tile<true>(T1, X + (int64_t)i * NB * ldx + j * NB, ldx, rows, jw);
    if (c > j && c != i)
        load_tile<true>(T2, X + (int64_t)c * NB * ldx + j * NB, ldx, cols, jw);
    else if (c < j)
        load_tile<false>(T2, X + (int64_t)j * NB * ldx + c * NB, ldx, jw, NB);
    else if (c == j)
        load_tile<false>(T2, D, NB, NB, NB);
    // this CTA's own tile, in flight during the products
    float own[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int r = ty * 4 + a, q = tx * 4 + b;
            own[a][b] = (grid16 && c != j && r < rows && q < cols) ? X[(int64_t)(i * NB + r) * ldx + c * NB + q] : 0.0f;
        }
    __syncthreads();
    if (grid16) {
        tile_mma(T1, Dt, ty, tx, acc);
#pragma unroll
        for (int b = 0; b < 4; ++b)
            *reinterpret_cast<float4*>(&T0[tx * 4 + b][ty * 4]) = make_float4(acc[0][b], acc[1][b], acc[2][b], acc[3][b]);
    }
    if (c != i && c != j) {  // the other operand: P_c (t-major) or W[j, c], over T1
        float other[4][4] = {};
        if (!grid16) {
        } else if (c > j)
            tile_mma(T2, Dt, ty, tx, other);
        else
            tile_mma(Dt, T2, ty, tx, other);
        __syncthreads();
#pragma unroll
        for (int b = 0; b < 4 && grid16; ++b) {
            if (c > j)
                *reinterpret_cast<float4*>(&T1[tx * 4 + b][ty * 4]) =
                    make_float4(other[0][b], other[1][b], other[2][b], other[3][b]);
            else
                *reinterpret_cast<float4*>(&T1[ty * 4 + b][tx * 4]) =
                    make_float4(other[b][0], other[b][1], other[b][2], other[b][3]);
        }
    }
    __syncthreads();
    if (grid16) {
        float upd[4][4] = {};
        tile_mma(T0, c == i ? T0 : c == j ? T2 : T1, ty, tx, upd);
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int r = ty * 4 + a, q = tx * 4 + b;
                own[a][b] -= upd[a][b];
                if (r < rows && q < cols) Y[(int64_t)(i * NB + r) * ldy + c * NB + q] = own[a][b];
            }
    }
    if (D_next) {
        if (grid16) {
#pragma unroll
            for (int a = 0; a < 4; ++a)
                *reinterpret_cast<float4*>(&Dt[ty * 4 + a][tx * 4]) =
                    make_float4(own[a][0], own[a][1], own[a][2], own[a][3]);
        }
        __syncthreads();
        chol_block(Dt, rows, D_next, status, &T1[0][0]);
    }
}

// All CTAs of a cooperative launch meet: true when they have all arrived `round` times (1, 2, ...).  Bounded.
__device__ bool meet(uint32_t* counter, uint32_t round, uint32_t* status) {
    __shared__ uint32_t met;
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t target = round * gridDim.x;
        uint32_t seen;
        __threadfence();
        atomicAdd(counter, 1u);
        const uint64_t t0 = globaltimer_ns();
        bool late = false;
        for (uint32_t n = 1;; ++n) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
            if (seen >= target) break;
            if ((n & 255u) == 0 && globaltimer_ns() - t0 > WAIT_LIMIT_NS) {
                late = true;
                break;
            }
        }
        __threadfence();
        if (late && atomicCAS(status, 0u, (uint32_t)ST_TIMEOUT_ACC) == 0u) status[1] = blockIdx.x;
        met = late ? 0u : 1u;
    }
    __syncthreads();
    return met != 0;
}

// Factors and inverts a diagonal block (kb x kb): CTA 0 takes the first tile and then every step's next diagonal tile,
// the others share the rest.  A cooperative launch of about as many CTAs as the largest step has tiles; meeting through
// a counter in the L2 between steps instead of one launch per step took the 512-wide block from 155 to 125 us.
__global__ void __launch_bounds__(STEP_THREADS) block_kernel(float* block, int64_t lda, int kb, float* blocks, float* dinv,
                                                             uint32_t* counter, uint32_t* status) {
    extern __shared__ __align__(16) float step_smem[];
    const int nt = (kb + NB - 1) / NB;
    if (blockIdx.x == 0) {
        Tile& S = *reinterpret_cast<Tile*>(step_smem);
        load_tile<false>(S, block, lda, min(NB, kb), min(NB, kb));
        __syncthreads();
        chol_block(S, min(NB, kb), dinv, status, step_smem + NB * TS);
    }
    for (int j = 0; j < nt; ++j) {
        if (!meet(counter, j + 1, status)) return;
        const float* X = j == 0 ? block : blocks + (size_t)((j - 1) & 1) * OUTER * OUTER;
        float* Y = blocks + (size_t)(j & 1) * OUTER * OUTER;
        const int64_t ldx = j == 0 ? lda : OUTER;
        const float* D = dinv + (size_t)j * NB * NB;
        if (blockIdx.x == 0) {
            if (j + 1 < nt)
                block_tile(step_smem, X, ldx, Y, OUTER, block, lda, kb, j, j + 1, j + 1, D,
                           dinv + (size_t)(j + 1) * NB * NB, status);
            continue;
        }
        int tiles = nt;  // row j of W, and the tiles (i, c), c <= i, of the rows below
        for (int i = j + 1; i < nt; ++i) tiles += i + 1;
        for (int t = (int)blockIdx.x - 1; t < tiles; t += (int)gridDim.x - 1) {
            int i = j, c = t;
            if (t >= nt) {
                c = t - nt;
                for (i = j + 1; c > i; ++i) c -= i + 1;
                if (i == j + 1 && c == j + 1) continue;  // CTA 0's
            }
            block_tile(step_smem, X, ldx, Y, OUTER, block, lda, kb, j, i, c, D, nullptr, status);
            __syncthreads();
        }
    }
}

// The three whole-matrix passes below walk rows per CTA and columns per thread (no index division), four
// columns at a time where the rows are 16-byte aligned.
__device__ __forceinline__ bool rows_are_vec4(const float* A, int64_t lda, int k) {
    return (k & 3) == 0 && (lda & 3) == 0 && (reinterpret_cast<uintptr_t>(A) & 15u) == 0;
}

constexpr int RED_BLOCKS = 1024;
__global__ void __launch_bounds__(256) abs_partial_kernel(const float* A, int64_t lda, int k, double* partial) {
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
    const float mean = mean_abs(partial, k);
    if (threadIdx.x == 0) *mean_out = mean;
}
// Every CTA sums the 8 KB of partial sums itself (about 1 us) instead of waiting for a launch that does.
__global__ void __launch_bounds__(256) scale_by_inverse_kernel(float* A, int64_t lda, int k, const double* partial,
                                                               float* mean_out) {
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
    off += align_up((size_t)((k + OUTER - 1) / OUTER) * sizeof(uint32_t), 256);
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

    uint32_t* counters = reinterpret_cast<uint32_t*>(base + l.counters);
    prepare_kernel<<<(K + 255) / 256, 256, 0, stream>>>(A, lda, K, lambda, counters, (K + OUTER - 1) / OUTER);
    if ((rc = record(side.s.forked, stream)) != TB_OK || (rc = wait(chain, side.s.forked)) != TB_OK) return rc;

    constexpr size_t step_smem = 4u * NB * TS * sizeof(float);
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
        cfg.dynamicSmemBytes = step_smem;
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
                                 partial_sums);
                if (rc != TB_OK) return rc;
                rc = launch_gemm(device, rest, tail, gt, tail, gt, TB_F32, r - d, r - d, A22 + d * lda + d, lda, nullptr,
                                 -1.0f, 1, 1, 1, partial_sums);
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
        abs_partial_kernel<<<RED_BLOCKS, 256, 0, stream>>>(A, lda, K, partial);
        if (rescale_by_mean_abs)
            scale_by_inverse_kernel<<<std::min(K, sm_count * 8), 256, 0, stream>>>(A, lda, K, partial, mean_abs_out);
        else
            abs_final_kernel<<<1, 256, 0, stream>>>(partial, K, mean_abs_out);
    }
    TB_CUDA(cudaGetLastError());
    return TB_OK;
}

}  // extern "C"
