// Coarsest-grid direct solve in FP64.
//
// The reference factors the coarsest Galerkin matrix once per setup with
// amd + sparse chol and applies eH = R\(R'\rH(perm)) in every cycle
// (I/SetupGMG.m:51-59, I/VCycle.m:40).  Here the coarsest matrix is assembled
// densely (fixed dofs decoupled with a unit diagonal, padded to a multiple of
// DB with identity) and inverted once per setup in place by a blocked
// symmetric sweep, so that each cycle's coarse solve is an FP64 GEMV, from L2
// when it fits (k_dense_gemv) or from half of the matrix (k_dense_symv).
#include <algorithm>
#include <vector>

#include "launch.cuh"
#include "tosp_internal.h"

namespace tosp {

constexpr int DB = DENSE_BLOCK;

__global__ void k_dense_scatter(const double *__restrict__ Ae, const uint8_t *__restrict__ fm, Grid g, double *A,
                                int64_t npad) {
    const int64_t total = g.nelem * 576;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t E = t / 576;
        const int e = (int)(t % 576), i = e / 24, j = e % 24;
        const int ey = (int)(E % g.nely), ex = (int)((E / g.nely) % g.nelx), ez = (int)(E / ((int64_t)g.nely * g.nelx));
        const int a = i / 3, ca = i % 3, b = j / 3, cb = j % 3;
        const int64_t na = ((int64_t)(ez + ((a >> 2) & 1)) * g.nx + (ex + ((a >> 1) & 1))) * g.ny + (ey + (a & 1));
        const int64_t nb = ((int64_t)(ez + ((b >> 2) & 1)) * g.nx + (ex + ((b >> 1) & 1))) * g.ny + (ey + (b & 1));
        const int64_t di = 3 * na + ca, dj = 3 * nb + cb;
        if (fm[di] && fm[dj]) atomicAdd(&A[di * npad + dj], Ae[t]);
    }
}

__global__ void k_dense_unitdiag(double *A, const uint8_t *fm, int64_t n, int64_t npad) {
    for (int64_t d = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; d < npad; d += (int64_t)gridDim.x * blockDim.x)
        if (d >= n || !fm[d]) A[d * npad + d] = 1.0;
}

void launch_dense_assemble(const double *Ae, const uint8_t *freemask, const Grid &g, double *A, int64_t npad,
                           cudaStream_t st) {
    cudaMemsetAsync(A, 0, sizeof(double) * npad * npad, st);
    k_dense_scatter<<<1024, 256, 0, st>>>(Ae, freemask, g, A, npad); count_launch();
    k_dense_unitdiag<<<64, 256, 0, st>>>(A, freemask, g.ndof, npad); count_launch();
}

// --- blocked symmetric sweep (block Gauss-Jordan) ----------------------------
// Sweeping block k of a symmetric matrix:  P = A_kk,  G_i = A_ik,
// C_i = G_i P^{-1},
//   A_ij -= C_i G_j' (i, j != k),  A_ik = C_i,  A_kk = -P^{-1}.
// After all blocks the array holds -A^{-1}, whatever their order.  Every pivot block is a Schur
// complement of the SPD matrix (a leading-block Cholesky factor exists), so no
// pivoting is needed.  Only the tiles on and below the diagonal are kept up to
// date; the last pass mirrors and negates them.
//
// Two launches per step, a block of 64 or two: the panel (G and C, stored transposed so that
// the update reads rows), and the rank-64 update by 64 x 64 tiles, whose first
// blocks take the next pivots' tiles and invert them while the others work.
// With blocks of 32, four launches each and the pivot on its own, the chain of
// small launches was the time: 1 911 dofs 3.0 -> 1.0 ms, 4 158 dofs 17 -> 4.0 ms
// one block a step and without regard to the band (see dense_sweep_inverse).
//
// The products run as FP64 matrix instructions (8 x 8 x 4): with FMAs and 4 x 4
// values per thread the shared-memory reads, four wavefronts for a 16-byte load
// whatever it broadcasts, held the update at 44 % of the FP64 rate.

// D += A B, A 8 x 4 (lane: row l / 4, column l % 4), B 4 x 8 (row l % 4, column
// l / 4), D 8 x 8 (row l / 4, columns 2 (l % 4) and the next).
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d[0]), "+d"(d[1])
        : "d"(a), "d"(b));
}

// A 64 x 64 tile of eight warps: warp w holds rows 16 (w / 2) .. + 15 and columns
// 32 (w % 2) .. + 31 as 2 x 4 blocks of 8 x 8; value (f, g, h) of thread t:
__device__ __forceinline__ int tile_row(int t, int f) { return (t >> 6) * 16 + f * 8 + ((t & 31) >> 2); }
__device__ __forceinline__ int tile_col(int t, int g) { return ((t >> 5) & 1) * 32 + g * 8 + 2 * (t & 3); }   // and + 1

// Row stride of shared k-major operands: 2 TS % 32 == 8 spreads a fragment's
// 4 x 4 half over all banks.
constexpr int TS = DB + 4;

// acc += X' Y over the first `rows` rows (a multiple of 4) of two k-major tiles.
__device__ __forceinline__ void tile_mma(const double *X, const double *Y, int rows, int t, double (&acc)[2][4][2]) {
    const int l = t & 31;
    const double *xr = X + (l & 3) * TS + (t >> 6) * 16 + (l >> 2);
    const double *yr = Y + (l & 3) * TS + ((t >> 5) & 1) * 32 + (l >> 2);
#pragma unroll 4
    for (int q = 0; q < rows; q += 4) {
        double a[2], b[4];
#pragma unroll
        for (int f = 0; f < 2; ++f) a[f] = xr[q * TS + 8 * f];
#pragma unroll
        for (int g = 0; g < 4; ++g) b[g] = yr[q * TS + 8 * g];
#pragma unroll
        for (int f = 0; f < 2; ++f)
#pragma unroll
            for (int g = 0; g < 4; ++g) mma_f64(acc[f][g], a[f], b[g]);
    }
}

__device__ __forceinline__ void dense_cp16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// P^{-1} of a tile V held by the block, swept by sub-blocks of 8: their eight
// rows R go through shared memory (by symmetry they serve as the columns), one
// warp inverts the 8 x 8 pivot in registers, and all warps apply
// V += R' (-Q R) with the inverse Q.  (A scalar sweep, with a barrier and a
// division by all threads per pivot, took 40 us; this takes 16.)
constexpr int SB = 8;
struct TileInverse {
    double R[2][SB * TS], QR[SB * TS], Q[SB][SB];   // QR: -Q R
};

// Inverse of the symmetric 8 x 8 block at R[.][p0 + .] by one warp: lane l holds
// (l / 4, 2 (l % 4)) and the element to its right.
__device__ __forceinline__ void block_inverse(const double *R, double (&Q)[SB][SB], int p0, int dof0, int *info) {
    const int l = threadIdx.x, r = l >> 2, c = 2 * (l & 3);
    double v0 = R[r * TS + p0 + c], v1 = R[r * TS + p0 + c + 1];
#pragma unroll
    for (int p = 0; p < SB; ++p) {
        const double d = __shfl_sync(0xffffffffu, (p & 1) ? v1 : v0, 4 * p + p / 2);
        const double fr = __shfl_sync(0xffffffffu, (p & 1) ? v1 : v0, (l & ~3) + p / 2);   // (r, p)
        const double c0 = __shfl_sync(0xffffffffu, v0, 4 * p + (l & 3));                   // (p, c)
        const double c1 = __shfl_sync(0xffffffffu, v1, 4 * p + (l & 3));
        if (l == 0 && !(d > 0.0)) atomicCAS(info, 0, 1 + dof0 + p0 + p);
        // (products before the reciprocal: the chain from pivot to pivot is the time)
        const double q = 1.0 / d, f0 = fr * c0, f1 = fr * c1;
        v0 = r == p ? (c == p ? -q : c0 * q) : (c == p ? fr * q : fma(-f0, q, v0));
        v1 = r == p ? (c + 1 == p ? -q : c1 * q) : (c + 1 == p ? fr * q : fma(-f1, q, v1));
    }
    Q[r][c] = -v0;
    Q[r][c + 1] = -v1;
}

__device__ __forceinline__ void tile_inverse(double (&v)[2][4][2], TileInverse &w, int t, int dof0, double *Pinv,
                                             int *info) {
    const int l = t & 31;
#pragma unroll 1
    for (int s = 0; s < DB / SB; ++s) {
        const int p0 = s * SB;
        double *R = w.R[s & 1];
        // which of this warp's 8-row and 8-column groups are the block's (as bits:
        // an index into v would put it into local memory)
        const unsigned rows = (t >> 6) == (s >> 1) ? 1u << (s & 1) : 0u;
        const unsigned cols = ((t >> 5) & 1) == (s >> 2) ? 1u << (s & 3) : 0u;
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            if (!((rows >> f) & 1u)) continue;
#pragma unroll
            for (int g = 0; g < 4; ++g)
                *reinterpret_cast<double2 *>(R + (l >> 2) * TS + tile_col(t, g)) = make_double2(v[f][g][0], v[f][g][1]);
        }
        __syncthreads();
        if (t < 32) block_inverse(R, w.Q, p0, dof0, info);
        __syncthreads();
        {
            // -Q R: warp w makes columns 8 w .. + 7
            const int c0 = (t >> 5) * 8;
            double o[2] = {0.0, 0.0};
#pragma unroll
            for (int k = 0; k < SB; k += 4)
                mma_f64(o, -w.Q[l >> 2][k + (l & 3)], R[(k + (l & 3)) * TS + c0 + (l >> 2)]);
            *reinterpret_cast<double2 *>(w.QR + (l >> 2) * TS + c0 + 2 * (l & 3)) = make_double2(o[0], o[1]);
        }
        __syncthreads();
        tile_mma(R, w.QR, SB, t, v);
        // the block's rows Q R, its columns (Q R)', the block itself -Q
#pragma unroll
        for (int f = 0; f < 2; ++f)
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = l >> 2, c = 2 * (l & 3) + h;
                    const bool pr = (rows >> f) & 1u, pc = (cols >> g) & 1u;
                    if (pr) v[f][g][h] = pc ? -w.Q[r][c] : -w.QR[r * TS + tile_col(t, g) + h];
                    else if (pc) v[f][g][h] = -w.QR[c * TS + tile_row(t, f)];
                }
    }
#pragma unroll
    for (int f = 0; f < 2; ++f)
#pragma unroll
        for (int g = 0; g < 4; ++g)
            *reinterpret_cast<double2 *>(Pinv + tile_row(t, f) * DB + tile_col(t, g)) =
                make_double2(-v[f][g][0], -v[f][g][1]);
}

// One step: np pivots k[p], the row tiles a[p] .. b[p] that each touches, and the
// next step's pivots (-1: none).  Buffers of pivot p: Gt and Ct at 2 p and 2 p + 1
// times DB npad in the work space, the pivot's inverse at p DB^2 in Pinv.
struct SweepStep {
    int np = 1, k[2] = {0, -1}, a[2] = {0, 0}, b[2] = {0, -1}, next[2] = {-1, -1};
};

__global__ void __launch_bounds__(256) k_sweep_first(const double *A, int64_t npad, const SweepStep s, double *Pinv,
                                                     int *info) {
    __shared__ __align__(16) TileInverse w;
    dep_enter();
    const int t = threadIdx.x, k = blockIdx.x ? s.k[1] : s.k[0];
    A += (int64_t)k * DB * (npad + 1);
    double v[2][4][2];
#pragma unroll
    for (int f = 0; f < 2; ++f)
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const double2 o = *reinterpret_cast<const double2 *>(A + tile_row(t, f) * npad + tile_col(t, g));
            v[f][g][0] = o.x;
            v[f][g][1] = o.y;
        }
    tile_inverse(v, w, t, k * DB, Pinv + blockIdx.x * DB * DB, info);
}

// PR rows of row tile i of block column k: Gt[q][i] = G_i', Ct[c][i] = C_i'
// (64 x npad each), and the column's new values.  Warp w makes columns 8 w .. + 7.
constexpr int PR = 16, GS = PR + 4;
constexpr int PANEL_SMEM = (DB * TS + DB * GS) * (int)sizeof(double);
__global__ void __launch_bounds__(256) k_sweep_panel(double *A, int64_t npad, const SweepStep s, const double *Pinv,
                                                     double *work) {
    extern __shared__ __align__(16) double sm[];
    dep_enter();
    double *P = sm, *G = sm + DB * TS;                    // P[q][c], G[q][r]
    const int rows0 = s.b[0] - s.a[0] + 1, row = (int)blockIdx.x / (DB / PR), p = row < rows0 ? 0 : 1, k = p ? s.k[1] : s.k[0];
    const int t = threadIdx.x, i = p == 0 ? s.a[0] + row : s.a[1] + row - rows0,
              r0 = i * DB + (int)(blockIdx.x % (DB / PR)) * PR;
    double *Gt = work + 2 * p * DB * npad, *Ct = Gt + DB * npad;
    Pinv += p * DB * DB;
    if (i == k) {
        for (int e = t; e < PR * DB; e += 256)
            A[(int64_t)(r0 + e / DB) * npad + k * DB + e % DB] = -Pinv[(r0 - k * DB) * DB + e];
        return;
    }
#pragma unroll
    for (int u = 0; u < DB * DB / 2 / 256; ++u) {
        const int e = t + 256 * u, q = e / (DB / 2), c = 2 * (e % (DB / 2));
        dense_cp16(P + q * TS + c, Pinv + q * DB + c);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    double gv[PR * DB / 256];
#pragma unroll
    for (int u = 0; u < PR * DB / 256; ++u) {
        const int e = t + 256 * u;
        gv[u] = i > k ? A[(int64_t)(r0 + e / DB) * npad + k * DB + e % DB]     // stored as (i, k)
                      : A[(int64_t)(k * DB + e / PR) * npad + r0 + e % PR];    // stored as (k, i)
    }
#pragma unroll
    for (int u = 0; u < PR * DB / 256; ++u) {
        const int e = t + 256 * u;
        if (i > k) G[(e % DB) * GS + e / DB] = gv[u];
        else G[(e / PR) * GS + e % PR] = gv[u];
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int u = 0; u < PR * DB / 256; ++u) {
        const int e = t + 256 * u, q = e / PR, rr = e % PR;
        Gt[(int64_t)q * npad + r0 + rr] = G[q * GS + rr];
    }
    // C[r][c] = sum_q G[q][r] P[q][c]
    const int l = t & 31, c0 = (t >> 5) * 8;
    double acc[2][2] = {};
#pragma unroll
    for (int q = 0; q < DB; q += 4) {
        const double b = P[(q + (l & 3)) * TS + c0 + (l >> 2)];
#pragma unroll
        for (int f = 0; f < 2; ++f) mma_f64(acc[f], G[(q + (l & 3)) * GS + 8 * f + (l >> 2)], b);
    }
    __syncthreads();
    double *T = sm;                                       // C[r][c], over P
#pragma unroll
    for (int f = 0; f < 2; ++f)
#pragma unroll
        for (int h = 0; h < 2; ++h) T[(8 * f + (l >> 2)) * (DB + 1) + c0 + 2 * (l & 3) + h] = acc[f][h];
    __syncthreads();
#pragma unroll
    for (int u = 0; u < PR * DB / 256; ++u) {
        const int e = t + 256 * u, c = e / PR, rr = e % PR;
        Ct[(int64_t)c * npad + r0 + rr] = T[rr * (DB + 1) + c];
        if (i < k) A[(int64_t)(k * DB + c) * npad + r0 + rr] = T[rr * (DB + 1) + c];
        else A[(int64_t)(r0 + e / DB) * npad + k * DB + e % DB] = T[e / DB * (DB + 1) + e % DB];
    }
}

// A_ij -= C_i G_j' for the tiles i >= j outside the pivots' rows and columns, for
// each pivot that touches both rows.  The first np blocks take the next pivots'
// tiles and invert them.
constexpr int DQ = 16;   // rows of Ct and Gt staged at a time (two stages)
__device__ __forceinline__ void tri_index(int e, int &i, int &j) {
    i = (int)((sqrt(8.0 * e + 1.0) - 1.0) * 0.5);
    while ((i + 1) * (i + 2) / 2 <= e) ++i;
    while (i * (i + 1) / 2 > e) --i;
    j = e - i * (i + 1) / 2;
}
__global__ void __launch_bounds__(256, 4) k_sweep_update(double *A, int64_t npad, const SweepStep s, const double *work,
                                                         double *Pinv, int *info) {
    __shared__ __align__(16) union {
        double st[2][2][DQ * TS];
        TileInverse w;
    } sm;
    dep_enter();
    const int t = threadIdx.x;
    int i, j;
    const bool pivot = (int)blockIdx.x < s.np;
    if (pivot) {
        i = j = blockIdx.x ? s.next[1] : s.next[0];
        if (i < 0) return;
    } else {
        const int e = (int)blockIdx.x - s.np, rows0 = s.b[0] - s.a[0] + 1, tri0 = rows0 * (rows0 + 1) / 2;
        tri_index(e < tri0 ? e : e - tri0, i, j);
        const int o = e < tri0 ? s.a[0] : s.a[1];
        i += o;
        j += o;
        if (e >= tri0 && i <= s.b[0]) return;   // (a[0] = 0: listed with the first pivot's)
        if (i == s.k[0] || j == s.k[0] || i == s.k[1] || j == s.k[1]) return;
        if (i == j && (i == s.next[0] || i == s.next[1])) return;
    }
    // the pivots that touch tile (i, j)
    const bool in0 = j >= s.a[0] && i <= s.b[0], in1 = s.np == 2 && j >= s.a[1] && i <= s.b[1];
    const int first = in0 ? 0 : 1, chunks = (in0 && in1 ? 2 : 1) * (DB / DQ);
    if (!in0 && !in1 && !pivot) return;
    auto stage = [&](int c) {
        double *X = sm.st[c & 1][0], *Y = sm.st[c & 1][1];
        const int p = c < DB / DQ ? first : 1;
        const double *Gt = work + (int64_t)2 * p * DB * npad + (int64_t)(c % (DB / DQ)) * DQ * npad, *Ct = Gt + DB * npad;
#pragma unroll
        for (int u = 0; u < DQ * DB / 2 / 256; ++u) {
            const int e = t + 256 * u, q = e / (DB / 2), col = 2 * (e % (DB / 2));
            dense_cp16(X + q * TS + col, Ct + (int64_t)q * npad + i * DB + col);
            dense_cp16(Y + q * TS + col, Gt + (int64_t)q * npad + j * DB + col);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double acc[2][4][2] = {};
    if (in0 || in1) {
        stage(0);
#pragma unroll 1
        for (int c = 0; c < chunks; ++c) {
            if (c + 1 < chunks) {
                stage(c + 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            tile_mma(sm.st[c & 1][0], sm.st[c & 1][1], DQ, t, acc);
            __syncthreads();
        }
    }
#pragma unroll
    for (int f = 0; f < 2; ++f)
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            double2 *p = reinterpret_cast<double2 *>(A + (int64_t)(i * DB + tile_row(t, f)) * npad + j * DB +
                                                     tile_col(t, g));
            double2 o = *p;
            o.x -= acc[f][g][0];
            o.y -= acc[f][g][1];
            *p = o;
            acc[f][g][0] = o.x;
            acc[f][g][1] = o.y;
        }
    if (pivot) tile_inverse(acc, sm.w, t, i * DB, Pinv + blockIdx.x * DB * DB, info);
}

// A = -(lower tiles), mirrored.
__global__ void __launch_bounds__(256) k_sweep_mirror(double *A, int64_t npad) {
    __shared__ double T[DB][DB + 1];
    dep_enter();
    const int e0 = (int)blockIdx.x, t = threadIdx.x;
    int i = (int)((sqrt(8.0 * e0 + 1.0) - 1.0) * 0.5);
    while ((i + 1) * (i + 2) / 2 <= e0) ++i;
    while (i * (i + 1) / 2 > e0) --i;
    const int j = e0 - i * (i + 1) / 2;
    for (int e = t; e < DB * DB; e += 256) {
        double *p = A + (int64_t)(i * DB + e / DB) * npad + j * DB + e % DB;
        const double v = -*p;
        T[e / DB][e % DB] = v;
        if (i != j) *p = v;
    }
    __syncthreads();
    // a diagonal tile takes its lower half on both sides
    for (int e = t; e < DB * DB; e += 256) {
        const int r = e / DB, c = e % DB;
        A[(int64_t)(j * DB + r) * npad + i * DB + c] = (i == j && c < r) ? T[r][c] : T[c][r];
    }
}

// The order of the pivots.  Entries more than `band` from the diagonal are zero on
// entry, and the Schur complements keep the band: a pivot k with all lower blocks
// swept touches the row tiles up to hi(k), one with all higher blocks swept those
// down to lo(k); the others hold zeros in column k and nothing of them changes.  So
// the sweep runs from both ends at once, two pivots a step, as long as neither
// touches the other (tiles that both touch take both updates), and then through
// what is left between, one a step, touching the lower part and, from where the
// upper part begins to couple, all.  That shortens the chain of steps, which is
// the time of small systems, and the updates, which are that of large ones: 1 911
// dofs (30 blocks, a band of 5) take 18 steps instead of 30, a whole setup 0.66 ms
// instead of 1.20; 4 158 dofs 2.1 for 4.4 ms, 8 619 dofs 6.5 for 26.8 (with the band
// alone 1.02, 3.3 and 13.6).
int dense_sweep_inverse(double *A, double *work, double *Pinv, int64_t npad, int64_t band, int *d_info,
                        cudaStream_t st) {
    const int nt = (int)(npad / DB), tiles = nt * (nt + 1) / 2;
    const int64_t bw = std::min<int64_t>(std::max<int64_t>(band, 1), npad);
    auto hi = [&](int k) { return (int)std::min<int64_t>(nt - 1, (DB * (int64_t)(k + 1) - 1 + bw) / DB); };
    auto lo = [&](int k) { return (int)(std::max<int64_t>(0, DB * (int64_t)k - bw) / DB); };
    int m = 0;   // steps of two pivots
    while (m < nt - 1 - m && hi(m) < nt - 1 - m && m < lo(nt - 1 - m)) ++m;
    std::vector<SweepStep> steps;
    for (int q = 0; q < m; ++q) {
        SweepStep s;
        s.np = 2;
        s.k[0] = q;
        s.b[0] = hi(q);
        s.k[1] = nt - 1 - q;
        s.a[1] = lo(s.k[1]);
        s.b[1] = nt - 1;
        steps.push_back(s);
    }
    for (int k = m; k < nt - m; ++k) {
        SweepStep s;
        s.k[0] = k;
        s.b[0] = k >= lo(nt - m) ? nt - 1 : hi(k);
        steps.push_back(s);
    }
    for (size_t q = 0; q + 1 < steps.size(); ++q)
        for (int p = 0; p < steps[q + 1].np; ++p) steps[q].next[p] = steps[q + 1].k[p];
    cudaFuncSetAttribute(k_sweep_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, PANEL_SMEM);
    cudaMemsetAsync(d_info, 0, sizeof(int), st);
    launch_dep(k_sweep_first, steps[0].np, 256, 0, st, A, npad, steps[0], Pinv, d_info);
    for (const SweepStep &s : steps) {
        const int r0 = s.b[0] - s.a[0] + 1, r1 = s.np == 2 ? s.b[1] - s.a[1] + 1 : 0;
        launch_dep(k_sweep_panel, (r0 + r1) * (DB / PR), 256, PANEL_SMEM, st, A, npad, s, Pinv, work);
        if (nt == 1) break;
        launch_dep(k_sweep_update, s.np + r0 * (r0 + 1) / 2 + r1 * (r1 + 1) / 2, 256, 0, st, A, npad, s, work, Pinv,
                   d_info);
    }
    launch_dep(k_sweep_mirror, tiles, 256, 0, st, A, npad);
    return 0;
}

// x = X b (X symmetric, npad x npad; only the first n entries are used).  A block
// makes GR rows at a time: lane t holds columns 2 t + 512 k of all of them, so a value
// of b serves GR, and a chunk of GK x 512 columns is in flight at once.  X is from the
// setup, which ends with a synchronisation: a grid that starts before its
// predecessor is done reads its first chunk ahead of the wait.  (Four warps a row, one
// value a lane and load, four in flight: 11 us for 1 911 dofs from memory, 2.6 TB/s.
// With the stencils' early reads 64 x 32 x 32 W 5.18 -> 4.88 ms, 96 x 48 x 48 4.16 -> 3.97,
// 192 x 96 x 96 FP64 61.0 -> 59.9.)
constexpr int GR = 2, GK = 4;
template <typename T>
__global__ void __launch_bounds__(256)
k_dense_gemv(const double *__restrict__ X, const T *b, T *x, int64_t n, int64_t npad) {
    __shared__ double part[GR][8];
    dep_start();
    const int t = threadIdx.x, w = t >> 5;
    const int64_t row = GR * (int64_t)blockIdx.x;   // (rows up to npad exist)
    double2 v[GR][GK];
    auto load = [&](int64_t c0) {
#pragma unroll
        for (int k = 0; k < GK; ++k) {
            const int64_t c = c0 + 512 * k + 2 * t;
#pragma unroll
            for (int r = 0; r < GR; ++r)
                v[r][k] = c < n ? __ldg(reinterpret_cast<const double2 *>(X + (row + r) * npad + c)) : make_double2(0.0, 0.0);
        }
    };
    load(0);
    dep_wait();
    double s[GR] = {};
    for (int64_t c0 = 0; c0 < n; c0 += 512 * GK) {
        if (c0) load(c0);
        T b0[GK], b1[GK];
#pragma unroll
        for (int k = 0; k < GK; ++k) {
            const int64_t c = c0 + 512 * k + 2 * t;
            b0[k] = c < n ? b[c] : T(0);
            b1[k] = c + 1 < n ? b[c + 1] : T(0);
        }
#pragma unroll
        for (int r = 0; r < GR; ++r)
#pragma unroll
            for (int k = 0; k < GK; ++k) s[r] += v[r][k].x * (double)b0[k] + v[r][k].y * (double)b1[k];
    }
#pragma unroll
    for (int r = 0; r < GR; ++r) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
        if ((t & 31) == 0) part[r][w] = s[r];
    }
    __syncthreads();
    if (t < GR && row + t < n) {
        double a = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) a += part[t][k];
        x[row + t] = (T)a;
    }
}

// The same from the lower tiles alone, for matrices that L2 does not keep: each is
// read once, for its own rows and, transposed, for its mirror image's.  A block
// takes up to SYM_CH tiles of a tile row: the sums of the tiles' columns go out
// by tile, those of its rows by block, and k_dense_symv_sum adds them up in a fixed
// order.  Half the bytes against a second launch and the partial sums: 4 158 dofs
// (138 MB) 17 us less of an FP64 iteration and 12 of a mixed one, 6 591 dofs 23,
// 9 126 dofs 51; 2 535 dofs (51 MB) 1 us more, 1 911 nothing.  So the line lies at half of L2.
constexpr int SYM_CH = 4;
// Partial sums (vectors of npad): 0 .. nt - 1 the column sums of tile row i, then
// the row sums of chunk c.
int64_t dense_partials(int64_t npad) { return npad / DB + (npad / DB + SYM_CH - 1) / SYM_CH; }

template <typename T>
__global__ void __launch_bounds__(256, 2) k_dense_symv(const double *X, const T *b, double *part, int64_t n, int64_t npad) {
    __shared__ double xi[DB], xj[SYM_CH][DB], cs[SYM_CH][8][DB];
    dep_enter();
    const int t = threadIdx.x, l = t & 31, w = t >> 5, nt = (int)(npad / DB);
    // tile rows SYM_CH q .. + 3 have q + 1 blocks each
    static_assert(SYM_CH == 4, "the index below");
    int q = (int)((sqrt(1.0 + 2.0 * blockIdx.x) - 1.0) * 0.5);
    while (2 * (q + 1) * (q + 2) <= (int)blockIdx.x) ++q;
    while (2 * q * (q + 1) > (int)blockIdx.x) --q;
    const int rem = (int)blockIdx.x - 2 * q * (q + 1), i = SYM_CH * q + rem / (q + 1), c = rem % (q + 1);
    const int j0 = SYM_CH * c, j1 = min(i + 1, j0 + SYM_CH);
    auto value = [&](int64_t d) { return d < n ? (double)b[d] : 0.0; };
    {
        const int jj = t / DB, r = t % DB;
        if (j0 + jj < j1) xj[jj][r] = value((int64_t)(j0 + jj) * DB + r);
        if (t < DB) xi[t] = value((int64_t)i * DB + t);
    }
    __syncthreads();
    double racc[8] = {};
#pragma unroll
    for (int jj = 0; jj < SYM_CH; ++jj) {
        if (j0 + jj >= j1) break;
        const double *p = X + ((int64_t)i * DB + 8 * w) * npad + (int64_t)(j0 + jj) * DB + 2 * l;
        double2 v[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) v[r] = *reinterpret_cast<const double2 *>(p + r * npad);
        const double b0 = xj[jj][2 * l], b1 = xj[jj][2 * l + 1];
        double c0 = 0.0, c1 = 0.0;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const double u = xi[8 * w + r];
            racc[r] += v[r].x * b0 + v[r].y * b1;
            c0 += v[r].x * u;
            c1 += v[r].y * u;
        }
        *reinterpret_cast<double2 *>(&cs[jj][w][2 * l]) = make_double2(c0, c1);
    }
    // the eight rows over the lanes: halving exchanges leave row l / 4 in lane l
#pragma unroll
    for (int h = 4; h > 0; h >>= 1) {
        const bool up = l & (4 * h);
#pragma unroll
        for (int r = 0; r < h; ++r) {
            const double keep = up ? racc[r + h] : racc[r], give = up ? racc[r] : racc[r + h];
            racc[r] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * h);
        }
    }
    racc[0] += __shfl_xor_sync(0xffffffffu, racc[0], 2);
    racc[0] += __shfl_xor_sync(0xffffffffu, racc[0], 1);
    if ((l & 3) == 0) part[(int64_t)(nt + c) * npad + (int64_t)i * DB + 8 * w + (l >> 2)] = racc[0];
    __syncthreads();
    const int jj = t / DB, r = t % DB;
    if (j0 + jj < j1 && j0 + jj != i) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) s += cs[jj][k][r];
        part[(int64_t)i * npad + (int64_t)(j0 + jj) * DB + r] = s;
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_dense_symv_sum(const double *part, T *x, int64_t n, int64_t npad) {
    __shared__ double sh[8][32];
    dep_enter();
    const int t = threadIdx.x, r = t & 31, w = t >> 5, nt = (int)(npad / DB);
    const int64_t d = (int64_t)blockIdx.x * 32 + r;
    const int k = (int)(d / DB), chunks = k / SYM_CH + 1;
    double s = 0.0;
#pragma unroll 4
    for (int q = w; q < chunks; q += 8) s += part[(int64_t)(nt + q) * npad + d];
#pragma unroll 4
    for (int q = k + 1 + w; q < nt; q += 8) s += part[(int64_t)q * npad + d];
    sh[w][r] = s;
    __syncthreads();
    if (w == 0 && d < n) {
        s = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) s += sh[q][r];
        x[d] = (T)s;
    }
}

static bool dense_symmetric(int64_t npad) { return npad * npad * (int64_t)sizeof(double) > (64 << 20); }

template <typename T>
void launch_dense_solve(const double *X, const T *b, T *x, int64_t n, int64_t npad, double *work, cudaStream_t st) {
    if (dense_symmetric(npad)) {
        const int nt = (int)(npad / DB), q = nt / SYM_CH, rest = nt % SYM_CH;   // full groups of tile rows
        launch_dep(k_dense_symv<T>, 2 * q * (q + 1) + rest * (q + 1), 256, 0, st, X, b, work, n, npad);
        launch_dep(k_dense_symv_sum<T>, (unsigned)(npad / 32), 256, 0, st, work, x, n, npad);
        return;
    }
    launch_dep(k_dense_gemv<T>, (unsigned)((n + GR - 1) / GR), 256, 0, st, X, b, x, n, npad);
}
template void launch_dense_solve<double>(const double *, const double *, double *, int64_t, int64_t, double *,
                                         cudaStream_t);
template void launch_dense_solve<float>(const double *, const float *, float *, int64_t, int64_t, double *,
                                        cudaStream_t);

}  // namespace tosp
