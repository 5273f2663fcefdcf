// Density filter (I/ApplyFilter.m:74-81 with W of I/ElemNeighborhood.m):
//   trans = 0:  y = (W x) ./ w        trans = 1:  y = W' (x ./ w) = W (x ./ w)
// W is symmetric with Gaussian/hat weights inside the radius; rows and
// columns of fixed elements are decoupled with a unit diagonal
// (I/ElemNeighborhood.m:173-179).
//
// k_filter_tiled: a CTA loads a 32 x 8 x 4 brick of the filter's inputs with
// its halo (the taps' radius) into shared memory once (v_j = x_j, x_j / w_j
// or 1, and 0 for fixed or absent neighbours) and each thread walks the tap
// list (weights and tile offsets in shared memory) over the tile for four
// outputs along z at once: every input is read from global memory about once
// per tile instead of once per tap, no branch separates the taps' loads, and
// each tap's weight and offset serve four independent sums.  The taps are summed in the same order as the
// per-element kernel, absent ones adding zero, so the results are the same.
// k_filter (one thread per element walking the tap list through L1/L2)
// serves radii whose tile would not fit in shared memory.
//
// k_filter_march does the same sums plane by plane on cubic cells, for radii of
// up to three cells: the taps are then all offsets with dx^2 + dy^2 + dz^2 <= D2,
// known when the kernel is compiled, and the weights depend on that square.
// The values of the columns (dx, dy) of equal dx^2 + dy^2 are added first, and
// their sum S over plane p adds w S to the outputs of the planes p + dz, held in
// registers while the block walks along z.  33 taps become 13 reads, 9 adds and
// 12 FMAs per element and plane (81: 21, 15 and 27), where the tile kernel
// reads every tap from shared memory.  The next plane is read while this one
// is summed.  384 x 192 x 192 cells, 33 taps: 237 -> 111 us (x, w and y once: 52);
// transposed, 480 x 240 x 120, 81 taps: 446 -> 171.
#include <algorithm>
#include <cmath>

#include "tosp_internal.h"

namespace tosp {

__global__ void k_filter(const double *__restrict__ x, double *__restrict__ y, const double *__restrict__ wsum,
                         const uint8_t *__restrict__ fixed, const FilterTap *__restrict__ taps, int ntaps, int nelx,
                         int nely, int nelz, int trans, int weights_only) {
    const int64_t n = (int64_t)nelx * nely * nelz;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int ey = (int)(i % nely), ex = (int)((i / nely) % nelx), ez = (int)(i / ((int64_t)nely * nelx));
        if (fixed && fixed[i]) {
            y[i] = weights_only ? 1.0 : (trans ? x[i] / wsum[i] : x[i]);
            continue;
        }
        double acc = 0.0;
        for (int t = 0; t < ntaps; ++t) {
            const FilterTap tp = taps[t];
            const int jx = ex + tp.dx, jy = ey + tp.dy, jz = ez + tp.dz;
            if (jx < 0 || jx >= nelx || jy < 0 || jy >= nely || jz < 0 || jz >= nelz) continue;
            const int64_t j = ((int64_t)jz * nelx + jx) * nely + jy;
            if (fixed && fixed[j]) continue;
            if (weights_only) acc += tp.w;
            else if (trans) acc += tp.w * (x[j] / wsum[j]);
            else acc += tp.w * x[j];
        }
        y[i] = (weights_only || trans) ? acc : acc / wsum[i];
    }
}

constexpr int FT_Y = 32, FT_X = 8, FT_Z = 4;   // outputs per CTA (256 threads, four along z each)

__global__ void __launch_bounds__(256)
k_filter_tiled(const double *__restrict__ x, double *__restrict__ y, const double *__restrict__ wsum,
               const uint8_t *__restrict__ fixed, const FilterTap *__restrict__ taps, int ntaps, int nelx, int nely,
               int nelz, int trans, int weights_only, int R) {
    extern __shared__ __align__(16) unsigned char ft_smem[];
    double *sw = reinterpret_cast<double *>(ft_smem);                 // tap weights
    double *tile = sw + ntaps;
    int *soff = reinterpret_cast<int *>(tile + (FT_Y + 2 * R) * (FT_X + 2 * R) * (FT_Z + 2 * R));   // tap offsets in the tile
    const int TY = FT_Y + 2 * R, TX = FT_X + 2 * R, TZ = FT_Z + 2 * R, TXY = TX * TY;
    const int y0 = blockIdx.x * FT_Y, x0 = blockIdx.y * FT_X, z0 = blockIdx.z * FT_Z;
    const int tid = threadIdx.x;
    for (int t = tid; t < ntaps; t += blockDim.x) {
        const FilterTap tp = taps[t];
        sw[t] = tp.w;
        soff[t] = tp.dz * TXY + tp.dx * TY + tp.dy;
    }
    for (int idx = tid; idx < TY * TX * TZ; idx += blockDim.x) {
        const int ty = idx % TY, tx = (idx / TY) % TX, tz = idx / TXY;
        const int gy = y0 - R + ty, gx = x0 - R + tx, gz = z0 - R + tz;
        double v = 0.0;
        if (gy >= 0 && gy < nely && gx >= 0 && gx < nelx && gz >= 0 && gz < nelz) {
            const int64_t j = ((int64_t)gz * nelx + gx) * nely + gy;
            if (!(fixed && fixed[j])) v = weights_only ? 1.0 : (trans ? x[j] / wsum[j] : x[j]);
        }
        tile[idx] = v;
    }
    __syncthreads();
    const int ly = tid % FT_Y, lx = tid / FT_Y;
    const int gy = y0 + ly, gx = x0 + lx;
    if (gy >= nely || gx >= nelx) return;
    // the four outputs along z share every tap's weight and offset
    const double *c = tile + (R * TX + (lx + R)) * TY + (ly + R);
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    for (int t = 0; t < ntaps; ++t) {
        const double w = sw[t];
        const double *ct = c + soff[t];
        a0 += w * ct[0];
        a1 += w * ct[TXY];
        a2 += w * ct[2 * TXY];
        a3 += w * ct[3 * TXY];
    }
    const double acc[FT_Z] = {a0, a1, a2, a3};
#pragma unroll
    for (int lz = 0; lz < FT_Z; ++lz) {
        const int gz = z0 + lz;
        if (gz >= nelz) break;
        const int64_t i = ((int64_t)gz * nelx + gx) * nely + gy;
        if (fixed && fixed[i]) y[i] = weights_only ? 1.0 : (trans ? x[i] / wsum[i] : x[i]);
        else y[i] = (weights_only || trans) ? acc[lz] : acc[lz] / wsum[i];
    }
}

constexpr int FM_Y = 32, FM_X = 8;   // outputs per plane (256 threads)

__host__ __device__ constexpr int isqrt(int v) {
    int r = 0;
    while ((r + 1) * (r + 1) <= v) ++r;
    return r;
}

constexpr int fm_resident(int d2) { return d2 >= 9 ? 4 : 5; }   // blocks per SM (registers)

template <int D2, bool TRANS>
__global__ void __launch_bounds__(256, fm_resident(D2))
k_filter_march(const double *__restrict__ x, double *__restrict__ y, const double *__restrict__ wsum,
               const uint8_t *__restrict__ fixed, const __grid_constant__ FilterPlan pl, int nelx, int nely, int nelz,
               int lz) {
    constexpr int R = isqrt(D2), TY = FM_Y + 2 * R, TX = FM_X + 2 * R, TP = TY * TX, NQ = (TP + 255) / 256;
    __shared__ double tile[2][TP];
    const int t = threadIdx.x;
    const int y0 = blockIdx.x * FM_Y, x0 = blockIdx.y * FM_X, z0 = blockIdx.z * lz, z1 = min(z0 + lz, nelz);
    const int64_t np = (int64_t)nelx * nely;
    // staged values of this thread: their place in a plane of the mesh (-1: outside)
    int src[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int f = t + 256 * q, gx = x0 - R + f / TY, gy = y0 - R + f % TY;
        src[q] = f < TP && gx >= 0 && gx < nelx && gy >= 0 && gy < nely ? gx * nely + gy : -1;
    }
    // (the divisions wait until the values are stored, behind this plane's sums)
    double v[NQ], w[NQ];
    auto fetch = [&](int p) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            v[q] = 0.0;
            w[q] = 1.0;
            if (src[q] < 0 || p < 0 || p >= nelz) continue;
            const int64_t j = p * np + src[q];
            if (fixed && fixed[j]) continue;
            v[q] = x[j];
            if (TRANS) w[q] = wsum[j];
        }
    };
    auto store = [&](int p) {
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            if (t + 256 * q < TP) tile[p & 1][t + 256 * q] = TRANS ? v[q] / w[q] : v[q];
    };
    const int ly = t % FM_Y, lx = t / FM_Y, gy = y0 + ly, gx = x0 + lx;
    const bool own = gy < nely && gx < nelx;
    const int64_t out = (int64_t)gx * nely + gy;
    double a[2 * R + 1];   // sums of the planes p - R .. p + R
#pragma unroll
    for (int d = 0; d <= 2 * R; ++d) a[d] = 0.0;
    fetch(z0 - R);
    store(z0 - R);
    __syncthreads();
#pragma unroll 1
    for (int p = z0 - R; p < z1 + R; ++p) {
        if (p + 1 < z1 + R) fetch(p + 1);
        const int z = p - R;                       // the plane whose sums this one completes
        const bool put = z >= z0 && own;
        const int64_t i = z * np + out;
        const double wo = !TRANS && put ? wsum[i] : 1.0;
        const double *c = &tile[p & 1][(lx + R) * TY + ly + R];
#pragma unroll
        for (int s2 = 0; s2 <= D2; ++s2) {         // columns with dx^2 + dy^2 = s2
            double s = 0.0;
            bool any = false;
#pragma unroll
            for (int dx = -R; dx <= R; ++dx)
#pragma unroll
                for (int dy = -R; dy <= R; ++dy)
                    if (dx * dx + dy * dy == s2) {
                        s = any ? s + c[dx * TY + dy] : c[dx * TY + dy];
                        any = true;
                    }
            if (!any) continue;
#pragma unroll
            for (int dz = -R; dz <= R; ++dz)
                if (s2 + dz * dz <= D2) a[R + dz] = fma(pl.w[s2 + dz * dz], s, a[R + dz]);
        }
        if (put) {
            if (fixed && fixed[i]) y[i] = TRANS ? x[i] / wsum[i] : x[i];
            else y[i] = TRANS ? a[0] : a[0] / wo;
        }
#pragma unroll
        for (int d = 0; d < 2 * R; ++d) a[d] = a[d + 1];
        a[2 * R] = 0.0;
        store(p + 1);
        __syncthreads();
    }
}

// Whether the taps are all offsets within a radius of at most three cells, with
// one weight per squared distance, and those weights.
bool filter_plan(const std::vector<FilterTap> &taps, FilterPlan &pl) {
    pl = FilterPlan();
    bool has[FilterPlan::D2MAX + 1] = {};
    for (const FilterTap &t : taps) {
        const int d2 = t.dx * t.dx + t.dy * t.dy + t.dz * t.dz;
        if (d2 > FilterPlan::D2MAX) return false;
        // (equal distances summed in another order differ in the last bit)
        if (has[d2] && std::abs(pl.w[d2] - t.w) > 1e-15 * t.w) return false;
        if (!has[d2]) pl.w[d2] = t.w;
        has[d2] = true;
        pl.d2 = std::max(pl.d2, d2);
    }
    size_t n = 0;
    for (int x = -3; x <= 3; ++x)
        for (int y = -3; y <= 3; ++y)
            for (int z = -3; z <= 3; ++z) n += x * x + y * y + z * z <= pl.d2;
    return pl.d2 > 0 && n == taps.size();
}

void launch_filter_march(const double *x, double *y, const double *wsum, const uint8_t *fixed, const FilterPlan &pl,
                         int nelx, int nely, int nelz, int trans, cudaStream_t st) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int by = (nely + FM_Y - 1) / FM_Y, bx = (nelx + FM_X - 1) / FM_X;
    // planes per block: the least of rounds x planes walked (a block of lz
    // planes walks 2 R more, and about two for its start)
    const int64_t slots = (int64_t)fm_resident(pl.d2) * std::max(sms, 1);
    int lz = nelz;
    int64_t least = INT64_MAX;
    for (int c = 1; c <= nelz; ++c) {
        const int l = (nelz + c - 1) / c;
        const int64_t rounds = ((int64_t)by * bx * ((nelz + l - 1) / l) + slots - 1) / slots;
        const int64_t cost = rounds * (l + 2 * isqrt(pl.d2) + 2);
        if (cost < least) {
            least = cost;
            lz = l;
        }
    }
    const dim3 grid((unsigned)by, (unsigned)bx, (unsigned)((nelz + lz - 1) / lz));
    auto kern = trans ? k_filter_march<9, true> : k_filter_march<9, false>;
    switch (pl.d2) {   // (seven is no sum of three squares)
        case 1: kern = trans ? k_filter_march<1, true> : k_filter_march<1, false>; break;
        case 2: kern = trans ? k_filter_march<2, true> : k_filter_march<2, false>; break;
        case 3: kern = trans ? k_filter_march<3, true> : k_filter_march<3, false>; break;
        case 4: kern = trans ? k_filter_march<4, true> : k_filter_march<4, false>; break;
        case 5: kern = trans ? k_filter_march<5, true> : k_filter_march<5, false>; break;
        case 6: kern = trans ? k_filter_march<6, true> : k_filter_march<6, false>; break;
        case 8: kern = trans ? k_filter_march<8, true> : k_filter_march<8, false>; break;
    }
    kern<<<grid, 256, 0, st>>>(x, y, wsum, fixed, pl, nelx, nely, nelz, lz);
    count_launch();
}

size_t filter_tile_bytes(int ntaps, int R) {
    return sizeof(double) * ntaps + sizeof(double) * (FT_Y + 2 * R) * (FT_X + 2 * R) * (FT_Z + 2 * R) +
           sizeof(int) * ntaps;
}

void launch_filter(const double *x, double *y, const double *wsum, const uint8_t *fixed, const FilterTap *taps_dev,
                   int ntaps, int nelx, int nely, int nelz, int trans, int weights_only, int radius, cudaStream_t st) {
    const size_t smem = radius >= 0 ? filter_tile_bytes(ntaps, radius) : 0;
    if (radius >= 0 && smem <= 160 * 1024) {
        static int attr_dev = -1;   // opt-in above 48 KB, per device
        int dev = 0;
        cudaGetDevice(&dev);
        if (attr_dev != dev) {
            cudaFuncSetAttribute(k_filter_tiled, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
            attr_dev = dev;
        }
        const dim3 grid((unsigned)((nely + FT_Y - 1) / FT_Y), (unsigned)((nelx + FT_X - 1) / FT_X),
                        (unsigned)((nelz + FT_Z - 1) / FT_Z));
        k_filter_tiled<<<grid, 256, smem, st>>>(x, y, wsum, fixed, taps_dev, ntaps, nelx, nely, nelz, trans,
                                                weights_only, radius);
        count_launch();
        return;
    }
    const int64_t n = (int64_t)nelx * nely * nelz;
    int64_t blocks = (n + 255) / 256;
    if (blocks > 16384) blocks = 16384;
    if (blocks < 1) blocks = 1;
    k_filter<<<(unsigned)blocks, 256, 0, st>>>(x, y, wsum, fixed, taps_dev, ntaps, nelx, nely, nelz, trans,
                                               weights_only); count_launch();
}

}  // namespace tosp
