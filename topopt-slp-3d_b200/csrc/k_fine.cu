// Setup and sensitivity kernels of the finest level: the diagonal of K(w), the
// SIMP factors and the compliance sensitivities.  (The operator itself:
// k_fine_modal.cu.)
#include <cuda_bf16.h>

#include "tosp_internal.h"

namespace tosp {

// Diagonal of K(w): one thread per element, atomics (setup only).  Reads the
// row-major packed blocks ke[s*300 + rowmajor(i,i)].
template <int N>
__global__ void k_fine_diag(double *__restrict__ y, const double *__restrict__ w, const uint8_t *__restrict__ freemask,
                            const double *__restrict__ ke, FineGeom fg) {
    constexpr int NS = N * N * N;
    const Grid &g = fg.g;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < g.nelem;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int ey = (int)(e % g.nely), ex = (int)((e / g.nely) % g.nelx), ez = (int)(e / ((int64_t)g.nely * g.nelx));
        for (int i = 0; i < 24; ++i) {
            const int t = pair_rowmajor(i, i);
            double d = 0.0;
            for (int s = 0; s < NS; ++s) {
                const int sy = s % N, sx = (s / N) % N, sz = s / (N * N);
                d += w[((int64_t)(ez * N + sz) * fg.nelx_d + (ex * N + sx)) * fg.nely_d + (ey * N + sy)] *
                     ke[s * KE_PACK + t];
            }
            const int a = i / 3, c = i % 3;
            const int64_t node = ((int64_t)(ez + ((a >> 2) & 1)) * g.nx + (ex + ((a >> 1) & 1))) * g.ny + (ey + (a & 1));
            if (freemask[3 * node + c]) atomicAdd(&y[3 * node + c], d);
        }
    }
}

static int num_sms() {
    static int n = 0;
    if (!n) {
        int dev;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    }
    return n;
}

void launch_fine_diag(double *y, const double *w, const uint8_t *freemask, const double *ke64, const FineGeom &fg,
                      int n, cudaStream_t st) {
    int64_t blocks = (fg.g.nelem + 255) / 256;
    if (blocks > 16 * num_sms()) blocks = 16 * num_sms();
    if (blocks < 1) blocks = 1;
    if (n == 1) { k_fine_diag<1><<<(unsigned)blocks, 256, 0, st>>>(y, w, freemask, ke64, fg); count_launch(); }
    else if (n == 2) { k_fine_diag<2><<<(unsigned)blocks, 256, 0, st>>>(y, w, freemask, ke64, fg); count_launch(); }
    else { k_fine_diag<3><<<(unsigned)blocks, 256, 0, st>>>(y, w, freemask, ke64, fg); count_launch(); }
}

// ---------------------------------------------------------------------------
// SIMP factors emin + (E - emin) rho^p (I/GlobalStiffMatrix.m:49,
// I/WOK/KelemProd.m:74).  Integer p uses repeated products.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double powp(double x, double p) {
    if (p == 1.0) return x;
    if (p == 2.0) return x * x;
    if (p == 3.0) return x * x * x;
    return pow(x, p);
}

// wq (optional) receives the BF16-rounded factors widened back to FP64, so
// that the mixed V-cycle's Galerkin hierarchy matches its finest operator;
// w32 (optional) the factors rounded to FP32 (the CG's FP32 product).
__global__ void k_simp(const double *rho, double *w64, __nv_bfloat16 *wbf, double *wq, float *w32, int64_t n,
                       double p, double emin, double E) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double w = emin + (E - emin) * powp(rho[i], p);
        w64[i] = w;
        if (w32) w32[i] = (float)w;
        if (wbf) {
            const __nv_bfloat16 b = __double2bfloat16(w);
            wbf[i] = b;
            if (wq) wq[i] = (double)__bfloat162float(b);
        }
    }
}

void launch_simp(const double *rho, double *w64, __nv_bfloat16 *wbf, double *wq, float *w32, int64_t n, double p,
                 double emin, double E, cudaStream_t st) {
    int64_t blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    k_simp<<<(unsigned)blocks, 256, 0, st>>>(rho, w64, wbf, wq, w32, n, p, emin, E); count_launch();
}

// ---------------------------------------------------------------------------
// Sensitivities (I/Grad.m:24-49, mr.interp = false):
//   g0(v_s) = -p rho_s^(p-1) (E-emin) u_e' KE_s u_e  for e in freeDensG.
// One thread per displacement element; KE_s packed in shared memory.
// ---------------------------------------------------------------------------
template <int N>
__global__ void __launch_bounds__(128)
k_grad(const double *__restrict__ u, const double *__restrict__ rho, const uint8_t *__restrict__ free_elem,
       const double *__restrict__ kepack, double *__restrict__ g0, FineGeom fg, double p, double emin, double E) {
    constexpr int NS = N * N * N;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *ke = reinterpret_cast<double *>(smem_raw);
    for (int i = threadIdx.x; i < NS * KE_PACK; i += blockDim.x) ke[i] = kepack[i];
    __syncthreads();
    const Grid &g = fg.g;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < g.nelem;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int ey = (int)(e % g.nely), ex = (int)((e / g.nely) % g.nelx), ez = (int)(e / ((int64_t)g.nely * g.nelx));
        const bool fr = free_elem[e] != 0;
        double ue[24];
        if (fr) {
#pragma unroll
            for (int a = 0; a < 8; ++a) {
                const int dx = (a >> 1) & 1, dy = a & 1, dz = (a >> 2) & 1;
                const int64_t node = ((int64_t)(ez + dz) * g.nx + (ex + dx)) * g.ny + (ey + dy);
#pragma unroll
                for (int c = 0; c < 3; ++c) ue[3 * a + c] = u[3 * node + c];
            }
        }
#pragma unroll 1
        for (int s = 0; s < NS; ++s) {
            const int sy = s % N, sx = (s / N) % N, sz = s / (N * N);
            const int64_t di = ((int64_t)(ez * N + sz) * fg.nelx_d + (ex * N + sx)) * fg.nely_d + (ey * N + sy);
            double out = 0.0;
            if (fr) {
                const double *k = ke + s * KE_PACK;
                double q = 0.0;
                int t = 0;
#pragma unroll
                for (int i = 0; i < 24; ++i) {
                    double row = 0.5 * k[t++] * ue[i];
#pragma unroll
                    for (int j = i + 1; j < 24; ++j) row += k[t++] * ue[j];
                    q += row * ue[i];
                }
                q *= 2.0;
                const double xs = rho[di];
                out = -p * powp(xs, p - 1.0) * (E - emin) * q;
            }
            g0[di] = out;
        }
    }
}

void launch_grad(const double *u, const double *rho, const uint8_t *free_elem, const double *kepack, double *g0,
                 const FineGeom &fg, int n, double p, double emin, double E, cudaStream_t st) {
    const int ns = n * n * n;
    const size_t smem = sizeof(double) * ns * KE_PACK;
    int64_t blocks = (fg.g.nelem + 127) / 128;
    if (blocks > 8 * num_sms()) blocks = 8 * num_sms();
    if (blocks < 1) blocks = 1;
    if (n == 1) {
        k_grad<1><<<(unsigned)blocks, 128, smem, st>>>(u, rho, free_elem, kepack, g0, fg, p, emin, E); count_launch();
    } else if (n == 2) {
        k_grad<2><<<(unsigned)blocks, 128, smem, st>>>(u, rho, free_elem, kepack, g0, fg, p, emin, E); count_launch();
    } else {
        static bool attr = false;
        if (!attr) {
            cudaFuncSetAttribute(k_grad<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            attr = true;
        }
        k_grad<3><<<(unsigned)blocks, 128, smem, st>>>(u, rho, free_elem, kepack, g0, fg, p, emin, E); count_launch();
    }
}

}  // namespace tosp
