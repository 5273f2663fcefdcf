// Coarse operators from the moments of the SIMP factors.
//
// The spaces of the grids are nested: a coarse element's trilinear functions are
// trilinear on each of its children, so the Galerkin matrix P'AP
// (I/SetupGMG.m:45-49) is the stiffness matrix of the coarse element with the
// same cell-wise factors, and in modal form (fine_modal.cuh) that takes the 27
// moments of the factors over the element, which are sums of the children's.
// This holds where P, restricted to the free rows and columns
// (I/Prolongation.m:53-55), drops nothing: when every parent of a fixed dof is
// fixed (moments_clean), as for supports on whole faces, edges or coarse nodes.
// Other supports build the coarse operators with the masked triple products of
// k_coarse.cu.
//
// A level then needs 27 values per element where the half-stored stencil has 126
// per node, and no element matrices: large levels apply the modal product,
// small ones (and the coarsest) get their element matrices column by column.
#include "fine_modal.cuh"
#include "tosp_internal.h"

namespace tosp {

// Moments here are means: per direction (1/2) int {1, sqrt(3) xi, 3 xi^2} w dxi, so
// that modal_coef(..., 1) applies on every level.
namespace {

constexpr double SQ3 = 1.73205080756887729353;

// C += the child's moments G seen from its parent; s: the child's side, -1 or 1
// per direction.  With xi = (eta + s) / 2:  {a, b, c} -> {a / 2, (b + s sqrt(3) a) / 4,
// (c + 2 sqrt(3) s b + 3 a) / 8}.
__device__ __forceinline__ void add_child(double (&G)[27], const double (&s)[3], double (&C)[27]) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int st = d == 0 ? 1 : (d == 1 ? 3 : 9);
        const double r = s[d] * SQ3;
#pragma unroll
        for (int q = 0; q < 27; ++q)
            if (q / st % 3 == 0) {
                const double a = G[q], b = G[q + st], c = G[q + 2 * st];
                G[q] = 0.5 * a;
                G[q + st] = 0.25 * fma(r, a, b);
                G[q + 2 * st] = 0.125 * fma(3.0, a, fma(2.0 * r, b, c));
            }
    }
#pragma unroll
    for (int q = 0; q < 27; ++q) C[q] += G[q];
}

__device__ __forceinline__ void elem_xyz(int64_t E, const Grid &g, int &x, int &y, int &z) {
    const int64_t q = E / g.nely;
    y = (int)(E - q * g.nely);
    z = (int)(q / g.nelx);
    x = (int)(q - (int64_t)z * g.nelx);
}

// The N^3 factors of element (x, y, z) as moments W of fine_modal.cuh.
template <int N>
__device__ __forceinline__ void cell_moments(const double *__restrict__ w, int nelx_d, int nely_d, int x, int y, int z,
                                             double (&W)[modal_moments<N>]) {
    double v[N * N * N];
#pragma unroll
    for (int s = 0; s < N * N * N; ++s)
        v[s] = w[((int64_t)(z * N + s / (N * N)) * nelx_d + (x * N + s / N % N)) * nely_d + (y * N + s % N)];
    modal_weights<N, double>(v, W);
}

}  // namespace

// Level-1 moments from the density cells.
template <int N>
__global__ void __launch_bounds__(128)
k_moments_fine(const double *__restrict__ w, int nelx_d, int nely_d, Grid gc, double *__restrict__ mom) {
    for (int64_t E = blockIdx.x * 128ll + threadIdx.x; E < gc.nelem; E += gridDim.x * 128ll) {
        int x, y, z;
        elem_xyz(E, gc, x, y, z);
        double C[27];
#pragma unroll
        for (int q = 0; q < 27; ++q) C[q] = 0.0;
#pragma unroll 1
        for (int c = 0; c < 8; ++c) {
            double W[modal_moments<N>], G[27];
            cell_moments<N>(w, nelx_d, nely_d, 2 * x + ((c >> 1) & 1), 2 * y + (c & 1), 2 * z + (c >> 2), W);
#pragma unroll
            for (int q = 0; q < 27; ++q) {
                // index by degree; n = 1, 2: by the parity of the degree
                const int tx = q % 3, ty = q / 3 % 3, tz = q / 9, par = (tx & 1) | ((ty & 1) << 1) | ((tz & 1) << 2);
                if (N == 3) G[q] = W[N == 3 ? q : 0] * (1.0 / 27.0);
                else if (N == 2) G[q] = W[N == 2 ? par : 0] * 0.125;
                else G[q] = par ? 0.0 : W[0];
            }
            const double s[3] = {(c & 2) ? 1.0 : -1.0, (c & 1) ? 1.0 : -1.0, (c & 4) ? 1.0 : -1.0};
            add_child(G, s, C);
        }
#pragma unroll
        for (int q = 0; q < 27; ++q) mom[q * gc.nelem + E] = C[q];
    }
}

// Moments of a level from the finer one's.
__global__ void __launch_bounds__(128) k_moments_coarse(const double *__restrict__ mf, Grid gf, Grid gc, double *__restrict__ mom) {
    for (int64_t E = blockIdx.x * 128ll + threadIdx.x; E < gc.nelem; E += gridDim.x * 128ll) {
        int x, y, z;
        elem_xyz(E, gc, x, y, z);
        double C[27];
#pragma unroll
        for (int q = 0; q < 27; ++q) C[q] = 0.0;
#pragma unroll 1
        for (int c = 0; c < 8; ++c) {
            const int64_t e = ((int64_t)(2 * z + (c >> 2)) * gf.nelx + (2 * x + ((c >> 1) & 1))) * gf.nely + 2 * y + (c & 1);
            double G[27];
#pragma unroll
            for (int q = 0; q < 27; ++q) G[q] = mf[q * gf.nelem + e];
            const double s[3] = {(c & 2) ? 1.0 : -1.0, (c & 1) ? 1.0 : -1.0, (c & 4) ? 1.0 : -1.0};
            add_child(G, s, C);
        }
#pragma unroll
        for (int q = 0; q < 27; ++q) mom[q * gc.nelem + E] = C[q];
    }
}

// Diagonal of the operator, added into diag (zeroed by the caller): cells
// (N = 1, 2, 3) or moments (N = 0).  A node's values of the elements below and
// above it along y are added in the warp first where both are in it.
template <int N>
__global__ void __launch_bounds__(128)
k_modal_diag(const double *__restrict__ w, int nelx_d, int nely_d, Grid g, const ModalCoef<double> k,
             const uint8_t *__restrict__ fm, double *diag) {
    const int64_t E = blockIdx.x * 128ll + threadIdx.x;
    const bool in = E < g.nelem;
    int x = 0, y = 0, z = 0;
    elem_xyz(in ? E : 0, g, x, y, z);
    double D[8][3];
    if (in) {
        double W[modal_moments<N>];
        if constexpr (N == 0) {
#pragma unroll
            for (int q = 0; q < 27; ++q) W[q] = w[q * g.nelem + E];
        } else {
            cell_moments<N>(w, nelx_d, nely_d, x, y, z, W);
        }
        modal_diagonal<N, double>(W, k, D);
    } else {
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int c = 0; c < 3; ++c) D[a][c] = 0.0;
    }
    // the upper corners of the element below (lane - 1) are this one's lower ones
    const int lane = threadIdx.x & 31;
    const bool below = in && lane > 0 && y > 0;
    const bool given = in && lane < 31 && y + 1 < g.nely;   // (the element above is then in the warp)
#pragma unroll
    for (int a = 0; a < 8; a += 2)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double up = __shfl_up_sync(0xffffffffu, D[a + 1][c], 1);
            if (below) D[a][c] += up;
        }
    if (!in) return;
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        if ((a & 1) && given && E + 1 < g.nelem) continue;
        const int64_t n = 3 * (((int64_t)(z + (a >> 2)) * g.nx + x + ((a >> 1) & 1)) * g.ny + y + (a & 1));
#pragma unroll
        for (int c = 0; c < 3; ++c)
            if (fm[n + c]) atomicAdd(&diag[n + c], D[a][c]);
    }
}

// Element matrices (24 x 24, row-major) from the moments: a thread applies the
// modal product to one unit vector.
constexpr int EM_ELEMS = 8;
__global__ void __launch_bounds__(24 * EM_ELEMS)
k_elem_matrix(const double *__restrict__ mom, int64_t nelem, const ModalCoef<double> k, double *__restrict__ Ae) {
    const int j = threadIdx.x % 24, node = j / 3, comp = j % 3;
    const int64_t E = (int64_t)blockIdx.x * EM_ELEMS + threadIdx.x / 24;
    if (E >= nelem) return;
    double W[27], m[3][8], r[3][8];
#pragma unroll
    for (int q = 0; q < 27; ++q) W[q] = mom[q * nelem + E];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double u[8];
#pragma unroll
        for (int a = 0; a < 8; ++a) u[a] = a == node && c == comp ? 1.0 : 0.0;
        element_modes<double>(plane_modes<double>(u[0], u[1], u[2], u[3]), plane_modes<double>(u[4], u[5], u[6], u[7]), m[c]);
    }
    modal_stress<0, double>(m, W, k, r);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double f[8];
        f[0] = 0.0;
#pragma unroll
        for (int p = 1; p < 8; ++p)
            f[p] = modal_deg(p) == 1 ? r[c][p] : (modal_deg(p) == 2 ? MODAL_R3 * r[c][p] : (1.0 / 3.0) * r[c][p]);
#pragma unroll
        for (int bit = 1; bit < 8; bit <<= 1)
#pragma unroll
            for (int b = 0; b < 8; ++b)
                if (!(b & bit)) {
                    const double e = f[b], o = f[b | bit];
                    f[b] = e - o;
                    f[b | bit] = e + o;
                }
#pragma unroll
        for (int a = 0; a < 8; ++a)
            Ae[E * 576 + (3 * a + c) * 24 + j] = f[((a >> 1) & 1) | ((a & 1) << 1) | (a & 4)];
    }
}

// bad |= 1 when a fixed dof of the fine grid has a free parent.
__global__ void k_clean(const uint8_t *__restrict__ fmf, const uint8_t *__restrict__ fmc, Grid gf, Grid gc, int *bad) {
    for (int64_t d = blockIdx.x * 256ll + threadIdx.x; d < gf.ndof; d += gridDim.x * 256ll) {
        if (fmf[d]) continue;
        const int64_t I = d / 3;
        const int c = (int)(d - 3 * I), y = (int)(I % gf.ny), x = (int)(I / gf.ny % gf.nx), z = (int)(I / ((int64_t)gf.ny * gf.nx));
        for (int k = 0; k < 8; ++k) {
            if (((k & 1) && !(y & 1)) || ((k & 2) && !(x & 1)) || ((k & 4) && !(z & 1))) continue;
            const int64_t J = ((int64_t)((z >> 1) + (k >> 2)) * gc.nx + (x >> 1) + ((k >> 1) & 1)) * gc.ny + (y >> 1) + (k & 1);
            if (fmc[3 * J + c]) *bad = 1;
        }
    }
}

static unsigned blocks_for(int64_t n, int threads) {
    const int64_t b = (n + threads - 1) / threads;
    return (unsigned)(b < 1 ? 1 : (b > 0x7fffffff ? 0x7fffffff : b));
}

void launch_moments_fine(const double *w, const FineGeom &fg, int n, const Grid &gc, double *mom, cudaStream_t st) {
    auto kern = n == 1 ? k_moments_fine<1> : (n == 2 ? k_moments_fine<2> : k_moments_fine<3>);
    kern<<<blocks_for(gc.nelem, 128), 128, 0, st>>>(w, fg.nelx_d, fg.nely_d, gc, mom);
    count_launch();
}
void launch_moments_coarse(const double *mf, const Grid &gf, const Grid &gc, double *mom, cudaStream_t st) {
    k_moments_coarse<<<blocks_for(gc.nelem, 128), 128, 0, st>>>(mf, gf, gc, mom);
    count_launch();
}
void launch_modal_diag(const double *w, const FineGeom &fg, int n, const ModalCoef<double> &k, const uint8_t *freemask,
                       double *diag, cudaStream_t st) {
    auto kern = n == 0 ? k_modal_diag<0> : (n == 1 ? k_modal_diag<1> : (n == 2 ? k_modal_diag<2> : k_modal_diag<3>));
    kern<<<blocks_for(fg.g.nelem, 128), 128, 0, st>>>(w, fg.nelx_d, fg.nely_d, fg.g, k, freemask, diag);
    count_launch();
}
void launch_elem_matrix(const double *mom, const Grid &g, const ModalCoef<double> &k, double *Ae, cudaStream_t st) {
    k_elem_matrix<<<blocks_for(g.nelem, EM_ELEMS), 24 * EM_ELEMS, 0, st>>>(mom, g.nelem, k, Ae);
    count_launch();
}
void launch_clean(const uint8_t *fmf, const uint8_t *fmc, const Grid &gf, const Grid &gc, int *bad, cudaStream_t st) {
    unsigned b = blocks_for(gf.ndof, 256);
    k_clean<<<b > 4096 ? 4096 : b, 256, 0, st>>>(fmf, fmc, gf, gc, bad);
    count_launch();
}

}  // namespace tosp
