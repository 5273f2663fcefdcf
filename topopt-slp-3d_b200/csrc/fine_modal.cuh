// Modal form of the multiresolution hex8 element product, shared by the
// finest-level operator and the sensitivities.
//
// On an element the displacement of component c is the trilinear polynomial
// u_c = sum_chi a_c[chi] xi^chi (chi in {0,1}^3, eight modes, a Walsh-Hadamard
// transform of the corner values), so its strains are polynomials in the
// monomials xi^p, p in {0,1}^3, whose coefficients are the modes themselves:
// d_d u_c has the coefficients a_c[p + e_d].  Integrating the elastic energy
// against the piecewise constant SIMP factors w needs the factors only through
// their moments
//
//     W[t] = sum_s w_s int_s  xi^t dxi,   t in {0,1,2}^3,
//
// because int w xi^p xi^q = W[p + q].  The element product is then: modes,
// strain coefficients (seven of the trace, four per normal strain, six per
// shear strain), one small Gram product S[p] = sum_q W[p + q] E[q] for each,
// and the transposes of the first two steps - about 390 operations for
// MR factor 2 (27 cells: 600) where forming K_e = sum_s w_s KE_s and
// multiplying takes 300 (n^3 + 2), since the moments carry all that the n^3
// blocks contribute.  The blocks KE_s of I/ElemStiffMatrixGQMR.m are integrated
// exactly by their 2-point rule (degree two per direction), so both forms are
// the same operator up to rounding.
//
// The monomials are scaled by sqrt(3) per degree, {1, sqrt(3) xi}, which has
// equal norms on [-1, 1]: for n = 1 and 2 the moments then depend on the
// parity of p + q only, W[p xor q] (n = 2: a Walsh-Hadamard transform of the
// eight factors; n = 1: W[0] alone), and n = 3 takes all 27.
#pragma once

#include "tosp_internal.h"

namespace tosp {

// N: cells per direction, 1 to 3, or 0 for an element whose 27 moments are given
// (a coarse element, see k_moments.cu).
template <int N> constexpr int modal_moments = N == 1 ? 1 : (N == 2 ? 8 : 27);
template <int N> constexpr int modal_values = N == 0 ? 27 : N * N * N;   // given per element

constexpr double MODAL_R3 = 0.57735026918962576451;   // 1 / sqrt(3)

// Bits of a mode or monomial: 1 x, 2 y, 4 z.
__host__ __device__ constexpr int modal_deg(int p) { return (p & 1) + ((p >> 1) & 1) + ((p >> 2) & 1); }
template <int N>
__host__ __device__ constexpr int modal_index(int p, int q) {
    return N == 1 ? 0
                  : (N == 2 ? (p ^ q)
                            : ((p & 1) + (q & 1)) + 3 * (((p >> 1) & 1) + ((q >> 1) & 1)) +
                                  9 * (((p >> 2) & 1) + ((q >> 2) & 1)));
}
// Monomials of the trace (all but xyz), of normal strain c and of the shear
// strain of components c, d.
__host__ __device__ constexpr bool modal_in_trace(int p) { return p != 7; }
__host__ __device__ constexpr bool modal_in_normal(int p, int c) { return !((p >> c) & 1); }
__host__ __device__ constexpr bool modal_in_shear(int p, int c, int d) { return !(((p >> c) & 1) && ((p >> d) & 1)); }

// Shear pairs (c, d).
__host__ __device__ constexpr int modal_sc(int k) { return k == 1 ? 1 : 0; }
__host__ __device__ constexpr int modal_sd(int k) { return k == 0 ? 1 : 2; }

// Moments of the factors w (y fastest, then x, then z) in the scaled basis,
// up to the constant that ModalCoef carries.
template <int N, typename T>
__device__ __forceinline__ void modal_weights(const T (&w)[modal_values<N>], T (&W)[modal_moments<N>]) {
    if constexpr (N == 0) {
#pragma unroll
        for (int q = 0; q < 27; ++q) W[q] = w[q];
    } else if constexpr (N == 1) {
        W[0] = w[0];
    } else if constexpr (N == 2) {
        // cell bits in w's order: 1 y, 2 x, 4 z; W's: 1 x, 2 y, 4 z
#pragma unroll
        for (int q = 0; q < 8; ++q) W[((q & 1) << 1) | ((q >> 1) & 1) | (q & 4)] = w[q];
#pragma unroll
        for (int bit = 1; bit < 8; bit <<= 1)
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (!(q & bit)) {
                    const T lo = W[q], hi = W[q | bit];
                    W[q] = lo + hi;
                    W[q | bit] = hi - lo;
                }
#pragma unroll
        for (int q = 1; q < 8; ++q)
            W[q] *= modal_deg(q) == 1 ? T(1.5 * MODAL_R3) : (modal_deg(q) == 2 ? T(0.75) : T(1.125 * MODAL_R3));
    } else {
        T v[27];
#pragma unroll
        for (int q = 0; q < 27; ++q) v[(q / 3 % 3) + 3 * (q % 3) + 9 * (q / 9)] = w[q];
#pragma unroll
        for (int s = 1; s < 27; s *= 3)
#pragma unroll
            for (int q = 0; q < 27; ++q)
                if (q / s % 3 == 0) {
                    const T l = v[q], m = v[q + s], r = v[q + 2 * s], o = l + r;
                    v[q] = o + m;
                    v[q + s] = T(2.0 * MODAL_R3) * (r - l);
                    v[q + 2 * s] = T(13.0 / 9.0) * o + T(1.0 / 9.0) * m;
                }
#pragma unroll
        for (int q = 0; q < 27; ++q) W[q] = v[q];
    }
}

// S[p] = sum_q W[p + q] E[q] over the monomials `in`.
template <int N, typename T, typename In>
__device__ __forceinline__ void modal_gram(const T (&W)[modal_moments<N>], const T (&E)[8], T (&S)[8], In in) {
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        if (!in(p)) continue;
        S[p] = W[modal_index<N>(p, p)] * E[p];
        if constexpr (N != 1) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (q != p && in(q)) S[p] += W[modal_index<N>(p, q)] * E[q];
        }
    }
}

// Strain coefficients of the modes m (m[c][chi], chi = 1..7, scaled by
// 3^(-(|chi| - 1) / 2)): trace (in units of 2 / el) and shear k (in units of
// 2 / h_d).  The normal strain c has the coefficients m[c][p | 1 << c].
template <typename T>
__device__ __forceinline__ void modal_trace(const T (&m)[3][8], const ModalCoef<T> &k, T (&E)[8]) {
#pragma unroll
    for (int p = 0; p < 7; ++p) {
        bool has = false;
        E[p] = T(0);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if ((p >> c) & 1) continue;
            const T v = m[c][p | (1 << c)];
            if (c == 0) E[p] = v;
            else E[p] = has ? E[p] + k.t[c] * v : k.t[c] * v;
            has = true;
        }
    }
}
template <typename T>
__device__ __forceinline__ void modal_shear(const T (&m)[3][8], const ModalCoef<T> &k, int kk, T (&E)[8]) {
    const int c = modal_sc(kk), d = modal_sd(kk);
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        const bool a = !((p >> d) & 1), b = !((p >> c) & 1);
        if (a && b) E[p] = m[c][p | (1 << d)] + k.sr[kk] * m[d][p | (1 << c)];
        else if (a) E[p] = m[c][p | (1 << d)];
        else if (b) E[p] = k.sr[kk] * m[d][p | (1 << c)];
    }
}

// r = energy gradient with respect to the scaled modes (r[c][0] is zero).
template <int N, typename T>
__device__ __forceinline__ void modal_stress(const T (&m)[3][8], const T (&W)[modal_moments<N>],
                                             const ModalCoef<T> &k, T (&r)[3][8]) {
    T E[8], S[8];
    modal_trace(m, k, E);
    modal_gram<N>(W, E, S, [](int p) { return modal_in_trace(p); });
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int p = 0; p < 7; ++p)
            if (!((p >> c) & 1)) r[c][p | (1 << c)] = k.kt[c] * S[p];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int p = 0; p < 8; ++p)
            if (!((p >> c) & 1)) E[p] = m[c][p | (1 << c)];
        modal_gram<N>(W, E, S, [c](int p) { return modal_in_normal(p, c); });
#pragma unroll
        for (int p = 0; p < 8; ++p)
            if (!((p >> c) & 1)) r[c][p | (1 << c)] = k.kn[c] * S[p] + r[c][p | (1 << c)];
    }
    // modes without bit c get their first contribution from the shears
    bool set[3][8];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int p = 0; p < 8; ++p) set[c][p] = (p >> c) & 1;
#pragma unroll
    for (int kk = 0; kk < 3; ++kk) {
        const int c = modal_sc(kk), d = modal_sd(kk);
        modal_shear(m, k, kk, E);
        modal_gram<N>(W, E, S, [c, d](int p) { return modal_in_shear(p, c, d); });
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            if (!((p >> d) & 1)) {
                T &o = r[c][p | (1 << d)];
                o = set[c][p | (1 << d)] ? o + k.s1[kk] * S[p] : k.s1[kk] * S[p];
                set[c][p | (1 << d)] = true;
            }
            if (!((p >> c) & 1)) {
                T &o = r[d][p | (1 << c)];
                o = set[d][p | (1 << c)] ? o + k.s2[kk] * S[p] : k.s2[kk] * S[p];
                set[d][p | (1 << c)] = true;
            }
        }
    }
}

// F[t] += k sum_{p + q = t} E[p] E[q] over the monomials `in`: the energy's
// derivative with respect to the moments.
template <int N, typename T, typename In>
__device__ __forceinline__ void modal_energy_gram(T k, const T (&E)[8], T (&F)[modal_moments<N>], In in) {
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        if (!in(p)) continue;
        const T kp = k * E[p];
        F[modal_index<N>(p, p)] += kp * E[p];
        if constexpr (N > 1) {
#pragma unroll
            for (int q = p + 1; q < 8; ++q)
                if (in(q)) F[modal_index<N>(p, q)] += (T(2) * kp) * E[q];
        }
    }
}

// Energies u' KE_s u of the cells from the modes m: the products of the strain
// coefficients gathered by moment, then the transpose of modal_weights.
template <int N, typename T>
__device__ __forceinline__ void modal_energies(const T (&m)[3][8], const ModalCoef<T> &k, T (&q)[N * N * N]) {
    T E[8], F[modal_moments<N>];
#pragma unroll
    for (int t = 0; t < modal_moments<N>; ++t) F[t] = T(0);
    modal_trace(m, k, E);
    modal_energy_gram<N>(k.kt[0], E, F, [](int p) { return modal_in_trace(p); });
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int p = 0; p < 8; ++p)
            if (!((p >> c) & 1)) E[p] = m[c][p | (1 << c)];
        modal_energy_gram<N>(k.kn[c], E, F, [c](int p) { return modal_in_normal(p, c); });
    }
#pragma unroll
    for (int kk = 0; kk < 3; ++kk) {
        const int c = modal_sc(kk), d = modal_sd(kk);
        modal_shear(m, k, kk, E);
        modal_energy_gram<N>(k.s1[kk], E, F, [c, d](int p) { return modal_in_shear(p, c, d); });
    }
    if constexpr (N == 1) {
        q[0] = F[0];
    } else if constexpr (N == 2) {
#pragma unroll
        for (int b = 1; b < 8; ++b)
            F[b] *= modal_deg(b) == 1 ? T(1.5 * MODAL_R3) : (modal_deg(b) == 2 ? T(0.75) : T(1.125 * MODAL_R3));
#pragma unroll
        for (int bit = 1; bit < 8; bit <<= 1)
#pragma unroll
            for (int b = 0; b < 8; ++b)
                if (!(b & bit)) {
                    const T e = F[b], o = F[b | bit];
                    F[b] = e - o;
                    F[b | bit] = e + o;
                }
#pragma unroll
        for (int s = 0; s < 8; ++s) q[s] = F[((s & 1) << 1) | ((s >> 1) & 1) | (s & 4)];
    } else {
#pragma unroll
        for (int s = 1; s < 27; s *= 3)
#pragma unroll
            for (int b = 0; b < 27; ++b)
                if (b / s % 3 == 0) {
                    const T f0 = F[b], f1 = T(2.0 * MODAL_R3) * F[b + s], f2 = F[b + 2 * s];
                    const T e = f0 + T(13.0 / 9.0) * f2;
                    F[b] = e - f1;
                    F[b + s] = f0 + T(1.0 / 9.0) * f2;
                    F[b + 2 * s] = e + f1;
                }
#pragma unroll
        for (int s = 0; s < 27; ++s) q[s] = F[(s / 3 % 3) + 3 * (s % 3) + 9 * (s / 9)];
    }
}

// Diagonal of the element matrix, D[a][c] at corner a (1 y, 2 x, 4 z) and
// component c.  For the derivative along d the products of modes chi, chi' with
// chi xor chi' = beta add up to H_d[beta], and a corner's value is the sum of
// sign^beta over beta.
template <int N, typename T>
__device__ __forceinline__ void modal_diagonal(const T (&W)[modal_moments<N>], const ModalCoef<T> &k, T (&D)[8][3]) {
    T H[3][8];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            H[d][b] = T(0);
            if ((b >> d) & 1) continue;
#pragma unroll
            for (int p = 0; p < 8; ++p) {
                if ((p >> d) & 1) continue;
                if (N == 1 && b) continue;
                const int n = modal_deg(p) + modal_deg(p ^ b);   // 3^(-n / 2)
                H[d][b] += T(n == 0 ? 1.0 : (n == 1 ? MODAL_R3 : (n == 2 ? 1.0 / 3.0 : (n == 3 ? MODAL_R3 / 3.0 : 1.0 / 9.0)))) *
                           W[modal_index<N>(p, p ^ b)];
            }
        }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        T f[8];
#pragma unroll
        for (int b = 0; b < 8; ++b) f[b] = (k.kt[c] * k.t[c] + k.kn[c]) * H[c][b];
#pragma unroll
        for (int kk = 0; kk < 3; ++kk) {
            const int sc = modal_sc(kk), sd = modal_sd(kk);
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                if (c == sc) f[b] += k.s1[kk] * H[sd][b];
                if (c == sd) f[b] += k.s2[kk] * k.sr[kk] * H[sc][b];
            }
        }
#pragma unroll
        for (int bit = 1; bit < 8; bit <<= 1)
#pragma unroll
            for (int b = 0; b < 8; ++b)
                if (!(b & bit)) {
                    const T e = f[b], o = f[b | bit];
                    f[b] = e - o;
                    f[b | bit] = e + o;
                }
#pragma unroll
        for (int a = 0; a < 8; ++a) D[a][c] = f[((a >> 1) & 1) | ((a & 1) << 1) | (a & 4)];
    }
}

// Two-dimensional modes (x, y) of one component on a node plane from the four
// corner values.  FP32 keeps the low corner apart and transforms the
// differences to it, which are exact or nearly so for the smooth fields of a
// solve: the coefficients then err relative to the element's deformation and
// not to its displacement (the constant mode is not used by the product).
template <typename T>
struct PlaneModes {
    T b, s, x, y, xy;   // low corner (FP32), sum (FP32: of the differences), modes
};
template <typename T>
__device__ __forceinline__ PlaneModes<T> plane_modes(T u00, T u0y, T ux0, T uxy) {
    PlaneModes<T> o;
    if constexpr (sizeof(T) == 4) {
        const T d1 = u0y - u00, d2 = ux0 - u00, d3 = uxy - u00;
        o.b = u00;
        o.xy = (d3 - d1) - d2;
        o.x = (d3 - d1) + d2;
        o.y = (d3 - d2) + d1;
        o.s = (d1 + d2) + d3;
    } else {
        const T p = u00 + u0y, q = ux0 + uxy, v = u0y - u00, w = uxy - ux0;
        o.b = T(0);
        o.s = p + q;
        o.x = q - p;
        o.y = v + w;
        o.xy = w - v;
    }
    return o;
}

// Scaled modes of one component from its two node planes.
template <typename T>
__device__ __forceinline__ void element_modes(const PlaneModes<T> &lo, const PlaneModes<T> &hi, T (&m)[8]) {
    m[0] = T(0);
    m[1] = lo.x + hi.x;
    m[2] = lo.y + hi.y;
    m[3] = T(MODAL_R3) * (lo.xy + hi.xy);
    if constexpr (sizeof(T) == 4) m[4] = T(4) * (hi.b - lo.b) + (hi.s - lo.s);
    else m[4] = hi.s - lo.s;
    m[5] = T(MODAL_R3) * (hi.x - lo.x);
    m[6] = T(MODAL_R3) * (hi.y - lo.y);
    m[7] = T(1.0 / 3.0) * (hi.xy - lo.xy);
}

}  // namespace tosp
