// Matrix-free Tet10 element kernels shared by the operator, the persistent PCG
// and the adjoint. No reference counterpart: the reference forms K_e
// explicitly (element.rs:23-61, mechanics/element.rs:33-65); these apply the
// same K_e to a vector without forming it.
#pragma once

#include "tet10.cuh"

namespace geo {

// Per-element geometric data ("qdata"), stored patch-major: for patch p, value j
// of the patch's element e sits at [(p * NQD + j) * kPatchElems + e]. Thermal: the
// symmetric 3x3 G = (k w / |det J|) adj(J) adj(J)^T packed as [xx xy xz yy yz zz], per
// quadrature point for curved elements (NQ = 4), once for affine elements (NQ = 1; in FP64
// times 4/5, see apply_affine). Elasticity: J^{-1} (9, row-major) and
// s = w |det J| E_e, once or per quadrature point.
template <class T, int NQ>
struct ThermalK {
    static constexpr int DPN = 1;
    static constexpr int NQD = 6 * NQ;

    // y = S K_e x. qd points at the element's first qdata value; value j sits at qd[j * stride].
    // The FP32 PCG takes the affine form like FP64 (128^3: 248 us per launch against 254
    // point by point): its rounding is the refinement's to correct. The FP32 operator apply
    // hands its rounding to the caller and keeps the point by point form (NQ == 1: one G for
    // the four points).
    template <bool PCG = false>
    __device__ __forceinline__ static void apply(const T* __restrict__ qd, int64_t stride, T, T, T S,
                                                 const T (&x)[10], T (&y)[10]) {
        if (NQ == 1 && (sizeof(T) == 8 || PCG)) apply_affine(qd, stride, sizeof(T) == 8 ? S : T(0.8) * S, x, y);
        else apply_quadrature(qd, stride, S, x, y);
    }

    // Affine element: the gradient is linear in L, so with its values c_m at the four
    // vertices, int grad.G.grad = sum_mn (1 + delta_mn) / 20 c_m.G c_n: the exact value
    // of the 4-point rule, on 4/5 of the rule's G (4 points / 20 x 4, the factor 4 of the
    // gradients folded in), which the FP64 qdata holds and S brings to the FP32 one. 114
    // operations, against 132 for the point by point form.
    __device__ __forceinline__ static void apply_affine(const T* __restrict__ qd, int64_t stride, T S,
                                                        const T (&x)[10], T (&y)[10]) {
        T G[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) G[j] = S * qd[j * stride];
        // c[m][a] = 4 (M_(a+1)m - M_0m) - (x_(a+1) - x_0), M the symmetric nodal matrix
        T d[3], c[4][3], sum[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) d[a] = x[a + 1] - x[0];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const T h0 = m == 0 ? x[0] : x[edge_of(0, m == 0 ? 1 : m)];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const T h = a + 1 == m ? x[m] : x[edge_of(a + 1, a + 1 == m ? 0 : m)];
                c[m][a] = T(4) * (h - h0) - d[a];
            }
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) sum[a] = (c[0][a] + c[1][a]) + (c[2][a] + c[3][a]);
        T f[4][4];  // f[m][j]: flux at vertex m in barycentric direction j
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const T w0 = c[m][0] + sum[0], w1 = c[m][1] + sum[1], w2 = c[m][2] + sum[2];
            f[m][1] = G[0] * w0 + G[1] * w1 + G[2] * w2;
            f[m][2] = G[1] * w0 + G[3] * w1 + G[4] * w2;
            f[m][3] = G[2] * w0 + G[4] * w1 + G[5] * w2;
            f[m][0] = -(f[m][1] + f[m][2] + f[m][3]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] = f[j][j] - T(0.25) * ((f[0][j] + f[1][j]) + (f[2][j] + f[3][j]));
#pragma unroll
        for (int k = 0; k < 6; ++k) y[4 + k] = f[edge_v(k, 0)][edge_v(k, 1)] + f[edge_v(k, 1)][edge_v(k, 0)];
    }

    // Curved element, G per quadrature point:
    // h_m(q) = base_m + D4 M_mq (M: nodal matrix), grad_xi = (h1-h0, h2-h0, h3-h0);
    // flux v_q = G grad_xi; phi_q = (-sum v, v); Phi = sum_q phi_q; then
    //   y_m = (B4 - 1) Phi_m + D4 phi_{m,m},  y_(mn) = B4 (Phi_m + Phi_n) + D4 (phi_{n,m} + phi_{m,n}).
    __device__ __forceinline__ static void apply_quadrature(const T* __restrict__ qd, int64_t stride, T S,
                                                            const T (&x)[10], T (&y)[10]) {
        const T B4 = T(4.0 * kQb), D4 = T(4.0 * (kQa - kQb)), B4m1 = T(4.0 * kQb - 1.0);
        T base[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            T s = x[m];
#pragma unroll
            for (int n = 0; n < 4; ++n)
                if (n != m) s += x[edge_of(m, n)];
            base[m] = B4 * s - x[m];
        }
        T phi[4][4], Phi[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            T G[6];
#pragma unroll
            for (int j = 0; j < 6; ++j) G[j] = qd[(NQ == 1 ? j : 6 * q + j) * stride];
            T h[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) h[m] = base[m] + D4 * (m == q ? x[m] : x[edge_of(m, m == q ? (q + 1) % 4 : q)]);
            const T g0 = h[1] - h[0], g1 = h[2] - h[0], g2 = h[3] - h[0];
            const T v0 = G[0] * g0 + G[1] * g1 + G[2] * g2;
            const T v1 = G[1] * g0 + G[3] * g1 + G[4] * g2;
            const T v2 = G[2] * g0 + G[4] * g1 + G[5] * g2;
            phi[q][0] = -(v0 + v1 + v2);
            phi[q][1] = v0;
            phi[q][2] = v1;
            phi[q][3] = v2;
#pragma unroll
            for (int m = 0; m < 4; ++m) Phi[m] = q == 0 ? phi[0][m] : Phi[m] + phi[q][m];
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) y[m] = S * (B4m1 * Phi[m] + D4 * phi[m][m]);
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const int m = edge_v(k, 0), n = edge_v(k, 1);
            y[4 + k] = S * (B4 * (Phi[m] + Phi[n]) + D4 * (phi[n][m] + phi[m][n]));
        }
    }
};

template <class T, int NQ>
struct ElasticK {
    static constexpr int DPN = 3;
    static constexpr int NQD = 10 * NQ;

    // x, y interleaved [3*i + c]; cl = nu/((1+nu)(1-2nu)), cm = 1/(2(1+nu))
    // y = S K_e x; S is applied to y last: times the element's stiffness it could overflow
    template <bool PCG = false>
    __device__ __forceinline__ static void apply(const T* __restrict__ qd, int64_t stride, T cl, T cm, T S,
                                                 const T (&x)[30], T (&y)[30]) {
        const T B4 = T(4.0 * kQb), D4 = T(4.0 * (kQa - kQb)), B4m1 = T(4.0 * kQb - 1.0);
        T base[3][4];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                T s = x[3 * m + c];
#pragma unroll
                for (int n = 0; n < 4; ++n)
                    if (n != m) s += x[3 * edge_of(m, n) + c];
                base[c][m] = B4 * s - x[3 * m + c];
            }
#pragma unroll
        for (int i = 0; i < 30; ++i) y[i] = T(0);
        T Ji[9], s = T(0);
        if (NQ == 1) {
#pragma unroll
            for (int j = 0; j < 9; ++j) Ji[j] = qd[j * stride];
            s = qd[9 * stride];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (NQ == 4) {
#pragma unroll
                for (int j = 0; j < 9; ++j) Ji[j] = qd[(10 * q + j) * stride];
                s = qd[(10 * q + 9) * stride];
            }
            // displacement gradient F[c][b] = sum_a H[c][a] Ji[a][b]
            T F[3][3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                T h[4];
#pragma unroll
                for (int m = 0; m < 4; ++m)
                    h[m] = base[c][m] + D4 * (m == q ? x[3 * m + c] : x[3 * edge_of(m, q) + c]);
                const T H0 = h[1] - h[0], H1 = h[2] - h[0], H2 = h[3] - h[0];
#pragma unroll
                for (int b = 0; b < 3; ++b) F[c][b] = H0 * Ji[b] + H1 * Ji[3 + b] + H2 * Ji[6 + b];
            }
            const T tr = cl * (F[0][0] + F[1][1] + F[2][2]);
            T S[3][3];
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int b = 0; b < 3; ++b) S[c][b] = s * (cm * (F[c][b] + F[b][c]) + (c == b ? tr : T(0)));
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                // P[c][a] = sum_b S[c][b] Ji[a][b]
                const T P0 = S[c][0] * Ji[0] + S[c][1] * Ji[1] + S[c][2] * Ji[2];
                const T P1 = S[c][0] * Ji[3] + S[c][1] * Ji[4] + S[c][2] * Ji[5];
                const T P2 = S[c][0] * Ji[6] + S[c][1] * Ji[7] + S[c][2] * Ji[8];
                const T phi[4] = {-(P0 + P1 + P2), P0, P1, P2};
#pragma unroll
                for (int m = 0; m < 4; ++m) y[3 * m + c] += (m == q ? B4m1 + D4 : B4m1) * phi[m];
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    const int m = edge_v(k, 0), n = edge_v(k, 1);
                    T t = B4 * (phi[m] + phi[n]);
                    if (q == n) t += D4 * phi[m];
                    if (q == m) t += D4 * phi[n];
                    y[3 * (4 + k) + c] += t;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 30; ++i) y[i] *= S;
    }
};

}  // namespace geo
