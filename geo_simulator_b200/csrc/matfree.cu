// K5/K6/K7: matrix-free Tet10 operator, persistent Jacobi-PCG (FP64 and mixed
// FP32/FP64 with on-device residual refresh), and the adjoint element gradient.
//
// Operator: K_bc of apply_dirichlet_bcs (assembly.rs:168-230) applied to a
// vector without assembling K (assembly.rs:69-117 / :389-437):
//   free rows  y_i = sum_{j free} K_ij x_j,   Dirichlet rows y_i = char_diag x_i.
// Elements are processed patch by patch (see patches.h): a CTA gathers the
// patch's nodal values into shared memory, every thread applies K_e of its
// elements from the per-element qdata, accumulates into shared memory, and the
// patch flushes its nodes: plain stores for nodes no other patch touches,
// red.global.add for the shared ones (so the matrix-free apply is not
// bit-reproducible in the last bit; the assembled path is). The PCG of the
// operator runs in halo mode instead: foreign contributions are stored to
// per-entry slots and added by the node update in slot order, with no atomics.
#include <algorithm>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <utility>

#include <cub/cub.cuh>

#include "mf_kernels.cuh"
#include "pcg_common.cuh"

struct geo_op;

namespace geo {

// f_bc: free rows f - (K_{F,D} g), Dirichlet rows g cd
__global__ void k_lift_finish(const uint8_t* flags, int dpn, int64_t n, double cd, const double* f,
                              const double* g, const double* kg, double* out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const bool dir = (flags[i / dpn] >> (i % dpn)) & 1;
        out[i] = dir ? g[i] * cd : f[i] - kg[i];
    }
}

__global__ void k_scale(double* v, int64_t n, double a) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        v[i] *= a;
}

template <class T>
__global__ void k_zero_dir(const uint8_t* flags, int dpn, int64_t n, T* v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        if ((flags[i / dpn] >> (i % dpn)) & 1) v[i] = T(0);
}

// out[new] = in[orig] / out[orig] = in[new] for interleaved dpn vectors
template <class Tin, class Tout>
__global__ void k_to_new(const int32_t* nperm, int dpn, int64_t N, const Tin* in, Tout* out) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < N * dpn; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t / dpn;
        const int c = (int)(t % dpn);
        out[t] = (Tout)in[(int64_t)nperm[i] * dpn + c];
    }
}
template <class Tin, class Tout>
__global__ void k_to_orig(const int32_t* nperm, int dpn, int64_t N, const Tin* in, Tout* out) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < N * dpn; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t / dpn;
        const int c = (int)(t % dpn);
        out[(int64_t)nperm[i] * dpn + c] = (Tout)in[t];
    }
}

// ------------------------------------------------------------------ set-up kernels
// node flags (Dirichlet bits, shared bit) and Dirichlet values in patch numbering
__global__ void k_node_flags(const int32_t* nperm, const uint8_t* shared, const uint8_t* mask, const double* vals,
                             int dpn, int64_t N, uint8_t* flags, double* g_new) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = nperm[i];
        uint8_t f = shared[i] ? kFlagShared : 0;
        for (int c = 0; c < dpn; ++c) {
            if (mask[o * dpn + c]) f |= (uint8_t)(kFlagDir0 << c);
            g_new[i * dpn + c] = vals[o * dpn + c];
        }
        flags[i] = f;
    }
}

__device__ __forceinline__ void load_elem(const double* __restrict__ xyz, const int32_t* __restrict__ conn,
                                          int64_t N, int64_t E, int64_t e, double (&X)[10][3]) {
#pragma unroll
    for (int l = 0; l < 10; ++l) {
        const int64_t nd = conn[l * E + e];
        X[l][0] = xyz[nd];
        X[l][1] = xyz[N + nd];
        X[l][2] = xyz[2 * N + nd];
    }
}

// flags[0] |= 1 when some element is not affine (a midpoint off its edge centre)
__global__ void k_affine_check(const double* xyz, const int32_t* conn, int64_t N, int64_t E, int* flag) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= E) return;
    double X[10][3];
    load_elem(xyz, conn, N, E, e, X);
    double h = 0.0;
    for (int k = 0; k < 6; ++k)
        for (int c = 0; c < 3; ++c) h = fmax(h, fabs(X[edge_v(k, 1)][c] - X[edge_v(k, 0)][c]));
    for (int k = 0; k < 6; ++k)
        for (int c = 0; c < 3; ++c) {
            const double mid = 0.5 * (X[edge_v(k, 0)][c] + X[edge_v(k, 1)][c]);
            if (fabs(X[4 + k][c] - mid) > 1e-13 * h) atomicOr(flag, 1);
        }
}

// geometry at QP q (NQ == 4) or the affine vertex Jacobian (NQ == 1)
template <int NQ>
__device__ __forceinline__ void elem_jacobian(const double (&X)[10][3], int q, double (&J)[3][3]) {
    if (NQ == 1) {
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) J[r][c] = X[c + 1][r] - X[0][r];
    } else {
        double L[4];
        qp4(q, L);
        jacobian10(X, L, J);
    }
}

// qdata in patch element order (see matfree.cuh)
template <int NQ>
__global__ void k_qdata(int phys, const double* xyz, const int32_t* conn, const int32_t* eperm, int64_t N,
                        int64_t E, const double* coef, double* qd64, float* qd32, int* err) {
    const int64_t ne = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (ne >= E) return;
    const int64_t e = eperm[ne];
    double X[10][3];
    load_elem(xyz, conn, N, E, e, X);
    const double k = coef[e];
    for (int q = 0; q < NQ; ++q) {
        double J[3][3], A[3][3];
        elem_jacobian<NQ>(X, q, J);
        const double d = det3(J);
        if (d == 0.0) {
            atomicOr(err, DEV_ERR_SINGULAR);
            return;
        }
        adj3(J, A);
        if (phys == 0) {
            const double s = kQw * k / fabs(d);
            double G[6];
            G[0] = s * (A[0][0] * A[0][0] + A[0][1] * A[0][1] + A[0][2] * A[0][2]);
            G[1] = s * (A[0][0] * A[1][0] + A[0][1] * A[1][1] + A[0][2] * A[1][2]);
            G[2] = s * (A[0][0] * A[2][0] + A[0][1] * A[2][1] + A[0][2] * A[2][2]);
            G[3] = s * (A[1][0] * A[1][0] + A[1][1] * A[1][1] + A[1][2] * A[1][2]);
            G[4] = s * (A[1][0] * A[2][0] + A[1][1] * A[2][1] + A[1][2] * A[2][2]);
            G[5] = s * (A[2][0] * A[2][0] + A[2][1] * A[2][1] + A[2][2] * A[2][2]);
            for (int j = 0; j < 6; ++j) {
                const int64_t at = ((ne / kPatchElems) * (6 * NQ) + 6 * q + j) * kPatchElems + ne % kPatchElems;
                qd64[at] = NQ == 1 ? 0.8 * G[j] : G[j];  // see ThermalK::apply_affine
                qd32[at] = (float)G[j];
            }
        } else {
            double v[10];
            for (int r = 0; r < 3; ++r)
                for (int c = 0; c < 3; ++c) v[3 * r + c] = A[r][c] / d;
            v[9] = kQw * fabs(d) * k;
            for (int j = 0; j < 10; ++j) {
                const int64_t at = ((ne / kPatchElems) * (10 * NQ) + 10 * q + j) * kPatchElems + ne % kPatchElems;
                qd64[at] = v[j];
                qd32[at] = (float)v[j];
            }
        }
    }
}

// Foreign ids and flags of every patch copied into segments that start at
// pfa[p] (multiples of kForeignAlign entries), so that the patch kernel's bulk
// copy brings them with the element data. One block per patch.
__global__ void k_patch_foreign(const int32_t* __restrict__ pf, const int32_t* __restrict__ pfa,
                               const int32_t* __restrict__ foreign, const uint8_t* __restrict__ flags,
                               int32_t* __restrict__ fids, uint8_t* __restrict__ fflags) {
    const int p = blockIdx.x;
    const int f0 = pf[p], nf = pf[p + 1] - f0, a0 = pfa[p];
    for (int k = threadIdx.x; k < nf; k += blockDim.x) {
        const int32_t nd = foreign[f0 + k];
        fids[a0 + k] = nd;
        fflags[a0 + k] = flags[nd];
    }
}

// Halo slots of the PCG (thermal and elasticity): every foreign entry a (patch p, its
// k-th foreign node n, a = pf[p] + k) gets a slot. Slots are ordered by node n,
// then by entry (a stable sort of the entries by node), so node n's slots are
// consecutive and follow those of the nodes before it.
__global__ void k_halo_count(const int32_t* __restrict__ foreign, int64_t n_app, int32_t* __restrict__ cnt) {
    for (int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; a < n_app; a += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&cnt[foreign[a]], 1);
}
__global__ void k_iota(int64_t n, int32_t* __restrict__ v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        v[i] = (int32_t)i;
}
__global__ void k_halo_slot_of(const int32_t* __restrict__ sorted_app, int64_t n_app, int32_t* __restrict__ slot_of) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_app; t += (int64_t)gridDim.x * blockDim.x)
        slot_of[sorted_app[t]] = (int32_t)t;
}
// the slots again in the per-patch segments of fids (one block per patch)
__global__ void k_patch_fslot(const int32_t* __restrict__ pf, const int32_t* __restrict__ pfa,
                              const int32_t* __restrict__ slot_of, int32_t* __restrict__ fslot) {
    const int p = blockIdx.x;
    const int f0 = pf[p], nf = pf[p + 1] - f0, a0 = pfa[p];
    for (int k = threadIdx.x; k < nf; k += blockDim.x) fslot[a0 + k] = slot_of[f0 + k];
}
// flag bits 3-6 = slot count (<= 15); chunk[c] = slots of nodes [32 c, 32 c + 32).
// The grid covers whole warps of 32 consecutive nodes.
__global__ void k_halo_flags(const int32_t* __restrict__ cnt, int64_t N, uint8_t* __restrict__ flags,
                             int32_t* __restrict__ chunk) {
    const int64_t N32 = (N + 31) / 32 * 32;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N32; i += (int64_t)gridDim.x * blockDim.x) {
        const int c = i < N ? cnt[i] : 0;
        if (i < N) flags[i] = (uint8_t)(flags[i] | (c << kHaloShift));
        const int sum = __reduce_add_sync(0xffffffffu, c);
        if ((threadIdx.x & 31) == 0) chunk[i / 32] = sum;
    }
}

// Largest number of a patch's elements that touch one patch-local node. One
// block per patch; counts in shared memory (max_local ints, by slot).
__global__ void k_patch_maxinc(const int32_t* __restrict__ pe, const int32_t* __restrict__ po,
                               const int32_t* __restrict__ pf, const uint32_t* __restrict__ lc, int32_t* maxinc) {
    extern __shared__ int cnt[];
    __shared__ int s_max;
    const int p = blockIdx.x;
    const int n_el = pe[p + 1] - pe[p];
    const int nloc = (po[p + 1] - patch_align(po[p])) + (pf[p + 1] - pf[p]);
    const int nslot = nloc > 0 ? patch_slot(nloc - 1) + 1 : 0;  // lc holds slots
    for (int u = threadIdx.x; u < nslot; u += blockDim.x) cnt[u] = 0;
    if (threadIdx.x == 0) s_max = 0;
    __syncthreads();
    for (int t = threadIdx.x; t < n_el * 10; t += blockDim.x) {
        const int j = t / 10, l = t % 10;
        const uint32_t w = lc[((int64_t)p * 5 + l / 2) * kPatchElems + j];
        const int u = (int)((l & 1) ? (w >> 16) : (w & 0xffffu));
        if (u < nslot) atomicAdd(&cnt[u], 1);
    }
    __syncthreads();
    int m = 0;
    for (int u = threadIdx.x; u < nslot; u += blockDim.x) m = max(m, cnt[u]);
    atomicMax(&s_max, m);
    __syncthreads();
    if (threadIdx.x == 0) maxinc[p] = s_max;
}

// max_e ||K_e||_inf per patch (row abs sums of K_e applied to the unit vectors,
// FP64 qdata), stored as double bits: non-negative doubles order like their bits.
template <class K>
__global__ void k_patch_knorm(const double* __restrict__ qd64, int64_t E, double cl, double cm,
                              unsigned long long* __restrict__ knorm) {
    constexpr int ND = 10 * K::DPN;
    const int64_t ne = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (ne >= E) return;
    const double* qd = qd64 + (ne / kPatchElems) * K::NQD * kPatchElems + ne % kPatchElems;
    double rs[ND];
#pragma unroll
    for (int i = 0; i < ND; ++i) rs[i] = 0.0;
    for (int j = 0; j < ND; ++j) {
        double x[ND], y[ND];
#pragma unroll
        for (int i = 0; i < ND; ++i) x[i] = i == j ? 1.0 : 0.0;
        K::apply(qd, kPatchElems, cl, cm, 1.0, x, y);
#pragma unroll
        for (int i = 0; i < ND; ++i) rs[i] += fabs(y[i]);
    }
    double m = 0.0;
#pragma unroll
    for (int i = 0; i < ND; ++i) m = fmax(m, rs[i]);
    atomicMax(&knorm[ne / kPatchElems], (unsigned long long)__double_as_longlong(m));
}

// bound32[p] = maxinc[p] * max_e ||K_e||_inf * 1.001 (margin for the FP32 qdata and
// the rounding of the contributions), rounded up to FP32.
__global__ void k_patch_bound(const int32_t* __restrict__ maxinc, const unsigned long long* __restrict__ knorm,
                              int P, float* __restrict__ b32) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    b32[p] = __double2float_ru((double)maxinc[p] * __longlong_as_double((long long)knorm[p]) * 1.001);
}

// Diagonal of every K_e, original element order: ediag[e][dpn*l + c].
__global__ void k_ediag(int phys, const double* xyz, const int32_t* conn, int64_t N, int64_t E, const double* coef,
                        double cl, double cm, double* ediag, int* err) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= E) return;
    double X[10][3];
    load_elem(xyz, conn, N, E, e, X);
    const double k = coef[e];
    const int dpn = phys == 0 ? 1 : 3;
    double acc[30];
    for (int i = 0; i < 30; ++i) acc[i] = 0.0;
    for (int q = 0; q < 4; ++q) {
        double L[4], J[3][3], A[3][3];
        qp4(q, L);
        jacobian10(X, L, J);
        const double d = det3(J);
        if (d == 0.0) {
            atomicOr(err, DEV_ERR_SINGULAR);
            return;
        }
        adj3(J, A);
        double Ji[3][3];
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c) Ji[r][c] = A[r][c] / d;
        const double w = kQw * fabs(d);
        for (int l = 0; l < 10; ++l) {
            double g[3], gc[3];
            ref_grad(l, L, g);
            cart_grad(Ji, g, gc);
            const double gg = gc[0] * gc[0] + gc[1] * gc[1] + gc[2] * gc[2];
            if (phys == 0) {
                acc[l] += k * gg * w;
            } else {
                for (int c = 0; c < 3; ++c)
                    acc[3 * l + c] += w * k * (cl * gc[c] * gc[c] + cm * (gg + gc[c] * gc[c]));
            }
        }
    }
    for (int i = 0; i < 10 * dpn; ++i) ediag[e * 10 * dpn + i] = acc[i];
}

__global__ void k_gather_diag(const int32_t* ptr, const int32_t* inc, const double* ediag, int64_t N, int dpn,
                              double* diag) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= N * dpn) return;
    const int64_t i = t / dpn;
    const int c = (int)(t % dpn);
    double s = 0.0;
    for (int32_t p = ptr[i]; p < ptr[i + 1]; ++p) {
        const int32_t el = inc[p];
        s += ediag[(int64_t)(el / 10) * 10 * dpn + dpn * (el % 10) + c];
    }
    diag[t] = s;
}

// max_i |v_i w_i| as the bit pattern of a non-negative double
__global__ void k_max_abs_scaled(const double* v, const double* w, int64_t n, unsigned long long* out) {
    double m = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        m = fmax(m, fabs(v[i] * w[i]));
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

__global__ void k_max_abs(const double* v, int64_t n, unsigned long long* out) {
    double m = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        m = fmax(m, fabs(v[i]));
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

// dinv in patch numbering (JacobiPreconditioner::new, preconditioner.rs:37-51 on K_bc)
__global__ void k_dinv(const int32_t* nperm, const uint8_t* flags, int dpn, int64_t N, const double* diag_orig,
                       double cd, double* d64, float* d32, double* dg_out) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < N * dpn; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t / dpn;
        const int c = (int)(t % dpn);
        const bool dir = (flags[i] >> c) & 1;
        const double dd = dir ? cd : diag_orig[(int64_t)nperm[i] * dpn + c];
        const double inv = fabs(dd) > 1e-14 ? 1.0 / dd : 1.0;
        d64[t] = inv;
        d32[t] = (float)inv;
        if (dg_out) dg_out[t] = dd;
    }
}

// Adjoint element gradient g_e = -lambda_e^T K_e u_e (original order, FP64),
// lambda read as zero on Dirichlet DOFs. Isoparametric, so curved elements too.
__global__ void k_elem_gradient(int phys, const double* xyz, const int32_t* conn, int64_t N, int64_t E,
                                const double* coef, double cl, double cm, const uint8_t* mask, const double* u,
                                const double* lam, double* g) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= E) return;
    double X[10][3];
    load_elem(xyz, conn, N, E, e, X);
    const double k = coef[e];
    const int dpn = phys == 0 ? 1 : 3;
    double ue[30], le[30];
    for (int l = 0; l < 10; ++l) {
        const int64_t nd = conn[l * E + e];
        for (int c = 0; c < dpn; ++c) {
            const int64_t dof = nd * dpn + c;
            ue[l * dpn + c] = u[dof];
            le[l * dpn + c] = mask[dof] ? 0.0 : lam[dof];
        }
    }
    double s = 0.0;
    for (int q = 0; q < 4; ++q) {
        double L[4], J[3][3], A[3][3];
        qp4(q, L);
        jacobian10(X, L, J);
        const double d = det3(J);
        if (d == 0.0) continue;
        adj3(J, A);
        double Ji[3][3];
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c) Ji[r][c] = A[r][c] / d;
        const double w = kQw * fabs(d);
        double Fu[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, Fl[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
        for (int l = 0; l < 10; ++l) {
            double gr[3], gc[3];
            ref_grad(l, L, gr);
            cart_grad(Ji, gr, gc);
            for (int c = 0; c < dpn; ++c)
                for (int b = 0; b < 3; ++b) {
                    Fu[c][b] += ue[l * dpn + c] * gc[b];
                    Fl[c][b] += le[l * dpn + c] * gc[b];
                }
        }
        if (phys == 0) {
            s += k * w * (Fu[0][0] * Fl[0][0] + Fu[0][1] * Fl[0][1] + Fu[0][2] * Fl[0][2]);
        } else {
            const double tu = Fu[0][0] + Fu[1][1] + Fu[2][2], tl = Fl[0][0] + Fl[1][1] + Fl[2][2];
            double ee = 0.0;
            for (int c = 0; c < 3; ++c)
                for (int b = 0; b < 3; ++b) ee += 0.5 * (Fu[c][b] + Fu[b][c]) * (Fl[c][b] + Fl[b][c]);
            // lambda tr(eps_u) tr(eps_l) + 2 mu eps_u : eps_l, with lambda = k cl, mu = k cm
            s += w * k * (cl * tu * tl + cm * ee);
        }
    }
    g[e] = -s;
}

}  // namespace geo

// ====================================================================== operator object
struct geo_op {
    geo_ctx* ctx = nullptr;
    geo::CtxRef ref;  // released after every buffer below
    const geo_mesh* mesh = nullptr;
    int phys = 0, dpn = 1, nq = 1;
    int64_t N = 0, E = 0, ndof = 0;
    int n_patches = 0, max_local = 0;
    double nu = 0, cl = 0, cm = 0, cd = 1.0, coef_scalar = 1.0;
    geo::DevBuf<int32_t> eperm, nperm, pe, po, pf, foreign;
    geo::DevBuf<uint32_t> lc, lc32;
    geo::DevBuf<uint8_t> flags;
    geo::DevBuf<uint8_t> mask_orig;  // Dirichlet mask, original DOF numbering
    geo::DevBuf<double> coef, qd64, g_new, diag_new, dinv64, ediag, diag_orig;
    geo::DevBuf<float> qd32, dinv32;
    // foreign ids and flags in aligned per-patch segments (bulk-copied with the elements)
    geo::DevBuf<int32_t> pfa, fids;
    geo::DevBuf<uint8_t> fflags;
    int max_for = 0;
    int max_own = 0;  // largest own-node count of a patch
    // halo mode of the PCG: slot of every foreign entry (fids
    // segments), slots before each 32-node chunk, and the slot arrays
    geo::DevBuf<int32_t> fslot, hbase;
    geo::DevBuf<double> halo64;
    geo::DevBuf<float> halo32;
    int64_t n_app = 0;
    bool halo_ok = false;  // slots built (every node has at most 15)
    int halo[2] = {0, 0};  // halo mode in use (FP64, FP32), see setup
    // per-patch bound of the fixed-point scatter (Scatter in mf_kernels.cuh)
    geo::DevBuf<int32_t> pmaxinc;
    geo::DevBuf<float> pbound32;
    geo::DevBuf<geo::PatchMeta> prec;  // per-patch records (PatchView::rec)
    // solver workspace
    geo::DevBuf<double> w64;
    geo::DevBuf<float> w32;
    geo::DevBuf<double> bvec, xvec;  // right-hand side and solution (patch numbering)
    // grow-only temporaries of the API calls (no cudaMalloc / cudaFree per call once
    // grown: cudaFree synchronises the device and can stall the caller)
    geo::DevBuf<double> tmp[7];
    geo::DevBuf<float> tmp32[2];
    geo::DevBuf<unsigned long long> tmpu[2];
    geo::DevBuf<geo::PcgState> state;
    geo::DevBuf<double> part, part_patch;  // per-block partials: node kernels, patch kernel
    geo::PcgState* h_state = nullptr;  // pinned mirror
    int patch_grid[2] = {0, 0};        // resident patch-kernel blocks (FP64, FP32)
    int nbuf[2] = {2, 2};              // element-data buffers of the patch kernel (FP64, FP32)
    int own_bulk[2] = {0, 0};          // own-node slices by bulk copy (PCG), see setup
    size_t patch_smem[2] = {0, 0};     // dynamic shared memory of the patch kernel
    int node_grid[2] = {0, 0};  // resident node-kernel blocks (FP64, mixed)
    // CUDA graphs of the PCG loop by precision, and the workspaces each one was built on: the
    // buffers in it that can move while the operator lives (pcg_args grows them)
    cudaGraphExec_t loop[2] = {nullptr, nullptr};
    const void* loop_on[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};
    ~geo_op() {
        for (auto& g : loop)
            if (g) cudaGraphExecDestroy(g);
        if (h_state) cudaFreeHost(h_state);
    }
};

namespace geo {
namespace {

// PCG iterations per pass of the graph's loop. A pass ends with k_pcg_decide and the loop's
// own test (3 us together); the iterations behind a refresh or the end are launched as
// no-ops (see ST_IDLE). 8, 16 per pass: 6^3 FP64 solve 935, 900 us, 64^3 FP64 54.6, 54.2 ms,
// viscoelastic step 27x22x13 13.1, 12.8, elastic 48x48x24 mixed 42.9, 42.5, inversion step
// 48x48x32 35.6, 35.5; 4 per pass is slower still (16^3 FP64 by 6%).
constexpr int kChunk = 16;

inline unsigned nblk(int64_t n, int bs = 256) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(cdiv(n, bs), 148 * 64));
}

// Length of a DOF vector that the patch kernel copies own ranges of, rounded outwards to
// kNodeAlign nodes: whole 64-entry blocks (sub-arrays of one workspace stay aligned).
inline size_t padded_dofs(const geo_op* op) {
    return (size_t)((op->N + kNodeAlign - 1) / kNodeAlign * kNodeAlign * op->dpn + 63) / 64 * 64;
}

template <class T>
T* grow(DevBuf<T>& b, size_t n) {
    b.ensure(n);
    return b.p;
}

PatchView view(const geo_op* op) {
    PatchView v;
    v.E = op->E;
    v.N = op->N;
    v.n_patches = op->n_patches;
    v.max_local = op->max_local;
    v.dpn = op->dpn;
    v.pe = op->pe.p;
    v.po = op->po.p;
    v.pf = op->pf.p;
    v.foreign = op->foreign.p;
    v.lc = op->lc.p;
    v.lc32 = op->lc32.p;
    v.flags = op->flags.p;
    v.bound32 = op->pbound32.p;
    v.pfa = op->pfa.p;
    v.fids = op->fids.p;
    v.fflags = op->fflags.p;
    v.max_for = op->max_for;
    v.max_own = op->max_own;
    v.own_bulk = 0;
    v.fslot = op->fslot.p;
    v.rec = op->prec.p;
    return v;
}

// dynamic shared memory of the patch kernel (see patch_smem_bytes)
template <class K, class T>
size_t smem_bytes(const geo_op* op, int nbuf, bool own, int halo) {
    return nbuf == 2 ? patch_smem_bytes<K, T, 2>(op->max_local, op->max_for, op->max_own, own, halo)
                     : patch_smem_bytes<K, T, 1>(op->max_local, op->max_for, op->max_own, own, halo);
}

constexpr size_t kSmemLimit = 227 * 1024;

template <class F>
void with_kernels(const geo_op* op, F&& f) {
    // dispatch (physics, NQ) to concrete element kernels
    if (op->phys == 0) {
        if (op->nq == 1) f(ThermalK<double, 1>{}, ThermalK<float, 1>{});
        else f(ThermalK<double, 4>{}, ThermalK<float, 4>{});
    } else {
        if (op->nq == 1) f(ElasticK<double, 1>{}, ElasticK<float, 1>{});
        else f(ElasticK<double, 4>{}, ElasticK<float, 4>{});
    }
}

// Calls f(kernel) for the patch kernel of one mode, buffer count and halo mode.
template <class K, class T, int MODE, class F>
void with_patch_kernel(int nbuf, int halo, F&& f) {
    if (nbuf == 2) {
        if (halo == 2) f(k_patch<K, T, MODE, 2, 2>);
        else if (halo == 1) f(k_patch<K, T, MODE, 2, 1>);
        else f(k_patch<K, T, MODE, 2, 0>);
    } else {
        if (halo == 2) f(k_patch<K, T, MODE, 1, 2>);
        else if (halo == 1) f(k_patch<K, T, MODE, 1, 1>);
        else f(k_patch<K, T, MODE, 1, 0>);
    }
}

// Lets a kernel take `bytes` of dynamic shared memory. The attribute belongs to the
// kernel, not to the operator, so it is only ever raised: a smaller operator made later
// must not take it from a larger one that is still in use. It is set each time, since a
// cudaDeviceReset puts it back to its default.
template <class Kernel>
void allow_smem(Kernel k, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> allowed;
    int dev = 0;
    GEO_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    size_t& a = allowed[{dev, (const void*)k}];
    a = std::max(a, bytes);
    GEO_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)a));
}

// Resident blocks per SM of the PCG-mode patch kernel.
template <class K, class T>
int patch_residency(int nbuf, int halo, size_t smem) {
    int per_sm = 0;
    if (smem > kSmemLimit) return 0;
    with_patch_kernel<K, T, MODE_PCG>(nbuf, halo, [&](auto k) {
        allow_smem(k, smem);
        GEO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kPatchBS, smem));
    });
    return per_sm;
}

// Chooses the form of the patch kernel, from its resident blocks per SM:
// - two element-data buffers when they fit in shared memory, else one;
// - halo mode when the operator has slots, the slot list in the bulk copy when that
//   costs no resident block, else read by the flush from global memory;
// - own-node slices by bulk copy (PCG) when their buffer costs no resident block:
//   about 13 bytes per own node took one block per SM away on meshes whose patches hold
//   more nodes, which was slower than the plain gather (80^3, 112^3).
// GEO_PATCH_NBUF=1 and GEO_PATCH_HALO (0: atomics, 1: slots in shared memory, 2: slots
// from global) force a form, so that tests cover all of them on small meshes. Returns
// the grid.
template <class K, class T>
int setup_patch_kernels(geo_op* op, int slot) {
    const char* force_nbuf = std::getenv("GEO_PATCH_NBUF");
    const char* force = std::getenv("GEO_PATCH_HALO");
    const int forced = force && force[0] >= '0' && force[0] <= '2' && force[1] == 0 ? force[0] - '0' : -1;
    const bool halo_ok = op->halo_ok && forced != 0;
    int halo = halo_ok ? 2 : 0;
    int nbuf = 2;
    if (smem_bytes<K, T>(op, 2, false, halo) > kSmemLimit || (force_nbuf && std::strcmp(force_nbuf, "1") == 0)) nbuf = 1;
    int per_sm = patch_residency<K, T>(nbuf, halo, smem_bytes<K, T>(op, nbuf, false, halo));
    if (per_sm < 1) fail(GEO_ERR_UNSUPPORTED, "patch tables exceed shared memory (too many nodes per patch)");
    bool own = false;
    if (const int with_own = patch_residency<K, T>(nbuf, halo, smem_bytes<K, T>(op, nbuf, true, halo)); with_own >= per_sm) {
        own = true;
        per_sm = with_own;
    }
    if (halo_ok && forced != 2) {
        const int in_copy = patch_residency<K, T>(nbuf, 1, smem_bytes<K, T>(op, nbuf, own, 1));
        if (in_copy > 0 && (forced == 1 || in_copy >= per_sm)) {
            halo = 1;
            per_sm = in_copy;
        }
    }
    op->nbuf[slot] = nbuf;
    op->own_bulk[slot] = own;
    op->halo[slot] = halo;
    op->patch_smem[slot] = smem_bytes<K, T>(op, nbuf, own, halo);
    // MODE_FREE and MODE_LIFT launch with the same shared memory
    with_patch_kernel<K, T, MODE_FREE>(nbuf, halo, [&](auto k) { allow_smem(k, op->patch_smem[slot]); });
    with_patch_kernel<K, T, MODE_LIFT>(nbuf, halo, [&](auto k) { allow_smem(k, op->patch_smem[slot]); });
    return per_sm * op->ctx->sm_count;
}

// The PCG loop's kernels use programmatic dependent launch up to this many dofs: the next
// kernel's blocks then start on the SMs that the last blocks of the one before leave, and
// set up shared memory and the first patch's element copies before they wait. us per
// iteration without and with, and M dofs:
//   thermal FP64   40^3 (0.5) 32.3, 31.6; 56^3 (1.4) 73.2, 72.4; 64^3 (2.1) 93.9, 92.0;
//                  72^3 (3.0) 148.3, 151.2; 88^3 (5.5) 253.8, 259.2
//   thermal mixed  40^3 23.4, 22.0; 64^3 54.3, 52.8; 72^3 80.2, 79.3; 88^3 132.4, 130.2;
//                  128^3 (17.0) 330, 342
//   elastic FP64   32^3 (0.8) 59.0, 58.4; 44^3 (2.1) 137.7, 143.0; 52^3 (3.5) 224.6, 235.8
//   elastic mixed  32^3 29.0, 27.9; 44^3 61.7, 61.4; 52^3 92.2, 92.4
// One threshold for all four: it is right for thermal FP64 and elastic mixed; FP64
// elasticity would end near 1 M, thermal mixed above 5.5 M.
constexpr int64_t kDependentDofs = 2500000;

// A graph under construction whose nodes run one after the other. Built node by node, not
// captured from a stream: a capture is lost when another thread of the process
// synchronises the device meanwhile.
struct GraphChain {
    cudaGraph_t g;
    cudaGraphNode_t last = nullptr;
};

// Where a launch goes: to a stream, or to the end of a chain.
struct LaunchTo {
    cudaStream_t s = nullptr;
    GraphChain* chain = nullptr;
    LaunchTo(cudaStream_t stream) : s(stream) {}
    LaunchTo(GraphChain& c) : chain(&c) {}
};

template <class... P, size_t... I>
void add_kernel(GraphChain& c, bool dependent, void (*k)(P...), unsigned grid, int bs, size_t smem, std::tuple<P...>& args,
                std::index_sequence<I...>) {
    void* params[] = {&std::get<I>(args)...};
    cudaGraphNodeParams p{};
    p.type = cudaGraphNodeTypeKernel;
    p.kernel.func = (void*)k;
    p.kernel.gridDim = dim3(grid);
    p.kernel.blockDim = dim3(bs);
    p.kernel.sharedMemBytes = (unsigned)smem;
    p.kernel.kernelParams = params;
    cudaGraphEdgeData edge{};
    if (dependent) {
        edge.from_port = cudaGraphKernelNodePortProgrammatic;
        edge.type = cudaGraphDependencyTypeProgrammatic;
    }
    cudaGraphNode_t node;
    GEO_CUDA(cudaGraphAddNode_v2(&node, c.g, c.last ? &c.last : nullptr, c.last ? &edge : nullptr, c.last ? 1 : 0, &p));
    c.last = node;
}

// Launches k; in a chain with programmatic dependent launch when `dependent`: its blocks may
// start, up to their griddepcontrol.wait, while the kernel before it still runs. Only for
// kernels of the loop: k_patch reads the operator's element data before its wait, which
// must not be the output of the kernel before it.
template <class... P, class... A>
void launch_kernel(LaunchTo to, bool dependent, void (*k)(P...), unsigned grid, int bs, size_t smem, A... args) {
    std::tuple<P...> a{P(args)...};
    if (to.chain) {
        add_kernel(*to.chain, dependent, k, grid, bs, smem, a, std::index_sequence_for<P...>{});
        return;
    }
    std::apply([&](auto&... v) { k<<<grid, bs, smem, to.s>>>(v...); }, a);
    GEO_CUDA(cudaGetLastError());
}

// Blocks of the patch kernel: the resident ones, or one per patch.
unsigned patch_blocks(const geo_op* op, int slot) { return (unsigned)std::min(op->patch_grid[slot], op->n_patches); }

template <class K, class T, int MODE>
void launch_patch(const geo_op* op, int slot, LaunchTo to, const T* qd, const PatchArgs<T>& pa, bool dependent = false) {
    PatchView v = view(op);
    v.own_bulk = op->own_bulk[slot];
    with_patch_kernel<K, T, MODE>(op->nbuf[slot], op->halo[slot], [&](auto k) {
        launch_kernel(to, dependent, k, patch_blocks(op, slot), kPatchBS, op->patch_smem[slot], v, qd, (T)op->cl,
                      (T)op->cm, pa);
    });
}

// Halo slots (see k_halo_count): fslot in the fids
// segments (seg_total entries), the slot counts in flag bits 3-6, hbase, and the
// FP64 / FP32 slot arrays. Leaves op->halo_ok false (atomics kept) when some node
// has more than 15 foreign entries.
void build_halo_slots(geo_op* op, int64_t seg_total) {
    geo_ctx* ctx = op->ctx;
    cudaStream_t s = ctx->stream;
    const int64_t N = op->N, A = op->n_app;
    DevBuf<int32_t> cnt(N), keys(A), vals(A), vals2(A), slot_of(A), mx(1);
    GEO_CUDA(cudaMemsetAsync(cnt.p, 0, cnt.bytes(), s));
    k_halo_count<<<nblk(A), 256, 0, s>>>(op->foreign.p, A, cnt.p);
    check_launch(ctx, "k_halo_count");
    size_t b1 = 0, b2 = 0;
    int bits = 1;
    while (bits < 31 && (int64_t(1) << bits) < N) ++bits;
    GEO_CUDA(cub::DeviceReduce::Max(nullptr, b1, cnt.p, mx.p, N, s));
    GEO_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b2, op->foreign.p, keys.p, vals.p, vals2.p, A, 0, bits, s));
    DevBuf<unsigned char> tmp(std::max(b1, b2));
    GEO_CUDA(cub::DeviceReduce::Max(tmp.p, b1, cnt.p, mx.p, N, s));
    int hmax = 0;
    GEO_CUDA(cudaMemcpyAsync(&hmax, mx.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    sync(ctx, "halo counts");
    if (hmax > 15) return;
    k_iota<<<nblk(A), 256, 0, s>>>(A, vals.p);
    check_launch(ctx, "k_iota");
    GEO_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, b2, op->foreign.p, keys.p, vals.p, vals2.p, A, 0, bits, s));
    k_halo_slot_of<<<nblk(A), 256, 0, s>>>(vals2.p, A, slot_of.p);
    check_launch(ctx, "k_halo_slot_of");
    op->fslot.alloc(seg_total + kForeignAlign);
    GEO_CUDA(cudaMemsetAsync(op->fslot.p, 0, op->fslot.bytes(), s));
    k_patch_fslot<<<(unsigned)op->n_patches, 128, 0, s>>>(op->pf.p, op->pfa.p, slot_of.p, op->fslot.p);
    check_launch(ctx, "k_patch_fslot");
    const int64_t nch = (N + 31) / 32;
    DevBuf<int32_t> chunk(nch + 1);
    GEO_CUDA(cudaMemsetAsync(chunk.p, 0, chunk.bytes(), s));
    k_halo_flags<<<nblk(nch * 32), 256, 0, s>>>(cnt.p, N, op->flags.p, chunk.p);
    check_launch(ctx, "k_halo_flags");
    op->hbase.alloc(nch + 1);
    size_t b3 = 0;
    GEO_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, b3, chunk.p, op->hbase.p, nch + 1, s));
    tmp.ensure(b3);
    GEO_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, b3, chunk.p, op->hbase.p, nch + 1, s));
    int total = 0;
    GEO_CUDA(cudaMemcpyAsync(&total, op->hbase.p + nch, sizeof(int), cudaMemcpyDeviceToHost, s));
    sync(ctx, "halo slots");
    if (total != A) fail(GEO_ERR_CUDA, "halo slot count mismatch");
    op->halo64.alloc(A * op->dpn);
    op->halo32.alloc(A * op->dpn);
    // every pass writes all slots, those of Dirichlet entries too (the node update ignores them)
    GEO_CUDA(cudaMemsetAsync(op->halo64.p, 0, op->halo64.bytes(), s));
    GEO_CUDA(cudaMemsetAsync(op->halo32.p, 0, op->halo32.bytes(), s));
    op->halo_ok = true;
}

// Recomputes qdata, diagonal, char_diag and the Jacobi inverse from op->coef.
void refresh_coefficients(geo_op* op) {
    geo_ctx* ctx = op->ctx;
    cudaStream_t s = ctx->stream;
    const geo_mesh* m = op->mesh;
    reset_dev_err(ctx);
    const int nqd = (op->phys == 0 ? 6 : 10) * op->nq;
    op->qd64.ensure((size_t)nqd * op->n_patches * kPatchElems);
    op->qd32.ensure((size_t)nqd * op->n_patches * kPatchElems);
    GEO_CUDA(cudaMemsetAsync(op->qd64.p, 0, op->qd64.bytes(), s));
    GEO_CUDA(cudaMemsetAsync(op->qd32.p, 0, op->qd32.bytes(), s));
    if (op->nq == 1)
        k_qdata<1><<<(unsigned)cdiv(op->E, 128), 128, 0, s>>>(op->phys, m->xyz.p, m->conn.p, op->eperm.p, op->N, op->E,
                                                    op->coef.p, op->qd64.p, op->qd32.p, ctx->dev_err.p);
    else
        k_qdata<4><<<(unsigned)cdiv(op->E, 128), 128, 0, s>>>(op->phys, m->xyz.p, m->conn.p, op->eperm.p, op->N,
                                                              op->E, op->coef.p, op->qd64.p, op->qd32.p,
                                                              ctx->dev_err.p);
    check_launch(ctx, "k_qdata");
    {
        unsigned long long* knorm = grow(op->tmpu[0], (size_t)op->n_patches);
        GEO_CUDA(cudaMemsetAsync(knorm, 0, (size_t)op->n_patches * sizeof(unsigned long long), s));
        with_kernels(op, [&](auto k64, auto) {
            k_patch_knorm<decltype(k64)><<<(unsigned)cdiv(op->E, 128), 128, 0, s>>>(op->qd64.p, op->E, op->cl,
                                                                                   op->cm, knorm);
        });
        check_launch(ctx, "k_patch_knorm");
        op->pbound32.ensure(op->n_patches);
        k_patch_bound<<<(unsigned)cdiv(op->n_patches, 256), 256, 0, s>>>(op->pmaxinc.p, knorm, op->n_patches,
                                                                         op->pbound32.p);
        check_launch(ctx, "k_patch_bound");
        op->prec.ensure(op->n_patches);
        k_patch_records<<<(unsigned)cdiv(op->n_patches, 256), 256, 0, s>>>(view(op), op->prec.p);
        check_launch(ctx, "k_patch_records");
        sync(ctx, "patch bounds");
    }
    op->ediag.ensure((size_t)op->E * 10 * op->dpn);
    k_ediag<<<(unsigned)cdiv(op->E, 128), 128, 0, s>>>(op->phys, m->xyz.p, m->conn.p, op->N, op->E, op->coef.p,
                                                       op->cl, op->cm, op->ediag.p, ctx->dev_err.p);
    check_launch(ctx, "k_ediag");
    raise_dev_err(ctx, read_dev_err(ctx), "operator set-up");
    op->diag_orig.ensure(op->ndof);
    k_gather_diag<<<(unsigned)cdiv(op->ndof, 256), 256, 0, s>>>(m->inc_ptr.p, m->inc.p, op->ediag.p, op->N,
                                                                op->dpn, op->diag_orig.p);
    check_launch(ctx, "k_gather_diag");
    unsigned long long* mx = grow(op->tmpu[1], 1);
    GEO_CUDA(cudaMemsetAsync(mx, 0, sizeof(unsigned long long), s));
    k_max_abs<<<nblk(op->ndof), 256, 0, s>>>(op->diag_orig.p, op->ndof, mx);
    check_launch(ctx, "k_max_abs");
    unsigned long long bits = 0;
    GEO_CUDA(cudaMemcpyAsync(&bits, mx, sizeof(bits), cudaMemcpyDeviceToHost, s));
    sync(ctx, "char_diag");
    double maxd;
    std::memcpy(&maxd, &bits, sizeof(double));
    op->cd = maxd > 1.0 ? maxd : 1.0;  // assembly.rs:184-193
    op->dinv64.ensure(padded_dofs(op));
    op->dinv32.ensure(padded_dofs(op));
    op->diag_new.ensure(op->ndof);
    k_dinv<<<nblk(op->ndof), 256, 0, s>>>(op->nperm.p, op->flags.p, op->dpn, op->N, op->diag_orig.p, op->cd,
                                         op->dinv64.p, op->dinv32.p, op->diag_new.p);
    check_launch(ctx, "k_dinv");
    sync(ctx, "operator coefficients");
}

void set_coef(geo_op* op, const double* coef_e, double coef) {
    cudaStream_t s = op->ctx->stream;
    op->coef.ensure(op->E);
    if (coef_e) {
        GEO_CUDA(cudaMemcpyAsync(op->coef.p, coef_e, op->E * sizeof(double), cudaMemcpyDefault, s));
    } else {
        std::vector<double> h(op->E, coef);
        GEO_CUDA(cudaMemcpyAsync(op->coef.p, h.data(), op->E * sizeof(double), cudaMemcpyHostToDevice, s));
        sync(op->ctx, "coefficients");
    }
    op->coef_scalar = coef;
}

geo_op* create_op(geo_ctx* ctx, const geo_mesh* mesh, const geo_dofs* dofs, int phys, const double* coef_e,
                  double coef, double nu) {
    GEO_CHECK_ARG(ctx && mesh && dofs, "NULL argument");
    GEO_CHECK_ARG(dofs->n_nodes == mesh->n_nodes, "DOF manager and mesh disagree on the node count");
    const int dpn = phys == 0 ? 1 : 3;
    GEO_CHECK_ARG(dofs->dpn == dpn, phys == 0 ? "thermal operator needs 1 DOF per node"
                                              : "Elasticity requires 3 DOF per node");
    auto op = std::make_unique<geo_op>();
    op->ctx = ctx;
    op->ref.set(ctx);
    op->mesh = mesh;
    op->phys = phys;
    op->dpn = dpn;
    op->N = mesh->n_nodes;
    op->E = mesh->n_elem;
    op->ndof = op->N * dpn;
    op->nu = nu;
    op->cl = phys == 1 ? nu / ((1.0 + nu) * (1.0 - 2.0 * nu)) : 0.0;
    op->cm = phys == 1 ? 1.0 / (2.0 * (1.0 + nu)) : 0.0;
    cudaStream_t s = ctx->stream;
    ensure_inverse_map(const_cast<geo_mesh*>(mesh));
    PatchLayout L;
    build_patches(s, op->N, mesh->xyz.p, op->E, mesh->conn.p, L);
    op->n_patches = L.n_patches;
    op->max_local = L.max_local;
    op->eperm = std::move(L.eperm);
    op->nperm = std::move(L.nperm);
    op->pe = std::move(L.patch_elem);
    op->po = std::move(L.patch_own);
    op->pf = std::move(L.patch_foreign);
    op->foreign = std::move(L.foreign);
    op->lc = std::move(L.lc);
    op->lc32 = std::move(L.lc32);
    op->mask_orig.alloc(op->ndof);
    GEO_CUDA(cudaMemcpyAsync(op->mask_orig.p, dofs->mask.p, op->ndof, cudaMemcpyDeviceToDevice, s));
    // padded to 16 bytes: the patch kernel copies flag ranges rounded outwards to 16
    op->flags.alloc((size_t)(op->N + 15) / 16 * 16);
    GEO_CUDA(cudaMemsetAsync(op->flags.p, 0, op->flags.bytes(), s));
    op->g_new.alloc(op->ndof);
    k_node_flags<<<nblk(op->N), 256, 0, s>>>(op->nperm.p, L.shared.p, dofs->mask.p, dofs->vals.p, dpn, op->N,
                                             op->flags.p, op->g_new.p);
    check_launch(ctx, "k_node_flags");
    sync(ctx, "operator layout");
    {
        const int P = op->n_patches;
        std::vector<int32_t> pf(P + 1), pfa(P + 1), po(P + 1);
        GEO_CUDA(cudaMemcpy(pf.data(), op->pf.p, (P + 1) * sizeof(int32_t), cudaMemcpyDeviceToHost));
        GEO_CUDA(cudaMemcpy(po.data(), op->po.p, (P + 1) * sizeof(int32_t), cudaMemcpyDeviceToHost));
        for (int p = 0; p < P; ++p) op->max_own = std::max(op->max_own, po[p + 1] - po[p]);
        int64_t acc = 0;
        for (int p = 0; p < P; ++p) {
            const int nfor = pf[p + 1] - pf[p];
            op->max_for = std::max(op->max_for, nfor);
            pfa[p] = (int32_t)acc;
            acc += (nfor + kForeignAlign - 1) / kForeignAlign * kForeignAlign;
        }
        if (acc > INT32_MAX) fail(GEO_ERR_UNSUPPORTED, "too many foreign patch nodes");
        pfa[P] = (int32_t)acc;
        op->pfa.alloc(P + 1);
        GEO_CUDA(cudaMemcpyAsync(op->pfa.p, pfa.data(), (P + 1) * sizeof(int32_t), cudaMemcpyHostToDevice, s));
        op->fids.alloc(acc + kForeignAlign);
        op->fflags.alloc(acc + kForeignAlign);
        GEO_CUDA(cudaMemsetAsync(op->fids.p, 0, op->fids.bytes(), s));
        GEO_CUDA(cudaMemsetAsync(op->fflags.p, 0, op->fflags.bytes(), s));
        k_patch_foreign<<<(unsigned)P, 128, 0, s>>>(op->pf.p, op->pfa.p, op->foreign.p, op->flags.p, op->fids.p,
                                                  op->fflags.p);
        check_launch(ctx, "k_patch_foreign");
        sync(ctx, "foreign segments");
        op->n_app = pf[P];
        if ((dpn == 1 || dpn == 3) && op->n_app > 0) build_halo_slots(op.get(), acc);
    }
    // affine (straight-sided) elements use one metric per element
    DevBuf<int> aff(1);
    GEO_CUDA(cudaMemsetAsync(aff.p, 0, sizeof(int), s));
    k_affine_check<<<(unsigned)cdiv(op->E, 128), 128, 0, s>>>(mesh->xyz.p, mesh->conn.p, op->N, op->E, aff.p);
    check_launch(ctx, "k_affine_check");
    int curved = 0;
    GEO_CUDA(cudaMemcpyAsync(&curved, aff.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    sync(ctx, "affine check");
    op->nq = curved ? 4 : 1;
    if (op->max_local > 12288) fail(GEO_ERR_UNSUPPORTED, "patch tables exceed shared memory (too many nodes per patch)");
    op->pmaxinc.alloc(op->n_patches);
    k_patch_maxinc<<<(unsigned)op->n_patches, 128, (size_t)op->max_local * sizeof(int), s>>>(
        op->pe.p, op->po.p, op->pf.p, op->lc.p, op->pmaxinc.p);
    check_launch(ctx, "k_patch_maxinc");
    set_coef(op.get(), coef_e, coef);
    refresh_coefficients(op.get());
    with_kernels(op.get(), [&](auto k64, auto k32) {
        using K64 = decltype(k64);
        using K32 = decltype(k32);
        op->patch_grid[0] = setup_patch_kernels<K64, double>(op.get(), 0);
        op->patch_grid[1] = setup_patch_kernels<K32, float>(op.get(), 1);
    });
    with_kernels(op.get(), [&](auto k64, auto k32) {
        int per_sm = 0;
        if (op->halo[0])
            GEO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                &per_sm, k_pcg_update_halo<double, decltype(k64)::DPN, false>, kNodeBS, 0));
        else
            GEO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                &per_sm, k_pcg_update<double, decltype(k64)::DPN, false>, kNodeBS, 0));
        op->node_grid[0] = std::max(1, per_sm) * ctx->sm_count;
        if (op->halo[1])
            GEO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                &per_sm, k_pcg_update_halo<float, decltype(k32)::DPN, true>, kNodeBS, 0));
        else
            GEO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                &per_sm, k_pcg_update<float, decltype(k32)::DPN, true>, kNodeBS, 0));
        op->node_grid[1] = std::max(1, per_sm) * ctx->sm_count;
    });
    op->bvec.alloc(op->ndof);
    op->xvec.alloc(op->ndof);
    op->state.alloc(2);
    op->part.alloc((size_t)2 * std::max(op->node_grid[0], op->node_grid[1]));
    op->part_patch.alloc((size_t)2 * std::max(op->patch_grid[0], op->patch_grid[1]));
    GEO_CUDA(cudaMemsetAsync(op->state.p, 0, op->state.bytes(), s));
    GEO_CUDA(cudaMallocHost(&op->h_state, sizeof(PcgState)));
    return op.release();
}

void to_new(geo_op* op, const double* in_orig, double* out_new) {
    k_to_new<double, double><<<nblk(op->ndof), 256, 0, op->ctx->stream>>>(op->nperm.p, op->dpn, op->N, in_orig,
                                                                          out_new);
    check_launch(op->ctx, "k_to_new");
}
void to_orig(geo_op* op, const double* in_new, double* out_orig) {
    k_to_orig<double, double><<<nblk(op->ndof), 256, 0, op->ctx->stream>>>(op->nperm.p, op->dpn, op->N, in_new,
                                                                           out_orig);
    check_launch(op->ctx, "k_to_orig");
}

// The patch pass y = K x (MODE_FREE) or K g (MODE_LIFT) in patch numbering, device vectors
// of type T, foreign contributions in the halo slots in halo mode. A wait that runs out
// shows in ctx->dev_err, which the caller reads with its results.
template <class T>
void patch_pass(geo_op* op, const T* x, T* y, int mode) {
    geo_ctx* ctx = op->ctx;
    cudaStream_t s = ctx->stream;
    constexpr int slot = std::is_same<T, double>::value ? 0 : 1;
    if (!op->halo[slot]) GEO_CUDA(cudaMemsetAsync(y, 0, op->ndof * sizeof(T), s));
    reset_dev_err(ctx);
    with_kernels(op, [&](auto k64, auto k32) {
        using K = typename std::conditional<slot == 0, decltype(k64), decltype(k32)>::type;
        const T* qd = slot == 0 ? (const T*)op->qd64.p : (const T*)op->qd32.p;
        PatchArgs<T> pa{};
        pa.x = x;
        pa.y = y;
        pa.err = ctx->dev_err.p;
        if (op->halo[slot]) pa.halo = slot == 0 ? (T*)op->halo64.p : (T*)op->halo32.p;
        if (mode == MODE_FREE) launch_patch<K, T, MODE_FREE>(op, slot, s, qd, pa);
        else launch_patch<K, T, MODE_LIFT>(op, slot, s, qd, pa);
    });
    check_launch(ctx, "k_patch");
}

template <class T, class F>
void halo_finish(geo_op* op, const T* y, const F& fin) {
    const T* h = std::is_same<T, double>::value ? (const T*)op->halo64.p : (const T*)op->halo32.p;
    k_halo_finish<T, F><<<nblk(op->N), kNodeBS, 0, op->ctx->stream>>>(op->flags.p, op->hbase.p, h, op->nperm.p, op->dpn,
                                                                      op->N, y, fin);
    check_launch(op->ctx, "k_halo_finish");
}

// y = K_bc x, both in the original numbering (device), x and y of the pass in patch
// numbering in xn, yn.
template <class T>
void apply_orig(geo_op* op, const double* x, T* xn, T* yn, double* y) {
    cudaStream_t s = op->ctx->stream;
    const int64_t n = op->ndof;
    k_to_new<double, T><<<nblk(n), 256, 0, s>>>(op->nperm.p, op->dpn, op->N, x, xn);
    check_launch(op->ctx, "k_to_new");
    patch_pass<T>(op, xn, yn, MODE_FREE);
    if (op->halo[std::is_same<T, double>::value ? 0 : 1]) {
        halo_finish(op, yn, ApplyOut<T>{op->cd, xn, y});
    } else {
        k_dir_rows<T><<<nblk(n), 256, 0, s>>>(op->flags.p, op->dpn, n, op->cd, xn, yn);
        k_to_orig<T, double><<<nblk(n), 256, 0, s>>>(op->nperm.p, op->dpn, op->N, yn, y);
        check_launch(op->ctx, "k_to_orig");
    }
}

// f_bc (patch numbering) from f (original numbering), device buffers. The caller calls
// check_pass when it has synchronised anyway.
void lift_new(geo_op* op, const double* f_orig_dev, double* fbc_new) {
    cudaStream_t s = op->ctx->stream;
    double* kg = grow(op->tmp[5], (size_t)op->ndof);
    patch_pass<double>(op, op->g_new.p, kg, MODE_LIFT);
    if (op->halo[0]) {
        halo_finish(op, kg, LiftOut{op->cd, f_orig_dev, op->g_new.p, fbc_new});
    } else {
        double* fn = grow(op->tmp[4], (size_t)op->ndof);
        to_new(op, f_orig_dev, fn);
        k_lift_finish<<<nblk(op->ndof), 256, 0, s>>>(op->flags.p, op->dpn, op->ndof, op->cd, fn, op->g_new.p, kg,
                                                    fbc_new);
        check_launch(op->ctx, "k_lift_finish");
    }
}

// Synchronises and raises what a patch_pass reported.
void check_pass(geo_op* op, const char* what) { raise_dev_err(op->ctx, read_dev_err(op->ctx), what); }

// p is memory of the context's device, which a kernel may write in place of a copy: aligned
// for doubles too, which a copy does not ask for.
bool on_device(const geo_op* op, const double* p) {
    if (reinterpret_cast<uintptr_t>(p) % alignof(double) != 0) return false;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice && a.device == op->ctx->device;
}

// Blocks of a node kernel whose threads take `items` items: one wave of resident
// blocks, or as many as there is work for. Every block of the node update costs a partial
// that all blocks of the next patch kernel add up (pcg_fold); one of the start and refresh
// kernels a ticket and a partial in the last block's sum.
unsigned node_blocks(const geo_op* op, int slot, int64_t items) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(op->node_grid[slot], cdiv(items, kNodeBS)));
}

// Blocks of the node update. Its items: a 16-byte vector (one DOF per node; the atomics
// form), else one node (FP64) or two (FP32) of the three-DOF halo form.
unsigned update_blocks(const geo_op* op, int slot) {
    return node_blocks(op, slot, op->dpn == 1 || !op->halo[slot] ? cdiv(op->ndof, slot ? 4 : 2)
                                                                 : (slot ? cdiv(op->N, 2) : op->N));
}

// The node update of the PCG loop: the halo-mode kernel when the patch kernel runs
// in halo mode.
template <class K, class T, bool MIXED>
void launch_update(const geo_op* op, LaunchTo to, const NodeArgs<T>& na, bool dependent = false) {
    constexpr int slot = std::is_same<T, double>::value ? 0 : 1;
    const unsigned g = update_blocks(op, slot);
    launch_kernel(to, dependent, op->halo[slot] ? k_pcg_update_halo<T, K::DPN, MIXED> : k_pcg_update<T, K::DPN, MIXED>, g,
                  kNodeBS, 0, na);
}

// Adds one PCG iteration (patch kernel in PCG mode + node update) to the loop's graph.
template <class K, class T, bool MIXED>
void add_iteration(geo_op* op, GraphChain& c, const PatchArgs<T>& pa, const NodeArgs<T>& na) {
    constexpr bool dbl = std::is_same<T, double>::value;
    const T* qd = dbl ? (const T*)op->qd64.p : (const T*)op->qd32.p;
    const bool dependent = op->ndof <= kDependentDofs;
    launch_patch<K, T, MODE_PCG>(op, dbl ? 0 : 1, c, qd, pa, dependent);
    launch_update<K, T, MIXED>(op, c, na, dependent);
}

// Kernel arguments of the PCG loop over the operator's workspace (FP64 mode: r, q,
// p0, p1 in w64; mixed: w64 plus xs, r, q, p0, p1 in w32), allocated on first use.
struct PcgLaunchArgs {
    NodeArgs<double> n64{};
    NodeArgs<float> n32{};
    PatchArgs<double> p64{};
    PatchArgs<float> p32{};
};

PcgLaunchArgs pcg_args(geo_op* op, bool mixed) {
    const int64_t n = op->ndof;
    // sub-arrays at a common stride of whole 256-byte blocks, so that all vectors of
    // the node update share 16-byte alignment
    const int64_t np = (int64_t)padded_dofs(op);
    op->w64.ensure((size_t)(mixed ? 1 : 4) * np);
    if (mixed) op->w32.ensure((size_t)5 * np);
    PcgLaunchArgs a;
    NodeArgs<double>& n64 = a.n64;
    NodeArgs<float>& n32 = a.n32;
    PatchArgs<double>& p64 = a.p64;
    PatchArgs<float>& p32 = a.p32;
    n64.flags = n32.flags = op->flags.p;
    n64.n = n32.n = n;
    n64.dpn = n32.dpn = op->dpn;
    // the patch kernel reads the first copy of the state and writes the second, the
    // node update the other way round; each kernel folds the other's partials in
    n64.st = n32.st = op->state.p;
    n64.st_in = n32.st_in = op->state.p + 1;
    p64.st = p32.st = op->state.p;
    p64.st_out = p32.st_out = op->state.p + 1;
    p64.err = p32.err = &op->state.p->err;
    n64.part = n32.part = op->part.p;
    p64.part_in = p32.part_in = op->part.p;
    p64.part = p32.part = op->part_patch.p;
    n64.part_in = n32.part_in = op->part_patch.p;
    p64.n_in = (int)update_blocks(op, 0);
    p32.n_in = (int)update_blocks(op, 1);
    n64.n_in = (int)patch_blocks(op, 0);
    n32.n_in = (int)patch_blocks(op, 1);
    n64.b = n32.b = op->bvec.p;
    n64.x64 = n32.x64 = op->xvec.p;
    if (!mixed) {
        n64.x = op->xvec.p;
        n64.r = op->w64.p;
        n64.q = op->w64.p + np;
        n64.pbuf0 = op->w64.p + 2 * np;
        n64.pbuf1 = op->w64.p + 3 * np;
        n64.dinv = op->dinv64.p;
        p64.r = n64.r;
        p64.dinv = n64.dinv;
        p64.pbuf0 = n64.pbuf0;
        p64.pbuf1 = n64.pbuf1;
        p64.y = n64.q;
    } else {
        n32.w64 = op->w64.p;
        n32.x = op->w32.p;
        n32.r = op->w32.p + np;
        n32.q = op->w32.p + 2 * np;
        n32.pbuf0 = op->w32.p + 3 * np;
        n32.pbuf1 = op->w32.p + 4 * np;
        n32.dinv = op->dinv32.p;
        p32.r = n32.r;
        p32.dinv = n32.dinv;
        p32.pbuf0 = n32.pbuf0;
        p32.pbuf1 = n32.pbuf1;
        p32.y = n32.q;
        p32.xsol = n32.x;  // updated by the patch kernel (z-form of the mixed solver)
    }
    if (op->halo[0]) {
        n64.halo = p64.halo = op->halo64.p;
        n64.hbase = op->hbase.p;
        n32.halo64 = op->halo64.p;  // the mixed solver's FP64 refresh apply
        n32.hbase = op->hbase.p;
    }
    if (op->halo[1]) {
        n32.halo = p32.halo = op->halo32.p;
        n32.hbase = op->hbase.p;
    }
    return a;
}

// Writes the initial PcgState and launches the start kernels (x = 0, r = b, ||b||).
void pcg_start(geo_op* op, bool mixed, const PcgState& init, const PcgLaunchArgs& a) {
    cudaStream_t s = op->ctx->stream;
    GEO_CUDA(cudaMemcpyAsync(op->state.p, &init, sizeof(init), cudaMemcpyHostToDevice, s));
    const unsigned ng = node_blocks(op, mixed ? 1 : 0, op->ndof);
    if (mixed) {
        k_mixed_init1<<<ng, kNodeBS, 0, s>>>(a.n32);
        k_mixed_init2<<<ng, kNodeBS, 0, s>>>(a.n32);
    } else {
        k_pcg_init<double><<<ng, kNodeBS, 0, s>>>(a.n64);
    }
    check_launch(op->ctx, "pcg init");
}

// A conditional node behind `dep` (nullptr: none) in g; returns its body graph.
cudaGraph_t add_conditional(cudaGraph_t g, const cudaGraphNode_t* dep, cudaGraphConditionalHandle h,
                            cudaGraphConditionalNodeType type) {
    cudaGraphNodeParams p{};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = type;
    p.conditional.size = 1;
    cudaGraphNode_t node;
    GEO_CUDA(cudaGraphAddNode(&node, g, dep, dep ? 1 : 0, &p));
    return p.conditional.phGraph_out[0];
}

// The PCG loop as one graph: WHILE (again) { kChunk iterations, k_pcg_decide, mixed: IF
// (refresh) { the FP64 refresh } }. The kernels of a chunk turn into no-ops once the state
// says done or refresh. The host used to read the state after each chunk and to launch the
// refreshes (12 us each time): per iteration, before and now: 6^3 FP64 11.6 -> 11.4 us,
// 16^3 mixed 15.1 -> 13.5, elastic 8^3 mixed 17.7 -> 16.2, 48x48x32 mixed 23.5 -> 22.6.
cudaGraphExec_t build_loop(geo_op* op, bool mixed, const PcgLaunchArgs& la) {
    struct Graph {
        cudaGraph_t g = nullptr;
        ~Graph() {
            if (g) cudaGraphDestroy(g);
        }
    } graph;
    GEO_CUDA(cudaGraphCreate(&graph.g, 0));
    cudaGraphConditionalHandle again, refresh = 0;
    GEO_CUDA(cudaGraphConditionalHandleCreate(&again, graph.g, 1, cudaGraphCondAssignDefault));
    GraphChain body{add_conditional(graph.g, nullptr, again, cudaGraphCondTypeWhile)};
    if (mixed) GEO_CUDA(cudaGraphConditionalHandleCreate(&refresh, body.g, 0, cudaGraphCondAssignDefault));
    with_kernels(op, [&](auto k64, auto k32) {
        for (int i = 0; i < kChunk; ++i) {
            if (mixed) add_iteration<decltype(k32), float, true>(op, body, la.p32, la.n32);
            else add_iteration<decltype(k64), double, false>(op, body, la.p64, la.n64);
        }
    });
    if (mixed) launch_kernel(body, false, k_pcg_decide<true>, 1, kNodeBS, 0, op->state.p, la.p32.part_in, la.p32.n_in, again, refresh);
    else launch_kernel(body, false, k_pcg_decide<false>, 1, kNodeBS, 0, op->state.p, la.p64.part_in, la.p64.n_in, again, refresh);
    if (mixed) {
        NodeArgs<float> n32 = la.n32;
        n32.again = again;
        PatchArgs<double> ra{};
        ra.x = op->xvec.p;
        ra.y = op->w64.p;
        ra.err = &op->state.p->err;
        if (op->halo[0]) ra.halo = op->halo64.p;  // fixed-order foreign sums: bit-reproducible refresh
        const unsigned ng = node_blocks(op, 1, op->ndof);
        GraphChain rest{add_conditional(body.g, &body.last, refresh, cudaGraphCondTypeIf)};
        launch_kernel(rest, false, k_refresh_flush, ng, kNodeBS, 0, n32);
        with_kernels(op, [&](auto k64, auto) {
            launch_patch<decltype(k64), double, MODE_FREE>(op, 0, rest, op->qd64.p, ra);
        });
        launch_kernel(rest, false, op->halo[0] ? k_refresh_residual_halo : k_refresh_residual, ng, kNodeBS, 0, n32);
        launch_kernel(rest, false, k_refresh_rescale, ng, kNodeBS, 0, n32);
    }
    cudaGraphExec_t exec = nullptr;
    GEO_CUDA(cudaGraphInstantiate(&exec, graph.g, 0));
    return exec;
}

// Jacobi-PCG on K_bc; b_new / x_new in patch numbering (device). The loop is one graph
// that the device steers; the host reads the state when it has ended.
int solve_new(geo_op* op, const geo_cg_opts& o, geo_solver_stats* st) {
    geo_ctx* ctx = op->ctx;
    cudaStream_t s = ctx->stream;
    GEO_CHECK_ARG(o.use_preconditioner, "the matrix-free solver is Jacobi-preconditioned only");
    const bool mixed = o.precision == GEO_PRECISION_MIXED;
    PcgState init{};
    init.tol = o.tolerance;
    init.abs_tol = o.abs_tolerance;
    init.delta = o.reliable_delta;
    init.cd = op->cd;
    init.max_it = o.max_iterations;
    init.max_chunks = o.max_iterations + 65LL;
    const PcgLaunchArgs la = pcg_args(op, mixed);
    const NodeArgs<float>& n32 = la.n32;
    const unsigned ng = node_blocks(op, mixed ? 1 : 0, op->ndof);
    GEO_CUDA(cudaEventRecord(ctx->ev0, s));
    pcg_start(op, mixed, init, la);
    // (re)build the loop's graph when a buffer in it has moved: an FP64 solve, or the timing of
    // one, grows w64, which the mixed loop's refresh works in
    const int pi = mixed ? 1 : 0;
    const void* on[2] = {op->w64.p, mixed ? op->w32.p : nullptr};
    if (!op->loop[pi] || op->loop_on[pi][0] != on[0] || op->loop_on[pi][1] != on[1]) {
        if (op->loop[pi]) cudaGraphExecDestroy(op->loop[pi]);
        op->loop[pi] = nullptr;
        op->loop[pi] = build_loop(op, mixed, la);
        op->loop_on[pi][0] = on[0];
        op->loop_on[pi][1] = on[1];
    }
    GEO_CUDA(cudaGraphLaunch(op->loop[pi], s));
    GEO_CUDA(cudaMemcpyAsync(op->h_state, op->state.p, sizeof(PcgState), cudaMemcpyDeviceToHost, s));
    sync(ctx, "PCG loop");
    if (op->h_state->err) fail(GEO_ERR_TIMEOUT, "matrix-free PCG: a bounded device-side wait timed out");
    long long launches = (mixed ? 2 : 1) + op->h_state->chunks * (2 * kChunk + 1) + op->h_state->nupd * 4;
    if (mixed && !(op->h_state->flags & ST_CONVERGED)) {
        k_refresh_flush<<<ng, kNodeBS, 0, s>>>(n32);  // keep the FP32 correction
        check_launch(ctx, "final flush");
        launches += 1;
    }
    GEO_CUDA(cudaEventRecord(ctx->ev1, s));
    sync(ctx, "matrix-free PCG");
    float ms = 0.f;
    GEO_CUDA(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
    const PcgState& h = *op->h_state;
    PcgResult r{h.it, h.res, h.bnorm, (h.flags & ST_CONVERGED) ? 1 : 0, (h.flags & ST_BREAKDOWN) ? 1 : 0, h.nupd};
    const int status = r.converged ? GEO_OK : (r.breakdown ? GEO_ERR_BREAKDOWN : GEO_NOT_CONVERGED);
    fill_stats(st, r, ms * 1e-3, status);
    if (st) st->kernel_launches = launches;
    return status;
}

// Device time of the two kernels of one PCG iteration, launch by launch: `iters`
// iterations from x = 0, r = op->bvec, with the stopping, refresh and
// iteration-limit tests unable to fire (tolerances 0, delta 0, no limit), so every
// launch does the full work of an iteration of a real solve. Events are
// recorded on the context stream between the launches.
void time_iterations(geo_op* op, bool mixed, int iters, double* patch_ms, double* update_ms) {
    geo_ctx* ctx = op->ctx;
    cudaStream_t s = ctx->stream;
    PcgState init{};
    init.cd = op->cd;
    init.max_it = 1LL << 60;
    const PcgLaunchArgs la = pcg_args(op, mixed);
    pcg_start(op, mixed, init, la);
    std::vector<cudaEvent_t> ev((size_t)2 * iters + 1, nullptr);
    struct Guard {
        std::vector<cudaEvent_t>& v;
        ~Guard() {
            for (auto e : v)
                if (e) cudaEventDestroy(e);
        }
    } guard{ev};
    for (auto& e : ev) GEO_CUDA(cudaEventCreate(&e));
    with_kernels(op, [&](auto k64, auto k32) {
        for (int i = 0; i < iters; ++i) {
            GEO_CUDA(cudaEventRecord(ev[2 * i], s));
            if (mixed) launch_patch<decltype(k32), float, MODE_PCG>(op, 1, s, op->qd32.p, la.p32);
            else launch_patch<decltype(k64), double, MODE_PCG>(op, 0, s, op->qd64.p, la.p64);
            GEO_CUDA(cudaEventRecord(ev[2 * i + 1], s));
            if (mixed) launch_update<decltype(k32), float, true>(op, s, la.n32);
            else launch_update<decltype(k64), double, false>(op, s, la.n64);
        }
    });
    GEO_CUDA(cudaEventRecord(ev[2 * iters], s));
    check_launch(ctx, "timed PCG iterations");
    sync(ctx, "timed PCG iterations");
    PcgState h{};
    GEO_CUDA(cudaMemcpy(&h, op->state.p, sizeof(h), cudaMemcpyDeviceToHost));
    if (h.err) fail(GEO_ERR_TIMEOUT, "matrix-free PCG: a bounded device-side wait timed out");
    if (h.flags & ST_DONE) fail(GEO_ERR_BREAKDOWN, "timed PCG iterations stopped early (breakdown)");
    double tp = 0.0, tu = 0.0;
    for (int i = 0; i < iters; ++i) {
        float a = 0.f, b = 0.f;
        GEO_CUDA(cudaEventElapsedTime(&a, ev[2 * i], ev[2 * i + 1]));
        GEO_CUDA(cudaEventElapsedTime(&b, ev[2 * i + 1], ev[2 * i + 2]));
        tp += a;
        tu += b;
    }
    *patch_ms = tp / iters;
    *update_ms = tu / iters;
}

int finish_status(geo_ctx* ctx, int status) {
    if (status != GEO_OK)
        record_error(ctx, status, status == GEO_ERR_BREAKDOWN ? "CG breakdown: |p^T A p| < 1e-30"
                                                              : "CG did not converge");
    return status;
}

// ---- failure-detection test kernel: block 0 leaves without arriving
__global__ void k_barrier_probe(GridSync* gs, unsigned long long timeout_ns) {
    if (blockIdx.x == 0) return;
    grid_barrier(gs, gridDim.x, timeout_ns);
}

}  // namespace
}  // namespace geo

using namespace geo;

extern "C" {

int geo_thermal_operator_create(geo_ctx* ctx, const geo_mesh* mesh, const geo_dofs* dofs, const double* k_e,
                                double k, geo_op** out) {
    GEO_API_BEGIN(ctx)
    GEO_CHECK_ARG(out, "out is NULL");
    *out = create_op(ctx, mesh, dofs, 0, k_e, k, 0.0);
    GEO_API_END
}

int geo_elasticity_operator_create(geo_ctx* ctx, const geo_mesh* mesh, const geo_dofs* dofs, const double* E_e,
                                   double E, double nu, geo_op** out) {
    GEO_API_BEGIN(ctx)
    GEO_CHECK_ARG(out, "out is NULL");
    GEO_CHECK_ARG(nu > -1.0 && nu < 0.5, "Poisson's ratio must be in (-1, 0.5)");
    *out = create_op(ctx, mesh, dofs, 1, E_e, E, nu);
    GEO_API_END
}

int geo_op_set_coefficients(geo_op* op, const double* coef_e, double coef) {
    GEO_API_BEGIN(op ? op->ctx : nullptr)
    GEO_CHECK_ARG(op, "NULL operator");
    set_coef(op, coef_e, coef);
    refresh_coefficients(op);
    GEO_API_END
}

int geo_op_info(const geo_op* op, int64_t* n_dofs, int64_t* n_elem, double* char_diag) {
    if (!op) return GEO_ERR_INVALID_ARG;
    if (n_dofs) *n_dofs = op->ndof;
    if (n_elem) *n_elem = op->E;
    if (char_diag) *char_diag = op->cd;
    return GEO_OK;
}

int geo_op_apply(geo_op* op, const double* x, double* y, int32_t precision) {
    GEO_API_BEGIN(op ? op->ctx : nullptr)
    GEO_CHECK_ARG(op && x && y, "NULL argument");
    cudaStream_t s = op->ctx->stream;
    const int64_t n = op->ndof;
    const double* dx = stage_in(x, n, op->tmp[0], s);
    double* yo = on_device(op, y) ? y : grow(op->tmp[3], (size_t)n);
    if (precision == GEO_PRECISION_MIXED)
        apply_orig<float>(op, dx, grow(op->tmp32[0], (size_t)n), grow(op->tmp32[1], (size_t)n), yo);
    else apply_orig<double>(op, dx, grow(op->tmp[1], (size_t)n), grow(op->tmp[2], (size_t)n), yo);
    if (yo != y) copy_out(y, yo, n, s);
    check_pass(op, "matrix-free apply");
    GEO_API_END
}

int geo_op_lift_rhs(geo_op* op, const double* f, double* f_bc) {
    GEO_API_BEGIN(op ? op->ctx : nullptr)
    GEO_CHECK_ARG(op && f && f_bc, "NULL argument");
    cudaStream_t s = op->ctx->stream;
    const int64_t n = op->ndof;
    const double* df = stage_in(f, n, op->tmp[0], s);
    double* fb = grow(op->tmp[1], (size_t)n);
    double* fo = on_device(op, f_bc) ? f_bc : grow(op->tmp[2], (size_t)n);
    lift_new(op, df, fb);
    to_orig(op, fb, fo);
    if (fo != f_bc) copy_out(f_bc, fo, n, s);
    check_pass(op, "matrix-free lift");
    GEO_API_END
}

int geo_op_diagonal(geo_op* op, double* diag) {
    GEO_API_BEGIN(op ? op->ctx : nullptr)
    GEO_CHECK_ARG(op && diag, "NULL argument");
    double* d = grow(op->tmp[0], (size_t)op->ndof);
    to_orig(op, op->diag_new.p, d);
    copy_out(diag, d, op->ndof, op->ctx->stream);
    sync(op->ctx, "geo_op_diagonal");
    GEO_API_END
}

int geo_cg_solve_matfree(geo_op* op, const double* b, const geo_cg_opts* opts, double* x, geo_solver_stats* st) {
    GEO_API_BEGIN(op ? op->ctx : nullptr)
    GEO_CHECK_ARG(op && b && x, "NULL argument");
    geo_cg_opts o;
    cg_opts_fill(opts, o);
    cudaStream_t s = op->ctx->stream;
    const int64_t n = op->ndof;
    const double* db = stage_in(b, n, op->tmp[0], s);
    to_new(op, db, op->bvec.p);
    const int status = solve_new(op, o, st);
    double* dst = x;
    if (!is_device_ptr(x)) dst = grow(op->tmp[1], (size_t)n);
    to_orig(op, op->xvec.p, dst);
    if (dst != x) copy_out(x, dst, n, s);
    sync(op->ctx, "geo_cg_solve_matfree");
    return finish_status(op->ctx, status);
    GEO_API_END
}

int geo_op_element_gradient(geo_op* op, const double* u, const double* lambda, double* grad_e) {
    GEO_API_BEGIN(op ? op->ctx : nullptr)
    GEO_CHECK_ARG(op && u && lambda && grad_e, "NULL argument");
    cudaStream_t s = op->ctx->stream;
    const double* du = stage_in(u, op->ndof, op->tmp[0], s);
    const double* dl = stage_in(lambda, op->ndof, op->tmp[1], s);
    double* g = grow(op->tmp[6], (size_t)op->E);
    const geo_mesh* m = op->mesh;
    k_elem_gradient<<<(unsigned)cdiv(op->E, 128), 128, 0, s>>>(op->phys, m->xyz.p, m->conn.p, op->N, op->E,
                                                               op->coef.p, op->cl, op->cm, op->mask_orig.p, du, dl,
                                                               g);
    check_launch(op->ctx, "k_elem_gradient");
    copy_out(grad_e, g, op->E, s);
    sync(op->ctx, "geo_op_element_gradient");
    GEO_API_END
}

int geo_forward(geo_op* op, const double* f, const geo_cg_opts* opts, double* u, geo_solver_stats* st) {
    GEO_API_BEGIN(op ? op->ctx : nullptr)
    GEO_CHECK_ARG(op && f && u, "NULL argument");
    geo_cg_opts o;
    cg_opts_fill(opts, o);
    cudaStream_t s = op->ctx->stream;
    const int64_t n = op->ndof;
    const double* df = stage_in(f, n, op->tmp[0], s);
    lift_new(op, df, op->bvec.p);
    const int status = solve_new(op, o, st);
    double* dst = u;
    if (!is_device_ptr(u)) dst = grow(op->tmp[1], (size_t)n);
    to_orig(op, op->xvec.p, dst);
    if (dst != u) copy_out(u, dst, n, s);
    check_pass(op, "matrix-free lift");
    return finish_status(op->ctx, status);
    GEO_API_END
}

int geo_vjp(geo_op* op, const double* f, const double* u, const double* dJ_du, const geo_cg_opts* opts,
            double* dJ_dlncoef, geo_solver_stats* st) {
    GEO_API_BEGIN(op ? op->ctx : nullptr)
    GEO_CHECK_ARG(op && dJ_du && dJ_dlncoef && (u || f), "NULL argument");
    geo_cg_opts o;
    cg_opts_fill(opts, o);
    cudaStream_t s = op->ctx->stream;
    const int64_t n = op->ndof;
    double* lo = grow(op->tmp[3], (size_t)n);
    double* ge = grow(op->tmp[6], (size_t)op->E);
    const double* du = nullptr;
    if (u) {
        du = stage_in(u, n, op->tmp[0], s);
    } else {
        // recompute the forward solution instead of storing it
        const double* df = stage_in(f, n, op->tmp[0], s);
        lift_new(op, df, op->bvec.p);
        const int fs = solve_new(op, o, nullptr);
        check_pass(op, "matrix-free lift");
        if (fs != GEO_OK) return finish_status(op->ctx, fs);
        double* uo = grow(op->tmp[2], (size_t)n);
        to_orig(op, op->xvec.p, uo);
        du = uo;
    }
    // adjoint right-hand side: dJ/du on free DOFs, zero on Dirichlet DOFs (K_bc
    // is symmetric and its Dirichlet rows are decoupled, so lambda_D = 0)
    const double* dg = stage_in(dJ_du, n, op->tmp[1], s);
    to_new(op, dg, op->bvec.p);
    k_zero_dir<double><<<nblk(n), 256, 0, s>>>(op->flags.p, op->dpn, n, op->bvec.p);
    check_launch(op->ctx, "adjoint rhs");
    // The adjoint system is linear in its right-hand side: solve with dJ/du scaled
    // so that its Jacobi-preconditioned form D^-1 b has unit max-norm (lambda is
    // then O(1)) and scale lambda back, so that the absolute breakdown and
    // stopping thresholds of the CG loop do not depend on the misfit's units or
    // on the stiffness scale.
    unsigned long long* mx = grow(op->tmpu[1], 1);
    GEO_CUDA(cudaMemsetAsync(mx, 0, sizeof(unsigned long long), s));
    k_max_abs_scaled<<<nblk(n), 256, 0, s>>>(op->bvec.p, op->dinv64.p, n, mx);
    unsigned long long bits = 0;
    GEO_CUDA(cudaMemcpyAsync(&bits, mx, sizeof(bits), cudaMemcpyDeviceToHost, s));
    sync(op->ctx, "adjoint scale");
    double zmax;
    std::memcpy(&zmax, &bits, sizeof(double));
    int status = GEO_OK;
    if (zmax > 0.0) {
        k_scale<<<nblk(n), 256, 0, s>>>(op->bvec.p, n, 1.0 / zmax);  // b / zmax
        status = solve_new(op, o, st);
        k_scale<<<nblk(n), 256, 0, s>>>(op->xvec.p, n, zmax);        // lambda = zmax * lambda_scaled
    } else {
        GEO_CUDA(cudaMemsetAsync(op->xvec.p, 0, n * sizeof(double), s));
    }
    to_orig(op, op->xvec.p, lo);
    const geo_mesh* m = op->mesh;
    k_elem_gradient<<<(unsigned)cdiv(op->E, 128), 128, 0, s>>>(op->phys, m->xyz.p, m->conn.p, op->N, op->E,
                                                               op->coef.p, op->cl, op->cm, op->mask_orig.p, du,
                                                               lo, ge);
    check_launch(op->ctx, "k_elem_gradient");
    copy_out(dJ_dlncoef, ge, op->E, s);
    sync(op->ctx, "geo_vjp");
    return finish_status(op->ctx, status);
    GEO_API_END
}

int geo_op_time_pcg_kernels(geo_op* op, const double* b, int32_t precision, int32_t iterations, double* patch_ms,
                            double* update_ms) {
    GEO_API_BEGIN(op ? op->ctx : nullptr)
    GEO_CHECK_ARG(op && b && patch_ms && update_ms, "NULL argument");
    GEO_CHECK_ARG(iterations >= 1 && iterations <= 4096, "iterations must be in [1, 4096]");
    cudaStream_t s = op->ctx->stream;
    const double* db = stage_in(b, op->ndof, op->tmp[0], s);
    to_new(op, db, op->bvec.p);
    time_iterations(op, precision == GEO_PRECISION_MIXED, iterations, patch_ms, update_ms);
    GEO_API_END
}

int geo_op_destroy(geo_op* op) {
    if (!op) return GEO_OK;
    cudaSetDevice(op->ctx->device);
    cudaStreamSynchronize(op->ctx->stream);
    delete op;
    return GEO_OK;
}

int geo_debug_barrier_timeout(geo_ctx* ctx, double timeout_seconds) {
    GEO_API_BEGIN(ctx)
    GEO_CHECK_ARG(ctx, "NULL context");
    GEO_CHECK_ARG(timeout_seconds > 0 && timeout_seconds <= 5.0, "timeout must be in (0, 5] seconds");
    DevBuf<GridSync> gs(1);
    GEO_CUDA(cudaMemsetAsync(gs.p, 0, sizeof(GridSync), ctx->stream));
    const int nb = std::min(persistent_blocks(ctx, k_barrier_probe, 128, 0), 2 * ctx->sm_count);
    GridSync* gp = gs.p;
    unsigned long long tns = (unsigned long long)(timeout_seconds * 1e9);
    void* params[] = {&gp, &tns};
    GEO_CUDA(cudaLaunchCooperativeKernel((const void*)k_barrier_probe, dim3(nb), dim3(128), params, 0, ctx->stream));
    GridSync g{};
    GEO_CUDA(cudaMemcpyAsync(&g, gs.p, sizeof(g), cudaMemcpyDeviceToHost, ctx->stream));
    sync(ctx, "barrier probe");
    if (g.error & DEV_ERR_TIMEOUT) fail(GEO_ERR_TIMEOUT, "device-side grid barrier timed out (as the probe intends)");
    GEO_API_END
}

}  // extern "C"
