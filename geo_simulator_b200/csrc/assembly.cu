// K2/K3: deterministic CSR assembly and Dirichlet elimination (FP64).
//
// The reference collects 100 (900) triplets per element and lets sprs sort and
// merge them (assembly.rs:69-117, :389-437). Here a node -> (element, local)
// inverse map, sorted by element, drives everything:
//   * the sparsity pattern of row i is the sorted union of the nodes of the
//     elements incident to node i (one warp per row, bitonic sort in shared
//     memory) -- identical to sprs' sorted, merged structure;
//   * each row sums its contributions in ascending element order, the order in
//     which the reference's triplets reach every (row, col) entry. The element rows are
//     formed from per-element geometry as they are added, so no element matrix is
//     stored, and the places of an element's nodes in a row come with the pattern;
//   * load vectors gather per node in the same order (assembly.rs:130-154).
// No atomics touch values, so every result is bit-reproducible run to run.
#include <cub/cub.cuh>

#include <algorithm>
#include <climits>

#include "objects.h"
#include "tet10.cuh"

namespace geo {

void element_thermal_load(geo_ctx* ctx, const geo_mesh* m, double Q, double* out);
void element_gravity_load(geo_ctx* ctx, const geo_mesh* m, double rho, const double g[3], double* out);

namespace {

constexpr int kPatCap = 1024;  // candidate columns per node row (10 x incident elements)
constexpr int kPatWarps = 4;

inline unsigned blocks(int64_t n, int bs) { return (unsigned)std::max<int64_t>(1, cdiv(n, bs)); }

template <class T>
void exclusive_scan(const T* in, T* out, int64_t n, cudaStream_t s) {
    size_t tmp_bytes = 0;
    GEO_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, in, out, n, s));
    DevBuf<unsigned char> tmp(tmp_bytes + 16);
    GEO_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tmp_bytes, in, out, n, s));
    GEO_CUDA(cudaStreamSynchronize(s));
}

// ---------------------------------------------------------------- inverse map
__global__ void k_inc_count(const int32_t* __restrict__ conn, int64_t E, int32_t* __restrict__ cnt) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= E * 10) return;
    atomicAdd(&cnt[conn[t]], 1);  // conn is SoA [10][E]; t = l*E + e
}

__global__ void k_inc_fill(const int32_t* __restrict__ conn, int64_t E, const int32_t* __restrict__ ptr,
                           int32_t* __restrict__ cursor, int32_t* __restrict__ inc) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= E * 10) return;
    const int64_t l = t / E, e = t % E;
    const int32_t n = conn[t];
    const int32_t pos = ptr[n] + atomicAdd(&cursor[n], 1);
    inc[pos] = (int32_t)(e * 10 + l);
}

// Sorts every node's incidence segment ascending (element-major) by insertion sort.
__global__ void k_inc_sort(const int32_t* __restrict__ ptr, int32_t* __restrict__ inc, int64_t N) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int32_t b = ptr[i], e = ptr[i + 1];
    for (int32_t p = b + 1; p < e; ++p) {
        const int32_t v = inc[p];
        int32_t q = p - 1;
        while (q >= b && inc[q] > v) {
            inc[q + 1] = inc[q];
            --q;
        }
        inc[q + 1] = v;
    }
}

// ---------------------------------------------------------------- node pattern
// One warp per node row: gather candidate columns, bitonic sort, count / emit
// the distinct ones and, with out_pos, the places of every incident element's nodes
// among them (geo_mesh::pat_pos). err[0] gets DEV_ERR_BOUNDS when a row exceeds
// kPatCap, err[1] the largest row beyond 256, err[2] is set when an element lists a node
// twice (two neighbouring incidences of the node, which are sorted by element).
__global__ void __launch_bounds__(32 * kPatWarps)
k_pattern(const int32_t* __restrict__ conn, int64_t E, const int32_t* __restrict__ ptr,
          const int32_t* __restrict__ inc, int64_t N, int64_t* __restrict__ row_cnt,
          const int64_t* __restrict__ out_ptr, int32_t* __restrict__ out_idx, uint32_t* __restrict__ out_pos,
          int* err) {
    __shared__ int32_t sbuf[kPatWarps][kPatCap];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int32_t* buf = sbuf[w];
    const int64_t nwarps = (int64_t)gridDim.x * kPatWarps;
    for (int64_t i = blockIdx.x * (int64_t)kPatWarps + w; i < N; i += nwarps) {
        const int32_t b = ptr[i];
        const int deg = ptr[i + 1] - b;
        const int nc = 10 * deg;
        if (nc > kPatCap) {
            if (lane == 0) {
                atomicOr(err, DEV_ERR_BOUNDS);
                if (row_cnt) row_cnt[i] = 0;
            }
            continue;
        }
        int P = 32;
        while (P < nc) P <<= 1;
        for (int t = lane; t < P; t += 32) {
            int32_t v = INT_MAX;
            if (t < nc) {
                const int32_t el = inc[b + t / 10];
                v = conn[(int64_t)(t % 10) * E + el / 10];
            }
            buf[t] = v;
        }
        __syncwarp();
        for (int k = 2; k <= P; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int t = lane; t < P; t += 32) {
                    const int ixj = t ^ j;
                    if (ixj > t) {
                        const int32_t a = buf[t], c = buf[ixj];
                        const bool up = (t & k) == 0;
                        if ((a > c) == up) {
                            buf[t] = c;
                            buf[ixj] = a;
                        }
                    }
                }
                __syncwarp();
            }
        int run = 0;
        const int64_t base = out_idx ? out_ptr[i] : 0;
        for (int t0 = 0; t0 < P; t0 += 32) {
            const int t = t0 + lane;
            const int32_t v = buf[t];
            const bool uniq = v != INT_MAX && (t == 0 || buf[t - 1] != v);
            const unsigned bal = __ballot_sync(0xffffffffu, uniq);
            const int at = run + __popc(bal & ((1u << lane) - 1u));  // <= t
            if (out_idx && uniq) out_idx[base + at] = v;
            // compacted in place; entry t0 + 31, which the next chunk compares with, keeps its value
            if (uniq) buf[at] = v;
            __syncwarp();
            run += __popc(bal);
        }
        if (row_cnt && lane == 0) {
            row_cnt[i] = run;
            if (run > 256) atomicMax(err + 1, run);
        }
        if (row_cnt)
            for (int t = lane; t + 1 < deg; t += 32)
                if (inc[b + t] / 10 == inc[b + t + 1] / 10) atomicOr(err + 2, 1);
        if (out_pos)
            for (int t = lane; t < 3 * deg; t += 32) {  // word t % 3 of incidence t / 3
                const int64_t e = inc[b + t / 3] / 10;
                uint32_t word = 0;
                for (int j = 0; j < 4; ++j) {
                    const int l = 4 * (t % 3) + j;
                    if (l >= 10) break;
                    const int32_t c = conn[(int64_t)l * E + e];
                    int lo = 0, hi = run;
                    while (lo < hi) {
                        const int m = (lo + hi) >> 1;
                        if (buf[m] < c) lo = m + 1;
                        else hi = m;
                    }
                    word |= (uint32_t)lo << (8 * j);
                }
                out_pos[3 * (int64_t)b + t] = word;
            }
        __syncwarp();
    }
}

__device__ __forceinline__ int64_t find_col(const int32_t* __restrict__ idx, int64_t b, int64_t e, int32_t c) {
    // lower_bound on the sorted column list [b, e)
    while (b < e) {
        const int64_t m = (b + e) >> 1;
        if (idx[m] < c) b = m + 1;
        else e = m;
    }
    return b;
}

// ---------------------------------------------------------------- values
// Rows (thermal: nodes, elastic: nodes with their three DOF rows) of one block of the
// value kernels. Its accumulators are the block's contiguous piece of the matrix in
// shared memory, copied out whole. A block of 64 thermal rows of the cube holds 11 KB (edge
// midpoints) to 33 KB (vertices), one of 32 elastic nodes 53 to 150 KB.
constexpr int kRowsT = 64;
constexpr int kRowsE = 32;
constexpr int kMetricT = 24;  // doubles per element: G (6) at the four points
constexpr int kMetricE = 40;  // J^{-1} (9) and w |det J| E at the four points

__global__ void k_block_max(const int64_t* __restrict__ pptr, int64_t N, unsigned long long* out) {
    const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (b * kRowsE >= N) return;
    const int64_t e0 = b * kRowsE;
    atomicMax(out + 1, (unsigned long long)(pptr[min(N, e0 + kRowsE)] - pptr[e0]));
    if (b % (kRowsT / kRowsE) == 0) atomicMax(out, (unsigned long long)(pptr[min(N, e0 + kRowsT)] - pptr[e0]));
}

// Isoparametric geometry at 4-point QP q of element e (basis.rs:196-247): adj(J) and det J.
__device__ __forceinline__ double metric_geometry(const double* __restrict__ xyz, const int32_t* __restrict__ conn,
                                                  int64_t N, int64_t E, int64_t e, int q, double (&A)[3][3]) {
    double X[10][3], L[4], J[3][3];
#pragma unroll
    for (int l = 0; l < 10; ++l) {
        const int64_t n = conn[l * E + e];
        X[l][0] = xyz[n];
        X[l][1] = xyz[N + n];
        X[l][2] = xyz[2 * N + n];
    }
    qp4(q, L);
    jacobian10(X, L, J);
    adj3(J, A);
    return det3(J);
}

// G_q = (k w / |det J|) adj(J) adj(J)^T, packed [xx xy xz yy yz zz]; thread (e, q)
__global__ void __launch_bounds__(128) k_thermal_metric(const double* __restrict__ xyz, const int32_t* __restrict__ conn,
                                                        int64_t N, int64_t E, const double* __restrict__ k_e, double k,
                                                        double* __restrict__ G, int* err) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= E * 4) return;
    const int64_t e = t / 4;
    double A[3][3];
    const double d = metric_geometry(xyz, conn, N, E, e, (int)(t % 4), A);
    if (d == 0.0) {
        atomicOr(err, DEV_ERR_SINGULAR);
        return;
    }
    const double s = (k_e ? k_e[e] : k) * kQw / fabs(d);
    double2* o = reinterpret_cast<double2*>(G + 6 * t);
    auto dot = [&](int r, int c) { return s * (A[r][0] * A[c][0] + A[r][1] * A[c][1] + A[r][2] * A[c][2]); };
    o[0] = make_double2(dot(0, 0), dot(0, 1));
    o[1] = make_double2(dot(0, 2), dot(1, 1));
    o[2] = make_double2(dot(1, 2), dot(2, 2));
}

// J^{-1} (row-major) and w |det J| E_e; thread (e, q)
__global__ void __launch_bounds__(128) k_elastic_metric(const double* __restrict__ xyz, const int32_t* __restrict__ conn,
                                                        int64_t N, int64_t E, const double* __restrict__ E_e, double Ey,
                                                        double* __restrict__ geom, int* err) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= E * 4) return;
    const int64_t e = t / 4;
    double A[3][3];
    const double d = metric_geometry(xyz, conn, N, E, e, (int)(t % 4), A);
    if (d == 0.0) {
        atomicOr(err, DEV_ERR_SINGULAR);
        return;
    }
    double* o = geom + 10 * t;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) o[3 * r + c] = A[r][c] / d;
    o[9] = kQw * fabs(d) * (E_e ? E_e[e] : Ey);
}

// Reference gradients of node l (0..9, known at run time) at the four points, from a
// shared table: g[q][a] = tab[(3 q + a) * 10 + l].
__device__ __forceinline__ void fill_gradients(double* tab) {
    for (int t = threadIdx.x; t < 40; t += blockDim.x) {
        const int q = t / 10, l = t % 10;
        double L[4], d[4] = {0.0, 0.0, 0.0, 0.0};
        for (int m = 0; m < 4; ++m) L[m] = m == q ? kQa : kQb;
        if (l < 4) {
            d[l] = 4.0 * L[l] - 1.0;
        } else {
            const int m = edge_v(l - 4, 0), n = edge_v(l - 4, 1);
            d[m] = 4.0 * L[n];
            d[n] = 4.0 * L[m];
        }
        for (int a = 0; a < 3; ++a) tab[(3 * q + a) * 10 + l] = d[a + 1] - d[0];
    }
}

// 32-byte load (one sector) of four doubles, 32-byte aligned
__device__ __forceinline__ void load4(const double* p, double& a, double& b, double& c, double& d) {
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a), "=d"(b), "=d"(c), "=d"(d) : "l"(p));
}

struct RowArgs {
    const int32_t* conn;
    const int32_t* ptr;
    const int32_t* inc;
    const int64_t* pptr;
    const int32_t* pidx;
    const uint32_t* pos;
    const double* metric;
    int64_t N, E;
    int32_t* indices;  // elastic: written here; thermal: the pattern's, copied by the host
    double* data;
    double lam, mu;
    int64_t lo, hi;  // the launch takes the blocks of more than lo and at most hi entries
};

// row[at[j]] += y[j] for an element's ten columns: all loads, then all stores, where they
// are distinct entries; one after the other where two may be the same (REPEATS: some element
// of the mesh lists a node twice).
template <bool REPEATS>
__device__ __forceinline__ void add_columns(double* row, const int (&at)[10], const double (&y)[10]) {
    if constexpr (REPEATS) {
#pragma unroll
        for (int j = 0; j < 10; ++j) row[at[j]] = __dadd_rn(row[at[j]], y[j]);
    } else {
        double v[10];
#pragma unroll
        for (int j = 0; j < 10; ++j) v[j] = row[at[j]];
#pragma unroll
        for (int j = 0; j < 10; ++j) row[at[j]] = __dadd_rn(v[j], y[j]);
    }
}

// Place of the element's local node j in its row: from the pattern's bytes, or by
// search in the row [rb, re).
template <bool SMEM>
__device__ __forceinline__ int row_place(const RowArgs& a, const uint32_t (&w)[3], int j, int64_t e, int64_t rb,
                                         int64_t re) {
    if (SMEM) return (int)((w[j / 4] >> (8 * (j % 4))) & 0xffu);
    return (int)(find_col(a.pidx, rb, re, a.conn[(int64_t)j * a.E + e]) - rb);
}

// Thermal rows, one thread per row. Per incident element, in element order, the row of
// K_e of the row's node l: K_e(l, j) = sum_q g_l(q).G_q g_j(q) (element.rs:23-61). The
// accumulation goes to shared memory and costs no search: 8.2 ms -> 0.92 ms at 64^3
// (60.9 M entries) against a thread per row that searched every entry's column and
// updated it in global memory, and the 1.26 GB of element matrices (2.5 ms) give way to
// 0.30 GB of geometry (0.17 ms). Bound by the L1 pipe: 192 bytes of geometry per
// incidence and the conflicts of the accumulation.
// SMEM = false (rows of more than 256 entries, a block beyond shared memory, REPEATS)
// searches and adds in global memory.
template <bool SMEM, bool REPEATS>
__global__ void __launch_bounds__(kRowsT) k_thermal_rows(RowArgs a) {
    extern __shared__ double acc[];
    __shared__ double tab[120];
    const int64_t i0 = blockIdx.x * (int64_t)kRowsT, i1 = min(a.N, i0 + kRowsT);
    const int64_t base = a.pptr[i0], total = a.pptr[i1] - base;
    if (total <= a.lo || total > a.hi) return;
    double* out = SMEM ? acc : a.data + base;
    fill_gradients(tab);
    for (int64_t t = threadIdx.x; t < total; t += kRowsT) out[t] = 0.0;
    __syncthreads();
    const int64_t i = i0 + threadIdx.x;
    if (i < i1) {
        const int64_t rb = a.pptr[i], re = a.pptr[i + 1];
        double* row = out + (rb - base);
        const int32_t p1 = a.ptr[i + 1];
        int32_t p = a.ptr[i], el_next = 0;
        uint32_t w_next[3] = {0u, 0u, 0u};
        auto fetch = [&](int32_t at) {
            el_next = a.inc[at];
            if (SMEM)
#pragma unroll
                for (int k = 0; k < 3; ++k) w_next[k] = a.pos[3 * (int64_t)at + k];
        };
        if (p < p1) fetch(p);
        for (; p < p1; ++p) {
            const int32_t el = el_next;
            const int64_t e = el / 10;
            const int l = el - (int)e * 10;
            const uint32_t w[3] = {w_next[0], w_next[1], w_next[2]};
            if (p + 1 < p1) fetch(p + 1);
            double G[kMetricT];
#pragma unroll
            for (int k = 0; k < kMetricT; k += 4) load4(a.metric + kMetricT * e + k, G[k], G[k + 1], G[k + 2], G[k + 3]);
            double y[10];
#pragma unroll
            for (int j = 0; j < 10; ++j) y[j] = 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double* g = G + 6 * q;
                const double x0 = tab[(3 * q) * 10 + l], x1 = tab[(3 * q + 1) * 10 + l], x2 = tab[(3 * q + 2) * 10 + l];
                double f[4];  // flux in the barycentric directions
                f[1] = g[0] * x0 + g[1] * x1 + g[2] * x2;
                f[2] = g[1] * x0 + g[3] * x1 + g[4] * x2;
                f[3] = g[2] * x0 + g[4] * x1 + g[5] * x2;
                f[0] = -(f[1] + f[2] + f[3]);
#pragma unroll
                for (int m = 0; m < 4; ++m) y[m] += (m == q ? 4.0 * kQa - 1.0 : 4.0 * kQb - 1.0) * f[m];
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    const int m = edge_v(k, 0), n = edge_v(k, 1);
                    y[4 + k] += 4.0 * (n == q ? kQa : kQb) * f[m] + 4.0 * (m == q ? kQa : kQb) * f[n];
                }
            }
            int at[10];
#pragma unroll
            for (int j = 0; j < 10; ++j) at[j] = row_place<SMEM>(a, w, j, e, rb, re);
            add_columns<REPEATS>(row, at, y);
        }
    }
    if (SMEM) {
        __syncthreads();
        for (int64_t t = threadIdx.x; t < total; t += kRowsT) a.data[base + t] = acc[t];
    }
}

// Elastic rows, thread 3 n + c for row c of the block's n-th node: K^{ij}_{cb} = sum_q
// w |det J| (lam g_ic g_jb + mu (g_ib g_jc + delta_cb g_i.g_j)) of the incident elements,
// in element order (mechanics/element.rs:33-65). The three threads of a node read the
// same geometry. Writes the column indices too. 1.40 -> 0.26 ms at 24x24x12 against element
// matrices, a searching row kernel and an index kernel. A warp per node with a lane per (c, j)
// took 0.41 ms at 24x24x12: its sixteen indexed loads of gradients per element weigh more
// than the divergence it avoids.
template <bool SMEM, bool REPEATS>
__global__ void __launch_bounds__(3 * kRowsE) k_elastic_rows(RowArgs a) {
    extern __shared__ double acc[];
    __shared__ double tab[120];
    const int64_t i0 = blockIdx.x * (int64_t)kRowsE, i1 = min(a.N, i0 + kRowsE);
    const int64_t base = 9 * a.pptr[i0], total = 9 * a.pptr[i1] - base;
    if (total <= a.lo || total > a.hi) return;
    double* out = SMEM ? acc : a.data + base;
    fill_gradients(tab);
    for (int64_t t = threadIdx.x; t < total; t += 3 * kRowsE) out[t] = 0.0;
    __syncthreads();
    const int64_t i = i0 + threadIdx.x / 3;
    const int c = threadIdx.x % 3;
    if (i < i1) {
        const int64_t rb = a.pptr[i], re = a.pptr[i + 1];
        double* row = out + (9 * rb + c * 3 * (re - rb) - base);
        const int32_t p1 = a.ptr[i + 1];
        int32_t p = a.ptr[i], el_next = 0;
        uint32_t w_next[3] = {0u, 0u, 0u};
        auto fetch = [&](int32_t at) {
            el_next = a.inc[at];
            if (SMEM)
#pragma unroll
                for (int k = 0; k < 3; ++k) w_next[k] = a.pos[3 * (int64_t)at + k];
        };
        if (p < p1) fetch(p);
        for (; p < p1; ++p) {
            const int32_t el = el_next;
            const int64_t e = el / 10;
            const int l = el - (int)e * 10;
            const uint32_t w[3] = {w_next[0], w_next[1], w_next[2]};
            if (p + 1 < p1) fetch(p + 1);
            double K[10][3];
#pragma unroll
            for (int j = 0; j < 10; ++j) K[j][0] = K[j][1] = K[j][2] = 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double2* g2 = reinterpret_cast<const double2*>(a.metric + kMetricE * e + 10 * q);
                double Ji[10];
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    const double2 t = g2[k];
                    Ji[2 * k] = t.x;
                    Ji[2 * k + 1] = t.y;
                }
                const double x0 = tab[(3 * q) * 10 + l], x1 = tab[(3 * q + 1) * 10 + l], x2 = tab[(3 * q + 2) * 10 + l];
                double gi[3];
#pragma unroll
                for (int b = 0; b < 3; ++b) gi[b] = Ji[9] * (Ji[b] * x0 + Ji[3 + b] * x1 + Ji[6 + b] * x2);
                const double lg = a.lam * (c == 0 ? gi[0] : (c == 1 ? gi[1] : gi[2]));
                const double m0 = a.mu * gi[0], m1 = a.mu * gi[1], m2 = a.mu * gi[2];
                // For the gradient h of a barycentric coordinate the block row is lg h +
                // mu (h_c g_i + (g_i.h) e_c), linear in h: formed for the four coordinates,
                // then combined into the shape functions'.
                double B[4][3];
#pragma unroll
                for (int m = 1; m < 4; ++m) {
                    const double* h = Ji + 3 * (m - 1);
                    const double hc = c == 0 ? h[0] : (c == 1 ? h[1] : h[2]);
                    const double dd = m0 * h[0] + m1 * h[1] + m2 * h[2];
                    B[m][0] = lg * h[0] + m0 * hc + (c == 0 ? dd : 0.0);
                    B[m][1] = lg * h[1] + m1 * hc + (c == 1 ? dd : 0.0);
                    B[m][2] = lg * h[2] + m2 * hc + (c == 2 ? dd : 0.0);
                }
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    B[0][b] = -(B[1][b] + B[2][b] + B[3][b]);
#pragma unroll
                    for (int m = 0; m < 4; ++m) K[m][b] += (m == q ? 4.0 * kQa - 1.0 : 4.0 * kQb - 1.0) * B[m][b];
#pragma unroll
                    for (int k = 0; k < 6; ++k) {
                        const int m = edge_v(k, 0), n = edge_v(k, 1);
                        K[4 + k][b] += 4.0 * (n == q ? kQa : kQb) * B[m][b] + 4.0 * (m == q ? kQa : kQb) * B[n][b];
                    }
                }
            }
            int at[10];
#pragma unroll
            for (int j = 0; j < 10; ++j) at[j] = 3 * row_place<SMEM>(a, w, j, e, rb, re);
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                double y[10];
#pragma unroll
                for (int j = 0; j < 10; ++j) y[j] = K[j][b];
                add_columns<REPEATS>(row + b, at, y);
            }
        }
    }
    if (SMEM) {
        __syncthreads();
        for (int64_t t = threadIdx.x; t < total; t += 3 * kRowsE) a.data[base + t] = acc[t];
    }
    // column indices: the node row's pattern expanded by 3x3 blocks, a warp per node
    for (int64_t n = i0 + threadIdx.x / 32; n < i1; n += 3 * kRowsE / 32) {
        const int64_t rb = a.pptr[n];
        const int L3 = (int)(3 * (a.pptr[n + 1] - rb));
        for (int t = threadIdx.x & 31; t < L3; t += 32) {
            const int32_t col = 3 * a.pidx[rb + t / 3] + t % 3;
#pragma unroll
            for (int r = 0; r < 3; ++r) a.indices[9 * rb + r * (int64_t)L3 + t] = col;
        }
    }
}

__global__ void k_elastic_indptr(const int64_t* __restrict__ pptr, int64_t N, int64_t* __restrict__ indptr) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t > 3 * N) return;
    const int64_t i = t / 3;
    indptr[t] = i == N ? 9 * pptr[N] : 9 * pptr[i] + (t % 3) * 3 * (pptr[i + 1] - pptr[i]);
}

// Launches a value kernel over all blocks of ROWS rows: a first launch takes the blocks of
// few entries with little shared memory each, so that more of them are resident (the
// vertices' rows of a Tet10 mesh are three times as long as the midpoints', in blocks of
// their own), a second one the others. The line lies at 28 entries per row, the mean of a
// Tet10 mesh, between the two kinds of block: one launch, 20, 28, 40, 60 entries take 1.01,
// 1.03, 0.92, 0.98, 1.01 ms (thermal 64^3) and 0.37, 0.39, 0.26, 0.30, 0.42 ms (elastic
// 24x24x12). Blocks beyond shared memory, and meshes without
// the pattern's places, go through the global form, meshes with repeated nodes through their
// own global form (a branch in the shared-memory form took it from 0.92 to 1.00 ms at 64^3).
template <int ROWS, class K>
void launch_rows(geo_ctx* ctx, const geo_mesh* m, int per_entry, int64_t block_max, K smem_form, K global_form,
                 K repeats_form, const double* metric, int32_t* indices, double* data, double lam, double mu) {
    cudaStream_t s = ctx->stream;
    const int64_t kMost = 200 * 1024 / 8;
    const int threads = per_entry == 1 ? ROWS : 3 * ROWS;
    const unsigned g = blocks(m->n_nodes, ROWS);
    RowArgs a{m->conn.p, m->inc_ptr.p, m->inc.p, m->pat_ptr.p, m->pat_idx.p, m->pat_pos.p, metric,
              m->n_nodes, m->n_elem, indices, data, lam, mu, 0, 0};
    int64_t done = -1;  // blocks of at most this many entries are launched
    if (m->pat_pos.p) {
        GEO_CUDA(cudaFuncSetAttribute(smem_form, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kMost * 8)));
        const int64_t small = (int64_t)ROWS * 28 * per_entry, top = std::min(block_max, kMost);
        for (int64_t cap : {std::min(small, top), top}) {
            if (cap <= done) continue;
            a.lo = done;
            a.hi = cap;
            smem_form<<<g, threads, (size_t)cap * 8, s>>>(a);
            check_launch(ctx, "row values");
            done = cap;
        }
    }
    if (done < block_max) {
        a.lo = done;
        a.hi = INT64_MAX;
        (m->pat_repeats ? repeats_form : global_form)<<<g, threads, 0, s>>>(a);
        check_launch(ctx, "row values (global)");
    }
}

// f_{dpn*i + a} = sum over incidences (element order) of fe[e][dpn*l + a]
__global__ void k_gather_load(const int32_t* __restrict__ ptr, const int32_t* __restrict__ inc,
                              const double* __restrict__ fe, int64_t N, int dpn, double* __restrict__ f) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= dpn * N) return;
    const int64_t i = t / dpn;
    const int a = (int)(t % dpn);
    double s = 0.0;
    for (int32_t p = ptr[i]; p < ptr[i + 1]; ++p) {
        const int32_t el = inc[p];
        s = __dadd_rn(s, fe[(int64_t)(el / 10) * (10 * dpn) + dpn * (el % 10) + a]);
    }
    f[t] = s;
}

// ---------------------------------------------------------------- Dirichlet
__global__ void k_max_abs_diag(const int64_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                               const double* __restrict__ data, int64_t n, unsigned long long* out) {
    double m = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = find_col(indices, indptr[i], indptr[i + 1], (int32_t)i);
        if (p < indptr[i + 1] && indices[p] == i) m = fmax(m, fabs(data[p]));
    }
    // non-negative doubles order like their bit patterns
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

__global__ void k_dirichlet_rhs(const int64_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                                const double* __restrict__ data, const uint8_t* __restrict__ mask,
                                const double* __restrict__ g, const double* __restrict__ f, double cd, int64_t n,
                                double* __restrict__ fbc, int64_t* __restrict__ rowcnt) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (mask[i]) {
        fbc[i] = __dmul_rn(g[i], cd);
        rowcnt[i] = 1;
        return;
    }
    double s = f[i];
    int64_t c = 0;
    for (int64_t p = indptr[i]; p < indptr[i + 1]; ++p) {
        const int32_t j = indices[p];
        if (mask[j]) s = __dsub_rn(s, __dmul_rn(data[p], g[j]));
        else ++c;
    }
    fbc[i] = s;
    rowcnt[i] = c;
}

// A row to kDirLanes lanes: its entries are read together, and the kept ones written
// together (1.59 -> 0.42 ms at 64^3 against a thread per row; for the right-hand side and
// the counts above, which write nothing per entry, a thread per row is the faster form:
// 0.12 against 0.33 ms).
constexpr int kDirLanes = 16;

__global__ void __launch_bounds__(256) k_dirichlet_fill(const int64_t* __restrict__ indptr,
                                                        const int32_t* __restrict__ indices,
                                                        const double* __restrict__ data,
                                                        const uint8_t* __restrict__ mask, double cd, int64_t n,
                                                        const int64_t* __restrict__ optr, int32_t* __restrict__ oidx,
                                                        double* __restrict__ odata) {
    const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kDirLanes;
    const int sub = threadIdx.x % kDirLanes;
    if (i >= n) return;  // uniform within the group
    int64_t o = optr[i];
    if (mask[i]) {
        if (sub == 0) {
            oidx[o] = (int32_t)i;
            odata[o] = cd;
        }
        return;
    }
    const int64_t b = indptr[i], e = indptr[i + 1];
    const int shift = threadIdx.x & 31 & ~(kDirLanes - 1);
    const unsigned group = ((1u << kDirLanes) - 1u) << shift;
    for (int64_t p0 = b; p0 < e; p0 += kDirLanes) {
        const int64_t p = p0 + sub;
        const int32_t j = p < e ? indices[p] : -1;
        const double v = p < e ? data[p] : 0.0;
        const bool keep = j >= 0 && !mask[j];
        const unsigned k = (__ballot_sync(group, keep) & group) >> shift;
        if (keep) {
            const int64_t at = o + __popc(k & ((1u << sub) - 1u));
            oidx[at] = j;
            odata[at] = v;
        }
        o += __popc(k);
    }
}

__global__ void k_set_last(int64_t* ptr, int64_t n, const int64_t* cnt) {
    if (threadIdx.x == 0 && blockIdx.x == 0) ptr[n] = ptr[n - 1] + cnt[n - 1];
}

// ---------------------------------------------------------------- SpMV
template <int VEC>
__global__ void k_spmv(const int64_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                       const double* __restrict__ data, const double* __restrict__ x, int64_t n,
                       double* __restrict__ y) {
    const int64_t gt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t row = gt / VEC;
    const int sub = (int)(gt % VEC);
    if (row >= n) return;
    double s = 0.0;
    for (int64_t p = indptr[row] + sub; p < indptr[row + 1]; p += VEC) s += data[p] * x[indices[p]];
#pragma unroll
    for (int o = VEC / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, VEC);
    if (sub == 0) y[row] = s;
}

}  // namespace

// ---------------------------------------------------------------- shared builders
void ensure_inverse_map(geo_mesh* m) {
    if (m->inc.p) return;
    geo_ctx* ctx = m->ctx;
    cudaStream_t s = ctx->stream;
    const int64_t N = m->n_nodes, E = m->n_elem;
    DevBuf<int32_t> cnt(N + 1), cursor(N);
    GEO_CUDA(cudaMemsetAsync(cnt.p, 0, (N + 1) * sizeof(int32_t), s));
    GEO_CUDA(cudaMemsetAsync(cursor.p, 0, N * sizeof(int32_t), s));
    k_inc_count<<<blocks(E * 10, 256), 256, 0, s>>>(m->conn.p, E, cnt.p);
    check_launch(ctx, "k_inc_count");
    m->inc_ptr.alloc(N + 1);
    exclusive_scan(cnt.p, m->inc_ptr.p, N + 1, s);
    m->inc.alloc(E * 10);
    k_inc_fill<<<blocks(E * 10, 256), 256, 0, s>>>(m->conn.p, E, m->inc_ptr.p, cursor.p, m->inc.p);
    check_launch(ctx, "k_inc_fill");
    k_inc_sort<<<blocks(N, 128), 128, 0, s>>>(m->inc_ptr.p, m->inc.p, N);
    check_launch(ctx, "k_inc_sort");
    sync(ctx, "inverse map");
}

void ensure_pattern(geo_mesh* m) {
    if (m->pat_nnz >= 0) return;
    ensure_inverse_map(m);
    geo_ctx* ctx = m->ctx;
    cudaStream_t s = ctx->stream;
    const int64_t N = m->n_nodes, E = m->n_elem;
    DevBuf<int64_t> cnt(N + 1);
    GEO_CUDA(cudaMemsetAsync(cnt.p, 0, (N + 1) * sizeof(int64_t), s));
    GEO_CUDA(cudaMemsetAsync(ctx->dev_err.p, 0, 3 * sizeof(int), s));
    const unsigned g = (unsigned)std::min<int64_t>(cdiv(N, kPatWarps), 1 << 20);
    k_pattern<<<g, 32 * kPatWarps, 0, s>>>(m->conn.p, E, m->inc_ptr.p, m->inc.p, N, cnt.p, nullptr, nullptr, nullptr,
                                           ctx->dev_err.p);
    check_launch(ctx, "k_pattern(count)");
    int h[3] = {0, 0, 0};  // error bits, largest row, repeated nodes
    GEO_CUDA(cudaMemcpyAsync(h, ctx->dev_err.p, sizeof h, cudaMemcpyDeviceToHost, s));
    sync(ctx, "pattern counts");
    if (h[0] & DEV_ERR_BOUNDS)
        fail(GEO_ERR_UNSUPPORTED, "a node is shared by more than 102 elements (row pattern buffer)");
    m->pat_ptr.alloc(N + 1);
    exclusive_scan(cnt.p, m->pat_ptr.p, N + 1, s);
    DevBuf<unsigned long long> bm(2);
    GEO_CUDA(cudaMemsetAsync(bm.p, 0, bm.bytes(), s));
    k_block_max<<<blocks(cdiv(N, kRowsE), 256), 256, 0, s>>>(m->pat_ptr.p, N, bm.p);
    check_launch(ctx, "k_block_max");
    unsigned long long hb[2];
    int64_t nnz = 0;
    GEO_CUDA(cudaMemcpyAsync(&nnz, m->pat_ptr.p + N, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    GEO_CUDA(cudaMemcpyAsync(hb, bm.p, sizeof hb, cudaMemcpyDeviceToHost, s));
    sync(ctx, "pattern size");
    m->pat_block_t = (int64_t)hb[0];
    m->pat_block_e = (int64_t)hb[1];
    m->pat_repeats = h[2] != 0;
    m->pat_idx.alloc(nnz);
    if (h[1] <= 256 && !m->pat_repeats) m->pat_pos.alloc(30 * (size_t)E);
    k_pattern<<<g, 32 * kPatWarps, 0, s>>>(m->conn.p, E, m->inc_ptr.p, m->inc.p, N, nullptr, m->pat_ptr.p,
                                           m->pat_idx.p, m->pat_pos.p, ctx->dev_err.p);
    check_launch(ctx, "k_pattern(fill)");
    sync(ctx, "pattern");
    m->pat_nnz = nnz;
}

void csr_spmv(geo_ctx* ctx, const geo_csr* A, const double* x, double* y) {
    const int64_t n = A->n_rows;
    k_spmv<8><<<blocks(n * 8, 256), 256, 0, ctx->stream>>>(A->indptr.p, A->indices.p, A->data.p, x, n, y);
    check_launch(ctx, "k_spmv");
}

}  // namespace geo

using namespace geo;

namespace {

std::unique_ptr<geo_csr> new_csr(geo_ctx* ctx, int64_t rows, int64_t cols, int64_t nnz) {
    auto A = std::make_unique<geo_csr>();
    A->ctx = ctx;
    A->ref.set(ctx);
    A->n_rows = rows;
    A->n_cols = cols;
    A->nnz = nnz;
    A->indptr.alloc(rows + 1);
    A->indices.alloc(std::max<int64_t>(nnz, 1));
    A->data.alloc(std::max<int64_t>(nnz, 1));
    return A;
}

void deliver(geo_ctx* ctx, double* out, const double* dev, size_t n) {
    copy_out(out, dev, n, ctx->stream);
    sync(ctx, "deliver");
}

}  // namespace

extern "C" {

int geo_assemble_thermal_stiffness(geo_ctx* ctx, const geo_mesh* mesh, const geo_dofs* dofs, const double* k_e,
                                   double k, geo_csr** K) {
    GEO_API_BEGIN(ctx)
    GEO_CHECK_ARG(ctx && mesh && K, "NULL argument");
    GEO_CHECK_ARG(!dofs || (dofs->dpn == 1 && dofs->n_nodes == mesh->n_nodes),
                  "thermal assembly needs 1 DOF per node on the same node set");
    geo_mesh* m = const_cast<geo_mesh*>(mesh);
    ensure_pattern(m);
    cudaStream_t s = ctx->stream;
    const int64_t N = m->n_nodes, E = m->n_elem;
    DevBuf<double> tk, G(E * kMetricT);
    const double* dk = k_e ? stage_in(k_e, E, tk, s) : nullptr;
    reset_dev_err(ctx);
    k_thermal_metric<<<blocks(E * 4, 128), 128, 0, s>>>(m->xyz.p, m->conn.p, N, E, dk, k, G.p, ctx->dev_err.p);
    check_launch(ctx, "k_thermal_metric");
    auto A = new_csr(ctx, N, N, m->pat_nnz);
    GEO_CUDA(cudaMemcpyAsync(A->indptr.p, m->pat_ptr.p, (N + 1) * sizeof(int64_t), cudaMemcpyDeviceToDevice, s));
    GEO_CUDA(cudaMemcpyAsync(A->indices.p, m->pat_idx.p, m->pat_nnz * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
    launch_rows<kRowsT>(ctx, m, 1, m->pat_block_t, k_thermal_rows<true, false>, k_thermal_rows<false, false>,
                        k_thermal_rows<false, true>, G.p, A->indices.p, A->data.p, 0.0, 0.0);
    raise_dev_err(ctx, read_dev_err(ctx), "thermal stiffness");
    *K = A.release();
    GEO_API_END
}

int geo_assemble_thermal_load(geo_ctx* ctx, const geo_mesh* mesh, const geo_dofs* dofs, double source,
                              double* f) {
    GEO_API_BEGIN(ctx)
    GEO_CHECK_ARG(ctx && mesh && f, "NULL argument");
    GEO_CHECK_ARG(!dofs || (dofs->dpn == 1 && dofs->n_nodes == mesh->n_nodes),
                  "thermal load needs 1 DOF per node on the same node set");
    geo_mesh* m = const_cast<geo_mesh*>(mesh);
    ensure_inverse_map(m);
    cudaStream_t s = ctx->stream;
    DevBuf<double> fe(m->n_elem * 10), out(m->n_nodes);
    reset_dev_err(ctx);
    element_thermal_load(ctx, m, source, fe.p);
    k_gather_load<<<blocks(m->n_nodes, 256), 256, 0, s>>>(m->inc_ptr.p, m->inc.p, fe.p, m->n_nodes, 1, out.p);
    check_launch(ctx, "k_gather_load");
    deliver(ctx, f, out.p, m->n_nodes);
    GEO_API_END
}

int geo_assemble_elasticity_stiffness(geo_ctx* ctx, const geo_mesh* mesh, const geo_dofs* dofs, const double* E_e,
                                      double E, double nu, geo_csr** K) {
    GEO_API_BEGIN(ctx)
    GEO_CHECK_ARG(ctx && mesh && K, "NULL argument");
    GEO_CHECK_ARG(!dofs || dofs->dpn == 3, "Elasticity requires 3 DOF per node");
    GEO_CHECK_ARG(!dofs || dofs->n_nodes == mesh->n_nodes, "DOF manager and mesh disagree on the node count");
    GEO_CHECK_ARG(nu > -1.0 && nu < 0.5, "Poisson's ratio must be in (-1, 0.5)");
    geo_mesh* m = const_cast<geo_mesh*>(mesh);
    ensure_pattern(m);
    cudaStream_t s = ctx->stream;
    const int64_t N = m->n_nodes, Ne = m->n_elem;
    DevBuf<double> tE, geom(Ne * kMetricE);
    const double* dE = E_e ? stage_in(E_e, Ne, tE, s) : nullptr;
    reset_dev_err(ctx);
    k_elastic_metric<<<blocks(Ne * 4, 128), 128, 0, s>>>(m->xyz.p, m->conn.p, N, Ne, dE, E, geom.p, ctx->dev_err.p);
    check_launch(ctx, "k_elastic_metric");
    auto A = new_csr(ctx, 3 * N, 3 * N, 9 * m->pat_nnz);
    k_elastic_indptr<<<blocks(3 * N + 1, 256), 256, 0, s>>>(m->pat_ptr.p, N, A->indptr.p);
    check_launch(ctx, "k_elastic_indptr");
    // constitutive.rs:63-102 with the modulus in the metric
    const double lam = nu / ((1.0 + nu) * (1.0 - 2.0 * nu)), mu = 1.0 / (2.0 * (1.0 + nu));
    launch_rows<kRowsE>(ctx, m, 9, 9 * m->pat_block_e, k_elastic_rows<true, false>,
                        k_elastic_rows<false, false>, k_elastic_rows<false, true>, geom.p, A->indices.p, A->data.p, lam, mu);
    raise_dev_err(ctx, read_dev_err(ctx), "elasticity stiffness");
    *K = A.release();
    GEO_API_END
}

int geo_assemble_gravity_load(geo_ctx* ctx, const geo_mesh* mesh, const geo_dofs* dofs, double density,
                              const double gravity[3], double* f) {
    GEO_API_BEGIN(ctx)
    GEO_CHECK_ARG(ctx && mesh && f && gravity, "NULL argument");
    GEO_CHECK_ARG(!dofs || dofs->dpn == 3, "Gravity load requires 3 DOF per node");
    geo_mesh* m = const_cast<geo_mesh*>(mesh);
    ensure_inverse_map(m);
    cudaStream_t s = ctx->stream;
    DevBuf<double> fe(m->n_elem * 30), out(3 * m->n_nodes);
    element_gravity_load(ctx, m, density, gravity, fe.p);
    k_gather_load<<<blocks(3 * m->n_nodes, 256), 256, 0, s>>>(m->inc_ptr.p, m->inc.p, fe.p, m->n_nodes, 3, out.p);
    check_launch(ctx, "k_gather_load");
    deliver(ctx, f, out.p, 3 * m->n_nodes);
    GEO_API_END
}

int geo_apply_dirichlet_bcs(geo_ctx* ctx, const geo_csr* K, const double* f, const geo_dofs* dofs,
                            geo_csr** K_bc, double* f_bc) {
    GEO_API_BEGIN(ctx)
    GEO_CHECK_ARG(ctx && K && f && dofs && K_bc && f_bc, "NULL argument");
    GEO_CHECK_ARG(K->n_rows == dofs->n_dofs && K->n_cols == dofs->n_dofs, "matrix and DOF manager disagree");
    cudaStream_t s = ctx->stream;
    const int64_t n = K->n_rows;
    DevBuf<double> tf, fbc(n);
    const double* df = stage_in(f, n, tf, s);
    DevBuf<unsigned long long> mx(1);
    GEO_CUDA(cudaMemsetAsync(mx.p, 0, sizeof(unsigned long long), s));
    k_max_abs_diag<<<blocks(std::min<int64_t>(n, 148 * 2048), 256), 256, 0, s>>>(K->indptr.p, K->indices.p,
                                                                                  K->data.p, n, mx.p);
    check_launch(ctx, "k_max_abs_diag");
    unsigned long long bits = 0;
    GEO_CUDA(cudaMemcpyAsync(&bits, mx.p, sizeof(bits), cudaMemcpyDeviceToHost, s));
    sync(ctx, "char_diag");
    double maxd;
    std::memcpy(&maxd, &bits, sizeof(double));
    const double cd = maxd > 1.0 ? maxd : 1.0;  // assembly.rs:184-193
    DevBuf<int64_t> cnt(n + 1);
    k_dirichlet_rhs<<<blocks(n, 256), 256, 0, s>>>(K->indptr.p, K->indices.p, K->data.p, dofs->mask.p,
                                                   dofs->vals.p, df, cd, n, fbc.p, cnt.p);
    check_launch(ctx, "k_dirichlet_rhs");
    DevBuf<int64_t> optr(n + 1);
    exclusive_scan(cnt.p, optr.p, n, s);
    k_set_last<<<1, 32, 0, s>>>(optr.p, n, cnt.p);
    int64_t nnz = 0;
    GEO_CUDA(cudaMemcpyAsync(&nnz, optr.p + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    sync(ctx, "dirichlet counts");
    auto B = new_csr(ctx, n, K->n_cols, nnz);
    GEO_CUDA(cudaMemcpyAsync(B->indptr.p, optr.p, (n + 1) * sizeof(int64_t), cudaMemcpyDeviceToDevice, s));
    k_dirichlet_fill<<<blocks(n * kDirLanes, 256), 256, 0, s>>>(K->indptr.p, K->indices.p, K->data.p, dofs->mask.p, cd, n,
                                                    optr.p, B->indices.p, B->data.p);
    check_launch(ctx, "k_dirichlet_fill");
    deliver(ctx, f_bc, fbc.p, n);
    *K_bc = B.release();
    GEO_API_END
}

int geo_csr_create(geo_ctx* ctx, int64_t n_rows, int64_t n_cols, int64_t nnz, const int64_t* indptr,
                   const int32_t* indices, const double* data, geo_csr** out) {
    GEO_API_BEGIN(ctx)
    GEO_CHECK_ARG(ctx && out && indptr && (nnz == 0 || (indices && data)), "NULL argument");
    GEO_CHECK_ARG(n_rows > 0 && n_cols > 0 && nnz >= 0, "bad dimensions");
    GEO_CHECK_ARG(n_rows < (int64_t(1) << 31) && n_cols < (int64_t(1) << 31), "dimensions exceed int32 indices");
    // validate structure on the host
    std::vector<int64_t> hp(n_rows + 1);
    std::vector<int32_t> hi(nnz);
    GEO_CUDA(cudaMemcpy(hp.data(), indptr, (n_rows + 1) * sizeof(int64_t), cudaMemcpyDefault));
    if (nnz) GEO_CUDA(cudaMemcpy(hi.data(), indices, nnz * sizeof(int32_t), cudaMemcpyDefault));
    GEO_CHECK_ARG(hp[0] == 0 && hp[n_rows] == nnz, "indptr must start at 0 and end at nnz");
    for (int64_t i = 0; i < n_rows; ++i) {
        GEO_CHECK_ARG(hp[i] <= hp[i + 1], "indptr must be non-decreasing");
        for (int64_t p = hp[i]; p < hp[i + 1]; ++p) {
            GEO_CHECK_ARG(hi[p] >= 0 && hi[p] < n_cols, "column index out of range");
            GEO_CHECK_ARG(p == hp[i] || hi[p - 1] < hi[p], "columns must be sorted and unique within a row");
        }
    }
    auto A = new_csr(ctx, n_rows, n_cols, nnz);
    GEO_CUDA(cudaMemcpyAsync(A->indptr.p, hp.data(), (n_rows + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, ctx->stream));
    if (nnz) {
        GEO_CUDA(cudaMemcpyAsync(A->indices.p, hi.data(), nnz * sizeof(int32_t), cudaMemcpyHostToDevice, ctx->stream));
        // behind the caller's work on the default stream, as the copies above that read it; the
        // context's stream does not wait for that one by itself
        GEO_CUDA(cudaMemcpyAsync(A->data.p, data, nnz * sizeof(double), cudaMemcpyDefault, cudaStreamLegacy));
        GEO_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
    }
    sync(ctx, "geo_csr_create");
    *out = A.release();
    GEO_API_END
}

int geo_csr_info(const geo_csr* A, int64_t* n_rows, int64_t* n_cols, int64_t* nnz) {
    if (!A) return GEO_ERR_INVALID_ARG;
    if (n_rows) *n_rows = A->n_rows;
    if (n_cols) *n_cols = A->n_cols;
    if (nnz) *nnz = A->nnz;
    return GEO_OK;
}

int geo_csr_copy(const geo_csr* A, int64_t* indptr, int32_t* indices, double* data) {
    GEO_API_BEGIN(A ? A->ctx : nullptr)
    GEO_CHECK_ARG(A, "NULL matrix");
    cudaStream_t s = A->ctx->stream;
    if (indptr) copy_out(indptr, A->indptr.p, A->n_rows + 1, s);
    if (indices) copy_out(indices, A->indices.p, A->nnz, s);
    if (data) copy_out(data, A->data.p, A->nnz, s);
    sync(A->ctx, "csr copy");
    GEO_API_END
}

int geo_csr_device_ptrs(const geo_csr* A, const int64_t** indptr, const int32_t** indices, const double** data) {
    if (!A) return GEO_ERR_INVALID_ARG;
    if (indptr) *indptr = A->indptr.p;
    if (indices) *indices = A->indices.p;
    if (data) *data = A->data.p;
    return GEO_OK;
}

int geo_csr_apply(geo_ctx* ctx, const geo_csr* A, const double* x, double* y) {
    GEO_API_BEGIN(ctx)
    GEO_CHECK_ARG(ctx && A && x && y, "NULL argument");
    cudaStream_t s = ctx->stream;
    DevBuf<double> tx, ty(A->n_rows);
    const double* dx = stage_in(x, A->n_cols, tx, s);
    csr_spmv(ctx, A, dx, ty.p);
    deliver(ctx, y, ty.p, A->n_rows);
    GEO_API_END
}

int geo_csr_destroy(geo_csr* A) {
    if (!A) return GEO_OK;
    cudaSetDevice(A->ctx->device);
    delete A;
    return GEO_OK;
}

}  // extern "C"
