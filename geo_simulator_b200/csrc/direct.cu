// Dense LU solve of a CSR system on the device: the drop-in for
// DirectSolver::solve (linalg/direct.rs:28-73), which copies the matrix into a
// dense nalgebra matrix, factors it with partial (row) pivoting and solves.
//
// The matrix and the right-hand side are scattered into a dense row-major n x (n + 1)
// buffer in HBM (n <= kMaxDenseN: 2 GiB), factored right-looking in panels of nb columns
// and solved by back substitution. Rows never move: every row keeps its place in memory
// and carries its position in the matrix with rows exchanged, so that the pivot rule
// (the first row of largest |a_ik|) sees the reference's order. Per panel:
//   P. k_lu_panel: one cluster of up to 8 blocks holds the panel in registers (a thread
//      has R rows of nb values, R nb = 32) and eliminates its columns. Every block sends
//      its best candidate with its whole panel row to all blocks of the cluster, so a
//      column costs one cluster barrier; all blocks then know pivot and pivot row.
//      Leaves the multipliers of the remaining rows, compacted, and the pivot rows.
//   U. k_lu_rows: the nb pivot rows right of the panel (and of b) by forward
//      substitution with the panel's unit triangle, a thread per column.
//   T. k_lu_trailing: A -= L U for the remaining rows, 64 x 64 tiles, each output
//      subtracting its nb products in column order, as the unblocked elimination does:
//      the blocked form changes no rounding. Tiles whose multipliers or pivot rows are
//      all zero (a banded matrix) are skipped.
// n = 3757 takes 11.8 ms (127 ms before, dense random matrices), n = 1000 2.6 ms (15.6): the
// unblocked form had two grid barriers and a pass over the trailing matrix per column.
// Bound by the panels' chain of columns, about 1.9 us each.
// Carrying b along leaves y = L^-1 P b in its column. Back substitution U x = y then
// runs over 32-row blocks from the bottom in one persistent cooperative kernel: every
// block solves the 32 x 32 diagonal triangle itself (one warp, identical in all blocks, so
// no barrier), and the grid subtracts its contribution from the rows above, one bounded
// grid barrier per row block.
// A zero pivot marks the matrix singular (the reference's solve then fails:
// "LU solve failed"); every block sees the same candidates and leaves together, and the
// kernels after it return at once.
// Infinities and NaN go the way of an elimination that leaves a row alone where its
// multiplier is zero: a NaN is never a pivot (a column with nothing else is singular), and a
// zero multiplier takes no part in a product with an infinity or a NaN. Each kernel does its
// plain work when what it multiplies by is finite, and looks at every multiplier when not.
// ||b - A x|| is formed on the CSR matrix afterwards (solver.rs:139-175).
#include <cooperative_groups.h>

#include "pcg_common.cuh"

namespace geo {
namespace {

namespace cg = cooperative_groups;

constexpr int kDBS = 256;
constexpr int64_t kMaxDenseN = 16384;
constexpr int kPanelBS = 512;   // threads of a panel block
constexpr int kPanelRegs = 32;  // panel values per thread: R rows x nb columns
constexpr int kMaxNb = 32;
constexpr int kMaxCluster = 8;
constexpr int kTile = 64;       // trailing tile, rows and columns

// M = [A | b], leading dimension ld
__global__ void k_densify(const int64_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                          const double* __restrict__ data, const double* __restrict__ b, int64_t n, int64_t ld,
                          double* __restrict__ M, int32_t* __restrict__ list, int32_t* __restrict__ pos) {
    const int lane = threadIdx.x & 31;
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 32; i < n;
         i += (int64_t)gridDim.x * blockDim.x / 32) {
        for (int64_t p = indptr[i] + lane; p < indptr[i + 1]; p += 32) M[i * ld + indices[p]] = data[p];
        if (lane == 0) {
            M[i * ld + n] = b[i];
            list[i] = pos[i] = (int32_t)i;
        }
    }
}

struct LuArgs {
    double* M;
    int64_t n, ld;
    int k0, nbw;           // first column and width of the panel
    int m;                 // rows not eliminated yet
    int tile0;             // first column tile of the trailing update
    const int32_t* list;   // those rows
    int32_t* list_out;     // the rows left after the panel
    int32_t* pos;          // per row: position with rows exchanged
    int32_t* piv;          // piv[k]: the row eliminated at column k
    double* lbuf;          // [m][nb] multipliers, in list_out's order
    double* l11;           // [kMaxNb][kMaxNb] the panel's unit lower triangle
    int* singular;         // 0, or 1 + the first column of the panel that met a zero pivot
    double* x;             // the solution
    GridSync* gs;
    unsigned long long timeout_ns;
};

// This panel, or one before it, met a zero pivot. The panel after it may find one while the
// rest of this one's trailing update runs beside it (see lu_panel), which must not stop some
// threads of a block and not others.
__device__ __forceinline__ bool panel_failed(const LuArgs& a) {
    const int at = cuda::atomic_ref<int, cuda::thread_scope_device>(*a.singular).load(cuda::memory_order_relaxed);
    return at != 0 && at <= a.k0 + 1;
}

// Bits of +infinity: |v| as an integer is above it for NaN, and at least it for both.
constexpr unsigned long long kInfBits = 0x7ff0000000000000ull;
__device__ __forceinline__ unsigned long long abs_bits(double v) {
    return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}

// A block's candidate for the pivot of one column: |value| as an integer key, the row's
// position, list index and place in M, and the row's panel values.
struct PanelSlot {
    double row[kMaxNb];
    unsigned long long key;
    int pos, at, mrow;  // mrow: the row in M
};

// Largest key of the warp, then the smallest position among its holders (the first
// maximum); every lane gets both. The upper halves alone mostly decide.
__device__ __forceinline__ void warp_best(unsigned long long& key, int& pos) {
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned holders = __ballot_sync(0xffffffffu, hi == mh);
    unsigned ml;
    if ((holders & (holders - 1u)) == 0u) {
        const int src = __ffs(holders) - 1;
        ml = __shfl_sync(0xffffffffu, lo, src);
        pos = __shfl_sync(0xffffffffu, pos, src);
    } else {
        ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
        pos = (int)__reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? (unsigned)pos : 0x7fffffffu);
    }
    key = (unsigned long long)mh << 32 | ml;
}

// One step of the panel is one pass of a rolled loop: the values are kept shifted, the
// current column in v[.][0], and the update writes v[j] from v[j + 1]. Unrolled over the
// columns (registers indexed by the column, half the FMAs) the kernel is 240 KB of
// instructions that each run once, and took 3.2 us per column, mostly waiting for them.
// The multipliers wait in shared memory for the end, when the remaining rows' places are
// known. Bound by latency: two block-wide reductions, a cluster barrier and a division per
// column, 1.9 us whatever the number of rows (2.45 with the results stored to global
// memory on the way, which every cluster barrier waits for; messages on mbarriers in place
// of the cluster barrier were no faster).
template <int NB>
__global__ void __launch_bounds__(kPanelBS) k_lu_panel(LuArgs a) {
    constexpr int R = kPanelRegs / NB;
    extern __shared__ double s_l[];  // [NB][R][blockDim.x] multipliers
    __shared__ PanelSlot s_slot[2][kMaxCluster];
    __shared__ unsigned long long s_key[kPanelBS / 32];
    __shared__ int s_pos[kPanelBS / 32];
    __shared__ double s_row[kMaxNb];
    __shared__ double s_up[NB][NB];  // block 0: the pivot rows from their column on
    __shared__ int s_piv[NB];
    if (panel_failed(a)) return;  // an earlier panel: the same for every block
    cg::cluster_group cluster = cg::this_cluster();
    const int ncta = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int bs = blockDim.x, nwarp = bs >> 5;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double v[R][NB];
    int row[R], pos[R], at[R], step[R], shift[R];
    auto load = [&]() {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            at[r] = (r * ncta + rank) * bs + (int)threadIdx.x;
            const bool in = at[r] < a.m;
            row[r] = in ? a.list[at[r]] : -1;
            pos[r] = in ? a.pos[row[r]] : 0x7fffffff;
            step[r] = in ? -1 : NB;  // column at which the row was the pivot; NB: no row; -2: see below
            shift[r] = 0;            // pivots at smaller list indices
#pragma unroll
            for (int j = 0; j < NB; ++j) v[r][j] = in && j < a.nbw ? a.M[row[r] * a.ld + a.k0 + j] : 0.0;
        }
    };
    bool singular = false;
    bool wild = false;     // last warp: a pivot row held an infinity or a NaN
    bool careful = false;  // second go at a panel that had one: looks at every multiplier
    // this warp's candidate in the current column
    auto candidate = [&]() {
        unsigned long long key = 0;
        int p = 0x7fffffff;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const unsigned long long kr = step[r] == -1 ? abs_bits(v[r][0]) : 0ull;
            const int pr = step[r] == -1 ? pos[r] : 0x7fffffff;
            if (kr > key || (kr == key && pr < p)) {
                key = kr;
                p = pr;
            }
        }
        warp_best(key, p);
        if (lane == 0) {
            s_key[warp] = key;
            s_pos[warp] = p;
        }
    };
    // One go at the panel, which stays as it was in memory until the end; a second, careful
    // one when a pivot row was not finite (looking in every column made all solves 2.5%
    // slower). Every block has seen the same pivot rows.
#pragma unroll 1
    for (;;) {
        load();
        candidate();
        cluster.sync();  // every block runs, and has read its slots, before they are written to
#pragma unroll 1
        for (int k = 0; k < a.nbw; ++k) {
            __syncthreads();
            unsigned long long key = lane < nwarp ? s_key[lane] : 0ull;
            int p = lane < nwarp ? s_pos[lane] : 0x7fffffff;
            warp_best(key, p);
            // the warp that holds the block's candidate sends it to every block
            bool mine = false;
            int my_at = 0, my_row = 0;
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (step[r] < 0 && pos[r] == p) {
                    mine = true;
                    my_at = at[r];
                    my_row = row[r];
#pragma unroll
                    for (int j = 0; j < NB; ++j) s_row[j] = v[r][j];
                }
            const unsigned who = __ballot_sync(0xffffffffu, mine);
            if (who || (p == 0x7fffffff && warp == 0)) {
                const int cat = __shfl_sync(0xffffffffu, my_at, who ? __ffs(who) - 1 : 0);
                const int crow = __shfl_sync(0xffffffffu, my_row, who ? __ffs(who) - 1 : 0);
                __syncwarp();
                const double mv = lane < NB ? s_row[lane] : 0.0;
                for (int c = 0; c < ncta; ++c) {
                    PanelSlot* dst = cluster.map_shared_rank(&s_slot[k & 1][rank], c);
                    if (lane < NB) dst->row[lane] = mv;
                    if (lane == 0) {
                        dst->key = key;
                        dst->pos = p;
                        dst->at = cat;
                        dst->mrow = crow;
                    }
                }
            }
            cluster.sync();
            const PanelSlot* slots = s_slot[k & 1];
            key = lane < ncta ? slots[lane].key : 0ull;
            p = lane < ncta ? slots[lane].pos : 0x7fffffff;
            const int lane_pos = p;
            warp_best(key, p);
            const int win = __ffs(__ballot_sync(0xffffffffu, lane < ncta && lane_pos == p)) - 1;
            if (key == 0ull) {  // no candidate, or a zero pivot: every block leaves the loop here
                singular = true;
                break;
            }
            if (careful && key > kInfBits) {
                // NaN: rows that have one in this column are no candidates from here on (their
                // multipliers and so all their values will be NaN), and the column is searched again
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (step[r] == -1 && abs_bits(v[r][0]) > kInfBits) step[r] = -2;
                cluster.sync();  // every block has read the slots
                candidate();
                --k;
                continue;
            }
            const PanelSlot& s = slots[win];
            const double d = s.row[0];
            const int pat = s.at;
            // kept for the end: a store to global memory here would be waited for at every
            // cluster barrier
            if (warp == nwarp - 1) {
                const double u = lane < NB ? s.row[lane] : 0.0;
                wild |= abs_bits(u) >= kInfBits;
                if (rank == 0) {
                    if (lane < NB) s_up[k][lane] = u;
                    if (lane == 0) s_piv[k] = s.mrow;
                }
            }
            double l[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                l[r] = 0.0;
                if (step[r] >= 0) continue;
                if (pos[r] == p) {
                    step[r] = k;
                    continue;
                }
                if (pos[r] == a.k0 + k) pos[r] = p;  // exchanged with the pivot row
                shift[r] += at[r] > pat;
                l[r] = v[r][0] / d;
                s_l[(k * R + r) * bs + threadIdx.x] = l[r];
            }
            if (careful) {
#pragma unroll
                for (int j = 0; j < NB; ++j)
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const double t = j + 1 < NB ? v[r][(j + 1) % NB] : 0.0;
                        v[r][j] = j + 1 < NB && l[r] != 0.0 ? t - l[r] * s.row[(j + 1) % NB] : t;
                    }
                candidate();
                continue;
            }
            // the next column first, so that its reduction overlaps the others' update
#pragma unroll
            for (int r = 0; r < R; ++r) v[r][0] = v[r][1] - l[r] * s.row[1];
            candidate();
#pragma unroll
            for (int j = 1; j + 1 < NB; ++j) {
                const double u = s.row[j + 1];
#pragma unroll
                for (int r = 0; r < R; ++r) v[r][j] = v[r][j + 1] - l[r] * u;
            }
#pragma unroll
            for (int r = 0; r < R; ++r) v[r][NB - 1] = 0.0;
        }
        if (careful || !__syncthreads_or(wild)) break;
        careful = true;
        singular = false;
    }
    if (singular && rank == 0 && threadIdx.x == 0)
        cuda::atomic_ref<int, cuda::thread_scope_device>(*a.singular).store(a.k0 + 1, cuda::memory_order_relaxed);
    __syncthreads();
    if (!singular) {
        if (rank == 0)
            for (int t = threadIdx.x; t < a.nbw * NB; t += bs) {
                const int k = t / NB, j = t % NB;
                if (j < a.nbw - k) a.M[s_piv[k] * a.ld + a.k0 + k + j] = s_up[k][j];
                if (j == 0) a.piv[a.k0 + k] = s_piv[k];
            }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (step[r] == NB) continue;
            const double* mine = s_l + r * bs + threadIdx.x;
            if (step[r] >= 0) {
                for (int j = 0; j < step[r]; ++j) a.l11[step[r] * kMaxNb + j] = mine[j * R * bs];
            } else {
                const int64_t to = at[r] - shift[r];
                a.list_out[to] = row[r];
                a.pos[row[r]] = pos[r];
                for (int j = 0; j < a.nbw; ++j) a.lbuf[to * NB + j] = mine[j * R * bs];
            }
        }
    }
    cluster.sync();  // no block leaves while another may still write to its shared memory
}

// Pivot rows right of the panel: u = L11^-1 a, column by column.
template <int NB>
__global__ void __launch_bounds__(64) k_lu_rows(LuArgs a) {
    __shared__ double l[NB][NB];
    const int lane = threadIdx.x & 31;
    const int mine = lane < a.nbw ? a.piv[a.k0 + lane] : 0;  // pivot row `lane`
    if (panel_failed(a)) return;
    const int64_t j = a.k0 + a.nbw + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    double u[NB];
#pragma unroll
    for (int r = 0; r < NB; ++r) {
        const int64_t row = __shfl_sync(0xffffffffu, mine, r);
        u[r] = r < a.nbw && j <= a.n ? a.M[row * a.ld + j] : 0.0;
    }
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
        const int r = t / NB, c = t % NB;
        l[r][c] = c < r && r < a.nbw ? a.l11[r * kMaxNb + c] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < NB; ++s)
#pragma unroll
        for (int r = s + 1; r < NB; ++r) u[r] -= l[r][s] * u[s];
    // an infinity or a NaN on the way is one in the end: that column again, row by row in
    // place, leaving out the zero multipliers
    bool wild = false;
#pragma unroll
    for (int r = 0; r < NB; ++r) wild |= abs_bits(u[r]) >= kInfBits;
    if (wild && j <= a.n) {
#pragma unroll 1
        for (int r = 1; r < a.nbw; ++r) {
            double* at = a.M + a.piv[a.k0 + r] * a.ld + j;
            double t = *at;
#pragma unroll 1
            for (int s = 0; s < r; ++s)
                if (l[r][s] != 0.0) t -= l[r][s] * a.M[a.piv[a.k0 + s] * a.ld + j];
            *at = t;
        }
    }
#pragma unroll
    for (int r = 1; r < NB; ++r) {
        const int64_t row = __shfl_sync(0xffffffffu, mine, r);
        if (!wild && r < a.nbw && j <= a.n) a.M[row * a.ld + j] = u[r];
    }
}

// Trailing tile: 128 threads, thread (tx, ty) holds rows 8 ty .. 8 ty + 7 and columns tx,
// tx + 16, tx + 32, tx + 48; per column of L it reads 12 values of shared memory for 32
// FMAs, so the FP64 pipe bounds it, or, below nb = 32, the pass over the trailing matrix.
template <int NB>
__global__ void __launch_bounds__(128) k_lu_trailing(LuArgs a) {
    __shared__ __align__(16) double L[NB][kTile + 2];
    __shared__ double U[NB][kTile];
    __shared__ int s_wild;  // the tile's multipliers or pivot rows hold an infinity or a NaN
    if (threadIdx.x == 0) s_wild = 0;
    if (panel_failed(a)) return;
    const int m = a.m - a.nbw;  // rows left
    const int r0 = blockIdx.y * kTile;
    const int64_t c0 = a.k0 + a.nbw + (a.tile0 + (int64_t)blockIdx.x) * kTile;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    bool any = false, wild = false;
    for (int t = threadIdx.x; t < kTile * NB; t += 128) {
        const int r = t / NB, k = t % NB;
        const double v = r0 + r < m && k < a.nbw ? a.lbuf[(int64_t)(r0 + r) * NB + k] : 0.0;
        L[k][r] = v;
        any |= v != 0.0;
        wild |= abs_bits(v) >= kInfBits;
    }
    if (!__syncthreads_or(any)) return;
    any = wild;  // times a zero of a pivot row it is not zero
    for (int t = threadIdx.x; t < kTile * NB; t += 128) {
        const int k = t / kTile, c = t % kTile;
        const double v = k < a.nbw && c0 + c <= a.n ? a.M[a.piv[a.k0 + k] * a.ld + c0 + c] : 0.0;
        U[k][c] = v;
        any |= v != 0.0;
        wild |= abs_bits(v) >= kInfBits;
    }
    if (wild) s_wild = 1;
    double* rows[8];
    double acc[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int i = r0 + 8 * ty + r;
        rows[r] = i < m ? a.M + a.list_out[i] * a.ld : nullptr;
#pragma unroll
        for (int c = 0; c < 4; ++c)
            acc[r][c] = rows[r] && c0 + tx + 16 * c <= a.n ? rows[r][c0 + tx + 16 * c] : 0.0;
    }
    if (!__syncthreads_or(any)) return;
    if (s_wild) {
#pragma unroll 1
        for (int k = 0; k < NB; ++k)
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const double l = L[k][8 * ty + r];
                if (l != 0.0)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[r][c] -= l * U[k][tx + 16 * c];
            }
    } else {
#pragma unroll 4
        for (int k = 0; k < NB; ++k) {
            double l[8], u[4];
#pragma unroll
            for (int r = 0; r < 8; r += 2) {
                const double2 t = *reinterpret_cast<const double2*>(&L[k][8 * ty + r]);
                l[r] = t.x;
                l[r + 1] = t.y;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) u[c] = U[k][tx + 16 * c];
#pragma unroll
            for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[r][c] -= l[r] * u[c];
        }
    }
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (rows[r] && c0 + tx + 16 * c <= a.n) rows[r][c0 + tx + 16 * c] = acc[r][c];
}

// Back substitution U x = y (y in column n) over 32-row blocks, bottom first. The
// diagonal block is brought to shared memory by the whole block and solved column by
// column by one warp; read from memory row by row it took 15 us per block.
__global__ void __launch_bounds__(kDBS) k_lu_back(LuArgs a) {
    __shared__ double s_u[32][33];
    __shared__ double s_x[32];
    if (*a.singular) return;
    const int64_t n = a.n;
    const int lane = threadIdx.x & 31;
    const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5, nw = (int64_t)gridDim.x * blockDim.x >> 5;
    for (int64_t r0 = (n - 1) / 32 * 32; r0 >= 0; r0 -= 32) {
        const int w = (int)std::min<int64_t>(n - r0, 32);
        for (int r = threadIdx.x >> 5; r < w; r += kDBS / 32) {
            const double* row = a.M + a.piv[r0 + r] * a.ld;
            if (lane < w) s_u[r][lane] = row[r0 + lane];
            if (lane == 0) s_u[r][32] = __ldcg(row + n);
        }
        __syncthreads();
        if (threadIdx.x < 32) {  // the same in every block
            double y = lane < w ? s_u[lane][32] : 0.0;
            const double diag = lane < w ? s_u[lane][lane] : 1.0;
            for (int r = w - 1; r >= 0; --r) {
                const double x = __shfl_sync(0xffffffffu, y / diag, r);
                if (lane < r) y -= s_u[lane][r] * x;
                if (lane == r) s_x[r] = x;
            }
            if (lane >= w) s_x[lane] = 0.0;
            __syncwarp();
            if (blockIdx.x == 0 && lane < w) a.x[r0 + lane] = s_x[lane];
        }
        __syncthreads();
        if (r0 == 0) break;
        for (int64_t i = gw; i < r0; i += nw) {  // rows above: y_i -= U[i, r0:r0+w] x
            double* row = a.M + a.piv[i] * a.ld;
            double t = lane < w ? row[r0 + lane] * s_x[lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
            if (lane == 0) __stcg(row + n, __ldcg(row + n) - t);
        }
        if (!grid_barrier(a.gs, gridDim.x, a.timeout_ns)) return;
    }
}

// Per-block partials of ||b - A x||^2 and ||b||^2 (CSR)
__global__ void __launch_bounds__(kDBS) k_residual(const int64_t* __restrict__ indptr,
                                                   const int32_t* __restrict__ indices,
                                                   const double* __restrict__ data, int64_t n,
                                                   const double* __restrict__ x, const double* __restrict__ b,
                                                   double* __restrict__ part) {
    double v[2] = {0.0, 0.0};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double ax = 0.0;
        for (int64_t p = indptr[i]; p < indptr[i + 1]; ++p) ax += data[p] * x[indices[p]];
        const double r = b[i] - ax;
        v[0] += r * r;
        v[1] += b[i] * b[i];
    }
    store_partial<2>(part, v);
}

// Stream of the panels and events of the look-ahead, for one solve. The stream has the
// highest priority: a panel's cluster needs 8 SMs at once, and would wait behind the
// thousands of blocks of the trailing update beside it.
struct LookAhead {
    cudaStream_t s = nullptr;
    cudaEvent_t rows = nullptr, rest = nullptr;  // pivot rows ready; rest of the trailing update done
    bool pending = false;                        // `rest` is recorded and not waited for
    void create() {
        int least = 0, greatest = 0;
        GEO_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
        GEO_CUDA(cudaStreamCreateWithPriority(&s, cudaStreamNonBlocking, greatest));
        GEO_CUDA(cudaEventCreateWithFlags(&rows, cudaEventDisableTiming));
        GEO_CUDA(cudaEventCreateWithFlags(&rest, cudaEventDisableTiming));
    }
    ~LookAhead() {
        if (s) cudaStreamSynchronize(s);
        if (rows) cudaEventDestroy(rows);
        if (rest) cudaEventDestroy(rest);
        if (s) cudaStreamDestroy(s);
    }
};

// Queues one panel of NB columns; returns the launches. With look-ahead the trailing
// update is split: the tile column that holds the next panel stays on the panels' stream,
// the others go to the context's stream and run beside the next panel's factorization,
// which leaves all but 8 SMs idle.
template <int NB>
int lu_panel(geo_ctx* ctx, LuArgs a, LookAhead* ahead) {
    cudaStream_t s = ahead ? ahead->s : ctx->stream;
    a.nbw = (int)std::min<int64_t>(NB, a.n - a.k0);
    // Blocks of at least two warps, spread over the cluster's SMs before they grow. A block
    // for every 32, 64, 128, 256, 512 rows: n = 500 takes 1.22, 1.21, 1.20, 1.24, 1.33 ms,
    // n = 2000 5.43, 5.41, 5.38, 5.44, 5.93: fewer, fuller blocks pay more for their own
    // reductions than they save at the cluster barrier.
    constexpr int R = kPanelRegs / NB;
    int ncta = 1;
    while (ncta < kMaxCluster && ncta * 64 * R < a.m) ncta *= 2;
    const int bs = (int)(cdiv(cdiv(a.m, ncta * R), 32) * 32);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ncta);
    cfg.blockDim = dim3(bs);
    cfg.dynamicSmemBytes = (size_t)kPanelRegs * bs * sizeof(double);
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = ncta;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    GEO_CUDA(cudaLaunchKernelEx(&cfg, k_lu_panel<NB>, a));
    const int64_t cols = a.n + 1 - (a.k0 + a.nbw);  // with the right-hand side
    if (ahead && ahead->pending) {
        GEO_CUDA(cudaStreamWaitEvent(s, ahead->rest, 0));
        ahead->pending = false;
    }
    k_lu_rows<NB><<<(unsigned)cdiv(cols, 64), 64, 0, s>>>(a);
    check_launch(ctx, "k_lu_rows");
    if (a.m == a.nbw) return 2;
    const unsigned ty = (unsigned)cdiv(a.m - a.nbw, kTile), tx = (unsigned)cdiv(cols, kTile);
    // 2, 8 or 16 tile columns: within 0.3% of each other at n = 700 to 5000
    const bool split = ahead && tx > 8;
    if (split) GEO_CUDA(cudaEventRecord(ahead->rows, s));
    k_lu_trailing<NB><<<dim3(split ? 1 : tx, ty), 128, 0, s>>>(a);
    check_launch(ctx, "k_lu_trailing");
    if (!split) return 3;
    GEO_CUDA(cudaStreamWaitEvent(ctx->stream, ahead->rows, 0));
    a.tile0 = 1;
    k_lu_trailing<NB><<<dim3(tx - 1, ty), 128, 0, ctx->stream>>>(a);
    check_launch(ctx, "k_lu_trailing");
    GEO_CUDA(cudaEventRecord(ahead->rest, ctx->stream));
    ahead->pending = true;
    return 4;
}

}  // namespace
}  // namespace geo

using namespace geo;

extern "C" {

int geo_direct_solve(geo_ctx* ctx, const geo_csr* A, const double* b, double* x, geo_solver_stats* stats) {
    GEO_API_BEGIN(ctx)
    GEO_CHECK_ARG(ctx && A && b && x, "NULL argument");
    GEO_CHECK_ARG(A->n_rows == A->n_cols, "matrix must be square");
    const int64_t n = A->n_rows;
    GEO_CHECK_ARG(n >= 1 && n <= kMaxDenseN, "dense LU: n must be in 1..16384 (n x n doubles on the device)");
    cudaStream_t s = ctx->stream;
    const int64_t ld = (n + 1 + 15) / 16 * 16;
    DevBuf<double> tb, M((size_t)n * ld), lbuf(2 * (size_t)n * kMaxNb), l11(kMaxNb * kMaxNb), xd(n);
    DevBuf<int32_t> idx(4 * (size_t)n);  // two row lists, positions, pivots
    DevBuf<int> sing(1);
    DevBuf<GridSync> gs(1);
    const double* db = stage_in(b, (size_t)n, tb, s);
    GEO_CUDA(cudaMemsetAsync(M.p, 0, M.bytes(), s));
    GEO_CUDA(cudaMemsetAsync(gs.p, 0, sizeof(GridSync), s));
    GEO_CUDA(cudaMemsetAsync(sing.p, 0, sizeof(int), s));
    GEO_CUDA(cudaEventRecord(ctx->ev0, s));
    LuArgs la{};
    la.M = M.p;
    la.n = n;
    la.ld = ld;
    la.pos = idx.p + 2 * n;
    la.piv = idx.p + 3 * n;
    la.l11 = l11.p;
    la.singular = sing.p;
    la.x = xd.p;
    la.gs = gs.p;
    la.timeout_ns = 10ull * 1000000000ull;
    k_densify<<<(unsigned)std::min<int64_t>(cdiv(n * 32, kDBS), 4096), kDBS, 0, s>>>(
        A->indptr.p, A->indices.p, A->data.p, db, n, ld, M.p, idx.p, la.pos);
    check_launch(ctx, "k_densify");
    const int panel_smem = kPanelRegs * kPanelBS * (int)sizeof(double);
    GEO_CUDA(cudaFuncSetAttribute(k_lu_panel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, panel_smem));
    GEO_CUDA(cudaFuncSetAttribute(k_lu_panel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, panel_smem));
    GEO_CUDA(cudaFuncSetAttribute(k_lu_panel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, panel_smem));
    // Panel width: the widest of which the rows left fit one cluster's registers (4096
    // rows at 32 columns, 8192 at 16, 16384 at 8).
    int64_t launches = 2;
    LookAhead ahead;
    // Look-ahead costs a stream, two events and a split launch per panel: with and without,
    // n = 300 0.77, 0.71 ms, 700 1.78, 1.72, 900 2.30, 2.25, 1200 3.08, 3.03, 1500 3.90, 3.90,
    // 2000 5.42, 5.56, 3757 11.8, 14.2. It is even at 1500; the line at 640 is early by 3%.
    LookAhead* pa = n > 10 * kTile ? &ahead : nullptr;
    if (pa) {
        ahead.create();
        GEO_CUDA(cudaEventRecord(ahead.rows, s));  // the matrix is in place
        GEO_CUDA(cudaStreamWaitEvent(ahead.s, ahead.rows, 0));
    }
    int flip = 0;
    for (int64_t k0 = 0; k0 < n; flip ^= 1) {
        la.k0 = (int)k0;
        la.m = (int)(n - k0);
        la.list = idx.p + flip * n;
        la.list_out = idx.p + (flip ^ 1) * n;
        la.lbuf = lbuf.p + (size_t)flip * n * kMaxNb;  // the panel before may still be in use
        const int64_t rows32 = (int64_t)kMaxCluster * kPanelBS;
        const int nb = la.m <= rows32 ? 32 : (la.m <= 2 * rows32 ? 16 : 8);
        launches += nb == 32 ? lu_panel<32>(ctx, la, pa) : (nb == 16 ? lu_panel<16>(ctx, la, pa) : lu_panel<8>(ctx, la, pa));
        k0 += std::min<int64_t>(nb, n - k0);
    }
    if (pa) {
        GEO_CUDA(cudaEventRecord(ahead.rows, ahead.s));
        GEO_CUDA(cudaStreamWaitEvent(s, ahead.rows, 0));
    }
    const int nback = (int)std::max<int64_t>(
        1, std::min<int64_t>(persistent_blocks(ctx, k_lu_back, kDBS, 0), cdiv(n, 4 * (kDBS / 32))));
    launch_persistent(ctx, k_lu_back, kDBS, 0, la, nback);
    GEO_CUDA(cudaEventRecord(ctx->ev1, s));
    int singular = 0;
    GridSync g{};
    GEO_CUDA(cudaMemcpyAsync(&singular, sing.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    GEO_CUDA(cudaMemcpyAsync(&g, gs.p, sizeof(g), cudaMemcpyDeviceToHost, s));
    sync(ctx, "dense LU");
    if (g.error & DEV_ERR_TIMEOUT) fail(GEO_ERR_TIMEOUT, "dense LU: grid barrier timed out");
    if (singular) fail(GEO_ERR_SINGULAR_MATRIX, "LU solve failed: the matrix is singular");
    const int rb = (int)std::min<int64_t>(cdiv(n, kDBS), 1024);
    DevBuf<double> part((size_t)rb * 2);
    k_residual<<<rb, kDBS, 0, s>>>(A->indptr.p, A->indices.p, A->data.p, n, xd.p, db, part.p);
    check_launch(ctx, "k_residual");
    std::vector<double> hp((size_t)rb * 2);
    GEO_CUDA(cudaMemcpyAsync(hp.data(), part.p, hp.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
    copy_out(x, xd.p, (size_t)n, s);
    sync(ctx, "geo_direct_solve");
    double rr = 0.0, bb = 0.0;
    for (int i = 0; i < rb; ++i) {
        rr += hp[2 * (size_t)i];
        bb += hp[2 * (size_t)i + 1];
    }
    float ms = 0.f;
    GEO_CUDA(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
    const double res = std::sqrt(rr), bn = std::sqrt(bb);
    const double rel = bn < 1e-14 ? res : res / bn;  // solver.rs:165-175
    if (stats) {
        *stats = geo_solver_stats{};
        stats->iterations = 0;  // direct.rs:62
        stats->residual_norm = res;
        stats->relative_residual = rel;
        stats->converged = rel < 1e-8;  // direct.rs:65
        stats->solve_time = ms * 1e-3;
        stats->kernel_time = ms * 1e-3;
        stats->status = GEO_OK;
        stats->b_norm = bn;
        stats->kernel_launches = launches + 1;
    }
    GEO_API_END
}

}  // extern "C"
