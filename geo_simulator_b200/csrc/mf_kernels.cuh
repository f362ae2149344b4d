// Kernels of the matrix-free operator and its PCG (see matfree.cu).
//
// Patch apply (k_patch): a CTA works through whole patches (patch = blockIdx.x,
// += gridDim.x). The patch's element data (16-bit local connectivity and the
// per-element qdata, contiguous per patch), its foreign node ids and flags
// (aligned per-patch segments) and its sizes are brought into shared memory with
// cp.async.bulk (bulk copy engine, mbarrier completion), double-buffered so the
// next patch's copy is in flight while the current one is processed; the gather
// then needs a single round trip to global memory. Per patch:
//   1. gather: every patch-local node's input value is read once from global
//      memory into a shared table (own nodes form one contiguous range, worked on in
//      aligned groups with 16-byte accesses);
//   2. element pass: each thread applies K_e to its elements from the shared
//      table and accumulates into a shared output table with shared atomics
//      (exact INT32 fixed point for FP32, see Scatter). Elements are ordered so
//      a warp's 32 elements share no node, so these atomics do not collide;
//   3. flush: a plain store for nodes no other patch touches, red.global.add
//      for the shared ones. In "halo" mode (every mode, when the operator has
//      halo slots) every own node is a plain store and every foreign node a
//      plain store to its own slot of a halo array; the slots are numbered by
//      owner node, so the node update (PCG) or k_halo_finish (operator apply,
//      lift) adds a node's foreign contributions from consecutive slots in a
//      fixed order. No global atomics are issued and results are bit-identical
//      from run to run.
// In PCG mode step 1 also forms the new search direction p = z + beta p_old
// (z = D^-1 r) on the fly: the Jacobi scaling and the p-update ride on the
// operator's gather. p is double-buffered by iteration parity.
//
// PCG node update (k_pcg_update): x += alpha p, r -= alpha q (Dirichlet rows
// q = char_diag p), z = D^-1 r, and the r.r / r.z partial sums; loads are
// issued for several entries before any store so they overlap.
//
// Reductions of the PCG loop: each block of a kernel writes its partial sums, and
// every block of the next kernel adds all of them in the same fixed order at its
// start, while its first loads are in flight, and derives the iteration's scalars
// from the totals (pcg_fold_update, pcg_fold_patch); block 0 stores them. A last-block
// sum at the end of each kernel instead (fence, ticket, one warp walking the partials,
// scalars, state store, then the next kernel's load of the state) put 3 to 4 us of
// dependent latency behind each of the two kernels: with the folds an iteration takes
// 13.0 instead of 19.0 us at 6^3 (FP64), 23.9 instead of 33.4 us at 48x48x32 (mixed)
// and 24.1 instead of 31.0 us for FP64 elasticity at 27x22x13. Two copies of PcgState
// alternate, so that block 0 never writes the copy that other blocks of its grid still
// read. The kernels outside the loop (start, refresh) keep the ticket form. The loop is
// one CUDA graph that the device steers (build_loop): no host round trip within a solve
// and no grid-wide spin wait.
#pragma once

#include <type_traits>

#include "matfree.cuh"
#include "patches.h"

namespace geo {

constexpr int kPatchBS = 192;  // threads of the patch kernel (2 elements each)
constexpr int kNodeBS = 256;   // threads of the node kernels
constexpr int kUnroll = 4;     // entries in flight per thread in the node kernels
constexpr int kForeignFlight = 2;  // foreign nodes in flight per thread in the gather

enum : int { MODE_FREE = 0, MODE_LIFT = 1, MODE_PCG = 2 };
enum : int { ST_DONE = 1, ST_REFRESH = 2, ST_CONVERGED = 4, ST_BREAKDOWN = 8 };
// Second copy of the state only: both copies say done or refresh, and the node updates left
// in the chunk return at once. Without it they loaded their vectors and folded the partials
// in first: a solve that ends at once takes 109 instead of 144 us at 6^3 (FP64), 100
// iterations with their refreshes 1.55 instead of 1.71 ms (mixed).
enum : int { ST_IDLE = 16 };

struct PatchMeta;

struct PatchView {
    int64_t E, N;
    int n_patches, max_local, dpn;
    const int32_t* pe;
    const int32_t* po;
    const int32_t* pf;
    const int32_t* foreign;
    const uint32_t* lc;    // patch-major paired connectivity [P][5][kPatchElems], FP64 kernels
    const uint32_t* lc32;  // the same for the FP32 kernels (PatchLayout::lc32)
    const uint8_t* flags;
    // scatter bound per patch (see Scatter): (max element incidences of a
    // patch-local node) x max_e ||K_e||_inf x 1.001, rounded up
    const float* bound32;
    // foreign ids and flags again, in per-patch segments that start at pfa[p]
    // (multiples of kForeignAlign entries) so that they travel with the patch's
    // bulk copy; max_for = the largest foreign count of a patch
    const int32_t* pfa;
    const int32_t* fids;
    const uint8_t* fflags;
    int max_for;
    int max_own;   // the largest own-node count of a patch
    int own_bulk;  // PCG: own-node slices by bulk copy (the launch's shared memory holds them)
    // halo mode: the halo slot of every foreign entry, in the same per-patch segments as fids
    const int32_t* fslot;
    // per patch: element count, own range, foreign count and segment start, scatter
    // bound, as one 32-byte record (16-byte aligned), so that the patch kernel's
    // copy issue needs one prefetched record instead of dependent global loads
    const PatchMeta* rec;
};

// ------------------------------------------------------------------ shared-memory scatter
// Element contributions are accumulated in shared memory as exact integers.
// Every contribution c of a patch is scaled by a power of two S chosen so that
// the sum of all contributions to one DOF stays below kLim, then rounded to an
// integer held in kWords INT32 words. Integer sums are exact, so the
// accumulation does not depend on the order of the atomics, and INT32 shared
// atomics cost a fraction of FP32 / FP64 ones (on B200, random banks: about 3.7
// SM cycles per warp operation against 13.4 for FP32 and 22 for FP64).
// The bound behind S is rigorous: K_e annihilates constants (thermal) and
// rigid translations (elasticity), so |(K_e x)_i| <= ||K_e||_inf * max_c h_c,
// h_c = half the range of component c of x over the patch; a margin of 2^-16
// max|x| covers the rounding of the apply, and the patch's largest number of
// element incidences per node bounds the sum (PatchView::bound32).
// FP32: one word (|sum| < 2^30, resolution 2^-30 of the bound). FP64: three
// words holding hi 2^42 + mid 2^21 + lo (|sum| < 2^62, resolution 2^-62 of the
// bound, below the FP64 rounding of the result).
template <class T>
struct Scatter;

template <>
struct Scatter<float> {
    static constexpr int kLimExp = 30;
    static constexpr int kWords = 1;
};

template <>
struct Scatter<double> {
    static constexpr int kLimExp = 62;
    static constexpr int kWords = 3;
};

// The patch-local node table: values x and fixed-point accumulators of every local
// node, addressed by the node's handle, which comes from the element connectivity
// (of_lc) or from the local index u (of_node; consecutive nodes of one aligned group
// are kStep apart).
template <class T, int DPN>
struct NodeTable;

// FP32: rows of 32 nodes, each row the nodes' values and then their accumulators, so
// that both sit at fixed distances from one byte address (see patch_slot32).
template <int DPN>
struct NodeTable<float, DPN> {
    unsigned char* tab;
    __device__ NodeTable(unsigned char* base, int) : tab(base) {}
    __host__ __device__ static size_t bytes(int max_local) { return (size_t)(max_local + 32) / 33 * (66 * 4 * DPN); }
    static constexpr int kStep = 4 * DPN;
    __device__ __forceinline__ static int of_lc(uint32_t v) { return (int)v * DPN; }
    __device__ __forceinline__ static int of_node(int u) { return patch_slot32(u) * (4 * DPN); }
    __device__ __forceinline__ float& x(int h, int c) const { return *reinterpret_cast<float*>(tab + h + 4 * c); }
    __device__ __forceinline__ int& acc(int h, int c) const {
        return *reinterpret_cast<int*>(tab + 33 * 4 * DPN + h + 4 * c);
    }
    __device__ __forceinline__ void add(int h, int c, float v) const { atomicAdd(&acc(h, c), __float2int_rn(v)); }
    // read and clear (the flush leaves the table zero for the next patch)
    __device__ __forceinline__ float take(int h, int c) const {
        int& a = acc(h, c);
        const int v = a;
        a = 0;
        return (float)v;
    }
};

// FP64: the values by slot, then the three accumulator words, word w of slot s at w M + s.
template <int DPN>
struct NodeTable<double, DPN> {
    double* xs;
    int* ys;
    int M;
    __device__ NodeTable(unsigned char* base, int max_local)
        : xs(reinterpret_cast<double*>(base)), ys(reinterpret_cast<int*>(base + (size_t)max_local * DPN * 8)),
          M(max_local * DPN) {}
    __host__ __device__ static size_t bytes(int max_local) { return (size_t)max_local * DPN * (8 + 3 * 4); }
    static constexpr int kStep = DPN;
    __device__ __forceinline__ static int of_lc(uint32_t v) { return (int)v * DPN; }
    __device__ __forceinline__ static int of_node(int u) { return patch_slot(u) * DPN; }
    __device__ __forceinline__ double& x(int h, int c) const { return xs[h + c]; }
    // v = hi 2^42 + mid 2^21 + lo; hi and mid are exact, lo rounds the last fraction
    __device__ __forceinline__ void add(int h, int c, double v) const {
        const int hi = __double2int_rn(v * 2.2737367544323206e-13);  // 2^-42
        const double r = fma(-(double)hi, 4398046511104.0, v);         // 2^42, exact
        const int mid = __double2int_rn(r * 4.76837158203125e-07);    // 2^-21
        const int lo = __double2int_rn(fma(-(double)mid, 2097152.0, r));
        int* acc = ys + h + c;
        atomicAdd(acc, hi);
        atomicAdd(acc + M, mid);
        atomicAdd(acc + 2 * M, lo);
    }
    __device__ __forceinline__ double take(int h, int c) const {
        int* acc = ys + h + c;
        const double v = fma((double)acc[0], 4398046511104.0, fma((double)acc[M], 2097152.0, (double)acc[2 * M]));
        acc[0] = acc[M] = acc[2 * M] = 0;
        return v;
    }
};

// S = the largest power of two <= 2^lim_exp / bx, clamped to [2^-100, 2^hi], and
// 1/S, both exact, from the exponent field of bx > 0 (no division): with
// bx = m 2^e, m in [1, 2), S = 2^(lim_exp - e) when m = 1, else 2^(lim_exp - e - 1);
// a subnormal bx gives the upper clamp, an infinite one the lower.
__device__ __forceinline__ void pow2_scale(float bx, int lim_exp, int hi, float& S, float& invS) {
    const unsigned bits = __float_as_uint(bx);
    const int ef = (int)(bits >> 23);
    int se = lim_exp - (ef - 127) - ((bits & 0x7fffffu) != 0u ? 1 : 0);
    if (ef == 0) se = hi;
    if (ef == 255) se = -100;
    se = min(max(se, -100), hi);
    S = __uint_as_float((unsigned)(se + 127) << 23);
    invS = __uint_as_float((unsigned)(127 - se) << 23);
}

// 16-byte vector of T
template <class T>
struct Vec16;
template <>
struct Vec16<float> {
    using type = float4;
    static constexpr int N = 4;
};
template <>
struct Vec16<double> {
    using type = double2;
    static constexpr int N = 2;
};

// float <-> unsigned key with the same order (for warp min/max reductions)
__device__ __forceinline__ unsigned float_key(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_float(unsigned k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Device-resident PCG scalars.
struct PcgScalars {
    double rz, rz_old, pAp, alpha, beta, bnorm, s_scale, rmax, res, ratio, s_new;
    double tol, abs_tol, delta, cd;
    long long it, max_it, nupd;
    int flags;
    int pending;  // the node update's partials (r.r, r.z) are not folded in yet
};
// With the words that the kernels of the loop do not copy along (first copy only): the
// DEV_ERR_* bits raised by bounded waits, the ticket counter, and the chunks run and
// allowed.
struct PcgState : PcgScalars {
    int err;
    unsigned int ticket;
    long long chunks, max_chunks;
};

template <class T>
struct PatchArgs {
    const T* x;  // FREE / LIFT input
    T* y;        // output (free rows)
    // PCG mode
    const T* r;
    const T* dinv;
    T* pbuf0;
    T* pbuf1;
    const PcgState* st;    // state left by the node update (or the start / refresh kernels)
    PcgState* st_out;      // the state the node update reads
    const double* part_in; // [n_in][2] partials of the node update
    int n_in;
    double* part;          // [gridDim.x][2] p.Ap partials of this kernel
    int* err;      // DEV_ERR_* bits (bounded waits)
    T* halo;       // halo mode: foreign contributions by slot (DPN values each)
    T* xsol;       // PCG z-form: the FP32 solution correction, updated on the own nodes
};

// ------------------------------------------------------------------ bulk copy + mbarrier
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
// global -> shared bulk copy (no multicast); dst/src 16-byte aligned, bytes % 16 == 0
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait (2 s of %globaltimer); returns false on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_timer_ns();
    while (!mbar_try_wait(bar, parity))
        if (global_timer_ns() - t0 > 2000000000ull) return false;
    return true;
}

// Programmatic dependent launch (kDependentDofs): lets the next kernel of the stream start
// its blocks once every block has come here, and waits until the kernels before this one
// are complete and their writes visible (a kernel triggers after its own wait, so this
// covers all earlier ones too). Both do nothing without the attribute. The trigger stands
// after a kernel's work: at its start the next kernel's blocks take the SM's issue slots
// (elastic 48x48x24 42.9 us per iteration against 40.8, thermal 64^3 94.4 against 92.5).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Last-block detection after every block stored its partial. Thread 0 wrote the
// partial (store_partial), so its fence alone orders it before the ticket; the
// block's other stores are for the next kernel.
__device__ __forceinline__ bool last_block(unsigned int* ticket) {
    __shared__ int s_last;
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (s_last) __threadfence();
    return s_last != 0;
}

// The scalars of an iteration that the kernels of the loop work with.
struct PcgHead {
    double alpha, beta, cd;
    int odd;  // parity of the iteration count
    int flags;
};

// The state after a node update whose sums of r.r and r.z are rr and rz: the stopping
// and refresh tests and beta (iterative.rs:95-110).
template <bool MIXED>
__device__ __forceinline__ void pcg_next_iteration(PcgScalars& s, double rr, double rz) {
    s.pending = 0;
    const double rn = sqrt(rr);
    if (!MIXED) {
        s.res = rn;
        if (rn < s.tol * s.bnorm || rn < s.abs_tol) {  // iterative.rs:95
            s.flags |= ST_DONE | ST_CONVERGED;
            return;
        }
    }
    s.beta = rz / s.rz;
    s.rz_old = s.rz;
    s.rz = rz;
    s.it += 1;
    if (MIXED) {
        s.rmax = fmax(s.rmax, rn);
        const double est = rn * s.s_scale;
        if (est < s.tol * s.bnorm || est < s.abs_tol || rn < s.delta * s.rmax || s.it >= s.max_it)
            s.flags |= ST_REFRESH;
    } else if (s.it >= s.max_it) {
        s.flags |= ST_DONE;
    }
}

// The state after a patch kernel whose sums are t[0] = sum_e p_e.K_e p_e and t[1] =
// p.p over Dirichlet rows: p.Ap, alpha, breakdown (iterative.rs:85).
__device__ __forceinline__ void pcg_step_length(PcgScalars& s, double t0, double t1) {
    if (s.flags & (ST_DONE | ST_REFRESH)) return;
    const double pAp = t0 + s.cd * t1;
    s.pAp = pAp;
    if (fabs(pAp) < 1e-30) {
        s.flags |= ST_DONE | ST_BREAKDOWN;
        s.alpha = 0.0;  // no step: the z-form's pending x update adds nothing
    } else {
        s.alpha = s.rz / pAp;
        s.pending = 1;
    }
}

// Start of a kernel of the loop: adds the previous kernel's partials and advances the
// state with step(scalars, t0, t1). Every thread gets the scalars, block 0 stores the
// state for the next kernel.
template <class Step>
__device__ __forceinline__ PcgHead pcg_fold(const PcgState* in, PcgState* out,
                                            const double* __restrict__ part, int n, Step&& step) {
    __shared__ PcgScalars s_st;  // worked on in place: few registers are live here
    constexpr int kWords = sizeof(PcgScalars) / 8;
    static_assert(sizeof(PcgScalars) % 8 == 0 && kWords <= 32, "the state is copied as 8-byte words by one warp");
    double* words = reinterpret_cast<double*>(&s_st);
    if (threadIdx.x < kWords)
        words[threadIdx.x] = __ldcg(reinterpret_cast<const double*>(static_cast<const PcgScalars*>(in)) + threadIdx.x);
    double t[2];
    grid_sum0<2>(part, n, t);  // its block barriers order s_st before the reads below
    if (threadIdx.x == 0) step(s_st, t[0], t[1]);
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x < kWords)
        reinterpret_cast<double*>(static_cast<PcgScalars*>(out))[threadIdx.x] = words[threadIdx.x];
    return PcgHead{s_st.alpha, s_st.beta, s_st.cd, (int)(s_st.it & 1), s_st.flags};
}

// End of a chunk of iterations: folds the last node update's partials in and decides
// whether the graph's loop runs another chunk (`again`) and whether the refresh comes
// first (`refresh`, mixed). One block.
template <bool MIXED>
__global__ void __launch_bounds__(kNodeBS) k_pcg_decide(PcgState* st, const double* __restrict__ part, int n,
                                                        cudaGraphConditionalHandle again,
                                                        cudaGraphConditionalHandle refresh) {
    const PcgHead h = pcg_fold(st, st, part, n, [](PcgScalars& s, double t0, double t1) {
        if (s.pending) pcg_next_iteration<MIXED>(s, t0, t1);
    });
    if (threadIdx.x == 0) {
        const long long chunks = ++st->chunks;
        const bool stop = (h.flags & ST_DONE) || st->err || chunks >= st->max_chunks;
        cudaGraphSetConditional(again, stop ? 0u : 1u);
        if (MIXED) cudaGraphSetConditional(refresh, !stop && (h.flags & ST_REFRESH) ? 1u : 0u);
    }
}

// bytes of one patch's element data (connectivity + qdata), 16-byte multiple
template <class K, class T>
__host__ __device__ constexpr uint32_t patch_bytes_lc() { return 5 * kPatchElems * 4; }
template <class K, class T>
__host__ __device__ constexpr uint32_t patch_bytes_qd() { return K::NQD * kPatchElems * (uint32_t)sizeof(T); }

constexpr int kForeignAlign = 16;  // foreign segments start at multiples of 16 entries

__host__ __device__ inline uint32_t round16(uint32_t b) { return (b + 15u) & ~15u; }

// A patch's sizes, written by the issuing thread next to its bulk copies.
struct __align__(16) PatchMeta {
    int n_el, o0, nown, nfor, fa;
    float bound;  // PatchView::bound32 of the patch
    int pad0, pad1;
};

// PatchView::rec from the per-patch offsets and bounds
__global__ void k_patch_records(PatchView pv, PatchMeta* __restrict__ rec) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= pv.n_patches) return;
    PatchMeta m;
    m.n_el = pv.pe[p + 1] - pv.pe[p];
    m.o0 = pv.po[p];
    m.nown = pv.po[p + 1] - m.o0;
    m.nfor = pv.pf[p + 1] - pv.pf[p];
    m.fa = pv.pfa[p];
    m.bound = pv.bound32[p];
    m.pad0 = m.pad1 = 0;
    rec[p] = m;
}

// 16-byte asynchronous copy global -> shared (cp.async, no bulk); completes at cp_async_wait_all
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// per-buffer bytes of [meta | foreign ids | foreign flags | halo slots (halo mode 1)]
__host__ __device__ inline uint32_t patch_aux_ids(int max_for) {
    return round16((uint32_t)((max_for + kForeignAlign - 1) / kForeignAlign * kForeignAlign) * 4u);
}
__host__ __device__ inline uint32_t patch_aux_flags(int max_for) {
    return round16((uint32_t)((max_for + kForeignAlign - 1) / kForeignAlign * kForeignAlign));
}
__host__ __device__ inline uint32_t patch_aux_bytes(int max_for, int halo) {
    return (uint32_t)sizeof(PatchMeta) + patch_aux_ids(max_for) + patch_aux_flags(max_for) +
           (halo == 1 ? patch_aux_ids(max_for) : 0u);
}

// Own-node slices (PCG mode): D^-1, r and p_old (z-form: z, p_old, x) over the patch's
// own nodes [o0, o1), rounded outwards to kNodeAlign nodes (components interleaved, so
// the range is contiguous and starts on 16 bytes), and the flags of its own nodes,
// copied with cp.async.bulk. Capacities: values per array, flag bytes.
template <class T>
__host__ __device__ inline uint32_t own_cap(int max_own, int dpn) {
    return (uint32_t)((max_own + 3 * kNodeAlign - 1) / kNodeAlign * kNodeAlign * dpn);
}
__host__ __device__ inline uint32_t own_capf(int max_own) { return (uint32_t)(max_own + 32 + 15) & ~15u; }
template <class T>
__host__ __device__ inline uint32_t own_bytes(int max_own, int dpn) {
    return 3u * own_cap<T>(max_own, dpn) * (uint32_t)sizeof(T) + own_capf(max_own);
}

// shared memory layout: [3 mbarriers (32 B) | node table | NBUF x (lc | qd) | NBUF x (meta | foreign ids |
// foreign flags | slots) | node flags (atomics mode) | own-node slices (PCG)]
constexpr uint32_t kPatchBars = 32;
template <class K, class T>
__host__ __device__ inline uint32_t patch_table_bytes(int max_local) {
    return round16((uint32_t)NodeTable<T, K::DPN>::bytes(max_local));
}
template <class K, class T>
__host__ __device__ constexpr uint32_t patch_elem_bytes() { return patch_bytes_lc<K, T>() + patch_bytes_qd<K, T>(); }
template <class K, class T, int NBUF>
__host__ __device__ inline uint32_t patch_flag_bytes(int max_local, int halo) {
    return halo ? 0u : round16((uint32_t)(max_local * NBUF));
}
template <class K, class T, int NBUF>
__host__ __device__ inline size_t patch_smem_bytes(int max_local, int max_for, int max_own, bool own, int halo) {
    return kPatchBars + patch_table_bytes<K, T>(max_local) + NBUF * patch_elem_bytes<K, T>() +
           NBUF * patch_aux_bytes(max_for, halo) + patch_flag_bytes<K, T, NBUF>(max_local, halo) +
           (own ? own_bytes<T>(max_own, K::DPN) : 0u);
}

// Resident blocks per SM the register allocation must allow (the minimum-blocks
// argument of the launch bounds): FP32 elasticity and FP64 thermal 2, FP64
// elasticity 1, as many as their shared memory allows on the bench meshes. FP32
// thermal gets no target (0): it compiles to 79-80 registers, 4 blocks of 192
// threads, by itself, and a target of 4 made the same register count run 2% slower.
template <class K, class T>
__host__ __device__ constexpr int patch_min_blocks() {
    return sizeof(T) == 4 ? (K::DPN == 1 ? 0 : 2) : (K::DPN == 1 ? 2 : 1);
}

// HM: 0 atomics, 1 halo mode with the slots in the bulk copy, 2 halo mode with the slots
// read from global memory by the flush.
//
// A patch's own nodes are gathered and flushed in aligned groups of V consecutive nodes
// (16 bytes per component array) by one thread, with 16-byte accesses; only the edge
// groups, which hold a neighbour patch's nodes too, go node by node. With the groups,
// the foreign values requested before the flush of the patch before, one copy schedule
// (late) for all kernels and the shorter affine apply, launches went from 264 to 249 us
// (FP32 thermal, 128^3), 83 to 75 us (FP64 thermal, 64^3) and 37.3 to 33.2 us (FP32
// elasticity, 48x48x24), events around each launch. No unit is saturated: in the FP32
// thermal kernel (96^3) the L1 data pipe, which gather and scatter share, is at 67% of its
// peak (21 M wavefronts, 11 M of them bank conflicts, for 5.3 M elements), issue at 60%; at
// 128^3 the card's 1 kW power cap holds the clock at 1.9 GHz. FP64: pipe 70%, issue 42%,
// two blocks of six warps per SM.
template <class K, class T, int MODE, int NBUF, int HM>
__global__ void __launch_bounds__(kPatchBS, patch_min_blocks<K, T>())
    k_patch(PatchView pv, const T* __restrict__ qd_all, T cl, T cm, PatchArgs<T> a) {
    constexpr int DPN = K::DPN;
    constexpr uint32_t LCB = patch_bytes_lc<K, T>(), QDB = patch_bytes_qd<K, T>();
    constexpr bool HALO = HM != 0;
    using VT = typename Vec16<T>::type;
    constexpr int V = Vec16<T>::N;  // nodes per group; DPN vectors of 16 bytes per array
    using Table = NodeTable<T, DPN>;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem);  // [0..NBUF): element data; [2]: own-node slices
    const bool OWNB = MODE == MODE_PCG && pv.own_bulk != 0;
    const uint32_t AUX = patch_aux_bytes(pv.max_for, HM), AIDS = patch_aux_ids(pv.max_for);
    const uint32_t AFL = patch_aux_flags(pv.max_for);
    const Table tab(smem + kPatchBars, pv.max_local);
    unsigned char* ebuf = smem + kPatchBars + patch_table_bytes<K, T>(pv.max_local);
    unsigned char* abuf = ebuf + NBUF * (LCB + QDB);  // NBUF x (meta | ids | flags | slots)
    uint8_t* sfl0 = abuf + NBUF * AUX;                // node flags (atomics mode)
    T* own_a = reinterpret_cast<T*>(sfl0 + patch_flag_bytes<K, T, NBUF>(pv.max_local, HM));
    const uint32_t OCAP = own_cap<T>(pv.max_own, DPN);
    T* own_b = own_a + OCAP;
    T* own_c = own_b + OCAP;
    uint8_t* own_f = reinterpret_cast<uint8_t*>(own_c + OCAP);
    // FP32 scatter: per component, min and max of x over the patch as order keys, by patch parity
    __shared__ unsigned s_lo[2][DPN], s_hi[2][DPN];
    // Preconditioned-residual form of the mixed solver's FP32 PCG (thermal and elasticity):
    // the node update keeps z = D^-1 r (a.r holds z) instead of r, so the gather
    // forms p = z + beta p_old from two vectors, and the solution update
    // x += alpha_prev p_old of the previous iteration rides here, on the own nodes'
    // p_old (a.xsol holds the FP32 solution). The FP64 drop-in keeps the
    // reference's form (iterative.rs:46-119).
    constexpr bool ZF = MODE == MODE_PCG && std::is_same<T, float>::value;
    if (threadIdx.x == 0) {
        for (int b = 0; b < NBUF; ++b) mbar_init(&bar[b], 1);
        if (OWNB) mbar_init(&bar[2], 1);
        mbar_fence_init();
        for (int c = 0; c < DPN; ++c) {
            s_lo[0][c] = s_lo[1][c] = 0xffffffffu;
            s_hi[0][c] = s_hi[1][c] = 0u;
        }
    }
    // the accumulators start at zero; each flush clears what it reads
    for (uint32_t i = threadIdx.x; i < patch_table_bytes<K, T>(pv.max_local) / 4; i += blockDim.x)
        reinterpret_cast<int*>(smem + kPatchBars)[i] = 0;
    __syncthreads();
    // Thread 0 issues the copies of patch q_j (the block's j-th patch) from its record
    // in s_rec[j & 1], prefetched by cp.async when q_(j-1) was issued, so that no
    // issue waits on a global load.
    __shared__ PatchMeta s_rec[2];
    auto prefetch_rec = [&](int patch, int slot) {
        cp_async16(&s_rec[slot], pv.rec + patch);
        cp_async16(reinterpret_cast<unsigned char*>(&s_rec[slot]) + 16,
                   reinterpret_cast<const unsigned char*>(pv.rec + patch) + 16);
        cp_async_commit();
    };
    // thread 0: the patch's element data, sizes, foreign ids and foreign flags into buffer b
    const uint32_t* lc_all = sizeof(T) == 4 ? pv.lc32 : pv.lc;
    auto issue = [&](const PatchMeta& m, int patch, int b) {
        unsigned char* ab = abuf + (size_t)b * AUX;
        *reinterpret_cast<PatchMeta*>(ab) = m;  // published by the arrive below
        const uint32_t ib = round16((uint32_t)m.nfor * 4u), fb = round16((uint32_t)m.nfor);
        unsigned char* dst = ebuf + (size_t)b * (LCB + QDB);
        mbar_expect_tx(&bar[b], LCB + QDB + ib + fb + (HM == 1 ? ib : 0u));
        bulk_g2s(dst, lc_all + (size_t)patch * 5 * kPatchElems, LCB, &bar[b]);
        bulk_g2s(dst + LCB, qd_all + (size_t)patch * K::NQD * kPatchElems, QDB, &bar[b]);
        if (ib) {
            bulk_g2s(ab + sizeof(PatchMeta), pv.fids + m.fa, ib, &bar[b]);
            bulk_g2s(ab + sizeof(PatchMeta) + AIDS, pv.fflags + m.fa, fb, &bar[b]);
            if (HM == 1) bulk_g2s(ab + sizeof(PatchMeta) + AIDS + AFL, pv.fslot + m.fa, ib, &bar[b]);
        }
    };
    // The first patch's element data and lists are the operator's: requested before the
    // wait for the kernel before this one.
    if (threadIdx.x == 0 && blockIdx.x < pv.n_patches) {
        issue(pv.rec[blockIdx.x], blockIdx.x, 0);
        if (blockIdx.x + gridDim.x < pv.n_patches) prefetch_rec(blockIdx.x + gridDim.x, 1);
    }
    // bit b: a copy into buffer b is in flight (tracked by thread 0, which issues them)
    uint32_t pend = blockIdx.x < pv.n_patches ? 1u : 0u;
    auto drain = [&]() {  // thread 0: lets the copies land before the block's shared memory is released
        for (int q = 0; q < 3; ++q)
            if ((pend >> q) & 1) mbar_wait(&bar[q], 0);
        cp_async_wait_all();
    };
    if (MODE == MODE_PCG) pdl_wait();
    T beta = T(0), alpha_prev = T(0);
    const T* pold = nullptr;
    T* pnew = nullptr;
    if (MODE == MODE_PCG) {
        if (a.st->flags & (ST_DONE | ST_REFRESH)) {  // nothing to do, for the node update either
            if (blockIdx.x == 0 && threadIdx.x == 0 && !(a.st_out->flags & ST_IDLE)) {
                *static_cast<PcgScalars*>(a.st_out) = *static_cast<const PcgScalars*>(a.st);
                a.st_out->flags |= ST_IDLE;
            }
            if (threadIdx.x == 0) drain();
            return;
        }
        // the direction's buffer after the fold below: it counts the pending iteration
        const bool odd = (a.st->it + a.st->pending) & 1;
        pold = odd ? a.pbuf1 : a.pbuf0;
        pnew = odd ? a.pbuf0 : a.pbuf1;
    }
    // the three own-node arrays: z-form z, p_old, x; else D^-1, r, p_old
    const T* ga = ZF ? a.r : a.dinv;
    const T* gb = ZF ? pold : a.r;
    const T* gc = ZF ? a.xsol : pold;
    // thread 0: the own-node slices and flags of the patch's own nodes (single buffer, bar[2])
    auto issue_own = [&](const PatchMeta& m) {
        const int o0 = m.o0, o1 = m.o0 + m.nown;
        const int n0 = patch_align(o0), nn = (o1 + kNodeAlign - 1) / kNodeAlign * kNodeAlign - n0;
        const int f0 = o0 & ~15, nf = ((o1 + 15) & ~15) - f0;  // flags, 16-byte aligned
        const uint32_t vb = (uint32_t)(nn * DPN) * (uint32_t)sizeof(T);
        mbar_expect_tx(&bar[2], 3u * vb + (uint32_t)nf);
        if (vb) {
            const int64_t at = (int64_t)n0 * DPN;
            bulk_g2s(own_a, ga + at, vb, &bar[2]);
            bulk_g2s(own_b, gb + at, vb, &bar[2]);
            bulk_g2s(own_c, gc + at, vb, &bar[2]);
        }
        if (nf) bulk_g2s(own_f, pv.flags + f0, (uint32_t)nf, &bar[2]);
    };
    // thread 0: patch + gridDim.x (the block's (k+1)-th) into buffer b from its prefetched
    // record, and the record after it into the slot just read from
    auto issue_next = [&](int patch, int k, int b) {
        cp_async_wait_all();
        const PatchMeta m = s_rec[(k + 1) & 1];
        issue(m, patch + gridDim.x, b);
        if (patch + 2 * (int)gridDim.x < pv.n_patches) prefetch_rec(patch + 2 * gridDim.x, k & 1);
    };
    if (OWNB && blockIdx.x < pv.n_patches) {
        if (threadIdx.x == 0) issue_own(pv.rec[blockIdx.x]);
        pend |= 4u;
    }
    uint32_t phase = 0;  // bit b = parity of buffer b; bit 2 = parity of the own-node buffer
    if (MODE == MODE_PCG) {  // the first patch's copies are in flight
        const PcgHead h = pcg_fold(a.st, a.st_out, a.part_in, a.n_in, [](PcgScalars& s, double t0, double t1) {
            if (s.pending) pcg_next_iteration<ZF>(s, t0, t1);
        });
        if (h.flags & (ST_DONE | ST_REFRESH)) {
            if (threadIdx.x == 0) drain();
            return;
        }
        beta = (T)h.beta;
        if (ZF) alpha_prev = (T)h.alpha;
    }
    // Foreign nodes go to scattered global addresses. Each thread has the values of up to
    // kForeignFlight of them in flight: with two element buffers they are requested
    // before the flush of the patch before (its element phase has brought the list), so
    // that the flush and the own nodes of the gather cover their latency.
    uint8_t ffl[kForeignFlight];
    T f0[kForeignFlight][DPN], f1[kForeignFlight][DPN], f2[kForeignFlight][DPN];
    auto f_load = [&](int b, int i, uint8_t& fl, T (&v0)[DPN], T (&v1)[DPN], T (&v2)[DPN]) {
        const unsigned char* ab = abuf + (size_t)b * AUX;
        if (i >= reinterpret_cast<const PatchMeta*>(ab)->nfor) return;
        const int64_t at = (int64_t)reinterpret_cast<const int*>(ab + sizeof(PatchMeta))[i] * DPN;
        fl = (ab + sizeof(PatchMeta) + AIDS)[i];
#pragma unroll
        for (int c = 0; c < DPN; ++c) {
            if (MODE != MODE_PCG) {
                v0[c] = a.x[at + c];
            } else {
                v0[c] = ga[at + c];
                v1[c] = gb[at + c];
                if (!ZF) v2[c] = gc[at + c];
            }
        }
    };
    // waits for the element data and lists in buffer b and requests the foreign values
    auto arrive = [&](int b) {
        if (!mbar_wait(&bar[b], (phase >> b) & 1)) return false;
        phase ^= 1u << b;
        pend &= ~(1u << b);
#pragma unroll
        for (int g = 0; g < kForeignFlight; ++g) f_load(b, threadIdx.x + g * kPatchBS, ffl[g], f0[g], f1[g], f2[g]);
        return true;
    };
    double dot = 0.0, pdd = 0.0;
    // A thread whose bounded wait ran out skips the next gather, and the gather barrier
    // ends the block.
    bool ok = true;
    if (NBUF == 2 && blockIdx.x < pv.n_patches) ok = arrive(0);
    int k = 0;
    for (int patch = blockIdx.x; patch < pv.n_patches; patch += gridDim.x, ++k) {
        const int b = NBUF == 2 ? (k & 1) : 0;
        const bool has_next = patch + (int)gridDim.x < pv.n_patches;
        if (NBUF == 1) ok = arrive(b);
        if (OWNB) {
            const bool ok2 = mbar_wait(&bar[2], (phase >> 2) & 1);
            if (ok2) {
                phase ^= 4u;
                pend &= ~4u;
            }
            ok = ok && ok2;
        }
        // node flags for the flush (atomics mode): with two buffers one table per patch
        // parity, since the flush of one patch reads them while faster warps gather the next
        uint8_t* sfl = sfl0 + b * pv.max_local;
        const unsigned char* ab = abuf + (size_t)b * AUX;
        const PatchMeta pm = *reinterpret_cast<const PatchMeta*>(ab);
        const int* __restrict__ sfor = reinterpret_cast<const int*>(ab + sizeof(PatchMeta));
        const int* __restrict__ sfsl = reinterpret_cast<const int*>(ab + sizeof(PatchMeta) + AIDS + AFL);
        const int o0 = pm.o0, o1 = pm.o0 + pm.nown, n0 = patch_align(o0);
        const int uf = o1 - n0;  // local index of the first foreign node
        float xlo[DPN], xhi[DPN];
#pragma unroll
        for (int c = 0; c < DPN; ++c) {
            xlo[c] = 3.0e38f;
            xhi[c] = -3.0e38f;
        }
        auto range = [&](int c, T v) {
            xlo[c] = fminf(xlo[c], (float)v);
            xhi[c] = fmaxf(xhi[c], (float)v);
        };
        // 1. gather
        const int nfor = ok ? pm.nfor : 0, ngrp = ok ? (o1 - n0 + V - 1) / V : 0;
        auto f_store = [&](int i, uint8_t fl, const T (&v0)[DPN], const T (&v1)[DPN], const T (&v2)[DPN]) {
            if (i >= nfor) return;
            const int h = Table::of_node(uf + i);
            if (!HALO) sfl[uf + i] = fl;
#pragma unroll
            for (int c = 0; c < DPN; ++c) {
                const bool dir = (fl >> c) & 1;
                T v;
                if (MODE == MODE_PCG) v = dir ? T(0) : (ZF ? v0[c] + beta * v1[c] : v0[c] * v1[c] + beta * v2[c]);
                else v = (MODE == MODE_FREE ? dir : !dir) ? T(0) : v0[c];
                tab.x(h, c) = v;
                range(c, v);
            }
        };
        for (int grp = threadIdx.x; grp < ngrp; grp += kPatchBS) {
            const int j0 = n0 + V * grp;  // first node of the group
            const bool full = j0 >= o0 && j0 + V <= o1;
            const int64_t at = (int64_t)(j0 / V) * DPN;  // in vectors
            VT va[DPN], vb[DPN], vc[DPN];
            unsigned fw;
            const uint8_t* fp = OWNB ? own_f + (j0 - (o0 & ~15)) : pv.flags + j0;
            if (V == 4) fw = *reinterpret_cast<const uint32_t*>(fp);
            else fw = *reinterpret_cast<const uint16_t*>(fp);
            if (MODE != MODE_PCG) {
                if (full) {
#pragma unroll
                    for (int q = 0; q < DPN; ++q) va[q] = reinterpret_cast<const VT*>(a.x)[at + q];
                } else {
#pragma unroll
                    for (int e = 0; e < V; ++e)
                        if (j0 + e >= o0 && j0 + e < o1)
#pragma unroll
                            for (int c = 0; c < DPN; ++c)
                                reinterpret_cast<T*>(va)[e * DPN + c] = a.x[(int64_t)(j0 + e) * DPN + c];
                }
            } else if (OWNB) {
#pragma unroll
                for (int q = 0; q < DPN; ++q) {
                    va[q] = reinterpret_cast<const VT*>(own_a)[grp * DPN + q];
                    vb[q] = reinterpret_cast<const VT*>(own_b)[grp * DPN + q];
                    vc[q] = reinterpret_cast<const VT*>(own_c)[grp * DPN + q];
                }
            } else {
#pragma unroll
                for (int q = 0; q < DPN; ++q) {
                    va[q] = reinterpret_cast<const VT*>(ga)[at + q];
                    vb[q] = reinterpret_cast<const VT*>(gb)[at + q];
                    vc[q] = reinterpret_cast<const VT*>(gc)[at + q];
                }
            }
            T* ta = reinterpret_cast<T*>(va);  // becomes p (PCG)
            const T* tb = reinterpret_cast<const T*>(vb);
            T* tc = reinterpret_cast<T*>(vc);  // z-form: becomes x
            const int h0 = Table::of_node(V * grp);
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const bool in = full || (j0 + e >= o0 && j0 + e < o1);
                if (!HALO && in) sfl[V * grp + e] = (uint8_t)(fw >> (8 * e));
#pragma unroll
                for (int c = 0; c < DPN; ++c) {
                    const int q = e * DPN + c;
                    const bool dir = (fw >> (8 * e + c)) & 1;
                    T v;
                    if (MODE == MODE_PCG) {
                        const T pn = ZF ? ta[q] + beta * tb[q] : ta[q] * tb[q] + beta * tc[q];
                        if (ZF) tc[q] = tc[q] + alpha_prev * tb[q];
                        ta[q] = pn;
                        if (dir && in) pdd += (double)(pn * pn);
                        v = dir ? T(0) : pn;
                    } else {
                        v = (MODE == MODE_FREE ? dir : !dir) ? T(0) : ta[q];
                    }
                    if (in) {
                        tab.x(h0 + e * Table::kStep, c) = v;
                        range(c, v);
                    }
                }
            }
            if (MODE == MODE_PCG) {
                if (full) {
#pragma unroll
                    for (int q = 0; q < DPN; ++q) {
                        reinterpret_cast<VT*>(pnew)[at + q] = va[q];
                        if (ZF) reinterpret_cast<VT*>(a.xsol)[at + q] = vc[q];
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < V; ++e)
                        if (j0 + e >= o0 && j0 + e < o1)
#pragma unroll
                            for (int c = 0; c < DPN; ++c) {
                                pnew[(int64_t)(j0 + e) * DPN + c] = ta[e * DPN + c];
                                if (ZF) a.xsol[(int64_t)(j0 + e) * DPN + c] = tc[e * DPN + c];
                            }
                }
            }
        }
#pragma unroll
        for (int g = 0; g < kForeignFlight; ++g) f_store(threadIdx.x + g * kPatchBS, ffl[g], f0[g], f1[g], f2[g]);
        for (int i = threadIdx.x + kForeignFlight * kPatchBS; i < nfor; i += kPatchBS) {
            f_load(b, i, ffl[0], f0[0], f1[0], f2[0]);
            f_store(i, ffl[0], f0[0], f1[0], f2[0]);
        }
#pragma unroll
        for (int c = 0; c < DPN; ++c) {
            const unsigned lo = __reduce_min_sync(0xffffffffu, float_key(xlo[c]));
            const unsigned hi = __reduce_max_sync(0xffffffffu, float_key(xhi[c]));
            if ((threadIdx.x & 31) == 0) {
                atomicMin(&s_lo[k & 1][c], lo);
                atomicMax(&s_hi[k & 1][c], hi);
            }
        }
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) {
                atomicOr(a.err, DEV_ERR_TIMEOUT);
                // let copies still in flight land (bounded waits) before the block's shared memory is released
                for (int q = 0; q < 3; ++q)
                    if ((pend >> q) & 1) mbar_wait(&bar[q], (phase >> q) & 1);
                cp_async_wait_all();
            }
            return;
        }
        // Every warp has left the previous patch's flush: with two buffers its buffer
        // takes the next patch's copy; the own-node buffer (read by the gather only)
        // takes the next patch's slices, during steps 2 and 3.
        if (threadIdx.x == 0 && has_next) {
            if (NBUF == 2) {
                issue_next(patch, k, b ^ 1);
                pend |= 1u << (b ^ 1);
            }
            if (OWNB) {
                // The record of patch + gridDim.x is in its slot: issue_next of this patch
                // waited for it (two buffers), or the previous patch's prefetched it (one
                // buffer). Waiting in the first case would wait for the prefetch just issued.
                if (NBUF == 1) cp_async_wait_all();
                issue_own(s_rec[(k + 1) & 1]);
                pend |= 4u;
            }
        }
        // 2. elements, scattered as fixed-point integers with scale S (see Scatter)
        T S = T(1), invS = T(1);
        {
            float half = 0.0f, mabs = 0.0f;
#pragma unroll
            for (int c = 0; c < DPN; ++c) {
                const float lo = key_float(s_lo[k & 1][c]), hi = key_float(s_hi[k & 1][c]);
                if (hi >= lo) {
                    half = fmaxf(half, __fmul_ru(__fsub_ru(hi, lo), 0.5f));
                    mabs = fmaxf(mabs, fmaxf(fabsf(lo), fabsf(hi)));
                }
            }
            const float bx = __fmul_ru(pm.bound, __fmaf_ru(mabs, 1.52587890625e-05f, half));  // 2^-16
            if (bx > 0.0f) {
                // S multiplies G of the affine thermal elements in the FP32 PCG
                // (ThermalK::apply_affine): it stays below 2^120 / bound, and G below the
                // bound on K_e's norm
                const int cap = min(100, 246 - (int)(__float_as_uint(pm.bound) >> 23));
                float sf, isf;
                pow2_scale(bx, Scatter<T>::kLimExp, MODE == MODE_PCG && DPN == 1 && sizeof(T) == 4 ? cap : 100, sf, isf);
                S = (T)sf;
                invS = (T)isf;
            }
            if (threadIdx.x < DPN) {  // next read by the patch after next
                s_lo[(k + 1) & 1][threadIdx.x] = 0xffffffffu;
                s_hi[(k + 1) & 1][threadIdx.x] = 0u;
            }
        }
        const uint32_t* lcs = reinterpret_cast<const uint32_t*>(ebuf + (size_t)b * (LCB + QDB));
        const T* qds = reinterpret_cast<const T*>(ebuf + (size_t)b * (LCB + QDB) + LCB);
        for (int el = threadIdx.x; el < pm.n_el; el += kPatchBS) {
            int h[10];
            T xe[10 * DPN], ye[10 * DPN];
#pragma unroll
            for (int l2 = 0; l2 < 5; ++l2) {
                const uint32_t w = lcs[l2 * kPatchElems + el];
                h[2 * l2] = Table::of_lc(w & 0xffffu);
                h[2 * l2 + 1] = Table::of_lc(w >> 16);
            }
#pragma unroll
            for (int l = 0; l < 10; ++l)
#pragma unroll
                for (int c = 0; c < DPN; ++c) xe[l * DPN + c] = tab.x(h[l], c);
            K::template apply<MODE == MODE_PCG>(qds + el, kPatchElems, cl, cm, S, xe, ye);
            if (MODE == MODE_PCG) {
                T d = T(0);
#pragma unroll
                for (int q = 0; q < 10 * DPN; ++q) d += xe[q] * ye[q];
                dot += (double)(d * invS);
            }
#pragma unroll
            for (int l = 0; l < 10; ++l)
#pragma unroll
                for (int c = 0; c < DPN; ++c) tab.add(h[l], c, ye[l * DPN + c]);
        }
        __syncthreads();
        if (NBUF == 2 && has_next) ok = arrive(b ^ 1);
        // 3. flush (node ids: the own range, then the foreign list still in the aux buffer)
        if (HALO) {
            // own nodes stored, foreign ones to their halo slots (DPN values each). Dirichlet
            // rows get a value too: no reader uses it.
            for (int grp = threadIdx.x; grp < (o1 - n0 + V - 1) / V; grp += kPatchBS) {
                const int j0 = n0 + V * grp;
                const int h0 = Table::of_node(V * grp);
                if (j0 >= o0 && j0 + V <= o1) {
                    VT yv[DPN];
#pragma unroll
                    for (int e = 0; e < V; ++e)
#pragma unroll
                        for (int c = 0; c < DPN; ++c)
                            reinterpret_cast<T*>(yv)[e * DPN + c] = tab.take(h0 + e * Table::kStep, c) * invS;
#pragma unroll
                    for (int q = 0; q < DPN; ++q) reinterpret_cast<VT*>(a.y)[(int64_t)(j0 / V) * DPN + q] = yv[q];
                } else {
#pragma unroll
                    for (int e = 0; e < V; ++e)
                        if (j0 + e >= o0 && j0 + e < o1)
#pragma unroll
                            for (int c = 0; c < DPN; ++c)
                                a.y[(int64_t)(j0 + e) * DPN + c] = tab.take(h0 + e * Table::kStep, c) * invS;
                }
            }
            for (int i = threadIdx.x; i < pm.nfor; i += kPatchBS) {
                const int h = Table::of_node(uf + i);
                const int64_t at = (int64_t)(HM == 2 ? __ldg(pv.fslot + pm.fa + i) : sfsl[i]) * DPN;
#pragma unroll
                for (int c = 0; c < DPN; ++c) a.halo[at + c] = tab.take(h, c) * invS;
            }
        } else {
            for (int u = o0 - n0 + (int)threadIdx.x; u < uf + pm.nfor; u += kPatchBS) {
                const uint8_t fl = sfl[u];
                const int node = u < uf ? n0 + u : sfor[u - uf];
                const bool plain = u < uf && !(fl & kFlagShared);
                const int h = Table::of_node(u);
#pragma unroll
                for (int c = 0; c < DPN; ++c) {
                    const T v = tab.take(h, c) * invS;
                    if ((fl >> c) & 1) continue;
                    T* dst = a.y + (int64_t)node * DPN + c;
                    if (plain) *dst = v;
                    else atomicAdd(dst, v);
                }
            }
        }
        // Two buffers need no barrier here: the next gather writes the node values (and
        // the other flag table), which no flush reads, and the accumulators are zero again.
        if (NBUF == 1) {
            __syncthreads();
            if (threadIdx.x == 0 && has_next) {
                issue_next(patch, k, 0);
                pend |= 1u;
            }
        }
    }
    if (MODE == MODE_PCG) {
        pdl_trigger();
        double v[2] = {dot, pdd};
        store_partial<2>(a.part, v);
    }
}

// ------------------------------------------------------------------ node kernels
template <class T>
struct NodeArgs {
    const uint8_t* flags;
    int64_t n;
    int dpn;
    T* x;  // solution (FP64 mode) or FP32 correction xs (mixed)
    T* r;
    T* q;
    const T* dinv;
    T* pbuf0;
    T* pbuf1;
    PcgState* st;   // state after the node update; the start and refresh kernels work on it
    const PcgState* st_in;  // node update: the state the patch kernel left
    const double* part_in;  // node update: the patch kernel's partials
    int n_in;
    double* part;
    // mixed refresh
    double* x64;
    double* w64;
    const double* b;
    // halo mode: foreign contributions by slot (dpn values each); node i's slots
    // follow those of nodes < i, hbase[c] = slots of nodes < 32 c, flag bits 3-6 =
    // the node's slot count
    const T* halo;
    const int32_t* hbase;
    const double* halo64;  // mixed refresh: FP64 slots of the FP64 apply (halo mode)
    cudaGraphConditionalHandle again;  // mixed refresh: cleared when it ends the solve
};

constexpr int kHaloShift = 3;  // flag bits 3-6: halo slots of the node (halo mode)

// ro / dj for the norms of the z-form (FP32: the fast reciprocal-multiply, within
// two units in the last place; the stopping and refresh tests do not need more)
__device__ __forceinline__ float fast_div(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ double fast_div(double a, double b) { return a / b; }

// The axpys of one row: x += alpha p, r -= alpha q (Dirichlet rows q = cd p), z = D^-1 r,
// and its terms of r.r and r.z. ZF (the mixed solver's z-form, see k_patch): r holds
// z = D^-1 r, x is not touched (the next patch kernel updates it).
template <class T, bool ZF>
struct PcgRow {
    T alpha, cd;
    T rr = T(0), rz = T(0);
    __device__ __forceinline__ void operator()(bool dir, T p, T q, T dinv, T& x, T& r) {
        const T qq = dir ? cd * p : q;
        if (ZF) {
            r = r - alpha * (dinv * qq);
            const T v = fast_div(r, dinv);
            rr += v * v;
            rz += v * r;
            return;
        }
        x = x + alpha * p;
        r = r - alpha * qq;
        rr += r * r;
        rz += r * (r * dinv);
    }
};

// Folds the patch kernel's partials in (see pcg_fold).
template <class T>
__device__ __forceinline__ PcgHead pcg_fold_patch(const NodeArgs<T>& a) {
    return pcg_fold(a.st_in, a.st, a.part_in, a.n_in,
                    [](PcgScalars& s, double t0, double t1) { pcg_step_length(s, t0, t1); });
}

// Exclusive prefix over the warp of the lanes' slot counts: added to the slots before
// the warp's first node (hbase) it gives a lane's first halo slot. Every lane of the
// warp calls it (lanes past the end pass cnt = 0).
__device__ __forceinline__ int halo_prefix(int cnt, int lane) {
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    return incl - cnt;
}

// First halo slot of node j alone, from the start of its 32-node chunk.
__device__ __forceinline__ int64_t halo_first(const uint8_t* __restrict__ flags, const int32_t* __restrict__ hbase,
                                              int64_t j) {
    int64_t s = hbase[j / 32];
    for (int64_t i = j & ~(int64_t)31; i < j; ++i) s += (flags[i] >> kHaloShift) & 15;
    return s;
}

// Node update of a one-DOF operator in halo mode: q_j = (own-patch sum, stored by the
// patch kernel) + (node j's halo slots, in slot order). Lane l of a warp takes vector
// iv (V nodes); the warp's 32 vectors are 32 V consecutive nodes starting at a multiple
// of 32, so its first slot is hbase[first / 32] and each lane's follows from a warp
// scan of the lanes' slot counts. Loop conditions are warp-uniform.
// The first vector's loads, slot scan and halo sums are issued before the partials of
// the patch kernel are folded in: they need none of the iteration's scalars. One
// vector per array in flight per thread: the halo loads wait on the slot scan, so
// warps hide that latency better than deeper unrolling (two vectors 0.107, four 0.20
// against 0.095 ms at 128^3, FP32).
template <class T, bool ZF>
__device__ __forceinline__ bool pcg_update_halo(const NodeArgs<T>& a, PcgRow<T, ZF>& row) {
    using VT = typename Vec16<T>::type;
    constexpr int V = Vec16<T>::N;
    const uint8_t* __restrict__ flags = a.flags;
    const T* __restrict__ dinv = a.dinv;
    const T* __restrict__ halo = a.halo;
    T* __restrict__ x = a.x;
    T* __restrict__ r = a.r;
    const T* __restrict__ q = a.q;
    const T* __restrict__ p = (a.st_in->it & 1) ? a.pbuf0 : a.pbuf1;
    const int lane = threadIdx.x & 31;
    const int64_t n = a.n, nth = (int64_t)gridDim.x * blockDim.x;
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nv = n / V;
    VT pv, qv, xv, rv, dv;
    unsigned dir;  // bit e: entry e is a Dirichlet row
    auto load = [&](int64_t iv) {
        const bool in = iv < nv;
        int cnt[V], tot = 0;
        dir = 0;
        if (in) {
            qv = reinterpret_cast<const VT*>(q)[iv];
            if (!ZF) xv = reinterpret_cast<const VT*>(x)[iv];
            rv = reinterpret_cast<const VT*>(r)[iv];
            dv = reinterpret_cast<const VT*>(dinv)[iv];
            if (!ZF) pv = reinterpret_cast<const VT*>(p)[iv];
        }
#pragma unroll
        for (int e = 0; e < V; ++e) {
            const uint8_t f = in ? flags[iv * V + e] : (uint8_t)0;
            dir |= (unsigned)(f & 1) << e;
            cnt[e] = (f >> kHaloShift) & 15;
            tot += cnt[e];
        }
        const int64_t first = (iv - lane) * V;
        int64_t sl = (int64_t)a.hbase[first / 32] + halo_prefix(tot, lane);
        T* qe = reinterpret_cast<T*>(&qv);
#pragma unroll
        for (int e = 0; e < V; ++e) {
            T h = T(0);
            for (int i = 0; i < cnt[e]; ++i) h += halo[sl + i];
            sl += cnt[e];
            qe[e] += h;
        }
    };
    int64_t iv = tid;
    if (a.st_in->flags & ST_IDLE) return false;
    if (iv - lane < nv) load(iv);
    const PcgHead h = pcg_fold_patch(a);
    if (h.flags & (ST_DONE | ST_REFRESH)) return false;
    row.alpha = (T)h.alpha;
    row.cd = (T)h.cd;
    while (iv - lane < nv) {
        if (iv < nv) {
            if (ZF && dir) pv = reinterpret_cast<const VT*>(p)[iv];  // z-form: p only where a Dirichlet row needs it
#pragma unroll
            for (int e = 0; e < V; ++e)
                row((dir >> e) & 1, reinterpret_cast<T*>(&pv)[e], reinterpret_cast<T*>(&qv)[e],
                    reinterpret_cast<T*>(&dv)[e], reinterpret_cast<T*>(&xv)[e], reinterpret_cast<T*>(&rv)[e]);
            if (!ZF) reinterpret_cast<VT*>(x)[iv] = xv;
            reinterpret_cast<VT*>(r)[iv] = rv;
        }
        iv += nth;
        if (iv - lane < nv) load(iv);
    }
    for (int64_t j = nv * V + tid; j < n; j += nth) {  // the last n mod V nodes
        const uint8_t f = flags[j];
        const int64_t sl = halo_first(flags, a.hbase, j);
        T hs = T(0), xo = ZF ? T(0) : x[j], ro = r[j];
        for (int i = 0; i < ((f >> kHaloShift) & 15); ++i) hs += halo[sl + i];
        row(f & 1, p[j], q[j] + hs, dinv[j], xo, ro);
        if (!ZF) x[j] = xo;
        r[j] = ro;
    }
    return true;
}

// Node update of a three-DOF operator in halo mode, as pcg_update_halo. FP32: two
// consecutive nodes per lane, so that each vector's six values are three 8-byte loads
// (a lane's pair starts at DOF 6 m) and a warp covers 64 nodes starting at a multiple
// of 64; FP64: one node per lane.
template <class T, bool ZF>
__device__ __forceinline__ bool pcg_update_halo3(const NodeArgs<T>& a, PcgRow<T, ZF>& row) {
    constexpr int P = std::is_same_v<T, float> ? 2 : 1;  // nodes per lane
    const uint8_t* __restrict__ flags = a.flags;
    const T* __restrict__ dinv = a.dinv;
    const T* __restrict__ halo = a.halo;
    T* __restrict__ x = a.x;
    T* __restrict__ r = a.r;
    const T* __restrict__ q = a.q;
    const T* __restrict__ p = (a.st_in->it & 1) ? a.pbuf0 : a.pbuf1;
    const int lane = threadIdx.x & 31;
    const int64_t nn = a.n / 3, nth = (int64_t)gridDim.x * blockDim.x;
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nm = nn / P;
    T pv[3 * P], qv[3 * P], xv[3 * P], rv[3 * P], dv[3 * P];
    unsigned f[P];
    auto get = [&](const T* __restrict__ src, int64_t m, T (&v)[3 * P]) {
        if constexpr (P == 2) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float2 t = reinterpret_cast<const float2*>(src)[3 * m + k];
                v[2 * k] = t.x, v[2 * k + 1] = t.y;
            }
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) v[c] = src[3 * m + c];
        }
    };
    auto put = [&](T* __restrict__ dst, int64_t m, const T (&v)[3 * P]) {
        if constexpr (P == 2) {
#pragma unroll
            for (int k = 0; k < 3; ++k) reinterpret_cast<float2*>(dst)[3 * m + k] = make_float2(v[2 * k], v[2 * k + 1]);
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) dst[3 * m + c] = v[c];
        }
    };
    auto load = [&](int64_t m) {
        const bool in = m < nm;
        int tot = 0;
#pragma unroll
        for (int e = 0; e < P; ++e) {
            f[e] = in ? flags[P * m + e] : 0u;
            tot += (f[e] >> kHaloShift) & 15;
        }
        if (in) {
            get(q, m, qv);
            if (!ZF) get(x, m, xv);
            get(r, m, rv);
            get(dinv, m, dv);
            if (!ZF) get(p, m, pv);
        }
        const int64_t first = (m - lane) * P;
        int64_t sl = (int64_t)a.hbase[first / 32] + halo_prefix(tot, lane);
#pragma unroll
        for (int e = 0; e < P; ++e) {
            const int cnt = (f[e] >> kHaloShift) & 15;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                T h = T(0);
                for (int i = 0; i < cnt; ++i) h += halo[3 * (sl + i) + c];
                qv[3 * e + c] += h;
            }
            sl += cnt;
        }
    };
    int64_t m = tid;
    // not in FP64, whose loads would all wait for it: 27x22x13 0.8% slower per solve
    if (ZF && (a.st_in->flags & ST_IDLE)) return false;
    if (m - lane < nm) load(m);
    const PcgHead h = pcg_fold_patch(a);
    if (h.flags & (ST_DONE | ST_REFRESH)) return false;
    row.alpha = (T)h.alpha;
    row.cd = (T)h.cd;
    while (m - lane < nm) {
        if (m < nm) {
            // z-form: p only where a Dirichlet row needs it
            if (ZF && ((f[0] | f[P - 1]) & 7u)) get(p, m, pv);
#pragma unroll
            for (int e = 0; e < P; ++e)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int v = 3 * e + c;
                    row((f[e] >> c) & 1, pv[v], qv[v], dv[v], xv[v], rv[v]);
                }
            if (!ZF) put(x, m, xv);
            put(r, m, rv);
        }
        m += nth;
        if (m - lane < nm) load(m);
    }
    for (int64_t nd = P * nm + tid; nd < nn; nd += nth) {  // an odd last node
        const unsigned fl = flags[nd];
        const int cnt = (fl >> kHaloShift) & 15;
        const int64_t sl = halo_first(flags, a.hbase, nd);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int64_t j = 3 * nd + c;
            T hs = T(0), xo = ZF ? T(0) : x[j], ro = r[j];
            for (int i = 0; i < cnt; ++i) hs += halo[3 * (sl + i) + c];
            row((fl >> c) & 1, p[j], q[j] + hs, dinv[j], xo, ro);
            if (!ZF) x[j] = xo;
            r[j] = ro;
        }
    }
    return true;
}

// Resident blocks per SM of the halo-mode node update: four (64 registers); the z-form
// of the mixed thermal solver streams four vectors instead of seven and fits six (40
// registers): 0.069 ms at 128^3 against 0.072 ms at five and 0.086 ms at four blocks.
constexpr int kHaloMinBlocks = 4;
constexpr int kHaloMinBlocksZ = 6;

// Node update of a PCG in halo mode (see pcg_update_halo / pcg_update_halo3).
template <class T, int DPN, bool MIXED>
__global__ void __launch_bounds__(kNodeBS, (MIXED && DPN == 1 && std::is_same<T, float>::value) ? kHaloMinBlocksZ
                                                                                             : kHaloMinBlocks)
    k_pcg_update_halo(NodeArgs<T> a) {
    PcgRow<T, MIXED && std::is_same<T, float>::value> row;
    pdl_wait();
    if (DPN == 1) {
        if (!pcg_update_halo(a, row)) return;
    } else {
        if (!pcg_update_halo3(a, row)) return;
    }
    pdl_trigger();
    double v[2] = {(double)row.rr, (double)row.rz};
    store_partial<2>(a.part, v);
}

// Node update in atomics mode (a mesh with a node of more than 15 foreign entries):
// every thread streams 16-byte vectors of p, q, x, r and D^-1, kUnroll in flight, and a
// scalar loop covers the tail. q is zeroed where another patch accumulates into it in
// the next iteration.
template <class T, int DPN, bool MIXED>
__global__ void __launch_bounds__(kNodeBS) k_pcg_update(NodeArgs<T> a) {
    constexpr bool ZF = MIXED && std::is_same<T, float>::value;
    pdl_wait();
    if (a.st_in->flags & ST_IDLE) return;
    const PcgHead h = pcg_fold_patch(a);
    if (h.flags & (ST_DONE | ST_REFRESH)) return;
    const T* __restrict__ p = h.odd ? a.pbuf0 : a.pbuf1;
    const uint8_t* __restrict__ flags = a.flags;
    const T* __restrict__ dinv = a.dinv;
    T* __restrict__ x = a.x;
    T* __restrict__ r = a.r;
    T* __restrict__ q = a.q;
    using VT = typename Vec16<T>::type;
    constexpr int V = Vec16<T>::N;
    const int64_t n = a.n, nth = (int64_t)gridDim.x * blockDim.x;
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    PcgRow<T, ZF> row;
    row.alpha = (T)h.alpha;
    row.cd = (T)h.cd;
    auto entry = [&](int64_t j, T pj, T qj, T dj, T& xj, T& rj) {
        const uint8_t f = flags[j / DPN];
        const bool dir = (f >> (j % DPN)) & 1;
        if (!dir && (f & kFlagShared)) q[j] = T(0);
        row(dir, pj, qj, dj, xj, rj);
    };
    const int64_t nv = n / V;
    int64_t iv = tid;
    for (; iv + (kUnroll - 1) * nth < nv; iv += kUnroll * nth) {
        VT pv[kUnroll], qv[kUnroll], xv[kUnroll], rv[kUnroll], dv[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const int64_t k = iv + u * nth;
            pv[u] = reinterpret_cast<const VT*>(p)[k];
            qv[u] = reinterpret_cast<const VT*>(q)[k];
            if (!ZF) xv[u] = reinterpret_cast<const VT*>(x)[k];
            rv[u] = reinterpret_cast<const VT*>(r)[k];
            dv[u] = reinterpret_cast<const VT*>(dinv)[k];
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const int64_t k = iv + u * nth;
#pragma unroll
            for (int e = 0; e < V; ++e)
                entry(k * V + e, reinterpret_cast<const T*>(&pv[u])[e], reinterpret_cast<const T*>(&qv[u])[e],
                      reinterpret_cast<const T*>(&dv[u])[e], reinterpret_cast<T*>(&xv[u])[e],
                      reinterpret_cast<T*>(&rv[u])[e]);
            if (!ZF) reinterpret_cast<VT*>(x)[k] = xv[u];
            reinterpret_cast<VT*>(r)[k] = rv[u];
        }
    }
    // the remaining vectors and the last n mod V entries
    for (int64_t k = iv; k < nv; k += nth)
        for (int e = 0; e < V; ++e) {
            const int64_t j = k * V + e;
            T xj = ZF ? T(0) : x[j], rj = r[j];
            entry(j, p[j], q[j], dinv[j], xj, rj);
            if (!ZF) x[j] = xj;
            r[j] = rj;
        }
    for (int64_t j = nv * V + tid; j < n; j += nth) {
        T xj = ZF ? T(0) : x[j], rj = r[j];
        entry(j, p[j], q[j], dinv[j], xj, rj);
        if (!ZF) x[j] = xj;
        r[j] = rj;
    }
    double v[2] = {(double)row.rr, (double)row.rz};
    store_partial<2>(a.part, v);
}

// FP64 mode start: x = 0, r = b, p_old = 0, q = 0; ||b||, r.z.
template <class T>
__global__ void __launch_bounds__(kNodeBS) k_pcg_init(NodeArgs<T> a) {
    const int64_t n = a.n, nth = (int64_t)gridDim.x * blockDim.x;
    double bb = 0.0, rz = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += nth) {
        const double bi = a.b[i];
        a.x[i] = T(0);
        a.r[i] = (T)bi;
        a.q[i] = T(0);
        a.pbuf0[i] = T(0);
        bb += bi * bi;
        rz += bi * (bi * (double)a.dinv[i]);
    }
    double v[2] = {bb, rz};
    store_partial<2>(a.part, v);
    if (last_block(&a.st->ticket)) {
        double t[2];
        grid_total<2>(a.part, gridDim.x, t);
        if (threadIdx.x == 0) {
            PcgState* st = a.st;
            st->ticket = 0;
            st->bnorm = sqrt(t[0]);
            st->res = st->bnorm;
            st->rz = t[1];
            st->beta = 0.0;
            st->it = 0;
            st->pending = 0;
            st->nupd = 0;
            st->s_scale = 1.0;
            st->rmax = 1.0;
            if (st->bnorm < 1e-25) {  // iterative.rs:60-68
                st->flags |= ST_DONE | ST_CONVERGED;
                st->res = 0.0;
            }
            if (st->max_it <= 0) st->flags |= ST_DONE;
        }
    }
}

// MIXED start, pass 1: x64 = 0, xs = 0, q = 0, w64 = 0, p_old = 0; ||b||.
__global__ void __launch_bounds__(kNodeBS) k_mixed_init1(NodeArgs<float> a) {
    const int64_t n = a.n, nth = (int64_t)gridDim.x * blockDim.x;
    double bb = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += nth) {
        const double bi = a.b[i];
        a.x64[i] = 0.0;
        a.w64[i] = 0.0;
        a.x[i] = 0.0f;
        a.q[i] = 0.0f;
        a.pbuf0[i] = 0.0f;
        bb += bi * bi;
    }
    double v[1] = {bb};
    store_partial<1>(a.part, v);
    if (last_block(&a.st->ticket)) {
        double t[1];
        grid_total<1>(a.part, gridDim.x, t);
        if (threadIdx.x == 0) {
            PcgState* st = a.st;
            st->ticket = 0;
            st->bnorm = sqrt(t[0]);
            st->res = st->bnorm;
            st->s_scale = st->bnorm;
            st->beta = 0.0;
            st->it = 0;
            st->pending = 0;
            st->nupd = 0;
            st->rmax = 1.0;
            if (st->bnorm < 1e-25) {
                st->flags |= ST_DONE | ST_CONVERGED;
                st->res = 0.0;
            }
            if (st->max_it <= 0) st->flags |= ST_DONE;
        }
    }
}

// MIXED start, pass 2: r = b / ||b|| (FP32), r.z.
__global__ void __launch_bounds__(kNodeBS) k_mixed_init2(NodeArgs<float> a) {
    if (a.st->flags & ST_DONE) return;
    const int64_t n = a.n, nth = (int64_t)gridDim.x * blockDim.x;
    const double inv = 1.0 / a.st->s_scale;
    double rz = 0.0;
    const bool zf = true;  // the mixed solver keeps z = D^-1 r (see k_patch)
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += nth) {
        const float ri = (float)(a.b[i] * inv);
        const float zi = ri * a.dinv[i];
        a.r[i] = zf ? zi : ri;
        rz += (double)(ri * zi);
    }
    double v[1] = {rz};
    store_partial<1>(a.part, v);
    if (last_block(&a.st->ticket)) {
        double t[1];
        grid_total<1>(a.part, gridDim.x, t);
        if (threadIdx.x == 0) {
            a.st->ticket = 0;
            a.st->rz = t[0];
        }
    }
}

// MIXED refresh 1: x64 += s xs, xs = 0. In the z-form xs still
// lacks the last step alpha p of the iteration that asked for the refresh (the next
// patch kernel would have added it): it is added here, and k_refresh_residual sets
// alpha to 0 so that no later patch kernel adds it again.
__global__ void __launch_bounds__(kNodeBS) k_refresh_flush(NodeArgs<float> a) {
    const double s = a.st->s_scale;
    const bool zf = true;  // z-form (see k_patch)
    const float alpha = zf ? (float)a.st->alpha : 0.0f;
    const float* p = (a.st->it & 1) ? a.pbuf1 : a.pbuf0;  // the last direction
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n; i += (int64_t)gridDim.x * blockDim.x) {
        const float xi = zf ? a.x[i] + alpha * p[i] : a.x[i];
        a.x64[i] += s * (double)xi;
        a.x[i] = 0.0f;
    }
}

// MIXED refresh 3: w = b - K_bc x64 (w holds K x64 on free rows); ||w|| decides
// convergence (FP64 true residual).
__global__ void __launch_bounds__(kNodeBS) k_refresh_residual(NodeArgs<float> a) {
    PcgState* st = a.st;
    const double cd = st->cd;
    double rr = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n; i += (int64_t)gridDim.x * blockDim.x) {
        const bool dir = (a.flags[i / a.dpn] >> (i % a.dpn)) & 1;
        const double kx = dir ? cd * a.x64[i] : a.w64[i];
        const double ri = a.b[i] - kx;
        a.w64[i] = ri;
        rr += ri * ri;
    }
    double v[1] = {rr};
    store_partial<1>(a.part, v);
    if (last_block(&st->ticket)) {
        double t[1];
        grid_total<1>(a.part, gridDim.x, t);
        if (threadIdx.x == 0) {
            st->ticket = 0;
            const double s_new = sqrt(t[0]);
            st->alpha = 0.0;  // the last step is in x64 now (k_refresh_flush)
            st->nupd += 1;
            st->res = s_new;
            st->s_new = s_new;
            if (s_new < st->tol * st->bnorm || s_new < st->abs_tol) {
                st->flags = (st->flags & ~ST_REFRESH) | ST_DONE | ST_CONVERGED;
                cudaGraphSetConditional(a.again, 0u);
            } else {
                st->ratio = st->s_scale / s_new;
            }
        }
    }
}

// MIXED refresh 3, halo mode: as k_refresh_residual, with K x64 on free rows =
// (own-patch sum in w) + (the node's FP64 halo slots, in slot order). Threads
// take nodes; the grid is a multiple of 32 threads, so warps cover aligned
// 32-node chunks and the loop condition is warp-uniform.
__global__ void __launch_bounds__(kNodeBS) k_refresh_residual_halo(NodeArgs<float> a) {
    PcgState* st = a.st;
    const double cd = st->cd;
    const int dpn = a.dpn, lane = threadIdx.x & 31;
    const int64_t nn = a.n / dpn, nth = (int64_t)gridDim.x * blockDim.x;
    double rr = 0.0;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j - lane < nn; j += nth) {
        const bool in = j < nn;
        const uint8_t f = in ? a.flags[j] : (uint8_t)0;
        const int cnt = (f >> kHaloShift) & 15;
        const int pre = halo_prefix(cnt, lane);
        if (!in) continue;
        const int64_t s0 = (int64_t)a.hbase[j >> 5] + pre;
        for (int c = 0; c < dpn; ++c) {
            const int64_t i = j * dpn + c;
            double kx;
            if ((f >> c) & 1) {
                kx = cd * a.x64[i];
            } else {
                kx = a.w64[i];
                for (int k = 0; k < cnt; ++k) kx += a.halo64[(s0 + k) * dpn + c];
            }
            const double ri = a.b[i] - kx;
            a.w64[i] = ri;
            rr += ri * ri;
        }
    }
    double v[1] = {rr};
    store_partial<1>(a.part, v);
    if (last_block(&st->ticket)) {
        double t[1];
        grid_total<1>(a.part, gridDim.x, t);
        if (threadIdx.x == 0) {
            st->ticket = 0;
            const double s_new = sqrt(t[0]);
            st->alpha = 0.0;  // the last step is in x64 now (k_refresh_flush)
            st->nupd += 1;
            st->res = s_new;
            st->s_new = s_new;
            if (s_new < st->tol * st->bnorm || s_new < st->abs_tol) {
                st->flags = (st->flags & ~ST_REFRESH) | ST_DONE | ST_CONVERGED;
                cudaGraphSetConditional(a.again, 0u);
            } else {
                st->ratio = st->s_scale / s_new;
            }
        }
    }
}

// After a FREE or LIFT pass in halo mode: h = y_j + node j's halo slots (slot order) on
// free rows, handed to fin(i, o, dir, h) with the dof's index in the patch numbering and in
// the original one (nperm: new node -> original). Every node is some patch's own, so the
// pass has stored all of y. Node-per-thread with warp-aligned 32-node chunks (grid a
// multiple of 32 threads). fin writes the caller's vector, which saves a pass over y and,
// at 45x37x29 (0.40 M dofs, FP64), the launches and copies around it: operator apply 108 ->
// 85 us.
template <class T, class F>
__global__ void __launch_bounds__(kNodeBS) k_halo_finish(const uint8_t* __restrict__ flags,
                                                         const int32_t* __restrict__ hbase,
                                                         const T* __restrict__ halo,
                                                         const int32_t* __restrict__ nperm, int dpn, int64_t nn,
                                                         const T* __restrict__ y, F fin) {
    const int lane = threadIdx.x & 31;
    const int64_t nth = (int64_t)gridDim.x * blockDim.x;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j - lane < nn; j += nth) {
        const bool in = j < nn;
        const uint8_t f = in ? flags[j] : (uint8_t)0;
        const int cnt = (f >> kHaloShift) & 15;
        const int pre = halo_prefix(cnt, lane);
        if (!in) continue;
        const int64_t s0 = (int64_t)hbase[j >> 5] + pre, o = nperm[j];
        for (int c = 0; c < dpn; ++c) {
            const bool dir = (f >> c) & 1;
            T h = T(0);
            if (!dir) {
                h = y[j * dpn + c];
                for (int k = 0; k < cnt; ++k) h += halo[(s0 + k) * dpn + c];
            }
            fin(j * dpn + c, o * dpn + c, dir, h);
        }
    }
}

// y = K_bc x in the original numbering: Dirichlet rows cd x
template <class T>
struct ApplyOut {
    double cd;
    const T* x;   // patch numbering
    double* out;  // original numbering
    __device__ void operator()(int64_t i, int64_t o, bool dir, T h) const {
        out[o] = (double)(dir ? (T)(cd * (double)x[i]) : h);
    }
};

// f_bc = f - K g on free rows, cd g on Dirichlet rows
struct LiftOut {
    double cd;
    const double* f;  // original numbering
    const double* g;  // patch numbering
    double* out;      // patch numbering
    __device__ void operator()(int64_t i, int64_t o, bool dir, double h) const { out[i] = dir ? g[i] * cd : f[o] - h; }
};

// MIXED refresh 4: r = w / ||w||, current p rescaled, r.z recomputed.
__global__ void __launch_bounds__(kNodeBS) k_refresh_rescale(NodeArgs<float> a) {
    PcgState* st = a.st;
    if (st->flags & ST_DONE) return;
    const double inv = 1.0 / st->s_new;
    const float ratio = (float)st->ratio;
    const bool zf = true;  // z-form: r holds z = D^-1 r
    float* p = (st->it & 1) ? a.pbuf1 : a.pbuf0;  // direction the next apply reads
    double rz = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint8_t fl = a.flags[i / a.dpn];
        const double wi = a.w64[i];
        if (!((fl >> (i % a.dpn)) & 1) && (fl & kFlagShared)) a.w64[i] = 0.0;
        const float ri = (float)(wi * inv);
        const float zi = ri * a.dinv[i];
        a.r[i] = zf ? zi : ri;
        p[i] *= ratio;
        rz += (double)(ri * zi);
    }
    double v[1] = {rz};
    store_partial<1>(a.part, v);
    if (last_block(&st->ticket)) {
        double t[1];
        grid_total<1>(a.part, gridDim.x, t);
        if (threadIdx.x == 0) {
            st->ticket = 0;
            const double ratio2 = st->ratio * st->ratio;
            st->beta = t[0] / (st->rz_old * ratio2);
            st->rz = t[0];
            st->s_scale = st->s_new;
            st->rmax = 1.0;
            st->flags &= ~ST_REFRESH;
            if (st->it >= st->max_it) {
                st->flags |= ST_DONE;
                cudaGraphSetConditional(a.again, 0u);
            }
        }
    }
}

// y_D = cd x_D after a MODE_FREE pass
template <class T>
__global__ void k_dir_rows(const uint8_t* flags, int dpn, int64_t n, double cd, const T* x, T* y) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        if ((flags[i / dpn] >> (i % dpn)) & 1) y[i] = (T)(cd * (double)x[i]);
}

}  // namespace geo
