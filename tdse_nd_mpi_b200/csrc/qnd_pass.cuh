// qnd_pass.cuh — the fused axis pass: every line of the N-D state along one axis
// is read once from HBM, transformed in registers/shared memory, combined with its
// phase tables and written once. All hot-path work is a sequence of these passes.
//
// State layout: row-major, axis 0 slowest (meshgrid.c:205-211). For the pass axis
// with length L and stride S (the product of the later axes' lengths) the lines are
// lam = o*S + s, element m of line lam sits at flat = o*L*S + m*S + s. A CTA owns G
// lines: for the contiguous axis (S = 1) G whole rows; for a strided axis G
// neighbouring s values, so every global access is a run of G consecutive values.
//
// Modes
//   PM_SANDWICH  psi <- epi(x) . IFFT[ spec(k) . FFT[ pro(x) . psi ] ]   (+ reductions)
//                The split-operator kernel/potential sub-steps: one read, one write.
//   PM_DOUBLE    psi <- epi . IFFT spec2 FFT [ mid(x) . IFFT spec FFT [ pro . psi ] ]: two kinetic
//                sandwiches along the same axis with the r-space factor between them, still one
//                read and one write (consecutive sandwiches alternate their axis order so that
//                the last axis of one is the first axis of the next).
//
// Full-grid tables (pro/mid/epi factors, WK_GRID weights) are stored LINE-MAJOR for the pass
// axis: entry lam*L + m for element m of line lam. Reads are then coalesced on every axis; for
// the contiguous axis this is the natural layout.
//   PM_FFT_FWD / PM_FFT_INV   psi <- scale . (I)FFT[psi]   (representation changes)
//   PM_SPECRED   reductions of |FFT psi|^2 weighted by k-space tables; no write
//   PM_APPLY     u = IFFT[spec . FFT psi] (+ V psi) (+ dst); optional store into dst and
//                reductions of |u|^2 or Re(conj(partner) u)   (energy moments, Lz)
//   PM_ROUNDTRIP psi <- FFT[ mid(x) . scale . IFFT[psi] ] (+ reductions before the FFT): the closing
//                inverse transform of one sandwich and the opening transform of the next on the
//                strided virtual axis of a long 1-D axis, with the r-space factors between. Every table,
//                those of the axis itself among them, is in the line-major order of this axis.
//
// Reductions are FP64 and deterministic: per-CTA partial sums, then the last CTA
// to finish (ticket counter) adds the partials in a fixed order.
#pragma once

#include <cuda.h>  // CUtensorMap (the type only; maps are encoded on the host)

#include "qnd_fft.cuh"

#include <type_traits>

namespace qnd {

constexpr int MAX_RED = 8;
constexpr int MAX_DIM = 6;  // grid dimensions (the reference reads DIMENSION from its parameters)

enum : int {
    PM_SANDWICH = 0,
    PM_FFT_FWD = 1,
    PM_FFT_INV = 2,
    PM_SPECRED = 3,
    PM_APPLY = 4,
    PM_DOUBLE = 5,        // runs the kernels of PM_SANDWICH with four turns
    PM_ROUNDTRIP = 6,
    PM_SANDWICH_RED = 7,  // with fused reductions: separate instantiations, so that the passes without them
    PM_ROUNDTRIP_RED = 8, // (most of a chain) keep their registers for the transform
    PM_SANDWICH_P = 9,    // the passes at a chain's ends in the momentum representation (PassArgs from_p, to_p):
                          // with their tests in the kernels of every pass those ran 2% slower
    PM_NMODES = 10
};
// The transform structure of a kernel's mode (the reducing variants share their base mode's), whether the
// mode can carry reductions at all, and the kernel mode of a pass.
__host__ __device__ constexpr int pass_base_mode(int m) {
    return m == PM_SANDWICH_RED || m == PM_SANDWICH_P ? PM_SANDWICH : (m == PM_ROUNDTRIP_RED ? PM_ROUNDTRIP : m);
}
__host__ __device__ constexpr bool pass_mode_reduces(int m) {
    return m == PM_SANDWICH_RED || m == PM_ROUNDTRIP_RED || m == PM_SPECRED || m == PM_APPLY;
}
__host__ __device__ constexpr int pass_kernel_mode(int m, bool reduces, bool ends_in_p = false) {
    return ends_in_p ? PM_SANDWICH_P
           : (m == PM_SANDWICH || m == PM_DOUBLE) ? (reduces ? PM_SANDWICH_RED : PM_SANDWICH)
           : m == PM_ROUNDTRIP ? (reduces ? PM_ROUNDTRIP_RED : PM_ROUNDTRIP) : m;
}
// |v|^2 w, Re(conj(partner) v) w, or (element-wise grid reductions only) the count of elements with a
// non-finite part
enum : int { RK_ABS2 = 0, RK_BILIN = 1, RK_NONFINITE = 2 };
enum : int { WK_ONE = 0, WK_AXIS = 1, WK_GRID = 2 }; // weight 1, table[idx_axis], line-major table

struct RedDesc {
    int n;                       // accumulators in use (0: no reduction)
    int accumulate;              // out[k] += result instead of out[k] = result
    int kind[MAX_RED];
    int wkind[MAX_RED];
    int waxis[MAX_RED];
    // WK_AXIS: the weight axis' log2 stride and index mask (set by the host from waxis, so that the
    // pass kernels index no parameter array by a run-time value)
    int wshift[MAX_RED];
    long long wmask[MAX_RED];
    const double* wtab[MAX_RED];
    double scale[MAX_RED];
    double* partials;            // [gridDim.x][MAX_RED] scratch
    unsigned int* counter;       // must be 0 at launch; the last CTA resets it
    double* out;                 // final values
};

template <typename R> struct PassArgs {
    using V = cplx_t<R>;
    V* psi;
    const V* src;                // contiguous axes: where the state is read (psi, or another state that stays)
    V* dst;
    const V* partner;
    const V* tw;
    int axis;                    // the pass axis (its index along a line is m)
    int log2S;
    long long nlines;
    int dim;
    int shift[MAX_DIM];
    long long nmask[MAX_DIM];
    const R* pro_real;
    const V* pro_cplx;
    const double* pro_scale_dev;
    const V* spec;
    int spec_full;               // spec is a full-grid table in line-major order (one row per line),
                                 // not one row shared by every line (the long-axis four-step pass)
    const V* spec2;              // PM_DOUBLE: the second sandwich's spectral factors
    const R* mid_real;           // PM_DOUBLE: r-space factors between the two sandwiches
    const V* mid_cplx;
    const V* mid2_cplx;          // reducing passes: a second full-grid factor there, after the reductions
    const V* mid_ax_cplx[MAX_DIM];
    const R* mid_ax_real[MAX_DIM];  // PM_DOUBLE: per-axis real factors between the sandwiches (step mask)
    int red_at_mid;                 // PM_DOUBLE: reduce the state between the sandwiches, not at the end
    int sandwiches;                 // of a propagating pass: 1 or 2
    // a pass at the end of a chain in the momentum representation: the first sandwich without its forward
    // transform, the last one without its inverse; each takes the place of two transforms and a scaling
    int from_p, to_p;
    R p_scale;                      // with either: sqrt(L) (the tables hold 1/L, the representation 1/sqrt(L))
    int points;                     // bits of the places with factors: 1 before, 2 between the sandwiches, 4 after
    const R* epi_real;
    const V* epi_cplx;
    const V* ax_cplx[MAX_DIM];   // per-axis factors (laser phases, step mask) applied ...
    const R* ax_real[MAX_DIM];
    int ax_in_prologue;          // complex factors before the forward transform (1) or after the inverse
                                 // (0); real factors (the step mask) always after the inverse
    R scale;
    int apply_acc;
    unsigned seed;               // FP32: the random stream of the stochastic rounding (one per launch)
    const double* apply_vtab;
    RedDesc red;
    // strided passes: the state as a 3-D tensor {contiguous sub-index, pass axis, outer} for TMA box
    // loads of a CTA's G lines, read by the SK = 2 instantiations (use_tma records the host's choice);
    // err: set when a wait for those loads runs out
    int use_tma;
    int* err;
    int tma_wait_tries;          // tries of the bounded wait for those loads before the CTA gives up
    int red_lm;                  // grid reductions: full-grid weights in the line-major order of `axis`
    CUtensorMap tmap;
};

// Threads-per-line, values-per-thread and lines-per-CTA for a line length.
//   E = 16 values per thread in registers (L itself up to 16 points; 32 values per thread, one
//   warp per 1024-point line, measured slower: WIDE). T = L/E threads per line; a CTA of NT = T*G
//   threads owns G lines. Lines along a strided axis are staged through shared memory, by
//   per-thread cp.async copies or by TMA boxes (the kernel's SK), so that the global accesses run
//   over G neighbouring lines; the stage buffer is then the exchange space.
//
// Shape variants VAR (the tile-shape autotuner picks one per geometry by timing, shape_choice in
// qnd_engine.cu): 0 the default, 1 half the lines per CTA (smaller CTAs, more of them per SM),
// 2 twice the lines per CTA (256-thread CTAs), 3 seven lines per CTA at L = 1024 (448 threads, one
// CTA per SM: a 1024-line pass then runs as 147 CTAs, 7 lines on every SM, where 2-line CTAs leave
// some SMs 8 lines and others 6). Variants exist for the two-sandwich and sandwich passes of lines
// of 256 to 2048 points; VALID says whether a variant differs from the default.
constexpr int NSHAPES = 4;
template <typename R, int L, int VAR = 0> struct PassShape {
    // FP64, L >= 1024: 32 values per thread (two radix-32 stages at L = 1024), one CTA per line, a
    // single warp per line at L = 1024 (warp-synchronous exchanges). Otherwise 16 values per thread
    // and 128-thread CTAs holding several lines.
    static constexpr bool WIDE = false;  // 32 values per thread for long FP64 lines: measured slower (too few warps per SM)
    static constexpr int E = L <= 16 ? L : (WIDE ? 32 : 16);
    static constexpr int T = L / E;
    static constexpr int G0 = WIDE ? 1 : (T >= 128 ? 1 : 128 / T);
    static constexpr int G = VAR == 1 ? (G0 > 1 ? G0 / 2 : 1) : (VAR == 2 ? 2 * G0 : (VAR == 3 ? 7 : G0));
    static constexpr bool VALID =
        VAR == 0 || (VAR == 3 ? (L == 1024 && T == 64)
                              : (L >= 256 && L <= 2048 && (VAR == 1 ? G0 > 1 : (T > 32 ? G <= 15 : true))));
    static constexpr int NT = T * G;
    static constexpr bool EXCHANGE = FFTPlan<L, E>::NSTAGE > 1;
    static constexpr int SLOTS = sizeof(R) == 8 ? 8 : 16;  // element slots per bank cycle (16 B / 8 B values)
    // Line stride. Lines of T >= SLOTS threads: the G lines touched in one bank cycle of the staging copy
    // land on distinct slots. Shorter lines share a bank cycle, SLOTS / T of them, in the exchanges too:
    // a stride of T (mod SLOTS) puts those on distinct slots, and line_off's shift by one slot per such
    // group keeps the copy's SLOTS neighbouring lines distinct. With an odd stride the exchanges of 32- and
    // 64-point FP64 lines (and 128-point FP32 lines) took two bank cycles each (64 x 256 x 128 velocity
    // gauge: 2.57 -> 2.47 ms).
    static constexpr int LS_TARGET = T < SLOTS ? T : (G >= SLOTS ? 1 : SLOTS / G);
    static constexpr int LINE_RAW = FFTPlan<L, E>::SMEM_LINE + (T < SLOTS ? T - 1 : 0);
    static constexpr int LS = LINE_RAW + ((LS_TARGET - LINE_RAW % SLOTS) % SLOTS + SLOTS) % SLOTS;
    __host__ __device__ static constexpr int line_off(int w) {
        return w * LS + (T < SLOTS ? w / (SLOTS / T) % T : 0);
    }
    // What LS and line_off are chosen for, checked where a shape is built (qnd_pass_inst.cu): no line reaches
    // into the next one or past the buffer, and ...
    static constexpr bool lines_apart() {
        for (int w = 0; w < G; ++w)
            if (line_off(w) + FFTPlan<L, E>::SMEM_LINE > (w + 1 < G ? line_off(w + 1) : G * LS)) return false;
        return true;
    }
    // ... for lines of fewer threads than a bank cycle has slots, the accesses of one bank cycle fall on
    // distinct slots: an exchange's store of register r by the threads of SLOTS / T lines, and the staging
    // copy's SLOTS neighbouring lines.
    static constexpr bool slots_distinct() {
        if (T >= SLOTS || G < SLOTS) return true;
        constexpr int Q = T < SLOTS ? SLOTS / T : 1;
        for (int w0 = 0; w0 + Q <= G; w0 += Q)
            for (int r = 0; r < E; ++r) {
                unsigned hit = 0;
                for (int w = w0; w < w0 + Q; ++w)
                    for (int t = 0; t < T; ++t) hit |= 1u << (line_off(w) + (E * t + r) + (E * t + r) / E) % SLOTS;
                if (hit != (1u << SLOTS) - 1) return false;
            }
        for (int w0 = 0; w0 + SLOTS <= G; w0 += SLOTS) {
            unsigned hit = 0;
            for (int w = w0; w < w0 + SLOTS; ++w) hit |= 1u << line_off(w) % SLOTS;
            if (hit != (1u << SLOTS) - 1) return false;
        }
        return true;
    }
    // stage twiddle entries: FP64 plans keep one base per butterfly position (TwiddledDFT)
    static constexpr int TW_ENTRIES = sizeof(R) == 8 ? FFTPlan<L, E>::twb_size() : FFTPlan<L, E>::tw_size();
    static constexpr int TWN_RAW = (TW_ENTRIES + 1) & ~1;
    // stage twiddles in shared memory when they are small and shared by several lines of the CTA;
    // otherwise read them through L1 (one copy per SM instead of one per CTA)
    static constexpr bool TW_SMEM = G > 1 && size_t(TWN_RAW) * sizeof(cplx_t<R>) <= 16 * 1024;
    // the line buffers start on a 128-byte boundary (TMA box destinations)
    static constexpr int TWN = TW_SMEM ? ((TWN_RAW * int(sizeof(cplx_t<R>)) + 127) / 128 * 128) / int(sizeof(cplx_t<R>)) : 0;
    // the 7-line shape (one CTA per SM, shared memory to spare) keeps the spectral rows of both
    // sandwiches in shared memory: read by 7 lines each, once per CTA from L2
    static constexpr bool SPEC_SMEM = VAR == 3;
    static constexpr int SPECN = SPEC_SMEM ? 2 * L : 0;
    static constexpr size_t SMEM = sizeof(cplx_t<R>) * (size_t(TWN) + size_t(G) * LS + size_t(SPECN));
    // 128-thread CTAs: <= 128 registers (4 CTAs per SM) when shared memory allows; one-line CTAs
    // of L >= 1024 keep their registers (the SM holds as many lines as its register file allows)
    static constexpr int MINB_DEFAULT =
        WIDE ? 1 : (SMEM <= 54 * 1024 ? 4 : (SMEM <= 72 * 1024 ? 3 : (SMEM <= 110 * 1024 ? 2 : 1)));
    // variants: as many CTAs as 128 registers a thread and the shared memory allow
    static constexpr int MINB_REGS = 65536 / (NT * 128) > 0 ? 65536 / (NT * 128) : 1;
    static constexpr int MINB_SMEM = int((227 * 1024) / (SMEM > 0 ? SMEM : 1)) > 0 ? int((227 * 1024) / (SMEM > 0 ? SMEM : 1)) : 1;
    static constexpr int MINB = VAR == 0 ? MINB_DEFAULT : (MINB_REGS < MINB_SMEM ? MINB_REGS : MINB_SMEM);
};

// Barrier over the threads of one line: a named barrier when a line spans whole warps,
// a warp barrier when several lines share a warp.
template <int T> struct LineSync {
    int id;
    __device__ __forceinline__ void operator()() const {
        if constexpr (T > 32) {
            asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(T) : "memory");
        } else {
            __syncwarp();
        }
    }
};

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
    return x;
}

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename V> __device__ __forceinline__ void cp_async_elem(V* smem_dst, const V* gsrc) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
    if constexpr (sizeof(V) == 16) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gsrc) : "memory");
    } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(gsrc) : "memory");
    }
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// ---- TMA box loads completing on an mbarrier (strided passes)
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t phase) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(phase)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, const void* src, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(smem_u32(src)), "r"(x), "r"(y), "r"(z)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// shared memory of the committed bulk stores read (the CTA may then leave; the writes complete
// before the grid does)
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// generic-proxy writes to shared memory visible to the bulk-copy (async) proxy
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Waits for phase `phase` of the barrier at most `limit` tries; false when they run out.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t phase, int limit) {
    for (int i = 0; i < limit; ++i)
        if (mbar_try_wait(bar, phase)) return true;
    return false;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A fused reduction's accumulators in shared memory, where they are indexed at run time: the loop over
// them is rolled. With a copy of the sums for each of the MAX_RED accumulators and each weight kind, a
// reducing 1024-point pass held up to 190 KB (FP64) and 237 KB (FP32) of code (64 and 81 KB now), and a
// launch finds the instruction caches cold.
struct RedRow {
    const double* w;  // weights: none (null), one for the line at w[(base >> shift) & mask], or a row
    long long mask;
    int shift;
    int how;          // 0 none, 1 one for the line, 2 a row over the pass axis, 3 a row of a line-major table
    int bilinear;
};
template <int NT> struct RedShared {
    static constexpr int NW = NT / 32 > 0 ? NT / 32 : 1;
    RedRow row[MAX_RED];
    double s[NW][MAX_RED];
    int is_last;
};

// The descriptor's accumulators for a pass along `axis` into shared memory, by the first threads
// (compile-time indices into the argument); visible after a CTA barrier.
template <int NT> __device__ __forceinline__ void load_red_rows(const RedDesc& rd, int axis, RedShared<NT>& sh) {
#pragma unroll
    for (int k = 0; k < MAX_RED; ++k)
        if (int(threadIdx.x) == k && k < rd.n) {
            const int wk = rd.wkind[k];
            sh.row[k] = RedRow{rd.wtab[k], rd.wmask[k], rd.wshift[k],
                               wk == WK_GRID ? 3 : (wk == WK_AXIS ? (rd.waxis[k] == axis ? 2 : 1) : 0),
                               rd.kind[k] == RK_BILIN};
        }
}

// One accumulator's sum over the E values a thread holds of one line (m = tid + u*T).
template <typename R, int E, int T>
__device__ __forceinline__ double line_sum(const RedRow& r, const cplx_t<R>* v, const cplx_t<R>* partner,
                                           long long base, int log2S, long long lbase, int tid) {
    const double* __restrict__ row = r.how == 2 ? r.w + tid : (r.how == 3 ? r.w + lbase + tid : nullptr);
    double sum = 0.0;
    if (!r.bilinear) {
        if (row) {
#pragma unroll
            for (int u = 0; u < E; ++u) {
                const double x = v[u].x, y = v[u].y;
                sum = fma(fma(x, x, y * y), __ldg(row + u * T), sum);
            }
        } else {
#pragma unroll
            for (int u = 0; u < E; ++u) {
                const double x = v[u].x, y = v[u].y;
                sum += fma(x, x, y * y);
            }
        }
    } else {
        const int step = row ? T : 0;
        const double one = 1.0;
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const cplx_t<R> p = partner[base + ((long long)(tid + u * T) << log2S)];
            sum += (double(p.x) * double(v[u].x) + double(p.y) * double(v[u].y)) * (row ? __ldg(row + u * step) : one);
        }
    }
    return r.how == 1 ? sum * __ldg(r.w + ((base >> r.shift) & r.mask)) : sum;
}

// Warm L2 with the line-major rows a pass will read later (a full-grid table), one 128-byte
// line per request.
template <int L, int T, typename X> __device__ __forceinline__ void prefetch_row_l2(const X* row, int tid) {
    constexpr int BYTES = L * int(sizeof(X));
    constexpr int NLINES = (BYTES + 127) / 128;
    const char* p = reinterpret_cast<const char*>(row);
#pragma unroll
    for (int q = tid; q < NLINES; q += T) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + 128 * q));
}

// Every warp's sums sh.s[warp][0..n) into partials, then the last CTA sums the partials in order.
// blk / nblk: this CTA's group and the number of groups (the grid, or a persistent kernel's groups
// of one pass).
template <int NT>
__device__ __forceinline__ void finish_red(const RedDesc& rd, RedShared<NT>& sh, unsigned blk, unsigned nblk) {
    constexpr int NW = RedShared<NT>::NW;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    __syncthreads();
    if (t < rd.n) {
        double s = 0.0;
        for (int w = 0; w < NW; ++w) s += sh.s[w][t];
        rd.partials[(long long)blk * MAX_RED + t] = s;
    }
    __threadfence();
    __syncthreads();
    if (t == 0) sh.is_last = (atomicAdd(rd.counter, 1u) == nblk - 1);
    __syncthreads();
    if (!sh.is_last) return;
    __threadfence();
    // every accumulator in one sweep over the partials (one round of L2 loads, one barrier): the
    // last CTA's tail is the critical path of the pass. Per accumulator the order of the sums is
    // the same as one accumulator at a time (thread-strided partials, warp sum, warps in order).
    double s[MAX_RED];
#pragma unroll
    for (int k = 0; k < MAX_RED; ++k) s[k] = 0.0;
    for (unsigned b = t; b < nblk; b += NT) {
        const double* pb = rd.partials + (long long)b * MAX_RED;
#pragma unroll
        for (int k = 0; k < MAX_RED; ++k)
            if (k < rd.n) s[k] += __ldcg(pb + k);
    }
#pragma unroll
    for (int k = 0; k < MAX_RED; ++k) {
        if (k >= rd.n) break;
        const double ws = warp_sum(s[k]);
        if (lane == 0) sh.s[wid][k] = ws;
    }
    __syncthreads();
    if (t < rd.n) {
        double tot = 0.0;
        for (int w = 0; w < NW; ++w) tot += sh.s[w][t];
        tot *= rd.scale[t];
        rd.out[t] = rd.accumulate ? rd.out[t] + tot : tot;
    }
    if (t == 0) *rd.counter = 0u;
}
// The same from each thread's accumulators acc[0..n).
template <int NT> __device__ __forceinline__ void finish_red(const RedDesc& rd, double* acc) {
    __shared__ RedShared<NT> sh;
#pragma unroll
    for (int k = 0; k < MAX_RED; ++k) {
        if (k >= rd.n) break;
        const double s = warp_sum(acc[k]);
        if ((threadIdx.x & 31) == 0) sh.s[threadIdx.x >> 5][k] = s;
    }
    finish_red<NT>(rd, sh, blockIdx.x, gridDim.x);
}

// The fused reductions of a pass: every line's values, the CTA's sums, the grid's.
template <typename R, int E, int T, int NT>
__device__ __forceinline__ void reduce_lines(const RedDesc& rd, RedShared<NT>& sh, const cplx_t<R>* v, bool active,
                                             const cplx_t<R>* partner, long long base, int log2S, long long lbase,
                                             int tid, int axis, unsigned blk, unsigned nblk) {
    load_red_rows<NT>(rd, axis, sh);
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < rd.n; ++k) {
        double s = 0.0;
        if (active) s = line_sum<R, E, T>(sh.row[k], v, partner, base, log2S, lbase, tid);
        s = warp_sum(s);
        if ((threadIdx.x & 31) == 0) sh.s[threadIdx.x >> 5][k] = s;
    }
    finish_red<NT>(rd, sh, blk, nblk);
}

// Point-wise r-space factors on the E values a thread holds of one line: full-grid tables tr (real) and
// tc (complex; line-major: entry lbase + m), the factors pc and pr along the pass axis (entry m), and for
// the whole line lf (the composed complex factors of the other axes) and lr (their real factors and a
// scalar). ROWS: pc and pr are rows of full tables in line-major order (entry lbase + m) too (the strided
// virtual axis of a long 1-D axis).
template <typename R, int E, int T, bool ROWS = false>
__device__ __forceinline__ void apply_tables(cplx_t<R>* v, int tid, long long lbase, const R* __restrict__ tr,
                                             const cplx_t<R>* __restrict__ tc, const cplx_t<R>* __restrict__ pc,
                                             const R* __restrict__ pr, bool use_lf, cplx_t<R> lf, bool use_lr, R lr,
                                             uint32_t key) {
    // One loop over the thread's elements per factor that is set, so that each loop is free of
    // branches and its table reads go out together: with the tests inside one loop over the elements
    // every read waited for the one before it, and the factor between the sandwiches of a 1024-point
    // two-sandwich pass took 16,500 of the pass's 55,000 cycles (FP64; 8,000 to 9,600 of 37,000 in
    // FP32). The order of an element's products is the same.
    auto grid_at = [&](int u) { return lbase + tid + u * T; };                            // full-grid tables
    auto axis_at = [&](int u) { return ROWS ? grid_at(u) : (long long)(tid + u * T); };  // pass-axis tables
    if (tr) {
#pragma unroll
        for (int u = 0; u < E; ++u) v[u] = cscale(v[u], __ldg(tr + grid_at(u)));
    }
    if (tc) {
#pragma unroll
        for (int u = 0; u < E; ++u) v[u] = fmul(v[u], __ldg(tc + grid_at(u)));
    }
    if (pc) {
#pragma unroll
        for (int u = 0; u < E; ++u) {
            // FP32: the per-axis laser phases near the origin, where the state lives, are rotations by
            // angles ~1e-4 and take the dithered product (fmul_dither): along the pass axis the elements
            // around the axis centre (a compile-time choice after unrolling), and the whole line when
            // the factor of the other axes is a small rotation (a line-uniform branch). The potential
            // tables rotate by h V, far from small where the state is.
            if (sizeof(R) == 4 && (u == E / 2 - 1 || u == E / 2)) {
                if constexpr (sizeof(R) == 4)
                    v[u] = fmul_dither(v[u], __ldg(pc + axis_at(u)), mix32(key + uint32_t(tid + u * T)));
            } else {
                v[u] = fmul(v[u], __ldg(pc + axis_at(u)));
            }
        }
    }
    if (pr) {
#pragma unroll
        for (int u = 0; u < E; ++u) v[u] = cscale(v[u], __ldg(pr + axis_at(u)));
    }
    if (use_lf) {
        bool dithered = false;
        if constexpr (sizeof(R) == 4) {
            if (lf.y != 0.0f && fabsf(lf.y) < 2e-3f) {
                dithered = true;
#pragma unroll
                for (int u = 0; u < E; ++u)
                    v[u] = fmul_dither(v[u], lf, mix32((key ^ 0x85ebca6bu) + uint32_t(tid + u * T)));
            }
        }
        if (!dithered) {
#pragma unroll
            for (int u = 0; u < E; ++u) v[u] = fmul(v[u], lf);
        }
    }
    if (use_lr) {
#pragma unroll
        for (int u = 0; u < E; ++u) v[u] = cscale(v[u], lr);
    }
}

// One CTA's share of a pass: line group g of ngroups (the CTA's G lines), with the dynamic shared
// memory smem_raw. `wait` runs after the prologue (twiddles to shared memory, read-only tables to
// L2), before the state is touched: the wait for the previous pass (programmatic dependent launch
// in qnd_pass_kernel, the pass's dependency counter in the persistent sweep kernel).
// SK: 0 a contiguous axis, 1 a strided axis staged by per-thread cp.async copies, 2 a strided axis
// staged by TMA boxes (separate instantiations: each staging gets its own register allocation).
template <typename R, int L, int SK, int KMODE, int VAR = 0, typename Wait>
__device__ __forceinline__ void pass_group(const PassArgs<R>& a, long long g, unsigned ngroups,
                                           unsigned char* smem_raw, Wait wait) {
    constexpr bool STRIDED = SK != 0;
    constexpr bool TMA = SK == 2;
    constexpr int MODE = pass_base_mode(KMODE);
    constexpr bool HAS_RED = pass_mode_reduces(KMODE);
    constexpr bool PROPAGATE = MODE == PM_SANDWICH, ENDS = KMODE == PM_SANDWICH_P;
    constexpr bool ONE_TRANSFORM = sizeof(R) == 8 && L >= 1024;  // see the sandwich below
    using V = cplx_t<R>;
    using SH = PassShape<R, L, VAR>;
    constexpr int E = SH::E, T = SH::T, G = SH::G, NT = SH::NT, LS = SH::LS;
    constexpr bool TWS = SH::TW_SMEM;
    V* tw_s = reinterpret_cast<V*>(smem_raw);   // [TWN] stage twiddles (when they fit)
    V* lines = tw_s + SH::TWN;                   // [G][LS]
    V* spec_s = lines + G * LS;                  // [2][L] spectral rows (SPEC_SMEM)

    const int t = threadIdx.x;
    const int w = t / T;  // line within the CTA (the threads of a line are consecutive)
    const int tid = t % T;
    const LineSync<T> lsync{1 + w};
    V* line = lines + SH::line_off(w);

    const long long nlines = a.nlines;
    const int log2S = a.log2S;
    const long long smask = (1ll << log2S) - 1;
    auto line_base = [&](long long lam) { return (((lam >> log2S) * L) << log2S) + (lam & smask); };
    const long long lam = g * G + w;
    const bool active = lam < nlines;
    const long long base = line_base(active ? lam : 0);
    const long long lbase = (active ? lam : 0) * L;  // line-major table offset of this line
    // stochastic-rounding stream of this line: two spectral multiplies of L elements per line
    const uint32_t key0 = mix32(a.seed) + uint32_t(lbase) * 2u;

    const V* tw = a.tw;
    if constexpr (TWS) {
        for (int i = t; i < SH::TW_ENTRIES; i += NT) tw_s[i] = a.tw[i];
        tw = tw_s;
    }
    // spectral rows to shared memory (read-only tables: before the wait for the previous pass);
    // visible after the CTA barrier that precedes the first transform
    const bool spec_row = a.spec && !a.spec_full;
    if constexpr (SH::SPEC_SMEM && PROPAGATE) {
        if (spec_row)
            for (int i = t; i < L; i += NT) spec_s[i] = __ldg(a.spec + i);
        if (a.spec2)
            for (int i = t; i < L; i += NT) spec_s[L + i] = __ldg(a.spec2 + i);
    }

    if constexpr (PROPAGATE || MODE == PM_ROUNDTRIP) {
        // the read-only tables: start their journey to L2 now, before the wait for the previous
        // pass (which writes only the state), so that it overlaps that pass's tail
        if (active) {
            if (a.pro_cplx) prefetch_row_l2<L, T>(a.pro_cplx + lbase, tid);
            if (a.mid_cplx) prefetch_row_l2<L, T>(a.mid_cplx + lbase, tid);
            if (a.mid_real) prefetch_row_l2<L, T>(a.mid_real + lbase, tid);
            if (a.epi_cplx) prefetch_row_l2<L, T>(a.epi_cplx + lbase, tid);
            if (a.epi_real) prefetch_row_l2<L, T>(a.epi_real + lbase, tid);
            if constexpr (HAS_RED) {
#pragma unroll
                for (int k = 0; k < MAX_RED; ++k)
                    if (k < a.red.n && a.red.wkind[k] == WK_GRID) prefetch_row_l2<L, T>(a.red.wtab[k] + lbase, tid);
                if (a.mid2_cplx) prefetch_row_l2<L, T>(a.mid2_cplx + lbase, tid);
            }
        }
    }

    wait();

    using RS = std::conditional_t<HAS_RED, RedShared<NT>, char>;
    __shared__ RS red_sh;
    (void)red_sh;

    V v[E];
    if constexpr (STRIDED) {
        if constexpr (TMA) {
            // the CTA's G lines as L/BOXL boxes {G lines, BOXL rows} in [row][line] order, loaded by TMA
            // (the host enables this only when every group lies inside one slab of lines and the boxes
            // meet the 16-byte rules; a partial last group reads the fill value past the last line)
            __shared__ __align__(8) uint64_t tma_bar;
            __shared__ int tma_gave_up;
            constexpr int BOXL = L < 256 ? L : 256;
            const long long lam0 = g * G;
            if (t == 0) {
                mbar_init(&tma_bar, 1);
                mbar_init_fence();
                tma_gave_up = 0;
            }
            __syncthreads();
            if (t == 0) {
                mbar_expect_tx(&tma_bar, uint32_t(G * L * sizeof(V)));
                const int x = int(lam0 & smask) * int(sizeof(V) / sizeof(uint64_t));
                const int z = int(lam0 >> log2S);
#pragma unroll 1
                for (int c = 0; c < L / BOXL; ++c) tma_load_3d(lines + c * BOXL * G, &a.tmap, x, c * BOXL, z, &tma_bar);
            }
            if (!mbar_wait_bounded(&tma_bar, 0, a.tma_wait_tries)) tma_gave_up = 1;
            __syncthreads();
            if (tma_gave_up) {
                // The CTA's lines did not arrive in time (one decision for the whole CTA). Give the
                // copies in flight a second bounded wait so that none lands after the CTA has left,
                // raise the error flag, and leave the state untouched: no transform, no store. The CTA
                // still takes its ticket in the grid reduction (with nothing), so that the last CTA
                // finishes it and resets the counter.
                mbar_wait_bounded(&tma_bar, 0, 1 << 20);
                if (t == 0 && a.err) atomicExch(a.err, 1);
                if constexpr (HAS_RED)
                    if (MODE == PM_SPECRED || a.red.n) {
                        for (int k = t; k < RedShared<NT>::NW * MAX_RED; k += NT) red_sh.s[k / MAX_RED][k % MAX_RED] = 0.0;
                        finish_red<NT>(a.red, red_sh, unsigned(g), ngroups);
                    }
                return;
            }
#pragma unroll
            for (int u = 0; u < E; ++u) v[u] = lines[(tid + u * T) * G + w];
            __syncthreads();  // every line has read its inputs before the exchanges reuse the buffer
        } else {
            // stage the CTA's G neighbouring lines: consecutive threads -> consecutive addresses
#pragma unroll 4
            for (int e = t; e < G * L; e += NT) {
                const int wl = e % G, m = e / G;
                const long long l2 = g * G + wl;
                if (l2 < nlines)
                    cp_async_elem(lines + SH::line_off(wl) + spad<E>(m), a.psi + line_base(l2) + ((long long)m << log2S));
            }
            cp_async_commit();
            cp_async_wait<0>();
            __syncthreads();
#pragma unroll
            for (int u = 0; u < E; ++u) v[u] = active ? line[spad<E>(tid + u * T)] : V{R(0), R(0)};
        }
    } else {
        const V* __restrict__ src = a.src;
#pragma unroll
        for (int u = 0; u < E; ++u) v[u] = active ? src[base + tid + u * T] : V{R(0), R(0)};
        if constexpr (TWS) __syncthreads();  // twiddles visible
    }

    if constexpr (STRIDED && !TMA) lsync();  // staged inputs read before the exchanges reuse the buffer

    auto reduce = [&] {
        if constexpr (HAS_RED)
            reduce_lines<R, E, T, NT>(a.red, red_sh, v, active, a.partner, base, log2S, lbase, tid, a.axis, unsigned(g),
                                      ngroups);
    };
    auto conjugate = [&] {
#pragma unroll
        for (int u = 0; u < E; ++u) v[u].y = -v[u].y;
    };
    auto spectral = [&](const V* row, uint32_t key) {
#pragma unroll
        for (int u = 0; u < E; ++u)
            v[u] = fmul_spec<L>(v[u], row[tid + u * T], key + uint32_t(tid + u * T), u == 0 || u == E - 1);
    };
    auto spectral_ldg = [&](const V* __restrict__ row, uint32_t key) {
#pragma unroll
        for (int u = 0; u < E; ++u)
            v[u] = fmul_spec<L>(v[u], __ldg(row + tid + u * T), key + uint32_t(tid + u * T), u == 0 || u == E - 1);
    };
    auto second_mid = [&] {
        if (active && a.mid2_cplx) {
#pragma unroll
            for (int u = 0; u < E; ++u) v[u] = fmul(v[u], __ldg(a.mid2_cplx + lbase + tid + u * T));
        }
    };
    // v <- IFFT[ between . FFT v ]. ONE_TRANSFORM: one copy of the transform, the inverse as the forward
    // transform of the conjugate, conjugated: less code to fetch against two sign flips per point.
    // Measured with one copy / with two, FP64: 2048^2 6.73 / 7.09 ms, 1024^2 7.48 / 7.51, 3-D grids of 64
    // to 256 points 2.74 / 2.66. FP32 passes keep both directions: 2048^2 13.2 / 12.5 ms, and the low parts
    // of their split constants round differently in the conjugate (the sweep of 256^2 to 1024^2 members
    // would gain 3%).
    // fwd / inv: whether the transforms run (PassArgs from_p, to_p).
    auto sandwich = [&](bool fwd, bool inv, auto between) {
        if constexpr (ONE_TRANSFORM) {
#pragma unroll 1
            for (int turn = 0; turn < 2; ++turn) {
                if (turn || fwd) fft_line_stages<L, E, -1, 0, TWS>(v, tid, line, tw, lsync);
                if (turn == 0) between();
                if (!inv) break;
                conjugate();
            }
        } else {
            if (fwd) fft_line_stages<L, E, -1, 0, TWS>(v, tid, line, tw, lsync);
            between();
            if (inv) fft_line_stages<L, E, +1, 0, TWS>(v, tid, line, tw, lsync);
        }
    };

    // A pass loops over one copy of the factors and reductions, at the places before, between and after
    // its sandwiches. A launch finds the instruction caches cold: with a copy per place, 71 KB of code in
    // the FP64 1024-point two-sandwich pass (30 KB now), its first transforms took 3,500 cycles each more
    // than the second ones of the same launch.
    bool store_out = false;  // write v back to psi at the end
    if constexpr (MODE == PM_FFT_FWD || MODE == PM_FFT_INV) {
        fft_line_stages<L, E, MODE == PM_FFT_FWD ? -1 : +1, 0, TWS>(v, tid, line, tw, lsync);
#pragma unroll
        for (int u = 0; u < E; ++u) v[u] = cscale(v[u], a.scale);
        store_out = true;
    } else if constexpr (MODE == PM_ROUNDTRIP) {
        fft_line_stages<L, E, +1, 0, TWS>(v, tid, line, tw, lsync);
#pragma unroll
        for (int u = 0; u < E; ++u) v[u] = cscale(v[u], a.scale);
        if (active)  // a 1-D axis: no other axes
            apply_tables<R, E, T, true>(v, tid, lbase, a.mid_real, a.mid_cplx, a.mid_ax_cplx[0], a.mid_ax_real[0],
                                        false, V{}, false, R(1), key0 ^ 0x2545f491u);
        if (HAS_RED && a.red.n) {
            reduce();
            second_mid();
        }
        fft_line_stages<L, E, -1, 0, TWS>(v, tid, line, tw, lsync);
        store_out = true;
    } else if constexpr (MODE == PM_SPECRED) {
        fft_line_stages<L, E, -1, 0, TWS>(v, tid, line, tw, lsync);
        reduce();
    } else if constexpr (MODE == PM_APPLY) {
        sandwich(true, true, [&] {
            if (a.spec) spectral_ldg(a.spec, key0);
        });
        if (active) {
            // a branch-free loop per term, so that its reads go out together
            auto flat_at = [&](int u) { return base + ((long long)(tid + u * T) << log2S); };
            if (a.apply_vtab) {
#pragma unroll
                for (int u = 0; u < E; ++u)
                    v[u] = cadd(v[u], cscale(a.psi[flat_at(u)], R(__ldg(a.apply_vtab + flat_at(u)))));
            }
            if (a.apply_acc) {
                const V* __restrict__ sum = a.dst;
#pragma unroll
                for (int u = 0; u < E; ++u) v[u] = cadd(v[u], sum[flat_at(u)]);
            }
        }
        // The sums before the store: their partner reads go across the stride of lines that other CTAs share
        // sectors with, and behind the store they waited for it (two energy moments at 1024^2: 97 us against
        // 123 in FP32, 118 against 130 in FP64).
        if (a.red.n) reduce();
        if (active && a.dst) {
#pragma unroll
            for (int u = 0; u < E; ++u) a.dst[base + ((long long)(tid + u * T) << log2S)] = v[u];
        }
    } else {
        // PROPAGATE: one sandwich or two; factors and reductions before the first, between them and after
        // the last
#pragma unroll 1
        for (int half = 0;; ++half) {
            const int place = half == 0 ? 0 : (half == a.sandwiches ? 2 : 1);
            if (active && (a.points >> place & 1)) {
                V lf = fone<V>();
                R lr = R(1);
                bool use_lf = false, use_lr = false;
                const V* pc = nullptr;  // of the pass axis
                const R* pr = nullptr;
#pragma unroll
                for (int k = 0; k < MAX_DIM; ++k) {
                    if (k >= a.dim) break;  // the grid's axes only (a 2-D pass runs two turns of the six)
                    const V* c = place == 1 ? a.mid_ax_cplx[k]
                                            : ((place == 0) == (a.ax_in_prologue != 0) ? a.ax_cplx[k] : nullptr);
                    const R* r = place == 1 ? a.mid_ax_real[k] : (place == 2 ? a.ax_real[k] : nullptr);
                    if (k == a.axis) {
                        pc = c;
                        pr = r;
                        continue;
                    }
                    const long long ik = (base >> a.shift[k]) & a.nmask[k];
                    if (c) { lf = fcompose(lf, c[ik]); use_lf = true; }
                    if (r) { lr *= r[ik]; use_lr = true; }
                }
                if (place == 0 && a.pro_scale_dev) { lr *= R(*a.pro_scale_dev); use_lr = true; }
                apply_tables<R, E, T>(v, tid, lbase,
                                      place == 0 ? a.pro_real : (place == 1 ? a.mid_real : a.epi_real),
                                      place == 0 ? a.pro_cplx : (place == 1 ? a.mid_cplx : a.epi_cplx), pc, pr,
                                      use_lf, lf, use_lr, lr,
                                      key0 ^ (place == 0 ? 0x51ed270bu : (place == 1 ? 0x2545f491u : 0x68e31da4u)));
            }
            if (HAS_RED && a.red.n && place == (a.red_at_mid ? 1 : 2)) {
                reduce();
                if (place == 1) second_mid();
            }
            if (place == 2) break;
            const bool fwd = !ENDS || half > 0 || !a.from_p, inv = !ENDS || half + 1 < a.sandwiches || !a.to_p;
            sandwich(fwd, inv, [&] {
                const V* __restrict__ sp = half ? a.spec2 : (a.spec ? a.spec + (a.spec_full ? lbase : 0ll) : nullptr);
                const uint32_t kh = key0 + uint32_t(half * L);
                if constexpr (SH::SPEC_SMEM) {  // host: never with spec_full
                    if (sp) spectral(spec_s + half * L, kh);
                } else {
                    if (sp) spectral_ldg(sp, kh);
                }
                if (!fwd || !inv) {
                    const R sc = (fwd || inv) ? a.p_scale : a.p_scale * a.p_scale;
#pragma unroll
                    for (int u = 0; u < E; ++u) v[u] = cscale(v[u], sc);
                }
            });
        }
        store_out = true;
    }

    if (store_out) {
        if constexpr (STRIDED) {
            if (TMA && g * G + G > nlines) {
                // the last group of a pass whose line count G does not divide: its boxes were loaded
                // with the missing lines filled in, and its lines go back by plain stores (a box store
                // would reach past the tensor)
                if (active) {
#pragma unroll
                    for (int u = 0; u < E; ++u) a.psi[base + ((long long)(tid + u * T) << log2S)] = v[u];
                }
            } else if constexpr (TMA) {
                // the G lines back in [row][line] order, then one thread stores the boxes
                constexpr int BOXL = L < 256 ? L : 256;
                __syncthreads();  // every line is done with its exchange buffer
#pragma unroll
                for (int u = 0; u < E; ++u) lines[(tid + u * T) * G + w] = v[u];
                fence_proxy_async_smem();
                __syncthreads();
                if (t == 0) {
                    const long long lam0 = g * G;
                    const int x = int(lam0 & smask) * int(sizeof(V) / sizeof(uint64_t));
                    const int z = int(lam0 >> log2S);
#pragma unroll 1
                    for (int c = 0; c < L / BOXL; ++c) tma_store_3d(&a.tmap, lines + c * BOXL * G, x, c * BOXL, z);
                    bulk_commit();
                    bulk_wait_read_all();
                }
            } else {
                // park the line in shared memory, then a coalesced copy-out over the G lines
                lsync();
#pragma unroll
                for (int u = 0; u < E; ++u) line[spad<E>(tid + u * T)] = v[u];
                __syncthreads();
#pragma unroll 4
                for (int e = t; e < G * L; e += NT) {
                    const int wl = e % G, m = e / G;
                    const long long l2 = g * G + wl;
                    if (l2 < nlines) a.psi[line_base(l2) + ((long long)m << log2S)] = lines[SH::line_off(wl) + spad<E>(m)];
                }
            }
        } else if (active) {
            V* __restrict__ out = a.psi;
#pragma unroll
            for (int u = 0; u < E; ++u) out[base + tid + u * T] = v[u];
        }
    }
}

template <typename R, int L, int SK, int KMODE, int VAR = 0>
__global__ void __launch_bounds__(PassShape<R, L, VAR>::NT, PassShape<R, L, VAR>::MINB)
    qnd_pass_kernel(const __grid_constant__ PassArgs<R> a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    pass_group<R, L, SK, KMODE, VAR>(a, blockIdx.x, gridDim.x, smem_raw, [] {
        pdl_wait();
        pdl_launch_dependents();
    });
}

// Element-wise reductions over a whole state in r-space (no transform): norm, dipole,
// acceleration, potential energy of an arbitrary state.
// Bound by the reads of the state, its partner and the weights: a thread has Q points of each on their way
// at a time, in 64 registers, so that all of the grid's 4 blocks per SM (reduce_blocks) run in one wave. Norm,
// dipoles and energy in FP32 take, with one, two and four points, 202, 192 and 191 us at 2^21 points and 139, 137
// and 145 at 1024^2 (code to fetch); with 79 registers, and so a second wave of blocks, 228 and 164.
template <typename R>
__global__ void __launch_bounds__(256, 4) qnd_grid_reduce_kernel(const __grid_constant__ PassArgs<R> a, long long n) {
    using V = cplx_t<R>;
    constexpr int Q = 2;
    double acc[MAX_RED];
#pragma unroll
    for (int k = 0; k < MAX_RED; ++k) acc[k] = 0.0;
    const int sa = a.shift[a.axis], log2L = __popcll(a.nmask[a.axis]);  // lengths are powers of two
    const long long step = (long long)gridDim.x * blockDim.x;
    for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += Q * step) {
        // a point past the end reads the last one again and is not added
        auto at = [&](int q) { return i0 + q * step < n ? i0 + q * step : n - 1; };
        double abs2[Q], other[Q];  // |v|^2; Re(conj(partner) v), or without a partner the test of RK_NONFINITE
        {
            V v[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) v[q] = a.psi[at(q)];
            if (a.partner) {
                V p[Q];
#pragma unroll
                for (int q = 0; q < Q; ++q) p[q] = a.partner[at(q)];
#pragma unroll
                for (int q = 0; q < Q; ++q) other[q] = double(p[q].x) * double(v[q].x) + double(p[q].y) * double(v[q].y);
            } else {
#pragma unroll
                for (int q = 0; q < Q; ++q) other[q] = isfinite(double(v[q].x)) && isfinite(double(v[q].y)) ? 0.0 : 1.0;
            }
#pragma unroll
            for (int q = 0; q < Q; ++q) abs2[q] = double(v[q].x) * double(v[q].x) + double(v[q].y) * double(v[q].y);
        }
#pragma unroll
        for (int k = 0; k < MAX_RED; ++k) {
            if (k >= a.red.n) break;
            const bool square = a.red.kind[k] == RK_ABS2;
            const int wk = a.red.wkind[k];
            double w[Q];
            if (wk == WK_ONE) {
#pragma unroll
                for (int q = 0; q < Q; ++q) w[q] = 1.0;
            } else {
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    long long li = at(q);
                    if (wk == WK_AXIS) {
                        li = (li >> a.red.wshift[k]) & a.red.wmask[k];
                    } else if (a.red_lm) {  // a full-grid weight in the line-major order of `axis`
                        const long long m = (li >> sa) & a.nmask[a.axis];
                        li = ((((li >> sa >> log2L) << sa) | (li & ((1ll << sa) - 1))) << log2L) + m;
                    }
                    w[q] = __ldg(a.red.wtab[k] + li);
                }
            }
#pragma unroll
            for (int q = 0; q < Q; ++q)
                if (i0 + q * step < n) acc[k] += (square ? abs2[q] : other[q]) * w[q];
        }
    }
    finish_red<256>(a.red, acc);
}

}  // namespace qnd
