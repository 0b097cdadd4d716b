// qnd_chain1d.cu — a whole chain of kinetic sandwiches on a 1-D grid of up to 4096 points in one
// launch: one CTA holds the line in registers from the first sandwich to the last, so that a chain
// reads and writes the state once and pays one launch, instead of one pass of one CTA per pair of
// sandwiches with the launches, the state's round trip through L2 and (imaginary time) the
// Gram-Schmidt kernels between them.
//
// What bounds it: one SM. A line of 4096 FP64 points needs 588 FP64 instructions per 16 points and
// transform, about 2,400 cycles of one SM's FP64 pipe, and its exchanges about 2,000 cycles of its
// shared memory; two transforms per sandwich. The tables come from L2: the spectral row is read into
// registers during the forward transform, the r-space factors one table after the other after the inverse.
#include <algorithm>

#include "qnd_kernels.cuh"

#ifndef QND_CHAIN_FP64
#error "compile with -DQND_CHAIN_FP64=0 or 1"
#endif

namespace qnd {

// Sums of n (at most MAX_RED) accumulators over the CTA's T threads (whole warps), to out[0..n) in shared memory,
// visible to every thread on return. red: [T / 32][MAX_RED] shared scratch.
template <int T> __device__ __forceinline__ void cta_sums(const double* acc, int n, double (*red)[MAX_RED], double* out) {
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
#pragma unroll
    for (int k = 0; k < MAX_RED; ++k) {
        if (k >= n) break;
        const double s = warp_sum(acc[k]);
        if (lane == 0) red[wid][k] = s;
    }
    __syncthreads();
    if (t < n) {
        double s = 0.0;
        for (int w = 0; w < T / 32; ++w) s += red[w][t];
        out[t] = s;
    }
    __syncthreads();
}

// Threads per line and the shared memory of a chain: E values per thread.
template <typename R, int L, int E> struct ChainShape {
    using P = FFTPlan<L, E>;
    static constexpr int T = L / E;
    static constexpr int NT = T < 32 ? 32 : T;  // threads: a shorter line's lanes are repeated over one warp
    static constexpr int TW = ((sizeof(R) == 8 ? P::twb_size() : P::tw_size()) + 1) & ~1;
    static constexpr size_t SMEM = sizeof(cplx_t<R>) * (size_t(TW) + P::SMEM_LINE);
};

template <typename R, int L, int E, int OPS>
__global__ void __launch_bounds__(ChainShape<R, L, E>::NT, 1)
    qnd_chain1d_kernel(const __grid_constant__ Chain1dArgs<R, OPS> a) {
    using V = cplx_t<R>;
    using SH = ChainShape<R, L, E>;
    constexpr int T = SH::T, NT = SH::NT;
    static_assert(T % 32 == 0 || 32 % T == 0, "whole warps, or lanes repeated over one");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ double red_s[NT / 32][MAX_RED];
    __shared__ RedShared<NT> red_sh;
    __shared__ double sum_s[MAX_RED];
    __shared__ double coef_s[2 * GS_MAXK];
    V* tw = reinterpret_cast<V*>(smem_raw);
    V* line = tw + SH::TW;
    const int t = threadIdx.x;
    // Lanes past T repeat the first ones' work on the same addresses with the same values; only the first
    // T count in sums.
    const int tid = t % T;
    const bool counts = t < T;
    const LineSync<T> lsync{1};

    // every twiddle's copy on its way at once: a line of one warp copies up to 30 of them a thread
    for (int i = t; i < (sizeof(R) == 8 ? SH::P::twb_size() : SH::P::tw_size()); i += NT) cp_async_elem(tw + i, a.tw + i);
    cp_async_commit();
    V v[E];
#pragma unroll
    for (int u = 0; u < E; ++u) v[u] = a.src[tid + u * T];
    load_red_rows<NT>(a.red, 0, red_sh);
    cp_async_wait<0>();
    __syncthreads();  // twiddles and reductions visible

    // the point-wise factor `mid` (a full-grid table) with the laser phases at `laser`, the step mask
    // and a device scalar
    auto factors = [&](int mid, int laser, bool mask, const double* scale, uint32_t key) {
        apply_tables<R, E, T>(v, tid, 0, mid >= 0 ? a.mid_real[mid] : nullptr, mid >= 0 ? a.mid_cplx[mid] : nullptr,
                              laser >= 0 ? a.field + laser : nullptr, mask ? a.mask : nullptr, false, V{},
                              scale != nullptr, scale ? R(*scale) : R(1), key);
    };
    factors(a.pre_mid, a.pre_laser, false, a.pre_scale, mix32(a.seed) ^ 0x51ed270bu);

#pragma unroll 1
    for (int i = 0; i < a.nops; ++i) {
        const Chain1dOp op = a.ops[i];
        const uint32_t key = mix32(a.seed + 0x9e3779b9u * uint32_t(i + 1));
        const V* __restrict__ sp = op.spec >= 0 ? a.spec[op.spec] : a.field + op.field_spec;
        V f[E];  // the spectral row, on its way during the forward transform
#pragma unroll
        for (int u = 0; u < E; ++u) f[u] = __ldg(sp + tid + u * T);
        fft_line_stages<L, E, -1, 0, true>(v, tid, line, tw, lsync);
#pragma unroll
        for (int u = 0; u < E; ++u)
            v[u] = fmul_spec<L>(v[u], f[u], key + uint32_t(tid + u * T), u == 0 || u == E - 1);
        fft_line_stages<L, E, +1, 0, true>(v, tid, line, tw, lsync);
        factors(op.mid, op.laser, op.mask != 0, nullptr, key ^ 0x2545f491u);
        if (op.obs >= 0) {
#pragma unroll 1
            for (int k = 0; k < a.red.n; ++k) {
                const double own = line_sum<R, E, T>(red_sh.row[k], v, static_cast<const V*>(nullptr), 0, 0, 0, tid);
                const double s = warp_sum(counts ? own : 0.0);
                if ((t & 31) == 0) red_sh.s[t >> 5][k] = s;
            }
            __syncthreads();
            if (t < a.red.n) {
                double s = 0.0;
                for (int w = 0; w < NT / 32; ++w) s += red_sh.s[w][t];
                a.red.out[op.obs + t] = s * a.red.scale[t];
            }
            __syncthreads();  // the warps' sums are read
        }
        if (op.gs) {
            // v = psi - sum_k <psi_k|psi> psi_k, then v / ||v|| (QuantumND_imag.c:280-310)
            for (int k0 = 0; k0 < a.ngs; k0 += MAX_RED / 2) {
                double acc[MAX_RED];
#pragma unroll
                for (int q = 0; q < MAX_RED / 2; ++q) {
                    acc[2 * q] = acc[2 * q + 1] = 0.0;
                    if (k0 + q >= a.ngs || !counts) continue;
                    const V* __restrict__ s = a.states[k0 + q];
#pragma unroll
                    for (int u = 0; u < E; ++u) {
                        const V p = s[tid + u * T];
                        acc[2 * q] += double(p.x) * double(v[u].x) + double(p.y) * double(v[u].y);
                        acc[2 * q + 1] += double(p.x) * double(v[u].y) - double(p.y) * double(v[u].x);
                    }
                }
                const int n = 2 * (a.ngs - k0 < MAX_RED / 2 ? a.ngs - k0 : MAX_RED / 2);
                cta_sums<NT>(acc, n, red_s, sum_s);
                if (t < n) coef_s[2 * k0 + t] = sum_s[t] * a.dNr;
                __syncthreads();
            }
            for (int k = 0; k < a.ngs; ++k) {
                const V* __restrict__ s = a.states[k];
                const R cr = R(coef_s[2 * k]), ci = R(coef_s[2 * k + 1]);
#pragma unroll
                for (int u = 0; u < E; ++u) {
                    const V p = s[tid + u * T];
                    v[u].x -= cr * p.x - ci * p.y;
                    v[u].y -= cr * p.y + ci * p.x;
                }
            }
            double acc[1] = {0.0};
#pragma unroll
            for (int u = 0; u < E; ++u) acc[0] += double(v[u].x) * double(v[u].x) + double(v[u].y) * double(v[u].y);
            if (!counts) acc[0] = 0.0;
            cta_sums<NT>(acc, 1, red_s, sum_s);
            const double n2 = sum_s[0] * a.dNr;
            double scale = 1.0;
            if (n2 < a.gs_tol || !(n2 == n2)) {
                if (t == 0) *a.gs_flag = 1;
            } else {
                scale = 1.0 / sqrt(n2);
            }
            const R sc = R(scale);
#pragma unroll
            for (int u = 0; u < E; ++u) v[u] = cscale(v[u], sc);
        }
        if (op.mid2 >= 0) factors(op.mid2, -1, false, nullptr, key ^ 0x68e31da4u);
    }
#pragma unroll
    for (int u = 0; u < E; ++u) a.psi[tid + u * T] = v[u];
}

template <typename R, int L, int OPS> static cudaError_t launch_args(const Chain1dArgs<R, OPS>& a, cudaStream_t st) {
    constexpr int E = chain1d_values(L, sizeof(R) == 8);
    using SH = ChainShape<R, L, E>;
    auto* fn = &qnd_chain1d_kernel<R, L, E, OPS>;
    if constexpr (SH::SMEM > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(SH::SMEM));
        if (e != cudaSuccess) return e;
    }
    fn<<<1, SH::NT, SH::SMEM, st>>>(a);
    return cudaGetLastError();
}

template <typename R, int L, int OPS>
static cudaError_t launch_ops(const Chain1dHead<R>& head, const Chain1dOp* ops, cudaStream_t st) {
    Chain1dArgs<R, OPS> a;
    static_cast<Chain1dHead<R>&>(a) = head;
    std::copy(ops, ops + head.nops, a.ops);
    return launch_args<R, L>(a, st);
}

template <typename R, int L>
static cudaError_t launch_one(const Chain1dHead<R>& head, const Chain1dOp* ops, cudaStream_t st) {
    static_assert(sizeof(Chain1dArgs<R, CHAIN1D_SHORT>) <= 4096, "the short list's arguments");
    return head.nops <= CHAIN1D_SHORT ? launch_ops<R, L, CHAIN1D_SHORT>(head, ops, st)
                                      : launch_ops<R, L, CHAIN1D_OPS>(head, ops, st);
}

template <typename R> cudaError_t launch_chain1d(int L, const Chain1dHead<R>& a, const Chain1dOp* ops, cudaStream_t st) {
    switch (L) {
    case 128: return launch_one<R, 128>(a, ops, st);
    case 256: return launch_one<R, 256>(a, ops, st);
    case 512: return launch_one<R, 512>(a, ops, st);
    case 1024: return launch_one<R, 1024>(a, ops, st);
    case 2048: return launch_one<R, 2048>(a, ops, st);
    case 4096: return launch_one<R, 4096>(a, ops, st);
    default: return cudaErrorInvalidValue;
    }
}

#if QND_CHAIN_FP64
template cudaError_t launch_chain1d<double>(int, const Chain1dHead<double>&, const Chain1dOp*, cudaStream_t);
#else
template cudaError_t launch_chain1d<float>(int, const Chain1dHead<float>&, const Chain1dOp*, cudaStream_t);
#endif

}  // namespace qnd
