// Observables: Pauli-sum application (lam = H psi), per-instance inner
// products and segment sums of FP64 partials.  All reductions accumulate in
// FP64 in a fixed order (deterministic).
#include <algorithm>

#include "common.cuh"
#include "pauli.cuh"

namespace qs {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxTerms = 128;
constexpr uint64_t kMaxInnerBlocks = 1024;  // partial sums per instance (workspace: 16 B each)

// Terms of one X mask together: group g is the terms [gbeg[g], gbeg[g+1]).
struct PauliTerms {
    int n, cplx, ngroups;
    int gbeg[kMaxTerms + 1];
    uint64_t gx[kMaxTerms];                  // per group
    uint64_t xs[kMaxTerms], zs[kMaxTerms];
    double cre[kMaxTerms], cim[kMaxTerms];  // coefficient times i^popc(x & z)
    __device__ __forceinline__ uint64_t x(int t) const { return xs[t]; }
    __device__ __forceinline__ uint64_t z(int t) const { return zs[t]; }
    __device__ __forceinline__ double re(int t) const { return cre[t]; }
    __device__ __forceinline__ double im(int t) const { return cim[t]; }
};

// out = H psi, eight amplitudes per thread (terms in pauli_before order).  2^24
// amplitudes in complex64, 31 terms with 17 X masks (B200): 446 us; 789 us with
// one parity per term and amplitude.
template <typename V, bool CPLX>
__global__ void __launch_bounds__(kThreads)
k_pauli_sum8(const V* __restrict__ psi, V* __restrict__ out, uint64_t N, const __grid_constant__ PauliTerms p) {
    static_assert(kThreads == 1 << kPauliShift, "one chunk per block and step");
    for (uint64_t c = blockIdx.x; c * kPauliChunk < N; c += gridDim.x) {
        const uint64_t base = c * kPauliChunk + threadIdx.x;
        double re[kPauliU], im[kPauliU];
        pauli8<CPLX>(p, p.n, base, [&](uint64_t i) { return psi[i]; }, re, im);
#pragma unroll
        for (int u = 0; u < kPauliU; ++u) out[base | (uint64_t(u) << kPauliShift)] = mk<V>(re[u], im[u]);
    }
}

// The same with one amplitude per thread: per group psi[j ^ x] is read once and
// multiplied by the group's signed coefficient sum (FP64).
template <typename V>
__global__ void __launch_bounds__(kThreads)
k_pauli_sum(const V* __restrict__ psi, V* __restrict__ out, uint64_t N, const __grid_constant__ PauliTerms p) {
    const uint64_t stride = uint64_t(gridDim.x) * kThreads;
    for (uint64_t j = uint64_t(blockIdx.x) * kThreads + threadIdx.x; j < N; j += stride) {
        double re = 0.0, im = 0.0;
        for (int g = 0; g < p.ngroups; ++g) {
            const uint64_t src = j ^ p.gx[g];
            const V a = psi[src];
            double sr = 0.0, si = 0.0;
            for (int t = p.gbeg[g]; t < p.gbeg[g + 1]; ++t) {
                const bool neg = __popcll(p.zs[t] & src) & 1;
                sr += neg ? -p.cre[t] : p.cre[t];
                si += neg ? -p.cim[t] : p.cim[t];
            }
            const double ar = double(a.x), ai = double(a.y);
            re += sr * ar - si * ai;
            im += sr * ai + si * ar;
        }
        out[j] = mk<V>(re, im);
    }
}

// Per-instance partial sums of conj(a) b: grid = (blocks per instance, instances).
template <typename V>
__global__ void __launch_bounds__(kThreads)
k_inner_partial(const V* __restrict__ a, const V* __restrict__ b, uint64_t inst_len, double* __restrict__ part) {
    const uint64_t inst = blockIdx.y;
    const V* ai = a + inst * inst_len;
    const V* bi = b + inst * inst_len;
    double re = 0.0, im = 0.0;
    for (uint64_t j = uint64_t(blockIdx.x) * kThreads + threadIdx.x; j < inst_len; j += uint64_t(gridDim.x) * kThreads) {
        const V u = ai[j], v = bi[j];
        re += double(u.x) * double(v.x) + double(u.y) * double(v.y);
        im += double(u.x) * double(v.y) - double(u.y) * double(v.x);
    }
    __shared__ double sr[kThreads / 32], si[kThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, o);
        im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if ((threadIdx.x & 31) == 0) {
        sr[threadIdx.x >> 5] = re;
        si[threadIdx.x >> 5] = im;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double r = 0.0, i = 0.0;
        for (int w = 0; w < kThreads / 32; ++w) { r += sr[w]; i += si[w]; }
        const uint64_t at = 2 * (inst * gridDim.x + blockIdx.x);
        part[at] = r;
        part[at + 1] = i;
    }
}

// Sums of `nseg` segments of `seglen` complex FP64 values, one warp per
// segment: lane l adds elements l, l + 32, ... (coalesced), then a fixed
// shuffle tree (the same order on every run).
__global__ void __launch_bounds__(kThreads) k_segsum(const double* __restrict__ in, int64_t nseg, int64_t seglen,
                                                     double* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = int64_t(gridDim.x) * (kThreads / 32);
    for (int64_t s = int64_t(blockIdx.x) * (kThreads / 32) + (threadIdx.x >> 5); s < nseg; s += warps) {
        const double2* p = reinterpret_cast<const double2*>(in) + s * seglen;
        double r = 0.0, i = 0.0;
        for (int64_t t = lane; t < seglen; t += 32) {
            const double2 v = p[t];
            r += v.x;
            i += v.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            r += __shfl_xor_sync(0xffffffffu, r, o);
            i += __shfl_xor_sync(0xffffffffu, i, o);
        }
        if (lane == 0) {
            out[2 * s] = r;
            out[2 * s + 1] = i;
        }
    }
}

}  // namespace
}  // namespace qs

using namespace qs;

extern "C" int qs_apply_pauli_sum(const void* psi, void* out, int n, int dtype, const uint64_t* xmask,
                                  const uint64_t* zmask, const double* coeff, int nterms, void* stream) {
    QS_REQUIRE(psi != nullptr && out != nullptr && psi != out, "psi and out must be distinct non-null vectors");
    QS_REQUIRE(n >= 1 && n <= 40, "qubit count %d outside [1, 40]", n);
    QS_REQUIRE(valid_dtype(dtype), "bad dtype %d", dtype);
    QS_REQUIRE(nterms >= 1 && nterms <= kMaxTerms, "term count %d outside [1, %d]", nterms, kMaxTerms);
    QS_REQUIRE(xmask != nullptr && zmask != nullptr && coeff != nullptr, "null term arrays");
    static thread_local PauliTerms p;
    p.n = nterms;
    int order[kMaxTerms];
    for (int t = 0; t < nterms; ++t) {
        QS_REQUIRE((xmask[t] >> n) == 0 && (zmask[t] >> n) == 0, "term %d acts on bits >= n", t);
        order[t] = t;
    }
    std::stable_sort(order, order + nterms, [&](int a, int b) { return xmask[a] < xmask[b]; });
    p.ngroups = 0;
    for (int i = 0; i < nterms; ++i)
        if (i == 0 || xmask[order[i]] != xmask[order[i - 1]]) {
            p.gx[p.ngroups] = xmask[order[i]];
            p.gbeg[p.ngroups++] = i;
        }
    p.gbeg[p.ngroups] = nterms;
    const uint64_t N = uint64_t(1) << n;
    // Eight amplitudes per thread from 2^20 amplitudes on, where the masks are
    // all different (a transform per term) from 2^22.  Below, an eighth of the
    // threads do not hide the terms' latency.  31 terms with 17 masks / 128 with
    // one / 100 with 100, complex64 (B200), one against eight amplitudes: 2^14
    // 6.3, 18.6 / 6.3, 19.8 / 24, 109 us; 2^18 16.6, 21.1 / 22.7, 20.6 / 64, 121
    // us; 2^20 54, 41 / 85, 37 / 250, 268 us; 2^22 202, 110 / 323, 94 / 966, 943 us.
    const bool eight = N >= (uint64_t(1) << (p.ngroups < nterms ? 20 : 22));
    if (eight)
        std::stable_sort(order, order + nterms,
                         [&](int a, int b) { return pauli_before(xmask[a], zmask[a], xmask[b], zmask[b]); });
    p.cplx = 0;
    for (int i = 0; i < nterms; ++i) {
        const int t = order[i];
        p.xs[i] = xmask[t];
        p.zs[i] = zmask[t];
        // fold i^popc(x & z) (Y = i X Z) into the coefficient
        double re = coeff[2 * t], im = coeff[2 * t + 1];
        for (int k = 0; k < (__builtin_popcountll(xmask[t] & zmask[t]) & 3); ++k) {
            double r2 = -im, i2 = re;
            re = r2;
            im = i2;
        }
        p.cre[i] = re;
        p.cim[i] = im;
        if (im != 0.0) p.cplx = 1;
    }
    const cudaStream_t st = as_stream(stream);
    auto launch = [&](auto zero) {
        using V = decltype(zero);
        const V* in = static_cast<const V*>(psi);
        V* o = static_cast<V*>(out);
        if (!eight) {
            k_pauli_sum<V><<<grid_for(N, kThreads, 8), kThreads, 0, st>>>(in, o, N, p);
            return;
        }
        const unsigned grid = grid_for(N / kPauliChunk, 1, 8);
        if (p.cplx) k_pauli_sum8<V, true><<<grid, kThreads, 0, st>>>(in, o, N, p);
        else        k_pauli_sum8<V, false><<<grid, kThreads, 0, st>>>(in, o, N, p);
    };
    if (dtype == QS_C128) launch(double2{});
    else                  launch(float2{});
    QS_CHECK_LAUNCH("qs_apply_pauli_sum");
    return QS_OK;
}

extern "C" int qs_inner_batched(const void* a, const void* b, int n, int dtype, int inst_bits, double* out_dev,
                                void* ws, size_t ws_bytes, void* stream) {
    QS_REQUIRE(a != nullptr && b != nullptr && out_dev != nullptr, "null argument");
    QS_REQUIRE(n >= 1 && n <= 40 && inst_bits >= 1 && inst_bits <= n, "bad sizes n=%d inst_bits=%d", n, inst_bits);
    QS_REQUIRE(valid_dtype(dtype), "bad dtype %d", dtype);
    const uint64_t ninst = uint64_t(1) << (n - inst_bits);
    const uint64_t len = uint64_t(1) << inst_bits;
    // blocks per instance: up to one per 2048 amplitudes, enough in total to
    // fill the GPU (8 CTAs per SM), at most kMaxInnerBlocks
    uint64_t per = (len + kThreads * 8 - 1) / (kThreads * 8);
    uint64_t fill = (uint64_t(sm_count()) * 8 + ninst - 1) / ninst;
    if (per > fill) per = fill;
    if (per > kMaxInnerBlocks) per = kMaxInnerBlocks;
    const uint64_t fits = ws == nullptr ? 0 : uint64_t(ws_bytes / (sizeof(double) * 2 * ninst));
    if (per > fits) per = fits;  // as many partials as the workspace holds
    if (per < 1) {
        set_error("qs_inner_batched needs at least %zu bytes of workspace", sizeof(double) * 2 * size_t(ninst));
        return QS_EWORKSPACE;
    }
    QS_REQUIRE(ninst <= 65535, "at most 65535 instances per call");
    const dim3 grid = dim3(unsigned(per), unsigned(ninst), 1u);
    double* part = static_cast<double*>(ws);
    if (dtype == QS_C128) k_inner_partial<double2><<<grid, kThreads, 0, as_stream(stream)>>>((const double2*)a, (const double2*)b, len, part);
    else                  k_inner_partial<float2><<<grid, kThreads, 0, as_stream(stream)>>>((const float2*)a, (const float2*)b, len, part);
    k_segsum<<<grid_for(ninst, kThreads / 32, 8), kThreads, 0, as_stream(stream)>>>(part, int64_t(ninst), int64_t(per),
                                                                                    out_dev);
    QS_CHECK_LAUNCH("qs_inner_batched");
    return QS_OK;
}

extern "C" int qs_segment_sum(const double* in_dev, int64_t nseg, int64_t seglen, double* out_dev, void* stream) {
    QS_REQUIRE(in_dev != nullptr && out_dev != nullptr && nseg >= 1 && seglen >= 1, "bad arguments");
    k_segsum<<<grid_for(uint64_t(nseg), kThreads / 32, 8), kThreads, 0, as_stream(stream)>>>(in_dev, nseg, seglen,
                                                                                              out_dev);
    QS_CHECK_LAUNCH("qs_segment_sum");
    return QS_OK;
}
