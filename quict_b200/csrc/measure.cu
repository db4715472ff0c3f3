// Measurement, reset, FP64 reductions and sampling.
//
// Sampling replaces the reference's shots x qubits loop (one reduction, one
// device->host read and one collapse kernel per qubit per shot,
// statevector_simulator.py:595-626) with a sum tree built once: FP64 sums of
// 2^B-amplitude blocks at the leaves, a binary tree above them.  Each shot is
// one warp that walks the tree from the root (qubit 0 = the vector's top bit
// first) and finishes inside its leaf block from the block's own amplitudes.
#include <mutex>

#include "common.cuh"

namespace qs {
namespace {

constexpr int kThreads = 256;
constexpr int kReduceCtas = 1024;     // partial-sum slots in the reduce workspace

// p_i of a probability source
template <typename V, int SRC>
__device__ __forceinline__ double prob_at(const V* __restrict__ s, uint64_t i, uint64_t dstride) {
    if (SRC == QS_SRC_SV) return cnorm2(s[i]);
    return double(s[i * dstride].x);
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Block-level sum; result valid in thread 0.
__device__ __forceinline__ double block_sum(double x) {
    __shared__ double part[32];
    x = warp_sum(x);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) part[w] = x;
    __syncthreads();
    double r = 0.0;
    if (w == 0) {
        r = (l < int(blockDim.x >> 5)) ? part[l] : 0.0;
        r = warp_sum(r);
    }
    __syncthreads();
    return r;
}

// Sum of p over the compact space with `bit` removed (bit < 0: everything).
// Eight loads in flight per thread: 25 qubits in complex64 (B200), half of
// the 256 MB: 33 us (51 us on the lowest bits, where every sector is read),
// 62-73 us with one.
template <typename V, int SRC>
__global__ void __launch_bounds__(kThreads)
k_partial(const V* __restrict__ s, uint64_t items, int bit, uint64_t dstride, double* __restrict__ part) {
    constexpr int U = 8;
    double acc = 0.0;
    const uint64_t stride = uint64_t(gridDim.x) * kThreads;
    uint64_t j = uint64_t(blockIdx.x) * kThreads + threadIdx.x;
    for (; j + (U - 1) * stride < items; j += U * stride) {
        V v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t q = j + u * stride, i = bit >= 0 ? insert0(q, bit) : q;
            v[u] = s[SRC == QS_SRC_SV ? i : i * dstride];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) acc += SRC == QS_SRC_SV ? cnorm2(v[u]) : double(v[u].x);
    }
    for (; j < items; j += stride) {
        uint64_t i = bit >= 0 ? insert0(j, bit) : j;
        acc += prob_at<V, SRC>(s, i, dstride);
    }
    acc = block_sum(acc);
    if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

__global__ void __launch_bounds__(kThreads) k_finish(const double* __restrict__ part, int nparts, double* out) {
    double acc = 0.0;
    for (int i = threadIdx.x; i < nparts; i += kThreads) acc += part[i];
    acc = block_sum(acc);
    if (threadIdx.x == 0) *out = acc;
}

// Collapse, amplitude by amplitude in vector order: every access of a warp is
// contiguous.
template <typename V>
__global__ void __launch_bounds__(kThreads)
k_collapse_each(V* __restrict__ v, uint64_t N, int bit, int outcome, double scale) {
    const uint64_t stride = uint64_t(gridDim.x) * kThreads;
    for (uint64_t i = uint64_t(blockIdx.x) * kThreads + threadIdx.x; i < N; i += stride) {
        if (int((i >> bit) & 1) == outcome) {
            V a = v[i];
            a.x *= scale; a.y *= scale;
            v[i] = a;
        } else {
            v[i] = mk<V>(0.0, 0.0);
        }
    }
}

// The two below walk the pairs of `bit`, U in flight per thread, and read only the
// half that is kept: 25 qubits in complex64 (B200), 256 MB: collapse 65-88 us
// (65-95 us amplitude by amplitude), reset 67 us (131 us with a division per
// component).
template <typename V>
__global__ void __launch_bounds__(kThreads) k_collapse(V* __restrict__ v, uint64_t items, int bit, int outcome, double scale) {
    constexpr int U = 4;
    const uint64_t stride = uint64_t(gridDim.x) * kThreads, off = uint64_t(1) << bit;
    const uint64_t keep = outcome ? off : 0;
    for (uint64_t j0 = uint64_t(blockIdx.x) * kThreads + threadIdx.x; j0 < items; j0 += U * stride) {
        V a[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (j0 + u * stride < items) a[u] = v[insert0(j0 + u * stride, bit) | keep];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (j0 + u * stride >= items) continue;
            const uint64_t i0 = insert0(j0 + u * stride, bit);
            a[u].x *= scale; a[u].y *= scale;
            v[i0 | keep] = a[u];
            v[i0 | (keep ^ off)] = mk<V>(0.0, 0.0);
        }
    }
}

// x / alpha for a given r = 1 / alpha: one correction step on x r gives the
// correctly rounded quotient (Markstein, IBM J. Res. Dev. 34(1), 1990).  A
// quotient of a component that is not finite or too small for the remainder
// to be exact is divided.
__device__ __forceinline__ double div_by(double x, double alpha, double r) {
    const double q = x * r;
    if (!(fabs(q) > 1e-280 && fabs(q) < 1e300)) return x / alpha;
    return fma(fma(-q, alpha, x), r, q);
}
__device__ __forceinline__ float div_by(float x, double alpha, double r) {
    return float(double(x) * r);  // within half a unit of the float result either way
}

// Reference reset rule: alpha = sqrt(P0); alpha < 1e-6 -> v0 <- v1, else
// v0 <- v0 / alpha; v1 <- 0 either way.
template <typename V, int U>
__global__ void __launch_bounds__(kThreads) k_reset(V* __restrict__ v, uint64_t items, int bit, double alpha, bool move) {
    const uint64_t stride = uint64_t(gridDim.x) * kThreads, off = uint64_t(1) << bit;
    const double r = 1.0 / alpha;
    for (uint64_t j0 = uint64_t(blockIdx.x) * kThreads + threadIdx.x; j0 < items; j0 += U * stride) {
        V a[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (j0 + u * stride < items) a[u] = v[insert0(j0 + u * stride, bit) | (move ? off : 0)];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (j0 + u * stride >= items) continue;
            const uint64_t i0 = insert0(j0 + u * stride, bit);
            if (!move) {
                a[u].x = div_by(a[u].x, alpha, r);
                a[u].y = div_by(a[u].y, alpha, r);
            }
            v[i0] = a[u];
            v[i0 | off] = mk<V>(0.0, 0.0);
        }
    }
}

// -------------------------------------------------------------- sum tree
// FP64 sums of leaf blocks of 2^bb probabilities, and above them every fifth
// level of the binary tree: level 0 holds the leaves, an entry of level j + 1
// sums 32 entries of level j (the top one fewer), the last level is the total.
// The four levels in between are never stored: a warp that holds the 32
// entries below a node has them from five butterfly steps, so a shot costs
// one coalesced load per five levels instead of a dependent load per level.
// 26 qubits in complex64, 100,000 shots (B200): a heap with every level stored,
// one dependent load per level and 32 elements per lane in the leaf took
// 649 us + 23 us for 16 launches of single levels; this takes 153 + 6 us, and
// the leaves 75 us (120 us with one load in flight).  What is left is the
// leaves' 8 KB a shot.
constexpr int kMaxLevels = 8;  // 30 tree bits over the leaves, five per level, and the root

struct TreeShape {
    int bb, levels;             // leaf bits; stored levels
    int lg[kMaxLevels];         // log2 of a level's entries
    uint64_t off[kMaxLevels];   // its first entry
    uint64_t total;             // entries of all levels
};

constexpr int kBlockBits = 10;  // leaf block = 2^10 probabilities: 32 rows of 32

TreeShape tree_shape(int n) {
    TreeShape t{};
    t.bb = n < kBlockBits ? n : kBlockBits;
    int lg = n - t.bb;
    for (;;) {
        t.lg[t.levels] = lg;
        t.off[t.levels++] = t.total;
        t.total += uint64_t(1) << lg;
        if (lg == 0) break;
        lg = lg > 5 ? lg - 5 : 0;
    }
    return t;
}

// Sum over the warp, lanes paired by ascending distance (the order in which
// the descent recomputes the levels between two stored ones).
__device__ __forceinline__ double tree_sum(double x) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// One warp per leaf, eight loads in flight per lane.
template <typename V, int SRC>
__global__ void __launch_bounds__(kThreads)
k_leaves(const V* __restrict__ s, int bb, uint64_t nleaf, uint64_t dstride, double* __restrict__ leaf) {
    constexpr int U = 8;
    const int lane = threadIdx.x & 31;
    const uint64_t warps = uint64_t(gridDim.x) * (kThreads / 32);
    for (uint64_t b = uint64_t(blockIdx.x) * (kThreads / 32) + (threadIdx.x >> 5); b < nleaf; b += warps) {
        const uint64_t base = (b << bb) + lane;
        double acc = 0.0;
        if (bb == kBlockBits) {
            for (int r = 0; r < 32; r += U) {
                V v[U];
#pragma unroll
                for (int i = 0; i < U; ++i) v[i] = s[(base + 32 * (r + i)) * (SRC == QS_SRC_SV ? 1 : dstride)];
#pragma unroll
                for (int i = 0; i < U; ++i) acc += SRC == QS_SRC_SV ? cnorm2(v[i]) : double(v[i].x);
            }
        } else {
            for (int e = lane; e < (1 << bb); e += 32) acc += prob_at<V, SRC>(s, base - lane + e, dstride);
        }
        acc = tree_sum(acc);
        if (lane == 0) leaf[b] = acc;
    }
}

// One warp per entry of the level above `in` (2^lg entries).
__global__ void __launch_bounds__(kThreads) k_level(const double* __restrict__ in, int lg, double* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const uint64_t warps = uint64_t(gridDim.x) * (kThreads / 32);
    const uint64_t cnt = lg > 5 ? uint64_t(1) << (lg - 5) : 1;
    const uint64_t size = uint64_t(1) << lg;
    for (uint64_t g = uint64_t(blockIdx.x) * (kThreads / 32) + (threadIdx.x >> 5); g < cnt; g += warps) {
        const double t = tree_sum(32 * g + lane < size ? in[32 * g + lane] : 0.0);
        if (lane == 0) out[g] = t;
    }
}

// All levels above `from`, in one block (from at most 2^14 entries): no launch
// between two small levels.
__global__ void __launch_bounds__(1024) k_top(double* __restrict__ tree, const __grid_constant__ TreeShape t, int from) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int j = from; j + 1 < t.levels; ++j) {
        const double* in = tree + t.off[j];
        const uint64_t size = uint64_t(1) << t.lg[j], cnt = uint64_t(1) << t.lg[j + 1];
        for (uint64_t g = w; g < cnt; g += 32) {
            const double x = tree_sum(32 * g + lane < size ? in[32 * g + lane] : 0.0);
            if (lane == 0) tree[t.off[j + 1] + g] = x;
        }
        __syncthreads();
    }
}

// CDF descent step: go right when u lies beyond the left half's mass, but
// never into a half of zero mass.  The in-block half sums are added in a
// different order from the leaf sums above them, so u can exceed a block's
// recomputed total by a rounding error; the guard then ends the descent on
// the block's last element of nonzero probability instead of one with p = 0.
__device__ __forceinline__ bool cdf_right(double uc, double acc, double sl, double sr) {
    if (!(sr > 0.0)) return false;
    if (!(sl > 0.0)) return true;
    return !(uc <= acc + sl);
}

// A shot's position in the decision sequence: the uniform in use and, in CDF
// mode, the mass strictly left of the current node.
struct Draw {
    const double* us;
    int lvl, n;
    double uc, acc;
};

// Walk down nb <= 5 levels below a node whose 2^nb entries are the lanes' x;
// returns the lane of the entry reached.
template <int MODE>
__device__ __forceinline__ int descend(double x, int nb, Draw& d) {
    double t[6];
    t[0] = x;
#pragma unroll
    for (int k = 0; k < 5; ++k) t[k + 1] = t[k] + __shfl_xor_sync(0xffffffffu, t[k], 1 << k);
    int lo = 0;
#pragma unroll
    for (int k = 4; k >= 0; --k) {
        if (k >= nb) continue;  // warp-uniform
        const double sl = __shfl_sync(0xffffffffu, t[k], lo), sr = __shfl_sync(0xffffffffu, t[k], lo + (1 << k));
        bool right;
        if (MODE == QS_SAMPLE_SEQ) {
            right = d.uc > sl / (sl + sr);
            ++d.lvl;
            d.uc = d.us[d.lvl < d.n ? d.lvl : d.n - 1];
        } else {
            right = cdf_right(d.uc, d.acc, sl, sr);
            if (right) d.acc += sl;
        }
        if (right) lo += 1 << k;
    }
    return lo;
}

// One warp per shot: through the stored levels, then the leaf block's rows of
// 32, then the row.
template <typename V, int SRC, int MODE>
__global__ void __launch_bounds__(kThreads)
k_sample(const V* __restrict__ s, int n, const __grid_constant__ TreeShape t, uint64_t dstride, const double* __restrict__ tree,
         const double* __restrict__ u, int64_t shots, int64_t* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = int64_t(gridDim.x) * (kThreads / 32);
    const int rowbits = t.bb > 5 ? t.bb - 5 : 0, lanebits = t.bb - rowbits;
    for (int64_t shot = int64_t(blockIdx.x) * (kThreads / 32) + (threadIdx.x >> 5); shot < shots; shot += warps) {
        Draw d;
        d.us = MODE == QS_SAMPLE_SEQ ? u + shot * n : u + shot;
        d.lvl = 0;
        d.n = n;
        d.acc = 0.0;
        // CDF mode compares against unnormalised FP64 partial sums, so the
        // uniform is scaled by the total mass (the root): a state whose norm
        // has drifted below 1 (complex64, a density matrix's trace) then
        // never runs off the end of the distribution
        d.uc = MODE == QS_SAMPLE_SEQ ? d.us[0] : d.us[0] * tree[t.off[t.levels - 1]];
        uint64_t node = 0;
        for (int j = t.levels - 2; j >= 0; --j) {
            const int nb = t.lg[j] - t.lg[j + 1];
            const double x = lane < (1 << nb) ? tree[t.off[j] + (node << nb) + lane] : 0.0;
            node = (node << nb) + descend<MODE>(x, nb, d);
        }
        uint64_t base = node << t.bb;
        if (rowbits == 5) {
            // the 32 rows' sums, lane r ending up with row r: five exchanges in
            // which each half of the lanes keeps half of the rows
            double p[32];
#pragma unroll
            for (int r = 0; r < 32; ++r) p[r] = prob_at<V, SRC>(s, base + 32 * r + lane, dstride);
#pragma unroll
            for (int h = 16; h > 0; h >>= 1) {
                const bool upper = lane & h;
#pragma unroll
                for (int i = 0; i < h; ++i) {
                    const double give = upper ? p[i] : p[i + h], keep = upper ? p[i + h] : p[i];
                    p[i] = keep + __shfl_xor_sync(0xffffffffu, give, h);
                }
            }
            base += 32 * uint64_t(descend<MODE>(p[0], 5, d));
        } else if (rowbits > 0) {
            double rows = 0.0;
            for (int r = 0; r < (1 << rowbits); ++r) {
                const double x = tree_sum(prob_at<V, SRC>(s, base + 32 * r + lane, dstride));
                if (lane == r) rows = x;
            }
            base += 32 * uint64_t(descend<MODE>(rows, rowbits, d));
        }
        const double p = lane < (1 << lanebits) ? prob_at<V, SRC>(s, base + lane, dstride) : 0.0;
        base += descend<MODE>(p, lanebits, d);
        if (lane == 0) out[shot] = int64_t(base);
    }
}

__global__ void k_hist(const int64_t* __restrict__ idx, int64_t shots, unsigned long long* counts, int64_t ncounts) {
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t s = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; s < shots; s += stride) {
        int64_t i = idx[s];
        if (i >= 0 && i < ncounts) atomicAdd(&counts[i], 1ull);
    }
}

int check_src(const void* src, int n, int dtype, int src_kind) {
    QS_REQUIRE(src != nullptr, "null source");
    QS_REQUIRE(valid_dtype(dtype), "bad dtype %d", dtype);
    QS_REQUIRE(src_kind == QS_SRC_SV || src_kind == QS_SRC_DM, "bad source kind %d", src_kind);
    QS_REQUIRE(n >= 1 && n <= (src_kind == QS_SRC_SV ? 40 : 20), "qubit count %d out of range", n);
    return QS_OK;
}

template <typename V>
int reduce_t(const void* src, int n, int src_kind, int bit, void* ws, double* out, cudaStream_t st) {
    const V* s = static_cast<const V*>(src);
    uint64_t items = uint64_t(1) << (bit >= 0 ? n - 1 : n);
    uint64_t dstride = (uint64_t(1) << n) + 1;
    unsigned grid = grid_for(items, kThreads * 4, 4);
    if (grid > kReduceCtas) grid = kReduceCtas;
    double* part = static_cast<double*>(ws);
    if (src_kind == QS_SRC_SV) k_partial<V, QS_SRC_SV><<<grid, kThreads, 0, st>>>(s, items, bit, dstride, part);
    else                       k_partial<V, QS_SRC_DM><<<grid, kThreads, 0, st>>>(s, items, bit, dstride, part);
    k_finish<<<1, kThreads, 0, st>>>(part, int(grid), out);
    QS_CHECK_LAUNCH("reduce");
    return QS_OK;
}

template <typename V>
int prepare_t(const void* src, int n, int src_kind, double* tree, cudaStream_t st) {
    const V* s = static_cast<const V*>(src);
    const TreeShape t = tree_shape(n);
    const uint64_t nleaf = uint64_t(1) << t.lg[0];
    const uint64_t dstride = (uint64_t(1) << n) + 1;
    const unsigned grid = grid_for(nleaf, kThreads / 32, 8, 4);
    if (src_kind == QS_SRC_SV) k_leaves<V, QS_SRC_SV><<<grid, kThreads, 0, st>>>(s, t.bb, nleaf, dstride, tree);
    else                       k_leaves<V, QS_SRC_DM><<<grid, kThreads, 0, st>>>(s, t.bb, nleaf, dstride, tree);
    int j = 0;
    for (; j + 1 < t.levels && t.lg[j] > 14; ++j)  // levels that one block would take long over
        k_level<<<grid_for(uint64_t(1) << t.lg[j + 1], kThreads / 32, 8), kThreads, 0, st>>>(tree + t.off[j], t.lg[j],
                                                                                            tree + t.off[j + 1]);
    if (j + 1 < t.levels) k_top<<<1, 1024, 0, st>>>(tree, t, j);
    QS_CHECK_LAUNCH("qs_sample_prepare");
    return QS_OK;
}

template <typename V>
int sample_t(const void* src, int n, int src_kind, const double* tree, const double* u, int64_t shots,
             int mode, int64_t* out, cudaStream_t st) {
    const V* s = static_cast<const V*>(src);
    const TreeShape t = tree_shape(n);
    uint64_t dstride = (uint64_t(1) << n) + 1;
    unsigned grid = grid_for(uint64_t(shots), kThreads / 32, 8, 4);
#define QS_SAMPLE_LAUNCH(SRC, MODE) \
    k_sample<V, SRC, MODE><<<grid, kThreads, 0, st>>>(s, n, t, dstride, tree, u, shots, out)
    if (src_kind == QS_SRC_SV) {
        if (mode == QS_SAMPLE_SEQ) QS_SAMPLE_LAUNCH(QS_SRC_SV, QS_SAMPLE_SEQ);
        else                       QS_SAMPLE_LAUNCH(QS_SRC_SV, QS_SAMPLE_CDF);
    } else {
        if (mode == QS_SAMPLE_SEQ) QS_SAMPLE_LAUNCH(QS_SRC_DM, QS_SAMPLE_SEQ);
        else                       QS_SAMPLE_LAUNCH(QS_SRC_DM, QS_SAMPLE_CDF);
    }
#undef QS_SAMPLE_LAUNCH
    QS_CHECK_LAUNCH("qs_sample");
    return QS_OK;
}

}  // namespace
}  // namespace qs

using namespace qs;

extern "C" size_t qs_reduce_ws_bytes(int) { return sizeof(double) * kReduceCtas; }

extern "C" int qs_prob0(const void* src, int n, int dtype, int src_kind, int bit, void* ws, size_t ws_bytes,
                        double* out_dev, void* stream) {
    int rc = check_src(src, n, dtype, src_kind);
    if (rc) return rc;
    QS_REQUIRE(bit >= 0 && bit < n, "bit %d outside [0, %d)", bit, n);
    QS_REQUIRE(out_dev != nullptr, "null output");
    if (ws == nullptr || ws_bytes < qs_reduce_ws_bytes(n)) {
        set_error("reduce workspace needs %zu bytes", qs_reduce_ws_bytes(n));
        return QS_EWORKSPACE;
    }
    if (dtype == QS_C128) return reduce_t<double2>(src, n, src_kind, bit, ws, out_dev, as_stream(stream));
    return reduce_t<float2>(src, n, src_kind, bit, ws, out_dev, as_stream(stream));
}

extern "C" int qs_norm2(const void* src, int n, int dtype, int src_kind, void* ws, size_t ws_bytes, double* out_dev,
                        void* stream) {
    int rc = check_src(src, n, dtype, src_kind);
    if (rc) return rc;
    QS_REQUIRE(out_dev != nullptr, "null output");
    if (ws == nullptr || ws_bytes < qs_reduce_ws_bytes(n)) {
        set_error("reduce workspace needs %zu bytes", qs_reduce_ws_bytes(n));
        return QS_EWORKSPACE;
    }
    if (dtype == QS_C128) return reduce_t<double2>(src, n, src_kind, -1, ws, out_dev, as_stream(stream));
    return reduce_t<float2>(src, n, src_kind, -1, ws, out_dev, as_stream(stream));
}

extern "C" int qs_collapse(void* vec, int n, int dtype, int bit, int outcome, double scale, void* stream) {
    int rc = check_src(vec, n, dtype, QS_SRC_SV);
    if (rc) return rc;
    QS_REQUIRE(bit >= 0 && bit < n, "bit %d outside [0, %d)", bit, n);
    QS_REQUIRE(outcome == 0 || outcome == 1, "outcome must be 0 or 1");
    uint64_t items = uint64_t(1) << (n - 1);
    unsigned grid = grid_for(items, kThreads * 4, 8);
    // Pairs for complex64 states beyond the L2's reach (2^23 amplitudes): 24 qubits
    // 39 - 49 us against 41 - 54 us (B200); below, and in complex128, the walk in
    // vector order is as fast or faster (20 qubits complex64 4.2 against 5.0 us; 26
    // qubits complex128, bit 0, 343 against 367 us, 24 qubits, bit 23, 70 against 75 us).
    const uint64_t N = 2 * items;
    const unsigned each = grid_for(N, kThreads * 4, 8);
    if (dtype == QS_C128) k_collapse_each<double2><<<each, kThreads, 0, as_stream(stream)>>>((double2*)vec, N, bit, outcome, scale);
    else if (n < 23)      k_collapse_each<float2><<<each, kThreads, 0, as_stream(stream)>>>((float2*)vec, N, bit, outcome, scale);
    else                  k_collapse<float2><<<grid, kThreads, 0, as_stream(stream)>>>((float2*)vec, items, bit, outcome, scale);
    QS_CHECK_LAUNCH("qs_collapse");
    return QS_OK;
}

extern "C" int qs_reset(void* vec, int n, int dtype, int bit, double p0, void* stream) {
    int rc = check_src(vec, n, dtype, QS_SRC_SV);
    if (rc) return rc;
    QS_REQUIRE(bit >= 0 && bit < n, "bit %d outside [0, %d)", bit, n);
    double alpha = sqrt(p0 > 0 ? p0 : 0.0);
    bool move = alpha < 1e-6;
    uint64_t items = uint64_t(1) << (n - 1);
    unsigned grid = grid_for(items, kThreads * 4, 8);
    // Bits 0 and 1 of complex64, whose pairs share a 32-byte sector: one pair in
    // flight (26 qubits, B200: 170 us, four 190 us).
    if (dtype == QS_C128) k_reset<double2, 4><<<grid, kThreads, 0, as_stream(stream)>>>((double2*)vec, items, bit, alpha, move);
    else if (bit < 2)     k_reset<float2, 1><<<grid, kThreads, 0, as_stream(stream)>>>((float2*)vec, items, bit, alpha, move);
    else                  k_reset<float2, 4><<<grid, kThreads, 0, as_stream(stream)>>>((float2*)vec, items, bit, alpha, move);
    QS_CHECK_LAUNCH("qs_reset");
    return QS_OK;
}

extern "C" size_t qs_sample_ws_bytes(int n) {
    const int bb = n < kBlockBits ? n : kBlockBits;
    return sizeof(double) * (size_t(2) << (n - bb));  // the levels take half of it and a bit
}

extern "C" int qs_sample_prepare(const void* src, int n, int dtype, int src_kind, void* ws, size_t ws_bytes,
                                 void* stream) {
    int rc = check_src(src, n, dtype, src_kind);
    if (rc) return rc;
    if (ws == nullptr || ws_bytes < qs_sample_ws_bytes(n)) {
        set_error("sample workspace needs %zu bytes", qs_sample_ws_bytes(n));
        return QS_EWORKSPACE;
    }
    if (dtype == QS_C128) return prepare_t<double2>(src, n, src_kind, (double*)ws, as_stream(stream));
    return prepare_t<float2>(src, n, src_kind, (double*)ws, as_stream(stream));
}

extern "C" int qs_sample(const void* src, int n, int dtype, int src_kind, const void* ws, size_t ws_bytes,
                         const double* u_dev, int64_t shots, int mode, int64_t* out_idx_dev, void* stream) {
    int rc = check_src(src, n, dtype, src_kind);
    if (rc) return rc;
    QS_REQUIRE(mode == QS_SAMPLE_CDF || mode == QS_SAMPLE_SEQ, "bad sample mode %d", mode);
    QS_REQUIRE(shots >= 0, "negative shot count");
    QS_REQUIRE(u_dev != nullptr && out_idx_dev != nullptr, "null uniforms or output");
    if (ws == nullptr || ws_bytes < qs_sample_ws_bytes(n)) {
        set_error("sample workspace needs %zu bytes", qs_sample_ws_bytes(n));
        return QS_EWORKSPACE;
    }
    if (shots == 0) return QS_OK;
    if (dtype == QS_C128)
        return sample_t<double2>(src, n, src_kind, (const double*)ws, u_dev, shots, mode, out_idx_dev, as_stream(stream));
    return sample_t<float2>(src, n, src_kind, (const double*)ws, u_dev, shots, mode, out_idx_dev, as_stream(stream));
}

extern "C" int qs_histogram(const int64_t* idx_dev, int64_t shots, int64_t* counts_dev, int64_t ncounts, void* stream) {
    QS_REQUIRE(shots >= 0 && ncounts >= 1, "bad sizes");
    QS_REQUIRE((shots == 0 || idx_dev != nullptr) && counts_dev != nullptr, "null pointer");
    if (shots == 0) return QS_OK;
    unsigned grid = grid_for(uint64_t(shots), 256, 4);
    k_hist<<<grid, 256, 0, as_stream(stream)>>>(idx_dev, shots, (unsigned long long*)counts_dev, ncounts);
    QS_CHECK_LAUNCH("qs_histogram");
    return QS_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free sampling.  The sum tree lives in a file-scope device array
// instead of a caller workspace, for callers that can only hand over the
// state, the uniforms and the output buffer (see include/qsim.h).
// ---------------------------------------------------------------------------
namespace {
constexpr int kNoAllocMaxQubits = QS_NOALLOC_SAMPLE_MAX_QUBITS;
constexpr size_t kNoAllocTreeDoubles = size_t(2) << (kNoAllocMaxQubits - kBlockBits);  // 1 MiB
}  // namespace

static __device__ __align__(256) double g_noalloc_tree[kNoAllocTreeDoubles];

namespace {
// Device address of g_noalloc_tree on the current device (the array's
// host-side name is not a device address).  It is looked up with that device
// current on every call made outside stream capture, so a context rebuilt
// after cudaDeviceReset gets its new address; inside a capture the address
// recorded by the last call outside one is used.
int noalloc_tree_ptr(cudaStream_t st, double** out) {
    static std::mutex mu;
    static double* addr[64] = {nullptr};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        set_error("qs_sample_noalloc: cudaGetDevice: %s", cudaGetErrorString(e));
        return QS_ECUDA;
    }
    QS_REQUIRE(dev >= 0 && dev < 64, "qs_sample_noalloc: device %d outside [0, 64)", dev);
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    e = cudaStreamIsCapturing(st, &cs);
    if (e != cudaSuccess) {
        set_error("qs_sample_noalloc: cudaStreamIsCapturing: %s", cudaGetErrorString(e));
        return QS_ECUDA;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (addr[dev] == nullptr || cs == cudaStreamCaptureStatusNone) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_tree);
        if (e != cudaSuccess || p == nullptr) {
            set_error("qs_sample_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
            return QS_ECUDA;
        }
        addr[dev] = static_cast<double*>(p);
    }
    *out = addr[dev];
    return QS_OK;
}
}  // namespace

extern "C" int qs_sample_noalloc(const void* src, int n, int dtype, int src_kind, const double* u_dev,
                                 int64_t shots, int mode, int64_t* out_idx_dev, void* stream) {
    int rc = check_src(src, n, dtype, src_kind);
    if (rc) return rc;
    if (n > kNoAllocMaxQubits) {
        set_error("qs_sample_noalloc: %d qubits exceed its fixed %d-qubit limit (a %zu-byte static sum tree); "
                  "use qs_sample_prepare/qs_sample with a workspace",
                  n, kNoAllocMaxQubits, sizeof(double) * kNoAllocTreeDoubles);
        return QS_EINVAL;
    }
    QS_REQUIRE(mode == QS_SAMPLE_CDF || mode == QS_SAMPLE_SEQ, "bad sample mode %d", mode);
    QS_REQUIRE(shots >= 0, "negative shot count");
    QS_REQUIRE(u_dev != nullptr && out_idx_dev != nullptr, "null uniforms or output");
    if (shots == 0) return QS_OK;
    cudaStream_t st = as_stream(stream);
    double* tree = nullptr;
    rc = noalloc_tree_ptr(st, &tree);
    if (rc) return rc;
    // every node the descent reads is written by the prepare step, so the
    // tree needs no clearing between calls
    if (dtype == QS_C128) {
        rc = prepare_t<double2>(src, n, src_kind, tree, st);
        return rc ? rc : sample_t<double2>(src, n, src_kind, tree, u_dev, shots, mode, out_idx_dev, st);
    }
    rc = prepare_t<float2>(src, n, src_kind, tree, st);
    return rc ? rc : sample_t<float2>(src, n, src_kind, tree, u_dev, shots, mode, out_idx_dev, st);
}
