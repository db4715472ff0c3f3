// Dense gates on 5 to 10 qubits as tiled matrix products.  In a translation unit
// of their own: compiled together with the one- and two-qubit kernels they
// changed those (a complex64 gate on bit 2 of 26 qubits took 215 us instead of
// 182 on B200, with the same registers).
#include "common.cuh"
#include "kq_tiles.h"

namespace qs {
namespace {

constexpr int kMaxIns = 48;
using Plan = InsertPlan<kMaxIns>;

Plan make_plan(uint64_t mask) {
    Plan p; p.nb = 0;
    for (int b = 0; b < 64; ++b)
        if ((mask >> b) & 1) p.b[p.nb++] = b;
    return p;
}

// The gate as a matrix product: a CTA gathers G groups of 2^K amplitudes into
// shared memory (columns), multiplies them by the matrix, which it reads in
// tiles of BK columns, and scatters them back.  A thread accumulates TM x TG
// outputs, rows and columns strided so that the shared-memory reads of a warp
// are contiguous; the sums run over the matrix columns in order: 16 outputs per
// thread and step take 8 shared loads for 64 multiply-adds.  Each matrix entry is
// read once per G groups (one CTA per group, one row per thread and strided
// matrix reads before: 6-qubit gate on 20 qubits, complex128, 325 us, now 53 us).
// Bound by latency: at 24 qubits (827 us) the FP64 pipe is 30 % active, one CTA
// of 8 warps an SM (132 registers a thread) waits for each tile of the matrix.
// With few groups k_kq_one (sv_gates.cu) is faster.
// The gather walks the target bits and the lowest free bits together in
// ascending vector order, so global accesses are as contiguous as the bits
// allow; column G pads the rows against bank conflicts.
struct KqMap {
    int nbits, gbits;      // bits of a tile; of them group bits
    uint8_t pos[20];       // vector bit, ascending
    int32_t at[20];        // its step in the shared tile
};

template <typename V, int K, int G, int THREADS, int TM, int TG, int BK>
__global__ void __launch_bounds__(THREADS)
k_kq_tile(V* __restrict__ v, uint64_t tiles, Plan plan, uint64_t cmask, const __grid_constant__ KqMap map,
          const double2* __restrict__ M) {
    constexpr int D = 1 << K, GP = G + 1, DP = D + 1;
    constexpr int RT = D / TM, CT = G / TG;
    static_assert(RT * CT == THREADS, "one thread per TM x TG outputs");
    constexpr int LT = THREADS == 512 ? 9 : THREADS == 256 ? 8 : 7;
    static_assert((1 << LT) == THREADS, "threads");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V* X = reinterpret_cast<V*>(smem_raw);  // [D][GP]
    V* A = X + D * GP;                      // [BK][DP]
    const int tid = threadIdx.x, tx = tid % CT, ty = tid / CT;
    uint64_t toff = 0;
    int tat = 0;
    for (int i = 0; i < LT && i < map.nbits; ++i)
        if ((tid >> i) & 1) {
            toff |= uint64_t(1) << map.pos[i];
            tat += map.at[i];
        }
    const int steps = map.nbits > LT ? 1 << (map.nbits - LT) : 1;
    const bool moves = map.nbits >= LT || tid < (1 << map.nbits);
    auto part = [&](int i, uint64_t& off, int& at) {
        off = toff;
        at = tat;
        for (int b = 0; b < map.nbits - LT; ++b)
            if ((i >> b) & 1) {
                off |= uint64_t(1) << map.pos[LT + b];
                at += map.at[LT + b];
            }
    };
    if ((1 << map.gbits) < G)  // fewer groups than columns: the others stay 0
        for (int i = tid; i < D * GP; i += THREADS) X[i] = mk<V>(0.0, 0.0);
    for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint64_t base = expand(t << map.gbits, plan) | cmask;
        __syncthreads();
        if (moves)
            for (int i = 0; i < steps; ++i) {
                uint64_t off;
                int at;
                part(i, off, at);
                X[at] = v[base | off];
            }
        V acc[TM][TG];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TG; ++j) acc[i][j] = mk<V>(0.0, 0.0);
        for (int c0 = 0; c0 < D; c0 += BK) {
            __syncthreads();
            for (int e = tid; e < D * BK; e += THREADS) {
                const int r = e / BK, c = e % BK;
                const double2 m = __ldg(&M[r * D + c0 + c]);
                A[c * DP + r] = mk<V>(m.x, m.y);
            }
            __syncthreads();
#pragma unroll
            for (int c = 0; c < BK; ++c) {
                V a[TM], x[TG];
#pragma unroll
                for (int i = 0; i < TM; ++i) a[i] = A[c * DP + i * RT + ty];
#pragma unroll
                for (int j = 0; j < TG; ++j) x[j] = X[(c0 + c) * GP + j * CT + tx];
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TG; ++j) acc[i][j] = cfma(a[i], x[j], acc[i][j]);
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TG; ++j) X[(i * RT + ty) * GP + j * CT + tx] = acc[i][j];
        __syncthreads();
        if (moves)
            for (int i = 0; i < steps; ++i) {
                uint64_t off;
                int at;
                part(i, off, at);
                v[base | off] = X[at];
            }
    }
}

template <typename V, int K, int G, int THREADS, int TM, int TG, int BK>
int launch_kq(V* v, int n, const int32_t* bits, uint64_t cmask, uint64_t tmask, const double2* M, cudaStream_t st) {
    constexpr int lg = G == 128 ? 7 : G == 64 ? 6 : G == 32 ? 5 : G == 16 ? 4 : 3;
    static_assert((1 << lg) == G, "G");
    const uint64_t fixed = cmask | tmask;
    const int free_bits = n - __builtin_popcountll(fixed);
    // Fewer wide tiles than SMs: narrow tiles of 8 columns spread the groups
    // over more SMs, at more matrix reads per group.
    if constexpr (G > 8)
        if ((uint64_t(1) << free_bits) / G < uint64_t(sm_count()))
            return launch_kq<V, K, 8, 128, (1 << K) / 16, 1, 8>(v, n, bits, cmask, tmask, M, st);
    KqMap map{};
    map.gbits = lg < free_bits ? lg : free_bits;
    int g = 0;
    for (int b = 0; b < n; ++b) {
        int step = -1;
        if ((tmask >> b) & 1) {
            for (int t = 0; t < K; ++t)
                if (bits[t] == b) step = (1 << (K - 1 - t)) * (G + 1);
        } else if (!((cmask >> b) & 1) && g < map.gbits) {
            step = 1 << g++;
        }
        if (step < 0) continue;
        map.pos[map.nbits] = uint8_t(b);
        map.at[map.nbits++] = step;
    }
    const Plan p = make_plan(fixed);
    const uint64_t tiles = uint64_t(1) << (free_bits - map.gbits);
    const size_t smem = sizeof(V) * (size_t(1 << K) * (G + 1) + size_t(BK) * ((1 << K) + 1));
    auto* fn = k_kq_tile<V, K, G, THREADS, TM, TG, BK>;
    // per call: the attribute belongs to the device, and costs nothing beside the launch
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) {
        set_error("qs_apply_kq: %s", cudaGetErrorString(e));
        return QS_ECUDA;
    }
    fn<<<grid_for(tiles, 1, smem > 110 * 1024 ? 1 : smem > 72 * 1024 ? 2 : 3), THREADS, smem, st>>>(v, tiles, p, cmask,
                                                                                                    map, M);
    QS_CHECK_LAUNCH("qs_apply_kq(tile)");
    return QS_OK;
}

template <typename V>
int apply_tiles(V* v, int n, int k, const int32_t* bits, uint64_t cmask, uint64_t tmask, const double2* M, cudaStream_t st) {
    switch (k) {
        case 5: return launch_kq<V, 5, 128, 256, 4, 4, 8>(v, n, bits, cmask, tmask, M, st);
        case 6: return launch_kq<V, 6, 64, 256, 4, 4, 8>(v, n, bits, cmask, tmask, M, st);
        case 7: return launch_kq<V, 7, 32, 256, 4, 4, 8>(v, n, bits, cmask, tmask, M, st);
        case 8: return launch_kq<V, 8, 16, 256, 4, 4, 8>(v, n, bits, cmask, tmask, M, st);
        case 9: return launch_kq<V, 9, 8, 256, 8, 2, 4>(v, n, bits, cmask, tmask, M, st);
        default: return launch_kq<V, 10, 8, 512, 8, 2, 4>(v, n, bits, cmask, tmask, M, st);
    }
}

}  // namespace

int apply_kq_tiles(int dtype, void* vec, int n, int k, const int32_t* bits, uint64_t cmask, uint64_t tmask,
                   const double2* M, cudaStream_t st) {
    return dtype == QS_C128 ? apply_tiles(static_cast<double2*>(vec), n, k, bits, cmask, tmask, M, st)
                            : apply_tiles(static_cast<float2*>(vec), n, k, bits, cmask, tmask, M, st);
}

}  // namespace qs
