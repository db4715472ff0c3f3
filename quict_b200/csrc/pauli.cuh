// Pauli sums, eight amplitudes at a time (observe.cu, batch.cuh).
//
// lam[j] = sum_t c_t (-1)^popc(z_t & src) psi[src], src = j ^ x_t.  A thread
// holds the amplitudes j | (u << 8), u = 0..7: a term's sign on them is its sign
// on j times (-1)^popc(m & u), m = the three bits of z_t at 8..10.  Terms of one
// X mask are added by m into eight sums (one parity per term for all eight
// amplitudes), and an 8-point Walsh transform turns those into the eight signed
// coefficient sums: per amplitude one parity an eighth of the terms instead of
// every term.  No unit is saturated: issue 58 % of its slots, the unit of the
// FP64 conversions and bit counts (XU) 44 %, ALU 42 % at 25 qubits, 31 terms
// (888 us); three CTAs an SM (76 registers) wait on dependent instructions.
#pragma once

#include "common.cuh"

namespace qs {
namespace {

constexpr int kPauliShift = 8, kPauliU = 8;
constexpr uint64_t kPauliChunk = uint64_t(kPauliU) << kPauliShift;  // 2048 amplitudes
constexpr uint64_t kPauliMask = uint64_t(kPauliU - 1) << kPauliShift;

// Order of the terms: by X mask, then by the three bits of the Z mask.
inline bool pauli_before(uint64_t x1, uint64_t z1, uint64_t x2, uint64_t z2) {
    return x1 != x2 ? x1 < x2 : (z1 & kPauliMask) < (z2 & kPauliMask);
}

__device__ __forceinline__ void walsh8(double (&w)[kPauliU]) {
#pragma unroll
    for (int h = 1; h < kPauliU; h <<= 1)
#pragma unroll
        for (int i = 0; i < kPauliU; ++i)
            if (!(i & h)) {
                const double a = w[i], b = w[i + h];
                w[i] = a + b;
                w[i + h] = a - b;
            }
}

// T: x(t), z(t), re(t), im(t) of terms in pauli_before order.  load(i): psi[i].
// base: amplitude index with bits 8..10 clear.  CPLX: some coefficient has an
// imaginary part.
template <bool CPLX, typename T, typename L>
__device__ __forceinline__ void pauli8(const T& tm, int nterms, uint64_t base, const L& load, double (&re)[kPauliU],
                                       double (&im)[kPauliU]) {
#pragma unroll
    for (int u = 0; u < kPauliU; ++u) re[u] = im[u] = 0.0;
    int t = 0;
    while (t < nterms) {
        const uint64_t x = tm.x(t);
        const uint32_t xm = uint32_t((x & kPauliMask) >> kPauliShift);
        const uint64_t src = base ^ (x & ~kPauliMask);
        double w[kPauliU], wi[kPauliU];
        bool flat = true;
#pragma unroll
        for (int m = 0; m < kPauliU; ++m) {
            w[m] = 0.0;
            if (CPLX) wi[m] = 0.0;
            // the transform gives the sums at the source index u ^ xm
            const bool twist = __popc(uint32_t(m) & xm) & 1;
            while (t < nterms && tm.x(t) == x && ((tm.z(t) & kPauliMask) >> kPauliShift) == uint64_t(m)) {
                const bool neg = ((__popcll(tm.z(t) & src) & 1) != 0) != twist;
                w[m] += neg ? -tm.re(t) : tm.re(t);
                if (CPLX) wi[m] += neg ? -tm.im(t) : tm.im(t);
                if (m) flat = false;
                ++t;
            }
        }
        if (flat) {  // no term tells the eight amplitudes apart
#pragma unroll
            for (int m = 1; m < kPauliU; ++m) {
                w[m] = w[0];
                if (CPLX) wi[m] = wi[0];
            }
        } else {
            walsh8(w);
            if (CPLX) walsh8(wi);
        }
#pragma unroll
        for (int u = 0; u < kPauliU; ++u) {
            const auto a = load(src | (uint64_t(uint32_t(u) ^ xm) << kPauliShift));
            const double ar = double(a.x), ai = double(a.y);
            re[u] = fma(w[u], ar, re[u]);
            im[u] = fma(w[u], ai, im[u]);
            if (CPLX) {
                re[u] = fma(-wi[u], ai, re[u]);
                im[u] = fma(wi[u], ar, im[u]);
            }
        }
    }
}

}  // namespace
}  // namespace qs
