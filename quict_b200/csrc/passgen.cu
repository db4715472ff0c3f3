// Run-time compiled passes: the source generator.
//
// A register pass planned by build_reg can also run as a kernel generated for
// it alone: every op, slot mask, control and relayout address is a constant
// of the generated code, so there is no per-op dispatch, plain exchanges
// (X, CX, SWAP without outside controls) become register renamings, zero and
// unit matrix entries drop out of the arithmetic, and the matrices are read
// as constant-bank operands from the launch's parameter block.  The source
// depends on the pass's structure and on which matrix entries are exactly
// 0, 1 or -1, not on the other matrix values, so passes of the same shape
// share one compiled kernel (jit.cu caches by source text).
#include <algorithm>
#include <array>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "common.cuh"
#include "passgen.h"
#include "regtile.cuh"

namespace qs {

bool jit_single_buffer(bool c128, bool tables) {
    static const int env = [] {
        const char* e = getenv("QS_JIT_SINGLE_BUFFER");
        return e && (*e == '0' || *e == '1') ? *e - '0' : -1;
    }();
    return env >= 0 ? env == 1 : c128 || tables;
}

namespace {

constexpr size_t kJitMaxParamBytes = 32000;  // below the 32764-byte kernel parameter limit

struct SrcBuf {
    std::string s;
    bool truncated = false;  // a formatted piece did not fit: the source is not used
    void add(const char* fmt, ...) __attribute__((format(printf, 2, 3))) {
        char tmp[1024];
        va_list ap;
        va_start(ap, fmt);
        int k = vsnprintf(tmp, sizeof(tmp), fmt, ap);
        va_end(ap);
        if (k >= int(sizeof(tmp))) {
            truncated = true;
            k = int(sizeof(tmp)) - 1;
        }
        s.append(tmp, size_t(k));
    }
};

// XOR of per-thread-bit images over the set bits of threadIdx.x, as an expression
std::string thread_xor_expr(const uint32_t* img, int nT) {
    std::string e;
    for (int i = 0; i < nT; ++i) {
        if (!img[i]) continue;
        char t[64];
        snprintf(t, sizeof(t), "%s(((tid >> %d) & 1u) * %uu)", e.empty() ? "" : " ^ ", i, img[i]);
        e += t;
    }
    return e.empty() ? std::string("0u") : e;
}

// ---------------------------------------------------------------- normalised matrices
// What bounds a pass over a large state is its multiply-add count, and most of
// its dense matrices are known only up to factors that need not be applied
// where they stand.  A dense matrix U is written as U = s (D_1 x D_2) U' with a
// scalar s and a diagonal D_i = diag(1, d_i) per target bit, chosen so that the
// diagonal entries of U' are exactly 1 (row r's factor is s times the d_i of
// its set index bits): an entry 1 costs nothing where a general one costs four
// instructions per amplitude, a real or imaginary one two.
//   - s commutes with everything: the scalars are multiplied into the next
//     diagonal that is general anyway (at no cost), or those of 8 ops
//     (complex128: 30) and what is left at the end into the op among them whose
//     cost grows least.
//   - D_i moves forward along its bit (through diagonals and controls, across
//     plain exchanges) into the next uncontrolled op on that bit; d_i = 1 when
//     no op takes it.
// The factors are products and quotients in extended precision (64 significand
// bits), rounded once into the parameter block: a coefficient changes by that
// rounding, or by its matrix's own where two entries are the same number (see
// same).  Row and scalar factors leave every product's
// relative rounding error as it is; only the range grows.  run() sums the
// factors' logarithms over the launch, and a launch whose amplitudes could leave
// the allowed range keeps its own matrices.
// Which entry becomes 1, the class of every other one and where the scalars go
// follow from the classes of the matrices' own entries, not from their sizes:
// new parameters of a circuit reuse its compiled kernels (a limit on the sum of
// the scalars decided op by op gave 4 to 6 kernels of one complex64 pass in 12
// parameter sets).  8 ops per carrier: the range holds as long as the scalars
// average above 2^-7.5, also when a layer repeats one angle; 30-qubit circuit,
// complex64, 4 / 8 / 16 / all ops of the launch: 2582 / 2557 / 2552 / 2552
// multiply-adds per amplitude.  complex128, 30 ops: no scalar is below 2^-20, so
// theirs never exceed the range; 2630, all ops 2630.
// 30-qubit spread circuit of 1000 gates at k = 12: 3284 -> 2630 multiply-adds
// per amplitude in complex128, 3158 -> 2557 in complex64 (B200, when this came
// in: 318.3 -> 276.3 and 202.4 -> 179.0 ms; now 264.4 and 140.8 ms).  The host
// takes 20 to 50 us a pass to make a parameter block with or without it.
// Per-instance tables and adjoint passes keep their matrices.
#pragma nv_diag_suppress 20208  // long double: host code only here
using Ld = long double;

// 0, 1, -1, general (3), real (4), imaginary (5)
template <typename T>
int value_class(T x, T y) {
    if (y == 0) return x == 0 ? 0 : x == 1 ? 1 : x == -1 ? 2 : 4;
    return x == 0 ? 5 : 3;
}

// A matrix entry, its class (what the generated code may assume about it) and
// the size of the rounding it came with: half a unit in the last place of its
// matrix's largest component.
struct Entry {
    Ld re, im;
    double err;
    int cl;
    Ld size() const { return std::max(std::abs(re), std::abs(im)); }
};
inline bool is_real(int cl) { return cl == 1 || cl == 2 || cl == 4; }
constexpr Entry kOne{1, 0, 0, 1};

int mul_class(int a, int b) {
    if (a == 0 || b == 0) return 0;
    if (a == 1 || b == 1) return a == 1 ? b : a;
    if (a == 2 && b == 2) return 1;
    if (a == 3 || b == 3) return 3;
    return is_real(a) == is_real(b) ? 4 : 5;
}
// an entry times a factor
Entry mul(const Entry& a, const Entry& f) {
    const int cl = mul_class(a.cl, f.cl);
    const double err = a.err == 0 ? 0 : a.err * double(f.size());
    if (cl == 0) return {0, 0, err, 0};
    if (is_real(f.cl)) return {a.re * f.re, a.im * f.re, err, cl};
    if (is_real(a.cl)) return {a.re * f.re, a.re * f.im, err, cl};
    return {a.re * f.re - a.im * f.im, a.re * f.im + a.im * f.re, err, cl};
}
// Two components that are the same number, or the same up to its sign (-1):
// merged matrices hold such pairs as sums rounded in different orders.  Each
// component is compared by itself (that of an angle of 2 pi, next to 0, counts),
// and a pair taken for equal changes its matrix by no more than the roundings it
// came with.
int same(Ld x, Ld u, Ld err) {
    const Ld d = std::abs(std::abs(x) - std::abs(u));
    if (!(d == 0 || (d <= err && d <= 0x1p-44L * std::abs(u) && x != 0))) return 0;
    return (x < 0) == (u < 0) ? 1 : -1;
}
// i^k with a = i^k b, or -1
int quarter_turns(const Entry& a, const Entry& b) {
    const Ld err = Ld(a.err) + Ld(b.err);
    int r = same(a.re, b.re, err), i = r ? same(a.im, b.im, err) : 0;
    if (r && i) {
        if (a.re == 0) return i == 1 ? 0 : 2;
        if (r == i || a.im == 0) return r == 1 ? 0 : 2;
    }
    r = same(a.re, b.im, err);
    i = r ? same(a.im, b.re, err) : 0;
    if (!r || !i) return -1;
    if (a.re == 0) return i == 1 ? 1 : 3;  // i times a real number
    if (a.im == 0) return r == 1 ? 3 : 1;
    return r != i ? (i == 1 ? 1 : 3) : -1;
}
// Class of a / b for two general entries: real or imaginary when they lie on one
// line through 0, or at a right angle (a row of real numbers times a phase), up
// to the same roundings; each product of components counts by itself.
int axis(const Entry& a, const Entry& b) {
    const Ld err = a.err * b.size() + b.err * a.size();
    const auto near = [err](Ld p, Ld q) {
        const Ld d = std::abs(p - q);
        return d <= err && d <= 0x1p-44L * std::abs(p);
    };
    if (near(a.im * b.re, a.re * b.im)) return 4;
    return near(a.re * b.re, -a.im * b.im) ? 5 : 3;
}
// class of a / b
int div_class(const Entry& a, const Entry& b, int* turns = nullptr) {
    if (a.cl == 0) return 0;
    const int t = quarter_turns(a, b);
    if (turns) *turns = t;
    if (t >= 0) return t == 0 ? 1 : t == 2 ? 2 : 5;
    if (b.cl == 1 || b.cl == 2) return a.cl;
    if (a.cl == 3 && b.cl == 3) return axis(a, b);
    if (a.cl == 3 || b.cl == 3) return 3;
    return is_real(a.cl) == is_real(b.cl) ? 4 : 5;
}
Entry div(const Entry& a, const Entry& b) {  // (a factor, or a final entry: err 0)
    int t = -1;
    const int cl = div_class(a, b, &t);
    if (cl == 0) return {0, 0, 0, 0};
    if (t >= 0) return {Ld(t == 0 ? 1 : t == 2 ? -1 : 0), Ld(t == 1 ? 1 : t == 3 ? -1 : 0), 0, cl};
    if (is_real(b.cl)) return {a.re / b.re, a.im / b.re, 0, cl};
    if (b.cl == 5) return {a.im / b.im, -a.re / b.im, 0, cl};
    const Ld q = 1 / (b.re * b.re + b.im * b.im);
    return {cl == 5 ? 0 : (a.re * b.re + a.im * b.im) * q, cl == 4 ? 0 : (a.im * b.re - a.re * b.im) * q, 0, cl};
}
double log2_abs(const Entry& e) { return 0.5 * std::log2(double(e.re * e.re + e.im * e.im)); }

// Instructions per amplitude of one row: the first term may be a unit entry
// (taken as is), which the generated code puts first.
struct RowCost {
    int c = 0;
    bool unit = false;
    void add(int cl) {
        if (cl == 0) return;
        if (cl <= 2) unit = true;
        c += cl == 3 ? 4 : 2;
    }
    int total() const { return unit ? c - 2 : c; }
};

template <typename V>
struct Normaliser {
    const RegArgs& a;
    V* const pm;                 // the block's matrices, in slot order
    std::vector<uint8_t>& ncls;  // and the classes of their entries
    // log2 bounds on how far the factors may raise (up) and lower (down) the
    // amplitudes between the launch's load and its store; bound on the largest
    // entry of a matrix and its inverse; ops whose scalars one carrier takes
    static constexpr bool C128 = sizeof(V) == 16;
    static constexpr double max_up = C128 ? 600 : 60, max_down = C128 ? 300 : 40;
    static constexpr Ld max_entry = C128 ? 0x1p700L : 0x1p80L;
    static constexpr int per_scalar = C128 ? 30 : 8;

    std::unique_ptr<Entry[]> store;
    std::vector<uint8_t> state;  // per op: 0 not loaded, 1 loaded, 2 changed
    std::vector<int> stage;      // per op
    Entry total = kOne;          // scalars taken out and not yet put back
    std::vector<Entry> late;     // those that appear at an op
    // log2 changes at each op of the state's scalar, and of the most and the
    // least that the factors under way make of it
    std::vector<double> scalar, high, low;

    Normaliser(const RegArgs& a_, V* pm_, std::vector<uint8_t>& ncls_)
        : a(a_), pm(pm_), ncls(ncls_), store(new Entry[ncls_.size()]), state(size_t(a_.nops), 0),
          stage(size_t(a_.nops), 0), late(size_t(a_.nops), kOne), scalar(size_t(a_.nops), 0.0),
          high(size_t(a_.nops), 0.0), low(size_t(a_.nops), 0.0) {
        for (int si = 0; si < a.nstages; ++si)
            for (int o = 0; o < a.st[si].op_count; ++o) stage[size_t(a.st[si].op_begin + o)] = si;
    }

    int count(int o) const { return a.cp[o].diag ? 1 << a.cp[o].m : 1 << (2 * a.cp[o].m); }
    int dim(int o) const { return 1 << a.cp[o].m; }
    // op o's matrix (MAT: row-major D x D; DIAG: 2^m entries)
    Entry* mat(int o) {
        Entry* const e = store.get() + a.cp[o].soff;
        if (state[size_t(o)]) return e;
        state[size_t(o)] = 1;
        const V* z = pm + a.cp[o].soff;
        double top = 0;
        const int cnt = count(o);
        for (int i = 0; i < cnt; ++i) top = std::max(top, double(std::max(std::abs(z[i].x), std::abs(z[i].y))));
        for (int i = 0; i < cnt; ++i) e[i] = {z[i].x, z[i].y, 0x1p-53 * top, value_class(z[i].x, z[i].y)};
        return e;
    }
    static bool controlled(const KOp& op) { return op.scm || op.tctrl || op.gctrl; }
    // index bit of tile bit b among op o's targets, or -1
    int index_bit(int o, int b) const {
        const KOp& op = a.ops[o];
        const KStage& S = a.st[stage[size_t(o)]];
        int i = 0;
        for (int j = 0; j < 6; ++j) {
            if (!((op.mask >> j) & 1)) continue;
            if (S.R[j] == b) return i;
            ++i;
        }
        if (op.code == QS_OP_DIAG)
            for (int q = 0; q < op.nh; ++q)
                if (op.hsrc[q] == b) return op.ns + (op.nh - 1 - q);
        return -1;
    }
    // a diagonal whose every entry is multiplied anyway takes factors for free
    bool free_diag(int o) {
        const KOp& op = a.ops[o];
        if (op.code != QS_OP_DIAG || controlled(op)) return false;
        if (op.nh > 0) return true;
        const Entry* v = mat(o);
        for (int i = 0; i < count(o); ++i)
            if (v[i].cl != 3) return false;
        return true;
    }
    // The op that takes a factor diag(1, d) of tile bit b from op o, the bit it
    // then sits on, and whether an odd number of exchanges inverts it; -1: none.
    int taker(int o, int b, int* bit, bool* inverted) {
        *inverted = false;
        for (int p = o + 1; p < a.nops; ++p) {
            const KOp& op = a.ops[p];
            const int ib = index_bit(p, b);
            if (ib < 0) continue;
            if (op.code == QS_OP_DIAG) {
                if (!free_diag(p)) continue;
            } else if (controlled(op)) {
                return -1;
            } else if (op.code == QS_OP_ANTI) {
                *inverted = !*inverted;
                continue;
            } else if (op.code == QS_OP_SWAP) {
                const KStage& S = a.st[stage[size_t(p)]];
                const int b0 = S.R[nth_bit(op.mask, 0)], b1 = S.R[nth_bit(op.mask, 1)];
                b = b == b0 ? b1 : b0;
                continue;
            } else if (op.code != QS_OP_MAT) {
                return -1;
            }
            *bit = b;
            return p;
        }
        return -1;
    }
    // m[p] <- m[p] diag(1, d) on index bit ib (columns; entries of a diagonal)
    void take(int p, int ib, const Entry& d) {
        Entry* v = mat(p);
        state[size_t(p)] = 2;
        const int D = dim(p);
        for (int e = 0; e < count(p); ++e)
            if (((e & (D - 1)) >> ib) & 1) v[e] = mul(v[e], d);
    }
    // instructions that a dense op costs more, over its rows, once it has taken
    // diag(1, d) on index bit ib: as it stands (more than two bits) or with its
    // rows scaled by their diagonal entries afterwards (an estimate)
    int take_cost(int p, int ib, const Entry& d) {
        const Entry* v = mat(p);
        const int D = dim(p);
        int cost = 0;
        for (int r = 0; r < D; ++r) {
            const Entry z = v[r * D + r], zd = ((r >> ib) & 1) && D <= 4 ? mul(z, d) : z;
            RowCost before, after;
            for (int c = 0; c < D; ++c) {
                const Entry& e = v[r * D + c];
                const bool taken = (c >> ib) & 1;
                if (D > 4 || z.cl == 0) {
                    before.add(e.cl);
                    after.add(taken ? mul_class(e.cl, d.cl) : e.cl);
                } else {
                    before.add(div_class(e, z));
                    after.add(div_class(taken ? mul(e, d) : e, zd));
                }
            }
            cost += after.total() - before.total();
        }
        return cost;
    }

    // Take factors out of every uncontrolled dense op on one or two bits.  False
    // (and nothing is changed): the range would be exceeded.
    bool run() {
        int begin = 0, taken = 0;  // of the scalars in `total`
        const auto put_back = [&](int o) {
            scalar[size_t(o)] += log2_abs(total);
            Entry* v = mat(o);
            state[size_t(o)] = 2;
            for (int e = 0; e < count(o); ++e) v[e] = mul(v[e], total);
            total = kOne;
            taken = 0;
        };
        for (int o = 0; o < a.nops; ++o) {
            total = mul(total, late[size_t(o)]);
            if (free_diag(o)) {
                if (total.cl != 1) put_back(o);
                begin = o;  // it can take the next ones as well, at no cost
            }
            if (take_out(o) && ++taken == per_scalar) {
                put_back(carrier(begin, o));
                begin = o + 1;
            }
        }
        if (total.cl != 1) put_back(carrier(begin, a.nops - 1));
        double c = 0, h = 0, l = 0;
        for (int o = 0; o < a.nops; ++o) {
            c += scalar[size_t(o)];
            h += high[size_t(o)];
            l += low[size_t(o)];
            // (written so that a value that is not finite is refused)
            if (!(c + h <= max_up && c + l >= -max_down)) return false;
            if (state[size_t(o)] != 2) continue;
            Ld top = 0;
            const Entry* v = mat(o);
            for (int e = 0; e < count(o); ++e) top = std::max(top, v[e].size());
            if (!(top <= max_entry && (top == 0 || top >= 1 / max_entry))) return false;
        }
        for (int o = 0; o < a.nops; ++o) {
            if (state[size_t(o)] != 2) continue;
            const Entry* v = mat(o);
            const size_t at = a.cp[o].soff;
            for (int e = 0; e < count(o); ++e) {
                pm[at + size_t(e)].x = decltype(V::x)(v[e].re);
                pm[at + size_t(e)].y = decltype(V::y)(v[e].im);
                ncls[at + size_t(e)] = uint8_t(v[e].cl);
            }
        }
        return true;
    }
    // The op of [begin, end] that takes the scalars: the one whose cost grows
    // least, the last of those.
    int carrier(int begin, int end) {
        int best = end;
        double least = 1e300;
        for (int o = end; o >= begin && least > 0; --o) {
            const KOp& op = a.ops[o];
            if (controlled(op) || (op.code != QS_OP_MAT && op.code != QS_OP_DIAG)) continue;
            const Entry* v = mat(o);
            const int D = dim(o), cnt = count(o);
            int more = 0;
            if (op.code == QS_OP_DIAG) {
                if (op.nh == 0)
                    for (int e = 0; e < cnt; ++e) more += diag_cost(mul_class(v[e].cl, total.cl)) - diag_cost(v[e].cl);
            } else {
                for (int r = 0; r < D; ++r) {
                    RowCost before, after;
                    for (int i = 0; i < D; ++i) {
                        before.add(v[r * D + i].cl);
                        after.add(mul_class(v[r * D + i].cl, total.cl));
                    }
                    more += after.total() - before.total();
                }
            }
            if (double(more) / D < least) {
                least = double(more) / D;
                best = o;
            }
        }
        return best;
    }
    static int diag_cost(int cl) { return cl == 1 ? 0 : cl == 3 ? 4 : 2; }

    // Op o's factors, if taking them out gains.
    bool take_out(int o) {
        const KOp& op = a.ops[o];
        const int M = a.cp[o].m, D = 1 << M;
        if (op.code != QS_OP_MAT || controlled(op) || M > 2) return false;
        Entry* const u = mat(o);
        const Entry s = u[0];
        Ld top = 0;
        int plain = 0;
        for (int r = 0; r < D; ++r) {
            RowCost row;
            for (int c = 0; c < D; ++c) {
                top = std::max(top, u[r * D + c].size());
                row.add(u[r * D + c].cl);
            }
            plain += row.total();
        }
        if (!usable(s, top)) return false;
        int own = 0;  // index bits whose d_i is taken out
        int best_cost = rows_cost(u, M, own);
        if (best_cost >= plain) return false;
        Entry d[2] = {kOne, kOne};
        int to[2] = {-1, -1}, tob[2] = {0, 0};
        bool inv[2] = {false, false};
        for (int i = 0; i < M; ++i) {
            const Entry& z = u[(1 << i) * D + (1 << i)];
            if (!usable(z, top)) continue;
            const Entry di = div(z, s);
            if (di.cl == 1) continue;
            bool iv = false;
            int bit = 0;
            const int p = taker(o, a.st[stage[size_t(o)]].R[nth_bit(op.mask, i)], &bit, &iv);
            if (p < 0) continue;
            // per amplitude: this op gains, a dense taker may lose
            const int cost = rows_cost(u, M, own | (1 << i));
            double gain = double(best_cost - cost) / D;
            if (gain > 0 && a.ops[p].code != QS_OP_DIAG) gain -= double(take_cost(p, index_bit(p, bit), di)) / dim(p);
            if (gain <= 0) continue;
            own |= 1 << i;
            best_cost = cost;
            d[i] = di;
            to[i] = p;
            tob[i] = bit;
            inv[i] = iv;
        }
        scale_rows(u, M, own);
        state[size_t(o)] = 2;
        total = mul(total, s);
        scalar[size_t(o)] -= log2_abs(s);
        for (int i = 0; i < M; ++i) {
            if (to[i] < 0) continue;
            Entry f = d[i];
            const size_t p = size_t(to[i]);
            const double ld = log2_abs(f);
            high[size_t(o)] += std::max(0.0, -ld);
            high[p] -= std::max(0.0, -ld);
            low[size_t(o)] += std::min(0.0, -ld);
            low[p] -= std::min(0.0, -ld);
            if (inv[i]) {  // X diag(1, d) = d diag(1, 1/d) X: the scalar is there once the factor is taken
                late[p] = mul(late[p], f);
                scalar[p] -= ld;
                f = div(kOne, f);
            }
            take(to[i], index_bit(to[i], tob[i]), f);
        }
        return true;
    }
    // a factor that is neither zero nor far below the matrix's largest entry
    // (then the matrix keeps its own form)
    static bool usable(const Entry& z, Ld top) {
        const Ld r = z.size();
        return r > top * 0x1p-20L && r >= 0x1p-20L && r <= 0x1p20L;
    }
    // Row r's factor when the index bits of `own` have theirs taken out: s times
    // the d_i of r's set bits in `own`, d_i = u_ii / s (so one such bit: u_ii
    // itself).
    static Entry row_factor(const Entry* u, int M, int own, int r) {
        const int D = 1 << M, w = r & own;
        if (w == 3) return mul(u[D + 1], div(u[2 * D + 2], u[0]));
        return u[w * D + w];
    }
    static int rows_cost(const Entry* u, int M, int own) {
        const int D = 1 << M;
        int cost = 0;
        for (int r = 0; r < D; ++r) {
            const Entry f = row_factor(u, M, own, r);
            RowCost row;
            for (int c = 0; c < D; ++c) row.add(div_class(u[r * D + c], f));
            cost += row.total();
        }
        return cost;
    }
    static void scale_rows(Entry* u, int M, int own) {
        const int D = 1 << M;
        Entry f[4];
        for (int r = 0; r < D; ++r) f[r] = row_factor(u, M, own, r);
        for (int r = 0; r < D; ++r)
            for (int c = 0; c < D; ++c) u[r * D + c] = div(u[r * D + c], f[r]);
    }
};

// devfn != nullptr: emit the pass as `extern "C" __device__ void <devfn>(vec,
// params, mats, partials, tile, tend, zero_in)` for the persistent batch
// kernel instead of a kernel: it runs tiles [tile, tend) of the calling CTA,
// reads its parameter block from global memory (params), may run in a CTA
// wider than its own thread count (the other threads share the loads, repeat
// the register work of thread tid mod threads, and store nothing), and with
// zero_in != 0 reads |0...0> instead of the vector.
template <typename V>
bool gen_reg_pass(const RegArgs& a, int R, const V* hm, JitPass& out, bool with_source = true,
                  const char* devfn = nullptr) {
    constexpr bool C128 = sizeof(V) == 16;
    const int E = 1 << R, nT = a.nT, K = a.K, L = a.L, H = a.H;
    const int threads = 1 << nT, nwarps = threads / 32;
    const int NM = a.nmats > 0 ? a.nmats : 1;
    const int NOPS = a.nops > 0 ? a.nops : 1;
    const int NEXP = a.nexp > 0 ? a.nexp : 1;
    const bool batched = a.batched != 0;
    // ---- parameter block (all fields 8-byte aligned, V first):
    //   V m[NM]; u64 ntiles, gthr[8], gslot[E], hibit[16], gctrl[NOPS], hsh[4 NOPS],
    //   mgoff[NOPS], mstride[NOPS], eslot[NEXP], misc[2]; u32 pe[NM]
    // m holds every op's matrix in slot order; for a batched pass the ops with
    // per-instance tables (stride != 0) are staged into shared memory per
    // instance instead: pe[g] = (op << 16) | offset within the instance block
    const size_t o_ntiles = sizeof(V) * size_t(NM), o_gthr = o_ntiles + 8, o_gslot = o_gthr + 64,
                 o_hibit = o_gslot + 8 * size_t(E), o_gctrl = o_hibit + 128, o_hsh = o_gctrl + 8 * size_t(NOPS),
                 o_mgoff = o_hsh + 32 * size_t(NOPS), o_mstride = o_mgoff + 8 * size_t(NOPS),
                 o_eslot = o_mstride + 8 * size_t(NOPS), o_misc = o_eslot + 8 * size_t(NEXP), o_pe = o_misc + 16;
    size_t bytes = o_pe + (batched ? 4 * size_t(NM) : 0);
    bytes = (bytes + 15) & ~size_t(15);
    if (bytes > kJitMaxParamBytes) return false;
    out.params.assign(bytes / 8, 0);
    unsigned char* pb = reinterpret_cast<unsigned char*>(out.params.data());
    auto put64 = [&](size_t off, uint64_t v) { memcpy(pb + off, &v, 8); };
    V* pm = reinterpret_cast<V*>(pb);
    std::vector<char> strided(size_t(NOPS), 0);
    for (int o = 0; o < a.nops; ++o) {
        const KCopy& c = a.cp[o];
        const int D = 1 << c.m;
        const int cnt = c.diag ? D : D * D;
        strided[o] = batched && c.stride != 0;
        put64(o_mgoff + 8 * size_t(o), uint64_t(c.goff));
        put64(o_mstride + 8 * size_t(o), uint64_t(c.stride));
        for (int e = 0; e < cnt; ++e) {
            const int kr = c.diag ? e : e / D, kc = c.diag ? 0 : e % D;
            int sr = 0, sc = 0;
            for (int i = 0; i < c.m; ++i) {
                sr |= ((kr >> i) & 1) << c.perm[i];
                sc |= ((kc >> i) & 1) << c.perm[i];
            }
            const int src = c.diag ? sr : sr * D + sc;
            if (strided[o]) {  // bit 31 marks a staged entry
                const uint32_t v = (1u << 31) | (uint32_t(o) << 16) | uint32_t(src);
                memcpy(pb + o_pe + 4 * size_t(c.soff + e), &v, 4);
            } else {
                pm[c.soff + e] = hm[c.goff + src];
            }
        }
    }
    if (a.nops > 32767) return false;
    std::vector<uint8_t> ncls(size_t(NM), 3);  // value classes of the entries in the block
    for (int i = 0; i < NM; ++i) ncls[size_t(i)] = uint8_t(value_class(pm[i].x, pm[i].y));
    if (!batched && a.nexp == 0) Normaliser<V>(a, pm, ncls).run();
    // tile position of the psi/lam pair bit (adjoint pair passes)
    int pair_tile = -1;
    for (int b = 0; b < 64 && a.pairmask; ++b)
        if ((a.pairmask >> b) & 1) {
            if (b < L) pair_tile = b;
            for (int t = 0; t < H; ++t)
                if (a.hi[t] == b) pair_tile = L + t;
        }
    auto gbit = [&](int b) -> uint64_t { return uint64_t(1) << (b < L ? b : a.hi[b - L]); };
    const KStage& SL = a.st[a.nstages - 1];
    put64(o_ntiles, uint64_t(1) << (a.n - K));
    for (int i = 0; i < nT; ++i) put64(o_gthr + 8 * i, gbit(SL.T[i]));
    for (int s = 0; s < E; ++s) {
        uint64_t v = 0;
        for (int j = 0; j < R; ++j)
            if ((s >> j) & 1) v |= gbit(SL.R[j]);
        put64(o_gslot + 8 * s, v);
    }
    for (int t = 0; t < H; ++t) put64(o_hibit + 8 * t, uint64_t(1) << a.hi[t]);
    for (int o = 0; o < a.nops; ++o) {
        put64(o_gctrl + 8 * o, a.ops[o].gctrl);
        for (int q = 0; q < a.ops[o].nh; ++q)
            put64(o_hsh + 32 * o + 8 * q, a.ops[o].hsrc[q] >= 64 ? uint64_t(a.ops[o].hsrc[q] - 64) : 0);
    }
    for (int e = 0; e < a.nexp; ++e) put64(o_eslot + 8 * e, uint64_t(a.eslot[e]));
    put64(o_misc, ~a.pairmask);
    put64(o_misc + 8, uint64_t(a.inst_shift));
    // value class of a matrix entry: 0, 1, -1, general (3), real (4), imaginary
    // (5).  An entry of a per-instance table gets the class that holds for
    // every instance's value (e.g. real for the entries of Ry tables, imaginary
    // for the off-diagonal entries of Rx tables); the value itself is read from
    // the staged table at run time.
    auto join_class = [](int c1, int c2) -> int {
        if (c1 == c2) return c1;
        const bool r1 = c1 == 0 || c1 == 1 || c1 == 2 || c1 == 4, r2 = c2 == 0 || c2 == 1 || c2 == 2 || c2 == 4;
        if (r1 && r2) return 4;
        if ((c1 == 0 || c1 == 5) && (c2 == 0 || c2 == 5)) return 5;
        return 3;
    };
    // instances of a batched pass: the vector bits above inst_shift, less the pair bit
    const int64_t ninst =
        batched && a.inst_shift > 0 ? (int64_t(1) << (a.n - a.inst_shift - (a.pairmask ? 1 : 0))) : int64_t(1);
    std::vector<uint8_t> scls(size_t(NM), 3);
    for (int o = 0; o < a.nops; ++o) {
        if (!strided[o]) continue;
        const KCopy& c = a.cp[o];
        const int D = 1 << c.m;
        const int cnt = c.diag ? D : D * D;
        for (int e = 0; e < cnt; ++e) {
            const int kr = c.diag ? e : e / D, kc = c.diag ? 0 : e % D;
            int sr = 0, sc = 0;
            for (int i = 0; i < c.m; ++i) {
                sr |= ((kr >> i) & 1) << c.perm[i];
                sc |= ((kc >> i) & 1) << c.perm[i];
            }
            const int64_t src = c.goff + (c.diag ? sr : sr * D + sc);
            int cl = value_class(hm[src].x, hm[src].y);
            for (int64_t i = 1; i < ninst && cl != 3; ++i) cl = join_class(cl, value_class(hm[src + i * c.stride].x, hm[src + i * c.stride].y));
            scls[size_t(c.soff + e)] = uint8_t(cl);
        }
    }
    auto vclass = [&](int o, int idx) -> int { return int((strided[o] ? scls : ncls)[size_t(idx)]); };
    auto mref = [&](int o, int idx) -> std::string {
        return (strided[o] ? "msm[" : "p.m[") + std::to_string(idx) + "]";
    };
    out.classes.resize(size_t(NM));
    for (int o = 0; o < a.nops; ++o) {
        const KCopy& c = a.cp[o];
        const int cnt = c.diag ? (1 << c.m) : (1 << (2 * c.m));
        for (int e = 0; e < cnt; ++e) out.classes[c.soff + e] = uint8_t(vclass(o, c.soff + e));
    }
    // Diagonal tables indexed by thread bits (a different entry per lane) are
    // copied to shared memory once per CTA: parameter-space loads with lane-
    // dependent addresses are serialised, shared-memory loads are not.
    std::vector<int> doff(size_t(NOPS), -1);
    int ndsm = 0;
    for (int o = 0; o < a.nops; ++o) {
        const KOp& op = a.ops[o];
        const bool dg = op.code == QS_OP_DIAG || (op.code == QS_OP_EXPECT && (op.flags & QS_OPF_DIAG));
        if (!dg || op.nh == 0 || strided[o]) continue;
        bool thr = false;
        for (int q = 0; q < op.nh; ++q) thr = thr || op.hsrc[q] < 64;
        if (!thr) continue;
        doff[size_t(o)] = ndsm;
        ndsm += 1 << a.cp[o].m;
    }
    // the table of a diagonal with other-bit index h, as an expression prefix
    auto dtab = [&](int o) -> std::string {
        if (strided[o]) return "msm[" + std::to_string(int(a.ops[o].moff)) + " + ";
        if (doff[size_t(o)] >= 0) return "dsm[" + std::to_string(doff[size_t(o)]) + " + ";
        return "p.m[" + std::to_string(int(a.ops[o].moff)) + " + ";
    };
    const unsigned hoff_n = (1u << H) < 2u ? 2u : (1u << H);  // a 16-byte multiple
    // One tile buffer instead of two (kernels only): the next tile is fetched
    // once the last stage has read this one, under that stage's arithmetic and
    // stores, and the smaller footprint lets more CTAs share an SM, whose loads
    // and arithmetic overlap.  Measured on the 30-qubit spread circuit (B200),
    // one buffer against two: complex128 k = 11 270 against 284 ms, complex64
    // k = 12 164.6 against 163.2 ms, k = 11 168.3 against 166.1 ms.  Passes with
    // per-instance tables and adjoint passes have registers for two CTAs per SM
    // at any width, where two 64 KB buffers leave room for one: gradients of 256
    // parameter sets of a 16-qubit ansatz in complex64 6.98 against 10.88 ms.  So
    // the default is double for plain complex64 passes only.  Fetching only after
    // the stores: complex128 k = 12 276 ms, now 261 ms (k = 10: 272, 269).
    // QS_JIT_SINGLE_BUFFER=0/1 overrides it.
    const bool single = devfn == nullptr && jit_single_buffer(C128, batched || a.nexp > 0);
    const int nbuf = single ? 1 : 2;
    out.threads = threads;
    out.smem = sizeof(V) * size_t(nbuf) * (size_t(1) << K) + 8 * size_t(hoff_n) +
               (a.nexp > 0 ? sizeof(double2) * size_t(nwarps) * size_t(a.nexp) : 0) +
               (batched ? sizeof(V) * size_t(NM) : 0) + sizeof(V) * size_t(ndsm);
    out.smem = (out.smem + 15) & ~size_t(15);
    // a device function keeps its parameter block in shared memory behind the
    // rest (see its prologue); the kernels read theirs from the parameter bank
    const size_t smem_main = out.smem;
    if (devfn) out.smem += 8 * out.params.size();
    if (!with_source) return true;
    const char* VT = C128 ? "double2" : "float2";
    const char* ST = C128 ? "double" : "float";
    const char* MK = C128 ? "make_double2" : "make_float2";
    const char* FMA = C128 ? "__fma_rn" : "__fmaf_rn";
    // resident threads per SM the register budget is sized for (launch bounds);
    // QS_JIT_THREADS_PER_SM overrides it
    static const int env_target = [] {
        const char* e = getenv("QS_JIT_THREADS_PER_SM");
        return e && *e ? atoi(e) : 0;
    }();
    // 512 threads per SM; plain complex64 passes (no per-instance tables, no
    // EXPECT ops) with 4 register bits 768 (30-qubit spread circuit, k = 12,
    // nlow 6, B200: 151.2 -> 148.1 ms; 28 qubits 14.5, 14.4 and at 1024 14.7
    // ms), with 5 register bits 256, i.e. the whole register file for 64-thread
    // CTAs (k = 11: 211.6 -> 189.7 ms; 384: 208.2 ms).  complex128 passes are
    // fastest at 512 (k = 12: 261 ms; 295 ms at 256; k = 10 at 640: 275 against
    // 269 ms).
    const bool plain64 = !C128 && !batched && a.nexp == 0;
    const int target = env_target > 0 ? env_target : !plain64 ? 512 : R == 4 ? 768 : 256;
    const int minb = threads >= target ? 1 : target / threads;
    SrcBuf g;
    g.add("// generated fused pass: n=%d K=%d L=%d R=%d stages=%d ops=%d expect=%d batched=%d\n", a.n, K, L, R,
          a.nstages, a.nops, a.nexp, int(batched));
    g.add("typedef unsigned long long u64;\ntypedef unsigned int u32;\ntypedef %s V;\ntypedef %s S;\n", VT, ST);
    g.add("static __device__ __forceinline__ V cmul(V a, V b) { V r; r.x = a.x * b.x - a.y * b.y; "
          "r.y = a.x * b.y + a.y * b.x; return r; }\n");
    g.add("static __device__ __forceinline__ V cfma(V a, V b, V c) { V r; r.x = %s(a.x, b.x, %s(-a.y, b.y, c.x)); "
          "r.y = %s(a.x, b.y, %s(a.y, b.x, c.y)); return r; }\n", FMA, FMA, FMA, FMA);
    g.add("static __device__ __forceinline__ V cadd(V a, V b) { V r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }\n");
    g.add("static __device__ __forceinline__ V cneg(V a) { V r; r.x = -a.x; r.y = -a.y; return r; }\n");
    g.add("static __device__ __forceinline__ V csel(bool c, V a, V b) { V r; r.x = c ? a.x : b.x; "
          "r.y = c ? a.y : b.y; return r; }\n");
    // products with a real entry a (rmul / rfma) or an imaginary one i*b (imul / ifma)
    g.add("static __device__ __forceinline__ V rmul(S a, V v) { V r; r.x = a * v.x; r.y = a * v.y; return r; }\n");
    g.add("static __device__ __forceinline__ V rfma(S a, V v, V c) { V r; r.x = %s(a, v.x, c.x); "
          "r.y = %s(a, v.y, c.y); return r; }\n", FMA, FMA);
    g.add("static __device__ __forceinline__ V imul(S b, V v) { V r; r.x = -b * v.y; r.y = b * v.x; return r; }\n");
    g.add("static __device__ __forceinline__ V ifma(S b, V v, V c) { V r; r.x = %s(-b, v.y, c.x); "
          "r.y = %s(b, v.x, c.y); return r; }\n", FMA, FMA);
    g.add("struct __align__(16) P { V m[%d]; u64 ntiles; u64 gthr[8]; u64 gslot[%d]; u64 hibit[16]; u64 gctrl[%d]; "
          "u64 hsh[%d]; u64 mgoff[%d]; u64 mstride[%d]; u64 eslot[%d]; u64 misc[2];%s };\n", NM, E, NOPS, 4 * NOPS,
          NOPS, NOPS, NEXP, batched ? (" u32 pe[" + std::to_string(NM) + "];").c_str() : "");
    // cooperative loops (no per-thread layout): all threads of the CTA
    const std::string CT = devfn ? "threadIdx.x" : "tid";
    const std::string CS = devfn ? "blockDim.x" : std::to_string(threads) + "u";
    if (devfn) {
        g.add("extern \"C\" __device__ void %s(V* __restrict__ vec, const void* __restrict__ pv, "
              "const V* __restrict__ mats, double* __restrict__ partials, u64 tile, const u64 tend, "
              "const u32 zero_in) {\n", devfn);
    } else {
        g.add("extern \"C\" __global__ void __launch_bounds__(%d, %d) qs_pass(V* __restrict__ vec, "
              "const __grid_constant__ P p, const V* __restrict__ mats, double* __restrict__ partials) {\n", threads,
              minb);
    }
    g.add("  extern __shared__ __align__(16) unsigned char smem_raw[];\n");
    if (devfn) {
        // the parameter block moves from the plan (global memory) to shared
        // memory behind the tile buffers: matrix entries are read at shared-
        // memory latency, as the kernels read them from the constant bank
        g.add("  { const uint4* __restrict__ src = reinterpret_cast<const uint4*>(pv);\n"
              "    uint4* dst = reinterpret_cast<uint4*>(smem_raw + %zuu);\n"
              "    for (u32 i = threadIdx.x; i < %zuu; i += blockDim.x) dst[i] = src[i]; }\n"
              "  __syncthreads();\n  const P& p = *reinterpret_cast<const P*>(smem_raw + %zuu);\n",
              smem_main, out.params.size() / 2, smem_main);
    }
    g.add("  V* const b0 = reinterpret_cast<V*>(smem_raw);\n  V* const b1 = b0 + %du;\n", single ? 0u : 1u << K);
    g.add("  u64* const hoff = reinterpret_cast<u64*>(b1 + %du);\n", 1u << K);
    g.add("  double2* const ered = reinterpret_cast<double2*>(hoff + %du);\n", hoff_n);
    g.add("  V* const msm = reinterpret_cast<V*>(ered + %d);\n", a.nexp > 0 ? nwarps * a.nexp : 0);
    g.add("  V* const dsm = msm + %d;\n", batched ? NM : 0);
    if (devfn) g.add("  const u32 tid = threadIdx.x & %du;\n  const bool act = threadIdx.x < %du;\n",
                     unsigned(threads - 1), unsigned(threads));
    else g.add("  const u32 tid = threadIdx.x;\n");
    g.add("  for (u32 j = %s; j < %du; j += %s) { u64 o = 0;\n", CT.c_str(), 1u << H, CS.c_str());
    g.add("#pragma unroll\n    for (int t = 0; t < %d; ++t) if ((j >> t) & 1u) o |= p.hibit[t];\n    hoff[j] = o; }\n", H);
    for (int o = 0; o < a.nops; ++o)
        if (doff[size_t(o)] >= 0)
            g.add("  for (u32 q = %s; q < %du; q += %s) dsm[%d + q] = p.m[%d + q];\n", CT.c_str(), 1u << a.cp[o].m,
                  CS.c_str(), doff[size_t(o)], int(a.ops[o].moff));
    g.add("  u64 gthr = 0;\n");
    for (int i = 0; i < nT; ++i) g.add("  if ((tid >> %d) & 1u) gthr |= p.gthr[%d];\n", i, i);
    for (int si = 0; si < a.nstages; ++si) {
        const KStage& S = a.st[si];
        uint32_t rt[8], wt[8], tb[8];
        for (int i = 0; i < 8; ++i) {
            rt[i] = S.rthr[i];
            wt[i] = S.wthr[i];
            tb[i] = S.tbit[i];
        }
        g.add("  const u32 RD%d = %s;\n", si, thread_xor_expr(rt, nT).c_str());
        if (si > 0) g.add("  const u32 WR%d = %s;\n", si, thread_xor_expr(wt, nT).c_str());
        g.add("  const u32 TH%d = %s;\n", si, thread_xor_expr(tb, nT).c_str());
    }
    g.add("  const u64 ntiles = p.ntiles;\n");
    g.add("  auto tile_base = [&](u64 t) -> u64 { u64 b = t << %d;\n", L);
    g.add("#pragma unroll\n    for (int i = 0; i < %d; ++i) { const u64 lo = p.hibit[i] - 1ull; "
          "b = ((b & ~lo) << 1) | (b & lo); }\n    return b; };\n", H);
    if (devfn) {  // the caller's tile range
        g.add("  const u64 tstep = 1;\n");
        if (batched) g.add("  u64 staged = ~0ull;\n");
    } else if (batched) {
        // per-instance tables: contiguous runs of tiles per CTA, so that a CTA
        // restages its instance's matrices once per instance
        g.add("  const u64 chunk = (ntiles + gridDim.x - 1) / gridDim.x;\n");
        g.add("  u64 tile = u64(blockIdx.x) * chunk;\n  const u64 tend = tile + chunk < ntiles ? tile + chunk : ntiles;\n");
        g.add("  const u64 tstep = 1;\n  u64 staged = ~0ull;\n");
    } else {
        g.add("  u64 tile = blockIdx.x;\n  const u64 tend = ntiles;\n  const u64 tstep = gridDim.x;\n");
    }
    g.add("  __syncthreads();\n");
    const int EPC = 16 / int(sizeof(V));
    g.add("  auto prefetch = [&](V* dst, u64 base) {\n");
    if (devfn)
        g.add("    if (zero_in) { for (u32 e = threadIdx.x; e < %du; e += blockDim.x) { V z; z.x = (base == 0 && e == 0) "
              "? 1 : 0; z.y = 0; dst[e] = z; } } else\n", 1u << K);
    g.add("    for (u32 c = %s; c < %du; c += %s) { const u32 e = c * %du;\n", CT.c_str(), (1u << K) / EPC, CS.c_str(),
          EPC);
    g.add("      const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(dst + e));\n");
    g.add("      asm volatile(\"cp.async.cg.shared.global [%%0], [%%1], 16;\\n\" :: \"r\"(sa), "
          "\"l\"(vec + (base | hoff[e >> %d] | (e & %du))) : \"memory\"); }\n", L, (1u << L) - 1u);
    g.add("    asm volatile(\"cp.async.commit_group;\\n\" ::: \"memory\"); };\n");
    g.add("  if (tile < tend) prefetch(b0, tile_base(tile));\n");
    g.add("  for (u32 it = 0; tile < tend; ++it, tile += tstep) {\n");
    g.add("    V* const cur = (it & 1u) ? b1 : b0;\n    const u64 base = tile_base(tile);\n");
    g.add("    asm volatile(\"cp.async.wait_group 0;\\n\" ::: \"memory\");\n    __syncthreads();\n");
    if (!single) g.add("    if (tile + tstep < tend) prefetch((it & 1u) ? b0 : b1, tile_base(tile + tstep));\n");
    if (batched) {
        g.add("    { const u64 inst = (base & p.misc[0]) >> p.misc[1];\n");
        g.add("      if (inst != staged) {\n");
        g.add("        for (u32 q = %s; q < %du; q += %s) { const u32 v = p.pe[q];\n", CT.c_str(), unsigned(a.nmats),
              CS.c_str());
        g.add("          if (v >> 31) { const u32 o = (v >> 16) & 0x7fffu; "
              "msm[q] = mats[p.mgoff[o] + inst * p.mstride[o] + (v & 0xffffu)]; } }\n");
        g.add("        staged = inst;\n        __syncthreads();\n      } }\n");
    }
    // ---- body
    int fresh = 0;
    std::vector<int> var(E);  // slot -> SSA value id
    auto vname = [&](int id) { return "v" + std::to_string(id); };
    auto slot_addr = [&](const uint16_t* img, int s) {
        uint32_t c = 0;
        for (int j = 0; j < R; ++j)
            if ((s >> j) & 1) c ^= img[j];
        return c;
    };
    // the sum over the nonzero entries of one row of a (slot-order) matrix
    auto row_expr = [&](int o, int base_idx, int D, const int* in) -> std::string {
        std::string e;
        int first = 0;  // start from a unit entry: it costs nothing
        for (int c = D - 1; c >= 0; --c)
            if (vclass(o, base_idx + c) == 1 || vclass(o, base_idx + c) == 2) first = c;
        for (int i = 0; i < D; ++i) {
            const int c = i == 0 ? first : i <= first ? i - 1 : i;
            const int idx = base_idx + c;
            const int cl = vclass(o, idx);
            if (cl == 0) continue;
            const std::string x = vname(in[c]);
            const std::string m = mref(o, idx);
            if (e.empty()) {
                if (cl == 1) e = x;
                else if (cl == 2) e = "cneg(" + x + ")";
                else if (cl == 4) e = "rmul(" + m + ".x, " + x + ")";
                else if (cl == 5) e = "imul(" + m + ".y, " + x + ")";
                else e = "cmul(" + m + ", " + x + ")";
            } else {
                if (cl == 1) e = "cadd(" + e + ", " + x + ")";
                else if (cl == 2) e = "cadd(" + e + ", cneg(" + x + "))";
                else if (cl == 4) e = "rfma(" + m + ".x, " + x + ", " + e + ")";
                else if (cl == 5) e = "ifma(" + m + ".y, " + x + ", " + e + ")";
                else e = "cfma(" + m + ", " + x + ", " + e + ")";
            }
        }
        if (e.empty()) e = std::string(MK) + "(0, 0)";
        return e;
    };
    // thread-dependent / outside-tile index bits of a diagonal (h), as an expression
    auto h_expr = [&](const KOp& op, int o, int si) -> std::string {
        std::string h;
        for (int q = 0; q < op.nh; ++q) {
            const int src = op.hsrc[q];
            const std::string t = src < 64 ? "((TH" + std::to_string(si) + " >> " + std::to_string(src) + ") & 1u)"
                                            : "u32((base >> p.hsh[" + std::to_string(4 * o + q) + "]) & 1ull)";
            h = h.empty() ? t : "((" + h + ") << 1) | " + t;
        }
        return h;
    };
    for (int s = 0; s < E; ++s) {
        var[s] = fresh++;
        g.add("    const V v%d = cur[RD0 ^ %uu];\n", var[s], slot_addr(a.st[0].rslot, s));
    }
    for (int si = 0; si < a.nstages; ++si) {
        const KStage& S = a.st[si];
        if (si > 0) {
            g.add("    __syncthreads();\n");
            for (int s = 0; s < E; ++s) g.add("    cur[WR%d ^ %uu] = v%d;\n", si, slot_addr(S.wslot, s), var[s]);
            g.add("    __syncthreads();\n");
            for (int s = 0; s < E; ++s) {
                var[s] = fresh++;
                g.add("    const V v%d = cur[RD%d ^ %uu];\n", var[s], si, slot_addr(S.rslot, s));
            }
        }
        if (single && si == a.nstages - 1)  // the buffer's last readers: the next tile comes in under the last stage
            g.add("    __syncthreads();\n    if (tile + tstep < tend) prefetch(b0, tile_base(tile + tstep));\n");
        for (int o = S.op_begin; o < S.op_begin + S.op_count; ++o) {
            const KOp& op = a.ops[o];
            std::string cond;
            if (op.gctrl) cond = "((base & p.gctrl[" + std::to_string(o) + "]) == p.gctrl[" + std::to_string(o) + "])";
            if (op.tctrl) {
                const std::string tc = std::to_string(unsigned(op.tctrl)) + "u";
                cond += (cond.empty() ? "" : " && ") + std::string("((TH") + std::to_string(si) + " & " + tc +
                        ") == " + tc + ")";
            }
            const int scm = op.scm;
            auto ctrl_ok = [&](int s) { return (s & scm) == scm; };
            if (!cond.empty() && op.code != QS_OP_EXPECT) g.add("    const bool c%d = %s;\n", o, cond.c_str());
            if (op.code == QS_OP_MAT) {
                const int mask = op.mask, M = popc_c(mask), D = 1 << M;
                g.add("    // op %d: dense on slot mask %d\n", o, mask);
                for (int s = 0; s < E; ++s) {
                    if ((s & mask) || !ctrl_ok(s)) continue;
                    int in[16], outid[16];
                    for (int c = 0; c < D; ++c) in[c] = var[s | pdep_c(c, mask)];
                    for (int r = 0; r < D; ++r) {
                        const std::string e = row_expr(o, op.moff + r * D, D, in);
                        outid[r] = fresh++;
                        if (cond.empty()) g.s += "    const V " + vname(outid[r]) + " = " + e + ";\n";
                        else g.s += "    const V " + vname(outid[r]) + " = c" + std::to_string(o) + " ? " + e + " : " +
                                    vname(in[r]) + ";\n";
                    }
                    for (int r = 0; r < D; ++r) var[s | pdep_c(r, mask)] = outid[r];
                }
            } else if (op.code == QS_OP_ANTI || op.code == QS_OP_SWAP) {  // plain exchanges
                int b0, b1;
                if (op.code == QS_OP_ANTI) {
                    b0 = 0;
                    b1 = op.mask;
                } else {
                    b0 = 1 << nth_bit(op.mask, 0);
                    b1 = 1 << nth_bit(op.mask, 1);
                }
                for (int s = 0; s < E; ++s) {
                    if ((s & op.mask) || !ctrl_ok(s)) continue;
                    const int x0 = var[s | b0], x1 = var[s | b1];
                    if (cond.empty()) {
                        var[s | b0] = x1;
                        var[s | b1] = x0;
                    } else {
                        const int n0 = fresh++, n1 = fresh++;
                        g.add("    const V v%d = csel(c%d, v%d, v%d);\n", n0, o, x1, x0);
                        g.add("    const V v%d = csel(c%d, v%d, v%d);\n", n1, o, x0, x1);
                        var[s | b0] = n0;
                        var[s | b1] = n1;
                    }
                }
            } else if (op.code == QS_OP_DIAG) {
                g.add("    // op %d: diagonal, %d register bits, %d other bits\n", o, op.ns, op.nh);
                if (op.nh > 0) g.s += "    const u32 h" + std::to_string(o) + " = " + h_expr(op, o, si) + ";\n";
                for (int s = 0; s < E; ++s) {
                    if (!ctrl_ok(s)) continue;
                    const int k = op.kidx[s];
                    std::string e;
                    if (op.nh == 0) {
                        const int idx = op.moff + k;
                        const int cl = vclass(o, idx);
                        if (cl == 1) continue;
                        if (cl == 2) e = "cneg(" + vname(var[s]) + ")";
                        else if (cl == 0) e = std::string(MK) + "(0, 0)";
                        else if (cl == 4) e = "rmul(" + mref(o, idx) + ".x, " + vname(var[s]) + ")";
                        else if (cl == 5) e = "imul(" + mref(o, idx) + ".y, " + vname(var[s]) + ")";
                        else e = "cmul(" + vname(var[s]) + ", " + mref(o, idx) + ")";
                    } else {
                        e = "cmul(" + vname(var[s]) + ", " + dtab(o) + "((h" + std::to_string(o) + " << " +
                            std::to_string(int(op.ns)) + ") | " + std::to_string(k) + "u)])";
                    }
                    const int nid = fresh++;
                    if (cond.empty()) g.s += "    const V " + vname(nid) + " = " + e + ";\n";
                    else g.s += "    const V " + vname(nid) + " = c" + std::to_string(o) + " ? " + e + " : " +
                                vname(var[s]) + ";\n";
                    var[s] = nid;
                }
            } else if (op.code == QS_OP_EXPECT) {
                // sum over the thread's psi/lam pairs (slot bit 0 = pair bit) of
                // conj(lam) (G psi) in the state's precision, then a warp sum in FP64
                if (!cond.empty() || scm != 0 || pair_tile < 0 || S.R[0] != pair_tile) return false;
                g.add("    { // op %d: <lam| G |psi>\n      S pr = 0, pi = 0;\n", o);
                const bool dg = op.flags & QS_OPF_DIAG;
                if (dg && op.nh > 0) g.s += "      const u32 h" + std::to_string(o) + " = " + h_expr(op, o, si) + ";\n";
                if (dg) {
                    for (int s = 0; s < E; s += 2) {
                        const int k = op.kidx[s];
                        std::string d = op.nh == 0 ? mref(o, op.moff + k)
                                                   : dtab(o) + "((h" + std::to_string(o) + " << " +
                                                         std::to_string(int(op.ns)) + ") | " + std::to_string(k) +
                                                         "u)]";
                        g.s += "      { const V acc = cmul(" + d + ", " + vname(var[s]) + "); const V l = " +
                               vname(var[s | 1]) + ";\n";
                        g.s += "        pr += l.x * acc.x + l.y * acc.y; pi += l.x * acc.y - l.y * acc.x; }\n";
                    }
                } else {
                    const int mask = op.mask, M = popc_c(mask), D = 1 << M;
                    if ((mask & 1) || M > 2) return false;
                    for (int s = 0; s < E; ++s) {
                        if ((s & mask) || (s & 1)) continue;
                        int in[4];
                        for (int c = 0; c < D; ++c) in[c] = var[s | pdep_c(c, mask)];
                        for (int r = 0; r < D; ++r) {
                            g.s += "      { const V acc = " + row_expr(o, op.moff + r * D, D, in) + "; const V l = " +
                                   vname(var[s | 1 | pdep_c(r, mask)]) + ";\n";
                            g.s += "        pr += l.x * acc.x + l.y * acc.y; pi += l.x * acc.y - l.y * acc.x; }\n";
                        }
                    }
                }
                g.add("      double re = pr, im = pi;\n");
                g.add("#pragma unroll\n      for (int off = 16; off > 0; off >>= 1) { re += __shfl_xor_sync(0xffffffffu, "
                      "re, off); im += __shfl_xor_sync(0xffffffffu, im, off); }\n");
                g.add("      if ((tid & 31u) == 0) ered[(tid >> 5) * %d + %d] = make_double2(re, im);\n    }\n", NEXP,
                      int(op.elocal));
            } else {
                return false;
            }
        }
    }
    if (devfn) g.add("    if (act) {\n");
    for (int s = 0; s < E; ++s) g.add("    vec[base | gthr | p.gslot[%d]] = v%d;\n", s, var[s]);
    if (devfn) g.add("    }\n");
    if (a.nexp > 0) {
        // per-tile partials: the warps' sums in a fixed order
        g.add("    __syncthreads();\n");
        g.add("    for (u32 e = %s; e < %du; e += %s) { double2 t = make_double2(0.0, 0.0);\n", CT.c_str(),
              unsigned(a.nexp), CS.c_str());
        g.add("      for (int w = 0; w < %d; ++w) { t.x += ered[w * %d + e].x; t.y += ered[w * %d + e].y; }\n", nwarps,
              NEXP, NEXP);
        g.add("      const u64 at = 2 * (p.eslot[e] * ntiles + tile);\n      partials[at] = t.x;\n"
              "      partials[at + 1] = t.y; }\n");
    }
    g.add("  }\n}\n");
    if (g.truncated) return false;
    out.src.swap(g.s);
    return true;
}

}  // namespace

bool gen_pass(const void* regargs, int R, bool c128, const void* mats_host, JitPass& out, bool with_source,
              const char* devfn) {
    const RegArgs& a = *static_cast<const RegArgs*>(regargs);
    return c128 ? gen_reg_pass<double2>(a, R, static_cast<const double2*>(mats_host), out, with_source, devfn)
                : gen_reg_pass<float2>(a, R, static_cast<const float2*>(mats_host), out, with_source, devfn);
}

bool gen_batch_pass(const void* regargs, int R, bool c128, const void* mats_host, const char* name, std::string* src,
                    std::vector<uint64_t>* params, size_t* smem, int* threads) {
    JitPass jp;
    if (!gen_pass(regargs, R, c128, mats_host, jp, true, name)) return false;
    src->swap(jp.src);
    params->swap(jp.params);
    *smem = jp.smem;
    *threads = jp.threads;
    return true;
}

}  // namespace qs
