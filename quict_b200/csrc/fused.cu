// Fused passes: one launch streams the state through on-chip tiles once and
// applies every op of the pass to each tile.
//
// A tile holds 2^k amplitudes: vector bits 0..nlow-1 (contiguous, so each
// warp moves 2^nlow consecutive amplitudes) plus k-nlow chosen higher bits.
// Ops whose non-diagonal targets lie in the tile run on chip; diagonal factors
// and controls on bits outside the tile are resolved per tile from the tile's
// base index, so they fuse into any pass.
//
// Register-resident kernel (k_fused_reg, tiles of 2^(R+5..R+8)):
//   each thread owns 2^R amplitudes in registers.  A "layout" assigns R tile
//   bits to register-slot bits and the remaining tile bits to the thread index
//   (lanes first).  Ops whose dense targets are slot bits run as fully
//   unrolled register code (one template per slot mask, no shared memory, no
//   barriers); between groups of ops ("stages") the tile is re-laid-out
//   through shared memory under a per-relayout XOR address map that keeps
//   both sides free of bank conflicts.  Loads and stores use a layout whose
//   lanes are tile bits 0..4, i.e. warp-contiguous global runs.  The host
//   (this file) plans the stages, translates each op into slot / thread /
//   outside-tile terms and permutes its matrix to the slot order.
// Shared-memory kernel (k_fused_smem): tiles too small for that layout.
//
// The reference has no fusion: one kernel and one full HBM pass per gate
// (statevector_simulator.py:155-164, gate_function.py:31-1031).
#include <algorithm>
#include <array>
#include <cstdarg>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <type_traits>
#include <unordered_map>
#include <utility>
#include <vector>

#include "common.cuh"
#include "jit.h"
#include "passgen.h"
#include "regtile.cuh"

namespace qs {
namespace {

constexpr int kFT = 256;

// =============================================================== shared-memory kernel
struct PassArgs {
    int n, k, nlow, nops, inst_shift;
    int hi[QS_MAX_TILE_BITS];
    qs_op ops[QS_MAX_PASS_OPS];
};

template <int M>
__device__ __forceinline__ void sort_bits(const int* t, int* s) {
#pragma unroll
    for (int i = 0; i < M; ++i) s[i] = t[i];
#pragma unroll
    for (int i = 0; i < M; ++i)
#pragma unroll
        for (int j = 0; j + 1 < M - i; ++j)
            if (s[j] > s[j + 1]) { int x = s[j]; s[j] = s[j + 1]; s[j + 1] = x; }
}

template <typename V, int M>
__device__ __forceinline__ void tile_mat(V* __restrict__ tile, int K, const qs_op& op, const V* __restrict__ mat) {
    constexpr int D = 1 << M;
    int t[M], s[M];
#pragma unroll
    for (int j = 0; j < M; ++j) t[j] = op.tgt[j];
    sort_bits<M>(t, s);
    uint32_t spread[D];
#pragma unroll
    for (int r = 0; r < D; ++r) {
        uint32_t o = 0;
#pragma unroll
        for (int j = 0; j < M; ++j)
            if ((r >> (M - 1 - j)) & 1) o |= 1u << t[j];
        spread[r] = o;
    }
    const uint32_t lctrl = op.lctrl;
    const uint32_t groups = 1u << (K - M);
    for (uint32_t g = threadIdx.x; g < groups; g += kFT) {
        uint32_t i0 = g;
#pragma unroll
        for (int j = 0; j < M; ++j) i0 = ins0(i0, s[j]);
        if ((i0 & lctrl) != lctrl) continue;
        V x[D];
#pragma unroll
        for (int r = 0; r < D; ++r) x[r] = tile[i0 | spread[r]];
#pragma unroll
        for (int r = 0; r < D; ++r) {
            V acc = cmul(__ldg(&mat[r * D]), x[0]);
#pragma unroll
            for (int c = 1; c < D; ++c) acc = cfma(__ldg(&mat[r * D + c]), x[c], acc);
            tile[i0 | spread[r]] = acc;
        }
    }
}

template <typename V>
__device__ __forceinline__ void tile_diag(V* __restrict__ tile, int K, uint64_t base, const qs_op& op,
                                          const V* __restrict__ mat) {
    const int m = op.m;
    uint32_t ext = 0;
    int lpos[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        lpos[j] = -1;
        if (j < m) {
            if (op.tgt[j] < 0) ext |= uint32_t((base >> op.gbit[j]) & 1) << (m - 1 - j);
            else lpos[j] = op.tgt[j];
        }
    }
    const uint32_t lctrl = op.lctrl;
    const uint32_t T = 1u << K;
    for (uint32_t e = threadIdx.x; e < T; e += kFT) {
        if ((e & lctrl) != lctrl) continue;
        uint32_t sidx = ext;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < m && lpos[j] >= 0) sidx |= ((e >> lpos[j]) & 1u) << (m - 1 - j);
        tile[e] = cmul(tile[e], __ldg(&mat[sidx]));
    }
}

// <lam| G |psi> over the tile for a generator on m <= 2 tile bits (dense) or
// a diagonal on bits anywhere (QS_OPF_DIAG); thread-partial sum returned.
template <typename V, int M>
__device__ __forceinline__ double2 tile_expect_dense(const V* __restrict__ psi, const V* __restrict__ lam, int K,
                                                     const qs_op& op, const V* __restrict__ g) {
    constexpr int D = 1 << M;
    int t[M], s[M];
#pragma unroll
    for (int j = 0; j < M; ++j) t[j] = op.tgt[j];
    sort_bits<M>(t, s);
    uint32_t spread[D];
#pragma unroll
    for (int r = 0; r < D; ++r) {
        uint32_t o = 0;
#pragma unroll
        for (int j = 0; j < M; ++j)
            if ((r >> (M - 1 - j)) & 1) o |= 1u << t[j];
        spread[r] = o;
    }
    double re = 0.0, im = 0.0;
    const uint32_t groups = 1u << (K - M);
    for (uint32_t gi = threadIdx.x; gi < groups; gi += blockDim.x) {
        uint32_t i0 = gi;
#pragma unroll
        for (int j = 0; j < M; ++j) i0 = ins0(i0, s[j]);
        if ((i0 & op.lctrl) != op.lctrl) continue;
        V x[D];
#pragma unroll
        for (int r = 0; r < D; ++r) x[r] = psi[i0 | spread[r]];
#pragma unroll
        for (int r = 0; r < D; ++r) {
            V acc = cmul(g[r * D], x[0]);
#pragma unroll
            for (int c = 1; c < D; ++c) acc = cfma(g[r * D + c], x[c], acc);
            const V l = lam[i0 | spread[r]];
            re += double(l.x) * double(acc.x) + double(l.y) * double(acc.y);
            im += double(l.x) * double(acc.y) - double(l.y) * double(acc.x);
        }
    }
    return make_double2(re, im);
}

template <typename V>
__device__ __forceinline__ double2 tile_expect_diag(const V* __restrict__ psi, const V* __restrict__ lam, int K,
                                                    uint64_t base, const qs_op& op, const V* __restrict__ d) {
    const int m = op.m;
    uint32_t ext = 0;
    int lpos[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        lpos[j] = -1;
        if (j < m) {
            if (op.tgt[j] < 0) ext |= uint32_t((base >> op.gbit[j]) & 1) << (m - 1 - j);
            else lpos[j] = op.tgt[j];
        }
    }
    double re = 0.0, im = 0.0;
    for (uint32_t e = threadIdx.x; e < (1u << K); e += blockDim.x) {
        if ((e & op.lctrl) != op.lctrl) continue;
        uint32_t sidx = ext;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < m && lpos[j] >= 0) sidx |= ((e >> lpos[j]) & 1u) << (m - 1 - j);
        const V acc = cmul(d[sidx], psi[e]);
        const V l = lam[e];
        re += double(l.x) * double(acc.x) + double(l.y) * double(acc.y);
        im += double(l.x) * double(acc.y) - double(l.y) * double(acc.x);
    }
    return make_double2(re, im);
}

// Shared-memory tile kernel.  ADJ: two vectors (psi, lam) move through the
// same tiles; apply-ops act on both and EXPECT ops write per-tile partials.
template <typename V, bool ADJ>
__global__ void __launch_bounds__(kFT) k_fused_smem(V* __restrict__ vec, V* __restrict__ vec2,
                                                     const __grid_constant__ PassArgs p, const V* __restrict__ mats,
                                                     double* __restrict__ partials) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double2 red[kFT / 32];
    const int K = p.k, L = p.nlow, H = K - L;
    const uint32_t T = 1u << K;
    V* tile = reinterpret_cast<V*>(smem_raw);
    V* tile2 = tile + (ADJ ? T : 0);
    uint64_t* hoff = reinterpret_cast<uint64_t*>(smem_raw + sizeof(V) * T * (ADJ ? 2 : 1));
    for (uint32_t j = threadIdx.x; j < (1u << H); j += kFT) {
        uint64_t o = 0;
        for (int t = 0; t < H; ++t)
            if ((j >> t) & 1) o |= uint64_t(1) << p.hi[t];
        hoff[j] = o;
    }
    __syncthreads();
    const uint32_t lmask = (1u << L) - 1u;
    const uint64_t ntiles = uint64_t(1) << (p.n - K);
    for (uint64_t tid = blockIdx.x; tid < ntiles; tid += gridDim.x) {
        uint64_t base = tid << L;
        for (int t = 0; t < H; ++t) base = insert0(base, p.hi[t]);
        const uint64_t inst = p.inst_shift > 0 ? (base >> p.inst_shift) : 0;
        for (uint32_t e = threadIdx.x; e < T; e += kFT) {
            const uint64_t gi = base | hoff[e >> L] | (e & lmask);
            tile[e] = vec[gi];
            if (ADJ) tile2[e] = vec2[gi];
        }
        __syncthreads();
        for (int o = 0; o < p.nops; ++o) {
            const qs_op& op = p.ops[o];
            const bool on = (base & op.gctrl) == op.gctrl;  // CTA-uniform
            const V* mat = mats + op.mat + int64_t(inst) * op.mat_stride;
            if (ADJ && op.kind == QS_OP_EXPECT) {
                double2 v = make_double2(0.0, 0.0);
                if (on) {
                    if (op.flags & QS_OPF_DIAG) v = tile_expect_diag<V>(tile, tile2, K, base, op, mat);
                    else if (op.m == 1) v = tile_expect_dense<V, 1>(tile, tile2, K, op, mat);
                    else v = tile_expect_dense<V, 2>(tile, tile2, K, op, mat);
                }
                // block reduction in a fixed order (deterministic)
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) {
                    v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
                    v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
                }
                if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
                __syncthreads();
                if (threadIdx.x == 0) {
                    double2 s2 = make_double2(0.0, 0.0);
                    for (int w = 0; w < kFT / 32; ++w) { s2.x += red[w].x; s2.y += red[w].y; }
                    const uint64_t at = 2 * (uint64_t(op.slot) * ntiles + tid);
                    partials[at] = s2.x;
                    partials[at + 1] = s2.y;
                }
                __syncthreads();
                continue;
            }
            if (!on) continue;
            if (op.kind == QS_OP_DIAG) {
                tile_diag<V>(tile, K, base, op, mat);
                if (ADJ) tile_diag<V>(tile2, K, base, op, mat);
            } else {
                switch (op.m) {
                    case 1: tile_mat<V, 1>(tile, K, op, mat); if (ADJ) tile_mat<V, 1>(tile2, K, op, mat); break;
                    case 2: tile_mat<V, 2>(tile, K, op, mat); if (ADJ) tile_mat<V, 2>(tile2, K, op, mat); break;
                    case 3: tile_mat<V, 3>(tile, K, op, mat); if (ADJ) tile_mat<V, 3>(tile2, K, op, mat); break;
                    default: tile_mat<V, 4>(tile, K, op, mat); if (ADJ) tile_mat<V, 4>(tile2, K, op, mat); break;
                }
            }
            __syncthreads();
        }
        for (uint32_t e = threadIdx.x; e < T; e += kFT) {
            const uint64_t gi = base | hoff[e >> L] | (e & lmask);
            vec[gi] = tile[e];
            if (ADJ) vec2[gi] = tile2[e];
        }
        __syncthreads();
    }
}

// One register pass over the whole vector.  Tile order: strided over the
// grid; batched passes take contiguous runs of tiles instead, so that a CTA
// restages per-instance matrices once per instance rather than once per tile.
template <typename V, int R, bool EXP, bool BIG>
__global__ void __launch_bounds__(256, 1) k_fused_reg(V* __restrict__ vec, const __grid_constant__ RegArgs p,
                                                      const V* __restrict__ mats, double* __restrict__ partials) {
    const uint64_t ntiles = uint64_t(1) << (p.n - p.K);
    uint64_t tile = blockIdx.x, tend = ntiles, tstep = gridDim.x;
    if (p.batched) {
        const uint64_t chunk = (ntiles + gridDim.x - 1) / gridDim.x;
        tile = uint64_t(blockIdx.x) * chunk;
        tend = tile + chunk < ntiles ? tile + chunk : ntiles;
        tstep = 1;
    }
    // one call: the body is inlined once
    reg_tiles<V, R, EXP, BIG>(vec, p, p.st, p.ops, p.cp, p.eslot, mats, partials, tile, tend, tstep, false);
}

template <typename V, bool ADJ>
int launch_smem(V* vec, V* vec2, int n, const qs_pass& ps, const qs_op* ops, const V* mats, double* partials,
                cudaStream_t st) {
    static thread_local PassArgs args;
    args.n = n; args.k = ps.k; args.nlow = ps.nlow; args.nops = ps.op_count; args.inst_shift = ps.inst_shift;
    for (int t = 0; t < QS_MAX_TILE_BITS; ++t) args.hi[t] = t < ps.k - ps.nlow ? ps.hi[t] : 0;
    for (int i = 0; i < ps.op_count; ++i) args.ops[i] = ops[ps.op_begin + i];
    size_t smem = sizeof(V) * (size_t(1) << ps.k) * (ADJ ? 2 : 1) + sizeof(uint64_t) * (size_t(1) << (ps.k - ps.nlow));
    config_smem((const void*)k_fused_smem<V, ADJ>);
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_fused_smem<V, ADJ>, kFT, smem);
    if (occ < 1) occ = 1;
    uint64_t ntiles = uint64_t(1) << (n - ps.k);
    uint64_t cap = uint64_t(sm_count()) * occ;
    k_fused_smem<V, ADJ><<<unsigned(ntiles < cap ? ntiles : cap), kFT, smem, st>>>(vec, vec2, args, mats, partials);
    QS_CHECK_LAUNCH(ADJ ? "qs_adjoint_fused" : "qs_apply_fused(smem)");
    return QS_OK;
}

// Launch memo: a planned register pass (the used parts of its RegArgs) and its
// parameter block determine the generated source completely, so repeated
// launches of the same plan (a replayed circuit, a gradient loop) reuse the
// loaded kernel without generating and hashing the source again.
struct JitMemo {
    std::string src;       // kept until the kernel is ready on some device
    void* fn[64] = {nullptr};
    int occ[64] = {0};
};

std::mutex& memo_mu() {  // guards the memos and their table
    static std::mutex mu;
    return mu;
}
std::unordered_map<uint64_t, std::shared_ptr<JitMemo>>& memo_table() {
    static std::unordered_map<uint64_t, std::shared_ptr<JitMemo>> t;
    return t;
}
std::shared_ptr<JitMemo> get_memo(uint64_t key) {
    std::lock_guard<std::mutex> lock(memo_mu());
    auto it = memo_table().find(key);
    return it == memo_table().end() ? nullptr : it->second;
}
// the memo of `key`: `m`, or the one another thread put there first
std::shared_ptr<JitMemo> put_memo(uint64_t key, std::shared_ptr<JitMemo> m) {
    std::lock_guard<std::mutex> lock(memo_mu());
    if (memo_table().size() > 4096) memo_table().clear();  // bounded: plans are cheap to regenerate
    return memo_table().emplace(key, std::move(m)).first->second;
}

uint64_t fnv(uint64_t h, const void* p, size_t n) {
    const unsigned char* c = static_cast<const unsigned char*>(p);
    for (size_t i = 0; i < n; ++i) h = (h ^ c[i]) * 1099511628211ull;
    return h;
}

// The source depends on the plan's structure and on the entries' value
// classes, not on the matrix values: the key hashes exactly those, so a new
// parameter set of the same circuit reuses the compiled kernel.
uint64_t plan_key(const RegArgs& a, int R, size_t vsize, const std::vector<uint8_t>& classes) {
    uint64_t h = 1469598103934665603ull;
    const int hdr[] = {a.n, a.K, a.L, a.H, a.nT, a.nstages, a.nops, a.nmats, a.inst_shift, a.batched, a.nexp,
                       R, int(vsize)};
    h = fnv(h, hdr, sizeof(hdr));
    h = fnv(h, &a.pairmask, sizeof(a.pairmask));
    h = fnv(h, a.hi, sizeof(int) * size_t(a.H));
    h = fnv(h, a.eslot, sizeof(int) * size_t(a.nexp));
    h = fnv(h, a.st, sizeof(KStage) * size_t(a.nstages));
    h = fnv(h, a.ops, sizeof(KOp) * size_t(a.nops));
    for (int o = 0; o < a.nops; ++o) {  // the table layout, not where the tables sit (goff)
        const KCopy& c = a.cp[o];
        const int f[] = {int(c.soff), int(c.m), int(c.diag), int(c.stride != 0), c.perm[0], c.perm[1], c.perm[2],
                         c.perm[3]};
        h = fnv(h, f, sizeof(f));
    }
    static const int target = [] {
        const char* e = getenv("QS_JIT_THREADS_PER_SM");
        return e && *e ? atoi(e) : 0;
    }();
    h = fnv(h, &target, sizeof(target));
    const int single = jit_single_buffer(vsize == 16, a.batched || a.nexp > 0) ? 1 : 0;
    h = fnv(h, &single, sizeof(single));
    return fnv(h, classes.data(), classes.size());
}

// ------------------------------------------------------- plans kept between launches
// Planning a register pass (build_reg scores every set of R tile bits for
// every stage) and generating its parameter block take 0.1 - 1 ms of host
// time, several times what the pass itself takes on a small state.  Both are
// functions of the pass's description alone, so they are kept: a plan under
// the exact contents of the pass and its ops, and, per plan, the parameter
// blocks of the matrix values it last ran with (none for per-instance tables,
// whose values are read on the device).  Contents are compared in full, and the
// store is dropped whole as soon as plans and parameter blocks together exceed
// kPlanBytes (plans in use live on with their callers).  run() of a known
// circuit with the keys of its ops kept as well (B200): 10 qubits, 60 gates
// 239 -> 81 us; 20 qubits, 200 gates 619 -> 243 us; 25 qubits, 300 gates in
// complex64 1.84 -> 1.46 ms (the host planned longer than the GPU ran).
struct ParamSet {
    std::vector<unsigned char> values;  // the matrix entries the block was made from
    JitPass jp;
    uint64_t key = 0;                   // plan_key: structure and value classes
    std::shared_ptr<JitMemo> memo;
};
struct PassPlan;
struct PlanLaunch {
    RegArgs args;
    PassPlan* plan;        // the plan it belongs to
    std::vector<int> rem;  // positions of the pass's ops that had not run before this launch
    std::mutex mu;  // guards sets
    std::vector<std::shared_ptr<const ParamSet>> sets;
};
struct PassPlan {
    std::vector<unsigned char> content;
    std::vector<std::unique_ptr<PlanLaunch>> launches;
    int64_t bytes = 0;    // guarded by g_plan_mu, as is
    bool stored = false;  // whether g_plans holds it (bytes are then part of g_plan_bytes)
};
constexpr int64_t kPlanBytes = int64_t(64) << 20;
constexpr size_t kParamSets = 8;  // per launch

std::mutex g_plan_mu;  // guards the two below
std::unordered_map<uint64_t, std::shared_ptr<PassPlan>> g_plans;
int64_t g_plan_bytes = 0;

// Account for a change of a plan's bytes.  With g_plan_mu held.
void plan_bytes(PassPlan& plan, int64_t change) {
    plan.bytes += change;
    if (!plan.stored) return;
    g_plan_bytes += change;
    if (g_plan_bytes <= kPlanBytes) return;
    for (auto& p : g_plans) p.second->stored = false;
    g_plans.clear();
    g_plan_bytes = 0;
}
int64_t set_bytes(const ParamSet& ps) {
    return int64_t(sizeof(ParamSet) + ps.values.size() + 8 * ps.jp.params.size() + ps.jp.classes.size());
}

// Word-wise hash of a byte string (the contents themselves are compared).
uint64_t hash_bytes(uint64_t h, const void* p, size_t n) {
    const unsigned char* c = static_cast<const unsigned char*>(p);
    for (; n >= 8; n -= 8, c += 8) {
        uint64_t w;
        memcpy(&w, c, 8);
        h = (h ^ w) * 0x9e3779b97f4a7c15ull;
        h ^= h >> 29;
    }
    return n ? fnv(h, c, n) : h;
}

// The plan of a pass: every launch it splits into.  nullptr with the error set
// when an op does not fit.
std::shared_ptr<PassPlan> get_plan(const qs_pass& ps, const qs_op* ops, int n, int R, int nb) {
    static thread_local std::vector<unsigned char> content;
    const int head[] = {n, R, nb, ps.k, ps.nlow, ps.inst_shift, ps.pair, ps.op_count};
    const size_t hb = sizeof(head), pb = sizeof(ps.hi), ob = sizeof(qs_op) * size_t(ps.op_count);
    content.resize(hb + pb + ob);
    memcpy(content.data(), head, hb);
    memset(content.data() + hb, 0, pb);
    memcpy(content.data() + hb, ps.hi, sizeof(int32_t) * size_t(ps.k - ps.nlow));
    memcpy(content.data() + hb + pb, ops + ps.op_begin, ob);
    const uint64_t key = hash_bytes(1469598103934665603ull, content.data(), content.size());
    {
        std::lock_guard<std::mutex> lock(g_plan_mu);
        auto it = g_plans.find(key);
        if (it != g_plans.end() && it->second->content == content) return it->second;
    }
    auto plan = std::make_shared<PassPlan>();
    plan->content = content;
    std::vector<int> rem(ps.op_count);
    for (int i = 0; i < ps.op_count; ++i) rem[i] = i;
    while (!rem.empty()) {
        const int next = ps.op_begin + rem.front();
        auto L = std::make_unique<PlanLaunch>();
        L->plan = plan.get();
        L->rem = rem;
        if (build_reg(ps, ops, rem, n, R, nb, L->args) <= 0) {
            set_error("qs_apply_fused: op %d does not fit a register tile", next);
            return nullptr;
        }
        plan->launches.push_back(std::move(L));
    }
    std::lock_guard<std::mutex> lock(g_plan_mu);
    std::shared_ptr<PassPlan>& slot = g_plans[key];
    if (slot) {  // the same hash: another thread's plan of this pass, or another pass
        slot->stored = false;
        g_plan_bytes -= slot->bytes;
    }
    slot = plan;
    plan->stored = true;
    plan_bytes(*plan, int64_t(sizeof(PassPlan) + content.size() +
                              (sizeof(PlanLaunch) + sizeof(int) * rem.capacity()) * plan->launches.size()));
    return plan;
}

// The parameter block of a planned launch for the values in `hm` (kept when
// the launch has no per-instance tables); nullptr when it is not generated.
template <typename V>
std::shared_ptr<const ParamSet> get_params(PlanLaunch& L, int R, const V* hm) {
    const RegArgs& a = L.args;
    static thread_local std::vector<unsigned char> values;
    values.clear();
    if (!a.batched) {
        for (int o = 0; o < a.nops; ++o) {
            const KCopy& c = a.cp[o];
            const size_t cnt = size_t(1) << (c.diag ? c.m : 2 * c.m);
            const unsigned char* p = reinterpret_cast<const unsigned char*>(hm + c.goff);
            values.insert(values.end(), p, p + cnt * sizeof(V));
        }
        std::lock_guard<std::mutex> lock(L.mu);
        for (const auto& s : L.sets)
            if (s->values == values) return s;
    }
    auto ps = std::make_shared<ParamSet>();
    if (!gen_pass(&a, R, sizeof(V) == 16, hm, ps->jp, false)) return nullptr;
    ps->key = plan_key(a, R, sizeof(V), ps->jp.classes);
    ps->memo = get_memo(ps->key);
    if (!ps->memo) {
        auto m = std::make_shared<JitMemo>();
        JitPass full;
        if (!gen_pass(&a, R, sizeof(V) == 16, hm, full, true)) return nullptr;
        m->src.swap(full.src);
        ps->memo = put_memo(ps->key, m);
    }
    if (!a.batched) {
        ps->values = values;
        int64_t change = set_bytes(*ps);
        {
            std::lock_guard<std::mutex> lock(L.mu);
            if (L.sets.size() >= kParamSets) {
                change -= set_bytes(*L.sets.front());
                L.sets.erase(L.sets.begin());
            }
            L.sets.push_back(ps);
        }
        std::lock_guard<std::mutex> lock(g_plan_mu);
        plan_bytes(*L.plan, change);
    }
    return ps;
}

// The run-time compiled kernel of a planned register pass with its parameter
// block.  fn is null when the compiler does not have it ready (mode SYNC: after
// compiling it; ASYNC: it is queued from here on) or the pass is not generated.
struct JitKernel {
    std::shared_ptr<const ParamSet> ps;
    void* fn = nullptr;
    int occ = 0;
};
template <typename V>
JitKernel jit_kernel(PlanLaunch& L, int R, const V* hm, cudaStream_t st) {
    JitKernel k;
    const int jm = jit::mode();
    int dev = 0;
    if (jm == QS_JIT_OFF || hm == nullptr || !(k.ps = get_params<V>(L, R, hm))) return k;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        k.ps = nullptr;
        return k;
    }
    JitMemo& m = *k.ps->memo;
    std::string src;
    {
        std::lock_guard<std::mutex> lock(memo_mu());
        k.fn = m.fn[dev];
        k.occ = m.occ[dev];
        if (k.fn == nullptr) src = m.src;
    }
    if (k.fn != nullptr) return k;
    // during stream capture nothing is compiled or loaded: a kernel that is
    // not loaded yet on this device leaves the pass to the generic kernel
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) cs = cudaStreamCaptureStatusActive;
    const bool capturing = cs != cudaStreamCaptureStatusNone;
    if (src.empty()) {  // loaded on another device only: regenerate the text
        JitPass full;
        if (!gen_pass(&L.args, R, sizeof(V) == 16, hm, full, true)) {
            k.ps = nullptr;
            return k;
        }
        src.swap(full.src);
    }
    k.fn = jit::lookup(src, "qs_pass", jm == QS_JIT_SYNC && !capturing, !capturing, k.ps->jp.threads, k.ps->jp.smem, &k.occ);
    if (k.fn != nullptr) {
        std::lock_guard<std::mutex> lock(memo_mu());
        m.fn[dev] = k.fn;
        m.occ[dev] = k.occ;
        std::string().swap(m.src);
    }
    return k;
}

// Launch that kernel; returns 1 when it was launched, 0 when the generic kernel
// has to run, < 0 on error.
template <typename V>
int launch_jit(V* vec, PlanLaunch& L, int R, const V* hm, const V* mats, double* partials, cudaStream_t st) {
    const JitKernel k = jit_kernel<V>(L, R, hm, st);
    if (!k.ps) return 0;
    if (k.fn == nullptr) {
        jit::count_launch(false);
        return 0;
    }
    const JitPass& jp = k.ps->jp;
    const uint64_t ntiles = uint64_t(1) << (L.args.n - L.args.K);
    const uint64_t cap = uint64_t(sm_count()) * uint64_t(k.occ < 1 ? 1 : k.occ);
    void* vp = vec;
    const void* mp = mats;
    void* pp = partials;
    void* params[] = {&vp, const_cast<uint64_t*>(jp.params.data()), &mp, &pp};
    const int rc = jit::launch(k.fn, unsigned(ntiles < cap ? ntiles : cap), unsigned(jp.threads), jp.smem, st, params);
    if (rc) return rc;
    jit::count_launch(true);
    return 1;
}

// Register bits per thread of generated passes.  complex128: 4, as the generic
// kernel.  complex64: 4 where a tile of 2^k amplitudes then has at most 256
// threads (k <= 12), else the generic kernel's 5.  Half the amplitudes per
// thread leave registers for three times the warps: three CTAs of 256 threads an
// SM issue 3.0 instructions a cycle (of 4), the FMA pipe 52 - 55 % active.  4
// against 5 (B200, k = 12): 30-qubit spread circuit of 1000 gates 147.6 against
// 163.2 ms (139.2 at nlow = 5), 28 qubits, 400 gates 14.4 against 15.6 ms, 24
// qubits 643 against 845 us, 18 qubits 27 against 37 us.  QS_JIT_REG_BITS (4 or
// 5) overrides both.
inline int jit_reg_bits(int generic_r, int k) {
    static const int env_r = [] {
        const char* e = getenv("QS_JIT_REG_BITS");
        const int v = e && *e ? atoi(e) : 0;
        return (v == 4 || v == 5) ? v : 0;
    }();
    if (env_r) return env_r;
    return generic_r == 5 && k <= 12 ? 4 : generic_r;
}

template <typename V, int R, bool EXP, bool BIG>
int launch_reg_k(V* vec, int n, const qs_pass& ps, const qs_op* ops, const V* mats, double* partials, cudaStream_t st,
                 const V* hm = nullptr) {
    const int nb = sizeof(V) == 16 ? 3 : 4;  // bank-group bits of a shared-memory phase
    const int RJ = jit_reg_bits(R, ps.k);
    qs_pass rest = ps;
    std::vector<qs_op> rest_ops;
    if (RJ != R && ps.k - RJ >= 5 && ps.k - RJ <= 8 && hm != nullptr && jit::mode() != QS_JIT_OFF) {
        // a generated pass with its own register width has its own plan; from
        // the first launch that is not ready on, the generic kernel's plan of
        // the remaining ops takes over
        if (const std::shared_ptr<PassPlan> plan = get_plan(ps, ops, n, RJ, nb)) {
            size_t done = 0;
            for (; done < plan->launches.size(); ++done) {
                const int jr = launch_jit<V>(vec, *plan->launches[done], RJ, hm, mats, partials, st);
                if (jr < 0) return jr;
                if (jr == 0) break;
            }
            if (done == plan->launches.size()) return QS_OK;
            // the ones after it do not run now, but are queued with it
            for (size_t li = done + 1; jit::mode() == QS_JIT_ASYNC && li < plan->launches.size(); ++li)
                jit_kernel<V>(*plan->launches[li], RJ, hm, st);
            for (int i : plan->launches[done]->rem) rest_ops.push_back(ops[ps.op_begin + i]);
            rest.op_begin = 0;
            rest.op_count = int(rest_ops.size());
            ops = rest_ops.data();
        }
    }
    const std::shared_ptr<PassPlan> plan = get_plan(rest, ops, n, R, nb);
    if (!plan) return QS_EINVAL;
    for (const auto& L : plan->launches) {
        const RegArgs& args = L->args;
        if (RJ == R) {
            const int jr = launch_jit<V>(vec, *L, R, hm, mats, partials, st);
            if (jr < 0) return jr;
            if (jr == 1) continue;
        }
        config_smem((const void*)k_fused_reg<V, R, EXP, BIG>);
        const int threads = 1 << (ps.k - R);
        const size_t smem = reg_smem_bytes<V>(args, R, EXP);
        if (smem > size_t(smem_optin())) {
            set_error("qs_apply_fused: a register pass needs %zu bytes of shared memory", smem);
            return QS_EINVAL;
        }
        uint64_t ntiles = uint64_t(1) << (n - ps.k);
        // persistent grid: as many CTAs as fit on the SMs at once (smaller
        // tiles run several CTAs per SM, whose relayouts and arithmetic overlap)
        int occ = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_fused_reg<V, R, EXP, BIG>, threads, smem);
        if (occ < 1) occ = 1;
        uint64_t cap = uint64_t(sm_count()) * uint64_t(occ);
        k_fused_reg<V, R, EXP, BIG><<<unsigned(ntiles < cap ? ntiles : cap), threads, smem, st>>>(vec, args, mats, partials);
        QS_CHECK_LAUNCH(EXP ? "qs_adjoint_pair" : "qs_apply_fused(reg)");
    }
    return QS_OK;
}

// Dense ops on 3 or 4 targets, and controlled dense ops, need the BIG kernel
// variant (adjoint pair passes take dense ops on at most 2 bits; their BIG
// variant only adds the controlled paths).
template <typename V, int R, bool EXP>
int launch_reg(V* vec, int n, const qs_pass& ps, const qs_op* ops, const V* mats, double* partials, cudaStream_t st,
               const V* hm = nullptr) {
    bool big = false;
    for (int i = 0; i < ps.op_count; ++i) {
        const qs_op& op = ops[ps.op_begin + i];
        const bool diag = op.kind == QS_OP_DIAG || (op.kind == QS_OP_EXPECT && (op.flags & QS_OPF_DIAG));
        if (op.m >= 3 && !diag) big = true;
        // dense here: MAT, and the anti-diagonal / swap ops that are not plain
        // exchanges (they run as dense matrices)
        const bool dense = op.kind == QS_OP_MAT ||
                           ((op.kind == QS_OP_ANTI || op.kind == QS_OP_SWAP) && !(op.flags & QS_OPF_UNIT));
        if (dense && op.lctrl != 0) big = true;
    }
    if constexpr (EXP) {
        for (int i = 0; i < ps.op_count; ++i) {
            const qs_op& op = ops[ps.op_begin + i];
            const bool diag = op.kind == QS_OP_DIAG || (op.kind == QS_OP_EXPECT && (op.flags & QS_OPF_DIAG));
            if (op.m >= 3 && !diag) {
                set_error("qs_adjoint_pair: pass ops act densely on at most 2 bits");
                return QS_EINVAL;
            }
        }
        return big ? launch_reg_k<V, R, true, true>(vec, n, ps, ops, mats, partials, st, hm)
                   : launch_reg_k<V, R, true, false>(vec, n, ps, ops, mats, partials, st, hm);
    } else {
        return big ? launch_reg_k<V, R, false, true>(vec, n, ps, ops, mats, partials, st, hm)
                   : launch_reg_k<V, R, false, false>(vec, n, ps, ops, mats, partials, st, hm);
    }
}

template <typename V>
constexpr int reg_bits() { return sizeof(V) == 16 ? 4 : 5; }

template <typename V>
int launch_pass(V* vec, int n, const qs_pass& ps, const qs_op* ops, const V* mats, cudaStream_t st,
                const V* hm = nullptr) {
    constexpr int R = reg_bits<V>();
    const int nT = ps.k - R;
    const size_t smem = sizeof(V) * (2 * (size_t(1) << ps.k) + QS_MAX_PASS_MATS) + 8 * ((size_t(1) << (ps.k - ps.nlow)) + (1 << R)) +
                        sizeof(KOp) * QS_MAX_PASS_OPS + 16 + sizeof(KStage) * kMaxStages + QS_MAX_PASS_MATS;
    if (nT >= 5 && nT <= 8 && ps.nlow >= 5 && smem <= size_t(smem_optin()))
        return launch_reg<V, R, false>(vec, n, ps, ops, mats, nullptr, st, hm);
    return launch_smem<V, false>(vec, nullptr, n, ps, ops, mats, nullptr, st);
}

}  // namespace

}  // namespace qs

using namespace qs;

extern "C" int64_t qs_plan_store_bytes(void) {
    std::lock_guard<std::mutex> lock(g_plan_mu);
    return g_plan_bytes;
}

extern "C" int qs_apply_fused(void* vec, int n, int dtype, const qs_pass* passes, int npasses, const qs_op* ops,
                              int64_t nops_total, const void* mats_dev, int64_t mats_count, void* stream) {
    return qs_apply_fused_ex(vec, n, dtype, passes, npasses, ops, nops_total, mats_dev, nullptr, mats_count, stream);
}

extern "C" int qs_apply_fused_ex(void* vec, int n, int dtype, const qs_pass* passes, int npasses, const qs_op* ops,
                                 int64_t nops_total, const void* mats_dev, const void* mats_host, int64_t mats_count,
                                 void* stream) {
    QS_REQUIRE(vec != nullptr, "null state vector");
    QS_REQUIRE(n >= 1 && n <= 40, "qubit count %d outside [1, 40]", n);
    QS_REQUIRE(valid_dtype(dtype), "bad dtype %d", dtype);
    QS_REQUIRE(npasses >= 0 && (npasses == 0 || passes != nullptr), "bad pass array");
    QS_REQUIRE(nops_total >= 0 && (nops_total == 0 || ops != nullptr), "bad op array");
    QS_REQUIRE(mats_count >= 0 && (mats_count == 0 || mats_dev != nullptr), "bad matrix table");
    size_t vsize = dtype == QS_C128 ? 16 : 8;
    for (int i = 0; i < npasses; ++i) {
        int rc = validate_pass(passes[i], n, ops, nops_total, mats_count);
        if (rc) return rc;
        size_t smem = vsize * (size_t(1) << passes[i].k) + 8 * (size_t(1) << (passes[i].k - passes[i].nlow));
        QS_REQUIRE(smem <= 160 * 1024, "pass %d: tile of 2^%d needs %zu bytes of shared memory", i, passes[i].k, smem);
    }
    for (int i = 0; i < npasses; ++i) {
        if (passes[i].op_count == 0) continue;
        int rc = dtype == QS_C128
                     ? launch_pass<double2>((double2*)vec, n, passes[i], ops, (const double2*)mats_dev,
                                            as_stream(stream), (const double2*)mats_host)
                     : launch_pass<float2>((float2*)vec, n, passes[i], ops, (const float2*)mats_dev,
                                           as_stream(stream), (const float2*)mats_host);
        if (rc) return rc;
    }
    return QS_OK;
}

extern "C" int qs_adjoint_fused(void* psi, void* lam, int n, int dtype, const qs_pass* passes, int npasses,
                                const qs_op* ops, int64_t nops_total, const void* mats_dev, int64_t mats_count,
                                double* partials_dev, int64_t partials_count, void* stream) {
    QS_REQUIRE(psi != nullptr && lam != nullptr && psi != lam, "psi and lam must be distinct non-null vectors");
    QS_REQUIRE(n >= 1 && n <= 40, "qubit count %d outside [1, 40]", n);
    QS_REQUIRE(valid_dtype(dtype), "bad dtype %d", dtype);
    QS_REQUIRE(npasses >= 0 && (npasses == 0 || passes != nullptr), "bad pass array");
    QS_REQUIRE(nops_total >= 0 && (nops_total == 0 || ops != nullptr), "bad op array");
    QS_REQUIRE(mats_count >= 0 && (mats_count == 0 || mats_dev != nullptr), "bad matrix table");
    QS_REQUIRE(partials_count >= 0 && (partials_count == 0 || partials_dev != nullptr), "bad partials buffer");
    size_t vsize = dtype == QS_C128 ? 16 : 8;
    for (int i = 0; i < npasses; ++i) {
        int rc = validate_pass(passes[i], n, ops, nops_total, mats_count, true, partials_count);
        if (rc) return rc;
        size_t smem = 2 * vsize * (size_t(1) << passes[i].k) + 8 * (size_t(1) << (passes[i].k - passes[i].nlow));
        QS_REQUIRE(smem <= 160 * 1024, "pass %d: two tiles of 2^%d need %zu bytes of shared memory", i,
                   passes[i].k, smem);
    }
    for (int i = 0; i < npasses; ++i) {
        if (passes[i].op_count == 0) continue;
        int rc = dtype == QS_C128
                     ? launch_smem<double2, true>((double2*)psi, (double2*)lam, n, passes[i], ops,
                                                  (const double2*)mats_dev, partials_dev, as_stream(stream))
                     : launch_smem<float2, true>((float2*)psi, (float2*)lam, n, passes[i], ops,
                                                 (const float2*)mats_dev, partials_dev, as_stream(stream));
        if (rc) return rc;
    }
    return QS_OK;
}

extern "C" int qs_adjoint_pair(void* psilam, int n, int dtype, const qs_pass* passes, int npasses, const qs_op* ops,
                               int64_t nops_total, const void* mats_dev, int64_t mats_count, double* partials_dev,
                               int64_t partials_count, void* stream) {
    return qs_adjoint_pair_ex(psilam, n, dtype, passes, npasses, ops, nops_total, mats_dev, nullptr, mats_count,
                              partials_dev, partials_count, stream);
}

extern "C" int qs_adjoint_pair_ex(void* psilam, int n, int dtype, const qs_pass* passes, int npasses,
                                  const qs_op* ops, int64_t nops_total, const void* mats_dev, const void* mats_host,
                                  int64_t mats_count, double* partials_dev, int64_t partials_count, void* stream) {
    QS_REQUIRE(psilam != nullptr, "null vector");
    QS_REQUIRE(n >= 2 && n <= 41, "bit count %d outside [2, 41]", n);
    QS_REQUIRE(valid_dtype(dtype), "bad dtype %d", dtype);
    QS_REQUIRE(npasses >= 0 && (npasses == 0 || passes != nullptr), "bad pass array");
    QS_REQUIRE(nops_total >= 0 && (nops_total == 0 || ops != nullptr), "bad op array");
    QS_REQUIRE(mats_count >= 0 && (mats_count == 0 || mats_dev != nullptr), "bad matrix table");
    QS_REQUIRE(partials_count >= 0 && (partials_count == 0 || partials_dev != nullptr), "bad partials buffer");
    const int R = dtype == QS_C128 ? reg_bits<double2>() : reg_bits<float2>();
    for (int i = 0; i < npasses; ++i) {
        int rc = validate_pass(passes[i], n, ops, nops_total, mats_count, true, partials_count);
        if (rc) return rc;
        QS_REQUIRE(passes[i].pair > 0, "pass %d: no pair bit", i);
        const int nT = passes[i].k - R;
        QS_REQUIRE(nT >= 5 && nT <= 8 && passes[i].nlow >= 5, "pass %d: tile 2^%d / nlow %d is not a register tile", i,
                   passes[i].k, passes[i].nlow);
    }
    for (int i = 0; i < npasses; ++i) {
        if (passes[i].op_count == 0) continue;
        int rc = dtype == QS_C128
                     ? launch_reg<double2, reg_bits<double2>(), true>((double2*)psilam, n, passes[i], ops,
                                                                      (const double2*)mats_dev, partials_dev,
                                                                      as_stream(stream), (const double2*)mats_host)
                     : launch_reg<float2, reg_bits<float2>(), true>((float2*)psilam, n, passes[i], ops,
                                                                    (const float2*)mats_dev, partials_dev,
                                                                    as_stream(stream), (const float2*)mats_host);
        if (rc) return rc;
    }
    return QS_OK;
}

namespace {

// Launch `launch_index` of one register pass as its generated kernel (source,
// parameter block), without a device.
int generated_launch(const char* who, int n, int dtype, const qs_pass* pass, const qs_op* ops, int64_t nops_total,
                     const void* mats_host, int64_t mats_count, int launch_index, JitPass& jp) {
    QS_REQUIRE(n >= 1 && n <= 40, "qubit count %d outside [1, 40]", n);
    QS_REQUIRE(valid_dtype(dtype), "bad dtype %d", dtype);
    QS_REQUIRE(pass != nullptr && mats_host != nullptr, "null argument");
    QS_REQUIRE(launch_index >= 0, "negative launch index");
    // pair passes (adjoint) carry EXPECT ops; their partials buffer is not touched here
    int rc = validate_pass(*pass, n, ops, nops_total, mats_count, pass->pair > 0, INT64_MAX / 4);
    if (rc) return rc;
    const int R = jit_reg_bits(dtype == QS_C128 ? reg_bits<double2>() : reg_bits<float2>(), pass->k);
    const int nT = pass->k - R;
    if (!(nT >= 5 && nT <= 8 && pass->nlow >= 5)) {
        set_error("%s: tile 2^%d / nlow %d is not a register tile", who, pass->k, pass->nlow);
        return QS_ENOTSUP;
    }
    static thread_local RegArgs args;
    std::vector<int> rem(pass->op_count);
    for (int i = 0; i < pass->op_count; ++i) rem[i] = i;
    for (int li = 0; li <= launch_index; ++li) {
        if (rem.empty()) {
            set_error("%s: the pass has %d launches", who, li);
            return QS_EINVAL;
        }
        if (build_reg(*pass, ops, rem, n, R, dtype == QS_C128 ? 3 : 4, args) <= 0) {
            set_error("%s: an op does not fit a register tile", who);
            return QS_EINVAL;
        }
    }
    if (!gen_pass(&args, R, dtype == QS_C128, mats_host, jp, true)) {
        set_error("%s: this launch is not generated (batched, EXPECT ops or parameters too large)", who);
        return QS_ENOTSUP;
    }
    return QS_OK;
}

}  // namespace

extern "C" int qs_jit_pass_source(int n, int dtype, const qs_pass* pass, const qs_op* ops, int64_t nops_total,
                                  const void* mats_host, int64_t mats_count, int launch_index, char* out,
                                  size_t out_size, int64_t* src_len) {
    QS_REQUIRE(src_len != nullptr, "null argument");
    JitPass jp;
    const int rc = generated_launch("qs_jit_pass_source", n, dtype, pass, ops, nops_total, mats_host, mats_count,
                                    launch_index, jp);
    if (rc) return rc;
    *src_len = int64_t(jp.src.size());
    if (out != nullptr && out_size > 0) {
        const size_t k = jp.src.size() < out_size - 1 ? jp.src.size() : out_size - 1;
        memcpy(out, jp.src.data(), k);
        out[k] = 0;
    }
    return QS_OK;
}

extern "C" int qs_jit_pass_params(int n, int dtype, const qs_pass* pass, const qs_op* ops, int64_t nops_total,
                                  const void* mats_host, int64_t mats_count, int launch_index, void* out,
                                  size_t out_size, int64_t* bytes) {
    QS_REQUIRE(bytes != nullptr, "null argument");
    JitPass jp;
    const int rc = generated_launch("qs_jit_pass_params", n, dtype, pass, ops, nops_total, mats_host, mats_count,
                                    launch_index, jp);
    if (rc) return rc;
    *bytes = int64_t(8 * jp.params.size());
    if (out != nullptr) memcpy(out, jp.params.data(), out_size < 8 * jp.params.size() ? out_size : 8 * jp.params.size());
    return QS_OK;
}
