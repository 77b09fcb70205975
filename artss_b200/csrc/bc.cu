// Boundary conditions as compiled assignment programs.
//
// The reference applies boundary conditions as a sequence of per-patch loops
// (ARTSS src/domain/Multigrid.cpp:555-572): obstacles in id order, each over
// its six patches, then the six domain patches LEFT..BACK, each cell doing
// x[t] = sign * x[t + ref] + value.  Later writes win on edges and corners and
// some assignments read cells an earlier one wrote.  Running that sequence as
// one GPU pass per patch would cost 6 + 6*obstacles launches per call.
//
// Here the host compiles the sequence once per (level, field type):
//   1. dead writes (overwritten before anyone reads them) are dropped;
//   2. read-after-write chains are folded: an assignment whose source was
//      written earlier re-evaluates that chain from its root cell, step by
//      step with the same roundings, so it no longer reads the intermediate;
//   3. the remaining ordering constraints (a cell read before it is written,
//      chains longer than kBcMaxDepth) are resolved by wave numbers;
//   4. a program of several waves (obstacles that touch each other) is also folded
//      onto the values from before it (flatten_bc), which needs no order but reads
//      before writes.
// The device executes one kernel per program (one per wave where a chain is too
// long for 4).  Results are identical to the sequential loops.
#include "internal.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <unordered_map>

namespace artss {

// A program as the kernels take it: assignments [begin, end) of a wave, or a flat
// program with its hazards first.
struct BcRun {
    double *f;
    const int64_t *target, *root;
    const uint8_t *depth, *neg;
    const double *value;
    int64_t begin, end, n;  // n: stride of value
    int64_t hazards;        // flat programs: the first block's share, staged in shared memory
};

// loop step of the last block of a launch; partials = nullptr: none
struct BcStep {
    const double *partials;
    int nblocks;
    const LoopState *rd;
    LoopState *wr;
    double tol;
    long long max_it;
};

// block `block` of `blocks` of a program
__device__ __forceinline__ void bc_blocks(const BcRun &p, int block, int blocks, const LoopState *pred, double *staged) {
    // FLAT: its values depend on cells from before the program only, so the
    // assignments may run in any order as long as every read of a cell comes before its
    // write: block 0 reads for all hazards, then writes them; the other blocks'
    // assignments touch no cell that another one touches
    const bool first = p.hazards > 0 && block == 0;
    const int64_t end = first ? p.hazards : p.end;
    int64_t q = (first ? 0 : p.begin + p.hazards) + threadIdx.x;
    int64_t stride = blockDim.x;
    if (!first) {
        const int skip = p.hazards > 0 ? 1 : 0;
        q += (int64_t) (block - skip) * blockDim.x;
        stride *= blocks - skip;
    }
    // the program's tables are constant: the first assignment's entries are
    // read before waiting for the kernel that wrote f
    int64_t t = 0, r = 0;
    int d = 0;
    uint8_t m = 0;
    double val[kBcMaxDepth];
    auto entry = [&]() {
        if (q < end) {
            t = p.target[q];
            r = p.root[q];
            d = p.depth[q] & ~kBcLagged;
            m = p.neg[q];
        }
#pragma unroll
        for (int s = 0; s < kBcMaxDepth; s++) val[s] = (q < end && s < d) ? p.value[s * p.n + q] : 0.0;
    };
    entry();
    pdl_wait();
    pdl_trigger();
    if (pred && !pred->cond) return;
    while (q < end) {
        double x = p.f[r];
#pragma unroll
        for (int s = 0; s < kBcMaxDepth; s++)
            if (s < d) x = ((m >> s) & 1 ? -x : x) + val[s];
        if (first) staged[q] = x;
        else p.f[t] = x;
        q += stride;
        if (q < end) entry();
    }
    if (first) {
        __syncthreads();
        for (int64_t h = threadIdx.x; h < p.hazards; h += blockDim.x) p.f[p.target[h]] = staged[h];
    }
}

__global__ void k_bc(BcRun p, BcStep step, const LoopState *__restrict__ pred) {
    extern __shared__ double staged[];  // [hazards]
    __shared__ double smem[32];
    const int blocks = (int) gridDim.x - (step.partials ? 1 : 0);
    if ((int) blockIdx.x == blocks) {
        pdl_wait();
        pdl_trigger();
        artss_loop_step(step.partials, step.nblocks, step.rd, step.wr, step.tol, step.max_it, smem);
        return;
    }
    bc_blocks(p, (int) blockIdx.x, blocks, pred, staged);
}

// three programs side by side, a row of blocks each
__global__ void k_bc3(BcRun a, BcRun b, BcRun c) {
    extern __shared__ double staged[];
    bc_blocks(blockIdx.y == 0 ? a : blockIdx.y == 1 ? b : c, (int) blockIdx.x, (int) gridDim.x, nullptr, staged);
}

namespace {

// the program as one launch, or false (several waves, not folded)
bool one_run(const BcProgram &p, double *f, BcRun *r) {
    if (p.flat.n) {
        const BcProgram::Flat &x = p.flat;
        *r = BcRun{f, x.d_target, x.d_root, x.d_depth, x.d_neg, x.d_value, 0, x.n, x.n, x.hazards};
        return true;
    }
    if (p.waves > 1) return false;
    *r = BcRun{f, p.d_target, p.d_root, p.d_depth, p.d_neg, p.d_value, p.wave_begin[0], p.wave_begin[p.waves], p.n, 0};
    return true;
}
unsigned run_blocks(const BcRun &r) {
    const int64_t rest = r.end - r.begin - r.hazards;
    return (r.hazards > 0 ? 1u : 0u) + (rest > 0 ? flat_blocks(rest) : 0u);
}

}  // namespace

// One launch for a program of one wave or a flat one, else one per wave.  On the
// room with a door (32^3, seven touching walls, 10952 assignments in three waves of
// 10836, 114 and 2) the flat form takes 57 launches a step instead of 171.
int apply_bc(artss_ctx *ctx, double *f, int level, int field_type, const LoopState *pred) {
    const BcProgram &p = ctx->bc[level][field_type];
    if (!p.present || p.n == 0) return ARTSS_OK;
    BcRun r{};
    if (one_run(p, f, &r)) {
        ARTSS_LAUNCH_PDL(ctx, FAM_BC, k_bc, run_blocks(r), 256, r.hazards * sizeof(double), r, BcStep{}, pred);
        ARTSS_LAUNCH_CK(ctx);
        return ARTSS_OK;
    }
    for (int w = 0; w < p.waves; w++) {
        r = BcRun{f, p.d_target, p.d_root, p.d_depth, p.d_neg, p.d_value, p.wave_begin[w], p.wave_begin[w + 1], p.n, 0};
        if (r.end <= r.begin) continue;
        ARTSS_LAUNCH_PDL(ctx, FAM_BC, k_bc, run_blocks(r), 256, 0, r, BcStep{}, pred);
        ARTSS_LAUNCH_CK(ctx);
    }
    return ARTSS_OK;
}

int apply_bc_step(artss_ctx *ctx, double *f, int level, int field_type, int slot, int parity, int nblocks, double tol,
                  long long max_it) {
    const BcProgram &p = ctx->bc[level][field_type];
    const LoopState *rd = ctx->d_loop + slot + parity;
    BcRun r{};
    if (p.present && p.n > 0 && one_run(p, f, &r)) {
        static_assert(kReduceThreads == 256, "the step block has the program's block size");
        const BcStep s{ctx->d_partials, nblocks, rd, ctx->d_loop + slot + 1 - parity, tol, max_it};
        ARTSS_LAUNCH_PDL(ctx, FAM_BC, k_bc, run_blocks(r) + 1, 256, r.hazards * sizeof(double), r, s, rd);
        ARTSS_LAUNCH_CK(ctx);
        return ARTSS_OK;
    }
    int st = apply_bc(ctx, f, level, field_type, rd);
    return st ? st : finalize_loop_pair(ctx, slot, parity, nblocks, tol, max_it);
}

int apply_bc_uvw(artss_ctx *ctx, double *u, double *v, double *w) {
    double *f[3] = {u, v, w};
    const int ft[3] = {ARTSS_FIELD_U, ARTSS_FIELD_V, ARTSS_FIELD_W};
    BcRun r[3]{};
    bool one = u != v && v != w && u != w;
    unsigned blocks = 0;
    int64_t hazards = 0;
    for (int c = 0; c < 3 && one; c++) {
        const BcProgram &p = ctx->bc[0][ft[c]];
        one = p.present && p.n > 0 && one_run(p, f[c], &r[c]);
        if (!one) break;
        blocks = std::max(blocks, run_blocks(r[c]));
        hazards = std::max(hazards, r[c].hazards);
    }
    if (one) {
        ARTSS_LAUNCH_PDL(ctx, FAM_BC, k_bc3, dim3(blocks, 3), 256, hazards * sizeof(double), r[0], r[1], r[2]);
        ARTSS_LAUNCH_CK(ctx);
        return ARTSS_OK;
    }
    int st = ARTSS_OK;
    for (int c = 0; c < 3 && !st; c++) st = apply_bc(ctx, f[c], 0, ft[c]);
    return st;
}

// The boundary program with every value taken as zero, on FP32 storage: the
// homogeneous conditions of a correction equation (mixed-precision pressure
// solve); only the sign chain of each folded assignment remains.
__global__ void k_bc_wave_f32(float *__restrict__ f, const int64_t *__restrict__ target,
                              const int64_t *__restrict__ root, const uint8_t *__restrict__ depth,
                              const uint8_t *__restrict__ neg, int64_t begin, int64_t end,
                              const LoopState *__restrict__ pred) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (pred && !pred->cond) return;
    for (int64_t q = begin + blockIdx.x * (int64_t) blockDim.x + threadIdx.x; q < end;
         q += (int64_t) gridDim.x * blockDim.x) {
        const int d = depth[q];
        const unsigned flips = __popc((unsigned) neg[q] & ((1u << d) - 1u));
        const float x = f[root[q]];
        f[target[q]] = (flips & 1u) ? -x : x;
    }
}

int apply_bc_f32(artss_ctx *ctx, float *f, int level, int field_type, const LoopState *pred) {
    const BcProgram &p = ctx->bc[level][field_type];
    if (!p.present || p.n == 0) return ARTSS_OK;
    for (int w = 0; w < p.waves; w++) {
        const int64_t b = p.wave_begin[w], e = p.wave_begin[w + 1];
        if (e <= b) continue;
        ARTSS_LAUNCH_PDL(ctx, FAM_BC, k_bc_wave_f32, flat_blocks(e - b), 256, 0, 
                                      f, p.d_target, p.d_root, p.d_depth, p.d_neg, b, e, pred);
        ARTSS_LAUNCH_CK(ctx);
    }
    return ARTSS_OK;
}

namespace {

struct Folded {
    int64_t target;
    int64_t root;
    int depth;
    uint8_t neg;
    double value[kBcMaxDepth];
    int wave;
};

}  // namespace

// Compile the ordered assignment list; exposed for the host-side unit test.
int compile_bc(const artss_bc_assign *ops, int64_t n, std::vector<Folded> &out, int &waves) {
    out.clear();
    waves = 0;
    // 1. dead-write elimination, scanning backwards
    std::vector<char> live(n, 0);
    {
        std::unordered_map<int64_t, char> overwritten;  // true: a later live write precedes any read
        overwritten.reserve(n * 2 + 1);
        for (int64_t k = n - 1; k >= 0; k--) {
            auto it = overwritten.find(ops[k].target);
            if (it != overwritten.end() && it->second) continue;  // dead
            live[k] = 1;
            overwritten[ops[k].target] = 1;
            overwritten[ops[k].source] = 0;
        }
    }
    // 2./3. forward pass: fold chains, assign waves
    std::unordered_map<int64_t, int64_t> last_writer;  // cell -> index in out
    std::unordered_map<int64_t, int> max_reader_wave;  // cell -> max wave of ops reading it
    std::unordered_map<int64_t, int> last_write_wave;  // cell -> wave of last write
    out.reserve(n);
    for (int64_t k = 0; k < n; k++) {
        if (!live[k]) continue;
        const artss_bc_assign &a = ops[k];
        Folded f{};
        f.target = a.target;
        int wave = 0;
        auto lw = last_writer.find(a.source);
        bool folded = false;
        if (lw != last_writer.end()) {
            const Folded &prev = out[lw->second];
            // fold only if the chain's root has not been written since it was read
            const bool root_written = last_writer.count(prev.root) != 0;
            if (prev.depth < kBcMaxDepth && !root_written) {
                f.root = prev.root;
                f.depth = prev.depth + 1;
                f.neg = prev.neg;
                for (int s = 0; s < prev.depth; s++) f.value[s] = prev.value[s];
                f.neg |= (a.sign < 0 ? 1 : 0) << prev.depth;
                f.value[prev.depth] = a.value;
                folded = true;
            } else {
                wave = std::max(wave, prev.wave + 1);
            }
        }
        if (!folded) {
            f.root = a.source;
            f.depth = 1;
            f.neg = a.sign < 0 ? 1 : 0;
            f.value[0] = a.value;
        }
        auto mr = max_reader_wave.find(a.target);
        if (mr != max_reader_wave.end()) wave = std::max(wave, mr->second + 1);
        auto ww = last_write_wave.find(a.target);
        if (ww != last_write_wave.end()) wave = std::max(wave, ww->second + 1);
        f.wave = wave;
        last_writer[a.target] = (int64_t) out.size();
        last_write_wave[a.target] = wave;
        auto &r = max_reader_wave[f.root];
        r = std::max(r, wave);
        waves = std::max(waves, wave + 1);
        out.push_back(f);
    }
    return ARTSS_OK;
}

// The ordered assignments as one assignment per target on the values from before
// the program: each assignment's source is replaced by the chain that last wrote
// it.  A step with a zero added joins the one before it where the result is the
// same for every x: (s1 x + z1) then (s2 y + z2) with z1 = -0 (which changes
// nothing) is s1 s2 x + z2, and z2 = +0 (which turns a -0 into +0) is s1 s2 x + 0
// for z1 = +0 as well.  False when a chain stays longer than kBcMaxDepth.
bool flatten_bc(const artss_bc_assign *ops, int64_t n, std::vector<Folded> &out) {
    struct Chain {
        int64_t root;
        int depth;
        uint8_t neg;
        double value[kBcMaxDepth];
    };
    std::unordered_map<int64_t, Chain> now;
    now.reserve((size_t) n * 2 + 1);
    for (int64_t k = 0; k < n; k++) {
        Chain c{ops[k].source, 0, 0, {}};
        const auto it = now.find(ops[k].source);
        if (it != now.end()) c = it->second;
        const bool neg = ops[k].sign < 0;
        const double z = ops[k].value;
        if (c.depth > 0 && z == 0.0 && c.value[c.depth - 1] == 0.0 &&
            (std::signbit(c.value[c.depth - 1]) || !std::signbit(z))) {
            c.neg ^= (neg ? 1 : 0) << (c.depth - 1);
            c.value[c.depth - 1] = z;
        } else {
            if (c.depth == kBcMaxDepth) return false;
            c.neg |= (neg ? 1 : 0) << c.depth;
            c.value[c.depth++] = z;
        }
        now[ops[k].target] = c;
    }
    out.clear();
    out.reserve(now.size());
    for (const auto &e : now) {
        Folded f{};
        f.target = e.first;
        f.root = e.second.root;
        f.depth = e.second.depth;
        f.neg = e.second.neg;
        for (int s = 0; s < kBcMaxDepth; s++) f.value[s] = e.second.value[s];
        out.push_back(f);
    }
    // the assignments that read a written cell or write a read one first, then by target
    std::unordered_map<int64_t, char> roots;
    roots.reserve(out.size() * 2 + 1);
    for (const Folded &f : out) roots[f.root] = 1;
    for (Folded &f : out) f.wave = now.count(f.root) || roots.count(f.target) ? 0 : 1;
    std::sort(out.begin(), out.end(),
              [](const Folded &a, const Folded &b) { return a.wave != b.wave ? a.wave < b.wave : a.target < b.target; });
    return true;
}

void free_flat(BcProgram::Flat &x) {
    cudaFree(x.d_target); cudaFree(x.d_root); cudaFree(x.d_depth); cudaFree(x.d_neg); cudaFree(x.d_value);
    x = BcProgram::Flat{};
}

// JacobiDiffuse copies in = out over the domain list after every iteration
// (JacobiDiffuse.cpp:85-89).  The two arrays may take turns instead where that copy
// gives the next iteration exactly what the array just written holds: every face
// neighbour of an inner cell is on the domain list (obstacles that leave cells off
// it keep their old values in `in`), the cells on it are the inner ones and the
// program's targets, and the program reads nothing that it writes (one wave).
// Decided when lists and programs are set: at 128^3 the check took 0.8 ms of a first solve.
void update_alternates(artss_ctx *ctx, int field_type) {
    const BcProgram &p = ctx->bc[0][field_type];
    const CellBits &in = ctx->inner_bits[0], &dom = ctx->domain_bits;
    bool ok = ctx->faces_in_domain && (!p.present || p.waves <= 1);
    if (ok) {
        CellBits set = in;
        for (int64_t t : p.h_target) set.set(t);
        for (int64_t r : p.h_root) ok = ok && dom.get(r);
        ok = ok && set.w == dom.w;
    }
    ctx->alternates[field_type] = ok;
}

// the flat form of a program of several waves, on the device
int build_flat(artss_ctx *ctx, BcProgram &p, const artss_bc_assign *ops, int64_t n_ops) {
    std::vector<Folded> f;
    if (!flatten_bc(ops, n_ops, f)) return ARTSS_OK;
    const int64_t n = (int64_t) f.size();
    BcProgram::Flat x;
    std::unordered_map<int64_t, char> targets;
    targets.reserve(f.size() * 2 + 1);
    for (const Folded &a : f) {
        targets[a.target] = 1;
        if (a.wave == 0) x.hazards++;
    }
    if (x.hazards > kBcMaxHazards) return ARTSS_OK;
    std::vector<uint8_t> neg((size_t) n);
    std::vector<double> val((size_t) kBcMaxDepth * n, 0.0);
    for (int64_t q = 0; q < n; q++) {
        const Folded &a = f[(size_t) q];
        x.h_target.push_back(a.target);
        x.h_root.push_back(a.root);
        x.h_depth.push_back((uint8_t) (a.depth | (targets.count(a.root) ? kBcLagged : 0)));
        neg[(size_t) q] = a.neg;
        for (int s = 0; s < a.depth; s++) val[(size_t) (s * n + q)] = a.value[s];
    }
    auto put = [&](auto **dst, const auto &src) -> int {
        const size_t bytes = src.size() * sizeof(src[0]);
        ARTSS_CK(cudaMalloc((void **) dst, bytes));
        ARTSS_CK(cudaMemcpy(*dst, src.data(), bytes, cudaMemcpyHostToDevice));
        return ARTSS_OK;
    };
    int st = ARTSS_OK;
    st = st ? st : put(&x.d_target, x.h_target);
    st = st ? st : put(&x.d_root, x.h_root);
    st = st ? st : put(&x.d_depth, x.h_depth);
    st = st ? st : put(&x.d_neg, neg);
    st = st ? st : put(&x.d_value, val);
    if (st) { free_flat(x); return st; }
    x.n = n;
    p.flat = x;
    return ARTSS_OK;
}

}  // namespace artss

using namespace artss;

extern "C" {

int artss_set_boundary_program(artss_ctx *ctx, int level, int field_type, const artss_bc_assign *ops, int64_t n_ops) {
    int st = check_level(ctx, level);
    if (st) return st;
    if ((st = check_field_type(field_type))) return st;
    if (n_ops < 0 || (n_ops && !ops)) { set_error("bad boundary program"); return ARTSS_ERR_ARG; }
    const Level &L = ctx->lvl[level];
    for (int64_t k = 0; k < n_ops; k++) {
        if (ops[k].target < 0 || ops[k].target >= L.size() || ops[k].source < 0 || ops[k].source >= L.size() ||
            (ops[k].sign != 1 && ops[k].sign != -1)) {
            set_error("boundary assignment " + std::to_string(k) + " out of range");
            return ARTSS_ERR_ARG;
        }
    }
    std::vector<Folded> folded;
    int waves = 0;
    compile_bc(ops, n_ops, folded, waves);
    // group by wave, targets ascending within a wave
    std::stable_sort(folded.begin(), folded.end(), [](const Folded &a, const Folded &b) {
        return a.wave != b.wave ? a.wave < b.wave : a.target < b.target;
    });
    const int64_t n = (int64_t) folded.size();
    std::vector<int64_t> tgt(n), root(n);
    std::vector<int8_t> sign(n);
    std::vector<uint8_t> depth(n), neg(n);
    std::vector<double> val((size_t) kBcMaxDepth * std::max<int64_t>(n, 1), 0.0);
    std::vector<int64_t> begin(waves + 1, 0);
    for (int64_t q = 0; q < n; q++) {
        tgt[q] = folded[q].target;
        root[q] = folded[q].root;
        depth[q] = (uint8_t) folded[q].depth;
        neg[q] = folded[q].neg;
        sign[q] = (__builtin_popcount((unsigned) folded[q].neg & ((1u << folded[q].depth) - 1u)) & 1) ? -1 : 1;
        for (int s = 0; s < kBcMaxDepth; s++) val[s * n + q] = s < folded[q].depth ? folded[q].value[s] : 0.0;
        begin[folded[q].wave + 1] = q + 1;
    }
    for (int w = 1; w <= waves; w++) begin[w] = std::max(begin[w], begin[w - 1]);

    BcProgram &p = ctx->bc[level][field_type];
    ARTSS_CK(cudaStreamSynchronize(ctx->stream));
    cudaFree(p.d_target); cudaFree(p.d_root); cudaFree(p.d_depth); cudaFree(p.d_neg); cudaFree(p.d_value);
    free_flat(p.flat);
    p = BcProgram{};
    p.present = true;
    p.waves = waves;
    p.wave_begin = begin;
    p.n = n;
    p.h_target = tgt;
    p.h_root = root;
    p.h_sign = sign;
    ctx->geom_version++;
    if (level == 0) update_alternates(ctx, field_type);
    p.zero_values = true;
    for (double v : val) {
        uint64_t bits;
        std::memcpy(&bits, &v, sizeof bits);
        if (bits != 0) p.zero_values = false;
    }
    p.homogeneous = waves <= 1;
    for (int64_t q = 0; q < n && p.homogeneous; q++) {
        // the steps x -> +-x + z from the last one back: x + (-0) is x; the step before
        // them adds +0, or there is none
        int d = folded[q].depth;
        for (int s = 0; s < d; s++) p.homogeneous = p.homogeneous && folded[q].value[s] == 0.0;
        while (d > 0 && std::signbit(folded[q].value[d - 1]) && !(folded[q].neg >> (d - 1) & 1)) d--;
        if (d > 0 && std::signbit(folded[q].value[d - 1])) p.homogeneous = false;
    }
    if (n == 0) return ARTSS_OK;
    ARTSS_CK(cudaMalloc(&p.d_target, n * sizeof(int64_t)));
    ARTSS_CK(cudaMalloc(&p.d_root, n * sizeof(int64_t)));
    ARTSS_CK(cudaMalloc(&p.d_depth, n));
    ARTSS_CK(cudaMalloc(&p.d_neg, n));
    ARTSS_CK(cudaMalloc(&p.d_value, kBcMaxDepth * n * sizeof(double)));
    ARTSS_CK(cudaMemcpyAsync(p.d_target, tgt.data(), n * sizeof(int64_t), cudaMemcpyHostToDevice, ctx->stream));
    ARTSS_CK(cudaMemcpyAsync(p.d_root, root.data(), n * sizeof(int64_t), cudaMemcpyHostToDevice, ctx->stream));
    ARTSS_CK(cudaMemcpyAsync(p.d_depth, depth.data(), n, cudaMemcpyHostToDevice, ctx->stream));
    ARTSS_CK(cudaMemcpyAsync(p.d_neg, neg.data(), n, cudaMemcpyHostToDevice, ctx->stream));
    ARTSS_CK(cudaMemcpyAsync(p.d_value, val.data(), kBcMaxDepth * n * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
    // the host vectors die with this call
    ARTSS_CK(cudaStreamSynchronize(ctx->stream));
    return waves > 1 ? build_flat(ctx, p, ops, n_ops) : ARTSS_OK;
}

int artss_boundary_program_waves(artss_ctx *ctx, int level, int field_type) {
    if (check_level(ctx, level) || check_field_type(field_type)) return -1;
    const BcProgram &p = ctx->bc[level][field_type];
    return p.present ? p.waves : 0;
}

int artss_apply_boundary(artss_ctx *ctx, double *field, int level, int field_type) {
    int st = check_level(ctx, level);
    if (st) return st;
    if ((st = check_field_type(field_type))) return st;
    if (!field) { set_error("null field"); return ARTSS_ERR_ARG; }
    return apply_bc(ctx, field, level, field_type);
}

}  // extern "C"
