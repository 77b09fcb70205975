// Mixed-precision pressure solve: FP64 defect correction around FP32 V-cycles.
//
// No counterpart in the reference; it plugs in where IPressure::pressure
// (src/interfaces/IPressure.h:17) is called and is judged against VCycleMG
// (src/pressure/VCycleMG.cpp) iterated to the same relative residual.
//
// Outer loop, FP64 on level 0:
//     r = b - A p                      stop when ||r||_2 <= rel_tol * ||b||_2
//     e = V(r)                         FP32 V-cycle on A e = r, e = 0 at start
//     p += e                           FP64
// and, for pure-Neumann problems (A 1 = 0), the mean of p over the inner
// cells is removed at the end.  b must lie in the range of A: with the
// reference's obstacle boundary programs (edge and corner cells copy one of
// their fluid neighbours) A is not symmetric, so a mean-free b is not enough
// for a pure-Neumann problem; artss_laplacian builds consistent right-hand
// sides.  The V-cycle has the structure of VCycleMG::VCycleMultigrid
// (n_relax weighted-Jacobi sweeps, each followed by the level's boundary
// program, residual, restriction, prolongation with the trilinear weights of
// VCycleMG::Prolongate), all in FP32 with the boundary values set to zero
// (the correction equation is homogeneous), and the coarsest level solved in
// FP64 by the cluster kernel to a relative tolerance.  Because the outer
// residual is FP64, the FP32 round-off limits only the convergence rate per
// cycle, not the final accuracy.
//
// All outer iterations run as predicated batches: every kernel of an
// iteration returns at once when the device loop state says the solve has
// converged, and the host reads that state once per batch.
#include "internal.cuh"

#include <algorithm>
#include <cstdlib>
#include <unordered_map>

struct artss_mixed {
    artss_ctx *ctx = nullptr;
    artss_mixed_cfg cfg{};
    int L = 0;  // levels 0 .. L-1
    float *r[artss::kMaxLevel + 1]{};    // right-hand side of level l
    float *q[artss::kMaxLevel + 1]{};    // residual of level l
    float *e[artss::kMaxLevel + 1]{};    // correction of level l
    float *t[artss::kMaxLevel + 1]{};    // Jacobi ping-pong partner of e
    // the level's homogeneous pressure program applied by the writers of the
    // inner cells instead of by a launch after each sweep (levels 0 .. L-2, when
    // fold[l]): nbm[l][x] bit 0 = inner, bits 1..7 = index of the cell's push
    // pattern in push[l]; bits 2d .. 2d + 1 of a pattern = what the boundary cell one
    // step (d % 3 - 1, d / 3 % 3 - 1, d / 9 - 1) away takes from inner cell x with
    // value v: 0 nothing, 1 +v, 2 -v
    uint8_t *nbm[artss::kMaxLevel + 1]{};
    uint64_t *push[artss::kMaxLevel + 1]{};  // 128 patterns per level (pattern 0: none)
    bool fold[artss::kMaxLevel + 1]{};
    bool whole[artss::kMaxLevel + 1]{};      // the patterns hold the whole program, edges and corners too
    bool q_bc_dead[artss::kMaxLevel + 1]{};  // the restriction of level l + 1 reads no boundary cell of level l
    uint64_t geom_version = ~0ull;       // ctx->geom_version the tables describe
    int64_t n_inner0 = 0;
    int64_t hint = 1;                    // outer iterations of the last solve
};

namespace artss {

namespace {

inline dim3 mx_grid(const Box3 &b) {
    dim3 g = box_grid(b);
    const int64_t xy = (int64_t) g.x * g.y;
    int64_t gz = b.nz();
    const int64_t cap = std::max<int64_t>(1, 2048 / std::max<int64_t>(xy, 1));
    if (gz > cap) gz = cap;
    g.z = (unsigned) std::max<int64_t>(gz, 1);
    return g;
}

// 32-bit cell indices: artss_ctx_create rejects levels of 2^31 cells or more
#define MX_COLUMN(box)                                                             \
    const int i = (int) (box).x0 + (int) (blockIdx.x * blockDim.x + threadIdx.x); \
    const int j = (int) (box).y0 + (int) (blockIdx.y * blockDim.y + threadIdx.y); \
    const bool col = (i <= (int) (box).x1) && (j <= (int) (box).y1)

// nbm of a boundary cell that takes +-the value of its inner partner in the pair of
// cells 2 n, 2 n + 1 (kept out of the partner's pattern)
constexpr unsigned kPartnerPlus = 2, kPartnerMinus = 4;

struct CoefF {
    float ax, ay, az, beta, w, omw;
};

// weighted Jacobi sweep of the pressure operator (the multigrid variant of
// JacobiDiffuse::JacobiStep, dsign = -1), FP32
// store v at inner cell x and the boundary cells whose homogeneous program
// value is +-x (the cell's push pattern)
template <class T>
__device__ __forceinline__ void mx_push(T *__restrict__ out, unsigned mask, const uint64_t *__restrict__ push, int x, T v,
                                        int nj, int nk) {
    uint64_t mm = __ldg((const unsigned long long *) push + (mask >> 1));
    while (mm) {
        const int d = (__ffsll((long long) mm) - 1) >> 1;
        out[x + (d % 3 - 1) + nj * (d / 3 % 3 - 1) + nk * (d / 9 - 1)] = (mm >> (2 * d)) & 1u ? v : -v;
        mm &= ~(3ull << (2 * d));
    }
}
template <class T>
__device__ __forceinline__ void mx_store(T *__restrict__ out, uint8_t mask, const uint64_t *__restrict__ push, int x, T v,
                                         int nj, int nk) {
    out[x] = v;
    if (mask >> 1) mx_push(out, mask, push, x, v, nj, nk);
}

// CORRECT (the last sweep of level 0 in a V-cycle): instead of storing the
// sweep's value v, add it to the FP64 iterate, p[x] += (double) v, which is
// k_mx_correct's update of the same value (out unused); push_p: p's boundary cells
// with it, where p's program is homogeneous and wholly in the patterns
template <bool CORRECT>
__global__ void __launch_bounds__(256, 8) k_mx_jacobi(float *__restrict__ out, const float *__restrict__ in, const float *__restrict__ b,
                            const uint8_t *__restrict__ nbm, const uint64_t *__restrict__ push, Level L, Box3 box,
                            CoefF c, const LoopState *__restrict__ pred, double *__restrict__ p, int push_p) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (pred && !pred->cond) return;
    MX_COLUMN(box);
    if (!col) return;
    const int nj = (int) L.Nx, nk = (int) L.nxy();
    column_march<2>(in, i + nj * j, nk, (int) box.z0, (int) box.z1, nbm,
        [&](int x, int, float km, float c0, float kp) {
            const float h = c.beta * (-b[x] + c.ax * (in[x + 1] + in[x - 1]) + c.ay * (in[x + nj] + in[x - nj]) +
                                      c.az * (kp + km));
            return c.omw * c0 + c.w * h;
        },
        [&](int x, int, float v, uint8_t fl) {
            if (CORRECT) mx_store(p, push_p ? fl : (uint8_t) 0, push, x, p[x] + (double) v, nj, nk);
            else mx_store(out, fl, push, x, v, nj, nk);
        });
}

// one colour of an in-place red-black Gauss-Seidel sweep of the same operator,
// FP32: cells with (i + j + k) % 2 == color; first != 0: the sweep starts from a
// zero correction, so the red cells get w * beta * (-b) and the black cells 0
__global__ void k_mx_rbgs(float *__restrict__ e, const float *__restrict__ b, const uint8_t *__restrict__ flags,
                          Level L, Box3 box, CoefF c, int color, int first, const LoopState *__restrict__ pred) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (pred && !pred->cond) return;
    MX_COLUMN(box);
    if (!col) return;
    const int nj = (int) L.Nx, nk = (int) L.nxy();
    // the cells of one colour read only cells of the other: no cell of the
    // launch is both read and written
    column_march((const float *) e, i + nj * j, nk, (int) box.z0, (int) box.z1, flags,
        [&](int x, int, float km, float c0, float kp) {
            if (first) return c.w * (c.beta * -b[x]);
            const float h = c.beta * (-b[x] + c.ax * (e[x + 1] + e[x - 1]) + c.ay * (e[x + nj] + e[x - nj]) +
                                      c.az * (kp + km));
            return c.omw * c0 + c.w * h;
        },
        [&](int x, int k, float v, auto) {
            if (((i + j + k) & 1) == color) e[x] = v;
            else if (first) e[x] = 0.f;
        });
}

// residual q = b - A e on inner cells, FP32 (VCycleMG::Residuum)
__global__ void __launch_bounds__(256, 8) k_mx_residuum(float *__restrict__ out, const float *__restrict__ e, const float *__restrict__ b,
                              const uint8_t *__restrict__ nbm, Level L, Box3 box, float rx, float ry, float rz,
                              const LoopState *__restrict__ pred) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (pred && !pred->cond) return;
    MX_COLUMN(box);
    if (!col) return;
    const int nj = (int) L.Nx, nk = (int) L.nxy();
    column_march<2>(e, i + nj * j, nk, (int) box.z0, (int) box.z1, nbm,
        [&](int x, int, float km, float c0, float kp) {
            const float c2 = 2.f * c0;
            return b[x] - (rx * (e[x - 1] - c2 + e[x + 1]) + ry * (e[x - nj] - c2 + e[x + nj]) +
                           rz * (km - c2 + kp));
        },
        [&](int x, int, float v, auto) { out[x] = v; });
}

// coarse inner cell = mean of its 8 children (VCycleMG::Restrict), FP32
__global__ void k_mx_restrict(float *__restrict__ out, const float *__restrict__ in,
                              const uint8_t *__restrict__ flags, Level C, Level F, Box3 box,
                              const LoopState *__restrict__ pred) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (pred && !pred->cond) return;
    MX_COLUMN(box);
    if (!col) return;
    const int fx = (int) F.Nx, fxy = (int) F.nxy();
    column_planes(i + (int) C.Nx * j, (int) C.nxy(), (int) box.z0, (int) box.z1, flags,
        [&](int, int k) {
            const int f = (2 * i - 1) + fx * (2 * j - 1) + fxy * (2 * k - 1);
            return 0.125f * (in[f] + in[f + 1] + in[f + fx] + in[f + fx + 1] + in[f + fxy] + in[f + fxy + 1] +
                             in[f + fxy + fx] + in[f + fxy + fx + 1]);
        },
        [&](int x, int, float v, auto) { out[x] = v; });
}

// Residual and restriction in one pass: a coarse inner cell takes the mean of its
// eight children's residuals, each with k_mx_residuum's expression, a child that is
// not inner counting 0 as in the residual array (q_bc_dead).  Written and read back,
// with its boundary program between, the residual cost 20 of 28 bytes a fine cell
// and two more launches.
__global__ void __launch_bounds__(256) k_mx_residuum_restrict(float *__restrict__ out, const float *__restrict__ e,
                                                              const float *__restrict__ b,
                                                              const uint8_t *__restrict__ cflags,
                                                              const uint8_t *__restrict__ nbm, Level C, Level F, Box3 box,
                                                              float rx, float ry, float rz,
                                                              const LoopState *__restrict__ pred) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (pred && !pred->cond) return;
    MX_COLUMN(box);
    if (!col) return;
    const int fx = (int) F.Nx, fxy = (int) F.nxy();
    const int f0 = 2 * i - 1 + fx * (2 * j - 1);
    for (int k = (int) box.z0 + (int) blockIdx.z; k <= (int) box.z1; k += (int) gridDim.z) {
        const int q = i + (int) C.Nx * j + (int) C.nxy() * k;
        if (!(cflags[q] & kInner)) continue;
        float r[8];
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const int x = f0 + (c & 1) + fx * ((c >> 1) & 1) + fxy * (2 * k - 1 + (c >> 2));
            const float c2 = 2.f * e[x];
            const float v = b[x] - (rx * (e[x - 1] - c2 + e[x + 1]) + ry * (e[x - fx] - c2 + e[x + fx]) +
                                    rz * (e[x - fxy] - c2 + e[x + fxy]));
            r[c] = (nbm[x] & kInner) ? v : 0.f;
        }
        out[q] = 0.125f * (r[0] + r[1] + r[2] + r[3] + r[4] + r[5] + r[6] + r[7]);
    }
}

// first Jacobi sweep from a zero correction: every neighbour is zero, so
// e = w * beta * (-b) on the inner cells
__global__ void k_mx_jacobi0(float *__restrict__ out, const float *__restrict__ b, const uint8_t *__restrict__ flags,
                             const uint64_t *__restrict__ push, Level L, Box3 box, CoefF c,
                             const LoopState *__restrict__ pred) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (pred && !pred->cond) return;
    MX_COLUMN(box);
    if (!col) return;
    const int nj = (int) L.Nx, nk = (int) L.nxy();
    column_planes(i + nj * j, nk, (int) box.z0, (int) box.z1, flags,
        [&](int x, int) { return c.w * (c.beta * -b[x]); },
        [&](int x, int, float v, uint8_t fl) { mx_store(out, fl, push, x, v, nj, nk); });
}

// fine correction += trilinear prolongation of the coarse correction
// (weights 27/9/3/1 over 64 of VCycleMG::Prolongate), on the fine inner
// children of each coarse inner cell, FP32
__global__ void k_mx_prolong_add(float *__restrict__ fine, const float *__restrict__ in,
                                 const uint8_t *__restrict__ cflags, const uint8_t *__restrict__ fflags,
                                 const uint64_t *__restrict__ push, Level C, Level F, Box3 fbox,
                                 const LoopState *__restrict__ pred) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (pred && !pred->cond) return;
    MX_COLUMN(fbox);  // one thread per fine column: fine cell 2c (side +1) or 2c - 1 (side -1) of coarse cell c
    if (!col) return;
    const int nj = (int) C.Nx, nk = (int) C.nxy();
    const int fx = (int) F.Nx, fxy = (int) F.nxy();
    const int ci = (i + 1) >> 1, cj = (j + 1) >> 1;
    const int sx = (i & 1) ? -1 : 1, sy = (j & 1) ? -1 : 1;
    struct Out { float v; uint8_t cf; };
    column_planes(i + fx * j, fxy, (int) fbox.z0, (int) fbox.z1, fflags,
        [&](int f, int k) {
            const int sz = (k & 1) ? -1 : 1;
            const int x = ci + nj * cj + nk * ((k + 1) >> 1);
            const float v = 0.015625f * (27.f * in[x] + 9.f * in[x + sx] + 9.f * in[x + sy * nj] + 9.f * in[x + sz * nk] +
                                         3.f * in[x + sx + sy * nj] + 3.f * in[x + sx + sz * nk] +
                                         3.f * in[x + sy * nj + sz * nk] + in[x + sx + sy * nj + sz * nk]);
            return Out{fine[f] + v, cflags[x]};
        },
        [&](int f, int, Out o, uint8_t fl) {
            if (o.cf & kInner) mx_store(fine, fl, push, f, o.v, fx, fxy);
        });
}

// The same prolongation, one thread per coarse column: the thread marches up
// its contiguous run of coarse planes keeping the 3 x 3 x 3 coarse
// neighbourhood in registers (one new 3 x 3 plane per step) and updates the 8
// fine children of each coarse inner cell, each with k_mx_prolong_add's
// expression, so every fine value is the same bit for bit.  The fine x pairs
// of a warp's 32 coarse columns are 64 consecutive cells.
__global__ void __launch_bounds__(256) k_mx_prolong_add8(float *__restrict__ fine, const float *__restrict__ in,
                                                         const uint8_t *__restrict__ cflags,
                                                         const uint8_t *__restrict__ fflags,
                                                         const uint64_t *__restrict__ push, Level C, Level F,
                                                         Box3 cbox, Box3 fbox, const LoopState *__restrict__ pred) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (pred && !pred->cond) return;
    MX_COLUMN(cbox);  // (i, j): the coarse column
    if (!col) return;
    const int nj = (int) C.Nx, nk = (int) C.nxy();
    const int fx = (int) F.Nx, fxy = (int) F.nxy();
    const int nzc = (int) cbox.nz();
    const int chunk = (nzc + (int) gridDim.z - 1) / (int) gridDim.z;
    const int k0 = (int) cbox.z0 + (int) blockIdx.z * chunk;
    const int k1 = min((int) cbox.z1, k0 + chunk - 1);
    if (k0 > k1) return;
    // w[p][b][a]: coarse value at (i + a - 1, j + b - 1, k + p - 1) for the current plane k
    float w[3][3][3];
    auto load_plane = [&](int k, float (&pl)[3][3]) {
        const int x = i + nj * j + nk * k;
#pragma unroll
        for (int b = 0; b < 3; b++)
#pragma unroll
            for (int a = 0; a < 3; a++) pl[b][a] = in[x + (a - 1) + nj * (b - 1)];
    };
    load_plane(k0 - 1, w[0]);
    load_plane(k0, w[1]);
    // fine children of this column that lie in the fine box
    const int fi0 = 2 * i - 1, fj0 = 2 * j - 1;
    const bool xa = fi0 >= (int) fbox.x0 && fi0 <= (int) fbox.x1, xb = fi0 + 1 >= (int) fbox.x0 && fi0 + 1 <= (int) fbox.x1;
    const bool ya = fj0 >= (int) fbox.y0 && fj0 <= (int) fbox.y1, yb = fj0 + 1 >= (int) fbox.y0 && fj0 + 1 <= (int) fbox.y1;
    for (int k = k0; k <= k1; k++) {
        // every load of the step first (the children lie in the fine array: 2 c <=
        // the fine inner box's end + 1), then the arithmetic and the stores
        const bool cin = (cflags[i + nj * j + nk * k] & kInner) != 0;
        uint8_t fl[8];
        float fv[8];
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const int f = fi0 + (c & 1) + fx * (fj0 + ((c >> 1) & 1)) + fxy * (2 * k - 1 + (c >> 2));
            fl[c] = fflags[f];
            fv[c] = fine[f];
        }
        load_plane(k + 1, w[2]);
        if (cin) {
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const int dx = c & 1, dy = (c >> 1) & 1, dz = c >> 2;
                const int fk = 2 * k - 1 + dz;
                if (fk < (int) fbox.z0 || fk > (int) fbox.z1 || !(dy ? yb : ya) || !(dx ? xb : xa) || !(fl[c] & kInner))
                    continue;
                const int px = dx ? 2 : 0, py = dy ? 2 : 0, pz = dz ? 2 : 0;  // s = +1 for the even child
                const int f = fi0 + dx + fx * (fj0 + dy) + fxy * fk;
                const float v = 0.015625f * (27.f * w[1][1][1] + 9.f * w[1][1][px] + 9.f * w[1][py][1] +
                                             9.f * w[pz][1][1] + 3.f * w[1][py][px] + 3.f * w[pz][1][px] +
                                             3.f * w[pz][py][1] + w[pz][py][px]);
                mx_store(fine, fl[c], push, f, fv[c] + v, fx, fxy);
            }
        }
#pragma unroll
        for (int b = 0; b < 3; b++)
#pragma unroll
            for (int a = 0; a < 3; a++) {
                w[0][b][a] = w[1][b][a];
                w[1][b][a] = w[2][b][a];
            }
    }
}

// Two neighbouring cells of x per thread, for rows of an even number of cells.  A plane
// is walked as one array, so a warp's 64 cells run on over the ends of rows, whose
// boundary cells are the 2 of Nx that are worked for nothing; the x neighbours come
// from the lanes beside, the warp's outer two from memory.
struct PairPos {
    int x0, lane;  // first cell within the plane, lane
    bool live;
};
__device__ __forceinline__ PairPos pair_pos(const Box3 &box, int nj) {
    const int p0 = (int) box.y0 * nj / 2, p1 = ((int) box.y1 + 1) * nj / 2;
    const int q = p0 + (int) (blockIdx.x * blockDim.x + threadIdx.x);
    return {2 * min(q, p1 - 1), (int) threadIdx.x & 31, q < p1};
}
__device__ __forceinline__ float2 ld2(const float *p) { return *(const float2 *) p; }
__device__ __forceinline__ double2 ld2(const double *p) { return *(const double2 *) p; }
// the values left of a pair's first and right of its second cell; edge: the lane's
// value from memory, for lanes 0 and 31
template <class T, class T2>
__device__ __forceinline__ void pair_sides(const T2 &c, T edge, int lane, T *l, T *r) {
    *l = __shfl_up_sync(~0u, c.y, 1);
    *r = __shfl_down_sync(~0u, c.x, 1);
    if (lane == 0) *l = edge;
    if (lane == 31) *r = edge;
}
// store a pair's inner cells, a boundary cell whose root is its partner in the pair
// (kPartnerPlus, kPartnerMinus) with it, and what the push patterns name.  Half the
// warps of a row hold one of its ends: by a pattern, those cost more instructions
// than the sweep.
template <class T, class T2>
__device__ __forceinline__ void pair_store(T *__restrict__ out, unsigned fl, const uint64_t *__restrict__ push, int x, T2 v,
                                           int nj, int nk) {
    if (fl == 0x0101u) {
        *(T2 *) (out + x) = v;
        return;
    }
    const unsigned f0 = fl & 0xffu, f1 = fl >> 8;
    const bool in0 = f0 & 1u, in1 = f1 & 1u;
    if (!in0) v.x = f0 == kPartnerMinus ? -v.y : v.y;
    if (!in1) v.y = f1 == kPartnerMinus ? -v.x : v.x;
    if (f0 && f1) *(T2 *) (out + x) = v;
    else if (f0) out[x] = v.x;
    else if (f1) out[x + 1] = v.y;
    if (in0 && f0 > 1u) mx_push(out, f0, push, x, v.x, nj, nk);
    if (in1 && f1 > 1u) mx_push(out, f1, push, x + 1, v.y, nj, nk);
}
// a pair's flags as those of its inner cells alone: nothing but them is stored
__device__ __forceinline__ unsigned pair_inner(unsigned fl) { return fl & 0x0101u; }

// A sweep's thread holds kPairPlanes planes with all their loads in flight.  256^3, one
// sweep / the two of kPairFromZero / the correcting one: 47 / 47 / 65 us here, 60 /
// 44 + 60 / 95 us by k_mx_jacobi0 and k_mx_jacobi (floors by their bytes: 33 / 23 /
// 63 us).  4 planes, 256 and 512 threads, a walk up the planes with the next one's
// loads in flight (53 / 55 / 85 us: a last wave half empty) and 4 cells per thread
// (61 us) were slower.  What bounds it now is the issue rate (87 % of the slots).
constexpr int kPairThreads = 128, kPairPlanes = 2;

enum PairMode : int { kPairSweep, kPairCorrect, kPairFromZero };

// k_mx_jacobi on pairs of cells.  kPairFromZero: the first two sweeps from a zero
// correction in one: the first one's result is e0 = w beta (-b) in inner cells and
// the same of their roots' b in the boundary cells, which b carries (its writers
// push it), so the second forms its neighbours from b alone (`in` = b).
template <int MODE>
__global__ void __launch_bounds__(kPairThreads) k_mx_jacobi2(float *__restrict__ out, const float *__restrict__ in,
                                                    const float *__restrict__ b, const uint8_t *__restrict__ nbm,
                                                    const uint64_t *__restrict__ push, Level L, Box3 box, CoefF c,
                                                    const LoopState *__restrict__ pred, double *__restrict__ p, int push_p) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (pred && !pred->cond) return;
    const int nj = (int) L.Nx, nk = (int) L.nxy(), z1 = (int) box.z1;
    const PairPos t = pair_pos(box, nj);
    constexpr int U = kPairPlanes;
    const int k0 = (int) box.z0 + (int) blockIdx.y * U;
    float2 cc[U + 2], ym[U], yp[U], bb[U];
    float edge[U];
    unsigned fl[U];
    double2 pp[U];
    const bool p2 = (uintptr_t) p % 16 == 0;
#pragma unroll
    for (int u = 0; u < U + 2; u++) cc[u] = ld2(in + t.x0 + nk * min(k0 - 1 + u, z1 + 1));
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int x = t.x0 + nk * min(k0 + u, z1);
        fl[u] = *(const uint16_t *) (nbm + x);
        ym[u] = ld2(in + x - nj);
        yp[u] = ld2(in + x + nj);
        if (MODE != kPairFromZero) bb[u] = ld2(b + x);
        edge[u] = 0.f;
        if (t.lane == 0 || t.lane == 31) edge[u] = in[x + (t.lane ? 2 : -1)];
        if (MODE == kPairCorrect) pp[u] = p2 ? ld2(p + x) : make_double2(p[x], p[x + 1]);
    }
    asm volatile("" ::: "memory");  // every load issued before the arithmetic
    const auto val = [&](float v) { return MODE == kPairFromZero ? c.w * (c.beta * -v) : v; };
    if (MODE == kPairFromZero) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            bb[u] = cc[u + 1];
            edge[u] = val(edge[u]);
            ym[u] = make_float2(val(ym[u].x), val(ym[u].y));
            yp[u] = make_float2(val(yp[u].x), val(yp[u].y));
        }
#pragma unroll
        for (int u = 0; u < U + 2; u++) cc[u] = make_float2(val(cc[u].x), val(cc[u].y));
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        float l, r;
        pair_sides(cc[u + 1], edge[u], t.lane, &l, &r);
        const float c0 = cc[u + 1].x, c1 = cc[u + 1].y;
        const float h0 = c.beta * (-bb[u].x + c.ax * (c1 + l) + c.ay * (yp[u].x + ym[u].x) + c.az * (cc[u + 2].x + cc[u].x));
        const float h1 = c.beta * (-bb[u].y + c.ax * (r + c0) + c.ay * (yp[u].y + ym[u].y) + c.az * (cc[u + 2].y + cc[u].y));
        const float v0 = c.omw * c0 + c.w * h0, v1 = c.omw * c1 + c.w * h1;
        if (!t.live || k0 + u > z1) continue;
        const int x = t.x0 + nk * (k0 + u);
        if (MODE == kPairCorrect) {
            if (p2) pair_store(p, push_p ? fl[u] : pair_inner(fl[u]), push, x, make_double2(pp[u].x + (double) v0, pp[u].y + (double) v1),
                            nj, nk);
            else {
                if (fl[u] & 1u) p[x] = pp[u].x + (double) v0;
                if (fl[u] & 0x100u) p[x + 1] = pp[u].y + (double) v1;
            }
        } else pair_store(out, fl[u], push, x, make_float2(v0, v1), nj, nk);
    }
}

// k_mx_residuum_restrict, a warp on 31 coarse cells of a row: lane n forms the residuals
// of fine cells 2 m and 2 m + 1 (m = its coarse cell) in the 4 rows of children and
// takes those of 2 m - 1 from the lane before.  A thread walks up its run of coarse
// planes with the next one's loads in flight.  256^3 to 128^3: 40 us (floor 24), 43
// by k_mx_residuum_restrict, 52 with a thread per coarse cell; at 128^3 and below
// 13 / 7 / 6 us.  push: the coarse cells' patterns,
// where the coarse level's first sweeps read r in its boundary cells.
__global__ void __launch_bounds__(256) k_mx_down2(float *__restrict__ out, const float *__restrict__ e,
                                                  const float *__restrict__ b, const uint8_t *__restrict__ cflags,
                                                  const uint8_t *__restrict__ nbm, const uint8_t *__restrict__ cnbm,
                                                  const uint64_t *__restrict__ cpush, Level C, Level F, Box3 box, int planes, float rx,
                                                  float ry, float rz, const LoopState *__restrict__ pred) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (pred && !pred->cond) return;
    const int lane = (int) threadIdx.x;
    const int m = (int) box.x0 - 1 + 31 * (int) blockIdx.x + lane, j = (int) box.y0 + (int) (blockIdx.y * 8 + threadIdx.y);
    if (j > (int) box.y1) return;
    const int ka = (int) box.z0 + (int) blockIdx.z * planes, ke = min(ka + planes - 1, (int) box.z1);
    const int fx = (int) F.Nx, fxy = (int) F.nxy(), mc = min(m, (int) box.x1);
    // rows 2 j - 2 .. 2 j + 1 of planes 2 k - 2 .. 2 k + 1, without the corners; a step up
    // keeps the inner rows of the upper two planes
    int x0 = 2 * mc + fx * (2 * j - 1) + fxy * (2 * ka - 1);
    float2 v[4][4];
#pragma unroll
    for (int z = 0; z < 2; z++)
#pragma unroll
        for (int y = 1; y < 3; y++) v[z][y] = ld2(e + x0 + fx * (y - 1) + fxy * (z - 1));
    struct In {
        float2 lo0, lo3, up[4], top1, top2, b[4];
        unsigned fl[4], cf, cm, side;
    };
    const auto load = [&](int x, int k) {
        In n;
        n.lo0 = ld2(e + x - fx);
        n.lo3 = ld2(e + x + 2 * fx);
#pragma unroll
        for (int y = 0; y < 4; y++) n.up[y] = ld2(e + x + fx * (y - 1) + fxy);
        n.top1 = ld2(e + x + 2 * fxy);
        n.top2 = ld2(e + x + fx + 2 * fxy);
#pragma unroll
        for (int c = 0; c < 4; c++) {
            n.b[c] = ld2(b + x + fx * (c & 1) + fxy * (c >> 1));
            n.fl[c] = *(const uint16_t *) (nbm + x + fx * (c & 1) + fxy * (c >> 1));
        }
        const int q = mc + (int) C.Nx * j + (int) C.nxy() * k;
        n.cf = cflags[q];
        n.cm = cnbm ? cnbm[q] : 0u;
        n.side = cnbm ? cnbm[q ^ 1] : 0u;
        return n;
    };
    In cur = load(x0, ka);
    for (int k = ka; k <= ke; k++, x0 += 2 * fxy) {
        v[1][0] = cur.lo0;
        v[1][3] = cur.lo3;
#pragma unroll
        for (int y = 0; y < 4; y++) v[2][y] = cur.up[y];
        v[3][1] = cur.top1;
        v[3][2] = cur.top2;
        In nxt = cur;
        if (k < ke) nxt = load(x0 + 2 * fxy, k + 1);
        float sum = 0.f;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int y = 1 + (c & 1), z = 1 + (c >> 1);
            const float2 o = v[z][y];
            float l, r;
            pair_sides(o, 0.f, lane, &l, &r);  // lane 0's first and lane 31's second residual go unused
            const float ax = 2.f * o.x, ay = 2.f * o.y;
            float r0 = cur.b[c].x - (rx * (l - ax + o.y) + ry * (v[z][y - 1].x - ax + v[z][y + 1].x) +
                                     rz * (v[z - 1][y].x - ax + v[z + 1][y].x));
            float r1 = cur.b[c].y - (rx * (o.x - ay + r) + ry * (v[z][y - 1].y - ay + v[z][y + 1].y) +
                                     rz * (v[z - 1][y].y - ay + v[z + 1][y].y));
            if (!(cur.fl[c] & 1u)) r0 = 0.f;
            if (!(cur.fl[c] & 0x100u)) r1 = 0.f;
            const float left = __shfl_up_sync(~0u, r1, 1);
            sum = c ? sum + left : left;
            sum += r0;
        }
        if (lane && m <= (int) box.x1 && (cur.cf & kInner)) {
            const int q = m + (int) C.Nx * j + (int) C.nxy() * k;
            const float mean = 0.125f * sum;
            mx_store(out, (uint8_t) cur.cm, cpush, q, mean, (int) C.Nx, (int) C.nxy());
            if (cur.side == kPartnerPlus || cur.side == kPartnerMinus) out[q ^ 1] = cur.side == kPartnerPlus ? mean : -mean;
        }
#pragma unroll
        for (int y = 1; y < 3; y++) {
            v[0][y] = v[2][y];
            v[1][y] = v[3][y];
        }
        cur = nxt;
    }
}

// k_mx_prolong_add8's values, a warp on 31 fine pairs (2 m, 2 m + 1) of 2 rows and 2
// planes: both cells' 8 coarse values lie in the columns m and m + 1, the lane's
// own and the next lane's, and a pair is stored in one piece.  128^3 to 256^3: 49 us
// (floor 24; instructions bound it), walking up the planes 52 to 58.
__global__ void __launch_bounds__(256) k_mx_prolong_add2(float *__restrict__ fine, const float *__restrict__ in,
                                                         const uint8_t *__restrict__ cflags,
                                                         const uint8_t *__restrict__ nbm,
                                                         const uint64_t *__restrict__ push, Level C, Level F,
                                                         Box3 cbox, Box3 fbox, const LoopState *__restrict__ pred) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (pred && !pred->cond) return;
    const int lane = (int) threadIdx.x;
    const int cm = (int) cbox.x0 - 1 + 31 * (int) blockIdx.x + lane, j = (int) cbox.y0 + (int) (blockIdx.y * 8 + threadIdx.y),
              k = (int) cbox.z0 + (int) blockIdx.z;
    if (j > (int) cbox.y1) return;
    const int m = min(cm, (int) cbox.x1 + 1);  // columns x0 - 1 .. x1 + 1, the last a right neighbour only
    const int nj = (int) C.Nx, nk = (int) C.nxy(), fx = (int) F.Nx, fxy = (int) F.nxy();
    const int x = m + nj * j + nk * k;
    const int mf = min(m, (int) cbox.x1);
    float w[3][3][2];
    float2 fv[4];
    unsigned fl[4];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) w[a][b][0] = in[x + nj * (b - 1) + nk * (a - 1)];
    const unsigned own = cflags[x] & kInner;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const int f = 2 * mf + fx * (2 * j - 1 + (c & 1)) + fxy * (2 * k - 1 + (c >> 1));
        fl[c] = *(const uint16_t *) (nbm + f);
        fv[c] = ld2(fine + f);
    }
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) w[a][b][1] = __shfl_down_sync(~0u, w[a][b][0], 1);
    const unsigned next = __shfl_down_sync(~0u, own, 1);
    if (lane == 31 || cm > (int) cbox.x1) return;
    const int i0 = 2 * m, i1 = 2 * m + 1;
    const bool in0 = own && m >= (int) cbox.x0 && i0 >= (int) fbox.x0 && i0 <= (int) fbox.x1;
    const bool in1 = next && m + 1 <= (int) cbox.x1 && i1 >= (int) fbox.x0 && i1 <= (int) fbox.x1;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const int fj = 2 * j - 1 + (c & 1), fk = 2 * k - 1 + (c >> 1);
        if (fj < (int) fbox.y0 || fj > (int) fbox.y1 || fk < (int) fbox.z0 || fk > (int) fbox.z1) continue;
        const int py = c & 1 ? 2 : 0, pz = c >> 1 ? 2 : 0;
        float2 v;
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const int o = 1 - s;
            const float g = 0.015625f * (27.f * w[1][1][s] + 9.f * w[1][1][o] + 9.f * w[1][py][s] + 9.f * w[pz][1][s] +
                                         3.f * w[1][py][o] + 3.f * w[pz][1][o] + 3.f * w[pz][py][s] + w[pz][py][o]);
            (s ? v.y : v.x) = (s ? fv[c].y : fv[c].x) + g;
        }
        unsigned f2 = fl[c];
        // an inner cell outside the children stays as it is, with its boundary cells
        if ((f2 & 1u) && !in0) f2 = f2 >> 8 & 1u ? f2 & 0xff00u : 0u;
        if ((f2 & 0x100u) && !in1) f2 = f2 & 1u ? f2 & 0x00ffu : 0u;
        pair_store(fine, f2, push, 2 * m + fx * fj + fxy * fk, v, fx, fxy);
    }
}

// the loop step of a kernel that reduces: thread 0 of each block has stored the block's
// partial sum; the last block to get here adds them in a fixed order
__device__ __forceinline__ void last_block_loop_step(const double *partials, LoopState *st, const LoopState *ref, double tol,
                                                     long long max_it, double *smem) {
    __shared__ bool last;
    const int blocks = (int) (gridDim.x * gridDim.y * gridDim.z), tid = (int) (threadIdx.x + blockDim.x * threadIdx.y);
    if (tid == 0) {
        __threadfence();
        last = atomicAdd(&st->blocks_done, 1) == blocks - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double v = 0.0;
    for (int n = tid; n < blocks; n += (int) (blockDim.x * blockDim.y)) v += __ldcg(partials + n);
    v = artss_block_sum(v, smem);
    if (tid == 0) {
        if (ref) tol = tol * sqrt(ref->sum);
        const double r = sqrt(v);
        st->blocks_done = 0;
        st->sum = v;
        st->residual = r;
        st->it += 1;
        st->cond = (r > tol && st->it < max_it) ? 1 : 0;
    }
}

// k_mx_outer_residual on pairs of cells, r's boundary cells with it (push); a thread walks
// up its run of planes with the next one's loads in flight.  256^3: 79 us (floor 50),
// 101 with two planes' loads at a time, 90 by k_mx_outer_residual and its finishing
// launch.
__global__ void __launch_bounds__(256) k_mx_outer_residual2(const double *__restrict__ p, const double *__restrict__ b,
                                                            float *__restrict__ r, const uint8_t *__restrict__ nbm,
                                                            const uint64_t *__restrict__ push, Level L, Box3 box, int planes,
                                                            double rx, double ry, double rz, double *__restrict__ partials,
                                                            LoopState *st, const LoopState *ref, double tol,
                                                            long long max_it) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    __shared__ double smem[32];
    if (!st->cond) return;  // nobody writes it before every block has passed here
    const int nj = (int) L.Nx, nk = (int) L.nxy();
    const PairPos t = pair_pos(box, nj);
    const int ka = (int) box.z0 + (int) blockIdx.y * planes, ke = min(ka + planes - 1, (int) box.z1);
    const bool p2 = ((uintptr_t) p | (uintptr_t) b) % 16 == 0;
    const auto ldp = [&](const double *q) { return p2 ? ld2(q) : make_double2(q[0], q[1]); };
    struct In {
        double2 ym, yp, b, kp;
        double edge;
        unsigned fl;
    };
    const auto load = [&](int x) {
        In v;
        v.kp = ldp(p + x + nk);
        v.ym = ldp(p + x - nj);
        v.yp = ldp(p + x + nj);
        v.b = ldp(b + x);
        v.edge = 0.0;
        if (t.lane == 0 || t.lane == 31) v.edge = p[x + (t.lane ? 2 : -1)];
        v.fl = *(const uint16_t *) (nbm + x);
        return v;
    };
    double acc = 0.0;
    int x = t.x0 + nk * ka;
    double2 km = ldp(p + x - nk), c0 = ldp(p + x);
    In cur = load(x);
#pragma unroll 2
    for (int k = ka; k <= ke; k++, x += nk) {
        In nxt = cur;
        if (k < ke) nxt = load(x + nk);
        double l, rr;
        pair_sides(c0, cur.edge, t.lane, &l, &rr);
        const double ax = 2 * c0.x, ay = 2 * c0.y;
        const double v0 = cur.b.x - (rx * (l - ax + c0.y) + ry * (cur.ym.x - ax + cur.yp.x) + rz * (km.x - ax + cur.kp.x));
        const double v1 = cur.b.y - (rx * (c0.x - ay + rr) + ry * (cur.ym.y - ay + cur.yp.y) + rz * (km.y - ay + cur.kp.y));
        if (t.live) {
            pair_store(r, cur.fl, push, x, make_float2((float) v0, (float) v1), nj, nk);
            if (cur.fl & 1u) acc += v0 * v0;
            if (cur.fl & 0x100u) acc += v1 * v1;
        }
        km = c0;
        c0 = cur.kp;
        cur = nxt;
    }
    acc = artss_block_sum(acc, smem);
    if (threadIdx.x == 0) partials[blockIdx.x + gridDim.x * blockIdx.y] = acc;
    __syncthreads();  // smem is rewritten
    last_block_loop_step(partials, st, ref, tol, max_it, smem);
}

// FP64 outer residual r = b - A p on level 0, stored as the FP32 right-hand
// side of the correction equation; the last block to finish adds the blocks' partial
// sums of ||r||^2 in a fixed order and does the loop step (state `st`, tolerance tol,
// times sqrt(ref->sum) with ref)
__global__ void __launch_bounds__(256, 8) k_mx_outer_residual(const double *__restrict__ p, const double *__restrict__ b,
                                    float *__restrict__ r, const uint8_t *__restrict__ flags, Level L, Box3 box,
                                    double rx, double ry, double rz, double *__restrict__ partials, LoopState *st,
                                    const LoopState *ref, double tol, long long max_it) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    __shared__ double smem[32];
    if (!st->cond) return;  // nobody writes it before every block has passed here
    MX_COLUMN(box);
    const int nj = (int) L.Nx, nk = (int) L.nxy();
    double acc = 0.0;
    if (col) {
        column_march<2>(p, i + nj * j, nk, (int) box.z0, (int) box.z1, flags,
            [&](int x, int, double km, double c0, double kp) {
                const double c2 = 2 * c0;
                return b[x] - (rx * (p[x - 1] - c2 + p[x + 1]) + ry * (p[x - nj] - c2 + p[x + nj]) +
                               rz * (km - c2 + kp));
            },
            [&](int x, int, double v, auto) {
                r[x] = (float) v;
                acc += v * v;
            });
    }
    acc = artss_block_sum(acc, smem);
    if (threadIdx.x == 0 && threadIdx.y == 0)
        partials[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = acc;
    __syncthreads();  // smem is rewritten
    last_block_loop_step(partials, st, ref, tol, max_it, smem);
}

// p += e on the inner cells (FP64 += FP32)
__global__ void k_mx_correct(double *__restrict__ p, const float *__restrict__ e, const uint8_t *__restrict__ flags,
                             Level L, Box3 box, const LoopState *__restrict__ pred) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (pred && !pred->cond) return;
    MX_COLUMN(box);
    if (!col) return;
    const int nj = (int) L.Nx, nk = (int) L.nxy();
    column_planes(i + nj * j, nk, (int) box.z0, (int) box.z1, flags,
        [&](int x, int) { return p[x] + (double) e[x]; },
        [&](int x, int, double v, auto) { p[x] = v; });
}

// block partials of sum(x - shift) and sum((x - shift)^2) over the inner cells
__global__ void k_mx_moments(const double *__restrict__ x, double shift, const uint8_t *__restrict__ flags, Level L,
                             Box3 box, double *__restrict__ p1, double *__restrict__ p2) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    __shared__ double smem[32];
    MX_COLUMN(box);
    const int64_t nj = L.Nx, nk = L.nxy();
    double s1 = 0.0, s2 = 0.0;
    if (col) {
        for (int64_t k = box.z0 + blockIdx.z; k <= box.z1; k += gridDim.z) {
            const int64_t q = i + nj * j + nk * k;
            if (!(flags[q] & kInner)) continue;
            const double v = x[q] - shift;
            s1 += v;
            s2 += v * v;
        }
    }
    const int bl = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    s1 = artss_block_sum(s1, smem);
    if (threadIdx.x == 0 && threadIdx.y == 0) p1[bl] = s1;
    __syncthreads();
    s2 = artss_block_sum(s2, smem);
    if (threadIdx.x == 0 && threadIdx.y == 0) p2[bl] = s2;
}

// out = A p on the inner cells (FP64)
__global__ void k_mx_laplacian(double *__restrict__ out, const double *__restrict__ p,
                               const uint8_t *__restrict__ flags, Level L, Box3 box, double rx, double ry, double rz) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    MX_COLUMN(box);
    if (!col) return;
    const int64_t nj = L.Nx, nk = L.nxy();
    for (int64_t k = box.z0 + blockIdx.z; k <= box.z1; k += gridDim.z) {
        const int64_t x = i + nj * j + nk * k;
        if (!(flags[x] & kInner)) continue;
        const double c2 = 2 * p[x];
        out[x] = rx * (p[x - 1] - c2 + p[x + 1]) + ry * (p[x - nj] - c2 + p[x + nj]) + rz * (p[x - nk] - c2 + p[x + nk]);
    }
}

}  // namespace

namespace {

constexpr int kSlotOuter = 6;  // device loop state of the outer iteration
constexpr int kSlotSum = 7;    // plain sums

CoefF coef_f(const artss_ctx *ctx, int level, double w) {
    const artss_grid_desc &g = ctx->grid;
    const double ax = 1. / (g.dx[level] * g.dx[level]), ay = 1. / (g.dy[level] * g.dy[level]),
                 az = 1. / (g.dz[level] * g.dz[level]);
    return CoefF{(float) ax, (float) ay, (float) az, (float) (1. / (2. * (ax + ay + az))), (float) w, (float) (1. - w)};
}

int mx_bc(artss_mixed *m, float *f, int level, const LoopState *pred) {
    return apply_bc_f32(m->ctx, f, level, ARTSS_FIELD_P, pred);
}

// the boundary program after a smoothing sweep, unless the level's stencils
// read their boundary neighbours through the program (m->fold[l])
int mx_bc_sweep(artss_mixed *m, float *f, int level, const LoopState *pred) {
    return m->fold[level] ? ARTSS_OK : mx_bc(m, f, level, pred);
}

// n_relax red-black Gauss-Seidel sweeps (ARTSS_MIXED_RBGS), in place on
// m->e[l], each colour followed by the level's boundary program
int mx_smooth_rbgs(artss_mixed *m, int l, bool from_zero, const LoopState *pred) {
    artss_ctx *ctx = m->ctx;
    const Level &L = ctx->lvl[l];
    const Box3 box = inner_box(L);
    const CoefF c = coef_f(ctx, l, m->cfg.w);
    int st;
    for (int s = 0; s < m->cfg.n_relax; s++) {
        for (int color = 0; color < 2; color++) {
            const int first = (from_zero && s == 0 && color == 0) ? 1 : 0;
            ARTSS_LAUNCH_PDL(ctx, FAM_MG_JACOBI, k_mx_rbgs, mx_grid(box), box_block(), 0, m->e[l],
                             (const float *) m->r[l], ctx->d_flags[l], L, box, c, color, first, pred);
            ARTSS_LAUNCH_CK(ctx);
            if ((st = mx_bc(m, m->e[l], l, pred))) return st;
        }
    }
    return ARTSS_OK;
}

// rows of whole pairs of cells take the two-cell kernels, which need the pairs aligned
// (256^3 pressure solve of 14 cycles: 7.2 ms by them, 9.5 by the one-cell kernels)
bool mx_pairs(const artss_mixed *m, const Level &L) {
    return L.Nx % 2 == 0 && m->cfg.n_relax > 1 && !(m->cfg.flags & (ARTSS_MIXED_BC_LAUNCH | ARTSS_MIXED_FINE_PROLONG));
}
// r carries its boundary cells, and the first two sweeps run as one
bool mx_zero_pair(const artss_mixed *m, int l) {
    return l + 1 < m->L && m->fold[l] && mx_pairs(m, m->ctx->lvl[l]);
}
inline dim3 pair_grid(const Level &L, const Box3 &b, int threads, int planes) {
    return dim3((unsigned) ((b.ny() * L.Nx / 2 + threads - 1) / threads), (unsigned) ((b.nz() + planes - 1) / planes));
}
// planes per thread of the kernels that walk up the planes: 8 blocks per SM for the
// latency of the loads, and no more, as each run reads the planes at its ends again
inline int pair_planes(const artss_ctx *ctx, const Box3 &b, int64_t blocks_xy) {
    return (int) std::max<int64_t>(1, std::min<int64_t>(32, blocks_xy * b.nz() / (8 * std::max(ctx->sm_count, 1))));
}

template <int MODE>
int mx_jacobi2(artss_mixed *m, int l, const CoefF &c, const LoopState *pred, double *p = nullptr, int push_p = 0) {
    artss_ctx *ctx = m->ctx;
    const Level &L = ctx->lvl[l];
    const Box3 box = inner_box(L);
    ARTSS_LAUNCH_PDL(ctx, FAM_MG_JACOBI, k_mx_jacobi2<MODE>, pair_grid(L, box, kPairThreads, kPairPlanes),
                     dim3(kPairThreads), 0, MODE == kPairFromZero ? m->e[l] : m->t[l],
                     MODE == kPairFromZero ? (const float *) m->r[l] : (const float *) m->e[l], (const float *) m->r[l],
                     (const uint8_t *) m->nbm[l], (const uint64_t *) m->push[l], L, box, c, pred, p, push_p);
    ARTSS_LAUNCH_CK(ctx);
    return ARTSS_OK;
}

// the correcting sweep writes p's boundary cells too: its program is homogeneous and
// wholly in level 0's patterns
int mx_pushes_p(const artss_mixed *m, const double *p) {
    return (uintptr_t) p % 16 == 0 && m->fold[0] && m->whole[0] && m->ctx->bc[0][ARTSS_FIELD_P].homogeneous;
}

// one weighted-Jacobi sweep m->t[l] <- m->e[l] (p: added to p instead, see
// k_mx_jacobi), in the launch shape tuned for the level (the p form repeats
// no launch, so it takes the shape the plain form was tuned to)
int mx_jacobi(artss_mixed *m, int l, const CoefF &c, const LoopState *pred, double *p, int push_p = 0) {
    artss_ctx *ctx = m->ctx;
    const Level &L = ctx->lvl[l];
    const Box3 box = inner_box(L);
    if (mx_pairs(m, L))
        return p ? mx_jacobi2<kPairCorrect>(m, l, c, pred, p, push_p) : mx_jacobi2<kPairSweep>(m, l, c, pred);
    return tuned_column_launch(ctx, kTuneMxJacobi, l, box, p == nullptr, [&](dim3 g, dim3 bl) -> int {
        if (p)
            ARTSS_LAUNCH_PDL(ctx, FAM_MG_JACOBI, k_mx_jacobi<true>, g, bl, 0, m->t[l], (const float *) m->e[l],
                             (const float *) m->r[l], (const uint8_t *) m->nbm[l], (const uint64_t *) m->push[l], L,
                             box, c, pred, p, push_p);
        else
            ARTSS_LAUNCH_PDL(ctx, FAM_MG_JACOBI, k_mx_jacobi<false>, g, bl, 0, m->t[l], (const float *) m->e[l],
                             (const float *) m->r[l], (const uint8_t *) m->nbm[l], (const uint64_t *) m->push[l], L,
                             box, c, pred, (double *) nullptr, 0);
        ARTSS_LAUNCH_CK(ctx);
        return ARTSS_OK;
    }, 256);
}

// n_relax weighted-Jacobi sweeps from e = 0 on level l, each followed by the
// boundary program; the result is left in m->e[l]
int mx_smooth_from_zero(artss_mixed *m, int l, const LoopState *pred) {
    if (m->cfg.flags & ARTSS_MIXED_RBGS) return mx_smooth_rbgs(m, l, true, pred);
    artss_ctx *ctx = m->ctx;
    const Level &L = ctx->lvl[l];
    const Box3 box = inner_box(L);
    const CoefF c = coef_f(ctx, l, m->cfg.w);
    int st, first = 1;
    if (mx_zero_pair(m, l)) {
        if ((st = mx_jacobi2<kPairFromZero>(m, l, c, pred))) return st;
        first = 2;
    } else if ((st = tuned_column_launch(ctx, kTuneMxJacobi0, l, box, true, [&](dim3 g, dim3 bl) -> int {
             ARTSS_LAUNCH_PDL(ctx, FAM_MG_JACOBI, k_mx_jacobi0, g, bl, 0, m->e[l], (const float *) m->r[l],
                              (const uint8_t *) m->nbm[l], (const uint64_t *) m->push[l], L, box, c, pred);
             ARTSS_LAUNCH_CK(ctx);
             return ARTSS_OK;
         })))
        return st;
    if (first == 1 && (st = mx_bc_sweep(m, m->e[l], l, pred))) return st;
    for (int s = first; s < m->cfg.n_relax; s++) {
        if ((st = mx_jacobi(m, l, c, pred, nullptr))) return st;
        std::swap(m->e[l], m->t[l]);
        if ((st = mx_bc_sweep(m, m->e[l], l, pred))) return st;
    }
    return ARTSS_OK;
}

// n_relax weighted-Jacobi sweeps continuing from m->e[l]; p: the last sweep
// adds its values to p (FP64) instead of storing them (the correction p += e
// of the outer loop, whose e is not read again); *corrected tells whether it did
int mx_smooth(artss_mixed *m, int l, const LoopState *pred, double *p = nullptr, bool *corrected = nullptr) {
    if (corrected) *corrected = false;
    if (m->cfg.flags & ARTSS_MIXED_RBGS) return mx_smooth_rbgs(m, l, false, pred);
    artss_ctx *ctx = m->ctx;
    const Level &L = ctx->lvl[l];
    const Box3 box = inner_box(L);
    const CoefF c = coef_f(ctx, l, m->cfg.w);
    int st;
    for (int s = 0; s < m->cfg.n_relax; s++) {
        if (p && s + 1 == m->cfg.n_relax) {
            if ((st = mx_jacobi(m, l, c, pred, p, mx_pushes_p(m, p)))) return st;
            if (corrected) *corrected = true;
            break;
        }
        if ((st = mx_jacobi(m, l, c, pred, nullptr))) return st;
        std::swap(m->e[l], m->t[l]);
        if ((st = mx_bc_sweep(m, m->e[l], l, pred))) return st;
    }
    return ARTSS_OK;
}

// Push patterns of levels 0 .. L-2 from the inner cells and the pressure
// boundary programs with every value zero (x_t = +-x_root after chain
// folding).  Every boundary cell that a smoothing or residual stencil reads
// (a face neighbour of an inner cell) must take its value from an inner cell one
// step away along an axis, which then writes it with each of its own values; where
// every other boundary cell takes its value from an inner cell among its 26
// neighbours too, the patterns hold the whole program.  A level where the former
// fails (a root that is not inner, not face-adjacent or itself written by
// the program, an inner target) or a solver with ARTSS_MIXED_RBGS /
// ARTSS_MIXED_BC_LAUNCH launches the program after each sweep instead, with a
// mask of inner bits only.  ARTSS_MIXED_BC_LAUNCH also keeps residual, its program
// and restriction apart and takes the one-cell kernels.
int mx_build_tables(artss_mixed *m) {
    artss_ctx *ctx = m->ctx;
    const bool allow = !(m->cfg.flags & (ARTSS_MIXED_RBGS | ARTSS_MIXED_BC_LAUNCH));
    for (int l = 0; l + 1 < m->L; l++) {
        const Level &L = ctx->lvl[l];
        const int64_t n = L.size();
        const CellBits &inner = ctx->inner_bits[l];
        const bool have_inner = inner.n == n;
        bool fold = allow && have_inner, whole = fold;
        const bool pairs = mx_pairs(m, L);
        std::vector<std::pair<int64_t, uint8_t>> partner;
        std::vector<std::pair<int64_t, uint64_t>> pat, far_pat;  // (inner cell, its share of the pattern): read targets, others
        const BcProgram &p = ctx->bc[l][ARTSS_FIELD_P];
        std::unordered_map<int64_t, std::pair<int64_t, int>> res;
        if (fold && p.present && p.n) {
            // final (root, sign) of every target, the program applied wave by wave
            res.reserve((size_t) p.n * 2);
            for (int64_t a = 0; a < p.n; a++) {
                int64_t r = p.h_root[(size_t) a];
                int sg = p.h_sign[(size_t) a];
                const auto it = p.waves > 1 ? res.find(r) : res.end();
                if (it != res.end()) {
                    r = it->second.first;
                    sg *= it->second.second;
                }
                res[p.h_target[(size_t) a]] = {r, sg};
            }
            const int64_t off[6] = {-1, 1, -L.Nx, L.Nx, -L.nxy(), L.nxy()};
            pat.reserve(res.size());
            for (const auto &kv : res) {
                const int64_t t = kv.first, r = kv.second.first;
                if (inner.get(t)) { fold = false; break; }
                bool read = false;  // t is a face neighbour of an inner cell
                for (int64_t d : off) read = read || (t - d >= 0 && t - d < n && inner.get(t - d));
                const int64_t tz = t / L.nxy(), ty = t / L.Nx % L.Ny, tx = t % L.Nx;
                const int64_t dx = tx - r % L.Nx, dy = ty - r / L.Nx % L.Ny, dz = tz - r / L.nxy();
                const int64_t far = std::max({std::abs(dx), std::abs(dy), std::abs(dz)});
                const bool root_ok = far == 1 && inner.get(r) && !res.count(r);
                if (read && !(root_ok && std::abs(dx) + std::abs(dy) + std::abs(dz) == 1)) { fold = false; break; }
                if (!root_ok) {
                    whole = false;
                    continue;
                }
                if (pairs && dy == 0 && dz == 0 && (std::min(tx, tx - dx) % 2 == 0)) {
                    partner.push_back({t, (uint8_t) (kv.second.second > 0 ? kPartnerPlus : kPartnerMinus)});
                    continue;
                }
                const int dir = (int) ((dx + 1) + 3 * (dy + 1) + 9 * (dz + 1));
                (read ? pat : far_pat).push_back({r, (kv.second.second > 0 ? 1ull : 2ull) << (2 * dir)});
            }
        }
        std::vector<uint8_t> nbm((size_t) n, 0);
        if (have_inner)
            for (int64_t i = 0; i < (int64_t) inner.w.size(); i++) {
                const uint64_t w = inner.w[(size_t) i];
                for (int64_t x = 64 * i; x < std::min(n, 64 * i + 64); x++) nbm[(size_t) x] = (uint8_t) (w >> (x & 63) & 1);
            }
        // distinct patterns -> ids 1..127, without the targets that no sweep reads
        // where they make too many
        std::vector<uint64_t> push(128, 0);
        std::vector<std::pair<int64_t, int>> of;
        const auto number = [&](std::vector<std::pair<int64_t, uint64_t>> v) {
            std::unordered_map<uint64_t, int> ids;
            std::sort(v.begin(), v.end());
            of.clear();
            std::fill(push.begin(), push.end(), (uint64_t) 0);
            for (size_t a = 0; a < v.size();) {
                const int64_t r = v[a].first;
                uint64_t bits = 0;
                for (; a < v.size() && v[a].first == r; a++) bits |= v[a].second;
                auto it = ids.find(bits);
                if (it == ids.end()) {
                    if (ids.size() >= 127) return false;
                    it = ids.emplace(bits, (int) ids.size() + 1).first;
                    push[(size_t) it->second] = bits;
                }
                of.push_back({r, it->second});
            }
            return true;
        };
        if (fold && whole) {
            far_pat.insert(far_pat.end(), pat.begin(), pat.end());
            whole = number(std::move(far_pat));
        }
        if (fold && !whole) fold = number(pat);
        if (fold)
            for (const auto &a : partner) nbm[(size_t) a.first] = a.second;
        if (fold)
            for (const auto &a : of) nbm[(size_t) a.first] = (uint8_t) (nbm[(size_t) a.first] | a.second << 1);
        else
            std::fill(push.begin(), push.end(), (uint64_t) 0);
        m->fold[l] = fold;
        m->whole[l] = fold && whole;
        // the children of the coarse inner cells are inner or touched by nothing
        const Level &C = ctx->lvl[l + 1];
        const CellBits &cin = ctx->inner_bits[l + 1];
        bool dead = have_inner && !(m->cfg.flags & ARTSS_MIXED_BC_LAUNCH) && cin.n == C.size() && C.i1 >= 1 && C.j1 >= 1 && C.k1 >= 1 &&
                    2 * C.i2 + 1 < L.Nx && 2 * C.j2 + 1 < L.Ny && 2 * C.k2 + 1 < L.Nz;
        for (int64_t t : p.h_target) {
            if (!dead) break;
            const int64_t ci = (t % L.Nx + 1) / 2, cj = (t / L.Nx % L.Ny + 1) / 2, ck = (t / L.nxy() + 1) / 2;
            dead = ci >= C.Nx || cj >= C.Ny || ck >= C.Nz || !cin.get(ci + C.Nx * cj + C.nxy() * ck);
        }
        m->q_bc_dead[l] = dead;
        // r's boundary cells are written from the patterns: none of an earlier geometry's
        ARTSS_CK(cudaMemsetAsync(m->r[l], 0, (size_t) n * sizeof(float), ctx->stream));
        if (!m->nbm[l]) ARTSS_CK(cudaMalloc(&m->nbm[l], (size_t) n));
        if (!m->push[l]) ARTSS_CK(cudaMalloc(&m->push[l], 128 * sizeof(uint64_t)));
        ARTSS_CK(cudaMemcpyAsync(m->push[l], push.data(), 128 * sizeof(uint64_t), cudaMemcpyHostToDevice, ctx->stream));
        ARTSS_CK(cudaMemcpyAsync(m->nbm[l], nbm.data(), (size_t) n, cudaMemcpyHostToDevice, ctx->stream));
        // the host vectors die with this iteration
        ARTSS_CK(cudaStreamSynchronize(ctx->stream));
    }
    m->geom_version = ctx->geom_version;
    return ARTSS_OK;
}

// FP32 V-cycle on A e = r[0] with e = 0 at start; result in m->e[0], or, with p,
// added to p by the last smoothing sweep where *corrected says so
int mx_vcycle(artss_mixed *m, const LoopState *pred, double *p = nullptr, bool *corrected = nullptr) {
    artss_ctx *ctx = m->ctx;
    const int Lc = m->L - 1;  // coarsest level
    const artss_grid_desc &g = ctx->grid;
    int st;
    for (int l = 0; l < Lc; l++) {
        if ((st = mx_smooth_from_zero(m, l, pred))) return st;
        const Level &L = ctx->lvl[l];
        const Box3 box = inner_box(L);
        if (m->q_bc_dead[l]) {
            const Level &C = ctx->lvl[l + 1];
            const Box3 cbox = inner_box(C);
            if (mx_pairs(m, L)) {
                const bool push = mx_zero_pair(m, l + 1);
                dim3 gr((unsigned) ((cbox.nx() + 30) / 31), (unsigned) ((cbox.ny() + 7) / 8));
                const int planes = pair_planes(ctx, cbox, (int64_t) gr.x * gr.y);
                gr.z = (unsigned) ((cbox.nz() + planes - 1) / planes);
                ARTSS_LAUNCH_PDL(ctx, FAM_MG_RESIDUUM, k_mx_down2, gr, dim3(32, 8), 0, m->r[l + 1],
                                 (const float *) m->e[l], (const float *) m->r[l], (const uint8_t *) ctx->d_flags[l + 1],
                                 (const uint8_t *) m->nbm[l], (const uint8_t *) (push ? m->nbm[l + 1] : nullptr),
                                 (const uint64_t *) m->push[l + 1], C, L, cbox, planes, (float) (1. / (g.dx[l] * g.dx[l])),
                                 (float) (1. / (g.dy[l] * g.dy[l])), (float) (1. / (g.dz[l] * g.dz[l])), pred);
                ARTSS_LAUNCH_CK(ctx);
            } else if ((st = tuned_column_launch(ctx, kTuneMxDown, l + 1, cbox, true, [&](dim3 gr, dim3 bl) -> int {
                     ARTSS_LAUNCH_PDL(ctx, FAM_MG_RESIDUUM, k_mx_residuum_restrict, gr, bl, 0, m->r[l + 1],
                                      (const float *) m->e[l], (const float *) m->r[l],
                                      (const uint8_t *) ctx->d_flags[l + 1], (const uint8_t *) m->nbm[l], C, L, cbox,
                                      (float) (1. / (g.dx[l] * g.dx[l])), (float) (1. / (g.dy[l] * g.dy[l])),
                                      (float) (1. / (g.dz[l] * g.dz[l])), pred);
                     ARTSS_LAUNCH_CK(ctx);
                     return ARTSS_OK;
                 }, 256)))
                return st;
            else if (mx_zero_pair(m, l + 1) && (st = mx_bc(m, m->r[l + 1], l + 1, pred)))
                return st;
            continue;
        }
        if ((st = tuned_column_launch(ctx, kTuneMxResiduum, l, box, true, [&](dim3 gr, dim3 bl) -> int {
                 ARTSS_LAUNCH_PDL(ctx, FAM_MG_RESIDUUM, k_mx_residuum, gr, bl, 0, m->q[l], (const float *) m->e[l],
                                  (const float *) m->r[l], (const uint8_t *) m->nbm[l], L, box,
                                  (float) (1. / (g.dx[l] * g.dx[l])), (float) (1. / (g.dy[l] * g.dy[l])),
                                  (float) (1. / (g.dz[l] * g.dz[l])), pred);
                 ARTSS_LAUNCH_CK(ctx);
                 return ARTSS_OK;
             }, 256)))
            return st;
        if ((st = mx_bc(m, m->q[l], l, pred))) return st;
        const Level &C = ctx->lvl[l + 1];
        const Box3 cbox = inner_box(C);
        if ((st = tuned_column_launch(ctx, kTuneMxRestrict, l + 1, cbox, true, [&](dim3 gr, dim3 bl) -> int {
                 ARTSS_LAUNCH_PDL(ctx, FAM_MG_RESTRICT, k_mx_restrict, gr, bl, 0, m->r[l + 1], m->q[l],
                                  ctx->d_flags[l + 1], C, L, cbox, pred);
                 ARTSS_LAUNCH_CK(ctx);
                 return ARTSS_OK;
             })))
            return st;
        if (mx_zero_pair(m, l + 1) && (st = mx_bc(m, m->r[l + 1], l + 1, pred))) return st;
    }
    // coarsest level: FP64 solve from zero
    {
        double w = m->cfg.coarse_w;
        if (w <= 0) {
            // red-black SOR with the optimal weight of the model problem on this grid
            const Level &C = ctx->lvl[Lc];
            const double n = (double) std::max({C.i2 - C.i1 + 1, C.j2 - C.j1 + 1, C.k2 - C.k1 + 1});
            w = m->cfg.coarse_smoother == ARTSS_SMOOTHER_CGS ? 2. / (1. + sin(M_PI / (n + 1.))) : 0.6666666667;
        }
        if ((st = coarse_cluster_f32(ctx, m->e[Lc], m->r[Lc], Lc, m->cfg.coarse_smoother, w, m->cfg.coarse_rel_tol,
                                     m->cfg.coarse_max_iter, pred, !(m->cfg.flags & ARTSS_MIXED_CLUSTER_COARSE),
                                     true)))
            return st;
    }
    for (int l = Lc - 1; l >= 0; l--) {
        // the prolongation reads the coarse correction's boundary cells (edges
        // and corners too): the level's program once, where the sweeps skipped it and
        // did not write them all
        if (l + 1 < Lc && m->fold[l + 1] && !m->whole[l + 1] && (st = mx_bc(m, m->e[l + 1], l + 1, pred))) return st;
        const Level &C = ctx->lvl[l + 1], &F = ctx->lvl[l];
        // the fine children 2c - 1, 2c of the coarse inner box, within the fine inner box
        const Box3 fbox{std::max(F.i1, 2 * C.i1 - 1), std::min(F.i2, 2 * C.i2), std::max(F.j1, 2 * C.j1 - 1),
                        std::min(F.j2, 2 * C.j2), std::max(F.k1, 2 * C.k1 - 1), std::min(F.k2, 2 * C.k2)};
        const Box3 cbox = inner_box(C);
        if (m->cfg.flags & ARTSS_MIXED_FINE_PROLONG) {
            ARTSS_LAUNCH_PDL(ctx, FAM_MG_PROLONGATE, k_mx_prolong_add, mx_grid(fbox), box_block(), 0,
                             m->e[l], (const float *) m->e[l + 1], (const uint8_t *) ctx->d_flags[l + 1],
                             (const uint8_t *) m->nbm[l], (const uint64_t *) m->push[l], C, F, fbox, pred);
        } else if (mx_pairs(m, F)) {
            const dim3 gr((unsigned) ((cbox.nx() + 31) / 31), (unsigned) ((cbox.ny() + 7) / 8), (unsigned) cbox.nz());
            ARTSS_LAUNCH_PDL(ctx, FAM_MG_PROLONGATE, k_mx_prolong_add2, gr, dim3(32, 8), 0, m->e[l],
                             (const float *) m->e[l + 1], (const uint8_t *) ctx->d_flags[l + 1],
                             (const uint8_t *) m->nbm[l], (const uint64_t *) m->push[l], C, F, cbox, fbox, pred);
        } else {
            ARTSS_LAUNCH_PDL(ctx, FAM_MG_PROLONGATE, k_mx_prolong_add8, mx_grid(cbox), box_block(), 0,
                             m->e[l], (const float *) m->e[l + 1], (const uint8_t *) ctx->d_flags[l + 1],
                             (const uint8_t *) m->nbm[l], (const uint64_t *) m->push[l], C, F, cbox, fbox, pred);
        }
        ARTSS_LAUNCH_CK(ctx);
        if ((st = mx_bc_sweep(m, m->e[l], l, pred))) return st;
        if ((st = mx_smooth(m, l, pred, l == 0 ? p : nullptr, l == 0 ? corrected : nullptr))) return st;
    }
    return ARTSS_OK;
}

// sum(x - shift) and sum((x - shift)^2) over level-0 inner cells, read back
int mx_moments(artss_mixed *m, const double *x, double shift, double *s1, double *s2) {
    artss_ctx *ctx = m->ctx;
    const Level &L = ctx->lvl[0];
    const Box3 box = inner_box(L);
    const dim3 grid = mx_grid(box);
    int st;
    if ((st = check_reduce_blocks(grid))) return st;
    const int nb = (int) (grid.x * grid.y * grid.z);
    ARTSS_LAUNCH_PDL(ctx, FAM_MG_RESNORM, k_mx_moments, grid, box_block(), 0, 
                                          x, shift, ctx->d_flags[0], L, box, ctx->d_partials, ctx->d_partials + nb);
    ARTSS_LAUNCH_CK(ctx);
    LoopState a{}, b{};
    if ((st = finalize_sum(ctx, kSlotSum, nb))) return st;
    if ((st = read_loop(ctx, kSlotSum, &a))) return st;
    ARTSS_CK(cudaMemcpyAsync(ctx->d_partials, ctx->d_partials + nb, nb * sizeof(double), cudaMemcpyDeviceToDevice,
                             ctx->stream));
    if ((st = finalize_sum(ctx, kSlotSum, nb))) return st;
    if ((st = read_loop(ctx, kSlotSum, &b))) return st;
    *s1 = a.sum;
    *s2 = b.sum;
    return ARTSS_OK;
}

}  // namespace
}  // namespace artss

using namespace artss;

extern "C" {

int artss_mixed_create(artss_ctx *ctx, const artss_mixed_cfg *cfg, artss_mixed **out) {
    if (!ctx || !cfg || !out) { set_error("null argument"); return ARTSS_ERR_ARG; }
    *out = nullptr;
    if (cfg->n_level < 2 || cfg->n_level > ctx->grid.n_levels + 1) {
        set_error("n_level must be at least 2 and at most the context's levels + 1"); return ARTSS_ERR_ARG;
    }
    if (cfg->n_relax < 1 || cfg->max_cycles < 0 || cfg->coarse_max_iter < 0 || !(cfg->rel_tol >= 0) ||
        (cfg->coarse_smoother != ARTSS_SMOOTHER_JACOBI && cfg->coarse_smoother != ARTSS_SMOOTHER_CGS)) {
        set_error("invalid mixed-precision settings"); return ARTSS_ERR_ARG;
    }
    auto *m = new artss_mixed();
    m->ctx = ctx;
    m->cfg = *cfg;
    m->L = cfg->n_level;
    int st = ARTSS_OK;
    for (int l = 0; l < m->L && !st; l++) {
        const size_t bytes = (size_t) ctx->lvl[l].size() * sizeof(float);
        for (float **f : {&m->r[l], &m->q[l], &m->e[l], &m->t[l]}) {
            cudaError_t e = cudaMalloc((void **) f, bytes);
            if (e == cudaSuccess) e = cudaMemsetAsync(*f, 0, bytes, ctx->stream);
            if (e != cudaSuccess) { st = cuda_fail(e, "mixed-precision level arrays"); break; }
        }
    }
    if (!st) {
        int cap = 0;
        int64_t smem = 0;
        const int buffers = cfg->coarse_smoother == ARTSS_SMOOTHER_CGS ? 1 : 2;
        if (!cluster_fits(ctx, m->L - 1, buffers, &cap, &smem) &&
            ((cfg->flags & ARTSS_MIXED_CLUSTER_COARSE) || !block_fits(ctx, m->L - 1, buffers, &smem))) {
            set_error("the coarsest level is too large for the cluster coarse solve; use more levels");
            st = ARTSS_ERR_LIMIT;
        }
    }
    if (!st) st = cudaStreamSynchronize(ctx->stream) == cudaSuccess ? ARTSS_OK : cuda_fail(cudaGetLastError(), "sync");
    if (!st) st = mx_build_tables(m);
    if (st) { artss_mixed_destroy(m); return st; }
    *out = m;
    return ARTSS_OK;
}

int artss_mixed_destroy(artss_mixed *m) {
    if (!m) return ARTSS_OK;
    cudaStreamSynchronize(m->ctx->stream);
    for (int l = 0; l <= kMaxLevel; l++) {
        for (float *f : {m->r[l], m->q[l], m->e[l], m->t[l]})
            if (f) cudaFree(f);
        if (m->nbm[l]) cudaFree(m->nbm[l]);
        if (m->push[l]) cudaFree(m->push[l]);
    }
    delete m;
    return ARTSS_OK;
}

int artss_laplacian(artss_ctx *ctx, double *out, double *p, int level) {
    if (!ctx || !out || !p || out == p) { set_error("null or aliased argument"); return ARTSS_ERR_ARG; }
    int st = check_level(ctx, level);
    if (st) return st;
    if ((st = apply_bc(ctx, p, level, ARTSS_FIELD_P))) return st;
    const Level &L = ctx->lvl[level];
    const Box3 box = inner_box(L);
    const artss_grid_desc &g = ctx->grid;
    ARTSS_LAUNCH_PDL(ctx, FAM_MG_RESIDUUM, k_mx_laplacian, mx_grid(box), box_block(), 0, 
                                           out, p, ctx->d_flags[level], L, box, 1. / (g.dx[level] * g.dx[level]),
                                           1. / (g.dy[level] * g.dy[level]), 1. / (g.dz[level] * g.dz[level]));
    ARTSS_LAUNCH_CK(ctx);
    return ARTSS_OK;
}

int artss_mixed_solve(artss_mixed *m, double *p, const double *b, artss_solve_stats *stats) {
    if (!m || !p || !b) { set_error("null argument"); return ARTSS_ERR_ARG; }
    artss_ctx *ctx = m->ctx;
    const Level &L = ctx->lvl[0];
    const Box3 box = inner_box(L);
    const artss_grid_desc &g = ctx->grid;
    const bool remove_mean = (m->cfg.flags & ARTSS_MIXED_REMOVE_MEAN) != 0;
    const int64_t n_inner = ctx->n_inner[0];
    int st;
    const dim3 grid = mx_grid(box);
    if ((st = check_reduce_blocks(grid))) return st;
    // at most 4096 partial sums for the last block to add, where planes allow it
    const int64_t pair_blocks = (box.ny() * L.Nx / 2 + 255) / 256;
    const int planes = (int) std::max<int64_t>(pair_planes(ctx, box, pair_blocks), pair_blocks * box.nz() / 4096);
    const dim3 pgrid = pair_grid(L, box, 256, planes);
    if ((st = check_reduce_blocks(pgrid))) return st;
    if (m->geom_version != ctx->geom_version) {
        // cell lists or boundary programs changed since the tables were built
        if (ctx->capturing) { set_error("the mixed solver's boundary tables are stale; solve once before capturing"); return ARTSS_ERR_ARG; }
        if ((st = mx_build_tables(m))) return st;
    }
    const int nb = (int) (grid.x * grid.y * grid.z);
    // ||b|| for the relative stopping rule: on the host, or (inside a capture)
    // kept in loop slot kSlotSum and applied by the loop step on the device
    double s1 = 0, s2 = 0;
    if (ctx->capturing) {
        if (remove_mean) { set_error("the mean removal reads sums on the host and cannot be captured"); return ARTSS_ERR_ARG; }
        ARTSS_LAUNCH_PDL(ctx, FAM_MG_RESNORM, k_mx_moments, grid, box_block(), 0, 
                                              b, 0.0, ctx->d_flags[0], L, box, ctx->d_partials, ctx->d_partials + nb);
        ARTSS_LAUNCH_CK(ctx);
        ARTSS_CK(cudaMemcpyAsync(ctx->d_partials, ctx->d_partials + nb, nb * sizeof(double), cudaMemcpyDeviceToDevice,
                                 ctx->stream));
        if ((st = finalize_sum(ctx, kSlotSum, nb))) return st;
    } else if ((st = mx_moments(m, b, 0.0, &s1, &s2))) {
        return st;
    }
    const double b_norm = sqrt(s2);
    const double tol = m->cfg.rel_tol * b_norm;
    if ((st = apply_bc(ctx, p, 0, ARTSS_FIELD_P))) return st;

    const double rx = 1. / (g.dx[0] * g.dx[0]), ry = 1. / (g.dy[0] * g.dy[0]), rz = 1. / (g.dz[0] * g.dz[0]);
    const long long max_eval = m->cfg.max_cycles + 1;
    if ((st = init_loop(ctx, kSlotOuter, 1e300, 0, 1))) return st;
    const LoopState *pred = ctx->d_loop + kSlotOuter;
    LoopState ls{};
    long long it = 0;
    bool cond = true;
    int64_t batch = std::max<int64_t>(1, std::min<int64_t>(m->hint, max_eval));
    GraphLoop gl;
    if (ctx->capturing) {
        // one outer iteration per body of a WHILE node decided on the device
        if ((st = gl.begin(ctx, 1))) return st;
        batch = 1;
    }
    while (cond) {
        for (int64_t r = 0; r < batch; r++) {
            const LoopState *ref = ctx->capturing ? ctx->d_loop + kSlotSum : nullptr;
            const double eps = ctx->capturing ? m->cfg.rel_tol : tol;
            if (mx_pairs(m, L))
                ARTSS_LAUNCH_PDL(ctx, FAM_MG_RESNORM, k_mx_outer_residual2, pgrid, dim3(256), 0, (const double *) p, b,
                                 m->r[0], (const uint8_t *) m->nbm[0], (const uint64_t *) m->push[0], L, box, planes,
                                 rx, ry, rz,
                                 ctx->d_partials, ctx->d_loop + kSlotOuter, ref, eps, max_eval);
            else
                ARTSS_LAUNCH_PDL(ctx, FAM_MG_RESNORM, k_mx_outer_residual, grid, box_block(), 0, (const double *) p, b,
                                 m->r[0], (const uint8_t *) ctx->d_flags[0], L, box, rx, ry, rz,
                                 ctx->d_partials, ctx->d_loop + kSlotOuter, ref, eps, max_eval);
            ARTSS_LAUNCH_CK(ctx);
            bool corrected = false;
            if ((st = mx_vcycle(m, pred, p, &corrected))) return st;
            if (!corrected) {
                ARTSS_LAUNCH_PDL(ctx, FAM_FIELD_OP, k_mx_correct, grid, box_block(), 0,
                                                    p, m->e[0], ctx->d_flags[0], L, box, pred);
                ARTSS_LAUNCH_CK(ctx);
            }
            if (!(corrected && mx_pushes_p(m, p)) && (st = apply_bc(ctx, p, 0, ARTSS_FIELD_P, pred))) return st;
        }
        if (ctx->capturing) {
            if ((st = gl.end(kSlotOuter, max_eval + 2))) return st;
            if (stats) *stats = artss_solve_stats{-1, -1.0, -1.0, -1.0};
            return ARTSS_OK;
        }
        if ((st = read_loop(ctx, kSlotOuter, &ls))) return st;
        it = ls.it;
        cond = ls.cond != 0;
        batch = std::max<int64_t>(1, std::min<int64_t>(2 * batch, max_eval - it));
    }
    m->hint = std::max<int64_t>(1, it);
    if (remove_mean && n_inner > 0) {
        double p1 = 0, p2 = 0;
        if ((st = mx_moments(m, p, 0.0, &p1, &p2))) return st;
        // a uniform shift keeps every Neumann ghost relation
        if ((st = artss_add_scalar(ctx, p, -p1 / (double) n_inner, 0))) return st;
    }
    if (stats) {
        stats->cycles = it - 1;
        stats->residual = ls.residual;
        stats->rel_residual = b_norm > 0 ? ls.residual / b_norm : ls.residual;
        stats->b_norm = b_norm;
    }
    return ARTSS_OK;
}

}  // extern "C"
