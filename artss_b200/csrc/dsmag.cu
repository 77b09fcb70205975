// DynamicSmagorinsky (src/turbulence/DynamicSmagorinsky.cpp:172-427): eddy
// viscosity of the dynamic Smagorinsky-Lilly model on level 0, FP64, with the
// reference's loops restated as passes over the inner cells:
//   1. u_f, v_f, w_f = explicit filter of u, v, w (trapezoidal 3x3x3 weights,
//      the sum over x offsets outermost and z offsets innermost, :384-427);
//   2. strain tensor S_ij of the filtered velocities and |S| (:200-282);
//   3. one pass for everything up to the coefficient: products of the filtered
//      velocities (the reference's "velocity products" are the filtered ones
//      too) and P_ij = |S| S_ij are formed where they are read, the filters of
//      the products (uu, vv, ww, uv, vw; the reference filters ww twice and never
//      uw, whose filter stays zero), of S_ij and of P_ij are summed side by side,
//      then Leonard stress, M_ij and Cs = num / den with the reference's products
//      of the 22 and 33 terms in num and den (:298-344);
//   4. the 27-cell average of Cs in place in list order, so that a cell sees
//      the averaged values of every neighbour before it in the list, then
//      ev = 2 Cs delta_s^2 |S| and ev = 0 where ev + nu < 0 (:350-376).
// Every sum keeps the reference's order; a filter weight is a power of two, so
// that fma(weight, value, sum) rounds exactly as sum + weight * value does.
// Step 4 is sequential in the reference.  Every neighbour that precedes a cell
// in the list has a smaller t = i + 2j + 4k, every one that follows has a larger
// t and no two neighbours share a t: any schedule in the order of t reads exactly
// what the sequential loop reads.  The work fields live in the context, zero
// outside the inner cells (the reference's fields start zero and only inner cells
// are written).
#include "internal.cuh"

#include <algorithm>
#include <cmath>
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace artss {
namespace {

enum DsArr : int { UF, VF, WF, S11, S22, S33, S12, S13, S23, SBAR, CS, DS_ARRAYS };
constexpr int kDsProgress = 512;  // ints behind the work fields: progress per block, the last one an error flag

#define DS_COLUMN(box)                                                             \
    const int i = (int) (box).x0 + (int) (blockIdx.x * blockDim.x + threadIdx.x); \
    const int j = (int) (box).y0 + (int) (blockIdx.y * blockDim.y + threadIdx.y); \
    if (i > (int) (box).x1 || j > (int) (box).y1) return

inline dim3 ds_grid(const Box3 &b) {
    dim3 g = box_grid(b);
    const int64_t xy = (int64_t) g.x * g.y;
    int64_t gz = b.nz();
    const int64_t cap = std::max<int64_t>(1, 2048 / std::max<int64_t>(xy, 1));
    if (gz > cap) gz = cap;
    g.z = (unsigned) std::max<int64_t>(gz, 1);
    return g;
}

// planes [k0, k1] of this block: a contiguous run of the box
__device__ __forceinline__ void ds_planes(const Box3 &box, int &k0, int &k1) {
    const int nz = (int) box.nz(), chunk = (nz + (int) gridDim.z - 1) / (int) gridDim.z;
    k0 = (int) box.z0 + (int) blockIdx.z * chunk;
    k1 = min((int) box.z1, k0 + chunk - 1);
}

// explicit_filtering of u, v, w: sum over l (x), m (y), n (z) of a[l] a[m] a[n]
// in[...], a = (1/4, 1/2, 1/4).  A thread marches up its column with the 3 x 3 x 3
// neighbourhood in registers, nine new values a plane.
__global__ void k_ds_filter(const double *__restrict__ u, const double *__restrict__ v, const double *__restrict__ w,
                            double *__restrict__ A, const uint8_t *__restrict__ flags, Level L, Box3 box, int64_t N) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    DS_COLUMN(box);
    const int nj = (int) L.Nx, nk = (int) L.nxy();
    int k0, k1;
    ds_planes(box, k0, k1);
    if (k0 > k1) return;
    const int q0 = i + nj * j;
    for (int f = 0; f < 3; f++) {
        const double *__restrict__ in = f == 0 ? u : f == 1 ? v : w;
        double *__restrict__ out = A + (UF + f) * N;
        double p[3][3][3];  // plane, x, y
        auto plane = [&](int k, double (&d)[3][3]) {
#pragma unroll
            for (int l = 0; l < 3; l++)
#pragma unroll
                for (int m = 0; m < 3; m++) d[l][m] = in[q0 + nk * k + l - 1 + nj * (m - 1)];
        };
        plane(k0 - 1, p[0]);
        plane(k0, p[1]);
        for (int k = k0; k <= k1; k++) {
            const int q = q0 + nk * k;
            const uint8_t fl = flags[q];
            plane(k + 1, p[2]);
            double sum = 0;
#pragma unroll
            for (int l = 0; l < 3; l++)
#pragma unroll
                for (int m = 0; m < 3; m++)
#pragma unroll
                    for (int n = 0; n < 3; n++)
                        sum = __fma_rn((l == 1 ? 0.5 : 0.25) * (m == 1 ? 0.5 : 0.25) * (n == 1 ? 0.5 : 0.25), p[n][l][m],
                                       sum);
            if (fl & kInner) out[q] = sum;
#pragma unroll
            for (int l = 0; l < 3; l++)
#pragma unroll
                for (int m = 0; m < 3; m++) {
                    p[0][l][m] = p[1][l][m];
                    p[1][l][m] = p[2][l][m];
                }
        }
    }
}

// strain tensor of the filtered velocities and |S|
__global__ void k_ds_strain(double *__restrict__ A, const uint8_t *__restrict__ flags, Level L, Box3 box, int64_t N,
                            double rdx, double rdy, double rdz) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    DS_COLUMN(box);
    const int nj = (int) L.Nx, nk = (int) L.nxy();
    const double *uf = A + UF * N, *vf = A + VF * N, *wf = A + WF * N;
    struct S { double s11, s22, s33, s12, s13, s23; };
    column_planes<2>(i + nj * j, nk, (int) box.z0, (int) box.z1, flags,
        [&](int q, int) {
            S s;
            s.s11 = (uf[q + 1] - uf[q - 1]) * 0.5 * rdx;
            s.s22 = (vf[q + nj] - vf[q - nj]) * 0.5 * rdy;
            s.s33 = (wf[q + nk] - wf[q - nk]) * 0.5 * rdz;
            s.s12 = 0.5 * ((uf[q + nj] - uf[q - nj]) * 0.5 * rdy + (vf[q + 1] - vf[q - 1]) * 0.5 * rdx);
            s.s13 = 0.5 * ((uf[q + nk] - uf[q - nk]) * 0.5 * rdz + (wf[q + 1] - wf[q - 1]) * 0.5 * rdx);
            s.s23 = 0.5 * ((vf[q + nk] - vf[q - nk]) * 0.5 * rdz + (wf[q + nj] - wf[q - nj]) * 0.5 * rdy);
            return s;
        },
        [&](int q, int, const S &s, uint8_t) {
            A[S11 * N + q] = s.s11;
            A[S22 * N + q] = s.s22;
            A[S33 * N + q] = s.s33;
            A[S12 * N + q] = s.s12;
            A[S13 * N + q] = s.s13;
            A[S23 * N + q] = s.s23;
            A[SBAR * N + q] = sqrt(2. * (s.s11 * s.s11 + s.s22 * s.s22 + s.s33 * s.s33 + 2. * (s.s12 * s.s12) +
                                         2. * (s.s13 * s.s13) + 2. * (s.s23 * s.s23)));
        });
}

// Products, the 17 filters, Leonard stress, M_ij and the dynamic coefficient Cs
// = num / den in one pass.  A thread owns two cells that are neighbours in y: 12
// of the 18 values an x column of theirs needs are shared, and the products are
// formed once for both.  Bound by the FP64 pipe and the L1 reads together (some
// 660 double-precision instructions and 180 loads a cell); kept apart, the
// products and the filtered fields cost 60 reads and writes of whole arrays.
constexpr int kDsCx = 32, kDsCy = 4;  // threads of a block: a tile of 32 x 8 cells
__global__ void __launch_bounds__(kDsCx * kDsCy)
k_ds_coefficient(double *__restrict__ A, const uint8_t *__restrict__ flags, Level L, Box3 box, int64_t N,
                 double delta_s, int *__restrict__ progress) {
    pdl_wait();  // launched by launch_pdl: the predecessor's writes are visible after this
    pdl_trigger();
    if (blockIdx.x + blockIdx.y + blockIdx.z == 0)  // for the averaging that follows
        for (int t = (int) (threadIdx.x + kDsCx * threadIdx.y); t < kDsProgress; t += kDsCx * kDsCy) progress[t] = 0;
    const int i = (int) box.x0 + (int) (blockIdx.x * kDsCx + threadIdx.x);
    const int j = (int) box.y0 + 2 * (int) (blockIdx.y * kDsCy + threadIdx.y);
    if (i > (int) box.x1 || j > (int) box.y1) return;
    const int nj = (int) L.Nx, nk = (int) L.nxy();
    const bool two = j + 1 <= (int) box.y1;
    const double *__restrict__ uf = A + UF * N, *__restrict__ vf = A + VF * N, *__restrict__ wf = A + WF * N,
                 *__restrict__ st = A + S11 * N, *__restrict__ sb = A + SBAR * N;
    const double alpha = 2.0;
    int k0, k1;
    ds_planes(box, k0, k1);
    for (int k = k0; k <= k1; k++) {
        const int q = i + nj * j + nk * k;
        double s[2][17];
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
            for (int t = 0; t < 17; t++) s[c][t] = 0;
#pragma unroll 1
        for (int l = -1; l <= 1; l++) {
            const double wl = l == 0 ? 0.5 : 0.25;
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int qr = q + l + nj * (r == 3 && !two ? 1 : r - 1);
#pragma unroll
                for (int n = -1; n <= 1; n++) {
                    const int x = qr + nk * n;
                    const double a = uf[x], b = vf[x], c = wf[x], sn = sb[x];
                    double v[17];
                    v[0] = a * a;
                    v[1] = b * b;
                    v[2] = c * c;
                    v[3] = a * b;
                    v[4] = b * c;
#pragma unroll
                    for (int t = 0; t < 6; t++) {
                        v[5 + t] = st[t * N + x];
                        v[11 + t] = sn * v[5 + t];
                    }
                    const double wn = wl * (n == 0 ? 0.5 : 0.25);
                    if (r < 3) {
                        const double w = wn * (r == 1 ? 0.5 : 0.25);
#pragma unroll
                        for (int t = 0; t < 17; t++) s[0][t] = __fma_rn(w, v[t], s[0][t]);
                    }
                    if (r > 0) {
                        const double w = wn * (r == 2 ? 0.5 : 0.25);
#pragma unroll
                        for (int t = 0; t < 17; t++) s[1][t] = __fma_rn(w, v[t], s[1][t]);
                    }
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const int x = q + nj * c;
            if ((c == 1 && !two) || !(flags[x] & kInner)) continue;
            const double *f = s[c];
            const double a = uf[x], b = vf[x], d = wf[x];
            const double l11 = f[0] - a * a;
            const double l22 = f[1] - b * b;
            const double l33 = f[2] - d * d;
            const double l12 = f[3] - a * b;
            const double l13 = 0.0 - a * d;  // the filter of uw is never formed: zero
            const double l23 = f[4] - b * d;
            const double f11 = f[5], f22 = f[6], f33 = f[7], f12 = f[8], f13 = f[9], f23 = f[10];
            const double sbf = sqrt(2. * (f11 * f11 + f22 * f22 + f33 * f33 + 2. * (f12 * f12) + 2. * (f13 * f13) +
                                          2. * (f23 * f23)));
            const double m11 = 2.0 * delta_s * delta_s * (f[11] - alpha * alpha * sbf * f11);
            const double m22 = 2.0 * delta_s * delta_s * (f[12] - alpha * alpha * sbf * f22);
            const double m33 = 2.0 * delta_s * delta_s * (f[13] - alpha * alpha * sbf * f33);
            const double m12 = 2.0 * delta_s * delta_s * (f[14] - alpha * alpha * sbf * f12);
            const double m13 = 2.0 * delta_s * delta_s * (f[15] - alpha * alpha * sbf * f13);
            const double m23 = 2.0 * delta_s * delta_s * (f[16] - alpha * alpha * sbf * f23);
            const double num = l11 * m11 + l22 * m22 * l33 * m33 + 2.0 * l12 * m12 + 2.0 * l13 * m13 + 2.0 * l23 * m23;
            const double den = m11 * m11 + m22 * m22 * m33 * m33 + 2.0 * m12 * m12 + 2.0 * m13 * m13 + 2.0 * m23 * m23;
            A[CS * N + x] = num / den;
        }
    }
}

// x / 27 by Markstein's correction (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990): with y = RN(1 / 27),
// which is off by a quarter of an ulp, q = RN(x y) is within one ulp of x / 27 and
// RN(q + (x - 27 q) y) is the correctly rounded quotient.  Numbers whose products
// leave the normal range, zeros, infinities and NaN take the division.
__device__ __forceinline__ double div27(double x) {
    const double y = 1.0 / 27.0, m = fabs(x);
    if (!(m > 1e-280 && m < 1e300)) return x / 27.0;
    const double q = x * y;
    return __fma_rn(__fma_rn(-27.0, q, x), y, q);
}

// The in-place 27-cell average of Cs.
//
// The order of t is a wave that needs nx + 2 ny + 4 nz steps, each a chain of 23
// dependent additions and a division, so the whole is bound by latency and by how
// a value gets to the next step.  A grid barrier per step and values through L2
// cost some 4.5 us a step; here a block owns kn neighbouring planes, one thread a
// (j, k) row of them, and a step's values travel through shared memory under a
// block barrier: step s updates cell i = x0 - 2 + s - 2 (j - y0) - 4 (k - k0) of
// every row.  A ring of kAvRing columns per row (the block's planes and one on
// each side, one row on each side) holds what the rows read; a thread keeps its
// 27 values in registers and reads the nine of the next column.
// At 192 x 96 x 96 (5 planes a block) the averaging takes 1.21 ms alone, 4.5 ms
// before; several calls in flight overlap, since a call uses 20 multiprocessors.
// Loader warps fill the ring kAvG steps ahead.  Rows of the plane before the
// block's first are read once the block that owns it has published that it has
// updated them (the wait is bounded; a block that gives up raises two flags and
// ends: k_ds_ev then writes NaN, and the context's next wait reports the error); every other row is read as the
// reference reads it, before its update: its columns are loaded at least one
// column before their own block, or the next one, gets to them.
// Blocks wait on the block before them, so all are resident (cooperative launch).
constexpr int kAvG = 8, kAvRing = 32, kAvPitch = 33;  // an odd pitch spreads the rows over the banks
constexpr int kAvRows = 512, kAvLoaders = 128;        // rows (threads) of a block at most; loading threads
constexpr size_t kAvSmemMax = 225 * 1024;             // of a block at most

inline size_t av_smem(int ny, int kn) { return (size_t) (kn + 2) * (ny + 2) * kAvPitch * sizeof(double); }

__global__ void __launch_bounds__(kAvRows + kAvLoaders, 1)
k_ds_average_wave(double *__restrict__ Cs, const uint8_t *__restrict__ flags, Level L, Box3 box, int K,
                  int *__restrict__ progress, int polls, int *__restrict__ err) {
    extern __shared__ double ring[];
    const int nj = (int) L.Nx, nk = (int) L.nxy();
    const int x0 = (int) box.x0, x1 = (int) box.x1, y0 = (int) box.y0;
    const int nx = (int) box.nx(), ny = (int) box.ny(), nz = (int) box.nz();
    const int kb = (int) blockIdx.x * K, kn = min(K, nz - kb);  // planes of this block (kn >= 1)
    const int z0 = (int) box.z0 + kb;
    const int rowsr = ny + 2;
    const int comp = (int) blockDim.x - kAvLoaders;
    const int tid = threadIdx.x;
    const int steps = nx + 2 + 2 * (ny - 1) + 4 * (kn - 1);          // of this block
    const int rounds = (steps + kAvG - 1) / kAvG;

    if (tid >= comp) {
        const int lt = tid - comp;
        const int prev = (int) blockIdx.x - 1;
        const int prev_steps = nx + 2 + 2 * (ny - 1) + 4 * (K - 1);
        // the last column of ring row (jr, kr) that round S needs: rows of the plane
        // before the block are read up to one column behind their own step, others up
        // to seven ahead
        auto last = [&](int jr, int kr, int S) {
            return x0 - 2 + kAvG * S + kAvG - 1 - 2 * (jr - 1) - 4 * (kr - 1) + (kr == 0 ? -1 : 7);
        };
        // eight lanes a row, one column each; the values go straight to shared memory, so
        // that a round's loads are all in flight together
        const int lane8 = lt % kAvG;
        auto fill = [&](int S) {
            int jr = lt / kAvG, kr = 1;
            while (true) {
                while (jr >= rowsr) {
                    jr -= rowsr;
                    kr++;
                }
                if (kr > kn + 1) break;
                const int e = last(jr, kr, S);
                const double *src = Cs + (int64_t) nj * (y0 + jr - 1) + (int64_t) nk * (z0 + kr - 1);
                double *dst = ring + (kr * rowsr + jr) * kAvPitch;
                for (int c = S == 0 ? x0 - 1 + lane8 : e - (kAvG - 1) + lane8; c <= min(e, x1 + 1); c += kAvG)
                    if (c >= x0 - 1) {
                        const unsigned d = (unsigned) __cvta_generic_to_shared(dst + ((c - (x0 - 1)) & (kAvRing - 1)));
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src + c) : "memory");
                    }
                jr += kAvLoaders / kAvG;
            }
        };
        // the rows of the plane before the block: past the L1 cache, which another
        // block's stores do not reach
        auto fill_prev = [&](int S) {
            const double *src = Cs + (int64_t) nj * (y0 - 1) + (int64_t) nk * (z0 - 1);
            constexpr int B = 8;  // rows of a lane in flight
            for (int j0 = lt / kAvG; j0 < rowsr; j0 += B * (kAvLoaders / kAvG)) {
                int n = 1;
                if (S == 0) n = (last(j0, 0, 0) - (x0 - 1)) / kAvG + 1;
                for (int t = 0; t < n; t++) {
                    double v[B];
                    int at[B];
#pragma unroll
                    for (int u = 0; u < B; u++) {
                        const int jr = j0 + u * (kAvLoaders / kAvG), e = last(jr, 0, S);
                        const int c = (S == 0 ? x0 - 1 + t * kAvG : e - (kAvG - 1)) + lane8;
                        at[u] = jr < rowsr && c >= x0 - 1 && c <= min(e, x1 + 1) ? c : -1;
                        v[u] = at[u] >= 0 ? __ldcg(src + (int64_t) nj * jr + c) : 0.0;
                    }
#pragma unroll
                    for (int u = 0; u < B; u++)
                        if (at[u] >= 0)
                            ring[(j0 + u * (kAvLoaders / kAvG)) * kAvPitch + ((at[u] - (x0 - 1)) & (kAvRing - 1))] = v[u];
                }
            }
        };
        bool bad = false;  // the first loader thread's wait gave up
        auto wait_prev = [&](int S) {  // the block before has updated the columns of round S
            if (prev < 0) return;
            if (lt == 0) {
                const int need = min(prev_steps, kAvG * (S + 1) + 4 * K - 1);
                bool ok = false;
                for (int n = 0; n < polls && !ok; n++) {
                    int v;
                    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(progress + prev) : "memory");
                    ok = v >= need;
                }
                bad = bad || !ok;
            }
            asm volatile("bar.sync 2, %0;" ::"n"(kAvLoaders) : "memory");
        };
        fill(0);
        wait_prev(0);
        fill_prev(0);
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        bool stop = __syncthreads_or(bad);  // every thread of the block sees the same
        for (int S = 0; S < rounds && !stop; S++) {
            if (lt == 0 && S > 0) {
                // every row's stores of the rounds before are ordered by the block barrier
                __threadfence();
                asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(progress + blockIdx.x), "r"(kAvG * S) : "memory");
            }
            if (S + 1 < rounds) {
                fill(S + 1);
                wait_prev(S + 1);
                fill_prev(S + 1);
                asm volatile("cp.async.wait_all;\n" ::: "memory");
            }
            stop = __syncthreads_or(bad);
        }
        if (lt == 0) {
            __threadfence();
            if (stop) {
                atomicExch(progress + kDsProgress - 1, 1);
                atomicExch(err, 1);
            }
            else asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(progress + blockIdx.x), "r"(1 << 30) : "memory");
        }
        return;
    }

    const bool row = tid < kn * ny;
    const int jr = row ? 1 + tid % ny : 1, kr = row ? 1 + tid / ny : 1;
    const double *rr = ring + (size_t) ((kr - 1) * rowsr + jr - 1) * kAvPitch;  // its first neighbour row
    double *own = ring + (size_t) (kr * rowsr + jr) * kAvPitch;
    const uint8_t *ofl = flags + (int64_t) nj * (y0 + jr - 1) + (int64_t) nk * (z0 + kr - 1);
    double *out = Cs + (int64_t) nj * (y0 + jr - 1) + (int64_t) nk * (z0 + kr - 1);
    double w[3][3][3];  // x, y, z
#pragma unroll
    for (int l = 0; l < 3; l++)
#pragma unroll
        for (int m = 0; m < 3; m++)
#pragma unroll
            for (int n = 0; n < 3; n++) w[l][m][n] = 0;
    int i = x0 - 2 - 2 * (jr - 1) - 4 * (kr - 1);  // this row's cell at step 0
    uint8_t fb[kAvG];                              // flags of the next round's cells
    auto flag_bytes = [&](int i0) {
#pragma unroll
        for (int g = 0; g < kAvG; g++) fb[g] = row && i0 + g >= x0 && i0 + g <= x1 ? __ldg(ofl + i0 + g) : (uint8_t) 0;
    };
    auto flag_mask = [&]() {
        unsigned m = 0;
#pragma unroll
        for (int g = 0; g < kAvG; g++) m |= (fb[g] & kInner) ? 1u << g : 0u;
        return m;
    };
    flag_bytes(i);
    unsigned mask = flag_mask();
    bool stop = __syncthreads_or(false);
    for (int S = 0; S < rounds && !stop; S++) {
        flag_bytes(i + kAvG);
        for (int g = 0; g < kAvG; g++, i++) {
            if (row && i + 1 >= x0 - 1 && i <= x1) {
                const int o = (i + 2 - x0) & (kAvRing - 1);
#pragma unroll
                for (int m = 0; m < 3; m++)
#pragma unroll
                    for (int n = 0; n < 3; n++) {
                        w[0][m][n] = w[1][m][n];
                        w[1][m][n] = w[2][m][n];
                        w[2][m][n] = rr[(n * rowsr + m) * kAvPitch + o];
                    }
                const int oc = (i + 1 - x0) & (kAvRing - 1);
                if (mask >> g & 1) {
                    double sum = 0;
#pragma unroll
                    for (int l = 0; l < 3; l++)
#pragma unroll
                        for (int m = 0; m < 3; m++)
#pragma unroll
                            for (int n = 0; n < 3; n++) sum = sum + w[l][m][n];
                    const double c = div27(sum);
                    w[1][1][1] = c;
                    own[oc] = c;
                    out[i] = c;
                }
            }
            if (g + 1 < kAvG) asm volatile("bar.sync 1, %0;" ::"r"(comp) : "memory");
        }
        mask = flag_mask();
        stop = __syncthreads_or(false);
    }
}

// ev of the averaged coefficient; NaN where the averaging gave up
__global__ void k_ds_ev(double *__restrict__ ev, const double *__restrict__ Cs, const double *__restrict__ sbar,
                        const int *__restrict__ fail, const uint8_t *__restrict__ flags, Level L, Box3 box,
                        double delta_s, double nu) {
    DS_COLUMN(box);
    const bool bad = *fail != 0;
    column_planes(i + (int) L.Nx * j, (int) L.nxy(), (int) box.z0, (int) box.z1, flags,
        [&](int q, int) {
            double e = 2.0 * Cs[q] * delta_s * delta_s * sbar[q];
            if ((e + nu) < 0) e = 0;
            return bad ? nan("") : e;
        },
        [&](int q, int, double v, uint8_t) { ev[q] = v; });
}

// The same hyperplane by hyperplane over the whole grid with a grid barrier
// between them, and ev: for levels whose rows do not fit k_ds_average_wave (more
// than kAvRows rows in y, or more planes than its blocks take).
__global__ void k_ds_average(double *__restrict__ Cs, double *__restrict__ ev, const double *__restrict__ sbar,
                             const uint8_t *__restrict__ flags, Level L, Box3 box, double delta_s, double nu) {
    cg::grid_group grid = cg::this_grid();
    const int nj = (int) L.Nx, nk = (int) L.nxy();
    const int x0 = (int) box.x0, x1 = (int) box.x1, y0 = (int) box.y0, z0 = (int) box.z0;
    const int ny = (int) box.ny(), nz = (int) box.nz();
    const int pairs = ny * nz;
    const int t0 = x0 + 2 * y0 + 4 * z0, t1 = x1 + 2 * (int) box.y1 + 4 * (int) box.z1;
    const int stride = (int) (gridDim.x * blockDim.x);
    const int first = (int) (blockIdx.x * blockDim.x + threadIdx.x);
    for (int t = t0; t <= t1; t++) {
        for (int p = first; p < pairs; p += stride) {
            const int j = y0 + p % ny, k = z0 + p / ny;
            const int i = t - 2 * j - 4 * k;
            if (i < x0 || i > x1) continue;
            const int q = i + nj * j + nk * k;
            if (!(flags[q] & kInner)) continue;
            double sum = 0;
#pragma unroll
            for (int l = 0; l < 3; l++)
#pragma unroll
                for (int m = 0; m < 3; m++)
#pragma unroll
                    for (int n = 0; n < 3; n++) sum = sum + Cs[q - 1 + l + nj * (m - 1) + nk * (n - 1)];
            const double c = sum / 27.0;
            Cs[q] = c;
            double e = 2.0 * c * delta_s * delta_s * sbar[q];
            if ((e + nu) < 0) e = 0;
            ev[q] = e;
        }
        grid.sync();
    }
}

// planes per block of k_ds_average_wave, 0 where it does not fit: as many as the
// rows of a block and its shared memory take (each block adds the lag of its own
// planes and some 20 steps to the wave), then the same number for every block
int ds_average_planes(const Box3 &box, int sms) {
    const int64_t ny = box.ny(), nz = box.nz();
    if (ny > kAvRows) return 0;
    int64_t K = std::min<int64_t>(nz, kAvRows / ny);
    while (K > 0 && av_smem((int) ny, (int) K) > kAvSmemMax) K--;
    if (K == 0) return 0;
    const int64_t blocks = (nz + K - 1) / K;
    if (blocks > sms || blocks >= kDsProgress) return 0;
    return (int) ((nz + blocks - 1) / blocks);
}

}  // namespace
}  // namespace artss

using namespace artss;

extern "C" {

int artss_turb_dynamic_smagorinsky(artss_ctx *ctx, double *ev, const double *u, const double *v, const double *w,
                                   double nu) {
    if (!ctx || !ev || !u || !v || !w) { set_error("null argument"); return ARTSS_ERR_ARG; }
    const Level &L = ctx->lvl[0];
    const int64_t N = L.size();
    const size_t bytes = (size_t) DS_ARRAYS * N * sizeof(double) + kDsProgress * sizeof(int);
    if (!ctx->dsmag || ctx->dsmag_version != ctx->geom_version) {
        if (ctx->capturing) {
            set_error("the dynamic Smagorinsky work fields are set up on an eager call; call it once before capturing");
            return ARTSS_ERR_ARG;
        }
        if (!ctx->dsmag) ARTSS_CK(cudaMalloc(&ctx->dsmag, bytes));
        // zero outside the inner cells, also after the inner set changed
        ARTSS_CK(cudaMemsetAsync(ctx->dsmag, 0, bytes, ctx->stream));
        ctx->dsmag_version = ctx->geom_version;
    }
    double *A = ctx->dsmag;
    const Box3 box = inner_box(L);
    const artss_grid_desc &g = ctx->grid;
    const double dx = g.dx[0], dy = g.dy[0], dz = g.dz[0];
    const double rdx = 1. / dx, rdy = 1. / dy, rdz = 1. / dz;
    const double delta_s = cbrt(dx * dy * dz);
    const dim3 grid = ds_grid(box), block = box_block();
    const uint8_t *flags = ctx->d_flags[0];

    int *progress = (int *) (A + DS_ARRAYS * N);
    ARTSS_LAUNCH_PDL(ctx, FAM_SMAGORINSKY, k_ds_filter, grid, block, 0, u, v, w, A, flags, L, box, N);
    ARTSS_LAUNCH_CK(ctx);
    ARTSS_LAUNCH_PDL(ctx, FAM_SMAGORINSKY, k_ds_strain, grid, block, 0, A, flags, L, box, N, rdx, rdy, rdz);
    ARTSS_LAUNCH_CK(ctx);
    // planes in runs that give every multiprocessor some four blocks
    dim3 gc((unsigned) ((box.nx() + kDsCx - 1) / kDsCx), (unsigned) ((box.ny() + 2 * kDsCy - 1) / (2 * kDsCy)));
    const int64_t runs = std::max<int64_t>(1, (8 * (int64_t) std::max(ctx->sm_count, 1)) / ((int64_t) gc.x * gc.y));
    gc.z = (unsigned) std::min<int64_t>(box.nz(), runs);
    ARTSS_LAUNCH_PDL(ctx, FAM_SMAGORINSKY, k_ds_coefficient, gc, dim3(kDsCx, kDsCy), 0, A, flags, L, box, N, delta_s,
                     progress);
    ARTSS_LAUNCH_CK(ctx);
    double *Cs = A + CS * N;
    const double *sb = A + SBAR * N;
    Level Lc = L;
    Box3 bc = box;
    double ds = delta_s, nuv = nu;
    // the averaging: one cooperative launch, every block resident
    int K = ds_average_planes(box, std::max(ctx->sm_count, 1));
    if (K > 0) {
        const int ny = (int) box.ny(), blocks = (int) ((box.nz() + K - 1) / K);
        const size_t smem = av_smem(ny, K);
        // one limit for every grid: the attribute is the function's, which contexts of other
        // sizes launch from other threads
        ARTSS_CK(cudaFuncSetAttribute(k_ds_average_wave, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kAvSmemMax));
        int polls = ctx->wait_polls, *err_flag = &ctx->d_loop[kDsErrSlot].pad;
        void *wargs[] = {&Cs, (void *) &flags, &Lc, &bc, &K, &progress, &polls, &err_flag};
        cudaError_t err;
        ARTSS_LAUNCH(ctx, FAM_SMAGORINSKY,
                     err = cudaLaunchCooperativeKernel((const void *) k_ds_average_wave, dim3((unsigned) blocks),
                                                       dim3((unsigned) ((K * ny + 31) / 32 * 32 + kAvLoaders)), wargs, smem,
                                                       ctx->stream));
        if (err != cudaSuccess) return cuda_fail(err, "cooperative launch");
        ARTSS_LAUNCH_CK(ctx);
        ARTSS_LAUNCH(ctx, FAM_SMAGORINSKY, k_ds_ev<<<grid, block, 0, ctx->stream>>>(
                                               ev, Cs, sb, progress + kDsProgress - 1, flags, L, box, delta_s, nu));
        ARTSS_LAUNCH_CK(ctx);
        return ARTSS_OK;
    }
    static int blocks_per_sm = -1;
    const int threads = 256;
    if (blocks_per_sm < 0) {
        int nb = 0;
        ARTSS_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_ds_average, threads, 0));
        blocks_per_sm = std::max(1, std::min(nb, 4));
    }
    void *args[] = {&Cs, &ev, (void *) &sb, (void *) &flags, &Lc, &bc, &ds, &nuv};
    cudaError_t err;
    ARTSS_LAUNCH(ctx, FAM_SMAGORINSKY,
                 err = cudaLaunchCooperativeKernel((const void *) k_ds_average,
                                                   dim3((unsigned) (blocks_per_sm * std::max(ctx->sm_count, 1))),
                                                   dim3(threads), args, 0, ctx->stream));
    if (err != cudaSuccess) return cuda_fail(err, "cooperative launch");
    ARTSS_LAUNCH_CK(ctx);
    return ARTSS_OK;
}

}  // extern "C"
