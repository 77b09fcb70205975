// BF16 implicit-GEMM 3-D convolution on the 5th-generation tensor cores
// (tcgen05.mma, FP32 accumulation in tensor memory) for the learned
// initial guess of the pressure solve.  No counterpart in the reference.
//
// Activations are channels-last, [D][H][W][C] bf16, C a multiple of 16.
// Kernel 3x3x3, stride 1, zero padding 1 (cross-correlation):
//     y[z,y,x,co] = bias[co] + sum_{t, ci} w[t][co][ci] * x[z+dz, y+dy, x+dx, ci]
// with tap t = 9 (dz+1) + 3 (dy+1) + (dx+1).
//
// GEMM view of the forward pass: M = 128 output voxels (8 in x, 16 in y), a
// block owns `zb` such planes above one another and `nt` output channels, K = 27
// taps x C_in.  Input planes with their halo (10 x 18 voxels, all C_in channels)
// arrive in shared memory ONCE, `pz` planes to a step, as 16-byte pieces
// [z][channel / 8][y][x][8 channels] by cp.async (zero filled outside the grid, which
// is the padding).  In that no-swizzle layout the 8 rows of a core matrix are 8
// neighbours in x and the 16 groups lie one y row apart, so every tap is the same
// tile at another start address: the tap needs no copy of its own.  The three taps of
// a (dy, dx) pair that differ in dz read the same input plane and write three
// neighbouring output planes, whose accumulators lie side by side in tensor memory:
// one MMA with N = 3 nt does all three, so the A tile, whose reading bounds these
// narrow layers (4 KB per MMA, 32 cycles, more than the arithmetic for N < 128), is
// read 9 instead of 27 times per plane.
//
// The order of the sum is part of the result: FP32 accumulation rounds after each
// MMA, the next layer rounds to BF16, and ten layers and a training step magnify the
// last bit (to 0.8 % of an output after two steps on 21 networks, 9.6 % at worst seen).  An output adds its products tap by
// tap, t = 0 .. 26, and within a tap 16 input channels at a time: planes in the order
// of z, for each its 9 taps, for each all its channels.  So the channels of a plane
// have to be in shared memory together.
//
// The weights stay for all of a block's planes where they fit beside them; else a block
// owns one output plane and the weights of a dz arrive with its input plane.  Several
// blocks share a multiprocessor, so that one block's loads and epilogue run under
// another's MMAs (a ring of stages within a block took the room of a second block and
// was slower).  The accumulators start from zero (tcgen05.st); the epilogue adds the
// bias, clamps and stores.  zb, nt and pz follow from a cost model (conv_plan).
// Measured at 64 x 64 x 128, 16 -> 16 channels: 27 us (272 TFLOP/s), 48 -> 16: 58 us
// (377); 32 x 32 x 64, 96 -> 32: 33 us.  With all taps of 16 channels before the next 16,
// in another order then, 25, 57 and 34 us.
//
// Every wait is bounded and raises an error flag.
#include "internal.cuh"
#include "tc.cuh"

#include <cmath>
#include <cuda_bf16.h>

namespace artss {

namespace {

constexpr int kConvPolls = 1 << 20;
constexpr int kConvThreads = 256;
constexpr size_t kConvSmemMax = 227 * 1024 - 1024;  // dynamic limit minus the kernels' static shared memory
constexpr int64_t kConvSmemSm = 228 * 1024;         // of a multiprocessor
constexpr int kTx = 8, kTy = 16;                    // output voxels of one MMA (M = 128)
constexpr int kHx = kTx + 2, kHy = kTy + 2;         // with halo
constexpr unsigned kRowB = kHx * 16;                // bytes between y rows of a channel group
constexpr unsigned kGroupB = kHy * kRowB;           // bytes between channel groups (8 channels) of a plane

struct ConvShape {
    int D, H, W, cin, cout;
    int tiles_x, tiles_y;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool valid) {
    const int n = valid ? 16 : 0;  // 0: the 16 bytes are zero-filled, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_done() {
    asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
    const uint32_t z = 0;
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
        "%1};\n" ::"r"(taddr),
        "r"(z)
        : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

// the tile at (x0, y0) with its halo, planes z0 - 1 .. z0 - 2 + planes, `groups`
// channel groups from c8 on, to [plane][group][y][x][16 bytes] at dst
__device__ __forceinline__ void load_halo(uint32_t dst, const __nv_bfloat16 *__restrict__ x, const ConvShape &s,
                                          int x0, int y0, int z0, int planes, int c8, int groups, int tid) {
    const int n = planes * groups * kHx * kHy;
    for (int e = tid; e < n; e += kConvThreads) {
        const int g = e % groups, v = e / groups;  // groups of a voxel are neighbours in memory
        const int xx = v % kHx, yy = (v / kHx) % kHy, zz = v / (kHx * kHy);
        const int gx = x0 - 1 + xx, gy = y0 - 1 + yy, gz = z0 - 1 + zz;
        const bool in = gx >= 0 && gx < s.W && gy >= 0 && gy < s.H && gz >= 0 && gz < s.D;
        const __nv_bfloat16 *src = in ? x + (((size_t) gz * s.H + gy) * s.W + gx) * s.cin + (c8 + g) * 8 : x;
        cp_async16(dst + (uint32_t) (zz * groups + g) * kGroupB + (uint32_t) yy * kRowB + (uint32_t) xx * 16, src, in);
    }
}

// KK: C_in / 16 where it is known when compiled (0: any).  One thread issues the MMAs, a
// tap and 16 channels each some 40 cycles of the tensor core: with the channel loop
// unrolled the operands' descriptors are one addition each (64 x 64 x 128, 16 -> 16
// channels: 25 us, 33 with a loop and its products).
template <int KK>
__global__ void __launch_bounds__(kConvThreads)
k_conv3d_fwd(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ wp,
             const float *__restrict__ bias, __nv_bfloat16 *__restrict__ y, ConvShape s, ConvPlan p, int relu,
             int *__restrict__ err) {
    extern __shared__ __align__(128) uint8_t cv_sm[];
    __shared__ __align__(8) uint64_t done;  // the step's MMAs have completed
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = (int) blockIdx.x;
    const int x0 = (tile % s.tiles_x) * kTx, y0 = ((tile / s.tiles_x) % s.tiles_y) * kTy,
              z0 = (tile / (s.tiles_x * s.tiles_y)) * p.zb;
    const int n0 = (int) blockIdx.y * p.nt;
    const int zb = min(p.zb, s.D - z0);  // output planes of this block
    const int nt = p.nt, groups = KK ? 2 * KK : s.cin / 8;
    const int steps = (zb + 2 + p.pz - 1) / p.pz;
    const int wrows = p.resident ? 3 * nt : nt;  // rows of the B operand of a tap's dz
    const unsigned tap_bytes = (unsigned) (groups * wrows * 16), plane_bytes = (unsigned) groups * kGroupB;
    const uint32_t base = tc::smem_addr(cv_sm);

    // input planes z0 - 1 + q, q = pz step ..; and the weights of dz = q - 1 for q < 3 as
    // [dy dx][channel / 8][dz][nt][8], dz descending, so that any run of dz is one operand
    // of neighbouring rows (an output plane has dz = q - 1 of step q's planes or an earlier one's)
    auto load = [&](int step) {
        const uint32_t a = base + p.w_bytes;
        const int q0 = step * p.pz, q1 = min(q0 + p.pz, zb + 2);
        load_halo(a, x, s, x0, y0, z0 + q0, q1 - q0, 0, groups, tid);
        for (int dz = q0; dz < min(q1, 3); dz++) {
            const uint32_t b = p.resident ? base + (uint32_t) ((2 - dz) * nt * 16) : a + p.a_bytes;
            for (int e = tid; e < 9 * groups * nt; e += kConvThreads) {
                const int n = e % nt, kc = (e / nt) % groups, t9 = e / (nt * groups);
                cp_async16(b + (uint32_t) t9 * tap_bytes + (uint32_t) (kc * wrows + n) * 16,
                           wp + (((size_t) (9 * dz + t9) * groups + kc) * s.cout + n0 + n) * 8, true);
            }
        }
    };
    load(0);
    if (tid == 0) {
        tc::mbar_init(&done, 1);
        tc::fence_barrier_init();
    }
    if (warp == 0) {
        tc::tmem_alloc(&tmem_base, (unsigned) p.cols);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_base;
    const uint32_t lanes = (uint32_t) (32 * (warp & 3)) << 16;
    for (int c0 = 16 * (warp >> 2); c0 < zb * nt; c0 += 32) tmem_zero16(tmem + lanes + (uint32_t) c0);
    tmem_store_wait();
    tc::tc_fence_before();

    bool ok = true;
    for (int c = 0; c < steps && ok; c++) {
        if (c > 0) {
            ok = tc::mbar_wait(&done, (unsigned) ((c - 1) & 1), kConvPolls);
            if (ok) load(c);
            // no thread leaves the loop before the others have seen the same
            ok = !__syncthreads_or(!ok);
            if (!ok) break;
        }
        cp_async_done();
        tc::fence_proxy_async();  // this thread's pieces, before the tensor core reads them
        __syncthreads();
        if (tid == 0) {
            tc::tc_fence_after();
            const uint8_t *a = cv_sm + p.w_bytes;
            const uint8_t *b = p.resident ? cv_sm : a + p.a_bytes;
            for (int q = c * p.pz; q < min((c + 1) * p.pz, zb + 2); q++) {
                // input plane q feeds output planes q - 2 (dz = +1), q - 1, q (dz = -1)
                const int lo = max(0, q - 2), hi = min(zb - 1, q), nz = hi - lo + 1;
                const int gz = z0 - 1 + q;
                if (gz < 0 || gz >= s.D) continue;  // padding adds nothing
                const uint32_t idesc = tc::idesc_bf16(128, nz * nt, 0, 0);
                // descriptors count 16 bytes
                const uint64_t a0 = tc::smem_desc(a + (size_t) (q - c * p.pz) * plane_bytes, kGroupB, kRowB);
                const uint64_t b0 = tc::smem_desc(b + (p.resident ? (size_t) (lo - q + 2) * nt * 16 : 0),
                                                  (unsigned) (wrows * 16), 128);
                uint64_t db = b0;
#pragma unroll
                for (int t = 0; t < 9; t++) {
                    const uint64_t da = a0 + ((t / 3) * kRowB + (t % 3) * 16) / 16;
#pragma unroll
                    for (int kk = 0; kk < groups / 2; kk++, db += 2 * (unsigned) wrows)  // a tap's channel groups follow the last one's
                        tc::mma_bf16(tmem + (uint32_t) (lo * nt), da + (uint64_t) (kk * (2 * kGroupB / 16)), db, idesc, 1);
                }
            }
            tc::mma_commit(&done);
        }
    }
    if (ok) ok = tc::mbar_wait(&done, (unsigned) ((steps - 1) & 1), kConvPolls);
    if (__syncthreads_or(!ok)) {
        if (tid == 0 && err) atomicExch(err, 1);
        cp_async_done();
    } else {
        tc::tc_fence_after();
        // lane = voxel of the tile, columns = planes x output channels
        const int row = 32 * (warp & 3) + lane, vx = x0 + row % kTx, vy = y0 + row / kTx;
        const bool in = vx < s.W && vy < s.H;
        for (int z = warp >> 2; z < zb; z += 2) {
            __nv_bfloat16 *yo = y + (((size_t) (z0 + z) * s.H + vy) * s.W + vx) * s.cout + n0;
            for (int c0 = 0; c0 < nt; c0 += 16) {
                float v[16];
                tc::tmem_ld16(tmem + lanes + (uint32_t) (z * nt + c0), v);
                __align__(16) __nv_bfloat16 o[16];
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    float r = v[i] + (bias ? __ldg(bias + n0 + c0 + i) : 0.f);
                    if (relu) r = fmaxf(r, 0.f);
                    o[i] = __float2bfloat16_rn(r);
                }
                if (in) {
                    uint4 *dst = reinterpret_cast<uint4 *>(yo + c0);
                    dst[0] = reinterpret_cast<const uint4 *>(o)[0];
                    dst[1] = reinterpret_cast<const uint4 *>(o)[1];
                }
            }
        }
        tc::tc_fence_before();
    }
    __syncthreads();
    tc::tc_fence_after();
    if (warp == 0) tc::tmem_dealloc(tmem, (unsigned) p.cols);
}

// Weight gradient dW[t][co][ci] += sum_v dY[v][co] x[v + off_t][ci] as a GEMM
// with M = C_out (128 rows, those past C_out ignored), N = (dz, C_in), K = voxels.
// The activation tiles keep the forward's shared-memory layout, which read as
// MN-major operands is 8 voxels (K) x 8 channels (M or N) per core matrix, the
// next 8 voxels one y row on (LBO) and the next 8 channels one channel group on
// (SBO); the channel groups of planes z - 1, z, z + 1 follow one another at the
// same distance, so the three dz taps are one operand of N = 3 ct columns and an
// x tile is loaded once for all its taps (before: one 256-row copy per tap).
// A block accumulates `tg` (dy, dx) pairs for `ct` input channels over `chain` of its
// voxel tiles in tensor memory and adds them to dW with FP32 atomics (dW must be
// zeroed by the caller), then starts the next ones from zero.  FP32 accumulation in
// tensor memory rounds towards zero, so a sum's error grows with the length of the
// chain and not with its root: at 56 x 64 x 128, 48 -> 16 channels, 592 MMAs in a row
// were off by 8.9e-6, 200 are by 2.5e-6.  The chains' sums are added up in shared memory
// where that has room, else every one goes to dW.
struct WgradPlan {
    int ct, tg, groups, cols;  // groups of (dy, dx) pairs
    int chain;                 // voxel tiles summed in tensor memory at a time
    unsigned sums;             // where the chains' sums lie in shared memory [column][C_out], 0: nowhere
    unsigned a_bytes, b_bytes;
    size_t smem;
};

__global__ void __launch_bounds__(kConvThreads)
k_conv3d_wgrad(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ dy, float *__restrict__ dw,
               ConvShape s, WgradPlan p, int *__restrict__ err) {
    extern __shared__ __align__(128) uint8_t cv_sm[];
    __shared__ __align__(8) uint64_t done[2];
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles = s.tiles_x * s.tiles_y * s.D;
    const int t0 = (int) blockIdx.y % p.groups * p.tg, nt = min(p.tg, 9 - t0);  // this block's (dy, dx) pairs
    const int ci0 = (int) blockIdx.y / p.groups * p.ct;
    const int g_in = p.ct / 8, g_out = s.cout / 8;
    const uint32_t base = tc::smem_addr(cv_sm);
    const unsigned stage_bytes = p.a_bytes + p.b_bytes;
    auto load = [&](int it) {
        const int tile = (int) blockIdx.x + it * (int) gridDim.x;
        const int x0 = (tile % s.tiles_x) * kTx, y0 = ((tile / s.tiles_x) % s.tiles_y) * kTy,
                  z = tile / (s.tiles_x * s.tiles_y);
        const uint32_t a = base + (uint32_t) (it & 1) * stage_bytes, b = a + p.a_bytes;
        // dY tile [channel / 8][y][x][8]
        for (int e = tid; e < g_out * kTx * kTy; e += kConvThreads) {
            const int g = e % g_out, v = e / g_out, gx = x0 + v % kTx, gy = y0 + v / kTx;
            const bool in = gx < s.W && gy < s.H;
            cp_async16(a + (uint32_t) g * (kTx * kTy * 16) + (uint32_t) v * 16,
                       in ? dy + (((size_t) z * s.H + gy) * s.W + gx) * s.cout + g * 8 : dy, in);
        }
        load_halo(b, x, s, x0, y0, z, 3, ci0 / 8, g_in, tid);
    };
    const int my_tiles = (tiles - (int) blockIdx.x + (int) gridDim.x - 1) / (int) gridDim.x;  // >= 1
    load(0);
    if (tid == 0) {
        tc::mbar_init(&done[0], 1);
        tc::mbar_init(&done[1], 1);
        tc::fence_barrier_init();
    }
    if (warp == 0) {
        tc::tmem_alloc(&tmem_base, (unsigned) p.cols);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_base;
    const uint32_t idesc = tc::idesc_bf16(128, 3 * p.ct, 1, 1);
    // lane = output channel co, columns = (pair, dz, input channel); a column of a lane
    // is always the same thread's
    auto drain = [&](bool first, bool last) {
        tc::tc_fence_after();
        const int co = 32 * (warp & 3) + lane;
        const uint32_t src = tmem + ((uint32_t) (32 * (warp & 3)) << 16);
        float *sums = (float *) (cv_sm + p.sums);
        const int nc = nt * 3 * p.ct / 16;
        if (32 * (warp & 3) < s.cout)
            for (int q = warp >> 2; q < nc; q += 2) {
                const int c = 16 * q, pair = t0 + c / (3 * p.ct), dz = c / p.ct % 3, ci = ci0 + c % p.ct;
                float v[16];
                tc::tmem_ld16(src + (uint32_t) c, v);
                if (co >= s.cout) continue;
                float *d = dw + ((size_t) (9 * dz + pair) * s.cout + co) * s.cin + ci, *m = sums + c * s.cout + co;
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    if (p.sums && !first) v[i] += m[i * s.cout];
                    if (p.sums && !last) m[i * s.cout] = v[i];
                    else atomicAdd(d + i, v[i]);
                }
            }
        tc::tc_fence_before();
    };
    bool ok = true;
    for (int it = 0; it < my_tiles && ok; it++) {
        cp_async_done();
        tc::fence_proxy_async();
        __syncthreads();
        if (tid == 0) {
            tc::tc_fence_after();
            const uint8_t *a = cv_sm + (size_t) (it & 1) * stage_bytes, *b = a + p.a_bytes;
            for (int t = 0; t < nt; t++) {
                const uint8_t *bt = b + ((t0 + t) / 3) * kRowB + ((t0 + t) % 3) * 16;
#pragma unroll
                for (int kk = 0; kk < kTy / 2; kk++)  // 16 voxels (two y rows) per MMA
                    tc::mma_bf16(tmem + (uint32_t) (t * 3 * p.ct),
                                 tc::smem_desc(a + kk * 2 * kTx * 16, kTx * 16, kTx * kTy * 16),
                                 tc::smem_desc(bt + kk * 2 * kRowB, kRowB, kGroupB), idesc, (it % p.chain | kk) != 0);
            }
            tc::mma_commit(&done[it & 1]);
        }
        const int n = it + 1;
        if (n < my_tiles) {
            if (n >= 2) ok = tc::mbar_wait(&done[n & 1], (unsigned) (((n - 2) >> 1) & 1), kConvPolls);
            if (ok) load(n);
            ok = !__syncthreads_or(!ok);
        }
        if (ok && (n == my_tiles || n % p.chain == 0)) {
            ok = tc::mbar_wait(&done[it & 1], (unsigned) ((it >> 1) & 1), kConvPolls);
            ok = !__syncthreads_or(!ok);
            if (ok) drain(it < p.chain, n == my_tiles);  // before the next chain's MMAs: the barrier above them
        }
    }
    if (!ok) {
        if (tid == 0 && err) atomicExch(err, 1);
        cp_async_done();
    }
    __syncthreads();
    tc::tc_fence_after();
    if (warp == 0) tc::tmem_dealloc(tmem, (unsigned) p.cols);
}

int tmem_cols(int n) {
    int c = 32;
    while (c < n) c *= 2;
    return c;
}

// the largest divisor of c that is a multiple of 16 and at most `most`
int channel_tile(int c, int most) {
    for (int t = std::min(c, most) / 16 * 16; t > 16; t -= 16)
        if (c % t == 0) return t;
    return 16;
}

int conv_shape(const artss_conv_desc *d, ConvShape *s) {
    if (d->D < 1 || d->H < 1 || d->W < 1 || d->cin < 16 || d->cin % 16 || d->cin > 256 ||
        d->cout < 16 || d->cout % 16 || d->cout > 256) {
        set_error("conv3d: channels must be multiples of 16, at most 256");
        return ARTSS_ERR_ARG;
    }
    if (!(d->W % 128 == 0 || (128 % d->W == 0 && d->W * d->H >= 128 && d->H % (128 / d->W) == 0) ||
          (128 % (d->W * d->H) == 0 && d->D % (128 / (d->W * d->H)) == 0))) {
        set_error("conv3d: 128-voxel tiles must fit: W a multiple of 128, or W dividing 128 with H a multiple of "
                  "128/W, or W*H dividing 128 with D a multiple of 128/(W*H)");
        return ARTSS_ERR_ARG;
    }
    // 128 voxels x C_in and C_out x C_in operands of more than 104 KB together are not taken
    if ((size_t) 2 * d->cin * (128 + d->cout) > 104 * 1024) { set_error("conv3d: stages too large"); return ARTSS_ERR_LIMIT; }
    *s = ConvShape{d->D, d->H, d->W, d->cin, d->cout, (d->W + kTx - 1) / kTx, (d->H + kTy - 1) / kTy};
    return ARTSS_OK;
}

// The forward kernel's plan: the one with the least time by a model of its parts, whose
// weights (microseconds) were fitted to the times of up to 90 plans for each of 15 layers
// from 8 x 8 x 16 to 64 x 64 x 128 voxels, 16 to 96 channels.  Rounds: of blocks that
// run side by side; a step is a wait for loads and two barriers, an MMA its issue and its
// operands.  A plan that leaves a multiprocessor to one block counts 1.3 times, and
// shared memory counts a little, as blocks of other streams run beside these: over the
// 15 layers the choice is 2.5 % (at most 9 %) off the fastest plan on one stream and 5 %
// on three, without these two 1 % and 20 %.
ConvPlan conv_plan(const ConvShape &s, int sms) {
    ConvPlan best{};
    double least = 0;
    const unsigned plane = (unsigned) s.cin / 8 * kGroupB;
    for (int resident = 1; resident >= 0; resident--)
        for (int zb = resident ? 8 : 1; zb >= 1; zb /= 2)
            for (int nt = channel_tile(s.cout, 64); nt >= 16; nt = nt > 16 ? channel_tile(s.cout, nt - 16) : 0)
                for (int pz = resident ? zb + 2 : 1; pz >= 1; pz--) {
                    ConvPlan p{};
                    p.zb = zb;
                    p.nt = nt;
                    p.pz = pz;
                    p.resident = resident;
                    p.tiles_z = (s.D + zb - 1) / zb;
                    p.cols = tmem_cols(zb * nt);
                    const unsigned dz = (unsigned) (9 * s.cin * nt * 2);  // the weights of one dz
                    p.w_bytes = resident ? 3 * dz : 0;
                    p.a_bytes = (unsigned) pz * plane;
                    p.smem = (size_t) p.w_bytes + p.a_bytes + (resident ? 0 : dz);
                    if (p.cols > 256 || p.smem > kConvSmemMax) continue;
                    const int64_t blocks = (int64_t) s.tiles_x * s.tiles_y * p.tiles_z * (s.cout / nt);
                    const int64_t share = std::min<int64_t>(kConvSmemSm / (int64_t) (p.smem + 1024), 512 / p.cols);
                    const double waves = (double) ((blocks + sms - 1) / sms);
                    const double rounds = std::max(1., (double) blocks / (double) (sms * share));
                    const double mmas = (zb + 2) * 9. * (s.cin / 16), rows = (resident ? 3. : 1.) * nt;
                    const double steps = (zb + 2 + pz - 1) / pz, bytes = (zb + 2) * (double) plane + 3. * dz;
                    const double us = rounds * (1.9 * steps + 0.026 * mmas) + waves * (1.2e-4 * mmas * rows + 4.7e-5 * bytes);
                    const double cost = us * (share > 1 ? 1. : 1.3) * std::pow((double) p.smem, 0.12);
                    if (least == 0 || cost < least) {
                        least = cost;
                        best = p;
                    }
                }
    return best;
}

}  // namespace

int conv3d_wgrad(artss_ctx *ctx, const artss_conv_desc *d, const void *x, const void *dy, float *dw) {
    ConvShape s;
    int st = conv_shape(d, &s);
    if (st) return st;
    if (d->cout > 128 || d->cin > 128) { set_error("conv3d wgrad: C_out and C_in at most 128"); return ARTSS_ERR_ARG; }
    if (((uintptr_t) x & 15) || ((uintptr_t) dy & 15)) { set_error("conv3d: arrays must be 16-byte aligned"); return ARTSS_ERR_ARG; }
    WgradPlan p{};
    p.ct = channel_tile(s.cin, 64);            // N = 3 ct <= 192
    p.tg = std::min(9, 512 / (3 * p.ct));      // accumulators of tg pairs fill tensor memory
    if (p.tg < 9) p.tg = p.tg >= 3 ? 3 : 1;    // whole dy rows
    p.groups = (9 + p.tg - 1) / p.tg;
    p.cols = tmem_cols(p.tg * 3 * p.ct);
    p.a_bytes = (unsigned) (s.cout / 8) * kTx * kTy * 16;
    p.b_bytes = 3u * (unsigned) (p.ct / 8) * kGroupB;
    // the A operand's rows past C_out read on behind the dY tile, within the block's shared memory
    p.smem = std::max<size_t>(2 * ((size_t) p.a_bytes + p.b_bytes),
                              (size_t) p.a_bytes + p.b_bytes + 16 * kTx * kTy * 16);
    if (p.smem > kConvSmemMax) { set_error("conv3d wgrad: stages too large"); return ARTSS_ERR_LIMIT; }
    ARTSS_CK(cudaFuncSetAttribute(k_conv3d_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kConvSmemMax));
    const int tiles = s.tiles_x * s.tiles_y * s.D, yb = p.groups * (s.cin / p.ct);
    // one block a multiprocessor (tensor memory), the parts of dW side by side
    const int sms = std::max(ctx->sm_count, 1), gx = std::max(1, std::min(tiles, sms / yb));
    // as many tiles as a block would have if every one had all of dW
    p.chain = (tiles + sms - 1) / sms;
    const size_t sums = (size_t) p.tg * 3 * p.ct * s.cout * sizeof(float);
    if ((tiles + gx - 1) / gx > p.chain && p.smem + sums <= kConvSmemMax) {
        p.sums = (unsigned) p.smem;
        p.smem += sums;
    }
    ARTSS_LAUNCH(ctx, FAM_CONV, k_conv3d_wgrad<<<dim3((unsigned) gx, (unsigned) yb), kConvThreads, p.smem, ctx->stream>>>(
                                    (const __nv_bfloat16 *) x, (const __nv_bfloat16 *) dy, dw, s, p,
                                    &ctx->d_loop[kNnErrSlot].pad));
    ARTSS_LAUNCH_CK(ctx);
    return ARTSS_OK;
}

int conv3d_fwd(artss_ctx *ctx, const artss_conv_desc *d, const void *x, const void *wp, const float *bias, void *y) {
    ConvShape s;
    int st = conv_shape(d, &s);
    if (st) return st;
    if (((uintptr_t) x & 15) || ((uintptr_t) wp & 15) || ((uintptr_t) y & 15)) {
        set_error("conv3d: arrays must be 16-byte aligned"); return ARTSS_ERR_ARG;
    }
    // the search takes some microseconds: a context keeps the plans of its layers
    const std::array<int, 5> key{s.D, s.H, s.W, s.cin, s.cout};
    auto known = ctx->conv_plans.find(key);
    if (known == ctx->conv_plans.end()) {
        if (ctx->conv_plans.size() >= 256) ctx->conv_plans.clear();
        known = ctx->conv_plans.emplace(key, conv_plan(s, std::max(ctx->sm_count, 1))).first;
    }
    const ConvPlan p = known->second;
    const auto kernel = s.cin == 16 ? k_conv3d_fwd<1> : s.cin == 32 ? k_conv3d_fwd<2> : s.cin == 48 ? k_conv3d_fwd<3>
                      : s.cin == 64 ? k_conv3d_fwd<4> : s.cin == 96 ? k_conv3d_fwd<6> : k_conv3d_fwd<0>;
    ARTSS_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kConvSmemMax));
    const dim3 grid((unsigned) (s.tiles_x * s.tiles_y * p.tiles_z), (unsigned) (s.cout / p.nt));
    ARTSS_LAUNCH(ctx, FAM_CONV, kernel<<<grid, kConvThreads, p.smem, ctx->stream>>>(
                                    (const __nv_bfloat16 *) x, (const __nv_bfloat16 *) wp, bias, (__nv_bfloat16 *) y, s,
                                    p, d->relu, &ctx->d_loop[kNnErrSlot].pad));
    ARTSS_LAUNCH_CK(ctx);
    return ARTSS_OK;
}

}  // namespace artss

using namespace artss;

extern "C" int artss_conv3d_fwd(artss_ctx *ctx, const artss_conv_desc *d, const void *x, const void *w_packed,
                                const float *bias, void *y) {
    if (!ctx || !d || !x || !w_packed || !y) { set_error("null argument"); return ARTSS_ERR_ARG; }
    return conv3d_fwd(ctx, d, x, w_packed, bias, y);
}

extern "C" int artss_nn_check(artss_ctx *ctx) {
    if (!ctx) { set_error("null argument"); return ARTSS_ERR_ARG; }
    LoopState ls{};
    int st = read_loop(ctx, kNnErrSlot, &ls);
    if (st) return st;
    if (ls.pad) {
        ARTSS_CK(cudaMemsetAsync(&ctx->d_loop[kNnErrSlot].pad, 0, sizeof(int), ctx->stream));
        ARTSS_CK(cudaStreamSynchronize(ctx->stream));
        set_error("a network kernel gave up waiting for its operands");
        return ARTSS_ERR_CUDA;
    }
    return ARTSS_OK;
}

extern "C" int artss_conv3d_wgrad(artss_ctx *ctx, const artss_conv_desc *d, const void *x, const void *dy, float *dw) {
    if (!ctx || !d || !x || !dy || !dw) { set_error("null argument"); return ARTSS_ERR_ARG; }
    return conv3d_wgrad(ctx, d, x, dy, dw);
}
