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
// taps x C_in.  Per 16 input channels the block's input planes with their halo
// (10 x 18 x (zb + 2) voxels) and the weights are brought into shared memory
// ONCE, as 16-byte pieces [z][channel / 8][y][x][8 channels] by cp.async (zero
// filled outside the grid, which is the padding).  In that no-swizzle layout the
// 8 rows of a core matrix are 8 neighbours in x and the 16 groups lie one y row
// apart, so every tap is the same tile at another start address: the tap needs no
// copy of its own.  The three taps of a (dy, dx) pair that differ in dz read the
// same input plane and write three neighbouring output planes, whose accumulators
// lie side by side in tensor memory: one MMA with N = 3 nt does all three, so the
// A tile, whose reading bounds these narrow layers (4 KB per MMA, 32 cycles, more
// than the arithmetic for N < 128), is read 9 instead of 27 times per plane.
//
// The accumulators start from zero (tcgen05.st); the epilogue adds the bias,
// clamps and stores.  Several blocks share a multiprocessor, so that one block's
// loads and epilogue run under another's MMAs; zb, nt and the number of stages
// follow from a cost model of the two (conv_plan).  Measured at 64 x 64 x 128, 16 ->
// 16 channels: 25 us (293 TFLOP/s), 48 -> 16: 56 us (390); with one TMA copy of the
// tile per tap, 256 rows of 16 bytes at some four cycles each, the ten layers of the
// network took 3008 us, now 260.
//
// Every wait is bounded and raises an error flag.
#include "internal.cuh"
#include "tc.cuh"

#include <cuda_bf16.h>

namespace artss {

namespace {

constexpr int kConvPolls = 1 << 20;
constexpr int kConvThreads = 256;
constexpr size_t kConvSmemMax = 227 * 1024 - 1024;  // dynamic limit minus the kernels' static shared memory
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

struct ConvPlan {
    int zb, nt, stages, tiles_z, cols;
    unsigned a_bytes, b_bytes;
    size_t smem;
};

__global__ void __launch_bounds__(kConvThreads)
k_conv3d_fwd(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ wp,
             const float *__restrict__ bias, __nv_bfloat16 *__restrict__ y, ConvShape s, ConvPlan p, int relu,
             int *__restrict__ err) {
    extern __shared__ __align__(128) uint8_t cv_sm[];
    __shared__ __align__(8) uint64_t done[2];  // the MMAs of the stage's last use have completed
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = (int) blockIdx.x;
    const int x0 = (tile % s.tiles_x) * kTx, y0 = ((tile / s.tiles_x) % s.tiles_y) * kTy,
              z0 = (tile / (s.tiles_x * s.tiles_y)) * p.zb;
    const int n0 = (int) blockIdx.y * p.nt;
    const int zb = min(p.zb, s.D - z0);  // output planes of this block
    const int nt = p.nt, chunks = s.cin / 16;
    const uint32_t base = tc::smem_addr(cv_sm);
    const unsigned stage_bytes = p.a_bytes + p.b_bytes;

    // input planes z0 - 1 .. z0 + zb and the weights of input channels 16 c ..: the
    // weights as [dy dx][channel / 8][dz][nt][8], dz descending, so that any run of
    // dz is one operand of neighbouring rows
    auto load = [&](int c) {
        const uint32_t a = base + (uint32_t) (c % p.stages) * stage_bytes, b = a + p.a_bytes;
        load_halo(a, x, s, x0, y0, z0, zb + 2, 2 * c, 2, tid);
        for (int e = tid; e < 54 * nt; e += kConvThreads) {
            const int n = e % nt, kc = (e / nt) & 1, tap = e / (2 * nt);
            const int dz = tap / 9, t9 = tap % 9;
            cp_async16(b + (uint32_t) ((t9 * 2 + kc) * 3 * nt + (2 - dz) * nt + n) * 16,
                       wp + (((size_t) tap * (s.cin / 8) + 2 * c + kc) * s.cout + n0 + n) * 8, true);
        }
    };
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
    const uint32_t lanes = (uint32_t) (32 * (warp & 3)) << 16;
    for (int c0 = 16 * (warp >> 2); c0 < zb * nt; c0 += 32) tmem_zero16(tmem + lanes + (uint32_t) c0);
    tmem_store_wait();
    tc::tc_fence_before();

    bool ok = true;
    for (int c = 0; c < chunks && ok; c++) {
        cp_async_done();
        tc::fence_proxy_async();  // this thread's pieces, before the tensor core reads them
        __syncthreads();
        if (tid == 0) {
            tc::tc_fence_after();
            const uint8_t *a = cv_sm + (size_t) (c % p.stages) * stage_bytes, *b = a + p.a_bytes;
            for (int q = 0; q < zb + 2; q++) {
                // input plane q feeds output planes q - 2 (dz = +1), q - 1, q (dz = -1)
                const int lo = max(0, q - 2), hi = min(zb - 1, q), nz = hi - lo + 1;
                const int gz = z0 - 1 + q;
                if (gz < 0 || gz >= s.D) continue;  // padding adds nothing
                const uint32_t idesc = tc::idesc_bf16(128, nz * nt, 0, 0);
                const uint8_t *aq = a + (size_t) q * 2 * kGroupB, *bq = b + (size_t) (lo - q + 2) * nt * 16;
#pragma unroll
                for (int t = 0; t < 9; t++)
                    tc::mma_bf16(tmem + (uint32_t) (lo * nt),
                                 tc::smem_desc(aq + (t / 3) * kRowB + (t % 3) * 16, kGroupB, kRowB),
                                 tc::smem_desc(bq + (size_t) t * 6 * nt * 16, (unsigned) (3 * nt * 16), 128), idesc, 1);
            }
            tc::mma_commit(&done[c % p.stages]);
        }
        const int n = c + 1;
        if (n < chunks) {
            // the stage of chunk n was last read by the MMAs of chunk n - stages
            const int u = n - p.stages;
            if (u >= 0) ok = tc::mbar_wait(&done[u % p.stages], (unsigned) ((u / p.stages) & 1), kConvPolls);
            if (ok) load(n);
            // no thread leaves the loop before the others have seen the same
            ok = !__syncthreads_or(!ok);
        }
    }
    if (ok) ok = tc::mbar_wait(&done[(chunks - 1) % p.stages], (unsigned) (((chunks - 1) / p.stages) & 1), kConvPolls);
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
// A block accumulates `tg` (dy, dx) pairs for `ct` input channels over all its
// voxel tiles in tensor memory and adds them to dW once, with FP32 atomics (dW
// must be zeroed by the caller).
struct WgradPlan {
    int ct, tg, groups, tiles_z, cols;  // groups of (dy, dx) pairs
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
                                 tc::smem_desc(bt + kk * 2 * kRowB, kRowB, kGroupB), idesc, (it | kk) != 0);
            }
            tc::mma_commit(&done[it & 1]);
        }
        const int n = it + 1;
        if (n < my_tiles) {
            if (n >= 2) ok = tc::mbar_wait(&done[n & 1], (unsigned) (((n - 2) >> 1) & 1), kConvPolls);
            if (ok) load(n);
            ok = !__syncthreads_or(!ok);
        }
    }
    if (ok) ok = tc::mbar_wait(&done[(my_tiles - 1) & 1], (unsigned) (((my_tiles - 1) >> 1) & 1), kConvPolls);
    if (__syncthreads_or(!ok)) {
        if (tid == 0 && err) atomicExch(err, 1);
        cp_async_done();
    } else {
        tc::tc_fence_after();
        // lane = output channel co, columns = (pair, dz, input channel)
        const int co = 32 * (warp & 3) + lane;
        const uint32_t src = tmem + ((uint32_t) (32 * (warp & 3)) << 16);
        const int nc = nt * 3 * p.ct / 16;
        if (32 * (warp & 3) < s.cout)
            for (int q = warp >> 2; q < nc; q += 2) {
                const int c = 16 * q, pair = t0 + c / (3 * p.ct), dz = c / p.ct % 3, ci = ci0 + c % p.ct;
                float v[16];
                tc::tmem_ld16(src + (uint32_t) c, v);
                if (co < s.cout) {
                    float *d = dw + ((size_t) (9 * dz + pair) * s.cout + co) * s.cin + ci;
#pragma unroll
                    for (int i = 0; i < 16; i++) atomicAdd(d + i, v[i]);
                }
            }
        tc::tc_fence_before();
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

// zb and nt of the forward kernel: the pair with the least
//     waves x (shared-memory cycles of its MMAs + cycles of its loads)
// where one MMA reads 4 KB of A and 96 nt bytes of B at 128 bytes a cycle and
// loads arrive at some 48 bytes a cycle and multiprocessor.  At 64 x 64 x 128
// this takes 8 planes for the 16-channel layers (512 blocks, 3 a multiprocessor)
// and 1 plane with 32 of the 64 channels on 16 x 16 x 32 (128 blocks: 64 with all
// channels would leave half of the chip idle).
ConvPlan conv_plan(const ConvShape &s, int sms) {
    ConvPlan best{};
    double least = 0;
    for (int zb = 8; zb >= 1; zb /= 2)
        for (int nt = channel_tile(s.cout, 64); nt >= 16; nt = nt > 16 ? channel_tile(s.cout, nt - 16) : 0) {
            ConvPlan p{};
            p.zb = zb;
            p.nt = nt;
            p.tiles_z = (s.D + zb - 1) / zb;
            p.cols = tmem_cols(zb * nt);
            p.a_bytes = (unsigned) (zb + 2) * 2 * kGroupB;
            p.b_bytes = (unsigned) (54 * nt * 16);
            const size_t stage = p.a_bytes + p.b_bytes;
            if (p.cols > 256 || stage > kConvSmemMax / 2) continue;  // two blocks a multiprocessor
            p.stages = s.cin > 16 && 2 * stage <= kConvSmemMax / 2 ? 2 : 1;
            p.smem = p.stages * stage;
            const int64_t blocks = (int64_t) s.tiles_x * s.tiles_y * p.tiles_z * (s.cout / nt);
            const double cost = (double) ((blocks + sms - 1) / sms) *
                                ((zb + 2) * 9. * (32. + 0.75 * nt) + (double) stage / 48.);
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
    const int gx = std::max(1, std::min(tiles, std::max(ctx->sm_count, 1) / yb));
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
    const ConvPlan p = conv_plan(s, std::max(ctx->sm_count, 1));
    ARTSS_CK(cudaFuncSetAttribute(k_conv3d_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kConvSmemMax));
    const dim3 grid((unsigned) (s.tiles_x * s.tiles_y * p.tiles_z), (unsigned) (s.cout / p.nt));
    ARTSS_LAUNCH(ctx, FAM_CONV, k_conv3d_fwd<<<grid, kConvThreads, p.smem, ctx->stream>>>(
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
