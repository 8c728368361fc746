// Learned coarse-slice closure: a complex-valued convolutional network that
// corrects an exit wave computed with 4x thicker slices toward the fine-slice
// result.  It has no counterpart in the reference; the reference's fine-slice
// loop (mulslice.cpp:706-739) is its fallback and the judge of its error.
//
// Network (complex channels, 3x3 taps, periodic boundaries as the wave itself):
//   x = psi / s                 (s = norm of psi / 256: its RMS on a 256^2 grid)
//   h1 = CReLU(conv(x; 1 -> C))
//   h2..h5 = CReLU(conv(h; C -> C))
//   d = conv(h5; C -> 1)
//   psi_out = psi + s d
// with CReLU applying max(0, .) to real and imaginary parts separately and
// C = 32.  A complex layer is held as a real layer over 2C channels (real parts
// then imaginary parts) whose weight blocks are [[Wr, -Wi], [Wi, Wr]].
//
// Kernels:
//   * conv_tc_kernel: the C -> C layers (K = 9 taps x 64 real channels,
//     N = 64) as an implicit GEMM on the tensor cores (tcgen05, FP32
//     accumulators in tensor memory, TMA in and out), bias + CReLU (or the
//     backward pass's ReLU mask) in the epilogue, bf16 activations out.  The same
//     kernel computes the input gradient of these layers with the flipped,
//     transposed weights.
//   * first_layer_kernel, last_layer_kernel, last_layer_dx_kernel: the 1 -> C and
//     C -> 1 layers and the latter's input gradient on the CUDA cores (FP32).
//   * dw_tc_kernel, dw_edge_kernel: weight gradients of the C -> C layers on the
//     tensor cores and of the edge layers on the CUDA cores, FP32 partial sums per
//     CTA reduced in a fixed order (deterministic).
// Weights are kept as FP32 master copies (Adam) and used as bf16.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <string>
#include <vector>

#include "../../include/msl.h"
#include "msl_internal.h"
#include "msl_tc.cuh"

namespace msl {
namespace closure {

constexpr int kC = 32;          // complex channels of the hidden layers
constexpr int kR = 2 * kC;      // real channels
constexpr int kLayers = 6;
constexpr int kTile = 128;      // output pixels per tensor-core tile
constexpr uint32_t kWait = 1u << 22;

// Parameter layout (FP32), per layer l with complex in/out counts (ci, co):
//   weights [9][co][ci][2] (re, im), then bias [co][2].
__host__ __device__ inline int layer_ci(int l) { return l == 0 ? 1 : kC; }
__host__ __device__ inline int layer_co(int l) { return l == kLayers - 1 ? 1 : kC; }
inline int layer_wsize(int l) { return 9 * layer_co(l) * layer_ci(l) * 2; }
inline int layer_size(int l) { return layer_wsize(l) + layer_co(l) * 2; }
inline int param_offset(int l) {
    int o = 0;
    for (int i = 0; i < l; ++i) o += layer_size(i);
    return o;
}
inline int param_count() { return param_offset(kLayers); }

// ------------------------------------------------------------------ helpers
// A running sum as three unevaluated floats, two error-free additions (Knuth's two-sum)
// and a plain one for what is left: some 72 bits, more than an FP64 sum keeps, at 13
// FP32 additions a value.  FP64 ones run at a few per clock and SM here.
struct TripleSum {
    float hi = 0.f, mid = 0.f, lo = 0.f;
    __device__ __forceinline__ static float two_sum(float &a, float x) {  // a <- a + x, the error returned
        const float s = __fadd_rn(a, x), b = __fsub_rn(s, a);
        const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, b)), __fsub_rn(x, b));
        a = s;
        return e;
    }
    __device__ __forceinline__ void add(float x) {
        float e = two_sum(hi, x);
        e = two_sum(mid, e);
        lo = __fadd_rn(lo, e);
    }
    __device__ __forceinline__ void add(const float *p, int stride) {  // another such sum
        add(p[0]);
        lo = __fadd_rn(lo, two_sum(mid, p[stride]));
        lo = __fadd_rn(lo, p[2 * stride]);
    }
    // NaN where a sum on the way overflowed (or a value was no number)
    __device__ __forceinline__ double value() const { return ((double)lo + (double)mid) + (double)hi; }
};
__device__ __forceinline__ float bf(const __nv_bfloat16 v) { return __bfloat162float(v); }

// Real weight of the expanded layer: output real channel n, input real channel k.
__device__ __forceinline__ float expand_w(const float *wl, int co, int ci, int tap, int n, int k) {
    const int o = n % co, a = n / co, i = k % ci, b = k / ci;
    const float *w = wl + (((size_t)tap * co + o) * ci + i) * 2;
    if (a == b) return w[0];
    return a == 0 ? -w[1] : w[1];
}

// wt[tap][n][k] (bf16, K-major) = expanded real weights; transposed = the
// input-gradient form: wt[tap'][k][n] with tap' the mirrored tap.
// for the four tensor-core layers at once (blockIdx.y = layer - 1): out holds each
// layer's forward form, then its input-gradient form.
__global__ void expand_kernel(const float *params, int first, int stride, __nv_bfloat16 *out) {
    constexpr int total = 9 * kR * kR;
    const float *wl = params + first + (size_t)blockIdx.y * stride;
    __nv_bfloat16 *wt = out + (size_t)blockIdx.y * 2 * total;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < 2 * total; idx += gridDim.x * blockDim.x) {
        const int at = idx % total, tap = at / (kR * kR), rem = at % (kR * kR);
        // forward [tap][n][k]; transposed [tap'][k][n] with source tap 8 - tap'
        const float v = idx < total ? expand_w(wl, kC, kC, tap, rem / kR, rem % kR)
                                    : expand_w(wl, kC, kC, 8 - tap, rem % kR, rem / kR);
        wt[idx] = __float2bfloat16_rn(v);
    }
}

// --------------------------------------------------------- padded activations
// Hidden activations are bf16 [B][H + 2][W + 2][64] with a one-pixel halo that
// repeats the opposite edge (periodic boundaries), so that a tile shifted by any
// of the 3x3 taps is one TMA box.  Whoever writes an edge pixel also writes its
// halo copies.
struct Pad {
    int H, W;
    __host__ __device__ size_t pixels(int B) const { return (size_t)B * (H + 2) * (W + 2); }
    // pixel (y, x) of image b, -1 <= y <= H, -1 <= x <= W
    __device__ __forceinline__ size_t at(int b, int y, int x) const {
        return ((size_t)b * (H + 2) + y + 1) * (W + 2) + x + 1;
    }
    // f(y, x) for every place pixel (y, x) is kept at (H, W >= 3)
    template <class F> __device__ __forceinline__ void each_copy(int y, int x, const F &f) const {
        const int ya = y == 0 ? H : y == H - 1 ? -1 : y, xa = x == 0 ? W : x == W - 1 ? -1 : x;
        f(y, x);
        if (ya != y) f(ya, x);
        if (xa != x) {
            f(y, xa);
            if (ya != y) f(ya, xa);
        }
    }
};

// --------------------------------------------------- tensor-core C -> C layer
// Implicit GEMM of a 64 -> 64 real-channel 3x3 layer, input stationary and warp
// specialised, one persistent CTA per SM.  A unit of work is a strip of 128
// columns by some rows of one image.  Warp 0 streams the strip's input rows, each
// as three 128-pixel tiles (shifts -1, 0, +1; 16 KB, 128-byte swizzle) by TMA
// through a ring of kRing slots; warp 1 multiplies every tile by the three row taps
// that use it -- one tcgen05.mma of N = 192 per 16 channels, the three taps'
// outputs being three neighbouring 64-column accumulators of tensor memory -- and
// two groups of four warps drain finished accumulators in turn (bias + CReLU, or the
// backward pass's ReLU mask) to bf16 through swizzled staging tiles and TMA stores.  Output row y keeps
// its accumulator while input rows y - 1, y, y + 1 pass, in tap order, so its FP32
// sum order is tap 0..8, channels ascending.  Eight accumulators rotate, so the
// epilogue may lag five rows; it leaves them zeroed, so that no row's first product
// needs an MMA of its own (an MMA costs some 90 cycles before its columns count: 64
// columns 100, 192 columns 122).
// An input tile is read from L2 three times (the shifts), not nine, and nothing but
// TMA moves operands: what bounds it is the activations' traffic (2 x 128 bytes a
// pixel) beside the MMAs (12 x 122 cycles per 128 pixels, measured).
// 16 waves of 512^2 (537 MB in, 537 MB out): 1.33 ms a layer with each tap tile copied by the threads
// that issued its MMAs, now 0.24 ms.
enum Epi { EPI_BIAS_RELU = 0, EPI_MASK = 1 };

constexpr size_t kWTile = 64 * 128;          // one tap's B tile: 64 rows x 128 bytes
constexpr size_t kATile = kTile * 128;       // 128 pixels x 128 bytes
constexpr int kRing = 7, kStage = 2, kAcc = 8;
constexpr int kDwThreads = 320;                    // TMA warp, MMA warp, eight that read the sums out
constexpr int kConvThreads = 64 + 128 * kStage;    // TMA warp, MMA warp, a four-warp epilogue group per staging tile
constexpr size_t kConvSmem = 1024 + 9 * kWTile + (kRing + kStage) * kATile;

// Strips of 128 columns cut into segments of `seg` rows.
struct Units {
    int B, H, W, seg;
    __host__ __device__ int segs() const { return (H + seg - 1) / seg; }
    __host__ __device__ int count() const { return B * (W / kTile) * segs(); }
    __device__ __forceinline__ void get(int u, int *b, int *x0, int *y0, int *y1) const {
        const int sg = u % segs(), rest = u / segs();
        *x0 = (rest % (W / kTile)) * kTile;
        *b = rest / (W / kTile);
        *y0 = sg * seg;
        *y1 = *y0 + seg < H ? *y0 + seg : H;
    }
};

// The segment length that needs the fewest row steps of the busiest of `ncta` CTAs,
// a unit of n rows costing n + extra (its halo rows).
inline Units plan_units(int B, int H, int W, int ncta, int extra) {
    Units best = {B, H, W, H};
    long best_cost = -1;
    for (int n = 1; n <= H; ++n) {
        Units u = {B, H, W, (H + n - 1) / n};
        const long waves = (u.count() + ncta - 1) / ncta, cost = waves * (u.seg + extra);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = u;
        }
    }
    return best;
}

// Bounded wait that also gives up when another role of the CTA has.
__device__ __forceinline__ bool wait_or_quit(uint64_t *bar, uint32_t parity, volatile int *failed) {
    for (uint32_t i = 0; i < kWait; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 63u) == 63u && *failed) return false;
    }
    *failed = 1;
    return false;
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// An output tile's 128 pixels of row y leave a swizzled staging tile by TMA, the first
// and last row also to their halo rows (one thread) ...
__device__ __forceinline__ void store_tile(const CUtensorMap *map, const void *st, int b, int y, int x0, int H) {
    const int row = b * (H + 2) + y + 1;
    tma_store_3d(map, 0, x0 + 1, row, st);
    if (y == 0) tma_store_3d(map, 0, x0 + 1, row + H, st);           // halo row H
    else if (y == H - 1) tma_store_3d(map, 0, x0 + 1, row - H, st);  // halo row -1
    tma_commit();
}
// ... and an edge pixel's 64 channels to the halo columns, from the thread that holds them.
__device__ __forceinline__ void store_halo_column(const Pad &pd, __nv_bfloat16 *out, int b, int y, int x,
                                                  const __nv_bfloat16 *px) {
    if (x != 0 && x != pd.W - 1) return;
    const int xa = x == 0 ? pd.W : -1;
    pd.each_copy(y, 1, [&](int yy, int) {
        uint4 *h = (uint4 *)(out + pd.at(b, yy, xa) * 64);
#pragma unroll
        for (int c = 0; c < 8; ++c) h[c] = *(const uint4 *)(px + c * 8);
    });
}

__global__ void __launch_bounds__(kConvThreads, 1)
    conv_tc_kernel(const __grid_constant__ CUtensorMap min, const __grid_constant__ CUtensorMap mout,
                   const __nv_bfloat16 *__restrict__ wt, const float *__restrict__ bias,
                   const __nv_bfloat16 *__restrict__ mask, __nv_bfloat16 *__restrict__ out, Units units, int epi,
                   int *err) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *base = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *sw = base;                              // 9 x 8 KB, [kx][ky]
    unsigned char *sa = base + 9 * kWTile;                 // kRing x 16 KB
    unsigned char *so = sa + kRing * kATile;               // kStage x 16 KB
    __shared__ uint64_t full[kRing], empty[kRing], acc_full[kAcc], acc_empty[kAcc], drained;
    __shared__ uint32_t tmem_base;
    __shared__ volatile int failed;
    __shared__ float sbias[64];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform
    // real channel n: the complex bias [o][2] holds (re, im) of channel n % 32
    if (epi == EPI_BIAS_RELU && tid < 64) sbias[tid] = bias[(tid & (kC - 1)) * 2 + (tid >> 5)];
    // all nine B tiles, resident for the whole kernel, the three row taps of a column tap together
    for (int i = tid; i < 9 * 64 * 8; i += kConvThreads) {
        const int tap = i / 512, r = (i / 8) % 64, c = i % 8, slot = (tap % 3) * 3 + tap / 3;
        const uint4 v = *(const uint4 *)(wt + ((size_t)tap * 64 + r) * 64 + c * 8);
        *(uint4 *)(sw + slot * kWTile + tc::sw128_offset(r, c * 8)) = v;
    }
    if (warp == 1) tc::tmem_alloc(&tmem_base, 512);
    if (tid == 0) {
        for (int i = 0; i < kRing; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < kAcc; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 4);
        }
        mbar_init(&drained, 1);
        mbar_fence_init();
        failed = 0;
    }
    fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    if (warp >= 2 && warp < 6) {  // four warps, one per lane quarter
#pragma unroll
        for (int i = 0; i < kAcc; ++i) tc::tmem_zero64(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 64u * i);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const int H = units.H, W = units.W, nunits = units.count();
    const Pad pd = {H, W};
    if (warp == 0) {
        if (lane == 0) {
            uint32_t n = 0;  // tiles requested
            bool ok = true;
            for (int u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
                int b, x0, y0, y1;
                units.get(u, &b, &x0, &y0, &y1);
                for (int r = y0 - 1; r <= y1 && ok; ++r)
                    for (int kx = 0; kx < 3; ++kx, ++n) {
                        const uint32_t s = n % kRing;
                        if (n >= kRing && !(ok = wait_or_quit(&empty[s], (n / kRing - 1) & 1, &failed))) break;
                        mbar_arrive_expect_tx(&full[s], (uint32_t)kATile);
                        tma_load_3d(sa + s * kATile, &min, 0, x0 + kx, b * (H + 2) + r + 1, &full[s]);
                    }
            }
            // loads still in flight land in this CTA's shared memory: let them finish
            for (uint32_t j = n > kRing ? n - kRing : 0; j < n; ++j)
                mbar_wait_bounded(&full[j % kRing], (j / kRing) & 1, kWait);
        }
        __syncwarp();
    } else if (warp == 1) {
        // the whole warp walks the loop (its control flow is uniform), one elected lane issues
        const uint32_t swa = smem_u32(sw), saa = smem_u32(sa);
        uint32_t n = 0, ob = 0;  // tiles consumed, output rows before this unit
        bool ok = true;
        for (int u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
            int b, x0, y0, y1;
            units.get(u, &b, &x0, &y0, &y1);
            const int rows = y1 - y0;
            for (int i = 0; i < rows + 2 && ok; ++i) {
                // input row y0 - 1 + i meets row tap ky for output row j = i - ky of the unit
                const int klo = i < rows ? 0 : i - rows + 1, khi = i < 2 ? i : 2;
                if (i < rows) {  // a new accumulator: drained from its last use?
                    const uint32_t o = ob + i;
                    if (o >= kAcc && !(ok = wait_or_quit(&acc_empty[o % kAcc], (o / kAcc - 1) & 1, &failed))) break;
                }
                // accumulator of output row j at column 64 (7 - j mod 8): the row taps' accumulators
                // ascend with the tap, up to the wrap, so taps klo..khi are one or two runs
                const uint32_t slot = 7u - ((ob + (uint32_t)(i - klo)) & 7u);
                const int taps = khi - klo + 1, n0 = taps < 8 - (int)slot ? taps : 8 - (int)slot;
                const uint32_t col0 = tmem + 64u * slot;
                for (int kx = 0; kx < 3; ++kx, ++n) {
                    const uint32_t s = n % kRing;
                    if (!(ok = wait_or_quit(&full[s], (n / kRing) & 1, &failed))) break;
                    tc::fence_after_sync();
                    if (tc::elect_one()) {
                        const uint64_t ad = tc::desc_sw128(saa + s * (uint32_t)kATile);
                        const uint64_t bd = tc::desc_sw128(swa + (kx * 3 + klo) * (uint32_t)kWTile);
                        if (n0 == 3) {  // by far the most: straight, every operand a constant step on
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)  // 16 channels: 32 bytes
                                tc::mma_bf16(col0, ad + 2 * kk, bd + 2 * kk, tc::idesc_bf16(kTile, 192), 1u);
                        } else {
                            const uint64_t wrap = bd + n0 * (kWTile >> 4);  // the weights past the wrap
                            const uint32_t id0 = tc::idesc_bf16(kTile, 64 * n0), id1 = tc::idesc_bf16(kTile, 64 * (taps - n0));
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk) {
                                tc::mma_bf16(col0, ad + 2 * kk, bd + 2 * kk, id0, 1u);
                                if (n0 < taps) tc::mma_bf16(tmem, ad + 2 * kk, wrap + 2 * kk, id1, 1u);
                            }
                        }
                        tc::mma_commit(&empty[s]);
                        if (kx == 2 && i >= 2) tc::mma_commit(&acc_full[(ob + i - 2) % kAcc]);
                    }
                    __syncwarp();
                }
            }
            ob += rows;
        }
        if (tc::elect_one()) tc::mma_commit(&drained);  // every MMA has completed before the CTA's memory goes
        mbar_wait_bounded(&drained, 0, kWait);
        __syncwarp();
    } else {
        // epilogue group g takes every kStage-th output row, through its own staging tile
        const int g = (tid - 64) / 128, et = (tid - 64) % 128;
        const int r = 32 * (warp & 3) + lane;  // this thread's pixel of the tile (TMEM lane)
        const uint32_t lane_base = (uint32_t)(32 * (warp & 3)) << 16, bar = 1u + (uint32_t)g;
        unsigned char *st = so + g * kATile;
        uint32_t ob = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
            int b, x0, y0, y1;
            units.get(u, &b, &x0, &y0, &y1);
            // output row y0 + j is the CTA's output ob + j
            for (int y = y0 + (int)((g + kStage - ob % kStage) % kStage); y < y1; y += kStage) {
                const uint32_t o = ob + (uint32_t)(y - y0), a = o % kAcc;
                const int x = x0 + r;
                const size_t pix = pd.at(b, y, x);
                __align__(16) __nv_bfloat16 ob16[64];
                if (epi == EPI_MASK) {
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        *(uint4 *)(ob16 + c * 8) = __ldg((const uint4 *)(mask + pix * 64 + c * 8));
                }
                const bool got = wait_or_quit(&acc_full[a], (o / kAcc) & 1, &failed);
                if (et == 0) tma_wait_read<0>();  // the group's last store has read its staging tile
                if (bar_group_or(bar, 128, !got)) {
                    ok = false;
                    break;
                }
                tc::fence_after_sync();
                float v[64];
                tc::tmem_ld64(tmem + lane_base + 64u * (7u - a), v);
                tc::tmem_zero64(tmem + lane_base + 64u * (7u - a));  // its next row adds from the first product on
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[a]);
#pragma unroll
                for (int n = 0; n < 64; ++n) {
                    if (epi == EPI_BIAS_RELU)
                        ob16[n] = __float2bfloat16_rn(fmaxf(v[n] + sbias[n], 0.0f));
                    else
                        ob16[n] = __float2bfloat16_rn(bf(ob16[n]) > 0.0f ? v[n] : 0.0f);
                }
#pragma unroll
                for (int c = 0; c < 8; ++c) *(uint4 *)(st + tc::sw128_offset(r, c * 8)) = *(const uint4 *)(ob16 + c * 8);
                store_halo_column(pd, out, b, y, x, ob16);
                fence_proxy_async();
                bar_group(bar, 128);
                if (et == 0) store_tile(&mout, st, b, y, x0, H);
            }
            ob += (uint32_t)(y1 - y0);
        }
        if (et == 0) tma_wait_all();
    }
    tc::fence_before_sync();
    __syncthreads();
    if (failed && tid == 0 && err) atomicExch(err, 1);
    if (warp == 1) tc::tmem_free(tmem, 512);
}

// ----------------------------------------------------- CUDA-core small layers
// A lane per complex channel of the wide side (first layer, input gradient of the
// last) or a thread per pixel (last layer); sums over the taps in tap order, each
// complex product as two FP32 products, the second fused into the first's negative
// or positive.
constexpr int kEdgeWarps = 8;

// Periodic index one step outside [0, n) at most.
__device__ __forceinline__ int wrap(int i, int n) { return i < 0 ? i + n : i >= n ? i - n : i; }

// a + w x, scalar operations: the packed FP32 pairs run on one of the SM's two FMA pipes
// only, at half the rate of scalar ones on both.
__device__ __forceinline__ float2 c_mac(float2 a, float2 w, float2 x) {
    return make_float2(__fadd_rn(a.x, fmaf(w.x, x.x, -__fmul_rn(w.y, x.y))),
                       __fadd_rn(a.y, fmaf(w.y, x.x, __fmul_rn(w.x, x.y))));
}

// First layer: x (complex64 [B][H][W], scaled by 1/s[b]) -> h1 = CReLU(conv + b)
// (padded bf16); the scaled input is also written as bf16 [B][H][W][2] for the
// weight gradient when xin is given.  A warp takes runs of 32 pixels of a row: the
// 3 x 34 inputs are scaled, rounded to bf16 (as the tensor-core layers see theirs)
// and kept in shared memory, and each lane holds its channel's weights in registers,
// so a pixel is 54 operations a lane and its stores are two whole 64-byte halves.
// (On the tensor cores the sums round differently, and a flipped bf16 rounding here
// grows to 5e-4 of the output over the layers.)  16 waves of 512^2: 0.39 ms (2.2 ms
// with a thread per pixel, whose 64 two-byte stores each touched a line of their own).
__global__ void __launch_bounds__(32 * kEdgeWarps, 3)
    first_layer_kernel(const float2 *__restrict__ psi, const float *__restrict__ inv_s, const float *__restrict__ wl,
                       __nv_bfloat162 *__restrict__ xin, __nv_bfloat16 *__restrict__ h, int B, int H, int W) {
    __shared__ float2 win[kEdgeWarps][3][34];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Pad pd = {H, W};
    float2 w[9];
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        w[t] = make_float2(bf(__float2bfloat16_rn(wl[(t * kC + lane) * 2])),
                           bf(__float2bfloat16_rn(wl[(t * kC + lane) * 2 + 1])));
    }
    const float2 bias = make_float2(wl[9 * kC * 2 + lane * 2], wl[9 * kC * 2 + lane * 2 + 1]);
    const unsigned rr = (unsigned)W / 32u, runs = (unsigned)B * H * rr;
    for (unsigned u = blockIdx.x * kEdgeWarps + warp; u < runs; u += gridDim.x * kEdgeWarps) {
        const unsigned line = u / rr;
        const int x0 = (int)(u - line * rr) * 32, b = (int)(line / H), y = (int)line - b * H;
        const float sc = inv_s[b];
        __syncwarp();
        for (int i = lane; i < 3 * 34; i += 32) {
            const int yy = wrap(y + i / 34 - 1, H), xx = wrap(x0 + i % 34 - 1, W);
            const float2 v = psi[((size_t)b * H + yy) * W + xx];
            win[warp][i / 34][i % 34] =
                make_float2(bf(__float2bfloat16_rn(v.x * sc)), bf(__float2bfloat16_rn(v.y * sc)));
        }
        __syncwarp();
        if (xin) {
            const float2 c = win[warp][1][1 + lane];
            xin[((size_t)b * H + y) * W + x0 + lane] = __floats2bfloat162_rn(c.x, c.y);
        }
        const bool edge = y == 0 || y == H - 1 || x0 == 0 || x0 == W - 32;  // the run touches a halo
        __nv_bfloat16 *o = h + pd.at(b, y, x0) * 64 + lane;
        for (int x = 0; x < 32; x += 4) {
            float2 v[3][6];
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int j = 0; j < 6; ++j) v[r][j] = win[warp][r][x + j];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float2 a = bias;
#pragma unroll
                for (int t = 0; t < 9; ++t) a = c_mac(a, w[t], v[t / 3][j + t % 3]);
                const __nv_bfloat162 v2 =
                    __hmax2(__floats2bfloat162_rn(a.x, a.y), __floats2bfloat162_rn(0.0f, 0.0f));
                if (edge) {
                    pd.each_copy(y, x0 + x + j, [&](int yy, int xx) {
                        __nv_bfloat16 *q = h + pd.at(b, yy, xx) * 64 + lane;
                        q[0] = v2.x;
                        q[kC] = v2.y;
                    });
                } else {
                    o[(x + j) * 64] = v2.x;
                    o[(x + j) * 64 + kC] = v2.y;
                }
            }
        }
    }
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// Last layer: d = conv(h5; C -> 1) + b; psi_out = psi + s d (FP32).  With a
// target, writes the loss terms and g = dL/dd (FP32 [B][H][W][2]).  A CTA walks a
// strip of 128 columns, a thread per pixel, the strip's input rows (130 pixels, 16-byte
// chunks xored by the pixel so that the threads' own-pixel reads are conflict-free)
// in a ring of four fed one row ahead by cp.async.  The 576-term sums run in order
// in each thread: bound by their FP32 and unpacking instructions.
// 16 waves of 512^2: 0.40 ms (8.0 ms with every channel read from global memory by
// two-byte loads).
constexpr int kLastRow = (kTile + 2) * 128;
constexpr size_t kLastSmem = 4 * kLastRow + (9 * kC + 1) * sizeof(float2) + kTile * sizeof(double);
__global__ void __launch_bounds__(kTile)
    last_layer_kernel(const __nv_bfloat16 *__restrict__ h, const float *__restrict__ wl,
                      const float2 *__restrict__ psi, const float *__restrict__ s_img,
                      const float2 *__restrict__ target, float2 *__restrict__ out, float2 *__restrict__ g,
                      double *__restrict__ loss_part, float gscale, Units units) {
    extern __shared__ __align__(16) unsigned char ring[];
    float2 *w = reinterpret_cast<float2 *>(ring + 4 * kLastRow);
    double *red = reinterpret_cast<double *>(w + 9 * kC + 1);
    const int t = threadIdx.x, H = units.H, W = units.W, nunits = units.count();
    const Pad pd = {H, W};
    for (int i = t; i < 9 * kC + 1; i += kTile)
        w[i] = i < 9 * kC ? make_float2(bf(__float2bfloat16_rn(wl[2 * i])), bf(__float2bfloat16_rn(wl[2 * i + 1])))
                          : make_float2(wl[2 * i], wl[2 * i + 1]);
    double acc = 0.0;
    for (int u = blockIdx.x; u < nunits; u += gridDim.x) {
        int b, x0, y0, y1;
        units.get(u, &b, &x0, &y0, &y1);
        auto fetch = [&](int y) {  // input row y into its slot
            const unsigned char *src = (const unsigned char *)(h + pd.at(b, y, x0 - 1) * 64);
            unsigned char *dst = ring + ((y - y0 + 1) & 3) * kLastRow;
            for (int i = t; i < (kTile + 2) * 8; i += kTile) {
                const int px = i >> 3, c = i & 7;
                cp_async16(dst + px * 128 + ((c ^ (px & 7)) << 4), src + (size_t)i * 16);
            }
        };
        __syncthreads();  // the previous unit's rows have been read
        fetch(y0 - 1);
        fetch(y0);
        fetch(y0 + 1);
        const float s = s_img[b];
        for (int y = y0; y < y1; ++y) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();  // rows up to y + 1 are here, row y - 2 has been read
            if (y + 1 < y1) fetch(y + 2);
            const size_t p = ((size_t)b * H + y) * W + x0 + t;
            const float2 c = psi[p], f = target ? target[p] : make_float2(0.f, 0.f);
            float2 d = w[9 * kC];
            for (int tap = 0; tap < 9; ++tap) {
                const int px = t + tap % 3;
                const unsigned char *src = ring + ((y - y0 + tap / 3) & 3) * kLastRow + px * 128;
#pragma unroll
                for (int q = 0; q < 4; ++q) {  // channels 8 q .. 8 q + 7, real and imaginary
                    const uint4 vr = *(const uint4 *)(src + ((q ^ (px & 7)) << 4));
                    const uint4 vi = *(const uint4 *)(src + (((q + 4) ^ (px & 7)) << 4));
                    const uint32_t rr[4] = {vr.x, vr.y, vr.z, vr.w}, ii[4] = {vi.x, vi.y, vi.z, vi.w};
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t a = rr[j >> 1], e = ii[j >> 1];
                        const float hr = __uint_as_float(j & 1 ? a & 0xFFFF0000u : a << 16);
                        const float hi = __uint_as_float(j & 1 ? e & 0xFFFF0000u : e << 16);
                        const float2 k = w[tap * kC + q * 8 + j];
                        d.x = __fadd_rn(d.x, fmaf(k.x, hr, -__fmul_rn(k.y, hi)));
                        d.y = __fadd_rn(d.y, fmaf(k.y, hr, __fmul_rn(k.x, hi)));
                    }
                }
            }
            if (out) out[p] = make_float2(c.x + s * d.x, c.y + s * d.y);
            if (target) {
                // target residual in the network's units: (fine - coarse) / s
                const float er = d.x - (f.x - c.x) / s, ei = d.y - (f.y - c.y) / s;
                acc += (double)er * er + (double)ei * ei;
                g[p] = make_float2(gscale * er, gscale * ei);
            }
        }
    }
    if (loss_part) {
        red[t] = acc;
        __syncthreads();
        for (int k = kTile / 2; k > 0; k >>= 1) {
            if (t < k) red[t] += red[t + k];
            __syncthreads();
        }
        if (t == 0) loss_part[blockIdx.x] = red[0];
    }
}

// Input gradient of the last layer, masked by h5 > 0: dh5 = mask * conv^T(g) (padded
// bf16).  As the first layer: a lane per complex channel, runs of 32 pixels.
__global__ void __launch_bounds__(32 * kEdgeWarps, 3)
    last_layer_dx_kernel(const float2 *__restrict__ g, const float *__restrict__ wl,
                         const __nv_bfloat16 *__restrict__ h5, __nv_bfloat16 *__restrict__ dh, int B, int H, int W) {
    __shared__ float2 win[kEdgeWarps][3][34];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Pad pd = {H, W};
    // d = sum W h: dL/dhr = wr gr + wi gi, dL/dhi = -wi gr + wr gi
    float2 w[9];
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        const float wr = bf(__float2bfloat16_rn(wl[(t * kC + lane) * 2])),
                    wi = bf(__float2bfloat16_rn(wl[(t * kC + lane) * 2 + 1]));
        w[t] = make_float2(wr, -wi);
    }
    const unsigned rr = (unsigned)W / 32u, runs = (unsigned)B * H * rr;
    for (unsigned u = blockIdx.x * kEdgeWarps + warp; u < runs; u += gridDim.x * kEdgeWarps) {
        const unsigned line = u / rr;
        const int x0 = (int)(u - line * rr) * 32, b = (int)(line / H), y = (int)line - b * H;
        __syncwarp();
        for (int i = lane; i < 3 * 34; i += 32) {
            const int yy = wrap(y + i / 34 - 1, H), xx = wrap(x0 + i % 34 - 1, W);
            win[warp][i / 34][i % 34] = g[((size_t)b * H + yy) * W + xx];
        }
        __syncwarp();
        const bool edge = y == 0 || y == H - 1 || x0 == 0 || x0 == W - 32;  // the run touches a halo
        const size_t at = pd.at(b, y, x0) * 64 + lane;
        for (int x = 0; x < 32; x += 4) {
            float2 v[3][6];
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int j = 0; j < 6; ++j) v[r][j] = win[warp][r][x + j];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float2 a = make_float2(0.f, 0.f);
#pragma unroll
                for (int t = 0; t < 9; ++t)  // the pixel that sees this one through tap t
                    a = c_mac(a, w[t], v[2 - t / 3][j + 2 - t % 3]);
                const size_t o = at + (size_t)(x + j) * 64;
                const __nv_bfloat16 vr = __float2bfloat16_rn(bf(h5[o]) > 0.f ? a.x : 0.f),
                                    vi = __float2bfloat16_rn(bf(h5[o + kC]) > 0.f ? a.y : 0.f);
                if (edge) {
                    pd.each_copy(y, x0 + x + j, [&](int yy, int xx) {
                        __nv_bfloat16 *q = dh + pd.at(b, yy, xx) * 64 + lane;
                        q[0] = vr;
                        q[kC] = vi;
                    });
                } else {
                    dh[o] = vr;
                    dh[o + kC] = vi;
                }
            }
        }
    }
}

// ------------------------------------------------------------ weight gradients
// dW[tap][n][k] = sum_p dy[p][n] x[p + tap][k] and db[n] = sum_p dy[p][n].  Every
// CTA writes FP32 sums over its own pixels, partial[cta][10][n][k] (row 9: the
// bias, k = 0); dw_reduce_kernel adds them in CTA order.
// A CTA's float sums run over kDwChain pixels at most, whatever the batch (their error
// grows with their length): an edge layer's lane over half of them, then over the warps;
// on the tensor cores in pieces of kDwRows rows, because adding into tensor memory
// truncates, which on 16384 pixels of random waves is off by 1.9e-5 where rounded sums
// are by 2.4e-6 (2.8e-6 in pieces).  Batches of more than that many pixels an SM (2.4 M in
// all) take more CTAs than SMs.
constexpr int kDwChain = 16384;
constexpr int kDwRows = 16;  // of 128 pixels
constexpr size_t kDwStage = 6 * kATile;      // three x rows, dy at three column shifts
constexpr size_t kDwSmem = 1024 + 2 * kDwStage + 2048;

// D[m][n] (+)= A^T B, both operands stored pixel by pixel (the K dimension) with the
// channels contiguous: M- and N-major tiles of 64 channels x 8 pixels per swizzle
// atom, the next 64 channels `lbo` bytes on, the next 8 pixels 1024 bytes on.
__device__ __forceinline__ uint64_t desc_pixel_major(uint32_t addr, uint32_t lbo) {
    return (tc::desc_sw128(addr) & ~((uint64_t)0x3FFF << 16)) | (uint64_t)(lbo >> 4) << 16;
}

// The 64 x 64-channel layers on the tensor cores.  Strips as in conv_tc_kernel; for
// each row y of dy a stage holds x rows y - 1, y, y + 1 (one TMA box) and dy shifted
// by each column tap, and per 16 pixels two MMAs of M = 128, N = 192 add every tap
// at once: A is x rows (y - 1, y), then (y + 1, a tile of ones for the bias sum), B
// the three shifted dy tiles.  The two accumulators (128 x 192) stay in tensor
// memory for kDwRows rows, after which eight warps add them, rounded, to the CTA's
// partial sums.  bf16 products are exact in FP32.  Bound by the stages' 96 KB per 128
// pixels from L2 beside 16 x 96 MMA cycles.
// 8 waves of 256^2 (64 x 64 channels): 5.7 ms on the CUDA cores, now 49 us (40 with one
// read-out at the end, 112 with four warps that fetch a sum when they add to it).
__global__ void __launch_bounds__(kDwThreads, 1)
    dw_tc_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mdy, Units units,
                 float *__restrict__ partial, int *err) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *base = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *ones = base + 2 * kDwStage;   // 16 pixels x 64 channels of 1
    __shared__ uint64_t full[2], empty[2], done, read, last;
    __shared__ uint32_t tmem_base;
    __shared__ volatile int failed;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform
    for (int i = tid; i < 512; i += kDwThreads) ((uint32_t *)ones)[i] = 0x3F803F80u;
    if (warp == 1) tc::tmem_alloc(&tmem_base, 512);
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(&done, 1);
        mbar_init(&read, 8);
        mbar_init(&last, 1);
        mbar_fence_init();
        failed = 0;
    }
    fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    const int H = units.H, nunits = units.count();
    if (warp == 0) {
        if (lane == 0) {
            uint32_t n = 0;
            bool ok = true;
            for (int u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
                int b, x0, y0, y1;
                units.get(u, &b, &x0, &y0, &y1);
                for (int y = y0; y < y1; ++y, ++n) {
                    const uint32_t s = n & 1u;
                    if (n >= 2 && !(ok = wait_or_quit(&empty[s], (n / 2 - 1) & 1, &failed))) break;
                    unsigned char *st = base + s * kDwStage;
                    const int row = b * (H + 2) + y;  // of padded row y - 1
                    mbar_arrive_expect_tx(&full[s], (uint32_t)kDwStage);
                    tma_load_3d(st, &mx, 0, x0 + 1, row, &full[s]);
                    for (int kx = 0; kx < 3; ++kx)  // pixel q of x meets dy at q - (kx - 1)
                        tma_load_3d(st + (3 + kx) * kATile, &mdy, 0, x0 + 2 - kx, row + 1, &full[s]);
                }
            }
            for (uint32_t j = n > 2 ? n - 2 : 0; j < n; ++j) mbar_wait_bounded(&full[j & 1], (j / 2) & 1, kWait);
        }
        __syncwarp();
    } else if (warp == 1) {
        const uint32_t sb = smem_u32(base), so = smem_u32(ones);
        constexpr uint32_t idesc = tc::idesc_bf16(128, 192) | (1u << 15) | (1u << 16);  // A and B M/N-major
        uint32_t n = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
            int b, x0, y0, y1;
            units.get(u, &b, &x0, &y0, &y1);
            for (int y = y0; y < y1; ++y, ++n) {
                const uint32_t s = n & 1u;
                if (!(ok = wait_or_quit(&full[s], (n / 2) & 1, &failed))) break;
                const uint32_t f = n / kDwRows, r = n % kDwRows;
                if (r == 0 && f > 0 && !(ok = wait_or_quit(&read, (f - 1) & 1, &failed))) break;
                tc::fence_after_sync();
                if (tc::elect_one()) {
                    const uint32_t st = sb + s * (uint32_t)kDwStage;
#pragma unroll
                    for (int k = 0; k < kTile / 16; ++k) {
                        const uint32_t x = st + k * 2048u, x2 = x + 2u * (uint32_t)kATile;
                        const uint64_t bd = desc_pixel_major(x + 3u * (uint32_t)kATile, (uint32_t)kATile);
                        const uint32_t acc = (r > 0 || k > 0) ? 1u : 0u;
                        tc::mma_bf16(tmem, desc_pixel_major(x, (uint32_t)kATile), bd, idesc, acc);
                        tc::mma_bf16(tmem + 256u, desc_pixel_major(x2, so - x2), bd, idesc, acc);
                    }
                    tc::mma_commit(&empty[s]);
                    if (r == kDwRows - 1) tc::mma_commit(&done);
                }
                __syncwarp();
            }
        }
        if (tc::elect_one()) {
            if (ok && n % kDwRows) tc::mma_commit(&done);
            tc::mma_commit(&last);  // every MMA has completed before the CTA's memory goes
        }
        if (!mbar_wait_bounded(&last, 0, kWait)) failed = 1;
        __syncwarp();
    } else {
        // lane m of the first accumulator: x channel m % 64 of row tap m / 64, column (column tap, n);
        // of the second: row tap 2, and from m = 64 on the bias sum
        float *p = partial + (size_t)blockIdx.x * 10 * 64 * 64;
        const int m = 32 * (warp & 3) + lane, k = m & 63;
        const uint32_t lane_base = (uint32_t)(32 * (warp & 3)) << 16;
        int rows = 0;
        for (int u = blockIdx.x; u < nunits; u += gridDim.x) {
            int b, x0, y0, y1;
            units.get(u, &b, &x0, &y0, &y1);
            rows += y1 - y0;
        }
        // a warp reads half the columns, kCols at a time, whose sums so far it fetches ahead
        constexpr int kCols = 32;
        const int cbeg = warp < 6 ? 0 : 96, cend = cbeg + 96;
        float old[2][kCols];
        auto at = [&](int half, int c) {
            const int tap = half ? 6 + c / 64 : (m >> 6) * 3 + c / 64;
            return half && m >= 64 ? (9 * 64 + c % 64) * 64 : (tap * 64 + c % 64) * 64 + k;
        };
        auto mine = [&](int half, int c) { return !half || m < 64 || (m == 64 && c / 64 == 1); };
        auto fetch = [&](int c0) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < kCols; ++j) old[i][j] = mine(i, c0 + j) ? p[at(i, c0 + j)] : 0.f;
        };
        for (int f = 0; f * kDwRows < rows; ++f) {
            if (f) fetch(cbeg);
            if (__any_sync(0xffffffffu, !wait_or_quit(&done, f & 1, &failed))) break;
            tc::fence_after_sync();
#pragma unroll 1
            for (int c0 = cbeg; c0 < cend; c0 += kCols) {
                float v[2][kCols];
#pragma unroll
                for (int j = 0; j < kCols; j += 16) {
                    tc::tmem_ld16(tmem + lane_base + (uint32_t)(c0 + j), &v[0][j]);
                    tc::tmem_ld16(tmem + 256u + lane_base + (uint32_t)(c0 + j), &v[1][j]);
                }
                if (f) {
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int j = 0; j < kCols; ++j) v[i][j] = __fadd_rn(old[i][j], v[i][j]);
                    if (c0 + kCols < cend) fetch(c0 + kCols);  // while these are stored
                }
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < kCols; ++j)
                        if (mine(i, c0 + j)) p[at(i, c0 + j)] = v[i][j];
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&read);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (failed && tid == 0 && err) atomicExch(err, 1);
    if (warp == 1) tc::tmem_free(tmem, 512);
}

// The edge layers (one complex channel on one side) on the CUDA cores: a lane per
// complex channel of the wide side, a warp per run of 32 pixels of a row,
//     acc[tap][c] += s[q + sgn tap][c] wide[q][channel],   both halves of the channel,
// s the narrow side's two values per pixel (FP32, or bf16 when it is the input).
//   first layer (wide = dy, s = x, sgn = +1):  dW[tap][n][k = c]
//   last layer (wide = x, s = dy, sgn = -1):   dW[tap][n = c][k]
// 36 FMAs a pixel and lane on values in registers: issue-bound, one read of the
// wide activation.  8 waves of 256^2: 48 us each (5.7 ms on 64 x 64 tiles of zeros).
template <bool LAST>
__global__ void __launch_bounds__(32 * kEdgeWarps)
    dw_edge_kernel(const __nv_bfloat16 *__restrict__ wide, const float2 *__restrict__ sf,
                   const __nv_bfloat162 *__restrict__ sb, int B, int H, int W, float *__restrict__ partial) {
    __shared__ float2 win[kEdgeWarps][3][34];
    __shared__ float red[kEdgeWarps][40][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Pad pd = {H, W};
    float acc[9][2][2] = {}, bias[2] = {};  // [tap][narrow value][re / im half of the wide channel]
    const unsigned rr = (unsigned)W / 32u, runs = (unsigned)B * H * rr;
    for (unsigned u = blockIdx.x * kEdgeWarps + warp; u < runs; u += gridDim.x * kEdgeWarps) {
        const unsigned line = u / rr;
        const int x0 = (int)(u - line * rr) * 32, b = (int)(line / H), y = (int)line - b * H;
        __syncwarp();
        for (int i = lane; i < 3 * 34; i += 32) {
            const int yy = wrap(y + i / 34 - 1, H), xx = wrap(x0 + i % 34 - 1, W);
            const size_t p = ((size_t)b * H + yy) * W + xx;
            win[warp][i / 34][i % 34] = LAST ? sf[p] : __bfloat1622float2(sb[p]);
        }
        __syncwarp();
        const __nv_bfloat16 *wp = wide + pd.at(b, y, x0) * 64 + lane;
        for (int x = 0; x < 32; x += 8) {
            float wr[8], wi[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                wr[j] = bf(wp[(x + j) * 64]);
                wi[j] = bf(wp[(x + j) * 64 + kC]);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    // the neighbour at +tap (first layer) or -tap (last layer)
                    const float2 v = win[warp][LAST ? 2 - t / 3 : t / 3][x + j + (LAST ? 2 - t % 3 : t % 3)];
                    acc[t][0][0] = fmaf(v.x, wr[j], acc[t][0][0]);
                    acc[t][0][1] = fmaf(v.x, wi[j], acc[t][0][1]);
                    acc[t][1][0] = fmaf(v.y, wr[j], acc[t][1][0]);
                    acc[t][1][1] = fmaf(v.y, wi[j], acc[t][1][1]);
                    if (LAST && t == 4) {
                        bias[0] += v.x;
                        bias[1] += v.y;
                    }
                }
                if (!LAST) {
                    bias[0] += wr[j];
                    bias[1] += wi[j];
                }
            }
        }
    }
#pragma unroll
    for (int t = 0; t < 9; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) red[warp][t * 4 + i][lane] = acc[t][i >> 1][i & 1];
    red[warp][36][lane] = bias[0];
    red[warp][37][lane] = bias[1];
    __syncthreads();
    for (int i = threadIdx.x; i < 38 * 32; i += 32 * kEdgeWarps) {
        const int e = i / 32, ch = i % 32, c = (e >> 1) & 1, half = e & 1;
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < kEdgeWarps; ++w) sum += red[w][e][ch];
        float *p = partial + (size_t)blockIdx.x * 10 * 64 * 64;
        if (e < 36) {
            const int n = LAST ? c : half * kC + ch, k = LAST ? half * kC + ch : c;
            p[((e >> 2) * 64 + n) * 64 + k] = sum;
        } else if (!LAST || ch == 0) {
            p[(9 * 64 + (LAST ? half : half * kC + ch)) * 64] = sum;
        }
    }
}

// The partial sums of one layer added in a fixed order and contracted to
// the complex parameters: the expanded layer holds [[Wr, -Wi], [Wi, Wr]], so dWr is
// the sum of its two Wr blocks and dWi the difference of the others; db likewise.
// 32 parameters a block, their partials shared among kRedParts threads each (one
// thread over all of them waited for its loads: 105 us for 152 CTAs of 64 x 64 channels,
// now 12.5), then each of a parameter's four sums a warp's.  The six of a gradient step
// of 8 waves of 256^2 take 15 us on average; 33 with FP64 sums.
constexpr int kRedParts = 16;
__global__ void __launch_bounds__(32 * kRedParts)
    dw_reduce_kernel(const float *__restrict__ partial, int nblocks, int co, int ci, float *__restrict__ g) {
    __shared__ float part[kRedParts][4][3][32];
    __shared__ double sums[4][32];
    const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5, nw = 9 * co * ci, idx = blockIdx.x * 32 + lane;
    const bool live = idx < nw + co, isb = idx >= nw;
    const int tap = isb ? 9 : idx / (co * ci), o = isb ? idx - nw : (idx / ci) % co, i = isb ? 0 : idx % ci;
    const int at[4] = {o * 64 + i, (co + o) * 64 + ci + i, (co + o) * 64 + i, o * 64 + ci + i};
    TripleSum ps[4];
    if (live) {
        const float *p = partial + ((size_t)grp * 10 + tap) * 64 * 64;
#pragma unroll 4
        for (int b = grp; b < nblocks; b += kRedParts, p += (size_t)kRedParts * 10 * 64 * 64) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (!isb || j == 0 || j == 2) ps[j].add(p[at[j]]);
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        part[grp][j][0][lane] = ps[j].hi;
        part[grp][j][1][lane] = ps[j].mid;
        part[grp][j][2][lane] = ps[j].lo;
    }
    __syncthreads();
    if (grp < 4 && live) {  // a warp a sum
        TripleSum t;
#pragma unroll
        for (int q = 0; q < kRedParts; ++q) t.add(&part[q][grp][0][lane], 32);
        double v = t.value();
        if (!isfinite(v)) {  // beyond float's range on the way: FP64 has room
            v = 0.0;
            for (int b = 0; b < nblocks; ++b) v += partial[((size_t)b * 10 + tap) * 64 * 64 + at[grp]];
        }
        sums[grp][lane] = v;
    }
    __syncthreads();
    if (grp == 0 && live) {
        const double s[4] = {sums[0][lane], sums[1][lane], sums[2][lane], sums[3][lane]};
        float *out = g + (size_t)2 * idx;  // weights [tap][o][i][2], then bias [o][2]
        out[0] = (float)s[0] + (isb ? 0.f : (float)s[1]);
        out[1] = (float)s[2] - (isb ? 0.f : (float)s[3]);
    }
}

// Per-image scale s = sqrt(sum |psi|^2 / 256^2) (and 1/s): the wave's norm over
// a fixed reference area of 256^2 pixels, so a probe keeps its per-pixel scale
// whatever the grid it is computed on.
constexpr double kRefPixels = 65536.0;
constexpr int kRmsBlocks = 64;  // CTAs an image (one CTA an image: 640 us for 16 of 512^2, now 48, of FP64 operations)
__device__ __forceinline__ double block_sum(double v, double *red) {  // 256 threads, thread 0's result
    red[threadIdx.x] = v;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
        if ((int)threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    return red[0];
}
__global__ void __launch_bounds__(256) rms_partial_kernel(const float2 *__restrict__ psi, int HW, double *__restrict__ part) {
    __shared__ double red[256];
    // images and their blocks both on x, which takes any number of images
    const int b = blockIdx.x / kRmsBlocks, q = blockIdx.x % kRmsBlocks;
    double acc = 0.0;
    for (int i = q * 256 + threadIdx.x; i < HW; i += kRmsBlocks * 256) {
        const float2 v = psi[(size_t)b * HW + i];
        acc += (double)v.x * v.x + (double)v.y * v.y;
    }
    const double sum = block_sum(acc, red);
    if (threadIdx.x == 0) part[blockIdx.x] = sum;
}
// A warp an image.
__global__ void rms_finish_kernel(const double *__restrict__ part, float *__restrict__ s, float *__restrict__ inv) {
    const int b = blockIdx.x, lane = threadIdx.x;
    static_assert(kRmsBlocks == 64, "two partial sums a lane");
    double r = part[(size_t)b * kRmsBlocks + lane] + part[(size_t)b * kRmsBlocks + 32 + lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    if (lane) return;
    r = sqrt(r / kRefPixels);
    if (!(r > 0)) r = 1.0;
    s[b] = (float)r;
    inv[b] = (float)(1.0 / r);
}

__global__ void adam_kernel(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

}  // namespace closure

// ------------------------------------------------------------------ host side
using namespace closure;

namespace {
inline int grid_for(size_t n, int threads, int nsm) {
    size_t g = (n + threads - 1) / threads;
    const size_t cap = (size_t)nsm * 8;
    return (int)(g < cap ? (g > 0 ? g : 1) : cap);
}
// Strips and CTAs of the tensor-core weight gradients.
inline Units dw_units(int B, int H, int W, int nsm, int *grid) {
    Units u = plan_units(B, H, W, nsm, 0);
    const int rows = kDwChain / kTile, n = u.count();
    *grid = n < nsm ? n : nsm;
    if ((n + *grid - 1) / *grid * u.seg > rows) {
        const int segs = (H + rows - 1) / rows;
        u.seg = (H + segs - 1) / segs;
        const int per = rows / u.seg;
        *grid = (u.count() + per - 1) / per;
    }
    return u;
}
// CTAs of the edge layers' weight gradients.
inline int dw_edge_grid(size_t npix, int nsm) {
    const size_t runs = npix / (32 * kEdgeWarps), most = kDwChain / 64;  // of 32 pixels a warp
    const size_t ctas = runs < 2 * (size_t)nsm ? (runs > 0 ? runs : 1) : 2 * (size_t)nsm;
    return (int)(runs > ctas * most ? (runs + most - 1) / most : ctas);
}
// CTAs of the kernels with a warp per 32 pixels
inline int edge_grid(size_t npix, int nsm) { return grid_for(npix, 32 * kEdgeWarps, nsm); }
}  // namespace

int closure_param_count() { return param_count(); }

cudaError_t ClosureNet::alloc_params() {
    const size_t n = (size_t)param_count();
    cudaError_t e;
    if ((e = cudaMalloc(&params, sizeof(float) * n)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&grads, sizeof(float) * n)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&adam_m, sizeof(float) * n)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&adam_v, sizeof(float) * n)) != cudaSuccess) return e;
    if ((e = cudaMemset(adam_m, 0, sizeof(float) * n)) != cudaSuccess) return e;
    if ((e = cudaMemset(adam_v, 0, sizeof(float) * n)) != cudaSuccess) return e;
    // expanded bf16 weights of the four tensor-core layers, forward and transposed
    if ((e = cudaMalloc(&wt, sizeof(__nv_bfloat16) * 8 * 9 * 64 * 64)) != cudaSuccess) return e;
    return cudaSuccess;
}

void ClosureNet::release() {
    void *ptrs[] = {params, grads, adam_m, adam_v, wt, acts, partial, loss_part, scale, rms_part};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    params = grads = adam_m = adam_v = partial = scale = nullptr;
    wt = nullptr;
    acts = nullptr;
    loss_part = rms_part = nullptr;
    cap_bytes = cap_pix = 0;
    cap_img = cap_part = 0;
}

// Bytes of one padded activation, and of the workspace of a batch: training keeps
// every layer's activation; inference only a ping-pong pair.
static size_t act_bytes(int B, int H, int W) { return ((Pad{H, W}.pixels(B) * 128 + 255) / 256) * 256; }
static size_t plain_bytes(size_t npix, size_t per) { return ((npix * per + 255) / 256) * 256; }

cudaError_t ClosureNet::ensure(int B, int H, int W, bool train, int nsm) {
    const size_t npix = (size_t)B * H * W;
    int part = 0;  // CTAs whose weight-gradient sums are kept
    if (train) {
        dw_units(B, H, W, nsm, &part);
        const int e = dw_edge_grid(npix, nsm);
        part = part > e ? part : e;
    }
    size_t bytes = train ? 7 * act_bytes(B, H, W) + plain_bytes(npix, 4) + plain_bytes(npix, 8)
                               : 2 * act_bytes(B, H, W);
    if (bytes > cap_bytes || npix > cap_pix || B > cap_img || part > cap_part) {
        // every part at least as large as it was, so that two shapes in turn allocate once
        bytes = bytes > cap_bytes ? bytes : cap_bytes;
        part = part > cap_part ? part : cap_part;
        const size_t pix = npix > cap_pix ? npix : cap_pix;
        const int img = B > cap_img ? B : cap_img;
        if (acts) cudaFree(acts);
        if (partial) cudaFree(partial);
        if (loss_part) cudaFree(loss_part);
        if (scale) cudaFree(scale);
        if (rms_part) cudaFree(rms_part);
        acts = nullptr;
        partial = nullptr;
        loss_part = nullptr;
        scale = nullptr;
        rms_part = nullptr;
        cap_bytes = cap_pix = 0;
        cap_img = cap_part = 0;
        cudaError_t e;
        if ((e = cudaMalloc(&acts, bytes)) != cudaSuccess) return e;
        if (part && (e = cudaMalloc(&partial, sizeof(float) * part * 10 * 64 * 64)) != cudaSuccess) return e;
        if ((e = cudaMalloc(&loss_part, sizeof(double) * 4096)) != cudaSuccess) return e;
        if ((e = cudaMalloc(&scale, sizeof(float) * 2 * img)) != cudaSuccess) return e;
        if ((e = cudaMalloc(&rms_part, sizeof(double) * kRmsBlocks * img)) != cudaSuccess) return e;
        cap_bytes = bytes;
        cap_pix = pix;
        cap_img = img;
        cap_part = part;
    }
    return cudaSuccess;
}

cudaError_t ClosureNet::expand(cudaStream_t s, int nsm, int64_t *launches) {
    // layers 1..4 (0-based) are the tensor-core layers
    expand_kernel<<<dim3((2 * 9 * kR * kR + 255) / 256, 4), 256, 0, s>>>(params, param_offset(1), layer_size(1), wt);
    ++*launches;
    return cudaGetLastError();
}

// Padded activations as rows of pixels, boxes of 64 channels x 128 pixels x `rows` rows.
static bool act_map(CUtensorMap *m, const __nv_bfloat16 *p, int B, int H, int W, uint32_t rows = 1) {
    const uint64_t dims[3] = {64, (uint64_t)W + 2, (uint64_t)B * (H + 2)};
    const uint64_t strides[2] = {128, 128 * ((uint64_t)W + 2)};
    const uint32_t box[3] = {64, kTile, rows};
    return encode_tensor_map(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, p, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

cudaError_t ClosureNet::conv_tc(const __nv_bfloat16 *in, const __nv_bfloat16 *w, const float *bias,
                                const __nv_bfloat16 *mask, __nv_bfloat16 *out, int B, int H, int W, int epi,
                                int *err, cudaStream_t s, int nsm, int64_t *launches) {
    static KernelSetup ks;
    int per_sm = 0;
    cudaError_t e = ks.get(conv_tc_kernel, kConvThreads, kConvSmem, false, &per_sm);
    if (e != cudaSuccess) return e;
    CUtensorMap mi, mo;
    if (!act_map(&mi, in, B, H, W) || !act_map(&mo, out, B, H, W)) return cudaErrorInvalidValue;
    const Units u = plan_units(B, H, W, nsm, 2);
    const int grid = u.count() < nsm ? u.count() : nsm;
    ++*launches;
    conv_tc_kernel<<<grid, kConvThreads, kConvSmem, s>>>(mi, mo, w, bias, mask, out, u, epi, err);
    return cudaGetLastError();
}

// Forward pass.  psi: complex64 [B][H][W]; out (may be null, may equal psi):
// psi + s d; target (training): the fine-slice waves -> loss and dL/dd.
cudaError_t ClosureNet::forward(const float2 *psi, int B, int H, int W, float2 *out, const float2 *target,
                                bool train, int *err, cudaStream_t s, int nsm, int64_t *launches) {
    if (W % kTile || H < 3 || W < 3) return cudaErrorInvalidValue;
    const size_t npix = (size_t)B * H * W;
    cudaError_t e = ensure(B, H, W, train, nsm);
    if (e != cudaSuccess) return e;
    if ((e = expand(s, nsm, launches)) != cudaSuccess) return e;
    float *sc = scale, *inv = scale + B;
    rms_partial_kernel<<<kRmsBlocks * B, 256, 0, s>>>(psi, H * W, rms_part);
    rms_finish_kernel<<<B, 32, 0, s>>>(rms_part, sc, inv);
    *launches += 2;
    unsigned char *a = (unsigned char *)acts;
    const size_t act = act_bytes(B, H, W);
    auto take = [&](size_t bytes) {
        unsigned char *p = a;
        a += bytes;
        return p;
    };
    __nv_bfloat16 *h[6];
    if (train) {
        for (int l = 1; l <= 5; ++l) h[l] = (__nv_bfloat16 *)take(act);
        dh[0] = (__nv_bfloat16 *)take(act);
        dh[1] = (__nv_bfloat16 *)take(act);
        xbuf = (__nv_bfloat16 *)take(plain_bytes(npix, 4));
        g6 = (float *)take(plain_bytes(npix, 8));
    } else {
        // inference: h1 -> A, h2 -> B, h3 -> A, ... ; the scaled input is not kept
        h[1] = h[3] = h[5] = (__nv_bfloat16 *)take(act);
        h[2] = h[4] = (__nv_bfloat16 *)take(act);
        xbuf = nullptr;
        g6 = nullptr;
    }
    for (int l = 1; l <= 5; ++l) hbuf[l] = h[l];
    first_layer_kernel<<<edge_grid(npix, nsm), 32 * kEdgeWarps, 0, s>>>(
        psi, inv, params + param_offset(0), (__nv_bfloat162 *)xbuf, h[1], B, H, W);
    ++*launches;
    for (int l = 1; l <= 4; ++l) {
        const __nv_bfloat16 *w = wt + (size_t)(2 * (l - 1)) * 9 * 64 * 64;
        const float *bias = params + param_offset(l) + layer_wsize(l);
        if ((e = conv_tc(h[l], w, bias, nullptr, h[l + 1], B, H, W, EPI_BIAS_RELU, err, s, nsm, launches)) !=
            cudaSuccess)
            return e;
    }
    static KernelSetup ks;
    int per_sm = 0;
    if ((e = ks.get(last_layer_kernel, kTile, kLastSmem, true, &per_sm)) != cudaSuccess) return e;
    const Units u = plan_units(B, H, W, nsm * per_sm, 2);
    const int nblk = u.count() < nsm * per_sm ? u.count() : nsm * per_sm;
    last_layer_kernel<<<nblk, kTile, kLastSmem, s>>>(h[5], params + param_offset(5), psi, sc, target, out, (float2 *)g6,
                                                     target ? loss_part : nullptr, target ? 2.0f / (float)npix : 0.f,
                                                     u);
    ++*launches;
    loss_blocks = target ? nblk : 0;
    return cudaGetLastError();
}

// Backward pass after forward(train = true, target): grads <- dL/dtheta.
cudaError_t ClosureNet::backward(int B, int H, int W, int *err, cudaStream_t s, int nsm, int64_t *launches) {
    const size_t npix = (size_t)B * H * W;
    cudaError_t e;
    auto reduce = [&](int l, int nblk) {
        const int co = layer_co(l), ci = layer_ci(l);
        dw_reduce_kernel<<<(9 * co * ci + co + 31) / 32, 32 * kRedParts, 0, s>>>(partial, nblk, co, ci, grads + param_offset(l));
        *launches += 2;
    };
    const int edge = dw_edge_grid(npix, nsm);
    auto wgrad = [&](int l, const __nv_bfloat16 *dy) -> cudaError_t {
        static KernelSetup ks;
        int per_sm = 0;
        cudaError_t e = ks.get(dw_tc_kernel, kDwThreads, kDwSmem, false, &per_sm);
        if (e != cudaSuccess) return e;
        CUtensorMap mx, mdy;
        if (!act_map(&mx, hbuf[l], B, H, W, 3) || !act_map(&mdy, dy, B, H, W, 1)) return cudaErrorInvalidValue;
        int grid;
        const Units u = dw_units(B, H, W, nsm, &grid);
        dw_tc_kernel<<<grid, kDwThreads, kDwSmem, s>>>(mx, mdy, u, partial, err);
        reduce(l, grid);
        return cudaGetLastError();
    };
    // layer 6 (C -> 1): dW from g6, then dh5 = mask(h5) conv6^T(g6)
    dw_edge_kernel<true><<<edge, 32 * kEdgeWarps, 0, s>>>(hbuf[5], (const float2 *)g6, nullptr, B, H, W, partial);
    reduce(5, edge);
    last_layer_dx_kernel<<<edge_grid(npix, nsm), 32 * kEdgeWarps, 0, s>>>(
        (const float2 *)g6, params + param_offset(5), hbuf[5], dh[1], B, H, W);
    ++*launches;
    int cur = 1;
    for (int l = 4; l >= 1; --l) {
        // dh[cur] = dL/dpre_{l+1} (masked); weight gradient of layer l with input h_l
        if ((e = wgrad(l, dh[cur])) != cudaSuccess) return e;
        const __nv_bfloat16 *wT = wt + (size_t)(2 * (l - 1) + 1) * 9 * 64 * 64;
        if ((e = conv_tc(dh[cur], wT, nullptr, hbuf[l], dh[cur ^ 1], B, H, W, EPI_MASK, err, s, nsm, launches)) !=
            cudaSuccess)
            return e;
        cur ^= 1;
    }
    // layer 1 (1 -> C): input the scaled bf16 wave
    dw_edge_kernel<false><<<edge, 32 * kEdgeWarps, 0, s>>>(dh[cur], nullptr, (const __nv_bfloat162 *)xbuf, B, H, W,
                                                           partial);
    reduce(0, edge);
    return cudaGetLastError();
}

cudaError_t ClosureNet::adam(float lr, cudaStream_t s, int nsm, int64_t *launches) {
    ++step;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    const int n = param_count();
    adam_kernel<<<grid_for(n, 256, nsm), 256, 0, s>>>(params, grads, adam_m, adam_v, n, lr, b1, b2, 1e-8f, c1, c2);
    ++*launches;
    return cudaGetLastError();
}

// He-style initial weights from the library's splitmix64 stream (host), zero biases.
void closure_init_params(uint64_t seed, std::vector<float> &h) {
    h.assign(param_count(), 0.f);
    auto mix = [](uint64_t x) {
        x += 0x9E3779B97F4A7C15ull;
        x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
        x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
        return x ^ (x >> 31);
    };
    uint64_t ctr = 0;
    for (int l = 0; l < kLayers; ++l) {
        const int co = layer_co(l), ci = layer_ci(l);
        // complex fan-in 9 ci; the last layer starts small so the closure starts near identity
        float sd = sqrtf(1.0f / (9.0f * ci));
        if (l == kLayers - 1) sd *= 0.1f;
        float *w = h.data() + param_offset(l);
        for (int i = 0; i < 9 * co * ci * 2; ++i) {
            const double u1 = ((mix(seed ^ mix(ctr++)) >> 11) + 1.0) * (1.0 / 9007199254740993.0);
            const double u2 = (mix(seed ^ mix(ctr++)) >> 11) * (1.0 / 9007199254740992.0);
            w[i] = (float)(sd * sqrt(-2.0 * log(u1)) * cos(2.0 * 3.14159265358979323846 * u2));
        }
    }
}

}  // namespace msl
