// Projected-potential gather kernel: the PotentialBuilder step.
//
// Reference: LMultiSlice ModelPotential::calculatePotentialGrid
// (ImageSimulation/LMultiSlice/ModelPotential.cu:27-99) bins atoms by z and, for
// every pixel, sums calculateProjectedPotential over all atoms of the slice in
// 4608-atom constant-memory batches (:125-230), evaluating K0 in FP64 for every
// pixel-atom pair before the cutoff test.  The atom form used here is Kirkland's
// vzatom (multislice/slicelib.cpp:2666-2716):
//     V(r) = AL sum_i a_i K0(2 pi r sqrt(b_i)) + AG sum_i (c_i/d_i) exp(-pi^2 r^2 / d_i)
// with FPARAMS coefficients, K0/I0 by the Abramowitz & Stegun 9.8.1/9.8.5/9.8.6
// polynomials the reference uses (slicelib.cpp:168-235).
//
// GB300 design: one CTA per 64 x 32 pixel tile of one slice, eight pixels per
// thread (independent accumulators for latency hiding).  The slice's atoms
// stream through in rounds of 512, two per thread; each round is culled against
// the tile's periodic bounding box (in float, from float copies of the
// coordinates, with a margin that keeps every atom the exact test would:
// culling only has to be conservative) and compacted in atom order (so the
// float sum order is fixed) into a list of at most 64 atoms at a time.  Each
// atom arrives as its nearest pixel (ic, jc) and the residue x - ic dxp,
// y - jc dyp, formed in FP64 (atom_sort_kernel) and rounded to float, so the offset of
// pixel column ix is |residue + m dxp| with m = ic - ix folded to the minimum
// image in integers: all in FP32, and an atom sitting exactly on a pixel keeps
// the FP64 residue there (r is then clamped to 1e-10 A as the reference does,
// never a float rounding residue).  The per-atom offsets of the tile's 32
// columns and 32 rows are formed once per tile and the pair loop runs in FP32
// on them.  Every pixel sums its atoms in atom order, whatever the tile shape.
// 64-pixel-wide tiles halve the per-pixel share of the per-atom work against
// 32 x 32 (Au 2048^2: 2.78 ms per configuration against 3.40).  A warp's pixels are
// blocks of 4 x 8, so that a block is mostly all inside or all outside a cutoff and its
// lanes look up neighbouring table pieces; the piece number comes from a float
// addition, not conversions (a quarter-rate pipe).  What bounds it: the
// 16-byte table gathers (shared-memory wavefronts at 78 % of peak) and issue (76 %):
// SrTiO3, 100 slices of 512^2, 5 A cutoff: 0.50 ms (0.69 with warps of 32 rows x 1
// column, converted piece numbers and a branch per pixel); Au 2048^2, 40 slices, 3 A:
// 1.08 ms (1.42).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "msl_internal.h"

namespace msl {

namespace {
// tile shape and list capacity picked by timing 16 / 32 / 64 / 128-pixel-wide tiles
// and 32 / 64 / 128-atom lists on the Au 2048^2 potentials
constexpr int TX = 64, TY = 32, THREADS = 256, PX = TX * TY / THREADS, CAP = 64;
static_assert(TX == 64 && TY == 32 && THREADS == 256 && PX == 8, "a warp covers 32 x 8 pixels in blocks of 4 x 8");
constexpr int KR = 2, ROUND = KR * THREADS, NW = THREADS / 32;  // atoms culled per thread per round
static_assert(KR * NW <= 32, "one warp scans the counts");

__device__ __forceinline__ float poly(const float *c, int n, float t) {
    float s = c[n - 1];
    for (int i = n - 2; i >= 0; --i) s = fmaf(s, t, c[i]);
    return s;
}

__constant__ float kI0A[7] = {1.0f, 3.5156229f, 3.0899424f, 1.2067492f, 0.2659732f, 0.0360768f, 0.0045813f};
__constant__ float kK0A[7] = {-0.57721566f, 0.42278420f, 0.23069756f, 0.03488590f, 0.00262698f,
                              0.00010750f, 0.00000740f};
__constant__ float kK0B[7] = {1.25331414f, -0.07832358f, 0.02189568f, -0.01062446f, 0.00587872f,
                              -0.00251540f, 0.00053208f};

constexpr float kRound = 12582912.0f;  // 1.5 2^23: adding it rounds to an integer
// Least |dy| of a pair, so that r^2 is never 0 or a denormal (whose reciprocal root
// below is infinite): far below the 1e-10 A at which r is clamped.
constexpr float kTiny = 1.2e-19f;
// 1 / sqrt(x) of a normal x > 0 (denormals are taken as 0).
__device__ __forceinline__ float rsqrt_normal(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// K0(x), x > 0 (A&S 9.8.5 for x <= 2 with I0 from 9.8.1, 9.8.6 above).
__device__ __forceinline__ float bessk0f(float x) {
    if (x <= 2.0f) {
        const float t = (x / 3.75f) * (x / 3.75f);
        const float i0 = poly(kI0A, 7, t);
        const float x2 = 0.25f * x * x;
        return -logf(0.5f * x) * i0 + poly(kK0A, 7, x2);
    }
    return expf(-x) * poly(kK0B, 7, 2.0f / x) * rsqrtf(x);
}
// vzatom at r = max(sqrt(r2), 1e-10 A); p: A1 B1 A2 B2 A3 B3 C1 D1 C2 D2 C3 D3
__device__ __noinline__ float pot_analytic(const float *p, float r2) {
    const float r = sqrtf(fmaxf(r2, 1.0e-20f));
    float v = __ldg(p + 0) * bessk0f(__ldg(p + 1) * r) + __ldg(p + 2) * bessk0f(__ldg(p + 3) * r) +
              __ldg(p + 4) * bessk0f(__ldg(p + 5) * r);
    const float rr = r * r;
    v += __ldg(p + 6) * expf(-__ldg(p + 7) * rr) + __ldg(p + 8) * expf(-__ldg(p + 9) * rr) +
         __ldg(p + 10) * expf(-__ldg(p + 11) * rr);
    return v;
}
}  // namespace

template <bool TAB>
__global__ void __launch_bounds__(THREADS, 4) potential_kernel(PotArgs a) {
    extern __shared__ float4 stab[];  // TAB: [nsp][kPotTabN] cubic pieces of the species' radial profiles
    __shared__ int sZ[CAP];
    __shared__ int sS[CAP];
    __shared__ int sic[CAP], sjc[CAP];
    __shared__ float sfx[CAP], sfy[CAP];
    __shared__ __align__(16) float sdx[CAP][TX];  // [half][lane column][block]: a thread's eight in a row
    __shared__ float sdy[CAP][TY];
    __shared__ int wcount[KR * NW];
    const int tid = threadIdx.x;
    if (TAB) {
        for (int i = tid; i < a.nsp * kPotTabN; i += THREADS) stab[i] = a.tab[i];
    }
    const int lane = tid & 31, warp = tid >> 5;
    // a warp's pixel block j: 4 columns (along x) of 8 neighbouring rows (along y)
    const int ty = 8 * (warp & 3) + (lane & 7), tx = 32 * (warp >> 2) + (lane >> 3);  // pixels (tx + 4 j, ty), j < PX
    const int txs = 8 * (4 * (warp >> 2) + (lane >> 3));
    const int iy0 = blockIdx.x * TY, ix0 = blockIdx.y * TX, s = blockIdx.z;

    // tile bounding box (pixel positions) for the culling, in float.  The culling only has
    // to keep every atom that can reach the tile (the pair loop tests r < radius), so the
    // margin covers the rounding of the positions at any cell size: the atom's, the tile
    // middle's (pixel size and product), the cell edge's and two differences, each at most
    // 2^-24 of the cell edge, 3.6e-7 of it together.
    const float xc = ((float)ix0 + 0.5f * (TX - 1)) * a.dxpf, hx = 0.5f * (TX - 1) * a.dxpf;
    const float yc = ((float)iy0 + 0.5f * (TY - 1)) * a.dypf, hy = 0.5f * (TY - 1) * a.dypf;
    const float axf = (float)a.ax, byf = (float)a.by;
    const float rad = sqrtf(a.rad2) * (1.0f + 1e-5f) + 1e-3f + 4e-7f * fmaxf(axf, byf);
    const int a0 = a.off[s], a1 = a.off[s + 1];
    float acc[PX];
#pragma unroll
    for (int j = 0; j < PX; ++j) acc[j] = 0.f;

    for (int c0 = a0; c0 < a1; c0 += ROUND) {
        // cull: atom c0 + k THREADS + tid; the kept atoms' pixel positions and
        // species are loaded right away so their latency overlaps the compaction
        bool keep[KR];
        unsigned ball[KR];
        int ia[KR], ja[KR], za[KR];
        float fxa[KR], fya[KR];
#pragma unroll
        for (int k = 0; k < KR; ++k) {
            const int ai = c0 + k * THREADS + tid;
            keep[k] = false;
            ia[k] = ja[k] = za[k] = 0;
            fxa[k] = fya[k] = 0.f;
            if (ai < a1) {
                float dx = fabsf(a.xf[ai] - xc);
                dx = fminf(dx, axf - dx);
                float dy = fabsf(a.yf[ai] - yc);
                dy = fminf(dy, byf - dy);
                keep[k] = (dx - hx < rad) && (dy - hy < rad);
                if (keep[k]) {
                    ia[k] = a.ic[ai];
                    ja[k] = a.jc[ai];
                    fxa[k] = a.fx[ai];
                    fya[k] = a.fy[ai];
                    za[k] = a.Z[ai];
                }
            }
            ball[k] = __ballot_sync(0xffffffffu, keep[k]);
        }
        __syncthreads();  // the previous round's pair loop is done with wcount and the lists
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < KR; ++k) wcount[k * NW + warp] = __popc(ball[k]);
        }
        __syncthreads();
        // order-preserving positions: atom order is (k, warp, lane); lane q < KR NW scans
        // the counts of the (k, warp) pairs in that order
        int scan = lane < KR * NW ? wcount[lane] : 0;
#pragma unroll
        for (int o = 1; o < KR * NW; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, scan, o);
            if (lane >= o) scan += up;
        }
        const int total = __shfl_sync(0xffffffffu, scan, KR * NW - 1);
        int pos[KR];
#pragma unroll
        for (int k = 0; k < KR; ++k)
            pos[k] = __shfl_sync(0xffffffffu, scan, k * NW + warp) - __popc(ball[k]) +
                     __popc(ball[k] & ((1u << lane) - 1u));
        for (int piece = 0; piece < total; piece += CAP) {
            if (piece > 0) __syncthreads();  // the previous piece's pair loop is done with the lists
#pragma unroll
            for (int k = 0; k < KR; ++k) {
                const int p = pos[k] - piece;
                if (keep[k] && p >= 0 && p < CAP) {
                    sZ[p] = za[k];
                    if (TAB) sS[p] = a.zslot[za[k]];
                    sic[p] = ia[k];
                    sjc[p] = ja[k];
                    sfx[p] = fxa[k];
                    sfy[p] = fya[k];
                }
            }
            __syncthreads();
            const int n = min(CAP, total - piece);
            // per-atom offsets of this tile's columns and rows: |residue + m pixel|,
            // m the pixel difference folded to the minimum image (ModelPotential.cu:154-203)
            for (int idx = tid; idx < n * TX; idx += THREADS) {
                const int k = idx / TX, i = idx % TX;
                int m = sic[k] - (ix0 + i);
                if (2 * m >= a.nx) m -= a.nx;
                else if (2 * m < -a.nx) m += a.nx;
                sdx[k][8 * (4 * (i >> 5) + (i & 3)) + ((i >> 2) & 7)] = fabsf(fmaf((float)m, a.dxpf, sfx[k]));
            }
            for (int idx = tid; idx < n * TY; idx += THREADS) {
                const int k = idx / TY, i = idx % TY;
                int m = sjc[k] - (iy0 + i);
                if (2 * m >= a.ny) m -= a.ny;
                else if (2 * m < -a.ny) m += a.ny;
                sdy[k][i] = fmaxf(fabsf(fmaf((float)m, a.dypf, sfy[k])), kTiny);
            }
            __syncthreads();
            for (int k = 0; k < n; ++k) {
                // the warp stays together: a block with no pixel inside the cutoff is skipped,
                // in any other every lane goes through the table and the outer ones drop it
                const float dy = sdy[k][ty], dy2 = dy * dy;
                if (!__any_sync(0xffffffffu, dy2 < a.rad2)) continue;
                const float4 d0 = *(const float4 *)&sdx[k][txs], d1 = *(const float4 *)&sdx[k][txs + 4];
                const float dx[PX] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
                const float4 *tb = TAB ? stab + sS[k] * kPotTabN : nullptr;
#pragma unroll
                for (int j = 0; j < PX; ++j) {
                    const float r2 = fmaf(dx[j], dx[j], dy2);
                    const bool in = r2 < a.rad2;
                    if (!__any_sync(0xffffffffu, in)) continue;
                    float v = 0.f;
                    bool near = true;  // below the table: the analytic form
                    if (TAB) {
                        // cubic piece of the tabulated profile in t = u - i, |t| <= 1/2, about the
                        // middle of the piece i nearest u: rounded by adding 1.5 2^23, so that no
                        // pair takes a conversion (a pixel beyond the cutoff lands on any piece)
                        const float u = fmaf(r2 * rsqrt_normal(r2), a.tab_inv_h, a.tab_off);
                        const float m = u + kRound;
                        const float t = u - (m - kRound);
                        const float4 c = tb[__float_as_int(m) & (kPotTabN - 1)];
                        v = fmaf(fmaf(fmaf(c.w, t, c.z), t, c.y), t, c.x);
                        near = !(u >= -0.5f);
                    }
                    if (near && in) v = pot_analytic(a.sp + sZ[k] * 12, r2);
                    if (in) acc[j] += v;
                }
            }
        }
    }
    const int iy = iy0 + ty;
#pragma unroll
    for (int j = 0; j < PX; ++j) {
        const int ix = ix0 + tx + 4 * j;
        if (ix < a.nx && iy < a.ny) a.v[((size_t)s * a.nx + ix) * a.ny + iy] = acc[j];
    }
}

cudaError_t launch_potential(const PotArgs &a, cudaStream_t s, int64_t *launches) {
    ++*launches;
    dim3 grid((a.ny + TY - 1) / TY, (a.nx + TX - 1) / TX, a.nslice);
    if (a.nsp > 0 && a.tab) {
        const size_t smem = sizeof(float4) * (size_t)a.nsp * kPotTabN;
        static KernelSetup ks;
        int per_sm = 0;
        cudaError_t e = ks.get(potential_kernel<true>, THREADS, sizeof(float4) * kPotMaxSp * kPotTabN, true, &per_sm);
        if (e != cudaSuccess) return e;
        potential_kernel<true><<<grid, THREADS, smem, s>>>(a);
    } else {
        potential_kernel<false><<<grid, THREADS, 0, s>>>(a);
    }
    return cudaGetLastError();
}

// ------------------------------------------------------------- atoms by slice
// (97 us on one host core for the 32,000 atoms of the SrTiO3 crystal)
namespace {
__global__ void atom_sort_kernel(AtomSort a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.natom) return;
    const AtomIn in = a.in[i];
    const int p = a.off[in.k] + in.rank;
    const double xw = in.x - a.ax * floor(in.x / a.ax), yw = in.y - a.by * floor(in.y / a.by);
    // nearest pixel and the FP64 residue (the same expression as |x - ix dxp| at that
    // pixel); the pixel index is then wrapped into the grid
    const double ci = floor(xw / a.dxp + 0.5), cj = floor(yw / a.dyp + 0.5);
    a.fx[p] = (float)(xw - ci * a.dxp);
    a.fy[p] = (float)(yw - cj * a.dyp);
    a.ic[p] = (int)ci % a.nx;
    a.jc[p] = (int)cj % a.ny;
    a.zd[p] = in.Z;
    a.xf[p] = (float)xw;
    a.yf[p] = (float)yw;
}
}  // namespace

cudaError_t launch_atom_sort(const AtomSort &a, cudaStream_t s, int64_t *launches) {
    if (a.natom < 1) return cudaSuccess;
    ++*launches;
    atom_sort_kernel<<<(a.natom + 127) / 128, 128, 0, s>>>(a);
    return cudaGetLastError();
}

// ------------------------------------------------------------ radial tables
// Cubic pieces of vzatom evaluated in FP64 (slicelib.cpp:2666-2716 with the A&S Bessel
// polynomials of :168-235), kPotTabN of width h from r0 per species: the cubic through
// the profile at t = -1/2, -1/6, 1/6, 1/2 about the middle of piece i, a thread per
// point.  On one host core the three species of SrTiO3 took 218 us a call.
namespace {
__device__ __forceinline__ double polyd(const double *c, double t) {
    double s = c[6];
#pragma unroll
    for (int i = 5; i >= 0; --i) s = s * t + c[i];
    return s;
}
__constant__ double kI0D[7] = {1.0, 3.5156229, 3.0899424, 1.2067492, 0.2659732, 0.0360768, 0.0045813};
__constant__ double kK0AD[7] = {-0.57721566, 0.42278420, 0.23069756, 0.03488590, 0.00262698, 0.00010750, 0.00000740};
__constant__ double kK0BD[7] = {1.25331414, -0.07832358, 0.02189568, -0.01062446, 0.00587872, -0.00251540, 0.00053208};
__device__ double bessk0d(double x) {
    if (x <= 2.0) {
        const double q = (x / 3.75) * (x / 3.75);
        return -log(0.5 * x) * polyd(kI0D, q) + polyd(kK0AD, 0.25 * x * x);
    }
    return exp(-x) * polyd(kK0BD, 2.0 / x) / sqrt(x);
}
__device__ double vz_double(const double *f, double r) {
    const double AL = 300.8242834, AG = 150.4121417, PIK = 3.141592654;
    const double x = 2.0 * PIK * r;
    double suml = 0.0, sumg = 0.0;
    for (int i = 0; i < 3; ++i) suml += f[2 * i] * bessk0d(x * sqrt(f[2 * i + 1]));
    const double x2 = (PIK * r) * (PIK * r);
    for (int i = 0; i < 3; ++i) sumg += f[6 + 2 * i] * exp(-x2 / f[7 + 2 * i]) / f[7 + 2 * i];
    return AL * suml + AG * sumg;
}
constexpr int TAB_THREADS = 64;
__global__ void __launch_bounds__(TAB_THREADS)
    potential_tables_kernel(const __grid_constant__ PotRows rows, double r0, double h, float4 *out) {
    // four neighbouring lanes hold a piece's four points
    const int piece = (blockIdx.x * TAB_THREADS + threadIdx.x) >> 2, q = threadIdx.x & 3;
    const double r = r0 + piece * h;
    const double y = vz_double(rows.r[blockIdx.y], q == 0 ? r : q == 1 ? r + h / 3 : q == 2 ? r + 2 * h / 3 : r + h);
    const int l0 = threadIdx.x & 28;
    const double y0 = __shfl_sync(0xffffffffu, y, l0), y1 = __shfl_sync(0xffffffffu, y, l0 + 1),
                 y2 = __shfl_sync(0xffffffffu, y, l0 + 2), y3 = __shfl_sync(0xffffffffu, y, l0 + 3);
    if (q == 0) {
        const double s0 = y1 + y2, s1 = y0 + y3, d0 = y2 - y1, d1 = y3 - y0;
        out[blockIdx.y * kPotTabN + piece] =
            make_float4((float)((9 * s0 - s1) / 16), (float)((27 * d0 - d1) / 8), (float)(9 * (s1 - s0) / 4),
                        (float)(9 * (d1 - 3 * d0) / 2));
    }
}
}  // namespace

cudaError_t launch_potential_tables(const PotRows &rows, int nsp, double r0, double h, float4 *out, cudaStream_t s,
                                    int64_t *launches) {
    ++*launches;
    static_assert(4 * kPotTabN % TAB_THREADS == 0, "whole blocks of pieces");
    potential_tables_kernel<<<dim3(4 * kPotTabN / TAB_THREADS, nsp), TAB_THREADS, 0, s>>>(
        rows, r0, h, out);
    return cudaGetLastError();
}

}  // namespace msl
