// Denoiser kernels (denoise_kernels.cuh). The convolutions are implicit GEMMs
// on the BF16 tensor cores with FP32 accumulators: tcgen05 MMAs into TMEM
// (the strip kernel, TMA-fed, for layers whose weights fit in shared memory;
// per-tile kernels for the rest), and the warp-level mma.sync m16n8k16 kernels
// (operand tiles read with ldmatrix) kept as a cross-check.
#include <algorithm>
#include <atomic>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "denoise_kernels.cuh"
#include "per_device.h"

namespace vvdn {

namespace {

__device__ __forceinline__ uint32_t smem_addr(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}

__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
                 "{%8, %9}, {%0, %1, %2, %3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Programmatic dependent launch: the network's launches follow each other
// closely, so each one starts while the previous one still runs, up to its
// first access to what earlier launches write (weights excepted, which a
// launch at least two back wrote): 12 us of launch and start-up per
// convolution are mostly hidden (a 256 x 256 frame, 27 launches: 289 us of
// kernel time one by one, 249 us as they run). pdl_wait returns when the previous launch
// is complete and its writes are visible; pdl_start, issued after it, lets the
// next launch begin.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Asynchronous 16-byte global -> shared copy; src_bytes = 0 writes zeros
// (padding, channels past cin, rows past cout).
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_addr(smem)), "l"(gmem),
                 "r"(valid ? 16 : 0));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// Forward tile: 256 threads = 8 warps; block tile 128 pixels x BN output
// channels (BN = 64: warps 4 x 2 of 32 x 32; BN = 32: warps 8 x 1 of 16 x 32,
// for the 32- and 16-channel layers). K runs over (tap, 32-channel chunk)
// with a 3-stage cp.async pipeline.
constexpr int kBM = 128, kBK = 32, kStages = 3, kLds = kBK + 8;

template <int BN, int WM>
__global__ void __launch_bounds__(256) k_conv3x3(ConvArgs a)
{
    constexpr int WN = 32;                // channels per warp
    constexpr int WARPS_M = kBM / WM;     // 4 or 8
    constexpr int MT = WM / 16, NT = WN / 8;
    static_assert(WARPS_M * (BN / WN) == 8, "8 warps");
    __shared__ __align__(128) bf16 sA[kStages][kBM][kLds];
    __shared__ __align__(128) bf16 sB[kStages][BN][kLds];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wm = warp % WARPS_M, wn = warp / WARPS_M;
    const long P = (long)a.n * a.h * a.wd;
    const long p0 = (long)blockIdx.x * kBM;
    const int c0 = blockIdx.y * BN;
    const int nchunks = (a.cin + kBK - 1) / kBK;
    const int KT = 9 * nchunks;
    // A loads: row tid / 2, two 8-channel vectors starting at (tid % 2) * 16
    const int ar = tid >> 1, av = (tid & 1) * 16;
    const long ap = p0 + ar;
    int an = 0, ay = 0, ax = 0;
    if (ap < P) {
        an = (int)(ap / ((long)a.h * a.wd));
        const int rem = (int)(ap - (long)an * a.h * a.wd);
        ay = rem / a.wd;
        ax = rem - ay * a.wd;
    }
    // B loads: row tid / 4, one 8-channel vector at (tid % 4) * 8 (BN * 4 threads)
    const int br = tid >> 2, bv = (tid & 3) * 8;
    const int bc = c0 + br;

    auto load_stage = [&](int stage, int kt) {
        const int tap = kt / nchunks, ci0 = (kt - tap * nchunks) * kBK;
        const int yy = ay + tap / 3 - 1, xx = ax + tap % 3 - 1;
        const bool pix_ok = ap < P && yy >= 0 && yy < a.h && xx >= 0 && xx < a.wd;
        const long pix = pix_ok ? (((long)an * a.h + yy) * a.wd + xx) : 0;
#pragma unroll
        for (int v = 0; v < 2; v++) {
            const int ci = ci0 + av + 8 * v;
            const bool ok = pix_ok && ci < a.cin;
            cp_async16(&sA[stage][ar][av + 8 * v], ok ? (const void *)(a.in + pix * a.cin + ci) : (const void *)a.in,
                       ok);
        }
        if (br < BN) {
            const int ci = ci0 + bv;
            const bool okb = bc < a.cout && ci < a.cin;
            cp_async16(&sB[stage][br][bv], okb ? (const void *)(a.wgt + ((long)bc * 9 + tap) * a.cin + ci)
                                               : (const void *)a.wgt,
                       okb);
        }
    };

    float acc[MT][NT][4];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++)
            acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.0f;

#pragma unroll
    for (int s = 0; s < kStages - 1; s++) {
        if (s < KT)
            load_stage(s, s);
        cp_async_commit();
    }
    for (int kt = 0; kt < KT; kt++) {
        cp_async_wait<kStages - 2>();
        __syncthreads();
        // refill the stage consumed in the previous iteration
        const int nk = kt + kStages - 1;
        if (nk < KT)
            load_stage(nk % kStages, nk);
        cp_async_commit();
        const int st = kt % kStages;
#pragma unroll
        for (int ks = 0; ks < kBK; ks += 16) {
            uint32_t af[MT][4], bfr[NT / 2][4];
#pragma unroll
            for (int mt = 0; mt < MT; mt++)
                ldsm_x4(smem_addr(&sA[st][wm * WM + mt * 16 + (lane & 15)][ks + (lane >> 4) * 8]), af[mt][0],
                        af[mt][1], af[mt][2], af[mt][3]);
#pragma unroll
            for (int j = 0; j < NT / 2; j++)
                ldsm_x4(smem_addr(&sB[st][wn * WN + 16 * j + (lane & 7) + ((lane >> 4) << 3)]
                                      [ks + ((lane >> 3) & 1) * 8]),
                        bfr[j][0], bfr[j][1], bfr[j][2], bfr[j][3]);
#pragma unroll
            for (int mt = 0; mt < MT; mt++)
#pragma unroll
                for (int j = 0; j < NT / 2; j++) {
                    mma_bf16(acc[mt][2 * j], af[mt][0], af[mt][1], af[mt][2], af[mt][3], bfr[j][0], bfr[j][1]);
                    mma_bf16(acc[mt][2 * j + 1], af[mt][0], af[mt][1], af[mt][2], af[mt][3], bfr[j][2], bfr[j][3]);
                }
        }
    }
    cp_async_wait<0>();
    // epilogue: c0,c1 at (row g, cols 2t, 2t+1), c2,c3 at row g + 8
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const long p = p0 + wm * WM + mt * 16 + g + half * 8;
            if (p >= P)
                continue;
#pragma unroll
            for (int j = 0; j < NT; j++) {
                const int col = c0 + wn * WN + 8 * j + 2 * t;
                if (col >= a.cout)
                    continue;
                float v0 = acc[mt][j][2 * half], v1 = acc[mt][j][2 * half + 1];
                if (a.bias) {
                    v0 += a.bias[col];
                    v1 += a.bias[col + 1];
                }
                if (a.relu) {
                    v0 = fmaxf(v0, 0.0f);
                    v1 = fmaxf(v1, 0.0f);
                }
                const long o = p * a.cout + col;
                if (a.mask) {
                    const __nv_bfloat162 m = *reinterpret_cast<const __nv_bfloat162 *>(a.mask + o);
                    if (!(__bfloat162float(m.x) > 0.0f))
                        v0 = 0.0f;
                    if (!(__bfloat162float(m.y) > 0.0f))
                        v1 = 0.0f;
                }
                if (a.out_f32)
                    *reinterpret_cast<float2 *>(reinterpret_cast<float *>(a.out) + o) = make_float2(v0, v1);
                else
                    *reinterpret_cast<__nv_bfloat162 *>(reinterpret_cast<bf16 *>(a.out) + o) =
                        __floats2bfloat162_rn(v0, v1);
            }
        }
}

__device__ __forceinline__ void unpack8(const uint4 &v, float (&f)[8])
{
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&v);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float2 t = __bfloat1622float2(h[k]);
        f[2 * k] = t.x;
        f[2 * k + 1] = t.y;
    }
}

// Weight (and bias) gradient, all nine taps in one pass over the pixels:
// dW_tap[co][ci] = sum_p dout[p][co] * in[p shifted by the tap][ci] on the
// warp-level mma.sync m16n8k16. A block owns 32 output x BN input channels and
// a set of units, a unit being a 64-pixel column of one image and a run of
// rows; warp t owns tap t and keeps its 32 x BN sums in registers over all
// units. Rows arrive by cp.async, two ahead: output row y reads input rows
// y - 1, y, y + 1 from a ring of five and its dout row, so a row of either is
// staged once for the nine taps. A tap's operand is the staged row shifted by
// a pixel or two, which ldmatrix takes as it is. The bias gradient is added up
// in FP32 by the threads that staged the values (the tensor cores cut the sums
// they accumulate off where an addition rounds: -1.3 units in the last place on
// average over rows of 64 pixels). Partial sums are added to dw and dbias with
// atomics, block b to copy b % copies of the gradients: hundreds of blocks
// adding to one value round as often, and with copies that are summed at the
// end the errors of n additions shrink from sqrt(n) to sqrt(n) / copies.
// Bound by shared-memory reads and MMA issue of the nine warps. Against one
// launch per layer that staged both tensors again for every tap (and a launch
// for the bias): 32 x 32 channels over 8 x 256 x 256 pixels 42 us, 157 + 10
// before; 80 x 32 channels 113 us, 314 + 10 before. (47 and 137 us with the bias
// as an MMA by ones and one copy of the gradients.) The weights' error against 64-bit sums of the same inputs, all layers,
// is 1.93e-6 there and 0.8e-7 at 8 x 64 x 64 (before the taps were taken together
// 4.6e-6 and 1.9e-7; with one copy 1.94e-6 and 2.1e-7), the bias's 0.2 to 0.6
// times that of the separate pass.
constexpr int kWgPx = 64, kWgM = 32, kWgThreads = 288, kWgRing = 5, kWgDRing = 3, kWgDRow = kWgM + 8;
template <int BN>
constexpr int wg_smem()
{
    return (kWgRing * (kWgPx + 2) * (BN + 8) + kWgDRing * kWgPx * kWgDRow) * (int)sizeof(bf16);
}

template <int BN>
__global__ void __launch_bounds__(kWgThreads, BN == 32 ? 3 : 2) k_conv3x3_wgrad(const bf16 *__restrict__ dout, int cout,
                                                              const bf16 *__restrict__ in, int cin, int n, int h,
                                                              int w, float *dw, float *dbias, int segs, int seg_rows,
                                                              int copies, long copy_stride)
{
    constexpr int G = BN / 8, XRow = BN + 8, XSlot = (kWgPx + 2) * XRow, DSlot = kWgPx * kWgDRow, NT = BN / 8;
    extern __shared__ __align__(16) uint8_t wg_raw[];
    bf16 *Xs = reinterpret_cast<bf16 *>(wg_raw); // [ring][pixel][BN + 8]
    bf16 *Ds = Xs + kWgRing * XSlot;             // [ring][pixel][kWgDRow]
    const int tid = threadIdx.x, tap = tid >> 5, lane = tid & 31;
    const int tiles_ci = (cin + BN - 1) / BN;
    const int co0 = ((int)blockIdx.y / tiles_ci) * kWgM, ci0 = ((int)blockIdx.y % tiles_ci) * BN;
    const int cols = (w + kWgPx - 1) / kWgPx, units = n * cols * segs;
    const int dy = tap / 3, dx = tap % 3;
    const bool bias = dbias && ci0 == 0 && tid < kWgPx * (kWgM / 8);
    const long copy = (long)((int)blockIdx.x % copies) * copy_stride;

    // A unit's copies: what a thread copies of a row is fixed within a unit
    // (element offsets within the row, -1: zeros), so a row costs it no
    // index arithmetic beyond the row's address.
    constexpr int NV = ((kWgPx + 2) * G + kWgThreads - 1) / kWgThreads;
    struct Unit {
        int u, x0, ya, nout;
        long row0; // the unit's first output row among all images' rows
        int xoff[NV], doff;
    };
    const int dpx = tid >> 2, dg = tid & 3;
    auto unit = [&](int u) {
        Unit t;
        t.u = u;
        const int sg = u % segs, c = (u / segs) % cols, nb = u / (segs * cols);
        t.x0 = c * kWgPx;
        t.ya = sg * seg_rows;
        t.nout = u < units ? min(h, t.ya + seg_rows) - t.ya : 0;
        t.row0 = (long)nb * h + t.ya;
#pragma unroll
        for (int k = 0; k < NV; k++) {
            const int v = tid + k * kWgThreads, px = v / G, g = v % G, xx = t.x0 - 1 + px, ci = ci0 + 8 * g;
            t.xoff[k] = xx >= 0 && xx < w && ci < cin ? xx * cin + ci : -1;
        }
        const int x = t.x0 + dpx, co = co0 + 8 * dg;
        t.doff = x < w && co < cout ? x * cout + co : -1;
        return t;
    };
    // rows of a unit: nout + 2 input rows; with input row r >= 2 comes the
    // dout row of output row r - 2
    auto load = [&](const Unit &t, int r, int at) {
        bf16 *xd = Xs + (at % kWgRing) * XSlot;
        const int yy = t.ya - 1 + r;
        const bool row_ok = yy >= 0 && yy < h;
        const bf16 *xrow = in + (t.row0 - 1 + r) * w * cin;
#pragma unroll
        for (int k = 0; k < NV; k++) {
            const int v = tid + k * kWgThreads;
            if (v < (kWgPx + 2) * G) {
                const bool ok = row_ok && t.xoff[k] >= 0;
                cp_async16(xd + (v / G) * XRow + 8 * (v % G), ok ? xrow + t.xoff[k] : in, ok);
            }
        }
        if (r >= 2 && tid < kWgPx * (kWgM / 8)) {
            const bool ok = t.doff >= 0;
            cp_async16(Ds + (at % kWgDRing) * DSlot + dpx * kWgDRow + 8 * dg,
                       ok ? dout + (t.row0 + r - 2) * w * cout + t.doff : dout, ok);
        }
    };
    auto advance = [&](Unit &t, int &r) {
        if (++r == t.nout + 2) {
            t = unit(t.u + (int)gridDim.x);
            r = 0;
        }
    };

    float acc[2][NT][4] = {}, sum[8] = {}; // sum: of the 8 output channels and the pixel this thread stages
    Unit cu = unit((int)blockIdx.x), lu = cu;
    int cr = 0, lr = 0;
    for (int k = 0; k < 2; k++) {
        if (lu.u < units) {
            load(lu, lr, k);
            advance(lu, lr);
        }
        cp_async_commit();
    }
    for (int at = 0; cu.u < units; at++) {
        cp_async_wait<1>(); // this thread's copies of row `at` landed
        __syncthreads();    // everyone's; and the ring slots of row at - 3 are read
        if (lu.u < units) {
            load(lu, lr, at + 2);
            advance(lu, lr);
        }
        cp_async_commit();
        if (cr >= 2) {
            const bf16 *D = Ds + (at % kWgDRing) * DSlot;
            const bf16 *X = Xs + ((at - 2 + dy) % kWgRing) * XSlot + dx * XRow;
            const int steps = (min(kWgPx, w - cu.x0) + 15) >> 4;
            for (int ks = 0; ks < 16 * steps; ks += 16) {
                // A[m = cout][k = pixel] from D[k][m], B[k = pixel][n = cin]
                // from X[k][n] (transposed loads)
                uint32_t a[2][4];
#pragma unroll
                for (int m = 0; m < 2; m++)
                    ldsm_x4_t(smem_addr(D + (ks + (lane & 7) + ((lane >> 4) << 3)) * kWgDRow + 16 * m +
                                        ((lane >> 3) & 1) * 8),
                              a[m][0], a[m][1], a[m][2], a[m][3]);
#pragma unroll
                for (int j = 0; j < NT / 2; j++) {
                    uint32_t b0, b1, b2, b3;
                    ldsm_x4_t(smem_addr(X + (ks + (lane & 7) + ((lane >> 3) & 1) * 8) * XRow + 16 * j +
                                        (lane >> 4) * 8),
                              b0, b1, b2, b3);
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        mma_bf16(acc[m][2 * j], a[m][0], a[m][1], a[m][2], a[m][3], b0, b1);
                        mma_bf16(acc[m][2 * j + 1], a[m][0], a[m][1], a[m][2], a[m][3], b2, b3);
                    }
                }
            }
            if (bias) {
                float v[8];
                unpack8(*reinterpret_cast<const uint4 *>(D + dpx * kWgDRow + 8 * dg), v);
#pragma unroll
                for (int k = 0; k < 8; k++)
                    sum[k] += v[k];
            }
        }
        advance(cu, cr);
    }
    cp_async_wait<0>();
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const int co = co0 + 16 * m + g + half * 8;
            if (co >= cout)
                continue;
#pragma unroll
            for (int j = 0; j < NT; j++) {
                const int ci = ci0 + 8 * j + 2 * t;
                if (ci < cin)
                    atomicAdd(reinterpret_cast<float2 *>(dw + copy + ((long)co * 9 + tap) * cin + ci),
                              make_float2(acc[m][j][2 * half], acc[m][j][2 * half + 1]));
            }
        }
    if (!dbias || ci0 != 0)
        return;
    // bias: over a warp's 8 pixels by halves, then the 8 warps' sums
    __syncthreads(); // the staged rows are read
    float(*red)[kWgM] = reinterpret_cast<float(*)[kWgM]>(wg_raw);
    if (tid < kWgPx * (kWgM / 8)) {
#pragma unroll
        for (int k = 0; k < 8; k++) {
#pragma unroll
            for (int o = 4; o < 32; o <<= 1)
                sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
            if (lane < 4)
                red[tid >> 5][8 * lane + k] = sum[k];
        }
    }
    __syncthreads();
    if (tid < kWgM && co0 + tid < cout) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; k++)
            v[k] = red[k][tid];
        atomicAdd(dbias + copy + co0 + tid, ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])));
    }
}

// The layout kernels below move 8 channels (16 bytes) per thread: channel
// counts are multiples of 8, so every access is one aligned 128-bit load or
// store and a warp covers 512 consecutive bytes. Index arithmetic is 32-bit
// (element counts stay below 2^31; the host checks).
__device__ __forceinline__ uint4 pack8(const float (&f)[8])
{
    uint4 v;
    __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&v);
#pragma unroll
    for (int k = 0; k < 4; k++)
        h[k] = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
    return v;
}

__device__ __forceinline__ uint4 ld16(const bf16 *p) { return __ldg(reinterpret_cast<const uint4 *>(p)); }
__device__ __forceinline__ void st16(bf16 *p, const uint4 &v) { *reinterpret_cast<uint4 *>(p) = v; }

// dbias[c] += sum_p dout[p][c]: a thread sums 8 channels (one 16-byte load
// per pixel) over a strided set of pixels, the block reduces its pixel lanes
// in shared memory and adds one value per channel.
constexpr int kBiasThreads = 256;
__global__ void __launch_bounds__(kBiasThreads) k_bias_grad(const bf16 *dout, int cout, long P, float *dbias)
{
    __shared__ float red[kBiasThreads * 8];
    const int G = cout >> 3, lanes = kBiasThreads / G;
    const int g = threadIdx.x % G, r = threadIdx.x / G;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (r < lanes) {
        for (long p = (long)blockIdx.x * lanes + r; p < P; p += (long)gridDim.x * lanes) {
            float v[8];
            unpack8(ld16(dout + p * cout + 8 * g), v);
#pragma unroll
            for (int k = 0; k < 8; k++)
                acc[k] += v[k];
        }
    }
#pragma unroll
    for (int k = 0; k < 8; k++)
        red[threadIdx.x * 8 + k] = acc[k];
    __syncthreads();
    for (int c = threadIdx.x; c < cout; c += kBiasThreads) {
        float sum = 0.0f;
        for (int q = 0; q < lanes; q++)
            sum += red[(q * G + (c >> 3)) * 8 + (c & 7)];
        atomicAdd(dbias + c, sum);
    }
}

// bf16 copies of all layers' weights, w16 as they are and wt16 transposed for
// the input gradients (wt[ci][8 - tap][co] = w[co][tap][ci]), in one launch.
__global__ void k_prepare_weights(const float *params, WeightTable t, bf16 *w16, bf16 *wt16)
{
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < t.start[t.layers]; i += gridDim.x * blockDim.x) {
        int l = 0;
        while (i >= t.start[l + 1])
            l++;
        const unsigned k = i - t.start[l], cin = t.cin[l], cout = t.cout[l];
        const bf16 v = __float2bfloat16_rn(params[t.param[l] + k]);
        w16[i] = v;
        const unsigned ci = k % cin, tap = (k / cin) % 9, co = k / (9 * cin);
        wt16[t.start[l] + (ci * 9 + (8 - tap)) * cout + co] = v;
    }
}

__global__ void k_pack_features(const float4 *rad, const float4 *alb, const float4 *nrm, bf16 *x, int npix)
{
    pdl_wait();
    pdl_start();
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
        const float4 r = rad[p], a = alb[p], q = nrm[p];
        __align__(16) bf16 v[16];
        v[0] = __float2bfloat16_rn(log1pf(fmaxf(r.x, 0.0f)));
        v[1] = __float2bfloat16_rn(log1pf(fmaxf(r.y, 0.0f)));
        v[2] = __float2bfloat16_rn(log1pf(fmaxf(r.z, 0.0f)));
        v[3] = __float2bfloat16_rn(a.x);
        v[4] = __float2bfloat16_rn(a.y);
        v[5] = __float2bfloat16_rn(a.z);
        v[6] = __float2bfloat16_rn(q.x);
        v[7] = __float2bfloat16_rn(q.y);
        v[8] = __float2bfloat16_rn(q.z);
#pragma unroll
        for (int k = 9; k < 16; k++)
            v[k] = __float2bfloat16_rn(0.0f);
        uint4 *dst = reinterpret_cast<uint4 *>(x + (long)p * 16);
        dst[0] = *reinterpret_cast<const uint4 *>(&v[0]);
        dst[1] = *reinterpret_cast<const uint4 *>(&v[8]);
    }
}

__global__ void k_avgpool2(const bf16 *in, bf16 *out, int n, int h, int w, int c)
{
    pdl_wait();
    pdl_start();
    const unsigned ho = h / 2, wo = w / 2, g = c / 8;
    const unsigned total = (unsigned)n * ho * wo * g;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const unsigned cg = i % g, q = i / g;
        const unsigned x = q % wo, y = (q / wo) % ho, b = q / (wo * ho);
        const size_t base = (((size_t)b * h + 2 * y) * w + 2 * x) * c + 8 * cg, row = (size_t)w * c;
        float a[8], t[8];
        unpack8(ld16(in + base), a);
        unpack8(ld16(in + base + c), t);
#pragma unroll
        for (int k = 0; k < 8; k++)
            a[k] += t[k];
        unpack8(ld16(in + base + row), t);
#pragma unroll
        for (int k = 0; k < 8; k++)
            a[k] += t[k];
        unpack8(ld16(in + base + row + c), t);
#pragma unroll
        for (int k = 0; k < 8; k++)
            a[k] = 0.25f * (a[k] + t[k]);
        st16(out + (size_t)i * 8, pack8(a));
    }
}

__global__ void k_upcat(const bf16 *coarse, int cc, const bf16 *skip, int cs, bf16 *out, int n, int h, int w)
{
    pdl_wait();
    pdl_start();
    const unsigned gc = cc / 8, gt = (cc + cs) / 8;
    const unsigned total = (unsigned)n * h * w * gt;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const unsigned cg = i % gt, p = i / gt;
        uint4 v;
        if (cg < gc) {
            const unsigned x = p % w, y = (p / w) % h, b = p / (w * h);
            v = ld16(coarse + (((size_t)b * (h / 2) + y / 2) * (w / 2) + x / 2) * cc + 8 * cg);
        } else {
            v = ld16(skip + (size_t)p * cs + 8 * (cg - gc));
        }
        st16(out + (size_t)i * 8, v);
    }
}

__global__ void k_upcat_backward_coarse(const bf16 *dcat, int cc, int cs, bf16 *dcoarse, int n, int h, int w)
{
    pdl_wait();
    pdl_start();
    const int ct = cc + cs;
    const unsigned ho = h / 2, wo = w / 2, g = cc / 8;
    const unsigned total = (unsigned)n * ho * wo * g;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const unsigned cg = i % g, q = i / g;
        const unsigned x = q % wo, y = (q / wo) % ho, b = q / (wo * ho);
        const size_t base = (((size_t)b * h + 2 * y) * w + 2 * x) * ct + 8 * cg, row = (size_t)w * ct;
        float a[8], t[8];
        unpack8(ld16(dcat + base), a);
        unpack8(ld16(dcat + base + ct), t);
#pragma unroll
        for (int k = 0; k < 8; k++)
            a[k] += t[k];
        unpack8(ld16(dcat + base + row), t);
#pragma unroll
        for (int k = 0; k < 8; k++)
            a[k] += t[k];
        unpack8(ld16(dcat + base + row + ct), t);
#pragma unroll
        for (int k = 0; k < 8; k++)
            a[k] += t[k];
        st16(dcoarse + (size_t)i * 8, pack8(a));
    }
}

__global__ void k_upcat_backward_skip(const bf16 *dcat, int cc, int cs, bf16 *dskip, unsigned npix)
{
    pdl_wait();
    pdl_start();
    const unsigned g = cs / 8, gt = (cc + cs) / 8, gc = cc / 8;
    const unsigned total = npix * g;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const unsigned cg = i % g, p = i / g;
        st16(dskip + (size_t)i * 8, ld16(dcat + ((size_t)p * gt + gc + cg) * 8));
    }
}

__global__ void k_pool_backward_combine(const bf16 *dskip, const bf16 *dpooled, const bf16 *e, bf16 *de, int n, int h,
                                        int w, int c)
{
    pdl_wait();
    pdl_start();
    const unsigned g = c / 8;
    const unsigned total = (unsigned)n * h * w * g;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const unsigned cg = i % g, p = i / g;
        const unsigned x = p % w, y = (p / w) % h, b = p / (w * h);
        float v[8], t[8], m[8];
        unpack8(ld16(dpooled + (((size_t)b * (h / 2) + y / 2) * (w / 2) + x / 2) * c + 8 * cg), v);
#pragma unroll
        for (int k = 0; k < 8; k++)
            v[k] *= 0.25f;
        if (dskip) {
            unpack8(ld16(dskip + (size_t)i * 8), t);
#pragma unroll
            for (int k = 0; k < 8; k++)
                v[k] += t[k];
        }
        unpack8(ld16(e + (size_t)i * 8), m);
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (!(m[k] > 0.0f))
                v[k] = 0.0f;
        st16(de + (size_t)i * 8, pack8(v));
    }
}

// Loss and its gradient from the output layer (`cout` f32 channels, the first 3
// used) and the target frame in one pass over the pixels.
__global__ void __launch_bounds__(256) k_l1_loss(const float *out, int cout, const float4 *target, bf16 *dout,
                                                 float *loss_sum, int npix)
{
    __shared__ float part[8];
    float local = 0.0f;
    const float scale = 1.0f / (3.0f * (float)npix);
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
        const float4 y = *reinterpret_cast<const float4 *>(out + (long)p * cout);
        const float4 v = target[p];
        const float t[3] = {log1pf(fmaxf(v.x, 0.0f)), log1pf(fmaxf(v.y, 0.0f)), log1pf(fmaxf(v.z, 0.0f))};
        const float d[3] = {y.x - t[0], y.y - t[1], y.z - t[2]};
        float g[8] = {};
#pragma unroll
        for (int c = 0; c < 3; c++) {
            local += fabsf(d[c]);
            g[c] = d[c] > 0.0f ? scale : (d[c] < 0.0f ? -scale : 0.0f);
        }
        bf16 *o = dout + (long)p * cout;
        st16(o, pack8(g));
        for (int c = 8; c < cout; c += 8)
            st16(o + c, make_uint4(0u, 0u, 0u, 0u));
    }
    for (int o = 16; o > 0; o >>= 1)
        local += __shfl_xor_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0)
        part[threadIdx.x >> 5] = local;
    __syncthreads();
    if (threadIdx.x == 0) {
        float sum = 0.0f;
        for (int k = 0; k < 8; k++)
            sum += part[k];
        atomicAdd(loss_sum, sum);
    }
}

// The sum of a gradient's copies (see k_conv3x3_wgrad).
__device__ __forceinline__ float sum_copies(const float *g, size_t stride)
{
    static_assert(kGradCopies == 4, "summed by halves");
    return (g[0] + g[stride]) + (g[2 * stride] + g[3 * stride]);
}
__global__ void k_sum_grads(const float *g, size_t stride, float *sum, size_t n)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        sum[i] = sum_copies(g + i, stride);
}

__global__ void k_adam(float *p, const float *g, size_t stride, float *m, float *v, size_t n, float lr, float b1,
                       float b2, float eps, float c1, float c2)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float gi = sum_copies(g + i, stride);
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

__global__ void k_unpack_output(const float *y, int cout, float4 *out, int npix)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
        const float *v = y + (long)p * cout;
        out[p] = make_float4(expm1f(fmaxf(v[0], 0.0f)), expm1f(fmaxf(v[1], 0.0f)), expm1f(fmaxf(v[2], 0.0f)), 1.0f);
    }
}

int grid_for(long n, int block = 256)
{
    return (int)std::max<long>(1, std::min<long>((n + block - 1) / block, 152L * 16));
}


// ---------------------------------------------------------------------------
// tcgen05 convolution (5th-generation tensor cores, accumulator in TMEM).
//
// CTA = kTcThreads threads, tile = 128 consecutive pixels of one image row (UMMA
// M = 128: pixel i of the tile is TMEM lane i) x all output channels (N =
// cout <= 256, one accumulator of N f32 columns). For each 32-channel chunk
// of the input the CTA stages a halo of 3 rows x 130 pixels once in shared
// memory; every one of the 9 taps is then an MMA over a shifted view of it
// (the operand descriptor starts 16 bytes per pixel and one halo row further),
// so the input is read once per chunk instead of once per tap. Layout, K-major
// without swizzle: for each halo row and 8-channel group the 130 pixels are
// consecutive 16-byte rows, so 8 consecutive pixels form a core matrix (SBO
// 128 B between pixel groups, LBO 130 x 16 B between channel groups). The
// weights of one (chunk, tap) step go to one of 4 stages. One thread issues
// the MMAs (two m128 nN k16 per step) and commits each step to its stage's
// mbarrier; refills wait on the mbarrier of the step two back (MMAs complete
// in issue order). Waits are bounded by the global timer; on a timeout the
// kernel records an error, stops issuing and still frees its TMEM.
constexpr int kTcM = 128, kTcBK = 32, kTcKC = kTcBK / 8, kTcBStages = 4, kTcHaloPx = kTcM + 2;
constexpr int kTcHaloRow = kTcKC * kTcHaloPx * 16;  // one halo row: 4 channel groups x 130 pixels x 16 B
constexpr int kTcHaloAlloc = 25088;                 // rounded up to 1 KB multiples
constexpr unsigned long long kTcWaitNs = 2000000000ull;
// threads of the per-tile kernels: what bounds a chunk is the index arithmetic
// of its copies, so 16 warps share them (and the drain): 160 to 64 channels at
// 960 x 540 274 us with 4 warps, 220 us with 16
constexpr int kTcThreads = 512;

__host__ __device__ constexpr int tc_smem_bytes(int N) { return 2 * kTcHaloAlloc + kTcBStages * N * kTcBK * 2; }

__device__ __forceinline__ unsigned long long globaltimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity)
{
    const unsigned long long t0 = globaltimer();
    for (;;) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}\n"
                     : "=r"(done)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (done)
            return true;
        if (globaltimer() - t0 > kTcWaitNs)
            return false;
    }
}

// The MMAs are issued by one elected lane, but by code that the whole warp runs
// with the same values: descriptors, instruction word and accumulator address
// of a tcgen05.mma are uniform registers, and code of a single lane moves each
// of them there for every MMA. Measured, MMAs of M 128, K 16 one after the
// other: 55 clocks each from a lane's own code whatever N, 32 + N / 4 (the
// operands' shared-memory reads) from the warp's.
__device__ __forceinline__ uint32_t elect_one()
{
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(e));
    return e;
}
__device__ __forceinline__ void umma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate,
                                     uint32_t elected)
{
    asm volatile("{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t"
                 "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
                 "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate), "r"(elected));
}

__device__ __forceinline__ void umma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar));
}

// shared-memory matrix descriptor: start, LBO, SBO (16-byte units),
// version 1, no swizzle
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                 "%14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15])
                 : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;");
}

__device__ __forceinline__ void tmem_ld8_issue(uint32_t addr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr));
}

__device__ __forceinline__ void tmem_ld16_issue(uint32_t addr, uint32_t (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                 "%14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15])
                 : "r"(addr));
}
// Every use of the loaded values depends on a value that passes through here.
__device__ __forceinline__ void tmem_wait8(uint32_t *r)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])::
                     "memory");
}

// 16 channels of a row accumulator of `nacc` (1, 2 or 4) partial sums, ncol
// columns apart, added in their order: as many loads in flight before a wait
// as fit 32 registers.
template <int nacc>
__device__ __forceinline__ void tmem_sum16(uint32_t addr, uint32_t ncol, uint32_t (&r)[16])
{
    static_assert(nacc == 1 || nacc == 2 || nacc == 4, "partial sums");
    if constexpr (nacc <= 2) {
        uint32_t t[16];
        tmem_ld16_issue(addr, r);
        if constexpr (nacc > 1)
            tmem_ld16_issue(addr + ncol, t);
        tmem_wait8(r);
        tmem_wait8(r + 8);
        if constexpr (nacc > 1)
#pragma unroll
            for (int k = 0; k < 16; k++)
                r[k] = __float_as_uint(__uint_as_float(r[k]) + __uint_as_float(t[k]));
    } else {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t t[3][8];
            tmem_ld8_issue(addr + 8 * h, *reinterpret_cast<uint32_t(*)[8]>(r + 8 * h));
#pragma unroll
            for (int q = 1; q < 4; q++)
                tmem_ld8_issue(addr + 8 * h + q * ncol, t[q - 1]);
            tmem_wait8(r + 8 * h);
#pragma unroll
            for (int k = 0; k < 8; k++) {
                float v = __uint_as_float(r[8 * h + k]) + __uint_as_float(t[0][k]);
                v += __uint_as_float(t[1][k]);
                v += __uint_as_float(t[2][k]);
                r[8 * h + k] = __float_as_uint(v);
            }
        }
    }
}

// 32 bytes per lane in one instruction (sm_100 and later): a whole sector. The
// operand reads of the MMAs take the same path, so what the epilogue saves
// there the MMAs get.
__device__ __forceinline__ void st32(void *p, const uint32_t (&v)[8])
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void ld32(const void *p, uint32_t (&v)[8])
{
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(p));
}

// Epilogue of one pixel row x 16 channels: bias, ReLU, mask, store (bf16, or
// f32 for the output layer). Channel counts are multiples of 16 and the arrays
// 32-byte aligned, so 16 bf16 channels are one sector.
struct Bias16 {
    float4 b[4];
};
__device__ __forceinline__ void load_bias(const ConvArgs &a, int c, Bias16 &b)
{
    if (a.bias && c < a.cout)
#pragma unroll
        for (int k = 0; k < 4; k++)
            b.b[k] = __ldg(reinterpret_cast<const float4 *>(a.bias + c) + k);
}
// (h: the 16 channels as stored, where they are stored as bf16.)
__device__ __forceinline__ void store_row16(const ConvArgs &a, long p, int c, const uint32_t (&r)[16], const Bias16 &b,
                                            uint32_t (&h)[8])
{
    float v[16];
#pragma unroll
    for (int k = 0; k < 16; k++)
        v[k] = __uint_as_float(r[k]);
    if (a.bias) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[4 * k] += b.b[k].x;
            v[4 * k + 1] += b.b[k].y;
            v[4 * k + 2] += b.b[k].z;
            v[4 * k + 3] += b.b[k].w;
        }
    }
    if (a.relu) {
#pragma unroll
        for (int k = 0; k < 16; k++)
            v[k] = fmaxf(v[k], 0.0f);
    }
    if (a.rgba) {
        // the output unpacking of the frame, in the epilogue (k_unpack_output)
        if (c == 0)
            a.rgba[p] = make_float4(expm1f(fmaxf(v[0], 0.0f)), expm1f(fmaxf(v[1], 0.0f)), expm1f(fmaxf(v[2], 0.0f)),
                                    1.0f);
        return;
    }
    const long o = p * a.cout + c;
    if (a.mask) {
        uint32_t m[8];
        ld32(a.mask + o, m);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&m[k]));
            if (!(f.x > 0.0f))
                v[2 * k] = 0.0f;
            if (!(f.y > 0.0f))
                v[2 * k + 1] = 0.0f;
        }
    }
    if (a.out_f32) {
        float4 *dst = reinterpret_cast<float4 *>(reinterpret_cast<float *>(a.out) + o);
#pragma unroll
        for (int k = 0; k < 4; k++)
            dst[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    } else {
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
            h[k] = *reinterpret_cast<const uint32_t *>(&b);
        }
        st32(reinterpret_cast<bf16 *>(a.out) + o, h);
    }
}
__device__ __forceinline__ void store_row16(const ConvArgs &a, long p, int c, const uint32_t (&r)[16], const Bias16 &b)
{
    uint32_t h[8];
    store_row16(a, p, c, r, b, h);
}

// 2x2 averages of 16 channels, of the row just stored (h) and the one above it,
// which the same thread stored: the lanes of an even and an odd pixel exchange
// halves, and each averages eight channels in the order of k_avgpool2. The
// whole warp calls it; `ok`: the lane's pixel and channels exist.
__device__ __forceinline__ void pool_row16(const ConvArgs &a, long p, long pool_p, int c, const uint32_t (&h)[8], bool ok)
{
    uint32_t up[8] = {};
    if (ok)
        ld32(reinterpret_cast<const bf16 *>(a.out) + (p - a.wd) * a.cout + c, up);
    const bool odd = threadIdx.x & 1;
    uint4 res;
    uint32_t *out = reinterpret_cast<uint32_t *>(&res);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t mu = odd ? up[4 + k] : up[k], mc = odd ? h[4 + k] : h[k];
        const uint32_t ou = __shfl_xor_sync(0xffffffffu, odd ? up[k] : up[4 + k], 1);
        const uint32_t oc = __shfl_xor_sync(0xffffffffu, odd ? h[k] : h[4 + k], 1);
        auto f = [](uint32_t w) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&w)); };
        const float2 f00 = f(odd ? ou : mu), f01 = f(odd ? mu : ou), f10 = f(odd ? oc : mc), f11 = f(odd ? mc : oc);
        const __nv_bfloat162 b = __floats2bfloat162_rn(0.25f * (((f00.x + f01.x) + f10.x) + f11.x),
                                                       0.25f * (((f00.y + f01.y) + f10.y) + f11.y));
        out[k] = *reinterpret_cast<const uint32_t *>(&b);
    }
    if (ok)
        *reinterpret_cast<uint4 *>(a.pool + pool_p * a.cout + c + (odd ? 8 : 0)) = res;
}

__global__ void __launch_bounds__(kTcThreads) k_conv3x3_tc(ConvArgs a, int ncols, uint32_t *err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint32_t tmem_holder;
    __shared__ __align__(8) uint64_t mbar[kTcBStages];
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int tiles_x = (a.wd + kTcM - 1) / kTcM;
    const int tx = blockIdx.x % tiles_x;
    const int y = (blockIdx.x / tiles_x) % a.h;
    const int nb = blockIdx.x / (tiles_x * a.h);
    const int x0 = tx * kTcM;
    const int N = (a.cout + 15) & ~15;
    const int bstage_bytes = N * kTcBK * 2;
    const int nchunks = (a.cin + kTcBK - 1) / kTcBK;
    const int S = 9 * nchunks;
    uint8_t *halo[2] = {smem, smem + kTcHaloAlloc};
    uint8_t *bst = smem + 2 * kTcHaloAlloc;
    const uint32_t sbase = smem_addr(smem);

    if (tid == 0) {
        for (int st = 0; st < kTcBStages; st++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&mbar[st])));
        abort_flag = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_holder)),
                     "r"(ncols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    pdl_wait();
    pdl_start();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_holder, 0), elected = elect_one();
    // D f32, A/B bf16, both K-major, N >> 3, M >> 4
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kTcM >> 4) << 24);

    auto load_step = [&](int st) {
        const int c = st / 9, tap = st - c * 9, ci0 = c * kTcBK;
        if (tap == 0) {
            // halo of chunk c: 3 rows x 130 pixels x 4 channel groups
            uint8_t *h = halo[c & 1];
            for (int i = tid; i < 3 * kTcKC * kTcHaloPx; i += kTcThreads) {
                const int px = i % kTcHaloPx, kc = (i / kTcHaloPx) % kTcKC, hr = i / (kTcHaloPx * kTcKC);
                const int yy = y + hr - 1, xx = x0 - 1 + px, ci = ci0 + 8 * kc;
                const bool ok = yy >= 0 && yy < a.h && xx >= 0 && xx < a.wd && ci < a.cin;
                const bf16 *src = ok ? a.in + (((long)nb * a.h + yy) * a.wd + xx) * a.cin + ci : a.in;
                cp_async16(h + ((hr * kTcKC + kc) * kTcHaloPx + px) * 16, src, ok);
            }
        }
        uint8_t *b = bst + (st % kTcBStages) * bstage_bytes;
        for (int i = tid; i < N * kTcKC; i += kTcThreads) {
            const int n = i / kTcKC, kc = i - n * kTcKC, ci = ci0 + 8 * kc;
            const bool ok = n < a.cout && ci < a.cin;
            const bf16 *src = ok ? a.wgt + ((long)n * 9 + tap) * a.cin + ci : a.wgt;
            cp_async16(b + (n >> 3) * (kTcKC * 128) + kc * 128 + (n & 7) * 16, src, ok);
        }
    };

    // prologue: steps 0 and 1
    for (int st = 0; st < 2; st++) {
        if (st < S)
            load_step(st);
        cp_async_commit();
    }
    for (int st = 0; st < S; st++) {
        cp_async_wait<1>(); // this thread's copies of step st landed
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (abort_flag)
            break;
        if (warp == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;");
            const int c = st / 9, tap = st - c * 9, dy = tap / 3, dx = tap % 3;
            const uint32_t a_addr = sbase + (c & 1) * kTcHaloAlloc + dy * kTcHaloRow + dx * 16;
            const uint32_t b_addr = sbase + 2 * kTcHaloAlloc + (st % kTcBStages) * bstage_bytes;
#pragma unroll
            for (int j = 0; j < kTcBK / 16; j++)
                umma(tmem, umma_desc(a_addr + j * 2 * kTcHaloPx * 16, kTcHaloPx * 16, 128),
                     umma_desc(b_addr + j * 2 * 128, 128, kTcKC * 128), idesc, st > 0 || j > 0, elected);
            if (elected)
                umma_commit(smem_addr(&mbar[st % kTcBStages]));
        }
        // step st + 2 reuses the weight stage of step st - 2 and, at a chunk
        // start, the halo of chunk (st + 2) / 9 - 2: both done once step st - 2
        // is (in-order completion)
        const int nx = st + 2;
        if (nx < S) {
            if (st >= 2) {
                const int prev = st - 2;
                if (!mbar_wait(smem_addr(&mbar[prev % kTcBStages]), (prev / kTcBStages) & 1))
                    atomicOr(&abort_flag, 1);
            }
            load_step(nx);
        }
        cp_async_commit();
    }
    cp_async_wait<0>();
    if (!abort_flag && S > 0) {
        const int last = S - 1;
        if (!mbar_wait(smem_addr(&mbar[last % kTcBStages]), (last / kTcBStages) & 1))
            atomicOr(&abort_flag, 1);
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (!abort_flag) {
        const int q = warp & 3, x = x0 + q * 32 + lane;
        const long p = ((long)nb * a.h + y) * a.wd + x;
        for (int c = 16 * (warp >> 2); c < N; c += 16 * (kTcThreads / 128)) {
            uint32_t r[16];
            Bias16 bias;
            load_bias(a, c, bias);
            tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c, r);
            if (x >= a.wd || c >= a.cout)
                continue;
            store_row16(a, p, c, r, bias);
        }
    } else if (tid == 0) {
        atomicOr(err, 1u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols));
}

// Chunk-batched variant for N <= 128 output channels: a stage holds the halo
// and the weights of all 9 taps of one 32-channel chunk, so a chunk is one
// barrier and 18 back-to-back MMAs; two stages alternate (the next chunk's
// copies overlap this chunk's MMAs). Same layouts, waits and error handling
// as k_conv3x3_tc.

// one stage when the layer has a single chunk, else two
// halo of `rows` output rows: rows + 2 halo rows, rounded up to 1 KB
__host__ __device__ constexpr int tc_chunk_halo_bytes(int rows) { return ((rows + 2) * kTcHaloRow + 1023) / 1024 * 1024; }

__host__ __device__ constexpr int tc_chunk_smem_bytes(int N, int nchunks, int rows)
{
    return (nchunks > 1 ? 2 : 1) * (tc_chunk_halo_bytes(rows) + 9 * N * kTcBK * 2);
}

// output rows per CTA of the chunk kernel: the chunk's weights are staged once
// for all of them (4 rows up to 64 output channels, else 2: two stages fit)
inline int tc_chunk_rows(int N) { return N <= 64 ? 4 : 2; }

__global__ void __launch_bounds__(kTcThreads) k_conv3x3_tc_chunk(ConvArgs a, int ncols, int rows, int ntile,
                                                                 uint32_t *err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint32_t tmem_holder;
    __shared__ __align__(8) uint64_t mbar[2];
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int tiles_x = (a.wd + kTcM - 1) / kTcM;
    const int yblocks = (a.h + rows - 1) / rows;
    const int tx = blockIdx.x % tiles_x;
    const int y0 = (blockIdx.x / tiles_x) % yblocks * rows;
    const int nb = blockIdx.x / (tiles_x * yblocks);
    const int x0 = tx * kTcM;
    const int N = ntile, n0 = (int)blockIdx.y * ntile; // this CTA's output channels
    const int tap_bytes = N * kTcBK * 2;
    const int halo_alloc = tc_chunk_halo_bytes(rows);
    const int stage_bytes = halo_alloc + 9 * tap_bytes;
    const int nchunks = (a.cin + kTcBK - 1) / kTcBK;
    const uint32_t sbase = smem_addr(smem);

    if (tid == 0) {
        for (int st = 0; st < 2; st++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&mbar[st])));
        abort_flag = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_holder)),
                     "r"(ncols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_holder, 0), elected = elect_one();
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kTcM >> 4) << 24);

    auto load_halo = [&](int c) {
        uint8_t *h = smem + (c & 1) * stage_bytes;
        const int ci0 = c * kTcBK;
        for (int i = tid; i < (rows + 2) * kTcKC * kTcHaloPx; i += kTcThreads) {
            const int px = i % kTcHaloPx, kc = (i / kTcHaloPx) % kTcKC, hr = i / (kTcHaloPx * kTcKC);
            const int yy = y0 + hr - 1, xx = x0 - 1 + px, ci = ci0 + 8 * kc;
            const bool ok = yy >= 0 && yy < a.h && xx >= 0 && xx < a.wd && ci < a.cin;
            const bf16 *src = ok ? a.in + (((long)nb * a.h + yy) * a.wd + xx) * a.cin + ci : a.in;
            cp_async16(h + ((hr * kTcKC + kc) * kTcHaloPx + px) * 16, src, ok);
        }
    };
    auto load_weights = [&](int c) {
        uint8_t *bw = smem + (c & 1) * stage_bytes + halo_alloc;
        const int ci0 = c * kTcBK;
        for (int i = tid; i < 9 * N * kTcKC; i += kTcThreads) {
            const int kc = i % kTcKC, n = (i / kTcKC) % N, tap = i / (kTcKC * N), ci = ci0 + 8 * kc;
            const bool ok = n0 + n < a.cout && ci < a.cin;
            const bf16 *src = ok ? a.wgt + ((long)(n0 + n) * 9 + tap) * a.cin + ci : a.wgt;
            cp_async16(bw + tap * tap_bytes + (n >> 3) * (kTcKC * 128) + kc * 128 + (n & 7) * 16, src, ok);
        }
    };

    load_weights(0);
    pdl_wait();
    pdl_start();
    load_halo(0);
    cp_async_commit();
    for (int c = 0; c < nchunks; c++) {
        cp_async_wait<0>(); // this thread's copies of chunk c landed
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (abort_flag)
            break;
        if (warp == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t h_addr = sbase + (c & 1) * stage_bytes, b_addr = h_addr + halo_alloc;
            // output row r of the block: accumulator r; the chunk's weights
            // serve all rows
            for (int r = 0; r < rows; r++) {
#pragma unroll
                for (int j = 0; j < kTcBK / 16; j++) {
#pragma unroll
                    for (int tap = 0; tap < 9; tap++) {
                        const int dy = tap / 3, dx = tap % 3;
                        umma(tmem + (uint32_t)(r * N),
                             umma_desc(h_addr + (r + dy) * kTcHaloRow + dx * 16 + j * 2 * kTcHaloPx * 16,
                                       kTcHaloPx * 16, 128),
                             umma_desc(b_addr + tap * tap_bytes + j * 2 * 128, 128, kTcKC * 128), idesc,
                             c > 0 || j > 0 || tap > 0, elected);
                    }
                }
            }
            if (elected)
                umma_commit(smem_addr(&mbar[c & 1]));
        }
        // chunk c + 1 goes to the stage chunk c - 1 was read from; the MMAs of
        // chunk c are queued behind it meanwhile
        if (c + 1 < nchunks) {
            if (c >= 1 && !mbar_wait(smem_addr(&mbar[(c - 1) & 1]), ((c - 1) >> 1) & 1))
                atomicOr(&abort_flag, 1);
            load_weights(c + 1);
            load_halo(c + 1);
        }
        cp_async_commit();
    }
    cp_async_wait<0>();
    if (!abort_flag && nchunks > 0) {
        const int last = nchunks - 1;
        if (!mbar_wait(smem_addr(&mbar[last & 1]), (last >> 1) & 1))
            atomicOr(&abort_flag, 1);
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (!abort_flag) {
        // warps w, w + 4, ... read the same 32 pixels, each its share of
        // (row, 16 channels)
        const int quarter = warp & 3, x = x0 + quarter * 32 + lane, groups = N / 16;
        for (int k = warp >> 2; k < rows * groups; k += kTcThreads / 128) {
            const int rr = k / groups, c = 16 * (k - rr * groups);
            if (y0 + rr >= a.h)
                break;
            const long p = ((long)nb * a.h + y0 + rr) * a.wd + x;
            const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(rr * N);
            uint32_t r[16];
            Bias16 bias;
            load_bias(a, n0 + c, bias);
            tmem_sum16<1>(lane_base + (uint32_t)c, 0u, r);
            if (x < a.wd && n0 + c < a.cout)
                store_row16(a, p, n0 + c, r, bias);
        }
    } else if (tid == 0) {
        atomicOr(err, 1u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols));
}

// Strip kernel: TMA-fed, weights resident, persistent over runs of rows.
//
// A unit of work is a 128-pixel-wide column of one image and a run of
// consecutive output rows (a segment); a CTA runs its units one after the
// other. The weights of the whole layer (9 x N x cin bf16) are loaded once and
// stay in shared memory. Input rows arrive by TMA into a ring of `ring` slots,
// each one halo row of 130 pixels x cin channels; the tensor map zero-fills
// pixels and rows outside the image, which is the convolution's zero padding.
// Output row i of a segment reads halo rows i, i + 1, i + 2, so every output
// row needs one new halo row (the input is read once, not three times).
// Slot layout (K-major, 32-byte swizzle): per 16 channels a plane of kStPlane
// bytes in which the 130 pixels are consecutive 32-byte rows (one TMA box of
// 16 channels x 130 pixels; boxes of 8 channels without swizzle copied 16
// bytes a pixel and took twice the requests); a tap (dy, dx) of output row i
// is the operand starting at slot(i + dy) + 32 dx (256 B between 8-pixel
// groups; the swizzle follows address bits, so a start inside a group of 8
// reads the pixels where they were stored). What bounds it: an MMA of M = 128,
// K = 16 and N <= 64 takes 32 + N / 4 clocks, the time to read its pixels from
// shared memory, if a whole warp reaches it and one elected lane issues it (55
// clocks when the code is one lane's own); layers with few channels are bound
// by memory instead. Two TMEM accumulators alternate between output
// rows; each holds `nacc` partial sums (taps spread over independent MMA
// chains) that the drain adds. The roles (k_conv3x3_strip below) are warp
// specialised: a producer warp, an MMA warp and four drain warps, linked by
// mbarriers only. Halo rows and output rows are counted over the CTA's whole
// run, so slot and accumulator phases carry across units. Every wait is
// bounded by the global timer; on a timeout the kernel records an error, the
// other roles stop at their next wait, copies and MMAs in flight are waited
// for (bounded) and the TMEM is freed.
constexpr int kStPlane = 4352; // 130 pixels x 32 B, padded to a multiple of the swizzle's 256 B
constexpr int kStHaloPx = kTcM + 2;
// byte of channel group g (8 channels) of pixel px in a ring slot: the 32-byte
// swizzle exchanges the two halves of a pixel where address bit 7 is set
__device__ __forceinline__ int st_chunk(int g, int px)
{
    return (g >> 1) * kStPlane + px * 32 + (((g & 1) ^ ((px >> 2) & 1)) << 4);
}
// at least the three halo rows one output row reads; three slots (no row
// prefetched ahead) are taken when they let more CTAs share an SM
constexpr int kStMaxRing = 8, kStMinRing = 3;

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}

// Bounded wait that also gives up once another role has aborted.
__device__ __forceinline__ bool mbar_wait_role(uint32_t bar, uint32_t parity, const volatile int *abort_flag)
{
    const unsigned long long t0 = globaltimer();
    for (;;) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}\n"
                     : "=r"(done)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (done)
            return true;
        if (*abort_flag || globaltimer() - t0 > kTcWaitNs)
            return false;
    }
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Warps 0-3 drain accumulators, and with two drain sets warps 6-9 too (TMEM
// lane quarter = warp % 4; the sets share a row's channels), warp 4 loads halo
// rows by TMA, warp 5 issues the MMAs, the last four warps (launched for it
// only) fill the upsampled channels of a fused upsample + concat input
// (a.coarse). The warps other than 4 and 5 first copy the weights, which the
// MMA warp waits for; the first rows are on their way meanwhile. (One warp for
// the upsampled channels bounded the full-resolution decoder input: 1037 us at
// 3840 x 2160, 782 us with four.) The roles run ahead of each other as far as
// the ring (`ring` halo-row slots) and the two accumulators allow, synchronised
// only by mbarriers:
//   full[s]   the halo row in slot s is complete: TMA bytes landed (producer)
//             and, fused, the upsampled channels stored -> MMA
//   empty[s]  the MMAs that read slot s completed (MMA commit -> producer)
//   acc_full[b]  row accumulator b is complete (MMA commit -> drain)
//   acc_empty[b] the drain warps have read accumulator b (drain -> MMA)
constexpr int kStThreads = 192, kStUpWarps = 4;

// (80 registers let four CTAs of 192 threads share an SM.)
// pool: the 2x2 averages are written in the drain of every odd row (rows start
// even in every unit). As a pass of their own they read the whole output again:
// 207 + 97 us for the second layer at 3840 x 2160, 262 together; 95 + 35 and 113
// a level down.
template <int nacc, bool pool>
__global__ void __maxnreg__(80)
    k_conv3x3_strip(ConvArgs a, const __grid_constant__ CUtensorMap tmap, int ncols, int ring, int segs, int seg_rows,
                    int ntile, int dsets, uint32_t *err, int withhold_acc_full)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ uint32_t tmem_holder;
    __shared__ __align__(8) uint64_t full[kStMaxRing], empty[kStMaxRing];
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2], weights_full;
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int tiles_x = (a.wd + kTcM - 1) / kTcM;
    const int units = a.n * tiles_x * segs;
    const int KC = a.cin >> 3;
    const int N = ntile, n0 = (int)blockIdx.y * ntile; // this CTA's output channels
    const int slot_bytes = (KC / 2) * kStPlane;
    const int tap_bytes = N * a.cin * 2;
    const uint32_t half_cols = (uint32_t)ncols >> 1;
    const uint32_t raw = smem_addr(smem_raw);
    const uint32_t ring_base = (raw + 1023u) & ~1023u;
    const uint32_t w_base = ring_base + (uint32_t)(ring * slot_bytes);
    uint8_t *w_ptr = smem_raw + (w_base - raw);
    const volatile int *abort_v = &abort_flag;

    const int CG = a.cc >> 3;  // channel groups filled by the last warps (upsampled coarse input)
    const int up_warp = 2 + 4 * dsets;
    if (tid == 0) {
        for (int r = 0; r < ring; r++) {
            mbar_init(&full[r], CG ? 1 + kStUpWarps : 1);
            mbar_init(&empty[r], 1);
        }
        for (int k = 0; k < 2; k++) {
            mbar_init(&acc_full[k], 1);
            mbar_init(&acc_empty[k], 4 * dsets);
        }
        mbar_init(&weights_full, blockDim.x - 64u); // every thread of the warps that copy them
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const bool copies = warp != 4 && warp != 5;
    if (copies) {
        const int ct = warp < 4 ? tid : tid - 64, cn = (int)blockDim.x - 64;
        for (int i = ct; i < 9 * N * KC; i += cn) {
            const int kc = i % KC, n = (i / KC) % N, tap = i / (KC * N);
            const bool ok = n0 + n < a.cout;
            const bf16 *src = ok ? a.wgt + ((long)(n0 + n) * 9 + tap) * a.cin + 8 * kc : a.wgt;
            cp_async16(w_ptr + tap * tap_bytes + (n >> 3) * (KC * 128) + kc * 128 + (n & 7) * 16, src, ok);
        }
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_holder)),
                     "r"(ncols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_holder, 0);
    if (copies) {
        cp_async_commit();
        cp_async_wait<0>();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_arrive(smem_addr(&weights_full));
    }
    pdl_wait();
    if (tid == 0)
        pdl_start();

    if (warp >= up_warp) {
        // ---- upsampled channels of a fused concat input: fine pixel x of
        // halo row y reads coarse pixel (x >> 1, y >> 1). 16-byte cp.async
        // copies (consecutive lanes on consecutive pixels, a lane all channel
        // groups of its pixel); a row is published (fence to the async proxy,
        // arrive on its full barrier) as soon as its copies have landed. (Held
        // back until two newer rows were on their way, it had to wait for the
        // slots of those: with the four slots of the half-resolution decoder
        // input the MMAs then waited for every row, 324 us at 3840 x 2160
        // against 211. The full-resolution one: 583 and 578 us.)
        if (CG) {
            const int hc = a.h >> 1, wc = a.wd >> 1;
            constexpr int kUp = 32 * kStUpWarps;
            const int first = 32 * (warp - up_warp) + lane;
            int slot = 0, phase = 0;
            bool ok = true;
            for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
                const int sg = u % segs, tx = (u / segs) % tiles_x, nb = u / (segs * tiles_x);
                const int x0 = tx * kTcM, ya = sg * seg_rows;
                const int nout = min(a.h, ya + seg_rows) - ya;
                if (nout <= 0)
                    continue;
                for (int h = 0; h < nout + 2 && ok; h++) {
                    bool w = true;
                    if (lane == 0)
                        w = mbar_wait_role(smem_addr(&empty[slot]), (uint32_t)(phase ^ 1), abort_v);
                    ok = __shfl_sync(0xffffffffu, w, 0);
                    if (!ok)
                        break;
                    const int yy = ya - 1 + h;
                    const bool row_ok = yy >= 0 && yy < a.h;
                    const bf16 *crow = a.coarse + ((long)nb * hc + (row_ok ? yy >> 1 : 0)) * wc * a.cc;
                    uint8_t *dst = smem_raw + (ring_base - raw) + slot * slot_bytes;
                    for (int pp = first; pp < kStHaloPx; pp += kUp) {
                        const int xx = x0 - 1 + pp;
                        const bool in = row_ok && xx >= 0 && xx < a.wd;
                        const bf16 *src = in ? crow + (long)(xx >> 1) * a.cc : a.coarse;
                        for (int g = 0; g < CG; g++)
                            cp_async16(dst + st_chunk(g, pp), src + (in ? 8 * g : 0), in);
                    }
                    cp_async_commit();
                    cp_async_wait<0>();
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(smem_addr(&full[slot]));
                    if (++slot == ring) {
                        slot = 0;
                        phase ^= 1;
                    }
                }
            }
            if (!ok)
                abort_flag = 1;
        }
    } else if (warp == 4) {
        // ---- producer: one TMA row ((KC - CG) / 2 boxes of 16 channels x 130
        // pixels of `in`) per halo row
        if (lane == 0) {
            const uint64_t tmap_ptr = reinterpret_cast<uint64_t>(&tmap);
            const uint32_t row_tx = (uint32_t)((KC - CG) * kStHaloPx * 16);
            int slot = 0, phase = 0, issued = 0;
            int last_phase[kStMaxRing];
            for (int r = 0; r < kStMaxRing; r++)
                last_phase[r] = -1;
            for (int u = blockIdx.x; u < units && !*abort_v; u += gridDim.x) {
                const int sg = u % segs, tx = (u / segs) % tiles_x, nb = u / (segs * tiles_x);
                const int x0 = tx * kTcM, ya = sg * seg_rows;
                const int nout = min(a.h, ya + seg_rows) - ya;
                if (nout <= 0)
                    continue;
                for (int h = 0; h < nout + 2; h++) {
                    if (!mbar_wait_role(smem_addr(&empty[slot]), (uint32_t)(phase ^ 1), abort_v)) {
                        abort_flag = 1;
                        break;
                    }
                    const uint32_t bar = smem_addr(&full[slot]);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(row_tx)
                                 : "memory");
                    const uint32_t dst = ring_base + (uint32_t)(slot * slot_bytes);
                    for (int kp = CG / 2; kp < KC / 2; kp++)
                        asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                                     "[%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst + (uint32_t)(kp * kStPlane)),
                                     "l"(tmap_ptr), "r"(16 * kp - 8 * CG), "r"(x0 - 1), "r"(ya - 1 + h), "r"(nb),
                                     "r"(bar)
                                     : "memory");
                    last_phase[slot] = phase;
                    issued++;
                    if (++slot == ring) {
                        slot = 0;
                        phase ^= 1;
                    }
                }
            }
            // every copy issued has landed before the CTA exits
            for (int r = 0; r < ring; r++)
                if (last_phase[r] >= 0 && !mbar_wait(smem_addr(&full[r]), (uint32_t)last_phase[r]))
                    abort_flag = 1;
        }
    } else if (warp == 5) {
        // ---- MMA issue: 9 taps x cin / 16 steps per output row
        const uint32_t elected = elect_one();
        const uint32_t idesc =
            (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kTcM >> 4) << 24);
        const uint64_t a_hi = umma_desc(0, 16, 256) | (6ull << 61), b_hi = umma_desc(0, 128, (uint32_t)(KC * 128));
        const uint32_t a_lo_base = ring_base >> 4, a_lo_slot = (uint32_t)slot_bytes >> 4;
        const uint32_t b_lo_base = w_base >> 4, b_lo_tap = (uint32_t)tap_bytes >> 4;
        // the whole warp waits, and goes on or gives up together
        auto wait = [&](uint64_t &bar, int phase) {
            return __all_sync(0xffffffffu, mbar_wait_role(smem_addr(&bar), (uint32_t)phase, abort_v)) != 0;
        };
        int row_slot = 0;            // slot of the unit's halo row i
        int wait_slot = 0, wait_phase = 0, waited = 0; // next halo row to see complete
        int gi = 0;                  // output rows so far
        int halo = 0;                // halo rows of earlier units
        bool ok = wait(weights_full, 0);
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
            const int sg = u % segs;
            const int ya = sg * seg_rows;
            const int nout = min(a.h, ya + seg_rows) - ya;
            if (nout <= 0)
                continue;
            for (int i = 0; i < nout && ok; i++, gi++) {
                while (ok && waited < halo + i + 3) {
                    ok = wait(full[wait_slot], wait_phase);
                    if (ok) {
                        waited++;
                        if (++wait_slot == ring) {
                            wait_slot = 0;
                            wait_phase ^= 1;
                        }
                    }
                }
                const int b = gi & 1;
                if (ok)
                    ok = wait(acc_empty[b], ((gi >> 1) & 1) ^ 1);
                if (!ok)
                    break;
                asm volatile("tcgen05.fence::after_thread_sync;");
                const uint32_t acc = tmem + (uint32_t)b * half_cols;
                uint32_t slot_lo[3];
#pragma unroll
                for (int dy = 0; dy < 3; dy++) {
                    int sl = row_slot + dy;
                    sl = sl >= ring ? sl - ring : sl;
                    slot_lo[dy] = a_lo_base + (uint32_t)sl * a_lo_slot;
                }
                for (int j = 0; j < KC / 2; j++) {
#pragma unroll
                    for (int tap = 0; tap < 9; tap++) {
                        const int dy = tap / 3, dx = tap % 3;
                        umma(acc + (uint32_t)((tap & (nacc - 1)) * N),
                             a_hi | (uint64_t)(slot_lo[dy] + (uint32_t)(2 * dx) + (uint32_t)j * (kStPlane / 16)),
                             b_hi | (uint64_t)(b_lo_base + (uint32_t)tap * b_lo_tap + (uint32_t)j * (2 * 128 / 16)),
                             idesc, j > 0 || tap >= nacc, elected);
                    }
                }
                if (elected) {
                    // (withhold_acc_full: a diagnostic launch that never signals
                    // the drain warps, whose bounded waits then run out)
                    if (!withhold_acc_full)
                        umma_commit(smem_addr(&acc_full[b]));
                    // halo row i is not read by later rows of the unit
                    umma_commit(smem_addr(&empty[row_slot]));
                }
                __syncwarp();
                row_slot = row_slot + 1 == ring ? 0 : row_slot + 1;
            }
            if (!ok)
                break;
            // the unit's last two halo rows
            for (int k = 0; k < 2; k++) {
                if (elected)
                    umma_commit(smem_addr(&empty[row_slot]));
                __syncwarp();
                row_slot = row_slot + 1 == ring ? 0 : row_slot + 1;
            }
            halo += nout + 2;
        }
        if (!ok)
            abort_flag = 1;
        // the MMAs of the last row issued are complete before TMEM is freed
        if (lane == 0 && gi > 0 && !mbar_wait(smem_addr(&acc_full[(gi - 1) & 1]), (uint32_t)(((gi - 1) >> 1) & 1)))
            abort_flag = 1;
    } else {
        // ---- drain: warp w reads TMEM lanes 32 (w % 4) .. + 31 (pixels x0 +
        // 32 (w % 4) + lane), 16 channels at a time, a set every `dsets`th 16.
        // A row's drain has to keep up with its MMAs, which hold the path that
        // loads and stores take, so what it loads is asked for early: the bias
        // one group ahead (loaded when it was needed, it made a drain of 64
        // channels 4000 clocks long against 1760 of MMAs).
        int gi = 0;
        bool ok = true;
        const int set = warp < 4 ? 0 : 1, quarter = warp & 3;
        Bias16 bias;
        load_bias(a, n0 + 16 * set, bias);
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
            const int sg = u % segs, tx = (u / segs) % tiles_x, nb = u / (segs * tiles_x);
            const int x0 = tx * kTcM, ya = sg * seg_rows;
            const int nout = min(a.h, ya + seg_rows) - ya;
            if (nout <= 0)
                continue;
            for (int i = 0; i < nout; i++, gi++) {
                const int b = gi & 1;
                ok = mbar_wait_role(smem_addr(&acc_full[b]), (uint32_t)((gi >> 1) & 1), abort_v);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok)
                    break;
                asm volatile("tcgen05.fence::after_thread_sync;");
                const int x = x0 + quarter * 32 + lane;
                const long p = ((long)nb * a.h + ya + i) * a.wd + x;
                const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)b * half_cols;
                for (int c = 16 * set; c < N; c += 16 * dsets) {
                    uint32_t r[16];
                    tmem_sum16<nacc>(acc + (uint32_t)c, (uint32_t)N, r);
                    const bool last = c + 16 * dsets >= N;
                    if (last) {
                        // the accumulator is read: hand it back to the MMA warp
                        asm volatile("tcgen05.fence::before_thread_sync;");
                        __syncwarp();
                        if (lane == 0)
                            mbar_arrive(smem_addr(&acc_empty[b]));
                    }
                    const bool ok_px = x < a.wd && n0 + c < a.cout;
                    uint32_t h[8] = {};
                    if (ok_px)
                        store_row16(a, p, n0 + c, r, bias, h);
                    if constexpr (pool)
                        if (i & 1)
                            pool_row16(a, p, ((long)nb * (a.h >> 1) + ((ya + i) >> 1)) * (a.wd >> 1) + (x >> 1), n0 + c, h,
                                       ok_px);
                    if (dsets * 16 < N)
                        load_bias(a, n0 + (last ? 16 * set : c + 16 * dsets), bias);
                }
            }
        }
        if (!ok)
            abort_flag = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (abort_flag && tid == 0)
        atomicOr(err, 1u);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols));
}

// Weight gradient on the tcgen05 tensor cores, one tap per CTA:
// dW_tap[co][ci] = sum_p dout[p][co] * in[p shifted by the tap][ci], a GEMM
// with M = 128 output channels (zero rows past cout), N = up to 128 input
// channels, K = a slice of pixels. Both operands are MN-major as they lie in
// NHWC memory (8 consecutive channels of a pixel are 16 contiguous bytes): a
// K chunk of 64 pixels is staged as [channel group][pixel][16 B], i.e. core
// matrices of 8 channels x 8 pixels, K groups 128 B apart (LBO) and channel
// groups 64 x 16 B apart (SBO). Three stages of cp.async copies; thread 0
// issues four m128 nN k16 MMAs per chunk and commits each stage to its
// mbarrier, refills wait for the MMAs of the stage's previous chunk. The
// accumulator (one TMEM column per input channel, lane = output channel) is
// added to dw with atomics. Waits are bounded as in the other tcgen05
// kernels.
constexpr int kWtK = 64, kWtStages = 3, kWtM = 128;

__host__ __device__ constexpr int wt_stage_bytes(int N) { return kWtK * (kWtM + N) * 2; }

__global__ void __launch_bounds__(128) k_conv3x3_wgrad_tc(const bf16 *__restrict__ dout, int cout,
                                                          const bf16 *__restrict__ in, int cin, int n, int h, int w,
                                                          float *dw, long slice, int ntile, int ncols, uint32_t *err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint32_t tmem_holder;
    __shared__ __align__(8) uint64_t mbar[kWtStages];
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tap = blockIdx.y % 9;
    const int tiles_ci = (cin + ntile - 1) / ntile;
    const int ct = blockIdx.y / 9;
    const int co0 = (ct / tiles_ci) * kWtM, ci0 = (ct % tiles_ci) * ntile;
    const int N = min(ntile, (cin - ci0 + 15) & ~15);
    const long P = (long)n * h * w;
    const long pbeg = (long)blockIdx.x * slice, pend = min(P, pbeg + slice);
    const int dy = tap / 3 - 1, dx = tap % 3 - 1;
    const int nchunks = (int)((pend - pbeg + kWtK - 1) / kWtK);
    const int stage_bytes = wt_stage_bytes(ntile);
    const uint32_t sbase = smem_addr(smem);

    if (tid == 0) {
        for (int st = 0; st < kWtStages; st++)
            mbar_init(&mbar[st], 1);
        abort_flag = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_holder)),
                     "r"(ncols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_holder;
    // D f32, A/B bf16, A and B MN-major (bits 15, 16), N >> 3, M >> 4
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kWtM >> 4) << 24);

    // A rows past cout stay zero: cleared once, never loaded
    const int ga = (min(cout - co0, kWtM) + 7) / 8; // A channel groups with data
    for (int i = tid; i < kWtStages * (kWtM / 8 - ga) * kWtK; i += 128) {
        const int st = i / ((kWtM / 8 - ga) * kWtK), r = i % ((kWtM / 8 - ga) * kWtK);
        *reinterpret_cast<uint4 *>(smem + st * stage_bytes + (ga * kWtK + r) * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
    // thread -> one pixel of the chunk (its position decoded once) and every
    // other channel group
    const int lpx = tid & (kWtK - 1), lhalf = tid / kWtK;
    auto load_chunk = [&](int c) {
        uint8_t *a_s = smem + (c % kWtStages) * stage_bytes;
        uint8_t *b_s = a_s + kWtK * kWtM * 2;
        const long p = pbeg + (long)c * kWtK + lpx;
        const bool pok = p < pend;
        bool xok = false;
        long q = 0;
        if (pok) {
            const int pn = (int)(p / ((long)h * w));
            const int rem = (int)(p - (long)pn * h * w);
            const int y = rem / w;
            const int yy = y + dy, xx = rem - y * w + dx;
            xok = yy >= 0 && yy < h && xx >= 0 && xx < w;
            q = ((long)pn * h + yy) * w + xx;
        }
        for (int g = lhalf; g < ga; g += 2) {
            const int co = co0 + 8 * g;
            const bool ok = pok && co < cout;
            cp_async16(a_s + g * (kWtK * 16) + lpx * 16, ok ? dout + p * cout + co : dout, ok);
        }
        for (int g = lhalf; g < N / 8; g += 2) {
            const int ci = ci0 + 8 * g;
            const bool ok = xok && ci < cin;
            cp_async16(b_s + g * (kWtK * 16) + lpx * 16, ok ? in + q * cin + ci : in, ok);
        }
    };

    for (int st = 0; st < kWtStages - 1; st++) {
        if (st < nchunks)
            load_chunk(st);
        cp_async_commit();
    }
    for (int c = 0; c < nchunks; c++) {
        cp_async_wait<kWtStages - 2>(); // this thread's copies of chunk c landed
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (abort_flag)
            break;
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t a_addr = sbase + (uint32_t)((c % kWtStages) * stage_bytes);
            const uint32_t b_addr = a_addr + (uint32_t)(kWtK * kWtM * 2);
#pragma unroll
            for (int j = 0; j < kWtK / 16; j++) {
                // K step j: pixels 16 j .. 16 j + 15 = two K groups of 8
                const uint64_t ad = umma_desc(a_addr + (uint32_t)(j * 256), 128, kWtK * 16);
                const uint64_t bd = umma_desc(b_addr + (uint32_t)(j * 256), 128, kWtK * 16);
                const uint32_t accumulate = (c > 0 || j > 0) ? 1u : 0u;
                asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                             "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
                             "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate));
            }
            umma_commit(smem_addr(&mbar[c % kWtStages]));
        }
        // chunk c + 2 reuses the stage of chunk c - 1
        const int nx = c + kWtStages - 1;
        if (nx < nchunks) {
            if (c >= 1) {
                const int prev = c - 1;
                if (!mbar_wait(smem_addr(&mbar[prev % kWtStages]), (uint32_t)((prev / kWtStages) & 1)))
                    atomicOr(&abort_flag, 1);
            }
            load_chunk(nx);
        }
        cp_async_commit();
    }
    cp_async_wait<0>();
    if (!abort_flag && nchunks > 0) {
        const int last = nchunks - 1;
        if (!mbar_wait(smem_addr(&mbar[last % kWtStages]), (uint32_t)((last / kWtStages) & 1)))
            atomicOr(&abort_flag, 1);
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (!abort_flag && nchunks > 0) {
        const int co = co0 + warp * 32 + lane;
        for (int c = 0; c < N; c += 16) {
            uint32_t r[16];
            tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, r);
            if (co >= cout)
                continue;
            float *d = dw + ((long)co * 9 + tap) * cin + ci0 + c;
#pragma unroll
            for (int k = 0; k < 16; k++)
                if (ci0 + c + k < cin)
                    atomicAdd(d + k, __uint_as_float(r[k]));
        }
    } else if (abort_flag && tid == 0) {
        atomicOr(err, 1u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols));
}

}  // namespace

namespace {

std::atomic<bool> g_inject_wait_timeout{false};

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

// The current device and what plans and launches need to know of it.
struct DeviceProps {
    int sms = 0, sm_smem = 0, optin = 0, reserved = 0;
};
int current_device()
{
    int dev = 0;
    cudaGetDevice(&dev);
    return dev;
}
const DeviceProps &device_props()
{
    static vvpt::PerDevice<DeviceProps> props;
    const int dev = current_device();
    return props.get(dev, [dev] {
        DeviceProps p;
        cudaDeviceGetAttribute(&p.sms, cudaDevAttrMultiProcessorCount, dev);
        cudaDeviceGetAttribute(&p.sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
        cudaDeviceGetAttribute(&p.optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        cudaDeviceGetAttribute(&p.reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
        return p;
    });
}

// Lets a kernel have up to `most` bytes of dynamic shared memory on the current
// device, once and for every launch of it there.
template <auto kernel>
void allow_smem(int most, bool carveout = false)
{
    static vvpt::PerDevice<bool> done;
    done.get(current_device(), [&] {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (carveout)
            cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        return true;
    });
}

// Launch that may start while the previous one runs (see pdl_wait).
template <class... P, class... A>
void launch_pdl(void (*kernel)(P...), dim3 grid, int threads, int smem, cudaStream_t s, A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// Output channels per CTA where `ctas` CTAs with all N leave SMs idle: the
// smallest share (a divisor of N, a multiple of 16) for which one CTA per SM
// still takes them all at once.
int split_channels(int N, long ctas)
{
    for (int nt = 16; nt < N; nt += 16)
        if (N % nt == 0 && ctas * (N / nt) <= device_props().sms)
            return nt;
    return N;
}

constexpr int kStStatic = 2048; // the strip kernel's mbarriers, TMEM address, flags (1 KB aligned)

struct StripPlan {
    int ntile = 0; // output channels per CTA
    int dsets = 1; // drain sets of four warps
    int ring = 0, smem = 0, grid = 0, segs = 0, seg_rows = 0, ncols = 0, nacc = 1;
};

// Occupancy first (up to 4 CTAs per SM, bounded by shared memory and by the
// 512 TMEM columns of an SM), then the deepest ring that fits; the rows of
// every 128-pixel column are cut into segments so that one wave of CTAs
// covers the layer.
bool plan_strip(const ConvArgs &a, StripPlan &pl)
{
    if (a.cin % 16 || a.cin < 16 || a.cout > 256 || a.cout < 1 || (reinterpret_cast<uintptr_t>(a.in) & 15))
        return false;
    if (a.cc && (a.cc % 16 || a.cc >= a.cin || a.h % 2 || a.wd % 2 || (reinterpret_cast<uintptr_t>(a.coarse) & 15)))
        return false;
    const DeviceProps &dp = device_props();
    const int nsm = dp.sms;
    if (!tensor_map_encoder())
        return false;
    const int N = (a.cout + 15) & ~15;
    const int slot = (a.cin / 16) * kStPlane;
    int share = N; // output channels whose weights a CTA holds
    int ncols = 32;
    while (ncols < 2 * N)
        ncols <<= 1;
    auto ring_of = [&](int c) {
        const int dyn = std::min(dp.optin - kStStatic, dp.sm_smem / c - dp.reserved - kStStatic);
        return std::min(kStMaxRing, (dyn - 1024 - 9 * share * a.cin * 2) / slot);
    };
    // accumulators per row (independent MMA chains, whose sums the drain adds):
    // 1, 2 or 4, as many as the TMEM of an SM holds beside the other CTAs of
    // the most that fit there with a ring of at most eight rows. This fixes
    // the order of the sums, whatever occupancy and ring are chosen below.
    int most = 0, nacc = 1;
    for (int c = 4; c >= 1 && !most; c--)
        if (c * ncols <= 512 && std::min(8, ring_of(c)) >= kStMinRing)
            most = c;
    const long cols = (long)a.n * ((a.wd + kTcM - 1) / kTcM);
    if (!most) {
        // The weights of all channels leave no room for three rows: shares of
        // them, one CTA per SM, each of which reads the whole input. The sums
        // are the per-tile kernel's (one accumulator, channels in the same
        // order), which keeps the layer where the image has less than a row of
        // 128 pixels per SM. 96 to 96 channels at 480 x 270: 65 to 35 us; 160 to
        // 64 at 960 x 540, fused: 249 to 238; whole images of 1024 x 512,
        // 1280 x 720 and 2560 x 1440: 383 to 378, 514 to 509 and 1378 to 1341.
        if (N > 128)
            return false;
        for (share = N - 16; share >= 16 && !most; share -= 16)
            if (N % share == 0 && ring_of(1) >= kStMinRing) {
                most = 1;
                break;
            }
        if (!most || cols * a.h * (N / share) < nsm)
            return false;
    }
    for (int q = 4; q >= 2 && nacc == 1 && share == N; q >>= 1) {
        int cq = 32;
        while (cq < 2 * q * N)
            cq <<= 1;
        if (most * cq <= 512)
            nacc = q;
    }
    int tcols = 32;
    while (tcols < 2 * nacc * N)
        tcols <<= 1;
    // CTAs per SM. A fused upsample + concat input takes one, with the deepest
    // ring: its upsample warps then run rows ahead of the MMAs (the
    // half-resolution decoder input at 3840 x 2160, 112 to 48 channels: 211 us,
    // against 450 us for upsampling, concatenating and convolving it
    // separately; the full-resolution one 578 against 650 with two per SM).
    const int c = a.cc ? 1 : most;
    const int ring = ring_of(c);
    const long ctas = (long)nsm * c / (N / share);
    int segs = (int)std::max<long>(1, std::min<long>(a.h, ctas / std::max<long>(1, cols)));
    int seg_rows = (a.h + segs - 1) / segs;
    if (a.pool)
        seg_rows = (seg_rows + 1) & ~1; // rows that are averaged together in one unit
    segs = (a.h + seg_rows - 1) / seg_rows;
    // a small image: fewer output channels per CTA (the accumulators stay as
    // planned for all of them)
    pl.grid = (int)std::min<long>(cols * segs, ctas);
    pl.ntile = std::min(split_channels(N, pl.grid), share);
    if (pl.ntile != N)
        for (tcols = 32; tcols < 2 * nacc * pl.ntile;)
            tcols <<= 1;
    // no more shared memory than the rows of a CTA's run need, so that the
    // next launch can begin beside this one
    pl.ring = (int)std::min<long>(ring, cols * segs <= ctas ? std::max(kStMinRing, seg_rows + 2) : kStMaxRing);
    pl.smem = 1024 + 9 * pl.ntile * a.cin * 2 + pl.ring * slot;
    pl.segs = segs;
    pl.seg_rows = seg_rows;
    pl.ncols = tcols;
    pl.nacc = nacc;
    // A second set of drain warps where the registers of the CTAs of an SM
    // leave room for it and there are channels to share (64 channels at
    // 960 x 540: 72 to 52 us; 48 at 1920 x 1080: 114 to 95). A fused
    // input keeps one: its MMAs bound it, and a second set only takes
    // shared-memory and issue slots from them (80 to 32 channels at
    // 3840 x 2160: 583 us with one, 615 with two).
    pl.dsets = c <= 2 && pl.ntile >= 32 && !a.cc ? 2 : 1;
    return true;
}

// rank-4 map over the NHWC input {C, W, H, N} (the cin - cc channels of `in`);
// box = 16 channels x 130 pixels, stored with the 32-byte swizzle (st_chunk)
bool encode_input_map(const ConvArgs &a, CUtensorMap &m)
{
    const int c = a.cin - a.cc;
    const cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)a.wd, (cuuint64_t)a.h, (cuuint64_t)a.n};
    const cuuint64_t strides[3] = {(cuuint64_t)c * 2, (cuuint64_t)a.wd * c * 2, (cuuint64_t)a.h * a.wd * c * 2};
    const cuuint32_t box[4] = {16, (cuuint32_t)kStHaloPx, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return tensor_map_encoder()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16 *>(a.in), dims, strides, box,
                                estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

namespace {

template <int nacc, bool pool>
void launch_strip_as(const ConvArgs &a, const CUtensorMap &tmap, const StripPlan &pl, int withhold, cudaStream_t s,
                       uint32_t *err)
{
    allow_smem<k_conv3x3_strip<nacc, pool>>(device_props().optin - kStStatic, true);
    launch_pdl(k_conv3x3_strip<nacc, pool>, dim3((unsigned)pl.grid, (unsigned)(((a.cout + 15) & ~15) / pl.ntile)),
               kStThreads + 128 * (pl.dsets - 1) + (a.cc ? 32 * kStUpWarps : 0), pl.smem, s, a, tmap, pl.ncols, pl.ring,
               pl.segs, pl.seg_rows, pl.ntile, pl.dsets, err, withhold);
}

// The strip kernel for `a` when it takes the layer; false (nothing launched)
// otherwise.
bool launch_strip(const ConvArgs &a, cudaStream_t s, uint32_t *err, ConvKernels kind)
{
    StripPlan pl;
    CUtensorMap tmap;
    if (!err || kind == kConvTiles || !plan_strip(a, pl) || !encode_input_map(a, tmap))
        return false;
    if (kind == kConvPersistent)
        pl.grid = std::min(pl.grid, 16);
    const int withhold = g_inject_wait_timeout.exchange(false) ? 1 : 0;
    if (pl.nacc == 4)
        a.pool ? launch_strip_as<4, true>(a, tmap, pl, withhold, s, err)
               : launch_strip_as<4, false>(a, tmap, pl, withhold, s, err);
    else if (pl.nacc == 2)
        a.pool ? launch_strip_as<2, true>(a, tmap, pl, withhold, s, err)
               : launch_strip_as<2, false>(a, tmap, pl, withhold, s, err);
    else
        a.pool ? launch_strip_as<1, true>(a, tmap, pl, withhold, s, err)
               : launch_strip_as<1, false>(a, tmap, pl, withhold, s, err);
    return true;
}

}  // namespace

void inject_wait_timeout() { g_inject_wait_timeout.store(true); }

bool conv3x3_concat(const ConvArgs &a, cudaStream_t s, uint32_t *err, ConvKernels kind)
{
    return kind != kConvNoFusion && a.coarse && a.cc > 0 && launch_strip(a, s, err, kind);
}

bool conv3x3(const ConvArgs &a_in, cudaStream_t s, uint32_t *err, ConvKernels kind)
{
    ConvArgs a = a_in;
    a.coarse = nullptr;
    a.cc = 0;
    const long P = (long)a.n * a.h * a.wd;
    if (launch_strip(a, s, err, kind))
        return a.pool != nullptr;
    a.pool = nullptr;
    if (err && a.cout <= 256) {
        allow_smem<k_conv3x3_tc>(tc_smem_bytes(256));
        allow_smem<k_conv3x3_tc_chunk>(std::max(tc_chunk_smem_bytes(128, 2, tc_chunk_rows(128)),
                                                tc_chunk_smem_bytes(64, 2, tc_chunk_rows(64))));
        const int sms = device_props().sms;
        const int N = (a.cout + 15) & ~15;
        int ncols = 32;
        while (ncols < N)
            ncols <<= 1;
        const long tiles = (long)a.n * a.h * ((a.wd + kTcM - 1) / kTcM);
        if (N <= 128) {
            // several output rows per CTA, one accumulator (one MMA chain)
            // per row
            const long columns = (long)a.n * ((a.wd + kTcM - 1) / kTcM);
            int rows = tc_chunk_rows(N);
            // a small image leaves SMs idle: fewer rows per CTA while the
            // CTAs still run at once, one per SM (224 to 96 channels at 32 x 32:
            // 28 us on 32 CTAs, 19 us on 96)
            while (rows > 1 && 2 * columns * ((a.h + rows - 1) / rows) <= sms)
                rows /= 2;
            const long blocks = columns * ((a.h + rows - 1) / rows);
            // ... and then fewer output channels per CTA, which share the
            // staging of the weights
            const int nt = split_channels(N, blocks);
            const int smem = tc_chunk_smem_bytes(nt, (a.cin + kTcBK - 1) / kTcBK, rows);
            int cols = 32;
            while (cols < rows * nt)
                cols <<= 1;
            launch_pdl(k_conv3x3_tc_chunk, dim3((unsigned)blocks, (unsigned)(N / nt)), kTcThreads, smem, s, a, cols, rows,
                       nt, err);
        }
        else
            launch_pdl(k_conv3x3_tc, dim3((unsigned)tiles), kTcThreads, tc_smem_bytes(N), s, a, ncols, err);
        return false;
    }
    // 32-wide channel tiles where they leave fewer channels of the last tile
    // empty than 64-wide ones (16, 32, 80, 96, 160, 224 channels)
    const int waste64 = (a.cout + 63) / 64 * 64 - a.cout, waste32 = (a.cout + 31) / 32 * 32 - a.cout;
    if (waste32 < waste64) {
        dim3 grid((unsigned)((P + kBM - 1) / kBM), (unsigned)((a.cout + 31) / 32));
        k_conv3x3<32, 16><<<grid, 256, 0, s>>>(a);
    } else {
        dim3 grid((unsigned)((P + kBM - 1) / kBM), (unsigned)((a.cout + 63) / 64));
        k_conv3x3<64, 32><<<grid, 256, 0, s>>>(a);
    }
    return false;
}

void conv3x3_wgrad(const bf16 *dout, int cout, const bf16 *in, int cin, int n, int h, int w, float *dw, float *dbias,
                   cudaStream_t s, uint32_t *err, long copy_stride)
{
    const long P = (long)n * h * w;
    if (err) {
        // tcgen05: 128 output channels x up to 128 input channels per tap and slice
        const int ntile = std::min(128, (cin + 15) & ~15);
        int ncols = 32;
        while (ncols < ntile)
            ncols <<= 1;
        const int tiles = ((cout + kWtM - 1) / kWtM) * ((cin + ntile - 1) / ntile);
        long slices = std::max<long>(1, (device_props().sms * 4L) / (9L * tiles));
        long slice = (P + slices - 1) / slices;
        slice = std::max<long>(kWtK, (slice + kWtK - 1) / kWtK * kWtK);
        slices = (P + slice - 1) / slice;
        const int smem = kWtStages * wt_stage_bytes(ntile);
        allow_smem<k_conv3x3_wgrad_tc>(kWtStages * wt_stage_bytes(128));
        dim3 grid((unsigned)slices, (unsigned)(9 * tiles));
        k_conv3x3_wgrad_tc<<<grid, 128, smem, s>>>(dout, cout, in, cin, n, h, w, dw, slice, ntile, ncols, err);
    } else {
        wgrad_mma_sync(dout, cout, in, cin, n, h, w, dw, dbias, s, copy_stride);
    }
    if (err && dbias) {
        // channel counts are multiples of 8 up to 256: 1-32 groups per pixel lane
        const int lanes = kBiasThreads / (cout / 8);
        const long blocks = std::min<long>(152L * 4, (P + 16L * lanes - 1) / (16L * lanes));
        k_bias_grad<<<(unsigned)std::max<long>(blocks, 1), kBiasThreads, 0, s>>>(dout, cout, P, dbias);
    }
}

template <int BN>
static void launch_wgrad(const bf16 *dout, int cout, const bf16 *in, int cin, int n, int h, int w, float *dw,
                         float *dbias, cudaStream_t s, long copy_stride)
{
    allow_smem<k_conv3x3_wgrad<BN>>(wg_smem<BN>());
    // three (BN = 32) or two blocks fit an SM: about one unit per block over
    // all channel tiles
    const int tiles = ((cout + kWgM - 1) / kWgM) * ((cin + BN - 1) / BN);
    const long cols = (long)n * ((w + kWgPx - 1) / kWgPx), blocks = std::max<long>(1, (long)device_props().sms * (BN == 32 ? 3 : 2) / tiles);
    int segs = (int)std::max<long>(1, std::min<long>(h, blocks / cols));
    const int seg_rows = (h + segs - 1) / segs;
    segs = (h + seg_rows - 1) / seg_rows;
    dim3 grid((unsigned)std::min<long>(cols * segs, blocks), (unsigned)tiles);
    k_conv3x3_wgrad<BN><<<grid, kWgThreads, wg_smem<BN>(), s>>>(dout, cout, in, cin, n, h, w, dw, dbias, segs, seg_rows,
                                                          copy_stride ? kGradCopies : 1, copy_stride);
}

void wgrad_mma_sync(const bf16 *dout, int cout, const bf16 *in, int cin, int n, int h, int w, float *dw, float *dbias,
                    cudaStream_t s, long copy_stride)
{
    // 64 input channels per block where that leaves no more of them empty
    // than 32 would (64, 112, 128 channels)
    if ((cin + 63) / 64 * 64 == (cin + 31) / 32 * 32)
        launch_wgrad<64>(dout, cout, in, cin, n, h, w, dw, dbias, s, copy_stride);
    else
        launch_wgrad<32>(dout, cout, in, cin, n, h, w, dw, dbias, s, copy_stride);
}

void prepare_weights(const float *params, const WeightTable &t, bf16 *w16, bf16 *wt16, cudaStream_t s)
{
    k_prepare_weights<<<grid_for((long)t.start[t.layers]), 256, 0, s>>>(params, t, w16, wt16);
}

void pack_features(const float *radiance, const float *albedo, const float *normal, bf16 *x, int npix, cudaStream_t s)
{
    launch_pdl(k_pack_features, dim3(grid_for(npix)), 256, 0, s, reinterpret_cast<const float4 *>(radiance),
               reinterpret_cast<const float4 *>(albedo), reinterpret_cast<const float4 *>(normal), x, npix);
}

// 8-channel groups of a layout kernel, indexed in 32 bits by the kernels: the
// denoiser's batch limit (n x h x w <= 2^27 pixels, at most 80 channels at
// full resolution) keeps every count below 2^31
static long groups8(long pixels, int c) { return pixels * (c / 8); }

void avgpool2(const bf16 *in, bf16 *out, int n, int h, int w, int c, cudaStream_t s)
{
    launch_pdl(k_avgpool2, dim3(grid_for(groups8((long)n * (h / 2) * (w / 2), c))), 256, 0, s, in, out, n, h, w, c);
}

void upcat(const bf16 *coarse, int cc, const bf16 *skip, int cs, bf16 *out, int n, int h, int w, cudaStream_t s)
{
    launch_pdl(k_upcat, dim3(grid_for(groups8((long)n * h * w, cc + cs))), 256, 0, s, coarse, cc, skip, cs, out, n, h, w);
}

void upcat_backward(const bf16 *dcat, int cc, int cs, bf16 *dcoarse, bf16 *dskip, int n, int h, int w, cudaStream_t s)
{
    launch_pdl(k_upcat_backward_coarse, dim3(grid_for(groups8((long)n * (h / 2) * (w / 2), cc))), 256, 0, s, dcat, cc,
               cs, dcoarse, n, h, w);
    if (dskip)
        launch_pdl(k_upcat_backward_skip, dim3(grid_for(groups8((long)n * h * w, cs + cc))), 256, 0, s, dcat, cc, cs,
                   dskip, (unsigned)((long)n * h * w));
}

void pool_backward_combine(const bf16 *dskip, const bf16 *dpooled, const bf16 *e, bf16 *de, int n, int h, int w, int c,
                           cudaStream_t s)
{
    launch_pdl(k_pool_backward_combine, dim3(grid_for(groups8((long)n * h * w, c))), 256, 0, s, dskip, dpooled, e, de, n,
               h, w, c);
}

void l1_loss(const float *out, int cout, const float *target, bf16 *dout, float *loss_sum, int npix, cudaStream_t s)
{
    k_l1_loss<<<std::min(grid_for(npix), 152 * 8), 256, 0, s>>>(out, cout, reinterpret_cast<const float4 *>(target),
                                                                dout, loss_sum, npix);
}

void sum_grads(const float *g, size_t stride, float *sum, size_t n, cudaStream_t s)
{
    k_sum_grads<<<grid_for((long)n), 256, 0, s>>>(g, stride, sum, n);
}

void adam(float *p, const float *g, size_t stride, float *m, float *v, size_t n, float lr, float b1, float b2, float eps, int t,
          cudaStream_t s)
{
    const float c1 = 1.0f - powf(b1, (float)t), c2 = 1.0f - powf(b2, (float)t);
    k_adam<<<grid_for((long)n), 256, 0, s>>>(p, g, stride, m, v, n, lr, b1, b2, eps, c1, c2);
}

void unpack_output(const float *y, int cout, float *out_rgba, int npix, cudaStream_t s)
{
    k_unpack_output<<<grid_for(npix), 256, 0, s>>>(y, cout, reinterpret_cast<float4 *>(out_rgba), npix);
}

}  // namespace vvdn
