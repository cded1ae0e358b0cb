// k_surrogate.cu — BF16 convolution kernels of the learned surrogate on the 5th-generation
// tensor cores (tcgen05.mma, FP32 accumulators in tensor memory).  No reference
// counterpart: the reference has no learned part.
//
// The network is a stack of 3x3 convolutions over NHWC BF16 activations.  Every layer is an
// implicit GEMM  D[p][n] = sum_k A[p][k] B[n][k]  with p an output pixel (the MMA's M, 128 per
// tile), n an output channel (the MMA's N) and k = (tap, input channel) (K = 9 x CIN, 16 at a
// time).  The four pixel mappings (same-size, its adjoint, stride-2 down, stride-2 up) give
// the forward pass and the data gradient (the adjoint mapping with the channel-transposed
// weights) the same kernel; the weight gradient takes the pixels as the reduction.
//
// Shared memory holds an activation tile once, not once per tap.  The images are laid out
// as one raster of padded rows (a zero column after every row, a zero row after every
// image), so that a tap is a constant offset along the raster; the tile is stored as planes
// of 8 channels, pixel after pixel at 16 bytes.  Eight consecutive pixels of a plane are a
// core matrix of the no-swizzle layout, as K-major rows (forward: pixels are M, channels K)
// and as MN-major columns (weight gradient: channels are M or N, pixels K), and a tap's
// operand is the same tile with a start address shifted by 16 bytes per pixel.  The stride-2
// mappings split the finer image into its parity sub-images, each a raster of its own.
// The raster's padding pixels take part in the MMAs (about 1/W + 1/H of the work) and are
// dropped by the epilogue.
//
// One elected thread issues the MMAs; tcgen05.commit arrives on an mbarrier that the CTA
// waits on with a bounded spin (on timeout: an error flag, a second bounded wait, the
// tensor memory freed, return).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/hydist_b200.h"

long long hyd_kernel_launches_add(long long n);

namespace {

constexpr int kTile = 128;            // output pixels per CTA tile (MMA M)
constexpr int kConvGroups = 4;        // the forward kernel's thread groups: a share of the accumulators each
constexpr int kConvWorkers = kTile * kConvGroups;  // threads that copy tiles and write results
constexpr int kConvThreads = kConvWorkers + 32;    // and the warp that issues the MMAs
constexpr int kWgGroups = 3;          // the weight gradient's thread groups: a third of the accumulator each
constexpr int kWgWorkers = kTile * kWgGroups;
constexpr int kWgThreads = kWgWorkers + 32;
constexpr int kWgChain = 2048;        // raster positions summed in one tensor-memory chain
constexpr long long kWaitCycles = 1LL << 32;  // bounded waits (about 2 s); then the error flag

// pixel mappings of a layer (the input pixel that output pixel p, tap t reads)
enum ConvMode { kSame = HYD_CONV_SAME, kSameAdj = HYD_CONV_SAME_ADJ, kDown = HYD_CONV_DOWN, kUp = HYD_CONV_UP };

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// sm_100 shared-memory matrix descriptor: start, leading and stride byte offsets (>> 4),
// version 1 (bits 46-47), no swizzle (bits 61-63 = 0), base offset 0.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}

// Instruction descriptor of kind::f16: D FP32 (bits 4-5 = 1), A and B BF16 (bits 7-9, 10-12
// = 1), both K-major, or with `mn` both MN-major (bits 15, 16), N >> 3 at bit 17, M >> 4 at
// bit 24.
__host__ __device__ constexpr uint32_t instr_desc(int M, int N, int mn = 0) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (mn ? (3u << 15) : 0u) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(accum));
}

// One lane of a converged warp.  The MMAs are issued by this lane inside control flow that is
// uniform over the warp, with warp-uniform operands: they then come from uniform registers,
// and an MMA of M = 128, N = 48, K = 16 takes 44 cycles (32 + N / 4: its operands' bytes over 128
// a cycle).  Issued under `threadIdx.x == 0` the same MMA took 76 to 96 cycles.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}\n" : "=r"(p));
    return p != 0;
}
// v of lane 0: tells the compiler that the value is the same on every lane
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }

__device__ __forceinline__ void mma_commit(uint64_t* mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(mbar))
                 : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t* mbar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(mbar)) : "memory");
}

// Bounded wait for phase `parity` of the mbarrier; false on timeout, or once another thread of
// the CTA has given up (*fail set).
__device__ __forceinline__ bool mbar_wait(uint64_t* mbar, uint32_t parity, volatile int* fail) {
    const uint32_t a = smem_u32(mbar);
    const long long t0 = clock64();
    do {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
        if (*fail) return false;
    } while (clock64() - t0 < kWaitCycles);
    *fail = 1;
    return false;
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Tensor memory of `cols` columns (a power of two >= 32), allocated by warp 0.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}

// 16 FP32 columns of this thread's tensor-memory lane (32x32b shape: warp w reads lanes
// 32w..32w+31, thread = lane).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = __uint_as_float(r[k]);
}

// 16-byte asynchronous copy global -> shared, cached in L1 (the two halves of a 32-byte
// sector and the taps of neighbouring pixels read the same lines); src_bytes 0 fills the
// 16 bytes with zeros (nothing is read).  A thread's copies are waited for with
// cp_async_wait_all.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// A run of raster positions p0 + start .. p0 + start + len - 1 (p0: the tile's first
// position) of parity sub-image (py, px), held at pixels off.. of a tile's planes.
struct TileSeg {
    int start, len, off, py, px;
};

// Division of 0 <= n < 2^31 by an invariant d >= 1 as a high multiplication and a shift
// (Granlund and Montgomery, PLDI 1994): mul = ceil(2^(31 + l) / d), l = ceil(log2 d).
struct FastDiv {
    uint32_t mul, sh, one;  // one: d == 1 (its multiplier does not fit 32 bits)
    __device__ __forceinline__ uint32_t operator()(uint32_t n) const { return one ? n : __umulhi(n, mul) >> sh; }
};

// How the tiles of one layer are laid out: the raster (Hp x Wp positions per image, nflat in
// all, the tiles starting at position p_first), the segments of the input image a tile holds
// (npix pixels per plane) and where in it each tap of the tile's first position lies.
// Built by the host (conv_plan, wgrad_plan).
struct TilePlan {
    int Hp, Wp;       // padded raster of one image
    FastDiv dW, dH, dI;  // division by Wp, Hp and Hp Wp
    int small;        // every raster position fits 31 bits
    int sub;          // 2: the input is split into its parity sub-images, else 1
    int xlim, ylim;   // raster columns / rows of an image at and beyond these are padding
    int T;            // forward: tiles of 128 positions per step
    int S;            // weight gradient: positions per step
    int nseg, npix;
    TileSeg seg[6];
    int tap[9];       // forward: pixel offset of tap t; weight gradient: of accumulator q
    long long nflat, p_first, nstep;
};

// Where raster position f lies: image b (-1 or past the last one for positions outside the
// batch), row y, column x.
__device__ __forceinline__ void raster_at(const TilePlan& pl, long long f, int& b, int& y, int& x) {
    const long long per = (long long)pl.Hp * pl.Wp;
    const long long g = f + per;  // tiles reach back less than an image
    if (pl.small) {
        const uint32_t bq = pl.dI((uint32_t)g), r = (uint32_t)g - bq * (uint32_t)per;
        b = (int)bq - 1;
        y = (int)pl.dW(r);
        x = (int)r - y * pl.Wp;
    } else {
        const long long bq = g / per, r = g - bq * per;
        b = (int)bq - 1;
        y = (int)(r / pl.Wp);
        x = (int)(r - (long long)y * pl.Wp);
    }
}

// The pixel k positions after raster place (b0, y0, x0) in an image array of nb x Hs x Ws
// pixels, of parity sub-image (py, px); -1 for padding.
__device__ __forceinline__ long long raster_pixel(const TilePlan& pl, int b0, int y0, int x0, int k, int Hs, int Ws,
                                                  int nb, int sub, int py, int px, int xlim, int ylim) {
    const int xs = x0 + k, yq = (int)pl.dW((uint32_t)xs);
    const int x = xs - yq * pl.Wp;
    const int ys = y0 + yq, bq = (int)pl.dH((uint32_t)ys);
    const int y = ys - bq * pl.Hp;
    const int b = b0 + bq;
    const int iy = sub * y + py, ix = sub * x + px;
    const bool in = b >= 0 && b < nb && y < ylim && x < xlim && iy < Hs && ix < Ws;
    return in ? ((long long)b * Hs + iy) * Ws + ix : -1;
}

// Copy segment `sg` of the tile at p0 into planes of 8 channels at dst (plane stride ch
// bytes): C channels per pixel of the image at src (Hs x Ws pixels per image, nb images),
// zeros for padding, by the first WARPS warps of the CTA.  A warp's lanes 0..15 take 16 pixels' first half of the planes, lanes
// 16..31 their second half: a quarter-warp writes 128 contiguous bytes of one plane.
template <int C, int WARPS>
__device__ __forceinline__ void fill_seg(const TilePlan& pl, const TileSeg& sg, long long p0, uint32_t dst,
                                         uint32_t ch, const __nv_bfloat16* src, int Hs, int Ws, int nb, int sub) {
    constexpr int HP = C / 16;  // planes per half-warp
    const int lane = threadIdx.x & 31, half = lane >> 4;
    int b0, y0, x0;
    raster_at(pl, p0 + sg.start, b0, y0, x0);
    for (int k = (threadIdx.x >> 5) * 16 + (lane & 15); k < sg.len; k += WARPS * 16) {
        const long long q = raster_pixel(pl, b0, y0, x0, k, Hs, Ws, nb, sub, sg.py, sg.px, pl.xlim, pl.ylim);
        const __nv_bfloat16* s = src + (q < 0 ? 0 : q * C + 8 * HP * half);
        const uint32_t n = q < 0 ? 0u : 16u, d = dst + (uint32_t)(HP * half) * ch + (uint32_t)(sg.off + k) * 16;
#pragma unroll
        for (int c = 0; c < HP; c++) cp_async16(d + (uint32_t)c * ch, q < 0 ? s : s + 8 * c, n);
    }
}

// The output gradient of S positions from p0 into planes 0.. and, one position further, into
// planes 8.. (the weight gradient's two row blocks), C channels per pixel.
template <int C, int WARPS>
__device__ __forceinline__ void fill_twice(const TilePlan& pl, long long p0, uint32_t dst, uint32_t ch,
                                           const __nv_bfloat16* src, int Hs, int Ws, int nb) {
    constexpr int HP = C / 16;
    const int lane = threadIdx.x & 31, half = lane >> 4;
    int b0, y0, x0;
    raster_at(pl, p0, b0, y0, x0);
    for (int k = (threadIdx.x >> 5) * 16 + (lane & 15); k <= pl.S; k += WARPS * 16) {
        const long long q = raster_pixel(pl, b0, y0, x0, k, Hs, Ws, nb, 1, 0, 0, Ws, Hs);
        const __nv_bfloat16* s = src + (q < 0 ? 0 : q * C + 8 * HP * half);
        const uint32_t n = q < 0 ? 0u : 16u, d = dst + (uint32_t)(HP * half) * ch + (uint32_t)k * 16;
#pragma unroll
        for (int c = 0; c < HP; c++) {
            const __nv_bfloat16* sc = q < 0 ? s : s + 8 * c;
            if (k < pl.S) cp_async16(d + (uint32_t)c * ch, sc, n);
            if (k > 0) cp_async16(d + (uint32_t)(8 + c) * ch - 16, sc, n);
        }
    }
}

struct ConvArgs {
    const uint4* w;          // packed weights: the shared-memory image of B (ksteps x ncols x 16)
    const float* bias;       // ncols (or null)
    const __nv_bfloat16* mask;  // null, or an NHWC activation with nout channels: output *= (mask > 0)
    void* y;                 // output, NHWC with nout channels (BF16, or FP32 with out_f32)
    int B, Hin, Win, Hout, Wout, nout;
    int relu, out_f32;
    const __nv_bfloat16* x;  // input activation, NHWC with cin channels
    int* err;
};

// zero the BF16 halves of v whose mask value is not > 0
__device__ __forceinline__ uint32_t mask_bf16x2(uint32_t v, uint32_t m) {
    const bool lo = __uint_as_float(m << 16) > 0.0f, hi = __uint_as_float(m & 0xFFFF0000u) > 0.0f;
    return (lo ? (v & 0xFFFFu) : 0u) | (hi ? (v & 0xFFFF0000u) : 0u);
}

// The accumulator of tap t: the up mapping keeps one per parity class (oy, ox) of the output
// pixel, 2 oy + ox, and each class takes only the taps that read a pixel for it.
template <int MODE>
__host__ __device__ constexpr int tap_class(int t) {
    return MODE == kUp ? 2 * ((t / 3) != 1 ? 1 : 0) + ((t % 3) != 1 ? 1 : 0) : 0;
}

// Forward / data-gradient convolution, all output columns (NCOL, a multiple of 16) at once.
// A CTA holds the whole K of weights in shared memory and walks steps of T tiles of 128
// raster positions (up mapping: one tile, four output pixels per position).  One warp issues
// the MMAs; sixteen copy tiles and write results, two steps in flight: while the tensor cores
// multiply step i + 1 from one buffer into one half of the tensor memory, the workers copy
// step i + 2 into the other buffer and write step i out of the other half.
// What bounds it: with 48 columns an MMA takes 44 cycles (32 of them to read its 4 KB of A
// from shared memory), 27 MMAs per 128 pixels, 50 us on 1.49M pixels of 48 channels; HBM is 44
// us there.  Measured on that layer (48 -> 48, same size): 98 us (2.9 TB/s of activations);
// copying a tile per tap (every pixel nine times, 16 bytes a lane) took 294 us, the
// tile once but the MMAs issued by a worker thread 133 us.
// Every output row leaves as full 32-byte sectors: neighbouring lanes swap halves of their 16
// columns, so that two lanes write one row's 32 bytes in one instruction.
template <int MODE, int CIN, int NCOL>
__global__ void __launch_bounds__(kConvThreads, 1) k_conv_tc(const __grid_constant__ ConvArgs a,
                                                             const __grid_constant__ TilePlan pl) {
    constexpr int CB = CIN / 16, KSTEPS = 9 * CB;
    constexpr int B_STEP = NCOL * 32;            // bytes of B per K step
    constexpr int CLS = MODE == kUp ? 4 : 1;
    constexpr uint32_t SETC = 4 * NCOL;          // tensor-memory columns of a step (at most 4 accumulators)
    constexpr uint32_t TCOLS = 2 * SETC <= 128 ? 128 : 512;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* sB = smem;
    float* sBias = reinterpret_cast<float*>(sB + KSTEPS * B_STEP);
    const uint32_t ch = (uint32_t)pl.npix * 16;  // plane stride
    const uint32_t buf0 = smem_u32(smem + KSTEPS * B_STEP + NCOL * 4), bufsz = ch * (CIN / 8);
    __shared__ uint64_t m_full[2], m_free[2], m_done[2];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_fail;
    const int tid = threadIdx.x, warp = (int)uniform(tid >> 5), lane = tid & 31;
    const int na = pl.T * CLS;  // accumulators of a step
    auto fill = [&](long long st, uint32_t buf) {
        const long long p0 = pl.p_first + st * (kTile * pl.T);
        for (int q = 0; q < pl.nseg; q++)
            fill_seg<CIN, kConvWorkers / 32>(pl, pl.seg[q], p0, buf, ch, a.x, a.Hin, a.Win, a.B, pl.sub);
    };
    const long long st0 = blockIdx.x, G = gridDim.x;
    const bool worker = warp < kConvWorkers / 32;
    if (worker) {
        fill(st0, buf0);
        // weights: a straight copy of the packed image; the bias (zero beyond nout)
        for (int q = tid; q < KSTEPS * B_STEP / 16; q += kConvWorkers) reinterpret_cast<uint4*>(sB)[q] = a.w[q];
        for (int c = tid; c < NCOL; c += kConvWorkers) sBias[c] = (a.bias && c < a.nout) ? a.bias[c] : 0.0f;
        if (st0 + G < pl.nstep) fill(st0 + G, buf0 + bufsz);
        cp_async_commit();
    } else {
        if (lane == 0) {
            for (int k = 0; k < 2; k++) {
                mbar_init(&m_full[k], kConvWorkers / 32);
                mbar_init(&m_free[k], kConvWorkers / 32);
                mbar_init(&m_done[k], 1);
            }
            s_fail = 0;
        }
        __syncwarp();
        tmem_alloc(&s_tmem, TCOLS);
    }
    cp_async_wait_all();
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = uniform(s_tmem);
    const uint32_t b0 = smem_u32(sB);
    constexpr uint32_t idesc = instr_desc(kTile, NCOL);
    const int nout = a.nout, odd = lane & 1;
    const bool vec = !a.out_f32 && nout % 8 == 0 && !(reinterpret_cast<uintptr_t>(a.y) & 15) &&
                     !(reinterpret_cast<uintptr_t>(a.mask) & 15);
    // buffer / accumulator set k of step i is i & 1; a set's r-th use has parity r & 1
    int i = 0;
    bool ok = true;
    if (!worker) {
        // ---- the MMA warp: a step once its tile is copied (the first two were, above) and its
        // accumulators have been read; the MMAs' completion arrives on m_done
        const bool lead = elect_one();
        for (long long st = st0; st < pl.nstep; st += G, i++) {
            const int set = i & 1;
            const uint32_t use = (uint32_t)(i >> 1);
            if (i >= 2) {
                ok = mbar_wait(&m_full[set], (use + 1) & 1, &s_fail) && mbar_wait(&m_free[set], (use + 1) & 1, &s_fail);
                if (!__all_sync(0xffffffffu, ok)) break;
                tc_fence_after();
            }
            const uint32_t buf = buf0 + (uint32_t)set * bufsz;
            const uint32_t d0 = tmem + (uint32_t)set * SETC;
            for (int tt = 0; tt < pl.T; tt++) {
                if (st * (kTile * pl.T) + tt * kTile >= pl.nflat) break;
                int seen = 0;
#pragma unroll
                for (int t = 0; t < 9; t++) {
                    const int cls = tap_class<MODE>(t);
#pragma unroll
                    for (int cb = 0; cb < CB; cb++) {
                        const uint32_t aa = buf + (uint32_t)(pl.tap[t] + tt * kTile) * 16 + (uint32_t)(2 * cb) * ch;
                        if (lead)
                            mma_bf16(d0 + (uint32_t)((tt * CLS + cls) * NCOL), smem_desc(aa, ch, 128),
                                     smem_desc(b0 + (t * CB + cb) * B_STEP, 128, 256), idesc, (seen >> cls) & 1);
                        seen |= 1 << cls;
                    }
                }
            }
            if (lead) mma_commit(&m_done[set]);
            __syncwarp();
        }
    }
    for (long long st = st0; worker && st < pl.nstep; st += G, i++) {
        const int set = i & 1;
        ok = mbar_wait(&m_done[set], (uint32_t)(i >> 1) & 1, &s_fail);
        if (!__all_sync(0xffffffffu, ok)) break;
        tc_fence_after();
        // this step's tile has been read: step i + 2 is copied under the epilogue
        const bool more = st + 2 * G < pl.nstep;
        if (more) fill(st + 2 * G, buf0 + (uint32_t)set * bufsz);
        cp_async_commit();
        // ---- epilogue: warp w reads tensor-memory lanes 32 (w % 4)..+31 (the lanes its
        // sub-partition may access); its group takes a contiguous share of the
        // (accumulator, 16 columns) units
        constexpr int NB = NCOL / 16;
        const int units = na * NB, per = (units + kConvGroups - 1) / kConvGroups;
        const int u0 = (warp >> 2) * per, u1 = min(u0 + per, units);
        const long long p0 = st * (kTile * pl.T);
        int last_tile = -1, b = 0, y = 0, x = 0;
        for (int u = u0; u < u1; u++) {  // warp-uniform
            const int acc = u / NB, c0 = (u % NB) * 16, tile = acc / CLS, cls = acc % CLS;
            if (p0 + tile * kTile >= pl.nflat) break;
            if (tile != last_tile) {
                raster_at(pl, p0 + tile * kTile + (warp & 3) * 32 + lane, b, y, x);
                last_tile = tile;
            }
            const int oy = MODE == kUp ? 2 * y + (cls >> 1) : y, ox = MODE == kUp ? 2 * x + (cls & 1) : x;
            const bool live = b < a.B && oy < a.Hout && ox < a.Wout;
            const int pix = live ? (b * a.Hout + oy) * a.Wout + ox : -1;  // the host keeps the pixel count below 2^31
            float v[16];
            tmem_ld16(tmem + (uint32_t)set * SETC + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(acc * NCOL + c0), v);
#pragma unroll
            for (int k = 0; k < 16; k++) {
                v[k] += sBias[c0 + k];
                if (a.relu) v[k] = fmaxf(v[k], 0.0f);
            }
            if (vec && c0 + 16 <= nout) {
                uint32_t w[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
                    w[k] = *reinterpret_cast<const uint32_t*>(&h);
                }
                uint32_t r[4];
#pragma unroll
                for (int k = 0; k < 4; k++) r[k] = __shfl_xor_sync(0xffffffffu, odd ? w[k] : w[4 + k], 1);
                const int other = __shfl_xor_sync(0xffffffffu, pix, 1);
                // the even lane's row, then the odd lane's: its first 16 bytes by the even
                // lane, its last by the odd
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int q = e == odd ? pix : other;
                    if (q < 0) continue;
                    uint4 o;
                    if (e == 0) o = odd ? make_uint4(r[0], r[1], r[2], r[3]) : make_uint4(w[0], w[1], w[2], w[3]);
                    else o = odd ? make_uint4(w[4], w[5], w[6], w[7]) : make_uint4(r[0], r[1], r[2], r[3]);
                    const long long el = (long long)q * nout + c0 + 8 * odd;
                    if (a.mask) {
                        const uint4 m = *reinterpret_cast<const uint4*>(a.mask + el);
                        o.x = mask_bf16x2(o.x, m.x);
                        o.y = mask_bf16x2(o.y, m.y);
                        o.z = mask_bf16x2(o.z, m.z);
                        o.w = mask_bf16x2(o.w, m.w);
                    }
                    *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.y) + el) = o;
                }
            } else if (live) {
#pragma unroll
                for (int k = 0; k < 16; k++) {
                    const int c = c0 + k;
                    if (c >= nout) break;
                    const long long el = (long long)pix * nout + c;
                    const bool keep = !a.mask || __bfloat162float(a.mask[el]) > 0.0f;
                    if (a.out_f32) reinterpret_cast<float*>(a.y)[el] = keep ? v[k] : 0.0f;
                    else reinterpret_cast<__nv_bfloat16*>(a.y)[el] = __float2bfloat16_rn(keep ? v[k] : 0.0f);
                }
            }
        }
        // this set's accumulators have been read; the next tile in its buffer is complete
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&m_free[set]);
        if (more) {
            cp_async_wait_all();
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&m_full[set]);
        }
    }
    cp_async_wait_all();  // no copy in flight past this point
    __syncthreads();
    if (s_fail) {
        if (tid == 0) atomicExch(a.err, 1);
        // MMAs may still be in flight: bounded waits for the completions before the memory is
        // freed (whichever parity the sets are in, one of the two passes at once)
        if (!worker) {
            int never = 0;
            for (int k = 0; k < 4; k++) mbar_wait(&m_done[k >> 1], k & 1, &never);
        }
        __syncthreads();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (!worker) tmem_free(tmem, TCOLS);
}

struct WgradArgs {
    const __nv_bfloat16* x;   // the layer's input activation, NHWC, cin channels
    const __nv_bfloat16* dy;  // gradient at the layer's output, NHWC, ncol channels
    int B, Hin, Win, Hout, Wout;
    int nout;                 // output channels to accumulate (<= NCOL)
    float* dw;                // [nout][9][cin] FP32, accumulated atomically
    int* err;
};

// The tap that row half h of accumulator q sums (-1: none).  Accumulator q = 2 r + s: r the
// tap row, s = 0 the pair of taps read at one place of the input, s = 1 the third.  Same-size
// and down: rows 64.. hold the output gradient one position further, so they sum the tap one
// input pixel back.  Up: they hold the odd output columns.
template <int MODE>
__host__ __device__ constexpr int wg_tap(int q, int h) {
    const int r = 3 * (q >> 1), s = q & 1;
    if (MODE == kSame) return s == 0 ? (h == 0 ? r + 2 : r + 1) : (h == 0 ? r : -1);  // dx +1, 0 | -1
    if (MODE == kDown) return s == 0 ? (h == 0 ? r + 2 : r) : (h == 0 ? r + 1 : -1);  // dx +1, -1 | 0
    return s == 0 ? (h == 0 ? r + 1 : r + 2) : (h == 0 ? -1 : r);                     // dx 0, +1 | -1
}

// The row half that sums tap t.
template <int MODE>
__device__ __forceinline__ int wg_half(int t) {
    for (int q = 0; q < 6; q++)
        if (wg_tap<MODE>(q, 1) == t) return 1;
    return 0;
}

// dW[n][t], all input channels, over the output pixels of raster positions p0..p1-1: each pixel's
// dY times the input pixel of the tap, times zero where the image has none.  Only for operands
// that are not finite (5.5 to 6.2 ms for a layer of 746k pixels of 48 channels, 0.1 ms with finite
// operands); U pixels' loads at a time, since a thread waits for each.
template <int MODE, int CIN, int NCOL>
__device__ __noinline__ void wgrad_tap(const WgradArgs& a, const TilePlan& pl, long long p0, long long p1, int n, int t) {
    constexpr int U = 2, V = CIN / 8;
    float sum[CIN];
#pragma unroll
    for (int k = 0; k < CIN; k++) sum[k] = 0.0f;
    const int dy = t / 3 - 1, dx = t % 3 - 1;
    int b, y, x;
    raster_at(pl, p0, b, y, x);
    // pixel by pixel: up, a position is four output pixels
    constexpr int per = MODE == kUp ? 4 : 1;
    const long long count = (p1 - p0) * per;
    int c = 0;  // which of them
    for (long long k0 = 0; k0 < count && b < a.B; k0 += U) {
        bool live[U];
        __nv_bfloat16 g[U];
        uint4 v[U][V];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int oy = MODE == kUp ? 2 * y + (c >> 1) : y, ox = MODE == kUp ? 2 * x + (c & 1) : x;
            live[u] = b >= 0 && b < a.B && oy < a.Hout && ox < a.Wout && k0 + u < count;
            int iy = MODE == kDown ? 2 * oy + dy : oy + dy, ix = MODE == kDown ? 2 * ox + dx : ox + dx;
            bool in = live[u];
            if (MODE == kUp) {
                in = in && !((oy - dy) & 1) && !((ox - dx) & 1);
                iy = (oy - dy) >> 1;
                ix = (ox - dx) >> 1;
            }
            in = in && iy >= 0 && iy < a.Hin && ix >= 0 && ix < a.Win;
            g[u] = a.dy[live[u] ? (((long long)b * a.Hout + oy) * a.Wout + ox) * NCOL + n : 0];
            const uint4* px = reinterpret_cast<const uint4*>(a.x + (in ? (((long long)b * a.Hin + iy) * a.Win + ix) * CIN : 0));
#pragma unroll
            for (int k = 0; k < V; k++) v[u][k] = in ? px[k] : make_uint4(0, 0, 0, 0);
            if (++c < per) continue;
            c = 0;
            if (++x < pl.Wp) continue;
            x = 0;
            if (++y < pl.Hp) continue;
            y = 0;
            b++;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (!live[u]) continue;
            const float f = __bfloat162float(g[u]);
#pragma unroll
            for (int k = 0; k < V; k++) {
                const uint32_t w[4] = {v[u][k].x, v[u][k].y, v[u][k].z, v[u][k].w};
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    sum[8 * k + 2 * m] = fmaf(f, __uint_as_float(w[m] << 16), sum[8 * k + 2 * m]);
                    sum[8 * k + 2 * m + 1] = fmaf(f, __uint_as_float(w[m] & 0xFFFF0000u), sum[8 * k + 2 * m + 1]);
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < CIN; k++) atomicAdd(a.dw + ((size_t)n * 9 + t) * CIN + k, sum[k]);
}

// Weight gradient: dW[n][t][ci] = sum_p dY[p][n] X[map(p, t)][ci].  MMAs with M = 128 rows (two
// blocks of 64: the output channels n of two taps), N = the CIN input channels and K = 16
// raster positions; both operands MN-major from planes of 8 channels, the taps as shifted
// start addresses, six accumulators (wg_tap) for the nine taps.  A CTA takes a contiguous run
// of steps of S positions, two steps in flight.  The tensor memory is read and cleared every
// kWgChain positions into registers, so a chain of FP32 additions in it is no longer than
// 128 MMAs, and the registers are added to dw once, with vector atomics.
// What bounds it: 6 MMAs of 44 cycles (operand reads from shared memory) per 16 positions, 81
// us for 1.49M pixels of 48 channels.  Measured there: 171 us; gathering every operand element
// by 2-byte loads, one thread per (tap, channel), took 3.13 ms.
// The raster's padding holds a zero output gradient beside real input pixels, so an input that is
// not finite next to an image's edge makes taps non-finite that never meet it.  A CTA whose sums
// are not all finite adds its output pixels one by one instead (wgrad_tap).
template <int MODE, int CIN, int NCOL>
__global__ void __launch_bounds__(kWgThreads, 1) k_conv_wgrad_tc(const __grid_constant__ WgradArgs a,
                                                                 const __grid_constant__ TilePlan pl,
                                                                 int steps_per_cta) {
    constexpr int NQ = 6;
    constexpr uint32_t TCOLS = NQ * CIN <= 128 ? 128 : 512;
    constexpr int YREG = MODE == kUp ? 2 : 1;     // output-gradient regions (up: even and odd output rows)
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t chx = (uint32_t)pl.npix * 16, chy = (uint32_t)pl.S * 16;
    const uint32_t ysz = YREG * 16 * chy, bufsz = ysz + chx * (CIN / 8);
    const uint32_t buf0 = smem_u32(smem);
    __shared__ uint64_t m_full[2], m_done[2], m_free;
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_fail;
    const int tid = threadIdx.x, warp = (int)uniform(tid >> 5), lane = tid & 31;
    const long long s0 = (long long)blockIdx.x * steps_per_cta;
    const long long s1 = s0 + steps_per_cta < pl.nstep ? s0 + steps_per_cta : pl.nstep;
    auto fill = [&](long long st, uint32_t buf) {
        const long long p0 = pl.p_first + st * pl.S;
        // the output gradient: planes 0.. and 8.. of each region (up: the parity sub-images of
        // the output, whose padding lies outside the output image)
        if (MODE == kUp) {
            for (int r = 0; r < YREG; r++)
                for (int h = 0; h < 2; h++)
                    fill_seg<NCOL, kWgWorkers / 32>(pl, TileSeg{0, pl.S, 0, r, h}, p0,
                                                    buf + (uint32_t)(r * 16 + h * 8) * chy, chy, a.dy, a.Hout, a.Wout,
                                                    a.B, 2);
        } else {
            fill_twice<NCOL, kWgWorkers / 32>(pl, p0, buf, chy, a.dy, a.Hout, a.Wout, a.B);
        }
        for (int q = 0; q < pl.nseg; q++)
            fill_seg<CIN, kWgWorkers / 32>(pl, pl.seg[q], p0, buf + ysz, chx, a.x, a.Hin, a.Win, a.B, pl.sub);
    };
    // the rows of the operand planes that no channel fills (NCOL..63 of each block) give
    // accumulator rows that are never read; they are cleared once so that they stay finite
    for (uint32_t q = tid * 16; q < 2 * bufsz; q += kWgThreads * 16)
        *reinterpret_cast<uint4*>(smem + q) = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const bool worker = warp < kWgWorkers / 32;
    if (worker) {
        fill(s0, buf0);
        if (s0 + 1 < s1) fill(s0 + 1, buf0 + bufsz);
        cp_async_commit();
    } else {
        if (lane == 0) {
            for (int k = 0; k < 2; k++) {
                mbar_init(&m_full[k], kWgWorkers / 32);
                mbar_init(&m_done[k], 1);
            }
            mbar_init(&m_free, kWgWorkers / 32);
            s_fail = 0;
        }
        __syncwarp();
        tmem_alloc(&s_tmem, TCOLS);
    }
    cp_async_wait_all();
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = uniform(s_tmem);
    constexpr uint32_t idesc = instr_desc(kTile, CIN, 1);
    const int chain = kWgChain / pl.S;  // steps per tensor-memory chain
    constexpr int NB = CIN / 16, UN = NQ * NB / kWgGroups;  // (accumulator, 16 columns) units per group
    float acc[UN][16];
#pragma unroll
    for (int u = 0; u < UN; u++)
#pragma unroll
        for (int k = 0; k < 16; k++) acc[u][k] = 0.0f;
    bool ok = true;
    const int n_steps = (int)(s1 - s0);
    if (!worker) {
        const bool lead = elect_one();
        for (int i = 0; i < n_steps; i++) {
            const int set = i & 1;
            const bool first = i % chain == 0;  // a new chain: the accumulators have been read
            if (i >= 2) ok = mbar_wait(&m_full[set], (uint32_t)((i >> 1) + 1) & 1, &s_fail);
            if (ok && first && i > 0) ok = mbar_wait(&m_free, (uint32_t)(i / chain - 1) & 1, &s_fail);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after();
            const uint32_t by = buf0 + (uint32_t)set * bufsz, bx = by + ysz;
            for (int s = 0; s < pl.S / 16; s++) {
#pragma unroll
                for (int q = 0; q < NQ; q++) {
                    const int r = MODE == kUp ? (q >= 2 && q < 4 ? 0 : 1) : 0;  // up: dy = 0 reads the even output rows
                    if (lead)
                        mma_bf16(tmem + q * CIN, smem_desc(by + (uint32_t)r * 16 * chy + s * 256, 128, chy),
                                 smem_desc(bx + (uint32_t)(pl.tap[q] + 16 * s) * 16, 128, chx), idesc,
                                 !(first && s == 0));
                }
            }
            if (lead) mma_commit(&m_done[set]);
            __syncwarp();
        }
    }
    for (int i = 0; worker && i < n_steps; i++) {
        const int set = i & 1;
        ok = mbar_wait(&m_done[set], (uint32_t)(i >> 1) & 1, &s_fail);
        if (!__all_sync(0xffffffffu, ok)) break;
        tc_fence_after();
        const bool more = i + 2 < n_steps;
        if (more) fill(s0 + i + 2, buf0 + (uint32_t)set * bufsz);
        cp_async_commit();
        if ((i + 1) % chain == 0 || i + 1 == n_steps) {
#pragma unroll
            for (int u = 0; u < UN; u++) {
                float v[16];
                tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(((warp >> 2) * UN + u) * 16), v);
#pragma unroll
                for (int k = 0; k < 16; k++) acc[u][k] += v[k];
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&m_free);
        }
        if (more) {
            cp_async_wait_all();
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&m_full[set]);
        }
    }
    cp_async_wait_all();
    const int row = (warp & 3) * 32 + lane, h = row >> 6, n = row & 63;
    bool finite = true;
    if (worker && n < a.nout) {
#pragma unroll
        for (int u = 0; u < UN; u++) {
            if (wg_tap<MODE>(((warp >> 2) * UN + u) / NB, h) < 0) continue;
#pragma unroll
            for (int k = 0; k < 16; k++) finite = finite && isfinite(acc[u][k]);
        }
    }
    const bool pixels = __syncthreads_or(!finite);
    if (s_fail) {
        if (tid == 0) atomicExch(a.err, 1);
        if (!worker) {  // as in k_conv_tc
            int never = 0;
            for (int k = 0; k < 4; k++) mbar_wait(&m_done[k >> 1], k & 1, &never);
        }
        __syncthreads();
    } else if (worker && pixels) {
        for (int k = warp; k < 9 * ((a.nout + 31) / 32); k += kWgWorkers / 32) {
            const int t = k % 9, nn = k / 9 * 32 + lane;
            // rows 64..: one position further (fill_twice)
            const long long p0 = pl.p_first + s0 * pl.S + (MODE == kUp ? 0 : wg_half<MODE>(t));
            if (nn < a.nout) wgrad_tap<MODE, CIN, NCOL>(a, pl, p0, p0 + (s1 - s0) * pl.S, nn, t);
        }
    } else if (worker && n < a.nout) {
        const bool v4 = !(reinterpret_cast<uintptr_t>(a.dw) & 15);
#pragma unroll
        for (int u = 0; u < UN; u++) {
            const int c = (warp >> 2) * UN + u, q = c / NB;
            const int t = wg_tap<MODE>(q, h);
            if (t < 0) continue;
            float* d = a.dw + ((size_t)n * 9 + t) * CIN + (c % NB) * 16;
            if (v4) {
#pragma unroll
                for (int k = 0; k < 16; k += 4)
                    atomicAdd(reinterpret_cast<float4*>(d + k),
                              make_float4(acc[u][k], acc[u][k + 1], acc[u][k + 2], acc[u][k + 3]));
            } else {
#pragma unroll
                for (int k = 0; k < 16; k++) atomicAdd(d + k, acc[u][k]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (!worker) tmem_free(tmem, TCOLS);
}

// Bias gradient: db[n] += sum over pixels of dY[p][n] (NHWC, ncol channels, a multiple of 8, 16-
// byte aligned rows), FP32.  A thread loads 16 bytes (8 channels) of every blockDim.y-th pixel
// of the grid into registers, four pixels in flight; a CTA's threads are added in shared memory
// and its sums to db with one atomic per channel.  Bound by HBM (143 MB at 1.49M pixels of 48
// channels: 22 us).
constexpr int kBiasPix = 32;  // pixels of a CTA (threads per channel block)
__global__ void __launch_bounds__(1024) k_bias_grad8(const uint4* __restrict__ dy, long long npix, int nout, float* db) {
    extern __shared__ float s_part[];  // [kBiasPix][8 blockDim.x]
    const int C8 = blockDim.x, c = threadIdx.x;
    float acc[8] = {};
    auto add = [&](const uint4& q) {
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            acc[2 * k] += __uint_as_float(w[k] << 16);
            acc[2 * k + 1] += __uint_as_float(w[k] & 0xFFFF0000u);
        }
    };
    const long long step = (long long)gridDim.x * kBiasPix;
    long long p = (long long)blockIdx.x * kBiasPix + threadIdx.y;
    for (; p + 3 * step < npix; p += 4 * step) {
        uint4 q[4];
#pragma unroll
        for (int k = 0; k < 4; k++) q[k] = dy[(p + k * step) * C8 + c];
#pragma unroll
        for (int k = 0; k < 4; k++) add(q[k]);
    }
    for (; p < npix; p += step) add(dy[p * C8 + c]);
#pragma unroll
    for (int k = 0; k < 8; k++) s_part[threadIdx.y * 8 * C8 + 8 * c + k] = acc[k];
    __syncthreads();
    const int t = threadIdx.y * C8 + c;
    if (t < nout) {
        float sum = 0.0f;
        for (int y = 0; y < kBiasPix; y++) sum += s_part[y * 8 * C8 + t];
        atomicAdd(&db[t], sum);
    }
}

// The same for any ncol and alignment.
__global__ void k_bias_grad(const __nv_bfloat16* dy, long long npix, int ncol, int nout, float* db) {
    __shared__ float acc[256];
    for (int c = threadIdx.x; c < nout; c += blockDim.x) acc[c] = 0.0f;
    __syncthreads();
    for (long long p = blockIdx.x * (long long)blockDim.y + threadIdx.y; p < npix; p += (long long)gridDim.x * blockDim.y)
        for (int c = threadIdx.x; c < nout; c += blockDim.x) atomicAdd(&acc[c], __bfloat162float(dy[p * ncol + c]));
    __syncthreads();
    for (int c = threadIdx.x; c < nout; c += blockDim.x)
        if (threadIdx.y == 0) atomicAdd(&db[c], acc[c]);
}

// Masked mean-squared error of FP32 predictions (npix x nc) against targets, weighted per
// pixel: loss += sum w (pred - tgt)^2 * scale; dY (BF16, npix x ncol, zero beyond nc) =
// 2 w (pred - tgt) * scale.  Bound by HBM (60 bytes a pixel for 3 of 16 channels); 2-byte stores
// took 185 us for 1.49M pixels.
template <bool WIDE>
__global__ void k_mse_grad(const float* pred, const float* tgt, const float* wgt, long long npix, int nc, int ncol,
                           float scale, __nv_bfloat16* dy, float* loss) {
    float l = 0.0f;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < npix; p += (long long)gridDim.x * blockDim.x) {
        const float w = wgt ? wgt[p] : 1.0f;
        if (WIDE) {  // nc <= 4, ncol a multiple of 8, dy 16-byte aligned: 16-byte stores
            uint32_t o[2] = {0u, 0u};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                if (c >= nc) break;
                const float d = pred[p * nc + c] - tgt[p * nc + c];
                l += w * d * d * scale;
                o[c >> 1] |= (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(2.0f * w * d * scale)) << (16 * (c & 1));
            }
            uint4* q = reinterpret_cast<uint4*>(dy + p * ncol);
            q[0] = make_uint4(o[0], o[1], 0u, 0u);
            for (int k = 1; k < ncol / 8; k++) q[k] = make_uint4(0u, 0u, 0u, 0u);
            continue;
        }
        for (int c = 0; c < ncol; c++) {
            float g = 0.0f;
            if (c < nc) {
                const float d = pred[p * nc + c] - tgt[p * nc + c];
                l += w * d * d * scale;
                g = 2.0f * w * d * scale;
            }
            dy[p * ncol + c] = __float2bfloat16_rn(g);
        }
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, l);
}

int sm_count() {
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}
constexpr int kSmemMax = 232448 - 1024;  // dynamic shared memory of a CTA (227 KB less the static part)

// Lets kernel f be launched with any plan's shared memory.  Always the same limit: it is the
// context's, shared by every thread, and one lowered to a small image's plan would fail the
// launch that another thread makes for a large one.
template <class F>
cudaError_t allow_smem(F* f) {
    return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
}

FastDiv fast_div(uint32_t d) {
    int l = 0;
    while ((1ull << l) < d) l++;
    if (l == 0) return FastDiv{0, 0, 1};
    return FastDiv{(uint32_t)(((1ull << (31 + l)) + d - 1) / d), (uint32_t)(l - 1), 0};
}

int round8(int n) { return (n + 7) / 8 * 8; }

// The raster of a layer: positions are output pixels (up: 2 x 2 blocks of them), with a
// padding column and row where a tap can step out of the image and no wider than needed.
TilePlan raster(int mode, int B, int Hin, int Win, int Hout, int Wout) {
    TilePlan pl{};
    pl.sub = mode == kDown ? 2 : 1;
    if (mode == kUp) {  // taps read the block's own input pixel and the next ones
        pl.Wp = (Wout + 1) / 2 + 1;
        pl.Hp = (Hout + 1) / 2 + 1;
        pl.xlim = pl.Wp;
        pl.ylim = pl.Hp;
    } else {
        // the column after the last output is both x = -1 of the next row (padding) and
        // x = Wout of this one, an input pixel only when the input is wider than the output:
        // then they get a column each (rows alike).  Down reads no pixel past its last output.
        pl.Wp = Wout + (mode != kDown && Win > Wout ? 2 : 1);
        pl.Hp = Hout + (mode != kDown && Hin > Hout ? 2 : 1);
        pl.xlim = pl.Wp - 1;
        pl.ylim = pl.Hp - 1;
    }
    const long long per = (long long)pl.Hp * pl.Wp;
    pl.nflat = B * per;
    pl.dW = fast_div(pl.Wp);
    pl.dH = fast_div(pl.Hp);
    pl.dI = fast_div(per < (1LL << 31) ? (uint32_t)per : 1u);  // read only where positions fit 31 bits
    // positions up to a step past the end, counted from one image before the start
    pl.small = pl.nflat + 2 * per + 8192 < (1LL << 31);
    return pl;
}

int add_seg(TilePlan& pl, int start, int len, int py, int px) {
    TileSeg& s = pl.seg[pl.nseg++];
    s = TileSeg{start, len, pl.npix, py, px};
    pl.npix += round8(len);
    return s.off;
}

// The segments that taps (sy in [sy0, sy1], sx in [sx0, sx1]) of n positions read of
// sub-image (py, px): one run over all rows of the taps, or one run per row when the raster
// rows are long enough for that to be fewer pixels.  row[sy - sy0]: the tile pixel that tap
// (sy, sx0) of the first position reads.
void tap_rows(TilePlan& pl, int n, int sy0, int sy1, int sx0, int sx1, int py, int px, int* row) {
    const int one = n + (sy1 - sy0) * pl.Wp + (sx1 - sx0), per = n + sx1 - sx0;
    if (one <= (sy1 - sy0 + 1) * round8(per)) {
        const int off = add_seg(pl, sy0 * pl.Wp + sx0, one, py, px);
        for (int s = sy0; s <= sy1; s++) row[s - sy0] = off + (s - sy0) * pl.Wp;
    } else {
        for (int s = sy0; s <= sy1; s++) row[s - sy0] = add_seg(pl, s * pl.Wp + sx0, per, py, px);
    }
}

// Segments and tap offsets of n positions per step (tap t at tap9[t]).
void tap_layout(TilePlan& pl, int mode, int n, int (&tap9)[9]) {
    pl.nseg = pl.npix = 0;
    int row[3];
    if (mode == kSame || mode == kSameAdj) {
        tap_rows(pl, n, -1, 1, -1, 1, 0, 0, row);
        for (int t = 0; t < 9; t++) {
            const int s = mode == kSame ? t : 8 - t;  // the adjoint reads the mirrored tap
            tap9[t] = row[s / 3] + s % 3;
        }
    } else if (mode == kUp) {
        tap_rows(pl, n, 0, 1, 0, 1, 0, 0, row);
        // output row 2a + 1 reads input row a + 1 through dy = -1 and row a through dy = 1
        for (int t = 0; t < 9; t++) tap9[t] = row[t / 3 == 0 ? 1 : 0] + (t % 3 == 0 ? 1 : 0);
    } else {
        // dy = 0 reads the even sub-image, dy = +-1 the odd one at this row or the row before
        for (int py = 0; py < 2; py++)
            for (int px = 0; px < 2; px++) {
                tap_rows(pl, n, py ? -1 : 0, 0, px ? -1 : 0, 0, py, px, row);
                for (int t = 0; t < 9; t++) {
                    const int dy = t / 3 - 1, dx = t % 3 - 1;
                    if ((dy != 0) != py || (dx != 0) != px) continue;
                    tap9[t] = (py ? row[dy == -1 ? 0 : 1] : row[0]) + (px && dx == 1 ? 1 : 0);
                }
            }
    }
}

// Tiles per step: up to 4 accumulators in each half of the tensor memory.  Of the shapes whose
// two buffers fit, the one with the least tiles on the busiest CTA, the larger on ties (its
// halo costs less); a batch of small crops thus spreads over the SMs.
template <int MODE>
TilePlan conv_plan(int B, int Hin, int Win, int Hout, int Wout, int cin, size_t fixed, int nsm, size_t* smem) {
    TilePlan best{};
    long long cost = -1;
    for (int T = MODE == kUp ? 1 : (MODE == kDown ? 2 : 4); T >= 1; T >>= 1) {
        TilePlan pl = raster(MODE, B, Hin, Win, Hout, Wout);
        tap_layout(pl, MODE, kTile * T, pl.tap);
        const size_t bytes = fixed + 2 * (size_t)pl.npix * cin * 2;
        if (bytes > (size_t)kSmemMax) continue;
        pl.T = T;
        pl.nstep = (pl.nflat + kTile * T - 1) / (kTile * T);
        const long long c = (pl.nstep + nsm - 1) / nsm * T;
        if (cost < 0 || c < cost) {
            best = pl;
            cost = c;
            *smem = bytes;
        }
    }
    return best;
}

// The packed weight image of a layer (hyd_conv_forward): element (n, k = t cinp + c) of w (n < nout,
// c < cin; element strides sn, st, sc) as BF16, zero beyond, at its place in K step k / 16.
__global__ void k_pack_weights(const float* __restrict__ w, int nout, int cin, long long sn, long long st, long long sc,
                               int ncol, int cinp, __nv_bfloat16* __restrict__ img) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ncol * 9 * cinp) return;
    // i: position in the image
    const int s = i / (ncol * 16), r = i % (ncol * 16);
    const int n = (r / 128) * 8 + (r / 8) % 8, kk = ((r / 64) % 2) * 8 + r % 8;
    const int k = s * 16 + kk, t = k / cinp, c = k % cinp;
    img[i] = __float2bfloat16_rn(n < nout && c < cin ? w[n * sn + t * st + c * sc] : 0.0f);
}

template <int MODE, int CIN, int NCOL>
cudaError_t launch_conv(const ConvArgs& a, cudaStream_t s) {
    const int nsm = sm_count();
    size_t smem = 0;
    const TilePlan pl = conv_plan<MODE>(a.B, a.Hin, a.Win, a.Hout, a.Wout, CIN, (size_t)(9 * CIN / 16) * NCOL * 32 + NCOL * 4,
                                        nsm, &smem);
    if (pl.T == 0) return cudaErrorInvalidConfiguration;
    cudaError_t e = allow_smem(k_conv_tc<MODE, CIN, NCOL>);
    if (e != cudaSuccess) return e;
    const int grid = (int)(pl.nstep < nsm ? pl.nstep : nsm);
    k_conv_tc<MODE, CIN, NCOL><<<grid, kConvThreads, smem, s>>>(a, pl);
    hyd_kernel_launches_add(1);
    return cudaGetLastError();
}

template <int MODE>
cudaError_t dispatch_conv(const ConvArgs& a, int cin, int ncol, cudaStream_t s) {
    if (cin == 16 && ncol == 48) return launch_conv<MODE, 16, 48>(a, s);
    if (cin == 48 && ncol == 48) return launch_conv<MODE, 48, 48>(a, s);
    if (cin == 48 && ncol == 16) return launch_conv<MODE, 48, 16>(a, s);
    return cudaErrorInvalidValue;
}

// Positions per step: 256 where two buffers fit, else 128.
template <int MODE>
TilePlan wgrad_plan(int B, int Hin, int Win, int Hout, int Wout, int cin, size_t* smem) {
    for (int S = 256; S >= 128; S >>= 1) {
        TilePlan pl = raster(MODE, B, Hin, Win, Hout, Wout);
        int tap9[9];
        tap_layout(pl, MODE, S, tap9);
        // accumulator q reads the input where its rows 0..63 (or, where they sum nothing, rows
        // 64..) need it
        for (int q = 0; q < 6; q++) pl.tap[q] = tap9[wg_tap<MODE>(q, 0) >= 0 ? wg_tap<MODE>(q, 0) : wg_tap<MODE>(q, 1)];
        pl.S = S;
        // same-size and down sum position p + 1 in rows 64..: from -1, so that position 0 is met
        pl.p_first = MODE == kUp ? 0 : -1;
        pl.nstep = (pl.nflat - pl.p_first + S - 1) / S;
        *smem = 2 * ((size_t)(MODE == kUp ? 2 : 1) * 16 * S * 16 + (size_t)pl.npix * cin * 2);
        if (*smem <= (size_t)kSmemMax) return pl;
    }
    return TilePlan{};
}

template <int MODE, int CIN, int NCOL>
cudaError_t launch_wgrad(const WgradArgs& a, cudaStream_t s) {
    if ((long long)a.B * a.Hout * a.Wout < 1) return cudaErrorInvalidConfiguration;
    size_t smem = 0;
    const TilePlan pl = wgrad_plan<MODE>(a.B, a.Hin, a.Win, a.Hout, a.Wout, CIN, &smem);
    if (pl.S == 0) return cudaErrorInvalidConfiguration;
    cudaError_t e = allow_smem(k_conv_wgrad_tc<MODE, CIN, NCOL>);
    if (e != cudaSuccess) return e;
    const int nsm = sm_count();
    const int per = (int)((pl.nstep + nsm - 1) / nsm);
    k_conv_wgrad_tc<MODE, CIN, NCOL><<<(unsigned)((pl.nstep + per - 1) / per), kWgThreads, smem, s>>>(a, pl, per);
    hyd_kernel_launches_add(1);
    return cudaGetLastError();
}

template <int MODE>
cudaError_t dispatch_wgrad(const WgradArgs& a, int cin, int ncol, cudaStream_t s) {
    if (ncol != 48 && ncol != 16) return cudaErrorInvalidValue;
    if (cin == 48) return ncol == 48 ? launch_wgrad<MODE, 48, 48>(a, s) : launch_wgrad<MODE, 48, 16>(a, s);
    return ncol == 48 ? launch_wgrad<MODE, 16, 48>(a, s) : launch_wgrad<MODE, 16, 16>(a, s);
}

// An aligned stand-in for a device array that does not start on a 16-byte boundary (the tiles
// are copied 16 bytes at a time); freed by the caller in stream order.
cudaError_t align16(const void** p, size_t bytes, void** tmp, cudaStream_t s) {
    *tmp = nullptr;
    if (!(reinterpret_cast<uintptr_t>(*p) & 15)) return cudaSuccess;
    cudaError_t e = cudaMallocAsync(tmp, bytes, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(*tmp, *p, bytes, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) *p = *tmp;
    return e;
}

}  // namespace

extern "C" {

int hyd_conv_forward(const void* x, int B, int Hin, int Win, int cin, const void* w_packed, const float* bias,
                     int ncol, int nout, int mode, int relu, const void* mask, void* y, int Hout, int Wout,
                     int out_f32, int* err, void* stream) {
    if (!x || !w_packed || !y || !err || B < 1 || Hin < 1 || Win < 1 || Hout < 1 || Wout < 1) return HYD_EINVAL;
    if (nout < 1 || nout > ncol) return HYD_EINVAL;
    if ((long long)B * Hout * Wout >= (1LL << 31)) return HYD_EINVAL;  // 32-bit pixel indices in the gather
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w_packed) & 15)) return HYD_EINVAL;
    ConvArgs a{(const uint4*)w_packed, bias, (const __nv_bfloat16*)mask, y, B, Hin, Win, Hout, Wout, nout, relu,
               out_f32, (const __nv_bfloat16*)x, err};
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e;
    switch (mode) {
        case HYD_CONV_SAME: e = dispatch_conv<kSame>(a, cin, ncol, s); break;
        case HYD_CONV_SAME_ADJ: e = dispatch_conv<kSameAdj>(a, cin, ncol, s); break;
        case HYD_CONV_DOWN: e = dispatch_conv<kDown>(a, cin, ncol, s); break;
        case HYD_CONV_UP: e = dispatch_conv<kUp>(a, cin, ncol, s); break;
        default: return HYD_EINVAL;
    }
    return e == cudaSuccess ? HYD_OK : (e == cudaErrorInvalidValue ? HYD_EINVAL : HYD_ECUDA);
}

int hyd_conv_wgrad(const void* x, int B, int Hin, int Win, int cin, int mode, const void* dy, int Hout, int Wout,
                   int ncol, int nout, float* dw, int* err, void* stream) {
    if (!x || !dy || !dw || !err || B < 1 || (cin != 16 && cin != 48) || nout < 1 || nout > ncol) return HYD_EINVAL;
    cudaStream_t s = (cudaStream_t)stream;
    void *tx = nullptr, *ty = nullptr;
    cudaError_t e = align16(&x, (size_t)B * Hin * Win * cin * 2, &tx, s);
    if (e == cudaSuccess) e = align16(&dy, (size_t)B * Hout * Wout * ncol * 2, &ty, s);
    const WgradArgs a{(const __nv_bfloat16*)x, (const __nv_bfloat16*)dy, B, Hin, Win, Hout, Wout, nout, dw, err};
    if (e == cudaSuccess) switch (mode) {
        case HYD_CONV_SAME: e = dispatch_wgrad<kSame>(a, cin, ncol, s); break;
        case HYD_CONV_DOWN: e = dispatch_wgrad<kDown>(a, cin, ncol, s); break;
        case HYD_CONV_UP: e = dispatch_wgrad<kUp>(a, cin, ncol, s); break;
        default: e = cudaErrorInvalidValue;
    }
    if (tx) cudaFreeAsync(tx, s);
    if (ty) cudaFreeAsync(ty, s);
    return e == cudaSuccess ? HYD_OK : (e == cudaErrorInvalidValue ? HYD_EINVAL : HYD_ECUDA);
}

int hyd_conv_pack(const float* w, int nout, int cin, long long sn, long long st, long long sc, int ncol, int cinp,
                  void* w_packed, void* stream) {
    if (!w || !w_packed || nout < 0 || cin < 0 || nout > ncol || cin > cinp || ncol < 16 || ncol % 16 || ncol > 256 ||
        cinp < 16 || cinp % 16 || cinp > 256)
        return HYD_EINVAL;
    k_pack_weights<<<(ncol * 9 * cinp + 255) / 256, 256, 0, (cudaStream_t)stream>>>(w, nout, cin, sn, st, sc, ncol, cinp,
                                                                                   (__nv_bfloat16*)w_packed);
    hyd_kernel_launches_add(1);
    return cudaGetLastError() == cudaSuccess ? HYD_OK : HYD_ECUDA;
}

int hyd_bias_grad(const void* dy, long long npix, int ncol, int nout, float* db, void* stream) {
    if (!dy || !db || npix < 1 || nout < 1 || nout > ncol || nout > 256) return HYD_EINVAL;
    if (ncol % 8 == 0 && ncol <= 256 && !(reinterpret_cast<uintptr_t>(dy) & 15)) {
        const dim3 block(ncol / 8, kBiasPix);
        const long long want = (npix + 8 * kBiasPix - 1) / (8 * kBiasPix);  // at least 8 pixels a thread
        const int per_sm = ncol <= 64 ? 8 : 2;
        k_bias_grad8<<<(int)(want < 148 * per_sm ? want : 148 * per_sm), block, sizeof(float) * kBiasPix * ncol,
                       (cudaStream_t)stream>>>((const uint4*)dy, npix, nout, db);
        hyd_kernel_launches_add(1);
        return cudaGetLastError() == cudaSuccess ? HYD_OK : HYD_ECUDA;
    }
    const dim3 block(64, 4);
    k_bias_grad<<<148, block, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)dy, npix, ncol, nout, db);
    hyd_kernel_launches_add(1);
    return cudaGetLastError() == cudaSuccess ? HYD_OK : HYD_ECUDA;
}

int hyd_mse_grad(const float* pred, const float* target, const float* weight, long long npix, int nc, int ncol,
                 float scale, void* dy, float* loss, void* stream) {
    if (!pred || !target || !dy || !loss || npix < 1 || nc < 1 || nc > ncol) return HYD_EINVAL;
    const bool wide = nc <= 4 && ncol % 8 == 0 && !(reinterpret_cast<uintptr_t>(dy) & 15);
    const auto k = wide ? k_mse_grad<true> : k_mse_grad<false>;
    k<<<8 * 148, 256, 0, (cudaStream_t)stream>>>(pred, target, weight, npix, nc, ncol, scale, (__nv_bfloat16*)dy, loss);
    hyd_kernel_launches_add(1);
    return cudaGetLastError() == cudaSuccess ? HYD_OK : HYD_ECUDA;
}

}  // extern "C"
