// 32 -> 32 3x3 convolutions of the learned smoother on the fifth-generation
// tensor cores (tcgen05.mma, accumulators in TMEM), fed by TMA: the forward
// layers and, with flipped channel-transposed weights and FP32 epilogues, the
// input gradients of the backward pass.
//
// Implicit GEMM per tile of 16 x 8 = 128 output pixels (the MMA's M):
//   D[p][co] = sum_{tap, ci} X[p + tap][ci] * W[co][tap * 32 + ci]
// with K = 9 taps x 32 channels = 288 = 18 MMAs of K = 16, N = 32.
//
// Shared-memory layout (canonical K-major, no swizzle: core matrices of 8
// rows x 16 bytes):
//  - the input halo (18 x 10 pixels) arrives by four TMA box loads of 8
//    channels each (box 8 x 10 x 18, zero fill outside the image), plane q of
//    a stage at q * 2944, pixel (hy, hx) at (hy * 10 + hx) * 16 inside it.
//    Because a tile is 8 pixels wide, the 8 rows of every core matrix of the A
//    operand of any tap are 8 consecutive halo pixels of one halo row, the
//    next core matrix (next tile row) is 160 bytes further and the next 8
//    channels one plane further: every tap's A operand is a descriptor view of
//    the halo (start, LBO = plane, SBO = halo row), nothing is copied;
//  - the weights W[co][k] at (co / 8) * 4608 + (k / 8) * 128 + (co % 8) * 16
//    + (k % 8) * 2 (LBO = 128, SBO = 4608).
// One accumulator per tap column dx, added in order in the epilogue (as
// k_conv_ws).  Two stages, software-pipelined: the TMA loads of a CTA's tiles run two
// tiles ahead and the MMAs of tile i + 1 run while tile i's epilogue reads
// its own TMEM accumulators (2 x 96 columns).  One thread issues the TMA loads
// and the 18 MMAs (committed to an mbarrier); after the bounded wait each warp reads its
// 32 TMEM lanes (one pixel per thread, 32 FP32 channels), adds the skip
// input, applies ReLU and stores BF16.  Persistent CTAs of 128 threads stride
// over the tiles (~42 KB of shared memory and 256 TMEM columns each).
#include <cudaTypedefs.h>

#include "jfg_ops.cuh"

namespace jfg {
namespace {

typedef __nv_bfloat16 bf16;

constexpr int kTH = 16, kTW = 8;                 // tile rows x columns (128 pixels)
constexpr int kHH = kTH + 2, kHW = kTW + 2;      // halo 18 x 10
constexpr int kPlaneData = kHH * kHW * 16;       // bytes one TMA box writes (2880)
constexpr int kPlane = 2944;                     // plane stride: 2880 rounded up to 128
constexpr int kHaloBytes = 4 * kPlane;           // 11,776 per stage
constexpr int kStages = 2;
constexpr int kWRowGroup = 36 * 128;             // bytes per 8 output channels (4608)
constexpr int kWBytes = 4 * kWRowGroup;          // 18,432
constexpr int kTcThreads = 128;
constexpr int kTcCtasPerSm = 2;                  // 256 TMEM columns each
// kind::f16 instruction descriptor: D FP32, A and B BF16, both K-major, N = 32, M = 128
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((32u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;      // descriptor version of sm_100; base offset 0, no swizzle
    return d;
}

// Bounded wait on an mbarrier phase (about a second at most).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity)
{
    for (int i = 0; i < (1 << 22); i++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (i > 32) __nanosleep(128);
    }
    return false;
}

__device__ __forceinline__ void tma_plane(uint32_t dst, const CUtensorMap* map, int c, int x, int y, int b,
                                          uint32_t bar)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
        "[%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c), "r"(x), "r"(y), "r"(b)
        : "memory");
}

// Epilogue modes (acc = the convolution, FP32 from TMEM; one pixel per thread):
//   kFwd:     out(bf16) = relu(acc)                          forward, no skip
//   kFwdSkip: out(bf16) = relu(acc + skip(bf16))             forward with the residual input
//   kBwdMask: out(f32) = acc * (mask(bf16) > 0), out16 = the same in BF16
//             (an input gradient through the next layer's ReLU, and its BF16
//             copy: the TMA input of the following input-gradient convolution)
//             (out may be null: only the BF16 image is wanted)
//   kBwdSkip: g = (acc + skip(f32)) * (mask(bf16) > 0): the input gradient plus
//             the skip path's through the ReLU of the layer before; out(f32) = g
//             and, where out16 is given, its BF16 copy
//   kFwdProj: the last 32 -> 32 layer (with skip) fused with the projection of
//   the 32 -> 1 output layer: h = relu(acc + skip) rounded to BF16 (the values
//   the output layer would read back), then u[t][p] = sum_c w6[c][t] h[c] for
//   the nine taps t, written as nine FP32 planes; y = sum_t u[t][p + off_t]
//   follows in a small kernel.  Warp-specialised kernel only.
constexpr int kFwd = 0, kFwdSkip = 1, kBwdMask = 2, kBwdSkip = 3, kFwdProj = 4;

// The image a mode's epilogue reads beside the accumulator, one pixel: 32
// BF16 (skip or mask) or 32 FP32 (skip; the mask beside it) channels.
template <int MODE>
struct AuxPx {
    static constexpr int kVecs = MODE == kFwd ? 0 : (MODE == kBwdSkip ? 8 : 4);
    uint4 q[kVecs ? kVecs : 1];
    uint4 m[MODE == kBwdSkip ? 4 : 1];
    __device__ __forceinline__ bool keep(int c) const     // kBwdSkip: the mask of channel c
    {
        const uint32_t u = reinterpret_cast<const uint32_t*>(m)[c >> 1];
        return __uint_as_float(c & 1 ? u & 0xFFFF0000u : u << 16) > 0.f;
    }
    __device__ __forceinline__ void load(const void* __restrict__ aux, const bf16* __restrict__ mask, size_t pix,
                                         bool inside)
    {
        if constexpr (MODE == kBwdSkip) {
#pragma unroll
            for (int i = 0; i < 4; i++)
                m[i] = inside ? __ldg(reinterpret_cast<const uint4*>(mask) + pix * 4 + i) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int i = 0; i < kVecs; i++)
            q[i] = inside ? __ldg(reinterpret_cast<const uint4*>(aux) + pix * kVecs + i) : make_uint4(0, 0, 0, 0);
    }
    __device__ __forceinline__ float at(int c) const      // channel c
    {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(q);
        if (MODE == kBwdSkip) return __uint_as_float(w[c]);
        const uint32_t u = w[c >> 1];
        return __uint_as_float(c & 1 ? u & 0xFFFF0000u : u << 16);
    }
};

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&p);
}
// 32 bytes (one sector) per thread in one store; p 32-byte aligned
__device__ __forceinline__ void st_sector(void* p, const uint32_t (&w)[8])
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                 "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}

// Channels c0 .. c0 + 15 of one output pixel: the sums v combined with the
// pixel's aux image and stored as MODE says (not kFwdProj).
template <int MODE>
__device__ __forceinline__ void conv_emit(const float (&v)[16], int c0, const AuxPx<MODE>& aux, size_t pix,
                                          void* __restrict__ out, bf16* __restrict__ out16)
{
    float f[16];
#pragma unroll
    for (int c = 0; c < 16; c++) {
        if (MODE == kFwd) f[c] = fmaxf(v[c], 0.f);
        if (MODE == kFwdSkip) f[c] = fmaxf(v[c] + aux.at(c0 + c), 0.f);
        if (MODE == kBwdMask) f[c] = aux.at(c0 + c) > 0.f ? v[c] : 0.f;
        if (MODE == kBwdSkip) f[c] = aux.keep(c0 + c) ? v[c] + aux.at(c0 + c) : 0.f;
    }
    const size_t base = pix * 32 + c0;
    constexpr bool bwd = MODE == kBwdMask || MODE == kBwdSkip;
    if (bwd && out) {
        float* of = static_cast<float*>(out) + base;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t w[8];
#pragma unroll
            for (int c = 0; c < 8; c++) w[c] = __float_as_uint(f[8 * h + c]);
            st_sector(of + 8 * h, w);
        }
    }
    if (!bwd || out16) {
        uint32_t w[8];
#pragma unroll
        for (int c = 0; c < 8; c++) w[c] = pack_bf16(f[2 * c], f[2 * c + 1]);
        st_sector((bwd ? out16 : static_cast<bf16*>(out)) + base, w);
    }
}

// 16 consecutive TMEM columns of this warp's 32 lanes
__device__ __forceinline__ void tmem_ld16(uint32_t addr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr)
        : "memory");
#pragma unroll
    for (int c = 0; c < 16; c++) v[c] = __uint_as_float(r[c]);
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

template <int MODE>
__global__ void __launch_bounds__(kTcThreads)
k_conv_mid_tc(const __grid_constant__ CUtensorMap tin, int B, int H, int W, const bf16* __restrict__ wk,
              const void* __restrict__ aux, const bf16* __restrict__ mask, void* __restrict__ out,
              bf16* __restrict__ out16, int* __restrict__ err)
{
    __shared__ __align__(128) unsigned char wsm[kWBytes];
    __shared__ __align__(128) unsigned char halo[kStages][kHaloBytes];
    __shared__ __align__(8) uint64_t full[kStages], mdone[kStages];
    __shared__ uint32_t tmem_sh;
    __shared__ int s_stop;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = tid; i < 32 * 36; i += kTcThreads) {
        const int co = i / 36, j = i % 36;
        const uint4 v = *reinterpret_cast<const uint4*>(wk + co * 288 + j * 8);
        *reinterpret_cast<uint4*>(wsm + (co >> 3) * kWRowGroup + j * 128 + (co & 7) * 16) = v;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(&tmem_sh))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        s_stop = 0;
        for (int s = 0; s < kStages; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mdone[s])) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // the weights written by threads are read by the tensor core (async proxy)
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_sh;
    const uint32_t wbase = smem_u32(wsm);
    const int tilesx = (W + kTW - 1) / kTW, tilesy = (H + kTH - 1) / kTH;
    const int per_img = tilesx * tilesy;
    const int ntiles = per_img * B;

    auto issue_load = [&](int t, int s) {       // thread 0 only
        const int b = t / per_img, rem = t - b * per_img;
        const int y0 = (rem / tilesx) * kTH, x0 = (rem % tilesx) * kTW;
        const uint32_t bar = smem_u32(&full[s]);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(4 * kPlaneData)
                     : "memory");
        const uint32_t dst = smem_u32(halo[s]);
#pragma unroll
        for (int q = 0; q < 4; q++) tma_plane(dst + q * kPlane, &tin, 8 * q, x0 - 1, y0 - 1, b, bar);
    };

    // tiles of this CTA: t_i = blockIdx.x + i * gridDim.x, i < cnt
    const int cnt = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    auto tile_of = [&](int i) { return (int)blockIdx.x + i * (int)gridDim.x; };
    auto issue_mma = [&](int i) -> bool {     // thread 0: wait for tile i's halo, MMAs into TMEM stage i & 1
        const int s = i & 1;
        if (!mbar_wait(smem_u32(&full[s]), (uint32_t)((i >> 1) & 1))) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t hb = smem_u32(halo[s]);
#pragma unroll
        for (int tap = 0; tap < 9; tap++) {
            const int dy = tap / 3, dx = tap % 3;
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const uint64_t da = umma_desc(hb + 2 * k * kPlane + (dy * kHW + dx) * 16, kPlane, kHW * 16);
                const uint64_t db = umma_desc(wbase + (4 * tap + 2 * k) * 128, 128, kWRowGroup);
                const uint32_t accum = (dy | k) ? 1u : 0u;     // one accumulator per tap column dx
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                    ::"r"(tmem + (uint32_t)(s * 128 + dx * 32)), "l"(da), "l"(db), "r"(kIdesc), "r"(accum)
                    : "memory");
            }
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(&mdone[s]))
                     : "memory");
        return true;
    };

    // Pipeline: loads run two tiles ahead, the MMAs of tile i + 1 run during
    // the epilogue of tile i.  Outstanding async work is tracked by thread 0
    // for the error path.
    int loads_issued = 0, loads_done = 0, mmas_issued = 0;
    if (tid == 0) {
        for (int i = 0; i < 2 && i < cnt; i++) {
            issue_load(tile_of(i), i);
            loads_issued++;
        }
        if (cnt > 0) {
            if (issue_mma(0)) {
                loads_done = 1;
                mmas_issued = 1;
            } else {
                s_stop = 1;
            }
        }
    }
    __syncthreads();
    int i = 0;
    for (; i < cnt && !s_stop; i++) {
        const int s = i & 1;
        const bool ok = mbar_wait(smem_u32(&mdone[s]), (uint32_t)((i >> 1) & 1));
        if (__syncthreads_or(!ok)) {
            if (tid == 0) s_stop = 1;
            break;
        }
        if (tid == 0) {
            if (i + 2 < cnt) {                   // its buffer held tile i, whose MMAs are complete
                issue_load(tile_of(i + 2), s);
                loads_issued++;
            }
            if (i + 1 < cnt) {
                if (issue_mma(i + 1)) {
                    loads_done++;
                    mmas_issued++;
                } else {
                    s_stop = 1;
                }
            }
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int t = tile_of(i);
        const int b = t / per_img, rem = t - b * per_img;
        const int y0 = (rem / tilesx) * kTH, x0 = (rem % tilesx) * kTW;
        const int m = warp * 32 + lane;
        const int gy = y0 + (m >> 3), gx = x0 + (m & 7);
        const bool inside = gy < H && gx < W;
        const size_t pix = inside ? ((size_t)b * H + gy) * W + gx : 0;
        AuxPx<MODE> ax;
        ax.load(aux, mask, pix, inside);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t col = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(s * 128 + 16 * h);
            float d0[16], d1[16], d2[16];
            tmem_ld16(col, d0);
            tmem_ld16(col + 32, d1);
            tmem_ld16(col + 64, d2);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 16; c++) d0[c] = (d0[c] + d1[c]) + d2[c];
            if (inside) conv_emit<MODE>(d0, 16 * h, ax, pix, out, out16);
        }
        // every thread's TMEM reads are done before the MMAs two tiles on overwrite this stage
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
    }
    if (s_stop && tid == 0) {
        // error path: report, then let the copies and MMAs still in flight finish (bounded) before TMEM is freed
        atomicOr(err, 1);
        for (int k = loads_done; k < loads_issued; k++) mbar_wait(smem_u32(&full[k & 1]), (uint32_t)((k >> 1) & 1));
        for (int k = i; k < mmas_issued; k++) mbar_wait(smem_u32(&mdone[k & 1]), (uint32_t)((k >> 1) & 1));
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem) : "memory");
    }
}

// ---------------------------------------------------------------------------
// Warp-specialised pipeline (the default).
//
// The three taps of a row are one MMA: for an input pixel q the products with
// the weights of dx = 0, 1, 2 (N = 3 x 32 outputs) go to three accumulators
// D_dx[q], summed over dy and the channels, and the output is
//   out[p] = (D_0[p - 1] + D_1[p]) + D_2[p + 1].
// A tile is kRY rows of kRX = 32 input pixels (M = 128, TMEM lane = row, x), so
// the lanes of an epilogue warp are one row's consecutive pixels, the shifts
// are two shuffles inside the warp and 30 of its 32 pixels are outputs.  The
// input arrives as ONE TMA box (32 channels x 32 pixels x kRY + 2 rows,
// 64-byte swizzle) which is the K-major A operand as it lies: tap row dy is
// dy * 2,048 bytes further.  6 MMAs of N = 96 per tile of 120 outputs instead
// of 18 of N = 32 per 128: each MMA of N = 32 held the tensor pipe ~40 cycles
// for 16 cycles of math, and the kernel that fed them from transposed 8-channel
// planes (shared memory read and written once more per tile) ran 55 us per
// layer at 1025 x 1025 pixels against 32.5 us here (63 -> 41.5 us with a skip
// input, 86 -> 65 us with the output projection); the image bytes (134 MB) take
// 20 us.
//
// Roles (320 threads, two CTAs per SM, 256 TMEM columns each):
//   warp 0 (one lane): TMA producer, kDxStages boxes ahead (`full` / `empty`);
//   warp 1 (one lane): MMA issuer -- waits for a box and a free accumulator
//     set (`tempty`), issues the 6 MMAs and commits them to `empty` and `tfull`;
//   warps 2-9: epilogue, two groups of four taking the tiles in turn (group =
//     accumulator set); a warp loads its pixels' aux channels before it waits.
// No CTA-wide barrier inside the tile loop.  Every wait is bounded
// (mbar_wait); a timeout sets *err, every role stops, and the copies and MMAs
// still in flight are waited for (bounded) before TMEM is released.
// ---------------------------------------------------------------------------
constexpr int kRX = 32, kRY = 4;                 // input pixels of a tile: 4 rows of 32
constexpr int kOutX = kRX - 2;                   // output pixels of a tile row
constexpr int kBoxRows = kRY + 2;
constexpr int kRowBytes = kRX * 64;              // one input row of the box
constexpr int kBoxBytes = kBoxRows * kRowBytes;  // 12,288
constexpr int kDxStages = 4;
constexpr int kDxAcc = 2;                        // accumulator sets of 96 columns, 128 apart
constexpr int kDxThreads = 320;
constexpr int kDxCtasPerSm = 2;
constexpr int kDxWGroup = 12 * 128;              // weights: bytes per 8 rows n = dx * 32 + co (k = dy * 32 + ci)
constexpr int kDxSmem = kDxStages * kBoxBytes + 12 * kDxWGroup + 1024;
constexpr uint32_t kIdesc96 = (1u << 4) | (1u << 7) | (1u << 10) | ((96u >> 3) << 17) | ((128u >> 4) << 24);

// K-major operand rows of 64 bytes, 64-byte swizzle (8-row groups 512 bytes apart)
__device__ __forceinline__ uint64_t umma_desc_sw64(uint32_t saddr)
{
    return umma_desc(saddr, 16, 512) | ((uint64_t)4 << 61);
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

template <int MODE>
__global__ void __launch_bounds__(kDxThreads, kDxCtasPerSm)
k_conv_ws(const __grid_constant__ CUtensorMap tin, int B, int H, int W, const bf16* __restrict__ wk,
          const void* __restrict__ aux, const bf16* __restrict__ mask, void* __restrict__ out,
          bf16* __restrict__ out16, int* __restrict__ err, const float* __restrict__ proj)
{
    extern __shared__ unsigned char dsm_raw[];
    unsigned char* boxes = reinterpret_cast<unsigned char*>(((uintptr_t)dsm_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* wsm = boxes + kDxStages * kBoxBytes;
    __shared__ __align__(8) uint64_t full[kDxStages], empty[kDxStages], tfull[kDxAcc], tempty[kDxAcc];
    __shared__ uint32_t tmem_sh;
    __shared__ volatile int s_stop;
    __shared__ int s_loads, s_mmas;                           // progress counts, for the error path
    __shared__ __align__(16) float w6s[MODE == kFwdProj ? 9 * 32 : 4];    // output-layer weights [tap][channel]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = tid; i < 32 * 36; i += kDxThreads) {
        const int co = i / 36, j = i % 36, tap = j >> 2, part = j & 3;
        const int n = (tap % 3) * 32 + co, kg = (tap / 3) * 4 + part;
        *reinterpret_cast<uint4*>(wsm + (n >> 3) * kDxWGroup + kg * 128 + (n & 7) * 16) =
            *reinterpret_cast<const uint4*>(wk + co * 288 + j * 8);
    }
    if constexpr (MODE == kFwdProj)
        for (int i = tid; i < 9 * 32; i += kDxThreads) w6s[(i % 9) * 32 + i / 9] = proj[i];
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(&tmem_sh))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 32) {
        s_stop = 0;
        s_loads = 0;
        s_mmas = 0;
        for (int q = 0; q < kDxStages; q++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[q])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[q])) : "memory");
        }
        for (int q = 0; q < kDxAcc; q++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&tfull[q])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(smem_u32(&tempty[q])) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // weights: generic writes, async-proxy reads
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_sh;
    const uint32_t wbase = smem_u32(wsm), bbase = smem_u32(boxes);
    const int tilesx = (W + kOutX - 1) / kOutX, tilesy = (H + kRY - 1) / kRY;
    const int per_img = tilesx * tilesy;
    const int ntiles = per_img * B;
    const int cnt = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    auto tile_of = [&](int i) { return (int)blockIdx.x + i * (int)gridDim.x; };

    if (warp == 0) {
        if (lane == 0) {                               // TMA producer
            for (int i = 0; i < cnt && !s_stop; i++) {
                const int q = i % kDxStages;
                if (i >= kDxStages && !mbar_wait(smem_u32(&empty[q]), (uint32_t)((i / kDxStages - 1) & 1))) {
                    s_stop = 1;
                    break;
                }
                const int t = tile_of(i);
                const int b = t / per_img, rem = t - b * per_img;
                const int y0 = (rem / tilesx) * kRY, x0 = (rem % tilesx) * kOutX;
                const uint32_t bar = smem_u32(&full[q]);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kBoxBytes)
                             : "memory");
                tma_plane(bbase + q * kBoxBytes, &tin, 0, x0 - 1, y0 - 1, b, bar);
                s_loads = i + 1;
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {                               // MMA issuer
            for (int i = 0; i < cnt && !s_stop; i++) {
                const int q = i % kDxStages, a = i % kDxAcc;
                if (!mbar_wait(smem_u32(&full[q]), (uint32_t)((i / kDxStages) & 1)) ||
                    (i >= kDxAcc && !mbar_wait(smem_u32(&tempty[a]), (uint32_t)((i / kDxAcc - 1) & 1)))) {
                    s_stop = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int dy = 0; dy < 3; dy++) {
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        const uint64_t da = umma_desc_sw64(bbase + q * kBoxBytes + dy * kRowBytes + k * 32);
                        const uint64_t db = umma_desc(wbase + (4 * dy + 2 * k) * 128, 128, kDxWGroup);
                        const uint32_t accum = (dy | k) ? 1u : 0u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                            ::"r"(tmem + (uint32_t)(a * 128)), "l"(da), "l"(db), "r"(kIdesc96), "r"(accum)
                            : "memory");
                    }
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_u32(&empty[q]))
                             : "memory");
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_u32(&tfull[a]))
                             : "memory");
                s_mmas = i + 1;
            }
        }
    } else {                                           // epilogue warps 2..9
        const int lg = warp & 3;                       // TMEM lane group this warp may access = tile row
        for (int i = (warp - 2) >> 2; i < cnt; i += kDxAcc) {
            const int a = i % kDxAcc;
            const int t = tile_of(i);
            const int b = t / per_img, rem = t - b * per_img;
            const int gy = (rem / tilesx) * kRY + lg, gx = (rem % tilesx) * kOutX + lane - 1;
            const bool inside = gy < H && gx < W && lane >= 1 && lane <= kOutX;
            const size_t pix = inside ? ((size_t)b * H + gy) * W + gx : 0;
            AuxPx<MODE> ax;
            ax.load(aux, mask, pix, inside);
            const bool ok = !s_stop && mbar_wait(smem_u32(&tfull[a]), (uint32_t)((i / kDxAcc) & 1));
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) s_stop = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float u9[9];
            if constexpr (MODE == kFwdProj) {
#pragma unroll
                for (int tp = 0; tp < 9; tp++) u9[tp] = 0.f;
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t col = tmem + ((uint32_t)(lg * 32) << 16) + (uint32_t)(a * 128 + 16 * h);
                float d0[16], d1[16], d2[16];
                tmem_ld16(col, d0);
                tmem_ld16(col + 32, d1);
                tmem_ld16(col + 64, d2);
                tmem_ld_wait();
                if (h == 1) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&tempty[a]));
                }
#pragma unroll
                for (int c = 0; c < 16; c++)
                    d0[c] = (__shfl_up_sync(0xffffffffu, d0[c], 1) + d1[c]) + __shfl_down_sync(0xffffffffu, d2[c], 1);
                if constexpr (MODE == kFwdProj) {
#pragma unroll
                    for (int c = 0; c < 16; c++)
                        d0[c] = __bfloat162float(__float2bfloat16_rn(fmaxf(d0[c] + ax.at(16 * h + c), 0.f)));
#pragma unroll
                    for (int tp = 0; tp < 9; tp++) {
                        const float4* w4 = reinterpret_cast<const float4*>(w6s + tp * 32 + 16 * h);
#pragma unroll
                        for (int c4 = 0; c4 < 4; c4++) {
                            const float4 w = w4[c4];
                            u9[tp] += w.x * d0[4 * c4];
                            u9[tp] += w.y * d0[4 * c4 + 1];
                            u9[tp] += w.z * d0[4 * c4 + 2];
                            u9[tp] += w.w * d0[4 * c4 + 3];
                        }
                    }
                } else {
                    if (inside) conv_emit<MODE>(d0, 16 * h, ax, pix, out, out16);
                }
            }
            if constexpr (MODE == kFwdProj) {
                float* u = static_cast<float*>(out);
                const size_t npx = (size_t)B * H * W;
                if (inside)
#pragma unroll
                    for (int tp = 0; tp < 9; tp++) u[(size_t)tp * npx + pix] = u9[tp];
            }
        }
    }
    __syncthreads();
    if (s_stop && tid == 32) {
        // report, then let the copies and MMAs still in flight finish (bounded) before TMEM is freed
        atomicOr(err, 1);
        const int nl = s_loads, nm = s_mmas;
        for (int k = nm; k < nl; k++) mbar_wait(smem_u32(&full[k % kDxStages]), (uint32_t)((k / kDxStages) & 1));
        if (nm > 0) mbar_wait(smem_u32(&tfull[(nm - 1) % kDxAcc]), (uint32_t)(((nm - 1) / kDxAcc) & 1));
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem) : "memory");
    }
}

// ---------------------------------------------------------------------------
// Weight gradient of a 32 -> 32 layer on the tensor cores:
//   dW[co][tap][ci] = sum_p G[p][co] X[p + tap][ci]
// The pixels are the contraction and both images hold a pixel's 32 channels
// contiguously, so both operands are MN-major as TMA writes them (64-byte
// swizzle, one pixel per 64-byte row): nothing is transposed or staged by
// threads.  For one row q of 16 pixels of X a single MMA (K = 16) covers all
// nine taps:
//   A = three copies of the row shifted by dx - 1 pixels (three TMA boxes;
//       M = dx * 32 + ci, the fourth block of M reads the G tile and its rows
//       of D are not used),
//   B = the rows q - 1, q, q + 1 of G (N = j * 32 + co, dy = 2 - j),
//   D[dx, ci][j, co] += A B, 96 FP32 columns of TMEM kept over all tiles of
//       the CTA.
// A tile is 8 rows x 16 pixels of X with 10 rows of G; the epilogue writes the
// CTA's partial dW (FP32, [co][tap * 32 + ci]) for the ordered reduction of
// k_wgrad_mid_reduce.  Bound by the boxes' bytes (34 KB per tile from L2);
// transposing both images into K-major planes with all threads and one MMA per
// tap took 85 us per layer at 16 x 128 x 128 pixels, against 13.4 us.
// Roles: warp 0 TMA producer, warp 1 MMA issuer, then warps 0-2 the epilogue.
// ---------------------------------------------------------------------------
constexpr int kGTH = 8, kGTW = 16;               // X rows x pixels of a tile
constexpr int kGRow = kGTW * 64;                 // bytes of one row of pixels
constexpr int kGXBytes = kGTH * kGRow;           // one shifted copy of X: 8,192
constexpr int kGGBytes = (kGTH + 2) * kGRow;     // the G rows: 10,240
constexpr int kGStage = 3 * kGXBytes + kGGBytes; // 34,816
constexpr int kGStages = 5;
constexpr int kWgSmem = kGStages * kGStage + 1024;
constexpr int kWgThreads = 128;
// M = 128, N = 96, both operands MN-major
constexpr uint32_t kIdescWg = kIdesc96 | (1u << 15) | (1u << 16);

// MN-major operand, 64-byte swizzle: 32-element blocks `blk` bytes apart, 8-row
// groups along K 512 bytes apart
__device__ __forceinline__ uint64_t umma_desc_mn64(uint32_t saddr, uint32_t blk)
{
    return umma_desc(saddr, blk, 512) | ((uint64_t)4 << 61);
}

__global__ void __launch_bounds__(kWgThreads, 1)
k_wgrad_tc(const __grid_constant__ CUtensorMap tg, const __grid_constant__ CUtensorMap txm, int B, int H, int W,
           float* __restrict__ part, int* __restrict__ err)
{
    extern __shared__ unsigned char dsm_raw[];
    const uint32_t sbase = (smem_u32(dsm_raw) + 1023u) & ~1023u;
    __shared__ __align__(8) uint64_t full[kGStages], empty[kGStages], mdone;
    __shared__ uint32_t tmem_sh;
    __shared__ volatile int s_stop;
    __shared__ int s_loads, s_mmas;                  // progress counts, for the error path
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 128;" ::"r"(smem_u32(&tmem_sh))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 32) {
        s_stop = 0;
        s_loads = 0;
        s_mmas = 0;
        for (int q = 0; q < kGStages; q++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[q])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[q])) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mdone)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_sh;
    const int tx = (W + kGTW - 1) / kGTW, ty = (H + kGTH - 1) / kGTH;
    const int ntiles = tx * ty * B;
    const int cnt = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

    if (warp == 0) {
        if (lane == 0) {                             // TMA producer
            for (int i = 0; i < cnt && !s_stop; i++) {
                const int q = i % kGStages;
                if (i >= kGStages && !mbar_wait(smem_u32(&empty[q]), (uint32_t)((i / kGStages - 1) & 1))) {
                    s_stop = 1;
                    break;
                }
                const int t = (int)blockIdx.x + i * (int)gridDim.x;
                const int b = t / (tx * ty), rem = t - b * (tx * ty);
                const int y0 = (rem / tx) * kGTH, x0 = (rem % tx) * kGTW;
                const uint32_t bar = smem_u32(&full[q]), dst = sbase + q * kGStage;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kGStage)
                             : "memory");
#pragma unroll
                for (int dx = 0; dx < 3; dx++) tma_plane(dst + dx * kGXBytes, &txm, 0, x0 - 1 + dx, y0, b, bar);
                tma_plane(dst + 3 * kGXBytes, &tg, 0, x0, y0 - 1, b, bar);
                s_loads = i + 1;
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {                             // MMA issuer
            for (int i = 0; i < cnt && !s_stop; i++) {
                const int q = i % kGStages;
                if (!mbar_wait(smem_u32(&full[q]), (uint32_t)((i / kGStages) & 1))) {
                    s_stop = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t xb = sbase + q * kGStage, gb = xb + 3 * kGXBytes;
#pragma unroll
                for (int r = 0; r < kGTH; r++) {
                    const uint64_t da = umma_desc_mn64(xb + r * kGRow, kGXBytes);
                    const uint64_t db = umma_desc_mn64(gb + r * kGRow, kGRow);
                    const uint32_t accum = (i | r) ? 1u : 0u;
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "setp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                        ::"r"(tmem), "l"(da), "l"(db), "r"(kIdescWg), "r"(accum)
                        : "memory");
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_u32(&empty[q]))
                             : "memory");
                s_mmas = i + 1;
            }
            // every MMA issued so far is complete when this arrives
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&mdone))
                         : "memory");
        }
    }
    __syncwarp();
    __syncthreads();
    const bool done = mbar_wait(smem_u32(&mdone), 0);
    const bool ok = __syncthreads_and(done && !s_stop);
    if (!ok && tid == 32) {
        // report, then let the copies still in flight finish (bounded)
        atomicOr(err, 1);
        for (int k = s_mmas; k < s_loads; k++) mbar_wait(smem_u32(&full[k % kGStages]), (uint32_t)((k / kGStages) & 1));
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp < 3) {                                  // warp = dx, lane = ci
        float* dst = part + (size_t)blockIdx.x * (32 * 288) + warp * 32 + lane;
#pragma unroll 1
        for (int h = 0; h < 6; h++) {                // columns 16 h ..: j = h / 2, co = 16 (h % 2) ..
            float v[16];
            tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(16 * h), v);
            tmem_ld_wait();
            const int dy = 2 - (h >> 1);
#pragma unroll
            for (int c = 0; c < 16; c++)
                dst[(size_t)(16 * (h & 1) + c) * 288 + dy * 96] = (cnt > 0 && ok) ? v[c] : 0.f;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 128;" ::"r"(tmem) : "memory");
    }
}

}  // namespace

// The driver's tensor-map encoder, fetched once through the runtime (no link
// against libcuda).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        JFG_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
        JFG_CHECK(q == cudaDriverEntryPointSuccess && p, JFG_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
        fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

// JFEM_CNN_WS=0 selects the single-role kernel (k_conv_mid_tc) instead of the
// warp-specialised pipeline (k_conv_ws)
static bool use_ws()
{
    const char* e = getenv("JFEM_CNN_WS");
    return !(e && e[0] == '0');
}

// A (B, H, W, 32) BF16 image as TMA boxes of box_c channels x box_x x box_y
// pixels; whole pixels (32 channels) with the 64-byte swizzle of the MMA
// operands, planes of 8 channels without; zero fill outside the image.
static CUtensorMap conv_input_map(int B, int H, int W, const __nv_bfloat16* in, int box_c, int box_x, int box_y)
{
    CUtensorMap map;
    const cuuint64_t dims[4] = {32, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)B};
    const cuuint64_t strides[3] = {64, (cuuint64_t)W * 64, (cuuint64_t)W * H * 64};
    const cuuint32_t box[4] = {(cuuint32_t)box_c, (cuuint32_t)box_x, (cuuint32_t)box_y, 1};
    const cuuint32_t estride[4] = {1, 1, 1, 1};
    CUresult r = tensor_map_encoder()(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<__nv_bfloat16*>(in), dims,
                                      strides, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                      box_c == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE,
                                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    JFG_CHECK(r == CUDA_SUCCESS, JFG_ERR_CUDA, "cuTensorMapEncodeTiled failed");
    return map;
}

template <int MODE>
static void launch_conv(cudaStream_t st, int B, int H, int W, const bf16* in, const bf16* w, const void* aux, void* out,
                        bf16* out16, int* err, const float* proj = nullptr, const bf16* mask = nullptr)
{
    const bool ws = use_ws();
    const long long ntiles = ws ? (long long)((W + kOutX - 1) / kOutX) * ((H + kRY - 1) / kRY) * B
                                : (long long)((W + kTW - 1) / kTW) * ((H + kTH - 1) / kTH) * B;
    JFG_CHECK(ntiles < (1LL << 30), JFG_ERR_UNSUPPORTED, "image too large for the tensor-core convolution");
    JFG_CHECK(((uintptr_t)in & 15) == 0, JFG_ERR_BAD_ARG, "convolution input not 16-byte aligned");
    const int grid = (int)std::min<long long>(ntiles, (long long)sm_count() * (ws ? kDxCtasPerSm : kTcCtasPerSm));
    if (grid <= 0) return;
    const CUtensorMap map = ws ? conv_input_map(B, H, W, in, 32, kRX, kBoxRows) : conv_input_map(B, H, W, in, 8, kHW, kHH);
    if (ws) {
        static PerDevice once;
        allow_smem(once, k_conv_ws<MODE>, kDxSmem);
        k_conv_ws<MODE><<<grid, kDxThreads, kDxSmem, st>>>(map, B, H, W, w, aux, mask, out, out16, err, proj);
    } else if constexpr (MODE != kFwdProj) {
        k_conv_mid_tc<MODE><<<grid, kTcThreads, 0, st>>>(map, B, H, W, w, aux, mask, out, out16, err);
    } else {
        JFG_CHECK(false, JFG_ERR_UNSUPPORTED, "the fused output projection needs the warp-specialised convolution");
    }
    JFG_CUDA(cudaGetLastError());
    note_launch();
}

// out = relu(conv3x3(in, wk) [+ skip]) for BF16 (B, H, W, 32) images; wk is
// BF16 [32 outputs][9 taps x 32 inputs].  err is set to 1 if a TMA or MMA
// wait timed out (the output is then incomplete).
void conv_mid_tc(cudaStream_t st, int B, int H, int W, const __nv_bfloat16* in, const __nv_bfloat16* wk,
                 const __nv_bfloat16* skip, __nv_bfloat16* out, int* err)
{
    if (skip)
        launch_conv<kFwdSkip>(st, B, H, W, in, wk, skip, out, nullptr, err);
    else
        launch_conv<kFwd>(st, B, H, W, in, wk, nullptr, out, nullptr, err);
}

// The last 32 -> 32 layer with its skip input fused with the projection of
// the 32 -> 1 output layer (kFwdProj): u receives nine FP32 planes of B*H*W
// entries, u[t][p] = sum_c w6[c][t] relu(conv + skip)[p][c] (BF16-rounded
// activations); w6 is FP32 [32 channels][9 taps].  Warp-specialised kernel
// only (the caller checks conv_proj_available()).
bool conv_proj_available() { return use_ws(); }

void conv_mid_tc_proj(cudaStream_t st, int B, int H, int W, const __nv_bfloat16* in, const __nv_bfloat16* wk,
                      const __nv_bfloat16* skip, const float* w6, float* u, int* err)
{
    launch_conv<kFwdProj>(st, B, H, W, in, wk, skip, u, nullptr, err, w6);
}

// Input gradient of a 32 -> 32 layer on the tensor cores: conv3x3 of the
// BF16 gradient image gin with the flipped, channel-transposed weights wt
// (the layout of wk), FP32 accumulation.  g = (acc [+ skip]) * (mask > 0): out
// = g in FP32 (null: not wanted), out16 = its BF16 copy (null: not wanted).
void conv_mid_tc_bwd(cudaStream_t st, int B, int H, int W, const __nv_bfloat16* gin, const __nv_bfloat16* wt,
                     const __nv_bfloat16* mask, const float* skip, float* out, __nv_bfloat16* out16, int* err)
{
    if (skip)
        launch_conv<kBwdSkip>(st, B, H, W, gin, wt, skip, out, out16, err, nullptr, mask);
    else
        launch_conv<kBwdMask>(st, B, H, W, gin, wt, mask, out, out16, err);
}

// Per-CTA partial weight gradients of a 32 -> 32 layer on the tensor cores
// (k_wgrad_tc) from the BF16 gradient image G16 and the BF16 layer input X:
// part[cta][co * 288 + tap * 32 + ci]; returns the number of CTAs (at most
// max_parts).  err is set to 1 if the MMA wait timed out.
int wgrad_mid_tc(cudaStream_t st, int B, int H, int W, const __nv_bfloat16* G16, const __nv_bfloat16* X,
                 float* part, int max_parts, int* err)
{
    const long long ntiles = (long long)((W + kGTW - 1) / kGTW) * ((H + kGTH - 1) / kGTH) * B;
    JFG_CHECK(ntiles < (1LL << 31), JFG_ERR_UNSUPPORTED, "image too large for the tensor-core weight gradient");
    const int ctas = (int)std::min<long long>(std::min<long long>(ntiles, sm_count()), max_parts);
    if (ctas <= 0) return 0;
    static PerDevice once;
    allow_smem(once, k_wgrad_tc, kWgSmem);
    const CUtensorMap tg = conv_input_map(B, H, W, G16, 32, kGTW, kGTH + 2);
    const CUtensorMap tx = conv_input_map(B, H, W, X, 32, kGTW, kGTH);
    k_wgrad_tc<<<ctas, kWgThreads, kWgSmem, st>>>(tg, tx, B, H, W, part, err);
    JFG_CUDA(cudaGetLastError());
    note_launch();
    return ctas;
}

}  // namespace jfg
