// Surrogate-denoiser inference on the 5th-generation tensor cores (tcgen05,
// sm_100a): the eight 3x3 convolutions of cpipe_b200/csrc/surrogate.cu in two
// kernels of four layers each, with no activation but the fourth layer's in
// device memory.
//
// A CTA owns a strip of up to 122 columns and walks down its rows.  The M = 128
// rows of every product are 128 neighbouring pixels of one image row, the strip
// and three halo pixels each side, so the valid pixels shrink by one a side and
// layer from 128 to 122.  Each of the four layers works on its own row, two
// rows behind the layer before it: a warp per layer issues the products of a
// row as it comes, and a warpgroup per layer turns finished rows into the next
// layer's input rows in shared memory (two-row rings).
//
//  * An input row [4 planes of 8 channels][pixel][8 ch] is a K-major, unswizzled
//    operand read in place: tap kx starts kx pixels (16 B each) further on, 8
//    pixels are one core matrix (SBO 128 B), the next 8 channels the next plane
//    (LBO).
//  * A row takes part in three output rows.  Their accumulators lie side by
//    side in TMEM (32 columns each, rows modulo 3), so one product with N = 96
//    serves all three: six MMAs a row (3 kx x 2 K slices) instead of the 18 of
//    N = 32 products per output row, which had bound the layers by the tensor
//    core's reads of A (4 KB per MMA).  Which 32 columns are the row above, at
//    and below the input row rotates with the row; the weights lie in shared
//    memory as the block sequence ky = 2 1 0 2 1, whose windows of three are the
//    three rotations.  Finished accumulators are cleared by the epilogue that
//    reads them.  An output pixel's sum runs over ky, kx and the two K slices in
//    that order, as in the mma.sync kernels.
//  * The first layer (8 input channels, two taps to a K slice, some pairs across
//    rows) keeps N = 32 products per output row over a ring of input rows whose
//    first row is stored again after the last, so that a row and the next are
//    always a constant distance apart.
//  * Rows outside the image take no products, pixels outside it are stored as
//    zeros: the convolutions' zero padding.
//
// Frames of at most 63 columns would leave most of the lanes to nothing.  Their
// kernels (PACK) lay the frames on top of one another, a row of zeros after each,
// cut that stack into bands of rows, as many as fit side by side with a column of
// zeros between them, and walk all bands at once; rows and pixels outside a frame
// are zeros everywhere.  16 x 187500 pixels: 2280 us a strip at a time, 752 with a
// kernel per layer, 520 so; 1000 frames of 16 x 16: 220, 115 and 84 us.
//
// Front kernel: RGBA -> the network's input (the mapping of sg_prep_kernel) by
// four warps -> layers 0-3 -> bf16 planes.  Back kernel: those planes by bulk
// copies -> layers 4-7 -> residual onto the RGBA frame.
//
// Bound by the tensor core's shared-memory reads, (4 + 3) KB per hidden MMA (42
// KB, 330 clocks, a row of 128 pixels and layer: 75 % of that path's rate in the
// back kernel, 58 % in the front one, 2048 x 2048), and by the epilogues' latency for the
// rest.  Measured, three frames of 1201 x 801: 778 -> 392 us against one kernel
// per layer with N = 32 (102 us a hidden layer); DRAM traffic 950 -> 152 B/px.
//
// Every mbarrier wait is bounded: a wait that runs out records an error code in
// *err, ends the CTA's roles, and the CTA still waits for its copies in flight
// and releases its TMEM, so the context stays usable.
#include <cuda_bf16.h>

#include "../../include/cpipe_node_abi.h"
#include "common.cuh"
#include "surrogate_tc.h"

namespace cpb {
namespace sgtc {

using bf16 = __nv_bfloat16;

constexpr int kLanes = 128;                   // pixels per product: the M of an MMA
constexpr int kStripMax = kLanes - 6;         // columns a strip of four layers keeps
constexpr int kRowPix = kLanes + 2;           // pixels of a stored row
constexpr int kPlane = 2176;                  // bytes per 8-channel plane of a row (130 x 16 B, 128-byte aligned)
constexpr int kRow = 4 * kPlane;              // bytes per 32-channel row
constexpr int kRing = 2;                      // rows between two layers (stepped as one bit)
constexpr int kEpiWarps = 16;                 // a warpgroup per layer
constexpr int kMmaWarps = 4;                  // one per layer
constexpr int kPrepWarps = 4;                 // front kernel: a thread per pixel of a row (two threads: two)
constexpr int kTmemCols = 512;
// A poll suspends its warp for up to this long: polls without the hint came back
// so often that they took a third of the shared-memory reads.
constexpr uint32_t kSuspendNs = 2000;
constexpr uint32_t kSpinLimit = 1U << 19;  // about a second in all

// ----------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(saddr(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(saddr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(saddr(bar)), "r"(bytes) : "memory");
}
// Bounded wait for the completion of phase `parity`.  A wait that runs out
// raises *stop and records `code` in *err; from then on the CTA's waits return
// at once and its roles run to their ends on whatever the buffers hold (every
// address stays within them).
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, volatile int* stop, int* err, int code) {
    const uint32_t a = saddr(bar);
    for (uint32_t i = 0;; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(a), "r"(parity), "r"(kSuspendNs)
            : "memory");
        if (ok || ((i & 7U) == 7U && *stop)) return;
        if (i == kSpinLimit) {
            *stop = 1;
            atomicCAS(err, 0, code);
            return;
        }
    }
}
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xFFFFFFFF;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// Shared-memory matrix descriptor: K-major, no swizzle (SM100 version field 1).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFU) | ((uint64_t)((lbo >> 4) & 0x3FFFU) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFU) << 32) | (1ULL << 46);
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     saddr(dst)),
                 "l"(src), "r"(bytes), "r"(saddr(bar))
                 : "memory");
}
// Instruction descriptor: D = F32, A = B = BF16, both K-major, M = 128, N.
template <int N>
__host__ __device__ constexpr uint32_t instr_desc() {
    return (1U << 4) | (1U << 7) | (1U << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
            d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(saddr(bar))
                 : "memory");
}


// A warp's 32 lanes x 16 columns.
__device__ __forceinline__ void tmem_load16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// 32 columns set to zero, for the next rows' sums.
__device__ __forceinline__ void tmem_clear32(uint32_t taddr) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,"
        "%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};\n" ::"r"(taddr),
        "r"(0)
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
}
// The last layer's columns, read and cleared.
__device__ __forceinline__ void tmem_take(uint32_t taddr, float (&v)[4]) {
    uint32_t r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%1,%1,%1};\n" ::"r"(taddr), "r"(0) : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
}

// Bias, rounding to bfloat16, ReLU (a NaN becomes 0, as with fmaxf).
__device__ __forceinline__ uint32_t bias_relu(float c0, float c1, float b0, float b1) {
    const float2 v = __fadd2_rn(make_float2(c0, c1), make_float2(b0, b1));
    uint32_t r;
    asm("{\n .reg .b32 t;\n cvt.rn.bf16x2.f32 t, %2, %1;\n max.bf16x2 %0, t, %3;\n}\n" : "=r"(r) : "f"(v.x), "f"(v.y), "r"(0));
    return r;
}

__device__ __forceinline__ uint4 bias_relu8(const float* c, const float* b) {
    return make_uint4(bias_relu(c[0], c[1], b[0], b[1]), bias_relu(c[2], c[3], b[2], b[3]),
                      bias_relu(c[4], c[5], b[4], b[5]), bias_relu(c[6], c[7], b[6], b[7]));
}

// Shared memory of a kernel: the layers' weights, the ring of rows that the
// first layer reads, the rings between the layers, barriers.
template <bool FRONT>
struct Smem {
    static constexpr int IN_RING = FRONT ? 6 : 4;                      // rows the first layer may have ahead
    static constexpr int IN_ROW = FRONT ? kPlane : kRow;
    static constexpr int W_HIDDEN = 12 * 20 * 128;                     // 12 K groups x (5 blocks x 4 N groups)
    static constexpr int W_FIRST = 10 * 4 * 128;                       // front, layer 0: 10 K groups x 4 N groups
    static constexpr int W_LAST = 12 * 10 * 128;                       // back, last layer: blocks of 16 channels
    __host__ __device__ static constexpr int w_off(int p) {
        return FRONT ? (p == 0 ? 0 : W_FIRST + (p - 1) * W_HIDDEN) : p * W_HIDDEN;
    }
    static constexpr int W_BYTES = FRONT ? W_FIRST + 3 * W_HIDDEN : 3 * W_HIDDEN + W_LAST;
    static constexpr int IN_OFF = W_BYTES;
    static constexpr int RING_OFF = IN_OFF + (IN_RING + (FRONT ? 1 : 0)) * IN_ROW;  // front: + the first row again
    static constexpr int BAR_OFF = RING_OFF + 3 * kRing * kRow;
    static constexpr int BARS = 2 * IN_RING + 2 * 3 * kRing + 2 * 4 * 2 + 4;
    static constexpr int BYTES = BAR_OFF + BARS * 8 + 16 + 128;        // + TMEM slot and stop flag, alignment slack
};

// A CTA's piece of one strip: output rows [oS[3], oE[3]) of the group's last
// layer, and the rows each earlier layer has to provide for them.
// PACK: rows of the bands, which all lie in one piece; no row is left out.
template <bool PACK>
struct Segment {
    int img, xs, xe, x0;  // strip columns [xs, xe); x0: the pixel of lane 0
    int oS[4], oE[4];
    __device__ __forceinline__ Segment(const TcNetArgs& a, long long pos, long long end) {
        if constexpr (PACK) {
            img = xs = xe = x0 = 0;
#pragma unroll
            for (int p = 0; p < 4; ++p) oS[p] = (int)pos - (3 - p), oE[p] = (int)end + (3 - p);
            return;
        }
        const long long strip = pos / a.h;
        img = (int)(strip / a.strips);
        const int s = (int)(strip - (long long)img * a.strips);
        xs = (int)((long long)s * a.w / a.strips);
        xe = (int)((long long)(s + 1) * a.w / a.strips);
        x0 = xs - 3;
        oS[3] = (int)(pos - strip * a.h);
        const long long left = end - pos;
        oE[3] = left < a.h - oS[3] ? oS[3] + (int)left : a.h;
#pragma unroll
        for (int p = 2; p >= 0; --p) {
            oS[p] = max(0, oS[p + 1] - 1);
            oE[p] = min(a.h, oE[p + 1] + 1);
        }
    }
    __device__ __forceinline__ int rows() const { return oE[3] - oS[3]; }
    // Layer p's input and output rows (constant indices, so the arrays stay in registers).
    __device__ __forceinline__ void layer(int p, int h, int* i0, int* i1, int* o0, int* o1) const {
        *i0 = PACK ? oS[0] - 1 : max(0, oS[0] - 1), *i1 = PACK ? oE[0] + 1 : min(h, oE[0] + 1);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k == p) *o0 = oS[k], *o1 = oE[k];
            if (k + 1 == p) *i0 = oS[k], *i1 = oE[k];
        }
    }
};

// PACK: the pixel of lane m of the product, in row y of the bands: column x of row
// yy of frame img, if `in`.
struct PackedPixel {
    int x, img, yy, h1, n;
    bool lane;
    __device__ __forceinline__ PackedPixel(const TcNetArgs& a, int m, int y) {
        const int band = m < 0 ? a.bands : m / (a.w + 1);
        x = m - band * (a.w + 1);
        lane = band < a.bands && x < a.w;
        h1 = a.h + 1;
        n = a.n;
        const int v = lane ? band * a.band_rows + y : -1;  // (rows above the first band: negative)
        img = v < 0 ? (v + 1) / h1 - 1 : v / h1;
        yy = v - img * h1;
    }
    __device__ __forceinline__ void next_row() {
        if (++yy == h1) yy = 0, ++img;
    }
    __device__ __forceinline__ bool in() const { return lane && yy < h1 - 1 && img >= 0 && img < n; }
};

template <bool FRONT, class T, bool PACK>
__global__ void __launch_bounds__(32 * (kEpiWarps + kMmaWarps + (FRONT ? kPrepWarps : 1)), 1) 
    sg_tc_net_kernel(const __grid_constant__ TcNetArgs a) {
    using S = Smem<FRONT>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
    uint8_t* s_in = smem + S::IN_OFF;
    uint64_t* in_full = reinterpret_cast<uint64_t*>(smem + S::BAR_OFF);
    uint64_t* in_empty = in_full + S::IN_RING;
    uint64_t* ring_full = in_empty + S::IN_RING;  // [3][kRing]: the ring that layer p + 1 reads
    uint64_t* ring_empty = ring_full + 3 * kRing;
    uint64_t* acc_full = ring_empty + 3 * kRing;  // [4][2]: the second of a pair is layer 0's of the front kernel only
    uint64_t* acc_free = acc_full + 8;
    uint64_t* drained = acc_free + 8;
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(drained + 4);
    volatile int* s_stop = reinterpret_cast<volatile int*>(s_tmem + 1);
    // (the shuffle tells the compiler that the warp's index is uniform)
    const int warp = __shfl_sync(0xFFFFFFFFU, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

    // weights into core-matrix order (8 output channels x 16 bytes of K each)
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        uint8_t* sw = smem + S::w_off(p);
        const bf16* wpk = a.weights[p];
        if (FRONT && p == 0) {
            for (int i = threadIdx.x; i < 32 * 10; i += blockDim.x) {
                const int n = i / 10, kg = i - n * 10;
                *reinterpret_cast<uint4*>(sw + (kg * 4 + n / 8) * 128 + (n % 8) * 16) =
                    *reinterpret_cast<const uint4*>(wpk + (size_t)n * 80 + kg * 8);
            }
        } else {
            const bool last = !FRONT && p == 3;
            const int nb = last ? 2 : 4;  // N groups per block
            for (int i = threadIdx.x; i < 12 * 5 * nb * 8; i += blockDim.x) {
                const int kg = i / (5 * nb * 8), r = i - kg * (5 * nb * 8), b = r / (nb * 8), n = r - b * (nb * 8);
                const int ky = b % 3 == 0 ? 2 : b % 3 == 1 ? 1 : 0;
                const int kx = kg / 4, ch = (kg & 3) * 8;
                uint4 v = make_uint4(0U, 0U, 0U, 0U);
                if (!last || n < 8) v = *reinterpret_cast<const uint4*>(wpk + (size_t)n * 288 + (ky * 3 + kx) * 32 + ch);
                *reinterpret_cast<uint4*>(sw + (kg * 5 * nb + b * nb + n / 8) * 128 + (n % 8) * 16) = v;
            }
        }
    }
    // the rings start as zeros: pixels 0 and 129 of a row are never written
    for (int i = threadIdx.x; i < (S::BAR_OFF - S::IN_OFF) / 16; i += blockDim.x)
        reinterpret_cast<uint4*>(s_in)[i] = make_uint4(0U, 0U, 0U, 0U);
    if (threadIdx.x == 0) {
        for (int s = 0; s < S::IN_RING; ++s) {
            mbar_init(&in_full[s], FRONT ? kPrepWarps : 1);
            mbar_init(&in_empty[s], 1);
        }
        for (int s = 0; s < 3 * kRing; ++s) {
            mbar_init(&ring_full[s], 4);
            mbar_init(&ring_empty[s], 1);
        }
        for (int s = 0; s < 8; ++s) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_free[s], 4);
        }
        for (int p = 0; p < 4; ++p) mbar_init(&drained[p], 1);
        *s_stop = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    // generic-proxy writes of weights and zeros must be visible to the tensor core (async proxy)
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    if (warp == kEpiWarps) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(saddr(s_tmem)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;
    // TMEM columns: front layer 0 two accumulators of 32, then 3 x 32 (last layer of the back kernel 3 x 16) a layer
    auto acc_col = [](int p) { return FRONT ? (p == 0 ? 0 : 64 + (p - 1) * 96) : p * 96; };
    if (warp < kEpiWarps && !(FRONT && warp < 4)) {  // a layer's accumulators start as zeros
        const uint32_t base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)acc_col(warp >> 2);
        for (int s = 0; s < 3; ++s) tmem_clear32(base + 32 * s);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    const long long total = PACK ? (long long)a.band_rows : (long long)a.n * a.strips * a.h;
    const long long begin = total * blockIdx.x / gridDim.x, end = total * (blockIdx.x + 1) / gridDim.x;
    auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
        mbar_wait(bar, parity, s_stop, a.err, code);
        __syncwarp();
    };

    if (warp >= kEpiWarps && warp < kEpiWarps + kMmaWarps) {
        // A warp per layer issues its products: a row as soon as the row is there
        // and the epilogue has taken the accumulator that it starts anew.  (One
        // warp issuing for all four layers in turn took 4600 clocks a step: its
        // waits and its issue, about 950 clocks a layer, came one after another.)
        const int p = warp - kEpiWarps;
        const bool first = FRONT && p == 0, last = !FRONT && p == 3;
        const uint32_t in_base = saddr(s_in), w_base = saddr(smem + S::w_off(p));
        const uint32_t row_base = p == 0 ? in_base : saddr(smem + S::RING_OFF) + (p - 1) * kRing * kRow;
        const uint32_t slots = p == 0 ? S::IN_RING : kRing;
        uint64_t* full = p == 0 ? in_full : ring_full + (p - 1) * kRing;
        uint64_t* empty = p == 0 ? in_empty : ring_empty + (p - 1) * kRing;
        const uint32_t d = tmem + (uint32_t)acc_col(p);
        uint32_t q = 0, par = 0, sums = 0;  // next row's slot and parity, accumulator rounds begun
        for (long long pos = begin; pos < end;) {
            const Segment<PACK> sg(a, pos, end);
            pos += sg.rows();
            int iS, iE, oS, oE;
            sg.layer(p, a.h, &iS, &iE, &oS, &oE);
            if (first) {
                for (int i = oS; i < oE; ++i) {
                    const uint32_t buf = sums & 1U;
                    const uint32_t q1 = q + 1 == slots ? 0 : q + 1, q2 = q1 + 1 == slots ? 0 : q1 + 1;
                    const uint32_t p1 = par ^ (q1 == 0 ? 1U : 0U), p2 = p1 ^ (q2 == 0 ? 1U : 0U);
                    if (i == oS) {
                        wait(&full[q], par, 1);
                        wait(&full[q1], p1, 1);
                    }
                    wait(&full[q2], p2, 1);
                    if (sums >= 2) wait(&acc_free[buf], ((sums >> 1) - 1U) & 1U, 2);
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t r0 = in_base + q * kPlane, r1 = in_base + q1 * kPlane, r2 = in_base + q2 * kPlane;
                        const uint64_t b0 = smem_desc(w_base, 4 * 128, 128);
                        const uint32_t dd = d + 32U * buf;
                        // K slices: taps (0,1) (2,3) (4,5) (6,7) (8, zero weights)
                        mma_f16(dd, smem_desc(r0, 16, 128), b0, instr_desc<32>(), 0U);
                        mma_f16(dd, smem_desc(r0 + 32, kPlane - 32, 128), b0 + 64, instr_desc<32>(), 1U);
                        mma_f16(dd, smem_desc(r1 + 16, 16, 128), b0 + 128, instr_desc<32>(), 1U);
                        mma_f16(dd, smem_desc(r2, 16, 128), b0 + 192, instr_desc<32>(), 1U);
                        mma_f16(dd, smem_desc(r2 + 32, 0, 128), b0 + 256, instr_desc<32>(), 1U);
                        mma_commit(&acc_full[buf]);
                        mma_commit(&empty[q]);
                        if (i == oE - 1) {  // the segment's last two rows go too
                            mma_commit(&empty[q1]);
                            mma_commit(&empty[q2]);
                        }
                    }
                    __syncwarp();
                    q = q1, par = p1;
                    if (i == oE - 1) {
                        q = q2 + 1 == slots ? 0 : q2 + 1;
                        par = p2 ^ (q == 0 ? 1U : 0U);
                    }
                    ++sums;
                }
            } else {
                // every input row sums into the accumulators of output rows -1, 0, +1; two more
                // rounds without a row let the epilogue take the last of them
                uint32_t off = 0;  // which of the three rotations: the weights' block that meets accumulator 0
                for (int i = iS; i < iE + 2; ++i) {
                    const bool has_row = i < iE;
                    if (has_row) wait(&full[q], par, 1);
                    if (sums > 0) wait(&acc_free[2 * p], (sums - 1U) & 1U, 2);
                    tc_fence_after();
                    if (elect_one()) {
                        if (has_row) {
                            const int nb = last ? 2 : 4;
                            const uint32_t idesc = last ? instr_desc<48>() : instr_desc<96>();
                            const uint64_t ad = smem_desc(row_base + q * kRow, kPlane, 128);
                            const uint64_t bd = smem_desc(w_base + off * (nb * 128), 5 * nb * 128, 128);
                            const uint32_t b_step = 2 * 5 * nb * 8;
#pragma unroll
                            for (int ks = 0; ks < 6; ++ks)
                                mma_f16(d, ad + (2 * (ks & 1) * kPlane + (ks >> 1) * 16) / 16, bd + ks * b_step, idesc, 1U);
                        }
                        mma_commit(&acc_full[2 * p]);
                        if (has_row) mma_commit(&empty[q]);
                    }
                    __syncwarp();
                    if (has_row) {
                        q = q + 1 == slots ? 0 : q + 1;
                        par ^= q == 0 ? 1U : 0U;
                    }
                    off = off == 0 ? 2 : off - 1;
                    ++sums;
                }
            }
        }
        if (*s_stop) {  // after a failure the products in flight finish before the TMEM goes
            volatile int go_on = 0;
            if (elect_one()) mma_commit(&drained[p]);
            __syncwarp();
            mbar_wait(&drained[p], 0, &go_on, a.err, 2);
        }
    } else if (warp >= kEpiWarps) {
        if constexpr (FRONT) {  // RGBA rows -> the network's input rows
            const int i = threadIdx.x - 32 * (kEpiWarps + kMmaWarps);
            const T* rgba = static_cast<const T*>(a.rgba);
            auto input = [&](const Rgba& p, float na, float nb) {  // a pixel's 8 channels
                const float L = ((p.r + p.g) + p.b) * (1.0F / 3.0F);
                const float var = fmaxf(0.0F, nb + na * fmaxf(L, 0.0F));
                const float sig = sqrtf(var) * a.sigma_scale;
                const __nv_bfloat162 v0 = __floats2bfloat162_rn(p.r, p.g), v1 = __floats2bfloat162_rn(p.b, sig);
                return make_uint4(*reinterpret_cast<const uint32_t*>(&v0), *reinterpret_cast<const uint32_t*>(&v1), 0U, 0U);
            };
            auto put = [&](const uint4& o, uint32_t slot, int pixel) {
                *reinterpret_cast<uint4*>(s_in + slot * kPlane + pixel * 16) = o;
                if (slot == 0) *reinterpret_cast<uint4*>(s_in + S::IN_RING * kPlane + pixel * 16) = o;
            };
            uint32_t q = 0, par = 0;  // next slot; the parity its release has once it was used
            bool used = false;
            for (long long pos = begin; pos < end;) {
                const Segment<PACK> sg(a, pos, end);
                pos += sg.rows();
                if constexpr (PACK) {
                    // thread i: stored pixel i (lane i - 1), threads 0 and 1 also pixels 128 and 129
                    const int y1 = sg.oE[0] + 1;
                    int y = sg.oS[0] - 1;
                    PackedPixel at[2] = {PackedPixel(a, i - 1, y), PackedPixel(a, i < kRowPix - kLanes ? i + kLanes - 1 : -1, y)};
                    struct Loaded {
                        Rgba p;
                        float na, nb;
                        bool in;
                    };
                    auto load = [&](const PackedPixel& c, bool on) {
                        Loaded l{Rgba{0.0F, 0.0F, 0.0F, 0.0F}, 0.0F, 0.0F, on && c.in()};
                        if (l.in) {
                            l.p = load_rgba(rgba + 4 * (((long long)c.img * a.h + c.yy) * a.w + c.x));
                            l.na = a.ab[2 * c.img], l.nb = a.ab[2 * c.img + 1];
                        }
                        return l;
                    };
                    Loaded cur[2] = {load(at[0], true), load(at[1], true)};
                    for (; y < y1; ++y) {
                        at[0].next_row();
                        at[1].next_row();
                        const Loaded nxt[2] = {load(at[0], y + 1 < y1), load(at[1], y + 1 < y1)};
                        if (used) wait(&in_empty[q], par, 3);
#pragma unroll
                        for (int k = 0; k < 2; ++k)
                            if (k == 0 || i < kRowPix - kLanes)
                                put(cur[k].in ? input(cur[k].p, cur[k].na, cur[k].nb) : make_uint4(0U, 0U, 0U, 0U), q,
                                    i + k * kLanes);
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&in_full[q]);
                        if (++q == S::IN_RING) {
                            q = 0;
                            par ^= used ? 1U : 0U;
                            used = true;
                        }
                        cur[0] = nxt[0];
                        cur[1] = nxt[1];
                    }
                    continue;
                }
                const T* img = rgba + 4LL * sg.img * a.h * a.w;
                const float na = a.ab[2 * sg.img], nb = a.ab[2 * sg.img + 1];
                // thread i: stored pixel i, threads 0 and 1 also pixels 128 and 129
                const int x = sg.x0 - 1 + i, x2 = x + kLanes;
                const bool in1 = x >= 0 && x < a.w, in2 = i < kRowPix - kLanes && x2 >= 0 && x2 < a.w;
                auto load = [&](bool in, int xx, int y) {
                    return in && y >= 0 && y < a.h ? load_rgba(img + 4 * ((long long)y * a.w + xx))
                                                   : Rgba{0.0F, 0.0F, 0.0F, 0.0F};
                };
                auto store = [&](bool in, const Rgba& p, uint32_t slot, int pixel) {
                    put(in ? input(p, na, nb) : make_uint4(0U, 0U, 0U, 0U), slot, pixel);
                };
                const int y1 = sg.oE[0] + 1;
                int y = sg.oS[0] - 1;
                Rgba p = load(in1, x, y), p2 = load(in2, x2, y);
                for (; y < y1; ++y) {
                    // the next row is asked for before this row's wait
                    const Rgba nxt = load(in1 && y + 1 < y1, x, y + 1), nxt2 = load(in2 && y + 1 < y1, x2, y + 1);
                    if (used) wait(&in_empty[q], par, 3);
                    const bool row_in = y >= 0 && y < a.h;
                    store(in1 && row_in, p, q, i);
                    if (i < kRowPix - kLanes) store(in2 && row_in, p2, q, i + kLanes);
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&in_full[q]);
                    if (++q == S::IN_RING) {
                        q = 0;
                        par ^= used ? 1U : 0U;
                        used = true;
                    }
                    p = nxt;
                    p2 = nxt2;
                }
            }
        } else {  // the front kernel's planes, row by row
            uint32_t n = 0;
            for (long long pos = begin; pos < end;) {
                const Segment<PACK> sg(a, pos, end);
                pos += sg.rows();
                if constexpr (PACK) {
                    // a lane copies the rows of bands `lane` and `lane` + 32 (at most 64 bands)
                    const int y0 = sg.oS[0] - 1, y1 = sg.oE[0] + 1, w1 = a.w + 1;
                    PackedPixel at[2] = {PackedPixel(a, lane * w1, y0), PackedPixel(a, (lane + 32) * w1, y0)};
                    for (int y = y0; y < y1; ++y, ++n) {
                        const uint32_t q = n % S::IN_RING;
                        if (n >= S::IN_RING) wait(&in_empty[q], (n / S::IN_RING - 1U) & 1U, 3);
                        uint8_t* row = s_in + q * kRow;
                        int copies = 0;
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const bool in = at[k].in();
                            const uint32_t ins = __ballot_sync(0xFFFFFFFFU, in);
                            copies += __popc(ins);
                            // bands that stand outside a frame: zeros
                            uint32_t outs = ~ins & __ballot_sync(0xFFFFFFFFU, at[k].lane);
                            for (; outs; outs &= outs - 1) {
                                const int first = (32 * k + __ffs((int)outs) - 1) * w1 + 1;
                                for (int i = lane; i < 4 * a.w; i += 32)
                                    *reinterpret_cast<uint4*>(row + (i / a.w) * kPlane + (first + i % a.w) * 16) =
                                        make_uint4(0U, 0U, 0U, 0U);
                            }
                        }
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_expect_tx(&in_full[q], (uint32_t)copies * 4U * (uint32_t)a.w * 16U);
                        __syncwarp();
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            if (at[k].in())
                                for (int pl = 0; pl < 4; ++pl)
                                    bulk_load(row + pl * kPlane + ((lane + 32 * k) * w1 + 1) * 16,
                                              a.act + ((((long long)at[k].img * 4 + pl) * a.h + at[k].yy) * a.w) * 8,
                                              (uint32_t)a.w * 16U, &in_full[q]);
                            at[k].next_row();
                        }
                        __syncwarp();
                    }
                    continue;
                }
                const int xl = max(0, sg.x0 - 1), xr = min(a.w, sg.x0 - 1 + kRowPix), lead = xl - (sg.x0 - 1);
                const int y0 = max(0, sg.oS[0] - 1), y1 = min(a.h, sg.oE[0] + 1);
                for (int y = y0; y < y1; ++y, ++n) {
                    const uint32_t q = n % S::IN_RING;
                    if (n >= S::IN_RING) wait(&in_empty[q], (n / S::IN_RING - 1U) & 1U, 3);
                    uint8_t* row = s_in + q * kRow;
                    if (y - y0 < S::IN_RING && xr - xl < kRowPix) {
                        // the slot's first row of this strip: zeros where the strip leaves the image
                        for (int i = lane; i < 4 * kRowPix; i += 32) {
                            const int pl = i / kRowPix, c = i - pl * kRowPix;
                            if (c < lead || c >= lead + (xr - xl))
                                *reinterpret_cast<uint4*>(row + pl * kPlane + c * 16) = make_uint4(0U, 0U, 0U, 0U);
                        }
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    }
                    __syncwarp();
                    if (lane == 0) {
                        const uint32_t bytes = (uint32_t)(xr - xl) * 16U;
                        mbar_expect_tx(&in_full[q], 4 * bytes);
#pragma unroll
                        for (int pl = 0; pl < 4; ++pl)
                            bulk_load(row + pl * kPlane + lead * 16,
                                      a.act + ((((long long)sg.img * 4 + pl) * a.h + y) * a.w + xl) * 8, bytes,
                                      &in_full[q]);
                    }
                    __syncwarp();
                }
            }
            if (*s_stop)  // after a failure the copies in flight land before the CTA goes
                for (uint32_t k = n > S::IN_RING ? n - S::IN_RING : 0; k < n; ++k) {
                    volatile int go_on = 0;
                    mbar_wait(&in_full[k % S::IN_RING], (k / S::IN_RING) & 1U, &go_on, a.err, 3);
                }
        }
    } else {  // epilogue of layer p: lane m is pixel x0 + m
        const int p = warp >> 2, m = (warp & 3) * 32 + lane;
        const bool first = FRONT && p == 0;
        const uint32_t t_base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)acc_col(p);
        // the biases stay in registers: reading them back for every row, against the
        // tensor core's own reads of shared memory, had doubled the row's time
        float bias[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) bias[k] = FRONT || p < 3 || k < 3 ? a.bias[p][k] : 0.0F;
        uint64_t* full = acc_full + 2 * p;
        uint64_t* freed = acc_free + 2 * p;
        uint8_t* rows_out = smem + S::RING_OFF + p * kRing * kRow + (m + 1) * 16;  // (p < 3)
        uint32_t ev = 0, out_n = 0;  // accumulators taken, rows handed on
        for (long long pos = begin; pos < end;) {
            const Segment<PACK> sg(a, pos, end);
            pos += sg.rows();
            const int x = sg.x0 + m;
            int iS, iE, oS, oE;
            sg.layer(p, a.h, &iS, &iE, &oS, &oE);
            const int y0 = first ? oS : iS - 1, y1 = first ? oE : iE + 1;
            const bool edge = sg.x0 < 0 || sg.x0 + kLanes > a.w;  // some lanes lie outside the image
            uint32_t turn = 0;  // which accumulator: rounds modulo 3
            PackedPixel at(a, PACK ? m : -1, y0);  // (PACK)
            for (int y = y0; y < y1; ++y, ++ev, turn = turn == 2 ? 0 : turn + 1, at.next_row()) {
                const bool wanted = y >= oS && y < oE;
                if constexpr (!FRONT) {
                    if (p == 3) {  // the last layer: residual onto the frame
                        const bool mine = wanted && (PACK ? at.in() : x >= sg.xs && x < sg.xe);
                        const long long px_n = PACK ? ((long long)at.img * a.h + at.yy) * a.w + at.x
                                                    : ((long long)sg.img * a.h + y) * a.w + x;
                        const T* src = static_cast<const T*>(a.rgba) + 4 * px_n;
                        const Rgba in = mine ? load_rgba(src) : Rgba{0.0F, 0.0F, 0.0F, 0.0F};
                        wait(full, ev & 1U, 4);
                        tc_fence_after();
                        float c[4];
                        tmem_take(t_base + 16 * turn, c);
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(freed);
                        if (mine)
                            store_rgb_keep_alpha(static_cast<T*>(a.out) + 4 * px_n,
                                                 Rgba{in.r + (c[0] + bias[0]), in.g + (c[1] + bias[1]),
                                                      in.b + (c[2] + bias[2]), 0.0F},
                                                 src);
                        continue;
                    }
                }
                const uint32_t q = out_n % kRing;
                if (p < 3 && wanted && out_n >= kRing)  // the slot's last row was read
                    wait(&ring_empty[p * kRing + q], (out_n / kRing - 1U) & 1U, 4);
                const uint32_t buf = first ? ev & 1U : 0U;
                wait(full + buf, (first ? ev >> 1 : ev) & 1U, 4);
                tc_fence_after();
                const uint32_t t = t_base + 32 * (first ? buf : turn);
                uint4 o[4];
                float c[16];
                tmem_load16(t, c);
                o[0] = bias_relu8(c, bias);
                o[1] = bias_relu8(c + 8, bias + 8);
                tmem_load16(t + 16, c);
                if (!first) tmem_clear32(t);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(freed + buf);
                if (!wanted) continue;
                o[2] = bias_relu8(c, bias + 16);
                o[3] = bias_relu8(c + 8, bias + 24);
                if (PACK ? !at.in() : edge && (x < 0 || x >= a.w)) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) o[k] = make_uint4(0U, 0U, 0U, 0U);
                }
                if (p < 3) {  // the next layer's input row
#pragma unroll
                    for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(rows_out + q * kRow + k * kPlane) = o[k];
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ring_full[p * kRing + q]);
                    ++out_n;
                } else if (PACK ? at.in() : x >= sg.xs && x < sg.xe) {  // the front kernel's output planes
                    uint4* dst = reinterpret_cast<uint4*>(a.act) +
                                 (PACK ? ((long long)at.img * 4 * a.h + at.yy) * a.w + at.x
                                       : ((long long)sg.img * 4 * a.h + y) * a.w + x);
#pragma unroll
                    for (int k = 0; k < 4; ++k) dst[(long long)k * a.h * a.w] = o[k];
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kEpiWarps) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kTmemCols));
    }
}

template <bool FRONT, class T, bool PACK>
cudaError_t launch(const TcNetArgs& a, int grid, cudaStream_t st) {
    using S = Smem<FRONT>;
    static_assert(S::BYTES <= 227 * 1024, "shared memory");
    // set on every call: the attribute belongs to the current device
    const cudaError_t e = cudaFuncSetAttribute(sg_tc_net_kernel<FRONT, T, PACK>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, S::BYTES);
    if (e != cudaSuccess) return e;
    sg_tc_net_kernel<FRONT, T, PACK><<<grid, 32 * (kEpiWarps + kMmaWarps + (FRONT ? kPrepWarps : 1)), S::BYTES, st>>>(a);
    return cudaGetLastError();
}
template <bool PACK>
cudaError_t launch_half(bool front, bool f16, const TcNetArgs& a, int grid, cudaStream_t st) {
    if (front) return f16 ? launch<true, __half, PACK>(a, grid, st) : launch<true, float, PACK>(a, grid, st);
    return f16 ? launch<false, __half, PACK>(a, grid, st) : launch<false, float, PACK>(a, grid, st);
}

}  // namespace sgtc

cudaError_t tc_net(bool front, bool f16, TcNetArgs a, cudaStream_t st) {
    using namespace sgtc;
    a.strips = (a.w + kStripMax - 1) / kStripMax;
    // A CTA takes at least eight rows: a segment costs about nine steps beyond its
    // rows (the layers' delays and the rows above and below).  Frames narrow enough
    // for two bands and more go by as many as leave the CTAs eight rows, up to what
    // fits (a band and the zeros after it take w + 1 lanes, the last band no zeros):
    // with fewer rows a CTA they would only pay for the bands' copies (16 x 1250
    // pixels, 7 bands: 61 us, a strip 50).  The stack's rows stay far inside 32 bits.
    constexpr int kCtaRows = 8;
    const long long stack = (long long)a.n * (a.h + 1LL) - 1;
    const long long useful = (stack + kCtaRows * kSmCount - 1) / (kCtaRows * kSmCount);
    const int fit = (kLanes + 1) / (a.w + 1);
    a.bands = (int)(useful < fit ? useful : fit);
    const bool pack = a.bands >= 2 && stack < (1LL << 30);
    a.band_rows = pack ? (int)((stack + a.bands - 1) / a.bands) : 0;
    const long long rows = pack ? a.band_rows : (long long)a.n * a.strips * a.h;
    const long long want = (rows + kCtaRows - 1) / kCtaRows;
    const int grid = (int)(want < kSmCount ? want : kSmCount);
    return pack ? launch_half<true>(front, f16, a, grid, st) : launch_half<false>(front, f16, a, grid, st);
}

}  // namespace cpb
