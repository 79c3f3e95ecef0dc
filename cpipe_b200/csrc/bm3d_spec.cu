// Two-stage colour BM3D on sm_100a (aot_id denoise_bm3d_spec).
//
// The algorithm is the published one (Dabov et al., IEEE TIP 2007; colour
// grouping on luminance; parameters of Lebrun, IPOL 2012).  The reference's
// denoise.bm3d node computes a 2x2 box blend instead
// (src/cpipe/nodes/denoise/bm3d_step1_generator.cpp:33-61); that form lives in
// kernels_nodes.cu and the fused chain.  The exact definition shared with the
// FP64 CPU oracle:
//   colour    orthonormal opponent Y=(R+G+B)/sqrt3, U=(R-B)/sqrt2, V=(R-2G+B)/sqrt6
//   refs      8x8 blocks at min(i*nstep, W-8), same in y
//   matching  integer sum of squared differences of q = rint(clamp(L,0,1)*255)
//             (L = ((R+G)+B)*(1/3) for step 1, Y_basic*(1/sqrt3) for step 2)
//             over all positions within +-(ns-1)/2, d <= floor(64*tau);
//             group = reference + best (d, raster) candidates, at most n2,
//             truncated to a power of two
//   transform orthonormal 8x8 DCT-II, then orthonormal Haar along the group
//   step 1    hard threshold |c| > lambda3d*sigma, weight 1/(sigma^2*kept)
//   step 2    Wiener W = B^2/(B^2+sigma^2) from the basic estimate's group,
//             weight 1/(sigma^2*max(sum W^2, 1e-20)) (1 when the sum is 0);
//             the kernels use the weights times sigma^2, which cancels in
//             num / den and keeps FP32 from overflowing
//   aggregate weight x Kaiser(beta) 8x8 window; estimate = num / den
//
// Kernels:
//   bm3d_prep_kernel    RGBA -> Y,U,V planes + 8-bit matching luminance
//   bm3d_match_kernel   block distances on the integer tensor cores, two passes
//                       (a bound, then the candidates it lets through); small
//                       windows: bm3d_match_each_kernel, a thread per reference
//   bm3d_filter_tc_kernel
//                       the default filter: one warp per group and channel, the
//                       separable DCTs on the FP16 tensor cores (hi/lo split, or
//                       single products for the spot check), the Haar in
//                       registers; one launch over all tiles, whose footprints
//                       overlap: the flush adds with global reductions
//   bm3d_filter_kernel  the FP32 form (transform 1; explicit fused multiply-adds,
//                       the library being built without contraction): lane =
//                       (block, row half); row DCT in registers, column DCT
//                       through a warp shared buffer, Haar along the group with
//                       warp shuffles; aggregation into a shared-memory footprint
//                       of the 8x8 reference tile, then added to the frame
//                       accumulators.  Tiles are launched in P x P phases so that
//                       tiles of one launch have disjoint footprints: the flush
//                       is a plain read-modify-write, no global atomics.
//   bm3d_basic_kernel   step-1 num/den -> basic estimate + step-2 luminance
//   bm3d_final_kernel   num/den -> RGB, alpha copied
#include "bm3d_spec.h"

#include <math.h>

#include <algorithm>
#include <type_traits>

#include "../../include/cpipe_node_abi.h"
#include "kernels.h"

namespace cpb {
namespace {

constexpr float kInvS3 = 0.57735026918962576451F;
constexpr float kInvS2 = 0.70710678118654752440F;
constexpr float kInvS6 = 0.40824829046386301637F;
constexpr float kMinWienerEnergy = 1e-20F;  // floor of sum W^2 in the step-2 weight

// cos(m * pi / 16) for any integer m.
__host__ __device__ constexpr float cos16(int m) {
    m = ((m % 32) + 32) % 32;
    if (m > 16) m = 32 - m;
    float sgn = 1.0F;
    if (m > 8) {
        m = 16 - m;
        sgn = -1.0F;
    }
    return sgn * (m == 0   ? 1.0F
                  : m == 1 ? 0.98078528040323044913F
                  : m == 2 ? 0.92387953251128675613F
                  : m == 3 ? 0.83146961230254523708F
                  : m == 4 ? 0.70710678118654752440F
                  : m == 5 ? 0.55557023301960222474F
                  : m == 6 ? 0.38268343236508977173F
                  : m == 7 ? 0.19509032201612826785F
                           : 0.0F);
}
// Orthonormal DCT-II basis: dctc(k, n) = a(k) cos((2n+1) k pi / 16).
__host__ __device__ constexpr float dctc(int k, int n) {
    return (k == 0 ? 0.35355339059327376220F : 0.5F) * cos16((2 * n + 1) * k);
}

__device__ __forceinline__ int refpos(int i, int n, int nstep) { return min(i * nstep, n - 8); }

__device__ __forceinline__ uint8_t quantise(float l) {
    l = l > 0.0F ? l : 0.0F;
    l = fminf(l, 1.0F);
    return (uint8_t)__float2int_rn(l * 255.0F);
}

// ------------------------------------------------------------------- prep
// gate (optional): the kernels of a gated run return at once unless *gate != 0.
__device__ __forceinline__ bool gated_off(const int* gate) { return gate != nullptr && *gate == 0; }

template <class T>
__global__ void bm3d_prep_kernel(Img in, float* __restrict__ yuv, uint8_t* __restrict__ q, long long npx,
                                 const int* gate) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= in.w || gated_off(gate)) return;
    for (int y = blockIdx.y; y < in.h; y += gridDim.y) {
        const Rgba p = load_rgba(px<const T>(in, x, y));
        const float s = (p.r + p.g) + p.b;
        const long long o = (long long)y * in.w + x;
        yuv[o] = s * kInvS3;
        yuv[npx + o] = (p.r - p.b) * kInvS2;
        yuv[2 * npx + o] = ((p.r + p.b) - 2.0F * p.g) * kInvS6;
        q[o] = quantise(s * (1.0F / 3.0F));
    }
}

// ------------------------------------------------------------------ match
struct MatchArgs {
    int w, h, nrx, nry, nstep, R, ns, n2;  // h: one image's height (blockIdx.z = image)
    int tile, wpr, plane, epitch;          // references per CTA edge; pitches of the staged region (words)
    uint32_t dthr;
    const uint8_t* q;
    uint32_t* list;
    uint8_t* cnt;
    const int* gate;
};

constexpr int kMatchQueue = 32;  // candidates a reference may have waiting
constexpr int kMatchStride = kMatchQueue + 1;  // words per reference: the queue and its length

// The distances come from the integer tensor cores.  With the block energies
// E(p) = sum of q^2 over the 8x8 block at p, a reference r and a candidate c
// are d = E(r) + E(c) - 2 r.c apart, and r.c for 16 references and 8
// neighbouring candidates is one m16n8k32 product for each half of a block.
// The candidates' half energies go in as the product's addend: what comes out
// is s = r.c - ceil(E(c) / 2), and d = E(r) - 2 s - (E(c) & 1).
__device__ __forceinline__ void mma_u8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1, int c0, int c1, int c2, int c3) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};\n"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
}

// A warp's references are 8 columns (lane / 4) x 4 rows (j).  It walks the union
// of their windows in tiles of 8 columns and one row, twice:
//   pass 1 keeps the largest s of 32 buckets a reference.  The 16th largest
//          bucket bounds the 15 best candidates (one bucket may hold nothing
//          better than the reference itself), and lets about 20 of 1521
//          candidates through;
//   pass 2 computes the same distances again, in raster order, and queues what
//          the bound lets through with its (distance, window index) key; a lane
//          sorts one reference's queue.  A queue about to overflow (flat areas
//          tie everywhere) is sorted in early; from then on only a smaller
//          distance than the 15th best passes.
//
// Shared memory: the search region of the CTA's references as four byte-shifted
// word copies (any 4 pixels are one aligned word; pitches 4 mod 8 and 8 mod 32
// keep the fragments' loads free of bank conflicts), the energies, the queues.
//
// Bound by instruction issue (half the cycles, 16 warps an SM): the products
// take a fifth of the integer tensor pipe, the rest is two to three
// instructions per distance, half of them for pairs outside a window, and the
// queueing of what passes.  12 MP chain frame, per stage: 4.7 -> 3.7 ms; 16
// tiles of 256 x 256: 636 -> 436 us, against a thread per reference with
// byte-SIMD |a - b|, dp4a and a sorted list.  (Visiting columns first, and
// with them letting equal distances through, cost 9 ms on the same frame.)
__global__ void __launch_bounds__(256, 2) bm3d_match_kernel(MatchArgs a) {
    extern __shared__ uint32_t s_w[];
    if (gated_off(a.gate)) return;
    const int img = blockIdx.z, row0 = img * a.h;  // images are stacked in rows
    const int i0 = blockIdx.x * a.tile, j0 = blockIdx.y * a.tile;
    const int iL = min(i0 + a.tile - 1, a.nrx - 1), jL = min(j0 + a.tile - 1, a.nry - 1);
    const int rx0 = max(0, refpos(i0, a.w, a.nstep) - a.R);
    const int rx1 = min(a.w, refpos(iL, a.w, a.nstep) + a.R + 8);
    const int ry0 = row0 + max(0, refpos(j0, a.h, a.nstep) - a.R);
    const int ry1 = row0 + min(a.h, refpos(jL, a.h, a.nstep) + a.R + 8);
    const int RW = rx1 - rx0, RH = ry1 - ry0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    int* s_e = reinterpret_cast<int*>(s_w + 4 * a.plane);  // minus the block energies
    uint32_t* s_q = reinterpret_cast<uint32_t*>(s_e + (size_t)a.epitch * (RH - 7)) + warp * 32 * kMatchStride;

    // copy 0: the region's bytes; copy s, row r, word k holds region bytes 4k+s .. 4k+s+3
    uint8_t* bytes = reinterpret_cast<uint8_t*>(s_w);
    for (int r = warp; r < RH; r += warps) {
        const uint8_t* src = a.q + (size_t)(ry0 + r) * a.w + rx0;
        for (int c = lane; c < 4 * a.wpr; c += 32) bytes[4 * r * a.wpr + c] = c < RW ? src[c] : (uint8_t)0;
    }
    __syncthreads();
    for (int r = warp; r < RH; r += warps)
        for (int k = lane; k < a.wpr; k += 32) {
            const uint32_t* p = s_w + r * a.wpr + k;
            const uint32_t lo = p[0], hi = k + 1 < a.wpr ? p[1] : 0U;
#pragma unroll
            for (int s = 1; s < 4; ++s) s_w[s * a.plane + r * a.wpr + k] = __funnelshift_r(lo, hi, 8 * s);
        }
    __syncthreads();
    // energies: a thread walks down a column with the last eight rows' sums in a ring
    {
        constexpr int kRows = 16;
        const int cols = RW - 7, rows = RH - 7;  // block positions
        // (columns past the last position read as zero: s and v stay below 2^22 there)
        for (int i = threadIdx.x; i < rows * (a.epitch - cols); i += blockDim.x) {
            const int y = i / (a.epitch - cols);
            s_e[y * a.epitch + cols + i - y * (a.epitch - cols)] = 0;
        }
        for (int item = threadIdx.x; item < cols * ((rows + kRows - 1) / kRows); item += blockDim.x) {
            const int seg = item / cols, x = item - seg * cols;
            const int y0 = seg * kRows, y1 = min(rows, y0 + kRows);
            const uint32_t* p = s_w + (x & 3) * a.plane + (x >> 2);
            auto row_energy = [&](int y) {
                const uint32_t w0 = p[y * a.wpr], w1 = p[y * a.wpr + 1];
                return (int)__dp4a(w1, w1, __dp4a(w0, w0, 0U));
            };
            int e = 0;
            for (int y = y0; y < y0 + 8; ++y) e += row_energy(y);
            for (int y = y0; y < y1; ++y) {
                s_e[y * a.epitch + x] = -e;
                if (y + 1 < y1) e += row_energy(y + 8) - row_energy(y);
            }
        }
    }
    __syncthreads();

    const int g = lane >> 2, q = lane & 3;
    const int wi = i0 + (warp % (a.tile / 8)) * 8, wj = j0 + (warp / (a.tile / 8)) * 4;  // a warp takes 8 x 4 references
    if (wi >= a.nrx || wj >= a.nry) return;  // (whole warps; no barrier follows)
    // positions of the lane's references (column g, rows j); past the last one the last again
    const int x = refpos(min(wi + g, a.nrx - 1), a.w, a.nstep);
    int y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = row0 + refpos(min(wj + j, a.nry - 1), a.h, a.nstep);
    const int ylo = max(row0, y[0] - a.R), yhi = min(row0 + a.h - 8, y[3] + a.R);
    const int xlo = max(0, refpos(wi, a.w, a.nstep) - a.R);
    const int xhi = min(a.w - 8, refpos(min(wi + 7, a.nrx - 1), a.w, a.nstep) + a.R);
    const int xs = rx0 + ((xlo - rx0) & ~1);  // even in the region, so two energies are one load

    // A fragments: K = 4 bytes (row q / 2, half q % 2) of two block rows; rows 2, 4, 6 further on
    uint32_t af[4][4];
    int er[4];
    {
        const int c = x - rx0 + 4 * (q & 1);
        const uint32_t* p = s_w + (c & 3) * a.plane + (c >> 2) + (q >> 1) * a.wpr;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = y[j] - ry0;
#pragma unroll
            for (int k = 0; k < 4; ++k) af[j][k] = p[(r + 2 * k) * a.wpr];
            er[j] = -s_e[r * a.epitch + x - rx0];
        }
    }
    constexpr int kNone = -0x20000000;  // below every s
    // a candidate may still enter the list when v = E(r) - d = 2 r.c - E(c) is
    // above lim[j]; first from the match threshold
    int lim[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) lim[j] = er[j] - (int)a.dthr - 1;
    uint32_t keys[15];
#pragma unroll
    for (int m = 0; m < 15; ++m) keys[m] = 0xFFFFFFFFU;
    auto insert = [&](uint32_t key) {
        if (key < keys[14]) {
#pragma unroll
            for (int m = 0; m < 15; ++m) {
                const uint32_t lo = min(keys[m], key);
                key = max(keys[m], key);
                keys[m] = lo;
            }
        }
    };

    // The walk over one tile of columns, four rows at a time: body(k, row, s of
    // row j = 0..3 x columns 2q, 2q + 1, the two (negated) energies, whether
    // every row j has the candidates in its window), k = 0..3 the row's place
    // among the four.  Rows that all references have take most of it.
    const int all0 = max(ylo, y[3] - a.R), all1 = min(yhi, y[0] + a.R);
    auto tile_walk = [&](int xt, auto&& body) {
        const int c = xt - rx0 + g + 4 * (q & 1);
        const uint32_t* bp = s_w + (c & 3) * a.plane + (c >> 2) + (ylo - ry0 + (q >> 1)) * a.wpr;
        const int* ep = s_e + (ylo - ry0) * a.epitch + xt - rx0 + 2 * q;
        auto row = [&](auto k, int yy, auto all) {
            const int2 e = *reinterpret_cast<const int2*>(ep + k * a.epitch);
            const int h0 = e.x >> 1, h1 = e.y >> 1;
            const uint32_t f0 = bp[k * a.wpr], f2 = bp[(k + 2) * a.wpr], f4 = bp[(k + 4) * a.wpr], f6 = bp[(k + 6) * a.wpr];
            int s[4][2];
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                int d[4];
                mma_u8(d, af[2 * m][0], af[2 * m + 1][0], af[2 * m][1], af[2 * m + 1][1], f0, f2, h0, h1, h0, h1);
                mma_u8(d, af[2 * m][2], af[2 * m + 1][2], af[2 * m][3], af[2 * m + 1][3], f4, f6, d[0], d[1], d[2], d[3]);
                s[2 * m][0] = d[0], s[2 * m][1] = d[1], s[2 * m + 1][0] = d[2], s[2 * m + 1][1] = d[3];
            }
            body(k, yy, s, e, all);
        };
        using std::integral_constant;
        for (int yy = ylo; yy <= yhi; yy += 4) {
            if (yy >= all0 && yy + 3 <= all1) {
                row(integral_constant<int, 0>{}, yy, std::true_type{});
                row(integral_constant<int, 1>{}, yy + 1, std::true_type{});
                row(integral_constant<int, 2>{}, yy + 2, std::true_type{});
                row(integral_constant<int, 3>{}, yy + 3, std::true_type{});
            } else {
                row(integral_constant<int, 0>{}, yy, std::false_type{});
                if (yy + 1 <= yhi) row(integral_constant<int, 1>{}, yy + 1, std::false_type{});
                if (yy + 2 <= yhi) row(integral_constant<int, 2>{}, yy + 2, std::false_type{});
                if (yy + 3 <= yhi) row(integral_constant<int, 3>{}, yy + 3, std::false_type{});
            }
            bp += 4 * a.wpr;
            ep += 4 * a.epitch;
        }
    };
    auto row_in = [&](int yy, int j) { return (unsigned)(yy - y[j] + a.R) <= 2U * a.R; };
    // whether columns 2q, 2q + 1 of the tile lie in the window of the lane's reference column
    auto column_in = [&](int xt, int c) {
        const int xx = xt + 2 * q + c;
        return xx >= x - a.R && xx <= x + a.R && xx >= 0 && xx <= a.w - 8;
    };

    if (a.n2 > 1) {
        // pass 1: a bucket is one residue of columns modulo 8 and of rows modulo
        // 4, so that good candidates lying together spread over the buckets
        int best[4][4][2];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int j = 0; j < 4; ++j) best[k][j][0] = best[k][j][1] = kNone;
        for (int xt = xs; xt <= xhi; xt += 8) {
            const int off0 = column_in(xt, 0) ? 0 : kNone, off1 = column_in(xt, 1) ? 0 : kNone;
            tile_walk(xt, [&](auto k, int yy, const int (&s)[4][2], const int2&, auto all) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const bool in = all || row_in(yy, j);
                    best[k][j][0] = __viaddmax_s32(s[j][0], in ? off0 : kNone, best[k][j][0]);
                    best[k][j][1] = __viaddmax_s32(s[j][1], in ? off1 : kNone, best[k][j][1]);
                }
            });
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int c = 0; c < 2; ++c) s_q[(8 * j + g) * kMatchStride + 8 * k + 2 * q + c] = (uint32_t)best[k][j][c];
        __syncwarp();
        {  // lane = reference (row lane / 8, column lane % 8): the 16th largest of its buckets
            int top[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) top[m] = kNone;
            for (int b = 0; b < kMatchQueue; ++b) {
                int v = (int)s_q[lane * kMatchStride + b];
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    const int hi = max(top[m], v);
                    v = min(top[m], v);
                    top[m] = hi;
                }
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; ++j) lim[j] = max(lim[j], 2 * __shfl_sync(0xFFFFFFFFU, top[15], 8 * j + g) - 1);
            s_q[lane * kMatchStride + kMatchQueue] = 0;
        }
        __syncwarp();
        // pass 2
        const int own = a.R * a.ns + a.R;  // window index of the reference itself
        int er_own = er[0];                // energy of the lane's reference as the queue's owner (row lane / 8, column lane % 8)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int v = __shfl_sync(0xFFFFFFFFU, er[j], 4 * (lane & 7));
            if (lane >> 3 == j) er_own = v;
        }
        auto drain = [&]() {
            __syncwarp();
            uint32_t* mine = s_q + lane * kMatchStride;
            const int n = (int)mine[kMatchQueue];
            const int most = __reduce_max_sync(0xFFFFFFFFU, n);
            for (int i = 0; i < most; ++i) {
                const uint32_t key = i < n ? mine[i] : 0xFFFFFFFFU;
                insert((key >> 11) <= a.dthr && (int)(key & 2047U) != own ? key : 0xFFFFFFFFU);
            }
            mine[kMatchQueue] = 0;
            __syncwarp();
        };
        bool full = false;
        // key of candidate (column, row) = key0[j] + row * ns + column - (v << 11)
        uint32_t key0[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            key0[j] = ((uint32_t)er[j] << 11) + (uint32_t)((a.R - y[j]) * a.ns + a.R - x + 2 * q);
        const int tiles = (xhi - xs) / 8 + 1;
        unsigned col0 = 0, col1 = 0;  // bit t: column 2q (2q + 1) of tile t lies in the window
        for (int t = 0; t < tiles; ++t) {
            col0 |= column_in(xs + 8 * t, 0) ? 1U << t : 0U;
            col1 |= column_in(xs + 8 * t, 1) ? 1U << t : 0U;
        }
        const int c = xs - rx0 + g + 4 * (q & 1);
        const uint32_t* brow = s_w + (c & 3) * a.plane + (c >> 2) + (ylo - ry0 + (q >> 1)) * a.wpr;
        const int* erow = s_e + (ylo - ry0) * a.epitch + xs - rx0 + 2 * q;
        for (int yy = ylo; yy <= yhi; ++yy, brow += a.wpr, erow += a.epitch) {
            unsigned rows = 0;  // bits of the rows j with this row in their windows
#pragma unroll
            for (int j = 0; j < 4; ++j) rows |= row_in(yy, j) ? 3U << (6 - 2 * j) : 0U;
#pragma unroll 2
            for (int t = 0; t < tiles; ++t) {
                const uint32_t* bp = brow + 2 * t;
                const int2 e = *reinterpret_cast<const int2*>(erow + 8 * t);
                const uint32_t f0 = bp[0], f2 = bp[2 * a.wpr], f4 = bp[4 * a.wpr], f6 = bp[6 * a.wpr];
                int v[4][2];
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const uint32_t(&u)[4] = af[2 * m];
                    const uint32_t(&w)[4] = af[2 * m + 1];
                    int d[4], p[4];  // twice r.c (two chains of products), minus E
                    mma_u8(d, u[0], w[0], u[1], w[1], f0, f2, e.x, e.y, e.x, e.y);
                    mma_u8(p, u[0], w[0], u[1], w[1], f0, f2, d[0], d[1], d[2], d[3]);
                    mma_u8(d, u[2], w[2], u[3], w[3], f4, f6, p[0], p[1], p[2], p[3]);
                    mma_u8(p, u[2], w[2], u[3], w[3], f4, f6, d[0], d[1], d[2], d[3]);
                    v[2 * m][0] = p[0], v[2 * m][1] = p[1], v[2 * m + 1][0] = p[2], v[2 * m + 1][1] = p[3];
                }
                unsigned pass = 0;  // bit 7 - (2 j + c): lim - v is negative
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    pass = __funnelshift_l((unsigned)(lim[j] - v[j][0]), pass, 1);
                    pass = __funnelshift_l((unsigned)(lim[j] - v[j][1]), pass, 1);
                }
                pass &= rows & ((col0 >> t & 1U ? 0xAAU : 0U) | (col1 >> t & 1U ? 0x55U : 0U));
                if (__any_sync(0xFFFFFFFFU, pass != 0)) {
                    while (pass) {
                        const int b = __clz(pass) - 24;  // 2 j + c
                        pass &= ~(128U >> b);
                        const bool c1 = b & 1;
                        const int j = b >> 1;
                        const int v0 = c1 ? v[0][1] : v[0][0], v1 = c1 ? v[1][1] : v[1][0];
                        const int v2 = c1 ? v[2][1] : v[2][0], v3 = c1 ? v[3][1] : v[3][0];
                        const int vv = j & 2 ? (j & 1 ? v3 : v2) : (j & 1 ? v1 : v0);
                        const uint32_t k0 = j & 2 ? (j & 1 ? key0[3] : key0[2]) : (j & 1 ? key0[1] : key0[0]);
                        uint32_t* mine = s_q + (8 * j + g) * kMatchStride;
                        const uint32_t at = atomicAdd(mine + kMatchQueue, 1U);
                        mine[at] = k0 + (uint32_t)(yy * a.ns + xs + 8 * t + c1) - ((uint32_t)vv << 11);
                        full |= at >= kMatchQueue - 8;
                    }
                    if (__any_sync(0xFFFFFFFFU, full)) {  // a tile's row may queue eight more
                        full = false;
                        drain();
                        // only a smaller distance than the 15th best can still enter:
                        // the walk is in raster order, so an equal one has a larger index
                        const int bound = keys[14] == 0xFFFFFFFFU ? 2 * kNone : er_own - (int)(keys[14] >> 11);
#pragma unroll
                        for (int j = 0; j < 4; ++j) lim[j] = max(lim[j], __shfl_sync(0xFFFFFFFFU, bound, 8 * j + g));
                    }
                }
            }
        }
        drain();
    }
    // lane = reference: write its list
    const int ri = wi + (lane & 7), rj = wj + (lane >> 3);
    if (ri >= a.nrx || rj >= a.nry) return;
    const int rx = refpos(ri, a.w, a.nstep), ry = row0 + refpos(rj, a.h, a.nstep);
    const long long ref = ((long long)img * a.nry + rj) * a.nrx + ri;
    uint32_t* out = a.list + ref * 16;
    out[0] = ((uint32_t)ry << 16) | (uint32_t)rx;
    int n = 1;
#pragma unroll
    for (int m = 0; m < 15; ++m) {
        if (m < a.n2 - 1 && keys[m] != 0xFFFFFFFFU) {
            const int widx = (int)(keys[m] & 2047U);
            const int dy = widx / a.ns - a.R, dx = widx % a.ns - a.R;
            out[1 + m] = ((uint32_t)(ry + dy) << 16) | (uint32_t)(rx + dx);
            ++n;
        }
    }
    a.cnt[ref] = (uint8_t)n;
}

// The same lists for small windows: a thread per reference visits its own
// candidates only, where the warp's 8 x 4 references above share the union of
// their windows (14 times a 5 x 5 window's pairs at step 3).  Distances with
// byte-SIMD |a - b| and dp4a; a sorted register list keeps the 15 best keys.
// The region of 16 x 16 references is staged as four byte-shifted word copies.
constexpr int kMatchEachTile = 16;
__global__ void __launch_bounds__(256) bm3d_match_each_kernel(MatchArgs a) {
    extern __shared__ uint32_t s_w[];
    const int wpr = a.wpr, plane = a.plane;  // words per staged row and per shifted copy
    if (gated_off(a.gate)) return;
    const int img = blockIdx.z, row0 = img * a.h;  // images are stacked in rows
    const int i0 = blockIdx.x * kMatchEachTile, j0 = blockIdx.y * kMatchEachTile;
    const int iL = min(i0 + kMatchEachTile - 1, a.nrx - 1), jL = min(j0 + kMatchEachTile - 1, a.nry - 1);
    const int rx0 = max(0, refpos(i0, a.w, a.nstep) - a.R);
    const int rx1 = min(a.w, refpos(iL, a.w, a.nstep) + a.R + 8);
    const int ry0 = row0 + max(0, refpos(j0, a.h, a.nstep) - a.R);
    const int ry1 = row0 + min(a.h, refpos(jL, a.h, a.nstep) + a.R + 8);
    const int RW = rx1 - rx0, RH = ry1 - ry0;
    // Copy s, row r, word k holds region bytes 4k+s .. 4k+s+3 (little endian).
    for (int idx = threadIdx.x; idx < 4 * RH * wpr; idx += blockDim.x) {
        const int s = idx / (RH * wpr), rem = idx - s * RH * wpr;
        const int r = rem / wpr, k = rem - r * wpr;
        const uint8_t* row = a.q + (size_t)(ry0 + r) * a.w + rx0;
        const int c0 = 4 * k + s;
        uint32_t word = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int cc = c0 + b;
            word |= (cc < RW ? (uint32_t)row[cc] : 0U) << (8 * b);
        }
        s_w[s * plane + r * wpr + k] = word;
    }
    __syncthreads();
    const int i = i0 + (int)(threadIdx.x % kMatchEachTile), j = j0 + (int)(threadIdx.x / kMatchEachTile);
    if (i >= a.nrx || j >= a.nry) return;
    const int x = refpos(i, a.w, a.nstep), y = row0 + refpos(j, a.h, a.nstep);
    uint32_t rw[16];
    {
        const int c = x - rx0;
        const uint32_t* p = s_w + (c & 3) * plane + (y - ry0) * wpr + (c >> 2);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            rw[2 * r] = p[r * wpr];
            rw[2 * r + 1] = p[r * wpr + 1];
        }
    }
    uint32_t keys[15];
#pragma unroll
    for (int m = 0; m < 15; ++m) keys[m] = 0xFFFFFFFFU;
    const int ylo = max(row0, y - a.R), yhi = min(row0 + a.h - 8, y + a.R);
    const int xlo = max(0, x - a.R), xhi = min(a.w - 8, x + a.R);
    if (a.n2 > 1) {
        // Columns of the search window outer, rows inner: the candidate's eight
        // rows sit in a register ring (slot = row & 7, rows counted from ylo), so
        // each candidate loads one new row.  Keys are unique (distance, window
        // index), so the sorted list does not depend on the visiting order.
        const int ny = yhi - ylo + 1;
        for (int xx = xlo; xx <= xhi; ++xx) {
            const int c = xx - rx0;
            const uint32_t* colp = s_w + (c & 3) * plane + (ylo - ry0) * wpr + (c >> 2);
            const uint32_t wcol = (uint32_t)((ylo - y + a.R) * a.ns + a.R - x + xx);
            uint32_t cw[8][2];
#pragma unroll
            for (int r = 0; r < 7; ++r) {
                cw[r][0] = colp[r * wpr];
                cw[r][1] = colp[r * wpr + 1];
            }
            cw[7][0] = cw[7][1] = 0U;
            for (int y0 = 0; y0 < ny; y0 += 8) {
                const uint32_t* rp = colp + (y0 + 7) * wpr;
#pragma unroll
                for (int st = 0; st < 8; ++st) {
                    if (y0 + st < ny) {
                        cw[(st + 7) & 7][0] = rp[st * wpr];
                        cw[(st + 7) & 7][1] = rp[st * wpr + 1];
                        uint32_t d = 0;
#pragma unroll
                        for (int r = 0; r < 8; ++r) {
                            const uint32_t a0 = __vabsdiffu4(rw[2 * r], cw[(st + r) & 7][0]);
                            d = __dp4a(a0, a0, d);
                            const uint32_t a1 = __vabsdiffu4(rw[2 * r + 1], cw[(st + r) & 7][1]);
                            d = __dp4a(a1, a1, d);
                        }
                        const int yy = ylo + y0 + st;
                        if (d <= a.dthr && (xx != x || yy != y)) {
                            uint32_t key = (d << 11) | (wcol + (uint32_t)((y0 + st) * a.ns));
                            if (key < keys[14]) {
#pragma unroll
                                for (int m = 0; m < 15; ++m) {
                                    const uint32_t lo = min(keys[m], key);
                                    key = max(keys[m], key);
                                    keys[m] = lo;
                                }
                            }
                        }
                    }
                }
            }
        }
    }
    const long long ref = ((long long)img * a.nry + j) * a.nrx + i;
    uint32_t* out = a.list + ref * 16;
    out[0] = ((uint32_t)y << 16) | (uint32_t)x;
    int n = 1;
#pragma unroll
    for (int m = 0; m < 15; ++m) {
        if (m < a.n2 - 1 && keys[m] != 0xFFFFFFFFU) {
            const int widx = (int)(keys[m] & 2047U);
            const int dy = widx / a.ns - a.R, dx = widx % a.ns - a.R;
            out[1 + m] = ((uint32_t)(y + dy) << 16) | (uint32_t)(x + dx);
            ++n;
        }
    }
    a.cnt[ref] = (uint8_t)n;
}

// ----------------------------------------------------------------- filter
struct FilterArgs {
    int w, h, nrx, nry, nstep, R, ntx, nty, phases, fw;
    float sigma2, thr;
    long long npx;
    const uint32_t* list;
    const uint8_t* cnt;
    const float* noisy;
    const float* basic;
    float* acc;  // num of channel c at c*npx, den at (3+c)*npx
    const int* gate;
    float kaiser[64];
    float kaiser1[8];
    int np;  // tensor-core form: row pitch of the footprint planes (= 4 mod 32)
};

constexpr int kBufStride = 65;                 // floats per block in a warp buffer
constexpr int kWarpBuf = 16 * kBufStride;      // one group of 16 blocks
constexpr int kFilterWarps = 8;
constexpr int kRefTile = 8;                    // reference blocks per tile edge

__device__ __forceinline__ void haar_forward(float (&Z)[32], int N, int b, bool act) {
    for (int s = 1; s < N; s <<= 1) {
        const bool part = act && (b & (s - 1)) == 0;
        const bool odd = (b & s) != 0;
#pragma unroll
        for (int e = 0; e < 32; ++e) {
            const float p = __shfl_xor_sync(0xFFFFFFFFU, Z[e], 2 * s);
            if (part) Z[e] = odd ? (p - Z[e]) * kInvS2 : (Z[e] + p) * kInvS2;
        }
    }
}
__device__ __forceinline__ void haar_inverse(float (&Z)[32], int N, int b, bool act) {
    for (int s = N >> 1; s >= 1; s >>= 1) {
        const bool part = act && (b & (s - 1)) == 0;
        const bool odd = (b & s) != 0;
#pragma unroll
        for (int e = 0; e < 32; ++e) {
            const float p = __shfl_xor_sync(0xFFFFFFFFU, Z[e], 2 * s);
            if (part) Z[e] = odd ? (p - Z[e]) * kInvS2 : (Z[e] + p) * kInvS2;
        }
    }
}

// 3D transform of the group held by one warp.  Lane (b, hh) loads rows
// 4hh..4hh+3 of block b; on return it holds frequency rows 0..7 of frequency
// columns 4hh..4hh+3 (Z[kr*4 + jj]) after the Haar transform along the group.
__device__ __forceinline__ void forward3d(const float* img, int fw, int bx, int by, int hh, int b, bool act, int N,
                                          float* buf, float (&Z)[32]) {
    if (act) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float* row = img + (by + 4 * hh + r) * fw + bx;
            float v[8];
#pragma unroll
            for (int n = 0; n < 8; ++n) v[n] = row[n];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                float s = dctc(k, 0) * v[0];
#pragma unroll
                for (int n = 1; n < 8; ++n) s = __fmaf_rn(dctc(k, n), v[n], s);
                buf[b * kBufStride + (4 * hh + r) * 8 + k] = s;
            }
        }
    }
    __syncwarp();
    float z[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) z[r][jj] = act ? buf[b * kBufStride + r * 8 + 4 * hh + jj] : 0.0F;
    __syncwarp();
#pragma unroll
    for (int kr = 0; kr < 8; ++kr)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
            float s = dctc(kr, 0) * z[0][jj];
#pragma unroll
            for (int r = 1; r < 8; ++r) s = __fmaf_rn(dctc(kr, r), z[r][jj], s);
            Z[kr * 4 + jj] = s;
        }
    haar_forward(Z, N, b, act);
}

template <int STAGE>
__global__ void __launch_bounds__(256, 2) bm3d_filter_kernel(FilterArgs a, int phx, int phy) {
    extern __shared__ float sm[];
    const int c = blockIdx.z % 3, img = blockIdx.z / 3, row0 = img * a.h;  // h: one image's height
    const int tx = blockIdx.x * a.phases + phx, ty = blockIdx.y * a.phases + phy;
    if (tx >= a.ntx || ty >= a.nty || gated_off(a.gate)) return;
    const int i0 = tx * kRefTile, j0 = ty * kRefTile;
    const int i1 = min(i0 + kRefTile, a.nrx), j1 = min(j0 + kRefTile, a.nry);
    const int fx0 = max(0, refpos(i0, a.w, a.nstep) - a.R);
    const int fx1 = min(a.w, refpos(i1 - 1, a.w, a.nstep) + a.R + 8);
    const int fy0 = row0 + max(0, refpos(j0, a.h, a.nstep) - a.R);
    const int fy1 = row0 + min(a.h, refpos(j1 - 1, a.h, a.nstep) + a.R + 8);
    const int fw = fx1 - fx0, fn = fw * (fy1 - fy0);
    const int FN = a.fw * a.fw;
    float* s_num = sm;
    float* s_den = sm + FN;
    float* s_img = sm + 2 * FN;
    float* s_bas = sm + 3 * FN;
    float* s_buf = sm + (STAGE == 2 ? 4 : 3) * FN;
    float* s_k = s_buf + kFilterWarps * kWarpBuf;
    const float* gz = a.noisy + (long long)c * a.npx;
    const float* gb = STAGE == 2 ? a.basic + (long long)c * a.npx : nullptr;
    for (int idx = threadIdx.x; idx < fn; idx += blockDim.x) {
        const int yy = idx / fw, xx = idx - yy * fw;
        const long long o = (long long)(fy0 + yy) * a.w + fx0 + xx;
        s_num[idx] = 0.0F;
        s_den[idx] = 0.0F;
        s_img[idx] = gz[o];
        if (STAGE == 2) s_bas[idx] = gb[o];
    }
    if (threadIdx.x < 64) s_k[threadIdx.x] = a.kaiser[threadIdx.x];
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, b = lane >> 1, hh = lane & 1;
    float* buf = s_buf + warp * kWarpBuf;
    const int nti = i1 - i0, nref = nti * (j1 - j0);
    for (int k = warp; k < nref; k += kFilterWarps) {
        const long long ref = ((long long)img * a.nry + j0 + k / nti) * a.nrx + i0 + k % nti;
        const int cnt = a.cnt[ref];
        const int N = cnt >= 16 ? 16 : cnt >= 8 ? 8 : cnt >= 4 ? 4 : cnt >= 2 ? 2 : 1;
        const bool act = b < N;
        int bx = 0, by = 0;
        if (act) {
            const uint32_t p = a.list[ref * 16 + b];
            bx = (int)(p & 0xFFFFU) - fx0;
            by = (int)(p >> 16) - fy0;
        }
        float Z[32];
        forward3d(s_img, fw, bx, by, hh, b, act, N, buf, Z);
        float wgt;
        if (STAGE == 1) {
            unsigned kept = 0;
#pragma unroll
            for (int e = 0; e < 32; ++e) {
                const bool keep = fabsf(Z[e]) > a.thr;
                Z[e] = keep ? Z[e] : 0.0F;
                kept += keep ? 1U : 0U;
            }
            kept = __reduce_add_sync(0xFFFFFFFFU, kept);
            // weight x sigma^2 (the factor cancels in num / den): 1/kept, or sigma^2
            wgt = kept > 0U ? 1.0F / (float)kept : a.sigma2;
        } else {
            float B[32];
            forward3d(s_bas, fw, bx, by, hh, b, act, N, buf, B);
            float sw2 = 0.0F;
#pragma unroll
            for (int e = 0; e < 32; ++e) {
                const float b2 = B[e] * B[e];
                const float W = b2 / (b2 + a.sigma2);
                Z[e] = Z[e] * W;
                sw2 = __fmaf_rn(W, W, sw2);
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) sw2 += __shfl_xor_sync(0xFFFFFFFFU, sw2, off);
            wgt = sw2 > 0.0F ? 1.0F / fmaxf(sw2, kMinWienerEnergy) : a.sigma2;
        }
        haar_inverse(Z, N, b, act);
        if (act) {
#pragma unroll
            for (int r = 0; r < 8; ++r)
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    float s = dctc(0, r) * Z[jj];
#pragma unroll
                    for (int kr = 1; kr < 8; ++kr) s = __fmaf_rn(dctc(kr, r), Z[kr * 4 + jj], s);
                    buf[b * kBufStride + r * 8 + 4 * hh + jj] = s;
                }
        }
        __syncwarp();
        if (act) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int row = 4 * hh + r;
                float v[8];
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) v[kk] = buf[b * kBufStride + row * 8 + kk];
                float* dn = s_num + (by + row) * fw + bx;
                float* dd = s_den + (by + row) * fw + bx;
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    float s = dctc(0, n) * v[0];
#pragma unroll
                    for (int kk = 1; kk < 8; ++kk) s = __fmaf_rn(dctc(kk, n), v[kk], s);
                    const float kw = wgt * s_k[row * 8 + n];
                    atomicAdd(dn + n, kw * s);
                    atomicAdd(dd + n, kw);
                }
            }
        }
        __syncwarp();
    }
    __syncthreads();
    float* gn = a.acc + (long long)c * a.npx;
    float* gd = a.acc + (long long)(3 + c) * a.npx;
    for (int idx = threadIdx.x; idx < fn; idx += blockDim.x) {
        const int yy = idx / fw, xx = idx - yy * fw;
        const long long o = (long long)(fy0 + yy) * a.w + fx0 + xx;
        gn[o] += s_num[idx];
        gd[o] += s_den[idx];
    }
}

// ------------------------------------------- filter on the tensor cores
// The 2D DCTs of a group as separable 8-point transforms on
// mma.sync.m16n8k8 (FP16 operands, FP32 accumulation).  Every operand is split
// hi/lo (x = hi + lo, both FP16): a*b ~ ahi*bhi + alo*bhi + ahi*blo, which keeps
// FP32-level accuracy for the threshold and Wiener decisions.  One m16 tile
// holds two blocks of the group (rows 0-7 block 2t, rows 8-15 block 2t+1):
//   forward  Rc = X^T C^T   rows (block, x), K = y  (columns of each block)
//            H  = Rc^T C^T  rows (block, v), K = x  (rows; Rc^T per 8x8 piece by
//                                                    movmatrix.trans in registers)
//   Haar     along the group, in FP32: a lane holds the same two coefficients
//            (v = g, u = 2q, 2q+1) of all 16 blocks, so every level is register
//            arithmetic (unnormalised butterflies; the normalisation is an exact
//            power of two applied in the shrink step)
//   shrink   hard threshold / Wiener on H (FP32)
//   inverse  Rr = H C       rows (block, v), K = u  (the accumulator is the A
//                                                    operand as it stands)
//            X' = Rr^T C    rows (block, x), K = v
// The DCT matrix enters only as B fragments: four registers per lane.
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 8x8 b16 matrix held as a fragment (row lane/4, columns 2(lane%4)..+1) -> its transpose.
__device__ __forceinline__ uint32_t movtrans(uint32_t x) {
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(y) : "r"(x));
    return y;
}
__device__ __forceinline__ void mma1688(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0));
}
// The same with a zero addend (one set of zero registers serves every call).
__device__ __forceinline__ void mma1688_0(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};\n"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0), "f"(0.0F));
}
// a - b, two at a time (the product with -1 is exact).
__device__ __forceinline__ float2 sub2(const float2& a, const float2& b) {
    return __ffma2_rn(b, make_float2(-1.0F, -1.0F), a);
}
// FP16 hi/lo halves of two floats, packed as (x0, x1) pairs.
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x0, x1);
    const float2 hf = __half22float2(h);
    const float2 r = sub2(make_float2(x0, x1), hf);
    const __half2 l = __floats2half2_rn(r.x, r.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
// c = A * B over one 8-wide k-step with A = (a0, a1) given as FP32 pairs and B split hi/lo.
__device__ __forceinline__ void mma_split(float (&c)[4], float a00, float a01, float a10, float a11, uint32_t bh,
                                          uint32_t bl) {
    uint32_t h0, l0, h1, l1;
    split2(a00, a01, h0, l0);
    split2(a10, a11, h1, l1);
    mma1688_0(c, h0, h1, bh);
    mma1688(c, l0, l1, bh);
    mma1688(c, h0, h1, bl);
}
// The same with A = each 8x8 piece of an accumulator tile transposed.
__device__ __forceinline__ void mma_split_t(float (&c)[4], const float (&r)[4], uint32_t bh, uint32_t bl) {
    uint32_t h0, l0, h1, l1;
    split2(r[0], r[1], h0, l0);
    split2(r[2], r[3], h1, l1);
    h0 = movtrans(h0);
    l0 = movtrans(l0);
    h1 = movtrans(h1);
    l1 = movtrans(l1);
    mma1688_0(c, h0, h1, bh);
    mma1688(c, l0, l1, bh);
    mma1688(c, h0, h1, bl);
}

// Single FP16 products (transform 2, the screening form): A rounded once to
// FP16, B = the DCT matrix's FP16 part, FP32 accumulation -- about 2^-11
// relative per product instead of the split form's FP32-level accuracy.
__device__ __forceinline__ uint32_t pack2(float x0, float x1) {
    const __half2 h = __floats2half2_rn(x0, x1);
    return *reinterpret_cast<const uint32_t*>(&h);
}
template <bool SPLIT>
__device__ __forceinline__ void mma_prod(float (&c)[4], float a00, float a01, float a10, float a11, uint32_t bh,
                                         uint32_t bl) {
    if (SPLIT) {
        mma_split(c, a00, a01, a10, a11, bh, bl);
    } else {
        mma1688_0(c, pack2(a00, a01), pack2(a10, a11), bh);
    }
}
template <bool SPLIT>
__device__ __forceinline__ void mma_prod_t(float (&c)[4], const float (&r)[4], uint32_t bh, uint32_t bl) {
    if (SPLIT) {
        mma_split_t(c, r, bh, bl);
    } else {
        mma1688_0(c, movtrans(pack2(r[0], r[1])), movtrans(pack2(r[2], r[3])), bh);
    }
}

struct DctFrags {
    uint32_t fh, fl;  // B[k][n] = C[n][k] (k = 2q, 2q+1; n = g): products with C^T
    uint32_t ih, il;  // B[k][n] = C[k][n]: products with C
};
__device__ __forceinline__ DctFrags dct_frags(int g, int q) {
    DctFrags d;
    split2(dctc(g, 2 * q), dctc(g, 2 * q + 1), d.fh, d.fl);
    split2(dctc(2 * q, g), dctc(2 * q + 1, g), d.ih, d.il);
    return d;
}

// One level of the unnormalised Haar along the group: block b = 2t + (e >= 2)
// pairs with b + S, (lo, hi) -> (lo + hi, lo - hi).  A level is its own
// transpose, so the inverse runs the same levels in reverse order.  The
// orthonormal transform's coefficient at position b is the unnormalised one
// times 2^(-k/2), k = log2 N for b = 0 and ctz(b) + 1 otherwise: the shrink
// step compares against thresholds scaled by 2^(k/2) (the Wiener step against
// sigma^2 2^k) and multiplies the kept coefficients by 2^-k, exactly, which is
// the forward and the inverse normalisation together.
template <int S>
__device__ __forceinline__ void haar_level(float (&H)[8][4]) {
    // (two coefficients to an instruction)
    auto butterfly = [](float& lo0, float& lo1, float& hi0, float& hi1) {
        const float2 lo = make_float2(lo0, lo1), hi = make_float2(hi0, hi1);
        const float2 sum = __fadd2_rn(lo, hi), dif = sub2(lo, hi);
        lo0 = sum.x, lo1 = sum.y, hi0 = dif.x, hi1 = dif.y;
    };
    if (S == 1) {
#pragma unroll
        for (int t = 0; t < 8; ++t) butterfly(H[t][0], H[t][1], H[t][2], H[t][3]);
    } else {
        constexpr int D = S / 2;  // distance in t
#pragma unroll
        for (int t = 0; t < 8; t += 2 * D) butterfly(H[t][0], H[t][1], H[t + D][0], H[t + D][1]);
    }
}
// k of position b > 0 (compile-time after unrolling); position 0 uses log2 N.
__device__ __forceinline__ constexpr int haar_k(int b) { return (b & 1) ? 1 : (b & 2) ? 2 : (b & 4) ? 3 : 4; }
// 2^e for a small integer e (exact).
__device__ __forceinline__ float exp2i(int e) { return __int_as_float((127 + e) << 23); }

// Forward 2D DCT and Haar of one group of N blocks read from `img` (row pitch P;
// off[b]: block b's offset in the footprint plane, block 0's for b >= N).
// H[t][e]: block 2t (e < 2) or 2t + 1 (e >= 2), coefficient (v = g, u = 2q + (e & 1)).
// The pairs of blocks are walked in the segments that a group size of 2, 4, 8 or
// 16 takes whole, so that a segment's pairs overlap without a branch between them.
template <bool SPLIT>
__device__ __forceinline__ void tc_forward(const float* img, int P, const int* off, int N, const DctFrags& d,
                                           float (&H)[8][4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    img += 2 * q * P + g;
    auto pair = [&](int t, int o0, int o1) {
        float rc[4];
        mma_prod<SPLIT>(rc, img[o0], img[o0 + P], img[o1], img[o1 + P], d.fh, d.fl);  // rows (block, x = g), columns v
        mma_prod_t<SPLIT>(H[t], rc, d.fh, d.fl);                                     // rows (block, v = g), columns u
    };
    auto segment = [&](int t0, int n) {  // n = 2 or 4 pairs
#pragma unroll
        for (int t = t0; t < t0 + n; t += 2) {
            const int4 o = *reinterpret_cast<const int4*>(off + 2 * t);
            pair(t, o.x, o.y);
            pair(t + 1, o.z, o.w);
        }
    };
#pragma unroll
    for (int t = 0; t < 8; ++t) H[t][0] = H[t][1] = H[t][2] = H[t][3] = 0.0F;
    const int4 o = *reinterpret_cast<const int4*>(off);
    pair(0, o.x, o.y);
    if (N == 1) H[0][2] = H[0][3] = 0.0F;
    if (N > 2) pair(1, o.z, o.w);
    if (N > 4) segment(2, 2);
    if (N > 8) segment(4, 4);
    if (N > 1) haar_level<1>(H);
    if (N > 2) haar_level<2>(H);
    if (N > 4) haar_level<4>(H);
    if (N > 8) haar_level<8>(H);
}

// Inverse Haar and 2D DCT of a group; its pixels, weighted by (kw0, kw1), are added
// to the plane `num` at the blocks' offsets: a lane holds (x = g, y = 2q, 2q + 1) of
// every block, so an atomic instruction covers 8 columns x every other row of a
// block, 32 pixels in 32 banks (P = 4 mod 32).
template <bool SPLIT>
__device__ __forceinline__ void tc_inverse_add(float (&H)[8][4], int N, const DctFrags& d, float kw0, float kw1, float* num,
                                               int P, const int* off) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    num += 2 * q * P + g;
    if (N > 8) haar_level<8>(H);
    if (N > 4) haar_level<4>(H);
    if (N > 2) haar_level<2>(H);
    if (N > 1) haar_level<1>(H);
    auto inverse = [&](int t) {  // in place: pixels (x = g, y = 2q + (e & 1))
        float rr[4];
        mma_prod<SPLIT>(rr, H[t][0], H[t][1], H[t][2], H[t][3], d.ih, d.il);  // rows (block, v = g), columns x
        mma_prod_t<SPLIT>(H[t], rr, d.ih, d.il);                             // rows (block, x = g), columns y
    };
    auto add = [&](int o, float p0, float p1) {
        atomicAdd(num + o, kw0 * p0);
        atomicAdd(num + o + P, kw1 * p1);
    };
    auto segment = [&](int t0, int n) {
#pragma unroll
        for (int t = t0; t < t0 + n; ++t) inverse(t);
#pragma unroll
        for (int t = t0; t < t0 + n; t += 2) {
            const int4 o = *reinterpret_cast<const int4*>(off + 2 * t);
            add(o.x, H[t][0], H[t][1]);
            add(o.y, H[t][2], H[t][3]);
            add(o.z, H[t + 1][0], H[t + 1][1]);
            add(o.w, H[t + 1][2], H[t + 1][3]);
        }
    };
    if (N > 2) {
        segment(0, 2);
    } else {
        inverse(0);
        add(off[0], H[0][0], H[0][1]);
        if (N > 1) add(off[1], H[0][2], H[0][3]);
    }
    if (N > 4) segment(2, 2);
    if (N > 8) segment(4, 4);
}

__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

constexpr int kTcWarps = 8;

// One launch per stage covers every tile: footprints of neighbouring tiles
// overlap, and the flush adds into the frame accumulators with global
// reductions.  The footprint planes use a row pitch P = 4 mod 32 (>= the
// footprint edge), which makes the column loads of the forward transform and
// the numerator atomics fall in 32 different banks.  Aggregation inside a tile:
//   numerator    added from the inverse transform's accumulators: a lane holds
//                two rows of one column, so each shared-memory atomic
//                instruction covers 32 distinct pixels of one block in 32 banks
//                (a staging buffer in between cost 48 shared accesses a group
//                and channel);
//   denominator  sum over placements of weight x Kaiser(pixel - origin): the
//                weights are added at the block origins (a weight map, one
//                atomic per block), and the separable Kaiser window is applied
//                to that map at the flush, four columns to a thread.
// Bound by issue (the split products' MMAs and splits, a Haar tree, the
// atomics), so what is not arithmetic counts: block offsets are read four at a
// time, nothing is staged, the pairs of a segment overlap, and stage 1 keeps two
// planes (64 registers: four CTAs an SM; stage 2 three).  12 MP chain frame, split
// products: stage 1 11.3 -> 8.4 ms, stage 2 15.5 -> 12.5 ms against a form with a
// staging buffer, an offset load and a branch per pair.  (The
// products are not merged into MMAs of k = 16: another order of the sums moves
// coefficients across the threshold.)
// ROWS: the flush adds whole rows (below).
template <int STAGE, bool SPLIT, bool ROWS>
__device__ __forceinline__ void filter_tc_tile(const FilterArgs& a, int tx, int ty, int c, int img) {
    extern __shared__ __align__(16) float sm[];
    const int row0 = img * a.h;
    const int i0 = tx * kRefTile, j0 = ty * kRefTile;
    const int i1 = min(i0 + kRefTile, a.nrx), j1 = min(j0 + kRefTile, a.nry);
    const int fx0 = max(0, refpos(i0, a.w, a.nstep) - a.R);
    const int fx1 = min(a.w, refpos(i1 - 1, a.w, a.nstep) + a.R + 8);
    const int fy0 = row0 + max(0, refpos(j0, a.h, a.nstep) - a.R);
    const int fy1 = row0 + min(a.h, refpos(j1 - 1, a.h, a.nstep) + a.R + 8);
    const int fw = fx1 - fx0, fh = fy1 - fy0;
    const int P = a.np, FP = a.fw * P;  // planes [a.fw rows][P]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* s_num = sm;
    float* s_img = sm + FP;                             // after the groups: the weight map, then den
    float* s_bas = s_img + FP;                          // stage 2: the basic estimate's footprint
    float* s_wgt = s_img + (STAGE == 2 ? 2 : 1) * FP;   // one aggregation weight per reference block of the tile
    uint32_t* s_list = reinterpret_cast<uint32_t*>((reinterpret_cast<uintptr_t>(s_wgt + kRefTile * kRefTile) + 15) &
                                                   ~(uintptr_t)15);
    uint32_t* s_cnt = s_list + kRefTile * kRefTile * 16;
    int* s_off = reinterpret_cast<int*>(s_cnt + kRefTile * kRefTile);  // [warp][16] block offsets of the group
    const float* gz = a.noisy + (long long)c * a.npx;
    const float* gb = STAGE == 2 ? a.basic + (long long)c * a.npx : nullptr;
    for (int yy = warp; yy < fh; yy += kTcWarps) {
        const long long o = (long long)(fy0 + yy) * a.w + fx0;
        for (int xx = lane; xx < fw; xx += 32) {
            cp_async4(s_img + yy * P + xx, gz + o + xx);
            if (STAGE == 2) cp_async4(s_bas + yy * P + xx, gb + o + xx);
        }
    }
    const int nti = i1 - i0, nref = nti * (j1 - j0);
    for (int i = threadIdx.x; i < nref * 4; i += blockDim.x) {
        const int k = i >> 2;
        const long long ref = ((long long)img * a.nry + j0 + k / nti) * a.nrx + i0 + k % nti;
        cp_async16(s_list + 4 * i, a.list + ref * 16 + 4 * (i & 3));
    }
    if (threadIdx.x < nref) {
        const int k = threadIdx.x;
        s_cnt[k] = a.cnt[((long long)img * a.nry + j0 + k / nti) * a.nrx + i0 + k % nti];
    }
    const float4 zero4 = make_float4(0.0F, 0.0F, 0.0F, 0.0F);
    for (int idx = threadIdx.x; idx < FP / 4; idx += blockDim.x) reinterpret_cast<float4*>(s_num)[idx] = zero4;
    cp_async_wait_all();
    __syncthreads();

    const int g = lane >> 2, q = lane & 3;
    const DctFrags dct = dct_frags(g, q);
    // hard thresholds of the unnormalised coefficients: lambda sigma 2^(k/2)
    const float thr1 = a.thr * 1.41421356237309515F, thr2 = a.thr * 2.0F, thr3 = a.thr * 2.82842712474619030F,
                thr4 = a.thr * 4.0F;
    // the window at the lane's two pixels of a block, (x, y) = (g, 2q) and (g, 2q + 1)
    const float kq0 = a.kaiser[2 * q * 8 + g], kq1 = a.kaiser[(2 * q + 1) * 8 + g];
    for (int k = warp; k < nref; k += kTcWarps) {
        const int cnt = (int)s_cnt[k];
        const int N = cnt >= 16 ? 16 : cnt >= 8 ? 8 : cnt >= 4 ? 4 : cnt >= 2 ? 2 : 1;
        const uint32_t* lst = s_list + k * 16;
        int* woff = s_off + warp * 16;
        __syncwarp();
        if (lane < 16) {
            const uint32_t p = lst[lane < N ? lane : 0];
            woff[lane] = ((int)(p >> 16) - fy0) * P + (int)(p & 0xFFFFU) - fx0;
        }
        __syncwarp();
        float H[8][4];
        tc_forward<SPLIT>(s_img, P, woff, N, dct, H);
        const int L = 31 - __clz(N);
        float wgt;
        if (STAGE == 1) {
            const float th0 = L == 0 ? a.thr : L == 1 ? thr1 : L == 2 ? thr2 : L == 3 ? thr3 : thr4;
            const float sc0 = exp2i(-L);
            unsigned kept = 0;
#pragma unroll
            for (int t = 0; t < 8; ++t)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int b = 2 * t + (e >> 1), kb = haar_k(b);
                    const float th = b == 0 ? th0 : kb == 1 ? thr1 : kb == 2 ? thr2 : kb == 3 ? thr3 : thr4;
                    const float sc = b == 0 ? sc0 : (kb == 1 ? 0.5F : kb == 2 ? 0.25F : kb == 3 ? 0.125F : 0.0625F);
                    const bool keep = fabsf(H[t][e]) > th;
                    H[t][e] = keep ? H[t][e] * sc : 0.0F;
                    kept += keep ? 1U : 0U;
                }
            kept = __reduce_add_sync(0xFFFFFFFFU, kept);
            wgt = kept > 0U ? 1.0F / (float)kept : a.sigma2;
        } else {
            float B[8][4];
            tc_forward<SPLIT>(s_bas, P, woff, N, dct, B);
            const float s0 = a.sigma2 * exp2i(L), sc0 = exp2i(-L);
            float sw2 = 0.0F;
#pragma unroll
            for (int t = 0; t < 8; ++t)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int b = 2 * t + (e >> 1), kb = haar_k(b);
                    const float sk = b == 0 ? s0 : a.sigma2 * (float)(1 << kb);
                    const float sc = b == 0 ? sc0 : (kb == 1 ? 0.5F : kb == 2 ? 0.25F : kb == 3 ? 0.125F : 0.0625F);
                    const float b2 = B[t][e] * B[t][e];
                    const float W = __fdividef(b2, b2 + sk);
                    H[t][e] = (H[t][e] * W) * sc;
                    sw2 = __fmaf_rn(W, W, sw2);
                }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) sw2 += __shfl_xor_sync(0xFFFFFFFFU, sw2, off);
            wgt = sw2 > 0.0F ? 1.0F / fmaxf(sw2, kMinWienerEnergy) : a.sigma2;
        }
        if (lane == 0) s_wgt[k] = wgt;
        tc_inverse_add<SPLIT>(H, N, dct, wgt * kq0, wgt * kq1, s_num, P, woff);
    }
    __syncthreads();
    // weight map at the block origins (in the footprint's own plane, now free)
    float* s_w = s_img;
    for (int idx = threadIdx.x; idx < FP / 4; idx += blockDim.x) reinterpret_cast<float4*>(s_w)[idx] = zero4;
    __syncthreads();
    for (int i = threadIdx.x; i < nref * 16; i += blockDim.x) {
        const int k = i >> 4, cnt = (int)s_cnt[k];
        const int N = cnt >= 16 ? 16 : cnt >= 8 ? 8 : cnt >= 4 ? 4 : cnt >= 2 ? 2 : 1;
        if ((i & 15) < N) {
            const uint32_t p = s_list[i];
            atomicAdd(s_w + ((int)(p >> 16) - fy0) * P + (int)(p & 0xFFFFU) - fx0, s_wgt[k]);
        }
    }
    __syncthreads();
    // den = map correlated with the Kaiser window (from the kernel arguments), in
    // place: rows, a band at a time, then columns, four columns to a thread (16-byte
    // loads); down the columns a thread keeps the last eight rows in registers.
    // With ROWS the frame's sums take whole rows after that: four columns to a
    // thread there, every lane in another sector, made a small window's stage a
    // tenth slower (2016 x 1512, 1 x 1 window at step 3: 1210 -> 1077 us; 12 MP
    // default 1 %).  The gated kernels add at once: with rows a 12 MP frame that
    // falls back took 34.77 ms against 34.38.
    const int gx = (fw + 3) / 4, segs = blockDim.x / gx;
    const int seg = threadIdx.x / gx, xx = 4 * (threadIdx.x - seg * gx);
    for (int b0 = 0; b0 < fh; b0 += segs) {
        float4* wr = reinterpret_cast<float4*>(s_w + (b0 + seg) * P + xx);
        const bool on = seg < segs && b0 + seg < fh;
        float h[4] = {0.0F, 0.0F, 0.0F, 0.0F};
        if (on) {
            const float4 w0 = xx >= 8 ? wr[-2] : zero4, w1 = xx >= 4 ? wr[-1] : zero4, w2 = wr[0];
            const float w[12] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w, w2.x, w2.y, w2.z, w2.w};
#pragma unroll
            for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int k = 0; k < 4; ++k) h[k] = __fmaf_rn(a.kaiser1[u], w[8 + k - u], h[k]);
        }
        __syncthreads();  // the band is read
        if (on) *wr = make_float4(h[0], h[1], h[2], h[3]);
    }
    __syncthreads();
    float* gn = a.acc + (long long)c * a.npx;
    float* gd = a.acc + (long long)(3 + c) * a.npx;
    const int seg_rows = (fh + segs - 1) / segs;
    const int y0 = seg * seg_rows, y1 = seg < segs ? min(fh, y0 + seg_rows) : 0;
    float4 r[8];  // r[v]: the row v above
#pragma unroll
    for (int v = 1; v < 8; ++v)
        r[v] = y0 < y1 && y0 - v >= 0 ? *reinterpret_cast<const float4*>(s_w + (y0 - v) * P + xx) : zero4;
    if (ROWS) __syncthreads();  // the rows above are read: den takes its place in the map
    for (int yy = y0; yy < y1; ++yy) {
        float4* row = reinterpret_cast<float4*>(s_w + yy * P + xx);
        r[0] = *row;
        float4 d = zero4;
#pragma unroll
        for (int v = 0; v < 8; ++v) {
            d.x = __fmaf_rn(a.kaiser1[v], r[v].x, d.x);
            d.y = __fmaf_rn(a.kaiser1[v], r[v].y, d.y);
            d.z = __fmaf_rn(a.kaiser1[v], r[v].z, d.z);
            d.w = __fmaf_rn(a.kaiser1[v], r[v].w, d.w);
        }
#pragma unroll
        for (int v = 7; v > 0; --v) r[v] = r[v - 1];
        if constexpr (ROWS) {
            *row = d;
        } else {
            const float4 n = *reinterpret_cast<const float4*>(s_num + yy * P + xx);
            const long long o = (long long)(fy0 + yy) * a.w + fx0 + xx;
            const float nv[4] = {n.x, n.y, n.z, n.w}, dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (xx + k < fw && dv[k] > 0.0F) {
                    atomicAdd(gn + o + k, nv[k]);
                    atomicAdd(gd + o + k, dv[k]);
                }
        }
    }
    if constexpr (!ROWS) return;
    __syncthreads();
    for (int yy = warp; yy < fh; yy += kTcWarps) {
        const long long o = (long long)(fy0 + yy) * a.w + fx0;
        for (int x = lane; x < fw; x += 32) {
            const float d = s_w[yy * P + x];
            if (d > 0.0F) {
                atomicAdd(gn + o + x, s_num[yy * P + x]);
                atomicAdd(gd + o + x, d);
            }
        }
    }
}

template <int STAGE, bool SPLIT>
__global__ void __launch_bounds__(32 * kTcWarps, STAGE == 1 ? 4 : 3) bm3d_filter_tc_kernel(const __grid_constant__ FilterArgs a) {
    filter_tc_tile<STAGE, SPLIT, true>(a, blockIdx.x, blockIdx.y, blockIdx.z % 3, blockIdx.z / 3);
}
// A gated run seldom happens: a grid of resident CTAs that walk the tiles, so
// that one which does not costs the launch (3 us) and not the start of every
// tile's CTA (46 us a stage at 12 MP).
template <int STAGE, bool SPLIT>
__global__ void __launch_bounds__(32 * kTcWarps, STAGE == 1 ? 4 : 3) bm3d_filter_tc_gated_kernel(const __grid_constant__ FilterArgs a,
                                                                               int tiles) {
    if (gated_off(a.gate)) return;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int z = t / (a.ntx * a.nty), r = t - z * (a.ntx * a.nty);
        filter_tc_tile<STAGE, SPLIT, false>(a, r % a.ntx, r / a.ntx, z % 3, z / 3);
        __syncthreads();
    }
}

// --------------------------------------------------------- basic / final
__global__ void bm3d_basic_kernel(const float* __restrict__ acc, float* __restrict__ basic, uint8_t* __restrict__ q,
                                  long long npx, const int* gate) {
    if (gated_off(gate)) return;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < npx; i += (long long)gridDim.x * blockDim.x) {
        float y = 0.0F;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float v = acc[c * npx + i] / acc[(3 + c) * npx + i];
            basic[c * npx + i] = v;
            if (c == 0) y = v;
        }
        q[i] = quantise(y * kInvS3);
    }
}

template <class T>
__global__ void bm3d_final_kernel(const float* __restrict__ acc, Img in, Img out, long long npx, const int* gate) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= in.w || gated_off(gate)) return;
    for (int y = blockIdx.y; y < in.h; y += gridDim.y) {
        const long long i = (long long)y * in.w + x;
        const float Y = acc[i] / acc[3 * npx + i];
        const float U = acc[npx + i] / acc[4 * npx + i];
        const float V = acc[2 * npx + i] / acc[5 * npx + i];
        const float yy = Y * kInvS3, uu = U * kInvS2, vv = V * kInvS6;
        const Rgba o{(yy + uu) + vv, yy - 2.0F * vv, (yy - uu) + vv, 0.0F};
        store_rgb_keep_alpha(px<T>(out, x, y), o, px<const T>(in, x, y));
    }
}

__global__ void bm3d_zero_kernel(float* __restrict__ p, long long n, const int* gate) {
    if (gated_off(gate)) return;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        p[i] = 0.0F;
}

double bessel_i0(double x) {
    double sum = 1.0, term = 1.0;
    const double hx = 0.5 * x;
    for (int k = 1; k < 64; ++k) {
        term *= (hx / k) * (hx / k);
        sum += term;
        if (term < 1e-18 * sum) break;
    }
    return sum;
}

int ref_count(int n, int nstep) {
    if (n < 8) return 0;
    int m = (n - 8) / nstep + 1;
    if ((n - 8) % nstep) ++m;
    return m;
}

size_t align256(size_t v) { return (v + 255U) & ~(size_t)255U; }

size_t filter_smem(const Bm3dPlan& p, int stage) {
    return sizeof(float) * ((size_t)(stage == 2 ? 4 : 3) * p.fw * p.fw + (size_t)kFilterWarps * kWarpBuf + 64);
}
// The match kernel's region for `tile` x `tile` references: its edge, the word
// pitches (rows 4 mod 8, copies 8 mod 32, with a spare row and the columns a
// last tile of eight may reach over), the energies' pitch, and the bytes.
size_t match_layout(Bm3dPlan& p, int tile) {
    p.mtile = tile;
    p.mwin = (tile - 1) * p.nstep + 2 * p.R + 8;
    const int wpr = (p.mwin + 11) / 4 + 1;
    p.mwpr = wpr + ((4 - wpr) % 8 + 8) % 8;
    const int plane = (p.mwin + 1) * p.mwpr;
    p.mplane = plane + ((8 - plane) % 32 + 32) % 32;
    p.mepitch = (p.mwin + 2) & ~1;
    return sizeof(uint32_t) *
           (4 * (size_t)p.mplane + (size_t)p.mepitch * (p.mwin - 7) + (size_t)(tile * tile) * kMatchStride);
}
// The same of the form with a thread per reference.
size_t match_each_layout(Bm3dPlan& p) {
    p.mtile = kMatchEachTile;
    p.mwin = (kMatchEachTile - 1) * p.nstep + 2 * p.R + 8;
    p.mwpr = (p.mwin + 3) / 4 + 1;
    p.mplane = p.mwin * p.mwpr;
    p.mepitch = 0;
    return sizeof(uint32_t) * 4 * (size_t)p.mplane;
}
// The smallest window that the matching on the tensor cores takes.  Its warps
// share the union of 8 x 4 references' windows, so small windows and large steps
// waste its products, and a thread per reference is faster; with CTAs for less
// than a quarter of the SMs that thread's serial walk counts instead.  Stage 1
// with either form (us; 320 x 240 has few, 2016 x 1512 many):
//   window, step           9, 3   21, 3  27, 3  33, 4  39, 4  39, 6  45, 6  39, 8
//   few:  tensor cores     162    207    223    257    281    314    330    338
//         thread           112    180    233    286    350    347    422    351
//   many: tensor cores     2542   2840   2930   2292   2557   1500   1682   1417
//         thread           2282   2688   2942   2029   2372   1301   1648   1023
// (Where the two are close on large frames the line keeps to the tensor cores.)
int match_from(const Bm3dPlan& p) {
    constexpr int few[8] = {21, 27, 27, 33, 33, 33, 39, 39}, many[8] = {21, 27, 27, 39, 39, 39, 47, 47};
    const int ctas = ((p.nrx + kMatchEachTile - 1) / kMatchEachTile) * ((p.nry + kMatchEachTile - 1) / kMatchEachTile);
    return (ctas * p.batch < kSmCount / 4 ? few : many)[p.nstep - 1];
}
// Row pitch of the tensor-core form's footprint planes: at least fw and 4 mod
// 32 (column loads of eight columns x two rows, and atomics of eight rows x
// four columns, fall in 32 different banks).
int tile_pitch(int fw) { return fw + ((4 - fw) % 32 + 32) % 32; }
size_t filter_tc_smem(const Bm3dPlan& p, int stage) {
    const size_t fp = (size_t)p.fw * tile_pitch(p.fw);
    const size_t floats = (stage == 2 ? 3 : 2) * fp + kRefTile * kRefTile;  // numerator, footprints, weights
    return sizeof(float) * floats + 16 + sizeof(uint32_t) * kRefTile * kRefTile * 17 + sizeof(int) * kTcWarps * 16;
}

}  // namespace

int bm3d_plan(const cpipe_Bm3dSpecParams* p, int w, int h, Bm3dPlan* out, int batch) {
    if (p == nullptr || out == nullptr) return CPIPE_BAD_INDEX;
    const int n2 = p->n2;
    if (!(n2 == 1 || n2 == 2 || n2 == 4 || n2 == 8 || n2 == 16)) return CPIPE_BAD_INDEX;
    if (p->ns < 1 || p->ns > 45 || (p->ns & 1) == 0) return CPIPE_BAD_INDEX;
    if (p->nstep < 1 || p->nstep > 8) return CPIPE_BAD_INDEX;
    if (!(p->tau_match1 >= 0.0F && p->tau_match1 <= 16000.0F)) return CPIPE_BAD_INDEX;
    if (!(p->tau_match2 >= 0.0F && p->tau_match2 <= 16000.0F)) return CPIPE_BAD_INDEX;
    if (p->stages != 1 && p->stages != 2) return CPIPE_BAD_INDEX;
    if (!(p->lambda3d >= 0.0F) || !(p->kaiser_beta >= 0.0F)) return CPIPE_BAD_INDEX;
    if (p->transform < 0 || p->transform > 2) return CPIPE_BAD_INDEX;
    if (w <= 0 || h <= 0 || batch < 1 || w > 65535 || (long long)h * batch > 65535) return CPIPE_BAD_INDEX;
    Bm3dPlan& q = *out;
    q = Bm3dPlan{};
    q.w = w;
    q.h = h;
    q.batch = batch;
    q.ns = p->ns;
    q.R = (p->ns - 1) / 2;
    q.n2 = n2;
    q.nstep = p->nstep;
    q.stages = p->stages;
    q.tensor = p->transform != 1;
    q.split = p->transform == 0;
    q.sigma = p->sigma;
    q.sigma2 = p->sigma * p->sigma;
    q.thr = p->lambda3d * p->sigma;
    q.dthr[0] = (uint32_t)floor(64.0 * (double)p->tau_match1);
    q.dthr[1] = (uint32_t)floor(64.0 * (double)p->tau_match2);
    q.copy = w < 8 || h < 8 || !(p->sigma > 0.0F) || !(q.sigma2 > 0.0F);
    if (q.copy) return CPIPE_OK;
    double k1[8];
    const double i0b = bessel_i0(p->kaiser_beta);
    for (int n = 0; n < 8; ++n) {
        const double t = (2.0 * n - 7.0) / 7.0;
        k1[n] = bessel_i0(p->kaiser_beta * sqrt(1.0 - t * t)) / i0b;
    }
    for (int v = 0; v < 8; ++v)
        for (int u = 0; u < 8; ++u) q.kaiser[v * 8 + u] = (float)(k1[v] * k1[u]);
    for (int n = 0; n < 8; ++n) q.kaiser1[n] = (float)k1[n];
    q.nrx = ref_count(w, q.nstep);
    q.nry = ref_count(h, q.nstep);
    q.fw = (kRefTile - 1) * q.nstep + 2 * q.R + 8;
    const int span = kRefTile * q.nstep;
    q.phases = (span + 2 * q.R + 8 + span - 1) / span;
    q.ntx = (q.nrx + kRefTile - 1) / kRefTile;
    q.nty = (q.nry + kRefTile - 1) / kRefTile;
    // 16 x 16 references a CTA share a region best; the largest windows and steps need 8 x 8
    q.match_each = n2 == 1 || q.ns < match_from(q);  // (n2 = 1: nothing to search)
    if (q.match_each) q.match_bytes = match_each_layout(q);
    else q.match_bytes = match_layout(q, 16);
    if (!q.match_each && q.match_bytes > 227 * 1024) q.match_bytes = match_layout(q, 8);
    const size_t npx = (size_t)w * h * batch, nref = (size_t)q.nrx * q.nry * batch;
    size_t o = 0;
    q.off_yuv = o;
    o = align256(o + 3 * npx * sizeof(float));
    q.off_basic = o;
    if (q.stages == 2) o = align256(o + 3 * npx * sizeof(float));
    q.off_acc = o;
    o = align256(o + 6 * npx * sizeof(float));
    q.off_q = o;
    o = align256(o + npx);
    q.off_list = o;
    o = align256(o + nref * 16 * sizeof(uint32_t));
    q.off_cnt = o;
    o = align256(o + nref);
    q.bytes = o;
    return CPIPE_OK;
}

cudaError_t bm3d_setup(const Bm3dPlan& p) {
    if (p.copy) return cudaSuccess;
    constexpr size_t kSmemOptIn = 227 * 1024;
    if (p.match_bytes > kSmemOptIn || filter_smem(p, 2) > kSmemOptIn) return cudaErrorInvalidConfiguration;
    if (p.tensor && filter_tc_smem(p, 2) > kSmemOptIn) return cudaErrorInvalidConfiguration;
    // The limit is a state of the kernel on the device, not of the plan: it is always
    // the most that any plan may take, so that plans and threads agree on it.
    static const void* const kernels[] = {
        (const void*)bm3d_match_kernel, (const void*)bm3d_match_each_kernel, (const void*)bm3d_filter_kernel<1>, (const void*)bm3d_filter_kernel<2>,
        (const void*)bm3d_filter_tc_kernel<1, true>, (const void*)bm3d_filter_tc_kernel<1, false>,
        (const void*)bm3d_filter_tc_kernel<2, true>, (const void*)bm3d_filter_tc_kernel<2, false>,
        (const void*)bm3d_filter_tc_gated_kernel<1, true>, (const void*)bm3d_filter_tc_gated_kernel<1, false>,
        (const void*)bm3d_filter_tc_gated_kernel<2, true>, (const void*)bm3d_filter_tc_gated_kernel<2, false>};
    for (const void* k : kernels)
        if (const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemOptIn);
            e != cudaSuccess)
            return e;
    return cudaSuccess;
}

cudaError_t bm3d_run(const Bm3dPlan& p, const Img& in, const Img& out, bool f16, void* scratch, cudaStream_t st,
                     bool setup, const int* gate) {
    if (p.copy && gate) return cudaSuccess;  // a gated run leaves the output alone
    if (p.copy) {
        const int elem = f16 ? 2 : 4;
        return launch_copy(in.data, in.row_stride * elem, out.data, out.row_stride * elem, (long long)in.w * 4 * elem,
                           in.h, st);
    }
    char* base = static_cast<char*>(scratch);
    float* yuv = reinterpret_cast<float*>(base + p.off_yuv);
    float* basic = reinterpret_cast<float*>(base + p.off_basic);
    float* acc = reinterpret_cast<float*>(base + p.off_acc);
    uint8_t* q = reinterpret_cast<uint8_t*>(base + p.off_q);
    uint32_t* list = reinterpret_cast<uint32_t*>(base + p.off_list);
    uint8_t* cnt = reinterpret_cast<uint8_t*>(base + p.off_cnt);
    const long long npx = (long long)p.w * p.h * p.batch;
    cudaError_t e;
    if (setup && (e = bm3d_setup(p)) != cudaSuccess) return e;
    const size_t fs1 = filter_smem(p, 1), fs2 = filter_smem(p, 2);
    const size_t ts1 = filter_tc_smem(p, 1), ts2 = filter_tc_smem(p, 2);

    // a gated run's kernels walk the frame with few CTAs: it seldom happens, and
    // should not cost the start of a CTA for every row when it does not
    const int prows = gate ? std::min(p.h * p.batch, std::max(1, 8 * kSmCount / ((p.w + 255) / 256))) : p.h * p.batch;
    const dim3 pgrid((p.w + 255) / 256, prows);
    const unsigned bgrid = (unsigned)(gate ? std::min((npx + 255) / 256, (long long)kSmCount * 8) : (npx + 255) / 256);
    if (f16) bm3d_prep_kernel<__half><<<pgrid, 256, 0, st>>>(in, yuv, q, npx, gate);
    else bm3d_prep_kernel<float><<<pgrid, 256, 0, st>>>(in, yuv, q, npx, gate);

    MatchArgs ma{p.w,    p.h,      p.nrx,     p.nry, p.nstep, p.R, p.ns, p.n2, p.mtile,
                 p.mwpr, p.mplane, p.mepitch, p.dthr[0], q, list, cnt, gate};
    const dim3 mgrid((p.nrx + p.mtile - 1) / p.mtile, (p.nry + p.mtile - 1) / p.mtile, p.batch);
    FilterArgs fa{};
    fa.w = p.w;
    fa.h = p.h;
    fa.nrx = p.nrx;
    fa.nry = p.nry;
    fa.nstep = p.nstep;
    fa.R = p.R;
    fa.ntx = p.ntx;
    fa.nty = p.nty;
    fa.phases = p.phases;
    fa.fw = p.fw;
    fa.sigma2 = p.sigma2;
    fa.thr = p.thr;
    fa.npx = npx;
    fa.list = list;
    fa.cnt = cnt;
    fa.noisy = yuv;
    fa.basic = basic;
    fa.acc = acc;
    fa.gate = gate;
    for (int i = 0; i < 64; ++i) fa.kaiser[i] = p.kaiser[i];
    for (int i = 0; i < 8; ++i) fa.kaiser1[i] = p.kaiser1[i];
    fa.np = tile_pitch(p.fw);
    FilterArgs ta = fa;  // tensor-core form: one launch over all tiles (global reductions at the flush)
    ta.phases = 1;
    const dim3 tgrid(p.ntx, p.nty, 3 * p.batch);
    const dim3 fgrid((p.ntx + p.phases - 1) / p.phases, (p.nty + p.phases - 1) / p.phases, 3 * p.batch);

    for (int stage = 1; stage <= p.stages; ++stage) {
        bm3d_zero_kernel<<<kSmCount * 8, 256, 0, st>>>(acc, 6 * npx, gate);
        ma.dthr = p.dthr[stage - 1];
        if (p.match_each) bm3d_match_each_kernel<<<mgrid, p.mtile * p.mtile, p.match_bytes, st>>>(ma);
        else bm3d_match_kernel<<<mgrid, p.mtile * p.mtile, p.match_bytes, st>>>(ma);
        if (p.tensor && gate) {
            const int tiles = p.ntx * p.nty * 3 * p.batch, g = std::min(tiles, kSmCount * (stage == 1 ? 4 : 3));
            if (p.split) {
                if (stage == 1) bm3d_filter_tc_gated_kernel<1, true><<<g, 32 * kTcWarps, ts1, st>>>(ta, tiles);
                else bm3d_filter_tc_gated_kernel<2, true><<<g, 32 * kTcWarps, ts2, st>>>(ta, tiles);
            } else {
                if (stage == 1) bm3d_filter_tc_gated_kernel<1, false><<<g, 32 * kTcWarps, ts1, st>>>(ta, tiles);
                else bm3d_filter_tc_gated_kernel<2, false><<<g, 32 * kTcWarps, ts2, st>>>(ta, tiles);
            }
        } else if (p.tensor) {
            if (p.split) {
                if (stage == 1) bm3d_filter_tc_kernel<1, true><<<tgrid, 32 * kTcWarps, ts1, st>>>(ta);
                else bm3d_filter_tc_kernel<2, true><<<tgrid, 32 * kTcWarps, ts2, st>>>(ta);
            } else {
                if (stage == 1) bm3d_filter_tc_kernel<1, false><<<tgrid, 32 * kTcWarps, ts1, st>>>(ta);
                else bm3d_filter_tc_kernel<2, false><<<tgrid, 32 * kTcWarps, ts2, st>>>(ta);
            }
        } else {
            for (int py = 0; py < p.phases; ++py)
                for (int pxh = 0; pxh < p.phases; ++pxh) {
                    if (stage == 1) bm3d_filter_kernel<1><<<fgrid, 32 * kFilterWarps, fs1, st>>>(fa, pxh, py);
                    else bm3d_filter_kernel<2><<<fgrid, 32 * kFilterWarps, fs2, st>>>(fa, pxh, py);
                }
        }
        if (stage == 1 && p.stages == 2)
            bm3d_basic_kernel<<<bgrid, 256, 0, st>>>(acc, basic, q, npx, gate);
    }
    if (f16) bm3d_final_kernel<__half><<<pgrid, 256, 0, st>>>(acc, in, out, npx, gate);
    else bm3d_final_kernel<float><<<pgrid, 256, 0, st>>>(acc, in, out, npx, gate);
    return cudaGetLastError();
}

}  // namespace cpb
