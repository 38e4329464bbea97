// kernels.cu — sm_103a kernels of the GB300 feature front-end.
//
//   k_pyramid       every pyramid level as f32 rows of 16-byte pitch (level 0 =
//                   u8 / 255, levels >= 1 one bilinear tap of LOD0): the
//                   source of k_detect's tile loads
//   k_detect   (K1) TMA-staged level tile + halo, FAST response + cull (or, in
//                   the cfg profile, FAST 9-of-16 at 20/255 + 3x3 NMS)
//   k_band_count, k_band_write
//                   ordered keypoint compaction over 32-row bands, cap; the
//                   list of blur tiles that the kept keypoints' tests read
//   k_blur          blur cache of the listed tiles, inside the level and
//                   beyond its edges (BRIEF points outside)
//   k_xsort         the matcher's lists: per horizontal band an x-sorted
//                   candidate list, and the band-grouped query order
//   k_describe (K2) orientation (one lane per keypoint of a warp's group) +
//                   256-bit rotated BRIEF (the warp's lanes take 8 tests each)
//   k_bacc_init     empties the accumulators before a k_match (the caller-
//                   owned and served forms, and batches of very large caps; others
//                   reset all of theirs by a memset)
//   k_match    (K3) windowed top-2 Hamming search of both directions, one
//                   distance per pair; a warp claims units: 32 x-adjacent
//                   queries of the previous set in one band against a part of
//                   one pool level
//   k_mutual        mutual cross-check (searches read from their accumulators)
//                   and ordered match output
//   k_bruteforce    brute-force top-2 matching (no window, no cross-check) on
//                   the integer pipes; the tensor-core form is k_bf_mma
//                   (bf_tc.cu)
//
// Arithmetic contract: binary32, round-to-nearest-even, no FMA contraction
// (the library is compiled with --fmad=false), evaluation order as in the
// reference shaders.  Every kernel is bit-exact against the CPU oracle.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/uslam_canon.h"
#include "bf_line.h"
#include "uslam_internal.h"

namespace uslam {

// K1 tile geometry: TW x TH output pixels (a template parameter pair, one of
// kTileShapes), halo HX columns / HY rows (HY_CFG with the cfg profile, whose
// 3x3 NMS needs the FAST score one pixel beyond the tile).
constexpr int HX = USLAM_TILE_HX;
constexpr int HY = USLAM_TILE_HY;
constexpr int HY_CFG = USLAM_TILE_HY_CFG;
constexpr int K1_THREADS = 256;
// Spin limit of a tile load's mbarrier wait (try_wait polls); past it the
// kernel records USLAM_ERR_TMA_TIMEOUT and leaves the tile.
constexpr uint32_t kTmaWaitLimit = 1u << 20;
// cfg detection profile threshold: 20 grey levels on the u8/255 scale.
constexpr float kCfgThreshold = 20.0f / 255.0f;

// Matcher band of a LOD-0 y in a frame of height H cut into n bands (rows
// [b H / n, (b + 1) H / n)).
__device__ __forceinline__ int match_band(float y, float H, int n) {
    const int b = (int)floorf(y * (float)n / H);
    return b < 0 ? 0 : (b >= n ? n - 1 : b);
}

// Bresenham circle of radius 3 (resources/detect_corners.wgsl:31-32) as
// compile-time constants: in the unrolled loops the shared-memory offsets fold
// into immediates.
__device__ __forceinline__ constexpr int circle_x(int i) {
    return i == 0 ? 0 : i == 1 ? 1 : i == 2 ? 2 : i <= 5 ? 3 : i == 6 ? 2 : i == 7 ? 1 : i == 8 ? 0
         : i == 9 ? -1 : i == 10 ? -2 : i <= 13 ? -3 : i == 14 ? -2 : -1;
}
// A quarter turn maps point i to point i + 4 ((x, y) -> (-y, x)), so y_i = -x_(i+4).
__device__ __forceinline__ constexpr int circle_y(int i) { return -circle_x((i + 4) & 15); }

// Tint robustness clamp of textureLoad coordinates: min(u32(c), n - 1).
__device__ __forceinline__ int tint_clamp(int c, int n) {
    const unsigned u = (unsigned)c;
    return u < (unsigned)n ? (int)u : n - 1;
}

// Clamp-to-edge index of an integer-valued float (may be huge or negative).
__device__ __forceinline__ int edge_index(float f, int n) {
    if (f <= 0.0f) return 0;
    if (f >= (float)(n - 1)) return n - 1;
    return (int)f;
}

// The top bit of each byte that is not 0.
__device__ __forceinline__ uint32_t nonzero_tops(uint32_t v) {
    return (((v & 0x7f7f7f7fu) + 0x7f7f7f7fu) | v) & 0x80808080u;
}
// Bit b of the result: byte b is not 0 (the product gathers the four bits, no
// two of its terms meet).
__device__ __forceinline__ uint32_t nonzero_mask(uint32_t v) { return ((nonzero_tops(v) >> 7) * 0x10204080u) >> 28; }
__device__ __forceinline__ uint32_t nonzero_mask16(const uint4& v) {
    return nonzero_mask(v.x) | nonzero_mask(v.y) << 4 | nonzero_mask(v.z) << 8 | nonzero_mask(v.w) << 12;
}
__device__ __forceinline__ uint32_t nonzero_bytes16(const uint4& v) {
    return (uint32_t)__popc(nonzero_tops(v.x) | nonzero_tops(v.y) >> 1 | nonzero_tops(v.z) >> 2 | nonzero_tops(v.w) >> 3);
}

__device__ __forceinline__ uint32_t warp_sum_u32(uint32_t v) { return __reduce_add_sync(0xffffffffu, v); }

// FAST response at smem cell (r, c): 1 + longest non-wrapping run of
// |centre - p_i| > 0.15, kept iff > 9 (detect_corners.wgsl:58-81).
template <int SW>
__device__ __forceinline__ uint32_t fast_response(const float (*sm)[SW], int r, int c) {
    const float center = sm[r][c];
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float p = sm[r + circle_y(i)][c + circle_x(i)];
        m |= (fabsf(center - p) > 0.15f ? 1u : 0u) << i;
    }
    // run >= 9 test: AND of the mask shifted by 0..8
    uint32_t t = m & (m >> 1);
    t &= t >> 2;
    t &= t >> 4;
    t &= t >> 1;
    // bit i of t starts a run of 9, so n + 1 adjacent bits of t are a run of 9 + n
    uint32_t run = t ? 9u : 0u;
    while (t) {
        t &= t << 1;
        ++run;
    }
    return run;
}

// Longest run of ones of a 16-bit circle mask, wrapping around (16 if all
// set), where it is at least 9; else 0.
__device__ __forceinline__ uint32_t circular_run9(uint32_t m) {
    if (m == 0xffffu) return 16u;
    const uint32_t x = m | (m << 16);
    uint32_t t = x & (x >> 1);
    t &= t >> 2;
    t &= t >> 4;
    t &= x >> 8;
    // bit i of t starts a run of 9, so n + 1 adjacent bits of t are a run of 9 + n
    uint32_t run = t ? 8u : 0u;
    while (t) {
        t &= t << 1;
        ++run;
    }
    return run;
}

// cfg profile corner test at smem cell (r, c): FAST 9-of-16 with wrap-around,
// brighter iff p - c > T, darker iff c - p > T (T = 20/255).  Returns the
// score (sum over i = 0..15 of (|p_i - c| - T) for the points of the
// qualifying polarity, added in index order) and the arc length (longest
// circular run, 9..16) in *arc; 0 and 0 if not a corner.
template <int SW>
__device__ __forceinline__ float cfg_corner(const float (*sm)[SW], int r, int c, uint32_t* arc) {
    const float center = sm[r][c];
    // d = p - c; brighter: the sign of T - d, darker (c - p = -d exactly): of
    // T + d, shifted in from point 15 down
    float d[16];
    uint32_t mb = 0, md = 0;
#pragma unroll
    for (int i = 15; i >= 0; --i) {
        d[i] = sm[r + circle_y(i)][c + circle_x(i)] - center;
        mb = __funnelshift_l(__float_as_uint(kCfgThreshold - d[i]), mb, 1);
        md = __funnelshift_l(__float_as_uint(kCfgThreshold + d[i]), md, 1);
    }
    const uint32_t rb = circular_run9(mb), rd = circular_run9(md);
    *arc = 0u;
    if ((rb | rd) == 0u) return 0.0f;
    const bool bright = rb >= 9u;
    const uint32_t m = bright ? mb : md;
    const float side = bright ? 1.0f : -1.0f;
    float score = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i)
        if ((m >> i) & 1u) score = score + __fmaf_rn(d[i], side, -kCfgThreshold);  // (+-d) - T, rounded once
    *arc = bright ? rb : rd;
    return score;
}

// Packed binary32 products (sm_100 family mul.f32x2): one instruction rounds
// each lane to nearest even exactly as the scalar mul.rn would, so two
// independent products cost one issue slot with unchanged bits.  Their sums
// are scalar here and take another form in k_blur (add2): ptxas (CUDA 13.0)
// contracts mul.rn.f32x2 feeding add.rn.f32x2 into one fused multiply-add (a
// single rounding) in spite of .rn and --fmad=false, while a packed product
// feeding a scalar add.rn is kept as two roundings.
__device__ __forceinline__ float2 mul2_rn(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 pa, pb, pd;\n\t"
        "mov.b64 pa, {%2, %3};\n\tmov.b64 pb, {%4, %5};\n\t"
        "mul.rn.f32x2 pd, pa, pb;\n\tmov.b64 {%0, %1}, pd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// f32(u8) / 255 of two bytes, correctly rounded: u hi + u lo in one fused step
// with hi + lo = 1/255 to 48 bits (multiplication by a constant held as two
// words, Brisebarre and Muller 2008); equal to the quotient for all 256 bytes.
// Five packed instructions (u is the byte as the low bits of 2^23 + u, less
// 2^23); a 256-entry shared table cost a load with bank conflicts each
// (k_pyramid on 32 frames of 752x480: 67 us with the table).
__device__ __forceinline__ float2 unit2_u8(uint32_t b0, uint32_t b1) {
    constexpr float hi = 1.0f / 255.0f, lo = (float)(1.0 / 255.0 - (double)hi);
    float2 d;
    asm("{\n\t.reg .b64 u, s, h, l, p;\n\t"
        "mov.b64 u, {%2, %3};\n\tmov.b64 s, {%4, %4};\n\tmov.b64 h, {%5, %5};\n\tmov.b64 l, {%6, %6};\n\t"
        "add.rn.f32x2 u, u, s;\n\tmul.rn.f32x2 p, u, l;\n\tfma.rn.f32x2 u, u, h, p;\n\tmov.b64 {%0, %1}, u;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(__uint_as_float(0x4B000000u | b0)), "f"(__uint_as_float(0x4B000000u | b1)), "f"(-8388608.0f), "f"(hi), "f"(lo));
    return d;
}

// ------------------------------------------------------ TMA + mbarrier ----
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    // make the initialised barrier visible to the async (TMA) proxy
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
// Bounded wait for phase `parity` of the barrier: true when it completed.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit) {
    const uint32_t a = smem_addr(bar);
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// 2D tiled TMA load of the map's box at element coordinates (x, y) into
// shared memory, completing on the barrier (x * 4 bytes is 16-byte aligned
// for every caller: x = tile origin - 8 or - 4, tile widths multiples of 32).
__device__ __forceinline__ void tma_load_2d(void* dst, const void* tmap, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
            "r"(smem_addr(dst)),
        "l"(tmap), "r"(x), "r"(y), "r"(smem_addr(bar))
        : "memory");
}

// ----------------------------------------------------------- pyramid ----
// Level l of one TW x TH tile into lvl[l] (row pitch lvl_pitch): l = 0 is
// f32(u8) / 255 (provider_base.cpp:121-124), read 8 pixels per 8-byte load
// and stored as two 16-byte vectors; l >= 1 is one canonical bilinear tap of
// LOD0 at the texel centre (create_pyramid.wgsl:11-12).  Sampling
// coordinates depend only on the row or only on the column, so they are
// computed once per tile row / column (the per-pixel operations, so the same
// bits).  The weights (na nb, a nb) and (na b, a b) are packed products and
// the sum is scalar in the written order.  Issue-bound (71 %): two columns a
// thread and packed conversions took four 3840x2160 frames from 162 to 141 us
// (366 MB, 2.6 TB/s).
template <int TW, int TH>
__global__ void __launch_bounds__(K1_THREADS)
k_pyramid(const FrameDev* __restrict__ frames, const TileItem* __restrict__ tiles, uint32_t* blur_count) {
    static_assert(K1_THREADS % TW == 0 && TW % 8 == 0, "tile shape");
    __shared__ int2 s_fx[TW];    // LOD0 source columns (x0, x1) per tile column
    __shared__ float2 s_fa[TW];  // (1 - a, a)
    __shared__ int2 s_fy[TH];    // offsets of the LOD0 source rows (y0, y1) per tile row
    __shared__ float2 s_fnb[TH], s_fb[TH];  // (1 - b, 1 - b), (b, b)
    const TileItem it = tiles[blockIdx.x];
    const FrameDev& F = frames[it.frame];
    const int l = it.level;
    const int w = F.w[l], h = F.h[l];
    const int X0 = it.tx * TW, Y0 = it.ty * TH;
    const int t = threadIdx.x;
    float* const out = F.lvl[l];
    const int lp = F.lvl_pitch[l];
    const uint8_t* img = F.img;
    const int pitch = F.img_pitch;
    // the run's counts and blur marks start empty: the first tile of a row
    // clears the bands it holds (a band is two rows of the 16-row shapes)
    if (it.tx == 0 && Y0 % 32 == 0) {
        const int nx = USLAM_BLUR_NX(w);
        uint32_t* f = F.btile[l];
        for (int band = Y0 / 32; band * 32 < min(Y0 + TH, h); ++band) {
            if (t < 2) F.bands[l][2 * band + t] = 0u;
            for (int i = t; i < nx; i += K1_THREADS) f[band * nx + i] = 0u;
            if (t == 0) f[USLAM_BLUR_AT_RIGHT(w, h) + band] = 0u;
        }
        if (Y0 == 0)
            for (int i = USLAM_BLUR_AT_BELOW(w, h) + t; i < USLAM_BLUR_TILES(w, h, F.margin); i += K1_THREADS) f[i] = 0u;
    }
    if (blockIdx.x == 0 && t < 2 && blur_count) blur_count[t] = 0u;
    if (l == 0) {
        // 8 pixels per thread (8-byte loads): a 64-wide tile of 32 rows is
        // 256 segments, one per thread.  16-byte loads left half the threads
        // without a segment and measured slower (0.151 against 0.144 ms on 64
        // frames of 752x480).
        constexpr int SEGS = TW / 8;
        for (int u = t; u < SEGS * TH; u += K1_THREADS) {
            const int r = u / SEGS;
            const int x = X0 + (u - r * SEGS) * 8, y = Y0 + r;
            if (y >= h || x >= w) continue;
            // x is a multiple of 8 below w, so x + 8 <= the 16-byte image pitch
            const uint2 q = *reinterpret_cast<const uint2*>(img + (size_t)y * pitch + x);
            float v[8];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 u2 = unit2_u8((q.x >> (8 * k)) & 255u, (q.y >> (8 * k)) & 255u);
                v[k] = u2.x;
                v[4 + k] = u2.y;
            }
            float* o = out + (size_t)y * lp + x;
            if (x + 8 <= lp) {
                reinterpret_cast<float4*>(o)[0] = make_float4(v[0], v[1], v[2], v[3]);
                reinterpret_cast<float4*>(o)[1] = make_float4(v[4], v[5], v[6], v[7]);
            } else {
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (x + k < w) o[k] = v[k];
            }
        }
        return;
    }
    for (int i = t; i < TW + TH; i += K1_THREADS) {
        if (i < TW) {
            const int gx = min(X0 + i, w - 1);
            const float u = (((float)gx + 0.5f) / (float)w) * (float)F.W0 - 0.5f;
            const float fi = floorf(u);
            const float a = u - fi;
            s_fa[i] = make_float2(1.0f - a, a);
            s_fx[i] = make_int2(edge_index(fi, F.W0), edge_index(fi + 1.0f, F.W0));
        } else {
            const int r = i - TW;
            const int gy = min(Y0 + r, h - 1);
            const float v = (((float)gy + 0.5f) / (float)h) * (float)F.H0 - 0.5f;
            const float fj = floorf(v);
            const float b = v - fj, nb = 1.0f - b;
            s_fb[r] = make_float2(b, b);
            s_fnb[r] = make_float2(nb, nb);
            s_fy[r] = make_int2(edge_index(fj, F.H0) * pitch, edge_index(fj + 1.0f, F.H0) * pitch);
        }
    }
    __syncthreads();
    // two adjacent columns a thread: the row's terms and the loop serve both
    constexpr int COLS = TW / 2;
    const int tx = t % COLS * 2;
    const int x = X0 + tx;
    if (x >= w) return;
    const float2 nab0 = s_fa[tx], nab1 = s_fa[tx + 1];
    const int2 fx0 = s_fx[tx], fx1 = s_fx[tx + 1];
    const bool both = x + 1 < w;
    auto pixel = [&](const float2& nab, const int2& fx, const int2& fy, const float2& nb, const float2& b) {
        const float2 t0 = unit2_u8(__ldg(img + (uint32_t)(fy.x + fx.x)), __ldg(img + (uint32_t)(fy.x + fx.y)));
        const float2 t1 = unit2_u8(__ldg(img + (uint32_t)(fy.y + fx.x)), __ldg(img + (uint32_t)(fy.y + fx.y)));
        const float2 p0 = mul2_rn(mul2_rn(nab, nb), t0);
        const float2 p1 = mul2_rn(mul2_rn(nab, b), t1);
        float val = p0.x;
        val = val + p0.y;
        val = val + p1.x;
        return val + p1.y;
    };
#pragma unroll 2
    for (int ty = t / COLS; ty < TH; ty += K1_THREADS / COLS) {
        const int y = Y0 + ty;
        if (y >= h) break;
        const int2 fy = s_fy[ty];
        const float2 nb = s_fnb[ty], b = s_fb[ty];
        const float v0 = pixel(nab0, fx0, fy, nb, b), v1 = pixel(nab1, fx1, fy, nb, b);
        float* const o = out + (size_t)y * lp + x;
        if (both) *reinterpret_cast<float2*>(o) = make_float2(v0, v1);
        else *o = v0;
    }
}

// ---------------------------------------------------------------- K1 ----
// One TW x TH tile of one level: one TMA load stages the level pixels plus
// halo (written by k_pyramid) in shared memory, then the corner test in two
// passes: a warp first rejects its cells on a few points (and, in the
// reference's detector, on the cull mask) and lists the rest, then evaluates
// the listed ones 32 at a time, so the full circle runs on full warps.  On
// the 752x480 workload 5 % of the pixels are listed, while nearly every warp
// ran the circle for one lane or another: 32 frames 0.155 -> 0.100 ms; the cfg
// profile on 16 frames 0.29 -> 0.144, and 0.109 with signs for its compares, the run
// test by shifts and 5 CTAs per SM instead of 4 (6: 0.113).  Issue-bound still, 8 CTAs of 32 registers
// per SM; the mask's bits by one lane per 32 pixels, joined to the ballot, took it
// to 0.084 (eight 3840x2160 frames 482 -> 404 us).  A persistent form with the next tile's load in flight was
// slower (0.140): the CTAs of a launch already hide each other's loads.
// The strengths go through shared memory to 16-byte stores, whose nonzero
// bytes are the band's keypoint counts (without per-cell caps).
template <int TW, int TH, bool CFG>
__global__ void __launch_bounds__(K1_THREADS, CFG ? 5 : 8)
k_detect(const FrameDev* __restrict__ frames, const TileItem* __restrict__ tiles, int shape, uint32_t* err) {
    constexpr int HY = CFG ? HY_CFG : uslam::HY;
    constexpr int SW = TW + 2 * HX;                   // staged columns [X0 - HX, X0 + TW + HX)
    constexpr int SH = TH + 2 * HY;                   // staged rows [Y0 - HY, Y0 + TH + HY)
    constexpr int BW = TW + 2 * USLAM_TILE_XPAD;      // TMA box columns [X0 - XPAD, X0 + TW + XPAD)
    constexpr int CX = USLAM_TILE_XPAD - HX;          // box column of staged column 0
    constexpr int WARPS = K1_THREADS / 32;
    constexpr int ROWS = TH / WARPS;                  // tile rows of a warp
    constexpr int CELLS = CFG ? (TW + 2) * (TH + 2) : TW * TH;  // tested cells (cfg: with a ring of one)
    // listed cells of one warp (the widest cfg tiles in rounds of 128, for their shared memory)
    constexpr int LIST = CFG && TW * TH > 2048 ? 128 : (CELLS + 32 * WARPS - 1) / (32 * WARPS) * 32;
    constexpr int ARC0 = 15;  // s_arc's column of ring column 0: the tile's columns start on 16 bytes
    static_assert(TH % WARPS == 0 && TW % 32 == 0 && CX >= 0 && (BW * 4) % 16 == 0 && BW <= 256 && SH <= 256, "tile shape");
    __shared__ __align__(128) float sbox[SH][BW];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ __align__(16) uint8_t s_out[CFG ? 1 : TH][TW];      // strengths of the tile
    __shared__ uint16_t s_list[WARPS][LIST];                       // cells that passed the quick test
    __shared__ float s_score[CFG ? TH + 2 : 1][CFG ? TW + 2 : 1];  // cfg: FAST score, tile + 1 ring
    __shared__ __align__(16) uint8_t s_arc[CFG ? TH + 2 : 1][TW + 32];  // cfg: arc lengths, then strengths
    const TileItem it = tiles[blockIdx.x];
    const FrameDev& F = frames[it.frame];
    const int l = it.level;
    const int w = F.w[l], h = F.h[l];
    const int X0 = it.tx * TW, Y0 = it.ty * TH;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;

    // 0. one thread starts the tile load.  Box cells outside the level arrive
    //    as 0 and are replaced below.
    if (t == 0) {
        const void* tmap = static_cast<const char*>(F.tmaps) +
                           (size_t)(l * USLAM_TMAPS_PER_LEVEL + shape) * USLAM_TMAP_BYTES;
        mbar_init(&s_bar, 1u);
        mbar_expect_tx(&s_bar, (uint32_t)(SH * BW * 4));
        tma_load_2d(&sbox[0][0], tmap, X0 - USLAM_TILE_XPAD, Y0 - HY, &s_bar);
    }
    if constexpr (!CFG)
        for (int i = t; i < TW * TH / 16; i += K1_THREADS) reinterpret_cast<uint4*>(s_out)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();  // the barrier is initialised before anyone polls it
    const uint32_t first_limit = F.detect_first_wait < 0 ? kTmaWaitLimit : (uint32_t)F.detect_first_wait;
    const bool landed = mbar_wait(&s_bar, 0u, first_limit);
    if (__syncthreads_or(!landed)) {
        if (t == 0) atomicOr(err, USLAM_ERR_TMA_TIMEOUT);
        mbar_wait(&s_bar, 0u, kTmaWaitLimit);  // the copy in flight lands before the tile is left (full limit)
        return;
    }

    // 1. halo cells outside the level follow the Tint clamp min(u32(c), n - 1)
    //    (a negative coordinate reads the far edge)
    //    Only those cells are visited: whole rows above and below the level,
    //    then the columns left and right of it in the rows between.
    if (X0 < HX || X0 + TW + HX > w || Y0 < HY || Y0 + TH + HY > h) {
        const float* lv = F.lvl[l];
        const int lp = F.lvl_pitch[l];
        const int top = min(max(HY - Y0, 0), SH), bot = min(max(Y0 - HY + SH - h, 0), SH - top);
        const int left = min(max(HX - X0, 0), SW), right = min(max(X0 - HX + SW - w, 0), SW - left);
        const int nrow = (top + bot) * SW, nside = (SH - top - bot) * (left + right);
        for (int idx = t; idx < nrow + nside; idx += K1_THREADS) {
            int r, c;
            if (idx < nrow) {
                const int k = idx / SW;
                r = k < top ? k : SH - bot + (k - top);
                c = idx - k * SW;
            } else {
                const int k = idx - nrow, rr = k / (left + right), cc = k - rr * (left + right);
                r = top + rr;
                c = cc < left ? cc : SW - right + (cc - left);
            }
            const int gy = Y0 - HY + r, gx = X0 - HX + c;
            sbox[r][c + CX] = __ldg(lv + (size_t)tint_clamp(gy, h) * lp + tint_clamp(gx, w));
        }
        __syncthreads();
    }
    // staged cell (r, c) = sm[r][c], c counted from X0 - HX
    const float(*sm)[BW] = reinterpret_cast<const float(*)[BW]>(&sbox[0][CX]);
    uint16_t* const list = s_list[warp];
    const uint32_t below = (1u << lane) - 1u;
    uint32_t nlist = 0;
    if constexpr (CFG) {
        // 2. cells of the tile and its 1-pixel ring; pixels within 3 of the
        //    level edge (and outside the level) are never corners.  An arc of 9
        //    of the 16 points holds two of the points 0, 4, 8 and 12.
        for (int i0 = 32 * warp; i0 < CELLS;) {
            for (nlist = 0; i0 < CELLS && nlist + 32u <= (uint32_t)LIST; i0 += 32 * WARPS) {
                const int i = i0 + lane, sr = i / (TW + 2), sc = i - sr * (TW + 2);
                const int y = Y0 - 1 + sr, x = X0 - 1 + sc;
                bool pass = false;
                if (i < CELLS) {
                    s_score[sr][sc] = 0.0f;
                    s_arc[sr][ARC0 + sc] = 0;
                    if (y >= 3 && y < h - 3 && x >= 3 && x < w - 3) {
                        const int r = sr - 1 + HY, c = sc - 1 + HX;
                        const float center = sm[r][c];
                        // two of them beyond the threshold: the second largest or smallest
                        // is (a rounded difference does not decrease with p)
                        const float p0 = sm[r + circle_y(0)][c + circle_x(0)], p4 = sm[r + circle_y(4)][c + circle_x(4)];
                        const float p8 = sm[r + circle_y(8)][c + circle_x(8)], p12 = sm[r + circle_y(12)][c + circle_x(12)];
                        const float h0 = fmaxf(p0, p4), l0 = fminf(p0, p4), h1 = fmaxf(p8, p12), l1 = fminf(p8, p12);
                        const float large = fmaxf(fminf(h0, h1), fmaxf(l0, l1)), small = fminf(fmaxf(l0, l1), fminf(h0, h1));
                        pass = large - center > kCfgThreshold || center - small > kCfgThreshold;
                    }
                }
                const uint32_t b = __ballot_sync(0xffffffffu, pass);
                if (pass) list[nlist + __popc(b & below)] = (uint16_t)i;
                nlist += __popc(b);
            }
            __syncwarp();
            for (uint32_t q = lane; q < nlist; q += 32u) {
                const int i = list[q], sr = i / (TW + 2), sc = i - sr * (TW + 2);
                uint32_t arc;
                s_score[sr][sc] = cfg_corner(sm, sr - 1 + HY, sc - 1 + HX, &arc);
                s_arc[sr][ARC0 + sc] = (uint8_t)arc;
            }
            __syncwarp();
        }
        __syncthreads();
        // 3. 3x3 NMS on the score; a tie goes to the first pixel in raster
        //    order (a cell's arc is read and replaced by its own thread alone)
        for (int i = lane; i < ROWS * TW; i += 32) {
            const int sr = warp * ROWS + i / TW + 1, sc = i % TW + 1;
            const uint32_t A = s_arc[sr][ARC0 + sc];
            if (A == 0u) continue;
            const float Sc = s_score[sr][sc];
            bool ok = true;
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
                for (int dx = -1; dx <= 1; ++dx) {
                    if (dy == 0 && dx == 0) continue;
                    const float v = s_score[sr + dy][sc + dx];
                    const bool earlier = dy < 0 || (dy == 0 && dx < 0);
                    ok = ok && (earlier ? (Sc > v) : (Sc >= v));
                }
            if (!ok) s_arc[sr][ARC0 + sc] = 0;
        }
        __syncwarp();
    } else {
        // 2. the warp's rows, 32 pixels at a time: the cull mask
        //    (resources/cull_corners.wgsl; a lane has one segment's bits, none
        //    outside the level), then points 7 and 8, which every
        //    non-wrapping run of 9 holds, and 4 or 12, one of which it holds
        constexpr int SEGS = TW / 32;
        static_assert(ROWS * SEGS <= 32, "a lane per segment");
        uint32_t mine = 0u;
        {
            const uint32_t* mask = F.mask[l];
            const int last = (w * h - 1) >> 5;  // (a level holds fewer than 2^31 pixels)
            const int y = Y0 + warp * ROWS + lane / SEGS, x = X0 + 32 * (lane % SEGS);
            if (lane < ROWS * SEGS && y < h && x < w) {
                const int p0 = y * w + x, q0 = p0 >> 5;
                mine = __funnelshift_r(__ldg(mask + min(q0, last)), __ldg(mask + min(q0 + 1, last)), p0 & 31);
                if (w - x < 32) mine &= (1u << (w - x)) - 1u;
            }
        }
#pragma unroll
        for (int k = 0; k < ROWS * SEGS; ++k) {
            const uint32_t m = __shfl_sync(0xffffffffu, mine, k);
            if (m == 0u) continue;
            const int ty = warp * ROWS + k / SEGS, tx = 32 * (k % SEGS) + lane;
            const int r = ty + HY, c = tx + HX;
            const float center = sm[r][c];
            const float d7 = fabsf(center - sm[r + 3][c + 1]), d8 = fabsf(center - sm[r + 3][c]);
            const float d4 = fabsf(center - sm[r][c + 3]), d12 = fabsf(center - sm[r][c - 3]);
            const uint32_t b = __ballot_sync(0xffffffffu, fminf(fminf(d7, d8), fmaxf(d4, d12)) > 0.15f) & m;
            if (b == 0u) continue;
            if ((b >> lane) & 1u) list[nlist + __popc(b & below)] = (uint16_t)(ty * TW + tx);
            nlist += __popc(b);
        }
        __syncwarp();
        // 3. the listed cells: FAST response (and the rest of the cull)
        for (uint32_t q = lane; q < nlist; q += 32u) {
            const int i = list[q], ty = i / TW, tx = i - ty * TW;
            const int r = ty + HY, c = tx + HX;
            const uint32_t S = fast_response(sm, r, c);
            uint32_t keep = S;
            if (S > 0u && Y0 + ty == 0) {
                // row 0: first arg-max of the 1x3 region [9k, min(9k+3, w))
                const int x = X0 + tx, start = x - x % 9, end = min(start + 3, w);
                for (int u = start; u < end; ++u) {
                    if (u == x) continue;
                    const uint32_t Sq = fast_response(sm, r, c + (u - x));
                    if ((u < x && Sq >= S) || (u > x && Sq > S)) keep = 0;
                }
            }
            s_out[ty][tx] = (uint8_t)keep;
        }
        __syncwarp();
    }
    // 4. the warp's rows of the map, 16 bytes a lane (X0 + 16 k < w lies within the row's pitch)
    uint8_t* const kpmap = F.kpmap[l];
    const int kp_pitch = F.kp_pitch[l];
    uint32_t found = 0;
    for (int q = lane; q < ROWS * TW / 16; q += 32) {
        const int ty = warp * ROWS + q / (TW / 16), tx = q % (TW / 16) * 16;
        if (Y0 + ty >= h || X0 + tx >= w) continue;
        const uint4 v = *reinterpret_cast<const uint4*>(CFG ? &s_arc[CFG ? ty + 1 : 0][ARC0 + 1 + tx] : &s_out[CFG ? 0 : ty][tx]);
        *reinterpret_cast<uint4*>(kpmap + (size_t)(Y0 + ty) * kp_pitch + X0 + tx) = v;
        found += nonzero_bytes16(v);
    }
    if (F.cell_cap <= 0) {
        // raw and kept counts of the 32-row band (equal), as one 64-bit word
        found = warp_sum_u32(found);
        if (lane == 0 && found > 0u)
            atomicAdd(reinterpret_cast<unsigned long long*>(F.bands[l] + 2 * ((Y0 + warp * ROWS) / 32)),
                      (unsigned long long)found << 32 | found);
    }
}

// -------------------------------------------------------------- blur ----
// The blur cache G(P) of generate_features.wgsl:149-172 at every integer
// point a described keypoint's tests can read.  9 bilinear taps at offsets
// -1.2, 0, 1.2: tap (i, j) is sv = (na nb) T00 + (a nb) T10 + (na b) T01 +
// (a b) T11 summed left to right, q = (sv wt_i) wt_j, and G = the q summed
// j-major, i-minor.  The sampling coordinates of a tap depend only on the
// column or only on the row.
//
// The samples of a keypoint lie within R = margin - 1 of it, so a run needs
// only the tiles that k_band_write listed: 71 % of the pixels on the 752x480
// workload (the level caps keep the first features in (y, x) order, so the
// lower part of most levels holds none), 55 % at 1920x1080 and a few per cent
// where a frame cap of 20000 is used up by the first level of a 4K frame.
// 64 frames of 752x480: 0.25 ms here and 0.16 in k_detect, where evaluating
// every pixel in k_detect and the margins in a kernel of their own took 0.72
// and 0.20; 8 frames of 3840x2160 with that cap: 0.16 and 0.40 against 1.77
// and 0.13.
constexpr int KBL_THREADS = 128;
constexpr int KBL_TW = USLAM_BLUR_TW, KBL_TH = USLAM_BLUR_TH;
constexpr int KBL_HY = USLAM_BLUR_HY, KBL_XPAD = USLAM_BLUR_XPAD;
constexpr int KBL_SH = KBL_TH + 2 * KBL_HY;    // staged rows [Y0 - HY, Y0 + TH + HY)
constexpr int KBL_BW = KBL_TW + 2 * KBL_XPAD;  // staged columns [X0 - XPAD, X0 + TW + XPAD)
constexpr int KBL_CTAS_PER_SM = 6;
static_assert(KBL_TW == 2 * 32 && KBL_THREADS % 32 == 0, "a warp covers a tile row, two columns a lane");

// Tap k = 0, 1, 2 of coordinate c in a level of n pixels: the lower texel
// (before the edge clamp) and the upper one's weight.
__device__ __forceinline__ float blur_tap(uint32_t c, int k, int n, float* weight) {
    const float tex = 1.0f / (float)n;
    const float off = k == 0 ? -1.2f : (k == 1 ? 0.0f : 1.2f);
    const float u = (((float)c + 0.5f) * tex + off * tex) * (float)n - 0.5f;
    const float f = floorf(u);
    *weight = u - f;
    return f;
}

// G at (px, py), taps read from the level in global memory: the cells beyond
// the level, where a coordinate of 0xffffffff stands for every negative one
// (u32 wrap: the same f32 2^32 for all of them).
__device__ __noinline__ float blur_cell(const float* lvl, int lp, int w, int h, uint32_t px, uint32_t py) {
    float a[3], b[3];
    int x0[3], x1[3];
    const float *r0[3], *r1[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float fi = blur_tap(px, k, w, &a[k]), fj = blur_tap(py, k, h, &b[k]);
        x0[k] = edge_index(fi, w);
        x1[k] = edge_index(fi + 1.0f, w);
        r0[k] = lvl + (size_t)edge_index(fj, h) * lp;
        r1[k] = lvl + (size_t)edge_index(fj + 1.0f, h) * lp;
    }
    float sum = 0.0f;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float na = 1.0f - a[i], nb = 1.0f - b[j];
            float sv = (na * nb) * __ldg(r0[j] + x0[i]);
            sv = sv + (a[i] * nb) * __ldg(r0[j] + x1[i]);
            sv = sv + (na * b[j]) * __ldg(r1[j] + x0[i]);
            sv = sv + (a[i] * b[j]) * __ldg(r1[j] + x1[i]);
            sum = sum + (sv * (i == 1 ? 0.375f : 0.3125f)) * (j == 1 ? 0.375f : 0.3125f);
        }
    return sum;
}

// Two binary32 values side by side (sm_100 family f32x2 operands).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// Packed sum: p * 1 + q with the 1 unknown to the compiler, so each lane is
// rounded once, exactly as add.rn (p * 1 is exact), and the product that made
// p keeps its own rounding (see mul2_rn).
__device__ __forceinline__ f32x2 add2(f32x2 p, f32x2 q, f32x2 one) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(p), "l"(one), "l"(q));
    return d;
}

// Persistent over the list: a CTA's first two items are fixed, the later ones
// claimed (items cost different amounts), and the next tile's TMA load is
// issued while this one is computed.
//
// A tile costs 36 weight products, 36 texel products, 18 tap weights and 35
// sums a pixel on the FMA pipe, which bounds it (a packed operation holds the
// pipe for two cycles, so packing saves issue slots only).  What is saved is
// work on values that repeat, with every remaining operation as written:
//  * the weights (b, 1 - b) of a row tap take about ten values in a whole
//    level and equal the row above's in two rows of three, so the twelve
//    products with the column weights are kept from row to row;
//  * the middle row tap sits on the row itself (b = 0 exactly) in three rows
//    of four: its products with 1 - b = 1 are the column weights and its lower
//    row adds zeros;
//  * a lane takes two adjacent columns as the halves of packed operations and
//    four rows: the 6 columns its taps touch are three aligned 8-byte shared
//    loads, and the rows of the outer taps are shared by consecutive rows.
// The taps of a pixel sit at -2, -1 | d, d + 1 | 1, 2 around it, d = -1 or 0
// per row and per column by rounding (a tile that holds another pixel takes
// blur_cell throughout), and the staged cells beyond the level hold the edge
// texel, so edge pixels take the same path.  one_f is 1.0f (see add2).
__global__ void __launch_bounds__(KBL_THREADS, KBL_CTAS_PER_SM)
k_blur(const FrameDev* __restrict__ frames, BlurList bl, uint32_t* err, float one_f) {
    constexpr int ROWS = 4;  // rows of a warp at a time
    __shared__ __align__(128) float sbox[2][KBL_SH][KBL_BW];
    __shared__ __align__(8) uint64_t s_bar[2];
    __shared__ __align__(16) float4 s_w[3][KBL_TH];  // (b, b, nb, nb) of the row taps
    __shared__ __align__(8) float s_a[3][KBL_TW];    // upper weights of the column taps
    __shared__ int s_dy[KBL_TH];                     // offset of the middle tap's rows
    __shared__ __align__(2) int8_t s_dx[KBL_TW];     // offset of the middle tap's columns
    __shared__ uint32_t s_claim[2];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t n = __ldcg(bl.count);
    const f32x2 one = pack2(one_f, one_f);
    auto fetch = [&](const TileItem& it, int buf) {  // one thread
        if (it.pad != USLAM_BLUR_TILE) return;
        const void* tmap = static_cast<const char*>(frames[it.frame].tmaps) +
                           (size_t)(it.level * USLAM_TMAPS_PER_LEVEL + USLAM_TMAP_BLUR) * USLAM_TMAP_BYTES;
        mbar_expect_tx(&s_bar[buf], (uint32_t)(KBL_SH * KBL_BW * 4));
        tma_load_2d(&sbox[buf][0][0], tmap, it.tx * KBL_TW - KBL_XPAD, it.ty * KBL_TH - KBL_HY, &s_bar[buf]);
    };
    if (blockIdx.x >= n) return;
    TileItem it = bl.items[blockIdx.x];
    if (t == 0) {
        mbar_init(&s_bar[0], 1u);
        mbar_init(&s_bar[1], 1u);
        fetch(it, 0);
    }
    __syncthreads();  // the barriers are initialised before anyone polls them
    uint32_t phase = 0u;  // bit b: parity of buffer b's next load
    int cur = 0;
    uint32_t inext = blockIdx.x + gridDim.x;
    while (true) {
        const bool more = inext < n;
        TileItem next{};
        if (more) next = bl.items[inext];
        uint32_t claimed = 0;
        if (more && t == 0) {
            fetch(next, cur ^ 1);  // that buffer was read before the last barrier
            claimed = 2u * gridDim.x + atomicAdd(bl.count + 1, 1u);
        }
        const FrameDev& F = frames[it.frame];
        const int l = it.level;
        const int w = F.w[l], h = F.h[l], bp = F.bl_pitch[l];
        float* const blur = F.blur[l];
        const int X0 = it.tx * KBL_TW, Y0 = it.ty * KBL_TH;
        bool regular = it.pad == USLAM_BLUR_TILE;
        int c0 = X0, r0 = Y0, nc = min(KBL_TW, w - X0), nr = min(KBL_TH, h - Y0);  // the item's cells
        if (regular) {
            float a;
            // taps of the tile's columns (threads 0 .. 63) and rows (64 .. 95)
            if (t < KBL_TW + KBL_TH) {
                const bool column = t < KBL_TW;
                const int c = column ? t : t - KBL_TW, x = (column ? X0 : Y0) + c, size = column ? w : h;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int d = (int)blur_tap((uint32_t)x, k, size, &a) - x;
                    if (column) s_a[k][c] = a;
                    else s_w[k][c] = make_float4(a, a, 1.0f - a, 1.0f - a);
                    if (k == 1 && column) s_dx[c] = (int8_t)d;
                    if (k == 1 && !column) s_dy[c] = d;
                    regular = regular && (k == 0 ? d == -2 : (k == 1 ? d == -1 || d == 0 : d == 1));
                }
            }
            const bool landed = mbar_wait(&s_bar[cur], (phase >> cur) & 1u, kTmaWaitLimit);
            if (__syncthreads_or(!landed)) {
                if (t == 0) atomicOr(err, USLAM_ERR_TMA_TIMEOUT);
                // the copies in flight land before the CTA leaves
                mbar_wait(&s_bar[cur], (phase >> cur) & 1u, kTmaWaitLimit);
                if (more && next.pad == USLAM_BLUR_TILE) mbar_wait(&s_bar[cur ^ 1], (phase >> (cur ^ 1)) & 1u, kTmaWaitLimit);
                return;
            }
            phase ^= 1u << cur;
            // cells up to two beyond the level take the edge texel
            if (X0 == 0 || X0 + KBL_TW + 2 > w || Y0 == 0 || Y0 + KBL_TH + 2 > h) {
                float(*sm)[KBL_BW] = sbox[cur];
                const int x1 = min(X0 + KBL_TW, w), y1 = min(Y0 + KBL_TH, h);  // one past the tile's cells
                auto edge = [&](int gy, int gx) {
                    const int ey = min(max(gy, 0), h - 1), ex = min(max(gx, 0), w - 1);
                    if (ey != gy || ex != gx)  // (the texel is inside the level, so no thread writes it, and in the box)
                        sm[gy - Y0 + KBL_HY][gx - X0 + KBL_XPAD] = sm[ey - Y0 + KBL_HY][ex - X0 + KBL_XPAD];
                };
                // the two rows above and below over the tile's columns and two
                // each side, the two columns left and right over its rows
                for (int q = t; q < 4 * (x1 - X0 + 4); q += KBL_THREADS)
                    edge((q & 2) ? y1 + (q & 1) : Y0 - 2 + (q & 1), X0 - 2 + (q >> 2));
                for (int q = t; q < 4 * (y1 - Y0); q += KBL_THREADS)
                    edge(Y0 + (q >> 2), (q & 2) ? x1 + (q & 1) : X0 - 2 + (q & 1));
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // a later load writes here again
            }
            regular = __syncthreads_and(regular);
        } else if (it.pad == USLAM_BLUR_RIGHT) {
            c0 = w;
            nc = F.margin;
        } else if (it.pad == USLAM_BLUR_BELOW) {
            r0 = h;
            nr = F.margin;
            nc = min(KBL_TW, w + F.margin + 1 - c0);
        } else if (it.pad == USLAM_BLUR_COL) {
            c0 = w + F.margin;
            nc = 1;
            r0 = it.ty * USLAM_BLUR_RUN;
            nr = min(USLAM_BLUR_RUN, h - r0);
        } else {
            r0 = h + F.margin;
            nr = 1;
            c0 = it.tx * USLAM_BLUR_RUN;
            nc = min(USLAM_BLUR_RUN, w + F.margin + 1 - c0);
        }
        if (regular) {
            const int x = X0 + 2 * lane;
            f32x2 pa[3], pna[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float2 a = *reinterpret_cast<const float2*>(&s_a[k][2 * lane]);
                pa[k] = pack2(a.x, a.y);
                pna[k] = pack2(1.0f - a.x, 1.0f - a.y);
            }
            const char2 dx = *reinterpret_cast<const char2*>(&s_dx[2 * lane]);
            const f32x2 w3 = pack2(0.3125f, 0.3125f), w4 = pack2(0.375f, 0.375f);
            // the left and right texels of the three column taps in a staged row
            auto texels = [&](const float* p, f32x2 (&lt)[3], f32x2 (&rt)[3]) {
                lt[0] = *reinterpret_cast<const f32x2*>(p - 2);
                const f32x2 mid = *reinterpret_cast<const f32x2*>(p);
                rt[2] = *reinterpret_cast<const f32x2*>(p + 2);
                const float2 f0 = unpack2(lt[0]), f1 = unpack2(mid), f2 = unpack2(rt[2]);
                rt[0] = pack2(f0.y, f1.x);
                lt[2] = pack2(f1.y, f2.x);
                lt[1] = pack2(dx.x ? f0.y : f1.x, dx.y ? f1.x : f1.y);
                rt[1] = pack2(dx.x ? f1.x : f1.y, dx.y ? f1.y : f2.x);
            };
            for (int ty0 = warp * ROWS; ty0 < nr; ty0 += KBL_THREADS / 32 * ROWS) {
                const float* const col = &sbox[cur][KBL_HY + ty0][2 * lane + KBL_XPAD];
                f32x2 sum[ROWS];
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const f32x2 wj = j == 1 ? w4 : w3;
                    f32x2 w00[3], w10[3], w01[3], w11[3];  // the products of the column and row weights
                    f32x2 lt[2][3], rt[2][3];
                    ulonglong2 had = make_ulonglong2(0ull, 0ull);
                    if (j != 1) texels(col + (j == 0 ? -2 : 1) * KBL_BW, lt[0], rt[0]);
#pragma unroll
                    for (int r = 0; r < ROWS; ++r) {
                        const ulonglong2 wr = *reinterpret_cast<const ulonglong2*>(&s_w[j][ty0 + r]);
                        if (j == 1 && wr.x == 0ull) {
                            // b = 0: one row, weights 1 - a and a
                            texels(col + (r + s_dy[ty0 + r]) * KBL_BW, lt[0], rt[0]);
#pragma unroll
                            for (int k = 0; k < 3; ++k) {
                                const f32x2 sv = add2(mul2(pa[k], rt[0][k]), mul2(pna[k], lt[0][k]), one);
                                sum[r] = add2(mul2(mul2(sv, k == 1 ? w4 : w3), wj), sum[r], one);
                            }
                            continue;
                        }
                        const int u = j == 1 ? 0 : r & 1, d = u ^ 1;  // the upper and the lower row's texels
                        if (j == 1) {
                            const float* p = col + (r + s_dy[ty0 + r]) * KBL_BW;
                            texels(p, lt[0], rt[0]);
                            texels(p + KBL_BW, lt[1], rt[1]);
                        } else {
                            texels(col + (r + (j == 0 ? -1 : 2)) * KBL_BW, lt[d], rt[d]);
                        }
                        if (j == 1 || r == 0 || wr.x != had.x) {  // (equal b, equal 1 - b)
#pragma unroll
                            for (int k = 0; k < 3; ++k) {
                                w00[k] = mul2(pna[k], wr.y);
                                w10[k] = mul2(pa[k], wr.y);
                                w01[k] = mul2(pna[k], wr.x);
                                w11[k] = mul2(pa[k], wr.x);
                            }
                            had = wr;
                        }
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            f32x2 sv = mul2(w00[k], lt[u][k]);
                            sv = add2(mul2(w10[k], rt[u][k]), sv, one);
                            sv = add2(mul2(w01[k], lt[d][k]), sv, one);
                            sv = add2(mul2(w11[k], rt[d][k]), sv, one);
                            const f32x2 q = mul2(mul2(sv, k == 1 ? w4 : w3), wj);
                            sum[r] = j == 0 && k == 0 ? q : add2(q, sum[r], one);  // 0 + q = q: no texel is negative
                        }
                    }
                }
                float* o = blur + (size_t)(Y0 + ty0) * bp + x;
#pragma unroll
                for (int r = 0; r < ROWS; ++r, o += bp) {
                    const float2 s = unpack2(sum[r]);
                    if (ty0 + r >= nr) break;
                    if (x + 1 < w) *reinterpret_cast<float2*>(o) = s;  // bp and x are even
                    else if (x < w) *o = s.x;
                }
            }
        } else {
            const int M = F.margin, lp = F.lvl_pitch[l];
            const float* lvl = F.lvl[l];
            for (int k = t; k < nc * nr; k += KBL_THREADS) {
                const int r = k / nc, ey = r0 + r, ex = c0 + (k - r * nc);
                blur[(size_t)ey * bp + ex] =
                    blur_cell(lvl, lp, w, h, ex < w + M ? (uint32_t)ex : 0xffffffffu, ey < h + M ? (uint32_t)ey : 0xffffffffu);
            }
        }
        if (!more) break;
        if (t == 0) s_claim[cur] = claimed;
        __syncthreads();  // the tables and this buffer are rewritten from here on
        inext = s_claim[cur];
        it = next;
        cur ^= 1;
    }
}

// ------------------------------------------------------------ compact ----
constexpr int KC_THREADS = 1024;

// Block-wide exclusive scan of one value per thread; returns the prefix and
// writes the block total to *total.
__device__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* s_warp, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = (blockDim.x + 31) >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t wv = lane < nwarps ? s_warp[lane] : 0u;
        uint32_t wi = wv;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < nwarps) s_warp[lane] = wi - wv;
        if (lane == 31) s_warp[32] = wi;
    }
    __syncthreads();
    const uint32_t res = s_warp[warp] + incl - v;
    *total = s_warp[32];
    __syncthreads();
    return res;
}

// (one 16-byte store; the orientation, its last word, is k_describe's)
__device__ __forceinline__ void write_header(uint32_t* feats, uint32_t pos, int x, int y, uint32_t s) {
    *reinterpret_cast<uint4*>(feats + (size_t)pos * 12u) =
        make_uint4(__float_as_uint((float)x), __float_as_uint((float)y), s, 0u);
}

// One lane's 32-pixel row segment of a 32x32 cell (the map's padding beyond w is 0).
__device__ __forceinline__ void load_cell_row(const uint8_t* kp, int kpitch, int w, int h, int x0, int y, uint4 (&v)[2]) {
    const uint8_t* row = kp + (size_t)y * kpitch + x0;
#pragma unroll
    for (int j = 0; j < 2; ++j)  // x0 + 16 j + 16 <= kpitch (a multiple of 16)
        v[j] = y < h && x0 + 16 * j < w ? *reinterpret_cast<const uint4*>(row + 16 * j) : make_uint4(0u, 0u, 0u, 0u);
}

// The lowest room set bits of mask, which has n.
__device__ __forceinline__ uint32_t first_bits(uint32_t mask, uint32_t n, uint32_t room) {
    for (; n > room; --n) mask ^= 1u << (31 - __clz((int)mask));
    return mask;
}
// A lane's keypoints in order: bit b of mask is one at x + b with the strength
// in byte b of v.  Every lane takes its own next keypoint, so a warp's steps
// are the most of a lane (2 or 3) instead of all 16 bytes.
__device__ __forceinline__ void write_headers16(uint32_t* feats, uint32_t mask, const uint4& v, uint32_t pos, int x, int y) {
    while (mask) {
        const int b = __ffs((int)mask) - 1;
        mask &= mask - 1u;
        const uint32_t s = b < 8 ? __byte_perm(v.x, v.y, b & 7) : __byte_perm(v.z, v.w, b & 7);
        write_header(feats, pos++, x + b, y, s & 0xffu);
    }
}

// LOD-0 y of a feature (match_features_cpu.cpp:58-64: f32 scale iterated).
__device__ __forceinline__ float lod0_y(uint32_t y_bits, float scale) {
    return (float)(uint32_t)__uint_as_float(y_bits) * scale;
}

// The matcher's index of one level.  The frame height is cut into
// B = F.nbands bands (LOD-0 rows [b H0 / B, (b + 1) H0 / B)):
//  * candidate list b = the features whose LOD-0 y lies in band b widened by
//    0.1 H0 + 2 (the window half-height plus slack), sorted by x, with the
//    first slot of each column; every feature inside the window of a query
//    of band b is in list b;
//  * query order = the features grouped by the band of their own LOD-0 y,
//    sorted by x within a band, with the band offsets after the column tables.
// One CTA per (frame, level, list): a counting sort by x in shared memory
// (s_hist of w + 1 counters), the candidate lists and the bands of the query
// order side by side (a CTA that made all six lists in turn took 51 us on the
// largest level of a 1920x1080 frame).  XU features a thread are in flight at
// a time.
constexpr int XU = 4;
__global__ void __launch_bounds__(KC_THREADS, 2)
k_xsort(const FrameDev* __restrict__ frames, const SegDev* __restrict__ segs) {
    extern __shared__ uint32_t s_hist[];  // [w + 1]
    __shared__ uint32_t s_warp[33];
    const SegDev sg = segs[blockIdx.x];
    const FrameDev& F = frames[sg.frame];
    const int NB = F.nbands;
    if ((int)blockIdx.y >= 2 * NB) return;  // a batch with frames of more bands
    const int l = sg.level, w = F.w[l];
    const bool query = (int)blockIdx.y >= NB;
    const int b = (int)blockIdx.y - (query ? NB : 0);
    const uint32_t kept = F.kept[l];
    const uint32_t* feats = F.feats[l];
    float scale = 1.0f;
    for (int i = 0; i < l; ++i) scale = scale * 1.2f;
    const float H = (float)(uint32_t)F.H0;
    const float margin = 0.1f * H + 2.0f;
    const float lo = (float)b * H / (float)NB - margin, hi = (float)(b + 1) * H / (float)NB + margin;
    const size_t cap = (size_t)(F.cap > 0 ? F.cap : 1);
    // -1: in an earlier band's list of the query order, 0: in this list, 1: in neither
    auto place = [&](float y) {
        if (!query) return y >= lo && y <= hi ? 0 : 1;
        const int q = match_band(y, H, NB);
        return q < b ? -1 : (q == b ? 0 : 1);
    };
    for (int i = threadIdx.x; i <= w; i += KC_THREADS) s_hist[i] = 0u;
    __syncthreads();
    uint32_t earlier = 0;
    for (uint32_t i0 = threadIdx.x; i0 < kept; i0 += XU * KC_THREADS) {
        uint2 xy[XU];
#pragma unroll
        for (int u = 0; u < XU; ++u) {
            const uint32_t i = i0 + u * KC_THREADS;
            if (i < kept) xy[u] = *reinterpret_cast<const uint2*>(feats + (size_t)i * 12u);
        }
#pragma unroll
        for (int u = 0; u < XU; ++u) {
            if (i0 + u * KC_THREADS >= kept) break;
            const int p = place(lod0_y(xy[u].y, scale));
            if (p == 0) atomicAdd(&s_hist[(int)__uint_as_float(xy[u].x)], 1u);
            earlier += p < 0 ? 1u : 0u;
        }
    }
    __syncthreads();
    // this band's queries start after the earlier bands'
    uint32_t base = 0;
    if (query) block_exclusive_scan(earlier, s_warp, &base);
    uint32_t* const qband = F.colstart[l] + (size_t)NB * (size_t)(w + 1);
    uint32_t* const order = query ? F.qorder[l] + base : F.xorder[l] + (size_t)b * cap;
    uint32_t* const colstart = F.colstart[l] + (size_t)b * (size_t)(w + 1);
    // the tensor-core matcher's positions (null without it): of the query
    // order, then of each list (~0: not in it)
    uint32_t* const inv = F.winv[l] ? F.winv[l] + (query ? 0 : cap * (size_t)(1 + b)) : nullptr;
    const int per = (w + KC_THREADS) / KC_THREADS;  // bins per thread over w + 1 bins
    const int b0 = threadIdx.x * per;
    uint32_t local = 0;
    for (int k = 0; k < per; ++k)
        if (b0 + k < w) local += s_hist[b0 + k];
    uint32_t tot;
    uint32_t run = block_exclusive_scan(local, s_warp, &tot);
    for (int k = 0; k < per; ++k) {
        if (b0 + k > w) break;
        const uint32_t c = b0 + k < w ? s_hist[b0 + k] : 0u;
        if (!query) colstart[b0 + k] = run;
        s_hist[b0 + k] = run;  // becomes the fill cursor
        run += c;
    }
    if (query && threadIdx.x == 0) {
        qband[b] = base;
        if (b == NB - 1) qband[NB] = base + tot;
    }
    __syncthreads();
    for (uint32_t i0 = threadIdx.x; i0 < kept; i0 += XU * KC_THREADS) {
        uint2 xy[XU];
#pragma unroll
        for (int u = 0; u < XU; ++u) {
            const uint32_t i = i0 + u * KC_THREADS;
            if (i < kept) xy[u] = *reinterpret_cast<const uint2*>(feats + (size_t)i * 12u);
        }
#pragma unroll
        for (int u = 0; u < XU; ++u) {
            const uint32_t i = i0 + u * KC_THREADS;
            if (i >= kept) break;
            if (place(lod0_y(xy[u].y, scale)) == 0) {
                const uint32_t pos = atomicAdd(&s_hist[(int)__uint_as_float(xy[u].x)], 1u);
                order[pos] = i;
                if (inv) inv[i] = base + pos;
            } else if (inv && !query) {
                inv[i] = 0xffffffffu;
            }
        }
    }
}

// --------------------------------------------------- banded compaction ----
// Keypoint compaction, spread over one CTA per 32-row band of every level (a
// band is also one row of 32x32 cells):
//   k_band_count  per band: raw keypoints and keypoints kept by the cell caps
//   k_band_write  per band: prefix of the earlier bands' kept counts, then the
//                 ordered write of the band's headers below the level cap;
//                 band 0 also writes the level's raw / kept totals
//   k_xsort       per level: counting sort of the kept features by x
// The list order ((y, x), or cell order with per-cell caps) is the band
// order followed by the order inside each band; the level cap keeps the
// first `cap` of it (generate_features.wgsl:67-70 appends in a racy order,
// so this canonical order is the deterministic policy).
// A CTA has one warp per row of its band: a lane reads 16 map bytes at a time
// (a 752-pixel row is two loads a lane); four rows per warp, 4 bytes a lane at
// a time, were 24 dependent scans (18 against 11 us on one 752x480 frame, with
// the list of blur items on top here).
// Cells mode: the warps take the band's cells in turn, a lane one cell row.
constexpr int KBAND_THREADS = 1024;
constexpr int KBAND_WARPS = KBAND_THREADS / 32;
static_assert(KBAND_WARPS == USLAM_BLUR_TH, "a warp per row of a band, which is a blur tile row");

__device__ __forceinline__ uint32_t warp_inclusive_scan(uint32_t v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}
// Map bytes x .. x + 15 of a row (the map's padding beyond w is 0; x a multiple of 16).
__device__ __forceinline__ uint4 map16(const uint8_t* row, int x, int w) {
    return x < w ? *reinterpret_cast<const uint4*>(row + x) : make_uint4(0u, 0u, 0u, 0u);
}

// This warp's share of a band and its counts: one row (rows mode), or cells
// warp, warp + KBAND_WARPS, ... (cells mode).
__device__ __forceinline__ uint32_t band_row_count(const FrameDev& F, int l, int y) {
    const int lane = threadIdx.x & 31, w = F.w[l];
    const uint8_t* row = F.kpmap[l] + (size_t)y * F.kp_pitch[l];
    uint32_t r = 0;
    if (y < F.h[l])
        for (int x = 16 * lane; x < w; x += 512) r += nonzero_bytes16(map16(row, x, w));
    return warp_sum_u32(r);
}

// Raw and kept counts of a band with per-cell caps (without them k_detect
// counts, and this kernel does not run).
__global__ void __launch_bounds__(KBAND_THREADS)
k_band_count(const FrameDev* __restrict__ frames, const BandItem* __restrict__ items) {
    __shared__ uint32_t s_raw[KBAND_WARPS], s_kept[KBAND_WARPS];
    const BandItem it = items[blockIdx.x];
    const FrameDev& F = frames[it.frame];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int l = it.level, w = F.w[l], h = F.h[l];
    const uint32_t ccap = (uint32_t)F.cell_cap;
    uint32_t r = 0, k = 0;
    for (int cx = warp; cx * 32 < w; cx += KBAND_WARPS) {
        uint4 v[2];
        load_cell_row(F.kpmap[l], F.kp_pitch[l], w, h, cx * 32, it.band * 32 + lane, v);
        const uint32_t n = warp_sum_u32(nonzero_bytes16(v[0]) + nonzero_bytes16(v[1]));
        r += n;
        k += n < ccap ? n : ccap;
    }
    if (lane == 0) {
        s_raw[warp] = r;
        s_kept[warp] = k;
    }
    __syncthreads();
    if (warp == 0) {
        const uint32_t R = warp_sum_u32(s_raw[lane]), K = warp_sum_u32(s_kept[lane]);
        if (lane == 0) {
            F.bands[l][2 * it.band] = R;
            F.bands[l][2 * it.band + 1] = K;
        }
    }
}

// The blur items that the tests of keypoints in columns x0 .. x1 and rows
// y0 .. y1 can read: they reach R = margin - 1 cells each way, past the level
// the margins, and for negative coordinates the last column / row.
// visit(kind, index within the kind).
template <typename Visit>
__device__ __forceinline__ void for_blur_items(int w, int h, int M, int x0, int x1, int y0, int y1, Visit visit) {
    const int R = M - 1, nx = USLAM_BLUR_NX(w);
    const int xa = max(x0 - R, 0), ya = max(y0 - R, 0), xe = min(x1 + R, w + M - 1), ye = min(y1 + R, h - 1);
    for (int ty = ya / USLAM_BLUR_TH; ty <= ye / USLAM_BLUR_TH; ++ty) {
        for (int tx = xa / USLAM_BLUR_TW; tx <= min(xe, w - 1) / USLAM_BLUR_TW; ++tx) visit(USLAM_BLUR_TILE, ty * nx + tx);
        if (x1 + R >= w) visit(USLAM_BLUR_RIGHT, ty);
    }
    if (x0 < R)
        for (int ty = ya / USLAM_BLUR_RUN; ty <= ye / USLAM_BLUR_RUN; ++ty) visit(USLAM_BLUR_COL, ty);
    if (y1 + R >= h) {
        for (int tx = xa / USLAM_BLUR_TW; tx <= xe / USLAM_BLUR_TW; ++tx) visit(USLAM_BLUR_BELOW, tx);
        if (x0 < R) visit(USLAM_BLUR_BELOW, (w + M) / USLAM_BLUR_TW);
    }
    if (y0 < R) {
        for (int tx = xa / USLAM_BLUR_RUN; tx <= xe / USLAM_BLUR_RUN; ++tx) visit(USLAM_BLUR_ROW, tx);
        if (x0 < R) visit(USLAM_BLUR_ROW, (w + M) / USLAM_BLUR_RUN);
    }
}

// Kept keypoints are noted per 8 x 8 cells of the band in shared memory, the
// items those cells need are gathered there too (where a band's reach is at
// most the tile rows beside it), and each joins the run's list once.
constexpr int KBAND_NOTES = 8192 / 8;                     // of the widest level
constexpr int KBAND_REACH = 32;                           // of gathered marks
constexpr int KBAND_NX = 8192 / USLAM_BLUR_TW;            // tile columns of the widest level
constexpr int KBAND_NEX = KBAND_NX + 1;                   // with its margin
constexpr int KBAND_MARKS = 3 * (KBAND_NX + 1) + 2 * KBAND_NEX + 2;

__global__ void __launch_bounds__(KBAND_THREADS, 2)
k_band_write(const FrameDev* __restrict__ frames, const BandItem* __restrict__ items, BlurList bl) {
    __shared__ uint8_t s_note[4][KBAND_NOTES];
    __shared__ uint8_t s_mark[KBAND_MARKS];
    __shared__ uint32_t s_red[3][KBAND_WARPS];
    __shared__ uint32_t s_wbase[KBAND_WARPS];
    const BandItem it = items[blockIdx.x];
    const FrameDev& F = frames[it.frame];
    const int l = it.level, band = it.band;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int w = F.w[l], h = F.h[l], kpitch = F.kp_pitch[l];
    const uint8_t* kp = F.kpmap[l];
    const int nb = (h + 31) / 32, notes = (w + 7) / 8;
    const uint32_t* bc = F.bands[l];
    uint32_t cap = (uint32_t)F.cap;
    if (F.frame_cap > 0) {
        // per-frame cap: what the earlier levels left of it (their kept
        // counts follow from their band counts, every level's being complete)
        uint32_t left = (uint32_t)F.frame_cap;
        for (int q = 0; q < l && left > 0u; ++q) {
            const int nbq = (F.h[q] + 31) / 32;
            uint32_t kq = 0;
            for (int b2 = lane; b2 < nbq; b2 += 32) kq += F.bands[q][2 * b2 + 1];
            kq = min(warp_sum_u32(kq), (uint32_t)F.cap);
            left -= min(kq, left);
        }
        cap = min(cap, left);
    }
    // prefix of the earlier bands' kept counts (band 0: also the level totals)
    uint32_t pk = 0, tr = 0, tk = 0;
    for (int q = threadIdx.x; q < nb; q += KBAND_THREADS) {
        const uint32_t kq = bc[2 * q + 1];
        if (q < band) pk += kq;
        tr += bc[2 * q];
        tk += kq;
    }
    pk = warp_sum_u32(pk);
    tr = warp_sum_u32(tr);
    tk = warp_sum_u32(tk);
    const uint32_t mine_in_row = F.cell_cap <= 0 ? band_row_count(F, l, band * 32 + warp) : 0u;
    if (lane == 0) {
        s_red[0][warp] = pk;
        s_red[1][warp] = tr;
        s_red[2][warp] = tk;
        s_wbase[warp] = mine_in_row;
    }
    for (int i = threadIdx.x; i < 4 * notes; i += KBAND_THREADS) s_note[i & 3][i >> 2] = 0;
    for (int i = threadIdx.x; i < KBAND_MARKS; i += KBAND_THREADS) s_mark[i] = 0;
    __syncthreads();
    const uint32_t prefix = warp_sum_u32(s_red[0][lane]);
    if (band == 0 && warp == 0) {
        const uint32_t R = warp_sum_u32(s_red[1][lane]), K = warp_sum_u32(s_red[2][lane]);
        if (lane == 0) {
            F.raw[l] = R;
            F.kept[l] = K < cap ? K : cap;
        }
    }
    if (prefix >= cap) return;
    uint32_t* feats = F.feats[l];
    if (F.cell_cap <= 0) {
        // (y, x) order: the band's earlier rows, then the row's earlier lanes
        uint32_t running = prefix + warp_sum_u32(lane < warp ? s_wbase[lane] : 0u);
        const int y = band * 32 + warp;
        const uint8_t* row = kp + (size_t)y * kpitch;
        for (int x0 = 0; y < h && x0 < w && running < cap; x0 += 512) {
            const int x = x0 + 16 * lane;
            const uint4 v = map16(row, x, w);
            uint32_t mask = nonzero_mask16(v);
            const uint32_t n = (uint32_t)__popc(mask);
            const uint32_t incl = warp_inclusive_scan(n, lane);
            const uint32_t pos = running + incl - n;
            mask = first_bits(mask, n, pos < cap ? cap - pos : 0u);
            if (mask & 0x00ffu) s_note[warp >> 3][x >> 3] = 1;
            if (mask & 0xff00u) s_note[warp >> 3][(x >> 3) + 1] = 1;
            write_headers16(feats, mask, v, pos, x, y);
            running += __shfl_sync(0xffffffffu, incl, 31);
        }
    } else {
        // cell order: the band's earlier cells (all warps' shares are
        // interleaved, so each cell's base comes from a pass over the counts)
        const uint32_t ccap = (uint32_t)F.cell_cap;
        const int ncx = (w + 31) / 32, y = band * 32 + lane;
        __shared__ uint32_t s_cell[KBAND_WARPS];
        uint32_t base = prefix;
        for (int c0 = 0; c0 < ncx; c0 += KBAND_WARPS) {
            const int cx = c0 + warp;
            uint4 v[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
            if (cx < ncx) load_cell_row(kp, kpitch, w, h, cx * 32, y, v);
            uint32_t mask = nonzero_mask16(v[0]) | nonzero_mask16(v[1]) << 16;
            const uint32_t n = (uint32_t)__popc(mask);
            const uint32_t incl = warp_inclusive_scan(n, lane);
            const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
            if (lane == 0) s_cell[warp] = min(tot, ccap);
            __syncthreads();
            const uint32_t mine = s_cell[lane];
            const uint32_t running = base + warp_sum_u32(lane < warp ? mine : 0u);
            base += warp_sum_u32(mine);
            const uint32_t rank = incl - n, end = running < cap ? min(ccap, cap - running) : 0u;
            mask = first_bits(mask, n, rank < end ? end - rank : 0u);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (mask & (0xffu << (8 * q))) s_note[lane >> 3][4 * cx + q] = 1;
            const uint32_t low = (uint32_t)__popc(mask & 0xffffu);
            write_headers16(feats, mask & 0xffffu, v[0], running + rank, cx * 32, y);
            write_headers16(feats, mask >> 16, v[1], running + rank + low, cx * 32 + 16, y);
            __syncthreads();  // s_cell is rewritten
        }
    }
    __syncthreads();
    const int M = F.margin, nx = USLAM_BLUR_NX(w);
    auto claim = [&](int kind, int k) {
        uint32_t* m = F.btile[l] + k;
        if (kind == USLAM_BLUR_RIGHT) m += USLAM_BLUR_AT_RIGHT(w, h);
        else if (kind == USLAM_BLUR_BELOW) m += USLAM_BLUR_AT_BELOW(w, h);
        else if (kind == USLAM_BLUR_COL) m += USLAM_BLUR_AT_COL(w, h, M);
        else if (kind == USLAM_BLUR_ROW) m += USLAM_BLUR_AT_ROW(w, h, M);
        if (atomicExch(m, 1u) != 0u) return;
        const bool tile = kind == USLAM_BLUR_TILE, down = kind == USLAM_BLUR_RIGHT || kind == USLAM_BLUR_COL;
        TileItem ti;
        ti.frame = it.frame;
        ti.level = it.level;
        ti.pad = (uint8_t)kind;
        ti.tx = (uint16_t)(tile ? k % nx : down ? 0 : k);
        ti.ty = (uint16_t)(tile ? k / nx : down ? k : 0);
        bl.items[atomicAdd(bl.count, 1u)] = ti;
    };
    // gathered marks: rows band - 1 .. band + 1 of tiles and their right
    // margin runs, then the runs below, of the last column and of the last row
    const bool gather = M - 1 <= KBAND_REACH;
    const int ty0 = band - 1, cy0 = max(band * 32 - (M - 1), 0) / USLAM_BLUR_RUN;
    const int g_below = 3 * (nx + 1), g_col = g_below + USLAM_BLUR_NX(w + M + 1), g_row = g_col + 2,
              g_end = g_row + USLAM_BLUR_DIV(w + M + 1, USLAM_BLUR_RUN);
    for (int i = threadIdx.x; i < 4 * notes; i += KBAND_THREADS) {
        const int g = i & 3, c = i >> 2;
        if (!s_note[g][c]) continue;
        const int y0 = band * 32 + 8 * g;
        for_blur_items(w, h, M, 8 * c, min(8 * c + 7, w - 1), y0, min(y0 + 7, h - 1), [&](int kind, int k) {
            if (!gather) claim(kind, k);
            else if (kind == USLAM_BLUR_TILE) s_mark[(k / nx - ty0) * (nx + 1) + k % nx] = 1;
            else if (kind == USLAM_BLUR_RIGHT) s_mark[(k - ty0) * (nx + 1) + nx] = 1;
            else if (kind == USLAM_BLUR_BELOW) s_mark[g_below + k] = 1;
            else if (kind == USLAM_BLUR_COL) s_mark[g_col + k - cy0] = 1;
            else s_mark[g_row + k] = 1;
        });
    }
    if (!gather) return;
    __syncthreads();
    for (int i = threadIdx.x; i < g_end; i += KBAND_THREADS) {
        if (!s_mark[i]) continue;
        if (i < g_below) {
            const int r = i / (nx + 1), c = i - r * (nx + 1);
            if (c < nx) claim(USLAM_BLUR_TILE, (ty0 + r) * nx + c);
            else claim(USLAM_BLUR_RIGHT, ty0 + r);
        } else if (i < g_col) {
            claim(USLAM_BLUR_BELOW, i - g_below);
        } else if (i < g_row) {
            claim(USLAM_BLUR_COL, cy0 + i - g_col);
        } else {
            claim(USLAM_BLUR_ROW, i - g_row);
        }
    }
}

// ------------------------------------------------------------- K2 ----
constexpr int KD_THREADS = 1024;
constexpr int MAX_SEGS = 4096;

// Prefix over per-segment counts, shared by the persistent kernels.
template <typename CountFn>
__device__ uint32_t segment_prefix(int nseg, uint32_t* s_pref, uint32_t* s_warp, CountFn count) {
    const int per = (nseg + blockDim.x - 1) / blockDim.x;
    const int b0 = threadIdx.x * per;
    uint32_t local = 0;
    for (int k = 0; k < per; ++k)
        if (b0 + k < nseg) local += count(b0 + k);
    uint32_t tot;
    uint32_t run = block_exclusive_scan(local, s_warp, &tot);
    for (int k = 0; k < per; ++k) {
        if (b0 + k < nseg) {
            s_pref[b0 + k] = run;
            run += count(b0 + k);
        }
    }
    if (threadIdx.x == 0) s_pref[nseg] = tot;
    __syncthreads();
    return tot;
}

__device__ __forceinline__ int find_segment(const uint32_t* s_pref, int nseg, uint32_t g) {
    int lo = 0, hi = nseg - 1;  // largest s with s_pref[s] <= g
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s_pref[mid] <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}


// FP8 E4M3 code of an integer 0..16 (all exact: 2^k (1 + m / 8) with
// k = floor(log2 v) <= 4 and m = (v - 2^k) 8 / 2^k an integer).
__device__ __forceinline__ uint32_t e4m3_small_int(int v) {
    if (v <= 0) return 0u;
    const int k = 31 - __clz(v);
    return (uint32_t)(((k + 7) << 3) | (((v - (1 << k)) << 3) >> k));
}

// FP8 operand row of a descriptor (bit k -> 0x50 = 8.0 or 0x00) at row R of
// a K-major no-swizzle operand array: lane j writes bits 8 j .. 8 j + 7 (K
// chunk j / 2, half j % 2); wj = the descriptor word holding them.
__device__ __forceinline__ void write_fp8_row(uint8_t* base, uint32_t R, uint32_t wj, int lane) {
    const uint32_t bits = (wj >> (8 * (lane & 3))) & 0xffu;
    uint32_t lo = 0u, hi = 0u;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        lo |= ((bits >> b) & 1u) * (0x50u << (8 * b));
        hi |= ((bits >> (b + 4)) & 1u) * (0x50u << (8 * b));
    }
    *reinterpret_cast<uint2*>(base + (size_t)(R >> 3) * 2048u + (lane >> 1) * 128u + (R & 7u) * 16u + (lane & 1) * 8u) =
        make_uint2(lo, hi);
}
// Extension row (32 E4M3 values) at row R, lanes 0-3: the popcount pc split
// into 16 integers <= 16, then 256, grp split into two integers <= 16, then 1.
__device__ __forceinline__ void write_ext_row(uint8_t* base, uint32_t R, uint32_t pc, int grp, int lane) {
    uint32_t ext[2] = {0u, 0u};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int e = 8 * lane + k;  // extension value index 0..31
        uint32_t code = 0u;
        if (e < 16) code = e4m3_small_int(min(16, max(0, (int)pc - 16 * e)));
        else if (e == 16) code = 0x78u;  // 256
        else if (e == 17) code = e4m3_small_int(min(grp, 16));
        else if (e == 18) code = e4m3_small_int(max(grp - 16, 0));
        else if (e == 19) code = 0x38u;  // 1
        ext[k >> 2] |= code << (8 * (k & 3));
    }
    *reinterpret_cast<uint2*>(base + (size_t)(R >> 3) * 256u + (lane >> 1) * 128u + (R & 7u) * 16u + (lane & 1) * 8u) =
        make_uint2(ext[0], ext[1]);
}
// Query-order position k of level l -> its operand row (each band's queries
// from a multiple of 128 rows).
__device__ __forceinline__ uint32_t win_query_row(const uint32_t* qband, int nb, int l, int wq_rows, uint32_t k) {
    uint32_t off = (uint32_t)l * (uint32_t)wq_rows, b = 0;
    while (b + 1 < (uint32_t)nb && k >= qband[b + 1]) {
        off += (qband[b + 1] - qband[b] + 127u) / 128u * 128u;
        ++b;
    }
    return off + (k - qband[b]);
}

// Finish one keypoint's record (the warp holds its 8 descriptor words, lane
// k the word k of every lane): orientation and descriptor into the record
// (generate_features.wgsl:170-172), plus the tensor-core operand rows (PACK,
// WIN) of the matchers that take them.
template <bool PACK, bool WIN>
__device__ __forceinline__ void emit_feature(const FrameDev& F, int l, uint32_t i, int y, float theta,
                                             const uint32_t (&words)[8], int lane) {
    uint32_t* rec = F.feats[l] + (size_t)i * 12u;
    uint32_t out = __float_as_uint(theta);
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (lane == 4 + k) out = words[k];
    if (lane >= 3 && lane < 12) rec[lane] = out;
    if constexpr (WIN) {
        uint32_t wj = words[0];
        uint32_t pc = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if ((lane >> 2) == k) wj = words[k];
            pc += (uint32_t)__popc(words[k]);
        }
        const uint32_t* inv = F.winv[l];
        const size_t cap = (size_t)(F.cap > 0 ? F.cap : 1);
        const int nb = F.nbands;
        const uint32_t* qband = F.colstart[l] + (size_t)nb * (size_t)(F.w[l] + 1);
        write_fp8_row(F.wq8, win_query_row(qband, nb, l, F.wq_rows, __ldg(inv + i)), wj, lane);
        for (int b = 0; b < nb; ++b) {
            const uint32_t pos = __ldg(inv + cap * (size_t)(1 + b) + i);
            if (pos == 0xffffffffu) continue;
            const uint32_t R = (uint32_t)(nb * l + b) * (uint32_t)F.wc_rows + pos;
            write_fp8_row(F.wc8, R, wj, lane);
            if (lane < 4) write_ext_row(F.wcext, R, pc, (int)(pos & 31u), lane);
            else if (lane == 4) F.wcy[R] = (uint16_t)y;
            else if (lane == 5) F.wcid[R] = USLAM_PACK(l, i);
        }
    }
    if constexpr (PACK) {
        // tensor-core operand rows of this feature (flat index f over
        // the levels): lane j writes the FP8 values of descriptor bits
        // 8j .. 8j + 7 (8.0 or 0; K chunk j / 2, half j % 2); lanes 0-3
        // write the 32-value extension row: the popcount split into 16
        // integers <= 16, then 256, the row's index within its 32-row
        // group split into two integers <= 16, then 1, then zeros
        uint32_t f = i;
        for (int q = 0; q < l; ++q) f += F.kept[q];
        uint32_t wj = words[0];
        uint32_t pc = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if ((lane >> 2) == k) wj = words[k];
            pc += (uint32_t)__popc(words[k]);
        }
        const uint32_t bits = (wj >> (8 * (lane & 3))) & 0xffu;
        uint32_t lo = 0u, hi = 0u;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            lo |= ((bits >> b) & 1u) * (0x50u << (8 * b));
            hi |= ((bits >> (b + 4)) & 1u) * (0x50u << (8 * b));
        }
        *reinterpret_cast<uint2*>(F.bf8 + (size_t)(f >> 3) * 2048u + (lane >> 1) * 128u + (f & 7u) * 16u +
                                  (lane & 1) * 8u) = make_uint2(lo, hi);
        if (lane < 4) {
            uint32_t ext[2] = {0u, 0u};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int e = 8 * lane + k;  // extension value index 0..31
                const int grp = (int)(f & 31u);
                uint32_t code = 0u;
                if (e < 16) code = e4m3_small_int(min(16, max(0, (int)pc - 16 * e)));
                else if (e == 16) code = 0x78u;  // 256
                else if (e == 17) code = e4m3_small_int(min(grp, 16));
                else if (e == 18) code = e4m3_small_int(max(grp - 16, 0));
                else if (e == 19) code = 0x38u;  // 1
                ext[k >> 2] |= code << (8 * (k & 3));
            }
            *reinterpret_cast<uint2*>(F.bfext + (size_t)(f >> 3) * 256u + (lane >> 1) * 128u + (f & 7u) * 16u +
                                      (lane & 1) * 8u) = make_uint2(ext[0], ext[1]);
        }
        if (lane == 0) {
            F.bfpop[f] = pc;
            F.bfid[f] = USLAM_PACK(l, i);
        }
    }
}

// PACK: also write the brute-force tensor-core matcher's operand rows of
// every feature (FrameDev::bf8 / bfext / bfpop / bfid).  WIN: the windowed
// tensor-core matcher's rows: the feature's query row (wq8) and its row in
// every candidate list that holds it (wc8, wcext, wcy, wcid), at the
// positions k_xsort recorded (winv).
//
// One CTA of 32 warps per SM over runs of consecutive keypoints, so that the
// blur-cache strip its warps gather from stays in L1 (97 % sector hits against
// 86 % with four CTAs of 8 warps over runs far apart: 32 frames of 752x480
// 186 -> 155 us).  The gathers are then bound by the cache lines that a warp
// load touches: in test order 22 of 32 lanes' points lie in lines of their
// own, in compact clusters of the pattern under 9 (DescTable), and the values
// reach their tests through shared memory (155 -> 145 us; 3840x2160 frames of
// the mixed batch 700 -> 553 in all).  The L1 data pipe bounds it now, three
// quarters busy.
constexpr size_t kDescSmem = 512 * sizeof(__half2) + KD_THREADS / 32 * 512 * sizeof(float);

template <bool PACK, bool WIN>
__global__ void __launch_bounds__(KD_THREADS)
k_describe(const FrameDev* __restrict__ frames, const SegDev* __restrict__ segs, int nseg,
           const DescTable* __restrict__ table) {
    extern __shared__ __align__(16) uint8_t kd_smem[];  // the table's points, then each warp's gathered values
    __shared__ uint32_t s_pref[MAX_SEGS + 1];
    __shared__ uint32_t s_warp[33];
    // the r = 3 disc in (dy outer, dx inner) order as compile-time constants, so
    // the unrolled moment sum multiplies by immediates (same f32 operations)
    constexpr int8_t kdx[29] = {0, -2, -1, 0, 1, 2, -2, -1, 0, 1, 2, -3, -2, -1, 0, 1, 2, 3, -2, -1, 0, 1, 2, -2, -1, 0, 1, 2, 0};
    constexpr int8_t kdy[29] = {-3, -2, -2, -2, -2, -2, -1, -1, -1, -1, -1, 0, 0, 0, 0, 0, 0, 0, 1, 1, 1, 1, 1, 2, 2, 2, 2, 2, 3};
    constexpr uint32_t WARPS = KD_THREADS / 32;
    const int lane = threadIdx.x & 31;
    const uint32_t warp = threadIdx.x >> 5;
    // (a point's coordinates are integers below 1024, exact in 16 bits: half the shared-memory reads)
    __half2* const s_pts = reinterpret_cast<__half2*>(kd_smem);
    float* const vals = reinterpret_cast<float*>(kd_smem + 512 * sizeof(__half2)) + warp * 512u;
    for (int i = threadIdx.x; i < 512; i += KD_THREADS)
        s_pts[i] = __floats2half2_rn(table->pts[i >> 5][i & 31][0], table->pts[i >> 5][i & 31][1]);
    uint32_t pair[8];  // this lane's tests
#pragma unroll
    for (int k = 0; k < 8; ++k) pair[k] = table->pair[k][lane];
    const uint32_t total = segment_prefix(nseg, s_pref, s_warp, [&](int s) {
        return frames[segs[s].frame].kept[segs[s].level];
    });
    // A CTA takes an equal share of consecutive keypoints in runs of WARPS * G
    // (G <= 32), of which warp q takes every WARPS-th from the q-th on: lane
    // j < G first computes the orientation of the warp's keypoint j, then the
    // warp runs the 256 tests of each in turn with its position and angle
    // broadcast from that lane.
    const uint32_t share = (total + gridDim.x - 1u) / gridDim.x;
    const uint32_t end = min(total, (blockIdx.x + 1u) * share);
    const uint32_t kq = max((share + 32u * WARPS - 1u) / (32u * WARPS), 1u);
    const uint32_t G = (share + kq * WARPS - 1u) / (kq * WARPS);
    for (uint32_t c0 = blockIdx.x * share; c0 < end; c0 += WARPS * G) {
        const uint32_t g0 = c0 + warp;
        if (g0 >= end) break;
        // orientation (generate_features.wgsl:80-99): intensity moments over
        // the r = 3 disc, summed in the reference's order, then atan2
        int my_seg = 0;
        uint32_t my_idx = 0, my_xy = 0;
        float my_theta = 0.0f, my_s = 0.0f, my_c = 0.0f;
        if ((uint32_t)lane < G && g0 + lane * WARPS < end) {
            my_seg = find_segment(s_pref, nseg, g0 + lane * WARPS);
            my_idx = g0 + lane * WARPS - s_pref[my_seg];
            const FrameDev& F = frames[segs[my_seg].frame];
            const int l = segs[my_seg].level;
            const int w = F.w[l], h = F.h[l];
            const uint32_t* rec = F.feats[l] + (size_t)my_idx * 12u;
            const int x = (int)__uint_as_float(rec[0]);
            const int y = (int)__uint_as_float(rec[1]);
            my_xy = (uint32_t)y << 16 | (uint32_t)x;
            const float* lvl = F.lvl[l];
            const int lp = F.lvl_pitch[l];
            float m10 = 0.0f, m01 = 0.0f;
#pragma unroll
            for (int k = 0; k < 29; ++k) {
                const int cx = tint_clamp(x + kdx[k], w);
                const int cy = tint_clamp(y + kdy[k], h);
                const float v = __ldg(lvl + (size_t)cy * (size_t)lp + cx);
                m10 = m10 + (float)kdx[k] * v;
                m01 = m01 + (float)kdy[k] * v;
            }
            my_theta = uslam_atan2f(m01, m10);
            uslam_sincosf(my_theta, &my_s, &my_c);
        }
        int seg = -1, l = 0, reach = 0;
        const FrameDev* F = frames;
        const float* blur = nullptr;
        uint32_t bp = 0;
        const int nk = (int)min(G, (end - g0 + WARPS - 1u) / WARPS);
        for (int kp = 0; kp < nk; ++kp) {
            const int sidx = __shfl_sync(0xffffffffu, my_seg, kp);
            const uint32_t i = __shfl_sync(0xffffffffu, my_idx, kp);
            const float theta = __shfl_sync(0xffffffffu, my_theta, kp);
            const float s = __shfl_sync(0xffffffffu, my_s, kp);
            const float c = __shfl_sync(0xffffffffu, my_c, kp);
            const uint32_t xy = __shfl_sync(0xffffffffu, my_xy, kp);
            const int x = (int)(xy & 0xffffu), y = (int)(xy >> 16);
            if (sidx != seg) {
                // the level's addresses are kept from keypoint to keypoint
                seg = sidx;
                F = frames + segs[sidx].frame;
                l = segs[sidx].level;
                blur = F->blur[l];
                bp = (uint32_t)F->bl_pitch[l];
                reach = F->margin - 1;
            }
            // The 512 points' samples.  Adding 1.5 2^23 rounds a rotated
            // coordinate to the nearest integer, ties to even, into the low
            // bits of the sum (|coordinate| < 2^22), so the cache index is two
            // integer operations on the sums' bits, modulo 2^32, where the
            // constants cancel.  Keypoints within the pattern's reach of the
            // left or top edge (the same for the whole warp) also replace
            // negative coordinates by the sentinel column / row.
            constexpr float kRound = 12582912.0f;
            constexpr uint32_t kRoundBits = 0x4B400000u;
            const uint32_t cx = (uint32_t)x - kRoundBits, cy = (uint32_t)y - kRoundBits;
            // at(rounded x bits, rounded y bits): the sample
            auto gather = [&](auto at) {
#pragma unroll
                for (int q0 = 0; q0 < USLAM_DESC_CLUSTERS; q0 += 8) {
                    float v[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float2 p = __half22float2(s_pts[(q0 + q) * 32 + lane]);
                        v[q] = at(__float_as_uint((p.x * c - p.y * s) + kRound), __float_as_uint((p.x * s + p.y * c) + kRound));
                    }
#pragma unroll
                    for (int q = 0; q < 8; ++q) vals[(q0 + q) * 32 + lane] = v[q];
                }
            };
            if (x >= reach && y >= reach) {
                const uint32_t origin = cy * bp + cx;
                gather([&](uint32_t xr, uint32_t yr) { return __ldg(blur + (yr * bp + (xr + origin))); });
            } else {
                const int sx = F->w[l] + F->margin, sy = F->h[l] + F->margin;
                gather([&](uint32_t xr, uint32_t yr) {
                    const int px = (int)(xr + cx), py = (int)(yr + cy);
                    return __ldg(blur + (size_t)(py < 0 ? sy : py) * bp + (px < 0 ? sx : px));
                });
            }
            __syncwarp();
            // lane j runs tests j, j + 32, ..., j + 224
            uint32_t words[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                words[k] = __ballot_sync(0xffffffffu, vals[pair[k] & 0xffffu] > vals[pair[k] >> 16]);
            emit_feature<PACK, WIN>(*F, l, i, y, theta, words, lane);
            __syncwarp();  // the values are rewritten for the next keypoint
        }
    }
}

// --------------------------------------------- K2 over staged tiles ----
// The same orientation and descriptor as k_describe, with the blur-cache
// samples read from shared memory: one CTA per item = (frame, level, 32-row
// band, chunk of KDT_CW columns).  One 2D TMA load stages the box of the
// blur cache that every test of the item's keypoints can reach (rows
// y0 - R .. y0 + 31 + R, columns x0 - RX .. x0 + KDT_CW - 1 + RX, R = margin
// - 1 >= the largest rotated test offset, RX = R rounded up to 4 so the box
// starts on a 16-byte boundary); cells at negative coordinates get the
// sentinel values the gather path reads for them.  The item's keypoints are
// those of the band's list range (the band order of the compaction) with x
// in the chunk, taken in rounds of up to KDT_THREADS.
constexpr int KDT_THREADS = 256;
constexpr int KDT_WARPS = KDT_THREADS / 32;

template <bool PACK, bool WIN>
__global__ void __launch_bounds__(KDT_THREADS)
k_describe_tiled(const FrameDev* __restrict__ frames, const BandItem* __restrict__ items,
                 const int32_t* __restrict__ pattern, uint32_t* err) {
    extern __shared__ __align__(128) float s_box[];  // [BH][BW] blur-cache box
    __shared__ float4 s_pat[256];
    __shared__ uint32_t s_list[KDT_THREADS];
    __shared__ uint32_t s_wcount[KDT_WARPS];
    __shared__ uint32_t s_pos[2];
    __shared__ __align__(8) uint64_t s_bar;
    constexpr int8_t kdx[29] = {0, -2, -1, 0, 1, 2, -2, -1, 0, 1, 2, -3, -2, -1, 0, 1, 2, 3, -2, -1, 0, 1, 2, -2, -1, 0, 1, 2, 0};
    constexpr int8_t kdy[29] = {-3, -2, -2, -2, -2, -2, -1, -1, -1, -1, -1, 0, 0, 0, 0, 0, 0, 0, 1, 1, 1, 1, 1, 2, 2, 2, 2, 2, 3};
    const BandItem it = items[blockIdx.x];
    const FrameDev& F = frames[it.frame];
    const int l = it.level, band = it.band;
    const int w = F.w[l], h = F.h[l], M = F.margin;
    const int R = M - 1, RX = (R + 3) & ~3;
    const int BW = KDT_CW + 2 * RX, BH = 32 + 2 * R;
    const int x0 = (int)it.pad2 * KDT_CW, y0 = band * 32;
    const int xs = x0 - RX, ys = y0 - R;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    // the band's range of the level's list: after the kept counts of the
    // earlier bands, clipped by the level's kept count (the cap); the box is
    // loaded only for a band that keeps keypoints
    if (warp == 0) {
        uint32_t pk = 0;
        for (int q = lane; q < band; q += 32) pk += F.bands[l][2 * q + 1];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) pk += __shfl_xor_sync(0xffffffffu, pk, o);
        if (lane == 0) {
            const uint32_t kept = F.kept[l];
            const uint32_t b0 = min(pk, kept), b1 = min(pk + F.bands[l][2 * band + 1], kept);
            s_pos[0] = b0;
            s_pos[1] = b1;
            if (b1 > b0) {
                const void* tmap = static_cast<const char*>(F.tmaps) +
                                   (size_t)(l * USLAM_TMAPS_PER_LEVEL + USLAM_NUM_TILE_SHAPES) * USLAM_TMAP_BYTES;
                mbar_init(&s_bar, 1u);
                mbar_expect_tx(&s_bar, (uint32_t)(BW * BH * 4));
                tma_load_2d(s_box, tmap, xs, ys, &s_bar);
            }
        }
    }
    __syncthreads();  // range, barrier initialised
    if (s_pos[1] <= s_pos[0]) return;  // no keypoint in the band: nothing loaded
    // while the box is in flight: the pattern, the selection and the
    // orientations of the first round (they read the level, not the box)
    for (int i = t; i < 256; i += KDT_THREADS) {
        s_pat[i] = make_float4((float)pattern[4 * i], (float)pattern[4 * i + 1], (float)pattern[4 * i + 2],
                               (float)pattern[4 * i + 3]);
    }
    const uint32_t pos0 = s_pos[0], pos1 = s_pos[1];
    const uint32_t* feats = F.feats[l];
    bool box_ready = false;
    for (uint32_t base = pos0; base < pos1; base += KDT_THREADS) {
        // this pass's keypoints with x in the chunk, in list order
        const uint32_t i = base + (uint32_t)t;
        bool sel = false;
        if (i < pos1) {
            const int x = (int)__uint_as_float(__ldg(feats + (size_t)i * 12u));
            sel = x >= x0 && x < x0 + KDT_CW;
        }
        const uint32_t bal = __ballot_sync(0xffffffffu, sel);
        if (lane == 0) s_wcount[warp] = (uint32_t)__popc(bal);
        __syncthreads();  // also the pattern of the first round
        uint32_t off = 0, nsel = 0;
        for (int q = 0; q < KDT_WARPS; ++q) {
            off += q < warp ? s_wcount[q] : 0u;
            nsel += s_wcount[q];
        }
        if (sel) s_list[off + (uint32_t)__popc(bal & ((1u << lane) - 1u))] = i;
        __syncthreads();
        // warp q takes G consecutive keypoints of the list (G <= 32); lane j
        // first computes the orientation of keypoint j
        const uint32_t G = (nsel + KDT_WARPS - 1) / KDT_WARPS;
        const uint32_t g0 = (uint32_t)warp * G;
        const int nk = (int)min(G, nsel > g0 ? nsel - g0 : 0u);
        float my_theta = 0.0f, my_s = 0.0f, my_c = 0.0f;
        if (lane < nk) {
            // orientation (generate_features.wgsl:80-99): intensity moments over
            // the r = 3 disc, summed in the reference's order, then atan2
            const uint32_t* rec = feats + (size_t)s_list[g0 + lane] * 12u;
            const int x = (int)__uint_as_float(rec[0]);
            const int y = (int)__uint_as_float(rec[1]);
            const float* lvl = F.lvl[l];
            const int lp = F.lvl_pitch[l];
            float m10 = 0.0f, m01 = 0.0f;
#pragma unroll
            for (int k = 0; k < 29; ++k) {
                const int cx = tint_clamp(x + kdx[k], w);
                const int cy = tint_clamp(y + kdy[k], h);
                const float v = __ldg(lvl + (size_t)cy * (size_t)lp + cx);
                m10 = m10 + (float)kdx[k] * v;
                m01 = m01 + (float)kdy[k] * v;
            }
            my_theta = uslam_atan2f(m01, m10);
            uslam_sincosf(my_theta, &my_s, &my_c);
        }
        if (!box_ready) {
            // the box has landed; cells at negative coordinates get the
            // sentinel column (x = w + M) / row (y = h + M) that every
            // negative coordinate reads
            const bool landed = mbar_wait(&s_bar, 0u, kTmaWaitLimit);
            if (__syncthreads_or(!landed)) {
                if (t == 0) atomicOr(err, USLAM_ERR_TMA_TIMEOUT);
                mbar_wait(&s_bar, 0u, kTmaWaitLimit);  // the copy in flight lands before the box is left
                return;
            }
            if (xs < 0 || ys < 0) {
                const float* blur = F.blur[l];
                const int bp = F.bl_pitch[l];
                const int nx = max(-xs, 0), ny = max(-ys, 0);
                const int n = ny * BW + (BH - ny) * nx;
                for (int k = t; k < n; k += KDT_THREADS) {
                    int r, c;
                    if (k < ny * BW) {
                        r = k / BW;
                        c = k - r * BW;
                    } else {
                        const int q = k - ny * BW;
                        r = ny + q / nx;
                        c = q - (q / nx) * nx;
                    }
                    const int gy = ys + r, gx = xs + c;
                    if (gy > h + M || gx > w + M) continue;  // past the cache: never read by a test
                    s_box[r * BW + c] = blur[(size_t)(gy < 0 ? h + M : gy) * bp + (gx < 0 ? w + M : gx)];
                }
                __syncthreads();
            }
            box_ready = true;
        }
        for (int kp = 0; kp < nk; ++kp) {
            const uint32_t i2 = s_list[g0 + kp];
            const float theta = __shfl_sync(0xffffffffu, my_theta, kp);
            const float sn = __shfl_sync(0xffffffffu, my_s, kp);
            const float cs = __shfl_sync(0xffffffffu, my_c, kp);
            const uint32_t* rec = feats + (size_t)i2 * 12u;
            const int x = (int)__uint_as_float(rec[0]);
            const int y = (int)__uint_as_float(rec[1]);
            // 256 tests, lane j owns tests j, j + 32, ..., j + 224: 16 reads of
            // the staged box at (y + dy - ys, x + dx - xs)
            const float* org = s_box + (y - ys) * BW + (x - xs);
            float ga[8], gb[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float4 tp = s_pat[lane + 32 * k];
                const int xa = (int)rintf(tp.x * cs - tp.y * sn);
                const int ya = (int)rintf(tp.x * sn + tp.y * cs);
                const int xb = (int)rintf(tp.z * cs - tp.w * sn);
                const int yb = (int)rintf(tp.z * sn + tp.w * cs);
                ga[k] = org[ya * BW + xa];
                gb[k] = org[yb * BW + xb];
            }
            uint32_t words[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) words[k] = __ballot_sync(0xffffffffu, ga[k] > gb[k]);
            emit_feature<PACK, WIN>(F, l, i2, y, theta, words, lane);
        }
        __syncthreads();  // s_list / s_wcount reused by the next pass
    }
    if (!box_ready) mbar_wait(&s_bar, 0u, kTmaWaitLimit);  // no keypoint in the chunk: the load lands first
}

// Dynamic shared memory of k_describe_tiled for a blur-cache margin M (0 if
// the box would exceed a TMA box's 256 cells per dimension).
size_t describe_tiled_smem(int margin) {
    const int R = margin - 1, RX = (R + 3) & ~3;
    const int BW = KDT_CW + 2 * RX, BH = 32 + 2 * R;
    if (R < 0 || BW > 256 || BH > 256) return 0;
    return (size_t)BW * (size_t)BH * 4u;
}

// One three-input logic operation; LUT: its value where the inputs are the
// bits of 0xf0, 0xcc, 0xaa.  Written out: with shared terms such as x ^ y in a
// sum and its carry the compiler keeps the term and needs an operation more.
template <int LUT>
__device__ __forceinline__ uint32_t lop3(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(a), "r"(b), "r"(c), "n"(LUT));
    return d;
}

// ------------------------------------------------- Hamming distance ----
// popcount(a ^ b) over 256 bits with 4 POPC instead of 8: with x = a ^ b, three
// carry-save adders fold x0..x6 into ones (o3) and twos (t1, t2, t3), a fourth
// folds the twos into twos (tw) and fours (f); x7 is added as ones.  Per bit
// position x0 + .. + x7 = o3 + x7 + 2 tw + 4 f, so the sum of the weighted
// popcounts is the exact distance (integer arithmetic, no rounding).
// 13 logic operations: both descriptors are in the form of parity_words, whose
// third inputs are replaced by the sums of words, so that the adders' sums o1,
// o2, o3 are differences of words, and a carry is taken from two inputs and
// the sum (x y | (x ^ y) ~o).  The weighted sum runs on the multiply-add pipe:
// two is 2 in a register the compiler does not see through (of a constant it
// makes shifted adds, which run on the ALU pipe beside the logic).
__device__ __forceinline__ void parity_words(uint4& d0, uint4& d1) {
    d0.z = d0.x ^ d0.y ^ d0.z;
    d1.x = d0.z ^ d0.w ^ d1.x;
    d1.z = d1.x ^ d1.y ^ d1.z;
}
__device__ __forceinline__ uint32_t hamming256_parity(const uint4& a0, const uint4& a1, const uint4& b0, const uint4& b1,
                                                      uint32_t two, uint32_t one) {
    const uint32_t x0 = a0.x ^ b0.x, x1 = a0.y ^ b0.y, o1 = a0.z ^ b0.z, x3 = a0.w ^ b0.w;
    const uint32_t o2 = a1.x ^ b1.x, x5 = a1.y ^ b1.y, o3 = a1.z ^ b1.z, x7 = a1.w ^ b1.w;
    const uint32_t t1 = lop3<0xd4>(x0, x1, o1), t2 = lop3<0xd4>(o1, x3, o2), t3 = lop3<0xd4>(o2, x5, o3);
    const uint32_t tw = lop3<0x96>(t1, t2, t3), f = lop3<0xe8>(t1, t2, t3);
    const uint32_t hi = (uint32_t)__popc(f) * two + (uint32_t)__popc(tw);
    return (uint32_t)__popc(x7) * one + (hi * two + (uint32_t)__popc(o3));
}

// ------------------------------------------------------------- K3 ----
constexpr int KM_THREADS = 256;
// k_match CTAs resident per SM: registers up to 85 a thread (no spills);
// measured faster than 4 CTAs at 64 registers (0.584 against 0.633 ms on
// the 64-frame step) and than 2 at 128.
constexpr int KM_CTAS_PER_SM = 3;
constexpr uint32_t KM_UNITS_PER_WARP = 4, KM_MAX_CHUNKS = 8;

struct MatchSegDev {
    int pair;
    int dir;    // tensor-core form: 0 queries = curr (b), pool = prev (a); 1 the reverse.
                // k_match searches both directions from the prev queries and ignores it.
    int level;
};

__device__ __forceinline__ float lod_scale(int lod) {
    float s = 1.0f;  // match_features_cpu.cpp:58-64
    for (int i = 0; i < lod; ++i) s = s * 1.2f;
    return s;
}

// First xb in [0, w] with (float)xb * s >= lo (w if none).
__device__ int first_col_ge(float lo, float s, int w) {
    int xb = (int)fminf(fmaxf(floorf(lo / s) - 1.0f, 0.0f), (float)w);
    while (xb > 0 && (float)(xb - 1) * s >= lo) --xb;
    while (xb < w && !((float)xb * s >= lo)) ++xb;
    return xb;
}

// Last xb in [-1, w - 1] with (float)xb * s <= hi (-1 if none).
__device__ int last_col_le(float hi, float s, int w) {
    int xb = (int)fminf(fmaxf(floorf(hi / s) + 1.0f, -1.0f), (float)(w - 1));
    while (xb < w - 1 && (float)(xb + 1) * s <= hi) ++xb;
    while (xb >= 0 && !((float)xb * s <= hi)) --xb;
    return xb;
}

// First xb in [0, w] with fl(fl(xb * s) + d) >= c (w if none): the first
// column of a list whose features have LOD-0 x = c inside their own window
// (the b -> a test of match_features_cpu.cpp:106-115 seen from a).
__device__ int first_col_reach(float c, float d, float s, int w) {
    int xb = (int)fminf(fmaxf(floorf((c - d) / s) - 1.0f, 0.0f), (float)w);
    while (xb > 0 && (float)(xb - 1) * s + d >= c) --xb;
    while (xb < w && !((float)xb * s + d >= c)) ++xb;
    return xb;
}

// Last xb in [-1, w - 1] with fl(fl(xb * s) - d) <= c (-1 if none).
__device__ int last_col_reach(float c, float d, float s, int w) {
    int xb = (int)fminf(fmaxf(floorf((c + d) / s) + 1.0f, -1.0f), (float)(w - 1));
    while (xb < w - 1 && (float)(xb + 1) * s - d <= c) ++xb;
    while (xb >= 0 && !((float)xb * s - d <= c)) --xb;
    return xb;
}

// Lane-wise minimum / maximum of two 16-bit keys per word.
__device__ __forceinline__ uint32_t min_u16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// Byte i = eight copies of the sign bit of byte (SEL >> 4 i) & 7 (the
// selector's upper bit asks for the sign; the __byte_perm function drops it).
template <int SEL>
__device__ __forceinline__ uint32_t byte_signs(uint32_t v) {
    static_assert((SEL & 0x8888) == 0x8888, "signs");
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(v), "n"(SEL));
    return r;
}
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// One warp's staging area: 32 candidates (LOD-0 y, packed (level, index),
// descriptor halves), the packed (level, index) of each lane's query, and the
// batch's column keys, two candidates in a word: halves 2 p and 2 p + 1 of
// col[p * 32 + lane] = distance << 5 | lane where lane's query meets candidate
// 2 p (2 p + 1), all ones otherwise.
struct CandBuf {
    float py[32];
    int32_t idx[32];
    uint4 d0[32], d1[32];
};
struct CandStage {
    CandBuf buf[2];
    uint32_t qid[32];
    uint32_t col[16 * 32];
};
constexpr int KM_MAX_SEGS = USLAM_MAX_MATCH_SEGS;

__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
                 "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Query groups of one (pair, level) segment: groups of 32 queries of the
// previous set, per band of its query order.
__device__ __forceinline__ uint32_t match_groups(const FrameDev* frames, const PairDev* pairs, const MatchSegDev& sg) {
    const FrameDev& Qf = frames[pairs[sg.pair].prev];
    const int ql = sg.level;
    const int nb = Qf.nbands;
    const uint32_t* qb = Qf.colstart[ql] + (size_t)nb * (size_t)(Qf.w[ql] + 1);
    uint32_t n = 0;
    for (int b = 0; b < nb; ++b) n += (qb[b + 1] - qb[b] + 31u) / 32u;
    return n;
}

// Band of group grp of a segment (grp becomes the group within the band).
__device__ __forceinline__ int match_group_band(const uint32_t* qband, int nb, uint32_t* grp) {
    int band = 0;
    while (band + 1 < nb && *grp >= (qband[band + 1] - qband[band] + 31u) / 32u) {
        *grp -= (qband[band + 1] - qband[band] + 31u) / 32u;
        ++band;
    }
    return band;
}

// The windowed mutual matcher (match_features_cpu.cpp:66-207), one Hamming
// distance per pair of features.  Both directions of FindMatches compare the
// same pairs: b in the window of a (a -> b, pool = the levels l - 1 .. l + 1
// of the current set) and a in the window of b (b -> a).  So the queries of a
// launch are the previous set's features alone, and every distance feeds
// both searches:
//  * a warp takes 32 queries a of one band that are consecutive in x (from
//    the query level's x order) and streams the union of their windows, level
//    by level of the pool, through shared memory, 32 candidates at a time
//    (asynchronous copies, one batch ahead);
//  * per lane two exact index ranges of the x-ordered list: [m0, m1), the b
//    inside a's window, and [n0, n1), the b whose window holds a (the same
//    features except where f32 rounding at the window's x edge differs);
//    the y test |ya - yb| <= 0.1 H0 is the same both ways;
//  * a lane takes the distances to all candidates of the batch (about half of
//    them are hits: picking those out, each lane its own, took more
//    instructions and the shared memory's time in bank conflicts), two to a
//    word with all ones in place of the others; it keeps a's two smallest keys
//    (distance << 5 | slot) in registers and writes the keys distance << 5 |
//    lane to the candidate's column; after the batch lane t folds column t
//    into b's two smallest and merges them into b's accumulator in HBM (atomic minimum of
//    (distance, packed a), then of the second distance), where the batches
//    of every query group that meets b meet;
//  * a's search is merged into its own accumulator the same way when its
//    units end; k_mutual reads both accumulators.
// The logic and popcount pipes bound it (ALU 68 %, XU 47 %, shared memory 43 %
// busy); 32 pairs of 752x480 frames: 318 us picking hits, 283 us so.
// A tied best leaves the second distance equal to the best, which fails the
// ratio test, so no result depends on the order of the candidates or of the
// merges.  The pool rule (fewer than two candidates: no match) is applied in
// k_mutual (to a here where a2b is written).
template <bool PARTS>
__global__ void __launch_bounds__(KM_THREADS, KM_CTAS_PER_SM)
k_match(const FrameDev* __restrict__ frames, const PairDev* __restrict__ pairs,
        const MatchSegDev* __restrict__ segs, int nseg, uint32_t* next_unit, uint32_t two) {
    __shared__ uint32_t s_pref[KM_MAX_SEGS + 1];
    __shared__ uint32_t s_warp[33];
    __shared__ __align__(16) CandStage s_stage[KM_THREADS / 32];
    // work units: groups of 32 queries of one band (band offsets follow the
    // query level's column tables)
    const uint32_t total =
        segment_prefix(nseg, s_pref, s_warp, [&](int s) { return match_groups(frames, pairs, segs[s]); });
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int gw = blockIdx.x * (KM_THREADS / 32) + warp;
    const int nw = gridDim.x * (KM_THREADS / 32);
    CandStage& S = s_stage[warp];
    const uint32_t one = two >> 1, n32 = two << 4, n64k = two << 15;
    // s_first[n]: the bits of the first n candidates of a batch.  Candidate i has
    // bit 8 (i % 4) + 7 - i / 4, so that after q shifts to the left candidates
    // 4 q .. 4 q + 3 have the bytes' signs, which a byte permute spreads.
    __shared__ uint32_t s_first[33];
    if (threadIdx.x < 33) {
        uint32_t m = 0u;
        for (int i = 0; i < (int)threadIdx.x; ++i) m |= 1u << (8 * (i & 3) + 7 - (i >> 2));
        s_first[threadIdx.x] = m;
    }
    __syncthreads();
    // PARTS: a group's search is cut by pool level and then into chunks of its
    // batches, for KM_UNITS_PER_WARP units a warp: a group in one piece takes 20
    // batches on a 752x480 frame, 70 on a 1920x1080 one, 5 to 7 us each, and the
    // groups cost very different amounts.  A warp's first unit is its own,
    // then it claims the next from *next_unit (zero before the launch; without
    // it warps take every nw-th unit).  The units of a group meet in aacc; else
    // a warp has all of a group and writes a2b.  All merging is by atomic
    // minima, so the order does not change the result.
    // One 752x480 / 1920x1080 frame with 1, 2, 4, 6, 8, 16 units a warp: 246, 245,
    // 240, 244, 246, 248 / 600, 620, 554, 544, 554, 572 us.  Whole groups in an
    // order of their cost (two kernels before) took 1438 us for 64 frames, units
    // 1431, the mixed batch 4689 and 4656.
    auto claim = [&](uint32_t c) -> uint32_t {
        if (!next_unit) return c + (uint32_t)nw;
        uint32_t n = 0;
        if (lane == 0) n = atomicAdd(next_unit, 1u);
        return __shfl_sync(0xffffffffu, n, 0) + (uint32_t)nw;
    };
    const uint32_t chunks = PARTS ? min(max((KM_UNITS_PER_WARP * (uint32_t)nw) / max(3u * total, 1u), 1u), KM_MAX_CHUNKS) : 1u;
    const uint32_t units = PARTS ? 3u * chunks * total : total;
    for (uint32_t c = (uint32_t)gw; c < units; c = claim(c)) {
        const uint32_t g = PARTS ? c / (3u * chunks) : c;
        const uint32_t part = PARTS ? c - g * (3u * chunks) : 0u;
        const int sidx = find_segment(s_pref, nseg, g);
        uint32_t grp = g - s_pref[sidx];
        const MatchSegDev sg = segs[sidx];
        const PairDev& P = pairs[sg.pair];
        const FrameDev& Q = frames[P.prev];
        const FrameDev& B = frames[P.curr];
        const int l = sg.level;
        const uint32_t* qband = Q.colstart[l] + (size_t)Q.nbands * (size_t)(Q.w[l] + 1);
        const int band = match_group_band(qband, Q.nbands, &grp);
        const uint32_t qk = qband[band] + grp * 32u + (uint32_t)lane;
        const bool valid = qk < qband[band + 1];
        const uint32_t qi = valid ? __ldg(Q.qorder[l] + qk) : 0u;
        const uint32_t* qrec = Q.feats[l] + (size_t)qi * 12u;
        const float ql = lod_scale(l);
        const float cx = (float)(uint32_t)__uint_as_float(qrec[0]) * ql;
        const float cy = (float)(uint32_t)__uint_as_float(qrec[1]) * ql;
        uint4 qd0 = *reinterpret_cast<const uint4*>(qrec + 4);
        uint4 qd1 = *reinterpret_cast<const uint4*>(qrec + 8);
        parity_words(qd0, qd1);
        const float dx = P.max_dx, dy = P.max_dy;
        const float lo = cx - dx, hi = cx + dx;
        S.qid[lane] = (uint32_t)USLAM_PACK(l, qi);
        __syncwarp();

        // a's best / second-best as 16-bit keys (distance << 5 | slot); a tie on the
        // best distance leaves second >> 5 == best >> 5, which fails the test
        uint32_t bestk = 0xffffu, secondk = 0xffffu;
        int32_t bidx = -1;
        const int L = B.levels;
        uint4* const bacc = P.bacc;
        const size_t capb = (size_t)(B.cap > 0 ? B.cap : 1);
        uint32_t* const colq = S.col + lane;
        const uint32_t lanes = (uint32_t)lane * 0x10001u;
        for (int k = PARTS ? (int)(part / chunks) : 0; k < 3; k = PARTS ? 3 : k + 1) {
            const int pl = k == 0 ? l : (k == 1 ? l - 1 : l + 1);
            if (pl < 0 || pl >= L) continue;
            const float ps = lod_scale(pl);
            const int wpl = B.w[pl];
            // the pool's candidate list of this band
            const uint32_t* colstart = B.colstart[pl] + (size_t)band * (size_t)(wpl + 1);
            uint32_t m0 = 0u, m1 = 0u, n0 = 0u, n1 = 0u;
            if (valid) {
                int xlo = first_col_ge(lo, ps, wpl), xhi = last_col_le(hi, ps, wpl);
                if (xlo <= xhi) {
                    m0 = __ldg(colstart + xlo);
                    m1 = __ldg(colstart + xhi + 1);
                }
                xlo = first_col_reach(cx, dx, ps, wpl);
                xhi = last_col_reach(cx, dx, ps, wpl);
                if (xlo <= xhi) {
                    n0 = __ldg(colstart + xlo);
                    n1 = __ldg(colstart + xhi + 1);
                }
            }
            // union over both ranges and the warp (lanes are x-sorted, so it is contiguous)
            uint32_t c0 = min(m0 < m1 ? m0 : 0xffffffffu, n0 < n1 ? n0 : 0xffffffffu);
            uint32_t c1 = max(m0 < m1 ? m1 : 0u, n0 < n1 ? n1 : 0u);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                c0 = min(c0, __shfl_xor_sync(0xffffffffu, c0, o));
                c1 = max(c1, __shfl_xor_sync(0xffffffffu, c1, o));
            }
            if (c0 >= c1) continue;
            if (PARTS) {
                const uint32_t nb = (c1 - c0 + 31u) / 32u, ch = part % chunks;
                const uint32_t from = c0 + 32u * (ch * nb / chunks), to = c0 + 32u * ((ch + 1u) * nb / chunks);
                c1 = min(c1, to);
                c0 = from;
                if (c0 >= c1) continue;
            }
            const uint32_t* xorder = B.xorder[pl] + (size_t)band * (size_t)(B.cap > 0 ? B.cap : 1);
            const uint32_t* feats = B.feats[pl];
            // Candidates are staged by asynchronous copies one batch ahead,
            // into two buffers: batch i + 1's copies are issued before batch i
            // is used, and batch i + 2's list entry is loaded meanwhile.
            uint32_t jn = 0u;  // list entry of this lane's slot in the next batch
            {
                // prologue: batch 0 in flight, batch 1's list entry in hand
                const uint32_t k0 = c0 + (uint32_t)lane;
                if (k0 < c1) {
                    const uint32_t j = __ldg(xorder + k0);
                    const uint32_t* rec = feats + (size_t)j * 12u;
                    CandBuf& N = S.buf[0];
                    cp_async4(&N.py[lane], rec + 1);
                    cp_async16(&N.d0[lane], rec + 4);
                    cp_async16(&N.d1[lane], rec + 8);
                    N.idx[lane] = USLAM_PACK(pl, j);
                }
                cp_async_commit();
                if (k0 + 32u < c1) jn = __ldg(xorder + k0 + 32u);
            }
            int cur = 0;
            for (uint32_t base = c0; base < c1; base += 32u, cur ^= 1) {
                const uint32_t kk = base + (uint32_t)lane;
                CandBuf& SB = S.buf[cur];
                {
                    // the next batch's copies go out before this batch is used
                    const uint32_t kn = kk + 32u;
                    if (kn < c1) {
                        const uint32_t* rec = feats + (size_t)jn * 12u;
                        CandBuf& N = S.buf[cur ^ 1];
                        cp_async4(&N.py[lane], rec + 1);
                        cp_async16(&N.d0[lane], rec + 4);
                        cp_async16(&N.d1[lane], rec + 8);
                        N.idx[lane] = USLAM_PACK(pl, jn);
                    }
                    cp_async_commit();
                    if (kn + 32u < c1) jn = __ldg(xorder + kn + 32u);
                    cp_async_wait<1>();
                    // the staged word is the record's f32 y; the LOD-0 y as in
                    // match_features_cpu.cpp:58-64
                    if (kk < c1) {
                        SB.py[lane] = (float)(uint32_t)SB.py[lane] * ps;
                        uint4 d0 = SB.d0[lane], d1 = SB.d1[lane];
                        parity_words(d0, d1);
                        SB.d0[lane] = d0;
                        SB.d1[lane] = d1;
                    }
                }
                __syncwarp();
                // |ya - yb| > dy of all 32 staged candidates, as the sign of
                // dy - |ya - yb| (exact) shifted in: one ALU operation each.
                // Candidates past the list's end lie outside both ranges.
                uint32_t f0 = 0u, f1 = 0u, f2 = 0u, f3 = 0u;
                const float4* py4 = reinterpret_cast<const float4*>(SB.py);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float4 v = py4[q];
                    f0 = __funnelshift_l(__float_as_uint(dy - fabsf(cy - v.x)), f0, 1);
                    f1 = __funnelshift_l(__float_as_uint(dy - fabsf(cy - v.y)), f1, 1);
                    f2 = __funnelshift_l(__float_as_uint(dy - fabsf(cy - v.z)), f2, 1);
                    f3 = __funnelshift_l(__float_as_uint(dy - fabsf(cy - v.w)), f3, 1);
                }
                const uint32_t far = __byte_perm(__byte_perm(f0, f1, 0x0040), __byte_perm(f2, f3, 0x0040), 0x5410);
                auto first = [&](uint32_t upto) { return s_first[min(max(upto, base) - base, 32u)]; };
                // candidates that are no hit: b outside a's window, a outside b's
                uint32_t no1 = ~first(m1) | first(m0) | far, no0 = ~first(n1) | first(n0) | far;
                uint32_t b2 = 0xffffffffu, s2 = 0xffffffffu, slots = 0x10000u;
                const int quads = (int)(min(c1 - base, 32u) + 3u) >> 2;
#pragma unroll 1
                for (int q = 0; q < quads; ++q) {
                    const uint4 *p0 = SB.d0 + 4 * q, *p1 = SB.d1 + 4 * q;
                    const uint32_t dA = hamming256_parity(p0[1], p1[1], qd0, qd1, two, one) * n64k +
                                        hamming256_parity(p0[0], p1[0], qd0, qd1, two, one);
                    const uint32_t dB = hamming256_parity(p0[3], p1[3], qd0, qd1, two, one) * n64k +
                                        hamming256_parity(p0[2], p1[2], qd0, qd1, two, one);
                    const uint32_t rA = (dA * n32 + slots) | byte_signs<0x9988>(no1);
                    const uint32_t rB = (dB * n32 + (slots + 0x20002u)) | byte_signs<0xbbaa>(no1);
                    s2 = min_u16x2(s2, max_u16x2(b2, rA));
                    b2 = min_u16x2(b2, rA);
                    s2 = min_u16x2(s2, max_u16x2(b2, rB));
                    b2 = min_u16x2(b2, rB);
                    colq[64 * q] = (dA * n32 + lanes) | byte_signs<0x9988>(no0);
                    colq[64 * q + 32] = (dB * n32 + lanes) | byte_signs<0xbbaa>(no0);
                    no1 += no1;
                    no0 += no0;
                    slots += 0x40004u;
                }
                {
                    const uint32_t bl = b2 & 0xffffu, bh = b2 >> 16, bb = min(bl, bh);
                    const uint32_t ss = min(max(bl, bh), min(s2 & 0xffffu, s2 >> 16));
                    secondk = min(min(secondk, ss), max(bestk, bb));
                    if (bb < bestk) {
                        bestk = bb;
                        bidx = SB.idx[bb & 31u];
                    }
                }
                __syncwarp();
                // column pass: lanes 2 p and 2 p + 1 fold a half of the queries' keys of
                // candidates 2 p and 2 p + 1 into the two smallest each, and
                // lane t merges candidate t's into b's accumulator
                {
                    const uint4* colt = reinterpret_cast<const uint4*>(S.col + 16 * lane);
                    b2 = s2 = 0xffffffffu;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint4 v = colt[(q + (lane >> 1)) & 3];  // no two lanes of a quarter warp in one bank
                        s2 = min_u16x2(s2, max_u16x2(b2, v.x));
                        b2 = min_u16x2(b2, v.x);
                        s2 = min_u16x2(s2, max_u16x2(b2, v.y));
                        b2 = min_u16x2(b2, v.y);
                        s2 = min_u16x2(s2, max_u16x2(b2, v.z));
                        b2 = min_u16x2(b2, v.z);
                        s2 = min_u16x2(s2, max_u16x2(b2, v.w));
                        b2 = min_u16x2(b2, v.w);
                    }
                    const uint32_t ob = __shfl_xor_sync(0xffffffffu, b2, 1), os = __shfl_xor_sync(0xffffffffu, s2, 1);
                    s2 = min_u16x2(min_u16x2(s2, os), max_u16x2(b2, ob));
                    b2 = min_u16x2(b2, ob);
                    const uint32_t cb = lane & 1 ? b2 >> 16 : b2 & 0xffffu, cs = lane & 1 ? s2 >> 16 : s2 & 0xffffu;
                    if (kk < c1 && cb != 0xffffu) {
                        const unsigned long long key =
                            ((unsigned long long)(cb >> 5) << 32) | (unsigned long long)S.qid[cb & 31u];
                        const int32_t id = SB.idx[lane];
                        uint4* acc = bacc + (size_t)USLAM_PACK_LEVEL(id) * capb + (size_t)USLAM_PACK_INDEX(id);
                        const unsigned long long old = atomicMin(reinterpret_cast<unsigned long long*>(acc), key);
                        // the larger of the old best and this best joins the
                        // second-best candidates
                        const uint32_t lose = (uint32_t)((old > key ? old : key) >> 32);
                        atomicMin(&acc->z, min(lose, cs == 0xffffu ? 0xffffffffu : cs >> 5));
                    }
                }
                __syncwarp();
            }
        }
        if (PARTS && bidx >= 0) {
            uint4* acc = P.aacc + (size_t)l * Q.cap + qi;
            const unsigned long long key = ((unsigned long long)(bestk >> 5) << 32) | (unsigned long long)(uint32_t)bidx;
            const unsigned long long old = atomicMin(reinterpret_cast<unsigned long long*>(acc), key);
            atomicMin(&acc->z, min((uint32_t)((old > key ? old : key) >> 32), secondk == 0xffffu ? 0xffffffffu : secondk >> 5));
        }
        if (!PARTS && valid) {
            uint32_t pool = B.kept[l];
            if (l > 0) pool += B.kept[l - 1];
            if (l + 1 < L) pool += B.kept[l + 1];
            int32_t res = -1;
            if (pool >= 2u && bidx >= 0 && (float)(bestk >> 5) < 0.85f * (float)(secondk >> 5)) res = bidx;
            P.a2b[(size_t)l * Q.cap + qi] = res;
        }
    }
}

// The accumulators start empty (all ones) before every k_match launch: one
// CTA per (pair, level).
__global__ void __launch_bounds__(256)
k_bacc_init(const FrameDev* __restrict__ frames, const PairDev* __restrict__ pairs, const SegDev* __restrict__ segs) {
    const int pi = segs[blockIdx.x].frame;  // pair index
    const int l = segs[blockIdx.x].level;
    const PairDev& P = pairs[pi];
    auto empty = [&](uint4* all, const FrameDev& F) {
        uint4* acc = all + (size_t)l * (size_t)(F.cap > 0 ? F.cap : 1);
        for (uint32_t i = threadIdx.x; i < F.kept[l]; i += blockDim.x) acc[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    };
    empty(P.bacc, frames[P.curr]);
    if (P.aacc) empty(P.aacc, frames[P.prev]);
}

// ----------------------------------------------------- brute force ----
constexpr int KB_THREADS = 64;
constexpr int KB_CTAS = 512 / KB_THREADS;  // per SM
constexpr int KB_PAIRS = 2;      // pairs of queries per thread: 256 queries per CTA
constexpr int KB_Q = 2 * KB_PAIRS;
constexpr int KB_TILE = 128;     // train descriptors per shared-memory tile
static_assert(256 * KB_TILE + KB_TILE - 1 < 0xffff, "distance and tile slot share 16 bits");

// Level of flat index f given the per-level prefix pre[0..L] (pre[L] = total).
__device__ __forceinline__ int flat_level(const uint32_t* pre, int L, uint32_t f) {
    int l = 0;
    while (l + 1 < L && pre[l + 1] <= f) ++l;
    return l;
}

// Brute-force top-2 matching (the benchmark's `cfg` matcher): every feature
// of frame prev (all levels) against every feature of frame curr, Lowe test
// best < ratio * second in f32, no window and no cross-check.  One CTA holds
// 256 queries in registers, four a thread, and streams the train set through
// shared memory in tiles of 128 descriptors.  A tied best fails the ratio
// test, so the result does not depend on the scan order; a train set of fewer
// than two features gives no match (the pool rule of
// match_features_cpu.cpp:80-82).
// Result per query a in a2b: packed (level, index) of its match in curr, or
// -1; or one record per part of a cut block (bf_line.h).
//
// The ALU and popcount pipes bound it (71 and 76 % busy).  So: descriptors as
// parity_words (13 logic operations and 4 popcounts a distance), weighted sums
// by multiply-add, and two queries' keys of 16 bits in a word, which min and
// max take together.  15 pairs of 8200 x 8200: 1.59 ms before, 1.05 now, 0.97 T
// distances/s; four queries a thread measured 8 % faster than two, tiles of 64
// or CTAs of 32 or 128 threads 1 to 3 % slower.
__global__ void __launch_bounds__(KB_THREADS, KB_CTAS)
k_bruteforce(const FrameDev* __restrict__ frames, const PairDev* __restrict__ pairs, const SegDev* __restrict__ psegs,
             int npairs, float ratio, uint32_t two) {
    extern __shared__ unsigned long long s_pref[];  // npairs + 1
    __shared__ unsigned long long s_warp[KB_THREADS / 32];
    __shared__ uint4 s_d[2 * KB_TILE];
    __shared__ int32_t s_id[KB_TILE];
    __shared__ uint32_t s_qpre[USLAM_MAX_LEVELS + 1], s_tpre[USLAM_MAX_LEVELS + 1];
    const int tid = threadIdx.x;
    const uint32_t one = two >> 1, two16 = two << 15, tile = two * (uint32_t)(KB_TILE / 2);
    BfLine line = bf_line<KB_Q * KB_THREADS, KB_TILE>(frames, pairs, psegs, npairs, s_pref, s_warp);
    BfUnit u;
    while (bf_next<KB_Q * KB_THREADS, KB_TILE>(frames, pairs, psegs, npairs, s_pref, line, u)) {
        const PairDev& P = *u.P;
        const uint32_t blk = u.blk;
        const FrameDev& A = frames[P.prev];
        const FrameDev& B = frames[P.curr];
        const int LA = A.levels, LB = B.levels;
        if (tid == 0) {
            uint32_t ra = 0, rb = 0;
            for (int l = 0; l <= USLAM_MAX_LEVELS; ++l) {
                s_qpre[l] = ra;
                s_tpre[l] = rb;
                if (l < LA) ra += A.kept[l];
                if (l < LB) rb += B.kept[l];
            }
        }
        __syncthreads();
        const uint32_t nq = u.nq, nt = u.nt;
        const bool busy = blk * (uint32_t)(KB_Q * KB_THREADS) + (uint32_t)(KB_Q * (tid & ~31)) < nq;  // the warp has queries
        uint4 q0[KB_Q], q1[KB_Q];
        uint32_t best[KB_PAIRS], second[KB_PAIRS];  // two queries' keys of 16 bits each: distance * KB_TILE + tile slot
        int32_t bidx[KB_Q];
        int ql[KB_Q];
        uint32_t qi[KB_Q];
        bool qv[KB_Q];
#pragma unroll
        for (int k = 0; k < KB_Q; ++k) {
            const uint32_t f = blk * (uint32_t)(KB_Q * KB_THREADS) + (uint32_t)(KB_Q * tid + k);
            qv[k] = f < nq;
            ql[k] = qv[k] ? flat_level(s_qpre, LA, f) : 0;
            qi[k] = qv[k] ? f - s_qpre[ql[k]] : 0u;
            const uint32_t* rec = A.feats[ql[k]] + (size_t)qi[k] * 12u;
            q0[k] = qv[k] ? *reinterpret_cast<const uint4*>(rec + 4) : make_uint4(0, 0, 0, 0);
            q1[k] = qv[k] ? *reinterpret_cast<const uint4*>(rec + 8) : make_uint4(0, 0, 0, 0);
            parity_words(q0[k], q1[k]);
            bidx[k] = -1;
        }
#pragma unroll
        for (int k = 0; k < KB_PAIRS; ++k) best[k] = second[k] = 0xffffffffu;
        const uint32_t t_end = min(nt, (u.tile + u.ntiles) * (uint32_t)KB_TILE);
        for (uint32_t t0 = u.tile * (uint32_t)KB_TILE; t0 < t_end; t0 += KB_TILE) {
            __syncthreads();
            for (int j = tid; j < KB_TILE; j += KB_THREADS) {
                const uint32_t f = t0 + (uint32_t)j;
                if (f < t_end) {
                    const int l = flat_level(s_tpre, LB, f);
                    const uint32_t i = f - s_tpre[l];
                    const uint32_t* rec = B.feats[l] + (size_t)i * 12u;
                    uint4 d0 = __ldg(reinterpret_cast<const uint4*>(rec + 4)), d1 = __ldg(reinterpret_cast<const uint4*>(rec + 8));
                    parity_words(d0, d1);
                    s_d[2 * j] = d0;
                    s_d[2 * j + 1] = d1;
                    s_id[j] = USLAM_PACK(l, i);
                }
            }
            __syncthreads();
            if (!busy) continue;
            const int n = (int)min((uint32_t)KB_TILE, t_end - t0);
            uint32_t prev[KB_PAIRS];
#pragma unroll
            for (int k = 0; k < KB_PAIRS; ++k) prev[k] = best[k];
            uint32_t slot = 0u;  // j in both halves
#pragma unroll 4
            for (int j = 0; j < n; ++j, slot += 0x10001u) {
                const uint4 d0 = s_d[2 * j], d1 = s_d[2 * j + 1];
#pragma unroll
                for (int k = 0; k < KB_PAIRS; ++k) {
                    const uint32_t lo = hamming256_parity(q0[2 * k], q1[2 * k], d0, d1, two, one);
                    const uint32_t hi = hamming256_parity(q0[2 * k + 1], q1[2 * k + 1], d0, d1, two, one);
                    // min/max keep the two smallest distances; a tie leaves
                    // equal distances in best and second
                    const uint32_t key = (hi * two16 + lo) * tile + slot;
                    second[k] = min_u16x2(second[k], max_u16x2(best[k], key));
                    best[k] = min_u16x2(best[k], key);
                }
            }
            // resolve this tile's winners to packed ids before the tile is overwritten
#pragma unroll
            for (int k = 0; k < KB_PAIRS; ++k) {
                const uint32_t diff = best[k] ^ prev[k];
                if (diff & 0xffffu) bidx[2 * k] = s_id[best[k] & (uint32_t)(KB_TILE - 1)];
                if (diff >> 16) bidx[2 * k + 1] = s_id[(best[k] >> 16) & (uint32_t)(KB_TILE - 1)];
            }
        }
#pragma unroll
        for (int k = 0; k < KB_Q; ++k) {
            if (!qv[k]) continue;
            const size_t q = (size_t)ql[k] * A.cap + qi[k];
            // distances; all ones: none
            const uint32_t bk = (best[k / 2] >> (16 * (k & 1))) & 0xffffu, sk = (second[k / 2] >> (16 * (k & 1))) & 0xffffu;
            const uint32_t bd = bk == 0xffffu ? 0xffffffu : bk / KB_TILE, sd = sk == 0xffffu ? 0xffffffu : sk / KB_TILE;
            if (u.parts == 1u && P.bf_part == nullptr) {
                const int32_t res = (nt >= 2u && bidx[k] >= 0 && (float)bd < ratio * (float)sd) ? bidx[k] : -1;
                P.a2b[q] = res;
            } else {
                bf_record(u, (size_t)A.levels * A.cap, q, bd, sd, bidx[k]);
            }
        }
        __syncthreads();  // s_qpre / s_tpre are rewritten by the next work unit
    }
}

// A pair of frames to match where they are: entries 0 and 1 of a frame table
// become a and b, and the run's error word 0.
__global__ void __launch_bounds__(256)
k_take_frames(FrameDev* __restrict__ dst, const FrameDev* __restrict__ a, const FrameDev* __restrict__ b, uint32_t* err) {
    static_assert(sizeof(FrameDev) % 8 == 0, "copied by 8-byte words");
    constexpr int N = (int)(sizeof(FrameDev) / 8);
    for (int i = threadIdx.x; i < 2 * N; i += blockDim.x)
        reinterpret_cast<unsigned long long*>(dst)[i] = reinterpret_cast<const unsigned long long*>(i < N ? a : b)[i < N ? i : i - N];
    if (threadIdx.x == 0) *err = 0u;
}

// ---------------------------------------------------------- mutual ----
constexpr int KU_THREADS = 1024;
constexpr int KU_ITEMS = 8;  // features of a thread in one round

// One CTA per (pair, level of a): keep (a, b) iff b2a[b] == a, in a order
// (match_features_cpu.cpp:196-205).
// MUTUAL = false: every a with a2b[a] >= 0 is emitted (brute-force mode,
// which has no cross-check).
// Latency bounds it: a round looks at 8192 features with all of a thread's
// loads in flight and orders them by one scan of the warps' counts (rounds of
// 256 took 53 us on the largest level of a 1920x1080 frame, 172 on a
// 3840x2160 one).
template <bool MUTUAL>
__global__ void __launch_bounds__(KU_THREADS)
k_mutual(const FrameDev* __restrict__ frames, const PairDev* __restrict__ pairs, const SegDev* __restrict__ segs,
         uint32_t* err, uint32_t* reset_word) {
    constexpr int WARPS = KU_THREADS / 32;
    static_assert(WARPS == 32, "the scan takes a warp per item index and a lane per warp");
    // k_match's unit counter for its next launch on this stream (k_mutual
    // always follows k_match, which has finished with it)
    if (reset_word && blockIdx.x == 0 && threadIdx.x == 0) *reset_word = 0u;
    __shared__ uint32_t s_cnt[KU_ITEMS][WARPS];  // matches per (item index, warp), then those before them in the row
    __shared__ uint32_t s_row[KU_ITEMS];
    const int pi = segs[blockIdx.x].frame;  // pair index
    const int l = segs[blockIdx.x].level;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const PairDev& P = pairs[pi];
    const FrameDev& A = frames[P.prev];
    const FrameDev& B = frames[P.curr];
    const uint32_t n = A.kept[l];
    int32_t* const a2b = P.a2b + (size_t)l * A.cap;
    uint32_t base = 0;
    uint32_t nt = 0;  // the train set of the brute-force matchers
    if (!MUTUAL)
        for (int q = 0; q < B.levels; ++q) nt += B.kept[q];
    for (uint32_t c0 = 0; c0 < n; c0 += KU_THREADS * KU_ITEMS) {
        int32_t m[KU_ITEMS];
        if (MUTUAL && P.aacc) {
            // a's search from its accumulator: the pool rule and the ratio test
            uint32_t pool = B.kept[l];
            if (l > 0) pool += B.kept[l - 1];
            if (l + 1 < B.levels) pool += B.kept[l + 1];
            const uint4* acc = P.aacc + (size_t)l * A.cap;
            uint4 e[KU_ITEMS];
#pragma unroll
            for (int u = 0; u < KU_ITEMS; ++u) {
                const uint32_t i = c0 + u * KU_THREADS + threadIdx.x;
                e[u] = i < n ? acc[i] : make_uint4(~0u, ~0u, ~0u, ~0u);
            }
#pragma unroll
            for (int u = 0; u < KU_ITEMS; ++u)
                m[u] = pool >= 2u && e[u].y != 0xffffffffu && (float)e[u].y < 0.85f * (float)e[u].z ? (int32_t)e[u].x : -1;
        } else if (MUTUAL || P.bf_part == nullptr) {
#pragma unroll
            for (int u = 0; u < KU_ITEMS; ++u) {
                const uint32_t i = c0 + u * KU_THREADS + threadIdx.x;
                m[u] = i < n && (MUTUAL || nt >= 2u) ? a2b[i] : -1;  // nt: the pool rule
            }
        } else {
            // merge the parts of each query's block: the two smallest distances
            // of the union of their (best, second) pairs; a tie on the best
            // leaves second == best, which fails the ratio test.  The records
            // of four items are in flight together.
            const size_t stride = (size_t)A.levels * A.cap;
#pragma unroll
            for (int h = 0; h < KU_ITEMS; h += 4) {
                const uint4* rec[4];
                uint4 e[4];
                uint32_t bd[4], sd[4];
                int32_t bi[4], parts[4], most = 1;
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const uint32_t i = c0 + (h + v) * KU_THREADS + threadIdx.x;
                    const bool any = i < n && nt >= 2u;  // the pool rule; such a pair may have no records
                    rec[v] = reinterpret_cast<const uint4*>(P.bf_part) + (size_t)l * A.cap + (any ? i : 0u);
                    e[v] = any ? *rec[v] : make_uint4(~0u, ~0u, ~0u, 0u);
                }
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    bd[v] = e[v].x >> 8;
                    sd[v] = e[v].y >> 8;
                    bi[v] = (int32_t)e[v].z;
                    parts[v] = min((int)e[v].w, P.bf_splits);
                    most = max(most, parts[v]);
                }
                for (int sp = 1; sp < most; ++sp) {
#pragma unroll
                    for (int v = 0; v < 4; ++v)
                        e[v] = sp < parts[v] ? rec[v][sp * stride] : make_uint4(~0u, ~0u, ~0u, 0u);
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        const uint32_t b = e[v].x >> 8, c = e[v].y >> 8;
                        if (b < bd[v]) {
                            sd[v] = min(bd[v], c);
                            bd[v] = b;
                            bi[v] = (int32_t)e[v].z;
                        } else {
                            sd[v] = min(sd[v], b);
                        }
                    }
                }
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const uint32_t i = c0 + (h + v) * KU_THREADS + threadIdx.x;
                    m[h + v] = bi[v] >= 0 && (float)bd[v] < P.bf_ratio * (float)sd[v] ? bi[v] : -1;
                    if (i < n) a2b[i] = m[h + v];
                }
            }
        }
        uint32_t ok = 0u;  // bit u: item u is a match
        if (!MUTUAL) {
#pragma unroll
            for (int u = 0; u < KU_ITEMS; ++u) ok |= (m[u] >= 0 ? 1u : 0u) << u;
        } else if (P.bacc) {
            // b's search from its accumulator (k_match): the pool rule over a's
            // levels bl - 1 .. bl + 1, the ratio test, and its nearest a is this a
            uint4 e[KU_ITEMS];
#pragma unroll
            for (int u = 0; u < KU_ITEMS; ++u)
                if (m[u] >= 0) e[u] = P.bacc[(size_t)USLAM_PACK_LEVEL(m[u]) * B.cap + USLAM_PACK_INDEX(m[u])];
#pragma unroll
            for (int u = 0; u < KU_ITEMS; ++u) {
                if (m[u] < 0) continue;
                const int bl = USLAM_PACK_LEVEL(m[u]);
                uint32_t pool = A.kept[bl];
                if (bl > 0) pool += A.kept[bl - 1];
                if (bl + 1 < A.levels) pool += A.kept[bl + 1];
                const uint32_t i = c0 + u * KU_THREADS + threadIdx.x;
                if (pool >= 2u && e[u].y != 0xffffffffu && (float)e[u].y < 0.85f * (float)e[u].z &&
                    e[u].x == (uint32_t)USLAM_PACK(l, i))
                    ok |= 1u << u;
            }
        } else {
            int32_t back[KU_ITEMS];
#pragma unroll
            for (int u = 0; u < KU_ITEMS; ++u)
                if (m[u] >= 0) back[u] = P.b2a[(size_t)USLAM_PACK_LEVEL(m[u]) * B.cap + USLAM_PACK_INDEX(m[u])];
#pragma unroll
            for (int u = 0; u < KU_ITEMS; ++u)
                if (m[u] >= 0 && back[u] == USLAM_PACK(l, c0 + u * KU_THREADS + threadIdx.x)) ok |= 1u << u;
        }
        uint32_t before[KU_ITEMS];  // matches of earlier lanes of the warp in the same item row
#pragma unroll
        for (int u = 0; u < KU_ITEMS; ++u) {
            const uint32_t bal = __ballot_sync(0xffffffffu, (ok >> u) & 1u);
            before[u] = (uint32_t)__popc(bal & ((1u << lane) - 1u));
            if (lane == 0) s_cnt[u][warp] = (uint32_t)__popc(bal);
        }
        __syncthreads();
        if (warp < KU_ITEMS) {
            const uint32_t v = s_cnt[warp][lane], incl = warp_inclusive_scan(v, lane);
            s_cnt[warp][lane] = incl - v;
            if (lane == 31) s_row[warp] = incl;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < KU_ITEMS; ++u) {
            if ((ok >> u) & 1u) {
                const uint32_t pos = base + s_cnt[u][warp] + before[u];
                if (pos < (uint32_t)P.max_matches_per_level) {
                    // (four stores: a caller's match buffer may be aligned to 4 bytes only)
                    int32_t* o = P.matches + ((size_t)l * P.max_matches_per_level + pos) * 4;
                    o[0] = l;
                    o[1] = (int32_t)(c0 + u * KU_THREADS + threadIdx.x);
                    o[2] = USLAM_PACK_LEVEL(m[u]);
                    o[3] = USLAM_PACK_INDEX(m[u]);
                } else {
                    atomicOr(err, USLAM_ERR_MATCH_OVERFLOW);
                }
            }
            base += s_row[u];
        }
        __syncthreads();  // s_cnt and s_row are rewritten
    }
    if (threadIdx.x == 0) P.match_count[l] = base;
}

// ------------------------------------------------------- frame ingest ----
// The reference's f32 pixel rule (data/src/provider_base.cpp:121-124 stores
// u8 / 255): the byte back, exact for those values; others become p * 255
// clamped to [0, 255] (NaN to 0) and rounded half to even.  One thread per 4
// pixels of a row.
__global__ void __launch_bounds__(128) k_frame_from_f32(const float* __restrict__ src, int W, int H, uint8_t* __restrict__ dst, int dpitch) {
    const int x4 = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (4 * x4 >= W || y >= H) return;
    const float* row = src + (size_t)y * W;
    uint32_t packed = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int x = 4 * x4 + k;
        if (x >= W) break;
        float t = row[x] * 255.0f;
        t = t > 0.0f ? (t < 255.0f ? t : 255.0f) : 0.0f;
        packed |= (uint32_t)__float2int_rn(t) << (8 * k);
    }
    uint8_t* out = dst + (size_t)y * dpitch + 4 * x4;
    if (4 * x4 + 4 <= W) {
        *reinterpret_cast<uint32_t*>(out) = packed;  // dpitch and the row start are multiples of 16
    } else {
        for (int k = 0; 4 * x4 + k < W; ++k) out[k] = (uint8_t)(packed >> (8 * k));
    }
}

}  // namespace uslam

// ------------------------------------------------------------ launch ----
namespace uslam {


template <bool CFG>
cudaError_t launch_detect_profile(const FrameDev* frames, const TileItem* tiles, int ntiles, int shape, uint32_t* err,
                                  cudaStream_t st) {
    switch (shape) {
        case 0: k_detect<64, 32, CFG><<<ntiles, K1_THREADS, 0, st>>>(frames, tiles, shape, err); break;
        case 1: k_detect<128, 32, CFG><<<ntiles, K1_THREADS, 0, st>>>(frames, tiles, shape, err); break;
        case 2: k_detect<64, 16, CFG><<<ntiles, K1_THREADS, 0, st>>>(frames, tiles, shape, err); break;
        case 3: k_detect<32, 32, CFG><<<ntiles, K1_THREADS, 0, st>>>(frames, tiles, shape, err); break;
        case 4: k_detect<128, 16, CFG><<<ntiles, K1_THREADS, 0, st>>>(frames, tiles, shape, err); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}
cudaError_t launch_pyramid(const FrameDev* frames, const TileItem* tiles, int ntiles, int shape, uint32_t* blur_count,
                           cudaStream_t st) {
    if (ntiles <= 0) return cudaSuccess;
    switch (shape) {
        case 0: k_pyramid<64, 32><<<ntiles, K1_THREADS, 0, st>>>(frames, tiles, blur_count); break;
        case 1: k_pyramid<128, 32><<<ntiles, K1_THREADS, 0, st>>>(frames, tiles, blur_count); break;
        case 2: k_pyramid<64, 16><<<ntiles, K1_THREADS, 0, st>>>(frames, tiles, blur_count); break;
        case 3: k_pyramid<32, 32><<<ntiles, K1_THREADS, 0, st>>>(frames, tiles, blur_count); break;
        case 4: k_pyramid<128, 16><<<ntiles, K1_THREADS, 0, st>>>(frames, tiles, blur_count); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_detect(const FrameDev* frames, const TileItem* tiles, int ntiles, int shape, int detector,
                          uint32_t* err, cudaStream_t st) {
    if (ntiles <= 0) return cudaSuccess;
    return detector == 1 ? launch_detect_profile<true>(frames, tiles, ntiles, shape, err, st)
                         : launch_detect_profile<false>(frames, tiles, ntiles, shape, err, st);
}

// The ordered lists and the list of blur tiles they need.
cudaError_t launch_compact_banded(const FrameDev* frames, const BandItem* bands, int nbands, int cell_cap, BlurList bl,
                                  cudaStream_t st) {
    if (nbands <= 0) return cudaSuccess;
    if (cell_cap > 0) {
        k_band_count<<<nbands, KBAND_THREADS, 0, st>>>(frames, bands);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    k_band_write<<<nbands, KBAND_THREADS, 0, st>>>(frames, bands, bl);
    return cudaGetLastError();
}

// max_bands: the largest FrameDev::nbands of the segments' frames.
cudaError_t launch_xsort(const FrameDev* frames, const SegDev* segs, int nseg, int max_w, int max_bands, cudaStream_t st) {
    if (nseg <= 0) return cudaSuccess;
    k_xsort<<<dim3(nseg, 2 * max_bands), KC_THREADS, (size_t)(max_w + 1) * sizeof(uint32_t), st>>>(frames, segs);
    return cudaGetLastError();
}

// max_tiles: the most items the list can hold.
cudaError_t launch_blur(const FrameDev* frames, BlurList bl, int max_tiles, int num_sms, uint32_t* err,
                        cudaStream_t st) {
    if (max_tiles <= 0) return cudaSuccess;
    k_blur<<<min(max_tiles, num_sms * KBL_CTAS_PER_SM), KBL_THREADS, 0, st>>>(frames, bl, err, 1.0f);
    return cudaGetLastError();
}

cudaError_t launch_describe(const FrameDev* frames, const SegDev* segs, int nseg, const DescTable* table,
                            int num_sms, bool pack, bool win, cudaStream_t st) {
    if (nseg <= 0) return cudaSuccess;
    if (pack) k_describe<true, false><<<num_sms, KD_THREADS, kDescSmem, st>>>(frames, segs, nseg, table);
    else if (win) k_describe<false, true><<<num_sms, KD_THREADS, kDescSmem, st>>>(frames, segs, nseg, table);
    else k_describe<false, false><<<num_sms, KD_THREADS, kDescSmem, st>>>(frames, segs, nseg, table);
    return cudaGetLastError();
}
cudaError_t set_describe_smem() {
    cudaError_t e = cudaFuncSetAttribute(k_describe<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDescSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_describe<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDescSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_describe<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDescSmem);
    return e;
}

cudaError_t launch_describe_tiled(const FrameDev* frames, const BandItem* items, int nitems, const int32_t* pattern,
                                  bool pack, bool win, int margin, uint32_t* err, cudaStream_t st) {
    if (nitems <= 0) return cudaSuccess;
    const size_t smem = describe_tiled_smem(margin);
    if (pack) k_describe_tiled<true, false><<<nitems, KDT_THREADS, smem, st>>>(frames, items, pattern, err);
    else if (win) k_describe_tiled<false, true><<<nitems, KDT_THREADS, smem, st>>>(frames, items, pattern, err);
    else k_describe_tiled<false, false><<<nitems, KDT_THREADS, smem, st>>>(frames, items, pattern, err);
    return cudaGetLastError();
}

cudaError_t set_describe_tiled_smem(int margin) {
    const int smem = (int)describe_tiled_smem(margin);
    cudaError_t e = cudaFuncSetAttribute(k_describe_tiled<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_describe_tiled<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_describe_tiled<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return e;
}

// k_match over all SMs (num_sms x its resident CTAs).
cudaError_t launch_match(const FrameDev* frames, const PairDev* pairs, const void* segs, int nseg, int num_sms,
                         cudaStream_t st) {
    if (nseg <= 0) return cudaSuccess;
    k_match<false><<<num_sms * KM_CTAS_PER_SM, KM_THREADS, 0, st>>>(frames, pairs, static_cast<const MatchSegDev*>(segs),
                                                                    nseg, nullptr, 2u);
    return cudaGetLastError();
}

// k_match with several units per query group, for the pairs' aacc; claim: a
// zero word that hands out the units after each warp's first (null: every
// warp takes its share of them).
cudaError_t launch_match_parts(const FrameDev* frames, const PairDev* pairs, const void* segs, int nseg, int num_sms,
                               uint32_t* claim, cudaStream_t st) {
    if (nseg <= 0) return cudaSuccess;
    k_match<true><<<num_sms * KM_CTAS_PER_SM, KM_THREADS, 0, st>>>(frames, pairs, static_cast<const MatchSegDev*>(segs),
                                                                   nseg, claim, 2u);
    return cudaGetLastError();
}
cudaError_t launch_bacc_init(const FrameDev* frames, const PairDev* pairs, const SegDev* segs, int nseg,
                             cudaStream_t st) {
    if (nseg <= 0) return cudaSuccess;
    k_bacc_init<<<nseg, 256, 0, st>>>(frames, pairs, segs);
    return cudaGetLastError();
}

cudaError_t launch_mutual(const FrameDev* frames, const PairDev* pairs, const SegDev* segs, int nseg,
                          uint32_t* err, cudaStream_t st) {
    if (nseg <= 0) return cudaSuccess;
    k_mutual<true><<<nseg, KU_THREADS, 0, st>>>(frames, pairs, segs, err, nullptr);
    return cudaGetLastError();
}
cudaError_t launch_mutual_reset(const FrameDev* frames, const PairDev* pairs, const SegDev* segs, int nseg,
                                uint32_t* err, uint32_t* next_group, cudaStream_t st) {
    if (nseg <= 0) return cudaSuccess;
    k_mutual<true><<<nseg, KU_THREADS, 0, st>>>(frames, pairs, segs, err, next_group);
    return cudaGetLastError();
}

cudaError_t launch_emit(const FrameDev* frames, const PairDev* pairs, const SegDev* segs, int nseg, uint32_t* err,
                        cudaStream_t st) {
    if (nseg <= 0) return cudaSuccess;
    k_mutual<false><<<nseg, KU_THREADS, 0, st>>>(frames, pairs, segs, err, nullptr);
    return cudaGetLastError();
}

cudaError_t launch_bruteforce(const FrameDev* frames, const PairDev* pairs, const SegDev* psegs, int npairs,
                              float ratio, int sms, cudaStream_t st) {
    if (npairs <= 0) return cudaSuccess;
    static_assert((MAX_SEGS + 1) * 8 <= 40 * 1024, "the pairs' table fits the default limit beside the tile");
    k_bruteforce<<<sms * KB_CTAS, KB_THREADS, (npairs + 1) * sizeof(unsigned long long), st>>>(frames, pairs, psegs, npairs, ratio, 2u);
    return cudaGetLastError();
}

cudaError_t launch_take_frames(FrameDev* dst, const FrameDev* a, const FrameDev* b, uint32_t* err, cudaStream_t st) {
    k_take_frames<<<1, 256, 0, st>>>(dst, a, b, err);
    return cudaGetLastError();
}

cudaError_t launch_frame_from_f32(const float* src, int W, int H, uint8_t* dst, int dpitch, cudaStream_t st) {
    if (W <= 0 || H <= 0) return cudaSuccess;
    const dim3 grid((W / 4 + 127) / 128 + 1, H);
    k_frame_from_f32<<<grid, 128, 0, st>>>(src, W, H, dst, dpitch);
    return cudaGetLastError();
}

cudaError_t set_compact_smem(int max_w) {
    const size_t smem = (size_t)(max_w + 1) * sizeof(uint32_t);
    if (smem <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(k_xsort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

}  // namespace uslam
