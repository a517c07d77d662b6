// The estimate's passes on integer luma: level 0 as pair planes (LumaPyrParams::pa / pc), a word holding a pixel and its
// right neighbour as 16-bit multiples of 1/16 level. Bilinear taps are two-way dot products (dp2a) of a word with byte
// weights, absolute differences one instruction (sad), all sums exact in 32 bits: the same values as the float kernels
// of fg_kernels.cu, which run where level 0 is not a multiple of 1/16 (flowScale 4 with 3-pixel cells).
//
// The searches and the sub-pixel pass are bound by instruction issue (76 and 83 % of the issue slots), the pixel field by
// issue and its barriers (66 %, 24 warps per SM). Measured (ncu, 3840x2160 at flowScale 2, float kernel -> this one; warp
// instructions): level-0 search 41.4 -> 29.7 us (30.1 -> 20.1 M), sub-pixel 65.9 -> 26.9 us (38.6 -> 20.1 M; it took the
// scene-cut sum then and takes level 0's median3 now), pixel field 80.4 -> 42.4 us (52.8 -> 25.4 M, the scene-cut sum with
// it). The pair planes cost the luma pass nothing: float level 0 is written only where a pass reads it.
#include "fg_device.h"

namespace fgk {

// ============================================================================================== seed + search
// interp.seed_from :131-144 and interp.search :116-124, as k_search_r (fg_kernels.cu), one warp per 8x8 block, for
// radii 1 and 2. Lane = (column x, rows 2 g and 2 g + 1) of the block: a candidate's score is two absolute differences
// per lane and one warp reduction. The window's rows stay in registers for all dy of one dx.
//
// kPair: level 0's pair planes (the pixel in a word's low half); else a float level whose values times qscale are
// integers below 2^23: the float 2^23 + v qscale holds them in its low bits, and the exponent cancels in differences.
template <bool kPair>
struct QSrc {
    const void* a;
    const void* c;
    float scale;
    __device__ __forceinline__ uint32_t ld(const void* plane, int i) const {
        if (kPair) return __ldg(reinterpret_cast<const uint32_t*>(plane) + i) & 0xFFFFu;
        return __float_as_uint(__fmaf_rn(__ldg(reinterpret_cast<const float*>(plane) + i), scale, 8388608.0f));
    }
};

// a warp reduction's result k to lane k
__device__ __forceinline__ void keepLane(uint32_t& mine, uint32_t r, int lane, int k) { mine = lane == k ? r : mine; }

template <int R, bool kPair>
__device__ __forceinline__ void searchQCta(const SearchParams& p, int ctaX, int by) {
    constexpr int T = 8 + 2 * R, TS = 12, D = 2 * R + 1;   // TS: two rows = 24 words, so the 4 row pairs hit all banks
    static_assert(T <= TS && D * D <= 32, "radius 1 or 2");
    __shared__ uint32_t win[4][2][T * TS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bx = ctaX * 4 + warp;
    if (bx >= p.bw) return;
    const QSrc<kPair> src = kPair ? QSrc<kPair>{p.pa, p.pc, 0.0f} : QSrc<kPair>{p.la, p.lc, p.qscale};
    const float unit = kPair ? 1.0f / 1024.0f : 1.0f / (64.0f * p.qscale);   // a block sum -> its mean in levels (exact)
    const int b = by * p.bw + bx, b0x = bx * kBlock, b0y = by * kBlock;
    const int lx = lane & 7, ly = (lane >> 3) * 2;
    // the seed: own parent, the 3 nearest other parents, zero, the global median (2x the parent level's vectors); the
    // first minimum. A candidate equal to an earlier one could never be picked.
    int sx = 0, sy = 0;
    if (!p.top) {
        int cxs[6], cys[6];
        bool pen0 = false;   // the first candidate pays lambda too
        if (p.cnn) {   // the seed net's two candidates, then zero (slots 3..5 repeat it)
            const float* o = p.cnn + (size_t)b * kSeedNetOut;
#pragma unroll
            for (int k = 0; k < 6; k++) {
                cxs[k] = k < 2 ? __float2int_rn(fminf(fmaxf(o[2 * k], -256.0f), 256.0f)) : 0;
                cys[k] = k < 2 ? __float2int_rn(fminf(fmaxf(o[2 * k + 1], -256.0f), 256.0f)) : 0;
            }
            pen0 = !(o[4] >= 0.0f);
        } else {
            const int px = min(bx >> 1, p.pw - 1), py = min(by >> 1, p.ph - 1);
            const int px1 = clampi(px + ((bx & 1) ? 1 : -1), 0, p.pw - 1), py1 = clampi(py + ((by & 1) ? 1 : -1), 0, p.ph - 1);
#pragma unroll
            for (int k = 0; k < 4; k++) {   // own, vertical, horizontal, diagonal neighbour
                const float2 v = __ldg(p.parent + ((k & 1) ? py1 : py) * p.pw + ((k & 2) ? px1 : px));
                cxs[k] = 2 * __float2int_rn(v.x);
                cys[k] = 2 * __float2int_rn(v.y);
            }
            cxs[4] = cys[4] = 0;
            cxs[5] = __float2int_rn(p.med[0]);
            cys[5] = __float2int_rn(p.med[1]);
        }
        const int qx = b0x + lx, qy = b0y + ly;
        float best = 0.0f;
#pragma unroll
        for (int k = 0; k < 6; k++) {
            bool dup = false;
#pragma unroll
            for (int j = 0; j < k; j++) dup |= cxs[j] == cxs[k] && cys[j] == cys[k];
            if (dup) continue;   // warp-uniform
            const int cx = cxs[k], cy = cys[k];
            uint32_t s;
            if (b0x - abs(cx) >= 0 && b0x + 7 + abs(cx) < p.w && b0y - abs(cy) >= 0 && b0y + 7 + abs(cy) < p.h) {
                const int ia = (qy - cy) * p.w + (qx - cx), ic = (qy + cy) * p.w + (qx + cx);
                s = __usad(src.ld(src.a, ia + p.w), src.ld(src.c, ic + p.w), __usad(src.ld(src.a, ia), src.ld(src.c, ic), 0u));
            } else {
                const int xa = clampi(qx - cx, 0, p.w - 1), xc = clampi(qx + cx, 0, p.w - 1);
                s = 0;
#pragma unroll
                for (int r = 0; r < 2; r++)
                    s = __usad(src.ld(src.a, clampi(qy + r - cy, 0, p.h - 1) * p.w + xa),
                               src.ld(src.c, clampi(qy + r + cy, 0, p.h - 1) * p.w + xc), s);
            }
            float cost = __fmul_rn((float)__reduce_add_sync(0xffffffffu, s), unit);
            if (k > 0 || pen0) cost = __fadd_rn(cost, p.lambda);
            if (k == 0 || cost < best) { best = cost; sx = cx; sy = cy; }
        }
    }
    // the T x T windows of a at q - s and c at q + s
    uint32_t* wa = win[warp][0];
    uint32_t* wc = win[warp][1];
    const int ax0 = b0x - sx - R, ay0 = b0y - sy - R, cx0 = b0x + sx - R, cy0 = b0y + sy - R;
    constexpr int LR = 32 / T;   // window rows staged per step
    const int tr = lane / T, tc = lane % T;
    if (tr < LR) {
        const bool in = ax0 >= 0 && ay0 >= 0 && ax0 + T <= p.w && ay0 + T <= p.h && cx0 >= 0 && cy0 >= 0 && cx0 + T <= p.w && cy0 + T <= p.h;
        if (in) {
            const int ia = (ay0 + tr) * p.w + ax0 + tc, ic = (cy0 + tr) * p.w + cx0 + tc;
#pragma unroll
            for (int r = 0; r < T; r += LR)
                if (T % LR == 0 || r + tr < T) {
                    wa[(r + tr) * TS + tc] = src.ld(src.a, ia + r * p.w);
                    wc[(r + tr) * TS + tc] = src.ld(src.c, ic + r * p.w);
                }
        } else {
            const int xa = clampi(ax0 + tc, 0, p.w - 1), xc = clampi(cx0 + tc, 0, p.w - 1);
            for (int r = tr; r < T; r += LR) {
                wa[r * TS + tc] = src.ld(src.a, clampi(ay0 + r, 0, p.h - 1) * p.w + xa);
                wc[r * TS + tc] = src.ld(src.c, clampi(cy0 + r, 0, p.h - 1) * p.w + xc);
            }
        }
    }
    __syncwarp();
    uint32_t mine = 0;   // lane i: the sum of candidate i = (dy + R) D + dx + R
    const uint32_t* pa = wa + ly * TS + lx;
    const uint32_t* pc = wc + ly * TS + lx;
#pragma unroll
    for (int dxi = 0; dxi < D; dxi++) {
        uint32_t a[D + 1], c[D + 1];   // rows ly - R .. ly + 1 + R of column lx -+ dx
#pragma unroll
        for (int i = 0; i <= D; i++) {
            a[i] = pa[i * TS + 2 * R - dxi];
            c[i] = pc[i * TS + dxi];
        }
#pragma unroll
        for (int dyi = 0; dyi < D; dyi++)
            keepLane(mine, __reduce_add_sync(0xffffffffu, __usad(a[2 * R - dyi + 1], c[dyi + 1], __usad(a[2 * R - dyi], c[dyi], 0u))),
                     lane, dyi * D + dxi);
    }
    const int dy = lane / D - R, dx = lane % D - R;
    const float sad = __fmul_rn((float)mine, unit);
    const float cost = __fadd_rn(sad, __fmul_rn(p.lambda, (float)(abs(dx) + abs(dy))));   // = fl32(lambda n) (interp.py:121)
    // the first minimum: costs are not negative, so their bits order as they do
    const uint32_t bits = lane < D * D ? __float_as_uint(cost) : 0xffffffffu;
    const int ci = __ffs(__ballot_sync(0xffffffffu, bits == __reduce_min_sync(0xffffffffu, bits))) - 1;
    if (lane == ci) {
        p.out[b] = make_float2((float)(sx + dx), (float)(sy + dy));
        if (p.sadOut) p.sadOut[b] = sad;
    }
}
template <int R, bool kPair>
__global__ void __launch_bounds__(128) k_search_q(const SearchParams p) {
    pdlEnter();
    searchQCta<R, kPair>(p, blockIdx.x, blockIdx.y);
}
template <int R, bool kPair>
__global__ void __launch_bounds__(128) k_search_q_m(const __grid_constant__ Merged<SearchParams> m) {
    pdlEnter();
    int bx, by;
    const int i = mergedItem(m, bx, by);
    searchQCta<R, kPair>(m.item[i], bx, by);
}

// ============================================================================================== sub-pixel refinement
// interp.flow :162-163: search(., 1, 0.5) then search(., 1, 0.25) around the median-filtered integer vector s, as
// k_subpix (fg_kernels.cu), one warp per finest-level block. Lane = (column x, rows 2 g and 2 g + 1). Both frames' pair
// words of rows and columns -1 .. 8 around the block (9 words a row) wait in shared memory; a pass takes, per column
// offset and frame, 4 rows of horizontal taps (one load and one dp2a each) and forms its 3 row offsets' vertical taps
// from them: offsets are compile-time per pass and chosen half-pixel row, so a vertical tap is at most one multiply-add.
constexpr int kQsS = 12, kQsRows = 10, kQsCols = 9;   // row stride (two rows = 24 words: conflict-free), rows, words a row

// 9 candidates (dx, dy) = quarter offsets (b4x + S4 {-1, 0, 1}, BY + S4 {-1, 0, 1}); returns in lane i = (dy + 1) 3 +
// dx + 1 its sum of absolute differences in units of 1/256 level
template <int S4, int BY>
__device__ __forceinline__ uint32_t subPass(const uint32_t* ta, const uint32_t* tc, int b4x, int lane) {
    uint32_t mine = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const int o = b4x + S4 * (d - 1);   // a at x - o / 4, c at x + o / 4
        const uint32_t wa = ((uint32_t)(-o) & 3u) * 255u + 4u, wc = ((uint32_t)o & 3u) * 255u + 4u;   // (4 - f) | f << 8
        const uint32_t* qa = ta + ((-o) >> 2);
        const uint32_t* qc = tc + (o >> 2);
        uint32_t ha[4], hc[4];   // rows y - 1 .. y + 2
#pragma unroll
        for (int i = 0; i < 4; i++) {
            ha[i] = __dp2a_lo(qa[i * kQsS], wa, 0u);
            hc[i] = __dp2a_lo(qc[i * kQsS], wc, 0u);
        }
#pragma unroll
        for (int e = 0; e < 3; e++) {
            constexpr int base[3] = {BY - S4, BY, BY + S4};
            const int oa = -base[e], oc = base[e];
            const int ra = 1 + (oa >> 2), rc = 1 + (oc >> 2), fa = oa & 3, fc = oc & 3;
            uint32_t s = 0;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                uint32_t va, vc;   // x 1 (f = 0), x 2 (f = 2) or x 4
                if (fa == 0) {
                    va = ha[i + ra];
                    vc = hc[i + rc];
                } else if (fa == 2) {
                    va = ha[i + ra] + ha[i + ra + 1];
                    vc = hc[i + rc] + hc[i + rc + 1];
                } else {
                    va = ha[i + ra] * (uint32_t)(4 - fa) + ha[i + ra + 1] * (uint32_t)fa;
                    vc = hc[i + rc] * (uint32_t)(4 - fc) + hc[i + rc + 1] * (uint32_t)fc;
                }
                s = __usad(va, vc, s);
            }
            keepLane(mine, __reduce_add_sync(0xffffffffu, s) << (fa == 0 ? 2 : (fa == 2 ? 1 : 0)), lane, e * 3 + d);
        }
    }
    return mine;
}

__device__ __forceinline__ void subpixQCta(const SubpixParams& p, int ctaX, int by) {
    __shared__ uint32_t tile[4][2][kQsRows * kQsS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bx = ctaX * 4 + warp;
    if (bx >= p.bw) return;
    const int b = by * p.bw + bx, b0x = bx * kBlock, b0y = by * kBlock;
    // interp.median3 :127-128 of the search's field at this block (level 0's medians feed nothing else: a launch of their own
    // cost more): lanes 0..8 hold the neighbours' x, 16..24 their y; the median is the one of rank 4
    int sx, sy;
    {
        const int i = lane & 15, j = min(i, 8);
        const float v = __ldg(reinterpret_cast<const float*>(p.in + clampi(by + j / 3 - 1, 0, p.bh - 1) * p.bw + clampi(bx + j % 3 - 1, 0, p.bw - 1)) +
                              (lane >> 4));
        int rank = i > 8 ? 16 : 0;
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const float u = __shfl_sync(0xffffffffu, v, (lane & 16) + k);
            rank += u < v || (u == v && k < i);
        }
        const uint32_t m = __ballot_sync(0xffffffffu, rank == 4);
        const float mx = __shfl_sync(0xffffffffu, v, __ffs(m & 0xffffu) - 1), my = __shfl_sync(0xffffffffu, v, 15 + __ffs(m >> 16));
        if (lane == 0) p.med[b] = make_float2(mx, my);
        sx = __float2int_rn(mx);
        sy = __float2int_rn(my);
    }
    uint32_t* wa = tile[warp][0];
    uint32_t* wc = tile[warp][1];
    const int ax0 = b0x - sx - 1, ay0 = b0y - sy - 1, cx0 = b0x + sx - 1, cy0 = b0y + sy - 1;
    const int tr = lane / kQsCols, tc = lane % kQsCols;   // 3 rows per step
    if (tr < 3) {
        const bool in = ax0 >= 0 && ay0 >= 0 && ax0 + kQsCols < p.w && ay0 + kQsRows <= p.h && cx0 >= 0 && cy0 >= 0 &&
                        cx0 + kQsCols < p.w && cy0 + kQsRows <= p.h;
        if (in) {
            const uint32_t* qa = p.pa + (ay0 + tr) * p.w + ax0 + tc;
            const uint32_t* qc = p.pc + (cy0 + tr) * p.w + cx0 + tc;
#pragma unroll
            for (int r = 0; r < kQsRows; r += 3)
                if (r + 3 <= kQsRows || r + tr < kQsRows) {
                    wa[(r + tr) * kQsS + tc] = __ldg(qa + r * p.w);
                    wc[(r + tr) * kQsS + tc] = __ldg(qc + r * p.w);
                }
        } else {   // clamped: left of the frame both halves are pixel 0 (the last column's word repeats its pixel)
            const int xa = clampi(ax0 + tc, 0, p.w - 1), xc = clampi(cx0 + tc, 0, p.w - 1);
            for (int r = tr; r < kQsRows; r += 3) {
                const uint32_t a = __ldg(p.pa + clampi(ay0 + r, 0, p.h - 1) * p.w + xa), c = __ldg(p.pc + clampi(cy0 + r, 0, p.h - 1) * p.w + xc);
                wa[r * kQsS + tc] = ax0 + tc < 0 ? __byte_perm(a, a, 0x1010) : a;
                wc[r * kQsS + tc] = cx0 + tc < 0 ? __byte_perm(c, c, 0x1010) : c;
            }
        }
    }
    __syncwarp();
    // this lane's column and first row in the tiles: pixel (x, y) is word (x + 1, y + 1); rows from y - 1
    const uint32_t* ta = wa + (lane >> 3) * 2 * kQsS + (lane & 7) + 1;
    const uint32_t* tcq = wc + (lane >> 3) * 2 * kQsS + (lane & 7) + 1;
    const int n = lane < 9 ? abs(lane % 3 - 1) + abs(lane / 3 - 1) : 0;
    int b4x = 0, b4y = 0;   // the offset chosen so far, quarter pixels
    float sadBest = 0.0f;
#pragma unroll
    for (int pass = 0; pass < 2; pass++) {
        uint32_t sum;
        if (pass == 0) sum = subPass<2, 0>(ta, tcq, 0, lane);
        else if (b4y == 0) sum = subPass<1, 0>(ta, tcq, b4x, lane);
        else if (b4y < 0) sum = subPass<1, -2>(ta, tcq, b4x, lane);
        else sum = subPass<1, 2>(ta, tcq, b4x, lane);
        const float sad = __fmul_rn((float)sum, 1.0f / 16384.0f);
        const float cost = __fadd_rn(sad, n == 0 ? p.pen[pass][0] : (n == 1 ? p.pen[pass][1] : p.pen[pass][2]));
        const uint32_t bits = lane < 9 ? __float_as_uint(cost) : 0xffffffffu;   // costs are not negative
        const int ci = __ffs(__ballot_sync(0xffffffffu, bits == __reduce_min_sync(0xffffffffu, bits))) - 1;
        const int step = pass ? 1 : 2;
        b4x += step * (ci % 3 - 1);
        b4y += step * (ci / 3 - 1);
        if (pass) sadBest = __shfl_sync(0xffffffffu, sad, ci);
        else if (p.out0 && lane == 0)
            p.out0[b] = make_float2(__fadd_rn((float)sx, (float)b4x * 0.25f), __fadd_rn((float)sy, (float)b4y * 0.25f));
    }
    if (lane == 0) {
        p.out[b] = make_float2(__fadd_rn((float)sx, (float)b4x * 0.25f), __fadd_rn((float)sy, (float)b4y * 0.25f));
        p.sads[b] = sadBest;   // summed for the scene cut by the pixel-field launch
    }
}
__global__ void __launch_bounds__(128) k_subpix_q(const SubpixParams p) {
    pdlEnter();
    subpixQCta(p, blockIdx.x, blockIdx.y);
}
__global__ void __launch_bounds__(128) k_subpix_q_m(const __grid_constant__ Merged<SubpixParams> m) {
    pdlEnter();
    int bx, by;
    const int i = mergedItem(m, bx, by);
    subpixQCta(m.item[i], bx, by);
}

// ============================================================================================== per-pixel field
// interp.pixel_field :167-183 at flow resolution, as k_pixfield (fg_kernels.cu): per pixel the candidate vectors
// bilinear block field, own block, block above / below / left / right, zero; each scored by the 5x5 replicate-border
// box of |a(q - h) - c(q + h)| where every window pixel uses its own candidate; the first minimum wins.
//
// One CTA = 60 x 32 outputs (4 block rows) with a 2 px apron, one candidate at a time. The vectors of a tile's blocks
// differ little, so the window of each frame that they reach is staged in shared memory first, clamped there to the frame
// (kWin): every tap after that is a shared load at a fixed offset, and frame edges cost nothing more. A thread owns a
// region column and the 8 rows of one block row, so a block candidate has one vector and one set of weights per run: per
// row and frame one load and one dp2a, the lower tap row reused as the next row's upper one. The 2 + 2 apron rows take one
// more pixel per thread. Errors stay in registers: the vertical 5-sums run down the thread's rows (2 rows above and below
// from the neighbours through shared memory), the horizontal 5-sums and the choice along rows, 8 pixels per thread. Tiles
// whose vectors differ by more than the window allows load their taps from the planes, clamped one by one.
constexpr int kQfE = 64, kQfAp = 2, kQfTW = kQfE - 2 * kQfAp, kQfTH = 32, kQfNC = 7;
constexpr int kQfG = kQfTH / 8;                             // block rows (thread rows) of a tile
constexpr int kQfBX = kQfE / 8 + 4, kQfBY = kQfG + 4;       // block-field region: the tile's, the apron's, +-1 around
constexpr int kQfWX = 80, kQfWY = 46;   // the windows: vectors of a tile within 16 px of each other across, 9 down
constexpr int kQfVS = kQfE + 4;   // row stride of the vertical sums: 16-byte loads down 8 rows hit all banks once

// (32 - f) | f << 8, f = X & 31: a tap pair's byte weights (left, right) at 1/32 position X
__device__ __forceinline__ uint32_t qWeights(int X) { return ((uint32_t)X & 31u) * 255u + 32u; }
// a pair-plane word, clamped (the last column's word repeats its pixel; left of the frame both halves are pixel 0)
__device__ __forceinline__ uint32_t ldPairClamped(const uint32_t* plane, int w, int h, int x, int y) {
    const uint32_t v = __ldg(plane + (size_t)clampi(y, 0, h - 1) * w + clampi(x, 0, w - 1));
    return x < 0 ? __byte_perm(v, v, 0x1010) : v;
}

struct QfTile {
    float2 bv[kQfBY][kQfBX];
    int2 bR[kQfBY][kQfBX];                     // rne(32 v)
    uint32_t above[kQfG + 1][2][kQfE];         // the errors of the 2 rows above each thread row (0: the apron's)
    uint32_t below[kQfG + 1][2][kQfE];         // ... below thread row i - 1 (kQfG: the apron's)
    alignas(16) uint32_t v[kQfTH][kQfVS];      // the vertical 5-sums
    uint8_t pick[kQfTH][kQfE];
    int4 range[4];                             // per warp: the least and largest R (x, y) of its block vectors
    uint32_t differ;                           // bit k: candidate k (2 .. 5) is not the own block's everywhere
    alignas(8) uint32_t win[2][kQfWY * kQfWX];   // pair words of a and c
};
// the windows' origins
struct QfWin {
    int ax, ay, cx, cy;
};
// |a(q - h) - c(q + h)| in units of 2^-14 at pixel (qx, qy) for R = rne(32 h)
template <bool kWin>
__device__ __forceinline__ uint32_t qErr(const PixfieldParams& p, const QfTile& t, const QfWin& o, int qx, int qy, int Rx, int Ry) {
    const int xa = qx + ((-Rx) >> 5), ya = qy + ((-Ry) >> 5), xc = qx + (Rx >> 5), yc = qy + (Ry >> 5);
    const uint32_t wa = qWeights(-Rx), wc = qWeights(Rx), fa = (uint32_t)(-Ry) & 31u, fc = (uint32_t)Ry & 31u;
    uint32_t a0, a1, c0, c1;
    if (kWin) {
        const uint32_t* qa = t.win[0] + (ya - o.ay) * kQfWX + xa - o.ax;
        const uint32_t* qc = t.win[1] + (yc - o.cy) * kQfWX + xc - o.cx;
        a0 = qa[0];
        a1 = qa[kQfWX];
        c0 = qc[0];
        c1 = qc[kQfWX];
    } else {
        a0 = ldPairClamped(p.pa, p.w, p.h, xa, ya);
        a1 = ldPairClamped(p.pa, p.w, p.h, xa, ya + 1);
        c0 = ldPairClamped(p.pc, p.w, p.h, xc, yc);
        c1 = ldPairClamped(p.pc, p.w, p.h, xc, yc + 1);
    }
    return __usad(__dp2a_lo(a0, wa, 0u) * (32u - fa) + __dp2a_lo(a1, wa, 0u) * fa,
                  __dp2a_lo(c0, wc, 0u) * (32u - fc) + __dp2a_lo(c1, wc, 0u) * fc, 0u);
}

template <bool kWin>
__device__ __forceinline__ void pixfieldQTile(const PixfieldParams& p, QfTile& t, const QfWin& o, int X0, int Y0) {
    const int tid = threadIdx.x, ex = tid & (kQfE - 1), g = tid >> 6;
    const int bx0 = (X0 >> 3) - 2, by0 = (Y0 >> 3) - 2;
    // this thread's column; the columns and weights of cv2.resize x8 (weights (1, 0) beyond the borders)
    const int qx = clampi(X0 - kQfAp + ex, 0, p.w - 1);
    const int bx = (qx >> 3) - bx0;
    int cx0;
    float ca0, ca1;
    {
        const float f0 = __fsub_rn(__fmul_rn((float)qx + 0.5f, 0.125f), 0.5f);
        const int s = (int)floorf(f0);
        const bool edge = s < 0 || s >= p.bw - 1;
        const float f = edge ? 0.0f : __fsub_rn(f0, (float)s);
        cx0 = clampi(s, 0, p.bw - 1) - bx0;
        ca0 = 1.0f - f;
        ca1 = f;
    }
    // this thread's run: rows qy0 .. qy0 + 7 of block row br (rows past the frame repeat its last row below); its
    // apron pixel: thread rows 0, 1 the 2 rows above the tile, 2, 3 the 2 below
    const int qy0 = min(Y0 + 8 * g, p.h - 1), br = (qy0 >> 3) - by0;
    const int ay = clampi(Y0 + (g < 2 ? g - 2 : kQfTH + g - 2), 0, p.h - 1), abr = (ay >> 3) - by0;
    const int rows = p.h - qy0;   // rows of the run inside the frame, >= 1
    // the bilinear block field in this column at region block row r (exact: dyadic values)
    auto colField = [&](int r) {
        return __ffma2_rn(t.bv[r][cx0 + 1], make_float2(ca1, ca1), pmul(t.bv[r][cx0], make_float2(ca0, ca0)));
    };
    // ... and at row qy of block row r: weights (2 (qy & 7) + 1) / 16 +- 1/2
    auto rowField = [&](const float2& lo, const float2& mid, const float2& hi, int i) {
        const float f = (float)(2 * i + 1) * 0.0625f + (i < 4 ? 0.5f : -0.5f);
        const float2 a = i < 4 ? lo : mid, b = i < 4 ? mid : hi;
        return __ffma2_rn(b, make_float2(f, f), pmul(a, make_float2(1.0f - f, 1.0f - f)));
    };
    const int r8 = tid & 31, c8 = (tid >> 5) * 8;   // the row run of the horizontal sums and the choice
    float best[8];
    int pk[8];
#pragma unroll
    for (int i = 0; i < 8; i++) { best[i] = FLT_MAX; pk[i] = 0; }
    const uint32_t cands = t.differ | 0x43u;   // the bilinear, own-block and zero candidates always
    for (int k = 0; k < kQfNC; k++) {
        if (!((cands >> k) & 1u)) continue;
        uint32_t e[8], ea;   // the run's and the apron pixel's errors
        if (k == 0) {   // the upsampled field: a vector per pixel
            const float2 lo = colField(br - 1), mid = colField(br), hi = colField(br + 1);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float2 r = rne32bits(rowField(lo, mid, hi, j));
                e[j] = qErr<kWin>(p, t, o, qx, qy0 + j, __float_as_int(r.x) - 0x4B400000, __float_as_int(r.y) - 0x4B400000);
            }
            if (qy0 & 7) {   // a run below the frame: its rows repeat row h - 1
                const float2 r = rne32bits(rowField(lo, mid, hi, qy0 & 7));
                e[0] = qErr<kWin>(p, t, o, qx, qy0, __float_as_int(r.x) - 0x4B400000, __float_as_int(r.y) - 0x4B400000);
            }
            const float2 r = rne32bits(rowField(colField(abr - 1), colField(abr), colField(abr + 1), ay & 7));
            ea = qErr<kWin>(p, t, o, qx, ay, __float_as_int(r.x) - 0x4B400000, __float_as_int(r.y) - 0x4B400000);
        } else if (k < kQfNC - 1) {   // the vector of the pixel's own block or of a 4-neighbour
            const int dx = k == 4 ? -1 : (k == 5 ? 1 : 0), dy = k == 2 ? -1 : (k == 3 ? 1 : 0);
            const int2 Ra = t.bR[abr + dy][bx + dx];
            ea = qErr<kWin>(p, t, o, qx, ay, Ra.x, Ra.y);
            const int2 R = t.bR[br + dy][bx + dx];
            if (kWin) {
                const uint32_t wa = qWeights(-R.x), wc = qWeights(R.x);
                const uint32_t fa = (uint32_t)(-R.y) & 31u, fc = (uint32_t)R.y & 31u, ga = 32u - fa, gc = 32u - fc;
                const uint32_t* qa = t.win[0] + (qy0 + ((-R.y) >> 5) - o.ay) * kQfWX + qx + ((-R.x) >> 5) - o.ax;
                const uint32_t* qc = t.win[1] + (qy0 + (R.y >> 5) - o.cy) * kQfWX + qx + (R.x >> 5) - o.cx;
                uint32_t ta = __dp2a_lo(qa[0], wa, 0u), tc = __dp2a_lo(qc[0], wc, 0u);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const uint32_t ua = __dp2a_lo(qa[(j + 1) * kQfWX], wa, 0u), uc = __dp2a_lo(qc[(j + 1) * kQfWX], wc, 0u);
                    e[j] = __usad(ta * ga + ua * fa, tc * gc + uc * fc, 0u);
                    ta = ua;
                    tc = uc;
                }
            } else {
#pragma unroll 1
                for (int j = 0; j < 8; j++) {
                    const uint32_t v = qErr<kWin>(p, t, o, qx, qy0 + j, R.x, R.y);
#pragma unroll
                    for (int i = 0; i < 8; i++) e[i] = i == j ? v : e[i];
                }
            }
        } else {   // zero: the pixels themselves (weights 32 x 32)
            auto err0 = [&](int y) {
                const size_t i = (size_t)clampi(y, 0, p.h - 1) * p.w + qx;
                return __usad(__ldg(p.pa + i) & 0xFFFFu, __ldg(p.pc + i) & 0xFFFFu, 0u) << 10;
            };
#pragma unroll
            for (int j = 0; j < 8; j++) e[j] = err0(qy0 + j);
            ea = err0(ay);
        }
        if (rows < 8) {   // the frame's last row stands for the rows below it
#pragma unroll
            for (int j = 1; j < 8; j++)
                if (j >= rows) e[j] = e[j - 1];
        }
        // the vertical 5-sums of this run
        t.below[g][0][ex] = e[0];
        t.below[g][1][ex] = e[1];
        t.above[g + 1][0][ex] = e[6];
        t.above[g + 1][1][ex] = e[7];
        if (g < 2) t.above[0][g][ex] = ea;
        else t.below[kQfG][g - 2][ex] = ea;
        __syncthreads();
        const uint32_t a0 = t.above[g][0][ex], a1 = t.above[g][1][ex], b0 = t.below[g + 1][0][ex], b1 = t.below[g + 1][1][ex];
        uint32_t S = a0 + a1 + e[0] + e[1] + e[2];
        uint32_t* vo = &t.v[8 * g][ex];
        vo[0] = S;
        S += e[3] - a0; vo[kQfVS] = S;
        S += e[4] - a1; vo[2 * kQfVS] = S;
        S += e[5] - e[0]; vo[3 * kQfVS] = S;
        S += e[6] - e[1]; vo[4 * kQfVS] = S;
        S += e[7] - e[2]; vo[5 * kQfVS] = S;
        S += b0 - e[3]; vo[6 * kQfVS] = S;
        S += b1 - e[4]; vo[7 * kQfVS] = S;
        __syncthreads();
        // the horizontal 5-sums of a run of 8 output pixels, the cost (cv2's box scale with the 2^-14 units folded in,
        // an exact scaling, in double as cv2), the running first minimum
        const double C = 0x1p-14 * (1.0 / 25.0);
        const float bonus = k == 0 ? p.smooth : (k == kQfNC - 1 ? p.zero : 0.0f);
        uint32_t u[12];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const uint4 q = *reinterpret_cast<const uint4*>(&t.v[r8][c8 + 4 * i]);
            u[4 * i] = q.x; u[4 * i + 1] = q.y; u[4 * i + 2] = q.z; u[4 * i + 3] = q.w;
        }
        uint32_t H = u[0] + u[1] + u[2] + u[3];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            H += u[i + 4];
            const float c = __fsub_rn((float)(__dadd_rn(__hiloint2double(0x43300000, (int)H), -4503599627370496.0) * C), bonus);
            if (c < best[i]) {
                best[i] = c;
                pk[i] = k;
            }
            H -= u[i];
        }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) t.pick[r8][c8 + i] = (uint8_t)pk[i];
    __syncthreads();
    // the chosen candidate's vector
    const int lx = ex - kQfAp;
    if ((unsigned)lx >= (unsigned)kQfTW || X0 + lx >= p.w || Y0 + 8 * g >= p.h) return;
    const float2 lo = colField(br - 1), mid = colField(br), hi = colField(br + 1);
    float2* dst = p.pf + (size_t)qy0 * p.w + X0 + lx;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        if (j >= rows) break;
        const int k = t.pick[8 * g + j][lx];
        float2 v = make_float2(0.0f, 0.0f);
        if (k == 0) v = rowField(lo, mid, hi, j);
        else if (k < kQfNC - 1) v = t.bv[br + (k == 2 ? -1 : (k == 3 ? 1 : 0))][bx + (k == 4 ? -1 : (k == 5 ? 1 : 0))];
        dst[(size_t)j * p.w] = v;
    }
}
// interp.estimate :189-190, the mean of the sub-pixel pass' SADs in numpy's pairwise order, by the pixel-field launch's first
// CTAs (beside its tiles; the synthesis is the first to need the decision). A warp sums a leaf of the tree: the leaf in
// registers by 4 coalesced loads, handed round by shuffles in numpy's order. The CTA that completes the last leaf adds the
// inner nodes, one height per step, from shared memory: a chain of dependent global loads per leaf and height took ~15 us
// and was the tail of this launch (43 us at 4K, 17 us at 640x360).
__device__ __forceinline__ float leafSum(const float* a, int n, int lane, unsigned int& s256) {
    float v[4];
    unsigned int s = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        v[k] = lane + 32 * k < n ? __ldcg(a + lane + 32 * k) : 0.0f;
        s += (unsigned int)__float2int_rn(__fmul_rn(v[k], 256.0f));
    }
    s256 = __reduce_add_sync(0xffffffffu, s);
    const int body = n >= 8 ? n - n % 8 : 0;   // below 8 elements they are added one by one from 0
    float res = 0.0f;
    if (body) {
        float r = v[0];   // lanes 0..7: numpy's 8 accumulators
#pragma unroll
        for (int m = 1; m < 16; m++) {
            const float x = __shfl_sync(0xffffffffu, v[m / 4], 8 * (m % 4) + (lane & 7));
            if (8 * m < body) r = __fadd_rn(r, x);
        }
        const float p2 = __fadd_rn(r, __shfl_down_sync(0xffffffffu, r, 1));      // lane 2k: r[2k] + r[2k + 1]
        const float p4 = __fadd_rn(p2, __shfl_down_sync(0xffffffffu, p2, 2));    // lane 4k: (r0 + r1) + (r2 + r3)
        res = __fadd_rn(p4, __shfl_down_sync(0xffffffffu, p4, 4));
    }
    for (int i = body; i < n; i++) {
        const float x = i < 32 ? v[0] : (i < 64 ? v[1] : (i < 96 ? v[2] : v[3]));
        res = __fadd_rn(res, __shfl_sync(0xffffffffu, x, i & 31));
    }
    return res;   // lane 0
}
__device__ __forceinline__ void cutMeanQCta(const PixfieldParams& p, int cta, uint32_t* sm, size_t smBytes) {
    const CutPlan& pl = p.plan;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, leaf = cta * 8 + warp;
    __shared__ unsigned int last, tot;
    if (leaf < pl.nLeaves) {
        const int2 lf = pl.leaves[leaf];
        unsigned int s256;
        const float v = leafSum(p.sads + lf.x, lf.y, lane, s256);
        if (lane == 0) {
            pl.gvals[leaf] = v;
            pl.leafS256[leaf] = s256;
        }
    }
    // the ticket: the thread that takes it fences on both sides, between two barriers, so that it releases the leaves of all
    // 8 warps (a fence by the warps that wrote them would not: release goes by the order within the ticket's thread) and
    // acquires the other CTAs' for this one
    __syncthreads();
    if (tid == 0) {
        const unsigned int n = (unsigned int)min(8, pl.nLeaves - cta * 8);
        __threadfence();
        last = atomicAdd(&p.st->subDone, n) + n == (unsigned int)pl.nLeaves;
        __threadfence();
        tot = 0;
    }
    __syncthreads();
    if (!last) return;
    // node values and the inner nodes' operands in shared memory where they fit (else the values stay in gvals)
    const bool fits = (size_t)pl.nLeaves * 16 <= smBytes;
    float* vals = fits ? reinterpret_cast<float*>(sm) : pl.gvals;
    int2* inner = reinterpret_cast<int2*>(sm + 2 * pl.nLeaves);
    unsigned int s = 0;
    for (int i = tid; i < pl.nLeaves; i += 256) {
        s += __ldcg(pl.leafS256 + i);
        if (fits) vals[i] = __ldcg(pl.gvals + i);
        if (fits && i < pl.nInner) inner[i] = __ldg(pl.inner + i);
    }
    s = __reduce_add_sync(0xffffffffu, s);
    if (lane == 0) atomicAdd(&tot, s);
    __syncthreads();
    for (int d = 0; d < pl.nSteps; d++) {
        for (int j = pl.depthStart[d] + tid; j < pl.depthStart[d + 1]; j += 256) {
            if (fits) {
                const int2 c = inner[j];
                vals[pl.nLeaves + j] = __fadd_rn(vals[c.x], vals[c.y]);
            } else {
                const int2 c = __ldg(pl.inner + j);
                __stcg(pl.gvals + pl.nLeaves + j, __fadd_rn(__ldcg(pl.gvals + c.x), __ldcg(pl.gvals + c.y)));
                __threadfence();
            }
        }
        __syncthreads();
    }
    if (tid == 0) {
        const float mean = __fdiv_rn(fits ? vals[pl.root] : __ldcg(pl.gvals + pl.root), (float)(p.bw * p.bh));
        p.st->sadMean = mean;
        p.st->cut = mean > p.cutSad ? 1u : 0u;
        p.st->sadSum256 = tot;
        p.st->subDone = 0;
    }
}

// CTA `cta` of an item: the CTAs of the scene-cut mean, then the tiles in raster order
__device__ __forceinline__ void pixfieldQCta(const PixfieldParams& p, int cta) {
    __shared__ QfTile t;
    const int cutCtas = (p.plan.nLeaves + 7) / 8;
    if (cta < cutCtas) {
        cutMeanQCta(p, cta, &t.win[0][0], sizeof(t.win));
        return;
    }
    cta -= cutCtas;
    const int gx = (p.w + kQfTW - 1) / kQfTW;
    const int X0 = cta % gx * kQfTW, Y0 = cta / gx * kQfTH;
    // the block-field region, clamped to the field (a replicated entry stands for every block outside), and the range of
    // its vectors (in 1/32 px): every candidate is one of them or a blend
    const int bx0 = (X0 >> 3) - 2, by0 = (Y0 >> 3) - 2;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    static_assert(kQfBX * kQfBY == 96, "three warps hold the block-field region");
    if (tid < 96) {
        const float2 v = __ldg(p.v + clampi(by0 + tid / kQfBX, 0, p.bh - 1) * p.bw + clampi(bx0 + tid % kQfBX, 0, p.bw - 1));
        t.bv[tid / kQfBX][tid % kQfBX] = v;
        const float2 r = rne32bits(v);
        const int2 R = make_int2(__float_as_int(r.x) - 0x4B400000, __float_as_int(r.y) - 0x4B400000);
        t.bR[tid / kQfBX][tid % kQfBX] = R;
        const int4 m = make_int4(__reduce_min_sync(0xffffffffu, R.x), __reduce_min_sync(0xffffffffu, R.y),
                                 __reduce_max_sync(0xffffffffu, R.x), __reduce_max_sync(0xffffffffu, R.y));
        if (lane == 0) t.range[warp] = m;
    }
    if (tid == 96) t.differ = 0;
    __syncthreads();
    // a neighbour candidate that names the own block's vector everywhere costs the same at every pixel and can never be
    // the first minimum: it is left out (still scenes, wide uniform motion)
    if (tid < 96) {
        const int r = tid / kQfBX, c = tid % kQfBX;
        const int2 R = t.bR[r][c], u = t.bR[max(r - 1, 0)][c], d = t.bR[min(r + 1, kQfBY - 1)][c];
        const int2 l = t.bR[r][max(c - 1, 0)], e = t.bR[r][min(c + 1, kQfBX - 1)];
        auto ne = [&](const int2& q) { return q.x != R.x || q.y != R.y; };
        const uint32_t m = (ne(u) ? 4u : 0u) | (ne(d) ? 8u : 0u) | (ne(l) ? 16u : 0u) | (ne(e) ? 32u : 0u);
        const uint32_t any = __reduce_or_sync(0xffffffffu, m);
        if (lane == 0 && any) atomicOr(&t.differ, any);
    }
    const int4 r0 = t.range[0], r1 = t.range[1], r2 = t.range[2];
    const int nx = min(r0.x, min(r1.x, r2.x)), ny = min(r0.y, min(r1.y, r2.y));
    const int mx = max(r0.z, max(r1.z, r2.z)), my = max(r0.w, max(r1.w, r2.w));
    QfWin o;
    o.ax = X0 - kQfAp + ((-mx) >> 5);
    o.ay = Y0 - kQfAp + ((-my) >> 5);
    o.cx = X0 - kQfAp + (nx >> 5);
    o.cy = Y0 - kQfAp + (ny >> 5);
    // columns and rows (and the taps' lower row) from the origin to the other end of the range
    const int ww = kQfE + max(((-nx) >> 5) - ((-mx) >> 5), (mx >> 5) - (nx >> 5));
    const int wh = kQfTH + 2 * kQfAp + 1 + max(((-ny) >> 5) - ((-my) >> 5), (my >> 5) - (ny >> 5));
    if (ww > kQfWX || wh > kQfWY) {
        __syncthreads();
        pixfieldQTile<false>(p, t, o, X0, Y0);
        return;
    }
    if (min(o.ax, o.cx) >= 0 && min(o.ay, o.cy) >= 0 && max(o.ax, o.cx) + ww <= p.w && max(o.ay, o.cy) + wh <= p.h) {
        const uint32_t* qa = p.pa + (size_t)(o.ay + warp) * p.w + o.ax + lane;
        const uint32_t* qc = p.pc + (size_t)(o.cy + warp) * p.w + o.cx + lane;
        uint32_t* wa = t.win[0] + warp * kQfWX + lane;
        const bool more = lane + 64 < ww;
        for (int r = warp; r < wh; r += 8) {   // (ww >= 64)
            const uint32_t a0 = __ldg(qa), a1 = __ldg(qa + 32), c0 = __ldg(qc), c1 = __ldg(qc + 32);
            const uint32_t a2 = more ? __ldg(qa + 64) : 0u, c2 = more ? __ldg(qc + 64) : 0u;
            qa += 8 * p.w;
            qc += 8 * p.w;
            wa[0] = a0;
            wa[32] = a1;
            wa[kQfWY * kQfWX] = c0;
            wa[kQfWY * kQfWX + 32] = c1;
            if (more) {
                wa[64] = a2;
                wa[kQfWY * kQfWX + 64] = c2;
            }
            wa += 8 * kQfWX;
        }
    } else {
        for (int r = warp; r < wh; r += 8)
            for (int c = lane; c < ww; c += 32) {
                t.win[0][r * kQfWX + c] = ldPairClamped(p.pa, p.w, p.h, o.ax + c, o.ay + r);
                t.win[1][r * kQfWX + c] = ldPairClamped(p.pc, p.w, p.h, o.cx + c, o.cy + r);
            }
    }
    __syncthreads();
    pixfieldQTile<true>(p, t, o, X0, Y0);
}
// 3 CTAs per SM: 4 (64 registers) spill in every candidate's loop (640x360's estimate 40 us against 48, 1080p 75 against
// 83, 4K the same)
__global__ void __launch_bounds__(256, 3) k_pixfield_q(const PixfieldParams p) {
    pdlEnter();
    pixfieldQCta(p, blockIdx.x);
}
// grids of at most 2 CTAs per SM: the registers of a third one (an estimate at 640x360 36 -> 34 us, 1080p 69 -> 66; 4K, 1120
// CTAs, 143 -> 147)
__global__ void __launch_bounds__(256, 2) k_pixfield_q_lat(const PixfieldParams p) {
    pdlEnter();
    pixfieldQCta(p, blockIdx.x);
}
__global__ void __launch_bounds__(256, 3) k_pixfield_q_m(const __grid_constant__ Merged<PixfieldParams> m) {
    pdlEnter();
    int bx, by;
    const int i = mergedItem(m, bx, by);
    pixfieldQCta(m.item[i], bx);
}

__global__ void __launch_bounds__(256) k_unpair(const uint32_t* pair, float* out, size_t n) {
    pdlEnter();
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (i < n) out[i] = __fmul_rn(i2f((int)(__ldg(pair + i) & 0xFFFFu)), 1.0f / 16.0f);
}

// ============================================================================================== launchers
cudaError_t launchUnpair(const uint32_t* pair, float* out, size_t n, cudaStream_t s) {
    return launchPdl(k_unpair, dim3((unsigned int)((n + 255) / 256)), dim3(256), 0, s, pair, out, n);
}
// one item as a merged launch: its grid is one-dimensional. The per-pair launches have a block row per grid row, and a grid
// ends at 65535 rows (a frame of 1048560 rows at flowScale 2; the passes before and after go to 3.6 M).
constexpr int kGridRows = 65535;
template <class P>
static Merged<P> alone(const P& p) {
    Merged<P> m{};
    m.n = 1;
    m.item[0] = p;
    return m;
}
cudaError_t launchSearchQ(const SearchParams& p, cudaStream_t s) {
    if (p.bh > kGridRows) {
        Merged<SearchParams> m = alone(p);
        return launchSearchQMerged(m, s);
    }
    const dim3 grid(divUp(p.bw, 4), p.bh);
    if (p.R == 1) return launchPdl(p.pa ? k_search_q<1, true> : k_search_q<1, false>, grid, dim3(128), 0, s, p);
    return launchPdl(p.pa ? k_search_q<2, true> : k_search_q<2, false>, grid, dim3(128), 0, s, p);
}
cudaError_t launchSearchQMerged(Merged<SearchParams>& m, cudaStream_t s) {
    const int total = layoutMerged(m, [](const SearchParams& p, int& gx) {
        gx = (int)divUp(p.bw, 4);
        return gx * p.bh;
    });
    const bool pair = m.item[0].pa != nullptr;
    if (m.item[0].R == 1) return launchPdl(pair ? k_search_q_m<1, true> : k_search_q_m<1, false>, dim3(total), dim3(128), 0, s, m);
    return launchPdl(pair ? k_search_q_m<2, true> : k_search_q_m<2, false>, dim3(total), dim3(128), 0, s, m);
}
cudaError_t launchSubpixQ(const SubpixParams& p, cudaStream_t s) {
    if (p.bh > kGridRows) {
        Merged<SubpixParams> m = alone(p);
        return launchSubpixQMerged(m, s);
    }
    return launchPdl(k_subpix_q, dim3(divUp(p.bw, 4), p.bh), dim3(128), 0, s, p);
}
cudaError_t launchSubpixQMerged(Merged<SubpixParams>& m, cudaStream_t s) {
    const int total = layoutMerged(m, [](const SubpixParams& p, int& gx) {
        gx = (int)divUp(p.bw, 4);
        return gx * p.bh;
    });
    return launchPdl(k_subpix_q_m, dim3(total), dim3(128), 0, s, m);
}
static int pixfieldQCtas(const PixfieldParams& p) {
    return (int)(divUp(p.w, kQfTW) * divUp(p.h, kQfTH) + divUp(p.plan.nLeaves, 8));
}
cudaError_t launchPixfieldQ(const PixfieldParams& p, cudaStream_t s) {
    const int ctas = pixfieldQCtas(p);
    return launchPdl(ctas <= 2 * smCount() ? k_pixfield_q_lat : k_pixfield_q, dim3(ctas), dim3(256), 0, s, p);
}
cudaError_t launchPixfieldQMerged(Merged<PixfieldParams>& m, cudaStream_t s) {
    const int total = layoutMerged(m, [](const PixfieldParams& p, int& gx) { return gx = pixfieldQCtas(p); });
    return launchPdl(k_pixfield_q_m, dim3(total), dim3(256), 0, s, m);
}

}  // namespace fgk
