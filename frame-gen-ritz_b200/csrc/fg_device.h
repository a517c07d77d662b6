// fg_device.h -- device helpers shared by the kernels of the V1 path (fg_kernels.cu: 8-bit RGBA, fg_formats.cu: the
// other frame formats), the synthesis tile shape and its field stage, and the launch helper.
#pragma once
#include <cfloat>
#include <cstdint>

#include "fg_params.h"

namespace fgk {

// Programmatic dependent launch: every kernel is launched with programmatic stream serialisation, lets the next kernel
// of the stream be scheduled at once (its CTAs only occupy the slots this grid frees) and then waits for the previous
// grid to complete and its memory to be visible before touching anything an earlier kernel wrote. The launch latency
// of each small dependent pass overlaps the tail of the one before it.
__device__ __forceinline__ void pdlEnter() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// the item of this CTA in a merged launch and the CTA's coordinates in the item's own grid
template <class P>
__device__ __forceinline__ int mergedItem(const Merged<P>& m, int& bx, int& by) {
    const int b = (int)blockIdx.x;
    int lo = 0, hi = m.n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (m.first[mid] <= b) lo = mid; else hi = mid - 1;
    }
    const int l = b - m.first[lo], gx = m.gx[lo];
    bx = l % gx;
    by = l / gx;
    return lo;
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return min(max(v, lo), hi); }

// luma texel with clamp-to-edge (== cv2 BORDER_REPLICATE and the replicate pad_to_block, interp.py:68-70)
__device__ __forceinline__ float Lc(const float* __restrict__ L, int w, int h, int x, int y) {
    return __ldg(L + (size_t)clampi(y, 0, h - 1) * w + clampi(x, 0, w - 1));
}

// cv2.remap INTER_LINEAR / BORDER_REPLICATE of a float plane at (x, y): coordinates rounded half-even to 1/32 px,
// taps clamped one by one, ((p00 w00 + p01 w01) + p10 w10) + p11 w11 with w = (1 - fy)(1 - fx) ... in float.
__device__ __forceinline__ float remapF(const float* __restrict__ L, int w, int h, float x, float y) {
    const int X = __float2int_rn(__fmul_rn(x, 32.0f)), Y = __float2int_rn(__fmul_rn(y, 32.0f));
    const int ix = X >> 5, iy = Y >> 5;
    const float fx = (float)(X & 31) * (1.0f / 32.0f), fy = (float)(Y & 31) * (1.0f / 32.0f);
    const float gx = 1.0f - fx, gy = 1.0f - fy;
    const int x0 = clampi(ix, 0, w - 1), x1 = clampi(ix + 1, 0, w - 1);
    const size_t r0 = (size_t)clampi(iy, 0, h - 1) * w, r1 = (size_t)clampi(iy + 1, 0, h - 1) * w;
    const float p00 = __ldg(L + r0 + x0), p01 = __ldg(L + r0 + x1), p10 = __ldg(L + r1 + x0), p11 = __ldg(L + r1 + x1);
    float r = __fmul_rn(p00, __fmul_rn(gy, gx));
    r = __fadd_rn(r, __fmul_rn(p01, __fmul_rn(gy, fx)));
    r = __fadd_rn(r, __fmul_rn(p10, __fmul_rn(fy, gx)));
    r = __fadd_rn(r, __fmul_rn(p11, __fmul_rn(fy, fx)));
    return r;
}

// the same on the 2-channel float field (fw x fh float2)
__device__ __forceinline__ float2 remapF2(const float2* __restrict__ F, int w, int h, float x, float y) {
    const int X = __float2int_rn(__fmul_rn(x, 32.0f)), Y = __float2int_rn(__fmul_rn(y, 32.0f));
    const int ix = X >> 5, iy = Y >> 5;
    const float fx = (float)(X & 31) * (1.0f / 32.0f), fy = (float)(Y & 31) * (1.0f / 32.0f);
    const float gx = 1.0f - fx, gy = 1.0f - fy;
    const float w00 = __fmul_rn(gy, gx), w01 = __fmul_rn(gy, fx), w10 = __fmul_rn(fy, gx), w11 = __fmul_rn(fy, fx);
    const int x0 = clampi(ix, 0, w - 1), x1 = clampi(ix + 1, 0, w - 1);
    const size_t r0 = (size_t)clampi(iy, 0, h - 1) * w, r1 = (size_t)clampi(iy + 1, 0, h - 1) * w;
    const float2 p00 = __ldg(F + r0 + x0), p01 = __ldg(F + r0 + x1), p10 = __ldg(F + r1 + x0), p11 = __ldg(F + r1 + x1);
    float2 r;
    r.x = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(p00.x, w00), __fmul_rn(p01.x, w01)), __fmul_rn(p10.x, w10)), __fmul_rn(p11.x, w11));
    r.y = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(p00.y, w00), __fmul_rn(p01.y, w01)), __fmul_rn(p10.y, w10)), __fmul_rn(p11.y, w11));
    return r;
}

// cv2.cvtColor BGR2GRAY on 8-bit input as OpenCV 4.13 computes it (15-bit fixed point; checked on all 2^24 colours)
__device__ __forceinline__ int gray8(uint32_t px, int ri, int gi, int bi) {
    const int r = (px >> (8 * ri)) & 255, g = (px >> (8 * gi)) & 255, b = (px >> (8 * bi)) & 255;
    return (b * 3735 + g * 19235 + r * 9798 + 16384) >> 15;
}
// the same with the weights in 16-bit lanes for the two-way dot products (byte 0, byte 1) and (byte 2, byte 3) of a
// pixel: wlo = w(byte 0) | w(byte 1) << 16, whi = w(byte 2) (byte 3, alpha, weighs 0); exact integer arithmetic
__device__ __forceinline__ int gray8dp(uint32_t px, uint32_t wlo, uint32_t whi) {
    return (int)(__dp2a_hi(whi, px, __dp2a_lo(wlo, px, 16384u)) >> 15);
}

// Paired fp32 multiply / add (two IEEE operations per instruction). The compiler may fuse a paired multiply and add into
// one paired FMA whatever rounding is asked for, so these are used only where every product and sum is exact (dyadic
// operands with few significant bits): there a fused and an unfused evaluation give the same bits. Chains that round
// (the field at t, its upsampling, the warp positions) use the scalar __fmul_rn / __fadd_rn, which are never fused.
__device__ __forceinline__ float2 pmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }

// CrosshairV2's warp-tap rejection: does the UI mask m (header + bytes, fg_params.h UiV2Params) mark a pixel of the
// rectangle (ax0, ay0) .. (ax1, ay1) of at most kN x kN frame pixels? At most 4 pixels lie in two words of a row, and all rows'
// words are loaded before any is looked at: a thread's rows are neighbours, and with a byte at a time, each behind the
// one before, a tile on the overlay waited for up to 8 x 16 loads in a row (a protected synthesis with its fallback
// check and paste: P010 1366x768 69 -> 48 us, 8-bit RGBA 1280x720 28.9 -> 23.1, with one vote for three below).
template <int kN>
__device__ __forceinline__ bool uiHitSpan(const uint32_t* __restrict__ m, int ax0, int ay0, int ax1, int ay1) {
    static_assert(kN <= 4, "two words a row");
    const uint4 hd = __ldg(reinterpret_cast<const uint4*>(m));   // kUiMaskHeader words: -, origin, size, row stride
    const int ox = (int)(hd.y & 0xFFFFu), oy = (int)(hd.y >> 16), w = (int)(hd.z & 0xFFFFu), h = (int)(hd.z >> 16);
    const int x0 = max(ax0 - ox, 0), y0 = max(ay0 - oy, 0), x1 = min(ax1 - ox, w - 1), y1 = min(ay1 - oy, h - 1);
    if (x0 > x1 || y0 > y1) return false;
    const uint32_t* q = m + kUiMaskHeader + y0 * (int)hd.w + (x0 >> 2);
    const bool two = (x1 >> 2) != (x0 >> 2);
    const uint32_t lo = 0xFFFFFFFFu << (8 * (x0 & 3)), hi = 0xFFFFFFFFu >> (24 - 8 * (x1 & 3));
    uint32_t v0 = 0u, v1 = 0u;
#pragma unroll
    for (int j = 0; j < kN; j++) {
        const bool ok = y0 + j <= y1;
        v0 |= ok ? __ldg(q + j * (int)hd.w) : 0u;
        v1 |= ok && two ? __ldg(q + j * (int)hd.w + 1) : 0u;
    }
    return ((v0 & (two ? lo : lo & hi)) | (v1 & hi)) != 0u;
}
// the pixels that the bilinear tap whose position rounded to 1/32 px is (X, Y) (in 1/32 px) reads with a non-zero weight
// (gpu/shaders/ui_reject.glsl): lo = (X >> 5, Y >> 5) .. lo + (the fraction is not 0) per axis
__device__ __forceinline__ bool uiHitMask(const uint32_t* __restrict__ m, int X, int Y) {
    const int lx = X >> 5, ly = Y >> 5;
    return uiHitSpan<2>(m, lx, ly, lx + ((X & 31) != 0), ly + ((Y & 31) != 0));
}

// CrosshairV2's estimate fill of one level-0 cell by a warp (gpu/shaders/ui_v2_lumafill.comp): if the fs x fs pixels from
// (px, py) hold a UI pixel, the sum and count of luma(x, y) over the window's not-UI pixels, the window widened by fs px a
// side per step up to 8 px while it has none. True (in every lane) where a sum was formed. The lanes share a window's
// pixels: with one thread per cell the up to 660 dependent mask and pixel reads of a cell took 113 us of an estimate, now 13.
template <class Luma>
__device__ __forceinline__ bool uiFillWindow(const uint32_t* __restrict__ m, int W, int H, int fs, int px, int py, int lane, Luma luma,
                                             int& sum, int& n) {
    const uint32_t o = __ldg(m + 1), wh = __ldg(m + 2);
    const int ox = (int)(o & 0xFFFFu), oy = (int)(o >> 16), w = (int)(wh & 0xFFFFu), h = (int)(wh >> 16), stride = (int)__ldg(m + 3);
    auto ui = [&](int x, int y) {
        x -= ox;
        y -= oy;
        if (x < 0 || y < 0 || x >= w || y >= h) return false;
        return ((__ldg(m + kUiMaskHeader + y * stride + (x >> 2)) >> (8 * (x & 3))) & 255u) != 0u;
    };
    const int cx = px + (lane & (fs - 1)), cy = py + lane / fs;   // fs = 1, 2, 4
    if (!__any_sync(0xffffffffu, lane < fs * fs && cx < W && cy < H && ui(cx, cy))) return false;
    for (int k = 0; k <= 8; k += fs) {
        const int side = fs + 2 * k;
        int s = 0, c = 0;
        for (int i = lane; i < side * side; i += 32) {
            const int x = px - k + i % side, y = py - k + i / side;
            if (x < 0 || y < 0 || x >= W || y >= H || ui(x, y)) continue;
            s += luma(x, y);
            c++;
        }
        n = __reduce_add_sync(0xffffffffu, c);
        if (n > 0) {
            sum = __reduce_add_sync(0xffffffffu, s);
            return true;
        }
    }
    return false;
}

// the same for a YUV sample (gpu/shaders/ui_reject.glsl uiFootprint, FG_YUV): the 2x2 texels of the half-resolution
// chroma plane around it, c = X - 16 in 1/64 chroma texels, i = c >> 6, the second texel only if the fraction is not
// 0: the pixels 2 i .. 2 (i + n) + 1 per axis, which contain the luma taps too
__device__ __forceinline__ bool uiHitMaskYuv(const uint32_t* __restrict__ m, int X, int Y) {
    const int cx = X - 16, cy = Y - 16, ix = cx >> 6, iy = cy >> 6;
    return uiHitSpan<4>(m, 2 * ix, 2 * iy, 2 * (ix + ((cx & 63) != 0)) + 1, 2 * (iy + ((cy & 63) != 0)) + 1);
}

// round-half-even(x * 32) for |x * 32| < 2^22 (cv2's saturate_cast<int>(x * INTER_TAB_SIZE)), as the float's bits
__device__ __forceinline__ float2 rne32bits(float2 v) {
    return __ffma2_rn(v, make_float2(32.0f, 32.0f), make_float2(12582912.0f, 12582912.0f));
}
__device__ __forceinline__ int rne32(float x) { return __float_as_int(__fmaf_rn(x, 32.0f, 12582912.0f)) - 0x4B400000; }
// exact float of 0 <= i < 2^23
__device__ __forceinline__ float i2f(int i) { return __int_as_float(0x4B000000 | i) - 8388608.0f; }
// floor of 0 <= v < 2^23
__device__ __forceinline__ int floorPos(float v) { return __float_as_int(__fadd_rz(v, 8388608.0f)) - 0x4B000000; }

__device__ __forceinline__ float warpSum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ============================================================================================== luma tower
constexpr int kTowerFloats = 1024 + 256 + 64 + 16 + 4 + 2;   // a 32x32 level-0 tile and its 16x16 .. 1x1 levels above

// round half-even to a multiple of 2^-10 (the grid of the other formats' coarse pyramid levels)
__device__ __forceinline__ float round10(float v) { return __fmul_rn(rintf(__fmul_rn(v, 1024.0f)), 1.0f / 1024.0f); }

// one pixel (lx, ly) of level L of a tile's tower: the mean of the valid 2x2 pixels below it (sum * 1/4 when full,
// sum / count at the odd edges), stored and kept in sl. ROUND: rounded to 2^-10.
template <bool ROUND, int L>
__device__ __forceinline__ void towerPx(const LumaPyrParams& p, float (*sl)[kTowerFloats], int tx0, int ty0, int lx, int ly) {
    constexpr int side = 32 >> (L - 1), ns = side / 2;
    constexpr int off = L == 1 ? 0 : L == 2 ? 1024 : L == 3 ? 1280 : L == 4 ? 1344 : 1360, noff = off + side * side;
    const int X = (tx0 >> L) + lx, Y = (ty0 >> L) + ly;
    float va = 0.0f, vc = 0.0f;
    if (X < p.lw[L] && Y < p.lh[L]) {
        const float* a = sl[0] + off + 2 * ly * side + 2 * lx;
        const float* c = sl[1] + off + 2 * ly * side + 2 * lx;
        const bool fx = 2 * X + 1 < p.lw[L - 1], fy = 2 * Y + 1 < p.lh[L - 1];
        float sa = a[0], sc = c[0];
        if (fx && fy) {
            va = __fmul_rn(__fadd_rn(__fadd_rn(__fadd_rn(sa, a[1]), a[side]), a[side + 1]), 0.25f);
            vc = __fmul_rn(__fadd_rn(__fadd_rn(__fadd_rn(sc, c[1]), c[side]), c[side + 1]), 0.25f);
        } else if (fx || fy) {
            const int o = fx ? 1 : side;
            va = __fmul_rn(__fadd_rn(sa, a[o]), 0.5f);
            vc = __fmul_rn(__fadd_rn(sc, c[o]), 0.5f);
        } else {
            va = sa;
            vc = sc;
        }
        if (ROUND) { va = round10(va); vc = round10(vc); }
        p.la[L][(size_t)Y * p.lw[L] + X] = va;
        p.lc[L][(size_t)Y * p.lw[L] + X] = vc;
    }
    sl[0][noff + ly * ns + lx] = va;
    sl[1][noff + ly * ns + lx] = vc;
}

// interp.pyramid :73-77 above one 32x32 level-0 tile held in sl[.][0..1023] (tx0, ty0: the tile's origin): levels
// 1 .. p.nlev-1 of the tile's tower, written to p.la / p.lc: level 1 by the whole CTA (a pixel per thread), the rest by
// the first warp alone (no CTA barrier).
template <bool ROUND>
__device__ __forceinline__ void lumaTower(const LumaPyrParams& p, float (*sl)[kTowerFloats], int tx0, int ty0) {
    const int t = threadIdx.x;
    if (p.nlev < 2) return;
    towerPx<ROUND, 1>(p, sl, tx0, ty0, t & 15, t >> 4);
    if (p.nlev < 3) return;
    __syncthreads();
    if (t >= 32) return;
    towerPx<ROUND, 2>(p, sl, tx0, ty0, t & 7, t >> 3);
    towerPx<ROUND, 2>(p, sl, tx0, ty0, t & 7, (t >> 3) + 4);
    __syncwarp();
    if (p.nlev < 4 || t >= 16) return;
    towerPx<ROUND, 3>(p, sl, tx0, ty0, t & 3, t >> 2);
    __syncwarp(0xffffu);
    if (p.nlev < 5 || t >= 4) return;
    towerPx<ROUND, 4>(p, sl, tx0, ty0, t & 1, t >> 1);
    __syncwarp(0xfu);
    if (p.nlev < 6 || t) return;
    towerPx<ROUND, 5>(p, sl, tx0, ty0, 0, 0);
}

// q = 16 x a level-0 luma value (a multiple of 1/16, at most 255) in the low 16 bits, as the float's bits
__device__ __forceinline__ uint32_t q16(float v) { return (uint32_t)__float_as_int(__fmaf_rn(v, 16.0f, 8388608.0f)); }

// the pair-plane words (LumaPyrParams::pa / pc) of a 32x32 level-0 tile held in sl[.][0..1023]: pixel x's word is the
// tile's own but for its column 31, whose high half belongs to the next tile's column 0 (each tile writes that half of
// the word to its left)
__device__ __forceinline__ void storePairs(const LumaPyrParams& p, const float (*sl)[kTowerFloats], int tx0, int ty0) {
    const int fw = p.lw[0], fh = p.lh[0];
    const int lx = threadIdx.x & 31, x = tx0 + lx;
    if (x >= fw) return;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        uint32_t* plane = k ? p.pc : p.pa;
        for (int ly = threadIdx.x >> 5; ly < 32 && ty0 + ly < fh; ly += 8) {
            uint32_t* o = plane + (size_t)(ty0 + ly) * fw + x;
            const uint32_t q = q16(sl[k][ly * 32 + lx]);
            if (x == fw - 1) *o = __byte_perm(q, q, 0x5410);
            else if (lx < 31) *o = __byte_perm(q, q16(sl[k][ly * 32 + lx + 1]), 0x5410);
            else *reinterpret_cast<unsigned short*>(o) = (unsigned short)q;
            if (lx == 0 && x > 0) reinterpret_cast<unsigned short*>(o)[-1] = (unsigned short)q;
        }
    }
}

// the pair words of two neighbouring pixels of a row (q0, q1; next: the pixel to their right) at the 8-byte aligned o;
// edge: the second word's high half is the next tile's; left: this tile writes the high half of the word to its left
__device__ __forceinline__ void storePairs2(uint32_t* o, uint32_t q0, uint32_t q1, uint32_t next, bool edge, bool left) {
    const uint32_t w0 = q0 | (q1 << 16);
    if (edge) {
        o[0] = w0;
        *reinterpret_cast<unsigned short*>(o + 1) = (unsigned short)q1;
    } else {
        *reinterpret_cast<uint2*>(o) = make_uint2(w0, q1 | (next << 16));
    }
    if (left) reinterpret_cast<unsigned short*>(o)[-1] = (unsigned short)q0;
}

// a level-0 value rewritten after the luma pass (CrosshairV2's estimate fill): its two halves in the pair plane
__device__ __forceinline__ void storePairPx(uint32_t* plane, int fw, int x, int y, float v) {
    unsigned short* o = reinterpret_cast<unsigned short*>(plane + (size_t)y * fw + x);
    const unsigned short q = (unsigned short)q16(v);
    o[0] = q;
    if (x > 0) o[-1] = q;
    if (x == fw - 1) o[1] = q;
}

// ============================================================================================== synthesis tile
// 64 x 64 mismatch region -> 58 x 58 output tile: the square tile recomputes the least halo (1.22 region pixels per
// output pixel, against 1.29 for 128 x 32) within the shared memory of 3 CTAs per SM.
//
// The synthesis kernels are bound by instruction issue and by the latency of the sample loads (8-bit RGBA at 3840x2160,
// t = 1/2: 74 % issue, 62.6 M warp instructions, 82.9 us under ncu; back to back with the fallback check 79.5 us, 92.3 before
// the rows of a thread became consecutive with the upsampled field in registers, interior tiles went without clamps, the
// row sums became byte dot products and fully trusted warps only blend; t = 1/3 110 -> 94 us). Other shapes measured within
// 3 % of it (64 x 60 with 4 x 384 threads, 64 x 72) or slower (64 x 40, 64 x 48). The forms of three CTAs per SM spill up
// to 48 bytes a thread at their 40 registers (-Xptxas -v); two CTAs per SM spill nothing and are slower on large grids but
// for Nv12 (fmtCtas).
constexpr int kSyE = 64, kSyEH = 64, kSyAp = 3;
constexpr int kSyT = kSyE - 2 * kSyAp, kSyTH = kSyEH - 2 * kSyAp;
constexpr int kSyThreads = 512, kSyK = kSyEH / (kSyThreads / kSyE);   // region rows per thread (512 = 64 columns x 8)
constexpr size_t kSyWarpBytes = (size_t)2 * kSyTH * kSyE * 4;   // k_synth: both warps of the output rows, after the row sums
// the output row (tile coordinates) of a thread's k-th output pixel: thread rows ey0 = 0..7 take kSyK consecutive rows
// each (the last only kSyTH - 7 kSyK of them), so the vertical 7-sums run as a sliding window
__device__ __forceinline__ int syOutRow(int ey0, int k) { return ey0 * kSyK + k; }
// row strides of the mismatch plane e (bytes) and of its horizontal 7-sums (uint16): one word of padding per row, so
// that the lanes of a warp can walk 32 different rows of one column group without bank conflicts
constexpr int kSyES = kSyE + 4, kSyHS = kSyE + 2;

// cv2.remap INTER_LINEAR / BORDER_REPLICATE of the 2-channel float field at (x, y): quantisation and weights paired
// (exact), the taps' weighted sum as cv2 rounds it, ((p00 w00 + p01 w01) + p10 w10) + p11 w11 per channel (paired
// products, scalar sums: never fused). One address where the four taps lie inside the field; kLat: clamped, without the
// branch (a latency form has the instructions to spare).
template <bool kLat>
__device__ __forceinline__ float2 remapF2m(const float2* __restrict__ F, int w, int h, float x, float y) {
    const float2 bits = rne32bits(make_float2(x, y));
    const int X = __float_as_int(bits.x) - 0x4B400000, Y = __float_as_int(bits.y) - 0x4B400000;
    const int ix = X >> 5, iy = Y >> 5;
    const float2 f = pmul(make_float2(i2f(X & 31), i2f(Y & 31)), make_float2(1.0f / 32.0f, 1.0f / 32.0f));
    const float2 g = padd(make_float2(1.0f, 1.0f), make_float2(-f.x, -f.y));
    const float2 wA = pmul(make_float2(g.y, g.y), make_float2(g.x, f.x));   // (w00, w01)
    const float2 wB = pmul(make_float2(f.y, f.y), make_float2(g.x, f.x));   // (w10, w11)
    float2 p00, p01, p10, p11;
    if (!kLat && (unsigned)ix < (unsigned)(w - 1) && (unsigned)iy < (unsigned)(h - 1)) {
        const float2* q = F + (iy * w + ix);
        p00 = __ldg(q);
        p01 = __ldg(q + 1);
        p10 = __ldg(q + w);
        p11 = __ldg(q + w + 1);
    } else {
        const int x0 = clampi(ix, 0, w - 1), x1 = clampi(ix + 1, 0, w - 1);
        const size_t r0 = (size_t)clampi(iy, 0, h - 1) * w, r1 = (size_t)clampi(iy + 1, 0, h - 1) * w;
        p00 = __ldg(F + r0 + x0); p01 = __ldg(F + r0 + x1); p10 = __ldg(F + r1 + x0); p11 = __ldg(F + r1 + x1);
    }
    const float2 m00 = pmul(p00, make_float2(wA.x, wA.x)), m01 = pmul(p01, make_float2(wA.y, wA.y));
    const float2 m10 = pmul(p10, make_float2(wB.x, wB.x)), m11 = pmul(p11, make_float2(wB.y, wB.y));
    return make_float2(__fadd_rn(__fadd_rn(__fadd_rn(m00.x, m01.x), m10.x), m11.x),
                       __fadd_rn(__fadd_rn(__fadd_rn(m00.y, m01.y), m10.y), m11.y));
}

struct SyCoef {   // one region column (or row): upsampling taps (relative to the tile's field region) and weights
    int i0, i1;
    float a0, a1;   // rows: already x fs (scaling by a power of 2 commutes with the rounding)
    float pos;      // the clamped pixel coordinate
};

// the clamped pixel of region column (or row) e, and cv2 resize's left tap and fraction of it, (d + 1/2) / fs - 1/2 in
// units of 1 / (2 fs): s = floor, rem the remainder (d: the crop [:H, :W] / edge pad of the upsampled field)
__device__ __forceinline__ int syPx(int e, int origin, int n) { return clampi(origin - kSyAp + e, 0, n - 1); }
__device__ __forceinline__ int syTap(int p, int un, int fs, int sh, int& rem) {
    const int num = 2 * min(p, un - 1) + 1 - fs;
    rem = num & (2 * fs - 1);
    return num >> sh;
}
__device__ __forceinline__ SyCoef syCoef(int e, int origin, int n, int un, int fn, int g0, int fs, float wscale, bool xaxis) {
    SyCoef c;
    const int p = syPx(e, origin, n), sh = fs == 1 ? 1 : (fs == 2 ? 2 : 3);
    int rem, s = syTap(p, un, fs, sh, rem);
    float f = __fmul_rn(i2f(rem), fs == 1 ? 0.5f : (fs == 2 ? 0.25f : 0.125f));   // exact
    if (xaxis) {   // cv2 resize: x weights forced to (1, 0) beyond the borders; y rows clamped, weights kept
        if (s < 0) { s = 0; f = 0.0f; }
        if (s >= fn - 1) { s = fn - 1; f = 0.0f; }
    }
    c.i0 = clampi(s, 0, fn - 1) - g0;
    c.i1 = clampi(s + 1, 0, fn - 1) - g0;
    c.a0 = __fmul_rn(1.0f - f, wscale);
    c.a1 = __fmul_rn(f, wscale);
    c.pos = (float)p;
    return c;
}

// One region row of a synthesis tile: (upsampling taps i0 | i1 << 16 relative to the tile's field region, weights x fs,
// the clamped pixel coordinate)
__device__ __forceinline__ float4 syRow(const SyCoef& c) { return make_float4(__int_as_float(c.i0 | (c.i1 << 16)), c.a0, c.a1, c.pos); }

// The field stage of a synthesis tile, shared by the kernels of every format: the tile's field region g (GW columns),
// the row coefficients (rowc) and this thread's column coefficients; the field at t on the region (interp.field_at:
// g <- pf(q - s g), twice, from g = pf(q)). Carves the dynamic shared memory sm into the field region, the mismatch
// plane e and the row sums hsum. Ends with a barrier.
//
// `in` (uniform over the CTA): flowScale 2, no coordinate of the tile clamped, and no warp of the tile, whatever blend of
// the region's vectors it takes, reaches within 2 px of the frame's border: the rows then follow a fixed pattern and
// the samples need no clamps. On a 4K frame 92 % of the tiles.
//
// `ui` (kUi; uniform over the CTA): some tap of the tile, with the footprint of any format, may touch a UI mask's rectangle.
// The other tiles need no rejection and run as a plain synthesis' (3840x2160: 115 -> 97 us a synthesis
// with its fallback check and paste; 81 without the protection).
struct SyField {
    const float2* g;
    int GW, gx0;
    SyCoef cx;
    bool in, ui;
};
// how far a tap of the region of tile origin `o` must move along an axis to touch [lo, lo + n) (4 px of footprint kept)
__device__ __forceinline__ int uiGap(int o, int side, int lo, int n) {
    return max(o - kSyAp - 4 - (lo + n - 1), lo - 4 - (o - kSyAp + side - 1));
}
// kSplit: a loop for the lookup at t and one for the plain field, the vectors' largest parts voted on after it. The 8-bit
// kernels, the latency forms and the protected ones gain by it (8-bit 1280x720 17.9 -> 17.4 us, unrelated frames of 1920x1080
// 27.0 -> 26.6); the formats' 40-register kernels lose 1 % at 3840x2160 and keep one loop.
template <bool kUi, bool kLat, bool kSplit>
__device__ __forceinline__ SyField syFieldStage(const SynthParams& p, int X0, int Y0, int tid, int ex, float4* rowc,
                                                unsigned char* sm, uint8_t*& e, unsigned short*& hsum) {
    const int fs = p.fs, uw = p.fw * fs, uh = p.fh * fs, sh = fs == 1 ? 1 : (fs == 2 ? 2 : 3);
    int rem;
    // the field region: from the first pixel's left tap to the last one's right tap (every thread, no barrier)
    const int gx0 = clampi(syTap(syPx(0, X0, p.W), uw, fs, sh, rem), 0, p.fw - 1);
    const int gy0 = clampi(syTap(syPx(0, Y0, p.H), uh, fs, sh, rem), 0, p.fh - 1);
    const int GW = clampi(syTap(syPx(kSyE - 1, X0, p.W), uw, fs, sh, rem) + 1, 0, p.fw - 1) - gx0 + 1;
    const int GH = clampi(syTap(syPx(kSyEH - 1, Y0, p.H), uh, fs, sh, rem) + 1, 0, p.fh - 1) - gy0 + 1;
    const float fsf = (float)fs;
    if (tid < kSyEH) rowc[tid] = syRow(syCoef(tid, Y0, p.H, uh, p.fh, gy0, fs, fsf, false));
    SyField f;
    f.cx = syCoef(ex, X0, p.W, uw, p.fw, gx0, fs, 1.0f, true);
    float2* g = reinterpret_cast<float2*>(sm);             // GH x GW
    f.g = g;
    f.GW = GW;
    f.gx0 = gx0;
    e = reinterpret_cast<uint8_t*>(g + GW * GH);           // kSyEH rows of kSyES bytes
    hsum = reinterpret_cast<unsigned short*>(e + kSyEH * kSyES);   // kSyEH rows of kSyHS (columns < kSyT used)
    // the room for |(2t) h|, |2(1 - t) h| (h: fs x a vector of the region) on each axis, negative where none is left
    const float kf = p.mid ? fsf : __fmul_rn(fmaxf(p.ka, p.kc), fsf);
    const int Ht = min(p.H, uh), Wt = min(p.W, uw);
    const bool wide = fs != 2 || (uint64_t)p.H * (p.pitch >> 2) >= 0xF0000000u;
    const float mx = wide ? -1.0f : (float)(min(X0 - kSyAp, Wt - (X0 - kSyAp + kSyE)) - 3);
    const float my = wide ? -1.0f : (float)(min(Y0 - kSyAp, Ht - (Y0 - kSyAp + kSyEH)) - 3);
    float gapX = FLT_MAX, gapY = FLT_MAX;   // the moves along each axis below which no tap touches a mask's rectangle
    if (kUi) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint32_t* m = k ? p.uiC : p.uiA;
            const uint32_t o = m ? __ldg(m + 1) : 0u, wh = m ? __ldg(m + 2) : 0u;
            if (wh == 0u) continue;
            gapX = fminf(gapX, (float)uiGap(X0, kSyE, (int)(o & 0xFFFFu), (int)(wh & 0xFFFFu)));
            gapY = fminf(gapY, (float)uiGap(Y0, kSyEH, (int)(o >> 16), (int)(wh >> 16)));
        }
    }
    // the region's GW x GH samples spread over all threads (GW is about half the CTA's width at flowScale 2): row
    // r = floor((i + 0.5) / GW), exact in float for these sizes (the quotient stays >= 0.5 / GW from an integer)
    const float invGW = 1.0f / (float)GW;
    auto sample = [&](int i, bool lookup) {
        const int r = (int)__fmul_rz(__int2float_rn(i) + 0.5f, invGW), c = i - r * GW;
        const int qx = gx0 + c, qy = gy0 + r;
        float2 v = __ldg(p.pf + (size_t)qy * p.fw + qx);
        if (lookup) {
            const float fx = (float)qx, fy = (float)qy;
#pragma unroll
            for (int it = 0; it < 2; it++)
                v = remapF2m<kLat>(p.pf, p.fw, p.fh, __fsub_rn(fx, __fmul_rn(p.s, v.x)), __fsub_rn(fy, __fmul_rn(p.s, v.y)));
        }
        g[i] = v;
        return v;
    };
    bool out = false, nearX = false, nearY = false;
    if (kSplit) {
        uint32_t ax = 0, ay = 0;   // the largest |v.x|, |v.y| as bits (a NaN is above every number)
        auto largest = [&](float2 v) {
            ax = max(ax, __float_as_uint(fabsf(v.x)));
            ay = max(ay, __float_as_uint(fabsf(v.y)));
        };
        if (p.lookup)
            for (int i = tid; i < GW * GH; i += kSyThreads) largest(sample(i, true));
        else
            for (int i = tid; i < GW * GH; i += kSyThreads) largest(sample(i, false));
        const float vx = __uint_as_float(ax) * kf, vy = __uint_as_float(ay) * kf;
        out = !(vx <= mx) || !(vy <= my);   // (a NaN is out too)
        nearX = !(vx < gapX);
        nearY = !(vy < gapY);
    } else {
        static_assert(kSplit || !kUi, "the protected kernels vote after the loop");
        for (int i = tid; i < GW * GH; i += kSyThreads) {
            const float2 v = sample(i, p.lookup);
            out |= !(fabsf(v.x) * kf <= mx) || !(fabsf(v.y) * kf <= my);
        }
    }
    f.ui = false;
    if (kUi) {   // three votes, one barrier
        __shared__ uint32_t vote[kSyThreads / 32];
        const uint32_t mine = __reduce_or_sync(0xffffffffu, (out ? 1u : 0u) | (nearX ? 2u : 0u) | (nearY ? 4u : 0u));
        if ((tid & 31) == 0) vote[tid >> 5] = mine;
        __syncthreads();
        const uint32_t all = __reduce_or_sync(0xffffffffu, vote[tid & (kSyThreads / 32 - 1)]);
        f.in = !(all & 1u);
        f.ui = (all & 6u) == 6u;
    } else {
        f.in = !__syncthreads_or(out);
    }
    return f;
}

// this thread's column of the horizontally upsampled field (cv2 resize: h = S0 a0 + S1 a1) at region row r
__device__ __forceinline__ float2 syColField(const SyField& f, int r) {
    const float2 s0 = f.g[r * f.GW + f.cx.i0], s1 = f.g[r * f.GW + f.cx.i1];
    return make_float2(__fadd_rn(__fmul_rn(s0.x, f.cx.a0), __fmul_rn(s1.x, f.cx.a1)),
                       __fadd_rn(__fmul_rn(s0.y, f.cx.a0), __fmul_rn(s1.y, f.cx.a1)));
}
// the vertical stage (x fs folded into the weights): the half-vector between two rows of it
__device__ __forceinline__ float2 syLerp(float2 h0, float2 h1, float a0, float a1) {
    return make_float2(__fadd_rn(__fmul_rn(h0.x, a0), __fmul_rn(h1.x, a1)), __fadd_rn(__fmul_rn(h0.y, a0), __fmul_rn(h1.y, a1)));
}

// Walks this thread's kSyK consecutive region rows (ey0 kSyK ..) top down and hands each to f(k, ey, posy, h). kIn (SyField
// ::in): rows follow flowScale 2's pattern, the tile's first row odd: two rows share their pair of field rows, weights
// (3/4, 1/4) and (1/4, 3/4) x 2. Else from the row coefficients, a field row loaded when the pair moves on. kRows rows
// per loop round: the 8-bit kernels stay rolled (2) where many CTAs share an SM (a 4K synthesis at t = 1/2: 78 us rolled,
// 83 us unrolled) and unroll (8) for grids of about one CTA per SM. kFlat: both field rows read for every row, no branch between
// the samples of neighbouring rows: for the latency forms, and for the border tiles of the 8-bit kernels, which
// end a small grid (with the mixed-trust rows unrolled: 1280x720 17.9 -> 16.9 us, 1920x1080 at flowScale 4 26.1 -> 24.7).
template <bool kIn, int kRows, bool kFlat = false, class F>
__device__ __forceinline__ void syWalk(const SyField& f, const float4* rowc, int ey0, F&& fn) {
    if (kIn) {
        const float y0 = rowc[ey0 * kSyK].w;
        float2 h0 = syColField(f, ey0 * (kSyK / 2));
#pragma unroll (kRows / 2)
        for (int k = 0; k < kSyK; k += 2) {
            const float2 h1 = syColField(f, ey0 * (kSyK / 2) + k / 2 + 1);
            fn(k, ey0 * kSyK + k, y0 + (float)k, syLerp(h0, h1, 1.5f, 0.5f));
            fn(k + 1, ey0 * kSyK + k + 1, y0 + (float)(k + 1), syLerp(h0, h1, 0.5f, 1.5f));
            h0 = h1;
        }
    } else {
        int c0 = -1, c1 = -1;
        float2 h0 = make_float2(0.0f, 0.0f), h1 = h0;
#pragma unroll kRows
        for (int k = 0; k < kSyK; k++) {
            const float4 r = rowc[ey0 * kSyK + k];
            const int i0 = __float_as_int(r.x) & 0xFFFF, i1 = __float_as_int(r.x) >> 16;
            if (kFlat) {   // no branch between the rows' samples
                fn(k, ey0 * kSyK + k, r.w, syLerp(syColField(f, i0), syColField(f, i1), r.y, r.z));
                continue;
            }
            if (i0 != c0) {   // uniform over the warp
                h0 = i0 == c1 ? h1 : syColField(f, i0);
                c0 = i0;
            }
            if (i1 != c1) {
                h1 = syColField(f, i1);
                c1 = i1;
            }
            fn(k, ey0 * kSyK + k, r.w, syLerp(h0, h1, r.y, r.z));
        }
    }
}

// Stage 3 of a synthesis tile: the horizontal 7-sums of the mismatch plane, one region row and 8 output columns per
// thread, as byte dot products with masks of ones (words w0 .. w3 hold columns c0 .. c0 + 15; the last group's columns
// past the region belong to outputs that no one reads); the lanes of a warp take the 32 rows of one column group
// (conflict-free strides)
__device__ __forceinline__ void syRowSums(const uint8_t* e, unsigned short* hsum, int tid) {
    const int r = tid & (kSyEH - 1), c0 = (tid / kSyEH) * 8;
    const uint32_t* q = reinterpret_cast<const uint32_t*>(e + r * kSyES + c0);
    const bool more = c0 + 8 < kSyE;
    const uint32_t w0 = q[0], w1 = q[1], w2 = more ? q[2] : 0u, w3 = more ? q[3] : 0u;
    const uint32_t m1 = __dp4a(w1, 0x01010101u, 0u), m2 = __dp4a(w2, 0x01010101u, 0u);
    const uint32_t s0 = __dp4a(w0, 0x01010101u, __dp4a(w1, 0x00010101u, 0u)), s1 = __dp4a(w0, 0x01010100u, m1);
    const uint32_t s2 = __dp4a(w0, 0x01010000u, __dp4a(w2, 0x00000001u, m1)), s3 = __dp4a(w0, 0x01000000u, __dp4a(w2, 0x00000101u, m1));
    const uint32_t s4 = __dp4a(w2, 0x00010101u, m1), s5 = __dp4a(w1, 0x01010100u, m2);
    const uint32_t s6 = __dp4a(w1, 0x01010000u, __dp4a(w3, 0x00000001u, m2)), s7 = __dp4a(w1, 0x01000000u, __dp4a(w3, 0x00000101u, m2));
    uint32_t* o = reinterpret_cast<uint32_t*>(hsum + r * kSyHS + c0);   // sums below 2^11: two per word
    o[0] = s0 | (s1 << 16);
    o[1] = s2 | (s3 << 16);
    o[2] = s4 | (s5 << 16);
    o[3] = s6 | (s7 << 16);
}

// ============================================================================================== scene-cut mean, spread
// One leaf of the pairwise tree by one warp, in numpy's order: lanes 0..7 are its 8 accumulators (independent loads),
// combined as ((r0 + r1) + (r2 + r3)) + ((r4 + r5) + (r6 + r7)), then the tail; leaves under 8 elements by lane 0
// alone. Also returns (in every lane) the leaf's sum of roundEven(sad * 256), the debug counter's share.
__device__ __forceinline__ float warpLeafSum(const float* a, int n, int lane, unsigned int& s256) {
    unsigned int s = 0;
    for (int i = lane; i < n; i += 32) s += (unsigned int)__float2int_rn(__fmul_rn(__ldcg(a + i), 256.0f));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    s256 = s;
    float res = 0.0f;
    if (n < 8) {
        if (lane == 0)
            for (int i = 0; i < n; i++) res = __fadd_rn(res, __ldcg(a + i));
        return __shfl_sync(0xffffffffu, res, 0);
    }
    const int body = n - (n % 8);
    float r = 0.0f;
    if (lane < 8) {
        r = __ldcg(a + lane);
        for (int i = 8 + lane; i < body; i += 8) r = __fadd_rn(r, __ldcg(a + i));
    }
    const float r1 = __shfl_down_sync(0xffffffffu, r, 1);   // lane 2k: r[2k] + r[2k+1]
    const float p2 = __fadd_rn(r, r1);
    const float p2b = __shfl_down_sync(0xffffffffu, p2, 2);  // lane 4k: (r0 + r1) + (r2 + r3)
    const float p4 = __fadd_rn(p2, p2b);
    const float p4b = __shfl_down_sync(0xffffffffu, p4, 4);
    if (lane == 0) {
        res = __fadd_rn(p4, p4b);
        for (int i = body; i < n; i++) res = __fadd_rn(res, __ldcg(a + i));
    }
    return __shfl_sync(0xffffffffu, res, 0);
}

// leaf `leaf` of the scene-cut mean (its SADs complete and visible), by one warp; the warp that completes the last leaf
// adds the inner nodes, one height per step, and writes the mean, the cut decision and the debug counter
__device__ __forceinline__ void cutMeanLeaf(const CutPlan& pl, const float* sads, int nb, float cutSad, DevState* st, int leaf,
                                            int lane) {
    const int2 lf = pl.leaves[leaf];
    unsigned int s256;
    const float v = warpLeafSum(sads + lf.x, lf.y, lane, s256);
    unsigned int done = 0;
    if (lane == 0) {
        pl.gvals[leaf] = v;
        pl.leafS256[leaf] = s256;
        __threadfence();
        done = atomicAdd(&st->subDone, 1u);
    }
    done = __shfl_sync(0xffffffffu, done, 0);
    if (done != (unsigned int)pl.nLeaves - 1u) return;
    __threadfence();
    for (int d = 0; d < pl.nSteps; d++) {
        for (int j = pl.depthStart[d] + lane; j < pl.depthStart[d + 1]; j += 32) {
            const int2 c = pl.inner[j];
            pl.gvals[pl.nLeaves + j] = __fadd_rn(__ldcg(pl.gvals + c.x), __ldcg(pl.gvals + c.y));
        }
        __threadfence_block();
        __syncwarp();
    }
    unsigned int tot = 0;
    for (int i = lane; i < pl.nLeaves; i += 32) tot += __ldcg(pl.leafS256 + i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    if (lane == 0) {
        const float mean = __fdiv_rn(__ldcg(pl.gvals + pl.root), (float)nb);
        st->sadMean = mean;
        st->cut = mean > cutSad ? 1u : 0u;
        st->sadSum256 = tot;
        st->subDone = 0;
    }
}

// the scene-cut mean's share of the warp that wrote the SAD of block b (warp-uniform call)
__device__ __forceinline__ void cutMeanShare(const SubpixParams& p, int b, int nb, int lane) {
    const CutPlan& pl = p.plan;
    const int leaf = pl.leafOf[b];
    unsigned int old = 0;
    if (lane == 0) {
        __threadfence();   // this warp's SAD before its arrival
        old = atomicAdd(pl.leafCnt + leaf, 1u);
    }
    old = __shfl_sync(0xffffffffu, old, 0);
    if (old != (unsigned int)pl.leaves[leaf].y - 1u) return;
    __threadfence();
    if (lane == 0) pl.leafCnt[leaf] = 0;
    cutMeanLeaf(pl, p.sads, nb, p.cutSad, p.st, leaf, lane);
}

inline unsigned int divUp(int a, int b) { return (unsigned int)((a + b - 1) / b); }

// the CTA ranges of a merged launch's items
template <class P, class F>
static int layoutMerged(Merged<P>& m, F ctasOf) {   // ctasOf(item, gx&) -> the item's CTA count
    int total = 0;
    for (int i = 0; i < m.n; i++) {
        int gx = 1;
        const int c = ctasOf(m.item[i], gx);
        m.first[i] = total;
        m.gx[i] = gx;
        total += c;
    }
    m.first[m.n] = total;
    return total;
}

// carveout: the launch's preferred share of shared memory in the SM's L1, in percent (0: no more than a CTA needs)
template <typename... KArgs, typename... Args>
cudaError_t launchPdlCarveout(int carveout, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[1].val.sharedMemCarveout = (unsigned int)carveout;
    cfg.attrs = attr;
    cfg.numAttrs = carveout < 0 ? 1 : 2;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}
// ... left to the driver
template <typename... KArgs, typename... Args>
cudaError_t launchPdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    return launchPdlCarveout(-1, kernel, grid, block, smem, s, args...);
}
// The carveout of a synthesis. A tile of flowScale 1 takes 75 to 105 KB (the whole field region); on a grid of at most one
// CTA per SM the driver splits the L1 for two or three of them, and each change of the split waits for an idle SM: such
// grids ask for one CTA's need (back to back with the fallback check, 640x360 at t = 1/3: 8-bit 17.7 -> 14.1 us, Rgb10 22.8
// -> 14.8, P010 28.4 -> 21.0; a pair doubled 63 -> 61, 69 -> 63, 77 -> 69). With more CTAs a second one per SM pays
// (1024x576, 180 tiles: 20.8 us, 23.4 so), and at flowScale 4 the estimate changes the split back (a Rgb10 pair at 640x360
// 48 -> 55).
inline int synthCarveout(const SynthParams& p, dim3 grid) { return p.fs == 1 && (int)(grid.x * grid.y) <= smCount() ? 0 : -1; }

}  // namespace fgk
