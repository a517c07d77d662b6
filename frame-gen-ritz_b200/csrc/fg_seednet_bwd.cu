// The seed proposer's training backward on the fifth-generation tensor cores (tcgen05, bf16 operands in shared memory,
// f32 accumulators in tensor memory): the weight gradient and the input gradient of every 3x3 convolution layer as
// implicit GEMMs, replacing per-element loops. Same layouts and semantics as the per-layer forward in fg_seednet.cu.
//
//   dwCta<CIN, COUT, S>  dW[co][tap][ci] += sum_p x[S p + tap - 1][ci] dpre[p][co], db[co] += sum_p dpre[p][co]
//       GEMM D[m][n] = sum_k A[m][k] B[n][k] with m = tap * CIN + ci (plus one row of ones at m = 9 CIN, which makes
//       that row of D the bias gradient), n = co, k = output pixel. Every CTA reduces a contiguous slice of the output
//       pixels in chunks of 64 (4 MMAs of K = 16 per 128-row chunk of m), the operands double-buffered, and stores its
//       partial D; k_sn_dw_sum then adds all layers' partials into dW / db in a fixed order, so the gradient is
//       deterministic.
//   dxCta<CIN, COUT, S>  dpre_in[q][ci] = [x[q][ci] > 0] sum_{tap, co} w[co][tap][ci] dpre[p(q, tap)][co], the
//       output pixels p with S p + tap - 1 = q: GEMM with m = input pixel q (128 per chunk), n = ci, k = tap * COUT + co
//       (padded to a multiple of 16); the weights are staged once per CTA.
// A layer's two gradients share one launch (k_sn_bwd: the first CTAs the weight gradient's, the others the input
// gradient's), so the chain of a step is one launch per layer and one sum.
//
// Latency bound (12 to 192 CTAs per layer at 24 to 64 crops). What the launches spent was the staging: a division and a
// 2-byte gather per element. It now works on 8 pixels x 8 channels at a time, 16-byte loads transposed in registers by byte
// permutes, with the pixels' coordinates worked out once per chunk. A step's backward on 64 crops of 256 x 256: 408 -> 181 us (zero_grads, forward and loss included).
// The gradient at a layer's output (float) enters the MMAs rounded to bf16, the way the forward's activations do;
// accumulation is f32. Operands are K-major without swizzle (fg_tc.h): a core matrix is 8 rows of 8 consecutive k.
// Waits on the MMAs' mbarriers are bounded (100 ms, then kErrSeedNet into *err, one more bounded wait, TMEM freed).
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdint>

#include "fg_device.h"
#include "fg_params.h"
#include "fg_seednet.h"
#include "fg_tc.h"

namespace fgk {
namespace {

using bf16 = __nv_bfloat16;
constexpr uint64_t kBwdWaitNs = 100000000ull;
constexpr int kBwdThreads = 256;
constexpr int kDwK = 64;   // output pixels per staged chunk of the weight gradient (8 k-groups)

__device__ __forceinline__ uint32_t bpack(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

template <int CIN, int COUT>
struct DwShape {
    static constexpr int MR = 9 * CIN + 1;                 // rows: (tap, ci), then the ones row (bias)
    static constexpr int NCH = (MR + 127) / 128;           // 128-row chunks of m
    static constexpr int NP = COUT < 16 ? 16 : COUT;       // N of the MMA (8 outputs padded to 16)
    static constexpr int KG = kDwK / 8;                    // k-groups per staged chunk
    // core matrices [m-group][k-group], 144 bytes apart along k: the 128 bytes of one and a gap that spreads the stores of
    // 8 k-groups over all banks
    static constexpr int LBO = 144, SBO = KG * LBO;
    static constexpr int A_BYTES = NCH * 16 * SBO;
    static constexpr int B_BYTES = NP / 8 * SBO;
    static constexpr int STAGE = A_BYTES + B_BYTES;
    static constexpr int TCOLS = NCH * NP <= 32 ? 32 : NCH * NP <= 64 ? 64 : 128;
    static constexpr size_t SMEM = 2 * (size_t)STAGE + 64;
};

// waits for the mbarrier's next phase (bounded); false when it gave up
__device__ __forceinline__ bool waitPhase(uint64_t* bar, uint32_t& ph) {
    const bool ok = mbarWait(bar, ph, kBwdWaitNs);
    ph ^= 1u;
    return ok;
}

}  // namespace

// CTA `cta` of the weight gradient: chunks cta chunksPerCta .. + chunksPerCta
template <int CIN, int COUT, int S>
__device__ __forceinline__ void dwCta(const SnBackArgs& a, int cta, int chunksPerCta, unsigned int* err, unsigned char* sm) {
    using Sh = DwShape<CIN, COUT>;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm + 2 * Sh::STAGE);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + 2 * Sh::STAGE + 16);
    __shared__ int2 pix[kDwK];   // per pixel of the chunk: the input pixel of tap (0, 0), and the taps inside the input
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int npix = a.B * a.Ho * a.Wo;
    const int nchunks = (npix + kDwK - 1) / kDwK;
    const int c0 = cta * chunksPerCta, c1 = min(nchunks, c0 + chunksPerCta);
    if (warp == 0) tmemAlloc(tslot, Sh::TCOLS);
    if (tid == 0) {
        mbarInit(&bars[0], 1);
        mbarInit(&bars[1], 1);
    }
    // the rows that no pixel changes, in both buffers: the ones row (its products with the gradient's zero rows past the
    // last pixel vanish) and the padding
    for (int i = tid; i < 2 * Sh::NCH * 16 * Sh::KG * 8; i += kBwdThreads) {
        const int r = i & 7, kg = (i >> 3) % Sh::KG, mg = (i >> 3) / Sh::KG % (Sh::NCH * 16), buf = (i >> 3) / Sh::KG / (Sh::NCH * 16);
        const int m = mg * 8 + r;
        const uint32_t v = m == 9 * CIN ? 0x3F803F80u : 0u;   // bf16 1, 1
        if (m >= 9 * CIN) *reinterpret_cast<uint4*>(sm + buf * Sh::STAGE + mg * Sh::SBO + kg * Sh::LBO + r * 16) = make_uint4(v, v, v, v);
    }
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    const uint32_t tbase = *tslot;
    const bf16* __restrict__ x = reinterpret_cast<const bf16*>(a.x);
    uint32_t ph[2] = {0u, 0u};
    bool ok = true;
    auto stage = [&](int chunk, int buf) {
        unsigned char* A = sm + buf * Sh::STAGE;
        unsigned char* Bm = A + Sh::A_BYTES;
        const int p0 = chunk * kDwK;
        if (tid < kDwK) {
            const int p = p0 + tid;
            int off = 0, mask = 0;
            if (p < npix) {
                const int b = p / (a.Ho * a.Wo), rem = p - b * (a.Ho * a.Wo), oy = rem / a.Wo, ox = rem - oy * a.Wo;
                const int iy = oy * S - 1, ix = ox * S - 1;
                off = (b * a.H + iy) * a.W + ix;
#pragma unroll
                for (int t = 0; t < 9; t++)
                    mask |= ((unsigned)(iy + t / 3) < (unsigned)a.H && (unsigned)(ix + t % 3) < (unsigned)a.W) << t;
            }
            pix[tid] = make_int2(off, mask);
        }
        __syncthreads();
        if (CIN == 32) {   // A: 8 channels of a tap x 8 pixels, loaded 16 bytes a pixel, transposed
            for (int i = tid; i < 9 * 4 * Sh::KG; i += kBwdThreads) {
                const int kg = i % Sh::KG, mg = i / Sh::KG, tap = mg >> 2;
                const int to = (tap / 3) * a.W + tap % 3;
                const bf16* xc = x + (mg & 3) * 8;
                uint32_t v[8][4];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int2 q = pix[kg * 8 + j];
                    uint4 u = make_uint4(0u, 0u, 0u, 0u);
                    if ((q.y >> tap) & 1) u = __ldg(reinterpret_cast<const uint4*>(xc + (ptrdiff_t)(q.x + to) * CIN));
                    v[j][0] = u.x; v[j][1] = u.y; v[j][2] = u.z; v[j][3] = u.w;
                }
                unsigned char* o = A + mg * Sh::SBO + kg * Sh::LBO;
#pragma unroll
                for (int r = 0; r < 8; r++) {
                    constexpr uint32_t sel[2] = {0x5410u, 0x7632u};
                    *reinterpret_cast<uint4*>(o + r * 16) =
                        make_uint4(__byte_perm(v[0][r / 2], v[1][r / 2], sel[r & 1]), __byte_perm(v[2][r / 2], v[3][r / 2], sel[r & 1]),
                                   __byte_perm(v[4][r / 2], v[5][r / 2], sel[r & 1]), __byte_perm(v[6][r / 2], v[7][r / 2], sel[r & 1]));
                }
            }
        } else {           // A, 2 channels: a tap's two rows x 8 pixels, 4 bytes a pixel
            for (int i = tid; i < 9 * Sh::KG; i += kBwdThreads) {
                const int kg = i % Sh::KG, tap = i / Sh::KG, to = (tap / 3) * a.W + tap % 3;
                uint32_t v[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int2 q = pix[kg * 8 + j];
                    v[j] = (q.y >> tap) & 1 ? __ldg(reinterpret_cast<const uint32_t*>(x + (ptrdiff_t)(q.x + to) * CIN)) : 0u;
                }
#pragma unroll
                for (int ci = 0; ci < 2; ci++) {
                    const int m = 2 * tap + ci;
                    const uint32_t sel = ci ? 0x7632u : 0x5410u;
                    *reinterpret_cast<uint4*>(A + (m >> 3) * Sh::SBO + kg * Sh::LBO + (m & 7) * 16) =
                        make_uint4(__byte_perm(v[0], v[1], sel), __byte_perm(v[2], v[3], sel), __byte_perm(v[4], v[5], sel), __byte_perm(v[6], v[7], sel));
                }
            }
        }
        // B: row co, 8 pixels of the output gradient
        for (int i = tid; i < Sh::NP / 8 * Sh::KG * 8; i += kBwdThreads) {
            const int r = i & 7, kg = (i >> 3) % Sh::KG, ng = (i >> 3) / Sh::KG;
            const int co = ng * 8 + r;
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int p = p0 + kg * 8 + j;
                v[j] = (p < npix && co < COUT) ? a.dy[(size_t)p * COUT + co] : 0.0f;
            }
            *reinterpret_cast<uint4*>(Bm + ng * Sh::SBO + kg * Sh::LBO + r * 16) =
                make_uint4(bpack(v[0], v[1]), bpack(v[2], v[3]), bpack(v[4], v[5]), bpack(v[6], v[7]));
        }
    };
    const uint32_t idesc = tcIdescBf16(128, Sh::NP);
    for (int c = c0; c < c1 && ok; c++) {
        const int i = c - c0, buf = i & 1;
        if (i >= 2) ok = waitPhase(&bars[buf], ph[buf]) && ok;   // the MMAs of chunk c - 2 read this buffer
        ok = __syncthreads_and(ok);
        if (!ok) break;
        stage(c, buf);
        fenceAsyncShared();
        __syncthreads();
        if (tid == 0) {
            tcFenceAfter();
            const uint32_t A = smemAddr(sm + buf * Sh::STAGE), Bm = A + Sh::A_BYTES;
            for (int ch = 0; ch < Sh::NCH; ch++)
                for (int s = 0; s < Sh::KG / 2; s++)
                    tcMma(tbase + ch * Sh::NP, tcDesc(A + (uint32_t)(ch * 16 * Sh::SBO + 2 * s * Sh::LBO), Sh::LBO, Sh::SBO),
                          tcDesc(Bm + (uint32_t)(2 * s * Sh::LBO), Sh::LBO, Sh::SBO), idesc, (i > 0 || s > 0) ? 1u : 0u);
            tcCommit(&bars[buf]);
        }
    }
    // the last (up to two) chunks' MMAs
    const int n = c1 - c0;
    for (int k = 0; k < 2; k++) {
        const int i = n - 1 - k;
        if (i < 0 || i < n - 2) continue;
        const bool w = waitPhase(&bars[i & 1], ph[i & 1]);
        ok = w && ok;
    }
    ok = __syncthreads_and(ok);
    tcFenceAfter();
    if (ok && n > 0) {   // epilogue: lanes 32 (warp % 4) .., columns half (warp / 4) of NP
        const int q = warp & 3, half = warp >> 2;
        for (int ch = 0; ch < Sh::NCH; ch++) {
            const int m = ch * 128 + 32 * q + lane;
            const uint32_t ta = tbase + ((uint32_t)(32 * q) << 16) + ch * Sh::NP + half * (Sh::NP / 2);
            float v[16];
            if (Sh::NP / 2 == 16) tmemLd16(ta, v);
            else tmemLd8(ta, v);
            float* part = a.part + (size_t)cta * (Sh::MR * COUT);
            for (int j = 0; j < Sh::NP / 2; j++) {
                const int co = half * (Sh::NP / 2) + j;
                if (co < COUT && m <= 9 * CIN) part[m * COUT + co] = v[j];
            }
        }
    }
    if (!ok && tid == 0 && err) atomicOr(err, kErrSeedNet);
    tcFenceBefore();
    __syncthreads();
    if (warp == 0) {
        tcFenceAfter();
        tmemFree(tbase, Sh::TCOLS);
    }
}

// dW / db += the sum of the CTAs' partial products of every layer: 32 elements x 8 slices of the CTAs per block, the
// slices added in order (a fixed order, whatever ran when)
__global__ void __launch_bounds__(256) k_sn_dw_sum(const SnSumArgs a) {
    pdlEnter();
    __shared__ float red[8][32];
    int l = 0;
    while (l < kSnLayers - 1 && (int)blockIdx.x >= a.first[l + 1]) l++;
    const SnSumLayer& y = a.layer[l];
    const int i = ((int)blockIdx.x - a.first[l]) * 32 + (threadIdx.x & 31), slice = threadIdx.x >> 5;
    const int n = (9 * y.cin + 1) * y.cout;
    float s = 0.0f;
    if (i < n) {
#pragma unroll 4
        for (int b = slice; b < y.ctas; b += 8) s += __ldcg(y.part + (size_t)b * n + i);
    }
    red[slice][threadIdx.x & 31] = s;
    __syncthreads();
    if (slice || i >= n) return;
#pragma unroll
    for (int k = 1; k < 8; k++) s += red[k][threadIdx.x];
    const int m = i / y.cout, co = i - m * y.cout;
    if (m < 9 * y.cin) y.dw[(co * 9 + m / y.cin) * y.cin + m % y.cin] += s;
    else y.db[co] += s;
}

template <int CIN, int COUT>
struct DxShape {
    static constexpr int K = 9 * COUT, KP = (K + 15) / 16 * 16, KG = KP / 8;
    static constexpr int A_BYTES = 16 * KG * 128;          // 128 rows (input pixels)
    static constexpr int B_BYTES = CIN / 8 * KG * 128;     // CIN rows
    static constexpr size_t SMEM = 2 * (size_t)A_BYTES + B_BYTES + 64;
};

// CTA `cta` of `ctas` of the input gradient: chunks cta, cta + ctas, ..
template <int CIN, int COUT, int S>
__device__ __forceinline__ void dxCta(const SnBackArgs& a, int cta, int ctas, unsigned int* err, unsigned char* sm) {
    static_assert(CIN == 32, "the input gradient is needed for the 32-channel inputs only");
    using Sh = DxShape<CIN, COUT>;
    __shared__ int4 row[128];   // per row (input pixel) of the chunk: its image's first output pixel (-1: none), y, x
    unsigned char* Bm = sm + 2 * Sh::A_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(Bm + Sh::B_BYTES);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(Bm + Sh::B_BYTES + 16);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nq = a.B * a.H * a.W;
    const int nchunks = (nq + 127) / 128;
    const bf16* __restrict__ w = reinterpret_cast<const bf16*>(a.w);
    const bf16* __restrict__ x = reinterpret_cast<const bf16*>(a.x);
    if (warp == 0) tmemAlloc(tslot, 64);
    if (tid == 0) {
        mbarInit(&bars[0], 1);
        mbarInit(&bars[1], 1);
    }
    // B: row ci, k = tap * COUT + co: w[co][tap][ci]
    for (int i = tid; i < CIN / 8 * Sh::KG * 8; i += kBwdThreads) {
        const int r = i & 7, kg = (i >> 3) % Sh::KG, ng = (i >> 3) / Sh::KG;
        const int ci = ng * 8 + r;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int k = kg * 8 + j;
            v[j] = k < Sh::K ? __bfloat162float(w[((k % COUT) * 9 + k / COUT) * CIN + ci]) : 0.0f;
        }
        reinterpret_cast<uint4*>(Bm)[(ng * Sh::KG + kg) * 8 + r] =
            make_uint4(bpack(v[0], v[1]), bpack(v[2], v[3]), bpack(v[4], v[5]), bpack(v[6], v[7]));
    }
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    const uint32_t tbase = *tslot;
    uint32_t ph[2] = {0u, 0u};
    bool ok = true;
    auto stage = [&](int chunk, int buf) {   // A: row q, k = tap * COUT + co: dpre[p(q, tap)][co]
        unsigned char* A = sm + buf * Sh::A_BYTES;
        if (tid < 128) {
            const int q = chunk * 128 + tid, b = q / (a.H * a.W), rem = q - b * (a.H * a.W), qy = rem / a.W;
            row[tid] = make_int4(q < nq ? b * a.Ho * a.Wo : -1, qy, rem - qy * a.W, 0);
        }
        __syncthreads();
#pragma unroll 3
        for (int i = tid; i < 16 * Sh::KG * 8; i += kBwdThreads) {
            const int r = i & 7, kg = (i >> 3) % Sh::KG, mg = (i >> 3) / Sh::KG;
            const int4 q = row[mg * 8 + r];
            const int k0 = kg * 8, tap = k0 / COUT, co0 = k0 % COUT;   // 8 consecutive k share a tap (COUT % 8 == 0)
            const int ty = q.y + 1 - tap / 3, tx = q.z + 1 - tap % 3;  // = S p
            uint4 o = make_uint4(0, 0, 0, 0);
            if (q.x >= 0 && k0 < Sh::K && ty >= 0 && tx >= 0 && ty % S == 0 && tx % S == 0 && ty / S < a.Ho && tx / S < a.Wo) {
                const float4* g = reinterpret_cast<const float4*>(a.dy + (size_t)(q.x + (ty / S) * a.Wo + tx / S) * COUT + co0);
                const float4 u = g[0], v = g[1];
                o = make_uint4(bpack(u.x, u.y), bpack(u.z, u.w), bpack(v.x, v.y), bpack(v.z, v.w));
            }
            reinterpret_cast<uint4*>(A)[(mg * Sh::KG + kg) * 8 + r] = o;
        }
    };
    const uint32_t idesc = tcIdescBf16(128, CIN);
    auto epi = [&](int chunk, int acc) {
        const int qw = warp & 3, half = warp >> 2;
        const int q = chunk * 128 + 32 * qw + lane;
        float v[16];
        tmemLd16(tbase + ((uint32_t)(32 * qw) << 16) + acc * 32 + half * 16, v);
        if (q >= nq) return;
        const bf16* xq = x + (size_t)q * CIN + half * 16;
        float* d = a.dx + (size_t)q * CIN + half * 16;
#pragma unroll
        for (int j = 0; j < 16; j++) d[j] = __bfloat162float(xq[j]) > 0.0f ? v[j] : 0.0f;
    };
    int it = 0, prev = -1;
    for (int c = cta; c < nchunks && ok; c += ctas, it++) {
        const int buf = it & 1;
        stage(c, buf);
        fenceAsyncShared();
        tcFenceBefore();
        ok = __syncthreads_and(ok);
        if (!ok) break;
        if (tid == 0) {
            tcFenceAfter();
            const uint32_t A = smemAddr(sm + buf * Sh::A_BYTES), B = smemAddr(Bm);
            for (int s = 0; s < Sh::KG / 2; s++)
                tcMma(tbase + buf * 32, tcDesc(A + (uint32_t)(2 * s * 128), 128, Sh::KG * 128),
                      tcDesc(B + (uint32_t)(2 * s * 128), 128, Sh::KG * 128), idesc, s > 0 ? 1u : 0u);
            tcCommit(&bars[buf]);
        }
        if (prev >= 0) {   // the previous chunk's epilogue overlaps this chunk's MMAs
            const bool done = waitPhase(&bars[buf ^ 1], ph[buf ^ 1]);
            ok = __syncthreads_and(done);   // (one answer for the whole CTA: the loop has barriers)
            tcFenceAfter();
            if (ok) epi(prev, buf ^ 1);
        }
        prev = c;
    }
    if (prev >= 0 && ok) {
        const int buf = (it - 1) & 1;
        ok = waitPhase(&bars[buf], ph[buf]) && ok;
        tcFenceAfter();
        if (ok) epi(prev, buf);
    }
    if (!ok) {
        if (tid == 0 && err) atomicOr(err, kErrSeedNet);
        for (int b = 0; b < 2; b++) mbarWait(&bars[b], ph[b], kBwdWaitNs);
    }
    tcFenceBefore();
    __syncthreads();
    if (warp == 0) {
        tcFenceAfter();
        tmemFree(tbase, 64);
    }
}

// one layer: CTAs 0 .. dwCtas - 1 the weight gradient, the others the input gradient (layers 2-6)
template <int CIN, int COUT, int S, bool kDx>
__global__ void __launch_bounds__(kBwdThreads) k_sn_bwd(const SnBackArgs a, int dwCtas, int chunksPerCta, unsigned int* err) {
    pdlEnter();
    extern __shared__ __align__(128) unsigned char sm[];
    if ((int)blockIdx.x < dwCtas) dwCta<CIN, COUT, S>(a, blockIdx.x, chunksPerCta, err, sm);
    else if constexpr (kDx) dxCta<CIN, COUT, S>(a, blockIdx.x - dwCtas, gridDim.x - dwCtas, err, sm);
}

namespace {

template <int CIN, int COUT, bool kDx>
constexpr size_t bwdSmem() {
    size_t n = DwShape<CIN, COUT>::SMEM;
    if constexpr (kDx) n = n > DxShape<CIN, COUT>::SMEM ? n : DxShape<CIN, COUT>::SMEM;
    static_assert(DwShape<CIN, COUT>::SMEM <= 227 * 1024, "shared memory");
    return n;
}

template <int CIN, int COUT, int S, bool kDx>
cudaError_t bwdLaunch(const SnBackArgs& a, int& ctas, unsigned int* err, cudaStream_t s) {
    const int nchunks = (a.B * a.Ho * a.Wo + kDwK - 1) / kDwK;
    const int most = std::min(nchunks, a.partCtas), per = (nchunks + most - 1) / most;
    ctas = (nchunks + per - 1) / per;
    // the SMs that the weight gradient leaves (one CTA each: the input gradient's operands fill the shared memory)
    const int dx = kDx ? std::min((a.B * a.H * a.W + 127) / 128, std::max(smCount() - ctas, smCount() / 2)) : 0;
    return launchPdl(k_sn_bwd<CIN, COUT, S, kDx>, dim3(ctas + dx), dim3(kBwdThreads), bwdSmem<CIN, COUT, kDx>(), s, a, ctas, per, err);
}

template <int CIN, int COUT, int S, bool kDx>
cudaError_t setSmem() {
    return cudaFuncSetAttribute(k_sn_bwd<CIN, COUT, S, kDx>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bwdSmem<CIN, COUT, kDx>());
}

}  // namespace

cudaError_t prepareSeedNetBackward() {
    cudaError_t e = setSmem<2, 32, 2, false>();
    if (e == cudaSuccess) e = setSmem<32, 32, 2, true>();
    if (e == cudaSuccess) e = setSmem<32, 32, 1, true>();
    if (e == cudaSuccess) e = setSmem<32, kSnOut, 1, true>();
    return e;
}

cudaError_t launchSnBackwardTc(int layer, const SnBackArgs& a, int& ctas, unsigned int* err, cudaStream_t s) {
    switch (layer) {
        case 0: return bwdLaunch<2, 32, 2, false>(a, ctas, err, s);
        case 1:
        case 2: return bwdLaunch<32, 32, 2, true>(a, ctas, err, s);
        case 3:
        case 4: return bwdLaunch<32, 32, 1, true>(a, ctas, err, s);
        case 5: return bwdLaunch<32, kSnOut, 1, true>(a, ctas, err, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launchSnDwSum(SnSumArgs& a, cudaStream_t s) {
    int total = 0;
    for (int l = 0; l < kSnLayers; l++) {
        a.first[l] = total;
        total += (int)divUp((9 * a.layer[l].cin + 1) * a.layer[l].cout, 32);
    }
    return launchPdl(k_sn_dw_sum, dim3(total), dim3(256), 0, s, a);
}

}  // namespace fgk
