// Deconvolution side of the serial major cycle on the GPU:
//   * serial coordinate descent, Core/Deconvolution/FastSerialCD.cs (Deconvolve, DeconvolvePath,
//     GetAbsMaxDiff, ResetLipschitzMap), bit-identical to the C# arithmetic: float values, no
//     FMA contraction, the same pixel choice (largest |change|, first in row-major order);
//   * the PSF preparation of Core/Common.cs (PSF.CalcPaddedFourierCorrelation, CalcPSFSquared,
//     CalcAMap, Cut, CalcMaxSidelobe, CalcMaxLipschitz, Residuals.GetMax) and the padded FFT
//     correlation of Core/PaddedConvolver.cs, in FP64 with cuFFT as the reference does with FFTW;
//   * MajorCycle.ReconstructSerialCD (SingleReconstruction/MajorCycle.cs:33-134) with the
//     visibilities, grids and images resident in HBM.
//
// Coordinate descent.  One iteration of FastSerialCD picks the pixel whose proximal update
// changes it most (a scan of the whole image), sets it, and adds the scaled PSF^2 to the
// gradient map in a window around it.  Only pixels in that window change, so the GPU keeps the
// best candidate of every 40 x 128 tile (one for each warp's rows of it) and re-evaluates only the
// rows that the window touches.  A candidate is ordered by one 64-bit key, (|change| bits << 32) |
// (0xFFFFFFFF - pixel index), so the largest key is the largest change and, among equal changes,
// the first pixel, which is the order in which GetAbsMax (FastSerialCD.cs:135-170) keeps its
// winner.  The iterations run inside one cooperative launch whose CTAs own fixed tiles and
// exchange nothing but their best candidates (cd_run_kernel).

#include <cuda_runtime.h>
#include <cufft.h>
#include <math_constants.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <vector>

#include "kernels.cuh"

using namespace p9idg;

namespace {

p9idg_status fail(p9idg_status st, const std::string &msg) {
    record_last_error(msg);
    return st;
}

p9idg_status cuda_fail(cudaError_t e, const char *what) {
    const p9idg_status st = (e == cudaErrorMemoryAllocation) ? P9IDG_OUT_OF_MEMORY
                            : (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) ? P9IDG_NO_DEVICE
                                                                                             : P9IDG_CUDA_ERROR;
    return fail(st, std::string(what) + ": " + cudaGetErrorString(e));
}

#define CK(x)                                                \
    do {                                                     \
        cudaError_t e_ = (x);                                \
        if (e_ != cudaSuccess) return cuda_fail(e_, #x);     \
    } while (0)

#define TRY(x)                         \
    do {                               \
        p9idg_status s_ = (x);         \
        if (s_ != P9IDG_OK) return s_; \
    } while (0)

#define CUFFT(x)                                                                              \
    do {                                                                                      \
        cufftResult r_ = (x);                                                                 \
        if (r_ != CUFFT_SUCCESS) return fail(P9IDG_CUDA_ERROR, std::string(#x) + " failed"); \
    } while (0)

struct Buf {  // device buffer, freed when it goes out of scope (every early return included)
    void *p = nullptr;
    size_t bytes = 0;
    Buf() = default;
    Buf(const Buf &) = delete;
    Buf &operator=(const Buf &) = delete;
    ~Buf() { release(); }
    cudaError_t ensure(size_t n) {
        if (n <= bytes && p) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
        cudaError_t e = device_alloc(&p, std::max<size_t>(n, 256));
        if (e == cudaSuccess) bytes = std::max<size_t>(n, 256);
        return e;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    template <typename T>
    T *as() const { return static_cast<T *>(p); }
};

p9idg_status have_device() {
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) return fail(P9IDG_NO_DEVICE, "no CUDA device available");
    return P9IDG_OK;
}

// ------------------------------------------------------------------------------------------
// device arithmetic in the reference's float semantics

// .NET Core 3.0 Math.Max(float, float): IEEE 754:2019 maximum (NaN wins, +0 above -0).
__device__ __forceinline__ float cs_maxf(float a, float b) {
    if (a != b) {
        if (!isnan(a)) return b < a ? a : b;
        return a;
    }
    return signbit(b) ? a : b;
}

// ElasticNet.ProximalOperator (Common.cs:28-29), un-fused: thr = lambda * alpha and slope = lambda *
// (1 - alpha), each rounded as the reference rounds it.  max(v, 0) is Math.Max
// as above: NaN stays, -0 becomes +0.  Most pixels of a sparse model are held at zero by the
// threshold, and 0 / den is +0 for every positive den, so a warp of such pixels makes no division.
__device__ __forceinline__ float prox(float x, float lipschitz, float thr, float slope) {
    const float v = __fsub_rn(x, thr);
    const float den = __fadd_rn(lipschitz, slope);
    if (v <= 0.0f && den > 0.0f) return 0.0f;
    return __fdiv_rn(v <= 0.0f ? 0.0f : v, den);
}

constexpr int kNT = 512, kWarps = kNT / 32;  // image reductions
// Coordinate descent: CTAs of kCdNT threads, tiles of kTX columns in which each warp has R = 1 or 2 rows.  A
// 768^2 update window (a 384^2 PSF) spans 21 x 7 = 147 tiles of two rows a warp, one for each CTA of the 152
// SMs.  Windows of few tiles take one row (cd_layout).
constexpr int kTX = 128, kCdNT = 640, kCdWarps = kCdNT / 32, kCdCols = kTX / 32;
// Slots of the exchange, three for each lane of the polling warp; pairs of CTAs share one from
// kCdPairFrom CTAs on.  Measured for the exchange alone: 1270 clocks with 30 CTAs, each polling every
// slot, 3500 with 147 (the polls of one line queue up), 2000 with 74 pairs; 30 CTAs in pairs take 1860.
constexpr int kCdPoll = 3, kCdSlots = 32 * kCdPoll, kCdPairFrom = 56;
// Iterations of one launch: few enough that other streams' kernels wait milliseconds for the SMs, not
// for a whole deconvolution, and enough that a launch does not show.
constexpr int kCdLaunchIters = 512;
// q / d = q * ceil(2^36 / d) >> 36 for q * d < 2^36; here q < 2^17, d < 2^15 and d >= 20, so the factor
// fits 32 bits.
constexpr int kCdInvBits = 36;
// Clocks (about 4 s) after which a CTA gives up waiting for another.  All CTAs of a cooperative launch are
// resident, so this is only met if one of them cannot run.
constexpr long long kCdPatience = 8000000000ll;

struct CdCtl {  // the state one launch hands to the next
    int32_t iter, done, converged, error;
};

// A candidate: x = |change| bits, y = 0xFFFFFFFF - (row << 16 | column), z = new value, w = current value;
// all zero for "none".  (x, y) is the key, larger is better: the largest change, and of equal changes the
// first pixel in row-major order.
using CdCand = uint4;

struct CdParams {
    float *x, *g;
    const float *a, *psf2;
    CdCand *cand;                  // [tile][warp]
    unsigned long long *tile_key;  // best key of each tile, left by the scan
    uint4 *slots;                  // [2][kCdSlots]: (epoch, candidate's y, z, w)
    CdCtl *ctl;
    CdCtl *report;  // pinned: [0] the state a launch leaves, [1].error set by a CTA that gave up
    int32_t n, ph, pw, tiles_x, tiles_y, max_iter;
    int32_t rows;                  // R
    int32_t ax, ay;                // tile (ty, tx) belongs to CTA (ty % ay) * ax + tx % ax
    uint32_t inv_row, inv_col;     // ceil(2^kCdInvBits / tile rows of a period), .. / tile columns
    int32_t local_x, local_tiles;  // tiles of one CTA: in a row, in all (at most)
    float lambda, alpha, eps;
};

// Max of a 64-bit key (hi, lo) over the warp as two 32-bit hardware reductions: the high words, then
// the low words of the lanes holding the highest one (the same lexicographic maximum).
__device__ __forceinline__ uint2 warp_max(unsigned hi, unsigned lo) {
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    return make_uint2(mh, ml);
}

__device__ __forceinline__ CdCand better(const CdCand &a, const CdCand &b) {
    return a.x > b.x || (a.x == b.x && a.y > b.y) ? a : b;
}

// The lane that holds the warp's best candidate (pixels are unique; of lanes without any, the first).
__device__ __forceinline__ int best_lane(const CdCand &c) {
    const uint2 m = warp_max(c.x, c.y);
    return __ffs(__ballot_sync(0xffffffffu, c.x == m.x && c.y == m.y)) - 1;
}

// One 16-byte access that no other can split: a packet carries its own epoch, so a reader that finds
// the epoch it waits for has the packet's other words too, without a fence.
__device__ __forceinline__ void st_packet(uint4 *p, const uint4 &v) {
    const unsigned long long lo = v.x | (static_cast<unsigned long long>(v.y) << 32),
                             hi = v.z | (static_cast<unsigned long long>(v.w) << 32);
    asm volatile("{\n.reg .b128 q;\nmov.b128 q, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], q;\n}\n" ::"l"(p), "l"(lo), "l"(hi)
                 : "memory");
}

__device__ __forceinline__ uint4 ld_packet(const uint4 *p) {
    unsigned long long lo, hi;
    asm volatile("{\n.reg .b128 q;\nld.relaxed.gpu.global.b128 q, [%2];\nmov.b128 {%0, %1}, q;\n}\n" : "=l"(lo), "=l"(hi) : "l"(p)
                 : "memory");
    return make_uint4(static_cast<unsigned>(lo), static_cast<unsigned>(lo >> 32), static_cast<unsigned>(hi),
                      static_cast<unsigned>(hi >> 32));
}

__device__ __forceinline__ uint32_t cd_shared(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ uint32_t cd_peer(uint32_t addr, unsigned rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// The same into another CTA's shared memory, and from this one's.  The packets carry their epoch at the scope of
// the pair, so nothing has to be acquired: a wait for st.async has to acquire at cluster scope, which empties
// L1, and the tiles' pixels then come from L2 in every iteration (1000 iterations at 3072^2, whole windows: 4.68 ms
// against 4.62, windows clipped by the edges 3.73 against 3.53 us an iteration).
__device__ __forceinline__ void st_peer(uint32_t dst, const uint4 &v) {
    const unsigned long long lo = v.x | (static_cast<unsigned long long>(v.y) << 32),
                             hi = v.z | (static_cast<unsigned long long>(v.w) << 32);
    asm volatile("{\n.reg .b128 q;\nmov.b128 q, {%1, %2};\nst.relaxed.cluster.shared::cluster.b128 [%0], q;\n}\n" ::"r"(dst),
                 "l"(lo), "l"(hi)
                 : "memory");
}

__device__ __forceinline__ uint4 ld_peer(uint32_t p) {
    unsigned long long lo, hi;
    asm volatile("{\n.reg .b128 q;\nld.relaxed.cluster.shared::cta.b128 q, [%2];\nmov.b128 {%0, %1}, q;\n}\n"
                 : "=l"(lo), "=l"(hi)
                 : "r"(p)
                 : "memory");
    return make_uint4(static_cast<unsigned>(lo), static_cast<unsigned>(lo >> 32), static_cast<unsigned>(hi),
                      static_cast<unsigned>(hi >> 32));
}

// A packet's candidate: |change| is not sent, it is the difference of the two values.
__device__ __forceinline__ CdCand cd_unpack(const uint4 &q) {
    return make_uint4(__float_as_uint(fabsf(__fsub_rn(__uint_as_float(q.w), __uint_as_float(q.z)))), q.y, q.z, q.w);
}

// Waits for the packet of this epoch at p (every lane its own, or the same one); false if it does not come.
__device__ __forceinline__ bool cd_await_peer(uint32_t p, unsigned epoch, CdCand &v) {
    const long long t0 = clock64();
    while (true) {
        const uint4 q = ld_peer(p);
        if (q.x == epoch) {
            v = cd_unpack(q);
            return true;
        }
        if (clock64() - t0 > kCdPatience) return false;
    }
}

__device__ __forceinline__ void cd_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// An arrival on another CTA's barrier, which only says that a packet is on its way: waiting for it spares the polls
// of its epoch (without it 4.69 ms and 3.63 us), which are what tells that the packet is there.
__device__ __forceinline__ void cd_signal(uint32_t bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// For what this CTA's own warps wrote to its shared memory.
__device__ __forceinline__ bool cd_wait(uint32_t bar, uint32_t phase) {
    long long t0 = 0;
    while (true) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(bar), "r"(phase)
            : "memory");
        if (done) return true;
        const long long t = clock64();
        if (t0 == 0) t0 = t;
        if (t - t0 > kCdPatience) return false;
    }
}

__device__ __forceinline__ void cd_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct Window {
    int py, px;          // selected pixel
    int yq, xq;          // of the update window's first pixel, which may lie outside the image
    int y0, y1, x0, x1;  // its part inside
    float xnew, xdiff;
};

// Two additions an instruction, rounded as __fadd_rn.  Products stay scalar: a packed mul.rn and the packed
// add.rn after it came out fused.
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 f2_get(F2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float rcp_approx(float a) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

// Evaluates (and with UPDATE first updates) the warp's R rows from yb of the tile at column xb; returns
// this thread's best candidate, which is the exact one wherever it is the warp's best.  COVER: what is known
// of the rows' pixels: nothing, that all lie in the image, or that all lie in the update window.  All of a
// thread's loads are issued before any is used, so the rows cost one memory latency rather than one per pixel.
//
// The kernel around this waits for what its warps issue here (five warps a scheduler), and most of it would
// be divisions for pixels that cannot win.  So the changes are first approximated with a reciprocal good to an
// ulp: for den in (1e-30, 1e30), quotient and change are off by at most Q 2^-22 + D 2^-23 (Q bounds the warp's
// quotients, D is its largest change), so the pixel with the largest change is among those within twice that
// of D, and only these (usually one in the warp) are evaluated as the reference does; rows whose pixels are
// all zero and held there by the threshold are left at once.  NaN and infinities fail the comparisons that
// leave a pixel out.
enum Cover { kAny, kImage, kWindow };

template <int R, bool UPDATE, Cover COVER>
__device__ __forceinline__ CdCand eval_rows(const CdParams &P, float thr, float slope, int yb, int xb, const Window &w) {
    const int x = xb + static_cast<int>(threadIdx.x & 31);
    constexpr int J = R * kCdCols;
    float gv[J], xv[J], av[J], pv[J], d[J];
    bool in[J], upd[J];
    const size_t i0 = static_cast<size_t>(yb) * P.n + x;
    float *gp = P.g + i0, *xp = P.x + i0;
    const float *ap = P.a + i0;
    const float *pp = P.psf2 + (static_cast<int64_t>(yb - w.yq) * P.pw + (x - w.xq));
    const auto off = [&](int j) { return (j / kCdCols) * P.n + 32 * (j % kCdCols); };
#pragma unroll
    for (int j = 0; j < J; j++) {
        const int r = j / kCdCols, k = j % kCdCols, y = yb + r, xc = x + 32 * k;
        in[j] = COVER != kAny || (y < P.n && xc < P.n);
        upd[j] = UPDATE && (COVER == kWindow || (y >= w.y0 && y < w.y1 && xc >= w.x0 && xc < w.x1));
        gv[j] = in[j] ? gp[off(j)] : 0.0f;
        xv[j] = in[j] ? xp[off(j)] : 0.0f;
        av[j] = in[j] ? __ldg(ap + off(j)) : 1.0f;
        pv[j] = upd[j] ? __ldg(pp + (r * P.pw + 32 * k)) : 0.0f;
    }
    if (UPDATE && w.py - yb < R && w.py >= yb) {  // the selected pixel takes its new value
#pragma unroll
        for (int j = 0; j < J; j++)
            if (w.py == yb + j / kCdCols && w.px == x + 32 * (j % kCdCols)) {
                xv[j] = w.xnew;
                xp[off(j)] = w.xnew;
            }
    }
    const F2 thr2 = f2(-thr, -thr), slope2 = f2(slope, slope);
    float dmax = 0.0f, vmax = 0.0f, den_lo = 1e30f, den_hi = 0.0f;
#pragma unroll
    for (int j = 0; j < J; j += 2) {
        if (UPDATE) {  // gradients[i, j] += psf2 * xDiff
            const float2 g = f2_get(
                f2_add(f2(gv[j], gv[j + 1]), f2(__fmul_rn(pv[j], w.xdiff), __fmul_rn(pv[j + 1], w.xdiff))));
            if (upd[j]) gp[off(j)] = gv[j] = g.x;
            if (upd[j + 1]) gp[off(j + 1)] = gv[j + 1] = g.y;
        }
        const F2 xa = f2(__fmul_rn(xv[j], av[j]), __fmul_rn(xv[j + 1], av[j + 1]));
        const float2 v = f2_get(f2_add(f2_add(xa, f2(gv[j], gv[j + 1])), thr2));
        const float2 den = f2_get(f2_add(f2(av[j], av[j + 1]), slope2));
        const float va = max_nan(v.x, 0.0f), vb = max_nan(v.y, 0.0f);
        d[j] = fabsf(__fsub_rn(xv[j], __fmul_rn(va, rcp_approx(den.x))));
        d[j + 1] = fabsf(__fsub_rn(xv[j + 1], __fmul_rn(vb, rcp_approx(den.y))));
        if (COVER == kAny) {
            d[j] = in[j] ? d[j] : 0.0f;
            d[j + 1] = in[j + 1] ? d[j + 1] : 0.0f;
        }
        dmax = fmaxf(dmax, fmaxf(d[j], d[j + 1]));
        vmax = max_nan(vmax, max_nan(va, vb));
        den_lo = fminf(den_lo, fminf(den.x, den.y));
        den_hi = fmaxf(den_hi, fmaxf(den.x, den.y));
    }
    const float q = den_lo > 1e-30f && den_hi < 1e30f ? __fmul_rn(vmax, 1.0001f * rcp_approx(den_lo)) : CUDART_NAN_F;
    const float D = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(dmax)));
    const float Q = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(q)));  // a NaN is the largest
    CdCand best = make_uint4(0u, 0u, 0u, 0u);
    if (D == 0.0f && __all_sync(0xffffffffu, vmax == 0.0f)) return best;
    const float least = D - (D + Q) * 0x1p-20f - 1e-37f;
#pragma unroll
    for (int j = 0; j < J; j++) {
        if (d[j] < least || !in[j]) continue;
        const float xt = prox(__fadd_rn(__fmul_rn(xv[j], av[j]), gv[j]), av[j], thr, slope);
        const float e = fabsf(__fsub_rn(xv[j], xt));
        if (e > __uint_as_float(best.x))  // pixels in index order: the first of equal changes stays
            best = make_uint4(__float_as_uint(e),
                              0xFFFFFFFFu - ((static_cast<uint32_t>(yb + j / kCdCols) << 16) | static_cast<uint32_t>(x + 32 * (j % kCdCols))),
                              __float_as_uint(xt), __float_as_uint(xv[j]));
    }
    return best;
}

// The same for an update, by what the window and the image cover.
template <int R>
__device__ __forceinline__ CdCand update_rows(const CdParams &P, float thr, float slope, int yb, int xb, const Window &w) {
    if (yb >= w.y0 && yb + R <= w.y1 && xb >= w.x0 && xb + kTX <= w.x1) return eval_rows<R, true, kWindow>(P, thr, slope, yb, xb, w);
    if (yb + R <= P.n && xb + kTX <= P.n) return eval_rows<R, true, kImage>(P, thr, slope, yb, xb, w);
    return eval_rows<R, true, kAny>(P, thr, slope, yb, xb, w);
}

// Full scan (GetAbsMax over the whole image): every warp's candidate of every tile, and each tile's best key.
template <int R>
__global__ void __launch_bounds__(kCdNT) cd_scan_kernel(const __grid_constant__ CdParams P) {
    __shared__ uint2 sm[kCdWarps];
    const float thr = __fmul_rn(P.lambda, P.alpha), slope = __fmul_rn(P.lambda, __fsub_rn(1.0f, P.alpha));
    const Window w{};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = blockIdx.y * P.tiles_x + blockIdx.x;
    const CdCand c = eval_rows<R, false, kAny>(P, thr, slope, (blockIdx.y * kCdWarps + warp) * R, blockIdx.x * kTX, w);
    if (lane == best_lane(c)) {
        P.cand[t * static_cast<int64_t>(kCdWarps) + warp] = c;
        sm[warp] = make_uint2(c.x, c.y);
    }
    __syncthreads();
    if (warp == 0) {
        const uint2 v = lane < kCdWarps ? sm[lane] : make_uint2(0u, 0u);
        const uint2 m = warp_max(v.x, v.y);
        if (lane == 0) P.tile_key[t] = (static_cast<unsigned long long>(m.x) << 32) | m.y;
    }
    if (t == 0) {
        if (threadIdx.x == 0) *P.ctl = CdCtl{0, 0, 0, 0};
        if (threadIdx.x < 2 * kCdSlots) P.slots[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
    }
}

// The largest key of the scan (GetAbsMax's result), for the host.
__global__ void __launch_bounds__(kCdNT) cd_pick_kernel(const unsigned long long *keys, int ntiles, unsigned long long *out) {
    __shared__ uint2 sm[kCdWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned long long best = 0;
    for (int base = 0; base < ntiles; base += 8 * kCdNT) {
        unsigned long long v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int t = base + j * kCdNT + static_cast<int>(threadIdx.x);
            v[j] = t < ntiles ? keys[t] : 0ull;
        }
#pragma unroll
        for (int j = 0; j < 8; j++) best = v[j] > best ? v[j] : best;
    }
    const uint2 m = warp_max(static_cast<unsigned>(best >> 32), static_cast<unsigned>(best));
    if (lane == 0) sm[warp] = m;
    __syncthreads();
    if (warp == 0) {
        const uint2 v = lane < kCdWarps ? sm[lane] : make_uint2(0u, 0u);
        const uint2 a = warp_max(v.x, v.y);
        if (lane == 0) *out = (static_cast<unsigned long long>(a.x) << 32) | a.y;
    }
}

// Up to kCdLaunchIters coordinate-descent iterations (FastSerialCD.cs:83-98) in one cooperative launch.
//
// An iteration is a latency chain: agree on the pixel, load the window, update and re-evaluate it, find
// the new candidates.  The only thing that CTAs need of each other is the best candidate, so a tile
// belongs to the same CTA (and a pixel to the same thread) throughout, the tiles dealt out as a torus of
// ay x ax CTAs: a window of at most that many tiles gives no CTA two of them.
//
// The exchange: every warp puts its best candidate into its cluster's first CTA (a cluster is one CTA or
// a PAIR), whose first warp posts the best of them as one 16-byte packet that carries the iteration's
// number, reads every cluster's packet until all carry it, and hands the best to the cluster's warps.  No
// fence, atomic or grid-wide counter is needed, and gradients and model stay out of it.  Buffers and
// slots alternate between two sets: a slot is overwritten only after every cluster has posted the
// iteration after it, hence read it.
//
// Measured for 1000 iterations at 3072^2 with a 768^2 window: 4.6 us an iteration, against 6.5 us for a
// launch per iteration (graph replays with programmatic dependent launches, every CTA reducing all tile
// keys).  Of the 4.6 us about 1.3 are the exchange and its two hops within a pair, 1.5 a warp's loads and
// evaluation, and the rest the wait for the slowest of 147 CTAs.
//
// A lane keeps in registers the candidate of its warp's rows of local tile `lane`; images of more than 32
// tiles a CTA (4864 tiles, 5000^2 with two rows a warp) keep them in P.cand, which only this warp touches.
template <int R, bool PAIR>
__global__ void __launch_bounds__(kCdNT, 1) cd_run_kernel(const __grid_constant__ CdParams P) {
    __shared__ CdCand sm_in[2][kCdWarps];  // candidates of the first CTA's warps
    __shared__ CdCand sm_sel[2];           // the selected candidate (first CTA)
    __shared__ __align__(16) uint4 sm_peer[2][kCdWarps];  // packets: candidates of the second CTA's warps (first CTA)
    __shared__ __align__(16) uint4 sm_told[2];            // the selected candidate (second CTA)
    __shared__ unsigned long long bar_in[2], bar_sel[2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const CdCtl c0 = *P.ctl;
    if (c0.done) {  // the same for all CTAs: an earlier launch wrote it
        if (blockIdx.x == 0 && threadIdx.x == 0) P.report[0] = c0;
        return;
    }
    constexpr unsigned csize = PAIR ? 2 : 1;
    unsigned rank = 0;
    if (PAIR) asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const CdCand none = make_uint4(0u, 0u, 0u, 0u);
    const int nslots = static_cast<int>(gridDim.x / csize), slot = static_cast<int>(blockIdx.x / csize);
    const uint32_t in_bar = cd_shared(bar_in), sel_bar = cd_shared(bar_sel);
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; b++) {
            // candidates: an arrival of each warp of the cluster; selection: one of its first warp
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(in_bar + 8 * b), "r"(csize * kCdWarps));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sel_bar + 8 * b));
        }
    }
    if (threadIdx.x < 2 * kCdWarps) sm_peer[threadIdx.x / kCdWarps][threadIdx.x % kCdWarps] = none;  // epochs start at 1
    if (threadIdx.x < 2) sm_told[threadIdx.x] = none;
    if (PAIR)
        cd_cluster_sync();
    else
        __syncthreads();

    const int cta = blockIdx.x, cy = static_cast<int>(static_cast<uint32_t>(cta) / static_cast<uint32_t>(P.ax)), cx = cta - cy * P.ax;
    const bool owner = cy < P.ay;  // the last CTA of an odd number in pairs owns nothing
    const bool in_regs = P.local_tiles <= 32;
    // this warp's candidate of local tile l = (ty / ay) * local_x + tx / ax; null past the image
    const auto at = [&](int l) -> CdCand * {
        const int q = l / P.local_x, ty = cy + q * P.ay, tx = cx + (l - q * P.local_x) * P.ax;
        return owner && l < P.local_tiles && ty < P.tiles_y && tx < P.tiles_x
                   ? P.cand + (static_cast<int64_t>(ty) * P.tiles_x + tx) * kCdWarps + warp
                   : nullptr;
    };
    const auto scan_held = [&]() {
        CdCand h = none;
        for (int l = lane; l < P.local_tiles; l += 32)
            if (const CdCand *p = at(l)) h = better(*p, h);
        return h;
    };
    const int row0 = (cy * kCdWarps + warp) * R, row_step = P.ay * kCdWarps * R, col0 = cx * kTX, col_step = P.ax * kTX;
    CdCand held = scan_held();  // best of the local tiles l = lane mod 32
    CdCand best = held;         // what this thread has to offer
    CdCand fresh = none;        // its candidate of local tile fresh_tile, not yet in held
    int fresh_tile = -1;
    const auto settle = [&]() {
        if (fresh_tile < 0) return;
        const int o = best_lane(fresh);
        const CdCand t = make_uint4(__shfl_sync(0xffffffffu, fresh.x, o), __shfl_sync(0xffffffffu, fresh.y, o),
                                    __shfl_sync(0xffffffffu, fresh.z, o), __shfl_sync(0xffffffffu, fresh.w, o));
        if (lane == fresh_tile) held = t;
        fresh_tile = -1;
    };
    const float thr = __fmul_rn(P.lambda, P.alpha), slope = __fmul_rn(P.lambda, __fsub_rn(1.0f, P.alpha));
    CdCtl c{c0.iter, 0, 0, 0};
    for (int step = 0;; step++) {
        if (c.iter >= P.max_iter) {  // while (!converged & iter < iterations)
            c.done = 1;
            break;
        }
        if (step == kCdLaunchIters) break;
        const int b = step & 1;
        const uint32_t phase = (step >> 1) & 1, in_b = in_bar + 8 * b, sel_b = sel_bar + 8 * b;
        const unsigned epoch = static_cast<unsigned>(c.iter) + 1u;
        bool ok = true;
        if (lane == best_lane(best)) {
            if (rank == 0) {
                sm_in[b][warp] = best;
                cd_arrive(in_b);
            } else {
                st_peer(cd_peer(cd_shared(&sm_peer[b][warp]), 0), make_uint4(epoch, best.y, best.z, best.w));
                cd_signal(cd_peer(in_b, 0));
            }
        }
        if (rank == 0 && warp == 0) {
            ok = cd_wait(in_b, phase);
            CdCand v = none;
            if (PAIR && ok && lane < kCdWarps) ok = cd_await_peer(cd_shared(&sm_peer[b][lane]), epoch, v);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) {
                uint4 *slots = P.slots + (c.iter & 1) * kCdSlots;
                if (lane < kCdWarps) v = PAIR ? better(sm_in[b][lane], v) : sm_in[b][lane];
                if (lane == best_lane(v)) st_packet(slots + slot, make_uint4(epoch, v.y, v.z, v.w));
                v = none;
                unsigned want = 0;
#pragma unroll
                for (int j = 0; j < kCdPoll; j++) want |= lane + 32 * j < nslots ? 1u << j : 0u;
                const long long t0 = clock64();
                while (true) {
                    uint4 q[kCdPoll];
#pragma unroll
                    for (int j = 0; j < kCdPoll; j++)
                        q[j] = (want >> j) & 1u ? ld_packet(slots + lane + 32 * j) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                    for (int j = 0; j < kCdPoll; j++) {
                        if (q[j].x != epoch) continue;  // epochs start at 1
                        want &= ~(1u << j);
                        v = better(cd_unpack(q[j]), v);
                    }
                    if (!__any_sync(0xffffffffu, want != 0u)) break;
                    if (__any_sync(0xffffffffu, clock64() - t0 > kCdPatience)) {
                        ok = false;
                        break;
                    }
                }
                if (ok && lane == best_lane(v)) {
                    if (PAIR) {
                        st_peer(cd_peer(cd_shared(&sm_told[b]), 1), make_uint4(epoch, v.y, v.z, v.w));
                        cd_signal(cd_peer(sel_b, 1));
                    }
                    sm_sel[b] = v;
                    cd_arrive(sel_b);
                }
            }
        }
        settle();  // while the exchange is under way
        CdCand s = none;
        ok = ok && cd_wait(sel_b, phase);
        if (PAIR && rank == 1) ok = ok && cd_await_peer(cd_shared(&sm_told[b]), epoch, s);
        ok = __all_sync(0xffffffffu, ok);
        if (rank == 0) s = sm_sel[b];
        if (!ok) {
            c = CdCtl{c.iter, 1, 0, 2};
            if (lane == 0) P.report[1].error = 2;
            break;
        }
        if (__uint_as_float(s.x) < P.eps) {  // converged = maxPixel.PixelMaxDiff < epsilon
            c = CdCtl{c.iter, 1, 1, 0};
            break;
        }
        if (s.y == 0u) {  // none: the reference would index pixel (-1, -1)
            c = CdCtl{c.iter, 1, 0, 1};
            break;
        }
        c.iter++;
        if (!owner) continue;
        Window w;
        w.py = static_cast<int>((0xFFFFFFFFu - s.y) >> 16);
        w.px = static_cast<int>((0xFFFFFFFFu - s.y) & 0xFFFFu);
        w.yq = w.py - P.ph / 2;
        w.xq = w.px - P.pw / 2;
        w.y0 = max(w.yq, 0);
        w.x0 = max(w.xq, 0);
        w.y1 = min(w.yq + P.ph, P.n);
        w.x1 = min(w.xq + P.pw, P.n);
        w.xnew = __uint_as_float(s.z);
        w.xdiff = __fsub_rn(__uint_as_float(s.w), w.xnew);  // pixelOld - maxPixel.PixelNew
        // this warp's first rows and this CTA's first tile column that reach into the window
        const auto first = [](int q, int d, uint32_t inv) {
            return static_cast<int>(__umulhi(static_cast<uint32_t>(max(q, 0) + d - 1), inv) >> (kCdInvBits - 32));
        };
        const int ly0 = first(w.y0 - (R - 1) - row0, row_step, P.inv_row), yb0 = row0 + ly0 * row_step;
        const int lx0 = first(w.x0 - (kTX - 1) - col0, col_step, P.inv_col), xb0 = col0 + lx0 * col_step;
        best = held;
        if (yb0 >= w.y1 || xb0 >= w.x1) continue;
        if (in_regs && yb0 + row_step >= w.y1 && xb0 + col_step >= w.x1) {
            // one tile: its pixels are offered at once, in place of the candidate held of it
            fresh_tile = ly0 * P.local_x + lx0;
            fresh = update_rows<R>(P, thr, slope, yb0, xb0, w);
            best = better(fresh, lane == fresh_tile ? none : held);
            continue;
        }
        for (int ly = ly0, yb = yb0; yb < w.y1; ly++, yb += row_step)
            for (int lx = lx0, xb = xb0; xb < w.x1; lx++, xb += col_step) {
                fresh_tile = ly * P.local_x + lx;
                fresh = update_rows<R>(P, thr, slope, yb, xb, w);
                if (in_regs) {
                    settle();
                } else {
                    if (lane == best_lane(fresh)) *at(fresh_tile) = fresh;
                    fresh_tile = -1;
                }
            }
        if (!in_regs) {
            __syncwarp();
            held = scan_held();
        }
        best = held;
    }
    settle();
    if (in_regs)
        if (CdCand *p = at(lane)) *p = held;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *P.ctl = c;
        P.report[0] = c;
    }
    if (PAIR) cd_cluster_sync();  // no CTA leaves while the other may still write to it
}

// ------------------------------------------------------------------------------------------
// PSF preparation and the padded correlation (FP64, as the reference)

// psfPadded of PSF.CalcPaddedFourierCorrelation (Common.cs:128-135), FFT.Shift-ed, as complex.
__global__ void corr_pad_kernel(const float *psf, int h, int w, int H, int yh, int xh, double2 *out) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= static_cast<int64_t>(H) * H) return;
    int r = static_cast<int>(i / H), c = static_cast<int>(i % H);
    shift_index(H, r, c);  // out[i] = padded[shifted position]
    const int y = r - yh - 1, x = c - xh - 1;
    double v = 0.0;
    if (y >= 0 && x >= 0 && y < h && x < w) v = psf[static_cast<int64_t>(h - y - 1) * w + (w - x - 1)];
    out[i] = make_double2(v, 0.0);
}

// PaddedConvolver.InsertImage (PaddedConvolver.cs:87-107): image at (yh, xh) of an H x W buffer.  One
// block per row and 512 columns, so no thread divides.
__global__ void __launch_bounds__(256) conv_pad_kernel(const float *img, int n, int W, int yh, int xh, double *out) {
    const int row = blockIdx.x, r = row - yh;
    double *dst = out + static_cast<int64_t>(row) * W;
    const float *src = img + static_cast<int64_t>(r) * n;
    const bool inside = r >= 0 && r < n;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int col = blockIdx.y * 512 + k * 256 + threadIdx.x, c = col - xh;
        if (col < W) dst[col] = inside && c >= 0 && c < n ? static_cast<double>(src[c]) : 0.0;
    }
}

// The correlation kernel of PSF.CalcPaddedFourierCorrelation (Common.cs:128-135) after its FFT.Shift, for a
// transform of M x M >= H x H: the shifted H x H image's element at the circular offset (dy, dx)
// from the origin, |dy|, |dx| < H / 2, goes to the same offset of the M x M one.
__global__ void corr_real_kernel(const float *psf, int h, int w, int H, int M, int yh, int xh, double *out) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= static_cast<int64_t>(M) * M) return;
    int r = static_cast<int>(i / M), c = static_cast<int>(i % M);
    double v = 0.0;
    if (M != H) {
        r = 2 * r > M ? r - M : r;
        c = 2 * c > M ? c - M : c;
    }
    if (M == H || (2 * abs(r) < H && 2 * abs(c) < H)) {
        r = r < 0 ? r + H : r;
        c = c < 0 ? c + H : c;
        shift_index(H, r, c);  // out[i] = padded[shifted position]
        const int y = r - yh - 1, x = c - xh - 1;
        if (y >= 0 && x >= 0 && y < h && x < w) v = psf[static_cast<int64_t>(h - y - 1) * w + (w - x - 1)];
    }
    out[i] = v;
}

// Half plane of the Hermitian part of a Fourier kernel, times f: with a real image's transform I,
// Re(IFFT(I K)) = IFFT(I (K(k) + conj K(-k)) / 2).
__global__ void conv_kernel_half(const double2 *full, int H, int W, double f, double2 *half) {
    const int Wh = W / 2 + 1;
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= static_cast<int64_t>(H) * Wh) return;
    const int r = static_cast<int>(i / Wh), c = static_cast<int>(i % Wh);
    const double2 a = full[static_cast<int64_t>(r) * W + c];
    const double2 b = full[static_cast<int64_t>(r ? H - r : 0) * W + (c ? W - c : 0)];
    half[i] = make_double2(0.5 * f * (a.x + b.x), 0.5 * f * (a.y - b.y));
}

__global__ void conv_scale_kernel(double2 *a, int64_t count, double f) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i < count) a[i] = make_double2(f * a[i].x, f * a[i].y);
}

// a *= b over the half plane.  Bound by HBM (48 bytes an element); two elements a thread in flight.
__global__ void __launch_bounds__(256) conv_mul_kernel(double2 *__restrict__ a, const double2 *__restrict__ b, int64_t count) {
    const int64_t i0 = static_cast<int64_t>(blockIdx.x) * 512 + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int64_t i = i0 + k * 256;
        if (i >= count) continue;
        const double2 x = a[i], y = b[i];
        a[i] = make_double2(fma(x.x, y.x, -x.y * y.y), fma(x.x, y.y, x.y * y.x));
    }
}

// out[i][j] = (float)buf[i + yh][j + xh]   (PaddedConvolver.cs:55-62; the division is in the kernel)
__global__ void __launch_bounds__(256) conv_crop_kernel(const double *buf, int W, int yh, int xh, int n, float *out) {
    const double *src = buf + (static_cast<int64_t>(blockIdx.x) + yh) * W + xh;
    float *dst = out + static_cast<int64_t>(blockIdx.x) * n;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int c = blockIdx.y * 512 + k * 256 + threadIdx.x;
        if (c < n) dst[c] = static_cast<float>(src[c]);
    }
}

// psfPadded of PSF.CalcPSFSquared (Common.cs:165-167): psf at (h/2, w/2) of a 2h x 2w buffer.
__global__ void sq_pad_kernel(const float *psf, int h, int w, double2 *out) {
    const int W = 2 * w;
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= static_cast<int64_t>(2 * h) * W) return;
    const int r = static_cast<int>(i / W) - h / 2, c = static_cast<int>(i % W) - w / 2;
    const double v = (r >= 0 && c >= 0 && r < h && c < w) ? static_cast<double>(psf[static_cast<int64_t>(r) * w + c]) : 0.0;
    out[i] = make_double2(v, 0.0);
}

// a *= b, System.Numerics.Complex multiplication (re = ac - bd, im = bc + ad), un-fused.
__global__ void cmul_kernel(double2 *a, const double2 *b, int64_t count) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= count) return;
    const double2 x = a[i], y = b[i];
    a[i] = make_double2(__dsub_rn(__dmul_rn(x.x, y.x), __dmul_rn(x.y, y.y)),
                        __dadd_rn(__dmul_rn(x.y, y.x), __dmul_rn(x.x, y.y)));
}

// out[i][j] = (float)(buf[i + yh][j + xh].Real / len)   (PaddedConvolver.cs:55-62)
__global__ void conv_extract_kernel(const double2 *buf, int W, int yh, int xh, int n, double len, float *out) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= static_cast<int64_t>(n) * n) return;
    const int r = static_cast<int>(i / n), c = static_cast<int>(i % n);
    out[i] = static_cast<float>(buf[static_cast<int64_t>(r + yh) * W + c + xh].x / len);
}

// PSF.QueryScan (Common.cs:46-74) per pixel of the image section, from the host-built scan.
__global__ void amap_kernel(const double *scan, int sh, int sw, int ty_end, int tx_end, int sy, int sx, int oh,
                            int ow, float *out) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= static_cast<int64_t>(oh) * ow) return;
    const int yPixel = sy + static_cast<int>(i / ow), xPixel = sx + static_cast<int>(i % ow);
#define S(a, b) scan[static_cast<int64_t>(a) * sw + (b)]
    int yOver = max(0, (yPixel + (sh - sh / 2)) - ty_end);
    int xOver = max(0, (xPixel + (sw - sw / 2)) - tx_end);
    const int yUnder = -(yPixel - sh / 2), xUnder = -(xPixel - sw / 2);
    const int yUi = max(1, yUnder) - 1, xUi = max(1, xUnder) - 1;
    double v;
    if (yOver <= 0 && xOver <= 0 && yUnder <= 0 && xUnder <= 0) {
        v = S(sh - 1, sw - 1);
    } else if (yUnder > 0 && xUnder > 0) {
        v = __dadd_rn(__dsub_rn(__dsub_rn(S(sh - 1, sw - 1), S(sh - 1, xUi)), S(yUi, sw - 1)), S(yUi, xUi));
    } else {
        double corr = 0.0;
        if (yUnder > 0) corr = __dadd_rn(corr, S(yUi, sw - xOver - 1));
        if (xUnder > 0) corr = __dadd_rn(corr, S(sh - yOver - 1, xUi));
        v = __dsub_rn(S(sh - 1 - yOver, sw - 1 - xOver), corr);
    }
#undef S
    out[i] = static_cast<float>(v);
}

// Residuals.GetMax (Common.cs:244-251) and PSF.CalcMaxSidelobe (Common.cs:203-214): max over
// non-negative values starting at 0 (NaN propagates), as uint bits with atomicMax.
__global__ void max_kernel(const float *img, int n, int cut_off, int cut_len, bool sidelobe, unsigned int *out) {
    __shared__ float sm[kWarps];
    float m = 0.0f;
    const int64_t total = static_cast<int64_t>(n) * n;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        float v = img[i];
        if (sidelobe) {
            const int y = static_cast<int>(i / n), x = static_cast<int>(i % n);
            if ((y >= cut_off && y < cut_off + cut_len) && (x >= cut_off && x < cut_off + cut_len)) continue;
            v = fabsf(v);
        }
        m = cs_maxf(m, v);
    }
    for (int o = 16; o; o >>= 1) m = cs_maxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kWarps; k++) m = cs_maxf(m, sm[k]);
        atomicMax(out, __float_as_uint(m));  // m is +0, positive or NaN: its bits order as uint
    }
}

// Partial sums of squares (PSF.CalcMaxLipschitz, Common.cs:107-114) per block, fixed assignment.
__global__ void sumsq_kernel(const float *psf, int64_t count, double *partial) {
    __shared__ double sm[kWarps];
    double s = 0.0;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < count;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const float v = __fmul_rn(psf[i], psf[i]);
        s = __dadd_rn(s, static_cast<double>(v));
    }
    for (int o = 16; o; o >>= 1) s = __dadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kWarps; k++) s = __dadd_rn(s, sm[k]);
        partial[blockIdx.x] = s;
    }
}

// The two sums of the major cycle's objective (MajorCycle.cs:102) in the reference's types:
// Residuals.CalcPenalty's float squares (Common.cs:253-260) and ElasticNet.CalcPenalty's
// lambda * ElasticNetPenalty (Common.cs:22-23, 31-41; a float expression widened to double),
// each summed in double: per-block partials, summed in block order on the host.
__global__ void objective_kernel(const float *dirty, const float *x, int64_t count, float lambda, float alpha,
                                 double *partial) {
    __shared__ double sm[2][kWarps];
    double sr = 0.0, sx = 0.0;
    const float half_1ma = __fmul_rn(1.0f / 2.0f, __fsub_rn(1.0f, alpha));
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < count;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const float r = dirty[i], v = x[i];
        sr = __dadd_rn(sr, static_cast<double>(__fmul_rn(r, r)));
        const float pen = __fadd_rn(__fmul_rn(half_1ma, __fmul_rn(v, v)), __fmul_rn(alpha, fabsf(v)));
        sx = __dadd_rn(sx, __dmul_rn(static_cast<double>(lambda), static_cast<double>(pen)));
    }
    for (int o = 16; o; o >>= 1) {
        sr = __dadd_rn(sr, __shfl_xor_sync(0xffffffffu, sr, o));
        sx = __dadd_rn(sx, __shfl_xor_sync(0xffffffffu, sx, o));
    }
    if ((threadIdx.x & 31) == 0) {
        sm[0][threadIdx.x >> 5] = sr;
        sm[1][threadIdx.x >> 5] = sx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kWarps; k++) {
            sr = __dadd_rn(sr, sm[0][k]);
            sx = __dadd_rn(sx, sm[1][k]);
        }
        partial[2 * blockIdx.x] = sr;
        partial[2 * blockIdx.x + 1] = sx;
    }
}

// PSF.Cut (Common.cs:216-226) of a square n x n image.
__global__ void cut_kernel(const float *psf, int n, int m, int off, float *out) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= static_cast<int64_t>(m) * m) return;
    const int y = static_cast<int>(i / m), x = static_cast<int>(i % m);
    out[i] = psf[static_cast<int64_t>(off + y) * n + off + x];
}

// psf2[i, j] *= (maxFull / maxCut)  (FastSerialCD.ResetLipschitzMap, FastSerialCD.cs:123-126)
__global__ void scale_kernel(float *a, int64_t count, float f) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i < count) a[i] = __fmul_rn(a[i], f);
}

// Visibilities.Substract (Common.cs:305-317) on complex64.
__global__ void vis_subtract_kernel(const float2 *v0, const float2 *v1, const uint8_t *flags, int64_t count,
                                    float2 *out) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= count) return;
    const float2 a = v0[i], b = v1[i];
    out[i] = flags[i] ? make_float2(0.0f, 0.0f) : make_float2(a.x - b.x, a.y - b.y);
}

// FFT.Shift(xImage) then the complex input of FFT.Forward (MajorCycle.cs:125-126).
__global__ void shifted_real_to_c64_kernel(const float *img, int n, float2 *out) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= static_cast<int64_t>(n) * n) return;
    int r = static_cast<int>(i / n), c = static_cast<int>(i % n);
    shift_index(n, r, c);
    out[i] = make_float2(img[static_cast<int64_t>(r) * n + c], 0.0f);
}

inline unsigned grid_for(int64_t count, int threads = 256) {
    return static_cast<unsigned>((count + threads - 1) / threads);
}

// ------------------------------------------------------------------------------------------
// host helpers

// The double prefix-sum scan of psf^2 in PSF.CalcAMap (Common.cs:84-93), in the reference's
// order (host: its dependencies make it sequential and it is psf-sized).
void amap_scan(const float *psf, int h, int w, std::vector<double> &scan) {
    scan.assign(static_cast<size_t>(h) * w, 0.0);
    for (int i = 0; i < h; i++)
        for (int j = 0; j < w; j++) {
            const double iB = i > 0 ? scan[static_cast<size_t>(i - 1) * w + j] : 0.0;
            const double jB = j > 0 ? scan[static_cast<size_t>(i) * w + j - 1] : 0.0;
            const double ijB = (i > 0 && j > 0) ? scan[static_cast<size_t>(i - 1) * w + j - 1] : 0.0;
            const float cur = psf[static_cast<size_t>(i) * w + j] * psf[static_cast<size_t>(i) * w + j];
            scan[static_cast<size_t>(i) * w + j] = static_cast<double>(cur) + iB + jB - ijB;
        }
}

struct Z2Z {
    cufftHandle h = 0;
    int ny = 0, nx = 0;
    p9idg_status get(int y, int x, cudaStream_t st) {
        if (h && (y != ny || x != nx)) {
            cufftDestroy(h);
            h = 0;
        }
        if (!h) {
            if (cufftPlan2d(&h, y, x, CUFFT_Z2Z) != CUFFT_SUCCESS) {
                h = 0;
                return fail(P9IDG_CUDA_ERROR, "cufftPlan2d (Z2Z) failed");
            }
            ny = y;
            nx = x;
        }
        CUFFT(cufftSetStream(h, st));
        return P9IDG_OK;
    }
    void release() {
        if (h) cufftDestroy(h);
        h = 0;
    }
};

// PSF.CalcPaddedFourierCorrelation on the device: psf (device h x w) -> out (device H x H complex).
p9idg_status dev_padded_correlation(const float *d_psf, int h, int w, int pad_y, int pad_x, double2 *d_out, Z2Z &fft,
                                    cudaStream_t st) {
    const int H = pad_y + h, W = pad_x + w;
    if (H != W) return fail(P9IDG_INVALID_ARGUMENT, "padded PSF must be square (FFT.Shift uses the row count)");
    corr_pad_kernel<<<grid_for(static_cast<int64_t>(H) * H), 256, 0, st>>>(d_psf, h, w, H, pad_y / 2, pad_x / 2, d_out);
    CK(cudaGetLastError());
    TRY(fft.get(H, W, st));
    CUFFT(cufftExecZ2Z(fft.h, reinterpret_cast<cufftDoubleComplex *>(d_out), reinterpret_cast<cufftDoubleComplex *>(d_out),
                       CUFFT_FORWARD));
    return P9IDG_OK;
}

// PSF.CalcPSFSquared on the device: psf (device h x w) -> out (device 2h x 2w float).
p9idg_status dev_psf_squared(const float *d_psf, int h, int w, float *d_out, Buf &b0, Buf &b1, Z2Z &fft,
                             cudaStream_t st) {
    const int64_t count = static_cast<int64_t>(2 * h) * (2 * w);
    CK(b0.ensure(sizeof(double2) * count));
    CK(b1.ensure(sizeof(double2) * count));
    TRY(dev_padded_correlation(d_psf, h, w, h, w, b0.as<double2>(), fft, st));
    sq_pad_kernel<<<grid_for(count), 256, 0, st>>>(d_psf, h, w, b1.as<double2>());
    CK(cudaGetLastError());
    auto *s = reinterpret_cast<cufftDoubleComplex *>(b1.p);
    CUFFT(cufftExecZ2Z(fft.h, s, s, CUFFT_FORWARD));
    cmul_kernel<<<grid_for(count), 256, 0, st>>>(b1.as<double2>(), b0.as<double2>(), count);
    CK(cudaGetLastError());
    CUFFT(cufftExecZ2Z(fft.h, s, s, CUFFT_INVERSE));
    // FFT.Backward(PSF2, (long)psfCorrelated.Length): Re / count
    conv_extract_kernel<<<grid_for(count), 256, 0, st>>>(b1.as<double2>(), 2 * w, 0, 0, 2 * w,
                                                         static_cast<double>(count), d_out);
    CK(cudaGetLastError());
    return P9IDG_OK;
}

// Residuals.GetMax / PSF.CalcMaxSidelobe on a device n x n image (synchronises the stream).
p9idg_status dev_max(const float *d_img, int n, int cut_factor, unsigned int *d_word, float *out, cudaStream_t st) {
    CK(cudaMemsetAsync(d_word, 0, sizeof(unsigned int), st));
    const int m = cut_factor > 0 ? n / cut_factor : 0;
    const int off = cut_factor > 0 ? n / 2 - m / 2 : 0;
    max_kernel<<<std::min<unsigned>(grid_for(static_cast<int64_t>(n) * n), 1024), kNT, 0, st>>>(d_img, n, off, m,
                                                                                                 cut_factor > 0, d_word);
    CK(cudaGetLastError());
    unsigned int bits = 0;
    CK(cudaMemcpyAsync(&bits, d_word, sizeof(bits), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    std::memcpy(out, &bits, sizeof(float));
    return P9IDG_OK;
}

// Residuals.CalcPenalty(dirty) + ElasticNet.CalcPenalty(x, lambda, alpha) (MajorCycle.cs:102).
p9idg_status dev_objective(const float *d_dirty, const float *d_x, int64_t count, float lambda, float alpha,
                           Buf &partial, double *out, cudaStream_t st) {
    constexpr int kBlocks = 256;
    CK(partial.ensure(sizeof(double) * 2 * kBlocks));
    objective_kernel<<<kBlocks, kNT, 0, st>>>(d_dirty, d_x, count, lambda, alpha, partial.as<double>());
    CK(cudaGetLastError());
    double h[2 * kBlocks];
    CK(cudaMemcpyAsync(h, partial.p, sizeof(h), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    double r = 0.0, x = 0.0;
    for (int b = 0; b < kBlocks; b++) {
        r += h[2 * b];
        x += h[2 * b + 1];
    }
    *out = 0.5 * r + x;
    return P9IDG_OK;
}

// PSF.CalcMaxLipschitz of a device image (deterministic: fixed partials summed in order).
p9idg_status dev_sumsq(const float *d_img, int64_t count, Buf &partial, double *out, cudaStream_t st) {
    constexpr int kBlocks = 256;
    CK(partial.ensure(sizeof(double) * kBlocks));
    sumsq_kernel<<<kBlocks, kNT, 0, st>>>(d_img, count, partial.as<double>());
    CK(cudaGetLastError());
    double h[kBlocks];
    CK(cudaMemcpyAsync(h, partial.p, sizeof(h), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    double s = 0.0;
    for (double v : h) s += v;
    *out = s;
    return P9IDG_OK;
}

}  // namespace

// ------------------------------------------------------------------------------------------
// PaddedConvolver

// The image and the result are real, so the two transforms are real-to-complex and complex-to-real
// over the half plane with the Hermitian part of the kernel: half the FP64 work and traffic of
// complex ones (FP64 arithmetic bounds them on this GPU).  A correlation made from a PSF is a linear
// one that the padding keeps from wrapping, so it may run at any larger size: the next one whose
// factors are 2, 3, 5 and 7 (a size with a large prime factor costs several times as much).
// 3072^2 with a 384^2 PSF: 5.26 -> 2.97 ms; 2.5 to 3.9 times faster at sizes with larger factors
// (in place, with one buffer less: 3.03 ms).
struct ConvSize {  // what the transforms of one size need
    int my = 0, mx = 0;
    Buf kernel, real, spec, work;  // half plane, padded image, its half plane, cuFFT's area
    cufftHandle fwd = 0, inv = 0;
    ~ConvSize() {
        if (fwd) cufftDestroy(fwd);
        if (inv) cufftDestroy(inv);
    }
};

struct p9idg_convolver {
    int device = -1;
    cudaStream_t stream = nullptr, own = nullptr;
    int H = 0, W = 0, ky = 0, kx = 0;  // the padded size and the PSF's
    int n_max = 0;                     // largest image that `made` serves
    std::unique_ptr<ConvSize> made;    // size >= H x W
    std::unique_ptr<ConvSize> padded;  // correlations: H x W, once an image larger than n_max has been seen
    Buf psf;                           // (correlations)
};

namespace {

int smooth_size(int n) {  // smallest even m >= n with no prime factor above 7
    for (int m = n + (n & 1);; m += 2) {
        int r = m;
        for (int p : {2, 3, 5, 7})
            while (r % p == 0) r /= p;
        if (r == 1) return m;
    }
}

p9idg_status conv_plans(ConvSize *z, int my, int mx) {
    z->my = my;
    z->mx = mx;
    const size_t half = static_cast<size_t>(my) * (mx / 2 + 1);
    CK(z->kernel.ensure(sizeof(double2) * half));
    CK(z->spec.ensure(sizeof(double2) * half));
    CK(z->real.ensure(sizeof(double) * static_cast<size_t>(my) * mx));
    size_t need = 0, w = 0;  // the two transforms never run at once: one work area
    for (int k = 0; k < 2; k++) {
        cufftHandle *h = k ? &z->inv : &z->fwd;
        CUFFT(cufftCreate(h));
        CUFFT(cufftSetAutoAllocation(*h, 0));
        CUFFT(cufftMakePlan2d(*h, my, mx, k ? CUFFT_Z2D : CUFFT_D2Z, &w));
        need = std::max(need, w);
    }
    CK(z->work.ensure(need));
    CUFFT(cufftSetWorkArea(z->fwd, z->work.p));
    CUFFT(cufftSetWorkArea(z->inv, z->work.p));
    return P9IDG_OK;
}

// What the unnormalised inverse of size my x mx is multiplied by: its own size, and the reference's
// count over its Length, a 32-bit int (PaddedConvolver.cs:57).
double conv_factor(const p9idg_convolver *c, const ConvSize *z) {
    const int64_t count = static_cast<int64_t>(c->H) * c->W;
    return static_cast<double>(count) / static_cast<double>(static_cast<int32_t>(count)) /
           (static_cast<double>(z->my) * z->mx);
}

p9idg_status conv_init(p9idg_convolver *c, int H, int W, int ky, int kx) {
    CK(cudaGetDevice(&c->device));
    CK(cudaStreamCreateWithFlags(&c->own, cudaStreamNonBlocking));
    c->stream = c->own;
    c->H = H;
    c->W = W;
    c->ky = ky;
    c->kx = kx;
    return P9IDG_OK;
}

void conv_release(p9idg_convolver *c) {
    if (c->stream) cudaStreamSynchronize(c->stream);
    c->made.reset();
    c->padded.reset();
    c->psf.release();
    if (c->own) cudaStreamDestroy(c->own);
}

// The transforms of m x m for a correlation with c->psf, made for images of n x n, into `out` once they are
// complete.
p9idg_status conv_correlation(p9idg_convolver *c, int m, int n, std::unique_ptr<ConvSize> &out) {
    std::unique_ptr<ConvSize> z(new (std::nothrow) ConvSize());
    if (!z) return fail(P9IDG_OUT_OF_MEMORY, "convolver allocation");
    TRY(conv_plans(z.get(), m, m));
    corr_real_kernel<<<grid_for(static_cast<int64_t>(m) * m), 256, 0, c->stream>>>(
        c->psf.as<float>(), c->ky, c->kx, c->H, m, n / 2, n / 2, z->real.as<double>());
    CK(cudaGetLastError());
    CUFFT(cufftSetStream(z->fwd, c->stream));
    CUFFT(cufftExecD2Z(z->fwd, z->real.as<double>(), reinterpret_cast<cufftDoubleComplex *>(z->kernel.p)));
    const int64_t half = static_cast<int64_t>(m) * (m / 2 + 1);
    conv_scale_kernel<<<grid_for(half), 256, 0, c->stream>>>(z->kernel.as<double2>(), half, conv_factor(c, z.get()));
    CK(cudaGetLastError());
    out = std::move(z);
    return P9IDG_OK;
}

// PaddedConvolver.Convolve (PaddedConvolver.cs:43-65) of a device n x n image.
p9idg_status conv_run(p9idg_convolver *c, const float *d_img, int n, float *d_out) {
    if (n + c->ky / 2 > c->H || n + c->kx / 2 > c->W)
        return fail(P9IDG_INVALID_ARGUMENT, "image larger than the convolver's padded buffer");
    // an image larger than the correlation was made for wraps at the padded size, which keeps transforms of its own
    const bool larger = n > c->n_max;
    if (larger && !c->padded) TRY(conv_correlation(c, c->H, c->n_max, c->padded));
    const ConvSize *z = larger ? c->padded.get() : c->made.get();
    const int64_t half = static_cast<int64_t>(z->my) * (z->mx / 2 + 1);
    const auto cols = [](int w) { return static_cast<unsigned>((w + 511) / 512); };
    conv_pad_kernel<<<dim3(z->my, cols(z->mx)), 256, 0, c->stream>>>(d_img, n, z->mx, c->ky / 2, c->kx / 2,
                                                                     z->real.as<double>());
    CK(cudaGetLastError());
    auto *s = reinterpret_cast<cufftDoubleComplex *>(z->spec.p);
    CUFFT(cufftSetStream(z->fwd, c->stream));
    CUFFT(cufftSetStream(z->inv, c->stream));
    CUFFT(cufftExecD2Z(z->fwd, z->real.as<double>(), s));
    conv_mul_kernel<<<static_cast<unsigned>((half + 511) / 512), 256, 0, c->stream>>>(
        z->spec.as<double2>(), z->kernel.as<double2>(), half);
    CK(cudaGetLastError());
    CUFFT(cufftExecZ2D(z->inv, s, z->real.as<double>()));
    conv_crop_kernel<<<dim3(n, cols(n)), 256, 0, c->stream>>>(z->real.as<double>(), z->mx, c->ky / 2, c->kx / 2, n, d_out);
    CK(cudaGetLastError());
    return P9IDG_OK;
}

}  // namespace

// ------------------------------------------------------------------------------------------
// FastSerialCD

struct p9idg_cd {
    int device = -1;
    cudaStream_t stream = nullptr, own = nullptr;
    int n = 0, ph = 0, pw = 0;  // image size, psf2 size
    int tiles_x = 0, tiles_y = 0;
    float max_lipschitz = 0.0f;
    Buf x, g, amap, psf2, tile_key, cand, slots, ctl, pick, word, partial, sq0, sq1, psf_tmp;
    Z2Z fft;
    CdParams hp{};
    CdCtl *h_ctl = nullptr;                // pinned [2]
    unsigned long long *h_pick = nullptr;  // pinned: selected key
    cudaEvent_t ev_ctl = nullptr;          // the control word of a launch has reached h_ctl
};

namespace {

p9idg_status cd_set_maps(p9idg_cd *cd, const float *h_psf, int h, int w) {
    // psf2 = PSF.CalcPSFSquared(psf); aMap = PSF.CalcAMap(psf, totalSize); MaxLipschitz = GetMax(psf2)
    const int n = cd->n;
    CK(cd->psf_tmp.ensure(sizeof(float) * static_cast<size_t>(h) * w));
    CK(cudaMemcpyAsync(cd->psf_tmp.p, h_psf, sizeof(float) * static_cast<size_t>(h) * w, cudaMemcpyHostToDevice,
                       cd->stream));
    CK(cd->psf2.ensure(sizeof(float) * static_cast<size_t>(4) * h * w));
    TRY(dev_psf_squared(cd->psf_tmp.as<float>(), h, w, cd->psf2.as<float>(), cd->sq0, cd->sq1, cd->fft, cd->stream));
    cd->ph = 2 * h;
    cd->pw = 2 * w;
    std::vector<double> scan;
    amap_scan(h_psf, h, w, scan);
    Buf d_scan;
    CK(d_scan.ensure(sizeof(double) * scan.size()));
    cudaError_t e = cudaMemcpyAsync(d_scan.p, scan.data(), sizeof(double) * scan.size(), cudaMemcpyHostToDevice,
                                    cd->stream);
    if (e == cudaSuccess) {
        amap_kernel<<<grid_for(static_cast<int64_t>(n) * n), 256, 0, cd->stream>>>(d_scan.as<double>(), h, w, n, n, 0,
                                                                                   0, n, n, cd->amap.as<float>());
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(cd->stream);
    d_scan.release();
    if (e != cudaSuccess) return cuda_fail(e, "aMap");
    // psf2 is square (2h x 2w with h == w for every caller); GetMax over it
    float m = 0.0f;
    if (cd->ph == cd->pw) {
        TRY(dev_max(cd->psf2.as<float>(), cd->ph, 0, cd->word.as<unsigned int>(), &m, cd->stream));
    } else {
        std::vector<float> host(static_cast<size_t>(cd->ph) * cd->pw);
        CK(cudaMemcpy(host.data(), cd->psf2.p, sizeof(float) * host.size(), cudaMemcpyDeviceToHost));
        for (float v : host) m = v > m ? v : m;
    }
    cd->max_lipschitz = m;
    return P9IDG_OK;
}

// Launch of the run kernel: nctas CTAs, in pairs from kCdPairFrom on.
struct CdLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    bool pairs;
    CdLaunch(int nctas, cudaStream_t stream) : pairs(nctas >= kCdPairFrom) {
        const unsigned c = pairs ? 2 : 1;
        cfg.gridDim = dim3((static_cast<unsigned>(nctas) + c - 1) / c * c);
        cfg.blockDim = dim3(kCdNT);
        cfg.stream = stream;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = c;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeCooperative;
        attr[1].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
    }
};

// Deals the tiles out to the CTAs of the run kernel: the ay x ax torus that leaves the fewest tiles of a
// whole window to one CTA.  Of several, the one of the fewest CTAs that keep their candidates in registers
// (at most 32 tiles each), since the exchange grows with them (1024^2 with a 256^2 window: 24 CTAs 2.97 ms a
// 1000 iterations, 104 CTAs 3.20 ms); if none does, the one of the fewest tiles a CTA.
p9idg_status cd_layout(p9idg_cd *cd) {
    CdParams &p = cd->hp;
    int coop = 0, pairs = 0;
    CK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, cd->device));
    CdLaunch two(kCdPairFrom, cd->stream);
    two.cfg.numAttrs = 1;
    CK(cudaOccupancyMaxActiveClusters(&pairs, cd_run_kernel<2, true>, &two.cfg));
    const int most = 2 * std::min(pairs, kCdSlots);
    if (!coop || most < 2) return fail(P9IDG_UNSUPPORTED, "the device cannot run the coordinate-descent kernel");
    const auto div = [](int a, int b) { return (a + b - 1) / b; };
    // One row a warp halves the evaluation, which is about half of an iteration, and doubles the CTAs that
    // exchange candidates.  1000 iterations at 376^2 with an 80^2 window: 2.30 ms with one row (10 tiles),
    // 2.85 with two; at 1024^2 with a 256^2 window: 3.29 ms with one row (42 tiles), 2.97 with two.
    p.rows = 1;
    const auto window_rows = [&]() { return std::min(div(cd->n, kCdWarps * p.rows), div(cd->ph, kCdWarps * p.rows) + 1); };
    cd->tiles_x = div(cd->n, kTX);
    const int wx = std::min(cd->tiles_x, div(cd->pw, kTX) + 1);
    if (window_rows() * wx > std::min(32, most)) p.rows = 2;
    cd->tiles_y = div(cd->n, kCdWarps * p.rows);
    const int wy = window_rows();
    int64_t best = INT64_MAX;
    for (int ax = 1; ax <= std::min(cd->tiles_x, most); ax++)
        for (int ay = 1; ay <= std::min(cd->tiles_y, most / ax); ay++) {
            const int64_t window = static_cast<int64_t>(div(wy, ay)) * div(wx, ax),
                          all = static_cast<int64_t>(div(cd->tiles_y, ay)) * div(cd->tiles_x, ax);
            const int64_t cost = (window << 32) + (all > 32 ? all << 8 : ax * ay);
            if (cost < best) {
                best = cost;
                p.ax = ax;
                p.ay = ay;
            }
        }
    p.tiles_x = cd->tiles_x;
    p.tiles_y = cd->tiles_y;
    const uint32_t row_step = static_cast<uint32_t>(p.ay * kCdWarps * p.rows), col_step = static_cast<uint32_t>(p.ax * kTX);
    p.inv_row = static_cast<uint32_t>(((1ull << kCdInvBits) + row_step - 1) / row_step);
    p.inv_col = static_cast<uint32_t>(((1ull << kCdInvBits) + col_step - 1) / col_step);
    p.local_x = div(cd->tiles_x, p.ax);
    p.local_tiles = div(cd->tiles_y, p.ay) * p.local_x;
    const size_t nt = static_cast<size_t>(cd->tiles_x) * cd->tiles_y;
    CK(cd->tile_key.ensure(sizeof(unsigned long long) * nt));
    CK(cd->cand.ensure(sizeof(CdCand) * kCdWarps * nt));
    p.cand = cd->cand.as<CdCand>();
    p.tile_key = cd->tile_key.as<unsigned long long>();
    return P9IDG_OK;
}

// Candidates of every tile with the parameters' lambda and alpha, control reset.
p9idg_status cd_scan(p9idg_cd *cd) {
    const dim3 grid(cd->tiles_x, cd->tiles_y);
    if (cd->hp.rows == 1)
        cd_scan_kernel<1><<<grid, kCdNT, 0, cd->stream>>>(cd->hp);
    else
        cd_scan_kernel<2><<<grid, kCdNT, 0, cd->stream>>>(cd->hp);
    CK(cudaGetLastError());
    return P9IDG_OK;
}

// FastSerialCD.Deconvolve on device buffers x, g (n x n float), in place.
p9idg_status cd_run(p9idg_cd *cd, float *d_x, float *d_g, float lambda, float alpha, int32_t max_iter, float eps,
                    p9idg_cd_result *res) {
    const auto t0 = std::chrono::steady_clock::now();
    cd->hp.x = d_x;
    cd->hp.g = d_g;
    cd->hp.lambda = lambda;
    cd->hp.alpha = alpha;
    cd->hp.eps = eps;
    cd->hp.max_iter = max_iter;
    TRY(cd_scan(cd));
    cd->h_ctl[0] = cd->h_ctl[1] = CdCtl{};
    if (max_iter <= 0) {
        CK(cudaStreamSynchronize(cd->stream));
        cd->h_ctl[0].done = 1;
    }
    // One launch stays in flight while the host looks at the state the previous one left, so the GPU never
    // waits on the host; a launch after the stopping one does nothing (it sees the done flag).
    const int64_t launches = (static_cast<int64_t>(std::max(max_iter, 0)) + kCdLaunchIters - 1) / kCdLaunchIters;
    CdLaunch run(cd->hp.ax * cd->hp.ay, cd->stream);
    const auto of_rows = [&](auto one, auto two) { return cd->hp.rows == 1 ? one : two; };
    const auto kernel = run.pairs ? of_rows(cd_run_kernel<1, true>, cd_run_kernel<2, true>)
                                  : of_rows(cd_run_kernel<1, false>, cd_run_kernel<2, false>);
    if (launches > 0) CK(cudaLaunchKernelEx(&run.cfg, kernel, cd->hp));
    for (int64_t r = 0; r < launches; r++) {
        CK(cudaEventRecord(cd->ev_ctl, cd->stream));
        if (r + 1 < launches) CK(cudaLaunchKernelEx(&run.cfg, kernel, cd->hp));
        CK(cudaEventSynchronize(cd->ev_ctl));
        if (static_cast<volatile CdCtl *>(cd->h_ctl)->done) break;
    }
    CK(cudaStreamSynchronize(cd->stream));  // the launch in flight, if any
    if (!cd->h_ctl[0].done || cd->h_ctl[1].error) return fail(P9IDG_DEVICE_CHECK_FAILED, "coordinate descent did not stop");
    if (cd->h_ctl[0].error)
        return fail(P9IDG_INVALID_ARGUMENT,
                    "no pixel changes and epsilon <= 0: the reference would index pixel (-1, -1)");
    if (res) {
        res->converged = cd->h_ctl[0].converged;
        res->iterations = cd->h_ctl[0].iter;
        res->elapsed_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }
    return P9IDG_OK;
}

p9idg_status cd_abs_max(p9idg_cd *cd, const float *d_x, const float *d_g, float lambda, float alpha, float *out) {
    cd->hp.x = const_cast<float *>(d_x);
    cd->hp.g = const_cast<float *>(d_g);
    cd->hp.lambda = lambda;
    cd->hp.alpha = alpha;
    TRY(cd_scan(cd));
    cd_pick_kernel<<<1, kCdNT, 0, cd->stream>>>(cd->hp.tile_key, cd->tiles_x * cd->tiles_y, cd->pick.as<unsigned long long>());
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(cd->h_pick, cd->pick.p, sizeof(unsigned long long), cudaMemcpyDeviceToHost, cd->stream));
    CK(cudaStreamSynchronize(cd->stream));
    const uint32_t bits = static_cast<uint32_t>(*cd->h_pick >> 32);
    std::memcpy(out, &bits, sizeof(float));
    return P9IDG_OK;
}

void cd_release(p9idg_cd *cd) {
    if (cd->stream) cudaStreamSynchronize(cd->stream);
    if (cd->ev_ctl) cudaEventDestroy(cd->ev_ctl);
    Buf *bufs[] = {&cd->x, &cd->g, &cd->amap, &cd->psf2, &cd->tile_key, &cd->cand, &cd->slots, &cd->ctl,
                   &cd->pick, &cd->word, &cd->partial, &cd->sq0, &cd->sq1, &cd->psf_tmp};
    for (Buf *b : bufs) b->release();
    cd->fft.release();
    if (cd->h_ctl) cudaFreeHost(cd->h_ctl);
    if (cd->h_pick) cudaFreeHost(cd->h_pick);
    if (cd->own) cudaStreamDestroy(cd->own);
}

p9idg_status cd_init(p9idg_cd *cd, int n, const float *psf, int h, int w) {
    CK(cudaGetDevice(&cd->device));
    CK(cudaStreamCreateWithFlags(&cd->own, cudaStreamNonBlocking));
    cd->stream = cd->own;
    CK(cudaMallocHost(reinterpret_cast<void **>(&cd->h_ctl), 2 * sizeof(CdCtl)));
    CK(cudaMallocHost(reinterpret_cast<void **>(&cd->h_pick), sizeof(unsigned long long)));
    CK(cudaEventCreateWithFlags(&cd->ev_ctl, cudaEventDisableTiming));
    cd->n = n;
    CK(cd->amap.ensure(sizeof(float) * static_cast<size_t>(n) * n));
    CK(cd->slots.ensure(sizeof(uint4) * 2 * kCdSlots));
    CK(cd->ctl.ensure(sizeof(CdCtl)));
    CK(cd->pick.ensure(sizeof(unsigned long long)));
    CK(cd->word.ensure(sizeof(unsigned int)));
    TRY(cd_set_maps(cd, psf, h, w));
    cd->hp = CdParams{};
    cd->hp.a = cd->amap.as<float>();
    cd->hp.psf2 = cd->psf2.as<float>();
    cd->hp.slots = cd->slots.as<uint4>();
    cd->hp.ctl = cd->ctl.as<CdCtl>();
    cd->hp.report = cd->h_ctl;
    cd->hp.n = n;
    cd->hp.ph = cd->ph;
    cd->hp.pw = cd->pw;
    return cd_layout(cd);
}

p9idg_status check_cd_args(int32_t n, const float *psf, int32_t h, int32_t w) {
    if (n <= 0 || n > 65535 || !psf || h <= 0 || w <= 0) return fail(P9IDG_INVALID_ARGUMENT, "invalid argument");
    if (h != w) return fail(P9IDG_INVALID_ARGUMENT, "the PSF must be square (FFT.Shift uses the row count)");
    return P9IDG_OK;
}

}  // namespace

extern "C" {

p9idg_status p9idg_cd_create(int32_t n, const float *psf, int32_t psf_h, int32_t psf_w, p9idg_cd **out) {
    if (!out) return fail(P9IDG_INVALID_ARGUMENT, "null output pointer");
    *out = nullptr;
    TRY(check_cd_args(n, psf, psf_h, psf_w));
    TRY(have_device());
    auto *cd = new (std::nothrow) p9idg_cd();
    if (!cd) return fail(P9IDG_OUT_OF_MEMORY, "deconvolver allocation");
    p9idg_status st = cd_init(cd, n, psf, psf_h, psf_w);
    if (st != P9IDG_OK) {
        cd_release(cd);
        delete cd;
        return st;
    }
    *out = cd;
    return P9IDG_OK;
}

p9idg_status p9idg_cd_max_lipschitz(const p9idg_cd *cd, float *out) {
    if (!cd || !out) return fail(P9IDG_INVALID_ARGUMENT, "null argument");
    *out = cd->max_lipschitz;
    return P9IDG_OK;
}

p9idg_status p9idg_cd_get_maps(p9idg_cd *cd, float *psf2_out, float *amap_out) {
    if (!cd) return fail(P9IDG_INVALID_ARGUMENT, "null deconvolver");
    CK(cudaSetDevice(cd->device));
    CK(cudaStreamSynchronize(cd->stream));
    if (psf2_out) CK(cudaMemcpy(psf2_out, cd->psf2.p, sizeof(float) * static_cast<size_t>(cd->ph) * cd->pw,
                                cudaMemcpyDeviceToHost));
    if (amap_out) CK(cudaMemcpy(amap_out, cd->amap.p, sizeof(float) * static_cast<size_t>(cd->n) * cd->n,
                                cudaMemcpyDeviceToHost));
    return P9IDG_OK;
}

p9idg_status p9idg_cd_psf2_size(const p9idg_cd *cd, int32_t *h, int32_t *w) {
    if (!cd || !h || !w) return fail(P9IDG_INVALID_ARGUMENT, "null argument");
    *h = cd->ph;
    *w = cd->pw;
    return P9IDG_OK;
}

p9idg_status p9idg_cd_set_stream(p9idg_cd *cd, void *cuda_stream) {
    if (!cd) return fail(P9IDG_INVALID_ARGUMENT, "null deconvolver");
    cudaStream_t s = cuda_stream ? static_cast<cudaStream_t>(cuda_stream) : cd->own;
    if (s != cd->stream) {
        CK(cudaStreamSynchronize(cd->stream));
        cd->stream = s;
    }
    return P9IDG_OK;
}

p9idg_status p9idg_cd_deconvolve_device(p9idg_cd *cd, float *d_x, float *d_bmap, float lambda, float alpha,
                                        int32_t max_iter, float epsilon, p9idg_cd_result *res) {
    if (!cd || !d_x || !d_bmap) return fail(P9IDG_INVALID_ARGUMENT, "null argument");
    CK(cudaSetDevice(cd->device));
    return cd_run(cd, d_x, d_bmap, lambda, alpha, max_iter, epsilon, res);
}

p9idg_status p9idg_cd_deconvolve(p9idg_cd *cd, float *x, float *bmap, float lambda, float alpha, int32_t max_iter,
                                 float epsilon, p9idg_cd_result *res) {
    if (!cd || !x || !bmap) return fail(P9IDG_INVALID_ARGUMENT, "null argument");
    CK(cudaSetDevice(cd->device));
    const size_t bytes = sizeof(float) * static_cast<size_t>(cd->n) * cd->n;
    CK(cd->x.ensure(bytes));
    CK(cd->g.ensure(bytes));
    CK(cudaMemcpyAsync(cd->x.p, x, bytes, cudaMemcpyHostToDevice, cd->stream));
    CK(cudaMemcpyAsync(cd->g.p, bmap, bytes, cudaMemcpyHostToDevice, cd->stream));
    TRY(cd_run(cd, cd->x.as<float>(), cd->g.as<float>(), lambda, alpha, max_iter, epsilon, res));
    // the reference updates reconstruction and bMap in place
    CK(cudaMemcpyAsync(x, cd->x.p, bytes, cudaMemcpyDeviceToHost, cd->stream));
    CK(cudaMemcpyAsync(bmap, cd->g.p, bytes, cudaMemcpyDeviceToHost, cd->stream));
    CK(cudaStreamSynchronize(cd->stream));
    return P9IDG_OK;
}

p9idg_status p9idg_cd_get_abs_max_diff_device(p9idg_cd *cd, const float *d_x, const float *d_bmap, float lambda,
                                              float alpha, float *out) {
    if (!cd || !d_x || !d_bmap || !out) return fail(P9IDG_INVALID_ARGUMENT, "null argument");
    CK(cudaSetDevice(cd->device));
    return cd_abs_max(cd, d_x, d_bmap, lambda, alpha, out);
}

p9idg_status p9idg_cd_get_abs_max_diff(p9idg_cd *cd, const float *x, const float *bmap, float lambda, float alpha,
                                       float *out) {
    if (!cd || !x || !bmap || !out) return fail(P9IDG_INVALID_ARGUMENT, "null argument");
    CK(cudaSetDevice(cd->device));
    const size_t bytes = sizeof(float) * static_cast<size_t>(cd->n) * cd->n;
    CK(cd->x.ensure(bytes));
    CK(cd->g.ensure(bytes));
    CK(cudaMemcpyAsync(cd->x.p, x, bytes, cudaMemcpyHostToDevice, cd->stream));
    CK(cudaMemcpyAsync(cd->g.p, bmap, bytes, cudaMemcpyHostToDevice, cd->stream));
    return cd_abs_max(cd, cd->x.as<float>(), cd->g.as<float>(), lambda, alpha, out);
}

p9idg_status p9idg_cd_deconvolve_path(p9idg_cd *cd, float *x, float *bmap, float lambda_min, float lambda_factor,
                                      float alpha, int32_t max_path_iter, int32_t max_iter, float epsilon,
                                      p9idg_cd_result *res) {
    // FastSerialCD.DeconvolvePath (FastSerialCD.cs:49-74)
    if (!cd || !x || !bmap) return fail(P9IDG_INVALID_ARGUMENT, "null argument");
    CK(cudaSetDevice(cd->device));
    const auto t0 = std::chrono::steady_clock::now();
    const size_t bytes = sizeof(float) * static_cast<size_t>(cd->n) * cd->n;
    CK(cd->x.ensure(bytes));
    CK(cd->g.ensure(bytes));
    CK(cudaMemcpyAsync(cd->x.p, x, bytes, cudaMemcpyHostToDevice, cd->stream));
    CK(cudaMemcpyAsync(cd->g.p, bmap, bytes, cudaMemcpyHostToDevice, cd->stream));
    bool converged = false;
    int32_t total = 0;
    for (int32_t p = 0; p < max_path_iter; p++) {
        float mx = 0.0f;
        TRY(cd_abs_max(cd, cd->x.as<float>(), cd->g.as<float>(), 0.0f, 1.0f, &mx));
        const float lambda_max = 1 / alpha * mx;
        float lambda_cur = lambda_max / lambda_factor;
        lambda_cur = lambda_cur > lambda_min ? lambda_cur : lambda_min;
        p9idg_cd_result r{};
        TRY(cd_run(cd, cd->x.as<float>(), cd->g.as<float>(), lambda_cur, alpha, max_iter, epsilon, &r));
        converged = (lambda_min == lambda_cur) && r.converged;
        total += r.iterations;
        if (converged) break;
    }
    CK(cudaMemcpyAsync(x, cd->x.p, bytes, cudaMemcpyDeviceToHost, cd->stream));
    CK(cudaMemcpyAsync(bmap, cd->g.p, bytes, cudaMemcpyDeviceToHost, cd->stream));
    CK(cudaStreamSynchronize(cd->stream));
    if (res) {
        res->converged = converged;
        res->iterations = total;
        res->elapsed_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }
    return P9IDG_OK;
}

p9idg_status p9idg_cd_reset_lipschitz_map(p9idg_cd *cd, const float *psf, int32_t h, int32_t w) {
    // FastSerialCD.ResetLipschitzMap (FastSerialCD.cs:116-127); aMap over the patch (= total size)
    if (!cd || !psf || h <= 0 || w <= 0 || h != w) return fail(P9IDG_INVALID_ARGUMENT, "invalid argument");
    CK(cudaSetDevice(cd->device));
    // maxCut = GetMax(psf2) of the current map
    float max_cut = 0.0f;
    if (cd->ph != cd->pw) return fail(P9IDG_UNSUPPORTED, "non-square PSF^2");
    TRY(dev_max(cd->psf2.as<float>(), cd->ph, 0, cd->word.as<unsigned int>(), &max_cut, cd->stream));
    // psf2Local = CalcPSFSquared(psf); maxFull = GetMax(psf2Local)
    Buf local;
    CK(local.ensure(sizeof(float) * static_cast<size_t>(4) * h * w));
    CK(cd->psf_tmp.ensure(sizeof(float) * static_cast<size_t>(h) * w));
    CK(cudaMemcpyAsync(cd->psf_tmp.p, psf, sizeof(float) * static_cast<size_t>(h) * w, cudaMemcpyHostToDevice,
                       cd->stream));
    p9idg_status st = dev_psf_squared(cd->psf_tmp.as<float>(), h, w, local.as<float>(), cd->sq0, cd->sq1, cd->fft,
                                      cd->stream);
    float max_full = 0.0f;
    if (st == P9IDG_OK) st = dev_max(local.as<float>(), 2 * h, 0, cd->word.as<unsigned int>(), &max_full, cd->stream);
    local.release();
    if (st != P9IDG_OK) return st;
    cd->max_lipschitz = max_full;
    std::vector<double> scan;
    amap_scan(psf, h, w, scan);
    Buf d_scan;
    CK(d_scan.ensure(sizeof(double) * scan.size()));
    CK(cudaMemcpyAsync(d_scan.p, scan.data(), sizeof(double) * scan.size(), cudaMemcpyHostToDevice, cd->stream));
    amap_kernel<<<grid_for(static_cast<int64_t>(cd->n) * cd->n), 256, 0, cd->stream>>>(
        d_scan.as<double>(), h, w, cd->n, cd->n, 0, 0, cd->n, cd->n, cd->amap.as<float>());
    CK(cudaGetLastError());
    const float f = max_full / max_cut;
    scale_kernel<<<grid_for(static_cast<int64_t>(cd->ph) * cd->pw), 256, 0, cd->stream>>>(
        cd->psf2.as<float>(), static_cast<int64_t>(cd->ph) * cd->pw, f);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(cd->stream));
    d_scan.release();
    return P9IDG_OK;
}

void p9idg_cd_destroy(p9idg_cd *cd) {
    if (!cd) return;
    cudaSetDevice(cd->device);
    cd_release(cd);
    delete cd;
}

// ---- PaddedConvolver ----

p9idg_status p9idg_convolver_create(const double *kernel, int32_t h, int32_t w, int32_t kernel_h, int32_t kernel_w,
                                    p9idg_convolver **out) {
    if (!out) return fail(P9IDG_INVALID_ARGUMENT, "null output pointer");
    *out = nullptr;
    if (!kernel || h <= 0 || w <= 0 || kernel_h <= 0 || kernel_w <= 0)
        return fail(P9IDG_INVALID_ARGUMENT, "invalid argument");
    TRY(have_device());
    auto *c = new (std::nothrow) p9idg_convolver();
    if (!c) return fail(P9IDG_OUT_OF_MEMORY, "convolver allocation");
    p9idg_status st = conv_init(c, h, w, kernel_h, kernel_w);
    if (st == P9IDG_OK) {
        c->made.reset(new (std::nothrow) ConvSize());
        st = c->made ? conv_plans(c->made.get(), h, w) : fail(P9IDG_OUT_OF_MEMORY, "convolver allocation");
    }
    if (st == P9IDG_OK) {
        Buf full;
        const int64_t half = static_cast<int64_t>(h) * (w / 2 + 1);
        cudaError_t e = full.ensure(sizeof(double2) * static_cast<size_t>(h) * w);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(full.p, kernel, sizeof(double2) * static_cast<size_t>(h) * w, cudaMemcpyHostToDevice,
                                c->stream);
        if (e == cudaSuccess) {
            conv_kernel_half<<<grid_for(half), 256, 0, c->stream>>>(full.as<double2>(), h, w,
                                                                    conv_factor(c, c->made.get()),
                                                                    c->made->kernel.as<double2>());
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess) st = cuda_fail(e, "convolver kernel upload");
        c->n_max = std::max(h, w);
    }
    if (st != P9IDG_OK) {
        conv_release(c);
        delete c;
        return st;
    }
    *out = c;
    return P9IDG_OK;
}

p9idg_status p9idg_convolver_create_correlation(const float *psf, int32_t psf_h, int32_t psf_w, int32_t n,
                                                p9idg_convolver **out) {
    if (!out) return fail(P9IDG_INVALID_ARGUMENT, "null output pointer");
    *out = nullptr;
    if (!psf || psf_h <= 0 || psf_w <= 0 || n <= 0) return fail(P9IDG_INVALID_ARGUMENT, "invalid argument");
    if (n + psf_h != n + psf_w) return fail(P9IDG_INVALID_ARGUMENT, "padded PSF must be square");
    TRY(have_device());
    auto *c = new (std::nothrow) p9idg_convolver();
    if (!c) return fail(P9IDG_OUT_OF_MEMORY, "convolver allocation");
    p9idg_status st = conv_init(c, n + psf_h, n + psf_w, psf_h, psf_w);
    if (st == P9IDG_OK) {
        cudaError_t e = c->psf.ensure(sizeof(float) * static_cast<size_t>(psf_h) * psf_w);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(c->psf.p, psf, sizeof(float) * static_cast<size_t>(psf_h) * psf_w,
                                cudaMemcpyHostToDevice, c->stream);
        if (e != cudaSuccess) st = cuda_fail(e, "psf upload");
    }
    // (tiny images keep the padded size: there the shifted PSF can reach the last row, which
    // FFT.Shift leaves in place)
    const int m = n >= 8 ? smooth_size(n + psf_h) : n + psf_h;
    if (st == P9IDG_OK) st = conv_correlation(c, m, n, c->made);
    if (st == P9IDG_OK) {
        c->n_max = m == c->H ? c->H : n;
        cudaError_t e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess) st = cuda_fail(e, "correlation kernel");
    }
    if (st != P9IDG_OK) {
        conv_release(c);
        delete c;
        return st;
    }
    *out = c;
    return P9IDG_OK;
}

p9idg_status p9idg_convolver_convolve_device(p9idg_convolver *c, const float *d_image, int32_t n, float *d_out) {
    if (!c || !d_image || !d_out || n <= 0) return fail(P9IDG_INVALID_ARGUMENT, "invalid argument");
    CK(cudaSetDevice(c->device));
    return conv_run(c, d_image, n, d_out);
}

p9idg_status p9idg_convolver_convolve(p9idg_convolver *c, const float *image, int32_t n, float *out) {
    if (!c || !image || !out || n <= 0) return fail(P9IDG_INVALID_ARGUMENT, "invalid argument");
    CK(cudaSetDevice(c->device));
    const size_t bytes = sizeof(float) * static_cast<size_t>(n) * n;
    Buf in, res;
    CK(in.ensure(bytes));
    CK(res.ensure(bytes));
    CK(cudaMemcpyAsync(in.p, image, bytes, cudaMemcpyHostToDevice, c->stream));
    p9idg_status st = conv_run(c, in.as<float>(), n, res.as<float>());
    if (st == P9IDG_OK) {
        cudaError_t e = cudaMemcpyAsync(out, res.p, bytes, cudaMemcpyDeviceToHost, c->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess) st = cuda_fail(e, "convolve");
    }
    in.release();
    res.release();
    return st;
}

void p9idg_convolver_destroy(p9idg_convolver *c) {
    if (!c) return;
    cudaSetDevice(c->device);
    conv_release(c);
    delete c;
}

// ---- PSF helpers on host arrays ----

p9idg_status p9idg_psf_padded_fourier_correlation(const float *psf, int32_t h, int32_t w, int32_t pad_y,
                                                  int32_t pad_x, double *out) {
    if (!psf || !out || h <= 0 || w <= 0 || pad_y < 0 || pad_x < 0) return fail(P9IDG_INVALID_ARGUMENT, "invalid argument");
    TRY(have_device());
    const int H = pad_y + h, W = pad_x + w;
    if (H != W) return fail(P9IDG_INVALID_ARGUMENT, "padded PSF must be square (FFT.Shift uses the row count)");
    cudaStream_t st = nullptr;
    Buf d_psf, d_out;
    Z2Z fft;
    CK(d_psf.ensure(sizeof(float) * static_cast<size_t>(h) * w));
    CK(d_out.ensure(sizeof(double2) * static_cast<size_t>(H) * W));
    CK(cudaMemcpy(d_psf.p, psf, sizeof(float) * static_cast<size_t>(h) * w, cudaMemcpyHostToDevice));
    p9idg_status s = dev_padded_correlation(d_psf.as<float>(), h, w, pad_y, pad_x, d_out.as<double2>(), fft, st);
    if (s == P9IDG_OK) {
        cudaError_t e = cudaMemcpy(out, d_out.p, sizeof(double2) * static_cast<size_t>(H) * W, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) s = cuda_fail(e, "correlation");
    }
    fft.release();
    d_psf.release();
    d_out.release();
    return s;
}

p9idg_status p9idg_psf_squared(const float *psf, int32_t h, int32_t w, float *out) {
    if (!psf || !out || h <= 0 || w <= 0 || h != w) return fail(P9IDG_INVALID_ARGUMENT, "invalid argument");
    TRY(have_device());
    Buf d_psf, d_out, b0, b1;
    Z2Z fft;
    CK(d_psf.ensure(sizeof(float) * static_cast<size_t>(h) * w));
    CK(d_out.ensure(sizeof(float) * static_cast<size_t>(4) * h * w));
    CK(cudaMemcpy(d_psf.p, psf, sizeof(float) * static_cast<size_t>(h) * w, cudaMemcpyHostToDevice));
    p9idg_status s = dev_psf_squared(d_psf.as<float>(), h, w, d_out.as<float>(), b0, b1, fft, nullptr);
    if (s == P9IDG_OK) {
        cudaError_t e = cudaMemcpy(out, d_out.p, sizeof(float) * static_cast<size_t>(4) * h * w, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) s = cuda_fail(e, "psf squared");
    }
    fft.release();
    Buf *bufs[] = {&d_psf, &d_out, &b0, &b1};
    for (Buf *b : bufs) b->release();
    return s;
}

p9idg_status p9idg_psf_amap(const float *psf, int32_t h, int32_t w, int32_t total_h, int32_t total_w, float *out) {
    if (!psf || !out || h <= 0 || w <= 0 || total_h <= 0 || total_w <= 0)
        return fail(P9IDG_INVALID_ARGUMENT, "invalid argument");
    TRY(have_device());
    std::vector<double> scan;
    amap_scan(psf, h, w, scan);
    Buf d_scan, d_out;
    CK(d_scan.ensure(sizeof(double) * scan.size()));
    CK(d_out.ensure(sizeof(float) * static_cast<size_t>(total_h) * total_w));
    CK(cudaMemcpy(d_scan.p, scan.data(), sizeof(double) * scan.size(), cudaMemcpyHostToDevice));
    amap_kernel<<<grid_for(static_cast<int64_t>(total_h) * total_w), 256>>>(d_scan.as<double>(), h, w, total_h, total_w,
                                                                            0, 0, total_h, total_w, d_out.as<float>());
    CK(cudaGetLastError());
    CK(cudaMemcpy(out, d_out.p, sizeof(float) * static_cast<size_t>(total_h) * total_w, cudaMemcpyDeviceToHost));
    d_scan.release();
    d_out.release();
    return P9IDG_OK;
}

}  // extern "C"

// ------------------------------------------------------------------------------------------
// MajorCycle.ReconstructSerialCD on device buffers

namespace {

struct McState {
    Buf layers, resid, model_vis, xgrid, grad, psf_cut, word, partial, own_model, own_resid, own_psf;
    cufftHandle c2c = 0;
    ~McState() {
        Buf *bufs[] = {&layers, &resid, &model_vis, &xgrid, &grad, &psf_cut, &word, &partial, &own_model, &own_resid,
                       &own_psf};
        for (Buf *b : bufs) b->release();
        if (c2c) cufftDestroy(c2c);
    }
};

double elapsed_ms(cudaEvent_t a, cudaEvent_t b) {
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, a, b);
    return ms;
}

p9idg_status major_cycle(p9idg_plan *plan, const p9idg_mc_params *mp, const float2 *d_vis, const uint8_t *d_flags,
                         float *d_model, float *d_residual, float *d_psf, p9idg_mc_cycle *cycles, int32_t *ncycles) {
    p9idg_plan_info info{};
    TRY(p9idg_plan_get_info(plan, &info));
    p9idg_params c{};
    TRY(p9idg_plan_get_params(plan, &c));
    TRY(p9idg_plan_init_device(plan));
    void *sv = nullptr;
    TRY(p9idg_plan_get_stream(plan, &sv));
    cudaStream_t st = static_cast<cudaStream_t>(sv);
    const int N = c.grid_size;
    const int64_t nn = static_cast<int64_t>(N) * N;
    const int64_t nvis = static_cast<int64_t>(info.nbl) * info.nt * info.nch;
    if (mp->psf_cut_factor <= 0 || N / mp->psf_cut_factor <= 0)
        return fail(P9IDG_INVALID_ARGUMENT, "psf cut factor must leave a PSF");
    const int P = N / mp->psf_cut_factor;
    if (mp->max_major_cycles < 0) return fail(P9IDG_INVALID_ARGUMENT, "negative cycle count");
    McState s;
    CK(s.layers.ensure(sizeof(float2) * nn * c.wlayer_count));
    CK(s.resid.ensure(sizeof(float2) * std::max<int64_t>(1, nvis)));
    CK(s.model_vis.ensure(sizeof(float2) * std::max<int64_t>(1, nvis)));
    CK(s.xgrid.ensure(sizeof(float2) * nn));
    CK(s.grad.ensure(sizeof(float) * nn));
    CK(s.psf_cut.ensure(sizeof(float) * static_cast<size_t>(P) * P));
    CK(s.word.ensure(sizeof(unsigned int)));
    if (!d_psf) {
        CK(s.own_psf.ensure(sizeof(float) * nn));
        d_psf = s.own_psf.as<float>();
    }
    cudaEvent_t ev[5];
    for (auto &e : ev) CK(cudaEventCreate(&e));
    struct EvGuard {
        cudaEvent_t *e;
        ~EvGuard() {
            for (int i = 0; i < 5; i++) cudaEventDestroy(e[i]);
        }
    } evg{ev};

    // PSF: unit visibilities where unflagged, GridW, WStackIFFTFloat, Shift (MajorCycle.cs:35-48)
    CK(launch_unit_vis(d_flags, nvis, s.resid.as<float2>(), st));
    TRY(p9idg_grid_w_device(plan, s.resid.p, s.layers.p));
    TRY(p9idg_wstack_image_device(plan, s.layers.p, d_psf, 1));
    // psfCut, maxSidelobe (MajorCycle.cs:54-55)
    cut_kernel<<<grid_for(static_cast<int64_t>(P) * P), 256, 0, st>>>(d_psf, N, P, N / 2 - P / 2, s.psf_cut.as<float>());
    CK(cudaGetLastError());
    float max_sidelobe = 0.0f;
    TRY(dev_max(d_psf, N, mp->psf_cut_factor, s.word.as<unsigned int>(), &max_sidelobe, st));
    TRY(p9idg_synchronize(plan));
    std::vector<float> h_cut(static_cast<size_t>(P) * P);
    CK(cudaMemcpy(h_cut.data(), s.psf_cut.p, sizeof(float) * h_cut.size(), cudaMemcpyDeviceToHost));

    // deconvolver = new FastSerialCD(totalSize, psfCut); gCalculator (MajorCycle.cs:57-73)
    p9idg_cd *cd = nullptr;
    TRY(p9idg_cd_create(N, h_cut.data(), P, P, &cd));
    struct CdGuard {
        p9idg_cd *cd;
        ~CdGuard() { p9idg_cd_destroy(cd); }
    } cdg{cd};
    TRY(p9idg_cd_set_stream(cd, st));
    p9idg_convolver *conv = nullptr;
    TRY(p9idg_convolver_create_correlation(h_cut.data(), P, P, N, &conv));
    struct ConvGuard {
        p9idg_convolver *c;
        ~ConvGuard() { p9idg_convolver_destroy(c); }
    } convg{conv};
    conv->stream = st;

    // maxLipschitz = CalcMaxLipschitz(psfCut): float squares summed in double in the reference's order
    double max_lipschitz = 0.0;
    for (float v : h_cut) {
        const float q = v * v;
        max_lipschitz += q;
    }
    const float lambda_lipschitz = static_cast<float>(mp->lambda * max_lipschitz);
    double lip_full = 0.0;
    TRY(dev_sumsq(d_psf, nn, s.partial, &lip_full, st));
    const float lambda_true = static_cast<float>(mp->lambda * lip_full);
    float lambda = mp->lambda;
    bool switched = false;

    CK(cudaMemsetAsync(d_model, 0, sizeof(float) * nn, st));
    const float2 *resid_src = d_vis;  // residualVis = data.Visibilities
    cufftHandle &c2c = s.c2c;
    CUFFT(cufftPlan2d(&c2c, N, N, CUFFT_C2C));
    CUFFT(cufftSetStream(c2c, st));
    *ncycles = 0;
    for (int cycle = 0; cycle < mp->max_major_cycles; cycle++) {
        p9idg_mc_cycle rec{};
        CK(cudaEventRecord(ev[0], st));
        TRY(p9idg_grid_w_device(plan, resid_src, s.layers.p));
        CK(cudaEventRecord(ev[1], st));
        TRY(p9idg_wstack_image_device(plan, s.layers.p, d_residual, 1));
        TRY(p9idg_synchronize(plan));
        float max_dirty = 0.0f, max_b = 0.0f;
        TRY(dev_max(d_residual, N, 0, s.word.as<unsigned int>(), &max_dirty, st));
        TRY(conv_run(conv, d_residual, N, s.grad.as<float>()));
        TRY(dev_max(s.grad.as<float>(), N, 0, s.word.as<unsigned int>(), &max_b, st));
        CK(cudaEventRecord(ev[2], st));
        // MajorCycle.cs:98-100 in the reference's types
        const double cf = static_cast<double>(max_b) / (static_cast<double>(max_dirty) * max_lipschitz);
        const double correction = cf > 1.0 ? cf : (std::isnan(cf) ? cf : 1.0);
        const double side = static_cast<double>(max_b * max_sidelobe) * correction;
        const double l1 = side / mp->alpha, l2 = lambda_lipschitz;
        const double lm = (l1 != l2) ? (!std::isnan(l1) ? (l2 < l1 ? l1 : l2) : l1) : (std::signbit(l2) ? l1 : l2);
        const float current_lambda = static_cast<float>(lm);
        float abs_max = 0.0f;
        TRY(p9idg_cd_get_abs_max_diff_device(cd, d_model, s.grad.as<float>(), lambda_true, mp->alpha, &abs_max));
        TRY(dev_objective(d_residual, d_model, nn, lambda_true, mp->alpha, s.partial, &rec.objective, st));
        rec.max_dirty = max_dirty;
        rec.max_b = max_b;
        rec.current_lambda = current_lambda;
        rec.abs_max = abs_max;
        if (abs_max >= mp->major_epsilon) {
            p9idg_cd_result r{};
            TRY(p9idg_cd_deconvolve_device(cd, d_model, s.grad.as<float>(), current_lambda, mp->alpha,
                                           mp->deconv_iterations, mp->deconv_epsilon, &r));
            rec.deconvolved = 1;
            rec.converged = r.converged;
            rec.iterations = r.iterations;
        }
        CK(cudaEventRecord(ev[3], st));
        if (lambda == current_lambda && !switched) {  // MajorCycle.cs:109-115
            lambda = lambda_true;
            max_lipschitz = lip_full;
            switched = true;
        }
        const bool stop = abs_max < mp->major_epsilon;
        if (!stop) {
            shifted_real_to_c64_kernel<<<grid_for(nn), 256, 0, st>>>(d_model, N, s.xgrid.as<float2>());
            CK(cudaGetLastError());
            CUFFT(cufftExecC2C(c2c, s.xgrid.as<cufftComplex>(), s.xgrid.as<cufftComplex>(), CUFFT_FORWARD));
            TRY(p9idg_degrid_w_device(plan, s.xgrid.p, s.model_vis.p));
            vis_subtract_kernel<<<grid_for(nvis), 256, 0, st>>>(d_vis, s.model_vis.as<float2>(), d_flags, nvis,
                                                                 s.resid.as<float2>());
            CK(cudaGetLastError());
            resid_src = s.resid.as<float2>();
        }
        CK(cudaEventRecord(ev[4], st));
        TRY(p9idg_synchronize(plan));
        rec.grid_ms = elapsed_ms(ev[0], ev[1]);
        rec.image_ms = elapsed_ms(ev[1], ev[2]);
        rec.deconv_ms = elapsed_ms(ev[2], ev[3]);
        rec.degrid_ms = elapsed_ms(ev[3], ev[4]);
        if (cycles) cycles[cycle] = rec;
        *ncycles = cycle + 1;
        if (stop) break;
    }
    return P9IDG_OK;
}

}  // namespace

extern "C" {

p9idg_status p9idg_major_cycle_serial_cd_device(p9idg_plan *plan, const p9idg_mc_params *params, const void *d_vis,
                                                const uint8_t *d_flags, float *d_model, float *d_residual,
                                                float *d_psf, p9idg_mc_cycle *cycles, int32_t *ncycles) {
    if (!plan || !params || !d_vis || !d_flags || !d_model || !d_residual || !ncycles)
        return fail(P9IDG_INVALID_ARGUMENT, "null argument");
    return major_cycle(plan, params, static_cast<const float2 *>(d_vis), d_flags, d_model, d_residual, d_psf, cycles,
                       ncycles);
}

p9idg_status p9idg_major_cycle_serial_cd(p9idg_plan *plan, const p9idg_mc_params *params, const double *vis,
                                         const uint8_t *flags, float *model_out, float *residual_out, float *psf_out,
                                         p9idg_mc_cycle *cycles, int32_t *ncycles) {
    if (!plan || !params || !vis || !flags || !model_out || !residual_out || !ncycles)
        return fail(P9IDG_INVALID_ARGUMENT, "null argument");
    TRY(have_device());
    p9idg_plan_info info{};
    TRY(p9idg_plan_get_info(plan, &info));
    p9idg_params c{};
    TRY(p9idg_plan_get_params(plan, &c));
    TRY(p9idg_plan_init_device(plan));
    const int64_t nvis = static_cast<int64_t>(info.nbl) * info.nt * info.nch;
    const int64_t nn = static_cast<int64_t>(c.grid_size) * c.grid_size;
    Buf v128, v64, fl, model, resid, psf;
    CK(v128.ensure(sizeof(double2) * std::max<int64_t>(1, nvis)));
    CK(v64.ensure(sizeof(float2) * std::max<int64_t>(1, nvis)));
    CK(fl.ensure(std::max<int64_t>(1, nvis)));
    CK(model.ensure(sizeof(float) * nn));
    CK(resid.ensure(sizeof(float) * nn));
    CK(psf.ensure(sizeof(float) * nn));
    void *sv = nullptr;
    TRY(p9idg_plan_get_stream(plan, &sv));
    cudaStream_t st = static_cast<cudaStream_t>(sv);
    CK(cudaMemcpyAsync(v128.p, vis, sizeof(double2) * nvis, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(fl.p, flags, nvis, cudaMemcpyHostToDevice, st));
    CK(launch_c128_to_c64(v128.as<double2>(), nvis, v64.as<float2>(), st));
    CK(cudaStreamSynchronize(st));
    v128.release();
    TRY(major_cycle(plan, params, v64.as<float2>(), fl.as<uint8_t>(), model.as<float>(), resid.as<float>(),
                    psf.as<float>(), cycles, ncycles));
    CK(cudaMemcpy(model_out, model.p, sizeof(float) * nn, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(residual_out, resid.p, sizeof(float) * nn, cudaMemcpyDeviceToHost));
    if (psf_out) CK(cudaMemcpy(psf_out, psf.p, sizeof(float) * nn, cudaMemcpyDeviceToHost));
    Buf *bufs[] = {&v64, &fl, &model, &resid, &psf};
    for (Buf *b : bufs) b->release();
    return P9IDG_OK;
}

}  // extern "C"
