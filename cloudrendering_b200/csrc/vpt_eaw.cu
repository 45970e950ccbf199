// vpt_eaw.cu - the EAW a-trous passes (Data/Shaders/Denoiser/EAWDenoise.glsl): 5x5 taps at step 2^i
// with Gaussian weights exp(-(x^2+y^2)/2), colour / position / normal edge stops
// min(exp(-|d|^2/phi), 1), taps outside the image clamped to the edge.  A unit of its own so that its
// multiply-adds are contracted (the other denoiser kernels are compiled without contraction): the
// passes are bound by instruction issue and shared-memory reads.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <algorithm>
#include <mutex>
#include "vpt_denoise.h"
#include "vpt_kernels.h"

namespace vpt {

constexpr int kMaxEawDevices = 64;
__constant__ float c_eaw_kernel[25];

__device__ __forceinline__ float dot4(float4 a, float4 b) {
    return ((a.x * b.x + a.y * b.y) + a.z * b.z) + a.w * b.w;
}
__device__ __forceinline__ float4 sub4(float4 a, float4 b) {
    return make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w);
}

// Edge-stopping weight min(exp(-|d|^2 / phi), 1) with the special-function unit's exponential and
// the reciprocal of phi computed once (a few ulp from the IEEE form; the filter is a normalised
// weighted mean, so its output moves by about as much).
__device__ __forceinline__ float eaw_stop(float4 d, float inv_phi) {
    return fminf(__expf(-dot4(d, d) * inv_phi), 1.0f);
}

// Packed pairs of fp32 (one 64-bit register pair): one instruction for two lanes.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float exp2_sfu(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void copy16(float4* dst, const float4* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
constexpr float kLog2e = 1.4426950408889634f;

struct EawPass {
    const float* color;
    const float* pos;  // nullptr: no position stop
    const float* nrm;  // nullptr: no normal stop
    float* out;
    int w, h, step, tiles_x, tiles_y;
    float phi_c, phi_p, phi_n;
    int use_c, quirk;
};

// A pixel's weighted sum.  A tap's weight is one exponential of its summed distances,
// 2^(log2 k - sum |d|^2 log2(e) / phi), in packed fp32 pairs: about 20 instructions a tap where three
// separate edge stops took about 45.  With phi >= 0 every stop min(exp(-|d|^2 / phi), 1) is the
// exponential itself except for a NaN distance (inf - inf, or 0 / 0), where it is 1: a NaN weight shows in
// the weight sum, and eaw_stops filters such a pixel again.
template <bool POS, bool NRM>
struct EawPixel {
    f32x2 nc[2], np[2], nn[2], s0, s1;  // the negated centre, the sums
    float acc;

    __device__ __forceinline__ void begin(float4 c, float4 p, float4 n) {
        nc[0] = pack2(-c.x, -c.y);
        nc[1] = pack2(-c.z, -c.w);
        if (POS) {
            np[0] = pack2(-p.x, -p.y);
            np[1] = pack2(-p.z, -p.w);
        }
        if (NRM) {
            nn[0] = pack2(-n.x, -n.y);
            nn[1] = pack2(-n.z, -n.w);
        }
        s0 = s1 = 0ull;
        acc = 0.0f;
    }
    // d2: squared distance of the tap on the 5 x 5 kernel; bias: log2 of a constant factor
    __device__ __forceinline__ void tap(int d2, float bias, ulonglong2 c, ulonglong2 p, ulonglong2 n, f32x2 lc,
                                        f32x2 lp, f32x2 ln) {
        f32x2 t = pack2(fmaf(-0.5f * kLog2e, (float)d2, bias), 0.0f);  // log2 of exp(-d2 / 2)
        f32x2 d = add2(c.x, nc[0]), e = add2(c.y, nc[1]);
        t = fma2(fma2(e, e, mul2(d, d)), lc, t);
        if (POS) {
            d = add2(p.x, np[0]);
            e = add2(p.y, np[1]);
            t = fma2(fma2(e, e, mul2(d, d)), lp, t);
        }
        if (NRM) {
            d = add2(n.x, nn[0]);
            e = add2(n.y, nn[1]);
            t = fma2(fma2(e, e, mul2(d, d)), ln, t);
        }
        float lo, hi;
        unpack2(t, lo, hi);
        const float wk = exp2_sfu(lo + hi);
        const f32x2 wk2 = pack2(wk, wk);
        s0 = fma2(c.x, wk2, s0);
        s1 = fma2(c.y, wk2, s1);
        acc += wk;
    }
    __device__ __forceinline__ bool valid() const { return acc == acc; }
    __device__ __forceinline__ float4 result() const {
        const float ia = 1.0f / acc;
        float4 o;
        unpack2(s0, o.x, o.y);
        unpack2(s1, o.z, o.w);
        return make_float4(o.x * ia, o.y * ia, o.z * ia, o.w * ia);
    }
};

// exponents' scales -log2(e) / phi.  The quirk's constant colour weight min(exp(-1 / phi_c), 1) is the same for every
// tap: it cancels in the quotient of the sums and is left out (as a factor it would take the weights out of the
// normal range for a small phi_c), except where it is 0, which leaves 0 / 0.
__device__ __forceinline__ f32x2 eaw_scale(float phi) {
    const float s = -kLog2e / phi;
    return pack2(s, s);
}
__device__ __forceinline__ f32x2 eaw_color_scale(const EawPass& a) {
    return a.use_c && !a.quirk ? eaw_scale(a.phi_c) : 0ull;
}
__device__ __forceinline__ float eaw_bias(const EawPass& a) {
    return a.use_c && a.quirk && expf(-1.0f / a.phi_c) == 0.0f ? -INFINITY : 0.0f;
}

// One pixel with the separate stops, its 25 taps taken from `taps` (fetch(i) gives the three maps).
template <class T>
__device__ __forceinline__ float4 eaw_stops(const EawPass& a, const T& taps) {
    float4 cc, cp, cn, oc, op, on;
    taps.fetch(12, cc, cp, cn);
    float4 sum = make_float4(0, 0, 0, 0);
    float acc = 0.0f;
    const float quirk_wc = fminf(expf(-1.0f / a.phi_c), 1.0f);
    const float inv_c = 1.0f / a.phi_c, inv_p = 1.0f / a.phi_p, inv_n = 1.0f / a.phi_n;
#pragma unroll 1
    for (int i = 0; i < 25; i++) {
        taps.fetch(i, oc, op, on);
        float weight = 1.0f;
        if (a.use_c) weight *= a.quirk ? quirk_wc : eaw_stop(sub4(cc, oc), inv_c);
        if (a.pos) weight *= eaw_stop(sub4(cp, op), inv_p);
        if (a.nrm) weight *= eaw_stop(sub4(cn, on), inv_n);
        const float wk = weight * c_eaw_kernel[i];
        sum.x += oc.x * wk;
        sum.y += oc.y * wk;
        sum.z += oc.z * wk;
        sum.w += oc.w * wk;
        acc += wk;
    }
    const float ia = 1.0f / acc;
    return make_float4(sum.x * ia, sum.y * ia, sum.z * ia, sum.w * ia);
}

struct GlobalTaps {
    const EawPass& a;
    int x, y;
    __device__ __forceinline__ size_t at(int i) const {
        const int sx = min(max(x + (i % 5 - 2) * a.step, 0), a.w - 1);
        const int sy = min(max(y + (i / 5 - 2) * a.step, 0), a.h - 1);
        return (size_t)sy * a.w + sx;
    }
    __device__ __forceinline__ void fetch(int i, float4& c, float4& p, float4& n) const {
        const size_t q = at(i);
        c = __ldg(reinterpret_cast<const float4*>(a.color) + q);
        p = a.pos ? __ldg(reinterpret_cast<const float4*>(a.pos) + q) : make_float4(0, 0, 0, 0);
        n = a.nrm ? __ldg(reinterpret_cast<const float4*>(a.nrm) + q) : make_float4(0, 0, 0, 0);
    }
};

// Every tap read from global memory, one thread a pixel: for images so small, or steps so large, that a
// lattice tile would be mostly empty, and (packed = 0) for negative phi, whose stops exceed 1 before the
// clamp.
template <bool POS, bool NRM>
__global__ void eaw_iteration_kernel(const __grid_constant__ EawPass a, int packed) {
    // blocks of 32 x 4 pixels, counted along x row by row, so that any height fits the grid
    const int blocks_x = (a.w + 31) / 32, by = (int)blockIdx.x / blocks_x;
    const int x = ((int)blockIdx.x - by * blocks_x) * 32 + (int)threadIdx.x;
    const int y = by * 4 + (int)threadIdx.y;
    if (x >= a.w || y >= a.h) return;
    const GlobalTaps taps{a, x, y};
    float4 o;
    bool done = false;
    if (packed) {
        const f32x2 lc = eaw_color_scale(a), lp = eaw_scale(a.phi_p), ln = eaw_scale(a.phi_n);
        const float bias = eaw_bias(a);
        float4 c, p, n;
        taps.fetch(12, c, p, n);
        EawPixel<POS, NRM> px;
        px.begin(c, p, n);
#pragma unroll
        for (int i = 0; i < 25; i++) {
            const int ox = i % 5 - 2, oy = i / 5 - 2;
            const size_t q = taps.at(i);
            const ulonglong2 tc = __ldg(reinterpret_cast<const ulonglong2*>(a.color) + q);
            ulonglong2 tp = tc, tn = tc;
            if (POS) tp = __ldg(reinterpret_cast<const ulonglong2*>(a.pos) + q);
            if (NRM) tn = __ldg(reinterpret_cast<const ulonglong2*>(a.nrm) + q);
            px.tap(ox * ox + oy * oy, bias, tc, tp, tn, lc, lp, ln);
        }
        done = px.valid();
        o = px.result();
    }
    if (!done) o = eaw_stops(a, taps);
    reinterpret_cast<float4*>(a.out)[(size_t)y * a.w + x] = o;
}

// The same iteration with the taps staged in shared memory.  The 25 taps of pixel (x, y) at step s lie
// on the lattice (x + i s, y + j s), so a block takes pixels of one residue class modulo s (at s = 1
// all pixels; at s >= 2 two horizontally adjacent classes, whose pixel pairs fill the 32-byte sectors
// that a single class would read half of): 32 x 16 of them, whose taps all fall on a 36 x 20 (40 x 20)
// patch of that lattice, loaded once.  Lattice points beyond the image are clamped to the edge pixel,
// as the taps are.  Same arithmetic, tap for tap, as eaw_iteration_kernel.
//
// The pass is bound by the multiply-add pipe and shared-memory reads, not by HBM.  So each thread filters
// kEawRowsOf vertically adjacent lattice pixels: the 5 columns of that many rows + 4 are read once and
// serve all of them (with both maps 45 instead of 75 16-byte reads a pixel).
// Measured, 1920 x 1080 with both maps, five passes: 688 us with one pixel a thread and loads through registers
// (shared-memory reads and the wait for the patch), 458 us so (the multiply-add pipe's time alone is about 250).
// Both maps with 4 rows a thread: 485 to 550 us; without maps 239 us with 4 rows, 265 with 2 (was 395).
constexpr int kEawTileW = 32;              // pixels of a block's row (two classes of 16 at step >= 2)
constexpr int kEawTileH = 16;              // lattice rows of a block
constexpr int kEawPatchH = kEawTileH + 4;
constexpr int kEawPatchW = kEawTileW + 8;  // 36 used at step 1
// rows a thread: 4, and 2 with both maps (whose 4 centres and sums would leave 12 warps an SM)
template <bool POS, bool NRM>
constexpr int kEawRowsOf = POS && NRM ? 2 : 4;

struct SharedTaps {
    const float4 *c, *p, *n;  // the maps' patches at the pixel; p / n null without that map
    int classes;
    __device__ __forceinline__ void fetch(int i, float4& oc, float4& op, float4& on) const {
        const int q = (i / 5 - 2) * kEawPatchW + (i % 5 - 2) * classes;
        oc = c[q];
        op = p ? p[q] : make_float4(0, 0, 0, 0);
        on = n ? n[q] : make_float4(0, 0, 0, 0);
    }
};

template <bool POS, bool NRM>
__global__ void __launch_bounds__(kEawTileW* kEawTileH / kEawRowsOf<POS, NRM>, POS&& NRM ? 3 : 4)
    eaw_lattice_kernel(const __grid_constant__ EawPass a) {
    constexpr int kEawRows = kEawRowsOf<POS, NRM>, kEawThreads = kEawTileW * kEawTileH / kEawRows;
    extern __shared__ float4 eaw_sm[];
    float4* sc = eaw_sm;
    float4* sp = sc + kEawPatchW * kEawPatchH;
    float4* sn = sp + (POS ? kEawPatchW * kEawPatchH : 0);
    // block -> (tile tx, ty; residue pair rx, residue ry)
    const int classes = a.step > 1 ? 2 : 1;
    const int cols = kEawTileW / classes;  // lattice columns of a class in the tile
    int b = blockIdx.x;
    const int tx = b % a.tiles_x;
    b /= a.tiles_x;
    const int ty = b % a.tiles_y;
    b /= a.tiles_y;
    const int pairs = (min(a.step, a.w) + classes - 1) / classes;
    const int rx = (b % pairs) * classes, ry = b / pairs;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int patch_w = (cols + 4) * classes;
    // asynchronous copies: the whole patch is in flight before the wait (loads through registers left the
    // block waiting for one patch row after the other)
    for (int k = threadIdx.x; k < patch_w * kEawPatchH; k += kEawThreads) {
        const int c = k / patch_w, i = k - c * patch_w;
        const int col = classes == 2 ? i >> 1 : i, cls = classes == 2 ? i & 1 : 0;
        const int py = min(max((ty * kEawTileH + c - 2) * a.step + ry, 0), a.h - 1);
        const int px = min(max((tx * cols + col - 2) * a.step + rx + cls, 0), a.w - 1);
        const size_t o = (size_t)py * a.w + px;
        const int q = c * kEawPatchW + i;
        copy16(sc + q, reinterpret_cast<const float4*>(a.color) + o);
        if (POS) copy16(sp + q, reinterpret_cast<const float4*>(a.pos) + o);
        if (NRM) copy16(sn + q, reinterpret_cast<const float4*>(a.nrm) + o);
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    const int x = (tx * cols + lane / classes) * a.step + rx + lane % classes;
    const int row0 = warp * kEawRows;  // the thread's first lattice row in the tile
    const int y0 = (ty * kEawTileH + row0) * a.step + ry;
    if (x >= a.w || y0 >= a.h) return;
    const int cx = lane + 2 * classes;

    const f32x2 lc = eaw_color_scale(a), lp = eaw_scale(a.phi_p), ln = eaw_scale(a.phi_n);
    const float bias = eaw_bias(a);
    EawPixel<POS, NRM> px[kEawRows];
#pragma unroll
    for (int r = 0; r < kEawRows; r++) {
        const int q = (row0 + r + 2) * kEawPatchW + cx;
        px[r].begin(sc[q], POS ? sp[q] : sc[q], NRM ? sn[q] : sc[q]);
    }
#pragma unroll
    for (int j = 0; j < kEawRows + 4; j++) {  // patch rows of the taps
#pragma unroll
        for (int ox = -2; ox <= 2; ox++) {
            const int q = (row0 + j) * kEawPatchW + cx + ox * classes;
            const ulonglong2 tc = *reinterpret_cast<const ulonglong2*>(sc + q);
            ulonglong2 tp = tc, tn = tc;
            if (POS) tp = *reinterpret_cast<const ulonglong2*>(sp + q);
            if (NRM) tn = *reinterpret_cast<const ulonglong2*>(sn + q);
#pragma unroll
            for (int r = 0; r < kEawRows; r++) {
                const int oy = j - 2 - r;
                if (oy >= -2 && oy <= 2) px[r].tap(ox * ox + oy * oy, bias, tc, tp, tn, lc, lp, ln);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < kEawRows; r++) {
        const int y = y0 + r * a.step;
        if (y >= a.h) break;
        float4 o = px[r].result();
        if (!px[r].valid()) {
            const int q = (row0 + r + 2) * kEawPatchW + cx;
            o = eaw_stops(a, SharedTaps{sc + q, POS ? sp + q : nullptr, NRM ? sn + q : nullptr, classes});
        }
        reinterpret_cast<float4*>(a.out)[(size_t)y * a.w + x] = o;
    }
}

template <bool POS, bool NRM>
static cudaError_t launch_pass(EawPass a, bool lattice, bool packed, cudaStream_t s) {
    // per residue class: ceil(w / step) x ceil(h / step) pixels, two classes side by side at step >= 2
    const int classes = a.step > 1 ? 2 : 1, cols = kEawTileW / classes;
    a.tiles_x = ((a.w + a.step - 1) / a.step + cols - 1) / cols;
    a.tiles_y = ((a.h + a.step - 1) / a.step + kEawTileH - 1) / kEawTileH;
    const long long blocks =
        (long long)a.tiles_x * a.tiles_y * ((std::min(a.step, a.w) + classes - 1) / classes) * std::min(a.step, a.h);
    // tiles at least a quarter full: below that most lanes and copies of a block would be for nothing.  The direct
    // pass costs about four times a full tile's pixel (25 x 3 reads a pixel through L1).
    if (lattice && packed && blocks * kEawTileW * kEawTileH <= 4LL * a.w * a.h) {
        constexpr int smem = (1 + POS + NRM) * kEawPatchW * kEawPatchH * (int)sizeof(float4);
        eaw_lattice_kernel<POS, NRM><<<(unsigned)blocks, kEawTileW * kEawTileH / kEawRowsOf<POS, NRM>, smem, s>>>(a);
    } else {
        const unsigned g = (unsigned)((a.w + 31) / 32) * (unsigned)((a.h + 3) / 4);
        eaw_iteration_kernel<POS, NRM><<<g, dim3(32, 4), 0, s>>>(a, packed);
    }
    count_launches(1);
    return cudaGetLastError();
}

// The 25 Gaussian tap weights live in constant memory, which is per device: upload once per device.
static cudaError_t upload_eaw_kernel(cudaStream_t s) {
    static std::mutex mu;
    static bool done[kMaxEawDevices] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxEawDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu);
    if (done[dev]) return cudaSuccess;
    float k[25];
    for (int i = 0; i < 25; i++) {
        int x = i % 5 - 2, y = i / 5 - 2;
        k[i] = expf(-float(x * x + y * y) / 2.0f);
    }
    e = cudaMemcpyToSymbolAsync(c_eaw_kernel, k, sizeof(k), 0, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) done[dev] = true;
    return e;
}

cudaError_t eaw_denoise(const float* color, const float* pos, const float* nrm, int w, int h, const EawSettings& s,
                        float* ping, float* pong, float** result, cudaStream_t stream) {
    cudaError_t e = upload_eaw_kernel(stream);
    if (e != cudaSuccess) return e;
    EawPass a;
    a.pos = s.use_position ? pos : nullptr;
    a.nrm = s.use_normal ? nrm : nullptr;
    a.w = w;
    a.h = h;
    a.phi_c = s.phi_color;
    a.phi_p = s.phi_position;
    a.phi_n = s.phi_normal;
    a.use_c = s.use_color;
    a.quirk = s.ref_compute_quirk;
    // the stops in use have phi >= 0
    const bool packed = (!a.use_c || s.phi_color >= 0.0f) && (!a.pos || s.phi_position >= 0.0f) &&
                        (!a.nrm || s.phi_normal >= 0.0f);
    const bool lattice = s.lattice_tiles != 0;
    // steps of 65,536 pixels and more are refused with lattice tiles
    if (lattice && s.iterations > 16) return cudaErrorInvalidValue;
    const float* src = color;
    float* bufs[2] = {ping, pong};
    a.step = 1;
    for (int i = 0; i < s.iterations; i++) {
        a.color = src;
        a.out = bufs[i & 1];
        e = a.pos ? (a.nrm ? launch_pass<true, true>(a, lattice, packed, stream)
                           : launch_pass<true, false>(a, lattice, packed, stream))
                  : (a.nrm ? launch_pass<false, true>(a, lattice, packed, stream)
                           : launch_pass<false, false>(a, lattice, packed, stream));
        if (e != cudaSuccess) return e;
        src = a.out;
        a.step = std::min(a.step * 2, 1 << 28);  // (taps that far are at the edge: the same image at any larger step)
    }
    *result = const_cast<float*>(src);
    return cudaGetLastError();
}

}  // namespace vpt
