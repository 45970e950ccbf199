// vpt_unet.cu - the learned denoiser's network kernels: a U-Net of 3x3 convolutions that predicts
// per-pixel 5x5 kernels (a kernel-predicting denoiser), trained on the GPU by these kernels.
//
// The reference runs its learned denoiser through libtorch (src/Denoiser/PyTorchDenoiser.cpp:637-800,
// a TorchScript forward).  It has no training code and no network of its own; this file is new.
//
// Tensors are NHWC bf16 ("pixels x channels", P = N*H*W rows, channels contiguous, every channel
// count a multiple of 16); accumulation is fp32.  A 3x3 convolution (stride 1, zero padding 1) is an
// implicit GEMM with K = 9 * Cin, k = tap * Cin + ci, tap = (dy + 1) * 3 + (dx + 1):
//
//   forward       y[p][co]  = act(bias[co] + sum_k x[p + off(tap)][ci] * w[co][k])       M = pixels
//   input grad    dx[p][ci] = sum_k' dy[p + off(tap')][co] * wrot[ci][k'],  wrot[ci][t'][co]
//                 = w[co][8 - t'][ci] (the same kernel, rotated weights)                   M = pixels
//   weight grad   dw[co][k] = sum_p dy[p][co] * x[p + off(tap)][ci]                      M = k, K = pixels
//
// Tensor-core path (sm_100a tcgen05): one CTA computes a 128 x N tile (N <= 256 output channels) of
// D = A * B^T with the fp32 accumulator in tensor memory (TMEM).  All 128 threads gather the A / B
// tiles of the next K-stages with 16-byte cp.async copies (zero-filled outside the image) into a
// 4-stage shared-memory ring laid out in the UMMA no-swizzle canonical form (8-row x 16-byte core
// matrices); one thread issues tcgen05.mma (kind::f16, bf16 x bf16 -> fp32) per 16-wide K step and
// tcgen05.commit signals a per-stage mbarrier when the stage's MMAs have read their operands, which
// frees the slot for the next gather.  The epilogue reads the accumulator with tcgen05.ld (each warp
// its 32 TMEM lanes = 32 tile rows) and fuses bias, ReLU, the ReLU-derivative mask of the backward
// pass and the bf16 / fp32 store.  Forward and input-gradient tiles have K-major operands (k
// contiguous: channels of one pixel); the weight-gradient tile has MN-major operands (channels
// contiguous, pixels along K) and writes per-split fp32 partial sums that the optimiser reduces in a
// fixed order (deterministic).  That is conv_tile_kernel, which takes any shape; most layers go through the kernels
// further down whose operands the tensor-memory-access unit loads: boxes of 128 pixels (conv_box_kernel), row
// strips (conv_stack_kernel, conv_ws_kernel) and the weight gradient on image rows (wgrad_rows_kernel).
//
// Every mbarrier wait is bounded: on expiry the kernel records VPT_ERR_ITER_LIMIT in *err, waits
// (bounded) for the MMAs it issued, frees its TMEM and returns.
#include <cuda.h>  // CUtensorMap (encoded through the runtime's driver entry point)
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>
#include <atomic>
#include <type_traits>
#include "../../include/vpt_b200.h"
#include "vpt_kernels.h"
#include "vpt_scratch.h"

namespace vpt {
namespace unet {

typedef __nv_bfloat16 bf16;

constexpr int kBM = 128;      // tile rows (TMEM lanes)
constexpr int kBK = 64;       // K elements per pipeline stage (4 MMAs of K = 16)
constexpr int kThreads = 128;
constexpr uint32_t kWaitLimit = 1u << 22;  // bounded mbarrier waits (error flag on expiry)

// ---------------------------------------------------------------------------------------------
// PTX helpers
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    const int n = valid ? 16 : 0;  // n = 0 writes 16 zero bytes and reads nothing
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async16_stream(uint32_t dst, const void* src) {  // L2 only
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, bool valid) {
    const int n = valid ? 4 : 0;  // n = 0 writes 4 zero bytes and reads nothing
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
// make this thread's generic-proxy shared-memory writes visible to the tensor core (async proxy)
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
// waits until the phase with the given parity has completed; false after kWaitLimit polls
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kWaitLimit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// whole warp: allocate `cols` TMEM columns (power of two >= 32), address written to shared memory
__device__ __forceinline__ void tmem_alloc(uint32_t dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(dst), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(cols) : "memory");
}

// Shared-memory matrix descriptor, no swizzle: start address, leading-dimension byte offset (between
// core matrices adjacent along K), stride-dimension byte offset (between core matrices adjacent
// along M/N), all in 16-byte units; bits 46-47 = 1 (descriptor version of sm_100).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}
// Instruction descriptor of kind::f16: D fp32 (bits 4-5 = 1), A and B bf16 (bits 7-9, 10-12 = 1),
// A / B major (bit 15 / 16: 0 = K-major, 1 = MN-major), N >> 3 (bits 17-22), M >> 4 (bits 24-28).
__host__ __device__ constexpr uint32_t instr_desc(int m, int n, int a_mn, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
            tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}
// true in one lane of a converged warp.  The issuing warps run their loops with all lanes and enter the MMA
// sequences through this: inside `if (lane == 0)` the compiler could not prove the operands warp-uniform and
// moved every descriptor word to the uniform registers separately, about 250 cycles an MMA.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n.reg .pred P;\nelect.sync _|P, 0xffffffff;\nselp.u32 %0, 1, 0, P;\n}\n" : "=r"(p));
    return p != 0;
}

// tcgen05.mma from descriptor halves.  No memory clobber: the MMA reads shared memory asynchronously
// and is ordered by the mbarrier waits, tcgen05 fences and commits around it (which carry clobbers);
// without one the issuing loop keeps its loop-invariant values in registers.
__device__ __forceinline__ void mma_bf16_halves(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo,
                                                uint32_t b_hi, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\n.reg .b64 da, db;\nmov.b64 da, {%1, %2};\nmov.b64 db, {%3, %4};\n"
        "setp.ne.b32 p, %6, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n}\n" ::"r"(tmem_d),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
                 : "memory");
}
// 32 lanes x 16 consecutive 32-bit columns: lane i of the warp gets TMEM lane (base + i)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 32 lanes x 16 columns of zeros (the caller waits with tcgen05.wait::st)
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};\n" ::"r"(taddr),
        "r"(0)
        : "memory");
}

// ---------------------------------------------------------------------------------------------
// the implicit-GEMM convolution tile
// ---------------------------------------------------------------------------------------------
enum Mode : int { kConv = 0, kWgrad = 1 };

struct ConvArgs {
    const bf16* x;       // conv: input [P][cin]; wgrad: forward input [P][cin]
    const bf16* w;       // conv: weights [cout][9][cin]; wgrad: output gradient dy [P][cout]
    const float* bias;   // conv: [cout] or null
    const bf16* mask;    // conv: [P][cout]; output multiplied by (mask > 0) (ReLU derivative) or null
    void* y;             // conv: [P][cout] bf16 or fp32; wgrad: fp32 partials [splits][m_pad][cout]
    int* err;            // device error word (VPT_ERR_ITER_LIMIT on an expired wait) or null
    int n, h, w_;        // batch and image size (pixels P = n * h * w_)
    int cin, cout;       // channel counts (multiples of 16)
    int n_tile;          // output columns per CTA (multiple of 16, <= 256)
    int tmem_cols;       // power of two >= n_tile, >= 32
    int relu, out_f32;   // conv epilogue
    int pix_per_split;   // wgrad: pixels (K) per CTA, multiple of kBK
    int m_pad;           // wgrad: rows of a partial (multiple of kBM)
    int ksplit;          // conv: K stages split over blockIdx.z (> 1: raw sums to `partial`)
    float* partial;      // conv split-K: fp32 [ksplit][P][cout]
};

__device__ __forceinline__ void pixel_coords(int p, int h, int w, int& n, int& y, int& x) {
    x = p % w;
    const int t = p / w;
    y = t % h;
    n = t / h;
}

// 16 output channels from co of pixel p: the split's raw sums, or bias, ReLU, mask and store
__device__ __forceinline__ void conv_store(const ConvArgs& a, int P, int p, int co, float (&v)[16]) {
    if (a.partial) {  // split-K: raw sums, finished by conv_finalize_kernel
        float4* dst = reinterpret_cast<float4*>(a.partial + ((size_t)blockIdx.z * P + p) * a.cout + co);
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        return;
    }
    if (a.bias) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] += a.bias[co + i];
    }
    if (a.relu) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = fmaxf(v[i], 0.0f);
    }
    if (a.mask) {
        const uint4* mp = reinterpret_cast<const uint4*>(a.mask + (size_t)p * a.cout + co);
        const uint4 m4[2] = {mp[0], mp[1]};
        const bf16* mb = reinterpret_cast<const bf16*>(m4);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = __bfloat162float(mb[i]) > 0.0f ? v[i] : 0.0f;
    }
    if (a.out_f32) {
        float4* dst = reinterpret_cast<float4*>(static_cast<float*>(a.y) + (size_t)p * a.cout + co);
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    } else {
        uint4 o[2];
        __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(o);
#pragma unroll
        for (int i = 0; i < 8; ++i) ob[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        uint4* dst = reinterpret_cast<uint4*>(static_cast<bf16*>(a.y) + (size_t)p * a.cout + co);
        dst[0] = o[0];
        dst[1] = o[1];
    }
}

template <int MODE, int kStages>
__global__ void __launch_bounds__(kThreads) conv_tile_kernel(const ConvArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t bars[kStages];
    __shared__ uint32_t tmem_slot;

    const int tid = threadIdx.x, warp_u = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int P = a.n * a.h * a.w_;
    const int n_tile = a.n_tile;
    const uint32_t a_bytes = kBM * kBK * 2;
    const uint32_t b_bytes = (uint32_t)n_tile * kBK * 2;
    const uint32_t stage_bytes = a_bytes + b_bytes;
    const uint32_t sbase = smem_u32(smem);
    const int n0 = blockIdx.y * n_tile;

    // K extent and tile origin
    int K, m0, kbeg = 0, kend = 0;
    int s_first = 0;  // conv split-K: first K stage of this CTA
    if (MODE == kConv) {
        K = 9 * a.cin;
        m0 = blockIdx.x * kBM;
    } else {
        m0 = blockIdx.x * kBM;  // rows m = tap * cin + ci
        kbeg = blockIdx.z * a.pix_per_split;
        kend = min(P, kbeg + a.pix_per_split);
        K = kend - kbeg;
    }
    const int M = (MODE == kConv) ? P : 9 * a.cin;
    int nk = (K + kBK - 1) / kBK;
    if (MODE == kConv && a.ksplit > 1) {
        const int per = (nk + a.ksplit - 1) / a.ksplit;
        s_first = blockIdx.z * per;
        nk = max(0, min(nk, s_first + per) - s_first);
    }

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) mbar_init(smem_u32(&bars[s]), 1);
        fence_mbar_init();
    }
    if (tid < 32) tmem_alloc(smem_u32(&tmem_slot), (uint32_t)a.tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);

    // per-thread gather state
    int pn = 0, py = 0, px = 0;
    bool p_ok = false;
    int wg_tap = 0, wg_ci = 0;
    bool wg_m_ok = false;
    if (MODE == kConv) {
        const int p = m0 + tid;  // this thread's A row
        p_ok = p < P;
        if (p_ok) pixel_coords(p, a.h, a.w_, pn, py, px);
    } else {
        const int m = m0 + ((tid >> 3) & 15) * 8;  // this thread's 8 A rows
        wg_m_ok = m < M;
        if (wg_m_ok) {
            wg_tap = m / a.cin;
            wg_ci = m - wg_tap * a.cin;
        }
    }

    // incremental gather state (stages are loaded in increasing order, so nothing is divided by a
    // runtime value inside the loop)
    int ld_tap = (s_first * kBK) / a.cin, ld_ci = (s_first * kBK) % a.cin;  // conv: next stage's first k
    int b_r0 = tid % n_tile, b_kc0 = tid / n_tile;   // conv: first B unit of this thread
    int wq_n = 0, wq_y = 0, wq_x = 0, wq_p = kbeg + (tid & 7);  // wgrad: this thread's next A pixel
    if (MODE == kWgrad && wq_p < P) pixel_coords(wq_p, a.h, a.w_, wq_n, wq_y, wq_x);
    const int nch = n_tile / 8;
    const int wb_rest0 = tid >> 3;
    const int wb_nc0 = wb_rest0 % nch, wb_kph0 = wb_rest0 / nch;

    auto load_stage = [&](int slot, int s) {
        const uint32_t sA = sbase + slot * stage_bytes;
        const uint32_t sB = sA + a_bytes;
        if (MODE == kConv) {
            const int k0 = (s_first + s) * kBK;
            // A: row tid, 8 chunks of 8 channels; unit (r, kc) at kc * kBM * 16 + r * 16
            int tap = ld_tap, ci = ld_ci;
#pragma unroll
            for (int kc = 0; kc < 8; ++kc) {
                const int kk = k0 + kc * 8;
                const bf16* src = a.x;
                bool v = false;
                if (p_ok && kk < K) {
                    const int dy = (tap * 11) >> 5, dx = tap - 3 * dy;  // tap / 3, tap % 3 for tap < 9
                    const int yy = py + dy - 1, xx = px + dx - 1;
                    if (yy >= 0 && yy < a.h && xx >= 0 && xx < a.w_) {
                        v = true;
                        src = a.x + ((size_t)(pn * a.h + yy) * a.w_ + xx) * a.cin + ci;
                    }
                }
                cp_async16(sA + kc * (kBM * 16) + tid * 16, src, v);
                ci += 8;
                while (ci >= a.cin) {
                    ci -= a.cin;
                    ++tap;
                }
            }
            ld_tap = tap;
            ld_ci = ci;
            // B: weight rows n0 .. n0 + n_tile; unit (r, kc) at kc * n_tile * 16 + r * 16
            int r = b_r0, kc = b_kc0;
            for (int q = tid; q < n_tile * 8; q += kThreads) {
                const int kk = k0 + kc * 8, co = n0 + r;
                const bool v = co < a.cout && kk < K;
                cp_async16(sB + kc * (n_tile * 16) + r * 16, v ? a.w + (size_t)co * K + kk : a.w, v);
                r += kThreads;
                while (r >= n_tile) {
                    r -= n_tile;
                    ++kc;
                }
            }
        } else {
            const int pbase = kbeg + s * kBK;
            // A (MN-major): unit (mc, kp) at (kp / 8) * 2048 + mc * 128 + (kp % 8) * 16 = 16 * q; this
            // thread's pixels advance by 8 per unit
            const int tdy = (wg_tap * 11) >> 5, tdx = wg_tap - 3 * tdy;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const bf16* src = a.x;
                bool v = false;
                if (wg_m_ok && wq_p < kend) {
                    const int yy = wq_y + tdy - 1, xx = wq_x + tdx - 1;
                    if (yy >= 0 && yy < a.h && xx >= 0 && xx < a.w_) {
                        v = true;
                        src = a.x + ((size_t)(wq_n * a.h + yy) * a.w_ + xx) * a.cin + wg_ci;
                    }
                }
                cp_async16(sA + (i * kThreads + tid) * 16, src, v);
                wq_p += 8;
                wq_x += 8;
                while (wq_x >= a.w_) {
                    wq_x -= a.w_;
                    if (++wq_y == a.h) {
                        wq_y = 0;
                        ++wq_n;
                    }
                }
            }
            // B (MN-major): dy rows; unit (nc, kp) at (kp / 8) * n_tile * 16 + nc * 128 + (kp % 8) * 16
            int nc = wb_nc0, kph = wb_kph0;
            for (int q = tid; q < n_tile * 8; q += kThreads) {
                const int p = pbase + kph * 8 + (tid & 7), co = n0 + nc * 8;
                const bool v = p < kend && co < a.cout;
                cp_async16(sB + q * 16, v ? a.w + (size_t)p * a.cout + co : a.w, v);
                nc += kThreads / 8;
                while (nc >= nch) {
                    nc -= nch;
                    ++kph;
                }
            }
        }
    };

    const uint32_t idesc = (MODE == kConv) ? instr_desc(kBM, n_tile, 0, 0) : instr_desc(kBM, n_tile, 1, 1);
    const uint32_t a_lbo = (MODE == kConv) ? kBM * 16 : (kBM / 8) * 128;
    const uint32_t b_lbo = (uint32_t)n_tile * 16;

    for (int s = 0; s < kStages - 1; ++s) {
        if (s < nk) load_stage(s, s);
        cp_async_commit();
    }
    int aborted = 0;
    int issued = -1;  // last stage whose MMAs were committed
    for (int s = 0; s < nk; ++s) {
        const int slot = s % kStages;
        cp_async_wait<kStages - 2>();
        fence_proxy_async();
        if (__syncthreads_or(aborted)) break;
        if (warp_u == 0) {
            tc_fence_after();
            if (elect_one()) {
                const uint32_t sA = sbase + slot * stage_bytes;
                const uint32_t sB = sA + a_bytes;
                const int steps = min(kBK / 16, (K - (s_first + s) * kBK + 15) / 16);
                const uint64_t da = smem_desc(sA, a_lbo, 128), db = smem_desc(sB, b_lbo, 128);
                const uint32_t a_lo = (uint32_t)da, a_hi = (uint32_t)(da >> 32);
                const uint32_t b_lo = (uint32_t)db, b_hi = (uint32_t)(db >> 32);
                for (int j = 0; j < steps; ++j)  // 16 K: two 8-channel planes of each operand
                    mma_bf16_halves(tmem, a_lo + (uint32_t)j * (a_lbo >> 3), a_hi, b_lo + (uint32_t)j * (b_lbo >> 3), b_hi,
                                    idesc, (s > 0 || j > 0) ? 1u : 0u);
                mma_commit(smem_u32(&bars[slot]));
            }
            __syncwarp();
        }
        issued = s;
        const int nxt = s + kStages - 1;
        if (nxt < nk) {
            bool ok = true;
            if (s >= 1) {  // the slot of stage s - 1 is refilled: its MMAs must have read it
                const int ps = s - 1;
                ok = mbar_wait(smem_u32(&bars[ps % kStages]), (uint32_t)((ps / kStages) & 1));
            }
            if (ok) load_stage(nxt % kStages, nxt);
            else aborted = 1;
        }
        cp_async_commit();
    }
    cp_async_wait<0>();
    // the last commit tracks every MMA this CTA issued
    bool done = true;
    if (issued >= 0) done = mbar_wait(smem_u32(&bars[issued % kStages]), (uint32_t)((issued / kStages) & 1));
    const bool fail = __syncthreads_or(aborted || !done || (issued != nk - 1 && nk > 0));
    tc_fence_after();

    if (!fail && nk == 0 && MODE == kConv && a.partial) {  // an empty K range contributes zeros
        const int p = m0 + tid;
        if (p < P)
            for (int co = n0; co < min(a.cout, n0 + n_tile); co += 4)
                *reinterpret_cast<float4*>(a.partial + ((size_t)blockIdx.z * P + p) * a.cout + co) =
                    make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    if (!fail && nk > 0) {
        const int warp = tid >> 5, lane = tid & 31;
        const int r = warp * 32 + lane;
        const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
        for (int c0 = 0; c0 < n_tile; c0 += 16) {
            float v[16];
            tmem_ld16(trow + (uint32_t)c0, v);  // whole warp, uniform
            const int co = n0 + c0;
            if (co >= a.cout) continue;
            if (MODE == kConv) {
                const int p = m0 + r;
                if (p >= P) continue;
                conv_store(a, P, p, co, v);
            } else {
                const int m = m0 + r;
                if (m >= M) continue;
                float4* dst = reinterpret_cast<float4*>(static_cast<float*>(a.y) +
                                                        ((size_t)blockIdx.z * a.m_pad + m) * a.cout + co);
#pragma unroll
                for (int i = 0; i < 4; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            }
        }
    }
    if (fail && tid == 0 && a.err) atomicExch(a.err, (int)VPT_ERR_ITER_LIMIT);
    tc_fence_before();
    __syncthreads();
    if (tid < 32) {
        tc_fence_after();
        tmem_dealloc(tmem, (uint32_t)a.tmem_cols);
    }
}

// Split-K convolution: y = act(bias + sum over the splits of partial[s]) (fixed order), times the
// ReLU-derivative mask, stored bf16 or fp32; 4 channels per thread.
template <class I>
__global__ void conv_finalize_kernel(const float* __restrict__ partial, int ksplit, long P, int cout,
                                     const float* __restrict__ bias, const bf16* __restrict__ mask, int relu,
                                     int out_f32, void* __restrict__ y) {
    const I c4 = (I)(cout / 4), total = (I)P * c4;
    for (I i = (I)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const size_t p = i / c4;
        const int c = (int)(i - (I)p * c4) * 4;
        float4 acc = reinterpret_cast<const float4*>(partial + p * cout + c)[0];
        for (int k = 1; k < ksplit; ++k) {
            const float4 u = reinterpret_cast<const float4*>(partial + ((size_t)k * P + p) * cout + c)[0];
            acc.x += u.x;
            acc.y += u.y;
            acc.z += u.z;
            acc.w += u.w;
        }
        float v[4] = {acc.x, acc.y, acc.z, acc.w};
        for (int j = 0; j < 4; ++j) {
            if (bias) v[j] += bias[c + j];
            if (relu) v[j] = fmaxf(v[j], 0.0f);
            if (mask) v[j] = __bfloat162float(mask[p * cout + c + j]) > 0.0f ? v[j] : 0.0f;
        }
        if (out_f32) {
            reinterpret_cast<float4*>(static_cast<float*>(y) + p * cout + c)[0] = make_float4(v[0], v[1], v[2], v[3]);
        } else {
            __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(static_cast<bf16*>(y) + p * cout + c);
            o[0] = __floats2bfloat162_rn(v[0], v[1]);
            o[1] = __floats2bfloat162_rn(v[2], v[3]);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// the row-strip convolution (forward and input gradient on images at least 128 pixels wide)
// ---------------------------------------------------------------------------------------------
// A persistent CTA owns segments of consecutive rows of one 128-pixel-wide image column
// (n, x0 .. x0 + 127).  The output tile of row y needs input rows y-1, y, y+1 at x0-1 .. x0+128: each
// input row is gathered once into a ring of 5 shared-memory row strips (130 pixels per 8-channel
// plane, 16 bytes per pixel, planes 2080 bytes apart), so that a row stays resident for the three
// output rows that use it and the row two ahead is in flight.  In the UMMA K-major no-swizzle layout
// (8-row core matrices of 16-byte rows, SBO = 128 between 8-pixel groups, LBO = plane stride between
// 8-channel chunks) the A operand of tap (dy, dx) is the strip of row y+dy with its start address
// moved by dx * 16 bytes: the three horizontal taps share one gather.  All 9 taps of the weights are
// resident in shared memory for the CTA's lifetime.  Two TMEM accumulators alternate: the epilogue
// of tile i-1 (tcgen05.ld, bias, ReLU, mask, store) runs while the tensor core computes tile i.
constexpr int kStripPix = kBM + 2;          // 130 pixels: x0-1 .. x0+128
constexpr int kPlane = kStripPix * 16;      // bytes per 8-channel plane of a row strip
constexpr int kRing = 5;                    // row strips resident

struct StripArgs {
    const bf16* x;       // [n][h][w][cin]
    const bf16* w;       // [cout][9][cin]
    const float* bias;   // [cout] or null
    const bf16* mask;    // [n][h][w][cout] or null
    void* y;             // [n][h][w][cout] bf16 / fp32
    int* err;
    int n, h, w_, cin, cout;   // cin: input channels of this pass (a group of the tensor's channels)
    int cin_total, c0;         // channels per pixel of x (and per tap of w); first channel of this pass
    const float* part_in;      // fp32 [n][h][w][cout] partial sum added before the epilogue, or null
    float* part_out;           // non-null: store the raw fp32 sum here (an intermediate pass), no epilogue
    int relu, out_f32;
    int xtiles;          // ceil(w / 128)
    int seg_rows;        // rows per segment
    int segs_per_col;
    int tmem_cols;
};

// TMEM lane quarter `quarter` (the warp's index mod 4) holds pixels x0 + 32 quarter .. + 31
__device__ __forceinline__ void strip_epilogue(const StripArgs& a, uint32_t tacc, int n_img, int yrow, int x0,
                                               int quarter, int lane) {
    const int x = x0 + quarter * 32 + lane;
    const bool ok = x < a.w_;
    const size_t p = ((size_t)n_img * a.h + yrow) * a.w_ + (ok ? x : 0);
    const uint32_t trow = tacc + ((uint32_t)(quarter * 32) << 16);
    for (int c0 = 0; c0 < a.cout; c0 += 16) {
        float v[16];
        tmem_ld16(trow + (uint32_t)c0, v);
        if (!ok) continue;
        if (a.part_in) {
            const float4* src = reinterpret_cast<const float4*>(a.part_in + p * a.cout + c0);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 u = src[i];
                v[4 * i] += u.x;
                v[4 * i + 1] += u.y;
                v[4 * i + 2] += u.z;
                v[4 * i + 3] += u.w;
            }
        }
        if (a.part_out) {
            float4* dst = reinterpret_cast<float4*>(a.part_out + p * a.cout + c0);
#pragma unroll
            for (int i = 0; i < 4; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            continue;
        }
        if (a.bias) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += a.bias[c0 + i];
        }
        if (a.relu) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = fmaxf(v[i], 0.0f);
        }
        if (a.mask) {
            const uint4* mp = reinterpret_cast<const uint4*>(a.mask + p * a.cout + c0);
            const uint4 m4[2] = {mp[0], mp[1]};
            const bf16* mb = reinterpret_cast<const bf16*>(m4);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __bfloat162float(mb[i]) > 0.0f ? v[i] : 0.0f;
        }
        if (a.out_f32) {
            float4* dst = reinterpret_cast<float4*>(static_cast<float*>(a.y) + p * a.cout + c0);
#pragma unroll
            for (int i = 0; i < 4; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        } else {
            uint4 o[2];
            __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(o);
#pragma unroll
            for (int i = 0; i < 8; ++i) ob[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            uint4* dst = reinterpret_cast<uint4*>(static_cast<bf16*>(a.y) + p * a.cout + c0);
            dst[0] = o[0];
            dst[1] = o[1];
        }
    }
}

__global__ void __launch_bounds__(kThreads) conv_strip_kernel(const StripArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t bars[2];
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x;
    const int nkc = a.cin / 8;
    const uint32_t w_bytes = 9u * (uint32_t)a.cin * (uint32_t)a.cout * 2u;
    const uint32_t row_bytes = (uint32_t)nkc * kPlane;
    const uint32_t sw = smem_u32(smem);
    const uint32_t sring = sw + ((w_bytes + 127u) & ~127u);

    if (tid == 0) {
        mbar_init(smem_u32(&bars[0]), 1);
        mbar_init(smem_u32(&bars[1]), 1);
        fence_mbar_init();
    }
    if (tid < 32) tmem_alloc(smem_u32(&tmem_slot), (uint32_t)a.tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    // resident weights: unit (t, kc, co) at ((t * nkc + kc) * cout + co) * 16
    for (int q = tid; q < 9 * nkc * a.cout; q += kThreads) {
        const int co = q % a.cout, rest = q / a.cout;
        const int kc = rest % nkc, t = rest / nkc;
        cp_async16(sw + (uint32_t)q * 16u, a.w + ((size_t)co * 9 + t) * a.cin_total + a.c0 + kc * 8, true);
    }
    cp_async_commit();

    auto load_row = [&](int n_img, int yy, int x0) {
        const uint32_t base = sring + (uint32_t)(((yy + 1) % kRing + kRing) % kRing) * row_bytes;
        const bool row_ok = yy >= 0 && yy < a.h;
        for (int q = tid; q < kStripPix * nkc; q += kThreads) {
            const int r = q % kStripPix, kc = q / kStripPix;
            const int xx = x0 - 1 + r;
            const bool v = row_ok && xx >= 0 && xx < a.w_;
            const bf16* src = v ? a.x + (((size_t)n_img * a.h + yy) * a.w_ + xx) * a.cin_total + a.c0 + kc * 8 : a.x;
            cp_async16(base + (uint32_t)kc * kPlane + (uint32_t)r * 16u, src, v);
        }
    };

    const uint32_t idesc = instr_desc(kBM, a.cout, 0, 0);
    const uint32_t b_lbo = (uint32_t)a.cout * 16u;
    const int total_segs = a.n * a.xtiles * a.segs_per_col;
    long g = 0;          // tiles computed by this CTA (accumulator index and mbarrier parity)
    int fail = 0;
    int pend_n = 0, pend_y = 0, pend_x0 = 0;
    bool pending = false;  // a tile whose epilogue has not run

    for (int seg = blockIdx.x; seg < total_segs && !fail; seg += gridDim.x) {
        const int col = seg / a.segs_per_col, part = seg % a.segs_per_col;
        const int n_img = col / a.xtiles, x0 = (col % a.xtiles) * kBM;
        const int y0 = part * a.seg_rows, y1 = min(a.h, y0 + a.seg_rows);
        if (y0 >= y1) continue;
        // every MMA of the previous segment has finished reading the ring
        if (pending) {
            if (!mbar_wait(smem_u32(&bars[(g - 1) & 1]), (uint32_t)(((g - 1) >> 1) & 1))) fail = 1;
            if (__syncthreads_or(fail)) break;
            tc_fence_after();
            strip_epilogue(a, tmem + (uint32_t)(((g - 1) & 1) * a.cout), pend_n, pend_y, pend_x0, tid >> 5, tid & 31);
            pending = false;
        }
        load_row(n_img, y0 - 1, x0);
        load_row(n_img, y0, x0);
        load_row(n_img, y0 + 1, x0);
        cp_async_commit();
        if (y0 + 2 <= y1) load_row(n_img, y0 + 2, x0);
        cp_async_commit();
        for (int yrow = y0; yrow < y1; ++yrow, ++g) {
            cp_async_wait<1>();  // rows yrow-1 .. yrow+1 (and the weights) have landed
            fence_proxy_async();
            tc_fence_before();
            if (__syncthreads_or(fail)) break;
            const int buf = (int)(g & 1);
            if (tid == 0) {
                tc_fence_after();
                const uint32_t dacc = tmem + (uint32_t)(buf * a.cout);
                int first = 1;
                for (int dy = 0; dy < 3; ++dy) {
                    const uint32_t rb = sring + (uint32_t)((yrow + dy) % kRing) * row_bytes;  // slot of row yrow+dy-1
                    for (int dx = 0; dx < 3; ++dx) {
                        const int t = dy * 3 + dx;
                        for (int j = 0; j < nkc / 2; ++j) {
                            const uint64_t da = smem_desc(rb + (uint32_t)(2 * j) * kPlane + (uint32_t)dx * 16u, kPlane,
                                                          128);
                            const uint64_t db = smem_desc(sw + (uint32_t)((t * nkc + 2 * j) * a.cout) * 16u, b_lbo, 128);
                            mma_bf16(dacc, da, db, idesc, first ? 0u : 1u);
                            first = 0;
                        }
                    }
                }
                mma_commit(smem_u32(&bars[buf]));
            }
            if (pending) {  // epilogue of the previous tile while this one computes
                if (!mbar_wait(smem_u32(&bars[(g - 1) & 1]), (uint32_t)(((g - 1) >> 1) & 1))) fail = 1;
                if (__syncthreads_or(fail)) break;
                tc_fence_after();
                strip_epilogue(a, tmem + (uint32_t)(((g - 1) & 1) * a.cout), pend_n, pend_y, pend_x0, tid >> 5, tid & 31);
            }
            pending = true;
            pend_n = n_img;
            pend_y = yrow;
            pend_x0 = x0;
            // the previous tile's MMAs are done: the slot of row yrow-2 is free for row yrow+3
            if (yrow + 3 <= y1) load_row(n_img, yrow + 3, x0);
            cp_async_commit();
        }
    }
    cp_async_wait<0>();
    if (pending && !fail) {
        if (!mbar_wait(smem_u32(&bars[(g - 1) & 1]), (uint32_t)(((g - 1) >> 1) & 1))) fail = 1;
        if (!__syncthreads_or(fail)) {
            tc_fence_after();
            strip_epilogue(a, tmem + (uint32_t)(((g - 1) & 1) * a.cout), pend_n, pend_y, pend_x0, tid >> 5, tid & 31);
        }
    } else if (pending) {
        // bounded wait for the MMAs in flight before the accumulator is freed
        mbar_wait(smem_u32(&bars[(g - 1) & 1]), (uint32_t)(((g - 1) >> 1) & 1));
    }
    if (__syncthreads_or(fail) && tid == 0 && a.err) atomicExch(a.err, (int)VPT_ERR_ITER_LIMIT);
    tc_fence_before();
    __syncthreads();
    if (tid < 32) {
        tc_fence_after();
        tmem_dealloc(tmem, (uint32_t)a.tmem_cols);
    }
}

// ---------------------------------------------------------------------------------------------
// the warp-specialised row-strip convolution (TMA-fed)
// ---------------------------------------------------------------------------------------------
// The tiling of conv_strip_kernel (persistent CTAs over segments of consecutive rows of one
// 128-pixel column; row strips of 130 pixels; A of tap (dy, dx) = the strip of row y+dy-1 with its
// start moved by dx pixel rows; the weights of all 9 taps resident), with the work split over warps
// and no CTA-wide barrier after the weights have landed:
//   warp 0     one lane loads input rows into a ring of `ring` slots with the tensor-memory-access
//              unit: one box {64 / 32 / 16 channels, 130 pixels} per channel group, written in the
//              swizzled K-major layout of that line width (pixel rows of 128 / 64 / 32 bytes), rows and
//              pixels outside the image arriving as zeros; full[s] completes on the bytes, empty[s] is
//              signalled by the tensor core once the last MMA reading the slot has completed;
//   warps 1, 6 each issue the 9 x cin/16 MMAs of every other output row (accumulator
//              index g: warp 1 the even, warp 6 the odd) into TMEM accumulator g % 2 (acc_full[b] on
//              completion, after acc_empty[b]): one issuing thread is the bound for small N (about 93
//              cycles per MMA against the tensor core's 48), two overlap their issue;
//   warps 2-5  the epilogue; warp w reads TMEM lane quarter w % 4 (pixels x0 + 32 (w % 4) .. + 31).
// All roles walk the same segment sequence, so ring and accumulator positions agree without
// communication.  Every wait is bounded: on expiry the role records the error and stops, and the
// CTA waits (bounded) for its copies and MMAs in flight before TMEM is released.
constexpr int kWsThreads = 224;  // 7 warps: producer, MMA issuer, 4 epilogue warps, second MMA issuer
constexpr int kWsMaxRing = 8;

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// tiled 4-D load (coordinates innermost first) into this CTA's shared memory, completing on `bar`
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];\n" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
        : "memory");
}

struct WsSegment {
    int n_img, x0, y0, y1;
};
__device__ __forceinline__ WsSegment ws_segment(const StripArgs& a, int seg) {
    const int col = seg / a.segs_per_col, part = seg % a.segs_per_col;
    WsSegment g;
    g.n_img = col / a.xtiles;
    g.x0 = (col % a.xtiles) * kBM;
    g.y0 = part * a.seg_rows;
    g.y1 = min(a.h, g.y0 + a.seg_rows);
    return g;
}

// Channel groups of a row: widths 64 / 32 / 16 channels = lines of 128 / 64 / 32 bytes per pixel in
// the 128B / 64B / 32B-swizzled K-major layout (what one TMA box of {width, 130 pixels} writes);
// each group buffer starts on a 1024-byte boundary.
constexpr int kWsMaxGroups = 4;
struct WsArgs {
    StripArgs s;
    int ngroups;
    int gc[kWsMaxGroups];    // first channel of the group (within this pass)
    int gw[kWsMaxGroups];    // channels of the group: 64, 32 or 16
    int goff[kWsMaxGroups];  // byte offset of the group buffer in a ring slot
    int row_bytes;           // ring slot size
    int tx_bytes;            // bytes the boxes of one row deliver
};

// K-major swizzled shared-memory descriptor: line = 128 / 64 / 32 bytes per row, 8-row groups
// `8 * line` apart (SBO), LBO unused (1), layout type 2 / 4 / 6 (bits 61-63).  The swizzle acts on
// absolute shared-memory address bits (as the TMA's does), so a start moved by whole rows (the dx
// taps) needs no base offset (measured: base offset 0 matches the oracle for every line width).
__device__ __forceinline__ uint64_t smem_desc_sw(uint32_t addr, uint32_t line) {
    uint64_t d = (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(((8u * line) >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    const uint64_t layout = line == 128 ? 2 : (line == 64 ? 4 : 6);
    d |= layout << 61;
    return d;
}

// high word of smem_desc_sw: SBO = 8 lines, version, layout type of the line width (2 * channels)
__device__ __forceinline__ uint32_t a_hi_of(int channels) {
    return (uint32_t)(smem_desc_sw(0, (uint32_t)channels * 2u) >> 32);
}

__global__ void __launch_bounds__(kWsThreads, 2) conv_ws_kernel(const __grid_constant__ CUtensorMap map64,
                                                             const __grid_constant__ CUtensorMap map32,
                                                             const __grid_constant__ CUtensorMap map16,
                                                             const __grid_constant__ WsArgs wa, int ring) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[kWsMaxRing], empty[kWsMaxRing], acc_full[2], acc_empty[2], done_bar[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int fail_any;
    const StripArgs& a = wa.s;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int nkc = a.cin / 8;
    const uint32_t w_bytes = 9u * (uint32_t)a.cin * (uint32_t)a.cout * 2u;
    const uint32_t row_bytes = (uint32_t)wa.row_bytes;
    const uint32_t sw = smem_u32(smem);
    const uint32_t sring = sw + ((w_bytes + 1023u) & ~1023u);
    const uint32_t acc_cols = (uint32_t)a.tmem_cols / 2;
    if (tid == 0) {
        for (int s = 0; s < ring; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 2);  // one release per MMA-issuing warp
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full[b]), 1);
            mbar_init(smem_u32(&acc_empty[b]), 4);  // one arrival per epilogue warp
            mbar_init(smem_u32(&done_bar[b]), 1);
        }
        fail_any = 0;
        fence_mbar_init();
    }
    if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), (uint32_t)a.tmem_cols);
    // resident weights: unit (t, kc, co) at ((t * nkc + kc) * cout + co) * 16
    for (int q = tid; q < 9 * nkc * a.cout; q += kWsThreads) {
        const int co = q % a.cout, rest = q / a.cout;
        const int kc = rest % nkc, t = rest / nkc;
        cp_async16(sw + (uint32_t)q * 16u, a.w + ((size_t)co * 9 + t) * a.cin_total + a.c0 + kc * 8, true);
    }
    cp_async_commit();
    cp_async_wait<0>();
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    const int total_segs = a.n * a.xtiles * a.segs_per_col;
    bool fail = false;

    if (warp == 0) {
        if (lane == 0) {
            int slot = 0;
            uint32_t phase = 0;
            long issued = 0;
            for (int seg = blockIdx.x; seg < total_segs && !fail; seg += gridDim.x) {
                const WsSegment g = ws_segment(a, seg);
                if (g.y0 >= g.y1) continue;
                for (int yy = g.y0 - 1; yy <= g.y1; ++yy) {
                    if (!mbar_wait(smem_u32(&empty[slot]), phase ^ 1u)) {
                        fail = true;
                        break;
                    }
                    const uint32_t dst = sring + (uint32_t)slot * row_bytes;
                    const uint32_t fb = smem_u32(&full[slot]);
                    mbar_arrive_expect_tx(fb, (uint32_t)wa.tx_bytes);
                    for (int k = 0; k < wa.ngroups; ++k) {
                        const CUtensorMap* m = wa.gw[k] == 64 ? &map64 : (wa.gw[k] == 32 ? &map32 : &map16);
                        tma_load_4d(dst + (uint32_t)wa.goff[k], m, a.c0 + wa.gc[k], g.x0 - 1, yy, g.n_img, fb);
                    }
                    ++issued;
                    if (++slot == ring) {
                        slot = 0;
                        phase ^= 1u;
                    }
                }
            }
            // the last loads (one per slot at most) have landed before the CTA can exit
            const long tail = issued < ring ? issued : ring;
            for (long k = 1; k <= tail; ++k) {
                int s = slot - (int)k;
                uint32_t ph = phase;
                if (s < 0) {
                    s += ring;
                    ph ^= 1u;
                }
                if (!mbar_wait(smem_u32(&full[s]), ph)) fail = true;
            }
        }
    } else if (warp == 1 || warp == 6) {
        const int mw = warp == 1 ? 0 : 1;  // this warp's accumulator parity
        const uint32_t idesc = instr_desc(kBM, a.cout, 0, 0);
        // descriptor words: A (swizzled, start field added per row / group / dx / step; LBO 1),
        // B (no swizzle, LBO = one 8-channel plane of the weights, SBO 128)
        const uint64_t bd0 = smem_desc(sw, (uint32_t)a.cout * 16u, 128);
        const uint32_t b_hi = (uint32_t)(bd0 >> 32), b_lo0 = (uint32_t)bd0;
        const uint32_t a_lo1 = 1u << 16;  // LBO field of the A descriptors
        const uint32_t b_step = 2u * (uint32_t)a.cout, b_tap = (uint32_t)(nkc * a.cout), b_row = 3u * b_tap;
        const int ngroups = wa.ngroups;
        int slot = 0;        // ring position of the segment's first row
        uint32_t phase = 0;
        long g = 0;          // accumulators used (both warps count every output row)
        // Ring slots are released by both issuing warps (empty[] counts 2): after output row i
        // its warp releases input rows i and i+1 (its last uses of them: it also computed row
        // i-2, the other warp rows i-1 and i+1).  Rows without such a row get the arrival at the
        // segment's start (input row 0 from the warp of row -1) or end (rows `rows`, `rows`+1).
        auto own = [&](long gi) { return (int)(gi & 1) == mw; };
        auto slot_of = [&](int r) { return (uint32_t)((slot + r) % ring); };
        for (int seg = blockIdx.x; seg < total_segs && !fail; seg += gridDim.x) {
            const WsSegment sgm = ws_segment(a, seg);
            if (sgm.y0 >= sgm.y1) continue;
            const int rows = sgm.y1 - sgm.y0;
            const long g0 = g;
            if (own(g0 - 1) && elect_one()) mbar_arrive(smem_u32(&empty[slot_of(0)]));
            __syncwarp();
            for (int i = 0; i < rows && !fail; ++i, ++g) {
                if (!own(g)) continue;
                // input rows i, i+1, i+2 of the segment (y-1, y, y+1)
                bool ok = true;
                for (int k = 0; k <= 2; ++k) {
                    const int pos = slot + i + k;
                    const uint32_t ph = phase ^ (uint32_t)((pos / ring) & 1);
                    ok = ok && mbar_wait(smem_u32(&full[pos % ring]), ph);
                }
                const int b = (int)(g & 1);
                ok = ok && mbar_wait(smem_u32(&acc_empty[b]), (uint32_t)(((g >> 1) & 1) ^ 1));
                if (!__all_sync(0xffffffffu, ok)) {
                    fail = true;
                    break;
                }
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t dacc = tmem + (uint32_t)b * acc_cols;
                    // descriptors walk affinely: per channel group, A's start advances by one pixel
                    // row per dx and 32 bytes per 16-channel step, B's by a tap (nkc * cout * 16
                    // bytes) per dx and two 8-channel planes per step
                    uint32_t acc = 0;
                    for (int dy = 0; dy < 3; ++dy) {
                        const uint32_t row16 = (sring + slot_of(i + dy) * row_bytes) >> 4;
                        for (int k = 0; k < ngroups; ++k) {
                            const int gw = wa.gw[k];
                            const uint32_t ahi = a_hi_of(gw);
                            uint32_t al = a_lo1 + row16 + ((uint32_t)wa.goff[k] >> 4);
                            uint32_t bl = b_lo0 + (uint32_t)dy * b_row + (uint32_t)((wa.gc[k] >> 3) * a.cout);
#pragma unroll
                            for (int dx = 0; dx < 3; ++dx) {
                                for (int jj = 0; jj < gw / 16; ++jj) {
                                    mma_bf16_halves(dacc, al + 2u * (uint32_t)jj, ahi, bl + (uint32_t)jj * b_step, b_hi,
                                                    idesc, acc);
                                    acc = 1;
                                }
                                al += (uint32_t)gw >> 3;
                                bl += b_tap;
                            }
                        }
                    }
                    mma_commit(smem_u32(&acc_full[b]));
                    mma_commit(smem_u32(&empty[slot_of(i)]));
                    mma_commit(smem_u32(&empty[slot_of(i + 1)]));
                }
                __syncwarp();
            }
            if (fail) break;
            if (elect_one()) {
                if (own(g0 + rows - 1)) mma_commit(smem_u32(&empty[slot_of(rows + 1)]));
                if (own(g0 + rows)) {
                    mma_commit(smem_u32(&empty[slot_of(rows)]));
                    mma_commit(smem_u32(&empty[slot_of(rows + 1)]));
                }
            }
            __syncwarp();
            const int adv = slot + rows + 2;
            slot = adv % ring;
            phase ^= (uint32_t)((adv / ring) & 1);
        }
        // every MMA this warp issued has completed before TMEM is released
        if (elect_one()) mma_commit(smem_u32(&done_bar[mw]));
        __syncwarp();
        if (!mbar_wait(smem_u32(&done_bar[mw]), 0)) fail = true;
    } else if (warp >= 2 && warp <= 5) {
        const int quarter = warp & 3;
        long g = 0;
        for (int seg = blockIdx.x; seg < total_segs && !fail; seg += gridDim.x) {
            const WsSegment sgm = ws_segment(a, seg);
            for (int y = sgm.y0; y < sgm.y1; ++y, ++g) {
                const int b = (int)(g & 1);
                const bool ok = mbar_wait(smem_u32(&acc_full[b]), (uint32_t)((g >> 1) & 1));
                if (!__all_sync(0xffffffffu, ok)) {
                    fail = true;
                    break;
                }
                tc_fence_after();
                strip_epilogue(a, tmem + (uint32_t)b * acc_cols, sgm.n_img, y, sgm.x0, quarter, lane);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&acc_empty[b]));
            }
        }
    }
    if (fail) atomicOr(&fail_any, 1);
    tc_fence_before();
    __syncthreads();
    if (fail_any && tid == 0 && a.err) atomicExch(a.err, (int)VPT_ERR_ITER_LIMIT);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, (uint32_t)a.tmem_cols);
    }
}


// ---------------------------------------------------------------------------------------------
// the warp-specialised row-strip convolution with stacked rows
// ---------------------------------------------------------------------------------------------
// conv_ws_kernel issues 9 x cin/16 MMAs of N = cout columns a row, and an MMA takes the same time for every N up to
// 96 (its issue, about 93 cycles; the tensor core's own minimum is 48).  This kernel turns the sum over dy around:
// the three output rows y-1, y, y+1 that read input row y have adjacent accumulators, and one MMA of N = 3 cout
// columns adds input row y's contribution to all of them, its B operand being the taps dy = +1, 0, -1 stacked:
// 3 x cin/16 (+ 1) MMAs a row.  A launch computes `cout` <= 80 of the layer's output channels.
//   Layer, us, 8 images of 256 x 256 (conv_ws_kernel / here): 96 -> 32 93.0 / 52.6, 32 -> 32 29.0 / 22.5, 16 -> 32
// 23.7 / 17.9; one image of 256 x 256, 32 -> 32 10.0 / 10.2, 48 -> 48 at half that size 17.2 / 13.2.  Bound: 8 us
// to start, load the weights and drain, then the bytes (32 -> 32 67 MB, 10 us at 6.65 TB/s; 96 -> 32 134 MB, 20 us)
// and the MMAs' issue (96 -> 32: 19 of about 90 cycles a row and 28 rows an SM, 25 us), which overlap in part.  (One loop over the pairs of group and dx, for both orders: 66.8.)
//   ring      input rows as in conv_ws_kernel, but a slot is free again after its own row's MMAs: two slots do.
//   TMEM      a ring of `blocks` accumulators of cout columns, output row g of the CTA in block g % blocks;
//             three adjacent rows are contiguous columns except around the ring's end (then two MMAs).
//   first use an output row's first MMA (its dy = -1 taps, dx = -1, first 16 channels) overwrites its block,
//             so that step is split into N = cout (overwrite) and the older rows (accumulate).
//   sums      an output's products are added row by row, in a row by channel group and in a group by tap, as
//             conv_ws_kernel adds them; or (by_tap) by tap and in a tap by channel, as conv_tile_kernel does.  A layer
//             of two passes over its input channels (ConvOrder) has a ring of accumulators for each, which the
//             epilogue adds.
//   order     one thread issues every MMA, so an accumulator's updates and the commits behind them are in
//             order: after input row q's MMAs one commit frees its ring slot, one hands row q-2 (counted
//             from the segment's start) to the epilogue.
// Warps: 0 loads input rows, 1 issues, 2-9 run the epilogue (two teams of four take the rows alternately: one
// team, 2700 cycles a row of 32 channels, was the kernel's bound).  The weights are copied by warps 1-9 while
// the first rows arrive.  Every wait is bounded, as in conv_ws_kernel.
constexpr int kStackThreads = 320;  // producer, issuer, 8 epilogue warps
constexpr int kStackMaxBlocks = 8;
constexpr int kStackMaxCout = 80;  // 3 cout <= 256 columns

struct StackArgs {
    WsArgs ws;
    int ring, blocks;
    int groups0;  // channel groups of the first pass (all of them: one ring of accumulators)
    int by_tap;   // order of an input row's products
    int co0, cout_total;  // first output channel of this launch, channels per pixel of y
};

// The image columns (at most 128 pixels wide) of a batch, their rows taken as one sequence that the CTAs split
// evenly: CTA i owns rows [i R / G, (i + 1) R / G), in segments of one column each.
struct RowRange {
    int row, end, h, xtiles;
    __device__ __forceinline__ RowRange(int n, int h_, int xtiles_) : h(h_), xtiles(xtiles_) {
        const long rows = (long)n * xtiles_ * h_;
        row = (int)(rows * blockIdx.x / gridDim.x);
        end = (int)(rows * (blockIdx.x + 1) / gridDim.x);
    }
    __device__ __forceinline__ bool next(WsSegment& g) {
        if (row >= end) return false;
        const int col = row / h;
        g.n_img = col / xtiles;
        g.x0 = (col % xtiles) * kBM;
        g.y0 = row - col * h;
        g.y1 = min(h, g.y0 + (end - row));
        row += g.y1 - g.y0;
        return true;
    }
};

// Epilogue of one accumulator row for this warp's 32 pixels (at: offset of the lane's pixel and this
// launch's first channel): partial sums
// of earlier passes, bias, ReLU, mask, store.  set2: column offset of a second accumulator that is added (0 = none).
__device__ __forceinline__ void stack_epilogue(const StripArgs& a, const float* bias, uint32_t tacc, uint32_t set2,
                                               size_t at, bool ok, const uint4 (&mask)[kStackMaxCout / 8]) {
#pragma unroll
    for (int k = 0; k < kStackMaxCout / 16; ++k) {
        const int c0 = 16 * k;
        if (c0 >= a.cout) break;
        float v[16];
        tmem_ld16(tacc + (uint32_t)c0, v);
        if (set2) {
            float v2[16];
            tmem_ld16(tacc + set2 + (uint32_t)c0, v2);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += v2[i];
        }
        if (!ok) continue;
        if (a.part_in) {
            const float4* src = reinterpret_cast<const float4*>(a.part_in + at + c0);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 t = src[i];
                v[4 * i] += t.x;
                v[4 * i + 1] += t.y;
                v[4 * i + 2] += t.z;
                v[4 * i + 3] += t.w;
            }
        }
        if (a.part_out) {
            float4* dst = reinterpret_cast<float4*>(a.part_out + at + c0);
#pragma unroll
            for (int i = 0; i < 4; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            continue;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] += bias[c0 + i];
        if (a.relu) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = fmaxf(v[i], 0.0f);
        }
        if (a.mask) {
            const uint4 m4[2] = {mask[2 * k], mask[2 * k + 1]};
            const bf16* mb = reinterpret_cast<const bf16*>(m4);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __bfloat162float(mb[i]) > 0.0f ? v[i] : 0.0f;
        }
        if (a.out_f32) {
            float4* dst = reinterpret_cast<float4*>(static_cast<float*>(a.y) + at + c0);
#pragma unroll
            for (int i = 0; i < 4; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        } else {
            uint4 o[2];
            __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(o);
#pragma unroll
            for (int i = 0; i < 8; ++i) ob[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            uint4* dst = reinterpret_cast<uint4*>(static_cast<bf16*>(a.y) + at + c0);
            dst[0] = o[0];
            dst[1] = o[1];
        }
    }
}

__global__ void __launch_bounds__(kStackThreads, 2)
    conv_stack_kernel(const __grid_constant__ CUtensorMap map64, const __grid_constant__ CUtensorMap map32,
                      const __grid_constant__ CUtensorMap map16, const __grid_constant__ StackArgs st) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[kWsMaxRing], empty[kWsMaxRing], acc_full[kStackMaxBlocks], acc_empty[kStackMaxBlocks],
        done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int fail_any;
    __shared__ __align__(16) float s_bias[kStackMaxCout];
    const WsArgs& wa = st.ws;
    const StripArgs& a = wa.s;
    const int ring = st.ring, blocks = st.blocks;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int nkc = a.cin / 8, cout = a.cout;
    const uint32_t w_bytes = 9u * (uint32_t)a.cin * (uint32_t)cout * 2u;
    const uint32_t row_bytes = (uint32_t)wa.row_bytes;
    const uint32_t sw = smem_u32(smem);
    const uint32_t sring = sw + ((w_bytes + 1023u) & ~1023u);
    if (tid == 0) {
        for (int k = 0; k < ring; ++k) {
            mbar_init(smem_u32(&full[k]), 1);
            mbar_init(smem_u32(&empty[k]), 1);
        }
        for (int k = 0; k < blocks; ++k) {
            mbar_init(smem_u32(&acc_full[k]), 1);
            mbar_init(smem_u32(&acc_empty[k]), 4);  // one arrival per epilogue warp
        }
        mbar_init(smem_u32(&done_bar), 1);
        fail_any = 0;
        fence_mbar_init();
    }
    if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), (uint32_t)a.tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    bool fail = false;

    if (warp > 0) {
        // weights: unit (dx, kc, p, co), p = 2 - dy, at (((dx * nkc + kc) * 3 + p) * cout + co) * 16
        for (int q = tid - 32; q < 9 * nkc * cout; q += kStackThreads - 32) {
            const int co = q % cout;
            int rest = q / cout;
            const int p = rest % 3;
            rest /= 3;
            const int kc = rest % nkc, dx = rest / nkc;
            const int t = (2 - p) * 3 + dx;
            cp_async16(sw + (uint32_t)q * 16u, a.w + ((size_t)(st.co0 + co) * 9 + t) * a.cin_total + a.c0 + kc * 8,
                       true);
        }
        for (int c = tid - 32; c < cout; c += kStackThreads - 32) s_bias[c] = a.bias ? a.bias[st.co0 + c] : 0.0f;
        cp_async_commit();
        cp_async_wait<0>();
        fence_proxy_async();
        asm volatile("bar.sync 1, %0;\n" ::"n"(kStackThreads - 32) : "memory");
    }

    if (warp == 0) {
        if (lane == 0) {
            int slot = 0;
            uint32_t phase = 0;
            long issued = 0;
            RowRange range(a.n, a.h, a.xtiles);
            WsSegment g;
            while (!fail && range.next(g)) {
                for (int yy = g.y0 - 1; yy <= g.y1; ++yy) {
                    if (!mbar_wait(smem_u32(&empty[slot]), phase ^ 1u)) {
                        fail = true;
                        break;
                    }
                    const uint32_t dst = sring + (uint32_t)slot * row_bytes;
                    const uint32_t fb = smem_u32(&full[slot]);
                    mbar_arrive_expect_tx(fb, (uint32_t)wa.tx_bytes);
                    for (int k = 0; k < wa.ngroups; ++k) {
                        const CUtensorMap* m = wa.gw[k] == 64 ? &map64 : (wa.gw[k] == 32 ? &map32 : &map16);
                        tma_load_4d(dst + (uint32_t)wa.goff[k], m, a.c0 + wa.gc[k], g.x0 - 1, yy, g.n_img, fb);
                    }
                    ++issued;
                    if (++slot == ring) {
                        slot = 0;
                        phase ^= 1u;
                    }
                }
            }
            // the last loads (one per slot at most) have landed before the CTA can exit
            const long tail = issued < ring ? issued : ring;
            for (long k = 1; k <= tail; ++k) {
                int sl = slot - (int)k;
                uint32_t ph = phase;
                if (sl < 0) {
                    sl += ring;
                    ph ^= 1u;
                }
                if (!mbar_wait(smem_u32(&full[sl]), ph)) fail = true;
            }
        }
    } else if (warp == 1) {
        // descriptor words: A (swizzled, start field added per row / group / dx / step; LBO 1), B (no
        // swizzle, LBO = one 8-channel plane of 3 cout rows, SBO 128)
        const uint32_t n3 = 3u * (uint32_t)cout;
        const uint64_t bd0 = smem_desc(sw, n3 * 16u, 128);
        const uint32_t b_hi = (uint32_t)(bd0 >> 32), b_lo0 = (uint32_t)bd0;
        const uint32_t a_lo1 = 1u << 16;
        const uint32_t b_step = 2u * n3, b_dx = (uint32_t)nkc * n3;
        const uint32_t id1 = instr_desc(kBM, cout, 0, 0);
        const uint32_t id_n = (uint32_t)(cout >> 3) << 17;  // one more block of columns
        const int ngroups = wa.ngroups;
        const uint32_t set_cols = (uint32_t)(blocks * cout);
        const int by_tap = st.by_tap;
        int slot = 0;
        uint32_t phase = 0;
        int blk0 = 0;        // block of the segment's first output row
        uint32_t use0 = 0;   // parity of that block's use count
        RowRange range(a.n, a.h, a.xtiles);
        WsSegment sgm;
        while (!fail && range.next(sgm)) {
            const int rows = sgm.y1 - sgm.y0;
            // block of output rows q - 2 and q, and the use parity of the latter's
            int b2 = blk0, b0 = blk0;
            uint32_t u0 = use0;
            for (int q = 0; q < rows + 2; ++q) {
                const int lo = q < 2 ? 0 : q - 2, hi = min(q, rows - 1);  // output rows that read input row q
                const int blo = q < 2 ? blk0 : b2;                        // block of row lo
                const bool fresh = q < rows;                              // row q starts here
                bool ok = mbar_wait(smem_u32(&full[slot]), phase);
                if (fresh) ok = ok && mbar_wait(smem_u32(&acc_empty[b0]), u0 ^ 1u);
                if (!__all_sync(0xffffffffu, ok)) {
                    fail = true;
                    break;
                }
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t row16 = (sring + (uint32_t)slot * row_bytes) >> 4;
                    const int cnt = hi - lo + 1;
                    const int n_first = min(cnt, blocks - blo);  // columns up to the ring's end, then the rest
                    const int n_rest = cnt - n_first;
                    const uint32_t p0 = (uint32_t)((2 - q + lo) * cout), p_rest = p0 + (uint32_t)(n_first * cout);
                    const uint32_t id_first = id1 + (uint32_t)(n_first - 1) * id_n;
                    const uint32_t id_rest = id1 + (uint32_t)(n_rest - 1) * id_n;
                    // 16-channel steps of a group and a dx; the first of a pass overwrites the new row's accumulator
                    auto steps = [&](uint32_t acc0, int gw, uint32_t ahi, uint32_t aj, uint32_t bj, bool first) {
                        for (int j = 0; j < gw / 16; ++j) {
                            if (first) {  // (the older rows accumulate)
                                first = false;
                                for (int i = lo; i <= hi; ++i) {
                                    const int bi = blo + (i - lo) < blocks ? blo + (i - lo) : blo + (i - lo) - blocks;
                                    mma_bf16_halves(acc0 + (uint32_t)(bi * cout), aj, ahi,
                                                    bj + (uint32_t)((2 - q + i) * cout), b_hi, id1, i < q ? 1u : 0u);
                                }
                            } else {
                                mma_bf16_halves(acc0 + (uint32_t)(blo * cout), aj, ahi, bj + p0, b_hi, id_first, 1u);
                                if (n_rest > 0) mma_bf16_halves(acc0, aj, ahi, bj + p_rest, b_hi, id_rest, 1u);
                            }
                            aj += 2u;
                            bj += b_step;
                        }
                    };
                    if (!by_tap) {
                        for (int k = 0; k < ngroups; ++k) {
                            const int gw = wa.gw[k];
                            const uint32_t ahi = a_hi_of(gw);
                            const uint32_t line16 = (uint32_t)gw >> 3;
                            // a ring of accumulators for each pass
                            const uint32_t acc0 = tmem + (k >= st.groups0 ? set_cols : 0u);
                            const bool first = fresh && (k == 0 || k == st.groups0);
                            const uint32_t al = a_lo1 + row16 + ((uint32_t)wa.goff[k] >> 4);
                            const uint32_t bl = b_lo0 + (uint32_t)(wa.gc[k] >> 3) * n3;
#pragma unroll
                            for (uint32_t dx = 0; dx < 3; ++dx)
                                steps(acc0, gw, ahi, al + dx * line16, bl + dx * b_dx, first && dx == 0);
                        }
                    } else {
                        for (uint32_t dx = 0; dx < 3; ++dx)
                            for (int k = 0; k < ngroups; ++k) {
                                const int gw = wa.gw[k];
                                steps(tmem, gw, a_hi_of(gw),
                                      a_lo1 + row16 + ((uint32_t)wa.goff[k] >> 4) + dx * ((uint32_t)gw >> 3),
                                      b_lo0 + (uint32_t)(wa.gc[k] >> 3) * n3 + dx * b_dx, fresh && dx == 0 && k == 0);
                            }
                    }
                    mma_commit(smem_u32(&empty[slot]));
                    if (q >= 2) mma_commit(smem_u32(&acc_full[b2]));
                }
                __syncwarp();
                if (++slot == ring) {
                    slot = 0;
                    phase ^= 1u;
                }
                if (q >= 2 && ++b2 == blocks) b2 = 0;
                if (fresh && ++b0 == blocks) {
                    b0 = 0;
                    u0 ^= 1u;
                }
            }
            blk0 = b0;
            use0 = u0;
        }
        // every MMA this warp issued has completed before TMEM is released
        if (elect_one()) mma_commit(smem_u32(&done_bar));
        __syncwarp();
        if (!mbar_wait(smem_u32(&done_bar), 0)) fail = true;
    } else {
        // two teams of four warps take the rows alternately; before it waits for its row a warp has the row's
        // ReLU mask on the way
        const int quarter = warp & 3, team = (warp - 2) >> 2;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        int b = 0, turn = 0;
        uint32_t u = 0;
        RowRange range(a.n, a.h, a.xtiles);
        WsSegment sgm;
        while (!fail && range.next(sgm)) {
            const int x = sgm.x0 + quarter * 32 + lane;
            const bool ok = x < a.w_;
            for (int y = sgm.y0; y < sgm.y1; ++y) {
                if (turn == team) {
                    const size_t at = (((size_t)sgm.n_img * a.h + y) * a.w_ + (ok ? x : 0)) * st.cout_total + st.co0;
                    uint4 mask[kStackMaxCout / 8];
                    if (a.mask) {
#pragma unroll
                        for (int k = 0; k < kStackMaxCout / 8; ++k)
                            if (k * 8 < cout) mask[k] = __ldg(reinterpret_cast<const uint4*>(a.mask + at) + k);
                    }
                    const bool full_ok = mbar_wait(smem_u32(&acc_full[b]), u);
                    if (!__all_sync(0xffffffffu, full_ok)) {
                        fail = true;
                        break;
                    }
                    tc_fence_after();
                    stack_epilogue(a, s_bias, tmem + lanes + (uint32_t)(b * cout),
                                   st.groups0 < wa.ngroups ? (uint32_t)(blocks * cout) : 0u, at, ok, mask);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&acc_empty[b]));
                }
                turn ^= 1;
                if (++b == blocks) {
                    b = 0;
                    u ^= 1u;
                }
            }
        }
    }
    if (fail) atomicOr(&fail_any, 1);
    tc_fence_before();
    __syncthreads();
    if (fail_any && tid == 0 && a.err) atomicExch(a.err, (int)VPT_ERR_ITER_LIMIT);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, (uint32_t)a.tmem_cols);
    }
}

// ---------------------------------------------------------------------------------------------
// the convolution on boxes of 128 pixels (TMA-fed tiles)
// ---------------------------------------------------------------------------------------------
// conv_tile_kernel's tiles (128 pixels x up to 256 output channels a CTA, K split over blockIdx.z for small grids) for
// images whose 128 consecutive pixels are a box: widths that divide 128 (whole rows, whole images where they are
// smaller) and multiples of 128.  A stage is one tap and up to 64 input channels: the box moved by (dx, dy), whose
// pixels outside the image arrive as zeros, and the tap's weights, both loaded by the tensor-memory-access unit
// into K-major swizzled lines of `cw` channels, four stages ahead; the gather kernel's threads compute 64 addresses
// and copies each a stage and meet at a barrier for it.  The stages follow the layer's order of products (ConvOrder):
// by tap and channel, or as the row-strip kernels add them, with an accumulator for each pass over the channels.
// Warps: 0 loads, 1 issues, 2-5 the epilogue.  Every wait is bounded, as in conv_ws_kernel.
//   us, gather kernel / here: 96 -> 96 8 images of 64 x 64 33.5 / 15.6, 224 -> 96 71 / 23, 96 -> 224 80 / 31; 128 -> 128
// 8 images of 16 x 16 17.3 / 13.1, one of 4 x 4 12.7 / 8.2; 224 -> 96 one image of 128 x 128 61 / 15.  Bound: the
// stages' bytes from L2 (28 KB for 96 channels) for large grids, the latency of a tile's serial stages for small ones.
constexpr int kBoxThreads = 192;
constexpr int kBoxStages = 4;

struct BoxArgs {
    ConvArgs c;
    int cw;              // channels of a stage: 64, 32 or 16 (a stage may use fewer)
    int bh, bn;          // rows and images of a box
    int passes, pass_ch; // order of the row-strip kernels: passes over pass_ch input channels each (0: by tap and channel)
    int kper;            // by tap: K (= tap * cin + channel) of a split
};

// The stages of a CTA in the layer's order of products.
struct BoxWalk {
    const BoxArgs& b;
    int tap = 0, ci = 0, len = 0;  // the stage: tap, first channel, channels
    int pass = -1;                 // its pass (by tap: 0)
    bool first = false;            // the first of its pass
    int k = 0, kend = 0;           // by tap: K so far, end of the split
    int c = 0, d = 0;              // by pass: channel within the pass, 3 dy + dx

    __device__ __forceinline__ explicit BoxWalk(const BoxArgs& b_) : b(b_) {
        if (b.passes) return;
        k = min((int)blockIdx.z * b.kper, 9 * b.c.cin);
        kend = min(k + b.kper, 9 * b.c.cin);
        tap = k / b.c.cin;
        ci = k - tap * b.c.cin;
    }
    __device__ __forceinline__ bool next() {
        if (!b.passes) {
            ci += len;
            if (ci == b.c.cin) {
                ci = 0;
                ++tap;
            }
            if (k >= kend) return false;
            len = min(min(b.cw, b.c.cin - ci), kend - k);
            k += len;
            first = pass < 0;
            pass = 0;
            return true;
        }
        // dy, channel group (64, then 32, then 16), dx
        int width = min(b.pass_ch, b.c.cin - max(pass, 0) * b.pass_ch);
        first = pass < 0;
        if (first) {
            pass = 0;
        } else if (++d % 3 == 0) {
            c += len;
            if (c < width) {
                d -= 3;
            } else {
                c = 0;
                if (d == 9) {
                    d = 0;
                    if (++pass == b.passes) return false;
                    first = true;
                    width = min(b.pass_ch, b.c.cin - pass * b.pass_ch);
                }
            }
        }
        tap = d;
        ci = pass * b.pass_ch + c;
        len = width - c >= 64 ? 64 : (width - c >= 32 ? 32 : 16);
        return true;
    }
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}

__global__ void __launch_bounds__(kBoxThreads)
    conv_box_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                    const __grid_constant__ BoxArgs b) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[kBoxStages], empty[kBoxStages], done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int fail_any;
    const ConvArgs& a = b.c;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int P = a.n * a.h * a.w_, n0 = blockIdx.y * a.n_tile;
    const uint32_t a_bytes = (uint32_t)(kBM * b.cw * 2), b_bytes = (uint32_t)(a.n_tile * b.cw * 2);
    const uint32_t stage_bytes = a_bytes + ((b_bytes + 1023u) & ~1023u);
    const uint32_t sbase = smem_u32(smem);
    if (tid == 0) {
        for (int k = 0; k < kBoxStages; ++k) {
            mbar_init(smem_u32(&full[k]), 1);
            mbar_init(smem_u32(&empty[k]), 1);
        }
        mbar_init(smem_u32(&done_bar), 1);
        fail_any = 0;
        fence_mbar_init();
    }
    if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), (uint32_t)a.tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    bool fail = false;

    if (warp == 0) {
        if (lane == 0) {
            int img, y0, x0;
            pixel_coords((int)blockIdx.x * kBM, a.h, a.w_, img, y0, x0);
            int slot = 0, issued = 0;
            uint32_t phase = 0;
            BoxWalk g(b);
            while (g.next()) {
                if (!mbar_wait(smem_u32(&empty[slot]), phase ^ 1u)) {
                    fail = true;
                    break;
                }
                const uint32_t dst = sbase + (uint32_t)slot * stage_bytes, fb = smem_u32(&full[slot]);
                mbar_arrive_expect_tx(fb, a_bytes + b_bytes);
                const int dy = g.tap / 3;
                tma_load_4d(dst, &xmap, g.ci, x0 + g.tap - 3 * dy - 1, y0 + dy - 1, img, fb);
                tma_load_3d(dst + a_bytes, &wmap, g.ci, g.tap, n0, fb);
                ++issued;
                if (++slot == kBoxStages) {
                    slot = 0;
                    phase ^= 1u;
                }
            }
            // the last loads (one per slot at most) have landed before the CTA can exit
            for (int k = 1; k <= min(issued, kBoxStages); ++k) {
                int q = slot - k;
                uint32_t ph = phase;
                if (q < 0) {
                    q += kBoxStages;
                    ph ^= 1u;
                }
                if (!mbar_wait(smem_u32(&full[q]), ph)) fail = true;
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc = instr_desc(kBM, a.n_tile, 0, 0), hi = a_hi_of(b.cw), lbo = 1u << 16;
        int slot = 0;
        uint32_t phase = 0;
        BoxWalk g(b);
        while (g.next()) {
            const bool ok = mbar_wait(smem_u32(&full[slot]), phase);
            if (!__all_sync(0xffffffffu, ok)) {
                fail = true;
                break;
            }
            tc_fence_after();
            if (elect_one()) {
                const uint32_t sA = (sbase + (uint32_t)slot * stage_bytes) >> 4;
                const uint32_t al = lbo + sA, bl = lbo + sA + (a_bytes >> 4);
                const uint32_t dacc = tmem + (uint32_t)(g.pass * a.n_tile);
                for (int j = 0; j < g.len / 16; ++j)
                    mma_bf16_halves(dacc, al + 2u * (uint32_t)j, hi, bl + 2u * (uint32_t)j, hi, idesc,
                                    (!g.first || j > 0) ? 1u : 0u);
                mma_commit(smem_u32(&empty[slot]));
            }
            __syncwarp();
            if (++slot == kBoxStages) {
                slot = 0;
                phase ^= 1u;
            }
        }
        // every MMA issued has completed before TMEM is read or released
        if (elect_one()) mma_commit(smem_u32(&done_bar));
        __syncwarp();
        if (!mbar_wait(smem_u32(&done_bar), 0)) fail = true;
    }
    if (fail) atomicOr(&fail_any, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp >= 2 && !fail_any) {
        const int q = warp & 3, p = (int)blockIdx.x * kBM + q * 32 + lane;
        const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16);
        const bool any = b.passes || (int)blockIdx.z * b.kper < 9 * a.cin;
        for (int c0 = 0; c0 < a.n_tile; c0 += 16) {
            float v[16] = {};  // an empty K range contributes zeros
            if (any) tmem_ld16(trow + (uint32_t)c0, v);  // whole warp, uniform
            if (b.passes == 2) {
                float v2[16];
                tmem_ld16(trow + (uint32_t)(a.n_tile + c0), v2);
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] += v2[i];
            }
            if (p < P && n0 + c0 < a.cout) conv_store(a, P, p, n0 + c0, v);
        }
    }
    if (fail_any && tid == 0 && a.err) atomicExch(a.err, (int)VPT_ERR_ITER_LIMIT);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, (uint32_t)a.tmem_cols);
    }
}

// ---------------------------------------------------------------------------------------------
// the weight gradient on image rows
// ---------------------------------------------------------------------------------------------
// dw[co][t][ci] = sum over pixels p of dy[p][co] * x[p + off(t)][ci].  Pixels are K, in steps of 16: a CTA walks
// segments of rows of an image column 128 pixels wide, or the rows of a run of pixels_per_split pixels (of images whose
// width is a multiple of 16, in tiles of 128 from left to right, the first and the last row in part), and sums
// them in TMEM, one after the other.  Both operands are rows as they lie in memory, [pixel][channels], read by the TMA
// into the MN-major swizzled layout (channels contiguous: MN; pixels: K), lines of 32 or 16 channels.  A tap's
// horizontal shift dx is a start moved by dx pixel lines, as in conv_stack_kernel; pixels and channels outside
// arrive as zeros.
//   One tensor (U) is the A operand, M = 64 or 128 of its channels; of the other (S) a chunk of at most 32
// channels is B, of the three rows that meet U's row in the three vertical taps at once: the rows lie in
// consecutive ring slots, so B's channel groups are the slots and one MMA of N = 3 x 32 columns serves
// three taps (two MMAs where the ring wraps).  Accumulators: one block of 3 x 32 columns per dx.
//   role 0: U = x, S = dy (row r of x meets rows r-1, r, r+1 of dy);
//   role 1: U = dy, S = x (row y of dy meets rows y-1, y, y+1 of x).
// The role with fewer passes (U chunks x S chunks, blockIdx.y) is taken.
// Warps: 0 loads (TMA), 1-3 issue the MMAs of dx = 0, 1, 2 (one thread's issue, about 93 cycles an MMA, is the
// bound of N <= 96), 4-7 zero the accumulators at the start and write the CTA's sums to
// partial[blockIdx.x][t * cin + ci][co] at the end (reduced in fixed order by reduce_grads_kernel).  M = 64
// accumulators occupy lanes 0-15 of each 32-lane quarter of TMEM.
//   us, 8 images of 256 x 256 (a strip kernel that copied both rows into 8-channel planes and issued one MMA a tap and
// 16 pixels / here): 96 -> 32 150 / 66, 32 -> 176 289 / 100; at half that size 64 -> 64 58 / 35, 160 -> 64 132 / 72;
// by the gather kernel in runs of pixels / here: 16 -> 32 108 / 41, 32 -> 32 154 / 55, 224 -> 96 at a quarter 123 / 47.
// Bound: the rows' bytes (96 -> 32: 134 MB, 21 us) and the MMAs (24 a row and 28 to 42 rows an SM: the segments are not
// split further, since their rows' order is part of the result), which overlap, then writing the accumulators.
constexpr int kWgThreads = 256;
constexpr int kWgMaxRing = 8;
constexpr int kWgURing = 3;

struct WgradArgs {
    float* partial;  // [gridDim.x][m_pad][cout]
    int* err;
    int n, h, w_, cin, cout, m_pad;
    int role;
    int s_group;               // channels of an S chunk: 32, or 16 when S has 16
    int u_chunks, s_chunks;    // blockIdx.y = u_chunk * s_chunks + s_chunk
    int xtiles, seg_rows, segs_per_col;  // segments of seg_rows rows of a column; CTA i takes i, i + gridDim.x, ...
    int pps;                   // or the run of pixels [i pps, (i + 1) pps) (0: segments)
    int tiles, row_groups;     // 128-pixel tiles and 16-pixel groups of a row of a segment
    int u_slot, u_group_bytes, s_tile, s_slot, s_ring;  // shared-memory strides (an S slot: a row's tiles); ring depth of S
    int u_lines, s_lines;      // pixel lines of a row (the x tensor's rows carry a halo of one)
    int tmem_cols;
};

// rows [y0, y1) of an image from x0; of the first row only the 16-pixel groups from g0 on, of the last those below g1
struct WgSegment {
    int n_img, x0, y0, y1, g0, g1;
};

// the segments of a CTA in order (RUNS: of a run of pixels)
template <bool RUNS>
struct SegWalk {
    const WgradArgs& a;
    long at, end;  // segment, or pixel of the run
    __device__ __forceinline__ explicit SegWalk(const WgradArgs& a_) : a(a_) {
        const long pixels = (long)a.n * a.h * a.w_;
        at = RUNS ? min((long)blockIdx.x * a.pps, pixels) : (long)blockIdx.x;
        end = RUNS ? min(at + a.pps, pixels) : (long)a.n * a.xtiles * a.segs_per_col;
    }
    __device__ __forceinline__ bool next(WgSegment& g) {
        if (at >= end) return false;
        if (RUNS) {  // the rest of the run, or of its image
            const int row = (int)(at / a.w_), img = row / a.h;
            const long stop = min(end, (long)(img + 1) * a.h * a.w_);
            const int last = (int)((stop - 1) / a.w_);
            g.n_img = img;
            g.x0 = 0;
            g.y0 = row - img * a.h;
            g.y1 = last + 1 - img * a.h;
            g.g0 = (int)(at - (long)row * a.w_) / 16;
            g.g1 = (int)(stop - (long)last * a.w_ + 15) / 16;
            at = stop;
            return true;
        }
        const int seg = (int)at, col = seg / a.segs_per_col, part = seg - col * a.segs_per_col;
        g.n_img = col / a.xtiles;
        g.x0 = (col % a.xtiles) * kBM;
        g.y0 = part * a.seg_rows;
        g.y1 = min(a.h, g.y0 + a.seg_rows);
        g.g0 = 0;
        g.g1 = a.row_groups;
        at += gridDim.x;
        return true;
    }
    // the 16-pixel groups [lo, hi) of dy row y that count, within tile t
    __device__ __forceinline__ int2 groups(const WgSegment& g, int y, int t) const {
        const int lo = (y == g.y0 ? g.g0 : 0) - t * (kBM / 16), hi = (y == g.y1 - 1 ? g.g1 : a.row_groups) - t * (kBM / 16);
        return make_int2(max(lo, 0), min(hi, kBM / 16));
    }
};

// MN-major swizzled descriptor: lines of `line` bytes (128 / 64 / 32: 64 / 32 / 16 channels), 8-pixel groups
// 8 lines apart (SBO), channel groups `lbo` bytes apart
__device__ __forceinline__ uint64_t smem_desc_mn(uint32_t line, uint32_t lbo) {
    uint64_t d = (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)(((8u * line) >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)(line == 128 ? 2 : (line == 64 ? 4 : 6)) << 61;
    return d;
}

template <bool RUNS>
__global__ void __launch_bounds__(kWgThreads, 1)
    wgrad_rows_kernel(const __grid_constant__ CUtensorMap umap, const __grid_constant__ CUtensorMap smap,
                      const __grid_constant__ WgradArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t u_full[kWgURing], u_empty[kWgURing], s_full[kWgMaxRing], s_empty[kWgMaxRing], done_bar[3];
    __shared__ uint32_t tmem_slot;
    __shared__ int fail_any;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int u_total = a.role == 0 ? a.cin : a.cout;
    const int u0 = ((int)blockIdx.y / a.s_chunks) * 128, s0 = ((int)blockIdx.y % a.s_chunks) * a.s_group;
    const int ma = u_total - u0 > 64 ? 128 : 64;
    const int n3 = 3 * a.s_group, tiles = RUNS ? a.tiles : 1;
    const uint32_t su = smem_u32(smem), ss = su + (uint32_t)(kWgURing * a.u_slot);
    if (tid == 0) {
        for (int k = 0; k < kWgURing; ++k) {
            mbar_init(smem_u32(&u_full[k]), 1);
            mbar_init(smem_u32(&u_empty[k]), 3);  // one release per issuing warp
        }
        for (int k = 0; k < a.s_ring; ++k) {
            mbar_init(smem_u32(&s_full[k]), 1);
            mbar_init(smem_u32(&s_empty[k]), 3);
        }
        for (int k = 0; k < 3; ++k) mbar_init(smem_u32(&done_bar[k]), 1);
        fail_any = 0;
        fence_mbar_init();
    }
    if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), (uint32_t)a.tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    bool fail = false;
    if (warp >= 4) {
        const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        for (int c = 0; c < 3 * n3; c += 16) tmem_zero16(trow + (uint32_t)c);
        asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
        tc_fence_before();
    }
    if (warp != 0) asm volatile("bar.sync 1, %0;\n" ::"n"(kWgThreads - 32) : "memory");

    // Row order of a segment [y0, y1) (both roles): steps r = first .. last of U's rows; before step r the S
    // rows up to r + 1 are there.  Role 0: r = y0 - 1 .. y1, S rows y0 .. y1 - 1; role 1: r = y0 .. y1 - 1, S
    // rows y0 - 1 .. y1.  An S row is released after the step that follows it.
    if (warp == 0) {
        if (lane == 0) {
            const int ugroups = ma / 32;
            const uint32_t u_tx = (uint32_t)(ugroups * a.u_lines * 64), s_tx = (uint32_t)(tiles * a.s_lines * a.s_group * 2);
            int us = 0, sl = 0;
            uint32_t uph = 0, sph = 0;
            long ui = 0, si = 0;
            auto load_s = [&](const WgSegment& g, int row) {
                if (!mbar_wait(smem_u32(&s_empty[sl]), sph ^ 1u)) {
                    fail = true;
                    return;
                }
                const uint32_t fb = smem_u32(&s_full[sl]);
                mbar_arrive_expect_tx(fb, s_tx);
                for (int t = 0; t < tiles; ++t)
                    tma_load_4d(ss + (uint32_t)(sl * a.s_slot + t * a.s_tile), &smap, s0,
                                g.x0 + t * kBM - (a.role == 1 ? 1 : 0), row, g.n_img, fb);
                ++si;
                if (++sl == a.s_ring) {
                    sl = 0;
                    sph ^= 1u;
                }
            };
            SegWalk<RUNS> range(a);
            WgSegment g;
            while (!fail && range.next(g)) {
                const int r0 = a.role == 0 ? g.y0 - 1 : g.y0, r1 = a.role == 0 ? g.y1 : g.y1 - 1;
                const int slo = a.role == 0 ? g.y0 : g.y0 - 1, shi = a.role == 0 ? g.y1 - 1 : g.y1;
                int next = slo;
                for (int r = r0; r <= r1 && !fail; ++r) {
                    while (next <= min(r + 1, shi) && !fail) load_s(g, next++);
                    for (int t = 0; t < tiles; ++t) {
                        if (fail || !mbar_wait(smem_u32(&u_empty[us]), uph ^ 1u)) {
                            fail = true;
                            break;
                        }
                        const uint32_t fb = smem_u32(&u_full[us]);
                        mbar_arrive_expect_tx(fb, u_tx);
                        for (int k = 0; k < ugroups; ++k)
                            tma_load_4d(su + (uint32_t)(us * a.u_slot + k * a.u_group_bytes), &umap, u0 + 32 * k,
                                        g.x0 + t * kBM - (a.role == 0 ? 1 : 0), r, g.n_img, fb);
                        ++ui;
                        if (++us == kWgURing) {
                            us = 0;
                            uph ^= 1u;
                        }
                    }
                }
            }
            // the last loads (one per slot at most) have landed before the CTA can exit
            for (long k = 1; k <= min(ui, (long)kWgURing); ++k) {
                int q = us - (int)k;
                uint32_t ph = uph;
                if (q < 0) {
                    q += kWgURing;
                    ph ^= 1u;
                }
                if (!mbar_wait(smem_u32(&u_full[q]), ph)) fail = true;
            }
            for (long k = 1; k <= min(si, (long)a.s_ring); ++k) {
                int q = sl - (int)k;
                uint32_t ph = sph;
                if (q < 0) {
                    q += a.s_ring;
                    ph ^= 1u;
                }
                if (!mbar_wait(smem_u32(&s_full[q]), ph)) fail = true;
            }
        }
    } else if (warp <= 3) {
        tc_fence_after();
        const int dx = warp - 1;
        const uint32_t s_line = (uint32_t)a.s_group * 2u;
        const uint64_t ud = smem_desc_mn(64, (uint32_t)a.u_group_bytes), sd = smem_desc_mn(s_line, (uint32_t)a.s_slot);
        const uint32_t u_hi = (uint32_t)(ud >> 32), s_hi = (uint32_t)(sd >> 32);
        // the x tensor's rows start at x0 - 1: its start moves by dx lines
        const uint32_t u_lo = (uint32_t)ud + ((su + (a.role == 0 ? (uint32_t)dx * 64u : 0u)) >> 4);
        const uint32_t s_lo = (uint32_t)sd + ((ss + (a.role == 1 ? (uint32_t)dx * s_line : 0u)) >> 4);
        const uint32_t u_step = 64, s_step = s_line;  // 16 lines, in 16-byte units
        const uint32_t id1 = instr_desc(ma, a.s_group, 1, 1), id_n = (uint32_t)(a.s_group >> 3) << 17;
        const uint32_t dacc = tmem + (uint32_t)(dx * n3);
        int us = 0;
        uint32_t uph = 0;
        int ws = 0;         // ring slot of the oldest S row in use
        uint32_t wph = 0;   // its phase
        SegWalk<RUNS> range(a);
        WgSegment g;
        while (!fail && range.next(g)) {
            const int r0 = a.role == 0 ? g.y0 - 1 : g.y0, r1 = a.role == 0 ? g.y1 : g.y1 - 1;
            const int slo = a.role == 0 ? g.y0 : g.y0 - 1, shi = a.role == 0 ? g.y1 - 1 : g.y1;
            int oldest = slo;  // S row in slot ws
            for (int r = r0; r <= r1 && !fail; ++r) {
                const int lo = max(r - 1, slo), hi = min(r + 1, shi);  // S rows of this step (lo == oldest)
                const int cnt = hi - lo + 1, n_first = min(cnt, a.s_ring - ws), n_rest = cnt - n_first;
                // S row r - 1 is last used here; the segment's last step releases the rest
                const int keep = r == r1 ? shi + 1 : max(r, slo);
                for (int t = 0; t < tiles; ++t) {
                    bool ok = mbar_wait(smem_u32(&u_full[us]), uph);
                    for (int k = 0; t == 0 && k < cnt; ++k) {
                        const int q = ws + k < a.s_ring ? ws + k : ws + k - a.s_ring;
                        ok = ok && mbar_wait(smem_u32(&s_full[q]), ws + k < a.s_ring ? wph : wph ^ 1u);
                    }
                    if (!__all_sync(0xffffffffu, ok)) {
                        fail = true;
                        break;
                    }
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t d0 = dacc + (uint32_t)((lo - (r - 1)) * a.s_group);
                        const uint32_t ub = u_lo + ((uint32_t)(us * a.u_slot) >> 4);
                        const uint32_t wrap = s_lo + ((uint32_t)(t * a.s_tile) >> 4);  // ring slot 0
                        const uint32_t sb = wrap + ((uint32_t)(ws * a.s_slot) >> 4);
                        const uint32_t d1 = d0 + (uint32_t)(n_first * a.s_group);
                        const uint32_t id_first = id1 + (uint32_t)(n_first - 1) * id_n;
                        const uint32_t id_rest = id1 + (uint32_t)(n_rest - 1) * id_n;
                        // the groups of the rows' dy that count: of row r, or (role 0) of each S row its own
                        int2 j0 = make_int2(0, kBM / 16);
                        bool same = true;
                        if (RUNS) {
                            j0 = range.groups(g, a.role == 1 ? r : lo, t);
                            if (a.role == 0) {
                                const int2 jm = range.groups(g, min(lo + 1, hi), t), j2 = range.groups(g, hi, t);
                                same = j0.x == jm.x && j0.y == jm.y && j0.x == j2.x && j0.y == j2.y;
                            }
                        }
                        if (same && j0.x == 0 && j0.y == kBM / 16) {
                            uint32_t ul = ub, sl = sb, sw = wrap;
                            for (int j = 0; j < kBM / 16; ++j) {
                                mma_bf16_halves(d0, ul, u_hi, sl, s_hi, id_first, 1u);
                                if (n_rest > 0) mma_bf16_halves(d1, ul, u_hi, sw, s_hi, id_rest, 1u);
                                ul += u_step;
                                sl += s_step;
                                sw += s_step;
                            }
                        } else if (same) {
                            for (uint32_t j = (uint32_t)j0.x; (int)j < j0.y; ++j) {
                                mma_bf16_halves(d0, ub + j * u_step, u_hi, sb + j * s_step, s_hi, id_first, 1u);
                                if (n_rest > 0)
                                    mma_bf16_halves(d1, ub + j * u_step, u_hi, wrap + j * s_step, s_hi, id_rest, 1u);
                            }
                        } else {  // around the ends of a run
                            for (int k = 0; k < cnt; ++k) {
                                const int2 jk = range.groups(g, lo + k, t);
                                const int q = ws + k < a.s_ring ? ws + k : ws + k - a.s_ring;
                                const uint32_t sk = wrap + ((uint32_t)(q * a.s_slot) >> 4);
                                for (uint32_t j = (uint32_t)jk.x; (int)j < jk.y; ++j)
                                    mma_bf16_halves(d0 + (uint32_t)(k * a.s_group), ub + j * u_step, u_hi, sk + j * s_step,
                                                    s_hi, id1, 1u);
                            }
                        }
                        mma_commit(smem_u32(&u_empty[us]));
                        if (t == tiles - 1)
                            for (int k = 0; k < keep - oldest; ++k)
                                mma_commit(smem_u32(&s_empty[ws + k < a.s_ring ? ws + k : ws + k - a.s_ring]));
                    }
                    __syncwarp();
                    if (++us == kWgURing) {
                        us = 0;
                        uph ^= 1u;
                    }
                }
                for (; oldest < keep; ++oldest)
                    if (++ws == a.s_ring) {
                        ws = 0;
                        wph ^= 1u;
                    }
            }
        }
        // every MMA this warp issued has completed before TMEM is read or released
        if (elect_one()) mma_commit(smem_u32(&done_bar[dx]));
        __syncwarp();
        if (!mbar_wait(smem_u32(&done_bar[dx]), 0)) fail = true;
    }
    if (fail) atomicOr(&fail_any, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp >= 4 && !fail_any) {
        const int q = warp & 3;
        const int row = ma == 128 ? q * 32 + lane : (lane < 16 ? q * 16 + lane : -1);
        const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16);
        const int s_total = a.role == 0 ? a.cout : a.cin;
        const bool ok = row >= 0 && u0 + row < u_total;
        float* part = a.partial + (size_t)blockIdx.x * a.m_pad * a.cout;
        for (int dx = 0; dx < 3; ++dx)
            for (int p = 0; p < 3; ++p) {
                const int t = (a.role == 0 ? 2 - p : p) * 3 + dx;
                for (int c = 0; c < a.s_group; c += 16) {
                    float v[16];
                    tmem_ld16(trow + (uint32_t)(dx * n3 + p * a.s_group + c), v);  // whole warp, uniform
                    if (!ok || s0 + c >= s_total) continue;  // (channel counts are multiples of 16)
                    if (a.role == 0) {
                        float4* dst = reinterpret_cast<float4*>(part + (size_t)(t * a.cin + u0 + row) * a.cout + s0 + c);
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            part[(size_t)(t * a.cin + s0 + c + i) * a.cout + u0 + row] = v[i];
                    }
                }
            }
    }
    if (fail_any && tid == 0 && a.err) atomicExch(a.err, (int)VPT_ERR_ITER_LIMIT);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, (uint32_t)a.tmem_cols);
    }
}

// ---------------------------------------------------------------------------------------------
// small kernels around the convolutions (NHWC bf16, 8 channels = 16 bytes per thread)
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void load8(const bf16* p, float (&f)[8]) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 t = __bfloat1622float2(b[i]);
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
    }
}
__device__ __forceinline__ void store8(bf16* p, const float (&f)[8]) {
    uint4 u;
    __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) b[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = u;
}

// wrot[ci][t][co] = w[co][8 - t][ci]
__global__ void rotate_weights_kernel(const bf16* __restrict__ w, bf16* __restrict__ wrot, int cin, int cout) {
    const int total = cout * 9 * cin;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int ci = i % cin, t = (i / cin) % 9, co = i / (9 * cin);
        wrot[((size_t)ci * 9 + (8 - t)) * cout + co] = w[i];
    }
}

// 2x2 average pooling, [n][h][w][c] -> [n][h/2][w/2][c]
template <class I>
__global__ void pool2_kernel(const bf16* __restrict__ in, bf16* __restrict__ out, int n, int h, int w, int c) {
    const int ho = h / 2, wo = w / 2, c8 = c / 8;
    const I total = (I)n * ho * wo * c8;
    for (I i = (I)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const I pix = i / (I)c8;
        const int cc = (int)(i - pix * c8) * 8;
        const I row = pix / (I)wo, img = row / (I)ho;
        const int x = (int)(pix - row * wo), y = (int)(row - img * ho), b = (int)img;
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int dy = 0; dy < 2; ++dy)
            for (int dx = 0; dx < 2; ++dx) {
                float f[8];
                load8(in + (((size_t)b * h + 2 * y + dy) * w + 2 * x + dx) * c + cc, f);
#pragma unroll
                for (int k = 0; k < 8; ++k) acc[k] += f[k];
            }
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] *= 0.25f;
        store8(out + (size_t)pix * c + cc, acc);
    }
}

// out[n][y][x] = (lo[n][y/2][x/2] (ca channels), skip[n][y][x] (cs channels)): nearest upsampling
// of the coarser level concatenated with the skip connection
template <class I>
__global__ void upcat_kernel(const bf16* __restrict__ lo, const bf16* __restrict__ skip, bf16* __restrict__ out,
                             int n, int h, int w, int ca, int cs) {
    const int c = ca + cs, c8 = c / 8;
    const I total = (I)n * h * w * c8;
    for (I i = (I)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const I pix = i / (I)c8;
        const int cc = (int)(i - pix * c8) * 8;
        const I row = pix / (I)w, img = row / (I)h;
        const int x = (int)(pix - row * w), y = (int)(row - img * h), b = (int)img;
        const uint4* src;
        if (cc < ca)
            src = reinterpret_cast<const uint4*>(lo + (((size_t)b * (h / 2) + y / 2) * (w / 2) + x / 2) * ca + cc);
        else
            src = reinterpret_cast<const uint4*>(skip + (size_t)pix * cs + (cc - ca));
        *reinterpret_cast<uint4*>(out + (size_t)pix * c + cc) = *src;
    }
}

// backward of upcat for the coarse part: dlo[n][y][x][k] = (lo > 0) * sum of the 2x2 children's
// gradient d[.][k] (k < ca); lo is the coarse level's ReLU output
template <class I>
__global__ void upcat_grad_lo_kernel(const bf16* __restrict__ d, const bf16* __restrict__ lo, bf16* __restrict__ dlo,
                                     int n, int h, int w, int ca, int cs) {
    const int ho = h / 2, wo = w / 2, c = ca + cs, c8 = ca / 8;
    const I total = (I)n * ho * wo * c8;
    for (I i = (I)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const I pix = i / (I)c8;
        const int cc = (int)(i - pix * c8) * 8;
        const I row = pix / (I)wo, img = row / (I)ho;
        const int x = (int)(pix - row * wo), y = (int)(row - img * ho), b = (int)img;
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int dy = 0; dy < 2; ++dy)
            for (int dx = 0; dx < 2; ++dx) {
                float f[8];
                load8(d + (((size_t)b * h + 2 * y + dy) * w + 2 * x + dx) * c + cc, f);
#pragma unroll
                for (int k = 0; k < 8; ++k) acc[k] += f[k];
            }
        float m[8];
        load8(lo + (size_t)pix * ca + cc, m);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = m[k] > 0.0f ? acc[k] : 0.0f;
        store8(dlo + (size_t)pix * ca + cc, acc);
    }
}

// gradient at an encoder level's ReLU output e (c channels): the skip part of the decoder's
// concatenated gradient (d_cat[p][cat_off + k], row stride cat_c; may be null) plus the pooled
// branch's gradient d_pool[n][y/2][x/2][k] / 4 (may be null), times (e > 0)
template <class I>
__global__ void encoder_grad_kernel(const bf16* __restrict__ d_cat, int cat_c, int cat_off,
                                    const bf16* __restrict__ d_pool, const bf16* __restrict__ e,
                                    bf16* __restrict__ out, int n, int h, int w, int c) {
    const int c8 = c / 8;
    const I total = (I)n * h * w * c8;
    for (I i = (I)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const I pix = i / (I)c8;
        const int cc = (int)(i - pix * c8) * 8;
        const I row = pix / (I)w, img = row / (I)h;
        const int x = (int)(pix - row * w), y = (int)(row - img * h), b = (int)img;
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0}, f[8];
        if (d_cat) {
            load8(d_cat + (size_t)pix * cat_c + cat_off + cc, f);
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] += f[k];
        }
        if (d_pool) {
            load8(d_pool + (((size_t)b * (h / 2) + y / 2) * (w / 2) + x / 2) * c + cc, f);
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] += 0.25f * f[k];
        }
        load8(e + (size_t)pix * c + cc, f);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = f[k] > 0.0f ? acc[k] : 0.0f;
        store8(out + (size_t)pix * c + cc, acc);
    }
}

// per-block column sums of dy [P][c] (bias gradient, first pass): partial[block][c]
__global__ void bias_grad_kernel(const bf16* __restrict__ dy, float* __restrict__ partial, int P, int c) {
    extern __shared__ float red[];  // [blockDim.x / c8 groups][c]
    const int c8 = c / 8;
    const int lane_c = threadIdx.x % c8, group = threadIdx.x / c8, groups = blockDim.x / c8;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (group < groups) {
        // eight loads at a time (with one, two blocks an SM keep 8 KB in flight; the sums' order does not change): the
        // 19 layers of a training step of 8 images of 256 x 256 144 -> 128 us
        const long step = (long)gridDim.x * groups;
        const bf16* src = dy + lane_c * 8;
        long p = (long)blockIdx.x * groups + group;
        for (; p + 7 * step < P; p += 8 * step) {
            float f[8][8];
#pragma unroll
            for (int u = 0; u < 8; ++u) load8(src + (p + u * step) * c, f[u]);
#pragma unroll
            for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int k = 0; k < 8; ++k) acc[k] += f[u][k];
        }
        for (; p < P; p += step) {
            float f[8];
            load8(src + p * c, f);
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] += f[k];
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) red[group * c + lane_c * 8 + k] = acc[k];
    }
    __syncthreads();
    for (int j = threadIdx.x; j < c; j += blockDim.x) {
        float s = 0.0f;
        for (int g = 0; g < groups; ++g) s += red[g * c + j];
        partial[(size_t)blockIdx.x * c + j] = s;
    }
}

// gradient of one layer into the flat fp32 gradient: g[co][t][ci] = sum_s wpart[s][t*cin+ci][co] and
// gb[co] = sum_b bpart[b][co], every sum one after the other from the first partial to the last.  The loads are whole
// lines, by the partials' own order (by the gradient's, ci fastest, they took a sector per lane).  A thread adds its own
// element's partials, 16 loads in flight, where the layer has an element for every lane of 128 blocks; below that, and
// for the biases, the eight warps of a block have 16 partials each of the same 32 elements on the way and put them into
// shared memory, where the first warp adds them while the next ones arrive.  Bound: the partials' bytes.  The
// 19 layers of a training step of 8 images of 256 x 256: 457 us by the gradient's order, 160 here (most of it
// the launches' 8 us each); all layers through shared memory 216.
constexpr int kReduceChunk = 128;  // partials in shared memory

__host__ __device__ constexpr bool reduce_shared(int splits, int nw) { return splits >= 8 && nw < 32768; }

__global__ void __launch_bounds__(256) reduce_grads_kernel(const float* __restrict__ wpart, int splits, int m_pad,
                                                           int cin, int cout, const float* __restrict__ bpart,
                                                           int bblocks, float* __restrict__ gw,
                                                           float* __restrict__ gb) {
    __shared__ float part[kReduceChunk][32];
    const int nw = cout * 9 * cin;  // a multiple of 256
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the blocks of the weights; then 32 biases a block
    const int wblocks = reduce_shared(splits, nw) ? nw / 32 : nw / 256;
    const bool weight = (int)blockIdx.x < wblocks;
    const bool own = weight && !reduce_shared(splits, nw);  // a thread's element is its own
    const int j = own ? (int)blockIdx.x * 256 + (int)threadIdx.x : ((int)blockIdx.x - (weight ? 0 : wblocks)) * 32 + lane;
    const float* src = weight ? wpart + j : bpart + j;
    const size_t stride = weight ? (size_t)m_pad * cout : (size_t)cout;
    const bool in = weight || j < cout;
    const int count = weight ? splits : (bpart ? bblocks : 0);
    float s = 0.0f;
    if (own) {
#pragma unroll 16
        for (int k = 0; k < count; ++k) s += __ldg(src + (size_t)k * stride);
    } else {
        constexpr int kMine = kReduceChunk / 8;
        float v[kMine];
        auto load = [&](int k0) {
#pragma unroll
            for (int i = 0; i < kMine; ++i) {
                const int k = k0 + 8 * i + warp;
                v[i] = in && k < count ? __ldg(src + (size_t)k * stride) : 0.0f;
            }
        };
        load(0);
        for (int k0 = 0; k0 < count; k0 += kReduceChunk) {
#pragma unroll
            for (int i = 0; i < kMine; ++i) part[8 * i + warp][lane] = v[i];
            __syncthreads();
            if (k0 + kReduceChunk < count) load(k0 + kReduceChunk);
            if (warp == 0) {
                const int n = min(kReduceChunk, count - k0);
#pragma unroll 8
                for (int k = 0; k < n; ++k) s += part[k][lane];
            }
            __syncthreads();
        }
        if (warp > 0) return;
    }
    if (weight) {
        const int m = j / cout, co = j - m * cout;  // m = t * cin + ci
        gw[(size_t)co * 9 * cin + m] = s;
    } else if (j < cout) {
        gb[j] = s;
    }
}

// Adam (Kingma & Ba 2015, Algorithm 1) on the flat fp32 master parameters; the bf16 copy the
// convolutions read is written in the same pass
__global__ void adam_kernel(float* __restrict__ param, bf16* __restrict__ param_bf16, float* __restrict__ m1,
                            float* __restrict__ m2, const float* __restrict__ grad, long count, float lr, float beta1,
                            float beta2, float eps, float bias1, float bias2, float grad_scale) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < count; i += (long)gridDim.x * blockDim.x) {
        const float g = grad[i] * grad_scale;
        const float a = beta1 * m1[i] + (1.0f - beta1) * g;
        const float b = beta2 * m2[i] + (1.0f - beta2) * g * g;
        m1[i] = a;
        m2[i] = b;
        const float mhat = a / bias1, vhat = b / bias2;
        const float p = param[i] - lr * mhat / (sqrtf(vhat) + eps);
        param[i] = p;
        if (param_bf16) param_bf16[i] = __float2bfloat16_rn(p);
    }
}

__global__ void f32_to_bf16_kernel(const float* __restrict__ in, bf16* __restrict__ out, long count) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < count; i += (long)gridDim.x * blockDim.x)
        out[i] = __float2bfloat16_rn(in[i]);
}

// ---------------------------------------------------------------------------------------------
// network input and the kernel-prediction head
// ---------------------------------------------------------------------------------------------
constexpr int kInputChannels = 16;  // 15 used: log radiance 3, albedo 3, normal 3, depth 1, transmittance 1,
                                    // noise level 1, log standard error of the pixel mean 3

// planes: [n][3][h][w] radiance (mean of the frames rendered so far), albedo [n][3][h][w], normal
// [n][3][h][w], depth [n][h][w], transmittance [n][h][w] (each may be null -> zeros); noise_level
// [n] (1 / sqrt(frames) of each image; may be null -> zeros); second_moment [n][3][h][w] (mean of the
// squared per-frame radiance; with noise_level gives log1p of the standard error of the pixel mean,
// sqrt(max(0, m2 - mean^2)) / sqrt(frames); may be null -> zeros)
__global__ void pack_input_kernel(const float* __restrict__ radiance, const float* __restrict__ albedo,
                                  const float* __restrict__ normal, const float* __restrict__ depth,
                                  const float* __restrict__ transmittance, const float* __restrict__ noise_level,
                                  const float* __restrict__ second_moment, bf16* __restrict__ out, int n, int h,
                                  int w) {
    const long plane = (long)h * w, total = (long)n * plane;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const long b = i / plane, q = i % plane;
        float f[16] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int c = 0; c < 3; ++c) {
            const float r = radiance[(b * 3 + c) * plane + q];
            f[c] = log1pf(fmaxf(r, 0.0f));
            if (albedo) f[3 + c] = albedo[(b * 3 + c) * plane + q];
            if (normal) f[6 + c] = normal[(b * 3 + c) * plane + q];
        }
        if (depth) f[9] = depth[b * plane + q];
        if (transmittance) f[10] = transmittance[b * plane + q];
        if (noise_level) {
            f[11] = noise_level[b];
            if (second_moment)
                for (int c = 0; c < 3; ++c) {
                    const float m1 = radiance[(b * 3 + c) * plane + q];
                    const float m2 = second_moment[(b * 3 + c) * plane + q];
                    f[12 + c] = log1pf(sqrtf(fmaxf(0.0f, m2 - m1 * m1)) * noise_level[b]);
                }
        }
        float lo[8], hi[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            lo[k] = f[k];
            hi[k] = f[8 + k];
        }
        store8(out + i * kInputChannels, lo);
        store8(out + i * kInputChannels + 8, hi);
    }
}

// Per-pixel k x k kernel application with the tap softmax fused, and (target != null) the relative
// MSE loss and its gradient with respect to the logits:
//   s = softmax(logits[p][0 .. k*k-1]);  d[c][p] = sum_j s_j x[c][p + off_j]  (taps outside skipped)
//   loss = sum_{p,c} (d - t)^2 / (t^2 + eps) * inv_count
//   dL/dlogit_j = s_j (g . x_j - g . d),  g_c = 2 (d_c - t_c) / (t_c^2 + eps) * inv_count
// logits: [P][hc] fp32 (NHWC, hc >= k*k a multiple of 8, channels k*k.. unused, their gradient 0);
// x, t, out: [n][3][h][w] fp32.  The softmax is recomputed per pass (no per-tap arrays in registers).
// One block per 64-pixel row segment at a time (grid-stride): the segment's logits (contiguous in
// NHWC) are staged in shared memory by asynchronous copies, a warp per pixel row, at a row stride of
// hc + 4 floats; the KS x (64 + KS - 1) radiance window likewise, with zeros outside the image (an
// out-of-image tap adds to the normalisation only).  Four lanes per pixel take the kernel rows
// sub, sub + 4, ... (columns unrolled: window offsets are immediates) and combine by shuffles.  Bank
// spread: the logit stride is 4 (mod 8) with an odd quotient, so the warp's 8 pixels start on banks
// 0, 4, .., 28 and the lanes' rows (KS odd) add 0..3; the window row length is 8 (mod 16), so the
// lanes' window rows start 8 banks apart.  The logit gradients overwrite the staged logits and leave
// as coalesced bf16 rows.
constexpr int kHeadSeg = 64;

__host__ __device__ constexpr int head_window_row(int ks) {  // >= kHeadSeg + ks - 1, = 8 (mod 16)
    return (kHeadSeg + ks - 1 + 7) / 16 * 16 + 8;
}

__device__ __forceinline__ float quad_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

template <int KS>
__global__ void __launch_bounds__(256) kpn_head_kernel(const float* __restrict__ logits, int hc,
                                                       const float* __restrict__ x, const float* __restrict__ target,
                                                       float* __restrict__ out, bf16* __restrict__ dlogits,
                                                       float* __restrict__ loss_partial, int n, int h, int w,
                                                       float eps, float inv_count) {
    constexpr int RW = head_window_row(KS), WIN = KS * RW, TAPS = KS * KS, RAD = KS / 2;
    extern __shared__ float hsm[];
    const int stride = hc + 4;
    float* lsm = hsm;                       // [kHeadSeg][stride]
    float* rsm = hsm + kHeadSeg * stride;   // [3][KS][RW]
    const long plane = (long)h * w;
    const int segs_w = (w + kHeadSeg - 1) / kHeadSeg;
    const long nseg = (long)n * h * segs_w;
    const int t = threadIdx.x, pl = t >> 2, sub = t & 3, warp = t >> 5, lane = t & 31;
    const int q4 = hc / 4;
    float local = 0.0f;
    for (long sg = blockIdx.x; sg < nseg; sg += gridDim.x) {
        const int sx = (int)(sg % segs_w);
        const long row = sg / segs_w;
        const int y = (int)(row % h);
        const long b = row / h;
        const int x0 = sx * kHeadSeg, np = min(kHeadSeg, w - x0);
        const long p0 = (b * h + y) * w + x0;
        __syncthreads();  // the previous segment is done with shared memory
        // asynchronous copies: every copy of the block is in flight before the first wait
        const float4* lg4 = reinterpret_cast<const float4*>(logits + p0 * hc);
        for (int p = warp; p < np; p += 8) {
            const float4* src = lg4 + (long)p * q4;
            const uint32_t dst = smem_u32(lsm + p * stride);
            for (int c = lane; c < q4; c += 32) cp_async16_stream(dst + 16 * c, src + c);
        }
        const float* xb = x + b * 3 * plane;
        for (int rr = warp; rr < 3 * KS; rr += 8) {  // window row rr = c * KS + r
            const int c = rr / KS, r = rr - c * KS;
            const int yy = y + r - RAD;
            const bool row_ok = yy >= 0 && yy < h;
            const float* src = xb + c * plane + (long)(row_ok ? yy : 0) * w;
            const uint32_t dst = smem_u32(rsm + rr * RW);
            for (int xx = lane; xx < kHeadSeg + KS - 1; xx += 32) {
                const int xq = x0 + xx - RAD;
                const bool v = row_ok && xq >= 0 && xq < w;
                cp_async4(dst + 4 * xx, v ? src + xq : xb, v);
            }
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        const bool pv = pl < np;
        const float* lp = lsm + pl * stride;
        const float* rp = rsm + pl;
        float mx = -INFINITY;
        if (pv)
            for (int r = sub; r < KS; r += 4) {
#pragma unroll
                for (int c = 0; c < KS; ++c) mx = fmaxf(mx, lp[r * KS + c]);
            }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        float sum = 0.0f, d0 = 0.0f, d1 = 0.0f, d2 = 0.0f;
        if (pv)
            for (int r = sub; r < KS; r += 4) {
                const float* lr = lp + r * KS;
                const float* xr = rp + r * RW;
#pragma unroll
                for (int c = 0; c < KS; ++c) {
                    const float e = __expf(lr[c] - mx);
                    sum += e;
                    d0 += e * xr[c];
                    d1 += e * xr[WIN + c];
                    d2 += e * xr[2 * WIN + c];
                }
            }
        sum = quad_sum(sum);
        d0 = quad_sum(d0);
        d1 = quad_sum(d1);
        d2 = quad_sum(d2);
        const float inv = 1.0f / sum;
        const float d[3] = {d0 * inv, d1 * inv, d2 * inv};
        const long q = (long)y * w + x0 + pl;
        if (pv && out && sub < 3) out[(b * 3 + sub) * plane + q] = sub == 0 ? d[0] : (sub == 1 ? d[1] : d[2]);
        if (target) {
            float g[3] = {0.0f, 0.0f, 0.0f};
            if (pv) {
                for (int c = 0; c < 3; ++c) {
                    const float tg = target[(b * 3 + c) * plane + q];
                    const float den = tg * tg + eps;
                    const float e = d[c] - tg;
                    if (sub == 0) local += e * e / den * inv_count;
                    g[c] = 2.0f * e / den * inv_count;
                }
            }
            const float gd = g[0] * d[0] + g[1] * d[1] + g[2] * d[2];
            float* lw = lsm + pl * stride;
            for (int r = sub; r < KS; r += 4) {
                float* lr = lw + r * KS;
                const float* xr = rp + r * RW;
#pragma unroll
                for (int c = 0; c < KS; ++c) {
                    const float gx = g[0] * xr[c] + g[1] * xr[WIN + c] + g[2] * xr[2 * WIN + c];
                    lr[c] = pv ? __expf(lr[c] - mx) * inv * (gx - gd) : 0.0f;
                }
            }
            for (int j = TAPS + sub; j < hc; j += 4) lw[j] = 0.0f;
            __syncthreads();
            for (int p = warp; p < np; p += 8) {
                const float* srow = lsm + p * stride;
                bf16* drow = dlogits + (p0 + p) * hc;
                for (int c = lane * 8; c < hc; c += 256) {
                    const float4 u = *reinterpret_cast<const float4*>(srow + c);
                    const float4 v = *reinterpret_cast<const float4*>(srow + c + 4);
                    const float f[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
                    store8(drow + c, f);
                }
            }
        }
    }
    if (loss_partial) {
        // block reduction (fixed order)
        __shared__ float red[256];
        red[threadIdx.x] = local;
        __syncthreads();
        for (int st = blockDim.x / 2; st > 0; st >>= 1) {
            if ((int)threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
            __syncthreads();
        }
        if (threadIdx.x == 0) loss_partial[blockIdx.x] = red[0];
    }
}

// ---------------------------------------------------------------------------------------------
// multi-scale reconstruction
// ---------------------------------------------------------------------------------------------
// Level l (l = 0 full resolution) has the noisy input x_l (x_{l+1} = 2x2 average of x_l), its kernel
// output d_l = apply(x_l, K_l), and the reconstruction
//     c_l = d_l + a_l * (up(c_{l+1}) - up(pool(d_l))),   a_l = sigmoid(logit_l[alpha channel])
// (the coarsest level: c = d): the low frequencies of the fine estimate are replaced, in the
// proportion a, by the coarser level's estimate.  up = nearest (each coarse pixel to its 2x2
// children), pool = 2x2 average.  Images are planar [n][3][h][w] fp32; logits NHWC [p][hc] fp32.
__device__ __forceinline__ float sigmoidf_(float v) { return 1.0f / (1.0f + __expf(-v)); }

__global__ void kpn_combine_kernel(const float* __restrict__ d, const float* __restrict__ c_coarse,
                                   const float* __restrict__ logits, int hc, int alpha_ch, float* __restrict__ c,
                                   int n, int h, int w) {
    const long plane = (long)h * w, total = (long)n * plane;
    const int hh = h / 2, wh = w / 2;
    const long cplane = (long)hh * wh;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const long b = i / plane, q = i % plane;
        const int y = (int)(q / w), x = (int)(q % w);
        const int y0 = y & ~1, x0 = x & ~1;
        const float a = sigmoidf_(logits[i * hc + alpha_ch]);
        for (int ch = 0; ch < 3; ++ch) {
            const float* dp = d + (b * 3 + ch) * plane;
            const float pool = 0.25f * ((dp[(long)y0 * w + x0] + dp[(long)y0 * w + x0 + 1]) +
                                        (dp[(long)(y0 + 1) * w + x0] + dp[(long)(y0 + 1) * w + x0 + 1]));
            const float cc = c_coarse[(b * 3 + ch) * cplane + (long)(y / 2) * wh + x / 2];
            c[(b * 3 + ch) * plane + q] = dp[q] + a * (cc - pool);
        }
    }
}

// Backward of one level.  g = dL/dc_l is read from g_in, or (level 0, target != null) computed here
// from the relative-MSE loss of c = c_l against the target (whose partial sums go to loss_partial).
// With a blend (alpha_ch >= 0): dL/dd = g - pool^T(up^T(a g)) (each pixel minus a quarter of its
// 2x2 family's sum of a g), dL/dc_{l+1} = up^T(a g) (written by the family's first pixel),
// dL/dlogit_alpha = a (1 - a) g . (up(c_{l+1}) - up(pool(d))); without: dL/dd = g.  Then the kernel
// application's gradient dL/dlogit_j = s_j (gd . x_j - gd . d) (taps outside skipped), all written
// to dlogits [p][hc] bf16 (0 in unused channels).
__global__ void kpn_level_grad_kernel(const float* __restrict__ logits, int hc, int ks, int alpha_ch,
                                      const float* __restrict__ x, const float* __restrict__ d,
                                      const float* __restrict__ c_coarse, const float* __restrict__ g_in,
                                      const float* __restrict__ c_out, const float* __restrict__ target, float eps,
                                      float inv_count, bf16* __restrict__ dlogits, float* __restrict__ g_coarse,
                                      float* __restrict__ loss_partial, int n, int h, int w) {
    const long plane = (long)h * w, total = (long)n * plane;
    const int taps = ks * ks, rad = ks / 2;
    const int hh = h / 2, wh = w / 2;
    const long cplane = (long)hh * wh;
    float local = 0.0f;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const long b = i / plane, q = i % plane;
        const int y = (int)(q / w), xx = (int)(q % w);
        // gradient at c for a pixel of this image
        auto g_at = [&](long qq, int ch) -> float {
            if (target) {
                const float t = target[(b * 3 + ch) * plane + qq];
                return 2.0f * (c_out[(b * 3 + ch) * plane + qq] - t) / (t * t + eps) * inv_count;
            }
            return g_in[(b * 3 + ch) * plane + qq];
        };
        float g[3], gd[3];
        for (int ch = 0; ch < 3; ++ch) g[ch] = g_at(q, ch);
        if (target) {
            for (int ch = 0; ch < 3; ++ch) {
                const float t = target[(b * 3 + ch) * plane + q];
                const float e = c_out[(b * 3 + ch) * plane + q] - t;
                local += e * e / (t * t + eps) * inv_count;
            }
        }
        float dalpha = 0.0f;
        bool has_alpha = alpha_ch >= 0;
        if (has_alpha) {
            const int y0 = y & ~1, x0 = xx & ~1;
            const long fam[4] = {(long)y0 * w + x0, (long)y0 * w + x0 + 1, (long)(y0 + 1) * w + x0,
                                 (long)(y0 + 1) * w + x0 + 1};
            const long base = i - q;  // first pixel of this image in NHWC order
            float sag[3] = {0.0f, 0.0f, 0.0f};
            for (int k = 0; k < 4; ++k) {
                const float ak = sigmoidf_(logits[(base + fam[k]) * hc + alpha_ch]);
                for (int ch = 0; ch < 3; ++ch) sag[ch] += ak * g_at(fam[k], ch);
            }
            const float a = sigmoidf_(logits[i * hc + alpha_ch]);
            const long parent = (long)(y / 2) * wh + xx / 2;
            for (int ch = 0; ch < 3; ++ch) {
                gd[ch] = g[ch] - 0.25f * sag[ch];
                const float* dp = d + (b * 3 + ch) * plane;
                const float pool = 0.25f * ((dp[fam[0]] + dp[fam[1]]) + (dp[fam[2]] + dp[fam[3]]));
                dalpha += g[ch] * (c_coarse[(b * 3 + ch) * cplane + parent] - pool);
            }
            dalpha *= a * (1.0f - a);
            if (g_coarse && (y & 1) == 0 && (xx & 1) == 0)
                for (int ch = 0; ch < 3; ++ch) g_coarse[(b * 3 + ch) * cplane + parent] = sag[ch];
        } else {
            for (int ch = 0; ch < 3; ++ch) gd[ch] = g[ch];
        }
        // kernel application backward
        const float* lg = logits + i * hc;
        float mx = -INFINITY;
        for (int j = 0; j < taps; ++j) mx = fmaxf(mx, lg[j]);
        float sum = 0.0f;
        for (int j = 0; j < taps; ++j) sum += __expf(lg[j] - mx);
        const float inv = 1.0f / sum;
        const float* xb = x + b * 3 * plane;
        const float gdd = gd[0] * d[(b * 3 + 0) * plane + q] + gd[1] * d[(b * 3 + 1) * plane + q] +
                          gd[2] * d[(b * 3 + 2) * plane + q];
        for (int j0 = 0; j0 < hc; j0 += 8) {
            float f[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int j = j0 + k;
                f[k] = 0.0f;
                if (j < taps) {
                    const float sj = __expf(lg[j] - mx) * inv;
                    const int yy = y + j / ks - rad, xq = xx + j % ks - rad;
                    float gx = 0.0f;
                    if (yy >= 0 && yy < h && xq >= 0 && xq < w) {
                        const long o = (long)yy * w + xq;
                        gx = gd[0] * xb[o] + gd[1] * xb[plane + o] + gd[2] * xb[2 * plane + o];
                    }
                    f[k] = sj * (gx - gdd);
                } else if (j == alpha_ch) {
                    f[k] = dalpha;
                }
            }
            store8(dlogits + i * hc + j0, f);
        }
    }
    if (loss_partial) {
        __shared__ float red[256];
        red[threadIdx.x] = local;
        __syncthreads();
        for (int st = blockDim.x / 2; st > 0; st >>= 1) {
            if ((int)threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
            __syncthreads();
        }
        if (threadIdx.x == 0) loss_partial[blockIdx.x] = red[0];
    }
}

// out = a + b (bf16, count a multiple of 8)
__global__ void add_bf16_kernel(const bf16* __restrict__ a, const bf16* __restrict__ b, bf16* __restrict__ out,
                                long count8) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < count8; i += (long)gridDim.x * blockDim.x) {
        float fa[8], fb[8];
        load8(a + i * 8, fa);
        load8(b + i * 8, fb);
#pragma unroll
        for (int k = 0; k < 8; ++k) fa[k] += fb[k];
        store8(out + i * 8, fa);
    }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
inline int grid_for(long work, int threads) {
    long b = (work + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 148L * 16) b = 148L * 16;
    return (int)b;
}

// An elementwise kernel over `units` 16-byte units, with 32-bit indices where they suffice (a 64-bit division by a
// runtime value is a long software routine, and these kernels divide several times per unit).
template <class K32, class K64, class... A>
void launch_units(long units, void* stream, K32 k32, K64 k64, A... args) {
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (units < (1L << 31)) k32<<<grid_for(units, 256), 256, 0, s>>>(args...);
    else k64<<<grid_for(units, 256), 256, 0, s>>>(args...);
}

inline int pow2_cols(int n) {
    int c = 32;
    while (c < n) c <<= 1;
    return c;
}

constexpr size_t kSmPerSm = 233472;   // shared memory of one SM (bytes)
constexpr size_t kSmPerCta = 232448;  // largest shared memory of one CTA

// Raises a kernel's limit of dynamic shared memory to all that a CTA can have, once on every device.  The limit is state
// of the process that every launch is checked against: set to the size of each launch, one thread could lower it
// between another's setting and its launch.  It is a limit only, and does not change what a launch occupies.
template <auto Kernel>
cudaError_t allow_smem() {
    static std::atomic<unsigned long long> done{0};  // a bit a device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    cudaFuncAttributes attr;
    if ((e = cudaFuncGetAttributes(&attr, Kernel)) != cudaSuccess) return e;
    e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kSmPerCta - attr.sharedSizeBytes));
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
}

template <int MODE, int STAGES>
cudaError_t launch_tile_n(const ConvArgs& a, dim3 grid, cudaStream_t s) {
    const size_t smem = (size_t)STAGES * (kBM * kBK * 2 + (size_t)a.n_tile * kBK * 2);
    const cudaError_t e = allow_smem<conv_tile_kernel<MODE, STAGES>>();
    if (e != cudaSuccess) return e;
    conv_tile_kernel<MODE, STAGES><<<grid, kThreads, smem, s>>>(a);
    count_launches(1);
    return cudaGetLastError();
}

static int g_gather_stages = 0;  // 0: 3 stages, except 4 for 64-column convolution tiles (measured)

template <int MODE>
cudaError_t launch_tile(const ConvArgs& a, dim3 grid, cudaStream_t s) {
    int st = g_gather_stages;
    if (st == 0) st = (MODE == kConv && a.n_tile == 64) ? 4 : 3;
    return st == 3 ? launch_tile_n<MODE, 3>(a, grid, s) : launch_tile_n<MODE, 4>(a, grid, s);
}

inline bool chan_ok(int c) { return c > 0 && c % 16 == 0; }

inline int sm_count() {
    int dev = 0, n = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 148;
}

constexpr size_t kStripSmemLimit = 200 * 1024;

inline size_t strip_smem_bytes(int cin, int cout) {
    return ((9ul * cin * cout * 2 + 127) & ~(size_t)127) + (size_t)kRing * (cin / 8) * kPlane;
}

// the row-strip kernel serves images at least one tile wide with at most 256 output channels; the
// input channels are split into groups whose weights and ring fit in shared memory (one pass each,
// summed through an fp32 partial)
inline int strip_groups(int width, int cin, int cout, bool any = false) {
    if (width < kBM || cout > 256) return 0;
    for (int g = 1; g <= 4; ++g) {
        const int cg = (cin / 16 + g - 1) / g * 16;
        // grouped passes re-stream an fp32 partial; they beat the gather kernel only for narrow
        // outputs (measured: 176 -> 32 faster, 160 -> 64 slower)
        if (strip_smem_bytes(cg, cout) <= kStripSmemLimit) return (g == 1 || cout <= 32 || any) ? g : 0;
    }
    return 0;
}

inline void strip_segments(int n, int h, int w, int slots, int& xtiles, int& seg_rows, int& segs_per_col,
                           int& total) {
    xtiles = (w + kBM - 1) / kBM;
    const int cols = n * xtiles;
    const int want = max(cols, 2 * slots);
    int spc = (want + cols - 1) / cols;
    spc = min(spc, max(1, h / 4));
    seg_rows = (h + spc - 1) / spc;
    segs_per_col = (h + seg_rows - 1) / seg_rows;
    total = cols * segs_per_col;
}

// The rule and the split of the weight gradient on image rows.  Which pixels a partial holds, and their order, are part
// of the result: one flipped rounding in the sum of a layer is as large as the error of a training step.  So
// images at least 128 pixels wide with 64 channels on a side are split by segments of rows, one partial for each CTA of
// a pass, where five 130-pixel rows of x and three 128-pixel rows of dy with their channels (one of the two in
// chunks of 64 or 128) take at most 220 KB; everything else in runs of pixels_per_split (wgrad_runs, conv_tile_kernel).
// `any`: also with fewer channels.
inline bool wgrad_by_rows(int width, int cin, int cout, bool any) {
    if (width < kBM || (!any && cin < 64 && cout < 64)) return false;
    for (int role = 0; role < 2; ++role) {
        const int u = role == 0 ? cin : cout, sc = role == 0 ? cout : cin;
        const int chunk = u > 64 ? 128 : 64, xc = role == 0 ? chunk : cin, dyc = role == 0 ? cout : chunk;
        if (sc <= 256 && 5 * kStripPix * 2 * xc + 3 * kBM * 2 * dyc <= 220 * 1024) return true;
    }
    return false;
}

struct WgradPlan {
    int role = 0, s_group = 32, u_chunks = 1, s_chunks = 1, passes = 1;
    int xtiles = 1, seg_rows = 1, segs_per_col = 1, grid = 1;
    int pps = 0, tiles = 1, row_groups = kBM / 16;  // runs of pixels
};

// Shared memory of wgrad_rows_kernel: strides and ring depth of S (as deep as fits, 0: less than the four rows it needs).
struct WgradSmem {
    int u_lines, s_lines, u_group_bytes, u_slot, s_tile, s_slot, s_ring;
    size_t bytes;
};
inline WgradSmem wgrad_smem(const WgradPlan& p, int cin, int cout) {
    WgradSmem m;
    const int pixels = std::min(kBM, p.row_groups * 16);
    m.u_lines = pixels + (p.role == 0 ? 2 : 0);
    m.s_lines = pixels + (p.role == 1 ? 2 : 0);
    // group, tile and slot strides: whole 1024-byte blocks (the swizzle acts on absolute addresses)
    auto up = [](int b) { return (b + 1023) / 1024 * 1024; };
    m.u_group_bytes = up(m.u_lines * 64);
    m.u_slot = m.u_group_bytes * ((p.role == 0 ? cin : cout) > 64 ? 4 : 2);
    m.s_tile = up(m.s_lines * p.s_group * 2);
    m.s_slot = m.s_tile * p.tiles;
    const int left = (int)kSmPerCta - 1024 - kWgURing * m.u_slot;
    m.s_ring = std::min(kWgMaxRing, left / m.s_slot);
    if (m.s_ring < 4) m.s_ring = 0;
    m.bytes = (size_t)kWgURing * m.u_slot + (size_t)m.s_ring * m.s_slot;
    return m;
}

inline WgradPlan wgrad_plan(int n, int h, int w, int cin, int cout, int sms) {
    WgradPlan p;
    int best = 0;
    for (int role = 0; role < 2; ++role) {  // the role with fewer passes
        const int u = role == 0 ? cin : cout, sc = role == 0 ? cout : cin;
        const int uc = (u + 127) / 128, sn = (sc + 31) / 32;
        if (best == 0 || uc * sn < best) {
            best = uc * sn;
            p.role = role;
            p.s_group = sc == 16 ? 16 : 32;
            p.u_chunks = uc;
            p.s_chunks = sn;
        }
    }
    p.passes = best;
    int total = 0;
    strip_segments(n, h, w, sms, p.xtiles, p.seg_rows, p.segs_per_col, total);
    p.grid = std::min(total, sms);
    return p;
}

// The row kernel on runs of pixels_per_split pixels, for whole 16-pixel groups a row: the gather kernel's order of pixels.
// For runs of 512 pixels (192 from 128 channels on both sides on), below which a CTA's nine accumulators cost more
// than the gather, and rows of 32 (a row costs its barriers).  us, gather / here, pixels of a run in brackets:
//     32 -> 32    8 x 64^2 [384] 14.4 / 15.1   256^2 [704] 22.4 / 16.5   512^2 [2,688] 72.3 / 31.5   8 x 256^2 [5,312] 141 / 53
//     48 -> 48    8 x 64^2 [448] 17.5 / 16.9   256^2 [896] 29.6 / 17.4   8 x 256^2 [7,104] 198 / 68
//     96 -> 96    64^2 [128] 12.9 / 14.5       112^2 [320] 19.0 / 18.4   8 x 64^2 [768] 49.2 / 26.6
//    224 -> 96    64^2 [256] 17.1 / 18.7       8 x 32^2 [448] 24.4 / 28.3   112^2 [704] 31.6 / 25.4   8 x 64^2 [1,728] 115 / 44
//    128 -> 128   64^2 [128] 14.4 / 13.6       8 x 32^2 [256] 19.6 / 18.3   8 x 64^2 [1,024] 55.3 / 29.0
inline bool wgrad_runs(int n, int h, int w, int cin, int cout, int pps, WgradPlan& p) {
    if (w % 16 || w < 32 || pps < w || pps < (cin >= 128 && cout >= 128 ? 192 : 512)) return false;
    p = wgrad_plan(n, h, w, cin, cout, sm_count());
    p.pps = pps;
    p.tiles = (w + kBM - 1) / kBM;
    p.row_groups = w / 16;
    p.grid = (int)(((long)n * h * w + pps - 1) / pps);
    return wgrad_smem(p, cin, cout).s_ring > 0;
}

cudaError_t launch_strip_pass(StripArgs a, cudaStream_t s) {
    a.xtiles = (a.w_ + kBM - 1) / kBM;
    a.tmem_cols = pow2_cols(2 * a.cout);
    const size_t smem = strip_smem_bytes(a.cin, a.cout);
    int per_sm = (int)(220 * 1024 / smem);
    per_sm = per_sm < 1 ? 1 : per_sm;
    per_sm = min(per_sm, 512 / a.tmem_cols);
    const int slots = sm_count() * per_sm;
    const int cols = a.n * a.xtiles;
    const int want = max(cols, 2 * slots);
    int spc = (want + cols - 1) / cols;
    spc = min(spc, max(1, a.h / 4));  // segments of at least 4 rows (2 halo rows per segment)
    a.seg_rows = (a.h + spc - 1) / spc;
    a.segs_per_col = (a.h + a.seg_rows - 1) / a.seg_rows;
    const int total = cols * a.segs_per_col;
    const int grid = min(total, slots);
    const cudaError_t e = allow_smem<conv_strip_kernel>();
    if (e != cudaSuccess) return e;
    conv_strip_kernel<<<grid, kThreads, smem, s>>>(a);
    count_launches(1);
    return cudaGetLastError();
}

// ---- the warp-specialised strip kernel ----
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static const EncodeTiledFn fn = []() -> EncodeTiledFn {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// NHWC bf16 activation [n][h][w][c] as a 4-D tensor (c, w, h, n) with boxes of `width` channels x
// 130 pixels, swizzled for lines of 2 * width bytes (the channel coordinate of every load is a
// multiple of 16 channels, i.e. 32 bytes)
bool encode_rows(CUtensorMap* map, const bf16* x, int n, int h, int w, int c, int width) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn || reinterpret_cast<uintptr_t>(x) % 16) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
    const cuuint64_t strides[3] = {(cuuint64_t)c * 2, (cuuint64_t)w * c * 2, (cuuint64_t)h * w * c * 2};
    const cuuint32_t box[4] = {(cuuint32_t)width, (cuuint32_t)kStripPix, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUtensorMapSwizzle sz = width == 64 ? CU_TENSOR_MAP_SWIZZLE_128B
                                              : (width == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(x), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, sz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// One tensor of a weight gradient, [n][h][w][c] bf16, as rows of `lines` pixels x `group` channels (64, 32 or
// 16: 128, 64 or 32-byte swizzled lines)
bool encode_wgrad(CUtensorMap* map, const bf16* x, int n, int h, int w, int c, int group, int lines) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
    const cuuint64_t strides[3] = {(cuuint64_t)c * 2, (cuuint64_t)w * c * 2, (cuuint64_t)h * w * c * 2};
    const cuuint32_t box[4] = {(cuuint32_t)group, (cuuint32_t)lines, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(x), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE,
              group == 64 ? CU_TENSOR_MAP_SWIZZLE_128B
                          : (group == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B),
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t launch_wgrad_rows(const bf16* x, const bf16* dy, float* partial, int* err, int n, int h, int w, int cin,
                              int cout, const WgradPlan& p, cudaStream_t s) {
    WgradArgs a{};
    a.partial = partial;
    a.err = err;
    a.n = n;
    a.h = h;
    a.w_ = w;
    a.cin = cin;
    a.cout = cout;
    a.m_pad = (9 * cin + kBM - 1) / kBM * kBM;
    a.role = p.role;
    a.s_group = p.s_group;
    a.u_chunks = p.u_chunks;
    a.s_chunks = p.s_chunks;
    a.xtiles = p.xtiles;
    a.seg_rows = p.seg_rows;
    a.segs_per_col = p.segs_per_col;
    a.pps = p.pps;
    a.tiles = p.tiles;
    a.row_groups = p.row_groups;
    const WgradSmem m = wgrad_smem(p, cin, cout);
    a.u_lines = m.u_lines;
    a.s_lines = m.s_lines;
    a.u_group_bytes = m.u_group_bytes;
    a.u_slot = m.u_slot;
    a.s_tile = m.s_tile;
    a.s_slot = m.s_slot;
    a.s_ring = m.s_ring;
    const int u_total = p.role == 0 ? cin : cout;
    const size_t smem = m.bytes;
    a.tmem_cols = pow2_cols(9 * p.s_group);
    CUtensorMap umap, smap;
    const bf16* ut = p.role == 0 ? x : dy;
    const bf16* st = p.role == 0 ? dy : x;
    if (!encode_wgrad(&umap, ut, n, h, w, u_total, 32, a.u_lines) ||
        !encode_wgrad(&smap, st, n, h, w, p.role == 0 ? cout : cin, p.s_group, a.s_lines))
        return cudaErrorInvalidValue;
    const dim3 grid((unsigned)p.grid, (unsigned)p.passes);
    const cudaError_t e = p.pps ? allow_smem<wgrad_rows_kernel<true>>() : allow_smem<wgrad_rows_kernel<false>>();
    if (e != cudaSuccess) return e;
    if (p.pps) wgrad_rows_kernel<true><<<grid, kWgThreads, smem, s>>>(umap, smap, a);
    else wgrad_rows_kernel<false><<<grid, kWgThreads, smem, s>>>(umap, smap, a);
    count_launches(1);
    return cudaGetLastError();
}

constexpr size_t kWsStatic = 2048;    // static shared memory + the per-CTA reservation, rounded up

// a pass's channels as groups of 64, then 32, then 16 (each a 1024-byte aligned buffer of 130 lines)
struct WsGroups {
    int n = 0, c[kWsMaxGroups] = {}, w[kWsMaxGroups] = {}, off[kWsMaxGroups] = {}, row_bytes = 0, tx = 0;
};
inline WsGroups ws_groups_of(int cin) {
    WsGroups g;
    int c = 0, off = 0;
    while (c < cin && g.n < kWsMaxGroups) {
        const int rem = cin - c, width = rem >= 64 ? 64 : (rem >= 32 ? 32 : 16);
        g.c[g.n] = c;
        g.w[g.n] = width;
        g.off[g.n] = off;
        off += (kStripPix * width * 2 + 1023) / 1024 * 1024;
        g.tx += kStripPix * width * 2;
        c += width;
        ++g.n;
    }
    g.row_bytes = c == cin ? off : 0;  // 0: more groups than supported
    return g;
}

inline size_t ws_weight_bytes(int cin, int cout) { return (9ul * cin * cout * 2 + 1023) & ~(size_t)1023; }
inline size_t ws_row_bytes(int cin) { return (size_t)ws_groups_of(cin).row_bytes; }

// the groups of `passes` (1 or 2) passes over the channels in one launch, pass by pass
inline int pass_channels(int cin, int passes) { return (cin / 16 + passes - 1) / passes * 16; }
inline WsGroups ws_groups_of(int cin, int passes) {
    if (passes == 1) return ws_groups_of(cin);
    const int cg = pass_channels(cin, 2);
    WsGroups g = ws_groups_of(cg);
    const WsGroups g1 = ws_groups_of(cin - cg);
    if (!g.row_bytes || !g1.row_bytes || g.n + g1.n > kWsMaxGroups) return WsGroups();
    for (int k = 0; k < g1.n; ++k) {
        g.c[g.n + k] = cg + g1.c[k];
        g.w[g.n + k] = g1.w[k];
        g.off[g.n + k] = g.row_bytes + g1.off[k];
    }
    g.n += g1.n;
    g.row_bytes += g1.row_bytes;
    g.tx += g1.tx;
    return g;
}

// The stacked kernel (cout <= kStackMaxCout a launch): a ring slot is free again after its own row's MMAs, so two slots
// do; two CTAs per SM when each gets three (their issuing threads overlap) and at least four accumulators.
bool stack_config(int cin, int cout, int passes, int& per_sm, int& ring) {
    const size_t rb = (size_t)ws_groups_of(cin, passes).row_bytes, wb = ws_weight_bytes(cin, cout);
    per_sm = 0;
    ring = 0;
    if (rb == 0) return false;
    for (int occ = 2; occ >= 1; --occ) {
        const size_t budget = std::min(kSmPerSm / occ - kWsStatic, kSmPerCta);
        if (wb >= budget || 512 / occ / (cout * passes) < 4) continue;
        const int r = (int)std::min<size_t>(kWsMaxRing, (budget - wb) / rb);
        if (r < (occ == 2 ? 3 : 2)) continue;
        per_sm = occ;
        ring = r;
        return true;
    }
    return false;
}

// CTAs per SM and ring depth: the most rows in flight per SM (CTAs x (ring - 3)), then more CTAs;
// TMEM holds two accumulators per CTA.  false when not even one CTA with a 4-slot ring fits.
bool ws_config(int cin, int cout, int& per_sm, int& ring) {
    const int acc = pow2_cols(cout);
    const size_t rb = ws_row_bytes(cin);
    per_sm = 0;
    ring = 0;
    if (rb == 0) return false;
    int best = -1;
    for (int occ = 1; occ <= 2 && occ * 2 * acc <= 512; ++occ) {  // 2: the registers of 2 CTAs fit an SM
        const size_t budget = kSmPerSm / occ - kWsStatic;
        const size_t wb = ws_weight_bytes(cin, cout);
        if (budget > kSmPerCta || wb >= budget) continue;
        const int r = (int)std::min<size_t>(kWsMaxRing, (budget - wb) / rb);
        if (r < 4) continue;
        const int score = occ * (r - 3);
        if (score > best || (score == best && occ > per_sm)) {
            best = score;
            per_sm = occ;
            ring = r;
        }
    }
    return per_sm > 0;
}


// input-channel passes of the row-strip kernels (0: the layer is not theirs).  Several passes, summed through an fp32
// partial: measured faster than the gather kernel for up to 64 output channels (176 -> 32, 160 -> 64), slower
// for 96 -> 96 and 224 -> 96.
inline int ws_passes(int width, int cin, int cout, bool any) {
    if (width < kBM || cout > 256) return 0;
    for (int g = 1; g <= 4; ++g) {
        int occ, ring;
        if (ws_config(pass_channels(cin, g), cout, occ, ring)) return (g == 1 || cout <= 64 || any) ? g : 0;
    }
    return 0;
}

// The order of a layer's sums.  It is part of the result and a function of the layer and the image alone, whichever
// kernel adds: fp32 sums in another order differ by 2e-7, which flips a few bf16 roundings and ReLU masks a layer, and
// twenty layers make that 2 to 4 % of a training step's gradient - as far as it is from its 64-bit value.
//   passes > 0: input channels in this many equal passes (the last may be smaller), whose sums are added in order; in
//   a pass by image row (dy), channel group (64, then 32, then 16 channels), dx, channel.
//   passes = 0: by K = tap * cin + channel, in ksplit runs of whole 64s, whose sums are added in order.
struct ConvOrder {
    int passes = 0, ksplit = 1;
};

// How the row-strip kernels take a layer.  Output channels: conv_stack_kernel for up to 80 of them, in chunks of at most
// 80 (each launch reads the input again) or all of them in conv_ws_kernel (chunk = 0) beyond.  One or two passes over the
// input channels in one launch where the weights and the rings fit, else a launch each through an fp32 partial.
// us on one image up to 256 rows of 128 pixels, images of 256 rows beyond (boxes in the layer's order; "before": conv_ws
// or, where it does not fit, the gather kernel, both without the kernels below):
//                 rows  128: stack, box, before   256              512              1,024            4,096
//     32 -> 32           8.3   6.4   9.6    8.9   7.0   9.6  10.2   8.9  10.2  12.3  14.3  11.9   24   41   29
//     48 -> 48          11.0   9.5  12.2   11.7  17.7  12.3  14.8  30.2  12.7  18.7  57.0  19.7   37  249   72
//     96 -> 32          13.3   9.0  14.4   14.9  10.2  14.6  18.5  18.8  14.8  24.8  35.2  24.1   67  122   94
//    160 -> 64          39.1  15.3  44.9   41.3  19.3  46.0  55.4  36.8  46.9  73.9  70.2  75.0  209  261  307
//    176 -> 32          20.4  14.1  30.9   21.3  16.0  31.4  29.0  30.2  32.1  37.8  57.7  49.6  109  214  211
//     96 -> 96          25.8  11.4  29.3   28.7  15.3  33.1  36.7  28.3  64.6  52.0  54.1   128  142  194  459
//     96 -> 224         53.1  16.6  40.3   57.7  30.5  79.2  73.7  57.6   156  96.1   102   275  235  385 1095
//     32 -> 176         25.4  10.4  25.6   25.7  12.1  25.9  26.7  22.5  27.1  42.0  44.9  42.3  129  150  163
// conv_box_kernel (on = false), whose tiles have a CTA each while these kernels read three rows for one and start with
// all nine taps' weights, where the width is a multiple of 128: up to two rows an SM, beyond one unless its stages would
// be more than half empty (48 channels in groups of 32 and 16); up to four with more than 80 output channels; up to
// eight with two passes and more than 48.  conv_ws_kernel: between two and four rows an SM (eight from 96 input channels
// on) for one pass of 48 input channels and more into at most 48; for 81 to 96 output channels; and for more of
// fewer than 16 rows an SM.  Output chunks from 64 rows a chunk.
struct StackPlan {
    bool on = false;
    int launches = 1;  // passes over the input channels with a launch each
    int chunk = 0;
};
inline StackPlan stack_plan(int n_img, int h, int width, int cin, int cout, const ConvOrder& order, bool any) {
    StackPlan p;
    if (width < kBM || cout > 256 || order.ksplit > 1) return p;
    const long rows = (long)n_img * ((width + kBM - 1) / kBM) * h;
    const long sms = sm_count();
    if (!any && width % kBM == 0 && order.passes <= 2) {
        const bool filled = order.passes == 0 || 2 * cin >= 64 * ws_groups_of(cin, order.passes).n;
        if (rows <= 2 * sms && cin > 16 && (filled || rows <= sms)) return p;
        if (rows <= 4 * sms && cout > kStackMaxCout && cin % 32 == 0) return p;
        if (rows <= 8 * sms && order.passes == 2 && cout > 48) return p;
    }
    // fewest output chunks of conv_stack_kernel with `passes` passes over c input channels
    int chunks = 0;
    auto fit = [&](int c, int passes) {
        int occ, ring;
        for (chunks = (cout + kStackMaxCout - 1) / kStackMaxCout; chunks <= 4; ++chunks) {
            const int n = (cout / 16 + chunks - 1) / chunks * 16;
            if (stack_config(c, n, passes, occ, ring)) return n;
        }
        return 0;
    };
    if (order.passes <= 2) p.chunk = fit(cin, std::max(1, order.passes));
    if (order.passes == 0) {
        p.on = p.chunk > 0 && (chunks == 1 || rows >= 64L * chunks || any);
        return p;
    }
    if (!p.chunk && order.passes > 1) {
        p.launches = order.passes;
        p.chunk = fit(pass_channels(cin, order.passes), 1);
    }
    // conv_ws_kernel fits (ws_passes)
    const bool narrow = order.passes == 1 && cin >= 48 && cout <= 48 && rows > 2 * sms && rows <= (cin >= 96 ? 8 : 4) * sms;
    const bool chunked = cout <= kStackMaxCout ? any || !narrow : cout > 96 && rows >= 16 * sms;
    if (!chunked || (chunks > 1 && rows < 64L * chunks && !any)) p.chunk = 0;
    if (!p.chunk) p.launches = order.passes;
    p.on = true;
    return p;
}

// the tensor maps (widths 64, 32, 16) and the channel groups of a launch
bool encode_groups(const StripArgs& a, int passes, WsArgs& wa, CUtensorMap (&maps)[3]) {
    const WsGroups gr = ws_groups_of(a.cin, passes);
    memset(maps, 0, sizeof(maps));
    bool have[3] = {false, false, false};
    for (int k = 0; k < gr.n; ++k) {
        const int mi = gr.w[k] == 64 ? 0 : (gr.w[k] == 32 ? 1 : 2);
        if (!have[mi] && !encode_rows(&maps[mi], a.x, a.n, a.h, a.w_, a.cin_total, gr.w[k])) return false;
        have[mi] = true;
        wa.gc[k] = gr.c[k];
        wa.gw[k] = gr.w[k];
        wa.goff[k] = gr.off[k];
    }
    wa.ngroups = gr.n;
    wa.row_bytes = gr.row_bytes;
    wa.tx_bytes = gr.tx;
    return true;
}

// the shared memory of a launch: at least what holds the CTAs per SM to per_sm (TMEM is sized for that many)
inline size_t ws_smem(int cin, int cout, int passes, int per_sm, int ring) {
    const size_t need = ws_weight_bytes(cin, cout) + (size_t)ring * ws_groups_of(cin, passes).row_bytes;
    return std::max(need, std::min(kSmPerCta, kSmPerSm / (per_sm + 1) - kWsStatic + 1024));
}

cudaError_t launch_ws(StripArgs a, cudaStream_t s) {
    int per_sm = 0, ring = 0;
    WsArgs wa{};
    CUtensorMap maps[3];
    if (!ws_config(a.cin, a.cout, per_sm, ring) || !encode_groups(a, 1, wa, maps)) return cudaErrorInvalidValue;
    a.tmem_cols = 2 * pow2_cols(a.cout);
    const int slots = sm_count() * per_sm;
    int total = 0;
    strip_segments(a.n, a.h, a.w_, slots, a.xtiles, a.seg_rows, a.segs_per_col, total);
    wa.s = a;
    const size_t smem = ws_smem(a.cin, a.cout, 1, per_sm, ring);
    const cudaError_t e = allow_smem<conv_ws_kernel>();
    if (e != cudaSuccess) return e;
    conv_ws_kernel<<<min(total, slots), kWsThreads, smem, s>>>(maps[0], maps[1], maps[2], wa, ring);
    count_launches(1);
    return cudaGetLastError();
}

// output channels [co0, co0 + cout) of the cout_total of a layer (a.cout is set here); passes: of this launch, 0 = the
// products by tap
cudaError_t launch_stack(StripArgs a, int co0, int cout, int cout_total, int passes, cudaStream_t s) {
    const int sets = std::max(1, passes);
    a.cout = cout;
    StackArgs sa{};
    int per_sm = 0;
    CUtensorMap maps[3];
    if (!stack_config(a.cin, cout, sets, per_sm, sa.ring) || !encode_groups(a, sets, sa.ws, maps))
        return cudaErrorInvalidValue;
    a.tmem_cols = 512 / per_sm;  // the CTAs of an SM share its 512 columns
    a.xtiles = (a.w_ + kBM - 1) / kBM;
    sa.groups0 = sets == 2 ? ws_groups_of(pass_channels(a.cin, 2)).n : sa.ws.ngroups;
    sa.by_tap = passes == 0;
    sa.blocks = std::min(kStackMaxBlocks, a.tmem_cols / (cout * sets));
    sa.co0 = co0;
    sa.cout_total = cout_total;
    sa.ws.s = a;
    const long rows = (long)a.n * a.xtiles * a.h;
    const int grid = (int)std::min<long>(std::max<long>(1, rows / 2), sm_count() * per_sm);  // at least two rows each
    const size_t smem = ws_smem(a.cin, cout, sets, per_sm, sa.ring);
    const cudaError_t e = allow_smem<conv_stack_kernel>();
    if (e != cudaSuccess) return e;
    conv_stack_kernel<<<grid, kStackThreads, smem, s>>>(maps[0], maps[1], maps[2], sa);
    count_launches(1);
    return cudaGetLastError();
}

// the box of 128 consecutive pixels of an image batch: rows and images, or false where they are not one
inline bool conv_box(int n, int h, int w, int& bh, int& bn) {
    bh = bn = 1;
    if (w % kBM == 0) return true;
    if (kBM % w) return false;
    const int rows = kBM / w;
    bh = std::min(rows, h);
    bn = rows / bh;
    return h % bh == 0 && rows % bh == 0;
}

cudaError_t launch_box(const ConvArgs& a, const ConvOrder& order, int bh, int bn, dim3 grid, cudaStream_t s) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return cudaErrorInvalidValue;
    BoxArgs b{};
    b.c = a;
    b.bh = bh;
    b.bn = bn;
    b.passes = order.passes;
    b.pass_ch = order.passes ? pass_channels(a.cin, order.passes) : 0;
    const int k64 = (9 * a.cin + 63) / 64;
    b.kper = (k64 + order.ksplit - 1) / order.ksplit * 64;
    if (order.passes == 2) b.c.tmem_cols = pow2_cols(2 * a.n_tile);
    b.cw = a.cin <= 16 ? 16 : (a.cin <= 32 ? 32 : 64);
    const CUtensorMapSwizzle sz = b.cw == 64 ? CU_TENSOR_MAP_SWIZZLE_128B
                                             : (b.cw == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    const cuuint64_t c = (cuuint64_t)a.cin, w = (cuuint64_t)a.w_, h = (cuuint64_t)a.h;
    const cuuint64_t xdims[4] = {c, w, h, (cuuint64_t)a.n}, xstr[3] = {c * 2, w * c * 2, h * w * c * 2};
    const cuuint32_t xbox[4] = {(cuuint32_t)b.cw, (cuuint32_t)std::min(a.w_, kBM), (cuuint32_t)bh, (cuuint32_t)bn};
    const cuuint64_t wdims[3] = {c, 9, (cuuint64_t)a.cout}, wstr[2] = {c * 2, 9 * c * 2};
    const cuuint32_t wbox[3] = {(cuuint32_t)b.cw, 1, (cuuint32_t)a.n_tile};
    const cuuint32_t one[4] = {1, 1, 1, 1};
    CUtensorMap xmap, wmap;
    auto encode = [&](CUtensorMap* m, int rank, const bf16* p, const cuuint64_t* dims, const cuuint64_t* str,
                      const cuuint32_t* box) {
        return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<bf16*>(p), dims, str, box, one,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, sz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    if (!encode(&xmap, 4, a.x, xdims, xstr, xbox) || !encode(&wmap, 3, a.w, wdims, wstr, wbox))
        return cudaErrorInvalidValue;
    const size_t smem = (size_t)kBoxStages * ((size_t)kBM * b.cw * 2 + ((size_t)a.n_tile * b.cw * 2 + 1023) / 1024 * 1024);
    const cudaError_t e = allow_smem<conv_box_kernel>();
    if (e != cudaSuccess) return e;
    conv_box_kernel<<<grid, kBoxThreads, smem, s>>>(xmap, wmap, b);
    count_launches(1);
    return cudaGetLastError();
}

static int g_strip_kernel = 0;  // 0: warp-specialised (TMA) strips, 1: the cp.async strip kernel

// groups: passes over the input channels with a launch each; passes, chunk: of a launch (launch_stack)
cudaError_t launch_strip(const ConvArgs& c, int groups, int chunk, int passes, cudaStream_t s) {
    StripArgs a{};
    a.x = c.x;
    a.w = c.w;
    a.err = c.err;
    a.n = c.n;
    a.h = c.h;
    a.w_ = c.w_;
    a.cout = c.cout;
    a.cin_total = c.cin;
    auto pass = [&](const StripArgs& p) {
        if (g_strip_kernel != 0) return launch_strip_pass(p, s);
        if (chunk == 0) return launch_ws(p, s);
        cudaError_t e = cudaSuccess;
        for (int co = 0; co < c.cout && e == cudaSuccess; co += chunk)
            e = launch_stack(p, co, min(chunk, c.cout - co), c.cout, passes, s);
        return e;
    };
    if (groups <= 1) {
        a.cin = c.cin;
        a.bias = c.bias;
        a.mask = c.mask;
        a.y = c.y;
        a.relu = c.relu;
        a.out_f32 = c.out_f32;
        return pass(a);
    }
    // fp32 partial sum of the earlier groups (stream-ordered scratch)
    float* part = nullptr;
    const size_t bytes = (size_t)c.n * c.h * c.w_ * c.cout * sizeof(float);
    cudaError_t e = vpt::scratch_alloc(reinterpret_cast<void**>(&part), bytes, s);
    if (e != cudaSuccess) return e;
    const int cg = pass_channels(c.cin, groups);
    for (int g = 0, c0 = 0; c0 < c.cin && e == cudaSuccess; ++g, c0 += cg) {
        const bool last = c0 + cg >= c.cin;
        StripArgs p = a;
        p.c0 = c0;
        p.cin = min(cg, c.cin - c0);
        p.part_in = g > 0 ? part : nullptr;
        p.part_out = last ? nullptr : part;
        if (last) {
            p.bias = c.bias;
            p.mask = c.mask;
            p.y = c.y;
            p.relu = c.relu;
            p.out_f32 = c.out_f32;
        }
        e = pass(p);
    }
    const cudaError_t f = cudaFreeAsync(part, s);
    return e != cudaSuccess ? e : f;
}

}  // namespace unet
}  // namespace vpt

using namespace vpt::unet;

static bool g_force_gather = false;  // conv path 1: the gather kernels everywhere
static bool g_force_strip = false;   // conv path 2: the strip kernels wherever they apply
static int g_conv_ksplit = 0;        // gather convolution K splits: 0 automatic, 1 none, k > 1 forced

static bool wgrad_on_rows(int w, int cin, int cout) {
    return !g_force_gather && wgrad_by_rows(w, cin, cout, g_force_strip) && encode_tiled();
}

extern "C" {

VptStatus vpt_unet_conv3x3(const void* x, const void* w, const float* bias, const void* mask, void* y, int n, int h,
                           int width, int cin, int cout, int relu, int out_f32, int* err, void* stream) {
    if (!x || !w || !y || n <= 0 || h <= 0 || width <= 0 || !chan_ok(cin) || !chan_ok(cout) || cout > 4096 ||
        (long)n * h * width > (1L << 30))
        return VPT_ERR_ARG;
    ConvArgs a{};
    a.x = static_cast<const bf16*>(x);
    a.w = static_cast<const bf16*>(w);
    a.bias = bias;
    a.mask = static_cast<const bf16*>(mask);
    a.y = y;
    a.err = err;
    a.n = n;
    a.h = h;
    a.w_ = width;
    a.cin = cin;
    a.cout = cout;
    const int ntiles = (cout + 255) / 256;
    a.n_tile = ((cout + ntiles - 1) / ntiles + 15) / 16 * 16;
    a.tmem_cols = pow2_cols(a.n_tile);
    a.relu = relu;
    a.out_f32 = out_f32;
    // tensor maps want a 16-byte aligned base (and the driver's encoder)
    const bool aligned = reinterpret_cast<uintptr_t>(x) % 16 == 0 && encode_tiled();
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    auto status = [](cudaError_t e) { return e == cudaSuccess ? VPT_OK : VPT_ERR_CUDA; };
    if (g_strip_kernel != 0 && !g_force_gather) {
        const int groups = strip_groups(width, cin, cout, g_force_strip);
        if (groups > 0) return status(launch_strip(a, groups, 0, 0, s));
    }
    const long P = (long)n * h * width;
    const unsigned gx = (unsigned)((P + kBM - 1) / kBM), gy = (unsigned)((cout + a.n_tile - 1) / a.n_tile);
    const int sms = sm_count();
    const long tiles = (long)gx * gy;
    ConvOrder order;
    if (g_strip_kernel == 0 && !g_force_gather && aligned) order.passes = ws_passes(width, cin, cout, g_force_strip);
    if (order.passes == 0) {
        // small grids (the deep levels): K split over more CTAs, raw fp32 sums finished by conv_finalize_kernel
        const int nk = (9 * cin + kBK - 1) / kBK;
        if (g_conv_ksplit > 1) order.ksplit = std::min(g_conv_ksplit, nk);
        else if (g_conv_ksplit == 0 && 2 * tiles <= sms)  // under half a wave: about two CTAs per SM (measured)
            order.ksplit = (int)std::max<long>(1, std::min<long>(std::min<long>(8, (2L * sms + tiles - 1) / tiles), nk / 2));
    }
    if (g_strip_kernel == 0 && !g_force_gather && aligned) {
        const StackPlan plan = stack_plan(n, h, width, cin, cout, order, g_force_strip);
        if (plan.on)
            return status(launch_strip(a, plan.launches, plan.chunk, plan.launches > 1 ? 1 : order.passes, s));
    }
    int bh = 1, bn = 1;
    const bool box = !g_force_gather && aligned && reinterpret_cast<uintptr_t>(w) % 16 == 0 &&
                     conv_box(n, h, width, bh, bn);
    const int ksplit = order.ksplit;
    if (ksplit == 1)
        return status(box ? launch_box(a, order, bh, bn, dim3(gx, gy, 1), s) : launch_tile<kConv>(a, dim3(gx, gy, 1), s));
    float* part = nullptr;
    if (vpt::scratch_alloc(reinterpret_cast<void**>(&part), (size_t)ksplit * P * cout * sizeof(float), s) != cudaSuccess)
        return VPT_ERR_OOM;
    a.ksplit = ksplit;
    a.partial = part;
    const dim3 grid(gx, gy, (unsigned)ksplit);
    cudaError_t e = box ? launch_box(a, order, bh, bn, grid, s) : launch_tile<kConv>(a, grid, s);
    if (e == cudaSuccess) {
        launch_units(P * (cout / 4), stream, conv_finalize_kernel<uint32_t>, conv_finalize_kernel<unsigned long long>,
                     (const float*)part, ksplit, P, cout, bias, static_cast<const bf16*>(mask), relu, out_f32, y);
        e = cudaGetLastError();
    }
    const cudaError_t f = cudaFreeAsync(part, s);
    return (e == cudaSuccess && f == cudaSuccess) ? VPT_OK : VPT_ERR_CUDA;
}

// 0: the warp-specialised (TMA) row-strip kernel, 1: the cp.async row-strip kernel (comparisons)
VptStatus vpt_unet_set_strip_kernel(int kind) {
    if (kind < 0 || kind > 1) return VPT_ERR_ARG;
    g_strip_kernel = kind;
    return VPT_OK;
}

// K splits of the gather convolution: 0 chosen by grid size, 1 never split, k > 1 always k (tests)
VptStatus vpt_unet_set_conv_ksplit(int ksplit) {
    if (ksplit < 0 || ksplit > 64) return VPT_ERR_ARG;
    g_conv_ksplit = ksplit;
    return VPT_OK;
}

// 1: every convolution uses the per-tile gather kernel (for comparisons); 0: row strips where eligible
VptStatus vpt_unet_set_conv_path(int path) {
    if (path < 0 || path > 2) return VPT_ERR_ARG;
    g_force_gather = path == 1;
    g_force_strip = path == 2;
    return VPT_OK;
}

// shared-memory ring depth of the gather kernel (3 or 4; 0 = by shape)
VptStatus vpt_unet_set_gather_stages(int stages) {
    if (stages != 0 && stages != 3 && stages != 4) return VPT_ERR_ARG;
    g_gather_stages = stages;
    return VPT_OK;
}

VptStatus vpt_unet_conv3x3_wgrad(const void* x, const void* dy, float* partial, int n, int h, int width, int cin,
                                 int cout, int pixels_per_split, int* err, void* stream) {
    if (!x || !dy || !partial || n <= 0 || h <= 0 || width <= 0 || !chan_ok(cin) || !chan_ok(cout) ||
        cout > 4096 || pixels_per_split <= 0 || pixels_per_split % kBK != 0 || (long)n * h * width > (1L << 30))
        return VPT_ERR_ARG;
    ConvArgs a{};
    a.x = static_cast<const bf16*>(x);
    a.w = static_cast<const bf16*>(dy);
    a.y = partial;
    a.err = err;
    a.n = n;
    a.h = h;
    a.w_ = width;
    a.cin = cin;
    a.cout = cout;
    const int ntiles = (cout + 255) / 256;
    a.n_tile = ((cout + ntiles - 1) / ntiles + 15) / 16 * 16;
    a.tmem_cols = pow2_cols(a.n_tile);
    a.pix_per_split = pixels_per_split;
    const int mtiles = (9 * cin + kBM - 1) / kBM;
    a.m_pad = mtiles * kBM;
    if (wgrad_on_rows(width, cin, cout)) {  // (its tensor maps want aligned tensors)
        if (reinterpret_cast<uintptr_t>(x) % 16 || reinterpret_cast<uintptr_t>(dy) % 16) return VPT_ERR_ARG;
        const WgradPlan plan = wgrad_plan(n, h, width, cin, cout, sm_count());
        return launch_wgrad_rows(a.x, a.w, partial, err, n, h, width, cin, cout, plan,
                                 static_cast<cudaStream_t>(stream)) == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
    }
    WgradPlan runs;
    if (!g_force_gather && reinterpret_cast<uintptr_t>(x) % 16 == 0 && reinterpret_cast<uintptr_t>(dy) % 16 == 0 &&
        encode_tiled() && wgrad_runs(n, h, width, cin, cout, pixels_per_split, runs))
        return launch_wgrad_rows(a.x, a.w, partial, err, n, h, width, cin, cout, runs,
                                 static_cast<cudaStream_t>(stream)) == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
    const long P = (long)n * h * width;
    const dim3 grid((unsigned)mtiles, (unsigned)((cout + a.n_tile - 1) / a.n_tile),
                    (unsigned)((P + pixels_per_split - 1) / pixels_per_split));
    return launch_tile<kWgrad>(a, grid, static_cast<cudaStream_t>(stream)) == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

int vpt_unet_wgrad_rows(int cin) { return (9 * cin + kBM - 1) / kBM * kBM; }

int vpt_unet_wgrad_splits(int n, int h, int width, int cin, int cout, int pixels_per_split) {
    if (n <= 0 || h <= 0 || width <= 0 || !chan_ok(cin) || !chan_ok(cout) || cout > 4096 || pixels_per_split <= 0) return 0;
    if (wgrad_on_rows(width, cin, cout)) return wgrad_plan(n, h, width, cin, cout, sm_count()).grid;
    const long P = (long)n * h * width;
    return (int)((P + pixels_per_split - 1) / pixels_per_split);
}

VptStatus vpt_unet_rotate_weights(const void* w, void* wrot, int cin, int cout, void* stream) {
    if (!w || !wrot || !chan_ok(cin) || !chan_ok(cout)) return VPT_ERR_ARG;
    rotate_weights_kernel<<<grid_for((long)cout * 9 * cin, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(w), static_cast<bf16*>(wrot), cin, cout);
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

VptStatus vpt_unet_pool2(const void* in, void* out, int n, int h, int w, int c, void* stream) {
    if (!in || !out || n <= 0 || h <= 1 || w <= 1 || h % 2 || w % 2 || c <= 0 || c % 8) return VPT_ERR_ARG;
    launch_units((long)n * (h / 2) * (w / 2) * (c / 8), stream, pool2_kernel<uint32_t>, pool2_kernel<unsigned long long>,
                 static_cast<const bf16*>(in), static_cast<bf16*>(out), n, h, w, c);
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

VptStatus vpt_unet_upcat(const void* lo, const void* skip, void* out, int n, int h, int w, int ca, int cs,
                         void* stream) {
    if (!lo || !skip || !out || n <= 0 || h <= 1 || w <= 1 || h % 2 || w % 2 || ca <= 0 || ca % 8 || cs <= 0 ||
        cs % 8)
        return VPT_ERR_ARG;
    launch_units((long)n * h * w * ((ca + cs) / 8), stream, upcat_kernel<uint32_t>, upcat_kernel<unsigned long long>,
                 static_cast<const bf16*>(lo), static_cast<const bf16*>(skip), static_cast<bf16*>(out), n, h, w, ca, cs);
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

VptStatus vpt_unet_upcat_grad_lo(const void* d, const void* lo, void* dlo, int n, int h, int w, int ca, int cs,
                                 void* stream) {
    if (!d || !lo || !dlo || n <= 0 || h <= 1 || w <= 1 || h % 2 || w % 2 || ca <= 0 || ca % 8 || cs <= 0 ||
        cs % 8)
        return VPT_ERR_ARG;
    launch_units((long)n * (h / 2) * (w / 2) * (ca / 8), stream, upcat_grad_lo_kernel<uint32_t>,
                 upcat_grad_lo_kernel<unsigned long long>,
                 static_cast<const bf16*>(d), static_cast<const bf16*>(lo), static_cast<bf16*>(dlo), n, h, w, ca, cs);
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

VptStatus vpt_unet_encoder_grad(const void* d_cat, int cat_c, int cat_off, const void* d_pool, const void* e,
                                void* out, int n, int h, int w, int c, void* stream) {
    if (!e || !out || n <= 0 || h <= 0 || w <= 0 || c <= 0 || c % 8 || (d_cat && (cat_off % 8 || cat_c % 8)) ||
        (d_pool && (h % 2 || w % 2)))
        return VPT_ERR_ARG;
    launch_units((long)n * h * w * (c / 8), stream, encoder_grad_kernel<uint32_t>, encoder_grad_kernel<unsigned long long>,
                 static_cast<const bf16*>(d_cat), cat_c, cat_off, static_cast<const bf16*>(d_pool),
                 static_cast<const bf16*>(e), static_cast<bf16*>(out), n, h, w, c);
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

VptStatus vpt_unet_bias_grad(const void* dy, float* partial, int pixels, int c, int blocks, void* stream) {
    if (!dy || !partial || pixels <= 0 || c <= 0 || c % 8 || c > 2048 || blocks <= 0) return VPT_ERR_ARG;
    const int c8 = c / 8;
    int threads = 256 / c8 * c8;
    if (threads < c8) threads = c8;
    const size_t smem = (size_t)(threads / c8) * c * sizeof(float);
    bias_grad_kernel<<<blocks, threads, smem, static_cast<cudaStream_t>(stream)>>>(static_cast<const bf16*>(dy),
                                                                                   partial, pixels, c);
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

VptStatus vpt_unet_reduce_grads(const float* wpartial, int splits, int cin, int cout, const float* bpartial,
                                int bblocks, float* grad_w, float* grad_b, void* stream) {
    if (!wpartial || !grad_w || !grad_b || splits <= 0 || !chan_ok(cin) || !chan_ok(cout) ||
        (bpartial && bblocks <= 0))
        return VPT_ERR_ARG;
    const int m_pad = (9 * cin + kBM - 1) / kBM * kBM;
    const int blocks = cout * 9 * cin / (reduce_shared(splits, cout * 9 * cin) ? 32 : 256) + (cout + 31) / 32;
    reduce_grads_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        wpartial, splits, m_pad, cin, cout, bpartial, bblocks, grad_w, grad_b);
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

VptStatus vpt_unet_adam(float* param, void* param_bf16, float* m1, float* m2, const float* grad, long count, float lr,
                        float beta1, float beta2, float eps, int step, float grad_scale, void* stream) {
    if (!param || !m1 || !m2 || !grad || count <= 0 || step <= 0) return VPT_ERR_ARG;
    const float bias1 = 1.0f - powf(beta1, (float)step), bias2 = 1.0f - powf(beta2, (float)step);
    adam_kernel<<<grid_for(count, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        param, static_cast<bf16*>(param_bf16), m1, m2, grad, count, lr, beta1, beta2, eps, bias1, bias2, grad_scale);
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

VptStatus vpt_unet_to_bf16(const float* in, void* out, long count, void* stream) {
    if (!in || !out || count <= 0) return VPT_ERR_ARG;
    f32_to_bf16_kernel<<<grid_for(count, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        in, static_cast<bf16*>(out), count);
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

VptStatus vpt_unet_pack_input(const float* radiance, const float* albedo, const float* normal, const float* depth,
                              const float* transmittance, const float* noise_level, const float* second_moment,
                              void* out, int n, int h, int w, void* stream) {
    if (!radiance || !out || n <= 0 || h <= 0 || w <= 0) return VPT_ERR_ARG;
    pack_input_kernel<<<grid_for((long)n * h * w, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        radiance, albedo, normal, depth, transmittance, noise_level, second_moment, static_cast<bf16*>(out), n, h, w);
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

int vpt_unet_head_blocks(int n, int h, int w) { return grid_for((long)n * h * w, 256); }

VptStatus vpt_unet_kpn_head(const float* logits, int head_channels, int kernel_size, const float* radiance,
                            const float* target, float* out, void* dlogits, float* loss_partial, int n, int h, int w,
                            float eps, void* stream) {
    if (!logits || !radiance || n <= 0 || h <= 0 || w <= 0 || (target && !dlogits) || eps <= 0.0f ||
        kernel_size <= 0 || kernel_size % 2 == 0 || kernel_size > 15 || head_channels % 8 ||
        head_channels < kernel_size * kernel_size || head_channels > 512 || reinterpret_cast<uintptr_t>(logits) % 16)
        return VPT_ERR_ARG;
    // the loss partials are per block: as many blocks as vpt_unet_head_blocks (never more than the
    // row segments, which the blocks stride over)
    const int blocks = grid_for((long)n * h * w, 256);
    const float inv_count = 1.0f / (3.0f * (float)n * (float)h * (float)w);
    const size_t smem =
        ((size_t)kHeadSeg * (head_channels + 4) + 3 * kernel_size * head_window_row(kernel_size)) * sizeof(float);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    bf16* dl = static_cast<bf16*>(dlogits);
    cudaError_t e = cudaErrorInvalidValue;
    auto go = [&](auto size) {
        constexpr int kSize = decltype(size)::value;
        if (allow_smem<kpn_head_kernel<kSize>>() != cudaSuccess) return cudaErrorInvalidValue;
        kpn_head_kernel<kSize><<<blocks, 256, smem, s>>>(logits, head_channels, radiance, target, out, dl, loss_partial, n, h, w,
                                         eps, inv_count);
        return cudaGetLastError();
    };
    switch (kernel_size) {
        case 1: e = go(std::integral_constant<int, 1>()); break;
        case 3: e = go(std::integral_constant<int, 3>()); break;
        case 5: e = go(std::integral_constant<int, 5>()); break;
        case 7: e = go(std::integral_constant<int, 7>()); break;
        case 9: e = go(std::integral_constant<int, 9>()); break;
        case 11: e = go(std::integral_constant<int, 11>()); break;
        case 13: e = go(std::integral_constant<int, 13>()); break;
        case 15: e = go(std::integral_constant<int, 15>()); break;
        default: return VPT_ERR_ARG;
    }
    if (e != cudaSuccess) return VPT_ERR_CUDA;
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

VptStatus vpt_unet_kpn_combine(const float* d, const float* c_coarse, const float* logits, int head_channels,
                               int alpha_channel, float* c, int n, int h, int w, void* stream) {
    if (!d || !c_coarse || !logits || !c || n <= 0 || h <= 1 || w <= 1 || h % 2 || w % 2 || alpha_channel < 0 ||
        alpha_channel >= head_channels)
        return VPT_ERR_ARG;
    kpn_combine_kernel<<<grid_for((long)n * h * w, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        d, c_coarse, logits, head_channels, alpha_channel, c, n, h, w);
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

VptStatus vpt_unet_kpn_level_grad(const float* logits, int head_channels, int kernel_size, int alpha_channel,
                                  const float* x, const float* d, const float* c_coarse, const float* g_in,
                                  const float* c_out, const float* target, float eps, void* dlogits, float* g_coarse,
                                  float* loss_partial, int n, int h, int w, void* stream) {
    if (!logits || !x || !d || !dlogits || n <= 0 || h <= 0 || w <= 0 || kernel_size <= 0 || kernel_size % 2 == 0 ||
        kernel_size > 15 || head_channels % 8 || head_channels < kernel_size * kernel_size ||
        (alpha_channel >= 0 && (alpha_channel < kernel_size * kernel_size || alpha_channel >= head_channels ||
                                !c_coarse || h % 2 || w % 2)) ||
        (target ? !c_out : !g_in) || eps <= 0.0f || (loss_partial && !target))
        return VPT_ERR_ARG;
    const float inv_count = 1.0f / (3.0f * (float)n * (float)h * (float)w);
    kpn_level_grad_kernel<<<grid_for((long)n * h * w, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        logits, head_channels, kernel_size, alpha_channel, x, d, c_coarse, g_in, c_out, target, eps, inv_count,
        static_cast<bf16*>(dlogits), g_coarse, loss_partial, n, h, w);
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

VptStatus vpt_unet_add(const void* a, const void* b, void* out, long count, void* stream) {
    if (!a || !b || !out || count <= 0 || count % 8) return VPT_ERR_ARG;
    add_bf16_kernel<<<grid_for(count / 8, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(a), static_cast<const bf16*>(b), static_cast<bf16*>(out), count / 8);
    vpt::count_launches(1);
    return cudaGetLastError() == cudaSuccess ? VPT_OK : VPT_ERR_CUDA;
}

}  // extern "C"
