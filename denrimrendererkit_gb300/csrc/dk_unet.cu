// Kernels of the learned denoiser (dk_unet_* in include/denrim_cuda.h): a
// 5-level U-Net over the tracer's beauty + albedo + normal + depth AOVs.
//
// Tensors are NHWC bf16 with channel counts that are multiples of 16; a
// tensor may be a channel slice of a wider buffer (leading dimension `ld`,
// channel offset), so the decoder's concat(upsampled, skip) inputs are written
// in place.  3x3 convolutions (stride 1, zero padding 1) are implicit GEMMs
// on the tensor cores with FP32 accumulation:
//   forward   out[p][co] = act(b[co] + sum_{tap, ci} in[p + tap][ci] w[co][tap][ci])
//             M = pixels, N = Cout, K = 9 Cin; also the input gradient, as a
//             forward convolution of the output gradient with the
//             tap-flipped, transposed weights;
//   wgrad     dW[co][tap][ci] += sum_p dOut[p][co] in[p + tap][ci]
//             M = taps x Cin, N = Cout, K = pixels, split over CTAs.
#include <cstdint>
#include <cstdlib>
#include <initializer_list>

#include <cuda.h>
#include <cuda_bf16.h>

#include "dk_host.h"
#include "dk_smem_limit.h"

namespace dk {
namespace {

__device__ __forceinline__ uint32_t smemAddr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Programmatic dependent launch: the forward pass's kernels are launched so
// that each may start (and set up shared memory, barriers and tensor memory)
// while the previous one drains.  pdlWait() blocks until the previous kernel
// in the stream has completed and its writes are visible; every thread calls
// it before its first global memory access.  pdlRelease() lets the next
// kernel be scheduled.  Both are no-ops for a kernel launched without the
// attribute.
__device__ __forceinline__ void pdlWait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdlRelease() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// 16-byte async copy; `bytes` 0 fills the destination with zeros.
__device__ __forceinline__ void cpAsync16(void* dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smemAddr(dst)), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cpAsyncWait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void ldmatrixX4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(smemAddr(p)));
}

__device__ __forceinline__ void ldmatrixX4T(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(smemAddr(p)));
}

// D = A (16x16 bf16, row) * B (16x8 bf16, col) + D (fp32).
__device__ __forceinline__ void mmaBf16(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ------------------------------------------------------------ forward ----
struct ConvArgs {
    const __nv_bfloat16* in;
    const __nv_bfloat16* w;  // [cout][9][cin]
    const float* bias;       // [cout] or null
    __nv_bfloat16* out;
    uint32_t n, h, w_, cin, ldi, cout, ldo, coOff;
    uint32_t M;  // n * h * w
    int act;     // 0 identity, 1 ReLU
    int accumulate;
};

constexpr int kBM = 128;  // pixels per block
constexpr int kBK = 32;   // channels per k step (4 chunks of 16 bytes)
constexpr int kStages = 3;

// Byte offset of 16-byte chunk `seg` (0..3) of row `r` in a 64-byte-row tile.
__device__ __forceinline__ uint32_t swz64(uint32_t r, uint32_t seg) { return r * 64u + ((seg ^ ((r >> 1) & 3u)) << 4); }

template <int BN>
__global__ void __launch_bounds__(128) k_conv3x3_fwd(ConvArgs a) {
    __shared__ __align__(128) unsigned char sA[kStages][kBM * 64];
    __shared__ __align__(128) unsigned char sB[kStages][BN * 64];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;
    const uint32_t HW = a.h * a.w_;
    // This thread loads A row `tid` (one output pixel).
    const uint32_t m = m0 + tid;
    const bool rowValid = m < a.M;
    const uint32_t img = rowValid ? m / HW : 0u, rem = rowValid ? m - img * HW : 0u;
    const int py = (int)(rem / a.w_), px = (int)(rem - (rem / a.w_) * a.w_);
    const uint32_t chunks = (a.cin + kBK - 1) / kBK;
    const uint32_t kIters = 9u * chunks;

    auto loadStage = [&](uint32_t it, int stage) {
        uint32_t tap = it / chunks, c0 = (it - tap * chunks) * kBK;
        int dy = (int)(tap / 3u) - 1, dx = (int)(tap % 3u) - 1;
        int yy = py + dy, xx = px + dx;
        bool inb = rowValid && yy >= 0 && yy < (int)a.h && xx >= 0 && xx < (int)a.w_;
        const __nv_bfloat16* src =
            inb ? a.in + ((size_t)(img * a.h + (uint32_t)yy) * a.w_ + (uint32_t)xx) * a.ldi + c0 : a.in;
#pragma unroll
        for (uint32_t seg = 0; seg < 4; ++seg) {
            bool v = inb && c0 + seg * 8u < a.cin;
            cpAsync16(&sA[stage][swz64(tid, seg)], v ? src + seg * 8u : a.in, v ? 16u : 0u);
        }
#pragma unroll
        for (uint32_t i = tid; i < (uint32_t)BN * 4u; i += 128u) {
            uint32_t row = i >> 2, seg = i & 3u;
            bool v = c0 + seg * 8u < a.cin;
            const __nv_bfloat16* wsrc = a.w + ((size_t)(n0 + row) * 9u + tap) * a.cin + c0 + seg * 8u;
            cpAsync16(&sB[stage][swz64(row, seg)], v ? wsrc : a.w, v ? 16u : 0u);
        }
    };

    float acc[2][BN / 8][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < BN / 8; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.0f;

#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) {
        if ((uint32_t)s < kIters) loadStage(s, s);
        cpAsyncCommit();
    }
    for (uint32_t it = 0; it < kIters; ++it) {
        cpAsyncWait<kStages - 2>();
        __syncthreads();
        uint32_t nxt = it + kStages - 1;
        if (nxt < kIters) loadStage(nxt, (int)(nxt % kStages));
        cpAsyncCommit();
        const int st = (int)(it % kStages);
#pragma unroll
        for (uint32_t kk = 0; kk < 2; ++kk) {
            uint32_t af[2][4];
#pragma unroll
            for (uint32_t mt = 0; mt < 2; ++mt) {
                uint32_t r = warp * 32u + mt * 16u + (lane & 15u);
                uint32_t seg = kk * 2u + (lane >> 4);
                ldmatrixX4(af[mt][0], af[mt][1], af[mt][2], af[mt][3], &sA[st][swz64(r, seg)]);
            }
#pragma unroll
            for (uint32_t np = 0; np < (uint32_t)BN / 16u; ++np) {
                uint32_t r = np * 16u + (lane & 7u) + ((lane >> 4) << 3);
                uint32_t seg = kk * 2u + ((lane >> 3) & 1u);
                uint32_t b0, b1, b2, b3;
                ldmatrixX4(b0, b1, b2, b3, &sB[st][swz64(r, seg)]);
#pragma unroll
                for (uint32_t mt = 0; mt < 2; ++mt) {
                    mmaBf16(acc[mt][2 * np], af[mt], b0, b1);
                    mmaBf16(acc[mt][2 * np + 1], af[mt], b2, b3);
                }
            }
        }
    }
    cpAsyncWait<0>();
    // Epilogue: bias, activation, optional accumulate, bf16 store.
#pragma unroll
    for (uint32_t mt = 0; mt < 2; ++mt) {
#pragma unroll
        for (uint32_t half = 0; half < 2; ++half) {
            uint32_t row = m0 + warp * 32u + mt * 16u + (lane >> 2) + half * 8u;
            if (row >= a.M) continue;
            __nv_bfloat16* orow = a.out + (size_t)row * a.ldo + a.coOff;
#pragma unroll
            for (uint32_t nt = 0; nt < (uint32_t)BN / 8u; ++nt) {
                uint32_t col = n0 + nt * 8u + (lane & 3u) * 2u;
                float v0 = acc[mt][nt][half * 2 + 0], v1 = acc[mt][nt][half * 2 + 1];
                if (a.bias) {
                    v0 += a.bias[col];
                    v1 += a.bias[col + 1];
                }
                if (a.act == 1) {
                    v0 = fmaxf(v0, 0.0f);
                    v1 = fmaxf(v1, 0.0f);
                }
                __nv_bfloat162* dst = reinterpret_cast<__nv_bfloat162*>(orow + col);
                if (a.accumulate) {
                    float2 o = __bfloat1622float2(*dst);
                    v0 += o.x;
                    v1 += o.y;
                }
                *dst = __floats2bfloat162_rn(v0, v1);
            }
        }
    }
}

// ------------------------------------------------- tcgen05 forward ----
// The same convolution on the 5th-generation tensor cores: one CTA computes
// 128 output pixels x all Cout (one tcgen05.mma of M = 128, N = Cout, K = 16
// per 16 input channels of a tap), accumulating in tensor memory.  Operand
// tiles are K-major with the 128-byte swizzle: 64 channels (128 bytes) per
// row, 8-row atoms of 1024 bytes; cp.async fills them (zero fill for the
// padding), one thread issues the MMAs and commits each stage to an
// mbarrier that the copies of the stage's next use wait on.  Every wait is
// bounded: on timeout the kernel records an error, waits (bounded) for its
// MMAs, frees its tensor memory and returns.
constexpr int kTcStages = 4;
constexpr uint32_t kTcRows = 128;

__device__ int g_unetError;

__device__ __forceinline__ uint64_t umaDesc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4)  // start address
           | ((uint64_t)1 << 16)                // leading byte offset (unused for swizzled K-major)
           | ((uint64_t)(1024u >> 4) << 32)     // stride byte offset: 8 rows x 128 B
           | ((uint64_t)1 << 46)                // descriptor version
           | ((uint64_t)2 << 61);               // 128-byte swizzle
}

// tcgen05.mma kind::f16 with both shared-memory descriptors given as their
// low words (start address >> 4 in bits 0-13, leading byte offset) and the
// high word they share (stride byte offset, version, 128-byte swizzle): an
// operand's position inside a tile is then one 32-bit add, and the single
// issuing thread spends a few instructions per MMA.
__device__ __forceinline__ uint32_t descLo(uint32_t saddr) { return (uint32_t)umaDesc(saddr); }
__device__ __forceinline__ uint32_t descHi() { return (uint32_t)(umaDesc(0u) >> 32); }
__device__ __forceinline__ void mmaF16(uint32_t d, uint32_t aLo, uint32_t bLo, uint32_t hi, uint32_t idesc,
                                       uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\n.reg .b64 da, db;\nsetp.ne.b32 p, %5, 0;\nmov.b64 da, {%1, %3};\nmov.b64 db, {%2, %3};\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n}\n" ::"r"(d),
        "r"(aLo), "r"(bLo), "r"(hi), "r"(idesc), "r"(acc));
}

// tcgen05.mma with the operands' own high descriptor words, skipped when `on` is 0.
__device__ __forceinline__ void mmaF16If(uint32_t on, uint32_t d, uint32_t aLo, uint32_t aHi, uint32_t bLo, uint32_t bHi,
                                         uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p, q;\n.reg .b64 da, db;\nsetp.ne.b32 p, %6, 0;\nsetp.ne.b32 q, %7, 0;\n"
        "mov.b64 da, {%1, %2};\nmov.b64 db, {%3, %4};\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n}\n" ::"r"(d),
        "r"(aLo), "r"(aHi), "r"(bLo), "r"(bHi), "r"(idesc), "r"(acc), "r"(on));
}

__device__ __forceinline__ bool mbarTryWait(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0u;
}
__device__ __forceinline__ bool mbarWait(uint32_t bar, uint32_t parity) {
    if (mbarTryWait(bar, parity)) return true;
    const long long start = clock64();
    for (;;) {
        if (mbarTryWait(bar, parity)) return true;
        if (clock64() - start > 4000000000ll) return false;  // about 2 s
    }
}

// The MMA role is run by its whole warp with values the compiler can keep in
// uniform registers (warp index and tensor-memory address broadcast by a
// shuffle, loop counters, ring positions), and one elected lane issues.  Issued
// from a divergent single thread, every tcgen05.mma moved its descriptors and
// addresses from vector to uniform registers first: about 96 cycles each,
// whatever N (a 128 x 64 x 16 MMA runs in 32 to 48).
__device__ __forceinline__ bool electOne() {
    uint32_t p;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0u;
}
__device__ __forceinline__ bool mbarWaitWarp(uint32_t bar, uint32_t parity) {
    return __all_sync(0xffffffffu, mbarWait(bar, parity));
}

// A slot of an n-slot ring and the parity of its current use, advanced one
// use at a time (no division on the issuing threads' path).
struct RingPos {
    uint32_t slot, phase;
    __device__ __forceinline__ void advance(uint32_t n) {
        if (++slot == n) {
            slot = 0u;
            phase ^= 1u;
        }
    }
};

__global__ void __launch_bounds__(128, 1) k_conv3x3_tc(ConvArgs a, uint32_t tmemCols) {
    extern __shared__ unsigned char dsm[];
    const uint32_t raw = smemAddr(dsm);
    unsigned char* sm = dsm + (((raw + 1023u) & ~1023u) - raw);
    const uint32_t N = a.cout;
    const uint32_t aBytes = kTcRows * 128u, bBytes = N * 128u;
    unsigned char* sA = sm;
    unsigned char* sB = sm + kTcStages * aBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sB + kTcStages * bBytes);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + kTcStages);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smemAddr(tslot)),
                     "r"(tmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        for (int s = 0; s < kTcStages; ++s)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smemAddr(&bars[s])));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t taddr = *tslot;

    const uint32_t m0 = blockIdx.x * kTcRows;
    const uint32_t HW = a.h * a.w_;
    const uint32_t m = m0 + tid;
    const bool rowValid = m < a.M;
    const uint32_t img = rowValid ? m / HW : 0u, rem = rowValid ? m - img * HW : 0u;
    const int py = (int)(rem / a.w_), px = (int)(rem - (rem / a.w_) * a.w_);
    const uint32_t chunks = (a.cin + 63u) / 64u;
    const uint32_t kIters = 9u * chunks;
    // kind::f16 instruction descriptor: D f32, A and B bf16, both K-major, N, M = 128.
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((kTcRows >> 4) << 24);

    auto loadStage = [&](uint32_t it, uint32_t stage) {
        uint32_t tap = it / chunks, c0 = (it - tap * chunks) * 64u;
        int yy = py + (int)(tap / 3u) - 1, xx = px + (int)(tap % 3u) - 1;
        bool inb = rowValid && yy >= 0 && yy < (int)a.h && xx >= 0 && xx < (int)a.w_;
        const __nv_bfloat16* src =
            inb ? a.in + ((size_t)(img * a.h + (uint32_t)yy) * a.w_ + (uint32_t)xx) * a.ldi + c0 : a.in;
        unsigned char* rowA = sA + stage * aBytes + tid * 128u;
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            bool v = inb && c0 + j * 8u < a.cin;
            cpAsync16(rowA + ((j ^ (tid & 7u)) << 4), v ? src + j * 8u : a.in, v ? 16u : 0u);
        }
        unsigned char* tileB = sB + stage * bBytes;
        for (uint32_t i = tid; i < N * 8u; i += 128u) {
            uint32_t row = i >> 3, j = i & 7u;
            bool v = c0 + j * 8u < a.cin;
            const __nv_bfloat16* wsrc = a.w + ((size_t)row * 9u + tap) * a.cin + c0 + j * 8u;
            cpAsync16(tileB + row * 128u + ((j ^ (row & 7u)) << 4), v ? wsrc : a.w, v ? 16u : 0u);
        }
    };

    bool failed = false;
    uint32_t lastCommitted = 0xffffffffu;
#pragma unroll
    for (int s = 0; s < kTcStages - 1; ++s) {
        if ((uint32_t)s < kIters) loadStage((uint32_t)s, (uint32_t)s);
        cpAsyncCommit();
    }
    for (uint32_t it = 0; it < kIters && !failed; ++it) {
        const uint32_t stage = it % kTcStages;
        cpAsyncWait<kTcStages - 2>();
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t c0 = (it % chunks) * 64u;
            const uint32_t aBase = smemAddr(sA + stage * aBytes), bBase = smemAddr(sB + stage * bBytes);
#pragma unroll
            for (uint32_t ks = 0; ks < 4; ++ks) {
                if (c0 + ks * 16u >= a.cin) break;
                uint64_t ad = umaDesc(aBase + ks * 32u), bd = umaDesc(bBase + ks * 32u);
                uint32_t acc = (it > 0 || ks > 0) ? 1u : 0u;
                asm volatile(
                    "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(taddr),
                    "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                             smemAddr(&bars[stage]))
                         : "memory");
        }
        lastCommitted = it;
        const uint32_t nxt = it + kTcStages - 1;
        if (nxt < kIters) {
            const uint32_t ps = nxt % kTcStages;
            if (nxt >= (uint32_t)kTcStages) {  // the buffer's previous MMAs (iteration nxt - stages) must be done
                uint32_t use = (nxt - kTcStages) / kTcStages;
                if (!mbarWait(smemAddr(&bars[ps]), use & 1u)) failed = true;
            }
            if (!failed) loadStage(nxt, ps);
        }
        cpAsyncCommit();
    }
    cpAsyncWait<0>();
    bool done = false;
    if (lastCommitted != 0xffffffffu)
        done = mbarWait(smemAddr(&bars[lastCommitted % kTcStages]), (lastCommitted / kTcStages) & 1u);
    if (!done || failed) {
        if (tid == 0) atomicExch(&g_unetError, 1);
    } else {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const uint32_t row = warp * 32u + lane;
        const uint32_t pix = m0 + row;
        __nv_bfloat16* orow = a.out + (size_t)pix * a.ldo + a.coOff;
        for (uint32_t c0 = 0; c0 < N; c0 += 16u) {
            uint32_t r[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                "%14, %15}, [%16];\n"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                : "r"(taddr + ((warp * 32u) << 16) + c0));
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
            if (pix >= a.M) continue;
#pragma unroll
            for (uint32_t k = 0; k < 16; k += 2) {
                float v0 = __uint_as_float(r[k]), v1 = __uint_as_float(r[k + 1]);
                uint32_t col = c0 + k;
                if (a.bias) {
                    v0 += a.bias[col];
                    v1 += a.bias[col + 1];
                }
                if (a.act == 1) {
                    v0 = fmaxf(v0, 0.0f);
                    v1 = fmaxf(v1, 0.0f);
                }
                __nv_bfloat162* dst = reinterpret_cast<__nv_bfloat162*>(orow + col);
                if (a.accumulate) {
                    float2 o = __bfloat1622float2(*dst);
                    v0 += o.x;
                    v1 += o.y;
                }
                *dst = __floats2bfloat162_rn(v0, v1);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(tmemCols));
}

size_t tcSmemBytes(uint32_t cout) { return (size_t)kTcStages * (kTcRows * 128u + cout * 128u) + 1024u + 64u; }

// ------------------------------------------- tcgen05 + TMA, persistent ----
// The convolution of the layers that neither the halo-row nor the tile kernel
// below takes.  Persistent CTAs (one per SM) walk output
// tiles of 128 pixels (th image rows x tw columns, tw a power of two <= 128)
// with three warp roles:
//   warp 0     TMA producer: per (tap, 64-channel chunk) one 4-D box of the
//              activation tensor {64 ch, tw, th, 1} at the tap-shifted
//              coordinate (out-of-range pixels and channels are zero filled
//              by the copy engine) and one 3-D box of the weights
//              {64 ch, 1 tap, Cout}, both into 128-byte-swizzled K-major tiles;
//   warp 1     MMA issuer: tcgen05.mma M = 128, N = Cout, K = 16 into one of
//              the tensor-memory accumulators, stage release and
//              accumulator hand-off through tcgen05.commit;
//   warps 2-9  epilogue: tcgen05.ld of their TMEM lane quarter (two warps
//              per quarter, each half of the channels), bias, ReLU, optional
//              accumulate, bf16 stores; the next tiles' MMAs run into the
//              other accumulators (up to four) meanwhile.
// Every mbarrier wait is bounded (about 2 s); a role that times out records
// the error and stops, the others then time out in turn, and the CTA frees
// its tensor memory before returning.
constexpr uint32_t kHaloPix = 130;          // 128 output pixels and one on each side
constexpr uint32_t kHaloSlotBytes = 17408;  // 130 rows of 128 B, padded to 17 x 1024 B
constexpr uint32_t kTmaStagesMin = 4;   // (tap, chunk) stages in flight: at least 4,
constexpr uint32_t kTmaStagesMax = 8;   // more where shared memory holds them
constexpr uint32_t kTmaBarBytes = 256;  // full[8] empty[8] accFull[4] accEmpty[4], TMEM slot, flag

struct TmaConvArgs {
    const float* bias;
    __nv_bfloat16* out;
    uint32_t n, h, w, cin, cout, ldo, coOff, tw, th, tilesX, tilesY, numTiles, chunks, cols;
    uint32_t stages;  // kTmaStagesMin..kTmaStagesMax
    int act, accumulate;
    int staged;  // epilogue rows through shared memory (see epilogueRow)
};

__device__ __forceinline__ void mbarInit(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbarArrive(uint32_t bar) {
    asm volatile("{\n.reg .b64 st;\nmbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbarExpectTx(uint32_t bar, uint32_t bytes) {
    asm volatile("{\n.reg .b64 st;\nmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}\n" ::"r"(bar),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void tmaLoad4(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                         uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];\n" ::"r"(dst),
        "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tmaLoad3(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(dst),
        "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void umaCommit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
                 : "memory");
}

// The epilogue: eight warps, two per tensor-memory lane quarter (32 output
// pixels each).  When Cout is a multiple of 32 the two warps of a quarter
// split every accumulator's channels in halves; otherwise the first takes all
// of them and the second has nothing to do.  Up to four accumulators (as many
// as tensor memory holds, at least two) let the MMA warp run ahead of them.
constexpr uint32_t kEpiWarps = 8;
__host__ __device__ constexpr bool epiSplit(uint32_t n) { return n % 32u == 0u; }
__host__ __device__ constexpr uint32_t epiCols(uint32_t n) { return epiSplit(n) ? n / 2u : n; }
// Shared memory one epilogue warp uses to transpose its part of an output
// row: 32 pixels of its channels at a pitch of 2 x channels + 16 bytes (an odd
// number of 16-byte units, so eight lanes' 16-byte writes fall on distinct
// banks), then the 32 pixels' global row pointers.
__host__ __device__ constexpr uint32_t epiPitch(uint32_t cols) { return 2u * cols + 16u; }
__host__ __device__ constexpr uint32_t epiWarpBytes(uint32_t n) { return 32u * epiPitch(epiCols(n)) + 32u * 8u; }
// The same for a warp that takes all N channels of its rows.
__host__ __device__ constexpr uint32_t epiWarpBytesAll(uint32_t n) { return 32u * epiPitch(n) + 32u * 8u; }
__host__ __device__ constexpr uint32_t accBuffers(uint32_t cols) { return 4u * cols <= 512u ? 4u : 2u; }

// This warp's channels [c0, c1) of one accumulator (its 32 TMEM lanes: 32
// output pixels) to global memory: bias, ReLU, bf16, optionally added to the
// destination.  `src` is the accumulator's TMEM address for the warp's lane
// quarter, `dst` this lane's pixel (its channel 0), nullptr outside the image.
// With `stage` the warp writes its part of the row into shared memory and then
// stores every pixel's channels as 16-byte pieces by consecutive lanes, and
// hands the accumulator back as soon as it is read; `stage` is null when the
// destination is accumulated into (its bf16 sum is formed from the FP32
// value, as on the direct path) or not 16-byte aligned.  With `zero` the
// warp clears the columns it read before handing the accumulator back.
__device__ __forceinline__ void zeroColumns(uint32_t src, uint32_t c0, uint32_t c1) {
    const uint32_t z = 0u;
    for (uint32_t c = c0; c < c1; c += 16u)
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
            "%1, %1};\n" ::"r"(src + c),
            "r"(z)
            : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
}

__device__ __forceinline__ void epilogueRow(uint32_t src, uint32_t c0, uint32_t c1, const float* bias, int act,
                                            int accumulate, __nv_bfloat16* dst, unsigned char* stage,
                                            uint32_t accEmptyBar, bool zero = false) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t pitch = epiPitch(c1 - c0);
    const bool biasVec = bias && (reinterpret_cast<uintptr_t>(bias) & 15u) == 0u;
    for (uint32_t c = c0; c < c1; c += 16u) {
        uint32_t rr[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
            "%12, %13, %14, %15}, [%16];\n"
            : "=r"(rr[0]), "=r"(rr[1]), "=r"(rr[2]), "=r"(rr[3]), "=r"(rr[4]), "=r"(rr[5]), "=r"(rr[6]), "=r"(rr[7]),
              "=r"(rr[8]), "=r"(rr[9]), "=r"(rr[10]), "=r"(rr[11]), "=r"(rr[12]), "=r"(rr[13]), "=r"(rr[14]),
              "=r"(rr[15])
            : "r"(src + c));
        float bv[16];
        if (biasVec) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float4 b4 = __ldg(reinterpret_cast<const float4*>(bias + c) + k);
                bv[4 * k] = b4.x;
                bv[4 * k + 1] = b4.y;
                bv[4 * k + 2] = b4.z;
                bv[4 * k + 3] = b4.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 16; ++k) bv[k] = bias ? __ldg(bias + c + k) : 0.0f;
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        float v2[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            float x = __uint_as_float(rr[k]);
            if (bias) x += bv[k];
            if (act == 1) x = fmaxf(x, 0.0f);
            v2[k] = x;
        }
        if (stage) {
            uint32_t packed[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                __nv_bfloat162 h2 = __floats2bfloat162_rn(v2[2 * k], v2[2 * k + 1]);
                packed[k] = *reinterpret_cast<uint32_t*>(&h2);
            }
            uint4* sp = reinterpret_cast<uint4*>(stage + lane * pitch + (c - c0) * 2u);
            sp[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            sp[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
            continue;
        }
        if (!dst) continue;
        __nv_bfloat162* d2 = reinterpret_cast<__nv_bfloat162*>(dst + c);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float x0v = v2[2 * k], x1v = v2[2 * k + 1];
            if (accumulate) {
                float2 o = __bfloat1622float2(d2[k]);
                x0v += o.x;
                x1v += o.y;
            }
            d2[k] = __floats2bfloat162_rn(x0v, x1v);
        }
    }
    if (zero) zeroColumns(src, c0, c1);  // the next row in this accumulator slot starts from zero
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    mbarArrive(accEmptyBar);
    if (!stage) return;
    __nv_bfloat16** rows = reinterpret_cast<__nv_bfloat16**>(stage + 32u * pitch);
    rows[lane] = dst ? dst + c0 : nullptr;
    __syncwarp();
    // 16-byte pieces: `per` per pixel; lane j takes pieces j, j + 32, ...
    const uint32_t per = (c1 - c0) / 8u;
    const bool pow2 = (per & (per - 1u)) == 0u;
    const uint32_t sh = 31u - __clz(per);
    uint32_t pix = pow2 ? lane >> sh : lane / per;
    uint32_t part = lane - pix * per;
    const uint32_t dq = pow2 ? 32u >> sh : 32u / per, dr = 32u - dq * per;
    for (; pix < 32u; pix += dq) {
        __nv_bfloat16* d = rows[pix];
        if (d) *reinterpret_cast<uint4*>(d + part * 8u) = *reinterpret_cast<const uint4*>(stage + pix * pitch + part * 16u);
        part += dr;
        if (part >= per) {
            part -= per;
            ++pix;
        }
    }
    __syncwarp();
}

// A row-tap stage's K steps: for dx = 0, 1, 2 the A operand is the stage's
// input row from pixel dx on (128 bytes further per pixel) and the B operand
// the weights of tap (dy, dx); steps past a partial last chunk are predicated
// off.
//
// kRowTap (images at least 128 pixels wide): an output tile is 128 pixels of
// one row and a pipeline stage is (dy, 64-channel chunk): one box of the input
// row y + dy - 1, 130 pixels wide, and the weights of the three taps (dy, 0..2),
// so a tile takes 3 x chunks stages and waits instead of 9 x chunks.
template <bool kRowTap>
__global__ void __launch_bounds__(320, 1)
    k_conv3x3_tma(const __grid_constant__ CUtensorMap mapIn, const __grid_constant__ CUtensorMap mapW, TmaConvArgs a) {
    extern __shared__ unsigned char dsm[];
    const uint32_t raw = smemAddr(dsm);
    unsigned char* sm = dsm + (((raw + 1023u) & ~1023u) - raw);
    const uint32_t N = a.cout;
    const uint32_t aBytes = kRowTap ? kHaloSlotBytes : 128u * 128u, bBytes = (kRowTap ? 3u : 1u) * N * 128u;
    unsigned char* sA = sm;
    const uint32_t S = a.stages;
    unsigned char* sB = sm + S * aBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sB + S * bBytes);
    // bars: full[S], empty[S], accFull[4], accEmpty[4]
    const uint32_t fullBar = smemAddr(bars), emptyBar = fullBar + 8u * kTmaStagesMax;
    const uint32_t accFullBar = emptyBar + 8u * kTmaStagesMax, accEmptyBar = accFullBar + 32u;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 2 * kTmaStagesMax + 8);
    const uint32_t nbuf = accBuffers(a.cols), bufShift = nbuf == 4u ? 2u : 1u;
    int* abortFlag = reinterpret_cast<int*>(tslot + 1);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smemAddr(tslot)),
                     "r"(nbuf * a.cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        for (uint32_t s = 0; s < S; ++s) {
            mbarInit(fullBar + 8u * s, 1);
            mbarInit(emptyBar + 8u * s, 1);
        }
        for (uint32_t b = 0; b < nbuf; ++b) {
            mbarInit(accFullBar + 8u * b, 1);
            mbarInit(accEmptyBar + 8u * b, epiSplit(N) ? 256u : 128u);
        }
        *abortFlag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&mapIn) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&mapW) : "memory");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    pdlRelease();
    pdlWait();
    const uint32_t taddr = __shfl_sync(0xffffffffu, *tslot, 0);
    const uint32_t txBytes = (kRowTap ? kHaloPix * 128u : aBytes) + bBytes;
    volatile int* abortV = abortFlag;

    if (warp == 0 && kRowTap) {
        if (lane == 0) {
            uint32_t g = 0;
            RingPos pos{0u, 0u};
            bool ok = true;
            for (uint32_t tile = blockIdx.x; ok && tile < a.numTiles && !*abortV; tile += gridDim.x) {
                uint32_t tx = tile % a.tilesX, rest = tile / a.tilesX;
                uint32_t ty = rest % a.tilesY, img = rest / a.tilesY;
                int x0 = (int)(tx * 128u), y0 = (int)ty;
                for (uint32_t dy = 0; ok && dy < 3u; ++dy) {
                    for (uint32_t c = 0; c < a.chunks; ++c, ++g, pos.advance(S)) {
                        if (g >= S && !mbarWait(emptyBar + 8u * pos.slot, pos.phase ^ 1u)) {
                            ok = false;
                            break;
                        }
                        const uint32_t full = fullBar + 8u * pos.slot;
                        mbarExpectTx(full, txBytes);
                        tmaLoad4(smemAddr(sA + pos.slot * aBytes), &mapIn, (int)(c * 64u), x0 - 1, y0 + (int)dy - 1,
                                 (int)img, full);
                        for (uint32_t dx = 0; dx < 3u; ++dx)
                            tmaLoad3(smemAddr(sB + pos.slot * bBytes + dx * N * 128u), &mapW, (int)(c * 64u),
                                     (int)(dy * 3u + dx), 0, full);
                    }
                }
            }
            if (!ok) *abortV = 1;
        }
    } else if (warp == 0) {
        if (lane == 0) {
            uint32_t g = 0;
            RingPos pos{0u, 0u};
            bool ok = true;
            for (uint32_t tile = blockIdx.x; ok && tile < a.numTiles && !*abortV; tile += gridDim.x) {
                uint32_t tx = tile % a.tilesX, rest = tile / a.tilesX;
                uint32_t ty = rest % a.tilesY, img = rest / a.tilesY;
                int x0 = (int)(tx * a.tw), y0 = (int)(ty * a.th);
                for (uint32_t tap = 0; ok && tap < 9u; ++tap) {
                    const int dy = (int)(tap / 3u), dx = (int)tap - 3 * dy;
                    for (uint32_t c = 0; c < a.chunks; ++c, ++g, pos.advance(S)) {
                        if (g >= S && !mbarWait(emptyBar + 8u * pos.slot, pos.phase ^ 1u)) {
                            ok = false;
                            break;
                        }
                        const uint32_t full = fullBar + 8u * pos.slot;
                        mbarExpectTx(full, txBytes);
                        tmaLoad4(smemAddr(sA + pos.slot * aBytes), &mapIn, (int)(c * 64u), x0 + dx - 1, y0 + dy - 1,
                                 (int)img, full);
                        tmaLoad3(smemAddr(sB + pos.slot * bBytes), &mapW, (int)(c * 64u), (int)tap, 0, full);
                    }
                }
            }
            if (!ok) *abortV = 1;
        }
    } else if (warp == 1) {
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((128u >> 4) << 24);
        const uint32_t hi = descHi(), aLo0 = descLo(smemAddr(sA)), bLo0 = descLo(smemAddr(sB));
        const uint32_t lastSteps = (a.cin - (a.chunks - 1u) * 64u + 15u) / 16u;
        RingPos pos{0u, 0u};
        uint32_t t = 0;
        bool ok = true;
        for (uint32_t tile = blockIdx.x; ok && tile < a.numTiles; tile += gridDim.x, ++t) {
            const uint32_t b = t & (nbuf - 1u), v = t >> bufShift;
            if (v > 0 && !mbarWaitWarp(accEmptyBar + 8u * b, (v - 1u) & 1u)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t dAddr = taddr + b * a.cols;
            uint32_t acc = 0u;
            for (uint32_t it = 0; ok && it < (kRowTap ? 3u : 9u); ++it) {
                for (uint32_t c = 0; c < a.chunks; ++c, pos.advance(S)) {
                    if (!mbarWaitWarp(fullBar + 8u * pos.slot, pos.phase)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    // K steps of 16 channels in this (tap, chunk): 4, fewer in a partial last chunk
                    const uint32_t steps = c + 1u < a.chunks ? 4u : lastSteps;
                    const uint32_t aLo = aLo0 + pos.slot * (aBytes >> 4), bLo = bLo0 + pos.slot * (bBytes >> 4);
                    if (electOne()) {
                        const uint32_t bTapU = (N * 128u) >> 4;
#pragma unroll
                        for (uint32_t dx = 0; dx < (kRowTap ? 3u : 1u); ++dx)
#pragma unroll
                            for (uint32_t ks = 0; ks < 4u; ++ks)
                                mmaF16If(ks < steps, dAddr, aLo + dx * 8u + 2u * ks, hi, bLo + dx * bTapU + 2u * ks, hi,
                                         idesc, (dx | ks) ? 1u : acc);
                        umaCommit(emptyBar + 8u * pos.slot);  // the stage is free once these MMAs are done
                    }
                    __syncwarp();
                    acc = 1u;
                }
            }
            if (ok && electOne()) umaCommit(accFullBar + 8u * b);  // the accumulator is complete
            __syncwarp();
        }
        if (!ok && lane == 0) *abortV = 1;
    } else {
        // Epilogue warps 2..9: TMEM lane quarter warp % 4, channel half (warp - 2) / 4.
        const uint32_t q = warp & 3u, half = (warp - 2u) >> 2;
        const uint32_t r = q * 32u + lane;
        const uint32_t cw = epiCols(N), c0 = half * cw, c1 = epiSplit(N) ? c0 + cw : (half ? 0u : N);
        unsigned char* stage =
            a.staged ? reinterpret_cast<unsigned char*>(bars) + kTmaBarBytes + (warp - 2u) * epiWarpBytes(N) : nullptr;
        uint32_t t = 0;
        for (uint32_t tile = blockIdx.x; c1 > c0 && tile < a.numTiles; tile += gridDim.x, ++t) {
            uint32_t b = t & (nbuf - 1u), v = t >> bufShift;
            if (!mbarWait(accFullBar + 8u * b, v & 1u)) {
                *abortV = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            uint32_t tx = tile % a.tilesX, rest = tile / a.tilesX;
            uint32_t ty = rest % a.tilesY, img = rest / a.tilesY;
            uint32_t px = tx * a.tw + r % a.tw, py = ty * a.th + r / a.tw;
            bool valid = px < a.w && py < a.h;
            __nv_bfloat16* orow = valid ? a.out + ((size_t)(img * a.h + py) * a.w + px) * a.ldo + a.coOff : nullptr;
            epilogueRow(taddr + ((q * 32u) << 16) + b * a.cols, c0, c1, a.bias, a.act, a.accumulate, orow, stage,
                        accEmptyBar + 8u * b);
        }
    }
    __syncthreads();
    if (*abortV && tid == 0) atomicExch(&g_unetError, 2);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(nbuf * a.cols));
}

size_t tmaSmemBytes(uint32_t cout, bool staged, uint32_t stages, bool rowTap) {
    const size_t stage = rowTap ? kHaloSlotBytes + 3u * cout * 128u : 128u * 128u + cout * 128u;
    return (size_t)stages * stage + 1024u + kTmaBarBytes + (staged ? kEpiWarps * epiWarpBytes(cout) : 0u);
}

// ------------------------------------- tcgen05 + TMA, 2-D halo tiles ----
// The convolution for the layers the halo-row kernel does not take (narrow
// images, or weights beyond one CTA's shared memory).  The per-tap kernel above
// re-reads every input pixel for each tap (9 x 16 KB a tile and chunk) and
// every tile re-reads the weights, and waits on L2 for both.  Here an output
// tile is 8 x 16 pixels and its input, 10 x 18 pixels per 64-channel chunk, is
// loaded once and stays for all nine taps: an MMA's A operand is sixteen groups
// of eight pixels, one image row apart (stride byte offset = the halo's row),
// starting at the tap's pixel.  With kT = 2 two tiles side by side share the
// halo and every weight box.  The weights stream through a ring in stages of
// three (tap, chunk) boxes, one run of straight-line MMAs each (stages of one
// box left the tensor core idle for 230 cycles a box: the 160-to-64-channel
// layer at 960 x 544 takes 118 us with three, 146 with one, and 135 with three
// waited for but released one by one); K steps past a partial last chunk are
// predicated off.  Few tiles split the output
// channels over CTAs.  Warps: 0 weights, 1 MMA, 2-9 epilogue, 10 input.
// The K order of an output is the replaced kernel's: (dy, chunk, dx) for images
// at least 128 pixels wide, (tap, chunk) for narrower ones.
constexpr uint32_t kTileW = 8u, kTileH = 16u;
constexpr uint32_t kTileChunksMax = 8u;
constexpr uint32_t kTilePairs = 3u;  // (tap, chunk) boxes of a weight stage
constexpr uint32_t kTileWStagesMax = 8u;
constexpr uint32_t kTileBars = 2u * kTileWStagesMax + 8u;
constexpr uint32_t kTileBarBytes = 8u * kTileBars + 9u * kTileChunksMax * 4u + 32u;
template <uint32_t kT>
__host__ __device__ constexpr uint32_t tilePitch() { return kT * kTileW + 2u; }  // halo pixels per row
template <uint32_t kT>
__host__ __device__ constexpr uint32_t tileChunkBytes() {
    return (tilePitch<kT>() * (kTileH + 2u) * 128u + 1023u) & ~1023u;
}

constexpr uint32_t kTileWStagesMin = 2u;
// The epilogue's staging: of four warps where the output channels are not split between two.
__host__ __device__ constexpr uint32_t tileStageBytes(uint32_t nB) {
    return (epiSplit(nB) ? kEpiWarps : kEpiWarps / 2u) * epiWarpBytes(nB);
}
struct TileConvArgs {
    const float* bias;
    __nv_bfloat16* out;
    uint32_t n, h, w, ldo, coOff;
    uint32_t tilesX, tilesY, items;  // groups of kT tiles; work items (image x tiles x channel blocks)
    uint32_t chunks, lastSteps, pairs, rowOrder;
    uint32_t nB, nSplit, cols;       // output channels per CTA, blocks of them, accumulator columns
    uint32_t aSlots, wStages;
    int act, accumulate, staged;
};

template <uint32_t kT>
__global__ void __launch_bounds__(352, 1)
    k_conv3x3_tile(const __grid_constant__ CUtensorMap mapIn, const __grid_constant__ CUtensorMap mapW,
                   TileConvArgs a) {
    constexpr uint32_t kPitch = tilePitch<kT>(), kChunk = tileChunkBytes<kT>();
    extern __shared__ unsigned char dsm[];
    const uint32_t raw = smemAddr(dsm);
    unsigned char* sm = dsm + (((raw + 1023u) & ~1023u) - raw);
    const uint32_t aBytes = a.chunks * kChunk, wBox = a.nB * 128u, wBytes = kTilePairs * wBox;
    unsigned char* sW = sm + a.aSlots * aBytes;
    unsigned char* sEpi = sW + a.wStages * wBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sEpi + (a.staged ? tileStageBytes(a.nB) : 0u));
    const uint32_t wFull = smemAddr(bars), wEmpty = wFull + 8u * kTileWStagesMax, aFull = wEmpty + 8u * kTileWStagesMax;
    const uint32_t aEmpty = aFull + 16u, accFull = aEmpty + 16u, accEmpty = accFull + 16u;
    uint32_t* table = reinterpret_cast<uint32_t*>(bars + kTileBars);  // the (tap, chunk) order of the weight boxes: tap | chunk << 8
    uint32_t* tslot = table + 9u * kTileChunksMax;
    int* abortFlag = reinterpret_cast<int*>(tslot + 1);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t tmemCols = 2u * kT * a.cols <= 64u ? 64u : 2u * kT * a.cols <= 128u ? 128u
                              : 2u * kT * a.cols <= 256u ? 256u : 512u;

    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smemAddr(tslot)),
                     "r"(tmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        for (uint32_t s = 0; s < a.wStages; ++s) {
            mbarInit(wFull + 8u * s, 1);
            mbarInit(wEmpty + 8u * s, 1);
        }
        for (uint32_t b = 0; b < 2u; ++b) {
            mbarInit(aFull + 8u * b, 1);
            mbarInit(aEmpty + 8u * b, 1);
            mbarInit(accFull + 8u * b, 1);
            mbarInit(accEmpty + 8u * b, kT * (epiSplit(a.nB) ? 256u : 128u));
        }
        *abortFlag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&mapIn) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&mapW) : "memory");
    }
    if (tid < a.pairs) {
        uint32_t tap, c;
        if (a.rowOrder) {  // (dy, chunk, dx)
            const uint32_t dy = tid / (3u * a.chunks), rest = tid - dy * 3u * a.chunks;
            c = rest / 3u;
            tap = 3u * dy + rest - 3u * c;
        } else {  // (tap, chunk)
            tap = tid / a.chunks;
            c = tid - tap * a.chunks;
        }
        table[tid] = tap | (c << 8);
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    pdlRelease();
    pdlWait();
    const uint32_t taddr = __shfl_sync(0xffffffffu, *tslot, 0);
    volatile int* abortV = abortFlag;
    const uint32_t stages = a.pairs / kTilePairs;  // weight stages of a work item

    if (warp == 0) {
        if (lane == 0) {  // weights
            uint32_t g = 0;
            RingPos pos{0u, 0u};
            bool ok = true;
            for (uint32_t item = blockIdx.x; ok && item < a.items && !*abortV; item += gridDim.x) {
                const int co0 = (int)((item % a.nSplit) * a.nB);
                for (uint32_t s = 0; s < stages; ++s, ++g, pos.advance(a.wStages)) {
                    if (g >= a.wStages && !mbarWait(wEmpty + 8u * pos.slot, pos.phase ^ 1u)) {
                        ok = false;
                        break;
                    }
                    const uint32_t full = wFull + 8u * pos.slot;
                    mbarExpectTx(full, wBytes);
#pragma unroll
                    for (uint32_t j = 0; j < kTilePairs; ++j) {
                        const uint32_t e = table[s * kTilePairs + j];
                        tmaLoad3(smemAddr(sW + pos.slot * wBytes + j * wBox), &mapW, (int)((e >> 8) * 64u),
                                 (int)(e & 255u), co0, full);
                    }
                }
            }
            if (!ok) *abortV = 1;
        }
    } else if (warp == 10) {
        if (lane == 0) {  // input halos
            RingPos pos{0u, 0u};
            uint32_t g = 0;
            for (uint32_t item = blockIdx.x; item < a.items && !*abortV; item += gridDim.x, ++g, pos.advance(a.aSlots)) {
                if (g >= a.aSlots && !mbarWait(aEmpty + 8u * pos.slot, pos.phase ^ 1u)) {
                    *abortV = 1;
                    break;
                }
                const uint32_t tile = item / a.nSplit, tx = tile % a.tilesX, rest = tile / a.tilesX;
                const uint32_t ty = rest % a.tilesY, img = rest / a.tilesY;
                const uint32_t full = aFull + 8u * pos.slot;
                mbarExpectTx(full, a.chunks * kPitch * (kTileH + 2u) * 128u);
                for (uint32_t c = 0; c < a.chunks; ++c)
                    tmaLoad4(smemAddr(sm + pos.slot * aBytes + c * kChunk), &mapIn, (int)(c * 64u),
                             (int)(tx * kT * kTileW) - 1, (int)(ty * kTileH) - 1, (int)img, full);
            }
        }
    } else if (warp == 1) {
        // MMAs
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((a.nB >> 3) << 17) | ((128u >> 4) << 24);
        const uint32_t bHi = descHi(), aHi = (bHi & ~0x3FFFu) | (kPitch * 8u);  // stride: a halo row, in 16 bytes
        const uint32_t aLo0 = descLo(smemAddr(sm)), bLo0 = descLo(smemAddr(sW));
        RingPos ap{0u, 0u}, wp{0u, 0u};
        uint32_t t = 0;
        bool ok = true;
        for (uint32_t item = blockIdx.x; ok && item < a.items; item += gridDim.x, ++t, ap.advance(a.aSlots)) {
            const uint32_t b = t & 1u, v = t >> 1;
            if ((v > 0 && !mbarWaitWarp(accEmpty + 8u * b, (v - 1u) & 1u)) ||
                !mbarWaitWarp(aFull + 8u * ap.slot, ap.phase)) {
                ok = false;
                break;
            }
            const uint32_t dAddr = taddr + b * kT * a.cols, aBase = aLo0 + ap.slot * (aBytes >> 4);
            uint32_t dy = 0u, dx = 0u, c = 0u, acc = 0u;  // the next (tap, chunk) pair
            for (uint32_t s = 0; s < stages; ++s, wp.advance(a.wStages)) {
                uint32_t aLo[kTilePairs], steps[kTilePairs];
#pragma unroll
                for (uint32_t j = 0; j < kTilePairs; ++j) {
                    aLo[j] = aBase + c * (kChunk >> 4) + (dy * kPitch + dx) * 8u;
                    steps[j] = c + 1u < a.chunks ? 4u : a.lastSteps;
                    if (a.rowOrder) {
                        if (++dx == 3u) {
                            dx = 0u;
                            if (++c == a.chunks) {
                                c = 0u;
                                ++dy;
                            }
                        }
                    } else if (++c == a.chunks) {
                        c = 0u;
                        if (++dx == 3u) {
                            dx = 0u;
                            ++dy;
                        }
                    }
                }
                if (!mbarWaitWarp(wFull + 8u * wp.slot, wp.phase)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t bBase = bLo0 + wp.slot * (wBytes >> 4);
                if (electOne()) {
#pragma unroll
                    for (uint32_t j = 0; j < kTilePairs; ++j)
#pragma unroll
                        for (uint32_t ks = 0; ks < 4u; ++ks)
#pragma unroll
                            for (uint32_t q = 0; q < kT; ++q)
                                mmaF16If(ks < steps[j], dAddr + q * a.cols, aLo[j] + q * (kTileW * 8u) + 2u * ks, aHi,
                                         bBase + j * (wBox >> 4) + 2u * ks, bHi, idesc, (j | ks) ? 1u : acc);
                    umaCommit(wEmpty + 8u * wp.slot);
                }
                __syncwarp();
                acc = 1u;
            }
            if (ok && electOne()) {
                umaCommit(aEmpty + 8u * ap.slot);
                umaCommit(accFull + 8u * b);
            }
            __syncwarp();
        }
        if (!ok && lane == 0) *abortV = 1;
    } else {
        // Epilogue warps 2..9: TMEM lane quarter warp % 4 (four rows of eight pixels), channel half (warp - 2) / 4.
        const uint32_t q = warp & 3u, half = (warp - 2u) >> 2, N = a.nB;
        const uint32_t cw = epiCols(N), c0 = half * cw, c1 = epiSplit(N) ? c0 + cw : (half ? 0u : N);
        unsigned char* stage = a.staged ? sEpi + (warp - 2u) * epiWarpBytes(N) : nullptr;
        uint32_t t = 0;
        for (uint32_t item = blockIdx.x; c1 > c0 && item < a.items; item += gridDim.x, ++t) {
            const uint32_t b = t & 1u, v = t >> 1;
            if (!mbarWait(accFull + 8u * b, v & 1u)) {
                *abortV = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t tile = item / a.nSplit, co0 = (item - tile * a.nSplit) * N;
            const uint32_t tx = tile % a.tilesX, rest = tile / a.tilesX, ty = rest % a.tilesY, img = rest / a.tilesY;
            const uint32_t py = ty * kTileH + q * 4u + (lane >> 3);
#pragma unroll
            for (uint32_t j = 0; j < kT; ++j) {
                const uint32_t px = (tx * kT + j) * kTileW + (lane & 7u);
                const bool valid = px < a.w && py < a.h;
                __nv_bfloat16* orow =
                    valid ? a.out + ((size_t)(img * a.h + py) * a.w + px) * a.ldo + a.coOff + co0 : nullptr;
                epilogueRow(taddr + ((q * 32u) << 16) + (b * kT + j) * a.cols, c0, c1, a.bias ? a.bias + co0 : nullptr,
                            a.act, a.accumulate, orow, stage, accEmpty + 8u * b);
            }
        }
    }
    __syncthreads();
    if (*abortV && tid == 0) atomicExch(&g_unetError, 5);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(tmemCols));
}

// -------------------------------------- tcgen05 + TMA, halo-row ring ----
// The convolution for wide, shallow layers (the full- and half-resolution
// levels of the U-Net, where the per-tap kernel above re-reads every input
// pixel nine times from L2 and waits on it).  An output tile is 128
// consecutive pixels of one image row; a persistent CTA walks its share of
// the output rows (an equal, contiguous range of the rows numbered image by
// image, tile column by tile column, top to bottom), down one tile column at
// a time, and keeps the input rows it needs in a ring
// of halo rows: one TMA box {64 channels, 130 pixels} per 64-channel chunk
// and input row, loaded once (zero filled outside the image).  For tap
// (dy, dx) the MMA's A operand is the 128 rows of halo row y - 1 + dy that
// start at pixel dx: a contiguous run of 128-byte rows inside the slot, so all
// nine taps read the same shared-memory rows and each input row crosses L2
// once per tile column.  The weights of the layer (9 x chunks boxes of
// {64 channels, Cout}) stay resident in shared memory for the whole launch.
//   warp 0     TMA producer: the weights once, then the halo rows in order;
//   warp 1     MMA issuer: per output row 9 taps x chunks x K-steps of
//              tcgen05.mma M = 128, N = Cout, K = 16 into one of the TMEM
//              accumulators; releases a halo row once its last reader is done;
//   warps 2-9  epilogue as in k_conv3x3_tma.
// Waits are bounded as there.
constexpr uint32_t kHaloRingMin = 4;        // halo-row slots: three rows in use and one loading at least,
constexpr uint32_t kHaloRingMax = 16;       // and as many more loading as shared memory holds
constexpr uint32_t kHaloBarBytes = 1024;    // full[16] empty[16] weights accFull[32] accEmpty[32], TMEM slot, flag
constexpr uint32_t kHaloAccMax = 32;

struct HaloConvArgs {
    const float* bias;
    __nv_bfloat16* out;
    uint32_t n, h, w, cin, cout, ldo, coOff;
    uint32_t tilesX, totalRows, chunks, cols;  // totalRows = n x tilesX x h output rows of 128 pixels
    uint32_t ring;  // halo-row slots, kHaloRingMin..kHaloRingMax
    uint32_t slots, logSlots;  // stacked variant: accumulator slots of Cout columns (a power of two)
    uint32_t tmaStore;         // stacked variant: output rows leave by TMA tensor stores (Cout 16, 32 or 64)
    int act, accumulate;
    int staged;  // epilogue rows through shared memory (see epilogueRow)
    // With tensor-store rows: the 2x2 average of the output (h, w even) is also
    // written here, [n][h / 2][w / 2][poolLd] (channels 0 .. Cout), or null.
    __nv_bfloat16* pool;
    uint32_t poolLd;
};

// One accumulator slot of the stacked halo kernel to global memory through a
// TMA tensor store: this warp's 32 pixels (TMEM lanes) x all N channels are
// staged as a box {N channels, 32 pixels} in shared memory, laid out with the
// store map's swizzle (16-byte chunk j of pixel row r at r * 2N + 16 (j ^ f(r)),
// f(r) the row's address bits 7.. -- XOR-swizzle over 2N-byte rows, which also
// keeps the eight lanes of a 16-byte store on distinct banks), then one lane
// issues the store of the box at (channel offset, pixel, row, image); pixels
// beyond the image width are clipped by the copy engine.  `buf` alternates
// between two boxes per warp: before writing one, the warp waits until the
// store issued from it two rows earlier has read it.
__device__ __forceinline__ void tmaStoreRow(uint32_t src, uint32_t N, const float* bias, int act,
                                            unsigned char* buf, uint32_t accEmptyBar, const CUtensorMap* mapOut,
                                            int cx, int px0, int py, int img) {
    const uint32_t lane = threadIdx.x & 31u;
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;\n" ::: "memory");
    __syncwarp();
    const uint32_t rowBytes = 2u * N;
    const uint32_t swzMask = (rowBytes >> 4) - 1u;                          // 16-byte chunks per row - 1
    const uint32_t f = ((lane * rowBytes) >> 7) & swzMask;                  // address bits 7.. of the row
    const bool biasVec = bias && (reinterpret_cast<uintptr_t>(bias) & 15u) == 0u;
    for (uint32_t c = 0; c < N; c += 16u) {
        uint32_t rr[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
            "%12, %13, %14, %15}, [%16];\n"
            : "=r"(rr[0]), "=r"(rr[1]), "=r"(rr[2]), "=r"(rr[3]), "=r"(rr[4]), "=r"(rr[5]), "=r"(rr[6]), "=r"(rr[7]),
              "=r"(rr[8]), "=r"(rr[9]), "=r"(rr[10]), "=r"(rr[11]), "=r"(rr[12]), "=r"(rr[13]), "=r"(rr[14]),
              "=r"(rr[15])
            : "r"(src + c));
        float bv[16];
        if (biasVec) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float4 b4 = __ldg(reinterpret_cast<const float4*>(bias + c) + k);
                bv[4 * k] = b4.x;
                bv[4 * k + 1] = b4.y;
                bv[4 * k + 2] = b4.z;
                bv[4 * k + 3] = b4.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 16; ++k) bv[k] = bias ? __ldg(bias + c + k) : 0.0f;
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        uint32_t packed[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float x0 = __uint_as_float(rr[2 * k]), x1 = __uint_as_float(rr[2 * k + 1]);
            if (bias) {
                x0 += bv[2 * k];
                x1 += bv[2 * k + 1];
            }
            if (act == 1) {
                x0 = fmaxf(x0, 0.0f);
                x1 = fmaxf(x1, 0.0f);
            }
            __nv_bfloat162 h2 = __floats2bfloat162_rn(x0, x1);
            packed[k] = *reinterpret_cast<uint32_t*>(&h2);
        }
        const uint32_t j = c >> 3;  // first 16-byte chunk of these 16 channels
        unsigned char* row = buf + lane * rowBytes;
        *reinterpret_cast<uint4*>(row + (((j) ^ f) << 4)) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        *reinterpret_cast<uint4*>(row + (((j + 1u) ^ f) << 4)) = make_uint4(packed[4], packed[5], packed[6], packed[7]);
    }
    zeroColumns(src, 0u, N);  // the next row in this accumulator slot starts from zero
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    mbarArrive(accEmptyBar);
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the box is visible to the copy engine
    __syncwarp();
    if (lane == 0) {
        asm volatile(
            "cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4}], [%5];\n" ::"l"(mapOut),
            "r"(cx), "r"(px0), "r"(py), "r"(img), "r"(smemAddr(buf))
            : "memory");
        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
    }
}

// The 2x2 average of the two rows a warp has just staged for tensor stores
// (`top`: row 2i, `bottom`: row 2i + 1; 32 pixels x N channels each, laid out
// as in tmaStoreRow): lane l takes pooled pixel l / 2 and half of its
// channels and writes them to `dst` (that pooled pixel's first channel, or
// null past the image's right edge).  The staged values are the output's
// bf16 bits, and the sum ((top-left + top-right) + bottom-left) +
// bottom-right, times 0.25, is the pooling kernel's own, so the result is the
// one a separate pooling pass over the stored output gives.  The boxes were
// written before the warp's last __syncwarp in tmaStoreRow; they are next
// overwritten after the next one.
__device__ __forceinline__ void poolPairRow(const unsigned char* top, const unsigned char* bottom, uint32_t N,
                                            __nv_bfloat16* dst) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t rowBytes = 2u * N, swzMask = (rowBytes >> 4) - 1u;
    const uint32_t left = lane & ~1u, right = left + 1u;
    const uint32_t fl = ((left * rowBytes) >> 7) & swzMask, fr = ((right * rowBytes) >> 7) & swzMask;
    const uint32_t per = N >> 4;  // 16-byte chunks (8 channels) per lane
    const uint32_t j0 = (lane & 1u) * per;
    for (uint32_t j = j0; j < j0 + per; ++j) {
        const uint4 tl = *reinterpret_cast<const uint4*>(top + left * rowBytes + ((j ^ fl) << 4));
        const uint4 tr = *reinterpret_cast<const uint4*>(top + right * rowBytes + ((j ^ fr) << 4));
        const uint4 bl = *reinterpret_cast<const uint4*>(bottom + left * rowBytes + ((j ^ fl) << 4));
        const uint4 br = *reinterpret_cast<const uint4*>(bottom + right * rowBytes + ((j ^ fr) << 4));
        const uint32_t a[4] = {tl.x, tl.y, tl.z, tl.w}, b[4] = {tr.x, tr.y, tr.z, tr.w};
        const uint32_t c[4] = {bl.x, bl.y, bl.z, bl.w}, d[4] = {br.x, br.y, br.z, br.w};
        uint32_t o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 s = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a[k]));
            const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&b[k]));
            const float2 u = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&c[k]));
            const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&d[k]));
            __nv_bfloat162 h2 = __floats2bfloat162_rn(0.25f * (s.x + t.x + u.x + v.x), 0.25f * (s.y + t.y + u.y + v.y));
            o[k] = *reinterpret_cast<uint32_t*>(&h2);
        }
        if (dst) *reinterpret_cast<uint4*>(dst + 8u * j) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// A run of output rows y0..y1-1 of tile column tx of image img.
struct RowSegment {
    uint32_t img, tx, y0, y1;
};
// The next segment of this CTA's rows [cur, end): the rest of the current
// tile column at most; false when the range is done.
__device__ __forceinline__ bool nextSegment(const HaloConvArgs& a, uint32_t& cur, uint32_t end, RowSegment& sg) {
    if (cur >= end) return false;
    const uint32_t col = cur / a.h;
    sg.y0 = cur - col * a.h;
    sg.y1 = min(a.h, sg.y0 + (end - cur));
    sg.tx = col % a.tilesX;
    sg.img = col / a.tilesX;
    cur += sg.y1 - sg.y0;
    return true;
}
// With pooling (h even), ranges hold whole row pairs, so that rows 2i and
// 2i + 1 of a tile column reach the same epilogue set one after the other.
__device__ __forceinline__ uint32_t rangeBegin(const HaloConvArgs& a, uint32_t cta) {
    if (a.pool) return 2u * (uint32_t)((uint64_t)cta * (a.totalRows >> 1) / gridDim.x);
    return (uint32_t)((uint64_t)cta * a.totalRows / gridDim.x);
}

// kC: 64-channel chunks of the input (Cin / 64 rounded up), kLast: K steps of
// 16 channels in the last chunk.  Both are compile-time so that each output
// row's MMAs are straight-line code: a branch between two tcgen05.mma costs
// the issuing warp a few hundred cycles (measured), about the time of a
// 128 x 32 x 16 MMA (40 cycles) ten times over.
template <bool kStack, uint32_t kC, uint32_t kLast>
__global__ void __launch_bounds__(320, 1)
    k_conv3x3_halo(const __grid_constant__ CUtensorMap mapIn, const __grid_constant__ CUtensorMap mapW,
                   const __grid_constant__ CUtensorMap mapOut, HaloConvArgs a) {
    extern __shared__ unsigned char dsm[];
    const uint32_t raw = smemAddr(dsm);
    unsigned char* sm = dsm + (((raw + 1023u) & ~1023u) - raw);
    const uint32_t N = a.cout, C = a.chunks;
    const uint32_t slotBytes = C * kHaloSlotBytes;
    const uint32_t wBoxBytes = N * 128u, wBytes = 9u * C * wBoxBytes;
    unsigned char* sRing = sm;
    const uint32_t R = a.ring;
    unsigned char* sW = sm + R * slotBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sW + wBytes);
    // bars: full[R], empty[R], weights, accFull[Q], accEmpty[Q]
    const uint32_t fullBar = smemAddr(bars), emptyBar = fullBar + 8u * kHaloRingMax;
    const uint32_t wBar = emptyBar + 8u * kHaloRingMax, accFullBar = wBar + 8u;
    const uint32_t accEmptyBar = accFullBar + 8u * kHaloAccMax;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 2 * kHaloRingMax + 1 + 2 * kHaloAccMax);
    // Accumulators: Q slots of Cout columns for the stacked variant (a rolling
    // window over the output rows), else nbuf buffers of `cols` columns.
    const uint32_t nbuf = kStack ? a.slots : accBuffers(a.cols);
    const uint32_t bufShift = kStack ? a.logSlots : (nbuf == 4u ? 2u : 1u);
    const uint32_t tmemCols = kStack ? 512u : nbuf * a.cols;
    int* abortFlag = reinterpret_cast<int*>(tslot + 1);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smemAddr(tslot)),
                     "r"(tmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        for (uint32_t s = 0; s < R; ++s) {
            mbarInit(fullBar + 8u * s, 1);
            mbarInit(emptyBar + 8u * s, 1);
        }
        mbarInit(wBar, 1);
        for (uint32_t b = 0; b < nbuf; ++b) {
            mbarInit(accFullBar + 8u * b, 1);
            mbarInit(accEmptyBar + 8u * b, (kStack || !epiSplit(N)) ? 128u : 256u);
        }
        *abortFlag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&mapIn) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&mapW) : "memory");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    pdlRelease();
    pdlWait();
    const uint32_t taddr = __shfl_sync(0xffffffffu, *tslot, 0);
    volatile int* abortV = abortFlag;

    if (warp == 0) {
        if (lane == 0) {
            mbarExpectTx(wBar, wBytes);
            // Stacked: per (dx, chunk) one tile of 3 x Cout weight rows, the taps
            // dy = 2, 1, 0 in that order (an MMA with N = 3 Cout then yields the
            // contributions of one halo row to output rows y - 2, y - 1, y).
            for (uint32_t tap = 0; tap < 9u; ++tap)
                for (uint32_t c = 0; c < C; ++c) {
                    const uint32_t dy = tap / 3u, dx = tap - 3u * dy;
                    const uint32_t box = kStack ? (dx * C + c) * 3u + (2u - dy) : tap * C + c;
                    tmaLoad3(smemAddr(sW + box * wBoxBytes), &mapW, (int)(c * 64u), (int)tap, 0, wBar);
                }
            uint32_t g = 0;
            RingPos pos{0u, 0u};
            uint32_t cur = rangeBegin(a, blockIdx.x);
            const uint32_t end = rangeBegin(a, blockIdx.x + 1u);
            RowSegment sg;
            while (!*abortV && nextSegment(a, cur, end, sg)) {
                const int x0 = (int)(sg.tx * 128u), y0 = (int)sg.y0, y1 = (int)sg.y1;
                const uint32_t img = sg.img;
                bool ok = true;
                for (int hy = y0 - 1; hy <= y1; ++hy, ++g, pos.advance(R)) {
                    if (g >= R && !mbarWait(emptyBar + 8u * pos.slot, pos.phase ^ 1u)) {
                        ok = false;
                        break;
                    }
                    const uint32_t full = fullBar + 8u * pos.slot;
                    mbarExpectTx(full, C * kHaloPix * 128u);
                    for (uint32_t c = 0; c < C; ++c)
                        tmaLoad4(smemAddr(sRing + pos.slot * slotBytes + c * kHaloSlotBytes), &mapIn, (int)(c * 64u),
                                 x0 - 1, hy, (int)img, full);
                }
                if (!ok) {
                    *abortV = 1;
                    break;
                }
            }
        }
    } else if (warp == 1 && kStack) {
        // Per halo row k of a segment of `rows` output rows: the row's
        // contributions to output rows k - 2, k - 1, k (taps dy = 2, 1, 0).
        // Between the segment's edges, and when the three rows' slots are
        // adjacent, that is one MMA per (dx, chunk, K step) with N = 3 Cout
        // into the three slots; otherwise one MMA with N = Cout per valid
        // row.  Slots start zeroed (the epilogue clears a slot when it has
        // read it), so every MMA accumulates.
        const uint32_t idesc1 = (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((128u >> 4) << 24);
        const uint32_t idesc3 = (1u << 4) | (1u << 7) | (1u << 10) | (((3u * N) >> 3) << 17) | ((128u >> 4) << 24);
        const uint32_t hi = descHi(), aLo0 = descLo(smemAddr(sRing)), bLo0 = descLo(smemAddr(sW));
        const uint32_t tileU = (3u * wBoxBytes) >> 4, dyU = wBoxBytes >> 4;  // in 16-byte units
        const uint32_t Q = nbuf;
        // One halo row's stacked MMAs (N = 3 Cout) into the slots from `d` on.
        auto stackedRow = [&](uint32_t aRow, uint32_t d) {
#pragma unroll
            for (uint32_t dx = 0; dx < 3u; ++dx)
#pragma unroll
                for (uint32_t c = 0; c < kC; ++c)
#pragma unroll
                    for (uint32_t ks = 0; ks < (c + 1u < kC ? 4u : kLast); ++ks)
                        mmaF16(d, aRow + dx * 8u + c * (kHaloSlotBytes >> 4) + 2u * ks,  // pixel dx: 128 B on
                               bLo0 + (dx * kC + c) * tileU + 2u * ks, hi, idesc3, 1u);
        };
        bool ok = mbarWaitWarp(wBar, 0u);
        uint32_t t0 = 0;      // output rows of the earlier segments
        RingPos hp{0u, 0u};   // the current halo row's ring slot
        uint32_t cur = rangeBegin(a, blockIdx.x);
        const uint32_t end = rangeBegin(a, blockIdx.x + 1u);
        RowSegment sg;
        while (ok && !__any_sync(0xffffffffu, *abortV) && nextSegment(a, cur, end, sg)) {
            const uint32_t rows = sg.y1 - sg.y0;
            for (uint32_t k = 0; k < rows + 2u;) {
                // Two interior halo rows at once when both stack into adjacent
                // slots: their waits first, then both rows' MMAs and commits as
                // one straight-line run (one branch per two rows).
                if (k >= 2u && k + 1u < rows && ((t0 + k - 2u) & (Q - 1u)) + 3u < Q) {
                    RingPos hp1 = hp;
                    hp1.advance(R);
                    const uint32_t t = t0 + k, sLo = (t0 + k - 2u) & (Q - 1u);
                    if (!mbarWaitWarp(accEmptyBar + 8u * (t & (Q - 1u)), (t >> bufShift) & 1u) ||
                        !mbarWaitWarp(accEmptyBar + 8u * ((t + 1u) & (Q - 1u)), ((t + 1u) >> bufShift) & 1u) ||
                        !mbarWaitWarp(fullBar + 8u * hp.slot, hp.phase) || !mbarWaitWarp(fullBar + 8u * hp1.slot, hp1.phase)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    if (electOne()) {
                        stackedRow(aLo0 + hp.slot * (slotBytes >> 4), taddr + sLo * N);
                        umaCommit(emptyBar + 8u * hp.slot);
                        umaCommit(accFullBar + 8u * sLo);
                        stackedRow(aLo0 + hp1.slot * (slotBytes >> 4), taddr + (sLo + 1u) * N);
                        umaCommit(emptyBar + 8u * hp1.slot);
                        umaCommit(accFullBar + 8u * (sLo + 1u));
                    }
                    __syncwarp();
                    k += 2u;
                    hp = hp1;
                    hp.advance(R);
                    continue;
                }
                if (k < rows) {  // output row k enters: its slot must have been read and cleared
                    const uint32_t t = t0 + k;
                    if (!mbarWaitWarp(accEmptyBar + 8u * (t & (Q - 1u)), (t >> bufShift) & 1u)) ok = false;
                }
                if (ok && !mbarWaitWarp(fullBar + 8u * hp.slot, hp.phase)) ok = false;
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t aRow = aLo0 + hp.slot * (slotBytes >> 4);
                const uint32_t jLo = k >= 2u ? k - 2u : 0u, jHi = min(k, rows - 1u);
                const uint32_t sLo = (t0 + jLo) & (Q - 1u);
                const bool stacked = k >= 2u && k < rows && sLo + 2u < Q;
                if (electOne()) {
                    if (stacked) stackedRow(aRow, taddr + sLo * N);
                    for (uint32_t j = jLo; !stacked && j <= jHi; ++j) {
                        const uint32_t dy = k - j;
                        const uint32_t d = taddr + ((t0 + j) & (Q - 1u)) * N;
#pragma unroll
                        for (uint32_t dx = 0; dx < 3u; ++dx)
#pragma unroll
                            for (uint32_t c = 0; c < kC; ++c)
#pragma unroll
                                for (uint32_t ks = 0; ks < (c + 1u < kC ? 4u : kLast); ++ks)
                                    mmaF16(d, aRow + dx * 8u + c * (kHaloSlotBytes >> 4) + 2u * ks,
                                           bLo0 + (dx * kC + c) * tileU + (2u - dy) * dyU + 2u * ks, hi, idesc1,
                                           1u);
                    }
                }
                if (electOne()) {
                    umaCommit(emptyBar + 8u * hp.slot);  // halo row k has no reader left
                    if (k >= 2u) umaCommit(accFullBar + 8u * ((t0 + k - 2u) & (Q - 1u)));  // row k - 2 is complete
                }
                __syncwarp();
                ++k;
                hp.advance(R);
            }
            t0 += rows;
        }
        if (!ok) *abortV = 1;
    } else if (warp == 1) {
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((128u >> 4) << 24);
        const uint32_t hi = descHi(), aLo0 = descLo(smemAddr(sRing)), bLo0 = descLo(smemAddr(sW));
        bool ok = mbarWaitWarp(wBar, 0u);
        uint32_t t = 0;
        RingPos top{0u, 0u};  // the item's first halo row
        uint32_t cur = rangeBegin(a, blockIdx.x);
        const uint32_t end = rangeBegin(a, blockIdx.x + 1u);
        RowSegment sg;
        while (ok && !__any_sync(0xffffffffu, *abortV) && nextSegment(a, cur, end, sg)) {
            const uint32_t rows = sg.y1 - sg.y0;
            // halo rows w0, w1, w2 feed the current output row
            RingPos w0 = top, w1 = top, w2;
            w1.advance(R);
            w2 = w1;
            w2.advance(R);
            if (!mbarWaitWarp(fullBar + 8u * w0.slot, w0.phase) || !mbarWaitWarp(fullBar + 8u * w1.slot, w1.phase))
                ok = false;
            for (uint32_t k = 0; ok && k < rows; ++k, ++t) {
                if (!mbarWaitWarp(fullBar + 8u * w2.slot, w2.phase)) ok = false;
                const uint32_t b = t & (nbuf - 1u), v = t >> bufShift;
                if (ok && v > 0 && !mbarWaitWarp(accEmptyBar + 8u * b, (v - 1u) & 1u)) ok = false;
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t dAddr = taddr + b * a.cols;
                // A run that starts inside the 1024-byte swizzle pattern (pixel dx)
                // takes the plain descriptor: the tensor core applies the 128-byte
                // swizzle to absolute shared-memory address bits, as the copy engine
                // wrote it (measured: a base offset of (start >> 7) & 7 gives wrong sums).
                const uint32_t rowLo[3] = {aLo0 + w0.slot * (slotBytes >> 4), aLo0 + w1.slot * (slotBytes >> 4),
                                           aLo0 + w2.slot * (slotBytes >> 4)};
                if (electOne()) {
#pragma unroll
                    for (uint32_t tap = 0; tap < 9u; ++tap) {
                        const uint32_t dy = tap / 3u, dx = tap - dy * 3u;
                        const uint32_t aT = rowLo[dy] + dx * 8u;  // pixel dx: 128 bytes further
                        const uint32_t bT = bLo0 + tap * kC * (wBoxBytes >> 4);
#pragma unroll
                        for (uint32_t c = 0; c < kC; ++c)
#pragma unroll
                            for (uint32_t ks = 0; ks < (c + 1u < kC ? 4u : kLast); ++ks)
                                mmaF16(dAddr, aT + c * (kHaloSlotBytes >> 4) + 2u * ks, bT + c * (wBoxBytes >> 4) + 2u * ks,
                                       hi, idesc, (tap | c | ks) ? 1u : 0u);
                    }
                    umaCommit(accFullBar + 8u * b);          // output row complete
                    umaCommit(emptyBar + 8u * w0.slot);      // its top halo row has no reader left
                }
                __syncwarp();
                w0 = w1;
                w1 = w2;
                w2.advance(R);
            }
            if (!ok) break;
            if (electOne()) {
                umaCommit(emptyBar + 8u * w0.slot);  // the item's last two halo rows
                umaCommit(emptyBar + 8u * w1.slot);
            }
            __syncwarp();
            top = w2;
        }
        if (!ok) *abortV = 1;
    } else {
        // Epilogue warps 2..9: TMEM lane quarter warp % 4 (one output pixel per
        // thread); set (warp - 2) / 4.  Stacked: set s takes every channel of
        // the rows of parity s (and owns the accumulator slots of that parity:
        // the slot count is even), two rows in flight -- with pooling, of the
        // row pairs of parity s (slot count a multiple of 4); otherwise both
        // sets take every row, each half of the channels.
        const uint32_t q = warp & 3u, set = (warp - 2u) >> 2;
        const uint32_t r = q * 32u + lane;
        const uint32_t cw = epiCols(N);
        const uint32_t c0 = kStack ? 0u : set * cw, c1 = kStack ? N : (epiSplit(N) ? c0 + cw : (set ? 0u : N));
        unsigned char* stage = a.staged ? reinterpret_cast<unsigned char*>(bars) + kHaloBarBytes +
                                              (warp - 2u) * (kStack ? epiWarpBytesAll(N) : epiWarpBytes(N))
                                        : nullptr;
        uint32_t t = 0;
        bool ok = c1 > c0;
        const uint32_t quarter = taddr + ((q * 32u) << 16);
        const uint32_t slotCols = kStack ? N : a.cols;
        const uint32_t pairShift = a.pool ? 1u : 0u;  // rows (or row pairs) alternate between the sets
        if (kStack) {
            // Every slot starts zeroed; its first release lets the MMA warp in.
            for (uint32_t b = 0; b < nbuf; ++b)
                if (((b >> pairShift) & 1u) == set) zeroColumns(quarter + b * slotCols, c0, c1);
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            for (uint32_t b = 0; b < nbuf; ++b)
                if (((b >> pairShift) & 1u) == set) mbarArrive(accEmptyBar + 8u * b);
        }
        uint32_t cur = rangeBegin(a, blockIdx.x);
        const uint32_t end = rangeBegin(a, blockIdx.x + 1u);
        RowSegment sg;
        // Stacked with TMA stores: two boxes of 32 pixels x N channels per warp.
        unsigned char* boxes = reinterpret_cast<unsigned char*>(bars) + kHaloBarBytes + (warp - 2u) * 128u * N;
        uint32_t stored = 0;
        while (ok && nextSegment(a, cur, end, sg)) {
            const uint32_t img = sg.img, px = sg.tx * 128u + r;
            for (uint32_t py = sg.y0; py < sg.y1; ++py, ++t) {
                if (kStack && ((t >> pairShift) & 1u) != set) continue;  // the other set's row
                if (kStack && a.tmaStore) {
                    const uint32_t b = t & (nbuf - 1u), v = t >> bufShift;
                    if (!mbarWait(accFullBar + 8u * b, v & 1u)) {
                        *abortV = 1;
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t box = stored & 1u;
                    tmaStoreRow(quarter + b * slotCols, N, a.bias, a.act, boxes + box * 64u * N, accEmptyBar + 8u * b,
                                &mapOut, (int)a.coOff, (int)(sg.tx * 128u + q * 32u), (int)py, (int)img);
                    ++stored;
                    if (a.pool && (py & 1u)) {  // rows py - 1 and py are in this warp's two boxes
                        const uint32_t left = sg.tx * 128u + q * 32u + (lane & ~1u);
                        __nv_bfloat16* dst =
                            left < a.w ? a.pool + ((size_t)(img * (a.h >> 1) + (py >> 1)) * (a.w >> 1) + (left >> 1)) *
                                                      a.poolLd
                                       : nullptr;
                        poolPairRow(boxes + (box ^ 1u) * 64u * N, boxes + box * 64u * N, N, dst);
                    }
                    continue;
                }
                const uint32_t b = t & (nbuf - 1u), v = t >> bufShift;
                if (!mbarWait(accFullBar + 8u * b, v & 1u)) {
                    *abortV = 1;
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                __nv_bfloat16* orow =
                    px < a.w ? a.out + ((size_t)(img * a.h + py) * a.w + px) * a.ldo + a.coOff : nullptr;
                epilogueRow(quarter + b * slotCols, c0, c1, a.bias, a.act, a.accumulate, orow, stage,
                            accEmptyBar + 8u * b, kStack);
            }
        }
        if (kStack && a.tmaStore && lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    if (*abortV && tid == 0) atomicExch(&g_unetError, 3);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(tmemCols));
}

size_t haloSmemBytes(uint32_t cout, uint32_t chunks, bool staged, uint32_t ring, bool stack, bool tmaStore = false) {
    const size_t epi = tmaStore ? kEpiWarps * 128u * cout  // two boxes of 32 pixels x Cout per warp
                                : (staged ? kEpiWarps * (stack ? epiWarpBytesAll(cout) : epiWarpBytes(cout)) : 0u);
    return 1024u + (size_t)ring * chunks * kHaloSlotBytes + 9u * (size_t)chunks * cout * 128u + kHaloBarBytes + epi;
}

// -------------------------------------------------------------- wgrad ----
// dW[co][tap][ci] += sum_p dOut[p][co] in[p + tap][ci] on the tensor cores:
// K = pixels, so both operands are read "MN-major" straight from NHWC tiles
// (the channels of a pixel are contiguous, the pixels are the K index).
//   A (M = 128)  four horizontal taps x 32 input channels: rows of 64 bytes
//                (32 channels, 64-byte swizzle), the next tap's block one pixel
//                further (leading byte offset 64), so one MMA covers dx = 0, 1,
//                2 of a vertical tap; the fourth block is the price of M = 128
//                and its rows are not read back;
//   B (N = coB)  the output gradient's channels in blocks of 32.
// A persistent CTA owns `cpc` blocks of 32 input channels and up to 160 output
// channels (3 x cpc x coB <= 512 accumulator columns, one set per vertical tap)
// and walks 16 x 16 pixel tiles: per tile one box {32 channels, 18, 18} per
// input block and one {32 channels, 16, 16} per output block, zero filled
// outside the image, then 16 K steps x 3 vertical taps of straight-line MMAs
// per input block.  The sums stay in tensor memory over all of a CTA's tiles
// (at most 64 to a set of accumulators, 1,024 K steps; launchWgrad) and are
// added to dW once, 32 consecutive input channels per warp instruction.
// Bound: shared-memory operand reads at 32 output channels (4 KB of A per MMA),
// and 10 to 20 us of set-up and read-out, which small problems avoid
// (k_conv3x3_wgrad_mma).  Measured over the 19 layers of a 16 x 256^2 training
// step: 694 us, two of the layers on mma.sync; all of them there took 4218 us.
// The tensor core truncates, so the error against 64 bits grows with the K steps
// of a sum: 1.8e-7 to 1.2e-5 on those gradients and 2.2e-5 for 96 to 32 channels,
// 1.8e-7 to 2.7e-5 on mma.sync, no layer above it there.
// An infinite or NaN activation in the last column or row of an image that ends
// inside a tile reaches all nine taps' sums of its channel, through its products
// with the zero fill; elsewhere the taps whose pixels are in the image.
struct WgradArgs {
    float* dw;  // [cout][9][cin], accumulated
    uint32_t cin, cout, tilesX, tilesY, numTiles;
    uint32_t chunks, cpc, ciGroups;  // 32-channel input blocks: in all, per CTA; groups of them
    uint32_t coB, coChunks;          // output channels per CTA and their 32-channel blocks
    uint32_t stages, cols;
    uint32_t n, w, h, sets;          // accumulator sets, which take a CTA's tiles in turn
};
constexpr uint32_t kWgTile = 16u;                                   // tile edge in pixels
constexpr uint32_t kWgHalo = kWgTile + 2u;
constexpr uint32_t kWgInBytes = kWgHalo * kWgHalo * 64u;            // one input box
constexpr uint32_t kWgInSlot = (kWgInBytes + 64u + 1023u) & ~1023u;  // + the fourth tap's last pixel
constexpr uint32_t kWgOutSlot = kWgTile * kWgTile * 64u;
constexpr uint32_t kWgStagesMax = 4u;
constexpr uint32_t kWgBarBytes = 128u;
constexpr uint32_t kWgCoMax = 160u;
constexpr uint32_t kWgRunMax = 64u;  // tiles of one sum

// Image and first pixel of a tile.  The order goes by kind -- whole tiles, then those cut by the right edge, by the
// lower edge, by both -- so that the tiles of a CTA, gridDim.x apart, hold the same share of every kind: in row
// order two CTAs' sums may hold the whole tiles and the slivers of an image 17 pixels wide.
__device__ __forceinline__ void wgradTile(const WgradArgs& a, uint32_t tile, uint32_t& img, int& x0, int& y0) {
    const uint32_t fx = a.w / kWgTile, fy = a.h / kWgTile;
    uint32_t nx = fx, ny = fy, bx = 0u, by = 0u;
    if (tile >= a.n * fx * fy) {
        tile -= a.n * fx * fy;
        const uint32_t right = a.tilesX > fx ? a.n * fy : 0u, lower = a.tilesY > fy ? a.n * fx : 0u;
        nx = 1u;
        bx = fx;
        if (tile >= right) {
            tile -= right;
            nx = fx;
            bx = 0u;
            ny = 1u;
            by = fy;
            if (tile >= lower) {
                tile -= lower;
                nx = 1u;
                bx = fx;
            }
        }
    }
    const uint32_t tx = tile % nx, rest = tile / nx, ty = rest % ny;
    img = rest / ny;
    x0 = (int)((bx + tx) * kWgTile);
    y0 = (int)((by + ty) * kWgTile);
}

// Sixteen accumulator columns of a warp's lanes.
__device__ __forceinline__ void wgradLoad(uint32_t taddr, float (&f)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
        "%12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int k = 0; k < 16; ++k) f[k] = __uint_as_float(r[k]);
}

__global__ void __launch_bounds__(128, 1)
    k_conv3x3_wgrad(const __grid_constant__ CUtensorMap mapIn, const __grid_constant__ CUtensorMap mapOut,
                    WgradArgs a) {
    extern __shared__ unsigned char dsm[];
    const uint32_t raw = smemAddr(dsm);
    unsigned char* sm = dsm + (((raw + 1023u) & ~1023u) - raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t coBlock = blockIdx.y / a.ciGroups, chunk0 = (blockIdx.y - coBlock * a.ciGroups) * a.cpc;
    const uint32_t co0 = coBlock * a.coB, nc = min(a.cpc, a.chunks - chunk0);
    const uint32_t stageBytes = a.cpc * kWgInSlot + a.coChunks * kWgOutSlot;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm + a.stages * stageBytes);
    const uint32_t fullBar = smemAddr(bars), emptyBar = fullBar + 8u * kWgStagesMax;
    const uint32_t doneBar = emptyBar + 8u * kWgStagesMax;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 2u * kWgStagesMax + 1u);
    int* abortFlag = reinterpret_cast<int*>(tslot + 1);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smemAddr(tslot)),
                     "r"(a.cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        for (uint32_t s = 0; s < a.stages; ++s) {
            mbarInit(fullBar + 8u * s, 1);
            mbarInit(emptyBar + 8u * s, 1);
        }
        mbarInit(doneBar, 1);
        *abortFlag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&mapIn) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&mapOut) : "memory");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t taddr = __shfl_sync(0xffffffffu, *tslot, 0);
    volatile int* abortV = abortFlag;

    if (tid == 0) {  // TMA producer
        const uint32_t txBytes = nc * kWgInBytes + a.coChunks * kWgOutSlot;
        RingPos pos{0u, 0u};
        uint32_t g = 0;
        for (uint32_t tile = blockIdx.x; tile < a.numTiles && !*abortV; tile += gridDim.x, ++g, pos.advance(a.stages)) {
            if (g >= a.stages && !mbarWait(emptyBar + 8u * pos.slot, pos.phase ^ 1u)) {
                *abortV = 1;
                break;
            }
            uint32_t img;
            int x0, y0;
            wgradTile(a, tile, img, x0, y0);
            const uint32_t full = fullBar + 8u * pos.slot, base = smemAddr(sm + pos.slot * stageBytes);
            mbarExpectTx(full, txBytes);
            for (uint32_t c = 0; c < nc; ++c)
                tmaLoad4(base + c * kWgInSlot, &mapIn, (int)((chunk0 + c) * 32u), x0 - 1, y0 - 1, (int)img, full);
            for (uint32_t j = 0; j < a.coChunks; ++j)
                tmaLoad4(base + a.cpc * kWgInSlot + j * kWgOutSlot, &mapOut, (int)(co0 + j * 32u), x0, y0, (int)img,
                         full);
        }
    } else if (warp == 1) {  // MMAs
        // kind::f16: D f32, A and B bf16, both MN-major, N = coB, M = 128.
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((a.coB >> 3) << 17) |
                               ((128u >> 4) << 24);
        // 8 pixels x 64 bytes between K groups (stride byte offset 512), version 1, 64-byte swizzle.
        const uint32_t hi = (512u >> 4) | (1u << 14) | (4u << 29);
        const uint32_t aLbo = (64u >> 4) << 16, bLbo = (kWgOutSlot >> 4) << 16;
        RingPos pos{0u, 0u};
        uint32_t t = 0u;
        bool ok = true;
        for (uint32_t tile = blockIdx.x; tile < a.numTiles; tile += gridDim.x, ++t, pos.advance(a.stages)) {
            if (!mbarWaitWarp(fullBar + 8u * pos.slot, pos.phase)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t base = smemAddr(sm + pos.slot * stageBytes);
            const uint32_t bLo = (((base + a.cpc * kWgInSlot) & 0x3FFFFu) >> 4) | bLbo;
            const uint32_t set = a.sets == 2u ? t & 1u : 0u, acc = t >= a.sets ? 1u : 0u;
            for (uint32_t c = 0; c < nc; ++c) {
                const uint32_t aLo = (((base + c * kWgInSlot) & 0x3FFFFu) >> 4) | aLbo;
                const uint32_t d = taddr + 3u * (set * a.cpc + c) * a.coB;
                if (electOne()) {
#pragma unroll
                    for (uint32_t r = 0; r < kWgTile; ++r)
#pragma unroll
                        for (uint32_t dy = 0; dy < 3u; ++dy)
                            mmaF16(d + dy * a.coB, aLo + (r + dy) * (kWgHalo * 64u / 16u),
                                   bLo + r * (kWgTile * 64u / 16u), hi, idesc, r ? 1u : acc);
                }
                __syncwarp();
            }
            if (electOne()) umaCommit(emptyBar + 8u * pos.slot);
            __syncwarp();
        }
        if (!ok) *abortV = 1;
        else if (electOne()) umaCommit(doneBar);
        __syncwarp();
    }
    __syncwarp();
    // Lanes of warp q hold rows 32 q..: horizontal tap q, input channel = lane.
    if (!mbarWait(doneBar, 0u)) *abortV = 1;
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (!*abortV && warp < 3u) {
        const bool second = a.sets == 2u && blockIdx.x + gridDim.x < a.numTiles;  // the CTA's second tile
        for (uint32_t c = 0; c < nc; ++c) {
            const uint32_t ci = (chunk0 + c) * 32u + lane;
            for (uint32_t dy = 0; dy < 3u; ++dy) {
                for (uint32_t k0 = 0; k0 < a.coB; k0 += 16u) {
                    float sum[16];
                    wgradLoad(taddr + ((warp * 32u) << 16) + (3u * c + dy) * a.coB + k0, sum);
                    if (second) {
                        float other[16];
                        wgradLoad(taddr + ((warp * 32u) << 16) + (3u * (a.cpc + c) + dy) * a.coB + k0, other);
#pragma unroll
                        for (uint32_t k = 0; k < 16; ++k) sum[k] += other[k];
                    }
#pragma unroll
                    for (uint32_t k = 0; k < 16; ++k) {
                        const uint32_t co = co0 + k0 + k;
                        if (ci < a.cin && co < a.cout)
                            atomicAdd(a.dw + ((size_t)co * 9u + dy * 3u + warp) * a.cin + ci, sum[k]);
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (*abortV && tid == 0) atomicExch(&g_unetError, 4);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(a.cols));
}

// The same sums on mma.sync for small problems: blocks of 64 x 64 channels of
// one tap over a run of pixels, operands by cp.async (zero fill for the padding)
// through an XOR swizzle that keeps the transposing ldmatrix conflict-free.  It
// has no set-up and packs the pixels of any image densely: 128 to 128 channels
// at 32 x 32 take 8.6 us against 18.7 in the kernel above, on 1,531 images of
// one pixel 8.5 against 64 (launchWgrad chooses).
struct WgradMmaArgs {
    const __nv_bfloat16* in;    // [M][ldi], channels [0, cin)
    const __nv_bfloat16* dout;  // [M][ldd], channels [0, cout)
    float* dw;                  // [cout][9][cin], accumulated
    uint32_t n, h, w_, cin, ldi, cout, ldd, M;
    uint32_t chunk;             // pixels per block (multiple of 32)
};

constexpr int kWB = 64;  // co and ci per block

// Byte offset of 16-byte chunk `seg` (0..7) of row `r` in a 128-byte-row tile.
__device__ __forceinline__ uint32_t swz128(uint32_t r, uint32_t seg) { return r * 128u + ((seg ^ (r & 7u)) << 4); }

__global__ void __launch_bounds__(128) k_conv3x3_wgrad_mma(WgradMmaArgs a) {
    __shared__ __align__(128) unsigned char sA[2][32 * 128];  // [pixel][64 co]
    __shared__ __align__(128) unsigned char sB[2][32 * 128];  // [pixel][64 ci]
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t tap = blockIdx.z;
    const uint32_t ciTiles = (a.cin + kWB - 1) / kWB;
    const uint32_t co0 = (blockIdx.y / ciTiles) * kWB, ci0 = (blockIdx.y % ciTiles) * kWB;
    const uint32_t p0 = blockIdx.x * a.chunk, p1 = min(p0 + a.chunk, a.M);
    const int dy = (int)(tap / 3u) - 1, dx = (int)(tap % 3u) - 1;
    const uint32_t HW = a.h * a.w_;
    const uint32_t wm = warp >> 1, wn = warp & 1u;  // 2 x 2 warps of 32 co x 32 ci

    auto loadStage = [&](uint32_t pb, int stage) {
        // 32 pixels x 8 chunks for each operand: 2 + 2 chunks per thread.
#pragma unroll
        for (uint32_t k = 0; k < 2; ++k) {
            uint32_t i = tid + k * 128u, row = i >> 3, seg = i & 7u;
            uint32_t p = pb + row;
            bool pv = p < p1;
            bool v = pv && co0 + seg * 8u < a.cout;
            const __nv_bfloat16* src = a.dout + (size_t)p * a.ldd + co0 + seg * 8u;
            cpAsync16(&sA[stage][swz128(row, seg)], v ? src : a.dout, v ? 16u : 0u);
            bool vb = false;
            const __nv_bfloat16* bsrc = a.in;
            if (pv && ci0 + seg * 8u < a.cin) {
                uint32_t img = p / HW, rem = p - img * HW;
                int yy = (int)(rem / a.w_) + dy, xx = (int)(rem % a.w_) + dx;
                if (yy >= 0 && yy < (int)a.h && xx >= 0 && xx < (int)a.w_) {
                    vb = true;
                    bsrc = a.in + ((size_t)(img * a.h + (uint32_t)yy) * a.w_ + (uint32_t)xx) * a.ldi + ci0 + seg * 8u;
                }
            }
            cpAsync16(&sB[stage][swz128(row, seg)], bsrc, vb ? 16u : 0u);
        }
    };

    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.0f;

    const uint32_t steps = (p1 > p0) ? (p1 - p0 + 31u) / 32u : 0u;
    if (steps > 0) loadStage(p0, 0);
    cpAsyncCommit();
    for (uint32_t s = 0; s < steps; ++s) {
        if (s + 1 < steps) loadStage(p0 + (s + 1) * 32u, (int)((s + 1) & 1u));
        cpAsyncCommit();
        cpAsyncWait<1>();
        __syncthreads();
        const int st = (int)(s & 1u);
#pragma unroll
        for (uint32_t kk = 0; kk < 2; ++kk) {  // 16 pixels each
            uint32_t af[2][4];
#pragma unroll
            for (uint32_t mt = 0; mt < 2; ++mt) {
                // A (co x p) from sA[p][co] through transposed 8x8 loads:
                // matrices (co 0-7, p 0-7), (co 8-15, p 0-7), (co 0-7, p 8-15), (co 8-15, p 8-15).
                uint32_t id = lane >> 3;
                uint32_t prow = kk * 16u + ((id >> 1) << 3) + (lane & 7u);
                uint32_t seg = (wm * 32u + mt * 16u) / 8u + (id & 1u);
                ldmatrixX4T(af[mt][0], af[mt][1], af[mt][2], af[mt][3], &sA[st][swz128(prow, seg)]);
            }
#pragma unroll
            for (uint32_t np = 0; np < 2; ++np) {
                // B (p x ci): matrices (p 0-7, ci 0-7), (p 8-15, ci 0-7), (p 0-7, ci 8-15), (p 8-15, ci 8-15).
                uint32_t id = lane >> 3;
                uint32_t prow = kk * 16u + ((id & 1u) << 3) + (lane & 7u);
                uint32_t seg = (wn * 32u + np * 16u) / 8u + (id >> 1);
                uint32_t b0, b1, b2, b3;
                ldmatrixX4T(b0, b1, b2, b3, &sB[st][swz128(prow, seg)]);
#pragma unroll
                for (uint32_t mt = 0; mt < 2; ++mt) {
                    mmaBf16(acc[mt][2 * np], af[mt], b0, b1);
                    mmaBf16(acc[mt][2 * np + 1], af[mt], b2, b3);
                }
            }
        }
        __syncthreads();
    }
    cpAsyncWait<0>();
#pragma unroll
    for (uint32_t mt = 0; mt < 2; ++mt)
#pragma unroll
        for (uint32_t half = 0; half < 2; ++half) {
            uint32_t co = co0 + wm * 32u + mt * 16u + (lane >> 2) + half * 8u;
            if (co >= a.cout) continue;
#pragma unroll
            for (uint32_t nt = 0; nt < 4; ++nt) {
                uint32_t ci = ci0 + wn * 32u + nt * 8u + (lane & 3u) * 2u;
                if (ci >= a.cin) continue;
                float* dst = a.dw + ((size_t)co * 9u + tap) * a.cin + ci;
                atomicAdd(dst, acc[mt][nt][half * 2 + 0]);
                atomicAdd(dst + 1, acc[mt][nt][half * 2 + 1]);
            }
        }
}

// ------------------------------------------------------- elementwise ----
__device__ __forceinline__ uint32_t gid() { return blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ uint32_t gstride() { return gridDim.x * blockDim.x; }

// dPre = dOut where out > 0 (ReLU), over `c` channels of every pixel.
__global__ void k_relu_backward(const __nv_bfloat16* out, uint32_t ldo, const __nv_bfloat16* dout, uint32_t ldd,
                                __nv_bfloat16* dpre, uint32_t ldp, uint32_t c, uint32_t M) {
    const uint32_t pairs = c / 2u;
    for (uint64_t i = gid(); i < (uint64_t)M * pairs; i += gstride()) {
        uint32_t p = (uint32_t)(i / pairs), k = (uint32_t)(i % pairs) * 2u;
        __nv_bfloat162 o = *reinterpret_cast<const __nv_bfloat162*>(out + (size_t)p * ldo + k);
        __nv_bfloat162 d = *reinterpret_cast<const __nv_bfloat162*>(dout + (size_t)p * ldd + k);
        float2 of = __bfloat1622float2(o), df = __bfloat1622float2(d);
        *reinterpret_cast<__nv_bfloat162*>(dpre + (size_t)p * ldp + k) =
            __floats2bfloat162_rn(of.x > 0.0f ? df.x : 0.0f, of.y > 0.0f ? df.y : 0.0f);
    }
}

// Per-channel sums of dPre (the bias gradient), accumulated into db.
__global__ void k_bias_grad(const __nv_bfloat16* dpre, uint32_t ld, uint32_t c, uint32_t M, float* db) {
    // blockDim.x = 256: thread handles channel (tid % c) over a pixel stripe.
    __shared__ float partial[256];
    uint32_t ch = threadIdx.x % c, lanes = 256u / c;
    uint32_t lanePix = threadIdx.x / c;
    float s = 0.0f;
    if (lanePix < lanes)
        for (uint32_t p = blockIdx.x * lanes + lanePix; p < M; p += gridDim.x * lanes)
            s += __bfloat162float(dpre[(size_t)p * ld + ch]);
    partial[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x < c) {
        float t = 0.0f;
        for (uint32_t k = 0; k < lanes; ++k) t += partial[k * c + threadIdx.x];
        atomicAdd(&db[threadIdx.x], t);
    }
}

// 2x2 average pooling: out (h/2, w/2).
__global__ void k_avgpool2(const __nv_bfloat16* in, uint32_t ldi, __nv_bfloat16* out, uint32_t ldo, uint32_t coOff,
                           uint32_t c, uint32_t n, uint32_t h, uint32_t w) {
    const uint32_t ho = h / 2u, wo = w / 2u, pairs = c / 2u;
    for (uint64_t i = gid(); i < (uint64_t)n * ho * wo * pairs; i += gstride()) {
        uint32_t k = (uint32_t)(i % pairs) * 2u;
        uint64_t q = i / pairs;
        uint32_t x = (uint32_t)(q % wo), y = (uint32_t)((q / wo) % ho), b = (uint32_t)(q / ((uint64_t)wo * ho));
        size_t base = ((size_t)(b * h + 2u * y) * w + 2u * x) * ldi + k;
        float2 s = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(in + base));
        float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(in + base + ldi));
        float2 u = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(in + base + (size_t)w * ldi));
        float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(in + base + (size_t)w * ldi + ldi));
        *reinterpret_cast<__nv_bfloat162*>(out + q * ldo + coOff + k) =
            __floats2bfloat162_rn(0.25f * (s.x + t.x + u.x + v.x), 0.25f * (s.y + t.y + u.y + v.y));
    }
}

// Gradient of the 2x2 average pool: din (+)= dout / 4 on each of the 4 inputs.
__global__ void k_avgpool2_backward(const __nv_bfloat16* dout, uint32_t ldd, __nv_bfloat16* din, uint32_t ldi,
                                    uint32_t c, uint32_t n, uint32_t h, uint32_t w, int accumulate) {
    const uint32_t wo = w / 2u, pairs = c / 2u;
    for (uint64_t i = gid(); i < (uint64_t)n * h * w * pairs; i += gstride()) {
        uint32_t k = (uint32_t)(i % pairs) * 2u;
        uint64_t q = i / pairs;
        uint32_t x = (uint32_t)(q % w), y = (uint32_t)((q / w) % h), b = (uint32_t)(q / ((uint64_t)w * h));
        float2 d = __bfloat1622float2(
            *reinterpret_cast<const __nv_bfloat162*>(dout + ((size_t)(b * (h / 2u) + y / 2u) * wo + x / 2u) * ldd + k));
        __nv_bfloat162* dst = reinterpret_cast<__nv_bfloat162*>(din + q * ldi + k);
        float2 v = make_float2(0.25f * d.x, 0.25f * d.y);
        if (accumulate) {
            float2 o = __bfloat1622float2(*dst);
            v.x += o.x;
            v.y += o.y;
        }
        *dst = __floats2bfloat162_rn(v.x, v.y);
    }
}

// Nearest 2x upsampling: out (2h, 2w).
__global__ void k_upsample2(const __nv_bfloat16* in, uint32_t ldi, __nv_bfloat16* out, uint32_t ldo, uint32_t coOff,
                            uint32_t c, uint32_t n, uint32_t h, uint32_t w) {
    const uint32_t H = 2u * h, W = 2u * w, pairs = c / 2u;
    for (uint64_t i = gid(); i < (uint64_t)n * H * W * pairs; i += gstride()) {
        uint32_t k = (uint32_t)(i % pairs) * 2u;
        uint64_t q = i / pairs;
        uint32_t x = (uint32_t)(q % W), y = (uint32_t)((q / W) % H), b = (uint32_t)(q / ((uint64_t)W * H));
        *reinterpret_cast<__nv_bfloat162*>(out + q * ldo + coOff + k) =
            *reinterpret_cast<const __nv_bfloat162*>(in + ((size_t)(b * h + y / 2u) * w + x / 2u) * ldi + k);
    }
}

// Gradient of the nearest upsampling: din = sum of the 4 output gradients.
__global__ void k_upsample2_backward(const __nv_bfloat16* dout, uint32_t ldd, uint32_t ciOff, __nv_bfloat16* din,
                                     uint32_t ldi, uint32_t c, uint32_t n, uint32_t h, uint32_t w) {
    const uint32_t W = 2u * w, pairs = c / 2u;
    for (uint64_t i = gid(); i < (uint64_t)n * h * w * pairs; i += gstride()) {
        uint32_t k = (uint32_t)(i % pairs) * 2u;
        uint64_t q = i / pairs;
        uint32_t x = (uint32_t)(q % w), y = (uint32_t)((q / w) % h), b = (uint32_t)(q / ((uint64_t)w * h));
        size_t base = ((size_t)(b * 2u * h + 2u * y) * W + 2u * x) * ldd + ciOff + k;
        float2 s = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(dout + base));
        float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(dout + base + ldd));
        float2 u = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(dout + base + (size_t)W * ldd));
        float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(dout + base + (size_t)W * ldd + ldd));
        *reinterpret_cast<__nv_bfloat162*>(din + q * ldi + k) =
            __floats2bfloat162_rn(s.x + t.x + u.x + v.x, s.y + t.y + u.y + v.y);
    }
}

// Channel-slice copy (skip connections into concat buffers, gradient routing).
__global__ void k_copy_channels(const __nv_bfloat16* src, uint32_t lds, uint32_t sOff, __nv_bfloat16* dst,
                                uint32_t ldd, uint32_t dOff, uint32_t c, uint32_t M, int accumulate) {
    const uint32_t pairs = c / 2u;
    for (uint64_t i = gid(); i < (uint64_t)M * pairs; i += gstride()) {
        uint32_t p = (uint32_t)(i / pairs), k = (uint32_t)(i % pairs) * 2u;
        float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(src + (size_t)p * lds + sOff + k));
        __nv_bfloat162* d = reinterpret_cast<__nv_bfloat162*>(dst + (size_t)p * ldd + dOff + k);
        if (accumulate) {
            float2 o = __bfloat1622float2(*d);
            v.x += o.x;
            v.y += o.y;
        }
        *d = __floats2bfloat162_rn(v.x, v.y);
    }
}

// The same element-wise layers over groups of 8 channels (one 16-byte load or
// store per group) with 32-bit indices: used when every channel count, leading
// dimension and offset is a multiple of 8, the pointers are 16-byte aligned
// and the element count fits 32 bits (the host checks); the arithmetic per
// channel is the one of the kernels above.
__device__ __forceinline__ void ld8(const __nv_bfloat16* p, float (&f)[8]) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[k]));
        f[2 * k] = t.x;
        f[2 * k + 1] = t.y;
    }
}
__device__ __forceinline__ void st8(__nv_bfloat16* p, const float (&f)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        __nv_bfloat162 h2 = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
        w[k] = *reinterpret_cast<uint32_t*>(&h2);
    }
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}

__global__ void k_relu_backward8(const __nv_bfloat16* out, uint32_t ldo, const __nv_bfloat16* dout, uint32_t ldd,
                                 __nv_bfloat16* dpre, uint32_t ldp, uint32_t groups, uint32_t total) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gstride()) {
        const uint32_t p = i / groups, k = (i - p * groups) * 8u;
        float o[8], d[8];
        ld8(out + (size_t)p * ldo + k, o);
        ld8(dout + (size_t)p * ldd + k, d);
#pragma unroll
        for (int j = 0; j < 8; ++j) d[j] = o[j] > 0.0f ? d[j] : 0.0f;
        st8(dpre + (size_t)p * ldp + k, d);
    }
}

// The bias gradient (db[c] += the sum of dout) over groups of 8 channels, with
// kRelu after the ReLU gradient (dpre = dout where out > 0, summed instead).  A
// thread keeps one channel group, so its eight sums stay in registers over its
// pixels; the block adds its partial sums in shared memory and issues one atomic
// per channel.  Memory-bound: each operand is read once, whole 64-byte runs of a
// pixel by neighbouring threads (32 channels of 2^20 pixels with both gradients:
// 36 us, 5.6 TB/s).  Over a 16 x 256^2 training step 341 us; the separate passes
// with one channel per thread took 236 + 719 us.  (The ReLU gradient alone keeps
// a group per thread: small tensors 4.4 us against 6.4 in blocks like these.)
constexpr uint32_t kRbThreads = 256u;
template <bool kRelu>
__global__ void __launch_bounds__(256) k_relu_bias8(const __nv_bfloat16* out, uint32_t ldo, const __nv_bfloat16* dout,
                                                    uint32_t ldd, __nv_bfloat16* dpre, uint32_t ldp, uint32_t groups,
                                                    uint32_t M, float* db) {
    const uint32_t lanes = kRbThreads / groups, lane = threadIdx.x / groups;
    const uint32_t g = threadIdx.x - lane * groups, k = g * 8u;
    float s[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (lane < lanes) {
        const uint64_t step = (uint64_t)gridDim.x * lanes;
#pragma unroll 4
        for (uint64_t p = (uint64_t)blockIdx.x * lanes + lane; p < M; p += step) {
            float d[8];
            ld8(dout + (size_t)p * ldd + k, d);
            if (kRelu) {
                float o[8];
                ld8(out + (size_t)p * ldo + k, o);
#pragma unroll
                for (int j = 0; j < 8; ++j) d[j] = o[j] > 0.0f ? d[j] : 0.0f;
                st8(dpre + (size_t)p * ldp + k, d);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j] += d[j];
        }
    }
    __shared__ float part[kRbThreads][9];
#pragma unroll
    for (int j = 0; j < 8; ++j) part[threadIdx.x][j] = s[j];
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < groups * 8u; c += kRbThreads) {
        float t = 0.0f;
        for (uint32_t l = 0; l < lanes; ++l) t += part[l * groups + (c >> 3)][c & 7u];
        atomicAdd(&db[c], t);
    }
}

__global__ void k_avgpool2_8(const __nv_bfloat16* in, uint32_t ldi, __nv_bfloat16* out, uint32_t ldo, uint32_t coOff,
                             uint32_t groups, uint32_t h, uint32_t w, uint32_t total) {
    pdlRelease();
    pdlWait();
    const uint32_t wo = w / 2u, ho = h / 2u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gstride()) {
        const uint32_t q = i / groups, k = (i - q * groups) * 8u;
        const uint32_t x = q % wo, r = q / wo, y = r % ho, b = r / ho;
        const size_t base = ((size_t)(b * h + 2u * y) * w + 2u * x) * ldi + k;
        float s[8], t[8], u[8], v[8];
        ld8(in + base, s);
        ld8(in + base + ldi, t);
        ld8(in + base + (size_t)w * ldi, u);
        ld8(in + base + (size_t)w * ldi + ldi, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] = 0.25f * (s[j] + t[j] + u[j] + v[j]);
        st8(out + (size_t)q * ldo + coOff + k, s);
    }
}

__global__ void k_avgpool2_backward8(const __nv_bfloat16* dout, uint32_t ldd, __nv_bfloat16* din, uint32_t ldi,
                                     uint32_t groups, uint32_t h, uint32_t w, int accumulate, uint32_t total) {
    // one thread per pooled pixel and group: its gradient goes to the 4 inputs
    const uint32_t wo = w / 2u, ho = h / 2u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gstride()) {
        const uint32_t q = i / groups, k = (i - q * groups) * 8u;
        const uint32_t x = q % wo, r = q / wo, y = r % ho, b = r / ho;
        float d[8];
        ld8(dout + (size_t)q * ldd + k, d);
#pragma unroll
        for (int j = 0; j < 8; ++j) d[j] *= 0.25f;
        const size_t base = ((size_t)(b * h + 2u * y) * w + 2u * x) * ldi + k;
        const size_t offs[4] = {0, ldi, (size_t)w * ldi, (size_t)w * ldi + ldi};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = d[j];
            if (accumulate) {
                float o[8];
                ld8(din + base + offs[c], o);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] += o[j];
            }
            st8(din + base + offs[c], v);
        }
    }
}

__global__ void k_upsample2_8(const __nv_bfloat16* in, uint32_t ldi, __nv_bfloat16* out, uint32_t ldo, uint32_t coOff,
                              uint32_t groups, uint32_t h, uint32_t w, uint32_t total) {
    // one thread per input pixel and group, written to its 2x2 outputs
    pdlRelease();
    pdlWait();
    const uint32_t W = 2u * w;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gstride()) {
        const uint32_t q = i / groups, k = (i - q * groups) * 8u;
        const uint32_t x = q % w, r = q / w, y = r % h, b = r / h;
        const uint4 v = *reinterpret_cast<const uint4*>(in + (size_t)q * ldi + k);
        const size_t o = ((size_t)(b * 2u * h + 2u * y) * W + 2u * x) * ldo + coOff + k;
        *reinterpret_cast<uint4*>(out + o) = v;
        *reinterpret_cast<uint4*>(out + o + ldo) = v;
        *reinterpret_cast<uint4*>(out + o + (size_t)W * ldo) = v;
        *reinterpret_cast<uint4*>(out + o + (size_t)W * ldo + ldo) = v;
    }
}

__global__ void k_upsample2_backward8(const __nv_bfloat16* dout, uint32_t ldd, uint32_t ciOff, __nv_bfloat16* din,
                                      uint32_t ldi, uint32_t groups, uint32_t h, uint32_t w, uint32_t total) {
    const uint32_t W = 2u * w;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gstride()) {
        const uint32_t q = i / groups, k = (i - q * groups) * 8u;
        const uint32_t x = q % w, r = q / w, y = r % h, b = r / h;
        const size_t base = ((size_t)(b * 2u * h + 2u * y) * W + 2u * x) * ldd + ciOff + k;
        float s[8], t[8], u[8], v[8];
        ld8(dout + base, s);
        ld8(dout + base + ldd, t);
        ld8(dout + base + (size_t)W * ldd, u);
        ld8(dout + base + (size_t)W * ldd + ldd, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] = s[j] + t[j] + u[j] + v[j];
        st8(din + (size_t)q * ldi + k, s);
    }
}

__global__ void k_copy_channels8(const __nv_bfloat16* src, uint32_t lds, uint32_t sOff, __nv_bfloat16* dst,
                                 uint32_t ldd, uint32_t dOff, uint32_t groups, int accumulate, uint32_t total) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gstride()) {
        const uint32_t p = i / groups, k = (i - p * groups) * 8u;
        float v[8];
        ld8(src + (size_t)p * lds + sOff + k, v);
        __nv_bfloat16* d = dst + (size_t)p * ldd + dOff + k;
        if (accumulate) {
            float o[8];
            ld8(d, o);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] += o[j];
        }
        st8(d, v);
    }
}

// Network input: 16 channels per pixel from the AOV planes (RGBA32F, image
// rows y0.., columns x0.. of a W_img-wide image; pixels outside the image are
// zero): log(1 + beauty) (3), albedo (3), normal in [-1, 1] (3), depth / (1 +
// depth) (1), zeros (6).
__global__ void k_pack_input(const float4* beauty, const float4* albedo, const float4* normal, const float4* depth,
                             uint32_t imgW, uint32_t imgH, uint32_t x0, uint32_t y0, __nv_bfloat16* out, uint32_t h,
                             uint32_t w, uint32_t batchIndex, bool wide) {
    for (uint32_t i = gid(); i < h * w; i += gstride()) {
        uint32_t x = i % w, y = i / w;
        uint32_t ix = x0 + x, iy = y0 + y;
        float v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = 0.0f;
        if (ix < imgW && iy < imgH) {
            size_t s = (size_t)iy * imgW + ix;
            float4 b = beauty[s], a = albedo[s], nm = normal[s], d = depth[s];
            v[0] = log1pf(fmaxf(b.x, 0.0f));
            v[1] = log1pf(fmaxf(b.y, 0.0f));
            v[2] = log1pf(fmaxf(b.z, 0.0f));
            v[3] = a.x;
            v[4] = a.y;
            v[5] = a.z;
            v[6] = nm.x * 2.0f - 1.0f;
            v[7] = nm.y * 2.0f - 1.0f;
            v[8] = nm.z * 2.0f - 1.0f;
            float dd = fmaxf(d.x, 0.0f);
            v[9] = dd / (1.0f + dd);
        }
        __nv_bfloat16* o = out + ((size_t)batchIndex * h * w + i) * 16u;
        if (wide) {  // a pixel's 32 bytes as two stores (eight cost 55 us instead of 28 at 1920 x 1088)
            st8(o, reinterpret_cast<const float(&)[8]>(v[0]));
            st8(o + 8, reinterpret_cast<const float(&)[8]>(v[8]));
            continue;
        }
#pragma unroll
        for (int k = 0; k < 16; k += 2)
            *reinterpret_cast<__nv_bfloat162*>(o + k) = __floats2bfloat162_rn(v[k], v[k + 1]);
    }
}

// A pixel's first three channels; `wide`: as one 8-byte load (leading dimension
// a multiple of 4, 8-byte aligned).
__device__ __forceinline__ void ld3(const __nv_bfloat16* p, bool wide, float (&f)[3]) {
    if (wide) {
        const uint2 u = *reinterpret_cast<const uint2*>(p);
        const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
        f[0] = t.x;
        f[1] = t.y;
        f[2] = __low2float(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) f[k] = __bfloat162float(p[k]);
    }
}

// L1 loss in log space against a target image (RGBA32F) and its gradient
// (scaled by 1 / (3 * pixels)) into the prediction's first 3 channels.  With
// `base` (the network input, whose first 3 channels are log(1 + noisy)), the
// prediction is a residual: the output is base + pred.
__global__ void k_l1_loss(const __nv_bfloat16* pred, uint32_t ldp, const __nv_bfloat16* base, uint32_t ldb,
                          const float4* target, uint32_t M, __nv_bfloat16* grad, uint32_t ldg, float* loss,
                          bool wideIn, bool wideGrad) {
    __shared__ float red[256];
    float s = 0.0f;
    const float scale = 1.0f / (3.0f * (float)M);
    for (uint32_t p = gid(); p < M; p += gstride()) {
        float4 t = target[p];
        float tl[3] = {log1pf(fmaxf(t.x, 0.0f)), log1pf(fmaxf(t.y, 0.0f)), log1pf(fmaxf(t.z, 0.0f))};
        float g[3], yp[3], yb[3];
        ld3(pred + (size_t)p * ldp, wideIn, yp);
        if (base) ld3(base + (size_t)p * ldb, wideIn, yb);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            float y = yp[k];
            if (base) y += yb[k];
            float d = y - tl[k];
            s += fabsf(d);
            g[k] = (d > 0.0f ? scale : (d < 0.0f ? -scale : 0.0f));
        }
        __nv_bfloat16* gp = grad + (size_t)p * ldg;
        if (wideGrad) {  // ldg 16: the pixel's 32 bytes as two stores
            const float lo[8] = {g[0], g[1], g[2], 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
            const float zero[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
            st8(gp, lo);
            st8(gp + 8, zero);
            continue;
        }
        gp[0] = __float2bfloat16_rn(g[0]);
        gp[1] = __float2bfloat16_rn(g[1]);
        gp[2] = __float2bfloat16_rn(g[2]);
        for (uint32_t k = 3; k < ldg; ++k) gp[k] = __float2bfloat16_rn(0.0f);
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (uint32_t o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(loss, red[0] * scale);
}

// Network output (log space, first 3 channels) to an RGBA32F image; alpha from
// `alphaSrc`.  With `base`: the output is base + pred (a residual over the
// network input's log(1 + noisy) channels), summed in FP32.
__global__ void k_unpack_output(const __nv_bfloat16* pred, uint32_t ldp, const __nv_bfloat16* base, uint32_t ldb,
                                uint32_t h, uint32_t w, const float4* alphaSrc, uint32_t imgW, uint32_t imgH,
                                uint32_t x0, uint32_t y0, float4* out, bool wideIn) {
    for (uint32_t i = gid(); i < h * w; i += gstride()) {
        uint32_t ix = x0 + i % w, iy = y0 + i / w;
        if (ix >= imgW || iy >= imgH) continue;
        size_t s = (size_t)iy * imgW + ix;
        float y[3];
        ld3(pred + (size_t)i * ldp, wideIn, y);
        if (base) {
            float b[3];
            ld3(base + (size_t)i * ldb, wideIn, b);
            y[0] += b[0];
            y[1] += b[1];
            y[2] += b[2];
        }
        out[s] = make_float4(fmaxf(expm1f(y[0]), 0.0f), fmaxf(expm1f(y[1]), 0.0f), fmaxf(expm1f(y[2]), 0.0f),
                             alphaSrc[s].w);
    }
}

// Adam on FP32 master weights; writes the bf16 forward weights and, for 3x3
// layers, the tap-flipped transposed copy the input gradient uses.
struct AdamRule {
    float lr, b1, b2, eps, c1, c2;
};
__device__ __forceinline__ float adamStep(const AdamRule& r, float w, float g, float& m, float& v) {
    // The new term is fused, the decayed one rounded, in both entry points: left to the compiler it was the other way
    // round in one build, which changes the last bit of every third m and every fourth v.
    m = __fmaf_rn(1.0f - r.b1, g, r.b1 * m);
    v = __fmaf_rn((1.0f - r.b2) * g, g, r.b2 * v);
    return w - r.lr * (m / r.c1) / (sqrtf(v / r.c2) + r.eps);
}
__global__ void k_adam(float* wts, const float* grad, float* m, float* v, uint32_t count, AdamRule rule,
                       __nv_bfloat16* wbf, __nv_bfloat16* wflip, uint32_t cout, uint32_t cin) {
    for (uint32_t i = gid(); i < count; i += gstride()) {
        float mi = m[i], vi = v[i];
        float wv = adamStep(rule, wts[i], grad[i], mi, vi);
        m[i] = mi;
        v[i] = vi;
        wts[i] = wv;
        if (wbf) wbf[i] = __float2bfloat16_rn(wv);
        if (wflip) {
            uint32_t ci = i % cin, tap = (i / cin) % 9u, co = i / (9u * cin);
            wflip[((size_t)ci * 9u + (8u - tap)) * cout + co] = __float2bfloat16_rn(wv);
        }
    }
}

// Every tensor of an optimiser step in one launch: blocks are dealt to the
// groups by a table in the kernel's parameters.  A block takes 1,024 elements:
// of a 3x3 layer a 32 x 32 tile of one tap, so that the transposed copy is
// written through shared memory in runs of output channels.  The 19 layers
// and their biases: 148 us of kernels in 38 launches, 12 us in one.
constexpr uint32_t kAdamGroups = 40;
struct AdamTable {
    dk_unet_adam_group g[kAdamGroups];
    uint32_t first[kAdamGroups + 1];  // first block of each group
    uint32_t groups;
};
__global__ void __launch_bounds__(256) k_adam_groups(const __grid_constant__ AdamTable t, AdamRule rule) {
    __shared__ __align__(8) __nv_bfloat16 tile[32][36];  // [ci][co], rows of 72 bytes, read in 8-byte pieces
    uint32_t lo = 0, hi = t.groups - 1u;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1u) >> 1;
        if (t.first[mid] <= blockIdx.x) lo = mid;
        else hi = mid - 1u;
    }
    const dk_unet_adam_group& g = t.g[lo];
    const uint32_t b = blockIdx.x - t.first[lo];
    __nv_bfloat16* wbf = static_cast<__nv_bfloat16*>(g.wbf16);
    __nv_bfloat16* wflip = static_cast<__nv_bfloat16*>(g.wflip);
    if (!wflip) {
        for (uint32_t i = b * 1024u + threadIdx.x; i < min(g.count, b * 1024u + 1024u); i += 256u) {
            float mi = g.m[i], vi = g.v[i];
            const float wv = adamStep(rule, g.weights[i], g.grad[i], mi, vi);
            g.m[i] = mi;
            g.v[i] = vi;
            g.weights[i] = wv;
            if (wbf) wbf[i] = __float2bfloat16_rn(wv);
        }
        return;
    }
    const uint32_t ciTiles = (g.cin + 31u) / 32u, coTiles = (g.cout + 31u) / 32u;
    const uint32_t tap = b / (ciTiles * coTiles), rest = b - tap * ciTiles * coTiles;
    const uint32_t co0 = rest / ciTiles * 32u, ci0 = rest % ciTiles * 32u;
    const uint32_t r = threadIdx.x >> 3, c4 = (threadIdx.x & 7u) * 4u;  // four input channels of an output channel
    if (co0 + r < g.cout && ci0 + c4 < g.cin) {
        const size_t i = ((size_t)(co0 + r) * 9u + tap) * g.cin + ci0 + c4;
        float4 w = *reinterpret_cast<const float4*>(g.weights + i), m = *reinterpret_cast<const float4*>(g.m + i);
        float4 v = *reinterpret_cast<const float4*>(g.v + i);
        const float4 d = *reinterpret_cast<const float4*>(g.grad + i);
        w.x = adamStep(rule, w.x, d.x, m.x, v.x);
        w.y = adamStep(rule, w.y, d.y, m.y, v.y);
        w.z = adamStep(rule, w.z, d.z, m.z, v.z);
        w.w = adamStep(rule, w.w, d.w, m.w, v.w);
        *reinterpret_cast<float4*>(g.weights + i) = w;
        *reinterpret_cast<float4*>(g.m + i) = m;
        *reinterpret_cast<float4*>(g.v + i) = v;
        __nv_bfloat162 h[2] = {__floats2bfloat162_rn(w.x, w.y), __floats2bfloat162_rn(w.z, w.w)};
        if (wbf) *reinterpret_cast<uint2*>(wbf + i) = *reinterpret_cast<const uint2*>(h);
        tile[c4 + 0u][r] = __low2bfloat16(h[0]);
        tile[c4 + 1u][r] = __high2bfloat16(h[0]);
        tile[c4 + 2u][r] = __low2bfloat16(h[1]);
        tile[c4 + 3u][r] = __high2bfloat16(h[1]);
    }
    __syncthreads();
    if (ci0 + r < g.cin && co0 + c4 < g.cout)
        *reinterpret_cast<uint2*>(wflip + ((size_t)(ci0 + r) * 9u + (8u - tap)) * g.cout + co0 + c4) =
            *reinterpret_cast<const uint2*>(&tile[r][c4]);
}

__global__ void k_weights_to_bf16(const float* wts, uint32_t count, __nv_bfloat16* wbf, __nv_bfloat16* wflip,
                                  uint32_t cout, uint32_t cin) {
    for (uint32_t i = gid(); i < count; i += gstride()) {
        float wv = wts[i];
        wbf[i] = __float2bfloat16_rn(wv);
        if (wflip) {
            uint32_t ci = i % cin, tap = (i / cin) % 9u, co = i / (9u * cin);
            wflip[((size_t)ci * 9u + (8u - tap)) * cout + co] = __float2bfloat16_rn(wv);
        }
    }
}

inline int gridFor(uint64_t work, int block = 256) {
    if (deviceProp().multiProcessorCount == 0) ensureDevice();
    uint64_t g = (work + block - 1) / block;
    uint64_t cap = (uint64_t)deviceProp().multiProcessorCount * 16u;
    return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

inline bool aligned16(uint32_t v) { return v % 16u == 0u; }

// The 8-channel element-wise kernels apply: channel counts, leading
// dimensions and offsets multiples of 8, pointers 16-byte aligned, and the
// element count within 32 bits.
inline bool vec8(std::initializer_list<uint32_t> counts, std::initializer_list<const void*> ptrs, uint64_t total) {
    for (uint32_t v : counts)
        if (v % 8u) return false;
    for (const void* q : ptrs)
        if (reinterpret_cast<uintptr_t>(q) % 16u) return false;
    return total > 0 && total < (1ull << 31);
}

// ld3's 8-byte loads apply to every tensor given.
inline bool wide4(std::initializer_list<uint32_t> lds, std::initializer_list<const void*> ptrs) {
    for (uint32_t v : lds)
        if (v % 4u) return false;
    for (const void* q : ptrs)
        if (reinterpret_cast<uintptr_t>(q) % 8u) return false;
    return true;
}

inline AdamRule adamRule(float lr, float b1, float b2, float eps, uint32_t step) {
    return AdamRule{lr, b1, b2, eps, 1.0f - powf(b1, (float)step), 1.0f - powf(b2, (float)step)};
}

// k_relu_bias8 over `pixels` pixels of `c` channels: up to six resident blocks
// per SM, at least eight pixels per thread.
template <bool kRelu>
int launchReluBias(const void* out, uint32_t ldo, const void* dout, uint32_t ldd, void* dpre, uint32_t ldp, uint32_t c,
                   uint32_t pixels, float* db, void* stream) {
    if (deviceProp().multiProcessorCount == 0) ensureDevice();
    const uint32_t groups = c / 8u, perBlock = kRbThreads / groups * 8u;
    const uint32_t blocks = (uint32_t)(((uint64_t)pixels + perBlock - 1u) / perBlock);
    const uint32_t grid = std::min(blocks, (uint32_t)deviceProp().multiProcessorCount * 6u);
    k_relu_bias8<kRelu><<<grid, kRbThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(out), ldo, static_cast<const __nv_bfloat16*>(dout), ldd,
        static_cast<__nv_bfloat16*>(dpre), ldp, groups, pixels, db);
    DK_CUDA(cudaGetLastError(), "relu / bias gradient launch");
    return DK_OK;
}

// 3 (default): the halo-row TMA + tcgen05 convolution where the layer fits it,
// else the tile kernel where it is the faster one (launchConvTile), else the
// row-tap or per-tap one, or mma.sync above 256 output channels; 2: the per-tap
// persistent TMA + tcgen05 convolution; 1: the cp.async + tcgen05 one; 0: the
// mma.sync one.
int g_convPath = 3;

// Launch with programmatic stream serialization (see pdlWait); DK_PDL=0 launches
// plainly.
template <typename... KArgs, typename... Args>
cudaError_t launchPdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                      Args... args) {
    static int enabled = -1;
    if (enabled < 0) {
        const char* e = getenv("DK_PDL");
        enabled = (e && e[0] == '0') ? 0 : 1;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = enabled ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// dependency on libcuda).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encodeTiled() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// The current device's opt-in shared memory for `kernel`, once per device.
template <typename... KArgs>
cudaError_t raiseSmemLimit(SmemLimit& limit, void (*kernel)(KArgs...)) {
    int device = 0;
    if (const cudaError_t e = cudaGetDevice(&device)) return e;
    return (cudaError_t)limit.raise(device, [&] {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)deviceProp().sharedMemPerBlockOptin);
    });
}

// Pipeline depth limit from the environment (a tuning knob, read at each
// launch), clamped to [lo, hi]; hi when unset.
uint32_t depthCap(const char* name, uint32_t lo, uint32_t hi) {
    const char* e = getenv(name);
    if (!e || !*e) return hi;
    const long v = strtol(e, nullptr, 10);
    return v < (long)lo ? lo : (v > (long)hi ? hi : (uint32_t)v);
}

// Output rows go through the epilogue's shared-memory transpose when the
// destination is overwritten and every pixel's channel run starts on a
// 16-byte boundary.
bool stagedStores(const ConvArgs& c) {
    return !c.accumulate && c.cout % 8u == 0u && c.ldo % 8u == 0u && c.coOff % 8u == 0u &&
           reinterpret_cast<uintptr_t>(c.out) % 16u == 0u;
}

// The halo-row kernel's launch, or kHaloUnfit (nothing launched) when the
// layer does not fit it: narrow images, or weights and halo ring beyond the
// shared memory of one CTA.
constexpr int kHaloUnfit = -1;
// `pool` (optional): where the 2x2 average of the output goes ([n][h / 2][w / 2]
// [poolLd]); *pooled says whether this launch writes it (tensor-store rows
// only), else the caller pools separately.
int launchConvHalo(const ConvArgs& c, cudaStream_t st, __nv_bfloat16* pool = nullptr, uint32_t poolLd = 0,
                   bool* pooled = nullptr) {
    if (pooled) *pooled = false;
    const uint32_t chunks = (c.cin + 63u) / 64u;
    const size_t optin = (size_t)deviceProp().sharedMemPerBlockOptin;
    // Vertical taps stacked into one MMA (N = 3 Cout <= 256) with a rolling
    // window of accumulator slots; DK_CONV_STACK=0 keeps one MMA per tap.
    const char* stackEnv = getenv("DK_CONV_STACK");
    const bool stack = c.cout * 3u <= 256u && !(stackEnv && stackEnv[0] == '0');
    // Stacked, a halo row is read only in its own step: two slots suffice
    // (one in use, one loading); else three rows are in use at a time.
    const uint32_t minRing = stack ? 2u : kHaloRingMin;
    if (c.w_ < 128u || c.cout > 256u || chunks > 2u || haloSmemBytes(c.cout, chunks, false, minRing, stack) > optin)
        return kHaloUnfit;
    const bool staged = stagedStores(c) && haloSmemBytes(c.cout, chunks, true, minRing, stack) <= optin;
    // Stacked layers of 16, 32 or 64 output channels write their rows with
    // TMA tensor stores (DK_CONV_TMA_STORE=0: through the lanes).
    const char* storeEnv = getenv("DK_CONV_TMA_STORE");
    const bool tmaStore = stack && staged && (c.cout == 16u || c.cout == 32u || c.cout == 64u) &&
                          !(storeEnv && storeEnv[0] == '0') &&
                          haloSmemBytes(c.cout, chunks, true, minRing, stack, true) <= optin;
    // The deepest ring that fits: every further slot is a row in flight.
    uint32_t ring = minRing;
    const uint32_t ringCap = depthCap("DK_CONV_HALO_RING", minRing, kHaloRingMax);
    while (ring < ringCap && haloSmemBytes(c.cout, chunks, staged, ring + 1u, stack, tmaStore) <= optin) ++ring;
    const size_t smem = haloSmemBytes(c.cout, chunks, staged, ring, stack, tmaStore);
    EncodeTiledFn enc = encodeTiled();
    if (!enc) return fail(DK_ERROR_COMMAND_FAILED, "cuTensorMapEncodeTiled is not available");
    HaloConvArgs a;
    a.bias = c.bias;
    a.out = c.out;
    a.n = c.n;
    a.h = c.h;
    a.w = c.w_;
    a.cin = c.cin;
    a.cout = c.cout;
    a.ldo = c.ldo;
    a.coOff = c.coOff;
    a.act = c.act;
    a.accumulate = c.accumulate;
    a.staged = staged ? 1 : 0;
    a.ring = ring;
    a.tmaStore = tmaStore ? 1u : 0u;
    a.slots = 0u;
    a.logSlots = 0u;
    if (stack) {
        a.slots = 1u;
        while (a.slots * 2u * c.cout <= 512u && a.slots * 2u <= kHaloAccMax) a.slots *= 2u;
        while ((1u << a.logSlots) < a.slots) ++a.logSlots;
    }
    // The pooled epilogue (DK_CONV_POOL=0: a separate pass): tensor-store rows,
    // slots in pairs of pairs, whole 2x2 windows, 16-byte pooled stores.
    const char* poolEnv = getenv("DK_CONV_POOL");
    const bool fusePool = pool && tmaStore && a.slots >= 4u && c.h % 2u == 0u && c.w_ % 2u == 0u && !c.accumulate &&
                          poolLd >= c.cout && poolLd % 8u == 0u && (reinterpret_cast<uintptr_t>(pool) & 15u) == 0u &&
                          !(poolEnv && poolEnv[0] == '0');
    a.pool = fusePool ? pool : nullptr;
    a.poolLd = fusePool ? poolLd : 0u;
    a.chunks = chunks;
    a.cols = 32u;
    while (a.cols < c.cout) a.cols <<= 1;
    a.tilesX = (c.w_ + 127u) / 128u;
    const uint32_t sms = (uint32_t)deviceProp().multiProcessorCount;
    const uint64_t rowsTotal = (uint64_t)c.n * a.tilesX * c.h;
    if (rowsTotal >= (1ull << 32)) return kHaloUnfit;
    a.totalRows = (uint32_t)rowsTotal;
    alignas(64) CUtensorMap mapIn, mapW;
    cuuint64_t dimIn[4] = {c.cin, c.w_, c.h, c.n};
    cuuint64_t strideIn[3] = {(cuuint64_t)c.ldi * 2u, (cuuint64_t)c.w_ * c.ldi * 2u, (cuuint64_t)c.h * c.w_ * c.ldi * 2u};
    cuuint32_t boxIn[4] = {64u, kHaloPix, 1u, 1u};
    cuuint32_t unit[4] = {1u, 1u, 1u, 1u};
    CUresult r = enc(&mapIn, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<__nv_bfloat16*>(c.in), dimIn, strideIn,
                     boxIn, unit, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(DK_ERROR_INVALID_ARGUMENT, "activation tensor map rejected");
    cuuint64_t dimW[3] = {c.cin, 9u, c.cout};
    cuuint64_t strideW[2] = {(cuuint64_t)c.cin * 2u, (cuuint64_t)9u * c.cin * 2u};
    cuuint32_t boxW[3] = {64u, 1u, c.cout};
    r = enc(&mapW, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(c.w), dimW, strideW, boxW, unit,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(DK_ERROR_INVALID_ARGUMENT, "weight tensor map rejected");
    // Output rows as boxes {Cout channels, 32 pixels} of the 4-D output (channels, x, y, image) at the
    // slice's channel offset; 2 Cout bytes per pixel row, swizzled like the staging boxes.
    alignas(64) CUtensorMap mapOut = mapIn;
    if (tmaStore) {
        cuuint64_t dimOut[4] = {c.ldo, c.w_, c.h, c.n};
        cuuint64_t strideOut[3] = {(cuuint64_t)c.ldo * 2u, (cuuint64_t)c.w_ * c.ldo * 2u,
                                   (cuuint64_t)c.h * c.w_ * c.ldo * 2u};
        cuuint32_t boxOut[4] = {c.cout, 32u, 1u, 1u};
        const CUtensorMapSwizzle swz = c.cout == 16u   ? CU_TENSOR_MAP_SWIZZLE_32B
                                       : c.cout == 32u ? CU_TENSOR_MAP_SWIZZLE_64B
                                                       : CU_TENSOR_MAP_SWIZZLE_128B;
        r = enc(&mapOut, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, c.out, dimOut, strideOut, boxOut, unit,
                CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail(DK_ERROR_INVALID_ARGUMENT, "output tensor map rejected");
    }
    using HaloKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, HaloConvArgs);
    const uint32_t last = (c.cin - (chunks - 1u) * 64u + 15u) / 16u;
    HaloKernel kernels[2][2][4] = {
        {{k_conv3x3_halo<false, 1, 1>, k_conv3x3_halo<false, 1, 2>, k_conv3x3_halo<false, 1, 3>,
          k_conv3x3_halo<false, 1, 4>},
         {k_conv3x3_halo<false, 2, 1>, k_conv3x3_halo<false, 2, 2>, k_conv3x3_halo<false, 2, 3>,
          k_conv3x3_halo<false, 2, 4>}},
        {{k_conv3x3_halo<true, 1, 1>, k_conv3x3_halo<true, 1, 2>, k_conv3x3_halo<true, 1, 3>,
          k_conv3x3_halo<true, 1, 4>},
         {k_conv3x3_halo<true, 2, 1>, k_conv3x3_halo<true, 2, 2>, k_conv3x3_halo<true, 2, 3>,
          k_conv3x3_halo<true, 2, 4>}}};
    HaloKernel kernel = kernels[stack][chunks - 1u][last - 1u];
    static SmemLimit limits[2][2][4];
    DK_CUDA(raiseSmemLimit(limits[stack][chunks - 1u][last - 1u], kernel), "conv3x3 (halo) shared memory");
    uint32_t grid = std::min(sms, a.totalRows);
    DK_CUDA(launchPdl(kernel, dim3(grid), dim3(320), smem, st, mapIn, mapW, mapOut, a), "conv3x3 (halo) launch");
    DK_CUDA(cudaGetLastError(), "conv3x3 (halo rows, TMA + tcgen05) launch");
    if (pooled) *pooled = fusePool;
    return DK_OK;
}

// Output pixels (w x h) of a per-tap tile: 128 columns of a row for the row-tap mode.
inline uint32_t tapTileWidth(uint32_t w, bool rowTap) {
    uint32_t tw = 1;
    while (tw * 2u <= w && tw < 128u) tw *= 2u;
    return rowTap ? 128u : tw;
}
// Estimated time in us of the kernel that takes a layer the tile kernel leaves: row-tap or per-tap up to 256
// output channels, mma.sync above.  Fitted with convTileTime to 740 pairs of times (400 shapes of 1 x 1 to 544 x 960
// pixels on 1 to 2,000 images, 16 to 480 channels, with and without staged stores); root mean square errors 12 %
// (mma.sync 25) and 11 %.  A round is one tile per CTA; its loads and MMAs run beside the previous one's stores.
float convTapTime(const ConvArgs& c, uint32_t sms, size_t optin) {
    const uint32_t chunks = (c.cin + 63u) / 64u;
    if (c.cout > 256u) {
        const float blocks = (float)((c.M + 127u) / 128u) * (float)c.cout / 64.0f;
        return 5.9f + 9.0f * (float)c.cin * (0.0095f + 1.28e-4f * blocks);
    }
    const bool rowTap = c.w_ >= 128u && tmaSmemBytes(c.cout, false, 2u, true) <= optin;
    const uint32_t tw = tapTileWidth(c.w_, rowTap), th = 128u / tw;
    const uint64_t tiles = (uint64_t)c.n * ((c.w_ + tw - 1u) / tw) * ((c.h + th - 1u) / th);
    const bool staged = stagedStores(c) && tmaSmemBytes(c.cout, true, rowTap ? 2u : kTmaStagesMin, rowTap) <= optin;
    const float N = (float)c.cout, fill = (float)c.M / (128.0f * (float)tiles);
    const float mma = 9.0f * (float)chunks * (rowTap ? 0.14f + 4.2e-4f * N : 0.245f + 5.4e-4f * N);
    return 4.1f + (float)((tiles + sms - 1u) / sms) * std::max(mma, (staged ? 0.044f : 0.107f) * N * fill);
}
// The same of the tile kernel: `items` work items of kT tiles, nB output channels each; `pixels` of them in all.
float convTileTime(const ConvArgs& c, uint32_t sms, uint32_t kT, uint32_t nB, uint64_t items, uint64_t pixels,
                   bool staged) {
    const float N = (float)nB, fill = (float)c.M / (float)pixels;
    const float mma = (float)((c.cin + 63u) / 64u) * (kT == 2u ? 1.9f + 0.0101f * N : 0.84f + 0.0119f * N);
    return 3.7f + (float)((items + sms - 1u) / sms) * std::max(mma, (staged ? 0.031f : 0.084f) * N * (float)kT * fill);
}

// The 2-D halo-tile kernel's launch, or kHaloUnfit (nothing launched).
int launchConvTile(const ConvArgs& c, cudaStream_t st) {
    const uint32_t chunks = (c.cin + 63u) / 64u;
    if (chunks > kTileChunksMax) return kHaloUnfit;
    const uint32_t sms = (uint32_t)deviceProp().multiProcessorCount;
    const size_t optin = (size_t)deviceProp().sharedMemPerBlockOptin;
    const uint64_t tiles = (uint64_t)c.n * ((c.w_ + kTileW - 1u) / kTileW) * ((c.h + kTileH - 1u) / kTileH);
    if (tiles >= (1ull << 27)) return kHaloUnfit;
    TileConvArgs a;
    auto bytes = [&](uint32_t kT, uint32_t nB, uint32_t aSlots, uint32_t wStages, bool staged) {
        return (size_t)aSlots * chunks * (kT == 2u ? tileChunkBytes<2>() : tileChunkBytes<1>()) +
               (size_t)wStages * kTilePairs * nB * 128u + (staged ? tileStageBytes(nB) : 0u) + 1024u +
               kTileBarBytes;
    };
    const bool wantStaged = stagedStores(c);
    // Two tiles per item, which halves the weights read, where there are enough of them and they fit with
    // their epilogue's staging; on narrow images with the fewest blocks of at least 64 output channels that
    // fit.  (Smaller blocks, or splitting where that leaves each SM an item or two, are slower: 240 to 96
    // channels on two images of 35 x 232 21 us, whole single tiles 11; wide images 141 us against the
    // row-tap kernel's 86, 192 to 128 on 13 of 225 x 82.)
    bool pair = false;
    const uint32_t most = c.w_ < 128u && tiles >= 2ull * sms ? std::max(1u, c.cout / 64u) : 1u;
    for (a.nSplit = 0u; !pair && a.nSplit < most;) {
        ++a.nSplit;
        a.nB = c.cout / a.nSplit;
        pair = c.cout % (16u * a.nSplit) == 0u && a.nB <= 128u && tiles >= 2ull * sms &&
               bytes(2u, a.nB, 1u, kTileWStagesMin, wantStaged) <= optin;
    }
    if (!pair) {
        // Wide images in single tiles (up to 256 output channels: the row-tap kernel takes no more) read
        // more weights than the row-tap kernel's rows: 96 to 128 channels at 240 x 136 15.5 against 12.1 us,
        // 224 to 96 at 480 x 272 63 against 52.
        if (c.w_ >= 128u && c.cout <= 256u) return kHaloUnfit;
        // Output channels per CTA: the most blocks of at least 32 that still find an SM each where the
        // tiles are few, and more where a block does not fit -- with its epilogue's staging while it keeps
        // 64 channels: 96 to 224 channels on 16 images of 64 x 64 took 60 us with lane-by-lane stores, 30 staged.
        a.nSplit = 1u;
        for (uint32_t k = 2u; k <= c.cout / 32u; ++k)
            if (c.cout % (16u * k) == 0u && tiles * k <= sms) a.nSplit = k;
        auto fits = [&](uint32_t k, bool staged) {
            return c.cout % (16u * k) == 0u && c.cout <= 256u * k &&
                   bytes(1u, c.cout / k, 1u, kTileWStagesMin, staged) <= optin;
        };
        uint32_t k = a.nSplit;
        while (!fits(k, wantStaged) && c.cout >= 64u * (k + 1u)) ++k;
        if (fits(k, wantStaged)) a.nSplit = k;
        while (!fits(a.nSplit, false) && a.nSplit < c.cout / 16u) ++a.nSplit;
        a.nB = c.cout / a.nSplit;
        if (bytes(1u, a.nB, 1u, kTileWStagesMin, false) > optin) return kHaloUnfit;
        // Many small blocks (channel counts with few divisors): 16 to 272 channels at 480 x 272 take 124 us
        // in single tiles, 83 in pairs.
        pair = a.nB < 64u && tiles * a.nSplit >= 2ull * sms &&
               bytes(2u, a.nB, 1u, kTileWStagesMin, wantStaged) <= optin;
    }
    if (tiles * a.nSplit >= (1ull << 31)) return kHaloUnfit;
    a.cols = (a.nB + 31u) / 32u * 32u;
    const uint32_t kT = pair ? 2u : 1u;
    const bool staged = wantStaged && bytes(kT, a.nB, 1u, kTileWStagesMin, true) <= optin;
    a.aSlots = bytes(kT, a.nB, 2u, kTileWStagesMin, staged) <= optin ? 2u : 1u;
    a.wStages = kTileWStagesMin;
    while (a.wStages < kTileWStagesMax && bytes(kT, a.nB, a.aSlots, a.wStages + 1u, staged) <= optin) ++a.wStages;
    const size_t smem = bytes(kT, a.nB, a.aSlots, a.wStages, staged);
    a.bias = c.bias;
    a.out = c.out;
    a.n = c.n;
    a.h = c.h;
    a.w = c.w_;
    a.ldo = c.ldo;
    a.coOff = c.coOff;
    a.tilesX = (c.w_ + kT * kTileW - 1u) / (kT * kTileW);
    a.tilesY = (c.h + kTileH - 1u) / kTileH;
    a.items = c.n * a.tilesX * a.tilesY * a.nSplit;
    // A tile is 8 x 16 pixels of one image whatever its shape, and a pair twice that: images a few pixels wide or
    // high go to the other kernels, which take up to 128 of their pixels in a tile (160 to 192 channels on 353 of
    // 1 x 40: 118 us in tiles, 28 per tap; 176 to 208 on 620 of 33 x 4 210 and 163; 208 to 288 on 1,299 of 3 x 1
    // 173, mma.sync 35).  Only where the estimates are 5 % apart: that is 69 of the 82 fitted pairs which
    // tiles slow down by more than 3 %, and one that they speed up (by 4 %).
    if (convTapTime(c, sms, optin) <
        0.95f * convTileTime(c, sms, kT, a.nB, a.items, (uint64_t)c.n * a.tilesX * a.tilesY * kT * kTileW * kTileH, staged))
        return kHaloUnfit;
    a.chunks = chunks;
    a.lastSteps = (c.cin - (chunks - 1u) * 64u + 15u) / 16u;
    a.pairs = 9u * chunks;
    a.rowOrder = c.w_ >= 128u && tmaSmemBytes(c.cout, false, 2u, true) <= optin ? 1u : 0u;  // launchConvTma's choice
    a.act = c.act;
    a.accumulate = c.accumulate;
    a.staged = staged ? 1 : 0;
    EncodeTiledFn enc = encodeTiled();
    if (!enc) return fail(DK_ERROR_COMMAND_FAILED, "cuTensorMapEncodeTiled is not available");
    alignas(64) CUtensorMap mapIn, mapW;
    cuuint32_t unit[4] = {1u, 1u, 1u, 1u};
    cuuint64_t dimIn[4] = {c.cin, c.w_, c.h, c.n};
    cuuint64_t strideIn[3] = {(cuuint64_t)c.ldi * 2u, (cuuint64_t)c.w_ * c.ldi * 2u, (cuuint64_t)c.h * c.w_ * c.ldi * 2u};
    cuuint32_t boxIn[4] = {64u, kT * kTileW + 2u, kTileH + 2u, 1u};
    CUresult r = enc(&mapIn, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<__nv_bfloat16*>(c.in), dimIn, strideIn,
                     boxIn, unit, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(DK_ERROR_INVALID_ARGUMENT, "activation tensor map rejected");
    cuuint64_t dimW[3] = {c.cin, 9u, c.cout};
    cuuint64_t strideW[2] = {(cuuint64_t)c.cin * 2u, (cuuint64_t)9u * c.cin * 2u};
    cuuint32_t boxW[3] = {64u, 1u, a.nB};
    r = enc(&mapW, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(c.w), dimW, strideW, boxW, unit,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(DK_ERROR_INVALID_ARGUMENT, "weight tensor map rejected");
    static SmemLimit limits[2];
    DK_CUDA(raiseSmemLimit(limits[pair], pair ? k_conv3x3_tile<2> : k_conv3x3_tile<1>), "conv3x3 (tiles) shared memory");
    const dim3 grid(std::min(sms, a.items));
    DK_CUDA(launchPdl(pair ? k_conv3x3_tile<2> : k_conv3x3_tile<1>, grid, dim3(352), smem, st, mapIn, mapW, a),
            "conv3x3 (tiles) launch");
    return DK_OK;
}

// rowTap: the row-tap mode (images at least 128 pixels wide); else one stage
// per (tap, chunk) over 2-D tiles.
int launchConvTma(const ConvArgs& c, cudaStream_t st, bool rowTap) {
    rowTap = rowTap && c.w_ >= 128u;
    EncodeTiledFn enc = encodeTiled();
    if (!enc) return fail(DK_ERROR_COMMAND_FAILED, "cuTensorMapEncodeTiled is not available");
    TmaConvArgs a;
    a.bias = c.bias;
    a.out = c.out;
    a.n = c.n;
    a.h = c.h;
    a.w = c.w_;
    a.cin = c.cin;
    a.cout = c.cout;
    a.ldo = c.ldo;
    a.coOff = c.coOff;
    a.act = c.act;
    a.accumulate = c.accumulate;
    a.tw = tapTileWidth(c.w_, rowTap);
    a.th = 128u / a.tw;
    a.tilesX = (c.w_ + a.tw - 1) / a.tw;
    a.tilesY = (c.h + a.th - 1) / a.th;
    a.numTiles = a.tilesX * a.tilesY * c.n;
    a.chunks = (c.cin + 63u) / 64u;
    a.cols = 32u;
    while (a.cols < c.cout) a.cols <<= 1;
    alignas(64) CUtensorMap mapIn, mapW;
    cuuint64_t dimIn[4] = {c.cin, c.w_, c.h, c.n};
    cuuint64_t strideIn[3] = {(cuuint64_t)c.ldi * 2u, (cuuint64_t)c.w_ * c.ldi * 2u, (cuuint64_t)c.h * c.w_ * c.ldi * 2u};
    cuuint32_t boxIn[4] = {64u, rowTap ? kHaloPix : a.tw, a.th, 1u};
    cuuint32_t unit[4] = {1u, 1u, 1u, 1u};
    CUresult r = enc(&mapIn, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<__nv_bfloat16*>(c.in), dimIn, strideIn,
                     boxIn, unit, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(DK_ERROR_INVALID_ARGUMENT, "activation tensor map rejected");
    cuuint64_t dimW[3] = {c.cin, 9u, c.cout};
    cuuint64_t strideW[2] = {(cuuint64_t)c.cin * 2u, (cuuint64_t)9u * c.cin * 2u};
    cuuint32_t boxW[3] = {64u, 1u, c.cout};
    r = enc(&mapW, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(c.w), dimW, strideW, boxW, unit,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(DK_ERROR_INVALID_ARGUMENT, "weight tensor map rejected");
    const size_t optin = (size_t)deviceProp().sharedMemPerBlockOptin;
    const uint32_t minStages = rowTap ? 2u : kTmaStagesMin;
    if (tmaSmemBytes(c.cout, false, minStages, rowTap) > optin) {
        if (rowTap) return launchConvTma(c, st, false);
        return fail(DK_ERROR_INVALID_ARGUMENT, "conv3x3: the layer does not fit shared memory");
    }
    const bool staged = stagedStores(c) && tmaSmemBytes(c.cout, true, minStages, rowTap) <= optin;
    uint32_t stages = minStages;
    const uint32_t stageCap = depthCap("DK_CONV_STAGES", minStages, kTmaStagesMax);
    while (stages < stageCap && tmaSmemBytes(c.cout, staged, stages + 1u, rowTap) <= optin) ++stages;
    a.staged = staged ? 1 : 0;
    a.stages = stages;
    size_t smem = tmaSmemBytes(c.cout, staged, stages, rowTap);
    static SmemLimit limits[2];
    DK_CUDA(raiseSmemLimit(limits[rowTap], rowTap ? k_conv3x3_tma<true> : k_conv3x3_tma<false>), "conv3x3 shared memory");
    uint32_t grid = (uint32_t)deviceProp().multiProcessorCount;
    if (grid > a.numTiles) grid = a.numTiles;
    if (rowTap)
        DK_CUDA(launchPdl(k_conv3x3_tma<true>, dim3(grid), dim3(320), smem, st, mapIn, mapW, a), "conv3x3 launch");
    else
        DK_CUDA(launchPdl(k_conv3x3_tma<false>, dim3(grid), dim3(320), smem, st, mapIn, mapW, a), "conv3x3 launch");
    DK_CUDA(cudaGetLastError(), "conv3x3 (TMA + tcgen05) launch");
    return DK_OK;
}

// Pixels per block of the mma.sync kernel: blocks for the GPU several times over, 256 pixels at least.
uint32_t wgradMmaChunk(uint64_t M, uint32_t cin, uint32_t cout) {
    const uint32_t tiles = ((cout + 63u) / 64u) * ((cin + 63u) / 64u);
    const uint64_t target = (uint64_t)deviceProp().multiProcessorCount * 8u;
    const uint64_t perTile = (target + 9u * tiles - 1u) / (9u * tiles);
    const uint64_t chunk = ((M + perTile - 1u) / perTile + 31u) / 32u * 32u;
    return (uint32_t)std::max<uint64_t>(chunk, 256u);
}

int launchWgradMma(const __nv_bfloat16* in, uint32_t ldi, const __nv_bfloat16* dout, uint32_t ldd, uint32_t n,
                   uint32_t h, uint32_t w, uint32_t cin, uint32_t cout, float* dw, cudaStream_t st) {
    const uint64_t M = (uint64_t)n * h * w;
    const uint32_t chunk = wgradMmaChunk(M, cin, cout), tiles = ((cout + 63u) / 64u) * ((cin + 63u) / 64u);
    const WgradMmaArgs a{in, dout, dw, n, h, w, cin, ldi, cout, ldd, (uint32_t)M, chunk};
    k_conv3x3_wgrad_mma<<<dim3((uint32_t)((M + chunk - 1u) / chunk), tiles, 9), 128, 0, st>>>(a);
    DK_CUDA(cudaGetLastError(), "conv3x3 wgrad launch");
    return DK_OK;
}

// The weight gradient's launch: input blocks per CTA from the accumulator
// columns (3 x coB per block of 32 channels) and two pipeline stages of shared
// memory, fewer where the pixel tiles alone would leave SMs idle, two at most.
// With three, 96 to 32 channels on 16 x 256^2 take 106 us instead of 133, up to
// 1 % of a training step, in twice as many sums: 9.0e-6 from 64 bits instead of
// 2.2e-5 (mma.sync 2.7e-5), and up to 3e-5 from the gradients that both the
// mma.sync kernel and this one have given so far.  Two keep those.
int launchWgrad(const __nv_bfloat16* in, uint32_t ldi, const __nv_bfloat16* dout, uint32_t ldd, uint32_t n, uint32_t h,
                uint32_t w, uint32_t cin, uint32_t cout, float* dw, cudaStream_t st) {
    if (deviceProp().multiProcessorCount == 0) ensureDevice();
    const uint32_t sms = (uint32_t)deviceProp().multiProcessorCount;
    const size_t budget = (size_t)deviceProp().sharedMemPerBlockOptin - 1024u - kWgBarBytes;
    WgradArgs a;
    a.dw = dw;
    a.n = n;
    a.w = w;
    a.h = h;
    a.cin = cin;
    a.cout = cout;
    a.tilesX = (w + kWgTile - 1u) / kWgTile;
    a.tilesY = (h + kWgTile - 1u) / kWgTile;
    a.numTiles = a.tilesX * a.tilesY * n;
    a.chunks = (cin + 31u) / 32u;
    const uint32_t coBlocks = (cout + kWgCoMax - 1u) / kWgCoMax;
    a.coB = ((cout + coBlocks - 1u) / coBlocks + 15u) / 16u * 16u;
    a.coChunks = (a.coB + 31u) / 32u;
    auto stageBytes = [&](uint32_t cpc) { return (size_t)cpc * kWgInSlot + (size_t)a.coChunks * kWgOutSlot; };
    a.cpc = 1u;
    while (a.cpc < std::min(a.chunks, 2u) && 3u * a.coB * (a.cpc + 1u) <= 512u && 2u * stageBytes(a.cpc + 1u) <= budget) ++a.cpc;
    while (a.cpc > 1u && (uint64_t)a.numTiles * coBlocks * ((a.chunks + a.cpc - 1u) / a.cpc) < sms) --a.cpc;
    a.ciGroups = (a.chunks + a.cpc - 1u) / a.cpc;
    a.cpc = (a.chunks + a.ciGroups - 1u) / a.ciGroups;
    const uint32_t groups = coBlocks * a.ciGroups;
    // The tensor core truncates when it accumulates, so a gradient's error grows with the K steps of one sum and
    // falls with the number of sums it is made of.  They are as many as the mma.sync kernel's (runs of up to 512
    // pixels are not worth a split), a K step with fewer than 16 pixels counting for a third more than its pixels or
    // as a whole one, and no sum takes more than kWgRunMax tiles.  Where one CTA per SM makes fewer, a CTA sums into two sets of
    // accumulators if they fit, and then the pixels are split further, in whole rounds of CTAs.
    const uint64_t M = (uint64_t)n * h * w;
    const float pieces = (float)M / (float)std::max(wgradMmaChunk(M, cin, cout), 512u);
    const float ragged = std::min(1.0f + 0.3f * (float)(w % kWgTile) / (float)w, (float)(a.tilesX * kWgTile) / (float)w);
    const uint32_t sums = std::max((uint32_t)(pieces * ragged), (a.numTiles + kWgRunMax - 1u) / kWgRunMax);
    uint32_t gx = std::max(1u, sms / groups);
    a.sets = sums > gx && 6u * a.cpc * a.coB <= 512u ? 2u : 1u;
    if (sums > gx * a.sets) {
        const uint64_t splits = (sums + a.sets - 1u) / a.sets, rounds = (splits * groups + sms - 1u) / sms;
        gx = (uint32_t)std::max<uint64_t>(splits, rounds * sms / groups);
    }
    gx = std::min(gx, a.numTiles);
    // Both kernels' times in us, fitted to 260 shapes from 1 x 1 pixel to 16 x 256^2 on 16 to 512 channels (root
    // mean square errors 7 and 6 %): this one's read-out of 9 x 32 x coB sums a block and its tiles, whatever
    // part of a tile the image fills, against the other's pixels.  The choice costs 8 % or more on two of
    // them (19 and 13 %); 128 to 160 channels at 16 x 16 22.8 -> 8.5 us, 80 to 144 on 2 of 20 x 25 24.9 -> 10.4.
    const float tilesPerCta = (float)((a.numTiles + gx - 1u) / gx), rounds = (float)((gx * (uint64_t)groups + sms - 1u) / sms);
    const float here = 5.5f + rounds * (0.1f * (float)(a.cpc * a.coB) +
                                        tilesPerCta * (0.2f + (float)a.cpc * (0.8f + 0.0062f * (float)a.coB)));
    const float mma = 4.2f + 0.013f * (float)std::min<uint64_t>(M, 256u) +
                      4.0e-4f * (float)M * (float)(((cin + 63u) / 64u) * ((cout + 63u) / 64u));
    if (mma < here) return launchWgradMma(in, ldi, dout, ldd, n, h, w, cin, cout, dw, st);
    EncodeTiledFn enc = encodeTiled();
    if (!enc) return fail(DK_ERROR_COMMAND_FAILED, "cuTensorMapEncodeTiled is not available");
    a.stages = 2u;
    while (a.stages < kWgStagesMax && (a.stages + 1u) * stageBytes(a.cpc) <= budget) ++a.stages;
    a.cols = 32u;
    while (a.cols < 3u * a.sets * a.cpc * a.coB) a.cols <<= 1;
    alignas(64) CUtensorMap mapIn, mapOut;
    cuuint32_t unit[4] = {1u, 1u, 1u, 1u};
    auto encode = [&](CUtensorMap* map, const __nv_bfloat16* p, uint32_t ld, uint32_t c, uint32_t edge) {
        cuuint64_t dims[4] = {c, w, h, n};
        cuuint64_t strides[3] = {(cuuint64_t)ld * 2u, (cuuint64_t)w * ld * 2u, (cuuint64_t)h * w * ld * 2u};
        cuuint32_t box[4] = {32u, edge, edge, 1u};
        return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<__nv_bfloat16*>(p), dims, strides, box, unit,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    if (encode(&mapIn, in, ldi, cin, kWgHalo) != CUDA_SUCCESS)
        return fail(DK_ERROR_INVALID_ARGUMENT, "activation tensor map rejected");
    if (encode(&mapOut, dout, ldd, cout, kWgTile) != CUDA_SUCCESS)
        return fail(DK_ERROR_INVALID_ARGUMENT, "gradient tensor map rejected");
    const size_t smem = a.stages * stageBytes(a.cpc) + 1024u + kWgBarBytes;
    static SmemLimit limit;
    DK_CUDA(raiseSmemLimit(limit, k_conv3x3_wgrad), "conv3x3 wgrad shared memory");
    k_conv3x3_wgrad<<<dim3(gx, groups), 128, smem, st>>>(mapIn, mapOut, a);
    DK_CUDA(cudaGetLastError(), "conv3x3 wgrad launch");
    return DK_OK;
}

}  // namespace
}  // namespace dk

using bf16 = __nv_bfloat16;

extern "C" {

int dk_unet_conv3x3(const void* in, uint32_t n, uint32_t h, uint32_t w, uint32_t cin, uint32_t ldi,
                    const void* weight, const float* bias, uint32_t cout, void* out, uint32_t ldo, uint32_t coOff,
                    int act, int accumulate, void* stream) {
    if (!in || !weight || !out) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_conv3x3: null argument");
    if (!dk::aligned16(cin) || !dk::aligned16(cout) || ldi < cin || ldo < coOff + cout || ldi % 8u || ldo % 2u ||
        coOff % 2u)
        return dk::fail(DK_ERROR_INVALID_ARGUMENT,
                        "dk_unet_conv3x3: channel counts must be multiples of 16 within their leading dimensions");
    uint64_t M = (uint64_t)n * h * w;
    if (M == 0) return DK_OK;
    if (M >= (1ull << 31)) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_conv3x3: tensor too large");
    dk::ConvArgs a{static_cast<const bf16*>(in), static_cast<const bf16*>(weight), bias, static_cast<bf16*>(out),
                   n, h, w, cin, ldi, cout, ldo, coOff, (uint32_t)M, act, accumulate};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // More than 256 output channels (one accumulator) go in tiles too, split over CTAs: 128 to 288 channels
    // on 16 images of 32 x 32 take 13 us, with the mma.sync kernel below 98; 16 to 272 at 480 x 272 82 and 192.
    if (dk::g_convPath == 3) {
        int rc = dk::launchConvHalo(a, st);
        if (rc == dk::kHaloUnfit) rc = dk::launchConvTile(a, st);
        if (rc != dk::kHaloUnfit) return rc;
    }
    if (dk::g_convPath >= 2 && cout <= 256u) {
        int rc = dk::launchConvTma(a, st, dk::g_convPath == 3);
        if (rc != DK_OK) return rc;
        return DK_OK;
    }
    if (dk::g_convPath == 1 && cout <= 256u) {
        uint32_t cols = 32u;
        while (cols < cout) cols <<= 1;
        size_t smem = dk::tcSmemBytes(cout);
        static dk::SmemLimit limit;
        DK_CUDA(dk::raiseSmemLimit(limit, dk::k_conv3x3_tc), "conv3x3 shared memory");
        dk::k_conv3x3_tc<<<(uint32_t)((M + dk::kTcRows - 1) / dk::kTcRows), 128, smem, st>>>(a, cols);
        DK_CUDA(cudaGetLastError(), "conv3x3 (tcgen05) launch");
        return DK_OK;
    }
    dim3 grid((uint32_t)((M + dk::kBM - 1) / dk::kBM), 1);
    if (cout % 64u == 0) {
        grid.y = cout / 64u;
        dk::k_conv3x3_fwd<64><<<grid, 128, 0, st>>>(a);
    } else if (cout % 32u == 0) {
        grid.y = cout / 32u;
        dk::k_conv3x3_fwd<32><<<grid, 128, 0, st>>>(a);
    } else {
        grid.y = cout / 16u;
        dk::k_conv3x3_fwd<16><<<grid, 128, 0, st>>>(a);
    }
    DK_CUDA(cudaGetLastError(), "conv3x3 launch");
    return DK_OK;
}

int dk_unet_conv3x3_wgrad(const void* in, uint32_t ldi, const void* dout, uint32_t ldd, uint32_t n, uint32_t h,
                          uint32_t w, uint32_t cin, uint32_t cout, float* dweight, void* stream) {
    if (!in || !dout || !dweight) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_conv3x3_wgrad: null argument");
    if (!dk::aligned16(cin) || !dk::aligned16(cout) || ldi < cin || ldd < cout || ldi % 8u || ldd % 8u)
        return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_conv3x3_wgrad: channel counts must be multiples of 16");
    if (reinterpret_cast<uintptr_t>(in) % 16u || reinterpret_cast<uintptr_t>(dout) % 16u)
        return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_conv3x3_wgrad: tensors must be 16-byte aligned");
    uint64_t M = (uint64_t)n * h * w;
    if (M == 0) return DK_OK;
    if (M >= (1ull << 31)) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_conv3x3_wgrad: tensor too large");
    return dk::launchWgrad(static_cast<const bf16*>(in), ldi, static_cast<const bf16*>(dout), ldd, n, h, w, cin, cout,
                           dweight, static_cast<cudaStream_t>(stream));
}

int dk_unet_relu_backward(const void* out, uint32_t ldo, const void* dout, uint32_t ldd, void* dpre, uint32_t ldp,
                          uint32_t c, uint32_t pixels, void* stream) {
    if (!out || !dout || !dpre || c % 2u) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_relu_backward");
    const uint64_t total8 = (uint64_t)pixels * (c / 8u);
    if (dk::vec8({c, ldo, ldd, ldp}, {out, dout, dpre}, total8)) {
        dk::k_relu_backward8<<<dk::gridFor(total8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
            static_cast<const bf16*>(out), ldo, static_cast<const bf16*>(dout), ldd, static_cast<bf16*>(dpre), ldp,
            c / 8u, (uint32_t)total8);
        DK_CUDA(cudaGetLastError(), "relu backward launch");
        return DK_OK;
    }
    dk::k_relu_backward<<<dk::gridFor((uint64_t)pixels * c / 2), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(out), ldo, static_cast<const bf16*>(dout), ldd, static_cast<bf16*>(dpre), ldp, c,
        pixels);
    DK_CUDA(cudaGetLastError(), "relu backward launch");
    return DK_OK;
}

int dk_unet_bias_grad(const void* dpre, uint32_t ld, uint32_t c, uint32_t pixels, float* dbias, void* stream) {
    if (!dpre || !dbias || c == 0 || c > 256u) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_bias_grad");
    if (dk::vec8({c, ld}, {dpre}, (uint64_t)pixels * (c / 8u)))
        return dk::launchReluBias<false>(nullptr, 0, dpre, ld, nullptr, 0, c, pixels, dbias, stream);
    uint32_t lanes = 256u / c;
    uint64_t blocks = ((uint64_t)pixels + lanes * 64u - 1) / (lanes * 64u);
    int grid = (int)(blocks < 1 ? 1 : (blocks > 1024 ? 1024 : blocks));
    dk::k_bias_grad<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const bf16*>(dpre), ld, c, pixels,
                                                                          dbias);
    DK_CUDA(cudaGetLastError(), "bias grad launch");
    return DK_OK;
}

int dk_unet_relu_bias_backward(const void* out, uint32_t ldo, const void* dout, uint32_t ldd, void* dpre, uint32_t ldp,
                               uint32_t c, uint32_t pixels, float* dbias, void* stream) {
    if (!out || !dout || !dpre || !dbias || c == 0 || c % 2u || c > 256u)
        return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_relu_bias_backward");
    if (dk::vec8({c, ldo, ldd, ldp}, {out, dout, dpre}, (uint64_t)pixels * (c / 8u)))
        return dk::launchReluBias<true>(out, ldo, dout, ldd, dpre, ldp, c, pixels, dbias, stream);
    const int rc = dk_unet_relu_backward(out, ldo, dout, ldd, dpre, ldp, c, pixels, stream);
    return rc != DK_OK ? rc : dk_unet_bias_grad(dpre, ldp, c, pixels, dbias, stream);
}

int dk_unet_avgpool2(const void* in, uint32_t ldi, void* out, uint32_t ldo, uint32_t coOff, uint32_t c, uint32_t n,
                     uint32_t h, uint32_t w, void* stream) {
    if (!in || !out || c % 2u || h % 2u || w % 2u) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_avgpool2");
    const uint64_t total8 = (uint64_t)n * (h / 2u) * (w / 2u) * (c / 8u);
    if (dk::vec8({c, ldi, ldo, coOff}, {in, out}, total8)) {
        DK_CUDA(dk::launchPdl(dk::k_avgpool2_8, dim3(dk::gridFor(total8)), dim3(256), 0,
                              static_cast<cudaStream_t>(stream), static_cast<const bf16*>(in), ldi,
                              static_cast<bf16*>(out), ldo, coOff, c / 8u, h, w, (uint32_t)total8),
                "avgpool launch");
        return DK_OK;
    }
    dk::k_avgpool2<<<dk::gridFor((uint64_t)n * h * w / 4 * c / 2), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(in), ldi, static_cast<bf16*>(out), ldo, coOff, c, n, h, w);
    DK_CUDA(cudaGetLastError(), "avgpool launch");
    return DK_OK;
}

int dk_unet_conv3x3_avgpool2(const void* in, uint32_t n, uint32_t h, uint32_t w, uint32_t cin, uint32_t ldi,
                             const void* weight, const float* bias, uint32_t cout, void* out, uint32_t ldo,
                             uint32_t coOff, int act, void* pool, uint32_t poolLd, void* stream) {
    if (!pool || h % 2u || w % 2u || poolLd < cout)
        return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_conv3x3_avgpool2: pool target or odd extent");
    if (dk::g_convPath == 3 && cout <= 256u && in && weight && out && dk::aligned16(cin) && dk::aligned16(cout) &&
        ldi >= cin && ldo >= coOff + cout && ldi % 8u == 0u && ldo % 2u == 0u && coOff % 2u == 0u &&
        (uint64_t)n * h * w > 0 && (uint64_t)n * h * w < (1ull << 31)) {
        dk::ConvArgs a{static_cast<const bf16*>(in), static_cast<const bf16*>(weight), bias, static_cast<bf16*>(out),
                       n, h, w, cin, ldi, cout, ldo, coOff, (uint32_t)((uint64_t)n * h * w), act, 0};
        bool pooled = false;
        int rc = dk::launchConvHalo(a, static_cast<cudaStream_t>(stream), static_cast<bf16*>(pool), poolLd, &pooled);
        if (rc != dk::kHaloUnfit) {
            if (rc != DK_OK || pooled) return rc;
            return dk_unet_avgpool2(static_cast<const bf16*>(out) + coOff, ldo, pool, poolLd, 0u, cout, n, h, w, stream);
        }
    }
    int rc = dk_unet_conv3x3(in, n, h, w, cin, ldi, weight, bias, cout, out, ldo, coOff, act, 0, stream);
    if (rc != DK_OK) return rc;
    return dk_unet_avgpool2(static_cast<const bf16*>(out) + coOff, ldo, pool, poolLd, 0u, cout, n, h, w, stream);
}

int dk_unet_avgpool2_backward(const void* dout, uint32_t ldd, void* din, uint32_t ldi, uint32_t c, uint32_t n,
                              uint32_t h, uint32_t w, int accumulate, void* stream) {
    if (!dout || !din || c % 2u || h % 2u || w % 2u)
        return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_avgpool2_backward");
    const uint64_t total8 = (uint64_t)n * (h / 2u) * (w / 2u) * (c / 8u);
    if (dk::vec8({c, ldd, ldi}, {dout, din}, total8)) {
        dk::k_avgpool2_backward8<<<dk::gridFor(total8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
            static_cast<const bf16*>(dout), ldd, static_cast<bf16*>(din), ldi, c / 8u, h, w, accumulate,
            (uint32_t)total8);
        DK_CUDA(cudaGetLastError(), "avgpool backward launch");
        return DK_OK;
    }
    dk::k_avgpool2_backward<<<dk::gridFor((uint64_t)n * h * w * c / 2), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(dout), ldd, static_cast<bf16*>(din), ldi, c, n, h, w, accumulate);
    DK_CUDA(cudaGetLastError(), "avgpool backward launch");
    return DK_OK;
}

int dk_unet_upsample2(const void* in, uint32_t ldi, void* out, uint32_t ldo, uint32_t coOff, uint32_t c, uint32_t n,
                      uint32_t h, uint32_t w, void* stream) {
    if (!in || !out || c % 2u) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_upsample2");
    const uint64_t total8 = (uint64_t)n * h * w * (c / 8u);
    if (dk::vec8({c, ldi, ldo, coOff}, {in, out}, total8)) {
        DK_CUDA(dk::launchPdl(dk::k_upsample2_8, dim3(dk::gridFor(total8)), dim3(256), 0,
                              static_cast<cudaStream_t>(stream), static_cast<const bf16*>(in), ldi,
                              static_cast<bf16*>(out), ldo, coOff, c / 8u, h, w, (uint32_t)total8),
                "upsample launch");
        return DK_OK;
    }
    dk::k_upsample2<<<dk::gridFor((uint64_t)n * h * w * 4 * c / 2), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(in), ldi, static_cast<bf16*>(out), ldo, coOff, c, n, h, w);
    DK_CUDA(cudaGetLastError(), "upsample launch");
    return DK_OK;
}

int dk_unet_upsample2_backward(const void* dout, uint32_t ldd, uint32_t ciOff, void* din, uint32_t ldi, uint32_t c,
                               uint32_t n, uint32_t h, uint32_t w, void* stream) {
    if (!dout || !din || c % 2u) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_upsample2_backward");
    const uint64_t total8 = (uint64_t)n * h * w * (c / 8u);
    if (dk::vec8({c, ldd, ciOff, ldi}, {dout, din}, total8)) {
        dk::k_upsample2_backward8<<<dk::gridFor(total8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
            static_cast<const bf16*>(dout), ldd, ciOff, static_cast<bf16*>(din), ldi, c / 8u, h, w, (uint32_t)total8);
        DK_CUDA(cudaGetLastError(), "upsample backward launch");
        return DK_OK;
    }
    dk::k_upsample2_backward<<<dk::gridFor((uint64_t)n * h * w * c / 2), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(dout), ldd, ciOff, static_cast<bf16*>(din), ldi, c, n, h, w);
    DK_CUDA(cudaGetLastError(), "upsample backward launch");
    return DK_OK;
}

int dk_unet_copy_channels(const void* src, uint32_t lds, uint32_t sOff, void* dst, uint32_t ldd, uint32_t dOff,
                          uint32_t c, uint32_t pixels, int accumulate, void* stream) {
    if (!src || !dst || c % 2u || sOff % 2u || dOff % 2u)
        return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_copy_channels");
    const uint64_t total8 = (uint64_t)pixels * (c / 8u);
    if (dk::vec8({c, lds, sOff, ldd, dOff}, {src, dst}, total8)) {
        dk::k_copy_channels8<<<dk::gridFor(total8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
            static_cast<const bf16*>(src), lds, sOff, static_cast<bf16*>(dst), ldd, dOff, c / 8u, accumulate,
            (uint32_t)total8);
        DK_CUDA(cudaGetLastError(), "copy channels launch");
        return DK_OK;
    }
    dk::k_copy_channels<<<dk::gridFor((uint64_t)pixels * c / 2), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(src), lds, sOff, static_cast<bf16*>(dst), ldd, dOff, c, pixels, accumulate);
    DK_CUDA(cudaGetLastError(), "copy channels launch");
    return DK_OK;
}

int dk_unet_pack_input(const float* beauty, const float* albedo, const float* normal, const float* depth,
                       uint32_t imgW, uint32_t imgH, uint32_t x0, uint32_t y0, void* out, uint32_t h, uint32_t w,
                       uint32_t batchIndex, void* stream) {
    if (!beauty || !albedo || !normal || !depth || !out) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_pack_input");
    dk::k_pack_input<<<dk::gridFor((uint64_t)h * w), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const float4*>(beauty), reinterpret_cast<const float4*>(albedo),
        reinterpret_cast<const float4*>(normal), reinterpret_cast<const float4*>(depth), imgW, imgH, x0, y0,
        static_cast<bf16*>(out), h, w, batchIndex, reinterpret_cast<uintptr_t>(out) % 16u == 0u);
    DK_CUDA(cudaGetLastError(), "pack input launch");
    return DK_OK;
}

int dk_unet_l1_loss(const void* pred, uint32_t ldp, const float* target, uint32_t pixels, void* grad, uint32_t ldg,
                    float* loss, void* stream) {
    if (!pred || !target || !grad || !loss || ldp < 3u || ldg < 3u)
        return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_l1_loss");
    dk::k_l1_loss<<<dk::gridFor(pixels), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(pred), ldp, nullptr, 0u, reinterpret_cast<const float4*>(target), pixels,
        static_cast<bf16*>(grad), ldg, loss,
        dk::wide4({ldp}, {pred}), ldg == 16u && reinterpret_cast<uintptr_t>(grad) % 16u == 0u);
    DK_CUDA(cudaGetLastError(), "loss launch");
    return DK_OK;
}

int dk_unet_l1_loss_residual(const void* pred, uint32_t ldp, const void* base, uint32_t ldb, const float* target,
                             uint32_t pixels, void* grad, uint32_t ldg, float* loss, void* stream) {
    if (!pred || !base || !target || !grad || !loss || ldp < 3u || ldb < 3u || ldg < 3u)
        return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_l1_loss_residual");
    dk::k_l1_loss<<<dk::gridFor(pixels), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(pred), ldp, static_cast<const bf16*>(base), ldb,
        reinterpret_cast<const float4*>(target), pixels, static_cast<bf16*>(grad), ldg, loss,
        dk::wide4({ldp, ldb}, {pred, base}), ldg == 16u && reinterpret_cast<uintptr_t>(grad) % 16u == 0u);
    DK_CUDA(cudaGetLastError(), "loss launch");
    return DK_OK;
}

int dk_unet_unpack_output(const void* pred, uint32_t ldp, uint32_t h, uint32_t w, const float* alphaSrc, uint32_t imgW,
                          uint32_t imgH, uint32_t x0, uint32_t y0, float* out, void* stream) {
    if (!pred || !alphaSrc || !out) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_unpack_output");
    dk::k_unpack_output<<<dk::gridFor((uint64_t)h * w), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(pred), ldp, nullptr, 0u, h, w, reinterpret_cast<const float4*>(alphaSrc), imgW, imgH,
        x0, y0, reinterpret_cast<float4*>(out), dk::wide4({ldp}, {pred}));
    DK_CUDA(cudaGetLastError(), "unpack output launch");
    return DK_OK;
}

int dk_unet_unpack_output_residual(const void* pred, uint32_t ldp, const void* base, uint32_t ldb, uint32_t h,
                                   uint32_t w, const float* alphaSrc, uint32_t imgW, uint32_t imgH, uint32_t x0,
                                   uint32_t y0, float* out, void* stream) {
    if (!pred || !base || !alphaSrc || !out || ldb < 3u)
        return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_unpack_output_residual");
    dk::k_unpack_output<<<dk::gridFor((uint64_t)h * w), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const bf16*>(pred), ldp, static_cast<const bf16*>(base), ldb, h, w,
        reinterpret_cast<const float4*>(alphaSrc), imgW, imgH, x0, y0, reinterpret_cast<float4*>(out),
        dk::wide4({ldp, ldb}, {pred, base}));
    DK_CUDA(cudaGetLastError(), "unpack output launch");
    return DK_OK;
}

int dk_unet_adam(float* weights, const float* grad, float* m, float* v, uint32_t count, float lr, float beta1,
                 float beta2, float eps, uint32_t step, void* wbf16, void* wflip, uint32_t cout, uint32_t cin,
                 void* stream) {
    if (!weights || !grad || !m || !v || step == 0) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_adam");
    dk::k_adam<<<dk::gridFor(count), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        weights, grad, m, v, count, dk::adamRule(lr, beta1, beta2, eps, step), static_cast<bf16*>(wbf16),
        static_cast<bf16*>(wflip), cout, cin);
    DK_CUDA(cudaGetLastError(), "adam launch");
    return DK_OK;
}

int dk_unet_adam_groups(const dk_unet_adam_group* groups, uint32_t groupCount, float lr, float beta1, float beta2,
                        float eps, uint32_t step, void* stream) {
    if ((groupCount && !groups) || step == 0) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_adam_groups");
    for (uint32_t k = 0; k < groupCount; ++k)
        if (!groups[k].weights || !groups[k].grad || !groups[k].m || !groups[k].v)
            return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_adam_groups: null tensor");
    const dk::AdamRule rule = dk::adamRule(lr, beta1, beta2, eps, step);
    dk::AdamTable t;
    t.groups = 0;
    uint32_t blocks = 0;
    auto flush = [&]() -> int {
        if (t.groups == 0) return DK_OK;
        t.first[t.groups] = blocks;
        dk::k_adam_groups<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(t, rule);
        DK_CUDA(cudaGetLastError(), "adam launch");
        t.groups = 0;
        blocks = 0;
        return DK_OK;
    };
    for (uint32_t k = 0; k < groupCount; ++k) {
        const dk_unet_adam_group& g = groups[k];
        if (g.count == 0) continue;
        // The tiles take whole [cout][9][cin] layers in 16-byte pieces; other layouts go one tensor at a time.
        const bool tiled = g.wflip && (uint64_t)g.cout * 9u * g.cin == g.count && g.cin % 4u == 0u && g.cout % 4u == 0u &&
                           dk::vec8({}, {g.weights, g.grad, g.m, g.v, g.wbf16, g.wflip}, 1u);
        if (g.wflip && !tiled) {
            const int rc = dk_unet_adam(g.weights, g.grad, g.m, g.v, g.count, lr, beta1, beta2, eps, step, g.wbf16,
                                        g.wflip, g.cout, g.cin, stream);
            if (rc != DK_OK) return rc;
            continue;
        }
        t.g[t.groups] = g;
        t.first[t.groups++] = blocks;
        blocks += tiled ? 9u * ((g.cin + 31u) / 32u) * ((g.cout + 31u) / 32u) : (g.count + 1023u) / 1024u;
        if (t.groups == dk::kAdamGroups)
            if (const int rc = flush()) return rc;
    }
    return flush();
}

int dk_unet_set_conv_path(int path) {
    if (path < 0 || path > 3) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_set_conv_path: 0, 1, 2 or 3");
    dk::g_convPath = path;
    return DK_OK;
}

int dk_unet_error(int* out) {
    if (!out) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_error: null argument");
    int zero = 0;
    DK_CUDA(cudaMemcpyFromSymbol(out, dk::g_unetError, sizeof(int)), "read denoiser error flag");
    DK_CUDA(cudaMemcpyToSymbol(dk::g_unetError, &zero, sizeof(int)), "clear denoiser error flag");
    return DK_OK;
}

int dk_unet_weights_to_bf16(const float* weights, uint32_t count, void* wbf16, void* wflip, uint32_t cout, uint32_t cin,
                            void* stream) {
    if (!weights || !wbf16) return dk::fail(DK_ERROR_INVALID_ARGUMENT, "dk_unet_weights_to_bf16");
    dk::k_weights_to_bf16<<<dk::gridFor(count), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        weights, count, static_cast<bf16*>(wbf16), static_cast<bf16*>(wflip), cout, cin);
    DK_CUDA(cudaGetLastError(), "weights launch");
    return DK_OK;
}

}  // extern "C"
