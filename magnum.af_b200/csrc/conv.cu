// 3x3 convolutions of the warm-start U-net as implicit GEMMs on the 5th-generation
// tensor cores (tcgen05.mma kind::f16, BF16 operands, FP32 accumulation in tensor
// memory): the forward pass and the data gradient (k_conv) and the weight gradient
// (k_conv_wgrad).  Activations are pixel-major [P][Cp] (BF16, Cp a multiple of 8);
// tap t of pixel (b, y, x) is pixel (b, y + t/3 - 1, x + t%3 - 1), zero outside.
//
// Why implicit: an im2col matrix is nine times the activation and went through HBM
// twice per GEMM (FP32, and through col2im, for the data gradient).  Here the taps are
// gathered from the activation straight into shared memory by 16-byte cp.async (a
// chunk of 8 channels of one tap of one pixel, zero-filled outside the image); the
// nine reads of a pixel hit L2.  At level 0 (262144 pixels, 32-96 channels) the kernel
// is bound on those copies (128 pixels x 9 Cp x 2 bytes per tile), not on the MMA.
//
// Pipeline: kStages shared-memory stages of 64 K values; per stage one barrier, four
// MMAs issued by thread 0 and committed to the stage's mbarrier; a stage is refilled
// when the MMA that read it has completed, so up to kStages - 1 copies are in flight
// under the MMAs.  Every wait is bounded: a wait that gives up raises the device's flag
// (tc_error.hpp) and the CTA leaves without storing, freeing its tensor memory.
#include <cuda_bf16.h>

#include <algorithm>

#include "../../include/maf_b200.h"
#include "capi_internal.hpp"
#include "engine.hpp"
#include "tc_error.hpp"

namespace mafb {

namespace {

using bf16 = __nv_bfloat16;
constexpr int kBM = 128;     // rows of the accumulator (TMEM lanes)
constexpr int kBK = 64;      // K values per stage: one 128-byte swizzled row of BF16
constexpr int kStages = 3;
constexpr unsigned long long kWaitCycles = 4000000000ull;  // about 2 s at the boost clock

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor: 128-byte swizzle (layout type 2), descriptor
// version 1, addresses and offsets in 16-byte units.  K-major: sbo between 8-row
// groups, lbo unused.  MN-major: lbo between blocks of 64 MN values, sbo between
// groups of 8 K rows.
__device__ __forceinline__ uint64_t sdesc128(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (2ull << 61);
}

// Instruction descriptor: D FP32, A and B BF16, M = 128, N = BN; MN: both operands MN-major.
template <int BN, bool MN> constexpr uint32_t idesc() {
    return (1u << 4) | (1u << 7) | (1u << 10) | (MN ? (1u << 15) | (1u << 16) : 0u) | ((uint32_t)(BN >> 3) << 17) |
           ((uint32_t)(kBM >> 4) << 24);
}

__device__ __forceinline__ void umma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t id, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(a), "l"(b), "r"(id), "r"(acc));
}

__device__ __forceinline__ void umma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t phase) {
    const unsigned long long t0 = clock64();
    while (true) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(mbar), "r"(phase)
            : "memory");
        if (done) return true;
        if (clock64() - t0 > kWaitCycles) return false;
    }
}

// 16 bytes from src (zeros when !ok; src must be a mapped address either way)
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The tensor memory and barriers of a CTA of 128 threads.
struct Cta {
    uint32_t tmem, mbar;
};
template <int COLS> __device__ __forceinline__ Cta cta_begin(uint64_t* mbar, uint32_t* tmem_sh) {
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_sh)),
                     "r"(COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar + s)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return Cta{*tmem_sh, smem_u32(mbar)};
}
template <int COLS> __device__ __forceinline__ void cta_end(const Cta& c) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem), "r"(COLS));
}

// The K loop: load(kb, stage) issues the copies of K block kb into a stage, mma(stage,
// first) its MMAs (thread 0).  Returns whether every MMA completed; the accumulator is
// then visible to tcgen05.ld.
template <typename LOAD, typename MMA>
__device__ __forceinline__ bool mainloop(const Cta& c, int nkb, LOAD&& load, MMA&& mma) {
    for (int kb = 0; kb < kStages - 1; ++kb) {
        if (kb < nkb) load(kb, kb);
        asm volatile("cp.async.commit_group;\n" ::);
    }
    bool ok = true;
    int st = 0;
    for (int kb = 0; kb < nkb; ++kb) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 2) : "memory");
        // the stage was written through the generic proxy; the MMA reads it through the async proxy
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (__syncthreads_or(!ok)) break;
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            mma(st, kb == 0);
            umma_commit(c.mbar + 8 * st);
        }
        const int prev = st == 0 ? kStages - 1 : st - 1;  // stage of kb - 1 and of kb + kStages - 1
        if (kb + kStages - 1 < nkb) {
            if (kb > 0) ok = mbar_wait(c.mbar + 8 * prev, (uint32_t)((kb - 1) / kStages) & 1u);
            load(kb + kStages - 1, prev);
        }
        asm volatile("cp.async.commit_group;\n" ::);
        st = st == kStages - 1 ? 0 : st + 1;
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    if (ok) ok = mbar_wait(c.mbar + 8 * ((nkb - 1) % kStages), (uint32_t)((nkb - 1) / kStages) & 1u);
    ok = !__syncthreads_or(!ok);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return ok;
}

struct ConvArgs {
    const bf16* act;    // [P][Cp]
    const bf16* w;      // [N][9 Cp]
    const float* bias;  // [N] or null
    float* out;         // [P][ldo], channels 0 .. N-1
    bf16* outb;         // [P][ldb] (zero beyond N) or null
    int H, W, Cp, N, ldo, ldb, relu;
    int64_t P;
    TcFlag* err;
};

// out[p][n] = relu?(bias[n] + sum_{t, c} act[tap t of p][c] w[n][t Cp + c]): CTA =
// 128 pixels x BN channels, both operands K-major.
template <int BN>
__global__ void __launch_bounds__(128) k_conv(ConvArgs a) {
    constexpr int kA = kBM * 128, kStage = kA + BN * 128;
    extern __shared__ uint8_t raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t mbar[kStages];
    __shared__ uint32_t tmem_sh;
    const int tid = threadIdx.x;
    const Cta cta = cta_begin<BN>(mbar, &tmem_sh);
    const uint32_t sbase = smem_u32(sm);
    const int64_t m0 = (int64_t)blockIdx.x * kBM;
    const int n0 = blockIdx.y * BN;
    const int K = 9 * a.Cp;
    // thread (row group r0, chunk kc): rows r0 + 16 i of both tiles, K values 8 kc .. 8 kc + 7
    const int r0 = tid >> 3, kc = tid & 7;
    uint32_t valid[4];  // per row: the taps inside the image, 9 bits, two rows per word
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int64_t p = m0 + r0 + 16 * i;
        uint32_t v = 0;
        if (p < a.P) {
            const int x = (int)(p % a.W), y = (int)(p / a.W % a.H);
            const uint32_t xs = (x > 0 ? 1u : 0u) | 2u | (x + 1 < a.W ? 4u : 0u);
            v = (y > 0 ? xs : 0u) | (xs << 3) | (y + 1 < a.H ? xs << 6 : 0u);
        }
        if (i & 1) valid[i >> 1] |= v << 16;
        else valid[i >> 1] = v;
    }
    const uint32_t dst0 = (uint32_t)(r0 * 128 + ((kc ^ (r0 & 7)) * 16));  // rows 16 apart: same swizzle
    int tap = kc * 8 / a.Cp, ch = kc * 8 - tap * a.Cp;                    // of the next K block to load
    const bf16* pix = a.act + (m0 + r0) * a.Cp;
    const bf16* wrow = a.w + (int64_t)(n0 + r0) * K;
    auto load = [&](int kb, int st) {
        const int k = kb * kBK + kc * 8;
        const uint32_t d = sbase + st * kStage + dst0;
        const bool kin = k < K;
        const int dy = tap / 3 - 1, dx = tap - (dy + 1) * 3 - 1;
        const bf16* src = pix + (int64_t)(dy * a.W + dx) * a.Cp + ch;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const bool in = kin && ((valid[i >> 1] >> ((i & 1) * 16 + tap)) & 1u);
            copy16(d + i * 2048, in ? src + (int64_t)16 * i * a.Cp : a.act, in);
        }
#pragma unroll
        for (int i = 0; i < BN / 16; ++i) {
            const bool in = kin && n0 + r0 + 16 * i < a.N;
            copy16(d + kA + i * 2048, in ? wrow + (int64_t)16 * i * K + k : a.w, in);
        }
        ch += kBK;
        while (ch >= a.Cp) {
            ch -= a.Cp;
            ++tap;
        }
    };
    auto mma = [&](int st, bool first) {
        const uint32_t sa = sbase + st * kStage;
#pragma unroll
        for (int s = 0; s < kBK / 16; ++s)
            umma(cta.tmem, sdesc128(sa + 32 * s, 16, 1024), sdesc128(sa + kA + 32 * s, 16, 1024), idesc<BN, false>(),
                 first && s == 0 ? 0u : 1u);
    };
    const bool ok = mainloop(cta, (K + kBK - 1) / kBK, load, mma);
    if (ok) {
        const int64_t p = m0 + tid;  // warp w reads TMEM lanes 32 w ..: row tid of the tile
        const bool vec = a.N % 4 == 0 && a.ldo % 4 == 0;
        const int nout = a.outb ? max(a.N, a.ldb) : a.N;
#pragma unroll 1
        for (int c0 = 0; c0 < BN && n0 + c0 < nout; c0 += 16) {
            uint32_t u[16];
            __syncwarp();
            tmem_ld16(cta.tmem + ((uint32_t)(tid & ~31) << 16) + (uint32_t)c0, u);
            if (p >= a.P) continue;
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int n = n0 + c0 + j;
                float f = __uint_as_float(u[j]);
                if (n < a.N) {
                    if (a.bias) f += __ldg(a.bias + n);
                    if (a.relu) f = fmaxf(f, 0.f);
                } else {
                    f = 0.f;
                }
                v[j] = f;
            }
            float* o = a.out + p * a.ldo + n0 + c0;
            if (vec) {
#pragma unroll
                for (int j = 0; j < 16; j += 4)
                    if (n0 + c0 + j < a.N) *reinterpret_cast<float4*>(o + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (n0 + c0 + j < a.N) o[j] = v[j];
            }
            if (a.outb) {
                bf16* ob = a.outb + p * a.ldb + n0 + c0;
#pragma unroll
                for (int j = 0; j < 16; j += 8) {
                    if (n0 + c0 + j >= a.ldb) continue;
                    __align__(16) bf16 h[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) h[q] = __float2bfloat16_rn(v[j + q]);
                    *reinterpret_cast<uint4*>(ob + j) = *reinterpret_cast<const uint4*>(h);
                }
            }
        }
    } else if (tid == 0) {
        tc_raise(a.err);
    }
    cta_end<BN>(cta);
}

struct WgradArgs {
    const bf16* act;  // [P][Cp]
    const bf16* dy;   // [P][Np]
    float* work;      // [splits][9 Cp][Np]
    int H, W, Cp, Np;
    int64_t P, chunk;  // pixels per split, a multiple of kBK
    TcFlag* err;
};

// work[s][t Cp + c][n] = sum over the split's pixels of act[tap t of p][c] dy[p][n]:
// CTA = 128 (tap, channel) rows x BN output channels, K = pixels.  Both operands are
// stored pixel by pixel as they lie in memory, so they are MN-major: 64 channels are a
// swizzled 128-byte row per pixel.
template <int BN>
__global__ void __launch_bounds__(128) k_conv_wgrad(WgradArgs a) {
    constexpr int kBlk = kBK * 128;                       // 64 channels of 64 pixels
    constexpr int kA = 2 * kBlk, kStage = kA + (BN + 63) / 64 * kBlk;
    extern __shared__ uint8_t raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t mbar[kStages];
    __shared__ uint32_t tmem_sh;
    const int tid = threadIdx.x;
    const Cta cta = cta_begin<BN>(mbar, &tmem_sh);
    const uint32_t sbase = smem_u32(sm);
    const int M = 9 * a.Cp;
    const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;
    const int64_t p0 = (int64_t)blockIdx.z * a.chunk;
    const int64_t p1 = min(a.P, p0 + a.chunk);
    // A: thread = (chunk q of 8 channels of one tap, pixels pr + 8 i); the pixel's (x, y)
    // advances by 8 from copy to copy
    const int q = tid & 15, pr = tid >> 4;
    const int mq = m0 + 8 * q;
    const int tap = mq / a.Cp, ch = mq - tap * a.Cp;
    const int dy = tap / 3 - 1, dx = tap % 3 - 1;
    const bool mok = mq < M;
    int64_t pa = p0 + pr;
    int x = (int)(pa % a.W), y = (int)(pa / a.W % a.H);
    const bf16* asrc = a.act + (pa + dy * a.W + dx) * a.Cp + ch;
    // B: chunks of 8 output channels, consecutive threads take consecutive chunks of a pixel
    constexpr int BQ = BN / 8;
    auto load = [&](int kb, int st) {
        const uint32_t d = sbase + st * kStage;
#pragma unroll
        for (int i = 0; i < kBK / 8; ++i) {
            const int r = pr + 8 * i;
            const bool in = mok && pa < p1 && (unsigned)(y + dy) < (unsigned)a.H && (unsigned)(x + dx) < (unsigned)a.W;
            copy16(d + (q >> 3) * kBlk + r * 128 + (((q & 7) ^ (r & 7)) * 16), in ? asrc : a.act, in);
            pa += 8;
            asrc += (int64_t)8 * a.Cp;
            x += 8;
            while (x >= a.W) {
                x -= a.W;
                if (++y == a.H) y = 0;
            }
        }
        const int64_t pb = p0 + (int64_t)kb * kBK;
#pragma unroll
        for (int i = 0; i < kBK * BQ / 128; ++i) {
            const int e = tid + 128 * i, r = e / BQ, n = e - r * BQ;
            const bool in = pb + r < p1 && n0 + 8 * n < a.Np;
            copy16(d + kA + (n >> 3) * kBlk + r * 128 + (((n & 7) ^ (r & 7)) * 16),
                   in ? a.dy + (pb + r) * a.Np + n0 + 8 * n : a.dy, in);
        }
    };
    auto mma = [&](int st, bool first) {
        const uint32_t sa = sbase + st * kStage;
#pragma unroll
        for (int s = 0; s < kBK / 16; ++s)
            umma(cta.tmem, sdesc128(sa + 2048 * s, kBlk, 1024), sdesc128(sa + kA + 2048 * s, kBlk, 1024),
                 idesc<BN, true>(), first && s == 0 ? 0u : 1u);
    };
    const bool ok = mainloop(cta, (int)((p1 - p0 + kBK - 1) / kBK), load, mma);
    if (ok) {
        const int m = m0 + tid;
        float* o = a.work + ((int64_t)blockIdx.z * M + m) * a.Np + n0;
#pragma unroll 1
        for (int c0 = 0; c0 < BN && n0 + c0 < a.Np; c0 += 16) {
            uint32_t u[16];
            __syncwarp();
            tmem_ld16(cta.tmem + ((uint32_t)(tid & ~31) << 16) + (uint32_t)c0, u);
            if (m >= M) continue;
#pragma unroll
            for (int j = 0; j < 16; j += 4)
                if (n0 + c0 + j < a.Np)
                    *reinterpret_cast<float4*>(o + c0 + j) =
                        make_float4(__uint_as_float(u[j]), __uint_as_float(u[j + 1]), __uint_as_float(u[j + 2]),
                                    __uint_as_float(u[j + 3]));
        }
    } else if (tid == 0) {
        tc_raise(a.err);
    }
    cta_end<BN>(cta);
}

// dW32 [Cout][9][Cin] = sum over the slabs in a fixed order: thread (z, o) of a block
// adds the slabs z, z + 8, .. of output o, then the eight sums are added (a single chain
// over up to 592 slabs is bound by its load latency)
__global__ void __launch_bounds__(256) k_wgrad_sum(const float* __restrict__ work, int ns, int Cp, int Cin, int Np,
                                                   int Cout, float* __restrict__ dW) {
    __shared__ float red[8][32];
    const int o = threadIdx.x & 31, z0 = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + o;
    const int64_t slab = (int64_t)9 * Cp * Np;
    const bool in = i < Cout * 9 * Cin;
    const int co = i % Cout, k = i / Cout, t = k / Cin, c = k - t * Cin;  // consecutive threads: channels of a row
    float s = 0.f;
    if (in) {
        const float* w = work + (int64_t)(t * Cp + c) * Np + co;
#pragma unroll 8
        for (int z = z0; z < ns; z += 8) s += w[z * slab];
    }
    red[z0][o] = s;
    __syncthreads();
    if (z0 == 0 && in) {
        for (int z = 1; z < 8; ++z) s += red[z][o];
        dW[((int64_t)co * 9 + t) * Cin + c] = s;
    }
}

// BF16 copies of the master weights W32 [Cout][9][Cin]: Wf [Cout][9 Cp] of the forward
// pass and Wd [Cin][9 CoutP] of the data gradient, whose tap u reads the output pixel
// that saw this input through tap 8 - u (zero padded)
__global__ void k_wcast_conv(const float* __restrict__ W32, int Cout, int Cin, int Cp, int CoutP, bf16* __restrict__ Wf,
                             bf16* __restrict__ Wd) {
    const int nf = Cout * 9 * Cp, nd = Cin * 9 * CoutP;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nf + nd; i += gridDim.x * blockDim.x) {
        if (i < nf) {
            const int co = i / (9 * Cp), k = i - co * 9 * Cp, t = k / Cp, c = k - t * Cp;
            Wf[i] = __float2bfloat16_rn(c < Cin ? W32[((int64_t)co * 9 + t) * Cin + c] : 0.f);
        } else {
            const int j = i - nf, c = j / (9 * CoutP), k = j - c * 9 * CoutP, u = k / CoutP, co = k - u * CoutP;
            Wd[j] = __float2bfloat16_rn(co < Cout ? W32[((int64_t)co * 9 + 8 - u) * Cin + c] : 0.f);
        }
    }
}

// dYb [P][Cp] = BF16(dA relu'(A)) (zero padded) and the per-block column sums of dA
// relu'(A) in FP64: thread = (pixel lane, channel), so rows are read as they lie.
// part [gridDim.x][C].  (A column sum with one block per channel read one value of
// each row's sectors: 179 us at 262144 x 32.)
constexpr int kRT = 256;
__global__ void __launch_bounds__(kRT) k_relu_bias_bwd(const float* __restrict__ dA, const float* __restrict__ A,
                                                       int64_t P, int C, int relu, bf16* __restrict__ dYb, int Cp,
                                                       double* __restrict__ part) {
    __shared__ double red[kRT];
    const int cw = min(Cp - (int)blockIdx.y * kRT, kRT);  // channels of this block
    const int lanes = kRT / cw, l = threadIdx.x / cw, c = blockIdx.y * kRT + threadIdx.x % cw;
    double s = 0.0;
    if (l < lanes) {
        for (int64_t p = (int64_t)blockIdx.x * lanes + l; p < P; p += (int64_t)gridDim.x * lanes) {
            float v = 0.f;
            if (c < C) {
                v = dA[p * C + c];
                if (relu && !(A[p * C + c] > 0.f)) v = 0.f;
                s += v;
            }
            dYb[p * Cp + c] = __float2bfloat16_rn(v);
        }
    }
    red[threadIdx.x] = s;
    __syncthreads();
    if (l == 0 && c < C) {
        for (int k = 1; k < lanes; ++k) s += red[k * cw + threadIdx.x];
        part[(int64_t)blockIdx.x * C + c] = s;
    }
}

// db[c] = sum of part[0..nb)[c] in a fixed order: a block takes 32 channels, eight
// groups of threads every eighth row of partials
__global__ void __launch_bounds__(256) k_bias_final(const double* __restrict__ part, int nb, int C, float* __restrict__ db) {
    __shared__ double red[8][32];
    const int l = threadIdx.x & 31, g = threadIdx.x >> 5, c = blockIdx.x * 32 + l;
    double s = 0.0;
    if (c < C) {
#pragma unroll 8
        for (int b = g; b < nb; b += 8) s += part[(int64_t)b * C + c];
    }
    red[g][l] = s;
    __syncthreads();
    if (g == 0 && c < C) {
        for (int k = 1; k < 8; ++k) s += red[k][l];
        db[c] = (float)s;
    }
}

constexpr int kReluBlocks = 592;  // 4 per SM

}  // namespace

template <int BN> static void launch_conv(const ConvArgs& a, cudaStream_t st) {
    constexpr size_t smem = (size_t)kStages * (kBM + BN) * 128 + 1024;
    MAF_CUDA(cudaFuncSetAttribute(k_conv<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid((unsigned)ceil_div(a.P, kBM), (unsigned)ceil_div(std::max(a.N, a.outb ? a.ldb : 0), BN));
    k_conv<BN><<<grid, 128, smem, st>>>(a);
    MAF_LAUNCH_CHECK();
}

template <int BN> static void launch_wgrad(const WgradArgs& a, int splits, cudaStream_t st) {
    constexpr size_t smem = (size_t)kStages * kBK * 128 * (2 + (BN + 63) / 64) + 1024;
    MAF_CUDA(cudaFuncSetAttribute(k_conv_wgrad<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid((unsigned)ceil_div(9 * a.Cp, kBM), (unsigned)ceil_div(a.Np, BN), (unsigned)splits);
    k_conv_wgrad<BN><<<grid, 128, smem, st>>>(a);
    MAF_LAUNCH_CHECK();
}

}  // namespace mafb

using namespace mafb;

extern "C" {

int maf_nn_conv(const void* act, int B, int H, int W, int Cp, const void* w, int N, const float* bias, int relu,
                float* out, int ldo, void* outb, int ldb, void* st) {
    return capi_run([&] {
        if (!act || !w || !out || B < 1 || H < 1 || W < 1 || N < 1 || Cp < 8 || Cp % 8 || ldo < N ||
            (outb && (ldb < N || ldb % 8)))
            throw Error(1, "maf_nn_conv: bad argument (Cp and ldb are multiples of 8, ldo and ldb at least N)");
        if (((uintptr_t)act | (uintptr_t)w | (uintptr_t)out | (uintptr_t)outb) % 16)
            throw Error(1, "maf_nn_conv: 16-byte aligned buffers expected");
        ConvArgs a{static_cast<const __nv_bfloat16*>(act), static_cast<const __nv_bfloat16*>(w), bias, out,
                   static_cast<__nv_bfloat16*>(outb), H, W, Cp, N, ldo, ldb, relu, (int64_t)B * H * W,
                   tc_flag()};
        cudaStream_t s = static_cast<cudaStream_t>(st);
        // the widest tile that the channels fill, so that a pixel's taps are gathered once;
        // narrower when the tiles would leave SMs idle (a single film's deeper levels)
        const int64_t mt = ceil_div(a.P, kBM);
        const int n = std::max(N, outb ? ldb : 0);
        int bn = n <= 32 ? 32 : n <= 64 ? 64 : 128;
        while (bn > 32 && mt * ceil_div(n, bn) < sm_count()) bn /= 2;
        if (bn == 32) launch_conv<32>(a, s);
        else if (bn == 64) launch_conv<64>(a, s);
        else launch_conv<128>(a, s);
    });
}

int maf_nn_conv_wgrad(const void* act, int B, int H, int W, int Cp, int Cin, const void* dy, int Cout, int CoutP,
                      float* work, int max_splits, float* dW, void* st) {
    return capi_run([&] {
        if (!act || !dy || !work || !dW || B < 1 || H < 1 || W < 1 || Cp % 8 || Cin < 1 || Cin > Cp || CoutP % 8 ||
            Cout < 1 || Cout > CoutP || max_splits < 1)
            throw Error(1, "maf_nn_conv_wgrad: bad argument (Cp and CoutP are multiples of 8)");
        if (((uintptr_t)act | (uintptr_t)dy | (uintptr_t)work) % 16)
            throw Error(1, "maf_nn_conv_wgrad: 16-byte aligned buffers expected");
        cudaStream_t s = static_cast<cudaStream_t>(st);
        WgradArgs a{static_cast<const __nv_bfloat16*>(act), static_cast<const __nv_bfloat16*>(dy), work, H, W, Cp,
                    CoutP, (int64_t)B * H * W, 0, tc_flag()};
        const int bn = CoutP <= 32 ? 32 : CoutP <= 64 ? 64 : 128;
        // about four CTAs per SM, at least four K blocks each
        const int64_t tiles = ceil_div(9 * Cp, kBM) * ceil_div(CoutP, bn);
        int64_t splits = std::min<int64_t>({ceil_div((int64_t)sm_count() * 4, tiles), ceil_div(a.P, 4 * kBK), max_splits});
        a.chunk = ceil_div(ceil_div(a.P, splits), kBK) * kBK;
        splits = ceil_div(a.P, a.chunk);
        if (bn == 32) launch_wgrad<32>(a, (int)splits, s);
        else if (bn == 64) launch_wgrad<64>(a, (int)splits, s);
        else launch_wgrad<128>(a, (int)splits, s);
        k_wgrad_sum<<<(unsigned)ceil_div(Cout * 9 * Cin, 32), 256, 0, s>>>(work, (int)splits, Cp, Cin, CoutP, Cout, dW);
        MAF_LAUNCH_CHECK();
    });
}

int maf_nn_wcast_conv(const float* W32, int Cout, int Cin, int Cp, int CoutP, void* Wf, void* Wd, void* st) {
    return capi_run([&] {
        if (!W32 || !Wf || !Wd || Cp % 8 || CoutP % 8 || CoutP < Cout || Cp < Cin)
            throw Error(1, "maf_nn_wcast_conv: bad padding");
        const int n = Cout * 9 * Cp + Cin * 9 * CoutP;
        k_wcast_conv<<<(unsigned)ceil_div(n, 256), 256, 0, static_cast<cudaStream_t>(st)>>>(
            W32, Cout, Cin, Cp, CoutP, static_cast<__nv_bfloat16*>(Wf), static_cast<__nv_bfloat16*>(Wd));
        MAF_LAUNCH_CHECK();
    });
}

int maf_nn_relu_bias_bwd(const float* dA, const float* A, long long P, int C, int relu, void* dYb, int Cp, float* db,
                         double* part, void* st) {
    return capi_run([&] {
        if (!dA || !A || !dYb || !db || !part || P < 1 || C < 1 || Cp % 8 || Cp < C)
            throw Error(1, "maf_nn_relu_bias_bwd: bad argument");
        cudaStream_t s = static_cast<cudaStream_t>(st);
        const int lanes = std::max(1, kRT / std::min(Cp, kRT));
        const int nb = (int)std::min<int64_t>(ceil_div(P, lanes), kReluBlocks);
        k_relu_bias_bwd<<<dim3((unsigned)nb, (unsigned)ceil_div(Cp, kRT)), kRT, 0, s>>>(
            dA, A, P, C, relu, static_cast<__nv_bfloat16*>(dYb), Cp, part);
        MAF_LAUNCH_CHECK();
        k_bias_final<<<(unsigned)ceil_div(C, 32), 256, 0, s>>>(part, nb, C, db);
        MAF_LAUNCH_CHECK();
    });
}

int maf_nn_relu_bias_bwd_parts(int* n) {
    if (n) *n = kReluBlocks;
    return n ? 0 : 1;
}

}  // extern "C"
