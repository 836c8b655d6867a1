// Layer kernels of the warm-start U-net (magnumaf/unet.py) beside the convolutions of
// conv.cu: the BF16 input, 2x2 average pooling, nearest 2x upsampling with skip
// concatenation, their backward passes, the normalising head with its loss gradient, and
// Adam.  Activations are pixel-major (NHWC): pixel p = (b, y, x) is row p = (b H + y) W + x;
// a layer's channel count C is padded to Cp (a multiple of 8) in the BF16 tensors that feed a
// convolution, the padding is zero.  Every reduction runs in a fixed order, so training is
// deterministic.
#include <cuda_bf16.h>

#include <initializer_list>

#include "../../include/maf_b200.h"
#include "capi_internal.hpp"
#include "engine.hpp"
#include "tc_error.hpp"

using namespace mafb;

namespace {

using bf16 = __nv_bfloat16;
constexpr int kT = 256;

unsigned grid_for(int64_t n) { return (unsigned)std::min<int64_t>(ceil_div(n, kT), (int64_t)sm_count() * 32); }

#define GRID_STRIDE(i, n) for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

// x [B][C][H][W] (FP32, channels first) -> act [P][Cp] BF16 (zero padded) and
// the magnetisation channels 0..2 as m [P][3] FP32
__global__ void k_in(const float* __restrict__ x, int B, int C, int H, int W, int Cp, bf16* __restrict__ act,
                     float* __restrict__ m) {
    const int64_t HW = (int64_t)H * W, P = B * HW;
    GRID_STRIDE(i, P * Cp) {
        const int64_t p = i / Cp;
        const int c = (int)(i - p * Cp);
        const int64_t b = p / HW, r = p - b * HW;
        const float v = c < C ? x[(b * C + c) * HW + r] : 0.f;
        act[i] = __float2bfloat16_rn(v);
        if (c < 3) m[p * 3 + c] = v;
    }
}

// The level-changing kernels below take one image row per block step (32-bit index
// arithmetic) and V channels per thread: 8 (two 16-byte FP32 loads, one 16-byte BF16
// store) when every channel count is a multiple of 8, else 1.  With one channel per
// thread and 64-bit divisions the skip concatenation of 16 x 128 x 128 x 96 channels took
// 79 us, its memory traffic 15.
template <int V> __device__ __forceinline__ void ldv(const float* __restrict__ p, float* v) {
    if constexpr (V == 8) {
        const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
        v[0] = *p;
    }
}
template <int V> __device__ __forceinline__ void stv(float* p, const float* v) {
    if constexpr (V == 8) {
        reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
    } else {
        *p = v[0];
    }
}
template <int V> __device__ __forceinline__ void stb(bf16* p, const float* v) {
    if constexpr (V == 8) {
        __align__(16) bf16 h[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) h[k] = __float2bfloat16_rn(v[k]);
        *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(h);
    } else {
        *p = __float2bfloat16_rn(v[0]);
    }
}
unsigned row_blocks(int64_t rows) { return (unsigned)std::min<int64_t>(rows, (int64_t)sm_count() * 16); }
#define ROW_LOOP(row, rows) for (int row = blockIdx.x; row < (rows); row += gridDim.x)

// 2x2 average pooling of in [B][H][W][C] -> out [B][H/2][W/2][C] (FP32 and BF16 [.][Cp])
template <int V>
__global__ void __launch_bounds__(kT) k_pool(const float* __restrict__ in, int rows, int W, int C, float* __restrict__ out,
                                             bf16* __restrict__ outb, int Cp) {
    const int w = W / 2, cv = Cp / V;
    ROW_LOOP(row, rows) {  // output row (b, y): input rows 2 row and 2 row + 1
        const float* s0 = in + (int64_t)2 * row * W * C;
        for (int i = threadIdx.x; i < w * cv; i += kT) {
            const int x = i / cv, c = (i - x * cv) * V;
            float v[V];
#pragma unroll
            for (int k = 0; k < V; ++k) v[k] = 0.f;
            if (c < C) {
                const float* s = s0 + (int64_t)2 * x * C + c;
                float a[V], b[V], d[V], e[V];
                ldv<V>(s, a);
                ldv<V>(s + C, b);
                ldv<V>(s + (int64_t)W * C, d);
                ldv<V>(s + (int64_t)W * C + C, e);
#pragma unroll
                for (int k = 0; k < V; ++k) v[k] = 0.25f * ((a[k] + b[k]) + (d[k] + e[k]));
                stv<V>(out + ((int64_t)row * w + x) * C + c, v);
            }
            stb<V>(outb + ((int64_t)row * w + x) * Cp + c, v);
        }
    }
}

template <int V>
__global__ void __launch_bounds__(kT) k_pool_bwd(const float* __restrict__ dout, int rows, int H, int W, int C,
                                                 float* __restrict__ din, int accumulate) {
    const int cv = C / V;
    ROW_LOOP(row, rows) {
        const int b = row / H, y = row - b * H;
        const float* s = dout + ((int64_t)b * (H / 2) + y / 2) * (W / 2) * C;
        float* o = din + (int64_t)row * W * C;
        for (int i = threadIdx.x; i < W * cv; i += kT) {
            const int x = i / cv, c = (i - x * cv) * V;
            float v[V], d[V];
            ldv<V>(s + (int64_t)(x / 2) * C + c, v);
            if (accumulate) ldv<V>(o + (int64_t)x * C + c, d);
#pragma unroll
            for (int k = 0; k < V; ++k) v[k] = accumulate ? d[k] + 0.25f * v[k] : 0.25f * v[k];
            stv<V>(o + (int64_t)x * C + c, v);
        }
    }
}

// out[B][H][W][Cp] BF16 = up2(a [B][H/2][W/2][Ca]) | s [B][H][W][Cs], zero padded
template <int V>
__global__ void __launch_bounds__(kT) k_up_cat(const float* __restrict__ a, int Ca, const float* __restrict__ s, int Cs,
                                               int rows, int H, int W, bf16* __restrict__ out, int Cp) {
    const int cv = Cp / V;
    ROW_LOOP(row, rows) {
        const int b = row / H, y = row - b * H;
        const float* ar = a + ((int64_t)b * (H / 2) + y / 2) * (W / 2) * Ca;
        const float* sr = s + (int64_t)row * W * Cs;
        bf16* o = out + (int64_t)row * W * Cp;
        for (int i = threadIdx.x; i < W * cv; i += kT) {
            const int x = i / cv, c = (i - x * cv) * V;
            float v[V];
#pragma unroll
            for (int k = 0; k < V; ++k) v[k] = 0.f;
            if (c < Ca)
                ldv<V>(ar + (int64_t)(x / 2) * Ca + c, v);
            else if (c < Ca + Cs)
                ldv<V>(sr + (int64_t)x * Cs + (c - Ca), v);
            stb<V>(o + (int64_t)x * Cp + c, v);
        }
    }
}

// backward of k_up_cat: da [B][H/2][W/2][Ca] = sum of the four children; ds [B][H][W][Cs] = the skip part
template <int V>
__global__ void __launch_bounds__(kT) k_up_cat_bwd(const float* __restrict__ dcat, int Cp, int Ca, int Cs, int rows, int W,
                                                   float* __restrict__ da, float* __restrict__ ds) {
    const int w = W / 2, av = Ca / V, sv = Cs / V;
    ROW_LOOP(row, rows) {  // coarse row: fine rows 2 row and 2 row + 1
        const float* d0 = dcat + (int64_t)2 * row * W * Cp;
        for (int i = threadIdx.x; i < w * av; i += kT) {
            const int x = i / av, c = (i - x * av) * V;
            const float* d = d0 + (int64_t)2 * x * Cp + c;
            float v[V], e[V], f[V], g[V];
            ldv<V>(d, v);
            ldv<V>(d + Cp, e);
            ldv<V>(d + (int64_t)W * Cp, f);
            ldv<V>(d + (int64_t)W * Cp + Cp, g);
#pragma unroll
            for (int k = 0; k < V; ++k) v[k] = (v[k] + e[k]) + (f[k] + g[k]);
            stv<V>(da + ((int64_t)row * w + x) * Ca + c, v);
        }
        for (int i = threadIdx.x; i < 2 * W * sv; i += kT) {
            const int x = i / sv, c = (i - x * sv) * V;  // x over both fine rows
            float v[V];
            ldv<V>(d0 + (int64_t)x * Cp + Ca + c, v);
            stv<V>(ds + ((int64_t)2 * row * W + x) * Cs + c, v);
        }
    }
}

// head: v = m + d, y = v / |v|; per-pixel loss |y - t|^2 and dL/dd (L = mean over
// pixels of |y - t|^2; t may be null: inference).  Where a convolution's wait gave up, y is
// NaN: its tiles hold another call's values, and an inference returns before the host could ask.
__global__ void k_head(const float* __restrict__ m, const float* __restrict__ d, int ldd,
                       const float* __restrict__ tgt, int64_t P, float* __restrict__ y, float* __restrict__ gd,
                       float* __restrict__ cell_loss, const int* __restrict__ failed) {
    const float inv = 1.f / (float)P;
    const bool bad = *failed != 0;
    GRID_STRIDE(p, P) {
        float v[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c] = bad ? __int_as_float(0x7fc00000) : m[p * 3 + c] + d[p * ldd + c];
        const float n = sqrtf(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
        const float in_ = n > 0.f ? 1.f / n : 0.f;
        float yy[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            yy[c] = v[c] * in_;
            if (y) y[p * 3 + c] = yy[c];
        }
        if (!tgt) continue;
        float gy[3], l = 0.f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float e = yy[c] - tgt[p * 3 + c];
            l += e * e;
            gy[c] = 2.f * e * inv;
        }
        cell_loss[p] = l;
        const float dot = yy[0] * gy[0] + yy[1] * gy[1] + yy[2] * gy[2];
#pragma unroll
        for (int c = 0; c < 3; ++c) gd[p * 3 + c] = (gy[c] - yy[c] * dot) * in_;
    }
}

// one block of kMeanT threads, sixteen values in flight per thread (a block of 256 with one
// load in flight took longer than the head itself)
constexpr int kMeanT = 1024;
__global__ void __launch_bounds__(kMeanT) k_mean(const float* __restrict__ v, int64_t n, float* __restrict__ out) {
    __shared__ double red[kMeanT / 32];
    double s = 0.0;
    int64_t i = threadIdx.x;
    for (; i + 15 * kMeanT < n; i += 16 * kMeanT) {
        float x[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = v[i + k * kMeanT];
#pragma unroll
        for (int k = 0; k < 16; ++k) s += x[k];
    }
    for (; i < n; i += kMeanT) s += v[i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < kMeanT / 32; ++k) t += red[k];
        *out = (float)(t / (double)n);
    }
}

__global__ void k_adam_nn(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m1,
                          float* __restrict__ m2, int64_t n, float lr, float c1, float c2) {
    GRID_STRIDE(i, n) {
        const float gi = g[i];
        const float a = 0.9f * m1[i] + 0.1f * gi;
        const float b = 0.999f * m2[i] + 0.001f * gi * gi;
        m1[i] = a;
        m2[i] = b;
        w[i] -= lr * (a / c1) / (sqrtf(b / c2) + 1e-8f);
    }
}

template <typename F> int run(F&& f) { return capi_run(f); }
cudaStream_t S(void* s) { return static_cast<cudaStream_t>(s); }

}  // namespace

extern "C" {

int maf_nn_input(const float* x, int B, int C, int H, int W, int Cp, void* act_bf16, float* m, void* st) {
    return run([&] {
        if (Cp % 8 || Cp < C || C < 3) throw Error(1, "maf_nn_input: Cp must be a multiple of 8 >= C >= 3");
        const int64_t n = (int64_t)B * H * W * Cp;
        k_in<<<grid_for(n), kT, 0, S(st)>>>(x, B, C, H, W, Cp, static_cast<bf16*>(act_bf16), m);
        MAF_LAUNCH_CHECK();
    });
}

// channel counts and buffers that the 8-channel kernels can take
static bool by8(std::initializer_list<int> c, std::initializer_list<const void*> p) {
    for (int v : c)
        if (v % 8) return false;
    for (const void* q : p)
        if ((uintptr_t)q % 16) return false;
    return true;
}

int maf_nn_pool(const float* in, int B, int H, int W, int C, float* out, void* outb, int Cp, void* st) {
    return run([&] {
        if (H % 2 || W % 2) throw Error(1, "maf_nn_pool: even H and W expected");
        const int rows = B * (H / 2);
        if (by8({C, Cp}, {in, out, outb}))
            k_pool<8><<<row_blocks(rows), kT, 0, S(st)>>>(in, rows, W, C, out, static_cast<bf16*>(outb), Cp);
        else
            k_pool<1><<<row_blocks(rows), kT, 0, S(st)>>>(in, rows, W, C, out, static_cast<bf16*>(outb), Cp);
        MAF_LAUNCH_CHECK();
    });
}

int maf_nn_pool_bwd(const float* dout, int B, int H, int W, int C, float* din, int accumulate, void* st) {
    return run([&] {
        if (by8({C}, {dout, din}))
            k_pool_bwd<8><<<row_blocks(B * H), kT, 0, S(st)>>>(dout, B * H, H, W, C, din, accumulate);
        else
            k_pool_bwd<1><<<row_blocks(B * H), kT, 0, S(st)>>>(dout, B * H, H, W, C, din, accumulate);
        MAF_LAUNCH_CHECK();
    });
}

int maf_nn_up_cat(const float* a, int Ca, const float* s, int Cs, int B, int H, int W, void* out, int Cp, void* st) {
    return run([&] {
        if (by8({Ca, Cs, Cp}, {a, s, out}))
            k_up_cat<8><<<row_blocks(B * H), kT, 0, S(st)>>>(a, Ca, s, Cs, B * H, H, W, static_cast<bf16*>(out), Cp);
        else
            k_up_cat<1><<<row_blocks(B * H), kT, 0, S(st)>>>(a, Ca, s, Cs, B * H, H, W, static_cast<bf16*>(out), Cp);
        MAF_LAUNCH_CHECK();
    });
}

int maf_nn_up_cat_bwd_set(const float* dcat, int Cp, int Ca, int Cs, int B, int H, int W, float* da, float* ds,
                          void* st) {
    return run([&] {
        const int rows = B * (H / 2);
        if (by8({Cp, Ca, Cs}, {dcat, da, ds}))
            k_up_cat_bwd<8><<<row_blocks(rows), kT, 0, S(st)>>>(dcat, Cp, Ca, Cs, rows, W, da, ds);
        else
            k_up_cat_bwd<1><<<row_blocks(rows), kT, 0, S(st)>>>(dcat, Cp, Ca, Cs, rows, W, da, ds);
        MAF_LAUNCH_CHECK();
    });
}

int maf_nn_head(const float* m, const float* d, int ldd, const float* tgt, long long P, float* y, float* gd,
                float* cell_loss, float* loss, void* st) {
    return run([&] {
        k_head<<<grid_for(P), kT, 0, S(st)>>>(m, d, ldd, tgt, P, y, gd, cell_loss, &tc_flag()->up);
        MAF_LAUNCH_CHECK();
        if (tgt && loss) {
            k_mean<<<1, kMeanT, 0, S(st)>>>(cell_loss, P, loss);
            MAF_LAUNCH_CHECK();
        }
    });
}

int maf_nn_adam(float* w, const float* g, float* m1, float* m2, long long n, float lr, int step, void* st) {
    return run([&] {
        const float c1 = 1.f - powf(0.9f, (float)step), c2 = 1.f - powf(0.999f, (float)step);
        k_adam_nn<<<grid_for(n), kT, 0, S(st)>>>(w, g, m1, m2, n, lr, c1, c2);
        MAF_LAUNCH_CHECK();
    });
}

}  // extern "C"
