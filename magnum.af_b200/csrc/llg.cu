// Runge-Kutta stage combine, error norm / candidate update, normalisation and
// small reductions for the adaptive LLG integrator.
//
// Reference: magnumaf/src/integrators/adaptive_runge_kutta.cpp:39-173,496-529
//   stage s:     m_s = m + sum_j a_sj k_j                    (FP64)
//   error norm:  err = max | rk_error / (atol + rtol |max(m, m + sumbk)|) |
//   accept:      m <- normalise(m + sumbk)   (normalize_even_zero_vectors, or
//                the zero-safe normalize when an Ms_field exists)
// magnumaf/src/math.cpp:6-8 (max_4d_abs), magnumaf/src/util/util.cpp:34-42.
#include "engine.hpp"
#include "rk.hpp"
#include "rng.cuh"

namespace mafb {

__global__ void k_combine(const double* __restrict__ m, KList kl, double* __restrict__ out64, float* __restrict__ out32,
                          int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double acc = m[i];
        for (int j = 0; j < kl.n; ++j) acc = acc + kl.c[j] * kl.k[j][i];
        out64[i] = acc;
        if (out32) out32[i] = (float)acc;
    }
}

// The same combine with the number of k's a compile-time constant and two
// values per thread through 16-byte loads: each thread issues its NK + 1
// independent loads before the first use (the generic loop above issues them
// one trip at a time).  Same arithmetic and summation order, so bit-identical.
// Needs n even and 16-byte aligned buffers.
template <int NK>
__global__ void __launch_bounds__(256) k_combine_v(const double* __restrict__ m, KList kl, double* __restrict__ out64,
                                                   float* __restrict__ out32, int64_t n2) {
    pdl_begin();
    const double2* m2 = reinterpret_cast<const double2*>(m);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += (int64_t)gridDim.x * blockDim.x) {
        double2 kv[NK];
#pragma unroll
        for (int j = 0; j < NK; ++j) kv[j] = reinterpret_cast<const double2*>(kl.k[j])[i];
        double2 acc = m2[i];
#pragma unroll
        for (int j = 0; j < NK; ++j) {
            acc.x = acc.x + kl.c[j] * kv[j].x;
            acc.y = acc.y + kl.c[j] * kv[j].y;
        }
        reinterpret_cast<double2*>(out64)[i] = acc;
        if (out32) reinterpret_cast<float2*>(out32)[i] = make_float2((float)acc.x, (float)acc.y);
    }
}

static bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

void rk_combine(const double* m, const KList& kl, double* out64, float* out32, int64_t n, cudaStream_t st) {
    bool vec = n % 2 == 0 && kl.n >= 1 && kl.n <= 7 && aligned16(m) && aligned16(out64) &&
               (!out32 || ((uintptr_t)out32 & 7) == 0);
    for (int j = 0; j < kl.n; ++j) vec = vec && aligned16(kl.k[j]);
    if (vec) {
        const int64_t n2 = n / 2;
        const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(n2, 256), (int64_t)sm_count() * 16);
        switch (kl.n) {
            case 1: launch_chain(k_combine_v<1>, dim3(blocks), 256, 0, st, m, kl, out64, out32, n2); break;
            case 2: launch_chain(k_combine_v<2>, dim3(blocks), 256, 0, st, m, kl, out64, out32, n2); break;
            case 3: launch_chain(k_combine_v<3>, dim3(blocks), 256, 0, st, m, kl, out64, out32, n2); break;
            case 4: launch_chain(k_combine_v<4>, dim3(blocks), 256, 0, st, m, kl, out64, out32, n2); break;
            case 5: launch_chain(k_combine_v<5>, dim3(blocks), 256, 0, st, m, kl, out64, out32, n2); break;
            case 6: launch_chain(k_combine_v<6>, dim3(blocks), 256, 0, st, m, kl, out64, out32, n2); break;
            default: launch_chain(k_combine_v<7>, dim3(blocks), 256, 0, st, m, kl, out64, out32, n2); break;
        }
        MAF_LAUNCH_CHECK();
        return;
    }
    const int64_t blocks = std::min<int64_t>(ceil_div(n, 256), (int64_t)sm_count() * 16);
    k_combine<<<(unsigned)blocks, 256, 0, st>>>(m, kl, out64, out32, n);
    MAF_LAUNCH_CHECK();
}

// max with NaN propagation (NaN wins)
__device__ __forceinline__ double nanmax(double a, double b) {
    if (a != a) return a;
    if (b != b) return b;
    return a > b ? a : b;
}

// The block's maximum to partials[block]; the block that arrives last writes the maximum
// over all blocks to *err (a kernel of its own for it was one more dependent launch per
// step).  *counter is zero before and after the launch.
__device__ __forceinline__ void block_max_final(double v, double* partials, unsigned* counter, double* err) {
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) v = nanmax(v, __shfl_down_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) red[wid] = v;
    __syncthreads();
    __shared__ bool last;
    const int nw = (blockDim.x + 31) >> 5;
    if (threadIdx.x == 0) {
        double s = red[0];
        for (int k = 1; k < nw; ++k) s = nanmax(s, red[k]);
        partials[blockIdx.x] = s;
        __threadfence();
        last = atomicInc(counter, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    v = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) v = nanmax(v, __ldcg(partials + b));
    for (int o = 16; o > 0; o >>= 1) v = nanmax(v, __shfl_down_sync(0xffffffffu, v, o));
    if (lane == 0) red[wid] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = red[0];
        for (int k = 1; k < nw; ++k) s = nanmax(s, red[k]);
        *err = s;
    }
}

// sumbk = sum bs_j k_j ; rk_error = (form 0) sum e_j k_j  or (form 1) sumbk - sum e_j k_j
__global__ void k_finalize(const double* __restrict__ m, KList kb, KList ke, int form, double atol, double rtol,
                           double* __restrict__ mcand, int norm_mode, int64_t N, double* partials, unsigned* counter, double* errout) {
    double vmax = 0.0;
    for (int64_t cell = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; cell < N;
         cell += (int64_t)gridDim.x * blockDim.x) {
        double out[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int64_t i = c * N + cell;
            double sumbk = kb.c[0] * kb.k[0][i];
            for (int j = 1; j < kb.n; ++j) sumbk = sumbk + kb.c[j] * kb.k[j][i];
            double e = ke.c[0] * ke.k[0][i];
            for (int j = 1; j < ke.n; ++j) e = e + ke.c[j] * ke.k[j][i];
            const double err = form == 0 ? e : sumbk - e;
            const double mi = m[i];
            const double mn = mi + sumbk;
            const double mx = mi > mn ? mi : mn;  // af::max(m, m + sumbk)
            const double sc = atol + rtol * fabs(mx);
            vmax = nanmax(vmax, fabs(err / sc));
            out[c] = mn;
        }
        if (norm_mode == 1) {
            const double nrm = sqrt(out[0] * out[0] + out[1] * out[1] + out[2] * out[2]);
            out[0] /= nrm; out[1] /= nrm; out[2] /= nrm;
        } else if (norm_mode == 2) {
            const double nrm = sqrt(out[0] * out[0] + out[1] * out[1] + out[2] * out[2]);
            if (nrm != 0) { out[0] /= nrm; out[1] /= nrm; out[2] /= nrm; }
            else { out[0] = 0; out[1] = 0; out[2] = 0; }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) mcand[c * N + cell] = out[c];
    }
    block_max_final(vmax, partials, counter, errout);
}

// The union of the b- and e-lists' k buffers, each loaded once: k[j] enters
// sumbk with cb[j] and the error sum with ce[j] (a zero coefficient: not in
// that list).  The lists' own orders are kept (checked by the caller), so the
// sums are formed in the same order as in k_finalize.
struct KUnion {
    const double* k[8] = {};
    double cb[8] = {};
    double ce[8] = {};
    int n = 0;
};

// vmax <- max(vmax, |err / sc|), NaN-propagating.  The FP64 division is skipped where the
// quotient is certainly below vmax or a zero (the finalize kernels are bound on FP64 division
// and square root as much as on HBM).  The comparisons are strict, so that 0 / 0 (atol = 0, a
// cell without m) and inf / inf are divided and give NaN, as a NaN does, which fails both.
__device__ __forceinline__ void err_max(double err, double sc, double& vmax) {
    if (!(fabs(err) < vmax * sc * (1.0 - 1e-12) || (err == 0.0 && sc > 0.0))) vmax = nanmax(vmax, fabs(err / sc));
}

__device__ __forceinline__ double fin_one(double sumbk, double e, int form, double mi, double atol, double rtol,
                                          double& vmax) {
    const double err = form == 0 ? e : sumbk - e;
    const double mn = mi + sumbk;
    const double mx = mi > mn ? mi : mn;  // af::max(m, m + sumbk)
    const double sc = atol + rtol * fabs(mx);
    err_max(err, sc, vmax);
    return mn;
}

__device__ __forceinline__ void fin_norm(double* o, int norm_mode) {
    if (norm_mode == 1) {
        const double nrm = sqrt(o[0] * o[0] + o[1] * o[1] + o[2] * o[2]);
        o[0] /= nrm; o[1] /= nrm; o[2] /= nrm;
    } else if (norm_mode == 2) {
        const double nrm = sqrt(o[0] * o[0] + o[1] * o[1] + o[2] * o[2]);
        if (nrm != 0) { o[0] /= nrm; o[1] /= nrm; o[2] /= nrm; }
        else { o[0] = 0; o[1] = 0; o[2] = 0; }
    }
}

// k_finalize with NU union buffers known at compile time and two cells per
// thread through 16-byte loads (N even, 16-byte aligned buffers); same
// arithmetic as k_finalize, bit-identical results.
template <int NU>
__global__ void __launch_bounds__(256, 4) k_finalize_v(const double* __restrict__ m, KUnion ku, int form, double atol,
                                                    double rtol, double* __restrict__ mcand, int norm_mode, int64_t N,
                                                    double* partials, unsigned* counter, double* errout) {
    pdl_begin();
    const int64_t N2 = N / 2;
    double vmax = 0.0;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < N2; p += (int64_t)gridDim.x * blockDim.x) {
        double o0[3], o1[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int64_t i = c * N2 + p;
            double2 kv[NU];
#pragma unroll
            for (int j = 0; j < NU; ++j) kv[j] = reinterpret_cast<const double2*>(ku.k[j])[i];
            const double2 mi = reinterpret_cast<const double2*>(m)[i];
            double b0 = 0.0, b1 = 0.0, e0 = 0.0, e1 = 0.0;
#pragma unroll
            for (int j = 0; j < NU; ++j) {
                if (ku.cb[j] != 0.0) {
                    b0 = b0 + ku.cb[j] * kv[j].x;
                    b1 = b1 + ku.cb[j] * kv[j].y;
                }
                if (ku.ce[j] != 0.0) {
                    e0 = e0 + ku.ce[j] * kv[j].x;
                    e1 = e1 + ku.ce[j] * kv[j].y;
                }
            }
            o0[c] = fin_one(b0, e0, form, mi.x, atol, rtol, vmax);
            o1[c] = fin_one(b1, e1, form, mi.y, atol, rtol, vmax);
        }
        fin_norm(o0, norm_mode);
        fin_norm(o1, norm_mode);
#pragma unroll
        for (int c = 0; c < 3; ++c) reinterpret_cast<double2*>(mcand)[c * N2 + p] = make_double2(o0[c], o1[c]);
    }
    block_max_final(vmax, partials, counter, errout);
}

// Union of the two lists with each list's order preserved, or false.
static bool make_union(const KList& kb, const KList& ke, KUnion& u) {
    for (int j = 0; j < kb.n; ++j) {
        if (kb.c[j] == 0.0) return false;
        u.k[u.n] = kb.k[j];
        u.cb[u.n] = kb.c[j];
        ++u.n;
    }
    int last = -1;
    for (int j = 0; j < ke.n; ++j) {
        if (ke.c[j] == 0.0) continue;  // adds nothing to the error sum
        int at = -1;
        for (int q = 0; q < u.n; ++q)
            if (u.k[q] == ke.k[j]) at = q;
        if (at < 0) {
            if (u.n == 8) return false;
            at = u.n++;
            u.k[at] = ke.k[j];
        }
        if (at <= last) return false;  // the e-list's order would change
        u.ce[at] = ke.c[j];
        last = at;
    }
    return u.n >= 1 && u.n <= 7;
}

int rk_finalize_blocks() { return 32 * sm_count(); }

void rk_finalize(const double* m, const KList& kb, const KList& ke, int form, double atol, double rtol, double* mcand,
                 int norm_mode, int64_t N, double* partials, double* err, cudaStream_t st) {
    const int threads = 256;
    KUnion u;
    bool vec = N % 2 == 0 && aligned16(m) && aligned16(mcand) && make_union(kb, ke, u);
    for (int j = 0; vec && j < u.n; ++j) vec = aligned16(u.k[j]);
    const int blocks = (int)std::min<int64_t>(ceil_div(vec ? N / 2 : N, threads), rk_finalize_blocks());
    unsigned* counter = reinterpret_cast<unsigned*>(partials + rk_finalize_blocks());
    if (vec) {
#define MAF_FIN(NU)                                                                                                 \
    launch_chain(k_finalize_v<NU>, dim3(blocks), threads, 0, st, m, u, form, atol, rtol, mcand, norm_mode, N, \
                 partials, counter, err)
        switch (u.n) {
            case 1: MAF_FIN(1); break;
            case 2: MAF_FIN(2); break;
            case 3: MAF_FIN(3); break;
            case 4: MAF_FIN(4); break;
            case 5: MAF_FIN(5); break;
            case 6: MAF_FIN(6); break;
            default: MAF_FIN(7); break;
        }
#undef MAF_FIN
    } else {
        k_finalize<<<blocks, threads, 0, st>>>(m, kb, ke, form, atol, rtol, mcand, norm_mode, N, partials,
                                               counter, err);
    }
    MAF_LAUNCH_CHECK();
}

// normalize_handle_zero_vectors (util.cpp:37-42); counts cells of zero norm
__global__ void k_normalize(double* __restrict__ m, int64_t N, int mode, unsigned long long* zero_count) {
    unsigned long long z = 0;
    for (int64_t cell = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; cell < N;
         cell += (int64_t)gridDim.x * blockDim.x) {
        double a = m[cell], b = m[N + cell], c = m[2 * N + cell];
        const double nrm = sqrt(a * a + b * b + c * c);
        if (mode == 1) {
            a /= nrm; b /= nrm; c /= nrm;
        } else if (nrm != 0) {
            a /= nrm; b /= nrm; c /= nrm;
        } else {
            a = 0; b = 0; c = 0;
            ++z;
        }
        m[cell] = a;
        m[N + cell] = b;
        m[2 * N + cell] = c;
    }
    if (zero_count && z) atomicAdd(zero_count, z);
}

void normalize_m(double* m, int64_t N, int mode, unsigned long long* zero_count_dev, cudaStream_t st) {
    const int64_t blocks = std::min<int64_t>(ceil_div(N, 256), (int64_t)sm_count() * 8);
    k_normalize<<<(unsigned)blocks, 256, 0, st>>>(m, N, mode, zero_count_dev);
    MAF_LAUNCH_CHECK();
}

// Ms_field = Ms * (|m| != 0)   (state.cpp:71-89)
__global__ void k_ms_from_m(const double* __restrict__ m, double Ms, double* __restrict__ msf, float* __restrict__ msf32,
                            int64_t N) {
    for (int64_t cell = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; cell < N;
         cell += (int64_t)gridDim.x * blockDim.x) {
        const double a = m[cell], b = m[N + cell], c = m[2 * N + cell];
        const double v = (sqrt(a * a + b * b + c * c) != 0) ? Ms : 0.0;
        msf[cell] = v;
        if (msf32) msf32[cell] = (float)v;
    }
}

void ms_field_from_m(const double* m, double Ms, double* msf, float* msf32, int64_t N, cudaStream_t st) {
    const int64_t blocks = std::min<int64_t>(ceil_div(N, 256), (int64_t)sm_count() * 8);
    k_ms_from_m<<<(unsigned)blocks, 256, 0, st>>>(m, Ms, msf, msf32, N);
    MAF_LAUNCH_CHECK();
}

// <m>: per-block sums of the three components and of the nonzero-cell count,
// then a fixed-order final pass (state.cpp:32-43).
__global__ void k_mean_partials(const double* __restrict__ m, int64_t N, double* __restrict__ part) {
    double s0 = 0, s1 = 0, s2 = 0, cnt = 0;
    for (int64_t cell = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; cell < N;
         cell += (int64_t)gridDim.x * blockDim.x) {
        const double a = m[cell], b = m[N + cell], c = m[2 * N + cell];
        s0 += a;
        s1 += b;
        s2 += c;
        cnt += (sqrt(a * a + b * b + c * c) != 0) ? 1.0 : 0.0;
    }
    __shared__ double red[4][32];
    double v[4] = {s0, s1, s2, cnt};
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
        if (lane == 0) red[q][wid] = v[q];
    }
    __syncthreads();
    if (wid == 0) {
        const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            double s = lane < nw ? red[q][lane] : 0.0;
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (lane == 0) part[4 * blockIdx.x + q] = s;
        }
    }
}

// one warp per sum (the three components and the cell count)
__global__ void k_mean_final(const double* __restrict__ part, int nb, double* __restrict__ out) {
    __shared__ double tot[4];
    const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
    double s = 0;
    for (int b = lane; b < nb; b += 32) s += part[4 * b + q];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) tot[q] = s;
    __syncthreads();
    if (threadIdx.x < 3) out[threadIdx.x] = tot[threadIdx.x] / tot[3];
}

int mean_m_blocks() { return 2 * sm_count(); }

void mean_m(const double* m, int64_t N, double* scratch, double* out_dev, cudaStream_t st) {
    const int blocks = (int)std::min<int64_t>(ceil_div(N, 256), mean_m_blocks());
    k_mean_partials<<<blocks, 256, 0, st>>>(m, N, scratch);
    MAF_LAUNCH_CHECK();
    k_mean_final<<<1, 128, 0, st>>>(scratch, blocks, out_dev);
    MAF_LAUNCH_CHECK();
}

// (a - b) -> d, with sum of squares partials (for the string method's Frobenius norm)
__global__ void k_f2d(const float* __restrict__ a, double* __restrict__ b, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = (double)a[i];
}

void f32_to_f64(const float* a, double* b, int64_t n, cudaStream_t st) {
    const int64_t blocks = std::min<int64_t>(ceil_div(n, 256), (int64_t)sm_count() * 16);
    k_f2d<<<(unsigned)blocks, 256, 0, st>>>(a, b, n);
    MAF_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// vector operations of the LBFGS minimiser (lbfgs_minimizer.cpp:44-46, 96-177)
// ---------------------------------------------------------------------------
// reduction blocks of the LBFGS vector operations (partials at scratch[0, n),
// the result at scratch[n])
int red_blocks() { return 2 * sm_count(); }

// per-block partials: mode 0 sum a*b, mode 1 max |a| (NaN-propagating),
// mode 2 sum (a-b)^2 (the string method's Frobenius norm of image differences)
__global__ void k_red_partials(const double* __restrict__ a, const double* __restrict__ b, int64_t n, int mode,
                               double* __restrict__ part) {
    double v = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (mode == 0) {
            v += a[i] * b[i];
        } else if (mode == 2) {
            const double d = a[i] - b[i];
            v += d * d;
        } else {
            v = nanmax(v, fabs(a[i]));
        }
    }
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) {
        const double w = __shfl_down_sync(0xffffffffu, v, o);
        v = mode != 1 ? v + w : nanmax(v, w);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) red[wid] = v;
    __syncthreads();
    if (wid == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        double s = lane < nw ? red[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            const double w = __shfl_down_sync(0xffffffffu, s, o);
            s = mode != 1 ? s + w : nanmax(s, w);
        }
        if (lane == 0) part[blockIdx.x] = s;
    }
}

// one block, 256 threads: the partials in a fixed tree (one thread adding the 192-296
// partials in a chain took 10.9 us, longer than the reduction itself)
__global__ void k_red_final(const double* __restrict__ part, int nb, int mode, double* __restrict__ out) {
    __shared__ double red[8];
    double v = 0.0;
    for (int i = threadIdx.x; i < nb; i += 256) v = mode != 1 ? v + part[i] : nanmax(v, part[i]);
    for (int o = 16; o > 0; o >>= 1) {
        const double w = __shfl_down_sync(0xffffffffu, v, o);
        v = mode != 1 ? v + w : nanmax(v, w);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = red[0];
        for (int i = 1; i < 8; ++i) s = mode != 1 ? s + red[i] : nanmax(s, red[i]);
        *out = s;
    }
}

double reduce_host(const double* a, const double* b, int64_t n, int mode, double* scratch, cudaStream_t st) {
    const int nred = red_blocks();
    const int blocks = (int)std::min<int64_t>(ceil_div(n, 256), nred);
    k_red_partials<<<blocks, 256, 0, st>>>(a, b, n, mode, scratch);
    MAF_LAUNCH_CHECK();
    k_red_final<<<1, 256, 0, st>>>(scratch, blocks, mode, scratch + nred);
    MAF_LAUNCH_CHECK();
    double v = 0;
    MAF_CUDA(cudaMemcpyAsync(&v, scratch + nred, sizeof(double), cudaMemcpyDeviceToHost, st));
    MAF_CUDA(cudaStreamSynchronize(st));
    return v;
}

double dot_host(const double* a, const double* b, int64_t n, double* scratch, cudaStream_t st) {
    return reduce_host(a, b, n, 0, scratch, st);
}

double maxabs_host(const double* a, int64_t n, double* scratch, cudaStream_t st) {
    return reduce_host(a, nullptr, n, 1, scratch, st);
}

double sqdiff_host(const double* a, const double* b, int64_t n, double* scratch, cudaStream_t st) {
    return reduce_host(a, b, n, 2, scratch, st);
}

// out = a + (c1 * (b - a)) / c2, the string method's linear re-interpolation
// in the reference's order of operations (string_method.cpp:94-95)
__global__ void k_lerp(double* __restrict__ out, const double* __restrict__ a, const double* __restrict__ b, double c1,
                       double c2, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = a[i] + (c1 * (b[i] - a[i])) / c2;
}

void lerp(double* out, const double* a, const double* b, double c1, double c2, int64_t n, cudaStream_t st) {
    const int64_t blocks = std::min<int64_t>(ceil_div(n, 256), (int64_t)sm_count() * 16);
    k_lerp<<<(unsigned)blocks, 256, 0, st>>>(out, a, b, c1, c2, n);
    MAF_LAUNCH_CHECK();
}

__global__ void k_inc_counter(unsigned long long* c) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *c += 1;
}

void inc_counter(unsigned long long* c, cudaStream_t st) {
    k_inc_counter<<<1, 32, 0, st>>>(c);
    MAF_LAUNCH_CHECK();
}

__global__ void k_axpby(double* out, double a, const double* x, double b, const double* y, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double v = a * x[i];
        out[i] = y ? v + b * y[i] : v;
    }
}

void axpby(double* out, double a, const double* x, double b, const double* y, int64_t n, cudaStream_t st) {
    const int64_t blocks = std::min<int64_t>(ceil_div(n, 256), (int64_t)sm_count() * 16);
    k_axpby<<<(unsigned)blocks, 256, 0, st>>>(out, a, x, b, y, n);
    MAF_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// LBFGS iteration kernels: an update and the reductions that follow it in one
// launch.  A film of 128x128 cells is 0.4 MB per vector, so an iteration is bound
// by the number of dependent launches (2.5-3.5 us each), not by bandwidth: with an
// update, a partial and a final kernel per dot product an iteration of 20 took
// 72 launches, 0.47 ms; with the last block of the update's grid forming the
// reduction's result it takes about 18.
// ---------------------------------------------------------------------------
constexpr int kLbThreads = 256;

// Block sums (or, bit r of maxmask, NaN-propagating maxima) of v[0..NR) to
// part[r * gridDim.x + block]; the block that arrives last combines every block's
// partials in a fixed tree, whatever the arrival order, and writes out[0..NR).
// *counter is zero before and after the launch.  Returns whether this is that block.
template <int NR>
__device__ __forceinline__ bool reduce_last_block(double (&v)[NR], unsigned maxmask, double* part, unsigned* counter,
                                                  double* out) {
    __shared__ double red[NR][kLbThreads / 32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    auto block_combine = [&](double (&x)[NR]) {  // the result in thread r < NR, x[0]
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            for (int o = 16; o > 0; o >>= 1) {
                const double w = __shfl_down_sync(0xffffffffu, x[r], o);
                x[r] = (maxmask >> r) & 1u ? nanmax(x[r], w) : x[r] + w;
            }
            if (lane == 0) red[r][wid] = x[r];
        }
        __syncthreads();
        if (threadIdx.x < NR) {
            const int r = threadIdx.x;
            double s = red[r][0];
            for (int k = 1; k < kLbThreads / 32; ++k) s = (maxmask >> r) & 1u ? nanmax(s, red[r][k]) : s + red[r][k];
            x[0] = s;
        }
    };
    block_combine(v);
    if (threadIdx.x < NR) {
        part[threadIdx.x * gridDim.x + blockIdx.x] = v[0];
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(counter, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double t[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        t[r] = 0.0;
        for (unsigned b = threadIdx.x; b < gridDim.x; b += kLbThreads) {
            const double w = __ldcg(part + r * gridDim.x + b);
            t[r] = (maxmask >> r) & 1u ? nanmax(t[r], w) : t[r] + w;
        }
    }
    block_combine(t);
    if (threadIdx.x < NR) out[threadIdx.x] = t[0];
    return true;
}

// One step of the two-loop recursion (lbfgs_minimizer.cpp:96-130):
//   q <- scale (q_in + b u),  b = -rho *d (first loop) or *alpha_in - rho *d (second),
// *alpha_out = rho *d, dir <- -q, and *d <- w . q for the next step.  u, alpha_*, dir
// and the copies (x_copy <- x, g_copy <- q_in) are optional.  The product order is
// that of separate kernels; *d is read by every thread before its block arrives, and
// written by the last block only.
__global__ void __launch_bounds__(kLbThreads) k_lb_recur(LbRecur a, int64_t n, double* part, unsigned* counter) {
    double b = 0.0;
    if (a.u) {
        const double t = a.rho * *a.d;
        b = a.alpha_in ? *a.alpha_in - t : -t;
        if (a.alpha_out && blockIdx.x == 0 && threadIdx.x == 0) *a.alpha_out = t;
    }
    double v[1] = {0.0};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double q = a.q_in[i];
        if (a.g_copy) a.g_copy[i] = q;
        if (a.x_copy) a.x_copy[i] = a.x[i];
        if (a.u) q = q + b * a.u[i];
        if (a.scaled) q = a.scale * q;
        a.q[i] = q;
        if (a.dir) a.dir[i] = -q;
        v[0] += a.w[i] * q;
    }
    reduce_last_block<1>(v, 0u, part, counter, a.d);
}

void lb_recur(const LbRecur& a, int64_t n, double* part, unsigned* counter, cudaStream_t st) {
    const int blocks = (int)std::min<int64_t>(ceil_div(n, kLbThreads), red_blocks());
    k_lb_recur<<<blocks, kLbThreads, 0, st>>>(a, n, part, counter);
    MAF_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// The whole two-loop recursion in one launch for films of up to 256x256 cells: one
// cluster of CTAs keeps q in registers, every dot product is a block sum and one
// hardware cluster barrier, after which each CTA adds the blocks' sums through
// distributed shared memory in rank order.  A step costs about a barrier and one pass
// over two vectors in L2 instead of a dependent launch with a last-block reduction
// (6.6 us at 128x128 cells).
// ---------------------------------------------------------------------------
constexpr int kLoopThreads = 1024;
constexpr int kLoopElems = 12;  // q values per thread at most (24 of the 64 registers)

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// sum over the cluster of v, to every thread; slot: the shared double of this step (two
// in turn: the barrier of the next step separates its readers from its next writer)
__device__ __forceinline__ double cluster_sum(double v, double* slot, double* red, double* total, int nctas) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[wid] = v;
    __syncthreads();
    if (wid == 0) {
        double s = red[lane];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) *slot = s;
    }
    cluster_barrier();
    if (wid == 0) {
        double s = 0.0;
        if (lane < nctas) {
            unsigned addr = (unsigned)__cvta_generic_to_shared(slot), remote;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(lane));
            asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(s) : "r"(remote) : "memory");
        }
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) *total = s;
    }
    __syncthreads();
    return *total;
}

template <int E> __global__ void __launch_bounds__(kLoopThreads) k_lb_loop(LbLoop a, int64_t n) {
    __shared__ double red[32], slot[2], total;
    const int nctas = gridDim.x;
    const int64_t i0 = (int64_t)blockIdx.x * kLoopThreads + threadIdx.x, step = (int64_t)nctas * kLoopThreads;
    double q[E], alpha[5], d = 0.0;
    auto dot = [&](const double* w, int turn) {
        double v = 0.0;
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (i0 + e * step < n) v += w[i0 + e * step] * q[e];
        return cluster_sum(v, slot + (turn & 1), red, &total, nctas);
    };
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int64_t i = i0 + e * step;
        q[e] = 0.0;
        if (i < n) {
            q[e] = a.grad[i];
            a.g_copy[i] = q[e];
            a.x_copy[i] = a.x[i];
        }
    }
    int turn = 0;
#pragma unroll
    for (int j = 4; j >= 0; --j) {
        if (j >= a.k) continue;
        d = dot(a.s[j], turn++);
        alpha[j] = a.rho[j] * d;
        const double b = -alpha[j];
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (i0 + e * step < n) q[e] = q[e] + b * a.y[j][i0 + e * step];
    }
#pragma unroll
    for (int e = 0; e < E; ++e) q[e] = a.scale * q[e];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        if (j >= a.k) continue;
        d = dot(a.y[j], turn++);
        const double b = alpha[j] - a.rho[j] * d;
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (i0 + e * step < n) q[e] = q[e] + b * a.s[j][i0 + e * step];
    }
    d = dot(a.grad, turn++);
#pragma unroll
    for (int e = 0; e < E; ++e)
        if (i0 + e * step < n) a.dir[i0 + e * step] = -q[e];
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.d = d;
    cluster_barrier();  // no CTA leaves while another reads its sums
}

// CTAs of the recursion's cluster on this device: 16 where such clusters can be resident, else 8
static int loop_cluster_size() {
    constexpr int kMaxOrdinals = 64;
    static int cache[kMaxOrdinals] = {};
    int dev = 0;
    MAF_CUDA(cudaGetDevice(&dev));
    int v = dev < kMaxOrdinals ? __atomic_load_n(&cache[dev], __ATOMIC_RELAXED) : 0;
    if (v) return v;
    MAF_CUDA(cudaFuncSetAttribute(k_lb_loop<kLoopElems>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 16;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(kLoopThreads);
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int nc = 0;
    v = cudaOccupancyMaxActiveClusters(&nc, k_lb_loop<kLoopElems>, &cfg) == cudaSuccess && nc > 0 ? 16 : 8;
    cudaGetLastError();
    if (dev < kMaxOrdinals) __atomic_store_n(&cache[dev], v, __ATOMIC_RELAXED);
    return v;
}

bool lb_loop(const LbLoop& a, int64_t n, cudaStream_t st) {
    const int cl = loop_cluster_size();
    const int64_t per = (int64_t)cl * kLoopThreads;
    if (n > kLoopElems * per) return false;
    const int e = (int)ceil_div(n, per);
    auto k = e <= 1 ? k_lb_loop<1> : e <= 3 ? k_lb_loop<3> : e <= 6 ? k_lb_loop<6> : k_lb_loop<kLoopElems>;
    if (cl > 8) MAF_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cl;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(cl);
    cfg.blockDim = dim3(kLoopThreads);
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    MAF_CUDA(cudaLaunchKernelEx(&cfg, k, a, n));
    return true;
}

// out[1] = g . s, and out[0] = the sum of the energy partials e[0, ne) in the order
// of k_sum_partials (one block of 256 threads)
__global__ void __launch_bounds__(kLbThreads) k_lb_slope(const double* __restrict__ g, const double* __restrict__ s,
                                                         int64_t n, const double* __restrict__ e, int ne, double* part,
                                                         unsigned* counter, double* out) {
    pdl_begin();
    double v[1] = {0.0};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        v[0] += g[i] * s[i];
    if (!reduce_last_block<1>(v, 0u, part, counter, out + 1)) return;
    __shared__ double red[kLbThreads / 32];
    double t = 0.0;
    for (int i = threadIdx.x; i < ne; i += kLbThreads) t += e[i];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x < 32) {
        double x = threadIdx.x < kLbThreads / 32 ? red[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (threadIdx.x == 0) out[0] = x;
    }
}

void lb_slope(const double* g, const double* s, int64_t n, const double* e, int ne, double* part, unsigned* counter,
              double* out, cudaStream_t st) {
    const int blocks = (int)std::min<int64_t>(ceil_div(n, kLbThreads), red_blocks());
    launch_chain(k_lb_slope, dim3(blocks), kLbThreads, 0, st, g, s, n, e, ne, part, counter, out);
}

// s = x - x_old, y = g - g_old; out = max|g|, max|s|, max|x|, y . s, y . y, s . s
__global__ void __launch_bounds__(kLbThreads) k_lb_pair(const double* __restrict__ x, const double* __restrict__ x_old,
                                                        const double* __restrict__ g, const double* __restrict__ g_old,
                                                        double* __restrict__ s, double* __restrict__ y, int64_t n,
                                                        double* part, unsigned* counter, double* out) {
    pdl_begin();
    double v[6] = {0, 0, 0, 0, 0, 0};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double xi = x[i], gi = g[i];
        const double si = xi - x_old[i], yi = gi - g_old[i];
        s[i] = si;
        y[i] = yi;
        v[0] = nanmax(v[0], fabs(gi));
        v[1] = nanmax(v[1], fabs(si));
        v[2] = nanmax(v[2], fabs(xi));
        v[3] += yi * si;
        v[4] += yi * yi;
        v[5] += si * si;
    }
    reduce_last_block<6>(v, 7u, part, counter, out);
}

void lb_pair(const double* x, const double* x_old, const double* g, const double* g_old, double* s, double* y,
             int64_t n, double* part, unsigned* counter, double* out, cudaStream_t st) {
    const int blocks = (int)std::min<int64_t>(ceil_div(n, kLbThreads), red_blocks());
    launch_chain(k_lb_pair, dim3(blocks), kLbThreads, 0, st, x, x_old, g, g_old, s, y, n, part, counter, out);
}

// m = normalize(wa + stp * s) with the zero-safe normalize (lbfgs_minimizer.cpp:274-275)
__global__ void k_normalize_combine(double* __restrict__ m, const double* __restrict__ wa, double stp,
                                    const double* __restrict__ s, int64_t N) {
    pdl_begin();
    for (int64_t cell = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; cell < N;
         cell += (int64_t)gridDim.x * blockDim.x) {
        double v[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c] = wa[c * N + cell] + stp * s[c * N + cell];
        const double nrm = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
#pragma unroll
        for (int c = 0; c < 3; ++c) m[c * N + cell] = nrm != 0 ? v[c] / nrm : 0.0;
    }
}

void normalize_combine(double* m, const double* wa, double stp, const double* s, int64_t N, cudaStream_t st) {
    const int64_t blocks = std::min<int64_t>(ceil_div(N, 256), (int64_t)sm_count() * 8);
    launch_chain(k_normalize_combine, dim3((unsigned)blocks), 256, 0, st, m, wa, stp, s, N);
}

// thermal field sigma * xi(seed, member, index, cell) [3][N] (the h_th of
// stochastic_integrator.cpp:11 as this library draws it)
__global__ void k_noise(double* __restrict__ out, int64_t N, double sigma, unsigned long long seed, unsigned member,
                        unsigned long long index) {
    for (int64_t cell = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; cell < N;
         cell += (int64_t)gridDim.x * blockDim.x) {
        double xi[3];
        normal3(seed, member, index, (uint64_t)cell, xi);
        out[cell] = sigma * xi[0];
        out[N + cell] = sigma * xi[1];
        out[2 * N + cell] = sigma * xi[2];
    }
}

void thermal_field(double* out, int64_t N, double sigma, unsigned long long seed, unsigned member,
                   unsigned long long index, cudaStream_t st) {
    const int64_t blocks = std::min<int64_t>(ceil_div(N, 256), (int64_t)sm_count() * 8);
    k_noise<<<(unsigned)blocks, 256, 0, st>>>(out, N, sigma, seed, member, index);
    MAF_LAUNCH_CHECK();
}

}  // namespace mafb
