// Effective-field kernels: the zero-padded demag FFT convolution in five (3-D)
// or three (nz == 1) passes, with the local terms and the chosen epilogue
// fused into the last pass.
//
// Reference: magnumaf/src/field_terms/micro/demag_field.cpp:215-264
//   H = IFFT( N^ . FFT(pad(Ms m)) ) / (Px Py Pz), truncated to the mesh,
// with P = (2nx, 2ny, nz == 1 ? 1 : 2nz) and the tensor of demag_field.cpp:104-147.
//
// HBM layout (x fastest everywhere):
//   m, H            [3][nz][ny][nx]            real (FP32 or FP64)
//   S1 half spectrum [3][nz][ny][pitch]         complex, kx in [0, nx]
//   S2               [3][nz][Py][pitch]         complex (3-D meshes only)
//   tensor (reduced) [ncomp][nz+1 or 1][ny+1][nx+1] real: the spectral Newell
//                    tensor is real and even/odd in ky and kz, so only the
//                    quadrant ky <= ny, kz <= nz is stored (6 components; 4
//                    when nz == 1 because Nxz = Nyz = 0 in a single layer).
//
// Passes (3-D): x-fwd R2C (zero pad fused into the load) -> y-fwd (pad fused)
//   -> z-fwd . tensor . z-inv (in place, truncation fused) -> y-inv (truncation
//   fused into the store) -> x-inv C2R + local terms + epilogue.
// Passes (nz == 1): x-fwd -> y-fwd . tensor . y-inv (in place) -> x-inv + epilogue.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>

#include "engine.hpp"
#include "epilogue.cuh"
#include "ct_dispatch.hpp"
#include "passes_generic.cuh"

namespace mafb {

// ---------------------------------------------------------------------------
// twiddles and plans
// ---------------------------------------------------------------------------
const std::vector<unsigned char>& Twiddles::host(int L, bool fp64) {
    std::vector<unsigned char>& tab = host_[std::make_pair(L, fp64 ? 1 : 0)];
    if (!tab.empty()) return tab;
    // W_L^k = exp(-2 pi i k / L) in long double, reduced to the first octant
    // so that the table is symmetric to the last bit.
    const long double pi = 3.141592653589793238462643383279502884L;
    std::vector<unsigned char> t((fp64 ? sizeof(double2) : sizeof(float2)) * (size_t)L);
    for (int k = 0; k < L; ++k) {
        // angle = 2 pi k / L; use k/L in [0,1)
        long double a = 2.0L * pi * (long double)k / (long double)L;
        // symmetric evaluation about the quarter points
        int64_t k4 = 4 * (int64_t)k;
        long double cv, sv;
        if (k4 == 0) { cv = 1; sv = 0; }
        else if (k4 == L) { cv = 0; sv = 1; }
        else if (k4 == 2 * (int64_t)L) { cv = -1; sv = 0; }
        else if (k4 == 3 * (int64_t)L) { cv = 0; sv = -1; }
        else { cv = cosl(a); sv = sinl(a); }
        sv = -sv;  // exp(-i a)
        if (fp64) reinterpret_cast<double2*>(t.data())[k] = make_double2((double)cv, (double)sv);
        else reinterpret_cast<float2*>(t.data())[k] = make_float2((float)cv, (float)sv);
    }
    tab = std::move(t);
    return tab;
}

// The upload is complete on return.  cudaMemcpy from pageable memory returns when a small
// buffer has been staged, before the device holds it, and orders the legacy stream only, which
// the library's non-blocking streams do not wait for: a pass could read a new table too early.
const void* Twiddles::upload(std::pair<int, int> key, const std::vector<unsigned char>& tab) {
    DevBuf buf(tab.size());
    MAF_CUDA(cudaMemcpyAsync(buf.p, tab.data(), tab.size(), cudaMemcpyHostToDevice, cudaStreamPerThread));
    MAF_CUDA(cudaStreamSynchronize(cudaStreamPerThread));
    return tables_.emplace(key, std::move(buf)).first->second.p;
}

const void* Twiddles::get(int L, bool fp64) {
    auto key = std::make_pair(L, fp64 ? 1 : 0);
    auto it = tables_.find(key);
    return it != tables_.end() ? it->second.p : upload(key, host(L, fp64));
}

const void* Twiddles::get_ct(int L, bool fp64, const int* radix, int nstages) {
    // (L, precision, radix sequence) identifies the layout
    int code = 0;
    for (int i = 0; i < nstages; ++i) code = code * 17 + radix[i];
    auto key = std::make_pair(L, 2 + (fp64 ? 1 : 0) + 2 * code);
    auto it = tables_.find(key);
    if (it != tables_.end()) return it->second.p;
    const size_t esz = fp64 ? sizeof(double2) : sizeof(float2);
    const std::vector<unsigned char>& tab = host(L, fp64);
    std::vector<unsigned char> out(tab);
    int NS = 1;
    for (int st = 0; st < nstages; ++st) {
        const int RAD = radix[st];
        if (NS > 1) {
            const int twst = L / (NS * RAD);
            for (int jm = 0; jm < NS; ++jm)
                for (int r = 1; r < RAD; ++r) {
                    const size_t k = (size_t)r * jm * twst;  // < L
                    out.insert(out.end(), tab.begin() + k * esz, tab.begin() + (k + 1) * esz);
                }
        }
        NS *= RAD;
    }
    return upload(key, out);
}

FFTPlan make_fft_plan(int L, const void* tw) {
    FFTPlan p;
    p.L = L;
    p.tw = tw;
    int n = L;
    auto push = [&](int r) {
        if (p.nstages >= kMaxStages) throw Error(6, "FFT plan: too many stages");
        p.radix[p.nstages++] = r;
    };
    while (n % 8 == 0) { push(8); n /= 8; }
    if (n % 4 == 0) { push(4); n /= 4; }
    if (n % 2 == 0) { push(2); n /= 2; }
    for (int r : {3, 5, 7, 11, 13}) {
        while (n % r == 0) { push(r); n /= r; }
    }
    if (n != 1)
        throw Error(6, "FFT length " + std::to_string(L) +
                           " has a prime factor > 13; choose mesh sizes whose doubled sizes factor into 2,3,5,7,11,13");
    return p;
}

// ---------------------------------------------------------------------------
// pass kernels
// ---------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(kMaxFftThreads) k_xfwd(const R* __restrict__ in, int n_in, int64_t rows, int64_t rows_pc,
                                               const R* __restrict__ msf, R ms, cplx_t<R>* __restrict__ out, int pitch,
                                               FFTPlan plan, const cplx_t<R>* __restrict__ twP, int nb) {
    xfwd_tile<R>(in, n_in, rows, rows_pc, msf, ms, out, pitch, plan, twP, nb, blockIdx.x);
}

// Strided batched column FFT: element i of column c of batch b at
// base + b*sbat + i*si + c.  Loads n_in values (zero pad to L), stores n_out.
template <typename R, int DIR>
__global__ void __launch_bounds__(kMaxFftThreads) k_fft_cols(const cplx_t<R>* in, cplx_t<R>* out, FFTPlan plan, int n_in,
                                                   int n_out, int ncols, int64_t in_si, int64_t out_si, int64_t in_sbat,
                                                   int64_t out_sbat, int nb) {
    using C = cplx_t<R>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* s = reinterpret_cast<C*>(smem_raw);
    const int L = plan.L;
    const SLay<true> lay{nb, 0};
    const int c0 = blockIdx.x * nb;
    const C* ib = in + (int64_t)blockIdx.y * in_sbat + c0;
    C* ob = out + (int64_t)blockIdx.y * out_sbat + c0;
    const int ncv = min(nb, ncols - c0);
    for (int idx = threadIdx.x; idx < L * nb; idx += blockDim.x) {
        const int i = idx / nb;
        const int b = idx - i * nb;
        C v = mk((R)0, (R)0);
        if (i < n_in && b < ncv) v = ib[i * in_si + b];
        s[lay.at(i, b)] = v;
    }
    __syncthreads();
    run_fft<R, DIR, true>(s, lay, plan);
    for (int idx = threadIdx.x; idx < n_out * nb; idx += blockDim.x) {
        const int i = idx / nb;
        const int b = idx - i * nb;
        if (b < ncv) ob[i * out_si + b] = s[lay.at(i, b)];
    }
}

template <typename R, bool PBC>
__global__ void __launch_bounds__(kMaxFftThreads) k_conv(cplx_t<R>* S, const R* __restrict__ Nred, FFTPlan fplan, FFTPlan iplan,
                                               int n_in, int64_t si, int64_t comp_stride, int64_t other_stride,
                                               int ncols, int nb, int axis_is_z, int ny, int nz, int nxh, PbcOp pop) {
    conv_tile<R, PBC>(S, Nred, fplan, iplan, n_in, si, comp_stride, other_stride, ncols, nb, axis_is_z, ny, nz, nxh,
                      pop, blockIdx.x, blockIdx.y);
}

template <typename R, int EPI>
__global__ void __launch_bounds__(kMaxFftThreads) k_xinv_epi(const cplx_t<R>* __restrict__ S1, int pitch, FFTPlan plan,
                                                   const cplx_t<R>* __restrict__ twP, Geom g, R scale,
                                                   const R* __restrict__ m, MsInfo ms, TermList tl, EpilogueArgs ep,
                                                   int nbr) {
    xinv_tile<R, EPI>(S1, pitch, plan, twP, g, scale, m, ms, tl, ep, nbr, blockIdx.x, 0);
}

// Local terms only (no demag in the term list).
template <typename R, int EPI>
__global__ void __launch_bounds__(256) k_local_epi(Geom g, const R* __restrict__ m, MsInfo ms, TermList tl,
                                                   EpilogueArgs ep) {
    double eacc = 0;
    const R hd[3] = {0, 0, 0};
    for (int64_t cell = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; cell < g.N;
         cell += (int64_t)gridDim.x * blockDim.x) {
        const int x = (int)(cell % g.nx);
        const int64_t r = cell / g.nx;
        const int y = (int)(r % g.ny);
        const int z = (int)(r / g.ny);
        epilogue_cell<R, EPI>(g, x, y, z, cell, m, ms, tl, ep, hd, eacc);
    }
    if constexpr (EPI == EPI_EDENS || EPI == EPI_EGRAD) block_sum_store(eacc, ep.partials);
}

// Local terms only, in runs of RN consecutive cells along x: the x-inverse's
// run epilogue with a zero demag contribution (eligibility: run_mode).
// Thread q takes run q of the flattened (row, run) index (fewer than 2^31 runs).
// FP32: capped for two CTAs per SM (128 registers); FP64 uncapped (it would spill).
template <typename R, int EPI, int RN, bool MSF, bool NEXT>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 2 : 1) k_local_run(Geom g, const R* __restrict__ m, MsInfo ms, TermList tl,
                                                                           EpilogueArgs ep, int nruns) {
    const int runs_row = g.nx / RN;
    double eacc = 0;
    R hd[RN][3];
#pragma unroll
    for (int i = 0; i < RN; ++i) hd[i][0] = hd[i][1] = hd[i][2] = (R)0;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nruns; q += gridDim.x * blockDim.x) {
        const int row = q / runs_row;
        const int x0 = (q - row * runs_row) * RN;
        const int z = row / g.ny;
        const int y = row - z * g.ny;
        const int64_t cell0 = (int64_t)row * g.nx + x0;
        RunN<R, RN> r;
        runN_load<R, RN>(m, g, x0, y, z, cell0, r);
        double Ms = ms.Ms;
        if constexpr (MSF) {
            Ms = ms.field64[cell0];
            r.ms = cell_Ms<R>(ms, cell0);
            r.inv = (R)1 / r.ms;
        }
        eacc += runN_epilogue<R, EPI, RN, MSF, NEXT>(tl, g, r, cell0, hd, ep, Ms);
    }
    if constexpr (EPI == EPI_EDENS || EPI == EPI_EGRAD) block_sum_store(eacc, ep.partials);
}

__global__ void k_sum_partials(const double* __restrict__ p, int n, double* out) {
    double v = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) v += p[i];
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        double s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) *out = s;
    }
}

__global__ void k_stage32(const double* __restrict__ a, float* __restrict__ b, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}

__global__ void k_widen(const float* __restrict__ a, double* __restrict__ b, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = (double)a[i];
}

void widen_m(const float* m32, double* m64, int64_t n, cudaStream_t st) {
    const int64_t blocks = std::min<int64_t>(ceil_div(n, 256), (int64_t)sm_count() * 16);
    k_widen<<<(unsigned)blocks, 256, 0, st>>>(m32, m64, n);
    MAF_LAUNCH_CHECK();
}

void stage_m32(const double* m64, float* m32, int64_t n, cudaStream_t st) {
    const int64_t blocks = std::min<int64_t>(ceil_div(n, 256), (int64_t)sm_count() * 16);
    k_stage32<<<(unsigned)blocks, 256, 0, st>>>(m64, m32, n);
    MAF_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// Parity of the tensor.  Component comp (0..5: xx, xy, xz, yy, yz, zz) is odd
// along the axes its letters name once (xy: x and y) and even along the others.
// On a periodic grid of even length L an odd function vanishes at j = 0 and at
// j = L/2 (the plane there never reaches the truncated output of the zero-padded
// convolution), so the entries at 0 <= j <= L/2 determine the component, its
// transform is real (odd axes come in pairs) and has the same parity.
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ bool tensor_odd(int comp, int axis) {
    return axis == 0 ? (comp == 1 || comp == 2) : axis == 1 ? (comp == 1 || comp == 4) : (comp == 2 || comp == 4);
}

// Entry at the wrapped index i of an axis of length L: the stored offset j, the
// sign, and whether it is zero by parity (odd).
__device__ __forceinline__ int wrap_offset(int i, int L, bool odd, bool& neg, bool& zero) {
    const int j = 2 * i <= L ? i : L - i;
    if (odd) {
        neg = neg != (2 * i > L);
        zero = zero || j == 0 || 2 * i == L;
    }
    return j;
}

// The components a launch completes (blockIdx.y), one array after the other.
struct TensorComps {
    int c[6];
};

// rows [nz][ny][L] of real values from the octant [o2][o1][o0] (zero beyond it): the
// x axis completed by parity; rows on the zero planes of the other axes are zero
__global__ void k_tensor_rows(const double* __restrict__ oct, double* __restrict__ out, TensorComps comps, int o0,
                              int o1, int o2, int ny, int nz, int Ly, int Lz, int L) {
    const int64_t total = (int64_t)L * ny * nz;
    const int comp = comps.c[blockIdx.y];
    oct += (int64_t)blockIdx.y * o0 * o1 * o2;
    out += blockIdx.y * total;
    const bool ox = tensor_odd(comp, 0), oy = tensor_odd(comp, 1), oz = tensor_odd(comp, 2);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int x = (int)(i % L);
        const int64_t r = i / L;
        const int y = (int)(r % ny), z = (int)(r / ny);
        bool neg = false, zero = (oy && (y == 0 || 2 * y == Ly)) || (oz && (z == 0 || 2 * z == Lz));
        const int j = wrap_offset(x, L, ox, neg, zero);
        const double v = zero || j >= o0 || y >= o1 || z >= o2 ? 0.0 : oct[((int64_t)z * o1 + y) * o0 + j];
        out[i] = neg ? -v : v;
    }
}

// spectrum rows completed along one axis by parity: out [A][L][B][pitch] from the
// rows a sa + j sj + b of in (rows_in of them per component), j <= L/2 (y: A = z planes,
// B = 1; z: A = 1, B = ky rows)
__global__ void k_tensor_wrap(const double2* __restrict__ in, double2* __restrict__ out, int64_t rows_in, int64_t A,
                              int L, int64_t B, int64_t sa, int64_t sj, TensorComps comps, int axis, int pitch,
                              int nxh) {
    const int64_t total = A * L * B * nxh;
    const bool odd = tensor_odd(comps.c[blockIdx.y], axis);
    in += blockIdx.y * rows_in * pitch;
    out += blockIdx.y * A * L * B * pitch;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int x = (int)(i % nxh);
        int64_t r = i / nxh;
        const int64_t o = r * pitch + x;
        const int64_t b = r % B;
        r /= B;
        const int l = (int)(r % L);
        const int64_t a = r / L;
        bool neg = false, zero = false;
        const int j = wrap_offset(l, L, odd, neg, zero);
        double2 v = make_double2(0.0, 0.0);
        if (!zero) v = in[(a * sa + j * sj + b) * pitch + x];
        out[o] = neg ? make_double2(-v.x, -v.y) : v;
    }
}

// scaled real part of the spectrum (rows_in rows per component) on the stored quadrant
__global__ void k_tensor_real(const double2* __restrict__ spec, int64_t rows_in, double* __restrict__ dst, int64_t rows,
                              int nxh, int pitch, double scale, int Ky, int spec_ky) {
    const int64_t total = rows * nxh;
    spec += blockIdx.y * rows_in * pitch;
    dst += blockIdx.y * total;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int kx = (int)(i % nxh);
        const int64_t r = i / nxh;
        dst[i] = scale * spec[((r / Ky) * spec_ky + r % Ky) * pitch + kx].x;
    }
}

// the parity-exact tensor on the padded grid [Pz][Py][Px] from its octant
__global__ void k_tensor_full(const double* __restrict__ oct, double* __restrict__ out, int comp, int o0, int o1,
                              int Px, int Py, int Pz) {
    const int64_t total = (int64_t)Px * Py * Pz;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int x = (int)(i % Px);
        const int64_t r = i / Px;
        bool neg = false, zero = false;
        const int jx = wrap_offset(x, Px, tensor_odd(comp, 0), neg, zero);
        const int jy = wrap_offset((int)(r % Py), Py, tensor_odd(comp, 1), neg, zero);
        const int jz = wrap_offset((int)(r / Py), Pz, tensor_odd(comp, 2), neg, zero);
        const double v = zero ? 0.0 : oct[((int64_t)jz * o1 + jy) * o0 + jx];
        out[i] = neg ? -v : v;
    }
}

__global__ void k_d2f(const double* __restrict__ a, float* __restrict__ b, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}

// ---------------------------------------------------------------------------
// launch helpers
// ---------------------------------------------------------------------------
void raise_smem(const void* kernel, size_t bytes) {
    // opt in above 32 KB: the 48 KB default also has to hold the static shared memory
    if (bytes <= 32 * 1024) return;
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    cudaFuncAttributes a;
    MAF_CUDA(cudaFuncGetAttributes(&a, kernel));
    if ((size_t)a.maxDynamicSharedSizeBytes < bytes)
        MAF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}
template <typename K> static void set_smem(K kernel, size_t bytes) { raise_smem((const void*)kernel, bytes); }


template <typename R>
static void launch_xfwd(const R* in, int n_in, int64_t rows, int64_t rows_pc, const R* msf, R ms, cplx_t<R>* out,
                        int pitch, int Px, Twiddles& tw, cudaStream_t st, bool try_ct = true) {
    if (try_ct && ct_xfwd<R>(in, n_in, rows, rows_pc, msf, ms, out, pitch, Px, tw, st)) return;
    const bool f64 = sizeof(R) == 8;
    const int Lc = Px / 2;
    FFTPlan plan = make_fft_plan(Lc, tw.get(Lc, f64));
    int nb = pick_nb(Lc, tile_target<R>(), (int)std::min<int64_t>(rows, 1 << 20), 64);
    int threads;
    while (true) {
        threads = fft_threads_needed(plan, nb);
        threads = std::max(threads, std::min(256, nb * Lc));
        if (threads <= kMaxFftThreads || nb == 1) break;
        nb = std::max(1, nb / 2);
    }
    threads = round_threads(threads);
    const size_t smem = sizeof(cplx_t<R>) * (size_t)nb * spad_len(Lc);
    set_smem(k_xfwd<R>, smem);
    const int64_t blocks = ceil_div(rows, nb);
    k_xfwd<R><<<(unsigned)blocks, threads, smem, st>>>(in, n_in, rows, rows_pc, msf, ms, out, pitch, plan,
                                                       static_cast<const cplx_t<R>*>(tw.get(Px, f64)), nb);
    MAF_LAUNCH_CHECK();
}

template <typename R, int DIR>
static void launch_cols(const cplx_t<R>* in, cplx_t<R>* out, int L, int n_in, int n_out, int ncols, int64_t in_si,
                        int64_t out_si, int64_t in_sbat, int64_t out_sbat, int nbat, Twiddles& tw,
                        const TuneChoice& tc, cudaStream_t st, bool try_ct = true) {
    if (try_ct && ct_cols<R, DIR>(in, out, L, n_in, n_out, ncols, in_si, out_si, in_sbat, out_sbat, nbat, tw, tc, st))
        return;
    const bool f64 = sizeof(R) == 8;
    FFTPlan plan = make_fft_plan(L, tw.get(L, f64));
    int nb = pick_nb(L, tile_target<R>(), ncols, 32);
    int threads;
    while (true) {
        threads = fft_threads_needed(plan, nb);
        threads = std::max(threads, std::min(256, nb * L));
        if (threads <= kMaxFftThreads || nb == 1) break;
        nb = std::max(1, nb / 2);
    }
    threads = round_threads(threads);
    const size_t smem = sizeof(cplx_t<R>) * (size_t)nb * spad_len(L);
    set_smem(k_fft_cols<R, DIR>, smem);
    dim3 grid((unsigned)ceil_div(ncols, nb), (unsigned)nbat);
    k_fft_cols<R, DIR><<<grid, threads, smem, st>>>(in, out, plan, n_in, n_out, ncols, in_si, out_si, in_sbat,
                                                    out_sbat, nb);
    MAF_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// Demag
// ---------------------------------------------------------------------------
// Lengths of the compile-time passes: packed x rows, y convolutions (2-D meshes), y
// passes (3-D) and z convolutions.
static const int kCtX[] = {16, 32, 64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048, 0};
static const int kCtY2[] = {16, 32, 64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048, 0};
static const int kCtY3[] = {16, 32, 64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048, 4096, 0};
static const int kCtZ[] = {8, 16, 32, 64, 96, 128, 0};

// the smallest length of the list that is at least n, 0 if there is none
static int ct_length(const int* list, int n) {
    for (; *list; ++list)
        if (*list >= n) return *list;
    return 0;
}

// Zero padding to any length of at least 2n - 1 gives the same linear convolution, so an axis
// whose doubled size has no compile-time kernel is padded to the next length that has one.  All
// axes are padded or, when one has no such length, none.  On 3-D meshes the y and z passes run
// over the padded x spectrum, so there x keeps its own length (on the run-time-plan kernel)
// where padding it costs the other passes more than it saves: when its spectrum grows by more
// than 1.6, or by more than 1.25 beside a y transform of 4096 points (whose CTAs take one or
// two columns, part of a sector per row); unless the padded spectrum has up to 2^16 values,
// where launches dominate.  Field times in us on B200, FP64 / FP32, x at its own length and
// padded (y and z padded in both), with x's growth:
//      1 x 1024 x 64  8.5     72 / 63     341 / 192
//      8 x 512 x 64   1.89   148 / 102    166 / 94
//      9 x 300 x 20   1.70    58 / 43      69 / 55
//     10 x 500 x 30   1.55    96 / 68      87 / 67
//    520 x 520 x 18   1.48  3318 / 1659  3260 / 1488
//   1040 x 600 x 9    1.48  3082 / 1727  2571 / 1168
//   1040 x 1040 x 9   1.48  8400 / 4507  12099 / 5370   (4096)
//   1100 x 1100 x 2   1.40  2184 / 1122  2389 / 1009    (4096)
//    600 x 1040 x 9   1.28  4437 / 2370  5639 / 2490    (4096)
//   1300 x 1300 x 4   1.18  5559 / 2880  4825 / 2017    (4096)
//      6 x 60 x 6     2.43    29 / 27      21 / 20      (35 k values)
//      1 x 256 x 4    8.5     23 / 21      35 / 28      (70 k values)
// y and z padded (x as above) against their own lengths: 520 x 520 x 9 3034 / 1830 -> 1287 /
// 607, 1040 x 1040 x 18 28650 / 14206 -> 20081 / 10563, 1024 x 1 x 16 31 / 25 -> 33 / 26.
// 2-D meshes, both padded against both own: 1040 x 1000 864 / 546 -> 316 / 169, 1 x 1000 71 /
// 60 -> 32 / 21.
void demag_lengths(int nx, int ny, int nz, int out[3]) {
    const int own[3] = {2 * nx, 2 * ny, nz == 1 ? 1 : 2 * nz};
    const int pad[3] = {2 * ct_length(kCtX, nx), ct_length(nz == 1 ? kCtY2 : kCtY3, 2 * ny - 1),
                        nz == 1 ? 1 : ct_length(kCtZ, 2 * nz - 1)};
    const bool padded = pad[0] && pad[1] && pad[2];
    for (int a = 0; a < 3; ++a) out[a] = padded ? pad[a] : own[a];
    if (!padded || nz == 1) return;
    const int64_t nxh = pad[0] / 2 + 1;
    if (nxh * pad[1] * pad[2] > (1 << 16) && nxh > (pad[1] == 4096 ? 1.25 : 1.6) * (nx + 1)) out[0] = own[0];
}

unsigned long long Demag::next_id() {
    static std::atomic<unsigned long long> n{0};
    return ++n;
}

Demag::Demag(const MeshDims& md, cudaStream_t st, const double* tensor_host, bool pbc) : md_(md), pbc_(pbc) {
    if (md.nx < 1 || md.ny < 1 || md.nz < 1) throw Error(1, "DemagField: empty mesh");
    if (pbc) {
        // the reference's inverse fftC2R(h, is_odd = false) returns 2*(nx/2) columns,
        // i.e. the field only has the mesh's shape for even nx (demag_field_pbc.cpp:70)
        if (md.nx % 2 != 0) throw Error(6, "DemagFieldPBC: nx must be even");
        pitch_ = (nxh() + 3) / 4 * 4;
        make_fft_plan(Px() / 2, nullptr);
        make_fft_plan(Py(), nullptr);
        make_fft_plan(Pz(), nullptr);
        return;
    }
    // complex pitch: multiple of 4 so that tiles of 4 complex values start on 32 B
    pitch_ = (nxh() + 3) / 4 * 4;
    int len[3];
    demag_lengths(md.nx, md.ny, md.nz, len);
    pad_x_ = len[0];
    pad_y_ = len[1];
    pad_z_ = len[2];
    padded_ = pad_x_ != Px() || pad_y_ != Py() || pad_z_ != Pz();
    // validate all FFT lengths early
    make_fft_plan(Px() / 2, nullptr);
    make_fft_plan(Py(), nullptr);
    make_fft_plan(Pz(), nullptr);
    if (tensor_host) {
        Nred64_.alloc(sizeof(double) * tensor_elems());
        MAF_CUDA(cudaMemcpyAsync(Nred64_.p, tensor_host, sizeof(double) * tensor_elems(), cudaMemcpyHostToDevice, st));
        MAF_CUDA(cudaStreamSynchronize(st));
    } else {
        build_tensor(st);
    }
}

Demag::~Demag() {
    std::vector<DevBuf*> v = {&Nred64_, &Nred32_, &Npad64_, &Npad32_, &S1_64_, &S2_64_, &S1_32_, &S2_32_};
    tw_.append_buffers(v);
    release_all(v);
}

// Real spectra (times scale) on the quadrant [Lz/2+1][Ly/2+1][Lx/2+1] (Lz = 1: one
// plane) of the periodic functions of lengths (Lx, Ly, Lz) that the octants `oct`
// [o2][o1][o0] of nc tensor components complete by parity (oct and quad: one component
// after the other).  The spectrum has the component's parity, so the transform of its
// quadrant over L values, divided by L, is the octant.  Each axis is completed just before
// its transform, so the x transforms run on a quarter of the rows, the y transforms on half
// of the planes and the z transforms on half of the rows.  The octants are read before the
// quadrants are written.  work: octant_work bytes.
static size_t octant_work_a(int Lx, int Ly, int Lz, int nc) {
    // the completed real rows, then the completed y columns
    const int Ky = Ly / 2 + 1, Kz = Lz == 1 ? 1 : Lz / 2 + 1, pitch = (Lx / 2 + 4) / 4 * 4;
    return (nc * std::max(sizeof(double) * (size_t)Lx * Ky * Kz, sizeof(double2) * (size_t)Kz * Ly * pitch) + 255) / 256 *
           256;
}
static size_t octant_work(int Lx, int Ly, int Lz, int nc) {
    // and the x spectra, then the completed z columns
    const int Ky = Ly / 2 + 1, Kz = Lz == 1 ? 1 : Lz / 2 + 1, pitch = (Lx / 2 + 4) / 4 * 4;
    const size_t b =
        sizeof(double2) * nc * (size_t)std::max<int64_t>((int64_t)Ky * Kz, Lz > 1 ? (int64_t)Lz * Ky : 0) * pitch;
    return octant_work_a(Lx, Ly, Lz, nc) + (b + 255) / 256 * 256;
}

// Components that are transformed together: all of them while the work buffers stay
// within kTensorBatch, else one by one: small tensors are launches of 3-15 us one after the
// other, 24 for the four components of a film.  A new tensor one by one and together: 24 x
// 24 x 1 302 and 184 us, 250 x 240 x 1 583 and 384, 66 x 91 x 6 816 and 501, 200 x 120 x 10
// (99 MB) 1947 and 1772.
constexpr size_t kTensorBatch = 128u << 20;
static int octant_batch(size_t work_all, int ncomp) { return work_all <= kTensorBatch ? ncomp : 1; }

void Demag::transform_octants(const double* oct, int o0, int o1, int o2, const int* comps, int nc, int Lx, int Ly,
                              int Lz, double* quad, double scale, char* work, cudaStream_t st) {
    const int nxh = Lx / 2 + 1, Ky = Ly / 2 + 1, Kz = Lz == 1 ? 1 : Lz / 2 + 1;
    const int pitch = (nxh + 3) / 4 * 4;
    TensorComps c = {};
    for (int i = 0; i < nc; ++i) c.c[i] = comps[i];
    char* work_b = work + octant_work_a(Lx, Ly, Lz, nc);
    auto grid = [nc](int64_t n) {
        return dim3((unsigned)std::min<int64_t>(ceil_div(n, 256), (int64_t)sm_count() * 16), (unsigned)nc);
    };
    double* rows = reinterpret_cast<double*>(work);
    double2* ycol = reinterpret_cast<double2*>(work);
    double2* xs = reinterpret_cast<double2*>(work_b);
    const int64_t xrows = (int64_t)Ky * Kz, yrows = (int64_t)Kz * Ly, zrows = (int64_t)Lz * Ky;
    k_tensor_rows<<<grid(Lx * xrows), 256, 0, st>>>(oct, rows, c, o0, o1, o2, Ky, Kz, Ly, Lz, Lx);
    MAF_LAUNCH_CHECK();
    launch_xfwd<double>(rows, Lx, nc * xrows, nc * xrows, nullptr, 1.0, xs, pitch, Lx, tw_, st);
    k_tensor_wrap<<<grid(yrows * nxh), 256, 0, st>>>(xs, ycol, xrows, Kz, Ly, 1, Ky, 1, c, 1, pitch, nxh);
    MAF_LAUNCH_CHECK();
    launch_cols<double, -1>(ycol, ycol, Ly, Ly, Ly, nxh, pitch, pitch, (int64_t)Ly * pitch, (int64_t)Ly * pitch,
                            nc * Kz, tw_, tune, st);
    if (Lz > 1) {
        // a component's columns are its rows of ky one after the other, the pitch's padding too
        double2* zcol = reinterpret_cast<double2*>(work_b);
        k_tensor_wrap<<<grid(zrows * nxh), 256, 0, st>>>(ycol, zcol, yrows, 1, Lz, Ky, 0, Ly, c, 2, pitch, nxh);
        MAF_LAUNCH_CHECK();
        launch_cols<double, -1>(zcol, zcol, Lz, Lz, Lz, Ky * pitch, (int64_t)Ky * pitch, (int64_t)Ky * pitch,
                                zrows * pitch, zrows * pitch, nc, tw_, tune, st);
        k_tensor_real<<<grid(xrows * nxh), 256, 0, st>>>(zcol, zrows, quad, xrows, nxh, pitch, scale, Ky, Ky);
    } else {
        k_tensor_real<<<grid((int64_t)Ky * nxh), 256, 0, st>>>(ycol, yrows, quad, Ky, nxh, pitch, scale, Ky, Ly);
    }
    MAF_LAUNCH_CHECK();
}

// tensor components that are stored, in order
static const int kComps6[6] = {0, 1, 2, 3, 4, 5};
static const int kComps4[4] = {0, 1, 3, 5};

void Demag::build_tensor(cudaStream_t st) {
    const int Kx = md_.nx + 1, Ky = md_.ny + 1, Kz = md_.nz == 1 ? 1 : md_.nz + 1;
    const int64_t cstride = (int64_t)Kz * Ky * Kx;
    const int* comps = md_.nz == 1 ? kComps4 : kComps6;
    Nred64_.alloc(sizeof(double) * cstride * ncomp());
    // the octants where the transforms replace them
    newell_octants(Nred64_.as<double>(), comps, ncomp(), md_, Kx, Ky, Kz, st);
    const int nb = octant_batch(octant_work(Px(), Py(), Pz(), ncomp()), ncomp());
    DevBuf work(octant_work(Px(), Py(), Pz(), nb));
    for (int ci = 0; ci < ncomp(); ci += nb) {
        double* t = Nred64_.as<double>() + ci * cstride;
        transform_octants(t, Kx, Ky, Kz, comps + ci, nb, Px(), Py(), Pz(), t, 1.0, work.as<char>(), st);
    }
    MAF_CUDA(cudaStreamSynchronize(st));
    work.release(true);
}

// The tensor at the padded lengths (FP64 or FP32), from the one at twice the mesh
// (assembled or read from a file: the same values either way): back to its octant of
// offsets, then forward at the other lengths.
void Demag::build_padded_tensor(double* out64, float* out32, cudaStream_t st) {
    const int Kx = md_.nx + 1, Ky = md_.ny + 1, Kz = md_.nz == 1 ? 1 : md_.nz + 1;
    const int64_t cstride = (int64_t)Kz * Ky * Kx, pstride = (int64_t)padded_elems() / ncomp();
    const int* comps = md_.nz == 1 ? kComps4 : kComps6;
    auto oct_bytes = [&](int nc) { return (sizeof(double) * nc * cstride + 255) / 256 * 256; };
    auto quad_bytes = [&](int nc) { return out32 ? (sizeof(double) * nc * pstride + 255) / 256 * 256 : (size_t)0; };
    auto bytes = [&](int nc) {
        return oct_bytes(nc) + quad_bytes(nc) +
               std::max(octant_work(Px(), Py(), Pz(), nc), octant_work(pad_x_, pad_y_, pad_z_, nc));
    };
    const int nb = octant_batch(bytes(ncomp()), ncomp());
    DevBuf scratch(bytes(nb));
    double* oct = scratch.as<double>();
    double* quad = reinterpret_cast<double*>(scratch.as<char>() + oct_bytes(nb));
    char* work = scratch.as<char>() + oct_bytes(nb) + quad_bytes(nb);
    const double scale = 1.0 / ((double)Px() * Py() * Pz());
    for (int ci = 0; ci < ncomp(); ci += nb) {
        transform_octants(Nred64_.as<double>() + ci * cstride, Kx, Ky, Kz, comps + ci, nb, Px(), Py(), Pz(), oct, scale,
                          work, st);
        transform_octants(oct, Kx, Ky, Kz, comps + ci, nb, pad_x_, pad_y_, pad_z_, out32 ? quad : out64 + ci * pstride,
                          1.0, work, st);
        if (out32) {
            const int64_t n = nb * pstride;
            k_d2f<<<(unsigned)std::min<int64_t>(ceil_div(n, 256), (int64_t)sm_count() * 16), 256, 0, st>>>(
                quad, out32 + ci * pstride, n);
            MAF_LAUNCH_CHECK();
        }
    }
    MAF_CUDA(cudaStreamSynchronize(st));
    scratch.release(true);
}

void Demag::download_tensor(double* host, cudaStream_t st) const {
    MAF_CUDA(cudaMemcpyAsync(host, Nred64_.p, sizeof(double) * tensor_elems(), cudaMemcpyDeviceToHost, st));
    MAF_CUDA(cudaStreamSynchronize(st));
}

void Demag::download_real_tensor(double* host, bool symmetric, cudaStream_t st) {
    const int64_t nreal = (int64_t)Px() * Py() * Pz();
    const int Kx = md_.nx + 1, Ky = md_.ny + 1, Kz = md_.nz == 1 ? 1 : md_.nz + 1;
    DevBuf real(sizeof(double) * nreal), oct;
    if (symmetric) oct.alloc(sizeof(double) * Kx * Ky * Kz);
    for (int c = 0; c < 6; ++c) {
        if (symmetric) {
            newell_octants(oct.as<double>(), &c, 1, md_, Kx, Ky, Kz, st);
            k_tensor_full<<<(unsigned)std::min<int64_t>(ceil_div(nreal, 256), (int64_t)sm_count() * 16), 256, 0, st>>>(
                oct.as<double>(), real.as<double>(), c, Kx, Ky, Px(), Py(), Pz());
            MAF_LAUNCH_CHECK();
        } else {
            newell_component(real.as<double>(), c, md_, Px(), Py(), Pz(), st);
        }
        MAF_CUDA(cudaMemcpyAsync(host + c * nreal, real.p, sizeof(double) * nreal, cudaMemcpyDeviceToHost, st));
    }
    MAF_CUDA(cudaStreamSynchronize(st));
}

template <> const double* Demag::tensor<double>(cudaStream_t) { return Nred64_.as<double>(); }
template <> const float* Demag::tensor<float>(cudaStream_t st) {
    if (!Nred32_.p) {
        const int64_t n = (int64_t)tensor_elems();
        DevBuf t(sizeof(float) * n);
        k_d2f<<<(unsigned)std::min<int64_t>(ceil_div(n, 256), (int64_t)sm_count() * 16), 256, 0, st>>>(
            Nred64_.as<double>(), t.as<float>(), n);
        MAF_LAUNCH_CHECK();
        MAF_CUDA(cudaStreamSynchronize(st));  // other streams may use it next
        Nred32_ = std::move(t);
    }
    return Nred32_.as<float>();
}

template <> cplx_t<double>* Demag::S1<double>(int pitch) {
    S1_64_.ensure(sizeof(double2) * 3 * md_.N() / md_.nx * pitch);
    return S1_64_.as<double2>();
}
template <> cplx_t<float>* Demag::S1<float>(int pitch) {
    S1_32_.ensure(sizeof(float2) * 3 * md_.N() / md_.nx * pitch);
    return S1_32_.as<float2>();
}
template <> cplx_t<double>* Demag::S2<double>(int Py, int pitch) {
    S2_64_.ensure(sizeof(double2) * 3 * (int64_t)md_.nz * Py * pitch);
    return S2_64_.as<double2>();
}
template <> cplx_t<float>* Demag::S2<float>(int Py, int pitch) {
    S2_32_.ensure(sizeof(float2) * 3 * (int64_t)md_.nz * Py * pitch);
    return S2_32_.as<float2>();
}

template <typename R> DemagPlan<R> Demag::plan(cudaStream_t st) {
    DemagPlan<R> p;
    if (padded_ && !tune.generic) {
        p.Px = pad_x_;
        p.Py = pad_y_;
        p.Pz = pad_z_;
        p.nxh = pad_x_ / 2 + 1;
        p.pitch = (p.nxh + 3) / 4 * 4;
        DevBuf& N = sizeof(R) == 8 ? Npad64_ : Npad32_;
        try {
            if (!N.p) {
                DevBuf t(sizeof(R) * padded_elems());
                if constexpr (sizeof(R) == 8)
                    build_padded_tensor(t.as<double>(), nullptr, st);
                else
                    build_padded_tensor(nullptr, t.as<float>(), st);
                N = std::move(t);
            }
            p.s1 = S1<R>(p.pitch);
            p.s2 = md_.nz > 1 ? S2<R>(p.Py, p.pitch) : nullptr;
            p.tensor = N.as<R>();
            p.padded = true;
            return p;
        } catch (const Error& e) {
            if (e.code != 3) throw;
            // no memory for the longer transforms: the mesh's own lengths from here on
            cudaGetLastError();
            N.release();
            padded_ = false;
        }
    }
    p.Px = Px();
    p.Py = Py();
    p.Pz = Pz();
    p.nxh = nxh();
    p.pitch = pitch_;
    p.s1 = S1<R>(pitch_);
    p.s2 = md_.nz > 1 ? S2<R>(Py(), pitch_) : nullptr;
    // the periodic form has no tensor and runs the run-time plans only
    p.tensor = pbc_ ? nullptr : tensor<R>(st);
    return p;
}

template <typename R> void Demag::forward_conv(const R* m, const MsInfo& ms, cudaStream_t st, PassMarks* marks) {
    using C = cplx_t<R>;
    const bool f64 = sizeof(R) == 8;
    const int nx = md_.nx, ny = md_.ny, nz = md_.nz;
    const int64_t rows_pc = (int64_t)ny * nz;
    const R* msf = nullptr;
    if (ms.field64) {
        if constexpr (sizeof(R) == 4) msf = reinterpret_cast<const R*>(ms.field32);
        else msf = reinterpret_cast<const R*>(ms.field64);
    }
    const bool ct = !pbc_ && !tune.generic;
    const DemagPlan<R> pl = plan<R>(st);
    C* s1 = pl.s1;
    const R* Nr = pl.tensor;
    const int Py_ = pl.Py, nxh_ = pl.nxh, pitch = pl.pitch;
    const PbcOp pop{nx, ny, nz, md_.dx, md_.dy, md_.dz};
    // pass 1: x forward (zero pad fused)
    launch_xfwd<R>(m, nx, 3 * rows_pc, rows_pc, msf, (R)ms.Ms, s1, pitch, pl.Px, tw_, st, ct);
    if (marks) marks->mark(st, "x_fwd");
    if (nz > 1) {
        C* s2 = pl.s2;
        // pass 2: y forward, S1 [3*nz][ny][pitch] -> S2 [3*nz][Py][pitch]
        launch_cols<R, -1>(s1, s2, Py_, ny, Py_, nxh_, pitch, pitch, (int64_t)ny * pitch,
                           (int64_t)Py_ * pitch, 3 * nz, tw_, tune, st, ct);
        if (marks) marks->mark(st, "y_fwd");
        // pass 3: z forward . tensor . z inverse, in place on S2
        if (!ct || !ct_convz<R>(s2, Nr, nz, pl.Pz, Py_ / 2, nxh_, pitch, tw_, tune, st)) {
            const int L = pl.Pz;
            FFTPlan fp = make_fft_plan(L, tw_.get(L, f64));
            FFTPlan ip = fp;
            int nb = pick_nb(3 * L, tile_target<R>(), nxh_, 64);
            int threads;
            while (true) {
                threads = std::max(fft_threads_needed(fp, 3 * nb), std::min(256, 3 * nb * L));
                if (threads <= kMaxFftThreads || nb == 1) break;
                nb = std::max(1, nb / 2);
            }
            threads = round_threads(threads);
            const size_t smem = sizeof(C) * (size_t)3 * nb * spad_len(L);
            dim3 grid((unsigned)ceil_div(nxh_, nb), (unsigned)Py_);
            if (pbc_) {
                set_smem(k_conv<R, true>, smem);
                k_conv<R, true><<<grid, threads, smem, st>>>(s2, Nr, fp, ip, nz, (int64_t)Py_ * pitch,
                                                             (int64_t)nz * Py_ * pitch, pitch, nxh_, nb, 1, ny,
                                                             nz, nxh_, pop);
            } else {
                set_smem(k_conv<R, false>, smem);
                k_conv<R, false><<<grid, threads, smem, st>>>(s2, Nr, fp, ip, nz, (int64_t)Py_ * pitch,
                                                              (int64_t)nz * Py_ * pitch, pitch, nxh_, nb, 1, Py_ / 2,
                                                              pl.Pz / 2, nxh_, pop);
            }
            MAF_LAUNCH_CHECK();
        }
        if (marks) marks->mark(st, "z_conv");
        // pass 4: y inverse, S2 -> S1, keep ky rows [0, ny)
        launch_cols<R, 1>(s2, s1, Py_, Py_, ny, nxh_, pitch, pitch, (int64_t)Py_ * pitch,
                          (int64_t)ny * pitch, 3 * nz, tw_, tune, st, ct);
        if (marks) marks->mark(st, "y_inv");
    } else {
        // pass 2 (2-D): y forward . tensor . y inverse, in place on S1
        if (ct && ct_convy<R>(s1, Nr, ny, Py_, nxh_, pitch, tw_, st)) {
            if (marks) marks->mark(st, "y_conv");
            return;
        }
        const int L = Py_;
        FFTPlan fp = make_fft_plan(L, tw_.get(L, f64));
        int nb = pick_nb(3 * L, tile_target<R>(), nxh_, 64);
        int threads;
        while (true) {
            threads = std::max(fft_threads_needed(fp, 3 * nb), std::min(256, 3 * nb * L));
            if (threads <= kMaxFftThreads || nb == 1) break;
            nb = std::max(1, nb / 2);
        }
        threads = round_threads(threads);
        const size_t smem = sizeof(C) * (size_t)3 * nb * spad_len(L);
        dim3 grid((unsigned)ceil_div(nxh_, nb), 1);
        if (pbc_) {
            set_smem(k_conv<R, true>, smem);
            k_conv<R, true><<<grid, threads, smem, st>>>(s1, Nr, fp, fp, ny, pitch, (int64_t)ny * pitch, 0, nxh_,
                                                         nb, 0, ny, nz, nxh_, pop);
        } else {
            set_smem(k_conv<R, false>, smem);
            k_conv<R, false><<<grid, threads, smem, st>>>(s1, Nr, fp, fp, ny, pitch, (int64_t)ny * pitch, 0, nxh_,
                                                          nb, 0, ny, nz, nxh_, pop);
        }
        MAF_LAUNCH_CHECK();
        if (marks) marks->mark(st, "y_conv");
    }
}

template <typename R>
void Demag::inverse_x_epilogue(const R* m, const MsInfo& ms, const TermList& tl, const EpilogueArgs& ep,
                               cudaStream_t st, int* nblocks_out, PassMarks* marks) {
    const bool f64 = sizeof(R) == 8;
    const DemagPlan<R> pl = plan<R>(st);
    const int Lc = pl.Px / 2;
    if (!pbc_ && !tune.generic) {
        const R scale = (R)(1.0 / ((double)pl.Px * pl.Py * pl.Pz));
        if (ct_xinv<R>(pl.s1, pl.pitch, pl.Px, tw_, md_.geom(), scale, m, ms, tl, ep, tune, st, nblocks_out)) {
            if (marks) marks->mark(st, "x_inv_local");
            return;
        }
    }
    FFTPlan plan = make_fft_plan(Lc, tw_.get(Lc, f64));
    const int64_t rows_pc = (int64_t)md_.ny * md_.nz;
    int nbr = pick_nb(3 * Lc, tile_target<R>(), (int)std::min<int64_t>(rows_pc, 1 << 20), 32);
    int threads;
    while (true) {
        threads = std::max(fft_threads_needed(plan, 3 * nbr), std::min(256, 3 * nbr * Lc));
        if (threads <= kMaxFftThreads || nbr == 1) break;
        nbr = std::max(1, nbr / 2);
    }
    threads = round_threads(threads);
    const size_t smem = sizeof(cplx_t<R>) * (size_t)3 * nbr * spad_len(Lc);
    const int64_t blocks = ceil_div(rows_pc, nbr);
    if (nblocks_out) *nblocks_out = (int)blocks;
    const R scale = (R)(1.0 / ((double)pl.Px * pl.Py * pl.Pz));
    const cplx_t<R>* tP = static_cast<const cplx_t<R>*>(tw_.get(pl.Px, f64));
    const Geom g = md_.geom();
    switch (ep.kind) {
        case EPI_H:
            set_smem(k_xinv_epi<R, EPI_H>, smem);
            k_xinv_epi<R, EPI_H><<<(unsigned)blocks, threads, smem, st>>>(pl.s1, pl.pitch, plan, tP, g, scale, m, ms,
                                                                          tl, ep, nbr);
            break;
        case EPI_LLG:
            set_smem(k_xinv_epi<R, EPI_LLG>, smem);
            k_xinv_epi<R, EPI_LLG><<<(unsigned)blocks, threads, smem, st>>>(pl.s1, pl.pitch, plan, tP, g, scale, m,
                                                                            ms, tl, ep, nbr);
            break;
        case EPI_EGRAD:
            set_smem(k_xinv_epi<R, EPI_EGRAD>, smem);
            k_xinv_epi<R, EPI_EGRAD><<<(unsigned)blocks, threads, smem, st>>>(pl.s1, pl.pitch, plan, tP, g, scale, m,
                                                                              ms, tl, ep, nbr);
            break;
        default:
            set_smem(k_xinv_epi<R, EPI_EDENS>, smem);
            k_xinv_epi<R, EPI_EDENS><<<(unsigned)blocks, threads, smem, st>>>(pl.s1, pl.pitch, plan, tP, g, scale, m,
                                                                              ms, tl, ep, nbr);
            break;
    }
    MAF_LAUNCH_CHECK();
    if (marks) marks->mark(st, "x_inv_local");
}

template DemagPlan<float> Demag::plan<float>(cudaStream_t);
template DemagPlan<double> Demag::plan<double>(cudaStream_t);
template void Demag::forward_conv<float>(const float*, const MsInfo&, cudaStream_t, PassMarks*);
template void Demag::forward_conv<double>(const double*, const MsInfo&, cudaStream_t, PassMarks*);
template void Demag::inverse_x_epilogue<float>(const float*, const MsInfo&, const TermList&, const EpilogueArgs&,
                                               cudaStream_t, int*, PassMarks*);
template void Demag::inverse_x_epilogue<double>(const double*, const MsInfo&, const TermList&, const EpilogueArgs&,
                                                cudaStream_t, int*, PassMarks*);

// ---------------------------------------------------------------------------
// field evaluation of a term list
// ---------------------------------------------------------------------------
Demag* term_demag(Term& t, const MeshDims& md, cudaStream_t st) {
    if (t.demag_pbc() && !(t.demag && t.demag_mesh == md)) {
        // DemagFieldPBC takes its mesh from the state: plan it on first use
        t.demag = std::make_unique<Demag>(md, st, nullptr, true);
        t.demag_mesh = md;
    }
    if (!(t.demag_mesh == md)) throw Error(1, "DemagField mesh differs from the state's mesh");
    return t.demag.get();
}

template <typename R>
void eval_terms(const std::vector<Term*>& terms, const MeshDims& md, const R* m, const MsInfo& ms,
                const EpilogueArgs& ep_in, cudaStream_t st, DevBuf& scratch, double* energy_out,
                PassMarks* marks) {
    if (terms.empty()) throw Error(1, "no field terms");
    if ((int)terms.size() > kMaxTerms) throw Error(1, "too many field terms (max 8)");
    TermList tl;
    Demag* demag = nullptr;
    for (Term* t : terms) {
        if (t->kind == TK_DEMAG) {
            if (demag) throw Error(1, "at most one DemagField per term list");
            demag = term_demag(*t, md, st);
        }
        if (t->field_cells && t->field_cells != md.N())
            throw Error(1, "field-term parameter array does not match the state's mesh");
        if (t->kind == TK_BULKDMI && (md.nx < 2 || md.ny < 2 || md.nz < 2))
            throw Error(1, "BulkDMIExchangeField needs at least 2 cells along x, y and z");
        tl.t[tl.n++] = t->desc();
    }
    EpilogueArgs ep = ep_in;
    int nblocks = 0;
    if (ep.kind == EPI_EDENS || ep.kind == EPI_EGRAD) {
        // upper bound of CTAs for the partial sums
        const int64_t maxb = std::max<int64_t>(md.N(), (int64_t)sm_count() * 8) + 1;
        scratch.ensure(sizeof(double) * (maxb + 1));
        ep.partials = scratch.as<double>();
    }
    if (demag) {
        if (marks) marks->mark(st, "start");
        demag->forward_conv<R>(m, ms, st, marks);
        demag->inverse_x_epilogue<R>(m, ms, tl, ep, st, &nblocks, marks);
    } else if (const int run = md.N() < (int64_t)INT32_MAX ? run_mode(md.geom(), m, ms, tl, ep, 2) : 0) {
        // scalar parameters: runs of cells with per-launch term constants
        // (no division in the cell loop); four cells per run where the rows allow it, two
        // for the energies (the energy and the field of four do not fit the registers)
        const Geom g = md.geom();
        prepare_run(tl, g, ms);
        // (and with the next Runge-Kutta stage)
        const bool four = run == 1 && g.nx % 4 == 0 && (ep.kind == EPI_H || (ep.kind == EPI_LLG && !ep.llg.next.out64));
        const int nruns = (int)(md.N() / (four ? 4 : run == 1 ? 2 : 1));
        const int threads = 256;
        const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(nruns, threads), (int64_t)sm_count() * 16);
        nblocks = (int)blocks;
        if (marks) marks->mark(st, "start");
#define MAF_LOCAL_RUN(EPI)                                                                                        \
    do {                                                                                                         \
        if (run == 1)                                                                                            \
            k_local_run<R, EPI, 2, false, true><<<blocks, threads, 0, st>>>(g, m, ms, tl, ep, nruns);                  \
        else if (run == 2)                                                                                       \
            k_local_run<R, EPI, 1, false, true><<<blocks, threads, 0, st>>>(g, m, ms, tl, ep, nruns);                  \
        else                                                                                                     \
            k_local_run<R, EPI, 1, true, true><<<blocks, threads, 0, st>>>(g, m, ms, tl, ep, nruns);                   \
    } while (0)
        if (four && ep.kind == EPI_H)
            k_local_run<R, EPI_H, 4, false, false><<<blocks, threads, 0, st>>>(g, m, ms, tl, ep, nruns);
        else if (four)
            k_local_run<R, EPI_LLG, 4, false, false><<<blocks, threads, 0, st>>>(g, m, ms, tl, ep, nruns);
        else if (ep.kind == EPI_H)
            MAF_LOCAL_RUN(EPI_H);
        else if (ep.kind == EPI_LLG)
            MAF_LOCAL_RUN(EPI_LLG);
        else if (ep.kind == EPI_EGRAD)
            MAF_LOCAL_RUN(EPI_EGRAD);
        else
            MAF_LOCAL_RUN(EPI_EDENS);
#undef MAF_LOCAL_RUN
        MAF_LAUNCH_CHECK();
        if (marks) marks->mark(st, "local");
    } else {
        const int threads = 256;
        const int64_t blocks = std::min<int64_t>(ceil_div(md.N(), threads), (int64_t)sm_count() * 8);
        nblocks = (int)blocks;
        const Geom g = md.geom();
        if (marks) marks->mark(st, "start");
        switch (ep.kind) {
            case EPI_H: k_local_epi<R, EPI_H><<<(unsigned)blocks, threads, 0, st>>>(g, m, ms, tl, ep); break;
            case EPI_LLG: k_local_epi<R, EPI_LLG><<<(unsigned)blocks, threads, 0, st>>>(g, m, ms, tl, ep); break;
            case EPI_EGRAD: k_local_epi<R, EPI_EGRAD><<<(unsigned)blocks, threads, 0, st>>>(g, m, ms, tl, ep); break;
            default: k_local_epi<R, EPI_EDENS><<<(unsigned)blocks, threads, 0, st>>>(g, m, ms, tl, ep); break;
        }
        MAF_LAUNCH_CHECK();
        if (marks) marks->mark(st, "local");
    }
    if (ep.kind == EPI_EDENS || ep.kind == EPI_EGRAD) {
        if (ep_in.npartials) {  // the caller sums them
            *ep_in.npartials = nblocks;
            return;
        }
        double* dst = ep.partials + nblocks;
        k_sum_partials<<<1, 256, 0, st>>>(ep.partials, nblocks, dst);
        MAF_LAUNCH_CHECK();
        double e = 0;
        MAF_CUDA(cudaMemcpyAsync(&e, dst, sizeof(double), cudaMemcpyDeviceToHost, st));
        MAF_CUDA(cudaStreamSynchronize(st));
        if (energy_out) *energy_out = e * md.dx * md.dy * md.dz;
    }
}

template void eval_terms<float>(const std::vector<Term*>&, const MeshDims&, const float*, const MsInfo&,
                                const EpilogueArgs&, cudaStream_t, DevBuf&, double*, PassMarks*);
template void eval_terms<double>(const std::vector<Term*>&, const MeshDims&, const double*, const MsInfo&,
                                 const EpilogueArgs&, cudaStream_t, DevBuf&, double*, PassMarks*);

}  // namespace mafb
