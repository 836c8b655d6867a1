// Newell demag tensor on the zero-padded grid, FP64.
//
// Follows magnumaf/src/field_terms/micro/demag_field.cpp:20-121 term for term:
// f() and g() keep the reference's expression order, Nxx/Nxy sum the 27
// stencil values in the reference's order, and the index wrap
// j = (i + P/2) % P - P/2 and the component mapping are the same.  This file
// is compiled with -fmad=false so that no multiply-add is contracted, which
// keeps the rounding of the (cancellation-prone) 27-point sums close to the
// reference's host build.  Only the elementary functions differ (CUDA's
// asinh/atan instead of the host libm), which perturbs far-field entries at
// the level of their own cancellation noise.
#include <algorithm>

#include "engine.hpp"

namespace mafb {

__device__ double newell_f(double x, double y, double z) {
    x = fabs(x);
    y = fabs(y);
    z = fabs(z);
    const double R = sqrt(x * x + y * y + z * z);
    const double xx = x * x;
    const double yy = y * y;
    const double zz = z * z;
    double result = 1.0 / 6.0 * (2.0 * xx - yy - zz) * R;
    if (xx + zz > 0) result += y / 2.0 * (zz - xx) * asinh(y / (sqrt(xx + zz)));
    if (xx + yy > 0) result += z / 2.0 * (yy - xx) * asinh(z / (sqrt(xx + yy)));
    if (x * R > 0) result += -x * y * z * atan(y * z / (x * R));
    return result;
}

__device__ double newell_g(const double x, const double y, double z) {
    z = fabs(z);
    const double R = sqrt(x * x + y * y + z * z);
    const double xx = x * x;
    const double yy = y * y;
    const double zz = z * z;
    double result = -x * y * R / 3.0;
    if (xx + yy > 0) result += x * y * z * asinh(z / (sqrt(xx + yy)));
    if (yy + zz > 0) result += y / 6.0 * (3.0 * zz - yy) * asinh(x / (sqrt(yy + zz)));
    if (xx + zz > 0) result += x / 6.0 * (3.0 * zz - xx) * asinh(y / (sqrt(xx + zz)));
    if (z * R > 0) result += -(z * z * z) / 6.0 * atan(x * y / (z * R));
    if (y * R != 0) result += -z * yy / 2.0 * atan(x * z / (y * R));
    if (x * R != 0) result += -z * xx / 2.0 * atan(y * z / (x * R));
    return result;
}

template <bool IS_F>
__device__ double newell_27(int ix, int iy, int iz, double dx, double dy, double dz) {
    const double x = dx * ix;
    const double y = dy * iy;
    const double z = dz * iz;
    auto F = [](double a, double b, double c) { return IS_F ? newell_f(a, b, c) : newell_g(a, b, c); };
    double result = 8.0 * F(x, y, z) - 4.0 * F(x + dx, y, z) - 4.0 * F(x - dx, y, z) - 4.0 * F(x, y + dy, z) -
                    4.0 * F(x, y - dy, z) - 4.0 * F(x, y, z + dz) - 4.0 * F(x, y, z - dz) + 2.0 * F(x + dx, y + dy, z) +
                    2.0 * F(x + dx, y - dy, z) + 2.0 * F(x - dx, y + dy, z) + 2.0 * F(x - dx, y - dy, z) +
                    2.0 * F(x + dx, y, z + dz) + 2.0 * F(x + dx, y, z - dz) + 2.0 * F(x - dx, y, z + dz) +
                    2.0 * F(x - dx, y, z - dz) + 2.0 * F(x, y + dy, z + dz) + 2.0 * F(x, y + dy, z - dz) +
                    2.0 * F(x, y - dy, z + dz) + 2.0 * F(x, y - dy, z - dz) - 1.0 * F(x + dx, y + dy, z + dz) -
                    1.0 * F(x + dx, y + dy, z - dz) - 1.0 * F(x + dx, y - dy, z + dz) -
                    1.0 * F(x + dx, y - dy, z - dz) - 1.0 * F(x - dx, y + dy, z + dz) -
                    1.0 * F(x - dx, y + dy, z - dz) - 1.0 * F(x - dx, y - dy, z + dz) - 1.0 * F(x - dx, y - dy, z - dz);
    return -result / (4.0 * 3.14159265358979323846 * dx * dy * dz);
}

__device__ __forceinline__ double newell_comp(int comp, int j0, int j1, int j2, double dx, double dy, double dz) {
    switch (comp) {
        case 0: return newell_27<true>(j0, j1, j2, dx, dy, dz);    // xx
        case 1: return newell_27<false>(j0, j1, j2, dx, dy, dz);   // xy
        case 2: return newell_27<false>(j0, j2, j1, dx, dz, dy);   // xz
        case 3: return newell_27<true>(j1, j2, j0, dy, dz, dx);    // yy
        case 4: return newell_27<false>(j1, j2, j0, dy, dz, dx);   // yz
        default: return newell_27<true>(j2, j0, j1, dz, dx, dy);   // zz
    }
}

// The reference's setup_N value at every padded index.
__global__ void k_newell(double* __restrict__ out, int comp, int Px, int Py, int Pz, double dx, double dy, double dz) {
    const int64_t total = (int64_t)Px * Py * Pz;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int i0 = (int)(idx % Px);
        const int i1 = (int)((idx / Px) % Py);
        const int i2 = (int)(idx / ((int64_t)Px * Py));
        const int j0 = (i0 + Px / 2) % Px - Px / 2;
        const int j1 = (i1 + Py / 2) % Py - Py / 2;
        const int j2 = (i2 + Pz / 2) % Pz - Pz / 2;
        out[idx] = newell_comp(comp, j0, j1, j2, dx, dy, dz);
    }
}

// The stored components (blockIdx.y) at the offsets 0 <= j < (o0, o1, o2) only.  The
// parity-exact tensor that the spectral pipeline transforms is even or odd along each
// axis, so these entries carry all of it (fields.cu, tensor_odd).  The kernel is bound on
// the FP64 pipe (27 evaluations of f or g with asinh and atan per entry) or, for small
// meshes, on their chain: a CTA takes 32 entries, lane = entry, and each of its 9 warps
// makes 3 of the 27 evaluations (so the offsets are uniform in a warp); the terms are added
// in newell_27's order, so the entries are the same bit for bit.  A new tensor (create,
// allocation and transforms included) with a thread for all 27, a warp per entry (lane =
// evaluation) and this split: 33 x 50 x 1 429, 373, 370 us; 400 x 400 x 1 1117, 1265, 858;
// 200 x 120 x 10 3118, 2762, 1952 (the evaluations of one offset branch alike).
struct NewellComps {
    int c[6];
};
constexpr int kOctWarps = 9;
// newell_27's order: centre, the 6 faces, the 12 edges, the 8 corners
__constant__ signed char kStencil[27][3] = {
    {0, 0, 0},   {1, 0, 0},  {-1, 0, 0},  {0, 1, 0},   {0, -1, 0},  {0, 0, 1},  {0, 0, -1},
    {1, 1, 0},   {1, -1, 0}, {-1, 1, 0},  {-1, -1, 0}, {1, 0, 1},   {1, 0, -1}, {-1, 0, 1},
    {-1, 0, -1}, {0, 1, 1},  {0, 1, -1},  {0, -1, 1},  {0, -1, -1}, {1, 1, 1},  {1, 1, -1},
    {1, -1, 1},  {1, -1, -1}, {-1, 1, 1}, {-1, 1, -1}, {-1, -1, 1}, {-1, -1, -1}};

__global__ void __launch_bounds__(32 * kOctWarps)
    k_newell_octant(double* __restrict__ out, NewellComps comps, int o0, int o1, int o2, double dx, double dy, double dz) {
    __shared__ double terms[27][32];
    const int64_t total = (int64_t)o0 * o1 * o2;
    const int comp = comps.c[blockIdx.y], lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    const bool is_f = comp == 0 || comp == 3 || comp == 5;
    for (int64_t base = (int64_t)blockIdx.x * 32; base < total; base += (int64_t)gridDim.x * 32) {
        const int64_t idx = base + lane < total ? base + lane : total - 1;
        const int j0 = (int)(idx % o0);
        const int j1 = (int)((idx / o0) % o1);
        const int j2 = (int)(idx / ((int64_t)o0 * o1));
        // newell_comp's mapping of the axes
        int ix = j0, iy = j1, iz = j2;
        double hx = dx, hy = dy, hz = dz;
        if (comp == 2) {
            iy = j2, iz = j1, hy = dz, hz = dy;
        } else if (comp == 3 || comp == 4) {
            ix = j1, iy = j2, iz = j0, hx = dy, hy = dz, hz = dx;
        } else if (comp == 5) {
            ix = j2, iy = j0, iz = j1, hx = dz, hy = dx, hz = dy;
        }
        for (int t = warp; t < 27; t += kOctWarps) {
            const double x = hx * ix + kStencil[t][0] * hx, y = hy * iy + kStencil[t][1] * hy,
                         z = hz * iz + kStencil[t][2] * hz;
            const double w = t == 0 ? 8.0 : t < 7 ? -4.0 : t < 19 ? 2.0 : -1.0;
            terms[t][lane] = w * (is_f ? newell_f(x, y, z) : newell_g(x, y, z));
        }
        __syncthreads();
        if (warp == 0 && base + lane < total) {
            double sum = terms[0][lane];
            for (int t = 1; t < 27; ++t) sum += terms[t][lane];
            out[blockIdx.y * total + base + lane] = -sum / (4.0 * 3.14159265358979323846 * hx * hy * hz);
        }
        __syncthreads();
    }
}

static unsigned newell_blocks(int64_t total) {
    return (unsigned)std::min<int64_t>(ceil_div(total, 128), (int64_t)sm_count() * 64);
}

void newell_component(double* out, int comp, const MeshDims& md, int Px, int Py, int Pz, cudaStream_t st) {
    k_newell<<<newell_blocks((int64_t)Px * Py * Pz), 128, 0, st>>>(out, comp, Px, Py, Pz, md.dx, md.dy, md.dz);
    MAF_LAUNCH_CHECK();
}

void newell_octants(double* out, const int* comps, int ncomp, const MeshDims& md, int o0, int o1, int o2,
                    cudaStream_t st) {
    NewellComps c = {};
    for (int i = 0; i < ncomp; ++i) c.c[i] = comps[i];
    const int64_t blocks = std::min<int64_t>(ceil_div((int64_t)o0 * o1 * o2, 32), (int64_t)sm_count() * 256);
    k_newell_octant<<<dim3((unsigned)blocks, (unsigned)ncomp), 32 * kOctWarps, 0, st>>>(out, c, o0, o1, o2, md.dx, md.dy,
                                                                                     md.dz);
    MAF_LAUNCH_CHECK();
}

}  // namespace mafb
