// Launch wrappers of the Runge-Kutta / normalisation kernels (llg.cu).
#pragma once
#include "common.cuh"

namespace mafb {

struct KList {
    const double* k[8] = {};
    double c[8] = {};
    int n = 0;
};

void rk_combine(const double* m, const KList& kl, double* out64, float* out32, int64_t n, cudaStream_t st);
// Candidate m and the error norm: *err receives
// the NaN-propagating max (device-accessible memory).  partials: rk_finalize_blocks() doubles
// and, behind them, one zeroed word, the block counter, which every launch leaves zero.
int rk_finalize_blocks();
void rk_finalize(const double* m, const KList& kb, const KList& ke, int form, double atol, double rtol, double* mcand,
                 int norm_mode, int64_t N, double* partials, double* err, cudaStream_t st);
void normalize_m(double* m, int64_t N, int mode, unsigned long long* zero_count_dev, cudaStream_t st);
void ms_field_from_m(const double* m, double Ms, double* msf, float* msf32, int64_t N, cudaStream_t st);
// partial-sum blocks of mean_m (its scratch needs 4 per block; out_dev may sit behind them)
int mean_m_blocks();
void mean_m(const double* m, int64_t N, double* scratch, double* out_dev, cudaStream_t st);
void f32_to_f64(const float* a, double* b, int64_t n, cudaStream_t st);
void thermal_field(double* out, int64_t N, double sigma, unsigned long long seed, unsigned member,
                   unsigned long long index, cudaStream_t st);
// LBFGS vector operations; scratch needs red_blocks() + 1 doubles; the reductions synchronise
int red_blocks();
double dot_host(const double* a, const double* b, int64_t n, double* scratch, cudaStream_t st);
double maxabs_host(const double* a, int64_t n, double* scratch, cudaStream_t st);
void axpby(double* out, double a, const double* x, double b, const double* y, int64_t n, cudaStream_t st);
// Device-resident LBFGS iteration kernels (no host synchronisation; llg.cu).  part:
// 6 red_blocks() doubles; counter: one zeroed word that every launch leaves zero.
struct LbRecur {
    const double* q_in = nullptr;   // q of the previous step, or the gradient
    double* q = nullptr;
    const double* u = nullptr;      // vector added with the coefficient formed from *d
    double* d = nullptr;            // in: the dot product of the previous step; out: w . q
    const double* w = nullptr;
    double rho = 0.0;
    const double* alpha_in = nullptr;
    double* alpha_out = nullptr;
    int scaled = 0;
    double scale = 1.0;
    double* dir = nullptr;          // -q
    const double* x = nullptr;      // copied to x_copy
    double* x_copy = nullptr;
    double* g_copy = nullptr;       // copy of q_in
};
void lb_recur(const LbRecur& a, int64_t n, double* part, unsigned* counter, cudaStream_t st);
// The recursion over k stored pairs (s[0..k), y[0..k), oldest first) in one launch: dir = -q,
// *d = grad . q, the copies as above; false (nothing done) when n is too large for it.
struct LbLoop {
    const double* grad = nullptr;
    const double* s[5] = {};
    const double* y[5] = {};
    double rho[5] = {};
    int k = 0;
    double scale = 1.0;
    const double* x = nullptr;
    double* x_copy = nullptr;
    double* g_copy = nullptr;
    double* dir = nullptr;
    double* d = nullptr;
};
bool lb_loop(const LbLoop& a, int64_t n, cudaStream_t st);
void lb_slope(const double* g, const double* s, int64_t n, const double* e, int ne, double* part, unsigned* counter,
              double* out, cudaStream_t st);
void lb_pair(const double* x, const double* x_old, const double* g, const double* g_old, double* s, double* y,
             int64_t n, double* part, unsigned* counter, double* out, cudaStream_t st);
void normalize_combine(double* m, const double* wa, double stp, const double* s, int64_t N, cudaStream_t st);
// string method: sum (a-b)^2 over n values (synchronises), out = a + (c1 (b - a)) / c2
double sqdiff_host(const double* a, const double* b, int64_t n, double* scratch, cudaStream_t st);
void lerp(double* out, const double* a, const double* b, double c1, double c2, int64_t n, cudaStream_t st);
// *c += 1 on the device (the step counter of a captured stochastic step)
void inc_counter(unsigned long long* c, cudaStream_t st);

}  // namespace mafb
