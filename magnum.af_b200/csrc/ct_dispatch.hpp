// Compile-time specialised demag passes (fields_ct.cu).  Each returns false when
// no specialisation exists for the transform length; the caller then runs the
// generic kernel of fields.cu.  The transform may be longer than twice the mesh:
// n_in or n_out of the y passes below L/2, nz (ny) planes (rows) of a z (y)
// convolution of length L with ny = Py/2, and rows of fewer than Px/2 cells.
#pragma once
#include "engine.hpp"

namespace mafb {

template <typename R>
bool ct_xfwd(const R* in, int n_in, int64_t rows, int64_t rows_pc, const R* msf, R ms, cplx_t<R>* out, int pitch,
             int Px, Twiddles& tw, cudaStream_t st);
template <typename R, int DIR>
bool ct_cols(const cplx_t<R>* in, cplx_t<R>* out, int L, int n_in, int n_out, int ncols, int64_t in_si, int64_t out_si,
             int64_t in_sbat, int64_t out_sbat, int nbat, Twiddles& tw, const TuneChoice& tc, cudaStream_t st);
template <typename R>
bool ct_convz(cplx_t<R>* S, const R* Nred, int nz, int L, int ny, int nxh, int pitch, Twiddles& tw,
              const TuneChoice& tc, cudaStream_t st);
template <typename R>
bool ct_convy(cplx_t<R>* S, const R* Nred, int ny, int L, int nxh, int pitch, Twiddles& tw, cudaStream_t st);
// (the lengths are instantiated in three groups G)
template <typename R, int G>
bool ct_xinv_group(const cplx_t<R>* S1, int pitch, int Px, Twiddles& tw, const Geom& g, R scale, const R* m,
                   const MsInfo& ms, const TermList& tl, const EpilogueArgs& ep, const TuneChoice& tc, cudaStream_t st,
                   int* nblocks);
template <typename R>
bool ct_xinv(const cplx_t<R>* S1, int pitch, int Px, Twiddles& tw, const Geom& g, R scale, const R* m,
             const MsInfo& ms, const TermList& tl, const EpilogueArgs& ep, const TuneChoice& tc, cudaStream_t st,
             int* nblocks) {
    return ct_xinv_group<R, 0>(S1, pitch, Px, tw, g, scale, m, ms, tl, ep, tc, st, nblocks) ||
           ct_xinv_group<R, 1>(S1, pitch, Px, tw, g, scale, m, ms, tl, ep, tc, st, nblocks) ||
           ct_xinv_group<R, 2>(S1, pitch, Px, tw, g, scale, m, ms, tl, ep, tc, st, nblocks);
}

// Batched compile-time passes: one launch runs the (item, tile) pairs of a
// device work table, every item of a launch with the same transform length
// (the ensembles' batched steps; the tile bodies are those of the per-state
// kernels, so an item's results equal its per-state pass bit for bit).
template <typename R> struct CtXfwdItem {
    const R* in;
    int n_in;
    int64_t rows;
    R ms;
    cplx_t<R>* out;
    int pitch;
};
template <typename R> struct CtConvyItem {
    cplx_t<R>* S;
    const R* Nred;
    int ny, nxh, pitch;
};
template <typename R> struct CtXinvItem {
    const cplx_t<R>* S1;
    int pitch;
    Geom g;
    R scale;
    const R* m;
    MsInfo ms;
    TermList tl;
    EpilogueArgs ep;  // EPI_LLG
    int run;  // run_mode
};
// pass: 0 x forward (L = Px / 2), 1 y convolution (L = Py), 2 x inverse (L = Px / 2).
// Rows (x passes) or kx columns (y convolution) per tile; 0: no compile-time kernel.
template <typename R> int ct_batch_tile(int pass, int L);
// The twiddle table the pass's kernel of length L reads (created on first use).
template <typename R> const void* ct_batch_twiddles(int pass, int L, Twiddles& tw);
// The launch class of an x-inverse item: `run` when its rows go in runs of that many cells,
// 0 for the other forms (the `run` argument of ct_batch_xinv).
template <typename R> int ct_batch_xinv_class(const CtXinvItem<R>& it, int run);
// The run-epilogue flag and constants of an x-inverse item (as the per-state launch prepares
// them for runs of `run` cells).
template <typename R> void ct_batch_xinv_prepare(CtXinvItem<R>& it, int run);
// Launches; tw from ct_batch_twiddles, twP the length-Px table (Twiddles::get).
template <typename R>
void ct_batch_xfwd(const CtXfwdItem<R>* items, const int2* work, int nwork, int L, const void* tw, const void* twP,
                   cudaStream_t st);
template <typename R>
void ct_batch_convy(const CtConvyItem<R>* items, const int2* work, int nwork, int L, bool rag, const void* tw,
                    cudaStream_t st);
template <typename R, int G>
bool ct_batch_xinv_group(const CtXinvItem<R>* items, const int2* work, int nwork, int L, int run, const void* tw,
                         const void* twP, cudaStream_t st);
template <typename R>
void ct_batch_xinv(const CtXinvItem<R>* items, const int2* work, int nwork, int L, int run, const void* tw,
                   const void* twP, cudaStream_t st) {
    if (nwork <= 0) return;
    ct_batch_xinv_group<R, 0>(items, work, nwork, L, run, tw, twP, st) ||
        ct_batch_xinv_group<R, 1>(items, work, nwork, L, run, tw, twP, st) ||
        ct_batch_xinv_group<R, 2>(items, work, nwork, L, run, tw, twP, st);
}

}  // namespace mafb
