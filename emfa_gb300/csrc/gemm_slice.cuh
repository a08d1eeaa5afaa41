// FP64- and FP32-accurate complex products on the tensor cores (gemm_slice.cu).
#pragma once
#include "gemm.cuh"

namespace emfa {

// `rows` rows of Z (n columns) as planes of signed 8-bit digits held in FP16
// (eight for complex128, four for complex64) and one of magnitudes, each rows x
// 2n (re, im interleaved), rows ldk halves apart, and a power-of-two scale per row.
struct SlicePlanes {
    const __half* d = nullptr;   // [planes][rows][ldk]
    const int* ex = nullptr;     // [rows] scales; SLICE_NONFINITE for a row with an infinity or NaN
    const void* Z = nullptr;     // the rows themselves
    size_t ldz = 0;
    int n = 0, rows = 0;
    size_t ldk = 0;
};

// FP64: whether a block of nrhs products of n unknowns is worth the planes; built:
// the planes exist already (a Krylov solve splits Z once).
bool slice_worthwhile(Ctx* c, int n, int nrhs, bool built, cudaStream_t st);
// Splits Z into workspace `slot` of the context.  EMFA_ERR_OOM: no room, the
// caller takes the CUDA-core product.
emfa_status_t slice_prepare(Ctx* c, int slot, const void* Z, size_t ldz, int n, SlicePlanes* out, cudaStream_t st);
// Y = Z X (complex128, RHS-major) with scratch from workspace `slot`; the error
// word of the pipeline's bounded waits turns Y into NaN, and slice_check tells
// (it reads the word of a solve's products, which slice_prepare zeroes)
emfa_status_t slice_apply(Ctx* c, int slot, const SlicePlanes& p, const void* X, int nrhs, void* Y, cudaStream_t st);
emfa_status_t slice_check(Ctx* c, cudaStream_t st);
// after a solve: gives its planes and scratch back where they are large
void slice_release(Ctx* c);
// The error word of single products.  It is not read after a product, which
// would wait for it: the product tells a page-locked word, and the next call
// that looks (slice_report: emfa_ctx_synchronize, emfa_matvec, emfa_residual)
// returns EMFA_ERR_TIMEOUT once and has the word zeroed.
emfa_status_t slice_word(Ctx* c, int** err, cudaStream_t st);
emfa_status_t slice_report(Ctx* c);
// one product in precision prec: splits Z, multiplies; false in *done where the
// CUDA cores are the better path or there is no room
emfa_status_t slice_matvec(Ctx* c, int prec, const void* Z, size_t ldz, const void* X, int n, int nrhs, void* Y,
                           cudaStream_t st, bool* done);

}  // namespace emfa
