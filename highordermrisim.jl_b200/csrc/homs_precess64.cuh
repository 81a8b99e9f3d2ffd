// Free precession of a whole segment in FP64, in parallel over time and spins
// (homs_precess64.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "homs_common.cuh"
#include "homs_fp64mma.cuh"

namespace homs {

// Spin table of a phantom: per spin the 16 phase coefficients (basis terms
// 1..15, dw/(2 pi)) and -log2(e)/T2, padded with zeros to whole 32-spin chunks.
size_t precess64_table_bytes(int64_t ns);
cudaError_t precess64_table(const double *x, const double *y, const double *z, const double *dw, const double *T2,
                            int64_t ns, void *table, cudaStream_t stream);

// How a segment is cut (homs_fp64mma.cuh); its partial sums take at most 256 MB.
CoilCut precess64_cut(int64_t ns, int32_t nc, int64_t nsamples);

// Upper bound of what the launches of a run of `nadc` samples take beside the spin
// table: prefix table and partial sums.
size_t precess64_run_bytes(int64_t ns, int32_t nc, int64_t nadc);

struct Precess64Args {
    int64_t ns, nsamples;
    int32_t nc;
    uint32_t method;
    const void *table;             // precess64_table
    const double *prefix;          // prefix table of the segment (split_prefix_launch)
    const cplx<double> *csm_rows;  // [ns][nc]
    const double *T1, *T2, *rho;
    cplx<double> *xy;  // state at the segment's start, replaced by the state at its end
    double *mz;
    cplx<double> *partial;  // cut.partial_bytes
    cplx<double> *sig;      // sample 0 of coil 0; coil stride ldsig
    int64_t ldsig;
};
// The segment's signal and its final state.  ev_start / ev_stop (may be NULL)
// bracket the main kernel's launches; *launches counts kernels.
cudaError_t precess64_run(const Precess64Args &a, const CoilCut &cut, cudaEvent_t ev_start,
                          cudaEvent_t ev_stop, unsigned ev_flags, int64_t *launches, cudaStream_t stream);

}  // namespace homs
