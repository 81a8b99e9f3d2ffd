// Free precession of a run of blocks in FP32 (homs_precess32.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "homs_common.cuh"
#include "homs_fp64mma.cuh"

namespace homs {

// Node table of a sequence and method: per node the 16 field coefficients (zero
// where the method leaves a term out, the nominal gradients in place of the
// first order where that is off), the interval that ends at the node, the
// block time at the node (`tp`, summed in FP32 node by node from the block's
// start) and the node's ADC and block-end flags.
size_t precess32_node_bytes(int64_t nnodes);
cudaError_t precess32_nodes(const SeqDev<float> &q, uint32_t method, const float *tp, void *nodes, cudaStream_t stream);

// A launch round: intervals [n_lo, n_hi) of one run, at most
// precess32_max_samples samples and precess32_max_blocks blocks.
int64_t precess32_max_samples(int64_t ns);
int64_t precess32_max_blocks(int64_t ns);
struct Precess32Args {
    PhantomDev<float> phantom;  // csm: spin-major rows [ns][nc]
    StateDev<float> state;      // xy, z, acc: at n_lo, replaced by their values at n_hi
    const void *nodes;          // precess32_nodes, of nnodes nodes
    int64_t nnodes;
    int64_t n_lo, n_hi;
    int block_start;  // n_lo is the first node of a block
    int64_t nsamples;
    int32_t nblocks;  // blocks that have intervals in the round
    uint32_t method;
    double gamma;
    void *work;              // precess32_work_bytes
    cplx<double> *partial;   // cut.partial_bytes
    cplx<float> *sig;        // the round's first sample of coil 0; coil stride ldsig
    int64_t ldsig;
};
size_t precess32_work_bytes(int64_t ns, int64_t nsamples, int32_t nblocks);
CoilCut precess32_cut(int64_t ns, int32_t nc, int64_t nsamples);
// Upper bound of what the launches of a run take: node table, a round's work area and
// partial sums.  block_adc: the most samples of a block.
size_t precess32_run_bytes(int64_t ns, int32_t nc, int64_t nnodes, int64_t nadc, int64_t nblocks, int64_t block_adc);
cudaError_t precess32_run(const Precess32Args &a, const CoilCut &cut, cudaEvent_t ev_start, cudaEvent_t ev_stop,
                          unsigned ev_flags, int64_t *launches, cudaStream_t stream);

}  // namespace homs
