// Tensor-core (tcgen05) Gram detection: entry points used by the detector.
#pragma once

#include "apsm_host.hpp"

namespace apsm {
void gram_workspace_free(GramWorkspace* g);

// out[u][s] = wL <w_u, x_s> + the sums part[split][u][s] in order, u < users <= kLinearUsers.
constexpr int kLinearUsers = 16;
cudaError_t launch_linear_part(const float* xs, int Dp, int D, const float* w, float wL, const float* part, int splits,
                               int users, int n_samples, float* out, size_t out_stride, cudaStream_t s);

// TF32 split form with the data tile in tensor memory (kernels_gram_tmem.cu).
constexpr int kGramTmemChunk = 128; // dictionary rows per chunk
struct GramTmemArgs {
    const float* rows;    // data rows (n_samples x Dp, FP32)
    const uint8_t* b_ops; // dictionary chunks of kGramTmemChunk rows, canonical K-major, hi | lo
    const float* xd;      // per chunk: norms and coefficients (gram_tmem_data_floats)
    float* part;          // splits x users x n_samples partial sums
    int* err;
    int n_samples, users, Kp, Dp;
    int chunks_per_split, n_chunks;
    float ewl2; // ew * log2(e)
    unsigned long long wait_ns; // limit of the bounded waits
};
size_t gram_tmem_data_floats(int users); // floats of one chunk's data
// Writes the chunk data (dictionary norms dn, coefficients a: users x a_stride, M rows) and runs the tiles.
cudaError_t launch_gram_tmem(const GramTmemArgs& g, const float* dn, const float* a, size_t a_stride, int M, float wG,
                             float* xd, int n_tiles, int splits, cudaStream_t s);
} // namespace apsm

// Detection of the packed data rows h->xs (2S rows) with the Gram form
// selected by h->cfg.detect_mode; soft outputs to d_out (users x 2S floats).
apsm_status detect_gram(apsm_detector* h, uint32_t S, float* d_out, cudaStream_t s);
// Expiry of a bounded wait in the last Gram detection of h (read after its
// stream synchronised): APSM_ERR_CUDA once, then cleared.
apsm_status detect_gram_check(apsm_detector* h);
