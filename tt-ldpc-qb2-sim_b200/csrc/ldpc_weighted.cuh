// Weighted Approximate-Min* decoder with a hand-written adjoint (training path).
//
// Row update of the layered decoder with per-iteration t, per-protograph-edge-class c parameters
// (scale alpha[t][c], offset beta[t][c]):
//     q_e = L_v - r_e
//     m_e = Approximate-Min* magnitude of edge e (as in the plain decoder: the recursive min* over the
//           row's other edges, ldpc_decoder_core.h:176-201)
//     r_e = sign_e * relu(alpha[t][c_e] * m_e - beta[t][c_e]),   sign_e = parity(q) * sign(q_e)
//     L_v = q_e + r_e
// With alpha = 1 and beta = 0 every value equals the plain fp32 decoder's bit for bit.  T iterations
// are unrolled with no early stop (the training graph); the posteriors after every iteration (or after
// the last) are the outputs.  The forward pass keeps q of every row of the last iterations, as many as
// fit the memory that checkpoints every ckpt_every iterations would take; the backward pass walks them
// back layer by layer (adjoints of L in shared memory, of r in global memory, parameter gradients
// reduced per warp into shared memory) and runs the iterations before them again from checkpoints of
// the state.
#pragma once
#include <cstddef>
#include <cstdint>
#include <string>

#include <cuda_runtime.h>

#include "ldpc_qc.cuh"

namespace ldpcb200 {

constexpr int W_MAX_ITER = 64;
constexpr int W_MAX_CLASSES = 64;
constexpr size_t W_ALIGN = 256;  // the workspace's arrays start at a multiple of this

// Edge slots of one iteration (the weight table's rows of qc_edge_slot), and the pairs of one
// message-shaped array (edges 2k and 2k+1 of a row share a pair, an odd degree's last pair half empty).
__host__ __device__ constexpr int wslots(int D) { return 4 * QC_DEG_LOW + 8 * D; }
__host__ __device__ constexpr int wedge_pairs(int Z, int D) { return Z * (4 * ((QC_DEG_LOW + 1) / 2) + 8 * ((D + 1) / 2)); }

struct WParams {
    int32_t edge[QC_LAYERS][QC_DMAX];  // block offset + circulant shift of edge e of layer l
    int32_t edge_class[QC_LAYERS][QC_DMAX];
    int32_t n_vars, n_tx;           // N, N - P
    int32_t n_iter, n_classes, post_all;
    int32_t row_uniform;            // 1: every edge of a layer has one class
    int32_t n_frames;
    int32_t keep;                   // iterations at the end whose q the forward pass keeps (weighted_plan)
    int32_t n_slots;                // message-adjoint slots, the most CTAs of the backward kernel
    size_t off_ckpt, off_gr, off_save, off_used;  // workspace offsets (elements); the stash is at 0
    // arrays of the kernel's real type (float, or double for adjoint checks)
    const void* llr;       // [B][n_tx]
    const void* alpha;     // [T][C]
    const void* beta;      // [T][C]
    void* post;            // [T or 1][B][N]
    void* stash;           // [B][keep][E] pairs: q of the kept iterations, then of a segment run again
    void* ckpt;            // states at the segments' starts (wckpt)
    void* gr;              // [slots][E] pairs: minus the adjoint of the messages
    void* save;            // [slots][N]: the adjoint of the posteriors while a segment runs again
    int32_t* used;         // [B] 1: a backward pass has run segments over the frame's kept q
    const void* gpost;     // [T or 1][B][N] adjoint of the posteriors
    void* galpha;          // [T][C] (accumulated)
    void* gbeta;           // [T][C] (accumulated)
    void* gllr;            // [B][n_tx] (optional)
};

// Host side (weighted.cu); real_bytes 4 (float) or 8 (double).  weighted_plan fills keep, n_slots and the
// workspace offsets from the sizes in p and returns the workspace's bytes.
size_t weighted_plan(WParams* p, int Z, int D, int ckpt_every, int n_sm, size_t real_bytes);
int weighted_launch(const WParams& p, int Z, int D, int real_bytes, bool fwd, int n_sm, cudaStream_t stream,
                    std::string& err);
bool weighted_supported(int Z, int D, int real_bytes);

}  // namespace ldpcb200
