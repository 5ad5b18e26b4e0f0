// Kernel variants for Z = 128, D = 6: AR4JA rate 1/2, K = 1024 (N = 2560, 1536 checks).
#include "ldpc_qc.cuh"
#include "ldpc_registry.h"

using namespace ldpcb200;

static const QcEntry qc_r12k1[] = {
    // simulation (Philox channel), Approximate-Min*, no clips: the benchmarked path
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(128, 6, 1, 2, STORE_FP32, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, false),
    // paired: two interleaved frames per thread, packed f32x2 arithmetic (16-bit messages)
    LDPC_QC_ENTRY_PAIR(128, 6, STORE_BF16, false, 0),
    LDPC_QC_ENTRY_PAIR(128, 6, STORE_BF16, false, 4),
    LDPC_QC_ENTRY_PAIR(128, 6, STORE_BF16, false, 5),
    LDPC_QC_ENTRY_PAIR(128, 6, STORE_FP16, false, 0),
    LDPC_QC_ENTRY_PAIR(128, 6, STORE_FP16, false, 4),
    LDPC_QC_ENTRY_PAIR(128, 6, STORE_FP16, false, 5),
    LDPC_QC_ENTRY_PAIR(128, 6, STORE_BF16, true, 0),
    LDPC_QC_ENTRY_PAIR(128, 6, STORE_FP16, true, 0),
    // register caps for more resident warps: 5 CTAs/SM (<= 96 registers), 6 (<= 80), 8 (<= 64)
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 5),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 6),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 5),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 6),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 8),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 5),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 6),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 8),
    // caller-supplied LLRs (parity tests, ldpc_decode_llr)
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, true),
    // reference-engine options: -n (NMS) and the -L/-R/-V/-G clips, reference numerics
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, true, false),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_NMS, false, false),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_NMS, true, false),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, true, true),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_NMS, false, true),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_NMS, true, true),
    // column offset table in shared memory (no circulant index arithmetic per edge)
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 5),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 6),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 6),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 8),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 8),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, true, 0),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, true, 0),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, true, 0),
    // layout 6: messages in registers, the code's layer descriptors compiled in (no offset table)
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 0, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 5, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 6, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 8, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 6, 5),
    // weighted Approximate-Min* (trained weights, LDPC_ALGO_WAMIN): simulation and caller-supplied LLRs
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP32, ALGO_WAMIN, false, false),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP16, ALGO_WAMIN, false, false),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_WAMIN, false, false),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_FP16, ALGO_WAMIN, false, false, 5),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_FP16, ALGO_WAMIN, false, false, 6),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_FP16, ALGO_WAMIN, false, false, 8),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_FP32, ALGO_WAMIN, false, false, 5),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP32, ALGO_WAMIN, false, true),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP16, ALGO_WAMIN, false, true),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_WAMIN, false, true),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP32, ALGO_WAMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP32, ALGO_WAMIN, false, false, 5),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP16, ALGO_WAMIN, false, false, 6),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP32, ALGO_WAMIN, false, true, 0),
    // the same shapes with one (alpha, beta) per row (weights of one class per protograph check row)
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP32, ALGO_WROW, false, false),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP16, ALGO_WROW, false, false),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_WROW, false, false),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_FP16, ALGO_WROW, false, false, 5),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_FP16, ALGO_WROW, false, false, 6),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_FP16, ALGO_WROW, false, false, 8),
    LDPC_QC_ENTRY_B(128, 6, 1, 1, STORE_FP32, ALGO_WROW, false, false, 5),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP32, ALGO_WROW, false, true),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP16, ALGO_WROW, false, true),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_WROW, false, true),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP32, ALGO_WROW, false, false, 0),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP32, ALGO_WROW, false, false, 5),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP16, ALGO_WROW, false, false, 6),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_FP32, ALGO_WROW, false, true, 0),
    // the storages' fastest shapes for caller-supplied LLRs
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, true, 8, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, true, 6, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, true, 5, 5),
    // the same for the -n and clip options
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_BF16, ALGO_NMS, false, false, 8, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, true, false, 8, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_BF16, ALGO_NMS, false, true, 8, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, true, true, 8, 5),
    // clips with fp16 and fp32 storage, caller-supplied LLRs (also the decoding without allocation)
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, true, true, 6, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, true, true, 5, 5),
    // layout 6 with more registers, for calls of few frames
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 5, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 5, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, true, 5, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, true, 5, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, true, 0, 5),
};
LDPC_QC_REGISTER(qc_r12k1)

// Default shapes.  us of the kernel at 1 / 440 / 1500 / 5000 / 100000 frames, 2.04 dB, all shapes in one run.  Few frames wait for
// the slowest of them, where fewer registers a thread do not help; with many, resident warps and instructions decide.
//   bf16: layout 6 cap 5 22.4 / 45.1 / 98.2 / 277 / 5007, cap 8 24.5 / 50.0 / 103 / 284 / 5084, layout 2 25.6 / 53.2 / 106 / 289 / 5141,
//         layout 0 cap 5 23.6 / 49.2 / 109 / 311 / 5675, (1,1,0,0) 25.6 / 55.3 / 120 / 341 / 6268
//   fp16: layout 6 cap 5 20.5 / 43.0 / 98.3 / 279 / 5103, cap 6 22.5 / 45.9 / 104 / 289 / 5220, layout 2 cap 6 24.5 / 49.1 / 104 / 289 /
//         5171, (1,1,0,0) 23.6 / 51.0 / 114 / 324 / 5960
//   fp32: layout 6 19.1 / 38.9 / 86.0 / 239 / 4356, its cap 5 19.1 / 38.9 / 84.0 / 236 / 4252, layout 2 cap 5 22.5 / 43.0 / 94.1 / 254 /
//         4530, (1,1,0,0) 21.2 / 43.8 / 99.1 / 281 / 5140
//   normalised min-sum bf16: layout 6 cap 8 21.2 / 49.3 / 102 / 281 / 5006, (1,1,0,0) 18.5 / 45.1 / 106 / 312 / 5750; with clips 26.5 /
//         56.2 / 122 / 335 / 6499 and 26.6 / 56.2 / 131 / 374 / 7405
//   weighted fp32: layout 2 31.7 / 61.4 / 122 / 335 / 6011, (1,1,0,0) 28.7 / 58.0 / 120 / 342 / 6241; fp16: cap 5 30.7 / 61.4 / 127 / 356 /
//         6499, (1,1,0,0) 31.6 / 63.5 / 135 / 384 / 7037
// The other lines are for options or matrices the first of their storage is not built for.
static const QcDefault qc_r12k1_default[] = {
    {128, 6, STORE_FP32, ALGO_WAMIN, 1500, 1, 1, 0, 2},
    {128, 6, STORE_FP32, ALGO_WAMIN, 0, 1, 1, 0, 0},
    {128, 6, STORE_FP16, ALGO_WAMIN, 0, 1, 1, 5, 0},
    {128, 6, STORE_BF16, -1, 0, 1, 1, 5, 6},
    {128, 6, STORE_BF16, -1, 1500, 1, 1, 8, 6},
    {128, 6, STORE_BF16, -1, 1500, 1, 1, 8, 2},
    {128, 6, STORE_BF16, -1, 1500, 1, 1, 0, 2},
    {128, 6, STORE_BF16, -1, 0, 1, 1, 5, 0},
    {128, 6, STORE_FP16, -1, 0, 1, 1, 5, 6},
    {128, 6, STORE_FP16, -1, 1500, 1, 1, 6, 2},
    {128, 6, STORE_FP16, -1, 1500, 1, 1, 6, 6},
    {128, 6, STORE_FP16, -1, 1500, 1, 1, 0, 2},
    {128, 6, STORE_FP16, -1, 0, 1, 1, 5, 0},
    {128, 6, STORE_FP32, -1, 1000, 1, 1, 5, 6},
    {128, 6, STORE_FP32, -1, 1500, 1, 1, 5, 2},
    {128, 6, STORE_FP32, -1, 1500, 1, 1, 0, 2},
    {128, 6, STORE_FP32, -1, 0, 1, 1, 0, 6},
};
LDPC_QC_DEFAULTS(qc_r12k1_default)
