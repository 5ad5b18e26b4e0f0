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

// Default shapes (us of the kernel at 1 / 440 / 1500 / 100000 frames, 2.04 dB, Approximate-Min*).  Few frames
// wait for the slowest of them, where fewer registers per thread do not help; with many, resident warps and
// instructions decide.  Layout 6 cap 5 is ahead at both ends since its min* step is one instruction shorter
// (amin_step_scaled): bf16 at 1 / 440 / 1500 / 5000 / 100000 frames 21.5 / 43.2 / 98 / 276 / 4982 against cap 8 25.6 / 54.1 /
// 109.5 / 284 / 5067, caller-supplied LLRs (8000 frames) 429 against 445; fp16 (20.5 / 48.2 / 102.4) / 285 / 5102 against
// layout 2 cap 6 289 / 5173.  The figures below were taken before that, of one run each.
//   bf16: layout 0 cap 5 25.0 / 47.5 / 110.8 / 5831, layout 6 cap 8 27.6 / 50.2 / 108.6 / 5269, layout 2 cap 8 - / 53.5 / 109.0 / 5335,
//         (1,1,0,0) 26.9 / 52.2 / 119.0 / 6268
//   fp16: layout 0 cap 5 23.5 / 46.3 / 110.8 / 5780, layout 2 cap 6 26.8 / 47.5 / 104.9 / 5171, layout 6 cap 6 24.9 / 45.4 / 104.8 /
//         5218, (1,1,0,0) 24.9 / 49.2 / 114.0 / 5966
//   fp32: layout 6 21.0 / 39.3 / 95.6 / 5057, its cap 5 22.8 / 39.1 / 92.5 / 4664, layout 2 cap 5 26.8 / 45.4 / 94.7 / 4678,
//         (1,1,0,0) 22.8 / 43.3 / 96.4 / 5143
//   normalised min-sum bf16: layout 6 cap 8 27.9 / 51.6 / 107.4 / 5013 against 22.8 / 48.5 / 109.8 / 5757; with clips 30.0 /
//   55.6 / 125.2 / 6028 against 29.0 / 56.2 / 135.1 / 6915; weighted fp32: layout 2 37.2 / 55.8 / 121.3 / 2396 (40000)
//   against 35.1 / 53.6 / 120.9 / 2483, its cap 5 2484; fp16: cap 5 35.9 / 57.7 / 129.1 / 2589 against 2799
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
