// Kernel variants for Z = 64, D = 10: AR4JA rate 2/3, K = 1024 (N = 1792, 768 checks).
#include "ldpc_qc.cuh"
#include "ldpc_registry.h"

using namespace ldpcb200;

static const QcEntry qc_r23k1[] = {
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_BF16, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_FP16, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_FP32, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_BF16, ALGO_AMIN, true, false),
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_BF16, ALGO_NMS, false, false),
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_BF16, ALGO_NMS, true, false),
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_BF16, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_FP16, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_FP32, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_BF16, ALGO_AMIN, true, true),
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_BF16, ALGO_NMS, false, true),
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_BF16, ALGO_NMS, true, true),
    // weighted Approximate-Min* (trained weights, LDPC_ALGO_WAMIN): simulation and caller-supplied LLRs
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_FP16, ALGO_WAMIN, false, false),
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_FP16, ALGO_WAMIN, false, true),
    LDPC_QC_ENTRY(64, 10, 1, 1, STORE_FP32, ALGO_WAMIN, false, true),
    // column offset table in shared memory (layout 2)
    LDPC_QC_ENTRY_OT(64, 10, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(64, 10, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(64, 10, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 0),
    // layout 6: the code's descriptors compiled in, no offset table
    LDPC_QC_ENTRY_RF(64, 10, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 0, 8),
    // layout 7: messages in global memory with the degree-10 layers in a loop that is not unrolled:
    // fp32 24.2 (offset table) -> 25.7, bf16 21.1 (layout 6) -> 22.4 M frames/s at threshold + 1.25 dB
    LDPC_QC_ENTRY_GR(64, 10, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_GR(64, 10, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 16),
    LDPC_QC_ENTRY_GR(64, 10, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 16),
    // the storages' fastest shapes for caller-supplied LLRs
    LDPC_QC_ENTRY_GR(64, 10, 1, 1, STORE_BF16, ALGO_AMIN, false, true, 16),
    LDPC_QC_ENTRY_RF(64, 10, 1, 1, STORE_BF16, ALGO_AMIN, false, true, 0, 8),
    LDPC_QC_ENTRY_OT(64, 10, 1, 1, STORE_FP16, ALGO_AMIN, false, true, 0),
    LDPC_QC_ENTRY_GR(64, 10, 1, 1, STORE_FP32, ALGO_AMIN, false, true, 0),
    LDPC_QC_ENTRY_OT(64, 10, 1, 1, STORE_FP32, ALGO_AMIN, false, true, 0),
    // the same for the -n and clip options
    LDPC_QC_ENTRY_GR(64, 10, 1, 1, STORE_BF16, ALGO_NMS, false, false, 16),
    LDPC_QC_ENTRY_GR(64, 10, 1, 1, STORE_BF16, ALGO_AMIN, true, false, 16),
    LDPC_QC_ENTRY_GR(64, 10, 1, 1, STORE_BF16, ALGO_NMS, false, true, 16),
    LDPC_QC_ENTRY_GR(64, 10, 1, 1, STORE_BF16, ALGO_AMIN, true, true, 16),
    LDPC_QC_ENTRY_RF(64, 10, 1, 1, STORE_BF16, ALGO_NMS, false, false, 0, 8),
    LDPC_QC_ENTRY_RF(64, 10, 1, 1, STORE_BF16, ALGO_AMIN, true, false, 0, 8),
    LDPC_QC_ENTRY_RF(64, 10, 1, 1, STORE_BF16, ALGO_NMS, false, true, 0, 8),
    LDPC_QC_ENTRY_RF(64, 10, 1, 1, STORE_BF16, ALGO_AMIN, true, true, 0, 8),
    // clips with fp16 and fp32 storage, caller-supplied LLRs (also the decoding without allocation)
    LDPC_QC_ENTRY_OT(64, 10, 1, 1, STORE_FP16, ALGO_AMIN, true, true, 0),
    LDPC_QC_ENTRY_GR(64, 10, 1, 1, STORE_FP32, ALGO_AMIN, true, true, 0),
    LDPC_QC_ENTRY_OT(64, 10, 1, 1, STORE_FP32, ALGO_AMIN, true, true, 0),
};
LDPC_QC_REGISTER(qc_r23k1)

// Default shapes.  us of the kernel at 1 / 440 / 1500 / 5000 / 100000 frames, 2.85 dB, all shapes in one run:
//   bf16: layout 6 25.5 / 45.1 / 82.8 / 232 / 4240, layout 7 27.7 / 49.2 / 89.0 / 224 / 3659, layout 2 28.7 / 50.2 / 90.1 / 251 / 4508,
//         (1,1,0,0) 30.7 / 55.3 / 104 / 309 / 5676; min-sum layout 6 19.5 / 39.8 / 70.7 / 187 / 3258, layout 7 23.5 / 51.2 / 90.1 / 238 /
//         3826, (1,1,0,0) 24.5 / 52.1 / 96.2 / 255 / 4472; with clips layout 6 28.7 / 52.1 / 1053 / 1178 / 6284, layout 7 30.7 / 57.3 /
//         1162 / 1312 / 5465, (1,1,0,0) 30.8 / 59.4 / 1164 / 1399 / 7984
//   fp16: layout 2 29.4 / 51.2 / 96.3 / 263 / 4828, (1,1,0,0) 30.7 / 53.4 / 104 / 299 / 5569
//   fp32: layout 2 25.4 / 42.0 / 77.8 / 225 / 3594, layout 7 28.6 / 50.1 / 87.0 / 247 / 3438, (1,1,0,0) 26.6 / 47.9 / 101 / 297 / 5181
static const QcDefault qc_r23k1_default[] = {
    {64, 10, STORE_BF16, ALGO_NMS, 0, 1, 1, 0, 6},
    {64, 10, STORE_BF16, -1, 5000, 1, 1, 16, 7},
    {64, 10, STORE_BF16, -1, 0, 1, 1, 0, 6},
    {64, 10, STORE_BF16, -1, 64, 1, 1, 0, 2},
    {64, 10, STORE_FP16, -1, 64, 1, 1, 0, 2},
    {64, 10, STORE_FP32, -1, 10000, 1, 1, 0, 7},
    {64, 10, STORE_FP32, -1, 64, 1, 1, 0, 2},
};
LDPC_QC_DEFAULTS(qc_r23k1_default)
