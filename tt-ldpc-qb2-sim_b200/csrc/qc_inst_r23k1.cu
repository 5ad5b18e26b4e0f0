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

// Default shapes (us of the kernel at 1 / 440 / 5000 / 100000 frames, 2.85 dB):
//   bf16: layout 6 29.1 / 64.8 / 241.0 / 4415, layout 7 33.0 / 74.1 / 238.9 / 3920, layout 2 30.9 / 68.0 / 270.7 / 4930,
//         (1,1,0,0) 31.0 / 75.1 / 300.2 / 5640; min-sum layout 6 22.9 / 75.0 / 187.7 / 3238, layout 7 25.9 / 100.4 / 250.2 /
//         3782, (1,1,0,0) 28.9 / 105.4 / 244.6 / 4332; with clips layout 6 28.7 / 69.7 / 288.1 / 5301, layout 7 35.0 / 77.2 /
//         261.5 / 4380, (1,1,0,0) 32.1 / 81.2 / 354.5 / 6727
//   fp16: layout 2 35.2 / 75.1 / 264.4 / 4823, (1,1,0,0) 33.1 / 77.1 / 295.2 / 5584
//   fp32: layout 2 29.2 / 59.8 / 215.4 / 3867, layout 7 31.9 / 73.9 / 227.6 / 3580, (1,1,0,0) 26.9 / 68.0 / 281.9 / 5184
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
