// Kernel variants for Z = 512, D = 6: AR4JA rate 1/2, K = 4096 (N = 10240, 6144 checks).
#include "ldpc_qc.cuh"
#include "ldpc_registry.h"

using namespace ldpcb200;

static const QcEntry qc_r12k4[] = {
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_BF16, ALGO_AMIN, true, false),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_BF16, ALGO_NMS, false, false),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_BF16, ALGO_NMS, true, false),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_BF16, ALGO_AMIN, true, true),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_BF16, ALGO_NMS, false, true),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_BF16, ALGO_NMS, true, true),
    // weighted Approximate-Min* (trained weights, LDPC_ALGO_WAMIN): simulation and caller-supplied LLRs
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_FP16, ALGO_WAMIN, false, false),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_FP16, ALGO_WAMIN, false, true),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_FP32, ALGO_WAMIN, false, true),
    // column offset table in shared memory (layout 2)
    LDPC_QC_ENTRY_OT(512, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(512, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(512, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 0),
    // layout 6: the code's descriptors compiled in, no offset table (its 120 KB held one CTA per SM)
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 1, 6),
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 2, 6),
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 2, 6),
    // the storages' fastest shapes for caller-supplied LLRs
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_BF16, ALGO_AMIN, false, true, 2, 6),
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_FP16, ALGO_AMIN, false, true, 2, 6),
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_FP32, ALGO_AMIN, false, true, 1, 6),
    // the same for the -n and clip options
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_BF16, ALGO_NMS, false, false, 2, 6),
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_BF16, ALGO_AMIN, true, false, 2, 6),
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_BF16, ALGO_NMS, false, true, 2, 6),
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_BF16, ALGO_AMIN, true, true, 2, 6),
    // clips with fp16 and fp32 storage, caller-supplied LLRs (also the decoding without allocation)
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_FP16, ALGO_AMIN, true, true, 2, 6),
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_FP32, ALGO_AMIN, true, true, 1, 6),
};
LDPC_QC_REGISTER(qc_r12k4)

// Default shapes.  us of the kernel at 1 / 100 / 440 / 1500 / 25000 frames, 2.04 dB, all shapes in one run: up to one frame per SM
// the uncapped kernel is about as fast; above, layout 6 holds two CTAs per SM
//   bf16: layout 6 42.0 / 51.9 / 120 / 362 / 5503, (1,1,0,0) 43.0 / 53.3 / 143 / 446 / 6886; min-sum 44.9 / 54.2 / 121 / 366 / 5504 and
//         43.9 / 54.1 / 138 / 429 / 6633; with clips 47.1 / 59.4 / 141 / 436 / 6521 and 50.0 / 61.4 / 167 / 521 / 8062
//   fp16: layout 6 41.0 / 53.2 / 123 / 385 / 5714, (1,1,0,0) 41.9 / 53.2 / 137 / 430 / 6628
//   fp32: layout 6 34.5 / 43.0 / 110 / 340 / 5212, layout 2 39.6 / 47.8 / 117 / 355 / 5401, (1,1,0,0) 39.6 / 49.9 / 127 / 398 / 6123
static const QcDefault qc_r12k4_default[] = {
    {512, 6, STORE_BF16, -1, 200, 1, 1, 2, 6},
    {512, 6, STORE_FP16, -1, 200, 1, 1, 2, 6},
    {512, 6, STORE_FP32, -1, 0, 1, 1, 1, 6},
    {512, 6, STORE_FP32, -1, 200, 1, 1, 0, 2},
};
LDPC_QC_DEFAULTS(qc_r12k4_default)
