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

// Default shapes (us of the kernel at 1 / 100 / 440 / 25000 frames, 2.04 dB): up to one frame per SM the
// uncapped kernel is as fast; above, layout 6 holds two CTAs per SM
//   bf16: layout 6 47.4 / 57.5 / 121.8 / 5673, (1,1,0,0) 47.3 / 58.7 / 143.7 / 6885; min-sum (12500 frames) 48.5 / 59.7 /
//         121.0 / 2226 against 48.2 / 57.6 / 139.6 / 2672; with clips 53.4 / 64.7 / 139.6 / 2637 against 55.6 / 67.7 / 168.1 / 3246
//   fp16: layout 6 47.1 / 53.3 / 120.0 / 5712, (1,1,0,0) 46.2 / 53.4 / 134.3 / 6631
//   fp32: layout 6 39.2 / 45.3 / 117.0 / 5565, layout 2 43.2 / 49.4 / 122.2 / 5632, (1,1,0,0) 43.2 / 49.4 / 129.2 / 6122
static const QcDefault qc_r12k4_default[] = {
    {512, 6, STORE_BF16, -1, 200, 1, 1, 2, 6},
    {512, 6, STORE_FP16, -1, 200, 1, 1, 2, 6},
    {512, 6, STORE_FP32, -1, 0, 1, 1, 1, 6},
    {512, 6, STORE_FP32, -1, 200, 1, 1, 0, 2},
};
LDPC_QC_DEFAULTS(qc_r12k4_default)
