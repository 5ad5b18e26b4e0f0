// Kernel variants for Z = 256, D = 10: AR4JA rate 2/3, K = 4096 (N = 7168, 3072 checks).
#include "ldpc_qc.cuh"
#include "ldpc_registry.h"

using namespace ldpcb200;

static const QcEntry qc_r23k4[] = {
    LDPC_QC_ENTRY(256, 10, 1, 1, STORE_BF16, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(256, 10, 1, 1, STORE_FP16, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(256, 10, 1, 1, STORE_FP32, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(256, 10, 1, 1, STORE_BF16, ALGO_AMIN, true, false),
    LDPC_QC_ENTRY(256, 10, 1, 1, STORE_BF16, ALGO_NMS, false, false),
    LDPC_QC_ENTRY(256, 10, 1, 1, STORE_BF16, ALGO_NMS, true, false),
    LDPC_QC_ENTRY(256, 10, 1, 1, STORE_BF16, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(256, 10, 1, 1, STORE_FP16, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(256, 10, 1, 1, STORE_FP32, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(256, 10, 1, 1, STORE_BF16, ALGO_AMIN, true, true),
    LDPC_QC_ENTRY(256, 10, 1, 1, STORE_BF16, ALGO_NMS, false, true),
    LDPC_QC_ENTRY(256, 10, 1, 1, STORE_BF16, ALGO_NMS, true, true),
    // column offset table in shared memory (layout 2)
    LDPC_QC_ENTRY_OT(256, 10, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(256, 10, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(256, 10, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 0),
    // layout 6: the code's descriptors compiled in, no offset table
    LDPC_QC_ENTRY_RF(256, 10, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 2, 7),
    LDPC_QC_ENTRY_RF(256, 10, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 2, 7),
    LDPC_QC_ENTRY_RF(256, 10, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 3, 7),
    // the storages' fastest shapes for caller-supplied LLRs
    LDPC_QC_ENTRY_RF(256, 10, 1, 1, STORE_BF16, ALGO_AMIN, false, true, 2, 7),
    LDPC_QC_ENTRY_RF(256, 10, 1, 1, STORE_FP16, ALGO_AMIN, false, true, 3, 7),
    LDPC_QC_ENTRY_RF(256, 10, 1, 1, STORE_FP32, ALGO_AMIN, false, true, 2, 7),
    // the same for the -n and clip options
    LDPC_QC_ENTRY_RF(256, 10, 1, 1, STORE_BF16, ALGO_NMS, false, false, 2, 7),
    LDPC_QC_ENTRY_RF(256, 10, 1, 1, STORE_BF16, ALGO_AMIN, true, false, 2, 7),
    LDPC_QC_ENTRY_RF(256, 10, 1, 1, STORE_BF16, ALGO_NMS, false, true, 2, 7),
    LDPC_QC_ENTRY_RF(256, 10, 1, 1, STORE_BF16, ALGO_AMIN, true, true, 2, 7),
    // clips with fp16 and fp32 storage, caller-supplied LLRs (also the decoding without allocation)
    LDPC_QC_ENTRY_RF(256, 10, 1, 1, STORE_FP16, ALGO_AMIN, true, true, 3, 7),
    LDPC_QC_ENTRY_RF(256, 10, 1, 1, STORE_FP32, ALGO_AMIN, true, true, 2, 7),
};
LDPC_QC_REGISTER(qc_r23k4)

// Default shapes (us of the kernel at 1 / 100 / 440 / 25000 frames, 2.85 dB):
//   bf16: layout 6 36.2 / 43.3 / 84.3 / 3731, layout 2 40.1 / 46.6 / 110.6 / 5068, (1,1,0,0) 37.2 / 45.4 / 114.0 / 5451;
//         min-sum (10000 frames) 28.8 / 37.0 / 74.0 / 1312 against 31.1 / 41.1 / 94.6 / 1800; with clips 39.2 / 45.2 / 92.5 / 1676
//         against 41.2 / 47.3 / 121.2 / 2347
//   fp16: layout 6 39.1 / 45.4 / 90.5 / 3737, layout 2 38.9 / 45.4 / 107.8 / 4951, (1,1,0,0) 37.2 / 43.2 / 110.9 / 5189
//   fp32: layout 6 34.9 / 41.2 / 78.2 / 3366, layout 2 36.1 / 43.3 / 99.4 / 4509, (1,1,0,0) 33.2 / 39.8 / 99.6 / 4664
static const QcDefault qc_r23k4_default[] = {
    {256, 10, STORE_BF16, -1, 0, 1, 1, 2, 6},
    {256, 10, STORE_BF16, -1, 200, 1, 1, 0, 2},
    {256, 10, STORE_FP16, -1, 200, 1, 1, 3, 6},
    {256, 10, STORE_FP16, -1, 200, 1, 1, 0, 2},
    {256, 10, STORE_FP32, -1, 200, 1, 1, 2, 6},
    {256, 10, STORE_FP32, -1, 1500, 1, 1, 0, 2},
};
LDPC_QC_DEFAULTS(qc_r23k4_default)
