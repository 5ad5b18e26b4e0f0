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

// Default shapes.  us of the kernel at 1 / 100 / 440 / 1500 / 25000 frames, 2.85 dB, all shapes in one run:
//   bf16: layout 6 30.7 / 40.7 / 81.9 / 238 / 3529, layout 2 34.4 / 43.0 / 86.0 / 249 / 3543, (1,1,0,0) 32.8 / 43.0 / 114 / 354 / 5454;
//         min-sum 28.7 / 34.8 / 73.7 / 223 / 3242 and (1,1,0,0) 30.7 / 38.9 / 97.3 / 296 / 4474; with clips 33.7 / 43.8 / 90.1 / 281 / 4151
//         and 35.8 / 46.3 / 121 / 377 / 5860
//   fp16: layout 6 34.8 / 43.0 / 90.1 / 272 / 3741, layout 2 34.8 / 43.0 / 107 / 328 / 4958, (1,1,0,0) 32.8 / 43.0 / 109 / 338 / 5198
//   fp32: layout 6 28.7 / 37.6 / 74.8 / 216 / 3167, layout 2 30.7 / 38.9 / 95.2 / 286 / 4293, (1,1,0,0) 29.7 / 38.9 / 98.3 / 305 / 4669
static const QcDefault qc_r23k4_default[] = {
    {256, 10, STORE_BF16, -1, 0, 1, 1, 2, 6},
    {256, 10, STORE_BF16, -1, 200, 1, 1, 0, 2},
    {256, 10, STORE_FP16, -1, 200, 1, 1, 3, 6},
    {256, 10, STORE_FP16, -1, 200, 1, 1, 0, 2},
    {256, 10, STORE_FP32, -1, 200, 1, 1, 2, 6},
    {256, 10, STORE_FP32, -1, 1500, 1, 1, 0, 2},
};
LDPC_QC_DEFAULTS(qc_r23k4_default)
