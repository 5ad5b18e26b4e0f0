// Kernel variants for Z = 128, D = 18: AR4JA rate 4/5, K = 4096 (N = 5632, 1536 checks).
// FP32 message storage is not built for D = 18: 156 fp32 messages per thread do not fit the
// register file next to the working set (16-bit storage packs them into 78 registers).
#include "ldpc_qc.cuh"
#include "ldpc_registry.h"

using namespace ldpcb200;

static const QcEntry qc_r45k4[] = {
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_BF16, ALGO_AMIN, true, false),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_BF16, ALGO_NMS, false, false),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_BF16, ALGO_NMS, true, false),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_BF16, ALGO_AMIN, true, true),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_BF16, ALGO_NMS, false, true),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_BF16, ALGO_NMS, true, true),
    // weighted Approximate-Min* (trained weights, LDPC_ALGO_WAMIN): simulation and caller-supplied LLRs
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_FP16, ALGO_WAMIN, false, false),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_BF16, ALGO_WAMIN, false, false),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_FP16, ALGO_WAMIN, false, true),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_BF16, ALGO_WAMIN, false, true),
    // column offset table in shared memory (layout 2)
    LDPC_QC_ENTRY_OT(128, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(128, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(128, 18, 1, 1, STORE_FP16, ALGO_WAMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(128, 18, 1, 1, STORE_BF16, ALGO_WAMIN, false, false, 0),
    // the same shapes with one (alpha, beta) per row (weights of one class per protograph check row)
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_FP16, ALGO_WROW, false, false),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_BF16, ALGO_WROW, false, false),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_FP16, ALGO_WROW, false, true),
    LDPC_QC_ENTRY(128, 18, 1, 1, STORE_BF16, ALGO_WROW, false, true),
    LDPC_QC_ENTRY_OT(128, 18, 1, 1, STORE_FP16, ALGO_WROW, false, false, 0),
    LDPC_QC_ENTRY_OT(128, 18, 1, 1, STORE_BF16, ALGO_WROW, false, false, 0),
    // check messages in global memory (layout 1): the 156 per-thread message registers of the
    // register layout leave room for only 8-10 warps per SM; without them the kernel holds more frames
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 0),
    // the same capped at 64 registers (8 CTAs of 128 threads per SM)
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 8),
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 8),
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 8),
    // layout 5: the register-capped shapes with the code's layer descriptors compiled in
    // (ar4ja_fixed_tables.h entry 4)
    LDPC_QC_ENTRY_GF(128, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 8, 4),
    LDPC_QC_ENTRY_GF(128, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 8, 4),
    LDPC_QC_ENTRY_GF(128, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 8, 4),
    // the weighted decoders in the same layout (per-edge and per-row weights)
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_BF16, ALGO_WAMIN, false, false, 8),
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_FP16, ALGO_WAMIN, false, false, 8),
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_FP32, ALGO_WAMIN, false, false, 8),
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_FP32, ALGO_WAMIN, false, true, 8),
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_BF16, ALGO_WROW, false, false, 8),
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_FP16, ALGO_WROW, false, false, 8),
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_FP32, ALGO_WROW, false, false, 8),
    LDPC_QC_ENTRY_G(128, 18, 1, 1, STORE_FP32, ALGO_WROW, false, true, 8),
    // layout 7: the degree-18 layers in a loop that is not unrolled (the instruction cache; 4-6
    // CTAs per SM at 80-112 registers): fp32 6.92 -> 8.32, bf16 6.45 -> 7.63 M frames/s at
    // threshold + 1.25 dB; and the weighted decoders in the same layout
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 6),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 4),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 6),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 5),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 6),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_FP32, ALGO_WAMIN, false, false, 6),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_BF16, ALGO_WAMIN, false, false, 6),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_FP16, ALGO_WAMIN, false, false, 6),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_FP32, ALGO_WROW, false, false, 6),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_BF16, ALGO_WROW, false, false, 6),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_FP16, ALGO_WROW, false, false, 6),
    // the storages' fastest shapes for caller-supplied LLRs
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, true, 6),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, true, 6),
    LDPC_QC_ENTRY_GR_NAN(128, 18, 1, 1, STORE_FP32, ALGO_AMIN, true, 6),
    // the same for the -n and clip options
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_BF16, ALGO_NMS, false, false, 6),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_BF16, ALGO_AMIN, true, false, 6),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_BF16, ALGO_NMS, false, true, 6),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_BF16, ALGO_AMIN, true, true, 6),
    // clips with fp16 and fp32 storage, caller-supplied LLRs (also the decoding without allocation)
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_FP16, ALGO_AMIN, true, true, 6),
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_FP32, ALGO_AMIN, true, true, 6),
    // fp32 caller-supplied LLRs at LLR_SCALE (the unscaled counterpart is the larger cap)
    LDPC_QC_ENTRY_GR(128, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, true, 5),
};
LDPC_QC_REGISTER(qc_r45k4)

// Default shapes.  us of the kernel at 1 / 100 / 440 / 1500 / 25000 frames, 3.80 dB, all shapes in one run: layout 7 at 6 CTAs per SM
//   bf16: 35.8 / 50.0 / 75.7 / 199 / 2729, (1,1,0,0) 38.8 / 53.2 / 96.3 / 303 / 5349; min-sum 32.7 / 38.8 / 69.6 / 181 / 2471 and 37.9 / 46.0 /
//         86.0 / 246 / 3913; with clips 40.9 / 55.3 / 88.1 / 242 / 4054 and 41.0 / 55.3 / 104 / 339 / 6325
//   fp16: 36.9 / 51.0 / 78.8 / 202 / 2767, (1,1,0,0) 37.7 / 52.0 / 93.1 / 296 / 5175;  fp32: 34.8 / 47.9 / 78.6 / 197 / 2600, layout 1 38.9 /
//         53.2 / 86.0 / 254 / 3677
//   weighted, per edge: bf16 72.4 / 84.8 / 99.1 / 225 / 3012, (1,1,0,0) 63.5 / 73.8 / 115 / 343 / 6103; fp16 62.2 / 72.4 / 93.0 / 236 / 3210 and
//         59.4 / 68.4 / 111 / 338 / 5963; fp32 72.5 / 84.0 / 103 / 256 / 3458, layout 1 cap 8 69.6 / 81.9 / 102 / 303 / 4706
static const QcDefault qc_r45k4_default[] = {
    {128, 18, STORE_FP32, ALGO_WAMIN, 1000, 1, 1, 6, 7},
    {128, 18, STORE_FP32, ALGO_WAMIN, 0, 1, 1, 8, 1},
    {128, 18, STORE_FP32, ALGO_WROW, 1000, 1, 1, 6, 7},
    {128, 18, STORE_FP32, ALGO_WROW, 0, 1, 1, 8, 1},
    {128, 18, STORE_BF16, -1, 300, 1, 1, 6, 7},
    {128, 18, STORE_FP16, -1, 300, 1, 1, 6, 7},
    {128, 18, STORE_FP32, -1, 0, 1, 1, 5, 7},  // (caller-supplied LLRs only)
    {128, 18, STORE_FP32, -1, 0, 1, 1, 6, 7},
};
LDPC_QC_DEFAULTS(qc_r45k4_default)
