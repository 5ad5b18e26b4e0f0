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

// Default shapes (us of the kernel at 1 / 100 / 440 / 25000 frames, 3.80 dB): layout 7 at 6 CTAs per SM
//   bf16: 43.3 / 52.5 / 81.3 / 2853, (1,1,0,0) 39.0 / 51.6 / 97.5 / 5365; min-sum (10000 frames) 33.0 / 41.2 / 72.0 / 1012 against
//         37.2 / 49.2 / 88.4 / 1567; with clips 47.4 / 55.6 / 90.8 / 1362 against 45.2 / 57.7 / 106.7 / 2404
//   fp16: 43.2 / 49.8 / 80.0 / 2760, (1,1,0,0) 37.1 / 54.6 / 97.6 / 5218;  fp32: 42.3 / 50.5 / 84.3 / 2681, layout 1 42.3 / 53.6 /
//         90.4 / 3705
//   weighted, per edge (10000 frames): bf16 70.2 / 82.3 / 98.4 / 1247, (1,1,0,0) 59.6 / 70.0 / 121.4 / 2429; fp16 61.8 / 70.1 /
//         94.7 / 1319 against 55.6 / 63.8 / 117.1 / 2372; fp32 (1500 frames: 254) 71.7 / 82.3 / 102.7 / 1418, layout 1 cap 8 (302)
//         67.8 / 78.2 / 98.6 / 1887
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
