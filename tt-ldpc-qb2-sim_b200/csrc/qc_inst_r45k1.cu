// Kernel variants for Z = 32, D = 18: AR4JA rate 4/5, K = 1024 (N = 1408, 384 checks).
// FP32 message storage is not built for D = 18: 156 fp32 messages per thread do not fit the
// register file next to the working set (16-bit storage packs them into 78 registers).
#include "ldpc_qc.cuh"
#include "ldpc_registry.h"

using namespace ldpcb200;

static const QcEntry qc_r45k1[] = {
    LDPC_QC_ENTRY(32, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(32, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false),
    LDPC_QC_ENTRY(32, 18, 1, 1, STORE_BF16, ALGO_AMIN, true, false),
    LDPC_QC_ENTRY(32, 18, 1, 1, STORE_BF16, ALGO_NMS, false, false),
    LDPC_QC_ENTRY(32, 18, 1, 1, STORE_BF16, ALGO_NMS, true, false),
    LDPC_QC_ENTRY(32, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(32, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, true),
    LDPC_QC_ENTRY(32, 18, 1, 1, STORE_BF16, ALGO_AMIN, true, true),
    LDPC_QC_ENTRY(32, 18, 1, 1, STORE_BF16, ALGO_NMS, false, true),
    LDPC_QC_ENTRY(32, 18, 1, 1, STORE_BF16, ALGO_NMS, true, true),
    // weighted Approximate-Min* (trained weights, LDPC_ALGO_WAMIN): simulation and caller-supplied LLRs
    LDPC_QC_ENTRY(32, 18, 1, 1, STORE_FP16, ALGO_WAMIN, false, false),
    LDPC_QC_ENTRY(32, 18, 1, 1, STORE_FP16, ALGO_WAMIN, false, true),
    // column offset table in shared memory (layout 2)
    LDPC_QC_ENTRY_OT(32, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_OT(32, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 0),
    // check messages in global memory (layout 1): the 156 per-thread message registers of the
    // register layout leave room for only 8-10 warps per SM; without them the kernel holds more frames
    LDPC_QC_ENTRY_G(32, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_G(32, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 0),
    LDPC_QC_ENTRY_G(32, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 0),
    // the same capped at 64 registers (32 CTAs of 32 threads per SM)
    LDPC_QC_ENTRY_G(32, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 32),
    LDPC_QC_ENTRY_G(32, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 32),
    LDPC_QC_ENTRY_G(32, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 32),
    // layout 5: the register-capped shapes with the code's layer descriptors compiled in
    // (ar4ja_fixed_tables.h entry 3)
    LDPC_QC_ENTRY_GF(32, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 32, 3),
    LDPC_QC_ENTRY_GF(32, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 32, 3),
    LDPC_QC_ENTRY_GF(32, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 32, 3),
    // layout 7: the eight degree-18 layers in a loop that is not unrolled.  The unrolled body does
    // not fit the instruction cache, and with one-warp CTAs each warp is somewhere else in it (ncu:
    // 9 no-instruction stalls per issue, issue 46 %).  Rolled, at 16-24 CTAs per SM (80-112
    // registers, no 64-register spills, a message scratch that stays in L2): fp32 23.1 -> 34.5,
    // bf16 21.3 -> 30.9 M frames/s at threshold + 1.25 dB.
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 24),
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 20),
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, false, 16),
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 24),
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 16),
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 16),
    // the storages' fastest shapes for caller-supplied LLRs
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, true, 16),
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, true, 16),
    LDPC_QC_ENTRY_GR_NAN(32, 18, 1, 1, STORE_FP32, ALGO_AMIN, true, 24),
    // the same for the -n and clip options
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_BF16, ALGO_NMS, false, false, 16),
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_BF16, ALGO_AMIN, true, false, 16),
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_BF16, ALGO_NMS, false, true, 16),
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_BF16, ALGO_AMIN, true, true, 16),
    // clips with fp16 and fp32 storage, caller-supplied LLRs (also the decoding without allocation)
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_FP16, ALGO_AMIN, true, true, 16),
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_FP32, ALGO_AMIN, true, true, 24),
    // fp32 caller-supplied LLRs at LLR_SCALE (the unscaled counterpart is the larger cap): us for 300 / 8000 frames with 15 CTAs'
    // registers 66.5 / 295, 16 66.5 / 293, 17 68.6 / 299, 22 69 / 329; 15, which no simulation kernel has, leaves
    // simulations their own default
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, true, 15),
};
LDPC_QC_REGISTER(qc_r45k1)

// Default shapes.  us of the kernel at 1 / 440 / 1500 / 5000 / 100000 frames, 3.80 dB, all shapes in one run: layout 7 at 16 or 24
// CTAs per SM
//   bf16: 28.7 / 73.8 / 94.2 / 248 / 3423, (1,1,0,0) 33.8 / 91.0 / 143 / 534 / 11715; min-sum 27.5 / 65.5 / 143 / 870 / 2786 and 33.6 / 84.9 /
//         187 / 1203 / 7767; with clips 30.7 / 83.9 / 1689 / 1737 / 4811 and 36.9 / 98.3 / 1939 / 2221 / 14962
//   fp16: 28.7 / 69.4 / 124 / 358 / 3419, (1,1,0,0) 32.8 / 78.7 / 160 / 638 / 11425
//   fp32: 24 CTAs 27.5 / 69.7 / 119 / 242 / 2405, 16 CTAs 26.7 / 65.5 / 119 / 246 / 2447, layout 1 32.4 / 77.8 / 150 / 389 / 5398
static const QcDefault qc_r45k1_default[] = {
    {32, 18, STORE_BF16, -1, 0, 1, 1, 16, 7},
    {32, 18, STORE_FP16, -1, 0, 1, 1, 16, 7},
    {32, 18, STORE_FP32, -1, 0, 1, 1, 15, 7},  // (caller-supplied LLRs only)
    {32, 18, STORE_FP32, -1, 0, 1, 1, 24, 7},
};
LDPC_QC_DEFAULTS(qc_r45k1_default)
