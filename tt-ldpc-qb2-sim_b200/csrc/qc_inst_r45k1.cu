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
    // fp32 caller-supplied LLRs at LLR_SCALE (the unscaled counterpart is the larger cap): us for 8000 / 300 frames with 16
    // CTAs' registers 293 / 65.5, 18 310 / 67.6, 20 310 / 65.5, 22 329 / 69
    LDPC_QC_ENTRY_GR(32, 18, 1, 1, STORE_FP32, ALGO_AMIN, false, true, 16),
};
LDPC_QC_REGISTER(qc_r45k1)

// Default shapes (us of the kernel at 1 / 440 / 5000 / 100000 frames, 3.80 dB): layout 7 at 16 or 24 CTAs per SM
//   bf16: 45.2 / 84.2 / 190.8 / 3067, (1,1,0,0) 45.9 / 97.2 / 478.5 / 11184; min-sum 34.0 / 54.3 / 175.5 / 2607 against 38.3 /
//         68.9 / 362.8 / 7348; with clips 46.4 / 87.3 / 209.8 / 4138 against 50.5 / 108.8 / 522.4 / 13509
//   fp16: 41.9 / 78.2 / 186.3 / 3140, (1,1,0,0) 44.2 / 98.6 / 457.6 / 11299
//   fp32: 43.2 / 80.1 / 188.7 / 2631, layout 1 43.4 / 92.2 / 289.0 / 5677
static const QcDefault qc_r45k1_default[] = {
    {32, 18, STORE_BF16, -1, 0, 1, 1, 16, 7},
    {32, 18, STORE_FP16, -1, 0, 1, 1, 16, 7},
    {32, 18, STORE_FP32, -1, 0, 1, 1, 16, 7},  // (caller-supplied LLRs only)
    {32, 18, STORE_FP32, -1, 0, 1, 1, 24, 7},
};
LDPC_QC_DEFAULTS(qc_r45k1_default)
