// Kernel variants for the K = 16384 AR4JA codes.  Their check messages (94,208 to 122,880 edges per
// frame) do not fit the register file, so they live in an L2-resident global scratch (RG kernels):
//   rate 1/2: Z = 2048, D = 6  (N = 40960, 24576 checks), 512 threads x 4 rows
//   rate 2/3: Z = 1024, D = 10 (N = 28672, 12288 checks), 512 threads x 2 rows
//   rate 4/5: Z = 512,  D = 18 (N = 22528,  6144 checks), 512 threads x 1 row
#include "ldpc_qc.cuh"
#include "ldpc_registry.h"

using namespace ldpcb200;

#define K16_SHAPE(Z, D, R)                                                          \
    LDPC_QC_ENTRY_G(Z, D, R, 1, STORE_BF16, ALGO_AMIN, false, false, 0),            \
    LDPC_QC_ENTRY_G(Z, D, R, 1, STORE_FP16, ALGO_AMIN, false, false, 0),            \
    LDPC_QC_ENTRY_G(Z, D, R, 1, STORE_FP32, ALGO_AMIN, false, false, 0),            \
    LDPC_QC_ENTRY_G(Z, D, R, 1, STORE_BF16, ALGO_AMIN, false, true, 0),             \
    LDPC_QC_ENTRY_G(Z, D, R, 1, STORE_FP16, ALGO_AMIN, false, true, 0),             \
    LDPC_QC_ENTRY_G(Z, D, R, 1, STORE_FP32, ALGO_AMIN, false, true, 0)

static const QcEntry qc_k16[] = {
    K16_SHAPE(2048, 6, 4),
    K16_SHAPE(1024, 10, 2),
    K16_SHAPE(512, 18, 1),
    // register cap of 64 (2 CTAs of 512 threads per SM) for the codes whose kernels need 77-110
    LDPC_QC_ENTRY_G(1024, 10, 2, 1, STORE_BF16, ALGO_AMIN, false, false, 2),
    LDPC_QC_ENTRY_G(1024, 10, 2, 1, STORE_FP16, ALGO_AMIN, false, false, 2),
    LDPC_QC_ENTRY_G(512, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 2),
    LDPC_QC_ENTRY_G(512, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 2),
    // layout 5: the same kernels with the code's layer descriptors compiled in (ar4ja_fixed_tables.h:
    // 0 = rate 1/2, 1 = rate 2/3, 2 = rate 4/5), so a circulant index costs no constant-bank operands
    LDPC_QC_ENTRY_GF(2048, 6, 4, 1, STORE_BF16, ALGO_AMIN, false, false, 0, 0),
    LDPC_QC_ENTRY_GF(2048, 6, 4, 1, STORE_FP16, ALGO_AMIN, false, false, 0, 0),
    LDPC_QC_ENTRY_GF(2048, 6, 4, 1, STORE_BF16, ALGO_AMIN, false, true, 0, 0),
    LDPC_QC_ENTRY_GF(1024, 10, 2, 1, STORE_BF16, ALGO_AMIN, false, false, 0, 1),
    LDPC_QC_ENTRY_GF(1024, 10, 2, 1, STORE_BF16, ALGO_AMIN, false, false, 2, 1),
    LDPC_QC_ENTRY_GF(1024, 10, 2, 1, STORE_FP16, ALGO_AMIN, false, false, 2, 1),
    LDPC_QC_ENTRY_GF(512, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 0, 2),
    LDPC_QC_ENTRY_GF(512, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, false, 2, 2),
    LDPC_QC_ENTRY_GF(512, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, false, 2, 2),
    // the same for caller-supplied LLRs
    LDPC_QC_ENTRY_GF(1024, 10, 2, 1, STORE_BF16, ALGO_AMIN, false, true, 2, 1),
    LDPC_QC_ENTRY_GF(1024, 10, 2, 1, STORE_FP16, ALGO_AMIN, false, true, 2, 1),
    LDPC_QC_ENTRY_GF(512, 18, 1, 1, STORE_BF16, ALGO_AMIN, false, true, 2, 2),
    LDPC_QC_ENTRY_GF(512, 18, 1, 1, STORE_FP16, ALGO_AMIN, false, true, 2, 2),
    LDPC_QC_ENTRY_GF(2048, 6, 4, 1, STORE_FP16, ALGO_AMIN, false, true, 0, 0),
    // normalised min-sum and the clips (reference numerics)
    LDPC_QC_ENTRY_GF(2048, 6, 4, 1, STORE_BF16, ALGO_NMS, false, false, 0, 0),
    LDPC_QC_ENTRY_GF(2048, 6, 4, 1, STORE_BF16, ALGO_AMIN, true, false, 0, 0),
    LDPC_QC_ENTRY_GF(2048, 6, 4, 1, STORE_BF16, ALGO_NMS, false, true, 0, 0),
    LDPC_QC_ENTRY_GF(2048, 6, 4, 1, STORE_BF16, ALGO_AMIN, true, true, 0, 0),
    LDPC_QC_ENTRY_GF(1024, 10, 2, 1, STORE_BF16, ALGO_NMS, false, false, 0, 1),
    LDPC_QC_ENTRY_GF(1024, 10, 2, 1, STORE_BF16, ALGO_AMIN, true, false, 0, 1),
    LDPC_QC_ENTRY_GF(1024, 10, 2, 1, STORE_BF16, ALGO_NMS, false, true, 0, 1),
    LDPC_QC_ENTRY_GF(1024, 10, 2, 1, STORE_BF16, ALGO_AMIN, true, true, 0, 1),
    LDPC_QC_ENTRY_GF(512, 18, 1, 1, STORE_BF16, ALGO_NMS, false, false, 2, 2),
    LDPC_QC_ENTRY_GF(512, 18, 1, 1, STORE_BF16, ALGO_AMIN, true, false, 2, 2),
    LDPC_QC_ENTRY_GF_NAN(512, 18, 1, 1, STORE_BF16, ALGO_NMS, true, 2, 2),
    LDPC_QC_ENTRY_GF(512, 18, 1, 1, STORE_BF16, ALGO_AMIN, true, true, 2, 2),
    // clips with fp16 and fp32 storage, caller-supplied LLRs (also the decoding without allocation)
    LDPC_QC_ENTRY_GF(2048, 6, 4, 1, STORE_FP16, ALGO_AMIN, true, true, 0, 0),
    LDPC_QC_ENTRY_G(2048, 6, 4, 1, STORE_FP32, ALGO_AMIN, true, true, 0),
    LDPC_QC_ENTRY_GF(2048, 6, 4, 1, STORE_BF16, ALGO_NMS, true, true, 0, 0),
    LDPC_QC_ENTRY_GF(1024, 10, 2, 1, STORE_FP16, ALGO_AMIN, true, true, 2, 1),
    LDPC_QC_ENTRY_G(1024, 10, 2, 1, STORE_FP32, ALGO_AMIN, true, true, 0),
    LDPC_QC_ENTRY_GF(1024, 10, 2, 1, STORE_BF16, ALGO_NMS, true, true, 0, 1),
    LDPC_QC_ENTRY_GF(512, 18, 1, 1, STORE_FP16, ALGO_AMIN, true, true, 2, 2),
    LDPC_QC_ENTRY_G(512, 18, 1, 1, STORE_FP32, ALGO_AMIN, true, true, 0),
    LDPC_QC_ENTRY_GF(512, 18, 1, 1, STORE_BF16, ALGO_NMS, true, true, 2, 2),
};
LDPC_QC_REGISTER(qc_k16)

// Default shapes.  us of the kernel at 1 / 100 / 440 / 6250 frames, threshold + 1.4 dB, all shapes in one run: the descriptors
// compiled in
//   r1/2 bf16 147 / 187 / 451 / 5816, parameters 165 / 210 / 527 / 6804; fp16 170 / 191 / 532 / 6984 and 182 / 206 / 573 / 7539
//   r2/3 bf16 cap 2 111 / 127 / 297 / 3767, uncapped 108 / 123 / 331 / 4278, parameters 114 / 132 / 356 / 4605; fp16 cap 2 113 / 133 / 360 /
//        4669, parameters 115 / 136 / 370 / 4793
//   r4/5 bf16 cap 2 86.0 / 101 / 231 / 2919, uncapped 88.1 / 102 / 231 / 2917, parameters 88.1 / 104 / 270 / 3520; fp16 cap 2 92.2 / 109 / 244 /
//        3055, parameters 88.9 / 105 / 271 / 3537
// Scaled kernels add up their rows' magnitudes (`hi` of row_update), which takes r2/3 bf16 without a cap past 64 registers, to
// one CTA an SM: 3750 frames 2270 us before, 2598 since, cap 2 2285; caller-supplied LLRs, 500 frames, 367, 423, 378.
// Min-sum and the clips have only these shapes: bf16 r1/2 156 / 195 / 455 / 5853 and 166 / 211 / 526 / 6750, r2/3 97.2 / 128 / 293 /
// 3646 and 124 / 142 / 343 / 4335, r4/5 77.8 / 96.3 / 212 / 2604 and 94.2 / 111 / 282 / 3261 (the general kernel before).
static const QcDefault qc_k16_default[] = {
    {2048, 6, STORE_BF16, -1, 0, 4, 1, 0, 5},
    {2048, 6, STORE_FP16, -1, 0, 4, 1, 0, 5},
    {1024, 10, STORE_BF16, -1, 0, 2, 1, 2, 5},
    {1024, 10, STORE_BF16, -1, 0, 2, 1, 0, 5},
    {1024, 10, STORE_FP16, -1, 0, 2, 1, 2, 5},
    {512, 18, STORE_BF16, -1, 200, 1, 1, 2, 5},
    {512, 18, STORE_BF16, -1, 0, 1, 1, 0, 5},
    {512, 18, STORE_FP16, -1, 200, 1, 1, 2, 5},
};
LDPC_QC_DEFAULTS(qc_k16_default)
