// Kernel variants of the circulant engine's decoder (ALGO_CIRC: pairwise min* tree, damping, its
// stop rules and tally) for the rate-1/2 AR4JA codes, the only ones with rows of degrees 3 and 6.
#include "ldpc_qc.cuh"
#include "ldpc_registry.h"

using namespace ldpcb200;

static const QcEntry qc_circ[] = {
    // K = 1024 (Z = 128): bf16 is the engine's storage; fp32 keeps L and r unrounded
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_CIRC, false, false),
    LDPC_QC_ENTRY_OT(128, 6, 1, 1, STORE_BF16, ALGO_CIRC, false, false, 0),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_BF16, ALGO_CIRC, false, true),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP32, ALGO_CIRC, false, false),
    LDPC_QC_ENTRY(128, 6, 1, 1, STORE_FP32, ALGO_CIRC, false, true),
    // K = 4096 (Z = 512)
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_BF16, ALGO_CIRC, false, false),
    LDPC_QC_ENTRY(512, 6, 1, 1, STORE_BF16, ALGO_CIRC, false, true),
    // K = 16384 (Z = 2048): check messages in global memory, 512 threads x 4 rows
    LDPC_QC_ENTRY_G(2048, 6, 4, 1, STORE_BF16, ALGO_CIRC, false, false, 0),
    LDPC_QC_ENTRY_G(2048, 6, 4, 1, STORE_BF16, ALGO_CIRC, false, true, 0),
    // layout 6: the code's layer descriptors compiled in
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_BF16, ALGO_CIRC, false, false, 5, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_BF16, ALGO_CIRC, false, true, 5, 5),
    LDPC_QC_ENTRY_RF(128, 6, 1, 1, STORE_FP32, ALGO_CIRC, false, false, 5, 5),
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_BF16, ALGO_CIRC, false, false, 2, 6),
    LDPC_QC_ENTRY_RF(512, 6, 1, 1, STORE_BF16, ALGO_CIRC, false, true, 2, 6),
};
LDPC_QC_REGISTER(qc_circ)

// Defaults.  us of the kernel at 440 / 5000 / 100000 frames (440 / 1500 / 25000 for K = 4096), 2.04 dB, all shapes in one run: bf16
// layout 6 51.9 / 334 / 6160, offset table 57.3 / 350 / 6374, parameters 57.4 / 420 / 7964; fp32 37.8 / 254 / 4654 and 45.1 / 316 /
// 5888; K = 4096 135 / 428 / 6440 and 167 / 524 / 8011.  K = 16384 keeps the parameter kernel: with the descriptors compiled in
// it spills and took 1.14 times as long.
static const QcDefault qc_circ_default[] = {
    {128, 6, STORE_BF16, ALGO_CIRC, 0, 1, 1, 5, 6},
    {128, 6, STORE_BF16, ALGO_CIRC, 440, 1, 1, 0, 2},
    {128, 6, STORE_FP32, ALGO_CIRC, 440, 1, 1, 5, 6},
    {512, 6, STORE_BF16, ALGO_CIRC, 300, 1, 1, 2, 6},
};
LDPC_QC_DEFAULTS(qc_circ_default)
