/* sg_cr.cu -- the decoder kernels with the correctly rounded exp/log (math
 * mode 1). */
#define SG_TU_CR true
#define SG_K_ARGS /* constants as launch arguments (sg_math.h) */
#include "sg_cr.h"
#include "sg_kernels.cuh"

const void* sg_cr_decode_fn(int v) { return k_variants[v].fn; }
const void* sg_cr_persist_fn(int v) { return k_pvariants[v].fn; }
const void* sg_cr_cluster_fn(int v) { return k_cvariants[v].fn; }
const void* sg_cr_bitso_fn(int v) { return k_bvariants[v].fn; }
cudaError_t sg_cr_load_code(const sg_code_tables& code) { return sg_load_code(code); }
