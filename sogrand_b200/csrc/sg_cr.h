/* sg_cr.h -- the kernels with the correctly rounded exp/log (sg_cr.cu). */
#pragma once
#include <cuda_runtime.h>
#include "sg_code.h"

const void* sg_cr_decode_fn(int v);  /* plain decoder configuration v */
const void* sg_cr_persist_fn(int v); /* batched configuration v */
const void* sg_cr_cluster_fn(int v); /* cluster configuration v */
const void* sg_cr_bitso_fn(int v);   /* line kernel v */
cudaError_t sg_cr_load_code(const sg_code_tables& code);
