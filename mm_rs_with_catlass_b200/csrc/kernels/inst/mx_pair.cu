// Instantiates the fused kernel for one operand kind and CTA flavour (see kernel_inst.cuh).
#include "catcoc/kernel_inst.cuh"

CATCOC_DEFINE_UNIT_PLAIN(mx_pair, catcoc::KIND_MX, true)
