// des_mixed.cuh -- launchers of the mixed-precision (DES_PREC_MIXED) kernels.
#pragma once

#include <cuda_runtime.h>

#include "des_common.cuh"

namespace des {

// outputs: also write the strain rate and edvoldt of a fused step (nothing
// in the step that follows reads them); ahead: the strain rate is the
// look-ahead geometry pass's (its shear components in KP::sh32)
int launch_update_stress_mixed(const KP &p, cudaStream_t s, bool fused, bool outputs = true, bool ahead = false);
int launch_strain_rate_mixed(const KP &p, cudaStream_t s);
int launch_heat_gather_mixed(const KP &p, cudaStream_t s);   // heat sums -> p.tdot
// fused step: strain rate + heat terms + dvoldt terms, then the nodal sums and the temperature update
int launch_elem_pass_mixed(const KP &p, cudaStream_t s, bool heat);
// mass_sums: first the compute_mass sums of the look-ahead geometry pass's
// element terms (k_mass_sum's), and the clock advance
int launch_node_pass_mixed(const KP &p, cudaStream_t s, bool heat, bool mass_sums = false);

}  // namespace des
