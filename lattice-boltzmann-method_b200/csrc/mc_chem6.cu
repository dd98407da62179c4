// The stiff chemistry's kernels for 6 species (mc_chem.cuh).
#include "mc_chem.cuh"

template int lbmh::chem_step<6>(lbmgpu *, const lbm::McArgs &);
