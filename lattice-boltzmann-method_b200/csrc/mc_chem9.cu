// The stiff chemistry's kernels for 9 species (mc_chem.cuh).
#include "mc_chem.cuh"

template int lbmh::chem_step<9>(lbmgpu *, const lbm::McArgs &);
