// The chemistry's kernels for 6 species (mc_chem.cuh).
#include "mc_chem.cuh"

template int lbmh::chem_step<6>(lbmgpu *, const lbm::McArgs &, cudaStream_t);
template int lbmh::explicit_step<6, double>(lbmgpu *, const lbm::McArgsT<double, double> &, cudaStream_t);
template int lbmh::explicit_step<6, float>(lbmgpu *, const lbm::McArgsT<float, double> &, cudaStream_t);
