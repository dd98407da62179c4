// The chemistry's kernels for 9 species (mc_chem.cuh).
#include "mc_chem.cuh"

template int lbmh::chem_step<9>(lbmgpu *, const lbm::McArgs &, cudaStream_t);
template int lbmh::explicit_step<9, double>(lbmgpu *, const lbm::McArgsT<double, double> &, cudaStream_t);
template int lbmh::explicit_step<9, float>(lbmgpu *, const lbm::McArgsT<float, double> &, cudaStream_t);
