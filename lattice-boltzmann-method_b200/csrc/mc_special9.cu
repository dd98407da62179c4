// The boundary cells' kernel for 9 species (mc_special.cuh).
#include "mc_special.cuh"

template int lbmh::special_step<9, double>(lbmgpu *, const lbm::McArgsT<double, double> &);
template int lbmh::special_step<9, float>(lbmgpu *, const lbm::McArgsT<float, double> &);
