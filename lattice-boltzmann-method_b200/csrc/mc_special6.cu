// The boundary cells' kernel for 6 species (mc_special.cuh).
#include "mc_special.cuh"

template int lbmh::special_step<6, double>(lbmgpu *, const lbm::McArgsT<double, double> &);
template int lbmh::special_step<6, float>(lbmgpu *, const lbm::McArgsT<float, double> &);
