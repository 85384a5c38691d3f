// Transform stages for channel grids of any 2-3-5 shape, float precision.
#include "general_kernels.cuh"

namespace cfft {

Status general_f32(const FastArgs& a, const GenShape& s, std::string* err) { return gen_unit_launch<float>(a, s, err); }
Status general_init_f32(std::string* err) { return gen_unit_init<float>(err); }

}  // namespace cfft
