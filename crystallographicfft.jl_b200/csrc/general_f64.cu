// Transform stages for channel grids of any 2-3-5 shape, double precision.
#include "general_kernels.cuh"

namespace cfft {

Status general_f64(const FastArgs& a, const GenShape& s, std::string* err) { return gen_unit_launch<double>(a, s, err); }
Status general_init_f64(std::string* err) { return gen_unit_init<double>(err); }

}  // namespace cfft
