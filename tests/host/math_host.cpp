// The CPU's side of math_device.cu.
#include "spc_math.h"

double host_log(std::uint64_t A) { return spc::neg2_log53(A); }
void host_sincos(double x, double &s, double &c) { spc::sincos_in_range(x, s, c); }
void host_turn(std::uint64_t b, double &s, double &c) { spc::sincos_turn53(b, s, c); }
