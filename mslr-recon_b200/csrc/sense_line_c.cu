// sense_line_c.cu — line kernels of the axis lengths 60,64,72,75.
#include "sense_line.cuh"

namespace mslr {
namespace line {
const LineOps* line_ops_c(int n) { return line_ops_pick<60, 64, 72, 75>(n); }
}  // namespace line
}  // namespace mslr
