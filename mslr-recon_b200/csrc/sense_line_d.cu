// sense_line_d.cu — line kernels of the axis lengths 80,81,90,96.
#include "sense_line.cuh"

namespace mslr {
namespace line {
const LineOps* line_ops_d(int n) { return line_ops_pick<80, 81, 90, 96>(n); }
}  // namespace line
}  // namespace mslr
