// sense_line_b.cu — line kernels of the axis lengths 40,45,48,50,54.
#include "sense_line.cuh"

namespace mslr {
namespace line {
const LineOps* line_ops_b(int n) { return line_ops_pick<40, 45, 48, 50, 54>(n); }
}  // namespace line
}  // namespace mslr
