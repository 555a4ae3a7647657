// sense_line_a.cu — line kernels of the axis lengths 8,9,10,12,15,16,18,20,24,25,27,30,32,36.
#include "sense_line.cuh"

namespace mslr {
namespace line {
const LineOps* line_ops_a(int n) { return line_ops_pick<8, 9, 10, 12, 15, 16, 18, 20, 24, 25, 27, 30, 32, 36>(n); }
}  // namespace line
}  // namespace mslr
