// The two-SM engine over convolution windows as the reduction, FP32 values.
#include "mm_tc2r_launch.cuh"

namespace thc {
namespace mm {

TC2R_ALL(Problem<RawOperand<true, kTf32>, WindowRowsOperand<kTf32>, false, kTf32>)
TC2R_ALL(Problem<WindowRowsOperand<kTf32>, RawOperand<true, kTf32>, false, kTf32>)
TC2R_ALL(Problem<WindowRowsOperand<kTf32>, WindowRowsOperand<kTf32>, false, kTf32>)

}  // namespace mm
}  // namespace thc
