// The two-SM engine over plain matrices, FP32 values.
#include "mm_tc2r_launch.cuh"

namespace thc {
namespace mm {

TC2R_ALL(Problem<RawOperand<false, kTf32>, RawOperand<false, kTf32>, false, kTf32>)
TC2R_ALL(Problem<RawOperand<true, kTf32>, RawOperand<false, kTf32>, false, kTf32>)
TC2R_ALL(Problem<RawOperand<false, kTf32>, RawOperand<true, kTf32>, false, kTf32>)
TC2R_ALL(Problem<RawOperand<true, kTf32>, RawOperand<true, kTf32>, false, kTf32>)

}  // namespace mm
}  // namespace thc
