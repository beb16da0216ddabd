// The two-SM engine over convolution windows, FP32 values.
#include "mm_tc2r_launch.cuh"

namespace thc {
namespace mm {

TC2R_ALL(Problem<PlanesWindowOperand<kTf32>, RawOperand<false, kTf32>, false, kTf32>)
TC2R_NARROW(Problem<PlanesWindowOperand<kTf32>, RawOperand<false, kTf32>, true, kTf32>)

}  // namespace mm
}  // namespace thc
