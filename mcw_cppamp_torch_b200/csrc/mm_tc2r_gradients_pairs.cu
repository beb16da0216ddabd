// The two-SM engine over convolution windows as the reduction, FP16 pairs.
#include "mm_tc2r_launch.cuh"

namespace thc {
namespace mm {

TC2R_BLOCKS(Problem<RawOperand<true, kPairs>, WindowRowsOperand<kPairs>, false, kPairs>)
TC2R_BLOCKS(Problem<WindowRowsOperand<kPairs>, RawOperand<true, kPairs>, false, kPairs>)
TC2R_BLOCKS(Problem<WindowRowsOperand<kPairs>, WindowRowsOperand<kPairs>, false, kPairs>)

}  // namespace mm
}  // namespace thc
