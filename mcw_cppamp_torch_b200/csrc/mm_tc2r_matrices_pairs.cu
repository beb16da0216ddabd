// The two-SM engine over plain matrices, FP16 pairs.
#include "mm_tc2r_launch.cuh"

namespace thc {
namespace mm {

TC2R_ALL(Problem<RawOperand<false, kPairs>, RawOperand<false, kPairs>, false, kPairs>)
TC2R_ALL(Problem<RawOperand<true, kPairs>, RawOperand<false, kPairs>, false, kPairs>)
TC2R_BLOCKS(Problem<RawOperand<false, kPairs>, RawOperand<true, kPairs>, false, kPairs>)
TC2R_BLOCKS(Problem<RawOperand<true, kPairs>, RawOperand<true, kPairs>, false, kPairs>)

}  // namespace mm
}  // namespace thc
