// The two-SM engine over plain matrices, BF16 values.
#include "mm_tc2r_launch.cuh"

namespace thc {
namespace mm {

TC2R_ALL(Problem<RawOperand<false, kBf16>, RawOperand<false, kBf16>, false, kBf16>)
TC2R_BLOCKS(Problem<RawOperand<true, kBf16>, RawOperand<true, kBf16>, false, kBf16>)

}  // namespace mm
}  // namespace thc
