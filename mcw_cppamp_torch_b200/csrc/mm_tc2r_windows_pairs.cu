// The two-SM engine over convolution windows, FP16 pairs.
#include "mm_tc2r_launch.cuh"

namespace thc {
namespace mm {

TC2R_ALL(Problem<PlanesWindowOperand<kPairs>, RawOperand<false, kPairs>, false, kPairs>)
TC2R_NARROW(Problem<PlanesWindowOperand<kPairs>, RawOperand<false, kPairs>, true, kPairs>)

}  // namespace mm
}  // namespace thc
