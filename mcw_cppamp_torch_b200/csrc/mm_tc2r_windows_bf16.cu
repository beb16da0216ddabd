// The two-SM engine over convolution windows, BF16 values.
#include "mm_tc2r_launch.cuh"

namespace thc {
namespace mm {

TC2R_ALL(Problem<PlanesWindowOperand<kBf16>, RawOperand<false, kBf16>, false, kBf16>)

}  // namespace mm
}  // namespace thc
