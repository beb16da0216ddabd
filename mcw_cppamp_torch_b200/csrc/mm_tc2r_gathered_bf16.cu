// The two-SM engine over gathered windows, BF16: first layers of up to 64 output planes.
#include "mm_tc2r_launch.cuh"

namespace thc {
namespace mm {

TC2R_WIDTH(64, Problem<GatheredWindowOperand, RawOperand<false, kBf16>, false, kBf16>)

}  // namespace mm
}  // namespace thc
