// double drains of the uneven stream, orders above 40.
#include "stream_launch.cuh"
namespace tsdx {
namespace host {
TSDX_STREAM_HI(double)
}  // namespace host
}  // namespace tsdx
