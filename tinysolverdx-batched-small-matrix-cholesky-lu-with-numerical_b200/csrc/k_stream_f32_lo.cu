// float drains of the uneven stream, orders up to 40.
#include "stream_launch.cuh"
namespace tsdx {
namespace host {
TSDX_STREAM_LO(float)
}  // namespace host
}  // namespace tsdx
