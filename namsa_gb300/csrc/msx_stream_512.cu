// Persistent all-slices kernel for rows of 512 (msx_stream.cuh).
#include "msx_stream.cuh"

namespace msx {
const StreamOps* stream_ops_512(int ny) { return stream_ops_of<StreamLine512>(ny); }
}  // namespace msx
