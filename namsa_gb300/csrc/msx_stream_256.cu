// Persistent all-slices kernel for rows of 256 (msx_stream.cuh).
#include "msx_stream.cuh"

namespace msx {
const StreamOps* stream_ops_256(int ny) { return stream_ops_of<StreamLine256>(ny); }
}  // namespace msx
