// Persistent all-slices kernel for rows of 768 (msx_stream.cuh).
#include "msx_stream.cuh"

namespace msx {
const StreamOps* stream_ops_768(int ny) { return stream_ops_of<StreamLine768>(ny); }
}  // namespace msx
