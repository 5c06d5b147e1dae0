// Persistent all-slices kernel for rows of 384 (msx_stream.cuh).
#include "msx_stream.cuh"

namespace msx {
const StreamOps* stream_ops_384(int ny) { return stream_ops_of<StreamLine384>(ny); }
}  // namespace msx
