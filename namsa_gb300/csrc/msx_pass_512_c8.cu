// The 512 schedule of four-warp CTAs (see msx_pass_512.cu).
#include "msx_sched.cuh"

namespace msx {
SchedOps schedule_512_c8() { return SchedImpl<Sched<512, 16, 8, 2, 32, 16>>::ops("t16_r32x16_c8"); }
}  // namespace msx
