// Whether a device takes an optional kernel form, asked once per plan and form.
#pragma once
#include <cuda_runtime.h>

namespace msx {

struct FormState {
  int state = 0;  // 0: not asked, 1: taken, -1: refused (the plan then does without)
  // configure: cudaError_t(); a refusal leaves no error behind
  template <class F>
  bool ready(F configure) {
    if (state == 0) {
      state = configure() == cudaSuccess ? 1 : -1;
      if (state < 0) cudaGetLastError();
    }
    return state > 0;
  }
};

}  // namespace msx
