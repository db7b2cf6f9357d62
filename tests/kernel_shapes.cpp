// Host-side launch arithmetic of the kernels, for the CPU tests (tests/test_kernel_shapes.py).
#include "../invariantq_b200/csrc/iq_kernels.h"

extern "C" void hh_shape_of(int n, int sms, long long* out) {
  const iqb::HhShape h = iqb::hh_shape(n, sms);
  out[0] = h.smem_rows;
  out[1] = h.threads;
  out[2] = h.rows;
  out[3] = h.grid;
  out[4] = (long long)h.smem;
}
