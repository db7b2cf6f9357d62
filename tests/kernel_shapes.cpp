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

// a gradient worker's memory as estimated, and the Hamiltonian partials (bytes per set) it allocates
extern "C" double worker_bytes(long long joint, long long mats, long long sets, long long grads, int grid) {
  iqb::AdjointBounds b;
  b.joint_amps = (uint64_t)joint;
  b.mats = (size_t)mats;
  b.sets = (size_t)sets;
  b.grads = (size_t)grads;
  return b.worker_bytes(grid);
}
extern "C" double ham_partial_bytes() { return 8.0 * (double)(iqb::kHamPartials + 1); }
