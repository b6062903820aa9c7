// FFT passes with lines in registers (native FP64 arithmetic, forward direction, the form along v1); see fft_reg.cuh.
#include "fft_reg.cuh"

int dmg_fft_reg_f64_fwd_v(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream) {
  return launch_reg_form<double, -1, false>(*p, *b, static_cast<cudaStream_t>(stream));
}
