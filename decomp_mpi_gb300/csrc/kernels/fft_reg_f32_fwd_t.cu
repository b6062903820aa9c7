// FFT passes with lines in registers (FP32 arithmetic, forward direction, the form along t); see fft_reg.cuh.
#include "fft_reg.cuh"

int dmg_fft_reg_f32_fwd_t(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream) {
  return launch_reg_form<float, -1, true>(*p, *b, static_cast<cudaStream_t>(stream));
}
