// FFT passes of any length (double-float arithmetic) reading complex128; see fft_gen.cuh.
#include "fft_gen.cuh"

int dmg_fft_gen_df_in(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream, int *taken) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return p->sign > 0 ? launch_gen<df, 1, 1>(*p, *b, s, taken) : launch_gen<df, -1, 1>(*p, *b, s, taken);
}
