// FFT passes of any length with butterflies in registers (FP32 arithmetic, both directions); see fft_gen.cuh.
#include "fft_gen.cuh"

int dmg_fft_gen_f32(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream, int *taken) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return p->sign > 0 ? launch_gen<float, 1>(*p, *b, s, taken) : launch_gen<float, -1>(*p, *b, s, taken);
}

int dmg_fft_gen_f32_group(const dmg_fft_group *g, void *stream, int *taken) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return g->job[0].p.sign > 0 ? launch_gen_group<float, 1>(*g, s, taken) : launch_gen_group<float, -1>(*g, s, taken);
}
