// FFT passes of any length with butterflies in registers (double-float arithmetic, both directions); see fft_gen.cuh.
#include "fft_gen.cuh"

// passes that convert complex128 in their first or last stage (fft_gen_df_{in,out}.cu)
int dmg_fft_gen_df_in(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream, int *taken);
int dmg_fft_gen_df_out(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream, int *taken);

int dmg_fft_gen_df(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream, int *taken) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (gen_conv<df>(*p)) {
    case 1: return dmg_fft_gen_df_in(p, b, stream, taken);
    case 2: return dmg_fft_gen_df_out(p, b, stream, taken);
    default: return p->sign > 0 ? launch_gen<df, 1>(*p, *b, s, taken) : launch_gen<df, -1>(*p, *b, s, taken);
  }
}

int dmg_fft_gen_df_group(const dmg_fft_group *g, void *stream, int *taken) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return g->job[0].p.sign > 0 ? launch_gen_group<df, 1>(*g, s, taken) : launch_gen_group<df, -1>(*g, s, taken);
}
