// Entry points of the FFT passes (dispatch by arithmetic) and the exponent
// pre-pass of double-float runs.  The passes are the execution of
// runSplitPlan (reference split_fft.c:622-744).
#include "fft_gen.cuh"

// per-arithmetic launchers (fft_pass_f64.cu, fft_pass_f32.cu, fft_pass_df.cu)
size_t dmg_fft_pass_smem_f64(const dmg_fft_pass *p);
size_t dmg_fft_pass_smem_f32(const dmg_fft_pass *p);
size_t dmg_fft_pass_smem_df(const dmg_fft_pass *p);
size_t dmg_fft_pass_smem_tc(const dmg_fft_pass *p);
int dmg_fft_pass_launch_tc(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream);
int dmg_fft_pass_launch_f64(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream);
int dmg_fft_pass_launch_f32(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream);
int dmg_fft_pass_launch_df(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream);
// grouped runtime-length passes (fft_pass_*_mixed.cu)
int dmg_fft_pass_f64_fwd_group(const dmg_fft_group *g, void *stream);
int dmg_fft_pass_f64_inv_group(const dmg_fft_group *g, void *stream);
int dmg_fft_pass_f32_fwd_group(const dmg_fft_group *g, void *stream);
int dmg_fft_pass_f32_inv_group(const dmg_fft_group *g, void *stream);
int dmg_fft_pass_df_fwd_group(const dmg_fft_group *g, void *stream);
int dmg_fft_pass_df_inv_group(const dmg_fft_group *g, void *stream);

// passes with their lines in registers (fft_reg_*.cu)
#define DMG_REG_DECL(a)                                                                    \
  int dmg_fft_reg_##a##_fwd_v(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream); \
  int dmg_fft_reg_##a##_fwd_t(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream); \
  int dmg_fft_reg_##a##_inv_v(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream); \
  int dmg_fft_reg_##a##_inv_t(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream);
DMG_REG_DECL(f64)
DMG_REG_DECL(f32)
DMG_REG_DECL(df)
#undef DMG_REG_DECL
// passes of any length with butterflies in registers (fft_gen_*.cu); taken: whether they ran
int dmg_fft_gen_f64(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream, int *taken);
int dmg_fft_gen_f32(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream, int *taken);
int dmg_fft_gen_df(const dmg_fft_pass *p, const dmg_fft_batch *b, void *stream, int *taken);
int dmg_fft_gen_f64_group(const dmg_fft_group *g, void *stream, int *taken);
int dmg_fft_gen_f32_group(const dmg_fft_group *g, void *stream, int *taken);
int dmg_fft_gen_df_group(const dmg_fft_group *g, void *stream, int *taken);

namespace {

// A pass's lines over every job, as the register kernels number them.
int64_t reg_line_count(const dmg_fft_pass &p, const dmg_fft_batch &b) {
  int64_t n = (int64_t)b.count * p.nv1 * p.nv2;
  for (int i = 0; i < p.nbatch; ++i) n *= p.blen[i];
  return n;
}

int check_batch_dtype(const dmg_fft_pass &p, const dmg_fft_batch &b, int dtype) {
  return dtype == 0 ? check_batch<double>(p, b) : dtype == 2 ? check_batch<df>(p, b) : check_batch<float>(p, b);
}

int launch_reg(const dmg_fft_pass *p, int dtype, const dmg_fft_batch *b, void *stream) {
  const int st = check_batch_dtype(*p, *b, dtype);
  if (st != DMG_OK) return st;
  const bool t = p->reg == DMG_FFT_REG_T, inv = p->sign > 0;
  using launcher = int (*)(const dmg_fft_pass *, const dmg_fft_batch *, void *);
  static const launcher table[3][2][2] = {
      {{dmg_fft_reg_f64_fwd_v, dmg_fft_reg_f64_fwd_t}, {dmg_fft_reg_f64_inv_v, dmg_fft_reg_f64_inv_t}},
      {{dmg_fft_reg_f32_fwd_v, dmg_fft_reg_f32_fwd_t}, {dmg_fft_reg_f32_inv_v, dmg_fft_reg_f32_inv_t}},
      {{dmg_fft_reg_df_fwd_v, dmg_fft_reg_df_fwd_t}, {dmg_fft_reg_df_inv_v, dmg_fft_reg_df_inv_t}}};
  return table[dtype == 3 ? 1 : dtype][inv][t](p, b, stream);
}

// Largest biased exponent of max(|re|, |im|) over every element of a layout.
// Coordinates enumerate the global array in C order; dimensions beyond ndim
// have length 1.
__global__ void __launch_bounds__(256) maxexp_kernel(const dmg_fft_layout lay, int ndim, int L0, int L1, int L2,
                                                     const double2 *__restrict__ src, int32_t *out) {
  const int64_t N = (int64_t)L0 * L1 * L2;
  int best = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
    int x[DMG_FFT_MAXDIM];
    int64_t r = i;
    x[2] = (int)(r % L2);
    r /= L2;
    x[1] = (int)(r % L1);
    x[0] = (int)(r / L1);
    const double2 v = src[layout_addr(lay, ndim, x)];
    const int ea = (int)((__double_as_longlong(v.x) >> 52) & 0x7FF);
    const int eb = (int)((__double_as_longlong(v.y) >> 52) & 0x7FF);
    best = max(best, max(ea, eb));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0 && best > 0) atomicMax(out, best);
}

// The same over a separable layout, a block per row of the last dimension
// at a time: the row's address part is formed once, the threads run along
// the row (contiguous in the usual layouts).
__global__ void __launch_bounds__(256) maxexp_rows_kernel(const dmg_fft_layout lay, int ndim, int L0, int L1, int L2,
                                                          const double2 *__restrict__ src, int32_t *out) {
  const int64_t rows = (int64_t)L0 * L1;
  int best = 0;
  for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
    const int x0 = (int)(r / L1), x1 = (int)(r - (int64_t)x0 * L1);
    const int64_t base = lay.base + __ldg(lay.tab[0] + x0) + (ndim > 1 ? __ldg(lay.tab[1] + x1) : 0);
    for (int x2 = threadIdx.x; x2 < L2; x2 += blockDim.x) {
      const double2 v = src[base + (ndim > 2 ? __ldg(lay.tab[2] + x2) : 0)];
      const int ea = (int)((__double_as_longlong(v.x) >> 52) & 0x7FF);
      const int eb = (int)((__double_as_longlong(v.y) >> 52) & 0x7FF);
      best = max(best, max(ea, eb));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0 && best > 0) atomicMax(out, best);
}

}  // namespace

extern "C" void dmg_fft_reg_radices(int dtype, int n, int reg, int sign, int *first, int *last) {
  const RegSched s = reg_sched(dtype == 3 ? 1 : dtype, n, reg == DMG_FFT_REG_T, sign > 0);
  *first = s.ns > 0 ? s.r[0] : 0;
  *last = s.ns > 0 ? s.r[s.ns - 1] : 0;
}

extern "C" int dmg_fft_tan_entries(int n, int reg, int sign, double *out) {
  const RegSched s = reg_sched(0, n, reg == DMG_FFT_REG_T, sign > 0);
  int at = 0, lp = 1;
  for (int f = 0; f < s.ns; ++f) {
    // (as RegShape<double>::tw_per_j: the twiddled stages' radices are 4 and 8)
    const int r = s.r[f];
    if (f > 0) {
      if (out) tan_table(r, lp, sign, out + 2 * (size_t)at);
      at += r * lp;
    }
    lp *= r;
  }
  return at;
}

extern "C" int dmg_fft_fixed_length(int n) { return fixed_length(n); }

extern "C" int dmg_fft_gen_fits(const dmg_fft_pass *p, int dtype) {
  gen_geom g;
  return dtype == 0 ? gen_make<double>(*p, 1, 0, &g)
                    : dtype == 2 ? gen_make<df>(*p, 1, 0, &g) : gen_make<float>(*p, 1, 0, &g);
}

extern "C" size_t dmg_fft_pass_smem(const dmg_fft_pass *p, int dtype) {
  return dtype == 0 ? dmg_fft_pass_smem_f64(p)
                    : dtype == 1 ? dmg_fft_pass_smem_f32(p)
                                 : dtype == 2 ? dmg_fft_pass_smem_df(p) : dmg_fft_pass_smem_tc(p);
}

extern "C" int dmg_fft_pass_launch_batch(const dmg_fft_pass *p, int dtype, const dmg_fft_batch *b, void *stream) {
  const int64_t most = p->wide ? 2 * DMG_FFT_TILE_MAX : DMG_FFT_TILE_MAX;
  if ((int64_t)p->M1 * p->M2 * p->n > most)
    return dmg_error(DMG_ERR_ARG, "fft tile %d exceeds %lld", p->M1 * p->M2 * p->n, (long long)most);
  if (p->wide && (dtype == 0 || (dtype == 3 && p->n == 1024) || p->radix_runtime || p->n < 8 || p->n > 2048 ||
                  (p->n & (p->n - 1))))
    return dmg_error(DMG_ERR_ARG, "fft pass: wide tiles for length %d in arithmetic %d", p->n, dtype);
  if ((p->perm_in || p->perm_out) && (p->perm_a < 1 || p->perm_b < 1 || (int64_t)p->perm_a * p->perm_b != p->n))
    return dmg_error(DMG_ERR_ARG, "fft slot order %d x %d does not match length %d", p->perm_a, p->perm_b, p->n);
  // (the register kernels number lines in 31 bits)
  if (p->reg && dtype >= 0 && dtype <= 3 && reg_line_count(*p, *b) < ((int64_t)1 << 31)) return launch_reg(p, dtype, b, stream);
  if (p->gen && dtype >= 0 && dtype <= 3) {
    int taken = 0, st = check_batch_dtype(*p, *b, dtype);
    if (st == DMG_OK)
      st = dtype == 0 ? dmg_fft_gen_f64(p, b, stream, &taken)
                      : dtype == 2 ? dmg_fft_gen_df(p, b, stream, &taken) : dmg_fft_gen_f32(p, b, stream, &taken);
    if (st != DMG_OK || taken) return st;
  }
  switch (dtype) {
    case 0: return dmg_fft_pass_launch_f64(p, b, stream);
    case 1: return dmg_fft_pass_launch_f32(p, b, stream);
    case 2: return dmg_fft_pass_launch_df(p, b, stream);
    case 3: return dmg_fft_pass_launch_tc(p, b, stream);
    default: return dmg_error(DMG_ERR_ARG, "fft dtype %d", dtype);
  }
}

static int launch_tiled_group(const dmg_fft_group *g, int dtype, bool inv, void *stream) {
  switch (dtype) {
    case 0: return inv ? dmg_fft_pass_f64_inv_group(g, stream) : dmg_fft_pass_f64_fwd_group(g, stream);
    case 1:
    case 3:  // the tensor-core form has no runtime-length kernel: its passes run in FP32
      return inv ? dmg_fft_pass_f32_inv_group(g, stream) : dmg_fft_pass_f32_fwd_group(g, stream);
    case 2: return inv ? dmg_fft_pass_df_inv_group(g, stream) : dmg_fft_pass_df_fwd_group(g, stream);
    default: return dmg_error(DMG_ERR_ARG, "fft dtype %d", dtype);
  }
}

extern "C" int dmg_fft_pass_launch_group(const dmg_fft_group *g, int dtype, void *stream) {
  if (g->count < 1 || g->count > DMG_FFT_MAXGROUP)
    return dmg_error(DMG_ERR_ARG, "grouped fft pass: %d passes (1 to %d)", g->count, DMG_FFT_MAXGROUP);
  const int sign = g->job[0].p.sign;
  for (int j = 0; j < g->count; ++j) {
    const dmg_fft_pass &p = g->job[j].p;
    if (!p.radix_runtime || p.wide || p.sign != sign)
      return dmg_error(DMG_ERR_ARG, "grouped fft pass %d: needs runtime stages, plain tiles and one direction", j);
    if ((int64_t)p.M1 * p.M2 * p.n > DMG_FFT_TILE_MAX)
      return dmg_error(DMG_ERR_ARG, "fft tile %d exceeds %d", p.M1 * p.M2 * p.n, DMG_FFT_TILE_MAX);
    if ((p.perm_in || p.perm_out) && (p.perm_a < 1 || p.perm_b < 1 || (int64_t)p.perm_a * p.perm_b != p.n))
      return dmg_error(DMG_ERR_ARG, "fft slot order %d x %d does not match length %d", p.perm_a, p.perm_b, p.n);
    const int st = check_batch_dtype(p, g->job[j].bt, dtype);
    if (st != DMG_OK) return st;
  }
  if (dtype < 0 || dtype > 3) return dmg_error(DMG_ERR_ARG, "fft dtype %d", dtype);
  // the passes the any-length register kernel takes run in its launch, the others in the tiled kernel's (the
  // choice depends on the pass alone, so that every plan's results are those of its own run)
  int taken[DMG_FFT_MAXGROUP] = {0}, left = 0;
  const int st = dtype == 0 ? dmg_fft_gen_f64_group(g, stream, taken)
                            : dtype == 2 ? dmg_fft_gen_df_group(g, stream, taken) : dmg_fft_gen_f32_group(g, stream, taken);
  if (st != DMG_OK) return st;
  for (int j = 0; j < g->count; ++j) left += !taken[j];
  if (left == 0) return DMG_OK;
  dmg_fft_group *rest = nullptr;
  if (left < g->count) {
    rest = static_cast<dmg_fft_group *>(malloc(sizeof(dmg_fft_group)));
    if (!rest) return dmg_error(DMG_ERR_NOMEM, "grouped fft pass: out of memory");
    rest->count = 0;
    for (int j = 0; j < g->count; ++j)
      if (!taken[j]) rest->job[rest->count++] = g->job[j];
  }
  const int done = launch_tiled_group(rest ? rest : g, dtype, sign > 0, stream);
  free(rest);
  return done;
}

extern "C" int dmg_fft_pass_launch(const dmg_fft_pass *p, int dtype, const void *src, void *dst, void *stream) {
  dmg_fft_batch b;
  b.count = 1;
  b.src[0] = src;
  b.dst[0] = dst;
  b.scale_exp[0] = p->scale_exp;
  return dmg_fft_pass_launch_batch(p, dtype, &b, stream);
}

extern "C" int dmg_fft_maxexp_launch(const dmg_fft_layout *lay, int ndim, const int32_t *A, const int32_t *L,
                                     const void *src, int32_t *out, void *stream) {
  (void)A;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(out, 0, sizeof(int32_t), s);
  if (e != cudaSuccess) return dmg_error(DMG_ERR_CUDA, "maxexp memset: %s", cudaGetErrorString(e));
  const int L0 = L[0], L1 = ndim > 1 ? L[1] : 1, L2 = ndim > 2 ? L[2] : 1;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (!lay->ranked) {
    const int64_t rows = (int64_t)L0 * L1;
    const int64_t grid = rows < (int64_t)nsm * 8 ? rows : (int64_t)nsm * 8;
    maxexp_rows_kernel<<<(unsigned)grid, 256, 0, s>>>(*lay, ndim, L0, L1, L2, static_cast<const double2 *>(src), out);
  } else {
    maxexp_kernel<<<nsm * 8, 256, 0, s>>>(*lay, ndim, L0, L1, L2, static_cast<const double2 *>(src), out);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return dmg_error(DMG_ERR_CUDA, "maxexp launch: %s", cudaGetErrorString(e));
  return DMG_OK;
}
