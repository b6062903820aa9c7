// FFT passes of any length, and of sides with per-rank strides, with a
// thread's butterflies in registers; alone, or several passes of different
// plans in one launch.
//
// The register kernels of fft_reg.cuh are compiled per length.  This kernel
// takes a pass's radices at run time (2 to 10, and 12, 14, 15, 16 in FP32,
// compiled one after the other; larger primes as direct DFTs): a block holds
// W lines, each stage's butterflies are spread over all threads, the first
// stage reads its values straight from the input layout, the last writes
// them straight to the output layout, and the values in between cross shared
// memory once per stage.  fft_pass.cuh's runtime stages did this with
// radices up to 8 only, every access predicated on the radix, a division and
// a table read in global memory per value, and two more trips through shared
// memory; ranked sides cost it a dozen table reads per value.
//
// Ranked sides (strides that differ between virtual ranks): along a line the
// rank only depends on the transform coordinate's process position, so a
// block tabulates, per line and position, the address of that rank's first
// value and its stride; a value then costs three shared-memory reads and one
// multiply-add.
//
// Measured on one GB300 against the tiled kernel's runtime stages (GB/s of a
// pass's bytes over 2^27 FP32 or 2^26 other values, along t / along v1):
// 105 points FP32 680 / 700 -> 2070 / 2680, double-float 520 / 590 -> 975 /
// 1575, native FP64 223 / 225 -> 527 / 531; 360 points FP32 540 / 810 -> 1600
// / 1880, native FP64 379 / 409 -> 464 / 471.  180 x 150 x 105 complex128
// double-float with uneven blocks 508 -> 267 us; 16 uneven small cubes in one
// launch per pass, native FP64, 488 -> 346 us.
#pragma once
#include "fft_reg.cuh"

namespace {

#define K_C7_1 0.623489801858733530525004884004239810, 0.6234897971153259f, 4.743407444607328e-09f
#define K_S7_1 0.781831482468029808708444526674057750, 0.7818315029144287f, -2.0446398352191864e-08f
#define K_C7_2 -0.22252093395631440428890256449679475, -0.22252093255519867f, -1.4011157789539652e-09f
#define K_S7_2 0.974927912181823607018131682993931217, 0.9749279022216797f, 9.960143820819667e-09f
#define K_C7_3 -0.90096886790241912623610231950744505, -0.9009688496589661f, -1.8243452970523322e-08f
#define K_S7_3 0.433883739117558120475768332848358754, 0.4338837265968323f, 1.252072578949992e-08f
#define K_C9_1 0.766044443118978035202392650555416673, 0.7660444378852844f, 5.2336934786012534e-09f
#define K_S9_1 0.642787609686539326322643409907263432, 0.6427876353263855f, -2.5639845802061245e-08f
#define K_C9_2 0.173648177666930348851716626769314796, 0.1736481785774231f, -9.10492736760915e-10f
#define K_S9_2 0.984807753012208059366743024589523013, 0.9848077297210693f, 2.3291137907222037e-08f
#define K_C9_4 -0.93969262078590838405410927732473146, -0.9396926164627075f, -4.323200908373792e-09f
#define K_S9_4 0.342020143325668733044099614682259580, 0.3420201539993286f, -1.0673660177928923e-08f

// ---------------------------------------------------------------- radices

template <typename T, int SIGN>
__device__ __forceinline__ void rdft7(C2<T> *a) {
  // sums and differences of the pairs q, 7 - q: three cosines and three sines
  const C2<T> s1 = add<T>(a[1], a[6]), s2 = add<T>(a[2], a[5]), s3 = add<T>(a[3], a[4]);
  const C2<T> d1 = sub<T>(a[1], a[6]), d2 = sub<T>(a[2], a[5]), d3 = sub<T>(a[3], a[4]);
  const T c1 = cst<T>(K_C7_1), c2 = cst<T>(K_C7_2), c3 = cst<T>(K_C7_3);
  const T n1 = cst<T>(K_S7_1), n2 = cst<T>(K_S7_2), n3 = cst<T>(K_S7_3);
  const C2<T> x0 = a[0];
  C2<T> p1, p2_, p3;
  if constexpr (std::is_same<T, df>::value) {
    p1 = add<T>(x0, add<T>(scl<T>(s1, c1), add<T>(scl<T>(s2, c2), scl<T>(s3, c3))));
    p2_ = add<T>(x0, add<T>(scl<T>(s1, c2), add<T>(scl<T>(s2, c3), scl<T>(s3, c1))));
    p3 = add<T>(x0, add<T>(scl<T>(s1, c3), add<T>(scl<T>(s2, c1), scl<T>(s3, c2))));
  } else {
    p1 = mac<T>(mac<T>(mac<T>(x0, s3, c3), s2, c2), s1, c1);
    p2_ = mac<T>(mac<T>(mac<T>(x0, s2, c3), s1, c2), s3, c1);
    p3 = mac<T>(mac<T>(mac<T>(x0, s1, c3), s3, c2), s2, c1);
  }
  const C2<T> q1 = mac<T>(mac<T>(scl<T>(d3, n3), d2, n2), d1, n1);
  const C2<T> q2 = mac<T>(mac<T>(scl<T>(d1, n2), d2, rneg(n3)), d3, rneg(n1));
  const C2<T> q3 = mac<T>(mac<T>(scl<T>(d1, n3), d2, rneg(n1)), d3, n2);
  a[0] = add<T>(x0, add<T>(s1, add<T>(s2, s3)));
  a[1] = add_rot<T, SIGN>(p1, q1);
  a[6] = sub_rot<T, SIGN>(p1, q1);
  a[2] = add_rot<T, SIGN>(p2_, q2);
  a[5] = sub_rot<T, SIGN>(p2_, q2);
  a[3] = add_rot<T, SIGN>(p3, q3);
  a[4] = sub_rot<T, SIGN>(p3, q3);
}
// v exp(sign i angle)
template <typename T, int SIGN>
__device__ __forceinline__ C2<T> rturn(C2<T> v, T c, T s) {
  return rmul<T>(v, pack_c(c, SIGN < 0 ? rneg(s) : s));
}
template <typename T, int SIGN>
__device__ __forceinline__ void rdft9(C2<T> *a) {
  C2<T> y[3][3];
#pragma unroll
  for (int i2 = 0; i2 < 3; ++i2) {
#pragma unroll
    for (int i1 = 0; i1 < 3; ++i1) y[i2][i1] = a[3 * i1 + i2];
    rdft3<T, SIGN>(y[i2]);
  }
  y[1][1] = rturn<T, SIGN>(y[1][1], cst<T>(K_C9_1), cst<T>(K_S9_1));
  y[1][2] = rturn<T, SIGN>(y[1][2], cst<T>(K_C9_2), cst<T>(K_S9_2));
  y[2][1] = rturn<T, SIGN>(y[2][1], cst<T>(K_C9_2), cst<T>(K_S9_2));
  y[2][2] = rturn<T, SIGN>(y[2][2], cst<T>(K_C9_4), cst<T>(K_S9_4));
#pragma unroll
  for (int k1 = 0; k1 < 3; ++k1) {
    C2<T> z[3] = {y[0][k1], y[1][k1], y[2][k1]};
    rdft3<T, SIGN>(z);
#pragma unroll
    for (int k2 = 0; k2 < 3; ++k2) a[k1 + 3 * k2] = z[k2];
  }
}
// Native FP64, eight points: the odd eighth turns as w - (1 - 1/sqrt(2)) w of w = (1 + sign i) v.  The rounding error
// of 1/sqrt(2) (0.62 units of 2^-53, upwards) would scale a quarter of every stage's values alike; the tiled kernel's
// partly makes up for that of its sqrt(3)/2 (0.52 downwards), which rdft3 no longer has, and 384 to 1536 points were 3
// to 4 % further off with it.  So it is 0.09, for four operations more per eight values.
template <int SIGN>
__device__ __forceinline__ void gdft8_f64(double2 *a) {
  double2 e0 = a[0], e1 = a[2], e2 = a[4], e3 = a[6];
  double2 o0 = a[1], o1 = a[3], o2 = a[5], o3 = a[7];
  rdft4<double, SIGN>(e0, e1, e2, e3);
  rdft4<double, SIGN>(o0, o1, o2, o3);
  const double k = -0.292893218813452475599155637895150961;
  double2 w1 = add_rot<double, SIGN>(o1, o1), w3 = sub_rot<double, SIGN>(o3, o3);  // (w3: subtracted below)
  w1 = mac<double>(w1, w1, k);
  w3 = mac<double>(w3, w3, k);
  a[0] = cadd(e0, o0);
  a[4] = csub(e0, o0);
  a[1] = cadd(e1, w1);
  a[5] = csub(e1, w1);
  a[2] = add_rot<double, SIGN>(e2, o2);
  a[6] = sub_rot<double, SIGN>(e2, o2);
  a[3] = csub(e3, w3);
  a[7] = cadd(e3, w3);
}
template <typename T, int SIGN, int R>
__device__ __forceinline__ void gdft(C2<T> *a) {
  if constexpr (R == 8 && std::is_same<T, double>::value) {
    gdft8_f64<SIGN>(a);
  } else if constexpr (R == 7) {
    rdft7<T, SIGN>(a);
  } else if constexpr (R == 9) {
    rdft9<T, SIGN>(a);
  } else if constexpr (R == 14) {
    // 2 x 7, coprime: input 7 i1 + 2 i2, output 7 k1 + 8 k2
    C2<T> e[7], o[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) {
      const C2<T> u = a[(2 * i) % 14], v = a[(7 + 2 * i) % 14];
      e[i] = add<T>(u, v);
      o[i] = sub<T>(u, v);
    }
    rdft7<T, SIGN>(e);
    rdft7<T, SIGN>(o);
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      a[(8 * k) % 14] = e[k];
      a[(7 + 8 * k) % 14] = o[k];
    }
  } else {
    rdft<T, SIGN, R>(a);
  }
}

// ---------------------------------------------------------------- geometry

// Threads per block (the launch's choice) and the values a block holds per
// thread: 512 threads per SM at 128 registers in any case, in small blocks
// for short lines (more of them in different phases, less to wait for at a
// barrier), in larger ones where a line needs the room.
constexpr int GEN_MAXNT = 512;
constexpr int GEN_SMS = 152;  // GB300's (the geometry is also made where there is no device to ask)
template <typename T>
constexpr int gen_per_thread() {
  return std::is_same<T, float>::value ? 16 : 8;
}
constexpr int GEN_STAGES = 12;
constexpr int GEN_MAXPOS = 64;       // process positions of a ranked side along the transform axis

// r = 1: moves values between a layout and the buffers (before or after a direct prime stage)
struct gen_stage {
  int32_t r, lp, m, nb;
  uint32_t m_mul, m_sh, nb_mul, nb_sh;  // divisions by m and nb
  int32_t pin, pout;                    // row pitches of the exchanges before and after
};
struct gen_side {
  int32_t ranked, np, rstep;  // ranked: positions along the transform axis, rank step between them
};
struct gen_geom {
  int32_t nst, w, nt;
  uint32_t w_mul, w_sh, n_mul, n_sh;
  int32_t s1, s2;              // buffer strides of a line's position and of a line
  int32_t load_t, store_t;     // lanes run along t (else along the lines) on that side
  int32_t slot_in, slot_out;   // read / write in slot order through the buffer
  int32_t srow_in, spitch_in, srow_out, spitch_out;
  uint32_t off_b, off_roots, off_tin, off_tout, off_lin, off_lout, off_lx;  // shared memory
  uint32_t smem;
  gen_side in, out;
  gen_stage st[GEN_STAGES];
};
__host__ __device__ inline void gen_divisor(uint32_t d, uint32_t *mul, uint32_t *sh) {
  uint32_t l = 0;
  while ((1ull << l) < (uint64_t)d) ++l;
  *sh = l;
  *mul = (uint32_t)(((1ull << 32) * ((1ull << l) - (uint64_t)d)) / (uint64_t)d + 1);
}
__device__ __forceinline__ uint32_t gen_div(uint32_t r, uint32_t mul, uint32_t sh) { return (__umulhi(r, mul) + r) >> sh; }

// whether a radix has a butterfly in registers
template <typename T>
constexpr bool gen_radix(int r) {
  return (r >= 2 && r <= 10) || (std::is_same<T, float>::value && (r == 12 || r == 14 || r == 15 || r == 16));
}

// Double-float passes that convert complex128 at one end have kernels whose
// first (1) or last (2) stage converts; with that long code in every radix
// the passes without conversions ran out of the instruction cache (105
// points along v1: 990 against 1570 GB/s).  0: conversions, where due, in
// stages of radix 1.
template <typename T>
int gen_conv(const dmg_fft_pass &p) {
  if (!std::is_same<T, df>::value) return 0;
  if (p.in_fp64 && !p.out_fp64 && p.twiddle != 2) return 1;
  if (p.out_fp64 && !p.in_fp64 && p.twiddle != 1) return 2;
  return 0;
}

// The fewest stages, then the smallest sum of radices, over the radices
// above: list gets them largest first.  Returns the stage count, or 0 when n
// has a larger prime factor.
template <typename T>
int gen_radices(int n, int *list) {
  int best = 0, sum = 0, cur[GEN_STAGES];
  auto walk = [&](auto &&self, int rest, int most, int depth, int total) -> void {
    if (rest == 1) {
      if (depth > 0 && (!best || depth < best || (depth == best && total < sum))) {
        best = depth;
        sum = total;
        for (int i = 0; i < depth; ++i) list[i] = cur[i];
      }
      return;
    }
    if (depth >= 8 || (best && depth + 1 > best)) return;
    for (int r = most; r >= 2; --r)
      if (gen_radix<T>(r) && rest % r == 0) {
        cur[depth] = r;
        self(self, rest / r, r, depth + 1, total + r);
      }
  };
  walk(walk, n, 16, 0, 0);
  return best;
}

// Geometry of a pass over `lines` lines (nt: the threads per block, 0 to choose); false when it does not fit.
template <typename T>
bool gen_make(const dmg_fft_pass &p, int64_t lines, int nt, gen_geom *g, int conv = 0) {
  memset(g, 0, sizeof(*g));
  const int es = (int)sizeof(C2<T>), n = p.n, V = 128 / es;
  int rad[2 * DMG_FFT_MAXFAC], nr = 0;
  int own[GEN_STAGES], no = p.radix_runtime ? 0 : gen_radices<T>(n, own);
  // double-float: values converted (or multiplied by the split twiddle) in a stage of their own at that end
  // where the kernel's stages do not (see gen_conv)
  const bool dfl = std::is_same<T, df>::value;
  const bool pre = dfl && ((p.in_fp64 && conv != 1) || p.twiddle == 2);
  const bool post = dfl && ((p.out_fp64 && conv != 2) || p.twiddle == 1);
  if (pre) rad[nr++] = 1;
  if (no > 0) {
    for (int i = 0; i < no; ++i) rad[nr++] = own[i];
  } else {
    // the plan's radices; a prime without a butterfly reads its values from the buffers
    for (int i = 0; i < p.nfac; ++i) {
      const bool big = !gen_radix<T>(p.fac[i]);
      if (big && i == 0 && !pre) rad[nr++] = 1;
      rad[nr++] = p.fac[i];
      if (big && i == p.nfac - 1 && !post) rad[nr++] = 1;
    }
  }
  if (post) rad[nr++] = 1;
  if (nr < 1 || nr > GEN_STAGES) return false;
  g->nst = nr;
  g->load_t = p.load_order[0] == 0;
  g->store_t = p.store_order[0] == 0;
  g->slot_in = g->load_t && p.perm_in;
  g->slot_out = g->store_t && p.perm_out;
  g->in.ranked = p.in.ranked;
  g->out.ranked = p.out.ranked;
  g->in.np = p.in.ranked ? p.gen_np_in : 1;
  g->out.np = p.out.ranked ? p.gen_np_out : 1;
  g->in.rstep = p.gen_rstep_in;
  g->out.rstep = p.gen_rstep_out;
  if (g->in.np > GEN_MAXPOS || g->out.np > GEN_MAXPOS) return false;
  const bool both_v = !g->load_t && !g->store_t;
  int lp = 1;
  for (int f = 0; f < nr; ++f) {
    gen_stage &s = g->st[f];
    s.r = rad[f];
    s.lp = lp;
    lp *= rad[f];
    s.m = n / lp;
    s.nb = n / rad[f];
    gen_divisor((uint32_t)s.m, &s.m_mul, &s.m_sh);
    gen_divisor((uint32_t)s.nb, &s.nb_mul, &s.nb_sh);
  }
  if (lp != n) return false;
  gen_divisor((uint32_t)n, &g->n_mul, &g->n_sh);
  g->srow_in = g->st[0].m;
  g->spitch_in = g->srow_in | 1;
  g->srow_out = g->st[nr - 1].lp;
  g->spitch_out = g->srow_out | 1;
  // threads for rows of 64 bytes along the lines, then the lines their registers hold
  const int row = both_v || !g->load_t || !g->store_t ? 64 / es : 2;
  g->nt = nt;
  if (!nt) {
    g->nt = 128;
    while (g->nt < GEN_MAXNT && g->nt * gen_per_thread<T>() < row * n) g->nt *= 2;
  }
  int w = g->nt * gen_per_thread<T>() / n;
  if (w < 1) w = 1;
  // (enough blocks for every SM where that leaves a warp of butterflies each)
  while (w > 1 && (lines + w - 1) / w < 2 * GEN_SMS && (w / 2) * n >= 32 * gen_per_thread<T>()) w /= 2;
  if (w >= 8) w &= ~3;
  // and, with more blocks than SMs, the threads for the lines that are left, as long as their block fits (in a 512-thread
  // block per SM over single lines 400 threads had nothing to do: 720 points along v1, 512 lines, double-float 54 us and
  // 33 in the tiled kernel, 29 so; native FP64 600 points 62, 47 and 40)
  const int most = g->nt;
  if (!nt && (lines + w - 1) / w > GEN_SMS)
    while (g->nt > 128 && g->nt / 2 * gen_per_thread<T>() >= w * n) g->nt /= 2;
  // and, with one block per SM, fewer lines where that shortens the last wave (rounds of blocks times lines) and leaves
  // half of the threads' work: 1080 points along v1, 1024 lines, native FP64 144 us with three (three rounds, the last a
  // quarter full), 122 in the tiled kernel, 124 with two; 1250 points 160, 148 and 148
  if (!nt && g->nt == GEN_MAXNT) {
    auto line_times = [&](int v) { return ((lines + v - 1) / v + GEN_SMS - 1) / GEN_SMS * v; };
    for (int v = w - 1; v >= 1 && 2 * v * n >= g->nt * gen_per_thread<T>(); --v)
      if ((v < 8 || v % 4 == 0) && 20 * line_times(v) < 19 * line_times(w)) w = v;
  }
  for (;;) {
    g->w = w;
    gen_divisor((uint32_t)w, &g->w_mul, &g->w_sh);
    // row pitches: neighbouring threads of the reading stage in different banks
    const int lanes = both_v ? (w >= V ? 1 : V / w) : V;
    int64_t line = n;
    for (int f = 0; f + 1 < nr; ++f) {
      int m = g->st[f].m, pitch = m;
      const int mn = g->st[f + 1].m;
      if (mn < lanes && (mn & (mn - 1)) == 0)
        while (pitch % (2 * mn) != mn) ++pitch;
      g->st[f].pout = g->st[f + 1].pin = pitch;
      if ((int64_t)g->st[f].lp * g->st[f].r * pitch > line) line = (int64_t)g->st[f].lp * g->st[f].r * pitch;
    }
    if (g->slot_in && (int64_t)(n / g->srow_in) * g->spitch_in > line) line = (int64_t)(n / g->srow_in) * g->spitch_in;
    if (g->slot_out && (int64_t)(n / g->srow_out) * g->spitch_out > line)
      line = (int64_t)(n / g->srow_out) * g->spitch_out;
    g->s1 = both_v ? w : 1;
    g->s2 = both_v ? 1 : (int)(line | 1);
    const size_t buf = (((size_t)w * (size_t)(both_v ? line : line | 1)) * es + 15) & ~(size_t)15;
    size_t pos = buf;
    g->off_b = (uint32_t)pos;
    pos += buf;
    g->off_roots = (uint32_t)pos;
    pos += (size_t)n * es;
    pos = (pos + 15) & ~(size_t)15;
    g->off_tin = (uint32_t)pos;
    pos += (size_t)n * 8;
    g->off_tout = (uint32_t)pos;
    pos += (size_t)n * 8;
    g->off_lin = (uint32_t)pos;
    pos += (size_t)w * g->in.np * 16;
    g->off_lout = (uint32_t)pos;
    pos += (size_t)w * g->out.np * 16;
    g->off_lx = (uint32_t)pos;
    pos += (size_t)w * 8;
    g->smem = (uint32_t)((pos + 15) & ~(size_t)15);
    if (g->smem <= 232448 / (512 / g->nt) - 1024) break;
    if (g->nt < most) g->nt *= 2;
    else if (--w < 1) return false;
  }
  return true;
}

// ---------------------------------------------------------------- the pass

// A value of the layouts by its address as an integer: the intrinsics say
// that it is global (a pass never writes the array half it reads).
template <typename T>
__device__ __forceinline__ C2<T> gen_load(long long at) {
  C2<T> r;
  if constexpr (sizeof(C2<T>) == 16) {
    const float4 v = __ldg(reinterpret_cast<const float4 *>(at));
    memcpy(&r, &v, 16);
  } else {
    r = __ldg(reinterpret_cast<const C2<T> *>(at));
  }
  return r;
}
template <typename T>
__device__ __forceinline__ void gen_store(long long at, C2<T> v) {
  if constexpr (sizeof(C2<T>) == 16) {
    float4 w;
    memcpy(&w, &v, 16);
    __stwb(reinterpret_cast<float4 *>(at), w);
  } else {
    __stwb(reinterpret_cast<C2<T> *>(at), v);
  }
}

template <typename T>
struct gen_ctx {
  const dmg_fft_pass &p;
  const gen_geom &g;
  const C2<T> *roots;
  const int2 *tin, *tout;           // offset, (position << 16) | place in the buffer
  const longlong2 *lin, *lout;      // per line (and position): address, stride in bytes; address 0 past the end
  const int2 *lx;                   // per line: twiddle y, scale exponent
  const C2<T> *twt;
  int tw_k, tw_y;
  int tid, nt;
};

template <typename T, int SIGN, int R, int CONV>
__device__ __forceinline__ void gen_run(const gen_ctx<T> &c, const gen_stage &st, bool first, bool last, const C2<T> *in,
                                        C2<T> *out) {
  const gen_geom &g = c.g;
  const dmg_fft_pass &p = c.p;
  constexpr bool DFT = std::is_same<T, df>::value;
  const bool from = first && !g.slot_in, to = last && !g.slot_out;
  const bool along_t = first ? g.load_t : last ? g.store_t : (g.s1 == 1);
  const int total = g.w * st.nb, ts = p.n / (st.lp * st.r);
  const int rstep = (first ? g.spitch_in : st.m) * g.s1;
  for (int e = c.tid; e < total; e += c.nt) {
    int l, b;
    if (along_t) {
      l = (int)gen_div((uint32_t)e, st.nb_mul, st.nb_sh);
      b = e - l * st.nb;
    } else {
      b = (int)gen_div((uint32_t)e, g.w_mul, g.w_sh);
      l = e - b * g.w;
    }
    const int j = (int)gen_div((uint32_t)b, st.m_mul, st.m_sh), k = b - j * st.m;
    C2<T> a[R];
    if (from) {
      if (g.in.ranked) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const int2 t = c.tin[b + q * st.m];
          const longlong2 s = c.lin[l * g.in.np + (int)((uint32_t)t.y >> 16)];
          a[q] = s.x ? gen_load<T>(s.x + (long long)t.x * s.y) : C2<T>{};
        }
      } else {
        const longlong2 s = c.lin[l];
        if (s.x) {
#pragma unroll
          for (int q = 0; q < R; ++q)
            a[q] = gen_load<T>(s.x + (long long)c.tin[b + q * st.m].x * (int)sizeof(C2<T>));
        } else {
#pragma unroll
          for (int q = 0; q < R; ++q) a[q] = C2<T>{};
        }
      }
    } else {
      const C2<T> *x = in + (first ? b : j * st.pin + k) * g.s1 + l * g.s2;
#pragma unroll
      for (int q = 0; q < R; ++q) a[q] = x[q * rstep];
    }
    // (double-float: the split twiddle, long code, in the stages of radix 1 only)
    if (first && (!DFT || R == 1 || CONV == 1)) {
      if (DFT && p.in_fp64) {
        const int sexp = c.lx[l].y;
#pragma unroll
        for (int q = 0; q < R; ++q) reg_convert<T>(a[q], sexp);
      }
      if ((!DFT || R == 1) && SIGN > 0 && p.twiddle == 2) {
        const int y = c.lx[l].x;
        if (y) {
#pragma unroll
          for (int q = 0; q < R; ++q) a[q] = rmul<T>(a[q], root_at<T, 1>(c.twt, (b + q * st.m) * c.tw_k + y * c.tw_y));
        }
      }
    }
    if constexpr (R > 1) {
      // (native FP64 multiplies its twiddles separately as well: inside the butterflies, in fma_node's radix-2 layers, they
      // take 72 operations instead of 84 per eight values, but the layers' doubled differences are rounded twice, and 20
      // to 1536 points came out 4 to 12 % further off than in the tiled kernel)
      auto twiddle = [&]() {
        const C2<T> *w = c.roots;
#pragma unroll
        for (int q = 1; q < R; ++q) {
          w += j * ts;
          a[q] = rmul<T>(a[q], *w);
        }
      };
      // (two paths: as one, with the products predicated, 12 and 16 points took a fifth longer)
      constexpr bool APART = std::is_same<T, double>::value && (R == 4 || R == 8);
      if (APART && st.lp == 1) {
        gdft<T, SIGN, R>(a);
      } else {
        if (APART || st.lp > 1) twiddle();
        gdft<T, SIGN, R>(a);
      }
    }
    if (last) {
      // outputs k = j + s lp (m = 1, b = j)
      if ((!DFT || R == 1) && SIGN < 0 && p.twiddle == 1) {
        const int y = c.lx[l].x;
        if (y) {
#pragma unroll
          for (int s = 0; s < R; ++s) a[s] = rmul<T>(a[s], root_at<T, -1>(c.twt, (b + s * st.lp) * c.tw_k + y * c.tw_y));
        }
      }
      if (DFT && (R == 1 || CONV == 2) && p.out_fp64) {
        const int sexp = c.lx[l].y;
#pragma unroll
        for (int s = 0; s < R; ++s) reg_unconvert<T>(a[s], sexp);
      }
      if (to) {
        if (g.out.ranked) {
#pragma unroll
          for (int s = 0; s < R; ++s) {
            const int2 t = c.tout[b + s * st.lp];
            const longlong2 d = c.lout[l * g.out.np + (int)((uint32_t)t.y >> 16)];
            if (d.x) gen_store<T>(d.x + (long long)t.x * d.y, a[s]);
          }
        } else {
          const longlong2 d = c.lout[l];
          if (d.x) {
#pragma unroll
            for (int s = 0; s < R; ++s)
              gen_store<T>(d.x + (long long)c.tout[b + s * st.lp].x * (int)sizeof(C2<T>), a[s]);
          }
        }
      } else {
        C2<T> *y = out + b * g.s1 + l * g.s2;
#pragma unroll
        for (int s = 0; s < R; ++s) y[s * g.spitch_out * g.s1] = a[s];
      }
    } else {
      C2<T> *y = out + (j * st.pout + k) * g.s1 + l * g.s2;
      const int ws = st.lp * st.pout * g.s1;
#pragma unroll
      for (int s = 0; s < R; ++s) y[s * ws] = a[s];
    }
  }
}

// A prime radix without a butterfly: direct DFTs from one buffer to the other, an output per thread (with a thread per
// butterfly, a block's few lines of a long prime left most lanes idle: 512 lines of 1009 points, native FP64, 1430 ms
// and 651 in the tiled kernel).
template <typename T, int SIGN>
__device__ __noinline__ void gen_prime(const gen_ctx<T> &c, const gen_stage &st, const C2<T> *in, C2<T> *out) {
  const gen_geom &g = c.g;
  const int n = c.p.n, r = st.r, ts = n / (st.lp * r), nr = n / r;
  const int per = g.w * st.nb;  // butterflies
  // (the input twiddle and the DFT's root are one root of n: a product a value, half of what two take; 1331 points,
  // 2048 lines, native FP64: 1717 us with two products, 1506 in the tiled kernel, 1020 so)
  for (int e = c.tid; e < per * r; e += c.nt) {
    const int s = e / per, i = e - s * per;
    const int l = (int)gen_div((uint32_t)i, st.nb_mul, st.nb_sh), b = i - l * st.nb;
    if (c.lin[l * g.in.np].x == 0) continue;  // past the last line
    const int j = (int)gen_div((uint32_t)b, st.m_mul, st.m_sh), k = b - j * st.m;
    const C2<T> *x = in + (j * st.pin + k) * g.s1 + l * g.s2;
    C2<T> acc = x[0];
    const int step = j * ts + s * nr;  // (each below n, step q = j q ts + q s n / r)
    int ro = 0;
    for (int q = 1; q < r; ++q) {
      ro += step;
      if (ro >= n) ro -= n;
      acc = add<T>(acc, rmul<T>(x[q * st.m * g.s1], c.roots[ro]));
    }
    out[(j * st.pout + k) * g.s1 + l * g.s2 + s * st.lp * st.pout * g.s1] = acc;
  }
}

// addresses of a side's lines of a tile: per line, and position of a ranked side
template <typename T>
__device__ __forceinline__ void gen_lines(const gen_side &s, const dmg_fft_layout &L, const dmg_fft_pass &p, int pos,
                                          const int *x, uint64_t base, longlong2 *to) {
  constexpr int ES = (int)sizeof(C2<T>);
  if (!s.ranked) {
    *to = make_longlong2((long long)(base + (uint64_t)line_address(L, p.ndim, x) * ES), ES);
    return;
  }
  const int d0 = p.kdim[0];
  int32_t R = s.rstep * pos;
#pragma unroll
  for (int d = 0; d < DMG_FFT_MAXDIM; ++d)
    if (d < p.ndim && d != d0) R += __ldg(L.rk[d] + x[d]);
  int64_t a = L.base + (int64_t)R * L.pitch;
#pragma unroll
  for (int d = 0; d < DMG_FFT_MAXDIM; ++d)
    if (d < p.ndim && d != d0) a += __ldg(L.tab[d] + x[d]) * __ldg(L.rstride + (size_t)d * L.nranks + R);
  *to = make_longlong2((long long)(base + (uint64_t)a * ES), (long long)__ldg(L.rstride + (size_t)d0 * L.nranks + R) * ES);
}

// The pass as block `bid` of `nblk` persistent blocks.
template <typename T, int SIGN, int CONV>
__device__ __forceinline__ void gen_body(const dmg_fft_pass &p, const dmg_fft_batch &bt, const line_axes &lines,
                                         const gen_geom &g, int64_t bid, int64_t nblk) {
  extern __shared__ __align__(16) unsigned char sm[];
  const int tid = threadIdx.x, nt = blockDim.x, n = p.n;
  C2<T> *const bufA = reinterpret_cast<C2<T> *>(sm), *const bufB = reinterpret_cast<C2<T> *>(sm + g.off_b);
  C2<T> *roots = reinterpret_cast<C2<T> *>(sm + g.off_roots);
  int2 *tin = reinterpret_cast<int2 *>(sm + g.off_tin), *tout = reinterpret_cast<int2 *>(sm + g.off_tout);
  longlong2 *lin = reinterpret_cast<longlong2 *>(sm + g.off_lin), *lout = reinterpret_cast<longlong2 *>(sm + g.off_lout);
  int2 *lx = reinterpret_cast<int2 *>(sm + g.off_lx);
  for (int i = tid; i < n; i += nt) roots[i] = root_at<T, SIGN>(reinterpret_cast<const C2<T> *>(p.roots), i);
  {
    const int d0 = p.kdim[0], m0 = p.kisz[0] ? p.A[d0] : 1;
    for (int s = tid; s < n; s += nt) {
      const int k = (p.perm_in || p.perm_out) ? s / p.perm_a + p.perm_b * (s % p.perm_a) : s;
      auto entry = [&](const dmg_fft_layout &L, const gen_side &sd, int place) {
        const int64_t v = __ldg(L.tab[d0] + (int64_t)s * m0);
        const int pos = sd.ranked ? __ldg(L.rk[d0] + s) / max(sd.rstep, 1) : 0;
        return make_int2((int32_t)(sd.ranked ? v : v - __ldg(L.tab[d0])), (int)(((uint32_t)pos << 16) | (uint32_t)place));
      };
      const int pi = (k / g.srow_in) * g.spitch_in + k % g.srow_in, po = (k / g.srow_out) * g.spitch_out + k % g.srow_out;
      tin[g.slot_in ? s : p.perm_in ? k : s] = entry(p.in, g.in, pi);
      tout[g.slot_out ? s : p.perm_out ? k : s] = entry(p.out, g.out, po);
    }
  }
  const int td = p.t >> 1;
  const bool kmaj = !g.store_t && p.kdim[1] == td && !p.kisz[1];
  const gen_ctx<T> c{p, g, roots, tin, tout, lin, lout, lx,
                     reinterpret_cast<const C2<T> *>(kmaj ? p.twk[td] : p.twy[td]), kmaj ? p.A[td] : 1, kmaj ? 1 : n, tid, nt};
  constexpr bool DFT = std::is_same<T, df>::value;
  const int64_t ntiles = ((int64_t)lines.total + g.w - 1) / g.w;
  for (int64_t tile = bid; tile < ntiles; tile += nblk) {
    __syncthreads();  // the previous tile's line table has been read (and the tables above are complete)
    const int npi = g.in.np, npo = g.out.np;
    for (int i = tid; i < g.w * (npi + npo); i += nt) {
      const bool o = i >= g.w * npi;
      const int ii = o ? i - g.w * npi : i, np = o ? npo : npi;
      const int l = ii / np, pos = ii - l * np;
      const int64_t line = tile * g.w + l;
      longlong2 v = make_longlong2(0, 0);
      if (!o && pos == 0) lx[l] = make_int2(0, 0);
      if (line < (int64_t)lines.total) {
        int x[DMG_FFT_MAXDIM], y;
        const uint32_t job = line_place(lines, (uint32_t)line, x, y);
        if (o) gen_lines<T>(g.out, p.out, p, pos, x, (uint64_t)bt.dst[job], &v);
        else gen_lines<T>(g.in, p.in, p, pos, x, (uint64_t)bt.src[job], &v);
        if (!o && pos == 0)
          lx[l] = make_int2(y, DFT && (p.in_fp64 || p.out_fp64) ? __ldg(bt.scale_exp[job]) - 1022 : 0);
      }
      (o ? lout : lin)[ii] = v;
    }
    __syncthreads();
    if (g.slot_in) {
      // slot order: lanes run along the slots of a line; 8 loads in flight per thread
      for (int e0 = tid; e0 < g.w * n; e0 += 8 * nt) {
        C2<T> v[8];
        int at[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int e = e0 + u * nt;
          at[u] = -1;
          if (e < g.w * n) {
            const int l = (int)gen_div((uint32_t)e, g.n_mul, g.n_sh), s = e - l * n;
            const int2 t = tin[s];
            const longlong2 b = lin[g.in.ranked ? l * npi + (int)((uint32_t)t.y >> 16) : l];
            if (b.x) {
              v[u] = gen_load<T>(b.x + (long long)t.x * b.y);
              at[u] = (t.y & 0xFFFF) * g.s1 + l * g.s2;
            }
          }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (at[u] >= 0) bufB[at[u]] = v[u];
      }
      __syncthreads();
    }
    const C2<T> *in = bufB;
    C2<T> *out = bufA;
    for (int f = 0; f < g.nst; ++f) {
      const gen_stage &st = g.st[f];
      const bool first = f == 0, last = f == g.nst - 1;
      switch (st.r) {
        case 1: gen_run<T, SIGN, 1, CONV>(c, st, first, last, in, out); break;
        case 2: gen_run<T, SIGN, 2, CONV>(c, st, first, last, in, out); break;
        case 3: gen_run<T, SIGN, 3, CONV>(c, st, first, last, in, out); break;
        case 4: gen_run<T, SIGN, 4, CONV>(c, st, first, last, in, out); break;
        case 5: gen_run<T, SIGN, 5, CONV>(c, st, first, last, in, out); break;
        case 6: gen_run<T, SIGN, 6, CONV>(c, st, first, last, in, out); break;
        case 7: gen_run<T, SIGN, 7, CONV>(c, st, first, last, in, out); break;
        case 8: gen_run<T, SIGN, 8, CONV>(c, st, first, last, in, out); break;
        case 9: gen_run<T, SIGN, 9, CONV>(c, st, first, last, in, out); break;
        case 10: gen_run<T, SIGN, 10, CONV>(c, st, first, last, in, out); break;
        default:
          if constexpr (std::is_same<T, float>::value) {
            if (st.r == 12) {
              gen_run<T, SIGN, 12, CONV>(c, st, first, last, in, out);
              break;
            } else if (st.r == 14) {
              gen_run<T, SIGN, 14, CONV>(c, st, first, last, in, out);
              break;
            } else if (st.r == 15) {
              gen_run<T, SIGN, 15, CONV>(c, st, first, last, in, out);
              break;
            } else if (st.r == 16) {
              gen_run<T, SIGN, 16, CONV>(c, st, first, last, in, out);
              break;
            }
          }
          gen_prime<T, SIGN>(c, st, in, out);
      }
      if (!last || g.slot_out) __syncthreads();
      const C2<T> *t = in;
      in = out;
      out = const_cast<C2<T> *>(t);
    }
    if (g.slot_out) {
      // (in: what the last stage wrote)
      for (int e0 = tid; e0 < g.w * n; e0 += 4 * nt) {
        C2<T> v[4];
        long long at[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int e = e0 + u * nt;
          at[u] = 0;
          if (e < g.w * n) {
            const int l = (int)gen_div((uint32_t)e, g.n_mul, g.n_sh), s = e - l * n;
            const int2 t = tout[s];
            const longlong2 d = lout[g.out.ranked ? l * npo + (int)((uint32_t)t.y >> 16) : l];
            v[u] = in[(t.y & 0xFFFF) * g.s1 + l * g.s2];
            if (d.x) at[u] = d.x + (long long)t.x * d.y;
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (at[u]) gen_store<T>(at[u], v[u]);
      }
    }
  }
}

template <typename T, int SIGN, int CONV>
__global__ void __launch_bounds__(GEN_MAXNT, 1)
    fft_gen_kernel(const __grid_constant__ dmg_fft_pass p, const __grid_constant__ dmg_fft_batch bt,
                   const __grid_constant__ line_axes lines, const __grid_constant__ gen_geom g) {
  gen_body<T, SIGN, CONV>(p, bt, lines, g, blockIdx.x, gridDim.x);
}

// Several passes in one launch: pass j owns blocks first_block ... first_block + nblocks - 1.
struct gen_job {
  dmg_fft_pass p;
  dmg_fft_batch bt;
  line_axes lines;
  gen_geom g;
  int64_t first_block, nblocks;
};
// (the jobs lie in device-visible constant parameters; a launch takes as many as fit in 32 KB)
constexpr int GEN_MAXJOBS = (int)((32764 - 16) / sizeof(gen_job));
struct gen_group {
  int32_t count;
  gen_job job[GEN_MAXJOBS];
};
template <typename T, int SIGN>
__global__ void __launch_bounds__(GEN_MAXNT, 1) fft_gen_group_kernel(const __grid_constant__ gen_group G) {
  int j = 0;
  while (j + 1 < G.count && (int64_t)blockIdx.x >= G.job[j + 1].first_block) ++j;
  const gen_job &job = G.job[j];
  gen_body<T, SIGN, 0>(job.p, job.bt, job.lines, job.g, (int64_t)blockIdx.x - job.first_block, job.nblocks);
}


// ---------------------------------------------------------------- launch

inline int64_t gen_lines_of(const dmg_fft_pass &p, const dmg_fft_batch &bt) {
  int64_t n = (int64_t)bt.count * p.nv1 * p.nv2;
  for (int b = 0; b < p.nbatch; ++b) n *= p.blen[b];
  return n;
}

template <typename K>
int gen_blocks(K k, int nt, size_t smem, int64_t *blocks) {
  int dev = 0, nsm = 0, per_sm = 0;
  cudaError_t e = allow_smem(k, smem);
  if (e == cudaSuccess) e = resident_blocks(k, nt, smem, &per_sm);
  if (e != cudaSuccess) return dmg_error(DMG_ERR_CUDA, "fft pass smem %zu: %s", smem, cudaGetErrorString(e));
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (per_sm < 1) return dmg_error(DMG_ERR_UNSUPPORTED, "fft pass does not fit on an SM (smem %zu)", smem);
  *blocks = (int64_t)nsm * per_sm;
  return DMG_OK;
}

// One pass; *taken says whether this kernel takes it.
template <typename T, int SIGN, int CONV = 0>
int launch_gen(const dmg_fft_pass &p, const dmg_fft_batch &bt, cudaStream_t s, int *taken) {
  gen_geom g;
  const int64_t n = gen_lines_of(p, bt);
  *taken = n < ((int64_t)1 << 31) && gen_make<T>(p, n, 0, &g, CONV);
  if (!*taken) return DMG_OK;
  auto k = fft_gen_kernel<T, SIGN, CONV>;
  int64_t grid = 0;
  const int st = gen_blocks(k, g.nt, g.smem, &grid);
  if (st != DMG_OK) return st;
  const int64_t ntiles = (n + g.w - 1) / g.w;
  if (grid > ntiles) grid = ntiles;
  if (grid < 1) return DMG_OK;
  k<<<(unsigned)grid, g.nt, g.smem, s>>>(p, bt, line_axes_of(p, bt), g);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return dmg_error(DMG_ERR_CUDA, "fft pass launch: %s", cudaGetErrorString(e));
  return DMG_OK;
}

// The passes of a group that this kernel takes (taken[j] set), in one launch:
// each gets blocks in proportion to its tiles (at least one, at most its tile
// count) out of those that fill the SMs at the largest job's shared memory.
template <typename T, int SIGN>
int launch_gen_group(const dmg_fft_group &in, cudaStream_t s, int *taken) {
  static_assert(GEN_MAXJOBS >= DMG_FFT_MAXGROUP, "a group is one launch");
  gen_group *G = static_cast<gen_group *>(malloc(sizeof(gen_group)));
  if (!G) return dmg_error(DMG_ERR_NOMEM, "grouped fft pass: out of memory");
  G->count = 0;
  size_t smem = 0;
  double work = 0;
  // one block size for all: the largest any of them asks for
  int nt = 0;
  double values = 0;
  for (int j = 0; j < in.count; ++j) {
    gen_geom g;
    values += (double)gen_lines_of(in.job[j].p, in.job[j].bt) * in.job[j].p.n;
    if (in.job[j].p.gen && gen_make<T>(in.job[j].p, (int64_t)1 << 30, 0, &g) && g.nt > nt) nt = g.nt;
  }
  const bool full = values >= 2.0 * GEN_SMS * nt * gen_per_thread<T>();  // (full tiles of all jobs fill the SMs)
  for (int j = 0; j < in.count; ++j) {
    const dmg_fft_pass &p = in.job[j].p;
    const int64_t n = gen_lines_of(p, in.job[j].bt);
    gen_job &job = G->job[G->count];
    taken[j] = p.gen && n < ((int64_t)1 << 31) && gen_make<T>(p, full ? (int64_t)1 << 30 : n, nt, &job.g);
    if (!taken[j]) continue;
    job.p = p;
    job.bt = in.job[j].bt;
    job.lines = line_axes_of(p, job.bt);
    smem = job.g.smem > smem ? job.g.smem : smem;
    work += (double)n * p.n;
    ++G->count;
  }
  int st = DMG_OK;
  if (G->count > 0) {
    auto k = fft_gen_group_kernel<T, SIGN>;
    int64_t budget = 0, first = 0;
    st = gen_blocks(k, nt, smem, &budget);
    for (int j = 0; j < G->count && st == DMG_OK; ++j) {
      gen_job &job = G->job[j];
      const int64_t tiles = ((int64_t)job.lines.total + job.g.w - 1) / job.g.w;
      int64_t nb = (int64_t)((double)budget * ((double)job.lines.total * job.p.n) / (work > 0 ? work : 1) + 0.999);
      if (nb > tiles) nb = tiles;
      if (nb < 1) nb = 1;
      job.first_block = first;
      job.nblocks = nb;
      first += nb;
    }
    if (st == DMG_OK) {
      k<<<(unsigned)first, nt, smem, s>>>(*G);
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) st = dmg_error(DMG_ERR_CUDA, "grouped fft pass launch: %s", cudaGetErrorString(e));
    }
  }
  free(G);
  return st;
}

}  // namespace
