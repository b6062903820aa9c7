// FFT passes whose lines live in registers: the kernel of every pass whose
// length has a schedule here, whose sides are separable and whose sides run
// along the same fastest tile axis (fft_gen.cuh serves other lengths, ranked
// sides and different fastest axes, fft_pass.cuh what is left).
//
// A block transforms W whole lines at a time with TL threads per line.  A
// thread loads the R values of its first butterfly straight from the input
// layout into registers, transforms them, and exchanges them with the line's
// other threads through shared memory once per further stage (n = R1 R2: one
// exchange, R1 R2 R3: two); the last stage's results go from registers to the
// output layout.  What bounds the kernels of fft_pass.cuh is not HBM but
// their instruction count (FP32 100 instructions per value, half of them
// index arithmetic; double-float 296; native FP64 219) at 16 warps per SM.
// Here a value costs one table read, one 64-bit address addition and one
// access per side; every shared-memory position is a thread's base plus a
// compile-time constant, and a line's values cross shared memory once or
// twice instead of four times.
//
// Lines.  A pass's lines (all tile and batch axes and the jobs of a batch)
// are numbered along v1, then v2, then the batch axes, then the jobs, and a
// block takes W consecutive ones, so that extents that do not divide by a
// tile leave no lanes idle except in the last tile.  A line's address on a
// side is the sum of its dimensions' table entries; the transform axis adds
// an offset that is the same for every line (the host checks this), kept in
// shared memory as int32 with the slot order of line passes folded in.
//
// Two forms: "along v1" (v1 is the fastest axis on both sides: neighbouring
// lanes hold neighbouring lines, shared memory is [position][line]) and
// "along t" (the transform axis is: neighbouring lanes hold neighbouring
// values of a line, shared memory is [line][position]).  Along t, a side in
// slot order is read or written in that order through one more exchange, so
// that its accesses stay contiguous.
//
// Measured on one GB300 against the tiled kernel (forward transforms, lines
// schedule): 1024^3 complex64 FP32 26.1 -> 9.9 ms (7.6 ms at the copy rate);
// 8 cubes of 240^3 complex64, moved, forward and back, 6.42 -> 2.16 ms;
// 512^3 complex128 double-float 7.95 -> 5.39 ms, native FP64 step (forward,
// inverse and two reshapes) 38.6 -> 34.2 ms, where the FP64 pipe binds.
#pragma once
#include <cmath>
#include <cstdlib>
#include <cstring>
#include "fft_pass.cuh"

namespace {

// ---------------------------------------------------------------- schedules

// Radices, threads per line, lines per block, resident blocks per SM the
// register budget allows, and how a block prepares its next tile (AHEAD_*).
// kind: 0 native FP64, 1 FP32, 2 double-float; t: the form along t.
struct RegSched {
  int ns;
  int r[3];
  int tl, w, minb;
  int ahead;
};
// The next tile of a block: loaded when its turn comes; its values asked
// into L2 behind this tile's first stage; or copied behind this tile's later
// stages into shared memory (each thread its own values, asynchronously).
enum { AHEAD_NONE = 0, AHEAD_L2 = 1, AHEAD_COPY = 2 };

// Each row is the fastest of the shapes timed for its length over 2^27 (FP32)
// or 2^26 values, in both forms (GB/s of a pass's bytes, read and written
// once; a plain copy runs at 6800):
// * FP32 is near HBM: two stages (radices up to 32) beat three throughout
//   (512 points along v1: 6290 against 4970); along v1 the rows of W lines
//   are 128 bytes where a block's registers hold the tile (512 points: 4750
//   with 64-byte rows); 1024 points take them in one 512-thread block that
//   asks L2 for its next tile (5100; 4610 in two blocks of 64-byte rows).
//   Along t small blocks, many per SM, are better (512: 6290 with 8 lines,
//   5580 with 16).
// * Double-float is bound by its FP32 operations (125 paired ones a value at
//   512 points) and by the phases in which a block has none to issue: radix 8
//   where a thread then needs no spills, 16 up to 256 points along v1 (256:
//   3260 against 2890 with three stages), copies ahead where two blocks still
//   fit (512 along v1: 2740; 2615 without).  The passes along t convert
//   complex128 on one side and take smaller radices and blocks (96: 2663
//   against 1328 with radices 12 and 8).
// * Native FP64 is bound by its pipe (86 % busy at 512 points): the odd
//   radices go first, where they need no twiddles, and the twiddled ones are
//   8 and 4, in their form with the fewest operations (240: 785 against 645
//   with radices 16 and 15; 256: 880 against 815 with 16 and 16).
__host__ __device__ constexpr RegSched reg_table(int kind, int n, bool t, bool inv) {
  if (kind == 1) {
    switch (n) {
      case 32: return t ? RegSched{2, {8, 4, 1}, 4, 32, 8, AHEAD_NONE} : RegSched{2, {8, 4, 1}, 4, 64, 3, AHEAD_L2};
      case 48: return t ? RegSched{2, {8, 6, 1}, 8, 16, 6, AHEAD_NONE} : RegSched{2, {8, 6, 1}, 8, 32, 4, AHEAD_L2};
      case 64: return t ? RegSched{2, {8, 8, 1}, 8, 16, 8, AHEAD_NONE} : RegSched{2, {8, 8, 1}, 8, 32, 3, AHEAD_L2};
      case 96: return t ? RegSched{2, {12, 8, 1}, 12, 8, 8, AHEAD_NONE} : RegSched{2, {12, 8, 1}, 12, 16, 4, AHEAD_L2};
      case 120: return t ? RegSched{2, {12, 10, 1}, 12, 8, 6, AHEAD_L2} : RegSched{2, {12, 10, 1}, 12, 16, 4, AHEAD_L2};
      case 128: return t ? RegSched{2, {16, 8, 1}, 8, 8, 12, AHEAD_NONE} : RegSched{2, {16, 8, 1}, 8, 32, 3, AHEAD_NONE};
      case 160: return t ? RegSched{2, {16, 10, 1}, 16, 4, 10, AHEAD_L2} : RegSched{2, {16, 10, 1}, 16, 16, 3, AHEAD_L2};
      case 192: return t ? RegSched{2, {16, 12, 1}, 16, 4, 10, AHEAD_L2} : RegSched{2, {16, 12, 1}, 16, 16, 3, AHEAD_L2};
      case 240: return t ? RegSched{2, {16, 15, 1}, 16, 4, 12, AHEAD_L2} : RegSched{2, {16, 15, 1}, 16, 16, 3, AHEAD_NONE};
      case 256: return t ? RegSched{2, {16, 16, 1}, 16, 8, 6, AHEAD_NONE} : RegSched{2, {16, 16, 1}, 16, 16, 3, AHEAD_NONE};
      case 320: return t ? RegSched{2, {20, 16, 1}, 20, 8, 4, AHEAD_L2} : RegSched{2, {20, 16, 1}, 20, 16, 2, AHEAD_L2};
      case 384: return t ? RegSched{2, {24, 16, 1}, 24, 8, 3, AHEAD_NONE} : RegSched{2, {24, 16, 1}, 24, 16, 1, AHEAD_L2};
      case 480: return t ? RegSched{2, {24, 20, 1}, 24, 4, 5, AHEAD_NONE} : RegSched{2, {24, 20, 1}, 24, 16, 1, AHEAD_L2};
      case 512: return t ? RegSched{2, {32, 16, 1}, 16, 8, 4, AHEAD_L2} : RegSched{2, {32, 16, 1}, 16, 16, 2, AHEAD_NONE};
      case 1024: return t ? (inv ? RegSched{2, {32, 32, 1}, 32, 4, 4, AHEAD_L2} : RegSched{2, {32, 32, 1}, 32, 8, 2, AHEAD_L2}) : RegSched{2, {32, 32, 1}, 32, 16, 1, AHEAD_L2};
      case 2048: return t ? RegSched{3, {16, 8, 16}, 128, 4, 2, AHEAD_L2} : RegSched{3, {16, 16, 8}, 128, 8, 1, AHEAD_L2};
      default: return {0, {1, 1, 1}, 1, 1, 1, AHEAD_NONE};
    }
  }
  if (kind == 0) {
    switch (n) {
      case 32: return {2, {8, 4, 1}, 4, 32, 3, AHEAD_NONE};
      case 48: return {2, {6, 8, 1}, 8, 16, 4, AHEAD_NONE};
      case 64: return {2, {8, 8, 1}, 8, 16, 4, AHEAD_NONE};
      case 96: return {2, {12, 8, 1}, 12, 8, 4, AHEAD_NONE};
      case 120: return t ? RegSched{2, {15, 8, 1}, 8, 8, 4, AHEAD_NONE} : RegSched{2, {15, 8, 1}, 15, 8, 4, AHEAD_NONE};
      case 128: return {3, {8, 4, 4}, 16, 8, 4, AHEAD_NONE};
      case 160: return {3, {5, 8, 4}, 20, 8, 3, AHEAD_NONE};
      case 192: return {3, {3, 8, 8}, 24, 8, 3, AHEAD_NONE};
      case 240: return {3, {15, 4, 4}, 16, 8, 3, AHEAD_NONE};
      case 256: return {3, {8, 8, 4}, 32, 4, 4, AHEAD_NONE};
      case 320: return {3, {20, 4, 4}, 16, 8, 2, AHEAD_NONE};
      case 384: return {3, {6, 8, 8}, 48, 4, 2, AHEAD_NONE};
      case 480: return {3, {15, 8, 4}, 32, 4, 3, AHEAD_NONE};
      case 512: return {3, {8, 8, 8}, 64, 2, 5, AHEAD_NONE};
      case 1024: return {3, {16, 8, 8}, 64, 4, 2, AHEAD_NONE};
      default: return {0, {1, 1, 1}, 1, 1, 1, AHEAD_NONE};
    }
  }
  switch (n) {
    case 32: return t ? RegSched{2, {8, 4, 1}, 4, 8, 16, AHEAD_NONE} : RegSched{2, {8, 4, 1}, 4, 32, 3, AHEAD_NONE};
    case 48: return t ? RegSched{3, {4, 4, 3}, 12, 8, 6, AHEAD_NONE} : RegSched{2, {8, 6, 1}, 8, 16, 5, AHEAD_COPY};
    case 64: return t ? RegSched{2, {8, 8, 1}, 8, 8, 10, AHEAD_NONE} : RegSched{2, {8, 8, 1}, 8, 16, 6, AHEAD_NONE};
    case 96: return t ? RegSched{3, {8, 4, 3}, 12, 8, 8, AHEAD_NONE} : RegSched{2, {12, 8, 1}, 12, 8, 5, AHEAD_COPY};
    case 120: return t ? RegSched{3, {8, 5, 3}, 15, 8, 5, AHEAD_NONE} : RegSched{2, {12, 10, 1}, 12, 16, 2, AHEAD_NONE};
    case 128: return t ? RegSched{3, {8, 4, 4}, 16, 4, 12, AHEAD_NONE} : RegSched{2, {16, 8, 1}, 8, 8, 6, AHEAD_COPY};
    case 160: return t ? RegSched{3, {8, 5, 4}, 20, 8, 3, AHEAD_NONE} : RegSched{3, {8, 5, 4}, 20, 8, 4, AHEAD_NONE};
    case 192: return t ? RegSched{3, {8, 6, 4}, 24, 4, 5, AHEAD_NONE} : RegSched{3, {8, 6, 4}, 24, 8, 2, AHEAD_COPY};
    case 240: return t ? RegSched{3, {8, 6, 5}, 30, 2, 8, AHEAD_NONE} : RegSched{2, {16, 15, 1}, 16, 8, 3, AHEAD_COPY};
    case 256: return t ? RegSched{3, {8, 8, 4}, 32, 4, 5, AHEAD_NONE} : RegSched{2, {16, 16, 1}, 16, 8, 4, AHEAD_NONE};
    case 320: return t ? RegSched{3, {8, 8, 5}, 40, 4, 3, AHEAD_NONE} : RegSched{3, {8, 10, 4}, 40, 4, 3, AHEAD_NONE};
    case 384: return t ? RegSched{3, {8, 8, 6}, 48, 2, 5, AHEAD_NONE} : RegSched{3, {8, 8, 6}, 48, 4, 2, AHEAD_COPY};
    case 480: return t ? RegSched{3, {8, 10, 6}, 60, 2, 4, AHEAD_NONE} : RegSched{3, {8, 6, 10}, 60, 4, 2, AHEAD_NONE};
    case 512: return t ? RegSched{3, {8, 8, 8}, 64, 2, 5, AHEAD_NONE} : RegSched{3, {8, 8, 8}, 64, 4, 2, AHEAD_COPY};
    case 1024: return {3, {8, 16, 8}, 64, 4, 2, AHEAD_NONE};
    default: return {0, {1, 1, 1}, 1, 1, 1, AHEAD_NONE};
  }
}
// The schedule of a pass.  Along t, inverse: the radices in reverse, so that
// the rows of the slot-order exchange (n / R1 values before the first stage,
// forward n / RL after the last) are as long as the distance of the values
// that neighbouring slots hold (the plans' larger factor B of n), whose odd
// pitch then spreads them over the banks.
// lines: the lines per block where not the table's (the results' bits do not depend on them).
__host__ __device__ constexpr RegSched reg_sched(int kind, int n, bool t, bool inv, int lines = 0) {
  RegSched s = reg_table(kind, n, t, inv);
  if (lines > 0) s.w = lines;
  // (native FP64 is bound by its pipe: there the odd radix comes first, where it needs no input twiddles)
  if (t && inv && s.ns > 1 && kind != 0) {
    const int first = s.r[0];
    s.r[0] = s.r[s.ns - 1];
    s.r[s.ns - 1] = first;
  }
  return s;
}
template <typename T>
__host__ __device__ constexpr int reg_kind() {
  return std::is_same<T, float>::value ? 1 : std::is_same<T, df>::value ? 2 : 0;
}
__host__ __device__ constexpr bool is_pow2(int n) { return n > 0 && (n & (n - 1)) == 0; }

// ---------------------------------------------------------------- butterflies in registers

// a * b with scalar FMAs in FP32 (the paired form has to build pairs of equal values first)
template <typename T>
__device__ __forceinline__ C2<T> rmul(C2<T> a, C2<T> b) {
  if constexpr (std::is_same<T, float>::value) {
    return make_float2(fmaf(a.x, b.x, -(a.y * b.y)), fmaf(a.x, b.y, a.y * b.x));
  } else {
    return mul<T>(a, b);
  }
}
// a + sign i b and a - sign i b
template <typename T, int SIGN, bool LAZY = false>
__device__ __forceinline__ C2<T> add_rot(C2<T> a, C2<T> b) {
  if constexpr (std::is_same<T, df>::value) {
    return LAZY ? addl<T>(a, rot90<T, SIGN>(b)) : add<T>(a, rot90<T, SIGN>(b));
  } else {
    C2<T> r;
    r.x = SIGN < 0 ? a.x + b.y : a.x - b.y;
    r.y = SIGN < 0 ? a.y - b.x : a.y + b.x;
    return r;
  }
}
template <typename T, int SIGN, bool LAZY = false>
__device__ __forceinline__ C2<T> sub_rot(C2<T> a, C2<T> b) {
  return add_rot<T, -SIGN, LAZY>(a, b);
}

// cos(pi k / 16), k = 0 ... 8, as a double and as two floats
template <typename T, int K>
__device__ __forceinline__ T cos16() {
  static_assert(K >= 0 && K <= 8, "first quadrant");
  if constexpr (K == 0) return cst<T>(1.0, 1.0f, 0.0f);
  else if constexpr (K == 1) return cst<T>(0.980785280403230449126182236134239036, 0.9807852506637573f, 2.9739473106360492e-08f);
  else if constexpr (K == 2) return cst<T>(0.923879532511286756128183189396788286, 0.9238795042037964f, 2.830748968563057e-08f);
  else if constexpr (K == 3) return cst<T>(0.831469612302545237078788377617905756, 0.8314695954322815f, 1.687026340846387e-08f);
  else if constexpr (K == 4) return cst<T>(K_SQRT1_2);
  else if constexpr (K == 5) return cst<T>(0.555570233019602224742830813948532874, 0.5555702447891235f, -1.1769521357507529e-08f);
  else if constexpr (K == 6) return cst<T>(0.382683432365089771728459984030398866, 0.3826834261417389f, 6.2233507236442165e-09f);
  else if constexpr (K == 7) return cst<T>(0.195090322016128267848284868477022240, 0.19509032368659973f, -1.670471427850373e-09f);
  else return cst<T>(0.0, 0.0f, 0.0f);
}
template <typename T>
__device__ __forceinline__ T rneg(T a) { return -a; }
// exp(sign i pi K / 16) as (re, im), any K
template <typename T, int SIGN, int K>
__device__ __forceinline__ void unit16(T &re, T &im) {
  constexpr int k = ((K % 32) + 32) % 32;
  constexpr int q = k / 8, r = k % 8;  // quadrant, angle within it
  const T c = cos16<T, r>(), s = cos16<T, 8 - r>();
  // e^{i (q pi/2 + a)} = i^q (c + i s)
  T x = q == 0 ? c : q == 1 ? rneg(s) : q == 2 ? rneg(c) : s;
  T y = q == 0 ? s : q == 1 ? c : q == 2 ? rneg(s) : rneg(c);
  re = x;
  im = SIGN < 0 ? rneg(y) : y;
}
__device__ __forceinline__ float2 pack_c(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ double2 pack_c(double x, double y) { return make_double2(x, y); }
__device__ __forceinline__ dfc pack_c(df x, df y) { return dfc{make_float2(x.h, y.h), make_float2(x.l, y.l)}; }
// v * exp(sign 2 pi i E / R), R a power of two up to 32
template <typename T, int SIGN, int R, int E>
__device__ __forceinline__ C2<T> mul_unit(C2<T> v) {
  constexpr int K = (E * (32 / R)) % 32;
  if constexpr (K == 0) {
    return v;
  } else if constexpr (K == 8) {
    return rot90<T, SIGN>(v);
  } else if constexpr (K % 8 == 4) {
    // (+-1 +- i) / sqrt 2: a sum with the rotated value, scaled
    const T c = cst<T>(K_SQRT1_2);
    if constexpr (K == 4) return scl<T>(add_rot<T, SIGN, true>(v, v), c);
    else return scl<T>(subl<T>(rot90<T, SIGN>(v), v), c);  // K == 12
  } else if constexpr (std::is_same<T, float>::value) {
    // The FP32 roundings of these few constants all make the factor shorter (by up to 2.9e-8): the trailing
    // part of the longer component goes in too, which keeps the bias from adding up over stages and passes
    // (1024-point round trip 2.39e-7 without it, 2.18e-7 in the tiled kernel's radix-8 and -4 stages).
    df re, im;
    unit16<df, SIGN, K>(re, im);
    constexpr int k = K % 16;
    if constexpr (k < 4 || k > 12) {
      return make_float2(fmaf(v.x, re.h, fmaf(v.x, re.l, -(v.y * im.h))), fmaf(v.y, re.h, fmaf(v.y, re.l, v.x * im.h)));
    } else {
      return make_float2(fmaf(-v.y, im.h, fmaf(-v.y, im.l, v.x * re.h)), fmaf(v.x, im.h, fmaf(v.x, im.l, v.y * re.h)));
    }
  } else {
    T re, im;
    unit16<T, SIGN, K>(re, im);
    return rmul<T>(v, pack_c(re, im));
  }
}

template <typename T, int SIGN, bool LAZY = false>
__device__ __forceinline__ void rdft4(C2<T> &a0, C2<T> &a1, C2<T> &a2, C2<T> &a3) {
  const C2<T> t0 = addl<T>(a0, a2), t1 = subl<T>(a0, a2), t2 = addl<T>(a1, a3), t3 = subl<T>(a1, a3);
  if constexpr (LAZY) {
    a0 = addl<T>(t0, t2);
    a2 = subl<T>(t0, t2);
  } else {
    a0 = add<T>(t0, t2);
    a2 = sub<T>(t0, t2);
  }
  a1 = add_rot<T, SIGN, LAZY>(t1, t3);
  a3 = sub_rot<T, SIGN, LAZY>(t1, t3);
}
template <typename T, int SIGN>
__device__ __forceinline__ void rdft8(C2<T> *a) {
  if constexpr (std::is_same<T, float>::value) {
    C2<T> e0 = a[0], e1 = a[2], e2 = a[4], e3 = a[6];
    C2<T> o0 = a[1], o1 = a[3], o2 = a[5], o3 = a[7];
    rdft4<T, SIGN>(e0, e1, e2, e3);
    rdft4<T, SIGN>(o0, o1, o2, o3);
    // o1 (1 + sign i) / sqrt 2 and o3 (-1 + sign i) / sqrt 2, the scale inside the last additions
    const float c = 0.70710678118654752440f;
    const float2 w1 = add_rot<T, SIGN>(o1, o1);
    const float2 w3 = make_float2(SIGN < 0 ? o3.y - o3.x : -o3.y - o3.x, SIGN < 0 ? -o3.x - o3.y : o3.x - o3.y);
    a[0] = cadd(e0, o0);
    a[4] = csub(e0, o0);
    a[1] = pfma(w1, splat(c), e1);
    a[5] = pfma(w1, splat(-c), e1);
    a[2] = add_rot<T, SIGN>(e2, o2);
    a[6] = sub_rot<T, SIGN>(e2, o2);
    a[3] = pfma(w3, splat(c), e3);
    a[7] = pfma(w3, splat(-c), e3);
  } else {
    dft8<T, SIGN>(a);
  }
}
// a + c v and a + sign i c v for a real constant c: one FMA per component where the arithmetic has it
template <typename T>
__device__ __forceinline__ C2<T> mac(C2<T> a, C2<T> v, T c) {
  if constexpr (std::is_same<T, df>::value) {
    return add<T>(a, scl<T>(v, c));
  } else if constexpr (std::is_same<T, float>::value) {
    return pfma(v, splat(c), a);
  } else {
    return make_double2(__fma_rn(c, v.x, a.x), __fma_rn(c, v.y, a.y));
  }
}
template <typename T, int SIGN>
__device__ __forceinline__ C2<T> mac_rot(C2<T> a, C2<T> v, T c) {
  if constexpr (std::is_same<T, df>::value) {
    return add_rot<T, SIGN>(a, scl<T>(v, c));
  } else {
    C2<T> r;
    r.x = fma(SIGN < 0 ? c : -c, v.y, a.x);
    r.y = fma(SIGN < 0 ? -c : c, v.x, a.y);
    return r;
  }
}
template <typename T, int SIGN>
__device__ __forceinline__ void rdft3(C2<T> *a) {
  const C2<T> s = add<T>(a[1], a[2]);
  const C2<T> d = sub<T>(a[1], a[2]);
  const C2<T> m = mac<T>(a[0], s, rneg(cst<T>(K_HALF)));
  a[0] = add<T>(a[0], s);
  if constexpr (std::is_same<T, df>::value) {
    const C2<T> r = scl<T>(d, cst<T>(K_SQRT3_2));
    a[1] = add_rot<T, SIGN>(m, r);
    a[2] = sub_rot<T, SIGN>(m, r);
  } else if constexpr (std::is_same<T, double>::value) {
    // The rounding error of sqrt(3)/2 would scale every value of every stage
    // alike and add up over stages, dimensions and directions (a 432^3 round
    // trip 7.2e-16, 72^3 5.8e-16): as d - (1 - sqrt(3)/2) d it is an eighth
    // of that, for two operations more.
    const T k = -0.133974596215561353236276829247063817;
    const C2<T> r = mac<T>(d, d, k);
    a[1] = add_rot<T, SIGN>(m, r);
    a[2] = sub_rot<T, SIGN>(m, r);
  } else {
    a[1] = mac_rot<T, SIGN>(m, d, cst<T>(K_SQRT3_2));
    a[2] = mac_rot<T, -SIGN>(m, d, cst<T>(K_SQRT3_2));
  }
}
template <typename T, int SIGN>
__device__ __forceinline__ void rdft5(C2<T> *a) {
  const C2<T> b1 = add<T>(a[1], a[4]), b2 = add<T>(a[2], a[3]);
  const C2<T> d1 = sub<T>(a[1], a[4]), d2 = sub<T>(a[2], a[3]);
  const T c1 = cst<T>(K_C72), c2 = cst<T>(K_C144), s1 = cst<T>(K_S72), s2 = cst<T>(K_S144);
  C2<T> p1, p2_;
  if constexpr (std::is_same<T, df>::value) {
    p1 = add<T>(a[0], add<T>(scl<T>(b1, c1), scl<T>(b2, c2)));
    p2_ = add<T>(a[0], add<T>(scl<T>(b1, c2), scl<T>(b2, c1)));
  } else {
    p1 = mac<T>(mac<T>(a[0], b2, c2), b1, c1);
    p2_ = mac<T>(mac<T>(a[0], b1, c2), b2, c1);
  }
  const C2<T> q1 = mac<T>(scl<T>(d2, s2), d1, s1);
  const C2<T> q2 = mac<T>(scl<T>(d1, s2), d2, rneg(s1));
  a[0] = add<T>(a[0], add<T>(b1, b2));
  a[1] = add_rot<T, SIGN>(p1, q1);
  a[4] = sub_rot<T, SIGN>(p1, q1);
  a[2] = add_rot<T, SIGN>(p2_, q2);
  a[3] = sub_rot<T, SIGN>(p2_, q2);
}

template <typename T, int SIGN, int R>
__device__ __forceinline__ void rdft(C2<T> *a);

// twiddles of the inner products: column k1 of row i2 times exp(sign 2 pi i i2 k1 / R)
template <typename T, int SIGN, int R, int A, int B, int I2, int K1>
__device__ __forceinline__ void ct_twiddle(C2<T> *row) {
  if constexpr (K1 < A) {
    row[K1] = mul_unit<T, SIGN, R, I2 * K1>(row[K1]);
    ct_twiddle<T, SIGN, R, A, B, I2, K1 + 1>(row);
  }
}
template <typename T, int SIGN, int R, int A, int B, int I2>
__device__ __forceinline__ void ct_rows(C2<T> (*y)[A], const C2<T> *a) {
  if constexpr (I2 < B) {
#pragma unroll
    for (int i1 = 0; i1 < A; ++i1) y[I2][i1] = a[i1 * B + I2];
    rdft<T, SIGN, A>(y[I2]);
    ct_twiddle<T, SIGN, R, A, B, I2, 1>(y[I2]);
    ct_rows<T, SIGN, R, A, B, I2 + 1>(y, a);
  }
}
// R = A B, powers of two: DFTs of A over the stride-B columns, twiddles, DFTs of B
template <typename T, int SIGN, int R, int A>
__device__ __forceinline__ void dft_ct(C2<T> *a) {
  constexpr int B = R / A;
  C2<T> y[B][A];
  ct_rows<T, SIGN, R, A, B, 0>(y, a);
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    C2<T> z[B];
#pragma unroll
    for (int i2 = 0; i2 < B; ++i2) z[i2] = y[i2][k1];
    rdft<T, SIGN, B>(z);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) a[k1 + A * k2] = z[k2];
  }
}
// the x of [0, m) with a x = 1 mod m
__host__ __device__ constexpr int mod_inverse(int a, int m) {
  for (int x = 1; x < m; ++x)
    if (a * x % m == 1) return x;
  return 0;
}
// R = A B, coprime: no twiddles (Good's index maps: input B i1 + A i2, output the k with remainders k1 mod A
// and k2 mod B)
template <typename T, int SIGN, int R, int A>
__device__ __forceinline__ void dft_pfa(C2<T> *a) {
  constexpr int B = R / A;
  constexpr int EA = B * mod_inverse(B, A), EB = A * mod_inverse(A, B);
  C2<T> y[B][A];
#pragma unroll
  for (int i2 = 0; i2 < B; ++i2) {
#pragma unroll
    for (int i1 = 0; i1 < A; ++i1) y[i2][i1] = a[(B * i1 + A * i2) % R];
    rdft<T, SIGN, A>(y[i2]);
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    C2<T> z[B];
#pragma unroll
    for (int i2 = 0; i2 < B; ++i2) z[i2] = y[i2][k1];
    rdft<T, SIGN, B>(z);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) {
      a[(EA * k1 + EB * k2) % R] = z[k2];
    }
  }
}

template <typename T, int SIGN, int R>
__device__ __forceinline__ void rdft(C2<T> *a) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const C2<T> t = add<T>(a[0], a[1]);
    a[1] = sub<T>(a[0], a[1]);
    a[0] = t;
  } else if constexpr (R == 3) {
    rdft3<T, SIGN>(a);
  } else if constexpr (R == 4) {
    rdft4<T, SIGN>(a[0], a[1], a[2], a[3]);
  } else if constexpr (R == 5) {
    rdft5<T, SIGN>(a);
  } else if constexpr (R == 8) {
    rdft8<T, SIGN>(a);
  } else if constexpr (R == 16) {
    dft_ct<T, SIGN, 16, 4>(a);
  } else if constexpr (R == 32) {
    dft_ct<T, SIGN, 32, 4>(a);
  } else if constexpr (R % 8 == 0) {
    dft_pfa<T, SIGN, R, 8>(a);  // 24
  } else if constexpr (R % 4 == 0) {
    dft_pfa<T, SIGN, R, 4>(a);  // 12, 20
  } else if constexpr (R % 2 == 0) {
    dft_pfa<T, SIGN, R, 2>(a);  // 6, 10
  } else {
    static_assert(R == 15, "radix");
    dft_pfa<T, SIGN, R, 3>(a);
  }
}

// Native FP64, power-of-two radix R without input twiddles (a first stage):
// every layer as radix-2 butterflies.  The even outputs of n values x_q are
// the transform of the sums x_q + x_{q+n/2}, the odd ones that of their
// differences with factors W_n^q; a node at depth d, reached by the choices
// in e, so adds its second half times W_{2^{d+1}}^e (y0 = a + t b,
// y1 = 2 a - y0: six FMAs; four additions where t is a quarter turn).
// Outputs in bit-reversed places.
__host__ __device__ constexpr int bit_reverse(int k, int R) {
  int r = 0;
  for (int b = 1; b < R; b <<= 1) {
    r = (r << 1) | (k & 1);
    k >>= 1;
  }
  return r;
}

template <int SIGN>
__device__ __forceinline__ void bfly_plain(double2 &a, double2 &b) {
  const double2 t = cadd(a, b);
  b = csub(a, b);
  a = t;
}
template <int SIGN>
__device__ __forceinline__ void bfly_plain_rot(double2 &a, double2 &b) {
  const double2 t = add_rot<double, SIGN>(a, b);
  b = sub_rot<double, SIGN>(a, b);
  a = t;
}
// N values at a, depth D, twiddle exponent E
template <int SIGN, int R, int N, int D, int E>
__device__ __forceinline__ void fma_node(double2 *a) {
  if constexpr (N > 1) {
    constexpr int H = N / 2;
    constexpr int HALF = D > 0 ? 1 << (D - 1) : 1;  // e and e + HALF differ by a quarter turn
    constexpr int EL = D > 0 ? E % HALF : 0;
    constexpr bool ROT = D > 0 && E >= HALF;
    if constexpr (EL == 0) {
#pragma unroll
      for (int q = 0; q < H; ++q) {
        if constexpr (ROT) bfly_plain_rot<SIGN>(a[q], a[q + H]);
        else bfly_plain<SIGN>(a[q], a[q + H]);
      }
    } else if constexpr (E * (32 >> (D + 1)) % 8 == 4) {
      // an odd eighth turn: (1 + sign i) b or (-1 + sign i) b by additions, its scale in the outputs' FMAs
      // (six operations as well, without the difference's doubled rounding)
      const double c = 0.707106781186547524400844362104849039;
#pragma unroll
      for (int q = 0; q < H; ++q) {
        const double2 b = a[q + H];
        double2 w = add_rot<double, SIGN>(b, b);
        if constexpr (ROT) w = SIGN < 0 ? make_double2(w.y, -w.x) : make_double2(-w.y, w.x);
        a[q + H] = make_double2(__fma_rn(-c, w.x, a[q].x), __fma_rn(-c, w.y, a[q].y));
        a[q] = make_double2(__fma_rn(c, w.x, a[q].x), __fma_rn(c, w.y, a[q].y));
      }
    } else {
      double re, im;
      unit16<double, SIGN, E * (32 >> (D + 1))>(re, im);
#pragma unroll
      for (int q = 0; q < H; ++q) bfly_tw<SIGN>(a[q], a[q + H], re, im);
    }
    fma_node<SIGN, R, H, D + 1, E>(a);
    fma_node<SIGN, R, H, D + 1, E + (1 << D)>(a + H);
  }
}

// Native FP64, twiddled radix 8 and 4 with fewer operations: a twiddle is
// w_q = i^m c_q (1 + i t_q) with |t_q| <= 1 (its angle within an eighth turn
// of i^m), so that x'_q = i^m x_q (1 + i t_q) takes two FMAs (the quarter
// turns are register selects and sign bits), and the scales c_q go into the
// butterflies' additions, which become FMAs with ratios of scales: 66
// operations per eight values against 72 in the radix-2 layers above, 22
// against 24 per four (after Linzer and Feig's FMA forms of the FFT).  The
// tables come from the host, rounded once: per j the t_q, the ratios, and the
// quarter turns, two bits a value.  512 points: 24.5 -> 23 operations a value,
// 720 -> 780 GB/s, and errors 2 % smaller (no doubled differences).
__device__ __forceinline__ double2 tan_turn(double2 v, double t, unsigned m) {
  const double p = (m & 1) ? v.y : v.x, r = (m & 1) ? v.x : v.y;
  // i^m v: the first part negative for m = 1, 2, the second for m = 2, 3
  const double x = __hiloint2double(__double2hiint(p) ^ (int)(((m ^ (m >> 1)) & 1u) << 31), __double2loint(p));
  const double y = __hiloint2double(__double2hiint(r) ^ (int)((m >> 1) << 31), __double2loint(r));
  return make_double2(__fma_rn(-t, y, x), __fma_rn(t, x, y));
}
template <int SIGN>
__device__ __forceinline__ void tan_dft8(double2 *a, const double2 *e) {
  const unsigned code = (unsigned)__double2loint(e[7].y);
  const double t[7] = {e[0].x, e[0].y, e[1].x, e[1].y, e[2].x, e[2].y, e[3].x};
#pragma unroll
  for (int q = 1; q < 8; ++q) a[q] = tan_turn(a[q], t[q - 1], (code >> (2 * (q - 1))) & 3u);
  const double rho[4] = {e[3].y, e[4].x, e[4].y, e[5].x};  // c_{q+4} / c_q
  const double c2 = e[5].y, c31 = e[6].x, c1 = e[6].y, c1h = e[7].x;
  double2 s[4], d[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    s[q] = mac<double>(a[q], a[q + 4], rho[q]);
    d[q] = mac<double>(a[q], a[q + 4], -rho[q]);
  }
  {
    const double2 A0 = mac<double>(s[0], s[2], c2), A1 = mac<double>(s[0], s[2], -c2);
    const double2 B0 = mac<double>(s[1], s[3], c31), B1 = mac<double>(s[1], s[3], -c31);
    a[0] = mac<double>(A0, B0, c1);
    a[4] = mac<double>(A0, B0, -c1);
    a[2] = mac_rot<double, SIGN>(A1, B1, c1);
    a[6] = mac_rot<double, -SIGN>(A1, B1, c1);
  }
  const double2 A0 = mac_rot<double, SIGN>(d[0], d[2], c2), A1 = mac_rot<double, -SIGN>(d[0], d[2], c2);
  const double2 B0 = mac_rot<double, SIGN>(d[1], d[3], c31), B1 = mac_rot<double, -SIGN>(d[1], d[3], c31);
  // times the eighth turn: (1 + sign i) / sqrt 2, its scale with c_1
  const double2 G = add_rot<double, SIGN>(B0, B0), H = add_rot<double, SIGN>(B1, B1);
  a[1] = mac<double>(A0, G, c1h);
  a[5] = mac<double>(A0, G, -c1h);
  a[3] = mac_rot<double, SIGN>(A1, H, c1h);
  a[7] = mac_rot<double, -SIGN>(A1, H, c1h);
}
template <int SIGN>
__device__ __forceinline__ void tan_dft4(double2 *a, const double2 *e) {
  const unsigned code = (unsigned)__double2loint(e[3].x);
  a[1] = tan_turn(a[1], e[0].x, code & 3u);
  a[2] = tan_turn(a[2], e[0].y, (code >> 2) & 3u);
  a[3] = tan_turn(a[3], e[1].x, (code >> 4) & 3u);
  const double c2 = e[1].y, c31 = e[2].x, c1 = e[2].y;
  const double2 A0 = mac<double>(a[0], a[2], c2), A1 = mac<double>(a[0], a[2], -c2);
  const double2 B0 = mac<double>(a[1], a[3], c31), B1 = mac<double>(a[1], a[3], -c31);
  a[0] = mac<double>(A0, B0, c1);
  a[2] = mac<double>(A0, B0, -c1);
  a[1] = mac_rot<double, SIGN>(A1, B1, c1);
  a[3] = mac_rot<double, -SIGN>(A1, B1, c1);
}
// Entries of a twiddled stage of radix r after lp points, [entry][j], from
// the host: for e in order t_1 ... t_{r-1}, then the ratios.  A scale is that
// of the rounded t, a ratio that to the rounded scales below it, so that a
// value's magnitude carries one rounding (48 points: 0.61 -> 0.34 half units
// rms; a 48^3 round trip 4.33e-16 with every entry rounded by itself).
inline void tan_table(int r, int lp, int sign, double *out) {
  const long double pi = 3.141592653589793238462643383279502884L;
  for (int j = 0; j < lp; ++j) {
    long double c[8], t[8];
    uint32_t code = 0;
    for (int q = 0; q < r; ++q) {
      // angle 2 pi q j / (r lp): quarter turns m and a rest within an eighth
      const long long num = (long long)q * j, den = (long long)r * lp;
      const long long m = (8 * num + den) / (2 * den);
      const long double phi = sign * 2 * pi * ((long double)(4 * num - m * den) / (long double)(4 * den));
      t[q] = (double)tanl(phi);
      c[q] = 1 / sqrtl(1 + t[q] * t[q]);
      if (q) code |= (uint32_t)((sign < 0 ? 4 - m % 4 : m) % 4) << (2 * (q - 1));
    }
    double bits;
    const uint64_t word = code;
    memcpy(&bits, &word, 8);
    double v[16];
    int k = 0;
    for (int q = 1; q < r; ++q) v[k++] = (double)t[q];
    const double c1 = (double)c[1], c2 = (double)c[2], c31 = (double)(c[3] / c1);
    if (r == 8) {
      const long double below[4] = {1, c1, c2, (long double)c31 * c1};
      for (int q = 0; q < 4; ++q) v[k++] = (double)(c[q + 4] / below[q]);
      v[k++] = c2;
      v[k++] = c31;
      v[k++] = c1;
      v[k++] = (double)(c[1] * sqrtl(0.5L));
      v[k++] = bits;
    } else {
      v[k++] = c2;
      v[k++] = c31;
      v[k++] = c1;
      v[k++] = bits;
      v[k++] = 0;
    }
    for (int e = 0; e < r; ++e) {
      out[2 * (e * lp + j)] = v[2 * e];
      out[2 * (e * lp + j) + 1] = v[2 * e + 1];
    }
  }
}

// ---------------------------------------------------------------- the lines of a pass

// An axis the lines are numbered along: its length (with the constants of a
// division by it), its dimension, the coordinate step and whether it is the
// twiddle's y.
struct reg_axis {
  uint32_t len, magic, shift;
  int32_t dim, mul, isy;
};
struct line_axes {
  uint32_t total;  // lines of all jobs
  uint32_t nax;
  reg_axis ax[5];
};
struct reg_lines : line_axes {
  dmg_fft_rows rows;
};
// r / len for r < 2^31
__device__ __forceinline__ uint32_t fast_div(uint32_t r, const reg_axis &a) {
  return (__umulhi(r, a.magic) + r) >> a.shift;
}

// coordinates of a line's first value, the twiddle's y, and its job (returned)
__device__ __forceinline__ uint32_t line_place(const line_axes &lines, uint32_t line, int *x, int &y) {
  uint32_t r = line;
  x[0] = x[1] = x[2] = 0;
  y = 0;
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    if (i < (int)lines.nax) {
      const reg_axis &ax = lines.ax[i];
      const uint32_t q = fast_div(r, ax);
      const int c = (int)(r - q * ax.len);
      r = q;
      const int step = c * ax.mul;
      x[0] += ax.dim == 0 ? step : 0;
      x[1] += ax.dim == 1 ? step : 0;
      x[2] += ax.dim == 2 ? step : 0;
      y += ax.isy ? c : 0;
    }
  }
  return r;
}
__device__ __forceinline__ int64_t line_address(const dmg_fft_layout &L, int ndim, const int *x) {
  int64_t a = L.base;
#pragma unroll
  for (int d = 0; d < DMG_FFT_MAXDIM; ++d)
    if (d < ndim) a += __ldg(L.tab[d] + x[d]);
  return a;
}

// LINES: the lines per block (0: the schedule's)
template <typename T, int NF, bool TF, bool INV, int LINES>
struct RegShape {
  static constexpr RegSched S = reg_sched(reg_kind<T>(), NF, TF, INV, LINES);
  static constexpr int TL = S.tl, W = S.w, NTH = TL * W;
  static constexpr int ES = (int)sizeof(C2<T>);
  static constexpr int V = 128 / ES;  // values per shared-memory wavefront
  // stage f: radix, product of the earlier radices, values per row after it, butterflies, rounds per thread
  static constexpr int R(int f) { return S.r[f]; }
  static constexpr int LP(int f) { return f == 0 ? 1 : LP(f - 1) * S.r[f - 1]; }
  static constexpr int M(int f) { return NF / (LP(f) * S.r[f]); }
  static constexpr int NB(int f) { return NF / S.r[f]; }
  static constexpr int TR(int f) { return (NB(f) + TL - 1) / TL; }
  // The exchange after stage f holds row J (of LP R) and value k (of m) at
  // J P + k; the next stage's thread (j', k') reads J = j', k = q m' + k'.
  // The row pitch P leaves consecutive threads of the next stage in
  // different banks: P an odd multiple of m' while m' is less than the lanes
  // of a wavefront that run along the line (the lines take the others in the
  // form along v1).
  static constexpr int pitch(int f) {
    const int m = M(f), mn = M(f + 1);
    const int lanes = !TF ? (W >= V ? 1 : V / W) : TL >= V ? V : TL >= 8 ? 8 : 4;
    if (mn >= lanes || !is_pow2(mn)) return m;
    int p = m;
    while (p % (2 * mn) != mn) ++p;
    return p;
  }
  static constexpr int rows(int f) { return LP(f) * S.r[f]; }
  // slot-order exchange (along t): rows of M(0) values before the first stage, of LP(last) after the last
  static constexpr int in_row = M(0), in_pitch = M(0) | 1;
  static constexpr int out_row = LP(S.ns - 1), out_pitch = LP(S.ns - 1) | 1;
  static constexpr int cmax(int a, int b) { return a > b ? a : b; }
  static constexpr int line_values() {
    int v = 0;
    for (int f = 0; f + 1 < S.ns; ++f) v = cmax(v, rows(f) * pitch(f));
    if (TF) v = cmax(v, cmax((NF / in_row) * in_pitch, (NF / out_row) * out_pitch));
    return v;
  }
  // line pitch along t: the lines of a wavefront start in different banks
  static constexpr int line_pitch() {
    int v = line_values();
    if (TL < V)
      while (v % V != TL % V) ++v;
    return v;
  }
  static constexpr size_t buf_bytes() { return (size_t)W * (TF ? line_pitch() : line_values()) * ES; }
  // twiddle table entries per j of stage f
  static constexpr bool tan(int f) { return std::is_same<T, double>::value && f > 0; }
  static constexpr bool tan_radices() {
    for (int f = 1; f < S.ns; ++f)
      if (tan(f) && S.r[f] != 4 && S.r[f] != 8) return false;
    return true;
  }
  static_assert(tan_radices(), "native FP64: the twiddled stages have radix 4 or 8");
  static constexpr bool fma(int f) { return std::is_same<T, double>::value && f == 0 && is_pow2(S.r[f]) && S.r[f] <= 32; }
  static constexpr int tw_per_j(int f) { return f == 0 ? 0 : tan(f) ? S.r[f] : S.r[f] - 1; }
  // (8-byte entries lie in pairs, so that one 16-byte read gives a thread two)
  static constexpr int tw_rows(int f) { return ES == 8 ? (tw_per_j(f) + 1) & ~1 : tw_per_j(f); }
  static constexpr int tw_base(int f) { return f <= 1 ? 0 : tw_base(f - 1) + tw_rows(f - 1) * LP(f - 1); }
  static constexpr int tw_total() { return tw_base(S.ns - 1) + tw_rows(S.ns - 1) * LP(S.ns - 1); }
  // place of entry e of row j (the schedule enters as constants: its object lives on the host)
  template <int F>
  __device__ static __forceinline__ int tw_at(int e, int j) {
    constexpr int base = tw_base(F), lp = LP(F);
    return base + (ES == 8 ? ((e >> 1) * lp + j) * 2 + (e & 1) : e * lp + j);
  }
  static constexpr size_t al16(size_t x) { return (x + 15) & ~(size_t)15; }
  // shared memory: exchange buffer, twiddles, the sides' offsets (8 bytes a slot on the side that may be in
  // slot order along t: the output forward, the input inverse), line pointers
  static constexpr size_t tw_off() { return al16(buf_bytes()); }
  static constexpr size_t tin_off() { return al16(tw_off() + (size_t)tw_total() * ES); }
  static constexpr size_t tout_off() { return al16(tin_off() + (size_t)NF * (TF && INV ? 8 : 4)); }
  static constexpr size_t ptr_off() {
    return al16(tout_off() + (size_t)NF * (TF && !INV ? 8 : 4));
  }
  // AHEAD_COPY: the next tile's values, [place in the thread][thread]
  static_assert(!TF || S.ahead != AHEAD_COPY, "copies ahead are written for the form along v1");
  static constexpr int stage_values() { return TR(0) * S.r[0]; }
  static constexpr size_t stage_off() { return al16(ptr_off() + (TF ? (size_t)W * 8 : 0)); }
  static constexpr size_t smem() {
    return stage_off() + (S.ahead == AHEAD_COPY ? al16((size_t)stage_values() * NTH * ES) : 0);
  }
};

// ---------------------------------------------------------------- the kernel

// (tan: the pass's host-made entries, at the places of the whole table)
template <typename T, int SIGN, int NF, bool TF, int LINES, int F>
__device__ __forceinline__ void reg_twiddles(const C2<T> *roots, const C2<T> *tan, C2<T> *tws, int tid) {
  using G = RegShape<T, NF, TF, (SIGN > 0), LINES>;
  if constexpr (F < G::S.ns) {
    constexpr int LP = G::LP(F), R = G::R(F), PJ = G::tw_per_j(F), TS = NF / (LP * R);
    for (int i = tid; i < PJ * LP; i += G::NTH) {
      const int e = i / LP, j = i - e * LP;
      if constexpr (G::tan(F)) {
        const int at = G::template tw_at<F>(e, j);
        tws[at] = __ldg(tan + at);
        continue;
      }
      tws[G::template tw_at<F>(e, j)] = root_at<T, SIGN>(roots, (e + 1) * j * TS % NF);
    }
    reg_twiddles<T, SIGN, NF, TF, LINES, F + 1>(roots, tan, tws, tid);
  }
}

// butterflies of stage F on the thread's registers, input twiddles included
template <typename T, int SIGN, int NF, bool TF, int LINES, int F>
__device__ __forceinline__ void reg_butterfly(C2<T> *a, const C2<T> *tws, int j) {
  using G = RegShape<T, NF, TF, (SIGN > 0), LINES>;
  constexpr int R = G::R(F), LP = G::LP(F);
  const C2<T> *tw = tws + G::template tw_at<F>(0, j);
  if constexpr (G::tan(F)) {
    double2 e[R];
#pragma unroll
    for (int i = 0; i < R; ++i) e[i] = tw[i * LP];
    if constexpr (R == 8) tan_dft8<SIGN>(a, e);
    else tan_dft4<SIGN>(a, e);
  } else if constexpr (G::fma(F)) {
    fma_node<SIGN, R, R, 0, 0>(a);
    C2<T> y[R];
#pragma unroll
    for (int s = 0; s < R; ++s) y[s] = a[bit_reverse(s, R)];
#pragma unroll
    for (int s = 0; s < R; ++s) a[s] = y[s];
  } else {
    if constexpr (F > 0 && G::ES == 8) {
#pragma unroll
      for (int e = 0; e < R - 1; e += 2) {
        const float4 w = *reinterpret_cast<const float4 *>(tw + e * LP);
        a[e + 1] = rmul<T>(a[e + 1], make_float2(w.x, w.y));
        if (e + 2 < R) a[e + 2] = rmul<T>(a[e + 2], make_float2(w.z, w.w));
      }
    } else if constexpr (F > 0) {
#pragma unroll
      for (int q = 1; q < R; ++q) a[q] = rmul<T>(a[q], tw[(q - 1) * LP]);
    }
    rdft<T, SIGN, R>(a);
  }
}

// the stages from F on: the exchange into stage F's registers and its
// butterflies; ends with the last stage's values in a (rounds of R each).
// after_write: called once the first exchange's values are written.
// bx: the thread's first buffer position (its line's).  STEP: distance of
// neighbouring positions of a line (W along v1, 1 along t).
template <typename T, int SIGN, int NF, bool TF, int LINES, int F, typename Then>
__device__ __forceinline__ void reg_exchange(const C2<T> *src, C2<T> *bx, const C2<T> *tws, int bl, C2<T> *out,
                                             Then &&after_write) {
  using G = RegShape<T, NF, TF, (SIGN > 0), LINES>;
  constexpr int STEP = TF ? 1 : G::W;
  constexpr int P = G::pitch(F - 1);
  // write stage F - 1's results
  {
    constexpr int R = G::R(F - 1), LP = G::LP(F - 1), M = G::M(F - 1), NB = G::NB(F - 1), TR = G::TR(F - 1);
    __syncthreads();  // the buffer's previous values have been read
#pragma unroll
    for (int tr = 0; tr < TR; ++tr) {
      const int b = bl + tr * G::TL;
      if (NB % G::TL == 0 || b < NB) {
        C2<T> *w = bx + ((b / M) * P + b % M) * STEP;
#pragma unroll
        for (int s = 0; s < R; ++s) w[s * LP * P * STEP] = src[tr * R + s];
      }
    }
    __syncthreads();
  }
  if constexpr (F == 1) after_write();
  constexpr int R = G::R(F), M = G::M(F), NB = G::NB(F), TR = G::TR(F);
  C2<T> a[TR * R];
#pragma unroll
  for (int tr = 0; tr < TR; ++tr) {
    const int b = bl + tr * G::TL;
    if (NB % G::TL == 0 || b < NB) {
      const int j = b / M, k = b % M;
      const C2<T> *x = bx + (j * P + k) * STEP;
#pragma unroll
      for (int q = 0; q < R; ++q) a[tr * R + q] = x[q * M * STEP];
    }
  }
#pragma unroll
  for (int tr = 0; tr < TR; ++tr) {
    const int b = bl + tr * G::TL;
    if (NB % G::TL == 0 || b < NB) reg_butterfly<T, SIGN, NF, TF, LINES, F>(a + tr * R, tws, b / M);
  }
  if constexpr (F + 1 < G::S.ns) {
    reg_exchange<T, SIGN, NF, TF, LINES, F + 1>(a, bx, tws, bl, out, after_write);
  } else {
#pragma unroll
    for (int i = 0; i < TR * R; ++i) out[i] = a[i];
  }
}

// a value as it lies in the input array (complex128 bits for a double-float pass that reads complex128)
template <typename T>
__device__ __forceinline__ C2<T> reg_load(const unsigned char *at) {
  if constexpr (sizeof(C2<T>) == 16) {
    const float4 v = *reinterpret_cast<const float4 *>(at);
    C2<T> r;
    memcpy(&r, &v, 16);
    return r;
  } else {
    return *reinterpret_cast<const C2<T> *>(at);
  }
}
template <typename T>
__device__ __forceinline__ void reg_store(unsigned char *at, C2<T> v) {
  if constexpr (sizeof(C2<T>) == 16) {
    float4 w;
    memcpy(&w, &v, 16);
    *reinterpret_cast<float4 *>(at) = w;
  } else {
    *reinterpret_cast<C2<T> *>(at) = v;
  }
}
template <typename T>
__device__ __forceinline__ void reg_convert(C2<T> &v, int sexp) {
  if constexpr (std::is_same<T, df>::value) {
    double2 d;
    memcpy(&d, &v, 16);
    const df re = to_df(d.x, sexp), im = to_df(d.y, sexp);
    v = dfc{make_float2(re.h, im.h), make_float2(re.l, im.l)};
  }
}

template <typename T>
__device__ __forceinline__ void reg_unconvert(C2<T> &v, int sexp) {
  if constexpr (std::is_same<T, df>::value) {
    const double2 d = make_double2(from_df(df{v.h.x, v.l.x}, sexp), from_df(df{v.h.y, v.l.y}, sexp));
    memcpy(&v, &d, 16);
  }
}

// Ask L2 for the values of a tile (the block's next one), a 128-byte line of
// memory per request where the lines (along v1) or the values of a line
// (along t) are contiguous; a hint only.
template <typename T, int SIGN, int NF, bool TF, int LINES>
__device__ __forceinline__ void reg_prefetch(const dmg_fft_pass &p, const dmg_fft_batch &bt, const reg_lines &lines,
                                             uint32_t tile, uint32_t ntiles, const int32_t *tin, const int2 *sin,
                                             bool slot_in, int tid, int l, int bl) {
  using G = RegShape<T, NF, TF, (SIGN > 0), LINES>;
  constexpr int PER = 128 / G::ES;                        // values per request
  constexpr int CH = G::W > PER ? (G::W + PER - 1) / PER : 1;  // requests per row of lines
  if (tile >= ntiles) return;
  const uint32_t line = tile * G::W + (TF ? l : (tid % CH) * PER);
  if (line >= lines.total) return;
  int x[DMG_FFT_MAXDIM], y;
  const uint32_t job = line_place(lines, line, x, y);
  const unsigned char *src = static_cast<const unsigned char *>(bt.src[job]) + line_address(p.in, p.ndim, x) * G::ES;
  if constexpr (TF) {
    for (int t = bl * PER; t < NF; t += G::TL * PER)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(src + (int64_t)(slot_in ? sin[t].y : tin[t]) * G::ES));
  } else {
    for (int t = tid / CH; t < NF; t += G::NTH / CH)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(src + (int64_t)tin[t] * G::ES));
  }
}

template <typename T, int SIGN, int NF, bool TF, int LINES>
__global__ void __launch_bounds__(RegShape<T, NF, TF, (SIGN > 0), LINES>::NTH, RegShape<T, NF, TF, (SIGN > 0), LINES>::S.minb)
    fft_reg_kernel(const __grid_constant__ dmg_fft_pass p, const __grid_constant__ dmg_fft_batch bt,
                   const __grid_constant__ reg_lines lines) {
  using G = RegShape<T, NF, TF, (SIGN > 0), LINES>;
  constexpr int TL = G::TL, W = G::W, NTH = G::NTH, ES = G::ES, NS = G::S.ns;
  constexpr bool DFT = std::is_same<T, df>::value;
  // (constants: device code must not evaluate the schedule's functions, whose table is a host object)
  constexpr size_t TW_AT = G::tw_off(), TIN_AT = G::tin_off(), TOUT_AT = G::tout_off(), PTR_AT = G::ptr_off();
  constexpr int LPITCH = G::line_pitch();
  extern __shared__ __align__(16) unsigned char sm[];
  C2<T> *buf = reinterpret_cast<C2<T> *>(sm);
  C2<T> *tws = reinterpret_cast<C2<T> *>(sm + TW_AT);
  // offsets along t: by transform coordinate (slot order folded in); along t in slot order: by slot, with
  // the position in the exchange buffer
  int32_t *tin = reinterpret_cast<int32_t *>(sm + TIN_AT);
  int32_t *tout = reinterpret_cast<int32_t *>(sm + TOUT_AT);
  int2 *sin = reinterpret_cast<int2 *>(tin), *sout = reinterpret_cast<int2 *>(tout);
  const unsigned char **lptr = reinterpret_cast<const unsigned char **>(sm + PTR_AT);
  const int tid = threadIdx.x;
  const bool slot_in = TF && SIGN > 0 && p.perm_in, slot_out = TF && SIGN < 0 && p.perm_out;

  reg_twiddles<T, SIGN, NF, TF, LINES, 1>(reinterpret_cast<const C2<T> *>(p.roots), reinterpret_cast<const C2<T> *>(p.tan), tws, tid);
  {
    const int d0 = p.kdim[0], m0 = p.kisz[0] ? p.A[d0] : 1;
    const int64_t *ti = p.in.tab[d0], *to = p.out.tab[d0];
    const int64_t i0 = __ldg(ti), o0 = __ldg(to);
    for (int s = tid; s < NF; s += NTH) {
      // layout slot s holds line position k of a side in slot order
      const int k = (p.perm_in || p.perm_out) ? s / p.perm_a + p.perm_b * (s % p.perm_a) : s;
      const int32_t oi = (int32_t)(__ldg(ti + (int64_t)s * m0) - i0), oo = (int32_t)(__ldg(to + (int64_t)s * m0) - o0);
      if (slot_in) sin[s] = make_int2((k / G::in_row) * G::in_pitch + k % G::in_row, oi);
      else tin[p.perm_in ? k : s] = oi;
      if (slot_out) sout[s] = make_int2((k / G::out_row) * G::out_pitch + k % G::out_row, oo);
      else tout[p.perm_out ? k : s] = oo;
    }
  }
  __syncthreads();

  const int l = TF ? tid / TL : tid % W, bl = TF ? tid % TL : tid / W;
  C2<T> *const bx = TF ? buf + l * LPITCH : buf + l;
  const bool in64 = DFT && p.in_fp64, out64 = DFT && p.out_fp64;
  // the twiddle's table and its strides along k and y (the order whose neighbouring entries the lanes read)
  const int td = p.t >> 1;
  const bool kmaj = !TF && p.kdim[1] == td && !p.kisz[1];
  const C2<T> *const twt = reinterpret_cast<const C2<T> *>(kmaj ? p.twk[td] : p.twy[td]);
  const int tw_k = kmaj ? p.A[td] : 1, tw_y = kmaj ? 1 : NF;

  const uint32_t ntiles = (lines.total + W - 1) / W;
  constexpr int R1 = G::R(0), M1 = G::M(0), NB1 = G::NB(0), TR1 = G::TR(0);
  // in slot order (along t, inverse): lines at a time, slots per thread and line
  constexpr int LS = NTH >= NF ? NTH / NF : 1, J = NTH >= NF ? 1 : (NF + NTH - 1) / NTH, LI = (W + LS - 1) / LS;
  const int s0 = NTH >= NF ? tid % NF : tid, l0 = NTH >= NF ? tid / NF : 0;

  // the copies of a tile's values into the staging area (AHEAD_COPY)
  constexpr bool COPY = G::S.ahead == AHEAD_COPY;
  constexpr size_t STAGE_AT = G::stage_off();
  C2<T> *const stg = reinterpret_cast<C2<T> *>(sm + STAGE_AT) + tid;
  auto source_of = [&](uint32_t tile) -> const unsigned char * {
    const uint32_t line = tile * W + l;
    if (line >= lines.total) return nullptr;
    int x[DMG_FFT_MAXDIM], y;
    const uint32_t job = line_place(lines, line, x, y);
    return static_cast<const unsigned char *>(bt.src[job]) + line_address(p.in, p.ndim, x) * ES;
  };
  auto start_copies = [&](uint32_t tile) {
    if (const unsigned char *src = source_of(tile)) {
#pragma unroll
      for (int tr = 0; tr < TR1; ++tr) {
        const int b = bl + tr * TL;
        if (NB1 % TL == 0 || b < NB1) {
          if (lines.rows.sum_in) {
            const unsigned char *sb = src + (int64_t)tin[b] * ES;
#pragma unroll
            for (int q = 0; q < R1; ++q)
              copy_async<ES>(stg + (tr * R1 + q) * NTH, sb + (int64_t)lines.rows.in[q] * ES);
          } else {
#pragma unroll
            for (int q = 0; q < R1; ++q)
              copy_async<ES>(stg + (tr * R1 + q) * NTH, src + (int64_t)tin[b + q * M1] * ES);
          }
        }
      }
    }
    copy_async_commit();
  };
  if constexpr (COPY) start_copies(blockIdx.x);

  for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const uint32_t line = tile * W + l;
    const bool act = line < lines.total;
    // the line's place: coordinates per dimension, then its address on each side
    const unsigned char *src = nullptr;
    unsigned char *dst = nullptr;
    int ytw = 0, sexp = 0;
    if (act) {
      int x[DMG_FFT_MAXDIM];
      const uint32_t r = line_place(lines, line, x, ytw);
      const int64_t ai = line_address(p.in, p.ndim, x), ao = line_address(p.out, p.ndim, x);
      src = static_cast<const unsigned char *>(bt.src[r]) + ai * ES;
      dst = static_cast<unsigned char *>(bt.dst[r]) + ao * ES;
      if (DFT && (in64 || out64)) sexp = __ldg(bt.scale_exp[r]) - 1022;
    }

    // ---- the first stage's values ----
    C2<T> a[TR1 * R1];
    if constexpr (COPY) copy_async_wait_all();  // (the thread's own copies)
    if (TF && slot_in) {
      // in slot order through shared memory: lanes run along the slots
      C2<T> v[LI * J];
      __syncthreads();  // the buffer and the pointers of the previous tile have been read
      if (bl == 0) lptr[l] = src;
      __syncthreads();
#pragma unroll
      for (int i = 0; i < LI; ++i) {
        const int lc = l0 + i * LS;
        const unsigned char *lp = l0 < LS && lc < W ? lptr[lc] : nullptr;
#pragma unroll
        for (int j = 0; j < J; ++j) {
          const int s = s0 + j * NTH;
          v[i * J + j] = C2<T>{};
          if (lp && (NTH >= NF || NF % NTH == 0 || s < NF)) v[i * J + j] = reg_load<T>(lp + (int64_t)sin[s].y * ES);
        }
      }
#pragma unroll
      for (int i = 0; i < LI; ++i) {
        const int lc = l0 + i * LS;
#pragma unroll
        for (int j = 0; j < J; ++j) {
          const int s = s0 + j * NTH;
          if (l0 < LS && lc < W && (NTH >= NF || NF % NTH == 0 || s < NF))
            buf[lc * LPITCH + sin[s].x] = v[i * J + j];
        }
      }
      __syncthreads();
#pragma unroll
      for (int tr = 0; tr < TR1; ++tr) {
        const int b = bl + tr * TL;
        if (NB1 % TL == 0 || b < NB1) {
#pragma unroll
          for (int q = 0; q < R1; ++q) a[tr * R1 + q] = bx[q * G::in_pitch + b];
        }
      }
    } else if (COPY && act) {
#pragma unroll
      for (int i = 0; i < TR1 * R1; ++i) a[i] = stg[i * NTH];
    } else if (act) {
#pragma unroll
      for (int tr = 0; tr < TR1; ++tr) {
        const int b = bl + tr * TL;
        if (NB1 % TL == 0 || b < NB1) {
          if (lines.rows.sum_in) {
            const unsigned char *sb = src + (int64_t)tin[b] * ES;
#pragma unroll
            for (int q = 0; q < R1; ++q) a[tr * R1 + q] = reg_load<T>(sb + (int64_t)lines.rows.in[q] * ES);
          } else {
#pragma unroll
            for (int q = 0; q < R1; ++q) a[tr * R1 + q] = reg_load<T>(src + (int64_t)tin[b + q * M1] * ES);
          }
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < TR1 * R1; ++i) a[i] = C2<T>{};
    }
    if constexpr (G::S.ahead == AHEAD_L2) reg_prefetch<T, SIGN, NF, TF, LINES>(p, bt, lines, tile + gridDim.x, ntiles, tin, sin, slot_in, tid, l, bl);
    if (in64) {
#pragma unroll
      for (int i = 0; i < TR1 * R1; ++i) reg_convert<T>(a[i], sexp);
    }
    if (SIGN > 0 && p.twiddle == 2 && act && ytw) {
#pragma unroll
      for (int tr = 0; tr < TR1; ++tr) {
        const int b = bl + tr * TL;
        if (NB1 % TL == 0 || b < NB1) {
#pragma unroll
          for (int q = 0; q < R1; ++q)
            a[tr * R1 + q] = rmul<T>(a[tr * R1 + q], root_at<T, 1>(twt, (b + q * M1) * tw_k + ytw * tw_y));
        }
      }
    }
#pragma unroll
    for (int tr = 0; tr < TR1; ++tr) {
      const int b = bl + tr * TL;
      if (NB1 % TL == 0 || b < NB1) reg_butterfly<T, SIGN, NF, TF, LINES, 0>(a + tr * R1, tws, 0);
    }

    // ---- the other stages ----
    constexpr int RL = G::R(NS - 1), LPL = G::LP(NS - 1), NBL = G::NB(NS - 1), TRL = G::TR(NS - 1);
    C2<T> y[TRL * RL];
    // (the staging area has been read by the exchange's barriers)
    reg_exchange<T, SIGN, NF, TF, LINES, 1>(a, bx, tws, bl, y, [&]() {
      if constexpr (COPY) start_copies(tile + gridDim.x);
    });
    if (SIGN < 0 && p.twiddle == 1 && act && ytw) {
#pragma unroll
      for (int tr = 0; tr < TRL; ++tr) {
        const int b = bl + tr * TL;
        if (NBL % TL == 0 || b < NBL) {
#pragma unroll
          for (int s = 0; s < RL; ++s)
            y[tr * RL + s] = rmul<T>(y[tr * RL + s], root_at<T, -1>(twt, (b + s * LPL) * tw_k + ytw * tw_y));
        }
      }
    }

    // ---- results to the output layout ----
    if (out64) {
#pragma unroll
      for (int i = 0; i < TRL * RL; ++i) reg_unconvert<T>(y[i], sexp);
    }
    if (TF && slot_out) {
      __syncthreads();
      if (bl == 0) lptr[l] = dst;
#pragma unroll
      for (int tr = 0; tr < TRL; ++tr) {
        const int b = bl + tr * TL;
        if (NBL % TL == 0 || b < NBL) {
#pragma unroll
          for (int s = 0; s < RL; ++s) bx[s * G::out_pitch + b] = y[tr * RL + s];
        }
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const int s = s0 + j * NTH;
        if (l0 < LS && (NTH >= NF || NF % NTH == 0 || s < NF)) {
          const int2 so = sout[s];
#pragma unroll
          for (int i = 0; i < LI; ++i) {
            const int lc = l0 + i * LS;
            if (W % LS == 0 || lc < W) {
              unsigned char *lp = const_cast<unsigned char *>(lptr[lc]);
              if (lp) reg_store<T>(lp + (int64_t)so.y * ES, buf[lc * LPITCH + so.x]);
            }
          }
        }
      }
    } else if (act) {
#pragma unroll
      for (int tr = 0; tr < TRL; ++tr) {
        const int b = bl + tr * TL;
        if (NBL % TL == 0 || b < NBL) {
          // (along t, inverse: the table form measured faster, 5040 against 4500 GB/s at 1024 points FP32)
          if (!(TF && SIGN > 0) && lines.rows.sum_out) {
            unsigned char *db = dst + (int64_t)tout[b] * ES;
#pragma unroll
            for (int s = 0; s < RL; ++s) reg_store<T>(db + (int64_t)lines.rows.out[s] * ES, y[tr * RL + s]);
          } else {
#pragma unroll
            for (int s = 0; s < RL; ++s) reg_store<T>(dst + (int64_t)tout[b + s * LPL] * ES, y[tr * RL + s]);
          }
        }
      }
    }
  }
}

// ---------------------------------------------------------------- launch

template <typename T, int SIGN, int NF, bool TF, int LINES = 0>
int launch_reg_k(const dmg_fft_pass &p, const dmg_fft_batch &bt, reg_lines lines, cudaStream_t s) {
  using G = RegShape<T, NF, TF, (SIGN > 0), LINES>;
  constexpr size_t smem = G::smem();
  static_assert((smem + 1024) * G::S.minb <= 233472, "shared memory of the resident blocks");
  // offsets made for other radices are no use here: the kernel reads its tables instead
  if (lines.rows.r_in != G::S.r[0]) lines.rows.sum_in = 0;
  if (lines.rows.r_out != G::S.r[G::S.ns - 1]) lines.rows.sum_out = 0;
  if (std::is_same<T, double>::value && !p.tan) return dmg_error(DMG_ERR_ARG, "fft pass: no twiddle table");
  auto k = fft_reg_kernel<T, SIGN, NF, TF, LINES>;
  int dev = 0, nsm = 0, per_sm = 0;
  cudaError_t es = allow_smem(k, smem);
  if (es == cudaSuccess) es = resident_blocks(k, G::NTH, smem, &per_sm);
  if (es != cudaSuccess) return dmg_error(DMG_ERR_CUDA, "fft pass smem %zu: %s", smem, cudaGetErrorString(es));
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (per_sm < 1) return dmg_error(DMG_ERR_UNSUPPORTED, "fft pass does not fit on an SM (smem %zu)", smem);
  int64_t grid = (int64_t)nsm * per_sm;
  const int64_t ntiles = ((int64_t)lines.total + G::W - 1) / G::W;
  if (grid > ntiles) grid = ntiles;
  if (grid < 1) return DMG_OK;
  k<<<(unsigned)grid, G::NTH, smem, s>>>(p, bt, lines);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return dmg_error(DMG_ERR_CUDA, "fft pass launch: %s", cudaGetErrorString(e));
  return DMG_OK;
}

// The axes a pass's lines are numbered along: v1, v2, the batch sub-axes (the
// jobs are what remains of the line number).
inline line_axes line_axes_of(const dmg_fft_pass &p, const dmg_fft_batch &bt) {
  line_axes g;
  memset(&g, 0, sizeof(g));
  uint64_t total = (uint64_t)bt.count;
  auto axis = [&](int sub, int len) {
    total *= (uint64_t)len;
    if (len <= 1) return;
    reg_axis &a = g.ax[g.nax++];
    uint32_t l = 0;
    while ((1ull << l) < (uint64_t)len) ++l;
    a.len = (uint32_t)len;
    a.shift = l;
    a.magic = (uint32_t)(((1ull << 32) * ((1ull << l) - (uint64_t)len)) / (uint64_t)len + 1);
    a.dim = sub >> 1;
    a.mul = (sub & 1) ? p.A[sub >> 1] : 1;
    a.isy = (sub >> 1) == (p.t >> 1) && !(sub & 1);
  };
  if (p.v1 >= 0) axis(p.v1, p.nv1);
  if (p.v2 >= 0) axis(p.v2, p.nv2);
  for (int b = 0; b < p.nbatch; ++b) axis(p.bsub[b], p.blen[b]);
  g.total = (uint32_t)total;
  return g;
}
inline reg_lines reg_lines_of(const dmg_fft_pass &p, const dmg_fft_batch &bt) {
  reg_lines g;
  memset(&g, 0, sizeof(g));
  static_cast<line_axes &>(g) = line_axes_of(p, bt);
  if (p.rows) g.rows = *p.rows;
  return g;
}

inline uint32_t sm_count() {
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return (uint32_t)nsm;
}

template <typename T, int SIGN, bool TF>
int launch_reg_form(const dmg_fft_pass &p, const dmg_fft_batch &bt, cudaStream_t s) {
  const reg_lines g = reg_lines_of(p, bt);
  switch (p.n) {
    case 32: return launch_reg_k<T, SIGN, 32, TF>(p, bt, g, s);
    case 48: return launch_reg_k<T, SIGN, 48, TF>(p, bt, g, s);
    case 64: return launch_reg_k<T, SIGN, 64, TF>(p, bt, g, s);
    case 96: return launch_reg_k<T, SIGN, 96, TF>(p, bt, g, s);
    case 120: return launch_reg_k<T, SIGN, 120, TF>(p, bt, g, s);
    case 128: return launch_reg_k<T, SIGN, 128, TF>(p, bt, g, s);
    case 160: return launch_reg_k<T, SIGN, 160, TF>(p, bt, g, s);
    case 192: return launch_reg_k<T, SIGN, 192, TF>(p, bt, g, s);
    case 240: return launch_reg_k<T, SIGN, 240, TF>(p, bt, g, s);
    case 256: return launch_reg_k<T, SIGN, 256, TF>(p, bt, g, s);
    case 320: return launch_reg_k<T, SIGN, 320, TF>(p, bt, g, s);
    case 384: return launch_reg_k<T, SIGN, 384, TF>(p, bt, g, s);
    case 480: return launch_reg_k<T, SIGN, 480, TF>(p, bt, g, s);
    case 512: return launch_reg_k<T, SIGN, 512, TF>(p, bt, g, s);
    case 1024:
      // Few lines in 16-byte values: one to a block, so that each has an SM (or half of one) to itself instead of
      // sharing it with three (64 lines, native FP64, 38 -> 27 us, 25 in the tiled kernel; double-float 22 -> 20).
      if constexpr (sizeof(C2<T>) == 16)
        if (g.total <= 2 * sm_count()) return launch_reg_k<T, SIGN, 1024, TF, 1>(p, bt, g, s);
      return launch_reg_k<T, SIGN, 1024, TF>(p, bt, g, s);
    case 2048:
      if constexpr (std::is_same<T, float>::value) return launch_reg_k<T, SIGN, 2048, TF>(p, bt, g, s);
    default: return dmg_error(DMG_ERR_ARG, "fft pass: no register schedule for length %d", p.n);
  }
}

}  // namespace
