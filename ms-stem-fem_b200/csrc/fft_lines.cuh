// Two FP32 lines, or one FP64 line, per thread: the Stockham FFT of the column
// passes and of the FP64 row pass.
//
// A thread holds E elements.  In FP32 an element is a Pair, the same element of
// two lines with both real parts in one register pair and both imaginary parts
// in another, so that every operation is one packed instruction (FADD2 / FMUL2 /
// FFMA2) and twiddles and propagators are loaded once for the two lines.
//
// A radix-R stage after NS-point sub-transforms computes
//   X[k + NS m] = sum_r v[r] W_(NS R)^(r (k + NS m))
// in one of two forms:
//
//  * product: v[r] W_(NS R)^(r k), R - 1 table entries, then an untwiddled
//    butterfly (32 points as 4 x 8, 16 as 4 x 4).  Every first stage is this one,
//    without the product.
//  * fused: log2 R decimation-in-time layers; the layer of block size B pairs m
//    and m + B/2 with the twiddle W_(NS B)^(k + NS m), so the stage's own
//    twiddles cost nothing beyond the butterflies'.  A butterfly is
//    r = a + w b (four FMAs), q = 2 a - r (two); m >= B/4 needs no twiddle of
//    its own, it is -i times that of m - B/4.  Half the entries of the other
//    form, but every layer multiplies, and q inherits the rounding of r.
//
// Which form a length takes is a matter of rounding first.  Exit waves' rms error
// outside the aperture against FP64 (FP32) and long double (FP64); first with the
// schedules of fft_core.cuh, products throughout, then with every stage fused and
// q = 2 a - r, then as it is here:
//   FP32, 1e-7:  64^2 4.33 4.93 4.32   128^2 6.42 7.29 6.41   256^2 6.86 7.41 6.87
//                512^2 7.57 7.73 7.55  1024^2 9.12 8.75 8.28  2048^2 5.24 5.62 5.24
//                4096 x 64 7.48 7.45 6.80
//   FP64, 1e-12: 64^2 0.43 0.47 0.41   128^2 1.69 1.74 1.31   256^2 1.90 2.84 1.85
//                512^2 8.06 8.17 5.97  1024^2 18.1 17.8 12.7  2048 x 64 6.44 7.02 4.90
// (part of the FP64 gain is the tables', see exact_root).  Stages are fused
// where that error is no larger and it is the faster form: FP64 rows of 512 points
// 1.69 us a probe against 3.57, 1024 6.4 against 12.1, 2048 39.8 against 47.4, 4096
// 181 against 231 (at 32 elements a thread the product form's table reads are
// exposed); FP32 columns of 4096 points 70.9 against 73.2, 1024 2.77 against 2.78.  At
// 2048 points fused later stages round 0.5 % worse (5.26), at 512 better (7.27) but
// take 0.735 us against 0.72.  Elsewhere the product form costs 1 to 4 % of a column
// pass (FP32 2048^2 13.3 -> 13.7 us a probe, 512^2 0.71 -> 0.72, 128^2 0.074 -> 0.076)
// and more of the FP64 rows of 128 and 256 points (0.098 -> 0.106, 0.338 -> 0.403 us).
#pragma once
#include <cmath>
#include <utility>
#include <vector>

#include "fft_core.cuh"

namespace msf {

struct Pair {
  float2 re, im;  // .x the first line, .y the second
};

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 f2neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 f2add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 f2sub(float2 a, float2 b) { return __fadd2_rn(a, f2neg(b)); }
__device__ __forceinline__ float2 f2mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 f2fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// Columns (rows) the band limit always removes: it keeps |k| < N/3 of the
// N-point line, so of the E slots (slot m holds elements T m .. T m + T - 1)
// those from ceil(E / 3) to E - ceil(E / 3) - 1 hold removed elements only.
template <int E> __host__ __device__ constexpr int dead_lo() { return (E + 2) / 3; }
template <int E> __host__ __device__ constexpr int dead_hi() { return E - (E + 2) / 3; }
template <int E> __host__ __device__ constexpr bool dead_slot(int m) {
  return m >= dead_lo<E>() && m < dead_hi<E>();
}

// An N-point schedule: E elements of each line per thread, T threads, radices
// R0 R1 [R2].
template <int N_, int E_, int R0_, int R1_, int R2_ = 1> struct LineShape {
  static constexpr int N = N_, E = E_, S = R2_ > 1 ? 3 : 2, T = N_ / E_;
  static_assert(R0_ * R1_ * R2_ == N_);
  __host__ __device__ static constexpr int radix(int s) {
    return s == 0 ? R0_ : s == 1 ? R1_ : R2_;
  }
  __host__ __device__ static constexpr int ns(int s) {
    return s == 0 ? 1 : s == 1 ? R0_ : R0_ * R1_;
  }
  // entries of one butterfly's twiddles: fused, one for B = 2 and 4 and B/4 after
  __host__ __device__ static constexpr int tw_rows(int r, bool fused) {
    return !fused ? r - 1 : r <= 2 ? r / 2 : r == 4 ? 2 : tw_rows(r / 2, true) + r / 4;
  }
  // stage s >= 1's table [row][k], k < ns(s), after the earlier stages'
  __host__ __device__ static constexpr int tw_off(int s, bool fused) {
    return s <= 1 ? 0 : tw_off(s - 1, fused) + tw_rows(radix(s - 1), fused) * ns(s - 1);
  }
};
// columns: the fewest stages
template <int N> struct ColShapeOf;
template <> struct ColShapeOf<64> { using type = LineShape<64, 8, 8, 8>; };
template <> struct ColShapeOf<128> { using type = LineShape<128, 16, 16, 8>; };
template <> struct ColShapeOf<256> { using type = LineShape<256, 16, 16, 16>; };
template <> struct ColShapeOf<512> { using type = LineShape<512, 32, 32, 16>; };
template <> struct ColShapeOf<1024> { using type = LineShape<1024, 32, 32, 32>; };
template <> struct ColShapeOf<2048> { using type = LineShape<2048, 32, 32, 8, 8>; };
template <> struct ColShapeOf<4096> { using type = LineShape<4096, 32, 32, 32, 4>; };
template <int N> using ColShape = typename ColShapeOf<N>::type;
// FP64 rows: the same up to 1024 points; beyond, where 32 elements a thread
// spill, 16 (2048: 40 us a probe against 59)
template <int N> struct RowShapeOf { using type = ColShape<N>; };
template <> struct RowShapeOf<2048> { using type = LineShape<2048, 16, 16, 16, 8>; };
template <> struct RowShapeOf<4096> { using type = LineShape<4096, 16, 16, 16, 16>; };
template <int N> using RowShape = typename RowShapeOf<N>::type;

// Whether a length's twiddled stages are fused (see the head of the file).
template <typename Real, int N> __host__ __device__ constexpr bool fused_twiddles() {
  return sizeof(Real) == 4 ? N == 1024 || N == 4096 : N >= 512;
}

// (cos, sin) of 2 pi num / den, den a power of two up to 4096, rounded from long
// double: an FP64 angle near 2 pi carries a rounding several times the entry's own.
// One octant is evaluated, once in a process (513 pairs of 0.44 us); the rest is
// its mirror images.
inline std::pair<double, double> exact_root(int num, int den) {
  constexpr int N = 4096, O = N / 8;
  static const std::vector<std::pair<double, double>> octant = [] {
    std::vector<std::pair<double, double>> t;
    for (int k = 0; k <= O; ++k) {
      const long double x = 6.283185307179586476925286766559005768L * k / N;
      t.emplace_back((double)std::cos(x), (double)std::sin(x));
    }
    return t;
  }();
  const int k = num * (N / den) % N, o = k / O;
  const auto& e = octant[o % 2 ? O - k % O : k % O];
  const bool swap = (o + 1) / 2 % 2;  // octants 1, 2, 5, 6
  const double c = swap ? e.second : e.first, s = swap ? e.first : e.second;
  return {o >= 2 && o < 6 ? -c : c, o >= 4 ? -s : s};
}

// A shape's twiddles, stage by stage in the order they are read, (cos, -sin) pairs.
template <class Sh, typename Real> void line_twiddles(std::vector<Real>& out) {
  auto put = [&](int num, int den) {
    const auto [c, s] = exact_root(num, den);
    out.push_back((Real)c);
    out.push_back((Real)-s);
  };
  for (int s = 1; s < Sh::S; ++s) {
    const int R = Sh::radix(s), NS = Sh::ns(s);
    if (fused_twiddles<Real, Sh::N>()) {
      for (int B = 2; B <= R; B *= 2)
        for (int m = 0; m < (B > 4 ? B / 4 : 1); ++m)
          for (int k = 0; k < NS; ++k) put(k + NS * m, NS * B);
    } else {
      for (int r = 1; r < R; ++r)
        for (int k = 0; k < NS; ++k) put(r * k, NS * R);
    }
  }
}

// Table entries from global or shared memory.
template <typename C> struct GlobalTable {
  using type = C;
  const C* p;
  __device__ __forceinline__ C operator()(int k) const { return __ldg(p + k); }
};
template <typename C> struct SharedTable {
  using type = C;
  const C* p;
  __device__ __forceinline__ C operator()(int k) const { return p[k]; }
};

// What a thread holds per element: a Pair (two FP32 lines) or a double2 (one
// FP64 line), 16 bytes either way, so both share the kernels' layouts.
template <class V> struct LineOf;
template <> struct LineOf<Pair> {
  using Real = float;
  using C = float2;     // a table entry
  using Half = float2;  // both lines' real or imaginary parts
  using Mem = float4;
};
template <> struct LineOf<double2> {
  using Real = double;
  using C = double2;
  using Half = double;
  using Mem = double2;
};
__device__ __forceinline__ void put(float4* p, const Pair& v) {
  *p = make_float4(v.re.x, v.re.y, v.im.x, v.im.y);
}
__device__ __forceinline__ void get(const float4* p, Pair& v) {
  const float4 x = *p;
  v = Pair{make_float2(x.x, x.y), make_float2(x.z, x.w)};
}
__device__ __forceinline__ void put(double2* p, const double2& v) { *p = v; }
__device__ __forceinline__ void get(const double2* p, double2& v) { v = *p; }
// two adjacent complex values in memory (re, im, re, im), or one FP64 one
__device__ __forceinline__ void put_cols(float4* p, const Pair& v) {
  *p = make_float4(v.re.x, v.im.x, v.re.y, v.im.y);
}
__device__ __forceinline__ void get_cols(const float4* p, Pair& v) {
  const float4 x = *p;
  v = Pair{make_float2(x.x, x.z), make_float2(x.y, x.w)};
}
__device__ __forceinline__ void put_cols(double2* p, const double2& v) { *p = v; }
__device__ __forceinline__ void get_cols(const double2* p, double2& v) { v = *p; }
__device__ __forceinline__ float2& re_of(Pair& v) { return v.re; }
__device__ __forceinline__ float2& im_of(Pair& v) { return v.im; }
__device__ __forceinline__ double& re_of(double2& v) { return v.x; }
__device__ __forceinline__ double& im_of(double2& v) { return v.y; }
__device__ __forceinline__ Pair vneg(const Pair& b) { return Pair{f2neg(b.re), f2neg(b.im)}; }
__device__ __forceinline__ double2 vneg(const double2& b) { return make_double2(-b.x, -b.y); }
template <class V> __device__ __forceinline__ V vzero();
template <> __device__ __forceinline__ Pair vzero<Pair>() { return Pair{f2(0.f), f2(0.f)}; }
template <> __device__ __forceinline__ double2 vzero<double2>() { return make_double2(0.0, 0.0); }

// a, b <- a + w b, a - w b, with w = c + i s (its conjugate when INV);
// NEED: bit 0 the sum is used, bit 1 the difference
template <bool INV, int NEED = 3>
__device__ __forceinline__ void bfly(Pair& a, Pair& b, float c, float s) {
  const float2 C = f2(c), S = f2(INV ? -s : s);
  if constexpr (NEED & 1) {
    Pair r;
    r.re = f2fma(f2neg(S), b.im, f2fma(C, b.re, a.re));
    r.im = f2fma(S, b.re, f2fma(C, b.im, a.im));
    if constexpr (NEED & 2) {
      b.re = f2fma(f2(2.f), a.re, f2neg(r.re));
      b.im = f2fma(f2(2.f), a.im, f2neg(r.im));
    }
    a = r;
  } else if constexpr (NEED & 2) {
    Pair q;
    q.re = f2fma(S, b.im, f2fma(f2neg(C), b.re, a.re));
    q.im = f2fma(f2neg(S), b.re, f2fma(f2neg(C), b.im, a.im));
    b = q;
  }
}
template <bool INV, int NEED = 3>
__device__ __forceinline__ void bfly(double2& a, double2& b, double c, double s0) {
  const double s = INV ? -s0 : s0;
  if constexpr (NEED & 1) {
    const double2 r = make_double2(fma(-s, b.y, fma(c, b.x, a.x)), fma(s, b.x, fma(c, b.y, a.y)));
    if constexpr (NEED & 2) b = make_double2(fma(2.0, a.x, -r.x), fma(2.0, a.y, -r.y));
    a = r;
  } else if constexpr (NEED & 2) {
    b = make_double2(fma(s, b.y, fma(-c, b.x, a.x)), fma(-s, b.x, fma(-c, b.y, a.y)));
  }
}
// Layers B, 2B, .. R of a fused stage over u[0..R) (bit-reversed in, natural
// out).  k: this butterfly's first entry of the table tw, rows NS apart.  ZOUT: E
// slots' dead range is not needed on exit (last layer).
template <int R, int B, int NS, bool INV, bool ZOUT, int NB, int BI, class V, class Tw>
__device__ __forceinline__ void fused_layers(V (&u)[R], const Tw& tw, int k) {
  if constexpr (B <= R) {
    constexpr int H = B / 2;
    constexpr int ROWS = H >= 2 ? H / 2 : 1;  // twiddles of this layer
    constexpr int ROW0 = B == 2 ? 0 : B == 4 ? 1 : B / 4;
    typename Tw::type w[ROWS];
#pragma unroll
    for (int m = 0; m < ROWS; ++m) w[m] = tw(k + (ROW0 + m) * NS);
    sfor<0, R, B>([&](auto baseI) {
      sfor<0, H>([&](auto mI) {
        constexpr int base = decltype(baseI)::value, m = decltype(mI)::value;
        V& a = u[base + m];
        V& b = u[base + m + H];
        // outputs of the last layer: element slots BI + NB m
        constexpr int E = R * NB;
        constexpr int need = !(ZOUT && B == R) ? 3
                             : (dead_slot<E>(BI + NB * m) ? 0 : 1) |
                                   (dead_slot<E>(BI + NB * (m + H)) ? 0 : 2);
        if constexpr (m < ROWS) bfly<INV, need>(a, b, w[m].x, w[m].y);
        else bfly<INV, need>(a, b, w[m - ROWS].y, -w[m - ROWS].x);  // -i w
      });
    });
    fused_layers<R, 2 * B, NS, INV, ZOUT, NB, BI>(u, tw, k);
  }
}

__device__ __forceinline__ Pair cadd(const Pair& a, const Pair& b) {
  return Pair{f2add(a.re, b.re), f2add(a.im, b.im)};
}
__device__ __forceinline__ Pair csub(const Pair& a, const Pair& b) {
  return Pair{f2sub(a.re, b.re), f2sub(a.im, b.im)};
}
// a * w (INV: its conjugate), the same w for both lines
template <bool INV> __device__ __forceinline__ Pair twiddle(const Pair& a, float2 w) {
  const float2 C = f2(w.x), S = f2(INV ? -w.y : w.y);
  return Pair{f2fma(C, a.re, f2mul(f2neg(S), a.im)), f2fma(C, a.im, f2mul(S, a.re))};
}
template <bool INV> __device__ __forceinline__ double2 twiddle(const double2& a, double2 w) {
  return INV ? cmulc(a, w) : cmul(a, w);
}
template <int K, int M, bool INV> __device__ __forceinline__ Pair twc(const Pair& a) {
  constexpr int k = (K * (64 / M)) & 63;
  if constexpr (k == 0) return a;
  else if constexpr (k == 16) return INV ? Pair{f2neg(a.im), a.re} : Pair{a.im, f2neg(a.re)};
  else if constexpr (k == 32) return vneg(a);
  else if constexpr (k == 48) return INV ? Pair{a.im, f2neg(a.re)} : Pair{f2neg(a.im), a.re};
  else return twiddle<INV>(a, make_float2((float)cos64(k), (float)-sin64(k)));
}
// x, y <- x + y, x - y; DX, DY: x, y is zero
template <bool DX, bool DY, class V> __device__ __forceinline__ void sum_diff(V& x, V& y) {
  if constexpr (DX && DY) {
  } else if constexpr (DY) {
    y = x;
  } else if constexpr (DX) {
    x = y;
    y = vneg(y);
  } else {
    const V t = cadd(x, y);
    y = csub(x, y);
    x = t;
  }
}
// Radix-2 decimation-in-frequency layers over u[OFF + r STR], r < R (natural order
// in, bit-reversed out).  Z: the dead slots of u are zero.
template <int R, int OFF, int STR, bool INV, bool Z, class V, int E>
__device__ __forceinline__ void line_dif(V (&u)[E]) {
  if constexpr (R > 1) {
    constexpr int H = R / 2;
    sfor<0, H>([&](auto kI) {
      constexpr int k = decltype(kI)::value, x = OFF + k * STR, y = OFF + (k + H) * STR;
      sum_diff<Z && dead_slot<E>(x), Z && dead_slot<E>(y)>(u[x], u[y]);
      u[y] = twc<k, R, INV>(u[y]);
    });
    line_dif<H, OFF, STR, INV, false>(u);
    line_dif<H, OFF + H * STR, STR, INV, false>(u);
  }
}
// DFT of u, natural order in; out(k) names the slot that holds output k.  32
// points as 4 x 8 and 16 as 4 x 4 (fft_core.cuh).
template <int R> __host__ __device__ constexpr int dft_out(int k) {
  if (R < 16) return bitrev(k, ilog2(R));
  const int R2 = R / 4, k1 = k & 3, k2 = k >> 2;
  return R2 * bitrev(k1, 2) + bitrev(k2, ilog2(R2));
}
template <int R, bool INV, bool Z, class V> __device__ __forceinline__ void line_dft(V (&u)[R]) {
  if constexpr (R < 16) {
    line_dif<R, 0, 1, INV, Z>(u);
  } else {
    constexpr int R2 = R / 4;
    sfor<0, R2>([&](auto nI) { line_dif<4, decltype(nI)::value, R2, INV, Z>(u); });
    sfor<1, 4>([&](auto kI) {
      constexpr int k1 = decltype(kI)::value;
      sfor<1, R2>([&](auto nI) {
        constexpr int n2 = decltype(nI)::value, at = R2 * bitrev(k1, 2) + n2;
        u[at] = twc<(n2 * k1) % R, R, INV>(u[at]);
      });
    });
    sfor<0, 4>([&](auto kI) { line_dif<R2, R2 * decltype(kI)::value, 1, INV, false>(u); });
  }
}

// One radix-R butterfly of a stage after NS-point sub-transforms: slots b + r NB
// of v, which hold its inputs and receive its outputs in natural order.
template <class Sh, int S, bool INV, bool ZIN, bool ZOUT, int BI, class V, class Tw>
__device__ __forceinline__ void stage_butterfly(V (&v)[Sh::E], int t, const Tw& tw) {
  constexpr int E = Sh::E, R = Sh::radix(S), NB = E / R, NS = Sh::ns(S);
  constexpr bool FUSED = fused_twiddles<typename LineOf<V>::Real, Sh::N>();
  const int k = (t + Sh::T * BI) & (NS - 1);
  V u[R];
  if constexpr (FUSED && NS > 1) {
    sfor<0, R>([&](auto rI) {
      constexpr int r = decltype(rI)::value;
      u[bitrev(r, ilog2(R))] = v[BI + r * NB];
    });
    fused_layers<R, 2, NS, INV, ZOUT && S + 1 == Sh::S, NB, BI>(u, tw, Sh::tw_off(S, true) + k);
    sfor<0, R>([&](auto rI) {
      constexpr int r = decltype(rI)::value;
      v[BI + r * NB] = u[r];
    });
  } else {
    u[0] = v[BI];
    sfor<1, R>([&](auto rI) {
      constexpr int r = decltype(rI)::value;
      if constexpr (NS > 1) {
        u[r] = twiddle<INV>(v[BI + r * NB], tw(Sh::tw_off(S, false) + (r - 1) * NS + k));
      } else {
        u[r] = v[BI + r * NB];
      }
    });
    line_dft<R, INV, ZIN && S == 0 && R == E>(u);
    sfor<0, R>([&](auto rI) {
      constexpr int r = decltype(rI)::value;
      v[BI + r * NB] = u[dft_out<R>(r)];
    });
  }
}

// Exchange slot of element a of a line: the low three bits are XORed
// with those of the stage-0 thread that writes it, so that the eight lanes of
// a 16-byte access phase hit eight different slots both in the stride-R0
// writes of the first exchange and in the unit-stride accesses of all others
// (whose lanes share a / R0 mod 8), with no padding: the buffer is exactly
// the line, and a column tile can be exchanged in place.
template <class Sh> __device__ __forceinline__ int line_slot(int a) {
  return a ^ ((a >> ilog2(Sh::radix(0))) & 7);
}

struct NoHook {
  __device__ __forceinline__ void operator()() const {}
};

// Transforms the thread's elements in place; v[m] holds element t + T m on
// entry and on exit.  at(a): where exchanged element a of this line lies in
// shared memory; tw: the shape's table; sync: a barrier over the T threads of
// the line, which must have passed one since they last read the buffer; hook:
// run once the buffer has been read for the last time.
template <class Sh, bool INV, bool ZIN, bool ZOUT, class V, class Tw, class At, class Sync,
          class Hook = NoHook>
__device__ __forceinline__ void fft_lines(V (&v)[Sh::E], int t, const Tw& tw, At&& at,
                                         Sync&& sync, Hook&& hook = Hook{}) {
  constexpr int N = Sh::N, E = Sh::E, T = Sh::T;
  sfor<0, Sh::S>([&](auto sI) {
    constexpr int s = decltype(sI)::value;
    constexpr int R = Sh::radix(s), NB = E / R, NS = Sh::ns(s);
    if constexpr (s > 0) {
      sfor<0, NB>([&](auto bI) {
        constexpr int b = decltype(bI)::value;
        const int j = t + T * b;
        sfor<0, R>([&](auto rI) {
          constexpr int r = decltype(rI)::value;
          get(at(j + r * (N / R)), v[b + r * NB]);
        });
      });
      if constexpr (s + 1 == Sh::S) hook();
      else sync();
    }
    sfor<0, NB>([&](auto bI) {
      stage_butterfly<Sh, s, INV, ZIN, ZOUT, decltype(bI)::value>(v, t, tw);
    });
    if constexpr (s + 1 < Sh::S) {
      sfor<0, NB>([&](auto bI) {
        constexpr int b = decltype(bI)::value;
        const int j = t + T * b;
        const int base = (j / NS) * NS * R + (j & (NS - 1));
        sfor<0, R>([&](auto rI) {
          constexpr int r = decltype(rI)::value;
          put(at(base + r * NS), v[b + r * NB]);
        });
      });
      sync();
    }
  });
}

// The same transform with the exchanges in two halves (real parts, then
// imaginary parts) through a buffer of 8 bytes an element: half the shared
// memory for two more barriers.  x(a): where exchanged element a of this line
// lies; start: the barrier that ends the buffer's previous use (a no-op when
// the caller has passed one); after: run once, after the first barrier.
template <class Sh, bool INV, bool ZIN, bool ZOUT, class V, class Tw, class X, class Sync,
          class Start, class After>
__device__ __forceinline__ void fft_lines_split(V (&v)[Sh::E], int t, const Tw& tw, X&& x,
                                               Sync&& sync, Start&& start, After&& after) {
  constexpr int N = Sh::N, E = Sh::E, T = Sh::T;
  sfor<0, Sh::S>([&](auto sI) {
    constexpr int s = decltype(sI)::value;
    constexpr int R = Sh::radix(s), NB = E / R, NS = Sh::ns(s);
    sfor<0, NB>([&](auto bI) {
      stage_butterfly<Sh, s, INV, ZIN, ZOUT, decltype(bI)::value>(v, t, tw);
    });
    if constexpr (s + 1 < Sh::S) {
      constexpr int R2 = Sh::radix(s + 1), NB2 = E / R2;
      sfor<0, 2>([&](auto hI) {
        constexpr int h = decltype(hI)::value;
        if constexpr (s == 0 && h == 0) start();
        else sync();
        sfor<0, NB>([&](auto bI) {
          constexpr int b = decltype(bI)::value;
          const int j = t + T * b;
          const int base = (j / NS) * NS * R + (j & (NS - 1));
          sfor<0, R>([&](auto rI) {
            constexpr int r = decltype(rI)::value;
            *x(base + r * NS) = h == 0 ? re_of(v[b + r * NB]) : im_of(v[b + r * NB]);
          });
        });
        sync();
        if constexpr (s == 0 && h == 0) after();
        typename LineOf<V>::Half w[E];
        sfor<0, NB2>([&](auto bI) {
          constexpr int b = decltype(bI)::value;
          sfor<0, R2>([&](auto rI) {
            constexpr int r = decltype(rI)::value;
            w[b + r * NB2] = *x(t + T * b + r * (N / R2));
          });
        });
        sfor<0, E>([&](auto mI) {
          constexpr int m = decltype(mI)::value;
          if constexpr (h == 0) re_of(v[m]) = w[m];
          else im_of(v[m]) = w[m];
        });
      });
    }
  });
}

}  // namespace msf
