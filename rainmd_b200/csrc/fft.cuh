// Register-resident DFTs of small lengths, and the two-factor line transform built from them.
//
// A line of N = R1 * R2 points is an R1 x R2 matrix, x[r * R2 + j] at (r, j). The forward
// transform is R1-point DFTs down the columns, a multiplication by W_N^(j k1), and R2-point DFTs
// along the rows, which leaves X[k1 + R1 * k2] at (k1, k2); the inverse runs the same steps
// backwards and returns to natural order (J. W. Cooley and J. W. Tukey, Math. Comp. 19, 297
// (1965), for one split). Each DFT is one thread's work in registers and reads and writes the
// same elements, so a transform is in place with one barrier, and its first and last steps can
// take their points from (and put them into) global memory or another block's shared memory
// without a copy of their own.
//
// The lengths a thread transforms are 1-6, 8, 9, 10, 12, 15, 16, 18, 20 and 25: with them every
// 5-smooth N up to 160, and most up to 400, is a product of two near-equal factors.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>
#include <utility>

namespace rmd {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// multiply by -i (forward) or +i (inverse)
__device__ __forceinline__ float2 rot(float2 a, bool inverse) {
  return inverse ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <int R>
__device__ __forceinline__ void dft_small(float2 *v, bool inv) {
  if (R == 2) {
    float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if (R == 4) {
    float2 a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
    float2 a2 = cadd(v[1], v[3]), a3 = rot(csub(v[1], v[3]), inv);
    v[0] = cadd(a0, a2);
    v[2] = csub(a0, a2);
    v[1] = cadd(a1, a3);
    v[3] = csub(a1, a3);
  } else if (R == 3) {
    const float h = 0.86602540378443864676f;  // sqrt(3)/2
    float2 t1 = cadd(v[1], v[2]), t2 = csub(v[1], v[2]);
    float2 b = make_float2(v[0].x - 0.5f * t1.x, v[0].y - 0.5f * t1.y);
    float2 r = rot(make_float2(h * t2.x, h * t2.y), inv);  // -i*h*t2 forward
    v[0] = cadd(v[0], t1);
    v[1] = cadd(b, r);
    v[2] = csub(b, r);
  } else if (R == 5) {
    const float c1 = 0.30901699437494742410f, c2 = -0.80901699437494742410f;
    const float s1 = 0.95105651629515357212f, s2 = 0.58778525229247312917f;
    float2 t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]);
    float2 t3 = csub(v[1], v[4]), t4 = csub(v[2], v[3]);
    float2 b1 = make_float2(v[0].x + c1 * t1.x + c2 * t2.x, v[0].y + c1 * t1.y + c2 * t2.y);
    float2 b2 = make_float2(v[0].x + c2 * t1.x + c1 * t2.x, v[0].y + c2 * t1.y + c1 * t2.y);
    float2 q1 = rot(make_float2(s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y), inv);
    float2 q2 = rot(make_float2(s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y), inv);
    v[0] = cadd(v[0], cadd(t1, t2));
    v[1] = cadd(b1, q1);
    v[4] = csub(b1, q1);
    v[2] = cadd(b2, q2);
    v[3] = csub(b2, q2);
  }
}

// cos and sin of 2 pi k / n at compile time: the Taylor series, on an angle reduced to [-pi, pi].
constexpr double root_angle(int k, int n) {
  return 6.283185307179586476925286766559 * (2 * (k % n) > n ? (k % n) - n : (k % n)) / n;
}
constexpr double root_cos(int k, int n) {
  const double x = root_angle(k, n);
  double term = 1.0, sum = 1.0;
  for (int m = 1; m <= 16; ++m) {
    term *= -x * x / ((2 * m - 1) * (2 * m));
    sum += term;
  }
  return sum;
}
constexpr double root_sin(int k, int n) {
  const double x = root_angle(k, n);
  double term = x, sum = x;
  for (int m = 1; m <= 16; ++m) {
    term *= -x * x / ((2 * m) * (2 * m + 1));
    sum += term;
  }
  return sum;
}

template <class F, int... I>
__device__ __forceinline__ void static_for_each(F &&f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F &&f) {
  static_for_each(f, std::make_integer_sequence<int, N>{});
}

constexpr int dft_split(int r) {  // the first factor of a composite length (1: transformed directly)
  return r <= 5 ? 1 : r == 6 || r == 10 ? 2 : r == 9 || r == 12 || r == 15 || r == 18 ? 3 : r == 25 ? 5 : r == 8 ? 2 : 4;
}

template <int R, bool INV>
__device__ __forceinline__ void dft(float2 (&v)[R]) {
  constexpr int A = dft_split(R), B = R / A;
  if constexpr (R <= 5) {
    dft_small<R>(v, INV);
  } else {
    float2 w[A][B];
    static_for<B>([&](auto nb) {
      constexpr int b = decltype(nb)::value;
      float2 t[A];
#pragma unroll
      for (int a = 0; a < A; ++a) t[a] = v[B * a + b];
      dft<A, INV>(t);
      static_for<A>([&](auto na) {
        constexpr int a = decltype(na)::value;
        if constexpr (a * b == 0) {
          w[a][b] = t[a];
        } else {
          constexpr float c = (float)root_cos(a * b, R), s = (float)root_sin(a * b, R);
          w[a][b] = cmul(t[a], make_float2(c, INV ? s : -s));
        }
      });
    });
#pragma unroll
    for (int a = 0; a < A; ++a) {
      dft<B, INV>(w[a]);
#pragma unroll
      for (int b = 0; b < B; ++b) v[a + A * b] = w[a][b];
    }
  }
}

// Call f with the length, at most MAXR, as a compile-time constant. A kernel's registers are those
// of its longest DFT, so the passes are built twice: for axes of factors up to RADIX_SMALL (every axis up
// to 144 points but 75, 125, 128 and 135) and for all. The longer form's blocks hold fewer to an SM (r2c 101 and
// 254 registers a thread, planes 96 and 128 with some spilled), which shows beside its neighbours' times:
// the reciprocal kernels of 42,000 atoms, us, against the Stockham passes that both replaced: 72^3 35 (66),
// 75^3 41 (68), 80^3 38 (83); 120^3 72 (167), 125^3 119 (178), 128^3 70 (178), 135^3 90 (264), 144^3 89 (290), 150^3 135 (325),
// 160^3 184 (261: its planes take the separate passes).
constexpr int RADIX_SMALL = 12, RADIX_ALL = 25;
template <int MAXR, class F>
__device__ __forceinline__ void with_radix(int r, F &&f) {
  switch (r) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    case 9: f(std::integral_constant<int, 9>{}); break;
    case 10: f(std::integral_constant<int, 10>{}); break;
    case 12: f(std::integral_constant<int, 12>{}); break;
    default:
      if constexpr (MAXR > RADIX_SMALL) {
        switch (r) {
          case 15: f(std::integral_constant<int, 15>{}); break;
          case 16: f(std::integral_constant<int, 16>{}); break;
          case 18: f(std::integral_constant<int, 18>{}); break;
          case 20: f(std::integral_constant<int, 20>{}); break;
          case 25: f(std::integral_constant<int, 25>{}); break;
        }
      }
  }
}

// The two factors of n (r1 <= r2, as near to each other as the lengths above allow), or false.
inline bool fft_two_factors(int n, int *r1, int *r2) {
  const int lengths[] = {1, 2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 18, 20, 25};
  int best = 0;
  for (int a : lengths)
    for (int b : lengths)
      if (a <= b && a * b == n && a > best) best = a, *r1 = a, *r2 = b;
  return best > 0;
}

}  // namespace rmd
