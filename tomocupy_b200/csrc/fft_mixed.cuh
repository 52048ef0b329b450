// Inverse FFT of contiguous lines whose length is a product of small primes, one
// line per CTA: self-sorting (Stockham) stages of radix 2 .. 18, twiddles from
// per-stage tables.  A stage's values go through registers (up to 18 per
// thread), so one shared-memory line buffer serves all stages.  Odd radices are summed directly
// (cosine terms of x_k + x_(r-k), sine terms of x_k - x_(r-k)): (r - 1)^2 / 2
// complex-by-real products each.
//
// Made for detector widths that are no powers of two (2n = 4896 = 17 18 16 for
// 2448 columns).  Bound: instruction issue (shared-memory addressing, twiddles,
// the odd radices' sums); lines are read and written in HBM once.  Few stages of
// large radix and three to four CTAs per SM matter most: 17 9 8 4 through two
// line buffers took twice as long.
#pragma once
#include <algorithm>
#include <cmath>
#include <vector>

namespace tcb {
namespace mixfft {

constexpr int MAX_STAGES = 4;
constexpr int MAX_T = 320, MIN_CTAS = 3;
constexpr int MAX_N = 18 * MAX_T;

// cos and sin of 2 pi m / r by their power series (m reduced to |angle| <= pi).
constexpr double series(double x, bool sine) {
  double term = sine ? x : 1.0, sum = term;
  for (int k = sine ? 1 : 0; k < 40; k += 2) {
    term *= -x * x / ((k + 1) * (k + 2));
    sum += term;
  }
  return sum;
}
constexpr double unit_angle(int m, int r) {
  int k = m % r;
  if (2 * k > r) k -= r;
  return 6.283185307179586476925286766559 * k / r;
}
template <int R> struct Roots {
  float c[R], s[R];
  constexpr Roots() : c(), s() {
    for (int m = 0; m < R; m++) {
      c[m] = (float)series(unit_angle(m, R), false);
      s[m] = (float)series(unit_angle(m, R), true);
    }
  }
};

struct Stage {
  int r, l;        // radix, product of the radices before it
  unsigned magic;  // ceil(2^32 / l): b / l = umulhi(b, magic) for b, l < 2^16
  int tw;          // first entry of its twiddles w^(p 2^j): [j][p], 2^j < r, p = 0 .. l - 1
};
struct Plan {
  int n = 0, nst = 0, threads = 0;
  Stage st[MAX_STAGES];
};

__host__ __device__ inline int pad(int i) { return i + (i >> 4); }
inline size_t smem_bytes(int n) { return (size_t)(pad(n - 1) + 1) * sizeof(float2); }
// butterflies of radix r that a thread holds at a time
__host__ __device__ constexpr int per_thread(int r) { return r > 9 ? 1 : 18 / r; }

// The stages of length n, or n = 0 when a prime above 17 divides it.
inline Plan make_plan(int n, std::vector<float2> &tw) {
  Plan p;
  std::vector<int> rs;
  int m = n;
  for (int r : {17, 13, 11}) while (m % r == 0) rs.push_back(r), m /= r;
  for (int r : {15, 9, 7, 5, 3}) while (m % r == 0) rs.push_back(r), m /= r;
  int two = 0;
  while (m % 2 == 0) two++, m /= 2;
  if (m != 1 || n < 2 || n > MAX_N) return p;
  if (two % 4 == 1)  // an odd two joins an odd radix
    for (int &r : rs)
      if (r <= 9) {
        r *= 2;
        two--;
        break;
      }
  std::stable_sort(rs.begin(), rs.end(), [](int x, int y) { return x % 2 > y % 2; });
  while (two > 0) {
    const int k = two >= 4 && two != 5 ? 4 : two >= 3 ? 3 : two;  // 16s, ends as 8 x 4, 8, 4 or 2
    rs.push_back(1 << k);
    two -= k;
  }
  if (rs.size() > MAX_STAGES) return p;
  int l = 1;
  tw.clear();
  for (size_t k = 0; k < rs.size(); k++) {
    const int r = rs[k];
    p.st[k] = {r, l, l > 1 ? (unsigned)((0x100000000ull + l - 1) / l) : 0u, (int)tw.size()};
    for (int q = 1; q < r; q *= 2)
      for (int j = 0; j < l; j++) {
        const double a = 6.283185307179586476925286766559 * ((double)q * j / ((double)r * l));
        tw.push_back(make_float2((float)std::cos(a), (float)std::sin(a)));
      }
    l *= r;
  }
  p.n = n;
  p.nst = (int)rs.size();
  for (int r : rs) {
    const int per = r * per_thread(r);
    p.threads = std::max(p.threads, ((n + per - 1) / per + 31) / 32 * 32);
  }
  if (p.threads > MAX_T) p.n = 0;
  return p;
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 muli(float2 a) { return make_float2(-a.y, a.x); }

// out(j, X_j) of the inverse DFT of v, odd R.
template <int R, typename Out>
__device__ __forceinline__ void dft_odd(const float2 (&v)[R], Out out) {
  constexpr Roots<R> w;
  constexpr int H = (R - 1) / 2;
  float2 t[H], d[H], s = v[0];
#pragma unroll
  for (int k = 0; k < H; k++) {
    t[k] = cadd(v[k + 1], v[R - 1 - k]);
    d[k] = csub(v[k + 1], v[R - 1 - k]);
    s = cadd(s, t[k]);
  }
  out(0, s);
#pragma unroll
  for (int j = 1; j <= H; j++) {
    float2 a = v[0], b = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 1; k <= H; k++) {
      const float c = w.c[j * k % R], e = w.s[j * k % R];
      a.x = fmaf(c, t[k - 1].x, a.x);
      a.y = fmaf(c, t[k - 1].y, a.y);
      b.x = fmaf(e, d[k - 1].x, b.x);
      b.y = fmaf(e, d[k - 1].y, b.y);
    }
    out(j, make_float2(a.x - b.y, a.y + b.x));
    out(R - j, make_float2(a.x + b.y, a.y - b.x));
  }
}

__device__ __forceinline__ void dft4(float2 &a, float2 &b, float2 &c, float2 &d) {
  const float2 s = cadd(a, c), t = csub(a, c), u = cadd(b, d), w = muli(csub(b, d));
  a = cadd(s, u);
  b = cadd(t, w);
  c = csub(s, u);
  d = csub(t, w);
}

template <int R, typename Out>
__device__ __forceinline__ void dft(float2 (&v)[R], Out out) {
  if constexpr (R % 2 == 1) {
    dft_odd<R>(v, out);
  } else if constexpr (R == 2) {
    out(0, cadd(v[0], v[1]));
    out(1, csub(v[0], v[1]));
  } else if constexpr (R == 4) {
    dft4(v[0], v[1], v[2], v[3]);
#pragma unroll
    for (int j = 0; j < 4; j++) out(j, v[j]);
  } else if constexpr (R % 4 == 2) {
    // R = 2 H: even outputs from the sums, odd ones from the turned differences
    constexpr int H = R / 2;
    constexpr Roots<R> w;
    float2 u[H];
#pragma unroll
    for (int q = 0; q < H; q++) u[q] = cadd(v[q], v[q + H]);
    dft_odd<H>(u, [&](int j, float2 x) { out(2 * j, x); });
#pragma unroll
    for (int q = 0; q < H; q++) {
      u[q] = csub(v[q], v[q + H]);
      if (q > 0) u[q] = cmul(u[q], make_float2(w.c[q], w.s[q]));
    }
    dft_odd<H>(u, [&](int j, float2 x) { out(2 * j + 1, x); });
  } else {
    // R = 4 S: S transforms of length 4 over v[q], v[q + S], .., twiddles, then S-point ones
    constexpr int S = R / 4;
    constexpr Roots<R> w;
#pragma unroll
    for (int q = 0; q < S; q++) {
      dft4(v[q], v[q + S], v[q + 2 * S], v[q + 3 * S]);
#pragma unroll
      for (int p = 1; p < 4; p++)
        if (q > 0) v[q + p * S] = cmul(v[q + p * S], make_float2(w.c[p * q], w.s[p * q]));
    }
#pragma unroll
    for (int p = 0; p < 4; p++) {  // X[p + 4 j] from v[p S .. p S + S - 1]
      if constexpr (S == 2) {
        out(p, cadd(v[2 * p], v[2 * p + 1]));
        out(p + 4, csub(v[2 * p], v[2 * p + 1]));
      } else {
        dft4(v[4 * p], v[4 * p + 1], v[4 * p + 2], v[4 * p + 3]);
#pragma unroll
        for (int j = 0; j < 4; j++) out(p + 4 * j, v[4 * p + j]);
      }
    }
  }
}

// One stage on the line buffer.
template <int R>
__device__ __forceinline__ void stage(const Stage &st, int n, const float2 *__restrict__ tw,
                                      float2 *sm) {
  constexpr int IT = per_thread(R);
  const int m = n / R;
  float2 v[IT][R];
#pragma unroll
  for (int t = 0; t < IT; t++) {
    const int b = threadIdx.x + t * blockDim.x;
    if (b < m) {
#pragma unroll
      for (int q = 0; q < R; q++) v[t][q] = sm[pad(b + q * m)];
    }
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < IT; t++) {
    const int b = threadIdx.x + t * blockDim.x;
    if (b < m) {
      int o = b * R;
      const int l = st.l;
      if (l > 1) {
        const int hi = (int)__umulhi((unsigned)b, st.magic), p = b - hi * l;
        const float2 *w = tw + st.tw + p;
        // w^(p q) by the bits of q: log2(r) loads, up to 4 roundings
#pragma unroll
        for (int j = 0; (1 << j) < R; j++) {
          const float2 wj = __ldg(w + j * l);
#pragma unroll
          for (int q = 1; q < R; q++)
            if (q >> j & 1) v[t][q] = cmul(v[t][q], wj);
        }
        o = hi * l * R + p;
      }
      dft<R>(v[t], [&](int j, float2 x) { sm[pad(o + j * l)] = x; });
    }
  }
  __syncthreads();
}

__device__ __forceinline__ void any_stage(const Stage &st, int n, const float2 *__restrict__ tw,
                                          float2 *sm) {
  switch (st.r) {
    case 2: stage<2>(st, n, tw, sm); break;
    case 3: stage<3>(st, n, tw, sm); break;
    case 4: stage<4>(st, n, tw, sm); break;
    case 5: stage<5>(st, n, tw, sm); break;
    case 6: stage<6>(st, n, tw, sm); break;
    case 7: stage<7>(st, n, tw, sm); break;
    case 8: stage<8>(st, n, tw, sm); break;
    case 9: stage<9>(st, n, tw, sm); break;
    case 10: stage<10>(st, n, tw, sm); break;
    case 11: stage<11>(st, n, tw, sm); break;
    case 13: stage<13>(st, n, tw, sm); break;
    case 14: stage<14>(st, n, tw, sm); break;
    case 15: stage<15>(st, n, tw, sm); break;
    case 16: stage<16>(st, n, tw, sm); break;
    case 17: stage<17>(st, n, tw, sm); break;
    default: stage<18>(st, n, tw, sm); break;
  }
}

// Lines of p.n values, one per CTA, in place in HBM; of the result only the
// values [k0, k1) are written.  (The stages are written out: in a loop the
// compiler keeps the constants of all radices in registers, and spills.)
__global__ void __launch_bounds__(MAX_T, MIN_CTAS)
    ifft_lines(float2 *__restrict__ x, const float2 *__restrict__ tw, Plan p, int k0, int k1) {
  extern __shared__ float2 mix_sm[];
  float2 *line = x + (size_t)blockIdx.x * p.n;
  for (int i = threadIdx.x; i < p.n; i += blockDim.x)  // all in flight at once
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(mix_sm + pad(i))),
                 "l"(line + i)
                 : "memory");
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  any_stage(p.st[0], p.n, tw, mix_sm);
  if (p.nst > 1) any_stage(p.st[1], p.n, tw, mix_sm);
  if (p.nst > 2) any_stage(p.st[2], p.n, tw, mix_sm);
  if (p.nst > 3) any_stage(p.st[3], p.n, tw, mix_sm);
  for (int i = k0 + threadIdx.x; i < k1; i += blockDim.x) line[i] = mix_sm[pad(i)];
}

}  // namespace mixfft
}  // namespace tcb
