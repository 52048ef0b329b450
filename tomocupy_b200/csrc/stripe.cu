// Fourier-wavelet ring removal (remove_stripe_fw).
//
// Same algorithm as the reference (src/tomocupy/processing/remove_stripe.py:
// _reflect/_mypad 51-84, afb1d 86-128, sfb1d 131-155, DWTForward 157-200,
// DWTInverse 202-246, remove_stripe_fw 253-293): the sinograms, padded along
// the angles to nproj + nproj/8 with zeros, go through `level` 2D DWT levels
// (stride-2 correlation with the reversed analysis filters along the
// detector, then along the angles, half-sample symmetric extension, output
// length floor((N + L - 1)/2)); at every level the band that is high-pass
// along the detector and low-pass along the angles (vertical stripes) is
// Fourier transformed along the angles, multiplied by
// -expm1(-k^2 / (2 sigma^2)) and transformed back; the inverse DWT (stride-2
// transposed convolution with the synthesis filters, cropped by L-2 on both
// sides) rebuilds the sinograms.
//
// Every tap is accumulated in the reference's order with explicit
// round-to-nearest multiplies and adds (no contraction), so the wavelet
// stages reproduce its float32 arithmetic; the band FFTs use cuFFT.
// B200 design: one kernel per filter pass over all slices of the chunk,
// both output channels of a pass from one read of the input window, the
// pyramid kept in HBM.  The damping y = irfft(rfft(x) (1 - g)) along the
// angles equals x - (1/H) sum_k g_k X_k e^{2 pi i k q / H}, and the
// Gaussian g_k = exp(-v_k^2 / (2 sigma^2)) (v_k = k, or k + 1/2 for even H,
// as the reference's ifftshifted grid gives) is below 1e-12 beyond a few
// modes (k <= 7 for sigma = 1): the band is damped in place by projecting
// each column onto those modes (sums of x cos, x sin) and subtracting the
// low-pass, one read and one write of the band, no transposes, no FFTs.
// Levels whose band is too short for the modes, or sigmas that need more
// than 32 (TCB_FW_DAMP=cufft forces it), transpose the band and use cuFFT
// R2C / C2R with 1/N folded into the damping factors.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "common.cuh"

namespace tcb {
namespace sw {

constexpr int MAXL = 64;

struct Taps {
  float h0[MAXL], h1[MAXL];  // analysis: dec_lo, dec_hi reversed
  float g0[MAXL], g1[MAXL];  // synthesis: rec_lo, rec_hi
  int L;
};

__device__ __forceinline__ int reflect(int m, int n) {
  int p = 2 * n;
  m %= p;
  if (m < 0) m += p;
  return m >= n ? p - 1 - m : m;
}

// The filter-bank kernels keep the reference's per-tap operation order
// (round-to-nearest multiply then add, tap by tap), so results are
// bit-identical; the taps live in shared memory and the symmetric reflection
// is only evaluated for outputs whose support crosses an edge.
struct SmemTaps {
  float a[MAXL], b[MAXL];
};

__device__ __forceinline__ void load_taps(SmemTaps &st, const float *a, const float *b, int L) {
  for (int k = threadIdx.x + threadIdx.y * blockDim.x; k < L; k += blockDim.x * blockDim.y) {
    st.a[k] = a[k];
    st.b[k] = b[k];
  }
  __syncthreads();
}

// afb1d along the last axis: x [B][H][W] (row stride sx, slice stride sz) ->
// out [B][2][H][Wo] (lo, hi).
__global__ void afb_rows(const float *__restrict__ x, long long sz, int sx, float *__restrict__ out,
                         int B, int H, int W, int Wo, int padl, const Taps *__restrict__ taps) {
  __shared__ SmemTaps st;
  const int L = taps->L;
  load_taps(st, taps->h0, taps->h1, L);
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)B * H * Wo;
  if (idx >= total) return;
  int j = (int)(idx % Wo);
  long long r = idx / Wo;
  int h = (int)(r % H);
  int b = (int)(r / H);
  const float *row = x + b * sz + (long long)h * sx;
  const int base = 2 * j - padl;
  float v = row[base >= 0 && base < W ? base : reflect(base, W)];
  float lo = __fmul_rn(st.a[0], v), hi = __fmul_rn(st.b[0], v);
  if (base >= 0 && base + L <= W) {
    for (int k = 1; k < L; k++) {
      v = row[base + k];
      lo = __fadd_rn(lo, __fmul_rn(st.a[k], v));
      hi = __fadd_rn(hi, __fmul_rn(st.b[k], v));
    }
  } else {
    for (int k = 1; k < L; k++) {
      v = row[reflect(base + k, W)];
      lo = __fadd_rn(lo, __fmul_rn(st.a[k], v));
      hi = __fadd_rn(hi, __fmul_rn(st.b[k], v));
    }
  }
  long long o = (((long long)b * 2) * H + h) * Wo + j;
  out[o] = lo;
  out[o + (long long)H * Wo] = hi;
}

// afb1d along the rows axis for both channels: in [B][2][H][W] ->
// out [B][4][Ho][W] (channel c -> 2c lo, 2c+1 hi).
__global__ void afb_cols(const float *__restrict__ in, float *__restrict__ out, int B, int H,
                         int W, int Ho, int padl, const Taps *__restrict__ taps) {
  __shared__ SmemTaps st;
  const int L = taps->L;
  load_taps(st, taps->h0, taps->h1, L);
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)B * 2 * Ho * W;
  if (idx >= total) return;
  int j = (int)(idx % W);
  long long r = idx / W;
  int i = (int)(r % Ho);
  long long bc = r / Ho;  // b*2 + c
  const float *col = in + bc * H * W + j;
  const int base = 2 * i - padl;
  float v = col[(long long)(base >= 0 && base < H ? base : reflect(base, H)) * W];
  float lo = __fmul_rn(st.a[0], v), hi = __fmul_rn(st.b[0], v);
  if (base >= 0 && base + L <= H) {
    const float *c0 = col + (long long)base * W;
    for (int k = 1; k < L; k++) {
      v = c0[(long long)k * W];
      lo = __fadd_rn(lo, __fmul_rn(st.a[k], v));
      hi = __fadd_rn(hi, __fmul_rn(st.b[k], v));
    }
  } else {
    for (int k = 1; k < L; k++) {
      v = col[(long long)reflect(base + k, H) * W];
      lo = __fadd_rn(lo, __fmul_rn(st.a[k], v));
      hi = __fadd_rn(hi, __fmul_rn(st.b[k], v));
    }
  }
  long long b = bc / 2, c = bc % 2;
  long long o = ((b * 4 + 2 * c) * Ho + i) * W + j;
  out[o] = lo;
  out[o + (long long)Ho * W] = hi;
}

// sfb1d along the rows axis: channel 0 = synth(lo0, hi0), 1 = synth(lo1, hi1)
// with lo0 = LL (stride sll), hi0 = band0, lo1 = band1, hi1 = band2 of a
// [B][4][Hi][Wb] pyramid level; LL may be cropped (Hi, W used).  Output
// [B][2][Ho][W], Ho = 2 Hi - L + 2.
__global__ void sfb_cols(const float *__restrict__ y, long long bstride, int Hi, int Wb, int W,
                         float *__restrict__ out, int B, int Ho, const Taps *__restrict__ taps) {
  __shared__ SmemTaps st;
  const int L = taps->L;
  load_taps(st, taps->g0, taps->g1, L);
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)B * 2 * Ho * W;
  if (idx >= total) return;
  int j = (int)(idx % W);
  long long r = idx / W;
  int t = (int)(r % Ho);
  long long bc = r / Ho;
  int b = (int)(bc / 2), c = (int)(bc % 2);
  const long long plane = (long long)Hi * Wb;
  const float *base = y + b * bstride;
  const float *lo = base + (c == 0 ? 0 : 2) * plane + j;  // LL or band1 (HL)
  const float *hi = base + (c == 0 ? 1 : 3) * plane + j;  // band0 (LH) or band2 (HH)
  int tt = t + L - 2;  // position in the uncropped output
  float acc = 0.f;
  for (int k = tt & 1; k < L; k += 2) {
    int h = (tt - k) >> 1;
    if (h < 0 || h >= Hi) continue;
    float v = __fadd_rn(__fmul_rn(st.a[k], lo[(long long)h * Wb]),
                        __fmul_rn(st.b[k], hi[(long long)h * Wb]));
    acc = __fadd_rn(acc, v);
  }
  out[(bc * Ho + t) * W + j] = acc;
}

// sfb1d along the last axis: in [B][2][H][Wi] -> out rows (b, h) of width
// Wo = 2 Wi - L + 2, written to dst[b*dsz + h*dsx + w] for h < Hd, w < Wd.
__global__ void sfb_rows(const float *__restrict__ in, int H, int Wi, float *__restrict__ dst,
                         long long dsz, int dsx, int Hd, int Wd, int B,
                         const Taps *__restrict__ taps) {
  __shared__ SmemTaps st;
  const int L = taps->L;
  load_taps(st, taps->g0, taps->g1, L);
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)B * Hd * Wd;
  if (idx >= total) return;
  int w = (int)(idx % Wd);
  long long r = idx / Wd;
  int h = (int)(r % Hd);
  int b = (int)(r / Hd);
  const float *lo = in + (((long long)b * 2) * H + h) * Wi;
  const float *hi = lo + (long long)H * Wi;
  int tt = w + L - 2;
  float acc = 0.f;
  for (int k = tt & 1; k < L; k += 2) {
    int q = (tt - k) >> 1;
    if (q < 0 || q >= Wi) continue;
    float v = __fadd_rn(__fmul_rn(st.a[k], lo[q]), __fmul_rn(st.b[k], hi[q]));
    acc = __fadd_rn(acc, v);
  }
  dst[b * dsz + (long long)h * dsx + w] = acc;
}

// ---- register-blocked filter banks for the supported filter lengths ------
// Same outputs, bit for bit, as the kernels above: every output keeps its
// multiply-then-add tap order, two outputs at a time in the halves of packed
// f32x2 instructions (two rows of the last axis, two columns of the other), so
// a tap costs one packed multiply and one packed add for both.  The multiply is
// a fused multiply-add of -0, which rounds as a multiply does and, unlike a
// packed multiply, cannot be contracted with the add that follows; the zero
// comes with the taps so that the compiler does not know it.
// These instructions (two cycles of the FP32 pipe each) are the bound: 0.13 ms per
// pass over the 7 levels of 16 slices of 1500 x 2048 at 32 taps.  Measured there,
// one output at a time and packed: analysis rows 0.43 and 0.40 ms, columns 0.39
// and 0.34, synthesis columns 0.49 and 0.30, rows 0.39 and 0.35; what is left is
// the staging's latency (rows) and the few warps 127 registers leave (columns of the
// analysis; the synthesis gains from three blocks per SM at 80: 0.36 with two).
// The small levels are latency: 2 slices of 360 x 512 take 0.21 ms, 0.23 one output
// at a time, of the call's 0.26 and 0.28.
struct TapPair {
  float4 c[MAXL];  // (a, a, b, b) of tap k
  float2 nz;       // -0, -0
};

typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pack2(float x, float y) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b, f32x2 nz) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(nz));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// The taps in shared memory, as one 16-byte broadcast per tap: the packed
// instructions take them from registers only, and a pair from the constant bank
// costs several moves.
template <int L>
__device__ __forceinline__ f32x2 stage_taps(ulonglong2 (&st)[L], const TapPair &t) {
  for (int k = threadIdx.x; k < L; k += blockDim.x)
    st[k] = make_ulonglong2(pack2(t.c[k].x, t.c[k].y), pack2(t.c[k].z, t.c[k].w));
  return pack2(t.nz.x, t.nz.y);
}

// Analysis: lo/hi[o] = sum over k of the taps times win(2 o + k), o < RO.
template <int L, int RO, class Win>
__device__ __forceinline__ void analyse(const ulonglong2 *taps, f32x2 nz, Win win,
                                        f32x2 (&lo)[RO], f32x2 (&hi)[RO]) {
  f32x2 v[2 * RO + L - 2];
#pragma unroll
  for (int q = 0; q < 2 * RO - 2; q++) v[q] = win(q);
#pragma unroll
  for (int k = 0; k < L; k++) {
    v[2 * RO - 2 + k] = win(2 * RO - 2 + k);
    const ulonglong2 c = taps[k];
#pragma unroll
    for (int o = 0; o < RO; o++) {
      const f32x2 x = mul2(c.x, v[2 * o + k], nz), y = mul2(c.y, v[2 * o + k], nz);
      lo[o] = k ? add2(lo[o], x) : x;
      hi[o] = k ? add2(hi[o], y) : y;
    }
  }
}

// Synthesis of 2 M consecutive outputs, the first at an even place t = 2 m0: with
// tt = t + L - 2, the taps k = tt & 1, tt & 1 + 2, ... meet h = (tt - k) / 2,
// which is m + L/2 - 1 - q for tap 2 q of output 2 m and for tap 2 q + 1 of
// output 2 m + 1 alike.  win(i) = the (lo, hi) samples at h = m0 + i, zero
// outside the band (a term of value zero leaves the sum, which starts at +0, as
// it is).
template <int L, int M, class Win>
__device__ __forceinline__ void synthesise(const ulonglong2 *taps, f32x2 nz, Win win,
                                           f32x2 (&acc)[2 * M]) {
  constexpr int NW = L / 2 + M - 1;
  f32x2 lo[NW], hi[NW];
#pragma unroll
  for (int i = 0; i < M - 1; i++) win(NW - 1 - i, lo[NW - 1 - i], hi[NW - 1 - i]);
#pragma unroll
  for (int r = 0; r < 2 * M; r++) acc[r] = 0ull;
#pragma unroll
  for (int q = 0; q < L / 2; q++) {
    const int i0 = L / 2 - 1 - q;
    win(i0, lo[i0], hi[i0]);
#pragma unroll
    for (int p = 0; p < 2; p++) {
      const ulonglong2 c = taps[2 * q + p];
#pragma unroll
      for (int m = 0; m < M; m++)
        acc[2 * m + p] = add2(acc[2 * m + p],
                              add2(mul2(c.x, lo[i0 + m], nz), mul2(c.y, hi[i0 + m], nz)));
    }
  }
}

// A warp's RO consecutive outputs per lane of NC rows, written through its shared
// buffer (32 NC RO floats) so that the stores run along the rows.  e0 = the warp's
// first group, ngrp groups per row; store(r, j, value) with r the block's pair of
// rows, j the column, value(c) the output of the c-th of its rows.
template <int RO, int NC, class Value, class Store>
__device__ __forceinline__ void store_rows(float *buf, Value value, int e0, int ngrp, int egrp,
                                           Store store) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
#pragma unroll
  for (int c = 0; c < NC; c++)
#pragma unroll
    for (int o = 0; o < RO; o += 4)
      *reinterpret_cast<float4 *>(buf + (c * 32 + lane) * RO + o) =
          make_float4(value(c, o), value(c, o + 1), value(c, o + 2), value(c, o + 3));
  __syncwarp();
  int r = e0 / ngrp, g = e0 - r * ngrp + lane / RO;
#pragma unroll
  for (int i = 0; i < RO; i++, g += 32 / RO) {
    if (e0 + lane / RO + i * (32 / RO) >= egrp) break;
    while (g >= ngrp) g -= ngrp, r++;
    store(r, g * RO + lane % RO, [=](int c) { return buf[(c * RO + i) * 32 + lane]; });
  }
}

constexpr int FB_PAIRS = 2;  // pairs of rows per block, at most

// Shared memory places of a row of n staged samples, one skipped after every g
// (an even count: the buffers behind are read in 16-byte pieces).
__host__ __device__ inline int fw_pad(int n, int g) { return (n + n / g + 2) & ~1; }

// afb1d along the last axis, two rows at a time: RB pairs of rows (of all the
// chunk's rows in a line) per block are staged in shared memory as float2 (row
// 2 i, row 2 i + 1) with the symmetric extension applied, one place skipped after
// every 2 RO so that lanes RO outputs apart meet different banks.
template <int L, int RO>
__global__ void __launch_bounds__(320) afb_rows_t(const float *__restrict__ x, long long sz,
                                                  int sx, float *__restrict__ out, int B, int H,
                                                  int W, int Wo, int padl, int RB,
                                                  const __grid_constant__ TapPair t) {
  extern __shared__ __align__(16) f32x2 frow[];
  __shared__ ulonglong2 taps[L];
  const f32x2 nz = stage_taps<L>(taps, t);
  const int ngrp = (Wo + RO - 1) / RO;
  const int SW = 2 * RO * ngrp + L - 2, SP = fw_pad(SW, 2 * RO);
  float *buf = reinterpret_cast<float *>(frow + RB * SP) + (threadIdx.x / 32) * 128 * RO;
  const long long nrows = (long long)B * H, row0 = 2LL * blockIdx.x * RB;
  const int np = (int)min((long long)RB, (nrows - row0 + 1) / 2);
  const long long band = (long long)H * Wo;
  __shared__ float *orow[2 * FB_PAIRS];  // the rows' low bands, null past the last row
  if (threadIdx.x < 2 * np) {
    const long long row = row0 + threadIdx.x;
    orow[threadIdx.x] = row < nrows ? out + row / H * 2 * band + row % H * Wo : nullptr;
  }
  for (int r = 0; r < np; r++) {
    const long long ra = row0 + 2 * r, rb = min(ra + 1, nrows - 1);
    const float *xa = x + ra / H * sz + ra % H * sx, *xb = x + rb / H * sz + rb % H * sx;
    f32x2 *sr = frow + r * SP;
#pragma unroll 4
    for (int u = threadIdx.x; u < SW; u += blockDim.x) {
      int m = u - padl;
      if ((unsigned)m >= (unsigned)W) m = reflect(m, W);
      sr[u + u / (2 * RO)] = pack2(xa[m], xb[m]);
    }
  }
  __syncthreads();
  const int egrp = np * ngrp;
  for (int e0 = threadIdx.x & ~31; e0 < egrp; e0 += blockDim.x) {
    const int e = min(e0 + (int)(threadIdx.x & 31), egrp - 1);
    const int r = e / ngrp, g = e - r * ngrp;
    const f32x2 *p = frow + r * SP + g * (2 * RO + 1);
    f32x2 lo[RO], hi[RO];
    analyse<L, RO>(taps, nz, [p](int q) { return p[q + q / (2 * RO)]; }, lo, hi);
    // low and high band of the first row, of the second
    store_rows<RO, 4>(
        buf,
        [&](int c, int o) {
          const float2 w = unpack2(c & 1 ? hi[o] : lo[o]);
          return c & 2 ? w.y : w.x;
        },
        e0, ngrp, egrp, [&](int rr, int j, auto val) {
          if (j >= Wo) return;
          float *oa = orow[2 * rr], *ob = orow[2 * rr + 1];
          oa[j] = val(0);
          oa[band + j] = val(1);
          if (ob) ob[j] = val(2), ob[band + j] = val(3);
        });
  }
}

// Column kernels: a warp takes 64 columns (a lane's two 32 apart in the halves of
// the packed values) and 8 warps adjacent runs of outputs, whose overlapping
// inputs meet in L1.

// afb1d along the rows axis: in [B][2][H][W] -> out [B][4][Ho][W].
template <int L, int RO>
__global__ void __launch_bounds__(256, 2) afb_cols_t(const float *__restrict__ in,
                                                     float *__restrict__ out, int B, int H, int W,
                                                     int Ho, int padl,
                                                     const __grid_constant__ TapPair t) {
  __shared__ ulonglong2 taps[L];
  const f32x2 nz = stage_taps<L>(taps, t);
  __syncthreads();
  const int ncolb = (W + 63) / 64;
  const int ngrp = (Ho + 8 * RO - 1) / (8 * RO);
  const unsigned blk = blockIdx.x;
  const int j = (int)(blk % ncolb) * 64 + threadIdx.x % 32;
  const unsigned rest = blk / ncolb;
  const long long bc = rest / ngrp;
  const int i0 = ((int)(rest % ngrp) * 8 + threadIdx.x / 32) * RO;
  if (i0 >= Ho) return;
  const float *ca = in + bc * H * W + min(j, W - 1), *cb = in + bc * H * W + min(j + 32, W - 1);
  const int r0 = 2 * i0 - padl;
  f32x2 lo[RO], hi[RO];
  if (r0 >= 0 && r0 + 2 * RO + L - 2 <= H) {
    ca += (long long)r0 * W;
    cb += (long long)r0 * W;
    analyse<L, RO>(taps, nz, [=](int q) { return pack2(ca[q * W], cb[q * W]); }, lo, hi);
  } else {
    analyse<L, RO>(taps, nz, [=](int q) {
      int rr = r0 + q;
      if ((unsigned)rr >= (unsigned)H) rr = reflect(rr, H);
      return pack2(ca[(long long)rr * W], cb[(long long)rr * W]);
    }, lo, hi);
  }
  const long long b = bc / 2, c = bc % 2;
  float *o0 = out + ((b * 4 + 2 * c) * Ho + i0) * (long long)W + j;
  float *o1 = o0 + (long long)Ho * W;
  const bool oka = j < W, okb = j + 32 < W;
#pragma unroll
  for (int r = 0; r < RO; r++)
    if (i0 + r < Ho) {
      const float2 l = unpack2(lo[r]), h = unpack2(hi[r]);
      if (oka) o0[r * W] = l.x, o1[r * W] = h.x;
      if (okb) o0[r * W + 32] = l.y, o1[r * W + 32] = h.y;
    }
}

// sfb1d along the rows axis (see sfb_cols).
template <int L, int M>
__global__ void __launch_bounds__(256, 3) sfb_cols_t(const float *__restrict__ y,
                                                     long long bstride, int Hi, int Wb, int W,
                                                     float *__restrict__ out, int B, int Ho,
                                                     const __grid_constant__ TapPair t) {
  static_assert(L % 2 == 0, "even filter length");
  __shared__ ulonglong2 taps[L];
  const f32x2 nz = stage_taps<L>(taps, t);
  __syncthreads();
  const int ncolb = (W + 63) / 64;
  const int ngrp = (Ho + 16 * M - 1) / (16 * M);
  const unsigned blk = blockIdx.x;
  const int j = (int)(blk % ncolb) * 64 + threadIdx.x % 32;
  const unsigned rest = blk / ncolb;
  const long long bc = rest / ngrp;
  const int t0 = ((int)(rest % ngrp) * 8 + threadIdx.x / 32) * 2 * M;
  if (t0 >= Ho) return;
  const int b = (int)(bc / 2), c = (int)(bc % 2);
  const long long plane = (long long)Hi * Wb;
  // channel 0 = LL and band 0 (LH), channel 1 = band 1 (HL) and band 2 (HH)
  const float *la = y + b * bstride + (c == 0 ? 0 : 2) * plane;
  const float *lb = la + min(j + 32, W - 1);
  la += min(j, W - 1);
  const int h0 = t0 / 2;
  f32x2 acc[2 * M];
  if (h0 + L / 2 + M - 1 <= Hi) {
    la += (long long)h0 * Wb;
    lb += (long long)h0 * Wb;
    const float *ha = la + plane, *hb = lb + plane;
    synthesise<L, M>(taps, nz, [=](int i, f32x2 &lo, f32x2 &hi) {
      lo = pack2(la[i * Wb], lb[i * Wb]);
      hi = pack2(ha[i * Wb], hb[i * Wb]);
    }, acc);
  } else {
    synthesise<L, M>(taps, nz, [=](int i, f32x2 &lo, f32x2 &hi) {
      const long long o = (long long)(h0 + i) * Wb;
      const bool ok = h0 + i < Hi;
      lo = ok ? pack2(la[o], lb[o]) : 0ull;
      hi = ok ? pack2(la[plane + o], lb[plane + o]) : 0ull;
    }, acc);
  }
  float *o0 = out + (bc * Ho + t0) * W + j;
  const bool oka = j < W, okb = j + 32 < W;
#pragma unroll
  for (int r = 0; r < 2 * M; r++)
    if (t0 + r < Ho) {
      const float2 v = unpack2(acc[r]);
      if (oka) o0[r * W] = v.x;
      if (okb) o0[r * W + 32] = v.y;
    }
}

// sfb1d along the last axis (see sfb_rows), two rows at a time: RB pairs of rows
// per block staged as float4 (low and high band of the first row and the second:
// the packed low, the packed high), one place skipped after every M.
template <int L, int M>
__global__ void __launch_bounds__(320) sfb_rows_t(const float *__restrict__ in, int H, int Wi,
                                                  float *__restrict__ dst, long long dsz, int dsx,
                                                  int Hd, int Wd, int B, int RB,
                                                  const __grid_constant__ TapPair t) {
  extern __shared__ __align__(16) f32x2 frow[];
  __shared__ ulonglong2 taps[L];
  const f32x2 nz = stage_taps<L>(taps, t);
  const int ngrp = (Wd + 2 * M - 1) / (2 * M);
  const int SW = M * ngrp + L / 2 - 1, SP = fw_pad(SW, M);
  ulonglong2 *srow = reinterpret_cast<ulonglong2 *>(frow);
  float *buf = reinterpret_cast<float *>(srow + RB * SP) + (threadIdx.x / 32) * 128 * M;
  const long long nrows = (long long)B * Hd, row0 = 2LL * blockIdx.x * RB;
  const int np = (int)min((long long)RB, (nrows - row0 + 1) / 2);
  const long long band = (long long)H * Wi;
  __shared__ float *orow[2 * FB_PAIRS];  // output rows, null past the last
  if (threadIdx.x < 2 * np) {
    const long long row = row0 + threadIdx.x;
    orow[threadIdx.x] = row < nrows ? dst + row / Hd * dsz + row % Hd * dsx : nullptr;
  }
  for (int r = 0; r < np; r++) {
    const long long ra = row0 + 2 * r, rb = min(ra + 1, nrows - 1);
    const float *la = in + (ra / Hd * 2 * H + ra % Hd) * Wi;
    const float *lb = in + (rb / Hd * 2 * H + rb % Hd) * Wi;
    ulonglong2 *sr = srow + r * SP;
#pragma unroll 4
    for (int u = threadIdx.x; u < SW; u += blockDim.x) {
      ulonglong2 w = make_ulonglong2(0ull, 0ull);
      if (u < Wi) {
        w.x = pack2(la[u], lb[u]);
        w.y = pack2(la[band + u], lb[band + u]);
      }
      sr[u + u / M] = w;
    }
  }
  __syncthreads();
  const int egrp = np * ngrp;
  for (int e0 = threadIdx.x & ~31; e0 < egrp; e0 += blockDim.x) {
    const int e = min(e0 + (int)(threadIdx.x & 31), egrp - 1);
    const int r = e / ngrp, g = e - r * ngrp;
    const ulonglong2 *p = srow + r * SP + g * (M + 1);
    f32x2 acc[2 * M];
    synthesise<L, M>(taps, nz, [p](int i, f32x2 &lo, f32x2 &hi) {
      const ulonglong2 w = p[i + i / M];
      lo = w.x;
      hi = w.y;
    }, acc);
    store_rows<2 * M, 2>(
        buf,
        [&](int c, int o) {
          const float2 w = unpack2(acc[o]);
          return c ? w.y : w.x;
        },
        e0, ngrp, egrp, [&](int rr, int j, auto val) {
          if (j >= Wd) return;
          float *oa = orow[2 * rr], *ob = orow[2 * rr + 1];
          oa[j] = val(0);
          if (ob) ob[j] = val(1);
        });
  }
}

// [B][R][C] <-> [B][C][R] (32x32 tiles)
__global__ void transpose_bands(const float *__restrict__ in, long long istride,
                                float *__restrict__ out, long long ostride, int R, int C) {
  __shared__ float t[32][33];
  int b = blockIdx.z;
  int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  const float *src = in + b * istride;
  float *dst = out + b * ostride;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    int r = r0 + k, c = c0 + threadIdx.x;
    if (r < R && c < C) t[k][threadIdx.x] = src[(long long)r * C + c];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    int c = c0 + k, r = r0 + threadIdx.x;
    if (r < R && c < C) dst[(long long)c * R + r] = t[threadIdx.x][k];
  }
}

__global__ void damp_kernel(float2 *__restrict__ spec, const float *__restrict__ damp, int nc,
                            long long total) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  float d = damp[i % nc];
  float2 v = spec[i];
  spec[i] = make_float2(v.x * d, v.y * d);
}

// Damping by the low Fourier modes, in place on band [B][H][W] (slice
// stride bstride): a block takes 32 adjacent columns (threadIdx.x) of one
// slice, 8 row phases (threadIdx.y).  cs[q * V1 + k] = (cos, sin)(2 pi k q / H)
// (read 16 bytes at a time)
// and gw[k] = g_k / H (k = 0) or 2 g_k / H (k >= 1, the mode and its mirror
// H - k).  Pass 1 sums A_k = sum_q x_q cos, S_k = sum_q x_q sin per column;
// pass 2 writes x_q - sum_k gw_k (A_k cos + S_k sin).
constexpr int DM_R = 8;

template <int V1>
__global__ void __launch_bounds__(32 * DM_R)
    damp_modes(float *__restrict__ band, long long bstride, int H, int W,
               const float4 *__restrict__ cs, const float *__restrict__ gw) {
  __shared__ float red[DM_R][V1][32];
  const int w = blockIdx.x * 32 + threadIdx.x, r = threadIdx.y;
  float *col = band + (long long)blockIdx.y * bstride + w;
  const bool on = w < W;
  float A[V1], S[V1];
#pragma unroll
  for (int k = 0; k < V1; k++) A[k] = S[k] = 0.f;
  if (on)
#pragma unroll 4
    for (int q = r; q < H; q += DM_R) {
      const float x = col[(long long)q * W];
#pragma unroll
      for (int k = 0; k < V1; k += 2) {
        const float4 t = __ldg(cs + (q * V1 + k) / 2);
        A[k] = fmaf(x, t.x, A[k]);
        S[k] = fmaf(x, t.y, S[k]);
        A[k + 1] = fmaf(x, t.z, A[k + 1]);
        S[k + 1] = fmaf(x, t.w, S[k + 1]);
      }
    }
  // the 8 row phases' partial sums, cosine then sine terms through one buffer
#pragma unroll
  for (int k = 0; k < V1; k++) red[r][k][threadIdx.x] = A[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < V1; k++) {
    float a = 0.f;
#pragma unroll
    for (int j = 0; j < DM_R; j++) a += red[j][k][threadIdx.x];
    A[k] = a * __ldg(gw + k);
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < V1; k++) red[r][k][threadIdx.x] = S[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < V1; k++) {
    float b = 0.f;
#pragma unroll
    for (int j = 0; j < DM_R; j++) b += red[j][k][threadIdx.x];
    S[k] = b * __ldg(gw + k);
  }
  if (!on) return;
#pragma unroll 4
  for (int q = r; q < H; q += DM_R) {
    float lp = 0.f;
#pragma unroll
    for (int k = 0; k < V1; k += 2) {
      const float4 t = __ldg(cs + (q * V1 + k) / 2);
      lp = fmaf(A[k], t.x, fmaf(S[k], t.y, lp));
      lp = fmaf(A[k + 1], t.z, fmaf(S[k + 1], t.w, lp));
    }
    col[(long long)q * W] -= lp;
  }
}

}  // namespace sw
}  // namespace tcb

using namespace tcb;
using namespace tcb::sw;

struct tcb_stripe_fw {
  int nproj, nz, ni, level, nproj_pad, L;
  std::vector<int> H, W;  // level sizes: H[0] = nproj_pad, W[0] = ni
  std::vector<float *> Y; // per level [nz][4][H[k+1]][W[k+1]]
  std::vector<float *> damp;  // per level damping factors (with 1/H)
  std::vector<cufftHandle> r2c, c2r;
  std::vector<int> modes;     // per level: modes of the direct damping (0 = cuFFT)
  std::vector<float4 *> mcs;  // per level [H][modes] (cos, sin)(2 pi k q / H)
  std::vector<float *> mgw;   // per level [modes] weights
  float *tmp = nullptr;    // [nz][2][H][W] scratch
  float *bt = nullptr;     // transposed band scratch
  float2 *spec = nullptr;  // band spectrum scratch
  Taps *taps = nullptr;    // device copy
  size_t tmp_elems = 0;
  TapPair ana{}, syn{};    // by-value taps of the register-blocked kernels
};

namespace {
// Outputs per thread of the analysis along the rows; the largest count along the
// columns, and of the synthesis half of it.
constexpr int FB_RO = 4, FB_CO = 8, FB_M = 4;
// Fewer outputs of a kernel in a level than this leave most of the chip idle, and
// what counts is how long one thread takes: half as many outputs per thread then.
// Measured over 512 to 2048 columns, 360 to 1500 angles, 2 to 16 slices, at the
// full and at half the count: analysis of columns 10.5 and 7.5 us at 10^5
// outputs, 14.0 and 14.2 at 1.6 10^6, 28.4 and 31.1 at 5.6 10^6; synthesis of
// columns 5.3 and 4.4, 6.9 and 6.6 at 5 10^5, 11.4 and 12.5; of rows 5.3 and 4.6,
// 7.0 and 5.6 at 4 10^5, 9.8 and 10.1 at 1.1 10^6, 25.2 and 26.1.
constexpr long long FB_AC_FEW = 1500000, FB_SC_FEW = 500000, FB_SR_FEW = 1000000;
// wide rows' shared memory (one value for every call: threads may launch at once)
constexpr int FB_MAX_SMEM = 220 * 1024;

// Pairs of rows and threads per block of a row kernel: `groups` threads' turns and
// `bytes` of shared memory per pair, `pairs` in all.  A block stages its pairs one
// after the other, so it takes one, or two where that leaves a block per SM and
// fewer lanes idle in the last turn; the smaller block where they are alike.  (Up
// to 16 pairs, chosen by the idle lanes alone: 10 to 15 us for the small levels,
// which take 4.5 so, and 190 against 171 us for 1690 x 1290 x 16.)
void rows_split(int groups, size_t bytes, long long pairs, int &RB, int &T) {
  const int most = pairs >= 2 * sm_count() ? FB_PAIRS : 1;
  double best = 0;
  for (int rb = 1; rb <= most && (rb == 1 || rb * bytes <= 40960); rb++)
    for (int th = 128; th <= 320; th += 32) {
      const int turns = (rb * groups + th - 1) / th;
      const double use = (double)rb * groups / ((double)turns * th);
      if (best == 0 || use > best + 0.02) best = use, RB = rb, T = th;
    }
}

template <int L>
void launch_afb_rows(const tcb_stripe_fw *h, const float *x, long long xsz, int xsx, int B,
                     int Hk, int Wk, int Wo, int padl, cudaStream_t s) {
  const int ngrp = (Wo + FB_RO - 1) / FB_RO;
  const size_t bytes = (size_t)fw_pad(2 * FB_RO * ngrp + L - 2, 2 * FB_RO) * sizeof(f32x2);
  int RB, T;
  rows_split(ngrp, bytes, ((long long)B * Hk + 1) / 2, RB, T);
  const size_t smem = RB * bytes + (size_t)T * 4 * FB_RO * sizeof(float);
  if (smem > 40960)
    cudaFuncSetAttribute(afb_rows_t<L, FB_RO>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         FB_MAX_SMEM);
  const long long nb = ((long long)B * Hk + 2 * RB - 1) / (2 * RB);
  afb_rows_t<L, FB_RO><<<(unsigned)nb, T, smem, s>>>(x, xsz, xsx, h->tmp, B, Hk, Wk, Wo, padl, RB,
                                                     h->ana);
}

template <int L, int RO>
void afb_cols_of(const tcb_stripe_fw *h, float *out, int B, int Hk, int Wo, int Ho, int padl,
                 cudaStream_t s) {
  const long long nb = (long long)ceil_div(Wo, 64) * (2LL * B) * ((Ho + 8 * RO - 1) / (8 * RO));
  afb_cols_t<L, RO><<<(unsigned)nb, 256, 0, s>>>(h->tmp, out, B, Hk, Wo, Ho, padl, h->ana);
}

template <int L>
void launch_afb_cols(const tcb_stripe_fw *h, float *out, int B, int Hk, int Wo, int Ho, int padl,
                     cudaStream_t s) {
  if (4LL * B * Ho * Wo < FB_AC_FEW)
    afb_cols_of<L, FB_CO / 2>(h, out, B, Hk, Wo, Ho, padl, s);
  else
    afb_cols_of<L, FB_CO>(h, out, B, Hk, Wo, Ho, padl, s);
}

template <int L, int M>
void sfb_cols_of(const tcb_stripe_fw *h, const float *y, int Hi, int Wi, int B, int Hc,
                 cudaStream_t s) {
  const long long nb = (long long)ceil_div(Wi, 64) * (2LL * B) * ((Hc + 16 * M - 1) / (16 * M));
  sfb_cols_t<L, M><<<(unsigned)nb, 256, 0, s>>>(y, 4LL * Hi * Wi, Hi, Wi, Wi, h->tmp, B, Hc,
                                                h->syn);
}

template <int L>
void launch_sfb_cols(const tcb_stripe_fw *h, const float *y, int Hi, int Wi, int B, int Hc,
                     cudaStream_t s) {
  if (2LL * B * Hc * Wi < FB_SC_FEW)
    sfb_cols_of<L, FB_M / 2>(h, y, Hi, Wi, B, Hc, s);
  else
    sfb_cols_of<L, FB_M>(h, y, Hi, Wi, B, Hc, s);
}

template <int L, int M>
void sfb_rows_of(const tcb_stripe_fw *h, int Hc, int Wi, float *dst, long long dsz, int Wd,
                 int Hrows, int B, cudaStream_t s) {
  const int ngrp = (Wd + 2 * M - 1) / (2 * M);
  const size_t bytes = (size_t)fw_pad(M * ngrp + L / 2 - 1, M) * sizeof(ulonglong2);
  int RB, T;
  rows_split(ngrp, bytes, ((long long)B * Hrows + 1) / 2, RB, T);
  const size_t smem = RB * bytes + (size_t)T * 4 * M * sizeof(float);
  if (smem > 40960)
    cudaFuncSetAttribute(sfb_rows_t<L, M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         FB_MAX_SMEM);
  const long long nb = ((long long)B * Hrows + 2 * RB - 1) / (2 * RB);
  sfb_rows_t<L, M><<<(unsigned)nb, T, smem, s>>>(h->tmp, Hc, Wi, dst, dsz, Wd, Hrows, Wd, B, RB,
                                                 h->syn);
}

template <int L>
void launch_sfb_rows(const tcb_stripe_fw *h, int Hc, int Wi, float *dst, long long dsz, int Wd,
                     int Hrows, int B, cudaStream_t s) {
  if ((long long)B * Hrows * Wd < FB_SR_FEW)
    sfb_rows_of<L, FB_M / 2>(h, Hc, Wi, dst, dsz, Wd, Hrows, B, s);
  else
    sfb_rows_of<L, FB_M>(h, Hc, Wi, dst, dsz, Wd, Hrows, B, s);
}

bool blocked_length(int L) { return L == 2 || L == 10 || L == 32; }
}  // namespace

static void fw_release(tcb_stripe_fw *h) {
  for (auto p : h->Y) cudaFree(p);
  for (auto p : h->damp) cudaFree(p);
  for (auto p : h->r2c) if (p) cufftDestroy(p);
  for (auto p : h->c2r) if (p) cufftDestroy(p);
  for (auto p : h->mcs) cudaFree(p);
  for (auto p : h->mgw) cudaFree(p);
  h->mcs.clear();
  h->mgw.clear();
  h->modes.clear();
  h->Y.clear();
  h->damp.clear();
  h->r2c.clear();
  h->c2r.clear();
  cudaFree(h->tmp);
  cudaFree(h->bt);
  cudaFree(h->spec);
  cudaFree(h->taps);
  h->tmp = h->bt = nullptr;
  h->spec = nullptr;
  h->taps = nullptr;
}

extern "C" int tcb_stripe_fw_create(tcb_stripe_fw **out, size_t nproj, size_t nz, size_t ni,
                                    int level, float sigma, const double *dec_lo,
                                    const double *dec_hi, const double *rec_lo,
                                    const double *rec_hi, int L) {
  TCB_CHECK_ARG(out, "tcb_stripe_fw_create: null out");
  *out = nullptr;
  TCB_CHECK_ARG(nproj >= 2 && nz >= 1 && ni >= 2 && level >= 1 && level <= 16,
                "tcb_stripe_fw_create: bad sizes");
  TCB_CHECK_ARG(L >= 2 && L <= MAXL && dec_lo && dec_hi && rec_lo && rec_hi,
                "tcb_stripe_fw_create: bad filter bank (L=%d)", L);
  TCB_CHECK_ARG(sigma > 0, "tcb_stripe_fw_create: sigma must be > 0");
  tcb_stripe_fw *h = new tcb_stripe_fw();
  h->nproj = (int)nproj;
  h->nz = (int)nz;
  h->ni = (int)ni;
  h->level = level;
  h->nproj_pad = (int)(nproj + nproj / 8);
  h->L = L;
  h->H.push_back(h->nproj_pad);
  h->W.push_back((int)ni);
  for (int k = 0; k < level; k++) {
    h->H.push_back((h->H[k] + L - 1) / 2);
    h->W.push_back((h->W[k] + L - 1) / 2);
  }
  auto fail = [&](int code, const char *what) {
    set_error("tcb_stripe_fw_create: %s", what);
    fw_release(h);
    delete h;
    return code;
  };
  Taps t{};
  t.L = L;
  for (int k = 0; k < L; k++) {  // float32 taps, analysis filters reversed
    t.h0[k] = (float)dec_lo[L - 1 - k];
    t.h1[k] = (float)dec_hi[L - 1 - k];
    t.g0[k] = (float)rec_lo[k];
    t.g1[k] = (float)rec_hi[k];
  }
  for (int k = 0; k < L; k++) {
    h->ana.c[k] = make_float4(t.h0[k], t.h0[k], t.h1[k], t.h1[k]);
    h->syn.c[k] = make_float4(t.g0[k], t.g0[k], t.g1[k], t.g1[k]);
  }
  h->ana.nz = h->syn.nz = make_float2(-0.f, -0.f);
  if (cudaMalloc(&h->taps, sizeof(Taps)) != cudaSuccess)
    return fail(TCB_ERR_OUT_OF_MEMORY, "cudaMalloc failed");
  if (cudaMemcpy(h->taps, &t, sizeof(Taps), cudaMemcpyHostToDevice) != cudaSuccess)
    return fail(TCB_ERR_CUDA, "cudaMemcpy failed");
  size_t maxband = 0, maxtmp = 0;
  for (int k = 0; k < level; k++) {
    int Ho = h->H[k + 1], Wo = h->W[k + 1];
    float *y = nullptr;
    if (cudaMalloc(&y, (size_t)nz * 4 * Ho * Wo * sizeof(float)) != cudaSuccess)
      return fail(TCB_ERR_OUT_OF_MEMORY, "cudaMalloc failed");
    h->Y.push_back(y);
    // damping factors (remove_stripe.py:270-274), 1/Ho of the inverse FFT folded in
    int nc = Ho / 2 + 1;
    std::vector<double> yh(Ho);
    for (int q = 0; q < Ho; q++) yh[q] = ((-Ho + 2 * q) + 1) / 2.0;
    std::vector<float> d(nc);
    for (int q = 0; q < nc; q++) {
      double v = yh[(q + Ho / 2) % Ho];  // ifftshift, first nc entries
      d[q] = (float)(-std::expm1(-v * v / (2.0 * (double)sigma * sigma)) / Ho);
    }
    float *dd = nullptr;
    if (cudaMalloc(&dd, nc * sizeof(float)) != cudaSuccess)
      return fail(TCB_ERR_OUT_OF_MEMORY, "cudaMalloc failed");
    h->damp.push_back(dd);
    if (cudaMemcpy(dd, d.data(), nc * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess)
      return fail(TCB_ERR_CUDA, "cudaMemcpy failed");
    cufftHandle p1 = 0, p2 = 0;
    int len[1] = {Ho};
    int batch = (int)(nz * Wo);
    if (cufftPlanMany(&p1, 1, len, nullptr, 1, Ho, nullptr, 1, nc, CUFFT_R2C, batch) !=
            CUFFT_SUCCESS ||
        cufftPlanMany(&p2, 1, len, nullptr, 1, nc, nullptr, 1, Ho, CUFFT_C2R, batch) !=
            CUFFT_SUCCESS)
      return fail(TCB_ERR_CUFFT, "cufftPlanMany failed");
    h->r2c.push_back(p1);
    h->c2r.push_back(p2);
    // the direct damping: modes k with g_k above 1e-12, padded to 8, 16 or 32
    // (the extra ones carry their exact, negligible weights); the mode and its
    // mirror H - k must be distinct
    int need = 0;
    while (need < Ho) {
      const double v = (Ho % 2) ? (double)need : need + 0.5;
      if (std::exp(-v * v / (2.0 * (double)sigma * sigma)) < 1e-12) break;
      need++;
    }
    int V1 = need <= 8 ? 8 : need <= 16 ? 16 : need <= 32 ? 32 : 0;
    if (2 * V1 >= Ho || std::getenv("TCB_FW_DAMP") != nullptr) V1 = 0;
    float2 *mc = nullptr;
    float *mg = nullptr;
    if (V1) {
      std::vector<float2> tab((size_t)V1 * Ho);
      std::vector<float> wt(V1);
      for (int k = 0; k < V1; k++) {
        for (int q = 0; q < Ho; q++) {
          // 2 pi k q / H reduced exactly: (k q mod H) / H
          const double a = 2.0 * M_PI * (double)(((long long)k * q) % Ho) / (double)Ho;
          tab[(size_t)q * V1 + k] = make_float2((float)std::cos(a), (float)std::sin(a));
        }
        const double v = (Ho % 2) ? (double)k : k + 0.5;
        const double g = std::exp(-v * v / (2.0 * (double)sigma * sigma)) / Ho;
        // bin 0 is its own mirror; bin k >= 1 comes with bin H - k, whose
        // factor the half-spectrum inverse takes from bin k
        wt[k] = (float)(k == 0 ? g : 2.0 * g);
      }
      if (cudaMalloc(&mc, tab.size() * sizeof(float2)) != cudaSuccess ||
          cudaMalloc(&mg, V1 * sizeof(float)) != cudaSuccess) {
        cudaFree(mc);
        return fail(TCB_ERR_OUT_OF_MEMORY, "cudaMalloc failed");
      }
      if (cudaMemcpy(mc, tab.data(), tab.size() * sizeof(float2), cudaMemcpyHostToDevice) !=
              cudaSuccess ||
          cudaMemcpy(mg, wt.data(), V1 * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaFree(mc);
        cudaFree(mg);
        return fail(TCB_ERR_CUDA, "cudaMemcpy failed");
      }
    }
    h->modes.push_back(V1);
    h->mcs.push_back(reinterpret_cast<float4 *>(mc));
    h->mgw.push_back(mg);
    maxband = std::max(maxband, (size_t)nz * Ho * Wo);
    maxtmp = std::max(maxtmp, (size_t)nz * 2 * h->H[k] * Wo);          // afb rows output
    maxtmp = std::max(maxtmp, (size_t)nz * 2 * (2 * Ho - L + 2) * Wo);  // sfb cols output
  }
  if (cudaMalloc(&h->tmp, maxtmp * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&h->bt, maxband * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&h->spec, (maxband / 2 + (size_t)nz * h->W[1] + 16) * sizeof(float2)) !=
          cudaSuccess)
    return fail(TCB_ERR_OUT_OF_MEMORY, "cudaMalloc failed");
  h->tmp_elems = maxtmp;
  *out = h;
  return TCB_OK;
}

// Ring removal in place on padded sinograms sino [nz][nproj_pad][ni] (slice
// stride sstride elements): rows [(pad)/2, (pad)/2 + nproj) hold the data,
// the other rows must be zero on entry (they are overwritten).
extern "C" int tcb_stripe_fw_apply_sino(tcb_stripe_fw *h, float *sino, size_t sstride,
                                        void *stream) {
  TCB_CHECK_ARG(h && h->taps, "tcb_stripe_fw_apply_sino: null or freed handle");
  TCB_CHECK_ARG(sino, "tcb_stripe_fw_apply_sino: null pointer");
  TCB_CHECK_ARG(sstride >= (size_t)h->nproj_pad * h->ni, "tcb_stripe_fw_apply_sino: stride");
  cudaStream_t s = (cudaStream_t)stream;
  const int B = h->nz, L = h->L;
  // forward
  for (int k = 0; k < h->level; k++) {
    int Hk = h->H[k], Wk = h->W[k], Ho = h->H[k + 1], Wo = h->W[k + 1];
    const float *x;
    long long xsz;
    int xsx;
    if (k == 0) {
      x = sino;
      xsz = (long long)sstride;
      xsx = Wk;
    } else {
      x = h->Y[k - 1];  // LL channel of the previous level
      xsz = 4LL * Hk * Wk;
      xsx = Wk;
    }
    int pw = 2 * (Wo - 1) - Wk + L, ph = 2 * (Ho - 1) - Hk + L;
    long long n1 = (long long)B * Hk * Wo;
    {
      StageTimer st("fw_afb_rows", s);
      switch (blocked_length(L) ? L : 0) {
        case 2: launch_afb_rows<2>(h, x, xsz, xsx, B, Hk, Wk, Wo, pw / 2, s); break;
        case 10: launch_afb_rows<10>(h, x, xsz, xsx, B, Hk, Wk, Wo, pw / 2, s); break;
        case 32: launch_afb_rows<32>(h, x, xsz, xsx, B, Hk, Wk, Wo, pw / 2, s); break;
        default:
          afb_rows<<<ceil_div(n1, 256), 256, 0, s>>>(x, xsz, xsx, h->tmp, B, Hk, Wk, Wo, pw / 2,
                                                     h->taps);
      }
    }
    TCB_LAUNCH_CHECK();
    long long n2 = (long long)B * 2 * Ho * Wo;
    {
      StageTimer st("fw_afb_cols", s);
      switch (blocked_length(L) ? L : 0) {
        case 2: launch_afb_cols<2>(h, h->Y[k], B, Hk, Wo, Ho, ph / 2, s); break;
        case 10: launch_afb_cols<10>(h, h->Y[k], B, Hk, Wo, Ho, ph / 2, s); break;
        case 32: launch_afb_cols<32>(h, h->Y[k], B, Hk, Wo, Ho, ph / 2, s); break;
        default:
          afb_cols<<<ceil_div(n2, 256), 256, 0, s>>>(h->tmp, h->Y[k], B, Hk, Wo, Ho, ph / 2,
                                                     h->taps);
      }
    }
    TCB_LAUNCH_CHECK();
    StageTimer std_("fw_damp", s);
    // damp band 1 (index 2 of the level: high-pass along the detector, low-pass along angles)
    float *band = h->Y[k] + 2LL * Ho * Wo;
    if (h->modes[k]) {
      const dim3 gd(ceil_div(Wo, 32), B), bd(32, DM_R);
      switch (h->modes[k]) {
        case 8: damp_modes<8><<<gd, bd, 0, s>>>(band, 4LL * Ho * Wo, Ho, Wo, h->mcs[k], h->mgw[k]); break;
        case 16: damp_modes<16><<<gd, bd, 0, s>>>(band, 4LL * Ho * Wo, Ho, Wo, h->mcs[k], h->mgw[k]); break;
        default: damp_modes<32><<<gd, bd, 0, s>>>(band, 4LL * Ho * Wo, Ho, Wo, h->mcs[k], h->mgw[k]);
      }
      TCB_LAUNCH_CHECK();
      count_launch();
      continue;
    }
    dim3 tb(32, 8);
    dim3 g1(ceil_div(Wo, 32), ceil_div(Ho, 32), B);
    transpose_bands<<<g1, tb, 0, s>>>(band, 4LL * Ho * Wo, h->bt, (long long)Ho * Wo, Ho, Wo);
    TCB_LAUNCH_CHECK();
    TCB_CUFFT(cufftSetStream(h->r2c[k], s));
    TCB_CUFFT(cufftSetStream(h->c2r[k], s));
    TCB_CUFFT(cufftExecR2C(h->r2c[k], h->bt, (cufftComplex *)h->spec));
    int nc = Ho / 2 + 1;
    long long tot = (long long)B * Wo * nc;
    damp_kernel<<<ceil_div(tot, 256), 256, 0, s>>>(h->spec, h->damp[k], nc, tot);
    TCB_LAUNCH_CHECK();
    TCB_CUFFT(cufftExecC2R(h->c2r[k], (cufftComplex *)h->spec, h->bt));
    dim3 g2(ceil_div(Ho, 32), ceil_div(Wo, 32), B);
    transpose_bands<<<g2, tb, 0, s>>>(h->bt, (long long)Ho * Wo, band, 4LL * Ho * Wo, Wo, Ho);
    TCB_LAUNCH_CHECK();
    count_launch(5);
  }
  // inverse
  for (int k = h->level - 1; k >= 0; k--) {
    int Hi = h->H[k + 1], Wi = h->W[k + 1];
    int Hc = 2 * Hi - L + 2;  // rows after the column synthesis
    long long n1 = (long long)B * 2 * Hc * Wi;
    {
      StageTimer st("fw_sfb_cols", s);
      switch (blocked_length(L) ? L : 0) {
        case 2: launch_sfb_cols<2>(h, h->Y[k], Hi, Wi, B, Hc, s); break;
        case 10: launch_sfb_cols<10>(h, h->Y[k], Hi, Wi, B, Hc, s); break;
        case 32: launch_sfb_cols<32>(h, h->Y[k], Hi, Wi, B, Hc, s); break;
        default:
          sfb_cols<<<ceil_div(n1, 256), 256, 0, s>>>(h->Y[k], 4LL * Hi * Wi, Hi, Wi, Wi, h->tmp,
                                                     B, Hc, h->taps);
      }
    }
    TCB_LAUNCH_CHECK();
    // reconstruction of level k's input, cropped to its size, into the LL
    // channel of the level above (or into the sinograms)
    int Hd = h->H[k], Wd = h->W[k];
    float *dst;
    long long dsz;
    if (k == 0) {
      dst = sino;
      dsz = (long long)sstride;
    } else {
      dst = h->Y[k - 1];
      dsz = 4LL * Hd * Wd;
    }
    int Hrows = std::min(Hd, Hc);
    long long n2 = (long long)B * Hrows * Wd;
    StageTimer st("fw_sfb_rows", s);
    switch (blocked_length(L) ? L : 0) {
      case 2: launch_sfb_rows<2>(h, Hc, Wi, dst, dsz, Wd, Hrows, B, s); break;
      case 10: launch_sfb_rows<10>(h, Hc, Wi, dst, dsz, Wd, Hrows, B, s); break;
      case 32: launch_sfb_rows<32>(h, Hc, Wi, dst, dsz, Wd, Hrows, B, s); break;
      default:
        sfb_rows<<<ceil_div(n2, 256), 256, 0, s>>>(h->tmp, Hc, Wi, dst, dsz, Wd, Hrows, Wd, B,
                                                   h->taps);
    }
    TCB_LAUNCH_CHECK();
    count_launch(2);
  }
  return TCB_OK;
}

extern "C" int tcb_stripe_fw_destroy(tcb_stripe_fw *h) {
  if (!h) return TCB_OK;
  fw_release(h);
  delete h;
  return TCB_OK;
}
