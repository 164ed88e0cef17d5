// A complex FFT of N = 2^LOGN points held in the registers of one CTA, for the envelope
// grid: N / V threads of V points each (V = 32; 16 or 8 for short rows).
//
// The factorisation is N = V x V x G, G = N / V^2 <= 16, decimation in frequency:
//   pass 1  thread t holds x[t + r T], r < V (T = N / V threads): a V-point DFT over r, the
//           twiddle w_N^(f t), output f to row f of shared memory (M = T points per row)
//   pass 2  row f belongs to G consecutive threads: thread j holds row points j + G r, a
//           V-point DFT over r, the twiddle w_M^(g j), output g to places g G .. + G - 1
//   pass 3  thread j holds the row's V consecutive points from j V: V / G DFTs of G points
// The result stays there, bin k = f + V (g + V h) of point (g, h): a product with a spectrum
// stored in that order needs no reordering, and the inverse runs the same passes backwards
// (decimation in time) to natural order x[t + r T] again.  So a forward and an inverse
// transform exchange points four times through shared memory, of which two stay inside a
// warp's G-thread groups; the passes of a shared-memory FFT (fft.cuh) would cross it eight
// times and once more for the bit-reversed product.
//
// An exchange moves the real parts, then the imaginary parts, through one plane of N reals,
// so that the caller keeps room for a second row.  The plane is padded by one element per V:
// every access above then has its 32 lanes (16 for FP64) on consecutive or V + 1 strided
// places, each in a bank of its own, at offsets known at compile time.
//
// Twiddles come from tables in the threads' order (coalesced): `outer` holds, for half p of a
// doubled row (below), w_2N^((2 f + p) t) at [(p V + f) T + t]; `inner` w_M^(g j) at [g G + j].
//
// A linear convolution on the doubled, zero-padded row of 2N points splits into two N-point
// transforms: the even bins 2k are FFT_N(x), the odd bins 2k + 1 are FFT_N(x[t] w_2N^t), with
// w_2N^(t + r T) = w_2N^t w_2V^r: a constant per register beside the table's p = 1 half.
#pragma once
#include "sp_common.cuh"

namespace sp {
namespace regs {

// cos(2 pi k / 64), k <= 16: the doubles nearest the exact values
__device__ constexpr double kCos64[17] = {
    1.0, 0.9951847266721969, 0.9807852804032304, 0.9569403357322088, 0.9238795325112867,
    0.881921264348355, 0.8314696123025452, 0.773010453362737, 0.7071067811865476,
    0.6343932841636455, 0.5555702330196023, 0.4713967368259978, 0.3826834323650898,
    0.29028467725446233, 0.19509032201612833, 0.0980171403295606, 0.0};

__device__ __forceinline__ constexpr double cos64(int e) {
  e &= 63;
  return e <= 16 ? kCos64[e] : e <= 32 ? -kCos64[32 - e] : e <= 48 ? -kCos64[e - 32] : kCos64[64 - e];
}

// a exp(-2 pi i e / 64) (conjugated for the inverse); e is a compile-time constant once unrolled
template <bool kInv, class C>
__device__ __forceinline__ C rotate64(C a, int e) {
  using T = decltype(a.x);
  e &= 63;
  if (e == 0) return a;
  if (e == 16) return kInv ? mul_pi(a) : mul_mi(a);
  if (e == 32) {
    a.x = -a.x;
    a.y = -a.y;
    return a;
  }
  if (e == 48) return kInv ? mul_mi(a) : mul_pi(a);
  C w;
  w.x = (T)cos64(e);
  w.y = kInv ? (T)cos64(e - 16) : (T)-cos64(e - 16);  // sin(x) = cos(x - pi / 2)
  return cmul(a, w);
}

__host__ __device__ constexpr int rev(int r, int bits) {
  int v = 0;
  for (int b = 0; b < bits; ++b) v |= ((r >> b) & 1) << (bits - 1 - b);
  return v;
}

// 2^K-point DFTs over registers x[at .. at + 2^K): natural order in, output o at register rev(o)
template <int K, class C>
__device__ __forceinline__ void dft_dif(C* x) {
#pragma unroll
  for (int level = K; level >= 1; --level) {
#pragma unroll
    for (int q = 0; q < (1 << (K - 1)); ++q) {
      const int half = 1 << (level - 1), i = q & (half - 1), at = ((q >> (level - 1)) << level) + i;
      const C u = x[at], v = x[at + half];
      x[at] = cadd(u, v);
      x[at + half] = rotate64<false>(csub(u, v), i << (6 - level));
    }
  }
}
// the inverse (unnormalised): register rev(o) holds input o, natural order out
template <int K, class C>
__device__ __forceinline__ void dft_dit_inverse(C* x) {
#pragma unroll
  for (int level = 1; level <= K; ++level) {
#pragma unroll
    for (int q = 0; q < (1 << (K - 1)); ++q) {
      const int half = 1 << (level - 1), i = q & (half - 1), at = ((q >> (level - 1)) << level) + i;
      const C u = x[at], v = rotate64<true>(x[at + half], i << (6 - level));
      x[at] = cadd(u, v);
      x[at + half] = csub(u, v);
    }
  }
}

// The tables are read with plain loads, not through the read-only path: those the compiler
// may keep in registers from the forward transform to the inverse, which reads the same
// twiddles, and the row is spilled to make room for them.

// 16 points a thread where the three passes allow it (N <= 4 096), 8 for N = 512: the same exchanges
// as with 32, half the unrolled code and twice the warps.  512 with 16, one warp a row: the inverse
// and the Raman spectrum of 15 FP64 columns 18.9 us, the forward 8.6; with 8 points 9.9 and 5.2
constexpr int default_log_v(int log_n) { return log_n <= 9 ? 3 : log_n <= 12 ? 4 : 5; }

template <class C, int LOGN, int LOGV = default_log_v(LOGN)>
struct Row {
  using R = decltype(C{}.x);
  static constexpr int kLogV = LOGV, V = 1 << kLogV;
  static constexpr int N = 1 << LOGN, T = N / V, M = T, G = M / V;
  static constexpr int kLogG = LOGN - 2 * kLogV;
  static_assert(kLogG >= 1 && G <= V && G <= 32 && T >= 32, "N = V V G with G threads of a warp per row");
  static constexpr int kPitch = M + G;                 // a padded row (one element per V)
  static constexpr size_t kPlane = (size_t)V * kPitch;  // reals of the exchange plane
  // offset of row point m = j + G r beside j < G (the padding (j + G r) / V does not depend on j)
  static __host__ __device__ constexpr int strided(int r) { return G * r + (G * r) / V; }

  // natural x[t + r T] -> point (f, m) of pass 3; the plane's last readers may be anywhere
  static __device__ __forceinline__ void forward(C (&x)[V], R* plane, const C* outer,
                                                 const C* inner, int half) {
    const int t = threadIdx.x, j = t % G;
    R* const column = plane + t + (t >> kLogV);
    R* const row = plane + (t / G) * kPitch;
    dft_dif<kLogV>(x);
    const C* const tw = outer + (size_t)half * N + t;
#pragma unroll
    for (int i = 0; i < V; ++i) x[i] = cmul(x[i], tw[rev(i, kLogV) * T]);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < V; ++i) column[rev(i, kLogV) * kPitch] = x[i].x;
    __syncthreads();
    R re[V];
#pragma unroll
    for (int r = 0; r < V; ++r) re[r] = row[j + strided(r)];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < V; ++i) column[rev(i, kLogV) * kPitch] = x[i].y;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < V; ++r) {
      x[r].x = re[r];
      x[r].y = row[j + strided(r)];
    }
    dft_dif<kLogV>(x);
    const C* const tw_row = inner + j;
#pragma unroll
    for (int i = 0; i < V; ++i)
      if (i > 0) x[i] = cmul(x[i], tw_row[rev(i, kLogV) * G]);
    __syncwarp();  // the row's other threads have read it
#pragma unroll
    for (int i = 0; i < V; ++i) row[j + strided(rev(i, kLogV))] = x[i].x;
    __syncwarp();
#pragma unroll
    for (int e = 0; e < V; ++e) re[e] = row[j * (V + 1) + e];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < V; ++i) row[j + strided(rev(i, kLogV))] = x[i].y;
    __syncwarp();
#pragma unroll
    for (int e = 0; e < V; ++e) {
      x[e].x = re[e];
      x[e].y = row[j * (V + 1) + e];
    }
#pragma unroll
    for (int s = 0; s < V; s += G) dft_dif<kLogG>(x + s);
  }

  // the bin of register e of pass 3: set e / G (g = j V / G + e / G), DFT output h
  static __host__ __device__ constexpr int bin(int t, int e) {
    return t / G + V * ((t % G) * (V / G) + e / G + V * rev(e % G, kLogG));
  }

  // the inverse (unnormalised) of forward: points of pass 3 -> natural x[t + r T]
  static __device__ __forceinline__ void inverse(C (&x)[V], R* plane, const C* outer,
                                                 const C* inner, int half) {
    const int t = threadIdx.x, j = t % G;
    R* const column = plane + t + (t >> kLogV);
    R* const row = plane + (t / G) * kPitch;
    R re[V];
#pragma unroll
    for (int s = 0; s < V; s += G) dft_dit_inverse<kLogG>(x + s);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < V; ++e) row[j * (V + 1) + e] = x[e].x;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < V; ++i) re[i] = row[j + strided(rev(i, kLogV))];
    __syncwarp();
#pragma unroll
    for (int e = 0; e < V; ++e) row[j * (V + 1) + e] = x[e].y;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < V; ++i) {
      x[i].x = re[i];
      x[i].y = row[j + strided(rev(i, kLogV))];
    }
    const C* const tw_row = inner + j;
#pragma unroll
    for (int i = 0; i < V; ++i)
      if (i > 0) x[i] = cmul(x[i], cconj(tw_row[rev(i, kLogV) * G]));
    dft_dit_inverse<kLogV>(x);
    __syncwarp();  // the row's other threads have read it
#pragma unroll
    for (int r = 0; r < V; ++r) row[j + strided(r)] = x[r].x;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < V; ++i) re[i] = column[rev(i, kLogV) * kPitch];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < V; ++r) row[j + strided(r)] = x[r].y;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < V; ++i) {
      x[i].x = re[i];
      x[i].y = column[rev(i, kLogV) * kPitch];
    }
    const C* const tw = outer + (size_t)half * N + t;
#pragma unroll
    for (int i = 0; i < V; ++i) x[i] = cmul(x[i], cconj(tw[rev(i, kLogV) * T]));
    dft_dit_inverse<kLogV>(x);
  }

  // x <- the first N samples of the circular convolution of length 2N of x (zero above N)
  // with the spectrum `table`: half p, register e, thread t at [(p V + e) T + t], 1 / 2N
  // inside.  x holds natural x[t + r T] on both sides; `stash` is a row of N of shared memory
  // of which every thread touches its own places alone.
  static __device__ __forceinline__ void convolve(C (&x)[V], R* plane, C* stash, const C* outer,
                                                  const C* inner, const C* table) {
    const int t = threadIdx.x;
#pragma unroll
    for (int r = 0; r < V; ++r) stash[r * T + t] = x[r];
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      if (half) {
#pragma unroll
        for (int r = 0; r < V; ++r) {
          const C drive = stash[r * T + t];
          stash[r * T + t] = x[r];
          x[r] = rotate64<false>(drive, r * (32 / V));
        }
      }
      forward(x, plane, outer, inner, half);
      const C* const h = table + (size_t)half * N + t;
#pragma unroll
      for (int e = 0; e < V; ++e) x[e] = cmul(x[e], h[e * T]);
      inverse(x, plane, outer, inner, half);
    }
#pragma unroll
    for (int r = 0; r < V; ++r) x[r] = cadd(rotate64<true>(x[r], r * (32 / V)), stash[r * T + t]);
  }
};

}  // namespace regs
}  // namespace sp
