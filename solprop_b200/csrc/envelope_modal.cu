// The envelope grid's modal route with many modes and nodes, on the modal transform's
// products (the GEMM route): the multimode generalised NLSE of a fibre or capillary on
// complex time samples.  backends/numpy_ref/passes/transforms.py:31-233 (ifft / fft with
// the crop, synthesis and projection), responses.py:65-139 (the analytic Kerr cubic),
// responses.py:218-498 (the Raman response on the doubled grid, drive |E|^2 / 2),
// stepping.py:286-369 (the in-stage absorber):
//
//   k_env_inverse  one CTA per modal column: a(t) = ifft(pad(lab)) into the modal field,
//                  interleaved (re, im) rows of 2 n_to; the absorber's spectrum
//                  FFT[-alpha a / 2], cropped, into its spectra block
//   products       E = tau S a and P_m = sum W P / tau over the interleaved rows
//                  (modal_gemm.cu), N = 2 n_to: FP64 products, or tcgen05 products of
//                  three-part BF16 splits accumulated in FP32 in the mixed form
//   k_env_pairs    one CTA per two nodes: the Kerr cubic, the Raman convolutions, the window g
//                  (k_env_kerr without Raman; k_env_nodes_long for FP64 rows of 16 384)
//   k_env_forward  one CTA per modal column: fft of the projected row, cropped
//
// Every transform is the register FFT of fft_regs.cuh (FP64 rows of 16 384 samples: the halves
// of fft_long.cuh over the table exp(-2 pi i m / (2 n_to)), m < n_to).  The inverse transform and
// the modal field are FP64 in both forms; the Kerr cubic, the Raman convolutions and the forward
// transform run in the form's type R (FP32 in the mixed form).
#include <algorithm>
#include <type_traits>

#include "fft.cuh"
#include "fft_long.cuh"
#include "fft_regs.cuh"
#include "kernels.cuh"

namespace sp {

namespace {

constexpr double kEps0 = 8.8541878188e-12;  // vacuum permittivity (F/m), CODATA 2022, as solprop.constants
constexpr int kEnvThreads = 1024;

// A column's (or kernel's) transform is one CTA's chain of passes, run once: what bounds it is
// latency, the instructions' own fetch included, so its threads hold 16 points where the three
// passes allow it (fft_regs.cuh).  30 columns of 4 096 and two Raman kernels, ncu: the inverse and
// the kernels' spectra 32.6 + 28.6 us with shared-memory radix-4 transforms in launches of their
// own -> 32.4 us, the FP32 forward 14.7 -> 13.4 (with 32 points per thread 28.6); FP64 columns of
// 8 192: 66 + 46 -> 57 us, the forward 34 us.

// The Raman kernels' spectra in k_env_pairs' order (rows of up to 8 192; longer ones take
// k_raman_kernel and k_raman_table): one CTA per kernel and half p transforms the damped
// kernel's samples s and s + n together, K[s] + K[s + n] for the even bins of the doubled row
// and (K[s] - K[s + n]) w_2n^s for the odd ones.  Both halves scale by the power of two that
// brings the kernel's sum of magnitudes, a bound of its bins, into [1, 2) (the mixed form).
template <class R, int LOGN>
__device__ __forceinline__ void raman_row(const EnvModalArgsT<R>& a, const RamanArgs& ra, cplx<R>* table, int kernel,
                                          int half, double* plane) {
  using Row = regs::Row<double2, LOGN>;
  constexpr int n = Row::N, T = Row::T, V = Row::V;
  const int t0 = threadIdx.x;
  double2 x[V];
  double sum = 0.0;
#pragma unroll 4
  for (int r = 0; r < V; ++r) {
    const double k0 = raman_sample(ra, kernel, t0 + r * T), k1 = raman_sample(ra, kernel, n + t0 + r * T);
    sum += fabs(k0) + fabs(k1);
    plane[r * T + t0] = half ? k0 - k1 : k0 + k1;  // each thread its own places
  }
#pragma unroll
  for (int r = 0; r < V; ++r) {
    x[r] = make_double2(plane[r * T + t0], 0.0);
    if (half) x[r] = regs::rotate64<false>(x[r], r * (32 / V));
  }
  int shift = 0;
  if (sizeof(R) == 4) {
    __shared__ double part[T / 32];
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if (t0 % 32 == 0) part[t0 / 32] = sum;
    __syncthreads();
    double all = 0.0;
    for (int w = 0; w < T / 32; ++w) all += part[w];
    all *= ra.dt;
    if (all > 0.0) shift = -ilogb(all);
    if (t0 == 0 && half == 0) ra.scale[kernel] = shift;
  }
  Row::forward(x, plane, a.row_outer, a.row_inner, half);
  const double f = scalbn(ra.dt, shift - (LOGN + 1));  // the convolution's 1 / 2n inside
  cplx<R>* out = table + ((size_t)kernel * 2 + half) * n;
#pragma unroll
  for (int e = 0; e < V; ++e)
    out[e * T + t0] = to_c<cplx<R>>(cscale(f, x[e]));
}

// The inverse transform of a column: the padded spectrum is gathered in the register
// transform's bin order (fine_to_coarse: -1 where the band is cropped), so that the inverse
// passes leave a(t) in natural order; the in-stage absorber's -alpha a / 2 goes forward from
// there and its bins are scattered to the cropped spectrum (stage output masks it).
// The Raman kernels' spectra take their CTAs of the same launch, ahead of the columns': they
// are as long a chain, and nothing of them depends on the field.
template <class R, int LOGN>
__global__ void __launch_bounds__(regs::Row<double2, LOGN>::T)
    k_env_inverse(EnvModalArgsT<R> a, RamanArgs ra, cplx<R>* table, int raman_rows) {
  using Row = regs::Row<double2, LOGN>;
  constexpr int n = Row::N, T = Row::T, V = Row::V;
  extern __shared__ __align__(16) double ei_plane[];
  if ((int)blockIdx.x < raman_rows) {
    raman_row<R, LOGN>(a, ra, table, blockIdx.x / 2, blockIdx.x % 2, ei_plane);
    return;
  }
  const int col = blockIdx.x - raman_rows, t0 = threadIdx.x;
  const double2* lab = a.lab + (size_t)col * a.n_omega;
  double2 x[V];
#pragma unroll
  for (int e = 0; e < V; ++e) {
    const int j = a.fine_to_coarse[Row::bin(t0, e)];
    x[e] = j >= 0 ? lab[j] : make_double2(0.0, 0.0);
  }
  Row::inverse(x, ei_plane, a.row_outer, a.row_inner, 0);
  const double inv_n = 1.0 / (double)n;  // scipy's ifft carries 1 / n_to
  double2* row = reinterpret_cast<double2*>(a.modal_t + (size_t)col * 2 * n) + t0;
#pragma unroll
  for (int r = 0; r < V; ++r) {
    x[r] = cscale(inv_n, x[r]);
    row[r * T] = x[r];
  }
  if (!a.alpha) return;
#pragma unroll
  for (int r = 0; r < V; ++r) x[r] = cscale(-0.5 * a.alpha[t0 + r * T], x[r]);
  Row::forward(x, ei_plane, a.row_outer, a.row_inner, 0);
  cplx<R>* absorber = a.spectra + (size_t)3 * a.n_cols * a.n_omega + (size_t)col * a.n_omega;
#pragma unroll
  for (int e = 0; e < V; ++e) {
    const int j = a.fine_to_coarse[Row::bin(t0, e)];
    if (j >= 0) absorber[j] = to_c<cplx<R>>(x[e]);
  }
}

constexpr int kNodeThreads = 512;

// One sample t of a node's gated polarisation: with drive 0 the Kerr cubic and the first
// convolution conv (already times eps0 rho) times the field; the later drives add
// conv [[1, 0], [0, -1]] (the difference) or conv [[0, 1], [1, 0]] (the coherence) times it.
template <class R>
__device__ __forceinline__ void node_sample(const EnvModalArgsT<R>& a, const cplx<R>* Ex, const cplx<R>* Ey,
                                            cplx<R>* Px, cplx<R>* Py, int t, double conv, int dr, int nc,
                                            double factor, R self, R conj) {
  using C = cplx<R>;
  const C x = Ex[t], y = Ey[t];
  const double g = a.t_window[t];
  const double2 dx = to_d2(x), dy = to_d2(y);
  if (dr == 0) {  // the Kerr cubic and the first convolution
    double2 px = make_double2(0.0, 0.0), py = px;
    if (a.kerr) {  // c rho (s (sum |a|^2) a_p + q (sum a^2) a_p*), summed over the components
      R mod = x.x * x.x + x.y * x.y;
      C sq = cmul(x, x);
      if (nc == 2) {
        mod += y.x * y.x + y.y * y.y;
        sq = cadd(sq, cmul(y, y));
      }
      const C cx = cadd(cscale(self * mod, x), cscale(conj, cmul(sq, cconj(x))));
      px = make_double2(factor * (double)cx.x, factor * (double)cx.y);
      if (nc == 2) {
        const C cy = cadd(cscale(self * mod, y), cscale(conj, cmul(sq, cconj(y))));
        py = make_double2(factor * (double)cy.x, factor * (double)cy.y);
      }
    }
    px = cadd(px, cscale(conv, dx));
    Px[t] = to_c<C>(cscale(g, px));
    if (nc == 2) {
      py = cadd(py, cscale(conv, dy));
      Py[t] = to_c<C>(cscale(g, py));
    }
  } else if (dr == 1) {  // + v [[1, 0], [0, -1]]
    Px[t] = to_c<C>(cadd(to_d2(Px[t]), cscale(g * conv, dx)));
    Py[t] = to_c<C>(csub(to_d2(Py[t]), cscale(g * conv, dy)));
  } else {  // + w [[0, 1], [1, 0]]
    Px[t] = to_c<C>(cadd(to_d2(Px[t]), cscale(g * conv, dy)));
    Py[t] = to_c<C>(cadd(to_d2(Py[t]), cscale(g * conv, dx)));
  }
}

// The nodes' responses without Raman: the gated Kerr cubic, sample by sample
template <class R>
__global__ void __launch_bounds__(256) k_env_kerr(EnvModalArgsT<R> a, int n_nodes) {
  const double factor = a.kerr ? a.kerr_coefficient * a.stage->kerr_density : 0.0;
  const int nc = a.n_components, n = a.n_to;
  const size_t total = (size_t)n_nodes * n;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t node = i >> a.log_n_to;
    const cplx<R>* Ex = reinterpret_cast<const cplx<R>*>(a.node_field) + node * nc * n;
    cplx<R>* Px = reinterpret_cast<cplx<R>*>(a.node_streams) + node * nc * n;
    const int step = nc == 2 ? n : 0;
    node_sample<R>(a, Ex, Ex + step, Px, Px + step, (int)(i & (n - 1)), 0.0, 0, nc, factor, R(a.kerr_self),
                   R(a.kerr_conjugate));
  }
}

// One sample of a node's gated polarisation with every convolution at hand: the Kerr cubic
// c rho (s (sum |a|^2) a_p + q (sum a^2) a_p*) and the Raman matrix [[u + v, w], [w, u - v]]
// (already times eps0 rho) times the field.  The cubic is formed in R and its SI coefficient
// (about 1e-37 for a gas) applied in FP64, so that it never rounds to an FP32 subnormal.
template <class R>
__device__ __forceinline__ void node_output(const EnvModalArgsT<R>& a, int nc, double factor, double gate,
                                            cplx<R> x, cplx<R> y, double u, double v, double w, cplx<R>& px,
                                            cplx<R>& py) {
  using C = cplx<R>;
  const R self = R(a.kerr_self), conj = R(a.kerr_conjugate);
  const double2 dx = to_d2(x), dy = to_d2(y);
  // without Kerr the cubic is of zeros (a field above 7e12 overflows it in FP32): selections, which
  // the unrolled samples carry better than a branch
  if (!a.kerr) x.x = x.y = y.x = y.y = R(0);
  R mod = x.x * x.x + x.y * x.y;
  C sq = cmul(x, x);
  if (nc == 2) {
    mod += y.x * y.x + y.y * y.y;
    sq = cadd(sq, cmul(y, y));
  }
  const double2 kx = to_d2(cadd(cscale(self * mod, x), cscale(conj, cmul(sq, cconj(x)))));
  const double rx = u + v;
  px = to_c<C>(make_double2(gate * fma(factor, kx.x, fma(rx, dx.x, w * dy.x)),
                            gate * fma(factor, kx.y, fma(rx, dx.y, w * dy.y))));
  if (nc == 2) {
    const double2 ky = to_d2(cadd(cscale(self * mod, y), cscale(conj, cmul(sq, cconj(y)))));
    const double ry = u - v;
    py = to_c<C>(make_double2(gate * fma(factor, ky.x, fma(ry, dy.x, w * dx.x)),
                              gate * fma(factor, ky.y, fma(ry, dy.y, w * dx.y))));
  }
}

// resident CTAs: the rows fill the registers of an SM (V points of 8 or 16 bytes and as much again,
// 64 or 128 registers a thread at least)
template <class R, int LOGN>
constexpr int pairs_resident() {
  using Row = regs::Row<cplx<R>, LOGN>;
  return (sizeof(R) == 4 ? 16384 : 8192) / (Row::V < 16 ? 16 : Row::V) / Row::T;
}

// The second drive of a complex row is brought to the first one's norm by a power of two: a
// transform's rounding is relative to its whole row, so beside a drive 1e6 times as strong the
// weaker one's convolution would keep no digit in FP32.  The norms are estimated as the root of
// peak times sum, which a rectangle meets.  undo: the factors of the two convolutions afterwards,
// zero for a drive of zeros, whose convolution is exactly zero again.
// What it costs: a barrier that waits for the drives' loads, and the sums.  16 384 nodes, rows of
// 16 384: 10.1 -> 10.5 ms an evaluation; 10.9 with both drives scaled and every thread adding the
// warps' sums, 11.5 with all signals gauged while the first one's drives are formed.
template <class R>
struct WarpGauge {
  int peak[2];  // the leading 32 bits of the largest magnitudes, ordered as the magnitudes are
  R sum[2];     // of the magnitudes
};
__device__ __forceinline__ int leading_bits(float a) { return __float_as_int(a); }
__device__ __forceinline__ int leading_bits(double a) { return __double2hiint(a); }
template <class R>
__device__ __forceinline__ int exponent_of(int leading) { return sizeof(R) == 4 ? leading >> 23 : leading >> 20; }
template <class R>
__device__ __forceinline__ R power_of_two(int e) {
  if constexpr (sizeof(R) == 4) return __int_as_float((127 + e) << 23);
  else return __hiloint2double((1023 + e) << 20, 0);
}
template <class Row, class R>
__device__ __forceinline__ void balance(cplx<R> (&x)[Row::V], WarpGauge<R>* part, double* undo) {
  constexpr int warps = Row::T / 32, limit = sizeof(R) == 4 ? 126 : 1022;
  WarpGauge<R> g = {};
#pragma unroll
  for (int r = 0; r < Row::V; ++r) {
    g.peak[0] = max(g.peak[0], leading_bits(fabs(x[r].x)));
    g.peak[1] = max(g.peak[1], leading_bits(fabs(x[r].y)));
    g.sum[0] += fabs(x[r].x);
    g.sum[1] += fabs(x[r].y);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    g.peak[i] = __reduce_max_sync(0xffffffffu, g.peak[i]);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) g.sum[i] += __shfl_xor_sync(0xffffffffu, g.sum[i], d);
  }
  if (threadIdx.x % 32 == 0) part[threadIdx.x / 32] = g;
  __syncthreads();
  g = part[threadIdx.x % warps];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    g.peak[i] = __reduce_max_sync(0xffffffffu, g.peak[i]);
#pragma unroll
    for (int d = warps / 2; d > 0; d >>= 1) g.sum[i] += __shfl_xor_sync(0xffffffffu, g.sum[i], d);
  }
  const int norm0 = exponent_of<R>(g.peak[0]) + exponent_of<R>(leading_bits(g.sum[0]));
  const int norm1 = exponent_of<R>(g.peak[1]) + exponent_of<R>(leading_bits(g.sum[1]));
  const int shift = g.peak[0] && g.peak[1] ? max(-limit, min(limit, (norm0 - norm1) / 2)) : 0;
  if (shift) {
    const R f = power_of_two<R>(shift);
#pragma unroll
    for (int r = 0; r < Row::V; ++r) x[r].y *= f;
  }
  if (threadIdx.x == 0) {
    undo[0] = g.peak[0] ? 1.0 : 0.0;
    undo[1] = g.peak[1] ? power_of_two<double>(-shift) : 0.0;
  }
}

// The nodes' responses with Raman, one CTA per two nodes A and B (or one node).  A convolution with a real
// kernel takes two real drives as one complex row: the trace drives of A and B together
// (drive |a|^2 / 2, or |a_x|^2 / 2 + |a_y|^2 / 2 of two field components), then, where the
// tensor response has a traceless kernel, each node's difference |a_x|^2 / 2 - |a_y|^2 / 2
// and coherence Re(a_x a_y*) (passes/responses.py:501-550).  The convolutions are linear on
// the doubled, zero-padded grid (Row::convolve of fft_regs.cuh), the spectra stored in the
// transform's bin order (k_raman_table), so that no spectrum is unpacked or reordered.  The
// trace convolutions wait for the traceless ones in the last node's polarisation row, each
// thread reading back what it wrote there before it writes the polarisation.
//
// What bounds it: the transforms' FP32 (FP64) issue and their exchanges through shared memory.
// The whole row lies in the registers of one CTA (32 points per thread) and crosses shared
// memory four times per convolution half, where a shared-memory transform of packed real
// drives (one CTA per node) crossed it nine times and gathered bit-reversed pairs besides.
// 16 384 nodes of two components, rows of 16 384, FP32: 33.0 -> 7 ms; 2 025 nodes, rows of
// 8 192, FP64: 2.78 -> 1.0 ms.
template <class R, int LOGN>
__global__ void __launch_bounds__(regs::Row<cplx<R>, LOGN>::T, pairs_resident<R, LOGN>())
    k_env_pairs(EnvModalArgsT<R> a, int n_nodes, int per_cta) {
  using C = cplx<R>;
  using Row = regs::Row<C, LOGN>;
  constexpr int n = Row::N, T = Row::T, V = Row::V;
  extern __shared__ __align__(16) unsigned char ep_raw[];
  C* stash = reinterpret_cast<C*>(ep_raw);
  R* plane = reinterpret_cast<R*>(stash + n);
  const int nc = a.n_components, t0 = threadIdx.x;
  const int first = per_cta * blockIdx.x, count = min(per_cta, n_nodes - first);
  const StageScalarsDev& st = *a.stage;
  const double factor = a.kerr ? a.kerr_coefficient * st.kerr_density : 0.0;
  const double density = kEps0 * (a.raman_mixture ? 1.0 : st.raman_density);  // a mixture's are inside
  const C* const field = reinterpret_cast<const C*>(a.node_field) + (size_t)first * nc * n + t0;
  C* const stream = reinterpret_cast<C*>(a.node_streams) + (size_t)first * nc * n + t0;
  const double* const window = a.t_window + t0;
  auto scale_of = [&](int kernel) {  // the mixed form's table carries the power of two 2^raman_scale
    if constexpr (sizeof(R) == 8) return density;
    else return scalbn(density, -a.raman_scale[kernel]);
  };
  const bool tensor = nc == 2 && a.raman_kernels == 2;
  const double trace_scale = scale_of(0), tensor_scale = tensor ? scale_of(1) : 0.0;
  C* const trace = stream + ((size_t)2 * count - 1) * n;  // tensor: the last node's y row
  const R half = R(0.5);
  C x[V];
  __shared__ WarpGauge<R> part[T / 32];
  __shared__ double undo[4];  // the trace drives' of both nodes, the tensor drives' of this one
  // signal 0: the trace drives of both nodes; signal 1 + q: the tensor drives of node q
#pragma unroll 1
  for (int signal = 0; signal <= (tensor ? count : 0); ++signal) {
    const C* const Ex = field + (size_t)(signal - 1) * 2 * n;  // signal > 0
    if (signal == 0) {
#pragma unroll
      for (int r = 0; r < V; ++r) {
        R d[2] = {R(0), R(0)};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (q < count) {
            const C e = field[(size_t)q * nc * n + r * T];
            d[q] = half * (e.x * e.x + e.y * e.y);
            if (nc == 2) {
              const C f = field[((size_t)q * 2 + 1) * n + r * T];
              d[q] += half * (f.x * f.x + f.y * f.y);
            }
          }
        }
        x[r].x = d[0];
        x[r].y = d[1];
      }
    } else {
#pragma unroll
      for (int r = 0; r < V; ++r) {
        const C e = Ex[r * T], f = Ex[n + r * T];
        x[r].x = half * (e.x * e.x + e.y * e.y) - half * (f.x * f.x + f.y * f.y);
        x[r].y = e.x * f.x + e.y * f.y;
      }
    }
    balance<Row, R>(x, part, undo + (signal ? 2 : 0));
    Row::convolve(x, plane, stash, a.outer_twiddles, a.inner_twiddles, a.raman_table + (signal ? (size_t)2 * n : 0));
    if (signal > 0) {
      C* const Px = stream + (size_t)(signal - 1) * 2 * n;
      const double us = trace_scale * undo[signal - 1], vs = tensor_scale * undo[2], ws = tensor_scale * undo[3];
#pragma unroll
      for (int r = 0; r < V; ++r) {
        const C u = trace[r * T];
        C px, py;
        node_output<R>(a, 2, factor, window[r * T], Ex[r * T], Ex[n + r * T],
                       us * (double)(signal == 2 ? u.y : u.x), vs * (double)x[r].x, ws * (double)x[r].y, px, py);
        Px[r * T] = px;
        Px[n + r * T] = py;
      }
    } else if (tensor) {
#pragma unroll
      for (int r = 0; r < V; ++r) trace[r * T] = x[r];
    } else {
      // rows of the stash carry the convolutions on, so that this rarer form stays a loop
#pragma unroll
      for (int r = 0; r < V; ++r) stash[r * T + t0] = x[r];
#pragma unroll 1
      for (int r = 0; r < V; ++r) {
        const C conv = stash[r * T + t0];
        for (int q = 0; q < count; ++q) {
          const size_t at = (size_t)q * nc * n + r * T;
          const C e = field[at];
          C px, py;
          node_output<R>(a, nc, factor, window[r * T], e, nc == 2 ? field[at + n] : e,
                         trace_scale * undo[q] * (double)(q ? conv.y : conv.x), 0.0, 0.0, px, py);
          stream[at] = px;
          if (nc == 2) stream[at + n] = py;
        }
      }
    }
  }
}

// The kernels' spectra in k_env_pairs' order: half p, register e, thread t at
// [(2 kernel + p) n + e T + t] holds bin 2 k + p of the doubled row, k = Row::bin(t, e), over
// 2n (the transform's normalisation) and, in the mixed form, times 2^raman_scale.
template <class R, int LOGN>
__global__ void __launch_bounds__(256) k_raman_table(const double2* __restrict__ spectrum, const int* scale,
                                                     cplx<R>* __restrict__ table) {
  using Row = regs::Row<cplx<R>, LOGN>;
  constexpr int n = Row::N;
  const int kernel = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
  const int half = i >> LOGN, e = (i & (n - 1)) / Row::T, t = i % Row::T;
  const int k = 2 * Row::bin(t, e) + half;
  const double2* row = spectrum + (size_t)kernel * (n + 1);
  const double2 h = k <= n ? row[k] : cconj(row[2 * n - k]);  // a real kernel's
  const int shift = (scale ? scale[kernel] : 0) - (LOGN + 1);
  table[(size_t)kernel * 2 * n + i] = to_c<cplx<R>>(make_double2(scalbn(h.x, shift), scalbn(h.y, shift)));
}

// The forward transform of a projected column, its bins scattered to the cropped spectrum
template <class R, int LOGN>
__global__ void __launch_bounds__(regs::Row<cplx<R>, LOGN>::T) k_env_forward(EnvModalArgsT<R> a) {
  using C = cplx<R>;
  using Row = regs::Row<C, LOGN>;
  extern __shared__ __align__(16) unsigned char ef_raw[];
  const int col = blockIdx.x, t0 = threadIdx.x;
  const C* row = reinterpret_cast<const C*>(a.projected) + (size_t)col * Row::N + t0;
  C x[Row::V];
#pragma unroll
  for (int r = 0; r < Row::V; ++r) x[r] = row[r * Row::T];
  Row::forward(x, reinterpret_cast<R*>(ef_raw), a.outer_twiddles, a.inner_twiddles, 0);
  C* spectra = a.spectra + (size_t)col * a.n_omega;
#pragma unroll
  for (int e = 0; e < Row::V; ++e) {
    const int j = a.fine_to_coarse[Row::bin(t0, e)];
    if (j >= 0) spectra[j] = x[e];
  }
}

// ---- FP64 rows of 16 384 samples: the halves of fft_long.cuh over each row's scratch
// (1.5 n_to complex: the n_to-point spectrum, then the even half's transform)

__global__ void __launch_bounds__(kEnvThreads) k_env_inverse_long(EnvModalArgsT<double> a) {
  extern __shared__ __align__(16) double2 el_raw[];
  const int n = a.n_to, h = n / 2, log_h = a.log_n_to - 1, col = blockIdx.x;
  double2* S = el_raw;
  double2* gz = a.scratch + (size_t)col * (n + h);
  double2* ge = gz + n;
  for (int k = threadIdx.x; k < n; k += blockDim.x) gz[k] = make_double2(0.0, 0.0);
  __syncthreads();
  const double2* lab = a.lab + (size_t)col * a.n_omega;
  for (int j = threadIdx.x; j < a.n_omega; j += blockDim.x) gz[a.crop[j]] = lab[j];
  __syncthreads();
  const double inv_n = 1.0 / (double)n;  // scipy's ifft carries 1 / n_to
  double2* row = reinterpret_cast<double2*>(a.modal_t + (size_t)col * 2 * n);
  for (int half = 0; half < 2; ++half) {
    long_inverse_half(gz, S, a.twiddles, log_h, half);
    for (int i = threadIdx.x; i < h; i += blockDim.x)
      row[2 * i + half] = cscale(inv_n, S[row_slot<double2>(bitrev(i, log_h))]);
    __syncthreads();
  }
  if (!a.alpha) return;
  long_forward([&](int m) { return cscale(-0.5 * a.alpha[m], row[m]); }, S, gz, ge, a.twiddles, log_h);
  double2* absorber = a.spectra + (size_t)3 * a.n_cols * a.n_omega + (size_t)col * a.n_omega;
  for (int j = threadIdx.x; j < a.n_omega; j += blockDim.x) absorber[j] = gz[a.crop[j]];
}

// the mixed form's inverse: the same FP64 transform, the absorber's spectrum in complex64
__global__ void __launch_bounds__(kEnvThreads) k_env_inverse_long32(EnvModalArgsT<float> a) {
  extern __shared__ __align__(16) double2 em_raw[];
  const int n = a.n_to, h = n / 2, log_h = a.log_n_to - 1, col = blockIdx.x;
  double2* S = em_raw;
  double2* gz = a.scratch + (size_t)col * (n + h);
  double2* ge = gz + n;
  for (int k = threadIdx.x; k < n; k += blockDim.x) gz[k] = make_double2(0.0, 0.0);
  __syncthreads();
  const double2* lab = a.lab + (size_t)col * a.n_omega;
  for (int j = threadIdx.x; j < a.n_omega; j += blockDim.x) gz[a.crop[j]] = lab[j];
  __syncthreads();
  const double inv_n = 1.0 / (double)n;
  double2* row = reinterpret_cast<double2*>(a.modal_t + (size_t)col * 2 * n);
  for (int half = 0; half < 2; ++half) {
    long_inverse_half(gz, S, a.twiddles, log_h, half);
    for (int i = threadIdx.x; i < h; i += blockDim.x)
      row[2 * i + half] = cscale(inv_n, S[row_slot<double2>(bitrev(i, log_h))]);
    __syncthreads();
  }
  if (!a.alpha) return;
  long_forward([&](int m) { return cscale(-0.5 * a.alpha[m], row[m]); }, S, gz, ge, a.twiddles, log_h);
  float2* absorber = a.spectra + (size_t)3 * a.n_cols * a.n_omega + (size_t)col * a.n_omega;
  for (int j = threadIdx.x; j < a.n_omega; j += blockDim.x) absorber[j] = to_c<float2>(gz[a.crop[j]]);
}

__global__ void __launch_bounds__(kEnvThreads) k_env_forward_long(EnvModalArgsT<double> a) {
  extern __shared__ __align__(16) double2 ef_long_raw[];
  const int n = a.n_to, h = n / 2, log_h = a.log_n_to - 1, col = blockIdx.x;
  double2* gz = a.scratch + (size_t)col * (n + h);
  const double2* row = reinterpret_cast<const double2*>(a.projected) + (size_t)col * n;
  long_forward([&](int m) { return row[m]; }, ef_long_raw, gz, gz + n, a.twiddles, log_h);
  double2* spectra = a.spectra + (size_t)col * a.n_omega;
  for (int j = threadIdx.x; j < a.n_omega; j += blockDim.x) spectra[j] = gz[a.crop[j]];
}

// The spectrum product of spectrum_product over a natural-order row in global memory: the
// thread of pair (k, n - k) reads and writes those two bins alone.
__device__ __forceinline__ void spectrum_product_global(double2* Z, const double2* __restrict__ H,
                                                        const double2* __restrict__ tw, int n) {
  for (int k = threadIdx.x; k <= n / 2; k += blockDim.x) {
    const int km = k == 0 ? 0 : n - k;
    const double2 a = Z[k], b = Z[km];
    if (k == 0) {
      const double y0 = cmul(H[0], make_double2(a.x + a.y, 0.0)).x, yn = cmul(H[n], make_double2(a.x - a.y, 0.0)).x;
      Z[0] = make_double2(0.5 * (y0 + yn), 0.5 * (y0 - yn));
      continue;
    }
    const double2 e = cscale(0.5, cadd(a, cconj(b)));
    const double2 o = cscale(0.5, mul_mi(csub(a, cconj(b))));
    const double2 wk = tw[k], wm = tw[km];
    const double2 xk = cadd(e, cmul(wk, o));
    const double2 om = cscale(0.5, mul_mi(csub(b, cconj(a))));
    const double2 xm = cadd(cconj(e), cmul(wm, om));
    const double2 yk = cmul(H[k], xk), ym = cmul(H[km], xm);
    Z[k] = cadd(cscale(0.5, cadd(yk, cconj(ym))), mul_pi(cscale(0.5, cmul(csub(yk, cconj(ym)), cconj(wk)))));
    if (k != n / 2)
      Z[km] = cadd(cscale(0.5, cadd(ym, cconj(yk))), mul_pi(cscale(0.5, cmul(csub(ym, cconj(yk)), cconj(wm)))));
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kNodeThreads, 1) k_env_nodes_long(EnvModalArgsT<double> a) {
  extern __shared__ __align__(16) double2 en_long_raw[];
  const int n = a.n_to, h = n / 2, log_h = a.log_n_to - 1, node = blockIdx.x, nc = a.n_components;
  double2* S = en_long_raw;
  double2* gz = a.scratch + (size_t)node * (n + h);
  double2* ge = gz + n;
  const StageScalarsDev& st = *a.stage;
  const double2* Ex = reinterpret_cast<const double2*>(a.node_field) + (size_t)node * nc * n;
  const double2* Ey = Ex + (nc == 2 ? n : 0);
  double2* Px = reinterpret_cast<double2*>(a.node_streams) + (size_t)node * nc * n;
  double2* Py = Px + (nc == 2 ? n : 0);
  const int drives = nc == 2 && a.raman_kernels == 2 ? 3 : 1;
  const double factor = a.kerr ? a.kerr_coefficient * st.kerr_density : 0.0;
  const double self = a.kerr_self, conj = a.kerr_conjugate;
  const double raman_scale = kEps0 * (a.raman_mixture ? 1.0 : st.raman_density);
  const double inv_n = 1.0 / (double)n;
  for (int dr = 0; dr < drives; ++dr) {
    // the drive on [0, n), zero on [n, 2n), packed b[m] = d(2m) + i d(2m + 1), transformed
    long_forward(
        [&](int m) {
          double v[2] = {0.0, 0.0};
          if (2 * m < n) {
            for (int q = 0; q < 2; ++q) {
              const double2 x = Ex[2 * m + q];
              const double xx = 0.5 * (x.x * x.x + x.y * x.y);
              if (nc == 1) {
                v[q] = xx;
              } else {
                const double2 y = Ey[2 * m + q];
                const double yy = 0.5 * (y.x * y.x + y.y * y.y);
                v[q] = dr == 0 ? xx + yy : dr == 1 ? xx - yy : 2.0 * 0.5 * (x.x * y.x + x.y * y.y);
              }
            }
          }
          return make_double2(v[0], v[1]);
        },
        S, gz, ge, a.twiddles, log_h);
    spectrum_product_global(gz, a.raman_spectrum + (dr == 0 ? 0 : (size_t)(n + 1)), a.twiddles, n);
    // the convolution at samples t < n: packed bins j = t >> 1 < h, j = 2 i + half
    for (int half = 0; half < 2; ++half) {
      long_inverse_half(gz, S, a.twiddles, log_h, half);
      for (int i = threadIdx.x; i < h / 2; i += blockDim.x) {
        const double2 z = S[row_slot<double2>(bitrev(i, log_h))];
        for (int q = 0; q < 2; ++q) {
          const int t = 4 * i + 2 * half + q;
          node_sample<double>(a, Ex, Ey, Px, Py, t, raman_scale * ((q ? z.y : z.x) * inv_n), dr, nc, factor,
                              self, conj);
        }
      }
      __syncthreads();  // the next half's inputs overwrite the row
    }
  }
}

}  // namespace

// ---- the pairs' kernels by row length
template <class R, int LOGN>
constexpr size_t pairs_smem() {
  using Row = regs::Row<cplx<R>, LOGN>;
  return (size_t)Row::N * sizeof(cplx<R>) + Row::kPlane * sizeof(R);
}
// FP32 rows of 512 to 16 384 samples, FP64 rows of up to 8 192 (the row and the exchange
// plane of the longest fill 194 KB of shared memory in either type)
template <class R, class F>
static cudaError_t with_row(int log_n, F&& f) {
  switch (log_n) {
    case 9: return f(std::integral_constant<int, 9>{});
    case 10: return f(std::integral_constant<int, 10>{});
    case 11: return f(std::integral_constant<int, 11>{});
    case 12: return f(std::integral_constant<int, 12>{});
    case 13: return f(std::integral_constant<int, 13>{});
    case 14:
      if constexpr (sizeof(R) == 4) return f(std::integral_constant<int, 14>{});
      [[fallthrough]];
    default: return cudaErrorInvalidValue;
  }
}

template <class C, int LOGN>
constexpr size_t plane_smem() { return regs::Row<C, LOGN>::kPlane * sizeof(typename regs::Row<C, LOGN>::R); }

// The kernels of one row length and form: each that is touched is loaded, a third of a millisecond of
// the first workspace that a process creates (all of them, for any grid: 17 -> 28 ms).
template <class R>
static cudaError_t configure_rows(int log_n) {
  return with_row<R>(log_n, [](auto log) {
    constexpr int LOGN = decltype(log)::value;
    const auto limit = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_env_pairs<R, LOGN>, limit, (int)pairs_smem<R, LOGN>());
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_env_forward<R, LOGN>, limit, (int)plane_smem<cplx<R>, LOGN>());
    if constexpr (LOGN <= 13) {
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_env_inverse<R, LOGN>, limit, (int)plane_smem<double2, LOGN>());
    }
    return e;
  });
}

cudaError_t configure_env_modal_kernels(int n_to, bool mixed) {
  if (n_to > kMaxEnvelopeRowF64) {
    const int row = (int)(kMaxEnvelopeRowF64 * sizeof(double2));  // half a long FP64 row
    for (const void* k : {mixed ? (const void*)k_env_inverse_long32 : (const void*)k_env_inverse_long,
                          (const void*)k_env_forward_long, (const void*)k_env_nodes_long}) {
      const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, row);
      if (e != cudaSuccess) return e;
    }
    if (!mixed) return cudaSuccess;
  }
  const int log_n = 31 - __builtin_clz((unsigned)n_to);
  return mixed ? configure_rows<float>(log_n) : configure_rows<double>(log_n);
}

void row_twiddles(int n_to, const std::vector<double2>& tw, std::vector<double2>& outer,
                  std::vector<double2>& inner) {
  // Row's V, T, M and G (the same for either type)
  const int log_v = regs::default_log_v(31 - __builtin_clz((unsigned)n_to)), V = 1 << log_v, T = n_to / V, M = T, G = M / V;
  auto root = [&](long q) {  // exp(-2 pi i q / 2n), q < 2n
    double2 w = tw[q & (n_to - 1)];
    if (q >= n_to) w = make_double2(-w.x, -w.y);
    return w;
  };
  outer.resize((size_t)2 * n_to);
  for (int p = 0; p < 2; ++p)
    for (int f = 0; f < V; ++f)
      for (int t = 0; t < T; ++t) outer[((size_t)p * V + f) * T + t] = root((long)(2 * f + p) * t);
  inner.resize((size_t)V * G);
  for (int g = 0; g < V; ++g)
    for (int j = 0; j < G; ++j) inner[(size_t)g * G + j] = root((long)g * j * (2 * n_to / M));
}

template <class R>
cudaError_t launch_env_inverse(const EnvModalArgsT<R>& a, const RamanArgs* raman, cplx<R>* table, cudaStream_t s) {
  const int kernels = !raman ? 0 : a.n_components == 2 ? a.raman_kernels : 1;
  if (a.n_to > kMaxEnvelopeRowF64) {
    const size_t half = (size_t)a.n_to / 2 * sizeof(double2);
    if constexpr (sizeof(R) == 8) k_env_inverse_long<<<a.n_cols, kEnvThreads, half, s>>>(a);
    else k_env_inverse_long32<<<a.n_cols, kEnvThreads, half, s>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !raman) return e;
    e = launch_raman_spectrum(*raman, s);
    if (e != cudaSuccess || sizeof(R) == 8) return e;  // k_env_nodes_long reads the spectrum itself
    return with_row<R>(a.log_n_to, [&](auto log) {
      k_raman_table<R, decltype(log)::value><<<dim3(2 * a.n_to / 256, kernels), 256, 0, s>>>(a.raman_spectrum,
                                                                                           raman->scale, table);
      return cudaGetLastError();
    });
  }
  return with_row<R>(a.log_n_to, [&](auto log) {
    constexpr int LOGN = decltype(log)::value;
    if constexpr (LOGN <= 13)
      k_env_inverse<R, LOGN><<<a.n_cols + 2 * kernels, regs::Row<double2, LOGN>::T, plane_smem<double2, LOGN>(), s>>>(
          a, raman ? *raman : RamanArgs{}, table, 2 * kernels);
    return cudaGetLastError();
  });
}

template <class R>
cudaError_t launch_env_nodes(const EnvModalArgsT<R>& a, int n_nodes, cudaStream_t s) {
  if (!a.raman) {
    const size_t total = (size_t)n_nodes * a.n_to;
    k_env_kerr<R><<<(unsigned)std::min<size_t>((total + 255) / 256, 148 * 16), 256, 0, s>>>(a, n_nodes);
    return cudaGetLastError();
  }
  if (sizeof(R) == 8 && a.n_to > kMaxEnvelopeRowF64) {
    if constexpr (sizeof(R) == 8)
      k_env_nodes_long<<<n_nodes, kNodeThreads, (size_t)a.n_to / 2 * sizeof(double2), s>>>(a);
    return cudaGetLastError();
  }
  // Two nodes a CTA take three convolutions of the tensor response where one takes two, and twice the
  // outputs: with no more nodes than SMs a CTA each is the shorter chain.  49 nodes, FP64 rows of
  // 1 024: 40 -> 27 us; 64 of one component: 27 -> 18 us.  Of 169, more than SMs, two a CTA.
  const int per_cta = n_nodes <= 148 ? 1 : 2;
  return with_row<R>(a.log_n_to, [&](auto log) {
    constexpr int LOGN = decltype(log)::value;
    k_env_pairs<R, LOGN><<<(n_nodes + per_cta - 1) / per_cta, regs::Row<cplx<R>, LOGN>::T, pairs_smem<R, LOGN>(), s>>>(
        a, n_nodes, per_cta);
    return cudaGetLastError();
  });
}

template <class R>
cudaError_t launch_env_forward(const EnvModalArgsT<R>& a, cudaStream_t s) {
  if (sizeof(R) == 8 && a.n_to > kMaxEnvelopeRowF64) {
    if constexpr (sizeof(R) == 8)
      k_env_forward_long<<<a.n_cols, kEnvThreads, (size_t)a.n_to / 2 * sizeof(double2), s>>>(a);
    return cudaGetLastError();
  }
  return with_row<R>(a.log_n_to, [&](auto log) {
    constexpr int LOGN = decltype(log)::value;
    k_env_forward<R, LOGN><<<a.n_cols, regs::Row<cplx<R>, LOGN>::T, plane_smem<cplx<R>, LOGN>(), s>>>(a);
    return cudaGetLastError();
  });
}

template cudaError_t launch_env_inverse<double>(const EnvModalArgsT<double>&, const RamanArgs*, double2*, cudaStream_t);
template cudaError_t launch_env_inverse<float>(const EnvModalArgsT<float>&, const RamanArgs*, float2*, cudaStream_t);
template cudaError_t launch_env_nodes<double>(const EnvModalArgsT<double>&, int, cudaStream_t);
template cudaError_t launch_env_nodes<float>(const EnvModalArgsT<float>&, int, cudaStream_t);
template cudaError_t launch_env_forward<double>(const EnvModalArgsT<double>&, cudaStream_t);
template cudaError_t launch_env_forward<float>(const EnvModalArgsT<float>&, cudaStream_t);

}  // namespace sp
