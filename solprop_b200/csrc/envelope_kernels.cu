// The source evaluation on the envelope grid (complex time samples, c2c transforms) for a
// single modal column on a single node -- the generalised NLSE of a single-mode fibre:
// passes/transforms.py:31-84 and 190-233 (ifft / fft with the crop), responses.py:65-139
// (the analytic Kerr cubic), responses.py:218-498 (the Raman response as a doubled-grid
// convolution), the projection, all in one launch:
//
//   a <- ifft(pad(lab))                                   the envelope a(t), E = tau S a
//   H <- dt rfft(f_R sum_r h_r e^{-g_r t})                the damped Raman kernel, length 2 n_to
//   conv <- irfft(H rfft(|E|^2 / 2))[:n_to]               the convolution
//   spectrum <- crop(fft((W / tau)(Kerr + eps0 rho_R E conv) g(t)))
//
// The transforms are the register FFT of fft_regs.cuh, whose doubled row comes as two halves
// (even and odd bins): a cluster of four CTAs takes a half of the field's convolution each
// (ranks 0 and 1, both forming the envelope) and a half of the kernel's spectrum each (ranks 2
// and 3, meanwhile); the spectra and rank 1's half of the convolution cross by distributed
// shared memory, and rank 0 forms the polarisation and its spectrum.
//
// What bounds it: latency, four transforms in a chain, the instructions' own fetch included
// (the loop below keeps one copy of each transform's code).  4 096 samples, ncu: 36 us; 84 in one CTA's
// shared-memory radix-4 transforms, with the kernel's spectrum in the chain.
#include <cooperative_groups.h>

#include <type_traits>

#include "fft_regs.cuh"
#include "kernels.cuh"

namespace cg = cooperative_groups;

namespace sp {

namespace {

constexpr double kEps0 = 8.8541878188e-12;  // vacuum permittivity (F/m), CODATA 2022, as solprop.constants
constexpr int kRanks = 4;

}  // namespace

template <int LOGN>
using EnvelopeRow = regs::Row<double2, LOGN>;
template <int LOGN>
constexpr size_t envelope_smem() {
  return EnvelopeRow<LOGN>::N * sizeof(double2) + EnvelopeRow<LOGN>::kPlane * sizeof(double);
}

template <int LOGN>
__global__ void __cluster_dims__(kRanks, 1, 1) __launch_bounds__(EnvelopeRow<LOGN>::T)
    k_envelope_source(EnvelopeArgs a) {
  await_previous_kernel();
  using Row = EnvelopeRow<LOGN>;
  constexpr int n = Row::N, T = Row::T, V = Row::V;
  extern __shared__ __align__(16) unsigned char env_raw[];
  double2* stash = reinterpret_cast<double2*>(env_raw);  // the envelope; a kernel rank's spectrum
  double* plane = reinterpret_cast<double*>(stash + n);
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), t0 = threadIdx.x, half = rank & 1;
  const bool kernel = rank >= 2, raman = a.raman_terms > 0;
  if (!raman && rank > 0) return;  // uniform over the cluster: nothing is exchanged
  const StageScalarsDev& st = *a.stage;
  double2 x[V];
  if (kernel) {
    // the kernel's samples s and s + n, together for this half's bins
#pragma unroll 4
    for (int r = 0; r < V; ++r) {
      double k[2] = {0.0, 0.0};
      for (int q = 0; q < 2; ++q) {
        const int s = t0 + r * T + q * n;
        for (int c = 0; c < a.raman_terms; ++c)
          k[q] += a.raman_undamped[(size_t)c * 2 * n + s] * exp(-st.raman_rates[c] * ((double)s * a.dt));
      }
      plane[r * T + t0] = a.raman_fraction * (half ? k[0] - k[1] : k[0] + k[1]);  // each thread its own places
    }
#pragma unroll
    for (int r = 0; r < V; ++r) x[r] = make_double2(plane[r * T + t0], 0.0);
  } else {
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const int j = a.fine_to_coarse[Row::bin(t0, e)];
      x[e] = j >= 0 ? a.lab[j] : make_double2(0.0, 0.0);
    }
  }
  const double es = st.taper * a.synthesis / (double)n;  // E = tau S a; scipy's ifft carries 1 / n_to
  const int last = raman ? 1 : 0;
#pragma unroll 1
  for (int it = 0; it <= last; ++it) {
    const bool at_half = raman && half;  // the odd bins' transforms
    if (!kernel) Row::inverse(x, plane, a.outer, a.inner, it == 1 ? half : 0);
    if (!kernel && it == 0) {  // the envelope, then its drive |E|^2 / 2
#pragma unroll
      for (int r = 0; r < V; ++r) {
        x[r] = cscale(es, x[r]);
        stash[r * T + t0] = x[r];
        if (raman) x[r] = make_double2(0.5 * (x[r].x * x[r].x + x[r].y * x[r].y), 0.0);
      }
    }
    if (it == 0 && at_half) {
#pragma unroll
      for (int r = 0; r < V; ++r) x[r] = regs::rotate64<false>(x[r], r * (32 / V));
    }
    if (it == last) {
      if (raman) {
        if (rank == 1) {  // its half of the convolution, over the envelope it needs no more
#pragma unroll
          for (int r = 0; r < V; ++r)
            reinterpret_cast<double*>(stash)[r * T + t0] = regs::rotate64<true>(x[r], r * (32 / V)).x;
        }
        cluster.sync();
        if (rank == 0) {
          const double* other = reinterpret_cast<const double*>(cluster.map_shared_rank(stash, 1));
#pragma unroll
          for (int r = 0; r < V; ++r) x[r].x += other[r * T + t0];
        }
        cluster.sync();  // rank 1 stays until it is read
        if (rank > 0) return;
      }
      // the polarisation, gated and projected
      const double factor = a.kerr ? a.kerr_coefficient * st.kerr_density : 0.0;
      const double raman_scale = raman ? kEps0 * st.raman_density : 0.0, proj = a.projection / st.taper;
#pragma unroll
      for (int r = 0; r < V; ++r) {
        const double2 e = stash[r * T + t0];
        const double conv = raman_scale * x[r].x;
        double2 p = make_double2(0.0, 0.0);
        if (a.kerr) {
          const double mod = e.x * e.x + e.y * e.y;
          p = cscale(factor, cadd(cscale(a.kerr_self * mod, e), cscale(a.kerr_conjugate, cmul(cmul(e, e), cconj(e)))));
        }
        if (raman) p = cadd(p, cscale(conv, e));
        x[r] = cscale(proj * a.t_window[t0 + r * T], p);
      }
    }
    Row::forward(x, plane, a.outer, a.inner, it == 0 && at_half);
    if (it < last) {
      if (kernel) {
        const double f = a.dt / (2.0 * (double)n);  // the convolution's 1 / 2n inside
#pragma unroll
        for (int e = 0; e < V; ++e) stash[e * T + t0] = cscale(f, x[e]);
      }
      cluster.sync();
      if (!kernel) {
        const double2* h = cluster.map_shared_rank(stash, 2 + half);
#pragma unroll
        for (int e = 0; e < V; ++e) x[e] = cmul(x[e], h[e * T + t0]);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < V; ++e) {
    const int j = a.fine_to_coarse[Row::bin(t0, e)];
    if (j >= 0) a.spectra[j] = x[e];
  }
}

template <class F>
static cudaError_t with_envelope_row(int log_n, F&& f) {
  switch (log_n) {
    case 9: return f(std::integral_constant<int, 9>{});
    case 10: return f(std::integral_constant<int, 10>{});
    case 11: return f(std::integral_constant<int, 11>{});
    case 12: return f(std::integral_constant<int, 12>{});
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_envelope(const EnvelopeArgs& a, cudaStream_t stream) {
  return with_envelope_row(a.log_n_to, [&](auto log) {
    constexpr int LOGN = decltype(log)::value;
    return launch_chained(k_envelope_source<LOGN>, kRanks, EnvelopeRow<LOGN>::T, envelope_smem<LOGN>(), 1, stream, a);
  });
}

cudaError_t configure_envelope_kernels(int n_to) {
  return with_envelope_row(31 - __builtin_clz((unsigned)n_to), [](auto log) {
    constexpr int LOGN = decltype(log)::value;
    return cudaFuncSetAttribute(k_envelope_source<LOGN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)envelope_smem<LOGN>());
  });
}

}  // namespace sp
