// fft_gen.cuh -- batched FP64 FFTs of any length in shared memory, out of
// place between two buffers, for the lengths without a compile-time kernel.
//
// NB = 1 << lg sequences side by side, element (e, b) at buf[(e << lg) + b],
// natural order in and out (Stockham's decimation in frequency): the pass of
// radix R and span s (the product of the radices before it) takes, for each
// t = q + s p < n / R (q < s), the elements t + r n / R, transforms them over
// r, multiplies output k by W_n^(s p k) and writes it to q + s (R p + k).
// Radices up to SPH_GEN_RADIX are one register butterfly per thread.  A larger
// prime is split over its outputs: a thread computes the pair (k, R - k) from
// cos and sin sums over the R inputs, which R - 1 FMAs per output cost, but
// (R + 1) / 2 threads share a butterfly (one thread per butterfly, with its
// inputs and outputs in local memory, measured 221 us for the 2 29 radial
// derivative of 528 columns, of which two passes over 32 columns were done by
// 64 threads).  The passes of one length are chosen on the host
// (fft_gen_plan): as few as possible, each a round trip through shared memory.
#pragma once
#include "fft3.cuh"
#include "sph_internal.cuh"

namespace fg {

// t / s for t < 2^16, s < 2^13 (mul = ceil(2^32 / s); s = 1 has no 32-bit mul)
__device__ __forceinline__ int div_span(int t, int s, unsigned mul) { return s == 1 ? t : (int)__umulhi((unsigned)t, mul); }

template <int SG>
__device__ __forceinline__ double2 tw_gen(const double2* __restrict__ tw, int e) {
  double2 w = __ldg(tw + e);
  if (SG > 0) w.y = -w.y;
  return w;
}

// the outputs of butterfly t (column b) of a pass
template <int R, int SG>
__device__ __forceinline__ void put(double2* dst, const double2 (&v)[R], int t, int b, const GenPass& g, int lg,
                                    const double2* __restrict__ tw) {
  const int p = div_span(t, g.s, g.mul), e = p * g.s;
  double2* o = dst + ((t - e + R * e) << lg) + b;
  o[0] = v[0];
#pragma unroll
  for (int k = 1; k < R; ++k) o[(g.s * k) << lg] = e ? ct::mul(v[k], tw_gen<SG>(tw, e * k)) : v[k];
}

template <int R, int SG>
__device__ __noinline__ void pass_reg(const double2* src, double2* dst, int n, GenPass g, int lg,
                                      const double2* __restrict__ tw) {
  const int nt = n / R;
  for (int it = threadIdx.x; it < nt << lg; it += blockDim.x) {
    const int b = it & ((1 << lg) - 1), t = it >> lg;
    double2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src[((t + r * nt) << lg) + b];
    ct::RD<double2, R, SG>::run(v);
    put<R, SG>(dst, v, t, b, g, lg, tw);
  }
}

// an odd prime radix above SPH_GEN_RADIX
template <int SG>
__device__ __noinline__ void pass_prime(const double2* src, double2* dst, int n, GenPass g, int lg,
                                        const double2* __restrict__ tw) {
  const int R = g.R, nt = n / R, H = (R - 1) / 2;
  for (int it = threadIdx.x; it < (nt * (H + 1)) << lg; it += blockDim.x) {
    const int b = it & ((1 << lg) - 1), u = it >> lg, k = u / nt, t = u - k * nt;
    const double2* x = src + (t << lg) + b;
    const int step = nt << lg;
    const int p = div_span(t, g.s, g.mul), e = p * g.s;
    double2* o = dst + ((t - e + R * e) << lg) + b;
    double2 a = x[0], c = make_double2(0.0, 0.0);
    int idx = 0;
    for (int j = 1; j <= H; ++j) {
      const double2 u1 = x[j * step], u2 = x[(R - j) * step];
      idx += k;
      if (idx >= R) idx -= R;
      const double2 w = __ldg(tw + idx * nt);  // (cos, -sin) of 2 pi j k / R
      a.x += w.x * (u1.x + u2.x);
      a.y += w.x * (u1.y + u2.y);
      c.x -= w.y * (u1.x - u2.x);
      c.y -= w.y * (u1.y - u2.y);
    }
    if (k == 0) {
      o[0] = a;
    } else {
      const double2 ic = ct::mul_si(c, SG);
      const double2 y1 = ct::add(a, ic), y2 = ct::sub(a, ic);
      o[(g.s * k) << lg] = e ? ct::mul(y1, tw_gen<SG>(tw, e * k)) : y1;
      o[(g.s * (R - k)) << lg] = e ? ct::mul(y2, tw_gen<SG>(tw, e * (R - k))) : y2;
    }
  }
}

#define SPH_GEN_RADICES(X) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13)

// Passes [first, last) of the list g on buffer a (b is the other one), with a
// barrier after each; returns the buffer that holds the result.
template <int SG>
__device__ __forceinline__ double2* run(double2* a, double2* b, int n, const GenPass* g, int first, int last, int lg,
                                        const double2* __restrict__ tw) {
  for (int ip = first; ip < last; ++ip) {
    switch (g[ip].R) {
#define CASE(r) \
  case r: pass_reg<r, SG>(a, b, n, g[ip], lg, tw); break;
      SPH_GEN_RADICES(CASE)
#undef CASE
      default: pass_prime<SG>(a, b, n, g[ip], lg, tw); break;
    }
    __syncthreads();
    double2* t = a;
    a = b;
    b = t;
  }
  return a;
}

}  // namespace fg

// The passes of a length-n transform: the primes up to SPH_GEN_RADIX grouped
// into register radices with the least cost (a pass moves every element
// through shared memory once, about 8 FMAs' worth per element, beside the
// butterfly's own), larger primes (at most 64) alone.  False: no plan.
// Fixed arrays only: sph_derivr_noalloc, which allocates no host memory,
// plans its transforms here too.
static inline bool fft_gen_plan(int n, FftDesc& fd) {
  const int cost[SPH_GEN_RADIX + 1] = {0, 0, 2, 4, 3, 6, 6, 8, 5, 8, 9, 12, 8, 14};
  int primes[SPH_GEN_PASSES], nprimes = 0, small = n;
  for (int q = SPH_GEN_RADIX + 1; q <= 64; ++q)  // ascending, so a composite q no longer divides
    for (; small % q == 0 && q % 2 && q % 3 && q % 5 && q % 7; small /= q) {
      if (nprimes == SPH_GEN_PASSES) return false;
      primes[nprimes++] = q;
    }
  // least cost over the divisors of the rest, built up from 1
  constexpr int MAXDIV = 256;
  int divs[MAXDIV], best[MAXDIV], take[MAXDIV], nd = 0;
  for (int d = 1; d <= small; ++d)
    if (small % d == 0) {
      if (nd == MAXDIV) return false;
      divs[nd] = d;
      best[nd] = d == 1 ? 0 : -1;
      take[nd++] = 0;
    }
  for (int i = 1; i < nd; ++i)
    for (int j = 0; j < i; ++j) {
      const int R = divs[i] / divs[j];
      if (divs[i] % divs[j] || R > SPH_GEN_RADIX || best[j] < 0) continue;
      if (best[i] < 0 || best[j] + 8 + cost[R] < best[i]) {
        best[i] = best[j] + 8 + cost[R];
        take[i] = R;
      }
    }
  if (best[nd - 1] < 0) return false;
  fd.ng = 0;
  for (int i = nd - 1; divs[i] > 1;) {
    if (fd.ng == SPH_GEN_PASSES) return false;
    fd.gf[fd.ng++].R = take[i];
    const int d = divs[i] / take[i];
    while (divs[i] != d) --i;
  }
  for (int i = 0; i < nprimes; ++i) {
    if (fd.ng == SPH_GEN_PASSES) return false;
    fd.gf[fd.ng++].R = primes[i];
  }
  for (int i = 0; i < fd.ng; ++i) fd.gl[i].R = fd.gf[fd.ng - 1 - i].R;
  for (GenPass* g : {fd.gf, fd.gl})
    for (int i = 0, s = 1; i < fd.ng; s *= g[i++].R) {
      g[i].s = s;
      g[i].mul = s > 1 ? (unsigned)(((1ull << 32) + s - 1) / s) : 0u;
    }
  return true;
}
