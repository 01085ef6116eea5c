// k_zfft.cu -- radial (z) transforms on the (lm, z) spectral layout.
//
// One CTA owns LB consecutive lm columns and all nz rows in shared memory
// (row-major: element (k, c) at sm[k*LB + c]), so every global access is a
// contiguous LB*16-byte run of one row.  The reference's steps, each a
// separate pass over HBM there, are fused here into one read and one write:
//   fftp1d_real_to_complex_z (src/sphp/sphp_sca.F90:332-397): continuation
//     of the last C rows from rows 1..d and N-d+1..N (sphp_sca.F90:369-381,
//     same summation order), DFT sign -1, divide by nz;
//   fftp1d_complex_to_real_z (sphp_sca.F90:495-530): DFT sign +1;
//   derivr_r (src/pseudo/pseudospec_hd.f90:101-135): forward, (i kz)^p,
//     inverse, without the reference's temporary copy;
//   fc_filter_r (pseudospec_hd.f90:443-467) and dlr (pseudospec_hd.f90:254-288)
//     likewise.
// Three kernels do the transform in shared memory: zfft2_kernel for the
// lengths N = R1 R2 with a two-step register split (every compile-time
// length up to 256: two shared-memory passes, results stored from
// registers), zfft_kernel with compile-time radix passes for nz 512, and
// zfft_gen_kernel with the out-of-place passes of fft_gen.cuh for every
// other length.  Batches run the
// forward transforms of all their problems with one z length as one launch
// of zfft2_group_kernel (the same body, one column block per CTA).
#include <algorithm>
#include <mutex>

#include "fft3.cuh"
#include "fft_ct.cuh"
#include "fft_gen.cuh"

namespace {

constexpr int ZTHREADS = 256;
constexpr int ZMAXCOL = 4096;  // LB*nz complex values per CTA (64 KB)

template <int IO>
struct ZIo {
  static constexpr bool FIN = IO == ZIO_FF || IO == ZIO_FD, FOUT = IO == ZIO_FF || IO == ZIO_DF;
};

struct ZArgs {
  const void* in;
  void* out;
  int nlm, nz, N, C, d, LB, order;
  const double* dir;      // C x d column-major
  const double2* kfac;    // (i kz)^order, nz entries
  const double* filt;     // nz
  const double* zinv2;    // nz
  const int* ell;         // nlm
  FftDesc fd;
  // the passes of the nonlinear step (Z_POT, Z_RHS, Z_DLADD)
  ZNlArgs nl;
  const double *z, *zinv;  // r, 1/r
  bool digits;  // general lengths: a mixed plan's passes of fft_engine.cuh
  int nbuf;     // buffers of a general length: one where every radix is done in place
};

// modes that keep the whole input column (every row) beside the transform's
constexpr bool zkeep(int mode) { return mode == Z_DLR || mode == Z_POT || mode == Z_DLADD; }

// The output of row r, column lm (at idx) of a spectral mode from the
// transformed value x and the kept input o.
template <int MODE, int IO>
__device__ __forceinline__ void zspectral_store(const ZArgs& a, int r, int lm, size_t idx, double2 x, double2 o);

// 16-byte global -> shared copy that lands asynchronously; src_bytes 0
// writes zeros (src is then not read but must be a valid address)
__device__ __forceinline__ void cp_async16z(void* dst, const void* src, int src_bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}

// column element (row r, column lm) of the input, widened to FP64
template <int IO>
__device__ __forceinline__ double2 zin(const ZArgs& a, size_t idx) {
  if constexpr (ZIo<IO>::FIN) {
    const float2 v = __ldg(static_cast<const float2*>(a.in) + idx);
    return make_double2((double)v.x, (double)v.y);
  } else {
    return __ldg(static_cast<const double2*>(a.in) + idx);
  }
}

// one column element into shared memory: by cp.async when the input is
// FP64, else loaded, widened and stored; zero past nlm
template <int IO>
__device__ __forceinline__ void zload(const ZArgs& a, double2* dst, size_t idx, bool in) {
  if constexpr (ZIo<IO>::FIN) {
    *dst = in ? zin<IO>(a, idx) : make_double2(0.0, 0.0);
  } else {
    const double2* src = static_cast<const double2*>(a.in);
    cp_async16z(dst, in ? src + idx : src, in ? 16 : 0);
  }
}

template <int IO>
__device__ __forceinline__ void zstore(const ZArgs& a, size_t idx, double2 v) {
  if constexpr (ZIo<IO>::FOUT)
    static_cast<float2*>(a.out)[idx] = make_float2((float)v.x, (float)v.y);
  else
    static_cast<double2*>(a.out)[idx] = v;
}

template <int MODE, int IO>
__device__ __forceinline__ void zspectral_store(const ZArgs& a, int r, int lm, size_t idx, double2 x, double2 o) {
  if constexpr (MODE == Z_DLR || MODE == Z_DLADD) {
    // b = b + z^-2 * (-l(l+1) a)   (laplang, multr(-2), saxpby_c)
    const double lf = -(double)(a.ell[lm] * (a.ell[lm] + 1));
    const double zi = a.zinv2[r];
    x.x = x.x + zi * (lf * o.x);
    x.y = x.y + zi * (lf * o.y);
  }
  if constexpr (MODE == Z_DLADD) {
    x = cscale(x, a.nl.nu);
    if (!a.nl.by_r || r < a.N) {
      const double f = a.nl.by_r ? a.z[r] : 1.0;
      const double2 v = __ldg(a.nl.add + idx);
      x = make_double2(f * v.x + x.x, f * v.y + x.y);
    }
    if (a.nl.base) {
      const double2 v = __ldg(a.nl.base + idx);
      x = make_double2(v.x + a.nl.c * x.x, v.y + a.nl.c * x.y);
    }
  }
  if constexpr (MODE == Z_RHS) {
    if (r < a.N) x = csub(x, __ldg(a.nl.q + idx));
  }
  if constexpr (MODE == Z_POT) {
    const double zi = a.zinv[r];
    a.nl.q[idx] = cscale(o, a.zinv2[r] * (double)(a.ell[lm] * (a.ell[lm] + 1)));
    if (a.nl.t) a.nl.t[idx] = cscale(o, zi);
    x = cscale(x, zi);
  }
  zstore<IO>(a, idx, x);
}

template <int MODE, int CTN, int IO>
__global__ void __launch_bounds__(ZTHREADS) zfft_kernel(ZArgs a) {
  grid_dependency_wait();
  extern __shared__ double2 sm[];
  const int LB = a.LB, nz = a.nz, nlm = a.nlm;
  const int lm0 = blockIdx.x * LB;
  const int tid = threadIdx.x;
  const bool cont = (MODE != Z_INV) && a.C > 0;
  const int nload = cont ? a.N : nz;
  double2* orig = sm + (size_t)LB * nz;  // D_l keeps the input column for the l(l+1)/r^2 term

  const int* __restrict__ rev = a.fd.rev;
  // every copy of the slab is in flight at once (no registers held); columns
  // past nlm are zero-filled
  for (int idx = tid; idx < nload * LB; idx += ZTHREADS) {
    int r = idx / LB, c = idx - r * LB;
    int lm = lm0 + c;
    // the inverse transform takes its input in digit-reversed order
    zload<IO>(a, sm + (MODE == Z_INV ? __ldg(rev + r) : r) * LB + c, (size_t)r * nlm + lm, lm < nlm);
  }
  if (MODE == Z_DLR) {
    for (int idx = tid; idx < nz * LB; idx += ZTHREADS) {
      int r = idx / LB, c = idx - r * LB;
      int lm = lm0 + c;
      zload<IO>(a, orig + idx, (size_t)r * nlm + lm, lm < nlm);
    }
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();

  if (cont) {
    // inout(n-C+ii) = sum_jj dir(ii,jj) inout(n-C-d+jj) + dir(C-ii+1,jj) inout(d-jj+1)
    const int C = a.C, d = a.d, N = a.N;
    for (int idx = tid; idx < C * LB; idx += ZTHREADS) {
      int ii = idx / LB, c = idx - ii * LB;  // ii is 0-based
      double2 acc;
      {
        double wr = __ldg(a.dir + ii), wl = __ldg(a.dir + (C - 1 - ii));
        double2 xr = sm[(N - d) * LB + c], xl = sm[(d - 1) * LB + c];
        acc = make_double2(wr * xr.x + wl * xl.x, wr * xr.y + wl * xl.y);
      }
      for (int jj = 1; jj < d; ++jj) {
        double wr = __ldg(a.dir + ii + C * jj), wl = __ldg(a.dir + (C - 1 - ii) + C * jj);
        double2 xr = sm[(N - d + jj) * LB + c], xl = sm[(d - 1 - jj) * LB + c];
        acc.x = (acc.x + wr * xr.x) + wl * xl.x;
        acc.y = (acc.y + wr * xr.y) + wl * xl.y;
      }
      sm[(N + ii) * LB + c] = acc;
    }
    __syncthreads();
  }

  const ct::Geo<CTN, 0, false> g{LB, 1, LB};
  if (MODE == Z_INV) ct::dit<double2, CTN, CTN>(sm, g, a.fd.twp, +1);
  else ct::dif<double2, CTN, CTN>(sm, g, a.fd.twp, -1);

  if (MODE == Z_DERIV || MODE == Z_FILTER || MODE == Z_DLR) {
    // spectral multiply in place (frequency k sits at row rev[k]), then back
    for (int idx = tid; idx < nz * LB; idx += ZTHREADS) {
      int k = idx / LB, c = idx - k * LB;
      int o = __ldg(rev + k) * LB + c;
      double2 v = div_nz(sm[o], nz);
      if (MODE == Z_FILTER) v = cscale(v, a.filt[k]);
      else v = cmul(a.kfac[k], v);
      sm[o] = v;
    }
    __syncthreads();
    ct::dit<double2, CTN, CTN>(sm, g, a.fd.twp, +1);
  }

  for (int idx = tid; idx < nz * LB; idx += ZTHREADS) {
    int r = idx / LB, c = idx - r * LB;
    int lm = lm0 + c;
    if (lm >= nlm) continue;
    double2 v;
    if (MODE == Z_FWD) {
      v = div_nz(sm[__ldg(rev + r) * LB + c], nz);
    } else {
      v = sm[idx];
    }
    if (MODE == Z_DLR) {
      // b = b + z^-2 * (-l(l+1) a)   (laplang, multr(-2), saxpby_c)
      double lf = -(double)(a.ell[lm] * (a.ell[lm] + 1));
      double2 o = orig[idx];
      double zi = a.zinv2[r];
      v.x = v.x + zi * (lf * o.x);
      v.y = v.y + zi * (lf * o.y);
    }
    zstore<IO>(a, (size_t)r * nlm + lm, v);
  }
}

// Lengths with a two-step split N = R1 R2 (ct::split2_r1, fft3.cuh): every
// mode, max(R1, R2) threads per column, the column slab in shared memory as
// in zfft_kernel (same loads and continuation, the inverse's input in
// natural order).  A plain transform is the two register steps, its results
// stored from registers; the spectral modes run the forward steps, multiply
// in registers and go back from there (dft2_back1/2: one more exchange).
// About 128 threads per CTA (8 columns at nz 96 and above), 80 registers: the
// kernels wait on loads and barriers, not on HBM or the FP64 pipe (29% busy
// in the derivative), so many small CTAs overlap best.  Derivative and D_l of
// 32896 columns: nz 96 55 and 64 -> 36 and 48 us, nz 128 53 and 66 -> 43 and
// 64 us, against the spectrum put back in natural order between two full
// splits, 128-148 registers and 16 columns.  The modes that keep the input
// column take the registers of the CTAs their shared memory lets share an SM
// (four at nz 192, three at 256), else they spill: D_l of 73920 columns nz 192
// 232 -> 196 us (217 before the exchange from registers), nz 256 292 -> 194
// (261).
__host__ __device__ constexpr int z2_lb(int nz) {
  int lb = 32;
  while (lb > 8 && lb * ct::split2_tpc(nz) > 128) lb >>= 1;
  return lb;
}
template <int MODE, int NZ, int TPC>
struct Z2Geo {
  static constexpr int LB = z2_lb(NZ), THREADS = LB * TPC;
  static constexpr bool PLAIN = MODE == Z_FWD || MODE == Z_INV;
  static constexpr int RPT = 84;
  static constexpr int SMEM = LB * NZ * (int)sizeof(double2) * (zkeep(MODE) ? 2 : 1);
  static constexpr int MINB = std::max(1, std::min(65536 / (THREADS * RPT), 227 * 1024 / (SMEM + 1024)));
};

// column block blk of the spectra a describes
template <int MODE, int R1, int R2, int IO>
__device__ __forceinline__ void zfft2_body(const ZArgs& a, int blk) {
  constexpr int NZ = R1 * R2, TPC = R1 > R2 ? R1 : R2;
  using GZ = Z2Geo<MODE, NZ, TPC>;
  constexpr bool PLAIN = GZ::PLAIN;
  constexpr int SG = MODE == Z_INV ? 1 : -1;  // first transform's sign
  constexpr int LB = GZ::LB, nthreads = GZ::THREADS;
  extern __shared__ double2 sm[];
  const int nlm = a.nlm, tid = threadIdx.x, lm0 = blk * LB;
  const bool cont = MODE != Z_INV && a.C > 0;
  const int nload = cont ? a.N : NZ;
  constexpr bool KEEP = zkeep(MODE);
  double2* in = KEEP ? sm + (size_t)LB * NZ : sm;
  for (int idx = tid; idx < (KEEP ? NZ : nload) * LB; idx += nthreads) {
    const int r = idx / LB, c = idx - r * LB, lm = lm0 + c;
    zload<IO>(a, in + idx, (size_t)r * nlm + lm, lm < nlm);
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  if constexpr (MODE == Z_RHS)  // r x, each thread the elements it copied
    for (int idx = tid; idx < nload * LB; idx += nthreads) sm[idx] = cscale(sm[idx], a.z[idx / LB]);
  __syncthreads();
  if (cont) {  // as in zfft_kernel
    const int C = a.C, d = a.d, N = a.N;
    for (int idx = tid; idx < C * LB; idx += nthreads) {
      const int ii = idx / LB, c = idx - ii * LB;
      sm[(N + ii) * LB + c] = fc_cont_elem(a.dir, C, d, N, ii, in + c, LB);
    }
    __syncthreads();
  }
  const int c = tid % LB, h = tid / LB, lm = lm0 + c;
  double2* col = sm + c;
  if constexpr (KEEP) {
    // step 1 with the physical rows from the kept column
    if (h < R2) {
      double2 w[R1];
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) {
        const int r = h + R2 * n1;
        w[n1] = r < nload ? in[r * LB + c] : col[r * LB];
      }
      ct::dft2_put1<R1, R2, SG>(w, col, LB, h, a.fd.tw);
    }
  } else {
    ct::dft2_step1<R1, R2, SG>(col, LB, h, a.fd.tw);
  }
  __syncthreads();
  double2 v[R2];
  ct::dft2_step2<R1, R2, SG>(col, LB, h, v);
  if constexpr (PLAIN) {
    if (h < R1 && lm < nlm) {
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2)
        zstore<IO>(a, (size_t)(h + R1 * k2) * nlm + lm, MODE == Z_FWD ? div_nz(v[k2], NZ) : v[k2]);
    }
  } else {
    // X[k] / nz times (i kz)^p or the filter, k = h + R1 k2, in registers, and back
    if (h < R1) {
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) {
        const int k = h + R1 * k2;
        const double2 x = div_nz(v[k2], NZ);
        v[k2] = MODE == Z_FILTER ? cscale(x, a.filt[k]) : cmul(a.kfac[k], x);
      }
    }
    ct::dft2_back1<R1, R2, 1>(v, col, LB, h, a.fd.tw);
    __syncthreads();
    double2 w[R1];
    ct::dft2_back2<R1, R2, 1>(col, LB, h, w);
    if (h < R2 && lm < nlm) {
#pragma unroll
      for (int b = 0; b < R1; ++b) {
        const int r = h + R2 * b;
        zspectral_store<MODE, IO>(a, r, lm, (size_t)r * nlm + lm, w[b], KEEP ? in[r * LB + c] : w[b]);
      }
    }
  }
}

template <int MODE, int R1, int R2, int IO>
__global__ void __launch_bounds__(Z2Geo<MODE, R1 * R2, (R1 > R2 ? R1 : R2)>::THREADS,
                                  Z2Geo<MODE, R1 * R2, (R1 > R2 ? R1 : R2)>::MINB) zfft2_kernel(ZArgs a) {
  grid_dependency_wait();
  zfft2_body<MODE, R1, R2, IO>(a, blockIdx.x);
}

// The same over the spectra of several plans with one z length (batches):
// job j owns the CTAs prefix[j] .. prefix[j+1]-1, one column block each.
template <int MODE, int R1, int R2, int IO>
__global__ void __launch_bounds__(Z2Geo<MODE, R1 * R2, (R1 > R2 ? R1 : R2)>::THREADS,
                                  Z2Geo<MODE, R1 * R2, (R1 > R2 ? R1 : R2)>::MINB)
    zfft2_group_kernel(const ZArgs* __restrict__ jobs, const int* __restrict__ prefix, int njobs) {
  grid_dependency_wait();
  int lo = 0, hi = njobs - 1;  // last job whose first CTA is <= blockIdx.x
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(prefix + mid) <= (int)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  zfft2_body<MODE, R1, R2, IO>(jobs[lo], (int)blockIdx.x - __ldg(prefix + lo));
}

// Lengths without a compile-time transform: the slab in natural order, the
// out-of-place passes of fft_gen.cuh between two buffers (a third keeps the
// D_l input), then one store.  Bound by the latency of the passes where a
// call has few columns and by shared memory where it has many.  Derivative of
// 528 columns at nz 58 (2 29) and 33 (3 11): 7.1 and 6.3 us, against 221 and
// 42 us with one thread per butterfly in place and 32 columns per CTA; nz 90,
// 14706 columns, plain: 19-27 against 52-59 us.
//
// DIGITS: the decimation-in-frequency and -in-time passes of fft_engine.cuh
// instead, the spectrum in digit-reversed order between them.  Wide slabs of
// some lengths take these (launch_gen), and mixed plans on FP64 arrays: the
// fp32 steps after a z transform round, and a forward continuation (weights up
// to 3.7e3) amplifies what a last-bit change flips there, so another order of
// the FP64 sums moves their results by 3e-6, and a run on a mixed plan would
// not repeat on another release of the library.
template <int MODE, int IO, bool DIGITS>
__global__ void __launch_bounds__(ZTHREADS, DIGITS ? 4 : 2) zfft_gen_kernel(ZArgs a, int lg) {
  grid_dependency_wait();
  extern __shared__ double2 sm[];
  const int LB = 1 << lg, nz = a.nz, nlm = a.nlm, lm0 = blockIdx.x << lg, tid = threadIdx.x;
  const bool cont = MODE != Z_INV && a.C > 0;
  const int nload = cont ? a.N : nz, total = nz << lg;
  constexpr bool KEEP = zkeep(MODE);
  double2* orig = sm + a.nbuf * total;
  const int* __restrict__ rev = a.fd.rev;
  // slot of frequency k
  auto slot = [&](int k) { return DIGITS ? __ldg(rev + k) : k; };
  for (int idx = tid; idx < (KEEP ? total : nload << lg); idx += ZTHREADS) {
    const int r = idx >> lg, c = idx & (LB - 1), lm = lm0 + c;
    const int to = MODE == Z_INV ? (slot(r) << lg) + c : idx;
    zload<IO>(a, (KEEP ? orig : sm) + to, (size_t)r * nlm + lm, lm < nlm);
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  // each thread the elements it copied: the transform's copy of a kept
  // column, or r x
  if constexpr (KEEP || MODE == Z_RHS)
    for (int idx = tid; idx < nload << lg; idx += ZTHREADS)
      sm[idx] = KEEP ? orig[idx] : cscale(sm[idx], a.z[idx >> lg]);
  __syncthreads();
  if (cont) {  // as in zfft_kernel
    for (int idx = tid; idx < a.C << lg; idx += ZTHREADS) {
      const int ii = idx >> lg, c = idx & (LB - 1);
      sm[((a.N + ii) << lg) + c] = fc_cont_elem(a.dir, a.C, a.d, a.N, ii, sm + c, LB);
    }
    __syncthreads();
  }
  constexpr int SG = MODE == Z_INV ? 1 : -1;  // first transform's sign
  const FftGeom g{nz, LB, 1, LB, 0, false};
  double2* x;
  if constexpr (!DIGITS) x = fg::run<SG>(sm, sm + total, nz, a.fd.gf, 0, a.fd.ng, lg, a.fd.tw);
  else if constexpr (MODE == Z_INV) x = fft_dit2(sm, sm + total, a.fd, g, 1);
  else x = fft_dif2(sm, sm + total, a.fd, g, -1);
  if constexpr (MODE != Z_FWD && MODE != Z_INV) {
    for (int idx = tid; idx < total; idx += ZTHREADS) {
      const int k = idx >> lg, o = (slot(k) << lg) + (idx & (LB - 1));
      const double2 v = div_nz(x[o], nz);
      x[o] = MODE == Z_FILTER ? cscale(v, a.filt[k]) : cmul(a.kfac[k], v);
    }
    __syncthreads();
    double2* y = x == sm ? sm + total : sm;
    if constexpr (DIGITS) x = fft_dit2(x, y, a.fd, g, 1);
    else x = fg::run<1>(x, y, nz, a.fd.gf, 0, a.fd.ng, lg, a.fd.tw);
  }
  for (int idx = tid; idx < total; idx += ZTHREADS) {
    const int r = idx >> lg, c = idx & (LB - 1), lm = lm0 + c;
    if (lm >= nlm) continue;
    const size_t o = (size_t)r * nlm + lm;
    if constexpr (MODE == Z_FWD) zstore<IO>(a, o, div_nz(x[(slot(r) << lg) + c], nz));
    else if constexpr (MODE == Z_INV) zstore<IO>(a, o, x[idx]);
    else zspectral_store<MODE, IO>(a, r, lm, o, x[idx], KEEP ? orig[idx] : x[idx]);
  }
}

// Columns per CTA of zfft_gen_kernel where the plan sets none: the default
// slab (32 KB), halved down to 4 columns while the grid has fewer than two
// CTAs for each of a B200's 148 SMs (a 528-column derivative at nz 58 then has 132 CTAs, not 17).
int zgen_lb(int nz, int nlm) {
  int lb = 64;
  while (lb > 1 && lb * nz > ZMAXCOL / 2) lb >>= 1;
  while (lb > 4 && (nlm + lb - 1) / lb < 2 * 148) lb >>= 1;
  return lb;
}

// Shared memory of a zfft_gen_kernel CTA at most, so that two share an SM:
// wider slabs (tuned widths) are cut to what fits.  D_l of a mixed plan, 8256
// columns, nz 400 at 8 columns: 407 us uncut, 239 cut to 4; nz 120 at 32
// columns, derivative, 75 and 53 (345 and 60 with the in-place passes of one
// thread per butterfly).
constexpr size_t ZGEN_SMEM = 112 * 1024;

template <int MODE, int IO, bool DIGITS>
int launch_gen_as(const ZArgs& a, cudaStream_t st) {
  static DeviceOnce once;
  if (!once.run([] {
        return cudaFuncSetAttribute(zfft_gen_kernel<MODE, IO, DIGITS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    200 * 1024) == cudaSuccess &&
               cudaFuncSetAttribute(zfft_gen_kernel<MODE, IO, DIGITS>,
                                    cudaFuncAttributePreferredSharedMemoryCarveout, 100) == cudaSuccess;
      }))
    return SPH_ECUDA;
  int lg = 0;
  while ((1 << lg) < a.LB) ++lg;
  const size_t col = (size_t)a.nz * sizeof(double2) * (a.nbuf + zkeep(MODE));
  while (lg > 0 && (col << lg) > ZGEN_SMEM) --lg;
  launch_dependent(zfft_gen_kernel<MODE, IO, DIGITS>, (a.nlm + (1 << lg) - 1) >> lg, ZTHREADS, col << lg, st, a, lg);
  SPH_LAUNCH_OK();
  return SPH_OK;
}

// The in-place passes (DIGITS) also where two buffers of a tuned slab would
// have to be cut, every radix is 2, 3, 4 or 8 and there are no more passes:
// one buffer keeps the columns (FP64 derivative, nz 1024 at 4 columns: 8256
// columns 247 us uncut, 206 in place; 18528 columns 560 uncut, 505 cut).
template <int MODE, int IO>
int launch_gen(ZArgs a, cudaStream_t st) {
  bool digits = IO == ZIO_DD && a.digits, inplace = true;
  for (int i = 0; i < a.fd.npass; ++i) inplace = inplace && fft_inplace_radix(a.fd.pass[i].R);
  if constexpr (!zkeep(MODE))
    digits = digits || (inplace && a.fd.npass <= a.fd.ng && a.LB > 1 &&
                        (size_t)a.LB * a.nz * sizeof(double2) * 2 > ZGEN_SMEM);
  a.nbuf = digits && inplace ? 1 : 2;
  if constexpr (IO == ZIO_DD || !zkeep(MODE))
    if (digits) return launch_gen_as<MODE, IO, true>(a, st);
  return launch_gen_as<MODE, IO, false>(a, st);
}

template <int MODE, int R1, int R2, int IO>
int launch_split(const ZArgs& a, int nblocks, cudaStream_t st) {
  using GZ = Z2Geo<MODE, R1 * R2, (R1 > R2 ? R1 : R2)>;
  static DeviceOnce once;
  if (!once.run([] {
        return cudaFuncSetAttribute(zfft2_kernel<MODE, R1, R2, IO>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    200 * 1024) == cudaSuccess &&
               cudaFuncSetAttribute(zfft2_kernel<MODE, R1, R2, IO>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                    100) == cudaSuccess;
      }))
    return SPH_ECUDA;
  const size_t smem = (size_t)GZ::LB * R1 * R2 * sizeof(double2) * (zkeep(MODE) ? 2 : 1);
  launch_dependent(zfft2_kernel<MODE, R1, R2, IO>, nblocks, GZ::THREADS, smem, st, a);
  SPH_LAUNCH_OK();
  return SPH_OK;
}

template <int MODE, int CTN, int IO>
int launch_ct(const ZArgs& a, int nblocks, size_t smem, cudaStream_t st) {
  if constexpr (ct::split2_r1(CTN) > 0) {  // a.LB is z2_lb(CTN): widths of these lengths are not tuned
    constexpr int R1 = ct::split2_r1(CTN);
    return launch_split<MODE, R1, CTN / R1, IO>(a, nblocks, st);
  } else {
    static DeviceOnce once;
    if (!once.run([] {
          return cudaFuncSetAttribute(zfft_kernel<MODE, CTN, IO>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      200 * 1024) == cudaSuccess &&
                 cudaFuncSetAttribute(zfft_kernel<MODE, CTN, IO>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                      100) == cudaSuccess;
        }))
      return SPH_ECUDA;
    launch_dependent(zfft_kernel<MODE, CTN, IO>, nblocks, ZTHREADS, smem, st, a);
    SPH_LAUNCH_OK();
    return SPH_OK;
  }
}

#define Z_SIZES(X) X(16) X(32) X(48) X(64) X(96) X(128) X(192) X(256) X(512)

// the two-step kernel's columns per CTA for the lengths that take it, else 0
int zsplit_lb(int nz) {
  switch (nz) {
#define CASE(n) \
  case n: return std::integral_constant<int, (ct::split2_r1(n) > 0 ? z2_lb(n) : 0)>::value;
    Z_SIZES(CASE)
#undef CASE
  }
  return 0;
}
bool zsplit_length(int nz) { return zsplit_lb(nz) > 0; }

bool ct_length(int nz) {
  switch (nz) {
#define CASE(n) case n:
    Z_SIZES(CASE)
#undef CASE
    return true;
  }
  return false;
}

template <int MODE, int IO>
int launch_mode(const ZArgs& a, int nblocks, size_t smem, cudaStream_t st) {
  switch (a.nz) {
#define CASE(n) \
  case n: return launch_ct<MODE, n, IO>(a, nblocks, smem, st);
    Z_SIZES(CASE)
#undef CASE
    default: return launch_gen<MODE, IO>(a, st);
  }
}

// the element types used with each mode: FP64 everywhere; single precision
// in and out for every mode; FP64 in, single out for the forward transform
// (after the analysis in FP64); single in, FP64 out for the inverse (before
// the synthesis)
template <int MODE>
int launch_mode_io(const ZArgs& a, int io, int nblocks, size_t smem, cudaStream_t st) {
  switch (io) {
    case ZIO_DD: return launch_mode<MODE, ZIO_DD>(a, nblocks, smem, st);
    case ZIO_FF: return launch_mode<MODE, ZIO_FF>(a, nblocks, smem, st);
    case ZIO_DF:
      if constexpr (MODE == Z_FWD) return launch_mode<MODE, ZIO_DF>(a, nblocks, smem, st);
      break;
    case ZIO_FD:
      if constexpr (MODE == Z_INV) return launch_mode<MODE, ZIO_FD>(a, nblocks, smem, st);
      break;
  }
  return SPH_EINVAL;
}

}  // namespace

int launch_zfft(const sph_plan* p, int mode, const double2* in, double2* out, int order,
                cudaStream_t st, bool cont) {
  return launch_zfft_io(p, mode, in, out, ZIO_DD, order, st, cont);
}

namespace {

// The arguments of one z transform of plan p's spectra and its CTA count.
int make_zargs(const sph_plan* p, int mode, const void* in, void* out, int order, bool cont, ZArgs* ap,
               int* nblocks) {
  ZArgs& a = *ap;
  a.in = in;
  a.out = out;
  a.nlm = p->nlmv;  // the caller's lm columns [lm0, lm0 + nlmv)
  a.nz = p->nz;
  a.N = cont ? p->N : p->nz;
  a.C = cont ? p->C : 0;
  a.d = p->d;
  a.order = order;
  a.dir = p->d_dir;
  a.kfac = (order >= 1 && order <= 4) ? p->kfac + (size_t)(order - 1) * p->nz : nullptr;
  a.filt = p->filt;
  a.zinv2 = p->zinv2;
  a.ell = p->d_ell + p->lm0;
  a.fd = p->fz;
  // columns per CTA: a power of two with LB*nz <= ZMAXCOL/2, at most 64
  // (32 KB slabs: 4 CTAs per SM, still full 128-byte lines per row at nz = 256)
  int LB = 64;
  while (LB > 1 && LB * p->nz > ZMAXCOL / 2) LB >>= 1;
  // a tuned width, except for the lengths with the two-step split, whose
  // kernel is compiled for the default width
  if (zsplit_length(p->nz)) LB = zsplit_lb(p->nz);
  if (!ct_length(p->nz)) LB = zgen_lb(p->nz, p->nlmv);
  if (p->tile_lb && !zsplit_length(p->nz)) LB = p->tile_lb;
  if (LB * p->nz > ZMAXCOL) return SPH_EINVAL;
  a.LB = LB;
  *nblocks = (p->nlmv + LB - 1) / LB;
  if (mode == Z_DLR || mode == Z_DLADD) a.kfac = p->kfac + (size_t)1 * p->nz;  // (i kz)^2
  a.nl = {};
  a.z = p->d_z;
  a.zinv = p->zinv;
  a.digits = p->precision == SPH_MIXED;
  return SPH_OK;
}

}  // namespace

int launch_zfft_io(const sph_plan* p, int mode, const void* in, void* out, int io, int order, cudaStream_t st,
                   bool cont) {
  ZArgs a;
  int nblocks = 0;
  const int rc = make_zargs(p, mode, in, out, order, cont, &a, &nblocks);
  if (rc != SPH_OK) return rc;
  size_t smem = (size_t)a.LB * p->nz * sizeof(double2) * (mode == Z_DLR ? 2 : 1);
  TimedLaunch tl(p, T_ZFFT, st);
  switch (mode) {
    case Z_FWD: return launch_mode_io<Z_FWD>(a, io, nblocks, smem, st);
    case Z_INV: return launch_mode_io<Z_INV>(a, io, nblocks, smem, st);
    case Z_DERIV:
      if (!a.kfac) return SPH_EINVAL;
      return launch_mode_io<Z_DERIV>(a, io, nblocks, smem, st);
    case Z_FILTER: return launch_mode_io<Z_FILTER>(a, io, nblocks, smem, st);
    case Z_DLR: return launch_mode_io<Z_DLR>(a, io, nblocks, smem, st);
  }
  return SPH_EINVAL;
}

namespace {

// the nonlinear step's passes: the two-step kernel for its lengths, the
// general one for the others
template <int MODE>
int launch_nl(const ZArgs& a, int nblocks, cudaStream_t st) {
  switch (a.nz) {
#define CASE(n)                                                                                             \
  case n:                                                                                                   \
    if constexpr (ct::split2_r1(n) > 0)                                                                     \
      return launch_split<MODE, std::max(1, ct::split2_r1(n)), n / std::max(1, ct::split2_r1(n)), ZIO_DD>(a, nblocks, st); \
    break;
    Z_SIZES(CASE)
#undef CASE
  }
  return launch_gen<MODE, ZIO_DD>(a, st);
}

}  // namespace

int launch_znl(const sph_plan* p, int mode, const double2* x, double2* out, const ZNlArgs& nl, cudaStream_t st) {
  ZArgs a;
  int nblocks = 0;
  const int rc = make_zargs(p, mode, x, out, 1, true, &a, &nblocks);
  if (rc != SPH_OK) return rc;
  a.nl = nl;
  TimedLaunch tl(p, T_ZFFT, st);
  switch (mode) {
    case Z_POT: return launch_nl<Z_POT>(a, nblocks, st);
    case Z_RHS: return launch_nl<Z_RHS>(a, nblocks, st);
    case Z_DLADD: return launch_nl<Z_DLADD>(a, nblocks, st);
  }
  return SPH_EINVAL;
}

// ---------------------------------------------------------------- grouped forward z (batches)
namespace {

template <int R1, int R2>
int zgroup_launch_len(const ZGroupLen& L, cudaStream_t st) {
  constexpr int NZ = R1 * R2;
  using GZ = Z2Geo<Z_FWD, NZ, ct::split2_tpc(NZ)>;
  static DeviceOnce once;
  if (!once.run([] {
        return cudaFuncSetAttribute(zfft2_group_kernel<Z_FWD, R1, R2, ZIO_DD>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) == cudaSuccess &&
               cudaFuncSetAttribute(zfft2_group_kernel<Z_FWD, R1, R2, ZIO_DD>,
                                    cudaFuncAttributePreferredSharedMemoryCarveout, 100) == cudaSuccess;
      }))
    return SPH_ECUDA;
  const size_t smem = (size_t)GZ::LB * NZ * sizeof(double2);
  zfft2_group_kernel<Z_FWD, R1, R2, ZIO_DD>
      <<<L.total, GZ::THREADS, smem, st>>>(static_cast<const ZArgs*>(L.jobs), L.prefix, L.njobs);
  SPH_LAUNCH_OK();
  return SPH_OK;
}

// the two-step lengths only (the others never reach a grouped launch)
template <int NZ>
int zgroup_launch_nz(const ZGroupLen& L, cudaStream_t st) {
  if constexpr (ct::split2_r1(NZ) > 0) {
    return zgroup_launch_len<ct::split2_r1(NZ), NZ / ct::split2_r1(NZ)>(L, st);
  } else {
    return SPH_EINVAL;
  }
}

}  // namespace

int zfwd_group_prepare(const std::vector<ZJob>& jobs, ZGroupLaunch* g, std::vector<int>* rest) {
  if (!g || !rest) return SPH_EINVAL;
  rest->clear();
  std::vector<int> lens;  // z lengths, in order of first appearance
  std::vector<std::vector<ZArgs>> args;
  std::vector<std::vector<int>> prefix;
  for (int k = 0; k < (int)jobs.size(); ++k) {
    const sph_plan* p = jobs[k].p;
    ZArgs a;
    int nb = 0;
    if (!p || !jobs[k].spec || !zsplit_length(p->nz) ||
        make_zargs(p, Z_FWD, jobs[k].spec, jobs[k].spec, 0, jobs[k].cont, &a, &nb) != SPH_OK || nb < 1 ||
        a.LB != zsplit_lb(p->nz)) {
      rest->push_back(k);
      continue;
    }
    int li = (int)(std::find(lens.begin(), lens.end(), p->nz) - lens.begin());
    if (li == (int)lens.size()) {
      lens.push_back(p->nz);
      args.emplace_back();
      prefix.emplace_back(1, 0);
    }
    args[li].push_back(a);
    prefix[li].push_back(prefix[li].back() + nb);
  }
  for (size_t li = 0; li < lens.size(); ++li) {
    ZGroupLen L;
    L.nz = lens[li];
    L.njobs = (int)args[li].size();
    L.total = prefix[li].back();
    g->lens.push_back(L);
    ZGroupLen& G = g->lens.back();
    if (cudaMalloc(&G.jobs, args[li].size() * sizeof(ZArgs)) != cudaSuccess ||
        cudaMalloc((void**)&G.prefix, prefix[li].size() * sizeof(int)) != cudaSuccess)
      return SPH_ENOMEM;
    if (cudaMemcpy(G.jobs, args[li].data(), args[li].size() * sizeof(ZArgs), cudaMemcpyHostToDevice) !=
            cudaSuccess ||
        cudaMemcpy(G.prefix, prefix[li].data(), prefix[li].size() * sizeof(int), cudaMemcpyHostToDevice) !=
            cudaSuccess)
      return SPH_ECUDA;
  }
  return SPH_OK;
}

int zfwd_group_launch(const ZGroupLaunch& g, cudaStream_t st) {
  for (const ZGroupLen& L : g.lens) {
    int rc = SPH_EINVAL;
    switch (L.nz) {
#define CASE(n)                    \
  case n:                          \
    rc = zgroup_launch_nz<n>(L, st); \
    break;
      Z_SIZES(CASE)
#undef CASE
    }
    if (rc != SPH_OK) return rc;
  }
  return SPH_OK;
}

void zgroup_free(ZGroupLaunch* g) {
  for (ZGroupLen& L : g->lens) {
    if (L.jobs) cudaFree(L.jobs);
    if (L.prefix) cudaFree(L.prefix);
  }
  g->lens.clear();
}

// ---------------------------------------------------------------- no-alloc derivative
// Radial derivative for callers that cannot allocate device memory: the
// device-resident tables the fused derivative kernel reads (twiddles,
// digit-reversal order, (i kz)^p factors, the FC-Gram operator) live in one
// file-scope array instead of a plan's cudaMalloc'd buffers.  The host side
// stages them in fixed static buffers, so the call allocates nothing on the
// host either.
namespace {

constexpr int NA_MAX_NZ = 4096;  // longest radial transform
constexpr int NA_MAX_CD = 2048;  // largest Cz*oz
constexpr size_t NA_TW = 0;                                              // double2[nz]
constexpr size_t NA_TWP = NA_TW + (size_t)NA_MAX_NZ * sizeof(double2);   // double2[< nz]
constexpr size_t NA_KF = NA_TWP + (size_t)NA_MAX_NZ * sizeof(double2);   // double2[nz]
constexpr size_t NA_DIR = NA_KF + (size_t)NA_MAX_NZ * sizeof(double2);   // double[Cz*oz]
constexpr size_t NA_REV = NA_DIR + (size_t)NA_MAX_CD * sizeof(double);   // int[nz]
constexpr size_t NA_BYTES = NA_REV + (size_t)NA_MAX_NZ * sizeof(int);    // 224 KiB

static __device__ __align__(256) unsigned char g_noalloc_tables[NA_BYTES];

// host staging, laid out like the device array; serialised by na_mutex
static unsigned char na_host[NA_BYTES];
static std::mutex na_mutex;
static void* na_dev[64];  // device address of g_noalloc_tables, per device

int na_setup(int dev) {
  if (dev < 0 || dev >= 64) return SPH_EINVAL;
  if (na_dev[dev]) return SPH_OK;
  void* ptr = nullptr;
  if (cudaGetSymbolAddress(&ptr, g_noalloc_tables) != cudaSuccess || !ptr) return SPH_ECUDA;
  na_dev[dev] = ptr;
  return SPH_OK;
}

}  // namespace

extern "C" int sph_derivr_noalloc(const double* a, double* b, int nlm, int nz, int Cz, int oz, double rint,
                                  double rext, const double* dir, int p, void* stream) {
  if (!a || !b || nlm < 1 || nz < 2 || nz > NA_MAX_NZ || p < 1 || p > 4) return SPH_EINVAL;
  if (Cz < 0 || oz < 0 || (Cz > 0 && (oz < 1 || nz - Cz < oz || !dir)) || (size_t)Cz * oz > NA_MAX_CD)
    return SPH_EINVAL;
  // radix plan (8s, then 4, 2, 3, other primes), as sph_plan_create builds it
  FftDesc fd = {};
  fd.n = nz;
  {
    int r = nz, Ns = 1;
    for (int q : {8, 4, 2, 3})
      while (r % q == 0) {
        if (fd.npass >= SPH_MAX_PASSES) return SPH_EINVAL;
        fd.pass[fd.npass++] = {q, Ns};
        Ns *= q;
        r /= q;
      }
    for (int q = 5; r > 1; q += 2)
      while (r % q == 0) {
        if (q > 64 || fd.npass >= SPH_MAX_PASSES) return SPH_EINVAL;
        fd.pass[fd.npass++] = {q, Ns};
        Ns *= q;
        r /= q;
      }
  }
  if (!fft_gen_plan(nz, fd)) return SPH_EINVAL;
  int LB = 64;
  // the column blocks of the plan path (so that both run the same kernel)
  while (LB > 1 && LB * nz > ZMAXCOL / 2) LB >>= 1;
  if (LB * nz > ZMAXCOL) return SPH_EINVAL;
  if (zsplit_length(nz)) LB = zsplit_lb(nz);
  if (!ct_length(nz)) LB = zgen_lb(nz, nlm);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return SPH_ECUDA;
  std::lock_guard<std::mutex> lock(na_mutex);
  int rc = na_setup(dev);
  if (rc != SPH_OK) return rc;

  const long double pi = 3.141592653589793238462643383279502884L;
  double2* tw = reinterpret_cast<double2*>(na_host + NA_TW);
  double2* twp = reinterpret_cast<double2*>(na_host + NA_TWP);
  double2* kf = reinterpret_cast<double2*>(na_host + NA_KF);
  double* dr = reinterpret_cast<double*>(na_host + NA_DIR);
  int* rev = reinterpret_cast<int*>(na_host + NA_REV);
  for (int e = 0; e < nz; ++e) {
    long double ang = -2.0L * pi * e / nz;
    tw[e] = make_double2((double)cosl(ang), (double)sinl(ang));
  }
  int ntp = 0;  // per-pass twiddles [pass][j][r-1] = W_L^{j r}
  for (int L = nz; L > 1;) {
    int R = L % 8 == 0 ? 8 : L % 4 == 0 ? 4 : L % 2 == 0 ? 2 : L % 3 == 0 ? 3 : L;
    int S = L / R;
    for (int j = 0; j < S; ++j)
      for (int r = 1; r < R; ++r) {
        long double ang = -2.0L * pi * (long double)((long)j * r) / L;
        twp[ntp++] = make_double2((double)cosl(ang), (double)sinl(ang));
      }
    L = S;
  }
  for (int k = 0; k < nz; ++k) {
    int t = k, s = nz, pos = 0;
    for (int ip = 0; ip < fd.npass; ++ip) {
      s /= fd.pass[ip].R;
      pos += (t % fd.pass[ip].R) * s;
      t /= fd.pass[ip].R;
    }
    rev[k] = pos;
  }
  // kz as box_init builds it (src/pseudo/pseudospec_mod.f90:196-227), times i^p
  const int N = nz - Cz;
  const double dz = N > 1 ? (rext - rint) / (nz - Cz - 1) : 1.0;
  const double Dkz = 2.0 * 3.14159265358979323846 / (dz * nz);
  for (int k = 0; k < nz; ++k) {
    double kzk;
    if (nz % 2 == 0) kzk = (double)(k < nz / 2 ? k : k - nz) * Dkz;
    else kzk = (double)(k < (nz + 1) / 2 ? k : k - nz) * Dkz;
    double kp = 1.0;
    for (int q = 0; q < p; ++q) kp *= kzk;
    double re = (p % 4 == 0) ? 1 : (p % 4 == 2) ? -1 : 0;
    double im = (p % 4 == 1) ? 1 : (p % 4 == 3) ? -1 : 0;
    kf[k] = make_double2(re * kp, im * kp);
  }
  for (int q = 0; q < Cz * oz; ++q) dr[q] = dir[q];

  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* dbase = static_cast<unsigned char*>(na_dev[dev]);
  const size_t spans[][2] = {{NA_TW, (size_t)nz * sizeof(double2)},
                             {NA_TWP, (size_t)(ntp > 0 ? ntp : 1) * sizeof(double2)},
                             {NA_KF, (size_t)nz * sizeof(double2)},
                             {NA_DIR, (size_t)(Cz * oz > 0 ? Cz * oz : 1) * sizeof(double)},
                             {NA_REV, (size_t)nz * sizeof(int)}};
  for (auto& sp : spans)
    if (cudaMemcpyAsync(dbase + sp[0], na_host + sp[0], sp[1], cudaMemcpyHostToDevice, st) != cudaSuccess)
      return SPH_ECUDA;

  fd.tw = reinterpret_cast<const double2*>(dbase + NA_TW);
  fd.twp = reinterpret_cast<const double2*>(dbase + NA_TWP);
  fd.rev = reinterpret_cast<const int*>(dbase + NA_REV);
  ZArgs z = {};
  z.in = reinterpret_cast<const double2*>(a);
  z.out = reinterpret_cast<double2*>(b);
  z.nlm = nlm;
  z.nz = nz;
  z.N = N;
  z.C = Cz;
  z.d = oz;
  z.LB = LB;
  z.order = p;
  z.dir = reinterpret_cast<const double*>(dbase + NA_DIR);
  z.kfac = reinterpret_cast<const double2*>(dbase + NA_KF);
  z.fd = fd;
  const int nblocks = (nlm + LB - 1) / LB;
  const size_t smem = (size_t)LB * nz * sizeof(double2);
  return launch_mode<Z_DERIV, ZIO_DD>(z, nblocks, smem, st);
}
