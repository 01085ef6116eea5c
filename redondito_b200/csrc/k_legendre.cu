// k_legendre.cu -- per-m Legendre contractions as FP64 tensor-core GEMMs.
//
// The reference does these inside SHTns, one plane at a time (spat_to_SH /
// SH_to_spat / spat_to_SHqst / SHqst_to_spat at src/sphp/sphp_sca.F90:312,485
// and src/sphp/sphp_vec.F90:89-91,157-159).  Here every plane and field is a
// column of one GEMM per m, so each Legendre table tile is read once per
// (m, row block) for all nz planes:
//   analysis   a[l][n]   = sum_i Pbar_lm(x_i) G_(l-m)%2[i][n]          K = nlat/2
//   synthesis  S_q[i][n] = sum_{l: (l-m)%2 = q} Pbar_lm(x_i) a[l][n]    K = lmax+1-m
// with n = (plane, re/im); folding mirror rings into even/odd parts halves K.
// The vector transforms fold their complex factors into the operand loads:
//   S_l  = 1/(l(l+1)) sum_i [ dP_l Vt_(1-p) + mPs_l (-i Vp_p) ]
//   T_l  = 1/(l(l+1)) sum_i [ mPs_l (-i Vt_p) - dP_l Vp_(1-p) ]
//   Vt_q = sum_(p=1-q) dP_l S_l + sum_(p=q) mPs_l (i T_l)
//   Vp_q = sum_(p=1-q) dP_l (-T_l) + sum_(p=q) mPs_l (i S_l)
// (p = (l-m)%2, fold 0 = F(i)+F(mirror), fold 1 = F(i)-F(mirror); Pbar has
// the parity of p, dPbar the opposite), so each output is one accumulator
// over a K twice as long.
//
// Bound by the FP64 tensor pipe (mma.sync.m16n8k4.f64; tcgen05 has no FP64
// kind), so the rest of the issue slots, the padding and the waits are what
// the layout is about:
//   - tiles arrive by cp.async through a 2- to 4-stage pipeline, every
//     thread's source addresses advanced by a constant per K tile;
//   - shared memory holds 128-byte rows with the 16-byte chunk index XORed by
//     the row, and the K order inside a fragment is chosen so that each
//     fragment load is one conflict-free 16-byte access: two nodes (or the two
//     nodes of an interleaved row pair) of a table row, or the re and im of one
//     coefficient.  Re and im are separate column tiles of 8 planes, so the
//     factors i and -1 of the vector forms become the choice of tile and of a
//     negated table fragment;
//   - a warp holds 16 accumulator tiles (32 FP64 values per thread); the vector
//     kernels form both outputs from one load of each operand;
//   - row tiles past lmax or nlat/2 and groups of 8 planes past the selection
//     issue no MMAs (103 physical planes cost 104);
//   - the plane blocks of one table tile are consecutive CTAs, so the tables
//     are read from HBM once.
#include <type_traits>

#include "sph_internal.cuh"

namespace {

// ---------------------------------------------------------------- primitives
// c (16 x 8) += a (16 x 4) b (4 x 8).  Lane (g = lane / 4, t = lane % 4):
// a0, a1 = rows g, g + 8 of column t; b = row t of column g; c[0..1] = row g,
// columns 2t, 2t + 1; c[2..3] = row g + 8.
__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b) {
  asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a0), "d"(a1), "d"(b));
}

// 16-byte global->shared copy; pred == false fills zeros (no global read).
__device__ __forceinline__ void cp16(unsigned dst, const void* gmem, bool pred) {
  const int sz = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}
__device__ __forceinline__ double2 frag(const unsigned char* p) { return *reinterpret_cast<const double2*>(p); }

// Two adjacent complex values, 32-byte aligned.
__device__ __forceinline__ void store2(double2* p, double a, double b, double c, double d) {
  asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};\n" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

struct LegArgs {
  const double* P;     // [nlm][ldn]
  const double* dP;    // [nlm][ldn]
  const double* mPs;   // [nlm][ldn]
  const double2* G;    // folded coefficients [field][m][2][nz][ldn]
  double2* Gw;
  size_t Gfield;
  int gfield;
  const double2* spec;  // (nz, nlm)
  const double2* spec2;
  double2* out;
  double2* out2;
  const LegTile* tiles;
  const int* mbase;
  const int* kzl;  // planes to transform (nullptr: all nz)
  int lmax, nlat2, ldn, nz, nlm, nkz;  // nodes past nlat2 are padding: G holds anything there
  int nkb;         // plane blocks of the launch
};

// Grouped launches: the CTAs of several plans' work sets in one grid; job j
// owns CTAs prefix[j] .. prefix[j+1]-1, laid out (tile, plane block).
struct LegGroup {
  const LegArgs* jobs;
  const int* prefix;
  int njobs;
};

// This CTA's arguments and (tile, plane block) indices, plane blocks fastest.
template <bool G>
__device__ __forceinline__ void leg_cta(const LegArgs& a0, const LegGroup& grp, LegArgs& a, int& bx, int& by) {
  int local = blockIdx.x;
  if constexpr (!G) {
    a = a0;
  } else {
    int lo = 0, hi = grp.njobs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(grp.prefix + mid) <= local) lo = mid;
      else hi = mid - 1;
    }
    a = grp.jobs[lo];
    local -= __ldg(grp.prefix + lo);
  }
  bx = local / a.nkb;
  by = local - bx * a.nkb;
}

// plane of local index kl; ok = within the selection
__device__ __forceinline__ int plane_of(const LegArgs& a, int kl, bool& ok) {
  ok = kl < a.nkz;
  return a.kzl ? (ok ? __ldg(a.kzl + kl) : 0) : kl;
}

constexpr int ROW = 128;  // bytes of a shared-memory row

// ================================================================ scalar analysis
// CTA: 128 consecutive l x 16 planes; K tile 16 nodes.  4 warps = (parity,
// half of the l), each 32 l of its parity x 16 planes.
// lmax 511, 256 planes: 2.51 -> 1.82 ms (28.3 TF/s, 77% of the FP64 tensor
// peak); with 8 warps and 32 planes per CTA, two CTAs per SM, 1.98: more and
// smaller CTAs hide each other's first loads and stores.
namespace an {
constexpr int L = 128, KZ = 16, K = 16, STAGES = 2;
constexpr int A_B = L * ROW, B_B = 4 * KZ * ROW;  // table rows; [parity][8 nodes][plane] coefficient rows
constexpr int STAGE = A_B + B_B;
constexpr int CP = L + 1;  // pitch of the output staging
constexpr int SMEM = STAGES * STAGE;
static_assert(KZ * CP * 16 <= SMEM, "output staging");
}  // namespace an

template <bool GROUP>
__global__ void __launch_bounds__(128, 4) leg_analysis_kernel(LegArgs a0, LegGroup grp) {
  grid_dependency_wait();
  using namespace an;
  extern __shared__ __align__(128) unsigned char sm[];
  LegArgs a;
  int bx, by;
  leg_cta<GROUP>(a0, grp, a, bx, by);
  const LegTile tile = a.tiles[bx];
  const int m = tile.m, l0 = tile.r0, kz0 = by * KZ;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int par = warp >> 1, lh = warp & 1;
  const size_t base_lm = (size_t)a.mbase[m] - m;
  const int nk = (a.ldn + K - 1) / K;

  // copies: chunk lc of row lr + 16 j, or of plane lr
  const int lc = tid & 7, lr = tid >> 3;
  const double* pa = a.P + (base_lm + l0 + lr) * a.ldn + 2 * lc;
  bool okb;
  const int kzb = plane_of(a, kz0 + lr, okb);
  const double2* pb = a.G + (size_t)a.gfield * a.Gfield + ((size_t)m * 2 * a.nz + kzb) * a.ldn + lc;
  const size_t parb = (size_t)a.nz * a.ldn;
  const unsigned s0 = (unsigned)__cvta_generic_to_shared(sm);
  const unsigned da = s0 + lr * ROW + ((lc ^ ((lr & 2) << 1)) << 4), db = s0 + A_B + lr * ROW + ((lc ^ (lr & 7)) << 4);
  const int na = a.lmax - l0 - lr;  // table row j is needed where 16 j <= na
  auto load = [&](int st, int k0) {
    const bool oka = k0 + 2 * lc < a.ldn;
#pragma unroll
    for (int j = 0; j < L / 16; ++j) {
      const bool ok = oka && 16 * j <= na;
      cp16(da + st * STAGE + j * 16 * ROW, ok ? pa + (size_t)(16 * j) * a.ldn + k0 : a.P, ok);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {  // (parity, block of 8 nodes)
      const bool ok = okb && k0 + (j & 1) * 8 + lc < a.nlat2;
      cp16(db + st * STAGE + j * KZ * ROW, ok ? pb + (j >> 1) * parb + k0 + (j & 1) * 8 : a.G, ok);
    }
  };

  // m16 tiles of 32 l and groups of 8 planes with work
  const int nmt = min(2, (a.lmax - l0 - lh * 64 + 32) / 32), ngr = min(2, (a.nkz - kz0 + 7) / 8);
  double acc[2][2][2][4] = {};  // [m16 tile][plane group][re, im]
  const unsigned char* fa = sm + (lh * 64 + 2 * g + par) * ROW;
  const unsigned char* fb = sm + A_B + (par * 2 * KZ + g) * ROW;
  const int sw = (g & 1) << 2;
  auto compute = [&](const unsigned char* A, const unsigned char* B, auto full) {
    constexpr bool FULL = decltype(full)::value;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      double2 av[2][2];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int r = 0; r < 2; ++r) av[mt][r] = frag(A + (mt * 32 + r * 16) * ROW + (((t + 4 * h) ^ sw) << 4));
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int gr = 0; gr < 2; ++gr) {
          if (!FULL && gr >= ngr) continue;
          const double2 b = frag(B + (h * KZ + gr * 8) * ROW + (((2 * t + s) ^ g) << 4));
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            if (!FULL && mt >= nmt) continue;
            const double x0 = s ? av[mt][0].y : av[mt][0].x, x1 = s ? av[mt][1].y : av[mt][1].x;
            dmma(acc[mt][gr][0], x0, x1, b.x);
            dmma(acc[mt][gr][1], x0, x1, b.y);
          }
        }
    }
  };

  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nk) load(s, s * K);
    cp_commit();
  }
  const bool full = nmt == 2 && ngr == 2, any = nmt > 0 && ngr > 0;
  for (int kt = 0, st = 0; kt < nk; ++kt, st = st + 1 == STAGES ? 0 : st + 1) {
    cp_wait<STAGES - 2>();
    __syncthreads();
    const int nx = kt + STAGES - 1;
    if (nx < nk) load(st == 0 ? STAGES - 1 : st - 1, nx * K);
    cp_commit();
    if (full) compute(fa + st * STAGE, fb + st * STAGE, std::true_type());
    else if (any) compute(fa + st * STAGE, fb + st * STAGE, std::false_type());
  }
  cp_wait<0>();
  __syncthreads();

  // Cs[plane][l], then contiguous rows of the (nz, nlm) output
  double2* Cs = reinterpret_cast<double2*>(sm);
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int gr = 0; gr < 2; ++gr)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int row = lh * 64 + 2 * (mt * 16 + (c >> 1) * 8 + g) + par, pl = gr * 8 + 2 * t + (c & 1);
        Cs[pl * CP + row] = make_double2(acc[mt][gr][0][c], acc[mt][gr][1][c]);
      }
  __syncthreads();
  const int nvalid = min(L, a.lmax + 1 - l0);
  for (int idx = tid; idx < KZ * L; idx += 128) {
    const int pl = idx / L, ll = idx % L;
    bool okz;
    const int kz = plane_of(a, kz0 + pl, okz);
    if (!okz || ll >= nvalid) continue;
    double2 v = Cs[pl * CP + ll];
    if (m == 0) v.y = 0.0;  // m = 0 coefficients of a real field are real
    a.out[(size_t)kz * a.nlm + base_lm + l0 + ll] = v;
  }
}

// ================================================================ scalar synthesis
// CTA: 64 nodes x 16 planes; K tile 16 consecutive l (8 per parity).
// 4 warps = (parity, half of the nodes).
// lmax 511, 256 planes: 2.06 -> 1.67 ms (30.9 TF/s, 84%); 8 warps and 32
// planes per CTA 1.79.
namespace sy {
constexpr int I = 64, KZ = 16, K = 16, STAGES = 4;
constexpr int A_B = (I / 16) * K * ROW, B_B = 2 * KZ * ROW;  // [16 nodes][l] table rows; [8 l][plane] spectra rows
constexpr int STAGE = A_B + B_B;
constexpr int SMEM = STAGES * STAGE;
}  // namespace sy

template <bool GROUP>
__global__ void __launch_bounds__(128, 4) leg_synthesis_kernel(LegArgs a0, LegGroup grp) {
  grid_dependency_wait();
  using namespace sy;
  extern __shared__ __align__(128) unsigned char sm[];
  LegArgs a;
  int bx, by;
  leg_cta<GROUP>(a0, grp, a, bx, by);
  const LegTile tile = a.tiles[bx];
  const int m = tile.m, i0 = tile.r0, kz0 = by * KZ;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int par = warp >> 1, mh = warp & 1;
  const size_t base_lm = (size_t)a.mbase[m];
  const int nl = a.lmax + 1 - m, nk = (nl + K - 1) / K;

  const int lc = tid & 7, ar = tid >> 3, bp = tid >> 3;
  const int ia = i0 + 2 * lc;
  const double* pa = a.P + (base_lm + ar) * a.ldn + ia;
  bool okb;
  const int kzb = plane_of(a, kz0 + bp, okb);
  const double2* pb = a.spec + (size_t)kzb * a.nlm + base_lm + lc;
  const unsigned s0 = (unsigned)__cvta_generic_to_shared(sm);
  const unsigned da = s0 + ar * ROW + ((lc ^ (ar & 7)) << 4), db = s0 + A_B + bp * ROW + ((lc ^ (bp & 7)) << 4);
  auto load = [&](int st, int q0) {  // degrees m + q0 ..
#pragma unroll
    for (int j = 0; j < I / 16; ++j) {
      const bool ok = q0 + ar < nl && ia + 16 * j < a.ldn;
      cp16(da + st * STAGE + j * K * ROW, ok ? pa + (size_t)q0 * a.ldn + 16 * j : a.P, ok);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const bool ok = okb && q0 + 8 * j + lc < nl;
      cp16(db + st * STAGE + j * KZ * ROW, ok ? pb + q0 + 8 * j : a.spec, ok);
    }
  };

  const int nmt = min(2, (a.ldn - i0 - mh * 32 + 15) / 16), ngr = min(2, (a.nkz - kz0 + 7) / 8);
  double acc[2][2][2][4] = {};  // [16 nodes][plane group][re, im]
  const int kr = par + 2 * t;   // this lane's l within a block of 8
  const unsigned char* fa = sm + (mh * 2 * K + kr) * ROW + ((g ^ kr) << 4);
  const unsigned char* fb = sm + A_B + g * ROW + ((kr ^ g) << 4);
  auto compute = [&](const unsigned char* A, const unsigned char* B, auto full) {
    constexpr bool FULL = decltype(full)::value;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      double2 av[2];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) av[mt] = frag(A + (mt * K + h * 8) * ROW);
#pragma unroll
      for (int gr = 0; gr < 2; ++gr) {
        if (!FULL && gr >= ngr) continue;
        const double2 b = frag(B + (h * KZ + gr * 8) * ROW);
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          if (!FULL && mt >= nmt) continue;
          dmma(acc[mt][gr][0], av[mt].x, av[mt].y, b.x);
          dmma(acc[mt][gr][1], av[mt].x, av[mt].y, b.y);
        }
      }
    }
  };

  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nk) load(s, s * K);
    cp_commit();
  }
  const bool full = nmt == 2 && ngr == 2, any = nmt > 0 && ngr > 0;
  for (int kt = 0, st = 0; kt < nk; ++kt, st = st + 1 == STAGES ? 0 : st + 1) {
    cp_wait<STAGES - 2>();
    __syncthreads();
    const int nx = kt + STAGES - 1;
    if (nx < nk) load(st == 0 ? STAGES - 1 : st - 1, nx * K);
    cp_commit();
    if (full) compute(fa + st * STAGE, fb + st * STAGE, std::true_type());
    else if (any) compute(fa + st * STAGE, fb + st * STAGE, std::false_type());
  }
  cp_wait<0>();

  double2* G = a.Gw + (size_t)a.gfield * a.Gfield + ((size_t)m * 2 + par) * a.nz * a.ldn;
#pragma unroll
  for (int gr = 0; gr < 2; ++gr)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      bool okz;
      const int kz = plane_of(a, kz0 + gr * 8 + 2 * t + c, okz);
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        const int i = i0 + mh * 32 + mt * 16 + 2 * g;
        if (okz && i < a.ldn)
          store2(G + (size_t)kz * a.ldn + i, acc[mt][gr][0][c], acc[mt][gr][1][c], acc[mt][gr][0][2 + c],
                 acc[mt][gr][1][2 + c]);
      }
    }
}

// ================================================================ vector analysis
// CTA: 64 consecutive l x 16 planes; K tile 16 nodes.  4 warps = (parity,
// group of 8 planes), each both outputs of 32 l:
//   l(l+1) S_re =  dP Vt'_re + mPs Vp_im     l(l+1) S_im =  dP Vt'_im - mPs Vp_re
//   l(l+1) T_re = -dP Vp'_re + mPs Vt_im     l(l+1) T_im = -dP Vp'_im - mPs Vt_re
// (' = fold 1 - p, else fold p); -T is accumulated.  Two stages: one K tile
// is 2048 cycles of tensor work per CTA, more than a load's latency.
// lmax 511, 256 planes: 8.42 -> 6.55 ms (31.5 TF/s, 85%), with 8 warps and 32
// planes per CTA 6.65; lmax 255, 10 planes: 181 -> 82 us, 137 with 32.
namespace va {
constexpr int L = 64, KZ = 16, K = 16, STAGES = 2, THREADS = 8 * KZ;
constexpr int A_B = 2 * L * ROW, B_B = 8 * KZ * ROW;  // [table][l]; [field][fold][8 nodes][plane]
constexpr int STAGE = A_B + B_B;
constexpr int CP = L + 1;
constexpr int SMEM = STAGES * STAGE;
static_assert(2 * KZ * CP * 16 <= SMEM, "output staging");
}  // namespace va

__global__ void __launch_bounds__(va::THREADS, 4) vec_analysis_kernel(LegArgs a) {
  grid_dependency_wait();
  using namespace va;
  extern __shared__ __align__(128) unsigned char sm[];
  const int bx = blockIdx.x / a.nkb, by = blockIdx.x - bx * a.nkb;
  const LegTile tile = a.tiles[bx];
  const int m = tile.m, l0 = tile.r0, kz0 = by * KZ;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int par = warp / (KZ / 8), gr = warp % (KZ / 8);
  const size_t base_lm = (size_t)a.mbase[m] - m;
  const int nk = (a.ldn + K - 1) / K;

  const int lc = tid & 7, lr = tid >> 3;
  const size_t arow = (base_lm + l0 + lr) * a.ldn + 2 * lc;
  bool okb;
  const int kzb = plane_of(a, kz0 + lr, okb);
  const double2* pb = a.G + a.Gfield + ((size_t)m * 2 * a.nz + kzb) * a.ldn + lc;  // field 1: v_theta, 2: v_phi
  const size_t parb = (size_t)a.nz * a.ldn;
  const unsigned s0 = (unsigned)__cvta_generic_to_shared(sm);
  const unsigned da = s0 + lr * ROW + ((lc ^ ((lr & 2) << 1)) << 4), db = s0 + A_B + lr * ROW + ((lc ^ (lr & 7)) << 4);
  const int na = a.lmax - l0 - lr;
  auto load = [&](int st, int k0) {
    const bool oka = k0 + 2 * lc < a.ldn;
#pragma unroll
    for (int j = 0; j < 2 * (L / KZ); ++j) {  // (table, block of KZ rows)
      const int r = j % (L / KZ) * KZ;
      const bool ok = oka && r <= na;
      const double* tab = j / (L / KZ) ? a.mPs : a.dP;
      cp16(da + st * STAGE + j * KZ * ROW, ok ? tab + arow + (size_t)r * a.ldn + k0 : a.dP, ok);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {  // (field, fold, block of 8 nodes)
      const bool ok = okb && k0 + (j & 1) * 8 + lc < a.nlat2;
      cp16(db + st * STAGE + j * KZ * ROW,
           ok ? pb + (j >> 2) * a.Gfield + ((j >> 1) & 1) * parb + k0 + (j & 1) * 8 : a.G, ok);
    }
  };

  const int nmt = kz0 + gr * 8 < a.nkz ? min(2, (a.lmax - l0 + 32) / 32) : 0;
  double acc[2][4][4] = {};  // [m16 tile][S_re, S_im, -T_re, -T_im]
  const unsigned char* fa = sm + (2 * g + par) * ROW;
  const unsigned char* fb = sm + A_B + (gr * 8 + g) * ROW;
  const int sw = (g & 1) << 2;
  const int f1 = (1 - par) * 2 * KZ * ROW, f0 = par * 2 * KZ * ROW, fp = 4 * KZ * ROW;
  auto compute = [&](const unsigned char* A, const unsigned char* B, int mts) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        if (mt >= mts) continue;
        double2 d[2], q[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const unsigned char* p = A + (mt * 32 + r * 16) * ROW + (((t + 4 * h) ^ sw) << 4);
          d[r] = frag(p);
          q[r] = frag(p + L * ROW);
        }
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const unsigned char* p = B + h * KZ * ROW + (((2 * t + s) ^ g) << 4);
          const double2 t1 = frag(p + f1), t0 = frag(p + f0), p1 = frag(p + fp + f1), p0 = frag(p + fp + f0);
          const double d0 = s ? d[0].y : d[0].x, d1 = s ? d[1].y : d[1].x;
          const double q0 = s ? q[0].y : q[0].x, q1 = s ? q[1].y : q[1].x;
          dmma(acc[mt][0], d0, d1, t1.x);
          dmma(acc[mt][1], d0, d1, t1.y);
          dmma(acc[mt][2], d0, d1, p1.x);
          dmma(acc[mt][3], d0, d1, p1.y);
          dmma(acc[mt][0], q0, q1, p0.y);
          dmma(acc[mt][3], q0, q1, t0.x);
          dmma(acc[mt][1], -q0, -q1, p0.x);
          dmma(acc[mt][2], -q0, -q1, t0.y);
        }
      }
  };

  load(0, 0);
  cp_commit();
  for (int kt = 0; kt < nk; ++kt) {
    cp_wait<0>();
    __syncthreads();
    if (kt + 1 < nk) load((kt + 1) & 1, (kt + 1) * K);
    cp_commit();
    const int o = (kt & 1) * STAGE;
    if (nmt == 2) compute(fa + o, fb + o, 2);
    else if (nmt == 1) compute(fa + o, fb + o, 1);
  }
  cp_wait<0>();
  __syncthreads();

  double2* Cs = reinterpret_cast<double2*>(sm);  // [out][plane][l]
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int row = 2 * (mt * 16 + (c >> 1) * 8 + g) + par, pl = gr * 8 + 2 * t + (c & 1);
      Cs[pl * CP + row] = make_double2(acc[mt][0][c], acc[mt][1][c]);
      Cs[(KZ + pl) * CP + row] = make_double2(-acc[mt][2][c], -acc[mt][3][c]);
    }
  __syncthreads();
  const int nvalid = min(L, a.lmax + 1 - l0);
  for (int idx = tid; idx < 2 * KZ * L; idx += THREADS) {
    const int ll = idx % L, r = idx / L, pl = r % KZ, o = r / KZ;
    bool okz;
    const int kz = plane_of(a, kz0 + pl, okz);
    if (!okz || ll >= nvalid) continue;
    const int l = l0 + ll;
    const double f = l ? 1.0 / ((double)l * (double)(l + 1)) : 0.0;
    double2 v = Cs[r * CP + ll];
    v.x *= f;
    v.y *= f;
    if (m == 0) v.y = 0.0;
    (o ? a.out2 : a.out)[(size_t)kz * a.nlm + base_lm + l] = v;
  }
}

// ================================================================ vector synthesis
// CTA: 32 nodes x 16 planes; K tile 16 consecutive l.  4 warps = (fold q,
// group of 8 planes), each both outputs of the 32 nodes:
//   Vt_re =  dP S_re - mPs T_im     Vt_im =  dP S_im + mPs T_re
//   Vp_re = -dP T_re - mPs S_im     Vp_im = -dP T_im + mPs S_re
// (rows of parity 1 - q through dP, of parity q through mPs); -Vp is accumulated.
// lmax 511, 256 planes: 7.41 -> 6.26 ms (33.0 TF/s, 89%), with 8 warps and 32
// planes per CTA 6.64; lmax 255, 10 planes: 128 -> 60 us, 108 with 32.
namespace vs {
constexpr int I = 32, KZ = 16, K = 16, STAGES = 3, THREADS = 8 * KZ;
constexpr int A_B = 2 * (I / 16) * K * ROW, B_B = 4 * KZ * ROW;  // [table][16 nodes][l]; [S, T][8 l][plane]
constexpr int STAGE = A_B + B_B;
constexpr int SMEM = STAGES * STAGE;
}  // namespace vs

__global__ void __launch_bounds__(vs::THREADS, 4) vec_synthesis_kernel(LegArgs a) {
  grid_dependency_wait();
  using namespace vs;
  extern __shared__ __align__(128) unsigned char sm[];
  const int bx = blockIdx.x / a.nkb, by = blockIdx.x - bx * a.nkb;
  const LegTile tile = a.tiles[bx];
  const int m = tile.m, i0 = tile.r0, kz0 = by * KZ;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int q = warp / (KZ / 8), gr = warp % (KZ / 8);
  const size_t base_lm = (size_t)a.mbase[m];
  const int nl = a.lmax + 1 - m, nk = (nl + K - 1) / K;

  const int lc = tid & 7, ar = tid >> 3, bp = tid >> 3;
  const int ia = i0 + 2 * lc;
  const size_t arow = (base_lm + ar) * a.ldn + ia;
  bool okb;
  const int kzb = plane_of(a, kz0 + bp, okb);
  const size_t brow = (size_t)kzb * a.nlm + base_lm + lc;
  const unsigned s0 = (unsigned)__cvta_generic_to_shared(sm);
  const unsigned da = s0 + ar * ROW + ((lc ^ (ar & 7)) << 4), db = s0 + A_B + bp * ROW + ((lc ^ (bp & 7)) << 4);
  auto load = [&](int st, int q0) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {  // (table, block of 16 nodes)
      const bool ok = ia + 16 * (j & 1) < a.ldn && q0 + ar < nl;
      cp16(da + st * STAGE + j * K * ROW, ok ? (j >> 1 ? a.mPs : a.dP) + arow + (size_t)q0 * a.ldn + 16 * (j & 1) : a.dP,
           ok);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {  // (S or T, block of 8 degrees); degree 0 has no vector part
      const int ql = q0 + 8 * (j & 1) + lc;
      const bool ok = okb && ql < nl && m + ql > 0;
      cp16(db + st * STAGE + j * KZ * ROW, ok ? (j >> 1 ? a.spec2 : a.spec) + brow + q0 + 8 * (j & 1) : a.spec, ok);
    }
  };

  const int nmt = kz0 + gr * 8 < a.nkz ? min(2, (a.ldn - i0 + 15) / 16) : 0;
  double acc[2][4][4] = {};  // [16 nodes][Vt_re, Vt_im, -Vp_re, -Vp_im]
  const int kd = 1 - q + 2 * t, km = q + 2 * t;  // this lane's l within a block of 8, for dP and mPs
  const unsigned char *fad = sm + kd * ROW + ((g ^ kd) << 4), *fam = sm + (2 * K + km) * ROW + ((g ^ km) << 4);
  const unsigned char* fb = sm + A_B + (gr * 8 + g) * ROW;
  const int bd = (kd ^ g) << 4, bm = (km ^ g) << 4;
  auto compute = [&](int o, int mts) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const unsigned char* p = fb + o + h * KZ * ROW;
      const double2 s1 = frag(p + bd), t1 = frag(p + 2 * KZ * ROW + bd);
      const double2 s0v = frag(p + bm), t0 = frag(p + 2 * KZ * ROW + bm);
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        if (mt >= mts) continue;
        const double2 d = frag(fad + o + (mt * K + h * 8) * ROW), r = frag(fam + o + (mt * K + h * 8) * ROW);
        dmma(acc[mt][0], d.x, d.y, s1.x);
        dmma(acc[mt][1], d.x, d.y, s1.y);
        dmma(acc[mt][2], d.x, d.y, t1.x);
        dmma(acc[mt][3], d.x, d.y, t1.y);
        dmma(acc[mt][1], r.x, r.y, t0.x);
        dmma(acc[mt][2], r.x, r.y, s0v.y);
        dmma(acc[mt][0], -r.x, -r.y, t0.y);
        dmma(acc[mt][3], -r.x, -r.y, s0v.x);
      }
    }
  };

  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nk) load(s, s * K);
    cp_commit();
  }
  for (int kt = 0, st = 0; kt < nk; ++kt, st = st + 1 == STAGES ? 0 : st + 1) {
    cp_wait<STAGES - 2>();
    __syncthreads();
    const int nx = kt + STAGES - 1;
    if (nx < nk) load(st == 0 ? STAGES - 1 : st - 1, nx * K);
    cp_commit();
    if (nmt == 2) compute(st * STAGE, 2);
    else if (nmt == 1) compute(st * STAGE, 1);
  }
  cp_wait<0>();

  double2* G = a.Gw + a.Gfield + ((size_t)m * 2 + q) * a.nz * a.ldn;  // field 1: v_theta, 2: v_phi
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    bool okz;
    const int kz = plane_of(a, kz0 + gr * 8 + 2 * t + c, okz);
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      const int i = i0 + mt * 16 + 2 * g;
      if (!okz || i >= a.ldn) continue;
      double2* o = G + (size_t)kz * a.ldn + i;
      store2(o, acc[mt][0][c], acc[mt][1][c], acc[mt][0][2 + c], acc[mt][1][2 + c]);
      store2(o + a.Gfield, -acc[mt][2][c], -acc[mt][3][c], -acc[mt][2][2 + c], -acc[mt][3][2 + c]);
    }
  }
}

// kz: planes per CTA of the kernel
LegArgs base_args(const sph_plan* p, int kz) {
  LegArgs a = {};
  a.P = p->P;
  a.dP = p->dP;
  a.mPs = p->mPs;
  a.G = p->G;
  a.Gw = p->G;
  a.Gfield = p->Gfield;
  a.mbase = p->d_mbase;
  a.lmax = p->lmax;
  a.nlat2 = p->nlat2;
  a.ldn = p->ldn;
  a.nz = p->nz;
  a.nlm = p->nlm;
  a.kzl = p->sel_kz;
  a.nkz = p->sel_kz ? p->sel_n : p->nz;
  a.nkb = (a.nkz + kz - 1) / kz;
  return a;
}

template <typename K>
bool set_smem(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess &&
         cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100) == cudaSuccess;
}

}  // namespace

int launch_leg_analysis(const sph_plan* p, int gfield, double2* spec, cudaStream_t st) {
  LegArgs a = base_args(p, an::KZ);
  a.gfield = gfield;
  a.out = spec;
  a.tiles = p->tilesA;
  static DeviceOnce once;
  if (!once.run([] { return set_smem(leg_analysis_kernel<false>, an::SMEM); })) return SPH_ECUDA;
  TimedLaunch tl(p, T_LEG_ANA, st);
  launch_dependent(leg_analysis_kernel<false>, p->ntilesA * a.nkb, 128, an::SMEM, st, a, LegGroup{});
  SPH_LAUNCH_OK();
  return SPH_OK;
}

int launch_leg_synthesis(const sph_plan* p, const double2* spec, int gfield, cudaStream_t st) {
  LegArgs a = base_args(p, sy::KZ);
  a.gfield = gfield;
  a.spec = spec;
  a.tiles = p->tilesS;
  static DeviceOnce once;
  if (!once.run([] { return set_smem(leg_synthesis_kernel<false>, sy::SMEM); })) return SPH_ECUDA;
  TimedLaunch tl(p, T_LEG_SYN, st);
  launch_dependent(leg_synthesis_kernel<false>, p->ntilesS * a.nkb, 128, sy::SMEM, st, a, LegGroup{});
  SPH_LAUNCH_OK();
  return SPH_OK;
}

int launch_vec_analysis(const sph_plan* p, double2* s, double2* t, cudaStream_t st) {
  LegArgs a = base_args(p, va::KZ);
  a.out = s;
  a.out2 = t;
  a.tiles = p->tilesA64;
  static DeviceOnce once;
  if (!once.run([] { return set_smem(vec_analysis_kernel, va::SMEM); })) return SPH_ECUDA;
  TimedLaunch tl(p, T_VEC_ANA, st);
  launch_dependent(vec_analysis_kernel, p->ntilesA64 * a.nkb, va::THREADS, va::SMEM, st, a);
  SPH_LAUNCH_OK();
  return SPH_OK;
}

int launch_vec_synthesis(const sph_plan* p, const double2* s, const double2* t, cudaStream_t st) {
  LegArgs a = base_args(p, vs::KZ);
  a.spec = s;
  a.spec2 = t;
  a.tiles = p->tilesS32;
  static DeviceOnce once;
  if (!once.run([] { return set_smem(vec_synthesis_kernel, vs::SMEM); })) return SPH_ECUDA;
  TimedLaunch tl(p, T_VEC_SYN, st);
  launch_dependent(vec_synthesis_kernel, p->ntilesS32 * a.nkb, vs::THREADS, vs::SMEM, st, a);
  SPH_LAUNCH_OK();
  return SPH_OK;
}

// ---------------------------------------------------------------- grouped launches
int leg_group_prepare(bool analysis, const std::vector<GroupJob>& jobs, GroupLaunch* g) {
  std::vector<LegArgs> args;
  std::vector<int> prefix;
  long long total = 0;
  for (const GroupJob& j : jobs) {
    if (j.p->precision != SPH_FP64 || j.field < 0 || j.field >= SPH_MAX_FIELDS) return SPH_EINVAL;
    LegArgs a = base_args(j.p, analysis ? an::KZ : sy::KZ);
    a.gfield = j.field;
    if (analysis) {
      a.out = j.spec;
      a.tiles = j.p->tilesA;
    } else {
      a.spec = j.spec;
      a.tiles = j.p->tilesS;
    }
    prefix.push_back((int)total);
    total += (long long)(analysis ? j.p->ntilesA : j.p->ntilesS) * a.nkb;
    args.push_back(a);
  }
  if (total > (1ll << 30)) return SPH_EINVAL;
  g->analysis = analysis;
  g->njobs = (int)jobs.size();
  g->total = (int)total;
  g->grid = (int)total;
  if (jobs.empty()) return SPH_OK;
  if (cudaMalloc(&g->jobs, args.size() * sizeof(LegArgs)) != cudaSuccess ||
      cudaMalloc((void**)&g->prefix, prefix.size() * sizeof(int)) != cudaSuccess)
    return SPH_ENOMEM;
  if (cudaMemcpy(g->jobs, args.data(), args.size() * sizeof(LegArgs), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(g->prefix, prefix.data(), prefix.size() * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess)
    return SPH_ECUDA;
  return SPH_OK;
}

int leg_group_launch(const GroupLaunch& g, cudaStream_t st) {
  if (g.total == 0) return SPH_OK;
  const LegGroup grp{static_cast<const LegArgs*>(g.jobs), g.prefix, g.njobs};
  if (g.analysis) {
    static DeviceOnce once;
    if (!once.run([] { return set_smem(leg_analysis_kernel<true>, an::SMEM); })) return SPH_ECUDA;
    launch_dependent(leg_analysis_kernel<true>, g.grid, 128, an::SMEM, st, LegArgs{}, grp);
  } else {
    static DeviceOnce once;
    if (!once.run([] { return set_smem(leg_synthesis_kernel<true>, sy::SMEM); })) return SPH_ECUDA;
    launch_dependent(leg_synthesis_kernel<true>, g.grid, 128, sy::SMEM, st, LegArgs{}, grp);
  }
  SPH_LAUNCH_OK();
  return SPH_OK;
}

void group_free(GroupLaunch* g) {
  if (g->jobs) cudaFree(g->jobs);
  if (g->prefix) cudaFree(g->prefix);
  g->jobs = nullptr;
  g->prefix = nullptr;
  g->njobs = g->total = g->grid = 0;
}
