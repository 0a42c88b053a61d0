// kmhd_leg_f64.cu -- FP64 equator-symmetric Legendre transforms on the FP64
// tensor pipe (mma.sync m8n8k4 f64, DMMA).
//
// Backward (reference: leg_b_trans_vec_sym_dgemm / leg_b_trans_scl_sym_dgemm,
// PARALLEL_src/SPH_SHELL_src/legendre_bwd_sym_matmul.f90:301-500, with the
// pack of set_sp_rlm_for_leg_matmul.f90:153-276 and the unpack of
// cal_vr_rtm_by_matmul.f90:163-352).  Per order m >= 0, per parity p of l-m:
//   V(theta, col) = sum_k Ptab[m][p][k][theta] * SB[m][p][k][col]
// for P and dP, then the N/S (sym +/- asym) recombination and the +-m cross
// terms are applied in registers and the grid spectra are written to
// the rtm_b records (layout: rtm_off, rtm_pair).
//
// Forward (leg_f_trans_vec_sym_dgemm, legendre_fwd_sym_matmul.f90:315-452,
// pack set_vr_rtm_for_leg_matmul.f90:170-364, unpack cal_sp_rlm_by_matmul.f90:172-360):
//   S(k, col) = sum_theta Ptab[m][p][k][theta] * X[m][p][theta][col]
// where X = (N +- S) * w (* 1/sin theta) is formed while staging rtm_f into
// shared memory, and the r, r^2, g7, g6, m factors are applied in the epilogue
// before the scatter into d_rj.
//
// Column blocks hold kRB = 4 radii of every field ("quads"): a vector quad has
// three 8-column tiles X = (b+, b-), Y = (c+, c-), Z = (a+, a-) per radius in the
// backward direction (a = S g3 / r^2, b = dS/dr / r, c = T / r), so the m8n8
// accumulator fragment of a thread (row g, columns 2t, 2t+1) holds the cos and
// sin slots of one radius.
#include <algorithm>
#include <type_traits>

#include "kmhd_internal.cuh"

namespace kmhd {
namespace {

template <int NV, int NS>
struct BwdGeo {
  static constexpr int CB = 24 * NV + 8 * NS;                       // columns per r-block
  // row strides = 32 B mod 128 B: a half warp (4 fragment rows x 32 B) spans all banks
  static constexpr int CBp = CB + ((4 - CB % 16) + 16) % 16;
  static constexpr int AS = kThBlk + 4;                              // A row stride (doubles)
  static constexpr int A_STAGE = 2 * kKC * AS;                       // P and dP
  static constexpr int B_STAGE = kKC * CBp;
  static constexpr size_t SMEM = sizeof(double) * 2 * (A_STAGE + B_STAGE);
  // both parities per stage, and two chunk pairs' recurrence coefficients
  static constexpr size_t SMEM_OTF = sizeof(double) * 4 * (A_STAGE + B_STAGE) + sizeof(double2) * 16 * kKC;
};

// ---------------------------------------------------------------------------
// d_rj -> SB packing.  CTA = (m, 32-wide l chunk, r block); both parities.  Warp
// (slot, radius u), lane = degree: the loads of every column go out together,
// the scaled values meet in shared memory and leave as whole SB rows.
// One item per thread in turn, with run-time divisions and a dependent chain of
// loads each, took 0.478 ms at L = 511, Nr = 17 where this takes 0.153.
template <int NV, int NS>
__global__ void __launch_bounds__(kThreads) k_pack_b(const __grid_constant__ Plan p, const double* __restrict__ d_rj,
                                                     long long ld, const int* __restrict__ cols) {
  constexpr int CB = 24 * NV + 8 * NS, ST = CB + 1;  // odd row stride: lanes (degrees) in different banks
  extern __shared__ double sm[];
  const int m = blockIdx.y;
  const int nrbw = win_nrb(p);
  const int lc = blockIdx.x / nrbw;
  const int rb = win_rb0(p) + blockIdx.x % nrbw;
  if (lc >= p.kpad[2 * m] / kKC) return;  // chunks of 32 l (16 k per parity)
  const int L = p.L;
  const int warp = threadIdx.x >> 5, lo = threadIdx.x & 31;
  static_assert(kWarps == 2 * kRB, "one warp per slot and radius");
  const int slot = warp / kRB, u = warp % kRB;
  const int l = m + 32 * lc + lo, r = kRB * rb + u;
  const bool ok = l <= L && r < p.nr && (slot == 0 || m > 0);
  const double* src = d_rj + (ok ? p.jmap[((long long)m * 2 + slot) * (L + 1) + l] + p.J * r : 0);
  double x[NV > 0 ? NV : 1][3], xs[NS > 0 ? NS : 1];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const double* c = src + ld * __ldg(cols + v);
#pragma unroll
    for (int q = 0; q < 3; ++q) x[v][q] = ok ? __ldg(c + q * ld) : 0.0;
  }
#pragma unroll
  for (int s = 0; s < NS; ++s) xs[s] = ok ? __ldg(src + ld * __ldg(cols + NV + s)) : 0.0;
  const double ar = r < p.nr ? 1.0 / p.radius[r] : 0.0;
  double* row = sm + lo * ST + 2 * u + slot;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    row[24 * v] = x[v][1] * ar;                        // dpoldt = dS/dr / r
    row[24 * v + 8] = x[v][2] * ar;                    // dtordt = T / r
    row[24 * v + 16] = x[v][0] * (ar * ar) * g3_of(l);  // pol = S / r^2 * g3
  }
#pragma unroll
  for (int s = 0; s < NS; ++s) row[24 * NV + 8 * s] = xs[s];
  __syncthreads();
#pragma unroll 5
  for (int it = threadIdx.x; it < 32 * CB; it += kThreads) {
    const int ll = it / CB, c = it - ll * CB;
    const int par = ll & 1, k = kKC * lc + (ll >> 1);
    if (k < p.kpad[2 * m + par])
      p.SB[p.sboff[2 * m + par] + (long long)k * (p.nrb * CB) + rb * CB + c] = sm[ll * ST + c];
  }
}

// +-m cross terms of a vector: products a(tile, parity, slot), tiles XP, XdP, YP, YdP, ZP, slots cos, sin ->
// (theta cos, theta sin, phi cos, phi sin), equator-symmetric and antisymmetric.
// theta: own slot dP*b, mirror slot -/+ m/sin * P*c;
// phi: own slot -dP*c, mirror slot +/- m/sin * P*b
template <typename F>
__device__ __forceinline__ void cross_terms(F a, double ms, double (&sy)[4], double (&as)[4]) {
  sy[0] = a(1, 1, 0) + ms * a(2, 0, 1);
  sy[1] = a(1, 1, 1) - ms * a(2, 0, 0);
  sy[2] = -a(3, 1, 0) + ms * a(0, 0, 1);
  sy[3] = -a(3, 1, 1) - ms * a(0, 0, 0);
  as[0] = a(1, 0, 0) + ms * a(2, 1, 1);
  as[1] = a(1, 0, 1) - ms * a(2, 1, 0);
  as[2] = -a(3, 0, 0) + ms * a(0, 1, 1);
  as[3] = -a(3, 0, 1) - ms * a(0, 1, 0);
}

// ---------------------------------------------------------------------------
constexpr int kGenThreadsB = 64;  // generator warps of the on-the-fly backward kernel (one per latitude)

// OTF: P / dP of the CTA's 64 latitudes come from two generator warps that run
// the recurrence one chunk pair ahead of the tensor warps (chunk pair c = the
// parity-0 and parity-1 chunks c, i.e. l = m + 32c .. m + 32c + 31); each
// parity still accumulates its chunks in order, so only P's last bits differ
// from the stored-table kernel.
template <int NV, int NS, bool OTF>
__global__ void __launch_bounds__(kThreads + (OTF ? kGenThreadsB : 0), 1) k_leg_bwd_f64(Plan p) {
  using G = BwdGeo<NV, NS>;
  extern __shared__ double sm[];
  double* sA = sm;                                   // [2 stages][(OTF: 2 parities)][2][kKC][AS]
  double* sB = sm + (OTF ? 4 : 2) * G::A_STAGE;      // [2 stages][(OTF: 2 parities)][kKC][CBp]
  const int nthb = p.nh_pad / kThBlk;
  int b = blockIdx.x;
  const int nrbw = win_nrb(p);
  const int rb = win_rb0(p) + b % nrbw;
  b /= nrbw;
  const int thb = b % nthb;
  const int m = b / nthb;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int th0 = thb * kThBlk;
  const int n0 = p.kpad[2 * m] / kKC, n1 = p.kpad[2 * m + 1] / kKC;
  const int total = n0 + n1;
  const long long rowB = (long long)p.nrb * G::CB;

  auto loadB = [&](double* bs, int par, int ch) {
    const double* Bg = p.SB + p.sboff[2 * m + par] + (long long)(ch * kKC) * rowB + rb * G::CB;
    for (int it = tid; it < kKC * (G::CB / 2); it += kThreads) {
      const int row = it / (G::CB / 2), c2 = it % (G::CB / 2);
      cp_async16(bs + row * G::CBp + 2 * c2, Bg + (long long)row * rowB + 2 * c2);
    }
  };
  auto load = [&](int stage, int step) {
    const int par = step < n0 ? 0 : 1;
    const int ch = step < n0 ? step : step - n0;
    const double* Pg = p.P + p.poff[2 * m + par] + (long long)(ch * kKC) * p.nh_pad + th0;
    const double* dPg = p.dP + p.poff[2 * m + par] + (long long)(ch * kKC) * p.nh_pad + th0;
    double* a = sA + stage * G::A_STAGE;
    // 2 tables x 16 rows x 64 doubles = 2 x 16 x 32 chunks of 16 B
    for (int it = tid; it < 2 * kKC * (kThBlk / 2); it += kThreads) {
      const int tb = it / (kKC * (kThBlk / 2));
      const int rem = it % (kKC * (kThBlk / 2));
      const int row = rem / (kThBlk / 2), c2 = rem % (kThBlk / 2);
      const double* src = (tb ? dPg : Pg) + (long long)row * p.nh_pad + 2 * c2;
      cp_async16(a + tb * kKC * G::AS + row * G::AS + 2 * c2, src);
    }
    loadB(sB + stage * G::B_STAGE, par, ch);
  };

  // accumulators: [field][tile][parity][2]; tiles XP, XdP, YP, YdP, ZP
  double acc[NV > 0 ? NV : 1][5][2][2];
  double accS[NS > 0 ? NS : 1][2][2];
#pragma unroll
  for (int v = 0; v < (NV > 0 ? NV : 1); ++v)
#pragma unroll
    for (int q = 0; q < 5; ++q)
#pragma unroll
      for (int s = 0; s < 2; ++s) acc[v][q][s][0] = acc[v][q][s][1] = 0.0;
#pragma unroll
  for (int v = 0; v < (NS > 0 ? NS : 1); ++v)
#pragma unroll
    for (int s = 0; s < 2; ++s) accS[v][s][0] = accS[v][s][1] = 0.0;

  auto compute = [&](const double* a, const double* bs, auto parc) {
    constexpr int par = decltype(parc)::value;
#pragma unroll
    for (int kk = 0; kk < kKC / 4; ++kk) {
      const int kr = 4 * kk + t;
      const double aP = a[kr * G::AS + warp * 8 + g];
      const double adP = a[kKC * G::AS + kr * G::AS + warp * 8 + g];
      const double* brow = bs + kr * G::CBp + g;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const double bX = brow[24 * v + 0], bY = brow[24 * v + 8], bZ = brow[24 * v + 16];
        dmma(acc[v][0][par][0], acc[v][0][par][1], aP, bX);
        dmma(acc[v][1][par][0], acc[v][1][par][1], adP, bX);
        dmma(acc[v][2][par][0], acc[v][2][par][1], aP, bY);
        dmma(acc[v][3][par][0], acc[v][3][par][1], adP, bY);
        dmma(acc[v][4][par][0], acc[v][4][par][1], aP, bZ);
      }
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const double bS = brow[24 * NV + 8 * s];
        dmma(accS[s][par][0], accS[s][par][1], aP, bS);
      }
    }
  };

  if constexpr (!OTF) {
    if (total > 0) {
      load(0, 0);
      cp_async_commit();
    }
    for (int step = 0; step < total; ++step) {
      if (step + 1 < total) {
        load((step + 1) & 1, step + 1);
        cp_async_commit();
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      const double* a = sA + (step & 1) * G::A_STAGE;
      const double* bs = sB + (step & 1) * G::B_STAGE;
      if (step < n0) compute(a, bs, std::integral_constant<int, 0>());
      else compute(a, bs, std::integral_constant<int, 1>());
      __syncthreads();
    }
  } else {
    const bool gen = warp >= kWarps;
    const int gi = tid - kThreads, ig = th0 + gi;  // generator thread: latitude ig
    double st6[6];
    double ct = 0.0;
    if (gen) {
      const double* sd = p.pseed + p.pseed_off[m] * 6 * p.nh_pad + ig;  // block 0: before l = m
#pragma unroll
      for (int q = 0; q < 6; ++q) st6[q] = sd[(long long)q * p.nh_pad];
      if (ig < p.nh) ct = p.cos_t[ig];
    }
    // recurrence coefficients of a chunk pair's 32 degrees, [2 buffers][j][4];
    // each call prefetches the next pair's into registers while it steps
    double2* cb = reinterpret_cast<double2*>(sm + 4 * (G::A_STAGE + G::B_STAGE));
    constexpr int kCE = 8 * kKC;  // coefficient pairs of one chunk pair
    if (gen)
      for (int e = gi; e < kCE; e += kGenThreadsB) cb[e] = pgen_coef(p, m, m + (e >> 2), e & 3);
    auto genA = [&](int stage, int c) {
      double* a = sA + stage * 2 * G::A_STAGE;
      asm volatile("bar.sync 1, %0;\n" ::"n"(kGenThreadsB));  // cb[c & 1] complete
      double2 nx[kCE / kGenThreadsB];
#pragma unroll
      for (int q = 0; q < kCE / kGenThreadsB; ++q) {
        const int e = gi + q * kGenThreadsB;
        nx[q] = c + 1 < n0 ? pgen_coef(p, m, m + 2 * kKC * (c + 1) + (e >> 2), e & 3) : make_double2(0.0, 0.0);
      }
      const double2* cc = cb + (c & 1) * kCE;
      const int l0 = m + 2 * kKC * c;
      const int nj = min(2 * kKC, p.L - l0 + 1);
      if (l0 >= m + 3 && ig < p.nh) {
#pragma unroll 4
        for (int j = 0; j < 2 * kKC; ++j) {
          double pv = 0.0, dpv = 0.0;
          if (j < nj) pgen_step_fast(st6, ct, cc + 4 * j, pv, dpv);
          double* ap = a + (j & 1) * G::A_STAGE + (j >> 1) * G::AS + gi;
          ap[0] = pv;
          ap[kKC * G::AS] = dpv;
        }
      } else {
        for (int j = 0; j < 2 * kKC; ++j) {
          double pv = 0.0, dpv = 0.0;
          if (j < nj && ig < p.nh) pgen_step(st6, p, m, l0 + j, ct, ig, cc + 4 * j, pv, dpv);
          double* ap = a + (j & 1) * G::A_STAGE + (j >> 1) * G::AS + gi;
          ap[0] = pv;
          ap[kKC * G::AS] = dpv;
        }
      }
      double2* cn = cb + ((c + 1) & 1) * kCE;
#pragma unroll
      for (int q = 0; q < kCE / kGenThreadsB; ++q) cn[gi + q * kGenThreadsB] = nx[q];
    };
    auto loadB2 = [&](int stage, int c) {
      loadB(sB + (2 * stage) * G::B_STAGE, 0, c);
      if (c < n1) loadB(sB + (2 * stage + 1) * G::B_STAGE, 1, c);
    };
    // separate loops (same __syncthreads count), so the generator state is
    // not live in the tensor warps
    if (gen) {
      genA(0, 0);
      for (int c = 0; c < n0; ++c) {
        __syncthreads();
        if (c + 1 < n0) genA((c + 1) & 1, c + 1);
      }
      return;  // the generator warps take no part in the epilogue
    }
    loadB2(0, 0);
    cp_async_commit();
    for (int c = 0; c < n0; ++c) {
      cp_async_wait<0>();
      __syncthreads();
      if (c + 1 < n0) {
        loadB2((c + 1) & 1, c + 1);
        cp_async_commit();
      }
      const double* a = sA + (c & 1) * 2 * G::A_STAGE;
      const double* bs = sB + (c & 1) * 2 * G::B_STAGE;
      compute(a, bs, std::integral_constant<int, 0>());
      if (c < n1) compute(a + G::A_STAGE, bs + G::B_STAGE, std::integral_constant<int, 1>());
    }
  }

  // ---- epilogue: N/S recombination and +-m cross terms
  const int i = th0 + warp * 8 + g;
  const int r = kRB * rb + t;
  if (i >= p.nh || r >= p.nr) return;
  const bool pair = i < p.nth / 2;
  const double ms = (double)m * p.asin_t[i];
  const int nc = p.ncb;
  double* outN = p.rtm_b + rtm_off(p, m, i, r, nc);
  double* outS = p.rtm_b + rtm_off(p, m, p.nth - 1 - i, r, nc);
  const bool al = rtm_aligned(p, nc);
  // (sym, asym) cos and sin of one component -> north and south values
  auto put = [&](int q, const double (&sy)[4], const double (&as)[4]) {
    const int o = rtm_pair(p, m, q, nc);
    if (pair) {
      st_sector(outN + o, al, sy[0] + as[0], sy[1] + as[1], sy[2] + as[2], sy[3] + as[3]);
      st_sector(outS + o, al, sy[0] - as[0], sy[1] - as[1], sy[2] - as[2], sy[3] - as[3]);
    } else {
      st_sector(outN + o, al, sy[0], sy[1], sy[2], sy[3]);
    }
  };
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    double sy[4], as[4];
    cross_terms([&](int tile, int par, int slot) { return acc[v][tile][par][slot]; }, ms, sy, as);
    put(v, sy, as);
  }
  // radial components and scalars, two list entries per pair
  constexpr int NF = NV + NS;
#pragma unroll
  for (int f = 0; f < NF; f += 2) {
    double sy[4] = {0.0, 0.0, 0.0, 0.0}, as[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int ff = f + e;
      if (ff >= NF) break;
      const double(&c)[2][2] = ff < NV ? acc[ff < NV ? ff : 0][4] : accS[ff < NV ? 0 : ff - NV];
      sy[2 * e] = c[0][0];
      sy[2 * e + 1] = c[0][1];
      as[2 * e] = c[1][0];
      as[2 * e + 1] = c[1][1];
    }
    if (f + 1 < NF) {
      put(NV + f / 2, sy, as);
    } else {  // odd count: the last pair holds one component
      const int o = rtm_pair(p, m, NV + f / 2, nc);
      *reinterpret_cast<double2*>(outN + o) =
          pair ? make_double2(sy[0] + as[0], sy[1] + as[1]) : make_double2(sy[0], sy[1]);
      if (pair) *reinterpret_cast<double2*>(outS + o) = make_double2(sy[0] - as[0], sy[1] - as[1]);
    }
  }
}

// ---------------------------------------------------------------------------
template <int NV, int NS>
struct FwdGeo {
  static constexpr int CF = 40 * NV + 8 * NS;
  static constexpr int CFp = CF + ((4 - CF % 16) + 16) % 16;
  static constexpr int AS = kKC + 4;                      // 160 B rows
  static constexpr int A_TILE = kLBlk * AS;
  static constexpr int B_TILE = kKC * CFp;
  static constexpr size_t SMEM = sizeof(double) * (4 * A_TILE + 2 * B_TILE);
  // A double-buffered, the block's recurrence coefficients and two chunks' seeds
  static constexpr size_t SMEM_OTF =
      sizeof(double) * (8 * A_TILE + 2 * B_TILE) + sizeof(double2) * 8 * kLBlk + sizeof(double) * 2 * 2 * 6 * kKC;
};

// OTF: the A tiles (P / dP of the block's 64 degrees at 16 latitudes) are
// generated by warp 0 one latitude chunk ahead, each latitude's recurrence
// starting from the seeds at the block's two 32-degree halves.
// Two CTAs per SM while the accumulators fit in 128 registers (up to ten
// components); one CTA with the whole register file for more (four or five
// vectors: 42-52 accumulators per lane), which would otherwise spill.
template <int NV, int NS, bool OTF>
__global__ void __launch_bounds__(kThreads, 3 * NV + NS > 10 ? 1 : 2)
k_leg_fwd_f64(Plan p, double* __restrict__ d_rj, long long ld, const int* __restrict__ cols) {
  using G = FwdGeo<NV, NS>;
  extern __shared__ double sm[];
  double* sA = sm;                              // [(OTF: 2 stages)][P_e, P_o, dP_e, dP_o][kLBlk][AS]
  double* sB = sm + (OTF ? 8 : 4) * G::A_TILE;  // [par][kKC][CFp]
  const int m = blockIdx.y;
  const int nrbw = win_nrb(p);
  const int kb = blockIdx.x / nrbw;
  const int rb = win_rb0(p) + blockIdx.x % nrbw;
  const int K0 = kcount(p.L, m, 0);
  if (kb * kLBlk >= K0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int par = warp & 1, rgi = warp >> 1;
  const int nc = p.ncf;
  const int nchunk = p.nh_pad / kKC;

  double acc[NV > 0 ? NV : 1][5][2];
  double accS[NS > 0 ? NS : 1][2];
#pragma unroll
  for (int v = 0; v < (NV > 0 ? NV : 1); ++v)
#pragma unroll
    for (int q = 0; q < 5; ++q) acc[v][q][0] = acc[v][q][1] = 0.0;
#pragma unroll
  for (int s = 0; s < (NS > 0 ? NS : 1); ++s) accS[s][0] = accS[s][1] = 0.0;

  constexpr int kItems = (kKC * kRB * (3 * NV + NS) + kThreads - 1) / kThreads;
  double2 pfN[kItems], pfS[kItems];
  // item it = tid + q kThreads of a chunk is (latitude row, radius u, component
  // in record order e), the same in every chunk: decomposed once, packed as
  // e | u << 8 | row << 12, or -1 past the chunk's items; neighbouring threads
  // read the two halves of one record sector
  constexpr int NC = 3 * NV + NS;
  int item[kItems];
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int it = tid + q * kThreads;
    const int rest = it / NC;
    item[q] = it < kKC * kRB * NC ? (it - rest * NC) | (rest % kRB) << 8 | (rest / kRB) << 12 : -1;
  }
  // global loads of one chunk's rtm_f values into registers (overlaps the MMAs)
  auto prefetch = [&](int ch) {
    const int th0 = ch * kKC;
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
      pfN[q] = make_double2(0.0, 0.0);
      pfS[q] = make_double2(0.0, 0.0);
      if (item[q] >= 0) {
        const int i = th0 + (item[q] >> 12), r = kRB * rb + ((item[q] >> 8) & 15);
        if (i < p.nh && r < p.nr) {
          const int e = item[q] & 255;
          const int ro = rtm_pair(p, m, e >> 1, nc) + 2 * (e & 1);
          pfN[q] = ld_global_v2(p.rtm_f + rtm_off(p, m, i, r, nc) + ro);
          if (i < p.nth / 2)
            pfS[q] = ld_global_v2(p.rtm_f + rtm_off(p, m, p.nth - 1 - i, r, nc) + ro);
        }
      }
    }
  };
  // OTF: warp 0 generates the next chunk's A tile (before its share of the
  // current chunk's MMAs).  Recurrence coefficients of the block's 64 degrees
  // [j][4] are loaded once; the seeds of the next chunk's 16 latitudes and two
  // 32-degree halves, [stage][half][6][kKC], arrive by cp.async a chunk ahead.
  double2* cb = reinterpret_cast<double2*>(sB + 2 * G::B_TILE);
  double* sS = reinterpret_cast<double*>(cb + 8 * kLBlk);
  const int nsd = (p.L - m + kSeedL) / kSeedL;  // seeds of order m
  auto seeds_async = [&](int stage, int ch) {
    for (int e = lane; e < 2 * 6 * (kKC / 2); e += 32) {
      const int h = e / (6 * (kKC / 2)), rem = e % (6 * (kKC / 2)), q = rem / (kKC / 2), c2 = rem % (kKC / 2);
      const int sdi = 2 * kb + h;
      if (sdi < nsd)
        cp_async16(sS + ((stage * 2 + h) * 6 + q) * kKC + 2 * c2,
                   p.pseed + ((p.pseed_off[m] + sdi) * 6 + q) * p.nh_pad + ch * kKC + 2 * c2);
    }
    cp_async_commit();
  };
  // lane: latitude ch * kKC + (lane & 15), degrees lh .. lh + 31 with
  // lh = l0 + 32 h (h = lane >> 4); block row j (l = l0 + j) is parity j & 1,
  // A row j >> 1
  auto genA = [&](int stage, int ch) {
    const int h = lane >> 4, tl = lane & 15;
    const int ig = ch * kKC + tl;
    double* a = sA + stage * 4 * G::A_TILE + tl;
    const int l0 = m + 2 * kLBlk * kb, lh = l0 + kSeedL * h;
    const int nj = min(kSeedL, p.L - lh + 1);
    const bool ok = ig < p.nh && nj > 0;
    double st6[6];
    const double* sd = sS + ((stage * 2 + h) * 6) * kKC + tl;
#pragma unroll
    for (int q = 0; q < 6; ++q) st6[q] = ok ? sd[q * kKC] : 0.0;
    const double ct = ok ? p.cos_t[ig] : 0.0;
    const double2* cc = cb + 4 * kSeedL * h;
    if (lh >= m + 3) {
#pragma unroll 4
      for (int jj = 0; jj < kSeedL; ++jj) {
        const int j = kSeedL * h + jj;
        double pv = 0.0, dpv = 0.0;
        if (ok && jj < nj) pgen_step_fast(st6, ct, cc + 4 * jj, pv, dpv);
        a[(j & 1) * G::A_TILE + (j >> 1) * G::AS] = pv;
        a[(2 + (j & 1)) * G::A_TILE + (j >> 1) * G::AS] = dpv;
      }
    } else {
      for (int jj = 0; jj < kSeedL; ++jj) {
        const int j = kSeedL * h + jj;
        double pv = 0.0, dpv = 0.0;
        if (ok && jj < nj) pgen_step(st6, p, m, lh + jj, ct, ig, cc + 4 * jj, pv, dpv);
        a[(j & 1) * G::A_TILE + (j >> 1) * G::AS] = pv;
        a[(2 + (j & 1)) * G::A_TILE + (j >> 1) * G::AS] = dpv;
      }
    }
  };
  if (OTF && warp == 0) {
    for (int e = lane; e < 8 * kLBlk; e += 32) cb[e] = pgen_coef(p, m, m + 2 * kLBlk * kb + (e >> 2), e & 3);
    seeds_async(0, 0);
    cp_async_wait<0>();
    __syncwarp();
    genA(0, 0);
    if (nchunk > 1) seeds_async(1, 1);
  }
  prefetch(0);
  for (int ch = 0; ch < nchunk; ++ch) {
    const int th0 = ch * kKC;
    // A: 4 tables x 32 k-rows x 16 theta
    for (int it = tid; !OTF && it < 4 * kLBlk * (kKC / 2); it += kThreads) {
      const int tb = it / (kLBlk * (kKC / 2));   // 0 P_e, 1 P_o, 2 dP_e, 3 dP_o
      const int rem = it % (kLBlk * (kKC / 2));
      const int row = rem / (kKC / 2), c2 = rem % (kKC / 2);
      const int pp = tb & 1;
      const int k = kb * kLBlk + row;
      double* dst = sA + tb * G::A_TILE + row * G::AS + 2 * c2;
      if (k < p.kpad[2 * m + pp]) {
        const double* src = (tb < 2 ? p.P : p.dP) + p.poff[2 * m + pp] + (long long)k * p.nh_pad + th0 + 2 * c2;
        cp_async16(dst, src);
      } else {
        dst[0] = 0.0;
        dst[1] = 0.0;
      }
    }
    cp_async_commit();
    // B: sym/asym with weights from the prefetched registers
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
      if (item[q] < 0) continue;
      const int c = item[q] & 255, u = (item[q] >> 8) & 15, row = item[q] >> 12;
      const int i = th0 + row;
      const int r = kRB * rb + u;
      double2 sy = make_double2(0.0, 0.0), as = sy, syn = sy, asn = sy;
      if (i < p.nh && r < p.nr) {
        const double wp = p.weight[i], ai = p.asin_t[i];
        const double2 nv = pfN[q];
        if (i < p.nth / 2) {
          const double2 sv = pfS[q];
          sy = make_double2((nv.x + sv.x) * wp, (nv.y + sv.y) * wp);
          as = make_double2((nv.x - sv.x) * wp, (nv.y - sv.y) * wp);
          syn = make_double2((nv.x + sv.x) * wp * ai, (nv.y + sv.y) * wp * ai);
          asn = make_double2((nv.x - sv.x) * wp * ai, (nv.y - sv.y) * wp * ai);
        } else {  // equator row
          sy = make_double2(nv.x * wp, nv.y * wp);
          syn = make_double2(nv.x * wp * ai, nv.y * wp * ai);
        }
      }
      double* b0 = sB + row * G::CFp;               // parity 0
      double* b1 = sB + G::B_TILE + row * G::CFp;   // parity 1
      if (c < 2 * NV) {
        const int v = c >> 1;
        const int base = 40 * v + 2 * u;
        if ((c & 1) == 0) {       // theta: U' tile (P, /sin), W tile (dP)
          *reinterpret_cast<double2*>(b0 + base + 16) = syn;
          *reinterpret_cast<double2*>(b1 + base + 16) = asn;
          *reinterpret_cast<double2*>(b0 + base + 24) = as;
          *reinterpret_cast<double2*>(b1 + base + 24) = sy;
        } else {                  // phi: U tile (P, /sin), W' tile (dP)
          *reinterpret_cast<double2*>(b0 + base + 8) = syn;
          *reinterpret_cast<double2*>(b1 + base + 8) = asn;
          *reinterpret_cast<double2*>(b0 + base + 32) = as;
          *reinterpret_cast<double2*>(b1 + base + 32) = sy;
        }
      } else {                    // list entry f: r of a vector (Zr tile, P) or a scalar
        const int f = c - 2 * NV;
        const int base = (f < NV ? 40 * f : 40 * NV + 8 * (f - NV)) + 2 * u;
        *reinterpret_cast<double2*>(b0 + base) = sy;
        *reinterpret_cast<double2*>(b1 + base) = as;
      }
    }
    if (ch + 1 < nchunk) prefetch(ch + 1);
    if (!OTF) cp_async_wait<0>();
    __syncthreads();
    if (OTF && warp == 0 && ch + 1 < nchunk) {
      cp_async_wait<0>();  // seeds of chunk ch + 1
      __syncwarp();
      if (ch + 2 < nchunk) seeds_async(ch & 1, ch + 2);
      genA((ch + 1) & 1, ch + 1);
    }
    const double* sAc = sA + (OTF ? (ch & 1) * 4 * G::A_TILE : 0);
    const double* aP = sAc + par * G::A_TILE + (rgi * 8 + g) * G::AS;
    const double* adP = sAc + (2 + par) * G::A_TILE + (rgi * 8 + g) * G::AS;
    const double* bb = sB + par * G::B_TILE;
#pragma unroll
    for (int kk = 0; kk < kKC / 4; ++kk) {
      const double a = aP[4 * kk + t], ad = adP[4 * kk + t];
      const double* brow = bb + (4 * kk + t) * G::CFp + g;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        dmma(acc[v][0][0], acc[v][0][1], a, brow[40 * v + 0]);    // Zr
        dmma(acc[v][1][0], acc[v][1][1], a, brow[40 * v + 8]);    // U
        dmma(acc[v][2][0], acc[v][2][1], a, brow[40 * v + 16]);   // U'
        dmma(acc[v][3][0], acc[v][3][1], ad, brow[40 * v + 24]);  // W
        dmma(acc[v][4][0], acc[v][4][1], ad, brow[40 * v + 32]);  // W'
      }
#pragma unroll
      for (int s = 0; s < NS; ++s) dmma(accS[s][0], accS[s][1], a, brow[40 * NV + 8 * s]);
    }
    __syncthreads();
  }

  // ---- epilogue (cal_sp_rlm_vector_sym_matmul / _scalar_)
  const int k = kb * kLBlk + rgi * 8 + g;
  const int l = m + 2 * k + par;
  const int r = kRB * rb + t;
  if (l > p.L || r >= p.nr) return;
  const double r1 = p.radius[r], r2 = r1 * r1;
  const double g7 = g7_of(l, m), gm = (double)m;
  const long long jp = p.jmap[((long long)m * 2 + 0) * (p.L + 1) + l] + p.J * r;
  const long long jn = m > 0 ? p.jmap[((long long)m * 2 + 1) * (p.L + 1) + l] + p.J * r : -1;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    double* o = d_rj + ld * cols[v];
    // + slot (cos), gm = +m
    o[jp] = acc[v][0][0] * r2 * g7;
    o[jp + ld] = acc[v][3][0] * r1 * g7 - acc[v][1][1] * r1 * g7 * gm;
    o[jp + 2 * ld] = -(acc[v][2][1] * r1 * g7 * gm) - acc[v][4][0] * r1 * g7;
    if (jn >= 0) {  // - slot (sin), gm = -m
      o[jn] = acc[v][0][1] * r2 * g7;
      o[jn + ld] = acc[v][3][1] * r1 * g7 - acc[v][1][0] * r1 * g7 * (-gm);
      o[jn + 2 * ld] = -(acc[v][2][0] * r1 * g7 * (-gm)) - acc[v][4][1] * r1 * g7;
    }
  }
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    double* o = d_rj + ld * cols[NV + s];
    const double g6 = g6_of(l, m);
    o[jp] = accS[s][0] * g6;
    if (jn >= 0) o[jn] = accS[s][1] * g6;
  }
}

// ---------------------------------------------------------------------------
// Forward kernel of the stored tables.  CTA = (m, 64 degrees per parity, 4 radii,
// field group); 8 warps = (parity, 16 degrees).  Each warp's m16n8k4 DMMAs use a
// B fragment for 16 degrees (the 8-degree kernel above reads one per 8: its
// shared-memory reads alone took 62% of the L1 data pipe at 45% DMMA), each
// staged B chunk serves 64 degrees instead of 32, and both operands are double
// buffered, so a chunk costs one barrier and its staging runs beside the other
// warps' DMMAs.  A field group holds at most three vectors (16 accumulator tiles
// of four doubles per lane; more would spill): groups share nothing but the A
// operand, so larger sets run group by group.  The sums are those of the 8-row
// kernel in the same order, so the two agree bit for bit.
constexpr int kLB16 = 64;  // degrees per parity of a CTA

template <int NV, int NS>
struct Fwd16Geo {
  static constexpr int CF = 40 * NV + 8 * NS;
  static constexpr int CFp = CF + ((4 - CF % 16) + 16) % 16;
  static constexpr int AS = kKC + 4;
  static constexpr int A_TILE = kLB16 * AS;
  static constexpr int B_TILE = kKC * CFp;
  static constexpr size_t SMEM = sizeof(double) * 2 * (4 * A_TILE + 2 * B_TILE);
};

// group: vectors v0 .. v0 + NV - 1 and scalars s0 .. s0 + NS - 1 of the plan's forward fields
template <int NV, int NS>
__global__ void __launch_bounds__(kThreads, 1)
k_leg_fwd16(const __grid_constant__ Plan p, double* __restrict__ d_rj, long long ld, const int* __restrict__ cols, int v0,
            int s0) {
  using G = Fwd16Geo<NV, NS>;
  extern __shared__ double sm[];
  double* sA = sm;                  // [2][P_e, P_o, dP_e, dP_o][kLB16][AS]
  double* sB = sm + 8 * G::A_TILE;  // [2][par][kKC][CFp]
  const int m = blockIdx.y;
  const int nrbw = win_nrb(p);
  const int kb = blockIdx.x / nrbw;
  const int rb = win_rb0(p) + blockIdx.x % nrbw;
  const int k0 = kb * kLB16;
  if (k0 >= kcount(p.L, m, 0)) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int par = warp & 1, rgi = warp >> 1;
  const int nc = p.ncf;
  const int nchunk = p.nh_pad / kKC;
  const bool active = k0 + 16 * rgi < kcount(p.L, m, par);  // else no degree of this warp exists

  double acc[NV > 0 ? NV : 1][5][4];
  double accS[NS > 0 ? NS : 1][4];
#pragma unroll
  for (int v = 0; v < (NV > 0 ? NV : 1); ++v)
#pragma unroll
    for (int q = 0; q < 5; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[v][q][e] = 0.0;
#pragma unroll
  for (int s = 0; s < (NS > 0 ? NS : 1); ++s)
#pragma unroll
    for (int e = 0; e < 4; ++e) accS[s][e] = 0.0;

  // items of a chunk: (latitude row, radius u, component e of the group in
  // record order), the same in every chunk: record offset and tile column
  // decomposed once
  constexpr int NC = 3 * NV + NS;
  constexpr int kItems = (kKC * kRB * NC + kThreads - 1) / kThreads;
  double2 pfN[kItems], pfS[kItems];
  int item[kItems];  // e | u << 8 | row << 12, or -1 past the items
  int roff[kItems];  // offset of the component inside the record
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int it = tid + q * kThreads;
    const int rest = it / NC, e = it - rest * NC;
    item[q] = it < kKC * kRB * NC ? e | (rest % kRB) << 8 | (rest / kRB) << 12 : -1;
    if (e < 2 * NV) {
      roff[q] = rtm_pair(p, m, v0 + (e >> 1), nc) + 2 * (e & 1);
    } else {
      const int f = e - 2 * NV, li = f < NV ? v0 + f : p.nvf + s0 + f - NV;
      roff[q] = rtm_pair(p, m, p.nvf + (li >> 1), nc) + 2 * (li & 1);
    }
    if (item[q] >= 0 && kRB * rb + ((item[q] >> 8) & 15) >= p.nr) item[q] |= 1 << 30;  // past the last radius: zeros
  }
  const long long rowTh = rtm_row(p, nc);
  const double* recN[kItems];
#pragma unroll
  for (int q = 0; q < kItems; ++q)
    recN[q] = p.rtm_f + rtm_off(p, m, 0, min(kRB * rb + ((item[q] >> 8) & 15), p.nr - 1), nc) + roff[q];
  auto prefetch = [&](int ch) {
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
      pfN[q] = make_double2(0.0, 0.0);
      pfS[q] = make_double2(0.0, 0.0);
      const int i = ch * kKC + ((item[q] >> 12) & 15);
      if (item[q] >= 0 && item[q] < (1 << 30) && i < p.nh) {
        pfN[q] = ld_global_v2(recN[q] + i * rowTh);
        if (i < p.nth / 2) pfS[q] = ld_global_v2(recN[q] + (p.nth - 1 - i) * rowTh);
      }
    }
  };
  const int rows0 = min(kLB16, p.kpad[2 * m] - k0), rows1 = min(kLB16, p.kpad[2 * m + 1] - k0);
  auto loadA = [&](int st, int ch) {
    // P_e, P_o, dP_e, dP_o: the degrees that exist (padded to kKC) x 16 latitudes
#pragma unroll
    for (int it = tid; it < 4 * kLB16 * (kKC / 2); it += kThreads) {
      const int tb = it / (kLB16 * (kKC / 2));
      const int rem = it % (kLB16 * (kKC / 2));
      const int row = rem / (kKC / 2), c2 = rem % (kKC / 2);
      if (row < ((tb & 1) ? rows1 : rows0))
        cp_async16(sA + (st * 4 + tb) * G::A_TILE + row * G::AS + 2 * c2,
                   (tb < 2 ? p.P : p.dP) + p.poff[2 * m + (tb & 1)] + (long long)(k0 + row) * p.nh_pad + ch * kKC + 2 * c2);
    }
    cp_async_commit();
  };
  // sym / asym of the prefetched values with the Gauss weights
  auto storeB = [&](int st, int ch) {
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
      if (item[q] < 0) continue;
      const int e = item[q] & 255, u = (item[q] >> 8) & 15, row = (item[q] >> 12) & 15;
      const int i = ch * kKC + row;
      const double wp = i < p.nh ? __ldg(p.weight + i) : 0.0;
      const double2 nv = pfN[q], sv = pfS[q];
      const bool eq = i >= p.nth / 2;  // equator row: no southern partner
      const double2 sy = make_double2((nv.x + sv.x) * wp, (nv.y + sv.y) * wp);
      const double2 as = eq ? make_double2(0.0, 0.0) : make_double2((nv.x - sv.x) * wp, (nv.y - sv.y) * wp);
      double* b0 = sB + (2 * st) * G::B_TILE + row * G::CFp;      // parity 0
      double* b1 = sB + (2 * st + 1) * G::B_TILE + row * G::CFp;  // parity 1
      if (e < 2 * NV) {
        const double ai = i < p.nh ? __ldg(p.asin_t + i) : 0.0;
        const double2 syn = make_double2(sy.x * ai, sy.y * ai), asn = make_double2(as.x * ai, as.y * ai);
        const int base = 40 * (e >> 1) + 2 * u;
        // theta: U' (P, /sin) and W (dP) tiles; phi: U (P, /sin) and W' (dP) tiles
        const int c1 = base + ((e & 1) ? 8 : 16), c2 = base + ((e & 1) ? 32 : 24);
        *reinterpret_cast<double2*>(b0 + c1) = syn;
        *reinterpret_cast<double2*>(b1 + c1) = asn;
        *reinterpret_cast<double2*>(b0 + c2) = as;
        *reinterpret_cast<double2*>(b1 + c2) = sy;
      } else {  // r of a vector (Zr tile, P) or a scalar
        const int f = e - 2 * NV;
        const int base = (f < NV ? 40 * f : 40 * NV + 8 * (f - NV)) + 2 * u;
        *reinterpret_cast<double2*>(b0 + base) = sy;
        *reinterpret_cast<double2*>(b1 + base) = as;
      }
    }
  };

  prefetch(0);
  loadA(0, 0);
  storeB(0, 0);
  if (nchunk > 1) prefetch(1);
  cp_async_wait<0>();
  __syncthreads();
  auto stage_next = [&](int ch) {
    if (ch + 1 < nchunk) {
      loadA((ch & 1) ^ 1, ch + 1);
      storeB((ch & 1) ^ 1, ch + 1);
      if (ch + 2 < nchunk) prefetch(ch + 2);
    }
  };
  auto compute = [&](int ch) {
    const int st = ch & 1;
    if (!active) return;
    const double* aP = sA + (st * 4 + par) * G::A_TILE + (rgi * 16 + g) * G::AS + t;
    const double* adP = sA + (st * 4 + 2 + par) * G::A_TILE + (rgi * 16 + g) * G::AS + t;
    const double* bb = sB + (2 * st + par) * G::B_TILE + t * G::CFp + g;
#pragma unroll
    for (int kk = 0; kk < kKC / 4; ++kk) {
      const double a0 = aP[4 * kk], a1 = aP[8 * G::AS + 4 * kk];
      const double d0 = adP[4 * kk], d1 = adP[8 * G::AS + 4 * kk];
      const double* brow = bb + 4 * kk * G::CFp;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        dmma16(acc[v][0], a0, a1, brow[40 * v + 0]);   // Zr
        dmma16(acc[v][1], a0, a1, brow[40 * v + 8]);   // U
        dmma16(acc[v][2], a0, a1, brow[40 * v + 16]);  // U'
        dmma16(acc[v][3], d0, d1, brow[40 * v + 24]);  // W
        dmma16(acc[v][4], d0, d1, brow[40 * v + 32]);  // W'
      }
#pragma unroll
      for (int s = 0; s < NS; ++s) dmma16(accS[s], a0, a1, brow[40 * NV + 8 * s]);
    }
  };
  // the two warps of a scheduler (warp, warp + 4) take staging and DMMAs in
  // opposite order, so the tensor pipe works through the staging too
  for (int ch = 0; ch < nchunk; ++ch) {
    if (warp < 4) stage_next(ch);
    compute(ch);
    if (warp >= 4) stage_next(ch);
    cp_async_wait<0>();
    __syncthreads();
  }

  // ---- epilogue (cal_sp_rlm_vector_sym_matmul / _scalar_)
  const int r = kRB * rb + t;
  if (!active || r >= p.nr) return;
  const double r1 = p.radius[r], r2 = r1 * r1, gm = (double)m;
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // accumulator rows g, g + 8
    const int l = m + 2 * (k0 + rgi * 16 + 8 * h + g) + par;
    if (l > p.L) continue;
    const double g7 = g7_of(l, m);
    const long long jp = p.jmap[((long long)m * 2 + 0) * (p.L + 1) + l] + p.J * r;
    const long long jn = m > 0 ? p.jmap[((long long)m * 2 + 1) * (p.L + 1) + l] + p.J * r : -1;
    const int e = 2 * h;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      double* o = d_rj + ld * cols[v0 + v];
      // + slot (cos), gm = +m
      o[jp] = acc[v][0][e] * r2 * g7;
      o[jp + ld] = acc[v][3][e] * r1 * g7 - acc[v][1][e + 1] * r1 * g7 * gm;
      o[jp + 2 * ld] = -(acc[v][2][e + 1] * r1 * g7 * gm) - acc[v][4][e] * r1 * g7;
      if (jn >= 0) {  // - slot (sin), gm = -m
        o[jn] = acc[v][0][e + 1] * r2 * g7;
        o[jn + ld] = acc[v][3][e + 1] * r1 * g7 - acc[v][1][e] * r1 * g7 * (-gm);
        o[jn + 2 * ld] = -(acc[v][2][e] * r1 * g7 * (-gm)) - acc[v][4][e + 1] * r1 * g7;
      }
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      double* o = d_rj + ld * cols[p.nvf + s0 + s];
      const double g6 = g6_of(l, m);
      o[jp] = accS[s][e] * g6;
      if (jn >= 0) o[jn] = accS[s][e + 1] * g6;
    }
  }
}

template <int NV, int NS>
cudaError_t run_fwd16(const Plan& p, double* d_rj, long long ld, const int* cols, cudaStream_t s, int m_count, int v0,
                      int s0) {
  auto kern = k_leg_fwd16<NV, NS>;
  const size_t smem = Fwd16Geo<NV, NS>::SMEM;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int nkb = (kcount(p.L, 0, 0) + kLB16 - 1) / kLB16;
  if (win_nrb(p) <= 0) return cudaSuccess;
  kern<<<dim3(nkb * win_nrb(p), m_count), kThreads, smem, s>>>(p, d_rj, ld, cols, v0, s0);
  return cudaGetLastError();
}
// ---------------------------------------------------------------------------
// Backward kernel of the stored tables.  8 warps of m16n8k4: one B fragment serves
// 16 rows where the 8-row kernel reads it twice.  The products and their order
// are the 8-row kernel's (P and dP of each parity summed on their own, the +-m
// terms scaled and added at the end), and both DMMA shapes round alike, so the
// two kernels agree bit for bit: which one a launch takes does not show in the
// results of a radial window or slab.  (Summing the +-m terms into the same
// accumulators, m/sin P as a third operand, takes 1% less time at L = 255, Nr =
// 129, but its theta and phi sums have 1.3 times the rounding error at L = 63 ..
// 511.)  Operands come through a ring of six
// cp.async stages, one barrier per two chunks.  A CTA takes one field group, at most
// two vectors (20 accumulator tiles of four doubles per lane, and two per
// scalar); groups start at even vectors, so no record pair is split between two
// of them.  A group of one vector takes twice the radii, so that its warps have
// as many columns to share the A fragments.  Default set, ms at L = 255, Nr = 129
// and L = 1023, Nr = 17: a launch per group, eight radii each 2.83, 22.8; sixteen for
// the last 2.74, 23.7; one launch 2.72, 22.6; six stages and half the barriers
// (four and one per chunk before) 2.67, 22.1.
constexpr int kRing16 = 6;

// group: CTA = (m, 64 latitudes, 8 RB radii), warp = (16 latitudes, 4 RB radii)
template <int NV, int NS>
struct Bwd16Geo {
  static constexpr int RB = NV == 1 && NS <= 1 ? 2 : 1;
  static constexpr int CB = 24 * NV + 8 * NS;
  static constexpr int CBp = CB + ((4 - CB % 16) + 16) % 16;
  static constexpr int AS = kThBlk + 4;
  static constexpr int A_STAGE = 2 * kKC * AS;
  static constexpr int B_STAGE = 2 * RB * kKC * CBp;
  static constexpr size_t SMEM = sizeof(double) * kRing16 * (A_STAGE + B_STAGE);
  __host__ __device__ static int radial_ctas(const Plan& p) { return (win_nrb(p) + 2 * RB - 1) / (2 * RB); }
};

// order m, latitudes from th0, radial CTA rp of the group of vectors v0 .. v0 + NV - 1 and scalars 0 .. NS - 1
template <int NV, int NS>
__device__ __forceinline__ void bwd16_group(const Plan& p, double* sm, int m, int th0, int rp, int v0) {
  using G = Bwd16Geo<NV, NS>;
  constexpr int RB = G::RB;
  double* sA = sm;                            // [ring][P, dP][kKC][AS]
  double* sB = sm + kRing16 * G::A_STAGE;     // [ring][2 RB radial blocks][kKC][CBp]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int tg = warp & 3, rbi = warp >> 2;  // radial blocks rbi, rbi + 2, ...
  const int nrb_here = min(2 * RB, win_nrb(p) - 2 * RB * rp);  // of this CTA
  const int rb0 = win_rb0(p) + 2 * RB * rp;
  const int n0 = p.kpad[2 * m] / kKC, n1 = p.kpad[2 * m + 1] / kKC;
  const int total = n0 + n1;
  const int CBt = 24 * p.nvb + 8 * p.nsb;     // columns of one radial block in SB
  const long long rowB = (long long)p.nrb * CBt;
  const bool active = rbi < nrb_here && th0 + 16 * tg < p.nh;

  auto load = [&](int step) {
    const int st = step % kRing16;
    const int par = step < n0 ? 0 : 1;
    const int ch = step < n0 ? step : step - n0;
    const long long po = p.poff[2 * m + par] + (long long)(ch * kKC) * p.nh_pad + th0;
    double* a = sA + st * G::A_STAGE;
#pragma unroll
    for (int it = tid; it < 2 * kKC * (kThBlk / 2); it += kThreads) {
      const int tb = it / (kKC * (kThBlk / 2));
      const int rem = it % (kKC * (kThBlk / 2));
      const int row = rem / (kThBlk / 2), c2 = rem % (kThBlk / 2);
      cp_async16(a + (tb * kKC + row) * G::AS + 2 * c2, (tb ? p.dP : p.P) + po + (long long)row * p.nh_pad + 2 * c2);
    }
    const double* Bg = p.SB + p.sboff[2 * m + par] + (long long)(ch * kKC) * rowB + (long long)rb0 * CBt;
    double* bs = sB + st * G::B_STAGE;
    constexpr int NV2 = 12 * NV, NP2 = 12 * NV + 4 * NS;  // 16-byte pieces of a row: vectors, all
    for (int it = tid; it < 2 * RB * kKC * NP2; it += kThreads) {
      const int rr = it / NP2, c2 = it - rr * NP2;  // rr = radial block * kKC + row
      const int q = rr / kKC, row = rr % kKC;
      if (q >= nrb_here) break;
      const int src = c2 < NV2 ? 24 * v0 + 2 * c2 : 24 * p.nvb + 2 * (c2 - NV2);
      cp_async16(bs + rr * G::CBp + 2 * c2, Bg + row * rowB + q * CBt + src);
    }
  };

  // accumulators: [radial block][field][tile][parity][row g, g + 8: cos, sin]; tiles XP, XdP, YP, YdP, ZP
  double acc[RB][NV][5][2][4];
  double accS[RB][NS > 0 ? NS : 1][2][4];
#pragma unroll
  for (int u = 0; u < RB; ++u) {
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int q = 0; q < 5; ++q)
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[u][v][q][s][e] = 0.0;
#pragma unroll
    for (int v = 0; v < (NS > 0 ? NS : 1); ++v)
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int e = 0; e < 4; ++e) accS[u][v][s][e] = 0.0;
  }

  // nu: radial blocks of this warp
  auto compute = [&](int st, auto parc, auto nuc) {
    constexpr int par = decltype(parc)::value, nu = decltype(nuc)::value;
    const double* a = sA + st * G::A_STAGE + t * G::AS + 16 * tg + g;
    const double* bs = sB + st * G::B_STAGE + (rbi * kKC + t) * G::CBp + g;
#pragma unroll
    for (int kk = 0; kk < kKC / 4; ++kk) {
      const double p0 = a[4 * kk * G::AS], p1 = a[4 * kk * G::AS + 8];
      const double d0 = a[(kKC + 4 * kk) * G::AS], d1 = a[(kKC + 4 * kk) * G::AS + 8];
#pragma unroll
      for (int u = 0; u < nu; ++u) {
        const double* br = bs + (2 * u * kKC + 4 * kk) * G::CBp;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const double bX = br[24 * v], bY = br[24 * v + 8], bZ = br[24 * v + 16];
          dmma16(acc[u][v][0][par], p0, p1, bX);
          dmma16(acc[u][v][1][par], d0, d1, bX);
          dmma16(acc[u][v][2][par], p0, p1, bY);
          dmma16(acc[u][v][3][par], d0, d1, bY);
          dmma16(acc[u][v][4][par], p0, p1, bZ);
        }
#pragma unroll
        for (int s = 0; s < NS; ++s) dmma16(accS[u][s][par], p0, p1, br[24 * NV + 8 * s]);
      }
    }
  };

  using One = std::integral_constant<int, 1>;
  using All = std::integral_constant<int, RB>;
  const bool all = RB == 1 || rbi + 2 * (RB - 1) < nrb_here;
  auto compute_step = [&](int step) {
    const int st = step % kRing16;
    if (step < n0) {
      if (all) compute(st, std::integral_constant<int, 0>(), All());
      else compute(st, std::integral_constant<int, 0>(), One());
    } else {
      if (all) compute(st, std::integral_constant<int, 1>(), All());
      else compute(st, std::integral_constant<int, 1>(), One());
    }
  };
  // two chunks per commit group and barrier
  auto load2 = [&](int step) {
    if (step < total) load(step);
    if (step + 1 < total) load(step + 1);
    cp_async_commit();
  };
#pragma unroll
  for (int q = 0; q < kRing16 - 2; q += 2) load2(q);
  for (int step = 0; step < total; step += 2) {
    cp_async_wait<kRing16 / 2 - 2>();
    __syncthreads();  // both chunks have landed; every warp is done with the stages that load2() overwrites
    load2(step + kRing16 - 2);
    if (!active) continue;
#pragma unroll 1  // the body is large
    for (int q = step; q < min(step + 2, total); ++q) compute_step(q);
  }
  cp_async_wait<0>();

  // ---- epilogue: N/S recombination and +-m cross terms
  if (!active) return;
  const int nc = p.ncb;
  const bool al = rtm_aligned(p, nc);
#pragma unroll
  for (int u = 0; u < RB; ++u) {
    const int r = kRB * (rb0 + rbi + 2 * u) + t;
    if (rbi + 2 * u >= nrb_here || r >= p.nr) continue;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = th0 + 16 * tg + 8 * h + g, e = 2 * h;
      if (i >= p.nh) continue;
      const bool pair = i < p.nth / 2;
      const double ms = (double)m * p.asin_t[i];
      double* outN = p.rtm_b + rtm_off(p, m, i, r, nc);
      double* outS = p.rtm_b + rtm_off(p, m, p.nth - 1 - i, r, nc);
      // (sym, asym) of two components -> one record sector of each hemisphere
      auto put = [&](int q, const double(&sy)[4], const double(&as)[4]) {
        const int o = rtm_pair(p, m, q, nc);
        if (pair) {
          st_sector(outN + o, al, sy[0] + as[0], sy[1] + as[1], sy[2] + as[2], sy[3] + as[3]);
          st_sector(outS + o, al, sy[0] - as[0], sy[1] - as[1], sy[2] - as[2], sy[3] - as[3]);
        } else {
          st_sector(outN + o, al, sy[0], sy[1], sy[2], sy[3]);
        }
      };
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        double sy[4], as[4];
        cross_terms([&](int tile, int par, int slot) { return acc[u][v][tile][par][e + slot]; }, ms, sy, as);
        put(v0 + v, sy, as);
      }
      // radial components and scalars, two list entries per pair (v0 is even; the
      // scalars follow the last group's vectors)
      constexpr int NF = NV + NS;
#pragma unroll
      for (int f = 0; f < NF; f += 2) {
        double sy[4] = {0.0, 0.0, 0.0, 0.0}, as[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int ff = f + k;
          if (ff >= NF) break;
          const double(&c)[2][4] = ff < NV ? acc[u][ff < NV ? ff : 0][4] : accS[u][ff < NV ? 0 : ff - NV];
          sy[2 * k] = c[0][e];
          sy[2 * k + 1] = c[0][e + 1];
          as[2 * k] = c[1][e];
          as[2 * k + 1] = c[1][e + 1];
        }
        if (f + 1 < NF) {
          put(p.nvb + (v0 + f) / 2, sy, as);
        } else {  // odd count: the last pair holds one component
          const int o = rtm_pair(p, m, p.nvb + (v0 + f) / 2, nc);
          *reinterpret_cast<double2*>(outN + o) =
              pair ? make_double2(sy[0] + as[0], sy[1] + as[1]) : make_double2(sy[0], sy[1]);
          if (pair) *reinterpret_cast<double2*>(outS + o) = make_double2(sy[0] - as[0], sy[1] - as[1]);
        }
      }
    }
  }
}

// One launch for every group: nfull groups of two vectors, then the last one of
// NV vectors with the scalars.  The groups of one (m, latitudes) are neighbours
// in the grid: they read the same P and dP (once from HBM at large L).
template <int NV, int NS>
__global__ void __launch_bounds__(kThreads, 1) k_leg_bwd16(const __grid_constant__ Plan p, int nfull) {
  extern __shared__ double sm[];
  const int full = Bwd16Geo<2, 0>::radial_ctas(p), last = Bwd16Geo<NV, NS>::radial_ctas(p);
  const int per = nfull * full + last, x = blockIdx.x % per, y = blockIdx.x / per;
  const int nthb = p.nh_pad / kThBlk, m = y / nthb, th0 = (y - m * nthb) * kThBlk;
  if (x < nfull * full) bwd16_group<2, 0>(p, sm, m, th0, x % full, 2 * (x / full));
  else bwd16_group<NV, NS>(p, sm, m, th0, x - nfull * full, 2 * nfull);
}

template <int NV, int NS>
cudaError_t run_bwd16(const Plan& p, cudaStream_t s) {
  auto kern = k_leg_bwd16<NV, NS>;
  const int nfull = (p.nvb - NV) / 2;
  const size_t smem = std::max(nfull ? Bwd16Geo<2, 0>::SMEM : 0, Bwd16Geo<NV, NS>::SMEM);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const long long nblk = (long long)(p.L + 1) * (p.nh_pad / kThBlk) *
                         (nfull * Bwd16Geo<2, 0>::radial_ctas(p) + Bwd16Geo<NV, NS>::radial_ctas(p));
  if (nblk <= 0) return cudaSuccess;
  kern<<<(unsigned)nblk, kThreads, smem, s>>>(p, nfull);
  return cudaGetLastError();
}
cudaError_t run_bwd16(const Plan& p, cudaStream_t s) {  // at least one vector
  switch ((p.nvb % 2 ? 1 : 2) * 3 + p.nsb) {
    case 3: return run_bwd16<1, 0>(p, s);
    case 4: return run_bwd16<1, 1>(p, s);
    case 5: return run_bwd16<1, 2>(p, s);
    case 6: return run_bwd16<2, 0>(p, s);
    case 7: return run_bwd16<2, 1>(p, s);
    case 8: return run_bwd16<2, 2>(p, s);
    default: return cudaErrorInvalidValue;
  }
}

// Field groups of the forward kernel: two vectors while more than three are left,
// then the rest with the scalars.
cudaError_t run_fwd16(const Plan& p, double* d_rj, long long ld, const int* cols, cudaStream_t s, int m_count) {
  auto group = [&](int nv, int ns, int v0) -> cudaError_t {
    switch (nv * 3 + ns) {
      case 1: return run_fwd16<0, 1>(p, d_rj, ld, cols, s, m_count, v0, 0);
      case 2: return run_fwd16<0, 2>(p, d_rj, ld, cols, s, m_count, v0, 0);
      case 3: return run_fwd16<1, 0>(p, d_rj, ld, cols, s, m_count, v0, 0);
      case 4: return run_fwd16<1, 1>(p, d_rj, ld, cols, s, m_count, v0, 0);
      case 5: return run_fwd16<1, 2>(p, d_rj, ld, cols, s, m_count, v0, 0);
      case 6: return run_fwd16<2, 0>(p, d_rj, ld, cols, s, m_count, v0, 0);
      case 7: return run_fwd16<2, 1>(p, d_rj, ld, cols, s, m_count, v0, 0);
      case 8: return run_fwd16<2, 2>(p, d_rj, ld, cols, s, m_count, v0, 0);
      case 9: return run_fwd16<3, 0>(p, d_rj, ld, cols, s, m_count, v0, 0);
      case 10: return run_fwd16<3, 1>(p, d_rj, ld, cols, s, m_count, v0, 0);
      case 11: return run_fwd16<3, 2>(p, d_rj, ld, cols, s, m_count, v0, 0);
      default: return cudaErrorInvalidValue;
    }
  };
  cudaError_t e = cudaSuccess;
  int v0 = 0;
  do {
    const int nv = p.nvf - v0 <= 3 ? p.nvf - v0 : 2;
    e = group(nv, v0 + nv == p.nvf ? p.nsf : 0, v0);
    v0 += nv;
  } while (e == cudaSuccess && v0 < p.nvf);
  return e;
}

template <int NV, int NS, bool OTF>
cudaError_t run_bwd_t(const Plan& p, cudaStream_t s) {
  using G = BwdGeo<NV, NS>;
  auto kern = k_leg_bwd_f64<NV, NS, OTF>;
  const size_t smem = OTF ? G::SMEM_OTF : G::SMEM;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const long long nblk = (long long)(p.L + 1) * (p.nh_pad / kThBlk) * win_nrb(p);
  if (nblk <= 0) return cudaSuccess;
  kern<<<(unsigned)nblk, kThreads + (OTF ? kGenThreadsB : 0), smem, s>>>(p);
  return cudaGetLastError();
}
template <int NV, int NS>
cudaError_t run_bwd(const Plan& p, cudaStream_t s) {
  return p.otf ? run_bwd_t<NV, NS, true>(p, s) : run_bwd_t<NV, NS, false>(p, s);
}

template <int NV, int NS, bool OTF>
cudaError_t run_fwd_t(const Plan& p, double* d_rj, long long ld, const int* cols, cudaStream_t s, int m_count) {
  using G = FwdGeo<NV, NS>;
  auto kern = k_leg_fwd_f64<NV, NS, OTF>;
  const size_t smem = OTF ? G::SMEM_OTF : G::SMEM;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int nkb = (kcount(p.L, 0, 0) + kLBlk - 1) / kLBlk;
  if (win_nrb(p) <= 0) return cudaSuccess;
  dim3 grid(nkb * win_nrb(p), m_count);
  kern<<<grid, kThreads, smem, s>>>(p, d_rj, ld, cols);
  return cudaGetLastError();
}
template <int NV, int NS>
cudaError_t run_fwd(const Plan& p, double* d_rj, long long ld, const int* cols, cudaStream_t s, int m_count) {
  return p.otf ? run_fwd_t<NV, NS, true>(p, d_rj, ld, cols, s, m_count)
               : run_fwd_t<NV, NS, false>(p, d_rj, ld, cols, s, m_count);
}

template <int NV, int NS>
cudaError_t run_pack(const Plan& p, int nlc_max, const double* d_rj, long long ld, const int* cols, cudaStream_t s) {
  if (win_nrb(p) <= 0) return cudaSuccess;
  constexpr size_t smem = sizeof(double) * 32 * (24 * NV + 8 * NS + 1);  // at most 35 KB
  k_pack_b<NV, NS><<<dim3(nlc_max * win_nrb(p), p.L + 1), kThreads, smem, s>>>(p, d_rj, ld, cols);
  return cudaGetLastError();
}

#define KMHD_DISPATCH(NVv, NSv, FN, ...)                                   \
  switch (NVv * 3 + NSv) {                                                 \
    case 1: return FN<0, 1>(__VA_ARGS__);                                  \
    case 2: return FN<0, 2>(__VA_ARGS__);                                  \
    case 3: return FN<1, 0>(__VA_ARGS__);                                  \
    case 4: return FN<1, 1>(__VA_ARGS__);                                  \
    case 5: return FN<1, 2>(__VA_ARGS__);                                  \
    case 6: return FN<2, 0>(__VA_ARGS__);                                  \
    case 7: return FN<2, 1>(__VA_ARGS__);                                  \
    case 8: return FN<2, 2>(__VA_ARGS__);                                  \
    case 9: return FN<3, 0>(__VA_ARGS__);                                  \
    case 10: return FN<3, 1>(__VA_ARGS__);                                 \
    case 11: return FN<3, 2>(__VA_ARGS__);                                 \
    case 12: return FN<4, 0>(__VA_ARGS__);                                 \
    case 13: return FN<4, 1>(__VA_ARGS__);                                 \
    case 14: return FN<4, 2>(__VA_ARGS__);                                 \
    case 15: return FN<5, 0>(__VA_ARGS__);                                 \
    case 16: return FN<5, 1>(__VA_ARGS__);                                 \
    case 17: return FN<5, 2>(__VA_ARGS__);                                 \
    default: return cudaErrorInvalidValue;                                 \
  }

}  // namespace

cudaError_t launch_pack_b(const Plan& p, int nlc_max, const double* d_rj, long long ld,
                               const int* cols, int nv, int ns, cudaStream_t s) {
  KMHD_DISPATCH(nv, ns, run_pack, p, nlc_max, d_rj, ld, cols, s);
}

static int sm_count() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

cudaError_t launch_leg_bwd_f64(const Plan& p, cudaStream_t s) {
  // The 16-row kernel takes a whole SM per CTA: it wins when there are two CTAs
  // (of eight radii) for each and at least two vectors to share a chunk's
  // operands.  ms 8-row -> 16-row: L = 255, Nr = 129 3.19 -> 2.67; L = 511, Nr = 17
  // 3.24 -> 3.01; L = 127, Nr = 17 (768 CTAs) 0.109 -> 0.101; but L = 31, Nr = 33
  // (160) 0.016 -> 0.019, L = 63, Nr = 9 (128) 0.018 -> 0.020, one vector at
  // L = 255, Nr = 33 0.309 -> 0.322.  The launch is a window or slab of the shell
  // as often as not; the results are the same on both sides.
  const long long ctas = (long long)(p.L + 1) * (p.nh_pad / kThBlk) * ((win_nrb(p) + 1) / 2);
  if (!p.otf && p.nvb >= 2 && ctas >= 2 * sm_count()) return run_bwd16(p, s);
  KMHD_DISPATCH(p.nvb, p.nsb, run_bwd, p, s);
}

cudaError_t launch_leg_fwd_f64(const Plan& p, double* d_rj, long long ld, const int* cols,
                               cudaStream_t s, int m_count) {
  if (m_count <= 0 || m_count > p.L + 1) m_count = p.L + 1;
  // 64 degrees per parity and a whole SM per CTA: for truncations that fill them
  // and launches of at least one CTA per SM (not the few orders of the split
  // tiers' dipole modes at small Nr).  ms 32-degree kernel -> this one: L = 127, Nr =
  // 65 0.447 -> 0.409, Nr = 5 (256 CTAs) 0.081 -> 0.060; L = 255, Nr = 3 0.168 ->
  // 0.142, Nr = 129 3.94 -> 3.62; L = 1023, Nr = 17 29.0 -> 25.9; the same at L = 95
  // and 106; but L = 63, Nr = 33 0.051 -> 0.065 (most warps without a degree).
  const long long ctas = (long long)((kcount(p.L, 0, 0) + kLB16 - 1) / kLB16) * win_nrb(p) * m_count;
  if (!p.otf && p.L >= 112 && ctas >= sm_count()) return run_fwd16(p, d_rj, ld, cols, s, m_count);
  KMHD_DISPATCH(p.nvf, p.nsf, run_fwd, p, d_rj, ld, cols, s, m_count);
}

size_t bwd_smem_bytes(int nv, int ns) {
  const int CB = 24 * nv + 8 * ns;
  const int CBp = CB + ((4 - CB % 16) + 16) % 16;
  return sizeof(double) * 2 * (2 * kKC * (kThBlk + 4) + kKC * CBp);
}

}  // namespace kmhd
