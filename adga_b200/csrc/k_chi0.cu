// chi0 bubble: chi0^q({i,j},{l,k}; nu) = -(beta/nkp) sum_k G_il(k, nu) G_kj(k-q, nu-omega)
// for a batch of q points at one omega -- the k-loop of src/main.F90:646-657
// over accumulate_chi0 (src/one_particle_quant_module.f90:228-290).
//
// Two kernels: k_chi0 for many points (the FP64 pipe bounds it: nd2 complex
// MACs per gathered 16-byte G(k-q) value; the G-table slices it reads stay in
// L2 across the batch) and k_chi0_few for a few points.
#include "ctx.cuh"
#include "zgemm.cuh"
#include <cooperative_groups.h>
#include <algorithm>

namespace cg = cooperative_groups;

// Thread (q, b) of a CTA owns one column b = (k', j) of G(k-q, nu-omega) and
// one point q, and accumulates the nd2 products with every entry a = (i, l)
// of G(k, nu) over k.  G(k, nu) is staged in shared memory in chunks of KC
// k-points and read as broadcasts; the k-q indices of the CTA's points are
// staged beside it.  Each gathered G(k-q) value feeds nd2 complex FMAs.
template <int ND, int QG>
__global__ void __launch_bounds__(QG * ND * ND)
k_chi0(DevCtx c, int iwb, const int *__restrict__ qidx, int npts, z64 *__restrict__ out, int nnu_all,
       const z64 *__restrict__ g2tab) {
  constexpr int ND2 = ND * ND, KC = 64, NTH = QG * ND2;
  __shared__ z64 g1s[KC][ND2];
  __shared__ int kqs[KC][QG];
  const int inu = blockIdx.x, p0 = blockIdx.y * QG;
  const int t = threadIdx.x, ql = t / ND2, bcol = t % ND2;
  const int p = p0 + ql;
  const bool act = p < npts;
  const int nu = c.iwstart + inu;
  const z64 *g1t = c.gtab + (size_t)(nu - c.nu_lo) * c.nkp * ND2;
  const z64 *g2t = (g2tab ? g2tab : c.gtab) + (size_t)(nu - iwb - c.nu_lo) * c.nkp * ND2;
  z64 acc[ND2];
#pragma unroll
  for (int a = 0; a < ND2; ++a) acc[a] = make_double2(0.0, 0.0);
  for (int k0 = 0; k0 < c.nkp; k0 += KC) {
    const int kc = min(KC, c.nkp - k0);
    __syncthreads();
    for (int e = t; e < kc * ND2; e += NTH) g1s[e / ND2][e % ND2] = __ldg(g1t + (size_t)k0 * ND2 + e);
    for (int e = t; e < kc * QG; e += NTH) {
      const int q_l = e / kc, kk = e % kc, pp = p0 + q_l;
      kqs[kk][q_l] = pp < npts ? __ldg(c.kq + (k0 + kk) + (size_t)qidx[pp] * c.nkp) : 0;
    }
    __syncthreads();
    if (act) {
#pragma unroll 4
      for (int kk = 0; kk < kc; ++kk) {
        const z64 g2 = __ldg(g2t + (size_t)kqs[kk][ql] * ND2 + bcol);
#pragma unroll
        for (int a = 0; a < ND2; ++a) cfma(acc[a], g1s[kk][a], g2);
      }
    }
  }
  if (!act) return;
  // a = i + l*nd (G_il(k)), bcol = k' + j*nd (G_k'j(k-q)): chi0({i,j},{l,k'})
  z64 *o = out + ((size_t)p * nnu_all + inu) * ND2 * ND2;
  const double f = -c.beta / (double)c.nkp;
  const int kp = bcol % ND, j = bcol / ND;
#pragma unroll
  for (int a = 0; a < ND2; ++a) {
    const int i = a % ND, l = a / ND;
    o[(i * ND + j) + (l * ND + kp) * ND2] = make_double2(acc[a].x * f, acc[a].y * f);
  }
}

// A few points: a block per (nu, point, column group j of G(k-q)), its warps split over the orbital l
// of G(k, nu) and, for one and two orbitals, over k; a lane owns a k-point and accumulates the ND x ND
// products G_il(k) G_k'j(k-q) of its (l, j), and the lanes' sums are added by shuffles at the end.  Both
// factors come through a double-buffered cp.async stage (rows of an odd number of 16-byte units:
// conflict-free reads), so the block is bound by the gather's latency and the L2; a cluster of S blocks
// shares the k-points of one output where nnu x points alone leaves SMs idle, and its first block adds
// the others' sums in rank order from their shared memory.
// With one thread per column of G(k-q) and all k in a row, one point took 3.3 ms on a 20^3 mesh with
// three orbitals and 120 frequencies and 175 us on a 10^3 mesh with one and 40; this form: 107 us and 7 us.
template <int ND> struct Few {
  static constexpr int JB = ND <= 3 ? ND : 1;                 // column groups per block
  static constexpr int WPG = ND == 1 ? 8 : ND == 2 ? 2 : 1;   // warps per (l, j)
  static constexpr int NT = 32 * ND * JB * WPG, KC = ND == 1 ? 512 : ND <= 3 ? 128 : 64;
  static constexpr int L1 = (ND * ND) | 1, L2 = (ND * JB) | 1;   // strides of a k-point's row
  static constexpr size_t SMEM = sizeof(z64) * 2 * KC * (L1 + L2);
};

template <int ND>
__global__ void __launch_bounds__(Few<ND>::NT)
k_chi0_few(DevCtx c, int iwb, const int *__restrict__ qidx, z64 *__restrict__ out, int nnu_all,
           const z64 *__restrict__ g2tab) {
  typedef Few<ND> F;
  constexpr int ND2 = ND * ND, NT = F::NT, KC = F::KC, NB = ND * F::JB;
  extern __shared__ __align__(16) unsigned char few_smem[];
  __shared__ z64 red[F::WPG][F::JB * ND][ND2];
  z64 *g1s = reinterpret_cast<z64 *>(few_smem), *g2s = g1s + 2 * KC * F::L1;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), S = (int)cl.num_blocks();
  const int inu = blockIdx.x / S, p = blockIdx.y / (ND / F::JB), j0 = blockIdx.y % (ND / F::JB) * F::JB;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int grp = warp / F::WPG, wk = warp % F::WPG, l = grp % ND, jl = grp / ND;
  const int nu = c.iwstart + inu;
  const z64 *g1t = c.gtab + (size_t)(nu - c.nu_lo) * c.nkp * ND2;
  const z64 *g2t = (g2tab ? g2tab : c.gtab) + (size_t)(nu - iwb - c.nu_lo) * c.nkp * ND2 + j0 * ND;
  const int *kq = c.kq + (size_t)qidx[p] * c.nkp;
  const int nch = (c.nkp + KC - 1) / KC;
  auto load = [&](int ch, int buf) {
    if (ch < nch) {
      const int k0 = ch * KC;
      for (int e = t; e < KC * NB; e += NT) {
        const int kk = e / NB, b = e % NB;
        const bool in = k0 + kk < c.nkp;
        zg::cp_async16(g2s + (buf * KC + kk) * F::L2 + b, in ? g2t + (size_t)__ldg(kq + k0 + kk) * ND2 + b : g2t,
                       in ? 16 : 0);
      }
      for (int e = t; e < KC * ND2; e += NT) {
        const int kk = e / ND2, a = e % ND2;
        const bool in = k0 + kk < c.nkp;
        zg::cp_async16(g1s + (buf * KC + kk) * F::L1 + a, in ? g1t + (size_t)k0 * ND2 + e : g1t, in ? 16 : 0);
      }
    }
    zg::cp_async_commit();
  };
  z64 acc[ND][ND];                       // [i][k']
#pragma unroll
  for (int i = 0; i < ND; ++i)
#pragma unroll
    for (int q = 0; q < ND; ++q) acc[i][q] = make_double2(0.0, 0.0);
  load(rank, 0);
  int buf = 0;
  for (int ch = rank; ch < nch; ch += S, buf ^= 1) {
    load(ch + S, buf ^ 1);
    zg::cp_async_wait<1>();
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KC / (32 * F::WPG); ++k) {
      const int kk = lane + 32 * (wk + F::WPG * k);
      const z64 *x = g1s + (buf * KC + kk) * F::L1 + l * ND, *y = g2s + (buf * KC + kk) * F::L2 + jl * ND;
      z64 xi[ND], yk[ND];
#pragma unroll
      for (int i = 0; i < ND; ++i) { xi[i] = x[i]; yk[i] = y[i]; }
#pragma unroll
      for (int i = 0; i < ND; ++i)
#pragma unroll
        for (int q = 0; q < ND; ++q) cfma(acc[i][q], xi[i], yk[q]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < ND; ++i)
#pragma unroll
    for (int q = 0; q < ND; ++q) {
      z64 v = acc[i][q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      }
      if (lane == 0) red[wk][grp][i * ND + q] = v;
    }
  cl.sync();
  if (rank == 0) {
    const double f = -c.beta / (double)c.nkp;
    z64 *o = out + ((size_t)p * nnu_all + inu) * ND2 * ND2;
    for (int e = t; e < F::JB * ND * ND2; e += NT) {
      const int g = e / ND2, iq = e % ND2, i = iq / ND, q = iq % ND;
      z64 v = make_double2(0.0, 0.0);
      for (int r = 0; r < S; ++r) {
        const z64 *rd = cl.map_shared_rank(&red[0][0][0], r);
        for (int w = 0; w < F::WPG; ++w) v = cadd(v, rd[(w * F::JB * ND + g) * ND2 + iq]);
      }
      // chi0({i,j},{l,k'})
      o[(i * ND + j0 + g / ND) + (g % ND * ND + q) * ND2] = make_double2(v.x * f, v.y * f);
    }
  }
  cl.sync();                             // the first block has read the others' sums
}

template <int ND>
static cudaError_t launch_chi0_few(const DevCtx &c, int iwb, const int *qidx, int npts, z64 *out, int nnu_all,
                                   const z64 *g2tab, cudaStream_t st) {
  typedef Few<ND> F;
  // blocks for about two per SM, at least two k-chunks each
  const int blocks = nnu_all * npts * (ND / F::JB), nch = (c.nkp + F::KC - 1) / F::KC;
  int S = 1;
  while (S < 8 && 2 * S * blocks <= 296 && 4 * S <= nch) S *= 2;
  cudaError_t e = smem_limit(k_chi0_few<ND>, (int)F::SMEM);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(S * nnu_all, npts * (ND / F::JB));      // a big box has more frequencies than y holds
  cfg.blockDim = dim3(F::NT);
  cfg.dynamicSmemBytes = F::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = S;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, k_chi0_few<ND>, c, iwb, qidx, out, nnu_all, g2tab);
  if (e != cudaSuccess) return e;
  return ADGA_LAUNCH_CHECK();
}

// From 32 points on k_chi0's reuse of G(k) among points pays (20^3 mesh, three orbitals, 120 frequencies:
// 16 points 1.30 against 1.55 ms, 32 points 2.37 against 1.89 ms; five orbitals, 16 points: equal)
constexpr int FEW_POINTS = 16;

cudaError_t launch_chi0(const DevCtx &c, int iwb, const int *qidx, int npts, z64 *chi0_all,
                        int nnu_all, cudaStream_t st, const z64 *g2tab, const z64 *g2hat) {
  if (npts <= 0) return cudaSuccess;
  if (c.dft.ghat && npts >= c.dft.min_points && (!g2tab || g2hat))
    return launch_chi0_dft(c, iwb, qidx, npts, chi0_all, nnu_all, c.dft.ghat, g2tab ? g2hat : c.dft.ghat, st);
  if (npts <= FEW_POINTS) switch (c.nd) {
    case 1: return launch_chi0_few<1>(c, iwb, qidx, npts, chi0_all, nnu_all, g2tab, st);
    case 2: return launch_chi0_few<2>(c, iwb, qidx, npts, chi0_all, nnu_all, g2tab, st);
    case 3: return launch_chi0_few<3>(c, iwb, qidx, npts, chi0_all, nnu_all, g2tab, st);
    case 4: return launch_chi0_few<4>(c, iwb, qidx, npts, chi0_all, nnu_all, g2tab, st);
    case 5: return launch_chi0_few<5>(c, iwb, qidx, npts, chi0_all, nnu_all, g2tab, st);
    default: return cudaErrorInvalidValue;
  }
#define CHI0(NDD, QGG)                                                                      \
  k_chi0<NDD, QGG><<<dim3(nnu_all, cdiv_u(npts, QGG)), QGG * NDD * NDD, 0, st>>>(c, iwb, qidx, \
                                                                                npts, chi0_all, nnu_all, g2tab)
  switch (c.nd) {
    case 1: CHI0(1, 128); break;
    case 2: CHI0(2, 32); break;
    case 3: CHI0(3, 16); break;
    case 4: CHI0(4, 8); break;
    case 5: CHI0(5, 8); break;
    default: return cudaErrorInvalidValue;
  }
#undef CHI0
  return ADGA_LAUNCH_CHECK();
}

// chi0q (small box) and bubble_nl = sum_{iwstart..iwstop} chi0 / beta^2 -
// bubble_loc_tmp (src/main.F90:655-663).  A lane per (i1, i2, point), the block's eight warps sharing the
// frequencies (added in warp order): one thread for all of them took 8 us on 125 points and 40
// frequencies and 29 us on 216 and 160; this form: 5.3 and 10.3 us.
__global__ void __launch_bounds__(256)
k_chi0_finish(DevCtx c, const z64 *__restrict__ all, int nnu_all, int npts, const z64 *__restrict__ bub_tmp,
              z64 *chi0q, z64 *bub_nl) {
  __shared__ z64 part[8][32];
  const size_t nd4 = (size_t)c.nd2 * c.nd2;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const size_t idx = blockIdx.x * (size_t)32 + lane;
  const bool act = idx < nd4 * npts;
  const size_t e = act ? idx % nd4 : 0, p = act ? idx / nd4 : 0;
  const z64 *a = all + p * nnu_all * nd4 + e;
  z64 s = make_double2(0.0, 0.0);
  const int off = -c.iwf - c.iwstart;   // index of nu = -iwf in the full list
  if (act)
#pragma unroll 4
    for (int inu = w; inu < nnu_all; inu += 8) {
      const z64 v = a[(size_t)inu * nd4];
      s = cadd(s, v);
      const int ism = inu - off;
      if (chi0q && ism >= 0 && ism < 2 * c.iwf) chi0q[(p * 2 * c.iwf + ism) * nd4 + e] = v;
    }
  part[w][lane] = s;
  __syncthreads();
  if (w == 0 && act && bub_nl) {
    for (int v = 1; v < 8; ++v) s = cadd(s, part[v][lane]);
    const double b2 = c.beta * c.beta;
    const z64 t = bub_tmp[e];
    bub_nl[p * nd4 + e] = make_double2(s.x / b2 - t.x, s.y / b2 - t.y);
  }
}

cudaError_t launch_chi0_finish(const DevCtx &c, const z64 *chi0_all, int nnu_all, int npts,
                               const z64 *bubloc_tmp, z64 *chi0q, z64 *bubble_nl, cudaStream_t st) {
  size_t total = (size_t)c.nd2 * c.nd2 * npts;
  if (!total) return cudaSuccess;
  k_chi0_finish<<<cdiv_u(total, 32), 256, 0, st>>>(c, chi0_all, nnu_all, npts, bubloc_tmp,
                                                    chi0q, bubble_nl);
  return ADGA_LAUNCH_CHECK();
}
