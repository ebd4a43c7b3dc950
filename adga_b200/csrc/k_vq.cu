// Non-local interaction V(q) (do_vq): the parts of the ladder that V(q)
// enters besides the BSE build and m_tot (k_bse.cu).
//   read_vq's index map   v(i1 = i nd + k, i2 = l nd + j, q) = vq(i, j, k, l, q)
//                         (src/interaction_module.f90:107-119)
//   calc_eom_static       non-local Hartree 2 v(q=0) n_dmft and Fock
//                         -v(q)/nqp n_fock(k-q) into sigma_hf (src/eom_module.f90:70-108)
//   mixed refinement      the density-channel residual term X blockdiag(S_nu) (1+gamma^w_d),
//                         S_nu = 2 beta^-2 chi0^q(nu) v(q), i.e. Y (1+gamma^w_d) with
//                         Y = 2 beta^-2 sum_nu X_nu chi0^q(nu) v(q)
#include "ctx.cuh"
#include <algorithm>

__global__ void k_vq_permute(int nd, int nqp, const z64 *__restrict__ raw, z64 *__restrict__ v) {
  const int nd2 = nd * nd;
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (idx >= (size_t)nd2 * nd2 * nqp) return;
  const int i1 = (int)(idx % nd2), i2 = (int)((idx / nd2) % nd2);
  const size_t q = idx / ((size_t)nd2 * nd2);
  const int i = i1 / nd, k = i1 % nd, l = i2 / nd, j = i2 % nd;
  v[idx] = raw[(size_t)i + nd * ((size_t)j + nd * ((size_t)k + nd * ((size_t)l + nd * q)))];
}

cudaError_t launch_vq_permute(int nd, int nqp, const z64 *raw, z64 *v, cudaStream_t st) {
  const size_t total = (size_t)nd * nd * nd * nd * nqp;
  k_vq_permute<<<cdiv_u(total, 256), 256, 0, st>>>(nd, nqp, raw, v);
  return ADGA_LAUNCH_CHECK();
}

// sigma_hf(i, l, ik) += for the points of one batch at omega = 0.  A lane owns a k-point and all nd x nd
// elements, so that an n_fock entry gathered at k-q feeds nd^2 of them and the gathers of a warp are
// neighbours; the block's warps share the points and their sums are added in warp order.  Bound by the
// gathers' latency: a thread per element walking all points took 1.52 ms (216 points, 1728 k-points,
// three orbitals); this form: 0.12 ms.
constexpr int HF_WARPS = 8;
template <int ND>
__global__ void __launch_bounds__(32 * HF_WARPS)
k_eom_static_vq(DevCtx c, const int *__restrict__ qidx, int npts, z64 *sigma_hf) {
  constexpr int ND2 = ND * ND;
  __shared__ z64 part[HF_WARPS][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, ik = blockIdx.x * 32 + lane;
  const bool act = ik < c.nkp_eom;
  z64 acc[ND2];                                  // i + l nd
#pragma unroll
  for (int e = 0; e < ND2; ++e) acc[e] = czero<z64>();
  const double f = 1.0 / c.nqp;
  for (int p = w; p < npts; p += HF_WARPS) {
    const int q = qidx[p];
    const z64 *v = c.vq + (size_t)q * ND2 * ND2;
    const int ikq = act ? c.kqe[ik + (size_t)q * c.nkp_eom] : 0;
#pragma unroll
    for (int j = 0; j < ND; ++j)                 // Fock: -v({ki},{jl})/nqp n_fock(k-q, j, k)
#pragma unroll
      for (int k = 0; k < ND; ++k) {
        const z64 nf = cscale(c.nfock[(size_t)ikq + (size_t)c.nkp * (j + (size_t)ND * k)], f);
#pragma unroll
        for (int l = 0; l < ND; ++l)
#pragma unroll
          for (int i = 0; i < ND; ++i) cfms(acc[i + l * ND], __ldg(v + (i * ND + k) + (l * ND + j) * ND2), nf);
      }
    if (q == 0)                                  // q = 0: non-local Hartree 2 v(q=0) n_dmft
#pragma unroll
      for (int i = 0; i < ND; ++i)
        for (int j = 0; j < ND; ++j) {
          const z64 t = cmul(v[(i * ND + i) + (j * ND + j) * ND2], c.ndmft[j]);
          acc[i + i * ND] = cadd(acc[i + i * ND], make_double2(2.0 * t.x, 2.0 * t.y));
        }
  }
#pragma unroll
  for (int e = 0; e < ND2; ++e) {
    part[w][lane] = acc[e];
    __syncthreads();
    if (w == 0 && act) {
      z64 s = sigma_hf[(size_t)ik * ND2 + e];
      for (int u = 0; u < HF_WARPS; ++u) s = cadd(s, part[u][lane]);
      sigma_hf[(size_t)ik * ND2 + e] = s;
    }
    __syncthreads();
  }
}

cudaError_t launch_eom_static_vq(const DevCtx &c, const int *qidx, int npts, z64 *sigma_hf, cudaStream_t st) {
  const unsigned g = cdiv_u(c.nkp_eom, 32);
  switch (c.nd) {
    case 1: k_eom_static_vq<1><<<g, 32 * HF_WARPS, 0, st>>>(c, qidx, npts, sigma_hf); break;
    case 2: k_eom_static_vq<2><<<g, 32 * HF_WARPS, 0, st>>>(c, qidx, npts, sigma_hf); break;
    case 3: k_eom_static_vq<3><<<g, 32 * HF_WARPS, 0, st>>>(c, qidx, npts, sigma_hf); break;
    case 4: k_eom_static_vq<4><<<g, 32 * HF_WARPS, 0, st>>>(c, qidx, npts, sigma_hf); break;
    case 5: k_eom_static_vq<5><<<g, 32 * HF_WARPS, 0, st>>>(c, qidx, npts, sigma_hf); break;
    default: return cudaErrorInvalidValue;
  }
  return ADGA_LAUNCH_CHECK();
}

// extra(p, i1, c) = sum_j Y_p(i1, j) (1+gamma^w_d)(j, c) for the density channel
// (matrix 2p of X); one block per point
// (81 of 256 threads on the sums over nu: 177 us a call on 216 points, 9 components, 54 frequencies; with
// 512 threads and the frequencies split: 46 us)
constexpr int VQ_THREADS = 512;
__global__ void __launch_bounds__(VQ_THREADS)
k_vq_resid_extra(DevCtx c, int ns, const int *__restrict__ qidx, const z64 *__restrict__ X,
                 const z64 *__restrict__ chi0q, const z64 *__restrict__ opg_d, z64 *__restrict__ extra) {
  extern __shared__ z64 sy[];                  // Z then Y, nd2 x nd2 each, then the parts of Z
  const int p = blockIdx.x, nd2 = c.nd2, nd4 = nd2 * nd2, N = c.N, t = threadIdx.x;
  const size_t per = (size_t)nd2 * N;
  const z64 *x = X + (size_t)(2 * p) * per;
  const z64 *cq = chi0q + (size_t)p * nd4 * 2 * c.iwf;
  z64 *Z = sy, *Y = sy + nd4, *P = Y + nd4;
  // Z(i1, n) = sum_nu sum_m X(i1, nu nd2 + m) chi0q(m, n, nu): the frequencies shared by ns slices, added in
  // slice order
  for (int e = t; e < nd4 * ns; e += blockDim.x) {
    const int i1 = e % nd2, n = e / nd2 % nd2, sl = e / nd4;
    z64 s = make_double2(0.0, 0.0);
    for (int nu = sl; nu < 2 * c.iwf; nu += ns)
      for (int m = 0; m < nd2; ++m)
        cfma(s, x[(size_t)i1 * N + nu * nd2 + m], cq[m + (size_t)n * nd2 + (size_t)nu * nd4]);
    P[e] = s;
  }
  __syncthreads();
  for (int e = t; e < nd4; e += blockDim.x) {
    z64 s = P[e];
    for (int sl = 1; sl < ns; ++sl) s = cadd(s, P[e + sl * nd4]);
    Z[e] = s;
  }
  __syncthreads();
  const z64 *v = c.vq + (size_t)qidx[p] * nd2 * nd2;
  const double f = 2.0 / (c.beta * c.beta);
  for (int e = t; e < nd2 * nd2; e += blockDim.x) {
    const int i1 = e % nd2, j = e / nd2;
    z64 s = make_double2(0.0, 0.0);
    for (int n = 0; n < nd2; ++n) cfma(s, Z[i1 + n * nd2], v[n + (size_t)j * nd2]);
    Y[e] = make_double2(f * s.x, f * s.y);
  }
  __syncthreads();
  z64 *o = extra + (size_t)p * per;
  for (size_t e = t; e < per; e += blockDim.x) {
    const int i1 = (int)(e / N), col = (int)(e % N);
    z64 s = make_double2(0.0, 0.0);
    for (int j = 0; j < nd2; ++j) cfma(s, Y[i1 + j * nd2], opg_d[j + (size_t)col * nd2]);
    o[e] = s;
  }
}

cudaError_t launch_vq_resid_extra(const DevCtx &c, int npts, const int *qidx, const z64 *X, const z64 *chi0q,
                                  const z64 *opg_d, z64 *extra, cudaStream_t st) {
  if (npts <= 0) return cudaSuccess;
  // slices: as many as the block's threads allow, no more than there are frequencies
  const int nd4 = c.nd2 * c.nd2, ns = std::min(std::max(1, VQ_THREADS / nd4), 2 * c.iwf);
  k_vq_resid_extra<<<npts, VQ_THREADS, sizeof(z64) * nd4 * (2 + ns), st>>>(c, ns, qidx, X, chi0q, opg_d, extra);
  return ADGA_LAUNCH_CHECK();
}
