// Per-point BSE kernels around the LU:
//   * build  -- A = 1 - blockdiag_nu(chi0^q chi0_loc^-1 - 1) F~ and gamma^q_d
//               (src/main.F90:674-732), written transposed (T = A^T) with the
//               right-hand sides (1 + gamma^w)^T appended as extra columns;
//   * post   -- eta = (1+gamma^w)(A^-1 - 1) from the solve, the chi(q,w)
//               frequency sums of calc_chi_qw (src/main.F90:665-667,766-769;
//               src/susc_module.f90:34-56) and the EOM vertex m_tot
//               (src/eom_module.f90:184-207);
//   * eom    -- Sigma(k, nu) += m_tot G(k-q, nu-w) over a batch of points
//               (src/eom_module.f90:209-230), one owner thread per (k, nu).
#include "ctx.cuh"
#include "zgemm.cuh"
#include <cooperative_groups.h>
#include <algorithm>
#include <type_traits>

namespace cg = cooperative_groups;

// ---------------------------------------------------------------------------
// build: T(c, r) = delta(c, r) - sum_i3 sw_nu(i1, i3) F~(i3 + nu*nd2, c), r = i1 + nu*nd2,
// sw_nu = chi0q(:,:,nu) diag(chi0_loc^-1(nu)) - 1, and gamma^q_d = sum_nu sw_nu F~_d(nu block).
// ---------------------------------------------------------------------------
// One orbital: element by element.  A warp takes 32 columns and every eighth nu, so that the
// frequencies are not one serial chain per column; gamma^q_d adds the warps' parts in their order.
// (A thread per column walking all nu took 18 us a channel on N = 40 and 65 us on N = 160 with 216
// points; this kernel, both channels: 5.4 and 47 us.)
template <typename T>
__global__ void __launch_bounds__(256)
k_bse_build_1(DevCtx c, const z64 *__restrict__ chi0q, const z64 *__restrict__ c0inv,
              const z64 *__restrict__ Frow_d, const z64 *__restrict__ Frow_m, const z64 *__restrict__ opg_d,
              const z64 *__restrict__ opg_m, T *Tm, size_t strideM, z64 *gammaqd, const int *__restrict__ qidx) {
  __shared__ z64 part[8][32];
  const int N = c.N, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cc = blockIdx.x * 32 + lane, ch = blockIdx.y, p = blockIdx.z;
  const z64 *F = ch == 0 ? Frow_d : Frow_m, *opg = ch == 0 ? opg_d : opg_m, *c0 = chi0q + (size_t)p * N;
  T *Tp = Tm + (size_t)(2 * p + ch) * strideM;
  const bool act = cc < N;
  z64 og = act ? opg[cc] : czero<z64>(), sv = czero<z64>();
  if (c.vq && ch == 0) sv = cscale(c.vq[qidx[p]], 2.0 / (c.beta * c.beta));    // src/main.F90:710-719
  z64 gq = czero<z64>();
#pragma unroll 4
  for (int nu = w; nu < N; nu += 8) {
    const z64 q = c0[nu];
    z64 sw = cmul(q, c0inv[nu]);
    sw.x -= 1.0;
    const z64 g = act ? cmul(sw, F[(size_t)nu * N + cc]) : czero<z64>();
    gq = cadd(gq, g);
    z64 t = cneg(g);
    if (c.vq && ch == 0) cfms(t, cmul(q, sv), og);
    if (nu == cc) t.x += 1.0;
    if (act) Tp[cc + (size_t)nu * N] = from64<T>(t);
  }
  part[w][lane] = gq;
  __syncthreads();
  if (w == 0 && act) {
    Tp[cc + (size_t)N * N] = from64<T>(og);
    if (ch == 0 && gammaqd) {
      for (int v = 1; v < 8; ++v) gq = cadd(gq, part[v][lane]);
      gammaqd[(size_t)p * N + cc] = gq;
    }
  }
}

// 2 beta^-2 chi0^q(nu) v(q) for every point and frequency, in chi0^q's layout (src/main.F90:710-719)
__global__ void k_vq_sv(DevCtx c, size_t n, const z64 *__restrict__ chi0q, const int *__restrict__ qidx,
                        z64 *__restrict__ sv) {
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (idx >= n) return;
  const int nd2 = c.nd2, nd4 = nd2 * nd2, i1 = (int)(idx % nd2), i3 = (int)(idx / nd2 % nd2);
  const z64 *cq = chi0q + idx / nd4 * nd4 + i1;
  const z64 *vq = c.vq + (size_t)qidx[idx / nd4 / (2 * c.iwf)] * nd4 + (size_t)i3 * nd2;
  z64 s = czero<z64>();
  for (int k = 0; k < nd2; ++k) cfma(s, cq[k * nd2], vq[k]);
  sv[idx] = cscale(s, 2.0 / (c.beta * c.beta));
}

// Four and five orbitals, and the density channel with V(q): per nu a product of the batch's sw rows (npts nd2 x nd2) with the nd2 x N block of F~
// on the FP64 tensor cores (m8n8k4, complex as four real products).  A CTA owns 32 rows (p, i1) and 64
// columns and walks nu: F~'s block of the next nu arrives by cp.async while sw of the next nu is formed
// from chi0^q into the other half of the stage; K = nd2 is padded with zeros to a multiple of four (4, 12,
// 16, 28).  Bound by the FP64 rate (padding included) with F~ read from L2 and T written once.  GQ (the
// density channel) keeps gamma^q_d's sum over nu in registers; with V(q) the term
// 2 beta^-2 chi0^q(nu) v(q) (1+gamma^w_d) (src/main.F90:710-719) is a second product with a resident
// operand, after gamma^q_d has taken the first.
// A thread per column with all products on the CUDA cores took 8.8 ms (both channels, 216 points,
// N = 1000, 25 components; this kernel 4.45 ms) and 0.81 ms (both, 216 points, N = 486, with V(q); this
// kernel for the density channel 0.51 ms, the magnetic one as without V(q) 0.25 ms).
template <int ND2> struct BuildTile {
  static constexpr int KP = (ND2 + 3) / 4 * 4;
  static constexpr int LDA = KP % 8 == 4 ? KP : KP + 4, LDB = 66;      // conflict-free fragment reads
  static constexpr int A_ELEMS = 32 * LDA, B_ELEMS = KP * LDB;
  static constexpr int smem(bool vterm) {
    return (int)sizeof(z64) * (2 * (A_ELEMS + B_ELEMS) + (vterm ? 2 * A_ELEMS + B_ELEMS : 0));
  }
};

template <typename TW, int ND2, bool GQ>
__global__ void __launch_bounds__(128, 2)
k_bse_build(DevCtx c, int npts, int ch, const z64 *__restrict__ chi0q, const z64 *__restrict__ c0inv,
            const z64 *__restrict__ F, const z64 *__restrict__ opg, TW *Tm, size_t strideM, z64 *gammaqd,
            const z64 *__restrict__ sv) {
  typedef BuildTile<ND2> L;
  constexpr int KP = L::KP, NE = (32 * ND2 + 127) / 128;
  extern __shared__ __align__(16) z64 bse_smem[];
  z64 *As = bse_smem, *Bs = As + 2 * L::A_ELEMS, *Vs = Bs + 2 * L::B_ELEMS, *Og = Vs + 2 * L::A_ELEMS;
  const int N = c.N, nnu = 2 * c.iwf, t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int c0 = blockIdx.x * 64, m0 = blockIdx.y * 32, rows = npts * ND2;
  const bool vterm = GQ && c.vq;
  for (int e = t; e < L::smem(vterm) / (int)sizeof(z64); e += 128) bse_smem[e] = czero<z64>();   // the padding
  __syncthreads();
  auto stage_f = [&](int nu, int buf) {
    for (int e = t; e < ND2 * 64; e += 128) {
      const int k = e >> 6, col = e & 63;
      const bool in = c0 + col < N;
      const z64 *g = F + (size_t)(k + nu * ND2) * N + c0 + col;
      zg::cp_async16(Bs + buf * L::B_ELEMS + k * L::LDB + col, in ? g : F, in ? 16 : 0);
    }
    zg::cp_async_commit();
  };
  // this thread's elements of sw: (row, i3) with i1 fastest, as chi0^q lies in memory
  z64 pq[NE], pv[NE];
  auto load_sw = [&](int nu) {
#pragma unroll
    for (int q = 0; q < NE; ++q) {
      const int e = t + 128 * q, i3 = e / 32, m = m0 + e % 32;
      if (e < 32 * ND2 && m < rows) {
        const size_t at = ((size_t)(m / ND2) * nnu + nu) * ND2 * ND2 + m % ND2 + i3 * ND2;
        pq[q] = chi0q[at];
        if (vterm) pv[q] = sv[at];
      }
    }
  };
  auto store_sw = [&](int nu, int buf) {
#pragma unroll
    for (int q = 0; q < NE; ++q) {
      const int e = t + 128 * q, i3 = e / 32, r = e % 32, m = m0 + r;
      if (e < 32 * ND2 && m < rows) {
        z64 v = cmul(pq[q], c0inv[nu * ND2 + i3]);
        if (m % ND2 == i3) v.x -= 1.0;
        As[buf * L::A_ELEMS + r * L::LDA + i3] = v;
        if (vterm) Vs[buf * L::A_ELEMS + r * L::LDA + i3] = pv[q];
      }
    }
  };
  if (vterm)
    for (int e = t; e < ND2 * 64; e += 128) {
      const int k = e % ND2, col = e / ND2;
      if (c0 + col < N) Og[k * L::LDB + col] = opg[k + (size_t)(c0 + col) * ND2];
    }
  // warp (wm, wn): rows 16 wm.., columns 32 wn..
  const int wm = warp & 1, wn = warp >> 1, kl = lane & 3;
  const int ra = 16 * wm + (lane >> 2), cb = 32 * wn + (lane >> 2);
  double re[2][4][2], im[2][4][2], gr[GQ ? 2 : 1][4][2], gi[GQ ? 2 : 1][4][2];
#pragma unroll
  for (int i = 0; i < (GQ ? 2 : 1); ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) gr[i][j][0] = gr[i][j][1] = gi[i][j][0] = gi[i][j][1] = 0.0;
  auto product = [&](const z64 *A, const z64 *B) {
#pragma unroll
    for (int k = 0; k < KP; k += 4) {
      z64 a[2], b[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) a[i] = A[(ra + 8 * i) * L::LDA + k + kl];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = B[(k + kl) * L::LDB + cb + 8 * j];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const double an = -a[i].y;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          zg::dmma(re[i][j], a[i].x, b[j].x);
          zg::dmma(im[i][j], a[i].x, b[j].y);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          zg::dmma(re[i][j], an, b[j].y);
          zg::dmma(im[i][j], a[i].y, b[j].x);
        }
      }
    }
  };
  stage_f(0, 0);
  load_sw(0);
  store_sw(0, 0);
  for (int nu = 0; nu < nnu; ++nu) {
    const int buf = nu & 1;
    const bool more = nu + 1 < nnu;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                   // stage nu complete, stage nu - 1 read
    if (more) {
      stage_f(nu + 1, buf ^ 1);
      load_sw(nu + 1);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
    product(As + buf * L::A_ELEMS, Bs + buf * L::B_ELEMS);
    if constexpr (GQ) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            gr[i][j][e] += re[i][j][e];
            gi[i][j][e] += im[i][j][e];
          }
      if (vterm) product(Vs + buf * L::A_ELEMS, Og);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int m = m0 + ra + 8 * i, r = m % ND2 + nu * ND2;
      if (m >= rows) continue;
      TW *o = Tm + (size_t)(2 * (m / ND2) + ch) * strideM + (size_t)r * N;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int cc = c0 + 32 * wn + 8 * j + 2 * kl;       // even, N is even
        if (cc >= N) continue;
        const z64 t0 = make_double2((r == cc ? 1.0 : 0.0) - re[i][j][0], -im[i][j][0]);
        const z64 t1 = make_double2((r == cc + 1 ? 1.0 : 0.0) - re[i][j][1], -im[i][j][1]);
        if constexpr (sizeof(TW) == sizeof(z32))
          *reinterpret_cast<float4 *>(o + cc) = make_float4((float)t0.x, (float)t0.y, (float)t1.x, (float)t1.y);
        else {
          o[cc] = t0;
          o[cc + 1] = t1;
        }
      }
    }
    if (more) store_sw(nu + 1, buf ^ 1);
  }
  // the right-hand sides, and gamma^q_d
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int m = m0 + ra + 8 * i, p = m / ND2, i1 = m % ND2;
    if (m >= rows) continue;
    TW *o = Tm + (size_t)(2 * p + ch) * strideM + (size_t)(N + i1) * N;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int cc = c0 + 32 * wn + 8 * j + 2 * kl + e;
        if (cc >= N) continue;
        o[cc] = from64<TW>(opg[i1 + (size_t)cc * ND2]);
        if constexpr (GQ)
          if (gammaqd) gammaqd[(size_t)p * ND2 * N + i1 + (size_t)cc * ND2] = make_double2(gr[i][j][e], gi[i][j][e]);
      }
  }
}

// Two and three orbitals without the V(q) term: one block per (128-column tile, P points) of one
// channel, on the CUDA cores: with K = nd2 = 4 or 9 the tensor-core form above spends a quarter of its
// products on padding and waits at its per-nu barrier (density and magnetic channel of 250 points,
// N = 1080, FP64: 1.48 and 1.38 ms here, 2.52 and 1.85 ms there).  A thread owns one column c of T; the F~ rows of each nu block are
// staged into shared memory one nu ahead by cp.async (each thread copies and
// reads only its own column), and sw_nu of the block's points is formed in
// shared memory one nu ahead from chi0^q / chi0_loc^-1 values prefetched into
// registers; one barrier per nu.  F32 selects complex FP32 arithmetic from an
// FP32 copy of F~ -- used for the magnetic channel of the mixed path, whose T
// only feeds the FP32 LU (the FP64 residual of the refinement restores the
// FP64 answer); GQ accumulates gamma^q_d (the density channel, always FP64).
template <int ND2, bool GQ> struct BuildP { static constexpr int P = GQ ? 1 : 2; };

__device__ __forceinline__ void cp_async_bytes(void *smem, const void *gmem, int pred16or8, int nbytes) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  if (pred16or8 == 16)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(nbytes));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(s), "l"(gmem), "r"(nbytes));
}

template <typename TW, int ND2, bool F32, bool GQ>
__global__ void __launch_bounds__(128)
k_bse_build_fast(DevCtx c, int npts, int ch, const z64 *__restrict__ chi0q, const z64 *__restrict__ c0inv,
                 const void *__restrict__ Fv, const z64 *__restrict__ opg, TW *Tm, size_t strideM, z64 *gammaqd) {
  typedef typename std::conditional<F32, z32, z64>::type A;
  constexpr int P = BuildP<ND2, GQ>::P, ND4 = ND2 * ND2, NE = P * ND4, EPT = (NE + 127) / 128;
  __shared__ __align__(16) A fs[2][ND2][128];
  __shared__ __align__(16) A sws[2][NE];
  const A *F = (const A *)Fv;
  const int N = c.N, nnu = 2 * c.iwf, t = threadIdx.x;
  const int cc = blockIdx.x * 128 + t, p0 = blockIdx.y * P;
  const bool act = cc < N;
  z64 pc[EPT], pinv[EPT];
  auto load_sw = [&](int dum) {
#pragma unroll
    for (int k = 0; k < EPT; ++k) {
      const int e = t + 128 * k;
      if (e < NE) {
        const int pp = e / ND4, el = e % ND4, i3 = el / ND2;
        const int p = p0 + pp;
        pc[k] = p < npts ? chi0q[((size_t)p * nnu + dum) * ND4 + el] : make_double2(0.0, 0.0);
        pinv[k] = c0inv[dum * ND2 + i3];
      }
    }
  };
  auto store_sw = [&](int buf) {
#pragma unroll
    for (int k = 0; k < EPT; ++k) {
      const int e = t + 128 * k;
      if (e < NE) {
        const int el = e % ND4, i1 = el % ND2, i3 = el / ND2;
        z64 v = cmul(pc[k], pinv[k]);
        if (i1 == i3) v.x -= 1.0;
        if constexpr (F32) sws[buf][e] = to32(v);
        else sws[buf][e] = v;
      }
    }
  };
  auto stage_f = [&](int dum, int buf) {
#pragma unroll
    for (int i3 = 0; i3 < ND2; ++i3) {
      const A *g = F + (size_t)(i3 + dum * ND2) * N + (act ? cc : 0);
      cp_async_bytes(&fs[buf][i3][t], g, (int)sizeof(A), act ? (int)sizeof(A) : 0);
    }
    asm volatile("cp.async.commit_group;");
  };
  z64 gq[GQ ? P * ND2 : 1];
  if constexpr (GQ) {
#pragma unroll
    for (int a = 0; a < P * ND2; ++a) gq[a] = make_double2(0.0, 0.0);
  }
  stage_f(0, 0);
  load_sw(0);
  store_sw(0);
  __syncthreads();
  for (int dum = 0; dum < nnu; ++dum) {
    const bool more = dum + 1 < nnu;
    if (more) {
      stage_f(dum + 1, (dum + 1) & 1);
      load_sw(dum + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    const A *sw = sws[dum & 1];
    A f[ND2];
#pragma unroll
    for (int i3 = 0; i3 < ND2; ++i3) f[i3] = fs[dum & 1][i3][t];
#pragma unroll
    for (int pp = 0; pp < P; ++pp) {
      const int p = p0 + pp;
      if (act && p < npts) {
        TW *Tp = Tm + (size_t)(2 * p + ch) * strideM;
#pragma unroll
        for (int i1 = 0; i1 < ND2; ++i1) {
          A w = cx<A>::make(0, 0);
#pragma unroll
          for (int i3 = 0; i3 < ND2; ++i3) cfma(w, sw[pp * ND4 + i1 + i3 * ND2], f[i3]);
          const int r = i1 + dum * ND2;
          A tv = cx<A>::make(-w.x, -w.y);
          if (r == cc) tv.x += 1;
          if constexpr (F32) Tp[cc + (size_t)r * N] = tv;
          else Tp[cc + (size_t)r * N] = from64<TW>(tv);
          if constexpr (GQ) gq[pp * ND2 + i1] = cadd(gq[pp * ND2 + i1], w);
        }
      }
    }
    if (more) store_sw((dum + 1) & 1);
    __syncthreads();
  }
  if (!act) return;
#pragma unroll
  for (int pp = 0; pp < P; ++pp) {
    const int p = p0 + pp;
    if (p >= npts) continue;
    TW *Tp = Tm + (size_t)(2 * p + ch) * strideM;
#pragma unroll
    for (int i1 = 0; i1 < ND2; ++i1) Tp[cc + (size_t)(N + i1) * N] = from64<TW>(opg[i1 + (size_t)cc * ND2]);
    if constexpr (GQ) {
      if (gammaqd) {
        z64 *g = gammaqd + (size_t)p * ND2 * N;
#pragma unroll
        for (int i1 = 0; i1 < ND2; ++i1) g[i1 + (size_t)cc * ND2] = gq[pp * ND2 + i1];
      }
    }
  }
}

__global__ void k_to32(size_t n, const z64 *__restrict__ x, z32 *__restrict__ y) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = to32(x[i]);
}

cudaError_t launch_to32(size_t n, const z64 *x, z32 *y, cudaStream_t st) {
  if (!n) return cudaSuccess;
  k_to32<<<(unsigned)std::min<size_t>(cdiv_u(n, 256), 4096), 256, 0, st>>>(n, x, y);
  return ADGA_LAUNCH_CHECK();
}

template <typename T, int ND2, bool GQ>
static cudaError_t launch_build_tile(const DevCtx &c, int npts, const z64 *chi0q, const z64 *c0inv, const z64 *F,
                                     const z64 *opg, T *Tmat, size_t strideM, z64 *gammaqd, const z64 *sv,
                                     cudaStream_t st) {
  typedef BuildTile<ND2> L;
  cudaError_t e = smem_limit(k_bse_build<T, ND2, GQ>, L::smem(true));
  if (e != cudaSuccess) return e;
  const dim3 g(cdiv_u(c.N, 64), cdiv_u((size_t)npts * ND2, 32));
  k_bse_build<T, ND2, GQ><<<g, 128, L::smem(GQ && c.vq), st>>>(c, npts, GQ ? 0 : 1, chi0q, c0inv, F, opg, Tmat,
                                                             strideM, GQ ? gammaqd : nullptr, sv);
  return ADGA_LAUNCH_CHECK();
}

template <typename T>
cudaError_t launch_bse_build(const DevCtx &c, int npts, const z64 *chi0q, const z64 *c0inv,
                             const z64 *Frow_d, const z64 *Frow_m, const z64 *opg_d,
                             const z64 *opg_m, T *Tmat, size_t strideM, z64 *gammaqd,
                             const int *qidx, z64 *vscr, cudaStream_t st, const z32 *F32_m) {
  if (npts <= 0) return cudaSuccess;
  if (c.nd2 == 1) {
    k_bse_build_1<T><<<dim3(cdiv_u(c.N, 32), 2, npts), 256, 0, st>>>(c, chi0q, c0inv, Frow_d, Frow_m, opg_d, opg_m,
                                                                    Tmat, strideM, gammaqd, qidx);
    return ADGA_LAUNCH_CHECK();
  }
  cudaError_t e = cudaErrorInvalidValue;
  if (c.vq) {
    const size_t n = (size_t)npts * 2 * c.iwf * c.nd2 * c.nd2;
    k_vq_sv<<<cdiv_u(n, 256), 256, 0, st>>>(c, n, chi0q, qidx, vscr);
    if ((e = ADGA_LAUNCH_CHECK()) != cudaSuccess) return e;
  }
#define TILE(NDD, GQ)                                                                                            \
  launch_build_tile<T, NDD, GQ>(c, npts, chi0q, c0inv, GQ ? Frow_d : Frow_m, GQ ? opg_d : opg_m, Tmat, strideM,  \
                                gammaqd, vscr, st)
#define FAST(NDD, F32, GQ, F)                                                                                    \
  (k_bse_build_fast<T, NDD, F32, GQ><<<dim3(cdiv_u(c.N, 128), cdiv_u(npts, BuildP<NDD, GQ>::P)), 128, 0, st>>>(  \
       c, npts, GQ ? 0 : 1, chi0q, c0inv, F, GQ ? opg_d : opg_m, Tmat, strideM, GQ ? gammaqd : nullptr),         \
   ADGA_LAUNCH_CHECK())
#define BUILD_FAST(NDD)                                                                                          \
  do {                                                                                                           \
    e = c.vq ? TILE(NDD, true) : FAST(NDD, false, true, Frow_d);                                                 \
    if (e != cudaSuccess) return e;                                                                              \
    if constexpr (std::is_same<T, z32>::value) {                                                                 \
      if (F32_m && !c.vq) return FAST(NDD, true, false, F32_m);                                                  \
    }                                                                                                            \
    e = FAST(NDD, false, false, Frow_m);                                                                         \
  } while (0)
#define BUILD_TILE(NDD)                                                                                          \
  do {                                                                                                           \
    e = TILE(NDD, true);                                                                                         \
    if (e == cudaSuccess) e = TILE(NDD, false);                                                                  \
  } while (0)
  switch (c.nd2) {
    case 4: BUILD_FAST(4); break;
    case 9: BUILD_FAST(9); break;
    case 16: BUILD_TILE(16); break;
    case 25: BUILD_TILE(25); break;
  }
#undef TILE
#undef FAST
#undef BUILD_FAST
#undef BUILD_TILE
  return e;
}
template cudaError_t launch_bse_build<z64>(const DevCtx &, int, const z64 *, const z64 *,
                                           const z64 *, const z64 *, const z64 *, const z64 *,
                                           z64 *, size_t, z64 *, const int *, z64 *, cudaStream_t,
                                           const z32 *);
template cudaError_t launch_bse_build<z32>(const DevCtx &, int, const z64 *, const z64 *,
                                           const z64 *, const z64 *, const z64 *, const z64 *,
                                           z32 *, size_t, z64 *, const int *, z64 *, cudaStream_t,
                                           const z32 *);

// ---------------------------------------------------------------------------
// post: one cluster of S blocks per point, the blocks sharing its frequencies.
//   X_ch(c, i1) (column-major, ld ldX) = ((1+gamma^w) A^-1)^T  -> eta = X^T - (1+gamma^w)
//   chi_ch = beta^-2 sum gamma (chi0q - chi0w) + beta^-2 sum eta chi0q
//   m_tot(:, nu >= 0 half) = -(u - u~/2) eta_d/(beta nqp) + 1.5 u~ eta_m/(beta nqp)
//                            + u gamma^q_d/(beta nqp)
// A block stages VB frequencies at a time (chi0^q and both channels' eta, which it transposes for the
// output on the way) and every product runs on ND x ND register tiles, so that an operand read from
// shared memory feeds ND products: thread (g, ch, ib, jb) owns rows ib + ND r and columns jb + ND s of
// frequency g of the stage.  The chi tiles stay in registers over all stages and are added over g and
// then over the blocks in rank order.  Bound by the shared-memory reads and, for a few points, by the
// stages' latency.
// One block per point with eight lanes per chi element and a thread per m_tot element, operands from
// global memory: 3.04 ms (216 points, 25 components, 40 frequencies), 1.78 ms (1000 points, 9, 120),
// 0.30 ms (one of those); this kernel: 1.13 ms, 0.79 ms and 55 us.
// ---------------------------------------------------------------------------
template <int ND> struct PostTile {
  static constexpr int ND2 = ND * ND, ND4 = ND2 * ND2;
  static constexpr int VB = ND == 1 ? 64 : ND == 2 ? 16 : ND == 3 ? 7 : ND == 4 ? 4 : 2;   // frequencies per stage
  static constexpr int ACT = 2 * ND2 * VB, NT = (ACT + 31) / 32 * 32;
  static constexpr int LE = VB * ND2 + 1;                        // row stride of the staged eta
  static constexpr size_t STAGE = (size_t)VB * ND4 + 2 * ND2 * LE;   // chi0^q, eta_d, eta_m
  static constexpr size_t RED = (size_t)ACT * ND2;                // the threads' chi tiles
  static constexpr int SMEM = (int)sizeof(z64) * (int)((STAGE > RED ? STAGE : RED) + 2 * ND4);
};

template <int ND>
__global__ void __launch_bounds__(PostTile<ND>::NT)
k_post(DevCtx c, const z64 *__restrict__ X, size_t sp, size_t sc, int ldX, const z64 *__restrict__ opg_d,
       const z64 *__restrict__ opg_m, const z64 *__restrict__ gam_d, const z64 *__restrict__ gam_m,
       const z64 *__restrict__ gammaqd, const z64 *__restrict__ chi0q, const z64 *__restrict__ c0w,
       z64 *chi_qw_d, z64 *chi_qw_m, z64 *mtot, z64 *etad, z64 *etam, const int *__restrict__ qidx) {
  typedef PostTile<ND> L;
  constexpr int ND2 = L::ND2, ND4 = L::ND4, VB = L::VB, NT = L::NT, LE = L::LE;
  extern __shared__ __align__(16) z64 post_smem[];
  z64 *uw = post_smem, *ut = uw + ND4;          // v + u - u~/2 and u~
  z64 *Cs = ut + ND4, *Es = Cs + VB * ND4;      // [VB][i2][i3] and [ch][i1][LE]
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), S = (int)cl.num_blocks();
  const int p = blockIdx.y, t = threadIdx.x, nnu = 2 * c.iwf, N = c.N;
  const size_t nd2N = (size_t)ND2 * N;
  const z64 *c0 = chi0q + (size_t)p * ND4 * nnu, *gq = gammaqd + (size_t)p * nd2N;
  // V(q) terms of m_tot (src/eom_module.f90:187-205)
  const z64 *vq = (mtot && c.vq && qidx) ? c.vq + (size_t)qidx[p] * ND4 : nullptr;
  for (int e = t; e < ND4; e += NT) {
    const z64 uu = c.u[e], tt = c.ut[e];
    z64 w = make_double2(uu.x - 0.5 * tt.x, uu.y - 0.5 * tt.y);
    if (vq) w = cadd(vq[e], w);                 // u_work = v + u - u~/2
    uw[e] = w;
    ut[e] = tt;
  }
  const bool act = t < L::ACT;
  const int jb = t % ND, ib = t / ND % ND, ch = t / ND2 % 2, g = t / (2 * ND2);
  z64 acc[ND][ND];
#pragma unroll
  for (int r = 0; r < ND; ++r)
#pragma unroll
    for (int s = 0; s < ND; ++s) acc[r][s] = czero<z64>();
  const double inv = 1.0 / c.beta / (double)c.nqp;
  for (int v0 = rank * VB; v0 < nnu; v0 += S * VB) {
    const int nv = min(VB, nnu - v0), w = nv * ND2;
    __syncthreads();                            // the last stage is read
    for (int e = t; e < nv * ND4; e += NT) Cs[e] = c0[(size_t)v0 * ND4 + e];
    for (int e = t; e < 2 * ND2 * w; e += NT) {
      const int row = e / w, col = e % w;       // row = ch nd2 + i1
      Es[row * LE + col] = X[(size_t)p * sp + (row / ND2) * sc + (size_t)(row % ND2) * ldX + v0 * ND2 + col];
    }
    __syncthreads();
    // eta = X^T - (1 + gamma^w), written with i1 fastest
    for (int e = t; e < 2 * ND2 * w; e += NT) {
      const int ce = e / (ND2 * w), r = e % (ND2 * w), i1 = r % ND2, col = r / ND2;
      const size_t o = (size_t)(v0 * ND2 + col) * ND2 + i1;
      z64 &x = Es[(ce * ND2 + i1) * LE + col];
      x = csub(x, (ce ? opg_m : opg_d)[o]);
      ((ce ? etam : etad) + p * nd2N)[o] = x;
    }
    __syncthreads();
    if (!act || g >= nv) continue;
    const int nu = v0 + g;
    const z64 *C = Cs + g * ND4, *E = Es + ch * ND2 * LE + g * ND2;
    const z64 *G = (ch ? gam_m : gam_d) + (size_t)nu * ND2 * ND2;
#pragma unroll 1
    for (int i3 = 0; i3 < ND2; ++i3) {
      z64 q[ND];
#pragma unroll
      for (int s = 0; s < ND; ++s) q[s] = C[(jb + ND * s) * ND2 + i3];
#pragma unroll
      for (int r = 0; r < ND; ++r) {
        const z64 x = E[(ib + ND * r) * LE + i3];
#pragma unroll
        for (int s = 0; s < ND; ++s) cfma(acc[r][s], x, q[s]);
      }
#pragma unroll
      for (int s = 0; s < ND; ++s)
        if (jb + ND * s == i3) q[s] = csub(q[s], c0w[nu * ND2 + i3]);
#pragma unroll
      for (int r = 0; r < ND; ++r) {
        const z64 x = __ldg(G + ib + ND * r + i3 * ND2);
#pragma unroll
        for (int s = 0; s < ND; ++s) cfma(acc[r][s], x, q[s]);
      }
    }
    // m_tot of a frequency nu >= 0: rows ib + ND r, columns jb + ND s, one half of the columns per ch thread
    if (mtot && nu >= c.iwf) {
      const z64 *Ed = Es + g * ND2, *Em = Ed + ND2 * LE;
#pragma unroll 1
      for (int s = ch; s < ND; s += 2) {
        const int j = jb + ND * s;
        z64 a1[ND], a2[ND], a3[ND];
#pragma unroll
        for (int r = 0; r < ND; ++r) a1[r] = a2[r] = a3[r] = czero<z64>();
#pragma unroll 1
        for (int i3 = 0; i3 < ND2; ++i3) {
          const z64 ed = Ed[i3 * LE + j], em = Em[i3 * LE + j], gv = __ldg(gq + i3 + (size_t)(nu * ND2 + j) * ND2);
#pragma unroll
          for (int r = 0; r < ND; ++r) {
            const int i1 = ib + ND * r;
            const z64 tt = ut[i1 + i3 * ND2];
            cfma(a1[r], uw[i1 + i3 * ND2], ed);
            cfma(a2[r], tt, em);
            cfma(a3[r], __ldg(c.u + i1 + i3 * ND2), gv);
          }
        }
#pragma unroll
        for (int r = 0; r < ND; ++r) {
          const int i1 = ib + ND * r;
          z64 v = cscale(a1[r], -inv);
          v = cadd(cscale(a2[r], 1.5 * inv), v);
          v = cadd(cscale(a3[r], inv), v);
          if (vq) {                             // v gamma^w_d
            z64 a4 = czero<z64>();
            for (int i3 = 0; i3 < ND2; ++i3) cfma(a4, vq[i1 + i3 * ND2], gam_d[i3 + (size_t)(nu * ND2 + j) * ND2]);
            v = cadd(cscale(a4, -inv), v);
          }
          mtot[(size_t)p * ND4 * c.iwf + i1 + (size_t)((nu - c.iwf) * ND2 + j) * ND2] = v;
        }
      }
    }
  }
  // the tiles of all frequencies: over the stage's slots, then over the cluster's blocks
  __syncthreads();
  z64 *red = Cs;                                // [element][thread]
  if (act)
#pragma unroll
    for (int r = 0; r < ND; ++r)
#pragma unroll
      for (int s = 0; s < ND; ++s) red[(r * ND + s) * L::ACT + t] = acc[r][s];
  __syncthreads();
  constexpr int OUT = 2 * ND4;
  for (int e = t; e < OUT; e += NT) {
    const int rs = e / (2 * ND2), th = e % (2 * ND2);
    z64 v = czero<z64>();
    for (int k = 0; k < VB; ++k) v = cadd(v, red[rs * L::ACT + k * 2 * ND2 + th]);
    red[rs * L::ACT + th] = v;                  // slot 0 of the same (element, thread) column
  }
  cl.sync();
  if (rank == 0) {
    const double b2 = c.beta * c.beta;
    for (int e = t; e < OUT; e += NT) {
      const int rs = e / (2 * ND2), th = e % (2 * ND2);
      z64 v = czero<z64>();
      for (int k = 0; k < S; ++k) v = cadd(v, cl.map_shared_rank(red, k)[rs * L::ACT + th]);
      const int i1 = th / ND % ND + ND * (rs / ND), i2 = th % ND + ND * (rs % ND);
      (th / ND2 ? chi_qw_m : chi_qw_d)[(size_t)p * ND4 + i1 + i2 * ND2] = make_double2(v.x / b2, v.y / b2);
    }
  }
  cl.sync();                                    // the first block has read the others' sums
}

template <int ND, typename... A>
static cudaError_t launch_post_nd(int npts, int nnu, cudaStream_t st, A... args) {
  typedef PostTile<ND> L;
  cudaError_t e = smem_limit(k_post<ND>, L::SMEM);
  if (e != cudaSuccess) return e;
  // blocks for about two waves of two per SM, at least one stage each
  const int stages = (nnu + L::VB - 1) / L::VB;
  int S = 1;
  while (S < 8 && 2 * S <= stages && 2 * S * npts <= 1184) S *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(S, npts);
  cfg.blockDim = dim3(L::NT);
  cfg.dynamicSmemBytes = L::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = S;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, k_post<ND>, args...);
  if (e != cudaSuccess) return e;
  return ADGA_LAUNCH_CHECK();
}

cudaError_t launch_post(const DevCtx &c, int npts, const z64 *X, size_t sp, size_t sc, int ldX,
                        const z64 *opg_d, const z64 *opg_m, const z64 *gam_d, const z64 *gam_m,
                        const z64 *gammaqd, const z64 *chi0q, const z64 *c0w, z64 *chi_qw_d,
                        z64 *chi_qw_m, z64 *mtot, z64 *etad, z64 *etam, const int *qidx, cudaStream_t st) {
  if (npts <= 0) return cudaSuccess;
#define POST(NDD)                                                                                                  \
  return launch_post_nd<NDD>(npts, 2 * c.iwf, st, c, X, sp, sc, ldX, opg_d, opg_m, gam_d, gam_m, gammaqd, chi0q,   \
                             c0w, chi_qw_d, chi_qw_m, mtot, etad, etam, qidx)
  switch (c.nd) {
    case 1: POST(1);
    case 2: POST(2);
    case 3: POST(3);
    case 4: POST(4);
    case 5: POST(5);
  }
#undef POST
  return cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------
// eom: Sigma(i,l,nu,k) += sum_p sum_{k',j} m_tot_p({j,i},{k',l,nu}) G_jk'(k - q_p, nu - w)
// One block per (k tile, nu >= 0); the m_tot slice of each point is staged in
// shared memory, G is gathered from the resident table.  Summation order per
// element follows the reference: points in order, k' outer, j inner.
// ---------------------------------------------------------------------------
template <int ND>
__global__ void __launch_bounds__(128)
k_eom_dyn(DevCtx c, int iwb, const int *__restrict__ qidx, int npts, const z64 *__restrict__ mtot,
          z64 *sigma) {
  constexpr int ND2 = ND * ND;
  __shared__ z64 M[ND2 * ND2];
  const int nu = blockIdx.y;                  // 0..iwf-1
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int iwf = c.iwf;
  const bool act = k < c.nkp_eom;
  z64 acc[ND2];
  z64 *so = sigma + ((size_t)k * 2 * iwf + nu + iwf) * ND2;
#pragma unroll
  for (int a = 0; a < ND2; ++a) acc[a] = act ? so[a] : make_double2(0.0, 0.0);
  const z64 *gt = c.gtab + (size_t)(nu - iwb - c.nu_lo) * c.nkp * ND2;
  for (int p = 0; p < npts; ++p) {
    __syncthreads();
    const z64 *mp = mtot + (size_t)p * ND2 * iwf * ND2 + (size_t)nu * ND2 * ND2;
    for (int e = threadIdx.x; e < ND2 * ND2; e += blockDim.x) M[e] = mp[e];
    __syncthreads();
    if (act) {
      int kk = c.kqe[k + (size_t)qidx[p] * c.nkp_eom];
      const z64 *g = gt + (size_t)kk * ND2;
      z64 G[ND2];
#pragma unroll
      for (int a = 0; a < ND2; ++a) G[a] = __ldg(g + a);
#pragma unroll
      for (int l = 0; l < ND; ++l)
#pragma unroll
        for (int k2 = 0; k2 < ND; ++k2)
#pragma unroll
          for (int i = 0; i < ND; ++i)
#pragma unroll
            for (int j = 0; j < ND; ++j)
              cfma(acc[i + l * ND], M[(i * ND + j) + (l * ND + k2) * ND2], G[j + k2 * ND]);
    }
  }
  if (act) {
#pragma unroll
    for (int a = 0; a < ND2; ++a) so[a] = acc[a];
  }
}

cudaError_t launch_eom_dynamic(const DevCtx &c, int iwb, const int *qidx, int npts,
                               const z64 *mtot, z64 *sigma_nl, cudaStream_t st) {
  if (npts <= 0) return cudaSuccess;
  if (c.dft.ghat && npts >= c.dft.eom_min_points)
    return launch_eom_dft(c, iwb, qidx, npts, mtot, c.dft.ghat, sigma_nl, st);
  dim3 grid(cdiv_u(c.nkp_eom, 128), c.iwf);
  switch (c.nd) {
    case 1: k_eom_dyn<1><<<grid, 128, 0, st>>>(c, iwb, qidx, npts, mtot, sigma_nl); break;
    case 2: k_eom_dyn<2><<<grid, 128, 0, st>>>(c, iwb, qidx, npts, mtot, sigma_nl); break;
    case 3: k_eom_dyn<3><<<grid, 128, 0, st>>>(c, iwb, qidx, npts, mtot, sigma_nl); break;
    case 4: k_eom_dyn<4><<<grid, 128, 0, st>>>(c, iwb, qidx, npts, mtot, sigma_nl); break;
    case 5: k_eom_dyn<5><<<grid, 128, 0, st>>>(c, iwb, qidx, npts, mtot, sigma_nl); break;
    default: return cudaErrorInvalidValue;
  }
  return ADGA_LAUNCH_CHECK();
}
