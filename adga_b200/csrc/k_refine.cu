// FP64 iterative refinement of the mixed-precision BSE solve.
//
// The unknown is X = (1+gamma^w) A^-1 (ndim2 x N), solved from
// X A = B with A = 1 - D F~ (D = blockdiag_nu(chi0^q chi0_loc^-1 - 1)).
// The residual never needs A in FP64:
//     r = B - X A = B - X + (X D) F~ ,
// a (ndim2 x N) x (N x N) product per point with F~ shared by all q of one
// omega (L2-resident), computed here as one batched FP64 GEMM per channel.
// The correction d A = r is solved with the FP32 LU factors (forward with
// L and the pivots, backward with U), and X += d in FP64.
//
// Buffers follow the LU batch order m = 2*p + ch.  X (FP64) and the FP32
// right-hand sides V are N x R column-major per matrix, which is the same
// memory as X stored R x N row-major.
#include "ctx.cuh"

cudaError_t launch_resid_z64(const DevCtx &c, int npts, const z64 *XD, const z64 *X,
                             const z64 *Frow_d, const z64 *Frow_m, const z64 *opg_d,
                             const z64 *opg_m, z32 *V, const z64 *extra_d, unsigned long long *rnorm,
                             const z64 *Bpt, cudaStream_t st);

// the n x n identity
__global__ void k_identity(int n, z64 *E) {
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (idx < (size_t)n * n) E[idx] = make_double2(idx % n == idx / n ? 1.0 : 0.0, 0.0);
}
cudaError_t launch_identity(int n, z64 *E, cudaStream_t st) {
  k_identity<<<cdiv_u((size_t)n * n, 256), 256, 0, st>>>(n, E);
  return ADGA_LAUNCH_CHECK();
}

// X64 = up(Y32) from the RHS columns of the FP32 factorised matrices
__global__ void k_init_x(const z32 *T32, size_t strideM, int N, int R, int nmat, z64 *X) {
  size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  size_t per = (size_t)N * R;
  if (idx >= per * nmat) return;
  size_t m = idx / per, e = idx % per;
  X[idx] = to64(T32[m * strideM + (size_t)N * N + e]);
}

// XD(i1, i3 + nu*nd2) = sum_i2 X(i1, i2 + nu*nd2) sw_nu(i2, i3), row-major R x N.
// A block takes VB frequencies of one point: sw (formed once for both channels) and the X rows are staged
// in shared memory, thread (g, ch, ib, jb) owns the ND x ND outputs of rows ib + ND r and columns
// jb + ND s of frequency g.  Bound by memory (X read, XD written); a thread per output with operands
// and sw from global memory took 734 us a call (216 points, 25 components, 40 frequencies) and 528 us
// (1000 points, 9, 120); this kernel: 173 us and 218 us.
template <int ND> struct XdTile {
  static constexpr int ND2 = ND * ND, ND4 = ND2 * ND2;
  static constexpr int VB = ND == 1 ? 64 : ND == 2 ? 16 : ND == 3 ? 7 : ND == 4 ? 4 : 2;
  static constexpr int ACT = 2 * ND2 * VB, NT = (ACT + 31) / 32 * 32, LX = VB * ND2 + 1;
  static constexpr int SMEM = (int)sizeof(z64) * (VB * ND4 + 2 * ND2 * LX);
};
template <int ND>
__global__ void __launch_bounds__(XdTile<ND>::NT)
k_xd(DevCtx c, const z64 *__restrict__ X, const z64 *__restrict__ chi0q, const z64 *__restrict__ c0inv,
     z64 *__restrict__ XD, int minus_one) {
  typedef XdTile<ND> L;
  constexpr int ND2 = L::ND2, ND4 = L::ND4, NT = L::NT, LX = L::LX;
  extern __shared__ __align__(16) z64 xd_smem[];
  z64 *Ss = xd_smem, *Xs = Ss + L::VB * ND4;        // [VB][i3][i2] and [ch][i1][LX]
  const int t = threadIdx.x, N = c.N, nnu = 2 * c.iwf, p = blockIdx.y;
  const int v0 = blockIdx.x * L::VB, nv = min(L::VB, nnu - v0), w = nv * ND2;
  const size_t per = (size_t)ND2 * N, base = (size_t)2 * p * per + (size_t)v0 * ND2;
  for (int e = t; e < nv * ND4; e += NT) {
    const int i2 = e % ND2, r = e / ND2;             // r = g nd2 + i3
    z64 s = cmul(chi0q[((size_t)p * nnu + v0) * ND4 + e], c0inv[v0 * ND2 + r]);
    if (i2 == r % ND2 && minus_one) s.x -= 1.0;
    Ss[e] = s;
  }
  for (int e = t; e < 2 * ND2 * w; e += NT) {
    const int row = e / w, col = e % w;
    Xs[row * LX + col] = X[base + (size_t)row * N + col];
  }
  __syncthreads();
  const int jb = t % ND, ib = t / ND % ND, ch = t / ND2 % 2, g = t / (2 * ND2);
  if (t >= L::ACT || g >= nv) return;
  const z64 *sx = Xs + ch * ND2 * LX + g * ND2, *ss = Ss + g * ND4;
  z64 acc[ND][ND];
#pragma unroll
  for (int r = 0; r < ND; ++r)
#pragma unroll
    for (int s = 0; s < ND; ++s) acc[r][s] = czero<z64>();
#pragma unroll 1
  for (int i2 = 0; i2 < ND2; ++i2) {
    z64 y[ND];
#pragma unroll
    for (int s = 0; s < ND; ++s) y[s] = ss[(jb + ND * s) * ND2 + i2];
#pragma unroll
    for (int r = 0; r < ND; ++r) {
      const z64 x = sx[(ib + ND * r) * LX + i2];
#pragma unroll
      for (int s = 0; s < ND; ++s) cfma(acc[r][s], x, y[s]);
    }
  }
#pragma unroll
  for (int r = 0; r < ND; ++r)
#pragma unroll
    for (int s = 0; s < ND; ++s)
      XD[base + (size_t)(ch * ND2 + ib + ND * r) * N + g * ND2 + jb + ND * s] = acc[r][s];
}

// max that keeps a NaN (fmax drops it, and a point whose factors are not finite would pass for converged)
__device__ __forceinline__ double nanmax(double a, double b) { return b > a || b != b ? b : a; }

// X += up(V); per-matrix max |d| and max |X| (|re|+|im|, NaN if any is) into norms[2*m], norms[2*m+1]
__global__ void k_update(int per, const z32 *V, z64 *X, unsigned long long *norms, const int *active) {
  const int m = blockIdx.y;
  if (active && !active[m]) return;
  __shared__ double sd[8], sx[8];
  double md = 0.0, mx = 0.0;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < per; e += gridDim.x * blockDim.x) {
    z64 d = to64(V[(size_t)m * per + e]);
    z64 x = X[(size_t)m * per + e];
    x.x += d.x; x.y += d.y;
    X[(size_t)m * per + e] = x;
    md = nanmax(md, fabs(d.x) + fabs(d.y));
    mx = nanmax(mx, fabs(x.x) + fabs(x.y));
  }
  for (int o = 16; o > 0; o >>= 1) {
    md = nanmax(md, __shfl_xor_sync(0xffffffffu, md, o));
    mx = nanmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if ((threadIdx.x & 31) == 0) { sd[threadIdx.x >> 5] = md; sx[threadIdx.x >> 5] = mx; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) { md = nanmax(md, sd[w]); mx = nanmax(mx, sx[w]); }
    // non-negative doubles order like their bit patterns, a NaN of either sign above them
    atomicMax(norms + 2 * m, (unsigned long long)__double_as_longlong(md));
    atomicMax(norms + 2 * m + 1, (unsigned long long)__double_as_longlong(mx));
  }
}

cudaError_t launch_init_x(const z32 *T32, size_t strideM, int N, int R, int nmat, z64 *X, cudaStream_t st) {
  size_t total = (size_t)N * R * nmat;
  k_init_x<<<cdiv_u(total, 256), 256, 0, st>>>(T32, strideM, N, R, nmat, X);
  return ADGA_LAUNCH_CHECK();
}

cudaError_t launch_residual(const DevCtx &c, int npts, const z64 *X, const z64 *chi0q,
                            const z64 *c0inv, const z64 *Frow_d, const z64 *Frow_m,
                            const z64 *opg_d, const z64 *opg_m, z64 *XD, z32 *V, const z64 *extra_d,
                            unsigned long long *rnorm, cudaStream_t st, const z64 *Bpt, void *ri8,
                            long long fgen) {
  cudaError_t e = launch_xd(c, npts, X, chi0q, c0inv, XD, true, st);
  if (e != cudaSuccess) return e;
  if (ri8)
    return ri8_residual(ri8, c, npts, XD, X, Frow_d, Frow_m, fgen, opg_d, opg_m, V, extra_d, rnorm, Bpt, st);
  return launch_resid_z64(c, npts, XD, X, Frow_d, Frow_m, opg_d, opg_m, V, extra_d, rnorm, Bpt, st);
}

// XD = X blockdiag(chi0q chi0_loc^-1 - 1), or without the -1 (a tangent direction)
cudaError_t launch_xd(const DevCtx &c, int npts, const z64 *X, const z64 *chi0q, const z64 *c0inv, z64 *XD,
                      bool minus_one, cudaStream_t st) {
  if (npts <= 0) return cudaSuccess;
#define XDL(ND)                                                                                                   \
  do {                                                                                                            \
    typedef XdTile<ND> L;                                                                                         \
    cudaError_t e = smem_limit(k_xd<ND>, L::SMEM);                                                                \
    if (e != cudaSuccess) return e;                                                                               \
    k_xd<ND><<<dim3(cdiv_u(2 * c.iwf, L::VB), npts), L::NT, L::SMEM, st>>>(c, X, chi0q, c0inv, XD, minus_one);    \
    return ADGA_LAUNCH_CHECK();                                                                                   \
  } while (0)
  switch (c.nd) {
    case 1: XDL(1);
    case 2: XDL(2);
    case 3: XDL(3);
    case 4: XDL(4);
    case 5: XDL(5);
  }
#undef XDL
  return cudaErrorInvalidValue;
}

cudaError_t launch_update(int per, int nmat, const z32 *V, z64 *X, unsigned long long *norms,
                          const int *active, cudaStream_t st) {
  dim3 g(cdiv_u(per, 256 * 4), nmat);
  k_update<<<g, 256, 0, st>>>(per, V, X, norms, active);
  return ADGA_LAUNCH_CHECK();
}
