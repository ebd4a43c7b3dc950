// Complex FP64 GEMMs built on zgemm.cuh:
//   * k_trail_z64  -- the FP64 LU trailing update A22 -= L21 U12 (batched);
//   * k_resid_z64  -- the refinement residual r = B - X + (X D) F~ of the
//                     mixed path (rows = points x ndim2, K = N, F~ shared).
#include "ctx.cuh"
#include "lu.cuh"
#include "zgemm.cuh"

using namespace zg;

// Bound by the FP64 rate (8 flops per complex product; the C read and write takes two fifths of
// that time).  C's lines are prefetched into L2 before the products, and the difference is taken
// at the end: the sum over k is rounded at its own size and C once.
__global__ void __launch_bounds__(NT, 3)
k_trail_z64(z64 *M, size_t strideM, int N, int ncols, int J, int jb) {
  extern __shared__ __align__(16) z64 zg_smem[];
  z64 *A = M + (size_t)blockIdx.z * strideM;
  const int r0 = J + jb + blockIdx.y * BM, c0 = J + jb + blockIdx.x * BN;
  auto la = [&](int r, int k) -> const z64 * {
    const int rr = r0 + r;
    return (rr < N && k < jb) ? A + rr + (size_t)(J + k) * N : nullptr;
  };
  auto lb = [&](int k, int c) -> const z64 * {
    const int cc = c0 + c;
    return (k < jb && cc < ncols) ? A + (J + k) + (size_t)cc * N : nullptr;
  };
  {
    const int c = c0 + (threadIdx.x >> 1), r = r0 + 32 * (threadIdx.x & 1);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c < ncols && r + 8 * q < N) asm volatile("prefetch.global.L2 [%0];" ::"l"(A + r + 8 * q + (size_t)c * N));
  }
  Acc acc;
  clear(acc);
  mainloop<false, false>(acc, zg_smem, jb, N - r0, ncols - c0, la, lb, A);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = r0 + row_of(i);
    z64 cv[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = c0 + col_of(j, e);
        cv[j][e] = (r < N && c < ncols) ? A[r + (size_t)c * N] : make_double2(0.0, 0.0);
      }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = c0 + col_of(j, e);
        if (r < N && c < ncols)
          A[r + (size_t)c * N] = make_double2(cv[j][e].x - acc.re[i][j][e], cv[j][e].y - acc.im[i][j][e]);
      }
  }
}

cudaError_t lu_trail_z64(z64 *M, const LUBatch &lb, int J, int jb, cudaStream_t st) {
  const int m = lb.N - J - jb, n = lb.ncols - J - jb;
  if (m <= 0 || n <= 0) return cudaSuccess;
  smem_limit(k_trail_z64, SMEM_BYTES);
  dim3 grid(cdiv_u(n, BN), cdiv_u(m, BM), lb.batch);
  k_trail_z64<<<grid, NT, SMEM_BYTES, st>>>(M, lb.strideM, lb.N, lb.ncols, J, jb);
  return ADGA_LAUNCH_CHECK();
}

// rows (p, i1) of channel ch, columns c:
//   V(p,i1,c) = fp32( opg(i1,c) - X(p,i1,c) + sum_m XD(p,i1,m) F~(m,c) )
__global__ void __launch_bounds__(NT, 3)
k_resid_z64(int N, int R, int npts, int ch, const z64 *__restrict__ XD, const z64 *__restrict__ X,
            const z64 *__restrict__ Frow, const z64 *__restrict__ opg, z32 *V, const z64 *__restrict__ extra,
            unsigned long long *rnorm, const z64 *__restrict__ Bpt) {
  extern __shared__ __align__(16) z64 zg_smem[];
  const int rows = npts * R;
  const int r0 = blockIdx.y * BM, c0 = blockIdx.x * BN;
  const size_t per = (size_t)R * N;
  auto la = [&](int r, int k) -> const z64 * {
    const int row = r0 + r;
    if (row >= rows || k >= N) return nullptr;
    const int p = row / R, i1 = row % R;
    return XD + (size_t)(2 * p + ch) * per + (size_t)i1 * N + k;
  };
  auto lb = [&](int k, int c) -> const z64 * {
    const int cl = c0 + c;
    return (k < N && cl < N) ? Frow + (size_t)k * N + cl : nullptr;
  };
  Acc acc;
  clear(acc);
  mainloop<true, true>(acc, zg_smem, N, rows - r0, N - c0, la, lb, Frow);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = r0 + row_of(i);
    const int p = row / R, i1 = row % R;
    const size_t m = (size_t)(2 * p + ch);
    double rmax = 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int cl = c0 + col_of(j, e);
        if (row >= rows || cl >= N) continue;
        // right-hand side: (1+gamma^w) shared by the slice, or per point (tangent solves)
        const z64 b = Bpt ? Bpt[m * per + (size_t)i1 * N + cl] : opg[i1 + (size_t)cl * R];
        const z64 x = X[m * per + (size_t)i1 * N + cl];
        z64 r = make_double2(b.x - x.x + acc.re[i][j][e], b.y - x.y + acc.im[i][j][e]);
        if (extra) r = cadd(r, extra[(size_t)p * per + (size_t)i1 * N + cl]);   // V(q) term (density)
        V[m * per + (size_t)i1 * N + cl] = to32(r);
        rmax = fmax(rmax, fabs(r.x) + fabs(r.y));
      }
    // max |re| + |im| of the FP64 residual per matrix (four lanes share a row)
    rmax = fmax(rmax, __shfl_xor_sync(0xffffffffu, rmax, 1));
    rmax = fmax(rmax, __shfl_xor_sync(0xffffffffu, rmax, 2));
    if (rnorm && threadIdx.x % 4 == 0 && row < rows && rmax > 0.0)
      atomicMax(rnorm + (size_t)(2 * p + ch), (unsigned long long)__double_as_longlong(rmax));
  }
}

cudaError_t launch_resid_z64(const DevCtx &c, int npts, const z64 *XD, const z64 *X,
                             const z64 *Frow_d, const z64 *Frow_m, const z64 *opg_d,
                             const z64 *opg_m, z32 *V, const z64 *extra_d, unsigned long long *rnorm,
                             const z64 *Bpt, cudaStream_t st) {
  smem_limit(k_resid_z64, SMEM_BYTES);
  dim3 g(cdiv_u(c.N, BN), cdiv_u((size_t)npts * c.R, BM));
  k_resid_z64<<<g, NT, SMEM_BYTES, st>>>(c.N, c.R, npts, 0, XD, X, Frow_d, opg_d, V, extra_d, rnorm, Bpt);
  cudaError_t e = ADGA_LAUNCH_CHECK();
  if (e != cudaSuccess) return e;
  k_resid_z64<<<g, NT, SMEM_BYTES, st>>>(c.N, c.R, npts, 1, XD, X, Frow_m, opg_m, V, nullptr, rnorm, Bpt);
  return ADGA_LAUNCH_CHECK();
}
