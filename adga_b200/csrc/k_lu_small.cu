// Small FP64 systems in one kernel: LU with partial pivoting of the N x N
// matrix with its R right-hand sides appended (lu.cuh's layout) and the back
// substitution, everything in shared memory, one CTA per matrix.
//
// Pivot choice and info are those of the blocked path (izamax: the largest
// |re|+|im|, the lowest row on ties).  Only U, its reciprocal pivots and the
// right-hand sides are kept: the multipliers of a column live in registers for
// the one rank-1 update that uses them, and the row interchange is done by that
// update (the row that takes the old diagonal row's place reads it from there).
//
// Bound by the serial chain of a column: warp 0 updates the next column first,
// searches it and takes the reciprocal of its pivot while the other warps
// update the rest, so a column costs one barrier.  The blocked path's five
// launches took 110 us (66 panel, 30 block inverses, 13 interchanges and
// solve) on one 40 x 40 matrix and 115 us on 250 of them; this kernel: 33 us
// and 43 us.
#include "ctx.cuh"
#include "lu.cuh"

namespace {

constexpr int NT = 256, NW = NT / 32, JU = 3;   // JU columns in flight per warp
constexpr int SMEM_MAX = 208 * 1024;

__host__ __device__ inline int small_ld(int N) { return N | 1; }
size_t small_smem(int N, int R) { return sizeof(z64) * ((size_t)small_ld(N) * (N + R) + N); }

// RL rows per lane: N <= 32 RL
template <int RL>
__global__ void __launch_bounds__(NT)
k_lu_small(z64 *M, size_t strideM, int N, int R, int *info_all) {
  extern __shared__ __align__(16) unsigned char small_raw[];
  z64 *A = reinterpret_cast<z64 *>(small_raw);
  const int LD = small_ld(N), NC = N + R, t = threadIdx.x, w = t >> 5, lane = t & 31;
  z64 *rcps = A + (size_t)LD * NC;             // 1 / U(k, k), NaN at a zero pivot
  __shared__ int s_p[2];
  z64 *G = M + (size_t)blockIdx.x * strideM;
  // columns by warps, rows by lanes
  for (int c = w; c < NC; c += NW)
#pragma unroll
    for (int q = 0; q < RL; ++q) {
      const int i = lane + 32 * q;
      if (i < N) A[i + c * LD] = G[i + (size_t)c * N];
    }
  __syncthreads();
  int info = 0;
  // warp 0: the pivot row of column k, whose rows x the lanes hold, and its reciprocal
  auto search = [&](int k, const z64 (&x)[RL]) {
    unsigned long long key = 0;
    int row = INT_MAX;
#pragma unroll
    for (int q = 0; q < RL; ++q) {
      const int i = lane + 32 * q;
      // 1 + the bits of a non-negative number order like the number; NaN is never a pivot
      unsigned long long u = (unsigned long long)__double_as_longlong(cabs1(x[q]));
      u = (i >= k && i < N && u <= 0x7ff0000000000000ULL) ? u + 1 : 0;
      if (u > key) { key = u; row = i; }
    }
    warp_argmax(key, row);
    int p = row;
    if (p == INT_MAX) p = k;                   // all NaN
    z64 piv = czero<z64>();                    // of lane p % 32
#pragma unroll
    for (int q = 0; q < RL; ++q) {
      const double a = __shfl_sync(0xffffffffu, x[q].x, p & 31), b = __shfl_sync(0xffffffffu, x[q].y, p & 31);
      if (RL == 1 || q == p >> 5) piv = make_double2(a, b);
    }
    const bool zero = key == 1;                // the largest |re|+|im| is zero
    if (zero && !info) info = k + 1;
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    const z64 r = zero ? make_double2(nan, nan) : crcp_scaled(piv);
    if (lane == 0) {
      rcps[k] = r;
      s_p[k & 1] = zero ? -1 - p : p;          // a zero pivot eliminates nothing
    }
  };
  if (w == 0) {
    z64 x[RL];
#pragma unroll
    for (int q = 0; q < RL; ++q) x[q] = lane + 32 * q < N ? A[lane + 32 * q] : czero<z64>();
    search(0, x);
  }
  __syncthreads();
  for (int k = 0; k < N; ++k) {
    const int pc = s_p[k & 1], p = pc < 0 ? -1 - pc : pc;
    const z64 rc = pc < 0 ? czero<z64>() : rcps[k];
    // this lane's rows: where they come from (rows k and p change places) and their multipliers
    int src[RL];
    z64 l[RL];
#pragma unroll
    for (int q = 0; q < RL; ++q) {
      const int i = min(lane + 32 * q, N - 1);
      src[q] = i == p ? k : i == k ? p : i;
      l[q] = cmul(A[src[q] + k * LD], rc);
    }
    // J columns j, j + NW - 1, ..: every load before a warp barrier, every store after it
    auto update = [&](int j, auto &v) {
      constexpr int J = sizeof(v) / sizeof(v[0]);
      z64 u[J];
#pragma unroll
      for (int c = 0; c < J; ++c) {
        const z64 *C = A + min(j + c * (NW - 1), NC - 1) * LD;
        u[c] = C[p];
#pragma unroll
        for (int q = 0; q < RL; ++q) v[c][q] = C[src[q]];
      }
      __syncwarp();
#pragma unroll
      for (int c = 0; c < J; ++c) {
        z64 *C = A + (j + c * (NW - 1)) * LD;
        const bool in = j + c * (NW - 1) < NC;
#pragma unroll
        for (int q = 0; q < RL; ++q) {
          const int i = lane + 32 * q;
          z64 x = v[c][q];
          cfms(x, l[q], u[c]);
          if (i > k) v[c][q] = x;              // row k takes the pivot row as it is
          if (in && i >= k && i < N) C[i] = v[c][q];
        }
      }
    };
    if (w == 0) {
      z64 v[1][RL];
      update(k + 1, v);
      if (k + 1 < N) search(k + 1, v[0]);
    } else {
      z64 v[JU][RL];
      for (int j = k + 1 + w; j < NC; j += JU * (NW - 1)) update(j, v);
    }
    __syncthreads();
  }
  // back substitution, one warp per right-hand side, its rows in registers
  for (int r = w; r < R; r += NW) {
    const z64 *Y = A + (N + r) * LD;
    z64 y[RL];
#pragma unroll
    for (int q = 0; q < RL; ++q) y[q] = lane + 32 * q < N ? Y[lane + 32 * q] : czero<z64>();
#pragma unroll
    for (int q = RL - 1; q >= 0; --q) {
      for (int k = min(N, 32 * q + 32) - 1; k >= 32 * q; --k) {
        const z64 xk = cmul(y[q], rcps[k]);    // of lane k % 32
        const z64 x = make_double2(__shfl_sync(0xffffffffu, xk.x, k & 31), __shfl_sync(0xffffffffu, xk.y, k & 31));
        const z64 *U = A + k * LD;
#pragma unroll
        for (int q2 = 0; q2 <= q; ++q2) {
          const int i = lane + 32 * q2;
          if (i < k) cfms(y[q2], U[i], x);
          else if (i == k) y[q2] = x;
        }
      }
    }
#pragma unroll
    for (int q = 0; q < RL; ++q)
      if (lane + 32 * q < N) G[lane + 32 * q + (size_t)(N + r) * N] = y[q];
  }
  if (t == 0) info_all[blockIdx.x] = info;
}

}  // namespace

// Up to N = 80 this kernel wins at every batch (us for 2 / 250 / 1000 matrices, here against the blocked
// path: N = 40 33 / 43 / 131 against 95 / 124 / 358, N = 80 125 / 168 / 594 against 193 / 257 / 753); at N = 96, one CTA per SM, it
// loses from about 250 matrices on (341 against 315 us).
constexpr int SMALL_N = 80;
bool lu_small_supported(int N, int R) { return N <= SMALL_N && small_smem(N, R) <= SMEM_MAX; }

cudaError_t lu_small_solve(z64 *M, size_t strideM, int N, int R, int batch, int *info, cudaStream_t st) {
  if (!lu_small_supported(N, R)) return cudaErrorInvalidValue;
  const int smem = (int)small_smem(N, R);
#define SMALL(RL)                                                                  \
  do {                                                                             \
    cudaError_t e = smem_limit(k_lu_small<RL>, SMEM_MAX);                          \
    if (e != cudaSuccess) return e;                                                \
    k_lu_small<RL><<<batch, NT, smem, st>>>(M, strideM, N, R, info);               \
  } while (0)
  if (N <= 32) SMALL(1);
  else if (N <= 64) SMALL(2);
  else SMALL(3);
#undef SMALL
  return ADGA_LAUNCH_CHECK();
}
