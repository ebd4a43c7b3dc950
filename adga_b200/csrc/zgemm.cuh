// Complex FP64 GEMM mainloop on the FP64 tensor cores (mma m8n8k4):
//     acc += sum_k A(r, k) B(k, c)
// for a 64 x 64 output tile, 128 threads, k-slices of BK = 16 through a
// double-buffered cp.async stage in shared memory.  A complex product is four
// real ones, re += Ar Br, re += (-Ai) Bi, im += Ar Bi, im += Ai Br, each
// accumulated in FP64 fused multiply-adds.
//
// The FP64 rate of the tensor cores is that of the CUDA cores (37.0 TFLOP/s
// measured either way); what they save is registers and operand reads: a warp's
// 32 x 32 tile needs 8 shared loads per 64 instructions and 128 accumulator
// registers, so three CTAs share an SM and one CTA's operand waits and its
// read-modify-write of C run under the others' products.  As 8 x 4 register
// tiles of fused multiply-adds (128 x 64 CTA tiles, one CTA per SM) the N = 1080
// trailing updates ran at 17.2 TFLOP/s, 46 % of that rate: 90.1 ms for 500
// matrices; this form: 52.8 ms (29.4 TFLOP/s).
//
// Operand access goes through loader functors returning the address of A(r, k)
// / B(k, c) (or nullptr outside the matrix, read as zero).  Shared layouts put
// the fast global index first; their strides (66 and 20 elements) make both the
// cp.async writes and the fragment reads (lane = 4 (r or c) + k) conflict-free.
#pragma once
#include "common.cuh"

namespace zg {

constexpr int BM = 64, BN = 64, BK = 16, NT = 128, STAGES = 2;
constexpr int LD_OUT = BM + 2, LD_K = BK + 4;       // [k][r] and [r][k] strides, elements
constexpr int ELEMS_OUT = BK * LD_OUT, ELEMS_K = BM * LD_K;
// one operand of a stage in each layout (A_KFAST == B_CFAST in every user): 73 KB, three CTAs per SM
constexpr int SMEM_BYTES = STAGES * (ELEMS_OUT + ELEMS_K) * 16;
static_assert(BM == BN, "square tiles");

// accumulators of a thread: element (mi, ni, e) is row row_of(mi), column col_of(ni, e) of the tile
struct Acc {
  double re[4][4][2], im[4][4][2];
};
__device__ __forceinline__ int row_of(int mi) {
  return 32 * ((threadIdx.x >> 5) & 1) + 8 * mi + ((threadIdx.x & 31) >> 2);
}
__device__ __forceinline__ int col_of(int ni, int e) { return 32 * (threadIdx.x >> 6) + 8 * ni + 2 * (threadIdx.x & 3) + e; }
__device__ __forceinline__ void clear(Acc &a) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) a.re[i][j][0] = a.re[i][j][1] = a.im[i][j][0] = a.im[i][j][1] = 0.0;
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, int nbytes) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(nbytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// A_KFAST: A(r, k) is contiguous in k (row-major A), else in r.
// B_CFAST: B(k, c) is contiguous in c (row-major B), else in k.
// `safe` is any valid global address (source of the zero-filled copies).
// mv, nv: rows and columns of the tile inside the matrix; a warp leaves out the 8 x 8 blocks
// beyond them (an LU with right-hand sides has a last column tile of a few columns).
template <bool A_KFAST, bool B_CFAST, class LA, class LB>
__device__ __forceinline__ void mainloop(Acc &acc, z64 *smem, int K, int mv, int nv, const LA &la, const LB &lb,
                                         const z64 *safe) {
  static_assert(A_KFAST == B_CFAST, "stage layout");
  constexpr int OFF_B = A_KFAST ? ELEMS_K : ELEMS_OUT, STAGE = ELEMS_OUT + ELEMS_K;
  constexpr int SA_R = A_KFAST ? LD_K : 1, SA_K = A_KFAST ? 1 : LD_OUT;
  constexpr int SB_C = B_CFAST ? 1 : LD_K, SB_K = B_CFAST ? LD_OUT : 1;
  const int t = threadIdx.x, lane = t & 31;
  const int nk = (K + BK - 1) / BK;
  auto load = [&](int kt) {
    if (kt < nk) {
      const int k0 = kt * BK;
      z64 *as = smem + (kt % STAGES) * STAGE, *bs = as + OFF_B;
#pragma unroll
      for (int q = 0; q < (BM * BK) / NT; ++q) {
        const int e = t + NT * q;
        const int r = A_KFAST ? e / BK : e % BM, kk = A_KFAST ? e % BK : e / BM;
        const z64 *g = la(r, k0 + kk);
        cp_async16(as + r * SA_R + kk * SA_K, g ? g : safe, g ? 16 : 0);
      }
#pragma unroll
      for (int q = 0; q < (BN * BK) / NT; ++q) {
        const int e = t + NT * q;
        const int kk = B_CFAST ? e / BN : e % BK, c = B_CFAST ? e % BN : e / BK;
        const z64 *g = lb(k0 + kk, c);
        cp_async16(bs + c * SB_C + kk * SB_K, g ? g : safe, g ? 16 : 0);
      }
    }
    cp_async_commit();
  };
  const int ra = 32 * ((t >> 5) & 1) + (lane >> 2), cb = 32 * (t >> 6) + (lane >> 2), kl = lane & 3;
  const int mi = min(4, (mv - 32 * ((t >> 5) & 1) + 7) >> 3), nj = min(4, (nv - 32 * (t >> 6) + 7) >> 3);
  const bool full = mi == 4 && nj == 4;
  load(0);
  for (int kt = 0; kt < nk; ++kt) {
    load(kt + 1);
    cp_async_wait<1>();
    __syncthreads();                 // slice kt landed
    const z64 *as = smem + (kt % STAGES) * STAGE + ra * SA_R + kl * SA_K;
    const z64 *bs = smem + (kt % STAGES) * STAGE + OFF_B + cb * SB_C + kl * SB_K;
    if (full) {
#pragma unroll
      for (int kk = 0; kk < BK; kk += 4) {
        z64 a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = as[8 * i * SA_R + kk * SA_K];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = bs[8 * j * SB_C + kk * SB_K];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const double an = -a[i].y;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            dmma(acc.re[i][j], a[i].x, b[j].x);
            dmma(acc.im[i][j], a[i].x, b[j].y);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            dmma(acc.re[i][j], an, b[j].y);
            dmma(acc.im[i][j], a[i].y, b[j].x);
          }
        }
      }
    } else if (mi > 0 && nj > 0) {
#pragma unroll 1
      for (int kk = 0; kk < BK; kk += 4) {
        z64 a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = as[8 * i * SA_R + kk * SA_K];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < nj) {
            const z64 b = bs[8 * j * SB_C + kk * SB_K];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (i < mi) {
                dmma(acc.re[i][j], a[i].x, b.x);
                dmma(acc.im[i][j], a[i].x, b.y);
                dmma(acc.re[i][j], -a[i].y, b.y);
                dmma(acc.im[i][j], a[i].y, b.x);
              }
          }
      }
    }
    __syncthreads();                 // slice kt read: its stage is free
  }
}

}  // namespace zg
