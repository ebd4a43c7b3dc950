// Batched blocked right-looking LU with partial pivoting (complex FP64 or
// FP32) and blocked triangular solves; see lu.cuh for the layout.
//
// Per step J (panel width NB):
//   k_panel      one CTA per matrix factors rows J..N of the NB panel columns
//                in 2- to 16-column sub-panels held in registers (pivot search,
//                row swap and rank-1 updates never leave the SM), with
//                right-looking updates of the rest of the panel;
//   k_triinv     inverts the unit-lower and upper NB x NB diagonal blocks;
//   k_swap_trsm  applies the panel's row interchanges to the other columns
//                and forms U12 = L11^-1 A12 as a small GEMM (FP64:
//                k_swap_trsm_d, on the tensor cores);
//   trailing     A22 -= L21 U12 (FP64: k_zgemm.cu; FP32: the CUDA-core GEMM
//                below, or the tensor-core BF16x3 kernel of the mixed path).
// Pivot choice follows izamax: the largest |re|+|im|, the lowest row on ties.
#include "lu.cuh"
#include "zgemm.cuh"
#include <algorithm>


// ---------------------------------------------------------------------------
// Panel factorisation, one CTA per matrix: SW-column sub-panels live in
// registers (thread t holds rows J + t + q nt), and the rest of the panel takes
// their interchanges, triangular solve and rank-SW update from global memory.
//
// Bound by the serial chain of a column on few rows, by the passes over the
// panel on many.  The pivot search is three integer warp reductions over the
// bit pattern of |re|+|im| (high word, low word, then the lowest row), every
// warp's candidate row is put in shared memory beside its key before the one
// barrier of the column, and after it every warp reduces the candidates itself,
// so that neither a second reduction stage nor a row broadcast needs another
// barrier; the buffers alternate with the column's parity.  Rows keep their
// registers: an interchange only swaps the positions they stand for.  The next
// column is updated and searched before the rest of the row.  Sub-panels of 16
// columns where one row per thread fits (rows <= 512: half the passes over the
// rest of the panel), else of 8 and less.
// With double-precision shuffles, three barriers a column, rows moved through
// shared memory and a serially composed interchange map: 137 us for a 40 x 40
// panel, 310 us for 357 x 64, 417 us for 1016 x 64, 1799 us for 500 of those;
// this form: 40 us, 110 us, 250 us and 1193 us.
// ---------------------------------------------------------------------------
template <typename T, int SW> struct PanelShared {
  unsigned long long key[2][32];
  int row[2][32];
  T cand[2][32][SW];           // each warp's candidate row, from the column on
  T Lss[SW * SW];
  int piv[SW], dst[2 * SW], src[2 * SW], cnt;
};

// the warp's candidate for column CC: the row with the largest key, put beside the key
template <typename T, int RPT, int SW, int CC>
__device__ __forceinline__ void panel_search(const T (&a)[RPT][SW], const int (&pos)[RPT], int N, int col,
                                             unsigned long long &key, int &row) {
  key = 0;
  row = INT_MAX;
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    // 1 + the bits of a non-negative number order like the number; NaN is never a pivot
    unsigned long long k = (unsigned long long)__double_as_longlong((double)cabs1(a[q][CC]));
    k = (pos[q] >= col && pos[q] < N && k <= 0x7ff0000000000000ULL) ? k + 1 : 0;
    if (k > key || (k == key && k && pos[q] < row)) { key = k; row = pos[q]; }
  }
  warp_argmax(key, row);
}

// One column CC of the register-resident sub-panel.  CC is a compile-time
// constant so that every index into the register array is static.  Rows do not
// move: pos is the row of the matrix that a register row stands for, and an
// interchange swaps two positions.  The next column is updated and searched
// before the rest of the row.
template <typename T, int RPT, int SW, int CC>
__device__ __forceinline__ void panel_column(T (&a)[RPT][SW], int (&pos)[RPT], PanelShared<T, SW> &S, int N, int c0,
                                             int sw, int t, int nt, int *ipiv, int &info, unsigned long long &key,
                                             int &row) {
  if (CC >= sw) return;
  const int lane = t & 31, warp = t >> 5, nw = nt >> 5, par = CC & 1;
  const int col = c0 + CC;
#pragma unroll
  for (int q = 0; q < RPT; ++q)
    if (key && pos[q] == row)
#pragma unroll
      for (int c2 = CC; c2 < SW; ++c2) S.cand[par][warp][c2] = a[q][c2];
  if (lane == 0) { S.key[par][warp] = key; S.row[par][warp] = row; }
  __syncthreads();
  unsigned long long k2 = lane < nw ? S.key[par][lane] : 0;
  int p = lane < nw ? S.row[par][lane] : INT_MAX;
  const int rl = p;
  warp_argmax(k2, p);
  const unsigned who = __ballot_sync(0xffffffffu, k2 && rl == p && lane < nw);
  T rcp = czero<T>();
  const T *prow = S.cand[par][who ? __ffs(who) - 1 : 0];
  const bool zero = k2 <= 1;               // the largest |re|+|im| is zero, or no row is eligible (all NaN)
  if (!who) p = col;
  if (k2 == 1 && info == 0) info = col + 1;
  if (!zero) rcp = crcp_scaled(prow[CC]);
  T l[RPT];
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    pos[q] = pos[q] == p ? col : pos[q] == col ? p : pos[q];
    const bool below = pos[q] > col && pos[q] < N;
    if (below && !zero) a[q][CC] = cmul(a[q][CC], rcp);
    l[q] = below ? a[q][CC] : czero<T>();       // all NaN: NaN, whatever prow holds then
  }
  if (CC + 1 < SW) {
    const T u = prow[CC + 1 < SW ? CC + 1 : CC];
#pragma unroll
    for (int q = 0; q < RPT; ++q) cfms(a[q][CC + 1 < SW ? CC + 1 : CC], l[q], u);
    panel_search<T, RPT, SW, (CC + 1 < SW ? CC + 1 : CC)>(a, pos, N, col + 1, key, row);
  }
#pragma unroll
  for (int c2 = CC + 2; c2 < SW; ++c2) {
    const T u = prow[c2];
#pragma unroll
    for (int q = 0; q < RPT; ++q) cfms(a[q][c2], l[q], u);
  }
  if (t == 0) { S.piv[CC] = p; ipiv[col] = p; }
}

template <typename T, int RPT, int SW, int CC>
__device__ __forceinline__ void panel_columns(T (&a)[RPT][SW], int (&pos)[RPT], PanelShared<T, SW> &S, int N, int c0,
                                              int sw, int t, int nt, int *ipiv, int &info, unsigned long long &key,
                                              int &row) {
  if constexpr (CC < SW) {
    panel_column<T, RPT, SW, CC>(a, pos, S, N, c0, sw, t, nt, ipiv, info, key, row);
    panel_columns<T, RPT, SW, CC + 1>(a, pos, S, N, c0, sw, t, nt, ipiv, info, key, row);
  }
}

// One row per thread (rows <= 512): the rank-16 update of the rest of the panel on the FP64 tensor cores, whose
// operands a warp reads once per 8 x 8 tile (a thread's row times broadcast U entries is bound by the shared-
// memory reads: 46k against 30k clocks for the first update at 357 rows).  More rows per thread: their update is
// bound by the memory passes, where a thread's own rows measured better (1016 rows: 250 against 278 us a panel).
template <typename T, int RPT> constexpr bool panel_mma() { return sizeof(T) == sizeof(z64) && RPT == 1; }
// stride of the staged multipliers: 2 mod 8 elements, conflict-free fragment reads (lane = 4 row + k)
__host__ __device__ inline int panel_lr(int rows) { return (rows + 7) / 8 * 8 + 2; }

template <typename T, int RPT, int SW, int NTMAX>
__global__ void __launch_bounds__(NTMAX, 1)
k_panel(T *M, size_t strideM, int N, int J, int jb, int *ipiv_all, int *info_all) {
  const int b = blockIdx.x;
  T *A = M + (size_t)b * strideM;
  int *ipiv = ipiv_all + (size_t)b * N;
  const int nt = blockDim.x, t = threadIdx.x;
  __shared__ PanelShared<T, SW> S;
  extern __shared__ __align__(16) unsigned char panel_dyn[];
  T *Gs = reinterpret_cast<T *>(panel_dyn);        // [jb - sw columns][2 SW]: moved rows, then U in the first SW
  T *Ls = Gs + 64 * 2 * SW;                        // panel_mma: the sub-panel's multipliers, [SW][LR]
  const int LR = panel_lr(N - J);
  int info = info_all[b];
  T a[RPT][SW];

#pragma unroll 1
  for (int s = 0; s < jb; s += SW) {
    const int sw = min(SW, jb - s), c0 = J + s;
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      const int r = J + t + q * nt;
#pragma unroll
      for (int cc = 0; cc < SW; ++cc)
        a[q][cc] = (r >= c0 && r < N && cc < sw) ? A[r + (size_t)(c0 + cc) * N] : czero<T>();
    }
    int pos[RPT], row;
    unsigned long long key;
#pragma unroll
    for (int q = 0; q < RPT; ++q) pos[q] = J + t + q * nt;
    panel_search<T, RPT, SW, 0>(a, pos, N, c0, key, row);
    panel_columns<T, RPT, SW, 0>(a, pos, S, N, c0, sw, t, nt, ipiv, info, key, row);
    // the sub-panel back to the matrix; its L block for the solve below
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      const int r = pos[q];
      if (r >= c0 && r < N) {
#pragma unroll
        for (int cc = 0; cc < SW; ++cc)
          if (cc < sw) A[r + (size_t)(c0 + cc) * N] = a[q][cc];
        const int i = r - c0;
        if (i < SW)
#pragma unroll
          for (int cc = 0; cc < SW; ++cc) S.Lss[i + cc * SW] = a[q][cc];
        else if (panel_mma<T, RPT>())
#pragma unroll
          for (int cc = 0; cc < SW; ++cc) Ls[(size_t)cc * LR + r - J] = a[q][cc];
      }
    }
    if (jb == sw) break;                           // the panel is this sub-panel
    __syncthreads();                               // S.piv complete
    if (t < 32) {
      // the interchanges as (dst <- src): the sub-panel's positions, then the other touched rows
      const int me = t % SW;
      const bool top = t < SW;
      const int pos = top ? c0 + me : S.piv[me];
      bool use = t < 2 * SW && me < sw && (top || pos >= c0 + sw);
      int x = pos;
#pragma unroll
      for (int i = SW - 1; i >= 0; --i) {
        if (i >= sw) continue;
        const int p = S.piv[i];
        if (x == c0 + i) x = p;
        else if (x == p) x = c0 + i;
        if (!top && i < me && p == pos) use = false;       // listed already
      }
      const unsigned m = __ballot_sync(0xffffffffu, use);
      if (use) {
        const int k = __popc(m & ((1u << t) - 1));
        S.dst[k] = pos;
        S.src[k] = x;
      }
      if (t == 0) S.cnt = __popc(m);
    }
    __syncthreads();
    // the touched rows of the other panel columns, and the rows of U to solve: every load before a
    // barrier, every store after it
    const int nother = jb - sw, mc = S.cnt;
#pragma unroll 2
    for (int e = t; e < nother * mc; e += nt) {
      const int u = e / mc, k = e - u * mc;
      const int col = u < s ? J + u : c0 + sw + (u - s);
      Gs[u * 2 * SW + k] = A[(size_t)S.src[k] + (size_t)col * N];
    }
    __syncthreads();
    const int nright = jb - s - sw;
#pragma unroll 2
    for (int e = t; e < nother * mc; e += nt) {
      const int u = e / mc, k = e - u * mc;
      const int col = u < s ? J + u : c0 + sw + (u - s);
      if (u < s ? S.src[k] != S.dst[k] : k >= sw) A[(size_t)S.dst[k] + (size_t)col * N] = Gs[u * 2 * SW + k];
    }
    // U rows of the right panel columns: unit-lower solve with Lss, one thread a column
    for (int u = nt - 1 - t; u < nright; u += nt) {
      T *g = Gs + (s + u) * 2 * SW, *Ac = A + c0 + (size_t)(c0 + sw + u) * N;
      // columns are left, so sw == SW; in blocks of at most 8 rows (registers)
      constexpr int HB = SW < 8 ? SW : 8;
#pragma unroll 1
      for (int h = 0; h < SW; h += HB) {
        T x[HB];
#pragma unroll
        for (int i = 0; i < HB; ++i) x[i] = g[h + i];
#pragma unroll 1
        for (int k = 0; k < h; ++k) {
          const T y = g[k];
#pragma unroll
          for (int i = 0; i < HB; ++i) cfms(x[i], S.Lss[h + i + k * SW], y);
        }
#pragma unroll
        for (int k = 0; k < HB - 1; ++k)
#pragma unroll
          for (int i = k + 1; i < HB; ++i) cfms(x[i], S.Lss[h + i + (h + k) * SW], x[k]);
#pragma unroll
        for (int i = 0; i < HB; ++i) { Ac[h + i] = x[i]; g[h + i] = x[i]; }
      }
    }
    __syncthreads();
    // rank-SW update of the rows below, right panel columns (a full sub-panel: sw == SW whenever columns
    // are left)
    if constexpr (panel_mma<T, RPT>()) {
      // warps take 8-row tiles, eight columns at a time, on the FP64 tensor cores: C - L U with C as the
      // accumulators' start
      const int warp = t >> 5, lane = t & 31, kl = lane & 3, rl = lane >> 2;
      const T *U = Gs + s * 2 * SW;
      for (int m0 = c0 + sw + 8 * warp; m0 < N; m0 += 8 * (nt >> 5)) {
        const int r = m0 + rl;
        z64 l[(SW + 3) / 4];
#pragma unroll
        for (int k = 0; k < (SW + 3) / 4; ++k)
          l[k] = 4 * k + kl < SW && r < N ? Ls[(size_t)(4 * k + kl) * LR + r - J] : czero<z64>();
        constexpr int NB = 2;                      // column tiles in flight
        for (int n0 = 0; n0 < nright; n0 += 8 * NB) {
          double re[NB][2], im[NB][2];
#pragma unroll
          for (int j = 0; j < NB; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int c = n0 + 8 * j + 2 * kl + e;
              const z64 v = r < N && c < nright ? A[r + (size_t)(c0 + sw + c) * N] : czero<z64>();
              re[j][e] = v.x;
              im[j][e] = v.y;
            }
#pragma unroll
          for (int k = 0; k < (SW + 3) / 4; ++k)
#pragma unroll
            for (int j = 0; j < NB; ++j) {
              const int c = n0 + 8 * j + rl;
              const z64 u = c < nright && 4 * k + kl < SW ? U[c * 2 * SW + 4 * k + kl] : czero<z64>();
              zg::dmma(re[j], -l[k].x, u.x);
              zg::dmma(im[j], -l[k].x, u.y);
              zg::dmma(re[j], l[k].y, u.y);
              zg::dmma(im[j], -l[k].y, u.x);
            }
#pragma unroll
          for (int j = 0; j < NB; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int c = n0 + 8 * j + 2 * kl + e;
              if (r < N && c < nright) A[r + (size_t)(c0 + sw + c) * N] = make_double2(re[j][e], im[j][e]);
            }
        }
      }
    } else if (nright > 0) {
      // the thread's own rows, in chunks of CW columns whose loads are all issued before their stores
      constexpr int CW = sizeof(T) == 8 ? 4 : 2;
      const T *U = Gs + s * 2 * SW;
      T *ar[RPT];
      bool in[RPT];
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        in[q] = pos[q] >= c0 + sw && pos[q] < N;
        ar[q] = A + pos[q] + (size_t)(c0 + sw) * N;
      }
#pragma unroll 1
      for (int u0 = 0; u0 < nright; u0 += CW) {
        T v[RPT][CW];
#pragma unroll
        for (int q = 0; q < RPT; ++q)
          if (in[q])
#pragma unroll
            for (int j = 0; j < CW; ++j)
              if (u0 + j < nright) v[q][j] = ar[q][(size_t)(u0 + j) * N];
#pragma unroll
        for (int j = 0; j < CW; ++j)
#pragma unroll
          for (int i = 0; i < SW; ++i) {
            const T y = U[(u0 + j) * 2 * SW + i];
#pragma unroll
            for (int q = 0; q < RPT; ++q) cfms(v[q][j], a[q][i], y);
          }
#pragma unroll
        for (int q = 0; q < RPT; ++q)
          if (in[q])
#pragma unroll
            for (int j = 0; j < CW; ++j)
              if (u0 + j < nright) ar[q][(size_t)(u0 + j) * N] = v[q][j];
      }
    }
    __syncthreads();
  }
  if (t == 0) info_all[b] = info;
}

// ---------------------------------------------------------------------------
// Inverses of the step's diagonal block, unit-lower L11^-1 and upper U11^-1,
// and the step's interchanges as one row map.
//
// One CTA per matrix, bound by latency (a 64 x 64 block is 175k complex FMAs).
// Both inverses live in the factored block's own array: strictly lower part
// L^-1, upper part U^-1.  Eight warps invert the 16 x 16 diagonal blocks of
// the two triangles (lane = column, right-looking so that the updates of a
// column step are independent), then two levels of recursive doubling join
// them, X10 = -X11 (L10 X00) and Y01 = -Y00 (U01 Y11), the inner product
// taking the place of L10 / U01.  Blocks wholly outside jb are skipped.  66 KB
// of shared memory in FP64: three CTAs per SM.
// The row map: the content of position x after the interchanges (J+i <-> p_i,
// in order) came from the position reached by undoing them from the last to
// the first, one thread per touched position.
// Column by column through shared memory (xTRTI2's order) with the map
// composed by one thread: 187 us on a single 64 x 64 block, 391 us per step of
// 500 blocks; this form: 30 us and 74 us.
// ---------------------------------------------------------------------------
constexpr int TI_LD = 65;
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 8 ? 4 : 3)
k_triinv(const T *M, size_t strideM, int N, int J, int jb, int NB, int nsteps, T *Linv, T *Uinv,
         const int *ipiv_all, int *rmap_all) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T *D = reinterpret_cast<T *>(smraw);          // [64][TI_LD], column-major
  __shared__ T rcps[64];
  __shared__ int piv[64], s_cnt;
  const int b = blockIdx.x, t = threadIdx.x, w = t >> 5, lane = t & 31;
  const T *A = M + (size_t)b * strideM;
  const T one = cx<T>::make(1, 0), zero = czero<T>();
#pragma unroll 4
  for (int e = t; e < 64 * 64; e += 256) {
    const int i = e & 63, j = e >> 6;           // identity outside the jb x jb block
    D[i + j * TI_LD] = (i < jb && j < jb) ? A[(size_t)(J + i) + (size_t)(J + j) * N] : (i == j ? one : zero);
  }
  if (t < jb) piv[t] = ipiv_all[(size_t)b * N + J + t];
  if (t == 0) s_cnt = 0;
  __syncthreads();
  if (t < 64) rcps[t] = crcp(D[t + t * TI_LD]);
  if (t >= 128 && (t & 63) < jb) {
    // warps 4..7: positions J + i (t < 192) and the pivots' own rows below the block
    const int me = t & 63, pos = t < 192 ? J + me : piv[me];
    bool use = t < 192 || pos >= J + jb;
    int x = pos;
    for (int i = jb - 1; i >= 0; --i) {
      const int p = piv[i];
      if (x == J + i) x = p;
      else if (x == p) x = J + i;
      if (t >= 192 && i < me && p == pos) use = false;     // listed by an earlier interchange
    }
    if (use && x != pos) {
      const int k = atomicAdd(&s_cnt, 1);
      int *rm = rmap_all + (size_t)b * RMAP_STRIDE;
      rm[1 + 2 * k] = pos;
      rm[2 + 2 * k] = x;
    }
  }
  __syncthreads();
  if (t == 0) rmap_all[(size_t)b * RMAP_STRIDE] = s_cnt;
  const int o16 = 16 * (w & 3);
  if (o16 < jb && lane < 16) {
    const int l = lane;
    T x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) x[r] = r == l ? one : zero;
    const T *B = D + o16 + o16 * TI_LD;
    if (w < 4) {
#pragma unroll
      for (int k = 0; k < 15; ++k)
#pragma unroll
        for (int r = k + 1; r < 16; ++r) cfms(x[r], B[r + k * TI_LD], x[k]);
    } else {
#pragma unroll
      for (int k = 15; k >= 0; --k) {
        x[k] = cmul(x[k], rcps[o16 + k]);
#pragma unroll
        for (int r = 0; r < k; ++r) cfms(x[r], B[r + k * TI_LD], x[k]);
      }
    }
    __syncwarp(0x0000ffffu);          // every lane has read its triangle of the block
    T *C = D + o16 + (o16 + l) * TI_LD;
#pragma unroll
    for (int r = 0; r < 16; ++r)
      if (w < 4 ? r > l : r <= l) C[r] = x[r];
  }
  __syncthreads();
  // entries of the two inverses: L^-1 with its unit diagonal and zeros above, U^-1 with zeros below
  auto xl = [&](int r, int c) { return r > c ? D[r + c * TI_LD] : (r == c ? one : zero); };
  auto xu = [&](int r, int c) { return r <= c ? D[r + c * TI_LD] : zero; };
  if (jb > 16) {
    // 16 -> 32, blocks at o = 0 and 32: warp w takes product w >> 1 (L at 0, 32, then U at 0, 32),
    // columns 8 (w & 1).. + 7; lane: row lane & 15, columns 4 (lane >> 4) + q
    const bool up = w >= 4;
    const int o = 32 * ((w >> 1) & 1), i = lane & 15, j0 = 8 * (w & 1) + 4 * (lane >> 4);
    T v[4], y[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = y[q] = zero;
    if (o + 16 < jb) {
#pragma unroll 4
      for (int k = 0; k < 16; ++k) {
        const T d = up ? D[(o + i) + (o + 16 + k) * TI_LD] : D[(o + 16 + i) + (o + k) * TI_LD];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          cfma(v[q], d, up ? xu(o + 16 + k, o + 16 + j0 + q) : xl(o + k, o + j0 + q));
      }
    }
    T *P = up ? D + o + (o + 16) * TI_LD : D + o + 16 + o * TI_LD;     // the off-diagonal block
    __syncthreads();
    if (o + 16 < jb) {
#pragma unroll
      for (int q = 0; q < 4; ++q) P[i + (j0 + q) * TI_LD] = v[q];
    }
    __syncthreads();
    if (o + 16 < jb) {
#pragma unroll 4
      for (int k = 0; k < 16; ++k) {
        const T x = up ? xu(o + i, o + k) : xl(o + 16 + i, o + 16 + k);
#pragma unroll
        for (int q = 0; q < 4; ++q) cfms(y[q], x, P[k + (j0 + q) * TI_LD]);
      }
    }
    __syncthreads();
    if (o + 16 < jb) {
#pragma unroll
      for (int q = 0; q < 4; ++q) P[i + (j0 + q) * TI_LD] = y[q];
    }
    __syncthreads();
  }
  if (jb > 32) {
    // 32 -> 64: warps 0..3 L, 4..7 U; warp columns 8 (w & 3) + q, lane = row.  X00(k, j) = 0 for
    // k < j and Y11(k, j) = 0 for k > j: the inner products take the triangular half of the work
    const bool up = w >= 4;
    const int i = lane, j0 = 8 * (w & 3);
    T v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = zero;
    T *P = up ? D + 32 * TI_LD : D + 32;
    const int k0 = up ? 0 : j0, k1 = up ? j0 + 8 : 32;
#pragma unroll 2
    for (int k = k0; k < k1; ++k) {
      const T d = P[i + k * TI_LD];
#pragma unroll
      for (int q = 0; q < 8; ++q) cfma(v[q], d, up ? xu(32 + k, 32 + j0 + q) : xl(k, j0 + q));
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      P[i + (j0 + q) * TI_LD] = v[q];
      v[q] = zero;
    }
    __syncwarp();                     // a warp's product columns are read by that warp only
#pragma unroll 2
    for (int k = 0; k < 32; ++k) {
      const T x = up ? xu(i, k) : xl(32 + i, 32 + k);
#pragma unroll
      for (int q = 0; q < 8; ++q) cfms(v[q], x, P[k + (j0 + q) * TI_LD]);
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 8; ++q) P[i + (j0 + q) * TI_LD] = v[q];
    __syncthreads();
  }
  const size_t off = ((size_t)b * nsteps + J / NB) * NB * NB;
#pragma unroll 4
  for (int e = t; e < NB * NB; e += 256) {
    const int i = e % NB, k = e / NB;
    const bool in = i < jb && k < jb;
    Linv[off + e] = in ? xl(i, k) : zero;
    Uinv[off + e] = in ? xu(i, k) : zero;
  }
}

// ---------------------------------------------------------------------------
// Row interchanges of one step on the columns outside the panel, then
// U12 = L11^-1 A12 on the right columns (a jb x jb x TW product).
//
// The interchange map of the step (at most 2*NB <= 128 rows for NB <= 64) is
// applied to a TW-column tile with every load issued before a barrier and
// every store after it; thread (t % 64, t / 64) moves rows t%64 and t%64 + 64
// of columns t/64 + 4v.  Left tiles (columns left of the panel, needed by the
// forward solves) only swap rows and run in k_swap_left, which holds no
// dynamic shared memory.  A k_swap_trsm CTA stages L11^-1 (lower triangle,
// zero above) once and walks TPC column tiles: swap, stage the A12 tile,
// multiply.  Both operands are arranged so that the FP32 path uses packed
// two-lane FMAs (L as (re, re, -im, im), A12 as (re, im, im, re)).  Warp w
// owns row blocks w and 15 - w (4 rows each), so every warp does the same
// triangular k work; lane (r, cq) owns row r of each block and columns
// cq + 8n (n < 4).
// ---------------------------------------------------------------------------
#define TW 32
constexpr int TS_LD = 65;        // A12 tile column stride (elements) in shared memory
constexpr int TPC = 4;           // column tiles per k_swap_trsm CTA (L11^-1 staged once)

template <typename T>
__device__ __forceinline__ int load_map(const int *rm, int *s_map) {
  const int cnt = min(rm[0], 128);
  for (int i = threadIdx.x; i < 2 * cnt; i += 256) s_map[i] = rm[1 + i];
  return cnt;
}
// every load of the tile before a barrier, every store after it (s_map loaded and synced)
template <typename T>
__device__ __forceinline__ void swap_tile(T *A, int N, int cnt, int cs, int nc, const int *s_map) {
  const int t = threadIdx.x, kk = t & 63, cc = t >> 6;
  T v[2][8];
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int k = kk + 64 * u, c = cc + 4 * w;
      if (k < cnt && c < nc) v[u][w] = A[(size_t)s_map[2 * k + 1] + (size_t)(cs + c) * N];
    }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int k = kk + 64 * u, c = cc + 4 * w;
      if (k < cnt && c < nc) A[(size_t)s_map[2 * k] + (size_t)(cs + c) * N] = v[u][w];
    }
}

template <typename T>
__global__ void __launch_bounds__(256)
k_swap_left(T *M, size_t strideM, int N, int J, const int *rmap_all) {
  __shared__ int s_map[4 * 64];
  const int cs = blockIdx.x * TW, b = blockIdx.y;
  const int cnt = load_map<T>(rmap_all + (size_t)b * RMAP_STRIDE, s_map);
  __syncthreads();
  swap_tile<T>(M + (size_t)b * strideM, N, cnt, cs, min(J, cs + TW) - cs, s_map);
}

struct TrsmOp {
  typedef float4 L;
  typedef float4 X;
  static __device__ __forceinline__ L packL(z32 l) { return make_float4(l.x, l.x, -l.y, l.y); }
  static __device__ __forceinline__ X packX(z32 x) { return make_float4(x.x, x.y, x.y, x.x); }
  static __device__ __forceinline__ void fma(z32 &acc, const L &l, const X &x) {
    acc = __ffma2_rn(make_float2(l.x, l.y), make_float2(x.x, x.y), acc);
    acc = __ffma2_rn(make_float2(l.z, l.w), make_float2(x.z, x.w), acc);
  }
};

__global__ void __launch_bounds__(256)
k_swap_trsm(z32 *M, size_t strideM, int N, int ncols, int J, int jb, int NB, int nsteps,
            const int *rmap_all, const z32 *Linv) {
  typedef z32 T;
  typedef TrsmOp Op;
  extern __shared__ __align__(16) unsigned char smraw[];
  Op::L *Ls = reinterpret_cast<Op::L *>(smraw);           // [64 k][64 i]
  Op::X *Xs = reinterpret_cast<Op::X *>(Ls + 64 * 64);    // [TW c][TS_LD k]
  __shared__ int s_map[4 * 64];
  const int b = blockIdx.y, t = threadIdx.x;
  T *A = M + (size_t)b * strideM;
  const T *L = Linv + ((size_t)b * nsteps + J / NB) * NB * NB;
  for (int e = t; e < 64 * 64; e += 256) {
    const int i = e & 63, k = e >> 6;
    Ls[e] = Op::packL((i < jb && k <= i) ? L[i + k * NB] : czero<T>());
  }
  const int cnt = load_map<T>(rmap_all + (size_t)b * RMAP_STRIDE, s_map);
  // warp w owns row blocks w and 15-w (4 rows each): equal k work per warp
  const int warp = t >> 5, lane = t & 31, r = lane & 3, cq = lane >> 2;
  const int ia = 4 * warp + r, ib = 4 * (15 - warp) + r;
  const int ka = min(4 * warp + 4, jb), kb = min(4 * (16 - warp), jb);
  for (int tile = 0; tile < TPC; ++tile) {
    const int cs = J + jb + (blockIdx.x * TPC + tile) * TW;
    if (cs >= ncols) break;
    const int nc = min(ncols, cs + TW) - cs;
    __syncthreads();               // map and L staged; the previous tile's Xs reads are done
    swap_tile<T>(A, N, cnt, cs, nc, s_map);
    __syncthreads();
    for (int e = t; e < 64 * TW; e += 256) {
      const int k = e & 63, c = e >> 6;
      Xs[k + c * TS_LD] =
          Op::packX((k < jb && c < nc) ? A[(size_t)(J + k) + (size_t)(cs + c) * N] : czero<T>());
    }
    __syncthreads();
    T acc[2][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n) acc[m][n] = czero<T>();
    int k = 0;
#pragma unroll 2
    for (; k < ka; ++k) {
      const Op::L la = Ls[ia + k * 64], lb = Ls[ib + k * 64];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const Op::X x = Xs[k + (cq + 8 * n) * TS_LD];
        Op::fma(acc[0][n], la, x);
        Op::fma(acc[1][n], lb, x);
      }
    }
#pragma unroll 2
    for (; k < kb; ++k) {
      const Op::L lb = Ls[ib + k * 64];
#pragma unroll
      for (int n = 0; n < 4; ++n) Op::fma(acc[1][n], lb, Xs[k + (cq + 8 * n) * TS_LD]);
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int i = m ? ib : ia;
      if (i < jb)
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const int c = cq + 8 * n;
          if (c < nc) A[(size_t)(J + i) + (size_t)(cs + c) * N] = acc[m][n];
        }
    }
  }
}

// The FP64 step: the interchanges and the product in one pass over a tile.  The rows of A12
// are fetched from where the interchanges take them (cp.async, straight to shared memory), the
// rows that move below the panel go through registers, and U12 = L11^-1 A12 runs on the tensor
// cores: L11^-1 as 8 x 4 fragments of its lower triangle (36 KB), staged once per CTA; warp w
// owns the row blocks w & 3 and 7 - (w & 3), 18 fragments each pair, of two of the four column
// blocks.  A lane reads its entries of L and of A12 as 16-byte words without bank conflicts
// (column stride 68).  71 KB of shared memory: three CTAs per SM, one's loads behind the
// others' products.  Bound by the FP64 tensor cores and the rows' traffic alike; the earlier
// kernel swapped in place, read the tile back and multiplied with FMAs whose operands took
// more shared-memory cycles than they did.  17 steps of 250 points
// (500 matrices, N = 1080) 9.4 -> 3.6 ms, of 389 two-orbital points (N = 320) 1.47 -> 0.63 ms.
constexpr int SD_LD = 68, SD_FRAGS = 72;

__global__ void __launch_bounds__(256, 3)
k_swap_trsm_d(z64 *M, size_t strideM, int N, int ncols, int J, int jb, int NB, int nsteps,
              const int *rmap_all, const z64 *Linv) {
  extern __shared__ __align__(16) unsigned char smraw[];
  z64 *Lf = reinterpret_cast<z64 *>(smraw);      // fragment rb (rb + 1) + s: rows 8 rb.., columns 4 s..
  z64 *Xs = Lf + SD_FRAGS * 32;                  // [TW c][SD_LD k]
  __shared__ int s_src[64], s_od[64], s_os[64], s_n;
  const int b = blockIdx.y, t = threadIdx.x, w = t >> 5, lane = t & 31;
  z64 *A = M + (size_t)b * strideM;
  const z64 *L = Linv + ((size_t)b * nsteps + J / NB) * NB * NB;
  if (t < 64) s_src[t] = J + t;
  if (t == 0) s_n = 0;
  for (int s = 0; s < 2 * w + 2; ++s) {
    const int i = 8 * w + (lane >> 2), k = 4 * s + (lane & 3);
    Lf[(w * (w + 1) + s) * 32 + lane] = (i < jb && k <= i) ? L[i + k * NB] : czero<z64>();
  }
  __syncthreads();
  {
    // sources of the panel's rows; the rows below it (one per interchange at most)
    const int *rm = rmap_all + (size_t)b * RMAP_STRIDE;
    const int cnt = min(rm[0], 128);
    if (t < cnt) {
      const int dst = rm[1 + 2 * t], src = rm[2 + 2 * t];
      if (dst < J + jb) {
        s_src[dst - J] = src;
      } else {
        const int o = atomicAdd(&s_n, 1);
        if (o < 64) {
          s_od[o] = dst;
          s_os[o] = src;
        }
      }
    }
  }
  const int cb = 16 * (w >> 2);
  const int kk = t & 63, cc = t >> 6;
  for (int tile = 0; tile < TPC; ++tile) {
    const int cs = J + jb + (blockIdx.x * TPC + tile) * TW;
    if (cs >= ncols) break;
    const int nc = min(ncols, cs + TW) - cs;
    __syncthreads();               // L and the map staged; the previous tile's Xs reads are done
    const int nout = min(s_n, 64);
    z64 v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int c = cc + 4 * q;
      const bool in = kk < jb && c < nc;
      zg::cp_async16(&Xs[kk + c * SD_LD], in ? &A[(size_t)s_src[kk] + (size_t)(cs + c) * N] : A, in ? 16 : 0);
    }
    zg::cp_async_commit();
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int c = cc + 4 * q;
      if (kk < nout && c < nc) v[q] = A[(size_t)s_os[kk] + (size_t)(cs + c) * N];
    }
    zg::cp_async_wait<0>();
    __syncthreads();               // every row of the tile has been read
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int c = cc + 4 * q;
      if (kk < nout && c < nc) A[(size_t)s_od[kk] + (size_t)(cs + c) * N] = v[q];
    }
    if (cb >= nc) continue;
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      const int rb = h ? 7 - (w & 3) : w & 3, r0 = 8 * rb;
      if (r0 >= jb) continue;
      double re[2][2] = {}, im[2][2] = {};
      const z64 *lf = Lf + rb * (rb + 1) * 32 + lane;
      const z64 *xs = Xs + (cb + (lane >> 2)) * SD_LD + (lane & 3);
#pragma unroll 2
      for (int s = 0; s < 2 * rb + 2; ++s) {
        const z64 l = lf[s * 32];
        const double ln = -l.y;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const z64 x = xs[8 * n * SD_LD + 4 * s];
          zg::dmma(re[n], l.x, x.x);
          zg::dmma(im[n], l.x, x.y);
          zg::dmma(re[n], ln, x.y);
          zg::dmma(im[n], l.y, x.x);
        }
      }
      const int i = r0 + (lane >> 2);
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int c = cb + 8 * n + 2 * (lane & 3) + u;
          if (i < jb && c < nc)
            A[(size_t)(J + i) + (size_t)(cs + c) * N] = cx<z64>::make(re[n][u], im[n][u]);
        }
    }
  }
}

// ---------------------------------------------------------------------------
// Unpivoted step (the FP32 factorisation of the mixed path, a preconditioner
// of the FP64 refinement): the BSE matrices are close to the identity (growth
// factor 1.00 and condition numbers of 1..40 on the t2g workload), so the
// factorisation needs no row interchanges.  Per step:
//   k_diag_inv    LU of the jb x jb diagonal block in shared memory with its
//                 inverted L11 / U11 blocks (one CTA per matrix); identity
//                 pivots and an empty interchange map;
//   k_tri_tile    L21 = A21 U11^-1 and U12 = L11^-1 A12, every row / column
//                 independent (no pivot search over the column).
// A zero pivot gives non-finite factors; the refinement then fails to
// converge and the point is re-solved in FP64 with partial pivoting.
// ---------------------------------------------------------------------------
constexpr int DN_LD = 65;

// Diagonal block of an unpivoted step with its inverses, one CTA per matrix
// (FP32): the jb x jb block is padded with the identity to 64 x 64 and
// factored right-looking, four columns a step, its entries in registers and
// the panel of a step in shared memory (see the body).  L11^-1 (strictly
// lower; unit diagonal implied) and U11^-1 (upper with the diagonal) then
// share one array: eight warps invert the 16 x 16 diagonal blocks of both
// triangles (lane = column, no barriers), and two levels of recursive doubling
// join them,
//   [X00 0; X10 X11] with X10 = -X11 (L10 X00)   (and the transposed form for U),
// 16 x 16 blocks, then 32 x 32 blocks, the products L10 X00 formed in place of
// L10 (the factored block goes to the matrix before the inversion).  67 KB of
// shared memory and 72 registers: three CTAs per SM.
//
// Bound by latency: 16 steps, each a chain of four reciprocals and two
// barriers, and by what three CTAs read from shared memory.  An entry per
// thread and pass (rows bi + 16 r, columns bj + 16 c) lets every warp work to
// the end, where 4 x 4 blocks per thread left two lanes of each warp to solve
// the panel; the factor of the next diagonal block, in a warp of its own, runs
// beside the update (with it on the owner's path 62 instead of 56 us); scalar
// FMAs, the packed ones cost more in moving their operands (+2 us).
// 432 matrices (one wave) 85 -> 56 us, 2000 matrices 354 -> 237 us.
constexpr int DI_THREADS = 288;
constexpr int DI_SCR = 4 * 16;

__device__ __forceinline__ void cfma2(z32 &acc, z32 a, z32 u) {
  acc = __ffma2_rn(make_float2(a.x, a.x), u, acc);
  acc = __ffma2_rn(make_float2(-a.y, a.y), make_float2(u.y, u.x), acc);
}
// 1 / z for the FP32 block LU: z = (a + i b) / s with s the power of two that brings
// max(|a|, |b|) into [1, 2) (a result beyond the type's range apart, exact), and one correctly
// rounded reciprocal.  A zero pivot gives non-finite factors, which the refinement reports.
__device__ __forceinline__ z32 crcp_lu(z32 z) {
  const int e = __float_as_int(fmaxf(fabsf(z.x), fabsf(z.y))) & 0x7f800000;
  const float s = __int_as_float(max(0x7f000000 - e, 0x00800000));
  const float a = z.x * s, b = z.y * s;
  const float f = __frcp_rn(fmaf(a, a, b * b)) * s;
  return make_float2(a * f, -b * f);
}

template <typename T>
__global__ void __launch_bounds__(DI_THREADS, 3)
k_diag_inv(T *M, size_t strideM, int N, int J, int jb, int NB, int nsteps, T *Linv, T *Uinv, int *ipiv_all,
           int *rmap_all) {
  static_assert(sizeof(T) == sizeof(z32), "the blocked LU is the FP32 path's");
  extern __shared__ __align__(16) unsigned char smraw[];
  T *D = reinterpret_cast<T *>(smraw);          // [64][DN_LD] factored block
  T *X = D + 64 * DN_LD;                        // L11^-1 below the diagonal, U11^-1 on and above it
  T *S = X + 64 * DN_LD;                        // the LU's panel exchange
  __shared__ T rcps[64];
  const int b = blockIdx.x, t = threadIdx.x;
  T *A = M + (size_t)b * strideM;
  const T one = cx<T>::make(1, 0), zero = czero<T>();
  {
    // Right-looking LU, four columns a step.  Thread (bi, bj) of warps 0..7 owns rows bi + 16 r
    // and columns bj + 16 c.  The owners write the panel's rows and columns to D; two warps,
    // another pair each step, solve row i of L and column i of U, one pair per thread; then
    // every owner takes its share of A -= L U from the panel in D.  Warp 8 has factored the
    // panel's diagonal block by then: from copies that the owners write a step ahead (nd: the
    // next diagonal block before this step, followed by its rows and columns of the panel) it
    // brings that block up to date while the panel is solved and factors it beside the update,
    // so that the chain of four reciprocals, the longest of a step, is nobody else's.  Rows and
    // columns before the current group of 16 drop out at compile time; those inside it that
    // are already final are updated with the rest and not used again.
    auto bar = [] { asm volatile("bar.sync 0, %0;" ::"n"(DI_THREADS) : "memory"); };
    T *nd = S, *fd = S + 48;
    if (t >= 256) {
      const int lane = t & 31, r = lane & 3, c = (lane >> 2) & 3;
      T g[4][4], rp[4];
      bar();
      for (int kb = 0; kb < 16; ++kb) {
        // factor the block of step kb, every lane for itself; lane 0 writes it
#pragma unroll
        for (int c2 = 0; c2 < 4; ++c2)
#pragma unroll
          for (int r2 = 0; r2 < 4; ++r2) g[r2][c2] = fd[r2 + 4 * c2];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          rp[k] = crcp_lu(g[k][k]);
#pragma unroll
          for (int r2 = k + 1; r2 < 4; ++r2) g[r2][k] = cmul(g[r2][k], rp[k]);
#pragma unroll
          for (int r2 = k + 1; r2 < 4; ++r2)
#pragma unroll
            for (int c2 = k + 1; c2 < 4; ++c2) g[r2][c2] = csub(g[r2][c2], cmul(g[r2][k], g[k][c2]));
        }
        if (lane == 0) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            rcps[4 * kb + k] = rp[k];
#pragma unroll
            for (int r2 = 0; r2 < 4; ++r2) D[(4 * kb + r2) + (4 * kb + k) * DN_LD] = g[r2][k];
          }
        }
        bar();
        T l[4], u[4], v = nd[r + 4 * c];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          l[k] = nd[16 + r + 4 * k];
          u[k] = nd[32 + k + 4 * c];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
#pragma unroll
          for (int k2 = 0; k2 < k; ++k2) {
            l[k] = csub(l[k], cmul(l[k2], g[k2][k]));
            u[k] = csub(u[k], cmul(g[k][k2], u[k2]));
          }
          l[k] = cmul(l[k], rp[k]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) v = csub(v, cmul(l[k], u[k]));
        if (lane < 16) fd[r + 4 * c] = v;
        __syncwarp();
        bar();
      }
      bar();
      return;                // the barriers below wait for the threads that are left
    }
    const int bi = t & 15, bj = t >> 4;
    T a[4][4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = bi + 16 * r, j = bj + 16 * c;
        a[r][c] = (i < jb && j < jb) ? A[(size_t)(J + i) + (size_t)(J + j) * N] : (i == j ? one : zero);
      }
    if (bi < 4 && bj < 4) fd[bi + 4 * bj] = a[0][0];
    bar();
#pragma unroll
    for (int p = 0; p < 4; ++p) {
#pragma unroll 1
      for (int q = 0; q < 4; ++q) {
        const int k0 = 16 * p + 4 * q, qn = (q + 1) & 3;
        const int pn = (p + 1) & 3;                      // group of the next block when q = 3
        const bool rown = (bi >> 2) == qn, coln = (bj >> 2) == qn;
        if ((bj >> 2) == q) {
#pragma unroll
          for (int r = p; r < 4; ++r)
            if (r > p || bi >= 4 * q + 4) D[(bi + 16 * r) + (k0 + (bj & 3)) * DN_LD] = a[r][p];
          if (rown) nd[16 + (bi & 3) + 4 * (bj & 3)] = q < 3 ? a[p][p] : a[pn][p];
        }
        if ((bi >> 2) == q) {
#pragma unroll
          for (int c = p; c < 4; ++c)
            if (c > p || bj >= 4 * q + 4) D[(k0 + (bi & 3)) + (bj + 16 * c) * DN_LD] = a[p][c];
          if (coln) nd[32 + (bi & 3) + 4 * (bj & 3)] = q < 3 ? a[p][p] : a[p][pn];
        }
        if (rown && coln) nd[(bi & 3) + 4 * (bj & 3)] = q < 3 ? a[p][p] : a[pn][pn];
        bar();
        const int idx = t & 63, i = k0 + 4 + idx;
        if ((t >> 6) == q && i < 64) {
          T l[4], u[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            l[c] = D[i + (k0 + c) * DN_LD];
            u[c] = D[(k0 + c) + i * DN_LD];
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
#pragma unroll
            for (int c2 = 0; c2 < c; ++c2) {
              l[c] = csub(l[c], cmul(l[c2], D[(k0 + c2) + (k0 + c) * DN_LD]));
              u[c] = csub(u[c], cmul(D[(k0 + c) + (k0 + c2) * DN_LD], u[c2]));
            }
            l[c] = cmul(l[c], rcps[k0 + c]);
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            D[i + (k0 + c) * DN_LD] = l[c];
            D[(k0 + c) + i * DN_LD] = u[c];
          }
        }
        bar();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          T l[4], u[4];
#pragma unroll
          for (int r = p; r < 4; ++r) {
            l[r] = D[(bi + 16 * r) + (k0 + k) * DN_LD];
            u[r] = D[(k0 + k) + (bj + 16 * r) * DN_LD];
          }
#pragma unroll
          for (int c = p; c < 4; ++c)
#pragma unroll
            for (int r = p; r < 4; ++r) cfms(a[r][c], l[r], u[c]);
        }
      }
    }
    bar();
    // the packed factors (multipliers below the diagonal, U on and above it) to the matrix
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = bi + 16 * r, j = bj + 16 * c;
        if (i < jb && j < jb) A[(size_t)(J + i) + (size_t)(J + j) * N] = D[i + j * DN_LD];
      }
  }
  // entries of the two inverses: L^-1 with its unit diagonal and zeros above, U^-1 with zeros below
  auto xl = [&](int r, int c) { return r > c ? X[r + c * DN_LD] : (r == c ? one : zero); };
  auto xu = [&](int r, int c) { return r <= c ? X[r + c * DN_LD] : zero; };
  {
    // the 16 x 16 diagonal blocks of both inverses: warp w < 4 column l of L block w, warp w >= 4
    // column l of U block w - 4, by substitution
    const int w = t >> 5, lane = t & 31;
    if (lane < 16) {
      const int o = 16 * (w & 3), l = lane;
      T x[16];
      const T xd = w < 4 ? one : rcps[o + l];    // diagonal entry of the inverse's column l
#pragma unroll
      for (int r = 0; r < 16; ++r) x[r] = r == l ? xd : zero;
      if (w < 4) {                                // unit lower: column l of the block inverse, below l
#pragma unroll
        for (int r = 1; r < 16; ++r) {
          if (r > l) {
            T s = zero;
#pragma unroll
            for (int kk = 0; kk < r; ++kk)
              if (kk >= l) cfma(s, D[(o + r) + (o + kk) * DN_LD], x[kk]);
            x[r] = cneg(s);
          }
        }
#pragma unroll
        for (int r = 0; r < 16; ++r)
          if (r > l) X[(o + r) + (o + l) * DN_LD] = x[r];
      } else {                                    // upper: column l, on and above the diagonal
#pragma unroll
        for (int r = 14; r >= 0; --r) {
          if (r < l) {
            T s = zero;
#pragma unroll
            for (int kk = r + 1; kk < 16; ++kk)
              if (kk <= l) cfma(s, D[(o + r) + (o + kk) * DN_LD], x[kk]);
            x[r] = cneg(cmul(rcps[o + r], s));
          }
        }
#pragma unroll
        for (int r = 0; r < 16; ++r)
          if (r <= l) X[(o + r) + (o + l) * DN_LD] = x[r];
      }
    }
  }
  __syncthreads();
  {
    // 16 -> 32: for the 32-blocks at o = 0, 32 of both triangles
    //   L: X10 = -X11 (L10 X00),   U: Y01 = -Y00 (U01 Y11),
    // warp w: product (w >> 1): L at o = 0, 32, then U at o = 0, 32; columns 8 (w & 1).. + 7;
    // lane: row i = lane & 15, columns 4 (lane >> 4) + q
    const int w = t >> 5, lane = t & 31;
    const bool up = w >= 4;
    const int o = 32 * ((w >> 1) & 1), i = lane & 15, j0 = 8 * (w & 1) + 4 * (lane >> 4);
    T v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = zero;
    if (!up) {
#pragma unroll 4
      for (int k = 0; k < 16; ++k) {
        const T d = D[(o + 16 + i) + (o + k) * DN_LD];
#pragma unroll
        for (int q = 0; q < 4; ++q) cfma2(v[q], d, xl(o + k, o + j0 + q));
      }
    } else {
#pragma unroll 4
      for (int k = 0; k < 16; ++k) {
        const T d = D[(o + i) + (o + 16 + k) * DN_LD];
#pragma unroll
        for (int q = 0; q < 4; ++q) cfma2(v[q], d, xu(o + 16 + k, o + 16 + j0 + q));
      }
    }
    __syncthreads();     // every product has read its block of D: the products replace them
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (!up) D[(o + 16 + i) + (o + j0 + q) * DN_LD] = v[q];
      else D[(o + i) + (o + 16 + j0 + q) * DN_LD] = v[q];
      v[q] = zero;
    }
    __syncthreads();
    if (!up) {
#pragma unroll 4
      for (int k = 0; k < 16; ++k) {
        const T x = xl(o + 16 + i, o + 16 + k);
#pragma unroll
        for (int q = 0; q < 4; ++q) cfma2(v[q], x, D[(o + 16 + k) + (o + j0 + q) * DN_LD]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) X[(o + 16 + i) + (o + j0 + q) * DN_LD] = cneg(v[q]);
    } else {
#pragma unroll 4
      for (int k = 0; k < 16; ++k) {
        const T x = xu(o + i, o + k);
#pragma unroll
        for (int q = 0; q < 4; ++q) cfma2(v[q], x, D[(o + k) + (o + 16 + j0 + q) * DN_LD]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) X[(o + i) + (o + 16 + j0 + q) * DN_LD] = cneg(v[q]);
    }
  }
  __syncthreads();
  {
    // 32 -> 64: L: X10 = -X11 (L10 X00), U: Y01 = -Y00 (U01 Y11) with 32 x 32 blocks;
    // warps 0..3 the L product, 4..7 the U product; lane: rows i, i + 16, columns j0 + q.  The
    // products with a triangle skip its zero quarter (and, by groups of 8 columns, its zeros)
    const int w = t >> 5, lane = t & 31, w4 = w & 3;
    const bool up = w >= 4;
    const int i = lane & 15, j0 = 8 * w4 + 4 * (lane >> 4);
    T v[2][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[0][q] = v[1][q] = zero;
    if (!up) {             // L10 X00: X00(k, j) = 0 for k < j
#pragma unroll 4
      for (int k = 8 * w4; k < 32; ++k) {
        const T d0 = D[(32 + i) + k * DN_LD], d1 = D[(48 + i) + k * DN_LD];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const T x = xl(k, j0 + q);
          cfma2(v[0][q], d0, x);
          cfma2(v[1][q], d1, x);
        }
      }
    } else {               // U01 Y11: Y11(k, j) = 0 for k > j
#pragma unroll 4
      for (int k = 0; k < 8 * w4 + 8; ++k) {
        const T d0 = D[i + (32 + k) * DN_LD], d1 = D[(16 + i) + (32 + k) * DN_LD];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const T x = xu(32 + k, 32 + j0 + q);
          cfma2(v[0][q], d0, x);
          cfma2(v[1][q], d1, x);
        }
      }
    }
    __syncthreads();
    const int ro = up ? 0 : 32, co = up ? 32 : 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        D[(ro + 16 * h + i) + (co + j0 + q) * DN_LD] = v[h][q];
        v[h][q] = zero;
      }
    __syncthreads();
    if (!up) {             // X11(i, k) = 0 for k > i
#pragma unroll 4
      for (int k = 0; k < 16; ++k) {
        const T x0 = xl(32 + i, 32 + k), x1 = X[(48 + i) + (32 + k) * DN_LD];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const T d = D[(32 + k) + (j0 + q) * DN_LD];
          cfma2(v[0][q], x0, d);
          cfma2(v[1][q], x1, d);
        }
      }
#pragma unroll 4
      for (int k = 16; k < 32; ++k) {
        const T x1 = xl(48 + i, 32 + k);
#pragma unroll
        for (int q = 0; q < 4; ++q) cfma2(v[1][q], x1, D[(32 + k) + (j0 + q) * DN_LD]);
      }
    } else {               // Y00(i, k) = 0 for k < i
#pragma unroll 4
      for (int k = 0; k < 16; ++k) {
        const T x0 = xu(i, k);
#pragma unroll
        for (int q = 0; q < 4; ++q) cfma2(v[0][q], x0, D[k + (32 + j0 + q) * DN_LD]);
      }
#pragma unroll 4
      for (int k = 16; k < 32; ++k) {
        const T x0 = X[i + k * DN_LD], x1 = xu(16 + i, k);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const T d = D[k + (32 + j0 + q) * DN_LD];
          cfma2(v[0][q], x0, d);
          cfma2(v[1][q], x1, d);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int h = 0; h < 2; ++h) X[(ro + 16 * h + i) + (co + j0 + q) * DN_LD] = cneg(v[h][q]);
  }
  __syncthreads();
  const size_t off = ((size_t)b * nsteps + J / NB) * NB * NB;
#pragma unroll 4
  for (int e = t; e < NB * NB; e += 256) {
    const int i = e % NB, k = e / NB;
    T lv = zero, uv = zero;
    if (i < jb && k < jb) {
      lv = xl(i, k);
      uv = xu(i, k);
    }
    Linv[off + e] = lv;
    Uinv[off + e] = uv;
  }
  int *ip = ipiv_all + (size_t)b * N + J;
  for (int i = t; i < jb; i += 256) ip[i] = J + i;
  if (t == 0) rmap_all[(size_t)b * RMAP_STRIDE] = 0;
}

// Off-diagonal tiles of an unpivoted step, 64 x 64 per CTA:
//   LEFT  U12 = L11^-1 A12  (rows J.., columns J+jb+64 x)
//   !LEFT L21 = A21 U11^-1  (rows J+jb+64 x.., columns J..)
// The tile and the triangle are staged in shared memory (column stride 65,
// conflict-free).  Along the triangle's free index (rows of U12, columns of
// L21) a thread owns 4 consecutive entries and the other index strides by
// 16; that index's owner, (t / 16), is nearly warp-uniform, so each warp
// stops at its own edge of the triangle and the product does the triangular
// half of the work.  U12 is written back through shared memory (coalesced).
// one element global -> shared by cp.async (8 or 16 bytes); zeros when !valid
template <typename T>
__device__ __forceinline__ void cp_async_elem(T *dst, const T *src, bool valid) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(valid ? 8 : 0));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0));
}

template <typename T, bool LEFT>
__global__ void __launch_bounds__(256)
k_tri_tile(T *M, size_t strideM, int N, int ncols, int J, int jb, int NB, int nsteps, const T *Tri) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T *Ts = reinterpret_cast<T *>(smraw);        // triangle, [k or row][DN_LD]
  T *Xs = Ts + 64 * DN_LD;                      // tile
  const int b = blockIdx.y, t = threadIdx.x;
  T *A = M + (size_t)b * strideM;
  const T *Q = Tri + ((size_t)b * nsteps + J / NB) * NB * NB;
  const int r0 = LEFT ? J : J + jb + blockIdx.x * 64;
  const int c0 = LEFT ? J + jb + blockIdx.x * 64 : J;
  const int nr = LEFT ? jb : min(64, N - r0);
  const int nc = LEFT ? min(64, ncols - c0) : jb;
  // asynchronous staging (zero-filled outside the triangle / tile): every load in flight at once
  for (int e = t; e < 64 * 64; e += 256) {
    const int i = e & 63, j = e >> 6;           // i fastest: coalesced loads, conflict-free stores
    const bool inq = i < jb && j < jb, inx = i < nr && j < nc;
    cp_async_elem<T>(Ts + i + j * DN_LD, inq ? Q + i + (size_t)j * NB : Q, inq);
    cp_async_elem<T>(Xs + i + j * DN_LD, inx ? A + (size_t)(r0 + i) + (size_t)(c0 + j) * N : A, inx);
  }
  asm volatile("cp.async.commit_group;");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const int w4 = 4 * (t >> 4), s16 = t & 15;    // 4 consecutive triangle-side entries, the rest by 16
  T acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = czero<T>();
  // LEFT: out(w4 + i, s16 + 16 j) = sum_{k <= row} L^-1(row, k) X(k, col)
  // !LEFT: out(s16 + 16 i, w4 + j) = sum_{k <= col} X(row, k) U^-1(k, col)
  const int kend = min(jb, w4 + 4);
#pragma unroll 2
  for (int k = 0; k < kend; ++k) {
    T a[4], u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = LEFT ? Ts[(w4 + i) + k * DN_LD] : Xs[(s16 + 16 * i) + k * DN_LD];
#pragma unroll
    for (int j = 0; j < 4; ++j) u[j] = LEFT ? Xs[k + (s16 + 16 * j) * DN_LD] : Ts[k + (w4 + j) * DN_LD];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) cfma2(acc[i][j], a[i], u[j]);
  }
  if (LEFT) {
    __syncthreads();                            // every Xs read is done
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) Xs[(w4 + i) + (s16 + 16 * j) * DN_LD] = acc[i][j];
    __syncthreads();
    for (int e = t; e < 64 * 64; e += 256) {
      const int i = e & 63, j = e >> 6;
      if (i < nr && j < nc) A[(size_t)(r0 + i) + (size_t)(c0 + j) * N] = Xs[i + j * DN_LD];
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = w4 + j;
      if (c >= nc) continue;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = s16 + 16 * i;
        if (r < nr) A[(size_t)(r0 + r) + (size_t)(c0 + c) * N] = acc[i][j];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Trailing update on CUDA cores: C[J+jb.., J+jb..] -= A[J+jb.., J:J+jb] * A[J:J+jb, J+jb..]
// 64 x 64 tiles, BK = 16, 256 threads with 4 x 4 complex outputs each.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
k_gemm_update(T *M, size_t strideM, int N, int ncols, int J, int jb) {
  __shared__ T As[16][64];
  __shared__ T Bs[16][64];
  const int b = blockIdx.z, t = threadIdx.x;
  const int tx = t & 15, ty = t >> 4;
  T *A = M + (size_t)b * strideM;
  const int r0 = J + jb + blockIdx.y * 64, c0 = J + jb + blockIdx.x * 64;
  T acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = czero<T>();
  for (int k0 = 0; k0 < jb; k0 += 16) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int e = t + 256 * i;
      int rr = e & 63, kk = e >> 6;
      int r = r0 + rr, k = k0 + kk;
      As[kk][rr] = (r < N && k < jb) ? A[r + (size_t)(J + k) * N] : czero<T>();
      int kk2 = e & 15, cc = e >> 4;
      int c = c0 + cc, k2 = k0 + kk2;
      Bs[kk2][cc] = (c < ncols && k2 < jb) ? A[(size_t)(J + k2) + (size_t)c * N] : czero<T>();
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      T av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = As[kk][tx + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = Bs[kk][ty + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) cfma(acc[i][j], av[i], bv[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = c0 + ty + 16 * j;
    if (c >= ncols) continue;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + tx + 16 * i;
      if (r < N) {
        T *p = A + r + (size_t)c * N;
        *p = csub(*p, acc[i][j]);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Blocked triangular solves with the inverted diagonal blocks.
// backsolve: U Y = C (bottom block first); fwdsolve: L z = P r (top first).
// ---------------------------------------------------------------------------
#define RT 16
template <typename T, bool UPPER>
__global__ void __launch_bounds__(256)
k_trisolve(const T *M, size_t strideM, int N, int NB, int nsteps, const T *Dinv, T *C,
           size_t strideC, int ldc, int R, const int *ipiv_all, T *work) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int nph = 256 / NB;
  T *red = reinterpret_cast<T *>(smraw);          // [nph][NB][RT]
  T *W = red + (size_t)nph * NB * RT;             // [NB][RT]
  int *perm = reinterpret_cast<int *>(W + (size_t)NB * RT);
  const int b = blockIdx.y, r0 = blockIdx.x * RT, t = threadIdx.x;
  const T *A = M + (size_t)b * strideM;
  T *Cb = C + (size_t)b * strideC;
  const int nr = min(RT, R - r0);
  if (!UPPER) {
    // apply the row interchanges P to the right-hand sides (through work)
    if (t == 0) {
      for (int i = 0; i < N; ++i) perm[i] = i;
      const int *ip = ipiv_all + (size_t)b * N;
      for (int i = 0; i < N; ++i) {
        int p = ip[i];
        if (p != i) { int x = perm[i]; perm[i] = perm[p]; perm[p] = x; }
      }
    }
    __syncthreads();
    T *Wk = work + (size_t)b * N * RT * gridDim.x + (size_t)blockIdx.x * N * RT;
    for (int e = t; e < N * nr; e += 256) {
      int i = e % N, r = e / N;
      Wk[e] = Cb[perm[i] + (size_t)(r0 + r) * ldc];
    }
    __syncthreads();
    for (int e = t; e < N * nr; e += 256) {
      int i = e % N, r = e / N;
      Cb[i + (size_t)(r0 + r) * ldc] = Wk[e];
    }
    __syncthreads();
  }
  const int row = t % NB, kph = t / NB;
  for (int s = 0; s < nsteps; ++s) {
    const int blk = UPPER ? nsteps - 1 - s : s;
    const int J = blk * NB, jb = min(NB, N - J);
    T acc[RT];
#pragma unroll
    for (int r = 0; r < RT; ++r) acc[r] = czero<T>();
    if (row < jb) {
      const int kb = UPPER ? J + jb : 0, ke = UPPER ? N : J;
      for (int k = kb + kph; k < ke; k += nph) {
        const T u = A[(size_t)(J + row) + (size_t)k * N];
#pragma unroll
        for (int r = 0; r < RT; ++r)
          if (r < nr) cfma(acc[r], u, Cb[k + (size_t)(r0 + r) * ldc]);
      }
    }
#pragma unroll
    for (int r = 0; r < RT; ++r) red[((size_t)kph * NB + row) * RT + r] = acc[r];
    __syncthreads();
    for (int e = t; e < jb * nr; e += 256) {
      int i = e % jb, r = e / jb;
      T v = Cb[(size_t)(J + i) + (size_t)(r0 + r) * ldc];
      for (int ph = 0; ph < nph; ++ph) v = csub(v, red[((size_t)ph * NB + i) * RT + r]);
      W[i * RT + r] = v;
    }
    __syncthreads();
    const T *Di = Dinv + ((size_t)b * nsteps + blk) * NB * NB;
    for (int e = t; e < jb * nr; e += 256) {
      int i = e % jb, r = e / jb;
      T v = czero<T>();
      const int kb = UPPER ? i : 0, ke = UPPER ? jb : i + 1;
      for (int k = kb; k < ke; ++k) cfma(v, Di[i + k * NB], W[k * RT + r]);
      Cb[(size_t)(J + i) + (size_t)(r0 + r) * ldc] = v;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Blocked triangular solve with the right-hand sides resident in shared
// memory (R <= RMAX columns, N*R elements): one CTA per matrix, right-looking
// over the NB-row blocks.  Per block: X_blk = Dinv * C_blk, then the rows not
// yet solved are updated with the matching column block of U (backward) or L
// (forward), one thread per row, so every element of the triangle is read
// from HBM exactly once with coalesced column accesses.  The forward solve
// applies the row interchanges P while loading the right-hand sides.
// ---------------------------------------------------------------------------
template <typename T, bool UPPER, int RMAX, int RPT>
__global__ void __launch_bounds__(512)
k_trisolve_smem(const T *M, size_t strideM, int N, int NB, int nsteps, const T *Dinv, T *C,
                size_t strideC, int ldc, int R, const int *ipiv_all, size_t stage_d) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T *Cs = reinterpret_cast<T *>(smraw);            // [R][N]
  T *Yt = Cs + (size_t)N * R;                        // [R][NB]
  int *perm = reinterpret_cast<int *>(Yt + (size_t)NB * R);
  // the diagonal-block inverse of the current step, staged when it fits
  T *Ds = stage_d ? reinterpret_cast<T *>(smraw + stage_d) : nullptr;
  const int b = blockIdx.x, t = threadIdx.x, nt = blockDim.x;
  const T *A = M + (size_t)b * strideM;
  T *Cb = C + (size_t)b * strideC;
  if (!UPPER) {
    if (t == 0) {
      for (int i = 0; i < N; ++i) perm[i] = i;
      const int *ip = ipiv_all + (size_t)b * N;
      for (int i = 0; i < N; ++i) {
        const int p = ip[i];
        if (p != i) { int x = perm[i]; perm[i] = perm[p]; perm[p] = x; }
      }
    }
    __syncthreads();
  }
  for (int e = t; e < N * R; e += nt) {
    const int i = e % N, r = e / N;
    Cs[e] = Cb[(size_t)(UPPER ? i : perm[i]) + (size_t)r * ldc];
  }
  __syncthreads();
  for (int s = 0; s < nsteps; ++s) {
    const int blk = UPPER ? nsteps - 1 - s : s;
    const int J = blk * NB, jb = min(NB, N - J);
    const T *Di = Dinv + ((size_t)b * nsteps + blk) * NB * NB;
    if (Ds) {
      for (int e = t; e < NB * jb; e += nt) Ds[e] = Di[e];
      __syncthreads();
    }
    const T *D = Ds ? Ds : Di;
    for (int e = t; e < jb * R; e += nt) {
      const int i = e % jb, r = e / jb;
      const int kb = UPPER ? i : 0, ke = UPPER ? jb : i + 1;
      T v0 = czero<T>(), v1 = czero<T>(), v2 = czero<T>(), v3 = czero<T>();
      int k = kb;
      for (; k + 3 < ke; k += 4) {
        cfma(v0, D[i + k * NB], Cs[(size_t)r * N + J + k]);
        cfma(v1, D[i + (k + 1) * NB], Cs[(size_t)r * N + J + k + 1]);
        cfma(v2, D[i + (k + 2) * NB], Cs[(size_t)r * N + J + k + 2]);
        cfma(v3, D[i + (k + 3) * NB], Cs[(size_t)r * N + J + k + 3]);
      }
      for (; k < ke; ++k) cfma(v0, D[i + k * NB], Cs[(size_t)r * N + J + k]);
      Yt[(size_t)r * NB + i] = cadd(cadd(v0, v1), cadd(v2, v3));
    }
    __syncthreads();
    for (int e = t; e < jb * R; e += nt) {
      const int i = e % jb, r = e / jb;
      Cs[(size_t)r * N + J + i] = Yt[(size_t)r * NB + i];
    }
    // rows still to solve: each thread owns RPT of them, so every Yt value
    // read from shared memory feeds RPT rows
    const int rb = UPPER ? 0 : J + jb, re = UPPER ? J : N;
    for (int base = rb + t; base < re; base += nt * RPT) {
      T acc[RPT][RMAX];
#pragma unroll
      for (int q = 0; q < RPT; ++q)
#pragma unroll
        for (int r = 0; r < RMAX; ++r) acc[q][r] = czero<T>();
#pragma unroll 8
      for (int k = 0; k < jb; ++k) {
        T y[RMAX];
#pragma unroll
        for (int r = 0; r < RMAX; ++r) y[r] = r < R ? Yt[(size_t)r * NB + k] : czero<T>();
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          const int i = base + q * nt;
          const T u = i < re ? A[(size_t)i + (size_t)(J + k) * N] : czero<T>();
#pragma unroll
          for (int r = 0; r < RMAX; ++r)
            if (r < R) cfma(acc[q][r], u, y[r]);
        }
      }
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        const int i = base + q * nt;
        if (i < re)
#pragma unroll
          for (int r = 0; r < RMAX; ++r)
            if (r < R) Cs[(size_t)r * N + i] = csub(Cs[(size_t)r * N + i], acc[q][r]);
      }
    }
    __syncthreads();
  }
  for (int e = t; e < N * R; e += nt) {
    const int i = e % N, r = e / N;
    Cb[(size_t)i + (size_t)r * ldc] = Cs[e];
  }
}

// ---------------------------------------------------------------------------
// host drivers
// ---------------------------------------------------------------------------
template <typename T, int RPT, int SW, int NTMAX>
static cudaError_t launch_panel_as(T *M, const LUBatch &lb, int J, int jb, cudaStream_t st) {
  const int rows = lb.N - J;
  const int nt = std::max(128, ((rows + RPT - 1) / RPT + 31) / 32 * 32);
  const size_t dyn = sizeof(T) * ((size_t)64 * 2 * SW + (panel_mma<T, RPT>() ? (size_t)SW * panel_lr(rows) : 0));
  smem_limit(k_panel<T, RPT, SW, NTMAX>, 200 * 1024);
  k_panel<T, RPT, SW, NTMAX><<<lb.batch, nt, dyn, st>>>(M, lb.strideM, lb.N, J, jb, lb.ipiv, lb.info);
  return ADGA_LAUNCH_CHECK();
}

template <typename T>
static cudaError_t launch_panel(T *M, const LUBatch &lb, int J, int jb, cudaStream_t st) {
  const int rows = lb.N - J;
  // rows x SW complex values fill the register file at 512 x 16, 1152 x 8, 2048 x 4 and 4096 x 2; wider
  // sub-panels halve the passes over the rest of the panel, spilled ones cost more than they save
  // (one 64-column panel, us, as listed against another form: 1016 rows 250 / 275 at three rows a thread,
  // 1080 rows 276 / 337 at <2, 4>, 1500 rows 415 / 606 and 2000 rows 539 / 795 with the update on the
  // tensor cores, 4000 rows 2700 / 3839 at <8, 4>)
  if (rows <= 512) return launch_panel_as<T, 1, 16, 512>(M, lb, J, jb, st);
  if (rows <= 1024) return launch_panel_as<T, 2, 8, 512>(M, lb, J, jb, st);
  if (rows <= 1152) return launch_panel_as<T, 3, 8, 384>(M, lb, J, jb, st);
  if (rows <= 1536) return launch_panel_as<T, 2, 4, 768>(M, lb, J, jb, st);
  if (rows <= 2048) return launch_panel_as<T, 4, 4, 512>(M, lb, J, jb, st);
  if (rows <= 4096) return launch_panel_as<T, 8, 2, 512>(M, lb, J, jb, st);
  return cudaErrorInvalidValue;   // N > 4096 is not supported
}

cudaError_t lu_trail_z64(z64 *M, const LUBatch &lb, int J, int jb, cudaStream_t st);

template <typename T>
cudaError_t lu_trail_cuda(T *M, const LUBatch &lb, int J, int jb, cudaStream_t st) {
  if constexpr (sizeof(T) == sizeof(z64)) return lu_trail_z64((z64 *)M, lb, J, jb, st);
  const int m = lb.N - J - jb, n = lb.ncols - J - jb;
  if (m <= 0 || n <= 0) return cudaSuccess;
  dim3 grid(cdiv_u(n, 64), cdiv_u(m, 64), lb.batch);
  k_gemm_update<T><<<grid, 256, 0, st>>>(M, lb.strideM, lb.N, lb.ncols, J, jb);
  return ADGA_LAUNCH_CHECK();
}

// trailing update of step (J, jb) through `trail` (or the plain GEMM), timed into tt
template <typename T>
static cudaError_t lu_trail_step(T *M, const LUBatch &lb, int J, int jb, trail_fn trail, void *trail_ctx,
                                 cudaStream_t st, TrailTiming *tt) {
  cudaError_t e;
  if (J + jb < lb.N) {
    cudaEvent_t ev0 = (tt && tt->ev) ? tt->ev[2 * tt->n] : nullptr;
    cudaEvent_t ev1 = (tt && tt->ev) ? tt->ev[2 * tt->n + 1] : nullptr;
    if (trail) {
      e = trail(trail_ctx, J, jb, st, ev0, ev1);
    } else {
      if (ev0) cudaEventRecord(ev0, st);
      e = lu_trail_cuda<T>(M, lb, J, jb, st);
      if (ev1) cudaEventRecord(ev1, st);
    }
    if (e != cudaSuccess) return e;
    if (tt && tt->ev) {
      const double m = lb.N - J - jb, n = lb.ncols - J - jb;
      tt->gflop += 8.0 * m * n * jb * lb.batch * 1e-9;
      tt->gbytes += (2.0 * sizeof(T) * m * n + sizeof(T) * (double)jb * (m + n)) * lb.batch * 1e-9;
      tt->n++;
    }
  }
  return cudaSuccess;
}

// kernels of one unpivoted FP32 step: block LU + inverses, L21, U12 (k_diag_inv, k_tri_tile;
// tiles = false: the block LU only)
static cudaError_t nopiv_step_kernels(z32 *M, const LUBatch &lb, int J, int jb, cudaStream_t st,
                                      bool tiles = true) {
  typedef z32 T;
  const int nsteps = lb.nsteps();
  cudaError_t e;
  const size_t sm_di = sizeof(T) * (2 * 64 * DN_LD + DI_SCR), sm_tt = sizeof(T) * 2 * 64 * DN_LD;
  smem_limit(k_diag_inv<T>, (int)sm_di);
  smem_limit(k_tri_tile<T, true>, (int)sm_tt);
  smem_limit(k_tri_tile<T, false>, (int)sm_tt);
  k_diag_inv<T><<<lb.batch, DI_THREADS, sm_di, st>>>(M, lb.strideM, lb.N, J, jb, lb.NB, nsteps, (T *)lb.Linv,
                                              (T *)lb.Uinv, lb.ipiv, lb.rmap);
  if ((e = ADGA_LAUNCH_CHECK()) != cudaSuccess) return e;
  if (!tiles) return cudaSuccess;
  if (J + jb < lb.N) {
    k_tri_tile<T, false><<<dim3(cdiv_u(lb.N - J - jb, 64), lb.batch), 256, sm_tt, st>>>(
        M, lb.strideM, lb.N, lb.ncols, J, jb, lb.NB, nsteps, (const T *)lb.Uinv);
    if ((e = ADGA_LAUNCH_CHECK()) != cudaSuccess) return e;
  }
  if (lb.ncols > J + jb) {
    k_tri_tile<T, true><<<dim3(cdiv_u(lb.ncols - J - jb, 64), lb.batch), 256, sm_tt, st>>>(
        M, lb.strideM, lb.N, lb.ncols, J, jb, lb.NB, nsteps, (const T *)lb.Linv);
    if ((e = ADGA_LAUNCH_CHECK()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

static void trail_account(TrailTiming *tt, double m, double n, double k, int batch) {
  if (!tt || !tt->ev || m <= 0 || n <= 0) return;
  tt->gflop += 8.0 * m * n * k * batch * 1e-9;
  tt->gbytes += (2.0 * sizeof(z32) * m * n + sizeof(z32) * k * (m + n)) * batch * 1e-9;
}

// Unpivoted FP32 factorisation with delayed updates in groups of G = 2..4 steps: after
// step g < G - 1 of a group only the parts of the group's updates that step g + 1 reads
// (narrow), after its last step all G steps' updates of the rest at once (wide)
cudaError_t lu_factor_groups(z32 *M, const LUBatch &lb, const GroupOps &ops, cudaStream_t st, TrailTiming *tt) {
  if (ops.G < 2 || ops.G > 4) return cudaErrorInvalidValue;
  const int nsteps = lb.nsteps();
  int Js[4], jbs[4];
  for (int s = 0; s < nsteps; ++s) {
    const int J = s * lb.NB, jb = min(lb.NB, lb.N - J), g = s % ops.G;
    Js[g] = J;
    jbs[g] = jb;
    cudaError_t e = nopiv_step_kernels(M, lb, J, jb, st, ops.tri == nullptr);
    if (e == cudaSuccess && ops.tri) e = ops.tri(ops.ctx, J, jb, g, st);
    if (e != cudaSuccess) return e;
    if (J + jb >= lb.N) break;
    cudaEvent_t ev0 = (tt && tt->ev) ? tt->ev[2 * tt->n] : nullptr;
    cudaEvent_t ev1 = (tt && tt->ev) ? tt->ev[2 * tt->n + 1] : nullptr;
    const bool wide = g == ops.G - 1;
    e = ops.update(ops.ctx, g + 1, Js, jbs, wide, st, ev0, ev1);
    int K = 0;
    for (int i = 0; i <= g; ++i) K += jbs[i];
    const int R = J + jb;
    if (wide) {
      trail_account(tt, lb.N - R, lb.ncols - R, K, lb.batch);
    } else {
      const int jt = min(lb.NB, lb.N - R);
      trail_account(tt, lb.N - R, jt, K, lb.batch);
      trail_account(tt, jt, lb.ncols - R - jt, K, lb.batch);
    }
    if (e != cudaSuccess) return e;
    if (tt && tt->ev) tt->n++;
  }
  return cudaSuccess;
}

template <typename T>
cudaError_t lu_step(T *M, const LUBatch &lb, int s, bool apply_left, trail_fn trail, void *trail_ctx,
                    cudaStream_t st, TrailTiming *tt, bool nopiv) {
  if (lb.NB > 64 || lb.NB % 8) return cudaErrorInvalidValue;   // the step kernels cover NB <= 64
  const int nsteps = lb.nsteps();
  cudaError_t e;
  const size_t sm_tri = sizeof(T) * 64 * TI_LD;
  smem_limit(k_triinv<T>, 200 * 1024);
  const int J = s * lb.NB, jb = min(lb.NB, lb.N - J);
  if constexpr (sizeof(T) == sizeof(z32)) {
    if (nopiv) {
      if ((e = nopiv_step_kernels(M, lb, J, jb, st)) != cudaSuccess) return e;
      return lu_trail_step<T>(M, lb, J, jb, trail, trail_ctx, st, tt);
    }
  }
  if (nopiv) return cudaErrorInvalidValue;     // the unpivoted step is the FP32 factorisation only
  if ((e = launch_panel<T>(M, lb, J, jb, st)) != cudaSuccess) return e;
  k_triinv<T><<<lb.batch, 256, sm_tri, st>>>(M, lb.strideM, lb.N, J, jb, lb.NB, nsteps,
                                             (T *)lb.Linv, (T *)lb.Uinv, lb.ipiv, lb.rmap);
  if ((e = ADGA_LAUNCH_CHECK()) != cudaSuccess) return e;
  const int nleft = apply_left ? (J + TW - 1) / TW : 0;
  const int nright = (lb.ncols - J - jb + TW - 1) / TW;
  if (nleft > 0) {
    k_swap_left<T><<<dim3(nleft, lb.batch), 256, 0, st>>>(M, lb.strideM, lb.N, J, lb.rmap);
    if ((e = ADGA_LAUNCH_CHECK()) != cudaSuccess) return e;
  }
  if (nright > 0) {
    const dim3 grid((nright + TPC - 1) / TPC, lb.batch);
    if constexpr (sizeof(T) == sizeof(z64)) {
      const size_t sm = sizeof(z64) * (SD_FRAGS * 32 + TW * SD_LD);
      smem_limit(k_swap_trsm_d, (int)sm);
      k_swap_trsm_d<<<grid, 256, sm, st>>>(M, lb.strideM, lb.N, lb.ncols, J, jb, lb.NB, nsteps, lb.rmap,
                                           (const z64 *)lb.Linv);
    } else {
      const size_t sm = sizeof(TrsmOp::L) * 64 * 64 + sizeof(TrsmOp::X) * TW * TS_LD;
      smem_limit(k_swap_trsm, (int)sm);
      k_swap_trsm<<<grid, 256, sm, st>>>(M, lb.strideM, lb.N, lb.ncols, J, jb, lb.NB, nsteps, lb.rmap,
                                         (const z32 *)lb.Linv);
    }
    if ((e = ADGA_LAUNCH_CHECK()) != cudaSuccess) return e;
  }
  return lu_trail_step<T>(M, lb, J, jb, trail, trail_ctx, st, tt);
}

template <typename T>
cudaError_t lu_factor(T *M, const LUBatch &lb, bool apply_left, trail_fn trail, void *trail_ctx,
                      cudaStream_t st, TrailTiming *tt, bool nopiv) {
  for (int s = 0; s < lb.nsteps(); ++s) {
    cudaError_t e = lu_step<T>(M, lb, s, apply_left, trail, trail_ctx, st, tt, nopiv);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <typename T>
static cudaError_t trisolve(const T *M, const LUBatch &lb, T *C, size_t strideC, int ldc, int R,
                            bool upper, T *work, cudaStream_t st) {
  // FP32 factors, up to 16 right-hand sides: the tensor-core solve (k_trsv_tc.cu)
  if constexpr (sizeof(T) == sizeof(z32))
    if (trsv_tc_supported(lb, R, upper))
      return launch_trsv_tc(reinterpret_cast<const z32 *>(M), lb, reinterpret_cast<z32 *>(C), strideC, ldc, R,
                            upper, st);
  // few right-hand sides and NB = 64: the streaming solve (k_trsv.cu)
  if (trsv_stream_supported<T>(lb, strideC, R, upper, lb.perm, work))
    return launch_trsv_stream<T>(M, lb, C, strideC, ldc, R, upper, lb.perm, work, st);
  // few right-hand sides that fit in shared memory: the resident-RHS kernel
  size_t sm_small = sizeof(T) * ((size_t)lb.N * R + (size_t)lb.NB * R) + sizeof(int) * lb.N;
  size_t stage_d = 0;
  const size_t dbytes = sizeof(T) * (size_t)lb.NB * lb.NB;
  if (sm_small + 16 + dbytes <= 112 * 1024) {       // keep two CTAs per SM
    stage_d = (sm_small + 15) / 16 * 16;
    sm_small = stage_d + dbytes;
  }
  if (R <= 25 && sm_small <= 200 * 1024) {
    const int np = lb.nsteps();
#define TS_LAUNCH(UP, RM)                                                                            \
    do {                                                                                             \
      smem_limit(k_trisolve_smem<T, UP, RM, 1>, 200 * 1024);                                         \
      k_trisolve_smem<T, UP, RM, 1><<<lb.batch, 512, sm_small, st>>>(                                \
          M, lb.strideM, lb.N, lb.NB, np, (const T *)(UP ? lb.Uinv : lb.Linv), C, strideC, ldc, R,   \
          lb.ipiv, stage_d);                                                                         \
    } while (0)
    if (upper) {
      if (R == 9) TS_LAUNCH(true, 9); else if (R <= 4) TS_LAUNCH(true, 4);
      else if (R <= 16) TS_LAUNCH(true, 16); else TS_LAUNCH(true, 25);
    } else {
      if (R == 9) TS_LAUNCH(false, 9); else if (R <= 4) TS_LAUNCH(false, 4);
      else if (R <= 16) TS_LAUNCH(false, 16); else TS_LAUNCH(false, 25);
    }
#undef TS_LAUNCH
    return ADGA_LAUNCH_CHECK();
  }
  const int nph = 256 / lb.NB;
  size_t sm = sizeof(T) * ((size_t)nph * lb.NB * RT + (size_t)lb.NB * RT) + sizeof(int) * lb.N;
  if (upper)
    smem_limit(k_trisolve<T, true>, 200 * 1024);
  else
    smem_limit(k_trisolve<T, false>, 200 * 1024);
  if (!upper && !work) return cudaErrorInvalidValue;
  dim3 g(cdiv_u(R, RT), lb.batch);
  if (upper)
    k_trisolve<T, true><<<g, 256, sm, st>>>(M, lb.strideM, lb.N, lb.NB, lb.nsteps(), (const T *)lb.Uinv,
                                            C, strideC, ldc, R, lb.ipiv, work);
  else
    k_trisolve<T, false><<<g, 256, sm, st>>>(M, lb.strideM, lb.N, lb.NB, lb.nsteps(), (const T *)lb.Linv,
                                             C, strideC, ldc, R, lb.ipiv, work);
  return ADGA_LAUNCH_CHECK();
}

template <typename T>
cudaError_t lu_backsolve(const T *M, const LUBatch &lb, T *C, size_t strideC, int ldc, int R,
                         cudaStream_t st) {
  return trisolve<T>(M, lb, C, strideC, ldc, R, true, nullptr, st);
}

// work: batch * ceil(R/16) * N * 16 elements
template <typename T>
cudaError_t lu_fwdsolve_ws(const T *M, const LUBatch &lb, T *V, size_t strideV, int ldv, int R,
                           T *work, cudaStream_t st) {
  return trisolve<T>(M, lb, V, strideV, ldv, R, false, work, st);
}

template cudaError_t lu_factor<z64>(z64 *, const LUBatch &, bool, trail_fn, void *, cudaStream_t, TrailTiming *,
                                    bool);
template cudaError_t lu_step<z64>(z64 *, const LUBatch &, int, bool, trail_fn, void *, cudaStream_t, TrailTiming *,
                                  bool);
template cudaError_t lu_step<z32>(z32 *, const LUBatch &, int, bool, trail_fn, void *, cudaStream_t, TrailTiming *,
                                  bool);
template cudaError_t lu_factor<z32>(z32 *, const LUBatch &, bool, trail_fn, void *, cudaStream_t, TrailTiming *,
                                    bool);
template cudaError_t lu_trail_cuda<z64>(z64 *, const LUBatch &, int, int, cudaStream_t);
template cudaError_t lu_trail_cuda<z32>(z32 *, const LUBatch &, int, int, cudaStream_t);
template cudaError_t lu_backsolve<z64>(const z64 *, const LUBatch &, z64 *, size_t, int, int, cudaStream_t);
template cudaError_t lu_backsolve<z32>(const z32 *, const LUBatch &, z32 *, size_t, int, int, cudaStream_t);
template cudaError_t lu_fwdsolve_ws<z64>(const z64 *, const LUBatch &, z64 *, size_t, int, int, z64 *,
                                         cudaStream_t);
template cudaError_t lu_fwdsolve_ws<z32>(const z32 *, const LUBatch &, z32 *, size_t, int, int, z32 *,
                                         cudaStream_t);
