// Dense complex FP64 LU factorisation with row pivoting, and the triangular
// solves, written for B200 with no library: the device replacement of the
// reference's dense solves (PARDISO mtype 13 on the global system,
// b_mkl_solver_pardiso_d, d3qd2_mkl_solver.c:18-148, called at
// bem3_aw_qd2_solve_bieq.c:347-368; LAPACKE_zgesv on each domain's dpv system,
// solve_dpv_bv, bem3_aw_qd2_solve_bieq.c:533-653).
//
// The matrix is row-major (the layout the assembly writes), factored in place
// as P A = L U, right-looking, 32 columns per panel.  Per panel three kernels:
//
//  k_lu_panel   picks the panel's 32 pivot rows by tournament pivoting
//               (communication-avoiding LU): each CTA runs partial pivoting on a
//               slice of 256 rows, one row per thread in registers; the last of
//               up to eight CTAs to finish goes on with their winners, and so on
//               up to the root, which gives the pivot order and the packed
//               L11\U11, inverts U11 and L11, and lists the row moves (at most 64
//               touched positions).  The matrix is not written here.
//  k_lu_apply   all SMs: L21 = A21 U11^-1 for every row below the panel,
//               the row moves on the columns outside the panel, and
//               U12 = L11^-1 A12 on the pivot rows.
//  k_lu_update  all SMs: A22 -= L21 U12 on the FP64 tensor cores
//               (mma.sync m16n8k8 f64; Blackwell's tcgen05 has no FP64 kind),
//               64 x 64 complex tiles, the complex product as four real ones.
//
// A small factorisation's sequence is captured once as a CUDA graph and replayed,
// a large one runs on two streams of its own (factor_blocks).
//
// Solves: forward substitution L y = P b and back substitution U x = y in one launch
// each, one CTA per 32-row block, its diagonal block applied as an inverse formed ahead.
// The values are their own flags: the output is filled with all-ones words before the
// launch, a block polls the values that it needs and takes each 8-byte component
// (4 in FP32) once it is no longer that pattern (a 16-byte access is not one atomic), and
// a value that comes out as the pattern, a NaN handed in, is stored as another NaN.
// Waits are bounded: one that gives up sets BEM_LU_ST_WAIT and the call reports it;
// nothing hangs.  The launches are cooperative, so every CTA is resident and blocks are
// taken in order: the waits cannot deadlock.
#include "bem_count.h"
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include "bem_lu.h"

#define LU_W BEM_LU_W
#define LU_OB BEM_LU_OB  // outer block: panels whose updates right of it are delayed and applied at once
#define LU_NSLOT (2 * LU_OB / LU_W)  // panel slots (row moves, L11^-1): two outer blocks in work
#define LU_ONE_BLOCK_N 2048  // default of bem_lu.one_block_max
static_assert(LU_OB == LU_OUTER_W, "the tensor-core update depth is the outer block");
#define LU_TH 256        // threads of a panel CTA: one row each
#define LU_MAXP (2 * LU_W)
#define FULL 0xffffffffu

// integer scratch (bem_lu.piv)
#define PV_SEL 0                     // [LU_W] pivot rows in order
#define PV_LIST (1 + 2 * LU_MAXP)    // count, then (dst, src) pairs of the row moves
#define PV_PERM (PV_SEL + LU_W)      // [LU_NSLOT] lists, one per panel of two outer blocks
#define PV_INTS (PV_PERM + LU_NSLOT * PV_LIST)
// complex scratch (bem_lu.u11)
#define U_LU 0                       // [LU_W][LU_W] packed L11\U11, row i = pivot row i
#define U_UINV (LU_W * LU_W)         // U11^-1 (upper)
#define U_STAGE (2 * LU_W * LU_W)    // panel values of the rows moved out of the pivot block
#define U_LINV (3 * LU_W * LU_W)     // [LU_NSLOT] L11^-1 (unit lower) of each panel of two outer blocks
#define U_COUNT ((3 + LU_NSLOT) * LU_W * LU_W)

// the slot of the panel at column k
__host__ __device__ __forceinline__ int lu_slot(int k) { return k % (2 * LU_OB) / LU_W; }

// ---------------------------------------------------------------- complex helpers
// complex double (double2) and complex float (float2): the same code in both
// precisions
template <class C2> struct cx;
template <> struct cx<double2> {
  using R = double;
  static __device__ __forceinline__ double2 mk(double a, double b) { return make_double2(a, b); }
};
template <> struct cx<float2> {
  using R = float;
  static __device__ __forceinline__ float2 mk(float a, float b) { return make_float2(a, b); }
};
template <class C2> __device__ __forceinline__ C2 czero() { return cx<C2>::mk(0, 0); }
template <class C2> __device__ __forceinline__ C2 cone() { return cx<C2>::mk(1, 0); }
template <class C2> __device__ __forceinline__ C2 cneg(C2 a) { return cx<C2>::mk(-a.x, -a.y); }
__device__ __forceinline__ double2 cz() { return make_double2(0.0, 0.0); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// c + a b
__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
// c - a b
__device__ __forceinline__ double2 cfms(double2 a, double2 b, double2 c) {
  return make_double2(fma(-a.x, b.x, fma(a.y, b.y, c.x)), fma(-a.x, b.y, fma(-a.y, b.x, c.y)));
}
__device__ __forceinline__ double2 crcp(double2 a) {
  const double d = 1.0 / fma(a.x, a.x, a.y * a.y);
  return make_double2(a.x * d, -a.y * d);
}
__device__ __forceinline__ double cabs1(double2 a) { return fabs(a.x) + fabs(a.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cfma(float2 a, float2 b, float2 c) {
  return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
}
__device__ __forceinline__ float2 cfms(float2 a, float2 b, float2 c) {
  return make_float2(fmaf(-a.x, b.x, fmaf(a.y, b.y, c.x)), fmaf(-a.x, b.y, fmaf(-a.y, b.x, c.y)));
}
__device__ __forceinline__ float2 crcp(float2 a) {
  const float d = 1.0f / fmaf(a.x, a.x, a.y * a.y);
  return make_float2(a.x * d, -a.y * d);
}
__device__ __forceinline__ float cabs1(float2 a) { return fabsf(a.x) + fabsf(a.y); }

// ---------------------------------------------------------------- partial pivoting in one CTA
#define LU_SB 8                // columns of a sub-block
#define LU_NW (LU_TH / 32)     // warps
template <class C2>
struct gepp_sh {
  uint4 wk[2][LU_NW / 4];      // each warp's pivot key
  C2 row[2][LU_NW][LU_SB];     // its row's sub-block columns
  C2 rcp[2][LU_NW];            // the reciprocal of its pivot
  C2 l8[LU_SB][LU_SB];         // multipliers of the sub-block's pivot rows
  C2 tr[LU_SB][LU_W - LU_SB];  // their columns right of the sub-block
};

// Pivot key of a candidate: the high word (FP64) or the word (FP32) of |re| +
// |im| (non-negative numbers order as their bits) with the low 8 bits replaced
// by 255 - t, so that one integer maximum gives the largest value and, among
// values equal to 2^-12 (2^-15), the lowest row: a pivot within that of the
// largest, which keeps partial pivoting's growth bound.  0 for a row that takes
// no part.
__device__ __forceinline__ unsigned pivot_key(double a, int t) {
  return ((unsigned)__double2hiint(a) & 0xFFFFFF00u) | (unsigned)(255 - t);
}
__device__ __forceinline__ unsigned pivot_key(float a, int t) {
  return (__float_as_uint(a) & 0xFFFFFF00u) | (unsigned)(255 - t);
}
// 1 / a for the elimination steps, without a branch (a division's slow path
// would keep the compiler from scheduling it beside the updates): a scaled by a
// power of two to |re| + |im| in [1, 2), so that re^2 + im^2 neither over- nor
// underflows, and 1 / (re^2 + im^2) from the hardware's approximation by one
// third-order Newton step r (1 + e + e^2), e = 1 - d r.  Of zero it is zero (a summand
// far below the least d keeps r finite; the scale comes last, whose product with r alone
// would overflow): a column without a non-zero entry among a slice's rows then leaves
// them as they are, and the columns after it still choose among them.
__device__ __forceinline__ double2 pivot_rcp(double2 a) {
  const int e = (__double2hiint(cabs1(a)) >> 20) & 2047;
  const double sc = __hiloint2double(max(2046 - e, 1) << 20, 0);
  const double x = a.x * sc, y = a.y * sc, d = fma(x, x, fma(y, y, 0x1p-200));
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double q = fma(-d, r, 1.0);
  r = fma(r, fma(q, q, q), r);
  return make_double2(x * r * sc, -y * r * sc);
}
__device__ __forceinline__ float2 pivot_rcp(float2 a) {
  const int e = (__float_as_int(cabs1(a)) >> 23) & 255;
  const float sc = __int_as_float(max(254 - e, 1) << 23);
  const float x = a.x * sc, y = a.y * sc, d = fmaf(x, x, fmaf(y, y, 0x1p-100f));
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  r = fmaf(r, fmaf(-d, r, 1.0f), r);
  return make_float2(x * r * sc, -y * r * sc);
}
// a pivot that counts as zero: below 2^-141, an FP32 number's smallest 255 steps
template <class R> __device__ __forceinline__ bool zero_pivot(R a) { return (__float_as_uint((float)a) >> 8) == 0u; }

// Partial pivoting (|re| + |im| as LAPACK's izamax, lowest row on ties) over
// the rr <= LU_TH rows held one per thread (thread t < rr: values v), w
// columns.  Rows stay with their threads: ord becomes the row's place in the
// pivot order (-1: not picked), and a picked row's v its packed row
// (multipliers left of the pivot, U from it on).  With rd: the pivots'
// reciprocals, and a zero pivot reported in status.
//
// Latency decides here (32 dependent steps, one CTA), so the columns go in
// sub-blocks of eight: a step publishes each warp's best row, takes one barrier
// and updates at most seven columns; the columns right of the sub-block are
// updated by all eight pivots at once.  A step takes about 450 cycles; one that
// publishes and updates all 32 columns behind two barriers takes 1900 (panel of
// n = 1728: 67 -> 40 us, of which the FP64 root 24).  The sub-block is kept
// in v[0 .. 7] by rotating the registers, so that one short body serves all four.
template <class C2>
__device__ void gepp(C2 (&v)[LU_W], int &ord, int rr, int w, gepp_sh<C2> &sh, unsigned *status, C2 *rd) {
  const int t = threadIdx.x, wid = t >> 5;
  const int steps = min(w, rr);
  bool act = t < rr;
  C2 piv = cone<C2>();  // the pivot of a picked row
  ord = -1;
#pragma unroll 1
  for (int sb = 0; sb < LU_W / LU_SB; ++sb) {
    const int j0 = sb * LU_SB, cnt = min(LU_SB, steps - j0);  // pivots of this sub-block
#pragma unroll
    for (int jj = 0; jj < LU_SB; ++jj) {
      if (jj >= cnt) continue;
      const int b = jj & 1;
      const unsigned key = act ? pivot_key(cabs1(v[jj]), t) : 0u;
      const unsigned wmax = __reduce_max_sync(FULL, key);
      const C2 rc = pivot_rcp(v[jj]);  // by every row, beside the search
      if (act && key == wmax) {  // this warp's best row (keys of active rows are distinct)
#pragma unroll
        for (int c = jj; c < LU_SB; ++c) sh.row[b][wid][c] = v[c];
        sh.rcp[b][wid] = rc;
        reinterpret_cast<unsigned *>(sh.wk[b])[wid] = wmax;
      }
      if (wmax == 0u && (t & 31) == 0) reinterpret_cast<unsigned *>(sh.wk[b])[wid] = 0u;
      __syncthreads();
      const uint4 ka = sh.wk[b][0], kb = sh.wk[b][1];
      const unsigned best = max(max(max(ka.x, ka.y), max(ka.z, ka.w)), max(max(kb.x, kb.y), max(kb.z, kb.w)));
      const int p = 255 - (int)(best & 255u), pw = p >> 5;
      // no branch from here to the next barrier: every warp waits for the
      // slowest, and the pivot's warp would pay for both sides
      ord = t == p ? j0 + jj : ord;
      piv = t == p ? v[jj] : piv;
      act = act && t != p;
      C2 l = cmul(v[jj], sh.rcp[b][pw]);
      v[jj] = act ? l : v[jj];
      l = act ? l : czero<C2>();
#pragma unroll
      for (int c = jj + 1; c < LU_SB; ++c) v[c] = cfms(l, sh.row[b][pw][c], v[c]);
    }
    if (sb < LU_W / LU_SB - 1 && cnt > 0) {
      // the columns right of the sub-block: U there from the pivot rows
      // (unit lower solve, a thread per column), then every other row
      const int nrem = LU_W - LU_SB - j0;
      const int i = ord - j0;
      if (i >= 0) {
#pragma unroll
        for (int c = 0; c < LU_SB; ++c) sh.l8[i][c] = v[c];
#pragma unroll
        for (int c = 0; c < LU_W - LU_SB; ++c)
          if (c < nrem) sh.tr[i][c] = v[LU_SB + c];
      }
      __syncthreads();
      if (t < nrem) {
        C2 x[LU_SB];
#pragma unroll
        for (int r = 0; r < LU_SB; ++r) x[r] = r < cnt ? sh.tr[r][t] : czero<C2>();
#pragma unroll
        for (int r = 1; r < LU_SB; ++r)
          if (r < cnt)
#pragma unroll
            for (int c = 0; c < r; ++c) x[r] = cfms(sh.l8[r][c], x[c], x[r]);
#pragma unroll
        for (int r = 0; r < LU_SB; ++r)
          if (r < cnt) sh.tr[r][t] = x[r];
      }
      __syncthreads();
      if (i >= 0) {
#pragma unroll
        for (int c = 0; c < LU_W - LU_SB; ++c)
          if (c < nrem) v[LU_SB + c] = sh.tr[i][c];
      } else if (act) {
#pragma unroll
        for (int ch = 0; ch < LU_W / LU_SB - 1; ++ch)
          if (ch * LU_SB < nrem)
#pragma unroll
            for (int r = 0; r < LU_SB; ++r)
              if (r < cnt)
#pragma unroll
                for (int c = 0; c < LU_SB; ++c)
                  v[LU_SB + ch * LU_SB + c] = cfms(v[r], sh.tr[r][ch * LU_SB + c], v[LU_SB + ch * LU_SB + c]);
      }
    }
    // rotate: the finished sub-block goes behind the others
    C2 f[LU_SB];
#pragma unroll
    for (int c = 0; c < LU_SB; ++c) f[c] = v[c];
#pragma unroll
    for (int c = 0; c < LU_W - LU_SB; ++c) v[c] = v[c + LU_SB];
#pragma unroll
    for (int c = 0; c < LU_SB; ++c) v[LU_W - LU_SB + c] = f[c];
  }
  if (rd && ord >= 0) {
    rd[ord] = crcp(piv);
    if (zero_pivot(cabs1(piv))) atomicOr(status, BEM_LU_ST_ZERO);  // no non-zero entry was left
  }
  __syncthreads();  // the shared buffers may be used again
}

// ---------------------------------------------------------------- panel
// The panel's columns of one row per thread (id: the row, -1 none) into
// registers, converted to T (the leaves' partial pivoting only selects rows, so
// it runs in complex FP32 for either precision of the factorisation).  A warp
// reads four rows' eight columns at a time, whole 128-byte lines, and turns
// them through stage (32 x 9 of T per warp) so that each lane gets its own row;
// read row by row the loads take 8000 cycles of the SM's load path, this 1000.
__device__ __forceinline__ void cvt(double2 x, double2 &y) { y = x; }
__device__ __forceinline__ void cvt(double2 x, float2 &y) { y = make_float2((float)x.x, (float)x.y); }
__device__ __forceinline__ void cvt(float2 x, float2 &y) { y = x; }
template <class T, class C2>
__device__ __forceinline__ void load_rows(T (&v)[LU_W], const C2 *A, long lda, int id, int k, int w, T *stage) {
  const int lane = threadIdx.x & 31, sub = lane >> 3, col = lane & 7;
  T *s = stage + (threadIdx.x >> 5) * (32 * 9);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = __shfl_sync(FULL, id, i * 4 + sub);
    const C2 *p = A + (size_t)(row < 0 ? 0 : row) * lda + k;
#pragma unroll
    for (int c = 0; c < LU_W / 8; ++c) {
      const C2 x = (row >= 0 && c * 8 + col < w) ? p[c * 8 + col] : czero<C2>();
      cvt(x, v[c * 8 + i]);
    }
  }
#pragma unroll
  for (int c = 0; c < LU_W / 8; ++c) {
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) s[(i * 4 + sub) * 9 + col] = v[c * 8 + i];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) v[c * 8 + i] = s[lane * 9 + i];
  }
}

template <class C2>
struct panel_sh {
  gepp_sh<C2> g;
  gepp_sh<float2> gl;
  union {
    struct {
      C2 lu[LU_W][LU_W + 1];
      C2 iv[2][LU_W][LU_W + 1];  // U11^-1, L11^-1
    };
    C2 stage[LU_NW * 32 * 9];    // load_rows
  };
  C2 rd[LU_W];                   // reciprocals of U11's diagonal
  int sel[LU_W], la[LU_W], lb[LU_W];
  int last;
};

// X = T^-1 of the two triangles of lu (b = 0: U, b = 1: unit L), by inverting
// the 8 x 8 diagonal blocks (a warp each) and doubling the block size twice:
// the off-diagonal block of the inverse is -T22^-1 T21 T11^-1 (L), -T11^-1 T12
// T22^-1 (U).  All threads; lu complete before, iv complete after.
template <class C2>
__device__ void tri_inverses(panel_sh<C2> &S, int w) {
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  for (int e = t; e < 2 * LU_W * (LU_W + 1); e += LU_TH) (&S.iv[0][0][0])[e] = czero<C2>();
  __syncthreads();
  {
    const int up = wid < 4, d = (wid & 3) * 8;  // this warp's diagonal block, a lane per column
    if (lane < 8) {
      C2 x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = (i == lane) ? cone<C2>() : czero<C2>();
      if (up) {
#pragma unroll
        for (int l = 7; l >= 0; --l) {
          // an identity beyond a short panel keeps the block regular
          const C2 dg = d + l < w ? S.rd[d + l] : cone<C2>();
          x[l] = cmul(x[l], dg);
#pragma unroll
          for (int i = 0; i < l; ++i) x[i] = cfms(S.lu[d + i][d + l], x[l], x[i]);
        }
      } else {
#pragma unroll
        for (int l = 0; l < 8; ++l)
#pragma unroll
          for (int i = l + 1; i < 8; ++i) x[i] = cfms(S.lu[d + i][d + l], x[l], x[i]);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) S.iv[up ? 0 : 1][d + i][d + lane] = x[i];
    }
  }
  __syncthreads();
#pragma unroll
  for (int bs = 8; bs < LU_W; bs *= 2) {
    // products of bs x bs blocks: 32 / (2 bs) of them for each triangle
    const int per = bs * bs, tot = 2 * (LU_W / (2 * bs)) * per;
    C2 y[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = t + h * LU_TH;
      y[h] = czero<C2>();
      if (e < tot) {
        const int b = e / (tot / 2), r = e % (tot / 2), blk = r / per, i = r % per / bs, j = r % bs;
        const int o = blk * 2 * bs, ro = b ? o + bs : o, co = b ? o : o + bs;  // the off-diagonal block
        // T_off T_(column's diagonal)^-1
        for (int l = 0; l < bs; ++l) y[h] = cfma(S.lu[ro + i][co + l], S.iv[b][co + l][co + j], y[h]);
      }
    }
    // the strictly other triangle of iv holds the intermediate product
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = t + h * LU_TH;
      if (e < tot) {
        const int b = e / (tot / 2), r = e % (tot / 2), blk = r / per, i = r % per / bs, j = r % bs;
        const int o = blk * 2 * bs, ro = b ? o + bs : o, co = b ? o : o + bs;
        S.iv[b][co + i][ro + j] = y[h];
      }
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = t + h * LU_TH;
      if (e < tot) {
        const int b = e / (tot / 2), r = e % (tot / 2), blk = r / per, i = r % per / bs, j = r % bs;
        const int o = blk * 2 * bs, ro = b ? o + bs : o, co = b ? o : o + bs;
        C2 z = czero<C2>();
        for (int l = 0; l < bs; ++l) z = cfma(S.iv[b][ro + i][ro + l], S.iv[b][co + l][ro + j], z);
        y[h] = cneg(z);
      }
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = t + h * LU_TH;
      if (e < tot) {
        const int b = e / (tot / 2), r = e % (tot / 2), blk = r / per, i = r % per / bs, j = r % bs;
        const int o = blk * 2 * bs, ro = b ? o + bs : o, co = b ? o : o + bs;
        S.iv[b][ro + i][co + j] = y[h];
        S.iv[b][co + i][ro + j] = czero<C2>();
      }
    }
    __syncthreads();
  }
}

// Tournament over ceil(m / LU_TH) leaves: block b eliminates its slice of the
// panel's rows and leaves its winners; the block that finishes last of up to
// eight goes on with their winners, and so on up to the root (no block waits
// for another).  tree: winners [node][1 + LU_W] (count, rows), then a counter
// per node, zero between launches.
template <class C2>
__global__ void __launch_bounds__(LU_TH, 1)
    k_lu_panel(C2 *A, long lda, int n, int k, int *pv, int *tree, int max_nodes, C2 *u, unsigned *status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  panel_sh<C2> &S = *reinterpret_cast<panel_sh<C2> *>(smem_raw);
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int w = min(LU_W, n - k), m = n - k;
  int id = -1, rr = m, ord = -1;
  if (gridDim.x > 1) {
    int *counter = tree + (size_t)max_nodes * (1 + LU_W);
    int nn = gridDim.x, node = blockIdx.x, base = 0;  // nodes of this level, this one, the level's first
    {
      const int q = (m + nn - 1) / nn, lo = k + node * q, hi = min(n, lo + q);
      rr = max(0, hi - lo);
      id = t < rr ? lo + t : -1;
    }
    while (true) {
      float2 vl[LU_W];
      load_rows(vl, A, lda, id, k, w, reinterpret_cast<float2 *>(S.stage));
      gepp(vl, ord, rr, w, S.gl, nullptr, (float2 *)nullptr);
      int *win = tree + (size_t)(base + node) * (1 + LU_W);
      if (ord >= 0) win[1 + ord] = id;
      if (t == 0) win[0] = min(w, rr);
      __threadfence();
      __syncthreads();
      const int parents = (nn + 7) / 8, par = node / 8;
      if (t == 0) {
        const int kids = min(8, nn - par * 8);
        S.last = atomicAdd(counter + base + nn + par, 1) == kids - 1;
        if (S.last) counter[base + nn + par] = 0;
      }
      __syncthreads();
      if (!S.last) return;
      __threadfence();
      // this block goes on as the parent: its children's winners, one per thread
      int total = 0, mine = -1;
      for (int c = par * 8; c < min(nn, par * 8 + 8); ++c) {
        const int *wc = tree + (size_t)(base + c) * (1 + LU_W);
        const int cnt = __ldcg(wc);
        if (t >= total && t < total + cnt) mine = __ldcg(wc + 1 + (t - total));
        total += cnt;
      }
      base += nn;
      nn = parents;
      node = par;
      id = mine;
      rr = total;
      if (nn == 1) break;
    }
  } else {
    id = t < m ? k + t : -1;
  }
  // root: partial pivoting over the last winners (or over all rows of a short
  // panel), with the values kept: the pivot order and L11\U11
  C2 v[LU_W];
  load_rows(v, A, lda, id, k, w, S.stage);
  gepp(v, ord, rr, w, S.g, status, S.rd);
  if (t < LU_W) {
    S.sel[t] = -1;
    if (t >= w)
#pragma unroll
      for (int c = 0; c < LU_W; ++c) S.lu[t][c] = czero<C2>();
  }
  __syncthreads();
  if (ord >= 0) {
#pragma unroll
    for (int c = 0; c < LU_W; ++c) S.lu[ord][c] = v[c];
    S.sel[ord] = id;
    pv[PV_SEL + ord] = id;
  }
  __syncthreads();
  tri_inverses(S, w);
  for (int e = t; e < LU_W * LU_W; e += LU_TH) {
    const int i = e / LU_W, j = e % LU_W;
    const bool in = i < w && j < w;  // entries outside a short panel (w < 32) are zero
    u[U_LU + e] = S.lu[i][j];
    u[U_UINV + e] = in ? S.iv[0][i][j] : czero<C2>();
    u[U_LINV + lu_slot(k) * (LU_W * LU_W) + e] = in ? S.iv[1][i][j] : czero<C2>();
  }
  if (wid == 2) {
    // row moves: pivot row i goes to position k + i; the rows of the pivot
    // block that were not picked (displaced) go to the positions the pivot
    // rows from below left, paired in lane order
    const int i = lane;
    const int p = (i < w) ? S.sel[i] : -1;
    const bool below = (i < w) && (p >= k + w);
    bool picked = false;
    for (int jj = 0; jj < w; ++jj) picked |= (S.sel[jj] == k + i);
    const bool displaced = (i < w) && !picked;
    const unsigned ba = __ballot_sync(FULL, below), bb = __ballot_sync(FULL, displaced);
    const unsigned lt = (1u << lane) - 1u;
    if (below) S.la[__popc(ba & lt)] = p;
    if (displaced) S.lb[__popc(bb & lt)] = k + i;
    __syncwarp();
    const int cnt = __popc(ba);
    int *perm = pv + PV_PERM + lu_slot(k) * PV_LIST;
    if (lane == 0) perm[0] = w + cnt;
    if (i < w) { perm[1 + 2 * i] = k + i; perm[2 + 2 * i] = p; }
    if (lane < cnt) { perm[1 + 2 * (w + lane)] = S.la[lane]; perm[2 + 2 * (w + lane)] = S.lb[lane]; }
    // the displaced rows' panel values, before anything overwrites them
    for (int r = 0; r < cnt; ++r)
      u[U_STAGE + r * LU_W + lane] = lane < w ? A[(size_t)S.lb[r] * lda + k + lane] : czero<C2>();
  }
}

// ---------------------------------------------------------------- row moves, L21, U12
#define AP_TH 128
#define AP_ROWS 32   // rows of an L21 block (4 threads per row)
#define AP_COLS 16   // columns of a row-move block

template <class C2>
__global__ void __launch_bounds__(AP_TH) k_lu_apply(C2 *A, long lda, int n, int k, int cbeg, int cend, const int *pv, const C2 *u,
                                                    int *rowmap, unsigned *status) {
  __shared__ C2 sm[LU_W][LU_W + 1];
  __shared__ C2 srow[LU_MAXP][AP_COLS + 1];
  __shared__ int sdst[LU_MAXP], ssrc[LU_MAXP], moved[AP_ROWS];
  const int t = threadIdx.x;
  const int w = min(LU_W, n - k);
  const int r0 = k + w;
  const int nL = (n - r0 + AP_ROWS - 1) / AP_ROWS;
  const int nCl = (k - cbeg + AP_COLS - 1) / AP_COLS, nCr = (cend - r0 + AP_COLS - 1) / AP_COLS;
  const int b = blockIdx.x;
  pv += PV_PERM + lu_slot(k) * PV_LIST;
  // everything read through the row list or needed beside it is loaded at
  // once: the kernel is a chain of latencies, not of work
  int nperm = __ldcg(pv);
  int md = k, ms = k;
  if (t < LU_MAXP) {
    md = __ldcg(pv + 1 + 2 * t);
    ms = __ldcg(pv + 2 + 2 * t);
  }
  const int ci = b - nL;  // column block
  const bool right = ci >= nCl;
  const int c0 = right ? r0 + (ci - nCl) * AP_COLS : cbeg + ci * AP_COLS;
  const bool u12 = b >= nL && b < nL + nCl + nCr && right;
  if (b < nL || b >= nL + nCl + nCr || u12) {
    const C2 *src = u + (u12 ? U_LINV + lu_slot(k) * (LU_W * LU_W) : U_UINV);
#pragma unroll
    for (int e = t; e < LU_W * LU_W; e += AP_TH) sm[e / LU_W][e % LU_W] = __ldcg(src + e);
  }
  if (t < AP_ROWS) moved[t] = 0;
  if (nperm < 0 || nperm > LU_MAXP) {
    if (t == 0) atomicOr(status, BEM_LU_ST_INTERNAL);
    nperm = 0;
  }
  if (t < nperm) {
    if (md < k || md >= n || ms < k || ms >= n) {  // a row move out of range: report, keep the row
      if (b == 0) atomicOr(status, BEM_LU_ST_INTERNAL);
      md = ms = k + (t < w ? t : 0);
    }
    sdst[t] = md;
    ssrc[t] = ms;
  }
  if (b < nL) {
    // (a launch at n = 1728: 12 us with strided U11^-1 columns per thread and
    // the loads one after another, 5 us)
    // L21 = A21 U11^-1 in place, for the rows below the pivot block that no move touches
    const int rb = r0 + b * AP_ROWS, row = rb + (t >> 2), part = t & 3;
    // the row's panel values, loaded at once (independent loads, not a chain)
    C2 a[LU_W];
    {
      const C2 *ap = A + (size_t)(row < n ? row : r0) * lda + k;
#pragma unroll
      for (int l = 0; l < LU_W; ++l) a[l] = (row < n && l < w) ? ap[l] : czero<C2>();
    }
    __syncthreads();
    if (t >= w && t < nperm && md >= rb && md < rb + AP_ROWS) moved[md - rb] = 1;
    C2 x[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) x[c] = czero<C2>();
#pragma unroll
    for (int l = 0; l < LU_W; ++l)
#pragma unroll
      for (int c = 0; c < 8; ++c) x[c] = cfma(a[l], sm[l][part + 4 * c], x[c]);  // four neighbours: no bank conflict
    __syncthreads();  // every read of the row before any write to it
    if (row < n && !moved[t >> 2]) {
      C2 *ap = A + (size_t)row * lda + k;
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (part + 4 * c < w) ap[part + 4 * c] = x[c];
    }
    return;
  }
  __syncthreads();  // sdst / ssrc, sm
  if (b < nL + nCl + nCr) {
    // the row moves on AP_COLS of the outer block's columns [cbeg, cend) outside
    // the panel; right of the panel also U12 = L11^-1 A12 on the pivot block
    // (outside the outer block the moves wait for k_lu_swap)
    const int nc = min(right ? cend : k, c0 + AP_COLS) - c0;
    const int cc = t % AP_COLS, grp = t / AP_COLS;  // 8 groups of 16 columns
#pragma unroll
    for (int q = 0; q < LU_MAXP * AP_COLS / AP_TH; ++q) {
      const int pr = grp + q * (AP_TH / AP_COLS);
      srow[pr][cc] = (pr < nperm && cc < nc) ? A[(size_t)ssrc[pr] * lda + c0 + cc] : czero<C2>();
    }
    __syncthreads();
    if (cc >= nc) return;
    if (u12) {
      // four rows at a time (L11^-1 is zero right of its diagonal)
      C2 s[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) s[q] = czero<C2>();
#pragma unroll 4
      for (int l = 0; l < LU_W; ++l) {
        const C2 x = srow[l][cc];
#pragma unroll
        for (int q = 0; q < 4; ++q) s[q] = cfma(sm[grp + 8 * q][l], x, s[q]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (grp + 8 * q < w) A[(size_t)(k + grp + 8 * q) * lda + c0 + cc] = s[q];
    }
#pragma unroll
    for (int q = 0; q < LU_MAXP * AP_COLS / AP_TH; ++q) {
      const int e = grp + q * (AP_TH / AP_COLS);
      if (e < nperm && !(u12 && e < w)) A[(size_t)sdst[e] * lda + c0 + cc] = srow[e][cc];
    }
    return;
  }
  // last block: the panel columns of the moved rows (the pivot block gets
  // L11\U11, a row moved below it its L21), and the row map
  for (int e = t; e < w * LU_W; e += AP_TH) {
    const int ii = e / LU_W, c = e % LU_W;
    if (c < w) A[(size_t)(k + ii) * lda + k + c] = __ldcg(u + U_LU + ii * LU_W + c);
  }
  {
    const int r = t >> 2, part = t & 3, e = w + r;
    if (e < nperm) {
      C2 a[LU_W];
#pragma unroll
      for (int l = 0; l < LU_W; ++l) a[l] = l < w ? __ldcg(u + U_STAGE + r * LU_W + l) : czero<C2>();
      C2 x[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) x[c] = czero<C2>();
#pragma unroll
      for (int l = 0; l < LU_W; ++l)
#pragma unroll
        for (int c = 0; c < 8; ++c) x[c] = cfma(a[l], sm[l][part + 4 * c], x[c]);
      C2 *ap = A + (size_t)sdst[e] * lda + k;
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (part + 4 * c < w) ap[part + 4 * c] = x[c];
    }
  }
  int old = 0;
  if (t < nperm) old = rowmap[ssrc[t]];
  __syncthreads();
  if (t < nperm) rowmap[sdst[t]] = old;
}

// The row moves of the np panels from column K on, on the columns [0, left) and
// [cbeg, cend), AP_COLS columns per CTA, panel after panel: kept back from the
// columns outside the outer block until the previous block's trailing update,
// which runs beside the panels, is done with their rows.
template <class C2>
__global__ void __launch_bounds__(AP_TH) k_lu_swap(C2 *A, long lda, int n, int K, int np, int left, int cbeg, int cend,
                                                   const int *pv) {
  __shared__ C2 srow[LU_MAXP][AP_COLS + 1];
  __shared__ int sdst[LU_OB / LU_W][LU_MAXP], ssrc[LU_OB / LU_W][LU_MAXP], scnt[LU_OB / LU_W];
  const int t = threadIdx.x;
  const int nCl = (left + AP_COLS - 1) / AP_COLS;
  const bool right = (int)blockIdx.x >= nCl;
  const int c0 = right ? cbeg + ((int)blockIdx.x - nCl) * AP_COLS : (int)blockIdx.x * AP_COLS;
  const int nc = min(right ? cend : left, c0 + AP_COLS) - c0;
  for (int e = t; e < np * LU_MAXP; e += AP_TH) {
    const int s = e / LU_MAXP, i = e % LU_MAXP;
    const int *l = pv + PV_PERM + lu_slot(K + s * LU_W) * PV_LIST;
    int d = __ldcg(l + 1 + 2 * i), sr = __ldcg(l + 2 + 2 * i);
    const int cnt = __ldcg(l);
    if (i == 0) scnt[s] = cnt < 0 || cnt > LU_MAXP ? 0 : cnt;  // (k_lu_apply reports a list out of range)
    if (d < K || d >= n || sr < K || sr >= n) d = sr = K;
    sdst[s][i] = d;
    ssrc[s][i] = sr;
  }
  __syncthreads();
  const int cc = t % AP_COLS, grp = t / AP_COLS;
  for (int s = 0; s < np; ++s) {
    const int cnt = scnt[s];
#pragma unroll
    for (int q = 0; q < LU_MAXP * AP_COLS / AP_TH; ++q) {
      const int e = grp + q * (AP_TH / AP_COLS);
      if (e < cnt && cc < nc) srow[e][cc] = A[(size_t)ssrc[s][e] * lda + c0 + cc];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < LU_MAXP * AP_COLS / AP_TH; ++q) {
      const int e = grp + q * (AP_TH / AP_COLS);
      if (e < cnt && cc < nc) A[(size_t)sdst[s][e] * lda + c0 + cc] = srow[e][cc];
    }
    __syncthreads();  // the moves of panel s before the reads of panel s + 1
  }
}

// ---------------------------------------------------------------- trailing update
#define UP_BM 64
#define UP_BN 64
#define UP_TH 256
#define UP_BK 8     // depth of a slice
#define UP_NST 5    // slices in flight
#define UP_LDA 12   // row strides (complex) of the slices: a quarter warp's 16-byte
#define UP_LDB 66   // fragment loads fall into distinct banks
#define UP_STAGE (UP_BM * UP_LDA + UP_BK * UP_LDB)
#define UP_SMEM (UP_NST * UP_STAGE * sizeof(double2))

// d = a b + d on a 16 x 8 x 8 FP64 tile, g = lane / 4, q = lane % 4: a holds
// rows g (a[0], a[2]) and g + 8 (a[1], a[3]) at columns q and q + 4, b column g
// at rows q and q + 4, d rows g and g + 8 at columns 2 q and 2 q + 1
__device__ __forceinline__ void dmma(const double (&a)[4], double b0, double b1, double (&d)[4]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}
// 16 bytes from global to shared memory, asynchronously; zeros when not live
__device__ __forceinline__ void cp16(double2 *dst, const double2 *src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(live ? 16 : 0)
               : "memory");
}

// C -= L U on the FP64 tensor cores: C = A[r0:n, c0:cend), L = A[r0:n, kk:kk+kw),
// U = A[kk:kk+kw, c0:cend), kw a multiple of 8.  A panel's update (kk = k, kw =
// 32, cend = the end of its outer block) and an outer block's (kk = its first
// column, kw = LU_OB, cend = n) alike.  64 x 64 complex tiles, 8 warps of 32 x
// 16, the complex product as four real ones; L and U pass through a ring of
// slices in shared memory filled by asynchronous copies (2 blocks per SM, 103 KB
// each), C is fetched into L2 meanwhile and met at the end.  30.7 TFLOP/s over a
// factorisation of n = 12288, 36.5 being what the instruction alone reaches;
// filling the ring and meeting C take 6 us of a tile's 35.  Blocks that took
// several tiles, the next one's first slices on their way while one ends, were
// slower (30.1), as were 16-deep slices (29.8).
__global__ void __launch_bounds__(UP_TH, 2) k_lu_update(double2 *A, long lda, int n, int kk, int kw, int r0,
                                                        int c0, int cend) {
  extern __shared__ __align__(16) unsigned char up_raw[];
  double2 *sm = reinterpret_cast<double2 *>(up_raw);
  const int t = threadIdx.x;
  const int rb = r0 + blockIdx.y * UP_BM, cb = c0 + blockIdx.x * UP_BN;
  const int lane = t & 31, wid = t >> 5, g = lane >> 2, q = lane & 3;
  const int wm = (wid & 1) * 32, wn = (wid >> 1) * 16;  // warp tile: 32 rows x 16 columns
  const int nk = kw / UP_BK;
  auto fill = [&](int st, int k0) {
    double2 *As = sm + st * UP_STAGE, *Bs = As + UP_BM * UP_LDA;
#pragma unroll
    for (int i = 0; i < UP_BM * UP_BK / UP_TH; ++i) {
      const int e = t + i * UP_TH, r = e / UP_BK, c = e % UP_BK;
      const bool live = rb + r < n;
      cp16(As + r * UP_LDA + c, A + (size_t)(live ? rb + r : r0) * lda + kk + k0 + c, live);
    }
#pragma unroll
    for (int i = 0; i < UP_BK * UP_BN / UP_TH; ++i) {
      const int e = t + i * UP_TH, r = e / UP_BN, c = e % UP_BN;
      const bool live = cb + c < cend;
      cp16(Bs + r * UP_LDB + c, A + (size_t)(kk + k0 + r) * lda + (live ? cb + c : c0), live);
    }
  };
#pragma unroll
  for (int s = 0; s < UP_NST - 1; ++s) {
    if (s < nk) fill(s, s * UP_BK);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  double cr[2][2][4], ci[2][2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) cr[i][j][c] = ci[i][j][c] = 0.0;
  {
    const int row = rb + (t >> 2), col = cb + (t & 3) * 16;
#pragma unroll
    for (int c = 0; c < 16; c += 8)
      if (row < n && col + c < cend) asm volatile("prefetch.global.L2 [%0];" ::"l"(A + (size_t)row * lda + col + c));
  }
  int st = 0;
  for (int it = 0; it < nk; ++it) {
    asm volatile("cp.async.wait_group %0;" ::"n"(UP_NST - 2) : "memory");
    __syncthreads();  // this slice is in, and every warp is done with the one before
    if (it + UP_NST - 1 < nk) fill(st == 0 ? UP_NST - 1 : st - 1, (it + UP_NST - 1) * UP_BK);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const double2 *As = sm + st * UP_STAGE, *Bs = As + UP_BM * UP_LDA;
    st = st == UP_NST - 1 ? 0 : st + 1;
    double2 b[2][2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int c = 0; c < 2; ++c) b[j][c] = Bs[(q + 4 * c) * UP_LDB + wn + j * 8 + g];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      // (cr, ci) -= (ar + i ai)(br + i bi)
      double nr[4], ai[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const double2 a = As[(wm + i * 16 + g + (c & 1) * 8) * UP_LDA + q + (c >> 1) * 4];
        nr[c] = -a.x;
        ai[c] = a.y;
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        dmma(nr, b[j][0].x, b[j][1].x, cr[i][j]);
        dmma(nr, b[j][0].y, b[j][1].y, ci[i][j]);
        dmma(ai, b[j][0].y, b[j][1].y, cr[i][j]);
        dmma(ai, -b[j][0].x, -b[j][1].x, ci[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    // eight loads in flight, then eight stores (one by one each load would wait
    // for the store before it)
    double2 x[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int row = rb + wm + i * 16 + g + (c >> 1) * 8, col = cb + wn + j * 8 + 2 * q + (c & 1);
        x[j][c] = (row < n && col < cend) ? A[(size_t)row * lda + col] : cz();
      }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int row = rb + wm + i * 16 + g + (c >> 1) * 8, col = cb + wn + j * 8 + 2 * q + (c & 1);
        if (row < n && col < cend)
          A[(size_t)row * lda + col] = make_double2(x[j][c].x + cr[i][j][c], x[j][c].y + ci[i][j][c]);
      }
  }
}

// The same on a few panels' columns, which the next panel waits for: 32 x 32
// tiles (4 warps of 16 x 16), so that the few tiles of a strip spread over the
// SMs and none of a tile's columns is empty; 32 of the kw columns of L in one
// load.  kw = 32 at n = 1728: 3.2 us, 7.5 with the 64 x 64 tiles.
#define SP_B 32
#define SP_TH 128
#define SP_LDA 36
#define SP_LDB 34
__global__ void __launch_bounds__(SP_TH) k_lu_strip(double2 *A, long lda, int n, int kk, int kw, int r0, int c0, int cend) {
  __shared__ __align__(16) double2 As[SP_B * SP_LDA], Bs[SP_B * SP_LDB];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, g = lane >> 2, q = lane & 3;
  const int rb = r0 + blockIdx.x * SP_B, wm = (wid & 1) * 16, wn = (wid >> 1) * 16;
  c0 += blockIdx.y * SP_B;
  auto fill = [&](int k0) {
#pragma unroll
    for (int i = 0; i < SP_B * SP_B / SP_TH; ++i) {
      const int e = t + i * SP_TH, r = e / SP_B, c = e % SP_B;
      const bool la = rb + r < n, lb = c0 + c < cend;
      cp16(As + r * SP_LDA + c, A + (size_t)(la ? rb + r : r0) * lda + kk + k0 + c, la);
      cp16(Bs + r * SP_LDB + c, A + (size_t)(kk + k0 + r) * lda + (lb ? c0 + c : c0), lb);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fill(0);
  double cr[2][4], ci[2][4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int row = rb + wm + g + (c >> 1) * 8, col = c0 + wn + j * 8 + 2 * q + (c & 1);
      const double2 x = (row < n && col < cend) ? A[(size_t)row * lda + col] : cz();
      cr[j][c] = x.x;
      ci[j][c] = x.y;
    }
  for (int k0 = 0; k0 < kw; k0 += SP_B) {
    if (k0) {
      __syncthreads();  // the previous columns' fragment loads are done
      fill(k0);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int k8 = 0; k8 < SP_B; k8 += 8) {
      double nr[4], ai[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const double2 a = As[(wm + g + (c & 1) * 8) * SP_LDA + k8 + q + (c >> 1) * 4];
        nr[c] = -a.x;
        ai[c] = a.y;
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const double2 b0 = Bs[(k8 + q) * SP_LDB + wn + j * 8 + g], b1 = Bs[(k8 + q + 4) * SP_LDB + wn + j * 8 + g];
        dmma(nr, b0.x, b1.x, cr[j]);
        dmma(nr, b0.y, b1.y, ci[j]);
        dmma(ai, b0.y, b1.y, cr[j]);
        dmma(ai, -b0.x, -b1.x, ci[j]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int row = rb + wm + g + (c >> 1) * 8, col = c0 + wn + j * 8 + 2 * q + (c & 1);
      if (row < n && col < cend) A[(size_t)row * lda + col] = make_double2(cr[j][c], ci[j][c]);
    }
}
// complex FP32, on the CUDA cores: two rows and four columns per thread
__global__ void __launch_bounds__(SP_TH) k_lu_strip_c32(float2 *A, long lda, int n, int kk, int kw, int r0, int c0, int cend) {
  __shared__ float2 As[SP_B][SP_B + 1], Bs[SP_B][SP_B + 1];
  const int t = threadIdx.x, ty = t >> 3, tx = t & 7;
  const int rb = r0 + blockIdx.x * SP_B;
  c0 += blockIdx.y * SP_B;
  float2 acc[2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int row = rb + ty + 16 * i, col = c0 + tx + 8 * j;
      acc[i][j] = (row < n && col < cend) ? A[(size_t)row * lda + col] : make_float2(0.f, 0.f);
    }
  for (int k0 = 0; k0 < kw; k0 += SP_B) {
    if (k0) __syncthreads();
#pragma unroll
    for (int i = 0; i < SP_B * SP_B / SP_TH; ++i) {
      const int e = t + i * SP_TH, r = e / SP_B, c = e % SP_B;
      As[r][c] = rb + r < n ? A[(size_t)(rb + r) * lda + kk + k0 + c] : make_float2(0.f, 0.f);
      Bs[r][c] = c0 + c < cend ? A[(size_t)(kk + k0 + r) * lda + c0 + c] : make_float2(0.f, 0.f);
    }
    __syncthreads();
#pragma unroll 8
    for (int l = 0; l < SP_B; ++l)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = cfms(As[ty + 16 * i][l], Bs[l][tx + 8 * j], acc[i][j]);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int row = rb + ty + 16 * i, col = c0 + tx + 8 * j;
      if (row < n && col < cend) A[(size_t)row * lda + col] = acc[i][j];
    }
}

// complex FP32: the same update on the CUDA cores, 64 x 64 tiles, 4 x 4
// outputs per thread (rows ty*4 + i, columns tx + 16 j: conflict-free shared
// loads and 128-byte runs of C per 16 threads)
#define UF_TH 256
__global__ void __launch_bounds__(UF_TH) k_lu_update_c32(float2 *A, long lda, int n, int kk, int kw, int r0,
                                                         int c0, int cend) {
  __shared__ float2 As[UP_BM][LU_W + 1];
  __shared__ float2 Bs[LU_W][UP_BN + 1];
  const int t = threadIdx.x;
  const int rb = r0 + blockIdx.y * UP_BM, cb = c0 + blockIdx.x * UP_BN;
  const int ty = t >> 4, tx = t & 15;
  float2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int row = rb + ty * 4 + i, col = cb + tx + 16 * j;
      acc[i][j] = (row < n && col < cend) ? A[(size_t)row * lda + col] : make_float2(0.f, 0.f);
    }
  for (int q0 = 0; q0 < kw; q0 += LU_W) {
    const int wq = min(LU_W, kw - q0), kc = kk + q0;
    if (q0) __syncthreads();
    for (int e = t; e < UP_BM * LU_W; e += UF_TH) {
      const int r = e / LU_W, c = e % LU_W;
      As[r][c] = (rb + r < n && c < wq) ? A[(size_t)(rb + r) * lda + kc + c] : make_float2(0.f, 0.f);
    }
    for (int e = t; e < LU_W * UP_BN; e += UF_TH) {
      const int r = e / UP_BN, c = e % UP_BN;
      Bs[r][c] = (r < wq && cb + c < cend) ? A[(size_t)(kc + r) * lda + cb + c] : make_float2(0.f, 0.f);
    }
    __syncthreads();
#pragma unroll 4
    for (int k1 = 0; k1 < LU_W; ++k1) {
      float2 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[ty * 4 + i][k1];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[k1][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = cfms(a[i], b[j], acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int row = rb + ty * 4 + i, col = cb + tx + 16 * j;
      if (row < n && col < cend) A[(size_t)row * lda + col] = acc[i][j];
    }
}

// ---------------------------------------------------------------- U12 of an outer block
// U12 = L11^-1 A12 in place for the outer block's rows K .. K + ob - 1 and the
// columns [cbeg, cend) right of it (L11 unit lower, in A's strictly lower part, its
// diagonal blocks' inverses in the LINV slots): block row ib gets
// Linv_ib (A12_ib - sum_{jb < ib} L_ib,jb U12_jb).  One CTA per TR_NC columns;
// thread (i, cq) holds row i of a block row and columns cq, cq + 8.  The ten
// 32 x 32 blocks pass through two buffers of shared memory, each loaded into
// registers while the one before it is used: 41 -> 15 us at n = 4096 against
// loads between barriers.
#define TR_TH 256
#define TR_NC 16
template <class C2>
struct trsm_sh {
  C2 X[LU_OB][TR_NC + 1];
  C2 L[2][LU_W][LU_W + 1];
  C2 Y[LU_W][TR_NC + 1];
};
template <class C2>
__global__ void __launch_bounds__(TR_TH) k_lu_trsm(C2 *A, long lda, int K, int ob, int cbeg, int cend, const C2 *u) {
  extern __shared__ __align__(16) unsigned char tr_raw[];
  trsm_sh<C2> &S = *reinterpret_cast<trsm_sh<C2> *>(tr_raw);
  const int t = threadIdx.x;
  const int c0 = cbeg + blockIdx.x * TR_NC;
  const int nbk = ob / LU_W;
  constexpr int PF = LU_W * LU_W / TR_TH;
  C2 pf[PF];
  // block (ib, jb) of L11, or the inverse of diagonal block ib (jb = ib)
  auto fetch = [&](int ib, int jb) {
#pragma unroll
    for (int h = 0; h < PF; ++h) {
      const int e = t + h * TR_TH, r = e / LU_W, c = e % LU_W;
      pf[h] = jb < ib ? A[(size_t)(K + ib * LU_W + r) * lda + K + jb * LU_W + c]
                      : __ldcg(u + U_LINV + lu_slot(K + ib * LU_W) * (LU_W * LU_W) + e);
    }
  };
  fetch(0, 0);
#pragma unroll
  for (int e = t; e < LU_OB * TR_NC; e += TR_TH) {
    const int r = e / TR_NC, c = e % TR_NC;
    S.X[r][c] = (r < ob && c0 + c < cend) ? A[(size_t)(K + r) * lda + c0 + c] : czero<C2>();
  }
  const int i = t >> 3, cq = t & 7;  // row i of a block row, columns cq, cq + 8
  int buf = 0;
  for (int ib = 0; ib < nbk; ++ib) {
    C2 acc[2];
    for (int jb = 0; jb <= ib; ++jb) {
#pragma unroll
      for (int h = 0; h < PF; ++h) {
        const int e = t + h * TR_TH;
        S.L[buf][e / LU_W][e % LU_W] = pf[h];
      }
      if (jb < ib) fetch(ib, jb + 1);
      else if (ib + 1 < nbk) fetch(ib + 1, 0);
      if (jb == 0) {
        if (ib == 0) __syncthreads();  // X is in
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[j] = S.X[ib * LU_W + i][cq + 8 * j];
      }
      if (jb == ib)
#pragma unroll
        for (int j = 0; j < 2; ++j) S.Y[i][cq + 8 * j] = acc[j];
      __syncthreads();  // L (and X of the blocks above, Y) are in; the other buffer is free
      if (jb < ib) {
#pragma unroll 8
        for (int l = 0; l < LU_W; ++l) {
          const C2 lv = S.L[buf][i][l];
#pragma unroll
          for (int j = 0; j < 2; ++j) acc[j] = cfms(lv, S.X[jb * LU_W + l][cq + 8 * j], acc[j]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[j] = czero<C2>();
#pragma unroll 8
        for (int l = 0; l < LU_W; ++l) {
          const C2 lv = S.L[buf][i][l];
#pragma unroll
          for (int j = 0; j < 2; ++j) acc[j] = cfma(lv, S.Y[l][cq + 8 * j], acc[j]);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) S.X[ib * LU_W + i][cq + 8 * j] = acc[j];
      }
      buf ^= 1;
    }
  }
  __syncthreads();
  for (int e = t; e < ob * TR_NC; e += TR_TH) {
    const int r = e / TR_NC, c = e % TR_NC;
    if (c0 + c < cend) A[(size_t)(K + r) * lda + c0 + c] = S.X[r][c];
  }
}

// R = B - A X in FP64 (refinement residual): A row-major n x n, X, B, R
// column-major n x NR; one warp per row
template <int NR>
__global__ void __launch_bounds__(256) k_resid_z(const double2 *A, int n, const double2 *X, const double2 *B,
                                                 double2 *R) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  double2 acc[NR];
#pragma unroll
  for (int q = 0; q < NR; ++q) acc[q] = cz();
  const double2 *a = A + (size_t)row * n;
  for (int col = lane; col < n; col += 32) {
    const double2 av = a[col];
#pragma unroll
    for (int q = 0; q < NR; ++q) acc[q] = cfma(av, X[(size_t)q * n + col], acc[q]);
  }
#pragma unroll
  for (int q = 0; q < NR; ++q)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      acc[q].x += __shfl_down_sync(FULL, acc[q].x, o);
      acc[q].y += __shfl_down_sync(FULL, acc[q].y, o);
    }
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      const double2 b = B[(size_t)q * n + row];
      R[(size_t)q * n + row] = make_double2(b.x - acc[q].x, b.y - acc[q].y);
    }
}

// the identity row map, and the tournament's counters at zero
__global__ void k_lu_iota(int *rowmap, int n, int *counter, int nodes) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nodes; i += gridDim.x * blockDim.x) counter[i] = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) rowmap[i] = i;
}

// ---------------------------------------------------------------- triangular solves
// Bound by a serial chain: block it of 32 unknowns needs block it - 1, so a solve
// is n / 32 hops from one SM to the next through L2 (the factor's entries stream
// in beside them).  Everything that does not need the last block's values is done
// before they arrive: with V the inverse of the diagonal block and M = V times
// the block beside it, x_it = V (rhs - sum of the others) - M x_{it-1}, and only
// the last product, one sum over four warps and one store stay on the chain.  The
// values are their own flag: out starts as all ones (no arithmetic yields that
// pattern), a reader polls the values that it needs, and a hop has no counter, no
// fence and no second round trip.  A pair of solves with three right-hand sides
// at n = 1999: 816 us with substitution in the block behind a counter, 176.
#define TS_TH 128
#define TS_WAIT_NS 1000000000ull  // one second

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned ld_relaxed(const unsigned *p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ double2 ts_load(const double2 *p) {
  double2 v;
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float2 ts_load(const float2 *p) {
  float2 v;
  asm volatile("ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool ts_unset(double2 v) {
  return __double_as_longlong(v.x) == -1ll || __double_as_longlong(v.y) == -1ll;
}
__device__ __forceinline__ bool ts_unset(float2 v) { return __float_as_int(v.x) == -1 || __float_as_int(v.y) == -1; }
// a value with the reserved pattern (a NaN handed in) is stored as another NaN
__device__ __forceinline__ void ts_store(double2 *p, double2 v) {
  if (__double_as_longlong(v.x) == -1ll) v.x = __longlong_as_double(0x7ff8000000000000ll);
  if (__double_as_longlong(v.y) == -1ll) v.y = __longlong_as_double(0x7ff8000000000000ll);
  asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void ts_store(float2 *p, float2 v) {
  if (__float_as_int(v.x) == -1) v.x = __int_as_float(0x7fc00000);
  if (__float_as_int(v.y) == -1) v.y = __int_as_float(0x7fc00000);
  asm volatile("st.relaxed.gpu.global.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(v.x), "f"(v.y) : "memory");
}
// The warp's eight unknowns from c0 on, into sx[c][q], once they are written (zero
// beyond n).  After one second a wait gives up with BEM_LU_ST_WAIT set, and once
// any wait has given up the others return at their next look.
template <class C2, int NR>
__device__ __forceinline__ void ts_get(const C2 *out, int n, int c0, bool next, C2 *sx, unsigned *status) {
  const int lane = threadIdx.x & 31, c = lane & 7, q = lane >> 3;
  const bool need = q < NR && c0 + c < n;
  const C2 *p = out + (need ? (size_t)q * n + c0 + c : 0);
  C2 v = czero<C2>();
  bool ok = !need;
  unsigned long long t0 = 0;
  for (unsigned it = 1;; ++it) {
    if (!ok) {
      const C2 x = ts_load(p);
      if (!ts_unset(x)) {
        v = x;
        ok = true;
      }
    }
    if (__all_sync(FULL, ok)) break;
    if (it == 1) t0 = gtimer();
    if ((it & 255) == 0 &&
        __any_sync(FULL, gtimer() - t0 > TS_WAIT_NS || (ld_relaxed(status) & BEM_LU_ST_WAIT) != 0)) {
      if (lane == 0) atomicOr(status, BEM_LU_ST_WAIT);
      break;
    }
    if (!next) __nanosleep(100);  // leave the line to the block that is next
  }
  __syncwarp();
  if (q < NR) sx[c * NR + q] = v;
  __syncwarp();
}

// lower = 1: out = L^-1 (P in), in read through rowmap (unit lower L);
// lower = 0: out = U^-1 in.  in / out are n x NR column-major, out all ones (bits)
// before.  The 32-row blocks go in dependency order (top down for L, bottom up for
// U): the block of position it needs those of positions 0 .. it - 1.  All blocks
// are resident, or take their positions in order.
template <class C2, int NR>
__global__ void __launch_bounds__(TS_TH) k_lu_trsv(const C2 *LU, long lda, int n, const int *rowmap, const C2 *in,
                                                   C2 *out, int lower, unsigned *status) {
  __shared__ C2 sd[32][33], sv[32][33];
  __shared__ C2 sx[4][8 * NR];
  // once M is formed, V's place holds the four warps' sums
  C2 (*sacc)[32][NR] = reinterpret_cast<C2 (*)[32][NR]>(&sv[0][0]);
  C2 (*sout)[32][NR] = sacc + 4;
  const int nb = (n + 31) / 32;
  const int t = threadIdx.x, r = t & 31, s = t >> 5;
  for (int it = blockIdx.x; it < nb; it += gridDim.x) {
    const int b = lower ? it : nb - 1 - it;
    const int r0 = b * 32, rows = min(32, n - r0);
    const int row = r0 + r;
    // V: a warp inverts onto eight columns, a lane per row
    for (int e = t; e < 32 * 32; e += TS_TH) {
      const int i = e >> 5, j = e & 31;
      sd[i][j] = (i < rows && j < rows) ? LU[(size_t)(r0 + i) * lda + r0 + j] : (i == j ? cone<C2>() : czero<C2>());
    }
    __syncthreads();
    C2 inv[8], m[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      inv[c] = r == 8 * s + c ? cone<C2>() : czero<C2>();
      m[c] = czero<C2>();
    }
    const C2 d = lower ? cone<C2>() : crcp(sd[r][r]);
#pragma unroll 2
    for (int kk = 0; kk < 32; ++kk) {
      const int k = lower ? kk : 31 - kk;
      const C2 f = sd[r][k];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (!lower && r == k) inv[c] = cmul(inv[c], d);
        const C2 w = cx<C2>::mk(__shfl_sync(FULL, inv[c].x, k), __shfl_sync(FULL, inv[c].y, k));
        if (lower ? r > k : r < k) inv[c] = cfms(f, w, inv[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) sv[r][8 * s + c] = inv[c];
    __syncthreads();
    const int jl = (lower ? it - 1 : nb - it) * 32;  // the last dependency's columns
    if (it > 0) {  // M = V times the block beside
      for (int e = t; e < 32 * 32; e += TS_TH) {
        const int i = e >> 5, j = e & 31;
        sd[i][j] = (i < rows && jl + j < n) ? LU[(size_t)(r0 + i) * lda + jl + j] : czero<C2>();
      }
      __syncthreads();
#pragma unroll 4
      for (int j = 0; j < 32; ++j) {
        const C2 f = sv[r][j];
#pragma unroll
        for (int c = 0; c < 8; ++c) m[c] = cfma(f, sd[j][8 * s + c], m[c]);
      }
    }
    __syncthreads();
    C2 acc[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) acc[q] = czero<C2>();
    if (s == 0 && r < rows) {
      const int src = lower ? rowmap[row] : row;
#pragma unroll
      for (int q = 0; q < NR; ++q) acc[q] = in[(size_t)q * n + src];
    }
    // dependency k is the block of position k: rows/columns jb * 32 ..
    // jb * 32 + 31 with jb = k (lower) or nb - 1 - k (upper).  The factor's
    // entries do not depend on the other blocks, so dependency k + 1's eight
    // are loaded before the wait for dependency k.
    const C2 *arow = LU + (size_t)(r < rows ? row : r0) * lda;
    C2 ac[8], an[8];
    {
      const int jb = lower ? 0 : nb - 1;
#pragma unroll
      for (int cc = 0; cc < 8; ++cc) {
        const int col = jb * 32 + s * 8 + cc;
        ac[cc] = (it > 1 && r < rows && col < n) ? arow[col] : czero<C2>();
      }
    }
    for (int k = 0; k + 1 < it; ++k) {
      const int jb = lower ? k : nb - 1 - k, jn = lower ? k + 1 : nb - 2 - k;
#pragma unroll
      for (int cc = 0; cc < 8; ++cc) {
        const int col = jn * 32 + s * 8 + cc;
        an[cc] = (k + 2 < it && r < rows && col < n) ? arow[col] : czero<C2>();
      }
      ts_get<C2, NR>(out, n, jb * 32 + s * 8, k + 3 >= it, sx[s], status);
#pragma unroll
      for (int cc = 0; cc < 8; ++cc) {
#pragma unroll
        for (int q = 0; q < NR; ++q) acc[q] = cfms(ac[cc], sx[s][cc * NR + q], acc[q]);
        ac[cc] = an[cc];
      }
    }
#pragma unroll
    for (int q = 0; q < NR; ++q) sacc[s][r][q] = acc[q];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NR; ++q) acc[q] = czero<C2>();
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        C2 x = sacc[0][8 * s + c][q];
#pragma unroll
        for (int u = 1; u < 4; ++u) x = cx<C2>::mk(x.x + sacc[u][8 * s + c][q].x, x.y + sacc[u][8 * s + c][q].y);
        acc[q] = cfma(inv[c], x, acc[q]);
      }
    if (it > 0) {
      ts_get<C2, NR>(out, n, jl + s * 8, true, sx[s], status);
#pragma unroll
      for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int q = 0; q < NR; ++q) acc[q] = cfms(m[c], sx[s][c * NR + q], acc[q]);
    }
#pragma unroll
    for (int q = 0; q < NR; ++q) sout[s][r][q] = acc[q];
    __syncthreads();
    if (s < NR && r < rows) {
      C2 x = sout[0][r][s];
#pragma unroll
      for (int u = 1; u < 4; ++u) x = cx<C2>::mk(x.x + sout[u][r][s].x, x.y + sout[u][r][s].y);
      ts_store(out + (size_t)s * n + row, x);
    }
  }
}

// ---------------------------------------------------------------- host side
#define CKL(call, what)                                                                     \
  do {                                                                                     \
    cudaError_t _e = (call);                                                               \
    if (_e != cudaSuccess) {                                                               \
      snprintf(w->err, sizeof(w->err), "%s: %s", what, cudaGetErrorString(_e));            \
      return -1;                                                                           \
    }                                                                                      \
  } while (0)

extern "C" int bem_lu_init(bem_lu *w, int device) {
  CKL(cudaDeviceGetAttribute(&w->sms, cudaDevAttrMultiProcessorCount, device), "SM count");
  CKL(cudaFuncSetAttribute(k_lu_panel<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(panel_sh<double2>)),
      "panel smem");
  CKL(cudaFuncSetAttribute(k_lu_panel<float2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(panel_sh<float2>)),
      "panel smem");
  CKL(cudaFuncSetAttribute(k_lu_update, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)UP_SMEM), "update smem");
  CKL(cudaFuncSetAttribute(k_lu_trsm<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(trsm_sh<double2>)),
      "U12 smem");
  CKL(cudaFuncSetAttribute(k_lu_trsm<float2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(trsm_sh<float2>)),
      "U12 smem");
  int per_sm = 0;
  CKL(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_lu_trsv<double2, 4>, TS_TH, 0), "solve occupancy");
  w->coop_blocks = per_sm * w->sms;
  if (w->coop_blocks <= 0) {
    snprintf(w->err, sizeof(w->err), "triangular solve: no resident block");
    return -1;
  }
  // the panels' blocks (on hi) go before those of the update that runs beside them
  int lo = 0, hi = 0;
  CKL(cudaDeviceGetStreamPriorityRange(&lo, &hi), "LU streams");
  CKL(cudaStreamCreateWithPriority(&w->side, cudaStreamNonBlocking, lo), "LU side stream");
  CKL(cudaStreamCreateWithPriority(&w->hi, cudaStreamNonBlocking, hi), "LU streams");
  CKL(cudaEventCreateWithFlags(&w->ev_fork, cudaEventDisableTiming), "LU events");
  CKL(cudaEventCreateWithFlags(&w->ev_join, cudaEventDisableTiming), "LU events");
  CKL(cudaEventCreateWithFlags(&w->ev_st, cudaEventDisableTiming), "LU events");
  CKL(cudaMalloc(&w->piv, PV_INTS * sizeof(int)), "LU scratch");
  CKL(cudaMalloc(&w->u11, U_COUNT * sizeof(double2)), "LU scratch");
  CKL(cudaMalloc(&w->status, sizeof(unsigned)), "LU status");
  CKL(cudaMemset(w->status, 0, sizeof(unsigned)), "LU status");
  return 0;
}

static void drop_graph(bem_lu *w) {
  if (w->gexec) cudaGraphExecDestroy(w->gexec);
  if (w->graph) cudaGraphDestroy(w->graph);
  w->gexec = nullptr;
  w->graph = nullptr;
  w->g_A = nullptr;
}

extern "C" void bem_lu_free(bem_lu *w) {
  drop_graph(w);
  cudaFree(w->rowmap);
  cudaFree(w->tree);
  cudaFree(w->piv);
  cudaFree(w->u11);
  cudaFree(w->status);
  cudaFree(w->y);
  if (w->ev_fork) cudaEventDestroy(w->ev_fork);
  if (w->ev_join) cudaEventDestroy(w->ev_join);
  if (w->ev_st) cudaEventDestroy(w->ev_st);
  if (w->side) cudaStreamDestroy(w->side);
  if (w->hi) cudaStreamDestroy(w->hi);
  *w = bem_lu();
}

static int grow_bytes(bem_lu *w, void **p, size_t *cap, size_t bytes, const char *what) {
  if (*cap >= bytes) return 0;
  if (*p) cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  CKL(cudaMalloc(p, bytes), what);
  *cap = bytes;
  return 0;
}

// C = A[r0:n, c0:cend) -= A[r0:n, kk:kk+kw) A[kk:kk+kw, c0:cend)
static void launch_update(double2 *A, int n, int kk, int kw, int r0, int c0, int cend, cudaStream_t st) {
  const dim3 grid((cend - c0 + UP_BN - 1) / UP_BN, (n - r0 + UP_BM - 1) / UP_BM);
  k_lu_update<<<grid, UP_TH, UP_SMEM, st>>>(A, n, n, kk, kw, r0, c0, cend);
}
static void launch_update(float2 *A, int n, int kk, int kw, int r0, int c0, int cend, cudaStream_t st) {
  const dim3 grid((cend - c0 + UP_BN - 1) / UP_BN, (n - r0 + UP_BM - 1) / UP_BM);
  k_lu_update_c32<<<grid, UF_TH, 0, st>>>(A, n, n, kk, kw, r0, c0, cend);
}

// the same on a few panels' columns [c0, cend), kw a multiple of 32
static void launch_strip(double2 *A, int n, int kk, int kw, int r0, int c0, int cend, cudaStream_t st) {
  k_lu_strip<<<dim3((n - r0 + SP_B - 1) / SP_B, (cend - c0 + SP_B - 1) / SP_B), SP_TH, 0, st>>>(A, n, n, kk, kw, r0, c0, cend);
}
static void launch_strip(float2 *A, int n, int kk, int kw, int r0, int c0, int cend, cudaStream_t st) {
  k_lu_strip_c32<<<dim3((n - r0 + SP_B - 1) / SP_B, (cend - c0 + SP_B - 1) / SP_B), SP_TH, 0, st>>>(A, n, n, kk, kw, r0, c0, cend);
}

// an outer block's update right of the next block's columns, for a complex FP32
// factorisation on the tensor cores when the LU has them (returns 1 when
// launched): its first column tile (as wide as an outer block), or the others
static int tc_update(bem_lu *w, double2 *, int, int, bool, cudaStream_t) { (void)w; return 0; }
static int tc_update(bem_lu *w, float2 *A, int n, int K, bool first, cudaStream_t st) {
  if (!w->tc || !w->tc->ready) return 0;
  bem_tc_launch(w->tc, A, n, n, K, first, w->status, st);
  return 1;
}

// nodes of the tournament over n rows
static int lu_nodes(int n) {
  int nn = (n + LU_TH - 1) / LU_TH, total = nn;
  while (nn > 1) {
    nn = (nn + 7) / 8;
    total += nn;
  }
  return total;
}

// One outer block (n <= one_block_max): the launches in order, captured into a
// graph whose replays count them.  Look-ahead: a panel's update is split into
// the next panel's 32 columns (on st, before the next panel) and the rest (on
// the side stream, beside the next panel); the next row moves wait for the rest.
template <class C2>
static int factor_one(bem_lu *w, C2 *A, int n, cudaStream_t st) {
  const int nodes = lu_nodes(n);
  k_lu_iota<<<(n + 255) / 256, 256, 0, st>>>(w->rowmap, n, w->tree + (size_t)nodes * (1 + LU_W), nodes);
  bool pending = false;  // update work on the side stream not yet joined
  for (int k = 0; k < n; k += LU_W) {
    const int wd = n - k < LU_W ? n - k : LU_W;
    const int r0 = k + wd;
    k_lu_panel<C2><<<(n - k + LU_TH - 1) / LU_TH, LU_TH, sizeof(panel_sh<C2>), st>>>(
        A, n, n, k, w->piv, w->tree, nodes, (C2 *)w->u11, w->status);
    if (pending) CKL(cudaStreamWaitEvent(st, w->ev_join, 0), "LU join");
    pending = false;
    const int nL = (n - r0 + AP_ROWS - 1) / AP_ROWS;
    const int nC = (k + AP_COLS - 1) / AP_COLS + (n - r0 + AP_COLS - 1) / AP_COLS;
    k_lu_apply<C2><<<nL + nC + 1, AP_TH, 0, st>>>(A, n, n, k, 0, n, w->piv, (const C2 *)w->u11, w->rowmap, w->status);
    if (r0 < n) {  // wd = 32: only the last panel is narrower
      const int nxt = n - r0 < LU_W ? n : r0 + LU_W;
      launch_strip(A, n, k, LU_W, r0, r0, nxt, st);
      if (nxt < n) {
        CKL(cudaEventRecord(w->ev_fork, st), "LU fork");
        CKL(cudaStreamWaitEvent(w->side, w->ev_fork, 0), "LU fork");
        launch_update(A, n, k, wd, r0, nxt, n, w->side);
        CKL(cudaEventRecord(w->ev_join, w->side), "LU join");
        pending = true;
      }
    }
  }
  CKL(cudaGetLastError(), "LU launch");
  return 0;
}

// Outer blocks of LU_OB columns, two lanes.  hi (high priority): a block's panels,
// which update only the rest of their block, and then the same block's row
// moves, U12 and update on the next block's columns alone, so that the next
// panels can go on.  lo: the block's row moves on all other columns, U12 and the
// rank-LU_OB update right of the next block, its first LU_OB columns ahead of the
// rest because hi needs them one block later.  hi runs up to a block ahead: the
// panels, bound by latency (a half of the time at n = 4096 when they run by
// themselves), hide behind the updates.  Launched on the streams, not as a
// graph: a graph's launches do not keep the lanes' priorities.
template <class C2>
static int factor_blocks(bem_lu *w, C2 *A, int n, cudaStream_t st) {
  const int nodes = lu_nodes(n);
  cudaStream_t hi = w->hi, lo = w->side;
  unsigned long long count = 1;
  CKL(cudaEventRecord(w->ev_st, st), "LU start");
  CKL(cudaStreamWaitEvent(hi, w->ev_st, 0), "LU start");
  CKL(cudaStreamWaitEvent(lo, w->ev_st, 0), "LU start");
  k_lu_iota<<<(n + 255) / 256, 256, 0, hi>>>(w->rowmap, n, w->tree + (size_t)nodes * (1 + LU_W), nodes);
  const C2 *u = (const C2 *)w->u11;
  for (int K = 0; K < n; K += LU_OB) {
    const int cend = n - K < LU_OB ? n : K + LU_OB, np = (cend - K + LU_W - 1) / LU_W;
    const int c1 = n - cend < LU_OB ? n : cend + LU_OB;  // end of the next block
    const int c2 = n - c1 < LU_OB ? n : c1 + LU_OB;      // and of the one after
    for (int k = K; k < cend; k += LU_W) {
      const int r0 = n - k < LU_W ? n : k + LU_W;
      k_lu_panel<C2><<<(n - k + LU_TH - 1) / LU_TH, LU_TH, sizeof(panel_sh<C2>), hi>>>(
          A, n, n, k, w->piv, w->tree, nodes, (C2 *)w->u11, w->status);
      const int nL = (n - r0 + AP_ROWS - 1) / AP_ROWS;
      const int nC = (k - K + AP_COLS - 1) / AP_COLS + (cend - r0 + AP_COLS - 1) / AP_COLS;
      k_lu_apply<C2><<<nL + nC + 1, AP_TH, 0, hi>>>(A, n, n, k, K, cend, w->piv, u, w->rowmap, w->status);
      if (r0 < cend) launch_strip(A, n, k, LU_W, r0, r0, cend, hi);
      count += r0 < cend ? 3 : 2;
    }
    // lo's update of the next block's columns by the previous block (it also
    // ends lo's use of that block's slots, which the next block's panels take)
    if (K > 0) CKL(cudaStreamWaitEvent(hi, w->ev_join, 0), "LU join");
    CKL(cudaEventRecord(w->ev_fork, hi), "LU fork");
    CKL(cudaStreamWaitEvent(lo, w->ev_fork, 0), "LU fork");
    if (cend < n) {
      const int nc = (c1 - cend + AP_COLS - 1) / AP_COLS;
      k_lu_swap<C2><<<nc, AP_TH, 0, hi>>>(A, n, n, K, np, 0, cend, c1, w->piv);
      k_lu_trsm<C2><<<(c1 - cend + TR_NC - 1) / TR_NC, TR_TH, sizeof(trsm_sh<C2>), hi>>>(A, n, K, LU_OB, cend, c1, u);
      launch_strip(A, n, K, LU_OB, cend, cend, c1, hi);
      count += 3;
    }
    const int nsw = (K + AP_COLS - 1) / AP_COLS + (n - c1 + AP_COLS - 1) / AP_COLS;
    if (nsw > 0) {
      k_lu_swap<C2><<<nsw, AP_TH, 0, lo>>>(A, n, n, K, np, K, c1, n, w->piv);
      ++count;
    }
    if (c1 < n) {
      k_lu_trsm<C2><<<(n - c1 + TR_NC - 1) / TR_NC, TR_TH, sizeof(trsm_sh<C2>), lo>>>(A, n, K, LU_OB, c1, n, u);
      if (!tc_update(w, A, n, K, true, lo)) launch_update(A, n, K, LU_OB, cend, c1, c2, lo);
      else ++count;
      count += 2;
    }
    CKL(cudaEventRecord(w->ev_join, lo), "LU join");
    if (c2 < n) {
      if (!tc_update(w, A, n, K, false, lo)) launch_update(A, n, K, LU_OB, cend, c2, n, lo);
      ++count;
    }
  }
  CKL(cudaGetLastError(), "LU launch");
  CKL(cudaEventRecord(w->ev_join, lo), "LU end");
  CKL(cudaStreamWaitEvent(hi, w->ev_join, 0), "LU end");
  CKL(cudaEventRecord(w->ev_st, hi), "LU end");
  CKL(cudaStreamWaitEvent(st, w->ev_st, 0), "LU end");
  bem_count_launches(count);
  return 0;
}

template <class C2>
static int lu_factor(bem_lu *w, void *Av, int n, cudaStream_t st) {
  if (n <= 0) return 0;
  C2 *A = (C2 *)Av;
  // the kept graph's kernels write the row map and the tree: it goes where either
  // moves, also for a system that is factored without a graph
  const size_t need_map = (size_t)n * sizeof(int), need_tree = (size_t)lu_nodes(n) * (2 + LU_W) * sizeof(int);
  if (need_map > w->rowmap_cap || need_tree > w->tree_cap) drop_graph(w);
  if (grow_bytes(w, (void **)&w->rowmap, &w->rowmap_cap, need_map, "row map") ||
      grow_bytes(w, (void **)&w->tree, &w->tree_cap, need_tree, "tournament"))
    return -1;
  if (n > (w->one_block_max > 0 ? w->one_block_max : LU_ONE_BLOCK_N)) return factor_blocks(w, A, n, st);
  if (!(w->gexec && w->g_A == Av && w->g_n == n && w->g_fp == (int)sizeof(C2))) {
    drop_graph(w);
    CKL(cudaStreamBeginCapture(w->hi, cudaStreamCaptureModeThreadLocal), "LU capture");
    const int rc = factor_one(w, A, n, w->hi);
    cudaGraph_t g = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(w->hi, &g);
    if (rc) {
      if (g) cudaGraphDestroy(g);
      return rc;
    }
    CKL(ce, "LU capture");
    w->graph = g;
    CKL(cudaGraphInstantiate(&w->gexec, g, 0), "LU graph");
    size_t nodes = 0;
    CKL(cudaGraphGetNodes(g, nullptr, &nodes), "LU graph");
    w->g_nodes = nodes;
    w->g_A = Av;
    w->g_n = n;
    w->g_fp = (int)sizeof(C2);
  }
  CKL(cudaGraphLaunch(w->gexec, st), "LU graph launch");
  bem_count_launches(w->g_nodes);
  return 0;
}

extern "C" void bem_lu_set_one_block(bem_lu *w, int nmax) { w->one_block_max = nmax; }
extern "C" int bem_lu_factor_z(bem_lu *w, double *A, int n, cudaStream_t st) { return lu_factor<double2>(w, A, n, st); }
extern "C" int bem_lu_factor_c(bem_lu *w, float *A, int n, cudaStream_t st) { return lu_factor<float2>(w, A, n, st); }

template <class C2, int NR>
static int launch_trsv(bem_lu *w, const C2 *LU, int n, const C2 *in, C2 *out, int lower, cudaStream_t st) {
  const int nb = (n + 31) / 32;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nb < w->coop_blocks ? nb : w->coop_blocks);
  cfg.blockDim = dim3(TS_TH);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  CKL(cudaMemsetAsync(out, 0xff, (size_t)n * NR * sizeof(C2), st), "triangular solve");
  CKL(cudaLaunchKernelEx(&cfg, k_lu_trsv<C2, NR>, LU, (long)n, n, (const int *)w->rowmap, in, out, lower, w->status),
      "triangular solve");
  bem_count_launches(1);
  return 0;
}

template <class C2>
static int lu_solve(bem_lu *w, const void *LUv, int n, int nrhs, void *Bv, cudaStream_t st) {
  if (n <= 0) return 0;
  if (nrhs < 1 || nrhs > 4) {
    snprintf(w->err, sizeof(w->err), "LU solve: %d right-hand sides (1..4)", nrhs);
    return -1;
  }
  if (grow_bytes(w, &w->y, &w->y_cap, (size_t)n * nrhs * sizeof(C2), "solve scratch"))
    return -1;
  const C2 *LU = (const C2 *)LUv;
  C2 *B = (C2 *)Bv, *Y = (C2 *)w->y;
  int rc = 0;
  switch (nrhs) {
    case 1: rc = launch_trsv<C2, 1>(w, LU, n, B, Y, 1, st) || launch_trsv<C2, 1>(w, LU, n, Y, B, 0, st); break;
    case 2: rc = launch_trsv<C2, 2>(w, LU, n, B, Y, 1, st) || launch_trsv<C2, 2>(w, LU, n, Y, B, 0, st); break;
    case 3: rc = launch_trsv<C2, 3>(w, LU, n, B, Y, 1, st) || launch_trsv<C2, 3>(w, LU, n, Y, B, 0, st); break;
    default: rc = launch_trsv<C2, 4>(w, LU, n, B, Y, 1, st) || launch_trsv<C2, 4>(w, LU, n, Y, B, 0, st); break;
  }
  return rc ? -1 : 0;
}

extern "C" int bem_lu_solve_z(bem_lu *w, const double *LU, int n, int nrhs, double *B, cudaStream_t st) {
  return lu_solve<double2>(w, LU, n, nrhs, B, st);
}
extern "C" int bem_lu_solve_c(bem_lu *w, const float *LU, int n, int nrhs, float *B, cudaStream_t st) {
  return lu_solve<float2>(w, LU, n, nrhs, B, st);
}

extern "C" int bem_lu_resid_z(const double *A, int n, int nrhs, const double *X, const double *B, double *R,
                              cudaStream_t st) {
  const int blocks = (n + 7) / 8;
  const double2 *a = (const double2 *)A, *x = (const double2 *)X, *b = (const double2 *)B;
  double2 *r = (double2 *)R;
  switch (nrhs) {
    case 1: k_resid_z<1><<<blocks, 256, 0, st>>>(a, n, x, b, r); bem_count_launches(1); break;
    case 2: k_resid_z<2><<<blocks, 256, 0, st>>>(a, n, x, b, r); bem_count_launches(1); break;
    case 3: k_resid_z<3><<<blocks, 256, 0, st>>>(a, n, x, b, r); bem_count_launches(1); break;
    case 4: k_resid_z<4><<<blocks, 256, 0, st>>>(a, n, x, b, r); bem_count_launches(1); break;
    default: return -1;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

extern "C" unsigned bem_lu_status(bem_lu *w, cudaStream_t st) {
  unsigned s = 0;
  if (cudaMemcpyAsync(&s, w->status, sizeof(unsigned), cudaMemcpyDeviceToHost, st) != cudaSuccess) return 0xffffffffu;
  if (cudaStreamSynchronize(st) != cudaSuccess) return 0xffffffffu;
  cudaMemsetAsync(w->status, 0, sizeof(unsigned), st);
  return s;
}
