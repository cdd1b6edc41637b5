// Panel step of the blocked partial LU: the NB x NB diagonal tile is
// factored in shared memory together with the inverses of its unit-lower
// and upper triangles; the rows below and the columns right of it are then
// finished as small dense products with those inverses, which keeps every
// global access a coalesced tile load or store.  The inverses stay with the
// factors: the triangular sweeps of the solve reuse them.
#pragma once
#include "kernels.cuh"

namespace snu {

// Shared-memory tile, column-major with one element of padding per column.
constexpr int TLD = NB + 1;

// Product tiles (the operands and results of the 64 x 64 products) are
// column-major with leading dimension PLD.  FP32: 68, a multiple of 16
// bytes, so a thread reads four rows of a column, or two rows of a column,
// as one vector, and the eight columns a warp reads at once sit in
// distinct banks.  FP64: the odd stride TLD (scalar loads).
template <typename T>
__host__ __device__ constexpr int pld() {
  return sizeof(T) == 4 ? NB + 4 : TLD;
}
// Elements per tile buffer (the larger of the two layouts).
template <typename T>
__host__ __device__ constexpr int tile_elems() {
  return NB * (pld<T>() > TLD ? pld<T>() : TLD);
}


// Vector shared/global accesses of four (or two) contiguous elements.
__device__ __forceinline__ void ld4(const float* p, float (&v)[4]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
}
__device__ __forceinline__ void ld4(const double* p, double (&v)[4]) {
  const double2 t0 = *reinterpret_cast<const double2*>(p);
  const double2 t1 = *reinterpret_cast<const double2*>(p + 2);
  v[0] = t0.x, v[1] = t0.y, v[2] = t1.x, v[3] = t1.y;
}
__device__ __forceinline__ void ld2(const float* p, float& x, float& y) {
  const float2 t = *reinterpret_cast<const float2*>(p);
  x = t.x, y = t.y;
}
__device__ __forceinline__ void ld2(const double* p, double& x, double& y) {
  const double2 t = *reinterpret_cast<const double2*>(p);
  x = t.x, y = t.y;
}
// four contiguous values from global memory through L2 (16-byte aligned)
__device__ __forceinline__ void ldg4(const float* p, float (&v)[4]) {
  const float4 t = __ldcg(reinterpret_cast<const float4*>(p));
  v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
}
__device__ __forceinline__ void ldg4(const double* p, double (&v)[4]) {
  const double2 t0 = __ldcg(reinterpret_cast<const double2*>(p));
  const double2 t1 = __ldcg(reinterpret_cast<const double2*>(p + 2));
  v[0] = t0.x, v[1] = t0.y, v[2] = t1.x, v[3] = t1.y;
}
__device__ __forceinline__ void st4(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void st4(double* p, const double (&v)[4]) {
  *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
  *reinterpret_cast<double2*>(p + 2) = make_double2(v[2], v[3]);
}
template <typename T>
__device__ __forceinline__ bool aligned16(const T* p) {
  return (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

// Correctly rounded reciprocal (CUDA intrinsics): multipliers are formed as
// x * (1/p) instead of x / p, one reciprocal per pivot.
__device__ __forceinline__ float recip_rn(float x) { return __frcp_rn(x); }
__device__ __forceinline__ double recip_rn(double x) { return __drcp_rn(x); }

// The pivot reciprocal of the tile factorization, on the pivot chain.
// FP32: the hardware approximation (rcp.approx.ftz.f32) refined by one
// Newton-Raphson step in its FMA form, e = 1 - x r0, r = r0 + r0 e
// (Markstein, "IA-64 and Elementary Functions", 2000): the refined value
// is within one ulp of the correctly rounded reciprocal and nearly always
// equal to it (snu_selftest_pivot_reciprocal measures both on the GPU).  The
// .ftz form is one instruction, where the form that keeps subnormals added
// 55 cycles to every pivot; pivots whose value or reciprocal it could flush
// (outside [2^-120, 2^120]) take the same steps on a scaled pivot, in
// pivot_recip only.  FP64: the correctly rounded reciprocal.  A zero or
// infinite FP32 pivot gives NaN here; the tile factorization flags such
// pivots either way.
__device__ __forceinline__ float pivot_recip_fast(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  const float e = fmaf(-x, r, 1.f);
  return fmaf(r, e, r);
}
__device__ __forceinline__ double pivot_recip_fast(double x) { return __drcp_rn(x); }
__device__ __forceinline__ float pivot_recip(float x) {
  const float a = fabsf(x);
  const float sc = a < 0x1p-120f ? 0x1p64f : a > 0x1p120f ? 0x1p-64f : 1.f;
  return pivot_recip_fast(x * sc) * sc;
}
__device__ __forceinline__ double pivot_recip(double x) { return __drcp_rn(x); }
// The pivots pivot_recip_fast serves: lo <= |x| <= hi.
template <typename T>
__device__ __forceinline__ T pivot_lo() { return sizeof(T) == 4 ? (T)0x1p-120 : (T)4.9406564584124654e-324; }
template <typename T>
__device__ __forceinline__ T pivot_hi() { return sizeof(T) == 4 ? (T)0x1p120 : (T)1.7976931348623157e308; }

// Dynamic shared memory of k_diag_lu_inv: the tile, Linv and the
// factorization's panels.
template <typename T>
constexpr size_t diag_smem() {
  return 3 * (size_t)tile_elems<T>() * sizeof(T);
}

constexpr int SB = 4;  // pivots per step of the tile factorization

// LU without pivoting of the diagonal tile at (k0, k0) of every active front
// and the inverses of its triangles, written to INV + inv_off + step*2*NB*NB
// (Linv, then Uinv; column-major, leading dimension NB).  Leaf fronts apply
// the reference's static pivot |p| < eps -> +-eps (kernel_sparse.cu:742-749);
// separator fronts do not guard, like cusolverDnDgetrf without a pivot
// array (kernel_cuda.cu:45-73).  flags[0] counts replaced pivots, flags[1]
// records a zero or non-finite pivot.
//
// The tile is bound by the latency of its 64 dependent pivots, so the
// inverses ride along with the factorization instead of following it: the
// bordered matrix [A I; I 0] is eliminated, whose L part below A is
// I U^-1 = Uinv and whose U part right of A is L^-1 I = Linv.  At every
// pivot as many rows of A are left as rows of Uinv have begun, so both fit
// one 64 x 64 array: where a row (column) of A has become final, the row of
// Uinv (column of Linv) takes its place, starting from zero.  The array is
// eliminated SB = 4 pivots at a time, one CTA barrier per step, by two
// halves of the CTA:
//
// * the chain (warps 0, 1): thread t finishes row t of the step's four
//   columns against the 4 x 4 pivot block (x U = a; the block's own rows
//   start from the identity) and column t of its four rows (L y = a).
//   Every thread factors the block for itself, in registers, which no
//   exchange between lanes can match.  The block, row and column of the
//   next step come from shared memory without the current step's rank-4
//   update, which the thread applies itself, so the chain never waits for
//   the rest of the array.
// * the update (warps 4-7): holds the array in registers, an 8 x 4 patch per
//   thread; applies each step's rank-4 update and publishes the columns and
//   rows of the step after next.
// * warps 2 and 3 collect the finished rows and columns.
//
// (Shared memory serves 128 requested bytes a cycle, broadcasts included,
// so every operand that several threads share is requested by as few of
// them as possible: a chain of four warps beside update warps that also
// collected took 1150 cycles a step where this takes 780.)  A full tile on
// one SM takes 16.3 thousand cycles in FP32 and 28.4 in FP64, where the
// factorization by 16 x 16 sub-blocks with the inverses joined afterwards
// took 21.5 and 44.7.
//
// Finished rows of Uinv leave by whole 128-byte lines at every step; the
// tile and Linv, whose columns a step finishes four elements of, are
// collected in shared memory: Linv is stored at the end, the tile by the
// caller.  A pivot costs the chain its reciprocal and two dependent
// operations; pivots that need the
// guard, the singularity test or a scaled reciprocal send the step through
// a second pass.  A tile smaller than NB is padded with the identity, which
// leaves its factors and inverses unchanged; blocks of padding are skipped.

// Slot of row (or column) r in the 64 x 4 panels: r = 4 t + a is at
// 18 a + t, so the rows of a fixed a and consecutive t and consecutive
// rows are both in distinct banks as 16-byte vectors.
__device__ __forceinline__ int sb_slot(int r) { return (r & 3) * 18 + (r >> 2); }
constexpr int SB_SLOTS = 72;

// A 64 x 4 panel: 16-byte vectors (FP64: two planes of them).
template <typename T>
struct SbPanel {
  static constexpr int PL = sizeof(T) / 4;  // vectors per row
  __align__(16) T v[PL][SB_SLOTS][4 / PL];
  __device__ __forceinline__ void get(int slot, T (&x)[SB]) const {
    if constexpr (PL == 1) {
      ld4(v[0][slot], x);
    } else {
      ld2(v[0][slot], x[0], x[1]);
      ld2(v[1][slot], x[2], x[3]);
    }
  }
  __device__ __forceinline__ void put(int slot, T x0, T x1, T x2, T x3) {
    if constexpr (PL == 1) {
      *reinterpret_cast<float4*>(v[0][slot]) = make_float4(x0, x1, x2, x3);
    } else {
      *reinterpret_cast<double2*>(v[0][slot]) = make_double2(x0, x1);
      *reinterpret_cast<double2*>(v[1][slot]) = make_double2(x2, x3);
    }
  }
};

// (the eight panels fit one tile buffer)
static_assert(8 * sizeof(SbPanel<float>) <= tile_elems<float>() * sizeof(float) &&
              8 * sizeof(SbPanel<double>) <= tile_elems<double>() * sizeof(double),
              "panels exceed a tile buffer");

__device__ __forceinline__ void sb_barrier() {  // all 256 threads
  asm volatile("bar.sync 1, 256;" ::: "memory");
}

// Four contiguous elements of a column of a shared tile.
template <typename T>
__device__ __forceinline__ void tile_st4(T* p, const T (&w)[4]) {
  if constexpr (pld<T>() % 4 == 0) {
    st4(p, w);
  } else {
#pragma unroll
    for (int k = 0; k < 4; k++) p[k] = w[k];
  }
}
template <typename T>
__device__ __forceinline__ void tile_ld4(const T* p, T (&w)[4]) {
  if constexpr (pld<T>() % 4 == 0) {
    ld4(p, w);
  } else {
#pragma unroll
    for (int k = 0; k < 4; k++) w[k] = p[k];
  }
}

// The tile factorization of one front by the whole CTA (256 threads).  D,
// XL: shared tiles (leading dimension PLD), scratch: eight panels in shared
// memory (16-byte aligned).  On return D holds the factored tile and XL
// Linv; both inverses are in INV; the caller stores the tile to the front
// (it is off the chain: no other task reads it here).  pre: D
// already holds the tile (entries past the tile's pivots are ignored),
// instead of loading it from the front.
template <typename T>
__device__ __forceinline__ void diag_tile(const FrontDev& f,
                                          T* __restrict__ F,
                                          T* __restrict__ INV, int k0,
                                          int step, double eps, int* flags,
                                          T* D, T* XL, SbPanel<T>* scratch,
                                          bool pre = false) {
  constexpr int P = pld<T>();
  // two buffers each: the columns (rawr, by rows) and rows (rawc, by
  // columns) of a step, one update short, and the finished ones
  SbPanel<T>*rawr = scratch, *rawc = scratch + 2, *finr = scratch + 4,
  *finc = scratch + 6;
  const int kb = min(NB, f.p - k0);
  const int tid = threadIdx.x;
  const int nsb = (kb + SB - 1) / SB;
  const int64_t ld = f.ld;
  T* base = F + f.off + k0 + k0 * ld;
  T* inv = INV + f.inv_off + (int64_t)step * 2 * NB * NB;
  const bool vec = kb == NB && aligned16(base) && (f.ld & 3) == 0;
  if (tid < NB) {
    // ------------------------------------------------------------ chain
    const int i = tid, slot = sb_slot(i);  // the thread's row and column
    const T teps = (T)eps, rteps = recip_rn(teps);
    const bool guard = f.guard != 0;
    const T lo = guard ? max(teps, pivot_lo<T>()) : pivot_lo<T>();
    int nguard = 0;
    bool bad = false;
    T x[SB], y[SB];
#pragma unroll
    for (int k = 0; k < SB; k++) x[k] = y[k] = (T)0;
    sb_barrier();
    for (int s = 0; s < nsb; s++) {
      const int par = s & 1, s0 = SB * s;
      // the pivot block with the previous step's update.  FP32: every lane
      // forms all of it (gathering it as below costs 0.7 thousand cycles a
      // tile).  FP64, where that is 64 multiply-adds at a sixteenth of a warp
      // each: lane 4 a + c (and its copy 16 up) forms element (a, c) and all
      // lanes gather the sixteen (28.4 against 30.1 thousand cycles a tile)
      T d[SB][SB], r[SB], xn[SB], yn[SB], e = (T)0;
      if constexpr (sizeof(T) == 8) {
        const int ea = (tid >> 2) & 3, ec = tid & 3;
        T row[SB];
        rawr[par].get(18 * ea + s, row);
        e = ec == 0 ? row[0] : ec == 1 ? row[1] : ec == 2 ? row[2] : row[3];
        if (s > 0) {
          T fr[SB], fc[SB];
          finr[par ^ 1].get(18 * ea + s, fr);
          finc[par ^ 1].get(18 * ec + s, fc);
#pragma unroll
          for (int m = 0; m < SB; m++) e -= fr[m] * fc[m];
        }
      }
      auto block = [&]() {
        if constexpr (sizeof(T) == 8) {
#pragma unroll
          for (int a = 0; a < SB; a++)
#pragma unroll
            for (int c = 0; c < SB; c++)
              d[a][c] = __shfl_sync(0xffffffffu, e, 4 * a + c);
        } else {
#pragma unroll
          for (int k = 0; k < SB; k++) rawr[par].get(18 * k + s, d[k]);
          if (s > 0) {
            T fr[SB][SB], fc[SB][SB];
#pragma unroll
            for (int k = 0; k < SB; k++) {
              finr[par ^ 1].get(18 * k + s, fr[k]);
              finc[par ^ 1].get(18 * k + s, fc[k]);
            }
#pragma unroll
            for (int m = 0; m < SB; m++)
#pragma unroll
              for (int a = 0; a < SB; a++)
#pragma unroll
                for (int c = 0; c < SB; c++) d[a][c] -= fr[a][m] * fc[c][m];
          }
        }
      };
      block();
      rawr[par].get(slot, xn);
      rawc[par].get(slot, yn);
      bool ok = true;
#pragma unroll
      for (int k = 0; k < SB; k++) {
        const T a = fabs(d[k][k]);
        ok &= (a >= lo) & (a <= pivot_hi<T>());
        r[k] = pivot_recip_fast(d[k][k]);
#pragma unroll
        for (int a = k + 1; a < SB; a++) {
          d[a][k] *= r[k];
#pragma unroll
          for (int c = k + 1; c < SB; c++) d[a][c] -= d[a][k] * d[k][c];
        }
      }
      if (!ok) {  // (the pivots are the same in every thread)
        block();
#pragma unroll 1
        for (int k = 0; k < SB; k++) {
          // (1 / +-eps is +-rteps exactly)
          T piv = k == 0 ? d[0][0] : k == 1 ? d[1][1] : k == 2 ? d[2][2] : d[3][3];
          const bool lv = s0 + k < kb;
          const bool g = guard & lv & (piv < teps) & (piv > -teps);
          const T rk = g ? (piv < (T)0 ? -rteps : rteps) : pivot_recip(piv);
          piv = g ? (piv < (T)0 ? -teps : teps) : piv;
          nguard += g;
          bad |= lv & (!(piv != (T)0) | !isfinite(piv));
#pragma unroll
          for (int q = 0; q < SB; q++)
            if (q == k) {
              r[q] = rk;
              d[q][q] = piv;
#pragma unroll
              for (int a = q + 1; a < SB; a++) {
                d[a][q] *= rk;
#pragma unroll
                for (int c = q + 1; c < SB; c++) d[a][c] -= d[a][q] * d[q][c];
              }
            }
        }
      }
      // the thread's row and column: the previous step's update (a row or
      // column that was final in that step starts the inverse's from zero)
      if (s > 0) {
        const bool zero = (i >> 2) == s - 1;
#pragma unroll
        for (int k = 0; k < SB; k++) {
          xn[k] = zero ? (T)0 : xn[k];
          yn[k] = zero ? (T)0 : yn[k];
        }
#pragma unroll
        for (int k = 0; k < SB; k++) {
          T fr[SB], fc[SB];
          finr[par ^ 1].get(18 * k + s, fr);
          finc[par ^ 1].get(18 * k + s, fc);
#pragma unroll
          for (int m = 0; m < SB; m++) {
            xn[k] -= x[m] * fc[m];
            yn[k] -= fr[m] * y[m];
          }
        }
      }
      // finished against the block (the block's own: from the identity)
#pragma unroll
      for (int k = 0; k < SB; k++) {
        x[k] = (i >> 2) == s ? ((i & 3) == k ? (T)1 : (T)0) : xn[k];
        y[k] = (i >> 2) == s ? ((i & 3) == k ? (T)1 : (T)0) : yn[k];
      }
#pragma unroll
      for (int k = 0; k < SB; k++) {
        x[k] *= r[k];
#pragma unroll
        for (int c = k + 1; c < SB; c++) {
          x[c] -= x[k] * d[k][c];
          y[c] -= d[c][k] * y[k];
        }
      }
      finr[par].put(slot, x[0], x[1], x[2], x[3]);
      finc[par].put(slot, y[0], y[1], y[2], y[3]);
      if (tid == 0) {
#pragma unroll
        for (int c = 0; c < SB; c++) {
          const T w[4] = {d[0][c], d[1][c], d[2][c], d[3][c]};
          tile_st4(D + s0 + (s0 + c) * P, w);
        }
      }
      sb_barrier();
    }
    if (tid == 0) {
      if (nguard) atomicAdd(flags, nguard);
      if (bad) flags[1] = 1;
    }
  } else if (tid < 2 * NB) {
    // ---------------------------------------------------------- collect
    const int i = tid - NB;  // the row and the column
    sb_barrier();
    for (int s = 0; s < nsb; s++) {
      const int par = s & 1, s0 = SB * s;
      sb_barrier();
      T w[SB];
      finr[par].get(sb_slot(i), w);
      // a row of Uinv, or of the tile's L below the block
      const bool done = i < s0 + SB;
#pragma unroll
      for (int k = 0; k < SB; k++) {
        if (!done) D[i + (s0 + k) * P] = w[k];
        inv[NB * NB + i + (s0 + k) * NB] = done ? w[k] : (T)0;
      }
      finc[par].get(sb_slot(i), w);
      if (!done) {  // a column of the tile's U right of the block
        tile_st4(D + s0 + i * P, w);
#pragma unroll
        for (int k = 0; k < SB; k++) w[k] = (T)0;
      }
      tile_st4(XL + s0 + i * P, w);  // Linv, zero above the diagonal
    }
    // identity padding of the inverses past the tile's blocks
    for (int j = SB * nsb; j < NB; j++) {
      const T id = i == j ? (T)1 : (T)0;
      XL[j + i * P] = id;
      inv[NB * NB + i + j * NB] = id;
    }
  } else {
    // ----------------------------------------------------------- update
    // rows 4 tx + a and 32 + 4 tx + a, columns 4 ty + c (a, c < 4)
    const int u = tid - 2 * NB, tx = u & 7, ty = u >> 3;
    T acc[8][4];
    if (kb == NB && (pre || vec)) {
      T v[2][4][4];
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
          if (pre)
            tile_ld4(D + 32 * h + 4 * tx + (4 * ty + c) * P, v[h][c]);
          else
            ldg4(base + 32 * h + 4 * tx + (4 * ty + c) * ld, v[h][c]);
        }
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
          for (int c = 0; c < 4; c++) acc[4 * h + a][c] = v[h][c][a];
    } else {
#pragma unroll
      for (int a = 0; a < 8; a++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const int i = 32 * (a >> 2) + 4 * tx + (a & 3), j = 4 * ty + c;
          acc[a][c] = (i < kb && j < kb)
                          ? (pre ? D[i + j * P] : __ldcg(base + i + j * ld))
                          : (i == j ? (T)1 : (T)0);
        }
    }
    // the columns and rows of step s into the raw panels
    auto publish = [&](int s) {
      const int par = s & 1;
      if (ty == s) {
#pragma unroll
        for (int a = 0; a < 8; a++)
          rawr[par].put(18 * (a & 3) + 8 * (a >> 2) + tx, acc[a][0], acc[a][1],
                        acc[a][2], acc[a][3]);
      }
      if (tx == (s & 7)) {
        if (s < 8) {
#pragma unroll
          for (int c = 0; c < 4; c++)
            rawc[par].put(18 * c + ty, acc[0][c], acc[1][c], acc[2][c], acc[3][c]);
        } else {
#pragma unroll
          for (int c = 0; c < 4; c++)
            rawc[par].put(18 * c + ty, acc[4][c], acc[5][c], acc[6][c], acc[7][c]);
        }
      }
    };
    publish(0);
    publish(1);
    sb_barrier();
    for (int s = 0; s < nsb; s++) {
      const int par = s & 1;
      sb_barrier();
      // the inverses' rows and columns of this step start from zero
      if (ty == s) {
#pragma unroll
        for (int a = 0; a < 8; a++)
#pragma unroll
          for (int c = 0; c < 4; c++) acc[a][c] = (T)0;
      }
      if (tx == (s & 7)) {
        if (s < 8) {
#pragma unroll
          for (int a = 0; a < 4; a++)
#pragma unroll
            for (int c = 0; c < 4; c++) acc[a][c] = (T)0;
        } else {
#pragma unroll
          for (int a = 0; a < 4; a++)
#pragma unroll
            for (int c = 0; c < 4; c++) acc[4 + a][c] = (T)0;
        }
      }
      if (s + 1 < nsb) {
        T qc[4][SB];
#pragma unroll
        for (int c = 0; c < 4; c++) finc[par].get(18 * c + ty, qc[c]);
#pragma unroll
        for (int a = 0; a < 8; a++) {
          T pr[SB];
          finr[par].get(18 * (a & 3) + 8 * (a >> 2) + tx, pr);
#pragma unroll
          for (int k = 0; k < SB; k++)
#pragma unroll
            for (int c = 0; c < 4; c++) acc[a][c] -= pr[k] * qc[c][k];
        }
        if (s + 2 < nsb) publish(s + 2);
      }
    }
  }
  sb_barrier();
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int e = tid + 256 * q, i = (e & 15) * 4, j = e >> 4;
    T w[4];
    tile_ld4(XL + i + j * P, w);
    st4(inv + i + j * NB, w);
  }
}

// The nr x nc tile S (leading dimension PLD) to dst (leading dimension ld),
// by 256 threads: whole 16-byte vectors along the columns where they are
// aligned.
template <typename T>
__device__ __forceinline__ void tile_store(T* dst, int64_t ld, int nr, int nc,
                                           const T* S) {
  constexpr int P = pld<T>();
  if (nr == NB && aligned16(dst) && (ld & 3) == 0) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int e = threadIdx.x + 256 * q, i = (e & 15) * 4, j = e >> 4;
      T w[4];
      tile_ld4(S + i + j * P, w);
      if (j < nc) st4(dst + i + j * ld, w);
    }
  } else {
    for (int e = threadIdx.x; e < NB * nc; e += 256) {
      const int i = e & (NB - 1), j = e / NB;
      if (i < nr) dst[i + j * ld] = S[i + j * P];
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
    k_diag_lu_inv(const int* __restrict__ active,
                  const FrontDev* __restrict__ fr, T* __restrict__ F,
                  T* __restrict__ INV, int k0, int step, double eps,
                  int* flags) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* D = reinterpret_cast<T*>(smem_raw);
  const FrontDev f = fr[active[blockIdx.x]];
  diag_tile<T>(f, F, INV, k0, step, eps, flags, D, D + tile_elems<T>(),
               reinterpret_cast<SbPanel<T>*>(D + 2 * tile_elems<T>()));
  const int kb = min(NB, f.p - k0);
  __syncthreads();
  tile_store(F + f.off + k0 + (int64_t)k0 * f.ld, (int64_t)f.ld, kb, kb, D);
}

// Dynamic shared memory of k_panel_apply: the panel tile and the inverse.
template <typename T>
constexpr size_t apply_smem() {
  return 2 * (size_t)NB * TLD * sizeof(T);
}

// Rows below the diagonal tile: L = A Uinv (trsm right/upper/non-unit of the
// reference, kernel_cuda.cu:98-121); columns right of it: U = Linv A (trsm
// left/lower/unit, kernel_cuda.cu:74-97).  One CTA per NB rows or columns;
// each thread computes a 4 x 4 block of the NB x NB product.
template <typename T>
__global__ void __launch_bounds__(256)
    k_panel_apply(const PanelTask* __restrict__ tasks,
                  const FrontDev* __restrict__ fr, T* __restrict__ F,
                  const T* __restrict__ INV, int k0, int step) {
  extern __shared__ unsigned char smem_raw[];
  T* A = reinterpret_cast<T*>(smem_raw);
  T* X = A + NB * TLD;
  const PanelTask t = tasks[blockIdx.x];
  const FrontDev f = fr[t.front];
  const int kb = min(NB, f.p - k0), k1 = k0 + kb, dim = f.p + f.q;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int s0 = k1 + t.chunk * NB;  // first row (kind 0) or column (kind 1)
  const int cnt = min(NB, dim - s0);
  const T* inv = INV + f.inv_off + (int64_t)step * 2 * NB * NB +
                 (t.kind == 0 ? NB * NB : 0);
  for (int j = ty; j < NB; j += 16)
    for (int i = tx; i < NB; i += 16) X[i + j * TLD] = inv[i + j * NB];
  if (t.kind == 0) {
    // A(r, m) = F(s0 + r, k0 + m), r < cnt, m < kb
    T* src = F + f.off + s0 + (int64_t)k0 * f.ld;
    for (int m = ty; m < kb; m += 16)
      for (int r = tx; r < NB; r += 16)
        A[r + m * TLD] = r < cnt ? src[r + (int64_t)m * f.ld] : (T)0;
    __syncthreads();
    T acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) acc[a][b] = (T)0;
    for (int m = 0; m < kb; m++) {
      T av[4], xv[4];
#pragma unroll
      for (int a = 0; a < 4; a++) av[a] = A[tx + 16 * a + m * TLD];
#pragma unroll
      for (int b = 0; b < 4; b++) xv[b] = X[m + (ty + 16 * b) * TLD];
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) acc[a][b] += av[a] * xv[b];
    }
#pragma unroll
    for (int b = 0; b < 4; b++) {
      int c = ty + 16 * b;
      if (c >= kb) continue;
#pragma unroll
      for (int a = 0; a < 4; a++) {
        int r = tx + 16 * a;
        if (r < cnt) src[r + (int64_t)c * f.ld] = acc[a][b];
      }
    }
  } else {
    // A(m, c) = F(k0 + m, s0 + c), m < kb, c < cnt
    T* src = F + f.off + k0 + (int64_t)s0 * f.ld;
    for (int c = ty; c < NB; c += 16)
      for (int m = tx; m < NB; m += 16)
        A[m + c * TLD] = (c < cnt && m < kb) ? src[m + (int64_t)c * f.ld] : (T)0;
    __syncthreads();
    T acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) acc[a][b] = (T)0;
    for (int m = 0; m < kb; m++) {
      T xv[4], av[4];
#pragma unroll
      for (int a = 0; a < 4; a++) xv[a] = X[tx + 16 * a + m * TLD];
#pragma unroll
      for (int b = 0; b < 4; b++) av[b] = A[m + (ty + 16 * b) * TLD];
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) acc[a][b] += xv[a] * av[b];
    }
#pragma unroll
    for (int b = 0; b < 4; b++) {
      int c = ty + 16 * b;
      if (c >= cnt) continue;
#pragma unroll
      for (int a = 0; a < 4; a++) {
        int i = tx + 16 * a;
        if (i < kb) src[i + (int64_t)c * f.ld] = acc[a][b];
      }
    }
  }
}

}  // namespace snu
