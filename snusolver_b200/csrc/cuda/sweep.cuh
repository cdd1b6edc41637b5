// Triangular sweeps of the solve over the front tree (the reference's
// core_trsm / core_update_b / trsm_Lxb / gemm on b in the factorization, and
// the back solve, SnuMat_factorize.cu:258-345, kernel_sparse.cu:915-944).
//
// The vectors of a sweep are n x nrhs, column-major, with the rows in
// elimination order (a front's pivots are rows [y_off, y_off + p)): Z, the
// right-hand side that a front's products update in place, in the rows of
// whichever ancestors pivot them, and Y, the forward result.  The backward
// sweep updates Y in place and leaves the solution in Z.  yidx maps every
// front index to its row.
//
// Where updates must be added in a fixed order (bit-reproducible runs) or
// exchanged between ranks, every front has its own work vector W (dim x
// nrhs) and pivot part of Y (p x nrhs) instead, and the update vectors go
// from front to front (k_solve_ea).  SweepVec addresses both.
//
// Each level of a sweep is two launches (more with work vectors):
//
// * the pivot block (rows and columns [0, p)): one launch over (front, 128-row
//   chunk) tasks, taken from a counter (not a cooperative launch: it starts
//   while the kernel before it runs).  The chunk holding a tile's rows solves the
//   tile with the stored inverse of the diagonal tile and publishes the
//   result in Y; the other chunks of the front wait for it (bounded spin) and
//   update their rows.  Y itself is the flag: it starts as a NaN that no
//   result is stored as (SweepNan), and a waiting thread spins on the
//   elements that it needs.  The factor columns a chunk needs for a tile are
//   staged into shared memory with cp.async while it waits.
// * the off-diagonal part (L21 y for the forward sweep, U12 x_Q for the
//   backward sweep): a tall-skinny product over (front, 64-row, 256-column)
//   blocks that adds into Z, Y or W with atomics.
#pragma once
#include "kernels.cuh"

namespace snu {

constexpr int RG = 16;          // right-hand sides per register group
// columns per pass of the level-by-level sweeps: the pivot-block sweeps run
// the pass's register groups as independent task chains of one launch (a
// group's tasks after the previous group's)
constexpr int SOLVE_COLS = 64;
constexpr int DIAG_ROWS = 128;  // rows of a pivot-block chunk (= threads)
constexpr long WAVE_SPIN_LIMIT = 1L << 22;

// Dynamic shared memory of the pivot-block sweeps: two buffers (the tile
// being applied and the next one) of the staged factor columns of a chunk
// [NB][DIAG_ROWS] and a tile inverse [NB][NB].
template <typename T>
constexpr size_t sweep_smem() {
  return 2 * (size_t)(NB * DIAG_ROWS + NB * NB) * sizeof(T);
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa),
               "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}
// all but the most recently committed group
__device__ __forceinline__ void cp_async_wait_prev() {
  asm volatile("cp.async.wait_group 1;\n" ::: "memory");
}

// Spins (bounded) until *flag is set; on timeout sets *err and returns false.
// The load is an acquire at GPU scope: the caller's CTA barrier after it
// orders the CTA's reads of the published data after the flag.
__device__ __forceinline__ bool wait_flag(const int* flag, int* err) {
  for (long it = 0; it < WAVE_SPIN_LIMIT; it++) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(flag)
                 : "memory");
    if (v) return true;
    __nanosleep(64);
  }
  atomicExch(err, 1);
  return false;
}

// Sets *flag with a release at GPU scope (called by one thread after the
// CTA barrier that follows the CTA's writes of the published data, which
// the release orders before the flag).
__device__ __forceinline__ void raise_flag(int* flag) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(flag), "r"(1)
               : "memory");
}

// Stages rows [r0, r1) of factor columns [k0, k0 + kb) of front f into
// Ls[m * DIAG_ROWS + (row - rbase)] (rbase = the chunk's first row; r0 and
// rbase are multiples of the 16-byte vector).  Rows up to r1 rounded up to
// the vector stay inside the column (ld is a multiple of 4).
template <typename T>
__device__ __forceinline__ void stage_cols(T* Ls, const T* F, const FrontDev& f,
                                           int rbase, int r0, int r1, int k0,
                                           int kb) {
  constexpr int V = 16 / sizeof(T);
  const int nv = (r1 - r0 + V - 1) / V;
  if (nv <= 0) return;
  const T* src = F + f.off + r0 + (int64_t)k0 * f.ld;
  T* dst = Ls + (r0 - rbase);
  for (int e = threadIdx.x; e < kb * nv; e += blockDim.x) {
    const int m = e / nv, v = e - m * nv;
    cp_async16(dst + m * DIAG_ROWS + v * V, src + (int64_t)m * f.ld + v * V);
  }
}

template <typename T>
__device__ __forceinline__ void stage_inv(T* Xs, const T* inv) {
  constexpr int V = 16 / sizeof(T);
  for (int e = threadIdx.x; e < NB * NB / V; e += blockDim.x)
    cp_async16(Xs + e * V, inv + e * V);
}

// Programmatic dependent launch: a sweep kernel may start while the one
// before it in the stream still runs.  Until grid_wait it touches only what no
// kernel of a solve writes (task lists, fronts, factors) and its own task
// counter, zeroed before the first kernel of the pass.  The vectors are no
// __restrict__ pointers: loads from one that a kernel only reads could be
// moved before the wait.
__device__ __forceinline__ void grid_start_next() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void grid_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Where a front's rows are in the vectors of a sweep: n > 0: vectors in
// elimination order, 0: per-front work vectors and pivot parts.
struct SweepVec {
  int n;
  const int* yidx;  // row of every front index (n > 0)
  // first pivot row of front f and the distance of its columns
  __device__ __forceinline__ int64_t piv(const FrontDev& f, int nrhs) const {
    return n ? f.y_off : f.y_off * nrhs;
  }
  __device__ __forceinline__ int64_t ldp(const FrontDev& f) const {
    return n ? n : f.p;
  }
  // the same of its work vector (whose pivot rows start from the right-hand
  // side: Z with n > 0)
  __device__ __forceinline__ int64_t work(const FrontDev& f, int nrhs) const {
    return n ? f.y_off : f.w_off * nrhs;
  }
  __device__ __forceinline__ int64_t ldw(const FrontDev& f) const {
    return n ? n : f.p + f.q;
  }
};

// The NaN that marks an element of Y that is not solved yet: every bit set,
// so a buffer is marked by a memset.  A result with those bits (a NaN that
// came in with the right-hand side) is published as the usual NaN instead.
template <typename T>
struct SweepNan;
template <>
struct SweepNan<float> {
  __device__ __forceinline__ static float mark() { return __uint_as_float(0xffffffffu); }
  __device__ __forceinline__ static bool is(float v) { return __float_as_uint(v) == 0xffffffffu; }
  __device__ __forceinline__ static float load(const float* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return __uint_as_float(v);
  }
  __device__ __forceinline__ static void publish(float* p, float v) {
    const uint32_t b = is(v) ? 0x7fffffffu : __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(b) : "memory");
  }
};
template <>
struct SweepNan<double> {
  __device__ __forceinline__ static double mark() { return __longlong_as_double(-1ll); }
  __device__ __forceinline__ static bool is(double v) { return __double_as_longlong(v) == -1ll; }
  __device__ __forceinline__ static double load(const double* p) {
    long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return __longlong_as_double(v);
  }
  __device__ __forceinline__ static void publish(double* p, double v) {
    const long long b = is(v) ? 0x7fffffffffffffffll : __double_as_longlong(v);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(b) : "memory");
  }
};

// Whether another wait of the solve has already run out.  A spinning thread
// looks after every WAVE_ROUND iterations (64^3 convection-diffusion, four
// columns: a solve 3.39 ms, 3.51 with the look inside its loop), so that a
// launch in which one wait runs out ends soon after it and not a limit per
// waiting task later.
constexpr int WAVE_ROUND = 256;
__device__ __forceinline__ bool wait_failed(const int* err) {
  int e;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(e) : "l"(err) : "memory");
  return e != 0;
}

// v[q] = src[off(q)] for the q that are wanted, once published (bounded
// spin of `limit` iterations; all loads in flight together); on timeout, or
// once *err is set, sets *err and returns false: the caller's block leaves
// its kernel without handing anything on.
template <typename T, int N, typename Off>
__device__ __forceinline__ bool poll_all(const T* src, Off off, T (&v)[N],
                                         int* err, long limit = WAVE_SPIN_LIMIT) {
  bool again = true;
#pragma unroll
  for (int q = 0; q < N; q++) v[q] = SweepNan<T>::mark();
  for (long r = 0; again && r < limit; r += WAVE_ROUND) {
    if (r > 0 && wait_failed(err)) break;
    for (int it = 0; again && it < WAVE_ROUND; it++) {
      again = false;
#pragma unroll
      for (int q = 0; q < N; q++) {
        const int64_t o = off(q);
        if (o >= 0 && SweepNan<T>::is(v[q])) v[q] = SweepNan<T>::load(src + o);
      }
#pragma unroll
      for (int q = 0; q < N; q++) again |= off(q) >= 0 && SweepNan<T>::is(v[q]);
      if (again && it > 4) __nanosleep(20);
    }
  }
  if (again) atomicExch(err, 1);
  return !again;
}

// Shared memory of a pivot-block chunk beside the staging buffers: a tile's
// solution and right-hand side, [NB][R] with padded rows.
template <typename T, int R>
struct ChunkSmem {
  static constexpr int RS = R >= 8 ? R + 16 / (int)sizeof(T) : R;
  __align__(16) T ys[NB][RS];
  __align__(16) T ws[NB][RS];
  int bad;
};

// N contiguous values from shared memory, as wide as N allows (aligned to
// N values, N a power of two).
template <int N, typename T>
__device__ __forceinline__ void lds(const T* p, T (&v)[N]) {
  constexpr int V = 16 / sizeof(T);
  if constexpr (N >= V) {
#pragma unroll
    for (int q = 0; q < N; q += V) {
      const uint4 t = *reinterpret_cast<const uint4*>(p + q);
      if constexpr (sizeof(T) == 4) {
        v[q] = __uint_as_float(t.x), v[q + 1] = __uint_as_float(t.y);
        v[q + 2] = __uint_as_float(t.z), v[q + 3] = __uint_as_float(t.w);
      } else {
        v[q] = __hiloint2double(t.y, t.x), v[q + 1] = __hiloint2double(t.w, t.z);
      }
    }
  } else if constexpr (N == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = t.x, v[1] = t.y;
  } else {
    v[0] = p[0];
  }
}

// One pivot-block chunk (rows [c0, c1) of the pivots of front f, columns
// [r0, r0 + nr) of the pass) of a forward (FWD) or backward sweep, by the
// DIAG_ROWS threads of a CTA.
//   forward, tile s: y_s = Linv_s w[k0:k1]; w[r] -= L[r, k0:k1] y_s, r >= k1
//   backward, tile s (from the last): x_s = Uinv_s w[k0:k1];
//            w[r] -= U[r, k0:k1] x_s, r < k0
// init(row, r): the chunk's starting right-hand side; done(row, r, v): what
// else becomes of a solved element; Yp (columns ldy apart, column r0 first): where tiles are published and waited for.
//
// The chain of tiles is bound by latency: its hand-overs between CTAs, and
// shared-memory loads and barriers in front of few warps (one or two CTAs of
// four warps an SM).  48^3 convection-diffusion, FP32, 64 columns (8): warps
// active 6-12% (6-12), issue slots 23-44% (21-32), shared-memory wavefronts
// 20-39% (20-34) of what the SM can serve, FMA pipe 13-28% (10-16).
// So the chunk's right-hand side stays in registers, a thread holding TR rows
// x TC columns (4 x 4 at 16 columns: two vector loads for 16 multiply-adds,
// where a row per thread takes five), and a tile is handed over
// through its values alone: no fence, flag or second load.  With the
// products below, 64 columns on a 54^3 grid 20.1 -> 15.6 ms (pivot blocks
// 9.5 -> 6.5, products 5.8 -> 3.9), 13 FP64 columns on 37^3 2.44 -> 1.66 ms.
template <typename T, int R, bool FWD, bool WAIT, typename Init, typename Done>
__device__ __forceinline__ bool chunk_sweep(const FrontDev& f,
                                            const T* __restrict__ F,
                                            const T* __restrict__ INV,
                                            int chunk, int nr, T* Yp,
                                            int64_t ldy, T* Ls0, T* Xs0, ChunkSmem<T, R>& sm,
                                            Init init, Done done, int* err,
                                            long limit = WAVE_SPIN_LIMIT) {
  constexpr int V = 16 / sizeof(T), RS = ChunkSmem<T, R>::RS;
  constexpr int TC = R >= 4 ? R / 4 : 1, TR = R / TC;  // register tile
  constexpr int NG = R / TC, NT = DIAG_ROWS / NG;      // column groups, lanes
  constexpr int VW = TR < V ? TR : V, NP = TR / VW;    // row pieces of VW rows
  static_assert(NT * TR == DIAG_ROWS, "a chunk is one register tile a thread");
  const int tid = threadIdx.x, tx = tid % NT, tc = (tid / NT) * TC;
  const int c0 = chunk * DIAG_ROWS, c1 = min(f.p, c0 + DIAG_ROWS);
  const int ntiles = (f.p + NB - 1) / NB;
  // first row (in the chunk) of piece p
  auto prow = [&](int p) { return (p * NT + tx) * VW; };
  // stages tile s into buffer s & 1: the rows of this chunk it updates and,
  // for the chunk that owns it, its inverse
  auto stage = [&](int s) {
    const int b = s & 1, k0 = s * NB, kb = min(NB, f.p - k0), k1 = k0 + kb;
    const T* inv = INV + f.inv_off + (int64_t)s * 2 * NB * NB;
    if (FWD) {
      stage_cols(Ls0 + b * NB * DIAG_ROWS, F, f, c0, max(c0, k1) & ~(V - 1), c1,
                 k0, kb);
      if (k0 >= c0) stage_inv(Xs0 + b * NB * NB, inv);
    } else {
      stage_cols(Ls0 + b * NB * DIAG_ROWS, F, f, c0, c0, min(c1, k0), k0, kb);
      if (k0 < c1) stage_inv(Xs0 + b * NB * NB, inv + NB * NB);
    }
  };
  // the chunk's tiles: forward from 0 to its last, backward from the last
  // of the front to its first
  const int sA = FWD ? 0 : ntiles - 1, sB = FWD ? (c1 - 1) / NB : c0 / NB;
  const int ds = FWD ? 1 : -1;
  // two tiles are in flight: what a tile needs is requested a whole tile
  // before the chunk can use it
  stage(sA);
  cp_async_commit();
  if (sA != sB) stage(sA + ds);
  cp_async_commit();
  if (WAIT) grid_wait();  // (nothing the previous kernel writes so far)
  T w[NP][VW][TC];
#pragma unroll
  for (int p = 0; p < NP; p++)
#pragma unroll
    for (int a = 0; a < VW; a++)
#pragma unroll
      for (int c = 0; c < TC; c++) {
        const int row = c0 + prow(p) + a, r = tc + c;
        w[p][a][c] = row < c1 && r < nr ? init(row, r) : (T)0;
      }
  for (int s = sA;; s += ds) {
    const int k0 = s * NB, kb = min(NB, f.p - k0);
    const bool owner = FWD ? k0 >= c0 : k0 < c1;
    const T* Ls = Ls0 + (s & 1) * NB * DIAG_ROWS;
    const T* Xs = Xs0 + (s & 1) * NB * NB;
    T(*ys)[RS] = sm.ys;
    if (owner) {
      // the tile's right-hand side from the registers that hold it
#pragma unroll
      for (int p = 0; p < NP; p++) {
        const int lr = c0 + prow(p) - k0;  // row in the tile
        if (lr >= 0 && lr < NB)
#pragma unroll
          for (int a = 0; a < VW; a++)
#pragma unroll
            for (int c = 0; c < TC; c++)
              sm.ws[lr + a][tc + c] = lr + a < kb ? w[p][a][c] : (T)0;
      }
      cp_async_wait_prev();
      __syncthreads();
      constexpr int AR = R >= 4 ? 2 : 1;                       // rows
      constexpr int AC = (NB * R / DIAG_ROWS + AR - 1) / AR;   // x columns
      constexpr int AL = NB / AR;                              // row lanes
      const int i0 = (tid % AL) * AR, g0 = (tid / AL) * (AC > 0 ? AC : 1);
      if (g0 < R) {
        T acc[AR][AC > 0 ? AC : 1];
        constexpr int C = AC > 0 ? AC : 1;
#pragma unroll
        for (int a = 0; a < AR; a++)
#pragma unroll
          for (int c = 0; c < C; c++) acc[a][c] = (T)0;
        if constexpr (C == 1) {
          // (few columns: four partial sums shorten the chain of adds)
          T part[4][AR];
#pragma unroll
          for (int q = 0; q < 4; q++)
#pragma unroll
            for (int a = 0; a < AR; a++) part[q][a] = (T)0;
#pragma unroll 4
          for (int m = 0; m < NB; m += 4)
#pragma unroll
            for (int q = 0; q < 4; q++) {
              T xv[AR];
              lds(Xs + i0 + (m + q) * NB, xv);
              const T v = sm.ws[m + q][g0];
#pragma unroll
              for (int a = 0; a < AR; a++) part[q][a] += xv[a] * v;
            }
#pragma unroll
          for (int a = 0; a < AR; a++)
            acc[a][0] = (part[0][a] + part[1][a]) + (part[2][a] + part[3][a]);
        } else {
          // (sixteen steps' operands in flight: 64 columns on 54^3 12.4 ms
          // with four, 12.1 with sixteen)
#pragma unroll 16
          for (int m = 0; m < NB; m++) {
            T xv[AR], v[C];
            lds(Xs + i0 + m * NB, xv);
            lds(&sm.ws[m][g0], v);
#pragma unroll
            for (int a = 0; a < AR; a++)
#pragma unroll
              for (int c = 0; c < C; c++) acc[a][c] += xv[a] * v[c];
          }
        }
#pragma unroll
        for (int c = 0; c < C; c++)
#pragma unroll
          for (int a = 0; a < AR; a++) {
            const int i = i0 + a, r = g0 + c;
            const bool in = i < kb && r < nr;
            ys[i][r] = in ? acc[a][c] : (T)0;
            if (in) {
              SweepNan<T>::publish(Yp + k0 + i + r * ldy, acc[a][c]);
              done(k0 + i, r, acc[a][c]);
            }
          }
      }
      if (s == sB) break;  // nothing of the chunk is left
    } else {
      constexpr int N = (NB * R + DIAG_ROWS - 1) / DIAG_ROWS;
      T v[N];
      auto off = [&](int q) -> int64_t {
        const int e = tid + DIAG_ROWS * q, i = e % NB, r = e / NB;
        return i < kb && r < nr ? k0 + i + r * ldy : -1;
      };
      if (!poll_all<T, N>(Yp, off, v, err, limit)) sm.bad = 1;
#pragma unroll
      for (int q = 0; q < N; q++) {
        const int e = tid + DIAG_ROWS * q, i = e % NB, r = e / NB;
        if (r < R) ys[i][r] = off(q) >= 0 ? v[q] : (T)0;
      }
      cp_async_wait_prev();
    }
    __syncthreads();
    if (sm.bad) return false;
    // rows [u0, u1) of the chunk take this tile's update
    const int u0 = FWD ? max(0, k0 + NB - c0) : 0;
    const int u1 = FWD ? c1 - c0 : min(c1, k0) - c0;
    bool any = false;
#pragma unroll
    for (int p = 0; p < NP; p++) any |= prow(p) >= u0 && prow(p) < u1;
    if (any) {
      T acc[NP][VW][TC];
#pragma unroll
      for (int p = 0; p < NP; p++)
#pragma unroll
        for (int a = 0; a < VW; a++)
#pragma unroll
          for (int c = 0; c < TC; c++) acc[p][a][c] = (T)0;
#pragma unroll 16
      for (int m = 0; m < kb; m++) {
        T y[TC];
        lds(&ys[m][tc], y);
#pragma unroll
        for (int p = 0; p < NP; p++) {
          T l[VW];
          lds(Ls + m * DIAG_ROWS + prow(p), l);
#pragma unroll
          for (int a = 0; a < VW; a++)
#pragma unroll
            for (int c = 0; c < TC; c++) acc[p][a][c] += l[a] * y[c];
        }
      }
#pragma unroll
      for (int p = 0; p < NP; p++)
        if (prow(p) >= u0 && prow(p) < u1)
#pragma unroll
          for (int a = 0; a < VW; a++)
#pragma unroll
            for (int c = 0; c < TC; c++) w[p][a][c] -= acc[p][a][c];
    }
    __syncthreads();  // the tile's buffers are read
    if (FWD ? s + 2 <= sB : s - 2 >= sB) stage(s + 2 * ds);
    cp_async_commit();
  }
  return true;
}

// Forward (FWD) or backward sweep of the pivot blocks of one level.  Tasks
// are (front, chunk) with the chunks of a front in ascending (backward:
// descending) order, so every chunk waits only on tasks of lower index; the
// blocks take tasks from a counter as they come free, so tasks start in
// ascending order and the lowest unfinished one never waits on a task that is
// not running, whatever part of the grid is resident.  A chunk's right-hand side comes from W (forward Z,
// backward Y, or the work vectors) and its tiles go to Y (forward Y, backward
// Z, or the pivot parts); the backward sweep also writes the final solution
// to X in original row order.
template <typename T, int R, bool FWD>
__device__ __forceinline__ void diag_sweep_body(
    const SweepTask* __restrict__ tasks, int nbase, int ngroups,
    const FrontDev* __restrict__ fr, const T* __restrict__ F,
    const T* __restrict__ INV, SweepVec vec, int nrhs, const T* W,
    T* Y, const int* __restrict__ gidx, double* X, int ldx,
    int* next_task, int* err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Ls0 = reinterpret_cast<T*>(smem_raw);  // [2][NB][DIAG_ROWS]
  T* Xs0 = Ls0 + 2 * NB * DIAG_ROWS;         // [2][NB * NB]
  __shared__ ChunkSmem<T, R> sm;
  __shared__ int s_task;
  if (threadIdx.x == 0) sm.bad = 0;
  grid_start_next();
  for (;;) {
    // tasks start in ascending order as blocks come free
    cp_async_wait_all();
    __syncthreads();
    if (threadIdx.x == 0) s_task = atomicAdd(next_task, 1);
    __syncthreads();
    const int task = s_task;
    if (task >= nbase * ngroups) break;
    // task = group g's copy of base task task - g nbase: columns
    // [g R, g R + nr) of the pass
    const int g = task / nbase;
    const SweepTask t = tasks[task - g * nbase];
    const int r0 = g * R, nr = min(R, nrhs - r0);
    const FrontDev f = fr[t.front];
    const int64_t ldw = vec.ldw(f), ldy = vec.ldp(f);
    const T* Wf = W + vec.work(f, nrhs) + r0 * ldw;
    T* Yf = Y + vec.piv(f, nrhs) + r0 * ldy;
    const int* gi = gidx + f.idx_off;
    const bool ok = chunk_sweep<T, R, FWD, true>(
        f, F, INV, t.chunk, nr, Yf, ldy, Ls0, Xs0, sm,
        [&](int row, int r) { return __ldcg(Wf + row + r * ldw); },
        [&](int row, int r, T v) {
          if (!FWD && X) X[gi[row] + (int64_t)(r0 + r) * ldx] = (double)v;
        },
        err);
    if (!ok) break;
  }
  cp_async_wait_all();
  grid_wait();  // (also by a block without a task: the kernel's end is then
                // behind the end of the one before it)
}

template <typename T, int R>
__global__ void __launch_bounds__(DIAG_ROWS)
    k_fwd_diag(const SweepTask* __restrict__ tasks, int nbase, int ngroups,
               const FrontDev* __restrict__ fr, const T* __restrict__ F,
               const T* __restrict__ INV, SweepVec vec, int nrhs,
               const T* W, T* Y, const int* __restrict__ gidx,
               double* X, int ldx, int* next_task, int* err) {
  diag_sweep_body<T, R, true>(tasks, nbase, ngroups, fr, F, INV, vec, nrhs, W,
                              Y, gidx, X, ldx, next_task, err);
}

template <typename T, int R>
__global__ void __launch_bounds__(DIAG_ROWS)
    k_bwd_diag(const SweepTask* __restrict__ tasks, int nbase, int ngroups,
               const FrontDev* __restrict__ fr, const T* __restrict__ F,
               const T* __restrict__ INV, SweepVec vec, int nrhs,
               const T* W, T* Y, const int* __restrict__ gidx,
               double* X, int ldx, int* next_task, int* err) {
  diag_sweep_body<T, R, false>(tasks, nbase, ngroups, fr, F, INV, vec, nrhs, W,
                               Y, gidx, X, ldx, next_task, err);
}

// Backward start of a front: W[0:p] = Y (the forward result; Y is marked
// unsolved again for the backward sweep) and W[p:dim] = X[gidx] (the
// non-pivot solution, already final).
template <typename T>
__global__ void k_bwd_init(const int* __restrict__ list,
                           const FrontDev* __restrict__ fr,
                           const int* __restrict__ gidx,
                           const double* __restrict__ X, int ldx, int nrhs,
                           T* __restrict__ Y, T* __restrict__ W) {
  const FrontDev f = fr[list[blockIdx.x / SOLVE_SPLIT]];
  const int dim = f.p + f.q;
  T* w = W + f.w_off * nrhs;
  T* y = Y + f.y_off * nrhs;
  const int* g = gidx + f.idx_off;
  // one row per thread (its index once), all right-hand sides
  for (int t = (blockIdx.x % SOLVE_SPLIT) * blockDim.x + threadIdx.x; t < dim;
       t += SOLVE_SPLIT * blockDim.x) {
    if (t < f.p) {
      for (int r = 0; r < nrhs; r++) {
        w[t + (int64_t)r * dim] = y[t + (int64_t)r * f.p];
        y[t + (int64_t)r * f.p] = SweepNan<T>::mark();
      }
    } else {
      const int64_t gt = g[t];
      for (int r = 0; r < nrhs; r++)
        w[t + (int64_t)r * dim] = (T)X[gt + (int64_t)r * ldx];
    }
  }
}

constexpr int GEMV_ROWS = 64, GEMV_K = 256;

// Off-diagonal products of the sweeps, one (64-row, 256-column) block per
// CTA; the column blocks of a front add into W with atomics.  kchunk -1:
// the CTA runs over every column block itself, so each row of W has one
// writer (the bit-reproducible schedule).
//   FWD:  Z[row of p + i] -= L21[i, :] Y    (i < q, over the p pivot columns)
//   !FWD: Y[i] -= U12[i, :] Z[rows of Q]    (i < p, over the q update columns)
// With work vectors: W[p + i] -= L21[i, :] Y and W[i] -= U12[i, :] W[p:dim].
// Blocks of one task are neighbours (they share its factor entries in L2)
// and take columns [g R, g R + R) of the pass each.
//
// A lane holds two rows (so a load of the vector slice serves two rows'
// multiply-adds), a warp an eighth of the columns; UB columns of its factor
// entries are in flight at a time, the first of them before the slice is
// staged.  Bound by latency (48^3 convection-diffusion, FP32, 64 columns:
// warps active 24%, issue slots 45-52%, shared-memory wavefronts 34-39%, FMA
// pipe 26-29%; 8 columns: waiting on the factor loads).
template <typename T, int R, bool FWD>
__device__ __forceinline__ void gemv_off(const SweepTask* __restrict__ tasks,
                                         int ngroups,
                                         const FrontDev* __restrict__ fr,
                                         const T* __restrict__ F, SweepVec vec,
                                         int nrhs, T* W, T* Y) {
  grid_start_next();
  constexpr int RS = ChunkSmem<T, R>::RS;
  constexpr int KW = GEMV_K / 8;  // columns per warp
  constexpr int UB = R <= 4 ? 16 : 8;  // columns in flight (two rows each)
  // the block's slice of the source vector, then (after the products) the
  // partial sums of four warps, in one buffer
  constexpr size_t YS = sizeof(T) * GEMV_K * RS,
                   RED = sizeof(T) * 4 * GEMV_ROWS * (R + 1);
  __shared__ __align__(16) unsigned char smb[YS > RED ? YS : RED];
  T(*ys)[RS] = reinterpret_cast<T(*)[RS]>(smb);
  T(*red)[GEMV_ROWS][R + 1] = reinterpret_cast<T(*)[GEMV_ROWS][R + 1]>(smb);
  const SweepTask t = tasks[blockIdx.x / ngroups];
  const int r0 = (blockIdx.x % ngroups) * R, nr = min(R, nrhs - r0);
  const FrontDev f = fr[t.front];
  const int nrows = FWD ? f.q : f.p, nk = FWD ? f.p : f.q;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i0 = t.chunk * GEMV_ROWS + lane;  // rows i0 and i0 + 32
  const int nkb = (nk + GEMV_K - 1) / GEMV_K;
  const int kb0 = t.kchunk < 0 ? 0 : t.kchunk,
            kb1 = t.kchunk < 0 ? nkb : t.kchunk + 1;
  // source and destination vectors (columns lsrc / ldst apart; with vec.n
  // the Q rows, src backward and dst forward, go through yidx), and the
  // operand block's first element
  const int64_t lq = vec.ldw(f), lp = FWD ? vec.ldp(f) : lq;
  T* q0 = W + (vec.n ? 0 : f.w_off * nrhs + f.p) + r0 * lq;
  T* p0 = FWD || vec.n ? Y + vec.piv(f, nrhs) + r0 * lp : W + f.w_off * nrhs + r0 * lp;
  const T* src = FWD ? p0 : q0;
  T* dst = FWD ? q0 : p0;
  const int64_t lsrc = FWD ? lp : lq, ldst = FWD ? lq : lp;
  const int* qrow = vec.n ? vec.yidx + f.idx_off + f.p : nullptr;
  const T* a = FWD ? F + f.off + f.p + i0 : F + f.off + i0 + (int64_t)f.p * f.ld;
  const bool in0 = i0 < nrows, in1 = i0 + 32 < nrows;
  T acc[2][R];
#pragma unroll
  for (int r = 0; r < R; r++) acc[0][r] = acc[1][r] = (T)0;
  for (int kb = kb0; kb < kb1; kb++) {
    const int kc0 = kb * GEMV_K, kc1 = min(nk, kc0 + GEMV_K);
    const int w0 = kc0 + warp * KW;
    T av[UB][2];
    auto load = [&](int k0) {
#pragma unroll
      for (int u = 0; u < UB; u++) {
        const bool ink = k0 + u < kc1;
        av[u][0] = ink && in0 ? a[(int64_t)(k0 + u) * f.ld] : (T)0;
        av[u][1] = ink && in1 ? a[(int64_t)(k0 + u) * f.ld + 32] : (T)0;
      }
    };
    load(w0);
    if (kb > kb0)
      __syncthreads();  // the previous block's slice is read
    else
      grid_wait();
    {
      const int k = threadIdx.x;
      const bool ink = kc0 + k < kc1;
      const int64_t row = !FWD && qrow && ink ? qrow[kc0 + k] : kc0 + k;
#pragma unroll
      for (int r = 0; r < R; r++)
        ys[k][r] = ink && r < nr ? __ldcg(src + row + r * lsrc) : (T)0;
    }
    __syncthreads();
#pragma unroll 1
    for (int k0 = 0; k0 < KW; k0 += UB) {
      if (w0 + k0 >= kc1) break;
      if (k0) load(w0 + k0);
#pragma unroll
      for (int u = 0; u < UB; u++) {
        T y[R];
        lds(ys[warp * KW + k0 + u], y);
#pragma unroll
        for (int r = 0; r < R; r++) {
          acc[0][r] += av[u][0] * y[r];
          acc[1][r] += av[u][1] * y[r];
        }
      }
    }
  }
  __syncthreads();  // ys is read
  // eight partial sums per row: warps 4-7 hand theirs to warps 0-3, those
  // four are then added up by all threads
  if (warp >= 4) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      red[warp - 4][lane][r] = acc[0][r];
      red[warp - 4][lane + 32][r] = acc[1][r];
    }
  }
  __syncthreads();
  if (warp < 4) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      red[warp][lane][r] += acc[0][r];
      red[warp][lane + 32][r] += acc[1][r];
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < GEMV_ROWS * R; e += 256) {
    const int i = e % GEMV_ROWS, r = e / GEMV_ROWS;
    const int row = t.chunk * GEMV_ROWS + i;
    if (row < nrows && r < nr) {
      const T s = (red[0][i][r] + red[1][i][r]) + (red[2][i][r] + red[3][i][r]);
      atomicAdd(dst + (FWD && qrow ? qrow[row] : row) + r * ldst, -s);
    }
  }
}

template <typename T, int R>
__global__ void __launch_bounds__(256)
    k_gemv_l21(const SweepTask* __restrict__ tasks, int ngroups,
               const FrontDev* __restrict__ fr, const T* __restrict__ F,
               SweepVec vec, int nrhs, T* W, T* Y) {
  gemv_off<T, R, true>(tasks, ngroups, fr, F, vec, nrhs, W, Y);
}

template <typename T, int R>
__global__ void __launch_bounds__(256)
    k_gemv_u12(const SweepTask* __restrict__ tasks, int ngroups,
               const FrontDev* __restrict__ fr, const T* __restrict__ F,
               SweepVec vec, int nrhs, T* W, T* Y) {
  gemv_off<T, R, false>(tasks, ngroups, fr, F, vec, nrhs, W, Y);
}

}  // namespace snu
