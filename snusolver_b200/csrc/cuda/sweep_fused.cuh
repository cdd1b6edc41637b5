// Dependency-driven triangular sweeps: the whole forward (or backward)
// solve over the front tree in ONE cooperative launch.
//
// The level-by-level sweeps (sweep.cuh) take two launches per level and
// direction (pivot blocks, off-diagonal products); on the smallest trees
// those launches are mostly latency.  Here every level's work is one task
// list and a front starts as soon as what it reads is final:
//
// * forward: Z (elimination order, as in sweep.cuh) starts as B.  Pivot-block
//   chunk task (f, c): waits until every off-diagonal task of f's children
//   has finished, solves the tile chain of f's pivot block (chunk_sweep: the
//   chunks of f hand tiles over through Y_f) and writes Y_f.  Off-diagonal
//   task (f, 64-row block, 256-column block): waits for its columns of Y_f,
//   then subtracts L21[i, :] Y_f from the rows of Z with atomics -- straight
//   into the rows of whichever ancestor pivots them (no extend-add: the
//   elimination tree guarantees only f's descendants update f's pivot rows).
// * backward: Z is marked unsolved again.  Off-diagonal task (f, 64-row block
//   of P, 256-column block of Q): waits for its rows of Z (ancestors'
//   solutions), Y_f[i] -= U12[i, :] Z with atomics.  Pivot-block chunk task:
//   waits for all of f's off-diagonal tasks, solves the chain with the tile
//   inverses (descending), writes x_P to Z and, in FP64, to X[gidx[...]].
//
// A front's "children" here are its nearest descendants with pivots (fronts
// without pivots pass their rows on; dep.effpar skips them).  Tasks are
// listed level by level (forward: pivot chunks of a level, then its
// off-diagonal tasks; backward from the root level: off-diagonal tasks, then
// pivot chunks in descending order), so every wait is on a task of lower
// index; the grid is co-resident (cooperative launch) and blocks take tasks
// from a counter in ascending order, so the lowest unfinished task never
// waits on an unfinished one.  Every wait is bounded: when it runs out, or
// another block's has, the block records the error and returns, handing on
// nothing of the task it was in and taking no other.
#pragma once
#include "sweep.cuh"

namespace snu {

struct SolveTask {
  int kind;   // 0: pivot-block chunk (a = chunk), 1: off-diagonal block
  int front;  //    (a = 64-row block, b = 256-column block)
  int a, b;
};

// Per-front dependency data of the fused sweeps.
struct SweepDep {
  int effpar;  // nearest ancestor with pivots (-1: none)
  int need;    // forward: off-diagonal tasks of the fronts whose effpar is f
  int ngq;     // backward: off-diagonal tasks of f
};

// Counters of one sweep (zeroed before it), per front: [0, nf) forward
// off-diagonal tasks finished of f's children, [nf, 2nf) backward
// off-diagonal tasks of f finished.
__device__ __forceinline__ bool wait_count(const int* ctr, int target,
                                           int* err, long limit) {
  for (long r = 0; r < limit; r += WAVE_ROUND) {
    if (r > 0 && wait_failed(err)) break;
    for (int it = 0; it < WAVE_ROUND; it++) {
      int v;
      asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(ctr)
                   : "memory");
      if (v >= target) return true;
      if (it > 4) __nanosleep(20);
    }
  }
  atomicExch(err, 1);
  return false;
}

// Adds one to a counter, with a release at GPU scope (by one thread after
// the CTA barrier that follows the CTA's writes, as raise_flag).
__device__ __forceinline__ void count_one(int* ctr) {
  asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(ctr) : "memory");
}

// Dynamic shared memory: the pivot-block part's staging (two buffers of
// factor columns and tile inverses); the off-diagonal part reuses it.
template <typename T>
constexpr size_t fused_smem() {
  return sweep_smem<T>();
}

// One off-diagonal block with DIAG_ROWS threads: 64 rows x 2 k-groups.
// FWD: Z[rows of p + i] -= L21[i, kc0:kc1] Y[kc0:kc1]
// !FWD: Y[i] -= U12[i, kc0:kc1] Z[rows of p + kc0:kc1]
// (q: the rows of Q; Yf: f's rows of Y; columns of both n apart)
// False (in every thread) if a wait ran out: nothing was added then.  bad: the
// block's shared flag for it, zero before.
template <typename T, int R, bool FWD>
__device__ __forceinline__ bool fused_offdiag(
    const FrontDev& f, const T* __restrict__ F, const int* __restrict__ q,
    int blk, int kblk, int nrhs, T* Z, int64_t n, T* Yf, unsigned char* sm,
    int* bad, int* err, long limit) {
  constexpr size_t YS = sizeof(T) * GEMV_K * R;
  T(*ys)[R] = reinterpret_cast<T(*)[R]>(sm);
  T(*red)[GEMV_ROWS][R + 1] = reinterpret_cast<T(*)[GEMV_ROWS][R + 1]>(sm + YS);
  const int nrows = FWD ? f.q : f.p, nk = FWD ? f.p : f.q;
  const int i = blk * GEMV_ROWS + (threadIdx.x & 63), grp = threadIdx.x >> 6;
  const int kc0 = kblk * GEMV_K, kc1 = min(nk, kc0 + GEMV_K);
  const T* a = FWD ? F + f.off + f.p + i : F + f.off + i + (int64_t)f.p * f.ld;
  for (int r0 = 0; r0 < nrhs; r0 += R) {
    const int nr = min(R, nrhs - r0);
    __syncthreads();  // the previous pass's reduction is read
    // published by this launch's pivot chunks
    constexpr int N = GEMV_K * R / DIAG_ROWS, U = N < 8 ? N : 8;
#pragma unroll 1
    for (int q0 = 0; q0 < N; q0 += U) {
      T v[U];
      auto off = [&](int u) -> int64_t {
        const int e = threadIdx.x + DIAG_ROWS * (q0 + u), k = kc0 + e % GEMV_K,
                  r = e / GEMV_K;
        if (k >= kc1 || r >= nr) return -1;
        return (FWD ? k : q[k]) + (r0 + r) * n;
      };
      if (!poll_all<T, U>(FWD ? Yf : Z, off, v, err, limit)) {
        *bad = 1;
        break;
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int e = threadIdx.x + DIAG_ROWS * (q0 + u);
        ys[e % GEMV_K][e / GEMV_K] = off(u) >= 0 ? v[u] : (T)0;
      }
    }
    __syncthreads();
    if (*bad) return false;
    T acc[R];
#pragma unroll
    for (int r = 0; r < R; r++) acc[r] = (T)0;
    if (i < nrows) {
      constexpr int UB = R <= 4 ? 8 : (R <= 8 ? 4 : 2);  // loads in flight
      for (int k0 = kc0 + grp; k0 < kc1; k0 += 2 * UB) {
        T av[UB], wv[UB][R];
#pragma unroll
        for (int u = 0; u < UB; u++) {
          const int k = k0 + 2 * u;
          av[u] = k < kc1 ? a[(int64_t)k * f.ld] : (T)0;
#pragma unroll
          for (int r = 0; r < R; r++) wv[u][r] = ys[min(k, kc1 - 1) - kc0][r];
        }
#pragma unroll
        for (int u = 0; u < UB; u++)
#pragma unroll
          for (int r = 0; r < R; r++) acc[r] += av[u] * wv[u][r];
      }
    }
#pragma unroll
    for (int r = 0; r < R; r++) red[grp][threadIdx.x & 63][r] = acc[r];
    __syncthreads();
    if (grp == 0 && i < nrows) {
      for (int r = 0; r < nr; r++) {
        const T s = red[0][threadIdx.x][r] + red[1][threadIdx.x][r];
        if (FWD)
          atomicAdd(Z + q[i] + (r0 + r) * n, -s);
        else
          atomicAdd(Yf + i + (r0 + r) * n, -s);
      }
    }
  }
  return true;
}

template <typename T, int R, bool FWD>
__global__ void __launch_bounds__(DIAG_ROWS)
    k_sweep_fused(const SolveTask* __restrict__ tasks, int ntasks,
                  const FrontDev* __restrict__ fr,
                  const SweepDep* __restrict__ dep,
                  const int* __restrict__ gidx, const int* __restrict__ yidx,
                  const T* __restrict__ F, const T* __restrict__ INV,
                  int nfronts, int nrhs, int64_t n, T* Z, T* Y, double* X,
                  int ldx, int* ctr, int* next_task, int* err, long limit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Ls0 = reinterpret_cast<T*>(smem_raw);  // [2][NB][DIAG_ROWS]
  T* Xs0 = Ls0 + 2 * NB * DIAG_ROWS;         // [2][NB * NB]
  __shared__ ChunkSmem<T, R> sm;
  __shared__ int s_task;
  const int tid = threadIdx.x;
  if (tid == 0) sm.bad = 0;
  for (;;) {
    cp_async_wait_all();  // (the staging buffers: the next task's, or scratch)
    __syncthreads();
    if (tid == 0) s_task = atomicAdd(next_task, 1);
    __syncthreads();
    const int task = s_task;
    if (task >= ntasks) break;
    const SolveTask t = tasks[task];
    const FrontDev f = fr[t.front];
    const SweepDep d = dep[t.front];
    const int* g = gidx + f.idx_off;
    T* Yf = Y + f.y_off;
    if (t.kind == 1) {
      // ------------------------------------------ off-diagonal block
      if (!fused_offdiag<T, R, FWD>(f, F, yidx + f.idx_off + f.p, t.a, t.b,
                                    nrhs, Z, n, Yf, smem_raw, &sm.bad, err,
                                    limit))
        break;
      __syncthreads();
      if (tid == 0) {  // (the release orders the CTA's atomics before it)
        if (!FWD)
          count_one(ctr + nfronts + t.front);
        else if (d.effpar >= 0)
          count_one(ctr + d.effpar);
      }
      continue;
    }
    // ------------------------------------------------ pivot-block chunk
    if (tid == 0) {
      const bool ok = FWD ? wait_count(ctr + t.front, d.need, err, limit)
                          : wait_count(ctr + nfronts + t.front, d.ngq, err, limit);
      if (!ok) sm.bad = 1;
    }
    __syncthreads();
    if (sm.bad) return;
    // the chunk's rows: forward from Z, backward from Y (the forward result
    // less U12 x_Q); both written by this launch: via L2
    T* Zf = Z + f.y_off;
    const bool ok = chunk_sweep<T, R, FWD, false>(
        f, F, INV, t.a, nrhs, FWD ? Yf : Zf, n, Ls0, Xs0, sm,
        [&](int row, int r) { return __ldcg((FWD ? Zf : Yf) + row + r * n); },
        [&](int row, int r, T v) {
          if (!FWD) X[g[row] + (int64_t)r * ldx] = (double)v;
        },
        err, limit);
    if (!ok) break;
  }
  cp_async_wait_all();
}

// Z = (T) B in elimination order (orig: the original row of every row): the
// forward sweep's starting vector.
template <typename T>
__global__ void k_sweep_init(int n, int nrhs, const int* __restrict__ orig,
                             const double* __restrict__ B, int ldb,
                             T* __restrict__ Z) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= (int64_t)n * nrhs) return;
  const int i = (int)(e % n), r = (int)(e / n);
  Z[e] = (T)B[orig[i] + (int64_t)r * ldb];
}

}  // namespace snu
