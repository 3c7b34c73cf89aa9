// trsv_local.cu -- incomplete-LU apply of tasks whose solved values are gathered from shared memory
// (k_trsv_local, the LocTask tables of solver_kernels.cuh).
//
// k_trsv_task takes one chunk of copies per level and sends every gather of a solved value to L2 and
// back.  On slabs of a few thousand rows that latency, not the bytes, sets the time.  Here a chunk
// spans levels (one set of copies per 32 KB of operands, issued by the lanes of the producer warp in
// parallel) and the solved values stay in shared memory.  Per apply, k_trsv_task before and
// k_trsv_local now: 50x20x60 bar, L = 1 (38 tasks, 7 + 7 levels) 17.2 and 12.3 us, 100x25x80 bar,
// L = 3 (52 tasks, 21 + 21 levels) 101 and 93 us.
#include <cuda_runtime.h>
#include <cstdint>

#include "solver_kernels.cuh"
#include "staging.cuh"
#include "kernels.h"

namespace vshe {

namespace {

constexpr int kLocU = 4;  // entries of a row held in registers across the level barrier (rows of ILU(0) hold 2 to 5)

// orders this thread's global writes before later bulk copies that read them (with the mbarrier
// arrival that follows)
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// What a warp reads of one slice from the stage before its level starts: lane = row.
template <typename P>
struct LocRow {
  int4 d0, d1;  // SliceLoc
  int dst;
  double base;
  P dinv;
  int c[kLocU];
  P v[kLocU];
};

// Barriers and source arrays of a task, by one thread.
template <typename P>
__device__ __forceinline__ void task_init(const SysDev<P> &S, const LocSys &Q, const unsigned char *heads, int which, int consumers,
                                          const unsigned char **bases, uint64_t *full, uint64_t *empty, uint64_t *fwd) {
  for (int i = 0; i < kLocStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], consumers); }
  mbar_init(fwd, consumers);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  bases[kLocHead] = heads;
  bases[kLocLCol] = (const unsigned char *)Q.lcol;
  bases[kLocLVal] = (const unsigned char *)S.lval;
  bases[kLocIn] = (const unsigned char *)(which == 0 ? S.p : S.s);
  bases[kLocFSlot] = (const unsigned char *)Q.fslot;
  bases[kLocUCol] = (const unsigned char *)Q.ucol;
  bases[kLocUVal] = (const unsigned char *)S.uval;
  bases[kLocYSlot] = (const unsigned char *)Q.yslot;
  bases[kLocURow] = (const unsigned char *)S.urow;
  bases[kLocUDinv] = (const unsigned char *)S.udinv;
}

// Everything of a slice that does not depend on the rows before it, from its stage (R.d0, R.d1 set).
template <typename P>
__device__ __forceinline__ void read_row(LocRow<P> &R, const unsigned char *stage, const LocHead &H, bool lower, int lane) {
  const int width = R.d0.w >> 6;
  const int32_t *c = (const int32_t *)(stage + R.d0.x) + lane;
  const P *v = (const P *)(stage + R.d0.y) + lane;
#pragma unroll
  for (int u = 0; u < kLocU; ++u) {
    R.c[u] = kLocPad; R.v[u] = P(0);
    if (u < width) { R.c[u] = c[32 * u]; R.v[u] = v[32 * u]; }
  }
  R.base = 0.0; R.dinv = P(1); R.dst = 0;
  if (lane < (R.d0.w & 63)) {
    const int op = R.d0.z + lane;
    R.base = ((const double *)(stage + H.offA))[op];
    R.dst = ((const int32_t *)(stage + H.offB))[op];
    if (!lower) R.dinv = ((const P *)(stage + H.offC))[op];
  }
}

// The producer warp of a task: lane i issues copies i, i + 32, ... of a chunk.  Leaves once its
// copies have landed.
__device__ __forceinline__ void produce(const LocTask &T, const LocChunk *chunks, const LocCopy *copies, const unsigned char *const *bases,
                                        unsigned char *stages, int stage_bytes, uint64_t *full, uint64_t *empty, uint64_t *fwd,
                                        unsigned long long limit, int32_t *err) {
  const int lane = threadIdx.x & 31;
  int issued = 0;
  bool fwd_done = false;
  LocChunk next = T.nchunk > 0 ? chunks[T.c0] : LocChunk{};
  for (int g = 0; g < T.nchunk; ++g) {
    const LocChunk c = next;
    if (g + 1 < T.nchunk) next = chunks[T.c0 + g + 1];
    LocCopy r0{};
    if (lane < c.nrec) r0 = copies[c.rec0 + lane];
    const int e = *((volatile int32_t *)err);
    const int stg = g % kLocStages, round = g / kLocStages;
    bool ok = e == 0;
    if (ok && round > 0 && lane == 0) ok = mbar_wait(&empty[stg], (round - 1) & 1, limit, err);
    if (!__all_sync(0xffffffffu, ok)) break;
    const bool late = c.nlate > 0 && !fwd_done;
    const int now = late ? c.nrec - c.nlate : c.nrec;
    if (lane == 0) {
      if (late) mbar_expect_tx(&full[stg], (unsigned)c.bytes);
      else mbar_arrive_expect_tx(&full[stg], (unsigned)(c.bytes + c.late_bytes));
    }
    __syncwarp();
    unsigned char *base = stages + (size_t)stg * stage_bytes;
    for (int i = lane; i < now; i += 32) {
      const LocCopy r = i == lane ? r0 : copies[c.rec0 + i];
      bulk_g2s(base + r.dst, bases[r.what >> 24] + r.src, (unsigned)(r.what & 0xffffff), &full[stg]);
    }
    issued = g + 1;
    if (late) {
      bool done = true;
      if (lane == 0) done = mbar_wait(fwd, 0, limit, err);
      done = __all_sync(0xffffffffu, done);
      // (after a failed wait the phase still completes with the copies issued, for the drain below)
      if (lane == 0) mbar_arrive_expect_tx(&full[stg], done ? (unsigned)c.late_bytes : 0u);
      __syncwarp();
      if (!done) break;
      fence_async_proxy();
      for (int i = now + lane; i < c.nrec; i += 32) {
        const LocCopy r = copies[c.rec0 + i];
        bulk_g2s(base + r.dst, bases[r.what >> 24] + r.src, (unsigned)(r.what & 0xffffff), &full[stg]);
      }
      fwd_done = true;
    }
  }
  __syncwarp();
  // copies of the last kLocStages chunks can be in flight; leave once they have landed
  if (lane == 0)
    for (int g = issued > kLocStages ? issued - kLocStages : 0; g < issued; ++g) mbar_drain(&full[g % kLocStages], (g / kLocStages) & 1);
}

}  // namespace

// The incomplete-LU apply of one task (a whole system or a run of preconditioner blocks) on one CTA:
// out = U^{-1} L^{-1} in, level by level.  Slice by slice and row by row it is the arithmetic of
// k_trsv_task (one row per lane, summed in index order with FP64 FMAs), so both give the same bits.
//
// One producer warp streams the task's chunks through kLocStages shared-memory stages.  The
// consumer warps take the slices the plan assigned to them, a named barrier between two levels.  A
// warp reads the columns, values and operands of its next slice from the stage before it sums
// the current one (kMaxThreads <= 512; with 1024 threads the registers do not allow it, and
// the other warps cover the latency), and the gathers older than the ring go out before the
// level barrier, so between two barriers there are only the gathers from the ring, the FMAs and the store.
// A warp waits for the next chunk only after it has passed the level barriers its predecessors in
// the current chunk need (LocHead::pass), so chunk waits and level barriers cannot hold each other
// up.  The forward result is written by backward slot (yslot): the backward sweep reads it in slot
// order, so it is copied into the stages like every other operand, by bulk copies that the producer
// issues once every consumer has fenced its writes (fwd).
//
// Every chunk wait is bounded (bar[2..3] polls).  After one has failed the error word is set, the
// warp takes the remaining level barriers without touching the stages and leaves, the others
// find the error word in their own waits, and the producer drains its copies in flight before it
// leaves.
template <typename P, int kMaxThreads>
__global__ void __launch_bounds__(kMaxThreads, 1)
    k_trsv_local(const SysDev<P> *sys, const BiState *st, const int32_t *active, const LocSys *lsys, const LocTask *tasks,
                 const LocChunk *chunks, const LocCopy *copies, const unsigned char *heads, int which, int ring_max, int stage_bytes,
                 const unsigned *bar, int32_t *err) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[kLocStages], empty[kLocStages], fwd;
  __shared__ const unsigned char *bases[kLocKinds];
  const LocTask T = tasks[blockIdx.x];
  const int s = T.sys;
  if (!active[s] || st[s].done || (which == 1 && st[s].s_conv)) return;
  const SysDev<P> &S = sys[s];
  const LocSys &Q = lsys[s];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, consumers = (int)(blockDim.x >> 5) - 1;
  double *win = (double *)smem;
  unsigned char *stages = smem + 8 * (size_t)ring_max + 128;
  if (threadIdx.x == 0) {
    task_init(S, Q, heads, which, consumers, bases, full, empty, &fwd);
    win[ring_max] = 0.0;  // the value of padding entries
  }
  __syncthreads();
  const unsigned long long limit = spin_limit_of(bar);

  if (warp == consumers) {
    produce(T, chunks, copies, bases, stages, stage_bytes, full, empty, &fwd, limit, err);
    return;
  }

  // consumers
  constexpr bool kAhead = kMaxThreads <= 512;
  const int zero = ring_max, m = T.m, threads = 32 * consumers;
  double *out = which == 0 ? S.ph : S.sh, *yslot = Q.yslot;
  int lev = 0;  // level barriers passed
  auto pass_to = [&](int target) {
    while (lev < target) {
      consumers_sync(threads);
      if (++lev == T.nlevF) {  // the forward result is complete: hand this thread's part to the bulk copies
        fence_async_proxy();
        __syncwarp();
        if (lane == 0) mbar_arrive(&fwd);
      }
    }
  };
  for (int g = 0; g < T.nchunk; ++g) {
    const int stg = g % kLocStages;
    const bool lower = g < T.nfwd;
    if (!mbar_wait(&full[stg], (g / kLocStages) & 1, limit, err)) { pass_to(T.nbar); return; }
    const unsigned char *stage = stages + (size_t)stg * stage_bytes;
    const LocHead H = *(const LocHead *)stage;
    const int32_t *wptr = (const int32_t *)(stage + sizeof(LocHead));
    const int4 *sd = (const int4 *)(stage + H.offD);
    auto read = [&](LocRow<P> &R) { read_row(R, stage, H, lower, lane); };
    auto solve = [&](const LocRow<P> &R) {
      const int width = R.d0.w >> 6, nr = R.d0.w & 63, loc = R.d1.x + lane;
      int idx[kLocU];
      double a[kLocU], x[kLocU];
#pragma unroll
      for (int u = 0; u < kLocU; ++u) {
        const int q = R.c[u];
        idx[u] = q >= m ? zero : q;
        a[u] = (double)R.v[u];
      }
      pass_to(R.d1.y);
      double sum = 0.0;
#pragma unroll
      for (int u = 0; u < kLocU; ++u)
        if (u < width) x[u] = win[idx[u]];
#pragma unroll
      for (int u = 0; u < kLocU; ++u)
        if (u < width) sum = fma(a[u], x[u], sum);
      if (width > kLocU) {
        const int32_t *c = (const int32_t *)(stage + R.d0.x) + lane;
        const P *v = (const P *)(stage + R.d0.y) + lane;
#pragma unroll 4
        for (int k = kLocU; k < width; ++k) {
          const int q = c[32 * k];
          sum = fma((double)v[32 * k], win[q >= m ? zero : q], sum);
        }
      }
      if (lane < nr) {
        const double y = lower ? R.base - sum : (R.base - sum) * (double)R.dinv;
        win[loc] = y;
        (lower ? yslot : out)[R.dst] = y;
      }
    };
    const int i1 = wptr[warp + 1];
    int i = wptr[warp];
    if constexpr (kAhead) {
      LocRow<P> A, B;
      int4 e0{}, e1{};  // the descriptor after the next
      auto ahead = [&](LocRow<P> &R) {
        if (i + 1 < i1) { R.d0 = e0; R.d1 = e1; read(R); }
        if (i + 2 < i1) { e0 = sd[2 * i + 4]; e1 = sd[2 * i + 5]; }
      };
      if (i < i1) { A.d0 = sd[2 * i]; A.d1 = sd[2 * i + 1]; read(A); }
      if (i + 1 < i1) { e0 = sd[2 * i + 2]; e1 = sd[2 * i + 3]; }
      while (i < i1) {
        ahead(B);
        solve(A);
        if (++i >= i1) break;
        ahead(A);
        solve(B);
        ++i;
      }
    } else {
      for (; i < i1; ++i) {
        LocRow<P> R;
        R.d0 = sd[2 * i]; R.d1 = sd[2 * i + 1];
        read(R);
        solve(R);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[stg]);
    pass_to(H.pass);
  }
}

// slot of every row as int32
__global__ void k_slots(int64_t n, const int64_t *dpos, int32_t *fslot) {
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) fslot[i] = (int32_t)dpos[i];
}
// out[k] = map[col[k]], kLocPad for padding (column n)
__global__ void k_map_columns(int64_t n, int64_t count, const int32_t *col, const int32_t *map, int32_t *out) {
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < count; k += step) {
    const int32_t c = col[k];
    out[k] = c < n ? map[c] : kLocPad;
  }
}

}  // namespace vshe

using namespace vshe;

template <typename P>
static int launch_local(int ntasks, int consumers, int ring, int stage_bytes, const void *sys, const void *st, const int32_t *act,
                        const void *lsys, const void *tasks, const void *chunks, const void *copies, const void *heads, int which,
                        const unsigned *bar, int32_t *err, cudaStream_t s) {
  constexpr int narrow = 32 * (kLocNarrow + 1), wide = 32 * (kLocWide + 1);
  const auto k = consumers > kLocNarrow ? k_trsv_local<P, wide> : k_trsv_local<P, narrow>;
  const int smem = (int)local_smem_bytes(ring, stage_bytes);
  cudaError_t e = cudaFuncSetAttribute((const void *)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLocSmemMax);
  if (e != cudaSuccess) return (int)e;
  vk_count_launches(1);
  k<<<ntasks, 32 * (consumers + 1), smem, s>>>((const SysDev<P> *)sys, (const BiState *)st, act, (const LocSys *)lsys, (const LocTask *)tasks,
                                               (const LocChunk *)chunks, (const LocCopy *)copies, (const unsigned char *)heads, which, ring,
                                               stage_bytes, bar, err);
  return (int)cudaGetLastError();
}

extern "C" {

int vk_trsv_local(int mixed, int ntasks, int consumers, int ring, int stage_bytes, const void *sys, const void *st, const int32_t *act,
                  const void *lsys, const void *tasks, const void *chunks, const void *copies, const void *heads, int which, const unsigned *bar,
                  int32_t *err, cudaStream_t s) {
  return mixed ? launch_local<float>(ntasks, consumers, ring, stage_bytes, sys, st, act, lsys, tasks, chunks, copies, heads, which, bar, err, s)
               : launch_local<double>(ntasks, consumers, ring, stage_bytes, sys, st, act, lsys, tasks, chunks, copies, heads, which, bar, err, s);
}

int vk_slots(int64_t n, const int64_t *dpos, int32_t *fslot, cudaStream_t s) {
  vk_count_launches(1);
  k_slots<<<592, 256, 0, s>>>(n, dpos, fslot);
  return (int)cudaGetLastError();
}

int vk_map_columns(int64_t n, int64_t count, const int32_t *col, const int32_t *map, int32_t *out, cudaStream_t s) {
  vk_count_launches(1);
  k_map_columns<<<592, 256, 0, s>>>(n, count, col, map, out);
  return (int)cudaGetLastError();
}

}  // extern "C"
