// trsv_stream.cu -- incomplete-LU apply of whole systems with many short levels, one CTA per system
// (k_trsv_stream; the tables are described at StreamEnt in solver_kernels.cuh).
//
// 1D devices in natural order, Poisson systems and ILUT factors have 250 to several thousand levels of a
// few slices.  Nothing there is bound by bytes or arithmetic: the time is the number of levels times
// the time from one level to the next, and that is instructions and latencies on one SM.  So the
// sweep's data are laid out for it once per factorisation (k_stream_fill: column and value of an entry
// in one word, columns as positions in the shared-memory ring of solved values, the lane's
// destination and inverse diagonal in another), a warp holds its next slice in registers before
// the barrier of the level, and between two barriers a warp only loads from the ring, multiplies and
// stores: 0.10 us from one level to the next.  Per apply, k_trsv_task before and k_trsv_stream now:
// 250-box diode (278 + 278 levels of 4 slices, FP32 factor) 385 and 69 us, 200x50 Poisson system
// (249 + 249 levels of 2 slices, FP64 factor) 416 and 51 us, 32-diode sweep (at most 1202 + 1202
// levels) 2333 and 672 us, ILUT of a 20 076-row L = 5 bar (1001 + 874 levels, rows of up to 151
// entries) 2139 and 580 us.  Tried on the diode and the Poisson system: one chunk across levels with
// k_trsv_task's slices and a barrier per level 205 and 183 us; no barrier, rows polling the ring for
// pending entries 102 and 104 us; this layout with conditional steps 287 and 153 us (a branch costs
// a lone warp some 20 cycles).
#include <cuda_runtime.h>
#include <cstdint>

#include "solver_kernels.cuh"
#include "staging.cuh"
#include "kernels.h"

namespace vshe {

namespace {

__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// Counts an arrival on the mbarrier once this thread's asynchronous copies so far have landed.
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// The ring starts the CTA's dynamic shared memory, the stages follow it.
extern __shared__ __align__(128) unsigned char g_smem[];

// A lane's part of one slice, as it waits for the level to start.
template <typename P, int W>
struct Held {
  StreamStep d;
  StreamEnt<P> e[W];
  StreamRow row;
  double base;
};
// two slices held at once, where the registers allow it
template <typename P, int W> constexpr bool kHeldAhead = W <= (sizeof(P) == 4 ? 8 : 6);

__device__ __forceinline__ double at_smem(int at) { return *(const double *)(g_smem + at); }

// Everything of a step's slice that does not depend on the levels before.  No branches here and in
// solve_held: with one or two warps per scheduler each costs some 20 cycles, as much as a shared-memory
// access, so a warp without a slice sums the chunk's empty one.
template <typename P, int W>
__device__ __forceinline__ void read_held(Held<P, W> &h, const StreamStep &d, unsigned stage, int lane) {
  h.d = d;
  const StreamEnt<P> *e = (const StreamEnt<P> *)(g_smem + stage + d.ent) + lane;
#pragma unroll
  for (int u = 0; u < W; ++u) h.e[u] = e[32 * u];
  h.row = ((const StreamRow *)(g_smem + stage + d.row))[lane];
  h.base = ((const double *)(g_smem + stage + d.op))[lane];
}

template <typename P, int W, bool kTail, bool kKeep>
__device__ __forceinline__ void solve_held(const Held<P, W> &h, unsigned stage, int lane, int threads, double *dst, double *keep) {
  consumers_sync(threads);
  double x[W];
#pragma unroll
  for (int u = 0; u < W; ++u) x[u] = at_smem(h.e[u].at);
  double sum = 0.0;
#pragma unroll
  for (int u = 0; u < W; ++u) sum = fma((double)h.e[u].v, x[u], sum);
  if constexpr (kTail) {
    const StreamEnt<P> *e = (const StreamEnt<P> *)(g_smem + stage + h.d.ent) + lane;
#pragma unroll 4
    for (int u = W; u < h.d.width; ++u) {
      const StreamEnt<P> t = e[32 * u];
      sum = fma((double)t.v, at_smem(t.at), sum);
    }
  }
  // (the forward rows carry 1: a multiplication by 1 changes no bit)
  const double y = (h.base - sum) * h.row.dinv;
  if (h.row.dst >= 0) {
    *(double *)(g_smem + h.row.pos) = y;
    dst[h.row.dst] = y;
    if (kKeep) keep[(h.d.op >> 3) + lane] = y;
  }
}

// What a warp needs to walk the chunks of one sweep.
struct Walk {
  const StreamChunk *chunks;
  uint64_t *full, *empty;
  double *dst, *ytmp;       // where results go by destination, and by number
  const unsigned *bar;
  int32_t *err;
  unsigned stages;
  int g0, g1, stage_bytes, nwarp;
};

// One sweep of a task on one consumer warp.  kTail: slices wider than W; kKeep: values are read after they
// left the ring, so they go to global memory by number too.  Functions of their own: inlined into one kernel the variants spill.  Returns false
// after a failed wait.
template <typename P, int W, bool kTail, bool kKeep>
__device__ __noinline__ bool walk(const Walk &wk) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nwarp = wk.nwarp, threads = 32 * nwarp, g1 = wk.g1, stage_bytes = wk.stage_bytes;
  const StreamChunk *chunks = wk.chunks;
  uint64_t *full = wk.full, *empty = wk.empty;
  double *dst = wk.dst, *ytmp = wk.ytmp;
  int32_t *err = wk.err;
  const unsigned stages = wk.stages;
  const unsigned long long limit = spin_limit_of(wk.bar);
  for (int g = wk.g0; g < g1; ++g) {
    const int stg = g % kLocStages;
    const int nstep = chunks[g].nstep;
    // operand offsets count from the stage's start: the row at stage offset o is number
    // op0 + (o - first operand's offset) / 8
    double *keep = kKeep ? ytmp + chunks[g].op0 - ((chunks[g].head_bytes + chunks[g].ent_bytes + chunks[g].row_bytes) >> 3) - chunks[g].nold : nullptr;
    if (!mbar_wait_warp(&full[stg], (g / kLocStages) & 1, limit, err)) {
      // the error word is set or this wait ran out: every warp takes the level barriers that are left
      for (int q = g; q < g1; ++q)
        for (int b = 0; b < chunks[q].nstep; ++b) consumers_sync(threads);
      return false;
    }
    const unsigned stage = stages + (unsigned)(stg * stage_bytes);
    const StreamStep *sd = (const StreamStep *)(g_smem + stage) + warp;
    // (an even number of steps, and two more descriptors)
    if constexpr (kHeldAhead<P, W>) {
      Held<P, W> A, B;
      StreamStep next = sd[nwarp];
      read_held<P, W>(A, sd[0], stage, lane);
      for (int i = 0; i < nstep; i += 2) {
        read_held<P, W>(B, next, stage, lane);
        next = sd[(i + 2) * nwarp];
        solve_held<P, W, kTail, kKeep>(A, stage, lane, threads, dst, keep);
        read_held<P, W>(A, next, stage, lane);
        next = sd[(i + 3) * nwarp];
        solve_held<P, W, kTail, kKeep>(B, stage, lane, threads, dst, keep);
      }
    } else {
      Held<P, W> A;
      StreamStep next = sd[0];
      for (int i = 0; i < nstep; ++i) {
        read_held<P, W>(A, next, stage, lane);
        next = sd[(i + 1) * nwarp];
        solve_held<P, W, kTail, kKeep>(A, stage, lane, threads, dst, keep);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[stg]);
  }
  return true;
}

template <typename P, bool kKeep>
__device__ __forceinline__ bool walk_any(const Walk &k, int width) {
  switch (width) {
    case 1: return walk<P, 1, false, kKeep>(k);
    case 2: return walk<P, 2, false, kKeep>(k);
    case 3: return walk<P, 3, false, kKeep>(k);
    case 4: return walk<P, 4, false, kKeep>(k);
    case 5: return walk<P, 5, false, kKeep>(k);
    case 6: return walk<P, 6, false, kKeep>(k);
    case 8: return walk<P, 8, false, kKeep>(k);
    default: return walk<P, 8, true, kKeep>(k);
  }
}

}  // namespace

// out = U^{-1} L^{-1} in for one whole system on one CTA.  The arithmetic of a row is that of
// k_trsv_task, bit for bit (padding entries multiply 0 by the ring's zero).  One producer warp
// streams the chunks through kLocStages stages: lane 0 with bulk copies, all lanes the values older than
// the ring with copies of 8 bytes whose completion is counted on the same mbarrier.  The forward result is written by slot
// (yslot), so the backward sweep's operands are copied like the forward sweep's once every warp has
// fenced its writes (fwd).  Every chunk wait is bounded (bar[2..3] polls); after one has failed the error
// word is set, the others find it in their own waits, and every warp walks the remaining level
// barriers without touching the stages (their number is in the chunk table).
template <typename P>
__global__ void __launch_bounds__(32 * (kStreamWarps + 1), 1)
    k_trsv_stream(const SysDev<P> *sys, const BiState *st, const int32_t *active, const StreamTask *tasks, int which, const unsigned *bar,
                  int32_t *err) {
  __shared__ __align__(8) uint64_t full[kLocStages], empty[kLocStages], fwd;
  const StreamTask &T = tasks[blockIdx.x];
  const int s = T.sys;
  if (!active[s] || st[s].done || (which == 1 && st[s].s_conv)) return;
  const SysDev<P> &S = sys[s];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, producer = (int)(blockDim.x >> 5) - 1;
  const unsigned stages = 8u * (unsigned)T.ring + 128u;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kLocStages; ++i) { mbar_init(&full[i], 1 + 32); mbar_init(&empty[i], T.nwarp); }
    mbar_init(&fwd, T.nwarp);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *(double *)(g_smem + 8 * (size_t)T.ring) = 0.0;  // the value of padding entries
  }
  __syncthreads();

  if (warp == producer) {
    const unsigned long long limit = spin_limit_of(bar);
    const double *in = which == 0 ? S.p : S.s, *ytmp = S.ytmp;
    const int nchunk = T.nchunk, nfwd = T.nfwd, stage_bytes = T.stage;
    int issued = 0;
    bool forward_done = false;
    StreamChunk next = T.chunks[0];
    for (int g = 0; g < nchunk; ++g) {
      const StreamChunk c = next;
      if (g + 1 < nchunk) next = T.chunks[g + 1];
      const int old = lane < c.nold ? T.olds[c.old0 + lane] : 0;
      const int stg = g % kLocStages, round = g / kLocStages;
      bool ok = *((volatile int32_t *)err) == 0;
      if (ok && round > 0 && lane == 0) ok = mbar_wait(&empty[stg], (round - 1) & 1, limit, err);
      if (!__all_sync(0xffffffffu, ok)) break;
      unsigned char *base = g_smem + stages + (unsigned)(stg * stage_bytes);
      const unsigned at_old = (unsigned)(c.head_bytes + c.ent_bytes + c.row_bytes), at_op = at_old + 8u * (unsigned)c.nold, ops = 8u * (unsigned)c.nop;
      const bool lower = g < nfwd;
      if (lane == 0) {
        mbar_expect_tx(&full[stg], at_old);
        bulk_g2s(base, T.heads + c.head, (unsigned)c.head_bytes, &full[stg]);
        bulk_g2s(base + c.head_bytes, T.ent + c.ent, (unsigned)c.ent_bytes, &full[stg]);
        bulk_g2s(base + c.head_bytes + c.ent_bytes, T.row + c.row, (unsigned)c.row_bytes, &full[stg]);
      }
      for (int i = lane; i < c.nold; i += 32) cp_async8(base + at_old + 8 * i, ytmp + (i == lane ? old : T.olds[c.old0 + i]));
      cp_async_arrive(&full[stg]);
      issued = g + 1;
      if (!lower && !forward_done) {
        if (lane == 0) ok = mbar_wait(&fwd, 0, limit, err);
        ok = forward_done = __all_sync(0xffffffffu, ok);
        fence_async_proxy();
      }
      if (lane == 0) {
        mbar_arrive_expect_tx(&full[stg], ok ? ops : 0u);
        if (ok) bulk_g2s(base + at_op, (lower ? in : T.yslot) + c.op0, ops, &full[stg]);
      }
      if (!ok) break;
    }
    __syncwarp();
    // copies of the last kLocStages chunks can be in flight; leave once they have landed
    if (lane == 0)
      for (int g = issued > kLocStages ? issued - kLocStages : 0; g < issued; ++g) mbar_drain(&full[g % kLocStages], (g / kLocStages) & 1);
    __syncwarp();
    return;
  }
  if (warp >= T.nwarp) return;

  Walk k{T.chunks, full, empty, T.yslot, S.ytmp, bar, err, stages, 0, T.nfwd, T.stage, T.nwarp};
  const bool ok = T.keep[0] ? walk_any<P, true>(k, T.width[0][warp]) : walk_any<P, false>(k, T.width[0][warp]);
  // the forward result is complete: hand this thread's part to the bulk copies
  fence_async_proxy();
  __syncwarp();
  if (!ok) {
    // (no further chunk wait: the phase parities tell nothing once a phase has been given up)
    for (int q = T.nfwd; q < T.nchunk; ++q)
      for (int b = 0; b < T.chunks[q].nstep; ++b) consumers_sync(k.nwarp * 32);
    return;
  }
  if (lane == 0) mbar_arrive(&fwd);
  k.dst = which == 0 ? S.ph : S.sh;
  k.g0 = T.nfwd;
  k.g1 = T.nchunk;
  if (T.keep[1]) walk_any<P, true>(k, T.width[1][warp]);
  else walk_any<P, false>(k, T.width[1][warp]);
}

// Entries and rows of a stream from the system's SELL slices: one warp per slice record; all = false:
// the factor's values only.  (k_stream_patch then names the values older than the ring.)
template <typename P>
__global__ void k_stream_fill(SysDev<P> S, int nrec, const StreamRec *recs, const int64_t *dpos, int ring, bool all, unsigned char *ent,
                              unsigned char *row) {
  const int lane = threadIdx.x & 31, nw = (int)(gridDim.x * blockDim.x >> 5);
  for (int r = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); r < nrec; r += nw) {
    const StreamRec R = recs[r];
    const bool lower = R.lower != 0;
    const int j = R.slice;  // negative: an empty slice
    int64_t off = 0;
    int w = 0;
    int32_t r0 = 0, nr = 0;
    if (j >= 0) {
      off = lower ? S.loff[j] : S.uoff[j];
      w = (int)(((lower ? S.loff[j + 1] : S.uoff[j + 1]) - off) >> 5);
      r0 = lower ? S.lrow0[j] : S.uslot0[j];
      nr = (lower ? S.lrow0[j + 1] : S.uslot0[j + 1]) - r0;
    }
    StreamEnt<P> *e = (StreamEnt<P> *)(ent + R.ent) + lane;
    StreamRow *t = (StreamRow *)(row + R.row) + lane;
    if (all) {
      for (int u = 0; u < R.width; ++u) {
        StreamEnt<P> z{};
        z.at = 8 * ring;  // padding: value 0 times the ring's zero
        if (u < w) {
          const int64_t k = off + 32 * u + lane;
          const int32_t c = lower ? S.lcol[k] : S.ucol[k];
          if (c < S.n) z.at = 8 * ((lower ? c : (int32_t)dpos[c]) & (ring - 1));
        }
        e[32 * u] = z;
      }
      StreamRow z{0, -1, 1.0};
      if (lane < nr) {
        const int32_t q = r0 + lane;
        z.pos = 8 * (q & (ring - 1));
        z.dst = lower ? (int32_t)dpos[q] : S.urow[q];
      }
      *t = z;
      continue;
    }
    for (int u = 0; u < w; ++u) e[32 * u].v = (lower ? S.lval : S.uval)[off + 32 * u + lane];
    if (!lower && lane < nr) t->dinv = (double)S.udinv[r0 + lane];
  }
}

template <typename P>
__global__ void k_stream_patch(int count, const int64_t *patch, unsigned char *ent) {
  for (int i = (int)(blockIdx.x * blockDim.x + threadIdx.x); i < count; i += (int)(gridDim.x * blockDim.x))
    ((StreamEnt<P> *)ent)[patch[2 * i]].at = (int32_t)patch[2 * i + 1];
}

}  // namespace vshe

using namespace vshe;

template <typename P>
static int launch_stream(int ntasks, int nwarp, int smem, const void *sys, const void *st, const int32_t *act, const void *tasks, int which,
                         const unsigned *bar, int32_t *err, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute((const void *)k_trsv_stream<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLocSmemMax);
  if (e != cudaSuccess) return (int)e;
  vk_count_launches(1);
  k_trsv_stream<P><<<ntasks, 32 * (nwarp + 1), smem, s>>>((const SysDev<P> *)sys, (const BiState *)st, act, (const StreamTask *)tasks, which, bar, err);
  return (int)cudaGetLastError();
}

template <typename P>
static int launch_fill(const void *sysdev, int nrec, const void *recs, const int64_t *dpos, int ring, int npatch, const int64_t *patch, bool all,
                       void *ent, void *row, cudaStream_t s) {
  const int blocks = nrec < 8 * 592 ? (nrec + 7) / 8 : 592;
  vk_count_launches(1);
  k_stream_fill<P><<<blocks, 256, 0, s>>>(*(const SysDev<P> *)sysdev, nrec, (const StreamRec *)recs, dpos, ring, all, (unsigned char *)ent,
                                          (unsigned char *)row);
  if (all && npatch > 0) {
    vk_count_launches(1);
    k_stream_patch<P><<<(npatch + 255) / 256, 256, 0, s>>>(npatch, patch, (unsigned char *)ent);
  }
  return (int)cudaGetLastError();
}

extern "C" {

int vk_trsv_stream(int mixed, int ntasks, int nwarp, int smem, const void *sys, const void *st, const int32_t *act, const void *tasks, int which,
                   const unsigned *bar, int32_t *err, cudaStream_t s) {
  return mixed ? launch_stream<float>(ntasks, nwarp, smem, sys, st, act, tasks, which, bar, err, s)
               : launch_stream<double>(ntasks, nwarp, smem, sys, st, act, tasks, which, bar, err, s);
}

int vk_stream_fill(int mixed, const void *sysdev, int nrec, const void *recs, const int64_t *dpos, int ring, int npatch, const int64_t *patch,
                   int all, void *ent, void *row, cudaStream_t s) {
  if (nrec <= 0) return 0;
  return mixed ? launch_fill<float>(sysdev, nrec, recs, dpos, ring, npatch, patch, all != 0, ent, row, s)
               : launch_fill<double>(sysdev, nrec, recs, dpos, ring, npatch, patch, all != 0, ent, row, s);
}

}  // extern "C"
