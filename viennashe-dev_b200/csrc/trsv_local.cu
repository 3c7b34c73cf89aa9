// trsv_local.cu -- incomplete-LU apply of block tasks whose solved values fit shared memory
// (k_trsv_local; the records are described at LocHead in solver_kernels.cuh).
//
// On slabs of a few thousand rows k_trsv_task is bound by latency, not by bytes: a level is a handful of
// slices per warp, every gather of a solved value goes to L2 and back, and all warps wait for each
// chunk of copies together.  Here the values stay in shared memory, every warp streams its own slices
// (bulk copies into its own slots, no hand-over between warps), and the warps meet only at the
// level barriers.  Per apply, k_trsv_task and k_trsv_local: bar 50 x 20 x 60, first order (38 tasks of up
// to 1040 rows) 17 and 9.0 us; bar 100 x 25 x 80, third order (52 of up to 15300) 101 and 76; bar 90 x
// 29 x 64, third order (37 of up to 16008) 127 and 87; bar 71 x 27 x 67, third order, FP64 factors
// (40 of up to 11826) 103 and 76.  What bounds the large ones is the chain of records of a warp, about 90
// of 450 cycles for the gathers and sums and as many for the loads, beside a level's imbalance and shared memory
// itself (a gather takes 3.8 passes over the banks); a task on a cluster of 2 to 4 CTAs, each with all
// values, measured no better (87 to 100 us on the third of these: a level then waits for stores and
// arrivals between SMs).
#include <cuda_runtime.h>
#include <cstdint>

#include "solver_kernels.cuh"
#include "staging.cuh"
#include "kernels.h"

namespace vshe {

namespace {

extern __shared__ __align__(128) unsigned char l_smem[];

// a record in registers; columns past its groups are zeros times the zero of padding
template <typename P>
struct Record {
  LocHead H;
  uint2 at[2];
  __align__(16) P v[8];
  P dinv;
  int loc;
  // loads the record at rec; returns the next
  __device__ __forceinline__ const unsigned char *load(const unsigned char *rec, int lane, int ring) {
    H = *(const LocHead *)rec;
    rec += sizeof(LocHead);
    const unsigned char *at_ = rec + 128 * sizeof(P) * H.groups;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      at[g] = make_uint2((unsigned)ring * 65537u, (unsigned)ring * 65537u);
#pragma unroll
      for (int u = 0; u < 4; ++u) v[4 * g + u] = P(0);
      if (g < H.groups) {
        at[g] = *(const uint2 *)(at_ + 256 * g + 8 * lane);
        const uint4 *q = (const uint4 *)(rec + g * 128 * sizeof(P) + 4 * sizeof(P) * lane);
#pragma unroll
        for (int u = 0; u < (int)sizeof(P) / 4; ++u) *(uint4 *)(v + 4 * g + u * 16 / (int)sizeof(P)) = q[u];
      }
    }
    rec = at_ + 256 * H.groups;
    loc = H.loc0 + lane;
    dinv = P(1);
    if (H.nr >= kLocBack) {
      dinv = ((const P *)rec)[lane];
      loc = ((const uint16_t *)(rec + 32 * sizeof(P)))[lane];
      rec += 32 * (sizeof(P) + 2);
    }
    return rec;
  }
  __device__ __forceinline__ double sum(double s) const {
    const double *val = (const double *)l_smem;
    double x[8];
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      x[4 * g] = val[at[g].x & 0xffff];
      x[4 * g + 1] = val[at[g].x >> 16];
      x[4 * g + 2] = val[at[g].y & 0xffff];
      x[4 * g + 3] = val[at[g].y >> 16];
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) s = fma((double)v[u], x[u], s);
    return s;
  }
};

}  // namespace

// out = U^{-1} L^{-1} in for one block task on one CTA.  The arithmetic of a row is that of k_trsv_task,
// bit for bit.  Waits for copies are bounded (bar[2..3] polls); after one has failed the error word is
// set, the warp takes the remaining barriers without touching its slots, waits for its copies in flight
// and leaves; the others find the error word in their own waits.
template <typename P>
__global__ void __launch_bounds__(32 * kLocWarps, 1)
    k_trsv_local(const SysDev<P> *sys, const BiState *st, const int32_t *active, const LocTask *tasks, const LocRun *runs, const LocWarp *warps,
                 const unsigned char *recs, int which, int ring, int slot_bytes, const unsigned *bar, int32_t *err) {
  __shared__ __align__(8) uint64_t full[kLocWarps * kLocSlots];
  const LocTask T = tasks[blockIdx.x];
  const int s = T.sys;
  if (!active[s] || st[s].done || (which == 1 && st[s].s_conv)) return;
  const SysDev<P> &S = sys[s];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, threads = (int)blockDim.x;
  double *val = (double *)l_smem;
  const LocWarp W = warps[T.warp0 + warp];
  uint64_t *mine = full + warp * kLocSlots;
  unsigned char *slot0 = l_smem + 8 * (size_t)ring + 128 + (size_t)(warp * kLocSlots) * slot_bytes;
  const unsigned long long limit = spin_limit_of(bar);
  const unsigned char *next = recs + W.off;  // lane 0: the next chunk to copy
  int issued = 0;
  auto issue = [&](int slot, int bytes) {
    mbar_arrive_expect_tx(&mine[slot], (unsigned)bytes);
    bulk_g2s(slot0 + slot * slot_bytes, next, (unsigned)bytes, &mine[slot]);
    next += bytes;
    ++issued;
  };
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < kLocSlots; ++i) mbar_init(&mine[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
#pragma unroll
    for (int i = 0; i < kLocSlots - 1; ++i)
      if (i < W.nchunk) issue(i, W.bytes[i]);
  }
  // the input in the order of the numbers; a lane holds one level's run of rows
  const double *in = which == 0 ? S.p : S.s;
  double *out = which == 0 ? S.ph : S.sh;
  auto each_run = [&](auto &&f) {
    for (int k0 = 0; k0 < T.nlevF; k0 += 32) {
      LocRun R{0, 0};
      if (k0 + lane < T.nlevF) R = runs[T.run0 + k0 + lane];
      int end = __shfl_down_sync(0xffffffffu, R.num, 1);
      if (k0 + lane + 1 == T.nlevF) end = T.m;
      else if (lane == 31 && k0 + 32 < T.nlevF) end = runs[T.run0 + k0 + 32].num;
      for (int k = 0; k < 32 && k0 + k < T.nlevF; ++k) {
        const int row = __shfl_sync(0xffffffffu, R.row, k), num = __shfl_sync(0xffffffffu, R.num, k);
        f(row, num, __shfl_sync(0xffffffffu, end, k) - num);
      }
    }
  };
  each_run([&](int row, int num, int n) {
    for (int i = (int)threadIdx.x; i < n; i += threads) cp_async8(val + num + i, in + row + i);
  });
  if (threadIdx.x == 0) val[ring] = 0.0;
  cp_async_wait_all();
  __syncthreads();
  // A record is loaded into registers before the one ahead of it is worked on, so that its loads pass
  // behind that one's gathers and barriers.
  Record<P> R0, R1;
  int passed = 0, chunk = -1, slot = -1, phase = 0, left = 0, ahead = 0;
  const unsigned char *rec = nullptr;
  double sum = 0.0;
  // (ends the thread here: a result handed up through the loops costs 2 %)
  auto give_up = [&]() {
    for (; passed < T.nlev; ++passed) consumers_sync(threads);
    if (lane == 0)
      for (int q = chunk; q < issued; ++q) mbar_drain(&mine[q % kLocSlots], (q / kLocSlots) & 1);
    __syncwarp();
    asm volatile("exit;");
  };
  auto load = [&](Record<P> &R) {
    if (left == 0) {
      if (++chunk == W.nchunk) return false;
      if (++slot == kLocSlots) { slot = 0; phase ^= 1; }
      if (!mbar_wait_warp(&mine[slot], phase, limit, err)) give_up();
      rec = slot0 + slot * slot_bytes;
      const LocChunk C = *(const LocChunk *)rec;
      rec += sizeof(LocChunk);
      left = C.nrec;
      ahead = C.bytes_ahead;
    }
    --left;
    rec = R.load(rec, lane, ring);
    return true;
  };
  // the copy that opening a chunk asks for: the slot before it is free, its last record is done
  auto copy_ahead = [&]() {
    if (ahead) {
      if (lane == 0) issue(slot == 0 ? kLocSlots - 1 : slot - 1, ahead);
      ahead = 0;
    }
  };
  auto work = [&](Record<P> &R) {
    for (; passed < R.H.lev; ++passed) consumers_sync(threads);
    const int nr = R.H.nr & (kLocBack - 1);
    const double base = lane < nr ? val[R.loc] : 0.0;
    sum = R.sum(sum);
    if (nr) {
      if (lane < nr) val[R.loc] = (base - sum) * (double)R.dinv;
      sum = 0.0;
    }
    __syncwarp();
    copy_ahead();
  };
  bool more = load(R0);
  // (chunk 0's goes into the slot not used yet: loading the second record may open chunk 1)
  copy_ahead();
  while (more) {
    more = load(R1);
    work(R0);
    if (!more) break;
    more = load(R0);
    work(R1);
  }
  for (; passed < T.nlev; ++passed) consumers_sync(threads);
  each_run([&](int row, int num, int n) {
    for (int i = (int)threadIdx.x; i < n; i += threads) out[row + i] = val[num + i];
  });
}

// Records from the SELL slices, one warp per record.  all: everything, with the rows' numbers (num, by
// solver row); else the factor's values only.
template <typename P>
__global__ void k_local_fill(SysDev<P> S, int nrec, const LocRec *recs, const int32_t *num, int ring, bool all, unsigned char *buf) {
  const int lane = threadIdx.x & 31, nw = (int)(gridDim.x * blockDim.x >> 5);
  for (int r = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); r < nrec; r += nw) {
    const LocRec R = recs[r];
    unsigned char *rec = buf + R.off;
    if (all && lane == 0) *(LocHead *)rec = R.head;
    if (R.slice < 0) continue;
    const bool lower = R.lower != 0, back = R.head.nr >= kLocBack;
    const int j = R.slice, W = 4 * R.head.groups, nr = R.head.nr & (kLocBack - 1);
    const int64_t off = (lower ? S.loff[j] : S.uoff[j]) + 32 * R.u0 + lane;
    rec += sizeof(LocHead);
    P *v = (P *)rec + 4 * lane;
    uint16_t *at = (uint16_t *)(rec + 32 * sizeof(P) * W) + 4 * lane;
    unsigned char *tail = rec + 32 * (sizeof(P) + 2) * W;
    const int32_t slot = lower ? 0 : S.uslot0[j] + lane;
    for (int u = 0; u < W; ++u) {
      const int e = 128 * (u >> 2) + (u & 3);
      if (all) {
        const int32_t c = u < R.ncol ? (lower ? S.lcol : S.ucol)[off + 32 * u] : (int32_t)S.n;
        at[e] = (uint16_t)(c < S.n ? num[c] : ring);
        v[e] = P(0);
      } else if (u < R.ncol) {
        v[e] = (lower ? S.lval : S.uval)[off + 32 * u];
      }
    }
    if (!back) continue;
    if (all) {
      ((P *)tail)[lane] = P(1);
      ((uint16_t *)(tail + 32 * sizeof(P)))[lane] = (uint16_t)(lane < nr ? num[S.urow[slot]] : ring);
    } else if (lane < nr) {
      ((P *)tail)[lane] = S.udinv[slot];
    }
  }
}

}  // namespace vshe

using namespace vshe;

template <typename P>
static int launch_local(int ntasks, int nwarp, int ring, int slot_bytes, const void *sys, const void *st, const int32_t *act,
                        const void *tasks, const void *runs, const void *warps, const void *recs, int which, const unsigned *bar,
                        int32_t *err, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute((const void *)k_trsv_local<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLocSmemMax);
  if (e != cudaSuccess) return (int)e;
  vk_count_launches(1);
  k_trsv_local<P><<<ntasks, 32 * nwarp, 8 * ring + 128 + nwarp * kLocSlots * slot_bytes, s>>>(
      (const SysDev<P> *)sys, (const BiState *)st, act, (const LocTask *)tasks, (const LocRun *)runs, (const LocWarp *)warps,
      (const unsigned char *)recs, which, ring, slot_bytes, bar, err);
  return (int)cudaGetLastError();
}

template <typename P>
static int launch_local_fill(const void *sysdev, int nrec, const void *recs, const int32_t *num, int ring, bool all, void *buf, cudaStream_t s) {
  vk_count_launches(1);
  const int blocks = nrec < 8 * 1184 ? (nrec + 7) / 8 : 1184;
  k_local_fill<P><<<blocks, 256, 0, s>>>(*(const SysDev<P> *)sysdev, nrec, (const LocRec *)recs, num, ring, all, (unsigned char *)buf);
  return (int)cudaGetLastError();
}

extern "C" {

int vk_trsv_local(int mixed, int ntasks, int nwarp, int ring, int slot_bytes, const void *sys, const void *st, const int32_t *act,
                  const void *tasks, const void *runs, const void *warps, const void *recs, int which, const unsigned *bar, int32_t *err,
                  cudaStream_t s) {
  return mixed ? launch_local<float>(ntasks, nwarp, ring, slot_bytes, sys, st, act, tasks, runs, warps, recs, which, bar, err, s)
               : launch_local<double>(ntasks, nwarp, ring, slot_bytes, sys, st, act, tasks, runs, warps, recs, which, bar, err, s);
}

int vk_local_fill(int mixed, const void *sysdev, int nrec, const void *recs, const int32_t *num, int ring, int all, void *buf, cudaStream_t s) {
  if (nrec <= 0) return 0;
  return mixed ? launch_local_fill<float>(sysdev, nrec, recs, num, ring, all != 0, buf, s)
               : launch_local_fill<double>(sysdev, nrec, recs, num, ring, all != 0, buf, s);
}

}  // extern "C"
