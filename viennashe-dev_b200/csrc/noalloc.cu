// noalloc.cu -- the one entry point of this library that allocates no device memory:
// r = b - A x and the squared norms ||r||^2, ||b||^2 of a caller-owned CSR system.
//
// Who needs it: callers whose device memory is owned by someone else -- a host application
// whose framework hands out every byte of HBM through its own arena or caching allocator, or a
// Gummel/Newton driver that must not call cudaMalloc inside its timed inner loop (cudaMalloc and
// cudaFree synchronise the device).  Such callers bring their own device buffers for the inputs
// and outputs; the only scratch this computation needs -- one pair of partial sums per block and a
// ticket counter for the last block's reduction -- lives in a fixed file-scope __device__ array
// instead of a cudaMalloc'd buffer.
//
// The array holds kMaxTiles pairs (512 KiB), of which a call uses one per block; the row limit
// (64 Mi rows: kMaxTiles tiles of 2048) is part of the entry point's contract.  Every
// GPU that loads this library holds it until the process exits.  All calls share it: two calls
// whose kernels overlap on the GPU (different streams, or different host threads on one
// device) race on it; calls on one stream are ordered and safe.  The partial sums are fully
// rewritten by every call; the ticket counter must start at zero, which the set-up clears
// once per device, and every call leaves it at zero again.
#include <cuda_runtime.h>
#include <cstdint>
#include <mutex>

#include "../../include/vshe_gpu.h"
#include "kernels.h"

namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int64_t kMaxTiles = 32768;
constexpr int64_t kMaxRows = kMaxTiles * 2048;
constexpr int kRows = kThreads;     // rows of a block's tile: one per thread
constexpr int kChunk = 12 * kRows;  // entries staged at a time: a tile of up to 12 a row (SHE rows hold 5 to 16) in one go
constexpr int kBlocksPerSm = 5;     // 37 KB of shared memory each
constexpr int kMaxDevices = 64;

struct NoAllocScratch {
  double partial[2 * kMaxTiles];  // (||r||^2, ||b||^2) of every block
  unsigned int ticket;            // blocks finished in the current call
};

static __device__ __align__(256) NoAllocScratch g_scratch;

// Per-device address of g_scratch (host code cannot use the symbol itself as a pointer).
std::mutex g_mu;
NoAllocScratch *g_addr[kMaxDevices] = {nullptr};
int g_sms[kMaxDevices] = {0};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// sums over the block, result valid in thread 0; fixed order (deterministic)
__device__ __forceinline__ void block_sum2(double &a, double &b) {
  __shared__ double sh[2][kWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  a = warp_sum(a); b = warp_sum(b);
  if (lane == 0) { sh[0][w] = a; sh[1][w] = b; }
  __syncthreads();
  if (w == 0) {
    a = warp_sum(lane < kWarps ? sh[0][lane] : 0.0);
    b = warp_sum(lane < kWarps ? sh[1][lane] : 0.0);
  }
  __syncthreads();
}

// Asynchronous copies of one entry into shared memory: the caller's arrays promise no more than
// their elements' alignment, so the copies are as wide as the elements.
__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Tiles of kRows rows, dealt round the blocks (block b takes tiles b, b + gridDim, ...).  The
// kernel is bound by HBM (12 bytes an entry, 32 a row): a tile's entries are one contiguous run, so
// the block's threads copy it to shared memory coalesced and asynchronously, the next tile's run
// while they sum the current one, and each thread sums one row from there with FMAs, in four partial
// sums; the x gathers of neighbouring rows fall into the same lines.  A row of more than kLongRow
// entries is summed by its warp instead, lanes striding it, so that it does not wait on one thread,
// whatever the rows around it.  Before, a warp walked a row at a time and 256 rows in series
// (10 of its 32 lanes busy, three dependent loads a row).  Rows of 9 entries, before and now:
// 1000 rows 94 and 6.5 us, 100 003 rows 199 and 10.4 us, 1 000 003 rows 301 and 41.2 us
// (3.4 TB/s), 8 M rows 1271 and 277 us (4.0 TB/s).  With one running sum a row, and 42.7 and 293 us on the
// last two: tiles of 256 rows, three blocks an SM 49 and 329 us; one buffer instead of two 48 and 329 us.
// L2 flushed, rows of 8 with one of 3000 in 128 937 and 59 us (200 000 rows), rows of 33 to 47 370 and
// 121 us (500 000 rows).
// The last block to finish adds the block partials in block order; the order of every sum is fixed
// by the matrix and the SM count.
// Four partial sums are no less accurate than a warp that strides the row and adds its lanes up in a tree
// up to 28 entries (root mean square error of 28: 5.6 against 5.7 units of 2^-53; one running sum 8.6),
// eight up to 48 (7.6 against 7.7; four 8.6).  Each row chooses for itself: where a warp chose for its rows,
// rows of 22 to 33 entries took 119 us instead of 107, of 33 to 47 154 instead of 121 (500 000 rows).
constexpr int kShortRow = 28, kLongRow = 48, kParts = 8;
template <int N>
__device__ __forceinline__ void add_row(const double *val, const int32_t *col, const double *__restrict__ x, int k0, int k1, double (&part)[kParts]) {
  for (int k = k0; k < k1; k += N)
#pragma unroll
    for (int u = 0; u < N; ++u)
      if (k + u < k1) part[u] = fma(val[k + u], x[col[k + u]], part[u]);
}
__global__ void __launch_bounds__(kThreads, kBlocksPerSm) k_residual_noalloc(int64_t n, const int64_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                                                             const double *__restrict__ av, const double *__restrict__ x,
                                                                             const double *__restrict__ b, double *__restrict__ r,
                                                                             double *__restrict__ norms2, NoAllocScratch *sc) {
  __shared__ double sval[2][kChunk];
  __shared__ int32_t scol[2][kChunk];
  const int t = threadIdx.x, lane = t & 31;
  const int64_t step = (int64_t)gridDim.x * kRows;
  // copies the first chunk of entries [e0, e1) into a buffer
  auto fetch = [&](int buf, int64_t e0, int64_t e1) {
    const int m = (int)(e1 - e0 < kChunk ? e1 - e0 : kChunk);
    for (int k = t; k < m; k += kThreads) {
      cp_async4(&scol[buf][k], ci + e0 + k);
      cp_async8(&sval[buf][k], av + e0 + k);
    }
  };
  auto row_end = [&](int64_t row0) { return row0 + kRows < n ? row0 + kRows : n; };
  double rr = 0.0, bb = 0.0;
  int64_t r0 = (int64_t)blockIdx.x * kRows;
  int64_t e0 = rp[r0], e1 = rp[row_end(r0)];
  int64_t f0 = 0, f1 = 0;  // the entries of the block's next tile
  if (r0 + step < n) { f0 = rp[r0 + step]; f1 = rp[row_end(r0 + step)]; }
  fetch(0, e0, e1);
  for (int buf = 0; r0 < n; r0 += step, buf ^= 1) {
    const int rows = (int)(row_end(r0) - r0);
    const bool mine = t < rows;
    const int64_t a = mine ? rp[r0 + t] : 0, z = mine ? rp[r0 + t + 1] : 0;
    const double bi = mine ? b[r0 + t] : 0.0;
    const bool longrow = z - a > kLongRow;
    double s = 0.0, part[kParts] = {0.0};
    cp_async_wait();
    __syncthreads();  // the tile's first chunk has landed, and the other buffer's readers are through
    int64_t g0 = 0, g1 = 0;
    if (r0 + step < n) fetch(buf ^ 1, f0, f1);
    if (r0 + 2 * step < n) { g0 = rp[r0 + 2 * step]; g1 = rp[row_end(r0 + 2 * step)]; }
    for (int64_t base = e0; base < e1; base += kChunk) {
      const int m = (int)(e1 - base < kChunk ? e1 - base : kChunk);
      if (base > e0) {  // a tile of several chunks reuses its buffer
        __syncthreads();
        fetch(buf, base, e1);
        cp_async_wait();
        __syncthreads();
      }
      const int k0 = (int)((a < base ? base : a < base + m ? a : base + m) - base);
      const int k1 = (int)((z < base ? base : z < base + m ? z : base + m) - base);
      if (z - a <= kShortRow) add_row<4>(sval[buf], scol[buf], x, k0, k1, part);
      else if (!longrow) add_row<kParts>(sval[buf], scol[buf], x, k0, k1, part);
      for (unsigned of = __ballot_sync(0xffffffffu, longrow && k0 < k1); of; of &= of - 1) {
        const int l = __ffs(of) - 1, q0 = __shfl_sync(0xffffffffu, k0, l), q1 = __shfl_sync(0xffffffffu, k1, l);
        double p = 0.0;
#pragma unroll 4
        for (int k = q0 + lane; k < q1; k += 32) p = fma(sval[buf][k], x[scol[buf][k]], p);
        p = warp_sum(p);
        if (lane == l) s += p;
      }
    }
#pragma unroll
    for (int h = kParts / 2; h > 0; h >>= 1)
#pragma unroll
      for (int u = 0; u < h; ++u) part[u] += part[u + h];
    if (mine) {
      const double ri = bi - (longrow ? s : part[0]);
      r[r0 + t] = ri;
      rr += ri * ri;
      bb += bi * bi;
    }
    e0 = f0; e1 = f1; f0 = g0; f1 = g1;
  }
  block_sum2(rr, bb);
  __shared__ int last;
  if (t == 0) {
    sc->partial[2 * blockIdx.x] = rr;
    sc->partial[2 * blockIdx.x + 1] = bb;
    __threadfence();
    last = (atomicAdd(&sc->ticket, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double ta = 0.0, tb = 0.0;
  for (int64_t q = t; q < gridDim.x; q += kThreads) {
    ta += ((volatile double *)sc->partial)[2 * q];
    tb += ((volatile double *)sc->partial)[2 * q + 1];
  }
  block_sum2(ta, tb);
  if (t == 0) {
    norms2[0] = ta;
    norms2[1] = tb;
    sc->ticket = 0;  // ready for the next call
  }
}

// Address of g_scratch on the current device; the first call on a device looks it up and
// clears the ticket counter.
int scratch_for_current_device(NoAllocScratch **out, int *sms) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return VSHE_E_CUDA;
  if (dev < 0 || dev >= kMaxDevices) return VSHE_E_UNSUPPORTED;
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_addr[dev]) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_scratch) != cudaSuccess) return VSHE_E_CUDA;
    NoAllocScratch *s = static_cast<NoAllocScratch *>(p);
    if (cudaMemset(&s->ticket, 0, sizeof(unsigned int)) != cudaSuccess) return VSHE_E_CUDA;
    if (cudaDeviceSynchronize() != cudaSuccess) return VSHE_E_CUDA;
    if (cudaDeviceGetAttribute(&g_sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return VSHE_E_CUDA;
    g_addr[dev] = s;
  }
  *out = g_addr[dev];
  *sms = g_sms[dev];
  return VSHE_OK;
}

}  // namespace

extern "C" int vshe_csr_residual_noalloc(int64_t n, int64_t nnz, const int64_t *d_row_ptr, const int32_t *d_col,
                                         const double *d_val, const double *d_x, const double *d_b, double *d_r,
                                         double *d_norms2, void *stream) {
  if (n <= 0 || nnz < 0 || !d_row_ptr || (nnz > 0 && (!d_col || !d_val)) || !d_x || !d_b || !d_r || !d_norms2)
    return VSHE_E_INVALID_ARGUMENT;
  if (n > kMaxRows || n >= (int64_t(1) << 31)) return VSHE_E_CAPACITY;
  NoAllocScratch *sc = nullptr;
  int sms = 0;
  int rc = scratch_for_current_device(&sc, &sms);
  if (rc) return rc;
  const int64_t tiles = (n + kRows - 1) / kRows, most = int64_t(sms) * kBlocksPerSm < kMaxTiles ? int64_t(sms) * kBlocksPerSm : kMaxTiles;
  const int blocks = int(tiles < most ? tiles : most);
  vk_count_launches(1);
  k_residual_noalloc<<<blocks, kThreads, 0, static_cast<cudaStream_t>(stream)>>>(n, d_row_ptr, d_col, d_val, d_x, d_b, d_r, d_norms2, sc);
  return cudaGetLastError() == cudaSuccess ? VSHE_OK : VSHE_E_CUDA;
}
