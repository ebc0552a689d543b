/*
 * noalloc.cu -- per-cell triangle offsets of one iso-level without any device
 * allocation: contour3d_gb300_cell_offsets_noalloc (include/contour3d_gb300.h).
 *
 * Some callers cannot let a library allocate device memory: an in-situ solver
 * that has reserved the GPU's memory for its own pool (a cudaMalloc would fail
 * or would break the pool's accounting), or a time-stepping loop that must
 * not stall on the implicit device synchronisation of cudaFree.  This entry
 * point serves them.  The caller passes the field and the output arrays; the
 * only other memory the kernel touches -- the tile states of the single-pass
 * scan -- lives in the file-scope array below, which every GPU that loads the
 * library holds (kScratchBytes) until the process exits.
 *
 * The kernel is a single-pass scan with decoupled look-back that computes
 * each cell's triangle count from the field itself (the classification rule
 * of kernels.cu) instead of reading a codes array, so no intermediate buffer
 * is needed.  Tiles are taken in order from an atomic counter, so every tile
 * a block waits on is running or done; the wait is bounded (2^22 polls) and
 * raises an error flag that the host reports.
 *
 * Contract:
 *   - at most kMaxCells cells ((nx-1)(ny-1)(nz-1)); larger fields are
 *     rejected with an error before anything is launched;
 *   - the first call on a device looks up the scratch array's device address
 *     (cudaGetSymbolAddress) with that device current; make that first call
 *     before any stream capture on that device;
 *   - every call shares the one scratch array and clears the part it uses at
 *     its start; calls that overlap on the GPU (other streams, other host
 *     threads) race on it and must be serialised by the caller;
 *   - `stream` must belong to the current device (checked);
 *   - every call copies the 4-byte error word back to the host and
 *     synchronises `stream` before it returns, so the return code covers the
 *     device work too;
 *   - the cached device address is only valid for the device context it was
 *     taken in: the library must not be used across a cudaDeviceReset;
 *   - no cudaMalloc, cudaFree or allocating library routine is called.
 */
#include <cuda_runtime.h>
#include <cuda/atomic>
#include <cmath>
#include <cstdint>
#include <mutex>
#include "contour3d_gb300.h"
#include "c3d_common.cuh"
#include "c3d_host.h"
#include "c3d_kernels.h"

namespace {

constexpr int kThreads = 256;
constexpr long long kTile = kThreads * 32;
constexpr long long kMaxTiles = 1 << 15;
/* the scan also writes the offset after the last cell, so tiles cover n + 1 positions */
constexpr long long kMaxCells = kMaxTiles * kTile - 1;
constexpr int kMaxDevices = 64;
constexpr unsigned long long kAgg = 1ULL << 62;
constexpr unsigned long long kPrefix = 2ULL << 62;
constexpr unsigned long long kValue = (1ULL << 62) - 1;
constexpr unsigned kErrTimeout = 1u;

/* word 0: tile counter, word 1: error flags, words 2..: one state per tile */
constexpr size_t kScratchWords = 2 + (size_t)kMaxTiles;
constexpr size_t kScratchBytes = kScratchWords * sizeof(unsigned long long);
static __device__ __align__(256) unsigned long long g_scratch[kScratchWords];

/* the field's layout and its threshold as a key range (ThrSet); cells and
   nodes number fewer than 2^32 */
struct Grid {
  const void* data;
  unsigned nx, ny, ncx, ncy;
  unsigned nnodes;
  unsigned long long lo, cnt; /* of the type's key width */
};

template <typename T>
struct Bits;
template <>
struct Bits<double> {
  typedef long long type;
};
template <>
struct Bits<float> {
  typedef int type;
};
/* a node's value as its bit pattern, and the threshold test on it */
template <typename T>
__device__ __forceinline__ typename Bits<T>::type node(const Grid& g, unsigned idx) {
  return __ldg(static_cast<const typename Bits<T>::type*>(g.data) + idx);
}
__device__ __forceinline__ bool above(const Grid& g, long long b) {
  const long long key = b ^ (long long)((unsigned long long)(b >> 63) >> 1);
  return (unsigned long long)key - g.lo < g.cnt;
}
__device__ __forceinline__ bool above(const Grid& g, int b) {
  const int key = b ^ (int)((unsigned)(b >> 31) >> 1);
  return (unsigned)key - (unsigned)g.lo < (unsigned)g.cnt;
}

/* the node at corner 0 of cell c */
__device__ __forceinline__ unsigned corner_node(const Grid& g, unsigned c, unsigned& i, unsigned& j) {
  const unsigned row = c / g.ncx, k = row / g.ncy;
  i = c - row * g.ncx;
  j = row - k * g.ncy;
  return (k * g.ny + j) * g.nx + i;
}

/* a + b + c bit by bit: the sum's low and high bits */
__device__ __forceinline__ void add3(unsigned a, unsigned b, unsigned c, unsigned& lo, unsigned& hi) {
  lo = a ^ b ^ c;
  hi = (a & b) | (a & c) | (b & c);
}

/*
 * The triangle counts of 32 cells from their corner bits (bit q of w[c]:
 * corner c of cell q is above the threshold), as four words of count bits
 * (bit q of k[b]: bit b of cell q's count).  Of the six tetrahedra sharing
 * the 0-7 diagonal (triangulate.c:145-270), one with an odd number of corners
 * above has one triangle, one with two has two.
 */
__device__ __forceinline__ void count_words(const unsigned w[8], unsigned k[4]) {
  constexpr int tet[6][2] = {{3, 1}, {1, 5}, {5, 4}, {4, 6}, {6, 2}, {2, 3}};
  unsigned one[6], two[6];
#pragma unroll
  for (int t = 0; t < 6; t++) {
    const unsigned p = w[0], q = w[7], r = w[tet[t][0]], s = w[tet[t][1]];
    one[t] = p ^ q ^ r ^ s;
    two[t] = ((p ^ q) | (p ^ r) | (p ^ s)) & ~one[t];
  }
  unsigned a0, a1, b0, b1, c0, c1, d0, d1, e0, e1, f0, f1;
  add3(one[0], one[1], one[2], a0, a1);
  add3(one[3], one[4], one[5], b0, b1);
  add3(two[0], two[1], two[2], c0, c1);
  add3(two[3], two[4], two[5], d0, d1);
  k[0] = a0 ^ b0;
  add3(a1, b1, a0 & b0, e0, e1); /* weight 2, carry 4 */
  add3(c0, d0, e0, k[1], f1);    /* carry 4 */
  add3(c1, d1, e1, f0, d0);      /* weight 4, carry 8 */
  k[2] = f0 ^ f1;
  k[3] = d0 ^ (f0 & f1); /* at most 12: no further carry */
}

/*
 * One tile of kTile consecutive cells per block, 32 of them per thread.
 *
 * BITS: the tile's cells lie between two node numbers, and so do the four
 * node rows that they touch; each of the two z-planes of that range is read
 * once, coalesced, and kept as one bit per node (a warp ballot per 32 nodes)
 * in shared memory.  A thread shifts its 32 cells' eight corner words out of
 * them (a piece per row that its cells touch) and counts all 32 cells'
 * triangles at once in bit-sliced sums (count_words).  Without BITS (rows so
 * long that a tile's node range does not fit, see kCapNodes): eight coalesced
 * loads and ballots per 32 cells make the corner words.
 *
 * The offsets go out one cell per lane: the running offset of the thread's 32
 * cells plus the count bits below the lane, so every store of a warp covers
 * 128 contiguous bytes.
 *
 * The bytes it cannot do without take 35 us at 389 x 301 x 257 f32.  There,
 * the whole call took 1.09 ms with eight strided loads and two 64-bit
 * divisions per cell, 185 us with a cell per lane on the bit planes (issue
 * slots: about 80 instructions per 32 cells), 115 us as here (the
 * kernel 95 us of them; 16 loads in flight per lane: 116 us).
 */
constexpr int kWarps = kThreads / 32;
constexpr int kLoads = 8;                                 /* node words per warp and round */
constexpr unsigned kCapNodes = 4 * (unsigned)kTile + 256; /* nodes of one plane kept as bits */
constexpr int kCapWords = (int)(kCapNodes / 32) + 1;      /* the last one is read by a funnel shift only */
static_assert(kTile == 32 * kThreads, "a thread has one word of cells");

template <typename T, bool BITS>
__global__ void __launch_bounds__(kThreads)
k_offsets_noalloc(Grid g, unsigned n, unsigned* __restrict__ offsets, unsigned long long* __restrict__ total,
                  unsigned long long* __restrict__ scratch) {
  __shared__ unsigned s_tile;
  __shared__ unsigned s_warp[kWarps];
  __shared__ unsigned long long s_excl;
  __shared__ unsigned s_bits[BITS ? 2 : 8][BITS ? kCapWords : kThreads]; /* node bits, or corner words */
  __shared__ uint4 s_count[kThreads];                                      /* count bits of each word of cells */
  __shared__ unsigned s_rel[kThreads];                                     /* its first offset in the warp */
  unsigned* counter = reinterpret_cast<unsigned*>(scratch);
  unsigned* err = reinterpret_cast<unsigned*>(scratch + 1);
  unsigned long long* state = scratch + 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1u);
  __syncthreads();
  const unsigned tile = s_tile;
  const unsigned c0 = tile * (unsigned)kTile;
  const unsigned c1 = c0 + (unsigned)kTile < n ? c0 + (unsigned)kTile : n; /* cells [c0, c1): none in a tile of position n alone */
  const unsigned sxy = g.nx * g.ny;
  unsigned cw[8] = {0, 0, 0, 0, 0, 0, 0, 0}; /* corner words; cells past c1 stay all below */
  if (BITS) {
    unsigned i, j;
    unsigned first = 0;
    if (c0 < c1) {
      first = corner_node(g, c0, i, j);
      /* nodes first .. (last cell's corner 0) + nx + 1 of each plane; the host
         checked that they fit (kCapNodes) */
      const unsigned nodes = corner_node(g, c1 - 1, i, j) - first + g.nx + 2;
      const unsigned words = (nodes + 31) / 32;
#pragma unroll
      for (int p = 0; p < 2; p++) {
        const unsigned base = first + (p ? sxy : 0u);
        for (unsigned w0 = warp * kLoads; w0 < words; w0 += kWarps * kLoads) {
          /* kLoads loads in flight; those past the range or the field read the last node */
          typename Bits<T>::type v[kLoads];
#pragma unroll
          for (int u = 0; u < kLoads; u++)
            v[u] = node<T>(g, min(base + 32 * min(w0 + u, words - 1) + lane, g.nnodes - 1));
          unsigned m = 0;
#pragma unroll
          for (int u = 0; u < kLoads; u++) {
            const unsigned x = __ballot_sync(0xFFFFFFFFu, above(g, v[u]));
            if (lane == u) m = x;
          }
          if (lane < kLoads && w0 + lane < words) s_bits[p][w0 + lane] = m;
        }
      }
    }
    __syncthreads();
    unsigned c = c0 + 32 * threadIdx.x, at = 0;
    if (c < c1) at = corner_node(g, c, i, j);
    for (unsigned pos = 0; pos < 32 && c < c1;) {
      /* the cells of one row: `len` of them from bit `pos` on */
      const unsigned len = min(min(32 - pos, g.ncx - i), c1 - c);
      const unsigned keep = 0xFFFFFFFFu >> (32 - len);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const unsigned rel = at - first + ((q & 1) ? g.nx : 0u);
        const unsigned lo = s_bits[q >> 1][rel >> 5], hi = s_bits[q >> 1][(rel >> 5) + 1];
        const unsigned x0 = __funnelshift_r(lo, hi, rel & 31);
        const unsigned x1 = __funnelshift_r(x0, hi >> (rel & 31), 1);
        cw[2 * q] |= (x0 & keep) << pos;
        cw[2 * q + 1] |= (x1 & keep) << pos;
      }
      pos += len;
      c += len;
      i += len;
      at += len;
      if (i == g.ncx) { /* a node more per row end, a row more per slice end */
        i = 0;
        at++;
        if (++j == g.ncy) {
          j = 0;
          at += g.nx;
        }
      }
    }
  } else {
    for (int s = 0; s < 32; s++) {
      const unsigned c = c0 + 1024 * warp + 32 * s + lane;
      unsigned i, j, at = 0;
      if (c < c1) at = corner_node(g, c, i, j);
      typename Bits<T>::type v[8];
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] = node<T>(g, at + (q & 1) + ((q >> 1) & 1) * g.nx + (q >> 2) * sxy);
      unsigned m = 0;
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const unsigned x = __ballot_sync(0xFFFFFFFFu, c < c1 && above(g, v[q]));
        if (lane == q) m = x;
      }
      if (lane < 8) s_bits[lane][32 * warp + s] = m;
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 8; q++) cw[q] = s_bits[q][threadIdx.x];
  }
  unsigned k[4];
  count_words(cw, k);
  const unsigned sum = __popc(k[0]) + 2 * __popc(k[1]) + 4 * __popc(k[2]) + 8 * __popc(k[3]);
  unsigned incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
    if (lane >= d) incl += y;
  }
  s_count[threadIdx.x] = make_uint4(k[0], k[1], k[2], k[3]);
  s_rel[threadIdx.x] = incl - sum;
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  unsigned agg = 0, before = 0; /* the tile's triangles, and those of earlier warps */
#pragma unroll
  for (int w = 0; w < kWarps; w++) {
    if (w < warp) before += s_warp[w];
    agg += s_warp[w];
  }
  if (warp == 0) {
    cuda::atomic_ref<unsigned long long, cuda::thread_scope_device> mine(state[tile]);
    if (lane == 0) mine.store((tile == 0 ? kPrefix : kAgg) | agg, cuda::memory_order_release);
    unsigned long long excl = 0;
    if (tile > 0) {
      long long pred = (long long)tile - 1;
      int spins = 0;
      bool done = false;
      while (!done) {
        const long long p = pred - lane;
        unsigned long long st = 0;
        if (p >= 0) {
          cuda::atomic_ref<unsigned long long, cuda::thread_scope_device> ps(state[p]);
          st = ps.load(cuda::memory_order_acquire);
        }
        const unsigned invalid = __ballot_sync(0xFFFFFFFFu, p >= 0 && (st >> 62) == 0);
        const unsigned prefix = __ballot_sync(0xFFFFFFFFu, p >= 0 && (st >> 62) == 2);
        const unsigned fi = invalid ? __ffs(invalid) - 1 : 32;
        const unsigned fp = prefix ? __ffs(prefix) - 1 : 32;
        unsigned take = 0;
        if (fp < fi) {
          take = fp + 1;
          done = true;
        } else if (fi > 0) {
          take = fi;
        }
        if (take) {
          unsigned long long v = (lane < (int)take && p >= 0) ? (st & kValue) : 0;
#pragma unroll
          for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, d);
          excl += v;
          pred -= take;
          if (pred < 0) done = true;
        } else if (++spins > (1 << 22)) {
          if (lane == 0) atomicOr(err, kErrTimeout);
          done = true;
        } else {
          __nanosleep(64);
        }
      }
      if (lane == 0) mine.store(kPrefix | ((excl + agg) & kValue), cuda::memory_order_release);
    }
    if (lane == 0) s_excl = excl;
  }
  __syncthreads();
  const unsigned long long base = s_excl + before;
  const unsigned below = (1u << lane) - 1u;
#pragma unroll 4
  for (int s = 0; s < 32; s++) {
    const unsigned c = c0 + 1024 * warp + 32 * s + lane;
    const uint4 q = s_count[32 * warp + s];
    const unsigned long long off = base + s_rel[32 * warp + s] + __popc(q.x & below) + 2 * __popc(q.y & below) +
                                   4 * __popc(q.z & below) + 8 * __popc(q.w & below);
    if (c <= n) offsets[c] = (unsigned)off;
    if (c == n) *total = off;
  }
}

std::mutex g_mu;
unsigned long long* g_scratch_ptr[kMaxDevices] = {};

template <typename T, bool BITS>
void launch(const Grid& g, unsigned n, unsigned tiles, unsigned* offsets, unsigned long long* total,
            unsigned long long* scratch, cudaStream_t st) {
  k_offsets_noalloc<T, BITS><<<tiles, kThreads, 0, st>>>(g, n, offsets, total, scratch);
}

}  // namespace

extern "C" int contour3d_gb300_cell_offsets_noalloc(const void* device_field, int dtype, const size_t sizes[3],
                                                    double threshold, uint32_t* device_offsets,
                                                    unsigned long long* device_total, void* stream) {
  if (!device_field || !sizes || !device_offsets || !device_total ||
      (dtype != CONTOUR3D_GB300_F64 && dtype != CONTOUR3D_GB300_F32)) {
    c3d::log_error("cell_offsets_noalloc: null pointer or unknown dtype");
    return 1;
  }
  if (sizes[0] < 2 || sizes[1] < 2 || sizes[2] < 2) {
    c3d::log_error("cell_offsets_noalloc: every size must be at least 2 nodes");
    return 1;
  }
  const double cells = (double)(sizes[0] - 1) * (double)(sizes[1] - 1) * (double)(sizes[2] - 1);
  if (cells > (double)kMaxCells) {
    c3d::log_error("cell_offsets_noalloc: %.0f cells exceed the no-allocation limit of %lld cells "
                   "(%zu bytes of static scratch); use contour3d_gb300_render_device instead",
                   cells, kMaxCells, kScratchBytes);
    return 1;
  }
  const long long n = (long long)(sizes[0] - 1) * (long long)(sizes[1] - 1) * (long long)(sizes[2] - 1);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    c3d::log_error("cell_offsets_noalloc: no usable current device");
    return 1;
  }
  unsigned long long* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_scratch_ptr[dev]) {
      /* once per device, with that device current: the host-side name of the
         array is not its device address */
      void* p = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&p, g_scratch);
      if (e != cudaSuccess || !p) {
        c3d::log_error("cell_offsets_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
        return 1;
      }
      g_scratch_ptr[dev] = static_cast<unsigned long long*>(p);
    }
    scratch = g_scratch_ptr[dev];
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (st) {
    int sdev = -1;
    if (cudaStreamGetDevice(st, &sdev) != cudaSuccess || sdev != dev) {
      cudaGetLastError();
      c3d::log_error("cell_offsets_noalloc: the stream does not belong to the current device %d", dev);
      return 1;
    }
  }
  const long long tiles = (n + kTile) / kTile;
  /* the counter, the error word and the tile states this call uses start at zero */
  if (cudaMemsetAsync(scratch, 0, sizeof(unsigned long long) * (size_t)(2 + tiles), st) != cudaSuccess) {
    c3d::log_error("cell_offsets_noalloc: clearing the scratch failed");
    return 1;
  }
  /* the threshold as a key range of the field's type */
  c3d::FieldDev F = {};
  c3d::set_threshold(F, threshold);
  c3d::ThrSet ts;
  c3d::thr_range(F, ts, 0);
  const bool f64 = dtype == CONTOUR3D_GB300_F64;
  Grid g;
  g.data = device_field;
  g.nx = (unsigned)sizes[0];
  g.ny = (unsigned)sizes[1];
  g.ncx = g.nx - 1;
  g.ncy = g.ny - 1;
  g.nnodes = (unsigned)(sizes[0] * sizes[1] * sizes[2]);
  g.lo = f64 ? ts.lo[0] : ts.flo[0];
  g.cnt = f64 ? ts.cnt[0] : ts.fcnt[0];
  /* the most nodes of one plane that a tile touches: its cells, one more per
     row end, a row more per slice end, and the rows above and to the right.
     Rows of up to about 12,000 nodes fit in bits */
  const long long row_ends = kTile / g.ncx + 1, slice_ends = kTile / ((long long)g.ncx * g.ncy) + 1;
  const bool bits = kTile + row_ends + slice_ends * g.nx + g.nx + 2 <= (long long)kCapNodes;
  if (f64 && bits) launch<double, true>(g, (unsigned)n, (unsigned)tiles, device_offsets, device_total, scratch, st);
  else if (f64) launch<double, false>(g, (unsigned)n, (unsigned)tiles, device_offsets, device_total, scratch, st);
  else if (bits) launch<float, true>(g, (unsigned)n, (unsigned)tiles, device_offsets, device_total, scratch, st);
  else launch<float, false>(g, (unsigned)n, (unsigned)tiles, device_offsets, device_total, scratch, st);
  cudaError_t e = cudaGetLastError();
  unsigned errw = 0;
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&errw, scratch + 1, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    c3d::log_error("cell_offsets_noalloc: %s", cudaGetErrorString(e));
    return 1;
  }
  if (errw) {
    c3d::log_error("cell_offsets_noalloc: the device scan did not complete (flags 0x%x)", errw);
    return 1;
  }
  return 0;
}
