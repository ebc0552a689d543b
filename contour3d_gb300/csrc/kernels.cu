/*
 * kernels.cu -- sm_103a kernels of the isosurface-to-image path.
 *
 * The contour objects of one field are classified together, then each
 * object is processed in z-slabs of cells, then shaded once:
 *   k_classify_tma  cell codes of up to four thresholds per pass over the
 *                   field (TMA node planes; k_classify_multi where TMA cannot
 *                   address the field)                         (HBM: field read)
 * per slab of an object:
 *   k_scan          packed (triangle, vertex) counts per segment of cells,
 *                   the segment's prefix by decoupled look-back, a word per
 *                   crossed cell and the triangle -> cell map, in one pass
 *   k_vertices      one FP32 screen vertex per crossed edge, with certified
 *                   bounds (two FP64 subtractions per vertex)
 *   k_emit          one thread per triangle: its three vertices through their
 *                   owner cells, culling, and the raster route (cover list,
 *                   by one pixel or a range of them, sliver list, tiny list,
 *                   or dropped)
 *   k_raster        one thread per listed triangle, over the cover list
 *                   and then the sliver list: FP32 coverage and depth
 *                   intervals over its pixel range; certainly drawn
 *                   fragments raise a per-pixel depth floor, the rest become
 *                   candidates; slivers (area the reference may clamp) the
 *                   bounds cannot settle go to the tiny list
 *   k_finish        drops candidates below the final depth floor, settles what
 *                   float pairs can of the others (inside or not, the depth
 *                   within 2^-20, a 128-bit max into the z-buffer) and lists
 *                   the rest; in frames whose depths are exact the reference's
 *                   FP64 test instead
 *   k_exact         the listed fragments and the tiny-list triangles, four lanes
 *                   each (a lane each of more fragments than that fills): the
 *                   reference's vertices (recomputed from the field),
 *                   projection, barycentric test and harmonic depth in FP64
 * per object, after its slabs:
 *   k_winners       the pixels the object owns, by patches
 *   k_shade_f       FP32 vertex normals and colour with certified bounds
 *                   (block-shared triangle normals)
 *   k_shade_amb     the reference's FP64 colour for the pixels FP32 cannot
 *                   settle: neighbour triangles in normal.c's order, their
 *                   weighted normals, ordered sums and the shading
 *   k_nb_list, k_nb_wn, k_shade
 *                   the same in three launches for every pixel of a field
 *                   with a converter
 * and once per frame k_canvas_init, k_lines and k_resolve.  k_exact_all and
 * k_normals compute every triangle's exact data for inspection only.
 *
 * The FP64 work runs on compacted lists so that warps stay converged: on GB300 an FP64 warp instruction costs the same whether 2
 * or 32 lanes are active.  Exact vertices are needed only for fragments that
 * can win, and weighted normals only around the triangles that finally own a
 * pixel, so they are computed for those alone.
 *
 * Reference correspondence (file:line of the reference tree):
 *   k_classify*, scan, k_emit   src/contour3d/contour/triangulate.c:95-342
 *   k_vertices, exact vertices  src/contour3d/contour/triangulate.c:40-73
 *   k_shade_f, k_shade_amb, k_nb_*, k_shade, k_normals
 *                               src/contour3d/contour/normal.c:6-165
 *   k_raster, k_finish, k_exact, shading factor
 *                               src/contour3d/contour/render.c:38-163,
 *                               src/contour3d/project.c:9-67
 *   k_lines                     src/contour3d/line.c:26-119
 *   k_resolve                   src/contour3d/output.c:10-30, 113-123
 *   slab / interior             src/contour3d/contour/main.c:38-112
 */
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <type_traits>
#include <cuda/atomic>
#include "c3d_common.cuh"
#include "c3d_cover.cuh"
#include "c3d_kernels.h"

namespace c3d {

__constant__ unsigned char c_code_count[256];
/* normal.c:78-158: per cube edge, the (dk, dj, di, local edge id) of the
   cells sharing it, in the reference's accumulation order */
__constant__ signed char c_nb[19][4][4];
__constant__ unsigned char c_nb_count[19];
/* per code and cube edge: bit r set when the cell's triangle of rank r has
   a vertex on that edge (read by lanes with different codes: global, cached) */
__device__ unsigned short g_edge_tris[256 * 19];

/* ------------------------------------------------------------------ */
/* field access                                                        */
/* ------------------------------------------------------------------ */
template <typename T>
__device__ __forceinline__ double load_value(const T* f, long long idx) {
  return (double)__ldg(f + idx);
}
template <>
__device__ __forceinline__ double load_value<double>(const double* f, long long idx) {
  return __longlong_as_double(ld_bits(f + idx));
}

/* bit c of the result: threshold < value at corner c of cell (i, j, k) */
template <typename T>
__device__ __forceinline__ unsigned cell_code(const FieldDev& F, long long i, long long j, long long k,
                                              double vals[8]) {
  const T* f = static_cast<const T*>(F.data);
  const long long sx = 1, sy = F.nx, sz = F.nx * F.ny;
  const long long base = k * sz + j * sy + i;
  unsigned code = 0;
  const long long tk = F.thr_key;
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const long long idx = base + ((c & 1) ? sx : 0) + ((c & 2) ? sy : 0) + ((c & 4) ? sz : 0);
    const double v = load_value<T>(f, idx);
    vals[c] = v;
    const bool above = !F.thr_nan && !d_isnan(v) && d_key(v) > tk;
    code |= (unsigned)above << c;
  }
  return code;
}

__device__ __forceinline__ unsigned fast_div(unsigned n, const FastDiv& d) {
  const unsigned t = __umulhi(d.m, n);
  return (t + ((n - t) >> d.s1)) >> d.s2;
}

/* cell (i, j, k-in-slab) of a slab-local linear cell index; 32-bit arithmetic */
__device__ __forceinline__ void cell_ijk(const FieldDev& F, unsigned c, unsigned& i, unsigned& j, unsigned& kl) {
  const unsigned ncx = (unsigned)(F.nx - 1), ncy = (unsigned)(F.ny - 1);
  const unsigned r = fast_div(c, F.div_cx);
  i = c - r * ncx;
  kl = fast_div(r, F.div_cy);
  j = r - kl * ncy;
}

/* ------------------------------------------------------------------ */
/* counts per cell                                                     */
/* ------------------------------------------------------------------ */
/*
 * Per cell, its triangle count and the number of its owned vertices (edges
 * from its corner 0 that the iso-level crosses), packed as tri | vert << 31:
 * every sum over a slab stays below 2^31 in both fields for slabs of at most
 * kMaxSlabCells cells, so packed additions never carry.  The scan runs over
 * segments of kScanTile cells, one block each (k_scan).
 *
 * Vertices are owned by cells: cell c owns the crossed edges that start at
 * its corner 0 and run to corner m = 1..7 (+x, +y, +x+y, +z, +x+z, +y+z,
 * +x+y+z).  Every edge of the six-tetrahedra split joins corners a, b with
 * a & b = a or b, so it starts at corner a & b of its cell and runs in
 * direction a ^ b: it is the edge m = a ^ b owned by the cell at offset a & b.
 */
constexpr int kScanThreads = 256;
constexpr int kScanItems = 32;  /* cells per thread */
constexpr int kScanTile = kScanThreads * kScanItems;
static_assert(kScanTile == 1 << kVSegShift, "the words' offsets are relative to scan segments");
static_assert(kScanTile == 8192, "a slot's 12 bits name a cell of half a segment");
constexpr unsigned long long kTriMask = (1ULL << 31) - 1;

/* the vertex offset of cell c */
__device__ __forceinline__ unsigned voff_at(const VOffDev& o, long long c) {
  return o.seg[c >> kVSegShift] + (o.word[c] & 0xFFFFu);
}

/* bit m - 1: the iso-level crosses edge m of the cell's corner 0 */
__device__ __forceinline__ unsigned owned_edges(unsigned code) {
  const unsigned flip = code ^ (0u - (code & 1u));
  return (flip >> 1) & 0x7Fu;
}

/* triangles | vertices << 16 of every code, in shared memory */
__device__ __forceinline__ void load_count_lut(unsigned* lut) {
  for (int q = threadIdx.x; q < 256; q += blockDim.x)
    lut[q] = (unsigned)c_code_count[q] | ((unsigned)__popc(owned_edges((unsigned)q)) << 16);
}


/* ------------------------------------------------------------------ */
/* cell codes                                                          */
/* ------------------------------------------------------------------ */
/*
 * Tiled over (x, y) and marching in z: each node's "above" bit is computed
 * once per brick into shared memory (two planes, double-buffered), and a cell's
 * 8-bit code is assembled from the bits of its corners.  The codes are
 * kept: the scan maps them to triangle counts, and the later passes read
 * them instead of comparing the eight corner values again.  A block owns
 * kClsX x kClsY cells of kClsZ consecutive slices.
 */
constexpr int kClsX = 128;
constexpr int kClsY = 8;
constexpr int kClsZ = 32; /* default slices per brick (LaunchShape::cls_z) */

template <typename T>
__device__ __forceinline__ unsigned char node_above(const FieldDev& F, const T* f, long long idx);
template <>
__device__ __forceinline__ unsigned char node_above<double>(const FieldDev& F, const double* f, long long idx) {
  const long long b = ld_bits(f + idx);
  return (!F.thr_nan && !d_isnan_bits(b) && d_key_bits(b) > F.thr_key) ? 1 : 0;
}
template <>
__device__ __forceinline__ unsigned char node_above<float>(const FieldDev& F, const float* f, long long idx) {
  /* threshold < (double)v  <=>  v >= the least float above the threshold */
  const float v = __ldg(f + idx);
  return (F.thr_f_ok && v == v && f_key(v) >= F.thr_f_key) ? 1 : 0;
}

/* the same test against threshold t of a set (k_classify_tma classifies the
   objects of one field together), on the value's bit pattern: the
   sign-folded key, then one unsigned range check (ThrSet) */
template <typename T>
struct NodeBits;
template <>
struct NodeBits<double> {
  using type = long long;
};
template <>
struct NodeBits<float> {
  using type = int;
};
__device__ __forceinline__ long long fold_key(long long b) { return b ^ (long long)((unsigned long long)(b >> 63) >> 1); }
__device__ __forceinline__ int fold_key(int b) { return b ^ (int)((unsigned)(b >> 31) >> 1); }
__device__ __forceinline__ bool key_above(const ThrSet& ts, int t, long long key) {
  return (unsigned long long)key - ts.lo[t] < ts.cnt[t];
}
__device__ __forceinline__ bool key_above(const ThrSet& ts, int t, int key) {
  return (unsigned)key - ts.flo[t] < ts.fcnt[t];
}

constexpr int kClsWords = kClsX / 32 + 1; /* of a row's node bits */

/*
 * Codes of a brick (kClsX x kClsY cells from (i0, j0) on) from its planes'
 * node bits, m[row][threshold], where word w holds the nodes x = 32w .. 32w +
 * 31 of the row and word kClsX / 32 the node x = kClsX.  A warp takes rows
 * warp and warp + 4, a lane the four cells from x = 4 lane on.
 *
 * A plane's part of the codes is four bits per byte: a funnel shift gives a
 * row's five node bits around the four cells, and one multiply puts bits q and
 * q + 1 into byte q (copies of five bits, seven places apart, do not meet).  A
 * slice's codes join the parts of the planes below (kept from the last call)
 * and above it.  A row of codes starts at any offset from a 4-byte boundary, so
 * each lane takes the bytes its neighbour has beyond the boundary and stores
 * one aligned word; the up to three cells before the first boundary and after
 * the last one are stored as bytes.
 *
 * Issue slots bound the classification.  A cell per lane, with its own shifts
 * in both planes and a byte per store, took 321 us on a 512^3 double field of
 * two levels (556 instructions per warp and plane), 579 us per slab of a 1536^3
 * float one of four, 168 us at 313 x 269 x 311 double and three; this 286, 478
 * and 115.
 */
template <int NT>
struct HalfCodes {
  unsigned h[2][NT]; /* a plane's part: rows warp and warp + 4 */
};

/* the plane m above slice kl (and below the next one): stores the slice's
   codes, unless `first`, and keeps the plane's part in `below` */
template <int NT>
__device__ __forceinline__ void plane_codes(const unsigned (*m)[NT][kClsWords], HalfCodes<NT>& below, bool first,
                                            unsigned char* const* codes, int nt, long long kl, unsigned i0,
                                            unsigned j0, unsigned ncx, unsigned ncy) {
  static_assert(kClsX == 128 && kClsY == 8, "a warp per row, four cells per lane, two rows each");
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, w = lane >> 3, sh = 4 * (lane & 7u);
  const unsigned width = min((unsigned)kClsX, ncx - i0);
#pragma unroll
  for (unsigned g = 0; g < 2; g++) {
    const unsigned j = j0 + warp + 4 * g;
    if (j >= ncy) break;
    const unsigned long long row = ((unsigned long long)kl * ncy + j) * ncx + i0;
    const unsigned s = (0u - (unsigned)row) & 3u, x = 4 * lane + s; /* codes[t] is aligned */
    const bool part = (x < width && x + 4 > width) || (lane == 0 && s != 0);
#pragma unroll
    for (int t = 0; t < NT; t++) {
      if (t >= nt) break;
      auto two = [&](unsigned r) {
        return ((__funnelshift_r(m[r][t][w], m[r][t][w + 1], sh) & 31u) * 0x00204081u) & 0x03030303u;
      };
      const unsigned here = two(warp + 4 * g) | (two(warp + 4 * g + 1) << 2);
      const unsigned own = below.h[g][t] | (here << 4);
      below.h[g][t] = here;
      if (first) continue;
      const unsigned next = __shfl_down_sync(0xFFFFFFFFu, own, 1), four = __funnelshift_r(own, next, 8 * s);
      unsigned char* to = codes[t] + row;
      if (x + 4 <= width) *reinterpret_cast<unsigned*>(to + x) = four;
      if (part) {
#pragma unroll
        for (unsigned q = 0; q < 3; q++) {
          if (lane == 0 && q < s && q < width) to[q] = (unsigned char)(own >> (8 * q));
          if (x + 4 > width && x + q < width) to[x + q] = (unsigned char)(four >> (8 * q));
        }
      }
    }
  }
}

/*
 * k_classify_queue: the cell codes of many fields (the frames of a batch) in
 * one launch of a persistent grid.  A work item is one field with up to
 * kMaxThr thresholds; its bricks are numbered item by item
 * (ClsItem::first).  Each block takes the next brick number from a device
 * counter, finds its item by binary search over the items' first numbers,
 * and classifies that brick for all of the item's thresholds in one pass
 * over its nodes.  The values of the next plane are loaded into registers
 * before the current plane pair is turned into codes, so the loads are in
 * flight during that work; a thread holds a column of the plane's rows, and
 * its warp's ballots are the rows' node bits (plane_codes).  Every brick number
 * is taken once, so the loop ends after at most nunits / grid bricks per
 * block.
 */
/* what a block keeps of its current item, in shared memory */
struct QueueBrick {
  const void* data;
  unsigned char* codes[kMaxThr];
  long long nx, ny, kfirst, k0, k1;
  unsigned i0, j0, ncx, ncy;
  int nt;
};

/* a plane's node bits.  A brick keeps two: slow warps may read one plane's while
   the others write the next one's, so one barrier per plane is enough */
typedef unsigned QueueMask[kClsY + 1][kMaxThr][kClsWords];

template <typename T>
__device__ __forceinline__ void classify_queue_brick(const QueueBrick& qb, const ThrSet& ts, QueueMask* mask) {
  using K = typename NodeBits<T>::type;
  const K* __restrict__ f = static_cast<const K*>(qb.data);
  const long long nx = qb.nx, ny = qb.ny, sxy = nx * ny;
  const unsigned i0 = qb.i0, j0 = qb.j0;
  const long long k0 = qb.k0, k1 = qb.k1, kfirst = qb.kfirst;
  const int nt = qb.nt;
  const unsigned tx = threadIdx.x, lane = tx & 31u, warp = tx >> 5;
  /* this thread's column of the plane's rows, and for threads 0 .. kClsY of
     warp 0 a node of column kClsX (nodes beyond the field read as 0: they
     belong to no cell) */
  const unsigned rows = (unsigned)min((long long)(kClsY + 1), ny - j0);
  const bool in_x = i0 + tx < nx, edge = tx < rows && i0 + kClsX < nx;
  const long long column = (long long)j0 * nx + i0 + tx, corner = (long long)(j0 + tx) * nx + i0 + kClsX;
  K v[kClsY + 1], ve = K(0);
  auto fetch = [&](long long k) {
    const K* plane = f + k * sxy;
#pragma unroll
    for (unsigned r = 0; r <= (unsigned)kClsY; r++) v[r] = in_x && r < rows ? __ldg(plane + column + r * nx) : K(0);
    ve = edge ? __ldg(plane + corner) : K(0);
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int r = 0; r <= kClsY; r++) v[r] = fold_key(v[r]);
    ve = fold_key(ve);
    for (int t = 0; t < nt; t++) {
#pragma unroll
      for (int r = 0; r <= kClsY; r++) {
        const unsigned m = __ballot_sync(0xFFFFFFFFu, key_above(ts, t, v[r]));
        if (lane == (unsigned)r) mask[buf][r][t][warp] = m;
      }
      if (tx <= (unsigned)kClsY) mask[buf][tx][t][kClsWords - 1] = key_above(ts, t, ve) ? 1u : 0u;
    }
  };
  HalfCodes<kMaxThr> below = {};
  fetch(kfirst + k0);
  store(0);
  fetch(kfirst + k0 + 1);
  __syncthreads();
  plane_codes<kMaxThr>(mask[0], below, true, qb.codes, nt, 0, i0, j0, qb.ncx, qb.ncy);
  for (long long kl = k0; kl < k1; kl++) {
    const int buf = (int)((kl - k0 + 1) & 1);
    store(buf); /* node plane kl + 1 */
    __syncthreads();
    if (kl + 1 < k1) fetch(kfirst + kl + 2);
    plane_codes<kMaxThr>(mask[buf], below, false, qb.codes, nt, kl, i0, j0, qb.ncx, qb.ncy);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kClsX, 5)
k_classify_queue(const ClsItem* __restrict__ items, int nitems, unsigned long long nunits,
                 unsigned long long* __restrict__ next) {
  pdl_enter();
  __shared__ QueueMask mask[2];
  __shared__ QueueBrick s_qb;
  __shared__ ThrSet s_ts;
  __shared__ int s_item;
  __shared__ unsigned long long s_unit;
  for (;;) {
    if (threadIdx.x == 0) {
      const unsigned long long u = atomicAdd(next, 1ULL);
      s_unit = u;
      if (u < nunits) {
        int lo = 0, hi = nitems - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (items[mid].first <= u) lo = mid;
          else hi = mid - 1;
        }
        const ClsItem& it = items[lo];
        const unsigned long long r = u - it.first;
        const unsigned bx = (unsigned)(r % it.nbx), by = (unsigned)((r / it.nbx) % it.nby);
        const unsigned bz = (unsigned)(r / ((unsigned long long)it.nbx * it.nby));
        s_item = lo;
        s_qb.data = it.data;
        for (int t = 0; t < kMaxThr; t++) s_qb.codes[t] = it.out.codes[t];
        s_qb.nx = it.nx;
        s_qb.ny = it.ny;
        s_qb.kfirst = it.S.kfirst;
        s_qb.k0 = (long long)bz * it.S.cls_z;
        s_qb.k1 = min(s_qb.k0 + it.S.cls_z, it.S.nslices);
        s_qb.i0 = bx * kClsX;
        s_qb.j0 = by * kClsY;
        s_qb.ncx = (unsigned)(it.nx - 1);
        s_qb.ncy = (unsigned)(it.ny - 1);
        s_qb.nt = it.ts.n;
        s_ts = it.ts;
      }
    }
    __syncthreads();
    if (s_unit >= nunits) return;
    if (items[s_item].is_f32) classify_queue_brick<float>(s_qb, s_ts, mask);
    else classify_queue_brick<double>(s_qb, s_ts, mask);
    /* the brick ends with a barrier: thread 0 may overwrite s_qb */
  }
}

/*
 * k_classify_multi: the codes of up to kMaxThr objects of one field in one
 * pass over its nodes, one brick per block (the brick code of
 * k_classify_queue) -- the classification of fields whose rows TMA cannot
 * address (a row pitch that is not a multiple of 16 bytes, such as an odd
 * node count along x for a double field).
 */
template <typename T>
__global__ void __launch_bounds__(kClsX, 5)
k_classify_multi(const void* __restrict__ data, long long nx, long long ny, SlabDev S, ThrSet ts, CodeOut out) {
  pdl_enter();
  __shared__ QueueMask mask[2];
  /* the brick's description in shared memory, as k_classify_queue keeps it
     (in registers it spilled) */
  __shared__ QueueBrick s_qb;
  __shared__ ThrSet s_ts;
  if (threadIdx.x == 0) {
    s_qb.data = data;
    for (int t = 0; t < kMaxThr; t++) s_qb.codes[t] = out.codes[t];
    s_qb.nx = nx;
    s_qb.ny = ny;
    s_qb.kfirst = S.kfirst;
    s_qb.k0 = (long long)blockIdx.z * S.cls_z;
    s_qb.k1 = min(s_qb.k0 + S.cls_z, S.nslices);
    s_qb.i0 = blockIdx.x * kClsX;
    s_qb.j0 = blockIdx.y * kClsY;
    s_qb.ncx = (unsigned)(nx - 1);
    s_qb.ncy = (unsigned)(ny - 1);
    s_qb.nt = ts.n;
    s_ts = ts;
  }
  __syncthreads();
  classify_queue_brick<T>(s_qb, s_ts, mask);
}

/*
 * k_classify_tma: the same codes, with the node planes staged by TMA.  A
 * block owns kClsX x kClsY cells of kClsZ slices; each of its node planes
 * (TmaBox<T>::kX x (kClsY + 1) nodes, x from the tile start, so the copy starts on
 * a 16-byte boundary) is one cp.async.bulk.tensor copy into a ring of
 * TmaBox<T>::kStages shared-memory buffers, each completed on its own
 * mbarrier, so that many planes are in flight while the block turns the
 * current one into node bits and the previous pair into cell codes.  Fewer
 * stages let more blocks share an SM: the bytes in flight per SM stay about
 * the same, and more warps hide the latency of the bit work.  Copies beyond
 * the field read zeros (those nodes belong to no cell of the tile).  Every
 * wait is bounded: on a timeout the block records kErrClassifyTimeout, waits
 * (again bounded) for its own copies in flight, and returns.
 *
 * Node bits are warp ballots (see plane_codes).
 */
/* f64: 2 stages (19.7 KB, 11 blocks per SM) measured 0.326 ms on the 512^3
   two-level field, 3 stages 0.331, 4 stages 0.342; f32 blocks are limited
   by registers first */
constexpr int kTmaStagesF64 = 2;
constexpr int kTmaStagesF32 = 4;
constexpr int kTmaWaitLimit = 1 << 22;
template <typename T>
struct TmaBox {
  static constexpr int kX = sizeof(T) == 8 ? 130 : 132; /* >= kClsX + 1, a multiple of 16 bytes */
  static constexpr int kBytes = kX * (kClsY + 1) * (int)sizeof(T);
  static constexpr int kStride = (kBytes + 127) / 128 * 128; /* every stage starts on 128 bytes */
  static constexpr int kStages = sizeof(T) == 8 ? kTmaStagesF64 : kTmaStagesF32;
};

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

/* bounded wait; false when the limit was reached */
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
  for (int it = 0; it < kTmaWaitLimit; it++)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

template <typename T, int NT>
__global__ void __launch_bounds__(kClsX)
k_classify_tma(const __grid_constant__ CUtensorMap tmap, FieldDev F, SlabDev S, ThrSet ts, CodeOut out,
               unsigned* __restrict__ err) {
  pdl_enter();
  static_assert(kClsX % 32 == 0 && kClsY + 1 <= 32, "classify tile: whole warps, a column of rows in one warp");
  using B = typename NodeBits<T>::type;
  constexpr int BX = TmaBox<T>::kX;
  constexpr int kStages = TmaBox<T>::kStages;
  __shared__ __align__(128) unsigned char stage_mem[kStages][TmaBox<T>::kStride];
  /* mask[plane parity][row][threshold][word]: slow warps may read plane p's while
     the others write plane p + 1's, so one barrier per plane is enough */
  __shared__ unsigned mask[2][kClsY + 1][NT][kClsWords];
  __shared__ __align__(8) unsigned long long bar[kStages];
  __shared__ int s_fail[2]; /* by plane parity: a fast warp may already wait for the next plane */
  const unsigned ncx = (unsigned)(F.nx - 1), ncy = (unsigned)(F.ny - 1);
  const int i0 = blockIdx.x * kClsX, j0 = blockIdx.y * kClsY;
  const long long k0 = (long long)blockIdx.z * S.cls_z;
  const long long k1 = min(k0 + S.cls_z, S.nslices);
  const int nplanes = (int)(k1 - k0) + 1; /* node planes k0 .. k1 of the slab */
  if (threadIdx.x == 0) {
    s_fail[0] = s_fail[1] = 0;
    for (int q = 0; q < kStages; q++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar[q])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto issue = [&](int p) { /* thread 0: plane p into stage p % kStages */
    const int st = p % kStages;
    const unsigned b = smem_u32(&bar[st]);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(TmaBox<T>::kBytes)
                 : "memory");
    const int z = (int)(S.kfirst + k0 + p);
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(&stage_mem[st][0])), "l"(&tmap), "r"(i0), "r"(j0), "r"(z), "r"(b)
        : "memory");
  };
  if (threadIdx.x == 0)
    for (int p = 0; p < kStages && p < nplanes; p++) issue(p);
  const int tx = threadIdx.x, lane = tx & 31, warp = tx >> 5;
  HalfCodes<NT> below = {};
  for (int p = 0; p < nplanes; p++) {
    const int st = p % kStages;
    if (!mbar_wait(smem_u32(&bar[st]), (unsigned)((p / kStages) & 1))) s_fail[p & 1] = 1;
    /* node bits of plane p: warp w takes word w of every row; the node column
       x = kClsX goes to the last warp's lanes 0 .. kClsY */
    {
      const B(*vp)[BX] = reinterpret_cast<const B(*)[BX]>(&stage_mem[st][0]);
      unsigned(*mp)[NT][kClsWords] = mask[p & 1];
#pragma unroll
      for (int jj = 0; jj <= kClsY; jj++) {
        const B v = fold_key(vp[jj][32 * warp + lane]);
#pragma unroll
        for (int t = 0; t < NT; t++) {
          const unsigned m = __ballot_sync(0xFFFFFFFFu, key_above(ts, t, v));
          if (lane == t) mp[jj][t][warp] = m;
        }
      }
      if (warp == kClsX / 32 - 1 && lane <= kClsY) {
        const B v = fold_key(vp[lane][kClsX]);
#pragma unroll
        for (int t = 0; t < NT; t++) mp[lane][t][kClsWords - 1] = key_above(ts, t, v) ? 1u : 0u;
      }
    }
    __syncthreads();
    if (s_fail[p & 1]) {
      /* give up: record it, let the copies in flight land (bounded), return */
      if (threadIdx.x == 0) {
        atomicOr(err, kErrClassifyTimeout);
        for (int q = p; q < nplanes && q < p + kStages; q++)
          mbar_wait(smem_u32(&bar[q % kStages]), (unsigned)((q / kStages) & 1));
      }
      return;
    }
    /* stage st is free again: refill it with plane p + kStages */
    if (threadIdx.x == 0 && p + kStages < nplanes) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      issue(p + kStages);
    }
    plane_codes<NT>(mask[p & 1], below, p == 0, out.codes, NT, k0 + p - 1, (unsigned)i0, (unsigned)j0, ncx, ncy);
  }
}

/* ------------------------------------------------------------------ */
/* the scan: segment offsets, then every cell's offsets                 */
/* ------------------------------------------------------------------ */
/* the thread's kScanItems codes, 4 per word (a code past the end reads as 0:
   no triangles, no vertices) */
__device__ __forceinline__ void load_scan_codes(const unsigned char* __restrict__ codes, long long base, long long n,
                                                unsigned wv[kScanItems / 4]) {
  if (base + kScanItems <= n) {
    /* 16-byte loads (base is a multiple of 32, the buffer 256-byte aligned) */
#pragma unroll
    for (int h = 0; h < kScanItems / 16; h++) {
      const uint4 v = *reinterpret_cast<const uint4*>(codes + base + 16 * h);
      wv[4 * h] = v.x;
      wv[4 * h + 1] = v.y;
      wv[4 * h + 2] = v.z;
      wv[4 * h + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int w = 0; w < kScanItems / 4; w++) {
      unsigned x = 0;
      for (int b = 0; b < 4; b++) {
        const long long c = base + 4 * w + b;
        if (c < n) x |= (unsigned)codes[c] << (8 * b);
      }
      wv[w] = x;
    }
  }
}

/*
 * The scan in one pass with decoupled look-back (Merrill and Garland,
 * "Single-pass Parallel Prefix Scan with Decoupled Look-back", NVIDIA
 * technical report NVR-2016-002).  Segment s's state word holds a packed
 * (triangle, vertex) sum in bits 0-61 and a status in bits 62-63: 1 = the
 * segment's own total, 2 = the total of segments 0..s.  A block takes the
 * next segment number from a ticket counter (the word after the states), so
 * every segment it waits for belongs to a block that is already running and
 * publishes its own total without waiting on anyone.  Warp 0 then walks back
 * 32 states at a time, adding own totals until it meets an inclusive one.
 * The walk is bounded: after kScanWaitLimit rounds the block records
 * kErrScanTimeout and goes on with what it has; its writes stay inside their
 * buffers whatever the prefix (the map is written only where it fits).
 */
constexpr unsigned long long kStAgg = 1ULL << 62, kStIncl = 2ULL << 62, kStValue = (1ULL << 62) - 1;
constexpr int kScanWaitLimit = 1 << 20;

__device__ __forceinline__ unsigned long long ld_state(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_state(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

/* the exclusive prefix of segment seg >= 1 (warp 0; every lane returns it) */
__device__ __forceinline__ unsigned long long look_back(const unsigned long long* state, long long seg,
                                                        unsigned* err) {
  const int lane = threadIdx.x & 31;
  unsigned long long prefix = 0;
  long long p = seg - 1; /* the nearest state not yet added */
  for (int rounds = 0;;) {
    const long long q = p - lane;
    const unsigned long long v = q >= 0 ? ld_state(state + q) : kStIncl; /* before segment 0: an inclusive 0 */
    const unsigned stt = (unsigned)(v >> 62);
    if (__any_sync(0xFFFFFFFFu, stt == 0)) {
      if (++rounds > kScanWaitLimit) {
        if (lane == 0) atomicOr(err, kErrScanTimeout);
        break;
      }
      __nanosleep(64);
      continue;
    }
    const unsigned incl = __ballot_sync(0xFFFFFFFFu, stt == 2);
    const int stop = incl ? __ffs(incl) - 1 : 31; /* lanes 0..stop are added */
    unsigned long long x = lane <= stop ? (v & kStValue) : 0ULL;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, d);
    prefix += x;
    if (incl) break;
    p -= 32;
  }
  return prefix;
}

/* the sum of x over the lanes before this one; total: over the warp */
__device__ __forceinline__ unsigned warp_exclusive(unsigned x, unsigned lane, unsigned& total) {
  unsigned incl = x;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
    if (lane >= d) incl += y;
  }
  total = __shfl_sync(0xFFFFFFFFu, incl, 31);
  return incl - x;
}

/* nonzero in the bytes of x that are neither 0 nor 255 (cells that own a crossed
   edge): their neighbouring bits differ somewhere */
__device__ __forceinline__ unsigned differing_bits(unsigned x) { return (x ^ (x >> 1)) & 0x7F7F7F7Fu; }

/* bit q: byte q of x is neither 0 nor 255 (adding 127 to the differences
   reaches the top bit) */
__device__ __forceinline__ unsigned mixed_bytes(unsigned x) {
  return ((((differing_bits(x) + 0x7F7F7F7Fu) & 0x80808080u) >> 7) * 0x01020408u) >> 24;
}

/*
 * One block per segment: its sums, its prefix by look-back, the word of every
 * cell that owns a crossed edge (and the offset of every 256th cell, where
 * k_vertices' tiles start; nobody reads the others), and the segment's part of
 * the triangle -> cell map when it fits tri_cap.  Few cells are crossed, so a
 * warp first lists the crossed ones of its 1024 cells (256 codes at a time,
 * eight per lane) with their sums, and after the block's prefixes goes through
 * that list, a cell per lane.  The offsets are relative to the segment
 * (VOffDev), so every warp stores them before the segment's prefix is known;
 * warp 0 then looks back and stores the segment's first offset.  The map goes
 * through a shared list of the segment's triangles when they fit it
 * (positions relative to the segment, then a coalesced copy), else it is
 * written directly once the prefix is known.  The block of the last segment
 * writes the slab totals and the end entries (triangle offset of cell n,
 * vertex offset of cell n).  OFFSETS (inspection): every cell's triangle
 * offset too, through a per-warp shared-memory stage (rows of kStagePitch
 * words) so that every store of a warp covers 512 contiguous bytes.
 *
 * Issue slots bound it.  Looking up every cell's count and storing every
 * cell's offset took 231 us per object of a 512^3 field, 36 at 192^3; this 185
 * and 20.  (Four segments per block and look-back: 225; 256 states per look-back
 * step instead of 32: 270, the reads meet in a few lines of the L2.)
 */
constexpr int kFillList = 8192; /* triangles of a segment listed in shared memory */
constexpr int kStagePitch = 33;  /* words per staged row: conflict-free transposes */
constexpr size_t kScanListBytes = sizeof(unsigned short) * kFillList;
constexpr size_t kScanStageBytes = sizeof(unsigned) * (kScanThreads / 32) * 32 * kStagePitch;

/* a warp's 1024 staged values into dst[wbase ..] (cells past n are skipped) */
__device__ __forceinline__ void store_stage(unsigned* __restrict__ dst, const unsigned* stage, long long wbase,
                                            long long n) {
  const int lane = threadIdx.x & 31;
  if (wbase + 32 * kScanItems <= n) {
    /* each store instruction writes 512 contiguous bytes (lane L: cells
       4L .. 4L + 3 of a 128-cell chunk, all in one staged row; wbase is a
       multiple of 1024, dst 256-byte aligned) */
#pragma unroll 4
    for (int k = 0; k < 8; k++) {
      const int e = 128 * k + 4 * lane, row = e >> 5, col = e & 31;
      const unsigned* sr = stage + kStagePitch * row + col;
      reinterpret_cast<uint4*>(dst + wbase)[32 * k + lane] =
          make_uint4(sr[0], sr[1], sr[2], sr[3]);
    }
  } else {
    for (int k = 0; k < 32; k++) {
      const long long c = wbase + 32 * k + lane;
      if (c < n) dst[c] = stage[kStagePitch * k + lane];
    }
  }
}

/* what the cell words need of the field and the slab */
struct ScanCells {
  FastDiv div_cx, div_cy;
  unsigned ncx, ncy, kfirst, krender0, krender1;
};

/* bits 16-24 of cell c's word (see VOffDev) */
__device__ __forceinline__ unsigned cell_bits(const ScanCells& b, unsigned c, unsigned code) {
  const unsigned row = fast_div(c, b.div_cx), i = c - row * b.ncx, kl = fast_div(row, b.div_cy), j = row - kl * b.ncy;
  const unsigned k = b.kfirst + kl;
  const bool rendered = i - 1u < b.ncx - 2u && j - 1u < b.ncy - 2u && k - b.krender0 < b.krender1 - b.krender0;
  return (owned_edges(code) << 16) | ((code & 1u) << 23) | (rendered ? kWordRendered : 0u);
}

template <bool OFFSETS>
__global__ void __launch_bounds__(kScanThreads, 6)
k_scan(ScanCells box, const unsigned char* __restrict__ codes, long long n, long long nseg,
       unsigned long long* __restrict__ state, unsigned* __restrict__ offsets, VOffDev voff,
       unsigned long long* __restrict__ totals, unsigned* __restrict__ tri_cell, unsigned long long tri_cap,
       unsigned* __restrict__ ovf, unsigned* __restrict__ err) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char scan_smem[];
  constexpr unsigned kWarps = kScanThreads / 32, kWarpCells = 32 * kScanItems;
  static_assert(kWarpCells == 1024, "four groups of 256 cells");
  __shared__ unsigned s_tri[kWarps], s_vert[kWarps]; /* the warps' sums */
  __shared__ unsigned s_cnt[256];
  __shared__ unsigned long long s_prefix;
  __shared__ unsigned s_seg;
  __shared__ unsigned short s_cells[kWarps][kWarpCells]; /* the warp's crossed cells, from its first one on */
  /* per triangle of the segment, its cell (12 bits: the segment's second half
     starts at a slot of its own) and rank */
  unsigned short* s_list = reinterpret_cast<unsigned short*>(scan_smem);
  if (threadIdx.x == 0) s_seg = (unsigned)atomicAdd(state + nseg, 1ULL);
  load_count_lut(s_cnt);
  __syncthreads();
  const long long seg = s_seg, c0 = seg * kScanTile;
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const long long wbase = c0 + (long long)(warp * kWarpCells); /* the warp's first cell */
  const unsigned char* wcodes = codes + wbase;
  const unsigned wn = (unsigned)max(0LL, min((long long)kWarpCells, n - wbase)); /* its cells */
  unsigned short* cells = s_cells[warp];
  uint2 cw[4];
#pragma unroll
  for (unsigned g = 0; g < 4; g++) {
    /* eight codes per lane (a code past the end reads as 0; wbase is a multiple of 1024) */
    const unsigned cf = 256 * g + 8 * lane;
    cw[g] = make_uint2(0u, 0u);
    if (cf + 8 <= wn) {
      cw[g] = __ldg(reinterpret_cast<const uint2*>(wcodes + cf));
    } else {
      for (unsigned q = 0; q < 8; q++)
        if (cf + q < wn) (q < 4 ? cw[g].x : cw[g].y) |= (unsigned)wcodes[cf + q] << (8 * (q & 3));
    }
  }
  unsigned nact = 0, group[4]; /* crossed cells, and those before each 256 cells */
#pragma unroll
  for (unsigned g = 0; g < 4; g++) {
    group[g] = nact;
    if (!__any_sync(0xFFFFFFFFu, (differing_bits(cw[g].x) | differing_bits(cw[g].y)) != 0u)) continue;
    const unsigned mixed = mixed_bytes(cw[g].x) | (mixed_bytes(cw[g].y) << 4);
    unsigned total;
    unsigned short* to = cells + (nact + warp_exclusive(__popc(mixed), lane, total));
#pragma unroll
    for (unsigned q = 0; q < 8; q++)
      if (mixed & (1u << q)) *to++ = (unsigned short)(256 * g + 8 * lane + q);
    nact += total;
  }
  __syncwarp();
  unsigned tris = 0, verts = 0;
  for (unsigned a = lane; a < nact; a += 32) {
    const unsigned cnt = s_cnt[__ldg(wcodes + cells[a])];
    tris += cnt; /* both sums in 16-bit fields: at most 384 and 224 per lane */
  }
  tris = __reduce_add_sync(0xFFFFFFFFu, tris & 0xFFFFu) | (__reduce_add_sync(0xFFFFFFFFu, tris >> 16) << 16);
  verts = tris >> 16;
  tris &= 0xFFFFu;
  if (lane == 0) {
    s_tri[warp] = tris;
    s_vert[warp] = verts;
  }
  __syncthreads();
  /* of earlier warps; of the segment; of its first half */
  unsigned rel_t = 0, rel_v = 0, seg_tris = 0, seg_verts = 0, half_tris = 0;
#pragma unroll
  for (unsigned w = 0; w < kWarps; w++) {
    if (w < warp) {
      rel_t += s_tri[w];
      rel_v += s_vert[w];
    }
    if (w == kWarps / 2) half_tris = seg_tris;
    seg_tris += s_tri[w];
    seg_verts += s_vert[w];
  }
  const unsigned long long agg = (unsigned long long)seg_tris | ((unsigned long long)seg_verts << 31);
  /* the segment's own total goes out at once */
  if (threadIdx.x == 0) st_state(state + seg, (seg == 0 ? kStIncl : kStAgg) | agg);
  const bool can_list = seg_tris <= (unsigned)kFillList;
  /* the crossed cells, one per lane: fn(its place in the warp's list, its cell
     in the warp, code, first triangle and first vertex in the segment, triangles) */
  auto for_cells = [&](auto fn) {
    unsigned t0 = rel_t, v0 = rel_v;
    for (unsigned a = 0; a < nact; a += 32) {
      const bool has = a + lane < nact;
      const unsigned lc = has ? cells[a + lane] : 0u;
      const unsigned code = has ? __ldg(wcodes + lc) : 0u, cnt = has ? s_cnt[code] : 0u;
      unsigned total;
      const unsigned ex = warp_exclusive(cnt, lane, total); /* 16-bit fields: at most 384 and 224 */
      if (has) fn(a + lane, lc, code, t0 + (ex & 0xFFFFu), v0 + (ex >> 16), cnt & 0xFFFFu);
      t0 += total & 0xFFFFu;
      v0 += total >> 16;
    }
  };
  unsigned* words = voff.word + wbase;
  const unsigned hi = (warp * kWarpCells) & 4095u; /* of the warp's cells within half a segment */
  for_cells([&](unsigned at, unsigned lc, unsigned code, unsigned slot, unsigned v, unsigned cnt) {
    words[lc] = v | cell_bits(box, (unsigned)wbase + lc, code);
#pragma unroll
    for (unsigned g = 0; g < 4; g++)
      if (at == group[g] && lc != 256 * g) words[256 * g] = v; /* the first crossed cell from there on */
    if (can_list)
      for (unsigned r = 0; r < cnt; r++) s_list[slot + r] = (unsigned short)((hi + lc) | (r << 12));
  });
  if (lane < 4) {
    const unsigned at = lane == 0 ? group[0] : (lane == 1 ? group[1] : (lane == 2 ? group[2] : group[3]));
    if (at == nact && 256 * lane < wn) words[256 * lane] = rel_v + verts;
  }
  if (warp == 0) {
    unsigned long long prefix = 0;
    if (seg > 0) {
      prefix = look_back(state, seg, err);
      if (lane == 0) st_state(state + seg, kStIncl | ((prefix + agg) & kStValue));
    }
    if (lane == 0) {
      s_prefix = prefix;
      voff.seg[seg] = (unsigned)(prefix >> 31);
      if (seg == nseg - 1) {
        const unsigned long long tot = prefix + agg;
        totals[0] = tot & kTriMask;
        totals[1] = tot >> 31;
        if (OFFSETS) offsets[n] = (unsigned)(tot & kTriMask);
        /* cell n: the end of this segment, or the start of segment nseg */
        voff.seg[nseg] = (unsigned)(tot >> 31);
        voff.word[n] = n - c0 < kScanTile ? (unsigned)(agg >> 31) : 0u;
      }
    }
  }
  __syncthreads();
  const unsigned long long seg0 = s_prefix;
  const unsigned ta = (unsigned)(seg0 & kTriMask);
  const bool fill = (unsigned long long)ta + seg_tris <= tri_cap;
  /* a map that does not fit: the caller runs the scan again with a larger
     map, or, when the buffers were sized before the count was known (ovf
     given), renders the frame again */
  if (!fill && ovf && threadIdx.x == 0) atomicOr(ovf, kOvfTriangles);
  if (OFFSETS) {
    /* 32 consecutive cells per lane */
    unsigned* stage = reinterpret_cast<unsigned*>(scan_smem + kScanListBytes) + warp * 32 * kStagePitch;
    unsigned wv[kScanItems / 4], sum = 0, total;
    load_scan_codes(codes, wbase + (long long)lane * kScanItems, n, wv);
#pragma unroll
    for (int q = 0; q < kScanItems; q++) sum += s_cnt[(wv[q >> 2] >> (8 * (q & 3))) & 255] & 0xFFFFu;
    unsigned run = ta + rel_t + warp_exclusive(sum, lane, total);
#pragma unroll
    for (int q = 0; q < kScanItems; q++) {
      stage[kStagePitch * lane + q] = run;
      run += s_cnt[(wv[q >> 2] >> (8 * (q & 3))) & 255] & 0xFFFFu;
    }
    __syncwarp();
    store_stage(offsets, stage, wbase, n);
  }
  if (fill && !can_list) {
    for_cells([&](unsigned, unsigned lc, unsigned, unsigned slot, unsigned, unsigned cnt) {
      for (unsigned r = 0; r < cnt; r++) tri_cell[ta + slot + r] = ((unsigned)wbase + lc) | (r << kTcRankShift);
    });
  }
  if (fill && can_list) {
    /* the list was complete at the barrier above */
    for (unsigned e = threadIdx.x; e < seg_tris; e += kScanThreads) {
      const unsigned v = s_list[e];
      tri_cell[ta + e] = ((unsigned)c0 + (e >= half_tris ? 4096u : 0u) + (v & 4095u)) | ((v >> 12) << kTcRankShift);
    }
  }
}

/* ------------------------------------------------------------------ */
/* exact triangles on demand (triangulate.c:40-93)                      */
/* ------------------------------------------------------------------ */
__device__ __forceinline__ d3 corner_pos(const FieldDev& F, long long i, long long j, long long k, int c) {
  const long long ii = i + (c & 1), jj = j + ((c >> 1) & 1), kk = k + (c >> 2);
  if (F.nodes) {
    const double* p = F.nodes + 3 * ((kk * F.ny + jj) * F.nx + ii);
    return {p[0], p[1], p[2]};
  }
  return {F.gx[ii], F.gy[jj], F.gz[kk]};
}

/* triangulate.c:40-73 */
__device__ __forceinline__ d3 interpolate(double vt, d3 p0, double v0, d3 p1, double v1) {
  const double dv = dsub(v1, v0);
  if (abs_lt_1e8(dv)) return p0;
  const double f = ddiv(dsub(vt, v0), dv);
  return v_add(p0, v_mul(f, v_sub(p1, p0)));
}

/* value at corner c of cell (i, j, k) */
__device__ __forceinline__ double corner_value(const FieldDev& F, long long i, long long j, long long k, int c) {
  const long long idx = ((k + (c >> 2)) * F.ny + j + ((c >> 1) & 1)) * F.nx + i + (c & 1);
  return F.is_f32 ? (double)__ldg(static_cast<const float*>(F.data) + idx)
                  : __ldg(static_cast<const double*>(F.data) + idx);
}

/* corner values and code of cell (i, j, k), element type chosen at run time */
__device__ __forceinline__ unsigned cell_code_any(const FieldDev& F, long long i, long long j, long long k,
                                                  double vals[8]) {
  return F.is_f32 ? cell_code<float>(F, i, j, k, vals) : cell_code<double>(F, i, j, k, vals);
}

/*
 * The reference's triangle (vertices in winding order) for emission index t
 * of the slab, recomputed from the field: the same operations as k_emit's
 * FP32 estimate stands for.  Returns the cube-edge ids in *edges.
 */
__device__ __forceinline__ void exact_vertices(const Geo& G, long long t, d3 v[3]) {
  const unsigned tc = G.tri_cell[t];
  const unsigned c = tc & kTcCellMask, r = tc >> kTcRankShift;
  unsigned ui, uj, ukl;
  cell_ijk(G.F, c, ui, uj, ukl);
  const long long i = ui, j = uj, k = G.S.kfirst + ukl;
  const unsigned code = G.codes[c];
  const unsigned long long e = __ldg(G.lut + code * 12 + r);
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const int a = (int)((e >> (6 * q)) & 7), b = (int)((e >> (6 * q + 3)) & 7);
    v[q] = interpolate(G.F.threshold, corner_pos(G.F, i, j, k, a), corner_value(G.F, i, j, k, a),
                       corner_pos(G.F, i, j, k, b), corner_value(G.F, i, j, k, b));
  }
}

/* triangulate.c:75-93 and normal.c:39-40: face normal, area, area * face normal */
__device__ __forceinline__ void face_normal(const d3 v[3], d3& fn, double& area, d3& wn) {
  fn = v_cross(v_sub(v[1], v[0]), v_sub(v[2], v[0]));
  area = dsqrt(v_dot(fn, fn));
  fn = v_mul(drcp(area), fn);
  wn = v_mul(area, fn);
}

/* ------------------------------------------------------------------ */
/* k_emit: single-precision triangles with certified bounds             */
/* ------------------------------------------------------------------ */
/* x >= 0 as a bfloat16 no smaller than x (bits of the high half; a NaN gives
   0x8000) */
__device__ __forceinline__ unsigned bf16_up(float x) { return (__float_as_uint(x) + 0xFFFFu) >> 16; }
__device__ __forceinline__ float bf16_value(unsigned h) { return __uint_as_float(h << 16); }

/* a field value as a float and the bound on its conversion error */
__device__ __forceinline__ float value_f(double v, float& e) {
  const float a = to_f(v); /* truncation: < 2u |a|, or < 2^-126 when flushed */
  e = 2.f * kU32 * fabsf(a) + 1.2e-38f;
  return a;
}
__device__ __forceinline__ float value_f(float v, float& e) {
  e = 0.f;
  return v;
}

/*
 * The interpolation parameter f = (vt - v0) / (v1 - v0) of triangulate.c:40-73
 * in FP32 with a bound e_f on its distance to the reference's value.
 * Returns 1 (f valid), 0 (the reference keeps p0: |v1 - v0| < 1e-8) or -1
 * (the bounds cannot decide that test).
 *   double fields: the two differences are formed in FP64 exactly as the
 *     reference forms them, then truncated to float (2u each), so the 1e-8
 *     test is exact and cancellation costs no accuracy (k_vertices: issue
 *     bound, two FP64 subtractions cost fewer slots than float pairs);
 *   float fields: the values are exact floats and the differences are FP32
 *     (u each), with the 1e-8 test decided by the bounds.
 * interp_shade below is the FP64-free form for double fields.
 */
__device__ __forceinline__ int interp_param(double vt, float, float, double v0, double v1, float& f, float& e_f) {
  const double dvd = dsub(v1, v0);
  if (abs_lt_1e8(dvd)) return 0;
  const float dv = to_f(dvd), dt = to_f(dsub(vt, v0));
  const float adv = fabsf(dv);
  const float e_dv = 2.f * kU32 * adv + 1.2e-38f, e_dt = 2.f * kU32 * fabsf(dt) + 1.2e-38f;
  if (!(adv > 1e-30f) || adv > 1e30f) return -1;
  const float rdv = __fdividef(1.f, adv); /* 2 ulp on [1e-30, 1e30] */
  const float xr = e_dv * rdv;
  f = __fdividef(dt, dv);
  const float fmax_ = 1.01f * (fabsf(dt) + e_dt) * rdv * (1.f + 1.02f * xr);
  e_f = 1.1f * (1.01f * (e_dt + fmax_ * e_dv) * rdv + 4.f * kU32 * fabsf(f));
  return 1;
}
__device__ __forceinline__ int interp_param(double, float vt, float e_vt, float v0, float v1, float& f, float& e_f) {
  const float dv = v1 - v0;
  const float e_dv = 1.01f * kU32 * fabsf(dv);
  const float adv = fabsf(dv);
  if (!(adv - e_dv > 1.00001e-8f)) return adv + e_dv < 0.99999e-8f ? 0 : -1;
  if (adv > 1e30f) return -1;
  /* 1 / |dv| to 2 ulp; 1 / (|dv| - e_dv) <= rdv (1 + 1.02 x) for x = e_dv rdv < 0.01 */
  const float rdv = __fdividef(1.f, adv);
  const float xr = e_dv * rdv;
  if (!(xr < 0.01f)) return -1;
  const float dt = vt - v0;
  const float e_dt = e_vt + 1.01f * kU32 * fabsf(dt);
  f = __fdividef(dt, dv); /* 2 ulp */
  /* |dt/dv - DT/DV| <= (e_dt + |DT/DV| e_dv) / |dv|, |DT/DV| <= fmax */
  const float fmax_ = 1.01f * (fabsf(dt) + e_dt) * rdv * (1.f + 1.02f * xr);
  e_f = 1.1f * (1.01f * (e_dt + fmax_ * e_dv) * rdv + 4.f * kU32 * fabsf(f));
  return 1;
}

/* the threshold in the forms the shading pass uses */
struct ThrF {
  float vt, e_vt; /* rounded to float, with its bound (float fields) */
  float hi, lo;   /* split (double fields) */
};
/* the same for k_vertices, where a kept tail corner (status 0) is undecided as
   well.  Double fields: |dv| >= 1e-8 after the exact test, so the truncations
   are relative (2u each, a flushed dt is below 1e-29 of dv), the quotient adds 4u */
__device__ __forceinline__ int interp_edge(double vt, const ThrF&, double v0, double v1, float& f, float& e_f) {
  const double dvd = dsub(v1, v0);
  if (abs_lt_1e8(dvd)) return 0;
  const float dv = to_f(dvd);
  if (!(fabsf(dv) < 1e30f)) return -1;
  f = __fdividef(to_f(dsub(vt, v0)), dv);
  e_f = __fmaf_rn(8.5f * kU32, fabsf(f), 1e-29f);
  return 1;
}
__device__ __forceinline__ int interp_edge(double, const ThrF& th, float v0, float v1, float& f, float& e_f) {
  return interp_param(0., th.vt, th.e_vt, v0, v1, f, e_f);
}

/*
 * A double as an unevaluated float pair hi + lo, by integer operations (the
 * FP64 pipe stays free): hi carries the top 24 significand bits, lo up to 24
 * of the next 29, both truncated; |hi + lo - v| <= 2^-47 |v| + 2^-126.  False
 * for NaN, infinities and magnitudes beyond float.
 */
__device__ __forceinline__ bool split_bits(unsigned long long b, float& hi, float& lo) {
  const unsigned sign = (unsigned)(b >> 63) << 31;
  const int ex = (int)((b >> 52) & 0x7FF);
  hi = lo = 0.f;
  if (ex == 0x7FF || ex - 1023 > 127) return false;
  const int fe = ex - 1023 + 127;
  if (fe <= 0) { /* below 2^-126: flushed */
    hi = __uint_as_float(sign);
    return true;
  }
  hi = __uint_as_float(sign | ((unsigned)fe << 23) | (unsigned)((b >> 29) & 0x7FFFFFu));
  /* lo = rem 2^(ex - 1075), rem the low 29 bits, truncated to 24 significant
     bits (an error below 2^-47 |v|); flushed to 0 below 2^-126 */
  const unsigned rem = (unsigned)(b & 0x1FFFFFFFu);
  if (rem == 0) return true;
  const int lz = __clz(rem);                      /* 3 .. 31 */
  const int le = (31 - lz) + (ex - 1075) + 127;   /* biased exponent of lo */
  if (le <= 0) return true;
  lo = __uint_as_float(sign | ((unsigned)le << 23) | ((rem << (lz + 1)) >> 9));
  return true;
}

__device__ __forceinline__ bool split_f(double v, float& hi, float& lo) {
  return split_bits((unsigned long long)__double_as_longlong(v), hi, lo);
}

/* s + t = a - b exactly (Knuth's two-sum; no fused operations in this build) */
__device__ __forceinline__ void two_diff(float a, float b, float& s, float& t) {
  s = a - b;
  const float bb = s - a;
  t = (a - (s - bb)) - (b + bb);
}

/* (ah + al) - (bh + bl) in FP32 and a bound on its distance to the
   difference of the two doubles the pairs stand for */
__device__ __forceinline__ float pair_diff(float ah, float al, float bh, float bl, float& e) {
  float s, t;
  two_diff(ah, bh, s, t);
  const float dl = al - bl, u = t + dl, d = s + u;
  e = 1.01f * (kU32 * (fabsf(dl) + fabsf(u) + fabsf(d)) + 1.43e-14f * (fabsf(ah) + fabsf(bh)) + 3e-38f);
  return d;
}

__device__ __forceinline__ ThrF thr_f(double t) {
  ThrF r;
  r.vt = value_f(t, r.e_vt);
  if (!split_f(t, r.hi, r.lo)) r.hi = r.lo = __int_as_float(0x7fc00000);
  return r;
}

/* interp_param for the shading pass, FP32 operations only: for a double
   field the differences are formed from float pairs (pair_diff), accurate to
   a few float ulps of the differences themselves */
__device__ __forceinline__ int interp_shade(const FieldDev& F, const ThrF& th, long long v0, long long v1, float& f,
                                            float& e_f) {
  float h0, l0, h1, l1;
  if (!split_bits((unsigned long long)v0, h0, l0) || !split_bits((unsigned long long)v1, h1, l1) || th.hi != th.hi)
    return -1;
  float e_dv, e_dt;
  const float dv = pair_diff(h1, l1, h0, l0, e_dv);
  const float adv = fabsf(dv);
  /* triangulate.c:40-73: |v1 - v0| < 1e-8 keeps p0 */
  if (!(adv - e_dv > 1.00001e-8f)) return adv + e_dv < 0.99999e-8f ? 0 : -1;
  if (adv > 1e30f) return -1;
  const float rdv = __fdividef(1.f, adv);
  const float xr = e_dv * rdv;
  if (!(xr < 0.01f)) return -1;
  const float dt = pair_diff(th.hi, th.lo, h0, l0, e_dt);
  f = __fdividef(dt, dv); /* 2 ulp */
  const float fmax_ = 1.01f * (fabsf(dt) + e_dt) * rdv * (1.f + 1.02f * xr);
  e_f = 1.1f * (1.01f * (e_dt + fmax_ * e_dv) * rdv + 4.f * kU32 * fabsf(f));
  return 1;
}
__device__ __forceinline__ int interp_shade(const FieldDev& F, const ThrF& th, float v0, float v1, float& f,
                                            float& e_f) {
  return interp_param(F.threshold, th.vt, th.e_vt, v0, v1, f, e_f);
}

/* a corner value as the shading pass takes it: a double's bit pattern, a float itself */
template <typename T>
struct ShadeVal;
template <>
struct ShadeVal<double> {
  typedef long long type;
  static __device__ __forceinline__ long long load(const double* f, long long idx) { return ld_bits(f + idx); }
};
template <>
struct ShadeVal<float> {
  typedef float type;
  static __device__ __forceinline__ float load(const float* f, long long idx) { return __ldg(f + idx); }
};


/*
 * FP32 estimate of one vertex (triangulate.c:40-73) relative to the camera,
 * q = vertex - camera, with a bound per component on the distance to the
 * reference's FP64 value: p = p0 + f (p1 - p0) with f from interp_param.
 * Returns false when interp_param cannot decide the reference's 1e-8 test, or
 * decides that the tail corner is kept (the triangle then takes the FP64 path).
 */
template <typename T>
__device__ __forceinline__ bool vertex_q(const SceneDev& s, const FieldDev& F, const ThrF& th, const float x0[3],
                                         T v0, const float x1[3], T v1, float ce, float q[3], float eq[3]) {
  /* x0, x1: corner coordinates rounded to float with error <= ce u |x| */
  const float pc[3] = {s.f_cam[0], s.f_cam[1], s.f_cam[2]};
  float f = 0.f, e_f = 0.f;
  const int st = interp_param(F.threshold, th.vt, th.e_vt, v0, v1, f, e_f);
  /* 0: the reference keeps the tail corner, which depends on the triangle */
  if (st <= 0) return false;
  const float af = fabsf(f);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    /* fused multiply-adds round once where the bound allows for two
       roundings, so every bound below still holds */
    const float d = x1[i] - x0[i];
    const float p = __fmaf_rn(f, d, x0[i]);
    q[i] = p - pc[i];
    const float cx0 = ce * fabsf(x0[i]);
    const float inner = __fmaf_rn(2.2f, fabsf(d), __fmaf_rn(ce, fabsf(x1[i]), cx0));
    const float ep = __fmaf_rn(e_f, fabsf(d), kU32 * __fmaf_rn(af, inner, cx0 + fabsf(p)));
    eq[i] = __fmaf_rn(1.1f, __fmaf_rn(kU32, fabsf(pc[i]) + fabsf(q[i]), ep), 1e-30f);
  }
  return true;
}

/* corner coordinates as floats, and the bound factor of their rounding */
__device__ __forceinline__ float corner_pos_f(const FieldDev& F, long long i, long long j, long long k, int c,
                                              float x[3]) {
  const long long ii = i + (c & 1), jj = j + ((c >> 1) & 1), kk = k + (c >> 2);
  if (F.nodes) {
    const double* p = F.nodes + 3 * ((kk * F.ny + jj) * F.nx + ii);
    x[0] = to_f(p[0]);
    x[1] = to_f(p[1]);
    x[2] = to_f(p[2]);
    return 2.f;
  }
  x[0] = __ldg(F.gxf + ii);
  x[1] = __ldg(F.gyf + jj);
  x[2] = __ldg(F.gzf + kk);
  return 1.f;
}

/*
 * Screen projection in single precision from q (bounded per component).
 * Uses the identity (exact in real arithmetic) of project.c:9-67
 *   x = [(cam - centre) . lx + D (q . lx) / (n . q)] / (lx . lx),
 *   D = n . centre - n . cam,  depth = n . q,  t = D / (n . q)
 * Each FP32 dot product a . q is within sum|a_i| eq_i + 4.2 u sum|a_i q_i|
 * of the real one.  Returns 1 = certainly projects, 0 = certainly fails
 * (render.c:62-72 drops the triangle), -1 = too close to a threshold of
 * project.c:39-46.
 */
__device__ __forceinline__ int project_dots(const SceneDev& s, float nq, float lq, float mq, float e_nq, float e_lq,
                                            float e_mq, float ref_eps, float& X, float& Y, float& Z, float& exy,
                                            float& ez, float& rz) {
  const float anq = fabsf(nq);
  X = Y = exy = rz = 0.f;
  Z = nq;
  ez = 1.1f * e_nq + 1e-30f;
  /* project.c:39-46: |nr| < 1e-8 or t outside (0, 1) => the point is dropped */
  if (anq + e_nq < 0.99e-8f) return 0;
  if (!(anq - e_nq > 1.01e-8f) || !(anq < 1e30f)) return -1;
  /* r = 1 / nq to 2 ulp (__fdividef, |nq| in [1e-8, 1e30]); with
     x = e_nq |r| < 0.01, 1 / (|nq| - e_nq) <= |r| (1 + 1.02 x) (1 + 4u) */
  const float r = __fdividef(1.f, nq);
  rz = fabsf(r);
  const float x = e_nq * rz;
  if (!(x < 0.01f)) return -1;
  const float rin = 1.01f * rz * (1.f + 1.02f * x);
  const float t = s.f_dq * r;
  const float et = fabsf(t) * (1.02f * x + 6.f * kU32) + 1e-30f;
  if (t + et < 0.f || t - et > 1.f) return 0;
  if (!(t - et > 0.f) || !(t + et < 1.f)) return -1;
  const float rx = lq * r, ry = mq * r;
  const float erx = __fmaf_rn(__fmaf_rn(fabsf(rx), e_nq, e_lq), rin, 6.f * kU32 * fabsf(rx));
  const float ery = __fmaf_rn(__fmaf_rn(fabsf(ry), e_nq, e_mq), rin, 6.f * kU32 * fabsf(ry));
  X = __fmaf_rn(s.f_bx, rx, s.f_ax);
  Y = __fmaf_rn(s.f_by, ry, s.f_ay);
  const float ex = __fmaf_rn(fabsf(s.f_bx), erx,
                             __fmaf_rn(kU32, __fmaf_rn(2.f, fabsf(s.f_bx * rx), fabsf(s.f_ax)) + fabsf(X), ref_eps));
  const float ey = __fmaf_rn(fabsf(s.f_by), ery,
                             __fmaf_rn(kU32, __fmaf_rn(2.f, fabsf(s.f_by * ry), fabsf(s.f_ay)) + fabsf(Y), ref_eps));
  /* (a NaN in either must not be lost in a maximum) */
  exy = 1.1f * (ex > ey ? ex : ey);
  if (!(ex < 1e30f)) exy = INFINITY;
  return 1;
}

/* the dot products of q and their bounds, with fused multiply-adds: one rounding
   fewer per step than the unfused sums the bounds allow for */
__device__ __forceinline__ int project_f(const SceneDev& s, const float q[3], const float eq[3], float ref_eps,
                                         float& X, float& Y, float& Z, float& exy, float& ez, float& rz) {
  const float ax = fabsf(q[0]), ay = fabsf(q[1]), az = fabsf(q[2]);
  const float nq = __fmaf_rn(s.f_n[2], q[2], __fmaf_rn(s.f_n[1], q[1], s.f_n[0] * q[0]));
  const float lq = __fmaf_rn(s.f_lx[2], q[2], __fmaf_rn(s.f_lx[1], q[1], s.f_lx[0] * q[0]));
  const float mq = __fmaf_rn(s.f_ly[2], q[2], __fmaf_rn(s.f_ly[1], q[1], s.f_ly[0] * q[0]));
  auto bound = [&](const float a[3]) {
    const float se = __fmaf_rn(fabsf(a[2]), eq[2], __fmaf_rn(fabsf(a[1]), eq[1], fabsf(a[0]) * eq[0]));
    const float sq = __fmaf_rn(fabsf(a[2]), az, __fmaf_rn(fabsf(a[1]), ay, fabsf(a[0]) * ax));
    return __fmaf_rn(4.2f * kU32, sq, se);
  };
  return project_dots(s, nq, lq, mq, bound(s.f_n), bound(s.f_lx), bound(s.f_ly), ref_eps, X, Y, Z, exy, ez, rz);
}

/* inspection: every triangle's exact vertices, face normal, area and weighted normal */
__global__ void __launch_bounds__(256) k_exact_all(Geo G, const unsigned long long* __restrict__ total_p, TriDev tri) {
  pdl_enter();
  const long long T_ = (long long)*total_p;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < T_;
       t += (long long)gridDim.x * blockDim.x) {
    d3 v[3], fn, wn;
    double area;
    exact_vertices(G, t, v);
    face_normal(v, fn, area, wn);
    tri.wn[0][t] = wn.x;
    tri.wn[1][t] = wn.y;
    tri.wn[2][t] = wn.z;
#pragma unroll
    for (int q = 0; q < 3; q++) {
      tri.vert[3 * q + 0][t] = v[q].x;
      tri.vert[3 * q + 1][t] = v[q].y;
      tri.vert[3 * q + 2][t] = v[q].z;
    }
    tri.dbg_fn[3 * t + 0] = fn.x;
    tri.dbg_fn[3 * t + 1] = fn.y;
    tri.dbg_fn[3 * t + 2] = fn.z;
    tri.dbg_area[t] = area;
  }
}

/* ------------------------------------------------------------------ */
/* vertex normals (normal.c:6-165)                                      */
/* ------------------------------------------------------------------ */
/*
 * Sum of area * face normal over the triangles of the cells sharing cube
 * edge `e` of cell `c`, visited in the reference's order (ascending cell,
 * then triangle order), then normalised.  wn must be present for every
 * triangle touching the edge.
 */
__device__ __forceinline__ d3 vertex_normal(long long c, int e, long long ncx, long long ncy,
                                            const unsigned* __restrict__ offsets, const TriDev& tri) {
  d3 sum = {0., 0., 0.};
  const int nn = c_nb_count[e];
  for (int q = 0; q < nn; q++) {
    const long long nc = c + (long long)c_nb[e][q][0] * ncx * ncy + (long long)c_nb[e][q][1] * ncx +
                         (long long)c_nb[e][q][2];
    const unsigned le = (unsigned)c_nb[e][q][3];
    const unsigned u0 = offsets[nc], u1 = offsets[nc + 1];
    for (unsigned u = u0; u < u1; u++) {
      const unsigned om = tri.meta[u];
      if (((om & 31) == le) || (((om >> 5) & 31) == le) || (((om >> 10) & 31) == le)) {
        const d3 w = {tri.wn[0][u], tri.wn[1][u], tri.wn[2][u]};
        sum = v_add(sum, w);
      }
    }
  }
  return v_normalise(sum);
}

/* inspection: every rendered triangle's vertex normals */
__global__ void __launch_bounds__(256)
k_normals(FieldDev F, SlabDev S, const unsigned* __restrict__ offsets, const unsigned* __restrict__ tri_cell,
          const unsigned long long* __restrict__ total_p, TriDev tri) {
  pdl_enter();
  const long long T_ = (long long)*total_p;
  const long long ncx = F.nx - 1, ncy = F.ny - 1;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < T_;
       t += (long long)gridDim.x * blockDim.x) {
    const unsigned meta = tri.meta[t];
    if (!(meta & kMetaRendered)) continue;
    const long long c = tri_cell[t] & kTcCellMask;
#pragma unroll 1
    for (int m = 0; m < 3; m++) {
      const d3 n = vertex_normal(c, (meta >> (5 * m)) & 31, ncx, ncy, offsets, tri);
      tri.vn[3 * m + 0][t] = n.x;
      tri.vn[3 * m + 1][t] = n.y;
      tri.vn[3 * m + 2][t] = n.z;
    }
  }
}

/* ------------------------------------------------------------------ */
/* raster: exact fragment arithmetic (render.c:48-163)                  */
/* ------------------------------------------------------------------ */
/* the reference's projected triangle, bounding box and inverse area */
struct ExactTri {
  d3 v0, v1, v2;
  long long imin, imax, jmin, jmax;
  double area;
  double area_inv;
};

/* the projected triangle and its inverse area (the box is left unset) */
__device__ __forceinline__ bool exact_tri_core(const SceneDev& s, const d3 w[3], ExactTri& x) {
  if (!project(s, w[0], x.v0) || !project(s, w[1], x.v1) || !project(s, w[2], x.v2)) return false;
  x.area = edge_fn(x.v0, x.v1, x.v2);
  x.area_inv = drcp(x.area < 0. ? fmin(x.area, -1.e-16) : fmax(x.area, +1.e-16));
  return true;
}

/* the reference's bounding box of a projected triangle */
__device__ __forceinline__ void exact_box(const SceneDev& s, ExactTri& x) {
  const long long W = s.width, H = s.height;
  const long long xmin = (long long)dsub(dmul(dadd(0.5, fmin(x.v0.x, fmin(x.v1.x, x.v2.x))), (double)W), 1.);
  const long long xmax = (long long)dadd(dmul(dadd(0.5, fmax(x.v0.x, fmax(x.v1.x, x.v2.x))), (double)W), 1.);
  const long long ymin = (long long)dsub(dmul(dadd(0.5, fmin(x.v0.y, fmin(x.v1.y, x.v2.y))), (double)H), 1.);
  const long long ymax = (long long)dadd(dmul(dadd(0.5, fmax(x.v0.y, fmax(x.v1.y, x.v2.y))), (double)H), 1.);
  x.imin = min(W - 1, max(0LL, xmin));
  x.imax = min(W - 1, max(0LL, xmax));
  x.jmin = min(H - 1, max(0LL, ymin));
  x.jmax = min(H - 1, max(0LL, ymax));
}

__device__ __forceinline__ bool exact_tri(const SceneDev& s, const d3 w[3], ExactTri& x) {
  if (!exact_tri_core(s, w, x)) return false;
  exact_box(s, x);
  return true;
}

/* the reference's barycentric weights at pixel (i, j) of its box; false when
   outside the triangle */
__device__ __forceinline__ bool exact_weights_in(const ExactTri& x, long long i, long long j, const double* xs,
                                                 const double* ys, double& w0, double& w1, double& w2) {
  const d3 v3 = {xs[i], ys[j], 0.};
  w0 = dmul(x.area_inv, edge_fn(x.v1, x.v2, v3));
  w1 = dmul(x.area_inv, edge_fn(x.v2, x.v0, v3));
  w2 = dmul(x.area_inv, edge_fn(x.v0, x.v1, v3));
  return !(w0 < -1.e-8 || w1 < -1.e-8 || w2 < -1.e-8);
}

/* the same at any pixel; false when outside the box or the triangle */
__device__ __forceinline__ bool exact_weights(const ExactTri& x, long long i, long long j, const double* xs,
                                              const double* ys, double& w0, double& w1, double& w2) {
  if (i < x.imin || i > x.imax || j < x.jmin || j > x.jmax) return false;
  return exact_weights_in(x, i, j, xs, ys, w0, w1, w2);
}

__device__ __forceinline__ double exact_depth(const ExactTri& x, double w0, double w1, double w2) {
  return drcp(dadd(dadd(ddiv(w0, x.v0.z), ddiv(w1, x.v1.z)), ddiv(w2, x.v2.z)));
}

__device__ __forceinline__ unsigned long long order_of(const Geo& G, unsigned long long order_base, long long t) {
  const unsigned tc = G.tri_cell[t];
  return order_base + 12ULL * (tc & kTcCellMask) + (tc >> kTcRankShift);
}

/* a fragment the reference draws: its depth key, two of its weights and the
   bound on their distance to the reference's; and for the self-check the bound
   on an approximate depth's */
struct Hit {
  unsigned long long key;
  float w0, w1, ew, ed;
};

/* floats of the reference's weights, NaN where they do not sum to 1 (a clamped
   or so small an area that the edge functions' rounding shows) */
__device__ __forceinline__ void hit_weights(double w0, double w1, double w2, Hit& h) {
  const bool usable = fabs(w0 + w1 + w2 - 1.) < 1e-8;
  h.w0 = usable ? to_f(w0) : __int_as_float(0x7fc00000);
  h.w1 = usable ? to_f(w1) : __int_as_float(0x7fc00000);
  h.ew = 2.5f * kU32; /* truncated to float, at most 1 */
}

/* the winning fragment's weights for shading (see RasterDev::winfo) */
__device__ __forceinline__ void keep_weights(const RasterDev& R, long long p, unsigned long long order, const Hit& h) {
  store128_atomic(R.winfo + p,
                  (unsigned long long)__float_as_uint(h.w0) | ((unsigned long long)__float_as_uint(h.w1) << 32),
                  (order << 24) | (bf16_up(h.ew) << 8) | R.epoch);
}

/* approximate depths are within kDepthTol of the reference's relatively; two
   depth keys farther apart than kNear (in units of the last place; 2 kDepthTol
   is at most 2^34 of them) are in the order of the reference's depths */
constexpr float kDepthTol = 9.5367431640625e-07f; /* 2^-20 */
constexpr unsigned long long kNear = (1ULL << 34) + (1ULL << 30);
/* in the colour bits of a slot that is not shaded yet: its key is exact */
constexpr unsigned long long kLoExact = 1;

/* the triangle of a cell of field F: the reference's vertices */
__device__ __forceinline__ void cell_vertices(const FieldDev& F, long long i, long long j, long long k,
                                              unsigned long long e, d3 v[3]) {
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const int a = (int)((e >> (6 * q)) & 7), b = (int)((e >> (6 * q + 3)) & 7);
    v[q] = interpolate(F.threshold, corner_pos(F, i, j, k, a), corner_value(F, i, j, k, a), corner_pos(F, i, j, k, b),
                       corner_value(F, i, j, k, b));
  }
}

struct WinCell;
__device__ __forceinline__ bool winner_cell(const FieldDev& F, unsigned long long lo, unsigned long long obase,
                                            WinCell& w);

/* the reference's depth key of the fragment of order `order` that holds pixel
   (i, j) with key `key`: recomputed when an object of the table drew it, the
   key itself otherwise (background, lines, fields with a converter) */
__device__ __noinline__ unsigned long long slot_exact_key(const FrameObjs& O, const SceneDev& s,
                                                          const unsigned long long* lut, const double* xs,
                                                          const double* ys, unsigned long long order, long long i,
                                                          long long j, unsigned long long key);

/* an approximate fragment (key, order << 24) against a pixel's slot: 0 = it lost, 1 =
   it was stored, 2 = the slot's depth is near: it has to be compared exactly */
__device__ __forceinline__ int slot_max_approx(Slot* slot, unsigned long long key, unsigned long long lo,
                                               unsigned* err) {
  unsigned long long cur_lo = 0, cur_hi = 0;
  cas128(slot, 0ULL, 0ULL, 0ULL, 0ULL, cur_lo, cur_hi);
  for (int guard = 0; guard < 1 << 20; guard++) {
    if (cur_lo >> 24 == lo >> 24) return 0;
    if (key - cur_hi + kNear <= 2 * kNear) return 2;
    if (key < cur_hi) return 0;
    unsigned long long o_lo, o_hi;
    cas128(slot, cur_lo, cur_hi, lo, key, o_lo, o_hi);
    if (o_lo == cur_lo && o_hi == cur_hi) return 1;
    cur_lo = o_lo;
    cur_hi = o_hi;
  }
  atomicOr(err, 1u);
  return 0;
}

/*
 * Raises a pixel's slot to the reference's maximum of (depth, order) over the
 * slot and this fragment; true when the fragment was stored.  Keys closer
 * than kNear may stand for depths in either order: the two depths are then
 * compared exactly (this fragment's key is exact).  Every update, here and in
 * slot_max_approx, decides between the slot's fragment and the new one as the
 * reference's depths do, so the final owner is the reference's whichever keys
 * were stored.  A slot of the group being drawn says itself that its key is
 * exact (kLoExact): surfaces that coincide, or the many triangles through one
 * node, are compared without computing the other depth again and again.
 * Bounded like slot_max.
 */
__device__ __forceinline__ bool slot_max_near(const FrameObjs& O, const SceneDev& s, const unsigned long long* lut,
                                              const double* xs, const double* ys, Slot* slot, long long i, long long j,
                                              unsigned long long key, unsigned long long lo, unsigned* err) {
  unsigned long long cur_lo = 0, cur_hi = 0;
  cas128(slot, 0ULL, 0ULL, 0ULL, 0ULL, cur_lo, cur_hi);
  const unsigned long long order = lo >> 24;
  for (int guard = 0; guard < 1 << 20; guard++) {
    const unsigned long long co = cur_lo >> 24;
    if (co == order) return false;
    unsigned long long theirs = cur_hi;
    if (O.n && key - cur_hi + kNear <= 2 * kNear && (co < O.group || !(cur_lo & kLoExact)))
      theirs = slot_exact_key(O, s, lut, xs, ys, co, i, j, cur_hi);
    if (key < theirs || (key == theirs && order < co)) return false;
    unsigned long long o_lo, o_hi;
    cas128(slot, cur_lo, cur_hi, lo, key, o_lo, o_hi);
    if (o_lo == cur_lo && o_hi == cur_hi) return true;
    cur_lo = o_lo;
    cur_hi = o_hi;
  }
  if (err) atomicOr(err, 1u);
  return false;
}

/*
 * One candidate fragment through the reference's test.  Candidates come from
 * the cover list only: triangles whose area is certainly not clamped, so a
 * pixel that passes the weight test lies in the triangle's extent and so
 * inside the reference's box, whose margins are a pixel wide; the box is not
 * computed (CHECK: it is, and a pixel outside it counts as a violation and is
 * not drawn).
 */
template <bool CHECK>
__device__ __forceinline__ bool exact_hit(const Geo& G, const SceneDev& s, long long t, long long i, long long j,
                                          const double* xs, const double* ys, unsigned* checks, Hit& h) {
  d3 w[3];
  exact_vertices(G, t, w);
  ExactTri x;
  if (!exact_tri_core(s, w, x)) return false;
  double w0, w1, w2;
  if (!exact_weights_in(x, i, j, xs, ys, w0, w1, w2)) return false;
  if (CHECK) {
    exact_box(s, x);
    if (i < x.imin || i > x.imax || j < x.jmin || j > x.jmax) {
      atomicAdd(checks + 2, 1u);
      return false;
    }
  }
  h.key = depth_key(exact_depth(x, w0, w1, w2));
  hit_weights(w0, w1, w2, h);
  return true;
}

/* the same as a call of its own: its registers stay out of the caller's */
template <bool CHECK>
__device__ __noinline__ bool exact_fragment(const Geo& G, const SceneDev& s, long long t, long long i, long long j,
                                            const double* xs, const double* ys, unsigned* checks, Hit& h) {
  return exact_hit<CHECK>(G, s, t, i, j, xs, ys, checks, h);
}

/* ------------------------------------------------------------------ */
/* k_raster: single-precision coverage / depth filter                  */
/* ------------------------------------------------------------------ */
/*
 * Per rendered triangle, every pixel whose centre can lie in the triangle
 * is classified with certified FP32 bounds:
 *   certainly outside        -> dropped
 *   certainly inside         -> raises the pixel's depth floor (zlo) to a
 *                               certain lower bound of its depth, and is a
 *                               candidate
 *   undecided                -> candidate
 * A candidate carries an upper bound of its depth; k_finish drops it when
 * that bound is below the final floor (a certainly drawn fragment is nearer,
 * so it cannot win) and settles it otherwise.
 */

/*
 * Block-wide reservation of list slots for two lists at once: every thread of
 * the block calls it at the same point with its item counts (block totals
 * below 65536 per list).  One global atomic per block and list instead of
 * one per warp: the list counters are single addresses that every block
 * appends to, and same-address atomics serialise in the L2.
 */
template <int kThreads>
__device__ __forceinline__ void block_reserve2(unsigned long long* count0, unsigned n0, unsigned long long* count1,
                                               unsigned n1, unsigned long long& r0, unsigned long long& r1) {
  __shared__ unsigned s_w[kThreads / 32];
  __shared__ unsigned long long s_b[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned x = n0 | (n1 << 16);
  unsigned incl = x;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
    if (lane >= d) incl += y;
  }
  if (lane == 31) s_w[warp] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned run = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; w++) {
      const unsigned v = s_w[w];
      s_w[w] = run;
      run += v;
    }
    const unsigned t0 = run & 0xFFFFu, t1 = run >> 16;
    s_b[0] = t0 ? atomicAdd(count0, (unsigned long long)t0) : 0ULL;
    s_b[1] = t1 ? atomicAdd(count1, (unsigned long long)t1) : 0ULL;
  }
  __syncthreads();
  const unsigned ex = s_w[warp] + incl - x;
  r0 = s_b[0] + (ex & 0xFFFFu);
  r1 = s_b[1] + (ex >> 16);
  __syncthreads();
}

template <int kThreads>
__device__ __forceinline__ unsigned long long block_reserve(unsigned long long* count, unsigned n) {
  unsigned long long r0, r1;
  block_reserve2<kThreads>(count, n, count, 0u, r0, r1);
  return r0;
}

/* pixel index range whose centres (i + 0.5) / n - 0.5 may lie in [lo, hi]
   (finite); in 32 bits throughout (conversions from and to 64-bit integers run
   on the FP64 pipe), and a conversion out of range saturates */
__device__ __forceinline__ void centre_range(float lo, float hi, const PixAxis& ax, int& a, int& b) {
  a = max(0, __float2int_ru(__fmaf_rn(lo, ax.nf, ax.lo)));
  b = min(ax.n - 1, __float2int_rd(__fmaf_rn(hi, ax.nf, ax.hi)));
}

/*
 * k_vertices: the FP32 screen position of every crossed edge of the slab,
 * once per edge (a surface vertex is shared by about six triangles).  Each
 * record: X, Y, Z, and one word of two bfloat16s: the bound on |X, Y - the
 * reference's value| above the relative depth bound, which is kVUndecided when
 * the bounds cannot decide whether the projection fails and kVFailed when it
 * certainly does (so that the maximum over a triangle's vertices is the
 * triangle's).  The edge runs from the owning corner to
 * corner m; the reference interpolates a triangle's vertex from its own tail
 * corner, which gives the same point up to FP64 rounding -- except where it
 * keeps the tail because |v1 - v0| < 1e-8, so that case is left undecided.
 *
 * Issue slots bound it, and a few percent of the cells own an edge, so a warp
 * works alone through a tile of consecutive cells in three steps that each
 * fill its lanes: 256 codes at a time are reduced to the cells that own an
 * edge, 32 of those to their edges, and 32 edges are computed; what is left
 * of a step waits in shared memory for the next one.  The vertices of a tile
 * are numbered in this order, so one offset per tile places them, and a tile
 * without any is skipped by its two offsets alone.  (A block of four warps
 * over 1024 cells computed its 76 to 141 edges in whole rounds of 128 and
 * spent half of its instructions on listing them.  With the shorter
 * vertex_record, per object at 512^3 f64 424 and 545 us -> 303 and 393, at 313 x
 * 269 x 311 125 and 160 -> 108 and 138; at 1536^3 f32 33 ms per frame -> 19.)
 */
constexpr int kVThreads = 128;
constexpr unsigned kVTileMax = 2048; /* cells of a warp's tile: a multiple of 256, numbered in at most 12 bits */

constexpr unsigned kVUndecided = 0x8000u, kVFailed = 0xFFFFu;

/* the record of a projected vertex (st: project_f's result; rz: 1 / |Z|) */
__device__ __forceinline__ float4 pack_vertex(int st, float X, float Y, float Z, float exy, float ez, float rz) {
  /* an infinite or NaN bound decides nothing */
  if (st > 0 && !(exy < 1e30f)) st = -1;
  const unsigned depth = st > 0 ? bf16_up(1.02f * ez * rz) : (st == 0 ? kVFailed : kVUndecided);
  return make_float4(X, Y, Z, __uint_as_float((bf16_up(st > 0 ? exy : 0.f) << 16) | depth));
}

/*
 * One crossed edge: from corner 0 of a cell to corner m.  Identity converter:
 * q = vertex - camera is the node's rounded camera-relative coordinate c plus
 * f times the rounded spacing d along the axes of m; with c and d within u and
 * f within e_f, each component is within
 *   1.02 u (|c| + |q|) + |d| (1.02 e_f + 1.02 u |f|) + coord_eps
 * of the reference's (coord_eps: its own FP64 rounding).  The dot products'
 * 4.2 u sum|a q| (see project_f) joins these bounds before the sums.
 */
template <typename T>
__device__ __forceinline__ float4 vertex_record(const FieldDev& F, const SlabDev& S, const SceneDev& s, const ThrF& th,
                                                const T* fd, unsigned cell, unsigned m, long long edge) {
  unsigned ui, uj, ukl;
  cell_ijk(F, cell, ui, uj, ukl);
  const unsigned k = (unsigned)S.kfirst + ukl;
  const T* at = fd + (((unsigned long long)k * (unsigned)F.ny + uj) * (unsigned)F.nx + ui);
  const T v0 = __ldg(at), v1 = __ldg(at + edge);
  const float2 ax = __ldg(F.vx + ui), ay = __ldg(F.vy + uj), az = __ldg(F.vz + k);
  float f = 0.f, e_f = 0.f;
  if (interp_edge(F.threshold, th, v0, v1, f, e_f) <= 0) return pack_vertex(-1, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f);
  const float c[3] = {ax.x, ay.x, az.x};
  const float d[3] = {(m & 1u) ? ax.y : 0.f, (m & 2u) ? ay.y : 0.f, (m & 4u) ? az.y : 0.f};
  const float ed = 1.02f * __fmaf_rn(kU32, fabsf(f), e_f);
  float q[3], e[3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    q[i] = __fmaf_rn(f, d[i], c[i]);
    /* 1.02 u (|c| + |q|) + 4.2 u |q| */
    e[i] = __fmaf_rn(fabsf(d[i]), ed, __fmaf_rn(1.02f * kU32, fabsf(c[i]), __fmaf_rn(5.23f * kU32, fabsf(q[i]), F.coord_eps)));
  }
  const float nq = __fmaf_rn(s.f_n[2], q[2], __fmaf_rn(s.f_n[1], q[1], s.f_n[0] * q[0]));
  const float lq = __fmaf_rn(s.f_lx[2], q[2], __fmaf_rn(s.f_lx[1], q[1], s.f_lx[0] * q[0]));
  const float mq = __fmaf_rn(s.f_ly[2], q[2], __fmaf_rn(s.f_ly[1], q[1], s.f_ly[0] * q[0]));
  auto bound = [&](const float a[3]) {
    return 1.0001f * __fmaf_rn(fabsf(a[2]), e[2], __fmaf_rn(fabsf(a[1]), e[1], fabsf(a[0]) * e[0]));
  };
  float X, Y, Z, exy, ez, rz;
  const int st = project_dots(s, nq, lq, mq, bound(s.f_n), bound(s.f_lx), bound(s.f_ly), fmaxf(1e-12f, F.proj_eps), X, Y,
                              Z, exy, ez, rz);
  return pack_vertex(st, X, Y, Z, exy, ez, rz);
}

/* the same with node positions in memory (a converter) */
template <typename T>
__device__ __forceinline__ float4 vertex_record_nodes(const FieldDev& F, const SlabDev& S, const SceneDev& scene,
                                                      const ThrF& th, const T* fd, unsigned cell, unsigned m,
                                                      long long edge) {
  unsigned ui, uj, ukl;
  cell_ijk(F, cell, ui, uj, ukl);
  const long long i = ui, j = uj, k = S.kfirst + ukl;
  float xa[3], xb[3], qv[3], eq[3];
  const float ce = corner_pos_f(F, i, j, k, 0, xa);
  corner_pos_f(F, i, j, k, (int)m, xb);
  const long long i0 = (k * F.ny + j) * F.nx + i;
  float X = 0.f, Y = 0.f, Z = 0.f, exy = 0.f, ez = 0.f, rz = 0.f;
  int st = -1;
  if (vertex_q<T>(scene, F, th, xa, __ldg(fd + i0), xb, __ldg(fd + i0 + edge), ce, qv, eq))
    st = project_f(scene, qv, eq, fmaxf(1e-12f, F.proj_eps), X, Y, Z, exy, ez, rz);
  return pack_vertex(st, X, Y, Z, exy, ez, rz);
}

template <typename T, bool NODES>
__global__ void __launch_bounds__(kVThreads)
k_vertices(FieldDev F, SlabDev S, SceneDev scene, const unsigned char* __restrict__ codes,
           VOffDev voff, long long n, unsigned tile, VertDev V) {
  pdl_enter();
  __shared__ unsigned s_cells[kVThreads / 32][32 + 256];      /* cell in the tile | code << 12 */
  __shared__ unsigned short s_edges[kVThreads / 32][32 * 8];  /* cell in the tile | corner m << 12 */
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  __shared__ long long s_off[8]; /* node offset of corner m */
  if (threadIdx.x < 8)
    s_off[threadIdx.x] = (threadIdx.x & 1u) + ((threadIdx.x >> 1) & 1u) * F.nx + (threadIdx.x >> 2) * F.nx * F.ny;
  __syncthreads();
  const long long c0 = (blockIdx.x * (long long)(kVThreads / 32) + warp) * tile;
  if (c0 >= n) return;
  const long long c1 = min(c0 + tile, n);
  const unsigned va = voff_at(voff, c0), vb = voff_at(voff, c1);
  if (va == vb) return;
  if (vb > V.cap) {
    /* more crossed edges than records (buffers sized before the count was known) */
    if (lane == 0) atomicOr(V.ovf, kOvfVertices);
    return;
  }
  unsigned* cells = s_cells[warp];
  unsigned short* edges = s_edges[warp];
  const T* fd = static_cast<const T*>(F.data);
  const ThrF th = thr_f(F.threshold);
  const unsigned len = (unsigned)(c1 - c0);
  unsigned at = 0;         /* the next cell of the tile to look at */
  unsigned nc = 0, hc = 0; /* cells waiting, from hc on */
  unsigned ne = 0, he = 0; /* edges waiting, from he on */
  unsigned out = va;       /* the next vertex */
  for (;;) {
    while (ne < 32 && (nc > 0 || at < len)) {
      while (nc < 32 && at < len) {
        /* the waiting cells to the front, then those of the next 256 codes (a
           code past the end reads as 0) */
        const unsigned cf = at + 8 * lane;
        uint2 cw = make_uint2(0u, 0u);
        if (cf + 8 <= len) {
          cw = __ldg(reinterpret_cast<const uint2*>(codes + c0 + cf)); /* c0 and cf are multiples of 8 */
        } else {
          for (unsigned q = 0; q < 8; q++)
            if (cf + q < len) (q < 4 ? cw.x : cw.y) |= (unsigned)codes[c0 + cf + q] << (8 * (q & 3));
        }
        at += 256;
        if (!__any_sync(0xFFFFFFFFu, (differing_bits(cw.x) | differing_bits(cw.y)) != 0u)) continue;
        const unsigned keep = lane < nc ? cells[hc + lane] : 0u;
        unsigned mixed = mixed_bytes(cw.x) | (mixed_bytes(cw.y) << 4), total;
        unsigned pos = nc + warp_exclusive(__popc(mixed), lane, total);
        __syncwarp();
        if (lane < nc) cells[lane] = keep;
        while (mixed) {
          const unsigned q = __ffs(mixed) - 1;
          mixed &= mixed - 1;
          const unsigned code = ((q < 4 ? cw.x : cw.y) >> (8 * (q & 3))) & 255u;
          cells[pos++] = (cf + q) | (code << 12);
        }
        __syncwarp();
        hc = 0;
        nc += total;
      }
      if (nc == 0) break;
      /* the waiting edges to the front, then those of up to 32 cells */
      const unsigned k = min(nc, 32u);
      const unsigned e = lane < k ? cells[hc + lane] : 0u; /* code 0: no edges */
      const unsigned keep = lane < ne ? edges[he + lane] : 0u;
      unsigned mask = owned_edges(e >> 12), total;
      unsigned pos = ne + warp_exclusive(__popc(mask), lane, total);
      __syncwarp();
      if (lane < ne) edges[lane] = (unsigned short)keep;
      while (mask) {
        const unsigned m = __ffs(mask); /* edge to corner m */
        mask &= mask - 1;
        edges[pos++] = (unsigned short)((e & 4095u) | (m << 12));
      }
      __syncwarp();
      he = 0;
      ne += total;
      hc += k;
      nc -= k;
    }
    if (ne == 0) break;
    const unsigned k = min(ne, 32u);
    if (lane < k) {
      const unsigned e = edges[he + lane];
      const unsigned cell = (unsigned)c0 + (e & 4095u), m = e >> 12;
      V.pos[out + lane] = NODES ? vertex_record_nodes<T>(F, S, scene, th, fd, cell, m, s_off[m])
                                : vertex_record<T>(F, S, scene, th, fd, cell, m, s_off[m]);
    }
    out += k;
    he += k;
    ne -= k;
  }
}

/*
 * One thread per triangle.  The render form gathers a rendered triangle's
 * FP32 screen vertices and their bounds (from k_vertices) and picks the
 * raster path that settles it: the tiny list (FP64 throughout) when the
 * bounds cannot decide its culling, the sliver list when its area may be
 * clamped, none when no pixel centre can lie in it, the cover list
 * otherwise -- only cover and sliver triangles are written, to the compact
 * lists k_raster reads.  The inspection form keeps the cube-edge ids and
 * flags of every triangle (tri.meta) and routes nothing.
 */
/* the depth of any covered fragment: the harmonic mean of the vertex depths
   with weights >= -1e-8 summing to 1, so within their range */
__device__ __forceinline__ void depth_interval(const float Z[3], float zr, float& dlo, float& dhi) {
  const float zmin = fminf(Z[0], fminf(Z[1], Z[2])), zmax = fmaxf(Z[0], fmaxf(Z[1], Z[2]));
  const float m = zr + 4e-6f;
  dlo = zmin - m * fabsf(zmin);
  dhi = zmax + m * fabsf(zmax);
}

/* what k_emit decided for one triangle */
struct EmitOut {
  int route; /* 0 no fragment, 1 tiny list, 2 cover list, 3 sliver list, 4 cover list with one pixel */
  float X[3], Y[3], Z[3], exy, zr; /* route 4: the depth interval in Z[0], Z[1], the pixel's i, j in zr, Z[2] */
};

/* inspection: a triangle's cube-edge ids, rendered flag and rank in the cell */
__device__ __forceinline__ unsigned emit_meta(const FieldDev& F, const SlabDev& S, const unsigned long long* lut,
                                              const unsigned char* __restrict__ codes, unsigned tc) {
  const unsigned ncx = (unsigned)(F.nx - 1), ncy = (unsigned)(F.ny - 1);
  const unsigned c = tc & kTcCellMask, r = tc >> kTcRankShift;
  unsigned ui, uj, ukl;
  cell_ijk(F, c, ui, uj, ukl);
  const unsigned uk = (unsigned)S.kfirst + ukl;
  const unsigned long long e = lut[codes[c] * 12 + r];
  /* rendered set: interior cells of the slab's own slices (contour/main.c:70-112) */
  const bool rendered = ui >= 1u && ui + 2u <= ncx && uj >= 1u && uj + 2u <= ncy && uk >= (unsigned)S.krender0 &&
                        uk < (unsigned)S.krender1;
  unsigned edges = 0;
#pragma unroll
  for (int q = 0; q < 3; q++) edges |= (unsigned)((e >> (18 + 5 * q)) & 31) << (5 * q);
  return edges | (rendered ? kMetaRendered : 0u) | (r << kMetaRankShift);
}

/*
 * One triangle of the render form: for a rendered triangle, its FP32 screen
 * vertices (gathered from k_vertices), its bounds and its raster route;
 * nothing is stored per triangle.  Vertex q lies on an edge owned by a cell at
 * one of the corner offsets s_off; the owner's word and its segment's offset
 * give the record.  The gathers' latency and the issue of their address
 * arithmetic bound the pass: one word per owner in place of its code and a
 * 16-bit offset, the rendered flag in place of the cell's coordinates, and a
 * 32-bit table entry with the masks ready (512^3, two levels: a frame 4.02 ->
 * 3.83 ms; 1536^3, four: 117.2 -> 111.4 ms; the scan, which writes the words,
 * 367 -> 366 us of the former).
 */
template <typename T, bool CHECK>
__device__ __forceinline__ void emit_one(const FieldDev& F, const SlabDev& S, const SceneDev& scene,
                                         const unsigned long long* lut, const unsigned* lut32, const unsigned* s_off,
                                         const unsigned char* __restrict__ codes, const VOffDev& voff,
                                         unsigned tc, const RasterDev& R, const VertDev& V,
                                         unsigned* __restrict__ checks, EmitOut& out) {
  int& route = out.route;
  float* X = out.X;
  float* Y = out.Y;
  float* Z = out.Z;
  route = 0;
  const unsigned c = tc & kTcCellMask, r = tc >> kTcRankShift;
  const unsigned own = __ldg(voff.word + c);
  if (!(own & kWordRendered)) return;
  const unsigned e32 = __ldg(lut32 + ((own >> 16) & 255u) * 12 + r);
  /* each step's three loads together: the chain's latency bounds the pass */
  unsigned oc[3], word[3], vi[3];
#pragma unroll
  for (int q = 0; q < 3; q++) oc[q] = c + s_off[(e32 >> (9 * q)) & 7u];
#pragma unroll
  for (int q = 0; q < 3; q++) word[q] = __ldg(voff.word + oc[q]);
#pragma unroll
  for (int q = 0; q < 3; q++) vi[q] = __ldg(voff.seg + (oc[q] >> kVSegShift));
#pragma unroll
  for (int q = 0; q < 3; q++)
    vi[q] += (word[q] & 0xFFFFu) + __popc((word[q] >> 16) & (e32 >> (9 * q + 3)) & 63u);
  unsigned exy_bits = 0, depth_bits = 0;
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const float4 p = __ldg(V.pos + vi[q]);
    const unsigned pk = __float_as_uint(p.w);
    X[q] = p.x;
    Y[q] = p.y;
    Z[q] = p.z;
    exy_bits = max(exy_bits, pk);
    depth_bits = max(depth_bits, pk & 0xFFFFu);
  }
  const float exy = out.exy = __uint_as_float(exy_bits & 0xFFFF0000u);
  const int status = depth_bits < kVUndecided ? 1 : (depth_bits == kVFailed ? 0 : -1);
  float& zr = out.zr;
  zr = status > 0 ? bf16_value(depth_bits) : 0.f;
  d3 v[3];
  bool ok = true;
  if (CHECK) {
    /* the reference's own vertices and projection */
    d3 p[3];
    unsigned ui, uj, ukl;
    cell_ijk(F, c, ui, uj, ukl);
    cell_vertices(F, ui, uj, S.kfirst + ukl, __ldg(lut + codes[c] * 12 + r), v);
#pragma unroll
    for (int q = 0; q < 3; q++) ok = project(scene, v[q], p[q]) && ok;
    if (status >= 0 && (status == 1) != ok) atomicAdd(checks + 0, 1u);
    if (status == 1 && ok) {
#pragma unroll
      for (int q = 0; q < 3; q++)
        if (fabs((double)X[q] - p[q].x) > exy || fabs((double)Y[q] - p[q].y) > exy ||
            fabs((double)Z[q] - p[q].z) > (double)zr * fabs((double)Z[q]))
          atomicAdd(checks + 1, 1u);
    }
  }
  if (status == 0) return;
  float errA;
  const float A = emit_area(X, Y, exy, errA);
  const bool decided = status > 0 && fabsf(A) < 3e38f && exy < 1e-3f && zr < 1e-3f;
  if (!decided) {
    route = 1;
  } else if (!area_unclamped(A, errA)) {
    /* the area may be clamped to +-1e-16 (render.c:108-111): the sliver
       pass tests the reference's whole box */
    route = 3;
  } else {
    /* the reference's area is certainly not clamped: its weights are
       barycentric up to the -1e-8 slack, so every covered pixel centre
       lies in the triangle's extent */
    const float xlo = fminf(X[0], fminf(X[1], X[2])), xhi = fmaxf(X[0], fmaxf(X[1], X[2]));
    const float ylo = fminf(Y[0], fminf(Y[1], Y[2])), yhi = fmaxf(Y[0], fmaxf(Y[1], Y[2]));
    const float mb = exy + 1e-6f * ((xhi - xlo) + (yhi - ylo)) + 1e-12f;
    int imin, imax, jmin, jmax;
    centre_range(xlo - mb, xhi + mb, scene.px, imin, imax);
    centre_range(ylo - mb, yhi + mb, scene.py, jmin, jmax);
    route = imin <= imax && jmin <= jmax ? (imin == imax && jmin == jmax ? 4 : 2) : 0;
    if (route == 4) {
      float dlo, dhi;
      depth_interval(Z, zr, dlo, dhi);
      Z[0] = dlo;
      Z[1] = dhi;
      Z[2] = __int_as_float(jmin);
      zr = __int_as_float(imin);
    }
    if (CHECK && route == 0 && ok) {
      /* no pixel of the reference's box may be covered */
      ExactTri ex;
      if (exact_tri(scene, v, ex))
        for (long long jj = ex.jmin; jj <= ex.jmax; jj++)
          for (long long ii = ex.imin; ii <= ex.imax; ii++) {
            double w0, w1, w2;
            if (exact_weights(ex, ii, jj, R.xs, R.ys, w0, w1, w2)) atomicAdd(checks + 2, 1u);
          }
    }
  }
}

/*
 * List appends without block barriers: each warp takes chunks of entries
 * from a list's counter (one atomic per chunk) and fills them with warp
 * ballots; a batch that does not fit the chunk's rest starts the next
 * chunk.  At the warp's end the rest of its last chunk is marked empty
 * (kNoTri), so a list holds its entries and fewer than one chunk of empty
 * ones per warp; the raster passes skip those.
 *
 * The cover list's chunks are 32 entries, one warp of k_raster.  A chunk holds
 * either triangles whose range is a single pixel (four of five; marked by the
 * sign of their error bound) or the others, so that a warp there runs one of
 * the two paths: lanes with one pixel do not wait for lanes that walk a range.
 * The sparse sliver list (about 2 % of the triangles) takes chunks of 8 so
 * that its empty entries stay few.
 */
constexpr unsigned kCoverChunk = 32, kSliverChunk = 8;
/* runs of 32 consecutive triangles per warp and window: 1 (grid-stride), 2,
   4 and 8 measured 5.57, 5.56, 5.51 and 5.51 ms per bench frame */
constexpr unsigned kEmitRun = 4;
constexpr unsigned kNoTri = 0xFFFFFFFFu;

/* record entries beyond the triangles that a grid of `blocks` k_emit blocks
   may leave empty (two kinds of cover chunks and one of slivers, one partial
   chunk each per warp) */
__host__ __device__ __forceinline__ unsigned long long emit_slack_for(unsigned long long blocks) {
  return (unsigned long long)(2 * kCoverChunk + kSliverChunk) * blocks * (256 / 32);
}

/* a warp's current chunk of a list: its next free slot and its end */
struct Chunk {
  unsigned next = 0, end = 0;
};

/* the list slot of this lane's entry (when `take`), every lane of the warp
   calling with the same chunk state */
template <unsigned kChunk>
__device__ __forceinline__ unsigned warp_append(unsigned long long* count, bool take, unsigned lane, Chunk& c) {
  const unsigned m = __ballot_sync(0xFFFFFFFFu, take);
  if (m == 0u) return 0u;
  const unsigned n = __popc(m), rank = __popc(m & ((1u << lane) - 1u)), room = c.end - c.next;
  unsigned slot = c.next + rank;
  if (n > room) {
    /* the next chunk: whole multiples of kChunk holding the batch's rest */
    const unsigned size = (n - room + kChunk - 1) / kChunk * kChunk;
    unsigned nb = 0;
    if (lane == 0) nb = (unsigned)atomicAdd(count, (unsigned long long)size);
    nb = __shfl_sync(0xFFFFFFFFu, nb, 0);
    if (rank >= room) slot = nb + (rank - room);
    c.next = nb + (n - room);
    c.end = nb + size;
  } else {
    c.next += n;
  }
  return slot;
}

template <typename T, bool CHECK, bool RENDER>
__global__ void __launch_bounds__(256, CHECK ? 1 : 8)
k_emit(FieldDev F, SlabDev S, SceneDev scene, const unsigned long long* __restrict__ lut_g,
       const unsigned char* __restrict__ codes, const unsigned* __restrict__ offsets,
       VOffDev voff, const unsigned* __restrict__ tri_cell,
       const unsigned long long* __restrict__ total_p, TriDev tri, RasterDev R, VertDev V,
       unsigned* __restrict__ checks) {
  pdl_trigger(); /* the table below does not depend on the preceding kernel */
  (void)offsets;
  /* the render form reads its table through L1 (one 12 KB copy per SM) rather
     than from a copy in each block's shared memory, which takes L1 from the
     gathers and shared memory from other kernels */
  __shared__ unsigned long long lut_s[RENDER ? 1 : kLutEntries];
  __shared__ unsigned s_off[8]; /* cell offset of corner m */
  if (RENDER) {
    const unsigned ncx = (unsigned)(F.nx - 1), ncxy = ncx * (unsigned)(F.ny - 1), m = threadIdx.x;
    if (m < 8) s_off[m] = (m & 1u) + ((m >> 1) & 1u) * ncx + (m >> 2) * ncxy;
  } else {
    for (int q = threadIdx.x; q < kLutEntries; q += blockDim.x) lut_s[q] = lut_g[q];
  }
  __syncthreads();
  const unsigned* lut32 = reinterpret_cast<const unsigned*>(lut_g + kLutEntries);
  pdl_wait();
  const long long T_ = (long long)*total_p;
  /* the record region holds the cover and sliver entries (at most the
     triangles) and every warp's unfilled chunk ends */
  const unsigned long long slack = RENDER ? emit_slack_for(gridDim.x) : 0ULL;
  if ((unsigned long long)T_ > tri.cap || (unsigned long long)T_ + slack > tri.rec_cap ||
      (V.pos && total_p[1] > V.cap)) {
    /* more triangles than the arrays hold, or more crossed edges than vertex
       records (sized before the counts were known): nothing is read or
       written, the frame is rendered again */
    if (blockIdx.x == 0 && threadIdx.x == 0)
      atomicOr(tri.ovf, (unsigned long long)T_ + slack > tri.rec_cap || (unsigned long long)T_ > tri.cap
                            ? kOvfTriangles
                            : kOvfVertices);
    return;
  }
  const unsigned lane = threadIdx.x & 31u;
  /* the grid works through windows of the slab's triangles, small enough
     that a window's cells and vertex records stay in L2 (blocks with ranges
     of their own measured slower: 1.59 -> 1.82 ms per frame); within a
     window each warp takes kEmitRun consecutive runs of 32, so the entries
     of a list chunk lie close together in the field and on screen, as the
     raster passes like them (a slab's triangles are numbered in 31 bits) */
  const unsigned tcount = (unsigned)T_;
  const unsigned window = gridDim.x * blockDim.x * kEmitRun;
  /* cover chunks of ranges and of single pixels, sliver chunks */
  Chunk cc, c1, cs;
  unsigned t = (blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) * kEmitRun + lane; /* this thread's triangle */
  /* a warp's lanes run the same iterations (warp-wide appends) */
  while (t - lane < tcount) {
    EmitOut e;
    e.route = 0;
    if (t < tcount) {
      const unsigned tc = tri_cell[t];
      if (RENDER) emit_one<T, CHECK>(F, S, scene, lut_g, lut32, s_off, codes, voff, tc, R, V, checks, e);
      else tri.meta[t] = emit_meta(F, S, lut_s, codes, tc);
    }
    if (RENDER) {
      /* the tiny list holds a few thousand entries per frame: one atomic each */
      if (e.route == 1) {
        const unsigned long long ti = atomicAdd(R.tiny_count, 1ULL);
        if (ti < R.tiny_cap) R.tiny[ti] = t; /* overflow: the host re-runs the slab */
      }
      const unsigned ci = warp_append<kCoverChunk>(R.cover_count, e.route == 2, lane, cc);
      const unsigned oi = warp_append<kCoverChunk>(R.cover_count, e.route == 4, lane, c1);
      const unsigned si = warp_append<kSliverChunk>(R.sliver_count, e.route == 3, lane, cs);
      if (e.route >= 2) {
        float4* rec = e.route == 3 ? R.sliver_rec - 3 * (long long)si : tri.rec + 3 * (long long)(e.route == 2 ? ci : oi);
        rec[0] = make_float4(e.X[0], e.Y[0], e.Z[0], e.X[1]);
        rec[1] = make_float4(e.Y[1], e.Z[1], e.X[2], e.Y[2]);
        rec[2] = make_float4(e.Z[2], e.route == 4 ? -e.exy : e.exy, e.zr, __uint_as_float(t));
      }
    }
    /* the next of the run, or the next window's first */
    t += 32;
    if (!(t & (32 * kEmitRun - 32))) t += window - 32 * kEmitRun;
  }
  if (RENDER) {
    /* the unfilled ends of the warp's last chunks are marked empty */
    const float4 none = make_float4(0.f, 0.f, 0.f, __uint_as_float(kNoTri));
    for (unsigned q = cc.next + lane; q < cc.end; q += 32) tri.rec[3 * (long long)q + 2] = none;
    for (unsigned q = c1.next + lane; q < c1.end; q += 32) tri.rec[3 * (long long)q + 2] = none;
    for (unsigned q = cs.next + lane; q < cs.end; q += 32) R.sliver_rec[2 - 3 * (long long)q] = none;
  }
}

/*
 * A pixel range holding the reference's bounding box (render.c:90-99):
 * [(0.5 + lo) n - 1, (0.5 + hi) n + 1] truncated and clamped to [0, n - 1],
 * for a triangle whose extent lies in [lo, hi].
 */
__device__ __forceinline__ void reference_box(float lo, float hi, int n, int& a, int& b) {
  /* in [-4, n + 4] the FP32 values are within 2u n + u of the exact ones:
     floor / ceil past a margin of 3u n hold the truncated bounds; NaN gives
     the whole axis */
  const float nf = (float)n;
  const float fa = fmaxf(-4.f, fminf(nf + 4.f, (0.5f + lo) * nf - 1.f));
  const float fb = fmaxf(-4.f, fminf(nf + 4.f, (0.5f + hi) * nf + 1.f));
  const float mg = 3.f * kU32 * nf + 1e-4f;
  /* both ends are clamped: a triangle off the image is tested at its border */
  a = fa == fa ? min(n - 1, max(0, __float2int_rd(fa - mg))) : 0;
  b = fb == fb ? max(0, min(n - 1, __float2int_ru(fb + mg))) : n - 1;
}

/* ------------------------------------------------------------------ */
/* triangles the single-precision filter cannot settle                 */
/* ------------------------------------------------------------------ */
/*
 * Triangles whose culling or bounds are too uncertain for the FP32 filter
 * (a vertex near the camera plane or the edge of the view, or an edge whose
 * value difference is near 1e-8).  The reference's vertices, projection
 * and area are computed once per triangle; when the area is not clamped
 * (|area| >= 1e-16, render.c:108-111) the covered pixel centres lie in the
 * triangle's extent, which holds no pixel centre for most of these
 * triangles; otherwise the reference's whole box is tested.  Fragments go
 * straight to the z-buffer.
 */
/* a double of lane `src` of the warp (every lane calls) */
__device__ __forceinline__ double shfl_d(double v, unsigned src) { return __shfl_sync(0xFFFFFFFFu, v, src); }

/*
 * Four lanes share one triangle: lane m < 3 of the four computes vertex m and
 * its projection, then every lane has all three (a warp-wide call; `has`:
 * this four's item exists).  An FP64 warp instruction takes as long for one
 * lane as for 32, so the chain is a third as long as one lane's alone: the
 * last fragments of a frame finish after 8 us instead of 26.
 */
__device__ __forceinline__ bool quad_project(const FieldDev& F, const SceneDev& s, long long i, long long j,
                                             long long k, unsigned long long e, bool has, ExactTri& x) {
  const unsigned lane = threadIdx.x & 31u, m = lane & 3u, g0 = lane & ~3u;
  d3 q = {0., 0., 0.};
  bool ok = false;
  if (has) {
    const unsigned v = m < 3 ? m : 0u;
    const int a = (int)((e >> (6 * v)) & 7), b = (int)((e >> (6 * v + 3)) & 7);
    const d3 p = interpolate(F.threshold, corner_pos(F, i, j, k, a), corner_value(F, i, j, k, a),
                             corner_pos(F, i, j, k, b), corner_value(F, i, j, k, b));
    ok = project(s, p, q);
  }
  const unsigned all = __ballot_sync(0xFFFFFFFFu, ok);
  x.v0 = {shfl_d(q.x, g0), shfl_d(q.y, g0), shfl_d(q.z, g0)};
  x.v1 = {shfl_d(q.x, g0 + 1), shfl_d(q.y, g0 + 1), shfl_d(q.z, g0 + 1)};
  x.v2 = {shfl_d(q.x, g0 + 2), shfl_d(q.y, g0 + 2), shfl_d(q.z, g0 + 2)};
  if (((all >> g0) & 7u) != 7u) return false;
  x.area = edge_fn(x.v0, x.v1, x.v2);
  x.area_inv = drcp(x.area < 0. ? fmin(x.area, -1.e-16) : fmax(x.area, +1.e-16));
  return true;
}

/* lane m's weight of that triangle at pixel (i, j): exact_weights_in by parts */
__device__ __forceinline__ double quad_weight(const ExactTri& x, unsigned m, double px, double py) {
  const d3 p = {px, py, 0.};
  const d3 va = m == 0 ? x.v1 : (m == 1 ? x.v2 : x.v0), vb = m == 0 ? x.v2 : (m == 1 ? x.v0 : x.v1);
  return dmul(x.area_inv, edge_fn(va, vb, p));
}

/* the same for emission index t of a slab */
__device__ __forceinline__ bool quad_triangle(const Geo& G, const SceneDev& s, long long t, bool has, ExactTri& x) {
  unsigned i = 0, j = 0, kl = 0;
  unsigned long long e = 0;
  if (has) {
    const unsigned tc = G.tri_cell[t];
    const unsigned c = tc & kTcCellMask, r = tc >> kTcRankShift;
    cell_ijk(G.F, c, i, j, kl);
    e = __ldg(G.lut + G.codes[c] * 12 + r);
  }
  return quad_project(G.F, s, i, j, G.S.kfirst + kl, e, has, x);
}

/* one tiny-list triangle by four lanes (a warp-wide call): the pixels of its
   range in turn over the four */
template <bool CHECK>
__device__ __forceinline__ void tiny_triangle(const Geo& G, const SceneDev& s, long long t, bool has,
                                              const RasterDev& R, unsigned long long order_base, const FrameObjs& O,
                                              unsigned* checks) {
  const unsigned m = threadIdx.x & 3u;
  ExactTri x;
  if (!quad_triangle(G, s, t, has, x)) return;
  exact_box(s, x);
  long long imin = x.imin, imax = x.imax, jmin = x.jmin, jmax = x.jmax;
  if (fabs(x.area) >= 1.e-16) {
    const double xlo = fmin(x.v0.x, fmin(x.v1.x, x.v2.x)), xhi = fmax(x.v0.x, fmax(x.v1.x, x.v2.x));
    const double ylo = fmin(x.v0.y, fmin(x.v1.y, x.v2.y)), yhi = fmax(x.v0.y, fmax(x.v1.y, x.v2.y));
    const double mb = 1e-6 * ((xhi - xlo) + (yhi - ylo)) + 1e-14;
    const long long W = s.width, H = s.height;
    const double ia = ceil((0.5 + (xlo - mb)) * (double)W - 0.5 - 1e-6);
    const double ib = floor((0.5 + (xhi + mb)) * (double)W - 0.5 + 1e-6);
    const double ja = ceil((0.5 + (ylo - mb)) * (double)H - 0.5 - 1e-6);
    const double jb = floor((0.5 + (yhi + mb)) * (double)H - 0.5 + 1e-6);
    imin = max(imin, (long long)fmax(ia, -1.0));
    imax = min(imax, (long long)fmin(ib, (double)W));
    jmin = max(jmin, (long long)fmax(ja, -1.0));
    jmax = min(jmax, (long long)fmin(jb, (double)H));
  }
  if (CHECK && m == 0) {
    for (long long j = x.jmin; j <= x.jmax; j++)
      for (long long i = x.imin; i <= x.imax; i++) {
        double w0, w1, w2;
        if (exact_weights(x, i, j, R.xs, R.ys, w0, w1, w2) && (i < imin || i > imax || j < jmin || j > jmax))
          atomicAdd(checks + 2, 1u);
      }
  }
  if (imin > imax || jmin > jmax) return;
  const unsigned long long order = order_of(G, order_base, t);
  long long i = imin + m, j = jmin; /* every fourth pixel, row by row */
  for (;;) {
    while (i > imax) {
      i -= imax - imin + 1;
      j++;
    }
    if (j > jmax) break;
    double w0, w1, w2;
    if (exact_weights(x, i, j, R.xs, R.ys, w0, w1, w2)) {
      const long long p = j * s.width + i;
      Hit h;
      h.key = depth_key(exact_depth(x, w0, w1, w2));
      hit_weights(w0, w1, w2, h);
      if (slot_max_near(O, s, G.lut, R.xs, R.ys, R.canvas + p, i, j, h.key, (order << 24) | kLoExact, R.zerr))
        keep_weights(R, p, order, h);
    }
    i += 4;
  }
}

/* a warp's buffer of candidates in shared memory; it is written out when
   fewer than kCandRoom are free (a chunk of ranges with more than that appends
   the rest one by one) */
constexpr unsigned kCandWarp = 96, kCandRoom = 48;

/* a warp's candidates, collected in shared memory and written to the list
   together: one atomic on the list's counter and coalesced stores per hundred
   of them, and no barrier between warps */
struct CandBuf {
  Candidate* buf;
  unsigned* count; /* the number in shared memory, while lanes append on their own */
  unsigned n = 0;
};

/* the buffer to the list; those past the capacity are dropped (the host sees
   the count and re-runs the slab) */
__device__ __forceinline__ void flush_candidates(const RasterDev& R, CandBuf& B) {
  if (B.n == 0) return;
  const unsigned lane = threadIdx.x & 31u;
  unsigned long long b = 0;
  if (lane == 0) b = atomicAdd(R.cand_count, (unsigned long long)B.n);
  b = __shfl_sync(0xFFFFFFFFu, b, 0);
  __syncwarp();
  for (unsigned u = lane; u < B.n; u += 32)
    if (b + u < R.cand_cap) R.cand[b + u] = B.buf[u];
  __syncwarp();
  B.n = 0;
}

__device__ __forceinline__ Candidate candidate(unsigned t, unsigned pixel, float dhi) {
  Candidate c;
  c.t = t;
  c.pixel = pixel;
  c.dhi = dhi;
  c.pad = 0;
  return c;
}

/* self-check of one triangle: every pixel that the reference covers lies in
   the tight range and the depth interval */
__device__ __noinline__ bool check_range(const Geo& G, const SceneDev& scene, const RasterDev& R, unsigned t, int imin,
                                         int imax, int jmin, int jmax, float dlo, float dhi, unsigned* checks,
                                         ExactTri& ex) {
  d3 wv[3];
  exact_vertices(G, t, wv);
  if (!exact_tri(scene, wv, ex)) return false;
  for (long long j = ex.jmin; j <= ex.jmax; j++)
    for (long long i = ex.imin; i <= ex.imax; i++) {
      double w0, w1, w2;
      if (exact_weights(ex, i, j, R.xs, R.ys, w0, w1, w2)) {
        if (i < imin || i > imax || j < jmin || j > jmax) atomicAdd(checks + 2, 1u);
        const double d = exact_depth(ex, w0, w1, w2);
        if (!(d <= (double)dhi && d >= (double)dlo)) atomicAdd(checks + 4, 1u);
      }
    }
  return true;
}
__device__ __noinline__ void check_pixel(const ExactTri& ex, const RasterDev& R, int i, int j, bool out, bool inside,
                                         unsigned* checks) {
  double x0, x1, x2;
  const bool cov = exact_weights(ex, i, j, R.xs, R.ys, x0, x1, x2);
  if (cov && out) atomicAdd(checks + 2, 1u);     /* dropped a covered pixel */
  if (!cov && inside) atomicAdd(checks + 3, 1u); /* called an uncovered pixel inside */
}

/* one chunk of the cover list: the 32 entries from `base` on (n in all, a
   multiple of 32), traversed front to back along z (the list is close to
   emission order, which follows z) so that near surfaces raise the floors
   early.  A warp-wide call; returns the chunk's entries */
template <bool CHECK>
__device__ __forceinline__ unsigned cover_warp(const Geo& G, const SceneDev& scene, const TriDev& tri,
                                               const RasterDev& R, unsigned* __restrict__ checks, long long base,
                                               long long n, CandBuf& B) {
  const int W = (int)scene.width, H = (int)scene.height;
  const unsigned lane = threadIdx.x & 31u;
  if (B.n + kCandRoom > kCandWarp) flush_candidates(R, B);
  const long long q = base + lane, qq = scene.z_descending ? n - 1 - q : q;
  const float4 r0 = __ldg(tri.rec + 3 * qq), r1 = __ldg(tri.rec + 3 * qq + 1), r2 = __ldg(tri.rec + 3 * qq + 2);
  const unsigned t = __float_as_uint(r2.w);
  const bool valid = t != kNoTri; /* an entry, not a chunk's empty end */
  const unsigned entries = __popc(__ballot_sync(0xFFFFFFFFu, valid));
  const bool single = __any_sync(0xFFFFFFFFu, valid && __float_as_int(r2.y) < 0);
  const float X[3] = {r0.x, r0.w, r1.z}, Y[3] = {r0.y, r1.x, r1.w};
  if (single) {
    bool cand = false;
    unsigned p = 0;
    const float dlo = r0.z, dhi = r1.y;
    if (valid) {
      const int i = __float_as_int(r2.z), j = __float_as_int(r2.x);
      bool out, inside;
      cover_test(cover_tri(X, Y, -r2.y), R.xsf[i], R.ysf[j], out, inside);
      p = (unsigned)j * (unsigned)W + (unsigned)i;
      if (CHECK) {
        ExactTri ex;
        if (check_range(G, scene, R, t, i, i, j, j, dlo, dhi, checks, ex)) check_pixel(ex, R, i, j, out, inside, checks);
      }
      if (inside) atomicMax(R.zlo + p, f_key(dlo));
      cand = !out;
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, cand);
    if (cand) B.buf[B.n + __popc(m & ((1u << lane) - 1u))] = candidate(t, p, dhi);
    B.n += __popc(m);
    return entries;
  }
  if (lane == 0) *B.count = B.n;
  __syncwarp();
  if (valid) {
    const float Z[3] = {r0.z, r1.y, r2.x};
    const float eps = r2.y, zr = r2.z;
    const CoverTri c = cover_tri(X, Y, eps);
    const float xlo = fminf(X[0], fminf(X[1], X[2])), xhi = fmaxf(X[0], fmaxf(X[1], X[2]));
    const float ylo = fminf(Y[0], fminf(Y[1], Y[2])), yhi = fmaxf(Y[0], fmaxf(Y[1], Y[2]));
    const float mb = eps + 1e-6f * ((xhi - xlo) + (yhi - ylo)) + 1e-12f;
    int imin, imax, jmin, jmax;
    centre_range(xlo - mb, xhi + mb, scene.px, imin, imax);
    centre_range(ylo - mb, yhi + mb, scene.py, jmin, jmax);
    float dlo, dhi;
    depth_interval(Z, zr, dlo, dhi);
    ExactTri ex;
    bool ex_ok = false;
    if (CHECK) ex_ok = check_range(G, scene, R, t, imin, imax, jmin, jmax, dlo, dhi, checks, ex);
    const unsigned dkey = f_key(dlo);
    for (int j = jmin; j <= jmax; j++) {
      const float py = R.ysf[j];
      for (int i = imin; i <= imax; i++) {
        bool out, inside;
        cover_test(c, R.xsf[i], py, out, inside);
        const unsigned p = (unsigned)j * (unsigned)W + (unsigned)i;
        if (CHECK && ex_ok) check_pixel(ex, R, i, j, out, inside, checks);
        if (inside) atomicMax(R.zlo + p, dkey);
        if (!out) {
          const unsigned at = atomicAdd(B.count, 1u);
          if (at < kCandWarp) {
            B.buf[at] = candidate(t, p, dhi);
          } else {
            const unsigned long long b = atomicAdd(R.cand_count, 1ULL);
            if (b < R.cand_cap) R.cand[b] = candidate(t, p, dhi);
          }
        }
      }
    }
  }
  __syncwarp();
  B.n = min(*B.count, kCandWarp);
  return entries;
}

/* |a - b| bound of a product of bounded factors, plus its rounding */
__device__ __forceinline__ float prod_err(float a, float ea, float b, float eb) {
  return fabsf(a) * eb + ea * fabsf(b) + ea * eb + kU32 * fabsf(a * b);
}

/*
 * One thread per requested triangle: its area-weighted face normal in FP32.
 * The reference's area * unit normal equals the cross product of two edges
 * up to a few FP64 ulps; the vertices are taken relative to the cell's corner
 * 0 (offsets from the rounded node spacings, interpolation as in vertex_q),
 * so the edge vectors keep their relative accuracy.  w: the largest bound of
 * the three components (infinite when none can be given).
 */
/*
 * The vertices of triangle u (triangulate.c:40-73) relative to its cell's
 * corner 0, in FP32 with a bound on each component's distance to the
 * reference's FP64 vertex minus that corner: corner offsets from the rounded
 * node spacings, the interpolation parameter from interp_param, and an
 * absolute allowance (coord_eps) for the reference's own FP64 rounding.  Edge
 * vectors formed from these keep their relative accuracy however far the
 * cell is from the origin.  False when a vertex cannot be bounded.  Needs
 * the spacing tables (identity converter).
 */
/* one vertex of that kind: on the edge from corner a to corner b at the
   interpolation parameter f (bound e_f), with the rounded node spacings sp of
   the cell */
__device__ __forceinline__ void rel_pos(const FieldDev& F, const float sp[3], unsigned a, unsigned b, float f,
                                        float e_f, float rv[3], float er[3]) {
#pragma unroll
  for (int d = 0; d < 3; d++) {
    /* corner offsets from corner 0 along axis d: the rounded spacing or 0 */
    const float oa = ((a >> d) & 1u) ? sp[d] : 0.f, ob = ((b >> d) & 1u) ? sp[d] : 0.f;
    const float dd = ob - oa;
    const float p = oa + f * dd;
    rv[d] = p;
    er[d] = 1.1f * (1.01f * kU32 * (fabsf(oa) + fabsf(f) * (fabsf(oa) + fabsf(ob))) + e_f * fabsf(dd) +
                    kU32 * (2.2f * fabsf(f * dd) + fabsf(p))) +
            F.coord_eps;
  }
}

template <typename T>
__device__ __forceinline__ bool cell_rel_vertices(const Geo& G, unsigned u, float rv[3][3], float er[3][3]) {
  const FieldDev& F = G.F;
  const T* fd = static_cast<const T*>(F.data);
  const ThrF th = thr_f(F.threshold);
  const unsigned tc = G.tri_cell[u];
  const unsigned c = tc & kTcCellMask, r = tc >> kTcRankShift;
  unsigned ui, uj, ukl;
  cell_ijk(F, c, ui, uj, ukl);
  const long long i = ui, j = uj, k = G.S.kfirst + ukl;
  const unsigned long long e = __ldg(G.lut + G.codes[c] * 12 + r);
  const float sp[3] = {__ldg(F.dgx + i), __ldg(F.dgy + j), __ldg(F.dgz + k)};
  const long long base = (k * F.ny + j) * F.nx + i;
  bool ok = true;
#pragma unroll
  for (int v = 0; v < 3; v++) {
    const unsigned a = (unsigned)((e >> (6 * v)) & 7), b = (unsigned)((e >> (6 * v + 3)) & 7);
    const long long ia = base + (a & 1u) + ((a >> 1) & 1u) * F.nx + (long long)(a >> 2) * F.nx * F.ny;
    const long long ib = base + (b & 1u) + ((b >> 1) & 1u) * F.nx + (long long)(b >> 2) * F.nx * F.ny;
    float f = 0.f, e_f = 0.f;
    if (interp_shade(F, th, ShadeVal<T>::load(fd, ia), ShadeVal<T>::load(fd, ib), f, e_f) < 0) ok = false;
    rel_pos(F, sp, a, b, f, e_f, rv[v], er[v]);
  }
  return ok;
}

/*
 * Slivers: triangles whose area may be clamped to +-1e-16 (render.c:108-111).
 * A covered pixel then need not lie in the triangle's extent, so the
 * reference's whole box is tested: with the clamped area a, w_k = e_k / a <
 * -1e-8 holds certainly when s e_k < -tau for the sign s of a (|a| < tau /
 * 1e-8), and the weights need not sum to 1.  A sliver whose pixels are all
 * certainly outside draws nothing; any other goes whole to the exact path
 * (tiny list).  One thread per sliver, in a list of their own so that a warp's
 * loops over these boxes stay converged.
 */
/*
 * The three screen edge vectors V_b - V_a of triangle t (edge k runs from
 * vertex (k + 1) % 3 to (k + 2) % 3, as the weights of render.c:115-133)
 * from its world edges dv (cell_rel_vertices) in the exact form
 *   dX = b_x ((l_x . dv) - rho_x (n . dv)) / (n . q_a + n . dv),
 *   rho_x = (X_a - a_x) / b_x = (l_x . q_a) / (n . q_a)
 * (and the same for Y), q_a = vertex a - camera, with a bound e on each
 * component.  A point-like triangle keeps the directions of its edges this
 * way, where its FP32 screen vertices (bounds ~1e-7) cannot.  False when no
 * bound can be given.
 */
template <typename T>
__device__ __forceinline__ bool screen_edges(const Geo& G, const SceneDev& s, unsigned t, const float X[3],
                                             const float Y[3], const float Z[3], float eps, float zr, float sdx[3],
                                             float sdy[3], float sde[3]) {
  float rv[3][3], er[3][3];
  if (!G.F.dgx || !cell_rel_vertices<T>(G, t, rv, er)) return false;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int a = (k + 1) % 3, b = (k + 2) % 3;
    float dv[3], edv[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      dv[d] = rv[b][d] - rv[a][d];
      edv[d] = er[a][d] + er[b][d] + kU32 * fabsf(dv[d]);
    }
    float nd = 0.f, ld = 0.f, md = 0.f, e_nd = 0.f, e_ld = 0.f, e_md = 0.f, an = 0.f, al = 0.f, am = 0.f;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      nd += s.f_n[d] * dv[d];
      ld += s.f_lx[d] * dv[d];
      md += s.f_ly[d] * dv[d];
      e_nd += fabsf(s.f_n[d]) * edv[d];
      e_ld += fabsf(s.f_lx[d]) * edv[d];
      e_md += fabsf(s.f_ly[d]) * edv[d];
      an += fabsf(s.f_n[d] * dv[d]);
      al += fabsf(s.f_lx[d] * dv[d]);
      am += fabsf(s.f_ly[d] * dv[d]);
    }
    /* the constants' rounding to float (u) and the dot products' (3u) */
    e_nd = 1.01f * (e_nd + 4.f * kU32 * an);
    e_ld = 1.01f * (e_ld + 4.f * kU32 * al);
    e_md = 1.01f * (e_md + 4.f * kU32 * am);
    const float nq = Z[a];
    const float Dn = nq + nd;
    const float e_Dn = 1.01f * (zr * fabsf(nq) + e_nd + kU32 * fabsf(Dn)) + 1e-37f;
    if (!(fabsf(Dn) > 4.f * e_Dn) || !isfinite(Dn)) return false;
    const float rx = (X[a] - s.f_ax) / s.f_bx, ry = (Y[a] - s.f_ay) / s.f_by;
    const float e_rx = 1.01f * (eps + kU32 * (fabsf(s.f_ax) + fabsf(X[a] - s.f_ax))) / fabsf(s.f_bx) + 3.f * kU32 * fabsf(rx);
    const float e_ry = 1.01f * (eps + kU32 * (fabsf(s.f_ay) + fabsf(Y[a] - s.f_ay))) / fabsf(s.f_by) + 3.f * kU32 * fabsf(ry);
    const float Nx = ld - rx * nd, Ny = md - ry * nd;
    const float e_Nx = e_ld + fabsf(rx) * e_nd + e_rx * fabsf(nd) + e_rx * e_nd + kU32 * (fabsf(ld) + 2.f * fabsf(rx * nd));
    const float e_Ny = e_md + fabsf(ry) * e_nd + e_ry * fabsf(nd) + e_ry * e_nd + kU32 * (fabsf(md) + 2.f * fabsf(ry * nd));
    const float iD = 1.f / Dn;
    sdx[k] = s.f_bx * Nx * iD;
    sdy[k] = s.f_by * Ny * iD;
    const float rel = e_Dn / (fabsf(Dn) - e_Dn);
    /* the reference forms V_b - V_a from two FP64 projections, each rounded by up to proj_eps */
    const float ex = 1.01f * fabsf(s.f_bx) * (e_Nx + fabsf(Nx) * rel) * fabsf(iD) + 5.f * kU32 * fabsf(sdx[k]) +
                     2.f * G.F.proj_eps;
    const float ey = 1.01f * fabsf(s.f_by) * (e_Ny + fabsf(Ny) * rel) * fabsf(iD) + 5.f * kU32 * fabsf(sdy[k]) +
                     2.f * G.F.proj_eps;
    sde[k] = fmaxf(ex, ey);
    if (!isfinite(sde[k]) || !isfinite(sdx[k]) || !isfinite(sdy[k])) return false;
  }
  return true;
}

/* 32 entries [base, base + 32) of the sliver list (n entries) by a warp;
   triangles the bounds cannot settle go to the tiny list.  Returns the entries */
template <typename T, bool CHECK>
__device__ __noinline__ unsigned sliver_warp(const Geo& G, const SceneDev& scene, const RasterDev& R,
                                             unsigned* __restrict__ checks, long long base, long long n) {
  const int W = (int)scene.width, H = (int)scene.height;
  unsigned entries = 0;
  {
    const long long q = base + (threadIdx.x & 31u);
    bool to_tiny = false;
    unsigned t32 = 0;
    const float4* rec = R.sliver_rec - 3 * q;
    float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0, r2 = make_float4(0.f, 0.f, 0.f, __uint_as_float(kNoTri));
    if (q < n) {
      r0 = __ldg(rec);
      r1 = __ldg(rec + 1);
      r2 = __ldg(rec + 2);
    }
    entries = __popc(__ballot_sync(0xFFFFFFFFu, __float_as_uint(r2.w) != kNoTri));
    if (__float_as_uint(r2.w) != kNoTri) { /* an entry, not a chunk's empty end */
      t32 = __float_as_uint(r2.w);
      const float X[3] = {r0.x, r0.w, r1.z}, Y[3] = {r0.y, r1.x, r1.w}, Z[3] = {r0.z, r1.y, r2.x};
      const float eps = r2.y, zr = r2.z;
      /* the screen edges from the world edges (exact form, tight bounds) */
      float sdx[3], sdy[3], sde[3];
      const bool refined = screen_edges<T>(G, scene, t32, X, Y, Z, eps, zr, sdx, sdy, sde);
      const EdgeF E0 = edge_f(X[1], Y[1], X[2], Y[2], eps);
      const EdgeF E1 = edge_f(X[2], Y[2], X[0], Y[0], eps);
      const EdgeF E2 = edge_f(X[0], Y[0], X[1], Y[1], eps);
      float errA;
      float A = edge_eval(E2, X[2], Y[2], eps, eps, errA);
      if (refined) {
        /* render.c:38-46 area from the refined edges: (V2 - V0) x (V1 - V0) */
        const float ax_ = -sdx[1], ay_ = -sdy[1], bx_ = sdx[2], by_ = sdy[2];
        const float p1 = ax_ * by_, p2 = ay_ * bx_;
        A = p1 - p2;
        errA = 1.1f * ((fabsf(ax_) + fabsf(ay_)) * sde[2] + sde[1] * (fabsf(bx_) + fabsf(by_)) +
                       2.f * sde[1] * sde[2] + kU32 * (fabsf(p1) + fabsf(p2) + fabsf(A))) +
               1e-15f * (fabsf(p1) + fabsf(p2)) + 1e-37f;
      }
      const float xlo = fminf(X[0], fminf(X[1], X[2])), xhi = fmaxf(X[0], fmaxf(X[1], X[2]));
      const float ylo = fminf(Y[0], fminf(Y[1], Y[2])), yhi = fmaxf(Y[0], fmaxf(Y[1], Y[2]));
      int imin, imax, jmin, jmax;
      /* area certainly not clamped after all: the weights are barycentric up
         to the -1e-8 slack, so every covered pixel centre lies in the
         triangle's extent (as for the cover list) and the per-pixel test runs over
         that box only */
      if (area_unclamped(A, errA)) {
        const float mb = eps + 1e-6f * ((xhi - xlo) + (yhi - ylo)) + 1e-12f;
        centre_range(xlo - mb, xhi + mb, scene.px, imin, imax);
        centre_range(ylo - mb, yhi + mb, scene.py, jmin, jmax);
      } else {
        reference_box(xlo - eps, xhi + eps, W, imin, imax);
        reference_box(ylo - eps, yhi + eps, H, jmin, jmax);
      }
      const float tau = 1.001e-8f * (fabsf(A) + errA + 1e-16f) + 1e-37f;
      const bool may_pos = A + errA >= 0.f; /* an area of exactly 0 is clamped to +1e-16 */
      const bool may_neg = A - errA < 0.f;
      ExactTri ex;
      bool ex_ok = false;
      if (CHECK) {
        d3 wv[3];
        exact_vertices(G, (long long)t32, wv);
        ex_ok = exact_tri(scene, wv, ex);
        if (ex_ok)
          for (long long j = ex.jmin; j <= ex.jmax; j++)
            for (long long i = ex.imin; i <= ex.imax; i++) {
              double w0, w1, w2;
              if (exact_weights(ex, i, j, R.xs, R.ys, w0, w1, w2) && (i < imin || i > imax || j < jmin || j > jmax))
                atomicAdd(checks + 2, 1u);
            }
      }
      for (int j = jmin; j <= jmax && (CHECK || !to_tiny); j++) {
        const float py = R.ysf[j];
        for (int i = imin; i <= imax && (CHECK || !to_tiny); i++) {
          const float px = R.xsf[i];
          const float ep = 0.5f * kU32;
          bool out;
          if (refined) {
            /* the edge values from the refined edges, for each possible sign of the area */
            bool po = false, no = false;
#pragma unroll
            for (int k = 0; k < 3; k++) {
              const int a = (k + 1) % 3;
              const float ux = px - X[a], uy = py - Y[a];
              const float eux = eps + ep + kU32 * fabsf(ux), euy = eps + ep + kU32 * fabsf(uy);
              const float f = ux * sdy[k] - uy * sdx[k];
              const float ef = 1.1f * (fabsf(ux) * sde[k] + eux * fabsf(sdy[k]) + eux * sde[k] + fabsf(uy) * sde[k] +
                                       euy * fabsf(sdx[k]) + euy * sde[k] +
                                       2.f * kU32 * (fabsf(ux * sdy[k]) + fabsf(uy * sdx[k])) + kU32 * fabsf(f));
              po = po || (f + ef < -tau);
              no = no || (f - ef > tau);
            }
            out = (!may_pos || po) && (!may_neg || no);
          } else {
            float e0, e1, e2;
            const float f0 = edge_eval(E0, px, py, ep, eps, e0);
            const float f1 = edge_eval(E1, px, py, ep, eps, e1);
            const float f2 = edge_eval(E2, px, py, ep, eps, e2);
            const bool pos_out = (f0 + e0 < -tau) || (f1 + e1 < -tau) || (f2 + e2 < -tau);
            const bool neg_out = (f0 - e0 > tau) || (f1 - e1 > tau) || (f2 - e2 > tau);
            out = (!may_pos || pos_out) && (!may_neg || neg_out);
          }
          if (CHECK && ex_ok) {
            double x0, x1, x2;
            if (exact_weights(ex, i, j, R.xs, R.ys, x0, x1, x2) && out) atomicAdd(checks + 2, 1u);
          }
          to_tiny = to_tiny || !out;
        }
      }
    }
    if (to_tiny) { /* a few hundred per frame */
      const unsigned long long rt = atomicAdd(R.tiny_count, 1ULL);
      if (rt < R.tiny_cap) R.tiny[rt] = t32; /* overflow: the host re-runs the slab */
    }
    __syncwarp();
  }
  return entries;
}

/*
 * k_raster: the cover list's chunks, then the sliver list in warps' worth, in
 * one grid of resident blocks.  Issue slots bound it.  A warp has triangles of
 * one kind (see the list appends), and the warps run independently: mixed
 * lanes walking their ranges used 21.6 of 32, block-wide candidate appends
 * had the warps wait on each other, and half as many instructions remain.  Per
 * object at 313 x 269 x 311 f64: 172 and 249 us -> 134 and 177; at 512^3 and
 * 1920 x 1080 222 and 305 -> 193 and 268.
 */
template <typename T, bool CHECK>
__global__ void __launch_bounds__(128, 8)
k_raster(const __grid_constant__ Geo G, const __grid_constant__ SceneDev scene, const __grid_constant__ TriDev tri,
         const __grid_constant__ RasterDev R, unsigned* __restrict__ checks) {
  pdl_enter();
  __shared__ Candidate s_cand[4][kCandWarp];
  __shared__ unsigned s_count[4];
  CandBuf B;
  B.buf = s_cand[threadIdx.x >> 5];
  B.count = s_count + (threadIdx.x >> 5);
  const long long nc = (long long)*R.cover_count, ns = (long long)*R.sliver_count;
  const long long wc = nc / 32, ws = (ns + 31) / 32;
  unsigned cover = 0, sliver = 0; /* the warp's entries, for the statistics */
  for (long long w = blockIdx.x * 4LL + (threadIdx.x >> 5); w < wc + ws; w += gridDim.x * 4LL) {
    if (w < wc) cover += cover_warp<CHECK>(G, scene, tri, R, checks, 32 * w, nc, B);
    else sliver += sliver_warp<T, CHECK>(G, scene, R, checks, 32 * (w - wc), ns);
  }
  flush_candidates(R, B);
  if ((threadIdx.x & 31u) == 0 && cover) atomicAdd(R.listed_count, (unsigned long long)cover);
  if ((threadIdx.x & 31u) == 0 && sliver) atomicAdd(R.listed_count + 1, (unsigned long long)sliver);
}

/* ------------------------------------------------------------------ */
/* k_finish: the candidates that can win                                 */
/* ------------------------------------------------------------------ */
/* a float pair's value hi + lo, |lo| about an ulp of hi */
struct fpair {
  float h, l;
};

/* a . c for float-pair vectors: exact products (fused multiply-adds give
   their rounding errors), two-sums, and one rounding of the low part; within
   2^-40 sum|a c| of the exact value with ample room (the terms dropped are of
   2^-47) */
__device__ __forceinline__ fpair dot_pair(const float ah[3], const float al[3], const float2 c[3], float& mag) {
  float p[3], e[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    p[d] = ah[d] * c[d].x;
    e[d] = __fmaf_rn(ah[d], c[d].x, -p[d]);
    e[d] = __fmaf_rn(ah[d], c[d].y, e[d]);
    e[d] = __fmaf_rn(al[d], c[d].x, e[d]);
  }
  mag = fabsf(p[0]) + fabsf(p[1]) + fabsf(p[2]);
  float s, t, s2, t2;
  two_diff(p[0], -p[1], s, t);
  two_diff(s, -p[2], s2, t2);
  const float lo = (t + t2) + (e[0] + e[1] + e[2]);
  fpair r;
  r.h = s2 + lo;
  r.l = (s2 - r.h) + lo;
  return r;
}

/* a b - c d for float pairs, and a bound on its distance to the exact value */
__device__ __forceinline__ fpair cross_pair(fpair a, fpair b, fpair c, fpair d) {
  const float p = a.h * b.h, q = c.h * d.h;
  float e = __fmaf_rn(a.h, b.h, -p), f = __fmaf_rn(c.h, d.h, -q);
  e = __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, e));
  f = __fmaf_rn(c.h, d.l, __fmaf_rn(c.l, d.h, f));
  fpair r;
  two_diff(p, q, r.h, r.l);
  r.l += e - f;
  return r;
}

/*
 * A candidate fragment without FP64: 0 = the reference does not draw it, 1 =
 * it does, with h's depth within kDepthTol and weights within h.ew of the
 * reference's, 2 = these bounds cannot be given or decide nothing (the exact
 * path).
 *
 * With q = vertex - camera, N = n . q, L = l_x . q, M = l_y . q, the pixel is
 * off the vertex by px - x = U / N, py - y = V / N (project.c:9-67), where
 *   U = (px - a_x) N - b_x L,  V = (py - a_y) N - b_y M,
 * so the edge functions of render.c:38-46 are
 *   e_0 = F_0 / (N_1 N_2),  F_0 = U_2 V_1 - U_1 V_2  (and cyclically),
 * the weights e_k / sum e = F_k N_k / sum F N and the harmonic depth
 * 1 / sum (w / N) = sum F N / sum F = N_c + sum F (N - N_c) / sum F for any
 * N_c.  U and V are small differences of large terms: they are formed for the
 * cell's corner 0 in float pairs, and the vertices add their offsets from it
 * (rounded node spacings times the interpolation parameter), which floats
 * hold to their own relative accuracy.  So U, V and N are good to about 1e-7 of
 * the triangle's size, however small it is on screen, and so are the weights.
 *
 * Errors: tau bounds a vertex's offset per component and the rounding of a
 * dot product with it (5u of its size), as the sum of |n| etc. (SceneDev's
 * f_n1, f_lx1, f_ly1) scales it; the reference's own rounding of a screen
 * coordinate (proj_eps) is added to U and V.  Per fragment about 600 FP32
 * instructions replace about 560 FP64 ones, each of which holds the pipe as
 * long as 64 of the former: at 128^3 f64 and 1024 x 1024 (166 k fragments, 1.4 k
 * of them left open) the FP64 test took 160 us, this 23 us and k_exact 17; at
 * 512^3 f64, two levels, 1920 x 1080, 265 us per object became 45 and 27.
 */
template <typename T>
__device__ __forceinline__ int fast_fragment(const Geo& G, const SceneDev& s, const RasterDev& R, unsigned t,
                                             unsigned pi, unsigned pj, Hit& h) {
  const FieldDev& F = G.F;
  const T* fd = static_cast<const T*>(F.data);
  const unsigned tc = G.tri_cell[t];
  const unsigned c = tc & kTcCellMask, r = tc >> kTcRankShift;
  unsigned i, j, kl;
  cell_ijk(F, c, i, j, kl);
  const long long k = G.S.kfirst + kl;
  const unsigned long long e = __ldg(G.lut + G.codes[c] * 12 + r);
  const float2 cc[3] = {__ldg(F.cgx + i), __ldg(F.cgy + j), __ldg(F.cgz + k)};
  const float sp[3] = {__ldg(F.dgx + i), __ldg(F.dgy + j), __ldg(F.dgz + k)};
  const float2 pa = __ldg(R.xsa + pi), pb = __ldg(R.ysa + pj);
  const long long base = (k * F.ny + j) * F.nx + i, sxy = F.nx * F.ny;
  const ThrF th = thr_f(F.threshold);
  /* offsets of the vertices from corner 0, their bound and size */
  const float hm = fmaxf(fabsf(sp[0]), fmaxf(fabsf(sp[1]), fabsf(sp[2])));
  float rv[3][3], er = 0.f, rm = 0.f;
  typename ShadeVal<T>::type va[3], vb[3];
  unsigned ca[3], cb[3];
#pragma unroll
  for (int v = 0; v < 3; v++) {
    ca[v] = (unsigned)((e >> (6 * v)) & 7);
    cb[v] = (unsigned)((e >> (6 * v + 3)) & 7);
    va[v] = ShadeVal<T>::load(fd, base + (ca[v] & 1u) + ((ca[v] >> 1) & 1u) * F.nx + (ca[v] >> 2) * sxy);
    vb[v] = ShadeVal<T>::load(fd, base + (cb[v] & 1u) + ((cb[v] >> 1) & 1u) * F.nx + (cb[v] >> 2) * sxy);
  }
#pragma unroll
  for (int v = 0; v < 3; v++) {
    float f = 0.f, e_f = 0.f;
    if (interp_shade(F, th, va[v], vb[v], f, e_f) < 0) return 2;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float oa = ((ca[v] >> d) & 1u) ? sp[d] : 0.f, ob = ((cb[v] >> d) & 1u) ? sp[d] : 0.f;
      rv[v][d] = __fmaf_rn(f, ob - oa, oa);
      rm = fmaxf(rm, fabsf(rv[v][d]));
    }
    /* spacings within u of the grid's, one rounding of the fused sum, f within e_f */
    er = fmaxf(er, hm * __fmaf_rn(1.02f, e_f, 3.2f * kU32 * (1.f + fabsf(f))));
  }
  const float tau = 1.01f * (er + F.coord_eps + 5.f * kU32 * rm) + 1e-37f;
  /* corner 0 in float pairs */
  float mN, mL, mM;
  const fpair N = dot_pair(s.f_n, s.n_lo, cc, mN), L = dot_pair(s.f_lx, s.lx_lo, cc, mL),
              M = dot_pair(s.f_ly, s.ly_lo, cc, mM);
  const fpair Uc = cross_pair({pa.x, pa.y}, N, {s.f_bx, s.bx_lo}, L), Vc = cross_pair({pb.x, pb.y}, N, {s.f_by, s.by_lo}, M);
  /* the vertices */
  float U[3], V[3], Nv[3], dN[3], Um = 0.f, Vm = 0.f, Nm = 0.f, dm = 0.f;
#pragma unroll
  for (int v = 0; v < 3; v++) {
    const float* q = rv[v];
    dN[v] = __fmaf_rn(s.f_n[2], q[2], __fmaf_rn(s.f_n[1], q[1], s.f_n[0] * q[0]));
    const float dL = __fmaf_rn(s.f_lx[2], q[2], __fmaf_rn(s.f_lx[1], q[1], s.f_lx[0] * q[0]));
    const float dM = __fmaf_rn(s.f_ly[2], q[2], __fmaf_rn(s.f_ly[1], q[1], s.f_ly[0] * q[0]));
    U[v] = (Uc.h + __fmaf_rn(pa.x, dN[v], -(s.f_bx * dL))) + Uc.l;
    V[v] = (Vc.h + __fmaf_rn(pb.x, dN[v], -(s.f_by * dM))) + Vc.l;
    Nv[v] = N.h + (N.l + dN[v]);
    Um = fmaxf(Um, fabsf(U[v]));
    Vm = fmaxf(Vm, fabsf(V[v]));
    Nm = fmaxf(Nm, fabsf(Nv[v]));
    dm = fmaxf(dm, fabsf(dN[v]));
  }
  constexpr float kPair = 9.1e-13f; /* 2^-40 */
  const float eN = s.f_n1 * tau;
  /* the offsets' errors and the roundings of their sums (the partial sums are
     at most |U| plus the offset's size in both parts), the corner's pairs, and
     the reference's rounding of the screen coordinate */
  const float bx = fabsf(s.f_bx), by = fabsf(s.f_by);
  const float sU = __fmaf_rn(fabsf(pa.x), s.f_n1, bx * s.f_lx1), sV = __fmaf_rn(fabsf(pb.x), s.f_n1, by * s.f_ly1);
  const float gx = fabsf(pa.x) + fabsf(s.f_ax) + 1.f, gy = fabsf(pb.x) + fabsf(s.f_ay) + 1.f;
  const float eU = 1.01f * (sU * tau + 3.f * kU32 * (Um + sU * rm) + kPair * (gx * mN + bx * mL) + Nm * F.proj_eps);
  const float eV = 1.01f * (sV * tau + 3.f * kU32 * (Vm + sV * rm) + kPair * (gy * mN + by * mM) + Nm * F.proj_eps);
  const float F0 = U[2] * V[1] - U[1] * V[2], F1 = U[0] * V[2] - U[2] * V[0], F2 = U[1] * V[0] - U[0] * V[1];
  const float eF = 2.04f * (Um * eV + Vm * eU + eU * eV) + 5.f * kU32 * Um * Vm;
  const float G0 = F0 * Nv[0], G1 = F1 * Nv[1], G2 = F2 * Nv[2];
  const float Fm = fmaxf(fabsf(F0), fmaxf(fabsf(F1), fabsf(F2)));
  const float eNv = 1.01f * eN + 2.f * kU32 * Nm + kPair * mN;
  const float eG = 1.02f * (Nm * eF + Fm * eNv + eF * eNv) + 2.f * kU32 * Nm * Fm;
  const float A = G0 + G1 + G2, SF = F0 + F1 + F2;
  const float rA = 6.f * kU32 * Nm * Fm; /* A's own rounding */
  if (!(fabsf(A) > 4.f * (3.f * eG + rA)) || !(fabsf(SF) > 4.f * (3.f * eF + 6.f * kU32 * Fm)) ||
      !(fabsf(A) > 1e-30f) || !(fabsf(A) < 1e30f) || !(fabsf(SF) > 1e-30f) || !(fabsf(SF) < 1e30f))
    return 2;
  const float iA = __fdividef(1.f, A), iS = __fdividef(1.f, SF); /* 2 ulp on this range */
  const float w0 = G0 * iA, w1 = G1 * iA, w2 = G2 * iA;
  /* with errors d of the G: w' - w = (d_k - w_k sum d) / A', so at most
     (|1 - w_k| + 2 |w_k|) e_G / (|A| - 3 e_G), and |A| - 3 e_G > 3/4 |A| */
  const float wm = fmaxf(1.f, fmaxf(fabsf(w0), fmaxf(fabsf(w1), fabsf(w2))));
  const float cm = fminf(w0, fminf(w1, w2)) >= 0.f ? 2.f : 1.f + 3.f * wm;
  const float ew = 1.4f * (cm * eG + wm * rA) * fabsf(iA) + 6.f * kU32 * wm;
  if (w0 + ew < kWOut || w1 + ew < kWOut || w2 + ew < kWOut) return 0;
  if (!(w0 - ew > kWIn && w1 - ew > kWIn && w2 - ew > kWIn) || !(ew < 0.01f)) return 2;
  const float corr = (F0 * dN[0] + F1 * dN[1] + F2 * dN[2]) * iS;
  /* likewise corr' - corr = sum d_k (dN_k - corr) / SF' + a mean of the dN's errors */
  const float ds = fmaxf(dN[0], fmaxf(dN[1], dN[2])) - fminf(dN[0], fminf(dN[1], dN[2]));
  const float ed = 1.4f * (3.f * eF * 1.01f * ds + 18.f * kU32 * Fm * dm) * fabsf(iS) + 1.02f * eN + 8.f * kU32 * dm +
                   kPair * mN + 1e-14f * fabsf(N.h);
  /* against the fragment's own depth: where a cell is not small against its
     distance, corner 0 may be several times as deep */
  if (!(ed < 0.9f * kDepthTol * fabsf(N.h + (N.l + corr)))) return 2;
  h.key = depth_key(dadd((double)N.h, dadd((double)N.l, (double)corr)));
  h.w0 = w0;
  h.w1 = w1;
  h.ew = ew;
  h.ed = ed;
  return 1;
}

/* self-check of a fast fragment against the reference's: f its result, x (when
   drawn) the exact one */
__device__ __forceinline__ void check_fast(int f, const Hit& h, bool drawn, const Hit& x, unsigned* checks) {
  if (f == 0 && drawn) atomicAdd(checks + 2, 1u);
  if (f == 1 && !drawn) atomicAdd(checks + 3, 1u);
  if (f == 1 && drawn) {
    const double a = depth_from_key(h.key), b = depth_from_key(x.key);
    /* the depth within its bound, and the bound within the tolerance of this depth */
    if (!(fabs(a - b) <= (double)h.ed) || !((double)h.ed <= (double)kDepthTol * fabs(b)) ||
        fabsf(h.w0 - x.w0) > h.ew + x.ew || fabsf(h.w1 - x.w1) > h.ew + x.ew)
      atomicAdd(checks + 4, 1u);
  }
}

/* one candidate by the reference's arithmetic, into a z-buffer that may hold approximate depths */
template <bool CHECK>
__device__ __noinline__ void finish_exact(const Geo& G, const SceneDev& scene, unsigned t, unsigned pixel,
                                          const RasterDev& R, unsigned long long order_base, const FrameObjs& O,
                                          unsigned* checks) {
  const unsigned pj = pixel / (unsigned)scene.width, pi = pixel - pj * (unsigned)scene.width;
  Hit h;
  if (!exact_fragment<CHECK>(G, scene, t, pi, pj, R.xs, R.ys, checks, h)) return;
  const unsigned long long order = order_of(G, order_base, t);
  if (slot_max_near(O, scene, G.lut, R.xs, R.ys, R.canvas + pixel, pi, pj, h.key, (order << 24) | kLoExact, R.zerr))
    keep_weights(R, pixel, order, h);
}

/*
 * k_finish: the candidates that can still win.  A block filters a chunk of
 * candidates at a time against the final depth floors into a shared list and
 * takes whole rounds of its threads from it once it holds kFinRun of them,
 * keeping the rest for the next round.  The grid is what is resident at once
 * (a round is a chain of loads that more blocks would not shorten), and the
 * chunk 1024 candidates, or the blocks' equal shares when there are fewer: a
 * small frame's 1500 fragments took 70 us on four blocks.
 *
 * kFinFast (frames whose depths nobody reads, with float-pair coordinates):
 * fast_fragment; the few fragments that it leaves open, and those near the
 * slot's depth, go to a list for k_exact, because a warp with one FP64 lane
 * holds the pipe as long as with 32 (run here, 2 % of them kept half of the
 * FP64 time, and the FP64 code's registers half of the warps away).
 * kFinExact (every depth of the frame is exact): the reference's FP64
 * fragment test for every candidate, in the registers of four blocks per SM.
 * kFinList (a converter's object in a frame with approximate depths): every
 * candidate to the list.
 */
constexpr unsigned kFinChunk = 1024, kFinRun = 512;
enum FinMode { kFinFast, kFinExact, kFinList };
__host__ __device__ constexpr int fin_per_sm(FinMode m) { return m == kFinFast ? 3 : 4; }
template <typename T, bool CHECK, FinMode MODE>
__global__ void __launch_bounds__(256, CHECK ? 1 : fin_per_sm(MODE))
k_finish(const __grid_constant__ Geo G, const __grid_constant__ SceneDev scene, const __grid_constant__ RasterDev R,
         unsigned long long order_base, unsigned* __restrict__ checks) {
  pdl_enter();
  /* before a chunk is filtered the list holds fewer than kFinRun entries */
  __shared__ Candidate s_live[kFinRun + kFinChunk];
  __shared__ unsigned s_n;
  const unsigned long long nc = min(*R.cand_count, R.cand_cap);
  const unsigned chunk = nc >= (unsigned long long)kFinChunk * gridDim.x
                             ? kFinChunk
                             : max(32u, ((unsigned)nc / gridDim.x + 32u) / 32u * 32u);
  const unsigned long long nb = (nc + chunk - 1) / chunk;
  if (threadIdx.x == 0) s_n = 0u;
  __syncthreads();
  unsigned have = 0; /* entries in the list (s_n between the filter passes) */
  for (unsigned long long b = blockIdx.x;; b += gridDim.x) {
    const bool more = b < nb;
    if (more) {
      /* a thread's candidates and their floors in flight together */
      Candidate c[kFinChunk / 256];
      unsigned floor[kFinChunk / 256];
#pragma unroll
      for (unsigned u = 0; u < kFinChunk / 256; u++) {
        const unsigned w = u * 256 + threadIdx.x;
        const unsigned long long q = b * chunk + w;
        c[u].t = kNoTri;
        if (w < chunk && q < nc) {
          const uint4 v = __ldg(reinterpret_cast<const uint4*>(R.cand + q));
          c[u] = {v.x, v.y, __uint_as_float(v.z), v.w};
        }
      }
#pragma unroll
      for (unsigned u = 0; u < kFinChunk / 256; u++) floor[u] = c[u].t != kNoTri ? R.zlo[c[u].pixel] : 0xFFFFFFFFu;
#pragma unroll
      for (unsigned u = 0; u < kFinChunk / 256; u++)
        /* a certainly drawn fragment of this pixel is nearer than anything this one can reach */
        if (c[u].t != kNoTri && f_key(c[u].dhi) >= floor[u]) s_live[atomicAdd(&s_n, 1u)] = c[u];
    }
    __syncthreads();
    const unsigned n = s_n;
    __syncthreads(); /* every thread has read n before the next filter pass adds to it */
    if (threadIdx.x == 0 && n > have) atomicAdd(R.live_count, (unsigned long long)(n - have));
    have = n;
    if (n >= kFinRun || !more) {
      const unsigned take = more ? n / 256 * 256 : n; /* whole rounds, all at the end */
      for (unsigned e = threadIdx.x; e < take; e += 256) {
        const Candidate c = s_live[e];
        const unsigned pj = c.pixel / (unsigned)scene.width, pi = c.pixel - pj * (unsigned)scene.width;
        Hit h;
        int f = 2;
        if (MODE == kFinFast) {
          f = fast_fragment<T>(G, scene, R, c.t, pi, pj, h);
          if (CHECK && f != 2) {
            Hit x;
            const bool drawn = exact_fragment<CHECK>(G, scene, c.t, pi, pj, R.xs, R.ys, checks, x);
            check_fast(f, h, drawn, x, checks);
          }
          if (f == 1) {
            const unsigned long long order = order_of(G, order_base, c.t);
            f = slot_max_approx(R.canvas + c.pixel, h.key, order << 24, R.zerr);
            if (f == 1) keep_weights(R, c.pixel, order, h);
          }
        }
        if (MODE == kFinExact) {
          f = 0;
          if (exact_hit<CHECK>(G, scene, c.t, pi, pj, R.xs, R.ys, checks, h)) {
            const unsigned long long order = order_of(G, order_base, c.t);
            if (slot_max(R.canvas + c.pixel, h.key, order << 24, R.zerr)) keep_weights(R, c.pixel, order, h);
          }
        }
        if (f == 2) R.hard[atomicAdd(R.hard_count, 1ULL)] = make_uint2(c.t, c.pixel); /* one entry per candidate: fits */
      }
      __syncthreads();
      /* the rest (fewer than 256, from take >= 256 on) to the front */
      const unsigned rest = n - take;
      Candidate c = {};
      if (threadIdx.x < rest) c = s_live[take + threadIdx.x];
      __syncthreads();
      if (threadIdx.x < rest) s_live[threadIdx.x] = c;
      if (threadIdx.x == 0) s_n = rest;
      __syncthreads();
      have = rest;
    }
    if (!more) break;
  }
}

/*
 * k_exact: the candidates that k_finish left open, then the tiny list (the
 * reference's arithmetic for the whole triangle), four lanes each.  Both end
 * in the z-buffer's maximum, so their order does not matter.  Blocks of one
 * warp, so that a short list spreads over all SMs; the tiny list goes to the
 * blocks after the last fragments'.  Bound by one item's chain of FP64
 * operations until the lists fill the grid.
 *
 * Of more open fragments than the grid has lanes (surfaces that coincide, a
 * field with a converter) whole rounds are taken a lane each first: the FP64
 * pipe bounds those, and its instructions cost the same for one lane as for
 * 32.  Four levels within 1e-7 of one another at 160^3 f64, 1280 x 720: 2.10 ms
 * per frame of k_finish and k_exact with four lanes for each and no kLoExact,
 * 1.07 like this.
 * (The tiny list a lane each: 20 M triangles of a 128^3 field of whole numbers
 * 8.1 ms, four lanes 4.0; a triangle's pixels differ too much in number.)
 */
constexpr int kExactPerSm = 16; /* one-warp blocks resident per SM: at most 128 registers */
template <bool CHECK>
__global__ void __launch_bounds__(32, CHECK ? 1 : kExactPerSm)
k_exact(const __grid_constant__ Geo G, const __grid_constant__ SceneDev scene, const __grid_constant__ RasterDev R,
        const __grid_constant__ FrameObjs O, unsigned long long order_base, unsigned* __restrict__ checks) {
  pdl_enter();
  const unsigned long long nh = *R.hard_count, nt = min(*R.tiny_count, R.tiny_cap);
  const unsigned lane = threadIdx.x, m = lane & 3u, g0 = lane & ~3u;
  const unsigned lanes = 32 * gridDim.x;
  const unsigned long long fh = nh / lanes * lanes; /* taken in whole rounds */
  for (unsigned long long q = 32 * blockIdx.x + lane; q < fh; q += lanes) {
    const uint2 c = R.hard[q];
    finish_exact<CHECK>(G, scene, c.x, c.y, R, order_base, O, checks);
  }
  __syncwarp();
  const unsigned long long wh = (nh - fh + 7) / 8, wt = (nt + 7) / 8; /* warps' worth of the rest and of the tiny list */
  for (unsigned long long w = blockIdx.x; w < wh + wt; w += gridDim.x) {
    if (w >= wh) {
      const unsigned long long q = (w - wh) * 8 + lane / 4;
      tiny_triangle<CHECK>(G, scene, q < nt ? R.tiny[q] : 0u, q < nt, R, order_base, O, checks);
      __syncwarp();
      continue;
    }
    const unsigned long long q = fh + w * 8 + lane / 4;
    const uint2 c = q < nh ? R.hard[q] : make_uint2(0u, 0u);
    const unsigned pj = c.y / (unsigned)scene.width, pi = c.y - pj * (unsigned)scene.width;
    ExactTri x;
    const bool ok = quad_triangle(G, scene, c.x, q < nh, x);
    /* lane m: weight m and its depth term (exact_weights_in, exact_depth) */
    double wk = 0., term = 0.;
    bool in = false;
    if (ok) {
      wk = quad_weight(x, m, R.xs[pi], R.ys[pj]);
      in = !(wk < -1.e-8);
      term = ddiv(wk, m == 0 ? x.v0.z : (m == 1 ? x.v1.z : x.v2.z));
    }
    const unsigned all = __ballot_sync(0xFFFFFFFFu, in);
    const double w0 = shfl_d(wk, g0), w1 = shfl_d(wk, g0 + 1), w2 = shfl_d(wk, g0 + 2);
    const double t0 = shfl_d(term, g0), t1 = shfl_d(term, g0 + 1), t2 = shfl_d(term, g0 + 2);
    if (m == 0 && ok && ((all >> g0) & 7u) == 7u) {
      bool box = true;
      if (CHECK) {
        exact_box(scene, x);
        if (pi < x.imin || pi > x.imax || pj < x.jmin || pj > x.jmax) {
          atomicAdd(checks + 2, 1u);
          box = false;
        }
      }
      Hit h;
      h.key = depth_key(drcp(dadd(dadd(t0, t1), t2)));
      hit_weights(w0, w1, w2, h);
      const unsigned long long order = order_of(G, order_base, c.x);
      if (box && slot_max_near(O, scene, G.lut, R.xs, R.ys, R.canvas + c.y, pi, pj, h.key, (order << 24) | kLoExact, R.zerr))
        keep_weights(R, c.y, order, h);
    }
    __syncwarp();
  }
}

/* shading (render.c:137-159, normal.c:6-165), once per contour object     */
/* ------------------------------------------------------------------ */
/*
 * After all slabs of an object, every pixel the object won is shaded from the
 * field itself: the winner's drawing order gives its cell and rank (order =
 * base + 12 cell + rank), cell codes are recomputed from the corner values,
 * and each vertex normal is the normalised sum of the area-weighted face
 * normals of the triangles that share the vertex's cube edge, over the
 * neighbour cells in the reference's order.  Four lanes take one pixel: lane
 * m < 3 builds the normal of vertex m, lane 0 then blends them.  The FP32
 * pass settles a pixel when each channel's truncation is certain; the
 * others go to the FP64 pass, which repeats the reference's arithmetic in
 * its order.
 */
struct WinCell {
  long long i, j, k;
  unsigned r;
};

/* the object's triangle that owns a pixel, from the slot's order */
__device__ __forceinline__ bool winner_cell(const FieldDev& F, unsigned long long lo, unsigned long long obase,
                                            WinCell& w) {
  const unsigned long long order = lo >> 24;
  const unsigned long long ncx = (unsigned long long)(F.nx - 1), ncy = (unsigned long long)(F.ny - 1);
  const unsigned long long ncz = (unsigned long long)(F.nz - 1);
  if (order < obase || order - obase >= 12ULL * ncx * ncy * ncz) return false;
  /* rel / 12 by a multiply-high (exact for every 64-bit rel), the rest by
     the 32-bit divisions while the cells fit (no 64-bit division) */
  const unsigned long long rel = order - obase, c = __umul64hi(rel, 0xAAAAAAAAAAAAAAABULL) >> 3;
  w.r = (unsigned)(rel - 12ULL * c);
  if (c < (1ULL << 32)) {
    const unsigned row = fast_div((unsigned)c, F.div_cx);
    w.i = (long long)((unsigned)c - row * (unsigned)ncx);
    const unsigned kk = fast_div(row, F.div_cy);
    w.k = kk;
    w.j = (long long)(row - kk * (unsigned)ncy);
  } else {
    const unsigned long long row = c / ncx;
    w.i = (long long)(c - row * ncx);
    w.k = (long long)(row / ncy);
    w.j = (long long)(row - (unsigned long long)w.k * ncy);
  }
  return true;
}

__device__ __noinline__ unsigned long long slot_exact_key(const FrameObjs& O, const SceneDev& s,
                                                          const unsigned long long* lut, const double* xs,
                                                          const double* ys, unsigned long long order, long long i,
                                                          long long j, unsigned long long key) {
  for (int q = 0; q < O.n; q++) {
    if (order - O.first[q] >= O.span[q]) continue;
    const FieldDev& F = O.F[q];
    WinCell w;
    if (!winner_cell(F, order << 24, O.first[q], w)) return key;
    double vals[8];
    const unsigned code = cell_code_any(F, w.i, w.j, w.k, vals);
    d3 v[3];
    cell_vertices(F, w.i, w.j, w.k, __ldg(lut + code * 12 + w.r), v);
    ExactTri x;
    double w0, w1, w2;
    if (!exact_tri_core(s, v, x) || !exact_weights_in(x, i, j, xs, ys, w0, w1, w2)) return key;
    return depth_key(exact_depth(x, w0, w1, w2));
  }
  return key;
}

/*
 * The pixels whose owner is one of the object's triangles, a block per 16 x 16
 * pixels and a warp per 8 x 4 of them: k_shade_f takes 32 of the list at a
 * time and computes each distinct triangle around their vertices once, and
 * pixels of a compact patch share more of them than pixels of a row.
 */
__global__ void __launch_bounds__(256)
k_winners(const Slot* __restrict__ canvas, unsigned width, unsigned height, unsigned long long obase,
          unsigned long long span, unsigned* __restrict__ win, unsigned long long* __restrict__ win_count) {
  pdl_enter();
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x / 32;
  const unsigned dx = 8 * (warp & 1u) + (lane & 7u), dy = 4 * (warp >> 1) + (lane >> 3);
  const unsigned across = (width + 15) / 16, tiles = across * ((height + 15) / 16);
  for (unsigned t = blockIdx.x; t < tiles; t += gridDim.x) {
    const unsigned ty = t / across, tx = t - ty * across, i = 16 * tx + dx, j = 16 * ty + dy;
    const unsigned p = j * width + i;
    bool won = false;
    if (i < width && j < height) {
      const unsigned long long order = canvas[p].lo >> 24;
      won = order >= obase && order - obase < span;
    }
    const unsigned long long w = block_reserve<256>(win_count, won);
    if (won) win[w] = p;
  }
}

/*
 * Area-weighted face normal in FP32: the reference's area * unit normal
 * equals the cross product of two edges up to a few FP64 ulps; with vertices
 * relative to the cell's corner 0 the edge vectors keep their relative
 * accuracy.  eC: the largest bound of the three components, infinite when
 * none can be given.
 */
__device__ __forceinline__ void tri_wn_f(bool ok, const float rv[3][3], const float er[3][3], float C[3],
                                         float& eC) {
  /* edges from vertex 0 and their cross product (triangulate.c:75-93) */
  float x1[3], x2[3], e1[3], e2[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    x1[d] = rv[1][d] - rv[0][d];
    x2[d] = rv[2][d] - rv[0][d];
    e1[d] = er[1][d] + er[0][d] + kU32 * fabsf(x1[d]);
    e2[d] = er[2][d] + er[0][d] + kU32 * fabsf(x2[d]);
  }
  eC = 0.f;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const int d1 = (d + 1) % 3, d2 = (d + 2) % 3;
    const float p1 = x1[d1] * x2[d2], p2 = x1[d2] * x2[d1];
    C[d] = p1 - p2;
    const float ec = prod_err(x1[d1], e1[d1], x2[d2], e2[d2]) + prod_err(x1[d2], e1[d2], x2[d1], e2[d1]) +
                     kU32 * fabsf(C[d]);
    eC = fmaxf(eC, 1.1f * ec + 1e-15f * (fabsf(p1) + fabsf(p2)));
  }
  /* a zero cross product (area exactly 0, also by FP64 underflow) makes the
     reference's weighted normal 0 * (0 * inf) = NaN, which propagates to the
     pixel: unless some component is certainly away from 0, the triangle is
     left to the FP64 pass (a small but nonzero one only adds its small
     absolute bound) */
  const float cmax = fmaxf(fabsf(C[0]), fmaxf(fabsf(C[1]), fabsf(C[2])));
  if (!ok || !isfinite(cmax) || !isfinite(eC) || !(cmax - eC > 1e-30f)) eC = INFINITY;
}

/* 1 / sqrt(x) by the hardware approximation (PTX rsqrt.approx.f32: relative
   error below 2^-22.9 = 4.3u; no FP64 pipe, unlike the correctly rounded
   square root and division of a build without fused multiply-adds) */
__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

/*
 * A / |A| in FP32 as A * rsqrt_approx(A . A): the sum of squares is within
 * 3u of its value, the approximation within 4.3u, the products within u,
 * so U is within 6.9u of the exact unit vector; len = (A . A) * r stands for
 * |A| within 5u.  For |A - B| <= e, all norms Euclidean,
 *   | A / |A| - B / |B| | <= 2 e / (|A| + |B|) <= 2 e / (2 |A| - e)
 * (Dunkl and Williams, 1964); the result bounds |U - the reference's unit
 * vector|, infinite when |A| is too small.
 */
__device__ __forceinline__ float unit_vec(const float A[3], float e, float U[3]) {
  const float ss = A[0] * A[0] + A[1] * A[1] + A[2] * A[2];
  const float r = rsqrt_approx(ss);
  const float len = ss * r * (1.f - 6.f * kU32);
#pragma unroll
  for (int d = 0; d < 3; d++) U[d] = A[d] * r;
  if (!(len > 4.f * e) || !(len > 1e-30f) || !isfinite(r)) return INFINITY;
  return 1.01f * 2.f * e / (2.f * len - e) + 8.f * kU32;
}

/* code of cell (i, j, k) whose corner 0 is node `base` */
template <typename T>
__device__ __forceinline__ unsigned cell_code_at(const FieldDev& F, long long base);

/* the same, read from the classification's codes when they are kept */
template <typename T>
__device__ __forceinline__ unsigned cell_code_ijk(const FieldDev& F, long long i, long long j, long long k) {
  if (F.codes) return __ldg(F.codes + (k * (F.ny - 1) + j) * (F.nx - 1) + i);
  return cell_code_at<T>(F, (k * F.ny + j) * F.nx + i);
}

template <typename T>
__device__ __forceinline__ unsigned cell_code_at(const FieldDev& F, long long base) {
  const T* f = static_cast<const T*>(F.data);
  unsigned code = 0;
#pragma unroll
  for (int c = 0; c < 8; c++)
    code |= (unsigned)node_above<T>(F, f, base + (c & 1) + ((c >> 1) & 1) * F.nx + (c >> 2) * F.nx * F.ny) << c;
  return code;
}


/* the pixel's colour from the three FP32 vertex normals: false when a
   channel's truncation is not certain */
__device__ __forceinline__ bool blend_f(const SceneDev& scene, const RasterDev& R, long long p, unsigned long long lo,
                                        const float N[3][3], const float en[3], unsigned rgb_in, unsigned& rgb_out) {
  const unsigned long long tag = ((lo >> 24) << 24) | R.epoch;
  const ulonglong2 kw = R.winfo[p];
  if ((kw.y ^ tag) & ~0xFFFF00ULL) return false;
  /* the third weight from the first two: the reference's sum to 1 within 1e-8
     (NaN weights otherwise: nothing is certain).  With errors d0, d1 (bound
     ew) of the two and -(d0 + d1) of the third, the sum of w N is off by
     d0 (N0 - N2) + d1 (N1 - N2) besides the normals' own errors.  Every bound
     is of a vector's Euclidean length, as unit_vec gives the normals':
     bounds per component, with a sqrt(3) at each step, a unit_vec twice as
     wide and the light's 1-norm left 4.1 % of the pixels of a 128^3 double
     field to k_shade_amb, 8.6 % at 192^3 float and 26 % at 1536^3 float;
     these leave 0.6, 1.7 and 4.3 % */
  const float ew = bf16_value((unsigned)(kw.y >> 8) & 0xFFFFu);
  const float w0 = __uint_as_float((unsigned)kw.x), w1 = __uint_as_float((unsigned)(kw.x >> 32));
  const float ww[3] = {w0, w1, 1.f - w0 - w1};
  float M[3] = {0.f, 0.f, 0.f}, eM = 0.f, wsum = 0.f;
  float dn = 0.f; /* |N0 - N2| + |N1 - N2| <= sqrt(2) sqrt(3) dn */
#pragma unroll
  for (int d = 0; d < 3; d++) {
    M[d] = ww[0] * N[0][d] + ww[1] * N[1][d] + ww[2] * N[2][d];
    dn = fmaxf(dn, fabsf(N[0][d] - N[2][d]) + fabsf(N[1][d] - N[2][d]));
  }
#pragma unroll
  for (int m = 0; m < 3; m++) {
    eM += fabsf(ww[m]) * en[m];
    wsum += fabsf(ww[m]);
  }
  eM = 1.01f * eM + 1.02f * ew * (2.45f * dn + en[0] + en[1] + 2.f * en[2]) + 3e-7f;
  eM += 4.f * kU32 * wsum * 1.01f;
  float U[3];
  const float eN = unit_vec(M, eM, U);
  if (!isfinite(eN)) return false;
  const float* L = scene.f_light;
  const float dotv = U[0] * L[0] + U[1] * L[1] + U[2] * L[2];
  /* the unit vector's bound, the light's rounding to float, and the dot
     product's rounding (relative to the sum of |n_i L_i| <= |L| (1 + eN)) */
  const float ed = (eN + 5.f * kU32 * (1.f + eN)) * scene.f_light_len + 1e-30f;
  const float alo = fmaxf(0.f, fabsf(dotv) - ed), ahi = fabsf(dotv) + ed;
  /* factor = max(0.15, |d|): certainly clamped, certainly not, or undecided */
  const bool clamped = ahi < 0.149999f, free = alo > 0.150001f;
  if (clamped) {
    rgb_out = R.clamp_rgb;
    return true;
  }
  if (!free) return false;
  unsigned out = 0;
#pragma unroll
  for (int ch = 0; ch < 3; ch++) {
    const float cc = (float)((rgb_in >> (16 - 8 * ch)) & 255u);
    const float xl = alo * cc * (1.f - 4.f * kU32), xh = ahi * cc * (1.f + 4.f * kU32);
    const float fl = floorf(xl);
    if (floorf(xh) != fl || !(xl >= 0.f)) return false;
    out |= ((unsigned)(int)fl & 255u) << (16 - 8 * ch);
  }
  rgb_out = out;
  return true;
}

constexpr unsigned kFull = 0xFFFFFFFFu;

/* appends each flagged lane's pixel to a list, one atomic per warp */
__device__ __forceinline__ void warp_append(bool flag, unsigned p, unsigned* list, unsigned long long* count) {
  const unsigned lane = threadIdx.x & 31u;
  const unsigned bal = __ballot_sync(kFull, flag);
  unsigned long long a0 = 0;
  if (lane == 0 && bal) a0 = atomicAdd(count, (unsigned long long)__popc(bal));
  a0 = __shfl_sync(kFull, a0, 0);
  if (flag) list[a0 + __popc(bal & ((1u << lane) - 1u))] = p;
}

/*
 * FP32 pass over the won pixels, 32 pixels per block and iteration, four
 * threads per pixel (blocks of 128 threads: 0.47 -> 0.46 ms per bench frame
 * against 64 pixels and 256 threads; the block barriers wait for fewer warps).  Neighbouring pixels share most of their vertices'
 * neighbourhoods, so each block first gathers the triangles around its
 * pixels' vertices into a shared hash of (cell, rank) keys, computes each
 * distinct triangle's FP32 weighted normal once, then every (pixel, vertex)
 * thread sums its triangles' normals (the bound covers any summation order)
 * and lane 0 of each pixel blends the three.  A pixel whose neighbourhood
 * does not fit goes to the FP64 pass.  Self-check: every pixel is listed for
 * the FP64 pass, and the FP32 colour, where certain, is kept for it to compare.
 */
constexpr int kShadeHash = 512; /* distinct triangles per block and iteration */
constexpr int kShadeList = 24;    /* triangles around one cube edge: at most 12 (six tetrahedra, two each) */
constexpr unsigned long long kEmptyKey = ~0ULL;

/* (cell, rank) as a hash key: i, j, k below 2^20 each, rank below 12 (never all ones) */
__device__ __forceinline__ unsigned long long tri_key(long long i, long long j, long long k, unsigned r) {
  return ((unsigned long long)k << 44) | ((unsigned long long)j << 24) | ((unsigned long long)i << 4) | r;
}

/* slot of `key` in the block's table (inserted when absent, fresh = true), -1 when full */
template <int kSize>
__device__ __forceinline__ int hash_slot(unsigned long long* keys, unsigned long long key, bool& fresh) {
  static_assert((kSize & (kSize - 1)) == 0 && kSize <= 1024, "a power of two within the hash");
  unsigned h = (unsigned)((key * 0x9E3779B97F4A7C15ULL) >> 54) & (kSize - 1);
  for (int probe = 0; probe < kSize; probe++) {
    const unsigned long long prev = atomicCAS(keys + h, kEmptyKey, key);
    if (prev == kEmptyKey || prev == key) {
      fresh = prev == kEmptyKey;
      return (int)h;
    }
    h = (h + 1) & (kSize - 1);
  }
  fresh = false;
  return -1;
}

template <typename T, bool CHECK>
__global__ void __launch_bounds__(128)
k_shade_f(FieldDev F, SceneDev scene, RasterDev R, const unsigned long long* __restrict__ lut,
          unsigned long long obase, unsigned rgb_in) {
  pdl_enter();
  __shared__ unsigned long long keys[kShadeHash];
  __shared__ float4 wnf[kShadeHash];
  __shared__ unsigned short lists[kShadeList][128];
  __shared__ unsigned short todo[kShadeHash];
  __shared__ unsigned ntodo;
  for (int q = threadIdx.x; q < kShadeHash; q += blockDim.x) keys[q] = kEmptyKey;
  if (threadIdx.x == 0) ntodo = 0;
  __syncthreads();
  const unsigned long long n = *R.win_count;
  const unsigned tid = threadIdx.x, lane = tid & 31u, m = tid & 3u, g0 = lane & ~3u;
  const ThrF th = thr_f(F.threshold);
  for (unsigned long long base = blockIdx.x * 32ULL; base < n; base += gridDim.x * 32ULL) {
    const unsigned long long q = base + tid / 4;
    /* gather: the (cell, rank) of every triangle around this thread's vertex */
    unsigned p = 0;
    unsigned long long lo = 0;
    WinCell wc;
    bool ok = false, full = false;
    int cnt = 0;
    if (q < n) {
      p = R.win[q];
      lo = R.canvas[p].lo;
      ok = winner_cell(F, lo, obase, wc);
    }
    if (ok && m < 3) {
      const unsigned code = cell_code_ijk<T>(F, wc.i, wc.j, wc.k);
      const int ed = (int)((__ldg(lut + code * 12 + wc.r) >> (18 + 5 * m)) & 31);
      const int nn = c_nb_count[ed];
      for (int s = 0; s < nn; s++) {
        const long long ni = wc.i + c_nb[ed][s][2], nj = wc.j + c_nb[ed][s][1], nk = wc.k + c_nb[ed][s][0];
        const unsigned le = (unsigned)c_nb[ed][s][3];
        const unsigned ncode = cell_code_ijk<T>(F, ni, nj, nk);
        for (unsigned mask = __ldg(g_edge_tris + ncode * 19 + le); mask; mask &= mask - 1) {
          const int r = __ffs(mask) - 1;
          bool fresh;
          const int slot = hash_slot<kShadeHash>(keys, tri_key(ni, nj, nk, (unsigned)r), fresh);
          if (slot < 0 || cnt >= kShadeList) {
            full = true;
            continue;
          }
          if (fresh) todo[atomicAdd(&ntodo, 1u)] = (unsigned short)slot;
          lists[cnt++][tid] = (unsigned short)slot;
        }
      }
    }
    __syncthreads();
    /* each distinct triangle's FP32 weighted normal, once */
    const unsigned nd = ntodo;
    for (unsigned w = tid; w < nd; w += blockDim.x) {
      const int slot = todo[w];
      const unsigned long long key = keys[slot];
      const long long i = (long long)((key >> 4) & 0xFFFFFu), j = (long long)((key >> 24) & 0xFFFFFu);
      const long long k = (long long)(key >> 44);
      const long long nb = (k * F.ny + j) * F.nx + i;
      const unsigned code = cell_code_ijk<T>(F, i, j, k);
      const unsigned long long e = __ldg(lut + code * 12 + (key & 15u));
      const float sp[3] = {__ldg(F.dgx + i), __ldg(F.dgy + j), __ldg(F.dgz + k)};
      const T* fd = static_cast<const T*>(F.data);
      float rv[3][3], er[3][3];
      bool tok = true;
#pragma unroll
      for (int v = 0; v < 3; v++) {
        const unsigned a = (unsigned)((e >> (6 * v)) & 7), b = (unsigned)((e >> (6 * v + 3)) & 7);
        const typename ShadeVal<T>::type va =
            ShadeVal<T>::load(fd, nb + (a & 1u) + ((a >> 1) & 1u) * F.nx + (long long)(a >> 2) * F.nx * F.ny);
        const typename ShadeVal<T>::type vb =
            ShadeVal<T>::load(fd, nb + (b & 1u) + ((b >> 1) & 1u) * F.nx + (long long)(b >> 2) * F.nx * F.ny);
        float f = 0.f, e_f = 0.f;
        if (interp_shade(F, th, va, vb, f, e_f) < 0) tok = false;
        rel_pos(F, sp, a, b, f, e_f, rv[v], er[v]);
      }
      float C[3], eC;
      tri_wn_f(tok, rv, er, C, eC);
      wnf[slot] = make_float4(C[0], C[1], C[2], eC);
    }
    __syncthreads();
    /* vertex normal: the normalised sum over the triangles around the edge (normal.c:78-158) */
    float N[3] = {0.f, 0.f, 0.f}, en = INFINITY;
    if (ok && m < 3 && !full) {
      float S[3] = {0.f, 0.f, 0.f}, eS = 0.f, asum = 0.f;
      for (int t = 0; t < cnt; t++) {
        const float4 c = wnf[lists[t][tid]];
        S[0] += c.x;
        S[1] += c.y;
        S[2] += c.z;
        eS += c.w;
        asum += fabsf(c.x) + fabsf(c.y) + fabsf(c.z);
      }
      eS += (float)(cnt + 1) * kU32 * asum + 1e-15f * asum; /* FP32 and the reference's FP64 summation */
      en = unit_vec(S, 1.7321f * eS, N); /* eS bounds each component */
    }
    float Nv[3][3], env[3];
#pragma unroll
    for (int mm = 0; mm < 3; mm++) {
#pragma unroll
      for (int d = 0; d < 3; d++) Nv[mm][d] = __shfl_sync(kFull, N[d], g0 + mm);
      env[mm] = __shfl_sync(kFull, en, g0 + mm);
    }
    bool listed = false;
    if (ok && m == 0) {
      unsigned rgb = 0;
      const bool sure = isfinite(env[0]) && isfinite(env[1]) && isfinite(env[2]) &&
                        blend_f(scene, R, p, lo, Nv, env, rgb_in, rgb);
      if (CHECK) {
        R.shade_check[p] = sure ? (1u << 24) | rgb : 0u;
        listed = true;
      } else if (sure) {
        R.canvas[p].lo = (lo & ~0xFFFFFFULL) | rgb;
      } else {
        listed = true;
      }
    }
    warp_append(listed, p, R.amb, R.amb_count); /* at most the won pixels: fits */
    /* empty the table for the next pixels */
    for (unsigned w = tid; w < nd; w += blockDim.x) keys[todo[w]] = kEmptyKey;
    __syncthreads();
    if (tid == 0) ntodo = 0;
    __syncthreads();
  }
}

/*
 * FP64 pass over the pixels the FP32 pass could not settle (one to four in a
 * hundred), 16
 * per block and iteration: the triangles around the pixels' vertices are
 * listed in the reference's order, one thread computes each distinct one's
 * weighted normal, then two warps sum and normalise them in that order while
 * the other two compute the winning fragments' weights, and 16 threads blend
 * and colour.  The FP64 pipe bounds it (an FP64 warp instruction takes 16
 * cycles of an SM's), so a triangle is computed once per block, through a
 * hash: the three vertices of a pixel share 13 of their 18 triangles, and
 * unsettled pixels lie next to one another.
 */
constexpr int kAmbPixels = 16, kAmbPer = 16; /* triangles around one cube edge: at most 12 (six tetrahedra, two each) */
template <typename T, bool CHECK>
__global__ void __launch_bounds__(128)
k_shade_amb(const __grid_constant__ FieldDev F, const __grid_constant__ SceneDev scene,
            const __grid_constant__ RasterDev R, const unsigned long long* __restrict__ lut, unsigned long long obase,
            unsigned rgb_in, unsigned long long* __restrict__ ent_count, unsigned* __restrict__ checks) {
  pdl_enter();
  constexpr int kSlots = 4 * kAmbPixels * kAmbPer; /* more than the triangles of 48 vertices: never full */
  __shared__ unsigned long long s_key[kSlots];
  __shared__ double s_wn[3][kSlots];
  __shared__ unsigned short s_list[kAmbPer][4 * kAmbPixels]; /* each (pixel, vertex)'s triangles, in order */
  __shared__ unsigned short s_todo[kSlots];                  /* the slots in use */
  __shared__ unsigned s_ntodo, s_total;
  __shared__ double s_nrm[3][4 * kAmbPixels], s_w[3][kAmbPixels];
  __shared__ unsigned char s_good[kAmbPixels];
  const unsigned long long n = *R.amb_count;
  const unsigned tid = threadIdx.x, lane = tid & 31u, m = tid & 3u, g0 = lane & ~3u;
  const unsigned px = (tid & 63u) / 4;
  const double colour[3] = {(double)((rgb_in >> 16) & 255), (double)((rgb_in >> 8) & 255), (double)(rgb_in & 255)};
  /* few pixels: fewer per block, so that the chain of a block's FP64 steps is
     short and every SM has some (128^3 double, 1010 pixels: 31 -> 23 us; 192^3
     float, 1724 per object: 32 -> 28) */
  const unsigned spread = max(1u, gridDim.x / 4);
  const unsigned per = min((unsigned)kAmbPixels, max(4u, ((unsigned)n + spread - 1) / spread));
  if (blockIdx.x * (unsigned long long)per >= n) return;
  for (int q = tid; q < kSlots; q += blockDim.x) s_key[q] = kEmptyKey;
  if (tid == 0) s_ntodo = s_total = 0;
  __syncthreads();
  for (unsigned long long base = blockIdx.x * (unsigned long long)per; base < n;
       base += gridDim.x * (unsigned long long)per) {
    const unsigned long long q = px < per ? base + px : n;
    unsigned p = 0;
    unsigned long long e = 0;
    WinCell wc = {0, 0, 0, 0};
    bool ok = false;
    if (q < n) {
      p = R.amb[q];
      ok = winner_cell(F, R.canvas[p].lo, obase, wc);
      if (ok) e = __ldg(lut + cell_code_ijk<T>(F, wc.i, wc.j, wc.k) * 12 + wc.r);
    }
    unsigned cnt = 0;
    if (tid < 64 && ok && m < 3) {
      const int ed = (int)((e >> (18 + 5 * m)) & 31);
      const int nn = c_nb_count[ed];
      for (int s = 0; s < nn; s++) {
        const long long ni = wc.i + c_nb[ed][s][2], nj = wc.j + c_nb[ed][s][1], nk = wc.k + c_nb[ed][s][0];
        const unsigned ncode = cell_code_ijk<T>(F, ni, nj, nk);
        for (unsigned mask = __ldg(g_edge_tris + ncode * 19 + (unsigned)c_nb[ed][s][3]); mask && cnt < kAmbPer;
             mask &= mask - 1) {
          bool fresh;
          const int slot = hash_slot<kSlots>(s_key, tri_key(ni, nj, nk, (unsigned)(__ffs(mask) - 1)), fresh);
          if (fresh) s_todo[atomicAdd(&s_ntodo, 1u)] = (unsigned short)slot;
          s_list[cnt++][tid] = (unsigned short)slot;
        }
      }
      atomicAdd(&s_total, cnt);
    }
    __syncthreads();
    const unsigned todo = s_ntodo;
    if (tid == 0 && s_total) atomicAdd(ent_count, (unsigned long long)s_total);
    for (unsigned w = tid; w < todo; w += 128) {
      const unsigned slot = s_todo[w];
      const unsigned long long key = s_key[slot];
      const long long i = (long long)((key >> 4) & 0xFFFFFu), j = (long long)((key >> 24) & 0xFFFFFu);
      const long long k = (long long)(key >> 44);
      d3 v[3], fn, wn;
      double area;
      cell_vertices(F, i, j, k, __ldg(lut + cell_code_ijk<T>(F, i, j, k) * 12 + (key & 15u)), v);
      face_normal(v, fn, area, wn);
      s_wn[0][slot] = wn.x;
      s_wn[1][slot] = wn.y;
      s_wn[2][slot] = wn.z;
      s_key[slot] = kEmptyKey; /* for the next pixels */
    }
    __syncthreads();
    if (tid < 64) {
      if (ok && m < 3) { /* normal.c:78-158: in order, then normalised */
        d3 sum = {0., 0., 0.};
        for (unsigned u = 0; u < cnt; u++) {
          const unsigned slot = s_list[u][tid];
          sum = v_add(sum, d3{s_wn[0][slot], s_wn[1][slot], s_wn[2][slot]});
        }
        const d3 nm = v_normalise(sum);
        s_nrm[0][tid] = nm.x;
        s_nrm[1][tid] = nm.y;
        s_nrm[2][tid] = nm.z;
      }
    } else {
      /* the fragment's weights as it was drawn (render.c:102-133) */
      ExactTri x;
      const bool drawn = quad_project(F, scene, wc.i, wc.j, wc.k, e, ok, x);
      bool in = false;
      if (drawn) {
        const unsigned pj = p / (unsigned)scene.width, pi = p - pj * (unsigned)scene.width;
        const double wk = quad_weight(x, m, R.xs[pi], R.ys[pj]);
        in = !(wk < -1.e-8);
        if (m < 3) s_w[m][px] = wk;
      }
      const unsigned all = __ballot_sync(kFull, in);
      if (m == 0) s_good[px] = ((all >> g0) & 7u) == 7u;
    }
    if (tid == 0) s_ntodo = s_total = 0;
    __syncthreads();
    if (tid < 64 && m == 0 && ok && s_good[px]) {
      d3 n3[3];
#pragma unroll
      for (int mm = 0; mm < 3; mm++) n3[mm] = {s_nrm[0][tid + mm], s_nrm[1][tid + mm], s_nrm[2][tid + mm]};
      const d3 nrm = v_normalise(
          v_add(v_mul(s_w[0][px], n3[0]), v_add(v_mul(s_w[1][px], n3[1]), v_mul(s_w[2][px], n3[2]))));
      const double factor = fmax(0.15, fabs(v_dot(nrm, scene.light)));
      unsigned rgb = 0;
#pragma unroll
      for (int ch = 0; ch < 3; ch++) rgb = (rgb << 8) | (unsigned)(unsigned char)(int)dmul(factor, colour[ch]);
      if (CHECK) {
        /* the FP32 colour, where it was certain, must be this one */
        const unsigned f = R.shade_check[p];
        if ((f >> 24) && (f & 0xFFFFFFu) != rgb) atomicAdd(checks + 5, 1u);
      }
      R.canvas[p].lo = (R.canvas[p].lo & ~0xFFFFFFULL) | rgb;
    }
    __syncthreads();
  }
}

/*
 * FP64 pass over every won pixel of a field without single-precision shading
 * (a converter), in three steps so
 * that the FP64 work runs on full warps: list every (pixel, vertex)'s
 * neighbour triangles in the reference's order, compute each listed
 * triangle's area-weighted face normal, then sum them in that order and
 * blend.  A list entry is (global cell) * 16 + rank.
 */
__device__ __forceinline__ int vertex_edge(const FieldDev& F, const unsigned long long* lut, const WinCell& wc, int m,
                                           double vals[8], unsigned long long& e) {
  const unsigned code = cell_code_any(F, wc.i, wc.j, wc.k, vals);
  e = lut[code * 12 + wc.r];
  return (int)((e >> (18 + 5 * m)) & 31);
}

/* visits the neighbour triangles around cube edge ed of cell (i, j, k) in the
   reference's order (normal.c:78-158): fn(entry) */
template <typename Fn>
__device__ __forceinline__ void for_edge_triangles(const FieldDev& F, const unsigned long long* lut, long long i,
                                                   long long j, long long k, int ed, Fn fn) {
  const long long ncx = F.nx - 1, ncy = F.ny - 1;
  const int nn = c_nb_count[ed];
  for (int q = 0; q < nn; q++) {
    const long long ni = i + c_nb[ed][q][2], nj = j + c_nb[ed][q][1], nk = k + c_nb[ed][q][0];
    const unsigned le = (unsigned)c_nb[ed][q][3];
    const unsigned long long cell = (unsigned long long)((nk * ncy + nj) * ncx + ni);
    double vals[8];
    const unsigned code = F.codes ? (unsigned)__ldg(F.codes + cell) : cell_code_any(F, ni, nj, nk, vals);
    /* ascending rank: the reference's order within the cell */
    for (unsigned mask = __ldg(g_edge_tris + code * 19 + le); mask; mask &= mask - 1)
      fn(cell * 16ULL + (unsigned long long)(__ffs(mask) - 1));
  }
}

/* step 1: one thread per (pixel, vertex); spans[q] = (first entry, count),
   count 0xFFFFFFFF when the entries did not fit */
__global__ void __launch_bounds__(256)
k_nb_list(FieldDev F, RasterDev R, const unsigned long long* __restrict__ lut_g, const unsigned* __restrict__ pixels,
          const unsigned long long* __restrict__ count, unsigned long long obase, unsigned long long* __restrict__ ent,
          unsigned long long ent_cap, unsigned long long* __restrict__ ent_count, uint2* __restrict__ spans) {
  pdl_trigger();
  /* the table through L1: a copy in each block's shared memory cost every
     block 24 KB of loads and a barrier */
  const unsigned long long* lut = lut_g;
  pdl_wait();
  const unsigned long long n = 3 * *count;
  const unsigned long long iters = (n + blockDim.x - 1) / blockDim.x;
  /* every lane of a warp runs the same iterations (warp-wide reservations) */
  for (unsigned long long it = blockIdx.x; it < iters; it += gridDim.x) {
    const unsigned long long q = it * blockDim.x + threadIdx.x;
    WinCell wc;
    bool ok = false;
    int ed = 0;
    unsigned cnt = 0;
    if (q < n) {
      const unsigned long long pq = q / 3;
      const int m = (int)(q - 3 * pq);
      ok = winner_cell(F, R.canvas[pixels[pq]].lo, obase, wc);
      if (ok) {
        double vals[8];
        unsigned long long e;
        ed = vertex_edge(F, lut, wc, m, vals, e);
        for_edge_triangles(F, lut, wc.i, wc.j, wc.k, ed, [&](unsigned long long) { cnt++; });
      }
    }
    /* warp-aggregated reservation */
    const unsigned lane = threadIdx.x & 31u;
    unsigned incl = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned y = __shfl_up_sync(kFull, incl, d);
      if ((int)lane >= d) incl += y;
    }
    unsigned long long w0 = 0;
    if (lane == 31 && incl) w0 = atomicAdd(ent_count, (unsigned long long)incl);
    w0 = __shfl_sync(kFull, w0, 31);
    const unsigned long long first = w0 + (incl - cnt);
    if (q < n) {
      const bool fits = first + cnt <= ent_cap;
      spans[q] = make_uint2((unsigned)first, ok && fits ? cnt : 0xFFFFFFFFu);
      if (ok) {
        /* the entries below ent_cap are written even when the span does not
           fit whole: k_nb_wn takes every entry below min(count, ent_cap),
           and one left unwritten would hold a stale (cell, rank) word */
        unsigned long long at = first;
        for_edge_triangles(F, lut, wc.i, wc.j, wc.k, ed, [&](unsigned long long x) {
          if (at < ent_cap) ent[at] = x;
          at++;
        });
      }
    }
  }
}

/*
 * Step 2: the listed triangles' exact area-weighted face normals
 * (triangulate.c:40-93, normal.c:39-40).  The FP64 pipe bounds it, and the
 * entries of neighbouring pixels name the same triangles, so a block takes
 * kNbEntries of them and computes each distinct one once, through a hash (2.07 M
 * entries of a 72 x 64 x 80 field: 346 -> 125 us).
 */
constexpr int kNbEntries = 512;
__global__ void __launch_bounds__(256)
k_nb_wn(FieldDev F, const unsigned long long* __restrict__ lut, const unsigned long long* __restrict__ ent,
        unsigned long long ent_cap, const unsigned long long* __restrict__ ent_count, double* __restrict__ wn_out) {
  pdl_enter();
  constexpr int kSlots = 2 * kNbEntries, kPer = kNbEntries / 256;
  __shared__ unsigned long long s_key[kSlots];
  __shared__ double s_wn[3][kSlots];
  __shared__ unsigned short s_todo[kNbEntries];
  __shared__ unsigned s_ntodo;
  const unsigned long long n = min(*ent_count, ent_cap);
  const unsigned long long ncx = (unsigned long long)(F.nx - 1), ncy = (unsigned long long)(F.ny - 1);
  const unsigned long long cells = ncx * ncy * (unsigned long long)(F.nz - 1);
  for (int w = threadIdx.x; w < kSlots; w += 256) s_key[w] = kEmptyKey;
  if (threadIdx.x == 0) s_ntodo = 0;
  __syncthreads();
  for (unsigned long long base = blockIdx.x * (unsigned long long)kNbEntries; base < n;
       base += gridDim.x * (unsigned long long)kNbEntries) {
    int slot[kPer];
#pragma unroll
    for (int u = 0; u < kPer; u++) {
      const unsigned long long q = base + 256 * u + threadIdx.x, x = q < n ? ent[q] : kEmptyKey;
      slot[u] = -1;
      if ((x >> 4) >= cells || (x & 15) >= 12) continue; /* not a cell of the field: never read past it */
      bool fresh;
      slot[u] = hash_slot<kSlots>(s_key, x, fresh);
      if (fresh) s_todo[atomicAdd(&s_ntodo, 1u)] = (unsigned short)slot[u];
    }
    __syncthreads();
    const unsigned todo = s_ntodo;
    for (unsigned w = threadIdx.x; w < todo; w += 256) {
      const unsigned at = s_todo[w];
      const unsigned long long x = s_key[at], cell = x >> 4, row = cell / ncx;
      const long long i = (long long)(cell - row * ncx), k = (long long)(row / ncy);
      const long long j = (long long)(row - (unsigned long long)k * ncy);
      double vals[8];
      const unsigned code = cell_code_any(F, i, j, k, vals);
      const unsigned long long e = __ldg(lut + code * 12 + (x & 15));
      d3 v[3], fn, wn;
      double area;
#pragma unroll
      for (int qv = 0; qv < 3; qv++) {
        const int a = (int)((e >> (6 * qv)) & 7), b = (int)((e >> (6 * qv + 3)) & 7);
        v[qv] = interpolate(F.threshold, corner_pos(F, i, j, k, a), vals[a], corner_pos(F, i, j, k, b), vals[b]);
      }
      face_normal(v, fn, area, wn);
      s_wn[0][at] = wn.x;
      s_wn[1][at] = wn.y;
      s_wn[2][at] = wn.z;
      s_key[at] = kEmptyKey; /* for the next entries */
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPer; u++) {
      const unsigned long long q = base + 256 * u + threadIdx.x;
      if (slot[u] >= 0) {
        wn_out[3 * q + 0] = s_wn[0][slot[u]];
        wn_out[3 * q + 1] = s_wn[1][slot[u]];
        wn_out[3 * q + 2] = s_wn[2][slot[u]];
      }
    }
    if (threadIdx.x == 0) s_ntodo = 0;
    __syncthreads();
  }
}

/*
 * Step 3, a pixel per lane.  What belongs to a triangle (the sums of its
 * vertices' normals in the reference's order, its projection) is computed once
 * for the warp's pixels that show it, by four lanes, a vertex each, eight
 * triangles at a time; then every lane weighs, blends and colours its pixel
 * (render.c:102-159).  The FP64 pipe bounds it, whose instructions cost the same
 * for one lane as for 32: with four lanes per pixel throughout, 112815 pixels of
 * a 72 x 64 x 80 field took 165 us; this 128 (80 registers and some spills:
 * at 114 the warps need a second wave, 155 us).
 */
__global__ void __launch_bounds__(128, 6)
k_shade(FieldDev F, SceneDev scene, RasterDev R, const unsigned long long* __restrict__ lut,
        const unsigned* __restrict__ pixels, const unsigned long long* __restrict__ count, unsigned long long obase,
        const uint2* __restrict__ spans, const double* __restrict__ wn_in, unsigned rgb_in) {
  pdl_enter();
  const unsigned long long n = *count;
  const unsigned lane = threadIdx.x & 31u, m = lane & 3u, g0 = lane & ~3u;
  const double cr = (double)((rgb_in >> 16) & 255), cg = (double)((rgb_in >> 8) & 255),
               cb = (double)(rgb_in & 255);
  const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long base = (unsigned long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n;
       base += step) {
    const unsigned long long q = base + lane;
    unsigned p = 0;
    WinCell wc = {0, 0, 0, 0};
    unsigned long long e = 0, lo = 0;
    bool won = false;
    if (q < n) {
      p = pixels[q];
      lo = R.canvas[p].lo;
      won = winner_cell(F, lo, obase, wc);
      if (won) {
        double vals[8];
        vertex_edge(F, lut, wc, 0, vals, e);
      }
    }
    /* the first lane of each triangle stands for its pixels */
    const unsigned first = __ffs(__match_any_sync(kFull, won ? lo >> 24 : ~0ULL)) - 1;
    const unsigned firsts = __ballot_sync(kFull, won && first == lane);
    const unsigned rank = __popc(firsts & ((1u << first) - 1u)), tris = __popc(firsts);
    d3 n3[3] = {{0., 0., 0.}, {0., 0., 0.}, {0., 0., 0.}};
    ExactTri x = {};
    bool ready = false;
    for (unsigned r = 0; r < tris; r += 8) {
      /* lane m of a four: vertex m's normal (its sum in the listed order) and projection */
      const bool has = r + lane / 4 < tris;
      const unsigned src = has ? __fns(firsts, 0, (int)(r + lane / 4 + 1)) : 0u;
      const long long i = __shfl_sync(kFull, wc.i, src), j = __shfl_sync(kFull, wc.j, src),
                      k = __shfl_sync(kFull, wc.k, src);
      const unsigned long long te = __shfl_sync(kFull, e, src), tq = base + src;
      d3 nm = {0., 0., 0.};
      bool good = false;
      if (has && m < 3) {
        const uint2 sp = spans[3 * tq + m];
        good = sp.y != 0xFFFFFFFFu;
        if (good) {
          d3 sum = {0., 0., 0.};
          for (unsigned t = 0; t < sp.y; t++) {
            const double* w = wn_in + 3 * ((unsigned long long)sp.x + t);
            sum = v_add(sum, d3{w[0], w[1], w[2]});
          }
          nm = v_normalise(sum);
        }
      }
      ExactTri tx = {};
      const bool drawn = quad_project(F, scene, i, j, k, te, has, tx);
      const unsigned oks = __ballot_sync(kFull, good && drawn);
      /* to the triangle's pixels */
      const unsigned from = 4 * (rank & 7u);
      const bool mine = won && rank - r < 8u;
#pragma unroll
      for (unsigned mm = 0; mm < 3; mm++) {
        const d3 y = {shfl_d(nm.x, from + mm), shfl_d(nm.y, from + mm), shfl_d(nm.z, from + mm)};
        if (mine) n3[mm] = y;
      }
      const d3 v0 = {shfl_d(tx.v0.x, from), shfl_d(tx.v0.y, from), 0.};
      const d3 v1 = {shfl_d(tx.v1.x, from), shfl_d(tx.v1.y, from), 0.};
      const d3 v2 = {shfl_d(tx.v2.x, from), shfl_d(tx.v2.y, from), 0.};
      const double inv = shfl_d(tx.area_inv, from);
      if (mine) {
        x.v0 = v0;
        x.v1 = v1;
        x.v2 = v2;
        x.area_inv = inv;
        ready = ((oks >> from) & 7u) == 7u;
      }
    }
    if (!ready) continue;
    /* the winning fragment's weights as it was drawn (render.c:102-133) */
    const unsigned pj = p / (unsigned)scene.width, pi = p - pj * (unsigned)scene.width;
    const double px = R.xs[pi], py = R.ys[pj];
    const double w0 = quad_weight(x, 0, px, py), w1 = quad_weight(x, 1, px, py), w2 = quad_weight(x, 2, px, py);
    if (w0 < -1.e-8 || w1 < -1.e-8 || w2 < -1.e-8) continue;
    const d3 nrm = v_normalise(v_add(v_mul(w0, n3[0]), v_add(v_mul(w1, n3[1]), v_mul(w2, n3[2]))));
    const double factor = fmax(0.15, fabs(v_dot(nrm, scene.light)));
    const unsigned r8 = (unsigned)(unsigned char)(int)dmul(factor, cr);
    const unsigned g8 = (unsigned)(unsigned char)(int)dmul(factor, cg);
    const unsigned b8 = (unsigned)(unsigned char)(int)dmul(factor, cb);
    const unsigned rgb = (r8 << 16) | (g8 << 8) | b8;
    R.canvas[p].lo = (lo & ~0xFFFFFFULL) | rgb;
  }
}

/* ------------------------------------------------------------------ */
/* lines (line.c:26-119), canvas init, resolve                          */
/* ------------------------------------------------------------------ */
/*
 * One segment per blockIdx.x (line.c:26-119), its pixels over the threads of
 * the blocks (x, *).  The host found the few pixels per column (or row) that
 * can lie near the line (line_pixels in runtime.cu); the reference tests the
 * whole box.  Its distance test is repeated as it is, the quotient only where
 * the products do not settle it.  One pixel per thread, because a pixel is a
 * chain of about 60 dependent FP64 operations: the unit cube's 48 segments at
 * 800 x 600 took 60.8 us with one block over each whole box and a division
 * per pixel, 8.3 us like this; at 160 x 120 10.2 us and 7.4 us.
 */
__global__ void __launch_bounds__(128)
k_lines(const LineSegDev* __restrict__ segs, int nseg, const __grid_constant__ SceneDev scene,
        const __grid_constant__ RasterDev R, const __grid_constant__ FrameObjs O, const unsigned long long* lut,
        unsigned long long order_base) {
  pdl_enter();
  const int sidx = blockIdx.x;
  if (sidx >= nseg) return;
  const LineSegDev& L = segs[sidx];
  const long long total = L.npix;
  const unsigned long long order = order_base + (unsigned long long)sidx;
  for (long long q = blockIdx.y * (long long)blockDim.x + threadIdx.x; q < total;
       q += (long long)gridDim.y * blockDim.x) {
    const long long n = L.across_n;
    const long long col = (unsigned long long)total >> 32 ? q / n : (long long)((unsigned)q / (unsigned)n);
    const long long v = L.v0 + col;
    long long u = q - col * n; /* the column's u-th pixel */
    if (L.narrow) u += (long long)floor(L.slope * (double)v + L.icept); /* from its first pixel near the line on */
    else u += L.u0;
    if (u < (long long)L.u0 || u > (long long)L.u1) continue;
    const long long i = L.by_x ? v : u, j = L.by_x ? u : v;
    const double di = (double)i, dj = (double)j;
    const double num = dadd(dadd(dmul(L.dy, di), dmul(-L.dx, dj)), L.c);
    const double sq = dmul(num, num);
    if (sq > L.sure_out) continue;
    if (!(sq < L.sure_in) && L.thr < ddiv(sq, L.dd)) continue;
    const double param = ddiv(dmul(-1., dadd(dmul(L.dx, dsub(L.p0x, di)), dmul(L.dy, dsub(L.p0y, dj)))), L.dd);
    const double dist0 = drcp(dadd(ddiv(param, L.p1z), ddiv(dsub(1., param), L.p0z)));
    const unsigned long long key = depth_key(dist0);
    slot_max_near(O, scene, lut, R.xs, R.ys, R.canvas + j * scene.width + i, i, j, key, (order << 24) | L.rgb, R.zerr);
  }
}

__global__ void k_canvas_init(Slot* canvas, unsigned* zlo, long long n, unsigned long long hi, unsigned long long lo) {
  pdl_enter();
  const unsigned floor_key = f_key(-__int_as_float(0x7f800000));
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    canvas[p].hi = hi;
    canvas[p].lo = lo;
    zlo[p] = floor_key;
  }
}

/* ppm body: rows flipped (output.c:113-123); optional canvas-order depth */
__global__ void k_resolve(const Slot* __restrict__ canvas, long long W, long long H, unsigned char* __restrict__ rgb,
                          double* __restrict__ depth) {
  pdl_enter();
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < W * H; p += (long long)gridDim.x * blockDim.x) {
    const long long r = p / W, i = p % W;
    const Slot s = canvas[(H - 1 - r) * W + i];
    rgb[3 * p + 0] = (unsigned char)(s.lo >> 16);
    rgb[3 * p + 1] = (unsigned char)(s.lo >> 8);
    rgb[3 * p + 2] = (unsigned char)(s.lo);
    if (depth) {
      const Slot sc = canvas[p];
      depth[p] = depth_from_key(sc.hi);
    }
  }
}

/* ------------------------------------------------------------------ */
/* launchers                                                           */
/* ------------------------------------------------------------------ */
/* SMs of the first device the library runs on (thread-safe one-time query) */
static int num_sms() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) {
      cudaGetLastError();
      v = 1;
    }
    return v;
  }();
  return n;
}

static std::atomic<int> g_cls_z{kClsZ}, g_emit_per_sm{8}, g_raster_per_sm{8};
static std::atomic<int> g_pdl{0};

void set_dependent_launch(int on) { g_pdl = on ? 1 : 0; }
int dependent_launch() { return g_pdl.load(); }

int set_launch_shape(const LaunchShape& s) {
  if (s.cls_z < 1 || s.cls_z > 1024 || s.emit_per_sm < 1 || s.emit_per_sm > 32 || s.raster_per_sm < 1 ||
      s.raster_per_sm > 32)
    return 1;
  g_cls_z = s.cls_z;
  g_emit_per_sm = s.emit_per_sm;
  g_raster_per_sm = s.raster_per_sm;
  return 0;
}

LaunchShape launch_shape() { return LaunchShape{g_cls_z.load(), g_emit_per_sm.load(), g_raster_per_sm.load()}; }

/* every kernel launch of the library: programmatic dependent launch (the
   kernels call pdl_wait() before they touch what earlier work produced) */
/* C3D_LAUNCH_CHECK=1 in the environment: every launch is followed by a
   synchronisation of its stream and an error check that names the kernel
   (debugging; changes timing) */
static bool launch_check() {
  static const bool on = [] {
    const char* e = getenv("C3D_LAUNCH_CHECK");
    return e && e[0] == '1';
  }();
  return on;
}

template <typename... KArgs, typename... Args>
static void launch_k(void (*kernel)(KArgs...), const char* name, dim3 grid, dim3 block, size_t smem,
                     cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = g_pdl.load() ? 1 : 0;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
  if (launch_check()) {
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess)
      fprintf(stderr, "[CONTOUR3D ERROR] %s (grid %u x %u x %u): %s\n", name, grid.x, grid.y, grid.z,
              cudaGetErrorString(e));
  }
}

static int grid_for(long long n, int threads, int per_sm) {
  const int g_num_sms = num_sms();
  long long b = (n + threads - 1) / threads;
  const long long cap = (long long)g_num_sms * per_sm;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

int upload_tables(const unsigned char code_count[256], const signed char nb[19][4][4],
                  const unsigned char nb_count[19], const unsigned short edge_tris[256 * 19]) {
  if (cudaMemcpyToSymbol(c_code_count, code_count, 256) != cudaSuccess) return 1;
  if (cudaMemcpyToSymbol(g_edge_tris, edge_tris, sizeof(unsigned short) * 256 * 19) != cudaSuccess) return 1;
  if (cudaMemcpyToSymbol(c_nb, nb, sizeof(signed char) * 19 * 16) != cudaSuccess) return 1;
  if (cudaMemcpyToSymbol(c_nb_count, nb_count, 19) != cudaSuccess) return 1;
  /* beyond the default 48 KB of shared memory: set once per device */
  if (cudaFuncSetAttribute(k_scan<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScanListBytes) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_scan<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(kScanListBytes + kScanStageBytes)) != cudaSuccess)
    return 1;
  return 0;
}

/* cuTensorMapEncodeTiled through the runtime's driver entry point (no libcuda
   link); looked up once, thread-safely (a function-local static) */
static PFN_cuTensorMapEncodeTiled_v12000 lookup_tensor_map_encoder() {
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
      q == cudaDriverEntryPointSuccess)
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  cudaGetLastError();
  return nullptr;
}

static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = lookup_tensor_map_encoder();
  return fn;
}

/* the field as a 3-D tensor map with one node plane of a classify tile per box,
   or false when TMA cannot address it (row or plane pitch not a multiple of 16
   bytes, base not 16-byte aligned, more than 2^31 nodes along an axis) */
static bool classify_tensor_map(const FieldDev& F, CUtensorMap* map) {
  const size_t es = F.is_f32 ? 4 : 8;
  if (((uintptr_t)F.data & 15) || (F.nx * es) % 16 || F.nx >= (1LL << 31) || F.ny >= (1LL << 31) ||
      F.nz >= (1LL << 31))
    return false;
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)F.nx, (cuuint64_t)F.ny, (cuuint64_t)F.nz};
  const cuuint64_t strides[2] = {(cuuint64_t)(F.nx * es), (cuuint64_t)(F.nx * F.ny * es)};
  const cuuint32_t box[3] = {(cuuint32_t)(F.is_f32 ? TmaBox<float>::kX : TmaBox<double>::kX), kClsY + 1, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(map, F.is_f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3,
                         const_cast<void*>(F.data), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

/* ThrSet's range form of a field's threshold.  thr_key is the key with -0
   taken as +0, so lo = thr_key + 1 and the keys above run up to key(+inf);
   thr_f_key is the unsigned float key of the least float above the
   threshold, turned back into the float's bits (a zero of either sign
   admits both zeros: lo = key(-0) = -1). */
void thr_range(const FieldDev& F, ThrSet& ts, int t) {
  const long long kInfKey = 0x7FF0000000000000LL;
  ts.lo[t] = (unsigned long long)F.thr_key + 1;
  ts.cnt[t] = F.thr_nan ? 0ULL : (unsigned long long)kInfKey - (unsigned long long)F.thr_key;
  const int kInfKeyF = 0x7F800000;
  const unsigned K = F.thr_f_key;
  const unsigned u = (K & 0x80000000u) ? (K & 0x7FFFFFFFu) : ~K; /* the float's bits */
  int flo;
  if ((u << 1) == 0) flo = -1;
  else flo = (u & 0x80000000u) ? (int)(u ^ 0x7FFFFFFFu) : (int)u;
  ts.flo[t] = (unsigned)flo;
  ts.fcnt[t] = F.thr_f_ok ? (unsigned)((long long)kInfKeyF - flo + 1) : 0u;
}

template <typename T>
static void launch_classify_tma(const CUtensorMap& map, const FieldDev& F, const SlabDev& S, const ThrSet& ts,
                                const CodeOut& out, unsigned* err, const dim3& grid, cudaStream_t st) {
  switch (ts.n) {
    case 1: launch_k(k_classify_tma<T, 1>, "k_classify_tma", grid, kClsX, 0, st, map, F, S, ts, out, err); break;
    case 2: launch_k(k_classify_tma<T, 2>, "k_classify_tma", grid, kClsX, 0, st, map, F, S, ts, out, err); break;
    case 3: launch_k(k_classify_tma<T, 3>, "k_classify_tma", grid, kClsX, 0, st, map, F, S, ts, out, err); break;
    default: launch_k(k_classify_tma<T, 4>, "k_classify_tma", grid, kClsX, 0, st, map, F, S, ts, out, err); break;
  }
}

int launch_classify(const FieldDev* Fs, int nf, const SlabDev& S0, unsigned char* const* codes, unsigned* err,
                    cudaStream_t st) {
  /* codes[q] receives the cell codes of threshold q; the scan turns them into counts */
  const FieldDev& F = Fs[0];
  SlabDev S = S0;
  /* bricks of the launch shape's depth, or shallower when the slab is thin:
     at least 16 bricks per SM, so that every SM has copies in flight (the
     deeper the brick, the fewer node planes are read twice) */
  const long long bxy = ((F.nx - 1 + kClsX - 1) / kClsX) * ((F.ny - 1 + kClsY - 1) / kClsY);
  const long long want_z = ((long long)num_sms() * 16 + bxy - 1) / bxy;
  S.cls_z = (int)std::max(std::min<long long>(launch_shape().cls_z, (S.nslices + want_z - 1) / want_z),
                          (long long)std::min(8, launch_shape().cls_z));
  const dim3 grid((unsigned)((F.nx - 1 + kClsX - 1) / kClsX), (unsigned)((F.ny - 1 + kClsY - 1) / kClsY),
                  (unsigned)((S.nslices + S.cls_z - 1) / S.cls_z));
  CUtensorMap map;
  if (classify_tensor_map(F, &map)) {
    /* one pass over the field for up to kMaxThr thresholds */
    for (int q0 = 0; q0 < nf; q0 += kMaxThr) {
      ThrSet ts;
      CodeOut out;
      ts.n = min(kMaxThr, nf - q0);
      for (int t = 0; t < ts.n; t++) {
        thr_range(Fs[q0 + t], ts, t);
        out.codes[t] = codes[q0 + t];
      }
      if (F.is_f32) launch_classify_tma<float>(map, F, S, ts, out, err, grid, st);
      else launch_classify_tma<double>(map, F, S, ts, out, err, grid, st);
    }
    return (nf + kMaxThr - 1) / kMaxThr;
  }
  /* rows TMA cannot address: plain loads, still one pass per kMaxThr objects */
  for (int q0 = 0; q0 < nf; q0 += kMaxThr) {
    ThrSet ts;
    CodeOut out;
    ts.n = min(kMaxThr, nf - q0);
    for (int t = 0; t < ts.n; t++) {
      thr_range(Fs[q0 + t], ts, t);
      out.codes[t] = codes[q0 + t];
    }
    for (int t = ts.n; t < kMaxThr; t++) out.codes[t] = nullptr;
    if (F.is_f32)
      launch_k(k_classify_multi<float>, "k_classify_multi", grid, kClsX, 0, st, F.data, F.nx, F.ny, S, ts, out);
    else
      launch_k(k_classify_multi<double>, "k_classify_multi", grid, kClsX, 0, st, F.data, F.nx, F.ny, S, ts, out);
  }
  return (nf + kMaxThr - 1) / kMaxThr;
}

void make_cls_item(const FieldDev* Fs, int nf, const SlabDev& S, unsigned char* const* codes, ClsItem* it) {
  const FieldDev& F = Fs[0];
  memset(it, 0, sizeof *it);
  it->data = F.data;
  it->is_f32 = F.is_f32;
  it->nx = F.nx;
  it->ny = F.ny;
  it->S = S;
  it->ts.n = min(nf, kMaxThr);
  for (int t = 0; t < it->ts.n; t++) {
    thr_range(Fs[t], it->ts, t);
    it->out.codes[t] = codes[t];
  }
  it->nbx = (unsigned)((F.nx - 1 + kClsX - 1) / kClsX);
  it->nby = (unsigned)((F.ny - 1 + kClsY - 1) / kClsY);
  it->nbz = (unsigned)((S.nslices + S.cls_z - 1) / S.cls_z);
}

void launch_classify_queue(const ClsItem* items, int nitems, unsigned long long nunits, unsigned long long* next,
                           cudaStream_t st) {
  if (nitems < 1 || nunits == 0) return;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_classify_queue, kClsX, 0) != cudaSuccess ||
      per_sm < 1)
    per_sm = 8;
  const unsigned long long cap = (unsigned long long)num_sms() * (unsigned long long)per_sm;
  const unsigned grid = (unsigned)(nunits < cap ? nunits : cap);
  launch_k(k_classify_queue, "k_classify_queue", grid, kClsX, 0, st, items, nitems, nunits, next);
}

long long scan_state_words(long long n) { return std::max((n + kScanTile - 1) / kScanTile, 1LL) + 1; }

size_t voff_bytes(long long n) {
  return ((size_t)(n + 1) * sizeof(unsigned) + 255) / 256 * 256 + sizeof(unsigned) * (size_t)scan_state_words(n);
}

VOffDev voff_layout(void* base, long long n) {
  const size_t word_bytes = ((size_t)(n + 1) * sizeof(unsigned) + 255) / 256 * 256;
  VOffDev o;
  o.word = static_cast<unsigned*>(base);
  o.seg = reinterpret_cast<unsigned*>(static_cast<char*>(base) + word_bytes);
  return o;
}

cudaError_t launch_scan(const FieldDev& F, const SlabDev& S, const unsigned char* codes, long long n,
                        unsigned long long* state, unsigned* offsets, const VOffDev& voff, unsigned long long* totals,
                        unsigned* tri_cell, unsigned long long tri_cap, bool want_offsets, unsigned* ovf,
                        unsigned* err, cudaStream_t st) {
  const long long nseg = scan_state_words(n) - 1;
  const cudaError_t e = cudaMemsetAsync(state, 0, sizeof(unsigned long long) * (size_t)(nseg + 1), st);
  if (e != cudaSuccess) return e;
  ScanCells box;
  box.div_cx = F.div_cx;
  box.div_cy = F.div_cy;
  box.ncx = (unsigned)(F.nx - 1);
  box.ncy = (unsigned)(F.ny - 1);
  box.kfirst = (unsigned)S.kfirst;
  box.krender0 = (unsigned)S.krender0;
  box.krender1 = (unsigned)std::max(S.krender0, S.krender1);
  if (want_offsets)
    launch_k(k_scan<true>, "k_scan", (unsigned)nseg, kScanThreads, kScanListBytes + kScanStageBytes, st, box, codes, n,
             nseg, state, offsets, voff, totals, tri_cell, tri_cap, ovf, err);
  else
    launch_k(k_scan<false>, "k_scan", (unsigned)nseg, kScanThreads, kScanListBytes, st, box, codes, n, nseg, state,
             offsets, voff, totals, tri_cell, tri_cap, ovf, err);
  return cudaSuccess;
}

void launch_vertices(const FieldDev& F, const SlabDev& S, const SceneDev& scene, const unsigned char* codes,
                     const VOffDev& voff, long long n, const VertDev& V, cudaStream_t st) {
  /* a warp's tile: a quarter of the cells' share of the resident warps (12
     blocks of four per SM), so that the last wave is short, within 256 ..
     2048 cells (512^3 f64, two levels: 0.74 ms per frame; tiles up to 4096
     0.78, 512 0.81, 256 0.96) */
  const long long share = n / ((long long)num_sms() * 48 * 4);
  const unsigned tile = (unsigned)std::min<long long>(kVTileMax, std::max(256LL, share / 256 * 256));
  const unsigned blocks = (unsigned)((n + 4LL * tile - 1) / (4LL * tile));
  auto go = [&](auto kernel) {
    launch_k(kernel, "k_vertices", blocks, kVThreads, 0, st, F, S, scene, codes, voff, n, tile, V);
  };
  if (F.vx) {
    if (F.is_f32) go(k_vertices<float, false>);
    else go(k_vertices<double, false>);
  } else {
    if (F.is_f32) go(k_vertices<float, true>);
    else go(k_vertices<double, true>);
  }
}

void launch_emit(const FieldDev& F, const SlabDev& S, const SceneDev& scene, const unsigned long long* lut,
                 const unsigned char* codes, const unsigned* offsets,
                 const VOffDev& voff, const unsigned* tri_cell, const unsigned long long* total,
                 long long tri_bound, const TriDev& tri, const RasterDev& R, const VertDev& V, unsigned* checks,
                 cudaStream_t st) {
  const int g = grid_for(tri_bound, 256, g_emit_per_sm);
  if (!R.cover_count) {
    /* inspection: edge ids and flags only */
    launch_k(k_emit<double, false, false>, "k_emit", g, 256, 0, st, F, S, scene, lut, codes, offsets, voff,
             tri_cell, total, tri, R, V, checks);
  } else if (checks) {
    if (F.is_f32)
      launch_k(k_emit<float, true, true>, "k_emit", g, 256, 0, st, F, S, scene, lut, codes, offsets, voff,
               tri_cell, total, tri, R, V, checks);
    else
      launch_k(k_emit<double, true, true>, "k_emit", g, 256, 0, st, F, S, scene, lut, codes, offsets, voff,
               tri_cell, total, tri, R, V, checks);
  } else {
    if (F.is_f32)
      launch_k(k_emit<float, false, true>, "k_emit", g, 256, 0, st, F, S, scene, lut, codes, offsets, voff,
               tri_cell, total, tri, R, V, checks);
    else
      launch_k(k_emit<double, false, true>, "k_emit", g, 256, 0, st, F, S, scene, lut, codes, offsets, voff,
               tri_cell, total, tri, R, V, checks);
  }
}

unsigned long long emit_list_slack(long long tri_bound) {
  return emit_slack_for((unsigned long long)grid_for(tri_bound, 256, g_emit_per_sm));
}

void launch_exact_all(const Geo& G, const unsigned long long* total, long long tri_bound, const TriDev& tri,
                      cudaStream_t st) {
  launch_k(k_exact_all, "k_exact_all", grid_for(tri_bound, 256, 8), 256, 0, st, G, total, tri);
}

void launch_normals(const FieldDev& F, const SlabDev& S, const unsigned* offsets, const unsigned* tri_cell,
                    const unsigned long long* total, long long tri_bound, const TriDev& tri, cudaStream_t st) {
  const int g = grid_for(tri_bound, 256, 8);
  launch_k(k_normals, "k_normals", g, 256, 0, st, F, S, offsets, tri_cell, total, tri);
}

void launch_raster(const Geo& G, const SceneDev& scene, long long tri_bound, const TriDev& tri,
                   const RasterDev& R, unsigned* checks, cudaStream_t st) {
  /* cover and sliver entries together number at most the slab's triangles */
  const int g = grid_for(tri_bound, 128, g_raster_per_sm);
  if (G.F.is_f32) {
    if (checks) launch_k(k_raster<float, true>, "k_raster", g, 128, 0, st, G, scene, tri, R, checks);
    else launch_k(k_raster<float, false>, "k_raster", g, 128, 0, st, G, scene, tri, R, checks);
  } else {
    if (checks) launch_k(k_raster<double, true>, "k_raster", g, 128, 0, st, G, scene, tri, R, checks);
    else launch_k(k_raster<double, false>, "k_raster", g, 128, 0, st, G, scene, tri, R, checks);
  }
}

int launch_finish(const Geo& G, const SceneDev& scene, long long cands, long long tiny, const RasterDev& R,
                  unsigned long long order_base, const FrameObjs& objs, unsigned* checks, cudaStream_t st) {
  const FinMode mode = objs.n == 0 ? kFinExact : (G.F.cgx ? kFinFast : kFinList);
  const int g = grid_for(cands, 32, fin_per_sm(mode));
  auto go = [&](auto kernel) { launch_k(kernel, "k_finish", g, 256, 0, st, G, scene, R, order_base, checks); };
  if (mode == kFinExact) {
    if (checks) go(k_finish<double, true, kFinExact>);
    else go(k_finish<double, false, kFinExact>);
  } else if (mode == kFinList) {
    go(k_finish<double, false, kFinList>);
  } else if (G.F.is_f32) {
    if (checks) go(k_finish<float, true, kFinFast>);
    else go(k_finish<float, false, kFinFast>);
  } else {
    if (checks) go(k_finish<double, true, kFinFast>);
    else go(k_finish<double, false, kFinFast>);
  }
  const int ge = grid_for(cands + tiny, 8, kExactPerSm);
  if (checks) launch_k(k_exact<true>, "k_exact", ge, 32, 0, st, G, scene, R, objs, order_base, checks);
  else launch_k(k_exact<false>, "k_exact", ge, 32, 0, st, G, scene, R, objs, order_base, checks);
  return 2;
}

void launch_shade_f(const FieldDev& F, const SceneDev& scene, const RasterDev& R, const unsigned long long* lut,
                    unsigned long long obase, unsigned rgb, cudaStream_t st) {
  const long long npx = scene.width * scene.height;
  const unsigned long long span = 12ULL * (unsigned long long)((F.nx - 1) * (F.ny - 1) * (F.nz - 1));
  const long long tiles = ((scene.width + 15) / 16) * ((scene.height + 15) / 16);
  launch_k(k_winners, "k_winners", grid_for(256 * tiles, 256, 8), 256, 0, st, R.canvas, (unsigned)scene.width,
           (unsigned)scene.height, obase, span, R.win, R.win_count);
  /* no single-precision shading without node spacings (a converter) or for
     axes of 2^20 nodes and more (hash keys): every pixel to the FP64 pass */
  if (!F.dgx || F.nx > (1 << 20) || F.ny > (1 << 20) || F.nz > (1 << 20)) return;
  const int gs = grid_for(4 * npx, 128, 16); /* four threads per pixel */
  if (F.is_f32) {
    if (R.shade_check) launch_k(k_shade_f<float, true>, "k_shade_f", gs, 128, 0, st, F, scene, R, lut, obase, rgb);
    else launch_k(k_shade_f<float, false>, "k_shade_f", gs, 128, 0, st, F, scene, R, lut, obase, rgb);
  } else {
    if (R.shade_check) launch_k(k_shade_f<double, true>, "k_shade_f", gs, 128, 0, st, F, scene, R, lut, obase, rgb);
    else launch_k(k_shade_f<double, false>, "k_shade_f", gs, 128, 0, st, F, scene, R, lut, obase, rgb);
  }
}

void launch_shade_amb(const FieldDev& F, const SceneDev& scene, const RasterDev& R, const unsigned long long* lut,
                      unsigned long long obase, unsigned rgb, unsigned long long* ent_count, unsigned* checks,
                      cudaStream_t st) {
  const int g = grid_for(scene.width * scene.height, kAmbPixels, 8);
  auto go = [&](auto kernel) {
    launch_k(kernel, "k_shade_amb", g, 128, 0, st, F, scene, R, lut, obase, rgb, ent_count, checks);
  };
  const bool check = checks && R.shade_check;
  if (F.is_f32) {
    if (check) go(k_shade_amb<float, true>);
    else go(k_shade_amb<float, false>);
  } else {
    if (check) go(k_shade_amb<double, true>);
    else go(k_shade_amb<double, false>);
  }
}

void launch_shade_exact(const FieldDev& F, const SceneDev& scene, const RasterDev& R, const unsigned long long* lut,
                        const unsigned* pixels, const unsigned long long* count, long long npix,
                        unsigned long long obase, unsigned long long* ent, unsigned long long ent_cap,
                        unsigned long long* ent_count, uint2* spans, double* wn, unsigned rgb, cudaStream_t st) {
  if (npix <= 0) return;
  launch_k(k_nb_list, "k_nb_list", grid_for(3 * npix, 256, 8), 256, 0, st, F, R, lut, pixels, count, obase, ent,
           ent_cap, ent_count, spans);
  launch_k(k_nb_wn, "k_nb_wn", grid_for((long long)ent_cap, kNbEntries, 8), 256, 0, st, F, lut, ent, ent_cap, ent_count, wn);
  launch_k(k_shade, "k_shade", grid_for(npix, 128, 24), 128, 0, st, F, scene, R, lut, pixels, count, obase, spans, wn,
           rgb);
}

void launch_lines(const LineSegDev* segs, int nseg, long long most, const SceneDev& scene, const RasterDev& R,
                  const unsigned long long* lut, const FrameObjs& objs, unsigned long long order_base, cudaStream_t st) {
  if (nseg <= 0) return;
  /* a block per 128 pixels of the longest segment while that fills the GPU, fewer for many segments */
  const long long room = std::max(1LL, (long long)num_sms() * 64 / nseg);
  const long long by = std::max(1LL, std::min(std::min((most + 127) / 128, room), 65535LL));
  launch_k(k_lines, "k_lines", dim3((unsigned)nseg, (unsigned)by), 128, 0, st, segs, nseg, scene, R,
           objs, lut, order_base);
}

void launch_canvas_init(Slot* canvas, unsigned* zlo, long long n, unsigned long long hi, unsigned long long lo,
                        cudaStream_t st) {
  launch_k(k_canvas_init, "k_canvas_init", grid_for(n, 256, 8), 256, 0, st, canvas, zlo, n, hi, lo);
}

void launch_resolve(const Slot* canvas, long long W, long long H, unsigned char* rgb, double* depth,
                    cudaStream_t st) {
  launch_k(k_resolve, "k_resolve", grid_for(W * H, 256, 8), 256, 0, st, canvas, W, H, rgb, depth);
}

}  // namespace c3d
