// Multi-layer z-buffer rasterizer for GB300: triangle setup, screen-tile
// binning and a persistent shared-memory fine rasterizer over an
// (image, tile) work queue. One launch sequence covers a whole ragged batch.
//
// Results are bit-identical to diffren's rasterizers
// (diffren/common/kernels/rasterize_triangles_impl_cuda.cu.cc:244-395 for
// DR_DEPTH_DISCRETIZED, rasterize_triangles_impl.cc:27-118 for
// DR_DEPTH_FLOAT): the per-fragment arithmetic is the reference's, and each
// pixel keeps the L smallest packed (depth | triangle id) keys, which is
// independent of the order fragments arrive in.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <string>

#include "common.cuh"
#include "internal.h"

static_assert(dr::kErrorFlagsOffset == 4, "error word is counters[1]");

namespace dr {
namespace {

// Fine-raster block = triangle chunk size. 128-thread blocks keep eight
// tiles in flight per SM (each tile's setup, scan and epilogue are serial
// latency chains), which measured faster than four 256-thread tiles and
// than sixteen 64-thread ones.
constexpr int kThreads = 128;
constexpr int kDefaultTile = 16;
constexpr int kDefaultLargeTiles = 16;

// What setup keeps of a triangle: its clip vertices and vertex indices, 64
// bytes in four 16-byte loads. With back-face culling the edge coefficients
// (72 bytes) are recomputed from it where they are needed, in about 50
// instructions: a scattered load costs an L1 cycle per lane, and nine of them
// per sample bounded the epilogue, as their stores did setup. The other
// culling modes round each coefficient to float precision, which costs three
// times that: setup keeps theirs (RasterArgs::edges). With 144-byte records
// of everything the fine kernel took 313 us on a 200k-triangle soup
// (8 x 512^2), 629 on the 4 x 2048^2 terrain and 1025 on the 64-mesh ragged
// batch, now 244, 548 and 974 (16x16 tiles); setup 109, 227 and 137 us, now
// 94, 138 and 114.
struct __align__(16) TriSetup {
  float4 v[3];
  int32_t vid[3];
  int32_t small;  // the coordinates fit 32 bits in fixed point (fits_fixed32)
};
static_assert(sizeof(TriSetup) == 64, "TriSetup layout");

// Workspace taken per triangle for the record and the coefficients; rounded
// up so that what a caller's or the static scratch's fixed size admits does
// not move with their layout.
constexpr size_t kSetupBytes = 144;
static_assert(sizeof(TriSetup) + 5 * sizeof(longlong2) <= kSetupBytes, "setup workspace");

struct RasterArgs {
  const float4* verts;
  const int32_t* tris;
  int culling, depth_mode, L, TW, TH, large_tiles;
  bool fg_only;  // DR_RASTER_FOREGROUND_ONLY: background ids / barycentrics unwritten
  bool fg_attr;  // DR_RASTER_FOREGROUND_ATTRIBUTES: background attributes unwritten
  int swizzle;  // min(2^k, 16) - 1 of the power of two in TW (see fine_raster_kernel)
  uint32_t inv_tw, inv_th;  // ceil(2^32 / TW), ceil(2^32 / TH) (see tile_index)
  int64_t total_tris;
  int32_t total_tiles;
  int scan_shift;  // tiles per block of tile_scan_kernel, as a power of two
  TriSetup* setup;
  longlong2* edges;  // [tris][5] (the tenth unused), for DR_CULL_NONE / FRONT
  uint2* box;   // left | right << 16, bottom | top << 16; empty when culled
  int2* place;  // inside one tile: {tile, slot}; in 2..large_tiles tiles:
                // {-2, -}; otherwise {-1, -}
  int32_t* tile_count;  // triangles inside one tile (their slots come from here)
  int32_t* tile_multi;  // triangles spanning 2..large_tiles tiles
  int32_t* tile_fill;   // bin slots taken by the multi-tile triangles
  uint32_t* order;      // [tiles][3] the fine rasterizer's queue (see pack_tile),
                        // over the three arrays above once the bins are filled
  int32_t* tile_first;  // first bin of each tile; the tiles of one scan block
                        // follow each other (see tile_end)
  int32_t* bins;        // global triangle indices grouped by tile
  int32_t* large_count;  // per image
  int32_t* large_list;   // per image, at tri_start[image]
  uint32_t* counters;    // [0] work queue head, [1] error flags, [2, 9) tiles
                         // per cost class, [9, 16) their fill counts, [16]
                         // bins taken, [17, 49) end of each scan block's bins
  int32_t* ids;
  float* z;
  float* bary;
  SampleOutputs so;
};

// Workspace: the zeroed block first, then the rest; 256-byte aligned parts.
struct Layout {
  size_t counters, tile_count, tile_multi, tile_fill, large_count, zero_end;  // order: tile_count
  size_t tile_first, setup, box, place, bins, large_list, total;
};

size_t align_up(size_t x) { return (x + 255) & ~size_t(255); }

Layout make_layout(int64_t tris, int64_t tiles, int images, int large_tiles) {
  Layout l;
  size_t o = 0;
  l.counters = o; o = align_up(o + 256);
  l.tile_count = o; o = align_up(o + 4 * tiles);
  l.tile_multi = o; o = align_up(o + 4 * tiles);
  l.tile_fill = o; o = align_up(o + 4 * tiles);
  l.large_count = o; o = align_up(o + 4 * size_t(images));
  l.zero_end = o;
  l.tile_first = o; o = align_up(o + 4 * (tiles + 1));
  l.setup = o; o = align_up(o + kSetupBytes * tris);
  l.box = o; l.place = o + 8 * tris; o = align_up(o + 16 * tris);
  l.bins = o; o = align_up(o + 4 * size_t(large_tiles) * tris);
  l.large_list = o; o = align_up(o + 4 * tris);
  l.total = o;
  return l;
}

// True when no pixel center of `box` can pass the inside test: the sum of
// the three edge functions is linear in the fixed-point pixel coordinates
// (which are monotone in the pixel index), so it is <= 0 over the whole box
// iff it is <= 0 at the four corners. Only used when no int64 term can
// overflow (|m| < 2^43), so the test is exact.
__device__ bool cannot_cover(const long long m[9], int4 box, int W, int H, bool fused) {
  const long long lim = 1LL << 43;
#pragma unroll
  for (int i = 0; i < 9; ++i)
    if (m[i] >= lim || m[i] <= -lim) return false;
  const long long A = m[0] + m[3] + m[6];
  const long long B = m[1] + m[4] + m[7];
  const long long C = (m[2] + m[5] + m[8]) * 65536;
  const long long x0 = pixel_center_fixed(box.x, W, fused);
  const long long x1 = pixel_center_fixed(box.y - 1, W, fused);
  const long long y0 = pixel_center_fixed(box.z, H, fused);
  const long long y1 = pixel_center_fixed(box.w - 1, H, fused);
  const long long s00 = A * x0 + B * y0 + C, s10 = A * x1 + B * y0 + C;
  const long long s01 = A * x0 + B * y1 + C, s11 = A * x1 + B * y1 + C;
  return s00 <= 0 && s10 <= 0 && s01 <= 0 && s11 <= 0;
}

// x / size for x < 2^16 and size <= 128, by the reciprocal ceil(2^32 / size)
// (of size 1 it would not fit).
__device__ __forceinline__ int tile_index(int x, int size, uint32_t inv) {
  return size == 1 ? x : int(__umulhi(uint32_t(x), inv));
}

__device__ __forceinline__ void tile_rect(const RasterArgs& a, int4 box, int& tx0, int& tx1,
                                          int& ty0, int& ty1) {
  tx0 = tile_index(box.x, a.TW, a.inv_tw);
  tx1 = tile_index(box.y - 1, a.TW, a.inv_tw);
  ty0 = tile_index(box.z, a.TH, a.inv_th);
  ty1 = tile_index(box.w - 1, a.TH, a.inv_th);
}

// Image sides are at most 32768, so a box's four bounds pack into 16 bits each.
__device__ __forceinline__ int4 unpack_box(uint2 b) {
  return make_int4(int(b.x & 0xffffu), int(b.x >> 16), int(b.y & 0xffffu), int(b.y >> 16));
}

// End of tile i's bins.
__device__ __forceinline__ int tile_end(const RasterArgs& a, int i) {
  const int mask = (1 << a.scan_shift) - 1;
  return (i & mask) == mask || i + 1 == a.total_tiles ? int(a.counters[17 + (i >> a.scan_shift)])
                                                      : a.tile_first[i + 1];
}

// Edge coefficients of a triangle that setup kept.
__device__ __forceinline__ void load_edges(const RasterArgs& a, int64_t g, const float4 (&v)[3],
                                           bool small, long long m[9]) {
  if (a.culling == DR_CULL_BACK) {
    edge_matrix(v[0], v[1], v[2], DR_CULL_BACK, small, m);
  } else {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const longlong2 e = __ldg(a.edges + 5 * g + k);
      m[2 * k] = e.x;
      if (k < 4) m[2 * k + 1] = e.y;
    }
  }
}

// One thread per triangle of the batch: bounding box, edge matrix, exact
// coverage cull, per-tile counts (small triangles) or the large list.
// Bounded to 64 registers so that 32 warps share an SM: the kernel waits on
// its index and vertex loads, and the extra warps hide more of that than the
// few bytes of spills cost (measured against 24 warps and 40; blocks of 128
// threads a little faster than of 256).
__global__ void __launch_bounds__(128, 8) setup_kernel(RasterArgs a, Batch B) {
  const int64_t g = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  // Lanes past the end still take part in the warp-wide tile match below.
  const bool live = g < a.total_tris;
  const int img = live ? find_segment(B.tri_start, B.n, g) : 0;
  const int64_t t = g - B.tri_start[img];
  const int W = B.width[img], H = B.height[img];
  const int32_t* tri = a.tris + 3 * (B.triangle_offset[img] + t);
  const int i0 = live ? tri[0] : 0, i1 = live ? tri[1] : 0, i2 = live ? tri[2] : 0;
  const unsigned nv = unsigned(B.num_vertices[img]);
  int4 box = make_int4(0, 0, 0, 0);
  bool valid = false;
  if (!live) {
  } else if (unsigned(i0) >= nv || unsigned(i1) >= nv || unsigned(i2) >= nv) {
    atomicOr(&a.counters[1], DR_FLAG_INDEX_OUT_OF_RANGE);
  } else {
    const float4* vb = a.verts + B.vertex_offset[img];
    const float4 v0 = vb[i0], v1 = vb[i1], v2 = vb[i2];
    // x - x == 0 exactly for finite x, NaN for NaN and infinities.
    const float probe = (v0.x - v0.x) + (v0.y - v0.y) + (v0.z - v0.z) + (v0.w - v0.w) +
                        (v1.x - v1.x) + (v1.y - v1.y) + (v1.z - v1.z) + (v1.w - v1.w) +
                        (v2.x - v2.x) + (v2.y - v2.y) + (v2.z - v2.z) + (v2.w - v2.w);
    if (probe != 0.0f) atomicOr(&a.counters[1], DR_FLAG_NONFINITE_VERTEX);
    const bool disc = a.depth_mode == DR_DEPTH_DISCRETIZED;
    valid = triangle_box(v0, v1, v2, W, H, box, disc);
    if (valid) {
      long long m[9];
      const bool small = fits_fixed32(v0, v1, v2);
      edge_matrix(v0, v1, v2, a.culling, small, m);
      valid = !cannot_cover(m, box, W, H, disc);
      if (valid) {
        TriSetup* t = a.setup + g;
        t->v[0] = v0;
        t->v[1] = v1;
        t->v[2] = v2;
        *reinterpret_cast<int4*>(t->vid) = make_int4(i0, i1, i2, small);
        if (a.culling != DR_CULL_BACK) {
#pragma unroll
          for (int k = 0; k < 5; ++k)
            a.edges[5 * g + k] = make_longlong2(m[2 * k], k < 4 ? m[2 * k + 1] : 0);
        }
      }
    }
  }
  if (!valid) box = make_int4(0, 0, 0, 0);
  if (live) a.box[g] = make_uint2(unsigned(box.x | box.y << 16), unsigned(box.z | box.w << 16));
  int tx0 = 0, tx1 = -1, ty0 = 0, ty1 = -1;
  if (valid) tile_rect(a, box, tx0, tx1, ty0, ty1);
  const int n = (tx1 - tx0 + 1) * (ty1 - ty0 + 1);
  const int base = B.tile_start[img], tx = B.tiles_x[img];
  // Triangles inside one tile count with one atomic per tile per warp.
  const bool single = valid && n == 1 && n <= a.large_tiles;
  const int tile0 = base + ty0 * tx + tx0;
  const unsigned group = __match_any_sync(0xffffffffu, single ? tile0 : -1 - lane);
  if (single) {
    // The warp's triangles in this tile take consecutive slots, so that the
    // binning pass needs no atomic.
    const int leader = __ffs(group) - 1;
    int first = 0;
    if (lane == leader) first = atomicAdd(&a.tile_count[tile0], __popc(group));
    first = __shfl_sync(group, first, leader);
    a.place[g] = make_int2(tile0, first + __popc(group & ((1u << lane) - 1u)));
    return;
  }
  if (live) a.place[g] = make_int2(valid && n <= a.large_tiles ? -2 : -1, 0);
  if (!valid) return;
  if (n <= a.large_tiles) {
    for (int y = ty0; y <= ty1; ++y)
      for (int x = tx0; x <= tx1; ++x) atomicAdd(&a.tile_multi[base + y * tx + x], 1);
  } else {
    const int slot = atomicAdd(&a.large_count[img], 1);
    a.large_list[B.tri_start[img] + slot] = int(g);
  }
}

// Tile order of the fine rasterizer: the most expensive tiles first, so that
// no block is left with a heavy tile while the others have run out of work
// (the per-tile cost spans three orders of magnitude in ragged batches). The
// cost of a tile is its triangle count (binned plus the image's large ones),
// in seven classes, heaviest first and the empty ones last; inside a class
// tiles keep roughly their index order (block by block), which keeps an
// image's tiles together in L2. The order does not change any output: tiles
// are independent.
constexpr int kCostClasses = 7, kEmptyClass = kCostClasses - 1;

__device__ __forceinline__ int cost_class(int c) {
  return c >= 512 ? 0 : c >= 128 ? 1 : c >= 32 ? 2 : c >= 8 ? 3 : c >= 2 ? 4 : c >= 1 ? 5 : 6;
}

// Bins of every tile, and the tiles of each cost class (counters[2 + class]).
// Blocks take 2^scan_shift tiles each (at most 32 blocks) and their bins from
// a counter: where a tile's bins lie does not matter, so no block waits for
// another. One block scanning every count took 30 us for 111k tiles, this 5.
__global__ void __launch_bounds__(1024) tile_scan_kernel(RasterArgs a, Batch B) {
  __shared__ int warp_sums[32];
  __shared__ int s_base;
  __shared__ int h[kCostClasses];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r0 = blockIdx.x << a.scan_shift;
  const int r1 = min(a.total_tiles, r0 + (1 << a.scan_shift));
  // Counts past the last tile are zeros (the arrays are padded and cleared).
  const auto counts = [&](int i) {
    const int4 c = *reinterpret_cast<const int4*>(a.tile_count + i);
    const int4 m = *reinterpret_cast<const int4*>(a.tile_multi + i);
    return make_int4(c.x + m.x, c.y + m.y, c.z + m.z, c.w + m.w);
  };
  if (threadIdx.x < kCostClasses) h[threadIdx.x] = 0;
  int sum = 0;
  for (int i = r0 + 4 * int(threadIdx.x); i < r1; i += 4 * 1024) {
    const int4 c = counts(i);
    sum += c.x + c.y + c.z + c.w;
  }
  sum = __reduce_add_sync(0xffffffffu, sum);
  if (lane == 0) warp_sums[warp] = sum;
  __syncthreads();
  if (warp == 0) {
    sum = __reduce_add_sync(0xffffffffu, warp_sums[lane]);
    if (lane == 0) {
      s_base = int(atomicAdd(&a.counters[16], unsigned(sum)));
      a.counters[17 + blockIdx.x] = unsigned(s_base + sum);
    }
  }
  __syncthreads();
  int carry = s_base;
  for (int base = r0; base < r1; base += 4 * 1024) {
    const int i = base + 4 * int(threadIdx.x);
    const int4 c = i < r1 ? counts(i) : make_int4(0, 0, 0, 0);
    const int four = c.x + c.y + c.z + c.w;
    const int inc = warp_inclusive_scan(four);
    __syncthreads();  // warp_sums of the pass before has been read
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < 32; ++w) {
      const int v = warp_sums[w];
      before += w < warp ? v : 0;
      all += v;
    }
    if (i < r1) {
      const int first = carry + before + inc - four;
      *reinterpret_cast<int4*>(a.tile_first + i) =
          make_int4(first, first + c.x, first + c.x + c.y, first + c.x + c.y + c.z);
      const int n[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (i + k < a.total_tiles)
          atomicAdd(&h[cost_class(n[k] + a.large_count[find_segment(B.tile_start, B.n, i + k)])], 1);
    }
    carry += all;
  }
  __syncthreads();
  if (threadIdx.x < kCostClasses && h[threadIdx.x])
    atomicAdd(&a.counters[2 + threadIdx.x], unsigned(h[threadIdx.x]));
}

// One thread per triangle: writes its index into the bin of every tile its
// box touches. Order inside a bin is irrelevant to the result. Triangles
// inside one tile (most of them) took their slot in setup; the multi-tile
// ones take theirs after the tile's single-tile triangles.
__global__ void __launch_bounds__(256) bin_scatter_kernel(RasterArgs a, Batch B) {
  const int64_t g = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (g >= a.total_tris) return;
  const int2 place = a.place[g];
  if (place.x >= 0) {
    a.bins[a.tile_first[place.x] + place.y] = int(g);
    return;
  }
  if (place.x != -2) return;
  int tx0, tx1, ty0, ty1;
  tile_rect(a, unpack_box(a.box[g]), tx0, tx1, ty0, ty1);
  const int img = find_segment(B.tri_start, B.n, g);
  const int base = B.tile_start[img], ntx = B.tiles_x[img];
  // Four tiles at a time, so that their atomics' latencies overlap.
  int x = tx0, y = ty0;
  while (y <= ty1) {
    int tile[4], pos[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      tile[k] = y <= ty1 ? base + y * ntx + x : -1;
      if (++x > tx1) {
        x = tx0;
        ++y;
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (tile[k] >= 0)
        pos[k] = a.tile_first[tile[k]] + a.tile_count[tile[k]] + atomicAdd(&a.tile_fill[tile[k]], 1);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (tile[k] >= 0) a.bins[pos[k]] = int(g);
  }
}

// A tile of the queue in three words: its first bin slot; its triangles in
// the bins (27 bits, saturated) and 5 bits of its image; its origin (15 bits
// each) and 2 more bits of the image (DR_MAX_BATCH_INLINE = 128). One load
// then tells a block all about its next tile, where looking the image up and
// reading the bin bounds was a chain of two more loads and two divisions.
constexpr uint32_t kMaxPackedCount = (1u << 27) - 1;
static_assert(DR_MAX_BATCH_INLINE <= 128 && DR_MAX_IMAGE_DIM <= 32768, "pack_tile's fields");

__device__ __forceinline__ void pack_tile(uint32_t* o, uint32_t bin0, uint32_t nbin, int img,
                                          int x0, int y0) {
  o[0] = bin0;
  o[1] = min(nbin, kMaxPackedCount) | uint32_t(img & 31) << 27;
  o[2] = uint32_t(x0) | uint32_t(y0) << 15 | uint32_t(img >> 5) << 30;
}

// Writes every tile to its place in the order: class c starts after the
// tiles of classes < c, and each block takes a run of its classes' slots
// (counters[9 + class]).
__global__ void __launch_bounds__(256) tile_order_kernel(RasterArgs a, Batch B) {
  __shared__ int h[kCostClasses], base[kCostClasses];
  if (threadIdx.x < kCostClasses) h[threadIdx.x] = 0;
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int c = 0, rank = 0, img = 0, first = 0, n_bin = 0;
  if (i < a.total_tiles) {
    img = find_segment(B.tile_start, B.n, i);
    first = a.tile_first[i];
    n_bin = tile_end(a, i) - first;
    c = cost_class(n_bin + a.large_count[img]);
    rank = atomicAdd(&h[c], 1);
  }
  __syncthreads();
  if (threadIdx.x < kCostClasses) {
    int start = 0;
    for (int k = 0; k < int(threadIdx.x); ++k) start += int(a.counters[2 + k]);
    const int n = h[threadIdx.x];
    base[threadIdx.x] =
        start + (n ? int(atomicAdd(&a.counters[2 + kCostClasses + threadIdx.x], unsigned(n))) : 0);
  }
  __syncthreads();
  if (i < a.total_tiles) {
    const int local = i - B.tile_start[img], ntx = B.tiles_x[img];
    const int ty = local / ntx, tx = local - ty * ntx;
    pack_tile(a.order + 3 * size_t(base[c] + rank), first, n_bin, img, tx * a.TW, ty * a.TH);
  }
}

// Per chunk of up to kChunk triangles overlapping the tile, compacted to
// those with at least one candidate pixel (slot = rank among them).
struct FineSmem {
  long long* m;          // [9][kChunk]
  float* row;            // [9][kChunk] row-span coefficients (see row_coefficients)
  float* vz;             // [3][kChunk]
  float* vw;             // [3][kChunk]
  int* tid;              // [kChunk] local triangle id
  int* geom;             // [kChunk] x0 | y0 << 8 | width << 16 (tile-local)
  int* off;              // [kChunk + 1] exclusive row offsets
  int* pxf;              // [TW] fixed-point pixel-center x
  int* pyf;              // [TH]
  unsigned long long* keys;  // [L][TW*TH]
  unsigned short* queue;  // [kThreads / 32][kQueue] candidate pixels of each warp
  unsigned char* first;  // [kThreads / 32 * TH] slot holding row 32 g, per g
};

// A row pushes up to kPush candidates at a time; fewer than 32 are carried
// from one push to the next.
constexpr int kPush = 8, kQueue = 32 * kPush + 32;
// Between chunks the queues hold gather_inline's list.
static_assert(kThreads / 32 * kQueue * sizeof(unsigned short) >= kThreads * sizeof(int),
              "gather_inline's list");

// Triangles a chunk holds. Up to 768 keys (16x16 pixels of three layers) eight
// blocks of 128 fit an SM's shared memory, as the registers allow, and every
// further chunk costs: the fine kernel takes 545 us on the 4 x 2048^2 terrain
// with 128, 574 with 96, 625 with 64. Above, 64 keep eight blocks up to eight
// layers of 16x16, where 128 leave seven or six: 800 us on the 64-mesh
// ragged batch in 32x16 tiles (883 with 128); setup to fine kernel for a
// 100k-triangle sphere (8 x 1024^2) 454 us (466) at four layers, 535 (579) at
// six, 612 (649) at eight.
__host__ __device__ inline int chunk_of(int L, int TW, int TH) {
  return L * TW * TH > 768 ? 64 : 128;
}

// The chunk's edge coefficients; the epilogue reuses the space for its list
// of occupied (layer, pixel) slots (16 bits each).
__host__ __device__ inline size_t chunk_m_bytes(int L, int TW, int TH) {
  const size_t m = size_t(9) * chunk_of(L, TW, TH) * 8, list = size_t(L) * TW * TH * 2;
  return ((m > list ? m : list) + 7) & ~size_t(7);
}

__host__ __device__ inline size_t fine_smem_bytes(int L, int TW, int TH) {
  const size_t chunk = chunk_of(L, TW, TH);
  return chunk_m_bytes(L, TW, TH) + size_t(TW + TH) * 4 + size_t(L) * TW * TH * 8 +
         17 * chunk * 4 + (chunk + 4) * 4 +
         size_t(kThreads / 32) * kQueue * 2 + size_t(kThreads / 32) * TH;
}

// Which pixels of a row can be inside a triangle, from float32: edge i at
// fixed-point pixel center (x, y) is e = m0 x + m1 y + 65536 m2, so on a row
// e >= 0 reads x >= t g where m0 > 0 and x <= t g where m0 < 0, with
// t = m1 y + 65536 m2 and g = -1 / m0. |x|, |y| <= 65536 (the pixel centers
// lie in [-1, 1]), so the float32 roundings of the m and of t move e by less
// than 2^-22 s, s = 65536 (|m0| + |m1| + |m2|): t is raised by 2^-20 s, which
// keeps every pixel that the exact test accepts. m0 = 0 gets g = +inf, so
// that t < 0 empties the row. Coefficients from 2^43 on, whose edge functions
// may wrap, constrain nothing.
template <int kChunk>
__device__ __forceinline__ void row_coefficients(const long long* m, float* row, int slot) {
  bool wraps = false;
#pragma unroll
  for (int i = 0; i < 9; ++i) wraps |= m[i] >= (1LL << 43) || m[i] <= -(1LL << 43);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float a = __ll2float_rn(m[3 * i]), b = __ll2float_rn(m[3 * i + 1]),
                c = __ll2float_rn(m[3 * i + 2]);
    const float s = fabsf(a) + fabsf(b) + fabsf(c);
    row[(3 * i) * kChunk + slot] =
        wraps || a == 0.0f ? __int_as_float(0x7f800000) : __fdividef(-1.0f, a);
    row[(3 * i + 1) * kChunk + slot] = wraps ? 0.0f : b;
    row[(3 * i + 2) * kChunk + slot] = wraps ? 1.0f : fmaf(s, 0.0625f, c * 65536.0f);
  }
}

// Fused interpolation of one occupied layer sample o, the record of its
// triangle and the barycentrics just written: the splat position of a
// foreground sample (splat.py:207-221) with its clip w, its three vertex
// indices when requested (the Framebuffer's vertex_ids,
// rasterize.py:111-113), and the attributes (interpolate.py:24-63). The same
// operations, in the same order, as samples_fwd_kernel on the stored buffers.
// A depth of exactly 1 is background: its attributes stay as
// fill_background left them.
__device__ __forceinline__ void write_sample(const RasterArgs& a, const Batch& B, int img,
                                          int4 vid, const float4 (&v)[3], float zz,
                                          const float b[3], int64_t o) {
  const SampleOutputs& so = a.so;
  const int K = so.K;
  const bool vec_rows = (K & 3) == 0;
  if (zz == 1.0f) return;
  const int v0 = vid.x, v1 = vid.y, v2 = vid.z;
  const float4 c = lerp_clip(v[0], v[1], v[2], b);
  if (so.attr) {
    float* ao = so.attr_out + o * K;
    const float* ab = so.attr + B.vertex_offset[img] * K;
    const float* a0 = ab + int64_t(v0) * K;
    const float* a1 = ab + int64_t(v1) * K;
    const float* a2 = ab + int64_t(v2) * K;
    if (K == 4) {  // RGBA vertex colors
      const float4 x = __ldg(reinterpret_cast<const float4*>(a0)),
                   y = __ldg(reinterpret_cast<const float4*>(a1)),
                   w = __ldg(reinterpret_cast<const float4*>(a2));
      *reinterpret_cast<float4*>(ao) =
          make_float4(lerp3(x.x, y.x, w.x, b), lerp3(x.y, y.y, w.y, b),
                      lerp3(x.z, y.z, w.z, b), lerp3(x.w, y.w, w.w, b));
    } else for (int k = 0; k < K; k += 4) {
      const int n = min(4, K - k);
      const float4 x = load_chunk(a0 + k, n, vec_rows), y = load_chunk(a1 + k, n, vec_rows),
                   w = load_chunk(a2 + k, n, vec_rows);
      store_chunk(ao + k,
                  make_float4(lerp3(x.x, y.x, w.x, b), lerp3(x.y, y.y, w.y, b),
                              lerp3(x.z, y.z, w.z, b), lerp3(x.w, y.w, w.w, b)),
                  n, vec_rows);
    }
  }
  // w carries the interpolated clip w, which the VJP needs (background
  // and foreground are told apart by the depth buffer).
  so.positions[o] = viewport_of(c, __int2float_rn(B.width[img]),
                                __int2float_rn(B.height[img]), c.w);
  if (so.vertex_ids) {
    int32_t* vo = so.vertex_ids + 3 * o;
    vo[0] = v0;
    vo[1] = v1;
    vo[2] = v2;
  }
}

// One tile of an image in the packed layered buffers.
struct TileBox {
  int64_t base;  // element of layer 0, pixel (0, 0)
  int64_t hw;    // elements per layer
  int img, W, x0, y0, tw, th;
  int bin0, nbin;
};

// Entry k of the queue, as packed by pack_tile.
__device__ __forceinline__ uint3 tile_words(const RasterArgs& a, int k) {
  const uint32_t* o = a.order + 3 * size_t(k);
  return make_uint3(__ldg(o), __ldg(o + 1), __ldg(o + 2));
}

__device__ __forceinline__ TileBox tile_box(const RasterArgs& a, const Batch& B, uint3 o, int L) {
  TileBox t;
  t.img = int((o.y >> 27) | (o.z >> 30) << 5);
  t.W = B.width[t.img];
  t.hw = int64_t(t.W) * B.height[t.img];
  t.base = int64_t(L) * B.pix_off[t.img];
  t.x0 = int(o.z & 0x7fffu);
  t.y0 = int((o.z >> 15) & 0x7fffu);
  t.tw = min(a.TW, t.W - t.x0);
  t.th = min(a.TH, B.height[t.img] - t.y0);
  t.bin0 = int(o.x);
  t.nbin = int(o.y & kMaxPackedCount);
  if (uint32_t(t.nbin) == kMaxPackedCount) {
    const int item = B.tile_start[t.img] + (t.y0 / a.TH) * B.tiles_x[t.img] + t.x0 / a.TW;
    t.nbin = tile_end(a, item) - t.bin0;
  }
  return t;
}

// The fine rasterizer's queue: the occupied tiles in order, then the empty
// ones in runs (they only write background samples). A run is as long as two
// for every block allow, up to kEmptyRun: always eight left most blocks without
// work in images of a few thousand tiles (1024x1024, eight layers, 300 tiny
// triangles: 58 us, 43 so).
constexpr unsigned kEmptyRun = 8;

struct Queue {
  unsigned occupied, items, run;
};

__device__ __forceinline__ Queue make_queue(const RasterArgs& a) {
  const unsigned empty = a.counters[2 + kEmptyClass];
  Queue q;
  q.occupied = unsigned(a.total_tiles) - empty;
  q.run = min(max(empty / (2 * gridDim.x), 1u), kEmptyRun);
  q.items = q.occupied + (empty + q.run - 1) / q.run;
  return q;
}

// One item as its block sees it.
struct QueueItem {
  int kind;  // 0 tile, 1 empty run, 2 end
  uint3 o;   // tile: its words; run: its first entry and the one after its last
};

__device__ __forceinline__ QueueItem queue_item(const RasterArgs& a, const Queue& q,
                                                unsigned head) {
  QueueItem it;
  it.kind = head < q.occupied ? 0 : head < q.items ? 1 : 2;
  const unsigned first = q.occupied + (head - q.occupied) * q.run;
  it.o = make_uint3(first, min(first + q.run, unsigned(a.total_tiles)), 0u);
  if (it.kind == 0) it.o = tile_words(a, int(head));
  return it;
}

// Writes v to the `ch` values of every layer sample of a tile, row by row:
// consecutive threads take consecutive float4s (floats where a row does not
// start and end on 16 bytes).
__device__ __forceinline__ void fill_rows(float* buf, int ch, float v, const TileBox& t, int L) {
  const int64_t first = (t.base + int64_t(t.y0) * t.W + t.x0) * ch;
  const int64_t layer = t.hw * ch;
  const int row = t.W * ch, n = t.tw * ch;
  const bool vec = (((row | n | int(first) | int(layer)) & 3) |
                    int(reinterpret_cast<uintptr_t>(buf) & 15)) == 0;
  const int cols = vec ? n >> 2 : n, step = vec ? 4 : 1;
  int y0, dy, dc = 0;
  if ((cols & (cols - 1)) == 0 && cols <= kThreads) {  // whole rows per step, no division
    const int lg = __ffs(cols) - 1;
    y0 = threadIdx.x >> lg;
    dy = kThreads >> lg;
  } else {
    y0 = threadIdx.x / cols;
    dy = kThreads / cols;
    dc = kThreads - dy * cols;
  }
  const int c0 = threadIdx.x - y0 * cols;
  float* p = buf + first;
  for (int l = 0; l < L; ++l, p += layer) {
    int c = c0;
    for (int y = y0; y < t.th; y += dy) {
      float* q = p + (y * row + step * c);
      if (vec)
        *reinterpret_cast<float4*>(q) = make_float4(v, v, v, v);
      else
        *q = v;
      c += dc;
      if (c >= cols) {
        c -= cols;
        ++y;
      }
    }
  }
}

// Every sample of a tile as background: depth 1, and the ids, barycentrics
// and attributes that the flags ask for (positions are left unwritten:
// consumers take background samples from the depth buffer). Tiles without
// triangles end here; in the others the occupied samples are overwritten
// after a block barrier. Whole rows of float4s instead of a test and a store
// per sample: with it and the packed queue the kernel takes 1029 us instead
// of 1128 on the 64-mesh ragged batch (28.4 Mpixel, 78% background), 652
// instead of 737 on the 4 x 2048^2 terrain; the fill itself is bound by HBM
// (1.7 GB in 0.2 ms of it on the ragged batch).
template <bool kFused>
__device__ __forceinline__ void fill_background(const RasterArgs& a, const TileBox& t, int L) {
  fill_rows(a.z, 1, 1.0f, t, L);
  if (!a.fg_only) {
    fill_rows(reinterpret_cast<float*>(a.ids), 1,
              __int_as_float(a.depth_mode == DR_DEPTH_DISCRETIZED ? 0 : -1), t, L);
    fill_rows(a.bary, 3, 0.0f, t, L);
  }
  if (kFused && a.so.attr && !a.fg_attr) fill_rows(a.so.attr_out, a.so.K, 0.0f, t, L);
}

// The next chunk of a tile whose image has more large triangles than a chunk
// holds: the nrest < kChunk triangles that its bins still have (none where
// negative), then those of the large list whose box meets the tile's. Taken as
// they lie, most chunks of such a list hold a handful of triangles for this
// tile, and a chunk costs its chain of loads and barriers whatever it holds:
// 100k triangles 110 pixels wide at 1024x1024 took 4.57 ms (3.41 before a
// chunk's rows were narrowed and queued), with full chunks 2.35. Boxes are
// looked at 128 at a time, four groups of loads in flight. list: kChunk
// integers. scan: the first triangle of the next group, and how many of that
// group's hits an earlier chunk took.
template <int kChunk>
__device__ __forceinline__ int gather_inline(const int32_t* large, int nlarge, const uint2* boxes,
                                             const int32_t* rest, int nrest, int4 tile, int* list,
                                             int* s_warp, int2* scan) {
  const int tid = threadIdx.x;
  int next = scan->x, skip = scan->y;
  int have = max(0, nrest);
  if (tid < have) list[tid] = rest[tid];
  while (have < kChunk && next < nlarge) {
    constexpr int kAhead = 4;
    int g[kAhead];
    uint2 box[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const int i = next + k * kThreads + tid;
      g[k] = i < nlarge ? large[i] : -1;
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k) box[k] = g[k] >= 0 ? boxes[g[k]] : make_uint2(0u, 0u);
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      if (have >= kChunk) break;
      const int4 b = unpack_box(box[k]);
      const bool hit = b.y > tile.x && b.x < tile.y && b.w > tile.z && b.z < tile.w;
      int rank;
      const int all = block_exclusive_scan<kThreads>(hit ? 1 : 0, s_warp, rank) - skip;
      const int at = have + rank - skip;
      if (hit && at >= have && at < kChunk) list[at] = g[k];
      if (all > kChunk - have) {  // the rest of this group is the next chunk's
        skip += kChunk - have;
        have = kChunk;
      } else {
        have += all;
        skip = 0;
        next += kThreads;
      }
    }
  }
  __syncthreads();
  if (tid == 0) *scan = make_int2(next, skip);
  __syncthreads();
  return tid < have ? list[tid] : -1;
}

// Inline where the layer count is fixed and the sample outputs are fused; the
// other instantiations spill 92 bytes with it inline (sphere, 8 x 1024^2: 222,
// 296 and 406 us at one, two and four layers) and 20 with a call (216, 282, 390),
// where a call costs the first kind 1 to 3%.
template <int kChunk>
__device__ __noinline__ int gather_call(const int32_t* large, int nlarge, const uint2* boxes,
                                        const int32_t* rest, int nrest, uint32_t x, uint32_t y,
                                        int* list, int* s_warp, int2* scan) {
  const int4 tile = make_int4(int(x & 0xffffu), int(x >> 16), int(y & 0xffffu), int(y >> 16));
  return gather_inline<kChunk>(large, nlarge, boxes, rest, nrest, tile, list, s_warp, scan);
}

template <int kChunk, bool kInline>
__device__ __forceinline__ int gather_large(const int32_t* large, int nlarge, const uint2* boxes,
                                            const int32_t* rest, int nrest, int4 tile, int* list,
                                            int* s_warp, int2* scan) {
  if constexpr (kInline)
    return gather_inline<kChunk>(large, nlarge, boxes, rest, nrest, tile, list, s_warp, scan);
  else
    return gather_call<kChunk>(large, nlarge, boxes, rest, nrest,
                               uint32_t(tile.x) | uint32_t(tile.y) << 16,
                               uint32_t(tile.z) | uint32_t(tile.w) << 16, list, s_warp, scan);
}

// Persistent fine rasterizer. Each block takes (image, tile) items from a
// global queue (heaviest tiles first, in tile_order_kernel's order), keeps
// the tile's L x TW x TH packed keys in shared memory, and spreads the rows
// of each chunk's triangles (clipped to the tile) evenly over its threads:
// each lane narrows one row to the pixels that can be inside in float32, the
// warp queues them, and full warps of queued pixels take the exact edge
// functions and the rest. Issue-bound: the bounding boxes hold 4 to 6 pixels
// for each one inside, an exact test costs about 90 instructions, and with a
// lane for every box pixel nearly every warp went through the 150 more of an
// accepted one with a fifth of its lanes. Row spans take the kernel from 428
// to 344 us on a 100k-triangle sphere (8 x 1024^2), from 341 to 313 us on a
// 200k-triangle soup (8 x 512^2) and from 87 to 42 us on one 1283x717 image.
// The key of pixel x of row y lies at x ^ (y & swizzle), within the power of two
// in TW: a warp often holds one x of many rows, whose keys would all meet in one
// bank (300 triangles 300 pixels wide at 1024x1024: 138 us without, 123 with it;
// 221 and 181 with eight layers).
// kFused adds the sample outputs to the epilogue. LT > 0 fixes the layer
// count at compile time (the common L = 3), LT = 0 reads it.
template <bool kFused, int LT, int kChunk>
__global__ void __launch_bounds__(kThreads, 8) fine_raster_kernel(RasterArgs a, Batch B) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_warp[kThreads / 32];
  __shared__ Queue s_queue;  // thread 0's: in registers it would take every thread's
  __shared__ QueueItem s_item;
  __shared__ int s_nfg;
  __shared__ int2 s_scan;  // where the scan of the image's large list stands
  const int TW = a.TW, TH = a.TH, TP = TW * TH, L = LT > 0 ? LT : a.L;
  FineSmem s;
  {
    unsigned char* p = smem_raw;
    s.keys = reinterpret_cast<unsigned long long*>(p); p += size_t(L) * TP * 8;
    s.m = reinterpret_cast<long long*>(p); p += chunk_m_bytes(L, TW, TH);
    s.pxf = reinterpret_cast<int*>(p); p += size_t(TW) * 4;
    s.pyf = reinterpret_cast<int*>(p); p += size_t(TH) * 4;
    s.row = reinterpret_cast<float*>(p); p += size_t(9) * kChunk * 4;
    s.vz = reinterpret_cast<float*>(p); p += size_t(3) * kChunk * 4;
    s.vw = reinterpret_cast<float*>(p); p += size_t(3) * kChunk * 4;
    s.tid = reinterpret_cast<int*>(p); p += kChunk * 4;
    s.geom = reinterpret_cast<int*>(p); p += kChunk * 4;
    s.off = reinterpret_cast<int*>(p); p += (kChunk + 4) * 4;
    s.queue = reinterpret_cast<unsigned short*>(p); p += size_t(kThreads / 32) * kQueue * 2;
    s.first = p;
  }
  const int inv_tw = ((1 << 20) + TW - 1) / TW;  // p / TW = (p inv_tw) >> 20 for p < 1024
  const unsigned long long kEmpty = empty_key(a.depth_mode);
  const bool disc = a.depth_mode == DR_DEPTH_DISCRETIZED;

  if (threadIdx.x == 0) s_queue = make_queue(a);
  for (;;) {
    if (threadIdx.x == 0) s_item = queue_item(a, s_queue, atomicAdd(&a.counters[0], 1u));
    __syncthreads();
    const QueueItem it = s_item;
    if (it.kind == 2) break;
    if (it.kind == 1) {
      for (int k = int(it.o.x); k < int(it.o.y); ++k)
        fill_background<kFused>(a, tile_box(a, B, tile_words(a, k), L), L);
      __syncthreads();
      continue;
    }
    const TileBox tb = tile_box(a, B, it.o, L);
    const int img = tb.img;
    const int W = tb.W, H = B.height[img], x0 = tb.x0, y0 = tb.y0, tw = tb.tw, th = tb.th;
    const int64_t tri0 = B.tri_start[img];

    fill_background<kFused>(a, tb, L);
    for (int p = threadIdx.x; p < L * TP; p += kThreads) s.keys[p] = kEmpty;
    for (int i = threadIdx.x; i < TW + TH; i += kThreads) {
      if (i < TW) s.pxf[i] = int(pixel_center_fixed(x0 + i, W, disc));
      else s.pyf[i - TW] = int(pixel_center_fixed(y0 + i - TW, H, disc));
    }
    const int bin0 = tb.bin0, nbin = tb.nbin;
    const int nlarge = a.large_count[img];
    int nsrc = nbin + nlarge;
    if (threadIdx.x == 0) s_scan = make_int2(0, 0);
    // Fixed-point x to pixel index: x = px W / 131072 + W / 2 - 1/2. Rounding
    // the pixel centers to fixed point moves them by at most 2 units, and
    // the float32 steps here stay below 0.02 pixels.
    const float to_x = __int2float_rn(W) * (1.0f / 131072.0f);
    const float slack = 2.5f * to_x + 0.03f;
    const float x_off = __int2float_rn(W) * 0.5f - 0.5f - __int2float_rn(x0);
    __syncthreads();

    for (int c0 = 0; c0 < nsrc; c0 += kChunk) {
      const int i = c0 + threadIdx.x;
      int cnt = 0, g = -1, cx0 = 0, cy0 = 0, cw = 1;
      if (nlarge > kChunk && c0 + kChunk > nbin) {
        g = gather_large<kChunk, (kFused && LT > 0)>(
            a.large_list + tri0, nlarge, a.box, a.bins + bin0 + c0, nbin - c0,
            make_int4(x0, x0 + tw, y0, y0 + th), reinterpret_cast<int*>(s.queue), s_warp, &s_scan);
        if (s_scan.x >= nlarge) nsrc = 0;  // the last chunk
      } else if ((kChunk == kThreads || threadIdx.x < kChunk) && i < nsrc) {
        g = i < nbin ? a.bins[bin0 + i] : a.large_list[tri0 + (i - nbin)];
      }
      if (g >= 0) {
        const int4 box = unpack_box(a.box[g]);
        cx0 = max(box.x, x0) - x0;
        cy0 = max(box.z, y0) - y0;
        const int cx1 = min(box.y, x0 + tw) - x0, cy1 = min(box.w, y0 + th) - y0;
        if (cx1 > cx0 && cy1 > cy0) {
          cw = cx1 - cx0;
          cnt = cy1 - cy0;
        }
      }
      // One scan gives each triangle with candidates its compacted slot
      // (bits 20+) and its first row (bits 0-19): at most kChunk * 128 rows
      // per chunk.
      int excl;
      const int tot = block_exclusive_scan<kThreads>(cnt | (cnt > 0 ? 1 << 20 : 0), s_warp, excl);
      const int total = tot & 0xfffff, ntri = tot >> 20;
      if (cnt > 0) {
        const int slot = excl >> 20, off = excl & 0xfffff;
        const TriSetup* st = a.setup + g;
        const float4 v[3] = {__ldg(st->v), __ldg(st->v + 1), __ldg(st->v + 2)};
        long long mm[9];
        load_edges(a, g, v, __ldg(&st->small), mm);
#pragma unroll
        for (int k = 0; k < 9; ++k) s.m[k * kChunk + slot] = mm[k];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          s.vz[k * kChunk + slot] = v[k].z;
          s.vw[k * kChunk + slot] = v[k].w;
        }
        s.tid[slot] = int(g - tri0);
        row_coefficients<kChunk>(mm, s.row, slot);
        s.geom[slot] = cx0 | (cy0 << 8) | (cw << 16);
        s.off[slot] = off;
        // This triangle holds row 32 q for every q with 32 q in
        // [off, off + cnt).
        for (int q = (off + 31) >> 5; (q << 5) < off + cnt; ++q) s.first[q] = (unsigned char)slot;
      }
      if (threadIdx.x == 0) s.off[ntri] = total;
      __syncthreads();

      // Warp-wide groups of 32 consecutive rows. The group's first row lies
      // in triangle j0 = first[q]; the triangles that start inside the group
      // mark their start positions in one 32-bit mask, and lane t's triangle
      // is j0 plus the marks at positions 1..t. Each lane narrows its row to
      // the pixels [xa, xa + n) and the warp queues them (lane | x << 5); the
      // last round (no group left) empties the queue.
      const int lane = threadIdx.x & 31;
      unsigned short* queue = s.queue + (threadIdx.x >> 5) * kQueue;
      int held = 0;       // queued pixels carried to the next push (< 32), ...
      unsigned held_px = 0;  // ... the lane-th of them: slot | y << 8 | x << 16
      for (int q = threadIdx.x >> 5;; q += kThreads / 32) {
        const bool more = (q << 5) < total;
        int n = 0, xa = 0;
        unsigned slot_y = 0;
        if (more) {
          const int base = q << 5;
          const int j0 = s.first[q];
          const int jn = j0 + 1 + lane;
          const int d = jn <= ntri ? s.off[jn] - base : 32;
          const unsigned starts = __reduce_or_sync(0xffffffffu, d > 0 && d < 32 ? 1u << d : 0u);
          if (base + lane < total) {
            const int j = j0 + __popc(starts & ((2u << lane) - 1u));
            const int geom = s.geom[j];
            const int ly = ((geom >> 8) & 255) + (base + lane - s.off[j]);
            const float y = __int2float_rn(int(s.pyf[ly]));
            float lo = -1.0e6f, hi = 1.0e6f;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              const float g = s.row[(3 * i) * kChunk + j];
              const float x = fmaf(s.row[(3 * i + 1) * kChunk + j], y,
                                   s.row[(3 * i + 2) * kChunk + j]) * g;
              if (g < 0.0f) lo = fmaxf(lo, x); else hi = fminf(hi, x);
            }
            const int cx0 = geom & 255;
            const int x_lo = __float2int_ru(fmaf(fminf(lo, 1.0e6f), to_x, x_off - slack));
            const int x_hi = __float2int_rd(fmaf(fmaxf(hi, -1.0e6f), to_x, x_off + slack));
            xa = max(cx0, x_lo);
            n = max(0, min(cx0 + (geom >> 16) - 1, x_hi) - xa + 1);
            slot_y = unsigned(j | (ly << 8));
          }
        }
        do {
          int count = held;
          for (int t = 0; t < kPush; ++t) {
            const unsigned on = __ballot_sync(0xffffffffu, t < n);
            if (!on) break;
            if (t < n)
              queue[count + __popc(on & ((1u << lane) - 1u))] =
                  (unsigned short)(lane | ((xa + t) << 5));
            count += __popc(on);
          }
          xa += min(n, kPush);
          n -= min(n, kPush);
          __syncwarp();
          // Full warps of queued pixels (and the rest in the last round).
          const int stop = more ? count & ~31 : count;
          for (int base = 0;; base += 32) {
            const int at = base + lane;
            const unsigned c = queue[at < count ? at : 0];
            unsigned px = __shfl_sync(0xffffffffu, slot_y, c & 31u) | ((c >> 5) << 16);
            if (at < held) px = held_px;
            if (base >= stop) {
              held_px = px;
              held = count - stop;
              break;
            }
            if (at >= count) continue;
            const int j = int(px & 255u), ly = int((px >> 8) & 255u), lx = int(px >> 16);
            long long m[9];
#pragma unroll
            for (int t = 0; t < 9; ++t) m[t] = s.m[t * kChunk + j];
            long long e[3];
            edge_values(m, s.pxf[lx], s.pyf[ly], e);
            if (!inside(e)) continue;
            float b[3];
            barycentrics_of(e, b);
            const float3 vz = make_float3(s.vz[j], s.vz[kChunk + j], s.vz[2 * kChunk + j]);
            const float3 vw = make_float3(s.vw[j], s.vw[kChunk + j], s.vw[2 * kChunk + j]);
            const float z = fragment_z(b, vz, vw, disc);
            unsigned long long key;
            if (disc) {
              if (z < -1.0f || z > 1.0f) continue;  // NaN passes, as in the reference
              key = ((unsigned long long)discretize_z(z) << 32) | uint32_t(s.tid[j]);
            } else {
              if (!(z >= -1.0f && z < 1.0f)) continue;
              key = ((unsigned long long)float_order_bits(z) << 32) | uint32_t(s.tid[j]);
            }
            if (key >= kEmpty) continue;
            unsigned long long* kp = s.keys + (ly * TW + (lx ^ (ly & a.swizzle)));
            // Slot values only decrease, so a key above the current last layer
            // can never be among the pixel's L smallest.
            if (key > *reinterpret_cast<volatile unsigned long long*>(kp + (L - 1) * TP)) continue;
            for (int l = 0; l < L; ++l) {
              const unsigned long long old = atomicMin(kp + l * TP, key);
              if (old == kEmpty) break;
              key = max(key, old);
            }
          }
          __syncwarp();
        } while (__any_sync(0xffffffffu, n > 0));
        if (!more) break;
      }
      __syncthreads();
    }

    // Epilogue: list the occupied slots (layer << 10 | pixel, in the chunk
    // arrays' space, dead by now), then with full warps unpack each, recompute
    // the barycentrics (and float depth) of its triangle and overwrite the
    // background that fill_background wrote; optionally also each sample's
    // splat position and interpolated attributes.
    unsigned short* list = reinterpret_cast<unsigned short*>(s.m);
    if (threadIdx.x == 0) s_nfg = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int p0 = 0; p0 < TP; p0 += kThreads) {
      const int p = p0 + threadIdx.x;
#pragma unroll
      for (int l = 0; l < L; ++l) {
        const bool full = p < TP && s.keys[l * TP + p] != kEmpty;
        const unsigned ball = __ballot_sync(0xffffffffu, full);
        if (!ball) break;  // layers fill front to back
        int slot0 = 0;
        if (lane == 0) slot0 = atomicAdd(&s_nfg, __popc(ball));
        slot0 = __shfl_sync(0xffffffffu, slot0, 0);
        if (full) list[slot0 + __popc(ball & ((1u << lane) - 1u))] = (unsigned short)(l << 10 | p);
      }
    }
    __syncthreads();
    const int nfg = s_nfg;
    for (int f = threadIdx.x; f < nfg; f += kThreads) {
      const int q = list[f];
      const int l = q >> 10, p = q & 1023;
      const int ly = (p * inv_tw) >> 20, lx = (p - ly * TW) ^ (ly & a.swizzle);
      const unsigned long long key = s.keys[l * TP + p];
      const int64_t o = tb.base + l * tb.hw + ((y0 + ly) * W + x0 + lx);
      float b[3] = {0.0f, 0.0f, 0.0f};
      const int id = int(uint32_t(key));
      const TriSetup* st = a.setup + tri0 + id;
      const float4 v[3] = {__ldg(st->v), __ldg(st->v + 1), __ldg(st->v + 2)};
      const int4 vid = __ldg(reinterpret_cast<const int4*>(st->vid));
      long long m[9];
      load_edges(a, tri0 + id, v, vid.w, m);
      long long e[3];
      edge_values(m, s.pxf[lx], s.pyf[ly], e);
      float bb[3];
      barycentrics_of(e, bb);
      float zz;
      if (disc) {
        zz = undiscretize_z(uint32_t(key >> 32));
      } else {
        const float3 vz = make_float3(v[0].z, v[1].z, v[2].z);
        const float3 vw = make_float3(v[0].w, v[1].w, v[2].w);
        zz = fragment_z(bb, vz, vw, false);
      }
      if (!disc || zz != 1.0f) { b[0] = bb[0]; b[1] = bb[1]; b[2] = bb[2]; }
      a.ids[o] = id;
      a.z[o] = zz;
      float* bo = a.bary + 3 * o;
      bo[0] = b[0];
      bo[1] = b[1];
      bo[2] = b[2];
      if (kFused) write_sample(a, B, img, vid, v, zz, b, o);
    }
    __syncthreads();
  }
}

// Compares the integer depth codec with the reference's double formulas on
// every input: all 2^32 discretized values, and every float in [-1, 1]
// plus NaNs. out: [0] discretize mismatches, [1] first bad float bits,
// [2] undiscretize mismatches, [3] first bad discretized value, [4] the
// discretized value of a NaN depth, [5] / [6] the int32 / int64 conversion
// of a NaN float (toward zero).
__global__ void depth_codec_selftest_kernel(unsigned long long* out) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const float nan = __uint_as_float(0x7fc00000u);
    out[4] = discretize_z_fp64(nan);
    out[5] = (unsigned long long)(unsigned)__float2int_rz(nan);
    out[6] = (unsigned long long)__float2ll_rz(nan);
  }
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < (1ull << 32);
       i += stride) {
    const uint32_t u = uint32_t(i);
    if (__float_as_uint(undiscretize_z(u)) != __float_as_uint(undiscretize_z_fp64(u))) {
      atomicAdd(&out[2], 1ull);
      atomicMin(&out[3], (unsigned long long)u);
    }
    const float z = __uint_as_float(u);
    const bool in_domain = (z != z) || (z >= -1.0f && z <= 1.0f);
    if (in_domain && discretize_z(z) != discretize_z_fp64(z)) {
      atomicAdd(&out[0], 1ull);
      atomicMin(&out[1], (unsigned long long)u);
    }
  }
}

// Raises the fine rasterizer's dynamic shared-memory limit and computes its
// persistent grid (resident blocks per SM x SMs) on the current device.
template <bool kFused, int LT, int kChunk>
bool prepare_fine(size_t smem, int& sms, int& per_sm, std::string& err) {
  static LaunchCache cache;
  return prepare_launch(cache, fine_raster_kernel<kFused, LT, kChunk>, kThreads, smem, sms, per_sm,
                        "tile and layer count need more shared memory than the device has",
                        err);
}

int resolve_tile(int v) { return v > 0 ? v : kDefaultTile; }

bool check_config(const dr_raster_config* cfg, int& L, int& TW, int& TH, int& large,
                  std::string& err) {
  if (!cfg) { err = "config is null"; return false; }
  L = cfg->num_layers;
  TW = resolve_tile(cfg->tile_width);
  TH = resolve_tile(cfg->tile_height);  // see group_batch where neither is given
  large = cfg->large_tiles > 0 ? cfg->large_tiles : kDefaultLargeTiles;
  if (L < 1 || L > DR_MAX_LAYERS) { err = "num_layers must be in [1, 16]"; return false; }
  if (cfg->face_culling_mode < 0 || cfg->face_culling_mode > 2) {
    err = "face_culling_mode must be 0, 1 or 2";
    return false;
  }
  if (cfg->depth_mode != DR_DEPTH_DISCRETIZED && cfg->depth_mode != DR_DEPTH_FLOAT) {
    err = "depth_mode must be 0 (discretized) or 1 (float)";
    return false;
  }
  if (TW > 128 || TH > 128 || TW * TH > 1024) {
    err = "tile must satisfy width, height <= 128 and width*height <= 1024";
    return false;
  }
  if ((cfg->flags & ~(DR_RASTER_FOREGROUND_ONLY | DR_RASTER_FOREGROUND_ATTRIBUTES)) != 0) {
    err = "unknown raster config flags";
    return false;
  }
  return true;
}

// Tile of a group of images whose configuration gives none, from its table
// with 16x16 tiles: another one only where sweeps over triangles from 3 pixels
// to a third of the image wide lost next to nothing. The numbers of tiles and
// triangles tell little else: a dense mesh of small triangles and a scene of
// wide ones, which every tile of the image looks at, count alike.
//
// Up to 840 tiles many of the resident blocks (eight on each SM) are idle, and
// where each tile has work enough smaller ones spread it. Setup to fine kernel,
// of the time with 16x16 tiles (16 to 2000 triangles a tile, 1 to 8 layers): 0.30
// to 1.02 with 8x8 up to 256 tiles, 0.58 to 1.04 with 16x8 up to 840. Below 16
// triangles a tile or 4096 in all the launches are what takes the time (up to
// 1.36 with 8x8). Above, both gain on closed meshes (100k-triangle sphere at
// 1283x717, one layer: fine kernel 32 us with 16x8, 49) and lose elsewhere: 8x8 up
// to 1.24 at 4 x 256x256, 16x8 up to 1.11 there, and 1.35 on 80k triangles 110
// pixels wide at 1024x1024. The threshold of the large list stays the same number
// of tiles: a fourfold one gained up to a third on triangles of 32 to 64 pixels,
// for four times the bins' memory.
//
// Many tiles with few triangles each are bound by the cost per tile: the
// 64-mesh ragged batch (111k tiles) takes 1002 us with 32x16, 1165 with 16x16,
// 2048x2048 images of triangles 11 to 600 pixels wide 0.44 to 1.04 of 16x16's
// time, smaller images up to 1.09 (the widest triangles). With more than 24
// triangles a tile 32x16 is no better (terrain 789, 761). An image whose tiles
// hold more than a 912th of all the triangles each (about a block's share) then
// sets the time: one with 1531 a tile among 979k took 805 us with 32x16, 514 with
// 16x16. Above four layers the keys of a 32x16 tile cost more blocks per SM than
// it gains (eight: 744, 612 on a sphere). 32x8 for rows that do not start on 32
// bytes gained up to 17% on small triangles and lost up to 18% on wider ones.
void default_tile(const Batch& b, int L, int& TW, int& TH) {
  const int64_t tiles = b.tile_start[b.n], tris = b.tri_start[b.n];
  TW = TH = kDefaultTile;
  if (tiles <= 840 && tris >= std::max(int64_t(4096), 16 * tiles)) {
    TW = tiles <= 256 ? 8 : 16;
    TH = 8;
  } else if (tiles >= 16384 && L <= 4 && tris <= 24 * tiles) {
    bool even = true;
    for (int i = 0; i < b.n; ++i) {
      const int64_t t = b.tile_start[i + 1] - b.tile_start[i];
      if (6 * kSms * (b.tri_start[i + 1] - b.tri_start[i]) > tris * t) even = false;
    }
    if (even) TW = 32;
  }
}

// Tiles a triangle may take bins in. Bin positions are 32-bit integers, so all
// triangles together get fewer than 2^31: from 134 million on at the default 16,
// the threshold falls (to 1 at the 2^31 triangles that make_batch refuses).
// Triangles above it go to the large list, whatever their size, and the results
// do not depend on it.
int bounded_large(int large, int64_t tris) {
  return tris > 0 ? int(std::min(int64_t(large), INT32_MAX / tris)) : large;
}

// The batch table of one group with its tiles, and the workspace it needs.
// With a tile by the rule that workspace may exceed the 16x16 one (by its
// tiles' counts), which is then enough too (at 16x16): `min_bytes` is what a
// call must bring.
bool group_batch(const dr_image_desc* images, int n, const dr_raster_config* cfg, int L,
                 size_t ws_bytes, int& TW, int& TH, int& large, Batch& b, Layout& lay,
                 size_t& min_bytes, std::string& err) {
  if (!make_batch(images, n, L, TW, TH, b, err)) return false;
  large = bounded_large(large, b.tri_start[n]);
  lay = make_layout(b.tri_start[n], b.tile_start[n], n, large);
  min_bytes = lay.total;
  if (cfg->tile_width > 0 || cfg->tile_height > 0) return true;
  int w, h;
  default_tile(b, L, w, h);
  if (w == TW && h == TH) return true;
  Batch ruled;
  std::string ignored;
  if (!make_batch(images, n, L, w, h, ruled, ignored)) return true;  // too many tiles
  const Layout l = make_layout(ruled.tri_start[n], ruled.tile_start[n], n, large);
  if (l.total > ws_bytes) return true;
  b = ruled;
  lay = l;
  TW = w;
  TH = h;
  return true;
}

}  // namespace

int depth_codec_selftest(unsigned long long* out, cudaStream_t stream, std::string& err) {
  if (!out) { err = "results buffer is null"; return DR_ERR_INVALID_ARGUMENT; }
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  depth_codec_selftest_kernel<<<sms * 8, 256, 0, stream>>>(out);
  return launch_status("depth codec self-test", err);
}

size_t raster_workspace_bytes(const dr_image_desc* images, int n,
                              const dr_raster_config* cfg, std::string& err) {
  int L, TW, TH, large;
  if (!check_config(cfg, L, TW, TH, large, err)) return 0;
  if (n < 0 || (n > 0 && !images)) { err = "invalid image table"; return 0; }
  size_t best = 256;
  for (int g0 = 0; g0 < n; g0 += DR_MAX_BATCH_INLINE) {
    const int cnt = std::min(n - g0, DR_MAX_BATCH_INLINE);
    Batch b;
    Layout lay;
    int w = TW, h = TH, tiles = large;
    size_t min_bytes;
    if (!group_batch(images + g0, cnt, cfg, L, SIZE_MAX, w, h, tiles, b, lay, min_bytes, err))
      return 0;
    best = std::max(best, std::max(min_bytes, lay.total));
  }
  return best;
}

int raster_launch(const float* vertices, const int32_t* triangles,
                  const dr_image_desc* images, int n, const dr_raster_config* cfg,
                  int32_t* ids, float* z, float* bary, void* workspace,
                  size_t ws_bytes, cudaStream_t stream, std::string& err,
                  const SampleOutputs* samples) {
  int L, TW, TH, large;
  if (!check_config(cfg, L, TW, TH, large, err)) return DR_ERR_INVALID_ARGUMENT;
  if (n < 0 || (n > 0 && !images)) { err = "invalid image table"; return DR_ERR_INVALID_ARGUMENT; }
  if (n == 0) return DR_OK;
  if (!ids || !z || !bary || !workspace) {
    err = "outputs and workspace must be non-null";
    return DR_ERR_INVALID_ARGUMENT;
  }
  if ((reinterpret_cast<uintptr_t>(vertices) & 15) != 0 ||
      (reinterpret_cast<uintptr_t>(workspace) & 255) != 0) {
    err = "vertices must be 16-byte aligned and the workspace 256-byte aligned";
    return DR_ERR_MISALIGNED;
  }
  SampleOutputs so{};
  if (samples) {
    so = *samples;
    if (!so.positions || (so.attr && (!so.attr_out || so.K < 1 || so.K > DR_MAX_CHANNELS))) {
      err = "positions must be non-null, and attributes need attributes_out and 1 to 16 "
            "channels";
      return DR_ERR_INVALID_ARGUMENT;
    }
    if (!so.attr) so.K = 0;
    const bool vec = so.attr && so.K % 4 == 0;
    if ((reinterpret_cast<uintptr_t>(so.positions) & 15) != 0 ||
        (vec && ((reinterpret_cast<uintptr_t>(so.attr) & 15) != 0 ||
                 (reinterpret_cast<uintptr_t>(so.attr_out) & 15) != 0))) {
      err = "positions (and, with a multiple of 4 channels, the attribute buffers) must be "
            "16-byte aligned";
      return DR_ERR_MISALIGNED;
    }
  }
  const bool fused = so.positions != nullptr;
  // Instantiations: fused or not, three layers or any, chunks of 128 or 64.
  using Fine = void (*)(RasterArgs, Batch);
  using Prep = bool (*)(size_t, int&, int&, std::string&);
  const Fine fine[8] = {fine_raster_kernel<false, 0, 128>, fine_raster_kernel<false, 3, 128>,
                        fine_raster_kernel<true, 0, 128>,  fine_raster_kernel<true, 3, 128>,
                        fine_raster_kernel<false, 0, 64>,  fine_raster_kernel<false, 3, 64>,
                        fine_raster_kernel<true, 0, 64>,   fine_raster_kernel<true, 3, 64>};
  const Prep prep[8] = {prepare_fine<false, 0, 128>, prepare_fine<false, 3, 128>,
                        prepare_fine<true, 0, 128>,  prepare_fine<true, 3, 128>,
                        prepare_fine<false, 0, 64>,  prepare_fine<false, 3, 64>,
                        prepare_fine<true, 0, 64>,   prepare_fine<true, 3, 64>};
  const int TW0 = TW, TH0 = TH, large0 = large;
  for (int g0 = 0; g0 < n; g0 += DR_MAX_BATCH_INLINE) {
    const int cnt = std::min(n - g0, DR_MAX_BATCH_INLINE);
    Batch b;
    Layout lay;
    size_t min_bytes;
    TW = TW0;
    TH = TH0;
    large = large0;
    if (!group_batch(images + g0, cnt, cfg, L, ws_bytes, TW, TH, large, b, lay, min_bytes, err))
      return DR_ERR_INVALID_ARGUMENT;
    const int64_t tris = b.tri_start[cnt];
    const int tiles = b.tile_start[cnt];
    if (min_bytes > ws_bytes) {
      err = "workspace too small: need " + std::to_string(min_bytes) + " bytes";
      return DR_ERR_WORKSPACE_TOO_SMALL;
    }
    const int variant =
        (fused ? 2 : 0) + (L == 3 ? 1 : 0) + (chunk_of(L, TW, TH) == 64 ? 4 : 0);
    const size_t smem = fine_smem_bytes(L, TW, TH);
    int sms = 0, per_sm = 0;
    if (!prep[variant](smem, sms, per_sm, err)) return DR_ERR_INVALID_ARGUMENT;
    char* ws = static_cast<char*>(workspace);
    RasterArgs a;
    a.verts = reinterpret_cast<const float4*>(vertices);
    a.tris = triangles;
    a.culling = cfg->face_culling_mode;
    a.depth_mode = cfg->depth_mode;
    a.fg_only = (cfg->flags & DR_RASTER_FOREGROUND_ONLY) != 0;
    a.fg_attr = (cfg->flags & DR_RASTER_FOREGROUND_ATTRIBUTES) != 0;
    a.L = L; a.TW = TW; a.TH = TH; a.large_tiles = large;
    a.total_tris = tris;
    a.total_tiles = tiles;
    a.swizzle = std::min(TW & -TW, 16) - 1;
    a.inv_tw = TW > 1 ? 0xffffffffu / unsigned(TW) + 1u : 0u;
    a.inv_th = TH > 1 ? 0xffffffffu / unsigned(TH) + 1u : 0u;
    a.scan_shift = 12;  // 4096 tiles per block, more above 32 blocks
    while (((int64_t(tiles) + (int64_t(1) << a.scan_shift) - 1) >> a.scan_shift) > 32) ++a.scan_shift;
    a.setup = reinterpret_cast<TriSetup*>(ws + lay.setup);
    a.edges = reinterpret_cast<longlong2*>(ws + lay.setup + sizeof(TriSetup) * size_t(tris));
    a.box = reinterpret_cast<uint2*>(ws + lay.box);
    a.place = reinterpret_cast<int2*>(ws + lay.place);
    a.tile_count = reinterpret_cast<int32_t*>(ws + lay.tile_count);
    a.tile_multi = reinterpret_cast<int32_t*>(ws + lay.tile_multi);
    a.tile_fill = reinterpret_cast<int32_t*>(ws + lay.tile_fill);
    a.tile_first = reinterpret_cast<int32_t*>(ws + lay.tile_first);
    a.order = reinterpret_cast<uint32_t*>(ws + lay.tile_count);
    a.bins = reinterpret_cast<int32_t*>(ws + lay.bins);
    a.large_count = reinterpret_cast<int32_t*>(ws + lay.large_count);
    a.large_list = reinterpret_cast<int32_t*>(ws + lay.large_list);
    a.counters = reinterpret_cast<uint32_t*>(ws + lay.counters);
    a.ids = ids;
    a.z = z;
    a.bary = bary;
    a.so = so;

    if (cudaMemsetAsync(ws, 0, lay.zero_end, stream) != cudaSuccess) {
      err = std::string("cudaMemsetAsync: ") + cudaGetErrorString(cudaGetLastError());
      return DR_ERR_CUDA;
    }
    if (tris > 0) {
      const unsigned grid = unsigned((tris + 127) / 128);
      setup_kernel<<<grid, 128, 0, stream>>>(a, b);
    }
    if (tiles > 0) {
      const unsigned grid = unsigned((int64_t(tiles) + (int64_t(1) << a.scan_shift) - 1) >> a.scan_shift);
      tile_scan_kernel<<<grid, 1024, 0, stream>>>(a, b);
    }
    if (tris > 0) {
      const unsigned grid = unsigned((tris + 255) / 256);
      bin_scatter_kernel<<<grid, 256, 0, stream>>>(a, b);
    }
    if (tiles > 0) {
      const unsigned grid = unsigned((tiles + 255) / 256);
      tile_order_kernel<<<grid, 256, 0, stream>>>(a, b);
    }
    const int blocks = std::max(1, std::min(tiles, sms * per_sm));
    fine[variant]<<<blocks, kThreads, smem, stream>>>(a, b);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      err = std::string("raster launch failed: ") + cudaGetErrorString(e);
      return DR_ERR_CUDA;
    }
  }
  return DR_OK;
}

}  // namespace dr
