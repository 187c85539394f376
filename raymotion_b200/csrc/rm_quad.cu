// rm_quad.cu - the 4-wide BVH, collapsed from the binary child-pair records.
//
// The one-thread-per-path kernels, the adjoint, the batch and the ray queries
// traverse it (QTrav); the wavefront's traversal, the shadow rays of a large
// frame's ReSTIR candidates and of spatial reuse, and the no-allocation query
// read the binary records (Trav).
//
// Traversal is bound by the chain of dependent node fetches of each ray (5 to
// 6 of 32 lanes active, DRAM 3 % busy), so a node holds up to four children in
// one 128-byte line: the four boxes as six float4 of bounds (lo.x, hi.x, lo.y,
// hi.y, lo.z, hi.z of the four children), four child words (8-bit triangle
// count / 24-bit link, the traversal's stack entry; 0: no child) and, for the
// refit, where each child's box stands in the binary records (record << 1 |
// slot, -1: no child).  Boxes are the binary records' own floats, so a ray's
// hits are those of the binary BVH.  The format and its traversal are in
// rm_device.cuh (QTrav).
//
// The collapse runs top-down, one launch per level without a read-back: a node
// starts from the two children of its binary record and opens the internal
// child of the largest surface area until it has four children or only
// leaves.  The number of levels is at most the binary tree's depth, which the
// host knows; a launch for an empty level ends at once.  The binary records
// stay: a refit updates their boxes bottom-up and k_refit_last copies them.
//
// That needs a tree of nested boxes.  A subtree that several nodes of a caller's
// BVH share would be written once for each path to it, and the box of an opened
// child is not tested, which hides subtrees whose boxes reach out of it.  Such
// records become a node each, of their two children (k_quad_pairs).
#include <cuda_runtime.h>

#include <algorithm>

#include "rm_device.cuh"
#include "rm_launch.h"

namespace rmd {

namespace {

struct QChild {
  float lo[3], hi[3];
  int link, cnt;  // cnt > 0: leaf of cnt triangles from record link; 0: binary record link; < 0: none
  int src;        // record << 1 | slot
};

__device__ __forceinline__ QChild read_child(const float4* __restrict__ rec, int r, int slot) {
  const float4* q = rec + size_t(r) * 4;
  const float4 b = q[slot], c = q[2];
  const int4 d = *reinterpret_cast<const int4*>(q + 3);
  QChild ch;
  ch.lo[0] = b.x; ch.hi[0] = b.y; ch.lo[1] = b.z; ch.hi[1] = b.w;
  ch.lo[2] = slot ? c.z : c.x;
  ch.hi[2] = slot ? c.w : c.y;
  ch.link = slot ? d.y : d.x;
  ch.cnt = slot ? d.w : d.z;
  ch.src = (r << 1) | slot;
  return ch;
}

__device__ __forceinline__ float half_area(const QChild& c) {
  const float ex = c.hi[0] - c.lo[0], ey = c.hi[1] - c.lo[1], ez = c.hi[2] - c.lo[2];
  return ex * ey + ey * ez + ez * ex;
}

// roots[i]: the binary record node i collapses; level_n[l]: nodes of level l.
__global__ void k_quad_init(int* roots, int* level_n, int levels) {
  const int i = threadIdx.x;
  if (i < levels) level_n[i] = i == 0 ? 1 : 0;
  if (i == 0) roots[0] = 0;
}

// The nodes [begin, begin + n_here) of a level; theirs to come follow them, counted in *next_n.
__device__ __forceinline__ void collapse_level(const float4* __restrict__ rec, int begin, int n_here, int first,
                                               int stride, int* roots, int* next_n, float4* __restrict__ quads) {
  for (int k = first; k < n_here; k += stride) {
    const int node = begin + k, r = __ldcg(roots + node);
    QChild ch[4];
    int n = 0;
    for (int s = 0; s < 2; ++s) {
      const QChild c = read_child(rec, r, s);
      if (c.cnt >= 0) ch[n++] = c;
    }
#pragma unroll
    for (int open = 0; open < 2; ++open) {
      int best = -1;
      float area = -1.0f;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < n && ch[j].cnt == 0) {
          const float a = half_area(ch[j]);
          if (a > area || best < 0) { area = a; best = j; }
        }
      if (best < 0) break;
      const int link = ch[best].link;
      const QChild a = read_child(rec, link, 0), b = read_child(rec, link, 1);
      // a reachable record has both children (only a lone leaf's has one)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j == best) ch[j] = a;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j == n) ch[j] = b;
      ++n;
    }
    int n_int = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < n && ch[j].cnt == 0) ++n_int;
    int next = begin + n_here + (n_int ? atomicAdd(next_n, n_int) : 0);
    uint32_t word[4];
    int src[4];
    float b[6][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool have = j < n;
      word[j] = 0u;
      src[j] = have ? ch[j].src : -1;
      if (have) {
        if (ch[j].cnt == 0) {
          roots[next] = ch[j].link;
          word[j] = uint32_t(next++);
        } else {
          word[j] = (uint32_t(ch[j].cnt) << 24) | uint32_t(ch[j].link);
        }
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        b[2 * a][j] = have ? ch[j].lo[a] : 0.0f;
        b[2 * a + 1][j] = have ? ch[j].hi[a] : 0.0f;
      }
    }
    float4* q = quads + size_t(node) * 8;
#pragma unroll
    for (int a = 0; a < 6; ++a) q[a] = make_float4(b[a][0], b[a][1], b[a][2], b[a][3]);
    reinterpret_cast<uint4*>(q)[6] = make_uint4(word[0], word[1], word[2], word[3]);
    reinterpret_cast<int4*>(q)[7] = make_int4(src[0], src[1], src[2], src[3]);
  }
}

__global__ void __launch_bounds__(128) k_quad_level(const float4* __restrict__ rec, int level, int* roots,
                                                    int* level_n, float4* __restrict__ quads) {
  int begin = 0;
  for (int l = 0; l < level; ++l) begin += level_n[l];
  collapse_level(rec, begin, level_n[level], int(blockIdx.x * blockDim.x + threadIdx.x), int(gridDim.x * blockDim.x),
                 roots, level_n + level + 1, quads);
}

// The levels from `level` to the last, one block: a launch per level takes 4 us,
// of which a small tree's levels use little and its empty ones (the binary
// tree's depth is the bound) nothing.
constexpr int kQuadRestThreads = 512;

__global__ void __launch_bounds__(kQuadRestThreads) k_quad_rest(const float4* __restrict__ rec, int level, int levels,
                                                                int* roots, int* level_n,
                                                                float4* __restrict__ quads) {
  __shared__ int next_n;
  const int tid = int(threadIdx.x);
  int begin = 0, n = 1;
  if (level == 0 && tid == 0) roots[0] = 0;
  if (level > 0) {
    for (int l = 0; l < level; ++l) begin += level_n[l];
    n = level_n[level];
  }
  int l = level;
  for (; l < levels && n > 0; ++l) {
    __syncthreads();
    if (tid == 0) {
      level_n[l] = n;
      next_n = 0;
    }
    __syncthreads();
    collapse_level(rec, begin, n, tid, kQuadRestThreads, roots, &next_n, quads);
    __syncthreads();
    begin += n;
    n = next_n;
  }
  if (tid == 0)
    for (; l < levels; ++l) level_n[l] = 0;
}

// One node per record, of its two children: node and record share their index.
__global__ void __launch_bounds__(128) k_quad_pairs(const float4* __restrict__ rec, int n_records, int* roots,
                                                    int* level_n, int levels, float4* __restrict__ quads) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < levels) level_n[r] = r == 0 ? n_records : 0;  // (all in one level: what k_refit_last sums)
  if (r >= n_records) return;
  roots[r] = r;
  float4* q = quads + size_t(r) * 8;
  const QChild a = read_child(rec, r, 0), b = read_child(rec, r, 1);
  // a box's bounds may come in either order: the test takes the lesser as near
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    q[2 * k] = make_float4(fminf(a.lo[k], a.hi[k]), fminf(b.lo[k], b.hi[k]), 0.0f, 0.0f);
    q[2 * k + 1] = make_float4(fmaxf(a.lo[k], a.hi[k]), fmaxf(b.lo[k], b.hi[k]), 0.0f, 0.0f);
  }
  auto word = [](const QChild& c) { return c.cnt < 0 ? 0u : (uint32_t(c.cnt) << 24) | uint32_t(c.link); };
  reinterpret_cast<uint4*>(q)[6] = make_uint4(word(a), word(b), 0u, 0u);
  reinterpret_cast<int4*>(q)[7] = make_int4(a.cnt < 0 ? -1 : a.src, b.cnt < 0 ? -1 : b.src, -1, -1);
}

// The last pass of a refit: each child's box copied from the (refitted) binary
// records, one thread per child, and the triangles' records written anew
// (blocks from `quad_blocks` on).  In one launch: a refit of twelve triangles 65
// -> 63 us, of 1,000 94 -> 90.
__global__ void __launch_bounds__(256) k_refit_last(const float4* __restrict__ rec, const int* __restrict__ level_n,
                                                    int levels, float4* __restrict__ quads, int quad_blocks,
                                                    const rm_triangle* __restrict__ tris,
                                                    const int32_t* __restrict__ order, int n_tris,
                                                    float4* __restrict__ tgeo) {
  if (int(blockIdx.x) >= quad_blocks) {
    const int i = (int(blockIdx.x) - quad_blocks) * 256 + int(threadIdx.x);
    if (i < n_tris) pack_record(tris[order[i]], order[i], tgeo + size_t(i) * 3);
    return;
  }
  __shared__ int nodes;
  if (threadIdx.x < 32) {
    int n = 0;
    for (int l = int(threadIdx.x); l < levels; l += 32) n += level_n[l];
    n = int(__reduce_add_sync(0xffffffffu, n));
    if (threadIdx.x == 0) nodes = n;
  }
  __syncthreads();
  const int n = nodes;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n * 4; i += quad_blocks * 256) {
    const int j = i & 3;
    float* q = reinterpret_cast<float*>(quads + size_t(i >> 2) * 8);
    const int src = reinterpret_cast<const int*>(q)[28 + j];
    if (src < 0) continue;
    const QChild c = read_child(rec, src >> 1, src & 1);
#pragma unroll
    for (int a = 0; a < 3; ++a) { q[8 * a + j] = c.lo[a]; q[8 * a + 4 + j] = c.hi[a]; }
  }
}

}  // namespace

int quad_bound(int n_records) {
  // a tree of n_records + 1 leaves at most: full nodes consume three leaves or
  // subtrees each, the others hold only leaves, at least two
  return 2 * (n_records + 1) / 3 + 2;
}

cudaError_t build_quads(DevBvh& b, cudaStream_t st) {
  if (b.n_records <= 0) return cudaSuccess;
  const int bound = b.tree ? quad_bound(b.n_records) : b.n_records;
  cudaError_t e;
  if ((e = b.quads.reserve(size_t(bound) * 8 * sizeof(float4))) != cudaSuccess) return e;
  if ((e = b.qroots.reserve((size_t(bound) + kStack + 2) * sizeof(int))) != cudaSuccess) return e;
  int* level_n = b.qroots.as<int>();
  int* roots = level_n + kStack + 2;
  if (!b.tree) {
    const int n = std::max(b.n_records, kStack + 2);
    k_quad_pairs<<<(n + 127) / 128, 128, 0, st>>>(b.records.as<float4>(), b.n_records, roots, level_n, kStack + 2,
                                                  b.quads.as<float4>());
    return cudaGetLastError();
  }
  // One block takes a small tree whole and the levels behind the twelfth of a
  // middling one (a caller's BVH of 60 and of 1,000 triangles uploaded: 90 and
  // 120 us against 105 and 155 with a launch per level; 20,000: within the
  // spread; a larger tree's late levels hold more than one block is fast with).
  const int depth = std::max(1, std::min(b.max_depth, kStack));
  const int launched = b.n_records <= 2048 ? 0 : b.n_records <= 65536 ? std::min(depth, 12) : depth;
  if (launched > 0) k_quad_init<<<1, 128, 0, st>>>(roots, level_n, kStack + 2);
  long long most = 1;
  for (int l = 0; l < launched; ++l) {
    const long long blocks = std::min<long long>(148 * 8, (std::min<long long>(most, bound) + 127) / 128);
    k_quad_level<<<unsigned(blocks), 128, 0, st>>>(b.records.as<float4>(), l, roots, level_n, b.quads.as<float4>());
    most = std::min<long long>(most * 4, bound);
  }
  if (launched < depth)
    k_quad_rest<<<1, kQuadRestThreads, 0, st>>>(b.records.as<float4>(), launched, kStack + 2, roots, level_n,
                                                b.quads.as<float4>());
  return cudaGetLastError();
}

cudaError_t refit_last(const rm_triangle* d_tris, DevBvh& b, cudaStream_t st) {
  if (b.n_records <= 0 || b.n_tris <= 0) return cudaSuccess;
  const long long n = 4ll * (b.tree ? quad_bound(b.n_records) : b.n_records);
  const int quad_blocks = int(std::min<long long>(148 * 8, (n + 255) / 256));
  k_refit_last<<<unsigned(quad_blocks + (b.n_tris + 255) / 256), 256, 0, st>>>(
      b.records.as<float4>(), b.qroots.as<int>(), kStack + 2, b.quads.as<float4>(), quad_blocks, d_tris,
      b.order.as<int32_t>(), b.n_tris, b.tgeo.as<float4>());
  return cudaGetLastError();
}

}  // namespace rmd
