// rm_bvh.cu - device BVH: caller-BVH conversion, LBVH build, refit, packing.
//
// The reference builds a binned-SAH binary BVH on the CPU in fp64
// (src/engine/bvh.cpp:29-248), refits it in reverse node order (:250-272),
// and its Metal backend flattens it to preorder escape-link nodes every frame
// (src/engine/metal.mm:129-144).  Here:
//  * a caller BVH in the reference layout is validated, converted to the
//    child-pair layout of rm_device.cuh on the host in O(nodes), and uploaded;
//  * without a caller BVH the device builds a linear BVH (Karras, "Maximizing
//    Parallelism in the Construction of BVHs, Octrees, and k-d Trees", HPG
//    2012): 30-bit Morton codes of the centroids, a radix sort (rm_sort.cu), one
//    thread per internal node to find its range and split, bottom-up boxes
//    with arrival counters; subtrees of at most `leaf_max` triangles collapse
//    into leaves;
//  * refit runs bottom-up on the device over the child-pair records with the
//    same arrival-counter scheme (one pass, no per-level launches).
// Triangle boxes come from the caller's fp32 vertices, so every box bounds its
// float triangle exactly.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <initializer_list>
#include <mutex>
#include <vector>

#include "rm_launch.h"
#include "rm_sort.h"

namespace rmd {

#define RM_TRY_(x)                         \
  do {                                     \
    cudaError_t e_ = (x);                  \
    if (e_ != cudaSuccess) return e_;      \
  } while (0)


namespace {

constexpr int kPoolDevices = 64;
struct DevicePool {
  std::mutex mu;
  int users = 0;
  cudaMemPool_t pool = nullptr;
  cudaStream_t stream = nullptr;  // orders the pool's own allocations and frees; carries no work
  void* anchor = nullptr;         // keeps the driver's block of small allocations, which wait_for_device takes from
};
DevicePool g_pools[kPoolDevices];

}  // namespace

void pool_open(int device) {
  if (device < 0 || device >= kPoolDevices) return;
  DevicePool& p = g_pools[device];
  std::lock_guard<std::mutex> lk(p.mu);
  if (p.users++ > 0) return;
  int supported = 0;
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = device;
  unsigned long long keep = kPoolKeep;
  if (cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, device) == cudaSuccess && supported &&
      cudaStreamCreateWithFlags(&p.stream, cudaStreamNonBlocking) == cudaSuccess &&
      cudaMemPoolCreate(&p.pool, &props) == cudaSuccess &&
      cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess) {
    if (cudaMalloc(&p.anchor, 256) != cudaSuccess) {
      cudaGetLastError();
      p.anchor = nullptr;
    }
    return;
  }
  // no pool here: cudaMalloc serves the buffers
  cudaGetLastError();
  if (p.pool) cudaMemPoolDestroy(p.pool);
  if (p.stream) cudaStreamDestroy(p.stream);
  p.pool = nullptr;
  p.stream = nullptr;
}

void pool_close(int device) {
  if (device < 0 || device >= kPoolDevices) return;
  DevicePool& p = g_pools[device];
  std::lock_guard<std::mutex> lk(p.mu);
  if (--p.users > 0) return;
  if (p.stream) cudaStreamSynchronize(p.stream);
  if (p.anchor) cudaFree(p.anchor);
  p.anchor = nullptr;
  if (p.pool) cudaMemPoolDestroy(p.pool);
  if (p.stream) cudaStreamDestroy(p.stream);
  p.pool = nullptr;
  p.stream = nullptr;
}

cudaError_t DevBuf::reserve(size_t bytes) {
  if (bytes <= cap && ptr) return cudaSuccess;
  if (ptr) release();
  const size_t want = std::max<size_t>(bytes, 256);
  int dev = -1;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kPoolDevices) {
    DevicePool& p = g_pools[dev];
    std::lock_guard<std::mutex> lk(p.mu);
    if (p.pool) {
      // complete before any other stream can be given the pointer
      cudaError_t e = cudaMallocFromPoolAsync(&ptr, want, p.pool, p.stream);
      if (e == cudaSuccess) e = cudaStreamSynchronize(p.stream);
      if (e != cudaSuccess) { ptr = nullptr; return e; }
      cap = want;
      device = dev;
      return cudaSuccess;
    }
  }
  cudaError_t e = cudaMalloc(&ptr, want);
  if (e != cudaSuccess) { ptr = nullptr; return e; }
  cap = want;
  device = -1;
  return cudaSuccess;
}

namespace {

// Waits for the device's work, as a cudaFree of a buffer does: any stream of any
// context may still use pool memory that is given back.  By a cudaFree (5 us with
// its cudaMalloc, 500 without the pool's anchor): cudaDeviceSynchronize is refused
// while another thread captures a stream, and ends that capture.
void wait_for_device(int device) {
  int now = device;
  cudaGetDevice(&now);
  if (now != device) cudaSetDevice(device);
  void* p = nullptr;
  if (cudaMalloc(&p, 256) == cudaSuccess) {
    cudaFree(p);
  } else {
    cudaGetLastError();
    cudaDeviceSynchronize();
  }
  if (now != device) cudaSetDevice(now);
}

void give_back(DevBuf& b) {
  if (b.ptr && b.device >= 0) {
    DevicePool& p = g_pools[b.device];
    std::lock_guard<std::mutex> lk(p.mu);
    if (p.pool) cudaFreeAsync(b.ptr, p.stream);
    else cudaFree(b.ptr);  // the pool went with its last context; its memory goes back here
  } else if (b.ptr) {
    cudaFree(b.ptr);
  }
  b = DevBuf{};
}

}  // namespace

void release_all(std::initializer_list<DevBuf*> bufs) {
  int waited = -1;
  for (DevBuf* b : bufs) {
    if (b->ptr && b->device >= 0 && b->device != waited) wait_for_device(waited = b->device);
    give_back(*b);
  }
}

void DevBuf::release() { release_all({this}); }

namespace {

struct Box { float mn[3], mx[3]; };

__device__ __forceinline__ Box tri_box(const rm_triangle& t) {
  Box b;
  b.mn[0] = fminf(t.v0.x, fminf(t.v1.x, t.v2.x)); b.mx[0] = fmaxf(t.v0.x, fmaxf(t.v1.x, t.v2.x));
  b.mn[1] = fminf(t.v0.y, fminf(t.v1.y, t.v2.y)); b.mx[1] = fmaxf(t.v0.y, fmaxf(t.v1.y, t.v2.y));
  b.mn[2] = fminf(t.v0.z, fminf(t.v1.z, t.v2.z)); b.mx[2] = fmaxf(t.v0.z, fmaxf(t.v1.z, t.v2.z));
  return b;
}
__device__ __forceinline__ void grow(Box& a, const Box& b) {
  for (int k = 0; k < 3; ++k) { a.mn[k] = fminf(a.mn[k], b.mn[k]); a.mx[k] = fmaxf(a.mx[k], b.mx[k]); }
}
__device__ __forceinline__ Box empty_box() {
  Box b;
  for (int k = 0; k < 3; ++k) { b.mn[k] = __int_as_float(0x7f800000); b.mx[k] = -__int_as_float(0x7f800000); }
  return b;
}

// Slot boxes live in the first three float4 of a record (see rm_device.cuh).
__device__ __forceinline__ void write_slot(float4* rec, int slot, const Box& b) {
  float* f = reinterpret_cast<float*>(rec);
  if (slot == 0) { f[0] = b.mn[0]; f[1] = b.mx[0]; f[2] = b.mn[1]; f[3] = b.mx[1]; f[8] = b.mn[2]; f[9] = b.mx[2]; }
  else { f[4] = b.mn[0]; f[5] = b.mx[0]; f[6] = b.mn[1]; f[7] = b.mx[1]; f[10] = b.mn[2]; f[11] = b.mx[2]; }
}
__device__ __forceinline__ Box read_slot_cg(const float4* rec, int slot) {
  const float4 a = __ldcg(rec + slot), c = __ldcg(rec + 2);
  Box b;
  b.mn[0] = a.x; b.mx[0] = a.y; b.mn[1] = a.z; b.mx[1] = a.w;
  if (slot == 0) { b.mn[2] = c.x; b.mx[2] = c.y; } else { b.mn[2] = c.z; b.mx[2] = c.w; }
  return b;
}

__global__ void k_pack_tgeo(const rm_triangle* __restrict__ tris, const int32_t* __restrict__ order, int n,
                            float4* __restrict__ tgeo) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  pack_record(tris[order[i]], order[i], tgeo + size_t(i) * 3);
}

// Refit: one thread per record; leaf slots are boxed from their triangles,
// then the last child to arrive at a record carries the union upward.
__global__ void k_refit(const rm_triangle* __restrict__ tris, const int32_t* __restrict__ order, float4* recs,
                        const int32_t* __restrict__ parents, int* counters, int n_records) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_records) return;
  float4* rec = recs + size_t(i) * 4;
  const int4 d = *reinterpret_cast<const int4*>(rec + 3);
  int ready = 0;
  for (int slot = 0; slot < 2; ++slot) {
    const int cnt = slot ? d.w : d.z, link = slot ? d.y : d.x;
    if (cnt < 0) { ++ready; continue; }
    if (cnt == 0) continue;
    Box b = empty_box();
    for (int k = 0; k < cnt; ++k) grow(b, tri_box(tris[order[link + k]]));
    write_slot(rec, slot, b);
    ++ready;
  }
  if (ready == 0) return;
  __threadfence();
  int node = i;
  int add = ready;
  for (;;) {
    const int old = atomicAdd(counters + node, add);
    if (old + add < 2) return;  // the other child is still on its way
    __threadfence();
    const int pr = parents[node];
    if (pr < 0) return;
    float4* nrec = recs + size_t(node) * 4;
    const int4 nd = __ldcg(reinterpret_cast<const int4*>(nrec + 3));
    Box b = empty_box();
    if (nd.z >= 0) grow(b, read_slot_cg(nrec, 0));
    if (nd.w >= 0) grow(b, read_slot_cg(nrec, 1));
    write_slot(recs + size_t(pr >> 1) * 4, pr & 1, b);
    __threadfence();
    node = pr >> 1;
    add = 1;
  }
}

// ---- LBVH -------------------------------------------------------------------

__device__ __forceinline__ unsigned int ordered(float f) {
  unsigned int u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unordered(unsigned int u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// Six atomics per block: as one set per warp over a full grid, the atomics on
// six words took 20 us whatever the size (1,000 triangles included).
__global__ void __launch_bounds__(256) k_centroid_bounds(const rm_triangle* __restrict__ tris, int n,
                                                         unsigned int* bounds) {
  __shared__ unsigned int sh[6];
  unsigned int mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0, 0, 0};
  if (threadIdx.x < 6) sh[threadIdx.x] = threadIdx.x < 3 ? 0xffffffffu : 0u;
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const rm_triangle& t = tris[i];
    const float c[3] = {t.v0.x + t.v1.x + t.v2.x, t.v0.y + t.v1.y + t.v2.y, t.v0.z + t.v1.z + t.v2.z};
    for (int k = 0; k < 3; ++k) { mn[k] = min(mn[k], ordered(c[k])); mx[k] = max(mx[k], ordered(c[k])); }
  }
  for (int k = 0; k < 3; ++k) {
    mn[k] = __reduce_min_sync(0xffffffffu, mn[k]);
    mx[k] = __reduce_max_sync(0xffffffffu, mx[k]);
  }
  if ((threadIdx.x & 31) == 0)
    for (int k = 0; k < 3; ++k) { atomicMin(sh + k, mn[k]); atomicMax(sh + 3 + k, mx[k]); }
  __syncthreads();
  if (threadIdx.x < 3) atomicMin(bounds + threadIdx.x, sh[threadIdx.x]);
  else if (threadIdx.x < 6) atomicMax(bounds + threadIdx.x, sh[threadIdx.x]);
}

static inline unsigned bounds_blocks(int n) { return unsigned(std::min(148 * 4, (n + 1023) / 1024)); }

__device__ __forceinline__ unsigned int expand_bits(unsigned int v) {
  v = (v * 0x00010001u) & 0xFF0000FFu;
  v = (v * 0x00000101u) & 0x0F00F00Fu;
  v = (v * 0x00000011u) & 0xC30C30C3u;
  v = (v * 0x00000005u) & 0x49249249u;
  return v;
}

// 30-bit Morton code of a centroid (times three) in the bounds.
__device__ __forceinline__ unsigned int morton_code(const float* c, const unsigned int* bounds) {
  unsigned int q[3];
  for (int k = 0; k < 3; ++k) {
    const float lo = unordered(bounds[k]), hi = unordered(bounds[3 + k]);
    const float span = hi - lo;
    float f = span > 0.0f ? (c[k] - lo) / span : 0.5f;
    f = fminf(fmaxf(f, 0.0f), 1.0f);
    q[k] = min(unsigned(f * 1024.0f), 1023u);
  }
  return (expand_bits(q[0]) << 2) | (expand_bits(q[1]) << 1) | expand_bits(q[2]);
}

__global__ void k_morton(const rm_triangle* __restrict__ tris, int n, const unsigned int* __restrict__ bounds,
                         unsigned int* __restrict__ keys, int* __restrict__ vals) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const rm_triangle& t = tris[i];
  const float c[3] = {t.v0.x + t.v1.x + t.v2.x, t.v0.y + t.v1.y + t.v2.y, t.v0.z + t.v1.z + t.v2.z};
  keys[i] = morton_code(c, bounds);
  vals[i] = i;
}

// Common-prefix length of keys i and j, with the sorted position breaking
// ties between equal codes (Karras 2012, section 4).
__device__ __forceinline__ int delta(const unsigned int* keys, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  const unsigned int a = keys[i], b = keys[j];
  if (a != b) return __clz(a ^ b);
  return 32 + __clz(unsigned(i) ^ unsigned(j));
}

struct KarrasNode {
  int left, right;  // child index
  bool left_leaf, right_leaf;
  int first, last;  // range of sorted positions
};

// Internal node i of n-1 (Karras 2012, algorithm 1); keys in global or shared memory.
__device__ __forceinline__ KarrasNode karras_node(const unsigned int* keys, int n, int i) {
  const int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
  const int dmin = delta(keys, n, i, i - d);
  int lmax = 2;
  while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t >= 1; t >>= 1)
    if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
  const int j = i + l * d;
  const int dnode = delta(keys, n, i, j);
  int s = 0;
  for (int t = (l + 1) >> 1;; t = (t + 1) >> 1) {
    if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    if (t == 1) break;
  }
  const int gamma = i + s * d + min(d, 0);
  KarrasNode k;
  k.first = min(i, j);
  k.last = max(i, j);
  k.left = gamma;
  k.right = gamma + 1;
  k.left_leaf = k.first == gamma;
  k.right_leaf = k.last == gamma + 1;
  return k;
}

// Children encoded as (index << 1) | is_leaf; ranges.
__global__ void k_karras(const unsigned int* __restrict__ keys, int n, int2* __restrict__ children,
                         int2* __restrict__ ranges, int* __restrict__ parent_int, int* __restrict__ parent_leaf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  const KarrasNode k = karras_node(keys, n, i);
  children[i] = make_int2((k.left << 1) | int(k.left_leaf), (k.right << 1) | int(k.right_leaf));
  ranges[i] = make_int2(k.first, k.last);
  if (k.left_leaf) parent_leaf[k.left] = i; else parent_int[k.left] = i;
  if (k.right_leaf) parent_leaf[k.right] = i; else parent_int[k.right] = i;
}

// Boxes of the Karras tree, bottom-up from the leaves; the sorted triangle
// order is vals[].  kbox: (n-1) internal boxes.
__global__ void k_karras_boxes(const rm_triangle* __restrict__ tris, const int* __restrict__ order, int n,
                               const int2* __restrict__ children, const int* __restrict__ parent_int,
                               const int* __restrict__ parent_leaf, Box* kbox, int* kcount) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int node = parent_leaf[i];
  while (node >= 0) {
    __threadfence();
    if (atomicAdd(kcount + node, 1) == 0) return;  // first arrival waits for the sibling
    __threadfence();
    const int2 ch = children[node];
    Box b = empty_box();
    for (int k = 0; k < 2; ++k) {
      const int c = k ? ch.y : ch.x;
      if (c & 1) grow(b, tri_box(tris[order[c >> 1]]));
      else {
        const Box* src = kbox + (c >> 1);
        Box cb;
        for (int q = 0; q < 3; ++q) { cb.mn[q] = __ldcg(&src->mn[q]); cb.mx[q] = __ldcg(&src->mx[q]); }
        grow(b, cb);
      }
    }
    kbox[node] = b;
    node = node == 0 ? -1 : parent_int[node];
  }
}

// Child-pair records from the Karras tree: record index = Karras index;
// children with at most leaf_max triangles become leaves.
__global__ void k_emit_records(const rm_triangle* __restrict__ tris, const int* __restrict__ order, int n,
                               int leaf_max, const int2* __restrict__ children, const int2* __restrict__ ranges,
                               const Box* __restrict__ kbox, float4* recs, int* parents) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  float4* rec = recs + size_t(i) * 4;
  const int2 ch = children[i];
  int links[2], counts[2];
  for (int k = 0; k < 2; ++k) {
    const int c = k ? ch.y : ch.x;
    Box b;
    if (c & 1) {
      b = tri_box(tris[order[c >> 1]]);
      links[k] = c >> 1; counts[k] = 1;
    } else {
      const int2 r = ranges[c >> 1];
      b = kbox[c >> 1];
      const int size = r.y - r.x + 1;
      if (size <= leaf_max) { links[k] = r.x; counts[k] = size; }
      else { links[k] = c >> 1; counts[k] = 0; parents[c >> 1] = (i << 1) | k; }
    }
    write_slot(rec, k, b);
  }
  rec[3] = make_float4(__int_as_float(links[0]), __int_as_float(links[1]), __int_as_float(counts[0]),
                       __int_as_float(counts[1]));
  if (i == 0) parents[0] = -1;
}

// The whole LBVH of a small scene in one block, for the no-allocation query,
// whose cost at a thousand triangles was its launches: bounds, codes, sort, tree
// and boxes ran as 17 kernels of 4 to 43 us (the boxes' climb, a fence and an
// atomic in L2 per level, the longest).  Here the triangles are read once into
// registers; the centroid bounds, the Morton codes, a bitonic sort of (code,
// triangle) - the order the stable radix sort gives - and the keys stay in the
// block (strides below a warp by shuffles); the boxes of every range of sorted
// triangles come from a segment tree in shared memory, so that each internal
// node finds its two children's boxes by itself, without a climb (the climb in
// shared memory took 11 of 65 thousand cycles, the sort through shared memory
// alone 19).  The records are those of the multi-kernel build.  4-wide nodes
// instead (each node's internal children opened once, in the same pass)
// traced 4,096 rays in 18.7 against 21.6 us and built in 30 against 25.
constexpr int kSmallTris = 2048;

struct SmallLbvh {
  unsigned long long sorted[kSmallTris];  // code << 32 | triangle
  unsigned int keys[kSmallTris];
  int position[kSmallTris];   // sorted position of a triangle
  Box tree[2 * kSmallTris];   // segment tree over the sorted triangles' boxes: leaf i at m + i
  unsigned int bounds[6];
};

__device__ __forceinline__ unsigned long long shfl_xor_u64(unsigned long long v, int m) {
  const unsigned lo = __shfl_xor_sync(0xffffffffu, unsigned(v), m);
  const unsigned hi = __shfl_xor_sync(0xffffffffu, unsigned(v >> 32), m);
  return ((unsigned long long)hi << 32) | lo;
}

// Box of the sorted positions [first, last] from a segment tree of m leaves.
__device__ __forceinline__ Box range_box(const Box* tree, int m, int first, int last) {
  Box b = empty_box();
  for (int l = first + m, r = last + m + 1; l < r; l >>= 1, r >>= 1) {
    if (l & 1) grow(b, tree[l++]);
    if (r & 1) grow(b, tree[--r]);
  }
  return b;
}

__global__ void __launch_bounds__(1024) k_lbvh_small(const rm_triangle* __restrict__ tris, int n, int leaf_max,
                                                     float4* __restrict__ recs, float4* __restrict__ tgeo,
                                                     uint32_t* err_word) {
  extern __shared__ __align__(16) unsigned char small_lbvh[];
  SmallLbvh& sh = *reinterpret_cast<SmallLbvh*>(small_lbvh);
  constexpr int kPer = kSmallTris / 1024;
  const int tid = int(threadIdx.x);
  if (tid == 0) *err_word = 0u;
  if (tid < 6) sh.bounds[tid] = tid < 3 ? 0xffffffffu : 0u;
  float v[kPer][9], c[kPer][3];
  unsigned int mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0, 0, 0};
  // the nine vertex floats of a 176-byte record: three 128-bit loads when the
  // caller's array is aligned for them (the scalar loads of a warp touch 32
  // lines nine times)
  const bool wide = (reinterpret_cast<uintptr_t>(tris) & 15u) == 0;
#pragma unroll
  for (int r = 0; r < kPer; ++r) {
    const int j = tid + 1024 * r;
    if (j >= n) continue;
    const rm_triangle& t = tris[j];
    if (wide) {
      const float4* q = reinterpret_cast<const float4*>(&t);
      const float4 a = q[0], b = q[1], d = q[2];
      v[r][0] = a.x; v[r][1] = a.y; v[r][2] = a.z; v[r][3] = a.w;
      v[r][4] = b.x; v[r][5] = b.y; v[r][6] = b.z; v[r][7] = b.w;
      v[r][8] = d.x;
    } else {
      v[r][0] = t.v0.x; v[r][1] = t.v0.y; v[r][2] = t.v0.z;
      v[r][3] = t.v1.x; v[r][4] = t.v1.y; v[r][5] = t.v1.z;
      v[r][6] = t.v2.x; v[r][7] = t.v2.y; v[r][8] = t.v2.z;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      c[r][k] = v[r][k] + v[r][3 + k] + v[r][6 + k];
      mn[k] = min(mn[k], ordered(c[r][k]));
      mx[k] = max(mx[k], ordered(c[r][k]));
    }
  }
  for (int k = 0; k < 3; ++k) {
    mn[k] = __reduce_min_sync(0xffffffffu, mn[k]);
    mx[k] = __reduce_max_sync(0xffffffffu, mx[k]);
  }
  __syncthreads();
  if ((tid & 31) == 0 && tid < n)
    for (int k = 0; k < 3; ++k) { atomicMin(sh.bounds + k, mn[k]); atomicMax(sh.bounds + 3 + k, mx[k]); }
  __syncthreads();
  int m = 32;
  while (m < n) m <<= 1;
  // element tid + 1024 r in e[r]
  unsigned long long e[kPer];
#pragma unroll
  for (int r = 0; r < kPer; ++r) {
    const int j = tid + 1024 * r;
    e[r] = j < n ? ((unsigned long long)(morton_code(c[r], sh.bounds)) << 32) | unsigned(j) : ~0ull;
  }
  for (int size = 2; size <= m; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (stride >= 1024) {  // both elements of a pair in this thread (size 2048: ascending)
        if (e[0] > e[kPer - 1]) { const unsigned long long t = e[0]; e[0] = e[kPer - 1]; e[kPer - 1] = t; }
        continue;
      }
      if (stride >= 32) {
#pragma unroll
        for (int r = 0; r < kPer; ++r)
          if (tid + 1024 * r < m) sh.sorted[tid + 1024 * r] = e[r];
        __syncthreads();
      }
#pragma unroll
      for (int r = 0; r < kPer; ++r) {
        const int i = tid + 1024 * r;
        const unsigned long long o =
            stride >= 32 ? (i < m ? sh.sorted[i ^ stride] : ~0ull) : shfl_xor_u64(e[r], stride);
        const bool low = (i & stride) == 0, up = (i & size) == 0;
        if ((o < e[r]) == (low == up)) e[r] = o;
      }
      if (stride >= 32) __syncthreads();
    }
#pragma unroll
  for (int r = 0; r < kPer; ++r) {
    const int i = tid + 1024 * r;
    if (i < n) {
      sh.keys[i] = unsigned(e[r] >> 32);
      sh.position[unsigned(e[r])] = i;
    } else if (i < m) {
      sh.tree[m + i] = empty_box();
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kPer; ++r) {
    const int j = tid + 1024 * r;
    if (j >= n) continue;
    const int pos = sh.position[j];
    float4* g = tgeo + size_t(pos) * 3;
    g[0] = make_float4(v[r][0], v[r][1], v[r][2], __int_as_float(j));
    g[1] = make_float4(v[r][3] - v[r][0], v[r][4] - v[r][1], v[r][5] - v[r][2], 0.f);
    g[2] = make_float4(v[r][6] - v[r][0], v[r][7] - v[r][1], v[r][8] - v[r][2], 0.f);
    Box b;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      b.mn[k] = fminf(v[r][k], fminf(v[r][3 + k], v[r][6 + k]));
      b.mx[k] = fmaxf(v[r][k], fmaxf(v[r][3 + k], v[r][6 + k]));
    }
    sh.tree[m + pos] = b;
  }
  __syncthreads();
  for (int w = m >> 1; w >= 1; w >>= 1) {
    for (int k = tid; k < w; k += 1024) {
      Box b = sh.tree[2 * (w + k)];
      grow(b, sh.tree[2 * (w + k) + 1]);
      sh.tree[w + k] = b;
    }
    __syncthreads();
  }
  for (int i = tid; i < n - 1; i += 1024) {
    const KarrasNode k = karras_node(sh.keys, n, i);
    const int ln = k.left - k.first + 1, rn = k.last - k.right + 1;  // triangles of the children
    const Box a = range_box(sh.tree, m, k.first, k.left), b = range_box(sh.tree, m, k.right, k.last);
    const bool lleaf = ln <= leaf_max, rleaf = rn <= leaf_max;
    float4* rec = recs + size_t(i) * 4;
    rec[0] = make_float4(a.mn[0], a.mx[0], a.mn[1], a.mx[1]);
    rec[1] = make_float4(b.mn[0], b.mx[0], b.mn[1], b.mx[1]);
    rec[2] = make_float4(a.mn[2], a.mx[2], b.mn[2], b.mx[2]);
    rec[3] = make_float4(__int_as_float(lleaf ? k.first : k.left), __int_as_float(k.right),
                         __int_as_float(lleaf ? ln : 0), __int_as_float(rleaf ? rn : 0));
  }
}

// Depth of each leaf slot (for the traversal stack bound).
__global__ void k_depth(const float4* __restrict__ recs, const int* __restrict__ parents, int n_records, int* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_records) return;
  const int4 d = *reinterpret_cast<const int4*>(recs + size_t(i) * 4 + 3);
  if (d.z <= 0 && d.w <= 0) return;
  int depth = 1, node = i, guard = 0;
  while (parents[node] >= 0 && guard < 4096) { node = parents[node] >> 1; ++depth; ++guard; }
  atomicMax(out, depth);
}

__global__ void k_single_leaf(const rm_triangle* __restrict__ tris, int n, float4* rec, int* parents, int* order) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  Box b = empty_box();
  for (int i = 0; i < n; ++i) { grow(b, tri_box(tris[i])); order[i] = i; }
  write_slot(rec, 0, b);
  write_slot(rec, 1, empty_box());
  rec[3] = make_float4(__int_as_float(0), __int_as_float(0), __int_as_float(n), __int_as_float(-1));
  parents[0] = -1;
}

__global__ void k_hash(const unsigned long long* __restrict__ w, size_t n, unsigned long long* out) {
  unsigned long long acc = 0;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
    unsigned long long z = w[i] ^ (0x9E3779B97F4A7C15ull * (i + 1));
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    acc += z ^ (z >> 31);
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, acc);
}

// flag[0] |= 1 where the two word arrays differ.
__global__ void k_differ(const uint4* __restrict__ a, const uint4* __restrict__ b, size_t n, int* flag) {
  bool d = false;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
    const uint4 x = a[i], y = b[i];
    d |= (x.x != y.x) | (x.y != y.y) | (x.z != y.z) | (x.w != y.w);
  }
  if (__any_sync(0xffffffffu, d) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

// What upload_scene asks of every triangle before it is used (see check_triangles).
__global__ void __launch_bounds__(256) k_check_triangles(const rm_triangle* __restrict__ tris, int n,
                                                         long long n_texels, int* flags) {
  int f = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const rm_triangle& t = tris[i];
    if (!(t.alpha >= 1.0f)) f |= 1;
    if (t.texture_offset >= 0 &&
        (t.texture_width <= 0 || t.texture_height <= 0 ||
         (long long)t.texture_offset + (long long)t.texture_width * t.texture_height > n_texels))
      f |= 2;
  }
  f = __reduce_or_sync(0xffffffffu, f);
  if ((threadIdx.x & 31) == 0 && f) atomicOr(flags, f);
}

__global__ void k_light_records(const rm_triangle* __restrict__ tris, const int32_t* __restrict__ lights, int n,
                                float4* __restrict__ rec) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const rm_triangle& t = tris[lights[i]];
  rec[size_t(i) * 4 + 0] = make_float4(t.v0.x, t.v0.y, t.v0.z, t.er);
  rec[size_t(i) * 4 + 1] = make_float4(t.v1.x, t.v1.y, t.v1.z, t.eg);
  rec[size_t(i) * 4 + 2] = make_float4(t.v2.x, t.v2.y, t.v2.z, t.eb);
  rec[size_t(i) * 4 + 3] = make_float4(t.nn.x, t.nn.y, t.nn.z, t.alpha);
}

// guide[g] = first index with cdf >= g * step (the last index if none);
// guide[G] = L - 1.
__global__ void k_light_guide(const float* __restrict__ cdf, int L, int G, float step, int32_t* __restrict__ guide) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g > G) return;
  if (g == G) { guide[g] = L - 1; return; }
  const float th = float(g) * step;
  int lo = 0, hi = L - 1;
  while (lo < hi) {
    int mid = (lo + hi) / 2;
    if (cdf[mid] >= th) hi = mid; else lo = mid + 1;
  }
  guide[g] = lo;
}

}  // namespace

cudaError_t prepare_lights(const rm_triangle* d_tris, const int32_t* d_lights, const float* d_cdf, int n_lights,
                           float light_total, DevBuf& rec, DevBuf& guide, int& guide_n, float& guide_inv,
                           cudaStream_t st) {
  guide_n = 0;
  guide_inv = 0.0f;
  if (n_lights <= 0 || !(light_total > 1e-12f)) return cudaSuccess;
  RM_TRY_(rec.reserve(size_t(n_lights) * 4 * sizeof(float4)));
  k_light_records<<<(n_lights + 255) / 256, 256, 0, st>>>(d_tris, d_lights, n_lights, rec.as<float4>());
  int G = 1;
  while (G < n_lights && G < 65536) G <<= 1;
  RM_TRY_(guide.reserve(size_t(G + 1) * sizeof(int32_t)));
  const float step = light_total / float(G);
  k_light_guide<<<(G + 1 + 255) / 256, 256, 0, st>>>(d_cdf, n_lights, G, step, guide.as<int32_t>());
  guide_n = G;
  guide_inv = float(G) / light_total;
  return cudaGetLastError();
}

namespace {

}  // namespace

cudaError_t pack_tgeo(const rm_triangle* d_tris, DevBvh& bvh, cudaStream_t st) {
  if (bvh.n_tris <= 0) return cudaSuccess;
  cudaError_t e = bvh.tgeo.reserve(size_t(bvh.n_tris) * 3 * sizeof(float4));
  if (e != cudaSuccess) return e;
  k_pack_tgeo<<<(bvh.n_tris + 255) / 256, 256, 0, st>>>(d_tris, bvh.order.as<int32_t>(), bvh.n_tris,
                                                       bvh.tgeo.as<float4>());
  return cudaGetLastError();
}

cudaError_t refit_bvh(const rm_triangle* d_tris, DevBvh& bvh, cudaStream_t st) {
  if (bvh.n_records <= 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(bvh.counters.ptr, 0, size_t(bvh.n_records) * sizeof(int), st);
  if (e != cudaSuccess) return e;
  k_refit<<<(bvh.n_records + 255) / 256, 256, 0, st>>>(d_tris, bvh.order.as<int32_t>(), bvh.records.as<float4>(),
                                                       bvh.parents.as<int32_t>(), bvh.counters.as<int>(),
                                                       bvh.n_records);
  e = cudaGetLastError();
  return e == cudaSuccess ? refit_last(d_tris, bvh, st) : e;
}

cudaError_t check_triangles(const rm_triangle* d_tris, int n, long long n_texels, int* d_flags, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(d_flags, 0, sizeof(int), st);
  if (e != cudaSuccess || n <= 0) return e;
  k_check_triangles<<<unsigned(std::min(148 * 4, (n + 255) / 256)), 256, 0, st>>>(d_tris, n, n_texels, d_flags);
  return cudaGetLastError();
}

cudaError_t device_differ(const void* a, const void* b, size_t n_bytes, int* d_flag, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(d_flag, 0, sizeof(int), st);
  if (e != cudaSuccess || n_bytes == 0) return e;
  if (n_bytes % 16) return cudaErrorInvalidValue;
  k_differ<<<148 * 4, 256, 0, st>>>(static_cast<const uint4*>(a), static_cast<const uint4*>(b), n_bytes / 16, d_flag);
  return cudaGetLastError();
}

cudaError_t device_hash(const void* d_bytes, size_t n_bytes, unsigned long long* d_out, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(d_out, 0, sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  size_t words = n_bytes / 8;
  if (words == 0) return cudaSuccess;
  k_hash<<<148 * 4, 256, 0, st>>>(static_cast<const unsigned long long*>(d_bytes), words, d_out);
  return cudaGetLastError();
}

#define RM_TRY(x)                          \
  do {                                     \
    cudaError_t e_ = (x);                  \
    if (e_ != cudaSuccess) return e_;      \
  } while (0)

cudaError_t build_lbvh(const rm_triangle* d_tris, int n, int leaf_max, DevBvh& b, cudaStream_t st, std::string& err) {
  b.n_tris = n;
  b.max_depth = 0;
  if (n <= 0) { b.n_records = 0; return cudaSuccess; }
  leaf_max = std::max(1, std::min(leaf_max, kMaxLeaf));
  if (n >= kMaxLink) { err = "scene exceeds 16777215 triangles"; return cudaErrorInvalidValue; }
  RM_TRY(b.order.reserve(size_t(n) * sizeof(int)));
  if (n <= leaf_max) {
    b.n_records = 1;
    RM_TRY(b.records.reserve(4 * sizeof(float4)));
    RM_TRY(b.parents.reserve(sizeof(int)));
    RM_TRY(b.counters.reserve(sizeof(int)));
    k_single_leaf<<<1, 1, 0, st>>>(d_tris, n, b.records.as<float4>(), b.parents.as<int>(), b.order.as<int>());
    RM_TRY(cudaGetLastError());
    b.max_depth = 1;
    b.shared = false;
    b.tree = true;
    b.leaf_tris = n;
    RM_TRY(build_quads(b, st));
    return pack_tgeo(d_tris, b, st);
  }
  const int ni = n - 1;
  RM_TRY(b.bounds.reserve(6 * sizeof(unsigned int)));
  RM_TRY(b.keys.reserve(size_t(n) * 4 * 2));
  RM_TRY(b.keys_alt.reserve(size_t(n) * 4));
  RM_TRY(b.vals_alt.reserve(size_t(n) * 4));
  RM_TRY(b.knodes.reserve(size_t(ni) * sizeof(int2) * 2));  // children + ranges
  RM_TRY(b.ranges.reserve(size_t(ni) * sizeof(int) + size_t(n) * sizeof(int)));  // parent_int + parent_leaf
  RM_TRY(b.kbox.reserve(size_t(ni) * sizeof(Box)));
  RM_TRY(b.kcount.reserve(size_t(ni) * sizeof(int)));
  RM_TRY(b.records.reserve(size_t(ni) * 4 * sizeof(float4)));
  RM_TRY(b.parents.reserve(size_t(ni) * sizeof(int)));
  RM_TRY(b.counters.reserve(size_t(ni) * sizeof(int)));
  RM_TRY(b.depth.reserve(sizeof(int)));
  unsigned int init[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
  RM_TRY(cudaMemcpyAsync(b.bounds.ptr, init, sizeof(init), cudaMemcpyHostToDevice, st));
  k_centroid_bounds<<<bounds_blocks(n), 256, 0, st>>>(d_tris, n, b.bounds.as<unsigned int>());
  unsigned int* keys = b.keys.as<unsigned int>();
  int* vals = reinterpret_cast<int*>(keys + n);
  k_morton<<<(n + 255) / 256, 256, 0, st>>>(d_tris, n, b.bounds.as<unsigned int>(), keys, vals);
  RM_TRY(cudaGetLastError());
  const size_t temp_bytes = radix_sort_temp_bytes(n);
  RM_TRY(b.temp.reserve(temp_bytes));
  bool in_alt = false;
  RM_TRY(radix_sort_pairs(keys, b.keys_alt.as<unsigned int>(), vals, b.vals_alt.as<int>(), n, 30, b.temp.ptr,
                          temp_bytes, in_alt, st));
  const unsigned int* skeys = in_alt ? b.keys_alt.as<unsigned int>() : keys;
  const int* sorder = in_alt ? b.vals_alt.as<int>() : vals;
  RM_TRY(cudaMemcpyAsync(b.order.ptr, sorder, size_t(n) * sizeof(int), cudaMemcpyDeviceToDevice, st));
  int2* children = b.knodes.as<int2>();
  int2* ranges = children + ni;
  int* parent_int = b.ranges.as<int>();
  int* parent_leaf = parent_int + ni;
  RM_TRY(cudaMemsetAsync(parent_int, 0xff, size_t(ni) * sizeof(int), st));
  k_karras<<<(ni + 255) / 256, 256, 0, st>>>(skeys, n, children, ranges, parent_int, parent_leaf);
  RM_TRY(cudaMemsetAsync(b.kcount.ptr, 0, size_t(ni) * sizeof(int), st));
  k_karras_boxes<<<(n + 255) / 256, 256, 0, st>>>(d_tris, b.order.as<int>(), n, children, parent_int, parent_leaf,
                                                  b.kbox.as<Box>(), b.kcount.as<int>());
  RM_TRY(cudaMemsetAsync(b.parents.ptr, 0xff, size_t(ni) * sizeof(int), st));
  k_emit_records<<<(ni + 255) / 256, 256, 0, st>>>(d_tris, b.order.as<int>(), n, leaf_max, children, ranges,
                                                   b.kbox.as<Box>(), b.records.as<float4>(), b.parents.as<int>());
  RM_TRY(cudaGetLastError());
  b.n_records = ni;
  // Records of subtrees that collapsed into a leaf are never reached from the
  // root; they keep parent -1, so refit ends at them and depth counts them as 1.
  RM_TRY(cudaMemsetAsync(b.depth.ptr, 0, sizeof(int), st));
  k_depth<<<(ni + 255) / 256, 256, 0, st>>>(b.records.as<float4>(), b.parents.as<int>(), ni, b.depth.as<int>());
  RM_TRY(cudaMemcpyAsync(&b.max_depth, b.depth.ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
  RM_TRY(cudaStreamSynchronize(st));
  if (b.max_depth > kStack) { err = "device BVH deeper than the traversal stack"; return cudaErrorInvalidValue; }
  b.shared = false;
  b.tree = true;
  b.leaf_tris = n;
  RM_TRY(build_quads(b, st));
  return pack_tgeo(d_tris, b, st);
}

cudaError_t build_lbvh_into(const rm_triangle* d_tris, int n, int leaf_max, const LbvhScratch& w, DevBvhView& out,
                            cudaStream_t st, std::string& err) {
  out.n_records = 0;
  leaf_max = std::max(1, std::min(leaf_max, kMaxLeaf));
  // One block up to kSmallTris triangles (above leaf_max), where the kernels of
  // the large build are mostly launch: the call for 978 triangles and 4,096 rays took 213 us and
  // takes 72, for 1,954 triangles 227 and 92.
  if (n > leaf_max && n <= kSmallTris) {
    RM_TRY(cudaFuncSetAttribute(k_lbvh_small, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(SmallLbvh))));
    k_lbvh_small<<<1, 1024, sizeof(SmallLbvh), st>>>(d_tris, n, leaf_max, w.records, w.tgeo, w.err_word);
    RM_TRY(cudaGetLastError());
    out.n_records = n - 1;
    out.records = w.records;
    out.tgeo = w.tgeo;
    return cudaSuccess;
  }
  // The error word lives in scratch shared by every call: clear it before any
  // early return, or an empty scene would report the last call's overflow.
  RM_TRY(cudaMemsetAsync(w.err_word, 0, sizeof(uint32_t), st));
  if (n <= 0) return cudaSuccess;
  if (n <= leaf_max) {
    k_single_leaf<<<1, 1, 0, st>>>(d_tris, n, w.records, w.parents, w.order);
    RM_TRY(cudaGetLastError());
    out.n_records = 1;
  } else {
    const int ni = n - 1;
    // centroid bounds start at (+max ordered, 0): min slots all ones, max slots zero
    RM_TRY(cudaMemsetAsync(w.bounds, 0xff, 3 * sizeof(unsigned int), st));
    RM_TRY(cudaMemsetAsync(w.bounds + 3, 0, 3 * sizeof(unsigned int), st));
    k_centroid_bounds<<<bounds_blocks(n), 256, 0, st>>>(d_tris, n, w.bounds);
    k_morton<<<(n + 255) / 256, 256, 0, st>>>(d_tris, n, w.bounds, w.keys, w.vals);
    RM_TRY(cudaGetLastError());
    if (radix_sort_temp_bytes(n) > w.sort_temp_bytes) { err = "sort scratch too small"; return cudaErrorInvalidValue; }
    bool in_alt = false;
    RM_TRY(radix_sort_pairs(w.keys, w.keys_alt, w.vals, w.vals_alt, n, 30, w.sort_temp, w.sort_temp_bytes, in_alt,
                            st));
    RM_TRY(cudaMemcpyAsync(w.order, in_alt ? w.vals_alt : w.vals, size_t(n) * sizeof(int), cudaMemcpyDeviceToDevice,
                           st));
    RM_TRY(cudaMemsetAsync(w.parent_int, 0xff, size_t(ni) * sizeof(int), st));
    k_karras<<<(ni + 255) / 256, 256, 0, st>>>(in_alt ? w.keys_alt : w.keys, n, w.children, w.ranges, w.parent_int,
                                               w.parent_leaf);
    RM_TRY(cudaMemsetAsync(w.kcount, 0, size_t(ni) * sizeof(int), st));
    k_karras_boxes<<<(n + 255) / 256, 256, 0, st>>>(d_tris, w.order, n, w.children, w.parent_int, w.parent_leaf,
                                                    reinterpret_cast<Box*>(w.kbox), w.kcount);
    RM_TRY(cudaMemsetAsync(w.parents, 0xff, size_t(ni) * sizeof(int), st));
    k_emit_records<<<(ni + 255) / 256, 256, 0, st>>>(d_tris, w.order, n, leaf_max, w.children, w.ranges,
                                                     reinterpret_cast<const Box*>(w.kbox), w.records, w.parents);
    RM_TRY(cudaGetLastError());
    out.n_records = ni;
  }
  k_pack_tgeo<<<(n + 255) / 256, 256, 0, st>>>(d_tris, w.order, n, w.tgeo);
  RM_TRY(cudaGetLastError());
  out.records = w.records;
  out.tgeo = w.tgeo;
  return cudaSuccess;
}

size_t lbvh_box_bytes() { return sizeof(Box); }

// ---- PLOC ---------------------------------------------------------------------
//
// Meister & Bittner, "Parallel Locally-Ordered Clustering for Bounding Volume
// Hierarchy Construction" (IEEE TVCG 2018).  Clusters start as the triangles in
// Morton order; every iteration each cluster finds, within a window of
// +-kPlocRadius neighbours in that order, the cluster whose union box has the
// smallest surface area; mutual nearest neighbours merge into a new node, and
// the survivors are compacted in order.  Node ids: leaves 0..n-1 (Morton
// position), internal nodes n.. in creation order, so a parent's id is larger
// than its children's.  The tree is then laid out like the LBVH: leaves in
// depth-first order, subtrees of at most `leaf_max` triangles as leaves, one
// child-pair record per remaining internal node (record of node k is
// 2n-2-k, the root is record 0).

namespace {

constexpr int kPlocRadius = 16;

__device__ __forceinline__ float half_area(const float4& lo, const float4& hi) {
  const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
  return dx * dy + dy * dz + dz * dx;
}

struct PlocState {
  int clusters;   // current count
  int next_node;  // id of the next node
  int force;      // the last round merged nothing: merge neighbours (0,1), (2,3), ...
  int side;       // which cluster list is current
  // the round being applied
  int in_clusters, in_side, in_next, merge;
  unsigned int done;  // blocks of k_ploc_round that have counted
};

__global__ void k_ploc_leaves(const rm_triangle* __restrict__ tris, const int* __restrict__ order, int n,
                              float4* __restrict__ blo, float4* __restrict__ bhi, int* __restrict__ cl, PlocState* state) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *state = PlocState{n, n, 0, 0, 0, 0, 0, 0, 0u};
  if (i >= n) return;
  const Box b = tri_box(tris[order[i]]);
  blo[i] = make_float4(b.mn[0], b.mn[1], b.mn[2], __int_as_float(1));
  bhi[i] = make_float4(b.mx[0], b.mx[1], b.mx[2], __int_as_float(-1));
  cl[i] = i;
}

// One round of the clustering is two launches, k_ploc_round and k_ploc_apply,
// that read the cluster count on the device, so rounds are enqueued without
// waiting for it; from kPlocSmall clusters on, one block runs the remaining
// rounds (about half of them) in shared memory.  As nine launches and a
// read-back a round, the 62 rounds of 400,000 triangles took
// 2.7 ms of kernels and 62 waits; now 0.7 ms and one.
constexpr int kPlocTile = 256;
constexpr int kPlocSmall = 2048;

// The nearest neighbour of cluster e of a staged window: lo / hi are the
// window's boxes, w its length.
__device__ __forceinline__ int ploc_nearest(const float4* lo, const float4* hi, int w, int e) {
  const float4 alo = lo[e], ahi = hi[e];
  float best = __int_as_float(0x7f800000);
  int bj = -1;
  const int j0 = max(0, e - kPlocRadius), j1 = min(w - 1, e + kPlocRadius);
  for (int j = j0; j <= j1; ++j) {
    if (j == e) continue;
    const float4 l = lo[j], h = hi[j];
    const float4 ulo = make_float4(fminf(alo.x, l.x), fminf(alo.y, l.y), fminf(alo.z, l.z), 0.f);
    const float4 uhi = make_float4(fmaxf(ahi.x, h.x), fmaxf(ahi.y, h.y), fmaxf(ahi.z, h.z), 0.f);
    const float area = half_area(ulo, uhi);
    if (area < best) { best = area; bj = j; }  // ties keep the smaller index (scanned in order)
  }
  return bj;
}

// The partner cluster i merges with, or -1; the smaller index creates the node.
__device__ __forceinline__ int ploc_force_partner(int i, int C) {
  const int j = (i & 1) ? i - 1 : i + 1;
  return j < C ? j : -1;
}

// Per cluster: its mutual partner (pair[i], -1 for none); per block the nodes it
// creates and the clusters that survive.  The boxes of a tile and of a halo of
// two radii are staged in shared memory, so that the neighbours' own nearest
// neighbours are found here as well.  The last block to finish scans the
// blocks' counts and moves the state on.
__global__ void __launch_bounds__(kPlocTile) k_ploc_round(const int* __restrict__ cl0, const int* __restrict__ cl1,
                                                          const float4* __restrict__ blo,
                                                          const float4* __restrict__ bhi, int* __restrict__ pair,
                                                          int2* block_count, PlocState* st) {
  constexpr int kHalo = 2 * kPlocRadius, kWin = kPlocTile + 2 * kHalo;
  __shared__ float4 lo[kWin], hi[kWin];
  __shared__ int near_[kPlocTile + 2 * kPlocRadius];
  __shared__ int2 warp_sum[kPlocTile / 32];
  __shared__ bool last;
  const int C = st->clusters;
  if (C <= kPlocSmall) {
    if (blockIdx.x == 0 && threadIdx.x == 0) st->merge = 0;  // nothing for k_ploc_apply
    return;
  }
  const int blocks = (C + kPlocTile - 1) / kPlocTile;
  if (int(blockIdx.x) >= blocks) return;
  const int force = st->force;
  const int* cl = st->side ? cl1 : cl0;
  const int tile0 = int(blockIdx.x) * kPlocTile;
  const int i = tile0 + int(threadIdx.x);
  int partner = -1;
  if (force) {
    if (i < C) partner = ploc_force_partner(i, C);
  } else {
    const int w0 = max(0, tile0 - kHalo), w1 = min(C, tile0 + kPlocTile + kHalo);
    for (int k = int(threadIdx.x); k < w1 - w0; k += kPlocTile) {
      const int c = cl[w0 + k];
      lo[k] = blo[c];
      hi[k] = bhi[c];
    }
    __syncthreads();
    const int n0 = max(0, tile0 - kPlocRadius), n1 = min(C, tile0 + kPlocTile + kPlocRadius);
    for (int k = int(threadIdx.x); k < n1 - n0; k += kPlocTile)
      near_[k] = w0 + ploc_nearest(lo, hi, w1 - w0, n0 + k - w0);
    __syncthreads();
    if (i < C) {
      const int j = near_[i - n0];
      if (j >= w0 && near_[j - n0] == i) partner = j;
    }
  }
  if (i < C) pair[i] = partner;
  const int creates = i < C && partner > i ? 1 : 0, stays = i < C && (partner < 0 || partner > i) ? 1 : 0;
  const int2 c = make_int2(__reduce_add_sync(0xffffffffu, creates), __reduce_add_sync(0xffffffffu, stays));
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int2 t = make_int2(0, 0);
    for (int w = 0; w < kPlocTile / 32; ++w) { t.x += warp_sum[w].x; t.y += warp_sum[w].y; }
    block_count[blockIdx.x] = t;
    __threadfence();
    last = atomicAdd(&st->done, 1u) == unsigned(blocks) - 1u;
  }
  __syncthreads();
  if (!last) return;
  // exclusive scan of the blocks' counts, in place
  __threadfence();
  int2 carry = make_int2(0, 0);
  for (int base = 0; base < blocks; base += kPlocTile) {
    const int k = base + int(threadIdx.x);
    int2 v = make_int2(0, 0);
    if (k < blocks) {
      v.x = __ldcg(&block_count[k].x);
      v.y = __ldcg(&block_count[k].y);
    }
    int2 x = v;
    const int lane = int(threadIdx.x & 31), warp = int(threadIdx.x >> 5);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int px = __shfl_up_sync(0xffffffffu, x.x, o), py = __shfl_up_sync(0xffffffffu, x.y, o);
      if (lane >= o) { x.x += px; x.y += py; }
    }
    if (lane == 31) warp_sum[warp] = x;
    __syncthreads();
    int2 before = carry, all = make_int2(0, 0);
    for (int w = 0; w < kPlocTile / 32; ++w) {
      if (w < warp) { before.x += warp_sum[w].x; before.y += warp_sum[w].y; }
      all.x += warp_sum[w].x;
      all.y += warp_sum[w].y;
    }
    if (k < blocks) block_count[k] = make_int2(before.x + x.x - v.x, before.y + x.y - v.y);
    carry.x += all.x;
    carry.y += all.y;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    st->in_clusters = C;
    st->in_side = st->side;
    st->in_next = st->next_node;
    st->merge = carry.x > 0 ? 1 : 0;
    st->done = 0u;
    if (carry.x > 0) {
      st->next_node += carry.x;
      st->clusters = carry.y;
      st->side ^= 1;
      st->force = 0;
    } else {
      st->force = 1;  // degenerate input: pair up neighbours
    }
  }
}

// A node of two clusters.
__device__ __forceinline__ void ploc_merge(int a, int b, int id, int n_leaves, float4* blo, float4* bhi, int2* child,
                                           float4& lo, float4& hi) {
  const float4 al = blo[a], ah = bhi[a], bl = blo[b], bh = bhi[b];
  const int size = __float_as_int(al.w) + __float_as_int(bl.w);
  lo = make_float4(fminf(al.x, bl.x), fminf(al.y, bl.y), fminf(al.z, bl.z), __int_as_float(size));
  hi = make_float4(fmaxf(ah.x, bh.x), fmaxf(ah.y, bh.y), fmaxf(ah.z, bh.z), __int_as_float(-1));
  blo[id] = lo;
  bhi[id] = hi;
  child[id - n_leaves] = make_int2(a, b);
  bhi[a].w = __int_as_float(id);  // parent links
  bhi[b].w = __int_as_float(id);
}

__global__ void __launch_bounds__(kPlocTile) k_ploc_apply(int* __restrict__ cl0, int* __restrict__ cl1,
                                                          const int* __restrict__ pair,
                                                          const int2* __restrict__ block_count, PlocState* st,
                                                          float4* __restrict__ blo, float4* __restrict__ bhi,
                                                          int2* __restrict__ child, int n_leaves) {
  __shared__ int2 warp_sum[kPlocTile / 32];
  const int C = st->in_clusters;
  if (C <= kPlocSmall || !st->merge || int(blockIdx.x) * kPlocTile >= C) return;
  const int* cl = st->in_side ? cl1 : cl0;
  int* ncl = st->in_side ? cl0 : cl1;
  const int i = int(blockIdx.x) * kPlocTile + int(threadIdx.x);
  const int lane = int(threadIdx.x & 31), warp = int(threadIdx.x >> 5);
  const int partner = i < C ? pair[i] : -1;
  const bool creates = i < C && partner > i, stays = i < C && (partner < 0 || partner > i);
  const unsigned cb = __ballot_sync(0xffffffffu, creates), sb = __ballot_sync(0xffffffffu, stays);
  if (lane == 0) warp_sum[warp] = make_int2(__popc(cb), __popc(sb));
  __syncthreads();
  int2 pos = block_count[blockIdx.x];
  for (int w = 0; w < warp; ++w) { pos.x += warp_sum[w].x; pos.y += warp_sum[w].y; }
  pos.x += __popc(cb & ((1u << lane) - 1u));
  pos.y += __popc(sb & ((1u << lane) - 1u));
  if (!stays) return;
  int out = cl[i];
  if (creates) {
    const int id = st->in_next + pos.x;
    float4 lo, hi;
    ploc_merge(out, cl[partner], id, n_leaves, blo, bhi, child, lo, hi);
    out = id;
  }
  ncl[pos.y] = out;
}

// The rounds from kPlocSmall clusters to the root, one block.
struct PlocSmall {
  float4 lo[2][kPlocSmall], hi[2][kPlocSmall];
  int id[2][kPlocSmall];
  int near_[kPlocSmall];
};

__global__ void __launch_bounds__(1024) k_ploc_small(const int* __restrict__ cl0, const int* __restrict__ cl1,
                                                     PlocState* st, float4* __restrict__ blo,
                                                     float4* __restrict__ bhi, int2* __restrict__ child,
                                                     int n_leaves, int* left) {
  extern __shared__ __align__(16) unsigned char ploc_small[];
  PlocSmall& sh = *reinterpret_cast<PlocSmall*>(ploc_small);
  __shared__ int2 warp_sum[32];
  const int tid = int(threadIdx.x), lane = tid & 31, warp = tid >> 5;
  int C = st->clusters, next = st->next_node;
  bool force = st->force != 0;
  if (C > kPlocSmall) {  // not reached yet
    if (tid == 0) *left = C;
    return;
  }
  const int* cl = st->side ? cl1 : cl0;
  for (int i = tid; i < C; i += 1024) {
    const int c = cl[i];
    sh.id[0][i] = c;
    sh.lo[0][i] = blo[c];
    sh.hi[0][i] = bhi[c];
  }
  __syncthreads();
  int cur = 0;
  for (int round = 0; C > 1 && round < 2 * kPlocSmall; ++round) {  // a round merges, or the next one does
    if (!force)
      for (int i = tid; i < C; i += 1024) sh.near_[i] = ploc_nearest(sh.lo[cur], sh.hi[cur], C, i);
    __syncthreads();
    int2 carry = make_int2(0, 0);
    for (int base = 0; base < C; base += 1024) {
      const int i = base + tid;
      int partner = -1;
      if (i < C) {
        if (force) partner = ploc_force_partner(i, C);
        else {
          const int j = sh.near_[i];
          if (j >= 0 && sh.near_[j] == i) partner = j;
        }
      }
      const bool creates = i < C && partner > i, stays = i < C && (partner < 0 || partner > i);
      const unsigned cb = __ballot_sync(0xffffffffu, creates), sb = __ballot_sync(0xffffffffu, stays);
      if (lane == 0) warp_sum[warp] = make_int2(__popc(cb), __popc(sb));
      __syncthreads();
      int2 pos = carry;
      for (int w = 0; w < 32; ++w) {
        const int2 q = warp_sum[w];
        if (w < warp) { pos.x += q.x; pos.y += q.y; }
        carry.x += q.x;
        carry.y += q.y;
      }
      pos.x += __popc(cb & ((1u << lane) - 1u));
      pos.y += __popc(sb & ((1u << lane) - 1u));
      if (stays) {
        const int o = cur ^ 1;
        sh.id[o][pos.y] = sh.id[cur][i];
        sh.lo[o][pos.y] = sh.lo[cur][i];
        sh.hi[o][pos.y] = sh.hi[cur][i];
        if (creates) {
          const int id = next + pos.x;
          float4 lo, hi;
          ploc_merge(sh.id[cur][i], sh.id[cur][partner], id, n_leaves, blo, bhi, child, lo, hi);
          sh.id[o][pos.y] = id;
          sh.lo[o][pos.y] = lo;
          sh.hi[o][pos.y] = hi;
        }
      }
      __syncthreads();
    }
    force = carry.x == 0;
    if (carry.x > 0) {
      next += carry.x;
      C = carry.y;
      cur ^= 1;
    }
    __syncthreads();
  }
  if (tid == 0) *left = C;
}

// Leaf position in depth-first order and depth: walk to the root adding the
// sizes of left siblings.  Only the n leaves walk; max depth -> *depth.  The
// layout kernels leave an unfinished tree (*left clusters, not one) alone.
__global__ void k_ploc_layout(int n, int root, const float4* __restrict__ blo, const float4* __restrict__ bhi,
                              const int2* __restrict__ child, const int* __restrict__ order, int* __restrict__ pos,
                              int* __restrict__ out_order, const int* __restrict__ left, int* __restrict__ depth) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || *left != 1) return;
  int off = 0, d = 1, cur = i;
  while (cur != root) {
    const int p = __float_as_int(bhi[cur].w);
    const int2 c = child[p - n];
    if (c.y == cur) off += __float_as_int(blo[c.x].w);
    cur = p;
    ++d;
    if (d > 4 * kStack) break;  // a corrupt tree cannot loop forever
  }
  pos[i] = off;
  out_order[off] = order[i];
  atomicMax(depth, d);
}

// Depth-first (pre-order) record index of each internal node among the
// internal nodes: one slot per ancestor, plus the internal nodes of every left
// sibling's subtree on the way up (a subtree of s leaves has s - 1).  The
// nearer child of a descent then usually sits in the next record.
__global__ void k_ploc_preorder(int n, int root, const float4* __restrict__ blo, const float4* __restrict__ bhi,
                                const int2* __restrict__ child, const int* __restrict__ left,
                                int* __restrict__ pre) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;  // internal node n + k
  if (k >= n - 1 || *left != 1) return;
  int off = 0, d = 0, cur = n + k;
  while (cur != root) {
    const int p = __float_as_int(bhi[cur].w);
    const int2 c = child[p - n];
    off += 1;
    if (c.y == cur) off += __float_as_int(blo[c.x].w) - 1;
    cur = p;
    if (++d > 4 * kStack) break;  // a corrupt tree cannot loop forever
  }
  pre[k] = off;
}

__device__ __forceinline__ int ploc_first(int node, int n, const int2* __restrict__ child,
                                          const int* __restrict__ pos) {
  while (node >= n) node = child[node - n].x;
  return pos[node];
}

__global__ void k_ploc_emit(int n, int leaf_max, const float4* __restrict__ blo, const float4* __restrict__ bhi,
                            const int2* __restrict__ child, const int* __restrict__ pos, const int* __restrict__ pre,
                            const int* __restrict__ left, float4* recs, int* parents) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;  // internal node n + k
  if (k >= n - 1 || *left != 1) return;
  const int node = n + k;
  const int rec_id = pre[k];
  float4* rec = recs + size_t(rec_id) * 4;
  if (__float_as_int(blo[node].w) <= leaf_max) {
    // collapsed into an ancestor's leaf: an unreachable record
    write_slot(rec, 0, empty_box());
    write_slot(rec, 1, empty_box());
    rec[3] = make_float4(__int_as_float(0), __int_as_float(0), __int_as_float(-1), __int_as_float(-1));
    parents[rec_id] = -1;
    return;
  }
  const int2 ch = child[k];
  int links[2], counts[2];
  for (int s = 0; s < 2; ++s) {
    const int c = s ? ch.y : ch.x;
    const float4 l = blo[c], h = bhi[c];
    Box b;
    b.mn[0] = l.x; b.mn[1] = l.y; b.mn[2] = l.z;
    b.mx[0] = h.x; b.mx[1] = h.y; b.mx[2] = h.z;
    write_slot(rec, s, b);
    const int size = __float_as_int(l.w);
    if (size <= leaf_max) {
      links[s] = ploc_first(c, n, child, pos);
      counts[s] = size;
    } else {
      links[s] = pre[c - n];
      counts[s] = 0;
      parents[links[s]] = (rec_id << 1) | s;
    }
  }
  rec[3] = make_float4(__int_as_float(links[0]), __int_as_float(links[1]), __int_as_float(counts[0]),
                       __int_as_float(counts[1]));
  if (rec_id == 0) parents[0] = -1;
}

}  // namespace

cudaError_t build_ploc(const rm_triangle* d_tris, int n, int leaf_max, DevBvh& b, cudaStream_t st, std::string& err) {
  b.n_tris = n;
  b.max_depth = 0;
  if (n <= 0) { b.n_records = 0; return cudaSuccess; }
  leaf_max = std::max(1, std::min(leaf_max, kMaxLeaf));
  if (n <= leaf_max) return build_lbvh(d_tris, n, leaf_max, b, st, err);  // one leaf
  if (n >= kMaxLink / 2) { err = "scene exceeds 8388607 triangles for the clustering build"; return cudaErrorInvalidValue; }
  const int total = 2 * n - 1;
  // Morton order (shared with the LBVH build)
  RM_TRY(b.order.reserve(size_t(n) * sizeof(int)));
  RM_TRY(b.bounds.reserve(6 * sizeof(unsigned int)));
  RM_TRY(b.keys.reserve(size_t(n) * 4 * 2));
  RM_TRY(b.keys_alt.reserve(size_t(n) * 4));
  RM_TRY(b.vals_alt.reserve(size_t(n) * 4));
  unsigned int init[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
  RM_TRY(cudaMemcpyAsync(b.bounds.ptr, init, sizeof(init), cudaMemcpyHostToDevice, st));
  k_centroid_bounds<<<bounds_blocks(n), 256, 0, st>>>(d_tris, n, b.bounds.as<unsigned int>());
  unsigned int* keys = b.keys.as<unsigned int>();
  int* vals = reinterpret_cast<int*>(keys + n);
  k_morton<<<(n + 255) / 256, 256, 0, st>>>(d_tris, n, b.bounds.as<unsigned int>(), keys, vals);
  RM_TRY(cudaGetLastError());
  const size_t sort_bytes = radix_sort_temp_bytes(n), scan_bytes = exclusive_scan_temp_bytes(n);
  RM_TRY(b.temp.reserve(std::max(sort_bytes, scan_bytes)));
  bool in_alt = false;
  RM_TRY(radix_sort_pairs(keys, b.keys_alt.as<unsigned int>(), vals, b.vals_alt.as<int>(), n, 30, b.temp.ptr,
                          sort_bytes, in_alt, st));
  const int* sorted = in_alt ? b.vals_alt.as<int>() : vals;
  // node and cluster arrays (kbox: box lo/hi; knodes: children; ranges: two cluster lists, pairs, block counts, state)
  const int tiles = (n + kPlocTile - 1) / kPlocTile;
  RM_TRY(b.kbox.reserve(size_t(total) * 2 * sizeof(float4)));
  RM_TRY(b.knodes.reserve(size_t(n) * sizeof(int2)));
  RM_TRY(b.ranges.reserve(size_t(n) * 3 * sizeof(int) + sizeof(int) + size_t(tiles) * sizeof(int2) + sizeof(PlocState)));
  RM_TRY(b.kcount.reserve(size_t(n) * sizeof(int)));
  RM_TRY(b.depth.reserve(2 * sizeof(int)));
  float4* blo = b.kbox.as<float4>();
  float4* bhi = blo + total;
  int2* child = b.knodes.as<int2>();
  int2* block_count = b.ranges.as<int2>();
  PlocState* state = reinterpret_cast<PlocState*>(block_count + tiles);
  int* cl0 = reinterpret_cast<int*>(state + 1);
  int* cl1 = cl0 + n;
  int* pair = cl1 + n;
  k_ploc_leaves<<<(n + 255) / 256, 256, 0, st>>>(d_tris, sorted, n, blo, bhi, cl0, state);
  RM_TRY(cudaGetLastError());
  RM_TRY(cudaFuncSetAttribute(k_ploc_small, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(PlocSmall))));
  // Rounds in batches: a round keeps about two thirds of the clusters, so the
  // first batch usually ends below kPlocSmall; the count read back after it
  // says whether more are needed (launches past the end return at once).
  long long rounds = 0;
  for (int C = n; C > kPlocSmall;) {
    const unsigned g = unsigned((C + kPlocTile - 1) / kPlocTile);
    int batch = 2;
    for (double c = C; c > kPlocSmall; c *= 0.66) ++batch;
    for (int k = 0; k < batch; ++k) {
      k_ploc_round<<<g, kPlocTile, 0, st>>>(cl0, cl1, blo, bhi, pair, block_count, state);
      k_ploc_apply<<<g, kPlocTile, 0, st>>>(cl0, cl1, pair, block_count, state, blo, bhi, child, n);
    }
    RM_TRY(cudaGetLastError());
    if ((rounds += batch) > 8ll * n + 64) { err = "clustering build did not converge"; return cudaErrorInvalidValue; }
    RM_TRY(cudaMemcpyAsync(&C, &state->clusters, sizeof(int), cudaMemcpyDeviceToHost, st));
    RM_TRY(cudaStreamSynchronize(st));
  }
  int* depth = b.depth.as<int>();  // the tree's depth, then the clusters left
  k_ploc_small<<<1, 1024, sizeof(PlocSmall), st>>>(cl0, cl1, state, blo, bhi, child, n, depth + 1);
  RM_TRY(cudaGetLastError());
  const int root = total - 1;
  int* pos = b.kcount.as<int>();
  RM_TRY(cudaMemsetAsync(depth, 0, sizeof(int), st));
  k_ploc_layout<<<(n + 255) / 256, 256, 0, st>>>(n, root, blo, bhi, child, sorted, pos, b.order.as<int>(), depth + 1,
                                                 depth);
  int* pre = pair;  // the cluster arrays are free once the tree is built
  k_ploc_preorder<<<(n - 1 + 255) / 256, 256, 0, st>>>(n, root, blo, bhi, child, depth + 1, pre);
  RM_TRY(b.records.reserve(size_t(n - 1) * 4 * sizeof(float4)));
  RM_TRY(b.parents.reserve(size_t(n - 1) * sizeof(int)));
  RM_TRY(b.counters.reserve(size_t(n - 1) * sizeof(int)));
  k_ploc_emit<<<(n - 1 + 255) / 256, 256, 0, st>>>(n, leaf_max, blo, bhi, child, pos, pre, depth + 1,
                                                   b.records.as<float4>(), b.parents.as<int>());
  RM_TRY(cudaGetLastError());
  int built[2] = {0, 0};
  RM_TRY(cudaMemcpyAsync(built, depth, sizeof(built), cudaMemcpyDeviceToHost, st));
  RM_TRY(cudaStreamSynchronize(st));
  if (built[1] != 1) { err = "clustering build produced a malformed tree"; return cudaErrorInvalidValue; }
  b.max_depth = built[0];
  if (b.max_depth > kStack) { err = "device BVH deeper than the traversal stack"; return cudaErrorInvalidValue; }
  b.n_records = n - 1;
  b.shared = false;
  b.tree = true;
  b.leaf_tris = n;
  RM_TRY(build_quads(b, st));
  return pack_tgeo(d_tris, b, st);
}

bool convert_caller_bvh(const rm_bvh_node* nodes, int M, const int32_t* bvh_tri, int n_tris, DevBvh& out,
                        cudaStream_t st, std::string& err) {
  out.n_tris = n_tris;
  if (M <= 0 || n_tris <= 0) { out.n_records = 0; return true; }
  if (!nodes || !bvh_tri) { err = "BVH nodes without bvh_tri"; return false; }
  if (n_tris >= kMaxLink || M >= kMaxLink) { err = "BVH exceeds 16777215 nodes or triangles"; return false; }
  for (int i = 0; i < n_tris; ++i)
    if (bvh_tri[i] < 0 || bvh_tri[i] >= n_tris) { err = "bvh_tri index out of range"; return false; }
  // record index of each internal node, in node order (parents precede children)
  std::vector<int> rec(size_t(M), -1);
  int n_rec = 0;
  for (int i = 0; i < M; ++i) {
    const rm_bvh_node& s = nodes[i];
    if (s.count > 0) {
      if (s.count > kMaxLeaf || s.offset < 0 || int64_t(s.offset) + s.count > n_tris) {
        err = "BVH leaf range invalid (or more than 255 triangles)";
        return false;
      }
    } else {
      if (s.left <= i || s.right <= i || s.left >= M || s.right >= M) {
        err = "BVH child index invalid (children must follow their parent)";
        return false;
      }
      rec[size_t(i)] = n_rec++;
    }
  }
  const bool root_leaf = nodes[0].count > 0;
  if (root_leaf) n_rec = 1;
  std::vector<float> recs(size_t(n_rec) * 16, 0.0f);
  std::vector<int> parents(size_t(n_rec), -1);
  std::vector<int> depth(size_t(M), 0);
  auto put = [&](int r, int slot, const rm_bvh_node* c, int link, int count) {
    float* f = recs.data() + size_t(r) * 16;
    const float inf = __builtin_inff();
    float mn[3] = {inf, inf, inf}, mx[3] = {-inf, -inf, -inf};
    if (c) { mn[0] = c->mn.x; mn[1] = c->mn.y; mn[2] = c->mn.z; mx[0] = c->mx.x; mx[1] = c->mx.y; mx[2] = c->mx.z; }
    int base = slot ? 4 : 0;
    f[base] = mn[0]; f[base + 1] = mx[0]; f[base + 2] = mn[1]; f[base + 3] = mx[1];
    f[8 + slot * 2] = mn[2]; f[9 + slot * 2] = mx[2];
    int* iv = reinterpret_cast<int*>(f + 12);
    iv[slot] = link;
    iv[2 + slot] = count;
  };
  int max_depth = 1;
  bool shared = false, nested = true;  // (the root's own box is not tested)
  auto ordered_box = [](const rm_bvh_node& c) {
    return c.mn.x <= c.mx.x && c.mn.y <= c.mx.y && c.mn.z <= c.mx.z;
  };
  auto inside = [](const rm_bvh_node& c, const rm_bvh_node& p) {
    return p.mn.x <= c.mn.x && p.mn.y <= c.mn.y && p.mn.z <= c.mn.z && c.mx.x <= p.mx.x && c.mx.y <= p.mx.y &&
           c.mx.z <= p.mx.z;
  };
  long long leaf_tris = 0;
  if (root_leaf) {
    leaf_tris = nodes[0].count;
    put(0, 0, &nodes[0], nodes[0].offset, nodes[0].count);
    put(0, 1, nullptr, 0, -1);
  } else {
    depth[0] = 1;
    for (int i = 0; i < M; ++i) {
      if (nodes[i].count > 0 || rec[size_t(i)] < 0) continue;
      const int r = rec[size_t(i)];
      if (depth[size_t(i)] == 0) continue;  // unreachable from the root
      for (int slot = 0; slot < 2; ++slot) {
        const int c = slot ? nodes[i].right : nodes[i].left;
        const rm_bvh_node& cn = nodes[c];
        if (depth[size_t(c)] != 0) shared = true;  // another parent reached it before
        if (!(ordered_box(cn) && (i == 0 || inside(cn, nodes[i])))) nested = false;
        depth[size_t(c)] = depth[size_t(i)] + 1;
        max_depth = std::max(max_depth, depth[size_t(c)]);
        if (cn.count > 0) {
          put(r, slot, &cn, cn.offset, cn.count);
          leaf_tris += cn.count;
        } else {
          put(r, slot, &cn, rec[size_t(c)], 0);
          parents[size_t(rec[size_t(c)])] = (r << 1) | slot;
        }
      }
    }
    // an unreachable internal node keeps an all-empty record
    for (int i = 0; i < M; ++i)
      if (rec[size_t(i)] >= 0 && depth[size_t(i)] == 0) {
        put(rec[size_t(i)], 0, nullptr, 0, -1);
        put(rec[size_t(i)], 1, nullptr, 0, -1);
      }
  }
  if (max_depth > kStack) { err = "BVH deeper than 64 levels"; return false; }
  if (shared) {
    // Shared subtrees are traversed once for each path to them: written out as
    // a tree, the nodes must stay within the limit of a BVH without sharing (64
    // levels that name one child twice would keep a ray busy for years).
    std::vector<double> size(size_t(M), 1.0);
    for (int i = M; i-- > 0;)
      if (rec[size_t(i)] >= 0) size[size_t(i)] += size[size_t(nodes[i].left)] + size[size_t(nodes[i].right)];
    if (size[0] >= double(kMaxLink)) { err = "BVH exceeds 16777215 nodes with its shared subtrees written out"; return false; }
  }
  out.max_depth = max_depth;
  out.shared = shared;
  out.tree = !shared && nested;
  out.leaf_tris = leaf_tris;
  out.n_records = n_rec;
  cudaError_t e;
  if ((e = out.records.reserve(recs.size() * sizeof(float))) != cudaSuccess ||
      (e = out.parents.reserve(parents.size() * sizeof(int))) != cudaSuccess ||
      (e = out.counters.reserve(parents.size() * sizeof(int))) != cudaSuccess ||
      (e = out.order.reserve(size_t(n_tris) * sizeof(int))) != cudaSuccess) {
    err = std::string("BVH allocation failed: ") + cudaGetErrorString(e);
    return false;
  }
  if ((e = cudaMemcpyAsync(out.records.ptr, recs.data(), recs.size() * sizeof(float), cudaMemcpyHostToDevice, st)) !=
          cudaSuccess ||
      (e = cudaMemcpyAsync(out.parents.ptr, parents.data(), parents.size() * sizeof(int), cudaMemcpyHostToDevice,
                           st)) != cudaSuccess ||
      (e = cudaMemcpyAsync(out.order.ptr, bvh_tri, size_t(n_tris) * sizeof(int), cudaMemcpyHostToDevice, st)) !=
          cudaSuccess ||
      (e = cudaStreamSynchronize(st)) != cudaSuccess) {
    err = std::string("BVH upload failed: ") + cudaGetErrorString(e);
    return false;
  }
  if ((e = build_quads(out, st)) != cudaSuccess) {
    err = std::string("BVH collapse failed: ") + cudaGetErrorString(e);
    return false;
  }
  return true;
}

}  // namespace rmd
