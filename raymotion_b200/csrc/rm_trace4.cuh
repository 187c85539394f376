// rm_trace4.cuh - rays traced by four lanes each through the 4-wide BVH
// (rm_quad.cu): the traversal of the ray-query and wavefront trace kernels.
#pragma once

#include "rm_device.cuh"

namespace rmd {

constexpr int kT4Warps = 2;        // warps per block
constexpr int kT4Threads = kT4Warps * 32;
constexpr int kT4Depth = 32;       // stack entries per ray in shared memory; the rest in local memory
constexpr uint32_t kT4Done = 0xFFFFFFFFu;

struct T4Shared {
  // [warp][depth][ray]: the eight rays of a warp never share a bank
  uint32_t stack[kT4Warps][kT4Depth][8];
};

// Source: bool fetch(int i, float4& o_tmax, float3& d, bool& any_hit) for ray i (all four lanes), and
// void emit(bool have, int i, TraceResult, bool write) called by all lanes of the warp together.
template <class Source>
__device__ __forceinline__ void trace_quads(const Scene& s, T4Shared& sh, Source& src, int n_rays, uint32_t* err,
                                            uint32_t& n_nodes, uint32_t& n_tests) {
  const unsigned full = 0xffffffffu;
  const int lane = int(threadIdx.x & 31), l4 = lane & 3;
  const int base_lane = lane & 28;
  uint32_t(*stk)[8] = sh.stack[threadIdx.x >> 5];
  const int g = lane >> 2;
  const int total = int(gridDim.x * blockDim.x) >> 2;
  uint32_t over[kQuadStack - kT4Depth + 4];
  int i = int(blockIdx.x * blockDim.x + threadIdx.x) >> 2;
  while (__any_sync(full, i < n_rays)) {
    const bool have = i < n_rays;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    float3 d = make_float3(0.f, 0.f, 1.f);
    bool any_hit = false;
    if (have) src.fetch(i, o, d, any_hit);
    const float ix = 1.0f / (d.x == 0.0f ? 1e-30f : d.x);
    const float iy = 1.0f / (d.y == 0.0f ? 1e-30f : d.y);
    const float iz = 1.0f / (d.z == 0.0f ? 1e-30f : d.z);
    float cxl, cxh, cyl, cyh, czl, czh;
    slab_addends(o.x, ix, cxl, cxh);
    slab_addends(o.y, iy, cyl, cyh);
    slab_addends(o.z, iz, czl, czh);
    float best_t = o.w, best_u = 0.f, best_v = 0.f;
    int best = -1;
    bool own = l4 == 0;
    int sp = 0;
    uint32_t cur = have && s.n_nodes > 0 ? 0u : kT4Done;
    for (;;) {
      const unsigned im = __ballot_sync(full, cur < (1u << 24));
      const unsigned lm = __ballot_sync(full, cur >= (1u << 24) && cur != kT4Done);
      if ((im | lm) == 0u) break;
      bool want_pop = false;
      if (im != 0u && __popc(lm) < 16) {
        // one node per ray: each lane boxes one child
        const bool in = cur < (1u << 24);
        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
        if (in && !bad_index(cur, s.n_nodes, err, kSiteNode)) {
          const float4* n = s.quads + (size_t(cur) * 4 + l4) * 2;
          lo = __ldg(n);
          hi = __ldg(n + 1);
        }
        const float lx = __fmaf_rn(lo.x, ix, cxl), hx = __fmaf_rn(hi.x, ix, cxh);
        const float ly = __fmaf_rn(lo.y, iy, cyl), hy = __fmaf_rn(hi.y, iy, cyh);
        const float lz = __fmaf_rn(lo.z, iz, czl), hz = __fmaf_rn(hi.z, iz, czh);
        const uint32_t word = __float_as_uint(lo.w);
        const float tn = fmax3(fminf(lx, hx), fminf(ly, hy), fmaxf(fminf(lz, hz), 0.0f));
        const float tf = fmin3(fmaxf(lx, hx), fmaxf(ly, hy), fminf(fmaxf(lz, hz), best_t));
        const bool hit = word != 0u && !(tn > tf * kFmaBoxSlack);
        const uint32_t k0 = hit ? ((__float_as_uint(tn) & ~3u) | uint32_t(l4)) : kT4Done;
        const uint32_t k1 = __shfl_xor_sync(full, k0, 1);
        const uint32_t k2 = __shfl_xor_sync(full, k0, 2);
        const uint32_t k3 = __shfl_xor_sync(full, k0, 3);
        const uint32_t m = min(min(k0, k1), min(k2, k3));
        const uint32_t next = __shfl_sync(full, word, base_lane | int(m & 3u));
        if (in) {
          if (l4 == 0) n_nodes += 2;
          if (m != kT4Done) {
            // the other hit children, farthest first
            const int after = int(k1 > k0 && k1 != kT4Done) + int(k2 > k0 && k2 != kT4Done) + int(k3 > k0 && k3 != kT4Done);
            const int hits = int(k0 != kT4Done) + int(k1 != kT4Done) + int(k2 != kT4Done) + int(k3 != kT4Done);
            if (sp + 3 <= kT4Depth) {
              if (hit && k0 != m) stk[sp + after][g] = word;
              sp += hits - 1;
            } else {
              if (sp + 3 > kQuadStack) { atomicOr(err, kErrStack); cur = kT4Done; sp = 0; }
              else {
                for (int q = 0; q < hits - 1; ++q) {
                  const bool mine = hit && k0 != m && q == after;
                  if (sp + q < kT4Depth) { if (mine) stk[sp + q][g] = word; }
                  else over[sp + q - kT4Depth] = mine ? word : 0u;
                }
                sp += hits - 1;
              }
            }
            if (cur != kT4Done) cur = next;
          } else {
            want_pop = true;
          }
        }
      } else {
        // leaves: four triangles of a ray at a time
        const bool leaf = cur >= (1u << 24) && cur != kT4Done;
        int first = int(cur & 0xFFFFFFu), count = leaf ? int(cur >> 24) : 0;
        if (kChecked && leaf && (bad_index(first, s.n_tris, err, kSiteLeaf) ||
                         bad_index(first + count - 1, s.n_tris, err, kSiteLeaf)))
          count = 0;
        bool found = false;
        for (int b = 0; __any_sync(full, b < count); b += 4) {
          TraceResult c{best_t, best, 0.f, 0.f};
          bool ok = false;
          if (b + l4 < count) {
            ++n_tests;
            ok = test_triangle(s.tgeo + size_t(first + b + l4) * 3, o.x, o.y, o.z, d.x, d.y, d.z, c);
          }
          const uint32_t kd = ok ? __float_as_uint(c.t) : kT4Done;  // t > 0: its bits order as an integer
          uint32_t md = min(kd, __shfl_xor_sync(full, kd, 1));
          md = min(md, __shfl_xor_sync(full, md, 2));
          const uint32_t kj = ok && kd == md ? uint32_t(c.tri) : kT4Done;
          uint32_t mj = min(kj, __shfl_xor_sync(full, kj, 1));
          mj = min(mj, __shfl_xor_sync(full, mj, 2));
          if (md != kT4Done) {
            best_t = __uint_as_float(md);
            best = int(mj);
            own = kj == mj;
            best_u = c.u;
            best_v = c.v;
            found = true;
          }
        }
        if (leaf) {
          if (found && any_hit) cur = kT4Done;
          else want_pop = true;
        }
      }
      __syncwarp();
      if (want_pop) {
        if (sp == 0) cur = kT4Done;
        else {
          --sp;
          if (sp < kT4Depth) cur = stk[sp][g];
          else {
            uint32_t v = over[sp - kT4Depth];
            const unsigned grp = 0xFu << base_lane;
            v |= __shfl_xor_sync(grp, v, 1);
            v |= __shfl_xor_sync(grp, v, 2);
            cur = v;
          }
        }
      }
      __syncwarp();
    }
    src.emit(have && own, i, TraceResult{best_t, best, best_u, best_v});
    i += total;
  }
}

}  // namespace rmd
