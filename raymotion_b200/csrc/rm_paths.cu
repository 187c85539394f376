// rm_paths.cu - the plain path tracer of one image: K1 render_paths
// (pathtrace.metal:739-769, one lane per pixel) and K2 render_paths_simd
// (:773-815, 8 or 32 lanes per pixel, each a strided subset of the samples).
//
// One thread per pixel lane that runs its samples to the end leaves most of a
// warp idle: a path ends after one vertex or after ten, and the lanes of a
// round wait for the longest.  Here a warp's lanes take tasks - the samples of
// one pixel lane - from a counter, and a lane whose sample has ended starts its
// next sample or task while the others go on, one vertex per pass of the loop:
// closest hit, shade, shadow ray (wf::vertex, as the wavefronts).  A lane's
// samples keep its random stream and order, so the values are those of the
// lane kernels.
//
// With several lanes a round's values are summed by K2's butterfly over the
// pixel's lanes, then added to the pixel's sum; samples that may run ahead of
// their round leave their value in memory and k_paths_combine forms the sums
// in K2's order.  The adaptive test (:759-764, :806-810) needs the sum before
// the next round may start, so the rounds are cut into segments that end where
// the test applies; a segment traces and combines the pixels still open, their
// list and count on the device.  One lane per pixel needs none of this: the
// task itself sums its samples in order and takes the test.
#include <cuda_runtime.h>

#include <algorithm>

#include "rm_device.cuh"
#include "rm_launch.h"
#include "rm_wf_common.cuh"

namespace rmd {

namespace {

using namespace wf;

// Bound by the traversal's dependent node loads (long_scoreboard 3.4 of 8 cycles
// between a warp's instructions, 8 of 32 lanes).  Four 128-thread blocks per SM
// (128 registers): 1280x720, 16 spp, 150 k triangles 9.9 ms, at five (96
// registers) 10.4, at six 9.7 with small frames slower; one thread per lane and
// round (k_render_paths) 19.0, and this loop 13.2 before its two traversals
// became one copy (Tracer::trace).  Cornell box at 320x180, 16 spp 1.0 against
// 2.2 ms.
//
// Kept out, measured against 13.2: shadow and extension rays of different lanes in one traversal pass
// (Cornell 2.0 ms, 512x512 18.1: each pass then shades half the lanes), a
// lane's shadow ray and next extension ray one after the other in one loop (18
// to 20 ms: the second ray's setup splits the warp).
constexpr int kPathThreads = 128, kPathBlocks = 4;
// Idle lanes of a warp that make it take new tasks: 16 (13.2 ms with two traversals; 8: 14.3, 12:
// 13.6, 22: 13.2 and the Cornell box 1.17 against 1.13).
constexpr int kRefill = 16;

__device__ __forceinline__ void write_pixel(const PathsArgs& a, uint32_t pixel, float sr, float sg, float sb, int n,
                                            uint32_t st) {
  const float cr = sr / float(n), cg = sg / float(n), cb = sb / float(n);
  if (a.hdr) {
    a.hdr[size_t(pixel) * 3] = cr; a.hdr[size_t(pixel) * 3 + 1] = cg; a.hdr[size_t(pixel) * 3 + 2] = cb;
  }
  if (a.rgb) {
    a.rgb[size_t(pixel) * 3] = tonemap8(cr); a.rgb[size_t(pixel) * 3 + 1] = tonemap8(cg);
    a.rgb[size_t(pixel) * 3 + 2] = tonemap8(cb);
  }
  if (a.dbg) { a.dbg[size_t(pixel) * 2] = st; a.dbg[size_t(pixel) * 2 + 1] = uint32_t(n); }
}

// NEE as in wf::vertex: 0 opaque scene with one light candidate, 2 opaque with
// any number, 1 any scene.
template <int NEE>
__global__ void __launch_bounds__(kPathThreads, kPathBlocks) k_paths(Scene s, Params p, uint64_t seed, PathsArgs a, int seg,
                                                           unsigned long long* ctr, uint32_t* err) {
  const unsigned full = 0xffffffffu;
  const int lane_id = int(threadIdx.x & 31);
  const int L = a.lanes;
  const unsigned tasks = unsigned(seg == 0 ? a.n_pixels : a.counts[seg]) * unsigned(L);
  const int* list = seg == 0 ? nullptr : a.list[seg & 1];
  Tracer pt(s, p, err);
  PathRegs r;
  bool active = false, fresh = false, more = true;  // fresh: the next sample's camera ray is to be made
  uint32_t x = 0, y = 0, taken = 0;
  uint32_t slot = 0;   // pixel within the chunk x lanes + lane
  int si = 0, n = 0;   // sample; one lane: samples summed
  float sr = 0, sg = 0, sb = 0, sum_l = 0, sum_l2 = 0;
  for (;;) {
    const unsigned idle = __ballot_sync(full, !active);
    if (more && (__popc(idle) >= kRefill)) {
      unsigned base = 0;
      if (lane_id == 0) base = atomicAdd(a.next + seg, unsigned(__popc(idle)));
      base = __shfl_sync(full, base, 0);
      more = base + unsigned(__popc(idle)) < tasks;
      const unsigned t = base + unsigned(__popc(idle & ((1u << lane_id) - 1u)));
      if (!active && t < tasks && t >= base) {
        const unsigned k = t / unsigned(L), lane = t % unsigned(L);
        const uint32_t local = list ? uint32_t(list[k]) : k;
        const uint32_t pixel = uint32_t(a.pixel0) + local;
        slot = local * uint32_t(L) + lane;
        x = pixel % uint32_t(p.width);
        y = pixel / uint32_t(p.width);
        if (seg == 0) {
          uint64_t sd = seed_pixel(seed, x, y);
          if (L > 1) sd ^= uint64_t(lane) * 0x94D049BB133111EBull;
          pt.rng.seed(sd);
        } else {
          pt.rng.state = a.state[slot];
        }
        si = a.round0 * L + int(lane);
        n = 0;
        sr = sg = sb = sum_l = sum_l2 = 0.0f;
        active = fresh = si < p.spp;
        if (L > 1 && !active) a.state[slot] = pt.rng.state;
      }
    }
    if (!__any_sync(full, active)) {
      if (!more) break;
      continue;
    }
    if (fresh) {
      // the camera ray of the next sample (pathtrace.metal:754-756, :792-794; sample_sensor :729-737)
      float sx, sy;
      pt.jitter(x, y, sx, sy);
      const rm_camera& cam = p.camera;
      const float focal2 = cam.focal * cam.focal;
      const float dist = 1.0f / sqrtf(sx * sx + (sy * sy + focal2));
      const float tx = sx * dist, ty = sy * dist, tz = cam.focal * dist;
      r.dx = tx * cam.m0 + (ty * cam.m1 + tz * cam.m2);
      r.dy = tx * cam.m3 + (ty * cam.m4 + tz * cam.m5);
      r.dz = tx * cam.m6 + (ty * cam.m7 + tz * cam.m8);
      r.ox = cam.x; r.oy = cam.y; r.oz = cam.z;
      r.ax = r.ay = r.az = 0.0f;
      r.tx = r.ty = r.tz = 1.0f;
      r.v = 0;
      r.meta = kDelta;
      r.last_pdf = 0.0f; r.psumW = 0.0f; r.pM = 0;
      r.pbr = r.pbg = r.pbb = r.pbcos = 0.0f;
      fresh = false;
    }
    if (active) {
      bool go = false;
      if (r.v < p.bounces) {
        // closest hit, through transparent crossings (pathtrace.metal:536-550)
        const Hit hit = NEE == 1 ? pt.cast_alpha_ray(r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, kFar)
                                 : pt.cast_ray(r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, kFar);
        if (hit.tri >= 0) {
          bool has_shadow = false;
          float4 so, sd, c;
          go = hit.ior > 1.0001f ? vertex<1, NEE>(pt, p, r, hit, has_shadow, so, sd, c)
                                 : vertex<0, NEE>(pt, p, r, hit, has_shadow, so, sd, c);
          if (NEE != 1 && has_shadow && !pt.shadow(so.x, so.y, so.z, sd.x, sd.y, sd.z, so.w)) {
            r.ax += c.x; r.ay += c.y; r.az += c.z;
          }
        }
      }
      if (!go) {
        // the sample is done
        float cr = r.ax, cg = r.ay, cb = r.az;
        clamp3(p, cr, cg, cb);
        ++taken;
        bool last;
        if (L == 1) {
          sr += cr; sg += cg; sb += cb;
          ++n;
          last = n >= p.spp;
          if (p.adapt_min > 0) {
            const float lum = cr * 0.2126f + cg * 0.7152f + cb * 0.0722f;
            sum_l += lum; sum_l2 += lum * lum;
            if (n >= p.adapt_min && n > 1 && n % p.adapt_step == 0) {
              const float mean = sum_l / float(n);
              const float var = fmaxf(0.0f, (sum_l2 - sum_l * mean) / float(n - 1));
              const float thr = p.adapt_rel * mean + p.adapt_abs;
              if (var < thr * thr) last = true;
            }
          }
          if (last) write_pixel(a, y * uint32_t(p.width) + x, sr, sg, sb, n, pt.rng.state);
        } else {
          a.val[size_t(si / L - a.round0) * size_t(a.n_pixels) * size_t(L) + slot] = make_float4(cr, cg, cb, 0.f);
          si += L;
          last = si >= p.spp || si / L >= a.round1;
          if (last) a.state[slot] = pt.rng.state;
        }
        active = fresh = !last;
      }
    }
  }
  __syncwarp();
  warp_add(ctr + 0, taken);
  warp_add(ctr + 1, pt.rays);
  warp_add(ctr + 2, pt.nodes);
  warp_add(ctr + 3, pt.tests);
}

// The open pixels of a segment, L lanes of a warp each: every round's
// butterfly sum exactly as K2 does it (pathtrace.metal:797-805), then the
// adaptive test (:806-810) and either the pixel's output (:811-814) or its
// entry in the next segment's list.
template <int L>
__global__ void __launch_bounds__(256) k_paths_combine(Params p, PathsArgs a, int seg, int mode,
                                                       unsigned long long* done, unsigned long long ticket) {
  const int n_open = seg == 0 ? a.n_pixels : a.counts[seg];
  if (n_open == 0) {
    if (done && blockIdx.x == 0 && threadIdx.x == 0) *static_cast<volatile unsigned long long*>(done) = ticket;
    return;
  }
  const int* list = seg == 0 ? nullptr : a.list[seg & 1];
  const int lane = int(threadIdx.x & 31) % L;
  const int stride = int(gridDim.x * blockDim.x) / L;
  for (int k = int(blockIdx.x * blockDim.x + threadIdx.x) / L; k - (int(threadIdx.x & 31) / L) < n_open; k += stride) {
    const bool valid = k < n_open;
    const uint32_t local = valid ? (list ? uint32_t(list[k]) : uint32_t(k)) : 0u;
    float4 gs = make_float4(0.f, 0.f, 0.f, 0.f);
    float sl2 = 0.0f;
    if (valid && seg > 0) {
      gs = a.gsum[local];
      sl2 = a.gsl2[local];
    }
    const uint32_t slot = local * uint32_t(L) + uint32_t(lane);
    int n = 0;
    for (int r = a.round0; r < a.round1; ++r) {
      float cr = 0.f, cg = 0.f, cb = 0.f;
      if (valid && r * L + lane < p.spp) {
        const float4 v = a.val[size_t(r - a.round0) * size_t(a.n_pixels) * size_t(L) + slot];
        cr = v.x; cg = v.y; cb = v.z;
      }
      float lum = cr * 0.2126f + cg * 0.7152f + cb * 0.0722f;
      float lum2 = lum * lum;
#pragma unroll
      for (int m = 1; m < L; m <<= 1) {
        cr += __shfl_xor_sync(0xffffffffu, cr, m, L);
        cg += __shfl_xor_sync(0xffffffffu, cg, m, L);
        cb += __shfl_xor_sync(0xffffffffu, cb, m, L);
        lum += __shfl_xor_sync(0xffffffffu, lum, m, L);
        lum2 += __shfl_xor_sync(0xffffffffu, lum2, m, L);
      }
      gs.x += cr; gs.y += cg; gs.z += cb; gs.w += lum;
      sl2 += lum2;
      n = min(r * L + L, p.spp);
    }
    uint32_t st = valid ? a.state[slot] : 0u;
#pragma unroll
    for (int m = 1; m < L; m <<= 1) st ^= __shfl_xor_sync(0xffffffffu, st, m, L);
    bool open = false;
    if (valid && lane == 0) {
      bool stop = mode == 2;
      if (mode == 1) {
        const float mean = gs.w / float(n);
        const float var = fmaxf(0.0f, (sl2 - gs.w * mean) / float(n - 1));
        const float thr = p.adapt_rel * mean + p.adapt_abs;
        stop = var < thr * thr;
      }
      if (stop) {
        write_pixel(a, uint32_t(a.pixel0) + local, gs.x, gs.y, gs.z, n, st);
      } else {
        a.gsum[local] = gs;
        a.gsl2[local] = sl2;
        open = true;
      }
    }
    if (mode != 2) append(a.list[(seg + 1) & 1], a.counts + seg + 1, open, int(local));
  }
}

template <int NEE>
cudaError_t run(const Scene& s, const Params& p, uint64_t seed, const PathsArgs& a, int seg, int blocks,
                unsigned long long* ctr, uint32_t* err, cudaStream_t st) {
  k_paths<NEE><<<unsigned(blocks), kPathThreads, 0, st>>>(s, p, seed, a, seg, ctr, err);
  return cudaGetLastError();
}

}  // namespace

long long paths_one_wave(int sms) { return (long long)sms * kPathBlocks * kPathThreads; }

cudaError_t launch_paths(const Scene& s, const Params& p, uint64_t seed, const PathsArgs& a, int seg, int sms,
                         unsigned long long* ctr, uint32_t* err, cudaStream_t st) {
  const long long tasks = (long long)a.n_pixels * a.lanes;
  const int blocks = int(std::min<long long>((long long)sms * kPathBlocks, (tasks + kPathThreads - 1) / kPathThreads));
  if (!p.opaque) return run<1>(s, p, seed, a, seg, blocks, ctr, err, st);
  if (p.restir_candidates <= 1) return run<0>(s, p, seed, a, seg, blocks, ctr, err, st);
  return run<2>(s, p, seed, a, seg, blocks, ctr, err, st);
}

cudaError_t launch_paths_combine(const Params& p, const PathsArgs& a, int seg, int mode, unsigned long long* done,
                                 unsigned long long ticket, int sms, cudaStream_t st) {
  const long long threads = (long long)a.n_pixels * a.lanes;
  const unsigned g = unsigned(std::min<long long>((long long)sms * 8, (threads + 255) / 256));
  if (a.lanes == 8) k_paths_combine<8><<<g, 256, 0, st>>>(p, a, seg, mode, done, ticket);
  else k_paths_combine<32><<<g, 256, 0, st>>>(p, a, seg, mode, done, ticket);
  return cudaGetLastError();
}

}  // namespace rmd
