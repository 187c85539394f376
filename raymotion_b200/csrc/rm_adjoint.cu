// rm_adjoint.cu - path-replay adjoint of the plain single-frame chain:
// gradients of an image loss with respect to per-material albedo, roughness,
// emission and index of refraction.
//
// The differentiated estimator is the frame of render_paths (K1) or the lane
// kernel (K2) (pathtrace.metal:739-815) with its sampling held fixed: every
// random decision, sampled direction, pdf, MIS weight, light-sample
// resampling weight (RIS NEE) and Russian-roulette probability keeps its
// value at the current parameters, and only the
// factors of the path integrand that depend on the materials are
// differentiated - the opaque BSDF value (albedo, roughness), the emission of
// hit and sampled lights, and for a dielectric the Fresnel and (eta_i/eta_t)^2
// factors (index of refraction) and the microfacet D and G terms (roughness),
// each as a ratio to its value at the current parameters (path replay
// backpropagation with detached sampling, Vicini, Speierer and Jakob,
// SIGGRAPH 2021).  With the sample's radiance C and the radiance S_k that the
// path gathers after vertex k, the derivative of a sample is
//     sum_k thr_k * d(E_k + N_k) + sum_k (dB_k / B_k) * S_k
// (E_k emission at vertex k, N_k its light sample, B_k the throughput factor
// of its scattering).  A pixel lane's samples are replayed in order from its
// random stream, each in one walk: a vertex's terms independent of C and the
// factors of those proportional to it are kept until the path ends and C is
// known (adjoint_step, adjoint_end); paths longer than the kept list walk
// twice (first for C).  The lanes of a warp take pixel lanes from a counter and
// advance one vertex per pass of a loop (k_adjoint), as the forward frame does.
// The refracted direction
// is held fixed when the index of refraction changes; its motion would need a
// reparameterised sampler and is not part of the estimator.
#include <cuda_runtime.h>

#include <algorithm>

#include "rm_device.cuh"
#include "rm_launch.h"

namespace rmd {

namespace {

constexpr int kMatParams = 8;  // albedo rgb, rough, emission rgb, ior

extern __shared__ float sh_sums[];  // the block's accumulators

// One copy of the atomic additions per kernel (a float addition in shared
// memory is a loop), so that a pass over a vertex stays within the
// instruction cache.
struct GradSink {
  bool shared;  // the block's accumulators, else the caller's gradient
  float* gl;
  __device__ __forceinline__ void one(int i, float v) const {
    if (v == 0.0f) return;
    if (shared) atomicAdd(sh_sums + i, v);
    else atomicAdd(gl + i, v);
  }
  // parameters k to k + 3 of material m
  __device__ __noinline__ void add4(int m, int k, float a, float b, float c, float d) const {
    if (m < 0) return;
    const int i = m * kMatParams + k;
    one(i, a);
    one(i + 1, b);
    one(i + 2, c);
    one(i + 3, d);
  }
  __device__ __forceinline__ void albedo_rough(int m, float a, float b, float c, float r) const {
    add4(m, 0, a, b, c, r);
  }
  __device__ __forceinline__ void emission(int m, float a, float b, float c) const { add4(m, 4, a, b, c, 0.0f); }
  __device__ __forceinline__ void ior_rough(int m, float ior, float r) const {
    add4(m, 0, 0.0f, 0.0f, 0.0f, r);
    add4(m, 4, 0.0f, 0.0f, 0.0f, ior);
  }
};

struct Dual {
  float v, d;
};
__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return Dual{a.v + b.v, a.d + b.d}; }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return Dual{a.v - b.v, a.d - b.d}; }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) { return Dual{a.v * b.v, a.d * b.v + a.v * b.d}; }
__device__ __forceinline__ Dual operator/(Dual a, Dual b) {
  return Dual{a.v / b.v, (a.d * b.v - a.v * b.d) / (b.v * b.v)};
}
__device__ __forceinline__ Dual dsqrt(Dual a) {
  const float r = sqrtf(a.v);
  return Dual{r, r > 0.0f ? a.d / (2.0f * r) : 0.0f};
}
__device__ __forceinline__ Dual dc(float v) { return Dual{v, 0.0f}; }

// Fresnel (pathtrace.metal:80-91) and its derivative along the dual parts of
// the two indices.
__device__ Dual fresnel_dual(float ci, Dual eta_in, Dual eta_out) {
  if (ci < 0.0f) ci = 0.0f;
  if (ci > 1.0f) ci = 1.0f;
  const Dual eta = eta_in / eta_out;
  const Dual s2 = eta * eta * dc(1.0f - ci * ci);
  if (s2.v >= 1.0f) return dc(1.0f);
  const Dual ct = dsqrt(dc(1.0f) - s2);
  const Dual c = dc(ci);
  const Dual rp = (eta_out * c - eta_in * ct) / (eta_out * c + eta_in * ct);
  const Dual rs = (eta_in * c - eta_out * ct) / (eta_in * c + eta_out * ct);
  return dc(0.5f) * (rp * rp + rs * rs);
}

// |h x n|^2: the squared sine between two unit vectors, accurate near 0.
__device__ __forceinline__ float sin2(float hx, float hy, float hz, float nx, float ny, float nz) {
  const float cx = hy * nz - hz * ny, cy = hz * nx - hx * nz, cz = hx * ny - hy * nx;
  return cx * cx + cy * cy + cz * cz;
}

// d/dalpha2 of log G1 for one direction (Smith G1 of pathtrace.metal:270-276).
__device__ __forceinline__ float dlog_g1(float c, float alpha2) {
  const float sq = sqrtf(c * c + alpha2 * (1.0f - c * c));
  return -(1.0f - c * c) / (2.0f * sq * (c + sq));
}

// The opaque BSDF value (pathtrace.metal:243-295) with its derivatives with
// respect to each albedo channel and alpha2.
struct BsdfGrad {
  float f[3], da[3], dal2[3];
};

__device__ __noinline__ BsdfGrad bsdf_grad(float wix, float wiy, float wiz, float wox, float woy, float woz, float nx, float ny,
                              float nz, float alpha2, float metallic, float ar, float ag, float ab) {
  BsdfGrad out;
#pragma unroll
  for (int c = 0; c < 3; ++c) out.f[c] = out.da[c] = out.dal2[c] = 0.0f;
  const float cos_i = wix * nx + (wiy * ny + wiz * nz);
  const float cos_o = wox * nx + (woy * ny + woz * nz);
  if (!(cos_i > 1e-8f && cos_o > 1e-8f)) return out;
  float hx = wix + wox, hy = wiy + woy, hz = wiz + woz;
  const float hl = sqrtf(hx * hx + hy * hy + hz * hz);
  if (!(hl > 1e-8f)) return out;
  const float inv = 1.0f / hl;
  hx *= inv; hy *= inv; hz *= inv;
  float cos_h = hx * nx + (hy * ny + hz * nz);
  float vo_h = wox * hx + (woy * hy + woz * hz);
  if (cos_h < 0.0f) { cos_h = -cos_h; vo_h = -vo_h; }
  if (!(vo_h > 1e-8f)) return out;
  // cos_h^2 (alpha2 - 1) + 1 = |h x n|^2 + alpha2 cos_h^2, without the
  // cancellation near the lobe's peak (alpha2 can be 6e-6)
  const float dd = sin2(hx, hy, hz, nx, ny, nz) + alpha2 * cos_h * cos_h;
  const float D = alpha2 / (kPi * dd * dd);
  const float g1 = 2.0f * cos_o / (cos_o + sqrtf(cos_o * cos_o + alpha2 * (1.0f - cos_o * cos_o)));
  const float g2 = 2.0f * cos_i / (cos_i + sqrtf(cos_i * cos_i + alpha2 * (1.0f - cos_i * cos_i)));
  const float G = g1 * g2;
  float om = 1.0f - vo_h;
  om *= om; om *= om; om *= 1.0f - vo_h;
  const float di = 1.0f - metallic;
  const float base = D * G / (4.0f * cos_i * cos_o);
  const float dlog = 1.0f / alpha2 - 2.0f * cos_h * cos_h / dd + dlog_g1(cos_o, alpha2) + dlog_g1(cos_i, alpha2);
  const float alb[3] = {ar, ag, ab};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float f0 = 0.04f * di + alb[c] * metallic;
    const float F = f0 + (1.0f - f0) * om;
    out.f[c] = alb[c] * di * (1.0f - F) / kPi + base * F;
    out.da[c] = (di * (1.0f - F) - alb[c] * di * metallic * (1.0f - om)) / kPi + base * metallic * (1.0f - om);
    out.dal2[c] = base * dlog * F;
  }
  return out;
}

// d alpha2 / d rough for alpha2 = r^4, r = max(clamp(rough, 0, 1), 0.02).
__device__ __forceinline__ float dalpha2(float rough) {
  if (!(rough > 0.02f && rough < 1.0f)) return 0.0f;
  return 4.0f * rough * rough * rough;
}

// A walk along one sample's path (pathtrace.metal:552-728, the arithmetic and
// random draws of Tracer::pathtrace), vertex by vertex.
struct Walk {
  float ox, oy, oz, dx, dy, dz;
  float acc[3], thr[3], g[3];  // radiance so far, throughput, the loss gradient of the sample's value
  float C[3];                  // the sample's radiance (walks that do not keep their terms)
  float last_pdf, prev_sumW, prev_b[3], prev_cos;
  uint32_t prev_M;
  int prev_delta, bounce, max_bounces;
  bool camera;  // from the camera; else from a vertex already shaded (the ReSTIR
                // shade's primary vertex, pathtrace.metal:1135-1255), whose BSDF
                // sample and light-sample sums the fields above carry in
  bool keep;    // C is not known yet: keep the vertices' terms
  bool mute;    // a walk for C alone
};

// The kept terms of a walk's scattering vertices.  Opaque: the albedo and
// roughness sums so far and the factors of C per channel; dielectric: the same
// of ior and roughness.
struct Kept {
  static constexpr int kMax = 24;
  int n;
  int m[kMax];          // material << 1 | dielectric
  float v[kMax][10];
};

__device__ __forceinline__ void walk_camera(Walk& w, Tracer& pt, uint32_t x, uint32_t y) {
  const Params& p = pt.p;
  float sx, sy;
  pt.jitter(x, y, sx, sy);
  const rm_camera& cam = p.camera;
  const float focal2 = cam.focal * cam.focal;
  const float dist = 1.0f / sqrtf(sx * sx + (sy * sy + focal2));
  const float tx = sx * dist, ty = sy * dist, tz = cam.focal * dist;
  w.dx = tx * cam.m0 + (ty * cam.m1 + tz * cam.m2);
  w.dy = tx * cam.m3 + (ty * cam.m4 + tz * cam.m5);
  w.dz = tx * cam.m6 + (ty * cam.m7 + tz * cam.m8);
  w.ox = cam.x; w.oy = cam.y; w.oz = cam.z;
  w.thr[0] = w.thr[1] = w.thr[2] = 1.0f;
  w.last_pdf = w.prev_sumW = w.prev_cos = 0.0f;
  w.prev_b[0] = w.prev_b[1] = w.prev_b[2] = 0.0f;
  w.prev_M = 0;
  w.prev_delta = 1;
  w.max_bounces = p.bounces;
  w.camera = true;
}

// One vertex of a walk, accumulating g . dC/dparams; false when the path ends.
// kNee as in wf::vertex: 0 opaque scene with one light candidate, 2 opaque
// with several (RIS), 1 any scene.
template <int kNee>
__device__ __forceinline__ bool adjoint_step(Tracer& pt, const int32_t* __restrict__ tri_mat, Walk& w,
                                             const GradSink& sink, Kept& kept) {
  const Scene& s = pt.s;
  const Params& p = pt.p;
  const Hit hit = kNee == 1 ? pt.cast_alpha_ray(w.ox, w.oy, w.oz, w.dx, w.dy, w.dz, kFar)
                            : pt.cast_ray(w.ox, w.oy, w.oz, w.dx, w.dy, w.dz, kFar);
  if (hit.tri < 0) return false;
  const int m = w.mute ? -1 : tri_mat[hit.tri];
  float pnx = hit.nix, pny = hit.niy, pnz = hit.niz;
  float geom = hit.ngx * pnx + (hit.ngy * pny + hit.ngz * pnz);
  if (geom < 0.0f) { pnx = -pnx; pny = -pny; pnz = -pnz; }
  float ndot = w.dx * pnx + (w.dy * pny + w.dz * pnz);
  bool front = true;
  if (ndot > 0.0f) { pnx = -pnx; pny = -pny; pnz = -pnz; front = false; }
  float wox = -w.dx, woy = -w.dy, woz = -w.dz;
  float rough = hit.rough;
  if (rough < 0.0f) rough = 0.0f;
  if (rough > 1.0f) rough = 1.0f;
  if (rough < 0.02f) rough = 0.02f;
  float alpha = rough * rough;
  float alpha2 = alpha * alpha;
  const float dal2 = dalpha2(hit.rough);
  const rm_triangle& lt = s.tris[hit.tri];
  float metallic = lt.metallic;
  if (metallic < 0.0f) metallic = 0.0f;
  if (metallic > 1.0f) metallic = 1.0f;
  float we = 1.0f;  // MIS weight of the emission term (held fixed)
  if ((w.camera && w.bounce == 0) || w.prev_delta == 1) {
    w.acc[0] += hit.er * w.thr[0]; w.acc[1] += hit.eg * w.thr[1]; w.acc[2] += hit.eb * w.thr[2];
  } else {
    float lx = hit.px - w.ox, ly = hit.py - w.oy, lz = hit.pz - w.oz;
    float dist2 = lx * lx + ly * ly + lz * lz;
    float dist = sqrtf(dist2);
    float pl = 1e30f;
    float lta = lt.alpha;
    bool area = false;
    if (dist > 1e-20f && w.last_pdf > 1e-20f && w.prev_M > 0 && w.prev_sumW > 1e-20f) {
      float ph = lum3(hit.er * w.prev_b[0] * w.prev_cos * lta, hit.eg * w.prev_b[1] * w.prev_cos * lta,
                      hit.eb * w.prev_b[2] * w.prev_cos * lta);
      if (ph > 1e-20f) pl = float(w.prev_M) * ph / w.prev_sumW;
      else area = true;
    } else if (dist > 1e-20f && w.last_pdf > 1e-20f) {
      area = true;
    }
    if (area) {
      float inv = 1.0f / dist;
      float lxn = lx * inv, lyn = ly * inv, lzn = lz * inv;
      float cos_l = -(lt.nn.x * lxn + (lt.nn.y * lyn + lt.nn.z * lzn));
      if (cos_l > 1e-8f) {
        float lum = lum3(lt.er, lt.eg, lt.eb);
        if (lum < 1e-6f) lum = 1e-6f;
        pl = dist2 * lum / (cos_l * p.light_total);
      }
    }
    we = p.nomis ? 0.0f : ((w.last_pdf + pl > 1e-20f) ? w.last_pdf / (w.last_pdf + pl) : 0.0f);
    w.acc[0] += hit.er * w.thr[0] * we; w.acc[1] += hit.eg * w.thr[1] * we; w.acc[2] += hit.eb * w.thr[2] * we;
  }
  sink.emission(m, w.g[0] * w.thr[0] * we, w.g[1] * w.thr[1] * we, w.g[2] * w.thr[2] * we);
  if (hit.ior > 1.0001f) {
    float nx2, ny2, nz2, es;
    float dp[7];
    bool valid = pt.sample_dielectric(wox, woy, woz, pnx, pny, pnz, w.dx, w.dy, w.dz, hit.ior, front, rough, alpha2,
                                      nx2, ny2, nz2, es, dp);
    if (!valid) return false;
    // B_k = es: d log B_k (ior, rough), times g . S_k
    float dlog_ior = 0.0f, dlog_r = 0.0f;
    const int event = int(dp[0]);
    if (event != 2) {
      const Dual ior{hit.ior, 1.0f};
      const Dual ei = front ? dc(1.0f) : ior, et = front ? ior : dc(1.0f);
      const Dual F = fresnel_dual(dp[1], ei, et);
      if (event == 0) dlog_ior = F.v > 0.0f ? F.d / F.v : 0.0f;
      else {
        dlog_ior = F.v < 1.0f ? -F.d / (1.0f - F.v) : 0.0f;
        dlog_ior += front ? -2.0f / hit.ior : 2.0f / hit.ior;  // (eta_i / eta_t)^2
      }
    }
    if (rough > 0.0201f && dal2 != 0.0f) {
      const float ch = dp[4];
      const float dd = dp[6] + alpha2 * ch * ch;
      dlog_r = 1.0f / alpha2 - 2.0f * ch * ch / dd;  // D
      if (dp[5] == 0.0f) dlog_r += dlog_g1(dp[3], alpha2) + dlog_g1(dp[2], alpha2);  // G, unless clamped
      dlog_r *= dal2;
    }
    if (w.keep) {
      // g . (C - acc_k) dlog: the acc half as it stands, the factor of g . C
      const float gA = w.g[0] * w.acc[0] + w.g[1] * w.acc[1] + w.g[2] * w.acc[2];
      const int k = kept.n++;
      kept.m[k] = m * 2 + 1;
      kept.v[k][0] = -gA * dlog_ior;
      kept.v[k][1] = -gA * dlog_r;
      kept.v[k][2] = dlog_ior;
      kept.v[k][3] = dlog_r;
    } else {
      const float gS = w.g[0] * (w.C[0] - w.acc[0]) + w.g[1] * (w.C[1] - w.acc[1]) + w.g[2] * (w.C[2] - w.acc[2]);
      sink.ior_rough(m, gS * dlog_ior, gS * dlog_r);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) w.thr[c] *= es;
    float sg = 1.0f;
    if (nx2 * pnx + (ny2 * pny + nz2 * pnz) < 0.0f) sg = -1.0f;
    w.ox = hit.px + pnx * 0.001f * sg;
    w.oy = hit.py + pny * 0.001f * sg;
    w.oz = hit.pz + pnz * 0.001f * sg;
    w.dx = nx2; w.dy = ny2; w.dz = nz2;
    w.prev_delta = 1;
    w.prev_sumW = 0; w.prev_M = 0;
  } else {
    float spec_prob = 0.05f + 0.95f * metallic;
    if (spec_prob > 0.98f) spec_prob = 0.98f;
    if (metallic >= 0.999f) spec_prob = 1.0f;
    const bool alb_grad = hit.shader != 1;
    const float tx[3] = {hit.txr, hit.txg, hit.txb};
    float cur_sumW = 0;
    uint32_t cur_M = 0;
    float galb[3] = {0.f, 0.f, 0.f}, grough = 0.0f;  // this vertex's albedo and roughness gradient
    {
      float dl[3], sdist, sox, soy, soz, sdx, sdy, sdz;
      bool has_ray;
      float parts[2];
      // single-candidate NEE (pathtrace.metal:319-384) or RIS over the
      // candidates (:385-469), with the same draws; the selection, its
      // resampling weight W and the MIS weight are held, so the light sample
      // N_k = Le f k moves only with the light's emission and this BSDF
      if (kNee == 2 || (kNee == 1 && p.restir_candidates > 1))
        pt.direct_lighting_deferred(hit.px, hit.py, hit.pz, pnx, pny, pnz, wox, woy, woz, rough, metallic, spec_prob,
                                    hit.ar, hit.ag, hit.ab, dl[0], dl[1], dl[2], cur_sumW, cur_M, has_ray, sox, soy,
                                    soz, sdx, sdy, sdz, sdist, parts);
      else
        pt.nee_single_deferred(hit.px, hit.py, hit.pz, pnx, pny, pnz, wox, woy, woz, rough, metallic, spec_prob,
                               hit.ar, hit.ag, hit.ab, dl[0], dl[1], dl[2], cur_sumW, cur_M, has_ray, sox, soy, soz,
                               sdx, sdy, sdz, sdist, parts);
      if (has_ray && !(kNee == 1 ? pt.occluded(sox, soy, soz, sdx, sdy, sdz, sdist)
                                 : pt.shadow(sox, soy, soz, sdx, sdy, sdz, sdist))) {
        // N_k = Le * f * k: derivative in the light's emission and this surface's BSDF
        const int li = __float_as_int(parts[0]);
        const LightRec L = load_light(s, li);
        const int ml = w.mute ? -1 : tri_mat[s.lights[li]];
        const BsdfGrad bg = bsdf_grad(sdx, sdy, sdz, wox, woy, woz, pnx, pny, pnz, alpha2, metallic, hit.ar, hit.ag,
                                      hit.ab);
        const float le[3] = {L.er, L.eg, L.eb};
        float gle[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          w.acc[c] += dl[c] * w.thr[c];
          const float gt = w.g[c] * w.thr[c] * parts[1];
          gle[c] = gt * bg.f[c];
          if (alb_grad) galb[c] = gt * le[c] * bg.da[c] * tx[c];
          grough += gt * le[c] * bg.dal2[c];
        }
        grough *= dal2;
        sink.emission(ml, gle[0], gle[1], gle[2]);
      }
    }
    float nx2, ny2, nz2;
    bool go = true;
    if (pt.U() < spec_prob) {
      float hx, hy, hz;
      pt.sample_ggx_half(alpha2, pnx, pny, pnz, hx, hy, hz);
      float md = wox * hx + (woy * hy + woz * hz);
      go = md > 1e-8f;
      nx2 = 2.0f * md * hx - wox;
      ny2 = 2.0f * md * hy - woy;
      nz2 = 2.0f * md * hz - woz;
      w.prev_delta = (rough <= 0.0201f) ? 1 : 0;
    } else {
      pt.sample_cosine(pnx, pny, pnz, nx2, ny2, nz2);
      w.prev_delta = 0;
    }
    if (go) go = nx2 * pnx + (ny2 * pny + nz2 * pnz) > 1e-8f;
    Bsdf e{0.f, 0.f, 0.f, 0.f};
    if (go) {
      float d = 1.0f / sqrtf(nx2 * nx2 + ny2 * ny2 + nz2 * nz2);
      nx2 *= d; ny2 *= d; nz2 *= d;
      e = Tracer::eval_bsdf(nx2, ny2, nz2, wox, woy, woz, pnx, pny, pnz, alpha2, metallic, spec_prob, hit.ar, hit.ag,
                            hit.ab);
      go = e.pdf > 1e-12f;
    }
    float qa[3] = {0.f, 0.f, 0.f}, qr[3] = {0.f, 0.f, 0.f};
    if (go) {
      // B_k = f * cos / pdf: d log B_k = df / f, times g . S_k per channel
      const BsdfGrad bg = bsdf_grad(nx2, ny2, nz2, wox, woy, woz, pnx, pny, pnz, alpha2, metallic, hit.ar, hit.ag,
                                    hit.ab);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const bool ok = bg.f[c] > 0.0f;
        qa[c] = (ok && alb_grad) ? w.g[c] * bg.da[c] * tx[c] / bg.f[c] : 0.0f;
        qr[c] = ok ? w.g[c] * bg.dal2[c] * dal2 / bg.f[c] : 0.0f;
        const float S = w.keep ? -w.acc[c] : w.C[c] - w.acc[c];
        galb[c] += qa[c] * S;
        grough += qr[c] * S;
      }
    }
    if (w.keep && go) {
      const int k = kept.n++;
      kept.m[k] = m * 2;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        kept.v[k][c] = galb[c];
        kept.v[k][4 + c] = qa[c];
        kept.v[k][7 + c] = qr[c];
      }
      kept.v[k][3] = grough;
    } else {
      sink.albedo_rough(m, galb[0], galb[1], galb[2], grough);
    }
    if (!go) return false;
    w.last_pdf = e.pdf;
    float cos_i = nx2 * pnx + (ny2 * pny + nz2 * pnz);
    w.thr[0] *= e.r * cos_i / e.pdf;
    w.thr[1] *= e.g * cos_i / e.pdf;
    w.thr[2] *= e.b * cos_i / e.pdf;
    w.prev_sumW = cur_sumW; w.prev_M = cur_M;
    w.prev_b[0] = e.r; w.prev_b[1] = e.g; w.prev_b[2] = e.b; w.prev_cos = cos_i;
    w.ox = hit.px + pnx * 0.001f;
    w.oy = hit.py + pny * 0.001f;
    w.oz = hit.pz + pnz * 0.001f;
    w.dx = nx2; w.dy = ny2; w.dz = nz2;
  }
#pragma unroll
  for (int c = 0; c < 3; ++c)
    if (w.thr[c] < 0.0f) w.thr[c] = 0.0f;
  float mx = fmaxf(w.thr[0], w.thr[1]);
  mx = fmaxf(mx, w.thr[2]);
  if (!(mx >= 1e-12f)) return false;
  if (p.rr && w.bounce >= 1) {
    float rr = mx;
    if (rr < 0.05f) rr = 0.05f;
    if (rr > 0.9f) rr = 0.9f;
    if (!(pt.U() <= rr)) return false;
    float ir = 1.0f / rr;
#pragma unroll
    for (int c = 0; c < 3; ++c) w.thr[c] *= ir;
  }
  return ++w.bounce < w.max_bounces;
}

// The end of a walk that kept its terms: acc is the sample's radiance C.
__device__ __forceinline__ void adjoint_end(const Walk& w, const GradSink& sink, const Kept& kept) {
  const float gC = w.g[0] * w.acc[0] + w.g[1] * w.acc[1] + w.g[2] * w.acc[2];
#pragma unroll 1
  for (int k = 0; k < kept.n; ++k) {
    const int m = kept.m[k] >> 1;
    if (kept.m[k] & 1) {
      sink.ior_rough(m, kept.v[k][0] + kept.v[k][2] * gC, kept.v[k][1] + kept.v[k][3] * gC);
    } else {
      const float* v = kept.v[k];
      sink.albedo_rough(m, v[0] + v[4] * w.acc[0], v[1] + v[5] * w.acc[1], v[2] + v[6] * w.acc[2],
                        v[3] + v[7] * w.acc[0] + v[8] * w.acc[1] + v[9] * w.acc[2]);
    }
  }
}

// The light sample of a kind-1 pixel's reservoir (pathtrace.metal:1100-1128):
// its contribution pd = Le f k, the factor k, direction, emission and light.
struct HeldLight {
  float pd[3], k, dx, dy, dz, le[3], sumWu;
  uint32_t M;
  int light;
};
struct Primary {  // a kind-1 pixel's first hit
  float px, py, pz, nx, ny, nz, wox, woy, woz, ar, ag, ab, rough, metallic, alpha2, spec_prob;
};

__device__ __forceinline__ Primary primary(const GBufSoA& gb, uint32_t id) {
  const float4 PK = gb.pos_kind[id], NR = gb.nor_rough[id], AM = gb.alb_met[id], WO = gb.wo_ior[id];
  Primary q;
  q.px = PK.x; q.py = PK.y; q.pz = PK.z;
  q.nx = NR.x; q.ny = NR.y; q.nz = NR.z;
  q.wox = WO.x; q.woy = WO.y; q.woz = WO.z;
  q.ar = AM.x; q.ag = AM.y; q.ab = AM.z;
  float rough = NR.w; if (rough < 0.0f) rough = 0.0f; if (rough > 1.0f) rough = 1.0f;
  float metallic = AM.w; if (metallic < 0.0f) metallic = 0.0f; if (metallic > 1.0f) metallic = 1.0f;
  float r2 = rough; if (r2 < 0.02f) r2 = 0.02f;
  q.rough = rough; q.metallic = metallic;
  q.alpha2 = (r2 * r2) * (r2 * r2);
  q.spec_prob = 0.05f + 0.95f * metallic; if (q.spec_prob > 0.98f) q.spec_prob = 0.98f;
  if (metallic >= 0.999f) q.spec_prob = 1.0f;
  return q;
}

__device__ __noinline__ HeldLight held_light(const Params& p, const ResSoA& rm, uint32_t id, const Primary& q) {
  HeldLight h;
  h.pd[0] = h.pd[1] = h.pd[2] = h.k = h.dx = h.dy = h.dz = h.le[0] = h.le[1] = h.le[2] = h.sumWu = 0.0f;
  h.M = 0;
  h.light = -1;
  const float4 R3 = rm.sumwu_m_valid[id];
  const float4 R0 = rm.lp_alpha[id], R1 = rm.ln_phat[id], R2 = rm.le_sumws[id];
  if (__float_as_int(R3.z) != 0 && __float_as_int(R3.y) != 0 && R3.x > 0.0f && R2.w > 0.0f && R1.w > 0.0f) {
    h.sumWu = R3.x; h.M = uint32_t(__float_as_int(R3.y));
    float ldx = R0.x - q.px, ldy = R0.y - q.py, ldz = R0.z - q.pz;
    float dist = sqrtf(ldx * ldx + ldy * ldy + ldz * ldz);
    if (dist > 0.003f) {
      float inv = 1.0f / dist;
      float dxn = ldx * inv, dyn = ldy * inv, dzn = ldz * inv;
      float lcos = -(R1.x * dxn + (R1.y * dyn + R1.z * dzn));
      float scos = q.nx * dxn + (q.ny * dyn + q.nz * dzn);
      if (lcos > 1e-8f && scos > 1e-8f) {
        Bsdf e = Tracer::eval_bsdf(dxn, dyn, dzn, q.wox, q.woy, q.woz, q.nx, q.ny, q.nz, q.alpha2, q.metallic,
                                   q.spec_prob, q.ar, q.ag, q.ab);
        float Fr = R2.x * e.r * scos * R0.w, Fg = R2.y * e.g * scos * R0.w, Fb = R2.z * e.b * scos * R0.w;
        float ph = lum3(Fr, Fg, Fb);
        if (ph > 0.0f) {
          float pdf_ris = float(h.M) * ph / h.sumWu;
          float wnee = 1.0f;
          if (!p.nomis && e.pdf > 1e-20f) wnee = pdf_ris / (pdf_ris + e.pdf);
          float Wt = R2.w / (float(h.M) * ph);
          h.pd[0] = Fr * Wt * wnee; h.pd[1] = Fg * Wt * wnee; h.pd[2] = Fb * Wt * wnee;
          h.k = scos * R0.w * Wt * wnee;
          h.dx = dxn; h.dy = dyn; h.dz = dzn;
          h.le[0] = R2.x; h.le[1] = R2.y; h.le[2] = R2.z;
          h.light = __float_as_int(R3.w);
        }
      }
    }
  }
  return h;
}

// The samples of K1 / K2 in their lanes' order (pathtrace.metal:749-758,
// :787-796), or (kRestir) the adjoint of K5, the ReSTIR shade (:1056-1258),
// from the frame's checkpoint: its G-buffer and merged reservoirs (the light
// sample each kind-1 pixel shades, with its light index) stay as the forward
// pass left them, and the pixel's K5 draws are replayed.  Kind-3 pixels (a
// dielectric first hit) are camera paths, as in K1.  A kind-1 pixel's value
// is the mean over samples of clamp(base + C_s): base = the first hit's
// emission + the reservoir sample's Le f cos alpha W w_MIS (sample, W and MIS
// weight held), C_s an indirect path that leaves the first hit with the BSDF
// sample B_0 = f cos / pdf and goes on as a camera path's vertices do (a walk
// from the first hit; Russian roulette from its second vertex).  d(base) moves
// with the first hit's emission, albedo and roughness and the sampled light's
// emission; C_s with its vertices (the walk) and with B_0 (dlog B_0 * C_s).
// The first hit's material is found by tracing K3's primary ray again
// (pathtrace.metal:829-840).
//
// A warp's lanes take pixel lanes from a counter (*next) and advance one vertex
// per pass, so that no lane waits for the others' paths.  A sample whose value
// is clamped in some channel is walked a second time with -g on that channel,
// which takes its terms back out (rare).
//
// Bound by instruction fetch and by the traversal's loads: as many
// instructions as the forward frame (7.2 and 6.5 G warp instructions at
// 512 x 512, 32 spp, 8 bounces, 200 k triangles), but the code of a vertex
// with its derivatives is larger than the instruction cache that the four
// schedulers share, so everything that can be one copy is one (the traversal,
// bsdf_grad, the additions, no alpha code in opaque scenes): that frame's
// adjoint 21.8 -> 18.9 ms by the loop, -> 17.1 by the copies.  Sixteen warps an
// SM (12: +0.6 ms, 20: no change).  One block of 512 threads: 4 of 128 take the
// same time but add 592 partial sums to each gradient instead of 148.
constexpr int kAdjThreads = 512, kAdjBlocks = 1;
constexpr int kAdjRefill = 16;  // idle lanes of a warp that make it take new pixel lanes

// A block's sums are of 32 bits, and so is the gradient: a sum of many terms and
// many sums are both inexact.  So a block holds two arrays of sums where they
// fit in 32 KB: terms go to the first, which passes on to the second about each
// time the block has taken this many pixel lanes (a warp's turn comes every 256
// of its own, the warps' turns evenly spread), and the second goes to the gradient
// at the end.  (One array passes on to the gradient itself.)
// Error against the sum of 64 bands' gradients in 64 bits: 512x512, 32 spp 2.0e-7
// of the gradient, 1024x1024, 32 spp 1.9e-7; with the first array passed on to the
// gradient 1.1e-6 and 1.4e-6, with one that is never passed on 3.0e-7 and 4.5e-7,
// but 1.6e-3 where all terms are equal (1024x1024, 100 spp), which the two
// hold to 9e-6.  The second array costs nothing at 512x512, 32 spp (10.65 ms) and
// 2 % at 256x256, 16 spp (2.40 -> 2.44).
constexpr unsigned kAdjFlush = 256;

struct AdjointArgs {
  const int32_t* tri_mat;
  int n_mat;
  const float* dLdI;
  const float* dLdalb;  // kRestir: through the denoiser's weights, or null
  float* grad;
  int sums, lanes;  // sums: arrays of n_mat x 8 sums in the block's memory (0: none)
  unsigned flush;   // pixel lanes of a warp between its turns to pass the sums on
  unsigned* next;
  unsigned long long* ctr;
  uint32_t* err;
};

// The block's n sums to its second array (grad null) or to the gradient, by one
// warp; a copy of its own, called seldom.
__device__ __noinline__ void pass_sums_on(int n, float* grad) {
#pragma unroll 1
  for (int i = int(threadIdx.x & 31); i < n; i += 32) {
    const float v = sh_sums[i] != 0.0f ? atomicExch(sh_sums + i, 0.0f) : 0.0f;
    if (v == 0.0f) continue;
    if (grad) atomicAdd(grad + i, v);
    else atomicAdd(sh_sums + n + i, v);
  }
}

template <int kNee, bool kRestir>
__global__ void __launch_bounds__(kAdjThreads, kAdjBlocks) k_adjoint(Scene s, Params p, uint64_t seed, GBufSoA gb,
                                                                     ResSoA rm, AdjointArgs a) {
  float* sh = sh_sums;
  const int n_sums = a.n_mat * kMatParams;
  if (a.sums > 0) {
    for (int i = threadIdx.x; i < n_sums * a.sums; i += blockDim.x) sh[i] = 0.0f;
    __syncthreads();
  }
  const unsigned full = 0xffffffffu;
  const GradSink sink{a.sums > 0, a.grad};
  const int lane_id = int(threadIdx.x & 31);
  const unsigned L = unsigned(a.lanes);
  const unsigned tasks = unsigned(p.width) * unsigned(p.height) * L;
  const float inv_n = 1.0f / float(p.spp);
  const bool cl = p.clamp_value > 0.0f;
  Tracer pt(s, p, a.err);
  Walk w;
  Kept kept;
  bool active = false, fresh = false, again = false, more = true, indirect = false;
  // pixel lanes that the warp took since it last passed the block's sums on; its
  // turns lie evenly between the other warps'
  unsigned taken = threadIdx.x / 32 * (a.flush / (blockDim.x / 32));
  // mode of the walk: 0 the only one (terms kept), 1 with C known, 2 for C alone
  int mode = 0, si = 0;
  uint32_t id = 0, start_state = 0, samples = 0;
  // kRestir: the pixel's first hit (material, texel, roughness factor), base and the gradient reaching it,
  // the direction of the current sample's first BSDF sample
  int m0 = -1;
  bool alb0 = false;
  float tx0[3] = {1.f, 1.f, 1.f}, dal0 = 0.0f, base[3] = {0.f, 0.f, 0.f}, gbase[3] = {0.f, 0.f, 0.f};
  float b0x = 0, b0y = 0, b0z = 0;
  for (;;) {
    const unsigned idle = __ballot_sync(full, !active);
    if (more && __popc(idle) >= kAdjRefill) {
      unsigned first = 0;
      if (lane_id == 0) first = atomicAdd(a.next, unsigned(__popc(idle)));
      first = __shfl_sync(full, first, 0);
      taken += unsigned(__popc(idle));
      if (taken >= a.flush) {
        taken -= a.flush;
        pass_sums_on(n_sums, a.sums == 2 ? nullptr : a.grad);
      }
      more = first + unsigned(__popc(idle)) < tasks;
      const unsigned t = first + unsigned(__popc(idle & ((1u << lane_id) - 1u)));
      if (!active && t < tasks && t >= first) {
        id = t / L;
        const unsigned lane = t % L;
        const uint32_t x = id % uint32_t(p.width), y = id / uint32_t(p.width);
        si = int(lane);
        active = si < p.spp;
        indirect = false;
        if (!kRestir) {
          uint64_t sd = seed_pixel(seed, x, y);
          if (L > 1) sd ^= uint64_t(lane) * 0x94D049BB133111EBull;
          pt.rng.seed(sd);
        } else {
          const int kind = __float_as_int(gb.pos_kind[id].w);
          active = kind != 0;
          indirect = kind == 1;
          m0 = -1;
          alb0 = false;
          if (kind == 1 || (kind != 0 && a.dLdalb)) {
            // the first hit's triangle: K3's primary ray (its own random stream)
            pt.rng.seed(seed_pixel(seed, x, y));
            float sx = float(x) + 1e-12f + (p.resolution - 2e-12f) * pt.U() - float(p.width) * 0.5f;
            float sy = float(p.height) * 0.5f - (float(y) + 1e-12f + (p.resolution - 2e-12f) * pt.U());
            const rm_camera& c = p.camera;
            float f2 = c.focal * c.focal;
            float dinv = 1.0f / sqrtf(sx * sx + sy * sy + f2);
            float tx = sx * dinv, ty = sy * dinv, tz = c.focal * dinv;
            float rdx = tx * c.m0 + (ty * c.m1 + tz * c.m2);
            float rdy = tx * c.m3 + (ty * c.m4 + tz * c.m5);
            float rdz = tx * c.m6 + (ty * c.m7 + tz * c.m8);
            const Hit h0 = pt.cast_ray(c.x, c.y, c.z, rdx, rdy, rdz, kFar);
            if (h0.tri >= 0) {
              m0 = a.tri_mat[h0.tri];
              tx0[0] = h0.txr; tx0[1] = h0.txg; tx0[2] = h0.txb;
              alb0 = h0.shader != 1;
              dal0 = dalpha2(h0.rough);
            }
          }
          // the denoiser's weights through this pixel's G-buffer albedo (the first
          // hit's albedo times its texel)
          if (a.dLdalb && alb0) {
            const float* d = a.dLdalb + size_t(id) * 3;
            sink.albedo_rough(m0, d[0] * tx0[0], d[1] * tx0[1], d[2] * tx0[2], 0.0f);
          }
          pt.rng.seed(seed ^ (uint64_t(id + 1) * 0xBF58476D1CE4E5B9ull) ^ 0x94D049BB133111EBull);
          if (indirect) {
            const HeldLight h = held_light(p, rm, id, primary(gb, id));
            const float4 EM = gb.emi[id];
            base[0] = EM.x + h.pd[0]; base[1] = EM.y + h.pd[1]; base[2] = EM.z + h.pd[2];
            gbase[0] = gbase[1] = gbase[2] = 0.0f;
            if (p.bounces <= 1) {
              for (int c = 0; c < 3; ++c)
                gbase[c] = (cl && !(base[c] < p.clamp_value)) ? 0.0f : a.dLdI[size_t(id) * 3 + c];
              si = p.spp;  // no indirect samples
            }
          }
        }
        fresh = active;
        again = false;
      }
    }
    if (!__any_sync(full, active)) {
      if (!more) break;
      continue;
    }
    if (fresh) {
      // start the next sample's walk, or (again) the same sample's second one
      fresh = false;
      float g[3];
      for (int c = 0; c < 3; ++c) g[c] = a.dLdI[size_t(id) * 3 + c] * inv_n;
      if (kRestir && indirect) {
        const Primary q = primary(gb, id);
        const HeldLight h = held_light(p, rm, id, q);
        float nx2 = b0x, ny2 = b0y, nz2 = b0z;
        int pdelta = 0;
        Bsdf e0{0.f, 0.f, 0.f, 0.f};
        if (again) pt.rng.state = start_state;
        while (si < p.spp) {
          if (!again) start_state = pt.rng.state;
          bool early = false;
          if (pt.U() < q.spec_prob) {
            float hx, hy, hz;
            pt.sample_ggx_half(q.alpha2, q.nx, q.ny, q.nz, hx, hy, hz);
            float md = q.wox * hx + (q.woy * hy + q.woz * hz);
            if (!(md > 1e-8f)) early = true;
            else {
              nx2 = 2.0f * md * hx - q.wox; ny2 = 2.0f * md * hy - q.woy; nz2 = 2.0f * md * hz - q.woz;
              pdelta = (q.rough <= 0.0201f) ? 1 : 0;
            }
          } else {
            pt.sample_cosine(q.nx, q.ny, q.nz, nx2, ny2, nz2);
            pdelta = 0;
          }
          if (!early) {
            float ncos = nx2 * q.nx + (ny2 * q.ny + nz2 * q.nz);
            if (!(ncos > 1e-8f)) early = true;
            else {
              float d = 1.0f / sqrtf(nx2 * nx2 + ny2 * ny2 + nz2 * nz2);
              nx2 *= d; ny2 *= d; nz2 *= d;
              e0 = Tracer::eval_bsdf(nx2, ny2, nz2, q.wox, q.woy, q.woz, q.nx, q.ny, q.nz, q.alpha2, q.metallic,
                                     q.spec_prob, q.ar, q.ag, q.ab);
              if (!(e0.pdf > 1e-12f)) early = true;
            }
          }
          if (!early) break;
          for (int c = 0; c < 3; ++c) gbase[c] += (cl && !(base[c] < p.clamp_value)) ? 0.0f : g[c];
          ++samples;
          ++si;
        }
        if (si < p.spp) {
          const float cos0 = nx2 * q.nx + (ny2 * q.ny + nz2 * q.nz);
          w.thr[0] = e0.r * cos0 / e0.pdf; w.thr[1] = e0.g * cos0 / e0.pdf; w.thr[2] = e0.b * cos0 / e0.pdf;
          w.last_pdf = e0.pdf;
          w.prev_b[0] = e0.r; w.prev_b[1] = e0.g; w.prev_b[2] = e0.b; w.prev_cos = cos0;
          w.prev_sumW = h.sumWu; w.prev_M = h.M; w.prev_delta = pdelta;
          w.ox = q.px + q.nx * 0.001f; w.oy = q.py + q.ny * 0.001f; w.oz = q.pz + q.nz * 0.001f;
          w.dx = b0x = nx2; w.dy = b0y = ny2; w.dz = b0z = nz2;
          w.max_bounces = p.bounces - 1;
          w.camera = false;
        } else {
          // every sample is done: the base's terms, the first hit's emission and
          // the held light sample Le f k
          sink.emission(m0, gbase[0], gbase[1], gbase[2]);
          if (h.light >= 0 && h.k != 0.0f) {
            const int ml = a.tri_mat[s.lights[h.light]];
            const BsdfGrad bg = bsdf_grad(h.dx, h.dy, h.dz, q.wox, q.woy, q.woz, q.nx, q.ny, q.nz, q.alpha2,
                                          q.metallic, q.ar, q.ag, q.ab);
            float drough = 0.0f, gle[3], ga[3];
            for (int c = 0; c < 3; ++c) {
              const float gt = gbase[c] * h.k;
              gle[c] = gt * bg.f[c];
              ga[c] = alb0 ? gt * h.le[c] * bg.da[c] * tx0[c] : 0.0f;
              drough += gt * h.le[c] * bg.dal2[c];
            }
            sink.emission(ml, gle[0], gle[1], gle[2]);
            sink.albedo_rough(m0, ga[0], ga[1], ga[2], drough * dal0);
          }
          active = false;
        }
      } else {
        if (again) pt.rng.state = start_state;
        else start_state = pt.rng.state;
        walk_camera(w, pt, id % uint32_t(p.width), id / uint32_t(p.width));
      }
      w.bounce = 0;
      if (!again) {
        mode = w.max_bounces <= Kept::kMax ? 0 : 2;
        for (int c = 0; c < 3; ++c) w.g[c] = g[c];
        w.C[0] = w.C[1] = w.C[2] = 0.0f;
      } else {
        // the second walk: what the first left undone (for C alone), or -g on
        // the clamped channels (the sample enters the pixel mean clamped,
        // pathtrace.metal:757)
        for (int c = 0; c < 3; ++c) {
          w.C[c] = w.acc[c];
          const bool cut = cl && !((indirect ? base[c] : 0.0f) + w.acc[c] < p.clamp_value);
          w.g[c] = mode == 2 ? (cut ? 0.0f : g[c]) : (cut ? -g[c] : 0.0f);
        }
        mode = 1;
      }
      w.keep = mode == 0;
      w.mute = mode == 2;
      w.acc[0] = w.acc[1] = w.acc[2] = 0.0f;
      kept.n = 0;
      again = false;
    }
    if (active) {
      const bool go = w.bounce < w.max_bounces && adjoint_step<kNee>(pt, a.tri_mat, w, sink, kept);
      if (!go) {
        if (mode == 0) adjoint_end(w, sink, kept);
        bool cut = false;
        if (mode != 1)
          for (int c = 0; c < 3; ++c)
            cut = cut || (cl && !((indirect ? base[c] : 0.0f) + w.acc[c] < p.clamp_value));
        if (kRestir && indirect && mode != 1) {
          // B_0 = f cos / pdf: dlog B_0 = df / f, times the walk's radiance C
          const Primary q = primary(gb, id);
          const BsdfGrad bg = bsdf_grad(b0x, b0y, b0z, q.wox, q.woy, q.woz, q.nx, q.ny, q.nz, q.alpha2, q.metallic,
                                        q.ar, q.ag, q.ab);
          float drough = 0.0f, ga[3] = {0.f, 0.f, 0.f};
          for (int c = 0; c < 3; ++c) {
            const float ge = (cl && !(base[c] + w.acc[c] < p.clamp_value)) ? 0.0f : a.dLdI[size_t(id) * 3 + c] * inv_n;
            gbase[c] += ge;
            if (!(bg.f[c] > 0.0f)) continue;
            const float v = ge * w.acc[c] / bg.f[c];
            if (alb0) ga[c] = v * bg.da[c] * tx0[c];
            drough += v * bg.dal2[c];
          }
          sink.albedo_rough(m0, ga[0], ga[1], ga[2], drough * dal0);
        }
        fresh = true;
        if (mode == 2 || cut) {
          again = true;
        } else {
          ++samples;
          si += int(L);
          if (!indirect && si >= p.spp) active = fresh = false;  // (an indirect pixel ends at its next start)
        }
      }
    }
  }
  __syncwarp();
  const unsigned long long tot = __reduce_add_sync(full, samples);
  if (lane_id == 0 && tot) atomicAdd(a.ctr, tot);
  if (a.sums > 0) {
    __syncthreads();
    for (int i = threadIdx.x; i < n_sums; i += blockDim.x) {
      const float v = a.sums == 2 ? sh[n_sums + i] + sh[i] : sh[i];
      if (v != 0.0f) atomicAdd(a.grad + i, v);
    }
  }
}

// Copy per-material parameters into the triangles (albedo, rough, emission, ior).
__global__ void k_apply_materials(rm_triangle* tris, const int32_t* __restrict__ tri_mat,
                                  const float* __restrict__ mats, int n_tris) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_tris) return;
  const int m = tri_mat[i];
  if (m < 0) return;
  const float* q = mats + size_t(m) * kMatParams;
  rm_triangle& t = tris[i];
  t.ar = q[0]; t.ag = q[1]; t.ab = q[2];
  t.rough = q[3];
  t.er = q[4]; t.eg = q[5]; t.eb = q[6];
  t.ior = q[7];
}

}  // namespace

namespace {

template <bool kRestir>
cudaError_t run_adjoint(const Scene& s, const Params& p, uint64_t seed, const GBufSoA& gb, const ResSoA& rm,
                        AdjointArgs a, int sms, cudaStream_t st) {
  const size_t one = size_t(a.n_mat) * kMatParams * sizeof(float);
  a.sums = one * 2 <= 32 * 1024 ? 2 : one <= 32 * 1024 ? 1 : 0;
  const size_t threads = size_t(p.width) * size_t(p.height) * size_t(a.lanes);
  a.flush = kAdjFlush;
  // fewer pixel lanes than the GPU's threads: narrower blocks, one on each SM
  // (64x64, 2 spp 0.72 ms against 0.84, its ReSTIR frame 1.30 / 1.51, 130x97, 8
  // spp 4.04 / 4.50)
  const size_t per_sm = (threads + size_t(sms) * 32 - 1) / (size_t(sms) * 32) * 32;
  const unsigned block = unsigned(std::min<size_t>(kAdjThreads, per_sm));
  const unsigned grid = unsigned(std::min<size_t>(size_t(sms) * kAdjBlocks, (threads + block - 1) / block));
  if (threads <= size_t(grid) * kAdjFlush && a.sums == 2) {
    // a block takes no more than one pass: the first array does (64x64 on the
    // ReSTIR chain 3.2 ms, with the second's memory gone from the cache 3.7)
    a.sums = 1;
    a.flush = 0xffffffffu;
  }
  if (a.sums == 0) a.flush = 0xffffffffu;
  const size_t sm = size_t(a.sums) * one;
  const cudaError_t e = cudaMemsetAsync(a.next, 0, sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  if (!kRestir && !p.opaque) k_adjoint<1, false><<<grid, block, sm, st>>>(s, p, seed, gb, rm, a);
  else if (p.restir_candidates > 1) k_adjoint<2, kRestir><<<grid, block, sm, st>>>(s, p, seed, gb, rm, a);
  else k_adjoint<0, kRestir><<<grid, block, sm, st>>>(s, p, seed, gb, rm, a);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_adjoint(int lanes, const Scene& s, const Params& p, uint64_t seed, const int32_t* tri_mat,
                           int n_mat, const float* dLdI, float* grad, unsigned* next, int sms, unsigned long long* ctr,
                           uint32_t* err, cudaStream_t st) {
  return run_adjoint<false>(s, p, seed, GBufSoA{}, ResSoA{},
                            AdjointArgs{tri_mat, n_mat, dLdI, nullptr, grad, 0, lanes, 0, next, ctr, err}, sms, st);
}

cudaError_t apply_materials(rm_triangle* tris, const int32_t* tri_mat, const float* mats, int n_tris,
                            cudaStream_t st) {
  if (n_tris <= 0) return cudaSuccess;
  k_apply_materials<<<(n_tris + 255) / 256, 256, 0, st>>>(tris, tri_mat, mats, n_tris);
  return cudaGetLastError();
}

cudaError_t launch_adjoint_restir(const Scene& s, const Params& p, uint64_t seed, const GBufSoA& gb, const ResSoA& rm,
                                  const int32_t* tri_mat, int n_mat, const float* dLdI, const float* dLdalb,
                                  float* grad, unsigned* next, int sms, unsigned long long* ctr, uint32_t* err,
                                  cudaStream_t st) {
  return run_adjoint<true>(s, p, seed, gb, rm,
                           AdjointArgs{tri_mat, n_mat, dLdI, dLdalb, grad, 0, 1, 0, next, ctr, err}, sms, st);
}

}  // namespace rmd
