// pixel.cuh -- the pixel function shared by the single-scene pixel kernel
// (trace.cu) and the batched form's render (batch_kernel.cuh).
#pragma once
#include "crt_internal.h"

namespace crt {

namespace {

enum PixelMode { kRender = 0, kRenderStats = 1, kAdjoint = 2 };

// Warp-reduced atomic add of a double (light gradient: few addresses).
__device__ __forceinline__ void warp_add(double* dst, double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v != 0.0) atomicAdd(dst, v);
}

// The mean colour of a pixel, in every form asked for.
__device__ __forceinline__ void write_pixel(const RenderArgs& A, int idx, D3 c) {
  if (A.rgbf) {
    A.rgbf[3 * (int64_t)idx] = (float)c.x;
    A.rgbf[3 * (int64_t)idx + 1] = (float)c.y;
    A.rgbf[3 * (int64_t)idx + 2] = (float)c.z;
  }
  if (A.rgbd) {
    A.rgbd[3 * (int64_t)idx] = c.x;
    A.rgbd[3 * (int64_t)idx + 1] = c.y;
    A.rgbd[3 * (int64_t)idx + 2] = c.z;
  }
  if (A.rgb8) {
    const double cc[3] = {c.x, c.y, c.z};
#pragma unroll
    for (int ch = 0; ch < 3; ch++) {
      double v = cc[ch];
      if (v < 0) v = 0.0;
      if (v > 1) v = 1.0;
      A.rgb8[3 * (int64_t)idx + ch] = (uint8_t)(255.0 * v);
    }
  }
}

// True when no camera ray of a block of pixels can hit anything: pixels x0..x1
// by y0..y1, every point of the lens.  All 32 lanes call it with the same
// arguments.
//
// A ray starts at (ox, oy, 0), |ox|, |oy| <= R = aperture / 2, and goes through
// lambda (x, y, -1), lambda = focal / |(x, y, -1)|, so at depth z its line is at
//   x(z) = -z x + (1 + z / lambda) ox
// (y alike): over a box's z range and the block's x, y and lambda that is an
// interval, and a box clear of it in x or y is clear of every line.  (A hit
// needs its triangle's box to pass the exact slab test on the ray's line,
// either way along it; FP32 roundings, the float root inside normalize() and
// the test's own double roundings are covered by 2^-16 of the interval's
// terms and 2^-18 of the scene.)  The warp walks the tree breadth first, eight
// nodes and their 32 slots a round; a leaf or more than eight nodes in the
// beam, or kBeamRounds rounds, end the walk without an answer.
//
// A block that misses is a constant, and without this a wave of 32 missing
// samples takes some 70 to 125 double instructions (rays, sums, divisions) at
// 16 cycles of the SM each and 64 random table loads, where the beam takes
// about a hundred single ones a round.  1,003,520 triangles: 1920x1080 at 16
// samples, 83% of them misses, 16.4 -> 13.8 ms; 1280x720 at 4, 2.83 -> 2.35 ms
// (4 rounds 14.4 ms, 6 14.0, 8 13.9, 10 13.8); a soup that fills the view shows
// no difference.
constexpr int kBeamRounds = 8;
constexpr int kBeamNodes = 8;
__device__ __forceinline__ bool beam_misses(const DScene& S, const RenderArgs& A, const float rb[6], float B, int x0,
                                            int x1, int y0, int y1) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const float focal = (float)A.focal, R = 0.5f * fabsf((float)A.aperture);
  // the block in the plane z = -1 (an upper edge of a pixel row is its lower y)
  const float sx = (float)(A.angle * A.aspect), sy = (float)A.angle;
  const float ex = fabsf(sx) * 4e-6f, ey = fabsf(sy) * 4e-6f;
  const float iw = 2.f / (float)A.W, ih = 2.f / (float)A.H;
  float ax = (((float)x0 + 0.5f) * iw - 1.f) * sx, bx = (((float)x1 + 0.5f) * iw - 1.f) * sx;
  float ay = (1.f - ((float)y1 + 0.5f) * ih) * sy, by = (1.f - ((float)y0 + 0.5f) * ih) * sy;
  const float xl = fminf(ax, bx) - ex, xh = fmaxf(ax, bx) + ex, yl = fminf(ay, by) - ey, yh = fmaxf(ay, by) + ey;
  const float mx = fmaxf(fabsf(xl), fabsf(xh)), my = fmaxf(fabsf(yl), fabsf(yh));
  // 1 / lambda over the block, widened
  const float nmax = sqrtf(1.f + mx * mx + my * my) * 1.000001f;
  const float il = 0.999999f / fabsf(focal), ih2 = nmax / fabsf(focal) * 1.000001f;
  // (anything out of the ordinary: no answer)
  if (!(fabsf(focal) > 1e-6f && fabsf(focal) < 1e12f && R < 1e12f && mx < 1e6f && my < 1e6f && B <= 1e18f)) return false;
  const float pad = 3.8146973e-06f * B;
  auto clear = [&](float lx, float hx, float ly, float hy, float lz, float hz) {
    const float z = fmaxf(fabsf(lz), fabsf(hz));
    // |1 + z / lambda| over z in [lz, hz], 1 / lambda in [il, ih2] (with the sign of focal)
    const float s = focal > 0.f ? 1.f : -1.f;
    const float a0 = fabsf(1.f + s * lz * il), a1 = fabsf(1.f + s * lz * ih2), a2 = fabsf(1.f + s * hz * il),
                a3 = fabsf(1.f + s * hz * ih2);
    const float lens = R * (fmaxf(fmaxf(a0, a1), fmaxf(a2, a3)) + 1.5258789e-05f * (1.f + z * ih2));
    const float px = lens + 1.5258789e-05f * z * mx + pad, py = lens + 1.5258789e-05f * z * my + pad;
    const float x00 = -lz * xl, x01 = -lz * xh, x10 = -hz * xl, x11 = -hz * xh;
    const float y00 = -lz * yl, y01 = -lz * yh, y10 = -hz * yl, y11 = -hz * yh;
    const float qxl = fminf(fminf(x00, x01), fminf(x10, x11)) - px, qxh = fmaxf(fmaxf(x00, x01), fmaxf(x10, x11)) + px;
    const float qyl = fminf(fminf(y00, y01), fminf(y10, y11)) - py, qyh = fmaxf(fmaxf(y00, y01), fmaxf(y10, y11)) + py;
    return qxh < lx || qxl > hx || qyh < ly || qyl > hy;
  };
  if (S.ntri <= 0) return true;
  if (clear(rb[0], rb[3], rb[1], rb[4], rb[2], rb[5])) return true;
  if (S.root < 0) return false;
  int count = 1, node = S.root;  // lane j < count holds node j of the round
  for (int round = 0; round < kBeamRounds; round++) {
    const int mine = __shfl_sync(full, node, lane >> 2), slot = lane & 3;
    bool in = false;
    int code = kNoChild;
    if ((lane >> 2) < count) {
      if (mine < 0 || mine >= S.ntri - 1) {  // only a corrupt tree gets here
        in = true, code = -1;
      } else {
        const WNode* w = S.wnodes + mine;
        code = w->code[slot];
        if (code != kNoChild) {
          float lo[3], hi[3];
#pragma unroll
          for (int k = 0; k < 3; k++) {
            const float o = w->o[k], s15 = w->s15[k];
            const uint32_t one = 0x3F800000u, ql = (w->lo[k] >> (8 * slot)) & 255u, qh = (w->hi[k] >> (8 * slot)) & 255u;
            lo[k] = __fmaf_rd(__uint_as_float(one | (ql << 8)), s15, o);
            hi[k] = __fmaf_ru(__uint_as_float(one | (qh << 8)), s15, o);
          }
          in = !clear(lo[0], hi[0], lo[1], hi[1], lo[2], hi[2]);
        }
      }
    }
    const unsigned m = __ballot_sync(full, in);
    if (m == 0u) return true;
    if (__any_sync(full, in && code < 0) || __popc(m) > kBeamNodes) return false;
    // the nodes in the beam move to lanes 0, 1, ...
    count = __popc(m);
    const int src = __fns(m, 0, lane + 1);
    node = __shfl_sync(full, code, src & 31);
  }
  return false;
}

// sum / spp: a power of two's inverse is exact, and so is the product's rounding.
__device__ __forceinline__ double sample_mean(double sum, int spp) {
  if ((spp & (spp - 1)) == 0) return sum * __hiloint2double((1023 - (31 - __clz(spp))) << 20, 0);
  return sum / (double)spp;
}

// Lane j of every four lanes has a row v0..v3; afterwards it has column j.
__device__ __forceinline__ void swap_if(bool p, double& a, double& b) {
  const double t = p ? b : a;
  b = p ? a : b;
  a = t;
}
__device__ __forceinline__ void quad_transpose(double& v0, double& v1, double& v2, double& v3) {
  const unsigned full = 0xffffffffu;
  const bool b0 = threadIdx.x & 1, b1 = threadIdx.x & 2;
  swap_if(b0, v0, v1), swap_if(b0, v2, v3), swap_if(b1, v0, v2), swap_if(b1, v1, v3);
  v1 = __shfl_xor_sync(full, v1, 1), v2 = __shfl_xor_sync(full, v2, 2), v3 = __shfl_xor_sync(full, v3, 3);
  swap_if(b0, v0, v1), swap_if(b0, v2, v3), swap_if(b1, v0, v2), swap_if(b1, v1, v3);
}

// The pixel this lane would have shaded, when the block's beam misses: every
// sample is a miss.  mean: 0.9 summed spp times in double and divided by spp,
// as the samples would be.
__device__ __forceinline__ double miss_mean(int spp) {
  double a = 0.0;
  for (int i = 0; i < spp; i++) a = a + 0.9;
  return sample_mean(a, spp);
}

// Writes a block's missing pixels (this lane's when it leads its group of G).
template <int MODE>
__device__ __forceinline__ void write_miss(const RenderArgs& A, int px, int py, bool valid, int G, double mean) {
  if (MODE == kAdjoint || !valid) return;  // (misses have no gradient)
  const int g = threadIdx.x & (G - 1);
  const int idx = (A.H - py - 1) * A.W + px;
  if (A.hit_id || A.hit_t || A.shadow || A.shadow_id)
    for (int k = g; k < A.spp; k += G) {
      const int64_t si = (int64_t)idx * A.spp + k;
      if (A.hit_id) A.hit_id[si] = -1;
      if (A.hit_t) A.hit_t[si] = 0.0;
      if (A.shadow) A.shadow[si] = -1;
      if (A.shadow_id) A.shadow_id[si] = -1;
    }
  if (g != 0) return;
  write_pixel(A, idx, d3(mean, mean, mean));
  if (A.depth) A.depth[idx] = 0.0;
}

// runRayTracerKernelRec (kernels/raytracer.cu:95-166) per pixel, with
// traceRay (raytracer.cu:169-249), Material::shade (kernels/material.cu:6-40)
// and the positional Light (kernels/Light.cu:5-86).  MODE kAdjoint re-runs the
// same samples (same rays, hits and shadow tests: nothing is stored between
// the forward and the adjoint) and accumulates d loss / d (vertices, light
// position, albedo) for the Lambert and distance terms; visibility (which
// triangle is hit, whether the shadow ray is blocked) is held fixed.
//
// All 32 lanes of the warp call it together.  G lanes (a power of two) share
// one pixel and trace G of its samples at once, in waves of G samples; valid
// false marks a pixel outside the image (its lanes compute and write
// nothing).  The samples of a pixel share one mrand stream: sample k draws
// two numbers for the lens and, when its primary ray hits, three for the
// light, so where sample k starts in the stream depends on which earlier
// samples hit.  Each lane guesses those hits (`pred`: the last wave's
// majority), traces, and the lanes whose guess of an earlier sample proved
// wrong trace again with the hits just observed; at least one more sample of
// every group is settled per round, and the settled rays are exactly the
// sequential ones.  Colours and depths are then summed in sample order; with four
// lanes or more each lane of four sums one of x, y, z and depth (an inactive
// lane's zeros change no sum: none is ever -0).
template <int MODE, int SHORT = 0, bool NC = true>
__device__ __forceinline__ void pixel(const DScene& S, const RenderArgs& A, int px, int py, bool valid, int G,
                                      unsigned& pred, float rb[6], float B, float D, TravStats& ts, D3& glight,
                                      int2* ring = nullptr) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int g = lane & (G - 1);
    const int base = lane - g;
    const unsigned gmask = (G == 32) ? full : (((1u << G) - 1u) << base);
    const unsigned below = gmask & ((1u << lane) - 1u);  // the lanes of my group before me
    const int gx = (A.W + 15) / 16;  // gridDim.x of the reference's 16x16 launch
    const D3 lpos = d3(A.lpos[0], A.lpos[1], A.lpos[2]);
    const int idx = (A.H - py - 1) * A.W + px;
    // getGlobalIdx_2D_2D (inc/indexing.h:4-9) of the pixel's thread in the
    // reference launch, seeded by initPNRG (kernels/mrand.cu:38-41).
    const uint32_t gid = (uint32_t)(((py / 16) * gx + px / 16) * 256 + (py % 16) * 16 + (px % 16));
    uint32_t wst = wang_hash(gid ^ A.seed_mix);  // stream position at the start of the wave
    const double xx = (2 * ((px + 0.5) * A.invW) - 1) * A.angle * A.aspect;
    const double yy = (1 - 2 * ((py + 0.5) * A.invH)) * A.angle;
    // the pinhole direction scaled to the focal plane: the same for every sample
    D3 fdir = normalize_exact(d3(xx, yy, -1.0));
    fdir = d3(fdir.x * A.focal, fdir.y * A.focal, fdir.z * A.focal);
    D3 acc = d3(0, 0, 0);
    double depth = 0.0;
    D3 G3 = d3(0, 0, 0);
    double Gd = 0.0;
    if (MODE == kAdjoint && valid) {
      const double inv = 1.0 / (double)A.spp;
      G3 = d3(A.grad_rgb[3 * (int64_t)idx] * inv, A.grad_rgb[3 * (int64_t)idx + 1] * inv,
              A.grad_rgb[3 * (int64_t)idx + 2] * inv);
      Gd = A.grad_depth ? A.grad_depth[idx] * inv : 0.0;
    }
    const int waves = (A.spp + G - 1) / G;
    for (int w = 0; w < waves; w++) {
      const int k = w * G + g;
      const bool act = valid && k < A.spp;
      const unsigned actm = __ballot_sync(full, act);
      const int64_t si = (int64_t)idx * A.spp + k;
      // primary rays, speculating on the hits of the group's earlier samples
      unsigned guess = pred;
      bool done = !act;
      HitRec h;
      int res = 0;
      D3 org = d3(0, 0, 0), dir = d3(0, 0, 1);
      uint32_t st = wst;
      unsigned hits;
      while (true) {
        RayC rc;
        if (!done) {
          st = wst;
          for (int t = 0; t < g; t++) {
            xorshift32(st);
            xorshift32(st);
            if ((guess >> (base + t)) & 1u) {
              xorshift32(st);
              xorshift32(st);
              xorshift32(st);
            }
          }
          // sincos gives sin and cos bit for bit (checked for every angle 2*pi*u
          // the float-valued mrand draw u can take)
          double ox, oy;
          lens_origin(A.lens_cs, A.lens_sqrt, A.aperture, st, ox, oy);
          org = d3(ox, oy, 0.0);
          dir = normalize_exact(fdir - org);
          ray_setup(rc, org.x, org.y, org.z, dir.x, dir.y, dir.z, B, D);
        } else {
          ray_setup(rc, 0.0, 0.0, 0.0, 0.0, 0.0, 1.0, B, D);
        }
        HitRec ht;
        const int r = traverse<false, MODE == kRenderStats, SHORT, NC, true>(S, rc, rb, ht, !done, &ts, ring);
        if (!done) h = ht, res = r;
        hits = __ballot_sync(full, act && res > 0);
        // a lane is settled when every earlier sample of its group was guessed right
        if (((guess ^ hits) & actm & below) == 0u) done = true;
        guess = hits;
        if (__all_sync(full, done)) break;
      }
      if (res < 0) atomicOr(&S.g->err, kErrStack);
      const bool hit = act && res > 0;
      if (MODE != kAdjoint && A.rays && act) {
        double* rr = A.rays + 6 * si;
        rr[0] = org.x, rr[1] = org.y, rr[2] = org.z, rr[3] = dir.x, rr[4] = dir.y, rr[5] = dir.z;
      }
      // traceRay up to the shadow ray (lanes with a hit): only what the
      // shadow ray needs is computed before it, to keep little state live
      // across the walk; the rest of the shading follows it
      D3 q, L;
      double sL = 0.0, dist = 0.0;
      RayC sr;
      if (hit) {
        q = org + (h.t * dir);
        // Light::getDirection: three draws (x, y, z), times radius, minus 0.5
        const double r0 = rand_double(st), r1 = rand_double(st), r2 = rand_double(st);
        const D3 off = d3(r0 * A.lradius - 0.5, r1 * A.lradius - 0.5, r2 * A.lradius - 0.5);
        const D3 Lp = lpos + off - q;
        sL = 1.0 / (double)sqrtf(__double2float_rn(Lp.x * Lp.x + Lp.y * Lp.y + Lp.z * Lp.z));
        L = d3(Lp.x * sL, Lp.y * sL, Lp.z * sL);
        dist = norm_exact(lpos - q);
        ray_setup(sr, q.x, q.y, q.z, L.x, L.y, L.z, B, D);
      } else {
        ray_setup(sr, 0.0, 0.0, 0.0, 0.0, 0.0, 1.0, B, D);
      }
      // the next wave starts where the group's last sample ended
      wst = __shfl_sync(full, st, base + G - 1);
      // Light::shadowAttenuation: any-hit from q towards the light
      HitRec s;
      sr.oself = fabsf((float)A.aperture);  // (at least the lens radius, which bounds the primary ray's origin)
      const int sres =
          traverse<true, MODE == kRenderStats, SHORT, NC, true>(S, sr, rb, s, hit, &ts, ring, (float)dist,
                                                                hit ? h.id : -1);
      if (sres < 0) atomicOr(&S.g->err, kErrStack);
      D3 N;
      double sN = 0.0, fall = 0.0, datt = 0.0;
      bool tiny = false;
      if (hit) {
        // smooth normal, bvh.cu:357-364 (hit_normal, kept apart for the adjoint)
        const int na = S.nidx[3 * h.id], nb = S.nidx[3 * h.id + 1], nc = S.nidx[3 * h.id + 2];
        const D3 nA = d3(S.normals[3 * na], S.normals[3 * na + 1], S.normals[3 * na + 2]);
        const D3 nB = d3(S.normals[3 * nb], S.normals[3 * nb + 1], S.normals[3 * nb + 2]);
        const D3 nC = d3(S.normals[3 * nc], S.normals[3 * nc + 1], S.normals[3 * nc + 2]);
        const D3 Nr = (1.0 - (h.alpha + h.beta)) * nA + h.alpha * nB + h.beta * nC;
        sN = 1.0 / (double)sqrtf(__double2float_rn(Nr.x * Nr.x + Nr.y * Nr.y + Nr.z * Nr.z));
        N = d3(Nr.x * sN, Nr.y * sN, Nr.z * sN);
        // Light::distanceAttenuation
        fall = A.latt[0] + (A.latt[1] + A.latt[2] * dist) * dist;
        tiny = fabs(fall) < kRayEps;
        fall = tiny ? 1.0 : 1.0 / fall;
        datt = fmin(1.0, fall);
      }
      D3 col = d3(0.9, 0.9, 0.9);
      int sh = -1, shid = -1;
      if (hit) {
        const int mid = __ldg(S.matid + h.id);
        const DMat m = S.mats[mid];
        D3 I = d3(m.ke[0] + m.ka[0] * 0.0, m.ke[1] + m.ka[1] * 0.0, m.ke[2] + m.ka[2] * 0.0);
        D3 satt = d3(1, 1, 1);
        sh = 0;
        int omid = -1;
        bool otrans = false;
        DMat om;
        if (sres > 0) {
          sh = 1;
          shid = s.id;
          omid = __ldg(S.matid + s.id);
          om = S.mats[omid];
          otrans = om.kt[0] == 0 && om.kt[1] == 0 && om.kt[2] == 0;  // Trans() = isZero(kt)
          satt = otrans ? d3(om.kd[0] * (1 - om.kt[0]), om.kd[1] * (1 - om.kt[1]), om.kd[2] * (1 - om.kt[2]))
                        : d3(0, 0, 0);
        }
        const D3 att = datt * satt;
        const double NL = dot(N, L);
        double lam = NL;
        if (lam < 0) lam = 0;
        const D3 diffuse = d3(m.kd[0] * lam, m.kd[1] * lam, m.kd[2] * lam);
        D3 ds = diffuse;
        if (!phong_vanishes(m, I)) ds = diffuse + phong_term(S.mats + mid, L, N, q, d3(A.eye[0], A.eye[1], A.eye[2]));
        I = I + d3(att.x * ds.x * A.lcol[0], att.y * ds.y * A.lcol[1], att.z * ds.z * A.lcol[2]);
        col = I;
        if (MODE == kAdjoint) {
          const double Gc[3] = {G3.x, G3.y, G3.z};
          const double sa[3] = {satt.x, satt.y, satt.z};
          const double dsv[3] = {ds.x, ds.y, ds.z};
          double S_lam = 0.0, gdatt = 0.0;
#pragma unroll
          for (int c = 0; c < 3; c++) {
            const double w = Gc[c] * A.lcol[c];
            // d/d kd of the hit triangle's material (Lambert term)
            const double gkd = w * datt * sa[c] * lam;
            if (gkd != 0.0) atomicAdd(A.grad_albedo + 3 * mid + c, gkd);
            // d/d kd of an opaque occluder's material: the reference's shadow
            // attenuation is kd % (1 - kt) of the occluder (Light.cu:22-24)
            if (sh == 1 && otrans) {
              const double go = w * datt * dsv[c] * (1 - om.kt[c]);
              if (go != 0.0) atomicAdd(A.grad_albedo + 3 * omid + c, go);
            }
            S_lam += w * datt * sa[c] * m.kd[c];
            gdatt += w * sa[c] * dsv[c];
          }
          if (!(NL > 0)) S_lam = 0.0;  // lam = max(N.L, 0)
          // datt = min(1, 1/fall(dist)), fall = a + (b + c dist) dist
          double gdist = 0.0;
          if (!tiny && fall < 1.0) {
            const double fr = 1.0 / fall;  // the falloff polynomial itself
            gdist = gdatt * (-(A.latt[1] + 2.0 * A.latt[2] * dist) / (fr * fr));
          }
          // lam through L = Lp / |Lp|, Lp = P + off - q
          const D3 gLp = d3((N.x - NL * L.x) * sL * S_lam, (N.y - NL * L.y) * sL * S_lam,
                            (N.z - NL * L.z) * sL * S_lam);
          const D3 u = (dist > 0.0) ? (1.0 / dist) * (lpos - q) : d3(0, 0, 0);
          const D3 gP = gLp + gdist * u;
          glight = glight + gP;
          const D3 gq = d3(-gP.x, -gP.y, -gP.z);
          // lam through N = Nr / |Nr|, Nr = (1-a-b) nA + a nB + b nC
          const int na = S.nidx[3 * h.id], nb = S.nidx[3 * h.id + 1], nc = S.nidx[3 * h.id + 2];
          const D3 nA = d3(S.normals[3 * na], S.normals[3 * na + 1], S.normals[3 * na + 2]);
          const D3 nB = d3(S.normals[3 * nb], S.normals[3 * nb + 1], S.normals[3 * nb + 2]);
          const D3 nC = d3(S.normals[3 * nc], S.normals[3 * nc + 1], S.normals[3 * nc + 2]);
          const D3 gN = d3((L.x - NL * N.x) * sN * S_lam, (L.y - NL * N.y) * sN * S_lam,
                           (L.z - NL * N.z) * sN * S_lam);
          const double g_al = dot(gN, nB - nA), g_be = dot(gN, nC - nA);
          const double g_t = dot(gq, dir) + Gd;  // q = o + t d, and the depth output
          // (t, alpha, beta) solve [-d | E1 | E2] x = o - A; moving the hit's
          // barycentric point by delta moves x by -M^-1 delta, so
          // d loss / d delta = -M^-T g, split over A, B, C by (1-a-b, a, b).
          const int ia = S.vidx[3 * h.id], ib = S.vidx[3 * h.id + 1], ic = S.vidx[3 * h.id + 2];
          const D3 Av = d3(S.verts[3 * ia], S.verts[3 * ia + 1], S.verts[3 * ia + 2]);
          const D3 Bv = d3(S.verts[3 * ib], S.verts[3 * ib + 1], S.verts[3 * ib + 2]);
          const D3 Cv = d3(S.verts[3 * ic], S.verts[3 * ic + 1], S.verts[3 * ic + 2]);
          const D3 ma = d3(-dir.x, -dir.y, -dir.z), mb = Bv - Av, mc = Cv - Av;
          const D3 bc = d3(mb.y * mc.z - mb.z * mc.y, mb.z * mc.x - mb.x * mc.z, mb.x * mc.y - mb.y * mc.x);
          const D3 ca = d3(mc.y * ma.z - mc.z * ma.y, mc.z * ma.x - mc.x * ma.z, mc.x * ma.y - mc.y * ma.x);
          const D3 ab = d3(ma.y * mb.z - ma.z * mb.y, ma.z * mb.x - ma.x * mb.z, ma.x * mb.y - ma.y * mb.x);
          const double det = dot(ma, bc);
          if (det != 0.0) {
            const double id = -1.0 / det;
            const D3 w = d3(id * (g_t * bc.x + g_al * ca.x + g_be * ab.x), id * (g_t * bc.y + g_al * ca.y + g_be * ab.y),
                            id * (g_t * bc.z + g_al * ca.z + g_be * ab.z));
            const double wa = 1.0 - (h.alpha + h.beta), wb = h.alpha, wc = h.beta;
            atomicAdd(A.grad_verts + 3 * ia, wa * w.x), atomicAdd(A.grad_verts + 3 * ia + 1, wa * w.y);
            atomicAdd(A.grad_verts + 3 * ia + 2, wa * w.z);
            atomicAdd(A.grad_verts + 3 * ib, wb * w.x), atomicAdd(A.grad_verts + 3 * ib + 1, wb * w.y);
            atomicAdd(A.grad_verts + 3 * ib + 2, wb * w.z);
            atomicAdd(A.grad_verts + 3 * ic, wc * w.x), atomicAdd(A.grad_verts + 3 * ic + 1, wc * w.y);
            atomicAdd(A.grad_verts + 3 * ic + 2, wc * w.z);
          }
        }
      }
      if (MODE != kAdjoint && act) {
        if (A.hit_id) A.hit_id[si] = hit ? h.id : -1;
        if (A.hit_t) A.hit_t[si] = hit ? h.t : 0.0;
        if (A.shadow) A.shadow[si] = sh;
        if (A.shadow_id) A.shadow_id[si] = shid;
      }
      // sum in sample order (the reference adds the samples one by one)
      if (MODE != kAdjoint) {
        double v0 = act ? col.x : 0.0, v1 = act ? col.y : 0.0, v2 = act ? col.z : 0.0, v3 = hit ? h.t : 0.0;
        if (G >= 4) {
          quad_transpose(v0, v1, v2, v3);
          for (int t = 0; t < G; t += 4) {
            const int src = base + t + (lane & 3);
            const double a0 = __shfl_sync(full, v0, src), a1 = __shfl_sync(full, v1, src),
                         a2 = __shfl_sync(full, v2, src), a3 = __shfl_sync(full, v3, src);
            acc.x = acc.x + a0;
            acc.x = acc.x + a1;
            acc.x = acc.x + a2;
            acc.x = acc.x + a3;
          }
        } else {
          for (int t = 0; t < G; t++) {
            acc = acc + d3(__shfl_sync(full, v0, base + t), __shfl_sync(full, v1, base + t),
                           __shfl_sync(full, v2, base + t));
            depth += __shfl_sync(full, v3, base + t);
          }
        }
      }
      // guess for the next wave: the group's majority
      const int nh = __popc(hits & gmask), na = __popc(actm & gmask);
      pred = __ballot_sync(full, 2 * nh >= na);
    }
    if (MODE == kAdjoint) return;
    if (G >= 4) {
      const double m = sample_mean(acc.x, A.spp);
      acc = d3(m, __shfl_sync(full, m, base + 1), __shfl_sync(full, m, base + 2));
      depth = __shfl_sync(full, m, base + 3);
    } else {
      acc = d3(sample_mean(acc.x, A.spp), sample_mean(acc.y, A.spp), sample_mean(acc.z, A.spp));
      depth = sample_mean(depth, A.spp);
    }
    if (!valid || g != 0) return;
    write_pixel(A, idx, acc);
    if (A.depth) A.depth[idx] = depth;
}

template <int MODE>
__device__ __forceinline__ void flush_stats(const RenderArgs& A, const TravStats& ts, const D3& glight) {
  if (MODE == kRenderStats) {
    unsigned long long a = ts.nodes, b = ts.tris;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(A.stats, a);
      atomicAdd(A.stats + 1, b);
    }
  }
  if (MODE == kAdjoint) {
    warp_add(A.grad_light, glight.x);
    warp_add(A.grad_light + 1, glight.y);
    warp_add(A.grad_light + 2, glight.z);
  }
}

}  // namespace

}  // namespace crt
