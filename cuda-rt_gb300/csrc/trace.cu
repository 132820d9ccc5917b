// trace.cu -- traversal and the pixel kernel on sm_103a.
//
// k_trace<ANY>  closest hit (BVH_d::intersect) or first hit in left-first
//               DFS order (BVH_d::intersectAny) for a batch of double rays,
//               the lanes of a warp refilled as their rays end.
// k_pixels      runRayTracerKernelRec (kernels/raytracer.cu:95-166) with
//               traceRay (raytracer.cu:169-249), Material::shade
//               (kernels/material.cu:6-40) and the positional Light
//               (kernels/Light.cu:5-86); also its adjoint.  Persistent: each
//               warp claims tiles of at most 32 / G pixels (G lanes per pixel), first
//               from its SM's rectangle of the image, then from the others;
//               a pixel's lanes trace its samples in waves, speculating on
//               how the mrand stream couples them (a hit consumes three
//               extra draws).
#include <cmath>

#include "pixel.cuh"

namespace crt {

namespace {

// Batched rays: a warp owns every stride-th chunk of `per` consecutive rays
// (per <= 32: neighbouring rays share their lanes' nodes, and the chunks
// spread the costly regions of the batch over the warps) and refills its
// lanes from them.  Eight blocks of 64 registers per SM: the walk waits for its
// node loads, and 32 warps hide more of that than the spills cost (the
// 1,000,000-ray closest-hit batch: 4 blocks 1.42, 5 1.34, 6 1.37, 7 1.28, 8
// 1.25 ms).
template <bool ANY>
__global__ void __launch_bounds__(128, 8) k_trace(const __grid_constant__ DScene S, const double* __restrict__ rays, int64_t n, int per,
                                               int* __restrict__ ids, double* __restrict__ tout,
                                               double* __restrict__ nout) {
  float rb[6], B, D;
  scene_consts(S, rb, B, D);
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const int64_t w = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t chunks = (n + per - 1) / per;
  const int64_t mine = w < chunks ? (chunks - 1 - w) / warps + 1 : 0;  // chunks w, w + warps, ...
  auto at = [&](int64_t i) { return (w + (i / per) * warps) * per + i % per; };
  walk_queue<ANY>(
      S, rb, (int)(mine * per),
      [&](int i, RayC& rc) {
        const int64_t k = at(i);
        if (k >= n) return false;
        const double* r = rays + 6 * k;
        ray_setup(rc, r[0], r[1], r[2], r[3], r[4], r[5], B, D);
        return true;
      },
      [&](int i, const RayC&, int res, const HitRec& h) {
        const int64_t k = at(i);
        if (res < 0) atomicOr(&S.g->err, kErrStack);
        const bool hit = res > 0;
        ids[k] = hit ? h.id : -1;
        if (tout) tout[k] = hit ? h.t : 0.0;
        if (!ANY && nout && hit) {
          const D3 N = hit_normal(S, h);
          nout[3 * k] = N.x, nout[3 * k + 1] = N.y, nout[3 * k + 2] = N.z;
        }
      });
}

// One scene: warps claim tiles of tile_w x tile_h pixels (at most 32 / G) of
// rows [row0, row1).  BPS: blocks per SM (launch_render).
// SHORT: traversal-stack entries kept in shared memory per thread.
constexpr int kPixelsShort = 0;
template <int MODE, int BPS>
__global__ void __launch_bounds__(128, BPS) k_pixels(DScene S, RenderArgs A) {
  extern __shared__ int2 s_ring[];
  int2* ring = kPixelsShort > 0 ? s_ring + threadIdx.x : nullptr;
  TravStats ts;
  D3 glight = d3(0, 0, 0);
  float rb[6], B, D;
  scene_consts(S, rb, B, D);
  const int lane = threadIdx.x & 31;
  const int G = A.group, tw = A.tile_w, th = A.tile_h;
  const int tiles_x = (A.W + tw - 1) / tw;
  const int tiles_y = (A.row1 - A.row0 + th - 1) / th;
  const int p = lane / G;  // this lane's pixel in the tile
  unsigned pred = 0xffffffffu;
  const bool cull = MODE == kAdjoint || !A.rays;  // (requested rays have to be made)
  double miss = 0.0;  // a missing pixel's mean, once this warp has met one
  int region = home_region(A.regions_x, A.regions_y);
  bool home = true;
  while (true) {
    int tile = 0;
    if (lane == 0) tile = claim_tile(A.counter, tiles_x, tiles_y, A.regions_x, A.regions_y, region, home);
    tile = __shfl_sync(0xffffffffu, tile, 0);
    if (tile < 0) break;
    const int tx = (tile % tiles_x) * tw, ty = A.row0 + (tile / tiles_x) * th;
    const int px = tx + (p % tw), py = ty + (p / tw);
    const bool valid = p < tw * th && px < A.W && py < A.row1;
    if (cull && beam_misses(S, A, rb, B, tx, tx + tw - 1, ty, ty + th - 1)) {
      if (miss == 0.0) miss = miss_mean(A.spp);
      write_miss<MODE>(A, px, py, valid, G, miss);
      continue;
    }
    pixel<MODE, kPixelsShort>(S, A, px, py, valid, G, pred, rb, B, D, ts, glight, ring);
  }
  flush_stats<MODE>(A, ts, glight);
}

}  // namespace

template <int MODE, int BPS>
static void launch_pixels(const DScene& S, const RenderArgs& a, cudaStream_t st) {
  const size_t smem = (size_t)kPixelsShort * 128 * sizeof(int2);
  int bps = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_pixels<MODE, BPS>, 128, smem);
  k_pixels<MODE, BPS><<<num_sms() * (bps > 0 ? bps : 1), 128, smem, st>>>(S, a);
}

cudaError_t set_tile_regions(RenderArgs& a, int tiles_x, int tiles_y, bool split, cudaStream_t st) {
  int rx = 1, ry = 1;
  const int R = min(num_sms(), kMaxTileRegions - 1);
  if (split && (int64_t)tiles_x * tiles_y >= (int64_t)kMinTilesPerRegion * R) {
    const double aspect = (double)max(tiles_x, 1) / (double)max(tiles_y, 1);
    rx = (int)(std::sqrt(R * aspect) + 0.5);
    rx = max(1, min(rx, min(R, tiles_x)));
    ry = max(1, min((R + rx - 1) / rx, tiles_y));
    while (rx * ry > kMaxTileRegions - 1) ry--;
  }
  a.regions_x = rx, a.regions_y = ry;
  return cudaMemsetAsync(a.counter, 0, sizeof(unsigned) * (size_t)(rx * ry + 1), st);
}

// Images of few pixels: what bounds them is not throughput but the slowest
// warp, so their work is spread over more warps.
//  - More lanes per pixel (up to gmax: fewer waves one after another) while
//    that leaves fewer than 288 / G warps' worth of lanes per SM (36 are
//    resident; with more lanes more samples start from wrong guesses).
//    100,000-triangle soup at 16 samples, 4 lanes against the rule's up to 16:
//    160x120 1035 -> 470 us, 320x240 1524 -> 1287; 7,080-triangle sphere, 64x48
//    530 -> 515, 240x180 1013 -> 790, 320x240 1096 -> 1060 (16 lanes there:
//    1105).  Depth-3 recursion at 4 samples, 2 lanes against up to 4: 640x360
//    7.7 -> 6.8 ms, 320x180 6.4 -> 5.5.
//  - Tiles of fewer pixels than a warp holds until every SM has 24 (the lanes
//    left over only vote): fewer different walks wait for one another.
//    2,000 triangles, 64x48 at 2 samples, with the build: 119 -> 100 us (12 per
//    SM 104, 16 to 36 100); 72 slow down 640x480 at one sample, 645 -> 800.
//    Recursion: 160x90 6.3 -> 4.0 ms (16 per SM 4.4), 64x48 5.5 -> 2.1.
void spread_pixels(RenderArgs& a, int gmax) {
  const int rows = a.row1 - a.row0;
  const int64_t sms = num_sms(), px = (int64_t)a.W * rows;
  while (2 * a.group <= min(a.spp, gmax) && px * a.group * a.group < 288 * 32 * sms) a.group *= 2;
  int tw = group_tile_w(a.group), th = group_tile_h(a.group);
  while (tw * th > 1 && (int64_t)((a.W + tw - 1) / tw) * ((rows + th - 1) / th) < 24 * sms) {
    if (tw >= th)
      tw /= 2;
    else
      th /= 2;
  }
  a.tile_w = tw, a.tile_h = th;
}

cudaError_t launch_render(const DScene& S, const RenderArgs& a0, cudaStream_t st) {
  RenderArgs a = a0;
  spread_pixels(a, 16);
  const int tiles_x = (a.W + a.tile_w - 1) / a.tile_w, tiles_y = (a.row1 - a.row0 + a.tile_h - 1) / a.tile_h;
  cudaError_t e = set_tile_regions(a, tiles_x, tiles_y, true, st);
  if (e != cudaSuccess) return e;
  // Nine blocks of 56 registers per SM, but seven of 72 below two tiles per
  // resident warp, where the warps' own time counts: 640x480 soup at one sample
  // 648 -> 600 us, 320x240 at 4 604 -> 585; above it 400x300 at 4 (99 tiles per
  // SM) is 752 us with nine against 777, the large frame 11.0 ms against 11.4.
  if (a.grad_rgb)
    launch_pixels<kAdjoint, 9>(S, a, st);
  else if (a.stats)
    launch_pixels<kRenderStats, 9>(S, a, st);
  else if ((int64_t)tiles_x * tiles_y < 72 * num_sms())
    launch_pixels<kRender, 7>(S, a, st);
  else
    launch_pixels<kRender, 9>(S, a, st);
  return cudaGetLastError();
}

cudaError_t launch_trace(const DScene& S, const double* rays, int64_t n, bool any, int* ids, double* t,
                         double* normals, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  int bps = 0;
  if (any)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_trace<true>, 128, 0);
  else
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_trace<false>, 128, 0);
  if (bps <= 0) bps = 1;
  // few rays are spread over more warps, down to one ray each: a walk's latency,
  // not the lanes, then bounds the call (4096 view rays against 19,220
  // triangles, with the rebuild before them: 32 to a warp 248 us, 4 144, 2 129, 1
  // 127; without it 2000 incoherent rays against 100,000 triangles: 4 214 us, 2
  // 171, 1 133; 8000: 234, 216, 188)
  const int64_t warps = (int64_t)num_sms() * bps * 4;
  int per = 32;
  while (per > 1 && (n + per - 1) / per < warps) per /= 2;
  const int64_t need = ((n + per - 1) / per + 3) / 4;
  const int grid = (int)(need < (int64_t)num_sms() * bps ? need : (int64_t)num_sms() * bps);
  if (any)
    k_trace<true><<<grid, 128, 0, st>>>(S, rays, n, per, ids, t, nullptr);
  else
    k_trace<false><<<grid, 128, 0, st>>>(S, rays, n, per, ids, t, normals);
  return cudaGetLastError();
}

}  // namespace crt
