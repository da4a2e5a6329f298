// Occluder depth pass (vgc_occluder_depth): the reference draws the occluder meshes' previous-frame camera cuts
// depth-only with the current camera into a small depth target before the HZB build (OcclusionCulling.ts:244-273,
// through the pools' vertex pulling, GeometryPool.ts:1095-1131). Here it is a CUDA rasterizer over the draw list of
// an output slot:
//
//  * one warp per draw-list entry of part 0 (drawn over every pixel; the blended ones are left out, as in the
//    reference's proxy) whose mesh is an occluder; clip = (P V M) p with the instance's model matrix;
//  * a triangle is clipped against the near plane (clip.z >= 0, WebGPU depth) as a GPU's clipper would: the part in
//    front is a triangle or a quad (two triangles) with the crossing points at depth 0; a triangle that faces away
//    (the reference's proxy is single-sided) is dropped;
//  * pixel centres (x + 0.5, y + 0.5) inside all three edge functions (edges included) take the depth interpolated
//    from the vertices' NDC depths (affine in screen space) through an atomic minimum on the float's bits (depth is
//    >= 0, so the unsigned order is the float order); the image starts at 1 (far);
//  * each meshlet vertex is transformed once, into the warp's shared-memory vertex buffer (meshlet-local ids < 256);
//    a meshlet's loads are issued together (its triangles, then its vertex ids, then positions, 128 at a time) and
//    the warp's next entry is fetched while it draws this one: every step of this pass waits on memory;
//  * triangles that face the camera and cover a pixel centre's row and column wait in a ring per warp and are taken 32
//    at a time (most do not: drawing each step's own left most lanes idle), sorted by the pixels of their bounding
//    box: small ones (at most kLaneRasterMax) are drawn by the warp, their pixels laid end to end, a lane per pixel;
//    medium ones (at most kWarpRasterMax) are queued, one atomic per 32 triangles on one of kSubQueues counters (a
//    different one each time: with one per warp, the warps of the nearest geometry filled theirs and drew the rest
//    themselves), and drawn by the second kernel, a warp per triangle; larger ones are queued as 32 x 16 pixel tiles
//    of their bounding box, a warp per tile. The second kernel spreads both over the whole grid: a meshlet close to
//    the camera, with a hundred triangles of a few hundred pixels each, would otherwise keep one warp drawing long
//    after the rest have finished. When a queue is full its triangles are drawn by the warp that set them up.
//    16 two-pass images of 960x540 (steady state): occluder kernel 650 -> 275 us, queue kernel 215 -> 250 us;
//  * the atomics' results are unused, so they do not wait (a load-then-atomic early depth test measured slower: it
//    puts an L2 round trip on every pixel). The image is the minimum over all drawn pixels, whatever the order.
//
// The visibility pass (vgc_visibility, below) draws a cut's expanded index buffer through the same triangle setup,
// size classes and queues, with 64-bit (depth | triangle id) fragments.
//
// Every expression rounds step by step in the written order (the library is compiled with -fmad=false), so the
// oracle's C restatement reproduces the image bit for bit.
#include "vgcut_host.h"
#include "vgcut_kernels.h"

namespace {

// Bounding-box pixels up to which a triangle is drawn by the warp that set it up, with 31 others, a lane per pixel.
// 16 / 32 / 64 measured: 16 two-pass images of 960x540, occluder kernel + queue kernel: 504 + 269 (the medium queue
// overflows) / 281 + 273 / 385 + 191 us; a 1080p visibility buffer: 734 + 170 / 765 + 122 / 832 + 82 us.
constexpr uint32_t kLaneRasterMax = 32;
constexpr uint32_t kWarpRasterMax = 1024;   // ... by one warp of the second kernel; beyond, as tiles
constexpr uint32_t kTileW = 32, kTileH = 16;
// Queue capacities: medium triangles in sub-queues (record i of sub-queue q at i * kSubQueues + q), 160 MB of them; a
// quarter of that for images of up to kManyPixels in all (as many records a pixel as a 1080p image then has), in a context
// with an HBM budget and where the device has no room for more. What the queue does not hold is drawn by the warp that set it
// up, long after the others have finished: 1080p visibility buffers of near geometry 2.40 -> 1.30 ms, 32 two-pass images
// of 960x540 2.06 -> 1.45 ms a step, against a quarter of the records.
constexpr uint32_t kQueuedMedium = 5u << 19, kQueuedMediumMin = 5u << 17, kManyPixels = 1u << 19;
constexpr uint32_t kSubQueues = 256;
constexpr uint32_t kClipCtl = 4 + kSubQueues;   // occluder pass: triangles crossing the near plane, queued
constexpr uint32_t kCtlWords = kClipCtl + 1;
constexpr uint32_t kClipQueue = 1u << 17;     // (draw-list entry, triangle) records, clipped by a later kernel
constexpr uint32_t kQueuedLarge = 5u << 14;   // large triangles,
constexpr uint32_t kTileUnits = 1u << 20;     // and their tiles
constexpr uint32_t kNoTri = 0xffffffffu;      // an empty tile record
constexpr uint32_t kRecord = 4;               // float4 per queued triangle
constexpr uint32_t kMaxImages = 64;           // occluder images per launch set (vgc_occluder_depth_batch)

// Where the fragments go, and the queues of the second kernel.
struct RasterArgs {
  uint32_t width, height;
  uint32_t *depth[kMaxImages];   // occluder pass: float bits per pixel of image i (a fragment's TriTag::id)
  unsigned long long *vis;       // visibility pass: (depth bits << 32 | id) per pixel
  uint32_t frame;                // visibility pass: lodBlendFrame
  // queues: ctl[0] = the visibility pass's next run of triangles, ctl[1] = large triangles, ctl[2..3] = tiles (64-bit),
  // ctl[4 + q] = medium triangles of sub-queue q; triangle records (kRecord float4, read_record); tile records (large
  // triangle, tile index in its bounding box, row-major)
  uint32_t *ctl;
  float4 *medium;
  uint32_t medium_each;  // medium records a sub-queue holds
  float4 *large;
  uint2 *tiles;
  uint2 *clip;  // occluder pass: crossing triangles (ctl[kClipCtl] of them)
};

// The occluder pass's inputs: per image, the camera and the cut it draws.
struct OccluderImage {
  float vp[16];  // P * V, row-major 4x4 (float of the double product)
  const uint4 *draw_list;      // cut 0 entries of the source slot
  const uint32_t *counters;    // its counter header
};
struct OccluderArgs {
  OccluderImage img[kMaxImages];
  uint32_t count, max_drawn;
};

struct ScreenTri {
  float ax, ay, az, bx, by, bz, cx, cy, cz, area;
  int x0, x1, y0, y1;  // pixel bounding box, inclusive
};

// What a fragment carries besides its depth: for the visibility pass the entry's blend range and the triangle's id,
// for the occluder pass (lo = hi = 0) the image it belongs to in `id`.
struct TriTag {
  uint32_t lo, hi, id;
};

// Clip coordinates of a position: (P V M) p.
__device__ __forceinline__ float4 clip_vertex(const float mvp[4][4], float4 v) {
  float c[4];
#pragma unroll
  for (int r = 0; r < 4; r++) c[r] = ((mvp[r][0] * v.x + mvp[r][1] * v.y) + mvp[r][2] * v.z) + mvp[r][3];
  return make_float4(c[0], c[1], c[2], c[3]);
}

// A clip-space vertex in screen space: x, y (pixels, y down), NDC depth; w = 1 when usable (in front of the near
// plane), else all 0.
__device__ __forceinline__ float4 screen_of(float4 c, float W, float H) {
  if (!(c.w > 0.0f) || !(c.z >= 0.0f)) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const float nx = c.x / c.w, ny = c.y / c.w, nz = c.z / c.w;
  return make_float4((nx * 0.5f + 0.5f) * W, (0.5f - ny * 0.5f) * H, nz, 1.0f);
}

__device__ __forceinline__ float4 screen_vertex(const float mvp[4][4], float4 v, float W, float H) {
  return screen_of(clip_vertex(mvp, v), W, H);
}

// Setup of one triangle from its screen-space corners; false when it is dropped.
__device__ __forceinline__ bool setup_triangle(float4 v0, float4 v1, float4 v2, float W, float H, ScreenTri &t) {
  if (v0.w == 0.0f || v1.w == 0.0f || v2.w == 0.0f) return false;  // a corner behind the near plane
  // screen space is y-down: a triangle facing the camera (counter-clockwise in NDC) has a negative area here
  const float area0 = (v1.x - v0.x) * (v2.y - v0.y) - (v2.x - v0.x) * (v1.y - v0.y);
  if (!(area0 < 0.0f)) return false;  // back-facing, degenerate or not finite
  // order A, B, C = 0, 2, 1: positive area
  t.ax = v0.x, t.ay = v0.y, t.az = v0.z;
  t.bx = v2.x, t.by = v2.y, t.bz = v2.z;
  t.cx = v1.x, t.cy = v1.y, t.cz = v1.z;
  t.area = (t.bx - t.ax) * (t.cy - t.ay) - (t.cx - t.ax) * (t.by - t.ay);
  if (!(t.area > 0.0f)) return false;
  float mnx = fminf(fminf(t.ax, t.bx), t.cx), mxx = fmaxf(fmaxf(t.ax, t.bx), t.cx);
  float mny = fminf(fminf(t.ay, t.by), t.cy), mxy = fmaxf(fmaxf(t.ay, t.by), t.cy);
  // pixel centres px + 0.5 in [mn, mx]; clamped in float before the integer conversion
  mnx = fmaxf(mnx, -1.0f), mxx = fminf(mxx, W + 1.0f);
  mny = fmaxf(mny, -1.0f), mxy = fminf(mxy, H + 1.0f);
  t.x0 = max(0, int(ceilf(mnx - 0.5f)));
  t.x1 = min(int(W) - 1, int(floorf(mxx - 0.5f)));
  t.y0 = max(0, int(ceilf(mny - 0.5f)));
  t.y1 = min(int(H) - 1, int(floorf(mxy - 0.5f)));
  return t.x0 <= t.x1 && t.y0 <= t.y1;
}

// Near-plane clipping (Sutherland-Hodgman against clip.z >= 0) of the triangle with clip-space corners c0, c1, c2;
// the part in front is a triangle or a quad, set up as screen triangles into t0 (and t1); returns how many (0..2),
// t0 holding the first. With A the corner in front (one in front) or the corner after the one behind (two in front)
// in the order c0 -> c1 -> c2, and B, C the next ones: one in front -> (A, AB, CA); two in front (A, B) ->
// (A, B, BC) and (A, BC, CA), where XY = X + s (Y - X), s = X.z / (X.z - Y.z), is the crossing point at depth 0.
// A triangle wholly in front gives exactly setup_triangle of its screen corners.
__device__ __forceinline__ float4 crossing(float4 p, float4 q) {
  const float s = p.z / (p.z - q.z);
  return make_float4(p.x + s * (q.x - p.x), p.y + s * (q.y - p.y), 0.0f, p.w + s * (q.w - p.w));
}

__device__ __forceinline__ float4 pick3(int i, float4 a, float4 b, float4 c) { return i == 0 ? a : (i == 1 ? b : c); }

__device__ __forceinline__ int setup_clipped(float4 c0, float4 c1, float4 c2, float W, float H, ScreenTri &t0,
                                             ScreenTri &t1) {
  const int in = (c0.z >= 0.0f ? 1 : 0) + (c1.z >= 0.0f ? 1 : 0) + (c2.z >= 0.0f ? 1 : 0);
  if (in == 3) return setup_triangle(screen_of(c0, W, H), screen_of(c1, W, H), screen_of(c2, W, H), W, H, t0) ? 1 : 0;
  if (in == 0) return 0;
  // the corner that starts the polygon: the one in front (in == 1) or the one after the corner behind (in == 2)
  const int lone = in == 1 ? (c0.z >= 0.0f ? 0 : (c1.z >= 0.0f ? 1 : 2)) : (c0.z < 0.0f ? 0 : (c1.z < 0.0f ? 1 : 2));
  const int ia = in == 1 ? lone : (lone + 1) % 3;
  const float4 A = pick3(ia, c0, c1, c2), B = pick3((ia + 1) % 3, c0, c1, c2), C = pick3((ia + 2) % 3, c0, c1, c2);
  const float4 sa = screen_of(A, W, H);
  if (in == 1)
    return setup_triangle(sa, screen_of(crossing(A, B), W, H), screen_of(crossing(A, C), W, H), W, H, t0) ? 1 : 0;
  const float4 sbc = screen_of(crossing(B, C), W, H);
  const bool first = setup_triangle(sa, screen_of(B, W, H), sbc, W, H, t0);
  const bool second = setup_triangle(sa, sbc, screen_of(crossing(A, C), W, H), W, H, t1);
  if (!first && second) t0 = t1;
  return int(first) + int(second);
}

// lodBlendMask (lodBlend.ts:36-45) at pixel (px, py): true when the pixel's step lies in [lo, hi).
__device__ __forceinline__ bool blend_keep(int px, int py, uint32_t frame, uint32_t lo, uint32_t hi) {
  const float x = (float(px) + 0.5f) + float(frame) * 5.588238f, y = float(py) + 0.5f;
  const float a = x * 0.06711056f + y * 0.00583715f;
  const float b = (a - floorf(a)) * 52.9829189f;
  const float step = floorf((b - floorf(b)) * 255.0f);
  return step >= float(lo) && step < float(hi);
}

// One pixel of t: covered when its centre is inside the three edge functions (edges included); the depth is the
// screen-space interpolation of the corners' NDC depths, kept as a minimum (depth >= 0, so the unsigned order of
// the bits is the float order; the atomics' results are unused, so they do not wait).
template <bool VIS>
__device__ __forceinline__ void shade_pixel(const RasterArgs &R, const ScreenTri &t, const TriTag &g, int px, int py) {
  const float x = float(px) + 0.5f, y = float(py) + 0.5f;
  const float wa = (t.cx - t.bx) * (y - t.by) - (t.cy - t.by) * (x - t.bx);  // edge B -> C
  const float wb = (t.ax - t.cx) * (y - t.cy) - (t.ay - t.cy) * (x - t.cx);  // edge C -> A
  const float wc = (t.bx - t.ax) * (y - t.ay) - (t.by - t.ay) * (x - t.ax);  // edge A -> B
  // the blend steps are 0 .. 254: the full range [0, 255) keeps every pixel
  if (wa >= 0.0f && wb >= 0.0f && wc >= 0.0f &&
      (!VIS || (g.lo == 0u && g.hi == 255u) || blend_keep(px, py, R.frame, g.lo, g.hi))) {
    float z = ((wa * t.az + wb * t.bz) + wc * t.cz) / t.area;
    z = z > 0.0f ? z : 0.0f;  // +0 for rounding below zero (and never -0, whose bits would sort last)
    const size_t at = (size_t)py * R.width + px;
    if (VIS)
      atomicMin(R.vis + at, ((unsigned long long)__float_as_uint(z) << 32) | g.id);
    else
      atomicMin(R.depth[g.id] + at, __float_as_uint(z));
  }
}

__device__ __forceinline__ ScreenTri read_record(const float4 *r, uint32_t &tx, TriTag &g) {
  const float4 a = r[0], b = r[1], c = r[2], d = r[3];
  const uint32_t xy = __float_as_uint(c.z), size = __float_as_uint(c.w), tag = __float_as_uint(d.x);
  ScreenTri t;
  t.ax = a.x, t.ay = a.y, t.bx = a.z, t.by = a.w;
  t.cx = b.x, t.cy = b.y, t.az = b.z, t.bz = b.w;
  t.cz = c.x, t.area = c.y;
  t.x0 = int(xy & 0xffffu), t.y0 = int(xy >> 16);
  t.x1 = t.x0 + int(size & 0xffffu) - 1, t.y1 = t.y0 + int(size >> 16) - 1;
  g.lo = tag & 255u, g.hi = (tag >> 8) & 255u, g.id = __float_as_uint(d.y);
  tx = __float_as_uint(d.z);
  return t;
}

// q / w of a small triangle's pixel q < 128 and width w <= 128 as q * inv >> 15, inv = floor(2^15 / w) + 1 (an
// approximate quotient may give one more): 0 < inv w - 2^15 <= 2 w, so q (inv w - 2^15) < 2^15 and the result is exact
constexpr uint32_t kInvShift = 15;

// The whole warp over t's bounding box, 32 consecutive pixels (row-major) per step.
template <bool VIS>
__device__ __forceinline__ void warp_draw(const RasterArgs &R, const ScreenTri &t, const TriTag &g, uint32_t lane) {
  const uint32_t bw = uint32_t(t.x1 - t.x0 + 1), count = bw * uint32_t(t.y1 - t.y0 + 1);
  // a step of 32 pixels: q rows and r columns. The quotients of 32 and of the lane as at kInvShift, exact for every
  // width: up to 511, 32 * 2 bw < 2^15; above, inv <= 66 and both quotients are 0
  const uint32_t inv = uint32_t(__fdividef(float(1u << kInvShift), float(bw))) + 1u;
  const uint32_t q = (32u * inv) >> kInvShift, r = 32u - q * bw;
  uint32_t y = (lane * inv) >> kInvShift, x = lane - y * bw;
  for (uint32_t i = lane; i < count; i += 32) {
    shade_pixel<VIS>(R, t, g, t.x0 + int(x), t.y0 + int(y));
    x += r, y += q;
    if (x >= bw) x -= bw, y++;
  }
}

__device__ __forceinline__ uint32_t warp_scan_incl(uint32_t v) {
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  return v;
}

// Per warp: the triangles waiting to be drawn, a ring filled as they are set up and emptied 32 at a time.
constexpr uint32_t kRing = 64;
struct TriRing {
  float4 a[kRing];  // ax, ay, bx, by
  float4 b[kRing];  // cx, cy, az, bz
  float4 c[kRing];  // cz, area, x0 | y0 << 16, bounding-box width | height << 16 (as bits)
  uint2 d[kRing];   // lo | hi << 8, id
  uint8_t order[32];
};
static_assert(kLaneRasterMax <= 128, "the packed division covers boxes of 128 pixels");

__device__ __forceinline__ ScreenTri ring_triangle(const TriRing &ring, uint32_t j, TriTag &g, uint32_t &meta,
                                                   uint32_t &inv) {
  const float4 a = ring.a[j], b = ring.b[j], c = ring.c[j];
  const uint2 d = ring.d[j];
  ScreenTri t;
  t.ax = a.x, t.ay = a.y, t.bx = a.z, t.by = a.w;
  t.cx = b.x, t.cy = b.y, t.az = b.z, t.bz = b.w;
  t.cz = c.x, t.area = c.y;
  t.x0 = int(__float_as_uint(c.z) & 0xffffu), t.y0 = int(__float_as_uint(c.z) >> 16);
  meta = __float_as_uint(c.w);
  g.lo = d.x & 255u, g.hi = (d.x >> 8) & 255u, g.id = d.y;
  inv = d.x >> 16;
  return t;
}

// The queued record of ring entry j (read_record's layout: the ring's, then the triangle's tile columns).
__device__ __forceinline__ void ring_record(const TriRing &ring, uint32_t j, float4 *r, uint32_t tx) {
  r[0] = ring.a[j], r[1] = ring.b[j], r[2] = ring.c[j];
  r[3] = make_float4(__uint_as_float(ring.d[j].x), __uint_as_float(ring.d[j].y), __uint_as_float(tx), 0.0f);
}

// Draws the ring's first n (<= 32) triangles, a lane for each. Medium and large ones are queued for the second kernel,
// one reservation of each kind for all; the small ones' bounding-box pixels are laid end to end and drawn a lane per
// pixel, so that a step's cost does not follow the largest of them.
template <bool VIS>
__device__ __forceinline__ void draw_ring(const RasterArgs &R, TriRing &ring, uint32_t head, uint32_t n) {
  __syncwarp();
  const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u;
  // the medium sub-queue: another one each time, or the warps with the nearest geometry fill theirs and draw the rest
  // themselves, long after the other warps have finished
  const uint32_t sub = (((blockIdx.x * blockDim.x + threadIdx.x) >> 5) + (head >> 5) * 37u) % kSubQueues;
  const uint32_t own = (head + lane) & (kRing - 1u);
  const uint32_t size = lane < n ? __float_as_uint(ring.c[own].w) : 0u, bw = size & 0xffffu, bh = size >> 16;
  const uint32_t px = bw * bh;
  if (__any_sync(0xffffffffu, px > kLaneRasterMax)) {
    const bool medium = px > kLaneRasterMax && px <= kWarpRasterMax, large = px > kWarpRasterMax;
    const uint32_t mm = __ballot_sync(0xffffffffu, medium), lm = __ballot_sync(0xffffffffu, large);
    bool left = false;
    if (mm) {
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(R.ctl + 4 + sub, __popc(mm));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(mm & below);
      if (medium && at < R.medium_each)
        ring_record(ring, own, R.medium + ((size_t)at * kSubQueues + sub) * kRecord, 0u);
      else if (medium)
        left = true;
    }
    if (lm) {
      const uint32_t tx = large ? (bw - 1u + kTileW) / kTileW : 0u;
      const uint32_t nt = large ? tx * ((bh - 1u + kTileH) / kTileH) : 0u;
      const uint32_t ts = warp_scan_incl(nt) - nt, total = __shfl_sync(0xffffffffu, ts + nt, 31);
      uint32_t tri = 0;
      unsigned long long at_t = 0;
      if (lane == 0) {
        tri = atomicAdd(R.ctl + 1, __popc(lm));
        at_t = atomicAdd(reinterpret_cast<unsigned long long *>(R.ctl + 2), (unsigned long long)total);
      }
      tri = __shfl_sync(0xffffffffu, tri, 0);
      at_t = __shfl_sync(0xffffffffu, at_t, 0);
      if (tri + __popc(lm) <= kQueuedLarge && at_t + total <= kTileUnits) {
        const uint32_t mine = tri + __popc(lm & below);
        if (large) ring_record(ring, own, R.large + (size_t)mine * kRecord, tx);
        for (uint32_t rest = lm; rest; rest &= rest - 1) {  // the tile records, a triangle at a time
          const uint32_t j = __ffs(rest) - 1;
          const uint32_t nj = __shfl_sync(0xffffffffu, nt, j), sj = __shfl_sync(0xffffffffu, ts, j);
          const uint32_t tj = __shfl_sync(0xffffffffu, mine, j);
          for (uint32_t i = lane; i < nj; i += 32) R.tiles[at_t + sj + i] = make_uint2(tj, i);
        }
      } else {  // a queue is full: reserved tile slots below its capacity become empty records
        for (unsigned long long i = at_t + lane; i < at_t + total && i < kTileUnits; i += 32)
          R.tiles[i] = make_uint2(kNoTri, 0u);
        if (large) left = true;
      }
    }
    // what a full queue turned away, one at a time by the whole warp
    for (uint32_t rest = __ballot_sync(0xffffffffu, left); rest; rest &= rest - 1) {
      TriTag h;
      uint32_t meta, inv;
      ScreenTri u = ring_triangle(ring, (head + __ffs(rest) - 1) & (kRing - 1u), h, meta, inv);
      u.x1 = u.x0 + int(meta & 0xffffu) - 1, u.y1 = u.y0 + int(meta >> 16) - 1;
      warp_draw<VIS>(R, u, h, lane);
    }
  }
  const bool small = px != 0 && px <= kLaneRasterMax;
  const uint32_t smalls = __ballot_sync(0xffffffffu, small), count = small ? px : 0u;
  const uint32_t incl = warp_scan_incl(count), all = __shfl_sync(0xffffffffu, incl, 31), start = incl - count;
  if (small) {
    ring.c[own].w = __uint_as_float(start | bw << 16);
    ring.d[own].x |= (uint32_t(__fdividef(float(1u << kInvShift), float(bw))) + 1u) << 16;
  }
  if (small) ring.order[__popc(smalls & below)] = uint8_t(own);  // the k-th small triangle's place
  __syncwarp();
  const uint32_t upto = (2u << lane) - 1u;
  uint32_t started = ~0u;  // the last small triangle starting before this step's first pixel
  for (uint32_t base = 0; base < all; base += 32) {
    const uint32_t rel = start - base;
    const uint32_t starts = __reduce_or_sync(0xffffffffu, small && rel < 32u ? 1u << rel : 0u);
    const uint32_t p = base + lane, k = started + __popc(starts & upto);
    started += __popc(starts);
    if (p < all) {
      TriTag h;
      uint32_t meta, inv;
      const ScreenTri u = ring_triangle(ring, ring.order[k], h, meta, inv);
      const uint32_t q = p - (meta & 0xffffu), w = meta >> 16, y = (q * inv) >> kInvShift;
      shade_pixel<VIS>(R, u, h, u.x0 + int(q - y * w), u.y0 + int(y));
    }
  }
  __syncwarp();  // the drawn places are filled again
}

// One triangle per lane of the warp (ok: set up; t, g: its setup and tag) joins the warp's ring (head: its first, n: how
// many wait, at most 31 before); the caller draws 32 when there are as many. Most triangles of a cut face away or cover
// no pixel centre (84% of a 1080p view's), so drawing each step's own would leave most lanes idle.
__device__ __forceinline__ void ring_add(TriRing &ring, uint32_t head, uint32_t &n, uint32_t lane, bool ok,
                                         const ScreenTri &t, const TriTag &g) {
  const uint32_t mask = __ballot_sync(0xffffffffu, ok);
  if (ok) {
    const uint32_t at = (head + n + __popc(mask & ((1u << lane) - 1u))) & (kRing - 1u);
    ring.a[at] = make_float4(t.ax, t.ay, t.bx, t.by);
    ring.b[at] = make_float4(t.cx, t.cy, t.az, t.bz);
    ring.c[at] = make_float4(t.cz, t.area, __uint_as_float(uint32_t(t.x0) | uint32_t(t.y0) << 16),
                             __uint_as_float(uint32_t(t.x1 - t.x0 + 1) | uint32_t(t.y1 - t.y0 + 1) << 16));
    ring.d[at] = make_uint2(g.lo | g.hi << 8, g.id);
  }
  n += __popc(mask);
}

// Clears the occluder images (1.0f) and the queues' control words.
__global__ void __launch_bounds__(256) k_occluder_clear(const __grid_constant__ RasterArgs R, uint32_t count,
                                                        size_t pixels) {
  if (blockIdx.x == 0)
    for (uint32_t i = threadIdx.x; i < kCtlWords; i += blockDim.x) R.ctl[i] = 0;
  const size_t n = pixels * count;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    R.depth[i / pixels][i % pixels] = 0x3f800000u;
}

// Clears the image and the queues' control words.
template <typename T>
__global__ void __launch_bounds__(256) k_target_clear(T *image, size_t n, T value, uint32_t *ctl) {
  if (blockIdx.x == 0)
    for (uint32_t i = threadIdx.x; i < kCtlWords; i += blockDim.x) ctl[i] = 0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    image[i] = value;
}

// The images' entries laid end to end: first[v] = entries of images before v, first[count] = all (block-shared).
__device__ __forceinline__ void image_starts(const OccluderArgs &O, uint32_t *first) {
  if (threadIdx.x < 32) {
    uint32_t carry = 0;
    for (uint32_t v0 = 0; v0 < O.count; v0 += 32) {
      const uint32_t v = v0 + threadIdx.x;
      const uint32_t c = v < O.count ? min(O.img[v].counters[VGC_COUNTER_CUT0 + VGC_CUT_SELECTED], O.max_drawn) : 0u;
      const uint32_t incl = warp_scan_incl(c);
      if (v < O.count) first[v] = carry + incl - c;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (threadIdx.x == 0) first[O.count] = carry;
  }
  __syncthreads();
}

// The image of laid-out entry e < first[count]: the last v with first[v] <= e.
__device__ __forceinline__ uint32_t image_of(const uint32_t *first, uint32_t count, uint32_t e) {
  uint32_t v = 0;
  for (uint32_t span = count; span > 1;) {
    const uint32_t half = span >> 1;
    if (first[v + half] <= e) v += half;
    span -= half;
  }
  return v;
}

__global__ void __launch_bounds__(128, 5) k_raster_occluders(Scene S, const __grid_constant__ OccluderArgs O,
                                                              const __grid_constant__ RasterArgs R) {
  __shared__ float4 verts[4][256];     // per warp: the current meshlet's vertices in screen space (local ids < 256)
  __shared__ uint32_t packed[4][128];  // ... and its packed triangles
  __shared__ TriRing rings[4];
  __shared__ uint32_t first[kMaxImages + 1];
  TriRing &ring = rings[threadIdx.x >> 5];
  float4 *sv = verts[threadIdx.x >> 5];
  uint32_t *st = packed[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31;
  image_starts(O, first);
  const uint32_t n = first[O.count];
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const float W = float(R.width), H = float(R.height);
  // Each step waits on memory several times (entry, instance and meshlet, vertices, triangles): the loads of a step
  // are issued together, and the next entry is fetched while this one is drawn. Entries of all images are laid end
  // to end; a warp's entry belongs to one image.
  uint32_t e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint32_t head = 0, waiting = 0;  // the ring of small triangles (of any image: the tag names it)
  uint32_t v_next = e < n ? image_of(first, O.count, e) : 0u;
  uint4 next = e < n ? O.img[v_next].draw_list[e - first[v_next]] : make_uint4(0u, 0u, 0u, 0u);
  for (;; e += warps) {
    if (e >= n) {
      if (waiting) draw_ring<false>(R, ring, head, waiting);
      break;
    }
    const uint4 d = next;
    const uint32_t v = v_next;
    if (e + warps < n) {
      v_next = image_of(first, O.count, e + warps);
      next = O.img[v_next].draw_list[e + warps - first[v_next]];
    }
    const TriTag none{0u, 0u, v};  // the fragments' image
    if ((d.w & 0xffff00u) != (255u << 16)) continue;  // part 1 (blended): not an occluder
    const uint32_t slot = S.inst_slot[d.x];
    const float4 *col = S.inst + (size_t)d.x * 4;
    const float4 c0 = col[0], c1 = col[1], c2 = col[2], c3 = col[3];
    const uint4 info = S.m_info[d.y];
    if (!S.meshes[slot].occluder) continue;
    const uint32_t tris = d.w & 255u, first_tri = info.y / 3, voff = info.w;
    uint32_t pk[4];  // the meshlet's packed triangles (at most 128), loaded at once
#pragma unroll
    for (uint32_t r = 0; r < 4; r++) pk[r] = r * 32 + lane < tris ? S.m_tris[first_tri + r * 32 + lane] : 0u;
    // M's rows from the instance's columns, then clip = (P V) M p
    const float m[4][4] = {{c0.x, c1.x, c2.x, c3.x}, {c0.y, c1.y, c2.y, c3.y}, {c0.z, c1.z, c2.z, c3.z},
                           {c0.w, c1.w, c2.w, c3.w}};
    const float *vp = O.img[v].vp;
    float mvp[4][4];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int k = 0; k < 4; k++)
        mvp[r][k] = ((vp[r * 4] * m[0][k] + vp[r * 4 + 1] * m[1][k]) + vp[r * 4 + 2] * m[2][k]) + vp[r * 4 + 3] * m[3][k];
    // the meshlet's vertices (local ids 0 .. the largest its triangles use), each transformed once, 128 at a time
    uint32_t top = 0;
#pragma unroll
    for (uint32_t r = 0; r < 4; r++)
      top = max(top, max(pk[r] & 255u, max((pk[r] >> 8) & 255u, (pk[r] >> 16) & 255u)));
    top = __reduce_max_sync(0xffffffffu, top);
    __syncwarp();
#pragma unroll
    for (uint32_t r = 0; r < 4; r++) st[r * 32 + lane] = pk[r];
    for (uint32_t base = 0; base <= top; base += 128) {
      uint32_t id[4];
#pragma unroll
      for (uint32_t k = 0; k < 4; k++) id[k] = base + k * 32 + lane <= top ? S.m_verts[voff + base + k * 32 + lane] : 0u;
      float4 pos[4];
#pragma unroll
      for (uint32_t k = 0; k < 4; k++) pos[k] = base + k * 32 + lane <= top ? S.positions[id[k]] : make_float4(0, 0, 0, 1);
#pragma unroll
      for (uint32_t k = 0; k < 4; k++)
        if (base + k * 32 + lane <= top) sv[base + k * 32 + lane] = screen_vertex(mvp, pos[k], W, H);
    }
    __syncwarp();
    for (uint32_t round = 0; round * 32 < tris; round++) {
      const uint32_t ti = round * 32 + lane, p = st[ti];
      ScreenTri t;
      bool ok = false, crossing = false;
      if (ti < tris) {
        const float4 a = sv[p & 255u], b = sv[(p >> 8) & 255u], c = sv[(p >> 16) & 255u];
        crossing = a.w == 0.0f || b.w == 0.0f || c.w == 0.0f;  // a corner behind the near plane
        if (!crossing) ok = setup_triangle(a, b, c, W, H, t);
      }
      // crossing triangles (rare) are clipped by k_raster_clipped: (entry, triangle) records, one atomic per warp
      const uint32_t cm = __ballot_sync(0xffffffffu, crossing);
      if (cm) {
        uint32_t at = 0;
        if (lane == __ffs(cm) - 1) at = atomicAdd(R.ctl + kClipCtl, __popc(cm));
        at = __shfl_sync(0xffffffffu, at, __ffs(cm) - 1) + __popc(cm & ((1u << lane) - 1u));
        if (crossing && at < kClipQueue) R.clip[at] = make_uint2(e - first[v], ti | (v << 8));
      }
      ring_add(ring, head, waiting, lane, ok, t, none);
      if (waiting >= 32) {
        draw_ring<false>(R, ring, head, 32);
        head += 32, waiting -= 32;
      }
    }
    __syncwarp();  // the vertex and triangle buffers are rewritten by the next entry
  }
}

// The occluder pass's triangles that cross the near plane, a lane each: the draw-list entry's (P V M), the triangle's
// corners in clip space, clipped (setup_clipped), and its one or two screen triangles through the same size classes
// and queues (k_raster_queued runs after this kernel).
__global__ void __launch_bounds__(128) k_raster_clipped(Scene S, const __grid_constant__ OccluderArgs O,
                                                          const __grid_constant__ RasterArgs R) {
  __shared__ TriRing rings[4];
  TriRing &ring = rings[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t n = min(R.ctl[kClipCtl], kClipQueue);
  const uint32_t stride = gridDim.x * blockDim.x;
  const float W = float(R.width), H = float(R.height);
  uint32_t head = 0, waiting = 0;
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n; base += stride) {
    const uint32_t i = base + lane;
    ScreenTri t, t2;
    int k = 0;
    TriTag none{0u, 0u, 0u};  // the fragments' image
    if (i < n) {
      const uint2 rec = R.clip[i];
      const uint32_t v = rec.y >> 8;
      none.id = v;
      const float *vp = O.img[v].vp;
      const uint4 d = O.img[v].draw_list[rec.x];
      const float4 *col = S.inst + (size_t)d.x * 4;
      const float4 c0 = col[0], c1 = col[1], c2 = col[2], c3 = col[3];
      const float m[4][4] = {{c0.x, c1.x, c2.x, c3.x}, {c0.y, c1.y, c2.y, c3.y}, {c0.z, c1.z, c2.z, c3.z},
                             {c0.w, c1.w, c2.w, c3.w}};
      float mvp[4][4];
#pragma unroll
      for (int r = 0; r < 4; r++)
#pragma unroll
        for (int kk = 0; kk < 4; kk++)
          mvp[r][kk] = ((vp[r * 4] * m[0][kk] + vp[r * 4 + 1] * m[1][kk]) + vp[r * 4 + 2] * m[2][kk]) +
                       vp[r * 4 + 3] * m[3][kk];
      const uint4 info = S.m_info[d.y];
      const uint32_t p = S.m_tris[info.y / 3 + (rec.y & 255u)], voff = info.w;
      const float4 va = clip_vertex(mvp, S.positions[S.m_verts[voff + (p & 255u)]]);
      const float4 vb = clip_vertex(mvp, S.positions[S.m_verts[voff + ((p >> 8) & 255u)]]);
      const float4 vc = clip_vertex(mvp, S.positions[S.m_verts[voff + ((p >> 16) & 255u)]]);
      k = setup_clipped(va, vb, vc, W, H, t, t2);
    }
    for (int part = 1; part <= 2; part++) {
      if (part == 2 && !__any_sync(0xffffffffu, k == 2)) break;
      ring_add(ring, head, waiting, lane, k >= part, part == 1 ? t : t2, none);
      if (waiting >= 32) {
        draw_ring<false>(R, ring, head, 32);
        head += 32, waiting -= 32;
      }
    }
  }
  if (waiting) draw_ring<false>(R, ring, head, waiting);
}

// The queued triangles, spread over the whole grid: a warp per medium triangle, then a warp per tile of a large one
// (a lane per column of the tile).
template <bool VIS>
__global__ void __launch_bounds__(128) k_raster_queued(const __grid_constant__ RasterArgs R) {
  __shared__ uint32_t counts[kSubQueues];  // medium triangles per sub-queue
  __shared__ uint32_t most;
  if (threadIdx.x == 0) most = 0;
  __syncthreads();
  for (uint32_t q = threadIdx.x; q < kSubQueues; q += blockDim.x) {
    counts[q] = min(R.ctl[4 + q], R.medium_each);
    atomicMax(&most, counts[q]);
  }
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31;
  // medium records are interleaved: slot u holds record u / kSubQueues of sub-queue u % kSubQueues
  const uint32_t n_medium = most * kSubQueues;
  const uint32_t n = n_medium + (uint32_t)min(*reinterpret_cast<const unsigned long long *>(R.ctl + 2),
                                              (unsigned long long)kTileUnits);
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5, mine = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint32_t tx;
  TriTag g;
  uint32_t u = mine;
  for (; u < n_medium; u += warps)
    if (u / kSubQueues < counts[u % kSubQueues]) {
      const ScreenTri t = read_record(R.medium + (size_t)u * kRecord, tx, g);
      warp_draw<VIS>(R, t, g, lane);
    }
  for (; u < n; u += warps) {
    const uint2 tile = R.tiles[u - n_medium];
    if (tile.x == kNoTri) continue;
    const ScreenTri t = read_record(R.large + (size_t)tile.x * kRecord, tx, g);
    const int px = t.x0 + int((tile.y % tx) * kTileW + lane), py0 = t.y0 + int((tile.y / tx) * kTileH);
    if (px > t.x1) continue;
    const int py1 = min(t.y1, py0 + int(kTileH) - 1);
    for (int py = py0; py <= py1; py++) shade_pixel<VIS>(R, t, g, px, py);
  }
}

// ------------------------------------------------------------------------------------------------ visibility
// Headless consumer of a cut (vgc_visibility): the cut's expanded index buffer drawn as the draw args say, with the
// reference's vertex pulling (GeometryPool.ts:1095-1131) and LOD blend mask (lodBlend.ts:36-45), into a visibility
// buffer: per pixel the 64-bit minimum of (depth bits << 32 | drawSlot << 7 | triangle in its meshlet).
//
//  * an index is (drawSlot << 7) | localVertex; drawSlot picks the draw-list entry (instance, meshlet), the local
//    vertex its meshletVertices entry and the position; the instance's model maps it to world space, shrunk toward
//    the instance origin by the draw-distance fade clamp((maxDrawDistance - |V origin|) / (0.15 maxDrawDistance),
//    0, 1), V the camera's view (GeometryPool.ts:1112-1119);
//  * triangles are set up as in the occluder pass (pixel centres, edges included, back faces and triangles reaching
//    in front of the near plane left out), one per lane, and drawn through the same size classes and queues;
//  * a fragment is kept when the step floor(255 n) of its pixel lies in the entry's blend range [lo, hi), n the
//    interleaved gradient noise fract(52.9829189 fract(0.06711056 x + 0.00583715 y)) at the pixel centre (x, y),
//    x shifted by 5.588238 per `frame` (lodBlendFrame);
//  * indices or entries outside the context's arrays (an index buffer not written by vgc_expand) drop their
//    triangle.
constexpr float kDrawDistanceFade = 0.15f;   // GeometryPool.ts:109

struct VisArgs {
  float vp[16];    // P * V, row-major
  float view[16];  // the camera's V (draw-distance fade), row-major
  uint32_t width, height, regions;  // regions: mesh slots * 2 (parts)
  const uint32_t *indices;
  uint64_t capacity;
  const uint4 *draw_list;  // the output slot's entries (draw slots of both cuts)
  const uint32_t *args;    // the cut's draw args, 5 u32 per (mesh slot, part)
  uint32_t draw_slots;     // entries in draw_list
  uint32_t meshlets, instances, meshlet_vertices, vertices;
};

// The clip-space position of index `idx` of the expanded buffer (ok: the index and its data are in range).
__device__ __forceinline__ float4 pulled_clip(const Scene &S, const VisArgs &A, uint32_t idx, bool &ok) {
  const uint32_t ds = idx >> kLocalVertexBits, lv = idx & ((1u << kLocalVertexBits) - 1u);
  ok = false;
  if (ds >= A.draw_slots) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const uint4 ent = A.draw_list[ds];
  if (ent.x >= A.instances || ent.y >= A.meshlets) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const MeshRec &mesh = S.meshes[S.inst_slot[ent.x]];
  const uint32_t mv = S.m_info[ent.y].w + lv;
  if (!mesh.vertices || mv >= A.meshlet_vertices) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const uint32_t vid = S.m_verts[mv];
  if (vid >= A.vertices) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  ok = true;
  const float4 p = S.positions[vid];
  const float4 *col = S.inst + (size_t)ent.x * 4;
  const float4 c0 = col[0], c1 = col[1], c2 = col[2], c3 = col[3];
  // draw-distance fade, from the camera's distance to the instance origin
  const float *V = A.view;
  const float ox = ((V[0] * c3.x + V[1] * c3.y) + V[2] * c3.z) + V[3];
  const float oy = ((V[4] * c3.x + V[5] * c3.y) + V[6] * c3.z) + V[7];
  const float oz = ((V[8] * c3.x + V[9] * c3.y) + V[10] * c3.z) + V[11];
  const float dist = sqrtf((ox * ox + oy * oy) + oz * oz);
  const float maxd = mesh.max_draw_distance;
  const float fade = fminf(fmaxf((maxd - dist) / (maxd * kDrawDistanceFade), 0.0f), 1.0f);
  const float wx = c3.x + ((c0.x * p.x + c1.x * p.y) + c2.x * p.z) * fade;
  const float wy = c3.y + ((c0.y * p.x + c1.y * p.y) + c2.y * p.z) * fade;
  const float wz = c3.z + ((c0.z * p.x + c1.z * p.y) + c2.z * p.z) * fade;
  float c[4];
#pragma unroll
  for (int r = 0; r < 4; r++) c[r] = ((A.vp[r * 4] * wx + A.vp[r * 4 + 1] * wy) + A.vp[r * 4 + 2] * wz) + A.vp[r * 4 + 3];
  return make_float4(c[0], c[1], c[2], c[3]);
}

// Vertices [from, upto) of draw slot ds's meshlet in screen space into `cache`, a lane each (screen_of; w = 0: behind
// the near plane, w = -1: the slot or the vertex is outside the context's arrays): pulled_clip's arithmetic, with what
// belongs to the slot read and computed once. `upto` is raised to the meshlet's vertex count, as the next meshlet's
// offset tells it (only how many are pulled at once depends on it); returns how many are cached.
__device__ __forceinline__ uint32_t pull_vertices(const Scene &S, const VisArgs &A, uint32_t ds, uint32_t from,
                                                  uint32_t upto, float4 *cache) {
  const float4 outside = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
  bool ok = ds < A.draw_slots;
  uint4 ent = make_uint4(0u, 0u, 0u, 0u);
  if (ok) ent = A.draw_list[ds], ok = ent.x < A.instances && ent.y < A.meshlets;
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float4 c0 = zero, c1 = zero, c2 = zero, c3 = zero;
  float maxd = 1.0f;
  uint32_t first = 0;
  if (ok) {
    const MeshRec &mesh = S.meshes[S.inst_slot[ent.x]];
    const float4 *col = S.inst + (size_t)ent.x * 4;
    c0 = col[0], c1 = col[1], c2 = col[2], c3 = col[3];
    first = S.m_info[ent.y].w;
    const uint32_t count = ent.y + 1 < A.meshlets ? S.m_info[ent.y + 1].w - first : 0u;
    if (count <= 1u << kLocalVertexBits) upto = max(upto, count);
    maxd = mesh.max_draw_distance;
    ok = mesh.vertices != 0;
  }
  const float *V = A.view;
  const float ox = ((V[0] * c3.x + V[1] * c3.y) + V[2] * c3.z) + V[3];
  const float oy = ((V[4] * c3.x + V[5] * c3.y) + V[6] * c3.z) + V[7];
  const float oz = ((V[8] * c3.x + V[9] * c3.y) + V[10] * c3.z) + V[11];
  const float dist = sqrtf((ox * ox + oy * oy) + oz * oz);
  const float fade = fminf(fmaxf((maxd - dist) / (maxd * kDrawDistanceFade), 0.0f), 1.0f);
  upto = (upto + 31u) & ~31u;
  for (uint32_t lv = from + (threadIdx.x & 31); lv < upto; lv += 32) {
    const uint32_t mv = first + lv;
    uint32_t vid = ~0u;
    if (ok && mv < A.meshlet_vertices) vid = S.m_verts[mv];
    if (vid >= A.vertices) {
      cache[lv] = outside;
      continue;
    }
    const float4 p = S.positions[vid];
    const float wx = c3.x + ((c0.x * p.x + c1.x * p.y) + c2.x * p.z) * fade;
    const float wy = c3.y + ((c0.y * p.x + c1.y * p.y) + c2.y * p.z) * fade;
    const float wz = c3.z + ((c0.z * p.x + c1.z * p.y) + c2.z * p.z) * fade;
    float c[4];
#pragma unroll
    for (int r = 0; r < 4; r++) c[r] = ((A.vp[r * 4] * wx + A.vp[r * 4 + 1] * wy) + A.vp[r * 4 + 2] * wz) + A.vp[r * 4 + 3];
    cache[lv] = screen_of(make_float4(c[0], c[1], c[2], c[3]), float(A.width), float(A.height));
  }
  return upto;
}

// A triangle with a corner behind the near plane, or whose indices name several draw slots: its own three pulls,
// clipped. Returns how many screen triangles (0..2) it left in out.
__device__ __noinline__ int pulled_triangle(const Scene &S, const VisArgs &A, uint32_t i0, uint32_t i1, uint32_t i2,
                                            ScreenTri *out) {
  bool k0, k1, k2;
  const float4 v0 = pulled_clip(S, A, i0, k0), v1 = pulled_clip(S, A, i1, k1), v2 = pulled_clip(S, A, i2, k2);
  if (!(k0 && k1 && k2)) return 0;
  return setup_clipped(v0, v1, v2, float(A.width), float(A.height), out[0], out[1]);
}

// The triangles of the cut in region order (mesh slot, then part), as the draw args give them: a warp takes a run of
// consecutive ones from a counter, a lane each, 32 per step. Consecutive triangles belong to one or two meshlets, so the
// warp transforms each meshlet's vertices once, a lane per vertex, into shared memory and the triangles pick their corners
// from there: about 70 pulls for the 80 triangles of a meshlet, where a pull per index took 240. Bound by instruction
// issue (pulls 35%, pixels 20%, the rest indices and set-up); the ring's draw stands at one place of the loop, so that its
// registers and the set-up's share the 72 that let 28 warps live on an SM (80 and 64 measured 760 and 735 us, the
// indices of the next step fetched ahead 765). 1080p, 290k meshlets of 24M triangles: 1433 -> 737 us, with a quarter of the
// medium queue; with all of it another such view takes 540, and the queue kernel 147.
constexpr uint32_t kVisRunMin = 64, kVisRunMax = 512;
__global__ void __launch_bounds__(128, 7) k_visibility(const __grid_constant__ Scene S,
                                                       const __grid_constant__ VisArgs A,
                                                       const __grid_constant__ RasterArgs R) {
  extern __shared__ uint32_t tri_start[];  // per region: first triangle in the laid-out order; [regions] = total
  __shared__ TriRing rings[4];
  __shared__ float4 vertices[4][1u << kLocalVertexBits];
  TriRing &ring = rings[threadIdx.x >> 5];
  float4 *cache = vertices[threadIdx.x >> 5];
  if (threadIdx.x < 32) {  // warp 0 scans the regions' triangle counts
    uint32_t carry = 0;
    for (uint32_t r0 = 0; r0 < A.regions; r0 += 32) {
      const uint32_t r = r0 + threadIdx.x;
      const uint32_t c = r < A.regions ? A.args[r * 5] / 3 : 0u;
      const uint32_t incl = warp_scan_incl(c);
      if (r < A.regions) tri_start[r] = carry + incl - c;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (threadIdx.x == 0) tri_start[A.regions] = carry;
  }
  __syncthreads();
  const uint32_t total = tri_start[A.regions];
  // triangles per run: long runs cut fewer meshlets in two, short ones leave no warp idle when there are few triangles
  const uint32_t share = total / (gridDim.x * 16u) & ~31u, length = min(max(share, kVisRunMin), kVisRunMax);
  const uint32_t runs = (total + length - 1) / length;
  const uint32_t lane = threadIdx.x & 31;
  WarpFeed feed;
  feed.start(R.ctl);
  uint32_t slot = kNoTri, known = 0;  // the cached draw slot and how many of its vertices are cached
  uint32_t head = 0, waiting = 0;     // the ring of small triangles
  constexpr uint32_t mask = (1u << kLocalVertexBits) - 1u;
  // a step's indices: the triangle's three, its rank in its region; false past the run or the index buffer
  struct Indices {
    uint32_t i0, i1, i2, rank;
    bool valid;
  };
  uint32_t run = feed.i, base = 0, end = 0, region = 0;
  auto fetch = [&](uint32_t from) {
    Indices x{0u, 0u, 0u, 0u, false};
    const uint32_t t_id = min(from + lane, end - 1);
    uint32_t r = region;
    while (tri_start[r + 1] <= t_id) r++;
    region = __shfl_sync(0xffffffffu, r, 31);
    x.rank = t_id - tri_start[r];
    const uint64_t first = (uint64_t)A.args[r * 5 + 2] + 3ull * x.rank;
    x.valid = from + lane < end && first + 2 < A.capacity;
    if (x.valid) x.i0 = A.indices[first], x.i1 = A.indices[first + 1], x.i2 = A.indices[first + 2];
    return x;
  };
  ScreenTri out[2];
  TriTag g{0u, 0u, 0u};
  int n = 0;
  bool second = false, last = false;  // a clipped quad's second triangle comes next; no run is left
  while (!last) {
    ScreenTri t;
    bool ok = false;
    if (second) {
      second = false;
      ok = n == 2;
      if (ok) t = out[1];
    } else {
      if (base >= end) {  // the next run
        last = run >= runs;
        if (!last) {
          base = run * length, end = min(total - base, length) + base;
          region = 0;  // the last region starting at or before the run
          for (uint32_t span = A.regions; span > 1;) {
            const uint32_t half = span >> 1;
            if (tri_start[region + half] <= base) region += half;
            span -= half;
          }
          run = feed.next();
        }
      }
      if (!last) {
        const Indices x = fetch(base);
        base += 32;
        const uint32_t ds = x.i0 >> kLocalVertexBits;
        const bool one = x.valid && x.i1 >> kLocalVertexBits == ds && x.i2 >> kLocalVertexBits == ds;
        float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a, c = a;
        for (uint32_t pending = __ballot_sync(0xffffffffu, one); pending;) {
          const uint32_t d = __shfl_sync(0xffffffffu, ds, __ffs(pending) - 1);
          const bool mine = one && ds == d;
          const uint32_t top =
              __reduce_max_sync(0xffffffffu, mine ? max(x.i0 & mask, max(x.i1 & mask, x.i2 & mask)) + 1u : 0u);
          if (d != slot) slot = d, known = 0;
          if (known < top) {
            known = pull_vertices(S, A, d, known, top, cache);
            __syncwarp();
          }
          if (mine) a = cache[x.i0 & mask], b = cache[x.i1 & mask], c = cache[x.i2 & mask];
          pending &= ~__ballot_sync(0xffffffffu, mine);
          __syncwarp();  // the cache may be rewritten for the next slot
        }
        n = 0;
        if (one && a.w > 0.0f && b.w > 0.0f && c.w > 0.0f) {
          n = setup_triangle(a, b, c, float(A.width), float(A.height), t) ? 1 : 0;
        } else if (x.valid && (!one || (a.w >= 0.0f && b.w >= 0.0f && c.w >= 0.0f))) {
          n = pulled_triangle(S, A, x.i0, x.i1, x.i2, out);
          if (n) t = out[0];
        }
        ok = n != 0;
        if (ok) {
          const uint4 ent = A.draw_list[ds];
          g.lo = (ent.w >> 8) & 255u, g.hi = (ent.w >> 16) & 255u;
          const uint64_t at = 3ull * x.rank;  // index in the region
          const uint32_t tri = at >= ent.z && at < 1ull << 32 ? (uint32_t(at) - ent.z) / 3 : uint32_t((at - ent.z) / 3);
          g.id = (ds << kLocalVertexBits) | (tri & mask);
        }
        second = __any_sync(0xffffffffu, n == 2);
      }
    }
    ring_add(ring, head, waiting, lane, ok, t, g);
    if (waiting >= 32 || (last && waiting)) {
      const uint32_t m = min(waiting, 32u);
      draw_ring<true>(R, ring, head, m);
      head += m, waiting -= m;
    }
  }
}

}  // namespace

// The queues of the second kernel for images of `pixels` in all (the passes of one context share them, so calls on
// different streams must not overlap). What a call has used is kept until the context ends, since a captured graph may
// hold it: a first call of larger images takes everything at once, one of smaller images the smaller medium queue, to
// which a larger one is added when larger images come.
static int raster_queues(vgc_context *ctx, RasterArgs &R, size_t pixels, cudaStream_t st) {
  const size_t large_bytes = (size_t)kQueuedLarge * kRecord * 16, tile_bytes = (size_t)kTileUnits * 8;
  const size_t ctl_bytes = 2048, clip_bytes = (size_t)kClipQueue * 8;
  static_assert(kCtlWords * 4 <= ctl_bytes, "control words");
  const size_t rest = ctl_bytes + large_bytes + tile_bytes + clip_bytes, record = kRecord * 16;
  const bool many = pixels > kManyPixels && !ctx->opts.hbm_budget_bytes;
  if (!ctx->d_raster.ptr) {
    int rc = many ? dev_alloc(ctx, ctx->d_raster, rest + kQueuedMedium * record) : VGC_OOM;
    if (rc == VGC_OOM) rc = dev_alloc(ctx, ctx->d_raster, rest + kQueuedMediumMin * record);
    if (rc) return rc;
  } else if (many && ctx->d_raster.bytes < rest + kQueuedMedium * record && !ctx->d_raster_medium.ptr) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;  // a capture allows no allocation
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone ||
        dev_alloc(ctx, ctx->d_raster_medium, kQueuedMedium * record))
      cudaGetLastError();
  }
  char *q = (char *)ctx->d_raster.ptr;
  R.ctl = (uint32_t *)q;
  R.large = (float4 *)(q + ctl_bytes);
  R.tiles = (uint2 *)(q + ctl_bytes + large_bytes);
  R.clip = (uint2 *)(q + ctl_bytes + large_bytes + tile_bytes);
  const bool added = many && ctx->d_raster_medium.ptr;
  R.medium = (float4 *)(added ? (char *)ctx->d_raster_medium.ptr : q + rest);
  R.medium_each = (uint32_t)((added ? ctx->d_raster_medium.bytes : ctx->d_raster.bytes - rest) / record) / kSubQueues;
  return VGC_OK;
}

// Up to kMaxImages images of the occluder pass in one launch set (arguments checked): image i draws output slot
// slots[i] with views[i] into depth[i].
static int occluder_depth_images(vgc_context *ctx, uint32_t count, const uint32_t *slots, const vgc_view *views,
                                 float *const *depth, uint32_t width, uint32_t height, cudaStream_t st) {
  int rc;
  OccluderArgs O{};
  RasterArgs R{};
  O.count = count;
  O.max_drawn = ctx->opts.max_meshlets;
  for (uint32_t v = 0; v < count; v++) {
    OccluderImage &I = O.img[v];
    for (int r = 0; r < 4; r++)
      for (int c = 0; c < 4; c++) {
        double s = 0;
        for (int i = 0; i < 4; i++) s += views[v].proj[i * 4 + r] * views[v].view[c * 4 + i];
        I.vp[r * 4 + c] = (float)s;
      }
    I.draw_list = (const uint4 *)ctx->d_draw.ptr + (size_t)slots[v] * 2 * ctx->opts.max_meshlets;
    I.counters = (const uint32_t *)ctx->d_counters.ptr + (size_t)slots[v] * ctx->counter_words;
    R.depth[v] = reinterpret_cast<uint32_t *>(depth[v]);
  }
  R.width = width;
  R.height = height;
  const size_t pixels = (size_t)width * height;
  if ((rc = raster_queues(ctx, R, pixels * count, st))) return rc;
  k_occluder_clear<<<(unsigned)std::min<size_t>((pixels * count + 255) / 256, (size_t)ctx->sm_count * 16), 256, 0,
                     st>>>(R, count, pixels);
  CUDA_TRY(cudaGetLastError());
  if (ctx->positions.empty()) return VGC_OK;  // no mesh carries vertex data: nothing is an occluder
  // persistent grids of exactly the resident blocks: a grid-stride loop over a grid larger than one wave leaves the
  // blocks of the second wave their full share of the work after the first has finished
  static int per_sm[2] = {0, 0};
  if (!per_sm[0]) {
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm[0], k_raster_occluders, 128, 0));
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm[1], k_raster_queued<false>, 128, 0));
  }
  k_raster_occluders<<<ctx->sm_count * std::max(1, per_sm[0]), 128, 0, st>>>(scene_of(ctx), O, R);
  CUDA_TRY(cudaGetLastError());
  k_raster_clipped<<<ctx->sm_count * 2, 128, 0, st>>>(scene_of(ctx), O, R);
  CUDA_TRY(cudaGetLastError());
  k_raster_queued<false><<<ctx->sm_count * std::max(1, per_sm[1]), 128, 0, st>>>(R);
  CUDA_TRY(cudaGetLastError());
  return VGC_OK;
}

static int occluder_checks(vgc_context *ctx, uint32_t src_slot, const vgc_view *view, const float *depth,
                           uint32_t width, uint32_t height) {
  if (!ctx || !view || !depth) return fail(VGC_INVALID_ARG, "null argument");
  if (width == 0 || height == 0 || width > 16384 || height > 16384)
    return fail(VGC_INVALID_ARG, "occluder depth size must be 1..16384 per side");
  if (src_slot >= ctx->out_slots) return fail(VGC_NOT_FOUND, "output slot not allocated");
  return VGC_OK;
}

extern "C" int vgc_occluder_depth(vgc_context *ctx, uint32_t src_slot, const vgc_view *view, float *depth,
                                  uint32_t width, uint32_t height, vgc_stream stream) {
  int rc = occluder_checks(ctx, src_slot, view, depth, width, height);
  if (rc) return rc;
  cudaSetDevice(ctx->device);
  if ((rc = sync_scene(ctx))) return rc;
  return occluder_depth_images(ctx, 1, &src_slot, view, &depth, width, height,
                               stream ? (cudaStream_t)stream : ctx->stream);
}

extern "C" int vgc_occluder_depth_batch(vgc_context *ctx, uint32_t count, const uint32_t *src_slots,
                                        const vgc_view *views, float *const *depth, uint32_t width, uint32_t height,
                                        vgc_stream stream) {
  if (!ctx || (count && (!src_slots || !views || !depth))) return fail(VGC_INVALID_ARG, "null argument");
  int rc;
  for (uint32_t i = 0; i < count; i++)
    if ((rc = occluder_checks(ctx, src_slots[i], &views[i], depth[i], width, height))) return rc;
  cudaSetDevice(ctx->device);
  if ((rc = sync_scene(ctx))) return rc;
  const cudaStream_t st = stream ? (cudaStream_t)stream : ctx->stream;
  for (uint32_t i = 0; i < count; i += kMaxImages)
    if ((rc = occluder_depth_images(ctx, std::min(kMaxImages, count - i), src_slots + i, views + i, depth + i, width,
                                    height, st)))
      return rc;
  return VGC_OK;
}

extern "C" int vgc_visibility(vgc_context *ctx, uint32_t slot, uint32_t cut, const vgc_view *view,
                              const vgc_view *fade_view, const uint32_t *indices, uint64_t capacity, uint64_t *vis,
                              uint32_t width, uint32_t height, uint32_t frame, vgc_stream stream) {
  if (!ctx || !view || !indices || !vis || cut > 1) return fail(VGC_INVALID_ARG, "bad arguments");
  if (width == 0 || height == 0 || width > 16384 || height > 16384)
    return fail(VGC_INVALID_ARG, "visibility buffer size must be 1..16384 per side");
  if (slot >= ctx->out_slots) return fail(VGC_NOT_FOUND, "output slot not allocated");
  if (ctx->out_slot_capacity != ctx->slot_capacity)
    return fail(VGC_INVALID_ARG, "vgc_visibility: meshes were added since the cut; cut and expand again first");
  cudaSetDevice(ctx->device);
  int rc = sync_scene(ctx);
  if (rc) return rc;
  cudaStream_t st = stream ? (cudaStream_t)stream : ctx->stream;
  const vgc_view *fv = fade_view ? fade_view : view;
  VisArgs A{};
  for (int r = 0; r < 4; r++)
    for (int c = 0; c < 4; c++) {
      double s = 0;
      for (int i = 0; i < 4; i++) s += view->proj[i * 4 + r] * view->view[c * 4 + i];
      A.vp[r * 4 + c] = (float)s;
      A.view[r * 4 + c] = (float)fv->view[c * 4 + r];
    }
  A.width = width;
  A.height = height;
  A.regions = ctx->out_slot_capacity * 2;
  A.indices = indices;
  A.capacity = capacity;
  A.draw_list = (const uint4 *)ctx->d_draw.ptr + (size_t)slot * 2 * ctx->opts.max_meshlets;
  A.args = (const uint32_t *)ctx->d_args.ptr + (size_t)slot * 2 * ctx->out_slot_capacity * 2 * 5 +
           (size_t)cut * ctx->out_slot_capacity * 2 * 5;
  A.draw_slots = 2 * ctx->opts.max_meshlets;
  A.meshlets = (uint32_t)ctx->m_info.size();
  A.instances = (uint32_t)ctx->inst_slot.size();
  A.meshlet_vertices = (uint32_t)ctx->m_verts.size();
  A.vertices = (uint32_t)ctx->positions.size();
  RasterArgs R{};
  R.width = width;
  R.height = height;
  R.vis = reinterpret_cast<unsigned long long *>(vis);
  R.frame = frame;
  const size_t pixels = (size_t)width * height;
  if ((rc = raster_queues(ctx, R, pixels, st))) return rc;
  k_target_clear<unsigned long long>
      <<<(unsigned)std::min<size_t>((pixels + 255) / 256, (size_t)ctx->sm_count * 16), 256, 0, st>>>(
          R.vis, pixels, (unsigned long long)VGC_VIS_EMPTY, R.ctl);
  CUDA_TRY(cudaGetLastError());
  if (ctx->positions.empty()) return VGC_OK;  // no mesh carries vertex data
  const size_t smem = (A.regions + 1) * sizeof(uint32_t);
  if (smem > 48 * 1024) return fail(VGC_INVALID_ARG, "too many mesh slots for vgc_visibility");
  int per_sm = 0, per_sm_queued = 0;
  CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_visibility, 128, smem));
  CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_queued, k_raster_queued<true>, 128, 0));
  k_visibility<<<ctx->sm_count * std::max(1, per_sm), 128, smem, st>>>(scene_of(ctx), A, R);
  CUDA_TRY(cudaGetLastError());
  k_raster_queued<true><<<ctx->sm_count * std::max(1, per_sm_queued), 128, 0, st>>>(R);
  CUDA_TRY(cudaGetLastError());
  return VGC_OK;
}
