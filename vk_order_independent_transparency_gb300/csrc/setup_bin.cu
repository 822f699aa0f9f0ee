// Triangle setup and order-preserving tile binning.
//
// The reference hands its triangles to the fixed-function pipeline
// (vkCmdDrawIndexed in oitRender.cpp:185, 226, 275, 287, 321, 367, 413), which
// runs object.vert.glsl and rasterises them while keeping primitive order for
// blending. Here the same work is split into:
//   k_setup       one thread per triangle: transform, cull, snap to 1/256 px,
//                 bbox, interpolation constants (the raster specification);
//   k_setup_clip  the same for the triangles that cross the near plane,
//                 clipped into one or two; the pair count of every
//                 512-triangle block;
//   scan + emit   the blocks' pair counts scanned, then one (tile, triangle)
//                 pair per 16x16 tile the bbox touches, written in triangle
//                 order; the key holds the tile id (bits 0-23) and the 8x4
//                 micro-tiles the bbox overlaps (bits 24-31);
//   radix sort    stable LSD sort of the pairs by tile id, 8 bits a pass, in
//                 chunks (digit counts, then a scatter with warp-private
//                 ranks), so every tile's list keeps primitive order (the
//                 mask bits ride along unsorted);
//   k_tile_lists  begin/end of each tile's list, and the tiles by list length.
#include <algorithm>
#include <cstdio>

#include "oit_device.cuh"
#include "oit_internal.h"
#include "oit_launch.cuh"

namespace oit {
using namespace oitd;

namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;  // 4096 elements per block
constexpr int kRadixThreads = 256;
constexpr int kRadixRounds = 8;
constexpr int kRadixBits = 8;
constexpr int kRadixBins = 1 << kRadixBits;

// ---------------------------------------------------------------------------
// Setup (object.vert.glsl:32-39 + near-plane clip + viewport transform +
// triangle setup)
// ---------------------------------------------------------------------------
// One clip-space vertex with the attributes the raster interpolates.
struct ClipVert {
  float x, y, z, w, vz, nx, ny, nz;
};

// The vertex where edge a -> b crosses the near plane z = 0 (Vulkan clip
// space): attributes interpolated linearly at t = za / (za - zb), z exactly 0.
__device__ __forceinline__ ClipVert near_cut(const ClipVert& a, const ClipVert& b) {
  const float t = __fdiv_rn(a.z, __fsub_rn(a.z, b.z));
  ClipVert r;
  r.x = __fmaf_rn(t, __fsub_rn(b.x, a.x), a.x);
  r.y = __fmaf_rn(t, __fsub_rn(b.y, a.y), a.y);
  r.z = 0.0f;
  r.w = __fmaf_rn(t, __fsub_rn(b.w, a.w), a.w);
  r.vz = __fmaf_rn(t, __fsub_rn(b.vz, a.vz), a.vz);
  r.nx = __fmaf_rn(t, __fsub_rn(b.nx, a.nx), a.nx);
  r.ny = __fmaf_rn(t, __fsub_rn(b.ny, a.ny), a.ny);
  r.nz = __fmaf_rn(t, __fsub_rn(b.nz, a.nz), a.nz);
  return r;
}

// The 8x4 micro-tiles that a triangle may cover, for a bbox over at most 2 x 2
// tiles: byte 2 * j + i holds the key bits of tile (i, j) of the bbox; all bits
// set stands for all of the bbox's. Half of the (triangle, micro-tile) pairs
// whose bboxes meet share no sample: a triangle of 3 to 6 pixels has a bbox of
// 16 to 26, over two or three micro-tiles.
__device__ __forceinline__ uint32_t micro_bits(uint32_t micro, int i, int j) {
  return (micro >> (8 * (2 * j + i))) & 0xFFu;
}

// Area (in 1/256 pixel squared, times four: 1.5 pixels) up to which a triangle's
// centres are tested. Against never testing them, 948x592 frames of 65,280 small
// triangles 51.4 us against 55.5 (linked list) and 53.5 (WBOIT), of 261,120 77.3
// against 78.2 and 71.9 against 74.8; testing every triangle's is within 1%.
constexpr int kSliverArea = 4 * 98304;

// Coverage of a small triangle (edge functions in 32 bits; E = 2 e + top_left
// - 1, no E negative: inside, as in the tile rasters). False when it covers no
// sample of its pixel bbox, as far as that is tested: every sample of at most
// 2x2 pixels; with want_micro and one sample a pixel, the centres of at most
// 8x16 of a sliver. `covered` is then its micro-tiles, without those that
// lie outside an edge. (With more samples few of them do: Simple 1283x717 4x
// MSAA 141 -> 138 us for the raster, 22 -> 27 us for its two setups.)
template <int S>
__device__ __forceinline__ bool small_coverage(const int (&X)[3], const int (&Y)[3], int tl, int bx0, int by0, int bx1,
                                               int by1, bool want_micro, uint32_t& covered) {
  const int w = bx1 - bx0, h = by1 - by0;
  const bool tiny = w <= 1 && h <= 1;
  if (!tiny && (S > 1 || !want_micro)) return true;
  const int t0 = tl & 1, t1 = (tl >> 1) & 1, t2 = (tl >> 2) & 1;
  // edge values per 1/256 pixel, and at the bbox's first pixel's corner
  const int A0 = 2 * (Y[1] - Y[2]), B0 = 2 * (X[2] - X[1]), A1 = 2 * (Y[2] - Y[0]), B1 = 2 * (X[0] - X[2]);
  const int ox = bx0 * 256, oy = by0 * 256;
  const int E0 = B0 * (oy - Y[1]) + A0 * (ox - X[1]) + t0 - 1, E1 = B1 * (oy - Y[2]) + A1 * (ox - X[2]) + t1 - 1;
  const int sum = 2 * ((X[1] - X[0]) * (Y[2] - Y[0]) - (Y[1] - Y[0]) * (X[2] - X[0])) + t0 + t1 + t2 - 3;
  if (tiny) {
    bool any = false;
#pragma unroll
    for (int y = 0; y < 2; ++y)
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const bool in = x <= w && y <= h;
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const int2 sp = sample_pos<S>(s);
          const int e0 = E0 + A0 * (256 * x + sp.x) + B0 * (256 * y + sp.y);
          const int e1 = E1 + A1 * (256 * x + sp.x) + B1 * (256 * y + sp.y);
          any |= in && (e0 | e1 | (sum - e0 - e1)) >= 0;
        }
      }
    if (!any) return false;
  }
  if (S > 1 || !want_micro) return true;
  // per edge: values per pixel, and at the first pixel's centre
  const int A[3] = {256 * A0, 256 * A1, -256 * (A0 + A1)}, B[3] = {256 * B0, 256 * B1, -256 * (B0 + B1)};
  int M[3] = {E0 + 128 * A0 + 128 * B0, E1 + 128 * A1 + 128 * B1, 0};
  M[2] = sum - M[0] - M[1];
  // (the centres are only worth testing where few of them are expected inside:
  // `sum` is four times the area)
  if (w <= 7 && h <= 15 && !tiny && sum < kSliverArea) {
    int none = -1;  // negative: no pixel yet
#pragma unroll 1
    for (int y = 0; y <= h && none < 0; ++y) {
      int e0 = M[0] + B[0] * y, e1 = M[1] + B[1] * y, e2 = M[2] + B[2] * y;
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        none &= e0 | e1 | e2;
        e0 += A[0];
        e1 += A[1];
        e2 += A[2];
      }
    }
    if (none < 0) return false;
  }
  const int mx0 = bx0 >> 3, my0 = by0 >> 2, mx1 = bx1 >> 3, my1 = by1 >> 2, tx0 = mx0 >> 1, ty0 = my0 >> 2;
  if ((mx1 >> 1) - tx0 > 1 || (my1 >> 2) - ty0 > 1) return true;
  uint32_t m = 0;
#pragma unroll 1
  for (int my = my0; my <= my1; ++my) {
    // the micro-tile's pixels within the bbox, relative to its first pixel; each
    // edge's largest value over them
    const int y0 = max(my * 4 - by0, 0), y1 = min(my * 4 + 3 - by0, h);
    int r[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) r[i] = M[i] + (B[i] > 0 ? y1 : y0) * B[i];
#pragma unroll 1
    for (int mx = mx0; mx <= mx1; ++mx) {
      const int x0 = max(mx * 8 - bx0, 0), x1 = min(mx * 8 + 7 - bx0, w);
      int e = 0;
#pragma unroll
      for (int i = 0; i < 3; ++i) e |= r[i] + (A[i] > 0 ? x1 : x0) * A[i];
      if (e >= 0) m |= 1u << (16 * ((my >> 2) - ty0) + 8 * ((mx >> 1) - tx0) + 2 * (my & 3) + (mx & 1));
    }
  }
  if (!m) return false;
  covered = m;
  return true;
}

// Setup of one triangle of clip-space vertices: the 0 <= z <= w, w > 0 test,
// projection, snap, orientation (back faces culled for opaque triangles), bbox,
// the small-triangle sample test and the record T (and Q). bb: the bbox (empty
// when dropped, bit 31 of .y = has_second). micro: its micro-tiles. Returns the
// number of its tiles (0 when dropped; T, Q and micro are not set then).
template <int S>
__device__ __forceinline__ uint32_t setup_half(const SetupParams& p, bool opaque, const ClipVert (&cv)[3],
                                               const float* c0, bool has_second, TriSetup& T, TriPersp& Q,
                                               uint2& bb, uint32_t& micro) {
  const uint32_t second_bit = has_second ? 0x80000000u : 0u;
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (!(cv[k].w > 0.0f) || !(cv[k].z >= 0.0f) || !(cv[k].z <= cv[k].w)) ok = false;
  int X[3], Y[3];
  float zz[3], q[3];
  if (ok) {
    const float halfW = 0.5f * (float)p.RW, halfH = 0.5f * (float)p.RH;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      q[k] = __fdiv_rn(1.0f, cv[k].w);
      const float ndx = __fmul_rn(cv[k].x, q[k]), ndy = __fmul_rn(cv[k].y, q[k]);
      zz[k] = __fmul_rn(cv[k].z, q[k]);
      const float sx = __fmaf_rn(ndx, halfW, halfW), sy = __fmaf_rn(ndy, halfH, halfH);
      if (!(fabsf(sx) < 16384.0f) || !(fabsf(sy) < 16384.0f)) ok = false;
      X[k] = __float2int_rn(__fmul_rn(sx, 256.0f));
      Y[k] = __float2int_rn(__fmul_rn(sy, 256.0f));
    }
  }
  long long area = 0;
  if (ok) {
    area = (long long)(X[1] - X[0]) * (long long)(Y[2] - Y[0]) - (long long)(Y[1] - Y[0]) * (long long)(X[2] - X[0]);
    if (area == 0) ok = false;
    // area > 0: clockwise on the y-down framebuffer = back face for
    // VK_FRONT_FACE_COUNTER_CLOCKWISE (main.cpp:520-525); only opaque
    // triangles cull back faces (transparent ones are double-sided, oit.cpp:703).
    if (area > 0 && opaque) ok = false;
  }
  // counter-clockwise (area < 0) triangles swap vertices 1 and 2 so that
  // every record winds one way; selects, not an index, keep it in registers
  const bool sw = ok && area < 0;
  if (sw) area = -area;
  int bx0 = 0, by0 = 0, bx1 = -1, by1 = -1;
  int PX[3], PY[3];
  if (ok) {
    PX[0] = X[0]; PY[0] = Y[0];
    PX[1] = sw ? X[2] : X[1]; PY[1] = sw ? Y[2] : Y[1];
    PX[2] = sw ? X[1] : X[2]; PY[2] = sw ? Y[1] : Y[2];
    bx0 = max(min(PX[0], min(PX[1], PX[2])) >> 8, 0);
    by0 = max(min(PY[0], min(PY[1], PY[2])) >> 8, 0);
    bx1 = min(max(PX[0], max(PX[1], PX[2])) >> 8, p.RW - 1);
    by1 = min(max(PY[0], max(PY[1], PY[2])) >> 8, p.RH - 1);
    if (bx0 > bx1 || by0 > by1) ok = false;
  }
  int tl = 0;
  if (ok) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int a = (i + 1) % 3, b = (i + 2) % 3;
      const int dx = PX[b] - PX[a], dy = PY[b] - PY[a];
      if (dy < 0 || (dy == 0 && dx > 0)) tl |= 1 << i;
    }
  }
  const int minX = min(PX[0], min(PX[1], PX[2])), maxX = max(PX[0], max(PX[1], PX[2]));
  const int minY = min(PY[0], min(PY[1], PY[2])), maxY = max(PY[0], max(PY[1], PY[2]));
  const bool small = maxX - minX < kSmallExtent && maxY - minY < kSmallExtent;
  // Triangles that cover no sample never reach the bins. A large one over a
  // bbox of at most 2x2 pixels (at the frame's edge) is tested in 64 bits.
  uint32_t covered = 0xFFFFFFFFu;
  if (ok && small) {
    ok = small_coverage<S>(PX, PY, tl, bx0, by0, bx1, by1, p.micro != nullptr, covered);
  } else if (ok && (bx1 - bx0) <= 1 && (by1 - by0) <= 1) {
    bool any = false;
    const int4 a = make_int4(PX[0], PY[0], PX[1], PY[1]), b = make_int4(PX[2], PY[2], tl, 0);
    for (int py = by0; py <= by1; ++py)
      for (int px = bx0; px <= bx1; ++px)
#pragma unroll 1
        for (int s = 0; s < S; ++s) {
          const int2 sp = sample_pos<S>(s);
          if (inside(edges_at(a, b, px * 256 + sp.x, py * 256 + sp.y), tl)) any = true;
        }
    ok = any;
  }
  if (!ok) {
    // an empty bbox (x0 > x1): the unbinned walk of an overflowed frame
    // tests every triangle's bbox
    bb = make_uint2(0xFFFFFFFFu, second_bit);
    return 0;
  }
  T.xy01 = make_int4(PX[0], PY[0], PX[1], PY[1]);
  float alpha = __fmaf_rn(c0[3], p.alpha_width, p.alpha_min);
  alpha = (alpha > 0.0f) ? alpha : 0.0f;
  alpha = (alpha < 1.0f) ? alpha : 1.0f;
  const int acode = __float2int_rn(__fmul_rn(alpha, 255.0f));
  T.xy2f = make_int4(PX[2], PY[2], tl | (small ? kFlagSmall : 0) | (acode << 8), __float_as_int(alpha));
  const float z0 = zz[0], z1 = sw ? zz[2] : zz[1], z2 = sw ? zz[1] : zz[2];
  T.zc = make_float4(z0, __fsub_rn(z1, z0), __fsub_rn(z2, z0), __fdiv_rn(1.0f, __ll2float_rn(area)));
  const float q0 = q[0], q1 = sw ? q[2] : q[1], q2 = sw ? q[1] : q[2];
  const ClipVert& v1 = sw ? cv[2] : cv[1];
  const ClipVert& v2 = sw ? cv[1] : cv[2];
  T.n0 = make_float4(__fmul_rn(cv[0].nx, q0), __fmul_rn(cv[0].ny, q0), __fmul_rn(cv[0].nz, q0), c0[0]);
  T.n1 = make_float4(__fmul_rn(v1.nx, q1), __fmul_rn(v1.ny, q1), __fmul_rn(v1.nz, q1), c0[1]);
  T.n2 = make_float4(__fmul_rn(v2.nx, q2), __fmul_rn(v2.ny, q2), __fmul_rn(v2.nz, q2), c0[2]);
  if (p.persp) {
    Q.q = make_float4(q0, q1, q2, 0.0f);
    Q.vzq = make_float4(__fmul_rn(cv[0].vz, q0), __fmul_rn(v1.vz, q1), __fmul_rn(v2.vz, q2), 0.0f);
  }
  bb = make_uint2((uint32_t)bx0 | ((uint32_t)by0 << 16), ((uint32_t)bx1 | ((uint32_t)by1 << 16)) | second_bit);
  micro = covered;
  const int tx0 = bx0 / kTile, tx1 = bx1 / kTile, ty0 = by0 / kTile, ty1 = by1 / kTile;
  uint32_t pairs = (uint32_t)((tx1 - tx0 + 1) * (ty1 - ty0 + 1));
  if (covered != 0xFFFFFFFFu) {  // the tiles with a micro-tile to test
    pairs = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) pairs += micro_bits(covered, k & 1, k >> 1) != 0u;
  }
  return pairs;
}

// Triangle t's clip-space vertices (object.vert.glsl:32-39) and colour.
// Flattened mesh: 10 floats per vertex, colour of the first vertex.
// Instanced: template vertex (6 floats) scaled by the instance's radius and
// moved to its centre, one multiply and one add each rounded (as a flattened
// copy of the template is built on the host), colour of the instance.
__device__ __forceinline__ const float* clip_vertices(const SetupParams& p, uint32_t t, ClipVert (&cv)[3]) {
  const uint32_t tg = p.first_triangle + t;
  const float* vtx = p.vertices;
  const float* inst = nullptr;
  uint32_t tri = tg;
  if (p.instances) {
    const uint32_t o = tg / p.template_triangles;
    tri = tg - o * p.template_triangles;
    inst = p.instances + 8 * (size_t)o;
  }
  const uint32_t i0 = p.indices[3 * (size_t)tri + 0];
  const uint32_t i1 = p.indices[3 * (size_t)tri + 1];
  const uint32_t i2 = p.indices[3 * (size_t)tri + 2];
  const uint32_t vid[3] = {i0, i1, i2};
  // scene constants from device memory (every thread reads the same 80 bytes)
  float m[16], v[16];
  {
    const float4* sc = reinterpret_cast<const float4*>(p.scene);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 c = sc[k];
      m[4 * k + 0] = c.x;
      m[4 * k + 1] = c.y;
      m[4 * k + 2] = c.z;
      m[4 * k + 3] = c.w;
    }
    // of the view matrix only row 2 (view-space z) is used: columns' z entries
#pragma unroll
    for (int k = 0; k < 4; ++k) v[4 * k + 2] = p.scene[16 + 4 * k + 2];
  }
  float4 ic = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
  if (inst) ic = *reinterpret_cast<const float4*>(inst);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float* pv = inst ? vtx + 6 * (size_t)vid[k] : vtx + 10 * (size_t)vid[k];
    float x = pv[0], y = pv[1], z = pv[2];
    if (inst) {
      x = __fadd_rn(__fmul_rn(x, ic.w), ic.x);
      y = __fadd_rn(__fmul_rn(y, ic.w), ic.y);
      z = __fadd_rn(__fmul_rn(z, ic.w), ic.z);
    }
    cv[k].x = __fmaf_rn(m[0], x, __fmaf_rn(m[4], y, __fmaf_rn(m[8], z, m[12])));
    cv[k].y = __fmaf_rn(m[1], x, __fmaf_rn(m[5], y, __fmaf_rn(m[9], z, m[13])));
    cv[k].z = __fmaf_rn(m[2], x, __fmaf_rn(m[6], y, __fmaf_rn(m[10], z, m[14])));
    cv[k].w = __fmaf_rn(m[3], x, __fmaf_rn(m[7], y, __fmaf_rn(m[11], z, m[15])));
    cv[k].vz = __fmaf_rn(v[2], x, __fmaf_rn(v[6], y, __fmaf_rn(v[10], z, v[14])));
    cv[k].nx = pv[3];
    cv[k].ny = pv[4];
    cv[k].nz = pv[5];
  }
  return inst ? inst + 4 : vtx + 10 * (size_t)i0 + 6;  // color.rgba
}

// pair_count of a triangle the near plane crosses, between k_setup and
// k_setup_clip (no triangle overlaps 2^32 - 1 tiles)
constexpr uint32_t kClipPending = 0xFFFFFFFFu;

// One thread per triangle. Triangles wholly in front of the near plane, or
// wholly behind it (dropped by the clip-volume test), are set up here; a
// crossing triangle is marked for k_setup_clip, which keeps this kernel's
// vertices in registers and free of the clip's extra state.
// A warp's records go through shared memory and out in whole 512-byte lines: a
// thread's own 16-byte stores at a stride of 96 bytes fill half a sector each.
// With that and 32-bit sample tests of tiny triangles: 983,040 triangles 35 ->
// 27 us, 15.7 million with WBOIT's records 550 -> 401 us (5.5 TB/s; 548 us with
// the micro-tile test, which saves the raster twice that).
constexpr int kSetupThreads = 256;
struct SetupStage {
  uint4 rec[32][7];    // TriSetup, padded: 32 lanes' 16-byte stores in distinct banks
  uint4 persp[32][3];  // TriPersp, padded
};

template <int S>
__global__ void __launch_bounds__(kSetupThreads, 4) k_setup(SetupParams p) {
  frame_order();
  extern __shared__ __align__(16) unsigned char setup_smem[];
  const uint32_t t = blockIdx.x * kSetupThreads + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const size_t stage_bytes = p.persp ? sizeof(SetupStage) : sizeof(SetupStage::rec);
  SetupStage& st = *reinterpret_cast<SetupStage*>(setup_smem + (threadIdx.x >> 5) * stage_bytes);
  bool record = false;
  if (t < p.num_triangles) {
    ClipVert cv[3];
    const float* c0 = clip_vertices(p, t, cv);
    const int nin = (cv[0].z >= 0.0f) + (cv[1].z >= 0.0f) + (cv[2].z >= 0.0f);
    if (nin == 1 || nin == 2) {
      p.pair_count[t] = kClipPending;
    } else {
      TriSetup T;
      TriPersp Q;
      uint2 bb;
      uint32_t micro = 0;
      const uint32_t pairs = setup_half<S>(p, t >= p.opaque_from, cv, c0, false, T, Q, bb, micro);
      p.pair_count[t] = pairs;
      p.bbox[t] = bb;
      if (p.micro) p.micro[t] = micro;
      record = pairs != 0;
      if (record) {
        const uint4* src = reinterpret_cast<const uint4*>(&T);
#pragma unroll
        for (int k = 0; k < 6; ++k) st.rec[lane][k] = src[k];
        if (p.persp) {
          st.persp[lane][0] = reinterpret_cast<const uint4*>(&Q)[0];
          st.persp[lane][1] = reinterpret_cast<const uint4*>(&Q)[1];
        }
      }
    }
  }
  const uint32_t records = __ballot_sync(0xffffffffu, record);
  __syncwarp();
  uint4* out = reinterpret_cast<uint4*>(p.setup) + (size_t)(t - lane) * 6;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const int i = lane + 32 * k, r = i / 6;
    if ((records >> r) & 1u) out[i] = st.rec[r][i - 6 * r];
  }
  if (blockIdx.x == 0) {
    if (p.clear_fragments && threadIdx.x == 0) *p.clear_fragments = 0ull;
    if (p.clear_counter && threadIdx.x == 0) *p.clear_counter = 0u;
    if (p.clear_order && threadIdx.x < 2 * kOrderBuckets) p.clear_order[threadIdx.x] = 0u;
  }
  if (!p.persp) return;
  uint4* outp = reinterpret_cast<uint4*>(p.persp) + (size_t)(t - lane) * 2;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int i = lane + 32 * k, r = i >> 1;
    if ((records >> r) & 1u) outp[i] = st.persp[r][i & 1];
  }
}

// The record of one half of a clipped triangle. Returns its pair count.
template <int S>
__device__ __forceinline__ uint32_t store_half(const SetupParams& p, uint32_t slot, bool opaque,
                                               const ClipVert (&cv)[3], const float* c0, bool has_second) {
  TriSetup T;
  TriPersp Q;
  uint2 bb;
  uint32_t micro = 0;
  const uint32_t pairs = setup_half<S>(p, opaque, cv, c0, has_second, T, Q, bb, micro);
  p.bbox[slot] = bb;
  if (p.micro) p.micro[slot] = micro;
  if (pairs) {
    reinterpret_cast<TriSetup*>(p.setup)[slot] = T;
    if (p.persp) reinterpret_cast<TriPersp*>(p.persp)[slot] = Q;
  }
  return pairs;
}

// A triangle k_setup marked: Sutherland-Hodgman against z = 0 over the edges
// 0->1, 1->2, 2->0 keeps the triangle's winding; 3 vertices give one triangle
// (record t), 4 the fan (0, 1, 2) in record t and (0, 2, 3) in record
// num_triangles + t. The vertices are derived from the mesh again, with the
// same rounded operations as in k_setup. Returns the pair count.
template <int S>
__device__ __forceinline__ uint32_t setup_clipped(const SetupParams& p, uint32_t t) {
  ClipVert cv[3];
  const float* c0 = clip_vertices(p, t, cv);
  const bool opaque = t >= p.opaque_from;
  const bool in[3] = {cv[0].z >= 0.0f, cv[1].z >= 0.0f, cv[2].z >= 0.0f};
  // the polygon: in-front vertices and edge cuts in edge order (3 or 4 of them)
  ClipVert poly[4];
  int n = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int k1 = k == 2 ? 0 : k + 1;
    if (in[k] && n < 4) poly[n++] = cv[k];
    if (in[k] != in[k1] && n < 4) poly[n++] = near_cut(cv[k], cv[k1]);
  }
  uint32_t pairs = 0;
  if (n >= 3) {
    const ClipVert first[3] = {poly[0], poly[1], poly[2]};
    pairs = store_half<S>(p, t, opaque, first, c0, n == 4);
    if (n == 4) {
      const ClipVert second[3] = {poly[0], poly[2], poly[3]};
      pairs += store_half<S>(p, p.num_triangles + t, opaque, second, c0, false);
    }
  } else {
    p.bbox[t] = make_uint2(0xFFFFFFFFu, 0u);  // not reached: a crossing triangle gives 3 or 4
  }
  p.pair_count[t] = pairs;
  return pairs;
}

// Triangles per block of the clip kernel (4 per thread) and of the emit
// kernel (one per thread): the pair-count sums are per 512 triangles.
constexpr int kClipThreads = 128;
constexpr int kEmitItems = 4;
constexpr int kEmitTile = kClipThreads * kEmitItems;

// The marked triangles of each 512-triangle block are clipped one by one;
// with block_sums, the block's pair count (after clipping) is written there,
// the first level of the pair-offset scan. pair_count is 16-byte aligned.
template <int S>
__global__ void __launch_bounds__(kClipThreads, 12) k_setup_clip(SetupParams p, uint32_t* block_sums) {
  frame_order();
  __shared__ uint32_t warp_sums[kClipThreads / 32];
  const uint32_t n = p.num_triangles;
  const uint32_t t0 = blockIdx.x * kEmitTile + threadIdx.x * kEmitItems;
  uint32_t c[kEmitItems] = {0u, 0u, 0u, 0u};
  if (t0 + 3 < n) {
    const uint4 v = *reinterpret_cast<const uint4*>(p.pair_count + t0);
    c[0] = v.x; c[1] = v.y; c[2] = v.z; c[3] = v.w;
  } else {
#pragma unroll
    for (int k = 0; k < kEmitItems; ++k) c[k] = t0 + k < n ? p.pair_count[t0 + k] : 0u;
  }
  uint32_t sum = 0;
#pragma unroll 1
  for (int k = 0; k < kEmitItems; ++k) {
    const uint32_t ck = c[k] == kClipPending ? setup_clipped<S>(p, t0 + (uint32_t)k) : c[k];
    sum += ck;
  }
  if (!block_sums) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t b = 0;
#pragma unroll
    for (int w = 0; w < kClipThreads / 32; ++w) b += warp_sums[w];
    block_sums[blockIdx.x] = b;
  }
}

// ---------------------------------------------------------------------------
// Exclusive scan (u32), 4096 elements per block, recursive over block sums.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total, uint32_t* smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    uint32_t w = lane < nw ? smem[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    smem[32 + lane] = w;  // inclusive warp prefix
  }
  __syncthreads();
  const uint32_t warp_prefix = warp ? smem[32 + warp - 1] : 0u;
  *total = smem[32 + (blockDim.x >> 5) - 1];
  __syncthreads();
  return warp_prefix + x - v;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_sums(const uint32_t* in, size_t n, uint32_t* sums) {
  frame_order();
  __shared__ uint32_t smem[64];
  const size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
  uint32_t s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i)
    if (base + i < n) s += in[base + i];
  uint32_t total;
  block_exclusive_scan(s, &total, smem);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_apply(const uint32_t* in, uint32_t* out, size_t n,
                                                             const uint32_t* offsets, uint32_t* grand_total) {
  frame_order();
  __shared__ uint32_t smem[64];
  const size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    v[i] = (base + i < n) ? in[base + i] : 0u;
    s += v[i];
  }
  uint32_t total;
  uint32_t pre = block_exclusive_scan(s, &total, smem) + (offsets ? offsets[blockIdx.x] : 0u);
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (base + i < n) out[base + i] = pre;
    pre += v[i];
  }
  if (grand_total && blockIdx.x == gridDim.x - 1 && threadIdx.x == kScanThreads - 1) *grand_total = pre;
}

// One block walks the tiles of a short array in order, carrying the running
// sum: one launch instead of three for up to kScanLoopTiles tiles.
constexpr int kScanLoopTiles = 8;

__global__ void __launch_bounds__(kScanThreads) k_scan_loop(const uint32_t* in, uint32_t* out, size_t n,
                                                            uint32_t* grand_total) {
  frame_order();
  __shared__ uint32_t smem[64];
  uint32_t carry = 0;
  for (size_t tile = 0; tile * kScanTile < n; ++tile) {
    const size_t base = tile * kScanTile + (size_t)threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
      v[i] = (base + i < n) ? in[base + i] : 0u;
      s += v[i];
    }
    uint32_t total;
    uint32_t pre = block_exclusive_scan(s, &total, smem) + carry;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
      if (base + i < n) out[base + i] = pre;
      pre += v[i];
    }
    carry += total;
  }
  if (grand_total && threadIdx.x == 0) *grand_total = carry;
}

size_t blocks_for(size_t n) { return (n + kScanTile - 1) / kScanTile; }

// Exclusive scan of n u32 values; grand_total (device, may be null) receives the sum.
cudaError_t scan_exclusive(const uint32_t* in, uint32_t* out, size_t n, uint32_t* tmp, uint32_t* grand_total,
                           cudaStream_t s, uint64_t* launches) {
  if (n == 0) {
    if (grand_total) return cudaMemsetAsync(grand_total, 0, 4, s);
    return cudaSuccess;
  }
  const size_t nb = blocks_for(n);
  if (nb == 1) {
    launch_in_frame(k_scan_apply, 1, kScanThreads, 0, s, in, out, n, nullptr, grand_total);
    ++*launches;
    return cudaGetLastError();
  }
  if (nb <= (size_t)kScanLoopTiles) {
    launch_in_frame(k_scan_loop, 1, kScanThreads, 0, s, in, out, n, grand_total);
    ++*launches;
    return cudaGetLastError();
  }
  uint32_t* sums = tmp;
  uint32_t* rest = tmp + nb;
  launch_in_frame(k_scan_sums, (unsigned)nb, kScanThreads, 0, s, in, n, sums);
  ++*launches;
  cudaError_t e = scan_exclusive(sums, sums, nb, rest, nullptr, s, launches);
  if (e != cudaSuccess) return e;
  launch_in_frame(k_scan_apply, (unsigned)nb, kScanThreads, 0, s, in, out, n, sums, grand_total);
  ++*launches;
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Pair emission: pair j of triangle t lands at pair_offset[t] + j.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t emit_bbox(uint2 bb, uint32_t micro, uint32_t t, uint32_t tile_base, int tiles_x,
                                              uint32_t off, uint32_t j, uint32_t* keys, uint32_t* tris,
                                              size_t capacity) {
  const int bx0 = bb.x & 0xFFFF, by0 = bb.x >> 16, bx1 = bb.y & 0xFFFF, by1 = (bb.y >> 16) & 0x7FFF;
  if (bx0 > bx1 || by0 > by1) return j;
  const int tx0 = bx0 / kTile, ty0 = by0 / kTile, tx1 = bx1 / kTile, ty1 = by1 / kTile;
  if (micro != 0xFFFFFFFFu) {  // at most 2 x 2 tiles
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t bits = micro_bits(micro, k & 1, k >> 1);
      if (!bits) continue;
      const size_t pos = (size_t)off + j;
      if (pos >= capacity) return j;
      keys[pos] = (tile_base + (uint32_t)((ty0 + (k >> 1)) * tiles_x + tx0 + (k & 1))) | (bits << kMaskShift);
      tris[pos] = t;
      ++j;
    }
    return j;
  }
  // (a loop of its own: with the micro-tiles' test in it, a step took half as
  // long again, and one thread makes the steps of a triangle over thousands of
  // tiles: 80 triangles over most of 1280x720, 154 us against 100)
  for (int ty = ty0; ty <= ty1; ++ty) {
    // rows of 8x4 micro-tiles the bbox overlaps in this tile row
    const int ly0 = max(by0 - ty * kTile, 0), ly1 = min(by1 - ty * kTile, kTile - 1);
    uint32_t rows = 0;
    for (int r = ly0 >> 2; r <= (ly1 >> 2); ++r) rows |= 3u << (2 * r);
    for (int tx = tx0; tx <= tx1; ++tx, ++j) {
      const size_t pos = (size_t)off + j;
      if (pos >= capacity) return j;
      const int lx0 = max(bx0 - tx * kTile, 0), lx1 = min(bx1 - tx * kTile, kTile - 1);
      const uint32_t cols = (lx0 <= 7 ? 0x55u : 0u) | (lx1 >= 8 ? 0xAAu : 0u);
      keys[pos] = (tile_base + (uint32_t)(ty * tiles_x + tx)) | ((rows & cols) << kMaskShift);
      tris[pos] = t;
    }
  }
  return j;
}

// The pairs of the block's 512 triangles, one per thread: a triangle's
// offset is the scanned block sum plus the exclusive prefix of the counts
// before it in the block (written to pair_offset, which the bin-overflow walk
// reads); it emits its first (or only) half's tiles, then the second half's
// (record n + t) when the near-plane clip split it.
__global__ void __launch_bounds__(kEmitTile) k_emit(const uint32_t* pair_count, uint32_t* pair_offset,
                                                    const uint32_t* block_offsets, const uint2* bbox,
                                                    const uint32_t* micro, uint32_t n, int tiles_x,
                                                    uint32_t opaque_from, uint32_t num_tiles, uint32_t* keys,
                                                    uint32_t* tris, size_t capacity, const uint32_t* total,
                                                    uint32_t* err) {
  frame_order();
  __shared__ uint32_t smem[64];
  if (blockIdx.x == 0 && threadIdx.x == 0 && *total > capacity) atomicOr(err, 1u);  // OIT_DEVERR_BIN_OVERFLOW
  const uint32_t t = blockIdx.x * kEmitTile + threadIdx.x;
  const uint32_t c = t < n ? pair_count[t] : 0u;
  uint32_t block_total;
  const uint32_t off = block_exclusive_scan(c, &block_total, smem) + block_offsets[blockIdx.x];
  if (t >= n) return;
  pair_offset[t] = off;
  if (!c) return;
  const uint2 bb = bbox[t];
  const uint32_t tile_base = t < opaque_from ? num_tiles : 0u;
  const uint32_t j =
      emit_bbox(bb, micro ? micro[t] : 0xFFFFFFFFu, t, tile_base, tiles_x, off, 0u, keys, tris, capacity);
  if (bb.y >> 31)
    emit_bbox(bbox[n + t], micro ? micro[n + t] : 0xFFFFFFFFu, n + t, tile_base, tiles_x, off, j, keys, tris, capacity);
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort of (key, value) pairs, 8-bit digits.
//
// The pairs are cut into chunks: at most kSortBlocks of a multiple of 2048
// pairs, or any number of 2048. k_radix_hist counts each chunk's digits;
// k_radix_scatter derives its chunk's output offset for every digit (the
// digit's start over all chunks plus the counts of the chunks before it) from
// those counts itself, or from their sums by k_digit_scan, and
// moves the chunk 2048 pairs at a time: each warp ranks its 256 consecutive
// pairs with its own shared-memory counters, so a sub-tile costs three block
// barriers. Pairs keep their order within a digit: the sort is stable. The next
// sub-tile's pairs are fetched before this one's are stored, a round trip less
// per sub-tile of a chunk of several: 11.6 us a pass of the 64-view batch's views
// on average against 17.7, for 77 registers against 64.
// ---------------------------------------------------------------------------
__device__ __forceinline__ size_t pair_count_of(const uint32_t* total, size_t capacity) {
  const size_t t = *total;
  return t < capacity ? t : capacity;
}

constexpr int kSortSubTile = kRadixThreads * kRadixRounds;  // 2048 pairs: 8 warps x 8 rounds of 32
constexpr int kSortWarps = kRadixThreads / 32;

// Digit counts of chunk blockIdx.x: counts[chunk * 256 + digit], or, with
// digit_major (many chunks, summed in place before the scatter),
// counts[digit * gridDim.x + chunk]. One shared-memory atomic per distinct
// digit per warp (tile ids of neighbouring pairs are mostly equal).
__global__ void __launch_bounds__(kRadixThreads) k_radix_hist(const uint32_t* keys, const uint32_t* total,
                                                              size_t capacity, int shift, size_t chunk,
                                                              bool digit_major, uint32_t* counts) {
  frame_order();
  __shared__ uint32_t h[kRadixBins];
  h[threadIdx.x] = 0;
  __syncthreads();
  const size_t n = pair_count_of(total, capacity);
  const size_t beg = (size_t)blockIdx.x * chunk;
  const size_t end = beg + chunk < n ? beg + chunk : n;
  const uint32_t lane = threadIdx.x & 31;
  for (size_t base = beg; base < end; base += kRadixThreads * 8) {
    uint32_t d[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const size_t i = base + (size_t)k * kRadixThreads + threadIdx.x;
      d[k] = i < end ? (keys[i] >> shift) & (kRadixBins - 1) : kRadixBins;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t peers = __match_any_sync(0xffffffffu, d[k]);
      if (d[k] < kRadixBins && (__ffs(peers) - 1) == (int)lane) atomicAdd(&h[d[k]], (uint32_t)__popc(peers));
    }
  }
  __syncthreads();
  if (digit_major) counts[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
  else counts[(size_t)blockIdx.x * kRadixBins + threadIdx.x] = h[threadIdx.x];
}

// Running sums, in place, of digit blockIdx.x's counts over the chunks
// (counts[digit * nchunks + chunk]); the scatter adds the digit's start, the
// sum of the last ones of the digits before it. A short kernel, bound by its
// launch and one or two rounds of loads; a scan of the whole array is three of
// them (Simple 1283x717 4x MSAA, sorting twice, 294 us with that and 278 with
// this; Spinlock 800x512 155 and 147; Loop64 1920x1080 286 and 281).
constexpr int kDigitScanItems = 8;

__global__ void __launch_bounds__(kRadixThreads) k_digit_scan(uint32_t* counts, uint32_t nchunks) {
  frame_order();
  __shared__ uint32_t smem[64];
  uint32_t* row = counts + (size_t)blockIdx.x * nchunks;
  uint32_t carry = 0;
  for (uint32_t base = 0; base < nchunks; base += kRadixThreads * kDigitScanItems) {
    const uint32_t first = base + threadIdx.x * kDigitScanItems;
    uint32_t v[kDigitScanItems], sum = 0;
#pragma unroll
    for (int i = 0; i < kDigitScanItems; ++i) {
      v[i] = first + i < nchunks ? row[first + i] : 0u;
      sum += v[i];
    }
    uint32_t total;
    uint32_t run = carry + block_exclusive_scan(sum, &total, smem);
#pragma unroll
    for (int i = 0; i < kDigitScanItems; ++i) {
      run += v[i];
      if (first + i < nchunks) row[first + i] = run;
    }
    carry += total;
  }
}

__global__ void __launch_bounds__(kRadixThreads) k_radix_scatter(const uint32_t* keys_in, const uint32_t* vals_in,
                                                                 uint32_t* keys_out, uint32_t* vals_out,
                                                                 const uint32_t* total, size_t capacity, int shift,
                                                                 size_t chunk, uint32_t nchunks, bool scanned,
                                                                 const uint32_t* counts) {
  frame_order();
  __shared__ uint32_t base[kRadixBins];             // output position of the chunk's next pair of each digit
  __shared__ uint32_t wcount[kSortWarps][kRadixBins];  // per warp: counts, then exclusive offsets in the sub-tile
  __shared__ uint32_t sub_total[kRadixBins];
  __shared__ uint32_t scan_s[64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const size_t n = pair_count_of(total, capacity);
  const size_t beg = (size_t)blockIdx.x * chunk;
  // this digit's pairs in all chunks, and in the chunks before this one
  if (scanned) {
    // the digit-major counts' running sums: of all chunks, and of those before this one
    const uint32_t* row = counts + (size_t)threadIdx.x * nchunks;
    const uint32_t before = blockIdx.x ? row[blockIdx.x - 1] : 0u;
    uint32_t sum_all;
    base[threadIdx.x] = block_exclusive_scan(row[nchunks - 1], &sum_all, scan_s) + before;
  } else {
    // 32 independent loads in flight per thread: the chunks' counts are read
    // by every block, so their latency, not their bytes, is the cost
    const uint32_t d = threadIdx.x;
    uint32_t all = 0, before = 0;
    for (uint32_t c0 = 0; c0 < nchunks; c0 += 32) {
      uint32_t v[32];
#pragma unroll
      for (int k = 0; k < 32; ++k) v[k] = c0 + k < nchunks ? counts[(size_t)(c0 + k) * kRadixBins + d] : 0u;
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        all += v[k];
        before += c0 + k < blockIdx.x ? v[k] : 0u;
      }
    }
    uint32_t sum_all;
    base[d] = block_exclusive_scan(all, &sum_all, scan_s) + before;
  }
  if (beg >= n) return;
  const size_t end = beg + chunk < n ? beg + chunk : n;
  uint32_t key[kRadixRounds], val[kRadixRounds], dr[kRadixRounds];
  auto fetch = [&](size_t sub, uint32_t (&k)[kRadixRounds], uint32_t (&v)[kRadixRounds]) {
    const size_t wbase = sub + (size_t)warp * (32 * kRadixRounds);
#pragma unroll
    for (int r = 0; r < kRadixRounds; ++r) {
      const size_t i = wbase + (size_t)r * 32 + lane;
      k[r] = i < end ? keys_in[i] : 0u;
      v[r] = i < end ? vals_in[i] : 0u;
    }
  };
  fetch(beg, key, val);
  for (size_t sub = beg; sub < end; sub += kSortSubTile) {
#pragma unroll
    for (int k = 0; k < kRadixBins / 32; ++k) wcount[warp][lane + 32 * k] = 0;
    __syncwarp();
    // this warp's 256 consecutive pairs of the sub-tile, 32 per round
    const size_t wbase = sub + (size_t)warp * (32 * kRadixRounds);
#pragma unroll
    for (int r = 0; r < kRadixRounds; ++r) {
      const size_t i = wbase + (size_t)r * 32 + lane;
      const uint32_t d = i < end ? (key[r] >> shift) & (kRadixBins - 1) : kRadixBins;
      const uint32_t peers = __match_any_sync(0xffffffffu, d);
      const int leader = __ffs(peers) - 1;
      uint32_t old = 0;
      if (lane == leader && d < kRadixBins) {
        old = wcount[warp][d];
        wcount[warp][d] = old + (uint32_t)__popc(peers);
      }
      old = __shfl_sync(0xffffffffu, old, leader);
      dr[r] = (d << 16) | (old + (uint32_t)__popc(peers & lt_mask));  // digit (256 = none), rank in the warp
    }
    __syncthreads();
    {
      const int d = threadIdx.x;
      uint32_t acc = 0;
#pragma unroll
      for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t c = wcount[w][d];
        wcount[w][d] = acc;
        acc += c;
      }
      sub_total[d] = acc;
    }
    __syncthreads();
    uint32_t nkey[kRadixRounds], nval[kRadixRounds];
    fetch(sub + kSortSubTile, nkey, nval);
#pragma unroll
    for (int r = 0; r < kRadixRounds; ++r) {
      const uint32_t d = dr[r] >> 16;
      if (d < kRadixBins) {
        const uint32_t pos = base[d] + wcount[warp][d] + (dr[r] & 0xFFFFu);
        keys_out[pos] = key[r];
        vals_out[pos] = val[r];
      }
    }
#pragma unroll
    for (int r = 0; r < kRadixRounds; ++r) {
      key[r] = nkey[r];
      val[r] = nval[r];
    }
    __syncthreads();
    base[threadIdx.x] += sub_total[threadIdx.x];
  }
}

// [begin, end) of every key's pair range in the sorted keys, one key a thread:
// its first pair by binary search, its end from the next key's thread. A search
// is ~20 loads deep, most of them shared by the block's threads; marking every
// change of the sorted keys instead reads all pairs and needs both arrays
// cleared.
// With `order`, each kind's tiles are also put into kOrderBuckets buckets by
// list length (a factor of two each), for the rasters to start with the longest
// lists: order[(kind * kOrderBuckets + bucket) * num_tiles + ...], order_count[kind * kOrderBuckets + bucket].
constexpr int kListKeys = 256;  // keys per block (of kListKeys + 32 threads)

__global__ void __launch_bounds__(kListKeys + 32) k_tile_lists(const uint32_t* keys, const uint32_t* total,
                                                              size_t capacity, uint32_t num_tiles, uint32_t* begin,
                                                              uint32_t* end, uint32_t* order, uint32_t* order_count,
                                                              uint32_t* host_total) {
  frame_order();
  __shared__ uint32_t first[kListKeys + 1];
  __shared__ uint32_t sample[kListKeys], range[2];
  __shared__ uint32_t cnt[2 * kOrderBuckets], base[2 * kOrderBuckets];
  const uint32_t n = (uint32_t)pair_count_of(total, capacity);
  const uint32_t k = blockIdx.x * kListKeys + threadIdx.x;
  if (host_total && blockIdx.x == 0 && threadIdx.x == 0) *host_total = *total;
  if (threadIdx.x < 2 * kOrderBuckets) cnt[threadIdx.x] = 0;
  // Twice, the block narrows the pairs its keys can start in by a factor of 256,
  // reading 256 of them at once, before each thread searches what is left: a
  // step of a search in memory is an L2 round trip.
  uint32_t lo = 0, hi = n;
#pragma unroll 1
  for (int level = 0; level < 2; ++level) {
    const uint32_t step = max((hi - lo + kListKeys - 1) / kListKeys, 1u);
    if (threadIdx.x < kListKeys) {
      const uint32_t i = lo + threadIdx.x * step;
      sample[threadIdx.x] = i < hi ? keys[i] & kTileKeyMask : 0xFFFFFFFFu;
    }
    __syncthreads();
    // the last sample below k is before k's first pair, the one after it is not
    uint32_t a = 0, c = kListKeys;
    while (a < c) {
      const uint32_t mid = (a + c) >> 1;
      if (sample[mid] < k) a = mid + 1; else c = mid;
    }
    const uint32_t klo = a ? lo + (a - 1) * step : lo, khi = min(lo + a * step, hi);
    if (level == 0) {
      if (threadIdx.x == 0) range[0] = klo;
      if (threadIdx.x == kListKeys) range[1] = khi;
      __syncthreads();
      lo = range[0];
      hi = range[1];
      __syncthreads();
    } else {
      lo = klo;
      hi = khi;
    }
  }
  if (threadIdx.x <= kListKeys) {
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if ((keys[mid] & kTileKeyMask) < k) lo = mid + 1; else hi = mid;
    }
    first[threadIdx.x] = lo;
  }
  __syncthreads();
  const bool mine = threadIdx.x < kListKeys && k < 2u * num_tiles;
  uint32_t slot = 0, rank = 0;
  if (mine) {
    const uint32_t lo = first[threadIdx.x], hi = first[threadIdx.x + 1];
    begin[k] = lo;
    end[k] = hi;
    // bucket 0: fewer than 64 pairs, then a factor of two each
    slot = (k < num_tiles ? 0u : (uint32_t)kOrderBuckets) +
           min((uint32_t)max(26 - __clz((hi - lo) | 1u), 0), (uint32_t)kOrderBuckets - 1u);
  }
  if (!order) return;
  if (mine) rank = atomicAdd(&cnt[slot], 1u);
  __syncthreads();
  if (threadIdx.x < 2 * kOrderBuckets && cnt[threadIdx.x])
    base[threadIdx.x] = atomicAdd(&order_count[threadIdx.x], cnt[threadIdx.x]);
  __syncthreads();
  if (mine) order[(size_t)slot * num_tiles + base[slot] + rank] = k < num_tiles ? k : k - num_tiles;
}

__global__ void k_fill_u32(uint32_t* dst, uint32_t v, size_t n) {
  frame_order();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) dst[i] = v;
}

__global__ void k_fill_f4(float4* dst, float4 v, size_t n) {
  frame_order();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) dst[i] = v;
}

}  // namespace

size_t scan_scratch_words(size_t n) {
  size_t words = 0;
  while (n > 1) {
    n = blocks_for(n);
    words += n;
  }
  return words + 1;
}

cudaError_t launch_fill_u32(uint32_t* dst, uint32_t value, size_t count, cudaStream_t s) {
  if (!count) return cudaSuccess;
  const unsigned blocks = (unsigned)std::min<size_t>((count + 255) / 256, 152 * 16);
  launch_in_frame(k_fill_u32, blocks, 256, 0, s, dst, value, count);
  return cudaGetLastError();
}

cudaError_t launch_fill_f4(float4* dst, float4 value, size_t count, cudaStream_t s) {
  if (!count) return cudaSuccess;
  const unsigned blocks = (unsigned)std::min<size_t>((count + 255) / 256, 152 * 16);
  launch_in_frame(k_fill_f4, blocks, 256, 0, s, dst, value, count);
  return cudaGetLastError();
}

namespace {
// k_setup, then k_setup_clip over the triangles it marked (and, with
// block_sums, the pair count of every 512-triangle block)
template <int S>
cudaError_t launch_setup_s(const SetupParams& sp, uint32_t* block_sums, cudaStream_t s, uint64_t* launches) {
  const uint32_t n = sp.num_triangles;
  const size_t smem = kSetupThreads / 32 * (sp.persp ? sizeof(SetupStage) : sizeof(SetupStage::rec));
  launch_in_frame(k_setup<S>, (n + kSetupThreads - 1) / kSetupThreads, kSetupThreads, smem, s, sp);
  ++*launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  launch_in_frame(k_setup_clip<S>, (unsigned)emit_blocks(n), kClipThreads, 0, s, sp, block_sums);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launch_setup(const SetupParams& sp, uint32_t* block_sums, cudaStream_t s, uint64_t* launches) {
  switch (sp.samples) {
    case 4: return launch_setup_s<4>(sp, block_sums, s, launches);
    case 8: return launch_setup_s<8>(sp, block_sums, s, launches);
    default: return launch_setup_s<1>(sp, block_sums, s, launches);
  }
}

// Pairs per chunk of the radix sort. Up to direct_max pairs: whole 2048-pair
// sub-tiles, at most kSortBlocks chunks, each scatter block summing the counts
// of the chunks before it. Beyond: one sub-tile per chunk (every block busy),
// each digit's counts summed over the chunks in place.
constexpr size_t kSortBlocks = 128;
bool sort_scanned(size_t capacity, size_t direct_max) { return capacity > direct_max; }
size_t sort_chunk(size_t capacity, size_t direct_max) {
  if (sort_scanned(capacity, direct_max)) return kSortSubTile;
  const size_t per = (capacity + kSortBlocks - 1) / kSortBlocks;
  const size_t sub = (per + kSortSubTile - 1) / kSortSubTile * kSortSubTile;
  return sub > (size_t)kSortSubTile ? sub : (size_t)kSortSubTile;
}
}  // namespace

size_t emit_blocks(size_t tris) { return (tris + kEmitTile - 1) / kEmitTile; }

size_t bin_scan_words(size_t tris) {
  const size_t nb = emit_blocks(tris > 0 ? tris : 1);
  return nb + scan_scratch_words(nb);
}

cudaError_t bin_setup_only(const SetupParams& sp, cudaStream_t s, uint64_t* launches) {
  const uint32_t n = sp.num_triangles;
  if (n == 0) return cudaSuccess;
  return launch_setup(sp, nullptr, s, launches);
}

// Binning, step 1: setup, clip, pair counts per 512-triangle block and their
// exclusive scan (in b.scan_tmp, read by k_emit); the number of (tile,
// triangle) pairs lands in b.total (device).
cudaError_t bin_setup_scan(const SetupParams& sp, Bins& b, cudaStream_t s, uint64_t* launches) {
  cudaError_t e;
  const uint32_t n = sp.num_triangles;
  if (n == 0) return cudaMemsetAsync(b.total, 0, 4, s);
  if ((e = launch_setup(sp, b.scan_tmp, s, launches)) != cudaSuccess) return e;
  const size_t nb = emit_blocks(n);
  return scan_exclusive(b.scan_tmp, b.scan_tmp, nb, b.scan_tmp + nb, b.total, s, launches);
}

// Binning, step 2: emit pairs in triangle order, stable radix sort by tile id,
// tile ranges. Every kernel reads the pair count from b.total and is bounded
// by b.capacity, so no host round trip is needed; pairs beyond the capacity
// are dropped and raise OIT_DEVERR_BIN_OVERFLOW.
cudaError_t bin_sort(const SetupParams& sp, Bins& b, int key_bits, int num_tiles, uint32_t* error, cudaStream_t s,
                     uint64_t* launches) {
  cudaError_t e;
  const uint32_t n = sp.num_triangles;
  if (n > 0) {
    launch_in_frame(k_emit, (unsigned)emit_blocks(n), kEmitTile, 0, s, sp.pair_count, b.pair_offset, b.scan_tmp,
                    sp.bbox, sp.micro, n, sp.tiles_x, sp.opaque_from, (uint32_t)sp.num_tiles, b.keys, b.tris,
                    b.capacity, b.total, error);
    ++*launches;
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  } else if (b.order && (e = cudaMemsetAsync(b.order_count, 0, 2 * kOrderBuckets * 4, s)) != cudaSuccess) {
    return e;  // (k_setup clears it otherwise)
  }
  const size_t chunk = sort_chunk(b.capacity, b.sort_direct_max);
  const uint32_t nchunks = (uint32_t)std::max<size_t>((b.capacity + chunk - 1) / chunk, 1);
  uint32_t *kin = b.keys, *vin = b.tris, *kout = b.keys_alt, *vout = b.tris_alt;
  const bool scanned = sort_scanned(b.capacity, b.sort_direct_max);
  for (int shift = 0; shift < key_bits; shift += kRadixBits) {
    launch_in_frame(k_radix_hist, nchunks, kRadixThreads, 0, s, kin, b.total, b.capacity, shift, chunk, scanned,
                    b.hist);
    ++*launches;
    if (scanned) {
      launch_in_frame(k_digit_scan, kRadixBins, kRadixThreads, 0, s, b.hist, nchunks);
      ++*launches;
    }
    launch_in_frame(k_radix_scatter, nchunks, kRadixThreads, 0, s, kin, vin, kout, vout, b.total, b.capacity, shift,
                    chunk, nchunks, scanned, b.hist);
    ++*launches;
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    std::swap(kin, kout);
    std::swap(vin, vout);
  }
  if (kin != b.keys) {
    std::swap(b.keys, b.keys_alt);
    std::swap(b.tris, b.tris_alt);
  }
  // ranges of both kinds: [0, num_tiles) opaque, [num_tiles, 2 num_tiles) transparent
  launch_in_frame(k_tile_lists, (unsigned)((2 * num_tiles + kListKeys - 1) / kListKeys), kListKeys + 32, 0, s, b.keys,
                  b.total, b.capacity, (uint32_t)num_tiles, b.tile_begin, b.tile_end, b.order, b.order_count,
                  b.host_total);
  ++*launches;
  return cudaGetLastError();
}

// Digit counts of the chunks.
size_t radix_hist_words(size_t pairs, bool with_scanned) {
  const size_t direct = kSortBlocks * kRadixBins;
  if (!with_scanned) return direct;
  const size_t words = (pairs + kSortSubTile - 1) / kSortSubTile * kRadixBins;
  return std::max(direct, words);
}

void srgb_host_tables(float* thr256, float* dec256) {
  static const float thr[256] = OIT_SRGB_THR_INIT;
  static const float dec[256] = OIT_SRGB_DEC_INIT;
  for (int i = 0; i < 256; ++i) {
    thr256[i] = thr[i];
    dec256[i] = dec[i];
  }
}

}  // namespace oit
