// Tile rasteriser + per-algorithm A-buffer construction.
//
// One warp per 8x4 micro-tile of a 16x16 tile, one lane per pixel. Each warp
// walks its tile's triangle list (primitive order, from the bins), collects the
// triangles whose bbox touches the micro-tile (the hits) and processes them 32
// at a time: one lane per hit prepares its edge equations and finds the pixels
// it covers, one lane per covered pixel shades a fragment, and the pixel's
// owner lane runs the algorithm's fragment body (the COLOR/DEPTH shader of the
// reference) on that pixel's state, so every pixel sees its fragments in
// primitive order -- the order the reference's hardware blender guarantees for
// tail blending and the order ordered interlock guarantees for its critical
// section. Per-pixel k-buffers live in shared memory or registers; the
// A-buffer, aux images and the tail-blended colour target are written to HBM
// once, at the end.
#pragma once

#include <cuda_fp16.h>

#include <algorithm>

#include "oit_device.cuh"
#include "oit_launch.cuh"

namespace oitd {

using oit::RasterParams;

constexpr uint32_t kFull = 0xffffffffu;
constexpr unsigned long long kEmpty64 = 0xFFFFFFFFFFFFFFFFull;

// A queued fragment as its owner lane sees it.
struct Frag {
  uint32_t depth;   // floatBitsToUint(gl_FragCoord.z)
  uint32_t cover;   // samples covered after early depth (gl_SampleMaskIn with post_depth_coverage)
  uint32_t packed;  // packUnorm4x8(unPremultLinearToSRGB(shading)) (WBOIT, FP32: 1 - alpha)
};

// Payload arrays of a warp's fragment queue.
struct FragPay {
  uint32_t* packed;  // one word per queued fragment
  float4* rgba;      // shading(): linear colour (unpremultiplied) and alpha, where the policy needs it
};

template <int S>
struct PixelTargets {
  float4 col[S];  // colour target per sample (premultiplied linear)

  __device__ __forceinline__ void tail(const float4& src, uint32_t cover) {
#pragma unroll
    for (int s = 0; s < S; ++s)
      if (cover & (1u << s)) rop_over(col[s], src);
  }
};

__device__ __forceinline__ float4 premult(float r, float g, float b, float a) {
  return make_float4(r * a, g * a, b * a, a);
}
__device__ __forceinline__ float4 premult(const float4& c) { return premult(c.x, c.y, c.z, c.w); }

// ---------------------------------------------------------------------------
// Policies. Each provides: kPasses, kDirect (fragments are written to the
// A-buffer by the lane that shaded them; else they are queued for their owner
// lane), kPack (needs the packed colour), kViewZ, payload_bytes() of a queued
// fragment beside its depth and coverage, smem_bytes_per_warp(L, coverage),
// init(p, smem, lane, sample, pixel), produce() on the shading lane and
// fragment() on the pixel's owner lane, once per fragment, in primitive order,
// and flush(p, valid). `sample` is the lane's sample with sample shading (each
// sample has its own A-buffer) and 0 otherwise.
// ---------------------------------------------------------------------------
// Queued fragments per warp. A feed takes as long as the lane with the most of
// them: with several samples a lane, where a fragment's blends dominate and
// shared memory is left at the registers' occupancy, it waits for more
// (Interlock 2560x1440 8x MSAA 2.75 -> 2.71 ms).
template <bool Samples>
constexpr int kQueueOf = Samples ? 96 : 64;

// oitSimple.frag.glsl:50-91
template <int S>
struct SimplePolicy {
  static constexpr bool kNodes = false;
  static constexpr bool kDirect = true;
  static constexpr bool kPack = true;
  static constexpr int kPasses = 1;
  // the most resident warps per SM it is compiled for (36: 56 registers)
  static constexpr int kWarpsPerSM = 36;
  static constexpr bool kViewZ = false;
  static __host__ __device__ size_t smem_bytes_per_warp(int, int, int = 0) { return 0; }
  // the colours and coverage that tail blending takes
  static __host__ __device__ int payload_bytes(int tail, int, int) { return tail ? 20 : 0; }
  uint32_t count;
  uint32_t eaux;
  __device__ void init(const RasterParams& p, void*, int, int sample, uint32_t pixel) {
    count = 0;
    eaux = (uint32_t)sample * p.P + pixel;
  }
  // the fragment's record at its rank among the pixel's fragments
  // (listPos = viewSize * OIT_LAYERS * sampleID + pixel, oitSimple.frag.glsl:60)
  static __device__ __forceinline__ void write(const RasterParams& p, uint32_t rank, int sample, uint32_t pixel,
                                               const Frag& f) {
    const size_t r = ((size_t)sample * p.L + rank) * p.P + pixel;
    if (p.coverage) {
      reinterpret_cast<uint4*>(p.abuf)[r] = make_uint4(f.packed, f.depth, f.cover, 0u);
    } else {
      reinterpret_cast<uint2*>(p.abuf)[r] = make_uint2(f.packed, f.depth);
    }
  }
  __device__ void flush(const RasterParams& p, bool valid) {
    if (valid) p.aux[eaux] = count;
  }
};

// oitLinkedList.frag.glsl:51-85. The node counter is a global atomic,
// aggregated per warp: one atomicAdd per batch of queued fragments hands out
// consecutive node indices in queue (primitive, then pixel) order, so a
// fragment's node index (imageAtomicAdd(imgCounter) + 1, :55) and the node it
// links to are known to the lane that shaded it.
template <int S>
struct LinkedListPolicy {
  static constexpr int kPasses = 1;
  // the most resident warps per SM it is compiled for (36: 56 registers)
  static constexpr int kWarpsPerSM = 36;
  static constexpr bool kViewZ = false;
  static constexpr bool kNodes = true;
  static constexpr bool kDirect = true;
  static constexpr bool kPack = true;
  static __host__ __device__ size_t smem_bytes_per_warp(int, int, int = 0) { return 0; }
  static __host__ __device__ int payload_bytes(int, int, int) { return 0; }
  uint32_t head;
  uint32_t eaux;
  __device__ void init(const RasterParams& p, void*, int, int sample, uint32_t pixel) {
    head = 0;
    eaux = (uint32_t)sample * p.P + pixel;
  }
  static __device__ __forceinline__ void write(const RasterParams& p, uint32_t node, uint32_t next, const Frag& f,
                                               const Shade& sh, float alpha) {
    const uint32_t mask = p.coverage ? f.cover : 0u;
    if (p.record_fp32) {
      // RGBA32F node: linear unpremultiplied colour, then depth, mask, next
      uint4* n = reinterpret_cast<uint4*>(p.abuf) + 2 * (size_t)node;
      n[0] = make_uint4(__float_as_uint(sh.r), __float_as_uint(sh.g), __float_as_uint(sh.b), __float_as_uint(alpha));
      n[1] = make_uint4(f.depth, mask, next, 0u);
    } else {
      reinterpret_cast<uint4*>(p.abuf)[node] = make_uint4(f.packed, f.depth, mask, next);
    }
  }
  __device__ void flush(const RasterParams& p, bool valid) {
    if (valid) p.aux[eaux] = head;
  }
};

// oitLoop64.frag.glsl:65-141. The per-pixel k-buffer of 64-bit keys
// (depth << 32 | rgba8) lives in shared memory, [layer][lane] per warp, kept
// sorted: the shader's atomicMin chain leaves the OIT_LAYERS smallest keys in
// ascending order and evicts the largest.
template <int S>
struct Loop64Policy {
  static constexpr bool kNodes = false;
  static constexpr bool kDirect = false;
  static constexpr bool kPack = true;
  static constexpr int kPasses = 1;
  // the most resident warps per SM it is compiled for (36: 56 registers)
  static constexpr int kWarpsPerSM = 36;
  static constexpr bool kViewZ = false;
  // keys, plus a float4 colour per slot with RGBA32F records
  static __host__ __device__ size_t smem_bytes_per_warp(int L, int, int fp32 = 0) {
    return (size_t)L * 32 * (fp32 ? 24 : 8);
  }
  static __host__ __device__ int payload_bytes(int, int fp32, int) { return fp32 ? 20 : 4; }
  unsigned long long* kb;
  float4* pay;  // RGBA32F payload moving with its key, or null
  int lane, count;
  size_t abase;
  __device__ void init(const RasterParams& p, void* smem, int, int sample, uint32_t pixel) {
    lane = threadIdx.x & 31;
    count = 0;
    abase = (size_t)sample * p.L * p.P + pixel;
    kb = reinterpret_cast<unsigned long long*>(smem);
    pay = p.record_fp32 ? reinterpret_cast<float4*>(kb + p.L * 32) : nullptr;
  }
  static __device__ __forceinline__ void produce(const RasterParams& p, int, const FragPay& q, int j, const Frag& f,
                                                 const Shade& sh, float alpha) {
    q.packed[j] = f.packed;
    if (p.record_fp32) q.rgba[j] = make_float4(sh.r, sh.g, sh.b, alpha);
  }
  __device__ __forceinline__ void fragment(const RasterParams& p, int, const Frag& f, const FragPay& q, int j,
                                           PixelTargets<S>& tg) {
    const int L = p.L;
    const unsigned long long z = ((unsigned long long)f.depth << 32) | f.packed;
    if (pay) {
      fragment_fp32(p, z, q.rgba[j], f.cover, tg);
      return;
    }
    int pos = count;
    if (count == L) {
      const unsigned long long last = kb[(L - 1) * 32 + lane];
      const bool in = z < last;  // the last key is evicted, else the fragment itself
      if (p.tail) tg.tail(decode_premult(in ? (uint32_t)last : f.packed), f.cover);
      if (!in) return;
      pos = L - 1;
    } else {
      ++count;
    }
    // from the back: half the k-buffer is read on average, all of it by the
    // shader's chain, which carries the evicted key on to the end
    while (pos > 0) {
      const unsigned long long k = kb[(pos - 1) * 32 + lane];
      if (!(z < k)) break;
      kb[pos * 32 + lane] = k;
      --pos;
    }
    kb[pos * 32 + lane] = z;
  }
  // RGBA32F: the shader's chain itself. Which of two colours with equal keys
  // moves on depends on it (a displaced key passes by its equals).
  __device__ __forceinline__ void fragment_fp32(const RasterParams& p, unsigned long long zcur, float4 pcur,
                                                uint32_t cover, PixelTargets<S>& tg) {
    for (int i = 0; i < count; ++i) {
      const unsigned long long ztest = kb[i * 32 + lane];
      if (zcur < ztest) {
        kb[i * 32 + lane] = zcur;
        const float4 t = pay[i * 32 + lane];
        pay[i * 32 + lane] = pcur;
        pcur = t;
        zcur = ztest;
      }
    }
    if (count < p.L) {
      kb[count * 32 + lane] = zcur;
      pay[count * 32 + lane] = pcur;
      ++count;
    } else if (p.tail) {
      tg.tail(premult(pcur), cover);
    }
  }
  __device__ void flush(const RasterParams& p, bool valid) {
    if (!valid) return;
    unsigned long long* ab = reinterpret_cast<unsigned long long*>(p.abuf);
    for (int i = 0; i < p.L; ++i) ab[abase + (size_t)i * p.P] = i < count ? kb[i * 32 + lane] : kEmpty64;
    if (pay) {
      // payload block after the keys of every sample: [sample][layer][pixel] float4
      float4* pb = reinterpret_cast<float4*>(ab + (size_t)p.ssn * p.L * p.P);
      for (int i = 0; i < count; ++i) pb[abase + (size_t)i * p.P] = pay[i * 32 + lane];
    }
  }
};

// oitLoop.frag.glsl:57-100 (DEPTH) and 120-173 (COLOR). The shader's two passes
// leave the OIT_LAYERS smallest distinct depths, with each the colour of its last
// fragment, and blend every farther fragment into the target, in order. Here
// pass 0 keeps depths and colours together; only a warp of which a pixel has
// dropped a fragment, and only with tail blending, walks the list again (pass 1)
// to blend what lies behind the kept depths. Loop32 1001x563 4x sample shading
// takes 260 us (327 with two walks of every list), dense scenes of 2000 spheres
// 342 us without tail blending (442) and 467 us with it (448): nearly every warp
// walks twice there, and shades some fragments twice.
template <int S>
struct LoopPolicy {
  static constexpr bool kNodes = false;
  static constexpr bool kDirect = false;
  static constexpr bool kPack = true;
  static constexpr int kPasses = 2;
  // the most resident warps per SM it is compiled for (32: 64 registers)
  static constexpr int kWarpsPerSM = 32;
  static constexpr bool kViewZ = false;
  static __host__ __device__ size_t smem_bytes_per_warp(int L, int, int = 0) { return (size_t)L * 32 * 8; }
  static __host__ __device__ int payload_bytes(int tail, int, int) { return tail ? 20 : 4; }
  uint32_t* dep;
  uint32_t* col;
  int lane, count;
  bool dropped;
  size_t abase;  // viewSize * OIT_LAYERS * 2 * sampleID + pixel (oitLoop.frag.glsl:231)
  __device__ void init(const RasterParams& p, void* smem, int, int sample, uint32_t pixel) {
    lane = threadIdx.x & 31;
    count = 0;
    dropped = false;
    abase = (size_t)sample * 2 * p.L * p.P + pixel;
    dep = reinterpret_cast<uint32_t*>(smem);
    col = dep + p.L * 32;
    dep[(p.L - 1) * 32 + lane] = 0xFFFFFFFFu;  // (not full)
  }
  // Is a fragment of owner lane `owner` to be shaded in this pass? Behind the
  // last depth of a full buffer it will not be kept, whatever follows, and only
  // pass 1 blends it.
  __device__ __forceinline__ bool wanted(const RasterParams& p, int pass, uint32_t z, int owner) const {
    return (dep[(p.L - 1) * 32 + owner] < z) == (pass != 0);
  }
  // Is pass 1 wanted? Warp-uniform.
  __device__ __forceinline__ bool again(const RasterParams& p) const {
    return p.tail && __any_sync(kFull, dropped);
  }
  static __device__ __forceinline__ void produce(const RasterParams&, int pass, const FragPay& q, int j, const Frag& f,
                                                 const Shade& sh, float alpha) {
    if (pass == 0) q.packed[j] = f.packed;
    else q.rgba[j] = make_float4(sh.r, sh.g, sh.b, alpha);
  }
  __device__ __forceinline__ void fragment(const RasterParams& p, int pass, const Frag& f, const FragPay& q, int j,
                                           PixelTargets<S>& tg) {
    const int L = p.L;
    const uint32_t z = f.depth;
    if (pass != 0) {
      tg.tail(premult(q.rgba[j]), f.cover);
      return;
    }
    int at = count;  // the fragment's place
    while (at > 0) {
      const uint32_t d = dep[(at - 1) * 32 + lane];
      if (d == z) {
        col[(at - 1) * 32 + lane] = f.packed;
        return;
      }
      if (d < z) break;
      --at;
    }
    if (count == L) {
      dropped = true;
      if (at == L) return;
    } else {
      ++count;
    }
    for (int i = count - 1; i > at; --i) {
      dep[i * 32 + lane] = dep[(i - 1) * 32 + lane];
      col[i * 32 + lane] = col[(i - 1) * 32 + lane];
    }
    dep[at * 32 + lane] = z;
    col[at * 32 + lane] = f.packed;
  }
  __device__ void flush(const RasterParams& p, bool valid) {
    if (!valid) return;
    for (int i = 0; i < p.L; ++i) {
      p.abuf[abase + (size_t)i * p.P] = i < count ? dep[i * 32 + lane] : 0xFFFFFFFFu;
      p.abuf[abase + (size_t)(p.L + i) * p.P] = i < count ? col[i * 32 + lane] : 0u;
    }
  }
};

// oitSpinlock.frag.glsl:49-129 / oitInterlock.frag.glsl:90-152. The pixel's
// owner lane is its critical section: no lock is needed because no other
// thread ever touches the pixel, and fragments arrive in primitive order.
template <int S>
struct LockPolicy {
  static constexpr bool kNodes = false;
  static constexpr bool kDirect = false;
  static constexpr bool kPack = true;
  static constexpr int kPasses = 1;
  // the most resident warps per SM it is compiled for (36: 56 registers)
  static constexpr int kWarpsPerSM = 36;
  static constexpr bool kViewZ = false;
  // depths, then colours (and coverage) of the k-buffer, [layer][lane]
  static constexpr bool kCover = S > 1;  // several samples a lane: coverage records
  static __host__ __device__ size_t smem_bytes_per_warp(int L, int, int = 0) {
    return (size_t)L * 32 * (kCover ? 12 : 8);
  }
  static __host__ __device__ int payload_bytes(int tail, int, int) { return tail ? 20 : 4; }
  uint32_t count, auxdepth;
  // the furthest record of a full k-buffer, searched again once it is replaced
  uint32_t maxDepth;
  int furthest;
  uint32_t* dep;
  uint32_t eaux;
  size_t abase;
  __device__ void init(const RasterParams& p, void* smem, int, int sample, uint32_t pixel) {
    dep = reinterpret_cast<uint32_t*>(smem) + (threadIdx.x & 31);
    eaux = (uint32_t)sample * p.P + pixel;
    abase = (size_t)sample * p.L * p.P + pixel;
    count = 0;
    auxdepth = 0xFFFFFFFFu;
    furthest = -1;
    maxDepth = 0;
  }
  // record i's colour, and with coverage records its coverage after it
  __device__ __forceinline__ uint32_t* colour(int L, int i) const {
    return dep + 32 * (L + i) + (kCover ? (int)(threadIdx.x & 31) + 32 * i : 0);
  }
  static __device__ __forceinline__ void produce(const RasterParams& p, int, const FragPay& q, int j, const Frag& f,
                                                 const Shade& sh, float alpha) {
    q.packed[j] = f.packed;
    if (p.tail) q.rgba[j] = make_float4(sh.r, sh.g, sh.b, alpha);
  }
  __device__ __forceinline__ void store(int L, int i, const Frag& f) const {
    dep[32 * i] = f.depth;
    if constexpr (kCover) *reinterpret_cast<uint2*>(colour(L, i)) = make_uint2(f.packed, f.cover);
    else *colour(L, i) = f.packed;
  }
  __device__ __forceinline__ void fragment(const RasterParams& p, int, const Frag& f, const FragPay& q, int j,
                                           PixelTargets<S>& tg) {
    const int L = p.L;
    uint32_t evicted = 0u;  // the packed colour of the record the fragment replaces
    bool own = true;        // the fragment's own colour goes to the tail
    if (f.depth <= auxdepth) {
      const uint32_t old = count++;
      if (old < (uint32_t)L) {
        store(L, (int)old, f);
        return;  // (a blend of nothing)
      }
      if (furthest < 0) {
        furthest = 0;
        maxDepth = 0;
        for (int i = 0; i < L; ++i) {
          const uint32_t d = dep[32 * i];
          if (d > maxDepth) {
            maxDepth = d;
            furthest = i;
          }
        }
      }
      if (maxDepth > f.depth) {
        evicted = *colour(L, furthest);
        own = false;
        store(L, furthest, f);
        auxdepth = maxDepth;
        furthest = -1;
      }
    }
    if (p.tail) tg.tail(own ? premult(q.rgba[j]) : decode_premult(evicted), f.cover);
  }
  __device__ void flush(const RasterParams& p, bool valid) {
    if (!valid) return;
    p.aux[eaux] = count;
    p.auxdepth[eaux] = auxdepth;
    const int n = count < (uint32_t)p.L ? (int)count : p.L;
    for (int i = 0; i < n; ++i) {
      const uint32_t* c = colour(p.L, i);
      const size_t o = abase + (size_t)i * p.P;
      if constexpr (kCover) reinterpret_cast<uint4*>(p.abuf)[o] = make_uint4(c[0], dep[32 * i], c[1], 0u);
      else reinterpret_cast<uint2*>(p.abuf)[o] = make_uint2(c[0], dep[32 * i]);
    }
  }
};

// oitWeighted.frag.glsl:53-79 with the blend state of main.cpp:559-577.
// FP16 mode rounds the accumulators to half after every blend, as an
// RGBA16F/R16F render target does. The shading lane computes a fragment's
// weighted colour; the owner lane only accumulates.
template <int S>
struct WeightedPolicy {
  static constexpr bool kNodes = false;
  static constexpr bool kDirect = false;
  static constexpr bool kPack = false;
  static constexpr int kPasses = 1;
  // the most resident warps per SM it is compiled for (36: 56 registers)
  static constexpr int kWarpsPerSM = 36;
  static constexpr bool kViewZ = true;
  static __host__ __device__ size_t smem_bytes_per_warp(int, int, int = 0) { return 0; }
  static __host__ __device__ int payload_bytes(int, int, int weighted_fp32) { return weighted_fp32 ? 20 : 16; }
  // FP16: acc.x and acc.y hold four halves
  float4 acc[S];
  float rev[S];
  uint32_t px_;
  __device__ void init(const RasterParams&, void*, int, int, uint32_t pixel) {
    px_ = pixel;
#pragma unroll
    for (int s = 0; s < S; ++s) {
      acc[s] = make_float4(0.f, 0.f, 0.f, 0.f);
      rev[s] = 1.0f;
    }
  }
  static __device__ __forceinline__ float h(float x) { return __half2float(__float2half_rn(x)); }
  static __device__ __forceinline__ float pair(__half2 v) { return __uint_as_float(*reinterpret_cast<uint32_t*>(&v)); }
  // half accumulators: adding two halves in half precision rounds like adding
  // them in float and rounding the sum to half (24 >= 2 * 11 + 2 bits)
  static __device__ __forceinline__ void add(float& acc, float src) {
    const uint32_t a = __float_as_uint(acc), b = __float_as_uint(src);
    acc = pair(__hadd2_rn(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b)));
  }
  // FP32: the weighted colour, and 1 - alpha in the packed word; FP16: four
  // halves of weighted colour, then 1 - half(alpha).
  static __device__ __forceinline__ void produce(const RasterParams& p, int, const FragPay& q, int j, const Frag&,
                                                 const Shade& sh, float alpha) {
    const float4 c = premult(sh.r, sh.g, sh.b, alpha);
    const float depthZ = -sh.view_z * 10.0f;
    const float x = depthZ / 200.0f;
    const float x2 = x * x;
    float distWeight = 0.03f / (1e-5f + x2 * x2);
    distWeight = fminf(fmaxf(distWeight, 1e-2f), 3e3f);
    float aw = fminf(1.0f, fmaxf(fmaxf(c.x, c.y), fmaxf(c.z, c.w)) * 40.0f + 0.01f);
    aw *= aw;
    const float w = aw * distWeight;
    if (p.weighted_fp32) {
      q.rgba[j] = make_float4(c.x * w, c.y * w, c.z * w, c.w * w);
      q.packed[j] = __float_as_uint(1.0f - c.w);
    } else {
      q.rgba[j] = make_float4(pair(__floats2half2_rn(c.x * w, c.y * w)), pair(__floats2half2_rn(c.z * w, c.w * w)),
                              1.0f - h(c.w), 0.0f);
    }
  }
  __device__ __forceinline__ void fragment(const RasterParams& p, int, const Frag& f, const FragPay& q, int j,
                                           PixelTargets<S>&) {
    const float4 c = q.rgba[j];
#pragma unroll
    for (int s = 0; s < S; ++s) {
      if (!(f.cover & (1u << s))) continue;
      if (!p.weighted_fp32) {
        add(acc[s].x, c.x);
        add(acc[s].y, c.y);
        rev[s] = h(rev[s] * c.z);
      } else {
        acc[s].x += c.x;
        acc[s].y += c.y;
        acc[s].z += c.z;
        acc[s].w += c.w;
        rev[s] *= __uint_as_float(f.packed);
      }
    }
  }
  __device__ void flush(const RasterParams& p, bool valid) {
    if (!valid) return;
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const size_t o = (size_t)s * p.P + px_;
      if (p.weighted_fp32) {
        reinterpret_cast<float4*>(p.accum)[o] = acc[s];
        reinterpret_cast<float*>(p.reveal)[o] = rev[s];
      } else {
        reinterpret_cast<uint2*>(p.accum)[o] = make_uint2(__float_as_uint(acc[s].x), __float_as_uint(acc[s].y));
        reinterpret_cast<__half*>(p.reveal)[o] = __float2half_rn(rev[s]);
      }
    }
  }
};

// ---------------------------------------------------------------------------
// Triangle-list walk shared by the transparent and opaque kernels.
// ---------------------------------------------------------------------------
// A warp's piece of a 16x16 tile. Without sample shading (SSN = 1) a warp
// owns an 8x4 micro-tile, one lane per pixel, and 8 warps cover the tile.
// With sample shading every sample has its own A-buffer, so a lane owns one
// sample: a warp covers 4x2 pixels x 4 samples or 2x2 pixels x 8 samples and
// 8 * SSN warps cover the tile.
struct WarpTile {
  int lane, px, py, rx0, ry0, rx1, ry1;
  int tile;
  int mt;      // the 8x4 micro-tile of the tile that holds the warp's pixels
  int sample;  // the lane's sample with sample shading, else 0
  bool valid;
  uint32_t pixel;
};

template <int SSN>
struct LaneMap {
  static constexpr int kPix = 32 / SSN;                  // pixels per warp
  static constexpr int kW = SSN == 1 ? 8 : (SSN == 4 ? 4 : 2);
  static constexpr int kH = kPix / kW;
  __device__ static int pix(int lane) { return lane % kPix; }
  __device__ static int sample(int lane) { return lane / kPix; }
};

// The pass's tile number q: q itself, or with the tiles in buckets by list
// length, taken in turn from the longest and from the shortest lists. A small
// frame is resident as a whole but for its last tiles, and then waits for the
// tile with the longest list; between them the short lists' tiles write their
// (empty) A-buffers, which all at the end would be bound by memory. Measured in
// tile order, longest first, in turn: Simple 1283x717 4x MSAA 382 / 344 / 346
// us, Spinlock 800x512 253 / 236 / 242, linked list 1280x720 251 / 244 / 237,
// Loop32 1001x563 4x sample shading 362 / 378 / 363; but WBOIT 3840x2160 3.25 /
// 3.25 / 3.37 ms and Loop64 1920x1080 346 / 360 / 354 us: neighbouring tiles
// read the same records, so larger frames keep the tile order. Warp-uniform.
__device__ __forceinline__ int ordered_tile(const RasterParams& p, int q, int lane) {
  if (!p.tile_order) return q;
  constexpr int B = oit::kOrderBuckets;
  q = (q & 1) ? p.tiles_x * p.tiles_y - 1 - (q >> 1) : q >> 1;
  const int bucket = B - 1 - lane;  // lane 0: the longest lists
  const uint32_t c = lane < B ? p.order_count[bucket] : 0u;
  uint32_t incl = c;
#pragma unroll
  for (int o = 1; o < B; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  const int at = __ffs((int)__ballot_sync(kFull, lane < B && (uint32_t)q < incl)) - 1;
  const uint32_t before = __shfl_sync(kFull, incl - c, at);
  return (int)p.tile_order[(size_t)(B - 1 - at) * (size_t)(p.tiles_x * p.tiles_y) + ((uint32_t)q - before)];
}

// cta: the CTA's index within its view's grid.
template <int SSN>
__device__ __forceinline__ WarpTile warp_tile(const RasterParams& p, int cta) {
  using M = LaneMap<SSN>;
  WarpTile w;
  const int warp = threadIdx.x >> 5;
  w.lane = threadIdx.x & 31;
  const int gw = cta * (int)(blockDim.x >> 5) + warp;   // warp within the pass
  const int tile = ordered_tile(p, gw / (oit::kWarpsPerTile * SSN), w.lane);
  const int part = gw % (oit::kWarpsPerTile * SSN);     // the warp's part of the tile
  const int tx = tile % p.tiles_x, ty = tile / p.tiles_x;
  const int lx = (part % (16 / M::kW)) * M::kW, ly = (part / (16 / M::kW)) * M::kH;
  w.tile = tile;
  w.mt = 2 * (ly >> 2) + (lx >> 3);
  w.rx0 = tx * 16 + lx;
  w.ry0 = ty * 16 + ly;
  w.rx1 = w.rx0 + M::kW - 1;
  w.ry1 = w.ry0 + M::kH - 1;
  const int pix = M::pix(w.lane);
  w.sample = M::sample(w.lane);
  w.px = w.rx0 + pix % M::kW;
  w.py = w.ry0 + pix / M::kW;
  w.valid = w.px < p.RW && w.py < p.RH;
  w.pixel = w.valid ? (uint32_t)w.py * (uint32_t)p.RW + (uint32_t)w.px : 0u;
  return w;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

__device__ __forceinline__ bool bbox_hits(uint2 bb, const WarpTile& w) {
  const int bx0 = bb.x & 0xFFFF, by0 = bb.x >> 16, bx1 = bb.y & 0xFFFF, by1 = (bb.y >> 16) & 0x7FFF;
  return !(bx1 < w.rx0 || bx0 > w.rx1 || by1 < w.ry0 || by0 > w.ry1);
}

// Hits a warp processes at once, the list entries its walk tests at a time,
// and the ring it collects hits in (at most kHits - 1 left over and kScan new
// ones).
constexpr int kHits = 32;
constexpr int kScan = 64;
constexpr int kRing = 128;

// Walks [beg, end) of the tile list in primitive order, kScan entries at a time,
// and collects the triangles whose bbox touches the warp's pixels in `ring`;
// chunk(head, nh, last) then processes ring entries head .. head + nh - 1
// (modulo kRing), kHits of them until the list ends, and once more with nh = 0
// and last = true. A tile's list has a handful of hits per 32 entries (8
// micro-tiles, triangles of a few pixels), so collecting them first fills the
// lanes of every later step. chunk is warp-uniform.
// The test is the 8x4 micro-tile's bit in the pair's sorted key (those that the
// bbox overlaps, or that the setup found covered); a warp with fewer pixels than
// that (Fine) also tests the bbox. List entries of triangles >= limit are
// skipped (the second half of a near-clipped triangle t, record num_tris + t,
// counts as triangle t). With `ident` (an overflowed draw's unbinned
// triangles) entry i of [beg, end) is half i & 1 of triangle i >> 1, tested by
// its bbox (a second half only when the first's bbox says it exists).
template <bool Fine, class Chunk>
__device__ __forceinline__ void walk_list(const RasterParams& p, const WarpTile& w, uint32_t* ring, uint32_t beg,
                                          uint32_t end, bool ident, uint32_t limit, Chunk&& chunk) {
  const uint32_t lt = (1u << w.lane) - 1u;
  const uint32_t mbit = 1u << (oit::kMaskShift + w.mt);
  const bool test = Fine || ident || limit != 0xFFFFFFFFu;
  // the lane's entries of the block at pos, fetched while the one before it is
  // tested: a block's loads take an L2 round trip whatever its size
  constexpr int kPer = kScan / 32;
  uint32_t key[kPer], t[kPer];
  auto fetch = [&](uint32_t pos) {
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const uint32_t i = pos + 32u * u + w.lane;
      key[u] = 0;
      if (i >= end) continue;
      if (ident) {
        key[u] = mbit;
        t[u] = (i & 1u) ? p.num_tris + (i >> 1) : (i >> 1);
      } else {
        key[u] = p.tile_keys[i];
        t[u] = p.tile_tris[i];
      }
    }
  };
  uint32_t pos = beg, head = 0, cnt = 0;
  fetch(pos);
#pragma unroll 1
  for (;;) {
#pragma unroll 1
    while (cnt < kHits && pos < end) {
      bool hit[kPer];
      uint32_t tc[kPer];
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        hit[u] = (key[u] & mbit) != 0u;
        tc[u] = t[u];
      }
      const uint32_t at = pos;
      pos += kScan;
      fetch(pos);
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        if (test && hit[u]) {
          const uint32_t i = at + 32u * u + w.lane;
          if (ident && (i & 1u) && !(p.bbox[i >> 1].y >> 31)) hit[u] = false;
          else if (Fine || ident) hit[u] = bbox_hits(p.bbox[tc[u]], w);
          if ((tc[u] >= p.num_tris ? tc[u] - p.num_tris : tc[u]) >= limit) hit[u] = false;
        }
        const uint32_t m = __ballot_sync(kFull, hit[u]);
        if (hit[u]) ring[(head + cnt + __popc(m & lt)) % kRing] = tc[u];
        cnt += __popc(m);
      }
    }
    const int nh = (int)min(cnt, (uint32_t)kHits);
    __syncwarp();
    chunk(head, nh, nh == 0);
    __syncwarp();
    if (nh == 0) break;
    head += (uint32_t)nh;
    cnt -= (uint32_t)nh;
  }
}

// Triangles of the draw binned whole: all of them, or after a bin overflow
// those before the first triangle whose pairs reach past the capacity (pairs
// are emitted in triangle order). Warp-uniform.
__device__ __forceinline__ uint32_t binned_triangles(const RasterParams& p) {
  if (!p.pair_total || *p.pair_total <= p.pair_capacity) return 0xFFFFFFFFu;
  uint32_t lo = 0, hi = p.num_tris;  // first t with pair_offset[t] + pair_count[t] > capacity
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (p.pair_offset[mid] + p.pair_count[mid] > p.pair_capacity) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// The pass's walk: the tile list (triangles binned whole), then, after a bin
// overflow, the unbinned triangles of the pass by bbox; primitive order is
// kept because every binned triangle precedes every unbinned one.
template <bool Fine, class Chunk>
__device__ __forceinline__ void walk_pass(const RasterParams& p, const WarpTile& w, uint32_t* ring, uint32_t beg,
                                          uint32_t end, Chunk&& chunk) {
  const uint32_t cut = binned_triangles(p);
  const bool rest = cut < p.pass_end;
  const uint32_t nph = rest ? 2u : 1u;
#pragma unroll 1
  for (uint32_t ph = 0; ph < nph; ++ph) {
    const bool ident = ph == 1;
    walk_list<Fine>(p, w, ring, ident ? 2u * max(cut, p.pass_first) : beg, ident ? 2u * p.pass_end : end, ident,
                    ident ? 0xFFFFFFFFu : cut, chunk);
  }
}

// ---------------------------------------------------------------------------
// Transparent COLOR (+DEPTH) pass.
// ---------------------------------------------------------------------------
// Per warp in shared memory:
//  rec   the setup records of the hits being processed; xy01 and xy2f of small
//        triangles (kFlagSmall) are replaced by their edge equations at the
//        warp's first pixel: {E0, E1, sum, alpha} and {dE0/dx, dE0/dy, dE1/dx,
//        dE1/dy} per pixel, where E = 2 e + top_left - 1 for the edge value e
//        (so a sample is inside when no E is negative, and e = (E + 1) >> 1)
//        and E2 = sum - E0 - E1 (the edge values add up to twice the area);
//  hit   the hits that cover a pixel: number of the first covered one (bits
//        0-10), record (bits 11-15), alpha code (bits 16-23), bit 31: not
//        small; and the covered pixels, one bit per owner lane;
//  ent   queued fragments: depth, and with several samples a lane the hit (bits
//        0-4), owner lane (bits 8-12) and coverage (bits 16-23);
//  mine  per 32 queued fragments and lane: the fragments of the lane's pixel;
//  ring  triangles collected by the walk;
//  then the policy's payload per queued fragment.
//  persp WBOIT: the hits' perspective terms. Read from memory per fragment they
//        were another round trip before it could be shaded: 3840x2160 3.03 ->
//        2.91 ms, 641x359 86 -> 79 us without it.
template <bool Samples>
struct QueueEntry {
  uint32_t depth;
};
template <>
struct QueueEntry<true> {
  uint32_t depth, info;
};
template <bool Samples, bool ViewZ>
struct WarpStage {
  static constexpr int kQueue = kQueueOf<Samples>;
  TriSetup rec[kHits];
  uint2 hit[kHits];
  TriPersp persp[ViewZ ? kHits : 1];
  QueueEntry<Samples> ent[Samples || !ViewZ ? kQueue : 4];  // (WBOIT needs no depths)
  uint32_t mine[kQueue / 32][32];
  uint32_t ring[kRing];
};
template <int S, bool ViewZ>
__host__ __device__ constexpr size_t warp_stage_bytes(int payload) {
  return sizeof(WarpStage<(S > 1), ViewZ>) + (size_t)kQueueOf<(S > 1)> * payload;
}

// Position of set bit n (0 = the lowest) of m; n < popc(m).
__device__ __forceinline__ int nth_bit(uint32_t m, uint32_t n) {
  int pos = 0;
#pragma unroll
  for (int w = 16; w >= 1; w >>= 1) {
    const uint32_t c = (uint32_t)__popc(m & ((1u << w) - 1u));
    if (n >= c) {
      n -= c;
      m >>= w;
      pos += w;
    }
  }
  return pos;
}

// Sample s of SSN in 1/256 pixel, s a run-time value.
template <int SSN>
__device__ __forceinline__ int2 sample_pos_at(int s) {
  const uint32_t x = SSN == 4 ? 0xA2E6u : 0xFB135D79u, y = SSN == 4 ? 0xEA62u : 0x1F7D39B5u;
  return make_int2((int)((x >> (4 * s)) & 15u) << 4, (int)((y >> (4 * s)) & 15u) << 4);
}

// Could a point of the rectangle (x0, y0) .. (x1, y1), in 1/256 pixel, be inside a
// large triangle (a, b: TriSetup's xy01 and xy2f)? Not if it lies outside an edge.
__device__ __forceinline__ bool large_meets(const int4& a, const int4& b, int x0, int y0, int x1, int y1) {
  const Edges e = edges_at<long long>(a, b, x0, y0);
  // the edge's largest value: its value at the first corner and what it gains across
  auto most = [&](long long v, int dx, int dy) {
    return v + (long long)max(-dy, 0) * (x1 - x0) + (long long)max(dx, 0) * (y1 - y0);
  };
  return (most(e.e0, b.x - a.z, b.y - a.w) | most(e.e1, a.x - b.x, a.y - b.y) | most(e.e2, a.z - a.x, a.w - a.y)) >= 0;
}

// The owner lanes (bits) of the warp's pixels in a bbox.
template <int SSN>
__device__ __forceinline__ uint32_t bbox_lanes(const WarpTile& w, int bx0, int by0, int bx1, int by1) {
  using M = LaneMap<SSN>;
  const int x0 = max(bx0 - w.rx0, 0), x1 = min(bx1 - w.rx0, M::kW - 1);
  const int y0 = max(by0 - w.ry0, 0), y1 = min(by1 - w.ry0, M::kH - 1);
  uint32_t m = 0;
#pragma unroll
  for (int y = 0; y < M::kH; ++y)
    if (y >= y0 && y <= y1 && x0 <= x1) m |= ((2u << x1) - (1u << x0)) << (y * M::kW);
  uint32_t all = m;
#pragma unroll
  for (int i = 1; i < SSN; ++i) all |= m << (i * M::kPix);
  return all;
}

// Stages ring entries head .. head + nh - 1 in rec, one lane per hit, and finds
// the pixels each covers, 32 sign tests a lane (with several samples a lane,
// or a large triangle: the pixels it may cover), for `hit`. Returns the number
// of the hit's first pixel, and the number of pixels of all hits. `lanes`: the
// owner lanes whose pixel exists. Normals: the records' normals and colours
// are wanted too.
template <int S, int SSN, bool Normals>
__device__ __forceinline__ int stage_hits(const WarpTile& w, const TriSetup* setup, const uint32_t* ring,
                                          TriSetup* rec, uint2* hit, uint32_t lanes, uint32_t head, int nh,
                                          int& total) {
  using M = LaneMap<SSN>;
  constexpr bool kCentre = S == 1 && SSN == 1;
  const uint32_t lt = (1u << w.lane) - 1u;
  uint32_t cover = 0, info = 0;
  if (w.lane < nh) {
    const TriSetup* src = setup + ring[(head + w.lane) % kRing];
    TriSetup& dst = rec[w.lane];
    cp_async16(&dst.zc, &src->zc);
    if (Normals) {
      cp_async16(&dst.n0, &src->n0);
      cp_async16(&dst.n1, &src->n1);
      cp_async16(&dst.n2, &src->n2);
    }
    const int4 a = src->xy01, b = src->xy2f;
    const int X0 = a.x, Y0 = a.y, X1 = a.z, Y1 = a.w, X2 = b.x, Y2 = b.y;
    const uint32_t flags = (uint32_t)b.z;
    info = ((uint32_t)w.lane << 11) | ((flags << 8) & 0xFF0000u);
    if (flags & kFlagSmall) {
      const int t0 = (int)(flags & 1u), t1 = (int)((flags >> 1) & 1u), t2 = (int)((flags >> 2) & 1u);
      const int A0 = (Y1 - Y2) * 512, B0 = (X2 - X1) * 512, A1 = (Y2 - Y0) * 512, B1 = (X0 - X2) * 512;
      const int ox = w.rx0 * 256 + (kCentre ? 128 : 0), oy = w.ry0 * 256 + (kCentre ? 128 : 0);
      const int E0 = 2 * ((X2 - X1) * (oy - Y1) + (Y1 - Y2) * (ox - X1)) + t0 - 1;
      const int E1 = 2 * ((X0 - X2) * (oy - Y2) + (Y2 - Y0) * (ox - X2)) + t1 - 1;
      const int sum = 2 * ((X1 - X0) * (Y2 - Y0) - (Y1 - Y0) * (X2 - X0)) + t0 + t1 + t2 - 3;
      dst.xy01 = make_int4(E0, E1, sum, b.w);
      dst.xy2f = make_int4(A0, B0, A1, B1);
      // from the last lane to the first, so that each sign shifts in below the ones before it
      uint32_t out = 0;
      if (S == 1) {
#pragma unroll
        for (int smp = SSN - 1; smp >= 0; --smp) {
          int s0 = E0, s1 = E1;
          if (!kCentre) {
            const int2 sp = sample_pos<SSN>(smp);
            s0 += (A0 >> 8) * sp.x + (B0 >> 8) * sp.y;
            s1 += (A1 >> 8) * sp.x + (B1 >> 8) * sp.y;
          }
#pragma unroll
          for (int y = M::kH - 1; y >= 0; --y)
#pragma unroll
            for (int x = M::kW - 1; x >= 0; --x) {
              const int e0 = s0 + A0 * x + B0 * y, e1 = s1 + A1 * x + B1 * y;
              out = __funnelshift_l((uint32_t)(e0 | e1 | (sum - e0 - e1)), out, 1);
            }
        }
      } else {
        // the largest value over the pixel's samples (all of them within 16 .. 240)
        const int A2 = -(A0 + A1), B2 = -(B0 + B1);
        auto most = [](int A, int B) {
          return (max(A, 0) >> 8) * 240 + (min(A, 0) >> 8) * 16 + (max(B, 0) >> 8) * 240 + (min(B, 0) >> 8) * 16;
        };
        const int s0 = E0 + most(A0, B0), s1 = E1 + most(A1, B1), s2 = sum - E0 - E1 + most(A2, B2);
#pragma unroll
        for (int y = M::kH - 1; y >= 0; --y)
#pragma unroll
          for (int x = M::kW - 1; x >= 0; --x) {
            const int e0 = s0 + A0 * x + B0 * y, e1 = s1 + A1 * x + B1 * y, e2 = s2 + A2 * x + B2 * y;
            out = __funnelshift_l((uint32_t)(e0 | e1 | e2), out, 1);
          }
      }
      cover = ~out & lanes;
    } else {
      info |= 0x80000000u;
      dst.xy01 = a;
      dst.xy2f = b;
      // With several samples a lane, and in the opaque pass, each of the warp's
      // pixels in the bbox costs a lane of a group its samples' 64-bit tests, so
      // micro-tiles outside the triangle are dropped first: panes over most of
      // 1280x720, 231 us without and 125 with it for the opaque pass of 60 at 8x,
      // 238 and 157 us for 25 in linked lists at 8x.
      constexpr int kFirst = kCentre ? 128 : 16, kLast = kCentre ? 128 : 240;  // of a pixel's samples
      const int x0 = w.rx0 * 256, y0 = w.ry0 * 256;
      if ((S == 1 && Normals) || large_meets(a, b, x0 + kFirst, y0 + kFirst, x0 + 256 * (M::kW - 1) + kLast,
                                             y0 + 256 * (M::kH - 1) + kLast))
        cover = bbox_lanes<SSN>(w, min(X0, min(X1, X2)) >> 8, min(Y0, min(Y1, Y2)) >> 8, max(X0, max(X1, X2)) >> 8,
                                max(Y0, max(Y1, Y2)) >> 8) & lanes;
    }
  }
  const int n = __popc(cover);
  int incl = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, incl, o);
    if (w.lane >= o) incl += y;
  }
  total = __shfl_sync(kFull, incl, 31);
  const uint32_t some = __ballot_sync(kFull, n > 0);
  if (n > 0) hit[__popc(some & lt)] = make_uint2(info | (uint32_t)(incl - n), cover);
  cp_async_wait_all();
  __syncwarp();
  return n > 0 ? incl - n : 0x40000000;
}

// S: samples each lane evaluates (MSAA coverage); SSN: samples mapped to
// lanes (sample shading, S = 1 then).
// The pass is bound by instruction issue (77-82% issue-active at 1920x1080 with
// 4096 spheres, WBOIT), so the work is laid out to fill a warp's lanes at each
// step: 32 hits are prepared at once, each finding the pixels it covers by 32
// sign tests of five integer operations (a triangle of 6 pixels has a bbox of
// 26, so testing (hit, bbox pixel) pairs one per lane is four to six tests per
// fragment, each with the finding of its hit and pixel around it), and 32
// fragments are shaded at once; what a fragment's algorithm computes from the
// fragment alone (its weight, its record, its list node) is done by the lane
// that shaded it. Whole frames when that was measured, with covered pixels / with
// bbox pairs / with hits taken per 32 list entries and the edge functions
// evaluated from the vertices: WBOIT 3840x2160, 16384 spheres 3.32 / 4.60 / 6.84
// ms; Interlock 2560x1440 8x MSAA 3.63 / 4.31 / 6.30 ms; Loop32 1001x563 4x sample
// shading 391 / 522 / 738 us; Spinlock 800x512 288 / 327 / 420 us; linked list
// 640x480 137 / 156 / 215 us; 24-view batch 4.31 / 4.78 / 6.18 ms.
// Triangles wider than 64 pixels (64-bit edges) are tested pixel by pixel.
// The warps of a tile work independently (each walks the tile's list for its
// own micro-tile), so a CTA holds kRasterWarpsPerBlock of them: a CTA's
// resources are released when its slowest warp is done, and micro-tiles of
// one tile differ in work (2 warps per CTA: the 64-view batch 5.6% faster
// than 8; Loop64 k-buffers at large OIT_LAYERS pack shared memory better).
using oit::kRasterWarpsPerBlock;
// Registers: a spilled value comes back from L2 more often than not, since the
// warps' stages leave L1 a tenth of the SM's memory. At 64 registers (32 warps
// per SM) nothing or nearly nothing spills, at 56 (36 warps) 16-40 bytes do:
// Loop64 1920x1080 324 -> 300 us, Spinlock 800x512 186 -> 173 us, a mostly empty
// Spinlock 1577x1183 2x2 supersampled frame 366 -> 241 us, WBOIT 3840x2160 the
// same. A batch's tuner may still take 36. MSAA lanes hold more
// (msaa_warps): at 24 warps with 8 samples Interlock 2560x1440 took 3.08 ms, at
// 20 2.83, at 16 3.02; at 24 with 4 samples Simple 1283x717 298 us, at 20 301.
template <template <int> class Policy, int S, int SSN>
__device__ __forceinline__ void raster_transparent_body(const RasterParams& p, int cta) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Pol = Policy<S>;
  using M = LaneMap<SSN>;
  constexpr bool kCentre = S == 1 && SSN == 1;  // the edge equations are taken at pixel centres (else at corners)
  constexpr int kQueue = kQueueOf<(S > 1)>;
  const int warp = threadIdx.x >> 5;
  const WarpTile w = warp_tile<SSN>(p, cta);
  const uint32_t elem = (uint32_t)w.sample * p.P + w.pixel;  // this lane's sample of the pixel
  const int payload = Pol::payload_bytes(p.tail, p.record_fp32, p.weighted_fp32);
  unsigned char* wbase = smem_raw + (size_t)warp * warp_stage_bytes<S, Pol::kViewZ>(payload);
  using Stage = WarpStage<(S > 1), Pol::kViewZ>;
  Stage& st = *reinterpret_cast<Stage*>(wbase);
  FragPay pay;
  pay.rgba = reinterpret_cast<float4*>(wbase + sizeof(Stage));
  pay.packed = reinterpret_cast<uint32_t*>(wbase + sizeof(Stage) + (payload >= 16 ? kQueue * 16 : 0));
  unsigned char* pol_smem = smem_raw + (size_t)(blockDim.x >> 5) * warp_stage_bytes<S, Pol::kViewZ>(payload) +
                            (size_t)warp * Pol::smem_bytes_per_warp(p.L, p.coverage, p.record_fp32);

  PixelTargets<S> tg;
#pragma unroll
  for (int s = 0; s < S; ++s)
    tg.col[s] = p.has_opaque && w.valid ? p.opaque_color[(size_t)(SSN > 1 ? w.sample : s) * p.P + w.pixel]
                                        : p.background;
  // this lane's opaque depth (1.0 without an opaque pass)
  const uint32_t depth = S == 1 && p.has_opaque && w.valid ? p.depth[elem] : 0x3F800000u;
  Pol pol;
  pol.init(p, pol_smem, w.lane, w.sample, w.pixel);
#pragma unroll
  for (int i = 0; i < kQueue / 32; ++i) st.mine[i][w.lane] = 0u;

  const int tile = w.tile + p.tile_offset;
  const uint32_t beg = p.tile_begin[tile], end = p.tile_end[tile];
  const TriSetup* setup = reinterpret_cast<const TriSetup*>(p.setup);
  const TriPersp* persp = reinterpret_cast<const TriPersp*>(p.persp);
  const uint32_t lt = (1u << w.lane) - 1u;
  // owner lanes whose pixel exists
  const uint32_t lanes = __ballot_sync(kFull, w.valid);
  uint32_t nfrag = 0;  // warp-uniform
  uint32_t got = 0;    // fragments delivered to this lane's pixel
  int qn = 0;          // warp-uniform: queued fragments

#pragma unroll 1
  for (int pass = 0; pass < Pol::kPasses; ++pass) {
    if constexpr (Pol::kPasses > 1) {
      if (pass > 0 && !pol.again(p)) break;
    }

    auto stage = [&](uint32_t head, int nh, int& total) {
      if (Pol::kViewZ && w.lane < nh) {  // (waited for with the records)
        const TriPersp* src = persp + st.ring[(head + w.lane) % kRing];
        cp_async16(&st.persp[w.lane].q, &src->q);
        cp_async16(&st.persp[w.lane].vzq, &src->vzq);
      }
      return stage_hits<S, SSN, true>(w, setup, st.ring, st.rec, st.hit, lanes, head, nh, total);
    };

    // Edge values of hit h, record T at owner lane `owner`'s shading point: its
    // pixel's centre, or its sample with sample shading. False when a large
    // triangle does not cover it.
    auto edges = [&](uint2 h, const TriSetup& T, int owner, float3& v, float& alpha) {
      const int4 a = T.xy01, b = T.xy2f;
      const int pl = M::pix(owner), dx = pl % M::kW, dy = pl / M::kW;
      const int2 sp = SSN > 1 ? sample_pos_at<SSN>(M::sample(owner)) : make_int2(128, 128);
      if (!(h.x >> 31)) {
        int e0 = a.x + b.x * dx + b.y * dy, e1 = a.y + b.z * dx + b.w * dy;
        if (!kCentre) {
          e0 += (b.x >> 8) * sp.x + (b.y >> 8) * sp.y;
          e1 += (b.z >> 8) * sp.x + (b.w >> 8) * sp.y;
        }
        const int e2 = a.z - e0 - e1;
        v = make_float3(to_float((e0 + 1) >> 1), to_float((e1 + 1) >> 1), to_float((e2 + 1) >> 1));
        alpha = __int_as_float(a.w);
        return true;
      }
      const Edges ed = edges_at<long long>(a, b, (w.rx0 + dx) * 256 + sp.x, (w.ry0 + dy) * 256 + sp.y);
      v = make_float3(to_float(ed.e0), to_float(ed.e1), to_float(ed.e2));
      alpha = __int_as_float(b.w);
      return inside(ed, b.z);
    };

    // Shading of record T from its edge values.
    auto shade_fragment = [&](uint2 h, const TriSetup& T, float3 v, Frag& f, Shade& sh) {
      const int k = (int)((h.x >> 11) & 31u);
      sh = shade_at(T, v.x, v.y, v.z, Pol::kViewZ ? &st.persp[k] : nullptr);
      f.packed = Pol::kPack ? pack_rgba8(sh, (h.x >> 16) & 255u) : 0u;
    };

    // Direct policies: every active lane holds a shaded fragment and writes its
    // own record. `lower`: the earlier ones of its pixel, `own`: this lane's
    // pixel's fragments (one bit per lane that holds one).
    auto write_direct = [&](bool act, uint32_t am, int owner, const Frag& f, const Shade& sh, float alpha,
                            uint32_t node0) {
      if (act) atomicOr(&st.mine[0][owner], 1u << w.lane);
      __syncwarp();
      const uint32_t lower = act ? st.mine[0][owner] & lt : 0u;
      const uint32_t own = st.mine[0][w.lane];
      __syncwarp();
      st.mine[0][w.lane] = 0u;
      if constexpr (Pol::kNodes) {
        node0 = __shfl_sync(kFull, node0, 0);
        const uint32_t before = __shfl_sync(kFull, pol.head, owner);
        const uint32_t node = node0 + (uint32_t)__popc(am & lt) + 1u;
        const bool stored = act && node < p.capacity;
        // the pixel's last earlier node: its lane's rank among the active ones
        auto node_of = [&](uint32_t lanes_of) {
          return node0 + (uint32_t)__popc(am & (0xFFFFFFFFu >> __clz(lanes_of)));
        };
        if (stored) Pol::write(p, node, lower ? node_of(lower) : before, f, sh, alpha);
        const uint32_t sm = __ballot_sync(kFull, stored);
        uint32_t tails = p.tail ? am & ~sm : 0u;
        while (tails) {  // a full pool: the fragments are tail blended one after the other
          const int j = __ffs(tails) - 1;
          tails &= tails - 1u;
          const float4 c = premult(__shfl_sync(kFull, sh.r, j), __shfl_sync(kFull, sh.g, j),
                                   __shfl_sync(kFull, sh.b, j), __shfl_sync(kFull, alpha, j));
          const uint32_t cover = __shfl_sync(kFull, f.cover, j);
          if (__shfl_sync(kFull, owner, j) == w.lane) tg.tail(c, cover);
        }
        if (own & sm) pol.head = node_of(own & sm);
      } else if constexpr (Pol::kDirect) {
        const uint32_t rank = __shfl_sync(kFull, pol.count, owner) + (uint32_t)__popc(lower);
        if (act) {
          if (rank < (uint32_t)p.L) {
            const int pl = M::pix(owner);
            Pol::write(p, rank, M::sample(owner),
                       (uint32_t)(w.ry0 + pl / M::kW) * (uint32_t)p.RW + (uint32_t)(w.rx0 + pl % M::kW), f);
          } else if (p.tail) {
            pay.rgba[w.lane] = premult(sh.r, sh.g, sh.b, alpha);
            pay.packed[w.lane] = f.cover;
          }
        }
        if (p.tail) {
          __syncwarp();
          uint32_t m = own;
          for (uint32_t k = pol.count; m && k < (uint32_t)p.L; ++k) m &= m - 1u;
          while (m) {
            const int j = __ffs(m) - 1;
            m &= m - 1u;
            tg.tail(pay.rgba[j], pay.packed[j]);
          }
        }
        pol.count += (uint32_t)__popc(own);
      }
      got += (uint32_t)__popc(own);
      nfrag += (uint32_t)__popc(am);
      __syncwarp();
    };

    // Two passes: the fragments that this one shades; pass 0 counts the others.
    auto select = [&](bool frag, uint32_t z, int owner) {
      bool want = frag;
      if constexpr (Pol::kPasses > 1) {
        want = frag && pol.wanted(p, pass, z, owner);
        if (pass == 0) {
          const uint32_t left = __ballot_sync(kFull, frag && !want);
          nfrag += (uint32_t)__popc(left);
          pol.dropped = pol.dropped || left != 0u;
        }
      }
      return want;
    };

    // Queued policies: hands every lane its pixel's fragments in queue order.
    auto feed = [&]() {
      __syncwarp();
      unsigned long long m = (unsigned long long)st.mine[0][w.lane] | ((unsigned long long)st.mine[1][w.lane] << 32);
      uint32_t rest = kQueue > 64 ? st.mine[kQueue / 32 - 1][w.lane] : 0u;  // the third word
#pragma unroll
      for (int i = 0; i < kQueue / 32; ++i) st.mine[i][w.lane] = 0u;
      if (pass == 0) {
        got += (uint32_t)(__popcll(m) + __popc(rest));
        nfrag += (uint32_t)qn;
      }
      int first = -1;
      while (true) {
        if (m == 0) {
          if (kQueue == 64 || rest == 0) break;
          m = rest;
          rest = 0;
          first = 63;
        }
        const int j = first + __ffsll((long long)m);
        m &= m - 1;
        const auto e = st.ent[Pol::kViewZ && S == 1 ? 0 : j];
        Frag f;
        f.depth = e.depth;
        f.cover = 1u;
        if constexpr (S > 1) f.cover = e.info >> 16;
        f.packed = Pol::kPack || p.weighted_fp32 ? pay.packed[j] : 0u;
        if constexpr (!Pol::kDirect) pol.fragment(p, pass, f, pay, j, tg);
      }
      qn = 0;
      __syncwarp();
    };

    walk_pass<(SSN > 1)>(p, w, st.ring, beg, end, [&](uint32_t head, int nh, bool last) {
      int total = 0;
      const int pre = stage(head, nh, total);
      // The covered pixels of all hits are numbered hit by hit; lane g of each
      // group of 32 takes number g, so fragments come in primitive order.
      int khi = -1;  // the last hit that starts before this group
      int qs = qn;   // queued fragments already shaded
#pragma unroll 1
      for (int base = 0; base < total || last; base += 32) {
        if (!last) {
          const uint32_t rel = (uint32_t)(pre - base);
          const uint32_t starts = __reduce_or_sync(kFull, rel < 32u ? 1u << rel : 0u);
          const int j = khi + __popc(starts & (lt | (1u << w.lane)));
          khi += __popc(starts);
          const bool act = base + w.lane < total;
          const uint2 h = st.hit[j];
          const int k = (int)((h.x >> 11) & 31u);
          const TriSetup& T = st.rec[k];
          const int owner = act ? nth_bit(h.y, (uint32_t)(base + w.lane) - (h.x & 0x7FFu)) : w.lane;
          if constexpr (S == 1) {
            const uint32_t od = __shfl_sync(kFull, depth, owner);
            Frag f;
            f.cover = 1u;
            float3 v;
            float alpha = 0.f;
            bool pass_z = act;
            if (act) {
              pass_z = edges(h, T, owner, v, alpha);
              f.depth = __float_as_uint(depth_from(T.zc, v.y, v.z));
              pass_z = pass_z && f.depth < od;
            }
            if constexpr (Pol::kPasses > 1) pass_z = select(pass_z, f.depth, owner);
            const uint32_t pm = __ballot_sync(kFull, pass_z);
            if (pm) {
              Shade sh;
              if constexpr (Pol::kDirect) {
                uint32_t node0 = 0;
                if (Pol::kNodes && w.lane == 0) node0 = atomicAdd(p.counter, (uint32_t)__popc(pm));
                if (pass_z) shade_fragment(h, T, v, f, sh);
                write_direct(pass_z, pm, owner, f, sh, alpha, node0);
              } else {
                if (pass_z) {
                  const int e = qn + __popc(pm & lt);
                  if (!Pol::kViewZ) st.ent[e].depth = f.depth;
                  atomicOr(&st.mine[e >> 5][owner], 1u << (e & 31));
                  shade_fragment(h, T, v, f, sh);
                  Pol::produce(p, pass, pay, e, f, sh, alpha);
                }
                qn += __popc(pm);
              }
            }
          } else {
            // coverage of the pixel's samples, then a queue of covered pixels
            uint32_t cover = 0;
            float zcen = 0.f;
            if (act) {
              const int4 a = T.xy01, b = T.xy2f;
              const float4 zc = T.zc;
              const int dx = owner % M::kW, dy = owner / M::kW;
              const uint32_t* odp = p.depth + (size_t)(w.ry0 + dy) * p.RW + (w.rx0 + dx);
              // opaque depth, from memory (in the owner lane it would take S registers)
              auto opaque_depth = [&](int s) { return p.has_opaque ? odp[(size_t)s * p.P] : 0x3F800000u; };
              // without an opaque pass, and with every vertex well in front of depth
              // 1, every covered sample passes: its depth lies between the vertices'
              const bool near = !p.has_opaque && zc.x + fmaxf(fmaxf(zc.y, zc.z), 0.0f) < 0.999f;
              if (!(h.x >> 31)) {
                const int E0 = a.x + b.x * dx + b.y * dy, E1 = a.y + b.z * dx + b.w * dy;
#pragma unroll
                for (int s = 0; s < S; ++s) {
                  const int2 sp = sample_pos<S>(s);
                  const int e0 = E0 + (b.x >> 8) * sp.x + (b.y >> 8) * sp.y;
                  const int e1 = E1 + (b.z >> 8) * sp.x + (b.w >> 8) * sp.y;
                  const int e2 = a.z - e0 - e1;
                  if (near) {
                    cover |= ((uint32_t)~(e0 | e1 | e2) >> 31) << s;
                  } else if ((e0 | e1 | e2) >= 0) {
                    const float z = depth_from(zc, to_float((e1 + 1) >> 1), to_float((e2 + 1) >> 1));
                    if (__float_as_uint(z) < opaque_depth(s)) cover |= 1u << s;
                  }
                }
                if (cover) {
                  const int e0 = E0 + (b.x >> 1) + (b.y >> 1), e1 = E1 + (b.z >> 1) + (b.w >> 1);
                  zcen = depth_from(zc, to_float((e1 + 1) >> 1), to_float((a.z - e0 - e1 + 1) >> 1));
                }
              } else {
                const int bxp = (w.rx0 + dx) * 256, byp = (w.ry0 + dy) * 256;
#pragma unroll 1
                for (int s = 0; s < S; ++s) {
                  const int2 sp = sample_pos_at<S>(s);
                  const Edges e = edges_at<long long>(a, b, bxp + sp.x, byp + sp.y);
                  if (inside(e, b.z) && __float_as_uint(depth_at(zc, e)) < opaque_depth(s)) cover |= 1u << s;
                }
                if (cover) zcen = depth_at(zc, edges_at<long long>(a, b, bxp + 128, byp + 128));
              }
            }
            if constexpr (Pol::kPasses > 1) {
              if (!select(cover != 0, __float_as_uint(zcen), owner)) cover = 0;
            }
            const uint32_t m = __ballot_sync(kFull, cover != 0);
            if (cover) {
              const int e = qn + __popc(m & lt);
              st.ent[e] = {__float_as_uint(zcen), (uint32_t)j | ((uint32_t)owner << 8) | (cover << 16)};
              if (!Pol::kDirect) atomicOr(&st.mine[e >> 5][owner], 1u << (e & 31));
            }
            qn += __popc(m);
            __syncwarp();
          }
        }
        // the next group may add 32 fragments; the next hits replace the records
        const bool done = base + 32 >= total;
        if constexpr (S > 1) {
          // shades the covered pixels
#pragma unroll 1
          while (qn > qs && (done || qn > kQueue - 32 || (Pol::kDirect && qn >= 32))) {
            const int e = qs + w.lane;
            const bool act = e < qn;
            const auto en = st.ent[e % kQueue];
            const int owner = (int)((en.info >> 8) & 31u);
            const uint2 h = st.hit[en.info & 31u];
            const TriSetup& T = st.rec[(h.x >> 11) & 31u];
            const int cnt = min(qn - qs, 32);
            uint32_t node0 = 0;
            if (Pol::kDirect && Pol::kNodes && w.lane == 0) node0 = atomicAdd(p.counter, (uint32_t)cnt);
            Frag f;
            Shade sh;
            float alpha = 0.f;
            if (act) {
              float3 v;
              f.cover = (en.info >> 16) & 255u;
              f.depth = en.depth;
              edges(h, T, owner, v, alpha);
              shade_fragment(h, T, v, f, sh);
            }
            if constexpr (Pol::kDirect) {
              write_direct(act, cnt == 32 ? kFull : (1u << cnt) - 1u, owner, f, sh, alpha, node0);
              const auto nx = st.ent[32 + w.lane];
              __syncwarp();
              st.ent[w.lane] = nx;
              qn -= cnt;
              __syncwarp();
            } else {
              if (act) Pol::produce(p, pass, pay, e, f, sh, alpha);
              qs += cnt;
            }
          }
        }
        if constexpr (!Pol::kDirect) {
          if (last || qn > kQueue - 32) {
            feed();
            qs = 0;
          }
        }
        if (last) break;
      }
    });
  }

  pol.flush(p, w.valid);
  if (w.valid && p.color) {
    float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int s = 0; s < S; ++s) {
      c.x += tg.col[s].x;
      c.y += tg.col[s].y;
      c.z += tg.col[s].z;
      c.w += tg.col[s].w;
    }
    const float k = 1.0f / (float)S;
    store_color(p.color, p.color_half != 0, elem, make_float4(c.x * k, c.y * k, c.z * k, c.w * k));
  }
  if (w.lane == 0 && nfrag && p.frag_count) atomicAdd(p.frag_count, (unsigned long long)nfrag);
  if (SSN == 1 && p.lens) {
    const uint32_t mx = __reduce_max_sync(kFull, w.valid ? got : 0u);
    // micro-tiles of edge tiles may lie wholly outside the image
    if (w.lane == 0 && w.rx0 < p.RW && w.ry0 < p.RH)
      p.lens[(size_t)(w.ry0 >> 2) * p.lens_stride + (w.rx0 >> 3)] = (uint8_t)min(mx, 255u);
  }
}

// The view of a multi-view launch that CTA `block` belongs to, and the CTA's
// index within that view's grid (block-uniform).
__device__ __forceinline__ int mv_view(const oit::MvRaster& mv, uint32_t block, int& cta) {
  int lo = 0, hi = mv.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (mv.cta_end[mid] > block) hi = mid; else lo = mid + 1;
  }
  cta = (int)(block - (lo ? mv.cta_end[lo - 1] : 0u));
  return lo;
}


// Resident warps per SM with S samples a lane (WBOIT: accumulators too).
template <int S>
constexpr int msaa_warps(bool weighted) {
  return S == 4 ? (weighted ? 20 : 24) : (weighted ? 16 : 20);
}

// One view's pass: one CTA per kRasterWarpsPerBlock micro-tile warps, compiled
// for WPSM resident warps per SM with one coverage sample per lane (the
// register budget: 36 -> 56 registers, 32 -> 64).
template <template <int> class Policy, int S, int SSN, int WPSM>
__global__ void __launch_bounds__(32 * kRasterWarpsPerBlock,
                                  (S == 1 ? WPSM : msaa_warps<S>(Policy<S>::kViewZ)) / kRasterWarpsPerBlock)
    k_raster_transparent(RasterParams p) {
  frame_order();
  raster_transparent_body<Policy, S, SSN>(p, (int)blockIdx.x);
}

// Several views' passes in one grid: the CTAs of view 0, then view 1, ...
// (the hardware hands out CTAs as earlier ones retire, so the views share the
// machine and small views fill what large ones leave).
template <template <int> class Policy, int S, int SSN>
__global__ void __launch_bounds__(32 * kRasterWarpsPerBlock,
                                  (S == 1 ? Policy<S>::kWarpsPerSM : msaa_warps<S>(Policy<S>::kViewZ)) /
                                      kRasterWarpsPerBlock)
    k_raster_transparent_mv(const __grid_constant__ oit::MvRaster mv) {
  frame_order();
  int cta;
  const int v = mv_view(mv, blockIdx.x, cta);
  raster_transparent_body<Policy, S, SSN>(mv.v[v], cta);
}

// ---------------------------------------------------------------------------
// Opaque pass: opaque.frag.glsl:30-35, depth LESS with write (main.cpp:542-547).
// ---------------------------------------------------------------------------
// Per sample the nearest triangle, the first in primitive order among equal
// depths, is kept in shared memory; each pixel is shaded at the end, once per
// distinct triangle of its samples. Coverage as in the transparent pass.
// Measured against every fragment shaded, hits tested one after the other by
// all lanes, and targets cleared by fills beforehand: frames of Loop64
// 1920x1080 with 40% opaque spheres 421 -> 353 us, Simple 1283x717 4x MSAA with
// 30% 458 -> 382 us.
// id: the triangle's place in primitive order, 2 t for triangle t or its first
// half and 2 t + 1 for its second.
template <int S>
struct OpaqueStage {
  TriSetup rec[kHits];  // (normals and colours unused)
  uint2 hit[kHits];
  uint32_t ring[kRing];
  uint32_t z[S][32];
  uint32_t id[S][32];
};
constexpr uint32_t kNoTriangle = 0xFFFFFFFFu;

// Of the warp's fragments (pass: nearer than the sample's depth z), keeps per
// sample the nearest, the lowest id among equal depths. Warp-uniform call.
__device__ __forceinline__ void keep_nearest(uint32_t* z, uint32_t* id, bool pass, int owner, uint32_t zf,
                                             uint32_t oid) {
  if (!__any_sync(kFull, pass)) return;
  if (pass) atomicMin(&z[owner], zf);
  __syncwarp();
  const bool win = pass && z[owner] == zf;  // (an earlier fragment of this depth would not have let it pass)
  if (win) id[owner] = kNoTriangle;
  __syncwarp();
  if (win) atomicMin(&id[owner], oid);
  __syncwarp();
}

template <int S>
__device__ __forceinline__ void raster_opaque_body(const RasterParams& p, int cta) {
  using M = LaneMap<1>;
  __shared__ OpaqueStage<S> st_all[kRasterWarpsPerBlock];
  const int warp = threadIdx.x >> 5;
  const WarpTile w = warp_tile<1>(p, cta);
  OpaqueStage<S>& st = st_all[warp];
  const TriSetup* setup = reinterpret_cast<const TriSetup*>(p.setup);
  const uint32_t lt = (1u << w.lane) - 1u;
  const uint32_t lanes = __ballot_sync(kFull, w.valid);
#pragma unroll
  for (int s = 0; s < S; ++s) {
    st.z[s][w.lane] = w.valid && !p.opaque_fresh ? p.depth[(size_t)s * p.P + w.pixel] : 0x3F800000u;
    st.id[s][w.lane] = kNoTriangle;
  }
  const int tile = w.tile + p.tile_offset;
  walk_pass<false>(p, w, st.ring, p.tile_begin[tile], p.tile_end[tile], [&](uint32_t head, int nh, bool) {
    int total = 0;
    const int pre = stage_hits<S, 1, false>(w, setup, st.ring, st.rec, st.hit, lanes, head, nh, total);
    int khi = -1;
#pragma unroll 1
    for (int base = 0; base < total; base += 32) {
      const uint32_t rel = (uint32_t)(pre - base);
      const uint32_t starts = __reduce_or_sync(kFull, rel < 32u ? 1u << rel : 0u);
      const int j = khi + __popc(starts & (lt | (1u << w.lane)));
      khi += __popc(starts);
      const bool act = base + w.lane < total;
      const uint2 h = st.hit[j];
      const int k = (int)((h.x >> 11) & 31u);
      const TriSetup& T = st.rec[k];
      const int owner = act ? nth_bit(h.y, (uint32_t)(base + w.lane) - (h.x & 0x7FFu)) : w.lane;
      const int dx = owner % M::kW, dy = owner / M::kW;
      const uint32_t t = st.ring[(head + k) % kRing];
      const uint32_t oid = t >= p.num_tris ? 2u * (t - p.num_tris) + 1u : 2u * t;
      uint32_t zs[S];
#pragma unroll
      for (int s = 0; s < S; ++s) zs[s] = 0xFFFFFFFFu;
      if (act) {
        const int4 a = T.xy01, b = T.xy2f;
        const float4 zc = T.zc;
        if (!(h.x >> 31)) {
          const int E0 = a.x + b.x * dx + b.y * dy, E1 = a.y + b.z * dx + b.w * dy;
#pragma unroll
          for (int s = 0; s < S; ++s) {
            const int2 sp = S > 1 ? sample_pos<S>(s) : make_int2(0, 0);  // (1x: taken at the centre)
            const int e0 = E0 + (b.x >> 8) * sp.x + (b.y >> 8) * sp.y;
            const int e1 = E1 + (b.z >> 8) * sp.x + (b.w >> 8) * sp.y;
            const int e2 = a.z - e0 - e1;
            if ((e0 | e1 | e2) >= 0)
              zs[s] = __float_as_uint(depth_from(zc, to_float((e1 + 1) >> 1), to_float((e2 + 1) >> 1)));
          }
        } else {
          const int bxp = (w.rx0 + dx) * 256, byp = (w.ry0 + dy) * 256;
#pragma unroll
          for (int s = 0; s < S; ++s) {
            const int2 sp = sample_pos<S>(s);
            const Edges e = edges_at<long long>(a, b, bxp + sp.x, byp + sp.y);
            if (inside(e, b.z)) zs[s] = __float_as_uint(depth_at(zc, e));
          }
        }
      }
#pragma unroll
      for (int s = 0; s < S; ++s) keep_nearest(st.z[s], st.id[s], zs[s] < st.z[s][owner], owner, zs[s], oid);
    }
  });
  if (!w.valid) return;
  uint32_t shaded = kNoTriangle;
  float4 c = p.background;
#pragma unroll 1
  for (int s = 0; s < S; ++s) {
    const uint32_t id = st.id[s][w.lane];
    if (id == kNoTriangle && !p.opaque_fresh) continue;
    if (id != shaded) {
      c = p.background;
      if (id != kNoTriangle) {
        const TriSetup& T = setup[(id & 1u) ? p.num_tris + (id >> 1) : id >> 1];
        const Shade sh = shade(T, edges_at<long long>(T.xy01, T.xy2f, w.px * 256 + 128, w.py * 256 + 128), nullptr);
        c = make_float4(sh.r, sh.g, sh.b, 1.0f);
      }
      shaded = id;
    }
    p.depth[(size_t)s * p.P + w.pixel] = st.z[s][w.lane];
    p.opaque_color[(size_t)s * p.P + w.pixel] = c;
  }
}

// (the bound is what the registers come to without it, less spills at 1x)
template <int S>
__global__ void __launch_bounds__(32 * kRasterWarpsPerBlock, S == 1 ? 19 : 16) k_raster_opaque(RasterParams p) {
  frame_order();
  raster_opaque_body<S>(p, (int)blockIdx.x);
}

template <int S>
__global__ void __launch_bounds__(32 * kRasterWarpsPerBlock)
    k_raster_opaque_mv(const __grid_constant__ oit::MvRaster mv) {
  frame_order();
  int cta;
  const int v = mv_view(mv, blockIdx.x, cta);
  raster_opaque_body<S>(mv.v[v], cta);
}

}  // namespace oitd

namespace oitd {

// Shared memory of a warp of one view's pass.
template <template <int> class Pol, int S>
size_t warp_smem_bytes(const RasterParams& p) {
  return warp_stage_bytes<S, Pol<S>::kViewZ>(Pol<S>::payload_bytes(p.tail, p.record_fp32, p.weighted_fp32)) +
         Pol<S>::smem_bytes_per_warp(p.L, p.coverage, p.record_fp32);
}

template <template <int> class Pol, int S, int SSN, int WPSM>
cudaError_t launch_transparent_w(const RasterParams& p, cudaStream_t s) {
  const size_t smem = (size_t)kRasterWarpsPerBlock *
                      warp_smem_bytes<Pol, S>(p);
  if (smem > 48 * 1024) {
    // raise the kernel's dynamic shared memory cap once per device (never
    // while a CUDA graph is being captured after the first frame)
    static int cap_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || cap_set[dev] < (int)smem) {
      cudaError_t e = cudaFuncSetAttribute(k_raster_transparent<Pol, S, SSN, WPSM>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      if (dev >= 0 && dev < 64) cap_set[dev] = (int)smem;
    }
  }
  const unsigned ctas = (unsigned)(p.tiles_x * p.tiles_y * SSN * (oit::kWarpsPerTile / kRasterWarpsPerBlock));
  launch_in_frame(k_raster_transparent<Pol, S, SSN, WPSM>, ctas, 32 * kRasterWarpsPerBlock, smem, s, p);
  return cudaGetLastError();
}

// One sample per lane: 32 warps per SM (64 registers), or where p.warps_per_sm
// asks for 36 and the policy has it, 36 (56 registers, some spilled).
template <template <int> class Pol, int S, int SSN>
cudaError_t launch_transparent_s(const RasterParams& p, cudaStream_t s) {
  if constexpr (S == 1 && SSN == 1 && Pol<S>::kWarpsPerSM != 32) {
    if (p.warps_per_sm == Pol<S>::kWarpsPerSM) return launch_transparent_w<Pol, S, SSN, Pol<S>::kWarpsPerSM>(p, s);
  }
  return launch_transparent_w<Pol, S, SSN, 32>(p, s);
}

// Multi-view launch of one policy: mv.v[0..n) share S / SSN; the dynamic
// shared memory covers the largest per-warp policy state among them.
template <template <int> class Pol, int S, int SSN>
cudaError_t launch_transparent_mv_s(const oit::MvRaster& mv, cudaStream_t s) {
  size_t per_warp = 0;
  for (int i = 0; i < mv.n; ++i)
    per_warp = std::max(per_warp, warp_smem_bytes<Pol, S>(mv.v[i]));
  const size_t smem = (size_t)kRasterWarpsPerBlock * per_warp;
  if (smem > 48 * 1024) {
    static int cap_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || cap_set[dev] < (int)smem) {
      cudaError_t e = cudaFuncSetAttribute(k_raster_transparent_mv<Pol, S, SSN>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      if (dev >= 0 && dev < 64) cap_set[dev] = (int)smem;
    }
  }
  const uint32_t ctas = mv.n > 0 ? mv.cta_end[mv.n - 1] : 0u;
  if (!ctas) return cudaSuccess;
  launch_in_frame(k_raster_transparent_mv<Pol, S, SSN>, ctas, 32 * kRasterWarpsPerBlock, smem, s, mv);
  return cudaGetLastError();
}

template <template <int> class Pol>
cudaError_t launch_transparent_mv(const oit::MvRaster& mv, cudaStream_t s) {
  if (mv.n <= 0) return cudaSuccess;
  const RasterParams& p = mv.v[0];
  if (p.ssn > 1) {
    switch (p.ssn) {
      case 4: return launch_transparent_mv_s<Pol, 1, 4>(mv, s);
      case 8: return launch_transparent_mv_s<Pol, 1, 8>(mv, s);
      default: return cudaErrorInvalidValue;
    }
  }
  switch (p.S) {
    case 1: return launch_transparent_mv_s<Pol, 1, 1>(mv, s);
    case 4: return launch_transparent_mv_s<Pol, 4, 1>(mv, s);
    case 8: return launch_transparent_mv_s<Pol, 8, 1>(mv, s);
    default: return cudaErrorInvalidValue;
  }
}

inline cudaError_t launch_opaque_mv(const oit::MvRaster& mv, cudaStream_t s) {
  if (mv.n <= 0) return cudaSuccess;
  const uint32_t ctas = mv.cta_end[mv.n - 1];
  if (!ctas) return cudaSuccess;
  constexpr int kThreads = 32 * kRasterWarpsPerBlock;
  switch (mv.v[0].S) {
    case 1: launch_in_frame(k_raster_opaque_mv<1>, ctas, kThreads, 0, s, mv); break;
    case 4: launch_in_frame(k_raster_opaque_mv<4>, ctas, kThreads, 0, s, mv); break;
    case 8: launch_in_frame(k_raster_opaque_mv<8>, ctas, kThreads, 0, s, mv); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <template <int> class Pol>
cudaError_t launch_transparent(const RasterParams& p, cudaStream_t s) {
  if (p.ssn > 1) {
    switch (p.ssn) {
      case 4: return launch_transparent_s<Pol, 1, 4>(p, s);
      case 8: return launch_transparent_s<Pol, 1, 8>(p, s);
      default: return cudaErrorInvalidValue;
    }
  }
  switch (p.S) {
    case 1: return launch_transparent_s<Pol, 1, 1>(p, s);
    case 4: return launch_transparent_s<Pol, 4, 1>(p, s);
    case 8: return launch_transparent_s<Pol, 8, 1>(p, s);
    default: return cudaErrorInvalidValue;
  }
}

inline cudaError_t launch_opaque(const RasterParams& p, cudaStream_t s) {
  const unsigned grid = (unsigned)(p.tiles_x * p.tiles_y * (oit::kWarpsPerTile / kRasterWarpsPerBlock));
  constexpr int kThreads = 32 * kRasterWarpsPerBlock;
  switch (p.S) {
    case 1: launch_in_frame(k_raster_opaque<1>, grid, kThreads, 0, s, p); break;
    case 4: launch_in_frame(k_raster_opaque<4>, grid, kThreads, 0, s, p); break;
    case 8: launch_in_frame(k_raster_opaque<8>, grid, kThreads, 0, s, p); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace oitd
