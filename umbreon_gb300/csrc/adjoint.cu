// adjoint.cu -- ubr_adjoint: reverse-mode derivative of a single-layer sphere
// frame (the forward path of render.cu restricted to one opaque layer of
// spheres, POV shading, hard shadows, legacy or enhanced AO, fog, box
// downsample and gamma) with respect to the scene and render parameters.
//
// Nothing from a forward render is stored or reused.  The adjoint re-traces:
//   k_adj_primary   closest hit of every hi-res primary ray (the hit record
//                   and the 3x3 interior test read it)
// then, over chunks of the pixels,
//   k_adj_surface   queues the hit samples that count, with their secondary
//                   rays' origin, normal, AO start node and tangent
//   k_adj_rays      one thread per AO ray (nearest hit and its sphere) and
//                   shadow ray (any hit)
//   k_adj_shade     per queued sample: recompute the shaded colour and push
//                   dL/d(colour) back through gamma, downsample, fog,
//                   shadeLocal (shading.hpp:76-192), the AO estimators
//                   (ambient_occlusion.hpp:33-57, 171-267) and the sphere hit
//                   (t, P, N, self-intersection epsilon)
// and, in k_adj_surface, the background.  When the assumed gamma is not 1, a
// forward pass of k_adj_shade over the same rays and k_adj_down give the
// downsampled value the gamma derivative needs.
// Visibility (which sphere a ray hits, each shadow bit, each AO sample's
// grazing test and occluder, the frame-from-normal branch) is a constant of
// the derivative; per-sphere gradients are scattered with float atomics,
// global ones reduced per warp and block and added in double.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "trace.cuh"

namespace ubr {
namespace {

constexpr int kAdjLights = UBR_ADJOINT_MAX_LIGHTS;

// global gradient slots
enum : int {
  gAmbient = 0,
  gDiffuse,
  gSpecular,
  gRoughness,
  gBrilliance,
  gPhong,
  gPhongSize,
  gReflection,
  gEmission,
  gAmbColor = 9,      // 3
  gBg = 12,           // 3
  gFogStart = 15,
  gFogEnd = 16,
  gFogColor = 17,     // 3
  gAoDistance = 20,
  gAoIntensity = 21,
  gSpecScale = 22,
  gLightL = 23,       // 3 per light: d/d (unit) light vector
  gLightC = 23 + 3 * kAdjLights,  // 3 per light: d/d light colour x intensity
  kGlobals = 23 + 6 * kAdjLights
};

struct AdjBufs {
  const float2* hit;        // per hi-res sample: t, ref bits
  const float4* dOut;       // dL/d(output colour), outW x outH
  const float4* outFwd;     // forward output colour (gamma derivative), or null
  float4* colorHi;          // forward mode: fogged hi-res colour
  const LightD* lights;
  float* gColor;            // per input sphere x 3
  float* gCenter;           // per input sphere x 3
  float* gRadius;           // per input sphere
  float4* acc;              // per input sphere: (centre, radius) (colour, -) sums, or null: the arrays above
  double* gGlobal;          // kGlobals
  unsigned long long* stats;  // 0 samples, 1 rays, 2 overflow, 3 a chunk's queue length
  uint32_t flags;
};

// A chunk's queue of hit samples and the results of their secondary rays.
struct AdjRays {
  uint32_t* count;
  uint32_t* pix;    // hi-res pixel
  float4* a;        // secondary-ray origin, eps
  float4* b;        // normal, AO start node
  float4* c;        // AO frame tangent
  float2* ao;       // per hit and AO ray: nearest t (inf: none), its reference; unset below the grazing cosine
  uint8_t* shadow;  // per hit and light: 1 = occluded; unset where the hit faces away
};

// Adds a sphere's (centre, radius) gradient: one 16-byte reduction into the
// packed sums, or four into the caller's arrays (an arena cap leaves no room
// for the sums).
UBR_D void addGeom(const AdjBufs& b, uint32_t k, f3 c, float r);
UBR_D void addColor(const AdjBufs& b, uint32_t k, f3 v);

UBR_D void atomicAdd3(float* a, uint32_t k, f3 v) {
  if (!a) return;
  atomicAdd(a + 3 * k, v.x);
  atomicAdd(a + 3 * k + 1, v.y);
  atomicAdd(a + 3 * k + 2, v.z);
}

UBR_D void addGeom(const AdjBufs& b, uint32_t k, f3 c, float r) {
  if (b.acc) {
    atomicAdd(b.acc + 2 * size_t(k), make_float4(c.x, c.y, c.z, r));
  } else {
    atomicAdd3(b.gCenter, k, c);
    if (b.gRadius) atomicAdd(b.gRadius + k, r);
  }
}
UBR_D void addColor(const AdjBufs& b, uint32_t k, f3 v) {
  if (b.acc) atomicAdd(b.acc + 2 * size_t(k) + 1, make_float4(v.x, v.y, v.z, 0.0f));
  else atomicAdd3(b.gColor, k, v);
}
__global__ void k_adj_unpack(uint32_t n, AdjBufs b) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const float4 g = b.acc[2 * size_t(k)], c = b.acc[2 * size_t(k) + 1];
  if (b.gCenter) {
    b.gCenter[3 * size_t(k)] = g.x;
    b.gCenter[3 * size_t(k) + 1] = g.y;
    b.gCenter[3 * size_t(k) + 2] = g.z;
  }
  if (b.gRadius) b.gRadius[k] = g.w;
  if (b.gColor) {
    b.gColor[3 * size_t(k)] = c.x;
    b.gColor[3 * size_t(k) + 1] = c.y;
    b.gColor[3 * size_t(k) + 2] = c.z;
  }
}

// Adds the block's sums of N per-thread values to global[0..N): floats within
// a warp and the block of 128, double across blocks.
template <int N>
UBR_D void addGlobals(double* global, const float (&G)[N]) {
  __shared__ float sAcc[N];
  for (int k = threadIdx.x; k < N; k += blockDim.x) sAcc[k] = 0.0f;
  __syncthreads();
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    float v = G[k];
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 16);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 8);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 4);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 2);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 1);
    if (lane == 0 && v != 0.0f) atomicAdd(&sAcc[k], v);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < N; k += blockDim.x)
    if (sAcc[k] != 0.0f) atomicAdd(&global[k], double(sAcc[k]));
}

UBR_D f3 mul3(f3 a, f3 b) { return f3{a.x * b.x, a.y * b.y, a.z * b.z}; }

// d(a / |a|) transposed applied to g: (g - n (n.g)) / |a| with n = a / |a|
UBR_D f3 normalizeBack(f3 n, float len, f3 g) {
  const float ng = dot(n, g);
  const float inv = 1.0f / len;
  return f3{(g.x - n.x * ng) * inv, (g.y - n.y * ng) * inv, (g.z - n.z * ng) * inv};
}

__global__ void __launch_bounds__(128) k_adj_primary(Params p, TravScene ts, float2* hit, uint32_t npix,
                                                     unsigned long long* stats) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t ovf = 0, traced = 0;
  if (k < npix) {
    const uint32_t i = tiledPixel(k, uint32_t(p.W), uint32_t(p.H));
    const int px = int(i % uint32_t(p.W)), py = int(i / uint32_t(p.W));
    f3 org, rd;
    primaryRay(p, px, py, org, rd);
    float tn, tf;
    clipRange(p, rd, tn, tf);
    Hit h;
    h.t = 0.0f;
    const bool any = traverse<false, kMaskSphere, false, false, true>(ts, Ray{org, rd, tn, tf}, h, ovf, nullptr, false);
    hit[i] = make_float2(any ? h.t : 0.0f, __uint_as_float(any ? h.ref : kInvalid));
    traced = 1;
  }
  warpCount(&stats[1], traced);
  warpCount(&stats[2], ovf);
}

// Fog factor of view-z z (fog.cpp:17-36) and its partial derivatives (zero
// where the factor is clamped or the fog is a step).
struct FogD {
  float f, dz, dStart, dEnd;
  bool on;
};
UBR_D FogD fogAt(const Params& p, float z) {
  FogD r{1.0f, 0.0f, 0.0f, 0.0f, false};
  if (!p.fogOn || !(z > 0.0f)) return r;
  r.on = true;
  const float denom = p.fogEnd - p.fogStart;
  if (denom <= 0.0f) {
    r.f = z < p.fogEnd ? 1.0f : 0.0f;
    return r;
  }
  const float f = (p.fogEnd - z) / denom;
  if (f < 0.0f) {
    r.f = 0.0f;
  } else if (f > 1.0f) {
    r.f = 1.0f;
  } else {
    r.f = f;
    r.dz = -1.0f / denom;
    r.dStart = (p.fogEnd - z) / (denom * denom);
    r.dEnd = (z - p.fogStart) / (denom * denom);
  }
  return r;
}

// dL/d(this sample's fogged colour); false when it is zero or the sample does
// not count (interior only).
UBR_D bool sampleGradient(const Params& p, const AdjBufs& b, uint32_t i, int px, int py, uint32_t ref, float4& g) {
  const int ox = px / p.ss, oy = py / p.ss;
  const uint32_t o = uint32_t(oy) * uint32_t(p.outW) + uint32_t(ox);
  g = b.dOut[o];
  if (!(fabsf(p.gamma - 1.0f) <= 1.0e-4f)) {
    // applyAssumedGamma: v > 0 ? v^gamma : 0 (image_ops.cpp:37-46)
    const float4 v = b.outFwd[o];
    g.x = v.x > 0.0f ? g.x * p.gamma * powf(v.x, p.gamma - 1.0f) : 0.0f;
    g.y = v.y > 0.0f ? g.y * p.gamma * powf(v.y, p.gamma - 1.0f) : 0.0f;
    g.z = v.z > 0.0f ? g.z * p.gamma * powf(v.z, p.gamma - 1.0f) : 0.0f;
  }
  if (p.ss > 1) {
    const float inv = 1.0f / float(p.ss * p.ss);
    g = make_float4(g.x * inv, g.y * inv, g.z * inv, g.w * inv);
  }
  if (!(g.x != 0.0f || g.y != 0.0f || g.z != 0.0f || g.w != 0.0f)) return false;
  if (b.flags & UBR_ADJOINT_INTERIOR_ONLY) {
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        const int qx = px + dx, qy = py + dy;
        if (qx < 0 || qy < 0 || qx >= p.W || qy >= p.H) continue;
        if (__float_as_uint(b.hit[uint32_t(qy) * uint32_t(p.W) + uint32_t(qx)].y) != ref) return false;
      }
  }
  return true;
}

// A hit sample's geometry: the hit point, normals and the secondary-ray origin
// P + safeNormalize(Ng toward N) * eps (k_surface).
struct AdjHit {
  f3 org, rd, P, Ng, nHat, N, ng, O, cc;
  float t, rad, ngLen, sgn, eps;
  uint32_t prim;
};
UBR_D AdjHit adjHit(const Params& p, const DScene& s, int px, int py, float2 hr) {
  AdjHit h;
  h.prim = refPrim(__float_as_uint(hr.y));
  const float4 sc = __ldg(&s.sph[h.prim]);
  h.cc = f3{sc.x, sc.y, sc.z};
  h.rad = sc.w;
  primaryRay(p, px, py, h.org, h.rd);
  h.t = hr.x;
  h.P = f3{h.org.x + h.rd.x * h.t, h.org.y + h.rd.y * h.t, h.org.z + h.rd.z * h.t};
  h.Ng = h.rd * h.t - (h.cc - h.org);  // isectSphere's geometric normal
  h.ngLen = length(h.Ng);
  h.nHat = normalize(h.Ng);
  h.sgn = dot(h.nHat, h.rd) > 0.0f ? -1.0f : 1.0f;  // faceForward
  h.N = h.nHat * h.sgn;
  h.eps = selfIntersectEps(h.P, h.rd, h.t);
  const f3 ng = dot(h.Ng, h.N) < 0.0f ? neg(h.Ng) : h.Ng;
  h.ng = safeNormalize(ng, h.N);
  h.O = h.P + h.ng * h.eps;
  return h;
}

// The chunk's hit samples that need shading, with what their secondary rays
// start from.  With `all` every hit sample (the forward pass of the gamma
// derivative), else those whose gradient is not zero.  BACKGROUND: the others
// too, as k_adj_background<true> does in a launch of its own (4 us of a small
// frame's 60, and the hits are read once).
template <bool BACKGROUND>
__global__ void __launch_bounds__(128) k_adj_surface(Params p, DScene s, AdjBufs b, AdjRays r, uint32_t i0, uint32_t n,
                                                     int all) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  bool take = false;
  uint32_t i = 0, used = 0;
  AdjHit h;
  float4 bg = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (k < n) {
    i = tiledPixel(i0 + k, uint32_t(p.W), uint32_t(p.H));
    const int px = int(i % uint32_t(p.W)), py = int(i / uint32_t(p.W));
    const float2 hr = b.hit[i];
    const uint32_t ref = __float_as_uint(hr.y);
    if (ref != kInvalid) {
      float4 g;
      take = all || sampleGradient(p, b, i, px, py, ref, g);
      if (take) h = adjHit(p, s, px, py, hr);
    } else if (BACKGROUND) {
      used = sampleGradient(p, b, i, px, py, kInvalid, bg) ? 1 : 0;
      if (!used) bg = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  }
  if (BACKGROUND) {
    const float cov = p.transparentBg ? 0.0f : 1.0f;
    const float G[3] = {bg.x * cov, bg.y * cov, bg.z * cov};
    addGlobals<3>(b.gGlobal + gBg, G);
    warpCount(&b.stats[0], used);
  }
  int off;
  const int q = warpPushBase(take, r.count, off) + off;
  if (!take) return;
  r.pix[q] = i;
  const bool aoOn = p.aoSamples > 0 && __ldg(&s.primFromEdge[kSphere][h.prim]) == 0;
  int start = 0;
  if (aoOn) {
    f3 lo, hi;
    aoBox(h.O, p.aoDistance, lo, hi);
    start = boxStartNode(travOf(s), lo, hi);
    const Frame3 fr = frameFromNormal(h.N);
    r.c[q] = make_float4(fr.t.x, fr.t.y, fr.t.z, 0.0f);
  }
  r.a[q] = make_float4(h.O.x, h.O.y, h.O.z, h.eps);
  r.b[q] = make_float4(h.N.x, h.N.y, h.N.z, __int_as_float(start));
}

// One thread per AO ray (hit-major: a warp holds the rays of two hits at 16
// samples) and per shadow ray (light-major) of the chunk's hits: nearest hit
// and its sphere for the enhanced estimator, else any hit.
template <bool NEAREST>
__global__ void __launch_bounds__(128, 9) k_adj_rays(Params p, DScene s, AdjBufs b, AdjRays r) {
  const uint64_t tid = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const uint32_t nq = *r.count;
  const uint64_t nAo = uint64_t(nq) * uint32_t(p.aoSamples);
  uint32_t traced = 0, ovf = 0;
  const TravScene ts = travOf(s);
  if (tid < nAo) {
    const uint32_t q = uint32_t(tid / uint32_t(p.aoSamples)), k = uint32_t(tid % uint32_t(p.aoSamples)), i = r.pix[q];
    if (__ldg(&s.primFromEdge[kSphere][refPrim(__float_as_uint(b.hit[i].y))]) == 0) {
      const float4 a = r.a[q], n4 = r.b[q];
      const f3 N = ld3(n4), T = ld3(r.c[q]);
      const f3 dir = aoDir(p, Frame3{T, cross(N, T), N}, int(i % uint32_t(p.W)), int(i / uint32_t(p.W)), int(k));
      if (!(dot(dir, N) < 0.01f)) {
        Hit h;
        const bool hit = traverse<false, kMaskSphere, !NEAREST>(ts, Ray{ld3(a), dir, a.w, p.aoDistance}, h, ovf, nullptr,
                                                                !NEAREST, __float_as_int(n4.w));
        r.ao[tid] = make_float2(hit ? h.t : kInfF, __uint_as_float(hit ? h.ref : kInvalid));
        traced = 1;
      }
    }
  } else if (p.shadowsActive && tid - nAo < uint64_t(nq) * uint32_t(p.nLights)) {
    const uint32_t t = uint32_t(tid - nAo), l = t / nq, q = t - l * nq, i = r.pix[q];
    const float4 a = r.a[q], n4 = r.b[q];
    const f3 L = b.lights[l].L;
    if (dot(ld3(n4), L) > 0.0f && __ldg(&s.primFromEdge[kSphere][refPrim(__float_as_uint(b.hit[i].y))]) == 0) {
      Hit h;
      r.shadow[size_t(q) * uint32_t(p.nLights) + l] =
          traverse<false, kMaskSphere, true>(ts, Ray{ld3(a), L, a.w, kInfF}, h, ovf, nullptr, true) ? 1 : 0;
      traced = 1;
    }
  }
  warpCount(&b.stats[1], traced);
  warpCount(&b.stats[2], ovf);
}

// Background samples: colour = bg * coverage, alpha = coverage, no fog (view-z
// 0).  GRAD as in k_adj_shade.
template <bool GRAD>
__global__ void __launch_bounds__(128) k_adj_background(Params p, AdjBufs b, uint32_t npix) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const float cov = p.transparentBg ? 0.0f : 1.0f;
  float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  uint32_t used = 0;
  if (i < npix && __float_as_uint(b.hit[i].y) == kInvalid) {
    if (GRAD) {
      used = sampleGradient(p, b, i, int(i % uint32_t(p.W)), int(i / uint32_t(p.W)), kInvalid, g) ? 1 : 0;
      if (!used) g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    } else {
      b.colorHi[i] = make_float4(p.bg.x * cov, p.bg.y * cov, p.bg.z * cov, cov);
    }
  }
  if (GRAD) {
    float G[3] = {g.x * cov, g.y * cov, g.z * cov};
    addGlobals<3>(b.gGlobal + gBg, G);
    warpCount(&b.stats[0], used);
  }
}

// One hit sample of the queue.  GRAD = false: forward colour after fog into
// colorHi.  GRAD = true: the sample's share of every gradient.  The secondary
// rays come traced (k_adj_rays): one thread that walked its sample's 17 rays
// in turn held 168 registers (18 % of the warps) and left its warp's other
// lanes waiting at every ray: 100 k spheres, 1024x1024, enhanced AO 16, one
// light and fog 4.60 -> 3.11 ms (rays 2.20, this kernel 0.60).  At most 128
// registers (unbounded 0.66, 96 0.62).  The samples in lockstep, not each
// lane's hits alone (0.93): hits are most samples, and lanes that drift apart
// scatter their reads and reductions.
template <bool GRAD>
__global__ void __launch_bounds__(128, GRAD ? 4 : 1) k_adj_shade(Params p, DScene s, AdjBufs b, AdjRays r) {
  float G[kGlobals];
#pragma unroll
  for (int k = 0; k < kGlobals; ++k) G[k] = 0.0f;
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x, nq = *r.count;
  if (blockIdx.x * blockDim.x >= nq) return;
  uint32_t used = 0;
  if (q < nq) {
    const uint32_t i = r.pix[q];
    const int px = int(i % uint32_t(p.W)), py = int(i / uint32_t(p.W));
    const float2 hr = b.hit[i];
    // dL/d(this sample's fogged colour)
    float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const bool active = !GRAD || sampleGradient(p, b, i, px, py, __float_as_uint(hr.y), g);
    if (active) {
      const AdjHit h = adjHit(p, s, px, py, hr);
      const uint32_t prim = h.prim, sk = s.baseSph ? prim % s.baseSph : prim;
      const float rad = h.rad, t = h.t, ngLen = h.ngLen, sgn = h.sgn, eps = h.eps;
      const f3 rd = h.rd, P = h.P, Ng = h.Ng, nHat = h.nHat, N = h.N, ng = h.ng, O = h.O;
      const f3 V = normalize(f3{-rd.x, -rd.y, -rd.z});
      const float4 fc = __ldg(&s.primColor[kSphere][prim]);
      const f3 C{fc.x, fc.y, fc.z};
      const ubr_material m = s.mats[__ldg(&s.primMat[kSphere][prim])];
      const bool fromEdge = __ldg(&s.primFromEdge[kSphere][prim]) != 0;
      const bool aoOn = !fromEdge && p.aoSamples > 0;
      const bool shOn = !fromEdge && p.shadowsActive != 0;
      // fog of this sample
      const float z = t * dot(rd, p.camDir);
      const FogD fog = fogAt(p, z);
      const f3 gc = (fog.on && !p.transparentBg) ? f3{g.x * fog.f, g.y * fog.f, g.z * fog.f} : f3{g.x, g.y, g.z};
      const LightD* lights = b.lights;
      const int nL = p.nLights;
      // shadow bits and N.L per light
      uint32_t lit = 0, shadowed = 0;
#pragma unroll
      for (int l = 0; l < kAdjLights; ++l) {
        if (l >= nL) break;
        const LightD L = lights[l];
        if (dot(N, L.L) > 0.0f) {
          lit |= 1u << l;
          if (shOn && r.shadow[size_t(q) * uint32_t(nL) + uint32_t(l)]) shadowed |= 1u << l;
        }
      }
      const float ambTerm = dot(mul3(gc, C), p.ambLight);  // sum_c g_c C_c amb_c
      // dL/d(openness), which does not depend on the openness itself
      float gOpen = 0.0f;
      if (GRAD && aoOn) {
        gOpen = m.ambient * ambTerm * p.aoIntensity;
        if (p.aoDiffuseFactor > 0.0f) {
          float sdiff = 0.0f;
#pragma unroll
          for (int l = 0; l < kAdjLights; ++l) {
            if (l >= nL) break;
            if (!(lit & (1u << l))) continue;
            const LightD L = lights[l];
            const float ndl = dot(N, L.L);
            float d;
            if (m.brilliance == 1.0f) d = ndl;
            else if (m.brilliance == 0.0f) d = 1.0f;
            else d = powf(ndl, m.brilliance);
            const float sf = (shadowed & (1u << l)) ? 0.0f : 1.0f;
            sdiff += m.diffuse * d * dot(mul3(gc, C), L.color) * sf;
          }
          gOpen += sdiff * p.aoDiffuseFactor;
        }
      }
      // --- AO: every sample's traced hit; accumulate openness and, for the
      // enhanced estimator, push dL/d(obs) into the occluder, the origin,
      // the sample direction (through the frame of N) and the AO distance
      float openness = 1.0f;
      f3 gO{0.0f, 0.0f, 0.0f}, gN{0.0f, 0.0f, 0.0f};
      if (aoOn) {
        const Frame3 fr = frameFromNormal(N);
        const float R = p.aoDistance;
        float radius[3], weight[3], scaleOf[3];
        int K;
        if (p.aoMultiScale) {
          K = 3;
          scaleOf[0] = 0.08f; scaleOf[1] = 0.30f; scaleOf[2] = 1.00f;
          radius[0] = 0.08f * R; radius[1] = 0.30f * R; radius[2] = 1.00f * R;
          weight[0] = 0.55f; weight[1] = 0.35f; weight[2] = 0.10f;
        } else {
          K = 1;
          scaleOf[0] = scaleOf[1] = scaleOf[2] = 1.0f;
          radius[0] = radius[1] = radius[2] = R;
          weight[0] = 1.0f; weight[1] = weight[2] = 0.0f;
        }
        const float gObs = -gOpen / float(p.aoSamples);
        float obsSum = 0.0f;
        f3 gT{0.0f, 0.0f, 0.0f}, gB{0.0f, 0.0f, 0.0f};
        float gR = 0.0f;
        for (int k = 0; k < p.aoSamples; ++k) {
          float u1, u2;
          aoUV(p, px, py, k, u1, u2);
          // cosineSampleHemisphere (secondary_rays.hpp:66-73) with its coefficients kept
          const float phi = 6.2831853072f * u1;
          const float rr = sqrtf(u2);
          const float cz = sqrtf(fmaxf(0.0f, 1.0f - u2));
          const float cx = cosf(phi) * rr;
          const float cy = sinf(phi) * rr;
          const f3 dir = fr.t * cx + fr.b * cy + fr.n * cz;
          if (dot(dir, N) < 0.01f) {
            obsSum += 1.0f;
            continue;
          }
          const float2 ah = r.ao[size_t(q) * uint32_t(p.aoSamples) + uint32_t(k)];
          if (__float_as_uint(ah.y) == kInvalid) continue;
          if (!p.aoEnhanced) {
            obsSum += 1.0f;
            continue;
          }
          const float th = ah.x;
          float per = 0.0f, dPerDt = 0.0f, dPerDR = 0.0f;
          for (int q = 0; q < K; ++q) {
            if (th < radius[q]) {
              float fk = 1.0f;
              if (p.aoFalloffPower > 0.0f) {
                float a = 1.0f - th / radius[q];
                if (a < 0.0f) a = 0.0f;
                fk = powf(a, p.aoFalloffPower);
                if (GRAD && a > 0.0f) {
                  const float da = p.aoFalloffPower * powf(a, p.aoFalloffPower - 1.0f);
                  dPerDt += weight[q] * da * (-1.0f / radius[q]);
                  dPerDR += weight[q] * da * th / (radius[q] * radius[q]) * scaleOf[q];
                }
              }
              per += weight[q] * fk;
            }
          }
          obsSum += per;
          if (GRAD && gObs != 0.0f) {
            gR += gObs * dPerDR;
            const float gth = gObs * dPerDt;
            if (gth != 0.0f) {
              // th solves |O + th dir - c_j|^2 = r_j^2
              const uint32_t pj = refPrim(__float_as_uint(ah.y));
              const float4 sj = __ldg(&s.sph[pj]);
              const f3 Q = O + dir * th - f3{sj.x, sj.y, sj.z};
              const float den = dot(Q, dir);
              if (den != 0.0f) {
                const float w = gth / den;
                const uint32_t kj = s.baseSph ? pj % s.baseSph : pj;
                addGeom(b, kj, Q * w, w * sj.w);
                gO = gO - Q * w;
                const f3 gDir = Q * (-w * th);
                gT = gT + gDir * cx;
                gB = gB + gDir * cy;
                gN = gN + gDir * cz;
              }
            }
          }
        }
        openness = 1.0f - obsSum / float(p.aoSamples);
        if (GRAD) {
          G[gAoDistance] += gR;
          // frame of N (scene.hpp:69-76): t = seed / |seed|, b = N x t
          // b = N x t:  dN += t x gB,  dt += gB x N
          gN = gN + cross(fr.t, gB);
          gT = gT + cross(gB, N);
          const bool useSeed0 = fabsf(N.x) < fabsf(N.y);
          const f3 seed = useSeed0 ? f3{0.0f, N.z, -N.y} : f3{-N.z, 0.0f, N.x};
          const float sl2 = dot(seed, seed);
          if (!(sl2 < 1.0e-18f)) {
            const f3 gSeed = normalizeBack(fr.t, sqrtf(sl2), gT);
            if (useSeed0) {
              gN.z += gSeed.y;
              gN.y -= gSeed.z;
            } else {
              gN.z -= gSeed.x;
              gN.x += gSeed.z;
            }
          }
        }
      }
      // --- shadeLocal, POV branch, forward and backward ---
      float aoF = 1.0f, diffuseAo = 1.0f;
      if (aoOn) {
        aoF = 1.0f - p.aoIntensity * (1.0f - openness);
        if (p.aoDiffuseFactor > 0.0f) diffuseAo = 1.0f - p.aoDiffuseFactor * (1.0f - openness);
      }
      f3 out{m.emission * C.x + aoF * m.ambient * C.x * p.ambLight.x,
             m.emission * C.y + aoF * m.ambient * C.y * p.ambLight.y,
             m.emission * C.z + aoF * m.ambient * C.z * p.ambLight.z};
      f3 gC{gc.x * (m.emission + aoF * m.ambient * p.ambLight.x),
            gc.y * (m.emission + aoF * m.ambient * p.ambLight.y),
            gc.z * (m.emission + aoF * m.ambient * p.ambLight.z)};
      if (GRAD) {
        G[gEmission] += dot(gc, C);
        G[gAmbient] += aoF * ambTerm;
        G[gAmbColor] += gc.x * aoF * m.ambient * C.x;
        G[gAmbColor + 1] += gc.y * aoF * m.ambient * C.y;
        G[gAmbColor + 2] += gc.z * aoF * m.ambient * C.z;
        if (aoOn) G[gAoIntensity] += m.ambient * ambTerm * (openness - 1.0f);
      }
      const float ex = blinnExp(m.roughness);
      float gEx = 0.0f;
#pragma unroll
      for (int l = 0; l < kAdjLights; ++l) {
        if (l >= nL) break;
        if (!(lit & (1u << l))) continue;
        const LightD L = lights[l];
        const float ndl = dot(N, L.L);
        const float sf = (shOn && (shadowed & (1u << l))) ? 0.0f : 1.0f;
        const f3 Lc = L.color * sf;
        float d, dDdn, dDdb;
        if (m.brilliance == 1.0f) {
          d = ndl;
          dDdn = 1.0f;
        } else if (m.brilliance == 0.0f) {
          d = 1.0f;
          dDdn = 0.0f;
        } else {
          d = powf(ndl, m.brilliance);
          dDdn = m.brilliance * powf(ndl, m.brilliance - 1.0f);
        }
        dDdb = d * logf(ndl);
        const float dk = m.diffuse * d * diffuseAo;
        out.x += dk * C.x * Lc.x;
        out.y += dk * C.y * Lc.y;
        out.z += dk * C.z * Lc.z;
        f3 gLc = mul3(gc, C) * dk;
        gC = gC + mul3(gc, Lc) * dk;
        const float gDk = dot(mul3(gc, C), Lc);
        float gNdl = 0.0f;
        f3 gL{0.0f, 0.0f, 0.0f};
        if (GRAD) {
          G[gDiffuse] += gDk * d * diffuseAo;
          const float gD = gDk * m.diffuse * diffuseAo;
          gNdl += gD * dDdn;
          G[gBrilliance] += gD * dDdb;
        }
        if (L.highlight) {
          f3 hl;
          float fr = 0.0f, dFr = 0.0f;
          if (m.metallic) {
            float c = ndl;
            if (c > 1.0f) c = 1.0f;
            const float x = acosf(c) * 0.63661977f;
            fr = 0.014567225f / ((x - 1.12f) * (x - 1.12f)) - 0.011612903f;
            const float dx = c < 1.0f ? -0.63661977f / sqrtf(1.0f - c * c) : 0.0f;
            dFr = -2.0f * 0.014567225f / ((x - 1.12f) * (x - 1.12f) * (x - 1.12f)) * dx;
            if (fr < 0.0f) {
              fr = 0.0f;
              dFr = 0.0f;
            }
            if (fr > 1.0f) {
              fr = 1.0f;
              dFr = 0.0f;
            }
            hl = f3{Lc.x * (fr + (1.0f - fr) * C.x), Lc.y * (fr + (1.0f - fr) * C.y),
                    Lc.z * (fr + (1.0f - fr) * C.z)};
          } else {
            hl = Lc;
          }
          float s1 = 0.0f, s2 = 0.0f, nh = 0.0f, rv = 0.0f;
          f3 H{0.0f, 0.0f, 0.0f}, LV{0.0f, 0.0f, 0.0f};
          if (m.specular > 0.0f) {
            LV = f3{L.L.x + V.x, L.L.y + V.y, L.L.z + V.z};
            H = normalize(LV);
            nh = dot(N, H);
            if (nh > 0.0f) s1 = m.specular * powf(nh, ex);
          }
          f3 Rr{0.0f, 0.0f, 0.0f};
          if (m.phong > 0.0f) {
            Rr = 2.0f * ndl * N - L.L;
            rv = dot(Rr, V);
            if (rv > 0.0f && (m.phong_size < 60.0f || rv > 0.0008f)) s2 = m.phong * powf(rv, m.phong_size);
          }
          const float specW = s1 + s2;
          if (specW > 0.0f) {
            const float scl = specW * p.specularScale;
            out.x += scl * hl.x;
            out.y += scl * hl.y;
            out.z += scl * hl.z;
            if (GRAD) {
              const f3 gHl = gc * scl;
              const float gSpecW = p.specularScale * dot(gc, hl);
              G[gSpecScale] += specW * dot(gc, hl);
              if (m.metallic) {
                const f3 mix{fr + (1.0f - fr) * C.x, fr + (1.0f - fr) * C.y, fr + (1.0f - fr) * C.z};
                gLc = gLc + mul3(gHl, mix);
                gC = gC + mul3(gHl, Lc) * (1.0f - fr);
                const float gFr = gHl.x * Lc.x * (1.0f - C.x) + gHl.y * Lc.y * (1.0f - C.y) +
                                  gHl.z * Lc.z * (1.0f - C.z);
                gNdl += gFr * dFr;
              } else {
                gLc = gLc + gHl;
              }
              if (s1 > 0.0f) {
                G[gSpecular] += gSpecW * powf(nh, ex);
                const float gNh = gSpecW * m.specular * ex * powf(nh, ex - 1.0f);
                gEx += gSpecW * s1 * logf(nh);
                gN = gN + H * gNh;
                gL = gL + normalizeBack(H, length(LV), N * gNh);
              }
              if (s2 > 0.0f) {
                G[gPhong] += gSpecW * powf(rv, m.phong_size);
                const float gRv = gSpecW * m.phong * m.phong_size * powf(rv, m.phong_size - 1.0f);
                G[gPhongSize] += gSpecW * s2 * logf(rv);
                const f3 gR = V * gRv;
                gNdl += 2.0f * dot(gR, N);
                gN = gN + gR * (2.0f * ndl);
                gL = gL - gR;
              }
            }
          }
        }
        if (GRAD) {
          gN = gN + L.L * gNdl;
          gL = gL + N * gNdl;
          G[gLightL + 3 * l] += gL.x;
          G[gLightL + 3 * l + 1] += gL.y;
          G[gLightL + 3 * l + 2] += gL.z;
          G[gLightC + 3 * l] += gLc.x * sf;
          G[gLightC + 3 * l + 1] += gLc.y * sf;
          G[gLightC + 3 * l + 2] += gLc.z * sf;
        }
      }
      if (m.reflection > 0.0f) {
        out.x += m.reflection * p.bg.x;
        out.y += m.reflection * p.bg.y;
        out.z += m.reflection * p.bg.z;
        if (GRAD) {
          G[gReflection] += dot(gc, p.bg);
          G[gBg] += m.reflection * gc.x;
          G[gBg + 1] += m.reflection * gc.y;
          G[gBg + 2] += m.reflection * gc.z;
        }
      } else if (GRAD) {
        G[gReflection] += dot(gc, p.bg);
      }
      if (!GRAD) {
        float4 c4 = make_float4(out.x, out.y, out.z, 1.0f);
        if (fog.on) {
          if (p.transparentBg) {
            c4.w *= fog.f;
          } else {
            c4.x = p.fogColor.x * (1.0f - fog.f) + c4.x * fog.f;
            c4.y = p.fogColor.y * (1.0f - fog.f) + c4.y * fog.f;
            c4.z = p.fogColor.z * (1.0f - fog.f) + c4.z * fog.f;
          }
        }
        b.colorHi[i] = c4;
      } else {
        // roughness -> Blinn exponent (shading.hpp:34-41), zero where clamped
        if (gEx != 0.0f && m.roughness >= 1e-6f) {
          const float e = 1.0f / m.roughness;
          if (e > 1.0f && e < 1.0e6f) G[gRoughness] += gEx * (-e * e);
        }
        // fog backward
        float gT = 0.0f;
        if (fog.on) {
          float gF;
          if (p.transparentBg) {
            gF = g.w;
          } else {
            G[gFogColor] += g.x * (1.0f - fog.f);
            G[gFogColor + 1] += g.y * (1.0f - fog.f);
            G[gFogColor + 2] += g.z * (1.0f - fog.f);
            gF = g.x * (out.x - p.fogColor.x) + g.y * (out.y - p.fogColor.y) + g.z * (out.z - p.fogColor.z);
          }
          G[gFogStart] += gF * fog.dStart;
          G[gFogEnd] += gF * fog.dEnd;
          gT += gF * fog.dz * dot(rd, p.camDir);
        }
        // secondary-ray origin O = P + ng eps (ng = N for a sphere)
        f3 gP = gO;
        gN = gN + gO * eps;
        const float gEps = dot(ng, gO);
        {
          // eps = K max(|Px|, |Py|, |Pz|, dirMax t)  (secondary_rays.hpp:38-46)
          const float K = 0x1.0fp-21f;
          const float dirMax = fmaxf(fabsf(rd.x), fmaxf(fabsf(rd.y), fabsf(rd.z)));
          const float ax = fabsf(P.x), ay = fabsf(P.y), az = fabsf(P.z), at = dirMax * t;
          const float mx = fmaxf(fmaxf(ax, ay), fmaxf(az, at));
          if (mx == ax) gP.x += gEps * K * copysignf(1.0f, P.x);
          else if (mx == ay) gP.y += gEps * K * copysignf(1.0f, P.y);
          else if (mx == az) gP.z += gEps * K * copysignf(1.0f, P.z);
          else gT += gEps * K * dirMax;
        }
        // N = sgn Ng / |Ng|, Ng = P - c, P = org + rd t(c, r)
        const f3 gNg = normalizeBack(nHat, ngLen, gN * sgn);
        gP = gP + gNg;
        f3 gCenter = neg(gNg);
        const float den = dot(Ng, rd);
        float gRad = 0.0f;
        if (den != 0.0f) {
          const float gtt = gT + dot(rd, gP);
          gCenter = gCenter + Ng * (gtt / den);
          gRad = gtt * rad / den;
        }
        addColor(b, sk, gC);
        addGeom(b, sk, gCenter, gRad);
        used = 1;
      }
    }
  }
  if (GRAD) {
    addGlobals<kGlobals>(b.gGlobal, G);
    warpCount(&b.stats[0], used);
  }
}

// Box average of the fogged hi-res colour with the non-finite guard
// (image_ops.cpp:9-35): the value the gamma derivative is taken at.
__global__ void k_adj_down(Params p, const float4* colorHi, float4* out, uint32_t nOut) {
  const uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= nOut) return;
  const int ox = int(o % uint32_t(p.outW)), oy = int(o / uint32_t(p.outW));
  float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  for (int dy = 0; dy < p.ss; ++dy)
    for (int dx = 0; dx < p.ss; ++dx) {
      const float4 c = colorHi[size_t(oy * p.ss + dy) * p.W + size_t(ox * p.ss + dx)];
      a[0] += isfinite(c.x) ? c.x : 0.0f;
      a[1] += isfinite(c.y) ? c.y : 0.0f;
      a[2] += isfinite(c.z) ? c.z : 0.0f;
      a[3] += isfinite(c.w) ? c.w : 0.0f;
    }
  const float inv = 1.0f / float(p.ss * p.ss);
  out[o] = make_float4(a[0] * inv, a[1] * inv, a[2] * inv, a[3] * inv);
}

// Workspace of a chunk of pixels: kAdjArrays arrays of queue and ray
// results, at most kAdjBytes of them.  They start on a block of the memory,
// or on a float4 where an arena cap leaves room for a few pixels only.
constexpr size_t kAdjAlign = 256, kAdjArrays = 6, kAdjBytes = size_t(256) << 20;
constexpr size_t adjHeader(size_t align) { return kAdjArrays * align; }
size_t adjAlign(size_t wsBytes, size_t pixBytes) {
  return wsBytes >= adjHeader(kAdjAlign) + 32 * pixBytes ? kAdjAlign : 16;
}

ubr_status adjointCheck(Context* c, const Scene& sc, const ubr_render_desc& d, const Params& p) {
  if (sc.primCount[kMesh] || sc.primCount[kRound] || sc.primCount[kCone])
    return setError(c, UBR_INVALID_ARGUMENT, "adjoint: only sphere scenes are differentiable");
  if (sc.primCount[kSphere] == 0) return setError(c, UBR_INVALID_ARGUMENT, "adjoint: scene has no spheres");
  if (p.maxIters > 1 && !sc.opaque)
    return setError(c, UBR_INVALID_ARGUMENT, "adjoint: needs one opaque layer (opaque spheres or transparency off)");
  if (d.env_lights > 0) return setError(c, UBR_INVALID_ARGUMENT, "adjoint: env dome lights are not differentiable");
  if (p.nLights > kAdjLights) return setError(c, UBR_INVALID_ARGUMENT, "adjoint: at most 4 lights");
  if (p.shadowsActive && p.shadowRays != p.nLights)
    return setError(c, UBR_INVALID_ARGUMENT, "adjoint: soft shadows are not differentiable");
  if (p.aoSamples > 0 && p.aoEnhanced && (p.aoBentNormal || p.aoMultibounce))
    return setError(c, UBR_INVALID_ARGUMENT, "adjoint: AO bent normal / multibounce are not differentiable");
  if (sc.principled) return setError(c, UBR_INVALID_ARGUMENT, "adjoint: principled materials are not differentiable");
  if (p.aaMode == 1 && (p.ss > 1 || d.aa_depth > 1))
    return setError(c, UBR_INVALID_ARGUMENT, "adjoint: adaptive AA is not differentiable (use the grid)");
  if ((d.ao_res_div < 0 ? p.ss : d.ao_res_div) > 1 && p.aoSamples > 0)
    return setError(c, UBR_INVALID_ARGUMENT, "adjoint: coarse-grid AO is not differentiable");
  return UBR_OK;
}

}  // namespace

ubr_status adjoint(Context* c, const Scene* sc, const ubr_render_desc& d, const float* dColor, ubr_grads& g) {
  ++c->call;
  Params p;
  std::vector<LightD> lights;
  ubr_status st = makeParams(c, d, p, lights);
  if (st != UBR_OK) return st;
  if ((st = adjointCheck(c, *sc, d, p)) != UBR_OK) return st;
  if (!dColor) return setError(c, UBR_INVALID_ARGUMENT, "adjoint: d_color is NULL");
  const bool dev = g.memory == UBR_MEMORY_DEVICE;
  const uint32_t npix = uint32_t(p.W) * uint32_t(p.H), nout = uint32_t(p.outW) * uint32_t(p.outH);
  const uint64_t nSph = sc->view.baseSph;
  const bool needFwd = !(std::fabs(p.gamma - 1.0f) <= 1.0e-4f);
  cudaStream_t s = c->stream;
  AdjBufs b{};
  float4* colorHi = needFwd ? scratchT<float4>(c, 61, npix, st) : nullptr;
  float4* outFwd = needFwd ? scratchT<float4>(c, 62, nout, st) : nullptr;
  LightD* dl = scratchT<LightD>(c, 63, lights.size() + 1, st);
  // global sums, then the counters
  double* gg = scratchT<double>(c, 64, kGlobals + 4, st);
  unsigned long long* stats = reinterpret_cast<unsigned long long*>(gg + kGlobals);
  const float4* dOut = reinterpret_cast<const float4*>(dColor);
  float4* dOutDev = nullptr;
  if (!dev) dOutDev = scratchT<float4>(c, 66, nout, st);
  // per-sphere accumulators: the caller's device arrays, or scratch copied back
  float* gCol = g.sphere_color;
  float* gCen = g.sphere_center;
  float* gRad = g.sphere_radius;
  if (!dev) {
    gCol = g.sphere_color ? scratchT<float>(c, 67, 3 * nSph, st) : nullptr;
    gCen = g.sphere_center ? scratchT<float>(c, 68, 3 * nSph, st) : nullptr;
    gRad = g.sphere_radius ? scratchT<float>(c, 69, nSph, st) : nullptr;
  }
  if (st != UBR_OK) return st;
  // one block: the primary hits, the packed gradient sums and a chunk's
  // workspace; where an arena cap leaves less or it does not fit, the hits
  // alone and whatever workspace the context has, with the sums in it if they
  // leave at least as much for the chunk
  const size_t pixBytes = 4 + 48 + size_t(p.aoSamples) * 8 + size_t(p.nLights);
  const size_t hitBytes = (size_t(npix) * sizeof(float2) + kAdjAlign) / kAdjAlign * kAdjAlign;
  // the caller's arrays get the packed sums spread over them at the end where
  // the device holds them whole; any others are cleared here and added to (the
  // clearing finds arrays it cannot write, with an error)
  DeviceMemory holds(c->device);
  const bool spread = !dev || ((!gCol || holds(gCol, 3 * nSph * sizeof(float))) &&
                               (!gCen || holds(gCen, 3 * nSph * sizeof(float))) &&
                               (!gRad || holds(gRad, nSph * sizeof(float))));
  const size_t accBytes = spread && (gCol || gCen || gRad) ? size_t(nSph) * 32 : 0;
  const size_t accPad = (accBytes + kAdjAlign - 1) / kAdjAlign * kAdjAlign;
  size_t wsBytes = adjHeader(kAdjAlign) + std::min<size_t>(size_t(npix) * pixBytes, std::max(kAdjBytes, pixBytes));
  void* ws = nullptr;
  void* block = nullptr;
  const size_t all = hitBytes + accPad + wsBytes;
  const size_t own = size_t(kAdjointSlot) < c->scratch.size() ? c->scratch[kAdjointSlot].bytes : 0;
  if ((own >= all || arenaHolds(c, all - own)) && scratchGet(c, kAdjointSlot, all, &block, c->arenaCap == 0) == UBR_OK) {
    ws = static_cast<char*>(block) + hitBytes + accPad;
    if (accBytes) b.acc = reinterpret_cast<float4*>(static_cast<char*>(block) + hitBytes);
  } else {
    cudaGetLastError();
    if ((st = scratchGet(c, 60, size_t(npix) * sizeof(float2), &block)) != UBR_OK) return st;
    size_t got = accPad + wsBytes;
    const size_t least = adjHeader(16) + pixBytes;
    if ((st = workspaceGet(c, kAdjointSlot, least, nullptr, 0, &ws, &got)) != UBR_OK) return st;
    if (accBytes && got >= accPad + std::max(least, accPad)) {
      b.acc = reinterpret_cast<float4*>(ws);
      ws = static_cast<char*>(ws) + accPad;
      got -= accPad;
    }
    wsBytes = std::min(wsBytes, got);
  }
  float2* hit = static_cast<float2*>(block);
  cudaEventRecord(c->ev[0], s);
  if (!dev) {
    UBR_CUDA(c, cudaMemcpyAsync(dOutDev, dColor, size_t(nout) * 16, cudaMemcpyHostToDevice, s));
    dOut = dOutDev;
  }
  if (!lights.empty())
    UBR_CUDA(c, cudaMemcpyAsync(dl, lights.data(), lights.size() * sizeof(LightD), cudaMemcpyHostToDevice, s));
  UBR_CUDA(c, cudaMemsetAsync(gg, 0, kGlobals * sizeof(double) + 4 * sizeof(unsigned long long), s));
  if (b.acc) {
    UBR_CUDA(c, cudaMemsetAsync(b.acc, 0, accBytes, s));
  } else {
    if (gCol) UBR_CUDA(c, cudaMemsetAsync(gCol, 0, 3 * nSph * sizeof(float), s));
    if (gCen) UBR_CUDA(c, cudaMemsetAsync(gCen, 0, 3 * nSph * sizeof(float), s));
    if (gRad) UBR_CUDA(c, cudaMemsetAsync(gRad, 0, nSph * sizeof(float), s));
  }
  b.hit = hit;
  b.dOut = dOut;
  b.outFwd = outFwd;
  b.colorHi = colorHi;
  b.lights = dl;
  b.gColor = gCol;
  b.gCenter = gCen;
  b.gRadius = gRad;
  b.gGlobal = gg;
  b.stats = stats;
  b.flags = g.flags;
  const int TB = 128;
  const uint32_t grid = (npix + TB - 1) / TB;
  cudaEventRecord(c->ev[2], s);
  k_adj_primary<<<grid, TB, 0, s>>>(p, travOf(sc->view), hit, npix, stats);
  // pixels per chunk: what the workspace's queue and ray results hold
  const uint32_t S = uint32_t(p.aoSamples), nL = uint32_t(p.nLights);
  const size_t align = adjAlign(wsBytes, pixBytes);
  char* at = static_cast<char*>(ws);
  auto take = [&](size_t n) {
    char* q = at;
    at += (n + align - 1) / align * align;
    return q;
  };
  const uint32_t chunk = uint32_t(std::min<size_t>(npix, (wsBytes - adjHeader(align)) / pixBytes));
  AdjRays r{};
  r.count = reinterpret_cast<uint32_t*>(stats + 3);  // cleared with the counters
  bool cleared = true;
  r.pix = reinterpret_cast<uint32_t*>(take(size_t(chunk) * 4));
  r.a = reinterpret_cast<float4*>(take(size_t(chunk) * 16));
  r.b = reinterpret_cast<float4*>(take(size_t(chunk) * 16));
  r.c = reinterpret_cast<float4*>(take(size_t(chunk) * 16));
  r.ao = reinterpret_cast<float2*>(take(size_t(chunk) * S * 8));
  r.shadow = reinterpret_cast<uint8_t*>(take(size_t(chunk) * nL));
  const uint64_t raysPer = uint64_t(S) + (p.shadowsActive ? nL : 0u);
  auto traceChunk = [&](uint32_t i0, uint32_t n, bool all) -> ubr_status {
    if (!cleared) UBR_CUDA(c, cudaMemsetAsync(r.count, 0, sizeof(uint32_t), s));
    cleared = false;
    const uint32_t gs = (n + TB - 1) / TB;
    if (needFwd) k_adj_surface<false><<<gs, TB, 0, s>>>(p, sc->view, b, r, i0, n, all ? 1 : 0);
    else k_adj_surface<true><<<gs, TB, 0, s>>>(p, sc->view, b, r, i0, n, all ? 1 : 0);
    const uint32_t g = uint32_t((uint64_t(n) * raysPer + TB - 1) / TB);
    if (g > 0) {
      if (p.aoEnhanced) k_adj_rays<true><<<g, TB, 0, s>>>(p, sc->view, b, r);
      else k_adj_rays<false><<<g, TB, 0, s>>>(p, sc->view, b, r);
    }
    return UBR_OK;
  };
  bool traced = false;  // the only chunk's rays are traced already
  if (needFwd) {
    k_adj_background<false><<<grid, TB, 0, s>>>(p, b, npix);
    for (uint32_t i0 = 0; i0 < npix; i0 += chunk) {
      const uint32_t n = std::min(chunk, npix - i0);
      if ((st = traceChunk(i0, n, true)) != UBR_OK) return st;
      k_adj_shade<false><<<(n + TB - 1) / TB, TB, 0, s>>>(p, sc->view, b, r);
    }
    traced = chunk >= npix;
    k_adj_down<<<(nout + 255) / 256, 256, 0, s>>>(p, colorHi, outFwd, nout);
  }
  if (needFwd) k_adj_background<true><<<grid, TB, 0, s>>>(p, b, npix);
  for (uint32_t i0 = 0; i0 < npix; i0 += chunk) {
    const uint32_t n = std::min(chunk, npix - i0);
    if (!traced && (st = traceChunk(i0, n, false)) != UBR_OK) return st;
    k_adj_shade<true><<<(n + TB - 1) / TB, TB, 0, s>>>(p, sc->view, b, r);
  }
  if (b.acc) k_adj_unpack<<<uint32_t((nSph + 255) / 256), 256, 0, s>>>(uint32_t(nSph), b);
  UBR_CUDA(c, cudaGetLastError());
  cudaEventRecord(c->ev[3], s);
  const cudaMemcpyKind back = cudaMemcpyDeviceToHost;
  if (!dev) {
    if (gCol) UBR_CUDA(c, cudaMemcpyAsync(g.sphere_color, gCol, 3 * nSph * sizeof(float), back, s));
    if (gCen) UBR_CUDA(c, cudaMemcpyAsync(g.sphere_center, gCen, 3 * nSph * sizeof(float), back, s));
    if (gRad) UBR_CUDA(c, cudaMemcpyAsync(g.sphere_radius, gRad, nSph * sizeof(float), back, s));
  }
  double* hg = reinterpret_cast<double*>(static_cast<char*>(c->pinned) + 2048);
  const unsigned long long* hs = reinterpret_cast<const unsigned long long*>(hg + kGlobals);
  UBR_CUDA(c, cudaMemcpyAsync(hg, gg, kGlobals * sizeof(double) + 4 * sizeof(unsigned long long), back, s));
  UBR_CUDA(c, cudaStreamSynchronize(s));
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, c->ev[2], c->ev[3]);
  // fill the host struct; light vectors: L = normalize(-direction),
  // colour x intensity (buildSceneLights, embree_renderer.cpp:436-458)
  for (int k = 0; k < 9; ++k) g.material[k] = float(hg[k]);
  for (int k = 0; k < 3; ++k) {
    g.ambient_color[k] = float(hg[gAmbColor + k]);
    g.background[k] = float(hg[gBg + k]);
    g.fog_color[k] = float(hg[gFogColor + k]);
  }
  g.fog_start = float(hg[gFogStart]);
  g.fog_end = float(hg[gFogEnd]);
  g.ao_distance = float(hg[gAoDistance]);
  g.ao_intensity = float(hg[gAoIntensity]);
  g.specular_scale = float(hg[gSpecScale]);
  for (int l = 0; l < kAdjLights; ++l) {
    for (int k = 0; k < 3; ++k) g.light_direction[l][k] = g.light_color[l][k] = 0.0f;
    g.light_intensity[l] = 0.0f;
    if (l >= int(d.light_count)) continue;
    const ubr_light& ul = d.lights[l];
    const double dir[3] = {ul.direction[0], ul.direction[1], ul.direction[2]};
    const double len = std::sqrt(dir[0] * dir[0] + dir[1] * dir[1] + dir[2] * dir[2]);
    const double gL[3] = {hg[gLightL + 3 * l], hg[gLightL + 3 * l + 1], hg[gLightL + 3 * l + 2]};
    if (len > 0.0) {
      const double Lv[3] = {-dir[0] / len, -dir[1] / len, -dir[2] / len};
      const double lg = Lv[0] * gL[0] + Lv[1] * gL[1] + Lv[2] * gL[2];
      for (int k = 0; k < 3; ++k) g.light_direction[l][k] = float(-(gL[k] - Lv[k] * lg) / len);
    }
    double gi = 0.0;
    for (int k = 0; k < 3; ++k) {
      const double gc = hg[gLightC + 3 * l + k];
      g.light_color[l][k] = float(gc * ul.intensity);
      gi += gc * ul.color[k];
    }
    g.light_intensity[l] = float(gi);
  }
  g.samples = hs[0];
  g.rays = hs[1];
  g.adjoint_ms = ms;
  return UBR_OK;
}

}  // namespace ubr
