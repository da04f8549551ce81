// Wavefront BDPT kernels for GB300 (sm_103a).
//
// One frame of the reference's streaming BDPT (src/cudaRTBDPTStream.cu:816-951)
// runs as a fixed sequence of launches with no host round trip:
//
//   light pass                  pt_genLightPathQueue_kernel + pt_traceLight_kernel
//                               loop with stable compaction (:875-906)
//   camera                      pt_genPathQueue_kernel (:619-640)
//   per bounce launch d (k_walk, then k_shade):
//     shadow (any hit)          the visibility test of GetLightFromRandLightVertices
//                               (:665-700) for bounce d-1's connections
//     trace  (closest hit)      the TracePrimitive half of pt_traceSample_kernel,
//                               for the walks launch d-1 carried and wave d
//     shade                     the rest of pt_traceSample_kernel (:365-543);
//                               survivors are appended to the other wave
//                               buffer with one atomic per warp (replaces
//                               thrust::remove_if, :930), connection requests
//                               likewise (replaces thrust::copy_if, :934)
//   tail (k_tail)               the remaining bounces of the paths still alive,
//                               one lane per path, and the last launch's carried walks
//   fold (k_fold)               the accumulate of pt_connectEyeLightPath_kernel
//                               (:703-723) and of the path's end, in bounce order
//   apply                       pt_applyPathQueueResult_kernel (:741-778)
//
// Queue lengths live in device memory (DevCounters) and every kernel runs a
// grid-stride loop or a persistent fetch loop over them, so the host never
// waits on a count.
#include <algorithm>
#include <atomic>
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdlib>

#include "launch.h"
#include "ordered.cuh"
#include "shade.cuh"
#include "texture.cuh"
#include "trace.cuh"

namespace gbpt {

using gb::f3;
using gb::mk;

namespace {

constexpr int kBlock = 256;

__device__ __forceinline__ f3 ld3(float4 v) { return mk(v.x, v.y, v.z); }
__device__ __forceinline__ float4 st4(f3 v, float w) { return make_float4(v.x, v.y, v.z, w); }
__device__ __forceinline__ float4 st4u(f3 v, uint32_t w) { return make_float4(v.x, v.y, v.z, __uint_as_float(w)); }
__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Lanes of a warp that take paths when n of them meet `warps` resident warps:
// a small frame's paths are spread over a quarter of the warps instead of
// filling the first few, so that a warp waits for the longest of fewer walks
// and more warps hide each other's latency.  Cornell 64x64 pass: full warps
// 0.224 ms, spread over all warps 0.194, half 0.197, a quarter 0.199, an eighth
// 0.206; at 256x256 all warps cost 4 %, a quarter nothing.
__device__ __forceinline__ uint32_t path_lanes(uint32_t n, uint32_t warps) {
  const uint32_t q = max(warps / 4u, 1u), w = max((n + q - 1u) / q, 1u);
  return w >= 32u ? 0xffffffffu : (1u << w) - 1u;
}

struct Mat {
  f3 diff, emis;
  float trans, spec, metal, rough;
  int32_t texD, texE;  // diffuseTexId, emissiveTexId (-1: none)
};
__device__ __forceinline__ Mat load_mat(const DevScene& S, uint32_t id) {
  float4 a = __ldg(S.mats + 3 * (size_t)id), b = __ldg(S.mats + 3 * (size_t)id + 1),
         c = __ldg(S.mats + 3 * (size_t)id + 2);
  Mat m;
  m.diff = ld3(a);
  m.trans = a.w;
  m.emis = ld3(b);
  m.spec = b.w;
  m.metal = c.x;
  m.rough = c.y;
  m.texD = __float_as_int(c.z);
  m.texE = __float_as_int(c.w);
  return m;
}

// The texture half of GetMaterialColors (src/cudaRTCommon.cu:369-406) at the
// barycentrics (w, u, v) of triangle `tri`: uv = ((uv0*w) + (uv1*u)) + uv2*v
// (the float2 operators of the reference's kernels, e.g.
// src/cudaRTBDPTStream.cu:379-382); a diffuse texture gives the diffuse
// colour and scales the transparency by its alpha, an emissive texture gives
// the emissive colour.
__device__ __forceinline__ void apply_textures(const DevScene& S, Mat& m, uint32_t tri, float w, float u, float v) {
  const float2* q = S.uvs + 3 * (size_t)tri;
  const float2 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
  const float tu = (a.x * w + b.x * u) + c.x * v;
  const float tv = (a.y * w + b.y * u) + c.y * v;
  if (m.texD >= 0) {
    const float4 t = tex_bilinear(S.texels, __ldg(S.texInfo + m.texD), tu, tv);
    m.diff = mk(t.x, t.y, t.z);
    m.trans = t.w * m.trans;
  }
  if (m.texE >= 0) {
    const float4 t = tex_bilinear(S.texels, __ldg(S.texInfo + m.texE), tu, tv);
    m.emis = mk(t.x, t.y, t.z);
  }
}
__device__ __forceinline__ Mat load_mat_at(const DevScene& S, uint32_t matId, uint32_t tri, float w, float u,
                                           float v) {
  Mat m = load_mat(S, matId);
  if (m.texD >= 0 || m.texE >= 0) apply_textures(S, m, tri, w, u, v);
  return m;
}

// interpolated normal, position and material id of a triangle at (w,u,v):
// ((x0*w) + (x1*u)) + (x2*v) as the reference's float3 operators.
struct Surf {
  f3 norm, pos;
  uint32_t mat;
};
__device__ __forceinline__ Surf load_surf(const DevScene& S, uint32_t tri, float w, float u, float v, bool wantPos) {
  const float4* r = S.shade + 5 * (size_t)tri;
  float4 a = __ldg(r), b = __ldg(r + 1), c = __ldg(r + 2), d = __ldg(r + 3);
  Surf s;
  s.norm = (ld3(a) * w + ld3(b) * u) + ld3(c) * v;
  s.mat = __float_as_uint(d.w);
  if (wantPos) {
    float4 e = __ldg(r + 4);
    s.pos = (mk(a.w, b.w, c.w) * w + ld3(d) * u) + ld3(e) * v;
  } else {
    s.pos = mk(0.f, 0.f, 0.f);
  }
  return s;
}

enum : uint32_t { kTypeEye = 0, kTypeDiff = 1, kTypeSpec = 2, kTypeLight = 3 };

// The bounce decision shared by eye and light paths (reflect / transmit /
// diffuse, src/cudaRTBDPTStream.cu:400-493 and :223-323).
// With wantPdf, also the sampling density of the filter-only variant
// (src/cudaRTBDPTStreamBilat.cu:515-518, :560, :575, :599): D*NoH/(4 VoH)
// times the probability of the branch taken.
struct Bounce {
  f3 nl, nOrig, nDir, lmt, F;
  uint32_t type;
  float pdf;
};
//
// ptTir: the unidirectional variant reflects on total internal reflection
// (src/cudaRTPTStream.cu:153-160: cos2t < 0 sets reflProb = 1); the BDPT
// variants compute the refracted direction regardless (the test is commented
// out there).  The refracted direction stays zero when it is not computed
// (uninitialised in the reference).
__device__ __forceinline__ void sample_bounce(f3 orig, f3 dir, float dist, f3 norm, const Mat& m, const float* u,
                                              bool specPush, bool wantPdf, bool ptTir, Bounce& B) {
  using namespace gb;
  B.nl = dot(norm, dir) < 0.f ? norm : -1.f * norm;
  const f3 nl = B.nl;
  f3 hDir = ggx_sample(u[0], u[1], m.rough, nl);
  f3 ndir = -1.f * dir;
  float voH = dot(ndir, hDir);
  f3 f0 = vlerp(kF0Spec * mk(m.spec, m.spec, m.spec), m.diff, m.metal);
  f3 F = f_schlick(f0, voH);
  B.F = F;
  B.pdf = 1.f;
  if (wantPdf) {
    const float NoH0 = dot(nl, hDir);
    B.pdf = (d_ggx(m.rough, NoH0) * NoH0) / (4.f * voH);
  }
  float reflProb = lerp(length(F), 1.0f, m.metal);
  float refrProb = m.trans;
  f3 reflDir = mk(0.f, 0.f, 0.f), refrDir = reflDir;
  if (refrProb > 0.f) {
    bool into = dot(nl, norm) > 0.f;
    float nt = m.spec * 0.8f + 1.f;
    float nnt = into ? 1.0f / nt : nt / 1.0f;
    float ddn = dot(hDir, dir);
    float cos2t = 1.f - (nnt * nnt) * (1.f - ddn * ddn);
    if (ptTir && cos2t < 0.f)
      reflProb = 1.0f;
    else
      refrDir = normalize(dir * nnt - hDir * (ddn * nnt + sqrtf(cos2t)));
  }
  if (reflProb > 0.f) {
    reflDir = normalize(dir - (hDir * 2.f) * dot(hDir, dir));
    if (dot(reflDir, nl) < 0.f) reflProb = 0.f;
  }
  if (prob_rand(reflProb, u[2])) {
    B.nOrig = orig + (dist - kBias) * dir;
    if (specPush) B.nOrig = B.nOrig + reflDir * kBias;
    B.nDir = reflDir;
    float VoH = dot(ndir, hDir), NoV = dot(nl, ndir), NoH = dot(nl, hDir), NoL = dot(nl, reflDir);
    float G = vis_smith(m.rough, NoV, NoL);
    B.lmt = ((F * G) * VoH) / ((NoV * NoH) * reflProb);
    B.type = kTypeSpec;
    B.pdf = B.pdf * reflProb;
  } else if (prob_rand(refrProb, u[3])) {
    B.nOrig = (orig + (dist + kBias) * dir) + refrDir * kBias;
    B.nDir = refrDir;
    float cosine = dot(-1.f * nl, refrDir);
    B.lmt = (cosine * m.diff) / (refrProb * (1.f - reflProb));
    B.type = kTypeSpec;
    B.pdf = B.pdf * (refrProb * (1.f - reflProb));
  } else {
    f3 dd = cos_dir(u[4], u[5], nl);
    B.nOrig = (orig + dist * dir) + dd * kBias;
    B.nDir = dd;
    B.lmt = (kPi * (m.diff * kInvPi)) / ((1.f - refrProb) * (1.f - reflProb));
    B.type = kTypeDiff;
    B.pdf = B.pdf * (((1.f - refrProb) * (1.f - reflProb)) * dot(dd, nl));
  }
}

// light-vertex cache record: 6 float4
//   {pos, specular} {norm, metallic} {irrad, roughness} {irradDir, 0} {diff, 0} {emissive, 0}
struct LV {
  f3 pos, norm, irrad, irradDir, diff, emis;
  float spec, metal, rough;
};
__device__ __forceinline__ void store_lv(float4* c, const LV& v) {
  c[0] = st4(v.pos, v.spec);
  c[1] = st4(v.norm, v.metal);
  c[2] = st4(v.irrad, v.rough);
  c[3] = st4(v.irradDir, 0.f);
  c[4] = st4(v.diff, 0.f);
  c[5] = st4(v.emis, 0.f);
}
__device__ __forceinline__ LV load_lv(const float4* c) {
  LV v;
  float4 a = c[0], b = c[1], d = c[2], e = c[3], f = c[4], g = c[5];
  v.pos = ld3(a);
  v.spec = a.w;
  v.norm = ld3(b);
  v.metal = b.w;
  v.irrad = ld3(d);
  v.rough = d.w;
  v.irradDir = ld3(e);
  v.diff = ld3(f);
  v.emis = ld3(g);
  return v;
}

// ---------------------------------------------------------------------------
// Light pass: a thread per light subpath in one CTA, or eight in a cluster of
// eight CTAs (ordered walk, up to 128 subpaths).  Cache slots are handed
// out exactly as the reference's stable remove_if does: a surviving path's
// position in the stream equals the number of surviving paths with a lower
// index, i.e. an exclusive scan of the "alive" flags.
//
// kLanes == 8: eight lanes a path (coop_walk) in a cluster of kLightBlocks
// blocks, whose counts go through distributed shared memory.  The pass is a
// chain of at most lightDepth + 1 walks whatever the number of paths, so only
// latency counts: hall 0.62 ms with a lane a path in one block, 0.47 with eight
// lanes a path in one block, whose 32 warps share four schedulers.
constexpr uint32_t kLightBlocks = 8;
template <int kLanes, bool kOrdered>
__global__ void __launch_bounds__(1024) k_light(DevScene S, FrameArgs a, float4* cache, uint32_t cacheCap,
                                                DevCounters* ctr) {
  using namespace gb;
  __shared__ uint32_t warpCnt[32], openN, blockCnt[2][kLightBlocks];
  extern __shared__ float4 capMem[];
  const uint32_t x = (blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
  const bool first = threadIdx.x % kLanes == 0;  // the path's lane that writes
  const uint32_t NL = a.lightPaths;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nWarps = (blockDim.x + 31) >> 5;
  bool alive = (x < NL) && (S.lightN > 0);
  f3 orig = mk(0.f, 0.f, 0.f), dir = orig, outMul = mk(1.f, 1.f, 1.f), sample = orig;
  uint32_t depth = 0;
  if (alive) {
    float u[8];
    draw8(a.key0, a.key1, x, a.frame, kLightGen, 0, 0, u);
    uint32_t id = (uint32_t)(u[0] * (float)S.lightN);
    if (id >= S.lightN) id = S.lightN - 1;
    float lw = u[1], lu = u[2];
    if (lw + lu > 1.0f) {
      lw = 1.f - lw;
      lu = 1.f - lu;
    }
    float lvv = 1.f - lw - lu;
    Surf sf = load_surf(S, S.lightTri[id], lw, lu, lvv, true);
    Mat m = load_mat_at(S, sf.mat, S.lightTri[id], lw, lu, lvv);
    dir = cos_dir(u[3], u[4], sf.norm);
    orig = sf.pos + kBias * sf.norm;
    sample = m.emis;
    LV v;
    v.pos = sf.pos;
    v.norm = sf.norm;
    v.irrad = m.emis;
    v.irradDir = mk(0.f, 0.f, 0.f);
    v.diff = m.diff;
    v.emis = m.emis;
    v.spec = m.spec;
    v.metal = m.metal;
    v.rough = m.rough;
    if (first) store_lv(cache + 6 * (size_t)x, v);
  }
  uint32_t size = (S.lightN > 0) ? NL : 0;
  // the cluster's blocks must all have started before one of them stores to
  // another's shared memory: co-scheduling alone does not promise it
  if constexpr (kLanes > 1)
    cooperative_groups::this_cluster().sync();
  else
    __syncthreads();
  for (uint32_t round = 0;; round++) {
    uint32_t bal = __ballot_sync(0xffffffffu, alive && first);
    if (lane == 0) warpCnt[warp] = __popc(bal);
    if (threadIdx.x == 0) openN = 0;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (uint32_t w = 0; w < nWarps; w++) {
      uint32_t c = warpCnt[w];
      if (w < warp) before += c;
      total += c;
    }
    if constexpr (kLanes > 1) {  // the other blocks' counts (two sets: one is read while the next is written)
      auto cluster = cooperative_groups::this_cluster();
      uint32_t* cnt = blockCnt[round & 1u];
      if (threadIdx.x < kLightBlocks) cluster.map_shared_rank(cnt, threadIdx.x)[blockIdx.x] = total;
      cluster.sync();
      total = 0;
      for (uint32_t k = 0; k < kLightBlocks; k++) {
        if (k < blockIdx.x) before += cnt[k];
        total += cnt[k];
      }
    } else {
      __syncthreads();
    }
    if (total == 0) break;
    TraceHit h;
    bool hit = false;
    if constexpr (kLanes > 1) {  // every lane of the block takes part
      OrdWalk w;
      uint2 stack[kOrdStack];
      w.any = false;
      w.eps = kBias;
      w.init(S, orig, dir, kInf);
      coop_walk(S, w, stack, alive);
      hit = alive && w.hit();
      h.t = w.minT, h.tri = w.best, h.u = w.bu, h.v = w.bv;
      // walks past the pop bound, one after another by the block
      CapShared& c = *reinterpret_cast<CapShared*>(capMem);
      const bool open = alive && w.capped();
      uint32_t turn = open && first ? atomicAdd(&openN, 1u) : 0u;
      turn = __shfl_sync(0xffffffffu, turn, (int)(lane & ~(uint32_t)(kLanes - 1)));
      __syncthreads();
      const uint32_t n = openN;
      for (uint32_t k = 0; k < n; k++) {
        __syncthreads();
        if (open && first && turn == k) {
          c.hit[0] = st4(orig, 0.f);
          c.hit[1] = st4(dir, 0.f);
        }
        __syncthreads();
        const f3 o = ld3(c.hit[0]), d = ld3(c.hit[1]);
        resolve_capped(S, c, o, d, kInf, kBias, false);
        __syncthreads();
        if (open && turn == k) {
          const float4 q = c.answer;
          hit = c.found != 0u;
          h.t = q.x, h.tri = __float_as_uint(q.y), h.u = q.z, h.v = q.w;
        }
      }
    }
    if (alive) {
      uint32_t slot = size + before + __popc(bal & ((1u << (lane & ~(uint32_t)(kLanes - 1))) - 1u));
      if (slot >= cacheCap) {
        atomicOr(&ctr->errFlags, 1u);
        alive = false;
      } else {
        float4* cs = cache + 6 * (size_t)slot;
        if constexpr (kLanes == 1) {
          uint32_t nn = 0, nt = 0;
          if constexpr (kOrdered)
            hit = trace_ord(S, orig, dir, kInf, kBias, h);
          else
            hit = trace_ref<false, false>(S, orig, dir, kInf, kBias, false, h, nn, nt);
        }
        if (!hit) {
          const float4* home = cache + 6 * (size_t)x;  // :358-362
          if (first)
            for (int k = 0; k < 6; k++) cs[k] = home[k];
          alive = false;
        } else {
          float u[8];
          draw8(a.key0, a.key1, x, a.frame, kLightBounce, depth, 0, u);
          float hw = 1.f - h.u - h.v;
          Surf sf = load_surf(S, h.tri, hw, h.u, h.v, true);
          Mat m = load_mat_at(S, sf.mat, h.tri, hw, h.u, h.v);
          Bounce B;
          sample_bounce(orig, dir, h.t, sf.norm, m, u, false, false, false, B);
          LV v;
          v.irrad = (B.type != kTypeDiff) ? mk(0.f, 0.f, 0.f) : sample;
          v.irradDir = -1.f * dir;
          v.norm = (dot(B.nDir, B.nl) < 0.f) ? -1.f * B.nl : B.nl;
          v.pos = sf.pos;
          v.diff = m.diff;
          v.emis = m.emis;
          v.spec = m.spec;
          v.metal = m.metal;
          v.rough = m.rough;
          if (first) store_lv(cs, v);
          sample = m.emis + vmul(sample, B.lmt);
          float contrib = length(outMul) * length(B.lmt);
          if (length(m.emis) > 0.f) contrib = 0.f;
          if (u[6] > contrib || depth + 1 >= a.lightDepth) {
            alive = false;
          } else {
            outMul = vmul(outMul, B.lmt);
            dir = B.nDir;
            orig = B.nOrig;
            depth++;
          }
        }
      }
    }
    size += total;
    __syncthreads();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) ctr->cacheSize[a.cacheSel] = size;
}

// ---------------------------------------------------------------------------
// Camera rays, one per pixel (pt_genPathQueue_kernel, :619-640), for the
// band's pixels b.base .. b.base + b.count - 1; a ray's wave index is its
// index inside the band.
// Wave item i of a whole-image wavefront -> its pixel: 4x8-pixel tiles, one
// warp's 32 camera rays per tile, tiles in row-major order, then the pixels
// right of and below the whole tiles in row-major order (a bijection for any
// width and height).  Camera rays of a compact tile walk more of the same
// nodes than a 32-pixel row: hall 1280x720 188.0 -> 190.1 Mpaths/s (8x4
// tiles 189.2, 16x2 187.8), interior even, Cornell 256x256 190.1 -> 187.2
// (cheap walks: its first-bounce slot writes in 4-pixel runs show).  Results
// do not depend on it: every path's random numbers and its slot follow from
// its pixel.
__device__ __forceinline__ uint32_t tiled_pixel(uint32_t i, uint32_t w, uint32_t h) {
  constexpr uint32_t TW = 4u, TH = 8u;
  const uint32_t tx = w / TW, ty = h / TH, nFull = tx * ty * TW * TH;
  if (i < nFull) {
    const uint32_t t = i / (TW * TH), k = i % (TW * TH);
    return ((t / tx) * TH + k / TW) * w + (t % tx) * TW + k % TW;
  }
  uint32_t j = i - nFull;
  const uint32_t rw = w - tx * TW, rightN = rw * ty * TH;
  if (j < rightN) return (j / rw) * w + tx * TW + j % rw;
  j -= rightN;
  return (ty * TH + j / w) * w + j % w;
}

__global__ void k_camera(FrameArgs a, RenderBuffers b) {
  using namespace gb;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    b.ctr->wave[0] = b.count;
    b.ctr->paths = b.count;
    b.ctr->fetchT = 0;
    b.ctr->carryN[0] = b.ctr->carryN[1] = b.ctr->carryN[2] = 0;
    b.ctr->fetchTail = 0;
    b.ctr->openN = b.ctr->openOver = b.ctr->checkN[0] = b.ctr->checkN[1] = b.ctr->fixN = 0;
    b.ctr->tailAt = 0xFFFFFFFFu;
  }
  if (i >= b.count) return;
  // local pixel (the band's range in row-major order when the frame is split)
  const uint32_t p = b.count == a.width * a.height ? tiled_pixel(i, a.width, a.height) : b.base + i;
  // pixel of the full image: its coordinates place the ray and its id keys
  // every random number of the path, so a window renders as in the full image
  const uint32_t x = a.winX0 + p % a.width, y = a.winY0 + p / a.width;
  const uint32_t gp = y * a.fullW + x;
  float u[4];
  draw4(a.key0, a.key1, gp, a.frame, kCamera, 0, 0, 0, u);
  const float W = a.W, H = a.H, th = a.tanHalf;
  float cu = ((((2.f * ((float)x + 0.5f)) / W) - 1.f) * th * W) / H;
  float cv = (((2.f * ((float)y + 0.5f)) / H) - 1.f) * th;
  float au = cu + ((u[0] - 0.5f) / H) * th;
  float av = cv + ((u[1] - 0.5f) / H) * th;
  f3 R = mk(a.camRight[0], a.camRight[1], a.camRight[2]);
  f3 U = mk(a.camUp[0], a.camUp[1], a.camUp[2]);
  f3 D = mk(a.camDir[0], a.camDir[1], a.camDir[2]);
  f3 dir = normalize((R * au + U * av) + D);
  Wave w = b.wave[0];
  w.o[i] = make_float4(a.camPos[0], a.camPos[1], a.camPos[2], __uint_as_float(p));
  w.d[i] = st4u(dir, gp);
  w.thr[i] = make_float4(1.f, 1.f, 1.f, 1.f);  // .w: path potential (filter-only mode)
  w.smp[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  b.res[p] = make_float4(0.f, 0.f, 0.f, __uint_as_float(0u));
  b.slotPix[p] = p;
  b.slotSmp[p] = 0;
  if (a.gbuffer) {
    b.gbuf[3 * (size_t)p] = make_float4(0.f, 0.f, 0.f, 0.f);
    b.gbuf[3 * (size_t)p + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
    b.gbuf[3 * (size_t)p + 2] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (a.bilat) b.dsm[p] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// Direct-light sample of a bounce-0 connection that reached its light vertex
// (pt_connectEyeLightPath_kernel, src/cudaRTBDPTStreamBilat.cu:905-913):
// (direct + L) / 5 when any channel is positive, else L / 4.
__device__ __forceinline__ void direct_connect(float4* dsm, uint32_t slot, float4 C) {
  using namespace gb;
  const float4 q = dsm[slot];
  const f3 L = ld3(C);
  const f3 d = (q.x > 0.f || q.y > 0.f || q.z > 0.f) ? (ld3(q) + L) / 5.f : L / 4.f;
  dsm[slot] = st4(d, q.w);
}

__device__ __forceinline__ void warp_add_u64(unsigned long long* dst, uint32_t v) {
  uint32_t s = v;
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(dst, (unsigned long long)s);
}

// ---------------------------------------------------------------------------
// One persistent kernel walks the BVH for the extension rays of bounce d
// (closest hit) and the shadow rays of bounce d-1 (any hit): the two sets
// are independent, so running them in one launch removes one kernel tail per
// bounce.  A lane takes a new ray as soon as its ray is finished (refill when
// at least kRefill lanes of the warp are idle), so warps stay full while rays
// last.  Shadow rays are handed out first: they cannot be carried to the next
// launch (a path's connection contributions are summed in bounce order), so
// the long ones must start early; then the walks the previous launch carried,
// then the extension rays (hall 1280x720: 181.4 -> 187.9 Mpaths/s against
// extension rays first; interior 169.0 -> 168.2).
// Every ray still reaches leaves in TracePrimitive's order, so per-ray
// results do not depend on this scheduling.  The any-hit walk stops at the
// first hit closer than maxDist: that is exactly when the reference's
// closest-hit walk with the same maxDist would report a hit.
// 4 resident CTAs per SM (64 registers, no spill) for both orders.  The
// reference order measured 1-2% faster at 5 (48 registers) than at 4 or 6
// before walks were carried and before 16-step batches; now (hall / interior
// / Cornell / hall adaptive, Mpaths/s) 3: 173.2 / 160.6 / 204.5 / 137.8, 4:
// 198.7 / 179.9 / 198.5 / 153.8, 5: 196.0 / 178.5 / 190.4 / 151.6, 6: 180.9 /
// 168.0 / 187.3 / 141.1.
// walk steps per refill check (measured in Mpaths/s on interior / hall /
// Cornell): reference order before carrying 1: 148.4 / 167.6 / 140.7, 2:
// 152.2 / 171.7 / 144.5, 4: 154.9 / 174.3 / 143.1, 6: 156.0 / 176.2 / 141.9,
// 8: 155.5 / 176.6 / 142.7; with carrying (a launch's end no longer waits on
// idle lanes) and refill at 2 idle lanes: hall / interior / hall adaptive 6
// (refill 8): 190.0 / 172.3 / 147.4, 12: 195.1 / 177.8 / 150.9, 16: 196.5 /
// 178.1 / 151.3, 24 (refill 4): 195.2 / 178.3 / 151.4; wide order 2: 170.0 /
// 180.7 / 159.2, 4: 171.2 / 181.8 / 157.4
template <int kKind>
__host__ __device__ constexpr int walk_steps() {
  return kKind == kWalkOrd ? 4 : kKind == kWalkWide ? 2 : 16;
}
// reference walk steps (pops) that one step stands for: an ordered step is a
// wide node and a leaf, in place of 6 pops on average
template <int kKind>
__host__ __device__ constexpr uint32_t step_pops() {
  return kKind == kWalkOrd ? 6u : 1u;
}

// Word 3.w of a carry record: the path's depth for an extension walk, this
// tag for a connection (shadow) walk, whose record holds the connection
// {origin, slot} {direction, maxDist} {contribution, bounce} instead of the path.
constexpr uint32_t kShadowRec = 0xFFFFFFFFu;

// Words of the list of walks k_resolve answers: the item of a launch's wave,
// of its connection queue, or of the carry records it resumed.
constexpr uint32_t kOpenShadow = 0x40000000u, kOpenCarried = 0x80000000u, kOpenItem = 0x3FFFFFFFu;

// One carried walk to carry record r (out of line: it runs for a few walks
// per launch, and keeping it out of the walk loop keeps that loop's
// registers): three float4 of the walk's ray at src, src + stride, src +
// 2 * stride (the path of a wave, or a connection record), the fourth at src
// + 3 * stride (the path's carried emission and depth) or the connection tag,
// then the walk's state (two float4) and its node stack (n words).
__device__ __noinline__ void save_carry(float4* r, const float4* src, size_t stride, bool shadow, float4 state0,
                                        float4 state1, const uint32_t* stack, uint32_t n) {
  r[0] = src[0];
  r[1] = src[stride];
  r[2] = src[2 * stride];
  r[3] = shadow ? make_float4(0.f, 0.f, 0.f, __uint_as_float(kShadowRec)) : src[3 * stride];
  r[4] = state0;
  r[5] = state1;
  for (uint32_t k = 0; 4 * k < n; k++)
    r[6 + k] = make_float4(__uint_as_float(stack[4 * k]), __uint_as_float(stack[4 * k + 1]),
                           __uint_as_float(stack[4 * k + 2]), __uint_as_float(stack[4 * k + 3]));
}
__device__ __forceinline__ void save_walk(float4* r, const float4* src, size_t stride, bool shadow, const Walk& w,
                                          const uint32_t* stack) {
  save_carry(r, src, stride, shadow, make_float4(w.minT, __uint_as_float(w.best), w.bu, w.bv),
             make_float4(w.bw, __uint_as_float(w.steps), __uint_as_float(w.tos), __int_as_float(w.sp)), stack, 32);
}
__device__ __forceinline__ void save_walk(float4* r, const float4* src, size_t stride, bool shadow, const OrdWalk& w,
                                          const uint2* stack) {
  save_carry(r, src, stride, shadow, make_float4(w.minT, __uint_as_float(w.best), w.bu, w.bv),
             make_float4(__uint_as_float(w.gA), __uint_as_float(w.gB), __uint_as_float(w.bound), __int_as_float(w.sp)),
             reinterpret_cast<const uint32_t*>(stack), 2u * (uint32_t)w.sp);
}
static_assert(kCarryF4 >= 6 + 8 && kCarryF4 >= 6 + kOrdStack / 2, "carry record holds either walk");

// The walk of carry record r, resumed at the step where it stopped; true for
// a connection walk (any hit up to its maxDist).
__device__ __forceinline__ bool resume_walk(const DevScene& S, const float4* r, Walk& w, uint32_t* stack) {
  const float4 r1 = r[1];
  const bool shadow = __float_as_uint(r[3].w) == kShadowRec;
  w.init(ld3(r[0]), ld3(r1), shadow ? r1.w : gb::kInf, gb::kBias, stack);
  const float4 q = r[4], z = r[5];
  w.minT = q.x;
  w.best = __float_as_uint(q.y);
  w.bu = q.z;
  w.bv = q.w;
  w.bw = z.x;
  w.steps = __float_as_uint(z.y);
  w.tos = __float_as_uint(z.z);
  w.sp = __float_as_int(z.w);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const float4 e = r[6 + k];
    stack[4 * k] = __float_as_uint(e.x);
    stack[4 * k + 1] = __float_as_uint(e.y);
    stack[4 * k + 2] = __float_as_uint(e.z);
    stack[4 * k + 3] = __float_as_uint(e.w);
  }
  return shadow;
}
__device__ __forceinline__ bool resume_walk(const DevScene& S, const float4* r, OrdWalk& w, uint2* stack) {
  const float4 r1 = r[1];
  const bool shadow = __float_as_uint(r[3].w) == kShadowRec;
  start_walk<kWalkOrd>(S, w, ld3(r[0]), ld3(r1), 0.f, shadow, stack);
  const float4 q = r[4], z = r[5];
  w.minT = q.x;
  w.best = __float_as_uint(q.y);
  w.bu = q.z;
  w.bv = q.w;
  w.gA = __float_as_uint(z.x);
  w.gB = __float_as_uint(z.y);
  w.bound = __float_as_uint(z.z);
  w.sp = __float_as_int(z.w);
  w.rescale(S);
#pragma unroll 1
  for (int k = 0; 2 * k < w.sp; k++) {
    const float4 e = r[6 + k];
    stack[2 * k] = make_uint2(__float_as_uint(e.x), __float_as_uint(e.y));
    stack[2 * k + 1] = make_uint2(__float_as_uint(e.z), __float_as_uint(e.w));
  }
  return shadow;
}

// An unoccluded connection: its contribution into the slot's entry for the
// bounce that made it (summed with the path's other connections, in bounce
// order, by k_fold once every walk of the frame is done).
__device__ __forceinline__ void connection_reached(const RenderBuffers& b, uint32_t bilat, float4 A, float4 C) {
  const uint32_t slot = __float_as_uint(A.w), bounce = __float_as_uint(C.w);
  b.conn[(size_t)bounce * b.cap + slot] = make_float4(C.x, C.y, C.z, 1.f);
  if (bilat && bounce == 0u) direct_connect(b.dsm, slot, C);
}

// walks carried out of bounce launch L (buffer L & 1, counter L % 3; the
// counter of launch L + 1 is reset by launch L, after its last reader)
__device__ __forceinline__ uint32_t carried_of(const RenderBuffers& b, uint32_t launch) {
  return b.carry[0] ? min(b.ctr->carryN[launch % 3u], b.carryCap) : 0u;
}

// What becomes of an ordered walk that ended past the reference's pop bound
// (about 0.01-0.02 % of them; hardly any really run out of pops): the
// reference's walk at once (scenes too small to run out, where only origins
// outside the walk's range come here); a list that k_resolve answers before
// the launch is shaded (the modes whose shading adds to per-path state); or
// taken as it is, with a record of the path at this point that k_verify checks
// while the frame goes on (every other mode).
enum : uint32_t { kOpenNow = 0, kOpenList = 1, kOpenCheck = 2 };

// A record to check: {path's four float4, or the connection's three and its
// tag} {t, triangle, u, v; t -1: no hit}.  list 0: bounce launches, 1: the tail
// kernel.  False when the list is full.
__device__ __forceinline__ bool note_check(const RenderBuffers& b, uint32_t list, float4 r0, float4 r1, float4 r2,
                                           float4 r3, float4 answer) {
  const uint32_t k = atomicAdd(&b.ctr->checkN[list], 1u);
  if (k >= b.checkCap) return false;
  float4* r = b.check + ((size_t)list * b.checkCap + k) * kCheckF4;
  r[0] = r0;
  r[1] = r1;
  r[2] = r2;
  r[3] = r3;
  r[4] = answer;
  return true;
}

// Carrying (reference order only): once the launch's ray queue is empty, a
// warp keeps stepping its walks for carrySteps more steps; walks still
// unfinished then are written, with their path (or connection) and complete
// walk state, to the launch's carry buffer, an extension walk's hit word
// marked -2 (k_shade skips it).  The next bounce launch resumes them after its
// shadow rays (items nS .. nS+nC-1; their hit words after its own extension
// rays' at nE + k, -2 for a connection) and its shading kernel shades the
// extension walks at their own depth, one bounce behind the paths around
// them; the tail kernel takes those of the last bounce launch.  Results are
// unchanged: every random number is keyed by the path's own depth, and
// connections do not add to the slot when their walk ends but store their
// contribution per bounce, summed in bounce order by k_fold (a path's
// connections may now finish out of order).  The filter-only mode's bounce-0
// connections, whose direct-light sample is read by the next bounce's
// shading, are never carried.
template <bool kCount, int kKind>
__global__ void __launch_bounds__(kBlock, 4) k_walk(DevScene S, RenderBuffers b, int in, int shIn,
                                                              int shReset, uint32_t bilat, uint32_t kRefill,
                                                              uint32_t launch, uint32_t carrySteps, uint32_t later) {
  if (b.ctr->tailAt <= launch) return;  // the frame's tail kernel carries this bounce
  const uint32_t nC = (kKind != kWalkWide && in >= 0 && launch > 0) ? carried_of(b, launch - 1) : 0u;
  const uint32_t nE = (in >= 0) ? b.ctr->wave[in] : 0u;
  const uint32_t nS = (shIn >= 0) ? b.ctr->shadow[shIn] : 0u;
  const uint32_t nCE = nC + nE;
  const uint32_t n = nCE + nS;
  uint32_t* fetch = &b.ctr->fetchT;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    atomicAdd(&b.ctr->rays, (unsigned long long)nS);
    atomicAdd(&b.ctr->shadowRays, (unsigned long long)nS);
    if (in >= 0) b.ctr->wave[in ^ 1] = 0;
    b.ctr->shadow[shReset] = 0;
    b.ctr->carryN[(launch + 1) % 3u] = 0;
  }
  const Wave wv = b.wave[in >= 0 ? in : 0];
  const float4* __restrict__ sh = b.sh[shIn >= 0 ? shIn : 0];
  const float4* prev = b.carry[(launch + 1) & 1u];  // launch - 1's carried walks
  const uint32_t lane = threadIdx.x & 31;
  typename WalkOf<kKind>::type w;
  typename WalkOf<kKind>::Entry stack[WalkOf<kKind>::kDepth];
  bool has = false, drained = false, any = false, res = false;
  uint32_t item = 0, nnE = 0, ntE = 0, nnS = 0, ntS = 0;
  uint32_t dryFor = 0;  // walk steps since this warp found the queue empty
  for (;;) {
    const uint32_t idle = __ballot_sync(0xffffffffu, !has);
    if (idle == 0xffffffffu && drained) break;
    if constexpr (kKind == kWalkOrd) w.stop_long();
    if constexpr (kKind != kWalkWide) {
      if (carrySteps && drained && in >= 0) {
        // once per warp, carrySteps steps after it found the queue empty: its
        // walks still running take carry records with one atomic for the warp
        // (walks that find the buffer full finish here)
        if (dryFor >= carrySteps && dryFor < carrySteps + walk_steps<kKind>() * step_pops<kKind>()) {
          const float4* src = res ? prev + (size_t)item * kCarryF4 : (any ? sh + 3 * (size_t)item : wv.o + item);
          const bool want = has && !(any && bilat && __float_as_uint(src[2].w) == 0u);
          const uint32_t m = __ballot_sync(0xffffffffu, want);
          uint32_t c0 = 0;
          if (m && lane == 0) c0 = atomicAdd(&b.ctr->carryN[launch % 3u], (uint32_t)__popc(m));
          c0 = __shfl_sync(0xffffffffu, c0, 0) + __popc(m & lanemask_lt());
          if (want && c0 < b.carryCap) {
            save_walk(b.carry[launch & 1u] + (size_t)c0 * kCarryF4, src, (res || any) ? 1 : (size_t)(wv.d - wv.o),
                      any && !res, w, stack);
            if (res || !any) b.hit[res ? nE + item : item] = make_float4(-2.f, 0.f, 0.f, 0.f);
            has = false;
          }
        }
        dryFor += walk_steps<kKind>() * step_pops<kKind>();
      }
    }
    if (!drained && (idle == 0xffffffffu || __popc(idle) >= kRefill)) {
      const uint32_t cnt = __popc(idle);
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(fetch, cnt);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base + cnt >= n) drained = true;
      if (!has) {
        const uint32_t k = base + __popc(idle & lanemask_lt());
        if (k < n) {
          has = true;
          any = k < nS;
          res = !any && k < nS + nC;
          item = any ? k : (res ? k - nS : k - nS - nC);
          if (res) {
            if constexpr (kKind != kWalkWide) any = resume_walk(S, prev + (size_t)item * kCarryF4, w, stack);
          } else if (any) {
            const float4 A = sh[3 * (size_t)item], B = sh[3 * (size_t)item + 1];
            start_walk<kKind>(S, w, ld3(A), ld3(B), B.w, true, stack);
          } else {
            start_walk<kKind>(S, w, ld3(wv.o[item]), ld3(wv.d[item]), gb::kInf, false, stack);
          }
        }
      }
    }
    // walk_steps() steps per refill check: the ballot and refill test are paid
    // once for them (a lane whose walk ends in the first waits out the rest)
#pragma unroll 1
    for (int u = 0; u < walk_steps<kKind>(); u++) {
      // one inlined walk step for both ray kinds (a runtime any-hit flag), so a
      // warp holding extension and shadow rays does not run two copies of it;
      // the counting variant keeps separate counters per kind
      bool fin = false;
      if constexpr (kKind == kWalkOrd) {
        fin = w.step_warp(S, stack, has);
      } else if (has) {
        if (kCount)
          fin = any ? step_walk<kKind, kCount>(S, w, stack, true, nnS, ntS)
                    : step_walk<kKind, kCount>(S, w, stack, false, nnE, ntE);
        else
          fin = step_walk<kKind, kCount>(S, w, stack, any, nnE, ntE);
      }
      if (fin) {
        has = false;
        bool open = false;
        if constexpr (kKind == kWalkOrd) {
          if (w.capped()) {
            bool now = later == kOpenNow;
            if (later == kOpenList) {
              const uint32_t k = atomicAdd(&b.ctr->openN, 1u);
              open = k < b.openCap;
              now = !open;
              if (open) b.open[k] = item | (res ? kOpenCarried : any ? kOpenShadow : 0u);
              else b.ctr->openOver = 1u;
            } else if (later == kOpenCheck) {
              now = w.bound >= kPopStop;  // an unfinished walk has no answer to take
            }
            if (later == kOpenCheck && !now) {
              const float4* q = res ? prev + (size_t)item * kCarryF4 : any ? sh + 3 * (size_t)item : wv.o + item;
              const size_t st = (res || any) ? 1 : (size_t)(wv.d - wv.o);
              now = !note_check(b, 0, q[0], q[st], q[2 * st],
                                any ? make_float4(0.f, 0.f, 0.f, __uint_as_float(kShadowRec)) : q[3 * st],
                                make_float4(w.hit() ? w.minT : -1.f, __uint_as_float(w.best), w.bu, w.bv));
            }
            if (now) {
              TraceHit h;
              uint32_t nn = 0, nt = 0;
              const float far = any ? (res ? prev + (size_t)item * kCarryF4 : sh + 3 * (size_t)item)[1].w : gb::kInf;
              const bool hit = trace_ref<false, false>(S, w.o, w.d, far, gb::kBias, false, h, nn, nt);
              w.settle(hit, make_float4(h.t, __uint_as_float(h.tri), h.u, h.v));
            }
          }
        }
        if (open) {
          // k_resolve stores its answer
        } else if (any) {
          const float4* q = res ? prev + (size_t)item * kCarryF4 : sh + 3 * (size_t)item;
          if (!w.hit()) connection_reached(b, bilat, q[0], q[2]);  // unoccluded: it counts (:716-721)
          if (res) b.hit[nE + item] = make_float4(-2.f, 0.f, 0.f, 0.f);
        } else {
          b.hit[res ? nE + item : item] = w.hit() ? make_float4(w.minT, __uint_as_float(w.best), w.bu, w.bv)
                                                  : make_float4(-1.f, 0.f, 0.f, 0.f);
        }
      }
    }
  }
  if (kCount) {
    warp_add_u64(&b.ctr->nodes, nnE);
    warp_add_u64(&b.ctr->tris, ntE);
    warp_add_u64(&b.ctr->nodesS, nnS);
    warp_add_u64(&b.ctr->trisS, ntS);
  }
}

// ---------------------------------------------------------------------------
// Shading of one path after its closest-hit walk (pt_traceSample_kernel after
// TracePrimitive, src/cudaRTBDPTStream.cu:381-543) and the connection set-up
// of GetLightFromRandLightVertices / pt_connectEyeLightPath_kernel
// (:665-723): everything but the visibility test, which the shadow walk does.
// io holds the path (origin+slot, direction+pixel, throughput, carried
// emission) on entry and the next ray's state on exit when cont is set.
struct PathIO {
  float4 o, d, t, s;
  bool cont, conn;
  float4 shA, shB, shC;
};

// learned allocator statistics: a finished path of pixel `pix` after `hits`
// surface hits, counted in its 8x8 tile's path-length histogram
__device__ __forceinline__ void count_path_length(const FrameArgs& a, const RenderBuffers& b, uint32_t pix,
                                                  uint32_t hits) {
  const uint32_t px = pix % a.width, py = pix / a.width;
  const uint32_t tile = (py >> 3) * a.tilesX + (px >> 3);
  atomicAdd(&b.hist[tile * 8u + (hits < 7u ? hits : 7u)], 1u);
}

__device__ __forceinline__ void shade_path(const DevScene& S, const FrameArgs& a, const RenderBuffers& b,
                                           const float4* __restrict__ cache, uint32_t cacheSize, uint32_t depth,
                                           float4 h4, PathIO& io) {
  using namespace gb;
  io.cont = false;
  io.conn = false;
  const uint32_t slot = __float_as_uint(io.o.w);
  const uint32_t pix = __float_as_uint(io.d.w);
  f3 orig = ld3(io.o), dir = ld3(io.d), outMul = ld3(io.t), pathSample = ld3(io.s);
  float pot = io.t.w;  // path potential (filter-only mode)
  if (h4.x < 0.f) {  // miss (:537-542), plus the optional environment term
    if (a.useEnv) pathSample = pathSample + vmul(mk(a.env[0], a.env[1], a.env[2]), outMul);
    // the path's end: its emission and how many bounces' connections k_fold sums before it
    b.res[slot] = make_float4(pathSample.x, pathSample.y, pathSample.z, __uint_as_float(depth));
    if (a.bilat) reinterpret_cast<float*>(b.dsm + slot)[3] = pot;
    if (a.moments) count_path_length(a, b, pix, depth);
    return;
  }
  const uint32_t smp = b.slotSmp[slot];
  float u[8];
  draw8(a.key0, a.key1, pix, a.frame, kEyeBounce, depth, smp, u);
  const float hu = h4.z, hv = h4.w, hw = 1.f - hu - hv;
  Surf sf = load_surf(S, __float_as_uint(h4.y), hw, hu, hv, a.gbuffer && depth == 0);
  Mat m = load_mat_at(S, sf.mat, __float_as_uint(h4.y), hw, hu, hv);
  Bounce B;
  sample_bounce(orig, dir, h4.x, sf.norm, m, u, a.specPush != 0, a.bilat != 0, a.ptsc != 0, B);
  pathSample = pathSample + vmul(m.emis, outMul);
  if (a.gbuffer && depth == 0) {  // AdapBilatAtomic.cu:471-476, Bilat.cu:632-638
    const bool be = a.bilat != 0;
    b.gbuf[3 * (size_t)slot] = st4(sf.pos, be ? m.emis.x : 0.f);
    b.gbuf[3 * (size_t)slot + 1] = st4(B.nl, be ? m.emis.y : 0.f);
    b.gbuf[3 * (size_t)slot + 2] = st4(m.diff, be ? m.emis.z : 0.f);
  }
  if (a.bilat) {  // Bilat.cu:628-631
    pot = pot * B.pdf;
    if (depth < 2) {
      const float4 q = b.dsm[slot];
      b.dsm[slot] = make_float4(q.x + pathSample.x, q.y + pathSample.y, q.z + pathSample.z, q.w);
    }
  }
  const f3 inMul = outMul;
  float contrib = length(outMul) * length(B.lmt);
  if (length(m.emis) > 0.f) contrib = 0.f;
  if (u[6] > contrib || depth + 1 >= a.eyeDepth) {
    b.res[slot] = make_float4(pathSample.x, pathSample.y, pathSample.z, __uint_as_float(depth));
    if (a.bilat) reinterpret_cast<float*>(b.dsm + slot)[3] = pot;
    if (a.moments) count_path_length(a, b, pix, depth + 1);
    return;
  }
  io.cont = true;
  b.conn[(size_t)depth * b.cap + slot] = make_float4(0.f, 0.f, 0.f, 0.f);  // no connection made
  outMul = vmul(outMul, B.lmt);
  io.o = st4u(B.nOrig, slot);
  io.d = st4u(B.nDir, pix);
  io.t = st4(outMul, pot);
  io.s = make_float4(pathSample.x, pathSample.y, pathSample.z, __uint_as_float(depth + 1));
  if (B.type != kTypeDiff || cacheSize == 0 || a.ptsc) return;
  // connection: pick a cached light vertex, shade both ends (:665-723)
  f3 pos = B.nOrig + B.nl * kBias;
  uint32_t li = (uint32_t)(u[7] * (float)cacheSize);
  if (li >= cacheSize) li = cacheSize - 1;
  LV lv = load_lv(cache + 6 * (size_t)li);
  f3 toDir = normalize(lv.pos - pos);
  float toDist = length(lv.pos - pos);
  if (!(length(lv.irrad) > 0.f && dot(B.nl, toDir) > 0.f)) return;
  f3 irrad, irradDir;
  if (toDist > kFltEps) {
    irrad = shading(-1.f * toDir, lv.irradDir, lv.irrad, lv.norm, lv.diff, lv.metal, lv.rough, lv.spec, 1.f, 1.f) +
            lv.emis;
    irradDir = toDir;
  } else {
    irrad = lv.irrad;
    irradDir = -1.f * lv.irradDir;
  }
  f3 c = vmax0(shading(-1.f * dir, irradDir, irrad, B.nl, m.diff, m.metal, m.rough, m.spec, 1.f - m.trans, 1.f));
  if (length(c) > 0.f) {
    io.conn = true;
    reinterpret_cast<float*>(b.conn + (size_t)depth * b.cap + slot)[3] = -1.f;  // occluded, until its walk says
    io.shA = st4u(pos, slot);
    io.shB = st4(toDir, toDist - kBias);
    const f3 cw = vmul(c, inMul);
    io.shC = make_float4(cw.x, cw.y, cw.z, __uint_as_float(depth));  // .w: the bounce that made it
  }
}

// Shading of bounce launch L: the paths of its wave, then the walks it
// resumed for launch L - 1 (carry records, their hits after the wave's), each
// at its own depth; survivors are appended to the other wave buffer and
// connection requests to queue L & 1, one atomic per warp each.
// attach != 0 (the last bounce launch before the tail kernel): each continuing
// path's connection record is stored at the path's own index j of queue
// L & 1 (slot word 0xffffffff when it has none), so that the tail kernel
// walks it on the path's lane before the path's next bounce.  Three CTAs per
// SM (80 registers, a few bytes of spill) beat two at 96 registers: shading
// time -10 to -12% on the interior and hall walks.
__global__ void __launch_bounds__(kBlock, 3) k_shade(DevScene S, FrameArgs a, RenderBuffers b, int in, uint32_t launch,
                                                     uint32_t attach) {
  if (b.ctr->tailAt <= launch) return;  // the frame's tail kernel carries this bounce
  const uint32_t n = b.ctr->wave[in];
  const uint32_t nC = launch > 0 ? carried_of(b, launch - 1) : 0u;
  const uint32_t total = n + nC;
  // the switch decided on the device: with fewer than tailBelow x the band's
  // camera paths alive at this launch, the paths that continue go to the tail
  // kernel from the next launch (every CTA reads the same counts and decides alike)
  if (!attach && a.tailBelow > 0.f && launch + 1 < a.eyeDepth && (float)total < a.tailBelow * (float)b.ctr->paths)
    attach = 2u;
  const uint32_t cacheSize = b.lctr->cacheSize[a.cacheSel];
  const float4* __restrict__ cache = b.cache[a.cacheSel];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    atomicAdd(&b.ctr->rays, (unsigned long long)n);  // resumed walks were counted by their own launch
    b.ctr->fetchT = 0;  // for the next walk (next bounce's rays + this bounce's shadow rays)
    b.ctr->openN = 0;
    if (attach == 2u) b.ctr->tailAt = launch + 1;
  }
  const Wave w = b.wave[in];
  const Wave wo = b.wave[in ^ 1];
  const float4* prev = b.carry[(launch + 1) & 1u];
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t lane = threadIdx.x & 31;
  float4* shq = b.sh[launch & 1u];
  for (uint32_t base = blockIdx.x * blockDim.x; base < total; base += stride) {
    const uint32_t i = base + threadIdx.x;
    PathIO io;
    io.cont = io.conn = false;
    if (i < total) {
      const float4 h = b.hit[i];
      if (h.x != -2.f) {  // -2: the walk was carried on, to the next launch or the tail kernel
        if (i < n) {
          io.o = w.o[i];
          io.d = w.d[i];
          io.t = w.thr[i];
          io.s = w.smp[i];
        } else {
          const float4* r = prev + (size_t)(i - n) * kCarryF4;
          io.o = r[0];
          io.d = r[1];
          io.t = r[2];
          io.s = r[3];
        }
        shade_path(S, a, b, cache, cacheSize, __float_as_uint(io.s.w), h, io);
      }
    }
    const uint32_t mc = __ballot_sync(0xffffffffu, io.cont);
    if (mc) {
      uint32_t basej = 0;
      if (lane == 0) basej = atomicAdd(&b.ctr->wave[in ^ 1], __popc(mc));
      basej = __shfl_sync(0xffffffffu, basej, 0);
      if (io.cont) {
        const uint32_t j = basej + __popc(mc & lanemask_lt());
        wo.o[j] = io.o;
        wo.d[j] = io.d;
        wo.thr[j] = io.t;
        wo.smp[j] = io.s;
        if (attach) {
          shq[3 * (size_t)j] = io.conn ? io.shA : make_float4(0.f, 0.f, 0.f, __uint_as_float(0xffffffffu));
          shq[3 * (size_t)j + 1] = io.shB;
          shq[3 * (size_t)j + 2] = io.shC;
        }
      }
    }
    if (attach) continue;
    const uint32_t ms = __ballot_sync(0xffffffffu, io.conn);
    if (ms) {
      uint32_t basej = 0;
      if (lane == 0) basej = atomicAdd(&b.ctr->shadow[launch & 1u], __popc(ms));
      basej = __shfl_sync(0xffffffffu, basej, 0);
      if (io.conn) {
        const uint32_t j = basej + __popc(ms & lanemask_lt());
        shq[3 * (size_t)j] = io.shA;
        shq[3 * (size_t)j + 1] = io.shB;
        shq[3 * (size_t)j + 2] = io.shC;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Tail of a frame: once few paths are left, per-bounce launches are bounded
// by their slowest ray.  This persistent kernel instead carries every path
// of the wave left by the last bounce launch run (t, the switch bounce or K)
// through all its remaining bounces on one lane, each at its own depth: the
// connection attached to it by that launch (queue (t - 1) & 1, same index;
// slot word 0xffffffff: none), then closest-hit walk, shading, connection and
// shadow walk bounce after bounce; then the walks that launch carried,
// resumed where they stopped.  A path executes exactly the operations of the
// wavefront kernels in the same order (a connection is applied before the
// next bounce is shaded), so results are identical.
enum : uint32_t { kIdle = 0, kPathExt = 1, kPathShadow = 2 };

// walk steps of the tail kernel between two refill checks: a lane whose walk
// ends early waits for the others, and the warp then shades its finished
// paths together.  Measured in Mpaths/s on interior / Cornell before walks
// were carried (the hall then ran no tail kernel): 1: 154.4 / 144.2, 4:
// 157.5 / 158.7, 16: 161.1 / 171.4, 64: 162.3 / 189.1, 512: 156.7 / 197.4;
// with carrying and 16-step walk batches (hall / interior / Cornell): 32:
// 194.3 / 175.4 / 171.6, 64: 195.9 / 178.8 / 190.4, 128: 195.2 / 178.1 /
// 192.7.  Three CTAs per SM (80 registers, some spill) against two (116
// registers): interior 167.0 -> 170.0, Cornell 195.6 -> 193.6 Mpaths/s; four
// (64 registers): hall 195.9 -> 194.6, Cornell 190.4 -> 183.1.
// The ordered walk's tail: two CTAs per SM (128 registers, no spill) against
// three (80, 390 bytes of spill stores) and four: Cornell 256x256 image 3.61 /
// 3.99 / 4.50 ms, unidirectional 333x217 image 4.46 / 4.86 / 5.34, hall pass 2.94 /
// 2.97 / 2.99; 12 and 24 steps between refill checks within 2 % of 16.
template <int kKind>
__host__ __device__ constexpr int tail_ctas() {
  return kKind == kWalkOrd ? 2 : 3;
}
template <int kKind>
__host__ __device__ constexpr int tail_steps() {
  return kKind == kWalkOrd ? 16 : 64;
}

// kLater: what becomes of walks past the pop bound (kOpenNow etc.), fixed at
// compile time so that a kernel holds only its own case's code.
template <bool kCount, int kKind, uint32_t kLater = kOpenNow>
__global__ void __launch_bounds__(kBlock, tail_ctas<kKind>()) k_tail(DevScene S, FrameArgs a, RenderBuffers b, uint32_t K,
                                                   uint32_t kRefill) {
  // t: the launch the bounce launches stopped before (the device switch or K)
  const uint32_t t = min(b.ctr->tailAt, K);
  const int in = (int)(t & 1u);
  const int shIn = t > 0 ? (int)((t - 1) & 1u) : -1;
  const uint32_t n = b.ctr->wave[in];
  const uint32_t nCarry = t > 0 ? carried_of(b, t - 1) : 0u;
  const float4* carried = b.carry[(t + 1) & 1u];  // launch t - 1's
  const uint32_t total = n + nCarry;
  const uint32_t cacheSize = b.lctr->cacheSize[a.cacheSel];
  const float4* __restrict__ cache = b.cache[a.cacheSel];
  const float4* __restrict__ sh = b.sh[shIn >= 0 ? shIn : 0];
  const Wave wv = b.wave[in];
  const uint32_t lane = threadIdx.x & 31;
  typename WalkOf<kKind>::type w;
  typename WalkOf<kKind>::Entry stack[WalkOf<kKind>::kDepth];
  PathIO io;
  uint32_t mode = kIdle;
  bool drained = false, resumed = false;
  uint32_t extRays = 0, shRays = 0, nnE = 0, ntE = 0, nnS = 0, ntS = 0;
  const uint32_t warps = gridDim.x * (kBlock / 32);
  // so few paths that four a warp hold them all: their walks run eight lanes each
  const uint32_t lanes = kKind == kWalkOrd && kLater != kOpenNow && total <= 4u * warps ? 0xFu : path_lanes(total, warps);
  for (;;) {
    const uint32_t idle = __ballot_sync(0xffffffffu, mode == kIdle) & lanes;
    if (idle == lanes && drained) break;
    if constexpr (kKind == kWalkOrd) w.stop_long();
    if (!drained && (idle == lanes || __popc(idle) >= kRefill)) {
      const uint32_t cnt = __popc(idle);
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(&b.ctr->fetchTail, cnt);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base + cnt >= total) drained = true;
      if ((idle >> lane) & 1u) {
        const uint32_t j = base + __popc(idle & lanemask_lt());
        if (j >= n && j < total) {  // a carried walk: resume it where it stopped
          const float4* r = carried + (size_t)(j - n) * kCarryF4;
          resumed = true;
          if constexpr (kKind != kWalkWide) {
            if (resume_walk(S, r, w, stack)) {  // a connection alone, without its path
              io.shA = r[0];
              io.shB = r[1];
              io.shC = r[2];
              mode = kPathShadow;
            } else {
              io.o = r[0];
              io.d = r[1];
              io.t = r[2];
              io.s = r[3];
              mode = kPathExt;
            }
          }
        } else if (j < n) {
          io.o = wv.o[j];
          io.d = wv.d[j];
          io.t = wv.thr[j];
          io.s = wv.smp[j];
          const float4 A = (shIn >= 0) ? sh[3 * (size_t)j] : make_float4(0.f, 0.f, 0.f, __uint_as_float(0xffffffffu));
          if (__float_as_uint(A.w) != 0xffffffffu) {
            io.shA = A;
            io.shB = sh[3 * (size_t)j + 1];
            io.shC = sh[3 * (size_t)j + 2];
            mode = kPathShadow;
            start_walk<kKind>(S, w, ld3(io.shA), ld3(io.shB), io.shB.w, true, stack);
          } else {
            mode = kPathExt;
            start_walk<kKind>(S, w, ld3(io.o), ld3(io.d), gb::kInf, false, stack);
          }
        }
      }
    }
    if (kKind != kWalkOrd && mode == kIdle) continue;
    const bool anyHit = mode == kPathShadow;
    bool done = false;
    if constexpr (kKind == kWalkOrd) {
      // No more than four paths left to this warp: eight lanes a walk.  A step
      // costs about 2200 cycles whether 2 or 30 lanes take it (370 instructions
      // at six cycles each, instruction latency and not memory: children touched
      // ahead into L1 changed nothing), and the longest warps of a hall frame
      // spend 70 % of their time with four paths or fewer.  Unidirectional
      // 333x217 image 4.46 -> 4.15 ms, hall pass 2.93 -> 2.88, binary 500x375
      // image 9.70 -> 9.51.  Trees of up to 2048 nodes (kOpenNow) end their walks
      // in a few steps, and moving them costs more: Cornell 256x256 image 3.62 ->
      // 4.25 ms with it.
      const bool together = kLater != kOpenNow && (drained || __popc(lanes) <= 4);
      // the warp's walks advance together until they are all over, at most tail_steps times
      const uint32_t live = __ballot_sync(0xffffffffu, mode != kIdle);
      if (together && __popc(live) <= 4) {
        if constexpr (kLater != kOpenNow) gather_walks(S, w, stack, live);
        done = true;
      } else {
#pragma unroll 1
        for (int u = 0; u < tail_steps<kKind>(); u++) {
          done = w.step_warp(S, stack, mode != kIdle);
          if (__all_sync(0xffffffffu, done || mode == kIdle)) break;
        }
      }
      if (mode == kIdle) continue;
      if (done && w.capped()) {
        const float4 got = make_float4(w.hit() ? w.minT : -1.f, __uint_as_float(w.best), w.bu, w.bv);
        // an extension walk of a mode whose shading cannot be undone waits for
        // its answer (t -2: to be run on from there whatever it is); so would the
        // connection whose direct-light sample the next shading reads
        const bool wait = kLater == kOpenList && !anyHit;
        const bool direct = kLater == kOpenList && anyHit && a.bilat && __float_as_uint(io.shC.w) == 0u;
        const bool noted =
            kLater != kOpenNow && !direct && (wait || w.bound < kPopStop) &&
            (anyHit ? note_check(b, 1, io.shA, io.shB, io.shC, make_float4(0.f, 0.f, 0.f, __uint_as_float(kShadowRec)), got)
                    : note_check(b, 1, io.o, io.d, io.t, io.s, wait ? make_float4(-2.f, 0.f, 0.f, 0.f) : got));
        if (noted && wait) {
          if (!resumed) extRays++;
          resumed = false;
          mode = kIdle;
          continue;
        }
        if (!noted) {
          TraceHit h;
          uint32_t nn = 0, nt = 0;
          const bool hit = trace_ref<false, false>(S, w.o, w.d, anyHit ? io.shB.w : gb::kInf, gb::kBias, false, h, nn, nt);
          w.settle(hit, make_float4(h.t, __uint_as_float(h.tri), h.u, h.v));
        }
      }
    } else
#pragma unroll 1
    for (int u = 0; u < tail_steps<kKind>() && !done; u++)
      done = kCount ? (anyHit ? step_walk<kKind, kCount>(S, w, stack, true, nnS, ntS)
                              : step_walk<kKind, kCount>(S, w, stack, false, nnE, ntE))
                    : step_walk<kKind, kCount>(S, w, stack, anyHit, nnE, ntE);
    if (!done) continue;
    if (anyHit) {
      if (!w.hit()) connection_reached(b, a.bilat, io.shA, io.shC);  // unoccluded connection (:716-721)
      if (resumed) {  // a carried connection alone (counted by its launch): done
        resumed = false;
        mode = kIdle;
        continue;
      }
      shRays++;
      mode = kPathExt;  // the path's next extension ray
      start_walk<kKind>(S, w, ld3(io.o), ld3(io.d), gb::kInf, false, stack);
      continue;
    }
    // closest hit of the path's current ray: shade it (a resumed walk was
    // counted by the bounce launch's shading kernel)
    if (!resumed) extRays++;
    resumed = false;
    const float4 h4 = w.hit() ? make_float4(w.minT, __uint_as_float(w.best), w.bu, w.bv)
                              : make_float4(-1.f, 0.f, 0.f, 0.f);
    shade_path(S, a, b, cache, cacheSize, __float_as_uint(io.s.w), h4, io);
    if (!io.cont) {
      mode = kIdle;
    } else {
      if (io.conn) {
        mode = kPathShadow;
        start_walk<kKind>(S, w, ld3(io.shA), ld3(io.shB), io.shB.w, true, stack);
      } else {
        start_walk<kKind>(S, w, ld3(io.o), ld3(io.d), gb::kInf, false, stack);
      }
    }
  }
  warp_add_u64(&b.ctr->rays, extRays + shRays);
  warp_add_u64(&b.ctr->shadowRays, shRays);
  if (kCount) {
    warp_add_u64(&b.ctr->nodes, nnE);
    warp_add_u64(&b.ctr->tris, ntE);
    warp_add_u64(&b.ctr->nodesS, nnS);
    warp_add_u64(&b.ctr->trisS, ntS);
  }
}

// ---------------------------------------------------------------------------
// Answers of the walks bounce launch `launch` listed, one block each, before it
// is shaded.  On the 332,180-triangle hall about 150 of a launch's million
// walks; 65 us, most of it the cold binary tree's latency level by level.
__global__ void __launch_bounds__(kCapThreads) k_resolve(DevScene S, RenderBuffers b, int in, int shIn, uint32_t bilat,
                                                         uint32_t launch) {
  extern __shared__ float4 capMem[];
  CapShared& c = *reinterpret_cast<CapShared*>(capMem);
  if (b.ctr->tailAt <= launch) return;
  const uint32_t n = min(b.ctr->openN, b.openCap), nE = (in >= 0) ? b.ctr->wave[in] : 0u;
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
    const uint32_t code = b.open[i], item = code & kOpenItem;
    const bool res = (code & kOpenCarried) != 0u;
    const float4* r = res ? b.carry[(launch + 1) & 1u] + (size_t)item * kCarryF4
                          : (code & kOpenShadow) ? b.sh[shIn] + 3 * (size_t)item : nullptr;
    const bool any = r && (!res || __float_as_uint(r[3].w) == kShadowRec);
    const float4 A = r ? r[0] : b.wave[in].o[item], B = r ? r[1] : b.wave[in].d[item];
    resolve_capped(S, c, ld3(A), ld3(B), any ? B.w : gb::kInf, gb::kBias, any);
    if (threadIdx.x == 0) {
      if (any) {
        if (!c.found) connection_reached(b, bilat, A, r[2]);
        if (res) b.hit[nE + item] = make_float4(-2.f, 0.f, 0.f, 0.f);
      } else {
        b.hit[res ? nE + item : item] = c.found ? c.answer : make_float4(-1.f, 0.f, 0.f, 0.f);
      }
    }
  }
}

// Checks the recorded answers of one list, one block each.  A connection's
// entry is set right here; a path whose closest hit was another gets its
// record's answer corrected and joins the list k_again runs from that bounce,
// which rewrites everything the path wrote from there on (its
// connection entries, its end, its first-hit planes).  The bounce launches'
// list is checked beside the tail kernel.
__global__ void __launch_bounds__(kCapThreads) k_verify(DevScene S, RenderBuffers b, uint32_t list) {
  extern __shared__ float4 capMem[];
  CapShared& c = *reinterpret_cast<CapShared*>(capMem);
  const uint32_t n = min(b.ctr->checkN[list], b.checkCap);
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
    const uint32_t rec = list * b.checkCap + i;
    float4* r = b.check + (size_t)rec * kCheckF4;
    const bool any = __float_as_uint(r[3].w) == kShadowRec;
    const float4 A = r[0], B = r[1], got = r[4];
    resolve_capped(S, c, ld3(A), ld3(B), any ? B.w : gb::kInf, gb::kBias, any);
    if (threadIdx.x != 0) continue;
    const bool hit = c.found != 0u, was = got.x >= 0.f;
    if (any) {
      if (hit != was) {
        const float4 C = r[2];
        const float4 none = make_float4(0.f, 0.f, 0.f, -1.f);
        b.conn[(size_t)__float_as_uint(C.w) * b.cap + __float_as_uint(A.w)] = hit ? none : make_float4(C.x, C.y, C.z, 1.f);
      }
    } else if (got.x == -2.f || hit != was || (hit && (c.answer.x != got.x || __float_as_uint(c.answer.y) != __float_as_uint(got.y)))) {
      r[4] = hit ? c.answer : make_float4(-1.f, 0.f, 0.f, 0.f);
      b.fix[atomicAdd(&b.ctr->fixN, 1u)] = rec;
    }
  }
}

// The paths k_verify listed, from the bounce of their record on with its
// answer, one block each: few and alone on the GPU, so their latency counts.
// Walks run eight lanes a ray (coop_walk, every group the same ray), those past
// the pop bound are resolved by the block at once; one thread shades.
__global__ void __launch_bounds__(kCapThreads) k_again(DevScene S, FrameArgs a, RenderBuffers b) {
  extern __shared__ float4 capMem[];
  CapShared& c = *reinterpret_cast<CapShared*>(capMem);
  __shared__ float4 path[7];
  __shared__ uint32_t flags;
  const uint32_t n = b.ctr->fixN;
  const uint32_t cacheSize = b.lctr->cacheSize[a.cacheSel];
  const float4* __restrict__ cache = b.cache[a.cacheSel];
  int32_t extRays = 0, shRays = 0;
  // the answer of one ray, for every thread; (-1, ...) on a miss
  auto walk = [&](float4 o, float4 d, float far, bool any) {
    OrdWalk w;
    uint2 stack[kOrdStack];
    w.any = any;
    w.eps = gb::kBias;
    w.init(S, ld3(o), ld3(d), far);
    coop_walk(S, w, stack, true);
    if (!w.capped()) return w.hit() ? make_float4(w.minT, __uint_as_float(w.best), w.bu, w.bv)
                                    : make_float4(-1.f, 0.f, 0.f, 0.f);
    resolve_capped(S, c, ld3(o), ld3(d), far, gb::kBias, any);
    __syncthreads();
    const float4 h = c.found ? c.answer : make_float4(-1.f, 0.f, 0.f, 0.f);
    __syncthreads();
    return h;
  };
  for (uint32_t k = blockIdx.x; k < n; k += gridDim.x) {
    const float4* r = b.check + (size_t)b.fix[k] * kCheckF4;
    PathIO io;
    io.o = r[0];
    io.d = r[1];
    io.t = r[2];
    io.s = r[3];
    float4 h = r[4];
    bool skip = false;  // a path corrected at an earlier bounce as well starts there
    for (uint32_t m = 0; m < n; m++) {
      const float4* q = b.check + (size_t)b.fix[m] * kCheckF4;
      skip |= __float_as_uint(q[0].w) == __float_as_uint(io.o.w) && __float_as_uint(q[3].w) < __float_as_uint(io.s.w);
    }
    if (skip) continue;  // block-uniform
    // the rays of the continuation that was wrong come off the counters: one per
    // bounce up to its end, one per connection it made.  (Paths that waited for
    // this answer have none.)
    if (!(a.bilat || a.moments)) {
      const uint32_t slot = __float_as_uint(io.o.w), from = __float_as_uint(io.s.w), end = __float_as_uint(b.res[slot].w);
      extRays -= (int32_t)(end - from);
      for (uint32_t d = from; d < end; d++) shRays -= b.conn[(size_t)d * b.cap + slot].w != 0.f ? 1 : 0;
    }
    if (a.gbuffer && threadIdx.x == 0 && __float_as_uint(io.s.w) == 0u) {  // as k_camera leaves them
      float4* g = b.gbuf + 3 * (size_t)__float_as_uint(io.o.w);
      g[0] = g[1] = g[2] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (;;) {
      __syncthreads();
      if (threadIdx.x == 0) {
        shade_path(S, a, b, cache, cacheSize, __float_as_uint(io.s.w), h, io);
        path[0] = io.o, path[1] = io.d, path[2] = io.t, path[3] = io.s;
        path[4] = io.shA, path[5] = io.shB, path[6] = io.shC;
        flags = (io.cont ? 1u : 0u) | (io.conn ? 2u : 0u);
      }
      __syncthreads();
      io.o = path[0], io.d = path[1], io.t = path[2], io.s = path[3];
      const uint32_t f = flags;
      if (!(f & 1u)) break;
      if (f & 2u) {
        const float4 A = path[4], B = path[5], C = path[6];
        const float4 q = walk(A, B, B.w, true);
        if (threadIdx.x == 0 && q.x < 0.f) connection_reached(b, a.bilat, A, C);
        shRays++;
      }
      h = walk(io.o, io.d, gb::kInf, false);
      extRays++;
    }
  }
  if (threadIdx.x == 0 && (extRays || shRays)) {  // (negative: the sums wrap to the right value)
    atomicAdd(&b.ctr->rays, (unsigned long long)(long long)(extRays + shRays));
    atomicAdd(&b.ctr->shadowRays, (unsigned long long)(long long)shRays);
  }
}

// ... and of caller-supplied rays (marked with triangle -2 by their kernel):
// a block looks through 256 rays and answers the marked ones.
__global__ void __launch_bounds__(kCapThreads) k_resolve_rays(DevScene S, const float* rays, uint32_t n, float maxDist,
                                                              float eps, float* t, int32_t* tri, float* w, float* u,
                                                              float* v) {
  extern __shared__ float4 capMem[];
  CapShared& c = *reinterpret_cast<CapShared*>(capMem);
  __shared__ uint32_t list[kCapThreads], count;
  // 64 bits: the step past the last ray can leave 32
  for (uint64_t base = (uint64_t)blockIdx.x * kCapThreads; base < n; base += (uint64_t)gridDim.x * kCapThreads) {
    const uint64_t i = base + threadIdx.x;
    const bool open = i < n && tri[i] == -2;
    if (!__syncthreads_or(open)) continue;
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    if (open) list[atomicAdd(&count, 1u)] = (uint32_t)i;
    __syncthreads();
    const uint32_t m = count;
    for (uint32_t k = 0; k < m; k++) {
      const uint32_t j = list[k];
      const float* r = rays + 6 * (size_t)j;
      resolve_capped(S, c, mk(r[0], r[1], r[2]), mk(r[3], r[4], r[5]), maxDist, eps, false);
      if (threadIdx.x == 0) {
        const float4 h = c.answer;
        t[j] = c.found ? h.x : -1.f;
        tri[j] = c.found ? (int32_t)__float_as_uint(h.y) : -1;
        w[j] = c.found ? 1.f - h.z - h.w : 0.f;
        u[j] = c.found ? h.z : 0.f;
        v[j] = c.found ? h.w : 0.f;
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Sum of each path of the band, once all its walks are done: the unoccluded
// connections of bounces 0 .. k-1 in bounce order, then the path's emission
// at its end (bounce k), with the count word the accumulation kernels read
// (4 per connection, 1 for the end): the additions the reference makes into
// the path's result as each connection and the end happen (:716-721,
// :520-542), in the same order, so the sums are equal to the bit.
__global__ void k_fold(RenderBuffers b) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.ctr->paths) return;
  const uint32_t s = b.base + i;
  const float4 e = b.res[s];
  const uint32_t k = min(__float_as_uint(e.w), b.connDepth);
  float x = 0.f, y = 0.f, z = 0.f;
  uint32_t n = 0;
  for (uint32_t d = 0; d < k; d++) {
    const float4 c = b.conn[(size_t)d * b.cap + s];
    if (c.w > 0.f) {
      x = x + c.x;
      y = y + c.y;
      z = z + c.z;
      n += 4u;
    }
  }
  b.res[s] = make_float4(x + e.x, y + e.y, z + e.z, __uint_as_float(n + 1u));
}

// ---------------------------------------------------------------------------
// Running mean of one path per pixel (pt_applyPathQueueResult_kernel :741-778);
// with G-buffer planes, also the count-weighted first-hit means
// (AdapBilatAtomic.cu:929-966).
__global__ void k_apply(FrameArgs a, RenderBuffers b, float* result, uint32_t* sampleN, float* gpos, float* gnorm,
                        float* gdiff) {
  const uint32_t np = a.width * a.height;
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  const float4 r = b.res[p];
  const uint32_t n = __float_as_uint(r.w);
  if (n == 0) return;
  uint32_t old = (a.frame == 0) ? 0u : sampleN[p];
  if (a.frame == 0) sampleN[p] = 0;
  const uint32_t nn = old + n;
  if (!(nn > old)) return;
  if (isinf(r.x) || isinf(r.y) || isinf(r.z)) return;
  const float rInf = 1.f / (float)nn;
  const float oInf = (float)old * rInf;
  float* q = result + 3 * (size_t)p;
  q[0] = fmaxf(rInf * r.x + oInf * q[0], 0.f);
  q[1] = fmaxf(rInf * r.y + oInf * q[1], 0.f);
  q[2] = fmaxf(rInf * r.z + oInf * q[2], 0.f);
  sampleN[p] = nn;
  if (a.moments) {  // running mean of acc^2 / n (the path's second moment weighted like its mean)
    const float fn = (float)n;
    float* m = b.m2 + 3 * (size_t)p;
    const float s0 = (r.x * r.x) / fn, s1 = (r.y * r.y) / fn, s2 = (r.z * r.z) / fn;
    m[0] = old ? rInf * s0 + oInf * m[0] : rInf * s0;
    m[1] = old ? rInf * s1 + oInf * m[1] : rInf * s1;
    m[2] = old ? rInf * s2 + oInf * m[2] : rInf * s2;
  }
  if (gpos) {
    float* planes[3] = {gpos, gnorm, gdiff};
    const float fn = (float)n;
    for (int k = 0; k < 3; k++) {
      float4 g = b.gbuf[3 * (size_t)p + k];
      float* o = planes[k] + 3 * (size_t)p;
      o[0] = rInf * (g.x * fn) + oInf * o[0];
      o[1] = rInf * (g.y * fn) + oInf * o[1];
      o[2] = rInf * (g.z * fn) + oInf * o[2];
    }
  }
}

// Filter-only mode (pt_applyPathQueueResult_kernel of
// src/cudaRTBDPTStreamBilat.cu:989-1051): the running means have no inf test
// here; direct light and 1 - potential are running means too; the first-hit
// planes hold this frame's values.
__global__ void k_apply_bilat(FrameArgs a, RenderBuffers b, float* result, uint32_t* sampleN, float* gpos,
                              float* gnorm, float* gdiff, float* gemis, float* direct, float* pot) {
  const uint32_t np = a.width * a.height;
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  const float4 r = b.res[p];
  const uint32_t n = __float_as_uint(r.w);
  if (n == 0) return;
  uint32_t old = (a.frame == 0) ? 0u : sampleN[p];
  if (a.frame == 0) sampleN[p] = 0;
  const uint32_t nn = old + n;
  if (!(nn > old)) return;
  const float rInf = 1.f / (float)nn;
  const float oInf = (float)old * rInf;
  const float4 ds = b.dsm[p];
  float* q = result + 3 * (size_t)p;
  q[0] = fmaxf(rInf * r.x + oInf * q[0], 0.f);
  q[1] = fmaxf(rInf * r.y + oInf * q[1], 0.f);
  q[2] = fmaxf(rInf * r.z + oInf * q[2], 0.f);
  pot[p] = fmaxf(rInf * (1.f - ds.w) + oInf * pot[p], 0.f);
  sampleN[p] = nn;
  float* dq = direct + 3 * (size_t)p;
  dq[0] = rInf * ds.x + oInf * dq[0];
  dq[1] = rInf * ds.y + oInf * dq[1];
  dq[2] = rInf * ds.z + oInf * dq[2];
  const float4 g0 = b.gbuf[3 * (size_t)p], g1 = b.gbuf[3 * (size_t)p + 1], g2 = b.gbuf[3 * (size_t)p + 2];
  const size_t o = 3 * (size_t)p;
  gpos[o] = g0.x, gpos[o + 1] = g0.y, gpos[o + 2] = g0.z;
  gnorm[o] = g1.x, gnorm[o + 1] = g1.y, gnorm[o + 2] = g1.z;
  gemis[o] = g0.w, gemis[o + 1] = g1.w, gemis[o + 2] = g2.w;
  gdiff[o] = g2.x, gdiff[o + 1] = g2.y, gdiff[o + 2] = g2.z;
}

// Unidirectional mode: one path per pixel, weights of the frame index.
__global__ void k_apply_pt(FrameArgs a, RenderBuffers b, float* result, uint32_t* sampleN) {
  using namespace gb;
  const uint32_t np = a.width * a.height;
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  const float4 r = b.res[p];
  const uint32_t n = __float_as_uint(r.w);
  if (n == 0) return;
  const f3 smp = ld3(r) / (float)n;
  const float rInf = 1.f / (float)(a.frame + 1);
  const float oInf = 1.f - rInf;
  float* q = result + 3 * (size_t)p;
  q[0] = fmaxf(rInf * smp.x + oInf * q[0], 0.f);
  q[1] = fmaxf(rInf * smp.y + oInf * q[1], 0.f);
  q[2] = fmaxf(rInf * smp.z + oInf * q[2], 0.f);
  sampleN[p] = a.frame + 1;  // frames so far (the reference keeps no count in this mode)
}

// Leaf records of the ordered walk, one thread each: 21 MB that would otherwise
// be gathered on the host and copied (hall: 332,180 records).
__global__ void k_ord_leaves(const float4* __restrict__ nodes, const float4* __restrict__ tris,
                             const uint32_t* __restrict__ bin, uint32_t n, float4* __restrict__ out) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const size_t i = bin[k];
  const float4 lo = nodes[2 * i], hi = nodes[2 * i + 1];
  const uint32_t first = __float_as_uint(lo.w), cnt = __float_as_uint(hi.w);
  const float4 p0 = tris[4 * (size_t)first], e0 = tris[4 * (size_t)first + 1], e1 = tris[4 * (size_t)first + 2];
  const bool many = cnt != 1u;  // several triangles: the record names them
  float4* r = out + 4 * (size_t)k;
  r[0] = make_float4(many ? __uint_as_float(cnt) : p0.x, p0.y, p0.z, e0.x);
  r[1] = make_float4(e0.y, e0.z, e1.x, e1.y);
  r[2] = make_float4(e1.z, lo.x, lo.y, lo.z);
  r[3] = make_float4(hi.x, hi.y, hi.z, __uint_as_float(many ? first | kOrdManyTris : first));
}

// How many of n random rays pass the pop bound, asked once per scene: every other
// one from anywhere in the scene's box, the rest from the middle of a random
// triangle, as most of a renderer's rays start (a model whose rays pass the bound
// may fill little of a large space).  Bound by the longest walk (146 visits reach
// the bound), so a warp a block spreads the rays over as many SMs as there are.
__global__ void k_probe_walks(DevScene S, uint32_t n, uint32_t* capped) {
  using namespace gb;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 lo = S.nodes[0], hi = S.nodes[1];
  float u[8];
  draw8(0u, 0u, i, 0u, kCamera, 0u, 0u, u);
  float sn, cs;
  sincos_p(kTwoPi * u[3], &sn, &cs);
  const float z = 2.f * u[4] - 1.f, q = sqrtf(1.f - z * z);
  const f3 d = mk(q * cs, q * sn, z);
  f3 o = mk(lo.x + (hi.x - lo.x) * u[0], lo.y + (hi.y - lo.y) * u[1], lo.z + (hi.z - lo.z) * u[2]);
  if (i & 1u) {
    const float4* t = S.tris + 4 * (size_t)min((uint32_t)(u[5] * (float)S.triN), S.triN - 1u);
    const float4 p0 = t[0], e0 = t[1], e1 = t[2];
    o = mk(p0.x + (e0.x + e1.x) / 3.f, p0.y + (e0.y + e1.y) / 3.f, p0.z + (e0.z + e1.z) / 3.f) + kBias * d;
  }
  OrdWalk w;
  uint2 stack[kOrdStack];
  w.any = false;
  w.eps = kBias;
  w.init(S, o, d, kInf);
  while (!w.capped() && !w.step(S, stack)) {
  }
  if (w.capped()) atomicAdd(capped, 1u);
}

__global__ void k_prob_view(const float* pot, uint32_t np, float minProb, float* out) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  const float v = fmaxf(minProb, pot[p]);
  out[3 * (size_t)p] = v;
  out[3 * (size_t)p + 1] = v;
  out[3 * (size_t)p + 2] = v;
}

// ---------------------------------------------------------------------------
// Caller-supplied rays by the ordered walk: a warp owns `chunk` of them (a
// multiple of 32), a lane takes the warp's next ray as its walk ends, and the
// warp's walks step together.  Bound like the bounce launches' walks, by issue;
// with a thread a ray (k_trace_rays) a warp waits for the longest of its 32
// walks.  A fixed share needs no counter in memory, and some 200 rays a warp even
// out.  A million rays in the hall 1.06 -> 0.85 ms.
__global__ void __launch_bounds__(kBlock, 4) k_trace_ord(DevScene S, const float* rays, uint32_t n, uint32_t chunk,
                                                         float maxDist, float eps, float* t, int32_t* tri, float* w,
                                                         float* u, float* v) {
  __shared__ uint32_t openN;
  if (threadIdx.x == 0) openN = 0;
  __syncthreads();
  const uint64_t first = (uint64_t)(blockIdx.x * (kBlock / 32) + threadIdx.x / 32) * chunk;
  if (first >= n) return;
  uint32_t next = (uint32_t)first;
  const uint32_t end = (uint32_t)min(first + chunk, (uint64_t)n);
  OrdWalk wk;
  uint2 stack[kOrdStack];
  wk.any = false;
  wk.eps = eps;
  bool has = false;
  uint32_t item = 0;
  for (;;) {
    wk.stop_long();
    const uint32_t idle = __ballot_sync(0xffffffffu, !has);
    if (next < end) {
      const uint32_t off = __popc(idle & lanemask_lt()), left = end - next;
      if (!has && off < left) {
        item = next + off;
        has = true;
        const float* r = rays + 6 * (size_t)item;
        wk.init_caller(S, mk(r[0], r[1], r[2]), mk(r[3], r[4], r[5]), maxDist);
      }
      next += min((uint32_t)__popc(idle), left);
    } else if (idle == 0xffffffffu) {
      break;
    }
#pragma unroll 1
    for (int k = 0; k < walk_steps<kWalkOrd>(); k++) {
      if (!wk.step_warp(S, stack, has)) continue;
      has = false;
      bool hit = wk.hit();
      TraceHit h;
      h.t = wk.minT;
      h.tri = wk.best;
      h.w = 1.f - wk.bu - wk.bv;
      h.u = wk.bu;
      h.v = wk.bv;
      if (wk.capped()) {
        // one in 64 of a block's rays waits for k_resolve_rays, more take the reference's walk
        if (atomicAdd(&openN, 1u) < chunk / 8u) {
          tri[item] = -2;
          continue;
        }
        uint32_t nn = 0, nt = 0;
        hit = trace_ref<false, false>(S, wk.o, wk.d, maxDist, eps, false, h, nn, nt);
      }
      t[item] = hit ? h.t : -1.f;
      tri[item] = hit ? (int32_t)h.tri : -1;
      w[item] = hit ? h.w : 0.f;
      u[item] = hit ? h.u : 0.f;
      v[item] = hit ? h.v : 0.f;
    }
  }
}

// Stand-alone TracePrimitive for caller-supplied rays.
template <bool kCount>
__global__ void k_trace_rays(DevScene S, const float* rays, uint32_t n, float maxDist, float eps, int cullback,
                             float* t, int32_t* tri, float* w, float* u, float* v, uint32_t* nodes,
                             uint32_t* trisTested) {
  __shared__ uint32_t openN;
  if (threadIdx.x == 0) openN = 0;
  __syncthreads();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* r = rays + 6 * (size_t)i;
  TraceHit h;
  uint32_t nn = 0, nt = 0;
  bool hit;
  if (S.traversal == 1 && S.wide && !cullback) {  // wide order (no back-face culling there)
    Walk4 wk;
    uint2 stack[kWideDepth];
    wk.init(mk(r[0], r[1], r[2]), mk(r[3], r[4], r[5]), maxDist, eps, stack);
    while (!wk.step<kCount>(S, stack, false, nn, nt)) {
    }
    hit = wk.hit();
    h.t = wk.minT;
    h.tri = wk.best;
    h.w = wk.bw;
    h.u = wk.bu;
    h.v = wk.bv;
  } else if (!kCount && S.ord && S.traversal == 0 && !cullback) {
    bool open = false;
    const f3 o = mk(r[0], r[1], r[2]), d = mk(r[3], r[4], r[5]);
    hit = trace_ord(S, o, d, maxDist, eps, h, &open);
    if (open) {
      // a few of a block's rays wait for k_resolve_rays, more take the reference's walk
      if (atomicAdd(&openN, 1u) < 4u) {
        tri[i] = -2;
        return;
      }
      hit = trace_ref<false, false>(S, o, d, maxDist, eps, false, h, nn, nt);
    }
  } else {
    hit = trace_ref<false, kCount>(S, mk(r[0], r[1], r[2]), mk(r[3], r[4], r[5]), maxDist, eps, cullback != 0, h,
                                   nn, nt);
  }
  t[i] = hit ? h.t : -1.f;
  tri[i] = hit ? (int32_t)h.tri : -1;
  w[i] = hit ? h.w : 0.f;
  u[i] = hit ? h.u : 0.f;
  v[i] = hit ? h.v : 0.f;
  if (kCount) {
    nodes[i] = nn;
    trisTested[i] = nt;
  }
}

int g_sm = 0;

// Idle lanes of a warp that trigger a refill in k_walk / k_tail (tuning
// knob, GBPT_WALK_REFILL, 1..32; 0 when unset).  Defaults, measured on the
// interior, hall and Cornell workloads: 2 (with carrying; before it 8, 4-10
// within 1%, 20 3-4% slower), 20 for the wide order (10-20 within 1%, 4 2-3%
// slower).
uint32_t walk_refill_env() {
  static uint32_t v = [] {
    const char* e = std::getenv("GBPT_WALK_REFILL");
    if (!e) return 0u;
    int x = std::atoi(e);
    return (uint32_t)(x < 1 ? 1 : x > 32 ? 32 : x);
  }();
  return v;
}

uint32_t grid_for(const void* kernel, size_t smem = 0) {
  int per = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kBlock, smem);
  if (per < 1) per = 1;
  return (uint32_t)(sm_count() * per);
}

}  // namespace

static std::atomic<uint64_t> g_launches{0};
void note_launches(uint32_t n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
uint64_t launch_count() { return g_launches.load(std::memory_order_relaxed); }

int sm_count() {
  if (!g_sm) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sm, cudaDevAttrMultiProcessorCount, dev);
    if (g_sm <= 0) g_sm = 1;
  }
  return g_sm;
}

// opens a kernel for the lists' shared memory
template <typename Kern>
cudaError_t cap_launchable(Kern kern) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CapShared));
}

cudaError_t launch_light_pass(const DevScene& S, const FrameArgs& a, const RenderBuffers& b, cudaStream_t st) {
  uint32_t threads = ((a.lightPaths + 31) / 32) * 32;
  if (threads == 0) threads = 32;
  float4* cache = b.cache[a.cacheSel];
  if (a.ordered && threads <= 128) {
    const cudaError_t e = cap_launchable(k_light<8, true>);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kLightBlocks);
    cfg.blockDim = dim3(threads * 8 / kLightBlocks);
    cfg.dynamicSmemBytes = sizeof(CapShared);
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kLightBlocks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    const cudaError_t le = cudaLaunchKernelEx(&cfg, k_light<8, true>, S, a, cache, b.cacheCap, b.ctr);
    if (le != cudaSuccess) return le;
  } else if (a.ordered) {
    k_light<1, true><<<1, threads, 0, st>>>(S, a, cache, b.cacheCap, b.ctr);
  } else {
    k_light<1, false><<<1, threads, 0, st>>>(S, a, cache, b.cacheCap, b.ctr);
  }
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_ord_leaves(const float4* nodes, const float4* tris, const uint32_t* bin, uint32_t n, float4* out,
                              cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_ord_leaves<<<(n + kBlock - 1) / kBlock, kBlock, 0, st>>>(nodes, tris, bin, n, out);
  note_launches(1);
  return cudaGetLastError();
}

// More of the 2,048 random rays than this past the bound, and the scene keeps the
// node-by-node walk, as resolving them costs more than the others gain.  Measured,
// node-by-node walk / ordered (100,000 rays; 640x360 passes, each of a new view), by
// their number: hall 0 1.69 / 1.97, finer interior 1 1.82 / 2.00, hair of 40,000
// strands 2 1.81 / 2.39, fur of 300,000 2 1.72 / 2.45; 2,000 crossing sticks 30 0.65
// / 2.03, longer hair 38 0.91 / 1.65, longer fur 58 0.87 / 1.26, hair 155 0.78 / 0.76,
// sticks 190 0.67 / 0.21, fur 241 0.76 / 0.43, 6,000 sticks 920 0.44 / 0.17 and in a
// large space 696 - / 0.16.
constexpr uint32_t kProbeRays = 2048, kMostCapped = 10;

bool walks_pass_bound(const DevScene& S, uint32_t* word, cudaStream_t st, cudaError_t* err) {
  if (S.nodeN <= kPopCap) return false;  // cannot
  uint32_t capped = 0;
  *err = cudaMemsetAsync(word, 0, 4, st);
  if (*err != cudaSuccess) return false;
  k_probe_walks<<<kProbeRays / 32, 32, 0, st>>>(S, kProbeRays, word);
  note_launches(1);
  *err = cudaGetLastError();
  if (*err == cudaSuccess) *err = cudaMemcpyAsync(&capped, word, 4, cudaMemcpyDeviceToHost, st);
  if (*err == cudaSuccess) *err = cudaStreamSynchronize(st);
  return *err == cudaSuccess && capped > kMostCapped;
}

cudaError_t launch_camera(const FrameArgs& a, const RenderBuffers& b, cudaStream_t st) {
  k_camera<<<(b.count + kBlock - 1) / kBlock, kBlock, 0, st>>>(a, b);
  note_launches(1);
  return cudaGetLastError();
}

// launch shapes, queried once per kernel
template <bool kCount, int kKind>
uint32_t walk_grid() {
  static uint32_t g = grid_for((const void*)k_walk<kCount, kKind>);
  return g;
}

template <bool kCount, int kKind, uint32_t kLater = kOpenNow>
uint32_t tail_grid() {
  static uint32_t g = grid_for((const void*)k_tail<kCount, kKind, kLater>);
  return g;
}

uint32_t shade_grid() {
  static uint32_t g = grid_for((const void*)k_shade);
  return g;
}

// persistent grid: every CTA that fits, or `ctasPerSm` per SM when that is
// fewer (requests that share the GPU leave SMs to each other)
uint32_t persistent_grid(uint32_t full, uint32_t ctasPerSm) {
  if (ctasPerSm == 0) return full;
  return std::min(full, (uint32_t)sm_count() * ctasPerSm);
}

template <bool kCount, int kKind>
void walk_variant(const DevScene& S, const RenderBuffers& b, int in, int shIn, int shReset, uint32_t bilat,
                  uint32_t refill, uint32_t ctas, uint32_t launch, uint32_t carrySteps, uint32_t later,
                  cudaStream_t st) {
  const uint32_t g = persistent_grid(walk_grid<kCount, kKind>(), ctas);
  k_walk<kCount, kKind><<<g, kBlock, 0, st>>>(S, b, in, shIn, shReset, bilat, refill, launch, carrySteps, later);
}

template <bool kCount, int kKind, uint32_t kLater = kOpenNow>
void tail_variant(const DevScene& S, const FrameArgs& a, const RenderBuffers& b, uint32_t K, cudaStream_t st) {
  const uint32_t g = persistent_grid(tail_grid<kCount, kKind, kLater>(), a.walkCtas);
  k_tail<kCount, kKind, kLater><<<g, kBlock, 0, st>>>(S, a, b, K, walk_refill_for(a.refill, kKind == kWalkWide));
}

uint32_t cap_grid() { return 4u * (uint32_t)sm_count(); }

// what becomes of walks past the pop bound: a tree of up to 2048 nodes cannot
// have any; the filter-only mode's direct-light sample and the learned
// allocator's path-length counts are added to as a path is shaded, so their
// paths cannot be run again
uint32_t open_rule(const DevScene& S, const FrameArgs& a) {
  if (S.nodeN <= kPopCap) return kOpenNow;
  return a.bilat || a.moments ? kOpenList : kOpenCheck;
}

cudaError_t launch_walk(const DevScene& S, const FrameArgs& a, const RenderBuffers& b, int in, int shIn,
                        int shReset, uint32_t launch, cudaStream_t st) {
  const uint32_t sd = a.bilat ? 1u : 0u;
  const bool wide = S.traversal == 1 && S.wide;
  const uint32_t rf = walk_refill_for(a.refill, wide);
  const uint32_t cs = b.carry[0] ? a.carrySteps : 0u;
  if (a.ordered) {
    walk_variant<false, kWalkOrd>(S, b, in, shIn, shReset, sd, rf, a.walkCtas, launch, cs, open_rule(S, a), st);
    if (open_rule(S, a) == kOpenList) {
      const cudaError_t e = cap_launchable(k_resolve);
      if (e != cudaSuccess) return e;
      k_resolve<<<cap_grid(), kCapThreads, sizeof(CapShared), st>>>(S, b, in, shIn, sd, launch);
      note_launches(1);
    }
  } else if (a.counting) {
    if (wide) walk_variant<true, kWalkWide>(S, b, in, shIn, shReset, sd, rf, a.walkCtas, launch, 0u, 0u, st);
    else walk_variant<true, kWalkRef>(S, b, in, shIn, shReset, sd, rf, a.walkCtas, launch, cs, 0u, st);
  } else {
    if (wide) walk_variant<false, kWalkWide>(S, b, in, shIn, shReset, sd, rf, a.walkCtas, launch, 0u, 0u, st);
    else walk_variant<false, kWalkRef>(S, b, in, shIn, shReset, sd, rf, a.walkCtas, launch, cs, 0u, st);
  }
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_tail(const DevScene& S, const FrameArgs& a, const RenderBuffers& b, uint32_t K, cudaStream_t st) {
  const bool wide = S.traversal == 1 && S.wide;
  if (a.ordered) {
    const uint32_t rule = open_rule(S, a);
    if (rule == kOpenNow) tail_variant<false, kWalkOrd, kOpenNow>(S, a, b, K, st);
    else if (rule == kOpenList) tail_variant<false, kWalkOrd, kOpenList>(S, a, b, K, st);
    else tail_variant<false, kWalkOrd, kOpenCheck>(S, a, b, K, st);
  } else if (a.counting) {
    if (wide) tail_variant<true, kWalkWide>(S, a, b, K, st);
    else tail_variant<true, kWalkRef>(S, a, b, K, st);
  } else {
    if (wide) tail_variant<false, kWalkWide>(S, a, b, K, st);
    else tail_variant<false, kWalkRef>(S, a, b, K, st);
  }
  note_launches(1);
  return cudaGetLastError();
}

bool checks_walks(const DevScene& S, const FrameArgs& a) { return a.ordered && open_rule(S, a) != kOpenNow; }

cudaError_t launch_verify(const DevScene& S, const RenderBuffers& b, uint32_t list, cudaStream_t st) {
  const cudaError_t e = cap_launchable(k_verify);
  if (e != cudaSuccess) return e;
  k_verify<<<cap_grid(), kCapThreads, sizeof(CapShared), st>>>(S, b, list);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_again(const DevScene& S, const FrameArgs& a, const RenderBuffers& b, cudaStream_t st) {
  const cudaError_t e = cap_launchable(k_again);
  if (e != cudaSuccess) return e;
  k_again<<<sm_count(), kCapThreads, sizeof(CapShared), st>>>(S, a, b);
  note_launches(1);
  return cudaGetLastError();
}

uint32_t walk_lanes() {
  return std::max(walk_grid<false, kWalkRef>(), walk_grid<false, kWalkOrd>()) * (uint32_t)kBlock;
}

void prepare_launches() {
  walk_grid<false, kWalkRef>();
  walk_grid<false, kWalkWide>();
  walk_grid<false, kWalkOrd>();
  walk_grid<true, kWalkRef>();
  walk_grid<true, kWalkWide>();
  tail_grid<false, kWalkRef>();
  tail_grid<false, kWalkWide>();
  tail_grid<false, kWalkOrd, kOpenNow>();
  tail_grid<false, kWalkOrd, kOpenList>();
  tail_grid<false, kWalkOrd, kOpenCheck>();
  tail_grid<true, kWalkRef>();
  tail_grid<true, kWalkWide>();
  shade_grid();
}

uint32_t tail_from(uint32_t eyeDepth, bool wide, bool ordered, int32_t requested, size_t paths, bool carrying,
                   bool beside) {
  // default for the ordered walk while carrying: a frame with fewer camera paths
  // than 1.5 x the tail grid's lanes (116,736) runs in the tail kernel alone, a
  // larger one hands over at bounce 3D/5 when D > 6, else never.  Measured (ms per
  // case; first bounce in the tail kernel): Cornell 64x64 pass, D = 8: 0 0.202, 2
  // 0.231, 4 0.254; Cornell 256x256 x 16: 0 3.62, 2 3.93, 4 4.03, 7 4.36;
  // unidirectional 333x217 x 8, D = 10: 0 4.49, 2 5.35, 5 6.19; 500x375 binary, D =
  // 6: 0 10.0, 4 9.40, none 9.64; interior 1024x768, D = 10: 0 4.20, 4 3.06, 5 2.88,
  // 6 2.80, 7 2.80; hall 1280x720, D = 5: 0 4.59, 4 3.06, none 2.94.
  //
  // A bidirectional frame traced beside others of its call need not end soon, and
  // bounce launches use the lanes better: from 3/4 of the tail's lanes (58,368
  // paths) on, D > 4, the tail starts at (D + 3) / 2.  Measured (ms an image, from 0
  // / from there): Cornell 256x256 x 16, D = 8 2.49 / 2.12; interior 256x256 x 8, D =
  // 8 4.74 / 4.10, D = 5 3.94 / 3.57; hall 256x256 x 8, D = 5 4.59 / 3.99; interior
  // 340x340 x 8, D = 5 5.70 / 4.71.  Below the line from 0 is as good or better
  // (interior 182x181 x 8, D = 8: 3.48 / 3.57; 256x192, D = 5: 3.37 / 3.35), as it is
  // for D <= 4 (215x215, D = 4: 2.80 / 3.01) and for unidirectional frames, which
  // shade little between walks (333x217: 2.89, from 2 3.16, from 6 3.58).
  //
  // default of the node-by-node walk while carrying: a frame with fewer camera paths
  // than the walk grid has lanes hands its paths to the tail kernel from bounce
  // 2 on, a larger one from bounce D/2 when D > 6, else never.  Measured with
  // carrying (Mpaths/s; the walk grid then had 194,560 lanes, now 155,648):
  // Cornell 256x256 (65,536 paths),
  // D = 8: from 2 204.6, 3 193.6, 4 180.6, 5 168.2; interior 1024x768, D = 10:
  // from 3 163.0, 4 167.5, 5 170.6, 6 169.7; hall 1280x720, D = 5: none 188.1
  // (launches past the cap: worse).  Against the rule without carrying: interior
  // 168.4 -> 172.3, Cornell 188.9 -> 194.6, hall and hall adaptive even.  The
  // same choice on the device (a shading launch switching once the live paths
  // fall below 1-3 x the lanes) cost Cornell 14 %: the host still issues the
  // skipped launches.
  // default without carrying, D > 6: from bounce D/2 - 1 in the reference
  // order, D/2 in the wide order; per-bounce launches throughout for D <= 6.
  // Measured in Mpaths/s (reference / wide order), tail kernel at three CTAs
  // per SM: interior, D = 10: from 4 174.3 / 169.6, from 5 170.6 / 174.8,
  // from 6 161.4 / 173.7; Cornell, D = 8: from 3 199.3 / 173.7, from 4 194.3
  // / 173.5; hall, D = 5: no tail 176.7 / 180.5, from 4 171.1 / 175.8, from 3
  // 158.9 (once few paths are alive the tail kernel's per-path schedule wins;
  // while many are, per-bounce launches keep more of them resident).
  static int v = [] {
    const char* e = std::getenv("GBPT_TAIL_FROM");
    return e ? std::atoi(e) : -2;
  }();
  if (requested >= 0) return (uint32_t)requested;
  if (v == -2 && carrying) {
    const size_t lanes = (size_t)tail_grid<false, kWalkOrd>() * kBlock;
    if (ordered && beside && eyeDepth > 4 && paths >= lanes * 3 / 4 && paths < lanes * 3 / 2) return (eyeDepth + 3) / 2;
    if (ordered && paths < lanes * 3 / 2) return 0u;
    if (!ordered && paths < walk_lanes()) return std::min(eyeDepth, 2u);
    return eyeDepth > 6 ? (ordered ? eyeDepth * 3 / 5 : eyeDepth / 2) : eyeDepth;
  }
  if (v == -2) return eyeDepth > 6 ? eyeDepth / 2 - (wide ? 0u : 1u) : eyeDepth;
  return v < 0 ? eyeDepth : (uint32_t)v;
}

uint32_t walk_refill_for(uint32_t requested, bool wide) {
  if (requested >= 1 && requested <= 32) return requested;
  if (walk_refill_env()) return walk_refill_env();
  return wide ? 20u : 2u;
}

cudaError_t launch_shade(const DevScene& S, const FrameArgs& a, const RenderBuffers& b, int in, uint32_t launch,
                         bool attach, cudaStream_t st) {
  const uint32_t g = shade_grid();
  k_shade<<<g, kBlock, 0, st>>>(S, a, b, in, launch, attach ? 1u : 0u);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_fold(const RenderBuffers& b, cudaStream_t st) {
  const uint32_t n = b.count ? b.count : b.cap;
  k_fold<<<(n + kBlock - 1) / kBlock, kBlock, 0, st>>>(b);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_apply(const FrameArgs& a, const RenderBuffers& b, float* result, uint32_t* sampleN, float* gpos,
                         float* gnorm, float* gdiff, cudaStream_t st) {
  const uint32_t np = a.width * a.height;
  k_apply<<<(np + kBlock - 1) / kBlock, kBlock, 0, st>>>(a, b, result, sampleN, gpos, gnorm, gdiff);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_apply_bilat(const FrameArgs& a, const RenderBuffers& b, float* result, uint32_t* sampleN,
                               float* gpos, float* gnorm, float* gdiff, float* gemis, float* direct, float* pot,
                               cudaStream_t st) {
  const uint32_t np = a.width * a.height;
  k_apply_bilat<<<(np + kBlock - 1) / kBlock, kBlock, 0, st>>>(a, b, result, sampleN, gpos, gnorm, gdiff, gemis,
                                                               direct, pot);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_apply_pt(const FrameArgs& a, const RenderBuffers& b, float* result, uint32_t* sampleN,
                            cudaStream_t st) {
  const uint32_t np = a.width * a.height;
  k_apply_pt<<<(np + kBlock - 1) / kBlock, kBlock, 0, st>>>(a, b, result, sampleN);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_prob_view(const float* pot, uint32_t np, float minProb, float* out, cudaStream_t st) {
  if (np == 0) return cudaSuccess;
  k_prob_view<<<(np + kBlock - 1) / kBlock, kBlock, 0, st>>>(pot, np, minProb, out);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_trace_rays(const DevScene& S, const float* rays, uint32_t n, float maxDist, float eps, int cullback,
                              float* t, int32_t* tri, float* w, float* u, float* v, uint32_t* nodes,
                              uint32_t* trisTested, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const uint32_t grid = n / kBlock + (n % kBlock != 0u);
  const bool ordered = !(nodes && trisTested) && S.ord && S.traversal == 0 && !cullback;
  if (ordered) {
    // Shares from two rays a lane of the grid on (311,296): at 400,000 rays hall
    // 0.56 -> 0.50 ms, interior 0.42 -> 0.37, at 1,500,000 1.43 -> 0.98 and 1.17 ->
    // 0.69; at 160,000, where no lane gets a second ray, a thread a ray takes 0.35
    // against 0.38.  Walks of trees of up to 2048 nodes are short and alike: Cornell
    // at 400,000 0.068 against 0.076 ms, at 1,500,000 even.
    static const uint32_t full = grid_for((const void*)k_trace_ord);
    if (n >= 2u * full * kBlock && S.nodeN > kPopCap) {
      const uint32_t warps = full * (kBlock / 32), chunk = ((n - 1) / warps / 32 + 1) * 32;
      k_trace_ord<<<full, kBlock, 0, st>>>(S, rays, n, chunk, maxDist, eps, t, tri, w, u, v);
    } else {
      k_trace_rays<false><<<grid, kBlock, 0, st>>>(S, rays, n, maxDist, eps, cullback, t, tri, w, u, v, nodes,
                                                     trisTested);
    }
    note_launches(1);
    const cudaError_t e = cap_launchable(k_resolve_rays);
    if (e != cudaSuccess) return e;
    k_resolve_rays<<<std::min<uint32_t>(grid, cap_grid()), kCapThreads, sizeof(CapShared), st>>>(
        S, rays, n, maxDist, eps, t, tri, w, u, v);
  } else if (nodes && trisTested) {
    k_trace_rays<true><<<grid, kBlock, 0, st>>>(S, rays, n, maxDist, eps, cullback, t, tri, w, u, v, nodes,
                                                  trisTested);
  } else {
    k_trace_rays<false><<<grid, kBlock, 0, st>>>(S, rays, n, maxDist, eps, cullback, t, tri, w, u, v, nodes,
                                                   trisTested);
  }
  note_launches(1);
  return cudaGetLastError();
}

}  // namespace gbpt
