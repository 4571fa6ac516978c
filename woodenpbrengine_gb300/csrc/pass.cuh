// pass.cuh — device pieces of one sample pass shared by the render kernels
// (render.cu) and the differentiable estimator (adjoint.cu): camera samples and
// rays, surface interactions of a hit, light pick and light sampling, the
// light evaluation for BSDF-sampled directions and the film gather.
#pragma once

#include "camera.cuh"
#include "common.cuh"
#include "sampler.cuh"
#include "shade.cuh"
#include "views.cuh"
#include "wpbr_sampling.h"

namespace wpbr {

namespace {

constexpr int kTB = 128;
// Resident blocks per SM of the spawn kernels (surface interaction and
// sampling, 127 registers unbounded): the light and environment sampling is
// a chain of dependent loads (CDF searches), so occupancy pays even with
// spills. 1080p full frame, RGB / Sampled64 Msamples/s: unbounded 1093 /
// 621, 8 blocks 1188 / 649, 12 blocks (40 registers) 1229 / 667, 14 blocks
// 1246 / 677 but the 256x256 frame 4% slower.
#ifndef WPBR_SPAWN_MIN_BLOCKS
#define WPBR_SPAWN_MIN_BLOCKS 12
#endif
// The same kernels compiled with the texture path (scenes with textured
// metal), whose EWA loops need registers. Textured scene, 1080p x 16 spp, ms:
// 5 blocks 9.47, 6 9.24, 7 9.13, 8 9.23, 10 9.30. (The other spawn kernel:
// 6 blocks 12.06, 8 11.84, 10 11.67, 12 11.68, 14 11.80.)
#ifndef WPBR_SPAWN_TEX_MIN_BLOCKS
#define WPBR_SPAWN_TEX_MIN_BLOCKS 7
#endif
// Textured spawns come in two builds. With few pixels in flight a launch lasts
// as long as its slowest warps: the wide one has a copy of every lookup and as
// many registers as it likes (95, none spilled). With many the compact one
// wins, at 7 blocks and with the lookups in loops (texture.cuh). Compact /
// wide, us: one RGB pass of 256 x 256 320 / 198, 512 x 512 374 / 269, 1080p 823 /
// 733; frames of 2 passes of 1080p 1,276 / 1,247, 4 of 1280 x 800 1,501 /
// 1,359, 16 (8 at a time) of 1001 x 563 3,082 / 3,076, of 1280 x 800 4,848 /
// 5,199, 4 of 1080p 2,232 / 2,373; Sampled64, one of 512 x 512 483 / 381, 4 of
// 1001 x 563 1,685 / 1,656, of 1280 x 800 2,838 / 2,905, of 1080p 5,489 / 5,622.
enum : int { kTexNone, kTexWide, kTexCompact };
constexpr uint64_t kTexWideMax = 1ull << 22, kTexWideMaxSpectral = 3ull << 20;  // pixels in flight
inline int tex_build(bool textured, bool spectral, uint64_t pixels) {
  return !textured ? kTexNone : (pixels <= (spectral ? kTexWideMaxSpectral : kTexWideMax) ? kTexWide : kTexCompact);
}
constexpr int spawn_min_blocks(int tex) {
  return tex == kTexNone ? WPBR_SPAWN_MIN_BLOCKS : (tex == kTexWide ? 1 : WPBR_SPAWN_TEX_MIN_BLOCKS);
}
// The differentiable estimator's spawn: forward 4.06 -> 3.84 ms at 12 blocks
// (512x512 x 16 spp).
#ifndef WPBR_ADJ_SPAWN_MIN_BLOCKS
#define WPBR_ADJ_SPAWN_MIN_BLOCKS 12
#endif
// ... and its reverse sweep: a 512 x 512 x 16 spp step 3.85 ms at 12 blocks, 10
// 3.91, 8 3.92, 6 3.96.
#ifndef WPBR_ADJ_BACK_MIN_BLOCKS
#define WPBR_ADJ_BACK_MIN_BLOCKS 12
#endif

struct PassCtx {
  SceneView S;
  BvhView Bv;
  Sampler rs;
  uint32_t W, H;
  FastDiv row;  // by W
  uint32_t* err;
};
inline PassCtx pass_ctx(const SceneView& S, const BvhView& Bv, wpbr_rng::Stream rs, uint32_t W, uint32_t H,
                        uint32_t* err) {
  return PassCtx{S, Bv, make_sampler(rs), W, H, fast_div(W), err};
}

__device__ __forceinline__ V3 ld3(const float* f, uint32_t i) { return V3{f[3 * i], f[3 * i + 1], f[3 * i + 2]}; }
__device__ __forceinline__ void st3(float* f, uint32_t i, V3 v) {
  f[3 * i] = v.x;
  f[3 * i + 1] = v.y;
  f[3 * i + 2] = v.z;
}
__device__ __forceinline__ RGB3 ldc(const float* f, uint32_t i) { return RGB3{f[3 * i], f[3 * i + 1], f[3 * i + 2]}; }
__device__ __forceinline__ void stc(float* f, uint32_t i, RGB3 c) {
  f[3 * i] = c.r;
  f[3 * i + 1] = c.g;
  f[3 * i + 2] = c.b;
}

__device__ __forceinline__ uint32_t prim_material(const SceneView& S, uint32_t prim) {
  return prim < S.ns ? S.sph_mat[prim] : S.tri_mat[prim - S.ns];
}

// ---- material-sorted pixel order ----------------------------------------------
// The reference shades each kind of surface in a job of its own over that
// kind's component group: one BSDF job per material kind
// (CBSDFConductorMicroface.cpp:84-115, CBSDFDielectricMicroface.cpp:84-115,
// CBSDFSpecularReflectance.cpp:63-93) after the sphere or the triangle
// surface-interaction job (CSSphere.cpp:122-186, CSTriangle.cpp:149-319).
// The wavefront shades the pixels of a pass in that grouping, tile by tile:
// after the camera traversal the pixels of every run of kCatTile are ordered
// by category = primitive kind x material type (2 x 5), camera misses (and
// scenes without lights) last, so the spawn and finish kernels' warps mostly
// run one code path. Within a category pixels keep their film order.
//
// One launch, a block a tile, no global atomics: at most ten of a tile's 256
// warps hold two categories, and a tile's pixels stay near each other. Over
// the whole film (a counting launch, then one that claimed runs by atomics)
// the order took 36 us of a 1080p pass. 1080p x 16 spp, ms: whole film full
// 10.70 / textured 9.19, tiles of 2,048 10.52 / 9.43, 8,192 10.20 / 9.02,
// 16,384 10.35 / 8.89, 32,768 10.32 / 8.87; 1001 x 563 Sampled64 3.44, 3.54,
// 3.45, 3.50, 3.52 (large tiles leave SMs idle). (The spawn kernel alone is
// slower for it, 91 -> 100 us: a tile's categories run side by side and its
// warps wait more for instructions.)
constexpr uint32_t kMatTypes = 5;                  // WPBR_MAT_CONDUCTOR .. WPBR_MAT_METAL_ISOTROPIC
constexpr uint32_t kPixCats = 2 * kMatTypes + 1;   // last: misses
constexpr uint32_t kCatBlock = 512, kCatItems = 16;  // pixels per thread
constexpr uint32_t kCatTile = kCatBlock * kCatItems;
// Films of fewer pixels are shaded in film order: four passes of 256 x 256 in
// film order / sorted, us: spheres 177 / 177, mesh 353 / 355, textured 396 /
// 384, of 200 x 180 151 / 148, 311 / 316, 346 / 338.
constexpr uint32_t kSortMinPixels = 1u << 17;

// order[]: the pixels of each tile grouped by category.
__global__ void __launch_bounds__(kCatBlock) k_cat_order(SceneView S, uint32_t n, const uint32_t* hit_prim,
                                                         uint32_t* order) {
  constexpr uint32_t kWarps = kCatBlock / 32, kRuns = kCatItems * kWarps;  // a run: 32 pixels
  constexpr uint32_t kPer = (kPixCats * kRuns + kCatBlock - 1) / kCatBlock;
  __shared__ uint32_t s_at[kPer * kCatBlock];  // per category and run: pixels, then their start
  __shared__ uint32_t s_sum[kWarps];
  const uint32_t base = blockIdx.x * kCatTile, lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  // a thread's loads go out together, level by level: hit, material, its type
  uint32_t prim[kCatItems], m[kCatItems], c[kCatItems];
#pragma unroll
  for (uint32_t k = 0; k < kCatItems; ++k) {
    const uint32_t i = base + k * kCatBlock + threadIdx.x;
    prim[k] = i < n && S.nlights ? hit_prim[i] : kNoHit;
  }
#pragma unroll
  for (uint32_t k = 0; k < kCatItems; ++k) {
    const bool sph = prim[k] < S.ns;
    const uint32_t* id = sph ? S.sph_mat + prim[k] : S.tri_mat + (prim[k] - S.ns);
    m[k] = prim[k] != kNoHit ? *id : 0u;
  }
#pragma unroll
  for (uint32_t k = 0; k < kCatItems; ++k) {
    const uint32_t t = prim[k] != kNoHit ? S.mats[m[k]].type : 0u;
    c[k] = (prim[k] < S.ns ? 0u : kMatTypes) + (t < kMatTypes ? t : kMatTypes - 1);
    if (prim[k] == kNoHit) c[k] = kPixCats - 1;
    if (base + k * kCatBlock + threadIdx.x >= n) c[k] = kPixCats;  // no pixel
  }
#pragma unroll
  for (uint32_t q = 0; q < kPer; ++q) s_at[q * kCatBlock + threadIdx.x] = 0;
  __syncthreads();
  uint32_t rank[kCatItems];
#pragma unroll
  for (uint32_t k = 0; k < kCatItems; ++k) {
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, c[k]);
    rank[k] = __popc(peers & ((1u << lane) - 1u));
    if (rank[k] == 0 && c[k] < kPixCats) s_at[c[k] * kRuns + k * kWarps + w] = __popc(peers);
  }
  __syncthreads();
  uint32_t v[kPer], sum = 0;
#pragma unroll
  for (uint32_t q = 0; q < kPer; ++q) {
    v[q] = s_at[threadIdx.x * kPer + q];
    sum += v[q];
  }
  uint32_t x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) s_sum[w] = x;
  __syncthreads();
  uint32_t run = x - sum;
#pragma unroll
  for (uint32_t q = 0; q < kWarps; ++q) run += q < w ? s_sum[q] : 0u;
#pragma unroll
  for (uint32_t q = 0; q < kPer; ++q) {
    s_at[threadIdx.x * kPer + q] = run;
    run += v[q];
  }
  __syncthreads();
#pragma unroll
  for (uint32_t k = 0; k < kCatItems; ++k)
    if (c[k] < kPixCats)
      order[base + s_at[c[k] * kRuns + k * kWarps + w] + rank[k]] = base + k * kCatBlock + threadIdx.x;
}

// Full interaction for the winning primitive: re-runs its intersection test
// (identical bits) and builds the surface interaction.
__device__ SurfInt make_si(const SceneView& S, uint32_t prim, V3 o, V3 d) {
  if (prim < S.ns) {
    V3 rlo, rld, ph;
    sphere_intersect(S.sph_w2o[prim], S.sph_r[prim], o, d, &rlo, &rld, &ph);
    return sphere_si(S.sph_o2w[prim], S.sph_w2o[prim], S.sph_r[prim], rld, ph);
  }
  uint32_t t = prim - S.ns;
  const uint32_t* ix = S.idx + 3 * (size_t)t;
  TriData td;
  uint32_t fl = S.tri_flags[t];
  td.has_ns = (fl & WPBR_MESH_NORMALS_TANGENTS) != 0;
  td.has_uv = (fl & WPBR_MESH_UVS) != 0;
  for (int k = 0; k < 3; ++k) {
    uint32_t v = ix[k];
    td.p[k] = V3{S.pos[3 * v], S.pos[3 * v + 1], S.pos[3 * v + 2]};
    td.n[k] = td.has_ns ? V3{S.nrm[3 * v], S.nrm[3 * v + 1], S.nrm[3 * v + 2]} : V3{0, 0, 0};
    td.s[k] = td.has_ns ? V3{S.tan[3 * v], S.tan[3 * v + 1], S.tan[3 * v + 2]} : V3{0, 0, 0};
    td.uv[k] = td.has_uv ? V2{S.uv[2 * v], S.uv[2 * v + 1]} : V2{0, 0};
  }
  float b0, b1, b2;
  tri_intersect(td.p[0], td.p[1], td.p[2], o, d, S.quirks, &b0, &b1, &b2);
  return triangle_si(td, d, b0, b1, b2);
}

// The material of a hit: the scene's, or for textured metal the conductor
// built from its textures at the hit's footprint (camera-ray differentials,
// sphere or uv mapping).
// TEX = kTexNone compiles the texture path out, for scenes without textured
// materials (the context knows: has_metal).
template <int TEX>
__device__ wpbr_material hit_material(const SceneView& S, uint32_t prim, uint32_t mid, const SurfInt& s,
                                      const RayD& r) {
  wpbr_material m = S.mats[mid];
  if (TEX == kTexNone || !WPBR_MAT_TEXTURED(m.type)) return m;
  SurfDiff D = surf_differentials(s, r);
  constexpr bool kCompact = TEX == kTexCompact;
  TexFootprint fp = prim < S.ns ? sphere_footprint<kCompact>(S.sph_w2o[prim], s, D) : uv_footprint(s, D);
  return metal_material<kCompact>(S.tex, m, fp);
}
// The part of a textured-metal material that varies per hit, packed in a
// float4 (alpha, k.rgb), and its inverse.
__device__ __forceinline__ float4 metal_pack(const wpbr_material& m) {
  return make_float4(m.alpha_x, m.k[0], m.k[1], m.k[2]);
}
__device__ __forceinline__ wpbr_material metal_unpack(float4 v) {
  wpbr_material e;
  e.type = WPBR_MAT_CONDUCTOR;
  e.alpha_x = v.x;
  e.alpha_y = v.x;
  for (int c = 0; c < 3; ++c) {
    e.R[c] = 1.0f;
    e.eta_i[c] = 1.0f;
    e.eta_t[c] = 1.5f;
  }
  e.k[0] = v.y;
  e.k[1] = v.z;
  e.k[2] = v.w;
  e.tex[0] = e.tex[1] = 0;
  return e;
}

// JobSamplerUpdateCameraSamples (CSSampler.cpp:7-23): pFilm = pixel + u2
__device__ __forceinline__ void camera_sample(const PassCtx& P, uint32_t pix, uint32_t pass, float* fx, float* fy) {
  uint32_t x;
  const uint32_t y = div_mod(pix, P.row, &x);
  float u0, u1;
  sample2d(P.rs, pix, pass, wpbr_rng::DIM_CAMERA, &u0, &u1);
  *fx = (float)x + u0;
  *fy = (float)y + u1;
}

// JobScatteringSampleLight (SScattering.cpp:82-88), index clamped
__device__ __forceinline__ uint32_t pick_light(const PassCtx& P, uint32_t pix, uint32_t pass) {
  uint32_t nl = P.S.nlights;
  if (nl == 1) return 0;  // whatever the sample
  float ul = sample1d(P.rs, pix, pass, wpbr_rng::DIM_LIGHT_PICK);
  float fl = (ul + 0.5f) * (float)(nl - 1);
  uint32_t li = (uint32_t)fl;
  return li > nl - 1 ? nl - 1 : li;
}

struct LightSample {
  V3 wi;
  RGB3 li;
  float pdf;
  bool ok;
};
__device__ LightSample sample_light(const PassCtx& P, const wpbr_light& lt, V3 p, uint32_t pix, uint32_t pass) {
  float u0, u1;
  sample2d(P.rs, pix, pass, wpbr_rng::DIM_LIGHT, &u0, &u1);
  LightSample s;
  s.wi = V3{0, 0, 0};
  s.li = rgb1(0.0f);
  s.pdf = 0.0f;
  s.ok = true;
  if (lt.type == WPBR_LIGHT_SPHERE) {
    sphere_light_sample(P.S.sph_o2w[lt.sphere_index], P.S.sph_r[lt.sphere_index], p, u0, u1, &s.wi, &s.pdf);
    s.li = RGB3{lt.Le[0], lt.Le[1], lt.Le[2]};
  } else {
    env_li_sample(P.S.env, P.S.quirks, u0, u1, &s.wi, &s.li, &s.pdf, &s.ok);
  }
  return s;
}

// Whether a light sample can contribute: the reference discards the looked-up
// radiance of an environment sample (CLightInfiniteArea.cpp:192-199), so
// without WPBR_Q_ENV_LI_SAMPLE_FIX its value is black whatever is drawn, and
// the fused passes leave out the draw (two CDF searches of about 20 dependent
// loads; the staged jobs record it).
__device__ __forceinline__ bool light_sample_counts(const SceneView& S, const wpbr_light& lt) {
  return lt.type == WPBR_LIGHT_SPHERE || (S.quirks & WPBR_Q_ENV_LI_SAMPLE_FIX);
}

__device__ void light_compute(const PassCtx& P, const wpbr_light& lt, V3 p, V3 wi, RGB3* li, float* pdf) {
  if (lt.type == WPBR_LIGHT_SPHERE) {
    *pdf = sphere_light_pdf(P.S.sph_o2w[lt.sphere_index], P.S.sph_r[lt.sphere_index], p, P.S.quirks);
    *li = RGB3{lt.Le[0], lt.Le[1], lt.Le[2]};
  } else {
    env_li_compute(P.S.env, wi, li, pdf);
  }
}

__device__ __forceinline__ uint32_t light_prim(const wpbr_light& lt) {
  return lt.type == WPBR_LIGHT_SPHERE ? lt.sphere_index : 0xFFFFFFFEu;
}

// JobAccumalateLIFromSamples (CSFilm.cpp:70-122) as a gather: each pixel
// sums, in the reference's row-major sample order, the Mitchell-weighted
// samples of its 32x32 tile whose splat footprint covers it. A sample's
// footprint is clipped to its own tile, so a block takes a tile's width and
// stages, once per sample of its rows and of two rows above and below in the
// tile: the value and the Mitchell factors of the five pixel columns and rows
// the sample can reach, zero outside the footprint. A thread then walks the
// samples around a column of two pixels and adds each to every pixel it can
// reach: weight = the same product of two factors, the same additions in the
// same order. Samples outside a pixel's footprint and black ones add a zero,
// which changes no sum (a sum that starts at +0 never becomes -0), so nothing
// is tested per pair; only a block that holds a non-finite sample, whose
// product with a zero weight would be NaN, takes the tested walk.
//
// What bounds it: issue slots (70 % busy) and the shared loads, which the two
// pixels of a thread share. 1920 x 1080: 72 us (77 M instructions) with one
// thread a pixel testing 25 staged samples over 16 x 16 blocks, 60 us (41 M)
// with two pixels a thread; one a thread 69 us, four 75 us (80 registers, 5
// blocks an SM). Frames of 16 spp, 72 -> 60 us: full 11.84 -> 11.63 ms,
// textured 10.53 -> 10.13.
constexpr int kFilmTile = 32;                // tile width: the reference's film tiles
constexpr int kFilmPix = 2;                  // pixels (one column) per thread
constexpr uint64_t kFilmFewBlocks = 608;     // 4 a SM
constexpr int kFilmPitch = kFilmTile + 4;    // staged columns, two empty ones either side

// One dimension of the MitchellFilter of radius 2, B = C = 1/3 (CSFilm.h:20-44),
// at a distance of t <= 2.5 pixels: both branches as one polynomial
// (the inner one adds a zero linear term).
__device__ __forceinline__ float mitchell_at(float t) {
  const float B = (float)(1.0 / 3.0f), C = (float)(1.0 / 3.0f);
  const bool outer = t > 1.0f;
  const float a = outer ? -B - 6.0f * C : 12.0f - 9.0f * B - 6.0f * C;
  const float b = outer ? 6.0f * B + 30.0f * C : -18.0f + 12.0f * B + 6.0f * C;
  const float c = outer ? -12.0f * B - 48.0f * C : 0.0f;
  const float d = outer ? 8.0f * B + 24.0f * C : 6.0f - 2.0f * B;
  return (((((a * t) * t) * t + ((b * t) * t)) + (c * t)) + d) * (1.0f / 6.0f);
}
// Its inner branch, t <= 1.
__device__ __forceinline__ float mitchell_inner(float t) {
  const float B = (float)(1.0 / 3.0f), C = (float)(1.0 / 3.0f);
  return (((((12.0f - 9.0f * B - 6.0f * C) * t) * t) * t + (((-18.0f + 12.0f * B + 6.0f * C) * t) * t)) +
          (6.0f - 2.0f * B)) *
         (1.0f / 6.0f);
}
// The factors of the pixels s - 2 .. s + 2 for a film position f in [s, s + 1]
// whose footprint is clipped to [lo, hi]. The two middle pixels lie within 1 of
// it; of the outermost two the footprint holds one, both only when f lies
// exactly half way.
__device__ __forceinline__ void film_factors(float f, int s, int lo, int hi, float m[5]) {
  const float d0 = f - 0.5f;
  const int pmin = max((int)ceilf(d0 - 2.0f), lo), pmax = min((int)floorf(d0 + 2.0f), hi);
  const float fs = (float)s;
  const bool first = s - 2 >= pmin && s - 2 <= pmax, last = s + 2 >= pmin && s + 2 <= pmax;
  const float e = mitchell_at(fabsf((first ? fs - 2.0f : fs + 2.0f) - f));
  m[0] = first ? e : 0.0f;
  m[1] = s - 1 >= pmin && s - 1 <= pmax ? mitchell_at(fabsf((fs - 1.0f) - f)) : 0.0f;
  m[2] = s >= pmin && s <= pmax ? mitchell_inner(fabsf(fs - f)) : 0.0f;
  m[3] = s + 1 >= pmin && s + 1 <= pmax ? mitchell_inner(fabsf((fs + 1.0f) - f)) : 0.0f;
  m[4] = last ? e : 0.0f;
  if (first && last) m[4] = mitchell_at(fabsf((fs + 2.0f) - f));
}

// ROWS: pixel rows of a block.
template <int ROWS>
__global__ void __launch_bounds__(kFilmTile * ROWS / kFilmPix) k_film_tiles(uint32_t W, uint32_t H, const float2* pf,
                                                                             const float4* Lb, float4* acc) {
  constexpr int kThreads = kFilmTile * ROWS / kFilmPix;
  constexpr int kRows = ROWS + 4;
  __shared__ float4 s_L[kRows * kFilmPitch], s_my[kRows * kFilmPitch];  // rows 0-3 of a sample's five
  __shared__ float s_my4[kRows * kFilmPitch], s_mx[5][kRows * kFilmPitch];
  const int bx0 = (int)blockIdx.x * kFilmTile, by0 = (int)blockIdx.y * ROWS;
  const int ty0 = by0 / 32 * 32;
  const int tx1 = min(bx0 + 31, (int)W - 1), ty1 = min(ty0 + 31, (int)H - 1);
  bool odd = false;
  for (int i = (int)threadIdx.x; i < kRows * kFilmPitch; i += kThreads) {
    const int sx = bx0 - 2 + i % kFilmPitch, sy = by0 - 2 + i / kFilmPitch;
    float mx[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f}, my[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (sx >= bx0 && sx <= tx1 && sy >= ty0 && sy <= ty1) {
      const size_t sp = (size_t)sy * W + sx;
      const float2 f = pf[sp];
      c = Lb[sp];
      film_factors(f.x, sx, bx0, tx1, mx);
      film_factors(f.y, sy, ty0, ty1, my);
      odd |= !(isfinite(c.x) && isfinite(c.y) && isfinite(c.z));
    }
    s_L[i] = c;
    s_my[i] = make_float4(my[0], my[1], my[2], my[3]);
    s_my4[i] = my[4];
#pragma unroll
    for (int k = 0; k < 5; ++k) s_mx[k][i] = mx[k];
  }
  const bool tested = __syncthreads_or(odd);
  const int lx = (int)threadIdx.x % kFilmTile, ly = (int)threadIdx.x / kFilmTile * kFilmPix;
  const int x = bx0 + lx, y = by0 + ly;
  if (x >= (int)W || y >= (int)H) return;
  float4 a[kFilmPix];
#pragma unroll
  for (int p = 0; p < kFilmPix; ++p)
    a[p] = y + p < (int)H ? acc[(size_t)(y + p) * W + x] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (!tested) {
    // sample rows y - 2 .. y + 3 (outer), columns x - 2 .. x + 2 (inner):
    // pixel p is row 4 - (r - p) and the column 4 - dx of a sample's reach
#pragma unroll
    for (int r = 0; r < kFilmPix + 4; ++r)
#pragma unroll
      for (int dx = 0; dx < 5; ++dx) {
        const int i = (ly + r) * kFilmPitch + lx + dx;
        const float4 c = s_L[i], m = s_my[i];
        const float my[5] = {m.x, m.y, m.z, m.w, s_my4[i]}, mx = s_mx[4 - dx][i];
#pragma unroll
        for (int p = 0; p < kFilmPix; ++p) {
          const int k = 4 - r + p;
          if (k < 0 || k > 4) continue;
          const float w = mx * my[k];
          a[p].x = a[p].x + c.x * w;
          a[p].y = a[p].y + c.y * w;
          a[p].z = a[p].z + c.z * w;
          a[p].w = a[p].w + w;
        }
      }
  } else {
    for (int p = 0; p < kFilmPix; ++p)
      for (int dy = 0; dy < 5; ++dy)
        for (int dx = 0; dx < 5; ++dx) {
          const int sx = x - 2 + dx, sy = y + p - 2 + dy;
          if (y + p >= (int)H || sx < bx0 || sx > tx1 || sy < ty0 || sy > ty1) continue;
          const float2 f = pf[(size_t)sy * W + sx];
          const float fx0 = f.x - 0.5f, fy0 = f.y - 0.5f;
          if (x < (int)ceilf(fx0 - 2.0f) || x > (int)floorf(fx0 + 2.0f) || y + p < (int)ceilf(fy0 - 2.0f) ||
              y + p > (int)floorf(fy0 + 2.0f))
            continue;
          const int i = (ly + p + dy) * kFilmPitch + lx + dx;
          const float4 m = s_my[i];
          const int k = 4 - dy;
          const float my = k == 0 ? m.x : (k == 1 ? m.y : (k == 2 ? m.z : (k == 3 ? m.w : s_my4[i])));
          const float w = s_mx[4 - dx][i] * my;
          const float4 c = s_L[i];
          if (!rblack(RGB3{c.x, c.y, c.z})) {
            a[p].x = a[p].x + c.x * w;
            a[p].y = a[p].y + c.y * w;
            a[p].z = a[p].z + c.z * w;
          }
          a[p].w = a[p].w + w;
        }
  }
#pragma unroll
  for (int p = 0; p < kFilmPix; ++p)
    if (y + p < (int)H) acc[(size_t)(y + p) * W + x] = a[p];
}
// Blocks of 16 pixel rows, of 8 where 16 would leave SMs without a block.
inline void film_tiles_launch(uint32_t W, uint32_t H, const float2* pf, const float4* Lb, float4* acc, cudaStream_t st) {
  const unsigned nx = div_up(W, kFilmTile);
  if ((uint64_t)nx * div_up(H, 16) >= kFilmFewBlocks)
    k_film_tiles<16><<<dim3(nx, div_up(H, 16)), kFilmTile * 16 / kFilmPix, 0, st>>>(W, H, pf, Lb, acc);
  else
    k_film_tiles<8><<<dim3(nx, div_up(H, 8)), kFilmTile * 8 / kFilmPix, 0, st>>>(W, H, pf, Lb, acc);
}

// Shadow rays of a pass, queued densely: a kernel that decides per pixel
// whether to trace a ray pushes only the rays it traces (one atomic per warp
// and call) with the slot of their result (2 * pixel + branch), and the
// traversal walks just the queue, so its warps do not refill lanes with
// empty slots. All lanes that reach a push call it, each with its own
// `want`.
struct ShadowQueue {
  float4* rays;     // 2 float4 per queued ray
  uint32_t* map;    // result slot of each queued ray
  uint32_t* count;  // rays queued in this pass (zeroed before the pass)
  __device__ __forceinline__ void push(bool want, uint32_t slot, V3 o, V3 d) const {
    const uint32_t act = __activemask();
    const uint32_t m = __ballot_sync(act, want);
    if (!m) return;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t leader = __ffs(m) - 1u;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(count, (uint32_t)__popc(m));
    base = __shfl_sync(act, base, leader);
    if (!want) return;
    const uint32_t q = base + __popc(m & ((1u << lane) - 1u));
    rays[2 * (size_t)q] = make_float4(o.x, o.y, o.z, 0.0f);
    rays[2 * (size_t)q + 1] = make_float4(d.x, d.y, d.z, inf_());
    map[q] = slot;
  }
};

// Camera rays generated inside the persistent traversal's ray source.
struct CameraSrc {
  PassCtx P;
  const uint32_t* pass_dev;
  __device__ __forceinline__ uint32_t limit(uint32_t n) const { return n; }
  __device__ __forceinline__ void load(uint32_t pix, float4* o, float4* d) const {
    float fx, fy;
    camera_sample(P, pix, *pass_dev, &fx, &fy);
    RayD r = camera_ray(P.S.cam, fx, fy);
    *o = make_float4(r.o.x, r.o.y, r.o.z, 0.0f);
    *d = make_float4(r.d.x, r.d.y, r.d.z, inf_());
  }
};

}  // namespace

}  // namespace wpbr
