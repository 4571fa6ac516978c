// render.cu — the per-sample job list of MEngine::render
// (WoodenPBREngine/MEngine.cpp:380-448) as wavefront kernels.
//
// Two forms share the same device functions:
//  * the staged path (wpbr_job_run): one kernel per reference job group over
//    per-pixel state buffers, each recordable for stage-by-stage parity;
//  * the fused path (wpbr_render_pass): camera+primary traversal, shading +
//    sample generation (spawn), one traversal launch for both shadow rays,
//    MIS finish, film gather — five kernels per sample pass (six on large films), captured once as
//    a CUDA graph that reads the pass index from device memory.
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "ctx.hpp"
#include "pass.cuh"
#include "pass_groups.hpp"
#include "traverse.cuh"
#include "traverse_persistent.cuh"

namespace wpbr {

namespace {

// Staged-path field slots (float and uint buffers in RenderState).
enum FF {
  F_PFILM, F_RAY_O, F_RAY_D, F_RAY_DX, F_RAY_DY, F_HIT_T, F_SI_P, F_SI_N, F_SI_WO, F_SI_SN, F_SI_SDPDU, F_SI_DPDU,
  F_SI_DPDV, F_SI_DNDU, F_SI_DNDV, F_FRAME, F_LE, F_L_WI, F_L_LI, F_L_PDF, F_L_F, F_L_FPDF, F_B_WI, F_B_F, F_B_PDF,
  F_B_LI, F_B_LPDF, F_L, F_MAT, F_COUNT
};
constexpr int kFW_h[F_COUNT] = {2, 3, 3, 3, 3, 1, 3, 3, 3, 3, 3, 3, 3, 3, 3, 9, 3, 3, 3, 1, 3, 1, 3, 3, 1, 3, 1, 3, 4};
__constant__ int kFW_d[F_COUNT] = {2, 3, 3, 3, 3, 1, 3, 3, 3, 3, 3, 3, 3, 3, 3, 9, 3, 3, 3, 1, 3, 1, 3, 3, 1, 3, 1, 3, 4};
#ifdef __CUDA_ARCH__
#define kFW kFW_d
#else
#define kFW kFW_h
#endif
enum UF { U_HIT_PRIM, U_LIGHT_IDX, U_L_FLAGS, U_B_FLAGS, U_LOK, U_COUNT };

struct Staged {
  float* f[F_COUNT];
  uint32_t* u[U_COUNT];
};

__device__ __forceinline__ uint32_t trace_closest(const PassCtx& P, V3 o, V3 d) {
  HitRec h = P.Bv.max_depth < 60 ? trace_ray<false, 64>(P.S, P.Bv, o, d, inf_(), nullptr, nullptr, P.err)
                                 : trace_ray<false, 256>(P.S, P.Bv, o, d, inf_(), nullptr, nullptr, P.err);
  return h.prim;
}

// ============================== staged jobs =================================
#define kNaN __int_as_float(0x7fc00000)

__global__ void kj_camera(PassCtx P, uint32_t pass, Staged G) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H) return;
  for (int f = 0; f < F_COUNT; ++f)
    for (int c = 0; c < kFW[f]; ++c) G.f[f][(size_t)pix * kFW[f] + c] = kNaN;
  for (int u = 0; u < U_COUNT; ++u) G.u[u][pix] = 0xFFFFFFFFu;
  float fx, fy;
  camera_sample(P, pix, pass, &fx, &fy);
  RayD r = camera_ray(P.S.cam, fx, fy);
  G.f[F_PFILM][2 * pix] = fx;
  G.f[F_PFILM][2 * pix + 1] = fy;
  st3(G.f[F_RAY_O], pix, r.o);
  st3(G.f[F_RAY_D], pix, r.d);
  st3(G.f[F_RAY_DX], pix, r.dxd);
  st3(G.f[F_RAY_DY], pix, r.dyd);
  stc(G.f[F_L], pix, rgb1(0.0f));
}

__global__ void kj_collide(PassCtx P, Staged G) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H) return;
  V3 o = ld3(G.f[F_RAY_O], pix), d = ld3(G.f[F_RAY_D], pix);
  HitRec h = P.Bv.max_depth < 60 ? trace_ray<false, 64>(P.S, P.Bv, o, d, inf_(), nullptr, nullptr, P.err)
                                 : trace_ray<false, 256>(P.S, P.Bv, o, d, inf_(), nullptr, nullptr, P.err);
  G.u[U_HIT_PRIM][pix] = h.prim;
  G.f[F_HIT_T][pix] = h.t;
  if (h.prim == kNoHit) return;
  SurfInt s = make_si(P.S, h.prim, o, d);
  st3(G.f[F_SI_P], pix, s.p);
  st3(G.f[F_SI_N], pix, s.n);
  st3(G.f[F_SI_WO], pix, s.wo);
  st3(G.f[F_SI_SN], pix, s.sn);
  st3(G.f[F_SI_SDPDU], pix, s.sdpdu);
  st3(G.f[F_SI_DPDU], pix, s.dpdu);
  st3(G.f[F_SI_DPDV], pix, s.dpdv);
  st3(G.f[F_SI_DNDU], pix, s.dndu);
  st3(G.f[F_SI_DNDV], pix, s.dndv);
}

__global__ void kj_emitted(PassCtx P, Staged G) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H) return;
  if (G.u[U_HIT_PRIM][pix] != kNoHit || !P.S.has_env) return;
  RGB3 le = env_le(P.S.env, ld3(G.f[F_RAY_D], pix));
  stc(G.f[F_LE], pix, le);
  stc(G.f[F_L], pix, radd(ldc(G.f[F_L], pix), le));
}

__device__ __forceinline__ Frame load_frame(const float* f, uint32_t pix) {
  const float* q = f + 9 * (size_t)pix;
  return Frame{V3{q[0], q[1], q[2]}, V3{q[3], q[4], q[5]}, V3{q[6], q[7], q[8]}};
}

__global__ void kj_bsdf_setup(PassCtx P, Staged G) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H || G.u[U_HIT_PRIM][pix] == kNoHit) return;
  uint32_t prim = G.u[U_HIT_PRIM][pix];
  uint32_t mid = prim_material(P.S, prim);
  if (WPBR_MAT_TEXTURED(P.S.mats[mid].type)) {
    // JobComputeDifferentialsForSurfInter + the uv mapping jobs +
    // JobGenerateBSDFMaterialMetal (MEngine.cpp:399-403)
    RayD r = camera_ray(P.S.cam, G.f[F_PFILM][2 * pix], G.f[F_PFILM][2 * pix + 1]);
    SurfInt hs = make_si(P.S, prim, r.o, r.d);
    float4 v = metal_pack(hit_material<kTexWide>(P.S, prim, mid, hs, r));
    float* q = G.f[F_MAT] + 4 * (size_t)pix;
    q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;
  }
  SurfInt s;
  s.sdpdu = ld3(G.f[F_SI_SDPDU], pix);
  s.sn = ld3(G.f[F_SI_SN], pix);
  Frame fr = bsdf_frame(s);
  float* q = G.f[F_FRAME] + 9 * (size_t)pix;
  q[0] = fr.ss.x; q[1] = fr.ss.y; q[2] = fr.ss.z;
  q[3] = fr.ts.x; q[4] = fr.ts.y; q[5] = fr.ts.z;
  q[6] = fr.ns.x; q[7] = fr.ns.y; q[8] = fr.ns.z;
}

__global__ void kj_sample_light(PassCtx P, uint32_t pass, Staged G) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H || G.u[U_HIT_PRIM][pix] == kNoHit || P.S.nlights == 0) return;
  uint32_t li = pick_light(P, pix, pass);
  G.u[U_LIGHT_IDX][pix] = li;
  LightSample ls = sample_light(P, P.S.lights[li], ld3(G.f[F_SI_P], pix), pix, pass);
  st3(G.f[F_L_WI], pix, ls.wi);
  stc(G.f[F_L_LI], pix, ls.li);
  G.f[F_L_PDF][pix] = ls.pdf;
  G.u[U_LOK][pix] = ls.ok ? 1u : 0u;
  G.u[U_L_FLAGS][pix] = 0u;
}

__global__ void kj_shadow_light(PassCtx P, Staged G) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H || G.u[U_HIT_PRIM][pix] == kNoHit || P.S.nlights == 0) return;
  if (!G.u[U_LOK][pix] || rblack(ldc(G.f[F_L_LI], pix))) return;
  V3 wi = ld3(G.f[F_L_WI], pix);
  V3 o = add(ld3(G.f[F_SI_P], pix), mul(wi, (float)0.1));
  uint32_t hp = trace_closest(P, o, wi);
  uint32_t lp = light_prim(P.S.lights[G.u[U_LIGHT_IDX][pix]]);
  G.u[U_L_FLAGS][pix] = 1u | ((hp == kNoHit || hp == lp) ? 2u : 0u);
}

__device__ __forceinline__ wpbr_material staged_material(const PassCtx& P, const Staged& G, uint32_t pix) {
  const wpbr_material& m = P.S.mats[prim_material(P.S, G.u[U_HIT_PRIM][pix])];
  if (!WPBR_MAT_TEXTURED(m.type)) return m;
  const float* q = G.f[F_MAT] + 4 * (size_t)pix;
  return metal_unpack(make_float4(q[0], q[1], q[2], q[3]));
}

__global__ void kj_bsdf_compute(PassCtx P, Staged G) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H || G.u[U_HIT_PRIM][pix] == kNoHit || P.S.nlights == 0) return;
  if (!(G.u[U_L_FLAGS][pix] & 2u)) return;
  Frame fr = load_frame(G.f[F_FRAME], pix);
  wpbr_material m = staged_material(P, G, pix);
  float pdf;
  RGB3 f = bsdf_eval(m, to_local(fr, ld3(G.f[F_SI_WO], pix)), to_local(fr, ld3(G.f[F_L_WI], pix)), &pdf);
  stc(G.f[F_L_F], pix, f);
  G.f[F_L_FPDF][pix] = pdf;
}

__global__ void kj_integrate_light(PassCtx P, Staged G) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H || G.u[U_HIT_PRIM][pix] == kNoHit || P.S.nlights == 0) return;
  if (!(G.u[U_L_FLAGS][pix] & 2u)) return;
  float bpdf = G.f[F_L_FPDF][pix];
  if (bpdf == 0.0f) return;
  float lpdf = G.f[F_L_PDF][pix];
  float w = power_heuristic(lpdf, bpdf);
  RGB3 c = rmuls(rmul(ldc(G.f[F_L_LI], pix), ldc(G.f[F_L_F], pix)), w / lpdf);
  stc(G.f[F_L], pix, radd(ldc(G.f[F_L], pix), c));
}

__global__ void kj_sample_bsdf(PassCtx P, uint32_t pass, Staged G) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H || G.u[U_HIT_PRIM][pix] == kNoHit || P.S.nlights == 0) return;
  Frame fr = load_frame(G.f[F_FRAME], pix);
  wpbr_material m = staged_material(P, G, pix);
  float u0, u1;
  sample2d(P.rs, pix, pass, wpbr_rng::DIM_BSDF, &u0, &u1);
  V3 wi_l;
  float pdf;
  bool valid;
  RGB3 f = bsdf_sample(m, to_local(fr, ld3(G.f[F_SI_WO], pix)), u0, u1, &wi_l, &pdf, &valid);
  st3(G.f[F_B_WI], pix, to_world(fr, wi_l));
  stc(G.f[F_B_F], pix, f);
  G.f[F_B_PDF][pix] = pdf;
  G.u[U_B_FLAGS][pix] = valid ? 1u : 0u;
}

__global__ void kj_shadow_bsdf(PassCtx P, Staged G) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H || G.u[U_HIT_PRIM][pix] == kNoHit || P.S.nlights == 0) return;
  uint32_t fl = G.u[U_B_FLAGS][pix];
  if (!(fl & 1u)) return;
  V3 wi = ld3(G.f[F_B_WI], pix);
  V3 o = add(ld3(G.f[F_SI_P], pix), mul(wi, (float)0.01));
  uint32_t hp = trace_closest(P, o, wi);
  uint32_t lp = light_prim(P.S.lights[G.u[U_LIGHT_IDX][pix]]);
  G.u[U_B_FLAGS][pix] = fl | 2u | ((hp == kNoHit || hp == lp) ? 4u : 0u);
}

__global__ void kj_light_compute(PassCtx P, Staged G) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H || G.u[U_HIT_PRIM][pix] == kNoHit || P.S.nlights == 0) return;
  if (!(G.u[U_B_FLAGS][pix] & 4u)) return;
  RGB3 li;
  float pdf;
  light_compute(P, P.S.lights[G.u[U_LIGHT_IDX][pix]], ld3(G.f[F_SI_P], pix), ld3(G.f[F_B_WI], pix), &li, &pdf);
  stc(G.f[F_B_LI], pix, li);
  G.f[F_B_LPDF][pix] = pdf;
}

__global__ void kj_integrate_bsdf(PassCtx P, Staged G) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H || G.u[U_HIT_PRIM][pix] == kNoHit || P.S.nlights == 0) return;
  if (!(G.u[U_B_FLAGS][pix] & 4u)) return;
  RGB3 li = ldc(G.f[F_B_LI], pix);
  if (rblack(li)) return;
  float bpdf = G.f[F_B_PDF][pix];
  float w = (bpdf == 1.0f) ? 1.0f : power_heuristic(bpdf, G.f[F_B_LPDF][pix]);
  RGB3 c = rmuls(rmul(li, ldc(G.f[F_B_F], pix)), w / bpdf);
  stc(G.f[F_L], pix, radd(ldc(G.f[F_L], pix), c));
}

__global__ void kj_film_pack(PassCtx P, Staged G, float2* pf, float4* Lb) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H) return;
  pf[pix] = make_float2(G.f[F_PFILM][2 * pix], G.f[F_PFILM][2 * pix + 1]);
  RGB3 L = ldc(G.f[F_L], pix);
  Lb[pix] = make_float4(L.r, L.g, L.b, 0.0f);
}


// ============================== fused pass ==================================
// Compact per-pixel state written by k_spawn and read by k_finish: one
// 128-byte line a pixel, what the BSDF branch needs in its first half and the
// light branch's in the second, so that a pixel moves only the sectors of the
// branches it has; camera misses move none (they are told by hit_prim). With
// seven float4 a pixel, all written and read for every hit, the 1080p full
// frame's finish read 267 MB a pass (57 us).
constexpr int kStateF4 = kPassStateF4;
enum : int { ST_BWI, ST_P, ST_BF, ST_METAL, ST_LI, ST_WI, ST_WO };  // float4 of a pixel's state
static_assert(kStateF4 == 8, "a 128-byte line");
enum : uint32_t { SF_TRACE_L = 2u, SF_TRACE_B = 4u, SF_METAL = 16u };

template <int TEX>
__global__ void __launch_bounds__(kTB, spawn_min_blocks(TEX)) k_spawn(PassCtx P, const uint32_t* pass_dev, const uint32_t* hit_prim,
                                               float4* state, ShadowQueue sq, float4* Lb, float2* pf,
                                               const uint32_t* order) {
  uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= P.W * P.H) return;
  uint32_t pix = order ? order[slot] : slot;  // material-sorted (large films)
  if (pix >= P.W * P.H) return;
  uint32_t pass = *pass_dev;
  float fx, fy;
  camera_sample(P, pix, pass, &fx, &fy);
  pf[pix] = make_float2(fx, fy);
  RayD r = camera_ray(P.S.cam, fx, fy);
  uint32_t prim = hit_prim[pix];
  float4* st = state + (size_t)pix * kStateF4;
  if (prim == kNoHit || P.S.nlights == 0) {
    RGB3 L = rgb1(0.0f);
    if (prim == kNoHit && P.S.has_env) L = radd(L, env_le(P.S.env, r.d));
    Lb[pix] = make_float4(L.r, L.g, L.b, 0.0f);
    return;
  }
  uint32_t flags = 0;
  SurfInt s = make_si(P.S, prim, r.o, r.d);
  Frame fr = bsdf_frame(s);
  uint32_t mid = prim_material(P.S, prim);
  const wpbr_material m = hit_material<TEX>(P.S, prim, mid, s, r);
  if (TEX != kTexNone && WPBR_MAT_TEXTURED(P.S.mats[mid].type)) {
    flags |= SF_METAL;
    st[ST_METAL] = metal_pack(m);
  }
  V3 wo_l = to_local(fr, s.wo);
  uint32_t li_idx = pick_light(P, pix, pass);
  const wpbr_light& lt = P.S.lights[li_idx];
  LightSample ls;
  ls.ok = false;
  ls.li = rgb1(0.0f);
  ls.wi = V3{0, 0, 0};
  if (light_sample_counts(P.S, lt)) ls = sample_light(P, lt, s.p, pix, pass);
  const bool trace_l = ls.ok && !rblack(ls.li);
  if (trace_l) {
    flags |= SF_TRACE_L;
    const V3 wi_l = to_local(fr, ls.wi);
    st[ST_LI] = make_float4(ls.li.r, ls.li.g, ls.li.b, ls.pdf);
    st[ST_WI] = make_float4(wi_l.x, wi_l.y, wi_l.z, 0.0f);
    st[ST_WO] = make_float4(wo_l.x, wo_l.y, wo_l.z, __uint_as_float(mid));
  }
  sq.push(trace_l, 2 * pix, add(s.p, mul(ls.wi, (float)0.1)), ls.wi);
  float u0, u1;
  sample2d(P.rs, pix, pass, wpbr_rng::DIM_BSDF, &u0, &u1);
  V3 bwi_l;
  float bpdf;
  bool valid;
  RGB3 bf = bsdf_sample(m, wo_l, u0, u1, &bwi_l, &bpdf, &valid);
  V3 bwi = to_world(fr, bwi_l);
  if (valid) {
    flags |= SF_TRACE_B;
    st[ST_BF] = make_float4(bf.r, bf.g, bf.b, bpdf);
  }
  sq.push(valid, 2 * pix + 1, add(s.p, mul(bwi, (float)0.01)), bwi);
  st[ST_BWI] = make_float4(bwi.x, bwi.y, bwi.z, __uint_as_float(flags));
  st[ST_P] = make_float4(s.p.x, s.p.y, s.p.z, __uint_as_float(li_idx));
}

__global__ void __launch_bounds__(kTB) k_finish(PassCtx P, const uint32_t* hit_prim, const float4* state,
                                                const uint32_t* shadow, float4* Lb, const uint32_t* order) {
  uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= P.W * P.H || P.S.nlights == 0) return;
  uint32_t pix = order ? order[slot] : slot;  // material-sorted (large films)
  if (pix >= P.W * P.H || hit_prim[pix] == kNoHit) return;
  const float4* st = state + (size_t)pix * kStateF4;
  const float4 s4 = st[ST_BWI], s5 = st[ST_P];
  const uint32_t flags = __float_as_uint(s4.w), li_idx = __float_as_uint(s5.w);
  const wpbr_light& lt = P.S.lights[li_idx];
  uint32_t lp = light_prim(lt);
  RGB3 L = rgb1(0.0f);
  if (flags & SF_TRACE_L) {
    uint32_t hp = shadow[2 * pix];
    if (hp == kNoHit || hp == lp) {
      const float4 s0 = st[ST_LI], s1 = st[ST_WI], s2 = st[ST_WO];
      const wpbr_material m = (flags & SF_METAL) ? metal_unpack(st[ST_METAL]) : P.S.mats[__float_as_uint(s2.w)];
      float bpdf;
      RGB3 f = bsdf_eval(m, V3{s2.x, s2.y, s2.z}, V3{s1.x, s1.y, s1.z}, &bpdf);
      if (bpdf != 0.0f) {
        float lpdf = s0.w;
        float w = power_heuristic(lpdf, bpdf);
        L = radd(L, rmuls(rmul(RGB3{s0.x, s0.y, s0.z}, f), w / lpdf));
      }
    }
  }
  if (flags & SF_TRACE_B) {
    uint32_t hp = shadow[2 * pix + 1];
    if (hp == kNoHit || hp == lp) {
      RGB3 li;
      float lpdf;
      light_compute(P, lt, V3{s5.x, s5.y, s5.z}, V3{s4.x, s4.y, s4.z}, &li, &lpdf);
      if (!rblack(li)) {
        const float4 s3 = st[ST_BF];
        float bpdf = s3.w;
        float w = (bpdf == 1.0f) ? 1.0f : power_heuristic(bpdf, lpdf);
        L = radd(L, rmuls(rmul(li, RGB3{s3.x, s3.y, s3.z}), w / bpdf));
      }
    }
  }
  Lb[pix] = make_float4(L.r, L.g, L.b, 0.0f);
}

// ============================== environment =================================
// Distribution1D over n values by one block: cdf[0..n] and the integral. The
// running sum is the reference's serial loop (one thread, the same rounding);
// the block makes its terms f[i] / n beforehand and divides by the integral
// afterwards. Values come in chunks through shared memory; a distribution of
// one chunk never reads its sums back.
//
// What bounds it is the chain of additions: about 5 cycles a value, 2.7 us for
// a row of 1,024, with the rows of a map side by side on all SMs. With one
// thread a row making the terms, sums and quotients (each load and store of a
// warp touching 32 rows) a 1024 x 512 map took 967 us; 256 x 128, 62 us.
constexpr int kDistThreads = 128;
constexpr uint32_t kDistChunk = 2048;
template <class F>
__device__ __forceinline__ void block_distribution(F value, uint32_t n, float* cdf, float* fint) {
  __shared__ __align__(16) float s_q[kDistChunk], s_c[kDistChunk];
  __shared__ float s_sum;
  float sum = 0.0f;  // thread 0's running sum
  for (uint32_t at = 0; at < n; at += kDistChunk) {
    const uint32_t m = min(kDistChunk, n - at);
    for (uint32_t i = threadIdx.x; i < m; i += kDistThreads) s_q[i] = value(at + i) / (float)n;
    __syncthreads();
    if (threadIdx.x == 0) {
      const float4* q4 = reinterpret_cast<const float4*>(s_q);
      float4* c4 = reinterpret_cast<float4*>(s_c);
      float4 next = q4[0];
      const uint32_t quads = m / 4;
      for (uint32_t j = 0; j < quads; ++j) {
        const float4 q = next;
        next = q4[min(j + 1, kDistChunk / 4 - 1)];
        float4 c;
        c.x = sum + q.x;
        c.y = c.x + q.y;
        c.z = c.y + q.z;
        c.w = c.z + q.w;
        sum = c.w;
        c4[j] = c;
      }
      for (uint32_t i = 4 * quads; i < m; ++i) {
        sum = sum + s_q[i];
        s_c[i] = sum;
      }
      s_sum = sum;
    }
    __syncthreads();
    if (n > kDistChunk)
      for (uint32_t i = threadIdx.x; i < m; i += kDistThreads) cdf[at + i + 1] = s_c[i];
    // (the next chunk's terms go to s_q, which thread 0 has finished reading,
    // and its sums to s_c only after the barrier that follows them)
  }
  const float fi = s_sum;
  if (threadIdx.x == 0) {
    cdf[0] = 0.0f;
    *fint = fi;
  }
  for (uint32_t i = threadIdx.x; i < n; i += kDistThreads) {
    // thread i wrote entry i + 1 of every chunk itself
    const float c = n > kDistChunk ? cdf[i + 1] : s_c[i];
    cdf[i + 1] = fi == 0.0f ? (float)(i + 1) / (float)n : c / fi;
  }
}

// JobLightInfiniteAreaPreprocessSampling (CLightInfiniteArea.cpp:113-139): the
// map function and the conditional distribution of one row per block. A row's
// sine (double, FP64) is computed once.
__device__ __forceinline__ float env_row_sine(uint32_t y, uint32_t H) {
  return (float)sin_d((kPI * (double)(float)((float)y + 0.5f)) / (double)(float)H);
}
__device__ __forceinline__ float env_map_value(const EnvView& e, uint32_t x, uint32_t y, float sine) {
  return env_bilerp(e, (float)x / (float)e.W, (float)y / (float)e.H).g * sine;
}
__global__ void __launch_bounds__(kDistThreads) k_env_rows(EnvView e, uint32_t quirks, float* func, float* cdf,
                                                           float* fint) {
  __shared__ float s_sine;
  const uint32_t W = e.W, H = e.H, row = blockIdx.x;
  float* f = func + (size_t)row * W;
  if (threadIdx.x == 0) s_sine = env_row_sine(row, H);
  __syncthreads();
  auto value = [&](uint32_t col) {
    float v;
    if (quirks & WPBR_Q_ENV_DISTRIB_INDEX_BUG) {
      // data[x + y*resY] written in row order: the last writer of index i is
      // the one with the largest row.
      const uint32_t i = row * W + col;
      const uint32_t y = min(H - 1, i / H), x = i - y * H;
      v = x < W ? env_map_value(e, x, y, env_row_sine(y, H)) : 0.0f;
    } else {
      v = env_map_value(e, col, row, s_sine);
    }
    f[col] = v;
    return v;
  };
  block_distribution(value, W, cdf + (size_t)row * (W + 1), fint + row);
}
// The marginal distribution over the rows' integrals.
__global__ void __launch_bounds__(kDistThreads) k_env_marginal(const float* cond_int, uint32_t H, float* func,
                                                               float* cdf, float* fint) {
  block_distribution(
      [&](uint32_t i) {
        const float v = cond_int[i];
        func[i] = v;
        return v;
      },
      H, cdf, fint);
}

// JobOutputFilmTitles (CSFilm.cpp:129-170): /(w*800000), clamp, sRGB-like
// curve with the reference's 12.98 linear slope, x255, truncated to bytes.
__device__ float gamma_correct(float v) {
  if (v <= 0.0031308f) return 12.98f * v;
  return 1.055f * expf_(logf_(v) * (float)(1.0f / 2.4f)) - 0.055f;
}
__global__ void k_tonemap(uint32_t n, const float4* acc, uint8_t* out) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 a = acc[i];
  if (a.x == 0.0f && a.y == 0.0f && a.z == 0.0f) {
    out[3 * i] = out[3 * i + 1] = out[3 * i + 2] = 0;
    return;
  }
  float d = a.w * 800000.f;
  float c[3] = {a.x / d, a.y / d, a.z / d};
  for (int k = 0; k < 3; ++k) {
    float v = clampf(c[k], 0.0f, 1.0f);
    v = gamma_correct(v) * 255.0f;
    out[3 * i + k] = (uint8_t)(int)v;
  }
}

__global__ void k_film_split(uint32_t n, const float4* acc, float* L, float* w) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 a = acc[i];
  L[3 * (size_t)i] = a.x;
  L[3 * (size_t)i + 1] = a.y;
  L[3 * (size_t)i + 2] = a.z;
  w[i] = a.w;
}

PassCtx make_pass_ctx(wpbr_ctx* ctx) {
  return pass_ctx(scene_view(ctx), render_traversal_view(ctx),
                  wpbr_rng::Stream{ctx->rs.seed, ctx->rs.stream, ctx->rs.spp, (ctx->quirks & WPBR_Q_REF_SAMPLER_ARRAYS) ? 1u : 0u},
                  ctx->rs.W, ctx->rs.H, ctx->d_err.p);
}

Staged staged_view(wpbr_ctx* ctx) {
  Staged G;
  for (int i = 0; i < F_COUNT; ++i) G.f[i] = ctx->rs.f[i].p;
  for (int i = 0; i < U_COUNT; ++i) G.u[i] = ctx->rs.u[i].p;
  return G;
}

wpbr_status ensure_staged(wpbr_ctx* ctx) {
  size_t n = (size_t)ctx->rs.W * ctx->rs.H;
  for (int i = 0; i < F_COUNT; ++i) WPBR_CUDA(ctx->rs.f[i].ensure(n * kFW[i]));
  for (int i = 0; i < U_COUNT; ++i) WPBR_CUDA(ctx->rs.u[i].ensure(n));
  return WPBR_OK;
}

}  // namespace

__global__ void k_rgb_to_texels(const float* rgb, uint64_t n, float4* out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = make_float4(rgb[3 * i], rgb[3 * i + 1], rgb[3 * i + 2], 0.0f);
}
cudaError_t rgb_to_texels(const float* d_rgb, uint64_t n, float4* d_out, cudaStream_t st) {
  k_rgb_to_texels<<<div_up(n, 256), 256, 0, st>>>(d_rgb, n, d_out);
  return cudaGetLastError();
}

wpbr_status env_distribution_build(wpbr_ctx* ctx, const float4* rgb, const EnvDist& out, float* marg_int_host) {
  SceneView S = scene_view(ctx);
  S.env.rgb = rgb;
  const uint32_t H = ctx->envH;
  cudaStream_t st = ctx->stream;
  k_env_rows<<<H, kDistThreads, 0, st>>>(S.env, ctx->quirks, out.cond_func, out.cond_cdf, out.cond_int);
  k_env_marginal<<<1, kDistThreads, 0, st>>>(out.cond_int, H, out.marg_func, out.marg_cdf, out.marg_int);
  WPBR_CUDA(cudaGetLastError());
  float mi = 0.0f;
  WPBR_CUDA(cudaMemcpyAsync(&mi, out.marg_int, 4, cudaMemcpyDeviceToHost, st));
  WPBR_CUDA(cudaStreamSynchronize(st));
  *marg_int_host = mi;
  return WPBR_OK;
}

wpbr_status env_preprocess(wpbr_ctx* ctx) {
  if (!ctx->has_env) return WPBR_OK;
  EnvDist d{ctx->cond_func.p, ctx->cond_cdf.p, ctx->cond_int.p, ctx->marg_func.p, ctx->marg_cdf.p, ctx->marg_int.p};
  return env_distribution_build(ctx, ctx->env_rgb.p, d, &ctx->env_marg_int);
}

wpbr_status render_setup(wpbr_ctx* ctx, uint32_t spp, uint32_t seed, uint32_t stream) {
  if (!ctx->has_scene) return set_err(ctx, WPBR_ERR_NOT_BUILT, "render_setup: no scene");
  if (!ctx->bvh.built) return set_err(ctx, WPBR_ERR_NOT_BUILT, "render_setup: BVH not built");
  if (spp == 0) return set_err(ctx, WPBR_ERR_INVALID_ARG, "render_setup: spp must be > 0");
  RenderState& R = ctx->rs;
  // not ready until every buffer below exists: a failed allocation here must
  // not leave an earlier setup's graph (or its freed buffers) usable
  R.ready = false;
  R.spp = spp;
  R.seed = seed;
  R.stream = stream;
  R.W = ctx->cam.W;
  R.H = ctx->cam.H;
  size_t n = (size_t)R.W * R.H;
  WPBR_CUDA(R.acc.ensure(n * 4 + n * 4));  // the accumulators, then what reads copy to the host
  WPBR_CUDA(R.hit_prim.ensure(n));
  WPBR_CUDA(R.shadow_rays.ensure(n * 4));
  WPBR_CUDA(R.shadow_map.ensure(n * 2));
  WPBR_CUDA(R.shadow_hit.ensure(n * 2));
  WPBR_CUDA(R.pstate.ensure(n * kStateF4));
  WPBR_CUDA(R.Lbuf.ensure(n));
  WPBR_CUDA(R.pfilm.ensure(n));
  WPBR_CUDA(R.pass_dev.ensure(RenderState::kMaxGroup));
  WPBR_CUDA(R.counters.ensure(kPassCounters));  // allocated before any graph capture
  WPBR_CUDA(R.order.ensure(n));
  WPBR_CUDA(cudaMemsetAsync(R.acc.p, 0, n * 4 * sizeof(float), ctx->stream));
  if (ctx->spectrum == WPBR_SPECTRUM_SAMPLED64) {
    wpbr_status sst = spectral_setup(ctx);
    if (sst != WPBR_OK) return sst;
  }
  R.ready = true;  // a captured pass graph stays valid while pass_graph_key is unchanged
  return WPBR_OK;
}


namespace {
// Bytes of one state slice: the per-pixel arrays, then the counters, each
// part 256-byte aligned.
constexpr size_t kSliceAlign = 256;
size_t slice_part(size_t bytes) { return (bytes + kSliceAlign - 1) / kSliceAlign * kSliceAlign; }
template <class F>
size_t slice_layout(size_t n, F&& part) {
  size_t at = 0;
  for (size_t bytes : {n * 4, n * kStateF4 * 16, n * 16, n * 8, n * 64, n * 8, n * 8, n * 4,
                       (size_t)kPassCounters * 4}) {
    part(at);
    at += slice_part(bytes);
  }
  return at;
}
size_t slice_bytes(size_t n) {
  return slice_layout(n, [](size_t) {});
}

// State slice g of a pass group: the context's own buffers for g = 0.
PassBufs pass_bufs(const wpbr_ctx* ctx, uint32_t g) {
  const RenderState& R = ctx->rs;
  if (g == 0)
    return PassBufs{R.hit_prim.p,   R.pstate.p,     R.Lbuf.p,  R.pfilm.p,   R.shadow_rays.p,
                    R.shadow_map.p, R.shadow_hit.p, R.order.p, R.counters.p};
  const size_t n = (size_t)R.W * R.H;
  unsigned char* at[9];
  int k = 0;
  unsigned char* base = R.slices.p + (size_t)(g - 1) * slice_bytes(n);
  slice_layout(n, [&](size_t off) { at[k++] = base + off; });
  return PassBufs{(uint32_t*)at[0], (float4*)at[1],   (float4*)at[2],   (float2*)at[3],  (float4*)at[4],
                  (uint32_t*)at[5], (uint32_t*)at[6], (uint32_t*)at[7], (uint32_t*)at[8]};
}

void film_launch(const wpbr_ctx* ctx, const PassBufs& B, cudaStream_t st) {
  const RenderState& R = ctx->rs;
  film_tiles_launch(R.W, R.H, B.pfilm, B.Lbuf, (float4*)R.acc.p, st);
}

// The kernels of one sample pass up to its samples (the film gather follows),
// on stream `st` in state slice B, reading the pass index at pass_ptr; `share`
// passes run at the same time. A Sampled64 pass writes sample slot spec_slot.
wpbr_status pass_kernels(wpbr_ctx* ctx, const PassBufs& B, const uint32_t* pass_ptr, cudaStream_t st,
                         uint32_t share, uint32_t spec_slot = 0) {
  RenderState& R = ctx->rs;
  PassCtx P = make_pass_ctx(ctx);
  const uint32_t n = R.W * R.H, grid = R.trace_grid;
  uint32_t* counters = B.counters;
  WPBR_CUDA(cudaMemsetAsync(counters, 0, kPassCounters * sizeof(uint32_t), st));
  const ShadowQueue sq{B.shadow_rays, B.shadow_map, counters + kQueueCounter};
  bool spectral = ctx->spectrum == WPBR_SPECTRUM_SAMPLED64;
  launch_traversal<false>(P.S, P.Bv, CameraSrc{P, pass_ptr}, PrimSink{B.hit_prim}, n, counters, P.err, st, grid,
                          share);
  // the pixels in material-sorted order for the spawn and finish kernels
  const uint32_t* order = nullptr;
  if (n >= kSortMinPixels) {
    k_cat_order<<<div_up(n, kCatTile), kCatBlock, 0, st>>>(P.S, n, B.hit_prim, B.order);
    order = B.order;
  }
  const int tex = tex_build(ctx->has_metal, spectral, (uint64_t)n * share);
  if (spectral)
    WPBR_CUDA(spectral_spawn_launch(ctx, B, pass_ptr, order, spec_slot, tex, st));
  else
    (tex == kTexNone ? k_spawn<kTexNone> : tex == kTexWide ? k_spawn<kTexWide> : k_spawn<kTexCompact>)
        <<<div_up(n, kTB), kTB, 0, st>>>(P, pass_ptr, B.hit_prim, B.pstate, sq, B.Lbuf, B.pfilm, order);
  // shadow rays: unoccluded iff no hit or the closest hit is the sampled
  // light's primitive; with environment lights only that is "no hit", which
  // the any-hit traversal decides with the same primitive tests, stopping at
  // the first hit (the stored id is then some hit, never a light's)
  // (the spawn queued only the rays it traces; the traversal walks the queue)
  const QueueSrc qsrc{sq.rays, sq.count};
  const MapSink qsink{B.shadow_hit, sq.map};
  if (ctx->env_lights_only)
    launch_traversal<true>(P.S, P.Bv, qsrc, qsink, 2 * n, counters + 1, P.err, st, grid, share);
  else
    launch_traversal<false>(P.S, P.Bv, qsrc, qsink, 2 * n, counters + 1, P.err, st, grid, share);
  if (spectral)
    WPBR_CUDA(spectral_finish_launch(ctx, B, order, spec_slot, st));
  else
    k_finish<<<div_up(n, kTB), kTB, 0, st>>>(P, B.hit_prim, B.pstate, B.shadow_hit, B.Lbuf, order);
  WPBR_CUDA(cudaGetLastError());
  return WPBR_OK;
}
}  // namespace

// Launches the kernels of one sample pass on the context's stream. The
// pass index is read from device memory (R.pass_ptr, shared across the scenes
// of a batch, else R.pass_dev); R.trace_grid caps the persistent traversal
// grids (0: one full wave of resident blocks).
wpbr_status render_pass_launch(wpbr_ctx* ctx) {
  RenderState& R = ctx->rs;
  const uint32_t n = R.W * R.H;
  WPBR_CUDA(R.counters.ensure(kPassCounters));
  WPBR_CUDA(R.shadow_map.ensure((size_t)2 * n));
  WPBR_CUDA(R.order.ensure(n));
  const PassBufs B = pass_bufs(ctx, 0);
  wpbr_status s = pass_kernels(ctx, B, R.pass_ptr ? R.pass_ptr : R.pass_dev.p, ctx->stream, R.trace_share);
  if (s != WPBR_OK) return s;
  if (ctx->spectrum == WPBR_SPECTRUM_SAMPLED64) {
    WPBR_CUDA(spectral_film_launch(ctx, 1, ctx->stream));
  } else {
    film_launch(ctx, B, ctx->stream);
    WPBR_CUDA(cudaGetLastError());
  }
  return WPBR_OK;
}

// Everything the captured pass graph bakes into its kernel arguments: the
// scene/BVH epoch, the sample-stream parameters, the film size and every
// device pointer the kernels receive.
static uint64_t pass_graph_key(const wpbr_ctx* ctx) {
  const RenderState& R = ctx->rs;
  uint64_t h = 0xCBF29CE484222325ull;
  auto mix = [&h](uint64_t v) {
    for (int i = 0; i < 8; ++i) {
      h ^= (v >> (8 * i)) & 0xFFu;
      h *= 0x100000001B3ull;
    }
  };
  mix(ctx->epoch);
  mix(R.spp);
  mix(R.seed);
  mix(R.stream);
  mix(((uint64_t)R.W << 32) | R.H);
  mix((uint64_t)R.trace_grid);
  mix((uint64_t)ctx->spectrum | ((uint64_t)ctx->quirks << 8));
  const void* ptrs[] = {R.acc.p,    R.hit_prim.p, R.shadow_rays.p,     R.shadow_hit.p,      R.shadow_map.p, R.pstate.p,
                        R.Lbuf.p,   R.pfilm.p,    R.pass_dev.p,        R.counters.p,        R.pass_ptr, R.order.p,
                        R.slices.p, ctx->d_err.p, ctx->bvh.view.nodes,
                        ctx->bvh.view.prims, R.spec_mats.p, R.spec_le.p, R.spec_L.p, R.spec_acc.p, R.spec_flags.p};
  for (const void* q : ptrs) mix((uint64_t)(uintptr_t)q);
  return h;
}

wpbr_status render_pass_fused(wpbr_ctx* ctx, uint32_t pass) {
  RenderState& R = ctx->rs;
  if (!R.ready) return set_err(ctx, WPBR_ERR_NOT_BUILT, "render_pass: render_setup not called");
  if (pass >= R.spp) return set_err(ctx, WPBR_ERR_INVALID_ARG, "render_pass: pass >= spp");
  cudaStream_t st = ctx->stream;
  WPBR_CUDA(cudaMemcpyAsync(R.pass_dev.p, &pass, 4, cudaMemcpyHostToDevice, st));
  if (ctx->spectrum == WPBR_SPECTRUM_SAMPLED64) R.spec_dirty = true;
  uint64_t key = pass_graph_key(ctx);
  if (R.graph && R.graph_key != key) {
    cudaGraphExecDestroy(R.graph);
    R.graph = nullptr;
    R.graph_ok = false;
  }
  if (!R.graph_ok) {
    R.graph_key = key;
    // capture the kernels once; later passes replay the graph
    cudaGraph_t g = nullptr;
    if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
      wpbr_status s = render_pass_launch(ctx);
      cudaError_t e = cudaStreamEndCapture(st, &g);
      if (s == WPBR_OK && e == cudaSuccess && g) {
        if (cudaGraphInstantiate(&R.graph, g, 0) == cudaSuccess) R.graph_ok = true;
      }
      if (g) cudaGraphDestroy(g);
    }
    // capture is not possible on the legacy default stream: clear the error
    // and launch the kernels directly
    cudaGetLastError();
    if (!R.graph_ok) return render_pass_launch(ctx);
  }
  WPBR_CUDA(cudaGraphLaunch(R.graph, st));
  return WPBR_OK;
}

// Captures (or reuses) the graph of a group of K passes. RGB: K branches, each
// pass in its own state slice, and the film gathers in pass order on the
// context's stream, each as soon as its branch is done. Sampled64: K branches
// writing sample slots 0 .. K - 1, then one film gather over the slots. Every
// pass computes what it computes alone and the film adds the passes in order,
// so the film is the one that K single passes make. Returns WPBR_OK with
// G.exec null when the stream cannot be captured (the legacy default stream).
static wpbr_status group_graph(wpbr_ctx* ctx, RenderState::GroupGraph& G, uint32_t K) {
  RenderState& R = ctx->rs;
  cudaStream_t st = ctx->stream;
  const bool spectral = ctx->spectrum == WPBR_SPECTRUM_SAMPLED64;
  const uint64_t key = pass_graph_key(ctx) * 0x100000001B3ull + K;
  if (G.exec && G.key == key) return WPBR_OK;
  if (G.exec) cudaGraphExecDestroy(G.exec);
  G.exec = nullptr;
  for (uint32_t g = 0; g < K; ++g)
    if (!R.gstream[g]) WPBR_CUDA(cudaStreamCreateWithFlags(&R.gstream[g], cudaStreamNonBlocking));
  if (!R.gfork) WPBR_CUDA(cudaEventCreateWithFlags(&R.gfork, cudaEventDisableTiming));
  for (uint32_t g = 0; g < K; ++g)
    if (!R.gjoin[g]) WPBR_CUDA(cudaEventCreateWithFlags(&R.gjoin[g], cudaEventDisableTiming));
  if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();
    return WPBR_OK;
  }
  wpbr_status s = WPBR_OK;
  cudaError_t e = cudaEventRecord(R.gfork, st);
  for (uint32_t g = 0; g < K && e == cudaSuccess && s == WPBR_OK; ++g) {
    e = cudaStreamWaitEvent(R.gstream[g], R.gfork, 0);
    if (e != cudaSuccess) break;
    s = pass_kernels(ctx, pass_bufs(ctx, g), R.pass_dev.p + g, R.gstream[g], K, g);
    if (s != WPBR_OK) break;
    e = cudaEventRecord(R.gjoin[g], R.gstream[g]);
  }
  for (uint32_t g = 0; g < K && e == cudaSuccess && s == WPBR_OK; ++g) {
    e = cudaStreamWaitEvent(st, R.gjoin[g], 0);
    if (e == cudaSuccess && !spectral) film_launch(ctx, pass_bufs(ctx, g), st);
  }
  if (e == cudaSuccess && s == WPBR_OK && spectral) e = spectral_film_launch(ctx, K, st);
  cudaGraph_t gr = nullptr;
  const cudaError_t e2 = cudaStreamEndCapture(st, &gr);
  if (s == WPBR_OK && e == cudaSuccess && e2 == cudaSuccess && gr) e = cudaGraphInstantiate(&G.exec, gr, 0);
  if (gr) cudaGraphDestroy(gr);
  if (s != WPBR_OK) {
    cudaGetLastError();
    return s;
  }
  if (e != cudaSuccess || e2 != cudaSuccess || !G.exec) {
    cudaGetLastError();
    G.exec = nullptr;
    return set_err(ctx, WPBR_ERR_CUDA, "render: pass-group graph capture failed");
  }
  G.key = key;
  return WPBR_OK;
}

// A whole frame (every pass of render_setup's spp) through the fused pass, in
// pass groups; spp that the group size does not divide ends with a smaller
// group (a graph of its own).
wpbr_status render_frame(wpbr_ctx* ctx) {
  RenderState& R = ctx->rs;
  if (!R.ready) return set_err(ctx, WPBR_ERR_NOT_BUILT, "render: render_setup not called");
  const size_t n = (size_t)R.W * R.H;
  const bool spectral = ctx->spectrum == WPBR_SPECTRUM_SAMPLED64;
  uint32_t K = R.pass_ptr ? 1u : group_passes(n, R.spp, spectral);
  const size_t pass_bytes = slice_bytes(n) + (spectral ? spectral_slot_bytes(n) : 0);
  if ((K - 1) * pass_bytes > kGroupUnasked &&
      (R.slices.n < (K - 1) * slice_bytes(n) || (spectral && R.spec_flags.n < K * n))) {
    size_t room = 0, total = 0;
    WPBR_CUDA(cudaMemGetInfo(&room, &total));
    K = group_passes_within(K, pass_bytes, room + R.slices.n);  // the old slices go first
  }
  if (K > 1) {
    // the group's buffers; a device without room for them renders one pass at
    // a time, in the buffers render_setup made (which a failure here leaves)
    cudaError_t e = R.slices.ensure((K - 1) * slice_bytes(n));
    if (e == cudaSuccess && spectral) e = spectral_slots(ctx, K);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      R.slices.release();
      K = 1;
    } else {
      WPBR_CUDA(e);
    }
  }
  uint32_t base = 0;
  cudaStream_t st = ctx->stream;
  while (K > 1 && base < R.spp) {
    const uint32_t k = std::min(K, R.spp - base);
    RenderState::GroupGraph& G = R.groups[k == K ? 0 : 1];
    wpbr_status s = group_graph(ctx, G, k);
    if (s != WPBR_OK) return s;
    if (!G.exec) break;
    if (spectral) R.spec_dirty = true;
    uint32_t passes[RenderState::kMaxGroup];
    for (uint32_t g = 0; g < k; ++g) passes[g] = base + g;
    WPBR_CUDA(cudaMemcpyAsync(R.pass_dev.p, passes, sizeof(uint32_t) * k, cudaMemcpyHostToDevice, st));
    WPBR_CUDA(cudaGraphLaunch(G.exec, st));
    base += k;
  }
  for (; base < R.spp; ++base) {
    wpbr_status s = render_pass_fused(ctx, base);
    if (s != WPBR_OK) return s;
  }
  return WPBR_OK;
}

wpbr_status job_run(wpbr_ctx* ctx, uint32_t job, uint32_t pass) {
  RenderState& R = ctx->rs;
  if (ctx->spectrum != WPBR_SPECTRUM_RGB)
    return set_err(ctx, WPBR_ERR_INVALID_ARG, "job_run: the staged jobs run in RGB mode only");
  if (!R.ready) return set_err(ctx, WPBR_ERR_NOT_BUILT, "job_run: render_setup not called");
  if (job >= WPBR_JOB_COUNT) return set_err(ctx, WPBR_ERR_INVALID_ARG, "job_run: unknown job id");
  if (pass >= R.spp) return set_err(ctx, WPBR_ERR_INVALID_ARG, "job_run: pass >= spp");
  wpbr_status s = ensure_staged(ctx);
  if (s != WPBR_OK) return s;
  PassCtx P = make_pass_ctx(ctx);
  Staged G = staged_view(ctx);
  uint32_t n = R.W * R.H;
  unsigned g = div_up(n, kTB);
  cudaStream_t st = ctx->stream;
  switch (job) {
    case WPBR_JOB_CAMERA_RAYS: kj_camera<<<g, kTB, 0, st>>>(P, pass, G); break;
    case WPBR_JOB_COLLIDE_PRIMARY: kj_collide<<<g, kTB, 0, st>>>(P, G); break;
    case WPBR_JOB_EMITTED_LIGHT: kj_emitted<<<g, kTB, 0, st>>>(P, G); break;
    case WPBR_JOB_BSDF_SETUP: kj_bsdf_setup<<<g, kTB, 0, st>>>(P, G); break;
    case WPBR_JOB_SAMPLE_LIGHT: kj_sample_light<<<g, kTB, 0, st>>>(P, pass, G); break;
    case WPBR_JOB_SHADOW_LIGHT: kj_shadow_light<<<g, kTB, 0, st>>>(P, G); break;
    case WPBR_JOB_BSDF_COMPUTE: kj_bsdf_compute<<<g, kTB, 0, st>>>(P, G); break;
    case WPBR_JOB_INTEGRATE_LIGHT: kj_integrate_light<<<g, kTB, 0, st>>>(P, G); break;
    case WPBR_JOB_SAMPLE_BSDF: kj_sample_bsdf<<<g, kTB, 0, st>>>(P, pass, G); break;
    case WPBR_JOB_SHADOW_BSDF: kj_shadow_bsdf<<<g, kTB, 0, st>>>(P, G); break;
    case WPBR_JOB_LIGHT_COMPUTE: kj_light_compute<<<g, kTB, 0, st>>>(P, G); break;
    case WPBR_JOB_INTEGRATE_BSDF: kj_integrate_bsdf<<<g, kTB, 0, st>>>(P, G); break;
    case WPBR_JOB_FILM_ACCUMULATE:
      kj_film_pack<<<g, kTB, 0, st>>>(P, G, R.pfilm.p, R.Lbuf.p);
      film_tiles_launch(R.W, R.H, R.pfilm.p, R.Lbuf.p, (float4*)R.acc.p, st);
      break;
  }
  WPBR_CUDA(cudaGetLastError());
  return WPBR_OK;
}

wpbr_status job_record(wpbr_ctx* ctx, uint32_t x0, uint32_t y0, uint32_t x1, uint32_t y1, wpbr_pass_record* rec) {
  RenderState& R = ctx->rs;
  if (!R.ready || !R.f[0].p) return set_err(ctx, WPBR_ERR_NOT_BUILT, "job_record: no staged pass");
  if (x1 > R.W || y1 > R.H || x0 >= x1 || y0 >= y1 || !rec)
    return set_err(ctx, WPBR_ERR_INVALID_ARG, "job_record: bad rectangle");
  float* fptr[F_COUNT] = {rec->pfilm, rec->ray_o, rec->ray_d, rec->ray_dx_d, rec->ray_dy_d, rec->hit_t,
                          rec->si_p, rec->si_n, rec->si_wo, rec->si_sn, rec->si_sdpdu, rec->si_dpdu,
                          rec->si_dpdv, rec->si_dndu, rec->si_dndv, rec->frame, rec->le, rec->l_wi,
                          rec->l_li, rec->l_pdf, rec->l_f, rec->l_fpdf, rec->b_wi, rec->b_f,
                          rec->b_pdf, rec->b_li, rec->b_lpdf, rec->L, nullptr};
  uint32_t* uptr[4] = {rec->hit_prim, rec->light_idx, rec->l_flags, rec->b_flags};
  cudaStream_t st = ctx->stream;
  uint32_t w = x1 - x0;
  for (uint32_t y = y0; y < y1; ++y) {
    size_t src = (size_t)y * R.W + x0;
    size_t dst = (size_t)(y - y0) * w;
    for (int f = 0; f < F_COUNT; ++f)
      if (fptr[f])
        WPBR_CUDA(cudaMemcpyAsync(fptr[f] + dst * kFW[f], R.f[f].p + src * kFW[f], sizeof(float) * w * kFW[f],
                                  cudaMemcpyDeviceToHost, st));
    for (int u = 0; u < 4; ++u)
      if (uptr[u])
        WPBR_CUDA(cudaMemcpyAsync(uptr[u] + dst, R.u[u].p + src, sizeof(uint32_t) * w, cudaMemcpyDeviceToHost, st));
  }
  WPBR_CUDA(cudaStreamSynchronize(st));
  return WPBR_OK;
}

// The accumulators as separate radiance and weight arrays, as the caller
// receives them. Larger films are split on the device into memory that reads
// alone use, behind the accumulators (the pass state's would do, but a caller
// may read on one stream while passes still run on another), so the host only
// receives the copies, into pages touched while the last passes still run:
// splitting 1920 x 1080 float4s on the host, through a vector of its own, took
// 3.4 ms, the copies alone take 0.24.
//
// Films of at most kFilmHostSplit pixels are copied as they are and split on
// the host: one copy instead of a launch and two. us a read into kept / new arrays, host and
// device split: 100 x 100 26.0 / 28.2 on the host; 110 x 111 29.1 / 31.7; 110 x
// 112 28.5 / 31.6 and 28.8 / 35.5; 128 x 128 33.5 / 37.0 and 29.3 / 37.6;
// 160 x 160 45.0 / 49.5 and 30.0 / 41.0. (A vector of float4s, which is
// initialised element by element, instead of floats: 28.3 at 100 x 100.)
constexpr uint32_t kFilmHostSplit = 12288;
wpbr_status film_read(wpbr_ctx* ctx, float* acc_L, float* acc_w) {
  RenderState& R = ctx->rs;
  if (!R.ready) return set_err(ctx, WPBR_ERR_NOT_BUILT, "film_read: render_setup not called");
  wpbr_status rs = spectral_resolve(ctx);
  if (rs != WPBR_OK) return rs;
  const uint32_t n = R.W * R.H;
  if (n <= kFilmHostSplit) {
    std::vector<float> a((size_t)n * 4);
    WPBR_CUDA(cudaMemcpyAsync(a.data(), R.acc.p, (size_t)n * 16, cudaMemcpyDeviceToHost, ctx->stream));
    WPBR_CUDA(cudaStreamSynchronize(ctx->stream));
    for (size_t i = 0; i < n; ++i) {
      if (acc_L) {
        acc_L[3 * i] = a[4 * i];
        acc_L[3 * i + 1] = a[4 * i + 1];
        acc_L[3 * i + 2] = a[4 * i + 2];
      }
      if (acc_w) acc_w[i] = a[4 * i + 3];
    }
    return WPBR_OK;
  }
  float* L = R.acc.p + 4 * (size_t)n;
  float* w = L + 3 * (size_t)n;
  k_film_split<<<div_up(n, 256), 256, 0, ctx->stream>>>(n, (const float4*)R.acc.p, L, w);
  WPBR_CUDA(cudaGetLastError());
  touch_pages(acc_L, (size_t)n * 12);
  touch_pages(acc_w, (size_t)n * 4);
  if (acc_L) WPBR_CUDA(cudaMemcpyAsync(acc_L, L, (size_t)n * 12, cudaMemcpyDeviceToHost, ctx->stream));
  if (acc_w) WPBR_CUDA(cudaMemcpyAsync(acc_w, w, (size_t)n * 4, cudaMemcpyDeviceToHost, ctx->stream));
  WPBR_CUDA(cudaStreamSynchronize(ctx->stream));
  return WPBR_OK;
}

wpbr_status film_tonemap(wpbr_ctx* ctx, uint8_t* out) {
  RenderState& R = ctx->rs;
  if (!R.ready) return set_err(ctx, WPBR_ERR_NOT_BUILT, "tonemap: render_setup not called");
  wpbr_status rs = spectral_resolve(ctx);
  if (rs != WPBR_OK) return rs;
  uint32_t n = R.W * R.H;
  uint8_t* rgb8 = (uint8_t*)(R.acc.p + 4 * (size_t)n);  // as film_read
  k_tonemap<<<div_up(n, 256), 256, 0, ctx->stream>>>(n, (const float4*)R.acc.p, rgb8);
  WPBR_CUDA(cudaGetLastError());
  touch_pages(out, (size_t)n * 3);
  WPBR_CUDA(cudaMemcpyAsync(out, rgb8, (size_t)n * 3, cudaMemcpyDeviceToHost, ctx->stream));
  WPBR_CUDA(cudaStreamSynchronize(ctx->stream));
  return WPBR_OK;
}

}  // namespace wpbr
