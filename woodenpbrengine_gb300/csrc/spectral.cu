// spectral.cu — the Sampled64 mode of the render pass: the same per-sample
// job list as the RGB path (MEngine::render, MEngine.cpp:393-442) with every
// radiance, reflectance and Fresnel value a 64-bin SampledSpectrum, as the
// reference computes it (Spectrum = SampledSpectrum, CSpectrum.h:8).
//
// Wavefront layout: the pass shares the RGB path's camera and shadow-ray
// persistent traversals (render.cu); k_sspawn (one thread per pixel) does
// the scalar part of shading and sampling and records, per pixel, the
// scalar factors every spectral term needs; k_sfinish gives each pixel a
// half-warp, 16 lanes x 4 bins, for the per-bin Fresnel terms and products;
// k_sfilm stages film tiles' rows of sample spectra in shared memory for the
// Mitchell film gather (4 threads x 16 bins per two pixels); k_sresolve
// converts the film to RGB once per frame (or before a film read). Every per-bin value is
// computed with the same operations in the same order as the one-thread
// restatement, so the film is bit-identical to it; sums over bins (toXYZ)
// stay sequential in bin order.

#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "ctx.hpp"
#include "pass.cuh"
#include "spectral.cuh"

namespace wpbr {

namespace {

// The binned tables in global memory: the lanes of a pixel read different
// bins, which the constant cache would serialise.
__device__ __align__(16) SpecTables g_spec;

// Per material: R, eta_i, eta_t, k as spectra.
struct SpecMat {
  S64 R, eta_i, eta_t, k;
};

struct SpecCtx {
  const SpecMat* mats;
  const S64* light_le;  // per light: sphere Le, or the environment's LEmit
  float* L;             // per pixel, 64 floats
  uint32_t* flags;      // per pixel: a bin is not finite
};

// Per-pixel record of k_sspawn (kSpecStateF4 float4, five used):
//  [0] flags, light index (environment light on a miss), material id, w/lpdf
//  [1] light branch: cos(wi, wh), scalar BSDF factor, |cos wi|;  w/bpdf
//  [2] BSDF branch:  cos(wi, wh), scalar BSDF factor, |cos wi|;  -
//  [3] environment (s, t) of the light sample (or of the camera miss), of the BSDF sample
//  [4] textured metal: k (RGB)
constexpr int kSpecStateF4 = kPassStateF4;  // a 128-byte line a pixel, as the RGB pass
enum : uint32_t {
  SS_HIT = 1u,        // the camera ray hit and the scene has lights
  SS_MISS_ENV = 2u,   // the camera ray missed into the environment
  SS_LB = 4u,         // light branch: shadow ray traced, contribution if unoccluded and Li not black
  SS_BB = 8u,         // BSDF branch: likewise
  SS_COND = 16u,      // conductor Fresnel per bin (else the scalar dielectric form)
  SS_TEX = 32u,       // textured metal: eta 1 / 1.5, k from RGB
  SS_LZERO = 64u,     // light-branch f is 0 (grazing wi or wo, or wh = 0)
  SS_BZERO = 128u,    // BSDF-branch f is 0
  SS_LENV = 256u,     // light-branch Li is the environment lookup (WPBR_Q_ENV_LI_SAMPLE_FIX)
  SS_BENV = 512u      // BSDF-branch Li is the environment lookup
};
constexpr int kBinLanes = 16;  // lanes per pixel in the spectral kernels; 4 bins each

// averageSpectrumSamples (CSpectrumSampled.h:45-87): piecewise-linear average
// over [l0, l1], the trapezoid of each segment times 0.5 in double as the
// reference writes it.
float avg_samples(const float* lambda, const float* vals, int n, float l0, float l1) {
  if (l1 <= lambda[0]) return vals[0];
  if (l0 >= lambda[n - 1]) return vals[n - 1];
  if (n == 1) return vals[0];
  float sum = 0.0f;
  if (l0 < lambda[0]) sum += vals[0] * (lambda[0] - l0);
  if (l1 > lambda[n - 1]) sum += vals[n - 1] * (l1 - lambda[n - 1]);
  int j = 0;
  while (l0 > lambda[j + 1]) ++j;
  auto interp = [&](float w, int i) {
    float t = (w - lambda[i]) / (lambda[i + 1] - lambda[i]);
    return (1.0f - t) * vals[i] + t * vals[i + 1];
  };
  for (; j + 1 < n && l1 >= lambda[j]; ++j) {
    float s0 = std::max(l0, lambda[j]);
    float s1 = std::min(l1, lambda[j + 1]);
    sum = (float)((double)sum + (double)((interp(s0, j) + interp(s1, j)) * (s1 - s0)) * 0.5);
  }
  return sum / (l1 - l0);
}

void build_tables(SpecTables* T) {
  using namespace wpbr_spec;
  const float* refl[7] = {kReflWhite, kReflCyan, kReflMagenta, kReflYellow, kReflRed, kReflGreen, kReflBlue};
  const float* illum[7] = {kIllumWhite, kIllumCyan, kIllumMagenta, kIllumYellow, kIllumRed, kIllumGreen, kIllumBlue};
  const float a = (float)kLambdaStart, b = (float)kLambdaEnd;
  for (int i = 0; i < kSpecN; ++i) {
    float t0 = (float)i / (float)kSpecN, t1 = (float)(i + 1) / (float)kSpecN;
    float wl0 = (1.0f - t0) * a + t0 * b;
    float wl1 = (1.0f - t1) * a + t1 * b;
    T->X[i] = avg_samples(kCieLambda, kCieX, kCieSamples, wl0, wl1);
    T->Y[i] = avg_samples(kCieLambda, kCieY, kCieSamples, wl0, wl1);
    T->Z[i] = avg_samples(kCieLambda, kCieZ, kCieSamples, wl0, wl1);
    for (int k = 0; k < 7; ++k) {
      T->refl[k][i] = avg_samples(kRgbLambda, refl[k], kRgbSamples, wl0, wl1);
      T->illum[k][i] = avg_samples(kRgbLambda, illum[k], kRgbSamples, wl0, wl1);
    }
  }
}

// ---- scalar part (one thread per pixel) -----------------------------------

// Scalar factors of mf_f_impl for (wo, wi, wh, D): the per-bin value is
// ((F_conductor(c) * R) * kf) * fcos for a conductor and (R * kf) * fcos
// otherwise; zero when either cosine or wh is zero (then 0 * fcos).
struct FScalars {
  float c, kf, fcos;
  bool zero;
};
__device__ __forceinline__ FScalars f_scalars(const wpbr_material& m, float d_wh, V3 wh, V3 wo, V3 wi) {
  FScalars F;
  F.fcos = abs_cos(wi);
  F.c = 0.0f;
  F.kf = 0.0f;
  float co = abs_cos(wo), ci = abs_cos(wi);
  F.zero = ci == 0.0f || co == 0.0f || (wh.x == 0.0f && wh.y == 0.0f && wh.z == 0.0f);
  if (F.zero) return F;
  F.c = dot(wi, wh);
  if (m.type == WPBR_MAT_CONDUCTOR) {
    F.kf = d_wh / ((4.0f * ci) * co);
  } else {
    float fr = fresnel_dielectric(F.c, m.eta_i[0], m.eta_t[0]);
    F.kf = (fr * d_wh) / ((4.0f * ci) * co);
  }
  return F;
}

template <int TEX>
__global__ void __launch_bounds__(kTB, spawn_min_blocks(TEX)) k_sspawn(PassCtx P, const uint32_t* pass_dev, const uint32_t* hit_prim,
                                                float4* state, ShadowQueue sq, float2* pf, const uint32_t* order) {
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
  float4* st = state + (size_t)pix * kSpecStateF4;
  uint32_t nl = P.S.nlights;
  if (prim == kNoHit || nl == 0) {
    uint32_t flags = 0, env_light = 0;
    if (prim == kNoHit && P.S.has_env) {
      flags = SS_MISS_ENV;
      for (uint32_t i = 0; i < nl; ++i)
        if (P.S.lights[i].type == WPBR_LIGHT_ENV) env_light = i;
      V3 dl = xvector(P.S.env.w2l, r.d);
      float s = div_const(sph_phi(dl), kTwoPiDiv);
      float t = div_const(sph_theta(dl), kPiDiv);
      st[3] = make_float4(s, t, 0.0f, 0.0f);
    }
    st[0] = make_float4(__uint_as_float(flags), __uint_as_float(env_light), 0.0f, 0.0f);
    return;
  }
  uint32_t flags = SS_HIT;
  SurfInt si = make_si(P.S, prim, r.o, r.d);
  Frame fr = bsdf_frame(si);
  uint32_t mid = prim_material(P.S, prim);
  const wpbr_material m = hit_material<TEX>(P.S, prim, mid, si, r);
  if (TEX != kTexNone && WPBR_MAT_TEXTURED(P.S.mats[mid].type)) {
    flags |= SS_TEX;
    st[4] = make_float4(m.k[0], m.k[1], m.k[2], 0.0f);
  }
  if (m.type == WPBR_MAT_CONDUCTOR) flags |= SS_COND;
  V3 wo_l = to_local(fr, si.wo);
  uint32_t li_idx = pick_light(P, pix, pass);
  const wpbr_light& lt = P.S.lights[li_idx];
  float4 s0 = make_float4(0.0f, __uint_as_float(li_idx), __uint_as_float(mid), 0.0f);
  float4 s1 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), s2 = s1, s3 = s1;
  // ---- light-sampling branch: Li is the sphere's LEmit, or (quirk fixed)
  // the environment lookup at the sampled (s, t); without the fix the
  // environment branch's Li is black and nothing is traced
  float u0, u1;
  V3 wi{0, 0, 0};
  float lpdf = 0.0f;
  bool ok = light_sample_counts(P.S, lt);
  if (ok) {
    sample2d(P.rs, pix, pass, wpbr_rng::DIM_LIGHT, &u0, &u1);
    if (lt.type == WPBR_LIGHT_SPHERE) {
      sphere_light_sample(P.S.sph_o2w[lt.sphere_index], P.S.sph_r[lt.sphere_index], si.p, u0, u1, &wi, &lpdf);
    } else {
      RGB3 li_rgb;
      float uv[3];
      env_li_sample(P.S.env, P.S.quirks, u0, u1, &wi, &li_rgb, &lpdf, &ok, uv);
      flags |= SS_LENV;
      s3.x = uv[0];
      s3.y = uv[1];
    }
  }
  if (ok && m.type != WPBR_MAT_SPECULAR) {
    // bsdf_eval: the specular lobe evaluates to pdf 0, which contributes nothing
    V3 wi_l = to_local(fr, wi);
    V3 wh = normalize(add(wo_l, wi_l));
    float d = tr_d(m.alpha_x, m.alpha_y, wh);
    float bpdf = (d * abs_cos(wh)) / (4.0f * dot(wo_l, wh));
    if (bpdf != 0.0f) {
      flags |= SS_LB;
      FScalars F = f_scalars(m, d, wh, wo_l, wi_l);
      if (F.zero) flags |= SS_LZERO;
      float w = power_heuristic(lpdf, bpdf);
      s0.w = w / lpdf;
      s1 = make_float4(F.c, F.kf, F.fcos, 0.0f);
      sq.push(true, 2 * pix, add(si.p, mul(wi, (float)0.1)), wi);
    }
  }
  // ---- BSDF-sampling branch
  sample2d(P.rs, pix, pass, wpbr_rng::DIM_BSDF, &u0, &u1);
  V3 wi_l;
  float bpdf = 0.0f;
  bool valid;
  FScalars F;
  if (m.type == WPBR_MAT_SPECULAR) {
    // SBXDFSpecularReflectance::sample_f: f = R * (Fr / |cos|) * |cos|
    wi_l = V3{-wo_l.x, -wo_l.y, wo_l.z};
    bpdf = 1.0f;
    valid = true;
    F.fcos = abs_cos(wi_l);
    F.c = 0.0f;
    F.zero = !(F.fcos != 0.0f);
    F.kf = F.zero ? 0.0f : fresnel_dielectric(wi_l.z, m.eta_i[0], m.eta_t[0]) / F.fcos;
  } else {
    float d;
    V3 wh = tr_sample(m.alpha_x, m.alpha_y, wo_l, u0, u1, &d);
    wi_l = reflect(wo_l, wh);
    valid = same_hemi(wi_l, wo_l);
    if (valid) {
      bpdf = (d * abs_cos(wh)) / (4.0f * dot(wo_l, wh));
      F = f_scalars(m, d, wh, wo_l, wi_l);
    }
  }
  if (valid) {
    V3 wi_w = to_world(fr, wi_l);
    bool contributes = true;
    float blpdf = 0.0f;
    if (lt.type == WPBR_LIGHT_SPHERE) {
      blpdf = sphere_light_pdf(P.S.sph_o2w[lt.sphere_index], P.S.sph_r[lt.sphere_index], si.p, P.S.quirks);
    } else {
      flags |= SS_BENV;
      V3 wl = xvector(P.S.env.w2l, wi_w);
      float theta = sph_theta(wl);
      float phi = sph_phi(wl);
      float uu = div_const(phi, kTwoPiDiv);
      float vv = div_const(theta, kPiDiv);
      float stt = sinf_(theta);
      contributes = stt != 0.0f;  // else Li stays black
      if (contributes) blpdf = div_by_scaled(env_pdf_uv(P.S.env, uu, vv), kTwoPiSqMul, stt);
      s3.z = uu;
      s3.w = vv;
    }
    if (contributes) {
      flags |= SS_BB;
      if (F.zero) flags |= SS_BZERO;
      float w = (bpdf == 1.0f) ? 1.0f : power_heuristic(bpdf, blpdf);
      s1.w = w / bpdf;
      s2 = make_float4(F.c, F.kf, F.fcos, 0.0f);
      sq.push(true, 2 * pix + 1, add(si.p, mul(wi_w, (float)0.01)), wi_w);
    }
  }
  s0.x = __uint_as_float(flags);
  st[0] = s0;
  st[1] = s1;
  st[2] = s2;
  st[3] = s3;
}

// ---- per-bin part (a half-warp per pixel, 4 bins per lane) -----------------

struct Bins4 {
  float v[4];
};
__device__ __forceinline__ Bins4 ld_bins(const float* p) {
  float4 q = *reinterpret_cast<const float4*>(p);
  return Bins4{{q.x, q.y, q.z, q.w}};
}
__device__ __forceinline__ void st_bins(float* p, const Bins4& b) {
  *reinterpret_cast<float4*>(p) = make_float4(b.v[0], b.v[1], b.v[2], b.v[3]);
}
__device__ __forceinline__ Bins4 bins_const(float v) { return Bins4{{v, v, v, v}}; }
__device__ __forceinline__ bool bins_nonzero(const Bins4& b) {
  return b.v[0] != 0.0f || b.v[1] != 0.0f || b.v[2] != 0.0f || b.v[3] != 0.0f;
}
// s64_from_rgb at bins b0..b0+3: the same three accumulation steps per bin.
__device__ __forceinline__ Bins4 bins_from_rgb(RGB3 c, bool illuminant, int b0) {
  const float(*B)[kSpecN] = illuminant ? g_spec.illum : g_spec.refl;
  float r = c.r, g = c.g, b = c.b;
  int k0, k1, k2;
  float a0, a1, a2;
  if (r <= g && r <= b) {
    k0 = kSpWhite; a0 = r;
    if (g <= b) { k1 = kSpCyan; a1 = g - r; k2 = kSpBlue; a2 = b - g; }
    else { k1 = kSpCyan; a1 = b - r; k2 = kSpGreen; a2 = g - b; }
  } else if (g <= r && g <= b) {
    k0 = kSpWhite; a0 = g;
    if (r <= b) { k1 = kSpMagenta; a1 = r - g; k2 = kSpBlue; a2 = b - r; }
    else { k1 = kSpMagenta; a1 = b - g; k2 = kSpRed; a2 = r - b; }
  } else {
    k0 = kSpWhite; a0 = b;
    if (r <= g) { k1 = kSpYellow; a1 = r - b; k2 = kSpGreen; a2 = g - r; }
    else { k1 = kSpYellow; a1 = g - b; k2 = kSpRed; a2 = r - g; }
  }
  Bins4 s;
  for (int j = 0; j < 4; ++j) {
    float v = 0.0f + B[k0][b0 + j] * a0;
    v = v + B[k1][b0 + j] * a1;
    s.v[j] = v + B[k2][b0 + j] * a2;
  }
  return s;
}
// Spectrum(Spectrum(RGB texel lookup, Illuminant) * LEmit), bins b0..b0+3
__device__ __forceinline__ Bins4 bins_env(const EnvView& e, float s, float t, const float* lemit, int b0) {
  Bins4 r = bins_from_rgb(env_bilerp(e, s, t), true, b0);
  Bins4 le = ld_bins(lemit + b0);
  for (int j = 0; j < 4; ++j) r.v[j] = r.v[j] * le.v[j];
  return r;
}

struct MatBins {
  Bins4 R, eta_i, eta_t, k;
};

__device__ __forceinline__ Bins4 bins_f(bool cond, bool zero, float c, float kf, float fcos, const MatBins& M) {
  Bins4 f;
  for (int j = 0; j < 4; ++j) {
    float v;
    if (zero)
      v = 0.0f;
    else if (cond)
      v = (fresnel_conductor(c, M.eta_i.v[j], M.eta_t.v[j], M.k.v[j]) * M.R.v[j]) * kf;
    else
      v = M.R.v[j] * kf;
    f.v[j] = v * fcos;
  }
  return f;
}

// 12 resident blocks per SM (40 registers): 1080p Sampled64 669 -> 682
// Msamples/s against the unbounded 64 registers (16 blocks: 675).
__global__ void __launch_bounds__(128, 12) k_sfinish(PassCtx P, SpecCtx C, const float4* state,
                                                     const uint32_t* shadow, const uint32_t* order) {
  uint32_t slot = (blockIdx.x * blockDim.x + threadIdx.x) / kBinLanes;
  if (slot >= P.W * P.H) return;  // the whole half-warp leaves together
  uint32_t pix = order ? order[slot] : slot;  // material-sorted (large films)
  if (pix >= P.W * P.H) return;
  uint32_t lane = threadIdx.x & 31u;
  uint32_t hmask = 0xFFFFu << (lane & 16u);
  int b0 = 4 * (int)(lane & 15u);
  const float4* st = state + (size_t)pix * kSpecStateF4;
  float4 s0 = st[0];
  uint32_t flags = __float_as_uint(s0.x);
  uint32_t li_idx = __float_as_uint(s0.y);
  Bins4 L = bins_const(0.0f);
  if (flags & SS_MISS_ENV) {
    float4 s3 = st[3];
    Bins4 le = bins_env(P.S.env, s3.x, s3.y, C.light_le[li_idx].v, b0);
    for (int j = 0; j < 4; ++j) L.v[j] = L.v[j] + le.v[j];
  } else if (flags & (SS_LB | SS_BB)) {
    const wpbr_light& lt = P.S.lights[li_idx];
    uint32_t lp = light_prim(lt);
    const float* lemit = C.light_le[li_idx].v;
    MatBins M;
    if (flags & SS_TEX) {
      // R = Spectrum(1.0), etaI = Spectrum(1.0f), etaT = Spectrum(1.5f),
      // k = (Spectrum)metallic (CMaterialMetal.cpp:44-48)
      float4 kr = st[4];
      M.R = bins_const(1.0f);
      M.eta_i = bins_const(1.0f);
      M.eta_t = bins_const(1.5f);
      M.k = bins_from_rgb(RGB3{kr.x, kr.y, kr.z}, false, b0);
    } else {
      const SpecMat& sm = C.mats[__float_as_uint(s0.z)];
      M.R = ld_bins(sm.R.v + b0);
      M.eta_i = ld_bins(sm.eta_i.v + b0);
      M.eta_t = ld_bins(sm.eta_t.v + b0);
      M.k = ld_bins(sm.k.v + b0);
    }
    float4 s1 = st[1], s3 = st[3];
    bool cond = (flags & SS_COND) != 0;
    if (flags & SS_LB) {
      uint32_t hp = shadow[2 * pix];
      if (hp == kNoHit || hp == lp) {
        Bins4 li = (flags & SS_LENV) ? bins_env(P.S.env, s3.x, s3.y, lemit, b0) : ld_bins(lemit + b0);
        if (__ballot_sync(hmask, bins_nonzero(li)) & hmask) {
          Bins4 f = bins_f(cond, (flags & SS_LZERO) != 0, s1.x, s1.y, s1.z, M);
          for (int j = 0; j < 4; ++j) L.v[j] = L.v[j] + (li.v[j] * f.v[j]) * s0.w;
        }
      }
    }
    if (flags & SS_BB) {
      uint32_t hp = shadow[2 * pix + 1];
      if (hp == kNoHit || hp == lp) {
        Bins4 bli = (flags & SS_BENV) ? bins_env(P.S.env, s3.z, s3.w, lemit, b0) : ld_bins(lemit + b0);
        if (__ballot_sync(hmask, bins_nonzero(bli)) & hmask) {
          float4 s2 = st[2];
          Bins4 f = bins_f(cond, (flags & SS_BZERO) != 0, s2.x, s2.y, s2.z, M);
          for (int j = 0; j < 4; ++j) L.v[j] = L.v[j] + (bli.v[j] * f.v[j]) * s1.w;
        }
      }
    }
  }
  st_bins(C.L + (size_t)pix * kSpecN + b0, L);
  const bool odd = !(isfinite(L.v[0]) && isfinite(L.v[1]) && isfinite(L.v[2]) && isfinite(L.v[3]));
  const uint32_t any = __ballot_sync(hmask, odd) & hmask;
  if ((lane & 15u) == 0) C.flags[pix] = any != 0u;
}

// Tile-clipped Mitchell gather of k_film_tiles, 64 bins per sample: a block
// takes a film tile's width and four of its rows, stages the spectra of those
// rows and of two above and below (asynchronous copies, while the Mitchell
// factors are computed), and four threads share a column of two pixels, 16
// bins each: every staged value is read once for both. As there, pairs outside
// the footprint and black samples add exact zeros instead of being tested,
// unless the block holds a sample with a non-finite bin (spec_flags, from
// k_sfinish). npass passes' samples (pass j's film positions at pf + j * W * H,
// spectra at L + j * W * H * 64, flags likewise) are added in pass order, each
// pass's neighbours in row-major order, to an accumulator held in registers:
// the same sums as npass one-pass gathers, with one read and one write of the
// 64-bin accumulator.
//
// What bounds it: FP32 issue (25 pairs x 64 bins of a product and a sum per
// pixel, 230 us of it below) and the shared loads (270 us), three blocks of 76
// KB an SM. 1001 x 563, 4 passes a launch: 893 us with 8x8 tiles (2.25 staged
// samples a pixel, each pair tested, one pixel a thread), 560 us in this
// layout with scalar sums, 430 us with two-lane ones and unrolled copies. An
// 8-spp frame: 4.35 -> 3.51 ms.
constexpr int kSRows = 4;                          // pixel rows of a block
constexpr unsigned kMaxGridRows = 65535;
constexpr int kSStage = kSRows + 4;                // staged sample rows
constexpr int kFilmThreads = kFilmTile * kSRows / 2 * 4;
constexpr int kSSamples = kSStage * kFilmTile;
constexpr int kSPitch = kFilmTile + 2;             // factors: two empty columns between rows,
constexpr int kSPad = kSStage * kSPitch + 2;       // before the first and after the last
constexpr size_t kSFilmSmem = sizeof(float) * (kSSamples * kSpecN + 10 * kSPad);
// A sample's float4 c sits at c ^ 4 in odd columns, so that the eight lanes
// of a shared load (two columns, four threads each) meet all banks.
__device__ __forceinline__ int spec_slot(int col, int c) { return c ^ ((col & 1) << 2); }
// Two bins as one two-lane value.
__device__ __forceinline__ uint64_t two(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
// a + t * w, the product rounded before the sum. A two-lane product that feeds
// a two-lane sum is contracted, so the sum is a multiply-add of the product by
// one, which rounds once: a + p. `ones` comes from the host, unknown to the
// compiler.
constexpr unsigned long long kOnes = 0x3F8000003F800000ull;
__device__ __forceinline__ void add_scaled(unsigned long long& a, unsigned long long t, unsigned long long w,
                                           unsigned long long ones) {
  unsigned long long p;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(t), "l"(w));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a) : "l"(p), "l"(ones));
}
__global__ void __launch_bounds__(kFilmThreads, 3) k_sfilm(uint32_t W, uint32_t H, const float2* pf, const float* L,
                                                           const uint32_t* flags, uint32_t npass, float* acc,
                                                           float4* accw, unsigned long long ones) {
  extern __shared__ __align__(16) float sfilm_smem[];
  ulonglong2* S = reinterpret_cast<ulonglong2*>(sfilm_smem);   // kSSamples x 16
  float(*s_mx)[kSPad] = reinterpret_cast<float(*)[kSPad]>(sfilm_smem + kSSamples * kSpecN);  // [5]
  float(*s_my)[kSPad] = s_mx + 5;                              // [5]
  const int tid = (int)threadIdx.x;
  // (rows of blocks beyond the second grid dimension's 65,535 in the third)
  const int bx0 = (int)blockIdx.x * kFilmTile, by0 = (int)(blockIdx.z * kMaxGridRows + blockIdx.y) * kSRows;
  if (by0 >= (int)H) return;
  const int ty0 = by0 / 32 * 32;
  const int tx1 = min(bx0 + 31, (int)W - 1), ty1 = min(ty0 + 31, (int)H - 1);
  const int q = tid % 4, lx = tid / 4 % kFilmTile, ly = tid / (4 * kFilmTile) * 2;
  const int x = bx0 + lx, y = by0 + ly;
  const size_t plane = (size_t)W * H;
  bool on[2];
  ulonglong2 a[2][4];  // bins 4 (q + 4 j) .. + 3 of each pixel
  float ws[2];
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    on[p] = x < (int)W && y + p < (int)H;
    const size_t pix = on[p] ? (size_t)(y + p) * W + x : 0;
    const ulonglong2* ap = reinterpret_cast<const ulonglong2*>(acc + pix * kSpecN);
#pragma unroll
    for (int j = 0; j < 4; ++j) a[p][j] = on[p] ? ap[q + 4 * j] : make_ulonglong2(0, 0);
    ws[p] = on[p] ? accw[pix].w : 0.0f;
  }
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(S);
  for (uint32_t ps = 0; ps < npass; ++ps) {
    const float2* pfp = pf + ps * plane;
    const float* Lp = L + ps * plane * kSpecN;
    // the samples: asynchronous 16-byte copies, zero-filled outside the tile;
    // a half-warp a sample, 16 columns a step
    const float* Lrow = Lp + ((ptrdiff_t)(by0 - 2) * W + bx0 + tid / 16) * (ptrdiff_t)kSpecN + tid % 16 * 4;
    const uint32_t srow = sbase + 256u * (tid / 16) + 16u * spec_slot(tid / 16, tid % 16);
#pragma unroll
    for (int k = 0; k < kSSamples * 16 / kFilmThreads; ++k) {
      const int sy = by0 - 2 + k / 2;
      const bool in = bx0 + tid / 16 + k % 2 * 16 <= tx1 && sy >= ty0 && sy <= ty1;
      const float* src = in ? Lrow + ((ptrdiff_t)(k / 2) * W + k % 2 * 16) * (ptrdiff_t)kSpecN : Lp;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(srow + 256u * 16u * k), "l"(src),
                   "r"(in ? 16 : 0)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    bool odd = false;
    for (int i = tid; i < kSPad; i += kFilmThreads) {
      const int sx = bx0 - 2 + i % kSPitch, sy = by0 - 2 + i / kSPitch;
      float mx[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f}, my[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
      if (sx >= bx0 && sx <= tx1 && sy >= ty0 && sy <= ty1) {
        const size_t sp = (size_t)sy * W + sx;
        const float2 f = pfp[sp];
        film_factors(f.x, sx, bx0, tx1, mx);
        film_factors(f.y, sy, ty0, ty1, my);
        odd |= flags[ps * plane + sp] != 0u;
      }
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        s_mx[k][i] = mx[k];
        s_my[k][i] = my[k];
      }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    const bool tested = __syncthreads_or(odd);
    if (!tested) {
      // sample rows y - 2 .. y + 3 (outer), columns x - 2 .. x + 2 (inner);
      // pixel p is row 4 - (r - p) of a sample's reach. The first row reaches
      // only the upper pixel, the last only the lower.
      auto row = [&](int r, bool up, bool down) {
#pragma unroll
        for (int dx = 0; dx < 5; ++dx) {
          const int i = (ly + r) * kSPitch + lx + dx;
          const int col = min(max(lx + dx - 2, 0), kFilmTile - 1);  // beyond the tile: weight zero
          const ulonglong2* sp = S + 16 * ((ly + r) * kFilmTile + col);
          const float mx = s_mx[4 - dx][i];
          const float w0 = up ? mx * s_my[4 - r][i] : 0.0f, w1 = down ? mx * s_my[5 - r][i] : 0.0f;
          const uint64_t u = two(w0, w0), v = two(w1, w1);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const ulonglong2 t = sp[spec_slot(col, q + 4 * j)];
            if (up) {
              add_scaled(a[0][j].x, t.x, u, ones);
              add_scaled(a[0][j].y, t.y, u, ones);
            }
            if (down) {
              add_scaled(a[1][j].x, t.x, v, ones);
              add_scaled(a[1][j].y, t.y, v, ones);
            }
          }
          if (up) ws[0] = ws[0] + w0;
          if (down) ws[1] = ws[1] + w1;
        }
      };
      row(0, true, false);
#pragma unroll 1
      for (int r = 1; r < 5; ++r) row(r, true, true);
      row(5, false, true);
    } else {
      for (int p = 0; p < 2; ++p)
        for (int k = 0; k < 25; ++k) {
          const int sx = x - 2 + k % 5, sy = y + p - 2 + k / 5;
          const bool in = on[p] && sx >= bx0 && sx <= tx1 && sy >= ty0 && sy <= ty1;
          bool valid = false;
          if (in) {
            const float2 f = pfp[(size_t)sy * W + sx];
            const float dx0 = f.x - 0.5f, dy0 = f.y - 0.5f;
            valid = x >= (int)ceilf(dx0 - 2.0f) && x <= (int)floorf(dx0 + 2.0f) && y + p >= (int)ceilf(dy0 - 2.0f) &&
                    y + p <= (int)floorf(dy0 + 2.0f);
          }
          const int col = min(max(sx - bx0, 0), kFilmTile - 1), row = min(max(sy - by0 + 2, 0), kSStage - 1);
          const ulonglong2* sp = S + 16 * (row * kFilmTile + col);
          ulonglong2 t[4];
          bool nz = false;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            t[j] = sp[spec_slot(col, q + 4 * j)];
            nz |= ((t[j].x | t[j].y) & 0x7FFFFFFF7FFFFFFFull) != 0;
          }
          // black in all 64 bins: the pixel's four threads
          const uint32_t any = __ballot_sync(0xFFFFFFFFu, nz) >> (threadIdx.x & 28u) & 0xFu;
          if (!valid) continue;
          const int i = row * kSPitch + sx - bx0 + 2;
          const float w = s_mx[4 - k % 5][i] * s_my[4 - k / 5][i];
          if (any) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              add_scaled(a[p][j].x, t[j].x, two(w, w), ones);
              add_scaled(a[p][j].y, t[j].y, two(w, w), ones);
            }
          }
          ws[p] = ws[p] + w;
        }
    }
    __syncthreads();  // the next pass restages the samples and factors
  }
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    if (!on[p]) continue;
    const size_t pix = (size_t)(y + p) * W + x;
    ulonglong2* ap = reinterpret_cast<ulonglong2*>(acc + pix * kSpecN);
#pragma unroll
    for (int j = 0; j < 4; ++j) ap[q + 4 * j] = a[p][j];
    if (q == 0) accw[pix].w = ws[p];
  }
}

// toRGB of the accumulated spectra (s64_to_rgb: per bin products, the three
// sums taken sequentially in bin order, bin width, XYZ to RGB matrix). A
// warp stages 32 pixels' spectra in shared memory with coalesced loads, then
// each lane sums one pixel.
constexpr int kResolveRow = kSpecN + 1;  // padded row: lane l reads bank (l + i) mod 32
__global__ void __launch_bounds__(128) k_sresolve(uint32_t n, const float* acc, float4* accw, uint32_t quirks) {
  __shared__ float sh[4][32 * kResolveRow];
  uint32_t warp = threadIdx.x / 32, lane = threadIdx.x & 31u;
  uint64_t base = ((uint64_t)blockIdx.x * 4 + warp) * 32;
  if (base >= n) return;
  float* row = sh[warp];
  for (int i = 0; i < kSpecN; ++i) {
    uint32_t k = (uint32_t)i * 32 + lane;  // element k of the warp's 32 x 64 block
    uint64_t p = base + k / kSpecN;
    if (p < n) row[(k / kSpecN) * kResolveRow + k % kSpecN] = acc[p * kSpecN + k % kSpecN];
  }
  __syncwarp();
  uint64_t p = base + lane;
  if (p >= n) return;
  const float* s = row + lane * kResolveRow;
  float X = 0.0f, Y = 0.0f, Z = 0.0f;
  for (int i = 0; i < kSpecN; ++i) {
    float v = s[i];
    X = X + v * g_spec.X[i];
    Y = Y + v * g_spec.Y[i];
    Z = Z + v * g_spec.Z[i];
  }
  float dl = (float)(wpbr_spec::kLambdaEnd - wpbr_spec::kLambdaStart) / (float)kSpecN;
  X = X * dl;
  Y = Y * dl;
  Z = Z * dl;
  float m20 = (quirks & WPBR_Q_XYZ_MATRIX_FIX) ? 0.055648f : 0.041556f;
  float r = (X * 3.240479f + Y * -1.537150f) + Z * -0.498535f;
  float g = (X * -0.969256f + Y * 1.875991f) + Z * 0.041556f;
  float b = (X * m20 + Y * -0.204043f) + Z * 1.057311f;
  float4 a = accw[p];
  accw[p] = make_float4(r, g, b, a.w);
}

}  // namespace

wpbr_status spectral_setup(wpbr_ctx* ctx) {
  RenderState& R = ctx->rs;
  size_t n = (size_t)R.W * R.H;
  SpecTables T;
  build_tables(&T);
  WPBR_CUDA(cudaMemcpyToSymbolAsync(g_spec, &T, sizeof(T), 0, cudaMemcpyHostToDevice, ctx->stream));
  // material and light spectra from the scene's RGB parameters
  std::vector<wpbr_material> mats(ctx->nmat);
  WPBR_CUDA(cudaMemcpyAsync(mats.data(), ctx->mats.p, sizeof(wpbr_material) * ctx->nmat, cudaMemcpyDeviceToHost,
                            ctx->stream));
  WPBR_CUDA(cudaStreamSynchronize(ctx->stream));
  std::vector<SpecMat> sm(ctx->nmat);
  for (uint32_t i = 0; i < ctx->nmat; ++i) {
    const wpbr_material& m = mats[i];
    sm[i].R = s64_of_param(T, RGB3{m.R[0], m.R[1], m.R[2]}, false);
    sm[i].eta_i = s64_of_param(T, RGB3{m.eta_i[0], m.eta_i[1], m.eta_i[2]}, false);
    sm[i].eta_t = s64_of_param(T, RGB3{m.eta_t[0], m.eta_t[1], m.eta_t[2]}, false);
    sm[i].k = s64_of_param(T, RGB3{m.k[0], m.k[1], m.k[2]}, false);
  }
  std::vector<S64> le(ctx->h_lights.size() ? ctx->h_lights.size() : 1);
  for (size_t i = 0; i < ctx->h_lights.size(); ++i) {
    const wpbr_light& l = ctx->h_lights[i];
    RGB3 c = l.type == WPBR_LIGHT_SPHERE ? RGB3{l.Le[0], l.Le[1], l.Le[2]} : ctx->env_le;
    le[i] = s64_of_param(T, c, false);
  }
  WPBR_CUDA(R.spec_mats.ensure(sizeof(SpecMat) * sm.size() / sizeof(float) + 1));
  WPBR_CUDA(R.spec_le.ensure(le.size() * kSpecN));
  WPBR_CUDA(cudaMemcpyAsync(R.spec_mats.p, sm.data(), sizeof(SpecMat) * sm.size(), cudaMemcpyHostToDevice,
                            ctx->stream));
  WPBR_CUDA(cudaMemcpyAsync(R.spec_le.p, le.data(), sizeof(S64) * le.size(), cudaMemcpyHostToDevice, ctx->stream));
  WPBR_CUDA(R.spec_L.ensure(n * kSpecN));
  WPBR_CUDA(R.spec_flags.ensure(n));
  WPBR_CUDA(R.spec_acc.ensure(n * kSpecN));
  WPBR_CUDA(cudaMemsetAsync(R.spec_acc.p, 0, sizeof(float) * n * kSpecN, ctx->stream));
  WPBR_CUDA(cudaStreamSynchronize(ctx->stream));
  return WPBR_OK;
}

static PassCtx spec_pass_ctx(wpbr_ctx* ctx) {
  return pass_ctx(scene_view(ctx), render_traversal_view(ctx),
                  wpbr_rng::Stream{ctx->rs.seed, ctx->rs.stream, ctx->rs.spp, (ctx->quirks & WPBR_Q_REF_SAMPLER_ARRAYS) ? 1u : 0u},
                  ctx->rs.W, ctx->rs.H, ctx->d_err.p);
}

size_t spectral_slot_bytes(size_t pixels) { return pixels * (sizeof(float2) + kSpecN * sizeof(float) + sizeof(uint32_t)); }

// Room for `slots` passes' film positions and sample spectra; without it the
// slots that are there stay.
cudaError_t spectral_slots(wpbr_ctx* ctx, uint32_t slots) {
  RenderState& R = ctx->rs;
  const size_t n = (size_t)R.W * R.H;
  cudaError_t e = R.pfilm.grow(slots * n);
  if (e == cudaSuccess) e = R.spec_L.grow(slots * n * kSpecN);
  if (e == cudaSuccess) e = R.spec_flags.grow(slots * n);
  return e;
}

// The scalar spawn of the Sampled64 pass, between the camera traversal and
// the shadow-ray traversal (render_pass_launch); the pass's film positions go
// to sample slot `slot`; tex: tex_build of the pass.
cudaError_t spectral_spawn_launch(wpbr_ctx* ctx, const PassBufs& B, const uint32_t* pass_ptr, const uint32_t* order,
                                  uint32_t slot, int tex, cudaStream_t st) {
  RenderState& R = ctx->rs;
  uint32_t n = R.W * R.H;
  const ShadowQueue sq{B.shadow_rays, B.shadow_map, B.counters + kQueueCounter};
  (tex == kTexNone ? k_sspawn<kTexNone> : tex == kTexWide ? k_sspawn<kTexWide> : k_sspawn<kTexCompact>)
      <<<div_up(n, kTB), kTB, 0, st>>>(spec_pass_ctx(ctx), pass_ptr, B.hit_prim, B.pstate, sq,
                                       R.pfilm.p + (size_t)slot * n, order);
  return cudaGetLastError();
}

// The per-bin finish after the shadow-ray traversal: the pass's spectra to
// sample slot `slot`.
cudaError_t spectral_finish_launch(wpbr_ctx* ctx, const PassBufs& B, const uint32_t* order, uint32_t slot,
                                   cudaStream_t st) {
  RenderState& R = ctx->rs;
  uint32_t n = R.W * R.H;
  SpecCtx C{(const SpecMat*)R.spec_mats.p, (const S64*)R.spec_le.p, R.spec_L.p + (size_t)slot * n * kSpecN,
            R.spec_flags.p + (size_t)slot * n};
  k_sfinish<<<div_up((uint64_t)n * kBinLanes, 128), 128, 0, st>>>(spec_pass_ctx(ctx), C, B.pstate, B.shadow_hit,
                                                                   order);
  return cudaGetLastError();
}

// The film gather of sample slots 0 .. film_slots - 1 in slot order.
cudaError_t spectral_film_launch(wpbr_ctx* ctx, uint32_t film_slots, cudaStream_t st) {
  RenderState& R = ctx->rs;
  cudaError_t e = cudaFuncSetAttribute((const void*)k_sfilm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kSFilmSmem);
  if (e != cudaSuccess) return e;
  const unsigned rows = div_up(R.H, kSRows);
  const dim3 fg(div_up(R.W, kFilmTile), std::min(rows, kMaxGridRows), div_up(rows, kMaxGridRows));
  k_sfilm<<<fg, kFilmThreads, kSFilmSmem, st>>>(R.W, R.H, R.pfilm.p, R.spec_L.p, R.spec_flags.p, film_slots,
                                                 R.spec_acc.p, (float4*)R.acc.p, kOnes);
  return cudaGetLastError();
}

// Converts the accumulated spectra to the RGB film (wpbr_film_read and
// wpbr_film_tonemap read it) when passes ran since the last conversion.
wpbr_status spectral_resolve(wpbr_ctx* ctx) {
  RenderState& R = ctx->rs;
  if (ctx->spectrum != WPBR_SPECTRUM_SAMPLED64 || !R.spec_dirty) return WPBR_OK;
  uint32_t n = R.W * R.H;
  k_sresolve<<<div_up(n, 128), 128, 0, ctx->stream>>>(n, R.spec_acc.p, (float4*)R.acc.p, ctx->quirks);
  WPBR_CUDA(cudaGetLastError());
  R.spec_dirty = false;
  return WPBR_OK;
}

}  // namespace wpbr
