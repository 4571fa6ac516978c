// adjoint.cu — the differentiable direct-lighting estimator: a forward /
// backward pair giving the gradient of an image L2 loss with respect to the
// per-material parameters (alpha, albedo R, eta, k) and the environment
// texels.
//
// The differentiated function is the frozen-direction estimator: every
// sample's directions (camera ray, light sample, BSDF sample), hit points and
// visibility come from the sampling parameters theta_s (set by
// wpbr_adjoint_freeze); the BSDF values, pdfs, MIS weights and emitted /
// incident radiance are evaluated at the current parameters theta. Its value
// at theta = theta_s is the render of MEngine::render's per-sample job list
// (WoodenPBREngine/MEngine.cpp:393-442), its derivative is the detached-
// sampling gradient, and central differences of it are well defined (no
// visibility or sampling-map discontinuities).
//
// Neither pass stores paths: the backward pass replays each sample pass
// (camera rays, primary traversal, light and BSDF sampling, shadow
// traversal) from the counter-based sample streams and runs the hand-written
// reverse sweep (shade_grad.cuh) per sample. Material gradients are summed in
// shared memory per block, then in double in global memory; texel gradients
// are atomics on a float array; the environment map's normalisation adds one
// global scalar that a final kernel spreads over every texel.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "ctx.hpp"
#include "pass.cuh"
#include "shade_grad.cuh"
#include "traverse_persistent.cuh"

namespace wpbr {

namespace {

constexpr int kAdjF4 = 6;  // float4 of frozen state per pixel
enum : uint32_t { AF_HIT = 1u, AF_TRACE_L = 2u, AF_TRACE_B = 4u };
constexpr uint32_t kMaxAdjMaterials = 1024;  // shared-memory material accumulators

struct AdjView {
  const wpbr_material* mats_s;  // sampling parameters
  const wpbr_material* mats_e;  // evaluation parameters
  EnvView env_s;                // sampling texels + distribution
  EnvView env_e;                // evaluation texels, map function, integral
};

struct AdjGrad {
  const float4* gpix;  // dLoss/dI / film weight, per pixel
  double* g_mat;       // nmat * 10
  float* g_env;        // W * H * 3, per texel and channel
  float* g_func;       // W * H, per map cell
  double* g_Z;         // derivative with respect to the map integral
  uint32_t nmat;
};

struct MatGrad {
  float a;
  float R[3], eta[3], k[3];
};

__device__ __forceinline__ bool finite3(RGB3 c) { return isfinite(c.r) && isfinite(c.g) && isfinite(c.b); }

// ---- sample generation with the sampling parameters --------------------------
__global__ void __launch_bounds__(kTB, WPBR_ADJ_SPAWN_MIN_BLOCKS) k_adj_spawn(PassCtx P, AdjView A, const uint32_t* pass_dev,
                                                   const uint32_t* hit_prim, float4* state, ShadowQueue sq, float2* pf) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H) return;
  uint32_t pass = *pass_dev;
  float fx, fy;
  camera_sample(P, pix, pass, &fx, &fy);
  pf[pix] = make_float2(fx, fy);
  RayD r = camera_ray(P.S.cam, fx, fy);
  uint32_t prim = hit_prim[pix];
  float4* st = state + (size_t)pix * kAdjF4;
  if (prim == kNoHit || P.S.nlights == 0) {
    st[0] = make_float4(r.d.x, r.d.y, r.d.z, __uint_as_float(prim == kNoHit ? 0u : AF_HIT));
    st[1] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(0xFFFFFFFFu));  // no light: nothing to shade
    return;
  }
  uint32_t flags = AF_HIT;
  SurfInt s = make_si(P.S, prim, r.o, r.d);
  Frame fr = bsdf_frame(s);
  uint32_t mid = prim_material(P.S, prim);
  const wpbr_material& ms = A.mats_s[mid];
  V3 wo_l = to_local(fr, s.wo);
  uint32_t li_idx = pick_light(P, pix, pass);
  const wpbr_light& lt = P.S.lights[li_idx];
  float u0, u1;
  V3 wi{0, 0, 0};
  RGB3 li = rgb1(0.0f);
  float lpdf = 0.0f;
  bool ok = light_sample_counts(P.S, lt);
  float uvs[3] = {0.0f, 0.0f, 0.0f};
  if (ok) {
    sample2d(P.rs, pix, pass, wpbr_rng::DIM_LIGHT, &u0, &u1);
    if (lt.type == WPBR_LIGHT_SPHERE) {
      sphere_light_sample(P.S.sph_o2w[lt.sphere_index], P.S.sph_r[lt.sphere_index], s.p, u0, u1, &wi, &lpdf);
      li = RGB3{lt.Le[0], lt.Le[1], lt.Le[2]};
    } else {
      env_li_sample(A.env_s, P.S.quirks, u0, u1, &wi, &li, &lpdf, &ok, uvs);
    }
  }
  const bool trace_l = ok && !rblack(li);
  if (trace_l) flags |= AF_TRACE_L;
  sq.push(trace_l, 2 * pix, add(s.p, mul(wi, (float)0.1)), wi);
  sample2d(P.rs, pix, pass, wpbr_rng::DIM_BSDF, &u0, &u1);
  V3 bwi_l;
  float bpdf;
  bool valid;
  bsdf_sample(ms, wo_l, u0, u1, &bwi_l, &bpdf, &valid);
  V3 bwi = to_world(fr, bwi_l);
  if (valid) flags |= AF_TRACE_B;
  sq.push(valid, 2 * pix + 1, add(s.p, mul(bwi, (float)0.01)), bwi);
  V3 wi_l = to_local(fr, wi);
  st[0] = make_float4(wo_l.x, wo_l.y, wo_l.z, __uint_as_float(flags));
  st[1] = make_float4(wi_l.x, wi_l.y, wi_l.z, __uint_as_float(li_idx));
  st[2] = make_float4(bwi_l.x, bwi_l.y, bwi_l.z, __uint_as_float(mid));
  st[3] = make_float4(bwi.x, bwi.y, bwi.z, lpdf);
  st[4] = make_float4(s.p.x, s.p.y, s.p.z, uvs[0]);
  st[5] = make_float4(uvs[1], uvs[2], 0.0f, 0.0f);
}

// ---- evaluation at theta and its reverse sweep ---------------------------------
struct EvalCtx {
  const PassCtx* P;
  const AdjView* A;
  float* smem_mat;  // block accumulators (backward only)
  float* g_env;
  float* g_func;
  double gZ;        // this thread's share of -Z dLoss/dZ
  // the sums that many lanes of a warp share (backward): a hit's material
  // partials under the material's index, or a camera miss's texel partials
  // under kTexelKey | first texel
  uint32_t key;
  float part[12];
};

__device__ __forceinline__ void add_env_taps(EvalCtx& E, const EnvView& e, float s, float t, RGB3 g) {
  int idx[4];
  float w[4];
  env_taps(e, s, t, idx, w);
  for (int k = 0; k < 4; ++k) {
    if (w[k] == 0.0f) continue;
    float* d = E.g_env + 3 * (size_t)idx[k];
    atomicAdd(d, g.r * e.le.r * w[k]);
    atomicAdd(d + 1, g.g * e.le.g * w[k]);
    atomicAdd(d + 2, g.b * e.le.b * w[k]);
  }
}

// pdf = func[cell] / Z / K: local term to the cell, global term to Z
__device__ __forceinline__ void add_env_pdf(EvalCtx& E, const EnvView& e, int cell, float pdf, float g_pdf) {
  if (g_pdf == 0.0f) return;
  float f = e.cond_func[cell];
  if (f != 0.0f) atomicAdd(E.g_func + cell, g_pdf * pdf / f);
  E.gZ += (double)g_pdf * (double)pdf;  // times -1 / Z once per block
}

constexpr uint32_t kNoKey = 0xFFFFFFFFu, kTexelKey = 0x80000000u;
__device__ __forceinline__ void add_mat(EvalCtx& E, uint32_t mid, const MatGrad& g) {
  E.key = mid;
  E.part[0] = g.a;
  for (int c = 0; c < 3; ++c) {
    E.part[1 + c] = g.R[c];
    E.part[4 + c] = g.eta[c];
    E.part[7 + c] = g.k[c];
  }
  E.part[10] = E.part[11] = 0.0f;
}
// A camera miss's texels: add_env_taps for lanes whose neighbours mostly see
// the same four texels.
__device__ __forceinline__ void share_env_taps(EvalCtx& E, const EnvView& e, float s, float t, RGB3 g) {
  int idx[4];
  float w[4];
  env_taps(e, s, t, idx, w);
  E.key = kTexelKey | (uint32_t)idx[0];
  for (int k = 0; k < 4; ++k) {
    E.part[3 * k] = g.r * e.le.r * w[k];
    E.part[3 * k + 1] = g.g * e.le.g * w[k];
    E.part[3 * k + 2] = g.b * e.le.b * w[k];
  }
}
// Adds each lane's 12 parts to their targets, one addition per target and
// distinct key of the warp instead of one per lane. Halving exchanges leave the sum
// of part 8 b4 + 4 b3 + 2 b2 + b1 in the lanes with those index bits. A warp's
// neighbouring pixels mostly share a material or four texels of the map: with
// one addition per lane the backward kernel took 118 us a pass of 512 x 512,
// most of it in the shared-memory compare-and-swap loops and the atomics'
// queues; 76 us with one per key.
__device__ __forceinline__ void add_shared(const EvalCtx& E, const EnvView& e) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t todo = __ballot_sync(0xFFFFFFFFu, E.key != kNoKey);
  while (todo) {
    const uint32_t key = __shfl_sync(0xFFFFFFFFu, E.key, __ffs(todo) - 1);
    const bool mine = E.key == key;
    todo &= ~__ballot_sync(0xFFFFFFFFu, mine);
    float v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = mine && i < 12 ? E.part[i < 12 ? i : 0] : 0.0f;
#pragma unroll
    for (int half = 8; half >= 1; half >>= 1) {
      const bool upper = lane & (2 * half);
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float keep = upper ? v[i + half] : v[i], send = upper ? v[i] : v[i + half];
        v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 2 * half);
      }
    }
    const float sum = v[0] + __shfl_xor_sync(0xFFFFFFFFu, v[0], 1);
    const uint32_t k = lane >> 1;
    if ((lane & 1u) || k >= 12 || sum == 0.0f) continue;
    if (key & kTexelKey) {
      const int i0 = (int)(key & ~kTexelKey), s0 = i0 % e.W, t0 = i0 / e.W;
      const int tap = (int)k / 3, s = min(s0 + (tap >> 1), e.W - 1), t = min(t0 + (tap & 1), e.H - 1);
      atomicAdd(E.g_env + 3 * ((size_t)t * e.W + s) + k % 3, sum);
    } else if (k < 10) {
      atomicAdd(E.smem_mat + 10 * key + k, sum);
    }
  }
}

// bsdf_eval at theta (value includes |cos wi|) and, given the upstream
// gradients of the value and the pdf, the material partials.
template <bool BACK>
__device__ RGB3 bsdf_eval_ad(const wpbr_material& m, V3 wo, V3 wi, float* pdf, RGB3 gf, float gpdf, MatGrad* g) {
  if (m.type == WPBR_MAT_SPECULAR) {
    *pdf = 0.0f;
    return rgb1(0.0f);
  }
  V3 wh = normalize(add(wo, wi));
  float dD;
  float D = tr_d_grad(m.alpha_x, m.alpha_y, wh, &dD);
  float cwh = abs_cos(wh), dow = dot(wo, wh);
  *pdf = (D * cwh) / (4.0f * dow);
  float co = abs_cos(wo), ci = abs_cos(wi);
  bool zero_f = (ci == 0.0f || co == 0.0f || (wh.x == 0.0f && wh.y == 0.0f && wh.z == 0.0f));
  float c = dot(wi, wh);
  float K = abs_cos(wi) / ((4.0f * ci) * co);
  RGB3 f = rgb1(0.0f);
  float gD = BACK ? gpdf * cwh / (4.0f * dow) : 0.0f;
  if (!zero_f) {
    if (m.type == WPBR_MAT_CONDUCTOR) {
      float Fc[3];
      for (int ch = 0; ch < 3; ++ch) {
        float de, dk;
        Fc[ch] = fresnel_conductor_grad(c, m.eta_i[ch], m.eta_t[ch], m.k[ch], &de, &dk);
        if (BACK) {
          float gfc = ch == 0 ? gf.r : (ch == 1 ? gf.g : gf.b);
          g->R[ch] += gfc * Fc[ch] * D * K;
          gD += gfc * Fc[ch] * m.R[ch] * K;
          float gF = gfc * m.R[ch] * D * K;
          g->eta[ch] += gF * de;
          g->k[ch] += gF * dk;
        }
      }
      f = RGB3{Fc[0] * m.R[0] * D * K, Fc[1] * m.R[1] * D * K, Fc[2] * m.R[2] * D * K};
    } else {
      float de;
      float Fd = fresnel_dielectric_grad(c, m.eta_i[0], m.eta_t[0], &de);
      if (BACK) {
        float gsum = 0.0f;
        for (int ch = 0; ch < 3; ++ch) {
          float gfc = ch == 0 ? gf.r : (ch == 1 ? gf.g : gf.b);
          g->R[ch] += gfc * Fd * D * K;
          gD += gfc * Fd * m.R[ch] * K;
          gsum += gfc * m.R[ch] * D * K;
        }
        g->eta[0] += gsum * de;
      }
      f = RGB3{m.R[0] * Fd * D * K, m.R[1] * Fd * D * K, m.R[2] * Fd * D * K};
    }
  }
  if (BACK) g->a += gD * dD;
  return f;
}

// value of a BSDF-sampled direction: the specular lobe's sample value, else
// the microfacet evaluation; pdf 1 marks the delta lobe.
template <bool BACK>
__device__ RGB3 bsdf_branch_f(const wpbr_material& m, V3 wo, V3 wi, float* pdf, RGB3 gf, float gpdf, MatGrad* g) {
  if (m.type != WPBR_MAT_SPECULAR) return bsdf_eval_ad<BACK>(m, wo, wi, pdf, gf, gpdf, g);
  *pdf = 1.0f;
  if (abs_cos(wi) == 0.0f) return rgb1(0.0f);
  float de;
  float fr = fresnel_dielectric_grad(wi.z, m.eta_i[0], m.eta_t[0], &de);
  if (BACK) {
    g->R[0] += gf.r * fr;
    g->R[1] += gf.g * fr;
    g->R[2] += gf.b * fr;
    g->eta[0] += (gf.r * m.R[0] + gf.g * m.R[1] + gf.b * m.R[2]) * de;
  }
  return RGB3{m.R[0] * fr, m.R[1] * fr, m.R[2] * fr};
}

// One branch of a sample at theta: what its value li f w / pdf and its
// derivatives are made of. pdf is the sampling density of the branch's
// direction (lpdf for the light branch, bpdf for the BSDF one), opdf the
// other strategy's.
struct AdjBranch {
  RGB3 li, f;
  float pdf, opdf, w, dw, dwo;  // weight and its derivatives with respect to pdf and opdf
  int cell;                     // environment map cell, -1: no environment light
  float eu, ev;                 // its map coordinates
  bool on;                      // contributes
};
__device__ __forceinline__ RGB3 branch_value(const AdjBranch& b) { return rmuls(rmul(b.li, b.f), b.w / b.pdf); }

// The light-sampling branch: L += li f w / lpdf.
__device__ __forceinline__ AdjBranch light_branch(const PassCtx& P, const AdjView& A, const wpbr_light& lt,
                                                  const wpbr_material& m, V3 wo, V3 wi, float lpdf, float es, float et,
                                                  float sin_theta) {
  AdjBranch b;
  b.cell = -1;
  b.eu = es;
  b.ev = et;
  if (lt.type == WPBR_LIGHT_SPHERE) {
    b.li = RGB3{lt.Le[0], lt.Le[1], lt.Le[2]};
    b.pdf = lpdf;
  } else {
    b.li = (P.S.quirks & WPBR_Q_ENV_LI_SAMPLE_FIX) ? rmul(env_bilerp(A.env_e, es, et), A.env_e.le) : rgb1(0.0f);
    b.cell = env_cell(A.env_e, es, et);
    b.pdf = (sin_theta != 0.0f) ? env_pdf_cell(A.env_e, b.cell, sin_theta) : 0.0f;
  }
  b.f = bsdf_eval_ad<false>(m, wo, wi, &b.opdf, rgb1(0.0f), 0.0f, nullptr);
  b.on = b.opdf != 0.0f;
  b.w = power_heuristic_grad(b.pdf, b.opdf, &b.dw, &b.dwo);
  return b;
}
// The BSDF-sampling branch: L += li f w / bpdf.
__device__ __forceinline__ AdjBranch bsdf_branch(const PassCtx& P, const AdjView& A, const wpbr_light& lt,
                                                 const wpbr_material& m, V3 wo, V3 wi, V3 wiw, V3 p) {
  AdjBranch b;
  b.cell = -1;
  b.eu = b.ev = 0.0f;
  b.on = false;
  b.f = rgb1(0.0f);
  b.pdf = b.w = b.dw = b.dwo = 0.0f;
  if (lt.type == WPBR_LIGHT_SPHERE) {
    b.opdf = sphere_light_pdf(P.S.sph_o2w[lt.sphere_index], P.S.sph_r[lt.sphere_index], p, P.S.quirks);
    b.li = RGB3{lt.Le[0], lt.Le[1], lt.Le[2]};
  } else {
    V3 wl = xvector(A.env_e.w2l, wiw);
    float theta = sph_theta(wl);
    float phi = sph_phi(wl);
    b.eu = div_const(phi, kTwoPiDiv);
    b.ev = div_const(theta, kPiDiv);
    float sth = sinf_(theta);
    b.li = rgb1(0.0f);
    b.opdf = 0.0f;
    if (sth != 0.0f) {
      b.cell = env_cell(A.env_e, b.eu, b.ev);
      b.opdf = env_pdf_cell(A.env_e, b.cell, sth);
      b.li = rmul(env_bilerp(A.env_e, b.eu, b.ev), A.env_e.le);
    }
  }
  if (rblack(b.li)) return b;
  b.f = bsdf_branch_f<false>(m, wo, wi, &b.pdf, rgb1(0.0f), 0.0f, nullptr);
  if (b.pdf == 0.0f) return b;
  b.on = true;
  b.w = (b.pdf == 1.0f) ? 1.0f : power_heuristic_grad(b.pdf, b.opdf, &b.dw, &b.dwo);
  return b;
}
// Upstream gradients of a branch's parts.
struct BranchGrad {
  RGB3 li, f;
  float pdf, opdf;
};
__device__ __forceinline__ BranchGrad branch_grad(const AdjBranch& b, RGB3 gL) {
  const float T = b.w / b.pdf;
  BranchGrad g;
  g.li = RGB3{gL.r * b.f.r * T, gL.g * b.f.g * T, gL.b * b.f.b * T};
  g.f = RGB3{gL.r * b.li.r * T, gL.g * b.li.g * T, gL.b * b.li.b * T};
  const float gT = gL.r * b.li.r * b.f.r + gL.g * b.li.g * b.f.g + gL.b * b.li.b * b.f.b;
  const float gw = gT / b.pdf;
  g.pdf = -gT * b.w / (b.pdf * b.pdf) + gw * b.dw;
  g.opdf = gw * b.dwo;
  return g;
}

// One sample at theta: the return value is L. BACK: gL(L) gives dLoss/dL of
// this sample (zero: nothing to propagate), and the partials are accumulated.
// Each branch is evaluated once and its value's parts are kept for the
// reverse sweep. (The backward kernel evaluated every sample first for its
// value, a second time for its parts and in the reverse sweep a third time:
// 47 M instructions and 134 us a pass of 512 x 512; once, 34 M and 118 us.)
template <bool BACK, class GL>
__device__ __forceinline__ RGB3 eval_sample(EvalCtx& E, const float4* st, const uint32_t* shadow, uint32_t pix, GL gL) {
  const PassCtx& P = *E.P;
  const AdjView& A = *E.A;
  const float4 s0 = st[0];
  const uint32_t flags = __float_as_uint(s0.w);
  if (!(flags & AF_HIT)) {
    if (!P.S.has_env) return rgb1(0.0f);
    const V3 dl = xvector(A.env_e.w2l, V3{s0.x, s0.y, s0.z});
    const float s = div_const(sph_phi(dl), kTwoPiDiv);
    const float t = div_const(sph_theta(dl), kPiDiv);
    const RGB3 L = rmul(env_bilerp(A.env_e, s, t), A.env_e.le);
    if (BACK) {
      const RGB3 g = gL(L);
      if (!rblack(g)) share_env_taps(E, A.env_e, s, t, g);
    }
    return L;
  }
  RGB3 L = rgb1(0.0f);
  const float4 s1 = st[1];
  const uint32_t li_idx = __float_as_uint(s1.w);
  if (li_idx == 0xFFFFFFFFu) return L;
  const float4 s2 = st[2], s3 = st[3], s4 = st[4], s5 = st[5];
  const uint32_t mid = __float_as_uint(s2.w);
  const wpbr_material& m = A.mats_e[mid];
  const wpbr_light& lt = P.S.lights[li_idx];
  const uint32_t lp = light_prim(lt);
  const V3 wo{s0.x, s0.y, s0.z}, wl{s1.x, s1.y, s1.z}, wb{s2.x, s2.y, s2.z};
  AdjBranch bl, bb;
  bl.on = bb.on = false;
  if ((flags & AF_TRACE_L) && (shadow[2 * pix] == kNoHit || shadow[2 * pix] == lp)) {
    bl = light_branch(P, A, lt, m, wo, wl, s3.w, s4.w, s5.x, s5.y);
    if (bl.on) L = radd(L, branch_value(bl));
  }
  if ((flags & AF_TRACE_B) && (shadow[2 * pix + 1] == kNoHit || shadow[2 * pix + 1] == lp)) {
    bb = bsdf_branch(P, A, lt, m, wo, wb, V3{s3.x, s3.y, s3.z}, V3{s4.x, s4.y, s4.z});
    if (bb.on) L = radd(L, branch_value(bb));
  }
  if (BACK && (bl.on || bb.on)) {
    const RGB3 up = gL(L);
    if (!rblack(up)) {
      MatGrad g{};
      float pdf;
      if (bl.on) {
        const BranchGrad q = branch_grad(bl, up);
        bsdf_eval_ad<true>(m, wo, wl, &pdf, q.f, q.opdf, &g);
        if (bl.cell >= 0) {
          if (P.S.quirks & WPBR_Q_ENV_LI_SAMPLE_FIX) add_env_taps(E, A.env_e, bl.eu, bl.ev, q.li);
          add_env_pdf(E, A.env_e, bl.cell, bl.pdf, q.pdf);
        }
      }
      if (bb.on) {
        const BranchGrad q = branch_grad(bb, up);
        bsdf_branch_f<true>(m, wo, wb, &pdf, q.f, q.pdf, &g);
        if (bb.cell >= 0) {
          add_env_taps(E, A.env_e, bb.eu, bb.ev, q.li);
          add_env_pdf(E, A.env_e, bb.cell, bb.opdf, q.opdf);
        }
      }
      add_mat(E, mid, g);
    }
  }
  return L;
}

// Forward: the sample's radiance (non-finite samples contribute nothing).
__global__ void __launch_bounds__(kTB) k_adj_eval(PassCtx P, AdjView A, const float4* state, const uint32_t* shadow,
                                                  float4* Lb) {
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= P.W * P.H) return;
  EvalCtx E{&P, &A, nullptr, nullptr, nullptr, 0.0, kNoKey};
  RGB3 L = eval_sample<false>(E, state + (size_t)pix * kAdjF4, shadow, pix, [](RGB3) { return rgb1(0.0f); });
  if (!finite3(L)) L = rgb1(0.0f);
  Lb[pix] = make_float4(L.r, L.g, L.b, 0.0f);
}


// dLoss/dL of a sample: the transpose of the tile-clipped film gather (the
// factors of k_film_tiles over the sample's own footprint).
__device__ __forceinline__ RGB3 film_adjoint(uint32_t W, uint32_t H, int sx, int sy, float2 f, const float4* gpix) {
  const int tx0 = sx / 32 * 32, ty0 = sy / 32 * 32;
  const int tx1 = min(tx0 + 31, (int)W - 1), ty1 = min(ty0 + 31, (int)H - 1);
  const float dx0 = f.x - 0.5f, dy0 = f.y - 0.5f;
  const int pminx = max((int)ceilf(dx0 - 2.0f), tx0), pmaxx = min((int)floorf(dx0 + 2.0f), tx1);
  const int pminy = max((int)ceilf(dy0 - 2.0f), ty0), pmaxy = min((int)floorf(dy0 + 2.0f), ty1);
  float mx[5], my[5];
  film_factors(f.x, sx, tx0, tx1, mx);
  film_factors(f.y, sy, ty0, ty1, my);
  RGB3 g = rgb1(0.0f);
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    const int y = sy - 2 + j;
    if (y < pminy || y > pmaxy) continue;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const int x = sx - 2 + i;
      if (x < pminx || x > pmaxx) continue;
      const float w = mx[i] * my[j];
      const float4 gp = gpix[(size_t)y * W + x];
      g = radd(g, RGB3{gp.x * w, gp.y * w, gp.z * w});
    }
  }
  return g;
}

// Backward: replayed sample, film adjoint, reverse sweep.
__global__ void __launch_bounds__(kTB, WPBR_ADJ_BACK_MIN_BLOCKS) k_adj_back(PassCtx P, AdjView A, const float4* state, const uint32_t* shadow,
                                                  const float2* pf, AdjGrad G) {
  extern __shared__ float smem[];
  __shared__ double zsum[kTB / 32];
  uint32_t nm = G.nmat * 10;
  for (uint32_t j = threadIdx.x; j < nm; j += blockDim.x) smem[j] = 0.0f;
  __syncthreads();
  uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
  EvalCtx E{&P, &A, smem, G.g_env, G.g_func, 0.0, kNoKey};
  if (pix < P.W * P.H) {
    eval_sample<true>(E, state + (size_t)pix * kAdjF4, shadow, pix, [&](RGB3 L) {
      if (!finite3(L)) return rgb1(0.0f);
      uint32_t x;
      const uint32_t y = div_mod(pix, P.row, &x);
      return film_adjoint(P.W, P.H, (int)x, (int)y, pf[pix], G.gpix);
    });
  }
  __syncwarp();
  add_shared(E, A.env_e);
  double z = E.gZ;
  for (int o = 16; o > 0; o >>= 1) z += __shfl_down_sync(0xFFFFFFFFu, z, o);
  if ((threadIdx.x & 31) == 0) zsum[threadIdx.x >> 5] = z;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kTB / 32; ++w) t += zsum[w];
    if (t != 0.0) atomicAdd(G.g_Z, -t / (double)A.env_e.marg_int);
  }
  for (uint32_t j = threadIdx.x; j < nm; j += blockDim.x)
    if (smem[j] != 0.0f) atomicAdd(G.g_mat + j, (double)smem[j]);
}

// Per pixel: I = acc.rgb / acc.w, loss += |I - T|^2, gpix = 2 (I - T) / (3 N acc.w).
__global__ void k_adj_loss(uint32_t n, const float4* acc, const float* target, float4* gpix, float* image,
                           double* loss) {
  __shared__ double part[256 / 32];
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  double l = 0.0;
  if (i < n) {
    float4 a = acc[i];
    float I[3] = {a.x / a.w, a.y / a.w, a.z / a.w};
    if (image) {
      image[3 * (size_t)i] = I[0];
      image[3 * (size_t)i + 1] = I[1];
      image[3 * (size_t)i + 2] = I[2];
    }
    if (target) {
      float g[3];
      float sc = 2.0f / (3.0f * (float)n * a.w);
      for (int c = 0; c < 3; ++c) {
        float d = I[c] - target[3 * (size_t)i + c];
        l += (double)d * (double)d;
        g[c] = d * sc;
      }
      gpix[i] = make_float4(g[0], g[1], g[2], 0.0f);
    }
  }
  for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xFFFFFFFFu, l, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = l;
  __syncthreads();
  if (threadIdx.x == 0 && target) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x / 32); ++w) t += part[w];
    atomicAdd(loss, t);
  }
}

// Map function cells -> texel green channel, through k_env_rows' lookups:
// func[i] = green(bilerp(x/W, y/H)) * sin(theta_y); every cell also carries
// dLoss/dZ * dZ/dfunc = g_Z / (W H).
__global__ void k_adj_env_finish(EnvView e, uint32_t quirks, const float* g_func, const double* g_Z, float* g_env) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t W = e.W, H = e.H;
  if (i >= W * H) return;
  uint32_t x, y;
  if (quirks & WPBR_Q_ENV_DISTRIB_INDEX_BUG) {
    uint32_t yy = min(H - 1, i / H);
    uint32_t xx = i - yy * H;
    if (xx >= W) return;
    x = xx;
    y = yy;
  } else {
    x = i % W;
    y = i / W;
  }
  float g = g_func[i] + (float)(*g_Z / ((double)W * (double)H));
  if (g == 0.0f) return;
  float yN = (float)y / (float)H;
  float sin_t = (float)sin_d((kPI * (double)(float)((float)y + 0.5f)) / (double)(float)H);
  float xN = (float)x / (float)W;
  int idx[4];
  float w[4];
  env_taps(e, xN, yN, idx, w);
  for (int k = 0; k < 4; ++k)
    if (w[k] != 0.0f) atomicAdd(g_env + 3 * (size_t)idx[k] + 1, g * sin_t * w[k]);
}

__global__ void k_apply_mat_params(const float* prm, uint32_t nmat, wpbr_material* mats) {
  uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= nmat) return;
  const float* p = prm + 10 * (size_t)m;
  wpbr_material& d = mats[m];
  d.alpha_x = p[0];
  d.alpha_y = p[0];
  for (int c = 0; c < 3; ++c) {
    d.R[c] = p[1 + c];
    d.eta_t[c] = p[4 + c];
    d.k[c] = p[7 + c];
  }
}

// pass index words, read by the passes' kernels
__global__ void k_iota(uint32_t n, uint32_t* out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = i;
}

__global__ void k_mat_grad_out(const double* g, uint32_t n, float* out) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (float)g[i];
}

}  // namespace

// ---- host side ---------------------------------------------------------------------

namespace {

EnvView env_view_of(const wpbr_ctx* ctx, const float4* rgb, const float* func, const float* cdf, const float* cint,
                    const float* mfunc, const float* mcdf, float Z) {
  EnvView e = scene_view(ctx).env;
  e.rgb = rgb;
  e.cond_func = func;
  e.cond_cdf = cdf;
  e.cond_int = cint;
  e.marg_func = mfunc;
  e.marg_cdf = mcdf;
  e.marg_int = Z;
  return e;
}

AdjView adj_view(const wpbr_ctx* ctx) {
  const AdjState& J = ctx->adj;
  AdjView A;
  A.mats_s = J.mats_s.p;
  A.mats_e = J.mats_e.p;
  A.env_s = env_view_of(ctx, J.rgb_s.p, J.s_func.p, J.s_cdf.p, J.s_int.p, J.s_mfunc.p, J.s_mcdf.p, J.Z_s);
  A.env_e = env_view_of(ctx, J.rgb_e.p, J.e_func.p, J.e_cdf.p, J.e_int.p, J.e_mfunc.p, J.e_mcdf.p, J.Z_e);
  return A;
}

PassCtx adj_pass_ctx(wpbr_ctx* ctx) {
  return pass_ctx(scene_view(ctx), render_traversal_view(ctx),
                  wpbr_rng::Stream{ctx->adj.seed, ctx->adj.stream, ctx->adj.spp, (ctx->quirks & WPBR_Q_REF_SAMPLER_ARRAYS) ? 1u : 0u},
                  ctx->adj.W, ctx->adj.H, ctx->d_err.p);
}

wpbr_status rebuild_eval_distribution(wpbr_ctx* ctx) {
  AdjState& J = ctx->adj;
  if (!ctx->has_env) return WPBR_OK;
  EnvDist d{J.e_func.p, J.e_cdf.p, J.e_int.p, J.e_mfunc.p, J.e_mcdf.p, J.e_mint.p};
  return env_distribution_build(ctx, J.rgb_e.p, d, &J.Z_e);
}

// ---- passes in flight ----------------------------------------------------------
// The passes are independent up to their film gathers (forward) and gradient
// sums (backward), and one pass of a 512 x 512 film leaves 60 % of the warp
// slots empty, so several run side by side, each in a state slice on a stream
// of its own; the film gathers follow in pass order on the context's stream.
// As many as hold 2^19 pixels together, at most 8. A 512 x 512 x 16 spp step: 1
// pass at a time 5.68 ms, 2 4.66, 4 4.79, 8 4.76 (more state than L2 holds).
constexpr uint64_t kLanePixels = 1ull << 19;

// One pass's per-pixel state.
struct AdjBufs {
  float4 *state, *rays, *Lb;
  float2* pf;
  uint32_t *hit_prim, *shadow_hit, *shadow_map;
};
template <class F>
size_t adj_slice_layout(size_t n, F&& part) {
  size_t at = 0;
  for (size_t bytes : {n * kAdjF4 * 16, n * 64, n * 16, n * 8, n * 4, n * 8, n * 8}) {
    part(at);
    at += (bytes + 255) / 256 * 256;
  }
  return at;
}
size_t adj_slice_bytes(size_t n) {
  return adj_slice_layout(n, [](size_t) {});
}
AdjBufs adj_bufs(const AdjState& J, uint32_t lane) {
  if (lane == 0) return AdjBufs{J.state.p, J.rays.p, J.Lb.p, J.pf.p, J.hit_prim.p, J.shadow_hit.p, J.shadow_map.p};
  const size_t n = (size_t)J.W * J.H;
  unsigned char *base = J.slices.p + (size_t)(lane - 1) * adj_slice_bytes(n), *at[7];
  int k = 0;
  adj_slice_layout(n, [&](size_t off) { at[k++] = base + off; });
  return AdjBufs{(float4*)at[0], (float4*)at[1], (float4*)at[2], (float2*)at[3],
                 (uint32_t*)at[4], (uint32_t*)at[5], (uint32_t*)at[6]};
}

// Slices, streams and events for the passes in flight; a device without room
// for them runs one pass at a time.
wpbr_status adj_lanes(wpbr_ctx* ctx, uint32_t* lanes) {
  AdjState& J = ctx->adj;
  const size_t n = (size_t)J.W * J.H;
  uint32_t K = (uint32_t)std::min<uint64_t>({AdjState::kLanes, J.spp, (kLanePixels + n - 1) / n});
  if (K > 1) {
    cudaError_t e = J.slices.ensure((K - 1) * adj_slice_bytes(n));
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      J.slices.release();
      K = 1;
    } else {
      WPBR_CUDA(e);
    }
  }
  if (K > 1) {
    for (uint32_t k = 0; k < K; ++k) {
      if (!J.lane[k]) WPBR_CUDA(cudaStreamCreateWithFlags(&J.lane[k], cudaStreamNonBlocking));
      for (cudaEvent_t* ev : {&J.ready_ev[k], &J.free_ev[k]})
        if (!*ev) WPBR_CUDA(cudaEventCreateWithFlags(ev, cudaEventDisableTiming));
    }
    if (!J.fork_ev) WPBR_CUDA(cudaEventCreateWithFlags(&J.fork_ev, cudaEventDisableTiming));
  }
  *lanes = K;
  return WPBR_OK;
}

// camera + primary traversal + sampling + shadow traversal of one pass
wpbr_status replay_pass(wpbr_ctx* ctx, const PassCtx& P, const AdjView& A, uint32_t pass, const AdjBufs& B,
                        uint32_t share, cudaStream_t st) {
  AdjState& J = ctx->adj;
  uint32_t n = J.W * J.H;
  const uint32_t* word = J.pass_dev.p + pass;
  uint32_t* counters = J.counters.p + 3 * (size_t)pass;  // two ray fetches, the queued shadow rays
  launch_traversal<false>(P.S, P.Bv, CameraSrc{P, word}, PrimSink{B.hit_prim}, n, counters, P.err, st, 0, share);
  // shadow rays: the spawn queues the ones it traces, the traversal walks the queue
  const ShadowQueue sq{B.rays, B.shadow_map, counters + 2};
  k_adj_spawn<<<div_up(n, kTB), kTB, 0, st>>>(P, A, word, B.hit_prim, B.state, sq, B.pf);
  launch_traversal<false>(P.S, P.Bv, QueueSrc{sq.rays, sq.count}, MapSink{B.shadow_hit, sq.map}, 2 * n, counters + 1,
                          P.err, st, 0, share);
  WPBR_CUDA(cudaGetLastError());
  return WPBR_OK;
}

// Every pass: its samples (replay_pass, then per_sample(pass, B, stream)) in a
// lane, then after(pass, B) on the context's stream in pass order.
template <class PerSample, class After>
wpbr_status adj_passes(wpbr_ctx* ctx, const PassCtx& P, const AdjView& A, PerSample&& per_sample, After&& after) {
  AdjState& J = ctx->adj;
  cudaStream_t st = ctx->stream;
  uint32_t K = 1;
  wpbr_status s = adj_lanes(ctx, &K);
  if (s != WPBR_OK) return s;
  WPBR_CUDA(cudaMemsetAsync(J.counters.p, 0, sizeof(uint32_t) * 3 * J.spp, st));
  if (K > 1) {
    WPBR_CUDA(cudaEventRecord(J.fork_ev, st));
    for (uint32_t k = 0; k < K; ++k) WPBR_CUDA(cudaStreamWaitEvent(J.lane[k], J.fork_ev, 0));
  }
  cudaError_t e = cudaSuccess;
  for (uint32_t p = 0; p < J.spp && e == cudaSuccess && s == WPBR_OK; ++p) {
    const uint32_t k = p % K;
    const AdjBufs B = adj_bufs(J, k);
    cudaStream_t ls = K > 1 ? J.lane[k] : st;
    if (K > 1 && p >= K) e = cudaStreamWaitEvent(ls, J.free_ev[k], 0);  // the slice's last pass is in the film
    if (e != cudaSuccess) break;
    s = replay_pass(ctx, P, A, p, B, K, ls);
    if (s != WPBR_OK) break;
    per_sample(p, B, ls);
    if (K > 1) {
      e = cudaEventRecord(J.ready_ev[k], ls);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(st, J.ready_ev[k], 0);
    }
    if (e == cudaSuccess) after(p, B);
    if (e == cudaSuccess && K > 1) e = cudaEventRecord(J.free_ev[k], st);
  }
  if (s != WPBR_OK || e != cudaSuccess) {  // nothing of this call runs on after it
    for (uint32_t k = 0; k < K && K > 1; ++k) cudaStreamSynchronize(J.lane[k]);
    if (s != WPBR_OK) return s;
  }
  WPBR_CUDA(e);
  WPBR_CUDA(cudaGetLastError());
  return WPBR_OK;
}

}  // namespace

wpbr_status adjoint_setup(wpbr_ctx* ctx, uint32_t spp, uint32_t seed, uint32_t stream) {
  if (!ctx->has_scene) return set_err(ctx, WPBR_ERR_NOT_BUILT, "adjoint_setup: no scene");
  if (!ctx->bvh.built) return set_err(ctx, WPBR_ERR_NOT_BUILT, "adjoint_setup: BVH not built");
  if (spp == 0) return set_err(ctx, WPBR_ERR_INVALID_ARG, "adjoint_setup: spp must be > 0");
  if (ctx->spectrum != WPBR_SPECTRUM_RGB)
    return set_err(ctx, WPBR_ERR_INVALID_ARG, "adjoint_setup: the differentiable estimator runs in RGB mode only");
  if (ctx->has_metal)
    return set_err(ctx, WPBR_ERR_INVALID_ARG, "adjoint_setup: textured metal materials have no material parameters");
  if (ctx->nmat > kMaxAdjMaterials)
    return set_err(ctx, WPBR_ERR_INVALID_ARG, "adjoint_setup: more than 1024 materials");
  AdjState& J = ctx->adj;
  cudaStream_t st = ctx->stream;
  J.ready = false;  // until every buffer below exists
  J.spp = spp;
  J.seed = seed;
  J.stream = stream;
  J.W = ctx->cam.W;
  J.H = ctx->cam.H;
  J.nmat = ctx->nmat;
  size_t n = (size_t)J.W * J.H;
  WPBR_CUDA(J.mats_s.ensure(J.nmat));
  WPBR_CUDA(J.mats_e.ensure(J.nmat));
  WPBR_CUDA(cudaMemcpyAsync(J.mats_s.p, ctx->mats.p, sizeof(wpbr_material) * J.nmat, cudaMemcpyDeviceToDevice, st));
  WPBR_CUDA(cudaMemcpyAsync(J.mats_e.p, ctx->mats.p, sizeof(wpbr_material) * J.nmat, cudaMemcpyDeviceToDevice, st));
  J.h_mats.resize(J.nmat);
  WPBR_CUDA(cudaMemcpyAsync(J.h_mats.data(), ctx->mats.p, sizeof(wpbr_material) * J.nmat, cudaMemcpyDeviceToHost, st));
  size_t nt = ctx->has_env ? (size_t)ctx->envW * ctx->envH : 0;
  J.n_texels = nt;
  if (ctx->has_env) {
    uint32_t EW = ctx->envW, EH = ctx->envH;
    for (DevBuf<float4>* b : {&J.rgb_s, &J.rgb_e}) WPBR_CUDA(b->ensure(nt));
    for (DevBuf<float>* b : {&J.s_func, &J.e_func}) WPBR_CUDA(b->ensure(nt));
    for (DevBuf<float>* b : {&J.s_cdf, &J.e_cdf}) WPBR_CUDA(b->ensure((size_t)EH * (EW + 1)));
    for (DevBuf<float>* b : {&J.s_int, &J.e_int, &J.s_mfunc, &J.e_mfunc}) WPBR_CUDA(b->ensure(EH));
    for (DevBuf<float>* b : {&J.s_mcdf, &J.e_mcdf}) WPBR_CUDA(b->ensure(EH + 1));
    for (DevBuf<float>* b : {&J.s_mint, &J.e_mint}) WPBR_CUDA(b->ensure(1));
    WPBR_CUDA(J.g_env.ensure(nt * 3));
    WPBR_CUDA(J.g_func.ensure(nt));
    WPBR_CUDA(J.env_prm.ensure(nt * 3));
    WPBR_CUDA(cudaMemcpyAsync(J.rgb_e.p, ctx->env_rgb.p, sizeof(float4) * nt, cudaMemcpyDeviceToDevice, st));
    WPBR_CUDA(cudaMemcpyAsync(J.rgb_s.p, ctx->env_rgb.p, sizeof(float4) * nt, cudaMemcpyDeviceToDevice, st));
    wpbr_status s = rebuild_eval_distribution(ctx);
    if (s != WPBR_OK) return s;
    EnvDist d{J.s_func.p, J.s_cdf.p, J.s_int.p, J.s_mfunc.p, J.s_mcdf.p, J.s_mint.p};
    s = env_distribution_build(ctx, J.rgb_s.p, d, &J.Z_s);
    if (s != WPBR_OK) return s;
  } else {
    WPBR_CUDA(J.g_env.ensure(1));
    WPBR_CUDA(J.g_func.ensure(1));
  }
  WPBR_CUDA(J.mat_prm.ensure((size_t)J.nmat * 10));
  WPBR_CUDA(J.g_mat.ensure((size_t)J.nmat * 10));
  WPBR_CUDA(J.g_scalar.ensure(2));
  WPBR_CUDA(J.state.ensure(n * kAdjF4));
  WPBR_CUDA(J.rays.ensure(n * 4));
  WPBR_CUDA(J.pf.ensure(n));
  WPBR_CUDA(J.Lb.ensure(n));
  WPBR_CUDA(J.acc.ensure(n));
  WPBR_CUDA(J.gpix.ensure(n));
  WPBR_CUDA(J.target.ensure(n * 3));
  WPBR_CUDA(J.image.ensure(n * 3));
  WPBR_CUDA(J.hit_prim.ensure(n));
  WPBR_CUDA(J.shadow_hit.ensure(2 * n));
  WPBR_CUDA(J.shadow_map.ensure(2 * n));
  WPBR_CUDA(J.pass_dev.ensure(spp));
  WPBR_CUDA(J.counters.ensure(3 * (size_t)spp));
  k_iota<<<div_up(spp, 256), 256, 0, st>>>(spp, J.pass_dev.p);
  WPBR_CUDA(cudaGetLastError());
  WPBR_CUDA(cudaStreamSynchronize(st));
  J.ready = true;
  J.param_gen += 1;
  J.fwd_gen = 0;
  return WPBR_OK;
}

wpbr_status adjoint_get_params(wpbr_ctx* ctx, float* mat, float* env) {
  AdjState& J = ctx->adj;
  if (!J.ready) return set_err(ctx, WPBR_ERR_NOT_BUILT, "adjoint: adjoint_setup not called");
  cudaStream_t st = ctx->stream;
  if (mat) {
    std::vector<wpbr_material> m(J.nmat);
    WPBR_CUDA(cudaMemcpyAsync(m.data(), J.mats_e.p, sizeof(wpbr_material) * J.nmat, cudaMemcpyDeviceToHost, st));
    WPBR_CUDA(cudaStreamSynchronize(st));
    for (uint32_t i = 0; i < J.nmat; ++i) {
      float* p = mat + 10 * (size_t)i;
      p[0] = m[i].alpha_x;
      for (int c = 0; c < 3; ++c) {
        p[1 + c] = m[i].R[c];
        p[4 + c] = m[i].eta_t[c];
        p[7 + c] = m[i].k[c];
      }
    }
  }
  if (env && J.n_texels) {
    std::vector<float4> t(J.n_texels);
    WPBR_CUDA(cudaMemcpyAsync(t.data(), J.rgb_e.p, sizeof(float4) * J.n_texels, cudaMemcpyDeviceToHost, st));
    WPBR_CUDA(cudaStreamSynchronize(st));
    for (size_t i = 0; i < J.n_texels; ++i) {
      env[3 * i] = t[i].x;
      env[3 * i + 1] = t[i].y;
      env[3 * i + 2] = t[i].z;
    }
  }
  return WPBR_OK;
}

wpbr_status adjoint_set_params(wpbr_ctx* ctx, const float* mat, const float* env, bool device) {
  AdjState& J = ctx->adj;
  if (!J.ready) return set_err(ctx, WPBR_ERR_NOT_BUILT, "adjoint: adjoint_setup not called");
  cudaStream_t st = ctx->stream;
  if (mat) {
    const float* src = mat;
    if (!device) {
      WPBR_CUDA(cudaMemcpyAsync(J.mat_prm.p, mat, sizeof(float) * 10 * J.nmat, cudaMemcpyHostToDevice, st));
      src = J.mat_prm.p;
    }
    k_apply_mat_params<<<div_up(J.nmat, 128), 128, 0, st>>>(src, J.nmat, J.mats_e.p);
    WPBR_CUDA(cudaGetLastError());
  }
  if (env && J.n_texels) {
    const float* src = env;
    if (!device) {
      WPBR_CUDA(cudaMemcpyAsync(J.env_prm.p, env, sizeof(float) * 3 * J.n_texels, cudaMemcpyHostToDevice, st));
      src = J.env_prm.p;
    }
    WPBR_CUDA(rgb_to_texels(src, J.n_texels, J.rgb_e.p, st));
    wpbr_status s = rebuild_eval_distribution(ctx);
    if (s != WPBR_OK) return s;
  }
  J.param_gen += 1;
  return WPBR_OK;
}

wpbr_status adjoint_freeze(wpbr_ctx* ctx) {
  AdjState& J = ctx->adj;
  if (!J.ready) return set_err(ctx, WPBR_ERR_NOT_BUILT, "adjoint: adjoint_setup not called");
  cudaStream_t st = ctx->stream;
  WPBR_CUDA(cudaMemcpyAsync(J.mats_s.p, J.mats_e.p, sizeof(wpbr_material) * J.nmat, cudaMemcpyDeviceToDevice, st));
  if (J.n_texels) {
    uint32_t EW = ctx->envW, EH = ctx->envH;
    size_t nt = J.n_texels;
    auto cp = [&](float* d, const float* s, size_t cnt) {
      return cudaMemcpyAsync(d, s, sizeof(float) * cnt, cudaMemcpyDeviceToDevice, st);
    };
    WPBR_CUDA(cudaMemcpyAsync(J.rgb_s.p, J.rgb_e.p, sizeof(float4) * nt, cudaMemcpyDeviceToDevice, st));
    WPBR_CUDA(cp(J.s_func.p, J.e_func.p, nt));
    WPBR_CUDA(cp(J.s_cdf.p, J.e_cdf.p, (size_t)EH * (EW + 1)));
    WPBR_CUDA(cp(J.s_int.p, J.e_int.p, EH));
    WPBR_CUDA(cp(J.s_mfunc.p, J.e_mfunc.p, EH));
    WPBR_CUDA(cp(J.s_mcdf.p, J.e_mcdf.p, EH + 1));
    WPBR_CUDA(cp(J.s_mint.p, J.e_mint.p, 1));
    J.Z_s = J.Z_e;
  }
  J.param_gen += 1;
  return WPBR_OK;
}

wpbr_status adjoint_forward(wpbr_ctx* ctx, const float* target, float* image, double* loss, bool device) {
  AdjState& J = ctx->adj;
  if (!J.ready) return set_err(ctx, WPBR_ERR_NOT_BUILT, "adjoint: adjoint_setup not called");
  cudaStream_t st = ctx->stream;
  uint32_t n = J.W * J.H;
  PassCtx P = adj_pass_ctx(ctx);
  AdjView A = adj_view(ctx);
  WPBR_CUDA(cudaMemsetAsync(J.acc.p, 0, sizeof(float4) * n, st));
  wpbr_status s = adj_passes(
      ctx, P, A,
      [&](uint32_t, const AdjBufs& B, cudaStream_t ls) {
        k_adj_eval<<<div_up(n, kTB), kTB, 0, ls>>>(P, A, B.state, B.shadow_hit, B.Lb);
      },
      [&](uint32_t, const AdjBufs& B) { film_tiles_launch(J.W, J.H, B.pf, B.Lb, J.acc.p, st); });
  if (s != WPBR_OK) return s;
  const float* d_target = nullptr;
  if (target) {
    d_target = target;
    if (!device) {
      WPBR_CUDA(cudaMemcpyAsync(J.target.p, target, sizeof(float) * 3 * n, cudaMemcpyHostToDevice, st));
      d_target = J.target.p;
    }
  }
  float* d_image = image ? (device ? image : J.image.p) : nullptr;
  WPBR_CUDA(cudaMemsetAsync(J.g_scalar.p, 0, sizeof(double) * 2, st));
  k_adj_loss<<<div_up(n, 256), 256, 0, st>>>(n, J.acc.p, d_target, J.gpix.p, d_image, J.g_scalar.p);
  WPBR_CUDA(cudaGetLastError());
  if (image && !device)
    WPBR_CUDA(cudaMemcpyAsync(image, J.image.p, sizeof(float) * 3 * n, cudaMemcpyDeviceToHost, st));
  double l = 0.0;
  WPBR_CUDA(cudaMemcpyAsync(&l, J.g_scalar.p, sizeof(double), cudaMemcpyDeviceToHost, st));
  WPBR_CUDA(cudaStreamSynchronize(st));
  if (loss) *loss = target ? l / (3.0 * (double)n) : 0.0;
  J.fwd_gen = target ? J.param_gen : 0;
  return WPBR_OK;
}

wpbr_status adjoint_backward(wpbr_ctx* ctx, float* grad_mat, float* grad_env, bool device) {
  AdjState& J = ctx->adj;
  if (!J.ready) return set_err(ctx, WPBR_ERR_NOT_BUILT, "adjoint: adjoint_setup not called");
  if (J.fwd_gen != J.param_gen)
    return set_err(ctx, WPBR_ERR_NOT_BUILT, "adjoint_backward: no forward pass with a target at these parameters");
  cudaStream_t st = ctx->stream;
  uint32_t n = J.W * J.H;
  PassCtx P = adj_pass_ctx(ctx);
  AdjView A = adj_view(ctx);
  WPBR_CUDA(cudaMemsetAsync(J.g_mat.p, 0, sizeof(double) * 10 * J.nmat, st));
  WPBR_CUDA(cudaMemsetAsync(J.g_scalar.p + 1, 0, sizeof(double), st));
  if (J.n_texels) {
    WPBR_CUDA(cudaMemsetAsync(J.g_env.p, 0, sizeof(float) * 3 * J.n_texels, st));
    WPBR_CUDA(cudaMemsetAsync(J.g_func.p, 0, sizeof(float) * J.n_texels, st));
  }
  AdjGrad G{J.gpix.p, J.g_mat.p, J.g_env.p, J.g_func.p, J.g_scalar.p + 1, J.nmat};
  size_t smem = sizeof(float) * 10 * J.nmat;
  wpbr_status s = adj_passes(
      ctx, P, A,
      [&](uint32_t, const AdjBufs& B, cudaStream_t ls) {
        k_adj_back<<<div_up(n, kTB), kTB, smem, ls>>>(P, A, B.state, B.shadow_hit, B.pf, G);
      },
      [](uint32_t, const AdjBufs&) {});
  if (s != WPBR_OK) return s;
  if (J.n_texels)
    k_adj_env_finish<<<div_up(J.n_texels, 256), 256, 0, st>>>(A.env_e, ctx->quirks, J.g_func.p, J.g_scalar.p + 1,
                                                              J.g_env.p);
  WPBR_CUDA(cudaGetLastError());
  float* d_gm = grad_mat ? (device ? grad_mat : J.mat_prm.p) : nullptr;
  if (d_gm) k_mat_grad_out<<<div_up(10 * J.nmat, 256), 256, 0, st>>>(J.g_mat.p, 10 * J.nmat, d_gm);
  if (grad_mat && !device)
    WPBR_CUDA(cudaMemcpyAsync(grad_mat, J.mat_prm.p, sizeof(float) * 10 * J.nmat, cudaMemcpyDeviceToHost, st));
  if (grad_env && J.n_texels) {
    WPBR_CUDA(cudaMemcpyAsync(grad_env, J.g_env.p, sizeof(float) * 3 * J.n_texels,
                              device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, st));
  }
  WPBR_CUDA(cudaGetLastError());
  WPBR_CUDA(cudaStreamSynchronize(st));
  return WPBR_OK;
}

}  // namespace wpbr

using namespace wpbr;

extern "C" {

WPBR_API wpbr_status wpbr_adjoint_setup(wpbr_ctx* ctx, uint32_t spp, uint32_t seed, uint32_t stream) {
  if (!ctx) return WPBR_ERR_INVALID_ARG;
  return adjoint_setup(ctx, spp, seed, stream);
}

WPBR_API wpbr_status wpbr_adjoint_param_counts(wpbr_ctx* ctx, uint32_t* n_mat_params, uint32_t* n_env_params) {
  if (!ctx) return WPBR_ERR_INVALID_ARG;
  if (!ctx->adj.ready) return set_err(ctx, WPBR_ERR_NOT_BUILT, "adjoint: adjoint_setup not called");
  if (n_mat_params) *n_mat_params = 10 * ctx->adj.nmat;
  if (n_env_params) *n_env_params = (uint32_t)(3 * ctx->adj.n_texels);
  return WPBR_OK;
}

WPBR_API wpbr_status wpbr_adjoint_get_params(wpbr_ctx* ctx, float* mat_params, float* env_params) {
  if (!ctx) return WPBR_ERR_INVALID_ARG;
  return adjoint_get_params(ctx, mat_params, env_params);
}

WPBR_API wpbr_status wpbr_adjoint_set_params(wpbr_ctx* ctx, const float* mat_params, const float* env_params) {
  if (!ctx) return WPBR_ERR_INVALID_ARG;
  return adjoint_set_params(ctx, mat_params, env_params, false);
}

WPBR_API wpbr_status wpbr_adjoint_set_params_device(wpbr_ctx* ctx, const float* d_mat_params,
                                                    const float* d_env_params) {
  if (!ctx) return WPBR_ERR_INVALID_ARG;
  return adjoint_set_params(ctx, d_mat_params, d_env_params, true);
}

WPBR_API wpbr_status wpbr_adjoint_freeze(wpbr_ctx* ctx) {
  if (!ctx) return WPBR_ERR_INVALID_ARG;
  return adjoint_freeze(ctx);
}

WPBR_API wpbr_status wpbr_adjoint_forward(wpbr_ctx* ctx, const float* target, float* image, double* loss) {
  if (!ctx) return WPBR_ERR_INVALID_ARG;
  return adjoint_forward(ctx, target, image, loss, false);
}

WPBR_API wpbr_status wpbr_adjoint_forward_device(wpbr_ctx* ctx, const float* d_target, float* d_image, double* loss) {
  if (!ctx) return WPBR_ERR_INVALID_ARG;
  return adjoint_forward(ctx, d_target, d_image, loss, true);
}

WPBR_API wpbr_status wpbr_adjoint_backward(wpbr_ctx* ctx, float* grad_mat, float* grad_env) {
  if (!ctx) return WPBR_ERR_INVALID_ARG;
  return adjoint_backward(ctx, grad_mat, grad_env, false);
}

WPBR_API wpbr_status wpbr_adjoint_backward_device(wpbr_ctx* ctx, float* d_grad_mat, float* d_grad_env) {
  if (!ctx) return WPBR_ERR_INVALID_ARG;
  return adjoint_backward(ctx, d_grad_mat, d_grad_env, true);
}

}  // extern "C"
