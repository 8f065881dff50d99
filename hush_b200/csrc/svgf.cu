// SVGF baseline (Schied et al. 2017) + TAA resolve: the reference's SVGF class (src/denoise/svgf.js) as CUDA
// kernels over rgba16float device buffers. Kept beside Hush as its fallback and as the judge of its error.
#include <cuda_runtime.h>

#include <cstring>
#include <string>
#include <type_traits>

#include "common.cuh"
#include "hush.h"
#include "hush_device.cuh"
#include "hush_pair.cuh"
#include "quotient.cuh"

using namespace hush;

namespace {

struct SvgfFrame {
  int W, H;
  int reset, use_taa;
  float sigma_l, sigma_n, sigma_z, alpha_color, alpha_moments, taa_alpha;
  const uint2 *rad, *nd, *mv, *mat, *emi, *pnd, *pmv;
  int p_rad, p_nd, p_mv, p_mat, p_emi, p_pnd, p_pmv;
  const uint2 *hist_prev, *mom_prev, *taa_prev;
  uint2 *tmp, *mom, *hist, *taa;
};

HD_INL float hi_half(uint32_t u) { return __half2float(__ushort_as_half((uint16_t)(u >> 16))); }

// The history test of a previous frame's texel (guide q, object id) against this pixel's (svgf.js:31-39).
HD_INL bool svgf_same(float4 q, float qobj, float4 n, float zPrev, float obj) {
  return !(q.w < 0.0f) && qobj == obj && !(fabsf(q.w - zPrev) > 0.05f * zPrev + 0.01f) && !(dot3(q, n) < 0.9f);
}
HD_INL bool svgf_consistent(const SvgfFrame &f, int qx, int qy, float4 n, float zPrev, float obj) {
  if (qx < 0 || qy < 0 || qx >= f.W || qy >= f.H) return false;
  return svgf_same(ldh(f.pnd, qy * f.p_pnd + qx), ldh(f.pmv, qy * f.p_pmv + qx).z, n, zPrev, obj);
}

// TEMPORAL (svgf.js:41-105). Bound: the latency of its dependent loads (motion, then the footprint): the four texels'
// guide, object, colour and moments are loaded together, not test by test (58 -> 53 us at 1920 x 1080). Its quotients round as
// the IEEE ones do: an ulp in the history length flips the variance pass's branch.
__global__ void __launch_bounds__(256) k_svgf_temporal(const SvgfFrame f) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= f.W || y >= f.H) return;
  const int o = y * f.W + x;
  const float4 mv = ldh(f.mv, y * f.p_mv + x);
  const float4 nd = ldh(f.nd, y * f.p_nd + x);
  const float ppx = (float)x + 0.5f + mv.x - 0.5f, ppy = (float)y + 0.5f + mv.y - 0.5f;
  const float flx = floorf(ppx), fly = floorf(ppy);
  const int bx = (int)flx, by = (int)fly;
  const float fx = ppx - flx, fy = ppy - fly;
  // the bilinear footprint's guide, object and history texels (clamped), all in flight before the first test
  const bool noHistory = f.reset != 0;
  uint2 pn[4], ph[4], pm[4];
  uint32_t po[4];
  if (!noHistory) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int qx = clampi(bx + (i & 1), 0, f.W - 1), qy = clampi(by + (i >> 1), 0, f.H - 1);
      pn[i] = __ldg(f.pnd + qy * f.p_pnd + qx);
      po[i] = __ldg(&f.pmv[qy * f.p_pmv + qx].y);
      ph[i] = __ldg(f.hist_prev + qy * f.W + qx);
      pm[i] = __ldg(f.mom_prev + qy * f.W + qx);
    }
  }
  if (nd.w < 0.0f) {
    sth(f.tmp, o, make_float4(0.f, 0.f, 0.f, 0.f));
    sth(f.mom, o, make_float4(0.f, 0.f, 0.f, 0.f));
    return;
  }
  const float4 alb = ldh(f.mat, y * f.p_mat + x);
  const float4 r = ldh(f.rad, y * f.p_rad + x);
  // the history length it blends into decides the spatial / temporal variance branch (m.z >= 4), so the weighted
  // sums are rounded product by product like an unfused shader (no FMA contraction)
  float sumW = 0.f, hcx = 0.f, hcy = 0.f, hcz = 0.f, hm0 = 0.f, hm1 = 0.f, hm2 = 0.f;
  const float wts[4] = {__fmul_rn(1.0f - fx, 1.0f - fy), __fmul_rn(fx, 1.0f - fy), __fmul_rn(1.0f - fx, fy),
                        __fmul_rn(fx, fy)};
  if (!noHistory) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int qx = bx + (i & 1), qy = by + (i >> 1);
      if (qx >= 0 && qy >= 0 && qx < f.W && qy < f.H && wts[i] > 0.0f &&
          svgf_same(h4_to_f4(pn[i]), unpack2(po[i]).x, nd, mv.w, mv.z)) {
        const float4 c = h4_to_f4(ph[i]), m = h4_to_f4(pm[i]);
        sumW += wts[i];
        hcx = __fadd_rn(hcx, __fmul_rn(wts[i], c.x)); hcy = __fadd_rn(hcy, __fmul_rn(wts[i], c.y));
        hcz = __fadd_rn(hcz, __fmul_rn(wts[i], c.z));
        hm0 = __fadd_rn(hm0, __fmul_rn(wts[i], m.x)); hm1 = __fadd_rn(hm1, __fmul_rn(wts[i], m.y));
        hm2 = __fadd_rn(hm2, __fmul_rn(wts[i], m.z));
      }
    }
  }
  if (sumW < 0.01f && !noHistory) {
    const int cx = (int)rintf(ppx), cy = (int)rintf(ppy);  // WGSL round(): ties to even
    for (int dy = -1; dy <= 1; dy++) {
      for (int dx = -1; dx <= 1; dx++) {
        const int qx = cx + dx, qy = cy + dy;
        if (svgf_consistent(f, qx, qy, nd, mv.w, mv.z)) {
          const float4 c = ldh(f.hist_prev, qy * f.W + qx), m = ldh(f.mom_prev, qy * f.W + qx);
          sumW += 1.0f;
          hcx += c.x; hcy += c.y; hcz += c.z;
          hm0 += m.x; hm1 += m.y; hm2 += m.z;
        }
      }
    }
  }
  // (last: the test below would hold the footprint's loads back)
  const float ax = fmaxf(alb.x, 1e-3f), ay = fmaxf(alb.y, 1e-3f), az = fmaxf(alb.z, 1e-3f);
  float ix = quot_rn(r.x, ax, rcp_rn(ax)), iy = quot_rn(r.y, ay, rcp_rn(ay)), iz = quot_rn(r.z, az, rcp_rn(az));
  if (!all_finite(ix + iy + iz)) {
    ix = quot_any(r.x, ax); iy = quot_any(r.y, ay); iz = quot_any(r.z, az);
  }
  const float l = __fadd_rn(__fadd_rn(__fmul_rn(ix, 0.2126f), __fmul_rn(iy, 0.7152f)), __fmul_rn(iz, 0.0722f));
  float len, cx = ix, cy = iy, cz = iz, m0 = l, m1 = __fmul_rn(l, l);
  if (sumW >= 0.01f) {
    hcx /= sumW; hcy /= sumW; hcz /= sumW;
    hm0 /= sumW; hm1 /= sumW; hm2 /= sumW;
    len = fminf(hm2 + 1.0f, 64.0f);
    const float ac = fmaxf(f.alpha_color, 1.0f / len), am = fmaxf(f.alpha_moments, 1.0f / len);
    cx = __fadd_rn(__fmul_rn(hcx, 1.0f - ac), __fmul_rn(ix, ac));
    cy = __fadd_rn(__fmul_rn(hcy, 1.0f - ac), __fmul_rn(iy, ac));
    cz = __fadd_rn(__fmul_rn(hcz, 1.0f - ac), __fmul_rn(iz, ac));
    m0 = __fadd_rn(__fmul_rn(hm0, 1.0f - am), __fmul_rn(m0, am));
    m1 = __fadd_rn(__fmul_rn(hm1, 1.0f - am), __fmul_rn(m1, am));
  } else {
    len = 1.0f;
  }
  sth(f.tmp, o, make_float4(cx, cy, cz, 0.f));
  sth(f.mom, o, make_float4(m0, m1, len, 0.f));
}

// VARIANCE (svgf.js:114-148): temporal where the history is long enough, else from a 7 x 7 neighbourhood. Only a CTA
// with such a pixel (a disocclusion, or the first frames) stages the neighbourhood's texels; outside the image they are
// marked as sky. Taps, weights and sums are the reference's in its order (exp and pow with their full accuracy, quotients rounded
// as IEEE ones); the tap distances and a row's divisors are formed once. Bound: the 49 pow of such a pixel. 1920 x 1080
// 39 -> 32 us, 641 x 363 22.7 -> 15.7 us with the set-up beside the pass before (a sequence of eight frames, two of them
// without a long enough history).
constexpr int VT_W = 32, VT_H = 8, VT_NT = VT_W * VT_H;
// sqrt(i^2 + j^2), correctly rounded
__constant__ const float VT_DIST[4][4] = {{0.0f, 1.0f, 2.0f, 3.0f},
                                          {1.0f, 1.41421356237f, 2.2360679775f, 3.16227766017f},
                                          {2.0f, 2.2360679775f, 2.82842712475f, 3.60555127546f},
                                          {3.0f, 3.16227766017f, 3.60555127546f, 4.24264068712f}};
__global__ void __launch_bounds__(VT_NT) k_svgf_variance(const SvgfFrame f, uint2 *out) {
  pass_begin();
  constexpr int TC = VT_W + 6, TR = VT_H + 6, N = TC * TR;
  __shared__ uint2 sN[N], sC[N], sM[N];
  const int li = threadIdx.x, tx = li % VT_W, ty = li / VT_W;
  const int bx = blockIdx.x * VT_W, by = blockIdx.y * VT_H, x = bx + tx, y = by + ty;
  const bool in_img = x < f.W && y < f.H;
  const int o = y * f.W + x;
  float4 nd = make_float4(0.f, 0.f, 0.f, -1.0f), c = make_float4(0.f, 0.f, 0.f, 0.f), m = c;
  if (in_img) {
    nd = ldh(f.nd, y * f.p_nd + x);
    c = ldh_pass(f.tmp, o);
    m = ldh_pass(f.mom, o);
  }
  const bool sky = nd.w < 0.0f, spatial = !sky && !(m.z >= 4.0f);
  if (!__syncthreads_or(spatial ? 1 : 0)) {
    if (in_img)
      sth(out, o, sky ? make_float4(0.f, 0.f, 0.f, 0.f) : make_float4(c.x, c.y, c.z, fmaxf(0.0f, m.y - m.x * m.x)));
    return;
  }
  for (int i = li; i < N; i += VT_NT) {
    const int gx = bx - 3 + i % TC, gy = by - 3 + i / TC;
    if (gx >= 0 && gy >= 0 && gx < f.W && gy < f.H) {
      cp_async8(sN + i, f.nd + gy * f.p_nd + gx);
      cp_async8(sC + i, f.tmp + gy * f.W + gx);
      cp_async8(sM + i, f.mom + gy * f.W + gx);
    } else {
      sN[i] = make_uint2(0u, 0xbc000000u);  // depth -1: sky
    }
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  if (!in_img) return;
  if (!spatial) {
    sth(out, o, sky ? make_float4(0.f, 0.f, 0.f, 0.f) : make_float4(c.x, c.y, c.z, fmaxf(0.0f, m.y - m.x * m.x)));
    return;
  }
  float sw = 0.f, scx = 0.f, scy = 0.f, scz = 0.f, sm0 = 0.f, sm1 = 0.f;
  const int t = (ty + 3) * TC + tx + 3;
#pragma unroll 1
  for (int dy = -3; dy <= 3; dy++) {
    float den[4], rcp[4];  // of a row's depth weights, by |dx|
#pragma unroll
    for (int i = 0; i < 4; i++) {
      den[i] = 0.02f * nd.w * VT_DIST[dy < 0 ? -dy : dy][i] + 1e-3f;
      rcp[i] = rcp_rn(den[i]);
    }
#pragma unroll
    for (int dx = -3; dx <= 3; dx++) {
      const int q = t + dy * TC + dx, i = dx < 0 ? -dx : dx;
      const float4 ndq = h4_to_f4(sN[q]);
      if (ndq.w < 0.0f) continue;
      const float dz = -fabsf(ndq.w - nd.w);
      float x = quot_rn(dz, den[i], rcp[i]);
      if (!all_finite(x)) x = quot_any(dz, den[i]);
      const float wz = expf(x);
      const float wn = powf(fmaxf(0.0f, dot3(ndq, nd)), f.sigma_n);
      const float w = wz * wn;
      const float4 cq = h4_to_f4(sC[q]);
      const float2 mq = unpack2(sM[q].x);
      sw += w;
      scx += w * cq.x; scy += w * cq.y; scz += w * cq.z;
      sm0 += w * mq.x; sm1 += w * mq.y;
    }
  }
  const float d = fmaxf(sw, 1e-6f);
  scx /= d; scy /= d; scz /= d; sm0 /= d; sm1 /= d;
  const float v = fmaxf(0.0f, sm1 - sm0 * sm0) * 4.0f / fmaxf(m.z, 1.0f);
  sth(out, o, make_float4(scx, scy, scz, v));
}

// ATROUS iteration (svgf.js:157-216), step 1 << iter; iteration 0 also writes the colour history.
//
// A CTA filters 64 columns x 8 rows, the rows STEP apart (one row phase of the iteration's lattice), so its staged
// footprint is (64 + 4 STEP) x 12 texels for every STEP: rows between two lattice rows are not loaded. A thread filters
// four pixels: columns x and x + 32 in the two lanes of packed FP32x2 arithmetic, times two neighbouring lattice rows,
// which share 20 of their 25 taps. The footprint is held in shared memory as the pairs of texels 32 columns apart, each
// converted to FP32 once, so that every tap of every STEP, 1 included, is a pair without a shuffle; texels outside
// the image are marked as sky (depth -1, colour 0), so no tap tests its position. The tap rows run as a loop over the rows that
// both pixels share, between one row of the upper and one of the lower alone (a row's depth factors come from shared memory):
// all unrolled, instruction fetch stalled the warps; with a test per pixel and row in one loop the pass took 8 % longer. A
// pixel's taps are summed in the order of their rows and every quotient is rounded as the IEEE one, so the frame is the one of a
// thread per pixel bit for bit (column by column, with quotients by a product, iterations 0-4 took 71 / 69 / 76 / 78 / 82 us).
// Bound: the FP32 pipe (the ~25 FP32 operations of a tap and pixel; packing saves issue slots, not pipe time). A float4 tile
// with a thread per pixel read 36 bytes a tap for one pixel, and steps 8 and 16 loaded every tap from global memory: iterations
// 0-4 at 1920 x 1080 were 93 / 96 / 99 / 125 / 125 us and are 81 / 72 / 81 / 85 / 86 us with the set-up beside the pass before.
constexpr int AT_P = 32, AT_W = 2 * AT_P, AT_H = 8, AT_NT = AT_P * AT_H / 2;

HD_INL float2 neg_abs2(float2 a) {
  return f2(__uint_as_float(__float_as_uint(a.x) | 0x80000000u), __uint_as_float(__float_as_uint(a.y) | 0x80000000u));
}
// The normal weight pow(max(n . n_q, 0), sigma_n): by seven squarings for the default sigma_n = 128 (no special-function
// unit), else as the hardware exp2(sigma_n log2 x); pow(x, 0) = 1.
template <bool N128>
HD_INL float2 svgf_wn2(float2 x, float sigma_n) {
  if constexpr (N128) {
#pragma unroll
    for (int i = 0; i < 7; i++) x = mul2(x, x);
    return x;
  } else {
    return sigma_n != 0.0f ? f2(__powf(x.x, sigma_n), __powf(x.y, sigma_n)) : f2(1.0f, 1.0f);
  }
}
// A texel pair of the footprint: (nx, nx', ny, ny'), (nz, nz', z, z'), (r, r', g, g'), (b, b', v, v').
struct TexelPair {
  float4 g0, g1, c0, c1;
};
HD_INL TexelPair widen(uint2 na, uint2 nb, uint2 ca, uint2 cb) {
  const float4 n0 = h4_to_f4(na), n1 = h4_to_f4(nb), c0 = h4_to_f4(ca), c1 = h4_to_f4(cb);
  return TexelPair{make_float4(n0.x, n1.x, n0.y, n1.y), make_float4(n0.z, n1.z, n0.w, n1.w),
                   make_float4(c0.x, c1.x, c0.y, c1.y), make_float4(c0.z, c1.z, c0.w, c1.w)};
}
HD_INL float2 lum2(const TexelPair &p) {
  return fma2(lo2(p.c1), bc2(0.0722f), fma2(lo2(p.c0), bc2(0.2126f), mul2(hi2(p.c0), bc2(0.7152f))));
}
// RAW: the pairs as stored (converted by each tap), 32 bytes instead of 64. Only STEP = 16 takes it, whose 96 x 12
// pairs would leave two CTAs an SM.
template <int STEP>
struct AtrousSmem {
  static constexpr bool RAW = STEP >= 16;
  static constexpr int A = 2 * STEP, TC = AT_P + 2 * A, TR = AT_H + 4, N = TR * TC;
  uint4 t[RAW ? 2 : 4][N];
  float2 izd[2][5][AT_NT];  // 1 / (sigma_z zg dist + 1e-3) per tap distance 1, sqrt 2, 2, sqrt 5, sqrt 8
  HD_INL void put(int i, uint2 na, uint2 nb, uint2 ca, uint2 cb) {
    if constexpr (RAW) {
      t[0][i] = make_uint4(na.x, na.y, nb.x, nb.y);
      t[1][i] = make_uint4(ca.x, ca.y, cb.x, cb.y);
    } else {
      const TexelPair p = widen(na, nb, ca, cb);
      *reinterpret_cast<float4 *>(&t[0][i]) = p.g0;
      *reinterpret_cast<float4 *>(&t[1][i]) = p.g1;
      *reinterpret_cast<float4 *>(&t[2][i]) = p.c0;
      *reinterpret_cast<float4 *>(&t[3][i]) = p.c1;
    }
  }
  HD_INL static TexelPair get(const uint4 *p) {  // p = &t[0][i]
    if constexpr (RAW) {
      const uint4 n = p[0], c = p[N];
      return widen(make_uint2(n.x, n.y), make_uint2(n.z, n.w), make_uint2(c.x, c.y), make_uint2(c.z, c.w));
    } else {
      const float4 *q = reinterpret_cast<const float4 *>(p);
      return TexelPair{q[0], q[N], q[2 * N], q[3 * N]};
    }
  }
  HD_INL float depth(int i, int lane) const {
    if constexpr (RAW) return hi_half((&t[0][i].y)[2 * lane]);
    else return __uint_as_float((&t[1][i].z)[lane]);
  }
  HD_INL float variance(int i, int lane) const {
    if constexpr (RAW) return hi_half((&t[1][i].y)[2 * lane]);
    else return __uint_as_float((&t[3][i].z)[lane]);
  }
};

template <int STEP, bool N128>
__global__ void __launch_bounds__(AT_NT, 5) k_svgf_atrous(const SvgfFrame f, const uint2 *in, uint2 *out, int iter) {
  pass_begin();
  using Smem = AtrousSmem<STEP>;
  constexpr int A = Smem::A, TC = Smem::TC;
  extern __shared__ __align__(16) unsigned char at_smem[];
  Smem &S = *reinterpret_cast<Smem *>(at_smem);
  const int li = threadIdx.x;
  const int bx = blockIdx.x * AT_W, phase = blockIdx.y, j0 = blockIdx.z * AT_H;
  const int tx = li % AT_P, jr = (li / AT_P) * 2;  // the thread's first lattice row in the tile
  const int x0 = bx + tx, y0 = (j0 + jr) * STEP + phase;
  // The centre's 3 x 3 variance blur and depth gradient read the rows y +- 1, which only STEP = 1 stages; the other
  // steps load them here (texels clamped to the image).
  float vu[2][2], vd[2][2][3], zu[2][2], zd[2][2];
  if constexpr (STEP > 1) {
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int y = min(y0 + k * STEP, f.H - 1);
      const uint2 *im = in + max(y - 1, 0) * f.W, *ip = in + min(y + 1, f.H - 1) * f.W;
      const uint2 *nm = f.nd + max(y - 1, 0) * f.p_nd, *np = f.nd + min(y + 1, f.H - 1) * f.p_nd;
#pragma unroll
      for (int l = 0; l < 2; l++) {
        const int xc = min(x0 + l * AT_P, f.W - 1), xm = max(xc - 1, 0), xp = min(xc + 1, f.W - 1);
        auto var = [](const uint2 *p) { return hi_half(ld_pass(&p->y)); };
        vu[k][l] = 0.0625f * var(im + xm) + 0.125f * var(im + xc) + 0.0625f * var(im + xp);
        vd[k][l][0] = var(ip + xm); vd[k][l][1] = var(ip + xc); vd[k][l][2] = var(ip + xp);
        zu[k][l] = hi_half(__ldg(&nm[xc].y));
        zd[k][l] = hi_half(__ldg(&np[xc].y));
      }
    }
  }
  // one warp a row of the footprint at a time
  for (int r = li / 32; r < Smem::TR; r += AT_NT / 32) {
    const int gy = (j0 - 2 + r) * STEP + phase, gx0 = bx - A + li % 32;
    const bool iy = gy >= 0 && gy < f.H;
    const uint2 *pn = f.nd + (gy * f.p_nd + gx0), *pc = in + (gy * f.W + gx0);
#pragma unroll
    for (int u = 0; u < TC; u += 32) {
      if (u + 32 > TC && u + li % 32 >= TC) break;
      const bool o0 = iy && gx0 + u >= 0 && gx0 + u < f.W, o1 = iy && gx0 + u + AT_P >= 0 && gx0 + u + AT_P < f.W;
      uint2 n[2] = {make_uint2(0u, 0xbc000000u), make_uint2(0u, 0xbc000000u)}, c[2] = {};  // depth -1: sky
      if (o0) { n[0] = __ldg(pn + u); c[0] = ld_pass(pc + u); }
      if (o1) { n[1] = __ldg(pn + u + AT_P); c[1] = ld_pass(pc + u + AT_P); }
      S.put(r * TC + u + li % 32, n[0], n[1], c[0], c[1]);
    }
  }
  __syncthreads();
  if (y0 >= f.H || x0 >= f.W) return;
  struct Centre {
    float2 nx, ny, nz, z, lp, il, sw, sr, sg, sb, sv;
  } C[2];
  const int base = (jr + 2) * TC + tx + A;  // tile entry of the first row
  constexpr float h0 = 3.0f / 8.0f, h1 = 1.0f / 4.0f, h2 = 1.0f / 16.0f;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int t = base + k * TC;
    const TexelPair p = Smem::get(&S.t[0][t]);
    Centre &c = C[k];
    c.nx = lo2(p.g0); c.ny = hi2(p.g0); c.nz = lo2(p.g1); c.z = hi2(p.g1);
    c.lp = lum2(p);
    float den[6][2];  // of the luminance weight, then of the depth weight by tap distance
    const int y = min(y0 + k * STEP, f.H - 1);
#pragma unroll
    for (int l = 0; l < 2; l++) {
      const int x = min(x0 + l * AT_P, f.W - 1);
      const int tl = x > 0 ? t - 1 : t, tr = x + 1 < f.W ? t + 1 : t;
      const float z = S.depth(t, l), zl = S.depth(tl, l), zr = S.depth(tr, l);
      // the blur's sums in the order of its rows
      float up, dn, gv, v0, v1, v2;
      if constexpr (STEP > 1) {
        gv = vu[k][l];
        v0 = vd[k][l][0]; v1 = vd[k][l][1]; v2 = vd[k][l][2];
        up = zu[k][l];
        dn = zd[k][l];
      } else {
        const int du = y > 0 ? -TC : 0, dd = y + 1 < f.H ? TC : 0;
        gv = 0.0625f * S.variance(tl + du, l) + 0.125f * S.variance(t + du, l) + 0.0625f * S.variance(tr + du, l);
        v0 = S.variance(tl + dd, l); v1 = S.variance(t + dd, l); v2 = S.variance(tr + dd, l);
        up = S.depth(t + du, l);
        dn = S.depth(t + dd, l);
      }
      gv = gv + 0.125f * S.variance(tl, l) + 0.25f * S.variance(t, l) + 0.125f * S.variance(tr, l);
      gv = gv + 0.0625f * v0 + 0.125f * v1 + 0.0625f * v2;
      const float gx = fminf(zr > 0.0f ? fabsf(zr - z) : 1e9f, zl > 0.0f ? fabsf(zl - z) : 1e9f);
      const float gy = fminf(dn > 0.0f ? fabsf(dn - z) : 1e9f, up > 0.0f ? fabsf(up - z) : 1e9f);
      const float zg = f.sigma_z * fminf(fmaxf(gx, gy), z);
      den[5][l] = f.sigma_l * sqrt_rn(fmaxf(gv, 0.0f)) + 1e-6f;
      const float dcls[5] = {1.0f, 1.41421356237f, 2.0f, 2.2360679775f, 2.82842712475f};
#pragma unroll
      for (int d = 0; d < 5; d++) den[d][l] = zg * (dcls[d] * (float)STEP) + 1e-3f;
    }
    float2 rcp[6], sum = f2(0.0f, 0.0f);
#pragma unroll
    for (int d = 0; d < 6; d++) {
      rcp[d] = f2(rcp_rn(den[d][0]), rcp_rn(den[d][1]));
      sum = add2(sum, rcp[d]);
    }
    if (!all_finite(sum.x + sum.y)) {
#pragma unroll
      for (int d = 0; d < 6; d++) rcp[d] = f2(quot_any(1.0f, den[d][0]), quot_any(1.0f, den[d][1]));
    }
    c.il = rcp[5];
#pragma unroll
    for (int d = 0; d < 5; d++) S.izd[k][d][li] = rcp[d];  // read back by this thread alone
    c.sw = f2(h0 * h0, h0 * h0);
    c.sr = mul2(lo2(p.c0), c.sw); c.sg = mul2(hi2(p.c0), c.sw); c.sb = mul2(lo2(p.c1), c.sw);
    c.sv = mul2(mul2(hi2(p.c1), c.sw), c.sw);
  }
  // One row of taps at a time: its five texel pairs serve both rows' filters.
  const uint4 *row = &S.t[0][base - 2 * TC];
  auto taps = [&](int r, auto first, auto last) {  // for the pixels first .. last
    float2 hh[2][3], iz[2][3];  // by row and |dx|
#pragma unroll
    for (int k = first; k <= last; k++) {
      const int b = r < k ? k - r : r - k;
      const float hy = b == 0 ? h0 : (b == 1 ? h1 : h2);
      const int cls[3] = {b == 2 ? 2 : 0, b == 0 ? 0 : (b == 1 ? 1 : 3), b == 0 ? 2 : (b == 1 ? 3 : 4)};
      hh[k][0] = bc2(h0 * hy); hh[k][1] = bc2(h1 * hy); hh[k][2] = bc2(h2 * hy);
#pragma unroll
      for (int a = 0; a < 3; a++) iz[k][a] = S.izd[k][cls[a]][li];
    }
#pragma unroll
    for (int dx = -2; dx <= 2; dx++) {
      const TexelPair q = Smem::get(row + dx * STEP);
      const float2 z = hi2(q.g1), lq = lum2(q);
      const bool ok0 = !(z.x < 0.0f), ok1 = !(z.y < 0.0f);
#pragma unroll
      for (int k = first; k <= last; k++) {
        const int a = dx < 0 ? -dx : dx;
        if (dx == 0 && r == k) continue;
        Centre &c = C[k];
        const float2 dot = fma2(lo2(q.g1), c.nz, fma2(hi2(q.g0), c.ny, mul2(lo2(q.g0), c.nx)));
        const float2 wn = svgf_wn2<N128>(f2(fmaxf(0.0f, dot.x), fmaxf(0.0f, dot.y)), f.sigma_n);
        const float2 dz = sub2(z, c.z), dl = sub2(lq, c.lp);
        const float2 e = mul2(fma2(neg_abs2(dz), iz[k][a], mul2(neg_abs2(dl), c.il)), bc2(LOG2E));
        float2 w = mul2(mul2(hh[k][a], wn), f2(ex2_approx(e.x), ex2_approx(e.y)));
        w = f2(ok0 ? w.x : 0.0f, ok1 ? w.y : 0.0f);
        c.sw = add2(c.sw, w);
        c.sr = fma2(w, lo2(q.c0), c.sr);
        c.sg = fma2(w, hi2(q.c0), c.sg);
        c.sb = fma2(w, lo2(q.c1), c.sb);
        c.sv = fma2(mul2(w, w), hi2(q.c1), c.sv);
      }
    }
  };
  const std::integral_constant<int, 0> k0;
  const std::integral_constant<int, 1> k1;
  taps(-2, k0, k0);
#pragma unroll 1
  for (int r = -1; r <= 2; r++) {
    row += TC;
    taps(r, k0, k1);
  }
  row += TC;
  taps(3, k1, k1);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int y = y0 + k * STEP;
    if (y >= f.H) break;
    const Centre &c = C[k];
#pragma unroll
    for (int l = 0; l < 2; l++) {
      const int x = x0 + l * AT_P;
      if (x >= f.W) break;
      const float sw = l ? c.sw.y : c.sw.x, sw2 = sw * sw, sr = l ? c.sr.y : c.sr.x, sg = l ? c.sg.y : c.sg.x,
                  sb = l ? c.sb.y : c.sb.x, sv = l ? c.sv.y : c.sv.x, rw = rcp_rn(sw);
      float4 o = make_float4(quot_rn(sr, sw, rw), quot_rn(sg, sw, rw), quot_rn(sb, sw, rw), quot_rn(sv, sw2, rcp_rn(sw2)));
      if (!all_finite(o.x + o.y + o.z + o.w))
        o = make_float4(quot_any(sr, sw), quot_any(sg, sw), quot_any(sb, sw), quot_any(sv, sw2));
      if ((l ? c.z.y : c.z.x) < 0.0f) o = make_float4(0.f, 0.f, 0.f, 0.f);
      sth(out, y * f.W + x, o);
      if (iter == 0) sth(f.hist, y * f.W + x, make_float4(o.x, o.y, o.z, 0.f));
    }
  }
}

template <int STEP, bool N128>
cudaError_t launch_atrous_n(const SvgfFrame &f, const uint2 *in, uint2 *out, int iter, cudaStream_t st) {
  constexpr int smem = (int)sizeof(AtrousSmem<STEP>);
  if constexpr (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k_svgf_atrous<STEP, N128>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
  }
  // phases and their tiles in two dimensions: their product may be more than a grid's 65535 where no other pass's rows are
  const dim3 grid((f.W + AT_W - 1) / AT_W, STEP, (f.H + AT_H * STEP - 1) / (AT_H * STEP));
  return launch_chained(k_svgf_atrous<STEP, N128>, grid, dim3(AT_NT), smem, false, st, f, in, out, iter);
}
template <int STEP>
cudaError_t launch_atrous(const SvgfFrame &f, const uint2 *in, uint2 *out, int iter, cudaStream_t st) {
  return f.sigma_n == 128.0f ? launch_atrous_n<STEP, true>(f, in, out, iter, st)
                             : launch_atrous_n<STEP, false>(f, in, out, iter, st);
}

// RESOLVE (svgf.js:241-270). The reference samples the history through a hardware bilinear sampler
// (clamp-to-edge); here the same texel footprint is weighted exactly in f32.
HD_INL float3 svgf_remod(const SvgfFrame &f, const uint2 *il, int qx, int qy) {
  const int cx = clampi(qx, 0, f.W - 1), cy = clampi(qy, 0, f.H - 1);
  const float4 a = ldh_pass(il, cy * f.W + cx), m = ldh(f.mat, cy * f.p_mat + cx), e = ldh(f.emi, cy * f.p_emi + cx);
  return make_float3(a.x * m.x + e.x, a.y * m.y + e.y, a.z * m.z + e.z);
}

// A 32 x 8 tile with an apron of one: each texel is remodulated, tone-mapped and converted to YCoCg once (a thread per
// pixel did that for its nine neighbours, 27 texel loads and 27 divisions a pixel: 90 us at 1920 x 1080 where the tile
// takes 53 with its set-up beside the pass before, 65 with the IEEE operators' branches). The motion and the history's bilinear
// footprint are loaded before the tile barrier.
// The luminance's two roundings and the blend's are written out: the compiler's choice of FMAs depends on the code around it.
HD_INL float lum_grb(float3 c) { return __fmaf_rn(c.z, 0.0722f, __fmaf_rn(c.x, 0.2126f, __fmul_rn(c.y, 0.7152f))); }
HD_INL float lum_rgb(float3 c) { return __fmaf_rn(c.z, 0.0722f, __fmaf_rn(c.y, 0.7152f, __fmul_rn(c.x, 0.2126f))); }
HD_INL float3 svgf_tm(float3 c) { return div3(c, 1.0f + lum_grb(c)); }
HD_INL float3 svgf_itm(float3 c) { return div3(c, fmaxf(1.0f - lum_grb(c), 1e-4f)); }
constexpr int RT_W = 32, RT_H = 8, RT_NT = RT_W * RT_H;
__global__ void __launch_bounds__(RT_NT) k_svgf_resolve(const SvgfFrame f, const uint2 *il) {
  pass_begin(true);
  constexpr int SW = RT_W + 2, SH = RT_H + 2, N = SW * SH;
  __shared__ float sRgb[3][N], sY[3][N];
  const int li = threadIdx.x, tx = li % RT_W, ty = li / RT_W;
  const int x = blockIdx.x * RT_W + tx, y = blockIdx.y * RT_H + ty;
  const bool in_img = x < f.W && y < f.H;
  if (!f.use_taa) {
    if (!in_img) return;
    const float3 r = svgf_itm(svgf_tm(svgf_remod(f, il, x, y)));
    sth(f.taa, y * f.W + x, make_float4(r.x, r.y, r.z, 1.0f));
    return;
  }
  const int cx = min(x, f.W - 1), cy = min(y, f.H - 1);
  const float4 mv = ldh(f.mv, cy * f.p_mv + cx);
  // (a motion that is not finite gives a position that is not, outside the image either way)
  const float wf = (float)f.W, hf = (float)f.H;
  const float uvx = quot_rn((float)x + 0.5f + mv.x, wf, rcp_rn(wf)), uvy = quot_rn((float)y + 0.5f + mv.y, hf, rcp_rn(hf));
  const bool hist_in = uvx >= 0.0f && uvy >= 0.0f && uvx <= 1.0f && uvy <= 1.0f && !f.reset;
  const float ppx = uvx * (float)f.W - 0.5f, ppy = uvy * (float)f.H - 0.5f;
  const float bxf = floorf(ppx), byf = floorf(ppy);
  uint2 hq[4] = {};
  if (hist_in) {
#pragma unroll
    for (int j = 0; j < 4; j++)
      hq[j] = __ldg(f.taa_prev + clampi((int)byf + (j >> 1), 0, f.H - 1) * f.W + clampi((int)bxf + (j & 1), 0, f.W - 1));
  }
  const int ox = blockIdx.x * RT_W - 1, oy = blockIdx.y * RT_H - 1;
  constexpr int NU = (N + RT_NT - 1) / RT_NT;
  float3 tl[NU];
#pragma unroll
  for (int u = 0; u < NU; u++) {
    const int i = min(li + u * RT_NT, N - 1);
    tl[u] = svgf_remod(f, il, ox + i % SW, oy + i / SW);
  }
#pragma unroll
  for (int u = 0; u < NU; u++) {
    const int i = li + u * RT_NT;
    if (i >= N) break;
    const float3 c = svgf_tm(tl[u]), q = to_ycocg(c);
    sRgb[0][i] = c.x; sRgb[1][i] = c.y; sRgb[2][i] = c.z;
    sY[0][i] = q.x; sY[1][i] = q.y; sY[2][i] = q.z;
  }
  __syncthreads();
  if (!in_img) return;
  const int t = (ty + 1) * SW + tx + 1;
  const float3 cur = make_float3(sRgb[0][t], sRgb[1][t], sRgb[2][t]);
  // E[c^2] - E[c]^2 cancels catastrophically when the neighbourhood is flat: its products are rounded separately
  // (no FMA contraction), as an unfused f32 shader computes them
  float3 m1 = make_float3(0.f, 0.f, 0.f), m2 = m1;
#pragma unroll
  for (int j = 0; j < 9; j++) {
    const int q = t + (j / 3 - 1) * SW + j % 3 - 1;
    const float3 c = make_float3(sY[0][q], sY[1][q], sY[2][q]);
    m1.x += c.x; m1.y += c.y; m1.z += c.z;
    m2.x = __fadd_rn(m2.x, __fmul_rn(c.x, c.x));
    m2.y = __fadd_rn(m2.y, __fmul_rn(c.y, c.y));
    m2.z = __fadd_rn(m2.z, __fmul_rn(c.z, c.z));
  }
  m1 = div3(m1, 9.0f);
  m2 = div3(m2, 9.0f);
  const float sdx = sqrt_rn(fmaxf(__fsub_rn(m2.x, __fmul_rn(m1.x, m1.x)), 0.0f)),
              sdy = sqrt_rn(fmaxf(__fsub_rn(m2.y, __fmul_rn(m1.y, m1.y)), 0.0f)),
              sdz = sqrt_rn(fmaxf(__fsub_rn(m2.z, __fmul_rn(m1.z, m1.z)), 0.0f));
  const float a = f.taa_alpha;
  float3 res = cur;
  if (hist_in) {
    const float fx = ppx - bxf, fy = ppy - byf;
    float3 hist = make_float3(0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float wb = ((j & 1) == 1 ? fx : 1.0f - fx) * ((j >> 1) == 1 ? fy : 1.0f - fy);
      const float4 h = h4_to_f4(hq[j]);
      hist.x += wb * h.x; hist.y += wb * h.y; hist.z += wb * h.z;
    }
    float3 hh = to_ycocg(div3(hist, 1.0f + lum_rgb(hist)));
    hh.x = fminf(fmaxf(hh.x, m1.x - 1.25f * sdx), m1.x + 1.25f * sdx);
    hh.y = fminf(fmaxf(hh.y, m1.y - 1.25f * sdy), m1.y + 1.25f * sdy);
    hh.z = fminf(fmaxf(hh.z, m1.z - 1.25f * sdz), m1.z + 1.25f * sdz);
    const float3 h = from_ycocg(hh);
    const float b = 1.0f - a;
    res = make_float3(__fmaf_rn(cur.x, a, __fmul_rn(h.x, b)), __fmaf_rn(cur.y, a, __fmul_rn(h.y, b)),
                      __fmaf_rn(cur.z, a, __fmul_rn(h.z, b)));
  }
  const float3 r = svgf_itm(res);
  sth(f.taa, y * f.W + x, make_float4(r.x, r.y, r.z, 1.0f));
}

thread_local std::string g_svgf_err;

}  // namespace

struct svgf_s {
  int dev = 0, W = 0, H = 0, frame = 0;
  bool reset = true;
  svgf_options o;
  char *pool = nullptr;
  uint2 *hist[2] = {}, *mom[2] = {}, *tmp = nullptr, *atrous[2] = {}, *taa[2] = {};
  const void *last_out = nullptr;
  std::string last_error;
};

static int svgf_fail(svgf_t *s, int code, const std::string &m) {
  if (s) s->last_error = m;
  g_svgf_err = m;
  return code;
}

extern "C" svgf_options svgf_options_default(void) {
  svgf_options o;
  o.iterations = 5;
  o.sigma_l = 4.0f; o.sigma_n = 128.0f; o.sigma_z = 1.0f;
  o.alpha_color = 0.2f; o.alpha_moments = 0.2f; o.taa_alpha = 0.1f;
  o.taa = 1;
  return o;
}

static int svgf_alloc(svgf_t *s, int W, int H) {
  const size_t img = ((size_t)W * H * 8 + 255) & ~(size_t)255;
  char *p = nullptr;
  cudaError_t e = cudaMalloc(&p, img * 9);
  if (e != cudaSuccess) return svgf_fail(s, HUSH_ERR_CUDA, std::string("SVGF: cudaMalloc: ") + cudaGetErrorString(e));
  cudaMemset(p, 0, img * 9);
  if (s->pool) cudaFree(s->pool);
  s->pool = p;
  uint2 **slots[9] = {&s->hist[0], &s->hist[1], &s->mom[0], &s->mom[1], &s->tmp,
                      &s->atrous[0], &s->atrous[1], &s->taa[0], &s->taa[1]};
  for (int i = 0; i < 9; i++) *slots[i] = (uint2 *)(p + img * i);
  s->W = W; s->H = H; s->frame = 0; s->reset = true; s->last_out = nullptr;
  return HUSH_OK;
}

extern "C" int svgf_create(int width, int height, const svgf_options *opts, int device, svgf_t **out) {
  if (!out) return svgf_fail(nullptr, HUSH_ERR_ARG, "svgf_create: out is NULL");
  *out = nullptr;
  if (!(width > 0 && height > 0))
    return svgf_fail(nullptr, HUSH_ERR_ARG, "SVGF: bad size " + std::to_string(width) + "x" + std::to_string(height));
  svgf_options o = opts ? *opts : svgf_options_default();
  if (o.iterations < 1 || o.iterations > 5)
    return svgf_fail(nullptr, HUSH_ERR_ARG, "SVGF: iterations must be 1..5 (got " + std::to_string(o.iterations) + ")");
  int dev = device;
  if (dev < 0 && cudaGetDevice(&dev) != cudaSuccess) return svgf_fail(nullptr, HUSH_ERR_CUDA, "SVGF: cudaGetDevice");
  if (cudaSetDevice(dev) != cudaSuccess) return svgf_fail(nullptr, HUSH_ERR_CUDA, "SVGF: cudaSetDevice");
  svgf_t *s = new svgf_t();
  s->dev = dev;
  s->o = o;
  int rc = svgf_alloc(s, width, height);
  if (rc != HUSH_OK) { delete s; return rc; }
  *out = s;
  return HUSH_OK;
}

extern "C" void svgf_destroy(svgf_t *s) {
  if (!s) return;
  cudaSetDevice(s->dev);
  if (s->pool) cudaFree(s->pool);
  delete s;
}

extern "C" int svgf_resize(svgf_t *s, int w, int h) {
  if (!s) return svgf_fail(nullptr, HUSH_ERR_ARG, "svgf_resize: NULL instance");
  if (!(w > 0 && h > 0)) return svgf_fail(s, HUSH_ERR_ARG, "SVGF: bad size " + std::to_string(w) + "x" + std::to_string(h));
  if (w == s->W && h == s->H) return HUSH_OK;
  cudaSetDevice(s->dev);
  return svgf_alloc(s, w, h);
}

extern "C" int svgf_reset(svgf_t *s) {
  if (!s) return svgf_fail(nullptr, HUSH_ERR_ARG, "svgf_reset: NULL instance");
  s->reset = true;
  return HUSH_OK;
}

static const char *SVGF_NAMES[7] = {"radiance", "normalDepth", "motion", "material", "emission", "prevNormalDepth",
                                    "prevMotion"};

extern "C" int svgf_encode(svgf_t *s, const svgf_inputs *in, void *stream, const void **out) {
  if (!s) return svgf_fail(nullptr, HUSH_ERR_ARG, "svgf_encode: NULL instance");
  if (!in) return svgf_fail(s, HUSH_ERR_ARG, "SVGF.encode: missing inputs");
  const void *p[7] = {in->radiance, in->normal_depth, in->motion, in->material, in->emission,
                      in->prev_normal_depth, in->prev_motion};
  int pt[7];
  for (int k = 0; k < 7; k++) {
    if (!p[k]) return svgf_fail(s, HUSH_ERR_ARG, std::string("SVGF.encode: missing input '") + SVGF_NAMES[k] + "'");
    if (in->pitch[k] && (in->pitch[k] % 8 || in->pitch[k] < (size_t)s->W * 8))
      return svgf_fail(s, HUSH_ERR_ARG, std::string("SVGF.encode: bad pitch for '") + SVGF_NAMES[k] + "'");
    pt[k] = in->pitch[k] ? (int)(in->pitch[k] / 8) : s->W;
  }
  cudaSetDevice(s->dev);
  cudaStream_t st = (cudaStream_t)stream;
  const int cur = s->frame & 1, prev = cur ^ 1;
  SvgfFrame f;
  std::memset(&f, 0, sizeof(f));
  f.W = s->W; f.H = s->H;
  f.reset = s->reset ? 1 : 0;
  f.use_taa = s->o.taa ? 1 : 0;
  f.sigma_l = s->o.sigma_l; f.sigma_n = s->o.sigma_n; f.sigma_z = s->o.sigma_z;
  f.alpha_color = s->o.alpha_color; f.alpha_moments = s->o.alpha_moments; f.taa_alpha = s->o.taa_alpha;
  f.rad = (const uint2 *)p[0]; f.nd = (const uint2 *)p[1]; f.mv = (const uint2 *)p[2]; f.mat = (const uint2 *)p[3];
  f.emi = (const uint2 *)p[4]; f.pnd = (const uint2 *)p[5]; f.pmv = (const uint2 *)p[6];
  f.p_rad = pt[0]; f.p_nd = pt[1]; f.p_mv = pt[2]; f.p_mat = pt[3]; f.p_emi = pt[4]; f.p_pnd = pt[5]; f.p_pmv = pt[6];
  f.hist_prev = s->hist[prev]; f.mom_prev = s->mom[prev]; f.taa_prev = s->taa[prev];
  f.tmp = s->tmp; f.mom = s->mom[cur]; f.hist = s->hist[cur]; f.taa = s->taa[cur];
  const dim3 blk(32, 8), grd((s->W + 31) / 32, (s->H + 7) / 8);
  const dim3 tgrd((s->W + RT_W - 1) / RT_W, (s->H + RT_H - 1) / RT_H);
  k_svgf_temporal<<<grd, blk, 0, st>>>(f);
  const dim3 vgrd((s->W + VT_W - 1) / VT_W, (s->H + VT_H - 1) / VT_H);
  // each pass is set up while the one before runs: 7 us less at 641x363 with 3 iterations, 11 at 1920x1080 with 5
  cudaError_t e = launch_chained(k_svgf_variance, vgrd, dim3(VT_NT), 0, false, st, f, s->atrous[0]);
  int src = 0;
  for (int i = 0; i < s->o.iterations; i++) {
    const uint2 *a = s->atrous[src];
    uint2 *b = s->atrous[src ^ 1];
    if (e != cudaSuccess) break;
    switch (i) {
      case 0: e = launch_atrous<1>(f, a, b, i, st); break;
      case 1: e = launch_atrous<2>(f, a, b, i, st); break;
      case 2: e = launch_atrous<4>(f, a, b, i, st); break;
      case 3: e = launch_atrous<8>(f, a, b, i, st); break;
      default: e = launch_atrous<16>(f, a, b, i, st); break;
    }
    src ^= 1;
  }
  if (e == cudaSuccess) e = launch_chained(k_svgf_resolve, tgrd, dim3(RT_NT), 0, false, st, f, s->atrous[src]);
  const cudaError_t last = cudaGetLastError();  // (the first pass's; asked for in any case, so that none is left behind)
  if (e == cudaSuccess) e = last;
  if (e != cudaSuccess) return svgf_fail(s, HUSH_ERR_CUDA, std::string("SVGF: kernel launch: ") + cudaGetErrorString(e));
  s->reset = false;
  s->frame++;
  s->last_out = s->taa[cur];
  if (out) *out = s->last_out;
  return HUSH_OK;
}

// The reference's getter returns taa[frame & 1] after frame++, i.e. the previous frame's image (svgf.js:327, 376);
// this returns the image encode() produced last.
extern "C" const void *svgf_output(const svgf_t *s) { return s ? s->last_out : nullptr; }
extern "C" const char *svgf_last_error(const svgf_t *s) { return s ? s->last_error.c_str() : g_svgf_err.c_str(); }
