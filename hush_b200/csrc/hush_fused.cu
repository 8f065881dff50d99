// The fused B200 frame. Same arithmetic as the per-pass kernels (hush_passes.cu); different kernel boundaries:
//
//   stage 0  temporal   TEMPORAL + block features + the MLP heads (hush.js:79-308, 312-365) in one kernel: the 2x2
//                       blocks align with the tile, so the 20 features never leave the SM (the reference writes
//                       F0/F1 and reads them back in INFER). Writes A0, mom, key, par0..2 and the half-res block
//                       means Ah (= F2.zw) and guide Gh (= F3.xy).
//   stage 1  mid1|c1    mid1 (INFER's a-trous, hush.js:366) and COARSE1 (hush.js:404-421) in one launch
//   stage 2  mid2|c2    mid2 (hush.js:753) and coarse2 (hush.js:752) in one launch
//   stage 3  mid3       hush.js:754
//   stage 4  fine+final hush.js:560-621
//   stage 5  taa        hush.js:639-677
//
// Levels with a neighbourhood (the a-trous levels, TAA) stay separate launches: fusing them needs recomputed halos,
// and on B200 these passes are bound by instruction issue rather than HBM, so recomputation costs more than the
// L2-resident round trip of a half-res image.
#include <cuda.h>  // CUtensorMap and its enums (types only: the encoder is fetched from the driver)
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "hush_device.cuh"
#include "hush_pair.cuh"
#include "hush_internal.h"
#include "umma.cuh"

namespace hush {

// ------------------------------------------------------------------------------------------------ loaders
HD_INL float4 gh_decode(float4 g) {  // (oct normal, depth, count) -> (normal, depth)
  float4 n = oct_dec(g.x, g.y);
  n.w = g.z;
  return n;
}

// ------------------------------------------------------------------------------------------------ stage 0
// TEMPORAL pixel() (hush.js:111-223), block() (hush.js:226-282) and INFER's MLP with its heads (hush.js:312-365) in
// one kernel, one thread per 2x2 block (k_temporal_block below).
constexpr uint32_t MBAR_POLLS = 1u << 22;
// L of a tile entry outside the image or on sky (a valid luminance is finite and far above it)
constexpr float L_INVALID = -1e30f;
HD_INL bool l_valid(float L) { return L > -1e29f; }
// 1 for a valid L, else 0: 1 + 1e-20 L saturated to [0, 1] (one FMA instead of a comparison and a selection)
HD_INL float l_counts(float L) { return __saturatef(fmaf(L, 1e-20f, 1.0f)); }

// Eight values as one 16-byte operand row segment (hi), and the rounding residuals v - hi rounded again (lo): a
// split-precision operand, hi + lo carrying 16 (bf16) or 22 (f16) significant bits of v. Two values per conversion
// (cvt.rn.bf16x2.f32 / cvt.rn.f16x2.f32) and per residual subtraction (FP32x2).
HD_INL uint32_t cvt2(float a, float b, std::true_type) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}
HD_INL uint32_t cvt2(float a, float b, std::false_type) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}
HD_INL float2 back2(uint32_t u, std::true_type) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
HD_INL float2 back2(uint32_t u, std::false_type) {
  return __half22float2(*reinterpret_cast<const __half2 *>(&u));
}
template <bool BF16>
HD_INL void pack8_split(const float *v, uint4 &hi, uint4 &lo) {
  using T = std::integral_constant<bool, BF16>;
  uint32_t h[4], l[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    h[k] = cvt2(v[2 * k], v[2 * k + 1], T{});
    const float2 r = __fadd2_rn(make_float2(v[2 * k], v[2 * k + 1]), [&] {
      const float2 b = back2(h[k], T{});
      return make_float2(-b.x, -b.y);
    }());
    l[k] = cvt2(r.x, r.y, T{});
  }
  hi = make_uint4(h[0], h[1], h[2], h[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// pixel()'s inputs to block() for a pixel with a surface: P0..P4 as block() reads them (P0.y, the quantised luminance, comes
// from the tile instead) and the decoded normal.
struct PixOut {
  float4 P0, P1, P2, P3, P4, Ns;
};

// A pixel's loads are issued as cp.async copies into a shared-memory slot (no registers held while they fly): slot
// entry k of this thread at g[k * stride]: 0 normalDepth, 1 material, 2 previous par0, 3-6 key, 7-10 colour history,
// 11-14 moments of the bilinear footprint. The caller commits the group.
template <int STRIDE>
HD_INL void pixel_issue_async(const HushFrame &f, int px, int py, uint2 mvr, uint2 *g) {
  const int W = f.W, H = f.H;
  cp_async8(g, f.nd + py * f.p_nd + px);
  cp_async8(g + STRIDE, f.mat + py * f.p_mat + px);
  if (f.reset) return;
  const float4 mv = h4_to_f4(mvr);
  const float ppx = (float)px + mv.x, ppy = (float)py + mv.y;
  const int bix = __float2int_rz(floorf(ppx)), biy = __float2int_rz(floorf(ppy));
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int q = clampi(biy + (i >> 1), 0, H - 1) * W + clampi(bix + (i & 1), 0, W - 1);
    cp_async8(g + (3 + i) * STRIDE, f.key_prev + q);
    cp_async8(g + (7 + i) * STRIDE, f.hist_prev + q);
    cp_async8(g + (11 + i) * STRIDE, f.mom_prev + q);
  }
  const int cx = __float2int_rz(floorf(ppx + 0.5f)), cy = __float2int_rz(floorf(ppy + 0.5f));
  cp_async8(g + 2 * STRIDE, f.par0_prev + (clampi(cy, 0, H - 1) >> 1) * f.W2 + (clampi(cx, 0, W - 1) >> 1));
}
// qf16 of a value that is at most 65504 or NaN (which becomes -65504, as in qf16).
HD_INL float qf16_low(float x) { return __uint_as_float(__float_as_uint(fmaxf(x, -65504.0f)) & 0xffffe000u); }

// qf16 of feature i: all but the material means (12-15) and the logarithm of a quotient (7), which a zero divisor makes
// infinite, are logarithms of finite values, bounded ratios or unit values.
HD_INL float feature_qf16(int i, float x) { return i == 7 || (i >= 12 && i < 16) ? qf16(x) : qf16_low(x); }

// check_key() without normalising the decoded normal: v . n >= 0.9 |v|, tol = 0.05 zPrev + 0.01.
HD_INL bool check_key_v(float4 k, float4 n, float zPrev, float obj, float tol) {
  const float vz = 1.0f - fabsf(k.x) - fabsf(k.y), t = fmaxf(-vz, 0.0f);
  const float vx = k.x - copysignf(t, k.x), vy = k.y - copysignf(t, k.y);
  const float d = vx * n.x + vy * n.y + vz * n.z, l2 = vx * vx + vy * vy + vz * vz;
  return k.z >= 0.0f && k.w == obj && fabsf(k.z - zPrev) <= tol && d >= 0.9f * sqrtf(l2);
}

// pixel() of hush.js:111-223 over the (r, g, b, L) tile from the pixel's load slot g (texel k at g[k * STRIDE]); same
// arithmetic as temporal_pixel(). Writes A0, mom, key; returns false on sky, else the pixel's inputs to block() in o.
template <int STRIDE, class Tile>
HD_INL bool temporal_pixel_fast(const HushFrame &f, int px, int py, const Tile &T, const uint2 *g, uint2 mvr, PixOut &o) {
  const int W = f.W, H = f.H;
  const float4 nd = h4_to_f4(g[0]), mv = h4_to_f4(mvr);
  const int oi = py * W + px;
  if (nd.w < 0.0f) {
    f.A0[oi] = make_uint2(0, 0);
    f.mom[oi] = make_uint2(0, 0);
    sth(f.key, oi, make_float4(0.f, 0.f, -1.0f, mv.z));
    return false;
  }
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  // 3x3 statistics of the illumination (valid neighbours), two passes
  const float4 illum = T(0, 0);
  const float l = illum.w;
  // (r, g) as one packed FP32x2 lane pair, b and (in the second pass) L as the other: the same arithmetic per lane
  const float4 c0 = T(-1, -1);
  float2 s1xy = lo2(c0);
  float s1z = c0.z, cnt = l_counts(c0.w);
#pragma unroll
  for (int j = 1; j < 9; j++) {
    const float4 c = T(j % 3 - 1, j / 3 - 1);
    s1xy = add2(s1xy, lo2(c));  // invalid entries hold rgb = 0
    s1z += c.z;
    cnt += l_counts(c.w);
  }
  cnt = fmaxf(cnt, 1.0f);
  const float mux = s1xy.x / cnt, muy = s1xy.y / cnt, muz = s1z / cnt;
  const float slm = lum3(mux, muy, muz);
  const float2 nmu_xy = f2(-mux, -muy), nmu_zl = f2(-muz, -slm);
  float2 svxy = f2(0.f, 0.f), svzl = f2(0.f, 0.f);
#pragma unroll
  for (int j = 0; j < 9; j++) {
    const float4 c = T(j % 3 - 1, j / 3 - 1);
    if (l_valid(c.w)) {
      const float2 dxy = add2(lo2(c), nmu_xy), dzl = add2(hi2(c), nmu_zl);
      svxy = fma2(dxy, dxy, svxy);
      svzl = fma2(dzl, dzl, svzl);
    }
  }
  const float sdx = sqrtf(fmaxf(svxy.x / cnt, 1e-12f)), sdy = sqrtf(fmaxf(svxy.y / cnt, 1e-12f)),
              sdz = sqrtf(fmaxf(svzl.x / cnt, 1e-12f));
  const float svar = svzl.y / cnt;
  bool has = false;
  float hcx = 0.f, hcy = 0.f, hcz = 0.f;
  float4 hm = z4;
  float v = 0.f, alpha = 1.0f, gamma = 1.0f;
  if (!f.reset) {
    const float ppx = (float)px + mv.x, ppy = (float)py + mv.y;
    const float bx = floorf(ppx), by = floorf(ppy);
    const float fx = ppx - bx, fy = ppy - by;
    const float tol = 0.05f * mv.w + 0.01f;
    const float wf = (float)W, hf = (float)H;
    const bool ix[2] = {bx >= 0.0f && bx < wf, bx >= -1.0f && bx < wf - 1.0f};
    const bool iy[2] = {by >= 0.0f && by < hf, by >= -1.0f && by < hf - 1.0f};
    float sumW = 0.f;
    const float wts[4] = {(1.0f - fx) * (1.0f - fy), fx * (1.0f - fy), (1.0f - fx) * fy, fx * fy};
    bool ok[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
      ok[i] = (wts[i] > 0.0f) & ix[i & 1] & iy[i >> 1] & check_key_v(h4_to_f4(g[(3 + i) * STRIDE]), nd, mv.w, mv.z, tol);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (ok[i]) {
        const float4 c = h4_to_f4(g[(7 + i) * STRIDE]), m = h4_to_f4(g[(11 + i) * STRIDE]);
        const float2 w2 = bc2(wts[i]);
        sumW += wts[i];
        const float2 hxy = fma2(w2, lo2(c), f2(hcx, hcy));
        hcx = hxy.x; hcy = hxy.y;
        hcz += wts[i] * c.z;
        const float2 mxy = fma2(w2, lo2(m), f2(hm.x, hm.y)), mzw = fma2(w2, hi2(m), f2(hm.z, hm.w));
        hm = make_float4(mxy.x, mxy.y, mzw.x, mzw.y);
      }
    }
    if (sumW >= 0.01f) {
      hcx /= sumW; hcy /= sumW; hcz /= sumW;
      hm.x /= sumW; hm.y /= sumW; hm.z /= sumW; hm.w /= sumW;
      v = sumW;
      has = true;
    } else {
      const int cx = __float2int_rz(floorf(ppx + 0.5f)), cy = __float2int_rz(floorf(ppy + 0.5f));
      float n3 = 0.f;
      hcx = hcy = hcz = 0.f;
      hm = z4;
#pragma unroll 1
      for (int j = 0; j < 9; j++) {
        const int qx = cx + j % 3 - 1, qy = cy + j / 3 - 1;
        if (qx >= 0 && qy >= 0 && qx < W && qy < H && check_key_v(ldh(f.key_prev, qy * W + qx), nd, mv.w, mv.z, tol)) {
          n3 += 1.0f;
          const float4 c = ldh(f.hist_prev, qy * W + qx), m = ldh(f.mom_prev, qy * W + qx);
          hcx += c.x; hcy += c.y; hcz += c.z;
          hm.x += m.x; hm.y += m.y; hm.z += m.z; hm.w += m.w;
        }
      }
      if (n3 > 0.0f) {
        hcx /= n3; hcy /= n3; hcz /= n3;
        hm.x /= n3; hm.y /= n3; hm.z /= n3; hm.w /= n3;
        v = 0.1f;
        has = true;
      }
    }
    const float2 ag = unpack2(g[2 * STRIDE].x);
    alpha = ag.x;
    gamma = ag.y;
  }
  has = has && hm.w > 0.0f;
  float colx = illum.x, coly = illum.y, colz = illum.z;
  float nmx = l, nmy = l * l, nfast = l, len1 = 1.0f, lag = 0.0f;
  if (has) {
    const float hclx = fminf(fmaxf(hcx, mux - gamma * sdx), mux + gamma * sdx);
    const float hcly = fminf(fmaxf(hcy, muy - gamma * sdy), muy + gamma * sdy);
    const float hclz = fminf(fmaxf(hcz, muz - gamma * sdz), muz + gamma * sdz);
    len1 = fminf(hm.w + 1.0f, HMAX);
    const float a = fmaxf(alpha, 1.0f / len1);
    colx = hclx + (illum.x - hclx) * a;
    coly = hcly + (illum.y - hcly) * a;
    colz = hclz + (illum.z - hclz) * a;
    nmx = hm.x + (l - hm.x) * a;
    nmy = hm.y + (l * l - hm.y) * a;
    nfast = hm.z + (l - hm.z) * fmaxf(1.0f / 6.0f, 1.0f / len1);
    const float lh = lum3(hcx, hcy, hcz);
    lag = fabsf(slm - lh) / (sqrtf(fmaxf(svar / cnt, 1e-12f)) + 0.02f * lh + 1e-3f);
  } else {
    v = 0.0f;
  }
  const float tvar = fmaxf(nmy - nmx * nmx, 0.0f);
  const float4 A = make_float4(colx, coly, colz, svar + (tvar - svar) * fminf(len1 / 4.0f, 1.0f));
  const float2 oc = oct_enc(nd.x, nd.y, nd.z);
  sth(f.A0, oi, A);
  sth(f.mom, oi, make_float4(nmx, nmy, nfast, len1));
  sth(f.key, oi, make_float4(oc.x, oc.y, nd.w, mv.z));
  const float E = f.exposure;
  const float4 Aq = make_float4(qf16(A.x), qf16(A.y), qf16(A.z), qf16(A.w));
  const float m1 = E * qf16(nmx);
  const float m2 = E * E * qf16(nmy);
  const float ox = qf16(oc.x), oy = qf16(oc.y);  // (beside a NaN component the others leave the unit square)
  o.P0 = make_float4(E * lum(Aq), 0.0f, fmaxf(m2 - m1 * m1, 0.0f), len1);
  o.P1 = make_float4(qf16_low(v), qf16(lag), E * qf16(nfast), m1);
  // (an f16 depth is its own qf16 but for infinity and NaN)
  o.P2 = make_float4(ox, oy, fminf(fmaxf(nd.w, -65504.0f), 65504.0f), qf16(sqrtf(mv.x * mv.x + mv.y * mv.y)));
  o.P3 = h4_to_f4(g[STRIDE]);
  o.P4 = Aq;
  o.Ns = oct_dec(ox, oy);  // block() decodes the stored oct normal (hush.js:238)
  return true;
}

HD_INL float4 scale4(float4 v, float k) { return make_float4(v.x * k, v.y * k, v.z * k, v.w * k); }

HD_INL float4 ffma4(float s, float4 w, float4 a) {  // a + s * w as two packed FP32x2 FMAs
  const float2 lo = __ffma2_rn(make_float2(s, s), make_float2(w.x, w.y), make_float2(a.x, a.y));
  const float2 hi = __ffma2_rn(make_float2(s, s), make_float2(w.z, w.w), make_float2(a.z, a.w));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}

// ------------------------------------------------------------------------------------------------ k_temporal_block
// One thread per 2x2 block: tile 64 x 16 pixels = 32 x 8 blocks, 256 threads (64 x 8 and 128 for small frames). Each thread
// runs pixel() for its four pixels in block order, accumulates block()'s sums in registers in the WGSL's order
// (hush.js:226-282), forms the 20 features once and runs the whole FP32 MLP (weights in the constant bank, a kernel
// parameter: each FMA takes its weight as a broadcast operand), so after the tile barrier no thread waits for another. The
// tile is stored column-parity-split (even and odd columns in separate rows of 33 entries): neighbouring threads, two pixel
// columns apart, then read consecutive 16-byte entries. The per-pixel loads (G-buffer texels and the dependent reprojection
// gathers) go by cp.async into two shared-memory slots per thread, one pixel ahead: pixel q + 2's gathers are in
// flight while pixel q + 1 computes, without holding registers; a slot's texels are read where they are used. The
// tensor-core forms instead write each block's features as one operand row and run each layer as two tcgen05 MMAs (M = 128,
// N = 16) over the CTA's 256 rows, FP32 accumulators in TMEM; bias, ReLU and the heads stay FP32.
// Bound: instruction issue and the gathers' latency at 16 warps an SM (registers and the load slots; 5 CTAs of 128 threads
// take the L1 that the gathers hit in: 109 -> 129 us). So what is left out counts: sky pixels skip the block's sums, the
// key test needs no normalised normal, a quantisation clamps only the sides its value can reach, a validity counts by one
// saturating FMA. 1920x1080 FP32 119 -> 109 us (75.0 -> 71.4 M instructions), 3840x2160 bf16 530 -> 491, 256x256 16.2 -> 12.8.
constexpr int KB_TW = 64, KB_TH = 16, KB_NT = (KB_TW / 2) * (KB_TH / 2);
// Frames whose 16-row tiles fill at most the one wave of 2 x 148 CTAs an SM holds take 8-row tiles of 128 threads (4 CTAs
// an SM) in the per-thread MLP forms, so the pixels spread over more SMs: 256x256 14.3 -> 12.8 us, 640x360 21.3 -> 18.7.
// Beyond a wave both are even up to 1280x720 (35.8 either way at 960x540) and the larger apron share then loses
// (1600x900 79.0 -> 82.1, 1920x1080 108.3 -> 114.4). The tensor-core forms need the CTA's 256 rows.
constexpr int KB_HALF_CTAS = 2 * 148;
constexpr int KB_SWL = KB_TW + 2, KB_HW = KB_SWL / 2;
HD_INL int kb_tix(int r, int c) { return (2 * r + (c & 1)) * KB_HW + (c >> 1); }

constexpr int KB_NTEX = 15;  // texels of one pixel's loads (pixel_issue_async)
template <int TH>
struct KbSmem {
  float4 I[KB_SWL * (TH + 2)];            // illumination (r, g, b) and L (luminance or L_INVALID), apron 1
  float Lq[KB_SWL * (TH + 2)];            // E * qf16(L), or L_INVALID
  uint2 G[2][KB_NTEX][KB_TW / 4 * TH];    // two pixels' loads in flight per thread, thread-minor (conflict-free)
};
// Tensor-core forms: the same tile plus the MMA operands of the CTA's 256 rows (one per block) in the K-major
// no-swizzle layout, each as a split-precision pair (hi, lo): A1 256 x 32 (features, zero padded), A2 256 x 16
// (hidden layers), then the weights B1 / B2 / B3 (hi, and for bf16 lo).
// The per-pixel load slots (pixel phase) and the MMA operands (MLP phase, after a CTA barrier) share their space.
struct KbTcSmem {
  float4 I[KB_SWL * (KB_TH + 2)];
  float Lq[KB_SWL * (KB_TH + 2)];
  union {
    uint2 G[2][KB_NTEX][KB_NT];
    struct {
      alignas(128) uint8_t a1[KB_NT * 32 * 2];
      alignas(128) uint8_t a1lo[KB_NT * 32 * 2];
      alignas(128) uint8_t a2[KB_NT * 16 * 2];
      alignas(128) uint8_t a2lo[KB_NT * 16 * 2];
    };
  };
  alignas(128) uint8_t b[2 * MLP_TC_BLOB_BYTES];
  alignas(8) uint64_t mbar[2];  // one per 128-row group
  uint32_t tmem;
};

// One MMA layer over the CTA's 256 rows, as two independent 128-row groups: warps 0-3 (rows 0-127, TMEM columns
// [0, 16)) and warps 4-7 (rows 128-255, columns [16, 32)). A group waits only for its own four warps (a named barrier
// of 128 threads), then its first thread issues the group's MMAs and commits them to the group's mbarrier, so one
// group's MMAs run while the other group's warps are still forming their rows. Per K block the products A_hi B_hi,
// A_lo B_hi and (with lo weights, bf16) A_hi B_lo accumulate into the same FP32 accumulator; the dropped A_lo B_lo
// term is 2^-16 (bf16) / 2^-22 (f16) of the product. Every thread waits on its group's mbarrier (bounded) and loads
// its own row: warp w reads lanes 32 (w % 4) of column block w / 4. Returns false if the wait gave up.
HD_INL bool tc_layer_256(KbTcSmem &S, int li, const uint8_t *a, const uint8_t *alo, uint32_t kcore_a, int kblocks,
                         uint32_t b_off, bool b_lo, uint32_t kcore_b, uint32_t idesc, uint32_t phase, float *d) {
  const int g = li >> 7;
  umma::fence_proxy_async();
  umma::fence_before_sync();
  if (g == 0) asm volatile("bar.sync 1, 128;" ::: "memory");  // named barriers 1 / 2 (0 is __syncthreads)
  else asm volatile("bar.sync 2, 128;" ::: "memory");
  const uint32_t mbar = umma::smem_u32(&S.mbar[g]);
  if ((li & 127) == 0) {
    umma::fence_after_sync();
    const uint32_t b = umma::smem_u32(S.b) + b_off;
    const uint32_t ah = umma::smem_u32(a) + (uint32_t)g * 16u * 128u * kcore_a;
    const uint32_t al = umma::smem_u32(alo) + (uint32_t)g * 16u * 128u * kcore_a;
    for (int kb = 0; kb < kblocks; kb++) {
      const uint64_t bh = umma::sdesc(b + 256u * kb, 128, 128 * kcore_b);
      umma::mma_f16(S.tmem + 16u * g, umma::sdesc(ah + 256u * kb, 128, 128 * kcore_a), bh, idesc, kb > 0 ? 1u : 0u);
      umma::mma_f16(S.tmem + 16u * g, umma::sdesc(al + 256u * kb, 128, 128 * kcore_a), bh, idesc, 1u);
      if (b_lo)
        umma::mma_f16(S.tmem + 16u * g, umma::sdesc(ah + 256u * kb, 128, 128 * kcore_a),
                      umma::sdesc(b + MLP_TC_BLOB_BYTES + 256u * kb, 128, 128 * kcore_b), idesc, 1u);
    }
    umma::commit(mbar);
  }
  const bool ok = umma::mbar_wait_bounded(mbar, phase, MBAR_POLLS);
  umma::fence_after_sync();
  const int w = li >> 5;
  umma::ld16(S.tmem + ((uint32_t)(32 * (w & 3)) << 16) + 16u * (uint32_t)(w >> 2), d);
  return ok;
}

struct ParityTile {
  const float4 *I;
  int r, c;  // tile row / column of the pixel
  HD_INL float4 operator()(int dx, int dy) const { return I[kb_tix(r + dy, c + dx)]; }
};

// MODE 0: FP32 MLP per thread; 1 / 2: tensor-core MLP on split bf16 / f16 operands (dynamic shared memory);
// 3: the reference's f16-arithmetic MLP per thread (the `f16` option).
template <int MODE, int TH>
__global__ void __launch_bounds__(KB_TW / 4 * TH, 2 * KB_TH / TH)
    k_temporal_block(const __grid_constant__ HushFrame f, const __grid_constant__ MlpConst wp,
                     const uint4 *__restrict__ blob) {
  constexpr bool TC = MODE == 1 || MODE == 2;
  constexpr int NT = KB_TW / 4 * TH;
  static_assert(!TC || TH == KB_TH, "the tensor-core forms map a CTA's blocks to 256 operand rows");
  using Smem = std::conditional_t<TC, KbTcSmem, KbSmem<TH>>;
  extern __shared__ __align__(128) unsigned char kb_smem[];
  Smem &S = *reinterpret_cast<Smem *>(kb_smem);
  const int li = threadIdx.x;
  const float E = f.exposure;
  if constexpr (TC) {
    if (li < 32) {
      umma::tmem_alloc(umma::smem_u32(&S.tmem), 32);
      umma::tmem_relinquish();
    }
    if (li == 0) {
      umma::mbar_init(umma::smem_u32(&S.mbar[0]), 1);
      umma::mbar_init(umma::smem_u32(&S.mbar[1]), 1);
    }
    constexpr int NB = (MODE == 1 ? 2 : 1) * MLP_TC_BLOB_BYTES / 16;  // bf16: hi and lo weights
    for (int i = li; i < NB; i += NT) reinterpret_cast<uint4 *>(S.b)[i] = __ldg(blob + i);
    umma::fence_proxy_async();
    umma::fence_before_sync();
  }
  const int lbx = li % (KB_TW / 2), lby = li / (KB_TW / 2);
  const int px0 = blockIdx.x * KB_TW + 2 * lbx, py0 = blockIdx.y * TH + 2 * lby;
  // phase 1: the four pixels' motion first (each pixel's reprojection gathers then wait for one load round trip, not
  // two), then the first pixels' loads and gathers in flight with the tile loads
  uint2 mvq[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int px = px0 + (q & 1), py = py0 + (q >> 1);
    mvq[q] = (px < f.W && py < f.H) ? __ldg(f.mv + py * f.p_mv + px) : make_uint2(0, 0);
  }
  const int ox = blockIdx.x * KB_TW - 1, oy = blockIdx.y * TH - 1;
  constexpr int N = KB_SWL * (TH + 2);
#pragma unroll 1
  for (int i0 = 0; i0 < N; i0 += 2 * NT) {
    uint2 tn[2], tr[2], tm[2];
    bool tin[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int i = i0 + u * NT + li;
      const int qx = ox + i % KB_SWL, qy = oy + i / KB_SWL;
      tin[u] = i < N && qx >= 0 && qy >= 0 && qx < f.W && qy < f.H;
      const int cx = clampi(qx, 0, f.W - 1), cy = clampi(qy, 0, f.H - 1);
      tn[u] = __ldg(f.nd + cy * f.p_nd + cx);
      tr[u] = __ldg(f.rad + cy * f.p_rad + cx);
      tm[u] = __ldg(f.mat + cy * f.p_mat + cx);
    }
    if (i0 == 0) {  // the first two pixels' loads (cp.async into their slots), behind the first tile loads
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int px = px0 + (q & 1), py = py0 + (q >> 1);
        if (px < f.W && py < f.H) pixel_issue_async<NT>(f, px, py, mvq[q], &S.G[q][0][li]);
        cp_async_commit();
      }
    }
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int i = i0 + u * NT + li;
      if (i >= N) continue;
      float4 e = make_float4(0.f, 0.f, 0.f, L_INVALID);
      float lq = L_INVALID;
      if (tin[u] && h4_to_f4(tn[u]).w >= 0.0f) {
        const float4 r = h4_to_f4(tr[u]), m = h4_to_f4(tm[u]);
        e.x = r.x / fmaxf(m.x, 1e-3f);
        e.y = r.y / fmaxf(m.y, 1e-3f);
        e.z = r.z / fmaxf(m.z, 1e-3f);
        e.w = lum3(e.x, e.y, e.z);
        lq = E * qf16(e.w);
      }
      const int t = kb_tix(i / KB_SWL, i % KB_SWL);
      S.I[t] = e;
      S.Lq[t] = lq;
    }
  }
  __syncthreads();
  if constexpr (TC) umma::fence_after_sync();
  // phase 2: pixel() of the four pixels (block order: top-left, top-right, bottom-left, bottom-right), block() sums
  float nv = 0.f, Nx = 0.f, Ny = 0.f, Nz = 0.f, MV = 0.f, Z = 0.f;
  float4 S0 = make_float4(0.f, 0.f, 0.f, 0.f), S1 = S0, S3 = S0, AC = S0;
  float la[4], zs[4], nx4[4], ny4[4], nz4[4];
  bool okp[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int px = px0 + (q & 1), py = py0 + (q >> 1);
    const bool pin = px < f.W && py < f.H;
    if (q < 3) cp_async_wait<1>();  // this pixel's group has landed (the next pixel's may still fly)
    else cp_async_wait<0>();
    PixOut p;
    okp[q] = pin && temporal_pixel_fast<NT>(f, px, py, ParityTile{S.I, 2 * lby + (q >> 1) + 1, 2 * lbx + (q & 1) + 1},
                                               &S.G[q & 1][0][li], mvq[q], p);
    if (okp[q]) {
      la[q] = p.P0.x;
      zs[q] = p.P2.z;
      nx4[q] = p.Ns.x; ny4[q] = p.Ns.y; nz4[q] = p.Ns.z;
      nv += 1.0f;
      S0.x += p.P0.x; S0.z += p.P0.z; S0.w += p.P0.w;
      S1.x += p.P1.x; S1.y += p.P1.y; S1.z += p.P1.z; S1.w += p.P1.w;
      Nx += p.Ns.x; Ny += p.Ns.y; Nz += p.Ns.z;
      S3.x += p.P3.x; S3.y += p.P3.y; S3.z += p.P3.z; S3.w += p.P3.w;
      AC.x += p.P4.x; AC.y += p.P4.y; AC.z += p.P4.z; AC.w += p.P4.w;
      MV += p.P2.w;
      Z += p.P2.z;
    }
    if (q < 2) {  // pixel q + 2 into the slot pixel q has finished reading
      const int qx = px0 + (q & 1), qy = py0 + 1;
      if (qx < f.W && qy < f.H) pixel_issue_async<NT>(f, qx, qy, mvq[q + 2], &S.G[q & 1][0][li]);
      cp_async_commit();
    }
  }
  // phase 3: block() (hush.js:226-282)
  const int X = blockIdx.x * (KB_TW / 2) + lbx, Y = blockIdx.y * (TH / 2) + lby;
  const bool valid = X < f.W2 && Y < f.H2;
  const bool ok = nv != 0.0f;
  float fe[N_FEAT];
  float4 G = make_float4(0.f, 0.f, -1.0f, 0.f);
  {
    const float k = ok ? 1.0f / nv : 0.0f;
    S0 = scale4(S0, k); S1 = scale4(S1, k); S3 = scale4(S3, k); AC = scale4(AC, k);
    Nx *= k; Ny *= k; Nz *= k;
    MV *= k;
    Z *= k;
    const float Lacc = S0.x;
    float VA = 0.f;
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (okp[q]) VA += (la[q] - Lacc) * (la[q] - Lacc);
    VA *= k;
    // 4x4 neighbourhood (block +-1) of the quantised luminance, row-major; its middle entries are the block's own pixels
    // (a pixel of NaN depth is one of them but no valid neighbour: its luminance counts as the lowest)
    float s1 = 0.f, n4 = 0.f, lq[16], ly[16];
    float own[4];
#pragma unroll
    for (int e = 0; e < 16; e++) {
      const float x = S.Lq[kb_tix(2 * lby + (e >> 2), 2 * lbx + (e & 3))];
      const int q = (e >> 2) * 2 + (e & 3) - 3;  // of a middle entry
      if (((e >> 2) == 1 || (e >> 2) == 2) && ((e & 3) == 1 || (e & 3) == 2)) own[q] = okp[q] ? fmaxf(x, E * -65504.0f) : 0.0f;
      ly[e] = l_counts(x);
      lq[e] = ly[e] * x;
      s1 += lq[e];
      n4 += ly[e];
    }
    S0.y = (own[0] + own[1] + own[2] + own[3]) * k;
    const float mu4 = s1 / fmaxf(n4, 1.0f);
    float var4 = 0.f;
#pragma unroll
    for (int e = 0; e < 16; e++) {
      const float d = lq[e] - mu4;
      var4 += ly[e] * d * d;
    }
    var4 /= fmaxf(n4, 1.0f);
    const float nl = fmaxf(sqrtf(Nx * Nx + Ny * Ny + Nz * Nz), 1e-6f);
    const float nnx = Nx / nl, nny = Ny / nl, nnz = Nz / nl;
    float zmax = -1e30f, zmin = 1e30f, mind = 1e30f;
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (okp[q]) {
        zmax = fmaxf(zmax, zs[q]);
        zmin = fminf(zmin, zs[q]);
        mind = fminf(mind, nx4[q] * nnx + ny4[q] * nny + nz4[q] * nnz);
      }
    const float dz = fminf(fmaxf((zmax - zmin) / fmaxf(zmin, 1e-6f), 0.0f), 1.0f);
    const float dn = fminf(fmaxf(1.0f - mind, 0.0f), 2.0f);
    const float2 oc = oct_enc(nnx, nny, nnz);
    fe[0] = log1p_w(Lacc); fe[1] = log1p_w(S0.y); fe[2] = log1p_w(S0.z); fe[3] = log1p_w(var4);
    fe[4] = S0.w / HMAX; fe[5] = S1.x; fe[6] = log1p_w(S1.y);
    fe[7] = log1p_w(fabsf(S1.z - S1.w) / (S1.w + 1e-3f));
    fe[8] = oc.x; fe[9] = oc.y; fe[10] = dz; fe[11] = dn;
    fe[12] = S3.x; fe[13] = S3.y; fe[14] = S3.z; fe[15] = S3.w;
    fe[16] = 1.0f - nv / 4.0f; fe[17] = log1p_w(MV); fe[18] = log1p_w(mu4); fe[19] = log1p_w(VA);
    if (ok) G = make_float4(oc.x, oc.y, Z, nv);
  }
  const int o = Y * f.W2 + X;
  if (valid) {
    // block means and guide: F2.zw and F3.xy of hush.js:280-281 (hush.js:241-244 without valid pixels)
    f.Ah[o] = ok ? make_uint2(pk(AC.x, AC.y), pk(AC.z, AC.w)) : make_uint2(0, 0);
    f.Gh[o] = ok ? make_uint2(pk(G.x, G.y), pk(G.z, G.w)) : make_uint2(pk(0.f, 0.f), pk(-1.0f, 0.f));
    // the decoded guide every half-res consumer forms from F3 (octDec of the stored oct normal, stored depth)
    float4 gd = oct_dec(ok ? quant1(qf16(G.x)) : 0.f, ok ? quant1(qf16(G.y)) : 0.f);
    gd.w = ok ? quant1(qf16(G.z)) : -1.0f;
    f.Gd[o] = gd;
  }
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  if constexpr (TC) {
    __syncthreads();  // every thread is done with its load slots, which the operand rows overwrite
    // phase 4 (tensor cores): every thread writes its block's operand row (zeros for blocks outside the image or
    // without valid pixels) and takes part in all three layers
    constexpr bool BF16 = MODE == 1;
    constexpr int B1 = 16 * N_FEAT, B2 = B1 + 16 + 16 * 16, B3 = B2 + 16 + N_OUT * 16;
    const float *wb = reinterpret_cast<const float *>(wp.w);  // the decoded weights (their biases)
    constexpr uint32_t ID = umma::idesc_f16(BF16 ? 1 : 0, 128, 16);
    auto put_row = [&](uint8_t *hi, uint8_t *lo, int k0, int kcore, const float *v) {
      uint4 h, l;
      pack8_split<BF16>(v, h, l);
      *reinterpret_cast<uint4 *>(hi + umma::kmajor_off(li, k0, kcore)) = h;
      *reinterpret_cast<uint4 *>(lo + umma::kmajor_off(li, k0, kcore)) = l;
    };
#pragma unroll
    for (int c = 0; c < 4; c++) {
      float v8[8];
#pragma unroll
      for (int e = 0; e < 8; e++)
        v8[e] = (8 * c + e < N_FEAT && valid && ok) ? __half2float(__ushort_as_half(f2h(feature_qf16(8 * c + e, fe[8 * c + e])))) : 0.f;
      put_row(S.a1, S.a1lo, 8 * c, 4, v8);
    }
    float row[16], d[16];
    bool good = tc_layer_256(S, li, S.a1, S.a1lo, 4, 2, 0, BF16, 4, ID, 0, d);
#pragma unroll
    for (int j = 0; j < 16; j++) row[j] = fmaxf(d[j] + wb[B1 + j], 0.0f);
    put_row(S.a2, S.a2lo, 0, 2, row);
    put_row(S.a2, S.a2lo, 8, 2, row + 8);
    good &= tc_layer_256(S, li, S.a2, S.a2lo, 2, 1, 1024, BF16, 2, ID, 1, d);
#pragma unroll
    for (int j = 0; j < 16; j++) row[j] = fmaxf(d[j] + wb[B2 + j], 0.0f);
    put_row(S.a2, S.a2lo, 0, 2, row);
    put_row(S.a2, S.a2lo, 8, 2, row + 8);
    good &= tc_layer_256(S, li, S.a2, S.a2lo, 2, 1, 1536, BF16, 2, ID, 0, d);
    float out[N_OUT];
#pragma unroll
    for (int j = 0; j < N_OUT; j++) out[j] = d[j] + wb[B3 + j];
    umma::fence_before_sync();
    __syncthreads();
    if (li < 32) {
      umma::fence_after_sync();
      umma::tmem_dealloc(S.tmem, 32);
    }
    if (!good) {
      atomicOr(f.err, 1u);
      return;
    }
    if (!valid) return;
    if (!ok) {
      sth(f.par0, o, z4); sth(f.par1, o, z4); sth(f.par2, o, z4);
      return;
    }
    float4 p0, p1, p2;
    mlp_heads(out, p0, p1, p2);
    sth(f.par0, o, p0);
    sth(f.par1, o, p1);
    sth(f.par2, o, p2);
    return;
  }
  if (!valid) return;
  if (!ok) {  // INFER on a block without valid pixels writes zeros (hush.js:343-346)
    sth(f.par0, o, z4); sth(f.par1, o, z4); sth(f.par2, o, z4);
    return;
  }
  if constexpr (MODE == 3) {
    // phase 4 (the `f16` option, hush.js:683-703): f16 products and running sums per unit in the WGSL's order (bias,
    // then the inputs in increasing index), two units per f16x2 instruction, weights as f16x2 unit pairs in the
    // constant bank; the features enter as stored (packed f16, hush.js:278-280)
    const uint32_t *Wh = reinterpret_cast<const uint32_t *>(wp.w);
    uint32_t a[8], b[8];
#pragma unroll
    for (int p = 0; p < 8; p++) a[p] = Wh[MLP_HALF_B1 + p];
#pragma unroll
    for (int i = 0; i < N_FEAT; i++) {
      const uint32_t x = hdup(f2h(feature_qf16(i, fe[i])));
#pragma unroll
      for (int p = 0; p < 8; p++) a[p] = hadd2_rn(a[p], hmul2_rn(x, Wh[MLP_HALF_W1 + i * 8 + p]));
    }
#pragma unroll
    for (int p = 0; p < 8; p++) { a[p] = hrelu2(a[p]); b[p] = Wh[MLP_HALF_B2 + p]; }
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const uint32_t x = hdup((i & 1) ? a[i >> 1] >> 16 : a[i >> 1]);
#pragma unroll
      for (int p = 0; p < 8; p++) b[p] = hadd2_rn(b[p], hmul2_rn(x, Wh[MLP_HALF_W2 + i * 8 + p]));
    }
#pragma unroll
    for (int p = 0; p < 8; p++) b[p] = hrelu2(b[p]);
#pragma unroll
    for (int p = 0; p < 6; p++) a[p] = Wh[MLP_HALF_B3 + p];
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const uint32_t x = hdup((i & 1) ? b[i >> 1] >> 16 : b[i >> 1]);
#pragma unroll
      for (int p = 0; p < 6; p++) a[p] = hadd2_rn(a[p], hmul2_rn(x, Wh[MLP_HALF_W3 + i * 6 + p]));
    }
    float out[N_OUT];
#pragma unroll
    for (int p = 0; p < 6; p++) { out[2 * p] = hlo(a[p]); out[2 * p + 1] = hhi(a[p]); }
    float4 p0, p1, p2;
    mlp_heads(out, p0, p1, p2);
    sth(f.par0, o, p0);
    sth(f.par1, o, p1);
    sth(f.par2, o, p2);
    return;
  }
  // phase 4: the MLP (hush.js:681-704) on the features as stored (packed f16, hush.js:278-280, 348-353); each unit
  // is its bias plus the inputs in increasing index, FP32 with packed FP32x2 FMAs
#pragma unroll
  for (int i = 0; i < N_FEAT; i++) fe[i] = __half2float(__ushort_as_half(f2h(feature_qf16(i, fe[i]))));
  const float4 *Wt;
  if constexpr (!TC) Wt = wp.w;
  float4 a[4];
#pragma unroll
  for (int q = 0; q < 4; q++) a[q] = Wt[MLP_FP32_B1 + q];
#pragma unroll
  for (int i = 0; i < N_FEAT; i++)
#pragma unroll
    for (int q = 0; q < 4; q++) a[q] = ffma4(fe[i], Wt[MLP_FP32_W1 + i * 4 + q], a[q]);
  float h[16];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    h[4 * q] = fmaxf(a[q].x, 0.f); h[4 * q + 1] = fmaxf(a[q].y, 0.f);
    h[4 * q + 2] = fmaxf(a[q].z, 0.f); h[4 * q + 3] = fmaxf(a[q].w, 0.f);
  }
#pragma unroll
  for (int q = 0; q < 4; q++) a[q] = Wt[MLP_FP32_B2 + q];
#pragma unroll
  for (int i = 0; i < 16; i++)
#pragma unroll
    for (int q = 0; q < 4; q++) a[q] = ffma4(h[i], Wt[MLP_FP32_W2 + i * 4 + q], a[q]);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    h[4 * q] = fmaxf(a[q].x, 0.f); h[4 * q + 1] = fmaxf(a[q].y, 0.f);
    h[4 * q + 2] = fmaxf(a[q].z, 0.f); h[4 * q + 3] = fmaxf(a[q].w, 0.f);
  }
#pragma unroll
  for (int q = 0; q < 4; q++) a[q] = Wt[MLP_FP32_B3 + q];  // (output q, 4 + q, 8 + q, 0)
#pragma unroll
  for (int i = 0; i < 16; i++)
#pragma unroll
    for (int q = 0; q < 4; q++) a[q] = ffma4(h[i], Wt[MLP_FP32_W3 + i * 4 + q], a[q]);
  float out[N_OUT];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    out[q] = a[q].x;
    out[4 + q] = a[q].y;
    out[8 + q] = a[q].z;
  }
  float4 p0, p1, p2;
  mlp_heads(out, p0, p1, p2);
  sth(f.par0, o, p0);
  sth(f.par1, o, p1);
  sth(f.par2, o, p2);
}

// ------------------------------------------------------------------------------------------------ half / quarter
// 16 x 8 tiles like the reference. One launch runs two kinds of tiles: blockIdx.x < nA runs kind A, the rest kind B.
constexpr int HT_W = 16, HT_H = 8;

// mid1 (hush.js:326, 366): 3x3 step 1 with prefilter on the block means, learned s_1 / c_1 (stored par1.y / par2.y
// are the qf16 values INFER passes).
// TMA staging of a mid level's halo tile (interior tiles): the guide Gd (float4 per texel, a 3-d FLOAT32 map
// {4, W2, H2}) lands in sG as is, the level (8-byte texels, a 2-d UINT64 map {W2, H2}) in a staging array that is
// widened to float4 afterwards. Both copies start at x = bx - STEP, even for STEP = 2 / 4, so the 8-byte map's
// innermost coordinate is 16-byte aligned; the boxes are (16 + 2 STEP) x (8 + 2 STEP) texels.
struct HalfMaps {
  CUtensorMap gd2, gd4, bh0, bh1;  // Gd with the step-2 / step-4 box; Bh0 (mid2's source) and Bh1 (mid3's)
  CUtensorMap gd1, ah;             // mid1: Gd with an 18 x 10 box at x = bx - 1; Ah with a 20 x 10 box at x = bx - 2
  CUtensorMap cgd, c1;             // coarse2 (quarter resolution): CGd and C1 with 24 x 16 boxes at x = bx - 4
  int ok;                          // 0: every tile loads with plain loads (odd W2, or no encoder)
  int qok;                         // the same for the quarter-resolution maps (odd W4)
};
constexpr uint32_t TMA_POLLS = 1u << 22;
// Waits (bounded) for a halo tile's TMA copies. On giving up it sets bit 3 of the error word and returns false: the
// caller then fills its tile with the plain clamped loads, so the output stays defined. Interior tiles need no
// clamping, so a copy that still lands later writes the very values those loads wrote.
HD_INL bool tma_wait_or_flag(const HushFrame &f, uint32_t mb) {
  if (umma::mbar_wait_bounded(mb, 0, TMA_POLLS)) return true;
  atomicOr(f.err, 8u);
  return false;
}
HD_INL void tma_expect(uint32_t mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}
HD_INL void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t mbar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(mbar)
      : "memory");
}
HD_INL void tma_load_3d(uint32_t dst, const CUtensorMap *map, int c, int x, int y, uint32_t mbar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
          "r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c), "r"(x), "r"(y), "r"(mbar)
      : "memory");
}

// mid1 (hush.js:326, 366): the block means Ah and the guide, apron 1. On interior tiles the guide lands in sG by TMA
// (3-d map, no alignment rule on x) and Ah in a staging array from x = bx - 2 (the 8-byte map's x must be even), the
// tile's column c being the staged column c + 1.
HD_INL void tile_mid1(const HushFrame &f, int tileX, int tileY, float4 *sA, float4 *sG, const HalfMaps *M) {
  constexpr int AP = 1, SW = HT_W + 2, SH = HT_H + 2, BW = HT_W + 4;
  __shared__ alignas(128) uint2 stage[BW * SH];
  __shared__ alignas(8) uint64_t mbar;
  const int li = threadIdx.x;
  const int bx = tileX * HT_W, by = tileY * HT_H;
  const bool interior = bx - 2 >= 0 && by - 1 >= 0 && bx + HT_W + 2 <= f.W2 && by + HT_H + 1 <= f.H2;
  const bool inner = M && interior;
  const int X = bx + li % HT_W, Y = by + li / HT_W;
  const bool in_img = X < f.W2 && Y < f.H2;
  const int o = Y * f.W2 + X;
  // this pixel's parameters, in flight while the tile arrives
  uint2 p1 = make_uint2(0, 0), p2 = make_uint2(0, 0);
  if (in_img) { p1 = __ldg(f.par1 + o); p2 = __ldg(f.par2 + o); }
  bool staged = false;
  if (inner) {
    const uint32_t mb = umma::smem_u32(&mbar);
    if (li == 0) umma::mbar_init(mb, 1);
    __syncthreads();
    if (li == 0) {
      tma_expect(mb, BW * SH * 8 + SW * SH * 16);
      tma_load_2d(umma::smem_u32(stage), &M->ah, bx - 2, by - 1, mb);
      tma_load_3d(umma::smem_u32(sG), &M->gd1, 0, bx - 1, by - 1, mb);
    }
    staged = tma_wait_or_flag(f, mb);
    if (staged)
      for (int i = li; i < SW * SH; i += HT_W * HT_H) sA[i] = h4_to_f4(stage[(i / SW) * BW + i % SW + 1]);
  }
  if (!staged) {
    for (int i = li; i < SW * SH; i += HT_W * HT_H) {
      const int q = clampi(by - AP + i / SW, 0, f.H2 - 1) * f.W2 + clampi(bx - AP + i % SW, 0, f.W2 - 1);
      sA[i] = ldh(f.Ah, q);
      sG[i] = __ldg(f.Gd + q);
    }
  }
  __syncthreads();
  if (!in_img) return;
  const int lx = li % HT_W + AP, ly = li / HT_W + AP;
  if (sG[ly * SW + lx].w < 0.0f) { sth(f.Bh0, o, make_float4(0.f, 0.f, 0.f, 0.f)); return; }
  const float s = h4_to_f4(p1).y, c = h4_to_f4(p2).y;
  sth(f.Bh0, o, interior ? filt_x<1, 1, true, SW, false>(sA, sG, lx, ly, X, Y, f.W2, f.H2, s, c)
                         : filt_x<1, 1, true, SW, true>(sA, sG, lx, ly, X, Y, f.W2, f.H2, s, c));
}

template <int STEP, int COMP>
HD_INL void tile_mid(const HushFrame &f, int tileX, int tileY, const uint2 *src, uint2 *dst, float4 *sA, float4 *sG,
                     const CUtensorMap *mg, const CUtensorMap *ms) {
  constexpr int AP = STEP, SW = HT_W + 2 * AP, SH = HT_H + 2 * AP;
  __shared__ alignas(128) uint2 stage[SW * SH];
  __shared__ alignas(8) uint64_t mbar;
  const int li = threadIdx.x;
  const int bx = tileX * HT_W, by = tileY * HT_H;
  const bool interior = bx - AP >= 0 && by - AP >= 0 && bx + HT_W + AP <= f.W2 && by + HT_H + AP <= f.H2;
  const bool inner = mg && interior;
  const int X = bx + li % HT_W, Y = by + li / HT_W;
  const bool in_img = X < f.W2 && Y < f.H2;
  const int o = Y * f.W2 + X;
  uint2 p1 = make_uint2(0, 0), p2 = make_uint2(0, 0);  // this pixel's parameters, in flight with the tile
  if (in_img) { p1 = __ldg(f.par1 + o); p2 = __ldg(f.par2 + o); }
  bool staged = false;
  if (inner) {
    const uint32_t mb = umma::smem_u32(&mbar);
    if (li == 0) umma::mbar_init(mb, 1);
    __syncthreads();
    if (li == 0) {
      tma_expect(mb, SW * SH * (8 + 16));
      tma_load_2d(umma::smem_u32(stage), ms, bx - AP, by - AP, mb);
      tma_load_3d(umma::smem_u32(sG), mg, 0, bx - AP, by - AP, mb);
    }
    staged = tma_wait_or_flag(f, mb);
    if (staged)
      for (int i = li; i < SW * SH; i += HT_W * HT_H) sA[i] = h4_to_f4(stage[i]);
  }
  if (!staged) {
    for (int i = li; i < SW * SH; i += HT_W * HT_H) {
      const int q = clampi(by - AP + i / SW, 0, f.H2 - 1) * f.W2 + clampi(bx - AP + i % SW, 0, f.W2 - 1);
      sA[i] = ldh(src, q);
      sG[i] = __ldg(f.Gd + q);
    }
  }
  __syncthreads();
  if (!in_img) return;
  const int lx = li % HT_W + AP, ly = li / HT_W + AP;
  if (sG[ly * SW + lx].w < 0.0f) { sth(dst, o, make_float4(0.f, 0.f, 0.f, 0.f)); return; }
  const float4 a = h4_to_f4(p1), b = h4_to_f4(p2);
  const float s = COMP == 2 ? a.z : a.w, c = COMP == 2 ? b.z : b.w;
  sth(dst, o, interior ? filt_x<1, STEP, false, SW, false>(sA, sG, lx, ly, X, Y, f.W2, f.H2, s, c)
                       : filt_x<1, STEP, false, SW, true>(sA, sG, lx, ly, X, Y, f.W2, f.H2, s, c));
}

// down() (hush.js:385-402) from the half-res planes.
HD_INL void down_h(const HushFrame &f, int Qx, int Qy, float4 &c, float4 &g) {
  float N = 0.f, vr = 0.f, z = 0.f, cx = 0.f, cy = 0.f, cz = 0.f, nx = 0.f, ny = 0.f, nz = 0.f;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int hx = Qx * 2 + (j & 1), hy = Qy * 2 + (j >> 1);
    if (hx >= f.W2 || hy >= f.H2) continue;
    const float w = ldh(f.Gh, hy * f.W2 + hx).w;  // pixel count of the block
    if (w <= 0.0f) continue;
    const float4 a = ldh(f.Ah, hy * f.W2 + hx);
    const float4 n = __ldg(f.Gd + hy * f.W2 + hx);
    N += w;
    cx += w * a.x; cy += w * a.y; cz += w * a.z;
    vr += w * a.w;
    nx += w * n.x; ny += w * n.y; nz += w * n.z;
    z += w * n.w;
  }
  if (N == 0.0f) {
    c = make_float4(0.f, 0.f, 0.f, 0.f);
    g = make_float4(0.f, 0.f, -1.0f, 0.f);
    return;
  }
  const float nl = fmaxf(sqrtf(nx * nx + ny * ny + nz * nz), 1e-6f);
  const float2 o = oct_enc(nx / nl, ny / nl, nz / nl);
  c = make_float4(qf16(cx / N), qf16(cy / N), qf16(cz / N), qf16(vr / N / N));
  g = make_float4(qf16(o.x), qf16(o.y), qf16(z / N), 0.0f);
}

HD_INL void tile_coarse1(const HushFrame &f, int tileX, int tileY, float4 *sA, float4 *sG) {
  constexpr int AP = 2, SW = HT_W + 2 * AP, SH = HT_H + 2 * AP;
  const int li = threadIdx.x;
  const int bx = tileX * HT_W, by = tileY * HT_H;
  for (int i = li; i < SW * SH; i += HT_W * HT_H) {
    const int lqx = bx - AP + i % SW, lqy = by - AP + i / SW;
    const int qx = clampi(lqx, 0, f.W4 - 1), qy = clampi(lqy, 0, f.H4 - 1);
    float4 c, g;
    down_h(f, qx, qy, c, g);
    sA[i] = c;
    sG[i] = gh_decode(g);
    if (lqx == qx && lqy == qy && lqx >= bx && lqy >= by && lqx < bx + HT_W && lqy < by + HT_H) {
      sth(f.CG, qy * f.W4 + qx, g);
      // coarse2 and FINE_FINAL read the guide back from its rgba16float texture
      f.CGd[qy * f.W4 + qx] = gh_decode(quant4(g));
    }
  }
  __syncthreads();
  const int X = bx + li % HT_W, Y = by + li / HT_W;
  if (X >= f.W4 || Y >= f.H4) return;
  const int lx = li % HT_W + AP, ly = li / HT_W + AP;
  if (sG[ly * SW + lx].w < 0.0f) { sth(f.C1, Y * f.W4 + X, make_float4(0.f, 0.f, 0.f, 0.f)); return; }
  const bool interior = bx - AP >= 0 && by - AP >= 0 && bx + HT_W + AP <= f.W4 && by + HT_H + AP <= f.H4;
  sth(f.C1, Y * f.W4 + X, interior ? filt_x<2, 1, true, SW, false>(sA, sG, lx, ly, X, Y, f.W4, f.H4, COARSE_S, 1.0f)
                                   : filt_x<2, 1, true, SW, true>(sA, sG, lx, ly, X, Y, f.W4, f.H4, COARSE_S, 1.0f));
}

// coarse2 (hush.js:482-525, kind coarse): C1 and the decoded quarter-res guide, apron 4; interior tiles by TMA as
// the mid levels (x = bx - 4 is even).
HD_INL void tile_coarse2(const HushFrame &f, int tileX, int tileY, float4 *sA, float4 *sG, const HalfMaps *M) {
  constexpr int AP = 4, SW = HT_W + 2 * AP, SH = HT_H + 2 * AP;
  __shared__ alignas(128) uint2 stage[SW * SH];
  __shared__ alignas(8) uint64_t mbar;
  const int li = threadIdx.x;
  const int bx = tileX * HT_W, by = tileY * HT_H;
  const bool inner = M && bx - AP >= 0 && by - AP >= 0 && bx + HT_W + AP <= f.W4 && by + HT_H + AP <= f.H4;
  bool staged = false;
  if (inner) {
    const uint32_t mb = umma::smem_u32(&mbar);
    if (li == 0) umma::mbar_init(mb, 1);
    __syncthreads();
    if (li == 0) {
      tma_expect(mb, SW * SH * (8 + 16));
      tma_load_2d(umma::smem_u32(stage), &M->c1, bx - AP, by - AP, mb);
      tma_load_3d(umma::smem_u32(sG), &M->cgd, 0, bx - AP, by - AP, mb);
    }
    staged = tma_wait_or_flag(f, mb);
    if (staged)
      for (int i = li; i < SW * SH; i += HT_W * HT_H) sA[i] = h4_to_f4(stage[i]);
  }
  if (!staged) {
    for (int i = li; i < SW * SH; i += HT_W * HT_H) {
      const int q = clampi(by - AP + i / SW, 0, f.H4 - 1) * f.W4 + clampi(bx - AP + i % SW, 0, f.W4 - 1);
      sA[i] = ldh_pass(f.C1, q);
      sG[i] = ld_pass(f.CGd + q);
    }
  }
  __syncthreads();
  const int X = bx + li % HT_W, Y = by + li / HT_W;
  if (X >= f.W4 || Y >= f.H4) return;
  const int lx = li % HT_W + AP, ly = li / HT_W + AP;
  if (sG[ly * SW + lx].w < 0.0f) { sth(f.C0, Y * f.W4 + X, make_float4(0.f, 0.f, 0.f, 0.f)); return; }
  const bool interior = bx - AP >= 0 && by - AP >= 0 && bx + HT_W + AP <= f.W4 && by + HT_H + AP <= f.H4;
  sth(f.C0, Y * f.W4 + X, interior ? filt_x<2, 2, true, SW, false>(sA, sG, lx, ly, X, Y, f.W4, f.H4, COARSE_S, 1.0f)
                                   : filt_x<2, 2, true, SW, true>(sA, sG, lx, ly, X, Y, f.W4, f.H4, COARSE_S, 1.0f));
}

// mid2 / mid3 (hush.js:482-525, 753-754) on 32 x 8 tiles in two-pixel lanes (filt_pair): the level and the decoded
// guide of the (32 + 2 STEP) x (8 + 2 STEP) window are loaded as texel pairs (one 16-byte load for the two 8-byte
// level texels of an even column pair when the row pitch allows it, clamped single loads at the image border), every
// load of the thread issued before the first is unpacked, and stored in the even-column pair layout.
constexpr int MP_W = 32;  // tile width of the two-pixel mid tiles (16 lanes x 8 rows)
template <int STEP>
constexpr int mid_pair_smem() {
  return 4 * ((MP_W + 2 * STEP) / 2) * (HT_H + 2 * STEP) * 16;
}
template <int STEP, int COMP>
HD_INL void tile_mid_pair(const HushFrame &f, int tileX, int tileY, const uint2 *src, uint2 *dst, float4 *smem) {
  constexpr int AP = STEP, SW = MP_W + 2 * AP, SH = HT_H + 2 * AP, EW = SW / 2, NE = EW * SH;
  constexpr int NT = HT_W * HT_H, NIT = (NE + NT - 1) / NT;
  const PairTile T{smem, smem + NE, smem + 2 * NE, smem + 3 * NE};
  const int li = threadIdx.x;
  const int bx = tileX * MP_W, by = tileY * HT_H;
  const bool interior = bx - AP >= 0 && by - AP >= 0 && bx + MP_W + AP <= f.W2 && by + HT_H + AP <= f.H2;
  const int tx = li % (MP_W / 2), ty = li / (MP_W / 2);
  const int X = bx + 2 * tx, Y = by + ty;
  const bool in0 = X < f.W2 && Y < f.H2, in1 = in0 && X + 1 < f.W2;
  const int o = Y * f.W2 + X;
  // this pair's parameters, in flight with the tile
  uint2 pa1 = make_uint2(0, 0), pa2 = pa1, pb1 = pa1, pb2 = pa1;
  if (in0) { pa1 = __ldg(f.par1 + o); pa2 = __ldg(f.par2 + o); }
  if (in1) { pb1 = __ldg(f.par1 + o + 1); pb2 = __ldg(f.par2 + o + 1); }
  const bool even_w = !(f.W2 & 1);
  uint4 lv[NIT];
  float4 qa[NIT], qb[NIT];
#pragma unroll
  for (int i = 0; i < NIT; i++) {
    const int e = li + i * NT;
    const int r = e / EW, k = e % EW;
    const int gy = clampi(by - AP + r, 0, f.H2 - 1), gx = bx - AP + 2 * k;
    const int x0 = clampi(gx, 0, f.W2 - 1), x1 = clampi(gx + 1, 0, f.W2 - 1);
    if (e < NE) {
      if (even_w && gx >= 0 && gx + 1 < f.W2) {
        lv[i] = ld_pass(reinterpret_cast<const uint4 *>(src + gy * f.W2 + gx));
      } else {
        const uint2 a = ld_pass(src + gy * f.W2 + x0), b = ld_pass(src + gy * f.W2 + x1);
        lv[i] = make_uint4(a.x, a.y, b.x, b.y);
      }
      qa[i] = __ldg(f.Gd + gy * f.W2 + x0);
      qb[i] = __ldg(f.Gd + gy * f.W2 + x1);
    }
  }
#pragma unroll
  for (int i = 0; i < NIT; i++) {
    const int e = li + i * NT;
    if (e < NE)
      pair_put(T, e, h4_to_f4(make_uint2(lv[i].x, lv[i].y)), h4_to_f4(make_uint2(lv[i].z, lv[i].w)), qa[i], qb[i]);
  }
  __syncthreads();
  if (!in0) return;
  const float4 a0 = h4_to_f4(pa1), b0 = h4_to_f4(pa2), a1 = h4_to_f4(pb1), b1 = h4_to_f4(pb2);
  const float2 s = COMP == 2 ? f2(a0.z, a1.z) : f2(a0.w, a1.w), c = COMP == 2 ? f2(b0.z, b1.z) : f2(b0.w, b1.w);
  const int row = ty + AP, col = 2 * tx + AP;
  float4 r0, r1;
  if (interior) filt_pair<1, STEP, false, false, false, EW>(T, row, col, X, Y, f.W2, f.H2, s, c, r0, r1);
  else filt_pair<1, STEP, false, false, true, EW>(T, row, col, X, Y, f.W2, f.H2, s, c, r0, r1);
  const float4 zc = T.g1[pe<false, EW>(row, col)];  // centre depths (z, z') in .z / .w
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  if (zc.z < 0.0f) r0 = z4;  // sky centres write zeros (hush.js:505)
  if (zc.w < 0.0f) r1 = z4;
  if (in1 && even_w) {
    const uint2 u0 = f4_to_h4(r0), u1 = f4_to_h4(r1);
    *reinterpret_cast<uint4 *>(dst + o) = make_uint4(u0.x, u0.y, u1.x, u1.y);
  } else {
    sth(dst, o, r0);
    if (in1) sth(dst, o + 1, r1);
  }
}

// The half-res levels, one kind of tile per launch (PART, a HalfPart): stage 1 mid1 (HP_MID) or COARSE1 (HP_COARSE)
// tiles, stage 2 mid2 or coarse2 tiles, stage 3 mid3 tiles; block b is mid tile b (nA of them, nAx per row) or
// coarse tile b (nBx per row).
template <int STAGE, int PART>
__global__ void __launch_bounds__(HT_W *HT_H) k_half_stage(const __grid_constant__ HushFrame f, int nAx, int nA,
                                                           int nBx, const __grid_constant__ HalfMaps M) {
  constexpr int SMAX = (HT_W + 8) * (HT_H + 8);
  __shared__ alignas(128) float4 sA[SMAX];
  __shared__ alignas(128) float4 sG[SMAX];
  const int b = (int)blockIdx.x;
  if (PART == HP_MID) {
    if (b >= nA) return;
    const int tX = b % nAx, tY = b / nAx;
    if (STAGE == 1) tile_mid1(f, tX, tY, sA, sG, M.ok ? &M : nullptr);
    else if (STAGE == 2) tile_mid<2, 2>(f, tX, tY, f.Bh0, f.Bh1, sA, sG, M.ok ? &M.gd2 : nullptr, &M.bh0);
    else tile_mid<4, 3>(f, tX, tY, f.Bh1, f.Bh0, sA, sG, M.ok ? &M.gd4 : nullptr, &M.bh1);
  } else {
    const int tX = b % nBx, tY = b / nBx;
    if (STAGE == 1) tile_coarse1(f, tX, tY, sA, sG);
    else if (STAGE == 2) tile_coarse2(f, tX, tY, sA, sG, M.qok ? &M : nullptr);
  }
}

// stages 2 and 3 with the two-pixel mid tiles: 32 x 8 mid2 / mid3 tiles (HP_MID), or stage 2's coarse2 tiles (16 x 8,
// quarter resolution; HP_COARSE). Dynamic shared memory: the pair tile, or coarse2's two float4 tiles.
template <int STAGE, int PART, bool NEXT>
__global__ void __launch_bounds__(HT_W *HT_H) k_half_pair(const __grid_constant__ HushFrame f, int nAx, int nA,
                                                          int nBx, const __grid_constant__ HalfMaps M) {
  if constexpr (NEXT) pass_begin(true);
  extern __shared__ __align__(128) float4 hp_smem[];  // 128-byte aligned: coarse2 stages its guide by TMA
  const int b = (int)blockIdx.x;
  if (PART == HP_MID) {
    if (b >= nA) return;
    if (STAGE == 2) tile_mid_pair<2, 2>(f, b % nAx, b / nAx, f.Bh0, f.Bh1, hp_smem);
    else tile_mid_pair<4, 3>(f, b % nAx, b / nAx, f.Bh1, f.Bh0, hp_smem);
  } else if (STAGE == 2) {
    constexpr int SMAX = (HT_W + 8) * (HT_H + 8);
    tile_coarse2(f, b % nBx, b / nBx, hp_smem, hp_smem + SMAX, M.qok ? &M : nullptr);
  }
}

// ------------------------------------------------------------------------------------------------ stage 4 / 5
constexpr int FT_W = 32, FT_H = 8;  // TAA's tile

// FINE_FINAL on a 32 x 16 tile, two vertically adjacent pixels of one 2 x 2 block per thread. Before the barrier the CTA
// stages, besides the A0 / guide tile of the fine filter, everything its pixels' recombination reads: the half-res
// footprint (guide Gd, block means Ah, mid level Bh0; 18 x 10 texels, decoded once), the quarter-res footprint (guide
// CGd, coarse level C0; 10 x 6) and the per-block filter parameters (s0, c0, beta, kappa; 16 x 8). A thread's two pixels
// share the loads of 10 of their 3 x 3 windows' 18 texels, one row of the half-res footprint, the whole quarter-res
// footprint and the parameters: 52 16-byte loads of shared memory for two pixels instead of 80. With a pixel per
// thread the kernel was at 70% of the shared-memory bandwidth and 67% of the issue slots, and half of its CTAs waited for their
// tile's texels (so they did with two pixels per thread and a CTA per tile): 70 us at 1920 x 1080 and 271 at 3840 x 2160,
// now 66 and 246. Three CTAs per SM (80 registers, with spills) measured the same at 1920 x 1080 and 0.6 us more at
// 256 x 256.
constexpr int FF_W = 32, FF_H = 16, FF_NT = FF_W * FF_H / 2;
constexpr int FH_W = FF_W / 2 + 2, FH_H = FF_H / 2 + 2, FQ_W = FF_W / 4 + 2, FQ_H = FF_H / 4 + 2;
constexpr int FB_W = FF_W + 4, FB_H = FF_H + 2;  // A0 / key texels as copied, from column -2 on

// filt_x<1, 1, true> for the pixel at tile entry ti and the one below it. The taps run as pairs of one tap of each
// pixel, on the same texel where both windows hold it: (n.n)^128, weights and their squares as packed FP32x2, lane by lane
// the scalar arithmetic.
template <int SW, bool CHECK>
HD_INL void filt_v2(const float4 *sA, const float4 *sG, int ti, int qx, int qy, int w, int h, float s, float c,
                    float4 &out0, float4 &out1) {
  const float4 g0 = sG[ti], g1 = sG[ti + SW], a0 = sA[ti], a1 = sA[ti + SW];
  auto v = [&](int dx, int dy) { return sA[ti + dy * SW + dx].w; };
  auto z = [&](int dx, int dy) { return sG[ti + dy * SW + dx].w; };
  const float vm[2] = {v(-1, 0), v(-1, 1)}, vp[2] = {v(1, 0), v(1, 1)};
  const float gv0 = 0.0625f * (v(-1, -1) + v(1, -1) + vm[1] + vp[1]) + 0.125f * (v(0, -1) + vm[0] + vp[0] + a1.w) + 0.25f * a0.w;
  const float gv1 = 0.0625f * (vm[0] + vp[0] + v(-1, 2) + v(1, 2)) + 0.125f * (a0.w + vm[1] + vp[1] + v(0, 2)) + 0.25f * a1.w;
  const float lc0 = lum(a0), lc1 = lum(a1);
  auto slope = [](float zc, float zl, float zr, float zu, float zd) {
    const float gx = fminf(zr > 0.0f ? fabsf(zr - zc) : 1e9f, zl > 0.0f ? fabsf(zl - zc) : 1e9f);
    const float gy = fminf(zd > 0.0f ? fabsf(zd - zc) : 1e9f, zu > 0.0f ? fabsf(zu - zc) : 1e9f);
    return fminf(fmaxf(gx, gy), zc);
  };
  const float zg0 = slope(g0.w, z(-1, 0), z(1, 0), z(0, -1), g1.w), zg1 = slope(g1.w, z(-1, 1), z(1, 1), g0.w, z(0, 2));
  const float sl0 = LOG2E * s / (sqrtf(fmaxf(gv0, 1e-12f)) + 1e-6f), sl1 = LOG2E * s / (sqrtf(fmaxf(gv1, 1e-12f)) + 1e-6f);
  const float iz0[2] = {LOG2E / (zg0 * 1.0f + 1e-3f), LOG2E / (zg0 * 1.41421356237309515f + 1e-3f)};
  const float iz1[2] = {LOG2E / (zg1 * 1.0f + 1e-3f), LOG2E / (zg1 * 1.41421356237309515f + 1e-3f)};
  const float cw = 0.25f * c;
  float sw0 = cw, sw1 = cw;
  float x0 = a0.x * cw, y0 = a0.y * cw, b0 = a0.z * cw, v0 = a0.w * cw * cw;
  float x1 = a1.x * cw, y1 = a1.y * cw, b1 = a1.z * cw, v1 = a1.w * cw * cw;
  // one tap of each pixel: texel (p, cp) at offset (dx, dyp) of pixel 0, texel (q, cq) at offset (dx, dyq) of pixel 1
  auto tap = [&](float4 p, float4 cp, int dyp, float4 q, float4 cq, int dyq, int dx) {
    bool ok0 = p.w >= 0.0f, ok1 = q.w >= 0.0f;
    if (CHECK) {
      const int tx = qx + dx, t0 = qy + dyp, t1 = qy + 1 + dyq;
      const bool ix = tx >= 0 && tx < w;
      ok0 = ok0 && ix && t0 >= 0 && t0 < h;
      ok1 = ok1 && ix && t1 >= 0 && t1 < h;
    }
    float2 pp = make_float2(fmaxf(dot3(p, g0), 0.0f), fmaxf(dot3(q, g1), 0.0f));
#pragma unroll
    for (int i = 0; i < 7; i++) pp = __fmul2_rn(pp, pp);  // (n.n)^128
    const float e0 = fmaf(-fabsf(p.w - g0.w), iz0[dx != 0 && dyp != 0], fmaf(-sl0, fabsf(lum(cp) - lc0), lg_h(1, dx) + lg_h(1, dyp)));
    const float e1 = fmaf(-fabsf(q.w - g1.w), iz1[dx != 0 && dyq != 0], fmaf(-sl1, fabsf(lum(cq) - lc1), lg_h(1, dx) + lg_h(1, dyq)));
    const float2 wt = __fmul2_rn(pp, make_float2(ex2_approx(e0), ex2_approx(e1)));
    const float2 ww = __fmul2_rn(wt, wt);
    if (ok0) { sw0 += wt.x; x0 += wt.x * cp.x; y0 += wt.x * cp.y; b0 += wt.x * cp.z; v0 += ww.x * cp.w; }
    if (ok1) { sw1 += wt.y; x1 += wt.y * cq.x; y1 += wt.y * cq.y; b1 += wt.y * cq.z; v1 += ww.y * cq.w; }
  };
#pragma unroll
  for (int dx = -1; dx <= 1; dx++) tap(sG[ti - SW + dx], sA[ti - SW + dx], -1, sG[ti + 2 * SW + dx], sA[ti + 2 * SW + dx], 1, dx);
  tap(g1, a1, 1, g0, a0, -1, 0);
#pragma unroll
  for (int dx = -1; dx <= 1; dx += 2) {
    const float4 p0 = sG[ti + dx], c0 = sA[ti + dx], p1 = sG[ti + SW + dx], c1 = sA[ti + SW + dx];
    tap(p0, c0, 0, p0, c0, -1, dx);
    tap(p1, c1, 1, p1, c1, 0, dx);
  }
  out0 = make_float4(x0 / sw0, y0 / sw0, b0 / sw0, v0 / (sw0 * sw0));
  out1 = make_float4(x1 / sw1, y1 / sw1, b1 / sw1, v1 / (sw1 * sw1));
}

// The texels of one tile as they lie in memory (the copies' targets) and decoded (what the taps read).
struct FineSmem {
  static constexpr int SW = FF_W + 2, SH = FF_H + 2;
  static constexpr int NH = FH_W * FH_H, NQ = FQ_W * FQ_H, NP = (FF_W / 2) * (FF_H / 2);
  float4 a[SW * SH], g[SW * SH];                // A0 and the decoded key, apron 1
  float4 hg[NH], ha[NH], hb[NH], qg[NQ], qc[NQ], par[NP];
  alignas(16) uint2 ra[FB_W * FB_H], rk[FB_W * FB_H];  // A0 / key from column bx - 2
  float4 rhg[NH], rqg[NQ];
  uint2 rha[NH], rhb[NH], rqc[NQ], rp0[NP], rp1[NP], rp2[NP], mat[2][FF_NT], emi[2][FF_NT];
};

// Starts the copies of tile (bx, by)'s texels into the raw half of S and commits them as one group.
HD_INL void fine_issue(const HushFrame &f, FineSmem &S, int li, int bx, int by) {
  constexpr int SW = FineSmem::SW, NH = FineSmem::NH, NQ = FineSmem::NQ, NP = FineSmem::NP;
  const bool interior = bx - 2 >= 0 && by - 1 >= 0 && bx + FF_W + 2 <= f.W && by + FF_H + 1 <= f.H;
  if (interior && !(f.W & 1)) {  // even rows and columns of 8-byte texels: 16-byte copies of texel pairs
    for (int i = li; i < FB_W / 2 * FB_H; i += FF_NT) {
      const int r = i / (FB_W / 2), c = 2 * (i % (FB_W / 2)), q = (by - 1 + r) * f.W + bx - 2 + c;
      cp_async16(S.ra + r * FB_W + c, f.A0 + q);
      cp_async16(S.rk + r * FB_W + c, f.key + q);
    }
  } else {
    for (int i = li; i < SW * FineSmem::SH; i += FF_NT) {
      const int r = i / SW, c = i % SW;
      const int q = clampi(by - 1 + r, 0, f.H - 1) * f.W + clampi(bx - 1 + c, 0, f.W - 1);
      cp_async8(S.ra + r * FB_W + c + 1, f.A0 + q);
      cp_async8(S.rk + r * FB_W + c + 1, f.key + q);
    }
  }
  if (li < NH) {
    const int q = clampi(by / 2 - 1 + li / FH_W, 0, f.H2 - 1) * f.W2 + clampi(bx / 2 - 1 + li % FH_W, 0, f.W2 - 1);
    cp_async16(S.rhg + li, f.Gd + q);
    cp_async8(S.rha + li, f.Ah + q);
    cp_async8(S.rhb + li, f.Bh0 + q);
  } else if (li < NH + NQ) {
    const int i = li - NH;
    const int r = clampi(by / 4 - 1 + i / FQ_W, 0, f.H4 - 1) * f.W4 + clampi(bx / 4 - 1 + i % FQ_W, 0, f.W4 - 1);
    cp_async16(S.rqg + i, f.CGd + r);
    cp_async8(S.rqc + i, f.C0 + r);
  }
  if (li >= FF_NT - NP) {
    const int i = li - (FF_NT - NP);
    const int hq = clampi(by / 2 + i / (FF_W / 2), 0, f.H2 - 1) * f.W2 + clampi(bx / 2 + i % (FF_W / 2), 0, f.W2 - 1);
    cp_async8(S.rp0 + i, f.par0 + hq);
    cp_async8(S.rp1 + i, f.par1 + hq);
    cp_async8(S.rp2 + i, f.par2 + hq);
  }
  const int px = min(bx + li % FF_W, f.W - 1), py = by + 2 * (li / FF_W);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int y = min(py + k, f.H - 1);
    cp_async8(&S.mat[k][li], f.mat + y * f.p_mat + px);
    cp_async8(&S.emi[k][li], f.emi + y * f.p_emi + px);
  }
  cp_async_commit();
}

// The two pixels of thread li of tile (bx, by) from the decoded half of S.
HD_INL void fine_pixels(const HushFrame &f, const FineSmem &S, int li, int bx, int by, const uint2 *mat_r,
                        const uint2 *emi_r) {
  constexpr int AP = 1, SW = FineSmem::SW;
  const bool interior = bx - 1 >= 0 && by - 1 >= 0 && bx + FF_W + 1 <= f.W && by + FF_H + 1 <= f.H;
  const int px = bx + li % FF_W, py = by + 2 * (li / FF_W);
  const bool in0 = px < f.W && py < f.H, in1 = in0 && py + 1 < f.H;
  if (!in0) return;
  const int hx0 = bx / 2 - 1, hy0 = by / 2 - 1, qx0 = bx / 4 - 1, qy0 = by / 4 - 1;
  const int ti = (py - by + AP) * SW + px - bx + AP;
  const float4 gp0 = S.g[ti], gp1 = S.g[ti + SW];
  const bool live0 = !(gp0.w < 0.0f), live1 = in1 && !(gp1.w < 0.0f);
  const int o = py * f.W + px;
  auto sky = [&](int oo, uint2 er) {
    const float4 emi = h4_to_f4(er);
    sth(f.hist, oo, make_float4(0.f, 0.f, 0.f, 0.f));
    sth(f.X, oo, make_float4(emi.x, emi.y, emi.z, 0.f));
  };
  if (!live0) sky(o, emi_r[0]);
  if (in1 && !live1) sky(o + f.W, emi_r[1]);
  if (!live0 && !live1) return;
  const float4 pr = S.par[((py - by) >> 1) * (FF_W / 2) + ((px - bx) >> 1)];
  float4 A0v, A1v;
  if (interior) filt_v2<SW, false>(S.a, S.g, ti, px, py, f.W, f.H, pr.x, pr.y, A0v, A1v);
  else filt_v2<SW, true>(S.a, S.g, ti, px, py, f.W, f.H, pr.x, pr.y, A0v, A1v);
  if (live0) sth(f.hist, o, A0v);
  if (live1) sth(f.hist, o + f.W, A1v);
  // recombination (hush.js:580-620) of both pixels with the half-res block means (Ah) and decoded guides (Gd, CGd)
  const float3 f0 = make_float3(qf16(A0v.x), qf16(A0v.y), qf16(A0v.z)), f1 = make_float3(qf16(A1v.x), qf16(A1v.y), qf16(A1v.z));
  const float2 rzl = make_float2(LOG2E / (0.05f * gp0.w + 1e-3f), LOG2E / (0.05f * gp1.w + 1e-3f));
  // jbw() of one tap of each pixel: the (n.n)^8 and weight products as packed FP32x2
  auto jbw2 = [&](float2 wb, float4 n0, float4 n1) {
    const float2 d = make_float2(fmaxf(dot3(n0, gp0), 0.0f), fmaxf(dot3(n1, gp1), 0.0f));
    const float2 d2 = __fmul2_rn(d, d), d4 = __fmul2_rn(d2, d2);
    const float2 e = make_float2(ex2_approx(-fabsf(n0.w - gp0.w) * rzl.x), ex2_approx(-fabsf(n1.w - gp1.w) * rzl.y));
    return __fmul2_rn(__fmul2_rn(__fmul2_rn(wb, e), d4), d4);
  };
  // the bilinear phase: py is even, so pixel 0 lies 3/4 and pixel 1 1/4 of a half-res row below its base row (rows
  // r, r + 1 and r + 1, r + 2), and both share their quarter-res rows
  const float hposx = ((float)px + 0.5f) / 2.0f - 0.5f, hbx = floorf(hposx), hfx = hposx - hbx;
  const float cposx = ((float)px + 0.5f) / 4.0f - 0.5f, cbx = floorf(cposx), cfx = cposx - cbx;
  const float cpos0 = ((float)py + 0.5f) / 4.0f - 0.5f, cpos1 = ((float)py + 1.5f) / 4.0f - 0.5f, cby = floorf(cpos0);
  struct Sum { float bx, by, bz, ax, ay, az, w; };
  Sum u0 = {}, u1 = {};
  auto add = [](Sum &u, float w, float4 m, float4 a) {
    u.w += w;
    u.bx += w * m.x; u.by += w * m.y; u.bz += w * m.z;
    u.ax += w * a.x; u.ay += w * a.y; u.az += w * a.z;
  };
  const int hr = (py >> 1) - 1, hc = (int)hbx;
#pragma unroll
  for (int j = 0; j < 2; j++) {  // columns: rows r of pixel 0 and r + 2 of pixel 1 as one pair, row r + 1 for both
    const int t = (hr - hy0) * FH_W + hc + j - hx0;
    const float wx = j ? hfx : 1.0f - hfx;
    const bool ix = hc + j >= 0 && hc + j < f.W2;
    const float4 ga = S.hg[t], gm = S.hg[t + FH_W], gb = S.hg[t + 2 * FH_W];
    const float2 wo = jbw2(make_float2(wx * 0.25f, wx * 0.25f), ga, gb);
    const float2 wm = jbw2(make_float2(wx * 0.75f, wx * 0.75f), gm, gm);
    if (ix && hr >= 0 && ga.w >= 0.0f) add(u0, wo.x, S.hb[t], S.ha[t]);
    if (ix && gm.w >= 0.0f) {
      const float4 m = S.hb[t + FH_W], a = S.ha[t + FH_W];
      add(u0, wm.x, m, a);
      add(u1, wm.y, m, a);
    }
    if (ix && hr + 2 < f.H2 && gb.w >= 0.0f) add(u1, wo.y, S.hb[t + 2 * FH_W], S.ha[t + 2 * FH_W]);
  }
  float3 i0 = f0, i1 = f1;
  auto mix = [&](float3 fv, const Sum &u) {
    if (!(u.w > 1e-4f)) return fv;
    return make_float3(u.bx / u.w + pr.w * (fv.x - u.ax / u.w), u.by / u.w + pr.w * (fv.y - u.ay / u.w),
                       u.bz / u.w + pr.w * (fv.z - u.az / u.w));
  };
  i0 = mix(f0, u0);
  i1 = mix(f1, u1);
  float c0x = 0.f, c0y = 0.f, c0z = 0.f, w0 = 0.f, c1x = 0.f, c1y = 0.f, c1z = 0.f, w1 = 0.f;
  const float cf0 = cpos0 - cby, cf1 = cpos1 - cby;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int ry = (int)cby + (j >> 1), rx = (int)cbx + (j & 1);
    const int t = (ry - qy0) * FQ_W + rx - qx0;
    const float4 g = S.qg[t];
    const float wx = (j & 1) ? cfx : 1.0f - cfx;
    const float2 w = jbw2(make_float2(wx * ((j >> 1) ? cf0 : 1.0f - cf0), wx * ((j >> 1) ? cf1 : 1.0f - cf1)), g, g);
    if (ry >= 0 && ry < f.H4 && rx >= 0 && rx < f.W4 && g.w >= 0.0f) {
      const float4 c = S.qc[t];
      w0 += w.x; c0x += w.x * c.x; c0y += w.x * c.y; c0z += w.x * c.z;
      w1 += w.y; c1x += w.y * c.x; c1y += w.y * c.y; c1z += w.y * c.z;
    }
  }
  auto finish = [&](int oo, float3 i, float cx, float cy, float cz, float w, uint2 mr, uint2 er) {
    const float4 alb = h4_to_f4(mr), emi = h4_to_f4(er);
    float3 up = i;
    if (w > 1e-4f) up = make_float3(cx / w, cy / w, cz / w);
    i = make_float3(i.x + (up.x - i.x) * pr.z, i.y + (up.y - i.y) * pr.z, i.z + (up.z - i.z) * pr.z);
    sth(f.X, oo, make_float4(i.x * alb.x + emi.x, i.y * alb.y + emi.y, i.z * alb.z + emi.z, 0.0f));
  };
  if (live0) finish(o, i0, c0x, c0y, c0z, w0, mat_r[0], emi_r[0]);
  if (live1) finish(o + f.W, i1, c1x, c1y, c1z, w1, mat_r[1], emi_r[1]);
}

// Each CTA walks over tiles (blockIdx.x, + gridDim.x, ...): the next tile's texels fly into the raw buffers while this
// tile's pixels are filtered, so only a CTA's first tile waits for memory.
__global__ void __launch_bounds__(FF_NT, 2) k_fine_final_fused(const __grid_constant__ HushFrame f, int tiles_x, int tiles) {
  constexpr int AP = 1, SW = FineSmem::SW, SH = FineSmem::SH;
  constexpr int NH = FineSmem::NH, NQ = FineSmem::NQ, NP = FineSmem::NP;
  static_assert(NH + NQ <= FF_NT && NP <= FF_NT, "one footprint texel and one block's parameters per thread");
  extern __shared__ __align__(16) unsigned char ff_smem[];
  FineSmem &S = *reinterpret_cast<FineSmem *>(ff_smem);
  const int li = threadIdx.x;
  int tile = blockIdx.x;
  fine_issue(f, S, li, tile % tiles_x * FF_W, tile / tiles_x * FF_H);
  for (; tile < tiles; tile += gridDim.x) {
    const int bx = tile % tiles_x * FF_W, by = tile / tiles_x * FF_H;
    cp_async_wait<0>();
    __syncthreads();  // the tile's texels are here, and the previous tile's taps are done with the decoded half
    for (int i = li; i < SW * SH; i += FF_NT) {
      const int t = (i / SW) * FB_W + i % SW + 1;
      S.a[i] = h4_to_f4(S.ra[t]);
      const float4 k = h4_to_f4(S.rk[t]);
      float4 g = oct_dec(k.x, k.y);
      g.w = k.z;
      S.g[i] = g;
    }
    if (li < NH) {
      S.hg[li] = S.rhg[li];
      S.ha[li] = h4_to_f4(S.rha[li]);
      S.hb[li] = h4_to_f4(S.rhb[li]);
    } else if (li < NH + NQ) {
      S.qg[li - NH] = S.rqg[li - NH];
      S.qc[li - NH] = h4_to_f4(S.rqc[li - NH]);
    }
    if (li >= FF_NT - NP) {
      const int i = li - (FF_NT - NP);
      const float4 p0 = h4_to_f4(S.rp0[i]);
      S.par[i] = make_float4(h4_to_f4(S.rp1[i]).x, h4_to_f4(S.rp2[i]).x, p0.z, p0.w);  // s0, c0, beta, kappa
    }
    const uint2 mat_r[2] = {S.mat[0][li], S.mat[1][li]}, emi_r[2] = {S.emi[0][li], S.emi[1][li]};
    __syncthreads();
    const int next = tile + gridDim.x;
    if (next < tiles) fine_issue(f, S, li, next % tiles_x * FF_W, next / tiles_x * FF_H);
    fine_pixels(f, S, li, bx, by, mat_r, emi_r);
  }
}

// TAA (hush.js:639-677) with a 32 x 8 tile. The pixel's motion, colour and the four history texels of its bilinear
// footprint are loaded before the tile barrier, so the motion -> history dependency overlaps the tile loads. The
// YCoCg tile is held as (Y, Co) pairs beside a Cg plane, so the 3x3 statistics, the history sum, the clip bounds and
// the blend run (Y, Co) as one packed FP32x2 operation and Cg as a scalar one, lane by lane the same arithmetic
// (40 registers: six CTAs per SM).
template <bool NEXT>  // launched as FINE_FINAL's programmatic successor
__global__ void __launch_bounds__(FT_W *FT_H) k_taa_fused(const __grid_constant__ HushFrame f) {
  if constexpr (NEXT) pass_begin(true);
  constexpr int SW = FT_W + 2, SH = FT_H + 2, NT = FT_W * FT_H, NIT = (SW * SH + NT - 1) / NT;
  __shared__ float2 sXY[SW * SH];
  __shared__ float sXZ[SW * SH];
  const int li = threadIdx.x;
  const int tx = li % FT_W, ty = li / FT_W;
  const int px = blockIdx.x * FT_W + tx, py = blockIdx.y * FT_H + ty;
  const int cpx = min(px, f.W - 1), cpy = min(py, f.H - 1);
  const uint2 mvr = __ldg(f.mv + cpy * f.p_mv + cpx);
  const int ox = blockIdx.x * FT_W - 1, oy = blockIdx.y * FT_H - 1;
  uint2 tl[NIT];
#pragma unroll
  for (int it = 0; it < NIT; it++) {
    const int i = min(li + it * NT, SW * SH - 1);
    tl[it] = ld_pass(f.X + clampi(oy + i / SW, 0, f.H - 1) * f.W + clampi(ox + i % SW, 0, f.W - 1));
  }
  const uint2 xr = ld_pass(f.X + cpy * f.W + cpx);
  // the history footprint (clamped loads; used only when the reprojected position lies inside the image)
  const float4 mv = h4_to_f4(mvr);
  const float szx = (float)f.W, szy = (float)f.H;
  const float uvx = ((float)px + 0.5f + mv.x) / szx, uvy = ((float)py + 0.5f + mv.y) / szy;
  const float ppx = uvx * szx - 0.5f, ppy = uvy * szy - 0.5f;
  const float bxf = floorf(ppx), byf = floorf(ppy);
  const int ibx = (int)bxf, iby = (int)byf;
  uint2 hq[4];
#pragma unroll
  for (int j = 0; j < 4; j++)
    hq[j] = __ldg(f.taa_prev + clampi(iby + (j >> 1), 0, f.H - 1) * f.W + clampi(ibx + (j & 1), 0, f.W - 1));
#pragma unroll
  for (int it = 0; it < NIT; it++) {
    const int i = li + it * NT;
    if (i >= SW * SH) continue;
    const float4 x = h4_to_f4(tl[it]);
    const float3 y = to_ycocg(tmap(make_float3(x.x, x.y, x.z)));
    sXY[i] = make_float2(y.x, y.y);
    sXZ[i] = y.z;
  }
  __syncthreads();
  if (px >= f.W || py >= f.H) return;
  const int o = py * f.W + px;
  const float4 x = h4_to_f4(xr);
  const float3 cur = tmap(make_float3(x.x, x.y, x.z));
  float3 r;
  if (f.reset) {
    r = itmap(cur);
  } else {
    const int ti = (ty + 1) * SW + tx + 1;
    auto c9 = [&](int j) {
      const int t = ti + (j / 3 - 1) * SW + (j % 3 - 1);
      const float2 a = sXY[t];
      return make_float4(a.x, a.y, sXZ[t], 0.0f);
    };
    float2 s2 = f2(0.f, 0.f);
    float s1 = 0.f;
#pragma unroll
    for (int j = 0; j < 9; j++) {
      const float4 c = c9(j);
      s2 = add2(s2, lo2(c));
      s1 += c.z;
    }
    const float m1x = s2.x / 9.0f, m1y = s2.y / 9.0f, m1z = s1 / 9.0f;
    const float2 nm = f2(-m1x, -m1y);
    float2 v2 = f2(0.f, 0.f);
    float v1 = 0.f;
#pragma unroll
    for (int j = 0; j < 9; j++) {
      const float4 c = c9(j);
      const float2 d = add2(lo2(c), nm);
      const float dz = c.z - m1z;
      v2 = fma2(d, d, v2);
      v1 += dz * dz;
    }
    const float sdx = sqrtf(fmaxf(v2.x / 9.0f, 1e-12f)), sdy = sqrtf(fmaxf(v2.y / 9.0f, 1e-12f)),
                sdz = sqrtf(fmaxf(v1 / 9.0f, 1e-12f));
    float3 res = cur;
    if (uvx >= 0.0f && uvy >= 0.0f && uvx <= 1.0f && uvy <= 1.0f) {
      const float fx = ppx - bxf, fy = ppy - byf;
      float2 h2 = f2(0.f, 0.f);
      float h1 = 0.f;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int oxj = j & 1, oyj = j >> 1;
        const float wb = (oxj == 1 ? fx : 1.0f - fx) * (oyj == 1 ? fy : 1.0f - fy);
        const float4 t = h4_to_f4(hq[j]);
        h2 = fma2(bc2(wb), lo2(t), h2);
        h1 += wb * t.z;
      }
      float3 hh = to_ycocg(tmap(make_float3(h2.x, h2.y, h1)));
      const float2 sd2 = f2(sdx, sdy), m12 = f2(m1x, m1y);
      const float2 lo = fma2(bc2(-1.25f), sd2, m12), hi = fma2(bc2(1.25f), sd2, m12);
      hh.x = fminf(fmaxf(hh.x, lo.x), hi.x);
      hh.y = fminf(fmaxf(hh.y, lo.y), hi.y);
      hh.z = fminf(fmaxf(hh.z, m1z - 1.25f * sdz), m1z + 1.25f * sdz);
      const float3 hr = from_ycocg(hh);
      const float2 hr2 = f2(hr.x, hr.y);
      const float2 b2 = fma2(add2(f2(cur.x, cur.y), f2(-hr.x, -hr.y)), bc2(0.1f), hr2);
      res = make_float3(b2.x, b2.y, hr.z + (cur.z - hr.z) * 0.1f);
    }
    r = itmap(res);
  }
  sth(f.taa, o, make_float4(r.x, r.y, r.z, 1.0f));
}

// ------------------------------------------------------------------------------------------------ launchers
static const char *STAGE_LABELS[6] = {"temporal+mlp", "mid1+coarse1", "mid2+coarse2", "mid3", "fine+final", "taa"};
int fused_stage_count() { return 6; }
const char *fused_stage_label(int s) { return (s >= 0 && s < 6) ? STAGE_LABELS[s] : "?"; }

// The half stages' tensor maps for the frame's buffers, encoded when the buffers or sizes change (per host thread).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

static const HalfMaps &half_maps(const HushFrame &f) {
  struct Cache {
    const void *gd = nullptr, *b0 = nullptr, *b1 = nullptr, *ah = nullptr, *cgd = nullptr, *c1 = nullptr;
    int w = -1, h = -1;
    HalfMaps m{};
  };
  static thread_local Cache c;
  if (c.gd == f.Gd && c.b0 == f.Bh0 && c.b1 == f.Bh1 && c.ah == f.Ah && c.cgd == f.CGd && c.c1 == f.C1 &&
      c.w == f.W2 && c.h == f.H2)
    return c.m;
  c.gd = f.Gd; c.b0 = f.Bh0; c.b1 = f.Bh1; c.ah = f.Ah; c.cgd = f.CGd; c.c1 = f.C1; c.w = f.W2; c.h = f.H2;
  std::memset(&c.m, 0, sizeof(c.m));
  const PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (enc && !(f.W4 & 1) && f.W4 >= HT_W + 8 && f.H4 >= HT_H + 8) {  // coarse2's quarter-resolution maps
    const cuuint32_t one3[3] = {1, 1, 1};
    const cuuint64_t gdim[3] = {4, (cuuint64_t)f.W4, (cuuint64_t)f.H4};
    const cuuint64_t gstr[2] = {16, (cuuint64_t)f.W4 * 16};
    const cuuint32_t gbox[3] = {4, (cuuint32_t)(HT_W + 8), (cuuint32_t)(HT_H + 8)};
    const cuuint64_t ldim[2] = {(cuuint64_t)f.W4, (cuuint64_t)f.H4};
    const cuuint64_t lstr[1] = {(cuuint64_t)f.W4 * 8};
    const cuuint32_t lbox[2] = {(cuuint32_t)(HT_W + 8), (cuuint32_t)(HT_H + 8)};
    c.m.qok = enc(&c.m.cgd, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void *)f.CGd, gdim, gstr, gbox, one3,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS &&
              enc(&c.m.c1, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, (void *)f.C1, ldim, lstr, lbox, one3,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
                  ? 1
                  : 0;
  }
  // the 8-byte level map needs a row pitch that is a multiple of 16 bytes
  if (!enc || (f.W2 & 1) || f.W2 < HT_W + 8 || f.H2 < HT_H + 8) return c.m;
  const cuuint32_t one[3] = {1, 1, 1};
  auto gd = [&](CUtensorMap *m, int ap) {
    const cuuint64_t dim[3] = {4, (cuuint64_t)f.W2, (cuuint64_t)f.H2};
    const cuuint64_t str[2] = {16, (cuuint64_t)f.W2 * 16};
    const cuuint32_t box[3] = {4, (cuuint32_t)(HT_W + 2 * ap), (cuuint32_t)(HT_H + 2 * ap)};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void *)f.Gd, dim, str, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  auto lv = [&](CUtensorMap *m, const uint2 *p, int ap) {
    const cuuint64_t dim[2] = {(cuuint64_t)f.W2, (cuuint64_t)f.H2};
    const cuuint64_t str[1] = {(cuuint64_t)f.W2 * 8};
    const cuuint32_t box[2] = {(cuuint32_t)(HT_W + 2 * ap), (cuuint32_t)(HT_H + 2 * ap)};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, (void *)p, dim, str, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  bool ok = gd(&c.m.gd2, 2) == CUDA_SUCCESS && gd(&c.m.gd4, 4) == CUDA_SUCCESS && gd(&c.m.gd1, 1) == CUDA_SUCCESS &&
            lv(&c.m.bh0, f.Bh0, 2) == CUDA_SUCCESS && lv(&c.m.bh1, f.Bh1, 4) == CUDA_SUCCESS;
  {  // Ah: box (16 + 4) x (8 + 2) from an even x
    const cuuint64_t dim[2] = {(cuuint64_t)f.W2, (cuuint64_t)f.H2};
    const cuuint64_t str[1] = {(cuuint64_t)f.W2 * 8};
    const cuuint32_t box[2] = {(cuuint32_t)(HT_W + 4), (cuuint32_t)(HT_H + 2)};
    ok = ok && enc(&c.m.ah, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, (void *)f.Ah, dim, str, box, one,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
  c.m.ok = ok ? 1 : 0;
  return c.m;
}

// stage 0's forms: by MODE at 16 rows, then MODE 0 and MODE 3 at 8 rows
static void (*const KB_KERN[6])(HushFrame, MlpConst, const uint4 *) = {
    k_temporal_block<0, KB_TH>, k_temporal_block<1, KB_TH>,     k_temporal_block<2, KB_TH>,
    k_temporal_block<3, KB_TH>, k_temporal_block<0, KB_TH / 2>, k_temporal_block<3, KB_TH / 2>};

// chained: the kernels that directly follow another one of the frame on their stream (mid2, mid3, coarse2, TAA) are set up while
// that one runs: directly launched frames 256x256 43.2 -> 39.7 us, 640x360 60.5 -> 55.0, 1283x717 144.5 -> 142.0.
cudaError_t launch_fused_stage(int stage, int part, const HushFrame &f, const MlpConst &mc, int mlp_mode,
                               const void *mlp_tc, bool chained, cudaStream_t st) {
  const int hx = (f.W2 + HT_W - 1) / HT_W, hy = (f.H2 + HT_H - 1) / HT_H;
  const int qx = (f.W4 + HT_W - 1) / HT_W, qy = (f.H4 + HT_H - 1) / HT_H;
  const int hpx = (f.W2 + MP_W - 1) / MP_W;  // two-pixel mid tiles per row
  const bool plain = !chained;
  switch (stage) {
    case 0: {
      // blob: the tensor-core forms' bf16 hi / lo operands and f16 operands; mc: the weights as a kernel parameter
      const uint4 *blob = (const uint4 *)mlp_tc;
      int dev = 0;
      cudaGetDevice(&dev);
      if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
      const int gx = (f.W + KB_TW - 1) / KB_TW;
      const int m = mlp_mode & 3;
      const bool tc = m == 1 || m == 2;
      const bool half = !tc && gx * ((f.H + KB_TH - 1) / KB_TH) <= KB_HALF_CTAS;
      const int th = half ? KB_TH / 2 : KB_TH;
      // most forms need more than 48 KB of dynamic shared memory: opt in once per device and form
      static bool opted[6][64] = {};
      const int ki = !half ? m : m == 0 ? 4 : 5;
      const int smem = tc ? (int)sizeof(KbTcSmem) : half ? (int)sizeof(KbSmem<KB_TH / 2>) : (int)sizeof(KbSmem<KB_TH>);
      if (!opted[ki][dev]) {
        const cudaError_t e = cudaFuncSetAttribute(KB_KERN[ki], cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        opted[ki][dev] = true;
      }
      const uint4 *b = m == 1 ? blob + MLP_BLOB_BF16 / 16 : m == 2 ? blob + MLP_BLOB_F16 / 16 : blob;
      KB_KERN[ki]<<<dim3(gx, (f.H + th - 1) / th), KB_TW / 4 * th, smem, st>>>(f, mc, b);
      break;
    }
    // stages 1 and 2: the mid tiles and the coarse tiles are separate kernels (each with its own register count);
    // both parts run them one after the other on `st`
    case 1:
      if (part != HP_COARSE)
        k_half_stage<1, HP_MID><<<hx * hy, HT_W * HT_H, 0, st>>>(f, hx, hx * hy, qx, half_maps(f));
      if (part != HP_MID)
        k_half_stage<1, HP_COARSE><<<qx * qy, HT_W * HT_H, 0, st>>>(f, hx, hx * hy, qx, half_maps(f));
      break;
    case 2: {
      constexpr int smc = 2 * (HT_W + 8) * (HT_H + 8) * 16;  // coarse2's two float4 tiles
      cudaError_t e = cudaSuccess;
      if (part != HP_COARSE)
        e = launch_chained(plain ? k_half_pair<2, HP_MID, false> : k_half_pair<2, HP_MID, true>, dim3(hpx * hy),
                           dim3(HT_W * HT_H), (size_t)mid_pair_smem<2>(), plain, st, f, hpx, hpx * hy, qx, half_maps(f));
      if (part != HP_MID && e == cudaSuccess)
        e = launch_chained(plain ? k_half_pair<2, HP_COARSE, false> : k_half_pair<2, HP_COARSE, true>, dim3(qx * qy),
                           dim3(HT_W * HT_H), (size_t)smc, plain, st, f, hpx, hpx * hy, qx, half_maps(f));
      if (e != cudaSuccess) return e;
      break;
    }
    case 3:
      if (part == HP_COARSE) break;  // no coarse level in stage 3
      if (const cudaError_t e = launch_chained(plain ? k_half_pair<3, HP_MID, false> : k_half_pair<3, HP_MID, true>,
                                               dim3(hpx * hy), dim3(HT_W * HT_H), (size_t)mid_pair_smem<4>(), plain, st, f, hpx,
                                               hpx * hy, qx, half_maps(f)))
        return e;
      break;
    case 4: {
      const int tx = (f.W + FF_W - 1) / FF_W, tiles = tx * ((f.H + FF_H - 1) / FF_H);
      int dev = 0;
      cudaGetDevice(&dev);
      if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
      static int sms[64] = {};  // and, once it is known, the shared-memory opt-in is done
      if (!sms[dev]) {
        int n = 0;
        cudaError_t e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess)
          e = cudaFuncSetAttribute(k_fine_final_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FineSmem));
        if (e != cudaSuccess) return e;
        sms[dev] = n;
      }
      k_fine_final_fused<<<std::min(tiles, 2 * sms[dev]), FF_NT, sizeof(FineSmem), st>>>(f, tx, tiles);
      break;
    }
    case 5:
      if (const cudaError_t e = launch_chained(plain ? k_taa_fused<false> : k_taa_fused<true>,
                                               dim3((f.W + FT_W - 1) / FT_W, (f.H + FT_H - 1) / FT_H), dim3(FT_W * FT_H), 0,
                                               plain, st, f))
        return e;
      break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

size_t fused_scratch_bytes(int, int) { return 0; }

int fused_kernel_param_count(const void *func) {
  for (auto *k : KB_KERN)
    if (func == (const void *)k) return 3;  // (f, wp, blob)
  const void *half[5] = {(const void *)k_half_stage<1, HP_MID>, (const void *)k_half_stage<1, HP_COARSE>,
                         (const void *)k_half_pair<2, HP_MID, false>, (const void *)k_half_pair<2, HP_COARSE, false>,
                         (const void *)k_half_pair<3, HP_MID, false>};
  for (const void *k : half)
    if (func == k) return 5;  // (f, nAx, nA, nBx, M)
  if (func == (const void *)k_fine_final_fused) return 3;  // (f, tiles_x, tiles)
  if (func == (const void *)k_taa_fused<false>) return 1;          // (f)
  return 0;
}

}  // namespace hush
