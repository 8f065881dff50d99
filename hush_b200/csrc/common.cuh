// Device helpers shared by the Hush kernels: f16 texel I/O and the reference's COMMON / TILE_FNS functions
// (src/denoise/hush.js:28-49, 67-74, 98-108).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define HD_INL __device__ __forceinline__

namespace hush {

// ------------------------------------------------------------------------------------------------ texels
// A texel of an rgba16float image is 8 bytes (uint2); a packed-feature texel (rgba32uint) is 16 bytes (uint4).
HD_INL float4 h4_to_f4(uint2 t) {
  __half2 a = *reinterpret_cast<__half2 *>(&t.x), b = *reinterpret_cast<__half2 *>(&t.y);
  float2 fa = __half22float2(a), fb = __half22float2(b);
  return make_float4(fa.x, fa.y, fb.x, fb.y);
}
// f32 -> f16 rounded toward zero: the storage-write rounding the reference models (hush.js:98).
HD_INL uint16_t f2h(float x) { return __half_as_ushort(__float2half_rz(x)); }
// Two values in one conversion (cvt.rz.f16x2.f32 puts its first source in the upper half): a in bits 0-15.
HD_INL uint32_t pack2(float a, float b) {
  uint32_t r;
  asm("cvt.rz.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
HD_INL uint2 f4_to_h4(float4 v) { return make_uint2(pack2(v.x, v.y), pack2(v.z, v.w)); }
HD_INL float2 unpack2(uint32_t u) {
  __half2 h = *reinterpret_cast<__half2 *>(&u);
  return __half22float2(h);
}
HD_INL float4 ldh(const uint2 *__restrict__ p, int idx) { return h4_to_f4(__ldg(p + idx)); }
// A texel that an earlier kernel of a programmatic chain (pass_begin(), below) writes: by an ordinary load. __ldg's
// ld.global.nc is for memory that nobody writes while the kernel is resident, and a kernel of such a chain is resident
// before its predecessor has written, so that no wait orders it.
template <class T>
HD_INL T ld_pass(const T *p) { return *p; }
HD_INL float4 ldh_pass(const uint2 *p, int idx) { return h4_to_f4(ld_pass(p + idx)); }
HD_INL void sth(uint2 *__restrict__ p, int idx, float4 v) { p[idx] = f4_to_h4(v); }
HD_INL float4 quant4(float4 v) {  // value after an rgba16float round trip
  return h4_to_f4(f4_to_h4(v));
}
HD_INL float quant1(float v) { return __half2float(__float2half_rz(v)); }

// One texel copied from global to shared memory without passing through registers; a thread's copies are committed as
// groups and waited for by the number of later groups that may still fly.
HD_INL void cp_async8(const uint2 *dst_smem, const uint2 *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src)
               : "memory");
}
HD_INL void cp_async16(const void *dst_smem, const void *src) {  // both 16-byte aligned
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src)
               : "memory");
}
HD_INL void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
HD_INL void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// qf16 (hush.js:68, 99): clamp to the f16 range, drop the low 13 mantissa bits.
HD_INL float qf16(float x) {
  return __uint_as_float(__float_as_uint(fminf(fmaxf(x, -65504.0f), 65504.0f)) & 0xffffe000u);
}
// pk (hush.js:101): pack2x16float of qf16 values.
HD_INL uint32_t pk(float a, float b) { return pack2(qf16(a), qf16(b)); }

// ------------------------------------------------------------------------------------------------ COMMON
HD_INL float lum3(float r, float g, float b) { return r * 0.2126f + g * 0.7152f + b * 0.0722f; }
HD_INL float lum(float4 c) { return lum3(c.x, c.y, c.z); }
HD_INL float dot3(float4 a, float4 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

HD_INL float2 oct_enc(float nx, float ny, float nz) {
  float den = fmaxf(fabsf(nx) + fabsf(ny) + fabsf(nz), 1e-20f);
  float vx = nx / den, vy = ny / den, vz = nz / den;
  float sx = vx >= 0.0f ? 1.0f : -1.0f, sy = vy >= 0.0f ? 1.0f : -1.0f;
  if (vz < 0.0f) return make_float2((1.0f - fabsf(vy)) * sx, (1.0f - fabsf(vx)) * sy);
  return make_float2(vx, vy);
}
// Decoded normal in xyz; w is left for the caller (depth).
HD_INL float4 oct_dec(float ex, float ey) {
  float vx = ex, vy = ey, vz = 1.0f - fabsf(ex) - fabsf(ey);
  float t = fmaxf(-vz, 0.0f);
  vx += vx >= 0.0f ? -t : t;
  vy += vy >= 0.0f ? -t : t;
  float l = fmaxf(sqrtf(vx * vx + vy * vy + vz * vz), 1e-20f);
  return make_float4(vx / l, vy / l, vz / l, 0.0f);
}
HD_INL float log1p_w(float x) { return logf(1.0f + x); }  // hush.js:47: log(1 + x)
HD_INL float pow128(float x) {
  float x2 = x * x, x4 = x2 * x2, x8 = x4 * x4, x16 = x8 * x8, x32 = x16 * x16, x64 = x32 * x32;
  return x64 * x64;
}
HD_INL float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }
HD_INL int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

constexpr float HMAX = 32.0f;
constexpr float COARSE_S = 0.25f;  // hush.js:26
constexpr int N_FEAT = 20;
constexpr int N_OUT = 12;

// A chain of short kernels, each launched as the next one's programmatic predecessor: a kernel's CTAs are set up while the one
// before runs, and pass_begin(), the first thing that every kernel of the chain but the first does, waits for the end of that
// one (which has waited for the end of its own predecessor, and so on). The first kernel waits for whatever the stream did
// before, as any kernel; so does the first kernel after the chain. What a kernel of the chain writes is read in it by ld_pass()
// and ldh_pass() and never through a `const __restrict__` parameter; the caller's inputs and former frames' images, which no
// kernel of the chain writes, may take the read-only path.
__device__ __forceinline__ void pass_begin(bool last = false) {
  if (!last) asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
inline cudaError_t launch_chained(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, bool first, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = first ? 0 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
  if (e != cudaSuccess) cudaGetLastError();  // it is returned, not left for the next call that asks
  return e;
}

}  // namespace hush
