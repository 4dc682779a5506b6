// Device-side building blocks shared by the quantization kernels (sm_100a).
#pragma once

#include <cmath>
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/dtq_b200.h"

namespace dtq {

// ---- streaming global memory access ----------------------------------------------------------
// Inputs are read exactly once and outputs written exactly once, so neither should displace
// anything in L1; reads go through the non-coherent path, writes are marked evict-first.
__device__ __forceinline__ uint4 ldg_stream(const void *p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
// The same load with an L2 eviction policy attached (see l2_policy_evict_last): for data that the
// same launch reads again and that should therefore outlive the streaming traffic in L2.
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint4 ldg_stream_hint(const void *p, uint64_t policy) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0,%1,%2,%3}, [%4], %5;"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p), "l"(policy));
  return v;
}
// Same access without the streaming hint: for data that is read again later in the same launch.
__device__ __forceinline__ uint4 ldg_keep(const void *p) {
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ void stg_stream(void *p, uint2 v) {
  asm volatile("st.global.cs.v2.u32 [%0], {%1,%2};" ::"l"(p), "r"(v.x), "r"(v.y) : "memory");
}
__device__ __forceinline__ void stg_stream(void *p, uint32_t v) {
  asm volatile("st.global.cs.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void stg_stream(void *p, uint4 v) {
  asm volatile("st.global.cs.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}

// ---- programmatic dependent launch ------------------------------------------------------------
// Two kernels queued back to back on one stream normally run strictly one after the other: the
// second is launched when the first has drained.  A kernel launched with the programmatic-
// serialization attribute (launch_after_dependency in dtq_host.h) may instead become resident as
// soon as every block of its predecessor has executed pdl_launch_dependents (or exited); it must
// then execute pdl_wait before it touches anything the predecessor reads or writes: the wait
// returns when the predecessor has completed and its memory operations are visible.  Launch
// latency and the ramp of the second kernel hide under the tail of the first.  Both instructions
// are no-ops in a kernel that was launched the ordinary way.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Asks L2 to fetch `bytes` (a multiple of 16) from the 16-byte aligned global address `p`.  Nothing is
// delivered to the thread and nothing observable changes: L2 is where this GPU's memory is kept coherent,
// so a line fetched early is the line a later load would have fetched, whoever writes it in between.
__device__ __forceinline__ void l2_prefetch_bulk(const void *p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// ---- thread-block clusters ----------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The address, in the cluster's shared address space, of `local` (an address of this CTA's shared memory) in CTA `rank`.
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
// The two halves of the barrier of all threads of the cluster: what a thread wrote before it arrives is visible to whoever
// has waited.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync_all() {
  cluster_arrive();
  cluster_wait();
}
__device__ __forceinline__ void st_cluster_u32(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}

// SMs of a B200, for what must be known when compiled: how many blocks ask ahead.  The count of the device, as the kernels' grids
// use it, costs more than it is worth there: as a fifth parameter 0.35 us of the static cast's launch in the host, read in
// the kernel (%nsmid) 0.3 us of every cast of 16 to 48 MiB.
constexpr int kB200Sms = 148;

// The first blocks of a stream kernel (its kAskers) call this before pdl_wait: the tile that the block will take,
// `chunks` 16-byte chunks from `first` of `nchunks` in all, is asked into L2 while the kernel before drains (harmless whatever that
// still writes, see l2_prefetch_bulk).  What it hides is the start of the stream.  asks_ahead (dtq_host.h) has the sizes.
// Measured, bf16 [rows, 4096], outputs that stay; us with nothing asked, and the change in percent with 8 / 16 / 24 (static cast)
// or 2 / 4 / 8 blocks per SM (the others).  From memory: inputs of 400 MB in turn; three: three inputs in turn, as much of them in
// L2 as fits; amax: behind an amax of the input from memory, the two together in a graph, with as many blocks as ask; product: behind an MXFP8
// product of K = 1024 that wrote the input, the two together.  The products release their dependents early, so that their lines are asked for in
// vain; the amax when it ends, and then the lines stand behind the end of its own.
//   static cast      from memory             three                   amax            product
//      16 MiB   4.66  -6.9  -6.7  -6.7    3.96  -0.4  -4.3  -4.6     9.1  +6.0       16.1 -0.4 +0.3 +0.2
//      32 MiB   7.92 -11.8 -12.3 -10.7    8.63 -13.1 -21.2 -24.0   15.0  +5.7       26.5 +0.5 +1.2 +1.7
//      47 MiB  12.10  -5.6  -6.7  -6.2   12.17  -5.7  -9.4 -10.9   19.5 +10.6       36.9 +0.5 +0.9 +1.5
//      64 MiB  16.09  -3.4  -3.7  -3.2   15.98  -3.5  -6.0  -6.0   25.9  +8.0       45.6 +0.6 +0.9 +1.1
//      80 MiB  19.53  -2.3  -2.6  -2.0   19.46  -2.4  -4.2  -4.0   32.9  +3.1       59.4 -0.4 -0.7 -0.9
//     128 MiB  29.82  -1.0  -1.4  -0.8   30.02  -0.7  -1.7  -1.5   52.7  -0.9       96.1 -0.7 -0.7 -0.8
//     256 MiB  57.26  +0.5  +0.7  +0.8
//   fp32  16   4.51  -3.5  -5.4  -5.5    3.69  +4.8  +3.6  +3.8     8.9  +2.8
//         28   6.58  -5.5  -6.0  -6.9    6.82  -6.6 -10.1 -12.4   12.6  -0.6
//         64  13.28  -7.8 -11.8 -10.1   13.68  -4.8 -10.7 -13.5   24.5  +4.5
//        128  25.68  -0.5  -1.7  -2.0   25.66   0.0  -1.7  -2.7   47.7  +0.8
//   Two waves of blocks (16 per SM), not of bf16 between 48 and 80 MiB: there input and output of the pair just fill L2, and what is
//   asked for pushes out what the cast behind the amax would have found.  That holds below as well, where the cast alone gains more.
//   MX cast (4 blocks per SM)
//      16 MiB   5.00  -9.2  -4.2  -6.4    4.44  -5.0  -4.7  -4.5   10.3  -9.1       17.2  0.0 +0.1 +0.5
//      32 MiB   8.65 -13.2 -12.6 -11.9    9.04  -8.6 -13.8 -16.9   15.8  +3.2       27.1 -0.3 +0.1 +0.4
//      64 MiB  16.8   -1.4  -3.3  -2.0   16.8   -1.6  -3.4  -5.4   29.5  -1.8       47.6 +0.6 +1.1 +1.0
//     128 MiB  31.4   -0.7  -1.2  -0.6   31.4   -0.7  -0.9  -0.4   54.6  -1.5       98.5 -0.4 -0.5 -0.9
//     512 MiB 120.1   -0.2  -0.3   0.0
//   MX cast, blocked scales (2 blocks per SM)
//      16 MiB   5.33  -6.4  -1.9  -5.1    4.97  +0.2  +1.6  -2.6                   17.6 +0.1 +0.1 +0.1
//      32 MiB   8.99  -9.8  -8.1  -6.7    9.31  -6.4  -8.7 -11.1                   27.7 +0.5 +0.6 +0.6
//      64 MiB  16.95  -1.7  -2.4  -1.2   17.0   -1.4  -2.8  -2.8                   48.3 +0.6 +0.9 +1.3
//     128 MiB  31.5   -0.5  -0.5  +0.9   31.5   -0.5  -0.5  +0.9                   98.8 -0.2 -0.1 -0.4
//     512 MiB 120.9   +0.5  +1.5  +3.6   so not beyond 128 MiB
//   row-wise (8 blocks per SM)
//      16 MiB   5.59  -7.2 -11.8 -12.0    5.17  -3.9  -5.2  -6.6                   17.3 -0.5 -0.1 -0.1
//      32 MiB   9.11  -8.7 -13.6 -15.1    9.28  -7.4 -11.6 -15.5                   27.9 -1.0 -1.0 -0.7
//     128 MiB  30.9   -2.1  -3.0  -4.0   31.0   -2.8  -3.7  -4.7                   96.8 -0.4 -0.6 -0.8
// Below 16 MiB the grid is not much more than what is resident at once, and the loads follow at the prefetch's heels.
// Up to 2 MiB it is on again, for the tokens of a decode step: the product queued behind asks for its weights as soon as it is
// resident, and the cast's reads would stand behind those.  Cast and product, weights from memory, us, without / with, two (MXFP8),
// four (MXFP4) and three (row-wise) stages of weights asked for by the product:
//   tokens of K = 8192, N = 8192    16 (0.25 MiB)    33 (0.5)         64 (1)           128 (2)
//   MXFP8                           16.77 / 16.67    17.38 / 17.26    18.31 / 18.22    21.37 / 21.24
//   MXFP4                           11.80 / 11.15    12.49 / 11.85    13.59 / 12.98    16.32 / 15.59
//   row-wise                        16.53 / 16.46    17.35 / 17.19    18.46 / 18.25    21.12 / 20.93
//   128 tokens of K = 4096 (1 MiB), N = 8192: 15.85 / 15.54, 11.43 / 11.25, 15.56 / 15.10; of K = 16384 (4), N = 4096: 23.37 / 23.37, 18.17 / 17.60,
//   23.12 / 22.86
// By themselves, from memory: static cast 1 MiB 1.76 / 1.57, 2 MiB 2.10 / 1.88; MX 2.04 / 1.89, 2.27 / 2.01; row-wise 2.20 / 2.08, 3.00 / 2.33; in L2 all
// of them equal but the blocked MX cast, 1.95 / 2.00 and 2.09 / 2.20.
__device__ __forceinline__ void prefetch_first_tile(const uint4 *in, int64_t first, int64_t chunks, int64_t nchunks) {
  const int64_t left = nchunks - first;
  if (left > 0) l2_prefetch_bulk(in + first, unsigned((left < chunks ? left : chunks) * sizeof(uint4)));
}

// ---- number formats --------------------------------------------------------------------------
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// Two fp32 -> two fp8 bytes, round-to-nearest-even, saturating to the largest finite value.
// `lo` lands in bits 0-7 (lower address), `hi` in bits 8-15.
template <int OUT>
__device__ __forceinline__ uint32_t cvt_fp8x2(float lo, float hi) {
  uint16_t r;
  if constexpr (OUT == DTQ_E4M3) {
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  } else {
    asm("cvt.rn.satfinite.e5m2x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  }
  return r;
}
template <int OUT>
__device__ __forceinline__ uint32_t cvt_fp8x4(float a, float b, float c, float d) {
  return cvt_fp8x2<OUT>(a, b) | (cvt_fp8x2<OUT>(c, d) << 16);
}
template <int OUT>
__device__ __forceinline__ uint8_t cvt_fp8(float a) {
  return static_cast<uint8_t>(cvt_fp8x2<OUT>(a, 0.0f) & 0xFFu);
}

// fp32 power of two -> E8M0 byte, rounding towards +inf, saturating (inf -> 0xFE): sm_100a only.
__device__ __forceinline__ uint8_t cvt_ue8m0(float s) {
  uint16_t r;
  asm("cvt.rp.satfinite.ue8m0x2.f32 %0, %1, %2;" : "=h"(r) : "f"(s), "f"(s));
  return static_cast<uint8_t>(r & 0xFFu);
}

template <int OUT>
__device__ __forceinline__ constexpr double fp8_max() {
  return OUT == DTQ_E4M3 ? 448.0 : 57344.0;
}

// The fused ops' scale: a double, because the reference adds the double literal 1e-12.
template <int OUT>
__device__ __forceinline__ double dsq_scale(float amax) {
  return fp8_max<OUT>() / (static_cast<double>(amax) + 1e-12);
}
// (float)(scale_d * (double)x): product in double, one narrowing to fp32.
__device__ __forceinline__ float dsq_mul(double sd, float x) {
  return __double2float_rn(__dmul_rn(sd, static_cast<double>(x)));
}

// ---- the double-precision product without the 64-bit conversion pipe -----------------------------
// Done literally, (float)(scale_d * (double)x) costs two 64-bit conversions per element on the
// conversion (XU) pipe, and that pipe, not HBM, then bounds the kernel.  Two exact substitutes:
//
// (A) compensated fp32, for bf16 x and a bf16-valued amax in [0.25, 2^64] -- the normal case, amax
//     being an element of the tensor.  With head = sd rounded towards zero to fp32, tail = fp32(sd - head) >= 0:
//       t = fp32(x*tail),  R' = fma(x, head, t) = fp32(x*head + t)
//     and x*head + t differs from P = x*sd by < 2^-45 |P| (tail < 2^-23 sd, and it and t are each rounded once), so R' equals
//     the reference R = fp32(fp64(P)) unless P lies within 2^-45 of an fp32 rounding midpoint.  It cannot:
//     P = Q(1+theta) with Q = 7n 2^k / m (n, m <= 255 the integer mantissas of x and amax; both fp8
//     maxima are 7 * 2^j) and |theta| <= 1e-12/amax + 2^-51 <= 2^-36.9.  If m divides 7n 2^i, Q has
//     at most 11 significant bits, is an fp32 number, and P stays within 2^-36.9 of it; otherwise
//     |Q - M| >= 2^-33 |Q| for every 25-bit midpoint M (the difference of the two fractions is a
//     non-zero integer over m times a power of two).  Where t underflows (for an sd that is an fp32 number the tail
//     is the 2^-126 below, and t does for every |x| < 1) it is off by at most 2^-149, which is below 2^-45 |P| from
//     |P| = 2^-100 on; a smaller P converts to a signed zero either way.  Both products have the sign of x, zeros included, because tail is not negative; it
//     is not zero either (at least 2^-126, less than 2^-70 sd), so an infinite x gives an infinity and not 0 * inf,
//     and saturates as in the reference.  Two packed instructions per pair; the form with the rounding error of x*head
//     taken separately took four and two sign copies, and the issue of instructions is what bounds these kernels as soon
//     as they do not read from HBM.  Measured, bf16 -> e4m3, four instructions -> two: fused op 64 MiB 24.7 -> 20.6 us,
//     128 MiB 49.2 -> 44.6; row-wise 256 MiB 62.4 -> 57.9; cast with a known amax 64 MiB 15.9 -> 13.0, 128 MiB 31.2 -> 27.4.
//     This matters because with bf16 data about one e4m3 product in 128 sits exactly on an fp8
//     rounding tie (sd is a ratio of small integers), so any scheme that falls back to fp64 "near
//     a boundary" falls back in almost every warp.
// (B) bracket, for everything else (fp32 x, arbitrary amax): fp8 conversion is monotone, so if
//       fp8(fp32(x * fp32(sd(1 - 2^-21)))) == fp8(fp32(x * fp32(sd(1 + 2^-21))))
//     that byte is fp8(R) (every rounding involved is within 2^-24; underflow keeps the sign,
//     overflow saturates on both sides, NaN stays NaN); otherwise the pair is recomputed in fp64 by
//     a never-inlined function, so that the 64-bit conversions stay behind a real branch.
struct DsqScale {
  double sd;
  float lo, hi;      // (B) bracket ends
  float head, tail;  // (A) sd = head + tail + O(2^-47 sd), 0 < tail < 2^-23 sd
  bool compensated;  // (A) is valid for bf16 inputs
};
template <int OUT>
__device__ __forceinline__ DsqScale make_dsq_scale(float amax) {
  DsqScale s;
  s.sd = dsq_scale<OUT>(amax);
  s.lo = __double2float_rn(s.sd * (1.0 - 0x1p-21));
  s.hi = __double2float_rn(s.sd * (1.0 + 0x1p-21));
  s.head = __double2float_rz(s.sd);
  s.tail = fmaxf(__double2float_rn(s.sd - static_cast<double>(s.head)), 0x1p-126f);
  s.compensated = (__float_as_uint(amax) & 0xFFFFu) == 0u && amax >= 0.25f && amax <= 0x1p64f;
  return s;
}

// (A) two bf16-valued elements -> two fp8 bytes.
template <int OUT>
__device__ __forceinline__ uint32_t dsq_pair_compensated(float x0, float x1, const DsqScale &s) {
  const float2 x = make_float2(x0, x1);
  const float2 t = __fmul2_rn(x, make_float2(s.tail, s.tail));
  const float2 r = __ffma2_rn(x, make_float2(s.head, s.head), t);
  return cvt_fp8x2<OUT>(r.x, r.y);
}

// (B) two elements -> the fp8 bytes of the lower bracket end and of the upper end.
template <int OUT>
__device__ __forceinline__ void dsq_pair_bracket(float x0, float x1, const DsqScale &s, uint32_t &lo_bytes,
                                                 uint32_t &hi_bytes) {
  const float2 x = make_float2(x0, x1);
  const float2 pl = __fmul2_rn(x, make_float2(s.lo, s.lo));
  const float2 ph = __fmul2_rn(x, make_float2(s.hi, s.hi));
  lo_bytes = cvt_fp8x2<OUT>(pl.x, pl.y);
  hi_bytes = cvt_fp8x2<OUT>(ph.x, ph.y);
}
// fp32 -> fp64 is exact, so normal numbers are widened on the integer pipe (re-bias the exponent,
// move the mantissa); zeros, subnormals, infinities and NaNs take the conversion instruction.
__device__ __forceinline__ double widen_exact(float x) {
  const uint32_t w = __float_as_uint(x);
  const uint32_t a = w & 0x7FFFFFFFu;
  const uint32_t e = a >> 23;
  if (e - 1u >= 254u) return static_cast<double>(x);
  return __hiloint2double(static_cast<int>((w & 0x80000000u) | ((a >> 3) + 0x38000000u)), static_cast<int>(w << 29));
}
template <int OUT>
__device__ __forceinline__ uint32_t dsq_pair_exact(float x0, float x1, double sd) {
  return cvt_fp8x2<OUT>(__double2float_rn(__dmul_rn(sd, widen_exact(x0))),
                        __double2float_rn(__dmul_rn(sd, widen_exact(x1))));
}
// `r` = bytes of the lower bracket end, `m` = xor with the upper end's bytes: a non-zero 16-bit
// half marks a pair to redo.
template <int OUT>
__device__ __noinline__ uint2 dsq_redo_bf16x8(uint4 v, uint2 r, uint2 m, double sd) {
  if (m.x & 0xFFFFu) r.x = (r.x & 0xFFFF0000u) | dsq_pair_exact<OUT>(bf16_lo(v.x), bf16_hi(v.x), sd);
  if (m.x >> 16) r.x = (r.x & 0xFFFFu) | (dsq_pair_exact<OUT>(bf16_lo(v.y), bf16_hi(v.y), sd) << 16);
  if (m.y & 0xFFFFu) r.y = (r.y & 0xFFFF0000u) | dsq_pair_exact<OUT>(bf16_lo(v.z), bf16_hi(v.z), sd);
  if (m.y >> 16) r.y = (r.y & 0xFFFFu) | (dsq_pair_exact<OUT>(bf16_lo(v.w), bf16_hi(v.w), sd) << 16);
  return r;
}
template <int OUT>
__device__ __noinline__ uint32_t dsq_redo_f32x4(uint4 v, uint32_t r, uint32_t m, double sd) {
  if (m & 0xFFFFu) r = (r & 0xFFFF0000u) | dsq_pair_exact<OUT>(__uint_as_float(v.x), __uint_as_float(v.y), sd);
  if (m >> 16) r = (r & 0xFFFFu) | (dsq_pair_exact<OUT>(__uint_as_float(v.z), __uint_as_float(v.w), sd) << 16);
  return r;
}
// Eight bf16 (four packed words) -> eight fp8 bytes.
template <int OUT>
__device__ __forceinline__ uint2 dsq_convert_bf16x8(uint4 v, const DsqScale &s) {
  if (s.compensated) {
    return make_uint2(dsq_pair_compensated<OUT>(bf16_lo(v.x), bf16_hi(v.x), s) |
                          (dsq_pair_compensated<OUT>(bf16_lo(v.y), bf16_hi(v.y), s) << 16),
                      dsq_pair_compensated<OUT>(bf16_lo(v.z), bf16_hi(v.z), s) |
                          (dsq_pair_compensated<OUT>(bf16_lo(v.w), bf16_hi(v.w), s) << 16));
  }
  uint32_t a0, a1, a2, a3, b0, b1, b2, b3;
  dsq_pair_bracket<OUT>(bf16_lo(v.x), bf16_hi(v.x), s, a0, b0);
  dsq_pair_bracket<OUT>(bf16_lo(v.y), bf16_hi(v.y), s, a1, b1);
  dsq_pair_bracket<OUT>(bf16_lo(v.z), bf16_hi(v.z), s, a2, b2);
  dsq_pair_bracket<OUT>(bf16_lo(v.w), bf16_hi(v.w), s, a3, b3);
  uint2 r = make_uint2(a0 | (a1 << 16), a2 | (a3 << 16));
  const uint2 m = make_uint2(r.x ^ (b0 | (b1 << 16)), r.y ^ (b2 | (b3 << 16)));
  if (__builtin_expect((m.x | m.y) != 0, 0)) r = dsq_redo_bf16x8<OUT>(v, r, m, s.sd);
  return r;
}
// Four fp32 -> four fp8 bytes.
template <int OUT>
__device__ __forceinline__ uint32_t dsq_convert_f32x4(uint4 v, const DsqScale &s) {
  uint32_t a0, a1, b0, b1;
  dsq_pair_bracket<OUT>(__uint_as_float(v.x), __uint_as_float(v.y), s, a0, b0);
  dsq_pair_bracket<OUT>(__uint_as_float(v.z), __uint_as_float(v.w), s, a1, b1);
  uint32_t r = a0 | (a1 << 16);
  const uint32_t m = r ^ (b0 | (b1 << 16));
  if (__builtin_expect(m != 0, 0)) r = dsq_redo_f32x4<OUT>(v, r, m, s.sd);
  return r;
}

// ---- reductions of non-negative floats (or -inf) ------------------------------------------------
// Such floats order like their bit patterns read as signed ints (-inf is negative), so the
// warp-wide integer max instruction does the job exactly.
__device__ __forceinline__ float warp_max_nonneg(float v) {
  int b = __reduce_max_sync(0xFFFFFFFFu, __float_as_int(v));
  return __int_as_float(b);
}

// Block-wide max for blockDim.x a multiple of 32, up to 1024; result valid in every thread
// of warp 0.  `smem` holds 32 floats.
__device__ __forceinline__ float block_max_nonneg(float v, float *smem, float identity) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  v = warp_max_nonneg(v);
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  float r = identity;
  if (warp == 0) {
    r = lane < nwarps ? smem[lane] : identity;
    r = warp_max_nonneg(r);
  }
  return r;
}

// |x| of a packed bf16 pair and of eight packed pairs' running max; NaNs are dropped by max.
__device__ __forceinline__ __nv_bfloat162 as_bf162(uint32_t w) {
  return *reinterpret_cast<__nv_bfloat162 *>(&w);
}
__device__ __forceinline__ uint32_t as_u32(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t *>(&v); }

__device__ __forceinline__ __nv_bfloat162 absmax_bf162(__nv_bfloat162 acc, uint32_t w) {
  return __hmax2(acc, as_bf162(w & 0x7FFF7FFFu));
}
__device__ __forceinline__ float bf162_hmax_to_float(__nv_bfloat162 acc) {
  return fmaxf(__bfloat162float(acc.x), __bfloat162float(acc.y));
}

}  // namespace dtq
