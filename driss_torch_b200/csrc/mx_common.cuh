// MX (block-32, E8M0 scale, e4m3 payload) arithmetic shared by the MX kernels; identical to the
// reference's (src/mx_cast.cu:44-86 for the scale, :146-153 for payload and scale byte).
#pragma once

#include "dtq_device.cuh"

namespace dtq {

// Per-half maximum of two words of packed 15-bit bf16 magnitudes (sign bits clear): one bf16x2
// max.  NaN-propagating, so a NaN (the largest magnitudes when read as integers) still wins; it
// comes out as the canonical 0x7FFF, which has the exponent field and the non-zero mantissa of
// every other NaN, hence the same block exponent.
__device__ __forceinline__ uint32_t packed_mag_max(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.NaN.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// The same on signed values: per-half max(|a|, |b|), with a sign bit that is the XOR of the operands'
// signs -- garbage to be masked off once at the end of a chain (a canonical NaN included).
__device__ __forceinline__ uint32_t packed_absmax_signed(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.NaN.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// Largest 15-bit magnitude among the eight bf16 of a 16-byte chunk.
__device__ __forceinline__ uint32_t chunk_absmax_bits(uint4 v) {
  const uint32_t m = packed_absmax_signed(packed_absmax_signed(v.x, v.y), packed_absmax_signed(v.z, v.w)) & 0x7FFF7FFFu;
  return max(m & 0xFFFFu, m >> 16);
}

// Biased exponent of the block scale from the block's largest magnitude bits.  The reference:
// e = ceil(log2 |x|) from the exponent field (+1 if the mantissa is non-zero; zero -> -128,
// subnormal -> -126), biased = clamp(e - 8 + 127, 0, 255); e is monotone in |x|, so taking the
// maximum of the raw magnitudes first gives the same block exponent as the maximum of the e_i.
// Here: (mag + 0x7F) >> 7 = exponent field + (mantissa != 0), so biased = that - 8 clamped at 0.
// For the exponent field 0 (zero and subnormals) both forms are negative before the clamp, and
// the upper clamp never acts: mag <= 0x7FFF gives at most 248.
__device__ __forceinline__ int block_biased_exponent(uint32_t mag) {
  return max(0, static_cast<int>((mag + 0x7Fu) >> 7) - 8);
}

// 1 / scale for scale = 2^(biased-127), as the reference's rcp.rn gives it: the exact power of
// two (a normal number, since biased <= 248), and +inf for scale 0 (biased 0).  Built from the
// exponent instead of running the reciprocal sequence.
__device__ __forceinline__ float inverse_scale(int biased) {
  return __uint_as_float(biased == 0 ? 0x7F800000u : static_cast<uint32_t>(254 - biased) << 23);
}

// Two packed bf16 -> two e4m3 bytes of x * inv.
__device__ __forceinline__ uint32_t mx_pair(uint32_t w, float inv) {
  const float2 p = __fmul2_rn(make_float2(bf16_lo(w), bf16_hi(w)), make_float2(inv, inv));
  return cvt_fp8x2<DTQ_E4M3>(p.x, p.y);
}

// The same from two values already widened to fp32.
__device__ __forceinline__ uint32_t mx_pair_f32(float lo, float hi, float inv) {
  const float2 p = __fmul2_rn(make_float2(lo, hi), make_float2(inv, inv));
  return cvt_fp8x2<DTQ_E4M3>(p.x, p.y);
}

__device__ __forceinline__ uint2 mx_payload(uint4 v, float inv) {
  uint2 r;
  r.x = mx_pair(v.x, inv) | (mx_pair(v.y, inv) << 16);
  r.y = mx_pair(v.z, inv) | (mx_pair(v.w, inv) << 16);
  return r;
}

// The scale byte.  The reference converts 2^(biased-127) with cvt.rp.satfinite.ue8m0x2.f32; for a
// power of two in range that is the exponent field itself, 0.0 (biased 0) gives 0, and the
// saturating case (biased 255) cannot occur (biased <= 248).
__device__ __forceinline__ uint8_t mx_scale_byte(int biased) { return static_cast<uint8_t>(biased); }

// Where the scale of MX block `blk` (row-major index over [rows, kblocks]) goes.
// Row-major: scales[blk], the reference's layout (src/mx_cast.cu:199,210-211).
// Blocked: the layout the reference's MX GEMM consumes (src/mx_fp8_bf16.cu:97-110, CUTLASS
// Sm1xxBlockScaledConfig::tile_atom_to_shape_SFA; the reference gets there through a separate
// `to_blocked` pass, test/test_mx.py:28-32): 128-row x 4-k-block atoms of 512 bytes, atoms ordered
// k-block-major within a 128-row band; inside an atom row r, k-block c sit at
// (r % 32) * 16 + (r / 32) * 4 + c.
template <bool BLOCKED>
__device__ __forceinline__ int64_t scale_offset(int64_t blk, int64_t kblocks, int64_t katoms) {
  if constexpr (!BLOCKED) return blk;
  // the number of MX blocks of a tensor that fits this GPU's memory is below 2^32: a 32-bit division, a fifth of the work
  const uint32_t r = static_cast<uint32_t>(blk) / static_cast<uint32_t>(kblocks);
  const uint32_t c = static_cast<uint32_t>(blk) - r * static_cast<uint32_t>(kblocks);
  const int64_t atom = (r >> 7) * katoms + (c >> 2);
  return atom * 512 + (r & 31) * 16 + ((r >> 5) & 3) * 4 + (c & 3);
}

// The padding of a blocked scale array: the rows up to the next multiple of 128 and, where kblocks % 4 != 0, the rest of
// every row's last atom.  Written as zeros by spare blocks of the cast itself: a separate fill of the array costs a
// launch, and one that keeps the cast from starting under the tail of the kernel before it.
// `thread` of `threads` in all takes its share.  One item is the four bytes that a row of the last row band has in one of
// its atoms (32 x 16 bytes: byte group q of chunk l is row 32 q + l; a thread takes a chunk), or the tail of one row.
// No divisions: 64-bit ones made these few bytes take longer than the cast (2016 x 4096: 4.8 us without padding, 8.5 with).
// And no single bytes where the array allows it: the scales of 8 or 16 rows are nearly all padding, and with four byte stores
// per group the padding blocks were still at it 2 us after the cast itself (16 x 4096: 3.2 us of a decode step's chain).
__host__ __device__ inline int64_t scale_padding_items(int64_t rows, int64_t kblocks) {
  return (rows % 128 ? (kblocks + 3) / 4 * 32 : 0) + (kblocks % 4 ? rows : 0);
}
__device__ __forceinline__ void zero_scale_padding(uint8_t *scales, int64_t rows, int64_t kblocks, int64_t thread, int64_t threads) {
  const int64_t katoms = (kblocks + 3) / 4;
  const int used = int(rows & 127);  // rows of the last band that exist
  if (used) {
    uint8_t *band = scales + (rows >> 7) * katoms * 512;
    const bool wide = (reinterpret_cast<uintptr_t>(scales) & 15) == 0;
    for (int64_t i = thread; i < katoms * 32; i += threads) {  // atom i / 32, chunk i % 32
      const int l = int(i & 31);
      if (wide && l >= used) {
        *reinterpret_cast<uint4 *>(band + i * 16) = make_uint4(0, 0, 0, 0);
        continue;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint8_t *p = band + i * 16 + q * 4;
        if (32 * q + l >= used) {
          if (wide) *reinterpret_cast<uint32_t *>(p) = 0;
          else p[0] = p[1] = p[2] = p[3] = 0;
        }
      }
    }
  }
  const int live = int(kblocks & 3);
  if (live)
    for (int64_t r = thread; r < rows; r += threads) {
      uint8_t *p = scales + ((r >> 7) * katoms + katoms - 1) * 512 + (r & 31) * 16 + ((r >> 5) & 3) * 4;
      for (int c = live; c < 4; ++c) p[c] = 0;
    }
}
// The tiles of block `block` of a grid whose first `pad_blocks` blocks write padding instead: its first, and the step to its
// next (the number of blocks that take tiles).
struct TileWalk {
  int64_t first, step;
};
__host__ __device__ constexpr TileWalk tile_walk(unsigned block, unsigned grid, unsigned pad_blocks) {
  return {int64_t(block) - pad_blocks, int64_t(grid) - pad_blocks};
}
constexpr bool takes_every_tile_once(int64_t tiles, unsigned grid, unsigned pad_blocks) {
  for (int64_t t = 0; t < tiles; ++t) {
    int taken = 0;
    for (unsigned b = pad_blocks; b < grid; ++b)
      for (int64_t i = tile_walk(b, grid, pad_blocks).first; i < tiles; i += tile_walk(b, grid, pad_blocks).step) taken += i == t;
    if (taken != 1) return false;
  }
  return true;
}
// as many blocks as tiles, as today's grids; blocks that take several, with and without padding
static_assert(takes_every_tile_once(7, 9, 2) && takes_every_tile_once(7, 7, 0) && takes_every_tile_once(13, 5, 2) &&
                  takes_every_tile_once(13, 3, 0) && takes_every_tile_once(1, 4, 3),
              "blocks beside the padding share out the tiles");

// Spare blocks of `threads` threads for it, about one item per thread.
inline int64_t scale_padding_blocks(int64_t rows, int64_t kblocks, int threads) {
  const int64_t n = (scale_padding_items(rows, kblocks) + threads - 1) / threads;
  return n < 1024 ? n : 1024;
}

}  // namespace dtq
