// mx_fp8_bf16: D[M,N] (bf16) = sum_k  A[m,k] * 2^(sa[m,k/32]-127) * B[n,k] * 2^(sb[n,k/32]-127)
//
// The consumer of the MX casts: e4m3 operands with one E8M0 scale per 32 elements along K, both
// scale tensors in the blocked (128 x 4 atoms of 512 bytes) layout that mx_fp8_quantize_blocked
// emits.  Replaces driss_torch::mx_fp8_bf16 (src/mx_fp8_bf16.cu:42-163 run_gemm, :168-215 validate,
// :217-241), which instantiates a CUTLASS Sm100 block-scaled collective with 128x128x128 tiles; and, from
// the same source, mx_fp4_bf16 (:243-271) and the row-wise scaled GEMM behind sweep_mm (src/sweep_mm.cu,
// src/scaled_mm_kernels/f8f8bf16_rowwise_kernel.h:151-175), see Format below.
//
// Hand-written for sm_100a.  Four kernels from one source (chosen per call by a measured cost model, see
// launch_gemm): an SM pair on a 256 x 256 tile (tcgen05.mma.cta_group::2, further down), one CTA per SM on a
// 128 x 256 or a 128 x 128 tile (this kernel), and for few tiles a cluster that splits K (last).  Common to all:
//   * persistent CTAs of 320 threads walk the output tiles (the split kernel: 192, one tile); K advances in stages of 128 bytes;
//   * warp 0 is the producer: per stage tiled TMA loads of the operands (boxes of 128 bytes of K, 128-byte
//     swizzle, rows and columns past the edges filled with zeros) and of the stage's scale atoms (a 3-D tensor
//     map over the blocked scale array, an atom past the end arrives as zeros), all counted on the stage's `full`
//     mbarrier;
//   * warp 1 issues the tensor-core work: tcgen05.cp moves the stage's scale atoms from shared memory into
//     tensor memory (32 rows x 16 bytes, replicated to the four lane quadrants, which is exactly one blocked
//     atom), then four tcgen05.mma (K = 32 bytes of every operand row each), the k-block picking its scale byte
//     through the descriptor's scale-factor id; tcgen05.commit releases the stage (`empty`) and finally hands
//     the accumulator (128 lanes x up to 256 fp32 columns of tensor memory) to the epilogue;
//   * both of those warps walk their loops as whole warps with one elected lane issuing (see elect_one);
//   * warps 2..9 are the epilogue.  Single CTA: tcgen05.ld 2 x 32 columns at a time, fp32 -> bf16, 64-byte row segments
//     straight to global memory; the accumulator is released as soon as it is in registers, so the next tile's MMAs
//     overlap the stores.  The SM pair stages 32 x 32 boxes in shared memory for TMA stores; the split kernel's four
//     warps leave partial sums in shared memory, which the cluster adds up.
// No load is shared between CTAs: every CTA loads its own operands (A and B of an 8192^3 problem both fit in
// L2).  Every wait is bounded: a wait that runs out records DTQ_ERR_TIMEOUT in the status word, raises the CTA's
// abort flag, the roles drain what they have in flight, tensor memory is freed and the kernel returns.  (Roles wait as
// whole warps, see mbar_wait_warp.)
#include <cuda.h>

#include <algorithm>
#include <atomic>

#include "dtq_device.cuh"
#include "dtq_host.h"

namespace dtq {
namespace {

constexpr int kBM = 128;        // tile rows (M)
constexpr int kBK = 128;        // K bytes per stage: one 128-byte swizzle span = 4 MX blocks of 32
constexpr int kGemmThreads = 320;  // producer warp, MMA warp, 8 epilogue warps
constexpr int kEpilogueWarps = 8;
constexpr int kSfaCol = 256;               // scales of A: 4 tensor-memory columns per atom (128 rows x 4 k-blocks)
constexpr int kSfbCol = 256 + 16;          // scales of B: 4 columns per atom, up to 2 (N) x 2 (K) atoms
// Element formats.  e4m3: one byte per element, a 128-byte stage is 128 elements = 4 MX blocks = one scale atom
// along K, tcgen05.mma kind::mxf8f6f4 (K = 32 per instruction, one scale byte each for A and B).  e2m1 (MXFP4): two
// elements per byte, a 128-byte stage is 256 elements = 8 MX blocks = two scale atoms along K, kind::mxf4 with
// block32 scaling (K = 64 per instruction, which uses two consecutive scale bytes).  Either way an instruction
// reads 32 bytes of every operand row, so the operand descriptors are the same.
//
// A third mode has no block scales at all: fp8 operands (e4m3, or e5m2 for A) through kind::f8f6f4, with one fp32
// scale per row of A and per row of B (and an optional bias per column) applied to the fp32 accumulator in the
// epilogue -- the row-wise scaled GEMM that consumes dtq_dynamic_scaled_quant_rowwise's scales.
constexpr int kMxFp8 = 0, kMxFp4 = 1, kRowwise = 2;
template <int MODE>
struct Format {
  static constexpr bool kScaled = MODE != kRowwise;            // block scales travel with the operands
  static constexpr int kKAtoms = MODE == kMxFp4 ? 2 : 1;      // scale atoms along K per stage (staging is sized for them)
  // k (0..3) = the instruction within a stage: which atom along K, and which byte (pair) of its 4-byte scale columns
  __device__ static constexpr uint32_t k_atom(uint32_t k) { return MODE == kMxFp4 ? k >> 1 : 0u; }
  __device__ static constexpr uint32_t sf_id(uint32_t k) { return MODE == kMxFp4 ? (k & 1u) * 2u : (MODE == kMxFp8 ? k : 0u); }
  // instruction-descriptor bits besides the shape: block-scaled kinds carry the scale format (bit 23 = E8M0) and for
  // kind::mxf4 the e2m1 operand format; kind::f8f6f4 carries the accumulator format (bits 4-5 = fp32), the operand
  // formats come with the call (e4m3 = 0 or e5m2 = 1 in bits 7-9 / 10-12)
  static constexpr uint32_t kFormatBits = MODE == kMxFp4 ? ((1u << 7) | (1u << 10) | (1u << 23)) : (MODE == kMxFp8 ? (1u << 23) : (1u << 4));
};
constexpr int kTmemCols = 512;             // allocation (power of two); one CTA: columns 0..255 hold the accumulator(s); pair: PairTmem

// Two tile shapes.  Wide: 128 x 256, one accumulator of 256 columns, 4 stages -- least operand traffic per
// output (every byte of B serves 128 rows, every byte of A 256 columns), the shape for large problems.
// Narrow: 128 x 128, two accumulators of 128 columns (the epilogue of one tile runs under the MMAs of the
// next), 6 stages -- twice the tiles, for problems whose wide tiles would leave a large part of the last wave
// of SMs idle.
template <int BN_, int STAGES_, int ACC_>
struct GemmShape {
  static constexpr int BN = BN_, STAGES = STAGES_, ACC = ACC_;
  static_assert(BN == 128 || BN == 256, "N tile");
  static_assert(ACC * BN <= 256, "accumulators live in tensor-memory columns 0..255");
};
using WideShape = GemmShape<256, 4, 1>;
using NarrowShape = GemmShape<128, 6, 2>;
template <int MAPS, typename PARAMS>
constexpr size_t kGemmParameterBytes = MAPS * sizeof(CUtensorMap) + sizeof(PARAMS);  // all but the padding, see LaunchPad
constexpr unsigned long long kWaitLimitNs = 2000000000ull;  // a wait gives up after two seconds of wall time (Workspace::wait_limit_us)

// Shared memory that a kernel asks for: its struct, and what aligning that to 1024 bytes may take.  A struct that outgrew
// the limit would fail in cudaFuncSetAttribute, and for the cluster kernels look like a device without them.
constexpr size_t kMaxDynamicSmem = 227 * 1024;
template <typename SMEM>
constexpr int smem_bytes() {
  static_assert(sizeof(SMEM) + 1024 <= kMaxDynamicSmem, "more shared memory than a block can have");
  return static_cast<int>(sizeof(SMEM) + 1024);
}

template <typename SH, int MODE>
struct __align__(1024) GemmSmem {
  uint8_t a[SH::STAGES][kBM * kBK];        // 16 KB per stage, 1024-byte aligned (swizzle atom = 8 rows x 128 B)
  uint8_t b[SH::STAGES][SH::BN * kBK];     // 16 or 32 KB per stage
  uint8_t sfa[SH::STAGES][Format<MODE>::kKAtoms * 512];                  // blocked atoms of 128 rows x 4 k-blocks
  uint8_t sfb[SH::STAGES][SH::BN / 128 * Format<MODE>::kKAtoms * 512];  // [128 tile columns][atom along K]
  alignas(512) uint8_t out[kEpilogueWarps][32 * 64];  // per epilogue warp 32 rows x 32 bf16 on their way out (store_chunk)
  uint64_t full[SH::STAGES];
  uint64_t empty[SH::STAGES];
  uint64_t tmem_full[SH::ACC];
  uint64_t tmem_empty[SH::ACC];
  uint64_t drained;  // only the way out of an abort commits to it: the others may still have commits on their way
  uint32_t tmem_base;
  int abort;
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// One poll of the phase with the given parity; the thread may sleep up to about a microsecond inside it.
__device__ __forceinline__ bool mbar_poll(uint32_t addr, unsigned parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(addr), "r"(parity), "r"(1000u)
      : "memory");
  return done != 0;
}
// What every wait of a role looks at besides its barrier: the CTA's abort flag, and the caller's workspace, which holds
// the limit and takes the status when a wait gives up.
struct Bounds {
  volatile int *abort;
  Workspace *ws;
  __device__ __forceinline__ void give_up() const {
    atomicExch(&ws->status, DTQ_ERR_TIMEOUT);
    *abort = 1;
  }
};
// Bounded wait of one thread for the phase of the given parity: false if it has not completed within the limit of wall
// time, or (`abort` not null) if the CTA is aborting.  Behind the two functions below, which the roles use.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity, volatile int *abort, const Workspace *ws) {
  const uint32_t addr = smem_addr(bar);
  if (mbar_poll(addr, parity)) return true;
  const unsigned long long start = global_ns();
  for (unsigned int spins = 1;; ++spins) {
    if (mbar_poll(addr, parity)) return true;
    if ((spins & 63u) == 0) {
      if (abort && *abort) return false;
      const unsigned int us = ws ? *const_cast<const volatile unsigned int *>(&ws->wait_limit_us) : 0u;
      if (global_ns() - start > (us ? us * 1000ull : kWaitLimitNs)) return false;
    }
  }
}
// The wait of a role, by all lanes of a converged warp, with one answer for the warp: what follows it is warp-wide
// (tcgen05.ld, shuffles, elect.sync), so no lane may leave on a flag that another lane has not seen.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, unsigned parity, const Bounds &b) {
  return __all_sync(0xFFFFFFFFu, mbar_wait(bar, parity, b.abort, b.ws));
}
// The wait of a single lane for its own copies or MMAs in flight on the way out; an abort does not cut it short.
__device__ __forceinline__ void mbar_drain(uint64_t *bar, unsigned parity) { mbar_wait(bar, parity, nullptr, nullptr); }
// True in one lane of a converged warp, the same lane every time.  The producer and the MMA issuer walk their
// loops as whole warps and let the elected lane issue the asynchronous instructions: everything those
// instructions take as operands (descriptors, coordinates, barrier addresses) is then the same in all lanes,
// which lets the compiler keep it in the warp's uniform registers, where TMA and tcgen05 instructions read
// their operands from.  A loop walked by a single lane instead pays a transfer into uniform registers for
// every operand of every instruction: measured here, 55 to 75 clocks per tcgen05 instruction, which made the
// issuing thread, not the tensor cores, the limit of the kernel.
__device__ __forceinline__ bool elect_one() {
  uint32_t elected;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
  return elected != 0;
}
// A value that is the same in every lane, in a form the compiler can see is.
__device__ __forceinline__ uint32_t warp_uniform(uint32_t v) { return __shfl_sync(0xFFFFFFFFu, v, 0); }

// Tiled TMA load of a box at (x = byte column, y = row) into this CTA's shared memory.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                   smem_addr(dst)),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
                   smem_addr(dst)),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(x), "r"(y), "r"(z)
               : "memory");
}

// Shared-memory matrix descriptor of a K-major operand tile whose rows are 128 bytes long and
// 128-byte swizzled (what the TMA loads above produce): start address, leading byte offset (unused
// for swizzled K-major tiles, encoded as 1), stride between 8-row groups = 1024 bytes, descriptor
// version 1, layout type 2 = 128-byte swizzle.  Addresses and offsets are in units of 16 bytes.
__device__ __forceinline__ uint64_t operand_desc(uint32_t saddr) {
  return uint64_t((saddr >> 4) & 0x3FFFu) | (uint64_t(1) << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) |
         (uint64_t(2) << 61);
}
// Descriptor of one scale atom for tcgen05.cp: 32 rows of 16 bytes, no swizzle; 8-row groups 128 bytes apart.
__device__ __forceinline__ uint64_t scale_desc(uint32_t saddr) {
  return uint64_t((saddr >> 4) & 0x3FFFu) | (uint64_t(128 >> 4) << 32) | (uint64_t(1) << 46);
}
// Instruction descriptor of tcgen05.mma kind::mxf8f6f4.block_scale: e4m3 x e4m3, both K-major, E8M0 scales,
// M = 128, N = `bn`; `k` (0..3) is the byte of the 4-byte scale column that this k-block uses, for A and B.
__device__ __forceinline__ uint32_t instr_desc(uint32_t sf_id, uint32_t bn, uint32_t m, uint32_t format_bits) {
  return (sf_id << 4) | format_bits | ((bn >> 3) << 17) | ((m >> 4) << 24) | (sf_id << 29);
}
// One MMA: D (tensor memory) (+)= A x B, block-scaled kinds with the scales found at the two tensor-memory addresses.
template <int MODE, bool PAIR>
__device__ __forceinline__ void issue_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate,
                                          uint32_t sfa_tmem, uint32_t sfb_tmem) {
#define DTQ_MMA(GROUP, KIND)                                                                                         \
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"                                                     \
               "tcgen05.mma.cta_group::" GROUP ".kind::" KIND " [%0], %1, %2, %3, [%5], [%6], p;\n\t}"                \
               :                                                                                                     \
               : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem)    \
               : "memory")
  if constexpr (MODE == kMxFp4 && PAIR) DTQ_MMA("2", "mxf4.block_scale.block32");
  else if constexpr (MODE == kMxFp4) DTQ_MMA("1", "mxf4.block_scale.block32");
  else if constexpr (MODE == kMxFp8 && PAIR) DTQ_MMA("2", "mxf8f6f4.block_scale");
  else if constexpr (MODE == kMxFp8) DTQ_MMA("1", "mxf8f6f4.block_scale");
  else if constexpr (PAIR)  // no block scales; the braces hold the (unused) mask of output lanes to leave alone
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
                 :
                 : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
                 : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                 :
                 : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
                 : "memory");
#undef DTQ_MMA
}
// Instructions of 32 operand bytes that stage `ks` takes: four, but the last one only as many as K has, for what lies behind it
// arrived as zeros.  Adding them cost as much as any others where the tensor cores are the limit (B200, us, three sets in turn): MXFP8
// 8721 x 1072 x 1728 22.9 -> 21.8, 933 x 6320 x 1312 12.9 -> 12.5, row-wise 12511 x 272 x 2144 14.2 -> 13.5.
__device__ __forceinline__ uint32_t live_k(int ks, int k_stages, int last_k) { return ks + 1 == k_stages ? uint32_t(last_k) : 4u; }

// One scale atom, shared memory -> 4 tensor-memory columns (32 rows x 16 bytes, replicated to the four lane quadrants).
template <bool PAIR>
__device__ __forceinline__ void copy_scale_atom(uint32_t tmem_col_addr, uint32_t smem_atom_addr) {
  if constexpr (PAIR)
    asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem_col_addr), "l"(scale_desc(smem_atom_addr)) : "memory");
  else
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(tmem_col_addr), "l"(scale_desc(smem_atom_addr)) : "memory");
}

__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// fp32 pair -> packed bf16x2 (lo in the low half).
__device__ __forceinline__ uint32_t pack_bf16(uint32_t lo, uint32_t hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(__uint_as_float(hi)), "f"(__uint_as_float(lo)));
  return r;
}

// Tile order: consecutive tile numbers (the tiles that the CTAs of one wave work on together) fill bands of
// kGroupM tile rows, n-tile by n-tile, so that a wave of 148 tiles touches about 16 x 9 tiles' worth of A
// and B (34 MB at K = 8192) instead of every row of A: what is re-read from L2 mostly stays there.
constexpr int kGroupM = 16;
__device__ __forceinline__ void tile_coords(int tile, int m_tiles, int n_tiles, int *mt, int *nt) {
  const int per_group = kGroupM * n_tiles;
  const int g = tile / per_group, idx = tile - g * per_group;
  const int rows = min(kGroupM, m_tiles - g * kGroupM);
  *mt = g * kGroupM + idx % rows;
  *nt = idx / rows;
}

// The row-wise mode's epilogue: out = bf16(fp32(fp32(acc * row_scale[m]) * col_scale[n]) + bias[n]), every step rounded
// to fp32 (src/scaled_mm_kernels/f8f8bf16_rowwise_kernel.h:151-175: Multiply(WScale, Multiply(XScale, Acc)), Add(Bias), Cast).
struct RowwiseEpilogue {
  const float *row_scale;  // [M]
  const float *col_scale;  // [N]
  const void *bias;        // [N] fp32 or bf16, or null
  int bias_is_bf16;
  uint32_t operand_format_bits;  // a_format << 7 | b_format << 10 (e4m3 = 0, e5m2 = 1)
};
// What a thread of the epilogue needs of the scales for one tile, fetched BEFORE it waits for the accumulator (none of
// it depends on the MMAs): its row's scale, and for each 32-column chunk of its columns the scale and bias of column
// `lane` of the chunk; the value for column i of a chunk then comes from lane i by shuffle.  Columns past N get 0.
template <int CHUNKS>
struct RowwiseRegs {
  float xs;
  float cs[CHUNKS], bs[CHUNKS];
  bool has_bias;
};
template <int CHUNKS>
__device__ __forceinline__ void load_rowwise(RowwiseRegs<CHUNKS> &r, const RowwiseEpilogue &e, int64_t row, int64_t col0, int lane,
                                             int M, int N) {
  r.xs = row < M ? __ldg(e.row_scale + row) : 0.0f;
  r.has_bias = e.bias != nullptr;
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    const int64_t col = col0 + c * 32 + lane;
    const bool live = col < N;
    r.cs[c] = live ? __ldg(e.col_scale + col) : 0.0f;
    r.bs[c] = 0.0f;
    if (live && r.has_bias)
      r.bs[c] = e.bias_is_bf16 ? __uint_as_float(uint32_t(__ldg(static_cast<const uint16_t *>(e.bias) + col)) << 16)
                               : __ldg(static_cast<const float *>(e.bias) + col);
  }
}
// 32 consecutive accumulator columns of one row (fp32 bit patterns) through the row-wise epilogue, in place:
// bf16((acc * x_scale[row]) * w_scale[col] + bias[col]), every step rounded to fp32 as the reference's epilogue tree does.
__device__ __forceinline__ void apply_rowwise(uint32_t (&v)[32], float xs, float cs, float bs, bool has_bias) {
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    float f = __fmul_rn(__fmul_rn(__uint_as_float(v[i]), xs), __shfl_sync(0xFFFFFFFFu, cs, i));
    const float b = __shfl_sync(0xFFFFFFFFu, bs, i);
    if (has_bias) f = __fadd_rn(f, b);
    v[i] = __float_as_uint(f);
  }
}

// The same with the 32 columns' scales and biases (null: none) in shared memory, 16-byte aligned.
__device__ __forceinline__ void apply_rowwise_shared(uint32_t (&v)[32], float xs, const float *cs, const float *bs) {
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    const float4 s = *reinterpret_cast<const float4 *>(cs + i);
    float f[4] = {__fmul_rn(__fmul_rn(__uint_as_float(v[i]), xs), s.x), __fmul_rn(__fmul_rn(__uint_as_float(v[i + 1]), xs), s.y),
                  __fmul_rn(__fmul_rn(__uint_as_float(v[i + 2]), xs), s.z), __fmul_rn(__fmul_rn(__uint_as_float(v[i + 3]), xs), s.w)};
    if (bs) {
      const float4 b = *reinterpret_cast<const float4 *>(bs + i);
      f[0] = __fadd_rn(f[0], b.x), f[1] = __fadd_rn(f[1], b.y), f[2] = __fadd_rn(f[2], b.z), f[3] = __fadd_rn(f[3], b.w);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) v[i + j] = __float_as_uint(f[j]);
  }
}

// 32 accumulator columns of this thread's lane of tensor memory into registers (asynchronous: tmem_load_wait).
__device__ __forceinline__ void tmem_load_32(uint32_t (&v)[32], uint32_t taddr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
}
// Waits for this thread's tensor-memory loads.  The registers pass through the statement, so that no use of them can
// be scheduled before it.
__device__ __forceinline__ void tmem_load_wait(uint32_t (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]),
                 "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), "+r"(v[16]),
                 "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]),
                 "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31])
               :
               : "memory");
}

// 32 columns of 32 rows of the output, a row per lane (16 bf16 pairs), to global memory through 2 KB of this warp's own
// shared memory: read back, four lanes hold 64 consecutive bytes of a row, and a store touches 8 rows instead of 32.
// With a row per lane and 16 bytes per store, every instruction sent a partial 32-byte sector to each of 32 lines, and these stores
// bounded the single-CTA kernels wherever K is short.  Three outputs in turn, B200, us, wide / narrow, before -> now: row-wise 19879 x
// 3072 x 640 89.4 / 93.3 -> 67.7 / 66.4, MXFP8 32768 x 4096 x 256 114.5 / 127.4 -> 74.7 / 82.5 (writing them alone: 72), 4096 x 4096 x 512 17.6 /
// 17.1 -> 13.4 / 13.0, 1216 x 1280 x 3360 16.0 / 11.3 -> 14.7 / 10.7, 1632 x 736 x 2272 12.3 / 8.6 -> 10.8 / 7.9, 721 x 1784 x 672 7.4 / 5.1 ->
// 6.6 / 4.7, row-wise 962 x 1392 x 944 11.4 / 7.4 -> 10.1 / 6.8.  The pair kernel stays with TMA stores: 32768 x 4096 x 256 76.9 / 84.8 this way,
// row-wise 32768 x 4096 x 512 105 / 115.
// `row0` / `col0`: the chunk's first row and column; N % 8 == 0, so 16 bytes are inside or outside as a whole.
__device__ __forceinline__ void store_chunk(uint8_t *staging, const uint32_t (&packed)[16], uint16_t *out, int64_t row0, int64_t col0,
                                            int M, int N, int lane) {
  __syncwarp();  // the chunk before has been read
#pragma unroll
  for (int q = 0; q < 4; ++q)  // 16-byte groups XOR-swizzled by the row pair: both ways free of bank conflicts
    *reinterpret_cast<uint4 *>(staging + lane * 64 + ((q ^ ((lane >> 1) & 3)) * 16)) =
        make_uint4(packed[4 * q], packed[4 * q + 1], packed[4 * q + 2], packed[4 * q + 3]);
  __syncwarp();
  const int q = lane & 3, r = lane >> 2;
  if (col0 + q * 8 >= N) return;
  uint16_t *dst = out + (row0 + r) * N + col0 + q * 8;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = r + 8 * i;
    const uint4 v = *reinterpret_cast<const uint4 *>(staging + row * 64 + ((q ^ ((row >> 1) & 3)) * 16));
    if (row0 + row < M) stg_stream(dst + int64_t(8 * i) * N, v);  // streaming store: the output must not push the operands out of L2
  }
}

struct GemmParams {
  RowwiseEpilogue rowwise;
  uint16_t *out;  // bf16 [M, N]
  int M, N, last_k;  // last_k: see live_k
  int m_tiles, n_tiles, k_stages;
  Workspace *ws;
};

template <typename SH, int MODE>
__global__ void __launch_bounds__(kGemmThreads, 1)
mx_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               const __grid_constant__ CUtensorMap map_sfa, const __grid_constant__ CUtensorMap map_sfb, GemmParams p,
               LaunchPad<kGemmParameterBytes<4, GemmParams>>) {
  constexpr int kBN = SH::BN, kStagesG = SH::STAGES, kAcc = SH::ACC, kAtomsB = SH::BN / 128;
  constexpr int kKAtoms = Format<MODE>::kKAtoms;
  extern __shared__ unsigned char smem_raw[];
  GemmSmem<SH, MODE> &sm =
      *reinterpret_cast<GemmSmem<SH, MODE> *>(smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u));
  const int warp = int(warp_uniform(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const Bounds bounds{&sm.abort, p.ws};
  // Programmatic dependent launch, both ways: what is queued behind this kernel with that attribute may become
  // resident as this grid's CTAs leave, and this kernel's own set-up below (barriers, tensor memory, the tensor
  // maps in its parameters) may run under the tail of the kernel before it; nothing in global memory is touched
  // before pdl_wait.
  pdl_launch_dependents();

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStagesG; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    for (int i = 0; i < kAcc; ++i) {
      mbar_init(&sm.tmem_full[i], 1);
      mbar_init(&sm.tmem_empty[i], kEpilogueWarps);
    }
    mbar_init(&sm.drained, 1);
    sm.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // the MMA warp owns tensor memory
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sm.tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  pdl_wait();  // the operands, the scales and the output buffer belong to this kernel from here on
  const uint32_t tmem = warp_uniform(sm.tmem_base);
  const int total_tiles = p.m_tiles * p.n_tiles;

  if (warp == 0) {
    // ---- producer: the warp walks the loop, the elected lane issues ------------------------------------
    uint32_t stage = 0, phase = 0;  // `phase`: parity of the current pass over the ring of stages
    bool first_pass = true, ok = true;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
      int mt, nt;
      tile_coords(tile, p.m_tiles, p.n_tiles, &mt, &nt);
      for (int ks = 0; ks < p.k_stages; ++ks) {
        // the MMAs that read this stage's previous contents (one pass ago) must have finished
        if (!first_pass && !mbar_wait_warp(&sm.empty[stage], phase ^ 1u, bounds)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          // a whole box always arrives: rows, columns and scale atoms past the end of the arrays come as zeros
          mbar_expect_tx(&sm.full[stage],
                         kBM * kBK + kBN * kBK + (Format<MODE>::kScaled ? (1 + kAtomsB) * kKAtoms * 512 : 0));
          tma_load_2d(sm.a[stage], &map_a, ks * kBK, mt * kBM, &sm.full[stage]);
          tma_load_2d(sm.b[stage], &map_b, ks * kBK, nt * kBN, &sm.full[stage]);
          if constexpr (Format<MODE>::kScaled) {  // one box each: A's atoms along K; B's for kAtomsB rows of atoms
            tma_load_3d(sm.sfa[stage], &map_sfa, 0, ks * kKAtoms, mt, &sm.full[stage]);
            tma_load_3d(sm.sfb[stage], &map_sfb, 0, ks * kKAtoms, nt * kAtomsB, &sm.full[stage]);
          }
        }
        __syncwarp();
        if (++stage == kStagesG) {
          stage = 0;
          phase ^= 1u;
          first_pass = false;
        }
      }
    }
    if (!ok && lane == 0) {
      // Give up, but not with copies on their way into this CTA's shared memory: wait (bounded) for the newest
      // copy of every stage (this pass's below `stage`, the previous pass's from there on); they complete
      // without anybody's help.
      bounds.give_up();
      for (uint32_t j = 0; j < uint32_t(kStagesG); ++j) {
        if (j < stage) mbar_drain(&sm.full[j], phase);
        else if (!first_pass) mbar_drain(&sm.full[j], phase ^ 1u);
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer: the warp walks the loop, the elected lane issues ---------------------------------------
    uint32_t stage = 0, phase = 0;
    int local_tile = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++local_tile) {
      // the epilogue must have taken this accumulator's previous tile out of tensor memory
      const int acc = local_tile % kAcc, use = local_tile / kAcc;
      if (use > 0 && !mbar_wait_warp(&sm.tmem_empty[acc], (use - 1) & 1u, bounds)) {
        ok = false;
        break;
      }
      tmem_fence_after();
      const uint32_t d_tmem = tmem + uint32_t(acc * kBN);
      for (int ks = 0; ks < p.k_stages; ++ks) {
        if (!mbar_wait_warp(&sm.full[stage], phase, bounds)) {
          ok = false;
          break;
        }
        tmem_fence_after();
        if (elect_one()) {
          // this stage's scales: shared memory -> tensor memory, ordered before the MMAs below.  Tensor-memory
          // columns: A's atom j along K at kSfaCol + 4 j; B's at kSfbCol + j * 4 kAtomsB + 4 h (h = 128 tile columns)
          if constexpr (Format<MODE>::kScaled) {
#pragma unroll
            for (int j = 0; j < kKAtoms; ++j) {
              copy_scale_atom<false>(tmem + kSfaCol + 4 * j, smem_addr(sm.sfa[stage] + j * 512));
#pragma unroll
              for (int h = 0; h < kAtomsB; ++h)
                copy_scale_atom<false>(tmem + kSfbCol + j * 4 * kAtomsB + 4 * h,
                                       smem_addr(sm.sfb[stage] + (h * kKAtoms + j) * 512));
            }
          }
          const uint32_t a_addr = smem_addr(sm.a[stage]), b_addr = smem_addr(sm.b[stage]);
          const uint32_t live = live_k(ks, p.k_stages, p.last_k);
#pragma unroll
          for (uint32_t k = 0; k < 4; ++k) {  // four instructions of 32 operand bytes inside the 128-byte swizzle span
            if (k >= live) break;
            const uint32_t accumulate = (ks > 0 || k > 0) ? 1u : 0u;
            const uint32_t j = Format<MODE>::k_atom(k), id = Format<MODE>::sf_id(k);
            issue_mma<MODE, false>(d_tmem, operand_desc(a_addr + k * 32), operand_desc(b_addr + k * 32),
                                  instr_desc(id, kBN, kBM, Format<MODE>::kFormatBits | p.rowwise.operand_format_bits), accumulate,
                                  (tmem + kSfaCol + 4 * j) | (id << 30), (tmem + kSfbCol + j * 4 * kAtomsB) | (id << 30));
          }
          umma_commit(&sm.empty[stage]);  // the stage is free once these MMAs have read it
        }
        __syncwarp();
        if (++stage == kStagesG) {
          stage = 0;
          phase ^= 1u;
        }
      }
      // the accumulator is complete once all MMAs so far have finished
      if (ok && elect_one()) umma_commit(&sm.tmem_full[acc]);
      __syncwarp();
    }
    if (!ok && lane == 0) {
      bounds.give_up();
    }
  } else {
    // ---- epilogue: 8 warps; warp w reads lanes 32 (w % 4) .. + 31, column half (w - 2) / 4 -------------------
    const int quad = warp & 3, half = (warp - 2) >> 2;
    constexpr int kHalfCols = kBN / 2, kChunks = kHalfCols / 32;  // each warp takes half the tile's columns, 32 at a time
    int local_tile = 0;
    for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++local_tile) {
      int mt, nt;
      tile_coords(tile, p.m_tiles, p.n_tiles, &mt, &nt);
      const int acc = local_tile % kAcc, use = local_tile / kAcc;
      const int64_t row = int64_t(mt) * kBM + quad * 32 + lane;
      RowwiseRegs<kChunks> rw;
      if constexpr (MODE == kRowwise)
        load_rowwise<kChunks>(rw, p.rowwise, row, int64_t(nt) * kBN + half * kHalfCols, lane, p.M, p.N);
      if (!mbar_wait_warp(&sm.tmem_full[acc], use & 1u, bounds)) {
        if (lane == 0) {
          bounds.give_up();
        }
        break;
      }
      tmem_fence_after();
      uint32_t packed[kChunks][16];  // this thread's columns of one row as bf16 pairs
#pragma unroll
      for (int c = 0; c < kChunks; c += 2) {  // two loads in flight per wait: the accumulator is handed back sooner
        uint32_t v[2][32];
        const uint32_t taddr = tmem + (uint32_t(quad * 32) << 16) + uint32_t(acc * kBN + half * kHalfCols + c * 32);
        tmem_load_32(v[0], taddr);
        tmem_load_32(v[1], taddr + 32);
        tmem_load_wait(v[0]);
        tmem_load_wait(v[1]);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if constexpr (MODE == kRowwise) apply_rowwise(v[u], rw.xs, rw.cs[c + u], rw.bs[c + u], rw.has_bias);
#pragma unroll
          for (int i = 0; i < 16; ++i) packed[c + u][i] = pack_bf16(v[u][2 * i], v[u][2 * i + 1]);
        }
      }
      // the accumulator is in registers: hand tensor memory back before storing
      tmem_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.tmem_empty[acc]);
      const int64_t col0 = int64_t(nt) * kBN + half * kHalfCols;
#pragma unroll
      for (int c = 0; c < kChunks; ++c) store_chunk(sm.out[warp - 2], packed[c], p.out, row - lane, col0 + c * 32, p.M, p.N, lane);
    }
  }

  // ---- teardown: everybody meets, then the warp that allocated tensor memory frees it ----------------------
  tmem_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*bounds.abort && elect_one()) {  // the lane that issued the MMAs: a commit follows the issuing thread's own
      // MMAs may still be in flight: a commit that arrives on a barrier nobody else uses, and a bounded wait for it
      umma_commit(&sm.drained);
      mbar_drain(&sm.drained, 0u);
    }
    __syncwarp();
    tmem_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// ---- two SMs on one tile ----------------------------------------------------------------------------------
// The kernel above is bound by what one SM can pull out of L2 (about 64 bytes per clock): a 128 x 256 tile
// needs 48 KB of operands per 128 of K.  Here two CTAs of a cluster (an SM pair) share a 256 x 256 tile:
// tcgen05.mma.cta_group::2 multiplies M = 256 (each CTA supplies 128 rows of A and receives their 128 x 256
// accumulator in its own tensor memory) by N = 256 (each CTA supplies 128 of the 256 rows of B), so every CTA
// loads 16 + 16 KB per stage instead of 16 + 32: a third less traffic per flop, and room for 6 stages.
//   * both CTAs' producers load their own halves (TMA, .cta_group::2, each CTA for itself) and signal the LEADER
//     CTA's `full` barrier (the even CTA of the pair); the leader alone expects the bytes of both;
//   * the scale atoms come in through a 3-D tensor map over the blocked scale array ([atom row][atom column]
//     [512 bytes]), so that a missing atom is simply filled with zeros; every CTA needs its own A atom and
//     both B atoms (its accumulator spans all 256 columns);
//   * the leader's MMA thread copies the scales (tcgen05.cp.cta_group::2: each CTA's shared memory into that
//     CTA's tensor memory), issues the MMAs, and commits to both CTAs' copies of a barrier at once;
//   * two accumulators alternate, so that the tensor cores work on the next tile while the epilogue empties this one
//     (see PairTmem); the peer's epilogue warps arrive on the leader's `tmem_empty` barriers through the cluster
//     address space.
// Every wait is bounded as above; an abort is forwarded to the other CTA, and both always meet at the cluster
// barrier before tensor memory is freed.
template <int MODE>
constexpr int PairStages = MODE == kMxFp4 ? 5 : 6;  // what fits beside the output staging (MXFP4 has twice the scale atoms)
constexpr int kPairBN = 256;  // tile columns; each CTA holds kPairBN / 2 rows of B

// Tensor memory of the pair kernel: two accumulators of 256 columns.  Without block scales they fill the 512 columns
// exactly.  With block scales 24 columns are needed beside them, so the second accumulator starts 32 columns early and
// shares columns 224..255 with the first: the MMAs of a tile may start as soon as the epilogue has taken those 32
// columns of the tile BEFORE it (which it reads first) and all of the tile before that.
// With one accumulator the tensor cores stood still for about 3 us per tile, from the last MMA of a tile until all of it
// had been read.  Measured (one against two, B200, steady state): MXFP4 2000 x 12288 x 4096 with its cast 65.6 -> 59.6 us,
// row-wise 32768 x 4096 x 4096 with its quantization 587 -> 547 us; an MXFP8 training step at 8192^3 stays at 1.57-1.59 ms,
// because the board's power limit sets its clock and busier tensor cores run at a lower one.
template <int MODE>
struct PairTmem {
  static constexpr bool kShared = Format<MODE>::kScaled;
  static constexpr int kAcc1 = kShared ? 224 : 256;  // first column of the second accumulator
  static constexpr int kSfa = 480, kSfb = 488;       // scales: A 4 columns per atom along K, B 8
};

template <int MODE>
struct __align__(1024) PairSmem {
  uint8_t a[PairStages<MODE>][kBM * kBK];             // this CTA's 128 rows of A
  uint8_t b[PairStages<MODE>][kPairBN / 2 * kBK];     // this CTA's 128 of the tile's 256 rows of B
  // scales of this CTA's 128 rows of A, and of all 256 rows of B ([128 columns][atom along K]); one dummy without block scales
  uint8_t sfa[Format<MODE>::kScaled ? PairStages<MODE> : 1][Format<MODE>::kKAtoms * 512];
  uint8_t sfb[Format<MODE>::kScaled ? PairStages<MODE> : 1][2 * Format<MODE>::kKAtoms * 512];
  alignas(512) uint8_t out[kEpilogueWarps][32 * 64];  // per epilogue warp 32 rows x 32 bf16 on their way out (64-byte swizzle)
  float scales[MODE == kRowwise ? kEpilogueWarps : 1][2][128];  // per epilogue warp its columns' scales and biases (row-wise)
  uint64_t full[PairStages<MODE>];               // used in the leader CTA only
  uint64_t empty[PairStages<MODE>];
  uint64_t tmem_full[2];                         // one per accumulator
  uint64_t tmem_empty[2];                        // used in the leader CTA only
  uint32_t tmem_base;
  int abort;
};

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA loads of the pair kernel: destination in this CTA, completion counted on a barrier given by its cluster address.
__device__ __forceinline__ void tma_pair_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_pair_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z,
                                                 uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
          smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// All MMAs issued so far, once done, arrive on the barrier at this offset in BOTH CTAs of the pair.
__device__ __forceinline__ void umma_commit_pair(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   smem_addr(bar)),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}

// TMA store of a box of the output from shared memory (bulk group of the issuing thread), and the waits for it.
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, const void *src, int x, int y, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group.L2::cache_hint [%0, {%2, %3}], [%1], %4;\n\t"
      "cp.async.bulk.commit_group;" ::"l"(reinterpret_cast<uint64_t>(map)),
      "r"(smem_addr(src)), "r"(x), "r"(y), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

struct PairParams {
  RowwiseEpilogue rowwise;
  int M, N;
  int m_pairs, n_tiles, k_stages;  // 256-row tile rows, 256-column tile columns, 128-byte K stages
  int last_k;                      // see live_k
  Workspace *ws;
};

template <int MODE>
__global__ void __launch_bounds__(kGemmThreads, 1)
mx_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ CUtensorMap map_sfa, const __grid_constant__ CUtensorMap map_sfb,
                    const __grid_constant__ CUtensorMap map_out, PairParams p, LaunchPad<kGemmParameterBytes<5, PairParams>>) {
  constexpr int kKAtoms = Format<MODE>::kKAtoms, kPairStages = PairStages<MODE>;
  extern __shared__ unsigned char smem_raw[];
  PairSmem<MODE> &sm = *reinterpret_cast<PairSmem<MODE> *>(smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u));
  const int warp = int(warp_uniform(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const uint32_t rank = warp_uniform(cluster_ctarank());  // 0 = leader
  const bool leader = rank == 0;
  const uint32_t peer = rank ^ 1u;
  const Bounds bounds{&sm.abort, p.ws};
  const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
  const int total_tiles = p.m_pairs * p.n_tiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kPairStages; ++s) {
      mbar_init(&sm.full[s], 1);   // the leader's producer arrives once, expecting both CTAs' bytes
      mbar_init(&sm.empty[s], 1);  // one commit of the leader's MMA thread per CTA
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sm.tmem_full[i], 1);
      mbar_init(&sm.tmem_empty[i], 2 * kEpilogueWarps);  // the epilogue warps of both CTAs
    }
    sm.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // one warp of each CTA, together: 512 columns in both CTAs' tensor memory
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sm.tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tmem_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anybody signals them
  tmem_fence_after();
  pdl_wait();
  const uint32_t tmem = warp_uniform(sm.tmem_base);

  if (warp == 0) {
    // ---- producer (in each CTA): the warp walks the loop, the elected lane issues ------------------------------
    uint32_t stage = 0, phase = 0;
    bool first_pass = true, ok = true;
    for (int tile = cluster_id; tile < total_tiles && ok; tile += n_clusters) {
      int mp, nt;
      tile_coords(tile, p.m_pairs, p.n_tiles, &mp, &nt);
      // What is queued behind this kernel may become resident once every CTA has come to its last tile, and not at once as in
      // the other kernels: a cast that becomes resident asks for its first tiles (prefetch_first_tile), and at the start of a
      // large product that took memory from the first operands, for lines that the product was about to write.  Measured, MXFP8
      // product and an operation on its output, us, released at once / here: 2000 x 12288 x 4096 product alone 78.0 / 77.5, static
      // cast 89.1 / 88.9, MX cast 90.8 / 90.0, amax 89.2 / 87.8, amax and both casts 106.5 / 104.1; 8192 x 4096 x 1024: 33.2 / 33.1, 47.0 / 46.7,
      // 49.4 / 48.7, 45.0 / 43.4, 69.6 / 66.6; 3000 x 8192 x 2048: 44.2 / 43.9, 54.7 / 54.4, 56.1 / 55.3, 56.2 / 54.4, 80.4 / 77.7.  Later still, with
      // eight stages of the last tile left, the operations gain up to 2 us more, but a product behind a product starts too late
      // where the last round of tiles leaves SMs idle: 2000 x 12288 x 4096 80.1.
      if (tile + n_clusters >= total_tiles) pdl_launch_dependents();
      for (int ks = 0; ks < p.k_stages; ++ks) {
        if (!first_pass && !mbar_wait_warp(&sm.empty[stage], phase ^ 1u, bounds)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          const uint32_t bar = map_to_cta(smem_addr(&sm.full[stage]), 0);  // the leader's barrier
          if (leader)
            mbar_expect_tx(&sm.full[stage],
                           2 * (kBM * kBK + kPairBN / 2 * kBK + (Format<MODE>::kScaled ? 3 * kKAtoms * 512 : 0)));
          tma_pair_load_2d(sm.a[stage], &map_a, ks * kBK, mp * 256 + int(rank) * kBM, bar);
          tma_pair_load_2d(sm.b[stage], &map_b, ks * kBK, nt * kPairBN + int(rank) * (kPairBN / 2), bar);
          if constexpr (Format<MODE>::kScaled) {
            tma_pair_load_3d(sm.sfa[stage], &map_sfa, 0, ks * kKAtoms, mp * 2 + int(rank), bar);
            tma_pair_load_3d(sm.sfb[stage], &map_sfb, 0, ks * kKAtoms, nt * 2, bar);
          }
        }
        __syncwarp();
        if (++stage == kPairStages) {
          stage = 0;
          phase ^= 1u;
          first_pass = false;
        }
      }
    }
    if (!ok && lane == 0) {
      bounds.give_up();
      st_cluster_u32(map_to_cta(smem_addr(&sm.abort), peer), 1u);
    }
  } else if (warp == 1) {
    // ---- MMA issuer: the leader's warp walks the loop, its elected lane drives both SMs' tensor cores ---------
    if (leader) {
      uint32_t stage = 0, phase = 0;
      int local_tile = 0;
      bool ok = true;
      for (int tile = cluster_id; tile < total_tiles && ok; tile += n_clusters, ++local_tile) {
        // shared columns: wait for the previous tile's (its epilogue has then also emptied the accumulator used here, two
        // tiles ago); separate accumulators: for the tile two before this one
        constexpr int kBack = PairTmem<MODE>::kShared ? 1 : 2;
        const int before = local_tile - kBack;
        if (before >= 0 && !mbar_wait_warp(&sm.tmem_empty[before & 1], (before >> 1) & 1u, bounds)) {
          ok = false;
          break;
        }
        tmem_fence_after();
        const uint32_t d_tmem = tmem + ((local_tile & 1) ? PairTmem<MODE>::kAcc1 : 0);
        for (int ks = 0; ks < p.k_stages; ++ks) {
          if (!mbar_wait_warp(&sm.full[stage], phase, bounds)) {
            ok = false;
            break;
          }
          tmem_fence_after();
          if (elect_one()) {
            if constexpr (Format<MODE>::kScaled) {
#pragma unroll
              for (int j = 0; j < kKAtoms; ++j) {  // each CTA's shared memory -> that CTA's tensor memory, columns as above
                copy_scale_atom<true>(tmem + PairTmem<MODE>::kSfa + 4 * j, smem_addr(sm.sfa[stage] + j * 512));
#pragma unroll
                for (int h = 0; h < 2; ++h)
                  copy_scale_atom<true>(tmem + PairTmem<MODE>::kSfb + j * 8 + 4 * h,
                                        smem_addr(sm.sfb[stage] + (h * kKAtoms + j) * 512));
              }
            }
            const uint32_t a_addr = smem_addr(sm.a[stage]), b_addr = smem_addr(sm.b[stage]);
            const uint32_t live = live_k(ks, p.k_stages, p.last_k);
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
              if (k >= live) break;
              const uint32_t accumulate = (ks > 0 || k > 0) ? 1u : 0u;
              const uint32_t j = Format<MODE>::k_atom(k), id = Format<MODE>::sf_id(k);
              issue_mma<MODE, true>(d_tmem, operand_desc(a_addr + k * 32), operand_desc(b_addr + k * 32),
                                   instr_desc(id, kPairBN, 256, Format<MODE>::kFormatBits | p.rowwise.operand_format_bits),
                                   accumulate, (tmem + PairTmem<MODE>::kSfa + 4 * j) | (id << 30),
                                   (tmem + PairTmem<MODE>::kSfb + j * 8) | (id << 30));
            }
            umma_commit_pair(&sm.empty[stage]);  // the stage is free in both CTAs once these MMAs have read it
          }
          __syncwarp();
          if (++stage == kPairStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        // both CTAs' halves of the accumulator are complete once all MMAs so far have finished
        if (ok && elect_one()) umma_commit_pair(&sm.tmem_full[local_tile & 1]);
        __syncwarp();
      }
      if (!ok && lane == 0) {
        bounds.give_up();
        st_cluster_u32(map_to_cta(smem_addr(&sm.abort), peer), 1u);
      }
    }
  } else {
    // ---- epilogue: this CTA's 128 rows of the tile, 8 warps as in the single-CTA kernel --------------------
    // A warp's 128 columns go 32 at a time, the next 32 on their way from tensor memory while these are converted and
    // staged in shared memory, from where a TMA store takes them (which also cuts off what lies past the edges).  With
    // stores from registers a lane owned a row, a warp's store touched 32 lines, and the epilogue took longer than the
    // MMAs of 1024 bytes of K; see launch_pair for the figures.
    // The half that holds the shared columns starts with them: half 1 at its end (columns 255..224 of the first
    // accumulator), half 0 at its beginning (columns 0..31 of the second, the same columns of tensor memory).
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const uint32_t leader_empty[2] = {map_to_cta(smem_addr(&sm.tmem_empty[0]), 0), map_to_cta(smem_addr(&sm.tmem_empty[1]), 0)};
    // The last tile's 32 columns each have a buffer of their own: the operands' stages are free by then.  A tile before takes
    // one buffer four times, and waits each time until the store before has read it, behind the loads of the next tile.  Us, one buffer ->
    // four: MXFP8 2048^3 10.3 -> 9.9, 3000 x 2000 x 1504 13.3 -> 12.9, 8192^3 429 -> 428; row-wise, whose conversion takes longer, within 1 %.
    uint8_t *const last_staging = sm.a[0] + (warp - 2) * (4 * 32 * 64);
    static_assert(kEpilogueWarps * 4 * 32 * 64 <= PairStages<MODE> * kBM * kBK, "the operands of A have the room");
    const uint64_t stream_policy = l2_policy_evict_first();  // the output must not push the operands out of L2
    int local_tile = 0;
    for (int tile = cluster_id; tile < total_tiles; tile += n_clusters, ++local_tile) {
      int mp, nt;
      tile_coords(tile, p.m_pairs, p.n_tiles, &mp, &nt);
      const int64_t row = int64_t(mp) * 256 + int64_t(rank) * kBM + quad * 32 + lane;
      const int64_t col0 = int64_t(nt) * kPairBN + half * 128;
      const int acc = local_tile & 1;
      const bool last = tile + n_clusters >= total_tiles;
      float xs = 0.0f;
      if constexpr (MODE == kRowwise) {
        // before the wait: the row's scale, and the columns' scales and biases to shared memory, read there by all lanes
        RowwiseRegs<4> rw;
        load_rowwise<4>(rw, p.rowwise, row, col0, lane, p.M, p.N);
        xs = rw.xs;
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          sm.scales[warp - 2][0][c * 32 + lane] = rw.cs[c];
          sm.scales[warp - 2][1][c * 32 + lane] = rw.bs[c];
        }
        __syncwarp();
      }
      if (!mbar_wait_warp(&sm.tmem_full[acc], (local_tile >> 1) & 1u, bounds)) {
        if (lane == 0) {
          bounds.give_up();
          st_cluster_u32(map_to_cta(smem_addr(&sm.abort), peer), 1u);
        }
        break;
      }
      tmem_fence_after();
      const uint32_t taddr = tmem + (uint32_t(quad * 32) << 16) + uint32_t((acc ? PairTmem<MODE>::kAcc1 : 0) + half * 128);
      // the i-th 32 columns of this warp in the order it takes them
      auto chunk_at = [&](int i) { return PairTmem<MODE>::kShared && half ? 3 - i : i; };
      // handed back after the shared columns (the other half has none to wait for) or after everything
      const int release_after = PairTmem<MODE>::kShared ? (half == acc ? -1 : 0) : 3;
      auto hand_back = [&] {
        tmem_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(acc ? leader_empty[1] : leader_empty[0]);
      };
      if (release_after < 0) hand_back();
      uint32_t v[2][32];
      tmem_load_32(v[0], taddr + chunk_at(0) * 32);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        tmem_load_wait(v[i & 1]);
        if (i == release_after) hand_back();
        if (i < 3) tmem_load_32(v[(i + 1) & 1], taddr + chunk_at(i + 1) * 32);
        const int c = chunk_at(i);
        if constexpr (MODE == kRowwise)
          apply_rowwise_shared(v[i & 1], xs, &sm.scales[warp - 2][0][c * 32], p.rowwise.bias ? &sm.scales[warp - 2][1][c * 32] : nullptr);
        uint32_t packed[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) packed[j] = pack_bf16(v[i & 1][2 * j], v[i & 1][2 * j + 1]);
        uint8_t *const staging = last ? last_staging + i * (32 * 64) : sm.out[warp - 2];
        if (!last) {
          if (lane == 0) tma_store_wait_read();  // the staging buffer has been read
          __syncwarp();
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          *reinterpret_cast<uint4 *>(staging + lane * 64 + ((q ^ ((lane >> 1) & 3)) * 16)) =
              make_uint4(packed[4 * q], packed[4 * q + 1], packed[4 * q + 2], packed[4 * q + 3]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0 && row < p.M && col0 + c * 32 < p.N)
          tma_store_2d(&map_out, staging, static_cast<int>(col0) + c * 32, static_cast<int>(row), stream_policy);
      }
    }
    if (lane == 0) tma_store_wait_all();
  }

  // ---- teardown ---------------------------------------------------------------------------------------------
  // whoever gave up has already raised both CTAs' abort flags
  tmem_fence_before();
  __syncthreads();
  if (*bounds.abort) {
    // Copies and MMAs may still be in flight into or out of this CTA's memories.  Loads complete by themselves
    // within microseconds and the leader's MMAs within a tile's time; neither CTA leaves before the other
    // (cluster barrier below), and a short sleep here covers what was issued last.
    __nanosleep(200000);
  }
  cluster_sync_all();  // nobody's shared or tensor memory goes away while the other CTA may still touch it
  if (warp == 1) {
    tmem_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// ---- few output tiles: weights as the M operand, K split over a cluster ------------------------------------
// A decode step multiplies a handful of token rows with all the weights: bound by reading B once.  The kernels above
// give it one CTA per 128 or 256 rows of B (64 CTAs for 8192 outputs, less than half of the SMs, 64 stages of K one after
// the other).  Here
//   * the roles are swapped: 128 rows of B are the MMA's M operand and the tokens its N operand (32, 64 or 128 wide), so
//     a stage carries 16 KB of weights and only as many token rows as there are;
//   * the CTAs of a cluster (1, 2, 4 or 8) take consecutive ranges of the K stages of one tile; two CTAs fit an SM, with
//     up to 160 KB of weights on their way per SM;
//   * partial sums (fp32) go to each CTA's own shared memory, and after a cluster barrier every CTA adds up all CTAs'
//     partials of its share of the tokens through distributed shared memory, in the order of K;
//   * while the kernel before this one drains, the first stages of weights are already asked into L2: that is where this
//     GPU's memory is coherent, so it does not matter whether that kernel still writes them.
// Measured (B200, products back to back, weights not in L2, 8 stages asked ahead at that time; 128 x 128 kernel -> this one; reading the weights
// alone at the measured copy rate): 8 x 8192 x 8192 MXFP8 27.9 -> 13.6 us (10.3), 16 x 8192 x 4096 row-wise 15.4 -> 8.5 (5.1),
// 16 x 256 x 8192 16.5 -> 5.0, 300 x 2048 x 8192 19.4 -> 14.3.
constexpr int kSplitThreads = 192;   // producer warp, MMA warp, 4 warps that empty tensor memory; all six add up and store
constexpr int kSplitWarps = kSplitThreads / 32;
constexpr int kMaxSplits = 8;        // portable cluster size
// Stages of weights asked into L2 ahead of the dependency.  Few: the kernel that the dependency waits for (the cast of the
// tokens) reads through the same memory, and it is what everybody waits for; but that cast asks for its tokens ahead of its own
// wait (asks_ahead in dtq_host.h).  Cast and product, us, with 2 / 3 / 4 stages:
//   tokens x N x K        MXFP8                    MXFP4                    row-wise
//    16 x 8192 x 4096     11.17 / 10.98 / 10.78     9.17 /  9.00 /  8.85    10.69 / 10.54 / 10.46
//    64 x 8192 x 4096     12.79 / 12.68 / 12.64    10.11 / 10.13 / 10.13    12.70 / 12.56 / 12.52
//    16 x 8192 x 8192     16.67 / 16.76 / 16.98    11.56 / 11.36 / 11.15    16.22 / 16.46 / 16.81
//    64 x 8192 x 8192     18.22 / 18.25 / 18.62    13.15 / 13.03 / 12.98    18.12 / 18.25 / 18.53
//   128 x 8192 x 8192     21.24 / 21.32 / 21.57    15.81 / 15.66 / 15.59    20.83 / 20.93 / 21.22
//    16 x 16384 x 8192    27.44 / 27.36 / 27.21    17.12 / 17.04 / 17.13    26.90 / 26.70 / 26.65
//    64 x 4096 x 16384    19.02 / 19.23 / 19.73    13.82 / 13.79 / 13.70    19.34 / 19.65 / 20.09
// None / eight: MXFP8 8 x 8192 x 8192 16.9 / 17.2, row-wise 16 x 8192 x 4096 11.5 / 10.8.  Three for the row-wise product because
// with four 64 x 8192 x 8192 was behind two without the cast's asking (18.53 against 18.37).
template <int MODE>
constexpr int kSplitPrefetch = MODE == kMxFp8 ? 2 : (MODE == kRowwise ? 3 : 4);

template <int BN, int STAGES, int MODE>
struct __align__(1024) SplitSmem {
  uint8_t w[STAGES][kBM * kBK];  // 128 rows of weights; with x, reused for the fp32 partial sums [token][128]
  uint8_t x[STAGES][BN * kBK];   // the tile's tokens
  uint8_t sfw[STAGES][Format<MODE>::kKAtoms * 512];
  uint8_t sfx[STAGES][Format<MODE>::kKAtoms * 512];
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t tmem_full;
  uint64_t drained;  // as in GemmSmem
  uint32_t tmem_base;
  int abort;
};

struct SplitParams {
  RowwiseEpilogue rowwise;
  uint16_t *out;  // bf16 [M, N]
  int M, N;
  int n_tiles, k_stages, splits;  // 128-column tiles of the output, 128-byte K stages, CTAs per cluster
  int last_k;                     // see live_k
  Workspace *ws;
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t cluster_addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(cluster_addr) : "memory");
  return v;
}
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap *map, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y)
               : "memory");
}

template <int BN, int STAGES, int MODE>
__global__ void __launch_bounds__(kSplitThreads, 2)
mx_gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                     const __grid_constant__ CUtensorMap map_sfw, const __grid_constant__ CUtensorMap map_sfx, SplitParams p,
                     LaunchPad<kGemmParameterBytes<4, SplitParams>>) {
  using Smem = SplitSmem<BN, STAGES, MODE>;
  static_assert(BN * kBM * 4 <= STAGES * (kBM + BN) * kBK, "partial sums fit the stage buffers");
  constexpr int kKAtoms = Format<MODE>::kKAtoms;
  constexpr uint32_t kSfw = BN, kSfx = BN + 8;             // tensor-memory columns of the scales (4 per atom)
  constexpr uint32_t kCols = BN == 32 ? 64 : 2 * BN;       // two CTAs' columns fit an SM's 512
  extern __shared__ unsigned char smem_raw[];
  Smem &sm = *reinterpret_cast<Smem *>(smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u));
  const int warp = int(warp_uniform(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const int rank = int(warp_uniform(cluster_ctarank()));
  const Bounds bounds{&sm.abort, p.ws};
  const int tile = blockIdx.x / p.splits;
  const int nt = tile % p.n_tiles, tt = tile / p.n_tiles;
  const int k0 = int(int64_t(p.k_stages) * rank / p.splits), k1 = int(int64_t(p.k_stages) * (rank + 1) / p.splits);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    mbar_init(&sm.tmem_full, 1);
    mbar_init(&sm.drained, 1);
    sm.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int ks = k0; ks < k1 && ks < k0 + kSplitPrefetch<MODE>; ++ks) tma_prefetch_2d(&map_w, ks * kBK, nt * kBM);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sm.tmem_base)), "r"(kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  // only now that this CTA has its tensor memory may a dependent's CTA become resident beside it and take some
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t tmem = warp_uniform(sm.tmem_base);

  if (warp == 0) {
    // ---- producer ------------------------------------------------------------------------------------------
    uint32_t stage = 0, phase = 0;
    bool first_pass = true, ok = true;
    for (int ks = k0; ks < k1; ++ks) {
      if (!first_pass && !mbar_wait_warp(&sm.empty[stage], phase ^ 1u, bounds)) {
        ok = false;
        break;
      }
      if (elect_one()) {
        mbar_expect_tx(&sm.full[stage], kBM * kBK + BN * kBK + (Format<MODE>::kScaled ? 2 * kKAtoms * 512 : 0));
        tma_load_2d(sm.w[stage], &map_w, ks * kBK, nt * kBM, &sm.full[stage]);
        tma_load_2d(sm.x[stage], &map_x, ks * kBK, tt * BN, &sm.full[stage]);
        if constexpr (Format<MODE>::kScaled) {
          tma_load_3d(sm.sfw[stage], &map_sfw, 0, ks * kKAtoms, nt, &sm.full[stage]);
          tma_load_3d(sm.sfx[stage], &map_sfx, 0, ks * kKAtoms, tt, &sm.full[stage]);  // tt > 0 only with BN = 128
        }
      }
      __syncwarp();
      if (++stage == STAGES) {
        stage = 0;
        phase ^= 1u;
        first_pass = false;
      }
    }
    if (!ok && lane == 0) {  // as in the single-CTA kernel: no copies left on their way when the CTA leaves
      bounds.give_up();
      for (uint32_t j = 0; j < uint32_t(STAGES); ++j) {
        if (j < stage) mbar_drain(&sm.full[j], phase);
        else if (!first_pass) mbar_drain(&sm.full[j], phase ^ 1u);
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer ------------------------------------------------------------------------------------------
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int ks = k0; ks < k1; ++ks) {
      if (!mbar_wait_warp(&sm.full[stage], phase, bounds)) {
        ok = false;
        break;
      }
      tmem_fence_after();
      if (elect_one()) {
        if constexpr (Format<MODE>::kScaled) {
#pragma unroll
          for (int j = 0; j < kKAtoms; ++j) {
            copy_scale_atom<false>(tmem + kSfw + 4 * j, smem_addr(sm.sfw[stage] + j * 512));
            copy_scale_atom<false>(tmem + kSfx + 4 * j, smem_addr(sm.sfx[stage] + j * 512));
          }
        }
        const uint32_t w_addr = smem_addr(sm.w[stage]), x_addr = smem_addr(sm.x[stage]);
        const uint32_t live = live_k(ks, p.k_stages, p.last_k);
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
          if (k >= live) break;
          const uint32_t accumulate = (ks > k0 || k > 0) ? 1u : 0u;
          const uint32_t j = Format<MODE>::k_atom(k), id = Format<MODE>::sf_id(k);
          issue_mma<MODE, false>(tmem, operand_desc(w_addr + k * 32), operand_desc(x_addr + k * 32),
                                 instr_desc(id, BN, kBM, Format<MODE>::kFormatBits | p.rowwise.operand_format_bits), accumulate,
                                 (tmem + kSfw + 4 * j) | (id << 30), (tmem + kSfx + 4 * j) | (id << 30));
        }
        umma_commit(&sm.empty[stage]);
      }
      __syncwarp();
      if (++stage == STAGES) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if (ok && elect_one()) umma_commit(&sm.tmem_full);
    __syncwarp();
    if (!ok && lane == 0) {
      bounds.give_up();
    }
  }

  // ---- partial sums: tensor memory -> this CTA's shared memory [token][128 outputs] -------------------------
  float *partial = reinterpret_cast<float *>(sm.w);
  const int live = min(BN, p.M - tt * BN);  // tokens of this tile
  const int64_t n0 = int64_t(nt) * kBM + lane * 4;  // this lane's four outputs in the sum below; N % 8 == 0
  const bool n_live = n0 < p.N;
  float4 cs = make_float4(0.0f, 0.0f, 0.0f, 0.0f), bs = cs;
  if constexpr (MODE == kRowwise) {
    if (n_live) {  // fetched before the wait below
      const float *c = p.rowwise.col_scale + n0;
      cs = make_float4(__ldg(c), __ldg(c + 1), __ldg(c + 2), __ldg(c + 3));
      if (p.rowwise.bias) {
        if (p.rowwise.bias_is_bf16) {
          const uint16_t *b = static_cast<const uint16_t *>(p.rowwise.bias) + n0;
          bs = make_float4(bf16_lo(__ldg(b)), bf16_lo(__ldg(b + 1)), bf16_lo(__ldg(b + 2)), bf16_lo(__ldg(b + 3)));
        } else {
          const float *b = static_cast<const float *>(p.rowwise.bias) + n0;
          bs = make_float4(__ldg(b), __ldg(b + 1), __ldg(b + 2), __ldg(b + 3));
        }
      }
    }
  }
  if (warp >= 2) {
    const int quad = warp & 3;  // the quarter of tensor memory that this warp can read
    // the barrier completes when all MMAs have, so nothing reads the stage buffers any more
    if (!mbar_wait_warp(&sm.tmem_full, 0u, bounds)) {
      if (lane == 0) {
        bounds.give_up();
      }
    } else {
      tmem_fence_after();
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) {
        if (c * 32 < live) {
          uint32_t v[32];
          tmem_load_32(v, tmem + (uint32_t(quad * 32) << 16) + uint32_t(c * 32));
          tmem_load_wait(v);
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i < live) partial[(c * 32 + i) * kBM + quad * 32 + lane] = __uint_as_float(v[i]);
        }
      }
      tmem_fence_before();
    }
  }
  __syncwarp();
  cluster_sync_all();

  // ---- sum over the cluster: token t by CTA t % splits, a warp per token, four outputs per lane --------------
  // A CTA that gave up has operand bytes where its partial sums should be: if there is one, nobody in the cluster stores.
  // Lane j asks CTA j, and the answer is looked at behind the first loads of partial sums.
  const uint32_t gave_up = lane < p.splits ? ld_cluster_u32(map_to_cta(smem_addr(&sm.abort), lane)) : 0u;
  for (int t = rank + p.splits * warp; t < live; t += p.splits * kSplitWarps) {
    const uint32_t mine = smem_addr(partial + t * kBM + lane * 4);
    float4 part[kMaxSplits];
#pragma unroll
    for (int j = 0; j < kMaxSplits; ++j)
      if (j < p.splits) part[j] = ld_cluster_f4(map_to_cta(mine, j));
    if (__any_sync(0xFFFFFFFFu, gave_up != 0)) break;
    float4 f = part[0];
#pragma unroll
    for (int j = 1; j < kMaxSplits; ++j)
      if (j < p.splits) f = make_float4(f.x + part[j].x, f.y + part[j].y, f.z + part[j].z, f.w + part[j].w);
    const int64_t row = int64_t(tt) * BN + t;
    if constexpr (MODE == kRowwise) {  // the same steps as apply_rowwise
      const float xs = __ldg(p.rowwise.row_scale + row);
      f = make_float4(__fmul_rn(__fmul_rn(f.x, xs), cs.x), __fmul_rn(__fmul_rn(f.y, xs), cs.y), __fmul_rn(__fmul_rn(f.z, xs), cs.z),
                      __fmul_rn(__fmul_rn(f.w, xs), cs.w));
      if (p.rowwise.bias)
        f = make_float4(__fadd_rn(f.x, bs.x), __fadd_rn(f.y, bs.y), __fadd_rn(f.z, bs.z), __fadd_rn(f.w, bs.w));
    }
    if (n_live)
      stg_stream(p.out + row * p.N + n0,
                 make_uint2(pack_bf16(__float_as_uint(f.x), __float_as_uint(f.y)), pack_bf16(__float_as_uint(f.z), __float_as_uint(f.w))));
  }
  __syncwarp();
  if (warp == 1 && *bounds.abort && elect_one()) {  // MMAs may still be in flight: wait (bounded) for them, as in the single-CTA kernel
    umma_commit(&sm.drained);
    mbar_drain(&sm.drained, 0u);
  }
  __syncwarp();
  cluster_sync_all();  // nobody leaves while another CTA may still read its partial sums
  if (warp == 1) {
    tmem_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
  }
}

// ---- host side --------------------------------------------------------------------------------------------

using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's tensor-map encoder, looked up through the runtime (no link against libcuda).
int encode_tiled_fn(EncodeTiledFn *fn) {
  static std::atomic<EncodeTiledFn> cached{nullptr};
  EncodeTiledFn f = cached.load(std::memory_order_acquire);
  if (!f) {
    void *sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    DTQ_CUDA_TRY(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres));
    if (qres != cudaDriverEntryPointSuccess || !sym) return DTQ_ERR_CUDA_BASE + static_cast<int>(cudaErrorNotSupported);
    f = reinterpret_cast<EncodeTiledFn>(sym);
    cached.store(f, std::memory_order_release);
  }
  *fn = f;
  return DTQ_OK;
}

// Map of a row-major [rows, k_bytes] byte matrix, boxes of box_rows x 128 bytes, 128-byte swizzle, zero fill.
int make_operand_map(CUtensorMap *map, const void *base, int64_t rows, int64_t k_bytes, int box_rows) {
  EncodeTiledFn encode = nullptr;
  if (int e = encode_tiled_fn(&encode)) return e;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k_bytes), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k_bytes)};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(kBK), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t elem_strides[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, elem_strides,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? DTQ_OK : DTQ_ERR_INVALID_ARGUMENT;
}

// Map of the bf16 output [rows, cols] for stores of boxes of 32 x 32 (64-byte swizzle).
int make_output_map(CUtensorMap *map, void *base, int64_t rows, int64_t cols) {
  EncodeTiledFn encode = nullptr;
  if (int e = encode_tiled_fn(&encode)) return e;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * 2};
  const cuuint32_t box[2] = {32, 32};
  const cuuint32_t elem_strides[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, elem_strides,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? DTQ_OK : DTQ_ERR_INVALID_ARGUMENT;
}

// Map of a blocked scale array as [atom rows][atoms along K][512 bytes]: boxes of `box_rows` x `box_katoms` atoms.
// Atoms past the end are delivered as zeros.
int make_scale_map(CUtensorMap *map, const void *base, int64_t atom_rows, int64_t katoms, int box_rows, int box_katoms) {
  EncodeTiledFn encode = nullptr;
  if (int e = encode_tiled_fn(&encode)) return e;
  const cuuint64_t dims[3] = {128, static_cast<cuuint64_t>(katoms), static_cast<cuuint64_t>(atom_rows)};
  const cuuint64_t strides[2] = {512, static_cast<cuuint64_t>(512 * katoms)};
  const cuuint32_t box[3] = {128, static_cast<cuuint32_t>(box_katoms), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t elem_strides[3] = {1, 1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<void *>(base), dims, strides, box, elem_strides,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? DTQ_OK : DTQ_ERR_INVALID_ARGUMENT;
}

constexpr int kMaxGemmDevices = 64;

// The instructions of 32 operand bytes in the last stage of K.
int last_k(int64_t k_bytes) { return static_cast<int>(ceil_div64(k_bytes - (ceil_div64(k_bytes, kBK) - 1) * kBK, 32)); }

// Clusters of `cluster` CTAs, launched as a programmatic dependent of what is before it on the stream (attr: room for two).
void cluster_launch_config(cudaLaunchConfig_t *cfg, cudaLaunchAttribute *attr, int grid, int threads, int cluster, size_t smem,
                           cudaStream_t st) {
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3(grid);
  cfg->blockDim = dim3(threads);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 2;
}

// The SM-pair kernel: clusters of two CTAs, as many as the device can hold at once (at most one CTA per SM).
// *max_clusters (cached per device and format) is 0 where cluster launches of this kernel are not possible.
template <int MODE>
int pair_cluster_capacity(int dev_id, int *max_clusters) {
  static std::atomic<int> known[kMaxGemmDevices];
  if (dev_id < 0 || dev_id >= kMaxGemmDevices) return DTQ_ERR_INVALID_ARGUMENT;
  *max_clusters = clusters_that_fit(known[dev_id], [](int *n) {
    constexpr int smem = smem_bytes<PairSmem<MODE>>();
    const cudaError_t e = cudaFuncSetAttribute(mx_gemm_pair_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    cluster_launch_config(&cfg, attr, 2, kGemmThreads, 2, smem, nullptr);
    cfg.numAttrs = 1;  // the occupancy query wants the cluster shape only
    return cudaOccupancyMaxActiveClusters(n, mx_gemm_pair_kernel<MODE>, &cfg);
  });
  return DTQ_OK;
}

// What every launcher needs: operand pointers, sizes (k_bytes = bytes per operand row), the caller's workspace.
struct GemmCall {
  RowwiseEpilogue rowwise;  // all zero for the block-scaled modes
  const void *a, *b, *sfa, *sfb;
  void *out;
  int64_t m, n, k_bytes, katoms;
  Workspace *ws;
  cudaStream_t st;
};

// Stores from registers against TMA stores from staged boxes (and, row-wise, scales by shuffle against shared memory),
// us, B200: K of 512 bytes, 32768 x 4096 outputs, where the epilogue is as long as the MMAs: row-wise 118.6 -> 83.1, MXFP8
// 89.0 -> 80.2, MXFP4 (K 512) 82.7 -> 67.2; K of 1024, 2048 x 9472: row-wise 23.0 -> 18.7; K of 4096 and more within 1 %
// (MXFP4 8192^3 170 -> 173, for the stage that its staging costs).
template <int MODE>
int launch_pair(const GemmCall &c, int max_clusters) {
  CUtensorMap map_a, map_b, map_sfa, map_sfb, map_out;
  constexpr int kKAtoms = Format<MODE>::kKAtoms;
  if (int e = make_operand_map(&map_a, c.a, c.m, c.k_bytes, kBM)) return e;
  if (int e = make_operand_map(&map_b, c.b, c.n, c.k_bytes, kPairBN / 2)) return e;
  if constexpr (Format<MODE>::kScaled) {
    if (int e = make_scale_map(&map_sfa, c.sfa, ceil_div64(c.m, 128), c.katoms, 1, kKAtoms)) return e;
    if (int e = make_scale_map(&map_sfb, c.sfb, ceil_div64(c.n, 128), c.katoms, 2, kKAtoms)) return e;
  } else {  // never dereferenced by the kernel
    map_sfa = map_a;
    map_sfb = map_a;
  }
  if (int e = make_output_map(&map_out, c.out, c.m, c.n)) return e;
  PairParams p;
  p.rowwise = c.rowwise;
  p.M = static_cast<int>(c.m);
  p.N = static_cast<int>(c.n);
  p.m_pairs = static_cast<int>(ceil_div64(c.m, 256));
  p.n_tiles = static_cast<int>(ceil_div64(c.n, kPairBN));
  p.k_stages = static_cast<int>(ceil_div64(c.k_bytes, kBK));
  p.last_k = last_k(c.k_bytes);
  p.ws = c.ws;
  const int64_t tiles = int64_t(p.m_pairs) * p.n_tiles;
  const int clusters = static_cast<int>(tiles < max_clusters ? tiles : max_clusters);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[2];
  cluster_launch_config(&cfg, attr, 2 * clusters, kGemmThreads, 2, smem_bytes<PairSmem<MODE>>(), c.st);
  return cuda_status(launch_quickly(cfg, mx_gemm_pair_kernel<MODE>, map_a, map_b, map_sfa, map_sfb, map_out, p,
                                    LaunchPad<kGemmParameterBytes<5, PairParams>>{}));
}

// One CTA per tile, tile shape SH.
template <typename SH, int MODE>
int launch_shape(const GemmCall &c, const DeviceInfo &dev) {
  static std::atomic<int> configured[kMaxGemmDevices];
  int dev_id = 0;
  DTQ_CUDA_TRY(cudaGetDevice(&dev_id));
  if (dev_id < 0 || dev_id >= kMaxGemmDevices) return DTQ_ERR_INVALID_ARGUMENT;
  constexpr int smem = smem_bytes<GemmSmem<SH, MODE>>();
  if (!configured[dev_id].load(std::memory_order_acquire)) {  // setting the attribute twice is harmless
    DTQ_CUDA_TRY(cudaFuncSetAttribute(mx_gemm_kernel<SH, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured[dev_id].store(1, std::memory_order_release);
  }
  CUtensorMap map_a, map_b, map_sfa, map_sfb;
  if (int e = make_operand_map(&map_a, c.a, c.m, c.k_bytes, kBM)) return e;
  if (int e = make_operand_map(&map_b, c.b, c.n, c.k_bytes, SH::BN)) return e;
  if constexpr (Format<MODE>::kScaled) {
    if (int e = make_scale_map(&map_sfa, c.sfa, ceil_div64(c.m, 128), c.katoms, 1, Format<MODE>::kKAtoms)) return e;
    if (int e = make_scale_map(&map_sfb, c.sfb, ceil_div64(c.n, 128), c.katoms, SH::BN / 128, Format<MODE>::kKAtoms)) return e;
  } else {  // never dereferenced by the kernel
    map_sfa = map_a;
    map_sfb = map_a;
  }
  GemmParams p;
  p.rowwise = c.rowwise;
  p.out = static_cast<uint16_t *>(c.out);
  p.M = static_cast<int>(c.m);
  p.N = static_cast<int>(c.n);
  p.m_tiles = static_cast<int>(ceil_div64(c.m, kBM));
  p.n_tiles = static_cast<int>(ceil_div64(c.n, SH::BN));
  p.k_stages = static_cast<int>(ceil_div64(c.k_bytes, kBK));
  p.last_k = last_k(c.k_bytes);
  p.ws = c.ws;
  const int64_t tiles = int64_t(p.m_tiles) * p.n_tiles;
  const int grid = static_cast<int>(tiles < dev.sm_count ? tiles : dev.sm_count);
  return cuda_status(launch_after_dependency(mx_gemm_kernel<SH, MODE>, dim3(grid), dim3(kGemmThreads), size_t(smem), c.st, map_a,
                                             map_b, map_sfa, map_sfb, p, LaunchPad<kGemmParameterBytes<4, GemmParams>>{}));
}

// Token rows per tile of the split kernel, and its stages.
int split_tokens(int64_t m) { return m <= 32 ? 32 : (m <= 64 ? 64 : 128); }
template <int BN>
constexpr int SplitStages = BN == 32 ? 5 : (BN == 64 ? 4 : 3);

// CTAs per tile of the split kernel: as many (1, 2, 4, 8) as fill the device's two CTAs per SM, with at least eight K
// stages each.
int split_count(int64_t m, int64_t n, int64_t stages, int sm_count) {
  const int64_t tiles = ceil_div64(n, 128) * ceil_div64(m, split_tokens(m));
  int splits = 1;
  while (splits < kMaxSplits && tiles * splits * 2 <= 2 * sm_count && stages >= 16 * splits) splits *= 2;
  return splits;
}

// How many clusters of `splits` CTAs of the split kernel the device can hold at once, asked once per device and size; 0
// where it cannot launch them.
template <int BN, int MODE>
int split_cluster_capacity(int dev_id, int splits, int *max_clusters) {
  static std::atomic<int> known[kMaxGemmDevices][kMaxSplits + 1];
  auto kernel = mx_gemm_split_kernel<BN, SplitStages<BN>, MODE>;
  if (dev_id < 0 || dev_id >= kMaxGemmDevices) return DTQ_ERR_INVALID_ARGUMENT;
  *max_clusters = clusters_that_fit(known[dev_id][splits], [=](int *n) {
    constexpr int smem = smem_bytes<SplitSmem<BN, SplitStages<BN>, MODE>>();
    static_assert(2 * (smem + 1024) <= 228 * 1024, "two CTAs per SM, with the kilobyte that each takes besides");
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    cluster_launch_config(&cfg, attr, splits, kSplitThreads, splits, smem, nullptr);
    cfg.numAttrs = 1;  // the occupancy query wants the cluster shape only
    return cudaOccupancyMaxActiveClusters(n, kernel, &cfg);
  });
  return DTQ_OK;
}
template <int MODE>
int split_cluster_capacity(int dev_id, int64_t m, int splits, int *max_clusters) {
  switch (split_tokens(m)) {
    case 32: return split_cluster_capacity<32, MODE>(dev_id, splits, max_clusters);
    case 64: return split_cluster_capacity<64, MODE>(dev_id, splits, max_clusters);
    default: return split_cluster_capacity<128, MODE>(dev_id, splits, max_clusters);
  }
}

// split_cluster_capacity has been asked for these sizes: it also sets the kernel's shared-memory attribute.
template <int BN, int MODE>
int launch_split(const GemmCall &c, int splits) {
  constexpr int smem = smem_bytes<SplitSmem<BN, SplitStages<BN>, MODE>>();
  CUtensorMap map_w, map_x, map_sfw, map_sfx;
  if (int e = make_operand_map(&map_w, c.b, c.n, c.k_bytes, kBM)) return e;
  if (int e = make_operand_map(&map_x, c.a, c.m, c.k_bytes, BN)) return e;
  if constexpr (Format<MODE>::kScaled) {
    if (int e = make_scale_map(&map_sfw, c.sfb, ceil_div64(c.n, 128), c.katoms, 1, Format<MODE>::kKAtoms)) return e;
    if (int e = make_scale_map(&map_sfx, c.sfa, ceil_div64(c.m, 128), c.katoms, 1, Format<MODE>::kKAtoms)) return e;
  } else {  // never dereferenced by the kernel
    map_sfw = map_w;
    map_sfx = map_w;
  }
  SplitParams p;
  p.rowwise = c.rowwise;
  p.rowwise.operand_format_bits = c.rowwise.operand_format_bits << 3;  // the caller's A is the MMA's B here, and its B is e4m3 (0)
  p.out = static_cast<uint16_t *>(c.out);
  p.M = static_cast<int>(c.m);
  p.N = static_cast<int>(c.n);
  p.n_tiles = static_cast<int>(ceil_div64(c.n, kBM));
  p.k_stages = static_cast<int>(ceil_div64(c.k_bytes, kBK));
  p.last_k = last_k(c.k_bytes);
  p.ws = c.ws;
  const int64_t tiles = int64_t(p.n_tiles) * ceil_div64(c.m, BN);
  p.splits = splits;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[2];
  cluster_launch_config(&cfg, attr, static_cast<int>(tiles * p.splits), kSplitThreads, p.splits, smem, c.st);
  return cuda_status(launch_quickly(cfg, mx_gemm_split_kernel<BN, SplitStages<BN>, MODE>, map_w, map_x, map_sfw, map_sfx, p,
                                    LaunchPad<kGemmParameterBytes<4, SplitParams>>{}));
}

// The CTAs per tile that the split kernel gets in the choice below; 1: the call is not one for it.
// Few tiles and a long K: once it gets four CTAs per tile, or two where a tile is only 32 tokens wide or, with 32 stages of K
// or more, 64.  Measured split against the best of the others, us: four CTAs, row-wise 64 x 8192 x 4096 9.9 / 12.1,
// 128 x 4096 x 4096 10.3 / 12.4, 300 x 2048 x 8192 14.3 / 19.4, MXFP4 512 x 1024 x 8192 10.3 / 12.0; two CTAs,
// 16 x 16384 x 8192 24.0 / 27.0, 64 x 16384 x 8192 25.8 / 28.7, MXFP4 16 x 8192 x 4096 6.7 / 9.2, but 512 x 4096 x 4096
// 14.3 / 13.4 and MXFP4 64 x 8192 x 4096 8.1 / 8.0; one CTA, 32 x 1024 x 1024 6.1 / 4.9.
int split_worthwhile(int64_t m, int64_t n, int64_t stages, int sm_count) {
  const int splits = split_count(m, n, stages, sm_count);
  const bool two_pay = m <= 32 || (m <= 64 && stages >= 32);
  return splits >= (two_pay ? 2 : 4) ? splits : 1;
}

// Which kernel, for a device with `sm_count` SMs that holds `pair_clusters` SM pairs and `split_clusters` clusters of the split
// kernel (0: cannot launch them).  Estimated time, in microseconds as measured on a B200 = a fixed part (launch, set-up,
// filling the pipeline, the last epilogue) plus, for every round of tiles on the busiest SM, the stages of 128 operand bytes
// along K at the time of one, and what a tile costs besides; a tile never takes less than its epilogue.
//   pair   256 x 256 tiles on SM pairs: 5.4 + rounds x max(0.333 stages + 0.6, 3.4); row-wise 5.8 + rounds x max(0.333 stages + 0.6, 2.3)
//   wide   128 x 256 on one SM: 4.2 + rounds x max(0.36 stages + 1.9, 3.2; row-wise 0.36 stages + 2.1, 4.6), its epilogue not overlapped
//   narrow 128 x 128 on one SM: 3.2 + rounds x max(0.23 stages + 1.1, 1.9; row-wise 0.23 stages + 1.3, 2.4)
// So large problems run on SM pairs, and problems of about a tile per SM on the narrow kernel, whose smaller tiles also
// spread a small output over more SMs.  The constants were fitted to random shapes (K of 256 to 8192, 256 to 16384 outputs, up to 32768
// tokens; three sets in turn); pair's, whose last tile's stores came later, to 255 others of them, and checked on 180 with K up to 2048.
// Over those 435 the kernel chosen takes longer than the quickest, on average and at most: MXFP8 0.5 % and 11 % (3815 x 12712 x 576, 48.1 instead of 43.3 us), MXFP4
// 0.45 % and 9 %, row-wise 1.4 % and 39 % (512 x 536 x 416, where the host is what is measured; 3518 x 2584 x 4656 36 %).  With 5.4 and 3.1 for
// pair in MXFP8 and MXFP4 1.0 % and 24 %, 0.9 % and 22 %; 5.4 for row-wise 1.4 % and 39 %.
// Measured, us, narrow / wide / pair: MXFP8 7666 x 4840 x 512 29.3 / 26.8 / 33.1, 6311 x 8264 x 320 37.7 / 36.6 / 45.4, MXFP4 25579 x 2912 x 384 38.7 / 36.4 /
// 44.5, 677 x 6608 x 2144 15.5 / 16.3 / 13.5.
int choose_kernel(bool row_wise, int64_t m, int64_t n, int64_t k_bytes, int sm_count, int pair_clusters, int split_clusters) {
  const int64_t k_stages = ceil_div64(k_bytes, kBK), m_tiles = ceil_div64(m, kBM);
  if (split_clusters > 0 && split_worthwhile(m, n, k_stages, sm_count) > 1) return DTQ_GEMM_SPLIT;
  const double stages = static_cast<double>(k_stages);
  auto rounds = [](int64_t tiles, int64_t slots) { return static_cast<double>(ceil_div64(tiles, slots)); };
  const double wide =
      4.2 + rounds(m_tiles * ceil_div64(n, 256), sm_count) * std::max(0.36 * stages + (row_wise ? 2.1 : 1.9), row_wise ? 4.6 : 3.2);
  const double narrow =
      3.2 + rounds(m_tiles * ceil_div64(n, 128), sm_count) * std::max(0.23 * stages + (row_wise ? 1.3 : 1.1), row_wise ? 2.4 : 1.9);
  const double pair = pair_clusters > 0 ? (row_wise ? 5.8 : 5.4) + rounds(ceil_div64(m, 256) * ceil_div64(n, 256), pair_clusters) *
                                                    std::max(0.333 * stages + 0.6, row_wise ? 2.3 : 3.4)
                                        : 1e30;
  return (pair < wide && pair < narrow) ? DTQ_GEMM_PAIR : (narrow <= wide ? DTQ_GEMM_NARROW : DTQ_GEMM_WIDE);
}

template <int MODE>
int launch_gemm(const GemmCall &c, int kernel, const DeviceInfo &dev) {
  const int64_t stages = ceil_div64(c.k_bytes, kBK);
  int dev_id = 0, pair_clusters = 0, split_clusters = 0;
  DTQ_CUDA_TRY(cudaGetDevice(&dev_id));
  if (int e = pair_cluster_capacity<MODE>(dev_id, &pair_clusters)) return e;
  const int splits = kernel == DTQ_GEMM_SPLIT  ? split_count(c.m, c.n, stages, dev.sm_count)
                     : kernel == DTQ_GEMM_AUTO ? split_worthwhile(c.m, c.n, stages, dev.sm_count)
                                               : 1;
  if (splits > 1)
    if (int e = split_cluster_capacity<MODE>(dev_id, c.m, splits, &split_clusters)) return e;
  if (kernel == DTQ_GEMM_AUTO)
    kernel = choose_kernel(MODE == kRowwise, c.m, c.n, c.k_bytes, dev.sm_count, pair_clusters, split_clusters);
  if (kernel == DTQ_GEMM_SPLIT) {
    if (splits < 2) return DTQ_ERR_SHAPE;  // named, but too many tiles or too little of K to split anything
    if (split_clusters <= 0) return DTQ_ERR_CUDA_BASE + static_cast<int>(cudaErrorNotSupported);
    switch (split_tokens(c.m)) {
      case 32: return launch_split<32, MODE>(c, splits);
      case 64: return launch_split<64, MODE>(c, splits);
      default: return launch_split<128, MODE>(c, splits);
    }
  }
  if (kernel == DTQ_GEMM_PAIR && pair_clusters <= 0) return DTQ_ERR_CUDA_BASE + static_cast<int>(cudaErrorNotSupported);
  if (kernel == DTQ_GEMM_PAIR) return launch_pair<MODE>(c, pair_clusters);
  if (kernel == DTQ_GEMM_NARROW) return launch_shape<NarrowShape, MODE>(c, dev);
  return launch_shape<WideShape, MODE>(c, dev);
}

}  // namespace
}  // namespace dtq

extern "C" int dtq_gemm_kernel_for(int row_wise, int64_t m, int64_t n, int64_t k_bytes, int sm_count, int pair_clusters,
                                   int split_clusters) {
  if (m <= 0 || n <= 0 || k_bytes <= 0 || sm_count <= 0) return DTQ_GEMM_AUTO;
  return dtq::choose_kernel(row_wise != 0, m, n, k_bytes, sm_count, pair_clusters, split_clusters);
}

extern "C" size_t dtq_mx_gemm_scale_bytes(int64_t rows, int64_t k) {
  if (rows <= 0 || k <= 0) return 0;
  return static_cast<size_t>((rows + 127) / 128) * static_cast<size_t>(((k + 31) / 32 + 3) / 4) * 512;
}

extern "C" int dtq_mx_gemm_bf16(const void *a, const void *b, const void *a_scales_blocked, const void *b_scales_blocked,
                                void *out_bf16, int64_t m, int64_t n, int64_t k, int elem_format, int kernel, void *workspace,
                                size_t workspace_bytes, void *stream) {
  using namespace dtq;
  if (m < 0 || n < 0 || k < 0) return DTQ_ERR_INVALID_ARGUMENT;
  if (elem_format != DTQ_E4M3 && elem_format != DTQ_E2M1) return DTQ_ERR_UNSUPPORTED_DTYPE;
  if (kernel < DTQ_GEMM_AUTO || kernel > DTQ_GEMM_SPLIT) return DTQ_ERR_INVALID_ARGUMENT;
  if (n % 8 != 0 || k % 32 != 0) return DTQ_ERR_SHAPE;  // 16-byte output vectors; whole MX blocks (also the TMA row pitch)
  if (m > 0x7FFFFFFF - 256 || n > 0x7FFFFFFF - 256 || k > 0x7FFFFFFF - 256) return DTQ_ERR_TOO_LARGE;
  if (!workspace || workspace_bytes < sizeof(Workspace) || !aligned_to(workspace, 256)) return DTQ_ERR_WORKSPACE;
  if (m == 0 || n == 0) return DTQ_OK;
  if (!out_bf16 || !aligned_to(out_bf16, 16)) return DTQ_ERR_INVALID_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (k == 0) return cuda_status(cudaMemsetAsync(out_bf16, 0, static_cast<size_t>(m) * n * 2, st));
  if (!a || !b || !a_scales_blocked || !b_scales_blocked) return DTQ_ERR_INVALID_ARGUMENT;
  if (!aligned_to(a, 16) || !aligned_to(b, 16) || !aligned_to(a_scales_blocked, 16) || !aligned_to(b_scales_blocked, 16))
    return DTQ_ERR_INVALID_ARGUMENT;
  DeviceInfo dev;
  if (int e = current_device_info(&dev)) return e;
  GemmCall c;
  c.rowwise = RowwiseEpilogue{};
  c.a = a;
  c.b = b;
  c.sfa = a_scales_blocked;
  c.sfb = b_scales_blocked;
  c.out = out_bf16;
  c.m = m;
  c.n = n;
  c.k_bytes = elem_format == DTQ_E2M1 ? k / 2 : k;
  c.katoms = ceil_div64(k / 32, 4);
  c.ws = static_cast<Workspace *>(workspace);
  c.st = st;
  return elem_format == DTQ_E2M1 ? launch_gemm<kMxFp4>(c, kernel, dev) : launch_gemm<kMxFp8>(c, kernel, dev);
}

extern "C" int dtq_rowwise_fp8_bf16(const void *a, const void *b, const float *a_row_scale, const float *b_row_scale,
                                    const void *bias, int bias_dtype, void *out_bf16, int64_t m, int64_t n, int64_t k,
                                    int a_format, int kernel, void *workspace, size_t workspace_bytes, void *stream) {
  using namespace dtq;
  if (m < 0 || n < 0 || k < 0) return DTQ_ERR_INVALID_ARGUMENT;
  if (a_format != DTQ_E4M3 && a_format != DTQ_E5M2) return DTQ_ERR_UNSUPPORTED_DTYPE;
  if (bias && bias_dtype != DTQ_F32 && bias_dtype != DTQ_BF16) return DTQ_ERR_UNSUPPORTED_DTYPE;
  if (kernel < DTQ_GEMM_AUTO || kernel > DTQ_GEMM_SPLIT) return DTQ_ERR_INVALID_ARGUMENT;
  if (n % 8 != 0 || k % 16 != 0) return DTQ_ERR_SHAPE;  // 16-byte output vectors; 16-byte operand row pitch (TMA)
  if (m > 0x7FFFFFFF - 256 || n > 0x7FFFFFFF - 256 || k > 0x7FFFFFFF - 256) return DTQ_ERR_TOO_LARGE;
  if (!workspace || workspace_bytes < sizeof(Workspace) || !aligned_to(workspace, 256)) return DTQ_ERR_WORKSPACE;
  if (m == 0 || n == 0) return DTQ_OK;
  if (!out_bf16 || !aligned_to(out_bf16, 16) || !a_row_scale || !b_row_scale) return DTQ_ERR_INVALID_ARGUMENT;
  if (k > 0 && (!a || !b || !aligned_to(a, 16) || !aligned_to(b, 16))) return DTQ_ERR_INVALID_ARGUMENT;
  DeviceInfo dev;
  if (int e = current_device_info(&dev)) return e;
  GemmCall c;
  c.rowwise.row_scale = a_row_scale;
  c.rowwise.col_scale = b_row_scale;
  c.rowwise.bias = bias;
  c.rowwise.bias_is_bf16 = bias_dtype == DTQ_BF16;
  c.rowwise.operand_format_bits = a_format == DTQ_E5M2 ? (1u << 7) : 0u;
  c.a = a;
  c.b = b;
  c.sfa = nullptr;
  c.sfb = nullptr;
  c.out = out_bf16;
  c.m = m;
  c.n = n;
  c.k_bytes = k;
  c.katoms = 0;
  c.ws = static_cast<Workspace *>(workspace);
  c.st = static_cast<cudaStream_t>(stream);
  return launch_gemm<kRowwise>(c, kernel, dev);
}

extern "C" int dtq_mx_fp8_bf16(const void *a, const void *b, const void *a_scales_blocked, const void *b_scales_blocked,
                               void *out_bf16, int64_t m, int64_t n, int64_t k, void *workspace, size_t workspace_bytes,
                               void *stream) {
  return dtq_mx_gemm_bf16(a, b, a_scales_blocked, b_scales_blocked, out_bf16, m, n, k, DTQ_E4M3, DTQ_GEMM_AUTO, workspace,
                          workspace_bytes, stream);
}

extern "C" int dtq_mx_fp4_bf16(const void *a, const void *b, const void *a_scales_blocked, const void *b_scales_blocked,
                               void *out_bf16, int64_t m, int64_t n, int64_t k, void *workspace, size_t workspace_bytes,
                               void *stream) {
  return dtq_mx_gemm_bf16(a, b, a_scales_blocked, b_scales_blocked, out_bf16, m, n, k, DTQ_E2M1, DTQ_GEMM_AUTO, workspace,
                          workspace_bytes, stream);
}
