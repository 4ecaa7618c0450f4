// Per-axis contraction on the 5th-generation tensor cores (sm_103a):
// TMA -> shared memory -> tcgen05.mma (kind::tf32) -> TMEM -> epilogue.
//
//   out[b][s][m][p] = alpha * epi( sum_k op[s][m][k] * in[b][s][p][k] ) + beta * out
//
// Precision: three-term split TF32.  Each FP32 input x is split exactly into
// hi = x with its low 13 mantissa bits cleared (a TF32 value) and lo = x - hi;
// the operator is pre-split the same way on the host.  The tensor cores then
// accumulate hi*hi + hi*lo + lo*hi in FP32, which gives FP32-level accuracy
// (about 2^-22 relative per product) at three TF32 MMAs per block.
//
// Tile: 128 rows of p (the MMA M dimension, one TMEM lane per row) by up to 128
// operator rows m (the MMA N dimension, one TMEM column each).  The kernel is
// persistent (one CTA per SM walking the tile list) with two TMEM accumulator
// buffers.  Three rings decouple the roles: input blocks (128 rows x 32 FP32,
// 16 KB), operator blocks (a 128-byte row of K: 32 TF32 or 64 16-bit elements,
// hi and lo; or the CTA's whole operator chunk, kept) and operand A slots in
// TMEM.  An input block is free again as soon as it has been split, an operator
// block and the A slots when the MMAs of its K are done (one commit for both).
// Warp roles:
//   warp 0     input producer (TMA, one thread)
//   warp 1     TMEM allocator and MMA issuer
//   warps 2-5  split each input block into hi and lo, operand A, in TMEM
//   warps 15-18 (plain epilogue of the 16-bit paths) a second splitting group,
//              the two taking K blocks in turn: 36.5 -> 32.6 us at K = 512
//   warps 6-13 epilogue: two warps per TMEM lane quarter, tcgen05.ld 32 lanes
//              x 16 columns, fused field multiply / eigenvalue divide / beta
//              accumulate, stores from registers
//   warp 14    operator producer (TMA, one thread)
// With one ring of (input, operator) stages that the MMAs released, and output
// boxes staged for bulk stores, the split-BF16 pass of 16 x 256^3 took 422 us
// (now 365, 88 % of the measured HBM rate), the split-FP16 passes of 128
// problems of N = 256 39 us (M = 512; now 34.5) and 64 us with the field (now
// 49), the 3-D split-TF32 field pass of 8 x 128^3 130 us (now 104).
// Every mbarrier wait is bounded by a global-timer budget; on expiry the
// kernel records JFG_ERR_DEVICE_TIMEOUT in a device status word, drains its own
// TMA copies (bounded), frees its TMEM and returns.
#include <cuda.h>
#include <cuda_fp16.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "jfg_internal.cuh"

namespace jfg {

__device__ int g_tc_status = 0;
// Budget of the pipeline waits (ns) and the test hook that makes the epilogue
// first wait on a barrier nothing arrives on (jfg_tc_set_wait_budget_ns,
// jfg_tc_test_hold): the timeout path can then be exercised without any
// broken kernel.  Drain waits always use the full WAIT_NS budget.
constexpr unsigned long long WAIT_NS_DEFAULT = 2000000000ull;
__device__ unsigned long long g_tc_wait_ns = WAIT_NS_DEFAULT;
__device__ int g_tc_test_hold = 0;

// Kernel variant: 1 keeps the split input tile in TMEM (default), 0 in shared
// memory (jfg_tc_set_variant).
static int g_operand_a_in_tmem = 1;
// Operator-stationary schedule for single-group launches whose operator chunk
// fits in shared memory: 0 off, 1 (default) when every CTA gets >= 2 tiles, the
// chunk leaves four input blocks, the inputs stay in L2 and the kernel has one
// splitting group, 2 whenever the chunk fits (jfg_tc_set_op_resident); a launch
// configuration's schedule field overrides it.  Measured against streaming (128
// problems, N = 256): field pass (split FP16) 49.8 against 53.0 us, plain BF16
// 16.4 against 18.4; 3-D 8 x 128^3 split TF32: 43 against 47.5.  Inputs beyond
// L2 (3 x 8 x 128^3): 117 against 104 us, so they stream.  The kernels with two
// splitting groups (plain epilogue of the split 16-bit paths) gain or lose by
// the size and stream by default, the autotuner tries both: split FP16, M = 512,
// 128 problems 35.5 against 34.9 us, 64 problems 21.7 against 22.6; split BF16
// 19.2 against 20.5 for 128 problems, 10.8 against 10.3 for 32.
static int g_op_resident = 1;

namespace {

constexpr int TILE_P = 128;
constexpr int KB = 32;                     // FP32 elements per K block (128 B)
constexpr int MT_MAX = 128;                // operator rows per tile (MMA N)
// 15 warps; four more that split where that is what bounds the pass: the plain
// epilogue of the 16-bit paths (their registers, 96 instead of 128 a thread,
// cost the other kernels more than the split gains)
__host__ __device__ constexpr int nthreads(int epi, bool beta, int prec) {
  return prec != 0 && epi == JFG_EPI_NONE && !beta ? 608 : 480;
}
constexpr uint32_t XBYTES = TILE_P * KB * 4;  // 16 KB
// K elements of one operator stage: a 128-byte row, 32 TF32 or 64 16-bit ones.
__host__ __device__ constexpr int op_ke(bool b16) { return b16 ? 64 : 32; }
constexpr int S_MAX = 16;                  // stages (or resident blocks) of a ring
constexpr unsigned long long WAIT_NS = 2000000000ull;  // 2 s budget per wait

constexpr int GMAX = 40;  // groups per launch of the grouped kernel

// One group of problems of a (grouped) launch.
struct TcGroup {
  jfg_contract_desc d;
  float* out;
  int Mtile;       // padded operator rows per tile (multiple of 16, <= MT_MAX)
  int seg_in_map;  // 1 if the input map has a segment dimension
  int bat_in_map;  // 1 if the input map has a batch dimension
  int seg_op_map;  // 1 if the operator maps have a segment dimension
  int mc_inner;    // tile order: operator chunks innermost (inputs beyond L2)
  // scaled split-FP16 variant: per-problem max |input| (float bits) that sets
  // the power-of-two input scale, per-problem max |output| recorded for the
  // next pass, and the inverse power-of-two row scales of the operator
  const unsigned* in_max;
  unsigned* out_max;
  const float* op_inv;  // op_inv[s * op_inv_seg + m]
  long long op_inv_seg;
  // fused dot (field / divide epilogues): partials of sum(acc * out) per
  // problem at dot_part[b * DOT_NBMAX + tile-of-problem * 8 + epilogue warp]
  float* dot_part;
};

// Kernel parameter block (__grid_constant__): groups and their tensor maps
// (input X, operator hi, operator lo).
constexpr int SMEM_MAX = 227 * 1024 - 1024;   // dynamic shared memory (static use < 1 KB)
template <int G>
struct TcLaunch {
  CUtensorMap maps[G][3];
  TcGroup g[G];
  int ngroups;
  int xstages;  // input blocks (128 rows x 32 FP32) in shared memory
  int aslots;   // split input blocks (MMA operand A): TMEM slots, or the input stages
  int ostages;  // operator blocks in shared memory (streaming schedule)
  int tmem_cols;
  int tmem_a;   // 1: split input tile (MMA operand A) kept in TMEM, not shared memory
  int mt_max;   // largest Mtile: sets the stage layout
  // 1 (one group): operator-stationary schedule.  CTA c
  // serves the operator slot c % nslots, slot = s * mchunks + mc, loads that
  // operator chunk (all K blocks, hi and lo) into shared memory once and
  // streams only the input tiles of its (problem, p-tile) pairs.
  int op_res;
  int nslots;
};

// TMEM column map when operand A lives in TMEM: accumulator buffers at
// columns [0, 128) and [128, 256); slot s of operand A at 256 + A_SLOT s, hi
// then lo (32 TF32 columns each, or 16 columns of 16-bit pairs).
constexpr int ACC_STRIDE_TA = 128;
constexpr int A_COL0 = 256;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: false (and the status word set) if the budget runs out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity,
                                          unsigned long long budget) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long t0 = gtimer();
  while (true) {
    for (int i = 0; i < 256; ++i)
      if (mbar_try(bar, parity)) return true;
    if (gtimer() - t0 > budget) {
      atomicExch(&g_tc_status, JFG_ERR_DEVICE_TIMEOUT);
      return false;
    }
  }
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar,
                                            int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar,
                                            int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2),
      "r"(c3)
      : "memory");
}

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, 8-row
// core-matrix groups 1024 B apart.
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);  // start address
  d |= (uint64_t)1 << 16;                     // leading byte offset (unused, SW128 K-major)
  d |= (uint64_t)(1024 >> 4) << 32;           // stride byte offset
  d |= (uint64_t)1 << 46;                     // descriptor version
  d |= (uint64_t)2 << 61;                     // SWIZZLE_128B
  return d;
}

// Instruction descriptor: kind::tf32, D = F32, A = B = TF32, both K-major.
__host__ __device__ constexpr uint32_t idesc_tf32(int M, int N) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_tf32(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accum));
}

// Same MMA with operand A read from TMEM (128 lanes x 8 TF32 columns).
__device__ __forceinline__ void mma_tf32_ta(uint32_t tmem, uint32_t a_tmem, uint64_t b,
                                            uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem),
      "r"(a_tmem), "l"(b), "r"(idesc), "r"(accum));
}

// Instruction descriptor: kind::f16 with BF16 A/B, D = F32, both K-major.
__host__ __device__ constexpr uint32_t idesc_b16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}

// BF16 MMA (K = 16) with operand A read from TMEM (128 lanes x 8 columns of
// packed BF16 pairs).
__device__ __forceinline__ void mma_b16_ta(uint32_t tmem, uint32_t a_tmem, uint64_t b,
                                           uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem),
      "r"(a_tmem), "l"(b), "r"(idesc), "r"(accum));
}

// Two FP32 -> packed BF16 pair (round to nearest even): lo16 <- a, hi16 <- b.
__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(b), "f"(a));
  return d;
}

// Two FP32 -> packed FP16 pair (round to nearest even): lo16 <- a, hi16 <- b.
__device__ __forceinline__ uint32_t pack_f16x2(float a, float b) {
  uint32_t d;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(b), "f"(a));
  return d;
}

__device__ __forceinline__ float2 unpack_f16x2(uint32_t h) {
  return __half22float2(*reinterpret_cast<const __half2*>(&h));
}

// Instruction descriptor: kind::f16 with FP16 A/B, D = F32, both K-major.
__host__ __device__ constexpr uint32_t idesc_f16(int M, int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Power-of-two input scale of the split-FP16 variant from the float bits of
// an upper bound on max |x|: the scaled values are below 2^15 (FP16 max is
// 65504) and the largest is at least 2^14, so FP16 hi and lo keep ~22 bits
// relative to the maximum and nothing overflows.  Zero, non-finite or
// missing bounds give scale 1; the exponent is clamped to [2^-126, 2^126]
// so the inverse is exact as well.
__device__ __forceinline__ void h16_scale_bits(unsigned bits, float& sc, float& inv) {
  sc = inv = 1.f;
  bits &= 0x7FFFFFFFu;
  const int e = (int)(bits >> 23);
  if (bits == 0 || e == 0xFF) return;
  int eb = 268 - e;  // biased exponent of 2^(15 - E), max |x| < 2^E, E = e - 126
  eb = eb < 1 ? 1 : (eb > 253 ? 253 : eb);
  sc = __uint_as_float((unsigned)eb << 23);
  inv = __uint_as_float((unsigned)(254 - eb) << 23);
}
// the recorded bound of problem b (0: none, scale 1)
__device__ __forceinline__ unsigned h16_bits(const unsigned* in_max, int b) {
  return (in_max && b >= 0) ? __ldg(in_max + b) : 0u;
}
__device__ __forceinline__ void h16_scale(const unsigned* in_max, int b, float& sc, float& inv) {
  h16_scale_bits(h16_bits(in_max, b), sc, inv);
}

// Store 32 consecutive 32-bit columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(
          taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
      "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]),
      "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]),
      "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}

// Store 16 consecutive 32-bit columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
      "r"(v[15])
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ float tf32_hi(float x) {
  return __uint_as_float(__float_as_uint(x) & 0xFFFFE000u);
}

// Persistent kernel over one or more groups of problems.  Group gi has its own
// descriptor, operator tile height Mtile and tensor maps; its tiles are
// t = tb[gi] + ((slot * nseg + s) * mchunks + mc) * nptiles + pt (or, for inputs
// larger than L2, ((slot * nseg + s) * nptiles + pt) * mchunks + mc), covering p rows
// [pt*128, +128) and operator rows [mc*Mtile, +Mtile) of problem slot / segment
// s.  Each CTA walks t = blockIdx.x, blockIdx.x + gridDim.x, ...; two TMEM
// accumulator buffers let the epilogue of tile i overlap the main loop of
// tile i+1.  The tile prefix tb[] is formed on the device from the active
// counts, so listed (active-subset) groups need no host round trip.
template <int EPI, bool BETA, int G, int PREC>
__global__ void __launch_bounds__(nthreads(EPI, BETA, PREC), 1)
    k_contract_tc(const __grid_constant__ TcLaunch<G> L) {
  // PREC: 0 split TF32 (kind::tf32), 1 split BF16, 2 scaled split FP16 (both
  // kind::f16: 16-bit operator pairs, 64-element K blocks), 3 plain BF16 (one
  // product hi*hi, the operator's hi only: ~2^-8 relative per product)
  constexpr bool B16 = PREC != 0;
  constexpr bool H16 = PREC == 2;
  constexpr bool B1 = PREC == 3;
  constexpr uint32_t NOP = B1 ? 1u : 2u;  // operator pieces per stage (hi, lo)
  constexpr int KO = op_ke(B16);       // K elements of an operator block
  constexpr int KXO = KO / KB;         // input blocks per operator block
  constexpr uint32_t OROW = 128u;      // bytes per operator row of a block
  // TMEM columns per slot of operand A (hi then lo)
  constexpr uint32_t A_SLOT = B1 ? 16u : B16 ? 32u : 64u;
  extern __shared__ uint8_t smem_raw[];
  __shared__ long long tb[G + 1];
  __shared__ int nbs[G];
  __shared__ unsigned long long s_budget;
  __shared__ int s_hold;
  // scaled split FP16: the input bound of each stage's problem, written by the
  // producer with the stage's loads (it reads the list and the bound well
  // ahead), read by the split warps after the stage's full barrier
  __shared__ unsigned s_xbits[S_MAX];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int SX = L.xstages, SA = L.aslots, SO = L.ostages;
  const bool ta = B16 || L.tmem_a != 0;
  const bool res = L.op_res != 0;
  const uint32_t omax = (uint32_t)L.mt_max * OROW;  // Mtile operator rows (hi or lo)
  const uint32_t obytes_max = NOP * omax;           // an operator block
  const uint32_t xstage = ta ? XBYTES : 2 * XBYTES;  // input block (+ its lo part when in SMEM)
  const uint32_t acc_stride = ta ? ACC_STRIDE_TA : 256;
  // operator-stationary schedule: this CTA's operator slot and tile stride
  const int r_slot = res ? (int)(blockIdx.x % (unsigned)L.nslots) : 0;
  const int r_mchunks = res ? (L.g[0].d.M + L.g[0].Mtile - 1) / L.g[0].Mtile : 1;
  const int r_s = r_slot / r_mchunks, r_mc = r_slot - r_s * r_mchunks;
  const long long r_j0 = res ? (long long)(blockIdx.x / (unsigned)L.nslots) : 0;
  const long long r_step =
      res ? (long long)((gridDim.x - (unsigned)r_slot + (unsigned)L.nslots - 1) / L.nslots) : 1;
  const int r_nko = res ? (L.g[0].d.K + KO - 1) / KO : 0;

  if (threadIdx.x == 0) {
    long long acc = 0;
    for (int gi = 0; gi < L.ngroups; ++gi) {
      const TcGroup& q = L.g[gi];
      const int nb = active_count(q.d.batch_list, q.d.batch_count, q.d.batch);
      nbs[gi] = nb;
      tb[gi] = acc;
      acc += (long long)((q.d.P + TILE_P - 1) / TILE_P) * ((q.d.M + q.Mtile - 1) / q.Mtile) *
             nb * q.d.nseg;
    }
    tb[L.ngroups] = acc;
    s_budget = g_tc_wait_ns;
    s_hold = g_tc_test_hold;
  }
  __syncthreads();
  const unsigned long long budget = s_budget;
  const long long ntiles = __shfl_sync(0xffffffffu, tb[L.ngroups], 0);
  const int r_nptiles = (L.g[0].d.P + TILE_P - 1) / TILE_P;
  const long long r_cnt =  // tiles of one slot
      res ? (long long)__shfl_sync(0xffffffffu, nbs[0], 0) * r_nptiles : 0;
  if (!res && (long long)blockIdx.x >= ntiles) return;  // no tile for this CTA (uniform)
  if (res && r_j0 >= r_cnt) return;

  // operator blocks (ring or resident) | input ring
  uint8_t* obase = smem;
  uint8_t* xbase = obase + (size_t)(res ? r_nko : SO) * obytes_max;
  uint64_t* bars = (uint64_t*)(xbase + (size_t)SX * xstage);
  uint64_t* xfull = bars;               // [S_MAX] input block landed
  uint64_t* xempty = bars + S_MAX;      // [S_MAX] input block read
  uint64_t* conv = bars + 2 * S_MAX;    // [S_MAX] operand A slot written
  uint64_t* ofull = bars + 3 * S_MAX;   // [S_MAX] operator block landed
  // [S_MAX] the MMAs of K block n (n % S_MAX) are done: its operator block and
  // its operand A slots are free.  One commit per K block serves both rings
  // (a commit costs the issuer 100-200 clocks); no ring is longer than S_MAX.
  uint64_t* kdone = bars + 4 * S_MAX;
  uint64_t* tfull = bars + 5 * S_MAX;       // [2] accumulator ready
  uint64_t* tempty = bars + 5 * S_MAX + 2;  // [2] accumulator drained
  uint64_t* hold = bars + 5 * S_MAX + 4;    // test hook: nothing arrives on it
  uint64_t* mma_done = bars + 5 * S_MAX + 5;  // MMA drain after a timeout
  uint32_t* tmem_slot = (uint32_t*)(bars + 5 * S_MAX + 6);

  // warp-uniform to the compiler, like the TMEM base below: the MMA issuer's
  // descriptors then stay in uniform registers
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < S_MAX; ++i) {
      mbar_init(&xfull[i], 1);
      mbar_init(&xempty[i], 4);  // the split warps (operand A in TMEM)
      mbar_init(&conv[i], 4);
      mbar_init(&ofull[i], 1);
      mbar_init(&kdone[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 8);
    }
    mbar_init(hold, 1);
    mbar_init(mma_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(L.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  auto Xh = [&](int st) { return xbase + (size_t)st * xstage; };
  auto Xl = [&](int st) { return xbase + (size_t)st * xstage + XBYTES; };
  auto Op = [&](int st) { return obase + (size_t)st * obytes_max; };  // hi, then lo
  // b = problem index (-1: an out-of-range list entry, computed but not stored);
  // roles that do not use b (need_b false) skip its list load.  Tile indices
  // below 2^32 take 32-bit division: the 64-bit one is a long software
  // sequence, paid by every role at every tile.
  auto decode = [&](long long t, int& gi, int& pt, int& mc, int& b, int& s, bool need_b) {
    gi = 0;
    if (G > 1)
      while (gi + 1 < L.ngroups && t >= tb[gi + 1]) ++gi;
    const TcGroup& q = L.g[gi];
    const unsigned nptiles = (unsigned)((q.d.P + TILE_P - 1) / TILE_P);
    const unsigned mchunks = (unsigned)((q.d.M + q.Mtile - 1) / q.Mtile);
    const long long r = t - tb[gi];
    int bs;
    if (r <= 0xFFFFFFFFLL) {
      unsigned ru = (unsigned)r;
      if (q.mc_inner) {  // the CTAs that share an input tile run it at the same time
        mc = (int)(ru % mchunks);
        ru /= mchunks;
        pt = (int)(ru % nptiles);
        bs = (int)(ru / nptiles);
      } else {           // the CTAs that share an operator chunk run it at the same time
        pt = (int)(ru % nptiles);
        ru /= nptiles;
        mc = (int)(ru % mchunks);
        bs = (int)(ru / mchunks);
      }
    } else if (q.mc_inner) {
      mc = (int)(r % mchunks);
      pt = (int)((r / mchunks) % nptiles);
      bs = (int)(r / mchunks / nptiles);
    } else {
      pt = (int)(r % nptiles);
      mc = (int)((r / nptiles) % mchunks);
      bs = (int)(r / nptiles / mchunks);
    }
    const int slot = bs / q.d.nseg;
    s = bs - slot * q.d.nseg;
    b = need_b ? active_problem(q.d.batch_list, nbs[gi], q.d.batch, slot) : 0;
  };
  // input blocks of a tile: whole operator blocks (zeros past K)
  auto nkx_of = [&](int gi) { return (L.g[gi].d.K + KO - 1) / KO * KXO; };
  // the MMAs of K block n are done (n < 0: there is none)
  auto wait_done = [&](long long n) {
    return n < 0 || mbar_wait(&kdone[n % S_MAX], (uint32_t)(n / S_MAX) & 1u, budget);
  };
  // the wait of a whole warp: one answer for all lanes, which are converged
  // after it, as the aligned TMEM instructions need
  auto warp_wait = [&](uint64_t* bar, uint32_t parity) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, budget)) != 0;
  };
  // tile li of this CTA (false past the last one)
  auto tile_of = [&](long long li, int& gi, int& pt, int& mc, int& b, int& s,
                     bool need_b = true) -> bool {
    if (!res) {
      const long long t = (long long)blockIdx.x + li * (long long)gridDim.x;
      if (t >= ntiles) return false;
      decode(t, gi, pt, mc, b, s, need_b);
      return true;
    }
    const long long j = r_j0 + li * r_step;
    if (j >= r_cnt) return false;
    const TcGroup& q = L.g[0];
    gi = 0;
    pt = (int)(j % r_nptiles);
    b = need_b ? active_problem(q.d.batch_list, nbs[0], q.d.batch, (int)(j / r_nptiles)) : 0;
    s = r_s;
    mc = r_mc;
    return true;
  };

  if (warp == 0) {
    // ---------------- input producer ----------------
    if (lane == 0) {
      long long issued = 0;
      bool ok = true;
      int gi, pt, mc, b, s;
      int st = 0;       // stage of the current block (kept running: no division)
      uint32_t ph = 0;  // its use count parity
      for (long long li = 0; ok && tile_of(li, gi, pt, mc, b, s); ++li) {
        const TcGroup& q = L.g[gi];
        const int cs = q.seg_in_map ? s : 0;
        const int cb = (q.bat_in_map && b > 0) ? b : 0;
        const int nkx = nkx_of(gi);
        const unsigned xbits = H16 ? h16_bits(q.in_max, b) : 0u;
        for (int kx = 0; kx < nkx; ++kx) {
          // operand A in shared memory: the MMAs read the stage itself
          if (ta ? issued >= SX && !mbar_wait(&xempty[st], ph ^ 1u, budget)
                 : !wait_done(issued - SX)) {
            ok = false;
            break;
          }
          if (H16) s_xbits[st] = xbits;
          mbar_expect_tx(&xfull[st], XBYTES);
          tma_load_4d(Xh(st), &L.maps[gi][0], &xfull[st], kx * KB, pt * TILE_P, cs, cb);
          ++issued;
          if (++st == SX) {
            st = 0;
            ph ^= 1u;
          }
        }
      }
      // drain: the latest use of every stage must have landed before exit
      for (long long q = (issued > SX ? issued - SX : 0); q < issued; ++q)
        mbar_wait(&xfull[q % SX], (uint32_t)(q / SX) & 1u, WAIT_NS);
    }
  } else if (warp == 14) {
    // ---------------- operator producer ----------------
    if (lane == 0) {
      if (res) {
        // the operator chunk of this CTA's slot, once
        const TcGroup& q = L.g[0];
        const uint32_t obytes = (uint32_t)q.Mtile * OROW;
        const int os = q.seg_op_map ? r_s : 0;
        for (int ko = 0; ko < r_nko; ++ko) {
          mbar_expect_tx(&ofull[ko], NOP * obytes);
          tma_load_3d(Op(ko), &L.maps[0][1], &ofull[ko], ko * KO, r_mc * q.Mtile, os);
          if (!B1)
            tma_load_3d(Op(ko) + omax, &L.maps[0][2], &ofull[ko], ko * KO, r_mc * q.Mtile, os);
        }
        for (int ko = 0; ko < r_nko; ++ko) mbar_wait(&ofull[ko], 0, WAIT_NS);
      } else {
        long long issued = 0;
        bool ok = true;
        int gi, pt, mc, b, s;
        int st = 0;
        for (long long li = 0; ok && tile_of(li, gi, pt, mc, b, s, false); ++li) {
          const TcGroup& q = L.g[gi];
          const int os = q.seg_op_map ? s : 0;
          const uint32_t obytes = (uint32_t)q.Mtile * OROW;
          const int nko = (q.d.K + KO - 1) / KO;
          for (int ko = 0; ko < nko; ++ko) {
            if (!wait_done(issued - SO)) {
              ok = false;
              break;
            }
            mbar_expect_tx(&ofull[st], NOP * obytes);
            tma_load_3d(Op(st), &L.maps[gi][1], &ofull[st], ko * KO, mc * q.Mtile, os);
            if (!B1)
              tma_load_3d(Op(st) + omax, &L.maps[gi][2], &ofull[st], ko * KO, mc * q.Mtile, os);
            ++issued;
            if (++st == SO) st = 0;
          }
        }
        for (long long q = (issued > SO ? issued - SO : 0); q < issued; ++q)
          mbar_wait(&ofull[q % SO], (uint32_t)(q / SO) & 1u, WAIT_NS);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // The whole warp walks the loop on warp-uniform values and one elected
    // lane issues: from a lane-0 branch every MMA cost ~99 clocks of address
    // and register moves, whatever its N; this way one of N = 128 takes the
    // tensor pipe's 64 (measured alone).  Same MMAs in the same order.
    // Every branch is on a warp-uniform value (waits through a vote), or the
    // addresses would leave the uniform registers.
    int li = 0;
    bool ok = true, issued_any = false;
    const uint64_t od0 = sdesc(smem_u32(obase));
    const uint64_t xd0 = sdesc(smem_u32(xbase));
    int gi, pt, mc, b, s;
    int sl = 0, so = 0;          // operand A slots of a block, operator stage
    uint32_t aph = 0, oph = 0;   // their use count parities
    unsigned kn = 0;             // K blocks so far, modulo S_MAX
    for (; ok && tile_of(li, gi, pt, mc, b, s, false); ++li) {
      if (G > 1) gi = __shfl_sync(0xffffffffu, gi, 0);
      const int mtile = __shfl_sync(0xffffffffu, L.g[gi].Mtile, 0);
      const uint32_t idesc = H16   ? idesc_f16(TILE_P, mtile)
                             : B16 ? idesc_b16(TILE_P, mtile)
                                   : idesc_tf32(TILE_P, mtile);
      const int nko = __shfl_sync(0xffffffffu, nkx_of(gi) / KXO, 0);
      const int buf = li & 1;
      const uint32_t use = (uint32_t)(li >> 1);
      if (li >= 2 && !warp_wait(&tempty[buf], (use & 1u) ^ 1u)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem + (uint32_t)buf * acc_stride;
      if (res) so = 0;
      for (int ko = 0; ko < nko; ++ko) {
        if (!warp_wait(&ofull[so], res ? 0u : oph) || !warp_wait(&conv[sl], aph)) {
          ok = false;
          break;
        }
        issued_any = true;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t oh = od0 + (((uint32_t)so * obytes_max) >> 4);
        const uint64_t ol = oh + (omax >> 4);
        const uint32_t ah = tmem + (uint32_t)A_COL0 + A_SLOT * KXO * (uint32_t)sl;
        const uint64_t xh = xd0 + (((uint32_t)sl * xstage) >> 4), xl = xh + (XBYTES >> 4);
        if (elect_one()) {
          if (B16) {
#pragma unroll
            for (int kk = 0; kk < KO / 16; ++kk) {
              // 16 elements = 32 B of the operator per MMA, 8 A columns (two
              // per slot of 32 elements)
              const uint32_t a1 = ah + A_SLOT * (kk / 2) + 8 * (kk % 2), a2 = a1 + A_SLOT / 2;
              mma_b16_ta(acc, a1, oh + 2 * kk, idesc, (ko | kk) ? 1u : 0u);
              if (!B1) {
                mma_b16_ta(acc, a1, ol + 2 * kk, idesc, 1u);
                mma_b16_ta(acc, a2, oh + 2 * kk, idesc, 1u);
              }
            }
          } else if (ta) {
            const uint32_t al = ah + A_SLOT / 2;
#pragma unroll
            for (int kk = 0; kk < KB / 8; ++kk) {
              // 8 TF32 = 32 B of the operator per MMA, 8 A columns
              mma_tf32_ta(acc, ah + 8 * kk, oh + 2 * kk, idesc, (ko | kk) ? 1u : 0u);
              mma_tf32_ta(acc, ah + 8 * kk, ol + 2 * kk, idesc, 1u);
              mma_tf32_ta(acc, al + 8 * kk, oh + 2 * kk, idesc, 1u);
            }
          } else {
#pragma unroll
            for (int kk = 0; kk < KB / 8; ++kk) {
              // 8 TF32 = 32 B per MMA
              mma_tf32(acc, xh + 2 * kk, oh + 2 * kk, idesc, (ko | kk) ? 1u : 0u);
              mma_tf32(acc, xh + 2 * kk, ol + 2 * kk, idesc, 1u);
              mma_tf32(acc, xl + 2 * kk, oh + 2 * kk, idesc, 1u);
            }
          }
          mma_commit(&kdone[kn]);
        }
        __syncwarp();
        if (++sl == SA / KXO) {
          sl = 0;
          aph ^= 1u;
        }
        kn = (kn + 1) % S_MAX;
        ++so;
        if (!res && so == SO) {
          so = 0;
          oph ^= 1u;
        }
      }
      if (ok && elect_one()) mma_commit(&tfull[buf]);
      __syncwarp();
    }
    // after a timeout the MMAs already issued must finish before the TMEM
    // they write is freed: one more commit tracks all of them
    if (!ok && issued_any) {
      if (elect_one()) mma_commit(mma_done);
      __syncwarp();
      mbar_wait(mma_done, 0, WAIT_NS);
    }
  } else if (warp < 6 || warp > 14) {
    // ---------------- split staged input tiles into TF32 hi (in place) / lo ----------------
    // Two groups of four warps (one per TMEM lane quarter) take K blocks in
    // turn.  A stage must then always be the same group's (a whole number of
    // turns per ring): a parity wait cannot skip a phase that the other group
    // waits for.  Else the first group takes all blocks.
    const int grp = warp < 6 ? 0 : 1;
    const bool two = nthreads(EPI, BETA, PREC) == 608 && SX % (2 * KXO) == 0;
    const int ct = threadIdx.x - (grp ? 480 : 64);  // 0..127
    // TMEM mode: thread = row r of the tile (its warp's lane quarter), reads
    // its 32 values from the 128-byte-swizzled tile and stores hi / lo into
    // its TMEM lane with tcgen05.st.
    const int row = 32 * (warp & 3) + lane;
    bool ok = true;
    int gi, pt, mc, b, s;
    int st = 0, sl = 0;          // input stage, operand A slot
    uint32_t ph = 0;             // use count parity of the stage
    long long kn = 0;            // K block
    float xsc = 1.f, xinv = 1.f;
    for (long long li = 0; ok && tile_of(li, gi, pt, mc, b, s, false); ++li) {
      const int nkx = nkx_of(gi);
      for (int kx = 0; kx < nkx; ++kx) {
        if ((two ? (int)(kn & 1) : 0) != grp) {
          if (++st == SX) {
            st = 0;
            ph ^= 1u;
          }
          if (++sl == SA) sl = 0;
          if (kx % KXO == KXO - 1) ++kn;
          continue;
        }
        if (!warp_wait(&xfull[st], ph)) {
          ok = false;
          break;
        }
        if (H16 && kx % KXO == 0) h16_scale_bits(s_xbits[st], xsc, xinv);
        const uint32_t tbase = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)A_COL0 +
                               A_SLOT * (uint32_t)sl;
        if (ta) {
          // 32 FP32 of this row -> hi and lo: TF32 words, or 16-bit pairs
          // packed two to a column (lower k in the lower half; FP16 scaled by
          // the problem's power of two)
          constexpr int W = B16 ? 16 : 32;
          uint32_t h[W], l[W];
          const float4* xr = (const float4*)(Xh(st) + row * 128);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float4 v = xr[c ^ (row & 7)];
            if constexpr (H16) {
              const float a0 = v.x * xsc, a1 = v.y * xsc, a2 = v.z * xsc, a3 = v.w * xsc;
              const uint32_t h0 = pack_f16x2(a0, a1), h1 = pack_f16x2(a2, a3);
              const float2 f0 = unpack_f16x2(h0), f1 = unpack_f16x2(h1);
              h[2 * c] = h0;
              h[2 * c + 1] = h1;
              l[2 * c] = pack_f16x2(a0 - f0.x, a1 - f0.y);
              l[2 * c + 1] = pack_f16x2(a2 - f1.x, a3 - f1.y);
            } else if constexpr (B16) {
              const uint32_t h0 = pack_bf16x2(v.x, v.y), h1 = pack_bf16x2(v.z, v.w);
              h[2 * c] = h0;
              h[2 * c + 1] = h1;
              if (!B1) {
                l[2 * c] = pack_bf16x2(v.x - __uint_as_float(h0 << 16),
                                       v.y - __uint_as_float(h0 & 0xFFFF0000u));
                l[2 * c + 1] = pack_bf16x2(v.z - __uint_as_float(h1 << 16),
                                           v.w - __uint_as_float(h1 & 0xFFFF0000u));
              }
            } else {
              const float hv[4] = {tf32_hi(v.x), tf32_hi(v.y), tf32_hi(v.z), tf32_hi(v.w)};
              const float vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                h[4 * c + e] = __float_as_uint(hv[e]);
                l[4 * c + e] = __float_as_uint(vv[e] - hv[e]);
              }
            }
          }
          if (kx % KXO == 0 && !__all_sync(0xffffffffu, wait_done(kn - SA / KXO))) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if constexpr (B16) {
            tmem_st16(tbase, h);
            if (!B1) tmem_st16(tbase + A_SLOT / 2, l);
          } else {
            tmem_st32(tbase, h);
            tmem_st32(tbase + A_SLOT / 2, l);
          }
          if (kx % KXO == KXO - 1) {  // hand over a whole operator block's K
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          }
        } else {
          float4* xh = (float4*)Xh(st);
          float4* xl = (float4*)Xl(st);
#pragma unroll
          for (int i = 0; i < (int)(XBYTES / 16 / 128); ++i) {
            const int idx = ct + i * 128;
            float4 v = xh[idx];
            float4 h = make_float4(tf32_hi(v.x), tf32_hi(v.y), tf32_hi(v.z), tf32_hi(v.w));
            xh[idx] = h;
            xl[idx] = make_float4(v.x - h.x, v.y - h.y, v.z - h.z, v.w - h.w);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncwarp();
        if (lane == 0) {
          if (kx % KXO == KXO - 1) mbar_arrive(&conv[sl / KXO]);
          // the block is read (its values are stored): its stage may be filled
          // again while the MMAs still work on earlier slots
          if (ta) mbar_arrive(&xempty[st]);
        }
        if (++st == SX) {
          st = 0;
          ph ^= 1u;
        }
        if (++sl == SA) sl = 0;
        if (kx % KXO == KXO - 1) ++kn;
      }
    }
  } else {
    // ---------------- epilogue: TMEM -> registers -> global ----------------
    // Eight warps: two per TMEM lane quarter, each taking every other group
    // of 32 accumulator columns in blocks of 16.  A lane holds one p of all m,
    // so that a store (or a field load) of one m is 128 contiguous bytes of
    // the warp: registers go straight to global memory.  Staging the tile in
    // shared memory for bulk tensor stores cost the epilogue the copy, a proxy
    // fence and a wait per 32 x 32 box.  Per-row factors (eigenvalues, operator
    // scales) are held one per lane and broadcast; the field values of block
    // k + 1 are loaded while block k is processed, those of block 0 before the
    // accumulator wait.
    const int q4 = warp & 3;  // TMEM lane quarter this warp may access
    const int half = (warp - 6) >> 2;
    const int row = 32 * q4 + lane;
    int li = 0;
    // test hook: a barrier nothing arrives on; its wait runs out (status set)
    // and this warp skips its tiles, so every other role's waits run out too
    const bool held = s_hold != 0 && !mbar_wait(hold, 0, budget);
    const int ew = warp - 6;
    int gi, pt, mc, b, s;
    for (; !held && tile_of(li, gi, pt, mc, b, s); ++li) {
      const TcGroup& q = L.g[gi];
      const jfg_contract_desc& d = q.d;
      const int Mt = q.Mtile;
      const float alpha = (float)d.alpha, beta = (float)d.beta;
      const int buf = li & 1;
      const int p = pt * TILE_P + row;
      const bool pin = p < d.P && b >= 0;
      const int bb = b < 0 ? 0 : b;
      const int mt0 = mc * Mt;
      const bool full = mt0 + Mt <= d.M;  // no row of the tile is past M
      float* outT = q.out + (long long)bb * d.out_batch + (long long)s * d.out_seg +
                    (long long)mt0 * d.out_ld + p;
      float c0 = 0.f, c1 = 1.f, lp = 0.f;
      if (EPI == JFG_EPI_DIV_EIG) {
        c0 = d.c0 ? __ldg((const float*)d.c0 + bb) : 0.f;
        c1 = d.c1 ? __ldg((const float*)d.c1 + bb) : 1.f;
        lp = pin ? __ldg((const float*)d.lam_p + p) : 0.f;
      }
      const float* __restrict__ fld = nullptr;
      if (EPI == JFG_EPI_MUL_FIELD)
        fld = (const float*)d.field + (long long)bb * d.field_batch + (long long)s * d.field_seg +
              (long long)mt0 * d.field_ld + p;
      float omax = 0.f, dsum = 0.f;
      const bool fdot = EPI != JFG_EPI_NONE && q.dot_part != nullptr;
      const int ncb = Mt / 16;
      // block k: columns 16 cb(k) .. + 15; pairs of blocks are 32 columns
      auto cb_of = [&](int k) { return half * 2 + 4 * (k >> 1) + (k & 1); };
      // this lane's row of each pair: operator scale times the problem's, eigenvalue
      float os0 = 0.f, os1 = 0.f, lm0 = 1.f, lm1 = 1.f;
      if (H16 || EPI == JFG_EPI_DIV_EIG) {
        const int ma = mt0 + 32 * half + lane, mb = ma + 64;
        const bool oka = 32 * half + lane < Mt && ma < d.M, okb = 32 * half + lane + 64 < Mt && mb < d.M;
        if (H16) {
          float xsc, xinv;
          h16_scale(q.in_max, b, xsc, xinv);
          const float* __restrict__ oinv = q.op_inv + (long long)s * q.op_inv_seg;
          os0 = oka ? __ldg(oinv + ma) * xinv : 0.f;
          os1 = okb ? __ldg(oinv + mb) * xinv : 0.f;
        }
        if (EPI == JFG_EPI_DIV_EIG) {
          lm0 = oka ? __ldg((const float*)d.lam_m + ma) : 1.f;
          lm1 = okb ? __ldg((const float*)d.lam_m + mb) : 1.f;
        }
      }
      auto load_field = [&](int cb, float* f) {
        const float* src = fld + (long long)(16 * cb) * d.field_ld;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          f[j] = pin && (full || mt0 + 16 * cb + j < d.M) ? __ldg(src) : 0.f;
          src += d.field_ld;
        }
      };
      float f[16], fn[16];
      if (EPI == JFG_EPI_MUL_FIELD && cb_of(0) < ncb) load_field(cb_of(0), f);
      if (!warp_wait(&tfull[buf], (uint32_t)(li >> 1) & 1u)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tacc = tmem + ((uint32_t)(32 * q4) << 16) + (uint32_t)buf * acc_stride;
#pragma unroll 1
      for (int k = 0; cb_of(k) < ncb; ++k) {
        const int cb = cb_of(k);
        const int mh = mt0 + 16 * cb;
        if (EPI == JFG_EPI_MUL_FIELD && cb_of(k + 1) < ncb) load_field(cb_of(k + 1), fn);
        float* o = outT + (long long)(16 * cb) * d.out_ld;
        float prev[16];
        if (BETA) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            prev[j] = pin && (full || mh + j < d.M) ? o[(long long)j * d.out_ld] : 0.f;
        }
        float v[16];
        tmem_ld16(tacc + (uint32_t)(cb * 16), v);
        const float osr = k < 2 ? os0 : os1, lmr = k < 2 ? lm0 : lm1;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int src = 16 * (k & 1) + j;
          float r = v[j];
          if (H16) r *= __shfl_sync(0xffffffffu, osr, src);
          const float a = r;  // the contraction before the epilogue factor
          if (EPI == JFG_EPI_MUL_FIELD) r *= f[j];
          if (EPI == JFG_EPI_DIV_EIG)
            r = __fdividef(r, c0 + c1 * (__shfl_sync(0xffffffffu, lmr, src) + lp));
          r *= alpha;
          if (fdot) dsum = fmaf(a, r, dsum);
          if (BETA) r += beta * prev[j];
          if (H16) omax = fmaxf(omax, fabsf(r));
          v[j] = r;
        }
        if (pin) {
          if (full) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              *o = v[j];
              o += d.out_ld;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              if (mh + j < d.M) *o = v[j];
              o += d.out_ld;
            }
          }
        }
        if (EPI == JFG_EPI_MUL_FIELD) {
#pragma unroll
          for (int j = 0; j < 16; ++j) f[j] = fn[j];
        }
        __syncwarp();  // the next block's TMEM load takes the whole warp
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[buf]);
      if (fdot) {
        // this warp's partial of the tile, one deterministic slot each
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dsum += __shfl_xor_sync(0xffffffffu, dsum, o);
        const int mch = (d.M + Mt - 1) / Mt, npt = (d.P + TILE_P - 1) / TILE_P;
        if (lane == 0 && b >= 0)
          q.dot_part[(long long)b * DOT_NBMAX + ((s * mch + mc) * npt + pt) * 8 + ew] = dsum;
      }
      if (H16 && q.out_max != nullptr) {
        // max |output| of this tile for the next pass's input scale (float
        // bits of non-negative values order like unsigned integers)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) omax = fmaxf(omax, __shfl_xor_sync(0xffffffffu, omax, o));
        if (lane == 0 && b >= 0) atomicMax(q.out_max + b, __float_as_uint(omax));
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(L.tmem_cols)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

int make_map(CUtensorMap* map, const void* base, int rank, const cuuint64_t* dims,
             const cuuint64_t* strides_bytes, const cuuint32_t* box,
             CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
             CUtensorMapSwizzle sw = CU_TENSOR_MAP_SWIZZLE_128B) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return JFG_ERR_UNSUPPORTED;
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = fn(map, dt, (cuuint32_t)rank, (void*)base, dims,
                  strides_bytes, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? JFG_OK : JFG_ERR_ARG;
}

// the plain BF16 kernel exists for the epilogues of the fast diagonalisation
template <int E>
int set_attr_b1(int mx) {
  if constexpr (E != JFG_EPI_MUL_FIELD)
    JFG_CUDA_TRY(cudaFuncSetAttribute(k_contract_tc<E, false, 1, 3>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
  return JFG_OK;
}

// Opt every kernel variant into the largest dynamic shared-memory size once
// per device (before any stream capture can be active in the caller).
int setup_kernel_attr() {
  static bool done[64] = {};
  int dev = 0;
  JFG_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return JFG_ERR_UNSUPPORTED;
  if (!done[dev]) {
    const int mx = SMEM_MAX;
#define JFG_SET_ATTR(E, B, G)                                                              \
  JFG_CUDA_TRY(cudaFuncSetAttribute(k_contract_tc<E, B, G, 0>,                             \
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, mx));     \
  JFG_CUDA_TRY(cudaFuncSetAttribute(k_contract_tc<E, B, G, 1>,                             \
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, mx));     \
  if (G == 1)                                                                              \
  JFG_CUDA_TRY(cudaFuncSetAttribute(k_contract_tc<E, B, 1, 2>,                             \
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, mx));     \
  if (G == 1 && !B) JFG_TRY(set_attr_b1<E>(mx))
#define JFG_SET_ATTR_G(G)                   \
  JFG_SET_ATTR(JFG_EPI_NONE, false, G);     \
  JFG_SET_ATTR(JFG_EPI_NONE, true, G);      \
  JFG_SET_ATTR(JFG_EPI_MUL_FIELD, false, G); \
  JFG_SET_ATTR(JFG_EPI_MUL_FIELD, true, G); \
  JFG_SET_ATTR(JFG_EPI_DIV_EIG, false, G);  \
  JFG_SET_ATTR(JFG_EPI_DIV_EIG, true, G)
    JFG_SET_ATTR_G(1);
    JFG_SET_ATTR_G(GMAX);
#undef JFG_SET_ATTR_G
#undef JFG_SET_ATTR
    done[dev] = true;
  }
  return JFG_OK;
}

// Validate one group and fill its descriptor, tile height and tensor maps.
// prec: 0 the operator is TF32 in FP32 words; 1 BF16 (hi, lo) and 2 FP16
// (hi, lo), both with 64-element K blocks; 3 BF16 hi only (op_lo unused).
int fill_group(const jfg_contract_desc& d, const void* op_hi, const void* op_lo,
               const float* in, float* out, TcGroup& q, CUtensorMap* maps, int prec,
               int mt_cap) {
  const bool b16 = prec != 0;
  JFG_TRY(validate_desc(d));
  const bool lo = prec != 3;
  if (!op_hi || (lo && !op_lo) || !in || !out) return JFG_ERR_ARG;
  // TMA: 16-byte aligned bases and strides
  auto al16 = [](const void* p) { return ((uintptr_t)p & 15u) == 0; };
  if (!al16(op_hi) || (lo && !al16(op_lo)) || !al16(in)) return JFG_ERR_ARG;
  const int om = b16 ? 7 : 3;  // operator strides in elements: multiples of 16 bytes
  if ((d.op_ld & om) || (d.in_ld & 3) || (d.op_seg & om) || (d.in_seg & 3) || (d.in_batch & 3))
    return JFG_ERR_ARG;
  if ((long long)d.batch * d.nseg > 65535) return JFG_ERR_ARG;
  q.d = d;
  q.out = out;
  const int cap = (mt_cap > 0 && mt_cap < MT_MAX) ? mt_cap : MT_MAX;
  q.Mtile = ((d.M > cap ? cap : d.M) + 15) / 16 * 16;
  q.seg_in_map = (d.nseg > 1 && d.in_seg != 0) ? 1 : 0;
  q.bat_in_map = (d.batch > 1 && d.in_batch != 0) ? 1 : 0;
  q.seg_op_map = (d.nseg > 1 && d.op_seg != 0) ? 1 : 0;
  // inputs that do not stay in L2 are read once if their operator chunks run together
  q.mc_inner = (double)d.P * d.K * 4.0 * d.batch * d.nseg > 64.0 * 1024 * 1024 ? 1 : 0;
  {
    cuuint64_t dims[4] = {(cuuint64_t)d.K, (cuuint64_t)d.P,
                          (cuuint64_t)(q.seg_in_map ? d.nseg : 1),
                          (cuuint64_t)(q.bat_in_map ? d.batch : 1)};
    cuuint64_t str[3] = {(cuuint64_t)d.in_ld * 4,
                         (cuuint64_t)(q.seg_in_map ? d.in_seg : d.in_ld * d.P) * 4,
                         (cuuint64_t)(q.bat_in_map ? d.in_batch : d.in_ld * d.P) * 4};
    cuuint32_t box[4] = {KB, TILE_P, 1, 1};
    JFG_TRY(make_map(&maps[0], in, 4, dims, str, box));
  }
  {
    const int eb = b16 ? 2 : 4;
    cuuint64_t dims[3] = {(cuuint64_t)d.K, (cuuint64_t)d.M,
                          (cuuint64_t)(q.seg_op_map ? d.nseg : 1)};
    cuuint64_t str[2] = {(cuuint64_t)d.op_ld * eb,
                         (cuuint64_t)(q.seg_op_map ? d.op_seg : d.op_ld * d.M) * eb};
    cuuint32_t box[3] = {(cuuint32_t)op_ke(b16), (cuuint32_t)q.Mtile, 1};
    const CUtensorMapDataType dt = prec == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                   : b16     ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                             : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    JFG_TRY(make_map(&maps[1], op_hi, 3, dims, str, box, dt));
    if (lo) JFG_TRY(make_map(&maps[2], op_lo, 3, dims, str, box, dt));
  }
  return JFG_OK;
}

long long group_tiles(const TcGroup& q) {
  return (long long)((q.d.P + TILE_P - 1) / TILE_P) * ((q.d.M + q.Mtile - 1) / q.Mtile) *
         q.d.batch * q.d.nseg;
}

// One launch over ng <= G groups (same epilogue kind and beta != 0 for all).
// The scaled split-FP16 kernel exists for single-group launches only.
template <int E, bool BETA, int G>
void launch_h16(dim3 grid, size_t smem, cudaStream_t st, const TcLaunch<G>& L) {
  if constexpr (G == 1) k_contract_tc<E, BETA, 1, 2><<<grid, nthreads(E, BETA, 2), smem, st>>>(L);
}
// ... and so does the plain BF16 kernel (the fast diagonalisation's passes:
// no beta, no field)
template <int E, bool BETA, int G>
void launch_b1(dim3 grid, size_t smem, cudaStream_t st, const TcLaunch<G>& L) {
  if constexpr (G == 1 && !BETA && E != JFG_EPI_MUL_FIELD)
    k_contract_tc<E, false, 1, 3><<<grid, nthreads(E, false, 3), smem, st>>>(L);
}

// h16 (one group only): the scaled split-FP16 auxiliaries of that group.
struct H16Aux {
  const unsigned* in_max;
  unsigned* out_max;
  const float* op_inv;
  long long op_inv_seg;
};

template <int G>
int launch_groups(int ng, const jfg_contract_desc* const* ds, const void* const* op_hi,
                  const void* const* op_lo, const float* const* in, float* const* out,
                  const jfg_tc_config& cfg, int prec, cudaStream_t st,
                  const H16Aux* h16 = nullptr, const DotOut* dot = nullptr) {
  if (dot && dot->nb) *dot->nb = 0;
  const bool b16 = prec != 0;
  if (prec == 2 && (G != 1 || ng != 1 || !h16 || !h16->op_inv)) return JFG_ERR_ARG;
  if (prec == 3 && (G != 1 || ng != 1 || ds[0]->beta != 0.0 ||
                    ds[0]->epilogue == JFG_EPI_MUL_FIELD))
    return JFG_ERR_ARG;
  static_assert(sizeof(TcLaunch<G>) <= 32000, "kernel parameter block too large");
  TcLaunch<G> L;
  memset(&L, 0, sizeof(L));
  L.ngroups = ng;
  const int epi = ds[0]->epilogue;
  const bool hb = ds[0]->beta != 0.0;
  long long tiles = 0;
  int mt_max = 16;
  for (int i = 0; i < ng; ++i) {
    if (ds[i]->epilogue != epi || (ds[i]->beta != 0.0) != hb) return JFG_ERR_ARG;
    JFG_TRY(fill_group(*ds[i], op_hi[i], op_lo[i], in[i], out[i], L.g[i], L.maps[i], prec,
                       cfg.mtile));
    if (h16) {
      L.g[i].in_max = h16->in_max;
      L.g[i].out_max = h16->out_max;
      L.g[i].op_inv = h16->op_inv;
      L.g[i].op_inv_seg = h16->op_inv_seg;
    }
    tiles += group_tiles(L.g[i]);
    if (L.g[i].Mtile > mt_max) mt_max = L.g[i].Mtile;
  }
  if (tiles == 0) return JFG_OK;
  int dev = 0, nsm = 0;
  JFG_CUDA_TRY(cudaGetDevice(&dev));
  JFG_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  int ctas = cfg.ctas > 0 && cfg.ctas < nsm ? cfg.ctas : nsm;
  const int ta = (b16 || cfg.operand_a_in_tmem) ? 1 : 0;
  // Shared memory: operator blocks and input blocks.  The input
  // ring holds blocks of 16 KB (32 with the lo part beside it); the operator's
  // blocks stream through a ring of their own, or (operator-stationary
  // schedule, one group) each CTA keeps one chunk of it, all K of hi and lo,
  // and streams only input tiles, halving the L2-to-SM traffic per tile.
  const size_t oblock = (prec == 3 ? 1 : 2) * (size_t)mt_max * 128;
  const size_t xblock = (ta ? 1 : 2) * (size_t)XBYTES;
  const size_t fixed = 1024 + (5 * S_MAX + 8) * 8;
  const size_t room = (size_t)SMEM_MAX - fixed;
  bool res = false;
  int nslots = 0, nko = 0;
  const int sched = cfg.schedule == 1 ? 0 : cfg.schedule == 2 ? 2 : g_op_resident;
  if (ng == 1 && sched) {
    const TcGroup& q = L.g[0];
    nslots = q.d.nseg * ((q.d.M + q.Mtile - 1) / q.Mtile);
    nko = (q.d.K + op_ke(b16) - 1) / op_ke(b16);
    const long long per_slot = (long long)((q.d.P + TILE_P - 1) / TILE_P) * q.d.batch;
    res = nslots <= ctas && nko <= S_MAX &&
          (sched == 2 ? nko * oblock + 2 * xblock <= room
                      : !q.mc_inner && (nthreads(epi, hb, prec) != 608 || prec == 3) &&
                            per_slot * nslots >= 2LL * ctas &&
                            nko * oblock + 4 * xblock <= room);
  }
  // operand A in TMEM: 256 accumulator columns plus the slots
  const int amax = ta ? (b16 ? 8 : 4) : S_MAX;
  const size_t left = room - (res ? nko * oblock : 0);
  int xs, os;
  if (res) {
    xs = (int)(left / xblock);
    os = 0;
  } else {
    // as many bytes of operator as of input in flight (per 64 K of 16-bit
    // operators 32 KB of each), at least two operator and two input blocks
    const int xper = op_ke(b16) / KB;  // input blocks per operator block
    os = (int)(left / (oblock + xper * xblock));
    if (os < 2) os = 2;
    if (os > S_MAX) os = S_MAX;
    if (left < os * oblock + 2 * xblock) return JFG_ERR_UNSUPPORTED;
    xs = (int)((left - os * oblock) / xblock);
  }
  if (xs > 12) xs = 12;
  // whole turns of the two splitting groups
  const int turn = 2 * op_ke(b16) / KB;
  if (nthreads(epi, hb, prec) == 608 && xs >= turn) xs = xs / turn * turn;
  if (cfg.stages >= 2 && cfg.stages < xs) xs = cfg.stages;
  if (cfg.stages >= 2 && cfg.stages < os) os = cfg.stages;
  if (xs < 2) return JFG_ERR_UNSUPPORTED;
  L.xstages = xs;
  L.ostages = os;
  L.aslots = ta ? amax : xs;
  L.tmem_cols = 512;  // two accumulator buffers (+ operand A slots in TMEM mode)
  L.tmem_a = ta;
  L.mt_max = mt_max;
  L.op_res = res ? 1 : 0;
  L.nslots = res ? nslots : 0;
  if (dot && dot->part && ng == 1) {
    // fused dot: field or divide epilogue, <= DOT_NBMAX partials per problem
    TcGroup& q = L.g[0];
    const int e = q.d.epilogue;
    const long long nb = (long long)q.d.nseg * ((q.d.M + q.Mtile - 1) / q.Mtile) *
                         ((q.d.P + TILE_P - 1) / TILE_P) * 8;
    if ((e == JFG_EPI_DIV_EIG || e == JFG_EPI_MUL_FIELD) && q.d.beta == 0.0 &&
        nb <= DOT_NBMAX) {
      q.dot_part = dot->part;
      if (dot->nb) *dot->nb = (int)nb;
    }
  }
  const size_t smem = fixed + (res ? nko : os) * oblock + xs * xblock;
  if (smem > (size_t)SMEM_MAX) return JFG_ERR_UNSUPPORTED;
  long long nct = tiles < ctas ? tiles : ctas;
  if (res) nct = (long long)(ctas / nslots) * nslots;  // the same CTA count per slot
  dim3 grid((unsigned)nct);
  JFG_TRY(setup_kernel_attr());
#define JFG_LAUNCH(E)                                                          \
  do {                                                                         \
    if (prec == 2) {                                                           \
      if (hb)                                                                  \
        launch_h16<E, true, G>(grid, smem, st, L);                             \
      else                                                                     \
        launch_h16<E, false, G>(grid, smem, st, L);                            \
    } else if (prec == 3) {                                                    \
      launch_b1<E, false, G>(grid, smem, st, L);                               \
    } else if (b16) {                                                          \
      if (hb)                                                                  \
        k_contract_tc<E, true, G, 1><<<grid, nthreads(E, true, 1), smem, st>>>(L);         \
      else                                                                     \
        k_contract_tc<E, false, G, 1><<<grid, nthreads(E, false, 1), smem, st>>>(L);        \
    } else {                                                                   \
      if (hb)                                                                  \
        k_contract_tc<E, true, G, 0><<<grid, nthreads(E, true, 0), smem, st>>>(L);         \
      else                                                                     \
        k_contract_tc<E, false, G, 0><<<grid, nthreads(E, false, 0), smem, st>>>(L);        \
    }                                                                          \
  } while (0)
  switch (epi) {
    case JFG_EPI_NONE:
      JFG_LAUNCH(JFG_EPI_NONE);
      break;
    case JFG_EPI_MUL_FIELD:
      JFG_LAUNCH(JFG_EPI_MUL_FIELD);
      break;
    case JFG_EPI_DIV_EIG:
      JFG_LAUNCH(JFG_EPI_DIV_EIG);
      break;
    default:
      return JFG_ERR_ARG;
  }
#undef JFG_LAUNCH
  JFG_LAUNCHED();
  return JFG_OK;
}

}  // namespace

int tc_setup() {
  if (!encode_fn()) return JFG_ERR_UNSUPPORTED;
  return setup_kernel_attr();
}

jfg_tc_config tc_default_config() {
  jfg_tc_config c;
  c.operand_a_in_tmem = g_operand_a_in_tmem;
  c.order = 0;
  c.ctas = 0;
  c.stages = 0;
  c.mtile = 0;
  c.schedule = 0;
  c.store = 0;
  return c;
}

// ---- single-group launches: tuned configurations -------------------------

struct SingleTuned {
  jfg_tc_config cfg;
  float ms;
};
std::mutex g_single_mu;
std::map<std::string, SingleTuned> g_single;
int g_tune_single = 0;

std::string single_signature(int prec, const jfg_contract_desc& d) {
  int dev = 0;
  cudaGetDevice(&dev);
  char buf[200];
  snprintf(buf, sizeof buf, "d%d:p%d:b%d:s%d:M%d:P%d:K%d:e%d:beta%d", dev, prec, d.batch, d.nseg,
           d.M, d.P, d.K, d.epilogue, d.beta != 0.0 ? 1 : 0);
  return buf;
}

// Time every candidate configuration of this launch on its own operands and
// keep the fastest for its signature.
int tune_single(int prec, const jfg_contract_desc& d, const void* oh, const void* ol,
                const float* in, float* out, const H16Aux* aux, cudaStream_t st,
                const std::string& key, jfg_tc_config* best) {
  const jfg_contract_desc* dp = &d;
  std::vector<jfg_tc_config> cands;
  for (int ta : {1, 0})
    for (int sched : {1, 2})
      for (int sg : {0, 3, 2})
        for (int mt : {0, 64}) {
            if (prec != 0 && ta == 0) continue;
            // the operator-stationary schedule only where the chunk fits beside
            // two input blocks (else the launch would stream anyway)
            const int ke = op_ke(prec != 0);
            if (sched == 2 && (size_t)((d.K + ke - 1) / ke) * (prec == 3 ? 1 : 2) *
                                          (mt ? mt : 128) * 128 +
                                      2 * (size_t)XBYTES >
                                  (size_t)SMEM_MAX - 4096)
              continue;
            jfg_tc_config c = tc_default_config();
            c.operand_a_in_tmem = ta;
            c.schedule = sched;
            c.stages = sg;
            c.mtile = mt;
            cands.push_back(c);
          }
  cudaEvent_t e0, e1;
  JFG_CUDA_TRY(cudaEventCreate(&e0));
  JFG_CUDA_TRY(cudaEventCreate(&e1));
  const int reps = 3;
  float bt = -1.f;
  jfg_tc_config bc = tc_default_config();
  int status = JFG_OK;
  for (const jfg_tc_config& c : cands) {
    int s = launch_groups<1>(1, &dp, &oh, &ol, &in, &out, c, prec, st, aux);  // warm
    if (s == JFG_ERR_UNSUPPORTED) continue;  // does not fit: not a candidate
    if (s != JFG_OK) {
      status = s;
      break;
    }
    if (cudaEventRecord(e0, st) != cudaSuccess) {
      status = JFG_ERR_CUDA;
      break;
    }
    for (int r = 0; r < reps && s == JFG_OK; ++r)
      s = launch_groups<1>(1, &dp, &oh, &ol, &in, &out, c, prec, st, aux);
    float ms = 0.f;
    if (s != JFG_OK || cudaEventRecord(e1, st) != cudaSuccess ||
        cudaEventSynchronize(e1) != cudaSuccess || cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) {
      status = s != JFG_OK ? s : JFG_ERR_CUDA;
      break;
    }
    ms /= (float)reps;
    if (bt < 0.f || ms < bt) {
      bt = ms;
      bc = c;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (status != JFG_OK) return status;
  if (bt >= 0.f) {
    std::lock_guard<std::mutex> lk(g_single_mu);
    g_single[key] = SingleTuned{bc, bt};
  }
  *best = bc;
  return JFG_OK;
}

// One single-group launch with the tuned configuration of its signature (or
// the default); with autotuning on, an untuned signature launched outside
// stream capture is tuned first.
// jfg_tc_force_config: one configuration for every single-group launch
// (tests and tuning studies), instead of the tuned or default one
bool g_force_on = false;
jfg_tc_config g_force_cfg;

int launch_single(int prec, const jfg_contract_desc& d, const void* oh, const void* ol,
                  const float* in, float* out, const H16Aux* aux, cudaStream_t st,
                  const DotOut* dot = nullptr) {
  const jfg_contract_desc* dp = &d;
  jfg_tc_config cfg = tc_default_config();
  const std::string key = single_signature(prec, d);
  bool found = false;
  {
    std::lock_guard<std::mutex> lk(g_single_mu);
    if (g_force_on) {
      cfg = g_force_cfg;
      found = true;
    } else {
      auto it = g_single.find(key);
      if (it != g_single.end()) {
        cfg = it->second.cfg;
        found = true;
      }
    }
  }
  if (!found && g_tune_single) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    JFG_CUDA_TRY(cudaStreamIsCapturing(st, &cs));
    if (cs == cudaStreamCaptureStatusNone)
      JFG_TRY(tune_single(prec, d, oh, ol, in, out, aux, st, key, &cfg));
  }
  return launch_groups<1>(1, &dp, &oh, &ol, &in, &out, cfg, prec, st, aux, dot);
}

int contract_tc(const jfg_contract_desc& d, const float* op_hi, const float* op_lo,
                const float* in, float* out, cudaStream_t st, const DotOut* dot) {
  if (dot && dot->nb) *dot->nb = 0;
  if (d.batch == 0 || d.M == 0 || d.P == 0) return validate_desc(d);
  return launch_single(0, d, op_hi, op_lo, in, out, nullptr, st, dot);
}

int contract_tc_b16(const jfg_contract_desc& d, const uint16_t* op_hi, const uint16_t* op_lo,
                    const float* in, float* out, cudaStream_t st, const DotOut* dot) {
  if (dot && dot->nb) *dot->nb = 0;
  if (d.batch == 0 || d.M == 0 || d.P == 0) return validate_desc(d);
  return launch_single(op_lo ? 1 : 3, d, op_hi, op_lo, in, out, nullptr, st, dot);
}

int contract_tc_h16(const jfg_contract_desc& d, const uint16_t* op_hi, const uint16_t* op_lo,
                    const float* op_inv, long long op_inv_seg, const unsigned* in_max,
                    unsigned* out_max, const float* in, float* out, cudaStream_t st,
                    const DotOut* dot) {
  if (dot && dot->nb) *dot->nb = 0;
  if (d.batch == 0 || d.M == 0 || d.P == 0) return validate_desc(d);
  if (!op_inv || !in_max) return JFG_ERR_ARG;
  const H16Aux aux{in_max, out_max, op_inv, op_inv_seg};
  return launch_single(2, d, op_hi, op_lo, in, out, &aux, st, dot);
}

void set_single_autotune(int on) { g_tune_single = on; }
int single_autotune() { return g_tune_single; }

int contract_tc_grouped(int ng, const jfg_contract_desc* ds, const float* const* op_hi,
                        const float* const* op_lo, const float* const* in, float* const* out,
                        const jfg_tc_config& cfg, cudaStream_t st) {
  if (ng < 0 || (ng > 0 && (!ds || !op_hi || !op_lo || !in || !out))) return JFG_ERR_ARG;
  if (cfg.order < 0 || cfg.order > 2 || cfg.stages < 0 || cfg.ctas < 0 ||
      (cfg.mtile != 0 && cfg.mtile != 64))
    return JFG_ERR_ARG;
  // launch order of the groups: as given, by operator-tile work (K * Mtile,
  // largest first), or by total work (largest first)
  std::vector<int> ord;
  ord.reserve(ng);
  for (int i = 0; i < ng; ++i)
    if (ds[i].batch > 0 && ds[i].M > 0 && ds[i].P > 0) ord.push_back(i);
    else JFG_TRY(validate_desc(ds[i]));
  auto work = [&](int i) {
    const double mt = ds[i].M < MT_MAX ? ds[i].M : MT_MAX;
    const double tile = (double)ds[i].K * mt;
    if (cfg.order == 1) return tile;
    return tile * (double)((ds[i].P + TILE_P - 1) / TILE_P) *
           (double)((ds[i].M + MT_MAX - 1) / MT_MAX) * ds[i].batch * ds[i].nseg;
  };
  if (cfg.order != 0)
    std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) { return work(a) > work(b); });
  for (size_t c0 = 0; c0 < ord.size(); c0 += GMAX) {
    const int n = (int)(ord.size() - c0 < (size_t)GMAX ? ord.size() - c0 : GMAX);
    const jfg_contract_desc* dp[GMAX];
    const void* oh[GMAX];
    const void* ol[GMAX];
    const float* ip[GMAX];
    float* op[GMAX];
    for (int k = 0; k < n; ++k) {
      const int i = ord[c0 + k];
      dp[k] = &ds[i];
      oh[k] = op_hi[i];
      ol[k] = op_lo[i];
      ip[k] = in[i];
      op[k] = out[i];
    }
    if (n == 1)
      JFG_TRY(launch_groups<1>(1, dp, oh, ol, ip, op, cfg, 0, st));
    else
      JFG_TRY(launch_groups<GMAX>(n, dp, oh, ol, ip, op, cfg, 0, st));
  }
  return JFG_OK;
}

int tc_status_take(int* status) {
  int zero = 0;
  JFG_CUDA_TRY(cudaMemcpyFromSymbol(status, g_tc_status, sizeof(int)));
  JFG_CUDA_TRY(cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int)));
  return JFG_OK;
}

}  // namespace jfg

extern "C" int jfg_contract_tc(const jfg_contract_desc* d, const float* op_hi,
                               const float* op_lo, const float* in, float* out, void* stream) {
  if (!d) return JFG_ERR_ARG;
  return jfg::contract_tc(*d, op_hi, op_lo, in, out, (cudaStream_t)stream);
}

extern "C" int jfg_contract_tc_bf16x3(const jfg_contract_desc* d, const uint16_t* op_hi,
                                      const uint16_t* op_lo, const float* in, float* out,
                                      void* stream) {
  if (!d) return JFG_ERR_ARG;
  return jfg::contract_tc_b16(*d, op_hi, op_lo, in, out, (cudaStream_t)stream);
}

extern "C" int jfg_contract_tc_f16x3(const jfg_contract_desc* d, const uint16_t* op_hi,
                                     const uint16_t* op_lo, const float* op_inv,
                                     long long op_inv_seg, const unsigned* in_max,
                                     unsigned* out_max, const float* in, float* out,
                                     void* stream) {
  if (!d) return JFG_ERR_ARG;
  return jfg::contract_tc_h16(*d, op_hi, op_lo, op_inv, op_inv_seg, in_max, out_max, in, out,
                              (cudaStream_t)stream);
}

extern "C" void jfg_split_bf16_host(size_t n, const double* src, uint16_t* hi, uint16_t* lo) {
  auto bits = [](float f) -> uint32_t {
    uint32_t u;
    memcpy(&u, &f, 4);
    if ((u & 0x7F800000u) == 0x7F800000u) return u >> 16;  // inf / nan: truncate
    return (u + 0x7FFFu + ((u >> 16) & 1u)) >> 16;         // round to nearest even
  };
  auto value = [](uint32_t b) -> float {
    const uint32_t u = b << 16;
    float f;
    memcpy(&f, &u, 4);
    return f;
  };
  for (size_t i = 0; i < n; ++i) {
    const uint32_t h = bits((float)src[i]);
    const uint32_t l = bits((float)(src[i] - (double)value(h)));
    hi[i] = (uint16_t)h;
    lo[i] = (uint16_t)l;
  }
}

extern "C" int jfg_tc_set_store_path(int tma_store) {
  return tma_store != 0 && tma_store != 1 ? JFG_ERR_ARG : JFG_OK;
}

extern "C" int jfg_tc_set_wait_budget_ns(unsigned long long ns) {
  const unsigned long long v = ns == 0 ? jfg::WAIT_NS_DEFAULT : ns;
  JFG_CUDA_TRY(cudaMemcpyToSymbol(jfg::g_tc_wait_ns, &v, sizeof(v)));
  return JFG_OK;
}

extern "C" int jfg_tc_test_hold(int on) {
  if (on != 0 && on != 1) return JFG_ERR_ARG;
  JFG_CUDA_TRY(cudaMemcpyToSymbol(jfg::g_tc_test_hold, &on, sizeof(on)));
  return JFG_OK;
}

extern "C" int jfg_tc_force_config(const jfg_tc_config* cfg) {
  std::lock_guard<std::mutex> lk(jfg::g_single_mu);
  jfg::g_force_on = cfg != nullptr;
  if (cfg) jfg::g_force_cfg = *cfg;
  return JFG_OK;
}

extern "C" int jfg_tc_set_autotune(int on) {
  if (on != 0 && on != 1) return JFG_ERR_ARG;
  jfg::set_single_autotune(on);
  return JFG_OK;
}

extern "C" int jfg_tc_tuned_count(void) {
  std::lock_guard<std::mutex> lk(jfg::g_single_mu);
  return (int)jfg::g_single.size();
}

extern "C" int jfg_tc_tuned_entry(int i, char* signature, size_t signature_len,
                                  jfg_tc_config* cfg, float* ms) {
  std::lock_guard<std::mutex> lk(jfg::g_single_mu);
  if (i < 0 || i >= (int)jfg::g_single.size()) return JFG_ERR_ARG;
  auto it = jfg::g_single.begin();
  std::advance(it, i);
  if (signature && signature_len > 0) snprintf(signature, signature_len, "%s", it->first.c_str());
  if (cfg) *cfg = it->second.cfg;
  if (ms) *ms = it->second.ms;
  return JFG_OK;
}

extern "C" int jfg_tc_set_op_resident(int on) {
  if (on < 0 || on > 2) return JFG_ERR_ARG;
  jfg::g_op_resident = on;
  return JFG_OK;
}

extern "C" int jfg_tc_set_variant(int operand_a_in_tmem) {
  if (operand_a_in_tmem != 0 && operand_a_in_tmem != 1) return JFG_ERR_ARG;
  jfg::g_operand_a_in_tmem = operand_a_in_tmem;
  return JFG_OK;
}

namespace {

// Tuned configurations by launch signature (shapes, batch, epilogue of every group).
std::mutex g_tune_mu;
std::map<std::string, jfg_tc_config> g_tuned;

std::string signature(int ng, const jfg_contract_desc* ds) {
  std::string key;
  char buf[160];
  int dev = 0;
  cudaGetDevice(&dev);
  snprintf(buf, sizeof buf, "d%d:", dev);
  key += buf;
  for (int i = 0; i < ng; ++i) {
    const jfg_contract_desc& d = ds[i];
    snprintf(buf, sizeof buf, "%d,%d,%d,%d,%d,%d,%d;", d.batch, d.nseg, d.M, d.P, d.K,
             d.epilogue, d.beta != 0.0 ? 1 : 0);
    key += buf;
  }
  return key;
}

}  // namespace

extern "C" int jfg_contract_tc_grouped(int ngroups, const jfg_contract_desc* descs,
                                       const float* const* op_hi, const float* const* op_lo,
                                       const float* const* in, float* const* out,
                                       const jfg_tc_config* cfg, void* stream) {
  if (ngroups < 0 || (ngroups > 0 && !descs)) return JFG_ERR_ARG;
  jfg_tc_config c = jfg::tc_default_config();
  if (cfg) {
    c = *cfg;
  } else {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tuned.find(signature(ngroups, descs));
    if (it != g_tuned.end()) c = it->second;
  }
  return jfg::contract_tc_grouped(ngroups, descs, op_hi, op_lo, in, out, c,
                                  (cudaStream_t)stream);
}

extern "C" int jfg_tc_autotune(int ngroups, const jfg_contract_desc* descs,
                               const float* const* op_hi, const float* const* op_lo,
                               const float* const* in, float* const* out, int reps,
                               jfg_tc_config* best, float* best_ms, void* stream) {
  if (ngroups < 1 || !descs || reps < 1) return JFG_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  JFG_CUDA_TRY(cudaStreamIsCapturing(st, &cap));
  if (cap != cudaStreamCaptureStatusNone) return JFG_ERR_ARG;  // timing needs real launches
  std::vector<jfg_tc_config> cands;
  const int orders = ngroups > 1 ? 3 : 1;
  for (int ta = 1; ta >= 0; --ta)
    for (int o = 0; o < orders; ++o)
      for (int sg : {0, 3, 2})
        for (int mt : {0, 64}) {
          jfg_tc_config c = jfg::tc_default_config();
          c.operand_a_in_tmem = ta;
          c.order = o;
          c.stages = sg;
          c.mtile = mt;
          cands.push_back(c);
        }
  cudaEvent_t e0, e1;
  JFG_CUDA_TRY(cudaEventCreate(&e0));
  JFG_CUDA_TRY(cudaEventCreate(&e1));
  float bt = -1.f;
  jfg_tc_config bc = cands[0];
  int status = JFG_OK;
  for (const jfg_tc_config& c : cands) {
    status = jfg::contract_tc_grouped(ngroups, descs, op_hi, op_lo, in, out, c, st);  // warm
    if (status != JFG_OK) break;
    if (cudaEventRecord(e0, st) != cudaSuccess) { status = JFG_ERR_CUDA; break; }
    for (int r = 0; r < reps && status == JFG_OK; ++r)
      status = jfg::contract_tc_grouped(ngroups, descs, op_hi, op_lo, in, out, c, st);
    if (status != JFG_OK) break;
    float ms = 0.f;
    if (cudaEventRecord(e1, st) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
        cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) {
      status = JFG_ERR_CUDA;
      break;
    }
    ms /= (float)reps;
    if (bt < 0.f || ms < bt) {
      bt = ms;
      bc = c;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (status != JFG_OK) return status;
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tuned[signature(ngroups, descs)] = bc;
  }
  if (best) *best = bc;
  if (best_ms) *best_ms = bt;
  return JFG_OK;
}

extern "C" int jfg_device_status(void) {
  int s = 0, g = 0, sl = 0;
  int r = jfg::tc_status_take(&s);
  if (r != JFG_OK) return r;
  r = jfg::gemm_status_take(&g);
  if (r != JFG_OK) return r;
  r = jfg::sl_status_take(&sl);
  if (r != JFG_OK) return r;
  return s != JFG_OK ? s : g != JFG_OK ? g : sl;
}

extern "C" void jfg_split_tf32_host(size_t n, const double* src, float* hi, float* lo) {
  for (size_t i = 0; i < n; ++i) {
    const float f = (float)src[i];
    uint32_t u;
    memcpy(&u, &f, 4);
    // round-to-nearest onto the TF32 grid (10 explicit mantissa bits)
    uint32_t r = (u + 0x1000u) & 0xFFFFE000u;
    float h;
    memcpy(&h, &r, 4);
    if (!(h == h) || (h - h != 0.0f)) h = f;  // keep inf/nan as is
    hi[i] = h;
    lo[i] = (float)(src[i] - (double)h);
  }
}
