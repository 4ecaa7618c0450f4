// FP64 per-axis contraction on the tensor cores by error-free slicing:
//
//   out[b][s][m][p] = alpha * epi(sum_k op[s][m][k] * in[b][s][p][k]) + beta * out
//
// with FP64 operands and FP64 results.  GB300 issues about 2 FP64 FMAs per
// clock per SM, so the CUDA-core contraction (contract_simt.cu) is bound by
// that pipe at ~1.24 TFLOP/s.  Here every operand row becomes a 63-bit
// fixed-point number per element (one power-of-two scale per row), cut into
// eight signed base-256 digits that FP16 holds exactly; products of digits are
// accumulated exactly by the tensor cores (kind::f16, FP32 accumulators that
// stay below 2^24 in magnitude), and the accumulators of equal weight are put
// together in integer arithmetic and rounded to FP64 once.  This is the
// error-free transformation of matrix products of Ozaki, Ogita, Oishi and
// Rump (Numerical Algorithms 59, 2012) in the form that Mukunoki, Ozaki,
// Ogita and Imamura (ISC 2020) gave it for tensor cores.
//
// Accuracy.  The operator's columns are first scaled by powers of two to a
// largest entry in [1, 2) and the input's columns by the inverse, so that a
// column of large entries against small coefficients (derivatives of spectral
// bases) does not cost digits.  An element then keeps 62 bits below its
// scaled row's largest one; the digit products left out are larger: 7 K of
// level 8, about sqrt(7 K) 2^-63.6 of the two rows' largest entries' product.
// So a sum is as accurate as by FMAs where the operator meets the input's
// largest entries with entries not far below its row's largest one, which
// k_sl_split judges by the operator.  Level d sums at most d + 1 digit pairs, each
// below 2^14 K: levels 0..3 cannot pass 2^24 for K <= 256 (0 and 1 for
// K <= 512; sums whose level 2 or 3 did are redone by FMAs), and the others
// could only lose their last bits, which weigh 2^-8d.  Rows with an infinity or a NaN (in the operator or the input) are
// summed by plain FP64 FMAs in the epilogue.
//
// Tile.  A CTA takes PT input rows (p) of one problem and segment, cuts them
// into digits and keeps all K of all eight digits in shared memory as the
// MMA's N operand: a block of PT zero rows, then PT rows per digit (K-major,
// 128-byte swizzle).  The operator's digits, cut once per call into a
// workspace, stream through TMA as the M operand (128 rows by 64 K of one
// digit, 16 KB).  Levels are accumulated in pairs (2h, 2h + 1), 2 PT columns
// of TMEM each: operator digit i meets input digits 2h - i and 2h + 1 - i,
// which are neighbouring blocks of the N operand (the zero block stands for
// digit -1), 20 MMAs of N = 2 PT per 16 K for 36 digit products.  Pairs are
// kept apart because only MMAs of one shape on one accumulator are ordered
// among themselves.  The MMAs of one operator digit share its tile through the
// collector buffer: 37 clocks per MMA of N = 64 against 48 when each reads the
// tile from shared memory (measured; 32 would be the tensor pipe's own).  Two
// accumulator sets of 8 PT columns (all 512 columns of TMEM for PT = 32) let
// the epilogue of one set run during the MMAs of the next, and with K <= 128
// two input tiles fit, so that cutting overlaps them too.  PT = 16 serves K in
// (256, 512] and launches too small to fill the chip with PT = 32.  When all
// operator digits fit in the stages (M <= 128, K <= 64) they are loaded once
// per CTA.
//
// The epilogue keeps FP64 instructions to the two that round a result: a warp
// instruction holds its scheduler's share of that pipe for 64 clocks.  alpha
// and beta are a template flag (LIN) for the same reason: as run-time
// conditions the product by alpha was computed and dropped.
//
// Warps: 0 TMA producer, 1 TMEM allocator and MMA issuer, 2-9 cut the input,
// 10-17 epilogue (two per TMEM lane quarter).  Every wait is bounded
// (tc_common.cuh); after a timeout the issued MMAs and loads are waited for
// before TMEM is freed, and jfg_device_status() reports it.
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>

#include "jfg_internal.cuh"
#include "tc_common.cuh"

namespace jfg {

__device__ int g_sl_status = 0;

namespace {

constexpr int NS = 8;             // digits
constexpr int NWS = 8;            // warps that cut the input
constexpr int NWE = 8;            // epilogue warps
constexpr int SL_NT = 64 + 32 * (NWS + NWE);
constexpr uint32_t ABYTES = 128 * 128;  // one operator stage: 128 rows x 64 FP16
constexpr int A_MAX = 8;          // operator stages
constexpr int STG_LD = 5;         // epilogue staging: 32 rows x 4 columns, padded
constexpr int RING = 8;           // input tiles whose row exponents are kept (a tile's are
                                  // read after its accumulators are handed back)
constexpr int COL_MAX = 3 * 512;  // column exponents (segments x K padded to 64)
constexpr int SPECIAL = 1 << 20;  // row exponent of a row with inf or NaN
// Sum of two row exponents from which a running FP64 sum of up to 512 products
// (each below 2^(sum - 2044)) could overflow; rows with specials are above it.
constexpr int BIG = 3068 - 10;
constexpr int NO_COLUMN = -3000;  // column exponent of an all-zero column
constexpr size_t SMEM_LIMIT = 227 * 1024;

struct SlLaunch {
  CUtensorMap amap;  // operator digits {K, M, segment x digit}
  jfg_contract_desc d;
  const double* op;
  const double* in;
  double* out;
  const int* row_e;      // [segments][M]
  const int16_t* col_e;  // [segments][kpad]
  const int* use;        // [segments] 0: FP64 FMAs instead of digits
  int ctas;              // CTAs that digits take; the others serve FMA sums alone
  int op_segs;           // segments of the operator (1: shared by all)
  int row_ld;            // row exponents per segment
  int kpad;              // K padded to 64
  int nkb;               // 64-element K blocks
  int bbuf;              // input tiles in shared memory
  int astages;
  int a_res;             // 1: every operator tile has its own stage, loaded once
  int vec2;              // input rows are 16-byte aligned
  int nptiles, mtiles;
};

// exponent field of x, at least 1 (subnormals), plus the column's exponent
__device__ __forceinline__ int elem_e(double x, int ce) {
  const int ex = (__double2hiint(x) >> 20) & 0x7FF;
  return (ex ? ex : 1) + ce;
}
__device__ __forceinline__ bool is_zero(double x) {
  return ((__double2hiint(x) & 0x7FFFFFFF) | __double2loint(x)) == 0;
}
__device__ __forceinline__ bool not_finite(double x) {
  return (__double2hiint(x) & 0x7FF00000) == 0x7FF00000;
}

// 16-bit integer e of eight packed in v
__device__ __forceinline__ int short_of(const uint4& v, int e) {
  const uint32_t w = e < 2 ? v.x : e < 4 ? v.y : e < 6 ? v.z : v.w;
  return (e & 1) ? (int)w >> 16 : (int)(w << 16) >> 16;
}

// The same with six bits of the mantissa below it; a row's exponent is row_e_of
// of the largest key: one more than the largest element's where its mantissa is
// within 2^-6 of 2.
__device__ __forceinline__ int elem_key(double x, int ce) {
  return max((__double2hiint(x) >> 14) & 0x1FFFF, 64) + 64 * ce;
}
constexpr int NO_KEY = -(1 << 25);  // a row of zeros
__device__ __forceinline__ int row_e_of(int key) { return (key + 1) >> 6; }
// x 2^(62 - E) truncated to an integer (|.| < 2^63 (1 - 2^-7), e = elem_e(x) <= E,
// E its row's exponent), plus 0x80 in every byte: byte 7 - j is then
// digit j + 128, and the sum has not passed 64 bits.
__device__ __forceinline__ unsigned long long biased_fixed(double x, int e, int E) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t mh = (hi & 0xFFFFFu) | ((hi & 0x7FF00000u) ? 0x100000u : 0u);
  const unsigned long long m = ((unsigned long long)mh << 32 | lo) << 10;
  const unsigned s = min((unsigned)(E - e), 63u);  // a zero with e > E wraps to 63
  const unsigned long long v = m >> s;
  const unsigned long long sg = (unsigned long long)((long long)((unsigned long long)hi << 32) >> 63);
  return (v ^ sg) - sg + 0x8080808080808080ull;
}

// digit j of eight consecutive elements as packed FP16: byte b - 128, formed
// as the FP16 number 1024 + b minus 1152 (both exact)
__device__ __forceinline__ uint32_t digit_pair(unsigned long long a, unsigned long long b, int j) {
  const uint32_t x = j < 4 ? (uint32_t)(a >> 32) : (uint32_t)a;
  const uint32_t y = j < 4 ? (uint32_t)(b >> 32) : (uint32_t)b;
  const uint32_t t = 3 - (j & 3);
  const uint32_t u = (__byte_perm(x, y, t | ((4 + t) << 8)) & 0x00FF00FFu) | 0x64006400u;
  const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&u), __floats2half2_rn(1152.f, 1152.f));
  return *reinterpret_cast<const uint32_t*>(&h);
}

// ---------------------------------------------------------------------------
// operator digits
// ---------------------------------------------------------------------------

constexpr int SPLIT_T = 512;
constexpr int SPLIT_CL = 8;
static_assert(SPLIT_T == SL_KMAX, "a thread per column");

struct SlSeg {
  const double* src;
  const double* lam;
  long long ld;
  int M, K, Kp, kpad;
  uint16_t* dig;  // [NS][M][Kp]
  int* row_e;
  int16_t* col_e;
  int* use;
  SlRule rule;
};
struct SlSplitArgs {
  SlSeg s[SL_MAX_SEGS];
};

// Whether digits keep what FP64 sums keep of every entry.  A digit sum is off by
// about sqrt(7 K) 2^-63.6 of (row's largest scaled entry) x (input row's largest),
// an FP64 sum by 2^-53 of the terms' magnitudes: the two compare when the
// operator meets the input's largest entries with entries of its own that are
// not far below their row's largest.  "Large" is an entry whose first digit is
// not zero: within 2^7 to 2^8 of it.
// SL_DENSE asks for large entries nearly everywhere (15/16 of all, 3/8 of every
// row and column: the transforms of the spaces have 0.98 or more and 0.49 or
// more, N = 24 to 256, both families), so that it does not matter which entries
// of the input are the largest.  Banded, triangular, diagonal and graded
// operators fall short of it: an identity on e^-k keeps nothing from k = 45 on.
// SL_FACTORS (eigenvector factors, the variable-coefficient operator) turns away
// the sparse ones alone (large entries: half of each factor is zero by parity,
// 0.335 or more are large for N = 17 to 400); those factors were measured entry
// by entry through the whole call instead.
__device__ __forceinline__ bool dense_enough(SlRule rule, long long large, long long rows,
                                             long long cols) {
  return rule == SL_DENSE ? 16 * large >= 15 * rows * cols : 32 * large >= 9 * rows * cols;
}
__device__ __forceinline__ bool line_dense(int large, int len) { return 8 * large >= 3 * len; }

// One cluster of 8 CTAs per operator segment: column maxima over each CTA's
// rows, combined through distributed shared memory; then one warp per row
// finds the row's exponent, writes its digits and counts its large entries, for
// *use: whether the contraction is to take the digits.  A few microseconds, bound
// by the latency of two reads of the rows (256 x 256: 4 rows per warp).
__global__ void __cluster_dims__(SPLIT_CL, 1, 1) __launch_bounds__(SPLIT_T)
    k_sl_split(const __grid_constant__ SlSplitArgs A) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ int cmax[512];
  __shared__ int16_t ce[512];
  // large entries of each column in this CTA's rows ([element][chunk], so that a
  // warp's adds lie in different banks) and, in rank 0, in all rows
  __shared__ int clarge[512], call[512];
  // columns that are not zero; rank 0: regular rows, their large entries, and
  // whether a row has too few
  __shared__ int cols, rows, large, thin;
  const SlSeg& q = A.s[blockIdx.x / SPLIT_CL];
  const int rank = (int)cl.block_rank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  cmax[threadIdx.x] = -1;
  clarge[threadIdx.x] = call[threadIdx.x] = 0;
  if (threadIdx.x == 0) cols = rows = large = thin = 0;
  __syncthreads();
  // as many threads as fit take rows of a column in turn
  const int kc = q.K <= 128 ? 128 : q.K <= 256 ? 256 : SPLIT_T, k1 = threadIdx.x % kc;
  if (k1 < q.K) {
    int mx = -1;
    for (int m = rank + SPLIT_CL * (threadIdx.x / kc); m < q.M; m += SPLIT_CL * (SPLIT_T / kc)) {
      const double x = q.src[(long long)m * q.ld + k1];
      if (!is_zero(x) && !not_finite(x)) mx = max(mx, elem_e(x, 0));
    }
    if (mx >= 0) atomicMax(&cmax[k1], mx);
  }
  cl.sync();
  if (const int k = threadIdx.x; k < q.kpad) {  // whole warps: kpad is a multiple of 64
    int c = 0;
    if (k < q.K) {
      int mx = -1;
#pragma unroll
      for (int r = 0; r < SPLIT_CL; ++r) mx = max(mx, cl.map_shared_rank(cmax, r)[k]);
      c = mx < 0 ? NO_COLUMN : mx - 1023;
      if (mx >= 0) {
        // half of the eigenvalue's exponent: the inputs fall off like its
        // inverse, so that it evens out both sides
        if (q.lam && !is_zero(q.lam[k]) && !not_finite(q.lam[k]))
          c += (elem_e(q.lam[k], 0) - 1023) >> 1;
      }
    }
    const unsigned any = __ballot_sync(0xffffffffu, c != NO_COLUMN && k < q.K);
    if (lane == 0) atomicAdd(&cols, __popc(any));
    ce[k] = (int16_t)c;
    if (rank == 0) q.col_e[k] = (int16_t)c;
  }
  cl.sync();  // also keeps cmax alive until every peer has read it
  const int ncol = cols;
  int cnt[2][8] = {}, nrow = 0, nlarge = 0;
  bool short_row = false;
  for (int m = rank + SPLIT_CL * warp; m < q.M; m += SPLIT_CL * (SPLIT_T / 32)) {
    const double* row = q.src + (long long)m * q.ld;
    int key = NO_KEY;
    bool bad = false;
    double x[2][8];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int k = 8 * (lane + 32 * i) + e;
        x[i][e] = k < q.K ? row[k] : 0.0;
        if (not_finite(x[i][e])) bad = true;
        // the column's exponent moves to the input: subtract it here
        else if (!is_zero(x[i][e])) key = max(key, elem_key(x[i][e], -(int)ce[k]));
      }
    int E = row_e_of(__reduce_max_sync(0xffffffffu, key));
    bad = __any_sync(0xffffffffu, bad);
    if (bad) E = SPECIAL;
    const bool regular = E > -(1 << 18) && !bad;
    if (lane == 0) q.row_e[m] = E < -(1 << 18) ? 0 : E;
    if (E < -(1 << 18)) E = 0;
    int n = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int k0 = 8 * (lane + 32 * i);
      if (k0 >= q.Kp) continue;
      unsigned long long f[8];
#pragma unroll
      for (int e = 0; e < 8; ++e)
        f[e] = biased_fixed(x[i][e], elem_e(x[i][e], k0 + e < q.K ? -(int)ce[k0 + e] : 0), E);
      if (regular) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int l = (uint32_t)(f[e] >> 56) != 0x80u;
          n += l;
          cnt[i][e] += l;
        }
      }
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        uint4 v;
        v.x = digit_pair(f[0], f[1], j);
        v.y = digit_pair(f[2], f[3], j);
        v.z = digit_pair(f[4], f[5], j);
        v.w = digit_pair(f[6], f[7], j);
        *reinterpret_cast<uint4*>(q.dig + ((long long)j * q.M + m) * q.Kp + k0) = v;
      }
    }
    if (regular) {
      n = __reduce_add_sync(0xffffffffu, n);
      ++nrow;
      nlarge += n;
      short_row = short_row || !line_dense(n, ncol);
    }
  }
  // all counts to rank 0, which judges
  if (q.rule == SL_DENSE) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (cnt[i][e]) atomicAdd(clarge + 64 * e + lane + 32 * i, cnt[i][e]);
    __syncthreads();
    const int c = clarge[threadIdx.x];
    if (c) atomicAdd(cl.map_shared_rank(call, 0) + threadIdx.x, c);
  }
  if (lane == 0) {
    atomicAdd(cl.map_shared_rank(&rows, 0), nrow);
    atomicAdd(cl.map_shared_rank(&large, 0), nlarge);
    if (short_row) atomicOr(cl.map_shared_rank(&thin, 0), 1);
  }
  cl.sync();
  if (rank == 0) {
    bool ok = dense_enough(q.rule, large, rows, ncol);
    if (q.rule == SL_DENSE) {
      const int k = threadIdx.x;
      ok = ok && !thin && (k >= q.K || ce[k] == NO_COLUMN ||
                           line_dense(call[64 * (k & 7) + (k >> 3)], rows));
      ok = __syncthreads_and(ok) != 0;
    }
    if (threadIdx.x == 0) *q.use = ok ? 1 : 0;
  }
}

// ---------------------------------------------------------------------------
// the contraction
// ---------------------------------------------------------------------------

// FP16 MMAs with the operand A use of the collector buffer (plain: read and
// dropped).  Issued by the lane with leader set, as one predicated instruction:
// the warp does not branch, so that descriptors (32-bit address words, the
// rest is constant) stay in uniform registers.
#define JFG_MMA_COLLECT(NAME, USAGE)                                                          \
  __device__ __forceinline__ void NAME(uint32_t d, uint32_t a, uint32_t b, uint32_t desc_hi,  \
                                       uint32_t idesc, uint32_t accum, uint32_t leader) {     \
    asm volatile(                                                                             \
        "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"                                       \
        "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"                                  \
        "setp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"                                  \
        "@q tcgen05.mma.cta_group::1.kind::f16" USAGE " [%0], da, db, %4, p;\n\t}" ::"r"(d),  \
        "r"(a), "r"(b), "r"(desc_hi), "r"(idesc), "r"(accum), "r"(leader));                   \
  }
JFG_MMA_COLLECT(mma_plain, "")
JFG_MMA_COLLECT(mma_fill, ".collector::a::fill")
JFG_MMA_COLLECT(mma_use, ".collector::a::use")
JFG_MMA_COLLECT(mma_lastuse, ".collector::a::lastuse")
#undef JFG_MMA_COLLECT
__device__ __forceinline__ void commit_if(uint64_t* bar, uint32_t leader) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(
          tc::smem_u32(bar)),
      "r"(leader)
      : "memory");
}

// The wait of a whole warp: one answer for all lanes, which are converged after
// it, as the aligned TMEM instructions and the issuers' uniform walk need.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity) {
  return __all_sync(0xffffffffu, tc::mbar_wait(bar, parity, &g_sl_status)) != 0;
}

__device__ __forceinline__ void tmem_ld4(uint32_t addr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
// wait for the loads into r[0..31] (the operands order the uses after it)
__device__ __forceinline__ void tmem_wait32(uint32_t* r) {
  asm volatile(
      "tcgen05.wait::ld.sync.aligned;"
      : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
        "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]),
        "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]),
        "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]),
        "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])::"memory");
}

__device__ __forceinline__ int level_int(uint32_t r) { return __float2int_rn(__uint_as_float(r)); }
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}
// four levels as one integer: ((a 2^8 + b) 2^8 + c) 2^8 + d
__device__ __forceinline__ long long level_join(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  return mad_wide(level_int(a), 1 << 24,
                  mad_wide(level_int(b), 1 << 16, mad_wide(level_int(c), 1 << 8, level_int(d))));
}

// A rare element of the epilogue, summed as it stands and in the CUDA-core
// path's order, so that it overflows, underflows and spreads specials the same
// way: one whose rows hold an infinity or a NaN, whose terms are large enough
// for a running sum to overflow, or whose exponent leaves the normal range.
__device__ __noinline__ double plain_sum(const double* a, const double* y, int K) {
  double v = 0.0;
  for (int k = 0; k < K; ++k) v = fma(a[k], y[k], v);
  return v;
}

// H + lo 2^-32 (integers below 2^51 in magnitude) rounded to nearest even as
// a double times 2^sh; rare is set when its exponent leaves the normal range.
// H and lo become doubles of 1.5 2^52 + H and + lo by one integer addition
// each; H - 1.5 2^20 is exact, and in the one fused multiply-add the offsets
// cancel.  The two FP64 instructions hold the scheduler's share of that pipe
// for 64 clocks each, but next to the MMAs it is idle: in integers (shifts,
// carries, leading zeros: some 60 instructions) 8 x 128^3 took 588 us, so 510.
__device__ __forceinline__ double level_value(long long H, long long lo, int sh, bool& rare) {
  const double h = __longlong_as_double(H + 0x4338000000000000ll);
  const double l = __longlong_as_double(lo + 0x4338000000000000ll);
  const double v = __fma_rn(__dadd_rn(h, -6755399442628608.0), 4294967296.0, l);
  const int hi = __double2hiint(v);
  const int ex = (hi >> 20) & 0x7FF;  // 0: the sum is zero
  rare = ex != 0 && (unsigned)(ex + sh - 33) >= 2046u;
  return __hiloint2double(ex ? hi + ((sh - 32) << 20) : 0, __double2loint(v));
}

// whether every operator segment of the launch is to be taken as digits
__device__ __forceinline__ bool use_digits(const SlLaunch& L) {
  int u = 1;
  for (int s = 0; s < L.op_segs; ++s) u &= __ldg(L.use + s);
  return u != 0;
}

// The whole launch by FP64 FMAs, for an operator whose digits would lose entries:
// tiles of 16 R operator rows by 32 R input rows over the CTAs, summed in the
// order of the CUDA-core contraction (the same bits).  Bound by the FP64 pipe:
// a thread reads 2 R values from shared memory per R^2 FMAs of 64 clocks.  R = 1
// unless there are many tiles of R = 2, for less idling in the last round.  The
// next 32 K are in registers while the present ones are multiplied.
constexpr int FMA_K = 32;
template <int EPI, int R>
__device__ __forceinline__ void fma_tiles_r(const SlLaunch& L, int nb, double* sm) {
  constexpr int TM = 16 * R, TP = 32 * R, T = 512;  // warps 0-15 multiply
  constexpr int LA = TM + 1, LB = TP + 1, NA = TM * FMA_K / T, NB = TP * FMA_K / T;
  const jfg_contract_desc& d = L.d;
  double* As = sm;                // [FMA_K][LA]
  double* Bs = sm + FMA_K * LA;   // [FMA_K][LB]
  const int t = threadIdx.x, tx = t & 31, ty = t >> 5, kk = t % FMA_K, r0 = t / FMA_K;
  const unsigned mt = (unsigned)((d.M + TM - 1) / TM), ptl = (unsigned)((d.P + TP - 1) / TP);
  const long long tiles = (long long)nb * d.nseg * ptl * mt;
  for (long long i = blockIdx.x; i < tiles; i += gridDim.x) {
    const int m0 = (int)(i % mt) * TM, p0 = (int)(i / mt % ptl) * TP;
    const int bs = (int)(i / ((long long)mt * ptl)), slot = bs / d.nseg, s = bs - slot * d.nseg;
    const int b = active_problem(d.batch_list, nb, d.batch, slot);
    if (b < 0) continue;  // the same for the whole CTA
    const double* a = L.op + (L.op_segs > 1 ? (long long)s * d.op_seg : 0);
    const double* y = L.in + (long long)b * d.in_batch + (long long)s * d.in_seg;
    double av[NA], bv[NB], acc[R][R] = {};
    auto load = [&](int k) {
#pragma unroll
      for (int j = 0; j < NA; ++j) {
        const int m = m0 + r0 + j * (T / FMA_K);
        av[j] = t < T && m < d.M && k < d.K ? __ldg(a + (long long)m * d.op_ld + k) : 0.0;
      }
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const int p = p0 + r0 + j * (T / FMA_K);
        bv[j] = t < T && p < d.P && k < d.K ? __ldg(y + (long long)p * d.in_ld + k) : 0.0;
      }
    };
    load(kk);
    for (int k0 = 0; k0 < d.K; k0 += FMA_K) {
      __syncthreads();
      if (t < T) {
#pragma unroll
        for (int j = 0; j < NA; ++j) As[kk * LA + r0 + j * (T / FMA_K)] = av[j];
#pragma unroll
        for (int j = 0; j < NB; ++j) Bs[kk * LB + r0 + j * (T / FMA_K)] = bv[j];
      }
      __syncthreads();
      if (k0 + FMA_K < d.K) load(k0 + FMA_K + kk);
      if (t < T) {
#pragma unroll 8
        for (int k = 0; k < FMA_K; ++k)
#pragma unroll
          for (int u = 0; u < R; ++u)
#pragma unroll
            for (int v = 0; v < R; ++v)
              acc[u][v] = fma(As[k * LA + ty + 16 * u], Bs[k * LB + tx + 32 * v], acc[u][v]);
      }
    }
    if (t >= T) continue;
    double c0 = 0.0, c1 = 1.0;
    if (EPI == JFG_EPI_DIV_EIG) {
      if (d.c0) c0 = ((const double*)d.c0)[b];
      if (d.c1) c1 = ((const double*)d.c1)[b];
    }
#pragma unroll
    for (int u = 0; u < R; ++u)
#pragma unroll
      for (int v = 0; v < R; ++v) {
        const int m = m0 + ty + 16 * u, p = p0 + tx + 32 * v;
        if (m >= d.M || p >= d.P) continue;
        double w = acc[u][v];
        if (EPI == JFG_EPI_MUL_FIELD)
          w *= ((const double*)d.field)[(long long)b * d.field_batch + (long long)s * d.field_seg +
                                        (long long)m * d.field_ld + p];
        else if (EPI == JFG_EPI_DIV_EIG)
          w = w / (c0 + c1 * (((const double*)d.lam_m)[m] + ((const double*)d.lam_p)[p]));
        double* o = L.out + (long long)b * d.out_batch + (long long)s * d.out_seg +
                    (long long)m * d.out_ld + p;
        w = d.alpha * w;
        if (d.beta != 0.0) w += d.beta * *o;
        *o = w;
      }
  }
}
template <int EPI>
__device__ __noinline__ void fma_tiles(const SlLaunch& L, int nb, double* sm) {
  const jfg_contract_desc& d = L.d;
  if ((long long)nb * d.nseg * ((d.M + 31) / 32) * ((d.P + 63) / 64) >= 8LL * gridDim.x)
    fma_tiles_r<EPI, 2>(L, nb, sm);
  else
    fma_tiles_r<EPI, 1>(L, nb, sm);
}
constexpr size_t FMA_SMEM = FMA_K * (33 + 65) * 8;

template <int EPI, bool LIN, int PT>
__global__ void __launch_bounds__(SL_NT, 1)
    k_contract_sl(const __grid_constant__ SlLaunch L) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_nb, s_dig;
  // aligned by an offset, so that accesses stay in the shared window for the
  // compiler (through an integer they become generic ones, which it must order
  // against the global stores)
  uint8_t* smem = smem_raw + ((0u - tc::smem_u32(smem_raw)) & 1023u);
  const jfg_contract_desc& d = L.d;
  constexpr uint32_t DBLK = (uint32_t)PT * 128;        // one digit of one K block
  constexpr uint32_t KBLK = (NS + 1) * DBLK;           // zero block and digits
  const uint32_t bbytes = (uint32_t)L.nkb * KBLK;
  uint8_t* bs = smem;                                   // [bbuf][nkb][1 + NS][PT][64]
  uint8_t* as = smem + (uint32_t)L.bbuf * bbytes;       // [astages]
  double* stg = (double*)(as + (uint32_t)L.astages * ABYTES);
  int* row_e = (int*)(stg + NWE * 32 * STG_LD);         // [RING][PT]
  int16_t* col_e = (int16_t*)(row_e + RING * PT);       // [op_segs][kpad]
  uint64_t* bars = (uint64_t*)(col_e + COL_MAX);
  uint64_t* afull = bars;
  uint64_t* aempty = bars + A_MAX;
  uint64_t* bfull = bars + 2 * A_MAX;
  uint64_t* bempty = bfull + 2;
  uint64_t* dfull = bfull + 4;
  uint64_t* dempty = bfull + 6;
  uint64_t* done = bfull + 8;
  uint32_t* tmem_slot = (uint32_t*)(bfull + 9);

  // warp-uniform to the compiler, so that the MMA issuer's addresses stay in
  // uniform registers
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  if (blockIdx.x >= (unsigned)L.ctas && use_digits(L)) return;
  if (threadIdx.x == 0) {
    s_nb = active_count(d.batch_list, d.batch_count, d.batch);
    for (int i = 0; i < A_MAX; ++i) {
      tc::mbar_init(&afull[i], 1);
      tc::mbar_init(&aempty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&bfull[i], NWS);
      tc::mbar_init(&bempty[i], 1);
      tc::mbar_init(&dfull[i], 1);
      tc::mbar_init(&dempty[i], NWE);
    }
    tc::mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = threadIdx.x; i < L.op_segs * L.kpad; i += SL_NT) col_e[i] = L.col_e[i];
  for (int i = threadIdx.x; i < L.bbuf * L.nkb * (int)(DBLK / 16); i += SL_NT)
    *reinterpret_cast<uint4*>(bs + (i / (DBLK / 16)) * KBLK + (i % (DBLK / 16)) * 16) =
        make_uint4(0, 0, 0, 0);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     tc::smem_u32(tmem_slot)),
                 "r"(2 * NS * PT)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  // items: (problem slot, segment, p tile), all operator tiles of each; with
  // fewer of these than CTAs, every operator tile is an item of its own
  const int nb = __shfl_sync(0xffffffffu, s_nb, 0);
  const unsigned base_items = (unsigned)nb * d.nseg * L.nptiles;
  const int msplit = (base_items < gridDim.x) ? L.mtiles : 1;
  const unsigned items = base_items * msplit;
  const int mt_n = msplit > 1 ? 1 : L.mtiles;
  auto decode = [&](unsigned t, int& mt0, int& pt, int& slot, int& s) {
    mt0 = 0;
    if (msplit > 1) {
      mt0 = (int)(t % (unsigned)msplit);
      t /= (unsigned)msplit;
    }
    pt = (int)(t % (unsigned)L.nptiles);
    t /= (unsigned)L.nptiles;
    slot = (int)(t / (unsigned)d.nseg);
    s = (int)t - slot * d.nseg;
  };

  // The digits are summed whether they are to be taken or not, so that nothing
  // waits for the verdict; results are stored only if they are.
  if (warp == 0) {
    // ---------------- operator producer ----------------
    if (lane == 0) {
      if (L.a_res) {
        for (int t = 0; t < L.mtiles * L.nkb * NS; ++t) {
          const int i = t % NS, kb = (t / NS) % L.nkb, mt = t / NS / L.nkb;
          tc::mbar_expect_tx(&afull[t], ABYTES);
          tc::tma_load_3d(as + t * ABYTES, &L.amap, &afull[t], kb * 64, mt * 128, i);
        }
        for (int t = 0; t < L.mtiles * L.nkb * NS; ++t) tc::mbar_wait(&afull[t], 0, &g_sl_status);
      } else {
        int st = 0;
        uint32_t ph = 0;
        long long issued = 0;
        bool ok = true;
        for (unsigned t = blockIdx.x; ok && t < items; t += gridDim.x) {
          int mt0, pt, slot, s;
          decode(t, mt0, pt, slot, s);
          const int os = L.op_segs > 1 ? s : 0;
          for (int mt = mt0; ok && mt < mt0 + mt_n; ++mt)
            for (int kb = 0; ok && kb < L.nkb; ++kb)
              for (int i = 0; i < NS; ++i) {
                if (issued >= L.astages && !tc::mbar_wait(&aempty[st], ph ^ 1u, &g_sl_status)) {
                  ok = false;
                  break;
                }
                tc::mbar_expect_tx(&afull[st], ABYTES);
                tc::tma_load_3d(as + st * ABYTES, &L.amap, &afull[st], kb * 64, mt * 128,
                                os * NS + i);
                ++issued;
                if (++st == L.astages) {
                  st = 0;
                  ph ^= 1u;
                }
              }
        }
        // the last use of every stage must have landed before exit
        for (long long q = issued > L.astages ? issued - L.astages : 0; q < issued; ++q)
          tc::mbar_wait(&afull[q % L.astages], (uint32_t)(q / L.astages) & 1u, &g_sl_status);
      }
      s_dig = use_digits(L) ? 1 : 0;
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // The whole warp walks the loop, one elected lane issues.  Every branch is
    // on a warp-uniform value (waits through a vote): otherwise the addresses
    // leave the uniform registers and an MMA costs 64 clocks instead of 40 (4 x
    // 256^3 round: 4.34 ms then, 3.56 ms so; 32 x 256^2: 139 and 122 us).
    const uint32_t ad0 = (uint32_t)tc::sdesc_sw128(tc::smem_u32(as));
    const uint32_t bd0 = (uint32_t)tc::sdesc_sw128(tc::smem_u32(bs));
    const uint32_t dhi = (uint32_t)(tc::sdesc_sw128(0) >> 32);
    const uint32_t leader = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc =  // FP16 x FP16 -> FP32, M = 128, N = 2 PT
        (1u << 4) | ((uint32_t)(2 * PT) >> 3 << 17) | ((128u >> 4) << 24);
    int st = 0, bslot = 0;
    uint32_t aph = 0, bph = 0, unit = 0;
    bool ok = true, any = false;
    for (unsigned t = blockIdx.x; ok && t < items; t += gridDim.x) {
      if (!warp_wait(&bfull[bslot], bph)) {
        ok = false;
        break;
      }
      const uint32_t bdt = bd0 + (((uint32_t)bslot * bbytes) >> 4);
      for (int mi = 0; ok && mi < mt_n; ++mi, ++unit) {
        const uint32_t db = unit & 1u;
        if (unit >= 2 && !warp_wait(&dempty[db], ((unit >> 1) & 1u) ^ 1u)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem + db * (NS * PT);
        if (L.a_res) st = mi * L.nkb * NS;
        for (int kb = 0; ok && kb < L.nkb; ++kb) {
          const int rest = d.K - kb * 64;
          const int n16 = rest >= 64 ? 4 : (rest + 15) / 16;
          const uint32_t bdk = bdt + (((uint32_t)kb * KBLK) >> 4);
#pragma unroll
          for (int i = 0; i < NS; ++i) {
            if (!warp_wait(&afull[st], aph)) {
              ok = false;
              break;
            }
            any = true;
            const uint32_t ad = ad0 + (((uint32_t)st * ABYTES) >> 4);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              if (kk >= n16) break;
              const uint32_t more = (kb | kk | i) ? 1u : 0u;
              // pairs h = i / 2 .. 3 share the operator tile: it stays in the
              // collector buffer from the first to the last
#pragma unroll
              for (int h = 3; h >= i / 2; --h) {
                const uint32_t bd = bdk + (((uint32_t)(2 * h - i + 1) * DBLK + 32 * kk) >> 4);
                const uint32_t D = acc + 2 * PT * h;
                if (h == 3 && h == i / 2)
                  mma_plain(D, ad + 2 * kk, bd, dhi, idesc, more, leader);
                else if (h == 3)
                  mma_fill(D, ad + 2 * kk, bd, dhi, idesc, more, leader);
                else if (h == i / 2)
                  mma_lastuse(D, ad + 2 * kk, bd, dhi, idesc, more, leader);
                else
                  mma_use(D, ad + 2 * kk, bd, dhi, idesc, more, leader);
              }
            }
            if (!L.a_res) commit_if(&aempty[st], leader);
            if (++st == L.astages) {
              st = 0;
              if (!L.a_res) aph ^= 1u;
            }
          }
        }
        if (ok) commit_if(&dfull[db], leader);
      }
      if (ok) commit_if(&bempty[bslot], leader);
      if (++bslot == L.bbuf) {
        bslot = 0;
        bph ^= 1u;
      }
    }
    if (any) {  // every MMA has finished before TMEM is freed
      commit_if(done, leader);
      tc::mbar_wait(done, 0, &g_sl_status);
    }
  } else if (warp < 2 + NWS) {
    // ---------------- cut the input rows into digits ----------------
    constexpr int RW = PT / NWS;  // rows per warp
    constexpr int UPR = 32 / RW;  // lanes per row, one chunk of 8 elements each per step
    constexpr int STEPS = 4;      // chunks per lane: 8 UPR STEPS elements = 256 (PT 32) or 512
    const int row = (warp - 2) * RW + lane % RW;
    const int u = lane / RW;
    // chunk of this lane within a step, so that the eight lanes of a
    // quarter-warp store to different 16-byte columns of the swizzled rows
    const int cu = PT == 32 ? ((u >> 1) | ((u & 1) << 2))
                            : (((u & 3) << 1) | ((u >> 2) & 1) | (u & 8));
    const int steps = (L.kpad + 8 * UPR - 1) / (8 * UPR);  // with any elements
    double x[STEPS][8];
    auto load = [&](unsigned t) {
      int mt0, pt, slot, s;
      decode(t, mt0, pt, slot, s);
      const int b = active_problem(d.batch_list, nb, d.batch, slot);
      const int p = pt * PT + row;
      const double* src = L.in + (long long)(b < 0 ? 0 : b) * d.in_batch +
                          (long long)s * d.in_seg + (long long)p * d.in_ld;
      const bool live = b >= 0 && p < d.P;
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        if (i >= steps) break;
        const int k0 = 8 * (cu + UPR * i);
        if (live && k0 + 8 <= d.K) {
          if (L.vec2) {
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
              const double2 v = __ldg((const double2*)(src + k0 + e));
              x[i][e] = v.x;
              x[i][e + 1] = v.y;
            }
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[i][e] = __ldg(src + k0 + e);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e)
            x[i][e] = live && k0 + e < d.K ? __ldg(src + k0 + e) : 0.0;
        }
      }
      return s;
    };
    int bslot = 0, ring = 0;
    uint32_t bph = 0;
    unsigned n = 0;
    int s = 0;
    if (blockIdx.x < items) s = load(blockIdx.x);
    for (unsigned t = blockIdx.x; t < items; t += gridDim.x, ++n) {
      const int16_t* ce = col_e + (L.op_segs > 1 ? s : 0) * L.kpad;
      int key = NO_KEY;
      bool bad = false;
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        if (i >= steps) break;
        const int k0 = 8 * (cu + UPR * i);
        if (k0 < L.kpad) {
          const uint4 c = *reinterpret_cast<const uint4*>(ce + k0);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            bad = bad || not_finite(x[i][e]);
            if (!is_zero(x[i][e])) key = max(key, elem_key(x[i][e], short_of(c, e)));
          }
        }
      }
#pragma unroll
      for (int o = RW; o < 32; o <<= 1) {
        key = max(key, __shfl_xor_sync(0xffffffffu, key, o));
        bad = __shfl_xor_sync(0xffffffffu, (int)bad, o) || bad;
      }
      int E = row_e_of(key);
      if (E < -(1 << 18)) E = 0;
      if (bad) E = SPECIAL;
      if (n >= (unsigned)L.bbuf && !warp_wait(&bempty[bslot], bph ^ 1u)) break;
      if (u == 0) row_e[ring * PT + row] = E;
      uint8_t* dst = bs + (uint32_t)bslot * bbytes + DBLK + row * 128;
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        if (i >= steps) break;
        const int q = cu + UPR * i, k0 = 8 * q;
        if (k0 < L.kpad) {
          const uint4 c = *reinterpret_cast<const uint4*>(ce + k0);
          unsigned long long f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = biased_fixed(x[i][e], elem_e(x[i][e], short_of(c, e)), E);
          uint8_t* o = dst + (uint32_t)(q >> 3) * KBLK + (((q & 7) ^ (row & 7)) << 4);
#pragma unroll
          for (int j = 0; j < NS; ++j) {
            uint4 v;
            v.x = digit_pair(f[0], f[1], j);
            v.y = digit_pair(f[2], f[3], j);
            v.z = digit_pair(f[4], f[5], j);
            v.w = digit_pair(f[6], f[7], j);
            *reinterpret_cast<uint4*>(o + j * DBLK) = v;
          }
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bfull[bslot]);
      if (t + gridDim.x < items) s = load(t + gridDim.x);
      ring = (ring + 1) & (RING - 1);
      if (++bslot == L.bbuf) {
        bslot = 0;
        bph ^= 1u;
      }
    }
  } else {
    // ---------------- epilogue ----------------
    const int ew = warp - 2 - NWS;
    const int quarter = warp & 3, half = ew >> 2;
    double* st4 = stg + ew * 32 * STG_LD;
    const int sr = lane >> 2, sc = lane & 3;
    const bool take = use_digits(L);
    int ring = 0;
    uint32_t unit = 0;
    bool ok = true;
    for (unsigned t = blockIdx.x; ok && t < items; t += gridDim.x) {
      int mt0, pt, slot, s;
      decode(t, mt0, pt, slot, s);
      const int b = take ? active_problem(d.batch_list, nb, d.batch, slot) : -1;
      const int os = L.op_segs > 1 ? s : 0;
      const long long ib = (long long)(b < 0 ? 0 : b) * d.in_batch + (long long)s * d.in_seg;
      double* outS = L.out + (long long)(b < 0 ? 0 : b) * d.out_batch + (long long)s * d.out_seg;
      double c0 = 0.0, c1 = 1.0;
      if (EPI == JFG_EPI_DIV_EIG && b >= 0) {
        if (d.c0) c0 = ((const double*)d.c0)[b];
        if (d.c1) c1 = ((const double*)d.c1)[b];
      }
      for (int mt = mt0; mt < mt0 + mt_n; ++mt, ++unit) {
        const int m0 = mt * 128 + 32 * quarter;
        const int m = m0 + lane;
        const int Ea = m < d.M ? __ldg(L.row_e + (long long)os * L.row_ld + m) : 0;
        const uint32_t db = unit & 1u;
        if (!warp_wait(&dfull[db], (unit >> 1) & 1u)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem + db * (NS * PT) + ((uint32_t)(32 * quarter) << 16);
        if (m0 >= d.M) {  // no row of this quarter
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&dempty[db]);
          continue;
        }
        // four columns of all levels at a time, staged for stores of 32 bytes a row
#pragma unroll 1
        for (int g = 0; g < PT / 8; ++g) {
          const int col4 = half * (PT / 2) + 4 * g;
          uint32_t r[32];
#pragma unroll
          for (int j = 0; j < NS; ++j) tmem_ld4(acc + j * PT + col4, r + 4 * j);
          tmem_wait32(r);
          if (g == PT / 8 - 1) {  // the accumulators are read: the next tile may have them
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&dempty[db]);
          }
          const int4 E4 = *reinterpret_cast<const int4*>(row_e + ring * PT + col4);
          const int Ep[4] = {E4.x, E4.y, E4.z, E4.w};
          double* cell = st4 + lane * STG_LD;
          unsigned rare = 0;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            bool x;
            cell[c] = level_value(level_join(r[c], r[4 + c], r[8 + c], r[12 + c]),
                                  level_join(r[16 + c], r[20 + c], r[24 + c], r[28 + c]),
                                  Ea + Ep[c] - 2082, x);
            rare |= (x || Ea + Ep[c] >= BIG) ? 1u << c : 0u;
            // K > 256 (PT 16): levels 2 and 3 may have lost bits past 2^24
            if (PT == 16 && L.nkb > 4 && fmaxf(fabsf(__uint_as_float(r[8 + c])),
                                  fabsf(__uint_as_float(r[12 + c]))) >= 16777216.f)
              rare |= 1u << c;
          }
          if (rare && m < d.M && b >= 0) {
            const double* a = L.op + (long long)os * d.op_seg + (long long)m * d.op_ld;
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              const int p = pt * PT + col4 + c;
              if ((rare >> c & 1u) && p < d.P)
                cell[c] = plain_sum(a, L.in + ib + (long long)p * d.in_ld, d.K);
            }
          }
          __syncwarp();
          const int p = pt * PT + col4 + sc;
          if (p < d.P && b >= 0) {
            const double lp = EPI == JFG_EPI_DIV_EIG ? __ldg((const double*)d.lam_p + p) : 0.0;
            double* o = outS + (long long)(m0 + sr) * d.out_ld + p;
            const double* f = (const double*)d.field + (long long)b * d.field_batch +
                              (long long)s * d.field_seg + (long long)(m0 + sr) * d.field_ld + p;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int mm = m0 + 8 * i + sr;
              if (mm < d.M) {
                double v = st4[(8 * i + sr) * STG_LD + sc];
                if (EPI == JFG_EPI_MUL_FIELD)
                  v *= __ldg(f);
                else if (EPI == JFG_EPI_DIV_EIG)
                  v = v / (c0 + c1 * (__ldg((const double*)d.lam_m + mm) + lp));
                if (LIN) {
                  v *= d.alpha;
                  if (d.beta != 0.0) v += d.beta * *o;
                }
                *o = v;
              }
              o += 8 * d.out_ld;
              if (EPI == JFG_EPI_MUL_FIELD) f += 8 * d.field_ld;
            }
          }
          __syncwarp();
        }
      }
      ring = (ring + 1) & (RING - 1);
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (!s_dig) fma_tiles<EPI>(L, nb, (double*)smem);  // every copy has landed
  __syncwarp();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(2 * NS * PT));
  }
}

// ---------------------------------------------------------------------------
// the contraction for small operators (M <= 64, K <= 64, shared by all rows)
// ---------------------------------------------------------------------------

// The roles of the operands are swapped: 128 input rows, flattened over the
// problems so that short ones leave no tile part empty, are the MMA's M
// operand, and the operator's digits (in two halves of 32 rows) its resident N
// operand.  Above, an operator of 64 rows fills half of the MMA's M, and half
// of the TMEM lanes and with them the epilogue of two of the four schedulers:
// 1024 problems of 64 x 62 spent 11.1k clocks per 32 rows, 8k of them in the
// epilogue.  Lanes are input rows here, so results go straight to memory,
// coalesced, without staging.  Two passes: 1024 x 64 x 62 167 -> 105 us, 3000 x
// 51 x 49 465 -> 176, 3000 x 33 x 31 334 -> 103.
//
// One input tile fits (eight digits of 128 rows, 128 KB), so cutting a tile
// waits for the MMAs of the one before; the epilogue of either half overlaps
// both (two accumulator sets of 256 columns).
constexpr int RT = 128;                            // input rows of a tile
constexpr int RM = 32;                             // operator rows of a unit
constexpr uint32_t RBLK = RM * 128;                // one digit of one unit
constexpr uint32_t RUNIT = (NS + 1) * RBLK;        // zero block and digits
constexpr size_t ROWS_SMEM = 1024 + NS * ABYTES + 2 * RUNIT + RING * RT * 4 + 64 * 4 + 16 * 8;

template <int EPI, bool LIN>
__global__ void __launch_bounds__(SL_NT, 1)
    k_contract_sl_rows(const __grid_constant__ SlLaunch L) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_nb, s_dig;
  uint8_t* smem = smem_raw + ((0u - tc::smem_u32(smem_raw)) & 1023u);
  const jfg_contract_desc& d = L.d;
  uint8_t* as = smem;                                 // [NS][RT][64]
  uint8_t* bs = as + NS * ABYTES;                     // [2][1 + NS][RM][64]
  int* row_e = (int*)(bs + 2 * RUNIT);                // [RING][RT]
  int* op_e = row_e + RING * RT;                      // [64]
  uint64_t* bars = (uint64_t*)(op_e + 64);
  uint64_t* ofull = bars;
  uint64_t* bfull = bars + 1;
  uint64_t* bempty = bars + 2;
  uint64_t* done = bars + 3;
  uint64_t* dfull = bars + 4;
  uint64_t* dempty = bars + 6;
  uint32_t* tmem_slot = (uint32_t*)(bars + 8);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int units = (d.M + RM - 1) / RM;  // 1 or 2
  if (blockIdx.x >= (unsigned)L.ctas && use_digits(L)) return;
  if (threadIdx.x == 0) {
    s_nb = active_count(d.batch_list, d.batch_count, d.batch);
    tc::mbar_init(ofull, 1);
    tc::mbar_init(bfull, NWS);
    tc::mbar_init(bempty, 1);
    tc::mbar_init(done, 1);
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&dfull[i], 1);
      tc::mbar_init(&dempty[i], NWE);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc::mbar_expect_tx(ofull, (uint32_t)units * NS * RBLK);
    for (int v = 0; v < units; ++v)
      for (int i = 0; i < NS; ++i)
        tc::tma_load_3d(bs + v * RUNIT + (i + 1) * RBLK, &L.amap, ofull, 0, v * RM, i);
  }
  if (threadIdx.x < 64) op_e[threadIdx.x] = (int)threadIdx.x < d.M ? __ldg(L.row_e + threadIdx.x) : 0;
  for (int i = threadIdx.x; i < 2 * (int)(RBLK / 16); i += SL_NT)
    *reinterpret_cast<uint4*>(bs + (i / (RBLK / 16)) * RUNIT + (i % (RBLK / 16)) * 16) =
        make_uint4(0, 0, 0, 0);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     tc::smem_u32(tmem_slot)),
                 "r"(2 * NS * RM)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  // items: (segment, tile of RT flattened rows)
  const int nb = __shfl_sync(0xffffffffu, s_nb, 0);
  const unsigned R = (unsigned)nb * (unsigned)d.P;
  const unsigned per_seg = (R + RT - 1) / RT;
  const unsigned items = per_seg * (unsigned)d.nseg;
  // row of an item: segment, problem slot and p
  auto locate = [&](unsigned t, int row, int& s, unsigned& slot, unsigned& p) {
    s = d.nseg > 1 ? (int)(t / per_seg) : 0;
    const unsigned r = (t - (unsigned)s * per_seg) * RT + (unsigned)row;
    slot = r / (unsigned)d.P;
    p = r - slot * (unsigned)d.P;
  };
  auto problem = [&](unsigned slot) {  // -1: past the last
    return active_problem(d.batch_list, nb, d.batch, (int)slot);
  };

  if (warp == 0) {
    // the operator has landed before the CTA may end
    if (lane == 0) {
      tc::mbar_wait(ofull, 0, &g_sl_status);
      s_dig = use_digits(L) ? 1 : 0;
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (uniform walk as above) ----------------
    const uint32_t ad0 = (uint32_t)tc::sdesc_sw128(tc::smem_u32(as));
    const uint32_t bd0 = (uint32_t)tc::sdesc_sw128(tc::smem_u32(bs));
    const uint32_t dhi = (uint32_t)(tc::sdesc_sw128(0) >> 32);
    const uint32_t leader = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc =  // FP16 x FP16 -> FP32, M = 128, N = 2 RM
        (1u << 4) | ((uint32_t)(2 * RM) >> 3 << 17) | ((128u >> 4) << 24);
    const int n16 = (d.K + 15) / 16;
    uint32_t unit = 0, ph = 0;
    bool any = false;
    bool ok = blockIdx.x >= items || warp_wait(ofull, 0);
    for (unsigned t = blockIdx.x; ok && t < items; t += gridDim.x, ph ^= 1u) {
      if (!warp_wait(bfull, ph)) break;
      for (int v = 0; v < units; ++v, ++unit) {
        const uint32_t db = unit & 1u;
        if (unit >= 2 && !warp_wait(&dempty[db], ((unit >> 1) & 1u) ^ 1u)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        any = true;
        const uint32_t acc = tmem + db * (NS * RM);
        const uint32_t bdv = bd0 + (((uint32_t)v * RUNIT) >> 4);
#pragma unroll
        for (int i = 0; i < NS; ++i) {
          const uint32_t ad = ad0 + (((uint32_t)i * ABYTES) >> 4);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            if (kk >= n16) break;
            const uint32_t more = (kk | i) ? 1u : 0u;
#pragma unroll
            for (int h = 3; h >= i / 2; --h) {
              const uint32_t bd = bdv + (((uint32_t)(2 * h - i + 1) * RBLK + 32 * kk) >> 4);
              const uint32_t D = acc + 2 * RM * h;
              if (h == 3 && h == i / 2)
                mma_plain(D, ad + 2 * kk, bd, dhi, idesc, more, leader);
              else if (h == 3)
                mma_fill(D, ad + 2 * kk, bd, dhi, idesc, more, leader);
              else if (h == i / 2)
                mma_lastuse(D, ad + 2 * kk, bd, dhi, idesc, more, leader);
              else
                mma_use(D, ad + 2 * kk, bd, dhi, idesc, more, leader);
            }
          }
        }
        commit_if(&dfull[db], leader);
      }
      if (ok) commit_if(bempty, leader);
    }
    if (any) {  // every MMA has finished before TMEM is freed
      commit_if(done, leader);
      tc::mbar_wait(done, 0, &g_sl_status);
    }
  } else if (warp < 2 + NWS) {
    // ---------------- cut the input rows into digits ----------------
    // a lane takes 8 consecutive elements of four rows 32 apart; the chunk
    // order lets a quarter-warp store to different 16-byte columns
    const int u = lane >> 2;
    const int cu = (u >> 1) | ((u & 1) << 2);
    const int k0 = 8 * cu;
    const int row0 = 4 * (warp - 2) + (lane & 3);
    const uint4 ce = __ldg((const uint4*)(L.col_e + k0));
    uint8_t* dst = as + row0 * 128 + ((cu ^ (row0 & 7)) << 4);
    const unsigned q32 = 32u / (unsigned)d.P, r32 = 32u - q32 * (unsigned)d.P;  // 32 rows on
    double x[4][8];
    auto load = [&](unsigned t) {
      int s;
      unsigned slot, p;
      locate(t, row0, s, slot, p);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int b = problem(slot);
        const double* src = L.in + (long long)(b < 0 ? 0 : b) * d.in_batch +
                            (long long)s * d.in_seg + (long long)p * d.in_ld + k0;
        if (b >= 0 && k0 + 8 <= d.K) {
          if (L.vec2) {
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
              const double2 v = __ldg((const double2*)(src + e));
              x[i][e] = v.x;
              x[i][e + 1] = v.y;
            }
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[i][e] = __ldg(src + e);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) x[i][e] = b >= 0 && k0 + e < d.K ? __ldg(src + e) : 0.0;
        }
        slot += q32;
        p += r32;
        if (p >= (unsigned)d.P) {
          p -= (unsigned)d.P;
          ++slot;
        }
      }
    };
    uint32_t n = 0;
    if (blockIdx.x < items) load(blockIdx.x);
    for (unsigned t = blockIdx.x; t < items; t += gridDim.x, ++n) {
      int E[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        E[i] = NO_KEY;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int v = not_finite(x[i][e]) ? 64 * SPECIAL : elem_key(x[i][e], short_of(ce, e));
          if (!is_zero(x[i][e])) E[i] = max(E[i], v);
        }
      }
#pragma unroll
      for (int o = 4; o < 32; o <<= 1)
#pragma unroll
        for (int i = 0; i < 4; ++i) E[i] = max(E[i], __shfl_xor_sync(0xffffffffu, E[i], o));
      if (n >= 1 && !warp_wait(bempty, (n & 1u) ^ 1u)) break;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        E[i] = row_e_of(E[i]);
        if (E[i] < -(1 << 18)) E[i] = 0;
        if (u == 0) row_e[(n & (RING - 1)) * RT + 32 * i + row0] = E[i];
        unsigned long long f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
          f[e] = biased_fixed(x[i][e], elem_e(x[i][e], short_of(ce, e)), E[i]);
#pragma unroll
        for (int j = 0; j < NS; ++j) {
          uint4 v;
          v.x = digit_pair(f[0], f[1], j);
          v.y = digit_pair(f[2], f[3], j);
          v.z = digit_pair(f[4], f[5], j);
          v.w = digit_pair(f[6], f[7], j);
          *reinterpret_cast<uint4*>(dst + i * (32 * 128) + j * ABYTES) = v;
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bfull);
      if (t + gridDim.x < items) load(t + gridDim.x);
    }
  } else {
    // ---------------- epilogue: a lane is an input row ----------------
    const int quarter = warp & 3, half = (warp - 2 - NWS) >> 2;
    const int row = 32 * quarter + lane;
    const bool take = use_digits(L);
    uint32_t unit = 0, n = 0;
    bool ok = true;
    for (unsigned t = blockIdx.x; ok && t < items; t += gridDim.x, ++n) {
      int s;
      unsigned slot, up;
      locate(t, row, s, slot, up);
      const int b = take ? problem(slot) : -1, p = (int)up;
      const long long ib = (long long)(b < 0 ? 0 : b);
      double* outP = L.out + ib * d.out_batch + (long long)s * d.out_seg + p;
      const double* f = (const double*)d.field + ib * d.field_batch + (long long)s * d.field_seg + p;
      double c0 = 0.0, c1 = 1.0, lp = 0.0;
      if (EPI == JFG_EPI_DIV_EIG && b >= 0) {
        if (d.c0) c0 = ((const double*)d.c0)[b];
        if (d.c1) c1 = ((const double*)d.c1)[b];
        lp = __ldg((const double*)d.lam_p + p);
      }
      int Ep = 0;
      for (int v = 0; v < units; ++v, ++unit) {
        const uint32_t db = unit & 1u;
        if (!warp_wait(&dfull[db], (unit >> 1) & 1u)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // read before any accumulator of the tile is handed back: the ring
        // may be written again three tiles on
        if (v == 0) Ep = row_e[(n & (RING - 1)) * RT + row];
        const uint32_t acc = tmem + db * (NS * RM) + ((uint32_t)(32 * quarter) << 16);
        const int col0 = half * (RM / 2);
        const int live = min(RM / 2, d.M - v * RM - col0);  // columns with an operator row
        const int steps = live > 0 ? (live + 3) / 4 : 0;
        if (steps == 0) {
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&dempty[db]);
        }
#pragma unroll 1
        for (int g = 0; g < steps; ++g) {
          const int col4 = col0 + 4 * g, m = v * RM + col4;
          uint32_t r[32];
#pragma unroll
          for (int j = 0; j < NS; ++j) tmem_ld4(acc + j * RM + col4, r + 4 * j);
          tmem_wait32(r);
          if (g == steps - 1) {  // the accumulators are read: the next unit may have them
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&dempty[db]);
          }
          const int4 A4 = *reinterpret_cast<const int4*>(op_e + m);
          const int Ea[4] = {A4.x, A4.y, A4.z, A4.w};
          double val[4];
          unsigned rare = 0;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            bool xr;
            val[c] = level_value(level_join(r[c], r[4 + c], r[8 + c], r[12 + c]),
                                 level_join(r[16 + c], r[20 + c], r[24 + c], r[28 + c]),
                                 Ea[c] + Ep - 2082, xr);
            rare |= (xr || Ea[c] + Ep >= BIG) ? 1u << c : 0u;
          }
          if (b >= 0) {
            if (rare) {
              const double* y =
                  L.in + ib * d.in_batch + (long long)s * d.in_seg + (long long)p * d.in_ld;
#pragma unroll
              for (int c = 0; c < 4; ++c)
                if ((rare >> c & 1u) && m + c < d.M)
                  val[c] = plain_sum(L.op + (long long)(m + c) * d.op_ld, y, d.K);
            }
            double* o = outP + (long long)m * d.out_ld;
            const double* fm = f + (long long)m * d.field_ld;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              if (m + c < d.M) {
                double w = val[c];
                if (EPI == JFG_EPI_MUL_FIELD)
                  w *= __ldg(fm);
                else if (EPI == JFG_EPI_DIV_EIG)
                  w = w / (c0 + c1 * (__ldg((const double*)d.lam_m + m + c) + lp));
                if (LIN) {
                  w *= d.alpha;
                  if (d.beta != 0.0) w += d.beta * *o;
                }
                *o = w;
              }
              o += d.out_ld;
              if (EPI == JFG_EPI_MUL_FIELD) fm += d.field_ld;
            }
          }
          __syncwarp();  // the next step's TMEM loads take the whole warp
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (!s_dig) fma_tiles<EPI>(L, nb, (double*)smem);  // every copy has landed
  __syncwarp();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(2 * NS * RM));
  }
}

template <int EPI, bool LIN>
int set_attr() {
  JFG_CUDA_TRY(cudaFuncSetAttribute(k_contract_sl_rows<EPI, LIN>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)ROWS_SMEM));
  JFG_CUDA_TRY(cudaFuncSetAttribute(k_contract_sl<EPI, LIN, 32>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)SMEM_LIMIT - 1024));
  JFG_CUDA_TRY(cudaFuncSetAttribute(k_contract_sl<EPI, LIN, 16>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)SMEM_LIMIT - 1024));
  return JFG_OK;
}

// once per device: shared-memory opt-in (call before a capture)
int device_setup(int* sms) {
  static int nsm[64] = {};
  int dev = 0;
  JFG_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return JFG_ERR_UNSUPPORTED;
  if (!nsm[dev]) {
    JFG_TRY((set_attr<JFG_EPI_NONE, false>()));
    JFG_TRY((set_attr<JFG_EPI_NONE, true>()));
    JFG_TRY((set_attr<JFG_EPI_MUL_FIELD, false>()));
    JFG_TRY((set_attr<JFG_EPI_MUL_FIELD, true>()));
    JFG_TRY((set_attr<JFG_EPI_DIV_EIG, false>()));
    JFG_TRY((set_attr<JFG_EPI_DIV_EIG, true>()));
    int n = 0;
    JFG_CUDA_TRY(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    nsm[dev] = n;
  }
  *sms = nsm[dev];
  return JFG_OK;
}

inline int kp8(int K) { return (K + 7) / 8 * 8; }
inline int kp64(int K) { return (K + 63) / 64 * 64; }

template <int PT>
int launch(const SlLaunch& L, dim3 grid, size_t smem, cudaStream_t st) {
  const bool lin = L.d.alpha != 1.0 || L.d.beta != 0.0;
#define JFG_SL(E)                                                        \
  if (lin)                                                               \
    k_contract_sl<E, true, PT><<<grid, SL_NT, smem, st>>>(L);            \
  else                                                                   \
    k_contract_sl<E, false, PT><<<grid, SL_NT, smem, st>>>(L)
  switch (L.d.epilogue) {
    case JFG_EPI_NONE:
      JFG_SL(JFG_EPI_NONE);
      break;
    case JFG_EPI_MUL_FIELD:
      JFG_SL(JFG_EPI_MUL_FIELD);
      break;
    default:
      JFG_SL(JFG_EPI_DIV_EIG);
      break;
  }
#undef JFG_SL
  JFG_LAUNCHED();
  return JFG_OK;
}

int launch_rows(const SlLaunch& L, dim3 grid, cudaStream_t st) {
  const bool lin = L.d.alpha != 1.0 || L.d.beta != 0.0;
#define JFG_SL(E)                                                            \
  if (lin)                                                                   \
    k_contract_sl_rows<E, true><<<grid, SL_NT, ROWS_SMEM, st>>>(L);          \
  else                                                                       \
    k_contract_sl_rows<E, false><<<grid, SL_NT, ROWS_SMEM, st>>>(L)
  switch (L.d.epilogue) {
    case JFG_EPI_NONE:
      JFG_SL(JFG_EPI_NONE);
      break;
    case JFG_EPI_MUL_FIELD:
      JFG_SL(JFG_EPI_MUL_FIELD);
      break;
    default:
      JFG_SL(JFG_EPI_DIV_EIG);
      break;
  }
#undef JFG_SL
  JFG_LAUNCHED();
  return JFG_OK;
}

}  // namespace

size_t sl_op_bytes(int nseg, int M, int K) {
  if (K < 1 || K > SL_KMAX || M < 1 || nseg < 1) return 0;
  return align_up((size_t)nseg * NS * M * kp8(K) * 2, 256) + align_up((size_t)nseg * M * 4, 256) +
         align_up((size_t)nseg * kp64(K) * 2, 256) +
         align_up((size_t)nseg * 4, 256);
}

SlOp sl_op(const double* src, long long ld, long long seg, int nseg, int M, int K, SlRule rule,
           void* work, const double* lam) {
  SlOp o;
  o.src = src;
  o.lam = lam;
  o.rule = rule;
  o.ld = ld;
  o.seg = seg;
  o.nseg = nseg;
  o.M = M;
  o.K = K;
  if (!work || K > SL_KMAX) return o;
  char* w = (char*)work;
  o.dig = (uint16_t*)w;
  w += align_up((size_t)nseg * NS * M * kp8(K) * 2, 256);
  o.row_e = (int*)w;
  w += align_up((size_t)nseg * M * 4, 256);
  o.col_e = (int16_t*)w;
  w += align_up((size_t)nseg * kp64(K) * 2, 256);
  o.use = (int*)w;
  return o;
}

int sl_split_ops(const SlOp* ops, int nops, cudaStream_t st) {
  SlSplitArgs A;
  int n = 0;
  for (int i = 0; i < nops; ++i) {
    const SlOp& o = ops[i];
    if (!o.dig) continue;
    if (!o.src || o.K > SL_KMAX) return JFG_ERR_ARG;
    const int Kp = kp8(o.K), kpad = kp64(o.K);
    for (int s = 0; s < o.nseg; ++s) {
      if (n == SL_MAX_SEGS) return JFG_ERR_ARG;
      A.s[n++] = SlSeg{o.src + s * o.seg,
                       o.lam,
                       o.ld,
                       o.M,
                       o.K,
                       Kp,
                       kpad,
                       o.dig + (size_t)s * NS * o.M * Kp,
                       o.row_e + (size_t)s * o.M,
                       o.col_e + (size_t)s * kpad,
                       o.use + s,
                       o.rule};
    }
  }
  if (n == 0) return JFG_OK;
  k_sl_split<<<n * SPLIT_CL, SPLIT_T, 0, st>>>(A);
  JFG_LAUNCHED();
  return JFG_OK;
}

bool sl_pays(const jfg_contract_desc& d, double min_work) {
  if (d.K > SL_KMAX || d.M < 1 || d.M > 65536 || d.P < 1 || d.batch < 1 || d.nseg > 3 ||
      (long long)d.batch * d.nseg > 65535 ||
      (long long)d.batch * d.nseg * ((d.P + 15) / 16) * ((d.M + 127) / 128) > 0x3FFFFFFF)
    return false;
  const int t = contract_f64_tile(d);
  const double tiles = (double)d.batch * d.nseg * ((d.M + t - 1) / t) * ((d.P + t - 1) / t);
  return tiles * t * t * ((d.K + 15) / 16 * 16) >= min_work && sl_us(d) < contract_f64_us(d);
}

// Fitted to calls at the least work that took digits, M = 5 to 512 by K = 16 to
// 510 in one to three dimensions: with the rule made of these and of
// contract_f64_us the slower way is taken nowhere by more than 7 % (by 9 to 90 %
// at every second shape before, by the work alone).
double sl_us(const jfg_contract_desc& d) {
  int sms = 0;
  if (sm_count(&sms) != JFG_OK) return 0.0;
  const int pt = d.K > 256 ? 16 : 32;
  const double items = (double)d.batch * d.nseg * ((d.P + pt - 1) / pt) * ((d.M + 127) / 128);
  return 6.0 + 0.02 * d.K + std::floor(items / sms) * (1.0 + 0.03 * d.K);
}
double sl_cut_us(int M, int K) { return 14.0 + 0.02 * M + 3e-5 * M * K; }

int contract_sl(const jfg_contract_desc& d, const SlOp& op, const double* in, double* out,
                cudaStream_t st) {
  JFG_TRY(validate_desc(d));
  if (!in || !out || !op.dig || d.K != op.K || d.M > op.M || d.K > SL_KMAX) return JFG_ERR_ARG;
  if (op.nseg != 1 && op.nseg < d.nseg) return JFG_ERR_ARG;
  if (d.batch == 0 || d.M == 0 || d.P == 0) return JFG_OK;
  if ((long long)d.batch * d.nseg > 65535) return JFG_ERR_ARG;
  int sms = 0;
  JFG_TRY(device_setup(&sms));
  EncodeTiledFn enc = tensor_map_encoder();
  if (!enc) return JFG_ERR_UNSUPPORTED;
  SlLaunch L = {};
  L.d = d;
  L.d.op_ld = op.ld;
  L.d.op_seg = op.seg;
  L.op = op.src;
  L.in = in;
  L.out = out;
  L.row_e = op.row_e;
  L.col_e = op.col_e;
  L.use = op.use;
  L.op_segs = d.nseg > 1 && op.nseg > 1 ? d.nseg : 1;
  L.row_ld = op.M;
  L.kpad = kp64(d.K);
  L.nkb = L.kpad / 64;
  L.mtiles = (d.M + 127) / 128;
  if (L.op_segs * L.kpad > COL_MAX) return JFG_ERR_UNSUPPORTED;
  // PT 32 streams each operator digit past twice the rows that 16 does; 16
  // where K > 256 would not fit, or 32 would leave half the SMs without work
  const long long t32 = (long long)d.batch * d.nseg * ((d.P + 31) / 32) * L.mtiles;
  const int PT = (d.K > 256 || (2 * t32 <= sms && d.P > 16)) ? 16 : 32;
  L.nptiles = (d.P + PT - 1) / PT;
  const long long items = (long long)d.batch * d.nseg * L.nptiles * L.mtiles;
  if (items > 0x3FFFFFFF) return JFG_ERR_UNSUPPORTED;
  const size_t bbytes = (size_t)L.nkb * PT * (NS + 1) * 128;
  L.bbuf = 2 * bbytes <= 144 * 1024 ? 2 : 1;
  const size_t fixed = 1024 + L.bbuf * bbytes + NWE * 32 * STG_LD * 8 + RING * PT * 4 +
                       COL_MAX * 2 + (2 * A_MAX + 10) * 8;
  const size_t room = (SMEM_LIMIT - 1024 - fixed) / ABYTES;
  L.astages = room > A_MAX ? A_MAX : (int)room;
  if (L.astages < 2) return JFG_ERR_UNSUPPORTED;
  L.a_res = L.op_segs == 1 && L.mtiles * L.nkb * NS <= L.astages ? 1 : 0;
  L.vec2 = ((uintptr_t)in & 15) == 0 && !(d.in_ld & 1) && !(d.in_seg & 1) && !(d.in_batch & 1);
  const int Kp = kp8(d.K);
  const cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)op.M, (cuuint64_t)(op.nseg * NS)};
  const cuuint64_t strides[2] = {(cuuint64_t)Kp * 2, (cuuint64_t)Kp * 2 * op.M};
  // Small operators: 128 flattened rows per tile, unless so few that the SMs
  // are better spread over 32-row tiles.  Two passes and the digits take about
  // 27 + 20 us per wave of 128-row tiles and 22 + 10.5 us per wave of 32-row
  // ones (64 x 62; less on either side for smaller ones): 150 problems (1 wave
  // to 2) 47 and 43 us, 200 (1 to 3) 47 and 52, 1024 (4 to 14) 105 and 167.
  const long long row_tiles = d.nseg * (((long long)d.batch * d.P + RT - 1) / RT);
  const bool rows = L.op_segs == 1 && d.M <= 64 && d.K <= 64 && row_tiles <= 0xFFFFFF &&
                    (items + sms - 1) / sms > 2 * ((row_tiles + sms - 1) / sms);
  const cuuint32_t box[3] = {64, rows ? (cuuint32_t)RM : 128u, 1}, estr[3] = {1, 1, 1};
  if (enc(&L.amap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (void*)op.dig, dims, strides, box, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return JFG_ERR_ARG;
  // where digits take half of the SMs at most, a CTA per tile of the FMA sums too,
  // should the operator's digits not be taken (of eigenvector factors and packed
  // operators they are)
  const long long fma_ctas = (long long)d.batch * d.nseg * ((d.M + 15) / 16) * ((d.P + 31) / 32);
  const long long tiles = rows ? row_tiles : items;
  const long long most = op.rule == SL_DENSE && 2 * tiles <= sms ? std::max(tiles, fma_ctas) : tiles;
  L.ctas = (int)(tiles < sms ? tiles : sms);
  const dim3 grid((unsigned)(most < sms ? most : sms));
  if (rows) return launch_rows(L, grid, st);
  const size_t smem = fixed + (size_t)L.astages * ABYTES;
  static_assert(FMA_SMEM <= 2 * ABYTES && FMA_SMEM <= ROWS_SMEM, "the FMA tiles fit");
  return PT == 32 ? launch<32>(L, grid, smem, st) : launch<16>(L, grid, smem, st);
}

int sl_setup() {
  int sms = 0;
  JFG_TRY(device_setup(&sms));
  return tensor_map_encoder() ? JFG_OK : JFG_ERR_UNSUPPORTED;
}

int sl_status_take(int* status) {
  int zero = 0;
  JFG_CUDA_TRY(cudaMemcpyFromSymbol(status, g_sl_status, sizeof(int)));
  JFG_CUDA_TRY(cudaMemcpyToSymbol(g_sl_status, &zero, sizeof(int)));
  return JFG_OK;
}

}  // namespace jfg
