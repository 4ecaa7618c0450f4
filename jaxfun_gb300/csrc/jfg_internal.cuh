// Internal helpers shared by the jaxfun_gb300 CUDA translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "jaxfun_gb300.h"

namespace jfg {

// Last CUDA error observed on this host thread (reported by jfg_last_cuda_error).
void set_last_cuda_error(cudaError_t e);

// Kernel-launch accounting (jfg_launch_count): every launch site adds its
// launches; while a stream is being captured into a graph nothing is counted
// and each graph replay adds its kernel-node count instead.
void count_launches(long long n);
void set_capturing(bool on);

#define JFG_CUDA_TRY(expr)                              \
  do {                                                  \
    cudaError_t _e = (expr);                            \
    if (_e != cudaSuccess) {                            \
      ::jfg::set_last_cuda_error(_e);                   \
      return JFG_ERR_CUDA;                              \
    }                                                   \
  } while (0)

#define JFG_CHECK_LAUNCH()                              \
  do {                                                  \
    cudaError_t _e = cudaGetLastError();                \
    if (_e != cudaSuccess) {                            \
      ::jfg::set_last_cuda_error(_e);                   \
      return JFG_ERR_CUDA;                              \
    }                                                   \
  } while (0)

// after a <<<>>> launch: check it and count it
#define JFG_LAUNCHED()                                  \
  do {                                                  \
    JFG_CHECK_LAUNCH();                                 \
    ::jfg::count_launches(1);                           \
  } while (0)

#define JFG_TRY(expr)                                   \
  do {                                                  \
    int _s = (expr);                                    \
    if (_s != JFG_OK) return _s;                        \
  } while (0)

// A contraction operator: hi part (always) and, for the split-TF32 tensor-core
// path, the lo part with the same layout.
template <typename T>
struct OpRef {
  const T* hi;
  const T* lo;
  OpRef offset(long long o) const { return OpRef{hi + o, lo ? lo + o : nullptr}; }
};

// Dispatch of one contraction pass to an engine.
// DF: FP64 data, double-FP32 arithmetic (contract_df.cu).  TB: FP32 data on
// the tensor cores with a split-BF16 operator (OpRef<float> then points at
// BF16 arrays).  TH: FP32 data on the tensor cores as scaled split-FP16 pairs
// with a split-FP16 operator scaled per row (variable-coefficient apply only).
enum class Engine { F64, F32, TC, DF, TB, TH };

// Auxiliaries of the TH engine: the inverse row scales of the packed FP16
// operators and four per-problem max |x| slots (float bits, [4][batch]): the
// apply's input (slot 0) and the inputs of its passes 2-4 (slots 1-3).
struct H16Ops {
  const float* op_inv = nullptr;
  unsigned* slots = nullptr;  // [H16_SLOTS][batch]: max |x| of each pass's input
};
// per-problem max slots of a scaled split-FP16 operator apply (the 3-D one
// chains six)
constexpr int H16_SLOTS = 6;

// Fused dot product of a field-multiply or eigenvalue-divide pass: the
// epilogue writes, per problem b, partials part[b * DOT_NBMAX + i], i < *nb,
// of sum(acc * out) (acc the contraction before the epilogue factor, out the
// written value) -- p.Ap of the variable-coefficient operator in its field
// pass, r.M^-1 r of the fast diagonalisation in its divide pass.  The launch
// sets *nb (its tiles per problem x 8 epilogue warps), or 0 when the pass
// cannot produce it (then the caller computes the dot itself).
constexpr int DOT_NBMAX = 128;
struct DotOut {
  float* part = nullptr;
  int* nb = nullptr;
};

int sm_count(int* n);  // SMs of the current device
// tile of the FP64 CUDA-core launch (64, 32 or 16)
int contract_f64_tile(const jfg_contract_desc& d);
// its time in us: an SM does two FMAs per clock, padding included
double contract_f64_us(const jfg_contract_desc& d);
int contract_f64(const jfg_contract_desc& d, const double* op, const double* in, double* out,
                 cudaStream_t st);
int contract_f32(const jfg_contract_desc& d, const float* op, const float* in, float* out,
                 cudaStream_t st);
int contract_df64(const jfg_contract_desc& d, const double* op, const float2* op_pairs,
                  const double* in, double* out, cudaStream_t st, bool in_pairs = false,
                  bool out_pairs = false);
// dst[i] = (hi, lo) FP32 split of src[i] (the DF engine's pre-split operator)
int split_pairs_f64(const double* src, float2* dst, long long n, cudaStream_t st);
int contract_tc(const jfg_contract_desc& d, const float* op_hi, const float* op_lo,
                const float* in, float* out, cudaStream_t st, const DotOut* dot = nullptr);
// the same contraction with the operator as BF16 (hi, lo): three BF16 MMAs per product
int contract_tc_b16(const jfg_contract_desc& d, const uint16_t* op_hi, const uint16_t* op_lo,
                    const float* in, float* out, cudaStream_t st, const DotOut* dot = nullptr);
// the same contraction in scaled split FP16: operator (hi, lo) FP16 scaled per
// row with inverse scales op_inv[s * op_inv_seg + m]; the input of problem b
// is scaled by a power of two from in_max[b] (float bits of an upper bound on
// max |in[b]|); out_max[b] (optional, atomicMax) receives max |out[b]|
int contract_tc_h16(const jfg_contract_desc& d, const uint16_t* op_hi, const uint16_t* op_lo,
                    const float* op_inv, long long op_inv_seg, const unsigned* in_max,
                    unsigned* out_max, const float* in, float* out, cudaStream_t st,
                    const DotOut* dot = nullptr);
// ngroups contractions in persistent grouped launches (contract_tc.cu)
int contract_tc_grouped(int ng, const jfg_contract_desc* ds, const float* const* op_hi,
                        const float* const* op_lo, const float* const* in, float* const* out,
                        const jfg_tc_config& cfg, cudaStream_t st);
jfg_tc_config tc_default_config();
// Process-wide autotuning of single-group tensor-core launches (contract_tc.cu)
void set_single_autotune(int on);
int single_autotune();
// One-time per-device setup of the tensor-core kernels (shared-memory opt-in,
// tensor-map encoder); call before capturing their first launch into a graph.
int tc_setup();

// An FP64 operator cut into FP16 digits for the tensor-core FP64 contraction
// (contract_sl.cu): where the operator itself lies and, in a workspace of
// sl_op_bytes, its digits, row exponents and column exponents.
constexpr int SL_KMAX = 512;      // largest contracted extent
constexpr int SL_MAX_SEGS = 8;    // operator segments cut in one launch
// CUDA-core multiply-adds of a pass (its tiles' padding included) from which
// the tensor-core contraction is tried: when the operator is cut in the same
// call, and when it has been cut before.  Two passes of 31 x 64^2 (8.1e6
// each): 29 us cut in the call against 41 us; of 16 x 64^2: 31.7 against
// 25.4 us.  Below them shapes differ little; above, sl_us and sl_cut_us tell the
// shapes that would lose.
constexpr double SL_MIN_WORK = 8e6;
constexpr double SL_MIN_WORK_CUT = 4e6;
// How an operator must look for its digits to be taken (contract_sl.cu); where
// it does not, the same launch sums it by FP64 FMAs.
enum SlRule { SL_DENSE = 0, SL_FACTORS = 1 };
struct SlOp {
  const double* src = nullptr;
  const double* lam = nullptr;  // eigenvalues that the inputs were divided by, or null
  long long ld = 0, seg = 0;
  int nseg = 0, M = 0, K = 0;
  SlRule rule = SL_DENSE;
  uint16_t* dig = nullptr;  // null: not cut, the CUDA-core contraction serves it
  int* row_e = nullptr;
  int16_t* col_e = nullptr;
  int* use = nullptr;  // per segment: 1 digits, 0 FMAs (written by the cut)
  // segment s alone
  SlOp segment(int s) const {
    SlOp o = *this;
    o.src += s * seg;
    o.nseg = 1;
    if (dig) {
      o.dig += (size_t)s * 8 * M * ((K + 7) / 8 * 8);
      o.row_e += (size_t)s * M;
      o.col_e += (size_t)s * ((K + 63) / 64 * 64);
      o.use += s;
    }
    return o;
  }
};
size_t sl_op_bytes(int nseg, int M, int K);  // 0 when K > SL_KMAX
SlOp sl_op(const double* src, long long ld, long long seg, int nseg, int M, int K, SlRule rule,
           void* work, const double* lam = nullptr);
int sl_split_ops(const SlOp* ops, int nops, cudaStream_t st);  // operators without dig are skipped
// a pass on the tensor cores against the CUDA cores: large enough, and faster
// (its operator cut before)
bool sl_pays(const jfg_contract_desc& d, double min_work = SL_MIN_WORK);
double sl_us(const jfg_contract_desc& d);  // a pass, us
double sl_cut_us(int M, int K);            // cutting operators of up to M x K, us
int contract_sl(const jfg_contract_desc& d, const SlOp& op, const double* in, double* out,
                cudaStream_t st);
int sl_setup();
int sl_status_take(int* status);

inline int contract(Engine e, const jfg_contract_desc& d, OpRef<double> op, const double* in,
                    double* out, cudaStream_t st) {
  // DF: op.lo, when set, holds the operator pre-split into interleaved FP32
  // (hi, lo) pairs with the FP64 operator's element indexing (split_pairs_f64)
  if (e == Engine::DF) return contract_df64(d, op.hi, (const float2*)op.lo, in, out, st);
  return contract_f64(d, op.hi, in, out, st);
}
inline int contract(Engine e, const jfg_contract_desc& d, OpRef<float> op, const float* in,
                    float* out, cudaStream_t st, const DotOut* dot = nullptr) {
  if (e == Engine::TC) return contract_tc(d, op.hi, op.lo, in, out, st, dot);
  if (e == Engine::TB)
    return contract_tc_b16(d, (const uint16_t*)op.hi, (const uint16_t*)op.lo, in, out, st, dot);
  if (dot && dot->nb) *dot->nb = 0;  // CUDA-core engines do not fuse the dot
  return contract_f32(d, op.hi, in, out, st);
}

// Internal epilogues of the FP64 CUDA-core contraction (not part of the C
// ABI's jfg_contract_desc.epilogue values): the coefficient of a
// variable-coefficient form from the last pass of its backward transform.
constexpr int EPI_EXP_WEIGHT = 8;  // kw = exp(c1[b] (v - c0[b])) lam_m[m] lam_p[p]
constexpr int EPI_MOMENTS = 9;     // v, plus (count, mean, M2) per tile
int contract_f64_coef(const jfg_contract_desc& d, int kind, const double* op, const double* in,
                      double* out, double* aux, float* aux32, double* part, long long* tiles,
                      cudaStream_t st);

// Optional device-side active subset of a batch (jfg_contract_desc.batch_list).
struct Active {
  const int* list = nullptr;
  const int* count = nullptr;
};

// Problem index of slot j of a (possibly listed) batch, or -1 when the slot is
// past the active count or the entry is out of range.  n_active is *count
// (or batch without a list), read once by the caller.
__device__ __forceinline__ int active_problem(const int* list, int n_active, int batch, int j) {
  if (j >= n_active) return -1;
  const int b = list ? list[j] : j;
  return (b >= 0 && b < batch) ? b : -1;
}
__device__ __forceinline__ int active_count(const int* list, const int* count, int batch) {
  if (!list) return batch;
  const int c = *count;
  return c < 0 ? 0 : (c > batch ? batch : c);
}

// One lane of the (converged) warp: the tcgen05 issuers run whole warps on
// warp-uniform values and let this lane issue.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "elect.sync _|P1, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(p));
  return p != 0;
}

// A zero-initialised descriptor for a single-segment pass with no epilogue.
inline jfg_contract_desc make_desc(int batch, int M, int P, int K, Active act = Active()) {
  jfg_contract_desc d = {};
  d.batch_list = act.list;
  d.batch_count = act.count;
  d.batch = batch;
  d.nseg = 1;
  d.M = M;
  d.P = P;
  d.K = K;
  d.op_ld = K;
  d.in_ld = K;
  d.in_batch = (long long)P * K;
  d.out_ld = P;
  d.out_batch = (long long)M * P;
  d.epilogue = JFG_EPI_NONE;
  d.alpha = 1.0;
  d.beta = 0.0;
  return d;
}

int validate_desc(const jfg_contract_desc& d);

// Higher-level sequences (ops.cu), shared by the FP64, FP32 and tensor-core paths.
template <typename T>
int tp_apply(Engine e, int ndim, const int* rows, const int* cols, int batch,
             const OpRef<T>* mats, const T* in, T* out, void* work, size_t work_bytes,
             cudaStream_t st, const T* shift = nullptr);
// sl (FP64): E and W cut by the caller (fd_sl_ops); null: cut in the call
// when the workspace has room for them and a pass is large enough
template <typename T>
int fd_solve(Engine e, int ndim, int n, int batch, OpRef<T> E, OpRef<T> W, const T* lam,
             const T* c0, const T* c1, const T* rhs, T* out, void* work, size_t work_bytes,
             cudaStream_t st, Active act = Active(), const DotOut* dot = nullptr,
             const SlOp* sl = nullptr);
// sl (FP64): the packed operators cut by the caller (varcoef_sl_ops)
template <typename T>
int varcoef_apply(Engine e, int ndim, int n, int nq, int batch, OpRef<T> ops, const T* kw,
                  const T* u, T* v, void* work, size_t work_bytes, cudaStream_t st,
                  Active act = Active(), const H16Ops* h16 = nullptr,
                  const DotOut* dot = nullptr, const SlOp* sl = nullptr);
// Workspace and layout of the cut operators of fd_solve (2: E, W) and
// varcoef_apply (SL_VARCOEF); sl_split_ops cuts them.
constexpr int SL_VARCOEF = 4;
size_t fd_sl_bytes(int n);
void fd_sl_ops(int n, const double* E, const double* W, const double* lam, void* work, SlOp* out);
// whether a varcoef_apply is large enough to cut its operators for it
bool varcoef_pays(int ndim, int n, int nq, int batch, double min_work);
size_t varcoef_sl_bytes(int ndim, int n, int nq);
void varcoef_sl_ops(int ndim, int n, int nq, const double* ops, void* work, SlOp* out);
// number of inverse row scales of the 2-D packed operators (TH engine)
inline long long varcoef_h16_rows(int n, int nq) { return 4LL * nq + 3LL * n; }
inline long long varcoef_h16_rows_nd(int ndim, int n, int nq) {
  return ndim == 3 ? 5LL * nq + 3LL * n : varcoef_h16_rows(n, nq);
}

// Read and clear the device status word of the BF16 GEMM kernel.
int gemm_status_take(int* status);

// Scratch of the pass sequences (with room for cut FP64 operators: *_ws_sl;
// the sequences accept either and cut in the call when there is room).
size_t tp_apply_ws(int ndim, const int* rows, const int* cols, int batch, int eb);
size_t tp_apply_ws_sl(int ndim, const int* rows, const int* cols, int batch, int eb);
size_t fd_ws(int ndim, int n, int batch, int eb);
size_t varcoef_ws(int ndim, int n, int nq, int batch, int eb);

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace jfg
