// Internal interface of the dense solve kernels (lu.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#define LU_NB 128  // LU block size (rows/columns of a diagonal block)
#define LU_SB 16   // sub-block of the diagonal factorization and of the panel solves
// floats per diagonal block of the 16 x 16 sub-block inverses (L^{-1}, U^{-1})
#define LU_SI (2 * (LU_NB / LU_SB) * LU_SB * LU_SB)

namespace bem {

// cs[j] = 2^s_j with max_i |A[i, j]| 2^s_j in [0.5, 1); A32 = A * diag(cs)
// rounded to FP32, identity padding up to Npad (a multiple of LU_NB).
void lu_prepare(const double* A64, int64_t lda, int N, int Npad, double* cs, float* A32,
                int64_t ld32, cudaStream_t st);
// In-place blocked LU without pivoting of the Npad x Npad FP32 matrix.
// Dinv (lu_dinv_floats(K) floats) receives, per diagonal block, the inverses
// of its unit-lower and upper triangles (2 x LU_NB^2 floats per block), and
// after all blocks the 16 x 16 sub-block inverses (LU_SI floats per block).
// info: first block with a vanishing pivot (1-based), untouched otherwise.
// x3: 3xTF32 updates.
inline size_t lu_dinv_floats(int K) { return (size_t)K * (2 * LU_NB * LU_NB + LU_SI); }
struct TcPlan;
int lu_factor(float* A, int64_t ld, int Npad, float* Dinv, int* info, int x3, cudaStream_t st,
              const TcPlan* tc = nullptr, int* err = nullptr);
// M_b couplings of the triangular sweeps (Mc: K * 2 * 128^2 floats), after
// the factorization
void lu_couplings(const float* A, int64_t ld, int Npad, const float* Dinv, float* Mc, cudaStream_t st);
// (epoch, value) words of the triangular sweeps: y of both sweeps (2 Npad)
// and the helpers' partial sums (at most LU_TRSV_PMAX CTAs per block row)
constexpr int LU_TRSV_PMAX = 4;
inline size_t lu_tag_words(int Npad) { return (size_t)(2 + 2 * LU_TRSV_PMAX) * (size_t)Npad; }
// z <- cs .* U^{-1} L^{-1} v (v, z FP64 of length N, the sweeps FP32) and
// w <- 0, in one launch.  tags: lu_tag_words(Npad) words of (epoch, value)
// scratch, zeroed before the first call; epoch: > 0 and different in every
// call on the same tags; err: timeout flag, set when a wait polled wait_limit
// times in vain.  rf: 2 Npad floats, used when the block rows do not all stay
// resident.  wepoch_shift (failure injection, normally 0): results are
// published under epoch + wepoch_shift, so that a nonzero shift makes every
// dependent wait run out.  pmax: at most this many CTAs per block row (the
// count also stays within what the GPU keeps resident).  Returns 0 or a CUDA
// error.
int lu_solve_vec(const float* A, int64_t ld, int N, int Npad, const float* Dinv, const float* Mc, const double* v,
                 const double* cs, double* z, double* w, float* rf, unsigned long long* tags, int epoch, int* err,
                 cudaStream_t st, int wait_limit = 1 << 20, int wepoch_shift = 0, int pmax = LU_TRSV_PMAX);

// The steps of the refinement return 0 or the CUDA error of their launch.
// y += alpha A x
int gemv64(const double* A, int64_t lda, int N, const double* x, double* y, double alpha, cudaStream_t st);
// Two passes of classical Gram-Schmidt of w against V[:, 0:m] (m <= 30) and
// the normalization vn = w / |w|.  host (page-locked, 64 doubles): the
// coefficients of the passes at [0] and [32], |w|^2 at [62]; hinfo: the two
// ints at info.  refuse (failure injection, normally 0): 1 no cluster above
// the portable size is launched, 2 none at all.
int gram_schmidt64(const double* V, int64_t ldv, int N, int m, double* w, double* vn, double* host, const int* info,
                   int* hinfo, cudaStream_t st, int refuse = 0);
// v = r / |r| (zeros for r = 0), x = 0 when given; *host = |r|^2; hcnt: the
// two ints at cnt, when given; refuse as above
int normalize64(const double* r, int N, double* v, double* x, double* host, const int* info, int* hinfo,
                cudaStream_t st, const int* cnt = nullptr, int* hcnt = nullptr, int refuse = 0);
// x += Z[:, 0:m] y (y on the host, m <= 32), w = b
int add_zy64(const double* Z, int64_t ldz, int N, int m, const double* y, double* x, const double* b, double* w,
             cudaStream_t st);

// C (M x N) = beta C + alpha A (M x 128) B (128 x N); M, N multiples of 128.
void gemm_tile128(const float* A, int64_t lda, const float* B, int64_t ldb, float* C, int64_t ldc,
                  int M, int N, float alpha, float beta, int x3, cudaStream_t st);

void diag_selftest(float* A1, float* A2, int64_t ld, float* D1, float* D2, float* SI, int* info,
                   cudaStream_t st);

// tcgen05 trailing update (gemm_tc.cu).  The plan holds the TMA maps of the
// transposed L panel, its lo part, the matrix (U panel) and the U lo part.
struct TcPlan {
  float* A = nullptr;
  int64_t ld = 0;
  int Npad = 0;
  float* Lt = nullptr;    // Npad x 128, K-major
  float* Ltlo = nullptr;  // Npad x 128
  float* Ulo = nullptr;   // 128 x Npad (K-major per column)
  alignas(64) unsigned char mA[128];
  alignas(64) unsigned char mAlo[128];
  alignas(64) unsigned char mB[128];
  alignas(64) unsigned char mBlo[128];
  alignas(64) unsigned char mC[128];  // the matrix as C (persistent kernel)
  alignas(64) unsigned char mB128[128];    // B and B lo with 128-column boxes
  alignas(64) unsigned char mBlo128[128];  // (the diagonal block's own update)
  bool ok = false;
  int variant = 1;  // 1: one CTA per tile; 2: persistent, warp-specialized
  int grid = 0;     // persistent kernel: CTAs (SMs) it may use
};
// variant 2 runs the persistent kernel on all SMs but `reserve`
bool tc_plan(TcPlan& p, float* A, int64_t ld, int Npad, float* Lt, float* Ltlo, float* Ulo, int variant = 1,
             int reserve = 0);
// Lt, Ltlo, Ulo of step k (from the factored panels)
void tc_split(const TcPlan& p, int k, cudaStream_t st);
// part of step k's trailing update: rows [ro, ro+M), columns [co, co+N) of
// the trailing matrix  A22 -= L21 U12.  ctr: two zeroed device ints that the
// persistent kernel's CTAs claim tiles from (and rearm when done), or null
// for a static tile order; launches sharing ctr must not overlap.
int tc_gemm_sub(const TcPlan& p, int k, int ro, int co, int M, int N, int* err, cudaStream_t st,
                int* ctr = nullptr);
// The update C -= L U of the trailing matrix from block `org` on by step k and,
// with q (step k + 1's plan), by step k + 1 in the same pass over C.  strips:
// only its first block column and row, without the diagonal block.  Plans of
// variant 2.
int tc_update(const TcPlan& p, const TcPlan* q, int k, int org, bool strips, int* err, cudaStream_t st,
              int* ctr = nullptr);
// Steps share bulk updates in pairs while more than LU_PAIR columns remain
// (lu_factor_lookahead in lu.cu says why), with plans of variant 2.
constexpr int LU_PAIR = 3328;
// ctr: two zeroed device ints for the bulk updates' tile counter (or null);
// tc: LU_PLANS plans, step k uses tc[k % LU_PLANS].  A pair's operands are in
// use until its bulk update ends, two steps after: four plans with buffers of
// their own then, else (lu_own_plans) two, each given twice.
constexpr int LU_PLANS = 4;
inline int lu_own_plans(int Npad, int variant) { return variant == 2 && Npad - 2 * LU_NB > LU_PAIR ? 4 : 2; }
int lu_factor_lookahead(float* A, int64_t ld, int Npad, float* Dinv, int* info, cudaStream_t st,
                        cudaStream_t la, cudaEvent_t fork, cudaEvent_t* evP, cudaEvent_t* evT,
                        cudaStream_t tl, cudaEvent_t* evR, const TcPlan* tc, int* err, int* ctr = nullptr);

}  // namespace bem
