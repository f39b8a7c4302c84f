// Batched complex GEMMs of the mixed-precision path (projections and Dyson products).
#pragma once

#include "common.cuh"

namespace cq {

// what of a packed matrix is graded
constexpr int kFacColumns = 1, kFacRows = 2;
// Matrices A (M x K) packed for tc_packed_product (split FP16 tiles, tc_fac.cuh).
struct TcFactorView {
  const unsigned char* packed = nullptr;  // matrices `stride` bytes apart
  const float* inv = nullptr;             // 1 / scale of each row, (nmat, M)
  const float* ks = nullptr;              // graded columns only: their powers of two, (nmat, K)
  bool rows = false;                      // rows of one matrix differ in `inv`
  int64_t M = 0, K = 0, stride = 0;
};
struct TcFactor {
  DevBuf<unsigned char> packed;
  DevBuf<float> inv;
  DevBuf<float> ks;
  DevBuf<uint32_t> mx;  // row maxima, kept for the next packing
  DevBuf<int> flag;
  int grade = 0;        // kFacColumns | kFacRows
  int64_t M = 0, K = 0, stride = 0;
  TcFactorView view() const {
    return {packed.p, inv.p, grade & kFacColumns ? ks.p : nullptr, (grade & kFacRows) != 0, M, K, stride};
  }
  void release() {
    packed.release();
    inv.release();
    ks.release();
    mx.release();
    flag.release();
  }
};
// nmat row-major complex128 matrices; level_k: graded columns are brought to one size, for a product
// whose Bt carries the inverse grading along K.  Waits for the stream.
void tc_pack_matrix(TcFactor& f, const double2* L, int64_t M, int64_t K, int64_t nmat, bool level_k,
                    cudaStream_t s);
// dst = the matrices idx of src
void tc_gather_matrices(TcFactor& dst, const TcFactor& src, const std::vector<int64_t>& idx,
                        cudaStream_t s);

// C[b](m, n) = sum_k A(m, k) opB(Bt[b])(n, k) for b < batch: A the packed matrix (q0 + b) % mod,
// upper (tri > 0: k >= m) or lower (tri < 0: k <= m) triangular or full; Bt (N x K) and C (M x N)
// row-major complex64, one after the other; conj_b conjugates Bt.  row_max holds the row maxima of
// Bt (bits of the largest |re|, |im| as float, (batch, N)); those of C are raised in out_max
// ((batch, M), may be null).  half < 0: only the 128 x 128 tiles on or below the diagonal are formed
// and written, half > 0: on or above it.
// Of a factor with levelled columns Bt is multiplied by ks along K; row_max is then that of the
// multiplied Bt (tc_row_max with ks).  b_has_ks: Bt was written with it already.  ks_c: C's columns
// (N = K of them) are written multiplied by ks, for a next product with the same factor.
void tc_packed_product(const TcFactorView& f, int tri, int64_t mod, int64_t q0, const float2* Bt,
                       bool conj_b, int64_t N, const uint32_t* row_max, float2* C,
                       uint32_t* out_max, int half, int64_t batch, cudaStream_t s,
                       bool b_has_ks = false, bool ks_c = false);

// THC collocation X (nk, Np, nb) prepared for the projection GEMMs.
struct TcOperand {
  const double2* X = nullptr;
  int64_t nk = 0, Np = 0, nb = 0;
  DevBuf<unsigned char> packed;  // complex64 X (nk, Np, nb) then X^T (nk, nb, Np)
  TcFactor Xp;                   // X packed, where the primary -> aux projection uses it
  DevBuf<uint32_t> rm;           // row maxima of a call's operand
  DevBuf<unsigned char> tmp, tmp2;  // per-call intermediates
  void release() {
    Xp.release();
    rm.release();
    packed.release();
    tmp.release();
    tmp2.release();
  }
};

// p2a: for tc_project_p2a too (the IBZ route's X per self-energy row only projects back)
void tc_pack_X(TcOperand& op, const double2* X, int64_t nk, int64_t Np, int64_t nb, bool p2a,
               cudaStream_t s);

// out[b] = X^k G^b X^k^H  (Np x Np, complex64) for nbatch problems b = (tau, k), k = b % nk;
// G (nbatch, nb, nb) complex128.
void tc_project_p2a(TcOperand& op, const double2* Gk, float2* out, int64_t nk, int64_t Np,
                    int64_t nb, int64_t nbatch, cudaStream_t s);

// out[b] = X^k^H S^b X^k  (nb x nb, complex128) for nbatch problems, k = b % nk; S (nbatch,
// Np, Np) complex64.
void tc_project_a2p(TcOperand& op, const float2* Sk, double2* out, int64_t nk, int64_t Np,
                    int64_t nb, int64_t nbatch, cudaStream_t s);

// Pre-split operand format: one float4 (hi.re, hi.im, lo.re, lo.im) per complex value with
// hi = rna_tf32(x), lo = rna_tf32(x - hi); built once for operands used by many GEMMs.
// in: nbatch blocks of (rows x cols) complex128; transpose writes each block transposed.
void to_split(const double2* in, float4* out, int64_t rows, int64_t cols, int64_t batch,
              bool transpose, cudaStream_t s);
// Complex64 copy of nbatch (rows x cols) complex128 blocks (transposed if asked).  The GEMM
// splits complex64 operands while staging them; the copy reads half the bytes of the
// pre-split format per K block, which is what bounds the long-K products.
void to_c64(const double2* in, float2* out, int64_t rows, int64_t cols, int64_t batch,
            bool transpose, cudaStream_t s);

// Split-TF32 tensor-core GEMM, "NT" form:
//   C[b](m, n) = sum_k opA(A[b])(m, k) * opB(Bt[b])(n, k)
// A: row-major M x K (lda), Bt: row-major N x K (ldb), each complex64 or pre-split (the
// *_split flags) and optionally conjugated; C: row-major complex64 (ldc).  Strides in
// complex elements; sA/sB/sC are the batch strides.
// Known zero structure lets a tile skip K blocks (and whole tiles):
//   a_upper: A(m, k) = 0 for k < m      a_lower: A(m, k) = 0 for k > m
//   b_lower: B(k, n) = 0 for k < n      b_upper: B(k, n) = 0 for k > n
//   lower_only: only tiles touching the lower triangle (m >= n) are written.
// a_mod / b_mod (> 0): the operand's batch index is (q0 + b) % mod (per-q operands shared
// by every frequency of a flattened (w, q) batch).
// a_ident / b_ident: the operand is used as (stored values + identity), with the identity on
// the operand's own diagonal (m == k for A, n == k for B); complex64 operands only.
struct TcStructure {
  bool a_upper = false, a_lower = false, b_lower = false, b_upper = false, lower_only = false;
  // tiles strictly below the diagonal are written as zeros without products (their entries
  // are not needed, and a later product may still read them)
  bool upper_zero = false;
  bool a_ident = false, b_ident = false;
  int64_t a_mod = 0, a_q0 = 0, b_mod = 0, b_q0 = 0;
};

void tc_cgemm_nt(const void* A, bool a_split, bool conj_a, int64_t lda, int64_t sA, const void* Bt,
                 bool b_split, bool conj_b, int64_t ldb, int64_t sB, float2* C, int64_t ldc,
                 int64_t sC, int64_t M, int64_t N, int64_t K, int64_t batch, cudaStream_t s,
                 const TcStructure& st = TcStructure{});

// Products of square triangular factors (M = N = K) of different sizes in one launch; a group's Bt
// and C hold `batch` matrices sB and sC elements apart, all with one factor.  table: device copy of
// the descriptors.
struct TcFactorGroup {
  TcFactorView f;
  bool upper = false, conj_b = false;
  const float2* Bt = nullptr;
  int64_t sB = 0;
  const uint32_t* row_max = nullptr;
  float2* C = nullptr;
  int64_t sC = 0;
  uint32_t* out_max = nullptr;
  int half = 0;
  int64_t batch = 1;
  bool b_has_ks = false, ks_c = false;
};
void tc_factor_grouped(const std::vector<TcFactorGroup>& groups, DevBuf<unsigned char>& table,
                       cudaStream_t s);
// Row maxima of `batch` n x n complex64 matrices sA apart into rm (batch, n), for every group.
struct TcRowMaxGroup {
  const float2* A;
  int64_t n, sA, batch;
  uint32_t* rm;
  const float* ks;    // along each row; may be null
  int64_t row_begin;  // filled in by the call
};
void tc_row_max_grouped(std::vector<TcRowMaxGroup> groups, DevBuf<unsigned char>& table,
                        cudaStream_t s);
// Row maxima of a (rows, n) complex64 array, as tc_packed_product reads them; ks (mod, n) along each
// row (may be null), `per` rows to a problem and problem b with the scales (q0 + b) % mod.
void tc_row_max(const float2* A, uint32_t* rm, int64_t rows, int64_t n, cudaStream_t s,
                const float* ks = nullptr, int64_t per = 1, int64_t mod = 1, int64_t q0 = 0);

// One group of a grouped product: a batched "NT" product as tc_cgemm_nt describes.
struct TcGroup {
  const void* A = nullptr;
  bool a_split = false, conj_a = false;
  int64_t lda = 0, sA = 0;
  const void* Bt = nullptr;
  bool b_split = false, conj_b = false;
  int64_t ldb = 0, sB = 0;
  float2* C = nullptr;
  int64_t ldc = 0, sC = 0;
  int64_t M = 0, N = 0, K = 0, batch = 1;
  TcStructure st;
};

// All groups in one launch (same operand formats; the tile configuration follows the largest
// K and N).  table is the device copy of the group descriptors.
void tc_cgemm_grouped(const std::vector<TcGroup>& groups, DevBuf<unsigned char>& table,
                      cudaStream_t s);

// Tile-configuration autotuner of tc_cgemm_nt (default on; COQUI_B200_AUTOTUNE=0 or
// tc_set_autotune(0) selects the built-in heuristic) and the number of tuned shape classes.
void tc_set_autotune(int on);
int64_t tc_tuned_shapes();
// Pins the tile configuration (-1: autotuner / heuristic); false for an unknown index.
bool tc_set_forced_cfg(int cfg);
int tc_num_cfgs();

// What tensor-core kernels reported, of the kinds in `mask`: a bounded wait was given up; a primary ->
// auxiliary projection saw NaN or Inf in G.  Returns and clears one kind, the input's first; the
// other stays for the next call.
constexpr int kTcTimeout = 1, kTcNonfinite = 2;
int tc_take_flags(int mask);
// Time limit of the tensor-core kernels' bounded waits on the current device (ns; <= 0: the
// default 2 s).
void tc_set_wait_ns(int64_t ns);

}  // namespace cq
