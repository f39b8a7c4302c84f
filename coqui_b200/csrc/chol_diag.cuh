// Diagonal block of the blocked FP64 Cholesky kernels: the inverse of the Cholesky factor of a
// 32 x 32 Hermitian block, and its log-determinant, in one elimination.  Included once inside a
// namespace (chol.cu), before the kernels that use it.
//
// Column c of the elimination, with pivot d_c and p = 1 / d_c, takes every row r > c to
//   x(r, s) <- x(r, s) - f v(s),  f = S(r, c) p,
// where v(s) is the adjoint column conj(S(s, c)) for s > c (the trailing Schur complement) and row
// c of the accumulated inverse for s < c, 1 at s = c, where x starts from 0: the factor's finished
// column c makes room for the inverse's column c.  In the end C^{-1}(r, s) = x(r, s) / sqrt(d_r),
// and the factor itself is never formed: the panels need C^{-1} only.
//
// The block is a serial chain of 32 pivots, so what counts is the latency of one: a row's 32
// values stay in registers of NTH / 32 neighbouring lanes, one barrier per column passes the
// vector v and the pivot through shared memory, the chain holds one reciprocal, and the square
// roots and logarithms are taken for all rows at once at the end.  200 problems of N_mu 128, four
// blocks each: 127 us in all (246 with a square root, a division and a logarithm per column inside
// the chain and the factor inverted afterwards); 5400 of 384: 18.0 ms (22.2).
//
// Each element's operations do not depend on NTH, so all kernels give identical results.
template <typename F, int... C>
__device__ __forceinline__ void static_for(F&& f, std::integer_sequence<int, C...>) {
  (f(std::integral_constant<int, C>{}), ...);
}

template <int NTH, typename In, typename Out>
__device__ __forceinline__ void factor_invert_diag(In&& S, Out&& X, int n, double* ld_acc,
                                                   int* bad) {
  constexpr int LPR = NTH / 32, EPL = 32 / LPR;  // lanes per row, elements per lane
  __shared__ double2 v[2][32];
  __shared__ double piv[2];
  __shared__ double lg[32];
  const int lane = threadIdx.x & 31, r = threadIdx.x / LPR, q = threadIdx.x % LPR;
  const int row_hi = (threadIdx.x / 32 + 1) * (32 / LPR) - 1;  // last row of this warp
  double2 e[EPL];
#pragma unroll
  for (int j = 0; j < EPL; ++j) {
    const int s = q + LPR * j;
    e[j] = (s <= r && r < n) ? S(r, s) : make_double2(0.0, 0.0);
  }
  // the vector and pivot of column c (static) from the rows that hold them
  auto publish = [&](auto cc) {
    constexpr int c = decltype(cc)::value, b = c & 1;
    if (r == c) {
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        const int s = q + LPR * j;
        if (s < c) v[b][s] = e[j];
        if (s == c) {
          piv[b] = e[j].x;
          v[b][c] = make_double2(1.0, 0.0);
        }
      }
    } else if (r > c && q == c % LPR) {
      v[b][r] = make_double2(e[c / LPR].x, -e[c / LPR].y);
    }
  };
  publish(std::integral_constant<int, 0>{});
  double my = 1.0;  // this row's pivot
  auto column = [&](auto cc) {
    constexpr int c = decltype(cc)::value, b = c & 1;
    if (c >= n) return;  // uniform
    __syncthreads();
    const double d = piv[b];
    const bool good = d > 0.0;
    const double p = good ? 1.0 / d : 1.0;
    if (r == c && good) my = d;
    if (!good && threadIdx.x == 0) *bad = 1;
    const int src = (lane & ~(LPR - 1)) | (c % LPR);
    const double fx = p * __shfl_sync(0xffffffffu, e[c / LPR].x, src);
    const double fy = p * __shfl_sync(0xffffffffu, e[c / LPR].y, src);
    if (row_hi > c) {  // uniform over the warp
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        const int s = q + LPR * j;
        if (LPR * j > row_hi) continue;  // beyond every row of this warp
        const double2 w = v[b][s];
        const double ox = s == c ? 0.0 : e[j].x, oy = s == c ? 0.0 : e[j].y;
        if (r > c) {
          e[j].x = fma(-fx, w.x, fma(fy, w.y, ox));
          e[j].y = fma(-fx, w.y, fma(-fy, w.x, oy));
        }
      }
    }
    if constexpr (c + 1 < 32)
      if (c + 1 < n) publish(std::integral_constant<int, c + 1>{});
  };
  static_for(column, std::make_integer_sequence<int, 32>{});
  const double root = sqrt(my), inv = 1.0 / root;
#pragma unroll
  for (int j = 0; j < EPL; ++j) {
    const int s = q + LPR * j;
    double2 x = make_double2(0.0, 0.0);
    if (r < n && s < r) x = make_double2(e[j].x * inv, e[j].y * inv);
    if (r < n && s == r) x.x = inv;
    X(r, s) = x;
  }
  if (q == 0) lg[r] = log(root);
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = lane < n ? lg[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) *ld_acc += t;
  }
  __syncthreads();
}
