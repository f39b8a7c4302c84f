// Products of a fixed triangular factor with a complex64 operand on the tensor cores, both split
// into FP16 hi + lo words (tcgen05 kind::f16, FP32 accumulation): C = A opB(Bt)^T with A one of
// the per-q factors L, L^H of V and Bt row-major n x n.  Part of tc_gemm.cu (included there,
// inside its anonymous namespace, after the barrier and descriptor helpers it uses).
//
// The four long-K products of the Dyson step have a factor of V on one side (L^H Pi, L^H P1^H,
// L E, L T^H).  In the split-TF32 kernel both operands pass through registers on their way to
// shared memory; per 16 complex K of a 128 x 128-complex tile that is 96 KB of stores and 144 KB of
// operand reads against 1536 cycles of MMA, and the tile took 2000 to 2400.  Here
//  * the factor is laid out once per set_thc as the very shared-memory tiles the MMA reads (hi and
//    lo planes, 128-byte swizzle), so a K block of A is one 32 KB bulk copy;
//  * the words are FP16: half the bytes per value and twice the K per MMA.  hi = fp16(s x),
//    lo = fp16(s x - hi) carry 22 bits for every value within 2^-18 of the largest of its row (of
//    Bt: the maximum comes from a pass over it or from the epilogue that wrote it) or of its matrix
//    (A), and smaller ones are off by 2^-40 of it; s is a power of two from that maximum, and the
//    epilogue takes the powers out again.  Half as many additions into the FP32 accumulator round
//    toward zero.
//
// FP16 has five exponent bits, where TF32 words have eight, so gradings have to be taken out first.
// THC data have a free scale per point (X_P -> s_P X_P with V_PQ -> V_PQ / (s_P^2 s_Q^2)): L's rows
// carry it and Pi its inverse, so in L^H Pi the small elements of one meet the large ones of the
// other along K.  Where the columns of a factor differ by more than 2^kFacGrade they are brought to
// one size by powers of two, `ks`, which the product puts on Bt instead (X's columns in the
// projection likewise: a free scale per orbital); where its rows do, each row gets a scale of its
// own (GR kernels: 2 % slower, for the row's multiplication in the epilogue).  Relative error of
// Sigma at N_mu 300 for s_P spread over 10^3 / 10^5 / 10^6: 1.8e-5 each; with one scale per matrix
// throughout 1.8e-5 / 3e-3 / 7e-2.
//
// Per 32 complex K: 96 KB stored and 144 KB read against 1536 cycles of MMA, and half the
// conversion work.  Measured (1600 problems of N_mu 512 / 675 of 1024; split TF32 -> this form): the
// M products with their row-maximum pass 6.87 -> 4.9 ms / 17.1 -> 11.3, the W group (T and W, and
// with them the D^H D product, E and its row maxima, which are as they were) 11.4 -> 9.8 /
// 25.2 -> 20.7; W of random Hermitian Pi is 3.8e-6 / 5.7e-6 (N_mu 512 / 768) from FP64 in the 2-norm
// where split TF32 gave 7.0e-6 / 1.05e-5.
//
// CTA: 128 rows x 128 complex columns (UMMA M = 128, N = 256 with the realified rows of
// tc_gemm.cu), K blocks of 32 complex = one 128-byte row, two stages of 96 KB.  Warps 0-7 stage B
// (global -> registers two K blocks ahead -> split -> swizzled stores) and drain the accumulator,
// one lane of warp 8 issues the MMAs, one lane of warp 9 the bulk copies.  Waits are bounded as in
// tc_gemm.cu; the copy lane sees every copy it issued land before the CTA ends.

constexpr int kFacKC = 32;                                  // complex K per stage
constexpr int kFacTile = 2 * kBM * 128;                     // bytes of a packed A tile (hi, lo)
constexpr int kFacBPlane = 2 * kFacN * 128;                 // bytes of a B plane (256 real rows)
constexpr int kFacStage = kFacTile + 2 * kFacBPlane;        // 96 KB
constexpr int kFacThreads = 320;
// ST stages: two for long K; one for K of a few blocks, where a second CTA on the SM (96 KB each)
// covers the first one's start and epilogue
template <int ST> constexpr int fac_smem() {
  return ST * kFacStage + 1024 /*align*/ + 256 /*barriers*/ + 512 /*scales*/;
}
template <int ST> constexpr int fac_epi_cols() { return ST == 2 ? kFacN : kFacN / 2; }
constexpr uint32_t kFacIdesc = (1u << 4) | ((uint32_t)(2 * kFacN >> 3) << 17) |
                               ((uint32_t)(kBM >> 4) << 24);  // F16 x F16 -> F32, K-major

// 2^(14 - exponent) of a row or matrix maximum (bits of a non-negative float): the scaled values
// stay below 2^15; 1 for zero and non-finite maxima (those values then propagate as they are)
__device__ __forceinline__ int fac_exp(uint32_t bits) {
  const int e = (int)(bits >> 23) - 127;
  return bits == 0u || e >= 128 ? 14 : max(e, -100);
}
__device__ __forceinline__ float pow2f(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }

__device__ __forceinline__ void mma_f16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc,
                                        uint32_t acc) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p; }"
      ::"r"(tmem), "l"(ad), "l"(bd), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}
// arrives with the number of bytes the bulk copy will bring, then starts it
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(bar),
               "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

struct FacParams {
  const unsigned char* A;  // packed factors, sA bytes apart; problem b uses (a_q0 + b) % a_mod
  int64_t sA, a_mod, a_q0;
  const float* invA;       // 1 / scale of each row of each factor, (a_mod, M)
  const float* kB;         // powers of two that Bt takes along K, (a_mod, K); may be null
  const float* nC;         // powers of two that C's columns take, (a_mod, N); may be null
  const float2* B;
  int64_t ldb, sB;
  const uint32_t* rmB;     // (batch, n) row maxima of Bt
  float2* C;
  int64_t ldc, sC;
  uint32_t* rmC;           // (batch, n) row maxima of C, raised by atomics; may be null
  int64_t M, N, K;
  int conj_b;
  int tri;   // A is upper (> 0: k >= m) or lower (< 0: k <= m) triangular, or full (0)
  int half;  // < 0: tiles on or below the diagonal only, > 0: on or above
  int b_al;
};

// 32 complex K of four rows of Bt per thread: four values (32 bytes) of rows r + 32 j; GR: with the
// scales of these K (1 without a kb)
template <bool GR> struct FacStaging {
  float4 v[4][2];
  float ck[4];
  __device__ __forceinline__ void load(const FacParams& p, const float2* base, const float* kb,
                                       uint32_t ok, int64_t k0) {
    const int64_t k = k0 + 4 * (threadIdx.x & 7);
    if constexpr (GR) {
#pragma unroll
      for (int i = 0; i < 4; ++i) ck[i] = kb && k + i < p.K ? __ldg(kb + k + i) : 1.f;
    }
    if (k0 + kFacKC <= p.K && p.b_al) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4* q = reinterpret_cast<const float4*>(base + (int64_t)(32 * j) * p.ldb + k0);
        const bool in = (ok >> j) & 1u;
        v[j][0] = in ? __ldg(q) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[j][1] = in ? __ldg(q + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2* q = base + (int64_t)(32 * j) * p.ldb + k0;
        float2 w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          w[i] = (((ok >> j) & 1u) && k + i < p.K) ? __ldg(q + i) : make_float2(0.f, 0.f);
        v[j][0] = make_float4(w[0].x, w[0].y, w[1].x, w[1].y);
        v[j][1] = make_float4(w[2].x, w[2].y, w[3].x, w[3].y);
      }
    }
  }
  // realified rows 2r = (re, -im) and 2r + 1 = (im, re) of b (or of its conjugate), hi and lo
  __device__ __forceinline__ void store(const float (&sc)[4], int conj_b, uint32_t hi,
                                        uint32_t lo) const {
    const int r = threadIdx.x >> 3, c = threadIdx.x & 7;
    const uint32_t s0 = conj_b ? 0u : 0x80000000u, s1 = conj_b ? 0x8000u : 0u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t h[4], l[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 q = v[j][i >> 1];
        const float sk = GR ? sc[j] * ck[i] : sc[j];
        const float x = sk * ((i & 1) ? q.z : q.x), y = sk * ((i & 1) ? q.w : q.y);
        const __half2 a = __floats2half2_rn(x, y);
        const float2 f = __half22float2(a);
        const __half2 b = __floats2half2_rn(x - f.x, y - f.y);
        h[i] = *reinterpret_cast<const uint32_t*>(&a);
        l[i] = *reinterpret_cast<const uint32_t*>(&b);
      }
      const int row = 2 * (r + 32 * j);
      const uint32_t o0 = sw128(row, c), o1 = sw128(row + 1, c);
      st_shared_v4(hi + o0, h[0] ^ s0, h[1] ^ s0, h[2] ^ s0, h[3] ^ s0);
      st_shared_v4(lo + o0, l[0] ^ s0, l[1] ^ s0, l[2] ^ s0, l[3] ^ s0);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        h[i] = __byte_perm(h[i], h[i], 0x1032) ^ s1;
        l[i] = __byte_perm(l[i], l[i], 0x1032) ^ s1;
      }
      st_shared_v4(hi + o1, h[0], h[1], h[2], h[3]);
      st_shared_v4(lo + o1, l[0], l[1], l[2], l[3]);
    }
  }
};

template <int ST, bool GR>
__device__ __forceinline__ void fac_tile(const FacParams& p, int64_t bz, int64_t m0, int64_t n0,
                                         unsigned char* smem_raw) {
  if (p.half < 0 && n0 > m0) return;  // tiles strictly above the diagonal
  if (p.half > 0 && n0 < m0) return;  // strictly below
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full_b = reinterpret_cast<uint64_t*>(smem + ST * kFacStage);
  uint64_t *full_a = full_b + ST, *empty = full_a + ST;
  uint64_t *acc_bar = empty + ST, *done_bar = acc_bar + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
  float* scale = reinterpret_cast<float*>(smem + ST * kFacStage + 256);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // a triangular factor is zero beyond its triangle
  const int kbs = (int)((p.K + kFacKC - 1) / kFacKC);
  const int kb_lo = p.tri > 0 ? (int)(m0 / kFacKC) : 0;
  const int kb_hi = p.tri < 0 ? min(kbs, (int)((m0 + kBM) / kFacKC)) : kbs;
  const int nkb = kb_hi - kb_lo;
  const int64_t ia = (p.a_q0 + bz) % p.a_mod;

  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) {
      mbar_init(smem_u32(&full_b[s]), 8);  // one arrival per producer warp
      mbar_init(smem_u32(&full_a[s]), 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    mbar_init(smem_u32(acc_bar), 1);
    mbar_init(smem_u32(done_bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < kFacN) {
    // takes the power of two of column n0 + threadIdx.x out again, and A's if all its rows have one
    // (then at least 2^-34: the pair is at least 2^-148, which a float holds)
    const int64_t c = n0 + threadIdx.x;
    const int e = c < p.N ? fac_exp(p.rmB[bz * p.N + c]) : 14;
    if constexpr (GR)
      scale[threadIdx.x] = pow2f(e - 14) * (p.nC && c < p.N ? p.nC[ia * p.N + c] : 1.f);
    else
      scale[threadIdx.x] = p.invA[ia * p.M] * pow2f(e - 14);
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"((uint32_t)(2 * kFacN))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp < 8) {
    // ---------------- B producers ----------------
    bool ok = true;
    const int r = threadIdx.x >> 3;
    const float2* base = p.B + bz * p.sB + (n0 + r) * p.ldb + 4 * (threadIdx.x & 7);
    const float* kb = GR && p.kB ? p.kB + ia * p.K : nullptr;
    uint32_t rows = 0;
    float sc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t row = n0 + r + 32 * j;
      if (row < p.N) rows |= 1u << j;
      sc[j] = pow2f(14 - (row < p.N ? fac_exp(p.rmB[bz * p.N + row]) : 14));
    }
    auto step = [&](FacStaging<GR>& st, int it) -> bool {
      const int s = it % ST;
      if (!mbar_wait(smem_u32(&empty[s]), ((uint32_t)(it / ST) & 1u) ^ 1u)) return false;
      const uint32_t hi = smem_u32(smem + s * kFacStage + kFacTile);
      st.store(sc, p.conj_b, hi, hi + kFacBPlane);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&full_b[s]));
      if (it + ST < nkb) st.load(p, base, kb, rows, (int64_t)(kb_lo + it + ST) * kFacKC);
      return true;
    };
    FacStaging<GR> st0;
    st0.load(p, base, kb, rows, (int64_t)kb_lo * kFacKC);
    if constexpr (ST == 2) {
      FacStaging<GR> st1;
      if (nkb > 1) st1.load(p, base, kb, rows, (int64_t)(kb_lo + 1) * kFacKC);
      for (int it = 0; it < nkb; it += 2) {
        if (!step(st0, it)) { ok = false; break; }
        if (it + 1 < nkb && !step(st1, it + 1)) { ok = false; break; }
      }
    } else {
      for (int it = 0; it < nkb; ++it)
        if (!step(st0, it)) { ok = false; break; }
    }
    // ---------------- epilogue: TMEM -> registers (scaled) -> smem -> coalesced rows -----------
    const int q = warp & 3, h = warp >> 2;  // TMEM lane quadrant, column half
    constexpr int EC = fac_epi_cols<ST>(), PITCH = EC + 4;  // columns drained at a time
    static_assert(8 * 32 * PITCH * 4 <= ST * kFacStage, "epilogue buffer");
    float* buf = reinterpret_cast<float*>(smem) + warp * 32 * PITCH;
    bool have = false;
    if (ok) {
      have = mbar_wait(smem_u32(acc_bar), 0u);
      if (have) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    // all producers are past their last stage before it is reused
    asm volatile("bar.sync 1, %0;" ::"r"(256) : "memory");
    float mx = 0.f;
    // GR: the row's power of two.  The smaller one of it and the column's goes first, so that the
    // pair neither overflows nor underflows where the result does not.
    const int64_t row = m0 + q * 32 + lane;
    const float ra = GR && row < p.M ? p.invA[ia * p.M + row] : 1.f;
#pragma unroll 1
    for (int c0 = 0; c0 < kFacN; c0 += EC) {
      const int col = h * kFacN + c0;  // first real column of this piece
      const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)col;
#pragma unroll 1
      for (int j = 0; j < EC / 32; ++j) {
        uint32_t v[32];
        if (have) {
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
              "%11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, "
              "%28, %29, %30, %31}, [%32];"
              : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
                "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
                "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
                "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
                "=r"(v[31])
              : "r"(trow + (uint32_t)(j * 32)));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        } else {
#pragma unroll
          for (int x = 0; x < 32; ++x) v[x] = 0u;
        }
        const float4* sc4 = reinterpret_cast<const float4*>(scale + (col + j * 32) / 2);
        float4* dst = reinterpret_cast<float4*>(buf + lane * PITCH + j * 32);
#pragma unroll
        for (int x = 0; x < 4; ++x) {  // four complex columns
          const float4 f4 = sc4[x];
          const float f[4] = {f4.x, f4.y, f4.z, f4.w};
          float o[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            o[i] = __uint_as_float(v[8 * x + i]);
            if constexpr (GR) o[i] = o[i] * fminf(f[i / 2], ra) * fmaxf(f[i / 2], ra);
            else o[i] *= f[i / 2];
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) mx = fmaxf(mx, fabsf(o[i]));
          dst[2 * x] = make_float4(o[0], o[1], o[2], o[3]);
          dst[2 * x + 1] = make_float4(o[4], o[5], o[6], o[7]);
        }
      }
      __syncwarp();
      // EC / 4 lanes (16 bytes each) per row
      constexpr int LPR = EC / 4;
#pragma unroll 4
      for (int i = lane; i < 32 * LPR; i += 32) {
        const int rr = i / LPR, x = (i % LPR) * 4;
        const int64_t m = m0 + q * 32 + rr, n = n0 + (col + x) / 2;
        if (m >= p.M) continue;
        float2* cp = p.C + bz * p.sC + m * p.ldc + n;
        const float4 val = *reinterpret_cast<const float4*>(buf + rr * PITCH + x);
        if (n + 1 < p.N && ((reinterpret_cast<uintptr_t>(cp) & 15) == 0)) {
          *reinterpret_cast<float4*>(cp) = val;
        } else {
          if (n < p.N) cp[0] = make_float2(val.x, val.y);
          if (n + 1 < p.N) cp[1] = make_float2(val.z, val.w);
        }
      }
      __syncwarp();
    }
    if (p.rmC && row < p.M) atomicMax(p.rmC + bz * p.M + row, __float_as_uint(mx));
  } else if (warp == 8) {
    if (lane == 0) {
      // ---------------- MMA issuer ----------------
      bool ok = true;
      for (int it = 0; it < nkb; ++it) {
        const int s = it % ST;
        const uint32_t ph = (uint32_t)(it / ST) & 1u;
        if (!mbar_wait(smem_u32(&full_a[s]), ph) || !mbar_wait(smem_u32(&full_b[s]), ph)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a_hi = smem_u32(smem + s * kFacStage), a_lo = a_hi + kFacTile / 2;
        const uint32_t b_hi = a_hi + kFacTile, b_lo = b_hi + kFacBPlane;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const uint32_t o = (uint32_t)kk * 32;  // 16 halves along K
          const uint64_t ah = make_desc(a_hi + o), al = make_desc(a_lo + o);
          const uint64_t bh = make_desc(b_hi + o), bl = make_desc(b_lo + o);
          const uint32_t acc = (it > 0 || kk > 0) ? 1u : 0u;
          mma_f16(tmem, al, bh, kFacIdesc, acc);
          mma_f16(tmem, ah, bl, kFacIdesc, 1u);
          mma_f16(tmem, ah, bh, kFacIdesc, 1u);
        }
        mma_commit(smem_u32(&empty[s]));
      }
      if (ok) mma_commit(smem_u32(acc_bar));
      mma_commit(smem_u32(done_bar));
      mbar_drain(smem_u32(done_bar), 0u);
    }
  } else if (lane == 0) {
    // ---------------- A copies ----------------
    const unsigned char* a = p.A + ia * p.sA + ((m0 / kBM) * kbs + kb_lo) * (int64_t)kFacTile;
    int issued = 0;
    for (; issued < nkb; ++issued) {
      const int s = issued % ST;
      if (!mbar_wait(smem_u32(&empty[s]), ((uint32_t)(issued / ST) & 1u) ^ 1u)) break;
      bulk_load(smem_u32(smem + s * kFacStage), a + (int64_t)issued * kFacTile, kFacTile,
                smem_u32(&full_a[s]));
    }
    // every copy issued has landed before the CTA ends, also when a wait gave up
    for (int it = max(0, issued - ST); it < issued; ++it)
      mbar_drain(smem_u32(&full_a[it % ST]), (uint32_t)(it / ST) & 1u);
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 8) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"((uint32_t)(2 * kFacN))
                 : "memory");
  }
}

template <int ST, bool GR>
__global__ void __launch_bounds__(kFacThreads, 3 - ST) k_tc_fac(const __grid_constant__ FacParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  fac_tile<ST, GR>(p, blockIdx.z, (int64_t)blockIdx.y * kBM, (int64_t)blockIdx.x * kFacN, smem_raw);
}

// Products of different sizes in one launch (a group each); the flattened tile index picks the
// group by binary search.
struct FacGroupDev {
  FacParams p;
  int64_t tiles, tile_begin;  // tiles per matrix edge
};
template <bool GR>
__global__ void __launch_bounds__(kFacThreads, 1)
    k_tc_fac_grouped(const FacGroupDev* __restrict__ groups, int ngroups) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ FacParams sp;
  __shared__ int64_t s_bz, s_m0, s_n0;
  if (threadIdx.x == 0) {
    const int64_t t = blockIdx.x;
    int lo = 0, hi = ngroups - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (groups[mid].tile_begin <= t) lo = mid;
      else hi = mid - 1;
    }
    const FacGroupDev& g = groups[lo];
    const int64_t local = t - g.tile_begin, per = g.tiles * g.tiles, r = local % per;
    sp = g.p;
    s_bz = local / per;
    s_m0 = r / g.tiles * kBM;
    s_n0 = r % g.tiles * kFacN;
  }
  __syncthreads();
  fac_tile<2, GR>(sp, s_bz, s_m0, s_n0, smem_raw);
}

// Packing a factor: column maxima, the powers of two that level graded columns, row maxima of what
// remains, their common value where the rows are not graded, then the tiles.  Maxima are the bits
// of the largest |re|, |im| as a float, rounded up.
__device__ __forceinline__ float fac_abs(double2 v) {
  return __double2float_ru(fmax(fabs(v.x), fabs(v.y)));
}
// one column per thread, eight rows at a time
__global__ void __launch_bounds__(256) k_fac_colmax(const double2* __restrict__ L,
                                                    uint32_t* __restrict__ cm, int64_t M, int64_t K) {
  __shared__ float red[8][32];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int64_t q = blockIdx.y, k = (int64_t)blockIdx.x * 32 + x;
  const double2* a = L + q * M * K;
  float m = 0.f;
  if (k < K)
    for (int64_t r = y; r < M; r += 8) m = fmaxf(m, fac_abs(a[r * K + k]));
  red[y][x] = m;
  __syncthreads();
  if (y == 0 && k < K) {
    for (int j = 1; j < 8; ++j) m = fmaxf(m, red[j][x]);
    cm[q * K + k] = __float_as_uint(m);
  }
}
// Columns, and rows, of a matrix may differ by this power of two and keep one scale.  The words are
// off by 2^-40 of the largest element; in a row that is 2^-8 of it the terms of a sum with a graded
// Bt weigh 2^-8, and a column 2^-8 of the largest meets a Bt of 2^8: 2^(-40 + 8 + 8) of the sum,
// where FP32 rounds it.
constexpr int kFacGrade = 8;
constexpr int kFacExp = 20;  // a scale common to all rows lies within 2^+-20
__device__ __forceinline__ int fac_max_exp(uint32_t bits) { return min((int)(bits >> 23) - 127, 127); }
// smallest and largest exponent of the n nonzero maxima of a matrix (block-wide; hi < lo: none)
__device__ __forceinline__ void fac_exp_range(const uint32_t* m, int64_t n, int* lo, int* hi) {
  __shared__ int r[2];
  if (threadIdx.x == 0) {
    r[0] = 1 << 20;
    r[1] = -(1 << 20);
  }
  __syncthreads();
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x)
    if (m[i]) {
      atomicMin(&r[0], fac_max_exp(m[i]));
      atomicMax(&r[1], fac_max_exp(m[i]));
    }
  __syncthreads();
  *lo = r[0];
  *hi = r[1];
}
// cm (bits) -> ks: of graded columns (*flag gets kFacColumns) a column's power of two over the
// largest one's, 0 for an empty column; else 1
__global__ void __launch_bounds__(256) k_fac_kscale(uint32_t* __restrict__ cm, int64_t K,
                                                    int* __restrict__ flag) {
  uint32_t* c = cm + (int64_t)blockIdx.x * K;
  int lo, hi;
  fac_exp_range(c, K, &lo, &hi);
  const bool graded = hi - lo > kFacGrade;
  for (int64_t k = threadIdx.x; k < K; k += blockDim.x) {
    const float s = !graded ? 1.f : c[k] ? pow2f(max(fac_max_exp(c[k]) - hi, -100)) : 0.f;
    c[k] = __float_as_uint(s);
  }
  if (threadIdx.x == 0 && graded) atomicOr(flag, kFacColumns);
}
// rm -> the matrix's maximum in every row, unless its rows are graded or it lies beyond 2^+-kFacExp
// (*flag gets kFacRows)
__global__ void __launch_bounds__(256) k_fac_rscale(uint32_t* __restrict__ rm, int64_t M,
                                                    int* __restrict__ flag) {
  uint32_t* r = rm + (int64_t)blockIdx.x * M;
  __shared__ uint32_t most;
  if (threadIdx.x == 0) most = 0u;
  int lo, hi;
  fac_exp_range(r, M, &lo, &hi);
  const bool one = hi - lo <= kFacGrade && hi <= kFacExp && hi >= -kFacExp;
  if (hi < lo || one) {
    for (int64_t i = threadIdx.x; i < M; i += blockDim.x) atomicMax(&most, r[i]);
    __syncthreads();
    for (int64_t i = threadIdx.x; i < M; i += blockDim.x) r[i] = most;
  } else if (threadIdx.x == 0) {
    atomicOr(flag, kFacRows);
  }
}
// one warp per row, after division by ks (may be null)
__global__ void __launch_bounds__(256) k_fac_rowmax(const double2* __restrict__ L,
                                                    const float* __restrict__ ks,
                                                    uint32_t* __restrict__ rm, int64_t M, int64_t K) {
  const int64_t r = (int64_t)blockIdx.x * 8 + threadIdx.x / 32, q = blockIdx.y;
  if (r >= M) return;
  const double2* a = L + (q * M + r) * K;
  float m = 0.f;
  for (int64_t k = threadIdx.x & 31; k < K; k += 32) {
    const float d = ks ? ks[q * K + k] : 1.f;
    if (d > 0.f)
      m = fmaxf(m, __double2float_ru(fmax(fabs(a[k].x), fabs(a[k].y)) / (double)d));
  }
  const uint32_t w = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
  if ((threadIdx.x & 31) == 0) rm[q * M + r] = w;
}

// The packed tiles of a factor: tile (mt, kb) holds rows 128 mt .. and complex K 32 kb .. as a
// 128 x 64 FP16 hi plane and a lo plane in the swizzled order of shared memory, zeros beyond the
// matrix.  One thread per 16-byte chunk (four values).
__global__ void k_fac_pack(const double2* __restrict__ L, const float* __restrict__ ks,
                           const uint32_t* __restrict__ rm, unsigned char* __restrict__ out,
                           float* __restrict__ inv, int64_t M, int64_t K, int64_t sA) {
  const int64_t q = blockIdx.y, kbs = (K + kFacKC - 1) / kFacKC;
  const double2* a = L + q * M * K;
  const int64_t chunks = (M + kBM - 1) / kBM * kbs * kBM * 8;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < chunks;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i & 7), r = (int)((i >> 3) % kBM);
    const int64_t tile = i / (8 * kBM), m = tile / kbs * kBM + r, k = tile % kbs * kFacKC + 4 * c;
    const int e = m < M ? fac_exp(rm[q * M + m]) : 14;
    if (m < M && k == 0) inv[q * M + m] = pow2f(e - 14);
    uint32_t h[4], l[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      double2 v = make_double2(0.0, 0.0);
      double s = (double)pow2f(14 - e);
      if (m < M && k + j < K) {
        const float d = ks ? ks[q * K + k + j] : 1.f;
        if (d > 0.f) v = a[m * K + k + j];
        if (d > 0.f) s /= (double)d;
      }
      const double x = s * v.x, y = s * v.y;
      const __half hx = __double2half(x), hy = __double2half(y);
      const __half lx = __double2half(x - (double)__half2float(hx));
      const __half ly = __double2half(y - (double)__half2float(hy));
      h[j] = (uint32_t)__half_as_ushort(hx) | ((uint32_t)__half_as_ushort(hy) << 16);
      l[j] = (uint32_t)__half_as_ushort(lx) | ((uint32_t)__half_as_ushort(ly) << 16);
    }
    unsigned char* t = out + q * sA + tile * kFacTile + sw128(r, c);
    *reinterpret_cast<uint4*>(t) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(t + kFacTile / 2) = make_uint4(l[0], l[1], l[2], l[3]);
  }
}

// Row maxima (bits of the largest |re|, |im|) of a complex64 n-column matrix times ks along the row
// (may be null), one warp per row
__device__ __forceinline__ void row_max(const float2* __restrict__ a, const float* __restrict__ ks,
                                        uint32_t* rm, int64_t n) {
  float m = 0.f;
  if (ks) {
#pragma unroll 4
    for (int64_t i = threadIdx.x & 31; i < n; i += 32)
      m = fmaxf(m, ks[i] * fmaxf(fabsf(a[i].x), fabsf(a[i].y)));
  } else {
#pragma unroll 4
    for (int64_t i = threadIdx.x & 31; i < n; i += 32)
      m = fmaxf(m, fmaxf(fabsf(a[i].x), fabsf(a[i].y)));
  }
  const uint32_t w = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
  if ((threadIdx.x & 31) == 0) *rm = w;
}
// row r belongs to problem r / per, which takes the scales (q0 + r / per) % mod
__global__ void __launch_bounds__(256) k_row_max(const float2* __restrict__ A,
                                                 const float* __restrict__ ks,
                                                 uint32_t* __restrict__ rm, int64_t rows, int64_t n,
                                                 int64_t per, int64_t mod, int64_t q0) {
  const int64_t r = (int64_t)blockIdx.x * 8 + threadIdx.x / 32;
  if (r < rows) row_max(A + r * n, ks ? ks + (q0 + r / per) % mod * n : nullptr, rm + r, n);
}
// the same for matrices of different sizes: group g has `batch` matrices of n rows, sA apart
__global__ void __launch_bounds__(256) k_row_max_grouped(const TcRowMaxGroup* __restrict__ groups,
                                                         int ngroups) {
  const int64_t r = (int64_t)blockIdx.x * 8 + threadIdx.x / 32;
  int lo = 0, hi = ngroups - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (groups[mid].row_begin <= r) lo = mid;
    else hi = mid - 1;
  }
  const TcRowMaxGroup g = groups[lo];
  const int64_t l = r - g.row_begin;
  if (l < g.n * g.batch) row_max(g.A + l / g.n * g.sA + l % g.n * g.n, g.ks, g.rm + l, g.n);
}
