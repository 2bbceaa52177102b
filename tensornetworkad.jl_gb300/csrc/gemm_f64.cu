// FP64 (DFMA) GEMM of the plain path, on matrices or on tensors in any label
// order: the row, column and inner index of each operand is a list of extents
// and strides (GemmMap), so a pairwise contraction needs no permutation pass.
//
// GB300 retires 1.7 DFMA a clock and SM, so everything but that pipe is cheap:
// index arithmetic, shared loads, even 16×16 tiles (one multiply-add per two
// shared loads).  What matters is that the 152 SMs get equal shares: the tile
// (16, 32 or 64 square) and the split of K are those with the least work on the
// busiest SM (gemm_f64_plan).  A split product is summed by the CTA that
// arrives last at its tile, in fixed order.  The next K slice is loaded to
// registers while the current one is multiplied.
#include <algorithm>

#include "tnad_internal.h"

namespace tnad {

namespace {

__device__ __forceinline__ int64_t map_off(const GemmMap& m, unsigned i) {
  if (m.nd == 1) return (int64_t)i * m.str[0];
  int64_t o = 0;
#pragma unroll
  for (int d = 0; d < GemmMap::kMax; ++d) {
    if (d + 1 < m.nd) {
      const unsigned q = i / m.dim[d];
      o += (int64_t)(i - q * m.dim[d]) * m.str[d];
      i = q;
    } else if (d + 1 == m.nd) {
      o += (int64_t)i * m.str[d];
    }
  }
  return o;
}

struct GemmArgs {
  unsigned M, N, K, kchunk;
  int ks;
  double alpha, beta;
  const double *A, *B;
  double *C, *part;
  int* cnt;
  GemmMap am, ak, bk, bn, cm, cn;
  int scaled, accum;   // alpha ≠ 1, beta ≠ 0: compared once on the host, each comparison is an FP64 instruction
  int a_rows, b_rows;  // lanes run along the rows (columns) of the tile, else along K
};

// SYM: C = Cᵀ, the tiles above the diagonal are the others' mirror images
template <int BM, bool SYM>
__global__ void __launch_bounds__(256) k_gemm_f64(const GemmArgs g) {
  constexpr int BK = 16, T = BM / 16;  // T×T outputs and T loads per operand and thread
  __shared__ double As[2][BK][BM + 1];
  __shared__ double Bs[2][BK][BM + 1];
  __shared__ int last;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  if (SYM && blockIdx.y > blockIdx.x) return;
  const unsigned m0 = blockIdx.x * BM, n0 = blockIdx.y * BM;
  const unsigned kbeg = blockIdx.z * g.kchunk, kend = min(g.K, kbeg + g.kchunk);
  // this thread's elements of a slice: (row ai[q], inner ak[q]) and (inner, column)
  int ai[T], aK[T], bi[T], bK[T];
  int64_t ao[T], bo[T];
#pragma unroll
  for (int q = 0; q < T; ++q) {
    ai[q] = g.a_rows ? tid % BM : ty + 16 * q;
    aK[q] = g.a_rows ? tid / BM + (256 / BM) * q : tx;
    bi[q] = g.b_rows ? tid % BM : ty + 16 * q;
    bK[q] = g.b_rows ? tid / BM + (256 / BM) * q : tx;
    ao[q] = m0 + ai[q] < g.M ? map_off(g.am, m0 + ai[q]) : -1;
    bo[q] = n0 + bi[q] < g.N ? map_off(g.bn, n0 + bi[q]) : -1;
  }
  double ra[T], rb[T], acc[T][T];
  auto load = [&](unsigned k0) {
#pragma unroll
    for (int q = 0; q < T; ++q) {
      const unsigned ka = k0 + aK[q], kb = k0 + bK[q];
      ra[q] = (ao[q] >= 0 && ka < kend) ? g.A[ao[q] + map_off(g.ak, ka)] : 0.0;
      rb[q] = (bo[q] >= 0 && kb < kend) ? g.B[bo[q] + map_off(g.bk, kb)] : 0.0;
    }
  };
#pragma unroll
  for (int i = 0; i < T; ++i)
#pragma unroll
    for (int j = 0; j < T; ++j) acc[i][j] = 0.0;
  load(kbeg);
  int buf = 0;
  for (unsigned k0 = kbeg; k0 < kend; k0 += BK, buf ^= 1) {
#pragma unroll
    for (int q = 0; q < T; ++q) {
      As[buf][aK[q]][ai[q]] = ra[q];
      Bs[buf][bK[q]][bi[q]] = rb[q];
    }
    __syncthreads();  // one barrier a slice: the other buffer was read before the last one
    if (k0 + BK < kend) load(k0 + BK);
    const int kn = min((unsigned)BK, kend - k0);
    if (kn == BK) {
#pragma unroll
      for (int k = 0; k < BK; ++k) {
        double a[T], b[T];
#pragma unroll
        for (int i = 0; i < T; ++i) a[i] = As[buf][k][tx + 16 * i];
#pragma unroll
        for (int j = 0; j < T; ++j) b[j] = Bs[buf][k][ty + 16 * j];
#pragma unroll
        for (int i = 0; i < T; ++i)
#pragma unroll
          for (int j = 0; j < T; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
      }
    } else {
      for (int k = 0; k < kn; ++k) {
#pragma unroll
        for (int i = 0; i < T; ++i)
#pragma unroll
          for (int j = 0; j < T; ++j) acc[i][j] = fma(As[buf][k][tx + 16 * i], Bs[buf][k][ty + 16 * j], acc[i][j]);
      }
    }
  }
  if (g.ks > 1) {
    const int64_t tiles = (int64_t)gridDim.x * gridDim.y, tile = blockIdx.x + (int64_t)gridDim.x * blockIdx.y;
    double* P = g.part + ((int64_t)blockIdx.z * tiles + tile) * (BM * BM);
#pragma unroll
    for (int i = 0; i < T; ++i)
#pragma unroll
      for (int j = 0; j < T; ++j) __stcg(&P[tid + 256 * (i * T + j)], acc[i][j]);
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(&g.cnt[tile], 1) == g.ks - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
#pragma unroll
    for (int i = 0; i < T; ++i)
#pragma unroll
      for (int j = 0; j < T; ++j) acc[i][j] = 0.0;
    for (int z = 0; z < g.ks; ++z) {
      const double* Pz = g.part + ((int64_t)z * tiles + tile) * (BM * BM);
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) acc[i][j] += __ldcg(&Pz[tid + 256 * (i * T + j)]);
    }
    if (tid == 0) g.cnt[tile] = 0;  // for the next product on this stream
  }
#pragma unroll
  for (int j = 0; j < T; ++j) {
    const unsigned gj = n0 + ty + 16 * j;
    if (gj >= g.N) continue;
    const int64_t cj = map_off(g.cn, gj);
#pragma unroll
    for (int i = 0; i < T; ++i) {
      const unsigned gi = m0 + tx + 16 * i;
      if (gi >= g.M) continue;
      double* c = g.C + cj + map_off(g.cm, gi);
      double v = acc[i][j];
      if (g.scaled) v *= g.alpha;
      *c = g.accum ? v + g.beta * (*c) : v;
      if (SYM && blockIdx.y < blockIdx.x) g.C[map_off(g.cm, gj) + map_off(g.cn, gi)] = *c;
    }
  }
}

// Tile and split with the least time on the busiest SM, in clocks: its share of
// the tiles at 1.7 DFMA a clock, ~1200 for a CTA's first loads and stores (partly
// hidden where an SM holds several), ~2500 more where K is split (partials,
// counter, the sum).  Measured with its launch: 32×32×32 12.6 µs with one 32×32
// tile, K in two halves and a second kernel, 7.8 µs by this rule; 1024³ stays at
// the pipe's limit (2.07 ms).
void gemm_f64_plan(int sms, int64_t M, int64_t N, int64_t K, int* tile, int* splits) {
  double best = 1e300;
  for (int t : {64, 32, 16}) {
    const int64_t tiles = ((M + t - 1) / t) * ((N + t - 1) / t);
    if (t < 64 && (N + t - 1) / t > 65535) continue;  // grid.y
    const int64_t kmax = tiles <= kGemmCounters ? std::min<int64_t>(64, std::max<int64_t>(1, K / 16)) : 1;
    for (int64_t ks = 1; ks <= kmax; ++ks) {
      const int64_t kc = ((K + ks - 1) / ks + 15) / 16 * 16;
      const int64_t per_sm = (tiles * ((K + kc - 1) / kc) + sms - 1) / sms;
      const double cost =
          (double)per_sm * ((double)t * t * (double)std::min(kc, K) / 1.7 + 400.0) + 1200.0 + (ks > 1 ? 2500.0 + 60.0 * ks : 0.0);
      if (cost < best) {
        best = cost;
        *tile = t;
        *splits = (int)ks;
      }
      if (tiles * ks > 8 * (int64_t)sms) break;
    }
  }
}

}  // namespace

void gemm_f64_map(tnad_ctx* c, int64_t M, int64_t N, int64_t K, double alpha, const double* A, const GemmMap& am,
                  const GemmMap& ak, const double* B, const GemmMap& bk, const GemmMap& bn, double beta, double* C,
                  const GemmMap& cm, const GemmMap& cn, bool sym) {
  TNAD_REQUIRE(M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31), TNAD_ERR_ARG, "gemm_f64: size");
  int tile = 64, ks = 1;
  gemm_f64_plan(c->sm_count, M, N, K, &tile, &ks);
  GemmArgs g;
  g.M = (unsigned)M;
  g.N = (unsigned)N;
  g.K = (unsigned)K;
  const int64_t kc = ks > 1 ? ((K + ks - 1) / ks + 15) / 16 * 16 : K;
  g.kchunk = (unsigned)kc;
  g.ks = (int)((K + kc - 1) / kc);
  g.alpha = alpha;
  g.beta = beta;
  g.scaled = alpha != 1.0;
  g.accum = beta != 0.0;
  g.A = A;
  g.B = B;
  g.C = C;
  g.am = am;
  g.ak = ak;
  g.bk = bk;
  g.bn = bn;
  g.cm = cm;
  g.cn = cn;
  g.a_rows = am.str[0] == 1 || ak.str[0] != 1;
  g.b_rows = bn.str[0] == 1 || bk.str[0] != 1;
  g.cnt = c->d_cnt;
  WsScope scope(c);
  const int64_t tm = (M + tile - 1) / tile, tn = (N + tile - 1) / tile;
  TNAD_REQUIRE(tn <= 65535, TNAD_ERR_ARG, "gemm_f64: too many columns");
  g.part = g.ks > 1 ? ws_d(c, (int64_t)g.ks * tm * tn * tile * tile) : nullptr;
  const dim3 grid((unsigned)tm, (unsigned)tn, (unsigned)g.ks);
  KernelTimer kt(c, "gemm_f64", 2.0 * (double)M * (double)N * (double)K);
  auto launch = [&](auto* kernel) { kernel<<<grid, 256, 0, c->stream>>>(g); };
  if (tile == 64)
    launch(sym ? k_gemm_f64<64, true> : k_gemm_f64<64, false>);
  else if (tile == 32)
    launch(sym ? k_gemm_f64<32, true> : k_gemm_f64<32, false>);
  else
    launch(sym ? k_gemm_f64<16, true> : k_gemm_f64<16, false>);
  count_launch(c);
  check_launch(c, "gemm_f64");
}

// Matrix-vector products (N = 1), the Gram–Schmidt steps of GMRES: a tiled
// GEMM would compute whole 32×32 tiles for one useful column.
// y(M) = alpha·A·x + beta·y with A M×K (lda), x K values (stride incx), K small:
// one thread per row, coalesced over the rows of A.
__global__ void k_gemv_n(int64_t M, int64_t K, double alpha, const double* __restrict__ A, int64_t lda,
                         const double* __restrict__ x, int64_t incx, double beta, double* __restrict__ y) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < M; i += (int64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int64_t k = 0; k < K; ++k) s = fma(A[i + k * lda], x[k * incx], s);
    const double v = alpha * s;
    y[i] = beta == 0.0 ? v : v + beta * y[i];
  }
}

// part[chunk, i] = Σ_{k in chunk} A[k + i·lda]·x[k] for the M ≤ 32 columns of
// A (K×M, lda): y = Aᵀx split over K chunks, threads strided over k (coalesced),
// a fixed-order block reduction per column.
constexpr int kGemvMaxM = 32;
__global__ void __launch_bounds__(256) k_gemv_t_part(int64_t M, int64_t K, int64_t kchunk,
                                                     const double* __restrict__ A, int64_t lda,
                                                     const double* __restrict__ x, int64_t incx,
                                                     double* __restrict__ part) {
  __shared__ double red[8][kGemvMaxM];
  const int64_t k0 = (int64_t)blockIdx.x * kchunk, k1 = min(K, k0 + kchunk);
  double acc[kGemvMaxM];
#pragma unroll
  for (int i = 0; i < kGemvMaxM; ++i) acc[i] = 0.0;
  for (int64_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
    const double xv = x[k * incx];
#pragma unroll
    for (int i = 0; i < kGemvMaxM; ++i)
      if (i < M) acc[i] = fma(A[k + i * lda], xv, acc[i]);
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < kGemvMaxM; ++i) {
    double v = acc[i];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[w][i] = v;
  }
  __syncthreads();
  if (threadIdx.x < M) {
    double s = 0.0;
    for (int ww = 0; ww < 8; ++ww) s += red[ww][threadIdx.x];
    part[blockIdx.x * M + threadIdx.x] = s;
  }
}

// y[i] = alpha·Σ_chunk part[chunk, i] + beta·y[i] (fixed order)
__global__ void k_gemv_t_sum(int64_t M, int nchunk, const double* __restrict__ part, double alpha, double beta,
                             double* __restrict__ y) {
  const int64_t i = threadIdx.x;
  if (i >= M) return;
  double s = 0.0;
  for (int z = 0; z < nchunk; ++z) s += part[z * M + i];
  const double v = alpha * s;
  y[i] = beta == 0.0 ? v : v + beta * y[i];
}

static GemmMap map1(int64_t n, int64_t stride) {
  GemmMap m;
  m.nd = 1;
  m.dim[0] = (unsigned)n;
  m.str[0] = stride;
  return m;
}

void gemm_f64_gram(tnad_ctx* c, int64_t n, int64_t K, const double* A, const double* B, double* C) {
  gemm_f64_map(c, n, n, K, 1.0, A, map1(n, K), map1(K, 1), B, map1(K, 1), map1(n, K), 0.0, C, map1(n, 1), map1(n, n),
               true);
}

void gemm_f64(tnad_ctx* c, char ta, char tb, int64_t M, int64_t N, int64_t K, double alpha, const double* A,
              int64_t lda, const double* B, int64_t ldb, double beta, double* C, int64_t ldc) {
  if (M <= 0 || N <= 0) return;
  if (K <= 0) {
    if (beta == 0.0) {
      for (int64_t j = 0; j < N; ++j) fill(c, C + j * ldc, M, 0.0);
    } else if (beta != 1.0) {
      for (int64_t j = 0; j < N; ++j) scale(c, M, beta, C + j * ldc);
    }
    return;
  }
  int ita = (ta == 'T' || ta == 't'), itb = (tb == 'T' || tb == 't');
  if (N == 1 && (!ita || M <= kGemvMaxM)) {
    // matrix-vector product: x = op(B) is a K-vector with stride ldb when tb = T
    const int64_t incx = itb ? ldb : 1;
    KernelTimer kt(c, "gemm_f64", 2.0 * (double)M * (double)K);
    if (!ita) {
      k_gemv_n<<<(int)std::min<int64_t>((M + 255) / 256, 4096), 256, 0, c->stream>>>(M, K, alpha, A, lda, B, incx,
                                                                                     beta, C);
      count_launch(c);
    } else {
      // K chunks of at least 512 values, at most 2 CTAs per SM: the FP64 pipe
      // of every SM takes part (34 chunks of 2048 at K = 69632 left the
      // product DFMA-bound on 34 SMs)
      const int64_t nch = std::max<int64_t>(1, std::min<int64_t>((K + 511) / 512, 2 * c->sm_count));
      const int64_t kchunk = (K + nch - 1) / nch;
      WsScope scope(c);
      double* part = ws_d(c, nch * M);
      k_gemv_t_part<<<(unsigned)nch, 256, 0, c->stream>>>(M, K, kchunk, A, lda, B, incx, part);
      k_gemv_t_sum<<<1, kGemvMaxM, 0, c->stream>>>(M, (int)nch, part, alpha, beta, C);
      count_launch(c, 2);
    }
    check_launch(c, "gemv_f64");
    return;
  }
  gemm_f64_map(c, M, N, K, alpha, A, map1(M, ita ? lda : 1), map1(K, ita ? 1 : lda), B, map1(K, itb ? ldb : 1),
               map1(N, itb ? 1 : ldb), beta, C, map1(M, 1), map1(N, ldc));
}

void gemm(tnad_ctx* c, int prec, char ta, char tb, int64_t M, int64_t N, int64_t K, double alpha, const double* A,
          int64_t lda, const double* B, int64_t ldb, double beta, double* C, int64_t ldc) {
  if (prec == TNAD_PREC_TF32X3) {
    TNAD_REQUIRE(c->tc_ok, TNAD_ERR_STATE, "TF32X3 contractions need an sm_100-family GPU (tcgen05)");
    gemm_tf32x3(c, ta, tb, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
  } else if (prec == TNAD_PREC_FP64_TC) {
    gemm_fp64tc(c, ta, tb, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, true);
  } else if (prec == TNAD_PREC_FP64 && c->fp64_tc) {
    gemm_fp64tc(c, ta, tb, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
  } else {
    gemm_f64(c, ta, tb, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
  }
}

}  // namespace tnad
