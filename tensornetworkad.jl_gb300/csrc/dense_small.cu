// Small dense kernels of the subspace eigensolver, in one CTA or one cluster:
//  - Cholesky of a p×p Gram matrix and the inverse of its triangular factor
//    (CholeskyQR of the n×p block: Q = Y·R⁻¹), in one cluster of 16 CTAs;
//  - parallel Jacobi eigendecompositions of a symmetric p×p matrix held in
//    shared memory (circle-method rounds of p/2 disjoint rotations): FP32,
//    one-sided (the Rayleigh–Ritz problems, refined by products where FP64 is
//    wanted), and FP64, two-sided (the gauge-fixing problems; its eigenvectors
//    accumulate in global memory);
//  - a counter-based Gaussian generator for deterministic start blocks.
#include <cfloat>
#include <cmath>

#include "fp64_fast.cuh"
#include "per_device.h"
#include "tnad_internal.h"

namespace tnad {

// ---------------------------------------------------------------- Cholesky
// G (p×p, column-major, symmetric positive semi-definite) → R⁻¹ (p×p, upper
// triangular, zeros below) with G + E = RᵀR and E ≥ 0 diagonal: a pivot below
// kPivotFloor·max_k G_kk (a column numerically inside the span of the previous
// ones, e.g. when the subspace is wider than the rank of the matrix it
// iterates on) is raised to that floor, so the factor stays finite and the
// column maps to a vector of norm ≲ 1.  *fail = 1 when G has no positive
// finite diagonal.
//
// One cluster of 16 CTAs.  GB300 retires 1.7 FP64 multiply-adds a clock and SM:
// the p³/3 of factor and inverse alone take 85 µs in one SM at p = 96, and the
// one-CTA factorisation with its quotient, square root and two barriers a
// pivot took 260 µs, the inverse 89 more.  Here the columns of G = L·Lᵀ and of
// Y = L⁻¹ (the right-hand sides of L·Y = I) are dealt to the CTAs in panels of
// 4, right-looking: the owner factors a panel (one row per thread; every warp
// carries a copy of the 4×4 diagonal block, so no barrier inside), one cluster
// barrier, every CTA reads the panel from the owner's shared memory and
// updates its own columns of both parts.  The owner of the next panel updates
// and factors that one first and leaves its other columns for the time between
// its arrival at the barrier and the others'.  R⁻¹ = Yᵀ.  Panels of 8 on 8 CTAs
// without that order took 107 µs, this 86 (p = 96, factor and inverse): a chain of
// p/4 panels, half of the warps' stalls at barriers, the FP64 pipe 15% busy.
//
// near > 0 (a second pass): where p·max|G − I|² ≤ near, R⁻¹ to first order instead of a
// factorisation (5 µs).  The callers' bounds are what the product that uses R⁻¹
// rounds: 2^-26 before a 3xTF32 one, where orthogonality is then good to 1.5e-8 (an FP32
// factorisation, which stood there before, left ~1e-7), 2^-55 before an FP64 one.
constexpr double kPivotFloor = 1e-14;
constexpr int kCholC = 16;    // CTAs of the cluster
constexpr int kCholNB = 4;    // columns of a panel
constexpr int kCholMaxP = 160;
constexpr int kCholLd = kCholMaxP + 1;  // column stride; slot kCholMaxP holds 1/L_kk
constexpr int kCholPanels = (kCholMaxP / kCholNB + kCholC - 1) / kCholC;  // panels of one CTA

__global__ void __launch_bounds__(256) k_chol_inv(const double* __restrict__ G, int p, double floor_rel, float near,
                                                  double* __restrict__ Rinv, int* __restrict__ fail) {
  extern __shared__ __align__(16) double csm[];
  double* A = csm;                                        // own columns of L, kCholPanels·kCholNB × kCholLd
  double* Y = A + kCholPanels * kCholNB * kCholLd;        // own columns of L⁻¹
  double* Lp = Y + kCholPanels * kCholNB * kCholLd;       // the current panel, kCholNB × kCholLd
  __shared__ double fl_sh;
  __shared__ unsigned emax_sh;  // FP32 bits of max|E| over the own columns
  const int rank = blockIdx.x;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int np = (p + kCholNB - 1) / kCholNB;
  auto gcol = [&](int lc) { return ((lc / kCholNB) * kCholC + rank) * kCholNB + lc % kCholNB; };
  if (threadIdx.x == 0) emax_sh = 0u;
  __syncthreads();
  unsigned emax = 0u;
  for (int lc = w; lc < kCholPanels * kCholNB; lc += 8) {
    const int j = gcol(lc);
    if (j >= p) continue;
    for (int i = lane; i < p; i += 32) {
      const double g = G[i + (int64_t)j * p];
      A[lc * kCholLd + i] = g;
      Y[lc * kCholLd + i] = i == j ? 1.0 : 0.0;
      if (near > 0.f) emax = max(emax, __float_as_uint(fabsf(d2f_rn(i == j ? g - 1.0 : g))));  // NaN: above all
    }
  }
  if (near > 0.f) {
    atomicMax(&emax_sh, emax);
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(remote)
                 : "r"((uint32_t)__cvta_generic_to_shared(&emax_sh)), "r"(lane % kCholC));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(emax) : "r"(remote));
    for (int o = 16; o > 0; o >>= 1) emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, o));
    const float e = __uint_as_float(emax);
    if ((float)p * e * e <= near) {  // false for NaN
      for (int lc = w; lc < kCholPanels * kCholNB; lc += 8) {
        const int j = gcol(lc);
        if (j >= p) continue;
        for (int i = lane; i < p; i += 32) {
          const double g = A[lc * kCholLd + i];
          Rinv[i + (int64_t)j * p] = i > j ? 0.0 : i < j ? -g : fma(-0.5, g, 1.5);
        }
      }
      asm volatile("barrier.cluster.arrive;\nbarrier.cluster.wait;" ::: "memory");  // emax_sh was read
      return;
    }
  }
  if (w == 0) {
    double mx = 0.0;
    for (int k = lane; k < p; k += 32) mx = fmax(mx, G[k + (int64_t)k * p]);
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) {
      const bool ok = mx > 0.0 && isfinite(mx);
      fl_sh = ok ? floor_rel * mx : 1e-30;
      if (!ok && rank == 0) *fail = 1;
    }
  }
  __syncthreads();
  const double flo = fl_sh;
  // Factor the panel J in its owner's shared memory: row k0 + tid in this thread,
  // rows k0..k0+3 also in lanes 0..3 of every warp
  auto factor = [&](int J) {
    const int k0 = J * kCholNB, nc = min(kCholNB, p - k0);
    double* Ap = A + (J / kCholC) * kCholNB * kCholLd;
    const int i = k0 + (int)threadIdx.x, id = k0 + (lane & (kCholNB - 1));
    double a[kCholNB], d[kCholNB];
#pragma unroll
    for (int c = 0; c < kCholNB; ++c) {
      a[c] = (c < nc && i < p) ? Ap[c * kCholLd + i] : 0.0;
      d[c] = (c < nc && id < p) ? Ap[c * kCholLd + id] : 0.0;
    }
    __syncthreads();  // every warp has its copy of the diagonal block
    if ((int)(threadIdx.x & ~31u) >= p - k0) return;  // no row of the panel in this warp
#pragma unroll
    for (int c = 0; c < kCholNB; ++c) {
      if (c < nc) {
        double piv = __shfl_sync(0xffffffffu, d[c], c);
        if (!(piv > flo)) piv = flo;
        const double inv = rsqrt_any(piv);
        a[c] = i == k0 + c ? piv * inv : a[c] * inv;
        d[c] *= inv;
#pragma unroll
        for (int b = c + 1; b < kCholNB; ++b) {
          if (b < nc) {
            const double lb = __shfl_sync(0xffffffffu, d[c], b);
            a[b] = fma(-a[c], lb, a[b]);
            d[b] = fma(-d[c], lb, d[b]);
          }
        }
        if (threadIdx.x == 0) Ap[c * kCholLd + kCholMaxP] = inv;
      }
    }
#pragma unroll
    for (int c = 0; c < kCholNB; ++c)
      if (c < nc && i < p) Ap[c * kCholLd + i] = a[c];
  };
  // col[r] −= Σ_c f_c·L(r, k0 + c) for the rows r = r0 + lane, r0 + lane + step...
  auto apply = [&](double* col, const double* f, int nc, int r0, int step, int from) {
    for (int r = r0 + lane; r < p; r += step) {
      if (r < from) continue;
      double v = col[r];
#pragma unroll
      for (int c = 0; c < kCholNB; ++c)
        if (c < nc) v = fma(-f[c], Lp[c * kCholLd + r], v);
      col[r] = v;
    }
  };
  if (rank == 0) factor(0);
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  for (int J = 0; J < np; ++J) {
    const int k0 = J * kCholNB, nc = min(kCholNB, p - k0), owner = J % kCholC;
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    {  // the panel, rows k0.. and the 1/L_kk slot, from the owner's shared memory
      const double* Ap = A + (J / kCholC) * kCholNB * kCholLd;
      uint32_t remote;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                   : "=r"(remote)
                   : "r"((uint32_t)__cvta_generic_to_shared(Ap)), "r"(owner));
      const int nr = p - k0 + 1;
      for (int c = w & (kCholNB - 1); c < nc; c += kCholNB)
        for (int e = lane + 32 * (w / kCholNB); e < nr; e += 64) {
          const int row = e < nr - 1 ? k0 + e : kCholMaxP;
          double v;
          asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(remote + (uint32_t)(c * kCholLd + row) * 8u));
          Lp[c * kCholLd + row] = v;
        }
    }
    __syncthreads();
    const int k1 = k0 + nc;  // first column of the next panel
    const bool next = J + 1 < np && rank == (J + 1) % kCholC;
    if (next) {
      const int c = w & (kCholNB - 1);
      if (k1 + c < p) {
        double f[kCholNB];
#pragma unroll
        for (int q = 0; q < kCholNB; ++q) f[q] = q < nc ? Lp[q * kCholLd + k1 + c] : 0.0;
        apply(A + (((J + 1) / kCholC) * kCholNB + c) * kCholLd, f, nc, k1 + 32 * (w / kCholNB), 64, k1 + c);
      }
      __syncthreads();
      factor(J + 1);
    }
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    // own columns: L part beyond the panel (and the next one, done above), Y part
    // up to the panel's last column
    for (int lc = w; lc < 2 * kCholPanels * kCholNB; lc += 8) {
      const bool yp = lc >= kCholPanels * kCholNB;
      const int l = yp ? lc - kCholPanels * kCholNB : lc, j = gcol(l);
      if (j >= p || (yp ? j >= k1 : j < (next ? k1 + kCholNB : k1))) continue;
      double* col = (yp ? Y : A) + l * kCholLd;
      double f[kCholNB];
      if (!yp) {
#pragma unroll
        for (int c = 0; c < kCholNB; ++c) f[c] = c < nc ? Lp[c * kCholLd + j] : 0.0;
      } else {
        // forward substitution within the panel's rows, lane c holding row k0 + c
        double v = lane < nc ? col[k0 + lane] : 0.0;
#pragma unroll
        for (int c = 0; c < kCholNB; ++c) {
          f[c] = 0.0;
          if (c < nc) {
            f[c] = __shfl_sync(0xffffffffu, v, c) * Lp[c * kCholLd + kCholMaxP];
            if (lane > c && lane < nc) v = fma(-f[c], Lp[c * kCholLd + k0 + lane], v);
          }
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < kCholNB; ++c)
          if (lane == c && c < nc) col[k0 + c] = f[c];
      }
      apply(col, f, nc, k1, 32, yp ? 0 : j);
    }
    __syncthreads();  // Lp is free, the own columns are up to date
  }
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  // R⁻¹(j, i) = Y(i, j): column j of Y is row j of R⁻¹
  for (int lc = w; lc < kCholPanels * kCholNB; lc += 8) {
    const int j = gcol(lc);
    if (j >= p) continue;
    for (int i = lane; i < p; i += 32) Rinv[j + (int64_t)i * p] = i >= j ? Y[lc * kCholLd + i] : 0.0;
  }
  // no CTA leaves while another may still read its shared memory
  asm volatile("barrier.cluster.arrive;\nbarrier.cluster.wait;" ::: "memory");
}

void chol_inv_upper(tnad_ctx* c, const double* G, int64_t p, double* Rinv, int* dev_fail, float near) {
  TNAD_REQUIRE(p >= 1 && p <= kCholMaxP, TNAD_ERR_SHAPE, "chol_inv_upper: p must be in [1,160]");
  constexpr size_t smem = (size_t)(2 * kCholPanels + 1) * kCholNB * kCholLd * sizeof(double);
  static PerDevice attr;
  if (!attr.has(c->device)) {
    TNAD_CK(cudaFuncSetAttribute(k_chol_inv, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    TNAD_CK(cudaFuncSetAttribute(k_chol_inv, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    attr.mark(c->device);
  }
  KernelTimer kt(c, "chol", (double)p * p * p / 3.0);
  cudaLaunchConfig_t cf = {};
  cf.gridDim = dim3(kCholC);
  cf.blockDim = dim3(256);
  cf.dynamicSmemBytes = smem;
  cf.stream = c->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kCholC;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cf.attrs = at;
  cf.numAttrs = 1;
  TNAD_CK(cudaLaunchKernelEx(&cf, k_chol_inv, G, (int)p, kPivotFloor, near, Rinv, dev_fail));
  count_launch(c);
  check_launch(c, "chol_inv");
}

// ---------------------------------------------------------------- Jacobi eigh
__device__ __forceinline__ void circle_pair(int r, int k, int NP, int* p, int* q) {
  if (k == 0) {
    *p = NP - 1;
    *q = r;
  } else {
    *p = (r + k) % (NP - 1);
    *q = (r - k + (NP - 1)) % (NP - 1);
  }
}

// A (p×p symmetric, FP64 in global) → lam (p, sorted by |λ| descending, or by λ
// descending when by_value), W (p×p eigenvectors as columns, same order).
// Z: p×p scratch for the unsorted vectors.  Sweeps until no rotation is needed
// (or max_sweeps; the sweep count goes to info[0]).
__global__ void k_eigh_jacobi(const double* __restrict__ A, int p, int max_sweeps, double* __restrict__ lam,
                              double* __restrict__ W, double* __restrict__ Z, int* __restrict__ info, int by_value) {
  extern __shared__ unsigned char smraw[];
  double* H = reinterpret_cast<double*>(smraw);  // p×p, leading dimension ld = p+1 (bank-conflict free)
  const int ld = p + 1;
  __shared__ double cs_[128], sn_[128];
  __shared__ int pp_[128], qq_[128];
  __shared__ int rotated;
  __shared__ double fro_part[32];
  const int NP = p + (p & 1);
  const double eps_t = DBL_EPSILON;
  const double tol = (double)(4.0 * eps_t * sqrt((double)p));
  double ss = 0.0;
  for (int e = threadIdx.x; e < p * p; e += blockDim.x) {
    const double v = A[e];
    ss += v * v;
    H[(e % p) + (e / p) * ld] = (double)v;
    Z[e] = (e % p == e / p) ? 1.0 : (double)0;
  }
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((threadIdx.x & 31) == 0) fro_part[threadIdx.x >> 5] = ss;
  __syncthreads();
  // Rounding floor of the stop rule: every rotation leaves noise of size
  // ~ε·‖H‖ in the off-diagonal entries of small eigenvalues, which a purely
  // relative rule would keep rotating until the sweep cap.
  double fro2 = 0.0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) fro2 += fro_part[w];
  const double absfl = (double)(2.0 * eps_t * sqrt((double)p) * sqrt(fro2));
  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    if (threadIdx.x == 0) rotated = 0;
    __syncthreads();
    for (int r = 0; r < NP - 1; ++r) {
      // rotation parameters for the NP/2 disjoint pairs of this round
      for (int k = threadIdx.x; k < NP / 2; k += blockDim.x) {
        int a, b;
        circle_pair(r, k, NP, &a, &b);
        double c = 1, s = 0;
        if (a < p && b < p) {
          if (a > b) {
            int t = a;
            a = b;
            b = t;
          }
          const double apq = H[a + b * ld], app = H[a + a * ld], aqq = H[b + b * ld];
          if (apq != (double)0 && fabs(apq) > tol * sqrt(fabs(app)) * sqrt(fabs(aqq)) && fabs(apq) > absfl) {
            const double tau = (aqq - app) / (2.0 * apq);
            const double t = (tau >= (double)0 ? 1.0 : -1.0) / (fabs(tau) + sqrt((double)1 + tau * tau));
            c = (double)1 / sqrt((double)1 + t * t);
            s = t * c;
            rotated = 1;
          }
        } else {
          a = b = -1;
        }
        pp_[k] = a;
        qq_[k] = b;
        cs_[k] = c;
        sn_[k] = s;
      }
      __syncthreads();
      // warp w takes pairs k ≡ w (mod warps), its lanes the matrix index (no
      // integer division in the inner loops)
      const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
      // rows: (row a, row b) ← (c·row a − s·row b, s·row a + c·row b)
      for (int k = wid; k < NP / 2; k += nwarp) {
        const int a = pp_[k], b = qq_[k];
        if (a < 0 || sn_[k] == (double)0) continue;
        const double c = cs_[k], s = sn_[k];
        for (int col = lane; col < p; col += 32) {
          const double x = H[a + col * ld], y = H[b + col * ld];
          H[a + col * ld] = c * x - s * y;
          H[b + col * ld] = s * x + c * y;
        }
      }
      __syncthreads();
      // columns of H and of Z; then the rotated pair's off-diagonal entry is 0
      for (int k = wid; k < NP / 2; k += nwarp) {
        const int a = pp_[k], b = qq_[k];
        if (a < 0 || sn_[k] == (double)0) continue;
        const double c = cs_[k], s = sn_[k];
        for (int row = lane; row < p; row += 32) {
          const double x = H[row + a * ld], y = H[row + b * ld];
          H[row + a * ld] = c * x - s * y;
          H[row + b * ld] = s * x + c * y;
          const double zx = Z[row + a * p], zy = Z[row + b * p];
          Z[row + a * p] = c * zx - s * zy;
          Z[row + b * p] = s * zx + c * zy;
        }
        __syncwarp();
        if (lane == 0) {
          H[a + b * ld] = (double)0;
          H[b + a * ld] = (double)0;
        }
      }
      __syncthreads();
    }
    const int done = (rotated == 0);
    __syncthreads();
    if (done) break;
  }
  // sort by key descending (ties by index): rank_j = #{i: k_i > k_j or (= and i<j)},
  // key |λ|, or λ itself when by_value
  for (int j = threadIdx.x; j < p; j += blockDim.x) {
    const double lj = (double)H[j + j * ld];
    const double kj = by_value ? lj : fabs(lj);
    int rk = 0;
    for (int i = 0; i < p; ++i) {
      const double li = (double)H[i + i * ld];
      const double ki = by_value ? li : fabs(li);
      rk += (ki > kj || (ki == kj && i < j)) ? 1 : 0;
    }
    lam[rk] = lj;
    for (int i = 0; i < p; ++i) W[i + (int64_t)rk * p] = (double)Z[i + (int64_t)j * p];
  }
  if (threadIdx.x == 0 && info) info[0] = sweep;
}

// The FP32 solve, one-sided: W = A·V and V in shared memory, the rotation of a
// pair from the 2×2 block of VᵀAV (a = v_p·w_p, b = v_q·w_q, g = (v_p·w_q +
// v_q·w_p)/2), so that ±λ pairs stay apart.  Columns in blocks of two, a block pair
// per 8 lanes and round of the circle method: its 4 columns come to registers by
// 16-byte shared loads, the cross pairs are rotated in two steps of two disjoint
// ones (in a sweep's first round the pairs inside the blocks before them) in packed
// FP32 (fma.rn.f32x2), and go back; one barrier a round.  With single columns W and
// V passed through shared memory once a rotation (128 bytes a clock: 1150 of a
// round's 1650 clocks at p = 96) and a sweep took p − 1 rounds (454 µs in the mean of a solve at p = 96, now 280);
// the two-sided form (k_eigh_jacobi), with three barriers and two passes, 758.
// Same stop rule.
__device__ __forceinline__ uint64_t pk2(float a, float b) {
  return ((uint64_t)__float_as_uint(b) << 32) | __float_as_uint(a);
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float hsum2(uint64_t a) {
  return __uint_as_float((unsigned)a) + __uint_as_float((unsigned)(a >> 32));
}

template <int RV>  // 16-byte row chunks per lane: ⌈p/32⌉
__global__ void __launch_bounds__(64 * RV, 1) k_eigh32(const double* __restrict__ A, int p, int max_sweeps,
                                                double* __restrict__ lam, double* __restrict__ Wout,
                                                int* __restrict__ info, int by_value) {
  extern __shared__ __align__(16) float esm[];
  const int pr = (p + 3) & ~3, cs = 2 * pr, q4 = pr >> 2;  // column: W rows, then V rows
  __shared__ float fro_part[10];
  __shared__ int rotated;
  __shared__ float lam_sh[kEigh32MaxP];
  const int nreal = (p + 1) >> 1, NB = nreal + (nreal & 1);  // blocks; columns from p on are zero
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l8 = lane & 7;
  float ss = 0.f;
  for (int e = threadIdx.x; e < 2 * NB * cs; e += blockDim.x) {
    const int i = e % cs, j = e / cs;
    float v = 0.f;
    if (i < pr) {
      v = i < p && j < p ? d2f_rn(A[i + (int64_t)j * p]) : 0.f;
      ss = fmaf(v, v, ss);
    } else if (j < p) {
      v = i - pr == j ? 1.f : 0.f;
    }
    esm[e] = v;
  }
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if (lane == 0) fro_part[warp] = ss;
  __syncthreads();
  float fro2 = 0.f;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) fro2 += fro_part[w];
  const float tol = 4.f * FLT_EPSILON * sqrtf((float)p);
  const float absfl = 2.f * FLT_EPSILON * sqrtf((float)p) * sqrtf(fro2);
  const int k = threadIdx.x >> 3;  // this lane group's block pair
  const bool on = k < (NB >> 1);
  ulonglong2 w[4][RV], v[4][RV];
  float f[4];  // v_i·w_i

  // rotate the pairs (i0, j0) and (i1, j1) of the four columns; true when one did
  auto step = [&](const int i0, const int j0, const int i1, const int j1) -> bool {
    uint64_t s0 = 0, s1 = 0;
#pragma unroll
    for (int e = 0; e < RV; ++e) {
      s0 = fma2(v[i0][e].x, w[j0][e].x, s0);
      s1 = fma2(v[i1][e].x, w[j1][e].x, s1);
      s0 = fma2(v[j0][e].x, w[i0][e].x, s0);
      s1 = fma2(v[j1][e].x, w[i1][e].x, s1);
      s0 = fma2(v[i0][e].y, w[j0][e].y, s0);
      s1 = fma2(v[i1][e].y, w[j1][e].y, s1);
      s0 = fma2(v[j0][e].y, w[i0][e].y, s0);
      s1 = fma2(v[j1][e].y, w[i1][e].y, s1);
    }
    float g[2] = {hsum2(s0), hsum2(s1)};  // 2g
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      g[0] += __shfl_xor_sync(0xffffffffu, g[0], o);
      g[1] += __shfl_xor_sync(0xffffffffu, g[1], o);
    }
    bool any = false;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = h ? i1 : i0, j = h ? j1 : j0;
      const float ag = 0.5f * fabsf(g[h]);
      if (ag > tol * fsqrt_ap(fabsf(f[i])) * fsqrt_ap(fabsf(f[j])) && ag > absfl) {
        const float t = jacobi_tan(f[j] - f[i], g[h]), tg = 0.5f * t * g[h];
        const float c = rsqrtf(fmaf(t, t, 1.f)), sn = c * t;
        const uint64_t c2 = pk2(c, c), s2 = pk2(sn, sn), n2 = pk2(-sn, -sn);
        f[i] -= tg;
        f[j] += tg;
#pragma unroll
        for (int e = 0; e < RV; ++e) {
          const ulonglong2 wi = w[i][e], wj = w[j][e], vi = v[i][e], vj = v[j][e];
          w[i][e] = make_ulonglong2(fma2(c2, wi.x, mul2(n2, wj.x)), fma2(c2, wi.y, mul2(n2, wj.y)));
          w[j][e] = make_ulonglong2(fma2(c2, wj.x, mul2(s2, wi.x)), fma2(c2, wj.y, mul2(s2, wi.y)));
          v[i][e] = make_ulonglong2(fma2(c2, vi.x, mul2(n2, vj.x)), fma2(c2, vi.y, mul2(n2, vj.y)));
          v[j][e] = make_ulonglong2(fma2(c2, vj.x, mul2(s2, vi.x)), fma2(c2, vj.y, mul2(s2, vi.y)));
        }
        any = true;
      }
    }
    return any;
  };

  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    if (threadIdx.x == 0) rotated = 0;
    __syncthreads();
    for (int r = 0; r < NB - 1; ++r) {
      int P = r, Q = NB - 1;
      if (k > 0) {
        P = r + k < NB - 1 ? r + k : r + k - (NB - 1);
        Q = r >= k ? r - k : r - k + NB - 1;
      }
      if (P > Q) {
        const int t = P;
        P = Q;
        Q = t;
      }
      ulonglong2* cp = reinterpret_cast<ulonglong2*>(esm + (on ? 2 * P : 0) * cs);
      ulonglong2* cq = reinterpret_cast<ulonglong2*>(esm + (on ? 2 * Q : 0) * cs);
      const int c4 = cs >> 2;
      const ulonglong2 z = make_ulonglong2(0, 0);
      uint64_t sd[4] = {0, 0, 0, 0};
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const ulonglong2* x = (l < 2 ? cp : cq) + (l & 1) * c4;
#pragma unroll
        for (int e = 0; e < RV; ++e) {
          const int i = l8 + 8 * e;
          const bool in = on && i < q4;
          w[l][e] = in ? x[i] : z;
          v[l][e] = in ? x[q4 + i] : z;
        }
      }
#pragma unroll
      for (int e = 0; e < RV; ++e)
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          sd[l] = fma2(v[l][e].x, w[l][e].x, sd[l]);
          sd[l] = fma2(v[l][e].y, w[l][e].y, sd[l]);
        }
#pragma unroll
      for (int l = 0; l < 4; ++l) f[l] = hsum2(sd[l]);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int l = 0; l < 4; ++l) f[l] += __shfl_xor_sync(0xffffffffu, f[l], o);
      bool any = false;
      if (r == 0) any = step(0, 1, 2, 3);
      any |= step(0, 2, 1, 3);
      any |= step(0, 3, 1, 2);
      if (any) {
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          ulonglong2* x = (l < 2 ? cp : cq) + (l & 1) * c4;
#pragma unroll
          for (int e = 0; e < RV; ++e) {
            const int i = l8 + 8 * e;
            if (i < q4) {
              x[i] = w[l][e];
              x[q4 + i] = v[l][e];
            }
          }
        }
        if (l8 == 0) rotated = 1;
      }
      __syncthreads();
    }
    const int done = (rotated == 0);
    __syncthreads();
    if (done) break;
  }
  // λ_j = v_j·w_j, columns sorted descending by |λ| (or λ), ties by index
  const int nw = blockDim.x >> 5;
  for (int j = warp; j < p; j += nw) {
    float s = 0.f;
    for (int i = lane; i < p; i += 32) s = fmaf(esm[j * cs + i], esm[j * cs + pr + i], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) lam_sh[j] = s;
  }
  __syncthreads();
  for (int j = warp; j < p; j += nw) {
    const float lj = lam_sh[j], kj = by_value ? lj : fabsf(lj);
    int rk = 0;
    for (int i = lane; i < p; i += 32) {
      const float ki = by_value ? lam_sh[i] : fabsf(lam_sh[i]);
      rk += (ki > kj || (ki == kj && i < j)) ? 1 : 0;
    }
    for (int o = 16; o > 0; o >>= 1) rk += __shfl_xor_sync(0xffffffffu, rk, o);
    if (lane == 0) lam[rk] = (double)lj;
    for (int i = lane; i < p; i += 32) Wout[i + (int64_t)rk * p] = f2d_any(esm[j * cs + pr + i]);
  }
  if (threadIdx.x == 0 && info) info[0] = sweep;
}

template <int RV>
void eigh32_launch(tnad_ctx* c, const double* A, int p, int max_sweeps, double* lam, double* W, int* info, int by_value) {
  static PerDevice attr;
  if (!attr.has(c->device)) {
    TNAD_CK(cudaFuncSetAttribute(k_eigh32<RV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 2 * kEigh32MaxP * kEigh32MaxP * 4));
    attr.mark(c->device);
  }
  const int pr = (p + 3) & ~3, nreal = (p + 1) / 2, NB = nreal + (nreal & 1);
  k_eigh32<RV><<<1, (4 * NB + 31) / 32 * 32, (size_t)2 * NB * 2 * pr * sizeof(float), c->stream>>>(
      A, p, max_sweeps, lam, W, info, by_value);
}

void eigh_small_prec(tnad_ctx* c, bool fp32, const double* A, int64_t p, double* W, double* lam, int max_sweeps,
                     int* dev_info, bool by_value) {
  TNAD_REQUIRE(p >= 1 && p <= (fp32 ? kEigh32MaxP : 256), TNAD_ERR_SHAPE,
               "eigh_small: p must be in [1,256] (FP32: [1,160])");
  KernelTimer kt(c, fp32 ? "eigh_f32" : "eigh_f64", 0.0);
  if (fp32) {
    const int bv = by_value ? 1 : 0;
    if (p <= 32)
      eigh32_launch<1>(c, A, (int)p, max_sweeps, lam, W, dev_info, bv);
    else if (p <= 64)
      eigh32_launch<2>(c, A, (int)p, max_sweeps, lam, W, dev_info, bv);
    else if (p <= 96)
      eigh32_launch<3>(c, A, (int)p, max_sweeps, lam, W, dev_info, bv);
    else if (p <= 128)
      eigh32_launch<4>(c, A, (int)p, max_sweeps, lam, W, dev_info, bv);
    else
      eigh32_launch<5>(c, A, (int)p, max_sweeps, lam, W, dev_info, bv);
  } else {
    WsScope scope(c);
    const size_t sm = (size_t)(p + 1) * p * 8;
    const size_t kMaxSm = 200 * 1024;
    TNAD_REQUIRE(sm <= kMaxSm, TNAD_ERR_SHAPE, "eigh_small: matrix does not fit in shared memory");
    static PerDevice attr64;
    if (!attr64.has(c->device)) {
      TNAD_CK(cudaFuncSetAttribute(k_eigh_jacobi, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSm));
      attr64.mark(c->device);
    }
    // eigenvectors accumulate in global memory (L1-cached); H lives in shared memory
    double* Z = ws_d(c, p * p);
    k_eigh_jacobi<<<1, 512, sm, c->stream>>>(A, (int)p, max_sweeps, lam, W, Z, dev_info, by_value ? 1 : 0);
  }
  count_launch(c);
  check_launch(c, "eigh_small");
}

void eigh_small(tnad_ctx* c, const double* A, int64_t p, double* W, double* lam) {
  eigh_small_prec(c, false, A, p, W, lam, 40, nullptr);
}

// ---------------------------------------------------------------- polar factor
// O = polar(X) for a χ×χ X (χ ≤ 128) by Newton–Schulz, O ← O·(3I − OᵀO)/2,
// in FP32 in one CTA (the caller polishes in FP64); larger χ take polar_ns_gemm.  info[0] = 1 when the
// result is orthogonal to 1e-4 (else the caller falls back to sign alignment).
//
// Each thread owns a 4×4 tile of the product (⌈m/4⌉² ≤ 1024 threads): two 16-byte
// shared loads per 16 multiply-adds.  That needs the iterate in both layouts
// (rows and columns contiguous) and uses that AᵀA is symmetric bit for bit; the
// next iterate waits in registers until every tile has read the old one;
// bound by the shared loads: 132 µs for m = 64 and 24 iterations (2×2 tiles with
// 4-byte loads: 335 µs), the same sums in the same order.
__global__ void __launch_bounds__(1024) k_polar_ns(const double* __restrict__ X, int m, int iters,
                                                   double* __restrict__ O, int* __restrict__ info) {
  extern __shared__ __align__(16) float psm[];
  const int nt = (m + 3) >> 2, ld = 4 * nt + 4;  // 16-byte columns, one float4 of padding
  float* A = psm;                                // A(i, k) at i + k·ld
  float* At = psm + 4 * nt * ld;                 // A(k, i) at i + k·ld
  float* G = psm + 8 * nt * ld;                  // AᵀA, symmetric
  __shared__ float red[32];
  const int mm = m * m;
  // scale by 1/‖X‖_F·√m so that all singular values are ≤ 1 < √3
  float s = 0.f;
  for (int e = threadIdx.x; e < mm; e += blockDim.x) s += (float)(X[e] * X[e]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    red[0] = t > 0.f ? sqrtf((float)m / t) : 1.f;
  }
  __syncthreads();
  const float sc = red[0] > 1.f ? fminf(red[0], 1.0f) * 0.999f : 1.0f;
  for (int e = threadIdx.x; e < 16 * nt * nt; e += blockDim.x) {
    const int i = e % (4 * nt), k = e / (4 * nt);
    const float v = (i < m && k < m) ? (float)X[i + k * m] * sc : 0.f;
    A[i + k * ld] = v;
    At[k + i * ld] = v;
  }
  __syncthreads();
  const bool act = (int)threadIdx.x < nt * nt;
  const int i0 = 4 * ((int)threadIdx.x % nt), j0 = 4 * ((int)threadIdx.x / nt);
  float worst = 0.f;
  for (int it = 0; it <= iters; ++it) {
    // G = AᵀA, and how far it is from I
    float g[4][4];
    float dev = 0.f;
    if (act) {
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) g[a][b] = 0.f;
#pragma unroll 4
      for (int k = 0; k < 4 * nt; ++k) {  // rows beyond m are zero
        const float4 x = *reinterpret_cast<const float4*>(&At[i0 + k * ld]);
        const float4 y = *reinterpret_cast<const float4*>(&At[j0 + k * ld]);
        const float xa[4] = {x.x, x.y, x.z, x.w}, ya[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) g[a][b] = fmaf(xa[a], ya[b], g[a][b]);
      }
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        *reinterpret_cast<float4*>(&G[i0 + (j0 + b) * ld]) = make_float4(g[0][b], g[1][b], g[2][b], g[3][b]);
#pragma unroll
        for (int a = 0; a < 4; ++a)
          if (i0 + a < m && j0 + b < m) dev = fmaxf(dev, fabsf(g[a][b] - (i0 + a == j0 + b ? 1.f : 0.f)));
      }
    }
    for (int o = 16; o > 0; o >>= 1) dev = fmaxf(dev, __shfl_xor_sync(0xffffffffu, dev, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = dev;
    __syncthreads();
    // all iterations run: stopping once AᵀA is at FP32 rounding (and polishing
    // in FP64) changed the converged gauge enough to make the fixed-point
    // adjoint's GMRES several times slower
    if (it == iters) {
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) worst = fmaxf(worst, red[w]);
      break;
    }
    // A ← A·(1.5 I − 0.5 G)
    float v[4][4];
    if (act) {
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) g[a][b] = 0.f;
#pragma unroll 4
      for (int k = 0; k < 4 * nt; ++k) {
        const float4 x = *reinterpret_cast<const float4*>(&A[i0 + k * ld]);
        const float4 y = *reinterpret_cast<const float4*>(&G[j0 + k * ld]);  // G(k, j) = G(j, k)
        const float xa[4] = {x.x, x.y, x.z, x.w}, ya[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) g[a][b] = fmaf(xa[a], ya[b], g[a][b]);
      }
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const float4 x = *reinterpret_cast<const float4*>(&A[i0 + (j0 + b) * ld]);
        v[0][b] = 1.5f * x.x - 0.5f * g[0][b];
        v[1][b] = 1.5f * x.y - 0.5f * g[1][b];
        v[2][b] = 1.5f * x.z - 0.5f * g[2][b];
        v[3][b] = 1.5f * x.w - 0.5f * g[3][b];
      }
    }
    __syncthreads();
    if (act) {
#pragma unroll
      for (int b = 0; b < 4; ++b)
        *reinterpret_cast<float4*>(&A[i0 + (j0 + b) * ld]) = make_float4(v[0][b], v[1][b], v[2][b], v[3][b]);
#pragma unroll
      for (int a = 0; a < 4; ++a)
        *reinterpret_cast<float4*>(&At[j0 + (i0 + a) * ld]) = make_float4(v[a][0], v[a][1], v[a][2], v[a][3]);
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < mm; e += blockDim.x) O[e] = (double)A[(e % m) + (e / m) * ld];
  if (threadIdx.x == 0) info[0] = worst < 1e-4f ? 1 : 0;
}

// info[0] = 1 when max |G − I| < 1e-4 for the m×m matrix G = OᵀO (one CTA)
__global__ void k_orth_info(const double* __restrict__ G, int64_t m, int* __restrict__ info) {
  __shared__ double red[32];
  double dev = 0.0;
  for (int64_t e = threadIdx.x; e < m * m; e += blockDim.x)
    dev = fmax(dev, fabs(G[e] - ((e % m) == (e / m) ? 1.0 : 0.0)));
  for (int o = 16; o > 0; o >>= 1) dev = fmax(dev, __shfl_xor_sync(0xffffffffu, dev, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = dev;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t = fmax(t, red[w]);
    info[0] = t < 1e-4 ? 1 : 0;
  }
}

// Polar factor for m > 128 (beyond one CTA's shared memory): the same
// Newton–Schulz iteration O ← O·(3I − OᵀO)/2 from O = 0.999·X (X is a product of
// two orthonormal bases, so its singular values are ≤ 1), with its products on
// the multi-CTA GEMMs (TF32X3 where the tensor cores are available; the caller
// polishes in FP64), and the same orthogonality flag.
static void polar_ns_gemm(tnad_ctx* c, const double* X, int64_t m, int iters, double* O, int* dev_info) {
  WsScope scope(c);
  double* G = ws_d(c, m * m);
  double* O2 = ws_d(c, m * m);
  const int pr = c->tc_ok ? TNAD_PREC_TF32X3 : TNAD_PREC_FP64;
  copy_d2d(c, O, X, m * m);
  scale(c, m * m, 0.999, O);
  for (int it = 0; it < iters; ++it) {
    gemm(c, pr, 'T', 'N', m, m, m, 1.0, O, m, O, m, 0.0, G, m);
    copy_d2d(c, O2, O, m * m);
    gemm(c, pr, 'N', 'N', m, m, m, -0.5, O, m, G, m, 1.5, O2, m);
    copy_d2d(c, O, O2, m * m);
  }
  gemm(c, pr, 'T', 'N', m, m, m, 1.0, O, m, O, m, 0.0, G, m);
  k_orth_info<<<1, 1024, 0, c->stream>>>(G, m, dev_info);
  count_launch(c);
  check_launch(c, "polar_ns_gemm");
}

void polar_ns(tnad_ctx* c, const double* X, int64_t m, int iters, double* O, int* dev_info) {
  TNAD_REQUIRE(m >= 1, TNAD_ERR_SHAPE, "polar_ns: m must be >= 1");
  if (m > 128) {
    polar_ns_gemm(c, X, m, iters, O, dev_info);
    return;
  }
  static PerDevice attr;
  if (!attr.has(c->device)) {
    TNAD_CK(cudaFuncSetAttribute(k_polar_ns, cudaFuncAttributeMaxDynamicSharedMemorySize, 3 * 128 * 132 * 4));
    attr.mark(c->device);
  }
  KernelTimer kt(c, "polar_ns", 0.0);
  const int nt = ((int)m + 3) / 4;
  k_polar_ns<<<1, (nt * nt + 31) / 32 * 32, (size_t)3 * 4 * nt * (4 * nt + 4) * 4, c->stream>>>(X, (int)m, iters, O,
                                                                                                 dev_info);
  count_launch(c);
  check_launch(c, "polar_ns");
}

// ---------------------------------------------------------------- Gaussian fill
__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x ^= x >> 30;
  x *= 0xbf58476d1ce4e5b9ull;
  x ^= x >> 27;
  x *= 0x94d049bb133111ebull;
  x ^= x >> 31;
  return x;
}

// x[i] = scale·N(0,1) sample from a counter-based hash (SplitMix64 finaliser + Box–Muller)
// With sumsq != null the scale is relative to the RMS of the existing entries
// (scale·√(Σx²/n)), read on the device so that no host synchronisation is needed.
__global__ void k_randn(double* __restrict__ x, int64_t n, uint64_t seed, double scale, int accumulate,
                        const double* __restrict__ sumsq) {
  if (sumsq) {
    const double ms = sumsq[0] / (double)n;
    scale *= ms > 0.0 ? sqrt(ms) : 1.0;
  }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t h1 = mix64(seed * 0x9e3779b97f4a7c15ull + 2 * (uint64_t)i + 1);
    const uint64_t h2 = mix64(h1 ^ 0xd6e8feb86659fd93ull);
    const double u1 = ((double)(h1 >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    const double u2 = (double)(h2 >> 11) * (1.0 / 9007199254740992.0);
    const double g = sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
    x[i] = accumulate ? x[i] + scale * g : scale * g;
  }
}

void randn(tnad_ctx* c, double* x, int64_t n, uint64_t seed, double scale, bool accumulate,
           const double* dev_sumsq) {
  int nb = (int)std::min<int64_t>((n + 255) / 256, 4096);
  k_randn<<<nb, 256, 0, c->stream>>>(x, n, seed, scale, accumulate ? 1 : 0, dev_sumsq);
  count_launch(c);
  check_launch(c, "randn");
}

}  // namespace tnad
