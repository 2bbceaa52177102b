// FP64 SVD at LAPACK-level accuracy (every triplet to ε·‖A‖) of matrices up to
// 1024 rows: rank-revealing QR, then one-sided Jacobi on the triangular factor
// (Drmač and Veselić, "New fast and accurate Jacobi SVD algorithm", SIAM J.
// Matrix Anal. Appl. 29, 2008).  It serves the decompositions of src/trg.jl:36
// and src/ctmrg.jl:136 that the product refinement (eig_refine.cu) does not.
//
//   A·P = Q·R          Householder QR with column pivoting, stopped at rank r
//                      once every remaining column is below ½ε of the first
//                      pivot (what is dropped is below the rounding of A)
//   Rᵀ·P₂ = Q₂·R₂      a second one (general A, or r < n), r×r
//   X·Vx = Wn·Σ        one-sided Jacobi, X = R₂ᵀ (or Rᵀ without the second QR)
//
// so that A = (Q·P₂·Wn)·Σ·(P·Q₂·Vx)ᵀ, completed by the trailing columns of Q
// and P·Q₂ where r < n.  Symmetric A with r = n skips the second QR and the
// accumulation of Vx: the singular vectors are P·Wn, and k_svd_sym_basis makes
// eigenvectors of them.
//
// Why: GB300 issues one FP64 instruction per warp and SM quadrant every 64
// clocks (76 with all four busy), so the sweeps are paid in instructions and in
// rounds.  The corners and TRG splits are graded (singular values from 1 to
// 1e-16): plain Jacobi sweeps took 9-36 of them there, on the triangular factor
// it is 6-10, and the rank cut leaves ~250 of 400 columns of a χ = 20 split.
// Each factorisation and each kind of sweep is one launch (one instead of n − 1 per
// sweep), cooperative, or a cluster where n is small.  From kPreMin columns on the
// FP32 sweeps are followed by a host wait (the rank sizes what comes next), two
// corrections of V as products, and W = X·V.
// Measured on one GB300 against FP64 element rounds (k_jacobi_round_cta): TRG at
// χ = 20, 7 steps with gradient 718 → 24 ms; D=3, χ=36 energy and gradient (n =
// 324) 366 → 48 ms; one n = 80 decomposition 4.9 → 1.1 ms, n = 255 26.7 → 4.5 ms.
// At n = 324 the first QR takes 1.5 ms, the FP32 sweeps 2.0, the FP64 ones 2.4.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "fp64_fast.cuh"
#include "per_device.h"
#include "sweep_rule.h"
#include "tc_common.cuh"
#include "tnad_internal.h"

namespace tnad {

namespace {

constexpr int kMaxSvdRows = 1024;
constexpr int kSvdSweeps = 60;
constexpr int kPreMin = 24;         // columns from which FP32 sweeps precede the FP64 ones
constexpr int kPreSweeps = 20;
constexpr int kEigSweeps = 30;      // cap of the corner's FP32 sweeps (their result is refined or replaced)
constexpr float kPreCos = 1e-3f;    // a sweep that rotated no larger |cos| leaves ~1e-6: hand over
constexpr int kQrCl = 16;           // CTAs of a QR's cluster, at most
constexpr int kScaleExp = 40;  // the largest |entry| is scaled to 2^40: squared norms of
                               // columns down to ½ε of it stay inside the FP32 range

// Per-problem counters (ints): rank, non-finite input, converged sweep count
// (0: none), scale, error, FP32 sweeps, multiplets to separate, barrier counter of each of the three kernels, rotations per sweep
// and the largest |cos| of a rotated pair per sweep (float bits).
enum { kiRank = 0, kiBad = 1, kiSweeps = 2, kiExp = 3, kiErr = 4, kiPre = 5, kiMulti = 6, kiBar = 8, kiRot = 16, kiCos = 16 + kSvdSweeps,
       kiTan = 16 + 2 * kSvdSweeps, kiRot32 = 16 + 3 * kSvdSweeps, kiCos32 = kiRot32 + kEigSweeps, kiCount = kiCos32 + kEigSweeps };

struct SvdProb {
  const double* A;
  double *X, *X2, *Vx;    // Rᵀ (n×n), R₂ᵀ and the accumulated rotations; leading dimension ldx
  double *H, *H2;         // Householder vectors of the two factorisations, n×n
  double *hinv, *hinv2;   // 2/vᵀv of each
  int *perm, *perm2;      // perm[k]: column at pivot position k
  double *cand;           // 2 × G × ldc candidate columns, each entry with its tag
  unsigned long long* key;  // 2 × G candidate keys, and G column maxima
  float *W32, *V32;       // FP32 copies of X and of the rotations; leading dimension ld32
  double *W, *Wbuf;       // X·V after the FP32 sweeps (W null: none)
  double *nrm, *sv;       // squared column norms, singular values (unsorted)
  double *U, *S, *V;
  int* info;
};

struct SvdArgs {
  SvdProb p[2];
  int n, ldx, ldc, ld32;
  int second;      // run the second QR also when r = n
  float trunc;     // rank cut relative to the first pivot
  double tol;      // Jacobi: |cos| above which a pair rotates (FP64 and FP32 sweeps)
  float tol32;
  const double* fro2;  // EIG: ‖A‖²_F
  int max_sweeps;
};

__device__ __forceinline__ double wsum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Both sums with the additions of one: the half-warps take one value each
__device__ __forceinline__ void wsum2_d(double& a, double& b) {
  const bool up = (threadIdx.x & 16) != 0;
  const double give = up ? a : b;
  double v = (up ? b : a) + __shfl_xor_sync(0xffffffffu, give, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  a = __shfl_sync(0xffffffffu, v, 0);
  b = __shfl_sync(0xffffffffu, v, 16);
}

__device__ __forceinline__ float wsum_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Barrier over the CTAs of one problem.  CL: they form one thread-block cluster
// (hardware barrier, 0.24 µs).  Otherwise a counter in global memory (1.1 µs
// for 16 to 152 CTAs): the wait is bounded (2 s of %globaltimer); a CTA that
// gives up sets *err, which the others see, and all of them return.
template <bool CL>
struct GridBar {
  unsigned* cnt;
  unsigned tgt, G;
  int* err;
  int* dead;  // shared: 1 once a wait gave up
  __device__ bool sync() {
    if (CL) {
      asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
      return true;
    }
    __syncthreads();
    tgt += G;
    if (threadIdx.x == 0) {
      // release and acquire at GPU scope; the CTA barriers around them order the
      // other threads' accesses
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(cnt) : "memory");
      unsigned v, spins = 0;
      const uint64_t t0 = tc::gtime();
      while (true) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(cnt) : "memory");
        if ((int)(v - tgt) >= 0) break;
        if ((++spins & 255u) == 0 && (tc::gtime() - t0 > 2000000000ull || atomicAdd(err, 0) != 0)) {
          atomicExch(err, 1);
          *dead = 1;
          break;
        }
      }
    }
    __syncthreads();
    return *dead == 0;
  }
};

// A value and its step's tag as one 16-byte access: whoever reads the tag has
// the value, without a fence on either side
__device__ __forceinline__ void st_tagged(void* p, double v, unsigned long long tag) {
  asm volatile("{.reg .b128 t;\nmov.b128 t, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], t;}" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ double ld_tagged(const void* p, unsigned long long* tag) {
  long long v;
  asm volatile("{.reg .b128 t;\nld.relaxed.gpu.global.b128 t, [%2];\nmov.b128 {%0, %1}, t;}"
               : "=l"(v), "=l"(*tag)
               : "l"(p)
               : "memory");
  return __longlong_as_double(v);
}

// Bounded spin: false once 2 s have passed or another CTA gave up (*err)
struct SpinLimit {
  unsigned n = 0;
  uint64_t t0 = 0;
  __device__ bool more(int* err) {
    if ((++n & 255u) != 0) return true;
    if (t0 == 0) t0 = tc::gtime();
    if (tc::gtime() - t0 > 2000000000ull || atomicAdd(err, 0) != 0) {
      atomicExch(err, 1);
      return false;
    }
    return true;
  }
};

// ---------------------------------------------------------------------------
// Householder QR with column pivoting.  One warp per column, the column in
// registers (R chunks of 32 rows); CTA b holds the columns b, b + G, b + 2G...
// Step k: every CTA publishes its longest remaining column with a key (norm,
// column); every warp finds the longest of all (ties: smallest index), reads that
// column, forms its Householder vector (the same arithmetic in every warp) and
// updates its own column.  The norms that only choose pivots are FP32 sums of
// squares.  A step is a chain of latencies, so
//   - across SMs keys and column entries carry the step's number and are polled
//     where they lie: no counter barrier, no fence and no read of the keys after
//     them; a CTA reads the column once, for all its warps (read by every warp, 456
//     requests queue on each of its lines);
//   - in a cluster (up to 64 columns) keys and columns are stored into every CTA's
//     shared memory before the barrier;
//   - ‖x‖² and xᵀc are summed in one pass over registers and shuffles (vᵀc =
//     xᵀc − β·c_k needs no v).
// Two buffers by parity: a CTA is at most one step ahead of the slowest.
// STAGE 0: A (n×n, scaled by a power of two) → H, hinv, perm, rank, X = Rᵀ in
// pivot order.  STAGE 1: the r columns of X → H2, hinv2, perm2, X2 = R₂ᵀ.
// ---------------------------------------------------------------------------
template <int R, bool CL, int STAGE>
__global__ void __launch_bounds__(256) k_qrcp(SvdArgs a) {
  const SvdProb& q = a.p[blockIdx.y];
  const int G = gridDim.x, cta = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  int m, n;
  if (STAGE == 0) {
    m = n = a.n;
  } else {
    m = a.n;
    n = q.info[kiRank];
    if (q.info[kiErr] || n == 0 || (!a.second && n == a.n)) return;  // uniform over the problem's CTAs
  }
  double* H = STAGE == 0 ? q.H : q.H2;
  double* hinv = STAGE == 0 ? q.hinv : q.hinv2;
  int* perm = STAGE == 0 ? q.perm : q.perm2;
  double* X = STAGE == 0 ? q.X : q.X2;
  __shared__ unsigned long long wkey[8], rkey[8], ckey[CL ? 2 : 1][CL ? kQrCl : 1];
  __shared__ double xs[CL ? 1 : 32 * R];  // the step's column
  __shared__ double ccol[CL ? 2 : 1][CL ? kQrCl : 1][CL ? 32 * R : 1];  // CL: candidate columns of every CTA
  __shared__ unsigned picked_mask[kMaxSvdRows / 32];
  __shared__ int dead;
  if (threadIdx.x == 0) dead = 0;
  for (int i = threadIdx.x; i < kMaxSvdRows / 32; i += blockDim.x) picked_mask[i] = 0u;
  __syncthreads();
  GridBar<CL> bar{reinterpret_cast<unsigned*>(q.info + kiBar + STAGE), 0u, (unsigned)G, q.info + kiErr, &dead};

  const int col = warp * G + cta;
  const bool have = col < n;
  double c[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = lane + 32 * i;
    c[i] = (have && row < m) ? (STAGE == 0 ? q.A[row + (int64_t)col * m] : __ldcg(&q.X[row + (int64_t)col * a.ldx]))
                             : 0.0;
  }
  if (STAGE == 0) {
    // scale so that the largest |entry| lies in [2^40, 2^41): exact, undone on S
    unsigned long long mx = 0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const unsigned long long b = (unsigned long long)__double_as_longlong(fabs(c[i]));
      mx = b > mx ? b : mx;  // NaN and infinities order above every finite value
    }
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long b = __shfl_xor_sync(0xffffffffu, mx, o);
      mx = b > mx ? b : mx;
    }
    if (lane == 0) wkey[warp] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < nwarp; ++w) mx = wkey[w] > mx ? wkey[w] : mx;
      __stcg(&q.key[2 * G + cta], mx);
    }
    if (!bar.sync()) return;
    mx = 0;
    for (int g = lane; g < G; g += 32) {
      const unsigned long long b = __ldcg(&q.key[2 * G + g]);
      mx = b > mx ? b : mx;
    }
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long b = __shfl_xor_sync(0xffffffffu, mx, o);
      mx = b > mx ? b : mx;
    }
    const double amax = __longlong_as_double((long long)mx);
    if (!(amax > 0.0) || !isfinite(amax)) {  // zero or non-finite A (uniform)
      if (cta == 0 && threadIdx.x == 0) {
        q.info[kiRank] = 0;
        q.info[kiBad] = amax == 0.0 ? 0 : 1;
      }
      for (int j = cta * blockDim.x + threadIdx.x; j < n; j += G * blockDim.x) perm[j] = j;
      return;
    }
    const int e = ilogb(amax) - kScaleExp;
#pragma unroll
    for (int i = 0; i < R; ++i) c[i] = scalbn(c[i], -e);
    if (cta == 0 && threadIdx.x == 0) q.info[kiExp] = e;
  }
  float nr = 0.f;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const float f = d2f(c[i]);
    nr = fmaf(f, f, nr);
  }
  nr = wsum_f(nr);
  int pos = -1;
  float thr2 = 0.f;
  const int kmax = min(m, n);
  int k = 0;
  for (; k < kmax; ++k) {
    // this CTA's longest remaining column: (norm, 1024 − column, step)
    const int buf = k & 1;
    const unsigned tag = (unsigned)(STAGE * 2048 + k + 1);
    const bool live = have && pos < 0;
    const unsigned long long mykey =
        live ? (((unsigned long long)__float_as_uint(nr) << 32) | ((unsigned)(kMaxSvdRows - col) << 21) | tag) : tag;
    if (lane == 0) wkey[warp] = mykey;
    __syncthreads();
    unsigned long long best = wkey[0];
    int bw = 0;
    for (int w = 1; w < nwarp; ++w)
      if (wkey[w] > best) {
        best = wkey[w];
        bw = w;
      }
    double* mine = q.cand + 2 * ((int64_t)buf * G + cta) * a.ldc;
    if (warp == bw) {
      if (CL ? lane < G : lane == 0) {
        if (CL) {
          uint32_t ra;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                       : "=r"(ra)
                       : "r"((uint32_t)__cvta_generic_to_shared(&ckey[buf][cta])), "r"(lane));
          asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(ra), "l"(best) : "memory");
        } else {
          asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&q.key[buf * G + cta]), "l"(best) : "memory");
        }
      }
      if (CL) {
        const uint32_t la = (uint32_t)__cvta_generic_to_shared(&ccol[buf][cta][0]);
        for (int g = 0; g < G; ++g) {
          uint32_t ra;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(la), "r"(g));
#pragma unroll
          for (int i = 0; i < R; ++i)
            if (32 * i < m && 32 * i + 31 >= k)
              asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra + 8u * (lane + 32 * i)), "d"(c[i]) : "memory");
        }
      } else if (live) {
#pragma unroll
        for (int i = 0; i < R; ++i)
          if (32 * i + 31 >= k && lane + 32 * i < m) st_tagged(&mine[2 * (lane + 32 * i)], c[i], tag);
      }
    }
    if (CL) {
      bar.sync();
      best = lane < G ? ckey[buf][lane] : 0ull;
    } else {
      best = 0;
      SpinLimit spin;
      for (int g0 = threadIdx.x; g0 < G; g0 += 5 * (int)blockDim.x) {
        while (true) {  // the loads of one pass do not wait for one another
          unsigned long long b[5];
#pragma unroll
          for (int u = 0; u < 5; ++u) {
            const int g = g0 + u * (int)blockDim.x;
            b[u] = tag;
            if (g < G) asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(b[u]) : "l"(&q.key[buf * G + g]) : "memory");
          }
          bool all = true;
#pragma unroll
          for (int u = 0; u < 5; ++u) {
            all = all && ((unsigned)b[u] & 0x1fffffu) == tag;
            best = b[u] > best ? b[u] : best;
          }
          if (all) break;
          best = 0;
          if (!spin.more(q.info + kiErr)) {
            dead = 1;
            break;
          }
        }
      }
    }
    {  // the largest of the warp: its norm, then the column among equal norms
      const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(best >> 32));
      const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(best >> 32) == hi ? (unsigned)best : 0u);
      best = ((unsigned long long)hi << 32) | lo;
    }
    if (!CL) {
      if (lane == 0) rkey[warp] = best;
      __syncthreads();
      if (dead) return;
      for (int w = 0; w < nwarp; ++w) best = rkey[w] > best ? rkey[w] : best;
    }
    const float n2 = __uint_as_float((unsigned)(best >> 32));
    const int wj = kMaxSvdRows - (int)((unsigned)best >> 21);
    if (STAGE == 0) {
      if (k == 0) thr2 = a.trunc * a.trunc * n2;
      if (n2 <= thr2) break;  // the rest is below the rounding of A
    }
    if (threadIdx.x == 0) picked_mask[wj >> 5] |= 1u << (wj & 31);
    if (!CL) {
      const double* win = q.cand + 2 * ((int64_t)buf * G + (wj % G)) * a.ldc;
      SpinLimit spin;
      for (int row0 = (k & ~31) + threadIdx.x; row0 < m; row0 += 4 * blockDim.x) {
        double v[4];
        while (true) {  // four loads in flight
          unsigned long long t[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int row = row0 + u * (int)blockDim.x;
            t[u] = tag;
            if (row < m) v[u] = ld_tagged(&win[2 * row], &t[u]);
          }
          if (t[0] == tag && t[1] == tag && t[2] == tag && t[3] == tag) break;
          if (!spin.more(q.info + kiErr)) {
            dead = 1;
            break;
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (row0 + u * (int)blockDim.x < m) xs[row0 + u * (int)blockDim.x] = v[u];
      }
      __syncthreads();
      if (dead) return;
    }
    if (!live && !(cta == 0 && warp == 0)) continue;  // nothing left to update
    const double* wsh = CL ? &ccol[CL ? buf : 0][CL ? wj % G : 0][0] : xs;
    double x[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = lane + 32 * i;
      x[i] = (32 * i + 31 >= k && row >= k && row < m) ? wsh[row] : 0.0;
    }
    // v = x − β·e_k, β = −sign(α)·‖x‖, H = I − hk·v·vᵀ with hk = 2/vᵀv = 1/(‖x‖² + |α|‖x‖)
    double s2 = 0.0, d = 0.0, s2b = 0.0, db = 0.0, al = 0.0, ck = 0.0;
#pragma unroll
    for (int i = 0; i < R; i += 2) {
      if (32 * i < m && 32 * i + 63 >= k) {  // (x is 0 outside the rows k..m)
        s2 = fma(x[i], x[i], s2);
        d = fma(x[i], c[i], d);
        s2b = fma(x[i + 1], x[i + 1], s2b);
        db = fma(x[i + 1], c[i + 1], db);
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (lane + 32 * i == k) {  // (by i == k / 32 the arrays would be indexed in local memory)
        al = x[i];
        ck = c[i];
      }
    }
    s2 += s2b;
    d += db;
    wsum2_d(s2, d);
    al = __shfl_sync(0xffffffffu, al, k & 31);
    ck = __shfl_sync(0xffffffffu, ck, k & 31);
    double beta = 0.0, hk = 0.0;
    if (__double2hiint(s2) > (923 << 20)) {  // ‖x‖² > 2^-100 (1e-30)
      // ‖x‖ and hk by one cubic step each from FP32 values (error ~ (2e-7)³)
      const double y = f2d(rsqrtf(d2f(s2))), g0 = s2 * y, e = fma(-g0, y, 1.0);
      const double sg = fma(g0 * e, fma(0.375, e, 0.5), g0);
      beta = __double2hiint(al) >= 0 ? -sg : sg;
      const double den = fma(fabs(al), sg, s2), h0 = f2d(__fdividef(1.f, d2f(den))), f = fma(-den, h0, 1.0);
      hk = fma(h0, fma(f, f, f), h0);
#pragma unroll
      for (int i = 0; i < R; ++i)
        if (lane + 32 * i == k) x[i] = al - beta;
    } else {
#pragma unroll
      for (int i = 0; i < R; ++i) x[i] = 0.0;
    }
    if (cta == 0 && warp == 0) {
#pragma unroll
      for (int i = 0; i < R; ++i)
        if (lane + 32 * i < m) H[lane + 32 * i + (int64_t)k * m] = x[i];
      if (lane == 0) {
        hinv[k] = hk;
        perm[k] = wj;
      }
    }
    if (have && pos < 0) {
      if (col == wj) {
        pos = k;
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const int row = lane + 32 * i;
          c[i] = row < k ? c[i] : (row == k ? beta : 0.0);
        }
      } else {
        d = fma(-beta, ck, d) * hk;
        nr = 0.f;
        float nr1 = 0.f;
#pragma unroll
        for (int i = 0; i < R; i += 2)
          if (32 * i < m && 32 * i + 63 >= k) {
            c[i] = fma(-d, x[i], c[i]);
            c[i + 1] = fma(-d, x[i + 1], c[i + 1]);
            const float f = lane + 32 * i > k ? d2f(c[i]) : 0.f, f1 = lane + 32 * i + 32 > k ? d2f(c[i + 1]) : 0.f;
            nr = fmaf(f, f, nr);
            nr1 = fmaf(f1, f1, nr1);
          }
        nr += nr1;
        nr = wsum_f(nr);
      }
    }
  }
  const int r = k;  // rank (STAGE 0: k < kmax when the rest was cut)
  __syncthreads();
  if (have && pos < 0) {  // columns that were never a pivot follow in index order
    int u = 0;
    for (int w = 0; w < (col >> 5); ++w) u += 32 - __popc(picked_mask[w]);
    u += (col & 31) - __popc(picked_mask[col >> 5] & ((1u << (col & 31)) - 1u));
    pos = r + u;
    if (lane == 0) perm[pos] = col;
  }
  if (have) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = lane + 32 * i;
      if (row < r) X[pos + (int64_t)row * a.ldx] = c[i];
    }
  }
  if (STAGE == 0 && cta == 0 && threadIdx.x == 0) q.info[kiRank] = r;
}

// ---------------------------------------------------------------------------
// One-sided Jacobi sweeps on the rc columns of X (mx rows), one launch.
// Columns are grouped in blocks of two; a round of the circle method pairs the
// blocks and CTA k takes the block pair (P, Q): its 4 columns come from L2 to
// shared memory (16-byte cp.async), the cross pairs are rotated in two inner
// rounds of two disjoint pairs (in a sweep's first round the pairs inside P and
// Q first), 64 threads per pair, and the columns go back; one barrier a round.
// Blocks of two halve the barriers of single columns and leave one pair per two
// SM quadrants; blocks of four leave half of the SMs without work.
//
// FP64 instructions are what a round costs, so the squared norms are carried
// (a ← a − tγ, b ← b + tγ; formed anew at each sweep's start), the angle starts
// in FP32 and takes one Newton step in FP64, and cos comes from rsqrt_fast: 14
// instructions where the quotients and square roots took ~4000 clocks.
// Sweeps end when no pair rotates, or when the largest |cos| that a sweep rotated
// times its largest |tan| is below half of tol: a rotation by t changes the
// |cos| of its columns with the others, zeroed before it, by t times theirs (not
// by the square where two singular values are close and t is large).
// ---------------------------------------------------------------------------
template <int RJ, bool ACCV, bool CL>
__global__ void __launch_bounds__(128) k_svd_sweeps(SvdArgs a) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  const SvdProb& q = a.p[blockIdx.y];
  const int rc = q.info[kiRank];
  const bool two = a.second || rc < a.n;
  const int mx = two ? rc : a.n;
  const int nreal = (rc + 1) >> 1, NB = nreal + (nreal & 1);
  const int active = NB >> 1, cta = blockIdx.x;
  if (!CL && cta >= max(active, 1)) return;
  if (q.info[kiErr]) return;
  double* W = q.W ? q.W : (two ? q.X2 : q.X);
  double* V = q.Vx;
  const int ldx = a.ldx;
  constexpr int ldw = 64 * RJ, cst = (ACCV ? 2 : 1) * ldw;
  double* sm = reinterpret_cast<double*>(sm_raw);  // 4 columns of cst doubles: W rows, then V rows
  __shared__ double nrm4[4], red[2][2];
  __shared__ int dead, nrot, cosmax, tanmax;
  if (threadIdx.x == 0) dead = nrot = cosmax = tanmax = 0;
  for (int i = threadIdx.x; i < 4 * cst; i += blockDim.x) sm[i] = 0.0;  // rows beyond mx stay 0 and need no guard
  __syncthreads();
  GridBar<CL> bar{reinterpret_cast<unsigned*>(q.info + kiBar + 2), 0u, (unsigned)max(active, 1), q.info + kiErr,
                  &dead};
  if (ACCV && !q.W) {  // Vx = I (each CTA its own share of the columns)
    const int nc = CL ? (int)gridDim.x : max(active, 1);
    for (int j = cta; j < rc; j += nc)
      for (int i = threadIdx.x; i < rc; i += blockDim.x) __stcg(&V[i + (int64_t)j * ldx], i == j ? 1.0 : 0.0);
    if (!bar.sync()) return;
  }
  const int grp = threadIdx.x >> 6, lt = threadIdx.x & 63, wip = (threadIdx.x >> 5) & 1, lane = threadIdx.x & 31;
  const float tolf = (float)a.tol;
  // a warp without rows in the last chunk leaves the FP64 units to the others (mx ≥ rc)
  const bool last = 64 * (RJ - 1) + 32 * wip < mx;

  // rotate local columns x < y (in global order) of this thread group; their W
  // rows stay in registers between the dot product and the rotation
  auto process = [&](int x, int y, bool present) {
    double g = 0.0, u[RJ], v[RJ];
    double* wx = sm + (int64_t)x * cst;
    double* wy = sm + (int64_t)y * cst;
    if (present) {
#pragma unroll
      for (int e = 0; e < RJ; ++e) {
        u[e] = wx[lt + 64 * e];
        v[e] = wy[lt + 64 * e];
      }
      double g1 = 0.0;
#pragma unroll
      for (int e = 0; e < RJ; ++e) {
        if (e < RJ - 1 || last) {
          if (e & 1) g1 = fma(u[e], v[e], g1);
          else g = fma(u[e], v[e], g);
        }
      }
      if (RJ > 1) g += g1;
      g = wsum_d(g);
      if (lane == 0) red[grp][wip] = g;
    }
    asm volatile("bar.sync %0, 64;" ::"r"(grp + 1) : "memory");
    if (present) {
      g = red[grp][0] + red[grp][1];
      const double na = nrm4[x], nb = nrm4[y];
      const float gf = d2f(g), cs2 = fsqrt_ap(d2f(na)) * fsqrt_ap(d2f(nb));
      if (fabsf(gf) > tolf * cs2) {
        const double dl = nb - na;
        const float df = d2f(dl), g2 = 2.f * gf;
        const float t0 = jacobi_tan(df, g2);
        // one Newton step on γt² + (b − a)t − γ = 0
        const double td = f2d(t0);
        const double fr = fma(fma(g, td, dl), td, -g);
        const double t = fma(-fr, f2d(__fdividef(1.f, fmaf(g2, t0, df))), td);
        const double cs = rsqrt_fast(fma(t, t, 1.0)), sn = cs * t;
#pragma unroll
        for (int e = 0; e < RJ; ++e) {
          const int i = lt + 64 * e;
          if (e < RJ - 1 || last) {
            wx[i] = cs * u[e] - sn * v[e];
            wy[i] = sn * u[e] + cs * v[e];
          }
        }
        if (ACCV) {
          double* vx = wx + ldw;
          double* vy = wy + ldw;
#pragma unroll
          for (int e = 0; e < RJ; ++e) {
            u[e] = vx[lt + 64 * e];
            v[e] = vy[lt + 64 * e];
          }
#pragma unroll
          for (int e = 0; e < RJ; ++e) {
            const int i = lt + 64 * e;
            if (e < RJ - 1 || last) {
              vx[i] = cs * u[e] - sn * v[e];
              vy[i] = sn * u[e] + cs * v[e];
            }
          }
        }
        asm volatile("bar.sync %0, 64;" ::"r"(grp + 1) : "memory");  // norms read by all of the group
        if (lt == 0) {
          const double tg = t * g;
          nrm4[x] = na - tg;
          nrm4[y] = nb + tg;
          atomicAdd(&nrot, 1);
          atomicMax(&cosmax, __float_as_int(cs2 > 0.f ? fminf(__fdividef(fabsf(gf), cs2), 1.f) : 1.f));
          atomicMax(&tanmax, __float_as_int(fabsf(t0)));
        }
      }
    }
  };

  const int rounds = NB - 1;
  int sweep = 0;
  bool done = rc < 2;
  for (; sweep < a.max_sweeps && !done; ++sweep) {
    for (int r = 0; r < rounds; ++r) {
      if (cta < active) {
        int P, Q;
        if (cta == 0) {
          P = r;
          Q = NB - 1;
        } else {
          P = (r + cta) % (NB - 1);
          Q = (r - cta + (NB - 1)) % (NB - 1);
        }
        if (P > Q) {
          const int t = P;
          P = Q;
          Q = t;
        }
        auto gc = [&](int l) { return l < 2 ? 2 * P + l : 2 * Q + l - 2; };  // (an array would be local memory)
        // 4 columns of W and V to shared memory
        for (int l = 0; l < 4; ++l) {
          if (gc(l) >= rc) continue;
          const double* ws = W + (int64_t)gc(l) * ldx;
          const uint32_t dst = tc::su32(sm + (int64_t)l * cst);
          for (int i = threadIdx.x; i < (mx >> 1); i += blockDim.x)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * i), "l"(ws + 2 * i) : "memory");
          if ((mx & 1) && threadIdx.x == blockDim.x - 1) sm[(int64_t)l * cst + mx - 1] = __ldcg(&ws[mx - 1]);
          if (ACCV) {
            const double* vs = V + (int64_t)gc(l) * ldx;
            if ((rc & 1) && threadIdx.x == blockDim.x - 2) sm[(int64_t)l * cst + ldw + rc - 1] = __ldcg(&vs[rc - 1]);
            for (int i = threadIdx.x; i < (rc >> 1); i += blockDim.x)
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 8u * ldw + 16u * i), "l"(vs + 2 * i)
                           : "memory");
          }
        }
        if (r > 0 && threadIdx.x < 4 && gc(threadIdx.x) < rc) nrm4[threadIdx.x] = __ldcg(&q.nrm[gc(threadIdx.x)]);
        asm volatile("cp.async.wait_all;" ::: "memory");
        // read before the barrier: after it the other group may already count a
        // rotation of this round, and the threads would not agree on the write-back
        const int rot0 = nrot;
        __syncthreads();
        if (r == 0) {  // norms anew: warp w takes column w
          const int w = threadIdx.x >> 5;
          double s = 0.0;
          if (gc(w) < rc) {
            const double* wc = sm + (int64_t)w * cst;
#pragma unroll 4
            for (int i = lane; i < mx; i += 32) s = fma(wc[i], wc[i], s);
            s = wsum_d(s);
            if (lane == 0) nrm4[w] = s;
          }
          __syncthreads();
          process(2 * grp, 2 * grp + 1, gc(2 * grp + 1) < rc);
          __syncthreads();
        }
        process(grp, 2 + grp, gc(grp) < rc && gc(2 + grp) < rc);
        __syncthreads();
        process(grp, 3 - grp, gc(grp) < rc && gc(3 - grp) < rc);
        __syncthreads();
        if (nrot != rot0 || r == 0) {
          for (int l = 0; l < 4; ++l) {
            if (gc(l) >= rc) continue;
            double2* wd = reinterpret_cast<double2*>(W + (int64_t)gc(l) * ldx);  // (ldx is even: room for the pair)
            const double2* s2 = reinterpret_cast<const double2*>(sm + (int64_t)l * cst);
            for (int i = threadIdx.x; i < ((mx + 1) >> 1); i += blockDim.x) __stcg(&wd[i], s2[i]);
            if (ACCV) {
              double2* vd = reinterpret_cast<double2*>(V + (int64_t)gc(l) * ldx);
              for (int i = threadIdx.x; i < ((rc + 1) >> 1); i += blockDim.x) __stcg(&vd[i], s2[(ldw >> 1) + i]);
            }
          }
          if (threadIdx.x < 4 && gc(threadIdx.x) < rc) __stcg(&q.nrm[gc(threadIdx.x)], nrm4[threadIdx.x]);
        }
      }
      if (r == rounds - 1) {
        __syncthreads();  // every thread has compared nrot with rot0
        if (threadIdx.x == 0 && nrot) {
          atomicAdd(&q.info[kiRot + sweep], nrot);
          atomicMax(&q.info[kiCos + sweep], cosmax);
          atomicMax(&q.info[kiTan + sweep], tanmax);
          nrot = cosmax = tanmax = 0;
        }
      }
      if (!bar.sync()) return;
    }
    const int rot = __ldcg(&q.info[kiRot + sweep]);
    const float cm = __int_as_float(__ldcg(&q.info[kiCos + sweep]));
    const float tm = __int_as_float(__ldcg(&q.info[kiTan + sweep]));
    done = rot == 0 || cm * tm < 0.5f * tolf;
  }
  if (cta == 0 && threadIdx.x == 0) q.info[kiSweeps] = done ? max(sweep, 1) : 0;
}

// ---------------------------------------------------------------------------
// FP32 Jacobi sweeps, one launch: they precede the FP64 sweeps (n ≥ kPreMin) and
// start the corner's product refinement (EIG).  Blocks of 8 columns; CTA k takes
// the block pair of the round from L2 to shared memory (16-byte cp.async), W and
// V of 16 columns, rotates the 64 cross pairs in 8 inner rounds of 8 disjoint
// pairs (in a sweep's first round the pairs inside the blocks too, 7 inner
// rounds), and stores them; one barrier a round, n/8 − 1 rounds a sweep.  WP
// warps per pair, RV 16-byte chunks per lane and column, packed arithmetic
// (fma.rn.f32x2).  Blocks this long because a round's barrier and L2 exchange
// cost as much as ~6 inner rounds; longer ones leave too few CTAs at n = 1024.
//
// Rules: one-sided (a, b, g from W's columns, relative: graded columns keep
// their relative accuracy in FP32, so X·V comes out with |cos| ~ 1e-6 between
// all columns, small ones included), ended by a sweep that rotated no |cos|
// above kPreCos; EIG: the 2×2 block of VᵀXV for symmetric X (±λ pairs are not
// mixed), absolute threshold, ended by a sweep with at most eig_sweep_last(n) rotations.
//
// A group keeps its column of P in registers through the inner rounds, so that
// shared memory carries Q's columns only (128 bytes a clock limit n = 1024).
// Measured: n = 1024 15 ms for 9-10 sweeps, as 255 launches a sweep of 4-column
// blocks 17.9; n = 324 2.0 ms, 3.4 in one 16-CTA cluster with scalar loads.  A wait
// for the round's two blocks only, by a flag a block, instead of the grid barrier
// took 16.8 ms at n = 1024.
// ---------------------------------------------------------------------------
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

template <int B, int RV, int WP, bool EIG, bool CL>
__global__ void __launch_bounds__(32 * B * WP) k_sweeps32(SvdArgs a) {
  constexpr int LP = 32 * WP, NW = B * WP;  // lanes per pair, warps
  extern __shared__ __align__(16) unsigned char sm_raw[];
  const SvdProb& q = a.p[blockIdx.y];
  const int rc = EIG ? a.n : q.info[kiRank];
  const bool two = !EIG && (a.second || rc < a.n);
  const int mx = two ? rc : a.n;
  const int nreal = (rc + B - 1) / B, NB = nreal + (nreal & 1);
  const int active = NB >> 1, cta = blockIdx.x;
  if (q.info[kiErr]) return;
  if (!CL && cta >= active) return;  // a cluster's idle CTAs keep to its barriers
  float* W = q.W32;
  float* V = q.V32;
  const int ld = a.ld32;
  const int q4 = (mx + 3) >> 2, v4 = (rc + 3) >> 2, c4 = q4 + v4;  // 16-byte chunks of W, V, a column
  ulonglong2* sm = reinterpret_cast<ulonglong2*>(sm_raw);          // 16 columns: W rows, then V rows
  __shared__ float red[B][WP][3];
  __shared__ int dead, nrot, cosmax;
  if (threadIdx.x == 0) dead = nrot = cosmax = 0;
  __syncthreads();
  GridBar<CL> bar{reinterpret_cast<unsigned*>(q.info + kiBar + 3), 0u, (unsigned)active, q.info + kiErr, &dead};
  const double* X = EIG ? q.A : (two ? q.X2 : q.X);
  for (int j = cta; j < rc; j += max(active, 1)) {
    for (int i = threadIdx.x; i < 4 * q4; i += blockDim.x)
      __stcg(&W[i + (int64_t)j * ld], i < mx ? d2f(X[i + (int64_t)j * a.ldx]) : 0.f);
    for (int i = threadIdx.x; i < 4 * v4; i += blockDim.x) __stcg(&V[i + (int64_t)j * ld], i == j ? 1.f : 0.f);
  }
  if (!bar.sync()) return;
  const float thr_abs = EIG ? 2.f * FLT_EPSILON * sqrtf((float)a.fro2[0]) : 0.f;
  const int grp = threadIdx.x / LP, lt = threadIdx.x % LP, wip = (threadIdx.x >> 5) % WP, lane = threadIdx.x & 31;

  int my_rot = 0;  // of this thread's pairs, in the current sweep
  float my_cos = 0.f;
  // rotation of the pair (W, V) = (wx, vx), (wy, vy) held in registers; true when
  // it rotates.  Every thread of the pair returns the same.
  const ulonglong2 z = make_ulonglong2(0, 0);
  auto rotate = [&](ulonglong2 (&wx)[RV], ulonglong2 (&vx)[RV], ulonglong2 (&wy)[RV], ulonglong2 (&vy)[RV],
                    bool present) -> bool {
    float na = 0.f, nb = 0.f, g2 = 0.f;  // a, b, 2g
    if (present) {
      uint64_t sa = 0, sb = 0, sg = 0;
#pragma unroll
      for (int e = 0; e < RV; ++e) {
        if (EIG) {
          sa = fma2(vx[e].x, wx[e].x, sa);
          sb = fma2(vy[e].x, wy[e].x, sb);
          sg = fma2(vx[e].x, wy[e].x, sg);
          sg = fma2(vy[e].x, wx[e].x, sg);
          sa = fma2(vx[e].y, wx[e].y, sa);
          sb = fma2(vy[e].y, wy[e].y, sb);
          sg = fma2(vx[e].y, wy[e].y, sg);
          sg = fma2(vy[e].y, wx[e].y, sg);
        } else {
          sa = fma2(wx[e].x, wx[e].x, sa);
          sb = fma2(wy[e].x, wy[e].x, sb);
          sg = fma2(wx[e].x, wy[e].x, sg);
          sa = fma2(wx[e].y, wx[e].y, sa);
          sb = fma2(wy[e].y, wy[e].y, sb);
          sg = fma2(wx[e].y, wy[e].y, sg);
        }
      }
      na = hsum2(sa);
      nb = hsum2(sb);
      g2 = EIG ? hsum2(sg) : 2.f * hsum2(sg);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        na += __shfl_xor_sync(0xffffffffu, na, o);
        nb += __shfl_xor_sync(0xffffffffu, nb, o);
        g2 += __shfl_xor_sync(0xffffffffu, g2, o);
      }
      if (WP > 1 && lane == 0) {
        red[grp][wip][0] = na;
        red[grp][wip][1] = nb;
        red[grp][wip][2] = g2;
      }
    }
    if (WP > 1) {
      asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "n"(LP) : "memory");
      if (present) {
        na = nb = g2 = 0.f;
#pragma unroll
        for (int w = 0; w < WP; ++w) {
          na += red[grp][w][0];
          nb += red[grp][w][1];
          g2 += red[grp][w][2];
        }
      }
    }
    if (!present) return false;
    const float ag = 0.5f * fabsf(g2), nn = fsqrt_ap(fabsf(na)) * fsqrt_ap(fabsf(nb));
    if (!(EIG ? ag > thr_abs : ag > a.tol32 * nn)) return false;
    const float t = jacobi_tan(nb - na, g2);
    const float c = rsqrtf(fmaf(t, t, 1.f)), sn = c * t;
    const uint64_t c2 = pk2(c, c), s2 = pk2(sn, sn), n2 = pk2(-sn, -sn);
#pragma unroll
    for (int e = 0; e < RV; ++e) {
      const ulonglong2 wu = wx[e], vu = vx[e];
      wx[e] = make_ulonglong2(fma2(c2, wu.x, mul2(n2, wy[e].x)), fma2(c2, wu.y, mul2(n2, wy[e].y)));
      wy[e] = make_ulonglong2(fma2(c2, wy[e].x, mul2(s2, wu.x)), fma2(c2, wy[e].y, mul2(s2, wu.y)));
      vx[e] = make_ulonglong2(fma2(c2, vu.x, mul2(n2, vy[e].x)), fma2(c2, vu.y, mul2(n2, vy[e].y)));
      vy[e] = make_ulonglong2(fma2(c2, vy[e].x, mul2(s2, vu.x)), fma2(c2, vy[e].y, mul2(s2, vu.y)));
    }
    ++my_rot;
    if (!EIG) my_cos = fmaxf(my_cos, nn > 0.f ? fminf(__fdividef(ag, nn), 1.f) : 1.f);
    return true;
  };
  auto fetch = [&](int l, ulonglong2 (&w)[RV], ulonglong2 (&v)[RV]) {
    const ulonglong2* c = sm + l * c4;
#pragma unroll
    for (int e = 0; e < RV; ++e) {
      const int i = lt + LP * e;
      w[e] = i < q4 ? c[i] : z;
      v[e] = i < v4 ? c[q4 + i] : z;
    }
  };
  auto keep = [&](int l, const ulonglong2 (&w)[RV], const ulonglong2 (&v)[RV]) {
    ulonglong2* c = sm + l * c4;
#pragma unroll
    for (int e = 0; e < RV; ++e) {
      const int i = lt + LP * e;
      if (i < q4) c[i] = w[e];
      if (i < v4) c[q4 + i] = v[e];
    }
  };

  const int rounds = NB - 1;
  bool done = rc < 2;
  for (int sweep = 0; sweep < (EIG ? kEigSweeps : kPreSweeps) && !done; ++sweep) {
    for (int r = 0; r < rounds; ++r) {
      if (cta < active) {
        int P, Q;
        if (cta == 0) {
          P = r;
          Q = NB - 1;
        } else {
          P = (r + cta) % (NB - 1);
          Q = (r - cta + (NB - 1)) % (NB - 1);
        }
        if (P > Q) {
          const int t = P;
          P = Q;
          Q = t;
        }
        auto gcol = [&](int l) { return l < B ? B * P + l : B * Q + l - B; };
        for (int l = threadIdx.x >> 5; l < 2 * B; l += NW) {  // one warp per column
          const int g = gcol(l);
          if (g >= rc) continue;
          const float* ws = W + (int64_t)g * ld;
          const float* vs = V + (int64_t)g * ld;
          const uint32_t dst = tc::su32(sm + l * c4);
          for (int i = lane; i < q4; i += 32)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * i), "l"(ws + 4 * i) : "memory");
          for (int i = lane; i < v4; i += 32)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * (q4 + i)), "l"(vs + 4 * i)
                         : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        ulonglong2 wx[RV], vx[RV], wy[RV], vy[RV];
        if (r == 0) {  // pairs inside P (first half of the groups) and inside Q: circle method over B
          for (int ir = 0; ir < B - 1; ++ir) {
            const int k = grp % (B / 2), off = grp < B / 2 ? 0 : B;
            int x = k == 0 ? B - 1 : (ir + k) % (B - 1);
            int y = k == 0 ? ir : (ir - k + (B - 1)) % (B - 1);
            if (x > y) {
              const int t = x;
              x = y;
              y = t;
            }
            const bool present = gcol(off + y) < rc;
            if (present) {
              fetch(off + x, wx, vx);
              fetch(off + y, wy, vy);
            }
            if (rotate(wx, vx, wy, vy, present)) {
              keep(off + x, wx, vx);
              keep(off + y, wy, vy);
            }
            __syncthreads();
          }
        }
        // cross pairs: a group keeps its column of P in registers through the B
        // inner rounds; Q's columns pass through shared memory
        fetch(grp, wx, vx);
        for (int ir = 0; ir < B; ++ir) {
          const int y = B + ((grp + ir) & (B - 1));
          const bool present = gcol(y) < rc;  // P comes before Q
          if (present) fetch(y, wy, vy);
          if (rotate(wx, vx, wy, vy, present)) keep(y, wy, vy);
          __syncthreads();
        }
        if (gcol(grp) < rc) {
          ulonglong2* wd = reinterpret_cast<ulonglong2*>(W + (int64_t)gcol(grp) * ld);
          ulonglong2* vd = reinterpret_cast<ulonglong2*>(V + (int64_t)gcol(grp) * ld);
#pragma unroll
          for (int e = 0; e < RV; ++e) {
            const int i = lt + LP * e;
            if (i < q4) __stcg(&wd[i], wx[e]);
            if (i < v4) __stcg(&vd[i], vx[e]);
          }
        }
        for (int l = B + (threadIdx.x >> 5); l < 2 * B; l += NW) {
          const int g = gcol(l);
          if (g >= rc) continue;
          ulonglong2* wd = reinterpret_cast<ulonglong2*>(W + (int64_t)g * ld);
          ulonglong2* vd = reinterpret_cast<ulonglong2*>(V + (int64_t)g * ld);
          const ulonglong2* s4 = sm + l * c4;
          for (int i = lane; i < q4; i += 32) __stcg(&wd[i], s4[i]);
          for (int i = lane; i < v4; i += 32) __stcg(&vd[i], s4[q4 + i]);
        }
      }
      if (r == rounds - 1) {
        if (lt == 0 && my_rot) {
          atomicAdd(&nrot, my_rot);
          atomicMax(&cosmax, __float_as_int(my_cos));
        }
        my_rot = 0;
        my_cos = 0.f;
        __syncthreads();
        if (threadIdx.x == 0 && nrot) {
          atomicAdd(&q.info[kiRot32 + sweep], nrot);
          atomicMax(&q.info[kiCos32 + sweep], cosmax);
          nrot = 0;
          cosmax = 0;
        }
      }
      if (!bar.sync()) return;
    }
    const int rot = __ldcg(&q.info[kiRot32 + sweep]);
    done = EIG ? rot <= eig_sweep_last(rc) : rot == 0 || __int_as_float(__ldcg(&q.info[kiCos32 + sweep])) < kPreCos;
    if (done && cta == 0 && threadIdx.x == 0) q.info[kiPre] = sweep + 1;
  }
  // V in FP64
  for (int j = cta; j < rc; j += max(active, 1))
    for (int i = threadIdx.x; i < rc; i += blockDim.x)
      q.Vx[i + (int64_t)j * a.ldx] = f2d(__ldcg(&V[i + (int64_t)j * ld]));
}

// F = VᵀV − I (r×r) → the factor of V ← V·(I − T): T_qp = F_qp below the
// diagonal, F_pp/2 on it.  A column is cleared of the later (smaller) ones
// only: the small columns of V carry their relative accuracy in tiny entries,
// which a symmetric correction would fill with rounding of the large ones.
__global__ void k_svd_tri(double* __restrict__ F, int r) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < r * r; e += gridDim.x * blockDim.x) {
    const int i = e % r, j = e / r;
    const double f = F[e];
    F[e] = i > j ? f : (i == j ? 0.5 * (f - 1.0) : 0.0);
  }
}

// σ_j = ‖W_j‖ (unsorted, still scaled); one warp per column
__global__ void k_svd_norms(SvdArgs a) {
  const SvdProb& q = a.p[blockIdx.y];
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int rc = q.info[kiRank];
  if (j >= a.n || q.info[kiErr]) return;
  double s = 0.0;
  if (j < rc) {
    const bool two = a.second || rc < a.n;
    const int mx = two ? rc : a.n;
    const double* w = (q.W ? q.W : (two ? q.X2 : q.X)) + (int64_t)j * a.ldx;
    for (int i = lane; i < mx; i += 32) s = fma(w[i], w[i], s);
    s = sqrt(wsum_d(s));
  }
  if (lane == 0) q.sv[j] = s;
}

// One CTA per column j: its rank among the σ (descending, ties by index; the
// cut columns follow) and the column in its sorted place:
//   U[:, rank] = P₂·Wn_j (to be multiplied by Q), V[:, rank] = Vx_j (by P·Q₂),
//   or V[:, rank] = P·Wn_j where the second QR was skipped (symmetric, r = n);
//   symmetric: only V is formed, from P₂·Wn_j.
template <bool SYM>
__global__ void __launch_bounds__(128) k_svd_place(SvdArgs a) {
  const SvdProb& q = a.p[blockIdx.y];
  const int j = blockIdx.x, n = a.n;
  const int rc = q.info[kiRank];
  if (q.info[kiErr]) return;  // a wait gave up: perm and perm2, which this kernel stores through, may be unwritten
  const bool two = a.second || rc < n;
  const double sj = q.sv[j];
  int rk = j;
  if (j < rc) {
    int cnt = 0;
    for (int i = threadIdx.x; i < rc; i += blockDim.x) {
      const double si = q.sv[i];
      cnt += (si > sj || (si == sj && i < j)) ? 1 : 0;
    }
    __shared__ int part[4];
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = cnt;
    __syncthreads();
    rk = part[0] + part[1] + part[2] + part[3];
  }
  double* u = SYM ? nullptr : q.U + (int64_t)rk * n;
  double* v = q.V + (int64_t)rk * n;
  if (q.info[kiBad]) {
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    if (!SYM)
      for (int i = threadIdx.x; i < n; i += blockDim.x) u[i] = nan;
    for (int i = threadIdx.x; i < n; i += blockDim.x) v[i] = nan;
    if (threadIdx.x == 0) q.S[rk] = nan;
    return;
  }
  if (threadIdx.x == 0) q.S[rk] = scalbn(sj, q.info[kiExp]);
  if (j >= rc) {
    if (!SYM)
      for (int i = threadIdx.x; i < n; i += blockDim.x) u[i] = i == j ? 1.0 : 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) v[i] = i == j ? 1.0 : 0.0;
    return;
  }
  const double inv = sj > 0.0 ? 1.0 / sj : 0.0;
  if (SYM && !two) {
    const double* w = (q.W ? q.W : q.X) + (int64_t)j * a.ldx;
    for (int i = threadIdx.x; i < n; i += blockDim.x) v[q.perm[i]] = w[i] * inv;
    return;
  }
  const double* w = (q.W ? q.W : q.X2) + (int64_t)j * a.ldx;
  double* o = SYM ? v : u;
  for (int i = rc + threadIdx.x; i < n; i += blockDim.x) o[i] = 0.0;
  for (int i = threadIdx.x; i < rc; i += blockDim.x) o[q.perm2[i]] = w[i] * inv;
  if (!SYM) {
    const double* x = q.Vx + (int64_t)j * a.ldx;
    for (int i = threadIdx.x; i < n; i += blockDim.x) v[i] = i < rc ? x[i] : 0.0;
  }
}

// B ← Q·B, Q = H_0·H_1···H_{r−1}: one warp per column of B, which it holds in
// registers; the reflectors are read through L1/L2, the next one prefetched
// while the current one is applied.  STAGE 0: Q of A on U (symmetric: on V);
// STAGE 1: Q₂ on V, rows then permuted by P.
template <int R, bool SYM, int STAGE>
__global__ void __launch_bounds__(128) k_svd_apply_q(SvdArgs a) {
  const SvdProb& q = a.p[blockIdx.y];
  const int rc = q.info[kiRank], n = a.n;
  if (q.info[kiErr] || q.info[kiBad]) return;
  if (SYM && rc == n) return;  // the eigenvectors are in place
  const int rows = n;
  const int col = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (col >= n) return;
  const double* H = STAGE == 0 ? q.H : q.H2;
  const double* hinv = STAGE == 0 ? q.hinv : q.hinv2;
  double* B = ((STAGE == 0 && !SYM) ? q.U : q.V) + (int64_t)col * rows;
  double c[R], x[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = lane + 32 * i;
    c[i] = row < rows ? B[row] : 0.0;
    x[i] = (row < rows && rc > 0) ? H[row + (int64_t)(rc - 1) * rows] : 0.0;
  }
  for (int k = rc - 1; k >= 0; --k) {
    double d = 0.0;
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (32 * i < rows && 32 * i + 31 >= k) d = fma(x[i], c[i], d);
    double xn[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = lane + 32 * i;
      xn[i] = (k > 0 && 32 * i + 31 >= k - 1 && row < rows) ? H[row + (int64_t)(k - 1) * rows] : 0.0;
    }
    d = wsum_d(d) * hinv[k];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (32 * i < rows && 32 * i + 31 >= k) c[i] = fma(-d, x[i], c[i]);
      x[i] = xn[i];
    }
  }
  __syncwarp();  // every lane has read its rows of the column
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = lane + 32 * i;
    if (row < rows) B[STAGE == 1 ? q.perm[row] : row] = c[i];
  }
}

// Eigenvectors of a symmetric A from its singular vectors X (σ descending in S).
// X spans what it has to, but only up to rotations by ~ε·‖A‖/||λ_i| − |λ_j|| between
// columns: where λ_i and λ_j have opposite signs and about the same size (exact ±λ
// pairs, any size; or close ones), x_j is then no eigenvector and ±x_j no left vector.
// M = XᵀAX shows it: an entry above thr_rel·σ_1, the rounding of M, is such a
// coupling.  A column without one is kept, a pair takes the eigenvectors of its 2×2
// block, and a column in a larger group (a multiplet of both signs) sets *multi,
// upon which the caller separates them by eigenvalue sweeps (eig_separate).
// U = V·sign(λ).  One CTA per column.
__global__ void __launch_bounds__(128) k_svd_sym_basis(int n, const double* __restrict__ X,
                                                       const double* __restrict__ M, const double* __restrict__ S,
                                                       double thr_rel, double* __restrict__ U, double* __restrict__ V,
                                                       int* __restrict__ multi) {
  const int j = blockIdx.x;
  const double thr = thr_rel * S[0];
  __shared__ int cnt[2], who[2];  // coupled columns of this one and of its partner
  if (threadIdx.x < 2) {
    cnt[threadIdx.x] = 0;
    who[threadIdx.x] = -1;
  }
  __syncthreads();
  auto scan = [&](int col, int slot) {
    for (int i = threadIdx.x; i < n; i += blockDim.x)
      if (i != col && fabs(M[i + (int64_t)col * n]) > thr) {
        atomicAdd(&cnt[slot], 1);
        who[slot] = i;
      }
  };
  scan(j, 0);
  __syncthreads();
  const int o = cnt[0] == 1 ? who[0] : -1;
  if (o >= 0) scan(o, 1);
  __syncthreads();
  // (M is symmetric up to rounding: at the threshold only one of the two may see the other)
  const bool pair = o >= 0 && cnt[1] == 1 && who[1] == j;
  if (cnt[0] > 0 && !pair && threadIdx.x == 0) *multi = 1;
  const int lo = pair ? min(j, o) : j, hi = pair ? max(j, o) : j;
  double cl = 1.0, ch = 0.0, lam = M[j + (int64_t)j * n];
  if (pair) {
    const double a = M[lo + (int64_t)lo * n], b = M[hi + (int64_t)hi * n], g = M[hi + (int64_t)lo * n];
    const double tau = (b - a) / (2.0 * g);
    const double t = copysign(1.0, tau) / (fabs(tau) + sqrt(fma(tau, tau, 1.0)));
    const double c = 1.0 / sqrt(fma(t, t, 1.0)), s = c * t, la = a - t * g, lb = b + t * g;
    const bool swap = fabs(la) < fabs(lb);  // S is in descending order
    if ((j == lo) != swap) {
      cl = c;
      ch = -s;
      lam = la;
    } else {
      cl = s;
      ch = c;
      lam = lb;
    }
  }
  const double sg = lam < 0.0 ? -1.0 : 1.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double v = pair ? cl * X[i + (int64_t)lo * n] + ch * X[i + (int64_t)hi * n] : X[i + (int64_t)j * n];
    V[i + (int64_t)j * n] = v;
    U[i + (int64_t)j * n] = sg * v;
  }
}

template <typename F>
void launch_grid(tnad_ctx* c, F* f, bool cluster, int G, int np, int threads, size_t smem, SvdArgs& a) {
  cudaLaunchConfig_t cf = {};
  cf.gridDim = dim3((unsigned)G, (unsigned)np);
  cf.blockDim = dim3((unsigned)threads);
  cf.dynamicSmemBytes = smem;
  cf.stream = c->stream;
  cudaLaunchAttribute at[1];
  if (cluster && G > 8) TNAD_CK(cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  if (cluster) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)G;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
  } else {
    at[0].id = cudaLaunchAttributeCooperative;  // the CTAs wait on one another: all resident or none
    at[0].val.cooperative = 1;
  }
  cf.attrs = at;
  cf.numAttrs = 1;
  TNAD_CK(cudaLaunchKernelEx(&cf, f, a));
  count_launch(c);
}

template <int R, int STAGE>
void launch_qrcp(tnad_ctx* c, int np, int cols, SvdArgs& a) {
  // Up to 64 columns in a cluster, 4 warps a CTA (one an SM quadrant).  Beyond, CTAs
  // over the whole GPU: a column each up to 128 (n = 121: 6200 clocks a step, 6800 in
  // CTAs of 4 warps, 8000 in a cluster of 16 CTAs of 8, whose FP64 instructions
  // share the quadrants), then 4 warps a CTA, or more where the SMs run out: fewer
  // CTAs read the step's keys and column (n = 324: 10300 clocks, 12600 with 152 CTAs).
  if constexpr (R == 2) {
    const int G = std::min(kQrCl, (cols + 3) / 4);
    launch_grid(c, k_qrcp<R, true, STAGE>, true, G, np, 32 * ((cols + G - 1) / G), 0, a);
  } else {
    const int G = std::min(cols <= 128 ? cols : (cols + 3) / 4, c->sm_count / np);
    launch_grid(c, k_qrcp<R, false, STAGE>, false, G, np, 32 * ((cols + G - 1) / G), 0, a);
  }
}

template <int RJ, bool ACCV>
void launch_sweeps_rj(tnad_ctx* c, int np, SvdArgs& a) {
  const int nreal = (a.n + 1) / 2, G = std::max(1, (nreal + (nreal & 1)) / 2);
  const size_t smem = (size_t)4 * 64 * RJ * (ACCV ? 2 : 1) * sizeof(double);
  if constexpr (RJ == 1) {
    if (G <= 16) {
      launch_grid(c, k_svd_sweeps<RJ, ACCV, true>, true, G, np, 128, smem, a);
      return;
    }
  }
  static PerDevice attr;
  if (!attr.has(c->device)) {
    TNAD_CK(cudaFuncSetAttribute(k_svd_sweeps<RJ, ACCV, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 4 * kMaxSvdRows * 2 * 8));
    attr.mark(c->device);
  }
  launch_grid(c, k_svd_sweeps<RJ, ACCV, false>, false, G, np, 128, smem, a);
}

// By the rows that there are, in steps of 64 (of 128 beyond 512): a guard on each
// of a thread's rows cost a third of the rotation at n = 324
template <bool ACCV>
void launch_sweeps(tnad_ctx* c, int np, int rows, SvdArgs& a) {
  switch ((rows + 63) / 64) {
    case 0:
    case 1: return launch_sweeps_rj<1, ACCV>(c, np, a);
    case 2: return launch_sweeps_rj<2, ACCV>(c, np, a);
    case 3: return launch_sweeps_rj<3, ACCV>(c, np, a);
    case 4: return launch_sweeps_rj<4, ACCV>(c, np, a);
    case 5: return launch_sweeps_rj<5, ACCV>(c, np, a);
    case 6: return launch_sweeps_rj<6, ACCV>(c, np, a);
    case 7: return launch_sweeps_rj<7, ACCV>(c, np, a);
    case 8: return launch_sweeps_rj<8, ACCV>(c, np, a);
    case 9:
    case 10: return launch_sweeps_rj<10, ACCV>(c, np, a);
    case 11:
    case 12: return launch_sweeps_rj<12, ACCV>(c, np, a);
    default: return launch_sweeps_rj<16, ACCV>(c, np, a);
  }
}

template <int B, int RV, int WP, bool EIG, bool CL>
void launch_sweeps32_rv(tnad_ctx* c, int np, SvdArgs& a) {
  const int nreal = (a.n + B - 1) / B, G = std::max(1, (nreal + (nreal & 1)) / 2);
  static PerDevice attr;
  if (!attr.has(c->device)) {
    TNAD_CK(cudaFuncSetAttribute(k_sweeps32<B, RV, WP, EIG, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 2 * B * 2 * 128 * WP * RV * 4));  // 2B columns of W and V
    attr.mark(c->device);
  }
  launch_grid(c, k_sweeps32<B, RV, WP, EIG, CL>, CL, G, np, 32 * B * WP, (size_t)2 * B * 2 * a.ld32 * sizeof(float), a);
}

// Up to 128 columns the at most 8 CTAs form a cluster.  One warp per pair up to
// 512 rows (a second one's share of the sums costs a barrier), two beyond, where a
// lane would hold 64 registers of each column; and there blocks of 4, which spread
// 1024 columns over 128 SMs' shared memories.
template <bool EIG>
void launch_sweeps32(tnad_ctx* c, int np, SvdArgs& a) {
  if (a.n <= 128)
    launch_sweeps32_rv<8, 1, 1, EIG, true>(c, np, a);
  else if (a.n <= 256)
    launch_sweeps32_rv<8, 2, 1, EIG, false>(c, np, a);
  else if (a.n <= 384)
    launch_sweeps32_rv<8, 3, 1, EIG, false>(c, np, a);
  else if (a.n <= 512)
    launch_sweeps32_rv<8, 4, 1, EIG, false>(c, np, a);
  else
    launch_sweeps32_rv<4, 4, 2, EIG, false>(c, np, a);
}

// FP32 sweeps, then V orthogonal to FP64 rounding (two first-order triangular
// corrections: 1e-6 → 1e-12 → 1e-24) and W = X·V, all in DFMA products: the
// tensor-core ones are accurate to the row and column scales only, not to the
// small columns of graded operands.
void pre_sweeps(tnad_ctx* c, int np, SvdArgs& a, int* info_host) {
  launch_sweeps32<false>(c, np, a);
  for (int p = 0; p < np; ++p)
    TNAD_CK(cudaMemcpyAsync(info_host + p * kiBar, a.p[p].info, sizeof(int) * kiBar, cudaMemcpyDeviceToHost, c->stream));
  TNAD_CK(cudaStreamSynchronize(c->stream));
  for (int p = 0; p < np; ++p) {
    SvdProb& q = a.p[p];
    const int r = info_host[p * kiBar + kiRank];
    const bool two = a.second || r < a.n;
    const int mx = two ? r : a.n;
    TNAD_REQUIRE(info_host[p * kiBar + kiErr] == 0, TNAD_ERR_TIMEOUT, "svd_qrj: a bounded barrier wait expired");
    if (r < 2) continue;  // (q.W stays null: nothing to hand over)
    WsScope scope(c);
    double* F = ws_d(c, (int64_t)r * r);
    double* V2 = ws_d(c, (int64_t)a.ldx * r);
    double *from = q.Vx, *to = V2;
    for (int it = 0; it < 2; ++it) {
      gemm_f64(c, 'T', 'N', r, r, r, 1.0, from, a.ldx, from, a.ldx, 0.0, F, r);
      k_svd_tri<<<(unsigned)std::min((r * r + 255) / 256, 4096), 256, 0, c->stream>>>(F, r);
      count_launch(c);
      copy_d2d(c, to, from, (int64_t)a.ldx * (r - 1) + r);
      gemm_f64(c, 'N', 'N', r, r, r, -1.0, from, a.ldx, F, r, 1.0, to, a.ldx);
      std::swap(from, to);
    }
    q.W = q.Wbuf;
    gemm_f64(c, 'N', 'N', mx, r, r, 1.0, two ? q.X2 : q.X, a.ldx, q.Vx, a.ldx, 0.0, q.W, a.ldx);
    check_launch(c, "svd_pre_sweeps");
  }
}

template <int R>
void svd_qrj_r(tnad_ctx* c, int np, bool symmetric, SvdArgs& a, int* info_host) {
  launch_qrcp<R, 0>(c, np, a.n, a);
  if (c->fault_once == kFaultQrTimeout) {  // failure-path test: as if a wait of the second QR had expired
    for (int p = 0; p < np; ++p) TNAD_CK(cudaMemsetAsync(a.p[p].info + kiErr, 1, sizeof(int), c->stream));
    c->fault_once = kFaultNone;
  }
  launch_qrcp<R, 1>(c, np, a.n, a);
  if (a.n >= kPreMin) pre_sweeps(c, np, a, info_host);
  int rows = 0;  // of the triangular factors
  for (int p = 0; p < np; ++p) {
    const int r = a.n >= kPreMin ? info_host[p * kiBar + kiRank] : a.n;
    rows = std::max(rows, a.second || r < a.n ? r : a.n);
  }
  if (symmetric)
    launch_sweeps<false>(c, np, rows, a);
  else
    launch_sweeps<true>(c, np, rows, a);
  const dim3 gw((unsigned)((a.n + 3) / 4), (unsigned)np), gc((unsigned)a.n, (unsigned)np);
  k_svd_norms<<<gw, 128, 0, c->stream>>>(a);
  if (symmetric) {
    k_svd_place<true><<<gc, 128, 0, c->stream>>>(a);
    k_svd_apply_q<R, true, 0><<<gw, 128, 0, c->stream>>>(a);
    count_launch(c, 3);
  } else {
    k_svd_place<false><<<gc, 128, 0, c->stream>>>(a);
    k_svd_apply_q<R, false, 0><<<gw, 128, 0, c->stream>>>(a);
    k_svd_apply_q<R, false, 1><<<gw, 128, 0, c->stream>>>(a);
    count_launch(c, 4);
  }
  check_launch(c, "svd_qrj");
}

}  // namespace

int sweeps32_eig(tnad_ctx* c, const double* A, int64_t n, const double* fro2, double* V) {
  TNAD_REQUIRE(n >= 2 && n <= kMaxSvdRows, TNAD_ERR_SHAPE, "sweeps32_eig: n must be in [2,1024]");
  WsScope scope(c);
  SvdArgs a = {};
  a.n = a.ldx = (int)n;
  a.ld32 = (int)((n + 3) & ~(int64_t)3);
  a.fro2 = fro2;
  SvdProb& q = a.p[0];
  q.A = A;
  q.W32 = ws_f(c, (int64_t)a.ld32 * n);
  q.V32 = ws_f(c, (int64_t)a.ld32 * n);
  q.Vx = V;
  q.info = (int*)c->ws.alloc(sizeof(int) * kiCount);
  TNAD_CK(cudaMemsetAsync(q.info, 0, sizeof(int) * kiCount, c->stream));
  {
    KernelTimer kt(c, "jacobi_round_f32", 0.0);
    launch_sweeps32<true>(c, 1, a);
    check_launch(c, "sweeps32_eig");
  }
  int h[kiBar];
  TNAD_CK(cudaMemcpyAsync(h, q.info, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
  TNAD_CK(cudaStreamSynchronize(c->stream));
  TNAD_REQUIRE(h[kiErr] == 0, TNAD_ERR_TIMEOUT, "sweeps32_eig: a bounded barrier wait expired");
  const int sweeps = h[kiPre] > 0 ? h[kiPre] : kEigSweeps;
  // algorithmic work: per pair 4 dot products and the rotation of W and V
  if (c->ktimer == "jacobi_round_f32") c->kt_work += 0.5 * sweeps * (double)n * (double)n * 20.0 * (double)n;
  return sweeps;
}

bool svd_qrj_fits(int64_t n) { return n >= 2 && n <= kMaxSvdRows; }

void svd_qrj(tnad_ctx* c, int np, const double* const* A, int64_t n, double* const* U, double* const* S,
             double* const* V, bool symmetric) {
  TNAD_REQUIRE(svd_qrj_fits(n) && (np == 1 || np == 2), TNAD_ERR_SHAPE, "svd_qrj: n must be in [2,1024]");
  if (np == 2 && n > 8 * (int64_t)(c->sm_count / 2)) {  // a CTA of the QR holds at most 8 columns
    svd_qrj(c, 1, A, n, U, S, V, symmetric);
    svd_qrj(c, 1, A + 1, n, U + 1, S + 1, V + 1, symmetric);
    return;
  }
  TNAD_REQUIRE(n <= 8 * (int64_t)(c->sm_count / np), TNAD_ERR_SHAPE, "svd_qrj: too many columns for this GPU");
  WsScope scope(c);
  SvdArgs a = {};
  a.n = (int)n;
  a.ldx = (int)((n + 1) & ~(int64_t)1);
  a.ldc = (int)n;
  a.ld32 = (int)((n + 3) & ~(int64_t)3);
  a.second = symmetric ? 0 : 1;
  a.trunc = 0.5f * (float)DBL_EPSILON;
  a.tol = 2.0 * std::sqrt((double)std::max<int64_t>(n, 16)) * DBL_EPSILON;
  a.tol32 = 4.0f * std::sqrt((float)n) * FLT_EPSILON;
  a.max_sweeps = kSvdSweeps;
  if (c->fault_once == kFaultJacobiCap) {  // failure-path test: one sweep only
    a.max_sweeps = 1;
    c->fault_once = kFaultNone;
  }
  const int64_t G = c->sm_count;
  // candidates, keys and counters start at zero (what an earlier call left could carry this one's tags)
  const int64_t cand = 2 * 2 * G * a.ldc;  // doubles of one problem
  const size_t nzero = (size_t)np * cand * sizeof(double) +
                       2 * (3 * G * sizeof(unsigned long long) + kiCount * sizeof(int));
  double* cands = (double*)c->ws.alloc(nzero);
  unsigned long long* zero = (unsigned long long*)(cands + np * cand);
  int* info = (int*)(zero + 2 * 3 * G);
  for (int p = 0; p < np; ++p) {
    SvdProb& q = a.p[p];
    q.A = A[p];
    q.X = ws_d(c, (int64_t)a.ldx * n);
    q.X2 = ws_d(c, (int64_t)a.ldx * n);
    const bool pre = n >= kPreMin;
    q.Vx = symmetric && !pre ? nullptr : ws_d(c, (int64_t)a.ldx * n);
    q.Wbuf = pre ? ws_d(c, (int64_t)a.ldx * n) : nullptr;
    q.W32 = pre ? ws_f(c, (int64_t)a.ld32 * n) : nullptr;
    q.V32 = pre ? ws_f(c, (int64_t)a.ld32 * n) : nullptr;
    q.H = ws_d(c, n * n);
    q.H2 = ws_d(c, n * n);
    q.hinv = ws_d(c, 2 * n);
    q.hinv2 = q.hinv + n;
    q.perm = (int*)c->ws.alloc(sizeof(int) * 2 * n);
    q.perm2 = q.perm + n;
    q.cand = cands + p * cand;
    q.key = zero + p * 3 * G;
    q.nrm = ws_d(c, n);
    q.sv = ws_d(c, n);
    q.U = U[p];
    q.S = S[p];
    q.V = symmetric ? ws_d(c, n * n) : V[p];  // the basis that k_svd_sym_basis starts from
    q.info = info + p * kiCount;
  }
  TNAD_CK(cudaMemsetAsync(cands, 0, nzero, c->stream));
  const double nn = (double)n;
  int h[2 * kiBar];
  {
    KernelTimer kt(c, "svd_qrj", np * 9.0 * nn * nn * nn, 8);
    if (n <= 64)
      svd_qrj_r<2>(c, np, symmetric, a, h);
    else if (n <= 128)
      svd_qrj_r<4>(c, np, symmetric, a, h);
    else if (n <= 256)
      svd_qrj_r<8>(c, np, symmetric, a, h);
    else if (n <= 512)
      svd_qrj_r<16>(c, np, symmetric, a, h);
    else
      svd_qrj_r<32>(c, np, symmetric, a, h);
  }
  const double couple = 8.0 * std::sqrt((double)std::max<int64_t>(n, 16)) * DBL_EPSILON;
  if (symmetric) {
    for (int p = 0; p < np; ++p) {  // DFMA products: M has to be accurate to the rounding of A
      WsScope inner(c);
      double* AX = ws_d(c, n * n);
      double* M = ws_d(c, n * n);
      gemm_f64(c, 'N', 'N', n, n, n, 1.0, A[p], n, a.p[p].V, n, 0.0, AX, n);
      gemm_f64_gram(c, n, n, a.p[p].V, AX, M);
      k_svd_sym_basis<<<(unsigned)n, 128, 0, c->stream>>>((int)n, a.p[p].V, M, S[p], couple, U[p], V[p],
                                                          a.p[p].info + kiMulti);
      count_launch(c);
      check_launch(c, "svd_sym_basis");
    }
  }
  for (int p = 0; p < np; ++p)
    TNAD_CK(cudaMemcpyAsync(h + p * kiBar, a.p[p].info, sizeof(int) * kiBar, cudaMemcpyDeviceToHost, c->stream));
  TNAD_CK(cudaStreamSynchronize(c->stream));
  for (int p = 0; p < np; ++p) {
    TNAD_REQUIRE(h[p * kiBar + kiErr] == 0, TNAD_ERR_TIMEOUT, "svd_qrj: a bounded barrier wait expired");
    TNAD_REQUIRE(h[p * kiBar + kiSweeps] > 0, TNAD_ERR_NOT_CONVERGED, "svd_qrj: no convergence within the sweep cap");
    if (std::getenv("TNAD_TRACE"))
      std::fprintf(stderr, "[tnad trace] svd_qrj n=%lld rank %d sweeps %d (FP32 %d)\n", (long long)n,
                   h[p * kiBar + kiRank], h[p * kiBar + kiSweeps], h[p * kiBar + kiPre]);
    if (symmetric && h[p * kiBar + kiMulti]) eig_separate(c, A[p], n, a.p[p].V, couple, U[p], S[p], V[p]);
  }
}

}  // namespace tnad
