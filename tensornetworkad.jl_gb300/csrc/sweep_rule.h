// Stop rule of the FP32 Jacobi sweeps with the eigenvalue rule (svd_qr.cu,
// k_sweeps32<EIG>), apart from the kernel so that a host compiler can check it.
#pragma once

#ifdef __CUDACC__
#define TNAD_HOST_DEVICE __host__ __device__
#else
#define TNAD_HOST_DEVICE
#endif

namespace tnad {

// Rotations up to which a sweep over n columns was the last one: 16n, but not more
// than an eighth of the pairs.  16n is 3% of them at n = 1024 and half of them at
// n = 65 (the smallest group of clustered eigenvalues that is solved this way),
// where graded groups stopped at 1e-5 of their norm; by this rule ~1e-6 or less
// at every n, at the price of one sweep for those.  From n = 257 on it is 16n.
TNAD_HOST_DEVICE inline int eig_sweep_last(int n) {
  const int pairs8 = n * (n - 1) / 16;
  return 16 * n < pairs8 ? 16 * n : pairs8;
}

}  // namespace tnad
