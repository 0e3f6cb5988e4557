// dg_lu.cuh -- the LU factorisation of an affine Gauss-Newton Hessian by one
// warp.  It stands alone (the warp intrinsics are all that it takes from CUDA),
// so that tests/cpp/lu_lanes.cpp can run it on the CPU with the lanes in any
// order between two synchronising calls.
#pragma once

namespace dg {

// LU with partial pivoting of the N x N matrix H (row major, N <= 6) in place:
// the unblocked DGETRF steps, IDAMAX, the row swap, the scaling by the pivot's
// reciprocal, the rank-1 update.  Lane l updates entry (1 + l / 5, 1 + l mod 5);
// the pivot is found by reductions over the lanes (the first largest
// magnitude; a NaN is taken only where it stands first, as IDAMAX's comparisons
// leave it).  `pos` becomes the row of the unit entry of P e_lane.  Returns 0,
// or one more than the first column with a zero pivot.  It waits for shared
// memory and the division: 4.1 k cycles at N = 6 (the rows in registers, with
// shuffles, took 4.6 k).
__device__ __forceinline__ int lu_affine(double* H, const int N, const int lane, int& pos) {
  const unsigned full = 0xffffffffu;
  const int ri = 1 + lane / 5, ck = 1 + lane % 5;
  int info = 0;
  pos = lane;
#pragma unroll 1
  for (int j = 0; j < N; ++j) {
    unsigned long long key = 0ull;
    if (lane >= j && lane < N) {
      key = (unsigned long long)__double_as_longlong(H[lane * N + j]) & 0x7fffffffffffffffull;
      if (key > 0x7ff0000000000000ull && lane != j) key = 0ull;
    }
    const unsigned kh = (unsigned)(key >> 32), mh = __reduce_max_sync(full, kh);
    const unsigned kl = kh == mh ? (unsigned)key : 0u, ml = __reduce_max_sync(full, kl);
    const int p = __ffs(__ballot_sync(full, lane >= j && lane < N && kh == mh && kl == ml)) - 1;
    const double pv = H[p * N + j];
    __syncwarp();   // every lane has its pivot before the swap writes over it
    if (pos == j) pos = p;
    else if (pos == p) pos = j;
    if (pv != 0.0) {
      const double rp = 1.0 / pv;
      if (p != j && lane < N) {
        const double t = H[j * N + lane];
        H[j * N + lane] = H[p * N + lane];
        H[p * N + lane] = t;
      }
      __syncwarp();
      if (lane > j && lane < N) H[lane * N + j] = H[lane * N + j] * rp;
    } else if (info == 0) {
      info = j + 1;
    }
    __syncwarp();
    if (ri > j && ck > j && ri < N && ck < N) H[ri * N + ck] = H[ri * N + ck] - H[ri * N + j] * H[j * N + ck];
    __syncwarp();
  }
  return info;
}

}  // namespace dg
