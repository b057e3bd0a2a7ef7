// kc_fold.cuh — ((0 + v[0]) + v[1]) + ... with the serial sum's bits, in parallel.
//
// A serial fold of n terms is n dependent FP64 additions: 16 ms for the 2.2 M
// mass terms of the 192x180x64 wedge, a quarter of a time step. But while the running sum
// stays inside one binade [2^e, 2^(e+1)) every addition is one of integers: the
// sum is a multiple of its ulp 2^(e-52), and adding v moves it by v / ulp rounded
// to the nearest integer; only a tie looks at the sum, and there only at its
// parity. So a run of terms is the map parity -> (move, parity after), two
// integers, and such maps compose associatively. The fold then is
//   k_fold_sums    the plain sum of every chunk of terms (an estimate of the
//                  running sum, which says which binade each chunk meets),
//   k_fold_exact   each chunk's map in that binade, with bounds on how far the
//                  running sum can go up or down inside it,
//   k_fold_finish  one warp that applies the maps in order: exact where the
//                  running sum is in the chunk's binade and cannot leave it by
//                  the bounds; any other chunk (the first, the few that cross a
//                  binade, a non-finite term) it adds term by term.
// Measured: the wedge's sums 16 ms to 0.5 ms a row of diagnostics, the 384x360
// grid's 0.86 to about 0.3 ms.
#pragma once
#include <math.h>

#include "../../include/koral/kmath.h"

namespace kc {

// the move of a sum of either parity, in ulps
struct FoldMap {
  long long d0, d1;
};
KC_HD FoldMap fold_then(const FoldMap& a, const FoldMap& b) {
  FoldMap r;
  r.d0 = a.d0 + ((a.d0 & 1) ? b.d1 : b.d0);
  r.d1 = a.d1 + ((a.d1 & 1) ? b.d0 : b.d1);  // parity after: 1 + d1
  return r;
}
// what a chunk's fold needs of its terms; lo, hi: how far the sum can fall, rise
struct FoldRun {
  FoldMap m;
  long long lo, hi;
  int ok;
};
KC_HD FoldRun fold_empty() {
  FoldRun r = {{0, 0}, 0, 0, 1};
  return r;
}
KC_HD FoldRun fold_join(const FoldRun& a, const FoldRun& b) {
  FoldRun r = {fold_then(a.m, b.m), a.lo + b.lo, a.hi + b.hi, a.ok & b.ok};
  return r;
}
// one term x = v / ulp (the scaling by a power of two is exact, or x is far below
// one half)
KC_HD FoldRun fold_term(double x) {
  FoldRun r = fold_empty();
  if (!(x < 0x1p+50 && x > -0x1p+50)) {
    r.ok = 0;
    return r;
  }
  // the midpoint f + 1/2 is exact for every |x| < 2^50; x - f is not (for x just
  // above -1/2 it rounds to 1/2, which would make a tie of x)
  const double f = ::floor(x), mid = f + 0.5;
  const long long F = (long long)f;
  if (x == mid) {
    // to the even sum
    r.m.d0 = F + (F & 1);
    r.m.d1 = F + ((F + 1) & 1);
  } else {
    r.m.d0 = r.m.d1 = F + (x > mid);
  }
  r.lo = F < 0 ? -F : 0;
  r.hi = F >= 0 ? F + 1 : 0;
  return r;
}
// A chunk as k_fold_exact leaves it: valid for a running sum of the sign and
// binade of `key` (its sign and exponent bits; 0: not valid)
struct FoldChunk {
  FoldMap m;
  long long lo, hi, key;
};
KC_HD long long fold_key(double acc) {
  const long long b = (long long)(kmath::to_bits(acc) >> 52);  // sign and exponent
  const long long e = b & 0x7ff;
  return e < 64 || e > 1980 ? 0 : b;  // away from subnormals and infinity
}
// 2^(52-e) with the sign of the sum: v times it is the term in ulps of a positive sum
KC_HD double fold_scale(long long key) {
  const double s = kmath::from_bits((uint64_t)(1023 + 52 + 1023 - (key & 0x7ff)) << 52);
  return (key & 0x800) ? -s : s;
}
// the chunk's fold of acc; false where it does not apply
KC_HD bool fold_apply(double& acc, const FoldChunk& c) {
  if (c.key == 0 || (long long)(kmath::to_bits(acc) >> 52) != c.key) return false;
  const long long one = 1LL << 52;
  long long a = (long long)(kmath::to_bits(acc) & (uint64_t)(one - 1)) + one;
  if (a - c.lo <= one || a + c.hi >= 2 * one) return false;
  a += (a & 1) ? c.m.d1 : c.m.d0;
  acc = kmath::from_bits(((uint64_t)c.key << 52) | (uint64_t)(a - one));
  return true;
}

#if defined(__CUDACC__)
constexpr int FOLD_TPB = 128, FOLD_PER = 8, FOLD_CHUNK = FOLD_TPB * FOLD_PER;
constexpr int FOLD_JOBS = 4;
constexpr long FOLD_SERIAL = 2048;  // up to here the finishing warp folds the terms alone
struct FoldJobs {
  const double* v[FOLD_JOBS];
  double* out[FOLD_JOBS];
  long n[FOLD_JOBS];
  long chunk0[FOLD_JOBS];  // the job's first chunk in the scratch arrays
};
__host__ __device__ inline long fold_chunks(long n) { return (n + FOLD_CHUNK - 1) / FOLD_CHUNK; }

__global__ void __launch_bounds__(FOLD_TPB) k_fold_sums(FoldJobs J, double* sums) {
  const int job = blockIdx.y;
  const long n = J.n[job], k0 = (long)blockIdx.x * FOLD_CHUNK;
  if (k0 >= n) return;
  double s = 0.0;
  for (long k = k0 + threadIdx.x; k < n && k < k0 + FOLD_CHUNK; k += FOLD_TPB) s += J.v[job][k];
  for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  __shared__ double w[FOLD_TPB / 32];
  if (threadIdx.x % 32 == 0) w[threadIdx.x / 32] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < FOLD_TPB / 32; ++i) s += w[i];
    sums[J.chunk0[job] + blockIdx.x] = s;
  }
}
__device__ __forceinline__ FoldRun fold_shfl_down(const FoldRun& r, int o) {
  FoldRun x;
  x.m.d0 = __shfl_down_sync(0xffffffffu, r.m.d0, o);
  x.m.d1 = __shfl_down_sync(0xffffffffu, r.m.d1, o);
  x.lo = __shfl_down_sync(0xffffffffu, r.lo, o);
  x.hi = __shfl_down_sync(0xffffffffu, r.hi, o);
  x.ok = __shfl_down_sync(0xffffffffu, r.ok, o);
  return x;
}
__global__ void __launch_bounds__(FOLD_TPB) k_fold_exact(FoldJobs J, const double* sums, FoldChunk* chunks) {
  const int job = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long n = J.n[job], k0 = (long)blockIdx.x * FOLD_CHUNK;
  if (k0 >= n) return;
  __shared__ double w[FOLD_TPB / 32], v[FOLD_CHUNK];
  __shared__ FoldRun run[FOLD_TPB / 32];
  // the running sum before this chunk, nearly
  const double* sj = sums + J.chunk0[job];
  double s = 0.0;
  for (long k = tid; k < blockIdx.x; k += FOLD_TPB) s += sj[k];
  for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) w[warp] = s;
  for (int k = tid; k < FOLD_CHUNK; k += FOLD_TPB) v[k] = k0 + k < n ? J.v[job][k0 + k] : 0.0;
  __syncthreads();
  s = 0.0;
  for (int i = 0; i < FOLD_TPB / 32; ++i) s += w[i];
  const long long key = fold_key(s);
  FoldChunk c = {{0, 0}, 0, 0, 0};
  if (key) {
    const double scale = fold_scale(key);
    FoldRun r = fold_empty();
    for (int i = 0; i < FOLD_PER; ++i) r = fold_join(r, fold_term(v[tid * FOLD_PER + i] * scale));
    for (int o = 1; o < 32; o <<= 1) {
      const FoldRun x = fold_shfl_down(r, o);
      if (lane + o < 32 && lane % (2 * o) == 0) r = fold_join(r, x);
    }
    if (lane == 0) run[warp] = r;
    __syncthreads();
    if (tid == 0) {
      for (int i = 1; i < FOLD_TPB / 32; ++i) r = fold_join(r, run[i]);
      c = {r.m, r.lo, r.hi, r.ok ? key : 0};
    }
  }
  if (tid == 0) chunks[J.chunk0[job] + blockIdx.x] = c;
}
// One warp per job. serial: no chunk maps were formed (short jobs).
__global__ void __launch_bounds__(32) k_fold_finish(FoldJobs J, const FoldChunk* chunks, int serial) {
  __shared__ double tile[FOLD_CHUNK];
  __shared__ FoldChunk cs[32];
  const int job = blockIdx.x, lane = threadIdx.x;
  const long n = J.n[job], nch = fold_chunks(n);
  double acc = 0.0;
  for (long c0 = 0; c0 < nch; c0 += 32) {
    if (!serial && c0 + lane < nch) cs[lane] = chunks[J.chunk0[job] + c0 + lane];
    __syncwarp();
    const int m = nch - c0 < 32 ? (int)(nch - c0) : 32;
    for (int i = 0; i < m; ++i) {
      if (!serial && fold_apply(acc, cs[i])) continue;
      const long k0 = (c0 + i) * FOLD_CHUNK;
      const int cnt = n - k0 < FOLD_CHUNK ? (int)(n - k0) : FOLD_CHUNK;
      for (int k = lane; k < FOLD_CHUNK; k += 32) tile[k] = k < cnt ? J.v[job][k0 + k] : 0.0;
      __syncwarp();
      // in pieces of 128 terms, by the map of the running sum's own binade where it
      // holds: only the piece that crosses a binade is added term by term
      for (int q = 0; q < cnt; q += 128) {
        const long long key = fold_key(acc);
        if (key) {
          const double scale = fold_scale(key);
          FoldRun r = fold_empty();
          for (int k = 0; k < 4; ++k) r = fold_join(r, fold_term(tile[q + lane * 4 + k] * scale));
          for (int o = 1; o < 32; o <<= 1) {
            const FoldRun x = fold_shfl_down(r, o);
            if (lane % (2 * o) == 0) r = fold_join(r, x);
          }
          FoldChunk c;
          c.m.d0 = __shfl_sync(0xffffffffu, r.m.d0, 0);
          c.m.d1 = __shfl_sync(0xffffffffu, r.m.d1, 0);
          c.lo = __shfl_sync(0xffffffffu, r.lo, 0);
          c.hi = __shfl_sync(0xffffffffu, r.hi, 0);
          c.key = __shfl_sync(0xffffffffu, r.ok, 0) ? key : 0;
          if (fold_apply(acc, c)) continue;
        }
        const int end = q + 128 < cnt ? q + 128 : cnt;
#pragma unroll 8
        for (int k = q; k < end; ++k) acc += tile[k];
      }
      __syncwarp();
    }
    __syncwarp();
  }
  if (lane == 0) *J.out[job] = acc;
}
#endif

}  // namespace kc
