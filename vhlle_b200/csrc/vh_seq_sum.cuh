// vh_seq_sum.cuh -- the ordered sum of the initial states' normalisations
// (src/icGlissando.cpp:164-181, src/icTrento.cpp:185-202: over the cells in
// loop order).
#pragma once

#include "vh_crmath.cuh"

namespace vh {
namespace icr {

// sum of t[0..n) from 0.0 in index order, rounded after every addition as
// the host loop, without its chain of additions.
//
// While the running sum s stays in one binade [2^k, 2^(k+1)) it is a whole
// number of u = 2^(k-52), and RN(s + t) = s + RN_u(t), t rounded to a
// multiple of u: the same for every s there, unless t lies halfway between
// two multiples (the tie goes by the last bit of s).  So the additions of a
// run of non-negative terms without ties, as long as their sum stays below
// 2^(k+1), are a sum of whole numbers below 2^53, in any order.  A sub-tile
// (the 256 terms of a warp) with a tie, a negative or non-finite term, or
// the step into the next binade is added term by term; over n terms of one
// size that happens about ln n times for ties and log2 n times for binades.
// One block, since each tile needs the sum before it.  A warp whose terms are
// all zeros skips the arithmetic, and a chain takes the non-zero terms only.
// 520,251 terms take 148 us, and 977 as a chain of additions (181 with the
// zeros treated as any term; 4 terms per thread and tile instead of 8 made a
// call 15 % slower).
constexpr int kSumThreads = 1024;
constexpr int kSumPer = 8;                       // terms per thread and tile
constexpr int kSumRun = 32 * kSumPer;            // a sub-tile
constexpr int kSumTile = kSumThreads * kSumPer;  // 32 sub-tiles

__global__ void __launch_bounds__(kSumThreads) k_seq_sum(const double* __restrict__ t, long long n,
                                                         double* __restrict__ out) {
  __shared__ double wsum[32], chain[kSumRun];
  __shared__ int wbad[32];
  __shared__ double s_sh;
  __shared__ int pos_sh;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double s = 0.0, v[kSumPer];
  auto load = [&](long long tile, double* x) {
    const long long base = tile * kSumTile + warp * kSumRun + lane;
#pragma unroll
    for (int r = 0; r < kSumPer; r++) {
      const long long k = base + 32 * r;
      x[r] = k < n ? t[k] : 0.0;
    }
  };
  const long long ntile = (n + kSumTile - 1) / kSumTile;
  load(0, v);
  for (long long tile = 0; tile < ntile; tile++) {
    double next[kSumPer];
    load(tile + 1, next);  // (zeros past the end)
    bool with = false;
#pragma unroll
    for (int r = 0; r < kSumPer; r++) with |= v[r] != 0.0;
    with = __any_sync(0xffffffffu, with);
    int pos = 0;           // the first sub-tile not added yet
    while (pos < 32) {
      // s in whole numbers of its last bit; s = 0 takes zero terms only
      const int ex = (int)((unsigned long long)__double_as_longlong(s) >> 52);  // sign included
      const bool fit = ex >= 60 && ex <= 1980;
      const double scale = fit ? crm::pow2i(52 + 1023 - ex) : 0.0;
      const double u = fit ? crm::pow2i(ex - 1023 - 52) : 0.0;
      double sum = 0.0;
      bool bad = !fit && s != 0.0;
      if (with) {  // (the warp's terms are not all zeros)
#pragma unroll
        for (int r = 0; r < kSumPer; r++) {
          const double x = v[r] * scale, w = rint(x);
          sum += w;
          bad |= fit ? !(v[r] >= 0.0 && x < 0x1p51) || fabs(x - w) == 0.5 : v[r] != 0.0;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      }
      const unsigned any = __ballot_sync(0xffffffffu, bad);
      if (lane == 0) {
        wsum[warp] = sum;
        wbad[warp] = any != 0;
      }
      __syncthreads();
      if (warp == 0) {
        double run = lane >= pos ? wsum[lane] : 0.0;  // inclusive prefix sums
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const double x = __shfl_up_sync(0xffffffffu, run, o);
          if (lane >= o) run += x;
        }
        const double S = s * scale;
        const bool stop = lane >= pos && (wbad[lane] || !(S + run < 0x1p53));
        const unsigned st = __ballot_sync(0xffffffffu, stop);
        const int f = st ? __ffs((int)st) - 1 : 32;  // the first sub-tile to add term by term
        const double before = __shfl_sync(0xffffffffu, run, f > 0 ? f - 1 : 0);
        if (f > pos) s = fit ? (S + before) * u : s;
        if (lane == 0) {
          s_sh = s;
          pos_sh = f;
        }
      }
      __syncthreads();
      pos = pos_sh;
      if (warp == pos) {  // its own sub-tile, from its registers
        int m = 0;  // without the zeros, which leave any sum as it is (s = -0 cannot be)
#pragma unroll
        for (int r = 0; r < kSumPer; r++) {
          const unsigned b = __ballot_sync(0xffffffffu, v[r] != 0.0);
          if (v[r] != 0.0) chain[m + __popc(b & ((1u << lane) - 1u))] = v[r];
          m += __popc(b);
        }
        __syncwarp();
        if (lane == 0) {
          s = s_sh;
#pragma unroll 16
          for (int j = 0; j < m; j++) s += chain[j];
          s_sh = s;
        }
      }
      __syncthreads();
      s = s_sh;
      pos++;
    }
#pragma unroll
    for (int r = 0; r < kSumPer; r++) v[r] = next[r];
  }
  if (threadIdx.x == 0) out[0] = s;
}

}  // namespace icr
}  // namespace vh
