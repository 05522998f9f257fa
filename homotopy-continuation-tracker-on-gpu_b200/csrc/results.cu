// results.cu -- result counts of every hypothesis of a batch, on the device.
//
// The reference's Evaluations (GPU-HC/magmaHC/Evaluations.cpp:88-110 and
// 127-176) restated for a batch, with the same rules as the host
// ghc_count_results:
//   converged / infinity   the tracker's flags;
//   real                   converged and every |Im x_v| <= imag_tol;
//   unique                 walk the paths bs in order; a converged bs outside the
//                          current skip set collects every later ds (whatever its
//                          flags) that agrees in every Re and Im within dup_tol;
//                          none -> bs counts as unique, otherwise the skip set is
//                          REPLACED by those ds and bs is not counted.
// Only the skip set makes the walk sequential; whether a path has any duplicate among the later
// ones does not depend on it.  So a group of threads (a warp for few paths, else a CTA)
// takes one hypothesis: every thread first looks for its own paths' duplicates, comparing the first
// coordinate's real part, staged in shared memory, with those of all later paths (one broadcast load
// and two FP64 operations per pair and warp, which bound it; nearly every pair ends there), and the
// group then walks the paths, 32 at a time between those that have duplicates.  B200, 12 unknowns,
// against one warp per hypothesis walking alone: 1,024 tracked hypotheses of 583 paths 2.1 ms -> 108 us; one
// hypothesis, a fiftieth of its paths on shared points, 1.42 ms -> 59 us.  A class byte per path
// (bit 0 converged, bit 1 real, bit 2 counted as unique) lets a caller compact the results without
// leaving the device.
#include <cuda_runtime.h>

#include <cstdint>

#include "ghc_internal.h"
#include "smem_limit.h"

namespace ghc {
namespace {

constexpr int kWarpPaths = 64;   // hypotheses of up to this many paths get one warp each
constexpr int kWarpPathsMany = 128;  // ... and in batches of more than kManyHyps hypotheses up to this many
constexpr long long kManyHyps = 10 * 148;
constexpr int kWarps = 4;        // such hypotheses per CTA
constexpr int kThreads = 256;    // threads of a CTA that takes one hypothesis
constexpr int kBitSets = 5;      // converged, real, has duplicates, skip set, unique
constexpr int kStagedPaths = 8192;  // up to this many paths the first coordinates fit into shared memory
constexpr int kBlock = 8;        // pairs tested between two branches
constexpr unsigned kFull = 0xffffffffu;

// duplicate sets that a CTA's warps may form ahead of the walk (at most 8 KB of them)
__host__ __device__ inline int sets_ahead(int words, int threads) {
  const int fit = 2048 / words;
  return threads == 32 ? 0 : fit < 48 ? fit : 48;
}
// shared memory of one hypothesis: first coordinates (STAGED), bit sets, the counts of paths at
// infinity and of paths with duplicates
__host__ __device__ inline size_t group_bytes(int paths, int threads, bool staged) {
  const size_t words = (size_t)(paths + 31) / 32;
  return ((staged ? 16 * 32 * words : 0) + 4 * ((kBitSets + sets_ahead((int)words, threads)) * words + 2) + 15) &
         ~(size_t)15;
}

// T threads per hypothesis (32: one of kWarps warps of the CTA; kThreads: the whole CTA)
template <int T, bool STAGED>
__global__ void __launch_bounds__((T == 32 ? 32 * kWarps : T), (T == 32 ? 8 : 5))
    results_kernel(int N, int paths, long long n_hyp, const double* __restrict__ z, const uint8_t* __restrict__ conv,
                   const uint8_t* __restrict__ inf, double imag_tol, double dup_tol, int* __restrict__ counts,
                   uint8_t* __restrict__ cls) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int kGroups = T == 32 ? kWarps : 1;
  const int lane = threadIdx.x & 31;
  const int tid = T == 32 ? lane : threadIdx.x;
  const int g = T == 32 ? threadIdx.x >> 5 : 0;
  const int words = (paths + 31) / 32;
  unsigned char* base = smem + g * group_bytes(paths, T, STAGED);
  const int padded = 32 * words;  // staged coordinates beyond the paths are NaN: they agree with nothing
  double* fre = reinterpret_cast<double*>(base);
  double* fim = fre + padded;
  unsigned* convw = reinterpret_cast<unsigned*>(STAGED ? base + 16 * (size_t)padded : base);
  unsigned* realw = convw + words;
  unsigned* dupw = realw + words;
  unsigned* skip = dupw + words;
  unsigned* uniq = skip + words;
  unsigned* ahead = uniq + words;
  const int n_ahead = sets_ahead(words, T);
  int* n_inf = reinterpret_cast<int*>(ahead + (size_t)n_ahead * words);
  int* n_dup = n_inf + 1;
  auto sync = [&]() {
    if constexpr (T == 32) __syncwarp(kFull);
    else __syncthreads();
  };
  for (long long h = (long long)blockIdx.x * kGroups + g; h < n_hyp; h += (long long)gridDim.x * kGroups) {
    const double* zh = z + 2 * h * paths * (long long)N;
    const uint8_t* ch = conv + h * paths;
    const uint8_t* ih = inf + h * paths;
    auto at = [&](int p) { return zh + 2 * (size_t)p * N; };
    auto re0 = [&](int p) { return STAGED ? fre[p] : at(p)[0]; };
    auto im0 = [&](int p) { return STAGED ? fim[p] : at(p)[1]; };
    // coordinates 1 .. N-1 of two paths agree
    auto rest_same = [&](int a, int b) {
      for (int v = 1; v < N; ++v)
        if (!(fabs(at(a)[2 * v] - at(b)[2 * v]) < dup_tol && fabs(at(a)[2 * v + 1] - at(b)[2 * v + 1]) < dup_tol))
          return false;
      return true;
    };
    // converged / infinity / real (Evaluations.cpp:88-110)
    if (tid == 0) *n_inf = *n_dup = 0;
    sync();
    for (int p = tid; p < padded; p += T) {
      const bool c = p < paths && ch[p] != 0;
      bool real = c;
      if (STAGED) {
        fre[p] = p < paths ? at(p)[0] : nan("");
        fim[p] = p < paths ? at(p)[1] : nan("");
      }
      if (p < paths) {
        for (int v = 0; v < N && real; ++v) real = fabs(at(p)[2 * v + 1]) <= imag_tol;
      }
      const unsigned mc = __ballot_sync(kFull, c), mr = __ballot_sync(kFull, real);
      const unsigned mi = __ballot_sync(kFull, p < paths && ih[p] != 0);
      if (lane == 0) {
        convw[p >> 5] = mc;
        realw[p >> 5] = mr;
        skip[p >> 5] = 0u;
        uniq[p >> 5] = 0u;
        atomicAdd(n_inf, __popc(mi));
      }
    }
    sync();
    // which converged paths have a later path on the same point
    for (int p = tid; p < padded; p += T) {
      const bool c = (convw[p >> 5] >> lane) & 1u;
      bool found = false;
      if (convw[p >> 5] != 0u) {
        const double ar = c ? re0(p) : 0.0;
        // kBlock later paths at a time: one branch for all of them
        for (int d0 = p & ~31; d0 < paths; d0 += kBlock) {
          unsigned hit = 0u;
          if (STAGED) {
#pragma unroll
            for (int u = 0; u < kBlock; u += 2) {
              const double2 v = *reinterpret_cast<const double2*>(fre + d0 + u);
              hit |= (fabs(ar - v.x) < dup_tol ? 1u << u : 0u) | (fabs(ar - v.y) < dup_tol ? 2u << u : 0u);
            }
          } else {
#pragma unroll
            for (int u = 0; u < kBlock; ++u)
              hit |= d0 + u < paths && fabs(ar - re0(d0 + u)) < dup_tol ? 1u << u : 0u;
          }
          if (hit == 0u || !c || found) continue;
          if (d0 <= p) hit &= ~1u << (p - d0);  // only later paths
          for (; hit != 0u; hit &= hit - 1u) {
            const int ds = d0 + __ffs((int)hit) - 1;
            if (fabs(im0(p) - im0(ds)) < dup_tol && rest_same(p, ds)) {
              found = true;
              break;
            }
          }
        }
      }
      const unsigned m = __ballot_sync(kFull, found);
      if (lane == 0) {
        dupw[p >> 5] = m;
        if (m != 0u) atomicAdd(n_dup, __popc(m));
      }
    }
    sync();
    // the later paths on path bs's point, in words first, first + step, ... of a set
    auto dup_set = [&](int bs, unsigned* set, int first, int step) {
      for (int j = first; j < words; j += step) {
        const int ds = 32 * j + lane;
        const bool same = ds > bs && ds < paths && fabs(re0(bs) - re0(ds)) < dup_tol &&
                          fabs(im0(bs) - im0(ds)) < dup_tol && rest_same(bs, ds);
        const unsigned b = __ballot_sync(kFull, same);
        if (lane == 0) set[j] = b;
      }
    };
    // The paths that have duplicates are few as a rule: a CTA's warps then form all their sets first, and
    // one warp walks alone.  Where they are many, most are skipped by the walk, or their sets do not fit:
    // all threads walk, and together form the set of each path that the walk reaches.  B200, 1,024
    // hypotheses of 583 paths, against at most 48 sets ahead and the rest by the walking warp: every path on
    // one point 2.26 -> 0.19 ms, a third of them on shared points 1.38 -> 1.11, a fiftieth 0.131 -> 0.124.
    const int warp = T == 32 ? 0 : (int)(threadIdx.x >> 5);
    const bool few = T != 32 && *n_dup <= n_ahead;
    if (few) {
      int at_set = 0;  // the sets in path order, one warp after the other
      for (int k = 0; k < words; ++k)
        for (unsigned d = dupw[k]; d != 0u; d &= d - 1u, ++at_set)
          if (at_set % (T / 32) == warp) dup_set(32 * k + __ffs((int)d) - 1, ahead + (size_t)at_set * words, k, 1);
      __syncthreads();
    }
    // unique (Evaluations.cpp:127-176)
    if (!few || warp == 0) {
      const unsigned* skipped = skip;  // the skip set in force (words before the walk's are not kept up)
      int nu = 0, nc = 0, nr = 0, before = 0;  // before: paths with duplicates in earlier words
      for (int k = 0; k < words; ++k) {
        unsigned left = convw[k];
        nc += __popc(left);
        nr += __popc(realw[k]);
        unsigned u = 0u;
        while (true) {
          const unsigned m = left & ~skipped[k];
          const unsigned d = m & dupw[k];
          if (d == 0u) {
            u |= m;
            break;
          }
          const unsigned low = d & (0u - d);  // the next path of this word that has duplicates
          u |= m & (low - 1u);
          if (few) {
            skipped = ahead + (size_t)(before + __popc(dupw[k] & (low - 1u))) * words;
          } else {
            sync();  // every thread has read the set that is replaced
            dup_set(32 * k + __ffs((int)low) - 1, skip, k + warp, T / 32);
            sync();
          }
          left = convw[k] & ~(low | (low - 1u));
        }
        nu += __popc(u);
        before += __popc(dupw[k]);
        if (lane == 0 && warp == 0) uniq[k] = u;
      }
      if (lane == 0 && warp == 0) {
        counts[4 * h + 0] = nc;
        counts[4 * h + 1] = nr;
        counts[4 * h + 2] = *n_inf;
        counts[4 * h + 3] = nu;
      }
    }
    sync();
    if (cls) {
      for (int p = tid; p < paths; p += T) {
        const int k = p >> 5;
        cls[h * paths + p] =
            (uint8_t)((convw[k] >> lane & 1u) | (realw[k] >> lane & 1u) << 1 | (uniq[k] >> lane & 1u) << 2);
      }
    }
    sync();
  }
}

template <int T, bool STAGED>
int launch_t(int N, int paths, long long n_hyp, const double* z, const uint8_t* conv, const uint8_t* inf,
             double imag_tol, double dup_tol, int* counts, uint8_t* cls, cudaStream_t s) {
  constexpr int kGroups = T == 32 ? kWarps : 1;
  const size_t smem = kGroups * group_bytes(paths, T, STAGED);
  if (smem > 48 * 1024 && !allow_smem<results_kernel<T, STAGED>>()) return -20;
  long long grid = (n_hyp + kGroups - 1) / kGroups;
  if (grid > 148LL * 32) grid = 148LL * 32;
  results_kernel<T, STAGED><<<(unsigned)grid, T == 32 ? 32 * kWarps : T, smem, s>>>(
      N, paths, n_hyp, z, conv, inf, imag_tol, dup_tol, counts, cls);
  return cudaGetLastError() == cudaSuccess ? 0 : -23;
}

}  // namespace

int launch_results(int N, int paths, long long n_hyp, const double* z, const uint8_t* conv, const uint8_t* inf,
                   double imag_tol, double dup_tol, int* counts, uint8_t* cls, void* stream) {
  if (n_hyp <= 0 || paths <= 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  // A warp per hypothesis up to kWarpPaths paths, where a CTA's threads would idle, and up to
  // kWarpPathsMany where the CTAs would come in several waves (128 paths, a fiftieth of them on shared
  // points, 1 / 1,184 / 3,000 hypotheses: by CTA 21 / 31 / 56 us, by warp 26 / 28 / 37); above kStagedPaths the
  // first coordinates are read where they are.
  if (paths <= kWarpPaths || (paths <= kWarpPathsMany && n_hyp > kManyHyps))
    return launch_t<32, true>(N, paths, n_hyp, z, conv, inf, imag_tol, dup_tol, counts, cls, s);
  if (paths <= kStagedPaths)
    return launch_t<kThreads, true>(N, paths, n_hyp, z, conv, inf, imag_tol, dup_tol, counts, cls, s);
  return launch_t<kThreads, false>(N, paths, n_hyp, z, conv, inf, imag_tol, dup_tol, counts, cls, s);
}

}  // namespace ghc
