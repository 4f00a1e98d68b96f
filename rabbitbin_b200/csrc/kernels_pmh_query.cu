// ProbMinHash4 sketch rows and sketch-vs-sketch queries on the device: the
// batch counterparts of ProbMinHash4::getWinners / getRegisters,
// jaccard_weighted, jaccard, distance, ani and merge (src/probmh.h:103-283,
// src/probmh.cpp:1325-1440).
//
// A sketch row is m 64-bit words: the winners (RNG state of the element that
// won each register, 0 when unset) or the register values (doubles, +inf when
// unset).  A comparison counts the registers whose words are equal and set --
// jaccard_weighted on winners (:1364-1376), jaccard on register values
// (:1325-1362, exact double equality) -- and maps the count through a table of
// m + 1 doubles the host made with the reference's own formulas (count / m,
// and the distance / ANI transforms of it with the host's libm), so every
// value equals the reference's bit for bit.
#include <algorithm>
#include <cstdint>

#include "rbg_internal.h"

namespace rbg {
namespace {

__global__ void k_pmh_rows(const uint8_t *__restrict__ win_elem,
                           const double *__restrict__ elem_winv, int64_t n, int m, int E,
                           const uint64_t *__restrict__ W64, const double *__restrict__ U,
                           uint64_t *__restrict__ w64_out, double *__restrict__ reg_out) {
  const int64_t total = n * (int64_t)m;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < total;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = q / m;
    const int r = (int)(q - c * m);
    const uint32_t e = win_elem[q];
    uint64_t w = 0;
    double v = __longlong_as_double(0x7ff0000000000000ll);     // +inf
    if (e != 0xFFu) {
      w = __ldg(W64 + (size_t)e * m + r);
      // the same rounded product the register minimum compared
      v = __dmul_rn(__ldg(elem_winv + c * E + e), __ldg(U + (size_t)e * m + r));
    }
    if (w64_out) w64_out[q] = w;
    if (reg_out) reg_out[q] = v;
  }
}

// A word as compared: register values that are not numbers never match (they take
// the pattern of an unset register), and zeros have one sign, so that equal
// doubles are equal bits.
template <bool REGS>
__device__ __forceinline__ uint64_t canonical(uint64_t w) {
  if (REGS) {
    const double x = __longlong_as_double((long long)w);
    if (x != x) return 0x7ff0000000000000ull;
    if (x == 0.0) return 0ull;
  }
  return w;
}

// CTA: a T x T tile of (A row, B row) pairs; thread (tx, ty) owns the pairs (ty + 16 u,
// tx + 16 v), u, v < T / 16.  Chunks of QC registers of A and B rows are staged in
// shared memory, the next chunk's words loading meanwhile.
//
// T = 64, QC = 16: bound by the integer pipe (76% busy, issue 82%): two half-word
// comparisons and a count a pair and register.  1,000 x 4,999 rows, m = 1,000: 1.16 ms
// with 4 pairs a thread and both words tested for every pair, 1.00 ms now.  Few rows
// leave most SMs idle and are bound by the chain of chunks, so they take smaller
// tiles of longer chunks (launch_pmh_compare).
template <bool REGS, int T, int QC>
__global__ void __launch_bounds__(256)
k_pmh_compare(const uint64_t *__restrict__ A, int64_t na, const uint64_t *__restrict__ B,
              int64_t nb, int m, const double *__restrict__ table, double *__restrict__ out) {
  constexpr int QS = QC + 2;                     // words of a staged row: 16-byte reads of 8
                                                 // rows hit every bank
  constexpr int P = T / 16;                      // pairs of a thread, a side
  constexpr int kPer = T * QC / 256;             // words of A and of B a thread stages
  constexpr int kRows = 256 / QC;                // rows that the threads stage at a time
  static_assert(kPer * kRows == T, "a thread stages one column of rows kRows apart");
  __shared__ __align__(16) uint64_t sa[2][T][QS], sb[2][T][QS];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int sc = threadIdx.x % QC, sr = threadIdx.x / QC;
  const int64_t a0 = (int64_t)blockIdx.y * T, b0 = (int64_t)blockIdx.x * T;
  int cnt[P][P] = {};
  const uint64_t unset = REGS ? 0x7ff0000000000000ull : 0ull;
  uint64_t ra[kPer], rb[kPer];
  // the next chunk's words load while a chunk is compared
  auto fetch = [&](int k0) {
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int row = sr + kRows * t, col = k0 + sc;
      ra[t] = (col < m && a0 + row < na) ? __ldg(A + (a0 + row) * m + col) : unset;
      rb[t] = (col < m && b0 + row < nb) ? __ldg(B + (b0 + row) * m + col) : unset;
    }
  };
  fetch(0);
  int s = 0;
  for (int k0 = 0; k0 < m; k0 += QC, s ^= 1) {
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      sa[s][sr + kRows * t][sc] = canonical<REGS>(ra[t]);
      sb[s][sr + kRows * t][sc] = canonical<REGS>(rb[t]);
    }
    __syncthreads();
    if (k0 + QC < m) fetch(k0 + QC);
#pragma unroll 2
    for (int k = 0; k < QC; k += 2) {
      ulonglong2 b[P];
#pragma unroll
      for (int v = 0; v < P; ++v) b[v] = *reinterpret_cast<const ulonglong2 *>(&sb[s][tx + 16 * v][k]);
#pragma unroll
      for (int u = 0; u < P; ++u) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(&sa[s][ty + 16 * u][k]);
        const bool set0 = a.x != unset, set1 = a.y != unset;
#pragma unroll
        for (int v = 0; v < P; ++v) {
          if (set0 && a.x == b[v].x) ++cnt[u][v];
          if (set1 && a.y == b[v].y) ++cnt[u][v];
        }
      }
    }
  }
#pragma unroll
  for (int u = 0; u < P; ++u)
#pragma unroll
    for (int v = 0; v < P; ++v) {
      const int64_t i = a0 + ty + 16 * u, j = b0 + tx + 16 * v;
      if (i < na && j < nb) out[i * nb + j] = __ldg(table + cnt[u][v]);
    }
}

template <int T, int QC>
void launch_compare_tiles(const uint64_t *A, int64_t na, const uint64_t *B, int64_t nb, int m,
                          bool regs, const double *table, double *out, cudaStream_t s) {
  const dim3 grid((unsigned)((nb + T - 1) / T), (unsigned)((na + T - 1) / T));
  if (regs) k_pmh_compare<true, T, QC><<<grid, 256, 0, s>>>(A, na, B, nb, m, table, out);
  else k_pmh_compare<false, T, QC><<<grid, 256, 0, s>>>(A, na, B, nb, m, table, out);
}

__global__ void k_pmh_merge(const double *__restrict__ a, const double *__restrict__ b,
                            int64_t count, double *__restrict__ out) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < count;
       q += (int64_t)gridDim.x * blockDim.x) {
    const double x = a[q], y = b[q];
    out[q] = (y < x) ? y : x;                 // std::min(x, y)
  }
}

}  // namespace

void launch_pmh_rows(const uint8_t *win_elem, const double *elem_winv, int64_t n, int m, int E,
                     const uint64_t *W64, const double *U, uint64_t *w64_out, double *reg_out,
                     cudaStream_t s) {
  const int64_t total = n * (int64_t)m;
  if (total == 0) return;
  const int64_t blocks = std::min<int64_t>((total + 255) / 256, 148 * 16);
  k_pmh_rows<<<(unsigned)blocks, 256, 0, s>>>(win_elem, elem_winv, n, m, E, W64, U, w64_out,
                                              reg_out);
}

void launch_pmh_compare(const uint64_t *A, int64_t na, const uint64_t *B, int64_t nb, int m,
                        bool regs, const double *table, double *out, cudaStream_t s) {
  if (na == 0 || nb == 0) return;
  const int64_t c64 = (na + 63) / 64 * ((nb + 63) / 64), c32 = (na + 31) / 32 * ((nb + 31) / 32);
  const int64_t few = std::min(na, nb);
  // A call in tiles of 64 / 32 / 16 (winner rows, m registers, ms): 1 x 1 (m = 1,000) 0.164 /
  // 0.092 / 0.074, 65 x 65 (4,000) 0.603 / 0.319 / 0.247, 10 x 300 (1,000) 0.219 / 0.143 /
  // 0.125, 1 x 20,000 (500) 1.68 / 1.61 / 1.59, 300 x 300 (1,000) 0.395 / 0.320 / 0.322,
  // 500 x 500 (1,000) 0.341 / 0.299 / 0.342, 700 x 700 (500) 0.277 / 0.289 / 0.325,
  // 1,000 x 4,999 (1,000) 2.20 / 2.44 / 3.42
  if (few > 32 && c64 >= 100) launch_compare_tiles<64, 16>(A, na, B, nb, m, regs, table, out, s);
  else if (few > 16 && c32 > 100) launch_compare_tiles<32, 32>(A, na, B, nb, m, regs, table, out, s);
  else launch_compare_tiles<16, 64>(A, na, B, nb, m, regs, table, out, s);
}

void launch_pmh_merge(const double *a, const double *b, int64_t count, double *out,
                      cudaStream_t s) {
  if (count == 0) return;
  const int64_t blocks = std::min<int64_t>((count + 255) / 256, 148 * 16);
  k_pmh_merge<<<(unsigned)blocks, 256, 0, s>>>(a, b, count, out);
}

}  // namespace rbg
