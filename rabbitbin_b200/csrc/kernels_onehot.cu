// Dense regime (no abundance prune) on the tensor cores.  A register column r
// holds at most 136 distinct codes over an assembly, and far fewer in practice
// (a few tens: the elements of smallest U win most contigs), so a contig's
// codes are a short binary one-hot row X_i over the (register, code) pairs
// that occur in the assembly.  The register-match count of contigs i and j
// (src/rabbitbin.cpp:1261-1293: equal nonzero codes) is the exact integer dot
// product X_i . X_j.  Here the rows X are made; kernels_onehot_mma.cu multiplies
// them.
#include <algorithm>
#include <cstdint>

#include "rbg_internal.h"

namespace rbg {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kPresCols = 512;          // register columns per presence block (16 KB)

// Which codes occur in each register column: 256 bits per column.  A block
// takes rows_per_block rows and 512 register columns; a thread reads 4
// columns of a row at a time (mpad is a multiple of 16, so the 4-byte loads
// are aligned) and the block's two row streams run side by side.
__global__ void k_code_presence(const uint8_t *__restrict__ codesA, int64_t n, int m, int mpad,
                                int64_t rows_per_block, uint32_t *__restrict__ pres) {
  __shared__ uint32_t sp[kPresCols * 8];
  const int c0 = blockIdx.y * kPresCols;
  const int nc = (m - c0 < kPresCols) ? m - c0 : kPresCols;
  for (int i = threadIdx.x; i < kPresCols * 8; i += blockDim.x) sp[i] = 0;
  __syncthreads();
  const int64_t r0 = (int64_t)blockIdx.x * rows_per_block;
  const int64_t r1 = (r0 + rows_per_block < n) ? r0 + rows_per_block : n;
  const int cq = (threadIdx.x & 127) * 4;               // blockDim.x == 256
  if (cq < nc) {
    for (int64_t i = r0 + (threadIdx.x >> 7); i < r1; i += 2) {
      const uint32_t w4 = __ldg(reinterpret_cast<const uint32_t *>(codesA + i * mpad + c0 + cq));
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t code = (w4 >> (8 * u)) & 0xFFu;
        const int r = cq + u;
        // a column holds a few distinct codes: test before the (contended) atomic
        if (code && r < nc && !(sp[r * 8 + (code >> 5)] & (1u << (code & 31))))
          atomicOr(&sp[r * 8 + (code >> 5)], 1u << (code & 31));
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nc * 8; i += blockDim.x)
    if (sp[i]) atomicOr(&pres[(int64_t)c0 * 8 + i], sp[i]);
}

// koff[r] = one-hot columns before register r (koff[m] = K), and
// map[r][code] = koff[r] + rank of code among the column's codes (-1 absent).
// Latency-bound: a block takes kMapRegs registers (a thread one code of each)
// and counts the columns before its first one itself, rather than one block
// walking the m x 256 map (m = 500: 40 us with one block, 7 us now).
constexpr int kMapRegs = 8;
__global__ void __launch_bounds__(256) k_onehot_map(const uint32_t *__restrict__ pres, int m,
                                                    int32_t *__restrict__ map,
                                                    int32_t *__restrict__ koff) {
  __shared__ int32_t part[8];
  __shared__ int32_t cnt[kMapRegs];
  __shared__ uint32_t bits[kMapRegs * 8];
  const int t = threadIdx.x, lane = t & 31, wib = t >> 5;
  const int ra = blockIdx.x * kMapRegs, rb = min(ra + kMapRegs, m);
  int s = 0;
  for (int w = t; w < ra * 8; w += 256) s += __popc(__ldg(pres + w));
  s = (int)__reduce_add_sync(FULL, (unsigned)s);
  if (lane == 0) part[wib] = s;
  if (t < kMapRegs) cnt[t] = 0;
  __syncthreads();
  if (t < (rb - ra) * 8) {
    const uint32_t b = __ldg(pres + ra * 8 + t);
    bits[t] = b;
    atomicAdd(&cnt[t >> 3], __popc(b));
  }
  __syncthreads();
  int run = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) run += part[q];
  for (int r = ra; r < rb; ++r) {
    if (t == 0) koff[r] = run;
    const uint32_t *p = bits + (r - ra) * 8;             // warp wib holds codes 32 wib ..
    int32_t v = -1;
    if ((p[wib] >> lane) & 1u) {
      int rank = __popc(p[wib] & ((1u << lane) - 1u));
      for (int w = 0; w < wib; ++w) rank += __popc(p[w]);
      v = run + rank;
    }
    map[(int64_t)r * 256 + t] = v;
    run += cnt[r - ra];
  }
  if (rb == m && t == 0) koff[m] = run;
}

// X[i][map[r][code_i(r)]] = 1 (X zeroed by the caller; row stride ldx bytes).
__global__ void k_onehot_fill(const uint8_t *__restrict__ codesA, int64_t n, int m, int mpad,
                              const int32_t *__restrict__ map, int8_t *__restrict__ X,
                              int64_t ldx) {
  const int64_t i = blockIdx.x;                     // one row per block
  for (int r = threadIdx.x; r < m; r += blockDim.x) {
    const uint32_t code = codesA[i * mpad + r];
    if (code) X[i * ldx + __ldg(map + r * 256 + code)] = 1;
  }
}

}  // namespace

void launch_code_presence(const uint8_t *codesA, int64_t n, int m, int mpad, uint32_t *pres,
                          cudaStream_t s) {
  cudaMemsetAsync(pres, 0, (size_t)m * 8 * sizeof(uint32_t), s);
  if (n == 0) return;
  // 64 rows a block amortise its shared table; fewer while that leaves SMs idle
  const int64_t rows_per_block = std::max<int64_t>(4, std::min<int64_t>(64, n / 296));
  const dim3 grid((unsigned)((n + rows_per_block - 1) / rows_per_block),
                  (unsigned)((m + kPresCols - 1) / kPresCols));
  k_code_presence<<<grid, 256, 0, s>>>(codesA, n, m, mpad, rows_per_block, pres);
}

void launch_onehot_map(const uint32_t *pres, int m, int32_t *map, int32_t *koff, cudaStream_t s) {
  k_onehot_map<<<(unsigned)((m + kMapRegs - 1) / kMapRegs), 256, 0, s>>>(pres, m, map, koff);
}

void launch_onehot_fill(const uint8_t *codesA, int64_t n, int m, int mpad, const int32_t *map,
                        int8_t *X, int64_t ldx, cudaStream_t s) {
  cudaMemsetAsync(X, 0, (size_t)n * ldx, s);
  if (n == 0 || m == 0) return;
  k_onehot_fill<<<(unsigned)n, 256, 0, s>>>(codesA, n, m, mpad, map, X, ldx);
}

}  // namespace rbg
