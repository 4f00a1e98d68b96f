// All-pairs pass: per row top-K of (similarity, id) keys plus the row maxima
// the calibration reads, over full rows (every ordered pair i != j).
//
// A work item is a block of 32 rows (lane = row) against kWarps column slices,
// one warp per slice; the plain launch maps items to the grid, the batch form
// runs a persistent kernel that pulls (assembly, row block, slice group)
// items from a device counter.  Each row keeps its candidate keys in a
// private global buffer per slice (L2-resident) with the admission threshold
// and fill count in shared memory; when a buffer fills, the owning warp
// selects the K best in registers (radix search of the K-th largest key) and
// raises the threshold to it.  A merge pass then keeps the K best over the
// slices.
//
// Two regimes:
//  * dense (no abundance prune: the N <= 25000 path, S <= 2, RABBIT_NO_ABDFIRST):
//    every pair's register-match count, 4 columns per step over 8-bit code
//    words (row words from shared memory, column words staged by cp.async);
//  * sparse (the abundance-first prune of the fused path): tensor-core FP16
//    products of the unit rows prune almost every pair under a rigorous error
//    bound; the few left are decided by an FP32 chain with its own band and
//    then the AVX-512 order of unit_dot_f exactly.  Survivors queue per warp
//    and are counted by the whole warp, one survivor at a time.
//
// Compiled with -fmad=false; __fmaf_rn marks every fused operation.
#include <algorithm>
#include <cstdint>
#include <cuda_fp16.h>

#include "rbg_internal.h"
#include "scan.cuh"
#include "select_topk.cuh"
#include "sim_bins.cuh"

namespace rbg {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kWarps = 4;         // warps per CTA (independent)

// One 16-byte shared-memory load (a single 128-bit access: lanes reading
// consecutive 16-byte blocks take 4 wavefronts for the warp, where four 32-bit
// loads of the same blocks would conflict 4-way each).  Volatile, so it stays
// ordered after the cp.async waits and warp barriers around it.
__device__ __forceinline__ uint4 lds128(const void *p) {
  uint4 v;
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(a));
  return v;
}

// Row stride (floats) of the unit rows staged in shared memory: an odd number
// of 16-byte units, so lanes gathering rows of random indices spread over all
// eight 16-byte bank groups.
__host__ __device__ __forceinline__ int su_stride(int Su) {
  return ((Su >> 2) & 1) ? Su : Su + 4;
}

// 0x80 in each byte where a and b agree, 0 elsewhere: the low seven bits of
// each byte of a ^ b are tested by an add that cannot carry out of the byte,
// the top bit directly.
__device__ __forceinline__ uint32_t eq_mask(uint32_t a, uint32_t b) {
  const uint32_t x = a ^ b;
  const uint32_t t = (x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu;
  return ~(t | x) & 0x80808080u;
}
// acc + 128 x (number of equal bytes of two 16-byte blocks); the byte dot
// product with 0x01010101 sums the masks on the FMA pipe, beside the ALU
// work of the masks.
__device__ __forceinline__ uint32_t eq16(const uint4 a, const uint4 b, uint32_t acc) {
  acc = __dp4a(eq_mask(a.x, b.x), 0x01010101u, acc);
  acc = __dp4a(eq_mask(a.y, b.y), 0x01010101u, acc);
  acc = __dp4a(eq_mask(a.z, b.z), 0x01010101u, acc);
  return __dp4a(eq_mask(a.w, b.w), 0x01010101u, acc);
}

// unit_dot_f (src/rabbitbin.cpp:754-796) as an AVX-512 build evaluates it:
// element t feeds lane t % 16 of acc1 in the upper half of a full 32-element
// block, else of acc0 (the masked tail included); then acc0 + acc1 and the
// _mm512_reduce_add_ps tree (lanes i + i+8, i + i+4, i + i+2, 0 + 1).
template <int SMAX>
__device__ __forceinline__ float dot_avx512(const float (&a)[SMAX], const float *b, int S) {
  float acc0[16], acc1[16];
#pragma unroll
  for (int l = 0; l < 16; ++l) { acc0[l] = 0.f; acc1[l] = 0.f; }
  const int lim32 = S & ~31;
#pragma unroll
  for (int t = 0; t < SMAX; ++t) {
    if (t < S) {
      const float bt = __ldg(b + t);
      if ((t & 16) && t < lim32) acc1[t & 15] = __fmaf_rn(a[t], bt, acc1[t & 15]);
      else acc0[t & 15] = __fmaf_rn(a[t], bt, acc0[t & 15]);
    }
  }
  float v[16];
#pragma unroll
  for (int l = 0; l < 16; ++l) v[l] = lim32 ? __fadd_rn(acc0[l], acc1[l]) : acc0[l];
#pragma unroll
  for (int l = 0; l < 8; ++l) v[l] = __fadd_rn(v[l], v[l + 8]);
#pragma unroll
  for (int l = 0; l < 4; ++l) v[l] = __fadd_rn(v[l], v[l + 4]);
  v[0] = __fadd_rn(v[0], v[2]);
  v[1] = __fadd_rn(v[1], v[3]);
  return __fadd_rn(v[0], v[1]);
}

// 16-byte asynchronous global->shared copies (per lane), and their groups.
__device__ __forceinline__ void cp16(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_wait1() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

// Survivor entries of k_sym_check: row of the block << 27 | kHiBit when both
// rows hold codes above kLowCodes | column (below 2^26).
constexpr unsigned kHiBit = 1u << 26, kIdMask = kHiBit - 1u;
constexpr unsigned kLowCodes = 62;
// words of a row's low planes: four planes of every group, then the other two
__host__ __device__ __forceinline__ int low_stride(int pg) { return (6 * pg + 3) & ~3; }

struct Warp {
  uint64_t *gbuf;     // [32 rows][cap] candidate keys of this warp's rows
  int *cnt;           // smem [32]
  uint64_t *thr;      // smem [32]
  uint32_t *mxc;      // smem [32]
  int cap, K;
};

// Compact every row of the warp whose buffer holds more than `limit` keys.
__device__ __forceinline__ void compact_full_rows(Warp &w, int limit) {
  const int lane = threadIdx.x & 31;
  unsigned full = __ballot_sync(FULL, w.cnt[lane] > limit);
  while (full) {
    const int r = __ffs(full) - 1;
    full &= full - 1;
    const uint64_t P = select_topk<false>(w.gbuf + (size_t)r * w.cap, w.cnt[r], w.K);
    if (lane == 0) { w.cnt[r] = w.K; w.thr[r] = P; }
    __syncwarp();
  }
}

// Register-match counts of up to 32 queued survivors, the warp working on one
// survivor at a time: row codes from shared memory (sA, [32][mpad]) and column
// codes as coalesced 16-byte loads, four survivors in flight.  Lane p ends
// with survivor p's count and admits it.
__device__ __forceinline__ void count_batch_coop(const GraphArgs &g, Warp &w, const int *q, int nq,
                                                 const unsigned char *sA) {
  const int lane = threadIdx.x & 31;
  const int m16 = g.mpad >> 4;
  uint32_t mine = 0;
  for (int p = 0; p < nq; p += 4) {
    const uint4 *ra[4], *cb[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const unsigned e = (unsigned)q[p + u < nq ? p + u : p];
      ra[u] = (const uint4 *)(sA + (size_t)(e >> 27) * g.mpad);
      cb[u] = (const uint4 *)(g.codesB + (int64_t)(e & 0x07FFFFFFu) * g.mpad);
    }
    uint32_t acc[4] = {0u, 0u, 0u, 0u};         // 128 x matches
    for (int t = lane; t < m16; t += 32) {
      uint4 b[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) b[u] = __ldg(cb[u] + t);
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[u] = eq16(lds128(ra[u] + t), b[u], acc[u]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t c = __reduce_add_sync(FULL, acc[u]) >> 7;
      if (lane == p + u) mine = c;
    }
  }
  // Row maxima and admission.  The row state is this warp's own, so lanes of
  // the same row combine in registers and one of them writes: no shared-memory
  // atomics, which serialise when survivors share a row.
  const unsigned act = __ballot_sync(FULL, lane < nq);
  if (lane < nq) {
    const unsigned e = (unsigned)q[lane];
    const int r = (int)(e >> 27);
    const int64_t j = e & 0x07FFFFFFu;
    const unsigned grp = __match_any_sync(act, r);
    const uint32_t mx = __reduce_max_sync(grp, mine);
    const uint64_t key = ((uint64_t)__ldg(g.sv_bits + mine) << 32) | (uint64_t)(~(uint32_t)j);
    const bool adm = key > w.thr[r];
    const unsigned ag = grp & __ballot_sync(act, adm);
    const int base = w.cnt[r];
    if (adm) w.gbuf[(size_t)r * w.cap + base + __popc(ag & ((1u << lane) - 1u))] = key;
    __syncwarp(act);
    if (lane == __ffs(grp) - 1) {
      if (mx > w.mxc[r]) w.mxc[r] = mx;
      w.cnt[r] = base + __popc(ag);
    }
  }
  __syncwarp();
  compact_full_rows(w, w.cap - 32);
}

// Up to 32 survivors (i = row0 + r, j) with their match counts (lane p:
// survivor p's count `mine`): each raises both rows' maxima (row i through the
// warp's own state, row j by an atomic) and, when its similarity passes the
// admission floor, is appended once to the pair list with both rows' counts
// raised.  grow0: the assembly's first row in the row space of the pair list;
// rc: the block's own rows' counts in shared memory (null: straight to o.rowcnt).
__device__ __forceinline__ void admit_sym(const GraphArgs &g, const SymOut &o, uint32_t *mxc,
                                          int64_t row0, int64_t grow0, const unsigned *q, int nq,
                                          uint32_t mine, unsigned id_mask, int *rc) {
  const int lane = threadIdx.x & 31;
  bool adm = false;
  int r = 0;
  uint32_t j = 0, svb = 0;
  if (lane < nq) {
    const unsigned e = q[lane];
    r = (int)(e >> 27);
    j = e & id_mask;
    // shared-memory atomics: they serialise only the survivors of one row
    // (grouping the lanes by row runs one step per row of the batch)
    atomicMax(mxc + r, mine);
    if (mine) atomicMax(g.maxcnt_cand + j, mine);
    if (o.defer) {
      svb = mine;                        // converted once the similarity table exists
      adm = mine > 0;
    } else {
      svb = __ldg(g.sv_bits + mine);
      adm = svb > (uint32_t)(g.key_floor >> 32);
    }
  }
  const unsigned am = __ballot_sync(FULL, adm);
  if (am) {
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(o.npairs, (unsigned long long)__popc(am));
    base = __shfl_sync(FULL, base, 0);
    if (adm) {
      const unsigned long long pos = base + (unsigned)__popc(am & ((1u << lane) - 1u));
      if (pos < o.cap) {
        const uint32_t gi = (uint32_t)(grow0 + row0 + r), gj = (uint32_t)(grow0 + j);
        o.pairs[pos] = make_uint4(gi, gj, svb, (uint32_t)grow0);
        if (rc) atomicAdd(rc + r, 1);
        else atomicAdd(o.rowcnt + gi, 1);
        atomicAdd(o.rowcnt + gj, 1);
      }
    }
  }
  __syncwarp();
}

// Symmetric form of count_batch_coop: the same counts, then admit_sym.
__device__ __forceinline__ void count_batch_sym(const GraphArgs &g, const SymOut &o, uint32_t *mxc,
                                                int64_t row0, int64_t grow0, const int *q, int nq,
                                                const unsigned char *sA) {
  constexpr int NF = 4;                            // survivors' column codes in flight
  const int lane = threadIdx.x & 31;
  const int m16 = g.mpad >> 4;
  uint32_t mine = 0;
  for (int p = 0; p < nq; p += NF) {
    const uint4 *ra[NF], *cb[NF];
#pragma unroll
    for (int u = 0; u < NF; ++u) {
      const unsigned e = (unsigned)q[p + u < nq ? p + u : p];
      ra[u] = (const uint4 *)(sA + (size_t)(e >> 27) * g.mpad);
      cb[u] = (const uint4 *)(g.codesB + (int64_t)(e & 0x07FFFFFFu) * g.mpad);
    }
    uint32_t acc[NF];
#pragma unroll
    for (int u = 0; u < NF; ++u) acc[u] = 0u;
    for (int t = lane; t < m16; t += 32) {
      uint4 b[NF];
#pragma unroll
      for (int u = 0; u < NF; ++u) b[u] = __ldg(cb[u] + t);
#pragma unroll
      for (int u = 0; u < NF; ++u) acc[u] = eq16(lds128(ra[u] + t), b[u], acc[u]);
    }
#pragma unroll
    for (int u = 0; u < NF; ++u) {
      const uint32_t c = __reduce_add_sync(FULL, acc[u]) >> 7;
      if (lane == p + u) mine = c;
    }
  }
  admit_sym(g, o, mxc, row0, grow0, (const unsigned *)q, nq, mine, 0x07FFFFFFu, nullptr);
}

// The same counts on bit planes (launch_code_planes).  A group of 32 registers
// is six words, word p holding bit p of the registers' low codes (the codes up
// to 62, which name the winners of all but a few registers in a million; a register with
// another code or none matches nothing here): the registers that differ are the
// OR over the planes of the two sides' XORs, six three-input logic operations
// and one population count for 32 registers, where bytes take five operations
// for every 4 codes.  A pair whose rows both hold codes above 62 (kHiBit of its
// entry) is counted on the eight planes of the whole codes instead.  LP lanes
// take one survivor (a group each; LP < 32 only when the row's groups fit and a
// count fits LP bits), 32 / LP survivors a step, four steps' column planes in
// flight.  sP: the block's low row planes.
template <int LP>
__device__ __forceinline__ void count_batch_planes(const GraphArgs &g, const SymOut &o,
                                                   uint32_t *mxc, int *rc, int64_t row0,
                                                   const unsigned *q, int nq,
                                                   const uint32_t *sP) {
  constexpr int PER = 32 / LP, U = 4;
  const int lane = threadIdx.x & 31, sub = lane & (LP - 1), which = lane / LP;
  const int pg = g.pg, ls = low_stride(pg);
  uint32_t mine = 0;
  for (int p = 0; p < nq; p += PER * U) {
    unsigned e[U];
    uint32_t cnt[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      e[u] = q[min(p + u * PER + which, nq - 1)];
      cnt[u] = 0;
    }
    for (int t = sub; t < pg; t += LP) {           // one round when LP >= pg
      uint4 b[U];
      uint2 b4[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t *c = g.lowB + (int64_t)(e[u] & kIdMask) * ls;
        b[u] = __ldg(reinterpret_cast<const uint4 *>(c) + t);
        b4[u] = __ldg(reinterpret_cast<const uint2 *>(c + 4 * pg) + t);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t *r = sP + (e[u] >> 27) * ls;
        const uint4 a = lds128(reinterpret_cast<const uint4 *>(r) + t);
        uint32_t d = a.x ^ b[u].x;
        d |= a.y ^ b[u].y;
        d |= a.z ^ b[u].z;
        d |= a.w ^ b[u].w;
        const uint2 a4 = reinterpret_cast<const uint2 *>(r + 4 * pg)[t];
        d |= a4.x ^ b4[u].x;
        d |= a4.y ^ b4[u].y;
        cnt[u] += __popc(~d);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (__any_sync(FULL, e[u] & kHiBit)) {
        if (e[u] & kHiBit) {
          const int64_t i = row0 + (e[u] >> 27), j = e[u] & kIdMask;
          uint32_t c = 0;
          for (int t = sub; t < pg; t += LP) {
            const uint4 *x = reinterpret_cast<const uint4 *>(g.planesA) + i * (2 * pg) + t;
            const uint4 *y = reinterpret_cast<const uint4 *>(g.planesB) + j * (2 * pg) + t;
            const uint4 x0 = __ldg(x), x1 = __ldg(x + pg), y0 = __ldg(y), y1 = __ldg(y + pg);
            c += __popc(~((x0.x ^ y0.x) | (x0.y ^ y0.y) | (x0.z ^ y0.z) | (x0.w ^ y0.w) |
                          (x1.x ^ y1.x) | (x1.y ^ y1.y) | (x1.z ^ y1.z) | (x1.w ^ y1.w)));
          }
          cnt[u] = c;
        }
        __syncwarp();
      }
      // the PER survivors' sums side by side in one word, LP bits each
      const uint32_t c = __reduce_add_sync(FULL, cnt[u] << ((LP & 31) * which));
      const unsigned rel = (unsigned)(lane - (p + u * PER));
      if (rel < (unsigned)PER)
        mine = LP == 32 ? c : (c >> ((LP & 31) * rel)) & ((1u << (LP & 31)) - 1u);
    }
  }
  admit_sym(g, o, mxc, row0, o.row_base, q, nq, mine, kIdMask, rc);
}


// Dense regime: one work item = 32 rows (row block bx) x the column slices
// kWarps*by .. kWarps*by+3, one warp per slice.
__device__ __forceinline__ void dense_item(const GraphArgs &g, uint64_t *gbuf, int32_t *gcnt,
                                           int cap, int P, int64_t bx, int by,
                                           unsigned char *smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t n = g.n;
  const int64_t rhi = g.row_hi < 0 ? n : g.row_hi;
  const int64_t row0 = g.row_lo + bx * 32;
  const int64_t row = row0 + lane;
  const bool vrow = row < rhi;
  const int mw = g.mpad >> 2;
  const int mwq = ((mw + 27) & ~31) + 4;           // = 4 mod 32 words: conflict-free LDS.128
  const int slice = by * kWarps + warp;              // column slice of this warp
  const int64_t jb = n * slice / P, je = n * (slice + 1) / P;

  // shared: per-warp state, then the 32 row-code rows of the block
  unsigned char *ws = smem + (size_t)warp * 1024;
  uint64_t *thr = (uint64_t *)ws;                  // [32]
  int *cnt = (int *)(thr + 32);                    // [32]
  uint32_t *mxc = (uint32_t *)(cnt + 32);          // [32]
  uint32_t *sA = (uint32_t *)(smem + (size_t)kWarps * 1024);   // [32][mwq]

  thr[lane] = g.key_floor;
  cnt[lane] = 0;
  mxc[lane] = 0;
  const size_t bufrow = ((size_t)bx * P + slice) * 32;  // first buffer row of the warp
  Warp w{gbuf + bufrow * cap, cnt, thr, mxc, cap, g.K};
  const uint8_t nz_row = vrow ? g.anynz[row] : 0;
  unsigned n_pref = 0, n_cmp = 0;
  uint32_t mx_a = 0, mx_c = 0;

  for (int i = threadIdx.x; i < 32 * (mw >> 2); i += blockDim.x) {
    const int r = i / (mw >> 2), t = i - r * (mw >> 2);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (row0 + r < n) v = __ldg((const uint4 *)(g.codesA + (row0 + r) * g.mpad) + t);
    *(uint4 *)(sA + r * mwq + 4 * t) = v;
  }
  __syncthreads();
  const uint32_t *ra = sA + lane * mwq;
  const int m4 = mw >> 2;
  // per-warp ring: 2 stages x 4 columns of B codes
  uint4 *ring = (uint4 *)(smem + (size_t)kWarps * 1024 + 32 * (size_t)mwq * 4) +
                (size_t)warp * 2 * 4 * m4;
  auto stage_cols = [&](int st, int64_t j0) {
    uint4 *dst = ring + (size_t)st * 4 * m4;
    for (int i = lane; i < 4 * m4; i += 32) {
      const int u = i / m4, t = i - u * m4;
      const int64_t j = j0 + u < je ? j0 + u : j0;
      cp16(dst + i, (const uint4 *)(g.codesB + j * g.mpad) + t);
    }
    cp_commit();
  };
  if (jb < je) stage_cols(0, jb);
  int st = 0;
  for (int64_t j0 = jb; j0 < je; j0 += 4, st ^= 1) {
    if (j0 + 4 < je) stage_cols(st ^ 1, j0 + 4); else cp_commit();
    cp_wait1();
    __syncwarp();
    const uint4 *c0 = ring + (size_t)st * 4 * m4;
    const uint4 *c1 = c0 + m4, *c2 = c1 + m4, *c3 = c2 + m4;
    uint32_t a0 = 0, a1 = 0, a2 = 0, a3 = 0;      // 128 x matches
#pragma unroll 2
    for (int t = 0; t < m4; ++t) {
      const uint4 a = lds128(ra + 4 * t);
      a0 = eq16(a, lds128(c0 + t), a0);
      a1 = eq16(a, lds128(c1 + t), a1);
      a2 = eq16(a, lds128(c2 + t), a2);
      a3 = eq16(a, lds128(c3 + t), a3);
    }
    const uint32_t cntq[4] = {a0 >> 7, a1 >> 7, a2 >> 7, a3 >> 7};
    __syncwarp();
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int64_t j = j0 + t;
      const bool other = vrow && j < je && j != row;
      const bool cand = other && (nz_row | __ldg(g.anynz + (j < je ? j : jb)));
      const uint32_t c = cntq[t];
      if (other && c > mx_a) mx_a = c;
      if (cand && c > mx_c) mx_c = c;
      n_cmp += other;
      if (cand) {
        const uint64_t key = ((uint64_t)__ldg(g.sv_bits + c) << 32) | (uint64_t)(~(uint32_t)j);
        if (key > thr[lane]) w.gbuf[(size_t)lane * cap + cnt[lane]++] = key;
      }
    }
    __syncwarp();
    compact_full_rows(w, cap - 4);
  }
  if (g.stats) {
    const unsigned a = __reduce_add_sync(FULL, n_pref), b = __reduce_add_sync(FULL, n_cmp);
    if (lane == 0) {
      if (a) atomicAdd(g.stats, (unsigned long long)a);
      if (b) atomicAdd(g.stats + 1, (unsigned long long)b);
    }
  }
  __syncwarp();
  // this slice's K best of each row stay in the buffer for the merge
  compact_full_rows(w, g.K);
  gcnt[bufrow + lane] = cnt[lane];
  if (vrow) {
    if (mx_c) atomicMax(g.maxcnt_cand + row, mx_c);
    if (mx_a) atomicMax(g.maxcnt_all + row, mx_a);
  }
}

template <int SMAX>
__global__ void __launch_bounds__(kWarps * 32)
k_allpairs(GraphArgs g, uint64_t *gbuf, int32_t *gcnt, int cap, int P) {
  extern __shared__ __align__(16) unsigned char smem[];
  dense_item(g, gbuf, gcnt, cap, P, blockIdx.x, blockIdx.y, smem);
}

// ── sparse regime on the tensor cores ──────────────────────────────────────
// The abundance prune is a threshold on U·Uᵀ.  A warp multiplies its 32 rows
// (FP16 copies of the unit rank rows, A fragments kept in registers) with
// 8-column tiles of its column slice (FP16, staged in shared memory, B
// fragments by ldmatrix) using mma.sync m16n8k16 with FP32 accumulation.  For
// unit rows, |c16 - c_ref| <= 2^-10·Σ|a_k b_k| + 2^-24·(|a|_1+|b|_1) + K·2^-22
// + |c_ref - a·b| < 1.1e-3 (FP16 rounding of both inputs, accumulation,
// the reference's own FP32 error), so every pair with c16 < eps - kTcDelta is
// pruned exactly as the reference prunes it.  The rest are checked one per
// lane: FP32 chain with its own band, then the AVX-512 order inside the band.
constexpr float kTcDelta = 2.5e-3f;
constexpr int kTCT = 16;          // columns per staged tile
// check-queue ring entries per warp: at least 31 left over + 256 new ones
// (32 rows x 8 columns) of one step; not a power of two, indexed modulo
constexpr int kCQ = 320;
constexpr int kTcWs = 768;        // per-warp workspace: thresholds, counts, maxima, survivors
constexpr int kScWs = 512;        // the same in k_sym_check: maxima, counts, survivors

__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void *p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}
__device__ __forceinline__ void ldsm_x2(uint32_t &r0, uint32_t &r1, const void *p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n"
               : "=r"(r0), "=r"(r1)
               : "r"(a));
}

// Exact prune decision of one candidate (row r of the block, column j) per
// lane: the FP32 chain, the AVX-512 order inside its band.
template <int SMAX>
__device__ __forceinline__ bool prune_pass(const GraphArgs &g, int r, int64_t j, float lo,
                                           float hi, const float *sU, int SuP) {
  const int Su = g.Su;
  const float4 *ua = (const float4 *)(sU + r * SuP);
  const float4 *ub = (const float4 *)(g.unit + j * Su);
  float ur[SMAX];
  float c1 = 0.f;
#pragma unroll
  for (int t4 = 0; t4 < SMAX; t4 += 4) {
    if (t4 < Su) {
      const float4 x = ua[t4 >> 2], y = __ldg(ub + (t4 >> 2));
      ur[t4] = x.x; ur[t4 + 1] = x.y; ur[t4 + 2] = x.z; ur[t4 + 3] = x.w;
      c1 = __fmaf_rn(x.x, y.x, c1);
      c1 = __fmaf_rn(x.y, y.y, c1);
      c1 = __fmaf_rn(x.z, y.z, c1);
      c1 = __fmaf_rn(x.w, y.w, c1);
    } else {
      ur[t4] = ur[t4 + 1] = ur[t4 + 2] = ur[t4 + 3] = 0.f;
    }
  }
  if (c1 >= hi) return true;
  return c1 >= lo && !(dot_avx512<SMAX>(ur, g.unit + j * Su, g.S) < g.prefilter_eps);
}

// prune_pass of up to 32 candidates of the check ring (at head, modulo kCQ),
// survivors appended to the counting queue.
template <int SMAX, bool SYM>
__device__ __forceinline__ void check_batch(const GraphArgs &g, Warp &w, const SymOut &o,
                                            int64_t grow0, const int *cq, unsigned head, int nq,
                                            int64_t row0, int *q, int &qn, float lo, float hi,
                                            unsigned long long &n_cmp, const float *sU,
                                            int SuP, const unsigned char *sA) {
  const int lane = threadIdx.x & 31;
  const bool act = lane < nq;
  const unsigned e = act ? (unsigned)cq[(head + lane) % kCQ] : 0u;
  const int r = (int)(e >> 27);
  const int64_t j = e & 0x07FFFFFFu, row = row0 + r;
  const bool pass = act && j != row && (__ldg(g.anynz + row) | __ldg(g.anynz + j)) &&
                    prune_pass<SMAX>(g, r, j, lo, hi, sU, SuP);
  const unsigned m = __ballot_sync(FULL, pass);
  if (pass) q[qn + __popc(m & ((1u << lane) - 1u))] = (int)e;
  qn += __popc(m);
  __syncwarp();
  if (qn >= 32) {
    if constexpr (SYM) count_batch_sym(g, o, w.mxc, row0, grow0, q, 32, sA);
    else count_batch_coop(g, w, q, 32, sA);
    n_cmp += 1;
    if (lane + 32 < qn) q[lane] = q[lane + 32];
    __syncwarp();
    qn -= 32;
  }
}

// SYM: the warp's slice is a slice of columns [row0, n) instead of [0, n), the
// block's own rows only pair with later rows (j > i), and survivors go to the
// pair list (count_batch_sym) instead of the rows' candidate buffers.
template <int KS, int SMAX, bool SYM>
__device__ __forceinline__ void tc_item(const GraphArgs &g, uint64_t *gbuf, int32_t *gcnt,
                                        int cap, int P, float lo, float hi, float lo16,
                                        int64_t bx, int by, unsigned char *smem,
                                        const SymOut &o, int64_t grow0, int64_t cb = 0,
                                        int64_t ce = -1) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  const int64_t n = g.n;
  const int64_t row0 = (SYM ? 0 : g.row_lo) + bx * 32;
  const int slice = by * kWarps + warp;
  // columns [c_lo, c_hi); rows at or past row_end are never candidates
  const int64_t c_hi = (SYM && ce >= 0) ? ce : n;
  const int64_t row_end = SYM ? c_hi : (g.row_hi < 0 ? n : g.row_hi);
  const int64_t c_lo = SYM ? (row0 > cb ? row0 : cb) : 0;
  const int64_t span = c_hi > c_lo ? c_hi - c_lo : 0;
  const int64_t jb = c_lo + span * slice / P, je = c_lo + span * (slice + 1) / P;
  const int Kp = KS * 16;
  const int cstride = Kp * 2 + 16;                 // bytes per staged column (conflict-free ldmatrix)

  unsigned char *ws = smem + (size_t)warp * kTcWs;
  uint64_t *thr = (uint64_t *)ws;
  int *cnt = (int *)(thr + 32);
  uint32_t *mxc = (uint32_t *)(cnt + 32);
  int *q = (int *)(mxc + 32);                      // [64] survivors to count
  int *cq = (int *)(smem + (size_t)kWarps * kTcWs) + (size_t)warp * kCQ;     // check ring
  unsigned char *rings = smem + (size_t)kWarps * kTcWs + (size_t)kWarps * kCQ * 4;
  unsigned char *ring = rings + (size_t)warp * 2 * kTCT * cstride;
  // the block's 32 rows: register codes [32][mpad] and unit rows [32][Su]
  unsigned char *sA = rings + (size_t)kWarps * 2 * kTCT * cstride;
  float *sU = (float *)(sA + (size_t)32 * g.mpad);
  const int SuP = su_stride(g.Su);
  {
    const int m16 = g.mpad >> 4, s4 = g.Su >> 2;
    for (int i = threadIdx.x; i < 32 * m16; i += blockDim.x) {
      const int r = i / m16, t = i - r * m16;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (row0 + r < n) v = __ldg((const uint4 *)(g.codesA + (row0 + r) * g.mpad) + t);
      *((uint4 *)(sA + (size_t)r * g.mpad) + t) = v;
    }
    for (int i = threadIdx.x; i < 32 * s4; i += blockDim.x) {
      const int r = i / s4, t = i - r * s4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row0 + r < n) v = __ldg((const float4 *)(g.unit + (row0 + r) * g.Su) + t);
      *((float4 *)(sU + (size_t)r * SuP) + t) = v;
    }
    __syncthreads();
  }
  thr[lane] = g.key_floor;
  cnt[lane] = 0;
  mxc[lane] = 0;
  const size_t bufrow = ((size_t)bx * P + slice) * 32;
  Warp w{SYM ? gbuf : gbuf + bufrow * cap, cnt, thr, mxc, cap, g.K};
  unsigned long long n_pref = 0, n_cmp = 0;

  // A fragments: rows mt*16 + gq (+8), k = ks*16 + 2*tq (+8)
  uint32_t af[2][KS][4];
#pragma unroll
  for (int mt = 0; mt < 2; ++mt) {
    const int64_t ra = row0 + mt * 16 + gq, rb = ra + 8;
    const uint32_t *pa = (const uint32_t *)(g.unit16 + (ra < n ? ra : 0) * Kp);
    const uint32_t *pb = (const uint32_t *)(g.unit16 + (rb < n ? rb : 0) * Kp);
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      af[mt][ks][0] = ra < n ? __ldg(pa + ks * 8 + tq) : 0u;
      af[mt][ks][1] = rb < n ? __ldg(pb + ks * 8 + tq) : 0u;
      af[mt][ks][2] = ra < n ? __ldg(pa + ks * 8 + 4 + tq) : 0u;
      af[mt][ks][3] = rb < n ? __ldg(pb + ks * 8 + 4 + tq) : 0u;
    }
  }
  auto stage_cols = [&](int st, int64_t jt) {
    const int nc = (int)(je - jt < kTCT ? je - jt : kTCT);
    unsigned char *dst = ring + (size_t)st * kTCT * cstride;
    const int per = Kp / 8;                        // 16-byte chunks per column
    for (int i = lane; i < nc * per; i += 32) {
      const int c = i / per, t = i - c * per;
      cp16(dst + c * cstride + 16 * t, g.unit16 + (jt + c) * Kp + 8 * t);
    }
    cp_commit();
  };
  unsigned head = 0, tail = 0;                     // check ring
  int qn = 0;
  if (jb < je) stage_cols(0, jb);
  int st = 0;
  for (int64_t jt = jb; jt < je; jt += kTCT, st ^= 1) {
    if (jt + kTCT < je) stage_cols(st ^ 1, jt + kTCT); else cp_commit();
    const int nc = (int)(je - jt < kTCT ? je - jt : kTCT);
    cp_wait1();
    __syncwarp();
    const unsigned char *tile = ring + (size_t)st * kTCT * cstride;
    const bool interior = nc == kTCT && row0 + 32 <= row_end && (!SYM || jt >= row0 + 32);
    for (int c0 = 0; c0 < nc; c0 += 8) {
      float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      // B fragments: ldmatrix rows = columns c0 + (lane & 7), k block by lane >> 3
      const unsigned char *bp = tile + (c0 + (lane & 7)) * cstride;
      if (KS == 1) {
        uint32_t b0, b1;
        ldsm_x2(b0, b1, bp + 16 * ((lane >> 3) & 1));
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) mma16816(acc[mt], af[mt][0], b0, b1);
      } else {
#pragma unroll
        for (int kp = 0; kp < KS; kp += 2) {
          uint32_t b[4];
          ldsm_x4(b, bp + 16 * (2 * kp + (lane >> 3)));
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            mma16816(acc[mt], af[mt][kp], b[0], b[1]);
            mma16816(acc[mt], af[mt][kp + 1], b[2], b[3]);
          }
        }
      }
      // candidates: value i of m-tile mt -> row mt*16 + gq + 8*(i>>1), column c0 + 2*tq + (i&1).
      // Away from the staged tile's end, the valid rows' end and the diagonal
      // (a warp-uniform test), the threshold alone decides.
      unsigned mk = 0;
      if (interior) {
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int i = 0; i < 4; ++i) mk |= (acc[mt][i] >= lo16 ? 1u : 0u) << (mt * 4 + i);
      } else {
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int rr = mt * 16 + gq + 8 * (i >> 1);
            const int cc = c0 + 2 * tq + (i & 1);
            if (acc[mt][i] >= lo16 && cc < nc && row0 + rr < row_end && (!SYM || jt + cc > row0 + rr))
              mk |= 1u << (mt * 4 + i);
          }
      }
      n_pref += 8;
      if (__any_sync(FULL, mk != 0)) {
        // each lane's slot: the candidates of the lanes below it, summed from
        // the bit planes of the per-lane counts (0..8: four votes) rather than
        // by a chain of dependent shuffles
        const unsigned cntl = (unsigned)__popc(mk), below = (1u << lane) - 1u;
        const unsigned v0 = __ballot_sync(FULL, cntl & 1u), v1 = __ballot_sync(FULL, cntl & 2u);
        const unsigned v2 = __ballot_sync(FULL, cntl & 4u), v3 = __ballot_sync(FULL, cntl & 8u);
        const int excl = __popc(v0 & below) + 2 * __popc(v1 & below) + 4 * __popc(v2 & below) +
                         8 * __popc(v3 & below);
        const int total = __popc(v0) + 2 * __popc(v1) + 4 * __popc(v2) + 8 * __popc(v3);
        unsigned pos = tail + (unsigned)excl;
        while (mk) {
          const int b = __ffs(mk) - 1;
          mk &= mk - 1;
          const int mt = b >> 2, i = b & 3;
          const int rr = mt * 16 + gq + 8 * (i >> 1);
          const int64_t jj = jt + c0 + 2 * tq + (i & 1);
          cq[pos % kCQ] = (int)(((unsigned)rr << 27) | (unsigned)jj);
          ++pos;
        }
        tail += (unsigned)total;
        __syncwarp();
        while (tail - head >= 32) {
          check_batch<SMAX, SYM>(g, w, o, grow0, cq, head, 32, row0, q, qn, lo, hi, n_cmp, sU, SuP, sA);
          head += 32;
        }
      }
    }
    __syncwarp();
  }
  while (tail != head) {
    const int nq = (int)(tail - head < 32 ? tail - head : 32);
    check_batch<SMAX, SYM>(g, w, o, grow0, cq, head, nq, row0, q, qn, lo, hi, n_cmp, sU, SuP, sA);
    head += (unsigned)nq;
  }
  if (qn > 0) {
    n_cmp += lane < qn;
    if constexpr (SYM) count_batch_sym(g, o, mxc, row0, grow0, q, qn, sA);
    else count_batch_coop(g, w, q, qn, sA);
  }
  if (g.stats) {
    // pairs evaluated: ordered pairs, or unordered ones in the symmetric pass
    const unsigned a = __reduce_add_sync(FULL, (unsigned)n_pref),
                   b = __reduce_add_sync(FULL, (unsigned)n_cmp);
    if (lane == 0) {
      if (a) atomicAdd(g.stats, (unsigned long long)a);
      if (b) atomicAdd(g.stats + 1, (unsigned long long)b);
    }
  }
  __syncwarp();
  if constexpr (!SYM) {
    compact_full_rows(w, g.K);
    gcnt[bufrow + lane] = cnt[lane];
  }
  const int64_t row = row0 + lane;
  if (row < n && mxc[lane]) atomicMax(g.maxcnt_cand + row, mxc[lane]);
}

template <int KS, int SMAX>
__global__ void __launch_bounds__(kWarps * 32)
k_allpairs_tc(GraphArgs g, uint64_t *gbuf, int32_t *gcnt, int cap, int P, float lo, float hi,
              float lo16) {
  extern __shared__ __align__(16) unsigned char smem[];
  tc_item<KS, SMAX, false>(g, gbuf, gcnt, cap, P, lo, hi, lo16, blockIdx.x, blockIdx.y, smem,
                           SymOut{}, 0);
}

// Symmetric pass: CTA x scores row block x and row block B-1-x (columns from
// the block's first row on), so every CTA's column work is about n + 32.
// With x0, xs: CTA x0 + blockIdx.x * xs of that layout (the share of one rank
// of a sharded assembly).
template <int KS, int SMAX>
__global__ void __launch_bounds__(kWarps * 32, KS == 2 ? 6 : 1)
k_allpairs_tc_sym(GraphArgs g, int P, float lo, float hi, float lo16, SymOut o, int x0, int xs) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int64_t B = (g.n + 31) / 32;
  const int64_t x = x0 + (int64_t)blockIdx.x * xs;
  const int64_t b1 = x, b2 = B - 1 - x;
  tc_item<KS, SMAX, true>(g, nullptr, nullptr, 0, P, lo, hi, lo16, b1, blockIdx.y, smem, o, 0);
  if (b2 > b1) {
    __syncthreads();
    tc_item<KS, SMAX, true>(g, nullptr, nullptr, 0, P, lo, hi, lo16, b2, blockIdx.y, smem, o, 0);
  }
}

// Window of the symmetric pass: CTA x scores row block x against the columns
// [max(cb, its first row), ce).
template <int KS, int SMAX>
__global__ void __launch_bounds__(kWarps * 32)
k_allpairs_tc_win(GraphArgs g, int P, float lo, float hi, float lo16, SymOut o, int64_t cb,
                  int64_t ce) {
  extern __shared__ __align__(16) unsigned char smem[];
  tc_item<KS, SMAX, true>(g, nullptr, nullptr, 0, P, lo, hi, lo16, blockIdx.x, blockIdx.y, smem, o,
                          0, cb, ce);
}

// Work items of k_sym_check: segments of the blocks' candidate lists.  seg[0 ..
// B] = first item of each block, seg[B + 1] = entries of a segment: about six
// items a CTA slot, so that the last ones leave few SMs idle (with a block
// pair's whole lists per CTA, 30% of the kernel's time was its tail).
__global__ void __launch_bounds__(1024) k_check_items(const int64_t *coff, const int32_t *ccnt,
                                                      int64_t B, int64_t n, int slots,
                                                      int32_t *seg, float *need) {
  __shared__ int part[1024];
  __shared__ unsigned long long all;
  const int t = threadIdx.x;
  auto listed = [&](int64_t b) { return (int)min((int64_t)ccnt[b], coff[b + 1] - coff[b]); };
  if (t == 0) all = 0;
  __syncthreads();
  const int64_t per = (B + 1023) / 1024;
  const int64_t lo = min(B, t * per), hi = min(B, lo + per);
  unsigned long long sum = 0;
  float kept = 0.f;                    // a block's pairs: 32 rows against the columns from its first on
  for (int64_t b = lo; b < hi; ++b) {
    sum += (unsigned)listed(b);
    // (past the 256 entries every list has room for)
    if (n - 32 * b > kTc5Tail)
      kept = fmaxf(kept, (float)(ccnt[b] - 256) / (32.f * (float)(n - 32 * b)));
  }
  // non-negative floats order as their bits
  kept = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(kept)));
  if ((t & 31) == 0) atomicMax((int *)need, __float_as_int(kept));
#pragma unroll
  for (int d = 16; d; d >>= 1) sum += __shfl_xor_sync(FULL, sum, d);
  if ((t & 31) == 0) atomicAdd(&all, sum);
  __syncthreads();
  const int len = (int)(min(4096ull, max(256ull, all / (6ull * slots))) + 127) & ~127;
  int s = 0;
  for (int64_t b = lo; b < hi; ++b) s += (listed(b) + len - 1) / len;
  part[t] = s;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    const int add = t >= d ? part[t - d] : 0;
    __syncthreads();
    part[t] += add;
    __syncthreads();
  }
  int run = t ? part[t - 1] : 0;
  for (int64_t b = lo; b < hi; ++b) {
    seg[b] = run;
    run += (listed(b) + len - 1) / len;
  }
  if (t == 1023) {
    seg[B] = part[1023];
    seg[B + 1] = len;
  }
}

// Symmetric pass, part 2 (after k_sym_prefilter, kernels_sym_tc5.cu).  CTAs
// pull segments of the 32-row blocks' candidate lists from a counter; with the
// block's low register planes and unit rows in shared memory, the warps work
// through the segment 32 entries at a time: the exact prune decision
// (prune_pass), then the survivors' register compares (count_batch_planes) and
// pair records (admit_sym).  Bound by the L1 data path: per survivor its column
// planes (24 bytes a group of 32 registers), the candidate's unit row, and the
// atomics of the later row's maximum and count (70% of its wavefronts; issue
// 52%).  m = 500: 30,000 contigs 722 us on bytes -> 515 us (S = 20, 7.0 M
// survivors), 4.25 -> 3.04 ms (S = 5, 51 M).
template <int SMAX, int LP>
__global__ void __launch_bounds__(kWarps * 32, SMAX <= 32 ? 6 : 1)
k_sym_check(GraphArgs g, float lo, float hi, SymOut o, const uint32_t *cand,
            const int64_t *coff, const int32_t *ccnt, int B, const int32_t *seg, unsigned *next) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_block, s_first;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t n = g.n;
  unsigned char *ws = smem + (size_t)warp * kScWs;
  uint32_t *mxc = (uint32_t *)ws;
  int *rc = (int *)(mxc + 32);                     // pairs listed of the block's rows
  unsigned *q = (unsigned *)(rc + 32);             // [64] survivors to count
  const int ls = low_stride(g.pg);
  uint32_t *sP = (uint32_t *)(smem + (size_t)kWarps * kScWs);
  float *sU = (float *)(sP + (size_t)32 * ls);
  const int SuP = su_stride(g.Su);
  const int len = seg[B + 1], items = seg[B];
  unsigned long long n_cmp = 0;
  for (;;) {
    if (warp == 0) {
      // the next item and its block: the last b with seg[b] <= item, by 32-ary search
      unsigned it = 0;
      if (lane == 0) it = atomicAdd(next, 1u);
      it = __shfl_sync(FULL, it, 0);
      int b0 = 0, span = B;                        // the block is in [b0, b0 + span)
      if (it < (unsigned)items) {
        while (span > 1) {
          const int step = (span + 31) / 32;
          const int b = b0 + lane * step;
          const bool le = lane * step < span && __ldg(seg + b) <= (int)it;
          const int k = 31 - __clz((int)__ballot_sync(FULL, le));   // lane 0 always holds
          const int left = span - k * step;
          b0 += k * step;
          span = left < step ? left : step;
        }
      } else {
        b0 = -1;
      }
      if (lane == 0) {
        s_block = b0;
        s_first = b0 < 0 ? 0 : ((int)it - __ldg(seg + b0)) * len;
      }
    }
    __syncthreads();
    const int bx = s_block;
    if (bx < 0) break;
    const int64_t row0 = (int64_t)bx * 32;
    {
      const int p16 = ls >> 2, s4 = g.Su >> 2;
      const uint4 *rows = reinterpret_cast<const uint4 *>(g.lowA) + row0 * p16;
      const int lim = (int)min((int64_t)32, n - row0) * p16;
      for (int i = threadIdx.x; i < 32 * p16; i += blockDim.x)
        ((uint4 *)sP)[i] = i < lim ? __ldg(rows + i) : make_uint4(0u, 0u, 0u, 0u);
      for (int i = threadIdx.x; i < 32 * s4; i += blockDim.x) {
        const int r = i / s4, t = i - r * s4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row0 + r < n) v = __ldg((const float4 *)(g.unit + (row0 + r) * g.Su) + t);
        *((float4 *)(sU + (size_t)r * SuP) + t) = v;
      }
    }
    mxc[lane] = 0;
    rc[lane] = 0;
    const int64_t off = coff[bx];
    const int cnt = min((int)min((int64_t)ccnt[bx], coff[bx + 1] - off), s_first + len);
    const uint32_t *list = cand + off;
    const uint32_t rflag = row0 + lane < n ? __ldg(g.pflag + row0 + lane) : 0u;
    const unsigned rhi = __ballot_sync(FULL, rflag & 1u);   // rows with codes above kLowCodes
    const unsigned rnz = __ballot_sync(FULL, rflag & 2u);   // rows with abundance
    int i0 = s_first + warp * 32;
    __syncthreads();
    int qn = 0;
    unsigned enext = i0 + lane < cnt ? list[i0 + lane] : 0u;
    for (; i0 < cnt; i0 += kWarps * 32) {
      const bool act = i0 + lane < cnt;
      unsigned e = enext;
      const int inext = i0 + kWarps * 32 + lane;     // the next entries load meanwhile
      enext = inext < cnt ? list[inext] : 0u;
      const int r = (int)(e >> 27);
      const int64_t j = e & 0x07FFFFFFu;
      // flag and unit row load together (an idle lane reads column 0)
      const unsigned jf = __ldg(g.pflag + j);
      const bool dot = prune_pass<SMAX>(g, r, j, lo, hi, sU, SuP);
      const bool pass = act && dot && (((rnz >> r) & 1u) | (jf & 2u));
      const unsigned m = __ballot_sync(FULL, pass);
      if (pass) {
        if ((rhi >> r) & jf & 1u) e |= kHiBit;
        q[qn + __popc(m & ((1u << lane) - 1u))] = e;
      }
      qn += __popc(m);
      __syncwarp();
      if (qn >= 32) {
        count_batch_planes<LP>(g, o, mxc, rc, row0, q, 32, sP);
        n_cmp += 1;
        if (lane + 32 < qn) q[lane] = q[lane + 32];
        __syncwarp();
        qn -= 32;
      }
    }
    if (qn > 0) {
      n_cmp += lane < qn;
      count_batch_planes<LP>(g, o, mxc, rc, row0, q, qn, sP);
    }
    __syncwarp();
    const int64_t row = row0 + lane;
    if (row < n && mxc[lane]) atomicMax(g.maxcnt_cand + row, mxc[lane]);
    if (rc[lane]) atomicAdd(o.rowcnt + o.row_base + row, rc[lane]);
    __syncthreads();                               // shared rows and the item are done with
  }
  if (g.stats) {
    const unsigned b = __reduce_add_sync(FULL, (unsigned)n_cmp);
    if (lane == 0 && b) atomicAdd(g.stats + 1, (unsigned long long)b);
  }
}

// Bits of 8 codes (bytes of x, then y) as 8 bytes: byte p of (x, y) gets one
// bit of each code, the same bit of every code for one p (an 8 x 8 bit
// transpose by three rounds of block swaps).
__device__ __forceinline__ void transpose8(uint32_t &x, uint32_t &y) {
  uint32_t t = (x ^ (x >> 7)) & 0x00AA00AAu;
  x ^= t ^ (t << 7);
  t = (y ^ (y >> 7)) & 0x00AA00AAu;
  y ^= t ^ (t << 7);
  t = (x ^ (x >> 14)) & 0x0000CCCCu;
  x ^= t ^ (t << 14);
  t = (y ^ (y >> 14)) & 0x0000CCCCu;
  y ^= t ^ (t << 14);
  t = (y & 0x0F0F0F0Fu) << 4 | (x & 0x0F0F0F0Fu);
  y = (x >> 4 & 0x0F0F0F0Fu) | (y & 0xF0F0F0F0u);
  x = t;
}

// Eight plane words of 32 codes (word p: bit p of each).
__device__ __forceinline__ void planes32(const uint4 v0, const uint4 v1, uint32_t (&w)[8]) {
  uint32_t x[4] = {v0.x, v0.z, v1.x, v1.z}, y[4] = {v0.y, v0.w, v1.y, v1.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) transpose8(x[k], y[k]);
  // word p of the group: byte p of the four 8-code transposes
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t(&z)[4] = h ? y : x;
    const uint32_t l01 = __byte_perm(z[0], z[1], 0x5140u), h01 = __byte_perm(z[0], z[1], 0x7362u);
    const uint32_t l23 = __byte_perm(z[2], z[3], 0x5140u), h23 = __byte_perm(z[2], z[3], 0x7362u);
    w[4 * h] = __byte_perm(l01, l23, 0x5410u);
    w[4 * h + 1] = __byte_perm(l01, l23, 0x7632u);
    w[4 * h + 2] = __byte_perm(h01, h23, 0x5410u);
    w[4 * h + 3] = __byte_perm(h01, h23, 0x7632u);
  }
}

// 0xFF in the bytes of x above kLowCodes.
__device__ __forceinline__ uint32_t above_low(uint32_t x) {
  const uint32_t hi = (x & 0x80808080u) |
                      ((x & 0x7F7F7F7Fu) + (0x7Fu - kLowCodes) * 0x01010101u & 0x80808080u);
  return (hi >> 7) * 0xFFu;
}

// Register planes of rows [r_lo, r_hi), both sides (blockIdx.y): thread = (row,
// group of 32 registers), rows_per rows a block.  Registers past mpad count as
// unset (A 0, B 0xFF).  Whole codes: [row][2][pg] of four planes; low codes (see
// count_batch_planes): [row] low_stride words, 0 (A) or 63 (B) where a register
// has no code up to kLowCodes; pflag[row]: bit 0 some code is above it, bit 1 anynz.
__global__ void __launch_bounds__(256) k_code_planes(const uint4 *__restrict__ A,
                                                     const uint4 *__restrict__ B, int64_t r_lo,
                                                     int64_t r_hi, int m16, int pg, int rows_per,
                                                     uint4 *__restrict__ pA, uint4 *__restrict__ pB,
                                                     uint32_t *__restrict__ lA,
                                                     uint32_t *__restrict__ lB,
                                                     const uint8_t *__restrict__ anynz,
                                                     uint8_t *__restrict__ pflag) {
  __shared__ int any[256];
  const int rl = threadIdx.x / pg, t = threadIdx.x - rl * pg;
  const int64_t row = r_lo + (int64_t)blockIdx.x * rows_per + rl;
  const bool side = blockIdx.y != 0;
  if (threadIdx.x < rows_per) any[threadIdx.x] = 0;
  __syncthreads();
  if (rl < rows_per && row < r_hi) {
    const uint4 *src = (side ? B : A) + row * m16;
    const uint32_t fill = side ? 0xFFFFFFFFu : 0u;
    uint4 v0 = __ldg(src + 2 * t);
    uint4 v1 = 2 * t + 1 < m16 ? __ldg(src + 2 * t + 1) : make_uint4(fill, fill, fill, fill);
    uint32_t w[8];
    planes32(v0, v1, w);
    uint4 *dst = (side ? pB : pA) + row * (2 * pg) + t;
    dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
    dst[pg] = make_uint4(w[4], w[5], w[6], w[7]);
    const uint32_t none = side ? 0x3F3F3F3Fu : 0u;
    uint32_t seen = 0;
    auto low = [&](uint32_t x) {
      const uint32_t h = above_low(x);
      seen |= h;
      return (x & ~h) | (h & none);
    };
    v0 = make_uint4(low(v0.x), low(v0.y), low(v0.z), low(v0.w));
    v1 = make_uint4(low(v1.x), low(v1.y), low(v1.z), low(v1.w));
    planes32(v0, v1, w);
    uint32_t *l = (side ? lB : lA) + row * low_stride(pg);
    reinterpret_cast<uint4 *>(l)[t] = make_uint4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<uint2 *>(l + 4 * pg)[t] = make_uint2(w[4], w[5]);
    if (!side && seen) any[rl] = 1;                // A: unset registers are 0
  }
  if (side) return;
  __syncthreads();
  if (rl < rows_per && row < r_hi && t == 0) pflag[row] = (uint8_t)(any[rl] | (anynz[row] ? 2 : 0));
}

// Persistent form over a batch: CTAs pull (assembly, row block, slice group)
// items from a device counter until the variant's items are exhausted.  The
// tensor-core variants run the symmetric pass (a row block's slices cover the
// columns from its first row on; items come in ascending row blocks, so the
// largest first).
template <int KS, int SMAX>
__global__ void __launch_bounds__(kWarps * 32)
k_allpairs_batch(const BatchAsm *B, const int32_t *list, const int64_t *item0s, int nv,
                 int64_t items, unsigned long long *next, SymOut o) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ long long s_item;
  for (;;) {
    __syncthreads();                     // the previous item is done with shared memory
    if (threadIdx.x == 0) s_item = (long long)atomicAdd(next, 1ull);
    __syncthreads();
    const int64_t it = s_item;
    if (it >= items) return;
    int lo = 0, hi = nv - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(item0s + mid) <= it) lo = mid; else hi = mid - 1;
    }
    const BatchAsm &b = B[list[lo]];
    const GraphArgs g = b.g;
    const int G = b.P / kWarps;
    const int64_t local = it - item0s[lo];
    const int64_t bx = local / G;
    const int by = (int)(local - bx * G);
    if constexpr (KS == 0) dense_item(g, b.gbuf, b.gcnt, b.cap, b.P, bx, by, smem);
    else tc_item<KS, SMAX, true>(g, nullptr, nullptr, 0, b.P, b.lo, b.hi, b.lo16, bx, by, smem, o,
                                 b.row0);
  }
}

// Warp per row: the K best keys among the P slices' partial lists.  The lists
// stream through a 512-key shared buffer per warp; whenever it fills, the
// register radix select keeps its K best (K <= 448 leaves room to refill).
constexpr int kMergeWarps = 8;
constexpr int kMergeBuf = 32 * kCapW;       // 512 keys per warp

__device__ __forceinline__ void merge_row(const GraphArgs &g, const uint64_t *gbuf,
                                          const int32_t *gcnt, int cap, int P, int64_t row,
                                          uint64_t *keys) {
  const int lane = threadIdx.x & 31;
  const int K = g.K;
  const int64_t rb = (row - g.row_lo) >> 5, rl = (row - g.row_lo) & 31;
  const size_t br0 = (size_t)rb * P * 32 + rl;          // slice s: br0 + 32 s
  const int cl = lane < P ? gcnt[br0 + (size_t)lane * 32] : 0;   // P <= 32
  int fill = 0;
  for (int s = 0; s < P; ++s) {
    const int c = __shfl_sync(FULL, cl, s);
    const uint64_t *src = gbuf + (br0 + (size_t)s * 32) * cap;
    for (int i0 = 0; i0 < c;) {
      const int take = min(c - i0, kMergeBuf - fill);
      for (int i = lane; i < take; i += 32) keys[fill + i] = src[i0 + i];
      fill += take;
      i0 += take;
      __syncwarp();
      if (fill == kMergeBuf) {
        select_topk(keys, fill, K);
        fill = K;
      }
    }
  }
  if (fill > K) {
    select_topk(keys, fill, K);
    fill = K;
  }
  for (int i = lane; i < fill; i += 32) g.topk[row * K + i] = keys[i];
  if (lane == 0) g.topk_cnt[row] = fill;
}

__global__ void __launch_bounds__(kMergeWarps * 32)
k_merge_topk(GraphArgs g, const uint64_t *gbuf, const int32_t *gcnt, int cap, int P) {
  __shared__ uint64_t mk[kMergeWarps][kMergeBuf];
  const int wib = threadIdx.x >> 5;
  const int64_t row = g.row_lo + (int64_t)blockIdx.x * kMergeWarps + wib;
  if (row < (g.row_hi < 0 ? g.n : g.row_hi)) merge_row(g, gbuf, gcnt, cap, P, row, mk[wib]);
}

__global__ void __launch_bounds__(kMergeWarps * 32)
k_merge_batch(const BatchAsm *B, const int64_t *row0s, int nb, int64_t r_begin, int64_t rows) {
  __shared__ uint64_t mk[kMergeWarps][kMergeBuf];
  const int wib = threadIdx.x >> 5;
  const int64_t r = r_begin + (int64_t)blockIdx.x * kMergeWarps + wib;
  if (r >= rows) return;
  int lo = 0, hi = nb - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(row0s + mid) <= r) lo = mid; else hi = mid - 1;
  }
  const BatchAsm &b = B[lo];
  if (b.variant != 0) return;          // top-K from the symmetric pass's pairs
  merge_row(b.g, b.gbuf, b.gcnt, b.cap, b.P, r - b.row0, mk[wib]);
}

// Admitted keys per row of a pair list gathered from several ranks (both ends).
__global__ void k_pair_rowcounts(const uint4 *__restrict__ pairs, unsigned long long np,
                                 int32_t *__restrict__ rowcnt) {
  for (unsigned long long p = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; p < np;
       p += (unsigned long long)gridDim.x * blockDim.x) {
    const uint4 x = pairs[p];
    atomicAdd(rowcnt + x.x, 1);
    atomicAdd(rowcnt + x.y, 1);
  }
}

// out[i] = the largest of the W ranks' partial maxima (blocks of `stride`).
__global__ void k_max_blocks(const uint32_t *__restrict__ blocks, int W, int64_t stride,
                             int64_t n, uint32_t *__restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t v = 0;
    for (int r = 0; r < W; ++r) v = max(v, blocks[(int64_t)r * stride + i]);
    out[i] = v;
  }
}

// Both keys of every admitted pair into their rows' segments (grid-stride over
// the pairs written).  Positions count down from each row's end, so the row
// counts return to zero.
__global__ void k_scatter_pairs(SymOut o, const int64_t *off, uint64_t *keys,
                                const uint32_t *svtab) {
  const unsigned long long np = *o.npairs < o.cap ? *o.npairs : o.cap;
  for (unsigned long long p = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; p < np;
       p += (unsigned long long)gridDim.x * blockDim.x) {
    const uint4 x = o.pairs[p];                 // ids in keys are the assembly's own
    const uint64_t hi = (uint64_t)(svtab ? __ldg(svtab + x.z) : x.z) << 32;
    const int64_t pi = off[x.x] + atomicSub(o.rowcnt + x.x, 1) - 1;
    keys[pi] = hi | (uint64_t)(~(x.y - x.w));
    const int64_t pj = off[x.y] + atomicSub(o.rowcnt + x.y, 1) - 1;
    keys[pj] = hi | (uint64_t)(~(x.x - x.w));
  }
}

// Keys of a row ranked by a histogram of their similarity (sim_bins.cuh).
constexpr int kSelWords = kBins;                    // 32-bit words of a warp's buffer
static_assert(kMergeBuf * 2 <= kSelWords, "the tie buffer lies over the histogram");

__device__ __forceinline__ int key_bin(uint64_t key) { return sim_bin((uint32_t)(key >> 32)); }

// Keeps the R largest of the cnt unique keys in buf, in place.  Up to 96 keys by
// their ranks (each lane counts the keys above its own), else by select_topk.
__device__ __forceinline__ void keep_largest(uint64_t *buf, int cnt, int R) {
  const int lane = threadIdx.x & 31;
  if (cnt > 96) {
    select_topk(buf, cnt, R);
    return;
  }
  uint64_t v[3];
  int rank[3] = {0, 0, 0};
#pragma unroll
  for (int t = 0; t < 3; ++t) v[t] = t * 32 + lane < cnt ? buf[t * 32 + lane] : 0ull;
  for (int i = 0; i < cnt; ++i) {
    const uint64_t x = buf[i];
#pragma unroll
    for (int t = 0; t < 3; ++t) rank[t] += x > v[t];
  }
  __syncwarp();
#pragma unroll
  for (int t = 0; t < 3; ++t)
    if (t * 32 + lane < cnt && rank[t] < R) buf[rank[t]] = v[t];
  __syncwarp();
}

// Warp per row: the K best keys of the row's segment (row space index gr,
// assembly row `row`).  Two passes over the segment: a histogram gives the bin
// that holds the K-th key; keys above it are kept as they stream by, keys in it
// are gathered (in a 512-key buffer over the histogram, cut when it fills) and
// the largest of them fill up.  A segment read twice against a bit-by-bit search
// over every 512 keys: 50,000 rows (470 keys each) 0.31 -> 0.13 ms, 30,011 rows
// at S = 5 (3,400 keys) 0.72 -> 0.23 ms.
__device__ __forceinline__ void select_row(const GraphArgs &g, int64_t row, int64_t gr,
                                           const int64_t *off, const uint64_t *keys,
                                           uint32_t *words) {
  const int lane = threadIdx.x & 31;
  const int K = g.K;
  const int64_t s0 = off[gr];
  const int64_t c = off[gr + 1] - s0;
  const uint64_t *src = keys + s0;
  uint64_t *top = g.topk + row * K;
  if (c <= K) {
    for (int64_t i = lane; i < c; i += 32) top[i] = src[i];
    if (lane == 0) g.topk_cnt[row] = (int32_t)c;
    return;
  }
  for (int i = lane; i < kBins / 4; i += 32)
    reinterpret_cast<uint4 *>(words)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncwarp();
  for (int64_t i = lane; i < c; i += 32) atomicAdd(words + key_bin(src[i]), 1u);
  __syncwarp();
  // bins from the top: lane l owns the 40 bins below kBins - 40 l
  constexpr int kPer = kBins / 32;
  const uint32_t *mine = words + kBins - kPer * (lane + 1);
  uint32_t sum = 0;
#pragma unroll
  for (int i = 0; i < kPer; i += 4) {
    const uint4 x = *reinterpret_cast<const uint4 *>(mine + i);
    sum += x.x + x.y + x.z + x.w;
  }
  uint32_t incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(FULL, incl, d);
    if (lane >= d) incl += t;
  }
  int bin = 0, above = 0;                            // the K-th key's bin, keys above it
  const unsigned own = __ballot_sync(FULL, incl >= (uint32_t)K);
  const int who = __ffs(own) - 1;                    // c > K: some lane reaches K
  if (lane == who) {
    uint32_t at = incl - sum;
    int i = kPer - 1;
    for (; i > 0 && at + mine[i] < (uint32_t)K; --i) at += mine[i];
    bin = kBins - kPer * (lane + 1) + i;
    above = (int)at;
  }
  bin = __shfl_sync(FULL, bin, who);
  above = __shfl_sync(FULL, above, who);
  __syncwarp();                                      // the histogram is done with
  uint64_t *buf = reinterpret_cast<uint64_t *>(words);
  const int need = K - above;                        // keys taken from the bin
  int out = 0, fill = 0;
  for (int64_t i0 = 0; i0 < c; i0 += 32) {
    const int64_t i = i0 + lane;
    const uint64_t key = i < c ? src[i] : 0ull;
    const int b = i < c ? key_bin(key) : -1;
    const unsigned hi = __ballot_sync(FULL, b > bin), eq = __ballot_sync(FULL, b == bin);
    const unsigned below = (1u << lane) - 1u;
    if (b > bin) top[out + __popc(hi & below)] = key;
    out += __popc(hi);
    if (eq) {
      if (fill + __popc(eq) > kMergeBuf) {
        select_topk(buf, fill, need);
        fill = need;
      }
      if (b == bin) buf[fill + __popc(eq & below)] = key;
      fill += __popc(eq);
      __syncwarp();
    }
  }
  if (fill > need) keep_largest(buf, fill, need);
  for (int i = lane; i < need; i += 32) top[above + i] = buf[i];
  if (lane == 0) g.topk_cnt[row] = K;
}

__global__ void __launch_bounds__(kMergeWarps * 32)
k_select_rows(GraphArgs g, const int64_t *off, const uint64_t *keys) {
  __shared__ __align__(16) uint32_t mk[kMergeWarps][kSelWords];
  const int wib = threadIdx.x >> 5;
  const int64_t row = (int64_t)blockIdx.x * kMergeWarps + wib;
  if (row < g.n) select_row(g, row, row, off, keys, mk[wib]);
}

__global__ void __launch_bounds__(kMergeWarps * 32)
k_select_rows_batch(const BatchAsm *B, const int64_t *row0s, int nb, int64_t rows,
                    const int64_t *off, const uint64_t *keys) {
  __shared__ __align__(16) uint32_t mk[kMergeWarps][kSelWords];
  const int wib = threadIdx.x >> 5;
  const int64_t r = (int64_t)blockIdx.x * kMergeWarps + wib;
  if (r >= rows) return;
  int lo = 0, hi = nb - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(row0s + mid) <= r) lo = mid; else hi = mid - 1;
  }
  const BatchAsm &b = B[lo];
  if (b.variant <= 0) return;          // dense: candidate buffers or the one-hot GEMM
  select_row(b.g, r - b.row0, r, off, keys, mk[wib]);
}

size_t dense_smem(int mpad) {
  const int mw = mpad >> 2;
  const int mwq = ((mw + 27) & ~31) + 4;
  return (size_t)kWarps * 1024 + 32 * (size_t)mwq * 4 + (size_t)kWarps * 2 * 4 * mpad;
}

size_t tc_smem(int KS, int mpad, int Su) {
  return (size_t)kWarps * kTcWs + (size_t)kWarps * kCQ * 4 +
         (size_t)kWarps * 2 * kTCT * (KS * 16 * 2 + 16) + (size_t)32 * mpad +
         (size_t)32 * su_stride(Su) * 4;
}

}  // namespace

int allpairs_cap(int K) { return (K + 64 + 31) & ~31; }

// Column slices per 32-row block: enough warps for several waves of the GPU, a
// multiple of the CTA's warp count.
int allpairs_slices(int64_t n, int K) { return allpairs_slices_rows(n, n, K); }

int allpairs_slices_rows(int64_t rows, int64_t n, int K) {
  const int64_t blocks = (rows + 31) / 32;
  int64_t P = (4 * 148 * 48 + blocks - 1) / std::max<int64_t>(blocks, 1);
  // at least 64 columns a slice (fewer lists to merge); 8 with few contigs, whose row
  // blocks leave most SMs idle
  P = std::min<int64_t>(P, std::max<int64_t>(n / (n <= 512 ? 8 : 64), 1));
  P = std::max<int64_t>(P, 1);
  const int pmax = std::max(kWarps, std::min(32, (6400 / std::max(K, 1)) / kWarps * kWarps));
  P = std::min<int64_t>(P, pmax);
  return (int)(((P + kWarps - 1) / kWarps) * kWarps);
}

int64_t allpairs_items(int64_t n, int P) { return ((n + 31) / 32) * (P / kWarps); }

size_t allpairs_batch_smem(int variant, int mpad, int Su) {
  return variant == 0 ? dense_smem(mpad) : tc_smem(variant, mpad, Su);
}

void prefilter_bands(int S, float eps, float *lo, float *hi, float *lo16) {
  // band of the exact-safe prefilter: |chain - AVX-512 order| < delta
  const double e = (double)eps;
  const double delta = (double)(S + (S + 15) / 16 + 8) * ldexp(1.0, -23);
  float l = (float)(e - delta), h = (float)(e + delta);
  if ((double)l > e - delta) l = nextafterf(l, -INFINITY);
  if ((double)h < e + delta) h = nextafterf(h, INFINITY);
  *lo = l;
  *hi = h;
  *lo16 = (float)(e - (double)kTcDelta);
}

int allpairs_variant(const GraphArgs &g) {
  if (!g.prefilter) return 0;
  return g.Kp == 16 ? 1 : (g.Kp == 32 ? 2 : 4);   // the FP16 rows are KS * 16 halves wide
}

void launch_allpairs(const GraphArgs &g, uint64_t *gbuf, int32_t *gcnt, cudaStream_t s) {
  const int64_t rows = (g.row_hi < 0 ? g.n : g.row_hi) - g.row_lo;
  if (g.n == 0 || rows <= 0) return;
  const int cap = allpairs_cap(g.K);
  const int P = allpairs_slices_rows(rows, g.n, g.K);
  const dim3 grid((unsigned)((rows + 31) / 32), (unsigned)(P / kWarps));
  float lo, hi, lo16;
  prefilter_bands(g.S, g.prefilter_eps, &lo, &hi, &lo16);
  const int v = allpairs_variant(g);
  const size_t smem = allpairs_batch_smem(v, g.mpad, g.Su);
#define RBG_TC(KS, SM)                                                                        \
  do {                                                                                        \
    smem_cap_max((const void *)k_allpairs_tc<KS, SM>);                                        \
    k_allpairs_tc<KS, SM><<<grid, kWarps * 32, smem, s>>>(g, gbuf, gcnt, cap, P, lo, hi, lo16); \
  } while (0)
  if (v == 1) RBG_TC(1, 16);
  else if (v == 2) RBG_TC(2, 32);
  else if (v == 4) RBG_TC(4, 64);
  else {
    smem_cap_max((const void *)k_allpairs<4>);
    k_allpairs<4><<<grid, kWarps * 32, smem, s>>>(g, gbuf, gcnt, cap, P);
  }
#undef RBG_TC
  k_merge_topk<<<(unsigned)((rows + kMergeWarps - 1) / kMergeWarps), kMergeWarps * 32, 0, s>>>(
      g, gbuf, gcnt, cap, P);
}

void launch_pair_rowcounts(const uint4 *pairs, unsigned long long np, int32_t *rowcnt,
                           cudaStream_t s) {
  if (np == 0) return;
  k_pair_rowcounts<<<(unsigned)std::min<unsigned long long>((np + 255) / 256, 148 * 8), 256, 0,
                     s>>>(pairs, np, rowcnt);
}

void launch_max_blocks(const uint32_t *blocks, int W, int64_t stride, int64_t n, uint32_t *out,
                       cudaStream_t s) {
  if (n == 0) return;
  k_max_blocks<<<(unsigned)std::min<int64_t>((n + 255) / 256, 148 * 8), 256, 0, s>>>(
      blocks, W, stride, n, out);
}

void launch_merge_topk(const GraphArgs &g, const uint64_t *gbuf, const int32_t *gcnt, int cap,
                       int P, cudaStream_t s) {
  const int64_t rows = (g.row_hi < 0 ? g.n : g.row_hi) - g.row_lo;
  if (rows <= 0) return;
  k_merge_topk<<<(unsigned)((rows + kMergeWarps - 1) / kMergeWarps), kMergeWarps * 32, 0, s>>>(
      g, gbuf, gcnt, cap, P);
}

size_t low_plane_words(int pg) { return (size_t)low_stride(pg); }

void launch_code_planes(const GraphArgs &g, int64_t r_lo, int64_t r_hi, uint32_t *planesA,
                        uint32_t *planesB, uint32_t *lowA, uint32_t *lowB, uint8_t *pflag,
                        cudaStream_t s) {
  if (r_hi <= r_lo) return;
  const int rows_per = 256 / g.pg;                 // pg <= 128
  const int64_t blocks = (r_hi - r_lo + rows_per - 1) / rows_per;
  k_code_planes<<<dim3((unsigned)blocks, 2), 256, 0, s>>>(
      (const uint4 *)g.codesA, (const uint4 *)g.codesB, r_lo, r_hi, g.mpad / 16, g.pg, rows_per,
      (uint4 *)planesA, (uint4 *)planesB, lowA, lowB, g.anynz, pflag);
}

void launch_sym_check(const GraphArgs &g, const SymOut &o, const uint32_t *cand,
                      const int64_t *coff, const int32_t *ccnt, int64_t B, int32_t *seg,
                      unsigned *next, float *need, int sms, cudaStream_t s) {
  if (g.n == 0 || B <= 0) return;
  float lo, hi, lo16;
  prefilter_bands(g.S, g.prefilter_eps, &lo, &hi, &lo16);
  const int v = allpairs_variant(g);
  const size_t smem = (size_t)kWarps * kScWs + (size_t)32 * low_stride(g.pg) * 4 +
                      (size_t)32 * su_stride(g.Su) * 4;
  // lanes a survivor: its groups, while a count fits as many bits
  const int lp = g.pg <= 8 && g.m <= 255 ? 8 : (g.pg <= 16 ? 16 : 32);
#define RBG_SC(SM, LP)                                                                        \
  do {                                                                                        \
    smem_cap_max((const void *)k_sym_check<SM, LP>);                                          \
    int per_sm = 1;                                                                           \
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sym_check<SM, LP>, kWarps * 32,  \
                                                  smem);                                      \
    const int grid = std::max(per_sm, 1) * sms;                                               \
    k_check_items<<<1, 1024, 0, s>>>(coff, ccnt, B, g.n, grid, seg, need);                    \
    k_sym_check<SM, LP><<<grid, kWarps * 32, smem, s>>>(g, lo, hi, o, cand, coff, ccnt,       \
                                                        (int)B, seg, next);                   \
  } while (0)
#define RBG_SCL(SM)                                                                           \
  do {                                                                                        \
    if (lp == 8) RBG_SC(SM, 8);                                                               \
    else if (lp == 16) RBG_SC(SM, 16);                                                        \
    else RBG_SC(SM, 32);                                                                      \
  } while (0)
  if (v == 1) RBG_SCL(16);
  else if (v == 2) RBG_SCL(32);
  else RBG_SCL(64);
#undef RBG_SCL
#undef RBG_SC
}

float prefilter_lo16(int S, float eps) {
  float lo, hi, lo16;
  prefilter_bands(S, eps, &lo, &hi, &lo16);
  return lo16;
}

void launch_allpairs_sym(const GraphArgs &g, const SymOut &o, cudaStream_t s, int x0, int xs) {
  if (g.n == 0) return;
  const int P = allpairs_slices(g.n, g.K);
  const int64_t B = (g.n + 31) / 32;
  const int64_t nx = (B + 1) / 2;                 // CTAs of the whole pass
  if (x0 >= nx) return;
  const dim3 grid((unsigned)((nx - x0 + xs - 1) / xs), (unsigned)(P / kWarps));
  float lo, hi, lo16;
  prefilter_bands(g.S, g.prefilter_eps, &lo, &hi, &lo16);
  const int v = allpairs_variant(g);
  const size_t smem = tc_smem(v, g.mpad, g.Su);
#define RBG_TS(KS, SM)                                                                        \
  do {                                                                                        \
    smem_cap_max((const void *)k_allpairs_tc_sym<KS, SM>);                                    \
    k_allpairs_tc_sym<KS, SM><<<grid, kWarps * 32, smem, s>>>(g, P, lo, hi, lo16, o, x0, xs); \
  } while (0)
  if (v == 1) RBG_TS(1, 16);
  else if (v == 2) RBG_TS(2, 32);
  else RBG_TS(4, 64);
#undef RBG_TS
}

void launch_allpairs_sym_window(const GraphArgs &g, const SymOut &o, int64_t cb, int64_t ce,
                                cudaStream_t s) {
  if (g.n == 0 || ce <= cb) return;
  // slices of about 1024 columns: a window is a fraction of the columns, and
  // every CTA stages its row block once
  const int Pfull = allpairs_slices(g.n, g.K);
  const int64_t want = (ce - cb) / 1024 / kWarps * kWarps;
  const int P = (int)std::max<int64_t>(kWarps, std::min<int64_t>(Pfull, want));
  const dim3 grid((unsigned)((ce + 31) / 32), (unsigned)(P / kWarps));
  float lo, hi, lo16;
  prefilter_bands(g.S, g.prefilter_eps, &lo, &hi, &lo16);
  const int v = allpairs_variant(g);
  const size_t smem = tc_smem(v, g.mpad, g.Su);
#define RBG_TW(KS, SM)                                                                        \
  do {                                                                                        \
    smem_cap_max((const void *)k_allpairs_tc_win<KS, SM>);                                    \
    k_allpairs_tc_win<KS, SM><<<grid, kWarps * 32, smem, s>>>(g, P, lo, hi, lo16, o, cb, ce); \
  } while (0)
  if (v == 1) RBG_TW(1, 16);
  else if (v == 2) RBG_TW(2, 32);
  else RBG_TW(4, 64);
#undef RBG_TW
}

void launch_rows_topk_counts(const GraphArgs &g, const SymOut &o, const uint32_t *svtab,
                             int64_t *rowoff, uint64_t *keys, cudaStream_t s) {
  if (g.n == 0) return;
  launch_exclusive_scan(o.rowcnt, rowoff, g.n, s);
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  k_scatter_pairs<<<(unsigned)(sms * 32), 256, 0, s>>>(o, rowoff, keys, svtab);
  k_select_rows<<<(unsigned)((g.n + kMergeWarps - 1) / kMergeWarps), kMergeWarps * 32, 0, s>>>(
      g, rowoff, keys);
}

void launch_rows_topk(const GraphArgs &g, const SymOut &o, int64_t *rowoff, uint64_t *keys,
                      cudaStream_t s) {
  if (g.n == 0) return;
  launch_exclusive_scan(o.rowcnt, rowoff, g.n, s);
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  k_scatter_pairs<<<(unsigned)(sms * 32), 256, 0, s>>>(o, rowoff, keys, nullptr);   // a few pairs per thread
  k_select_rows<<<(unsigned)((g.n + kMergeWarps - 1) / kMergeWarps), kMergeWarps * 32, 0, s>>>(
      g, rowoff, keys);
}

void launch_rows_topk_batch(const BatchAsm *B, const int64_t *row0s, int nb, int64_t rows,
                            const SymOut &o, int64_t *rowoff, uint64_t *keys, cudaStream_t s) {
  if (rows == 0) return;
  launch_exclusive_scan(o.rowcnt, rowoff, rows, s);
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  k_scatter_pairs<<<(unsigned)(sms * 32), 256, 0, s>>>(o, rowoff, keys, nullptr);
  k_select_rows_batch<<<(unsigned)((rows + kMergeWarps - 1) / kMergeWarps), kMergeWarps * 32, 0,
                        s>>>(B, row0s, nb, rows, rowoff, keys);
}

void launch_allpairs_batch(const BatchAsm *B, int variant, const int32_t *list,
                           const int64_t *item0s, int nv, int64_t items, size_t smem,
                           unsigned long long *next, const SymOut &o, cudaStream_t s) {
  if (items == 0 || nv == 0) return;
  int dev = 0, sms = 148, per_sm = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
#define RBG_PB(KS, SM)                                                                         \
  do {                                                                                         \
    smem_cap_max((const void *)k_allpairs_batch<KS, SM>);                                      \
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_allpairs_batch<KS, SM>,           \
                                                  kWarps * 32, smem);                          \
    const int64_t grid = std::min<int64_t>(items, (int64_t)std::max(per_sm, 1) * sms);         \
    k_allpairs_batch<KS, SM><<<(unsigned)grid, kWarps * 32, smem, s>>>(B, list, item0s, nv,    \
                                                                       items, next, o);        \
  } while (0)
  if (variant == 1) RBG_PB(1, 16);
  else if (variant == 2) RBG_PB(2, 32);
  else if (variant == 4) RBG_PB(4, 64);
  else RBG_PB(0, 4);
#undef RBG_PB
}

void launch_merge_batch(const BatchAsm *B, const int64_t *row0s, int nb, int64_t rows,
                        cudaStream_t s, int64_t r_begin) {
  if (rows <= r_begin) return;
  k_merge_batch<<<(unsigned)((rows - r_begin + kMergeWarps - 1) / kMergeWarps), kMergeWarps * 32,
                  0, s>>>(B, row0s, nb, r_begin, rows);
}

}  // namespace rbg
