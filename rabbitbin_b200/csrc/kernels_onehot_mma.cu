// Dense regime on the 5th-generation tensor cores, hand-written for sm_100a.
//
// The register-match count of contigs i and j (pmh_match_count16,
// src/rabbitbin.cpp:1261-1293: registers with equal nonzero codes) is the dot
// product X_i . X_j of their binary one-hot rows over the (register, code)
// pairs that occur in the assembly (kernels_onehot.cu builds X).  The small
// path (build_graph_allpairs, src/impl/rb_graph.cpp:7-72) needs every pair's
// count, so the counts are one int8 contraction X X^T, computed here with
// tcgen05.mma kind::i8 into TMEM and consumed in the same kernel: no count
// matrix is written to memory.
//
// CTA tile: 256 rows x 256 columns = two UMMA 128x256 accumulators (A rows
// 0-127 and 128-255 against the same B columns), which fill the 512 TMEM
// columns of the SM.  The one-hot width is walked in chunks of 128 bytes (one
// 128-byte swizzle atom): TMA brings the chunk of the 256 A rows and the 256
// B rows (64 KB) into a 3-stage shared-memory ring.  Warp 0 issues the TMA
// loads, warp 1 allocates TMEM and issues the MMAs (4 K-steps of 32 per
// chunk per accumulator), warps 2-17 are the epilogue: each thread owns one
// row and one 128-column half of the tile, reads its 128 counts from TMEM in
// one load as 16-bit values (tcgen05.ld 32x32b .pack::16b; the counts are at
// most m < 4096), frees TMEM for the next tile's MMAs at once, and then keeps
// the row maxima and appends the candidates above the admission floor to its
// own list in global memory while the next tile's MMAs run.
//
// List keys are 32 bits: rank << 20 | (0xFFFFF - j), where rank is the dense
// rank of the pair's similarity among the distinct values of the similarity
// table (k_sv_rank; the table is non-decreasing in the count).  Their order is
// the order of the similarity keys (similarity bits << 32 | ~j) the other
// dense kernels rank by, ties in the similarity included, for j < 2^20.  A
// list holds up to 1024 keys; with room for every column of its group no cut
// ever runs in the kernel, otherwise a list that reaches its capacity is cut
// to the K best by the warp together (select_topk32), which raises its
// threshold.
//
// Work split: the CTAs form a GR x GC grid; CTA (a, b) takes the row blocks
// a, a + GR, ... and, in each, the column tiles of column group b, so at any
// moment GR row blocks and GC column tiles are in use (their operands stay in
// L2).  Each (row, column group, half) has its own list: k_merge_onehot then
// selects a row's top-K from its 2 GC lists and writes the similarity keys,
// exactly what the other dense kernels produce (top-K keys over the
// candidates above the admission floor, maxima over all other contigs and
// over the candidates).
//
// That form scores every ordered pair.  It takes the rows of a rank of a sharded
// assembly and assemblies above 32,768 contigs; up to there a whole assembly goes
// through k_onehot_sym below, which computes each pair once.
//
// Every wait on an mbarrier is bounded (2 s of %globaltimer); a wait that
// runs out records an error code for the host and the CTA stops issuing work,
// waits (bounded) for its own copies and MMAs in flight, frees its TMEM and
// returns.  No TMA load uses cluster multicast.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>

#include "rbg_internal.h"
#include "select_topk.cuh"
#include "tc05.cuh"

namespace rbg {
namespace {

using namespace tc05;

constexpr int kTM = 256;                      // rows per CTA tile
constexpr int kTN = 256;                      // columns per CTA tile
constexpr int kKC = 128;                      // one-hot bytes per stage (one swizzle atom)
constexpr int kStages = 3;
constexpr int kHalfBytes = 128 * kKC;         // one 128-row operand block: 16 KB
constexpr int kStageBytes = (kTM + kTN) * kKC;   // 64 KB
constexpr int kEpiWarps = 16;
constexpr int kCapW32 = 32;                   // list capacity: 32 * kCapW32 keys
constexpr int kThreads = (2 + kEpiWarps) * 32;
constexpr unsigned FULL = 0xffffffffu;

// instruction descriptor: D s32 (bits 4-5 = 2), A and B unsigned 8-bit (bits
// 7-9, 10-12 = 0), both K-major (bits 15, 16 = 0), N >> 3 at bits 17-22,
// M >> 4 at bits 24-28
constexpr uint32_t kIdesc = (2u << 4) | ((uint32_t)(kTN >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);

struct OhArgs {
  GraphArgs g;
  int64_t rows;          // rows scored: [g.row_lo, g.row_lo + rows)
  int nkc;               // one-hot chunks of 128 bytes
  int RB, NT;            // 256-row blocks, 256-column tiles
  int GR, GC;            // CTA grid: row groups x column groups
  uint32_t *cand;        // [rows32 x 2 GC x 32] lists of cap keys
  int cap;               // keys per list (multiple of 32, <= 1024, >= K + 136)
  int32_t *cand_cnt;     // [rows32 x 2 GC x 32]
  const uint32_t *tab;   // rank[m + 1], value[m + 1], admission count, count-key flag
  int *err;              // set when a bounded wait runs out
};

__device__ __forceinline__ void mma_i8_id(uint32_t dt, uint64_t ad, uint64_t bd, uint32_t idesc,
                                          uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(dt), "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void mma_i8(uint32_t dt, uint64_t ad, uint64_t bd, uint32_t acc) {
  mma_i8_id(dt, ad, bd, kIdesc, acc);
}

// 128 consecutive TMEM columns of this warp's 32 lanes as 16-bit values, two
// per register (column 2k in the low half of v[k]); the counts are below 2^16.
__device__ __forceinline__ void tmem_ld128_pack16(uint32_t taddr, uint32_t (&v)[64]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.pack::16b.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, %48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31]), "=r"(v[32]), "=r"(v[33]), "=r"(v[34]), "=r"(v[35]), "=r"(v[36]), "=r"(v[37]), "=r"(v[38]), "=r"(v[39]), "=r"(v[40]), "=r"(v[41]), "=r"(v[42]), "=r"(v[43]), "=r"(v[44]), "=r"(v[45]), "=r"(v[46]), "=r"(v[47]), "=r"(v[48]), "=r"(v[49]), "=r"(v[50]), "=r"(v[51]), "=r"(v[52]), "=r"(v[53]), "=r"(v[54]), "=r"(v[55]), "=r"(v[56]), "=r"(v[57]), "=r"(v[58]), "=r"(v[59]), "=r"(v[60]), "=r"(v[61]), "=r"(v[62]), "=r"(v[63])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Named barrier 1 of the epilogue warps; returns the OR of every thread's flag.
__device__ __forceinline__ uint32_t epi_barrier_or(uint32_t flag) {
  uint32_t out;
  asm volatile(
      "{\n\t.reg .pred pi, po;\n\t"
      "setp.ne.u32 pi, %1, 0;\n\t"
      "barrier.cta.red.or.pred po, 1, %2, pi;\n\t"
      "selp.u32 %0, 1, 0, po;\n\t}"
      : "=r"(out)
      : "r"(flag), "n"(kEpiWarps * 32)
      : "memory");
  return out;
}

// Smallest count whose similarity rank is at least R (rank is non-decreasing).
__device__ __forceinline__ uint32_t rank_floor(const uint16_t *rank, int m, uint32_t R) {
  int lo = 0, up = m + 1;
  while (lo < up) {
    const int mid = (lo + up) >> 1;
    if (rank[mid] >= R) up = mid; else lo = mid + 1;
  }
  return (uint32_t)max(lo, 1);
}

// The tiles of CTA (a, b): row blocks a, a + GR, ...; columns tiles
// [c0, c1) of column group b.
__device__ __forceinline__ void col_range(const OhArgs &A, int b, int &c0, int &c1) {
  c0 = (int)((int64_t)b * A.NT / A.GC);
  c1 = (int)((int64_t)(b + 1) * A.NT / A.GC);
}

__global__ void __launch_bounds__(kThreads, 1)
k_onehot_mma(const __grid_constant__ CUtensorMap tmap, const OhArgs A) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // 1024-byte aligned stage ring (the swizzle pattern follows address bits)
  uint8_t *ring = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *bars = (uint64_t *)(ring + kStages * kStageBytes);
  // bars: full[kStages], empty[kStages], tmem_full, tmem_empty, mma_done
  uint32_t *tmem_slot = (uint32_t *)(bars + 2 * kStages + 3);
  uint32_t *nzw = tmem_slot + 4;               // [2][8] candidate-flag words of a tile
  int *abort_flag = (int *)(nzw + 16);
  uint16_t *rank = (uint16_t *)(abort_flag + 4);   // [m + 1] similarity rank of a count
  // [11][512] staged keys of the epilogue threads (slot k of thread t at k * 512 + t)
  uint32_t *stage = (uint32_t *)(((uintptr_t)(rank + A.g.m + 1) + 15) & ~(uintptr_t)15);

  const GraphArgs &g = A.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a = blockIdx.x / A.GC, b = blockIdx.x % A.GC;
  int c0, c1;
  col_range(A, b, c0, c1);
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (kStages + s); };
  const uint32_t tfull = bar0 + 8u * (2 * kStages), tempty = tfull + 8u, mdone = tfull + 16u;

  for (int i = threadIdx.x; i <= g.m; i += kThreads) rank[i] = (uint16_t)A.tab[i];
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, kEpiWarps * 32);
    mbar_init(mdone, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {                               // TMEM: all 512 columns
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;"
                 ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tbase = *tmem_slot;
  const int nrb = (A.RB - a + A.GR - 1) / A.GR;  // row blocks of this CTA

  if (warp == 0) {
    // ── TMA producer ──
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      uint32_t issued = 0;                       // bit s: stage s holds an issued load
      uint32_t last_ph = 0;                      // bit s: phase of its last load
      bool ok = true;
      for (int r = 0; r < nrb && ok; ++r) {
        const int y_a = (int)(g.row_lo + (int64_t)(a + r * A.GR) * kTM);
        for (int ct = c0; ct < c1 && ok; ++ct) {
          for (int kc = 0; kc < A.nkc; ++kc) {
            if (!mbar_wait(empty_bar(s), ph ^ 1u, A.err, 1) || *(volatile int *)abort_flag) {
              ok = false;
              *(volatile int *)abort_flag = 1;
              break;
            }
            const uint32_t dst = smem_u32(ring + (size_t)s * kStageBytes);
            mbar_expect_tx(full_bar(s), kStageBytes);
            tma_load(dst, &tmap, kc * kKC, y_a, full_bar(s));
            tma_load(dst + 2 * kHalfBytes, &tmap, kc * kKC, ct * kTN, full_bar(s));
            issued |= 1u << s;
            last_ph = (last_ph & ~(1u << s)) | (ph << s);
            if (++s == kStages) { s = 0; ph ^= 1u; }
          }
        }
      }
      // copies in flight land before the CTA leaves (already true when the
      // MMAs consumed them)
      for (int t = 0; t < kStages; ++t)
        if ((issued >> t) & 1u) mbar_wait(full_bar(t), (last_ph >> t) & 1u, A.err, 2);
    }
  } else if (warp == 1) {
    // ── MMA issuer ──
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0, tph = 0;
      bool ok = true;
      for (int r = 0; r < nrb && ok; ++r) {
        for (int ct = c0; ct < c1 && ok; ++ct) {
          if (!mbar_wait(tempty, tph ^ 1u, A.err, 3) || *(volatile int *)abort_flag) {
            ok = false;
            *(volatile int *)abort_flag = 1;
            break;
          }
          fence_after();
          for (int kc = 0; kc < A.nkc; ++kc) {
            if (!mbar_wait(full_bar(s), ph, A.err, 4) || *(volatile int *)abort_flag) {
              ok = false;
              *(volatile int *)abort_flag = 1;
              break;
            }
            fence_after();
            const uint32_t st = smem_u32(ring + (size_t)s * kStageBytes);
            const uint64_t da0 = sdesc128(st), da1 = sdesc128(st + kHalfBytes),
                           db = sdesc128(st + 2 * kHalfBytes);
#pragma unroll
            for (int k = 0; k < kKC / 32; ++k) {
              const uint32_t acc = (kc | k) ? 1u : 0u;
              // +32 bytes of K per step: +2 in the descriptor's 16-byte units
              mma_i8(tbase, da0 + 2 * k, db + 2 * k, acc);
              mma_i8(tbase + kTN, da1 + 2 * k, db + 2 * k, acc);
            }
            mma_commit(empty_bar(s));            // the stage is free once these finish
            if (++s == kStages) { s = 0; ph ^= 1u; }
          }
          if (!ok) break;
          mma_commit(tfull);                     // the tile's counts are in TMEM
          tph ^= 1u;
        }
      }
      mma_commit(mdone);                         // every MMA issued has finished
      mbar_wait(mdone, 0, A.err, 5);
    }
  } else {
    // ── epilogue: thread = (row, column half of the tile) ──
    const int e = warp - 2;                      // 0..15
    const int q = warp & 3;                      // TMEM lane quarter of this warp
    const int half = (e >> 2) & 1;               // accumulator 0 or 1
    const int ch = e >> 3;                       // columns [128 ch, 128 ch + 128) of the tile
    const int K = g.K, m = g.m;
    const int n = (int)g.n;                      // < 2^20 (onehot_mma_fits)
    const int P = 2 * A.GC;                      // lists per row: column group x half
    const uint32_t cf = max(A.tab[2 * (m + 1)], 1u);   // counts above the floor
    const bool ident = A.tab[2 * (m + 1) + 1] != 0u;    // keys carry the count
    // Keys go to the list eight at a time (two 16-byte stores): they are staged
    // in shared memory first (up to 11 per thread).  fill (keys in the list)
    // stays a multiple of 8 except after the row's last drain.
    uint32_t *stg = stage + (threadIdx.x - 64);
    uint32_t tph = 0;
    int tcount = 0;
    bool ok = true;
    for (int r = 0; r < nrb && ok; ++r) {
      const int rb = a + r * A.GR;
      const int li = rb * kTM + half * 128 + q * 32 + lane;   // local row
      const int i = (int)g.row_lo + li;
      const bool valid_row = li < A.rows;
      const uint32_t nz_i = valid_row ? g.anynz[i] : 0u;
      uint32_t *buf = nullptr;
      size_t slot = 0;
      if (valid_row) {
        slot = ((size_t)(li >> 5) * P + 2 * b + ch) * 32 + (size_t)(li & 31);
        buf = A.cand + slot * (size_t)A.cap;
      }
      int fill = 0, qn = 0;                      // keys in the list, staged keys
      auto push = [&](uint32_t key) {
        stg[qn * 512] = key;
        ++qn;
      };
      // after every 4 candidates (at most 11 staged): 8 keys to the list
      auto flush = [&]() {
        if (qn >= 8) {
          const uint4 lo = make_uint4(stg[0], stg[512], stg[1024], stg[1536]);
          const uint4 hi = make_uint4(stg[2048], stg[2560], stg[3072], stg[3584]);
          *reinterpret_cast<uint4 *>(buf + fill) = lo;
          *reinterpret_cast<uint4 *>(buf + fill + 4) = hi;
          fill += 8;
          qn -= 8;
          for (int k = 0; k < qn; ++k) stg[k * 512] = stg[(k + 8) * 512];
        }
      };
      auto drain = [&]() {
        for (int k = 0; k < qn; ++k) buf[fill + k] = stg[k * 512];
        fill += qn;
        qn = 0;
      };
      uint32_t thr = 0;                          // after a cut: keys <= thr are out
      uint32_t cthr = cf;
      uint32_t mx_a = 0, mx_c = 0;
      for (int ct = c0; ct < c1; ++ct, ++tcount) {
        // candidate flags of the tile's columns (anynz), one word per warp of the first 8
        if (e < kTN / 32) {
          const int j = ct * kTN + e * 32 + lane;
          const unsigned w = __ballot_sync(FULL, j < n && g.anynz[j]);
          if (lane == 0) nzw[(tcount & 1) * 8 + e] = w;
        }
        uint32_t bad = mbar_wait(tfull, tph, A.err, 6) ? 0u : 1u;
        if (*(volatile int *)abort_flag) bad = 1u;
        // one decision for all epilogue threads (they meet at this barrier every tile)
        bad = epi_barrier_or(bad);
        if (bad) {
          ok = false;
          *(volatile int *)abort_flag = 1;
          break;
        }
        fence_after();
        const uint32_t *nzt = nzw + (tcount & 1) * 8 + ch * 4;
        uint32_t pk[64];                         // the 128 counts, two per register
        tmem_ld128_pack16(tbase + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * kTN + ch * 128),
                          pk);
        fence_before();
        mbar_arrive(tempty);                     // TMEM is free for the next tile's MMAs
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int j0 = ct * kTN + ch * 128 + c * 32;
          // valid columns: j < n and j != i; candidates: valid and (nz_i or nz_j)
          uint32_t vm = ~0u;
          if (j0 + 32 > n) vm = (n <= j0) ? 0u : (~0u >> (32 - (n - j0)));
          if (i >= j0 && i < j0 + 32) vm &= ~(1u << (i - j0));
          if (!valid_row) vm = 0u;
          const uint32_t cm = vm & (nz_i ? ~0u : nzt[c]);
          bool hit = false;
          const bool full = __all_sync(FULL, vm == ~0u && cm == ~0u);   // warp-uniform
          if (full) {
            // both halves at once: maximum and the test against the count threshold
            uint32_t m2 = 0, h2 = 0;
            const uint32_t c2 = cthr * 0x10001u;  // cthr <= m + 1 < 2^16
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              m2 = __vmaxu2(m2, pk[c * 16 + k]);
              h2 |= __vcmpgeu2(pk[c * 16 + k], c2);
            }
            const uint32_t cmx = max(m2 & 0xFFFFu, m2 >> 16);
            mx_a = max(mx_a, cmx);
            mx_c = max(mx_c, cmx);
            hit = h2 != 0u;
          } else {
#pragma unroll
            for (int t = 0; t < 32; ++t) {
              const uint32_t v = (pk[c * 16 + (t >> 1)] >> (16 * (t & 1))) & 0xFFFFu;
              const uint32_t va = ((vm >> t) & 1u) ? v : 0u;
              const uint32_t vc = ((cm >> t) & 1u) ? v : 0u;
              mx_a = max(mx_a, va);
              mx_c = max(mx_c, vc);
              hit |= vc >= cthr;
            }
          }
          if (hit) {
            const uint32_t jr = 0xFFFFFu - (uint32_t)j0;
            if (ident && full) {                 // the common case: count keys, every column
#pragma unroll
              for (int t = 0; t < 32; ++t) {
                const uint32_t v = (pk[c * 16 + (t >> 1)] >> (16 * (t & 1))) & 0xFFFFu;
                const uint32_t key = (v << 20) + (jr - (uint32_t)t);
                if (v >= cthr && key > thr) push(key);
                if ((t & 3) == 3) flush();
              }
            } else {
#pragma unroll
              for (int t = 0; t < 32; ++t) {
                const uint32_t v = (pk[c * 16 + (t >> 1)] >> (16 * (t & 1))) & 0xFFFFu;
                if (((cm >> t) & 1u) && v >= cthr) {
                  const uint32_t key = ((ident ? v : (uint32_t)rank[v]) << 20) | (jr - (uint32_t)t);
                  if (key > thr) push(key);
                }
                if ((t & 3) == 3) flush();
              }
            }
          }
        }
        // lists that could not take another tile (128 keys) are cut to the K best
        unsigned need = __ballot_sync(FULL, fill + qn > A.cap - 128);
        if ((need >> lane) & 1u) drain();
        while (need) {
          const int L = __ffs(need) - 1;
          need &= need - 1;
          uint32_t *lb = (uint32_t *)__shfl_sync(FULL, (unsigned long long)buf, L);
          const int lc = __shfl_sync(FULL, fill, L);
          __syncwarp();
          const uint32_t t = select_topk32<kCapW32>(lb, lc, K);
          if (lane == L) {
            thr = t;
            fill = (K + 7) & ~7;                 // zero keys pad to a multiple of 8
            for (int k = K; k < fill; ++k) buf[k] = 0u;
            cthr = ident ? max(t >> 20, 1u) : rank_floor(rank, m, t >> 20);
          }
        }
        tph ^= 1u;
      }
      if (!ok) break;
      // this half's list of the column group (cut by the merge), the maxima
      drain();
      if (valid_row) {
        A.cand_cnt[slot] = fill;
        if (mx_a) atomicMax(g.maxcnt_all + i, mx_a);
        if (mx_c) atomicMax(g.maxcnt_cand + i, mx_c);
      }
      if (b == 0 && ch == 0 && g.stats) {        // every other contig, once per row
        const unsigned vr = __ballot_sync(FULL, valid_row);
        if (lane == 0 && vr)
          atomicAdd(g.stats + 1, (unsigned long long)__popc(vr) * (unsigned long long)(n - 1));
      }
    }
  }
  __syncthreads();
  fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tbase) : "memory");
}

size_t oh_smem(int m) {
  return 1024 + (size_t)kStages * kStageBytes + (2 * kStages + 3) * 8 + 16 + 64 + 16 +
         (size_t)(m + 1) * 2 + 16 + (size_t)11 * kEpiWarps * 32 * 4;
}

// One warp: rank[c] = distinct similarity values below sv[c] (sv is
// non-decreasing in the count), value[rank] = sv bits, the admission count
// (the first count whose similarity is above the floor; m + 1 when none is)
// and the flag of the common case where the similarity strictly increases
// from the admission count on: keys then carry the count instead of the rank
// (the same order) and value[] is indexed by the count.
// tab: rank at [0, m], value at [m + 1, 2m + 1], admission count at 2m + 2,
// the flag at 2m + 3.
__global__ void k_sv_rank(const uint32_t *__restrict__ sv, int m, uint32_t fbits,
                          uint32_t *__restrict__ tab) {
  const int lane = threadIdx.x;
  const int n1 = m + 1, per = (n1 + 31) / 32;
  const int a = min(lane * per, n1), b = min(a + per, n1);
  int ch = 0;
  uint32_t first = (uint32_t)n1;
  for (int c = a; c < b; ++c) {
    const uint32_t x = sv[c];
    if (c > 0 && x != sv[c - 1]) ++ch;
    if (first == (uint32_t)n1 && x > fbits) first = (uint32_t)c;
  }
  int inc = ch;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(FULL, inc, d);
    if (lane >= d) inc += t;
  }
  uint32_t r = (uint32_t)(inc - ch);
  for (int c = a; c < b; ++c) {
    const uint32_t x = sv[c];
    if (c > 0 && x != sv[c - 1]) ++r;
    tab[c] = r;
    tab[n1 + r] = x;                             // equal values for equal ranks
  }
  first = __reduce_min_sync(FULL, first);
  __syncwarp();
  // the similarity strictly increases from the admission count on: the count
  // itself orders the keys, and value[] is indexed by the count
  const bool ident = first < (uint32_t)n1 && tab[m] - tab[first] == (uint32_t)m - first;
  if (ident) {
    __syncwarp();
    for (int c = a; c < b; ++c) tab[n1 + c] = sv[c];
  }
  if (lane == 0) {
    tab[2 * n1] = first;
    tab[2 * n1 + 1] = ident ? 1u : 0u;
  }
}

// Warp per row: the K best of the row's P lists of 32-bit keys (list of row
// r, list s at ((r/32 * P + s) * 32 + r%32) * cap), 32 keys a step into a
// 1024-key shared buffer that select_topk32 cuts to K when it could not take
// another step; after the first cut only keys above the K-th best so far are
// kept.  The kept keys leave as similarity keys (similarity bits << 32 | ~j).
constexpr int kOmWarps = 8;
constexpr int kOmBuf = 32 * kCapW32;
constexpr int kOmDepth = 8;                    // steps of 32 keys loaded ahead

__global__ void __launch_bounds__(kOmWarps * 32)
k_merge_onehot(GraphArgs g, const uint32_t *__restrict__ cand, const int32_t *__restrict__ cnt,
               int cap, int P, const uint32_t *__restrict__ tab, int64_t rows) {
  __shared__ uint32_t mk[kOmWarps][kOmBuf];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int64_t q = (int64_t)blockIdx.x * kOmWarps + wib;
  if (q >= rows) return;
  const int64_t row = g.row_lo + q;
  const int K = g.K;
  uint32_t *keys = mk[wib];
  const size_t br0 = (size_t)(q >> 5) * P * 32 + (size_t)(q & 31);
  const int cl = lane < P ? cnt[br0 + (size_t)lane * 32] : 0;    // P <= 32
  const unsigned below = (1u << lane) - 1u;
  int fill = 0;
  uint32_t thr = 0;
  for (int s = 0; s < P; ++s) {
    const int c = __shfl_sync(FULL, cl, s);
    const uint32_t *src = cand + (br0 + (size_t)s * 32) * cap;
    for (int i0 = 0; i0 < c; i0 += 32 * kOmDepth) {
      uint32_t kv[kOmDepth];                     // the loads of several steps in flight
#pragma unroll
      for (int u = 0; u < kOmDepth; ++u) {
        const int i = i0 + 32 * u + lane;
        kv[u] = i < c ? __ldg(src + i) : 0u;
      }
#pragma unroll
      for (int u = 0; u < kOmDepth; ++u) {
        const bool take = kv[u] > thr;
        const unsigned m = __ballot_sync(FULL, take);
        if (take) keys[fill + __popc(m & below)] = kv[u];
        fill += __popc(m);
        __syncwarp();
        if (fill > kOmBuf - 32) {
          thr = select_topk32<kCapW32>(keys, fill, K);
          fill = K;
        }
      }
    }
  }
  if (fill > K) {
    select_topk32<kCapW32>(keys, fill, K);
    fill = K;
  }
  const uint32_t *value = tab + g.m + 1;
  for (int i = lane; i < fill; i += 32) {
    const uint32_t key = keys[i];
    const uint32_t j = 0xFFFFFu - (key & 0xFFFFFu);
    g.topk[row * K + i] = ((uint64_t)__ldg(value + (key >> 20)) << 32) | (uint64_t)(~j);
  }
  if (lane == 0) g.topk_cnt[row] = fill;
}

// ── whole assemblies: every pair once, counts to memory ─────────────────────
// The count of (i, j) is that of (j, i), so the tiles on and above the diagonal
// hold every count: half the contraction, which bounds the kernel above.  A tile
// cannot feed the lists of its columns' rows, though (a row's list belongs to one
// thread), so each tile leaves its 16-bit counts in a matrix C, in both
// orientations (a 32 x 32 block is transposed in registers), and
// k_select_counts takes every row's top-K from its row of C.  A tile on the
// diagonal loads its rows once.  20,011 contigs, m = 500 (rows of 5,760 bytes):
// 1.37 ms + 0.50 ms for the lists' merge -> 0.72 ms + 0.35 ms; of that the tensor
// pipe needs about 0.5 ms at 4.5 PFLOP/s and the 0.8 GB of counts 0.25 ms, written
// and read.
//
// MB 128-row blocks a side: tiles of 256 x 256 read each operand byte for 256
// counts and run at the tensor rate; with few contigs 128 x 128 tiles occupy
// more SMs.  Tiles are walked in bands of kBandRows row blocks, down each
// column: the CTAs of a wave share about 12 + 12 blocks' rows in L2.  A staged call in
// bands of 3 / 12 / all: 20,011 contigs 2.20 / 2.16 / 2.21 ms, 32,000 4.12 / 4.03 /
// 4.31, up to 12,000 all within 1%.
constexpr int kBandRows = 12;

template <int MB>
struct SymCfg {
  static constexpr int T = 128 * MB;                       // rows and columns of a tile
  static constexpr int kStageB = 2 * T * kKC;
  static constexpr int kSt = 3 * 65536 / kStageB;          // 192 KB of stages
  static constexpr int kBlk = MB == 2 ? 4 : 1;             // 32-column blocks of an epilogue warp
  static constexpr uint32_t kId =
      (2u << 4) | ((uint32_t)(T >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
};

struct SymArgs {
  int n, NB;             // contigs, tile blocks a side
  int nkc;               // one-hot chunks of 128 bytes
  int tiles;             // NB (NB + 1) / 2
  uint16_t *C;           // [n][ldc] counts
  int64_t ldc;
  int *err;
};

// Tile t: row block I and column block J >= I.
__device__ __forceinline__ void sym_tile(int t, int NB, int &I, int &J) {
  int s0 = 0, h = 0;
  for (;; s0 += h) {
    h = min(kBandRows, NB - s0);
    const int cnt = h * (h + 1) / 2 + h * (NB - s0 - h);
    if (t < cnt) break;
    t -= cnt;
  }
  const int tri = h * (h + 1) / 2;
  if (t < tri) {
    int c = 0;
    while ((c + 1) * (c + 2) / 2 <= t) ++c;
    I = s0 + t - c * (c + 1) / 2;
    J = s0 + c;
  } else {
    const int u = t - tri;
    J = s0 + h + u / h;
    I = s0 + u % h;
  }
}

// 32 consecutive TMEM columns as 16-bit values, two per register (no wait).
__device__ __forceinline__ void tmem_ld32_pack16(uint32_t taddr, uint32_t *v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.pack::16b.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}

// 64 bytes (16-byte aligned pointer, 64-byte aligned here) in two 32-byte stores.
__device__ __forceinline__ void store64(uint16_t *p, const uint32_t *v) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p + 16 * h),
                 "r"(v[8 * h]), "r"(v[8 * h + 1]), "r"(v[8 * h + 2]), "r"(v[8 * h + 3]),
                 "r"(v[8 * h + 4]), "r"(v[8 * h + 5]), "r"(v[8 * h + 6]), "r"(v[8 * h + 7])
                 : "memory");
}

// 32 x 32 16-bit values, lane = row, columns 2k and 2k + 1 in v[k]; afterwards
// lane = column, rows 2k and 2k + 1 in v[k].  Bit b of the row (lane) and column
// (register, half) indices are exchanged one b at a time.
__device__ __forceinline__ void transpose32(uint32_t *v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int b = 4; b >= 1; --b) {
    const bool up = (lane >> b) & 1;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      if (k & (1 << (b - 1))) continue;
      const int k1 = k | (1 << (b - 1));
      const uint32_t got = __shfl_xor_sync(FULL, up ? v[k] : v[k1], 1 << b);
      v[k] = up ? got : v[k];
      v[k1] = up ? v[k1] : got;
    }
  }
  const uint32_t sel = (lane & 1) ? 0x3276u : 0x5410u;     // odd: (partner's, my) high halves
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = __byte_perm(v[k], __shfl_xor_sync(FULL, v[k], 1), sel);
}

template <int MB>
__global__ void __launch_bounds__(kThreads, 1)
k_onehot_sym(const __grid_constant__ CUtensorMap tmap, const SymArgs A) {
  using F = SymCfg<MB>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *ring = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *bars = (uint64_t *)(ring + F::kSt * F::kStageB);
  // bars: full[kSt], empty[kSt], tmem_full, tmem_empty, mma_done
  uint32_t *tmem_slot = (uint32_t *)(bars + 2 * F::kSt + 3);
  int *abort_flag = (int *)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (F::kSt + s); };
  const uint32_t tfull = bar0 + 8u * (2 * F::kSt), tempty = tfull + 8u, mdone = tfull + 16u;

  if (threadIdx.x == 0) {
    for (int s = 0; s < F::kSt; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, kEpiWarps * 32);
    mbar_init(mdone, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;"
                 ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tbase = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0, issued = 0, last_ph = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < A.tiles && ok; t += gridDim.x) {
        int I, J;
        sym_tile(t, A.NB, I, J);
        for (int kc = 0; kc < A.nkc; ++kc) {
          if (!mbar_wait(empty_bar(s), ph ^ 1u, A.err, 11) || *(volatile int *)abort_flag) {
            ok = false;
            *(volatile int *)abort_flag = 1;
            break;
          }
          const uint32_t dst = smem_u32(ring + (size_t)s * F::kStageB);
          mbar_expect_tx(full_bar(s), I == J ? F::kStageB / 2 : F::kStageB);
          tma_load(dst, &tmap, kc * kKC, I * F::T, full_bar(s));
          if (I != J) tma_load(dst + F::T * kKC, &tmap, kc * kKC, J * F::T, full_bar(s));
          issued |= 1u << s;
          last_ph = (last_ph & ~(1u << s)) | (ph << s);
          if (++s == F::kSt) { s = 0; ph ^= 1u; }
        }
      }
      // copies in flight land before the CTA leaves
      for (int t = 0; t < F::kSt; ++t)
        if ((issued >> t) & 1u) mbar_wait(full_bar(t), (last_ph >> t) & 1u, A.err, 12);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0, tph = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < A.tiles && ok; t += gridDim.x) {
        int I, J;
        sym_tile(t, A.NB, I, J);
        if (!mbar_wait(tempty, tph ^ 1u, A.err, 13) || *(volatile int *)abort_flag) {
          *(volatile int *)abort_flag = 1;
          break;
        }
        fence_after();
        for (int kc = 0; kc < A.nkc; ++kc) {
          if (!mbar_wait(full_bar(s), ph, A.err, 14) || *(volatile int *)abort_flag) {
            ok = false;
            *(volatile int *)abort_flag = 1;
            break;
          }
          fence_after();
          const uint32_t st = smem_u32(ring + (size_t)s * F::kStageB);
          const uint64_t db = sdesc128(I == J ? st : st + F::T * kKC);
#pragma unroll
          for (int k = 0; k < kKC / 32; ++k) {
            const uint32_t acc = (kc | k) ? 1u : 0u;
#pragma unroll
            for (int h = 0; h < MB; ++h)
              mma_i8_id(tbase + h * F::T, sdesc128(st + h * kHalfBytes) + 2 * k, db + 2 * k, F::kId,
                        acc);
          }
          mma_commit(empty_bar(s));
          if (++s == F::kSt) { s = 0; ph ^= 1u; }
        }
        if (!ok) break;
        mma_commit(tfull);
        tph ^= 1u;
      }
      mma_commit(mdone);                         // every MMA issued has finished
      mbar_wait(mdone, 0, A.err, 15);
    }
  } else {
    const int grp = (warp - 2) >> 2, q = warp & 3;   // four warps of a group: the TMEM lane quarters
    const int half = MB == 2 ? grp & 1 : 0;
    const int col = MB == 2 ? (grp >> 1) * 128 : grp * 32;
    uint32_t tph = 0;
    for (int t = blockIdx.x; t < A.tiles; t += gridDim.x) {
      int I, J;
      sym_tile(t, A.NB, I, J);
      const bool bad = !mbar_wait(tfull, tph, A.err, 16) || *(volatile int *)abort_flag;
      if (__any_sync(FULL, bad)) {
        *(volatile int *)abort_flag = 1;
        break;
      }
      fence_after();
      uint32_t v[16 * F::kBlk];                  // 32 columns (16 registers) a block
#pragma unroll
      for (int c = 0; c < F::kBlk; ++c)
        tmem_ld32_pack16(tbase + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * F::T + col + 32 * c),
                         v + 16 * c);
      tmem_wait_ld();
      fence_before();
      mbar_arrive(tempty);                       // TMEM is free for the next tile's MMAs
      const int i0 = I * F::T + half * 128 + q * 32, j0 = J * F::T + col;
#pragma unroll
      for (int c = 0; c < F::kBlk; ++c) {
        const int jc = j0 + 32 * c;
        if (i0 + lane < A.n) store64(A.C + (int64_t)(i0 + lane) * A.ldc + jc, v + 16 * c);
        if (I != J) {                            // warp-uniform
          transpose32(v + 16 * c);
          if (jc + lane < A.n) store64(A.C + (int64_t)(jc + lane) * A.ldc + i0, v + 16 * c);
        }
      }
      tph ^= 1u;
    }
  }
  __syncthreads();
  fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tbase) : "memory");
}

template <int MB>
size_t sym_smem() {
  using F = SymCfg<MB>;
  return 1024 + (size_t)F::kSt * F::kStageB + (2 * F::kSt + 3) * 8 + 16;
}

constexpr uint32_t kTop = 0x80008000u;

// Largest of a lane's counts, and how many (with bit 15 set) are at least T.
template <int R>
__device__ __forceinline__ uint32_t largest(const uint32_t (&x)[R]) {
  uint32_t m2 = 0;
#pragma unroll
  for (int k = 0; k < R; ++k) m2 = __vmaxu2(m2, x[k]);
  return max(m2 & 0xFFFFu, m2 >> 16);
}

template <int R>
__device__ __forceinline__ uint32_t at_least(const uint32_t (&x)[R], uint32_t T) {
  const uint32_t t2 = T * 0x10001u;
  uint32_t acc = 0;
#pragma unroll
  for (int k = 0; k < R; ++k) acc += ((x[k] - t2) & kTop) >> 15;
  return (acc & 0xFFFFu) + (acc >> 16);
}

// A lane's 16-byte words w0, w0 + 32, ... of a row of counts (the row's own and
// those past the row's end 0); the two halves of word r of a 16-byte word are
// columns 8 q + 2 r and 8 q + 2 r + 1.
template <int NV>
__device__ __forceinline__ void load_counts(const uint16_t *C, int64_t ldc, int row, int w0,
                                            uint32_t (&x)[4 * NV]) {
  const uint4 *src = reinterpret_cast<const uint4 *>(C + (int64_t)row * ldc);
  const int words = (int)(ldc >> 3);
  const uint32_t keep = (row & 1) ? 0x0000FFFFu : 0xFFFF0000u;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int q = w0 + 32 * k;
    const uint4 v = q < words ? __ldg(src + q) : make_uint4(0u, 0u, 0u, 0u);
    const int self = q == (row >> 3) ? (row >> 1) & 3 : 4;
    x[4 * k] = self == 0 ? v.x & keep : v.x;
    x[4 * k + 1] = self == 1 ? v.y & keep : v.y;
    x[4 * k + 2] = self == 2 ? v.z & keep : v.z;
    x[4 * k + 3] = self == 3 ? v.w & keep : v.w;
  }
}

// Abundance bits of the columns, eight a byte, when one of the block's rows has
// none (its candidates are then the columns with abundance only).
__device__ __forceinline__ void abundance_bits(const GraphArgs &g, int row0, int rows,
                                               uint8_t *nzb) {
  const int n = (int)g.n;
  if (!__syncthreads_or((int)threadIdx.x < rows && !g.anynz[row0 + threadIdx.x])) return;
  for (int q = threadIdx.x; 8 * q < n; q += blockDim.x) {
    uint32_t b = 0;
    for (int u = 0; u < 8 && 8 * q + u < n; ++u) b |= (g.anynz[8 * q + u] ? 1u : 0u) << u;
    nzb[q] = (uint8_t)b;
  }
  __syncthreads();
}

template <int NV>
__device__ __forceinline__ void mask_counts(const uint8_t *nzb, int n, int w0,
                                            uint32_t (&x)[4 * NV]) {
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int q = w0 + 32 * k;
    const uint32_t b = 8 * q < n ? nzb[q] : 0u;
#pragma unroll
    for (int r = 0; r < 4; ++r)
      x[4 * k + r] &= ((b >> 2 * r & 1u) * 0xFFFFu) | ((b >> (2 * r + 1) & 1u) * 0xFFFF0000u);
  }
}

// Top-K of a row from its counts: W warps a row hold it in registers (NV
// 16-byte words a lane; warp w a contiguous range of columns), find the K-th
// count by halving the range of counts, and write the keys above it, then those
// of its similarity in ascending column order until there are K: the set the
// list kernels keep.  Counts carry bit 15, so that (x - T) keeps bit 15 exactly
// where the count is at least T, two counts a subtraction.
template <int NV, int W>
__device__ __forceinline__ void select_row(const GraphArgs &g, const uint16_t *__restrict__ C,
                                           int64_t ldc, const uint32_t *__restrict__ tab, int row,
                                           uint32_t (&red)[2][8], int (&s_pos)[8],
                                           const uint8_t *nzb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wr = warp & (W - 1);
  const int n = (int)g.n, m = g.m, K = g.K;
  int turn = 0;
  // sum or maximum over the row's warps
  auto combine = [&](uint32_t x, bool mx) -> uint32_t {
    x = mx ? __reduce_max_sync(FULL, x) : __reduce_add_sync(FULL, x);
    if constexpr (W > 1) {
      if (lane == 0) red[turn][warp] = x;
      __syncthreads();
      x = red[turn][0];
#pragma unroll
      for (int w = 1; w < W; ++w) x = mx ? max(x, red[turn][w]) : x + red[turn][w];
      turn ^= 1;
    }
    return x;
  };
  const int w0 = wr * NV * 32 + lane;
  uint32_t x[4 * NV];
  load_counts<NV>(C, ldc, row, w0, x);
  const uint32_t mx_a = combine(largest(x), true);
  uint32_t mx_c = mx_a;
  if (!g.anynz[row]) {
    mask_counts<NV>(nzb, n, w0, x);
    mx_c = combine(largest(x), true);
  }
#pragma unroll
  for (int k = 0; k < 4 * NV; ++k) x[k] |= kTop;
  const uint32_t cf = max(tab[2 * (m + 1)], 1u);       // counts above the floor
  const bool ident = tab[2 * (m + 1) + 1] != 0u;
  uint32_t t_lo = cf, t_hi = cf;                 // [t_lo, t_hi): the K-th similarity's counts
  uint32_t c_hi = 0, total = 0;
  if (mx_c >= cf) total = combine(at_least(x, cf), false);
  if (total > (uint32_t)K) {
    uint32_t lo = cf, hi = mx_c + 1;             // at least K from lo on, fewer from hi on
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (combine(at_least(x, mid), false) >= (uint32_t)K) lo = mid; else hi = mid;
    }
    t_lo = lo;
    t_hi = lo + 1;
    if (!ident) {                                // counts of one similarity
      const uint32_t R = tab[lo];
      while (t_lo > cf && tab[t_lo - 1] == R) --t_lo;
      while (t_hi <= (uint32_t)m && tab[t_hi] == R) ++t_hi;
    }
    c_hi = t_hi <= mx_c ? combine(at_least(x, t_hi), false) : 0u;
  } else {
    c_hi = total;                                // all of them
  }
  if (W == 1 ? lane == 0 : threadIdx.x == 0) {
    s_pos[warp] = 0;
    if (mx_a) atomicMax(g.maxcnt_all + row, mx_a);
    if (mx_c) atomicMax(g.maxcnt_cand + row, mx_c);
    g.topk_cnt[row] = (int)min(total, (uint32_t)K);
  }
  const uint32_t need = total > (uint32_t)K ? (uint32_t)K - c_hi : 0u;   // keys of the K-th similarity
  // candidates of that similarity in the lower columns' warps
  uint32_t eq_before = 0;
  {
    uint32_t eq = 0;
    if (need) {
      const uint32_t lo2 = t_lo * 0x10001u, hi2 = t_hi * 0x10001u;
      uint32_t acc = 0;
#pragma unroll
      for (int k = 0; k < 4 * NV; ++k) acc += (((x[k] - lo2) & ~(x[k] - hi2)) & kTop) >> 15;
      eq = __reduce_add_sync(FULL, (acc & 0xFFFFu) + (acc >> 16));
    }
    if constexpr (W > 1) {
      if (lane == 0) red[turn][warp] = eq;
      __syncthreads();                           // (s_pos, too)
      for (int w = 0; w < wr; ++w) eq_before += red[turn][w];
    } else {
      __syncwarp();
    }
  }
  const uint32_t *value = tab + m + 1;
  uint64_t *out = g.topk + (int64_t)row * K;
  int *pos = &s_pos[W == 1 ? warp : 0];
  const uint32_t lo2 = t_lo * 0x10001u, hi2 = t_hi * 0x10001u;
  const uint16_t *src16 = C + (int64_t)row * ldc;
  auto put = [&](uint32_t at, uint32_t j) {
    const uint32_t cnt = __ldg(src16 + j);
    out[at] = ((uint64_t)__ldg(value + (ident ? cnt : tab[cnt])) << 32) | (uint64_t)(~j);
  };
  if (total == 0) return;
  // a byte of hits for each 16-byte word, four words at a time
  constexpr int KG = NV < 4 ? NV : 4;
#pragma unroll
  for (int k0 = 0; k0 < NV; k0 += KG) {
    uint32_t h4 = 0, e4 = 0;                     // above the K-th similarity, of it
#pragma unroll
    for (int r = 0; r < 4 * KG; ++r) {
      const uint32_t above = (x[4 * k0 + r] - hi2) & kTop;
      const uint32_t tie = (x[4 * k0 + r] - lo2) & ~above & kTop;
      h4 |= ((above >> 15 & 1u) | (above >> 30)) << (2 * r);
      e4 |= ((tie >> 15 & 1u) | (tie >> 30)) << (2 * r);
    }
    if (!need) e4 = 0;
    if (!__any_sync(FULL, (h4 | e4) != 0u)) continue;
#pragma unroll 1
    for (int k = 0; k < KG; ++k, h4 >>= 8, e4 >>= 8) {
      const uint32_t j = 8u * (uint32_t)(w0 + 32 * (k0 + k));
      const uint32_t h = h4 & 0xFFu, e = e4 & 0xFFu;
      if (h) {
        uint32_t at = (uint32_t)atomicAdd(pos, __popc(h));
        for (uint32_t b = h; b; b &= b - 1) put(at++, j + (uint32_t)(__ffs(b) - 1));
      }
      if (!__any_sync(FULL, e != 0u)) continue;
      uint32_t incl = (uint32_t)__popc(e);
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(FULL, incl, d);
        if (lane >= d) incl += o;
      }
      uint32_t at = eq_before + incl - (uint32_t)__popc(e);
      for (uint32_t b = e; b && at < need; b &= b - 1, ++at)
        put(c_hi + at, j + (uint32_t)(__ffs(b) - 1));
      eq_before += __shfl_sync(FULL, incl, 31);
    }
  }
}

__device__ __forceinline__ void count_pairs(const GraphArgs &g) {
  if (g.stats && blockIdx.x == 0 && threadIdx.x == 0)    // every other contig, once per row
    atomicAdd(g.stats + 1, (unsigned long long)g.n * (unsigned long long)(g.n - 1));
}

// A warp a row.
template <int NV>
__global__ void __launch_bounds__(256, NV <= 8 ? 4 : 2)
k_select_counts(GraphArgs g, const uint16_t *__restrict__ C, int64_t ldc,
                const uint32_t *__restrict__ tab) {
  __shared__ uint32_t red[2][8];
  __shared__ int s_pos[8];
  __shared__ uint8_t nzb[NV * 32];
  count_pairs(g);
  const int row0 = (int)blockIdx.x * 8, row = row0 + (threadIdx.x >> 5);
  abundance_bits(g, row0, min(8, (int)g.n - row0), nzb);
  if (row < (int)g.n) select_row<NV, 1>(g, C, ldc, tab, row, red, s_pos, nzb);
}

// Eight warps a row, R <= 8 rows in turn.  Each thread's even and odd columns, of
// each of H parts of them, give 512 H disjoint groups; K of their maxima reach the
// K-th largest maximum, so at least K counts do: H values a thread are searched
// instead of the whole row, and few counts pass (about 1.2 K of 20,000 at K = 200,
// but -512 H ln(1 - K / 512 H) as K nears the groups: over 1,024 at K = 448 of 512).
// These are listed, and each warp selects one row's K best from its list.  A row
// whose list overflows (ties) is selected from registers, as above.
template <int NV, int H>
__global__ void __launch_bounds__(256, NV <= 12 ? 3 : 2)
k_select_counts_rows(GraphArgs g, const uint16_t *__restrict__ C, int64_t ldc,
                     const uint32_t *__restrict__ tab, int R) {
  __shared__ uint32_t list[8][kOmBuf];
  __shared__ uint32_t mx[2][H][256];
  __shared__ unsigned cnt[8];
  __shared__ uint32_t red[2][8];
  __shared__ int s_pos[8];
  __shared__ uint8_t nzb[NV * 32 * 8];
  count_pairs(g);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = (int)g.n, m = g.m, K = g.K;
  const int row0 = (int)blockIdx.x * R, rows = min(R, n - row0);
  const uint32_t cf = max(tab[2 * (m + 1)], 1u);
  const bool ident = tab[2 * (m + 1) + 1] != 0u;
  const int w0 = warp * NV * 32 + lane;
  if (threadIdx.x < 8) cnt[threadIdx.x] = 0;
  abundance_bits(g, row0, rows, nzb);
  for (int r = 0; r < rows; ++r) {
    const int row = row0 + r;
    uint32_t x[4 * NV];
    load_counts<NV>(C, ldc, row, w0, x);
    const bool nz = g.anynz[row] != 0;
    if (!nz) {
      const uint32_t all = __reduce_max_sync(FULL, largest(x));
      if (lane == 0 && all) atomicMax(g.maxcnt_all + row, all);
      mask_counts<NV>(nzb, n, w0, x);
    }
#pragma unroll
    for (int h = 0; h < H; ++h) {
      uint32_t m2 = 0;
#pragma unroll
      for (int k = 4 * NV / H * h; k < 4 * NV / H * (h + 1); ++k) m2 = __vmaxu2(m2, x[k]);
      mx[r & 1][h][threadIdx.x] = m2;
    }
    __syncthreads();
    uint32_t y[8 * H];
#pragma unroll
    for (int k = 0; k < 8 * H; ++k) y[k] = mx[r & 1][k >> 3][32 * (k & 7) + lane];
    const uint32_t top = __reduce_max_sync(FULL, largest(y));
    if (threadIdx.x == 0 && top) {
      if (nz) atomicMax(g.maxcnt_all + row, top);
      atomicMax(g.maxcnt_cand + row, top);
    }
    if (top < cf) continue;
#pragma unroll
    for (int k = 0; k < 8 * H; ++k) y[k] |= kTop;
    uint32_t T = cf, hi = top + 1;               // K maxima reach T, or T = cf
    while (hi - T > 1) {
      const uint32_t mid = (T + hi) >> 1;
      if (__reduce_add_sync(FULL, at_least(y, mid)) >= (uint32_t)K) T = mid; else hi = mid;
    }
    if (!ident)                                  // with every count of T's similarity
      while (T > cf && tab[T - 1] == tab[T]) --T;
    const uint32_t t2 = T * 0x10001u;
    uint32_t hit[(4 * NV + 31) / 32] = {};
#pragma unroll
    for (int k = 0; k < 4 * NV; ++k)
      if (((x[k] | kTop) - t2) & kTop) hit[k >> 5] |= 1u << (k & 31);
#pragma unroll
    for (int h = 0; h < (4 * NV + 31) / 32; ++h)
      for (uint32_t b = hit[h]; b; b &= b - 1) {
        const int k = 32 * h + __ffs(b) - 1;
        const int j = 8 * (w0 + 32 * (k >> 2)) + 2 * (k & 3);
        // (the same masks as the registers had)
        const uint32_t v = __ldg(reinterpret_cast<const uint32_t *>(C + (int64_t)row * ldc + j));
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint32_t c = u ? v >> 16 : v & 0xFFFFu;
          if (c >= T && j + u != row && (nz || g.anynz[j + u])) {
            const unsigned at = atomicAdd(&cnt[r], 1u);
            if (at < kOmBuf)
              list[r][at] = ((ident ? c : tab[c]) << 20) | (0xFFFFFu - (uint32_t)(j + u));
          }
        }
      }
  }
  __syncthreads();
  if (warp < rows && cnt[warp] <= kOmBuf) {
    const int row = row0 + warp;
    uint32_t *keys = list[warp];
    int fill = (int)cnt[warp];
    if (fill > K) {
      if (fill <= 16 * 32) select_topk32<16>(keys, fill, K);
      else select_topk32<kCapW32>(keys, fill, K);
      fill = K;
    }
    const uint32_t *value = tab + m + 1;
    for (int i = lane; i < fill; i += 32) {
      const uint32_t key = keys[i], j = 0xFFFFFu - (key & 0xFFFFFu);
      g.topk[(int64_t)row * K + i] = ((uint64_t)__ldg(value + (key >> 20)) << 32) | (uint64_t)(~j);
    }
    if (lane == 0) g.topk_cnt[row] = fill;
  }
  for (int r = 0; r < rows; ++r)
    if (cnt[r] > kOmBuf) {                       // block-uniform
      select_row<NV, 8>(g, C, ldc, tab, row0 + r, red, s_pos, nzb);
      __syncthreads();
    }
}

template <int NV>
void launch_select_rows_nv(const GraphArgs &g, const uint16_t *C, int64_t ldc, const uint32_t *tab,
                           cudaStream_t s) {
  // Rows a block: fewer with few rows (a staged call, 4 / 8 rows: 5,003 contigs 0.590 /
  // 0.609 ms, 8,000 0.783 / 0.786, 20,011 2.170 / 2.163, 32,000 4.06 / 4.03; 1 row
  // 3 to 8% more).
  const int R = g.n > 8192 ? 8 : 4;
  const unsigned blocks = (unsigned)((g.n + R - 1) / R);
  // A staged call with 512 / 1,024 groups, 25,000 contigs: K = 200 2.87 / 2.90 ms, 300
  // 3.10 / 3.04, 350 3.20 / 3.11, 400 5.04 / 3.17, 448 5.87 / 3.21; 8,000: 350 0.838 /
  // 0.842, 448 0.955 / 0.855
  if (g.K <= 320) k_select_counts_rows<NV, 1><<<blocks, 256, 0, s>>>(g, C, ldc, tab, R);
  else k_select_counts_rows<NV, 2><<<blocks, 256, 0, s>>>(g, C, ldc, tab, R);
}

// A warp a row up to 4,096 columns (16 words a lane), a block above.  (20,011
// contigs: 0.89 ms searching the whole row's registers, 0.35 ms with the lists.)
void launch_select_counts(const GraphArgs &g, const uint16_t *C, int64_t ldc, const uint32_t *tab,
                          cudaStream_t s) {
  const unsigned blocks = (unsigned)((g.n + 7) / 8);
  if (ldc <= 1024) k_select_counts<4><<<blocks, 256, 0, s>>>(g, C, ldc, tab);
  else if (ldc <= 2048) k_select_counts<8><<<blocks, 256, 0, s>>>(g, C, ldc, tab);
  else if (ldc <= 4096) k_select_counts<16><<<blocks, 256, 0, s>>>(g, C, ldc, tab);
  else if (ldc <= 8192) launch_select_rows_nv<4>(g, C, ldc, tab, s);
  else if (ldc <= 16384) launch_select_rows_nv<8>(g, C, ldc, tab, s);
  else if (ldc <= 24576) launch_select_rows_nv<12>(g, C, ldc, tab, s);
  else launch_select_rows_nv<16>(g, C, ldc, tab, s);
}

// Tensor map of the one-hot rows: boxes of one 128-byte chunk of `rows` rows.
bool onehot_map(CUtensorMap *map, const int8_t *X, int64_t ldx, int64_t n, int rows) {
  auto enc = encode_fn();
  if (!enc) return false;
  std::memset(map, 0, sizeof(*map));
  const cuuint64_t dims[2] = {(cuuint64_t)ldx, (cuuint64_t)n};
  const cuuint64_t strides[1] = {(cuuint64_t)ldx};
  const cuuint32_t box[2] = {(cuuint32_t)kKC, (cuuint32_t)rows};
  const cuuint32_t estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void *)X, dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MB>
cudaError_t launch_sym_mb(const CUtensorMap &map, const SymArgs &A, int sms, cudaStream_t s) {
  cudaError_t e;
  {
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    e = cudaFuncSetAttribute(k_onehot_sym<MB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sym_smem<MB>());
  }
  if (e != cudaSuccess) return e;
  k_onehot_sym<MB><<<(unsigned)std::min(A.tiles, sms), kThreads, sym_smem<MB>(), s>>>(map, A);
  return cudaGetLastError();
}

}  // namespace

bool onehot_mma_fits(int64_t n, int m) { return n < ((int64_t)1 << 20) && m < 4096; }

// Keys per (row, column group, half) list: every column the list covers (no
// cut in the kernel) up to 1024, and at least K + 136 so that a tile's 128
// columns always fit after a cut to K (padded to a multiple of 8).  cap_max
// (> 0) lowers it, down to that floor.
int onehot_mma_cap(int64_t n, int GC, int K, int cap_max) {
  const int64_t NT = (n + 255) / 256;
  const int64_t cols = std::min<int64_t>(n, (NT + GC - 1) / GC * 128);
  int cap = (int)std::min<int64_t>(32 * kCapW32, (cols + 136 + 31) / 32 * 32);
  if (cap_max > 0) cap = std::min(cap, cap_max);
  return std::max(cap, (K + 136 + 31) & ~31);
}

// GR x GC CTA grid for RB row blocks and NT column tiles on `sms` SMs: the
// split with the smallest largest share of tiles, then the fewest column
// groups (fewer lists per row), then the fewest CTAs.
void onehot_mma_grid(int RB, int NT, int sms, int *GR, int *GC) {
  int bestR = 1, bestC = 1;
  int64_t best = INT64_MAX;
  for (int gr = 1; gr <= std::min(RB, sms); ++gr)
    for (int gc = 1; gc <= std::min(NT, std::min(16, sms / gr)); ++gc) {
      const int64_t load = (int64_t)((RB + gr - 1) / gr) * ((NT + gc - 1) / gc);
      if (load < best || (load == best && (gc < bestC || (gc == bestC && gr * gc < bestR * bestC)))) {
        best = load;
        bestR = gr;
        bestC = gc;
      }
    }
  *GR = bestR;
  *GC = bestC;
}

// X: [n][ldx] one-hot rows (ldx a multiple of 128, zero padded); the rows
// [g.row_lo, g.row_lo + rows) against every column, on a GR x GC CTA grid.
// cand/cand_cnt hold ceil(rows / 32) * 32 * 2 GC lists of cap keys (cand_cnt
// is zeroed here); tab [2m + 4] receives the rank tables.  The three launches:
// ranks, counts and lists, top-K per row.  Returns RBG_OK or a status with
// *why set.
int launch_onehot_mma(const GraphArgs &g, const int8_t *X, int64_t ldx, int64_t rows,
                      uint32_t *cand, int cap, int32_t *cand_cnt, uint32_t *tab, int *err, int GR,
                      int GC, cudaStream_t s, const char **why) {
  if (ldx % kKC != 0 || ((uintptr_t)X & 15u) != 0 || !onehot_mma_fits(g.n, g.m) || GC > 16 ||
      g.K < 1 || g.K > 448 || cap > 32 * kCapW32 || cap < g.K + 136 || cap % 32 != 0) {
    *why = "one-hot operand layout";
    return RBG_ERR_ARG;
  }
  CUtensorMap map;
  if (!onehot_map(&map, X, ldx, g.n, kTM)) {
    *why = "cuTensorMapEncodeTiled failed";
    return RBG_ERR_CUDA;
  }
  OhArgs A;
  A.g = g;
  A.rows = rows;
  A.nkc = (int)(ldx / kKC);
  A.RB = (int)((rows + kTM - 1) / kTM);
  A.NT = (int)((g.n + kTN - 1) / kTN);
  A.GR = GR;
  A.GC = GC;
  A.cand = cand;
  A.cap = cap;
  A.cand_cnt = cand_cnt;
  A.tab = tab;
  A.err = err;
  const size_t nslots = (size_t)((rows + 31) / 32) * 32 * 2 * GC;
  cudaError_t e = cudaMemsetAsync(cand_cnt, 0, nslots * sizeof(int32_t), s);
  if (e == cudaSuccess) {
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    e = cudaFuncSetAttribute(k_onehot_mma, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)oh_smem(4096));
  }
  if (e == cudaSuccess) {
    k_sv_rank<<<1, 32, 0, s>>>(g.sv_bits, g.m, (uint32_t)(g.key_floor >> 32), tab);
    k_onehot_mma<<<GR * GC, kThreads, oh_smem(g.m), s>>>(map, A);
    if (rows > 0)
      k_merge_onehot<<<(unsigned)((rows + kOmWarps - 1) / kOmWarps), kOmWarps * 32, 0, s>>>(
          g, cand, cand_cnt, cap, 2 * GC, tab, rows);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    *why = cudaGetErrorString(e);
    return RBG_ERR_CUDA;
  }
  return RBG_OK;
}

// Whole assemblies whose count matrix (2 n^2 bytes) and rows (registers of
// k_select_counts) fit.
bool onehot_sym_fits(int64_t n, int m) { return n <= 32768 && m < 4096; }

int64_t onehot_sym_ldc(int64_t n) { return (n + 255) / 256 * 256; }

// X as launch_onehot_mma takes it; C: [n][onehot_sym_ldc(n)] 16-bit counts; tab
// [2m + 4].  The three launches: ranks, counts, top-K and maxima per row.
//
// 128 x 128 tiles while all of them run at once (up to 2,048 contigs on 148 SMs):
// the whole dense pass takes 108 us at 2,000 contigs, 117 with 256 x 256; 144 and
// 134 us at 3,000, where they take a third round.
int launch_onehot_sym(const GraphArgs &g, const int8_t *X, int64_t ldx, uint16_t *C, uint32_t *tab,
                      int *err, int sms, cudaStream_t s, const char **why) {
  if (ldx % kKC != 0 || ((uintptr_t)X & 15u) != 0 || ((uintptr_t)C & 31u) != 0 ||
      !onehot_sym_fits(g.n, g.m) || g.K < 1 || g.row_lo != 0 ||
      (g.row_hi >= 0 && g.row_hi != g.n)) {
    *why = "one-hot operand layout";
    return RBG_ERR_ARG;
  }
  SymArgs A;
  A.n = (int)g.n;
  A.nkc = (int)(ldx / kKC);
  A.C = C;
  A.ldc = onehot_sym_ldc(g.n);
  A.err = err;
  const int nb2 = (int)((g.n + 255) / 256);
  const bool small = nb2 * (2 * nb2 + 1) <= sms;
  const int T = small ? 128 : 256;
  // (columns up to ldc are written with 128-row blocks, too)
  A.NB = small ? 2 * nb2 : nb2;
  A.tiles = A.NB * (A.NB + 1) / 2;
  CUtensorMap map;
  if (!onehot_map(&map, X, ldx, g.n, T)) {
    *why = "cuTensorMapEncodeTiled failed";
    return RBG_ERR_CUDA;
  }
  k_sv_rank<<<1, 32, 0, s>>>(g.sv_bits, g.m, (uint32_t)(g.key_floor >> 32), tab);
  cudaError_t e = small ? launch_sym_mb<1>(map, A, sms, s) : launch_sym_mb<2>(map, A, sms, s);
  if (e == cudaSuccess) {
    launch_select_counts(g, C, A.ldc, tab, s);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    *why = cudaGetErrorString(e);
    return RBG_ERR_CUDA;
  }
  return RBG_OK;
}

}  // namespace rbg
