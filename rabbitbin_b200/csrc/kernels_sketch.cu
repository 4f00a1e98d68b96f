// Sketch stage kernels: 2-bit packing, canonical k-mer counting with GC-norm
// weights, and the ProbMinHash register minimum.
//
// Compiled with -fmad=false: every double operation below rounds exactly like
// the reference's (which has no contracted expression in build_pmh_winners).
#include <algorithm>
#include <cstdint>
#include <mutex>
#include <set>
#include <utility>

#include "rbg_internal.h"

namespace rbg {
namespace {

// Spread the 16 bits of x to the even bit positions of a 32-bit word.
__device__ __forceinline__ uint32_t spread16(uint32_t x) {
  x = (x | (x << 8)) & 0x00FF00FFu;
  x = (x | (x << 4)) & 0x0F0F0F0Fu;
  x = (x | (x << 2)) & 0x33333333u;
  x = (x | (x << 1)) & 0x55555555u;
  return x;
}

// Base encoding: A/a->0, C/c->1, G/g->2, T/t->3, anything else invalid
// (RB_BASE_ENC_LUT, src/rabbit_sketch.h:56-75).
// One thread per 32 bases: two 128-bit loads of ASCII, two packed words out
// (first base in the top two bits) and the mask word of the pair (16 invalid
// bits per word, the first word in the high half).  Four bases per 32-bit
// step: with l = byte | 0x20, ((l >> 1) ^ (l >> 2)) & 3 is 0, 1, 2, 3 for a,
// c, g, t; the letter rebuilt from that code (a byte permute of "acgt") equals
// l exactly for the eight valid letters, which a zero-byte test of the
// difference marks.  Two dot products of four bytes gather the codes and the valid
// bits, first base highest.  Bases past nbases are invalid.  Bound by the integer
// pipe; 406 MB: 158 us with 64-bit multiplies and shifts (pipe 90% busy), 113 us
// so (0.56 GB moved, 85 us at the copy rate).
__device__ __forceinline__ void pack16(const uint4 v, int64_t w, int64_t nbases, uint32_t &word,
                                       uint32_t &bad16) {
  const uint32_t q[4] = {v.x, v.y, v.z, v.w};
  uint32_t good = 0;                                     // 128 x the valid bits
  word = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t l = q[k] | 0x20202020u;
    const uint32_t cw = ((l >> 1) ^ (l >> 2)) & 0x03030303u;
    // the codes as selectors of the letters they stand for
    const uint32_t sel = __byte_perm(cw | (cw >> 4), 0u, 0x4420u);
    const uint32_t y = __byte_perm(0x74676361u, 0u, sel) ^ l;
    const uint32_t ok = ~(((y & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | y) & 0x80808080u;
    word = __dp4a(cw, 0x01041040u, word << 8);
    good = __dp4a(ok, 0x01020408u, good << 4);
  }
  bad16 = ~(good >> 7) & 0xFFFFu;
  if (bad16) word &= ~(spread16(bad16) * 3u);            // rare: invalid bases have code 0
  const int64_t lim = nbases - w * 16;
  if (lim < 16) {
    const int keep = lim > 0 ? (int)lim : 0;
    bad16 |= 0xFFFFu >> keep;
    word &= ~(0xFFFFFFFFu >> (2 * keep));
  }
}

// Words [w_begin, w_end) (w_begin even): thread t packs words w_begin + 2t, + 1.
__global__ void k_pack(const uint4 *__restrict__ ascii, int64_t nbases, int64_t nwords,
                       int64_t w_begin, int64_t w_end, uint32_t *__restrict__ packed,
                       uint32_t *__restrict__ nmask) {
  const int64_t w = w_begin + 2 * ((int64_t)blockIdx.x * blockDim.x + threadIdx.x);
  if (w >= w_end) return;
  const bool two = w + 1 < w_end;
  const uint4 v0 = ascii[w];
  const uint4 v1 = two ? ascii[w + 1] : make_uint4(0u, 0u, 0u, 0u);
  uint32_t p0, b0, p1, b1;
  pack16(v0, w, nbases, p0, b0);
  pack16(v1, w + 1, nbases, p1, b1);
  if (two) {
    *reinterpret_cast<uint2 *>(packed + w) = make_uint2(p0, p1);   // w even: 8-byte aligned
  } else {
    packed[w] = p0;
  }
  nmask[w >> 1] = (b0 << 16) | ((w + 1 < nwords) ? b1 : 0xFFFFu);
}

// Invalid bits of the 16 bases of packed word wi, restricted to [s, e)
// (base t of the word at bit 15 - t; bases before s or from e on are invalid).
__device__ __forceinline__ uint32_t invalid16(const uint32_t *__restrict__ nmask, int64_t wi,
                                              int64_t s, int64_t e) {
  if (wi < 0) return 0xFFFFu;
  const uint32_t mw = __ldg(nmask + (wi >> 1));
  uint32_t b = (wi & 1) ? (mw & 0xFFFFu) : (mw >> 16);
  const int64_t g0 = wi * 16;
  const int64_t dl = s - g0, dh = e - g0;             // first valid, first invalid offset
  if (dl > 0) b |= dl >= 16 ? 0xFFFFu : (0xFFFFu << (16 - (int)dl)) & 0xFFFFu;
  if (dh < 16) b |= dh <= 0 ? 0xFFFFu : 0xFFFFu >> (int)dh;
  return b;
}

// Per contig: histogram of canonical k-mers (k <= 4) and base counts over the
// packed sequence, then the GC-normalised weights of build_pmh_winners
// (src/rabbitbin.cpp:1459-1516) and the ascending element list (rank, 1/w).
// W warps share a contig (W = 1, or all kCountWarps of the CTA).  A lane takes
// one packed word (16 bases) per step, the 3 bases before it come from the
// previous lane; base counts use popcounts over the 2-bit fields.  For k = 4 a
// word whose 16 windows are all valid adds 8 5-mers ending at its odd bases,
// each of which stands for two 4-mers (its first and its last four bases):
// half the shared-memory atomics; the 1,024 5-mer counts are folded into the
// 4-mer histogram once per contig.
// Bound by instruction issue (71% of the slots) around the shared atomics.  Words
// are indexed in 32 bits from the contig's first one, only the first and last take
// an end mask, and k = 4 is compiled on its own: 450 -> 343 us at 50,000 contigs of
// 8 kb (330 -> 249 us at 30,000).
constexpr int kCountWarps = 8;
constexpr int kH5 = 1024;               // 5-mer counters of a group

// A group's (the W warps of a contig) shared memory.
struct CountGroup {
  uint32_t h5[kH5];
  uint32_t hist[256];
  double p[4];                          // base frequencies (mode 2: with pseudocounts)
  double pc[16];                        // mode 2: P(next | prev)
  uint32_t bc[4], dn[16];
  uint32_t tot, pos;
  unsigned next;
  uint32_t pad;
};

// GC2: GC-norm mode 2 (dinucleotide model); K4: k = 4.
template <bool GC2, int W, bool K4>
__global__ void __launch_bounds__(kCountWarps * 32) k_count(SketchArgs a) {
  extern __shared__ __align__(16) unsigned char sh_count[];
  __shared__ uint8_t code_of[kMaxElems];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  constexpr int kG = kCountWarps / W;   // groups per CTA
  constexpr int GT = 32 * W;            // threads of a group
  const int gi = W == 1 ? wib : 0;
  const int gt = W == 1 ? lane : (int)threadIdx.x;
  const int wig = W == 1 ? 0 : wib;     // warp within the group
  CountGroup &G = reinterpret_cast<CountGroup *>(sh_count)[gi];
  auto gsync = [] {
    if constexpr (W == 1) __syncwarp();
    else __syncthreads();
  };
  const int k = K4 ? 4 : a.k;
  const int nb = 1 << (2 * k);
  const uint32_t kmask = (uint32_t)nb - 1u;
  for (int v = threadIdx.x; v < nb; v += blockDim.x) {
    const int e = a.rank_of_code[v];
    if (e >= 0) code_of[e] = (uint8_t)v;
  }
  for (int v = gt; v < kH5; v += GT) G.h5[v] = 0;
  __syncthreads();
  // A group takes its next contig from a.work (a counter zeroed before the
  // launch) when the caller gives one, else every groups-th contig: contig
  // lengths vary by an order of magnitude, and the counter keeps every group
  // busy until the last contigs.
  const int64_t groups = (int64_t)gridDim.x * kG;
  auto next_contig = [&](int64_t cur, bool first) -> int64_t {
    if (a.work == nullptr) return first ? (int64_t)blockIdx.x * kG + gi : cur + groups;
    if constexpr (W == 1) {
      unsigned t = 0;
      if (lane == 0) t = atomicAdd(a.work, 1u);
      return (int64_t)__shfl_sync(0xffffffffu, t, 0);
    } else {
      if (threadIdx.x == 0) G.next = atomicAdd(a.work, 1u);
      __syncthreads();
      return (int64_t)G.next;
    }
  };
  for (int64_t c = next_contig(0, true); c < a.n; c = next_contig(c, false)) {
  for (int v = gt; v < 256; v += GT) G.hist[v] = 0;
  if (gt < 4) G.bc[gt] = 0;
  if (gt < 16) G.dn[gt] = 0;
  if (gt == 0) { G.tot = 0; G.pos = 0; }
  const int64_t s = a.offsets[c], e = a.offsets[c + 1];
  uint32_t bc0 = 0, bc1 = 0, bc2 = 0, bc3 = 0;
  uint32_t dn[GC2 ? 16 : 1] = {};      // mode 2: dinucleotides (prev, next) = dn[4 prev + next]
  gsync();
  if (e - s >= k) {
    // words of the contig by their index j from its first one (contigs are
    // shorter than 2^31 words); only the first and last hold other contigs' bases
    const int64_t w0 = s >> 4;
    const int nw = (int)(((e + 15) >> 4) - w0);
    const uint32_t *words = a.packed + w0;
    const uint32_t *masks = a.nmask + (w0 >> 1);
    const uint32_t odd = (uint32_t)w0 & 1u;
    const uint32_t bad_first = 0xFFFFu & ~(0xFFFFu >> (int)(s & 15));
    const uint32_t bad_last = (e & 15) ? 0xFFFFu >> (int)(e & 15) : 0u;
    auto fetch = [&](int j, uint32_t &cur, uint32_t &bad) {
      cur = 0;
      bad = 0xFFFFu;
      if (j < nw) {
        cur = __ldg(words + j);
        const uint32_t q = (uint32_t)j + odd;
        const uint32_t mw = __ldg(masks + (q >> 1));
        bad = ((q & 1u) ? mw : mw >> 16) & 0xFFFFu;
        if (j == 0) bad |= bad_first;
        if (j == nw - 1) bad |= bad_last;
      }
    };
    // the next step's words, and for lane 0 the word before them
    uint32_t ncur, nbad, npre = 0, nprebad = 0xFFFFu;
    int j0 = 32 * wig;
    fetch(j0 + lane, ncur, nbad);
    if (lane == 0 && j0 > 0) fetch(j0 - 1, npre, nprebad);
    for (; j0 < nw; j0 += 32 * W) {
      const uint32_t cur = ncur, bad = nbad;
      uint32_t prev = __shfl_up_sync(0xffffffffu, cur, 1);
      uint32_t prevbad = __shfl_up_sync(0xffffffffu, bad, 1);
      if (lane == 0) { prev = npre; prevbad = nprebad; }
      const int jn = j0 + 32 * W;
      fetch(jn + lane, ncur, nbad);
      if (lane == 0) fetch(jn - 1, npre, nprebad);
      if (j0 + lane < nw) {
        // base counts of the valid bases (base t occupies bits 31-2t .. 30-2t)
        const uint32_t vs = spread16(~bad & 0xFFFFu);
        const uint32_t hi = (cur >> 1) & 0x55555555u, lo = cur & 0x55555555u;
        bc3 += __popc(hi & lo & vs);
        bc2 += __popc(hi & ~lo & vs);
        bc1 += __popc(~hi & lo & vs);
        bc0 += __popc(~hi & ~lo & vs);
        if constexpr (GC2) {
          // consecutive valid bases (t-1, t); base -1 is the previous word's last
          const uint32_t vprev = ((((~prevbad & 0xFFFFu) << 16) | (~bad & 0xFFFFu)) >> 1) & 0xFFFFu;
          const uint32_t vp = spread16(~bad & vprev & 0xFFFFu);
          const uint32_t q = (uint32_t)((((uint64_t)prev << 32) | cur) >> 2);
          const uint32_t qh = (q >> 1) & 0x55555555u, ql = q & 0x55555555u;
          const uint32_t mb[4] = {~hi & ~lo & vp, ~hi & lo & vp, hi & ~lo & vp, hi & lo & vp};
          const uint32_t ma[4] = {~qh & ~ql, ~qh & ql, qh & ~ql, qh & ql};
#pragma unroll
          for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) dn[4 * x + y] += __popc(ma[x] & mb[y]);
        }
        // k-mers ending at base t: window bases t-k+1 .. t all valid; forward
        // codes are counted and folded onto canonical codes per contig
        const uint32_t winbad = (prevbad << 16) | bad;
        uint32_t any = winbad;
        if constexpr (K4) any |= winbad >> 1 | winbad >> 2 | winbad >> 3;
        else
          for (int q = 1; q < k; ++q) any |= winbad >> q;
        uint32_t kv = ~any & 0xFFFFu;                   // bit 15-t: k-mer ending at t
        const uint64_t win = ((uint64_t)prev << 32) | cur;
        if (K4 && kv == 0xFFFFu) {
          // bases -3 .. 15 are valid: the 5-mers ending at t = 1, 3, .., 15
#pragma unroll
          for (int bp = 14; bp >= 0; bp -= 2)
            atomicAdd(&G.h5[__funnelshift_r(cur, prev, 2 * bp) & (kH5 - 1)], 1u);
        } else if (kv == 0xFFFFu) {
#pragma unroll
          for (int bp = 15; bp >= 0; --bp)
            atomicAdd(&G.hist[(uint32_t)(win >> (2 * bp)) & kmask], 1u);
        } else {
          while (kv) {
            const int bp = __ffs(kv) - 1;               // = 15 - t
            kv &= kv - 1;
            atomicAdd(&G.hist[(uint32_t)(win >> (2 * bp)) & kmask], 1u);
          }
        }
      }
    }
  }
  // base counts of the group
  bc0 = __reduce_add_sync(0xffffffffu, bc0);
  bc1 = __reduce_add_sync(0xffffffffu, bc1);
  bc2 = __reduce_add_sync(0xffffffffu, bc2);
  bc3 = __reduce_add_sync(0xffffffffu, bc3);
  if (lane < 4) atomicAdd(&G.bc[lane], lane == 0 ? bc0 : lane == 1 ? bc1 : lane == 2 ? bc2 : bc3);
  if constexpr (GC2) {
#pragma unroll
    for (int x = 0; x < 16; ++x) {
      const uint32_t t = __reduce_add_sync(0xffffffffu, dn[x]);
      if (lane == 0) atomicAdd(&G.dn[x], t);
    }
  }
  gsync();
  if constexpr (K4) {
    // 5-mer (first four = x, or last four = x) -> 4-mer x
    for (int x = gt; x < 256; x += GT) {
      const uint4 f = *reinterpret_cast<const uint4 *>(&G.h5[4 * x]);
      G.hist[x] += f.x + f.y + f.z + f.w +
                   G.h5[x] + G.h5[256 + x] + G.h5[512 + x] + G.h5[768 + x];
    }
    gsync();
    for (int v = gt; v < kH5 / 4; v += GT)
      reinterpret_cast<uint4 *>(G.h5)[v] = make_uint4(0u, 0u, 0u, 0u);
  }
  // fold each reverse-complement code onto its canonical (the smaller) code
  uint32_t tot = 0;
  for (int v = gt; v < nb; v += GT) {
    uint32_t rev = 0, x = (uint32_t)v;
#pragma unroll
    for (int q = 0; q < k; ++q) { rev = (rev << 2) | (3u - (x & 3u)); x >>= 2; }
    if ((uint32_t)v > rev) continue;
    uint32_t cnt = G.hist[v];
    if ((uint32_t)v < rev) {
      cnt += G.hist[rev];
      G.hist[v] = cnt;
    }
    tot += cnt;
  }
  tot = __reduce_add_sync(0xffffffffu, tot);
  if (lane == 0) atomicAdd(&G.tot, tot);
  gsync();
  tot = G.tot;
  bc0 = G.bc[0]; bc1 = G.bc[1]; bc2 = G.bc[2]; bc3 = G.bc[3];
  const uint64_t vb = (uint64_t)bc0 + bc1 + bc2 + bc3;
  if constexpr (GC2) {
    // mode 2 (src/rabbitbin.cpp:1517-1554): base frequencies with pseudocount 1,
    // P(next | prev) with Laplace pseudocount 1
    if (gt < 4) G.p[gt] = vb > 0 ? ((double)G.bc[gt] + 1.0) / ((double)vb + 4.0) : 0.25;
    if (gt < 16) {
      const int x = gt >> 2;
      double rs = 4.0;
#pragma unroll
      for (int y = 0; y < 4; ++y) rs += (double)G.dn[4 * x + y];
      G.pc[gt] = ((double)G.dn[gt] + 1.0) / rs;
    }
  } else {
    if (gt < 4) G.p[gt] = vb > 0 ? (double)G.bc[gt] / (double)vb : 0.25;
  }
  gsync();
  double *ewinv = a.elem_winv + c * a.n_elems;
  const double inf = __longlong_as_double(0x7FF0000000000000LL);
  const double inv = tot > 0 ? 1.0 / (double)tot : 0.0;
  int pos = 0;
  for (int el = gt; el < a.n_elems; el += GT) {
    const uint32_t v = code_of[el];
    double w = 0.0;
    if (tot > 0) {
      const uint32_t cnt = G.hist[v];
      if (cnt) {
        if (a.gc_norm == 0) {
          w = (double)cnt * inv;
        } else if constexpr (GC2) {
          // bases[i] = (v >> 2i) & 3; forward and reverse-complement chains
          double pf = G.p[v & 3u];
          for (int q = 1; q < k; ++q)
            pf = __dmul_rn(pf, G.pc[4 * ((v >> (2 * q - 2)) & 3u) + ((v >> (2 * q)) & 3u)]);
          double pr = G.p[3u - ((v >> (2 * k - 2)) & 3u)];
          for (int q = 1; q < k; ++q)
            pr = __dmul_rn(pr, G.pc[4 * (3u - ((v >> (2 * (k - q))) & 3u)) +
                                    (3u - ((v >> (2 * (k - 1 - q))) & 3u))]);
          const double obs = (double)cnt * inv;
          const double ex = __dadd_rn(pf, pr);
          if (ex > 1e-16) {
            const double r = obs / ex;
            w = (a.gc_cap < r) ? a.gc_cap : r;
          }
        } else {
          double pf = 1.0, pr = 1.0;
          uint32_t code = v;
          for (int q = 0; q < k; ++q) {
            const uint32_t b = code & 3u;
            pf = __dmul_rn(pf, G.p[b]);
            pr = __dmul_rn(pr, G.p[3u - b]);
            code >>= 2;
          }
          const double obs = (double)cnt * inv;
          const double ex = __dadd_rn(pf, pr);
          if (ex > 1e-14) {
            const double r = obs / ex;
            w = (a.gc_cap < r) ? a.gc_cap : r;
          }
        }
      }
    }
    const bool take = w > 0.0;
    pos += take;
    ewinv[el] = take ? 1.0 / w : inf;
  }
  pos = (int)__reduce_add_sync(0xffffffffu, (unsigned)pos);
  if constexpr (W == 1) {
    if (lane == 0) a.elem_cnt[c] = pos;
    __syncwarp();                      // the next contig clears the histogram
  } else {
    if (lane == 0) atomicAdd(&G.pos, (uint32_t)pos);
    __syncthreads();
    if (threadIdx.x == 0) a.elem_cnt[c] = (int32_t)G.pos;
    __syncthreads();
  }
  }
}

// Register minimum with an exact early exit.  The winner of register r for a
// contig is the element e with the smallest rounded product h = (1/w_e) * U[e][r],
// ties to the smallest e (the reference inserts elements in ascending order with
// a strict <), so the result is the lexicographic minimum of (h, e).
//
// Per contig, the kMHeavy elements with the smallest 1/w are evaluated directly;
// the others are bounded below by wb, the next smallest 1/w.  The elements of
// register r are then visited in ascending U (table `order`, ties by e): once
// round(wb * U_next) > best, no element left can reach best, since each remaining
// element is either already evaluated or has 1/w >= wb and U >= U_next, and a
// rounded product is monotonic in both factors.  Elements met again on the walk
// change nothing.  Absent elements (1/w = +inf) give inf or NaN, never below or
// equal to a finite best.
//
// A CTA holds 32 contigs (lane = contig) with their 1/w rows transposed in shared
// memory ([E][33]: the per-step gather is conflict-free, and so are the stores that
// transpose the rows).  Each warp takes one
// register at a time: the first 32 entries of its visiting order and its U row
// (by element, table UT) are loaded into registers one register ahead, stored in
// the warp's shared slot, and walked in lock step until every lane's bound has
// passed (entries past 32 come straight from the table), two entries a vote and no
// branch on a lane's own bound: with one entry a vote the loop waited on each
// vote and branch.  Winners go to a shared tile and leave as 4-byte code words,
// padding columns included.
//
// Bound by the shared-memory reads of the walk (L1 wavefronts 79%, issue 63% of
// peak); 50,000 contigs, m = 500: 790 -> 491 us (30,000: 600 -> 444 with 8 heavy
// elements; 4 leave half of the direct products out for less than one more step).
constexpr int kMC = 32;          // contigs per CTA, one per lane
constexpr int kMThreads = 256;
constexpr int kMWarps = kMThreads / 32;
constexpr int kMHeavy = 4;       // smallest-1/w elements evaluated directly
constexpr int kMRow = kMC + 1;   // row stride of sW: the transposing stores hit every bank
constexpr int kMChunk = 256;     // registers per pass; a multiple of 16
constexpr int kMWinStride = kMChunk + 4;
constexpr int kMRec = 32;        // visiting-order entries staged per register (one per lane)
constexpr int kMUcPerLane = (kMaxElems / 2 + 31) / 32;   // 16-byte chunks of a U row per lane
static_assert(kMaxElems % 2 == 0 && kMaxElems <= 5 * 32, "U rows in 16-byte chunks, 5 values per lane");

__host__ __device__ constexpr size_t minreduce_smem(int E) {
  return (size_t)E * kMRow * sizeof(double)          // sW   [E][kMRow]
         + (size_t)kMHeavy * kMC * sizeof(double)     // sHw  [kMHeavy][kMC]
         + (size_t)kMC * sizeof(double)               // sWb  [kMC]
         + (size_t)kMWarps * kMRec * 16               // sRec [kMWarps][kMRec]
         + (size_t)kMWarps * E * sizeof(double)       // sUc  [kMWarps][E]
         + (size_t)kMHeavy * kMC                      // sHe  [kMHeavy][kMC]
         + (size_t)kMC * kMWinStride;                 // sWin [kMC][kMWinStride]
}

__device__ __forceinline__ void lex_min(double h, int e, double &best, int &win) {
  if (h <= best) {                       // false for NaN
    if (h < best || e < win) win = e;
    best = h;
  }
}

__device__ __forceinline__ void cswap(uint64_t &a, int &ia, uint64_t &b, int &ib) {
  if (b < a) {
    const uint64_t t = a; a = b; b = t;
    const int u = ia; ia = ib; ib = u;
  }
}

// One register's staging data, loaded a register ahead: entry `lane` of the
// visiting order and the lane's 16-byte chunks of the U row.
struct MinStage {
  double2 rec;
  double2 uc[kMUcPerLane];
};

__device__ __forceinline__ void min_fetch(MinStage &st, const double2 *ord, const double2 *ut,
                                          int r, int E, int lane) {
  const int half = E >> 1;
  st.rec = lane < E ? __ldg(ord + (size_t)r * E + lane) : make_double2(0.0, 0.0);
#pragma unroll
  for (int q = 0; q < kMUcPerLane; ++q) {
    const int ch = lane + 32 * q;
    st.uc[q] = ch < half ? __ldg(ut + (size_t)r * half + ch) : make_double2(0.0, 0.0);
  }
}

__global__ void __launch_bounds__(kMThreads, 3) k_minreduce(SketchArgs a) {
  extern __shared__ __align__(16) unsigned char msh[];
  const int E = a.n_elems, m = a.m, mpad = a.mpad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double *sW = reinterpret_cast<double *>(msh);
  double *sHw = sW + (size_t)E * kMRow;
  double *sWb = sHw + kMHeavy * kMC;
  double2 *sRec = reinterpret_cast<double2 *>(sWb + kMC);
  double *sUc = reinterpret_cast<double *>(sRec + kMWarps * kMRec);
  uint8_t *sHe = reinterpret_cast<uint8_t *>(sUc + (size_t)kMWarps * E);
  uint8_t *sWin = sHe + kMHeavy * kMC;
  double2 *myRec = sRec + warp * kMRec;
  double *myUc = sUc + (size_t)warp * E;
  const int64_t c0 = (int64_t)blockIdx.x * kMC;
  const int nc = (int)(a.n - c0 < kMC ? a.n - c0 : kMC);
  const double inf = __longlong_as_double(0x7FF0000000000000LL);
  const uint64_t kNone = ~0ull;                      // key of a slot that is no element
  for (int i = threadIdx.x; i < kMC * E; i += kMThreads) {
    const int c = i / E, e = i - c * E;
    sW[e * kMRow + c] = c < nc ? __ldg(a.elem_winv + c0 * E + i) : inf;
  }
  // Heavy sets.  A non-negative double orders as its bit pattern, so 1/w values
  // are compared as 64-bit keys.  Each lane sorts its (up to 5) values; kMHeavy + 1
  // rounds of a warp minimum over the lanes' heads take one element each (the
  // lowest lane on ties), the last round giving the bound.
  for (int c = warp; c < kMC; c += kMWarps) {
    uint64_t v[5];
    int id[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const int e = lane + 32 * j;
      id[j] = e;
      v[j] = (c < nc && e < E) ? (uint64_t)__double_as_longlong(__ldg(a.elem_winv + (c0 + c) * E + e))
                                : kNone;
    }
    cswap(v[0], id[0], v[1], id[1]); cswap(v[3], id[3], v[4], id[4]);
    cswap(v[2], id[2], v[4], id[4]); cswap(v[2], id[2], v[3], id[3]);
    cswap(v[0], id[0], v[3], id[3]); cswap(v[0], id[0], v[2], id[2]);
    cswap(v[1], id[1], v[4], id[4]); cswap(v[1], id[1], v[3], id[3]);
    cswap(v[1], id[1], v[2], id[2]);
    for (int i = 0; i <= kMHeavy; ++i) {
      uint64_t mn = v[0];
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        const uint64_t ov = __shfl_xor_sync(0xffffffffu, mn, o);
        mn = ov < mn ? ov : mn;
      }
      const int src = __ffs(__ballot_sync(0xffffffffu, v[0] == mn)) - 1;
      const int ej = __shfl_sync(0xffffffffu, id[0], src);
      if (i < kMHeavy) {
        if (lane == src) {
#pragma unroll
          for (int j = 0; j < 4; ++j) { v[j] = v[j + 1]; id[j] = id[j + 1]; }
          v[4] = kNone;
        }
        if (lane == 0) {
          const bool real = mn != kNone;
          sHe[i * kMC + c] = real ? (uint8_t)ej : (uint8_t)0;
          sHw[i * kMC + c] = real ? __longlong_as_double((long long)mn) : inf;
        }
      } else if (lane == 0) {
        sWb[c] = mn != kNone ? __longlong_as_double((long long)mn) : inf;
      }
    }
  }
  __syncthreads();
  int he[kMHeavy];
  double hw[kMHeavy];
#pragma unroll
  for (int i = 0; i < kMHeavy; ++i) {
    he[i] = sHe[i * kMC + lane];
    hw[i] = sHw[i * kMC + lane];
  }
  const double wb = sWb[lane];
  const bool empty = lane >= nc || !(hw[0] < inf);
  const double2 *ord = reinterpret_cast<const double2 *>(a.order);
  const double2 *ut = reinterpret_cast<const double2 *>(a.UT);
  const int half = E >> 1;
  const int staged = E < kMRec ? E : kMRec;            // both even
  // this CTA's registers (gridDim.y ranges of whole 16-column groups)
  const int groups = mpad >> 4;
  const int r_lo = 16 * (int)((int64_t)blockIdx.y * groups / gridDim.y);
  const int r_hi = 16 * (int)((int64_t)(blockIdx.y + 1) * groups / gridDim.y);
  for (int rb = r_lo; rb < r_hi; rb += kMChunk) {
    const int rn = min(min(m, r_hi) - rb, kMChunk);
    MinStage st;
    if (warp < rn) min_fetch(st, ord, ut, rb + warp, E, lane);
    for (int rl = warp; rl < rn; rl += kMWarps) {
      const int r = rb + rl;
      myRec[lane] = st.rec;
#pragma unroll
      for (int q = 0; q < kMUcPerLane; ++q) {
        const int ch = lane + 32 * q;
        if (ch < half) reinterpret_cast<double2 *>(myUc)[ch] = st.uc[q];
      }
      __syncwarp();
      if (rl + kMWarps < rn) min_fetch(st, ord, ut, r + kMWarps, E, lane);
      double best = inf;
      int win = -1;
      // an empty lane's products are all infinite and leave win at -1
#pragma unroll
      for (int i = 0; i < kMHeavy; ++i) lex_min(__dmul_rn(hw[i], myUc[he[i]]), he[i], best, win);
      // Two entries a vote.  A lane whose bound has passed keeps evaluating with
      // the others: its products are above its best and change nothing.
      bool done = empty;
      int k = 0;
      for (; k < staged; k += 2) {
        const double2 v0 = myRec[k], v1 = myRec[k + 1];
        done |= __dmul_rn(wb, v0.x) > best;
        if (__all_sync(0xffffffffu, done)) break;
        const int e0 = __double2loint(v0.y), e1 = __double2loint(v1.y);
        const double h0 = __dmul_rn(sW[e0 * kMRow + lane], v0.x);
        const double h1 = __dmul_rn(sW[e1 * kMRow + lane], v1.x);
        lex_min(h0, e0, best, win);
        lex_min(h1, e1, best, win);
      }
      if (k >= staged) {
        for (; k < E; ++k) {                             // past the staged entries
          const double2 v = __ldg(ord + (size_t)r * E + k);
          done |= __dmul_rn(wb, v.x) > best;
          if (__all_sync(0xffffffffu, done)) break;
          const int e = __double2loint(v.y);
          lex_min(__dmul_rn(sW[e * kMRow + lane], v.x), e, best, win);
        }
      }
      if (lane < nc) sWin[lane * kMWinStride + rl] = win < 0 ? (uint8_t)0xFF : (uint8_t)win;
      __syncwarp();
    }
    __syncthreads();
    // code words: columns [rb, rend) of the nc rows; padding columns A = 0, B = 0xFF
    const int rend = min(rb + kMChunk, r_hi);
    const int q4 = (rend - rb) >> 2;
    for (int i = threadIdx.x; i < nc * q4; i += kMThreads) {
      const int cc = i / q4, rl = (i - cc * q4) * 4, r4 = rb + rl;
      const uint32_t wins = *reinterpret_cast<const uint32_t *>(sWin + cc * kMWinStride + rl);
      uint32_t va = 0, vb = 0;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int rr = r4 + b;
        uint32_t code = 0;
        if (rr < m) {
          const uint32_t wi = (wins >> (8 * b)) & 0xFFu;
          uint32_t w32 = 0;
          if (wi != 0xFFu) {
            code = __ldg(a.codeA + (size_t)wi * m + rr);
            w32 = __ldg(a.W32 + (size_t)wi * m + rr);
          }
          if (a.winners32) a.winners32[(c0 + cc) * m + rr] = w32;
          if (a.win_elem) a.win_elem[(c0 + cc) * m + rr] = (uint8_t)wi;
        }
        va |= code << (8 * b);
        vb |= (code ? code : 0xFFu) << (8 * b);
      }
      *reinterpret_cast<uint32_t *>(a.codesA + (c0 + cc) * mpad + r4) = va;
      *reinterpret_cast<uint32_t *>(a.codesB + (c0 + cc) * mpad + r4) = vb;
    }
    __syncthreads();
  }
}

}  // namespace

void launch_pack(const char *ascii, int64_t nbases, uint32_t *packed, uint32_t *nmask,
                 cudaStream_t s) {
  launch_pack_range(ascii, nbases, 0, (nbases + 15) / 16, packed, nmask, s);
}

void launch_pack_range(const char *ascii, int64_t nbases, int64_t w_begin, int64_t w_end,
                       uint32_t *packed, uint32_t *nmask, cudaStream_t s) {
  const int64_t nwords = (nbases + 15) / 16;
  if (w_end > nwords) w_end = nwords;
  if (w_end <= w_begin) return;
  const int tb = 256;
  const int64_t pairs = (w_end - w_begin + 1) / 2;
  const int64_t grid = (pairs + tb - 1) / tb;
  k_pack<<<(unsigned)grid, tb, 0, s>>>((const uint4 *)ascii, nbases, nwords, w_begin, w_end,
                                      packed, nmask);
}

namespace {

// Column-side codes from row-side ones: B = A, with 0xFF where A is 0 (unset).
__global__ void k_codes_b(const uint4 *__restrict__ A, uint4 *__restrict__ B, int64_t n16) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n16) return;
  const uint4 a = A[i];
  uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    // 0x80 in each zero byte (the add cannot carry out of a byte)
    const uint32_t z = ~(((w[q] & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | w[q]) & 0x80808080u;
    w[q] |= (z >> 7) * 0xFFu;
  }
  B[i] = make_uint4(w[0], w[1], w[2], w[3]);
}

}  // namespace

void launch_codes_b(const uint8_t *codesA, uint8_t *codesB, int64_t bytes, cudaStream_t s) {
  const int64_t n16 = bytes / 16;
  if (n16 == 0) return;
  k_codes_b<<<(unsigned)((n16 + 255) / 256), 256, 0, s>>>((const uint4 *)codesA, (uint4 *)codesB,
                                                          n16);
}

namespace {
template <bool GC2, int W>
void launch_count_w(const SketchArgs &a, int64_t grid, cudaStream_t s) {
  const size_t smem = (size_t)(kCountWarps / W) * sizeof(CountGroup);
  if (a.k == 4) {
    smem_cap_max((const void *)k_count<GC2, W, true>);
    k_count<GC2, W, true><<<(unsigned)grid, kCountWarps * 32, smem, s>>>(a);
  } else {
    smem_cap_max((const void *)k_count<GC2, W, false>);
    k_count<GC2, W, false><<<(unsigned)grid, kCountWarps * 32, smem, s>>>(a);
  }
}
}  // namespace

// Contigs up to which a CTA shares each contig (W = 8).  With a warp per contig
// the longest contig (80 kb) alone takes about 80 us; sharing cuts that to an
// eighth but pays the per-contig fold and weights with CTA barriers.  Measured
// (kernel time, warp / CTA per contig): 97 contigs 81 / 17 us, 2,000 142 / 38,
// 8,000 178 / 98, 16,000 226 / 180, 50,000 450 / 523.
constexpr int64_t kCountShare = 20000;

void launch_count(const SketchArgs &a, cudaStream_t s) {
  if (a.n == 0) return;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const bool share = a.n <= kCountShare;
  // with the contig counter, as many warps as fit (five blocks per SM);
  // without it, about eight contigs per group to even out the contig lengths
  const int64_t blocks = share ? a.n : (a.n + kCountWarps - 1) / kCountWarps;
  const int64_t grid =
      std::max<int64_t>(1, std::min<int64_t>(blocks, (int64_t)sms * (a.work ? 5 : 4)));
  if (a.gc_norm == 2) {
    if (share) launch_count_w<true, kCountWarps>(a, grid, s);
    else launch_count_w<true, 1>(a, grid, s);
  } else {
    if (share) launch_count_w<false, kCountWarps>(a, grid, s);
    else launch_count_w<false, 1>(a, grid, s);
  }
}

void smem_cap_max(const void *func) {
  static std::mutex mu;
  static std::set<std::pair<int, const void *>> done;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  if (!done.insert({dev, func}).second) return;
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaFuncAttributes fa;
  if (cudaFuncGetAttributes(&fa, func) != cudaSuccess) return;   // the launch reports it
  cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       optin - (int)fa.sharedSizeBytes);
}

// Ranges the registers are split into, one per blockIdx.y.  A CTA costs its
// set-up (the heavy sets, about as long as three registers of a warp) plus
// kMWarps registers at a time; few contigs leave SMs idle without a split,
// many fill them alone.  The smallest cost over the waves of three CTAs per SM
// (97 contigs: 163 -> 24 us, 2,000: 170 -> 61 us; from 25,000 contigs on
// unsplit).
static int minreduce_split(int64_t gx, int mpad, int sms) {
  const int groups = mpad / 16;
  const int64_t slots = 3 * (int64_t)sms;
  int best = 1;
  int64_t best_cost = INT64_MAX;
  for (int y = 1; y <= groups; ++y) {
    const int64_t waves = (gx * y + slots - 1) / slots;
    const int64_t regs = 16 * ((groups + y - 1) / y);
    const int64_t cost = waves * (3 * kMWarps + regs);
    if (cost < best_cost) {
      best_cost = cost;
      best = y;
    }
  }
  return best;
}

void launch_minreduce(const SketchArgs &a, cudaStream_t s) {
  if (a.n == 0) return;
  const size_t smem = minreduce_smem(a.n_elems);
  smem_cap_max((const void *)k_minreduce);
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t gx = (a.n + kMC - 1) / kMC;
  const dim3 grid((unsigned)gx, (unsigned)minreduce_split(gx, a.mpad, sms));
  k_minreduce<<<grid, kMThreads, smem, s>>>(a);
}

namespace {

// ── One-permutation MinHash (the RABBIT_PMH=0 metric, src/rabbit_sketch.h) ──
// KmerSketch::update (src/rabbit_sketch.h:199-238): every window of K bases
// that are all A/C/G/T offers h = murmur3_fmix(min(forward, reverse
// complement), seed) to bucket ((h >> 32) * m) >> 32 with value (uint32_t)h,
// kept if smaller.  buildSig (:264-281) gives an empty bucket the value that
// densify (:245-259) borrows along its probe sequence, and keeps `bits` low
// bits of every bucket (bit-planes); a sketch with no k-mer at all has an
// all-zero signature.  Here a bucket's kept bits + 1 are its 8-bit code (A
// side; the B side is the same), so equal codes are exactly the buckets whose
// bit-planes all agree (jaccard_raw, src/rabbitbin.cpp:1035-1130).

__device__ __forceinline__ uint64_t oph_fmix(uint64_t x, uint64_t seed) {
  x ^= seed;
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdull;
  x ^= x >> 33;
  x *= 0xc4ceb9fe1a85ec53ull;
  x ^= x >> 33;
  return x;
}

__device__ __forceinline__ uint32_t oph_bucket(uint64_t h, uint32_t m) {
  return (uint32_t)(((h >> 32) * (uint64_t)m) >> 32);
}

// Reverse complement of a K-base word (2 bits a base, first base highest).
__device__ __forceinline__ uint64_t oph_revcomp(uint64_t x, int K) {
  x = __brevll(~x);                        // complement, then every bit reversed
  x = ((x >> 1) & 0x5555555555555555ull) | ((x & 0x5555555555555555ull) << 1);
  return x >> (64 - 2 * K);                // the base pairs back in order
}

constexpr int kOphWarps = 4;

// Warp per contig (warps stride over the contigs); the warp's m registers in
// shared memory; a lane takes one 16-base word per step and the windows that
// end in it.
__global__ void __launch_bounds__(kOphWarps * 32)
k_oph(SketchArgs a, int K, int bits, uint64_t seed) {
  extern __shared__ uint32_t sh_oph[];
  constexpr uint32_t kEmpty = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t m = (uint32_t)a.m;
  uint32_t *reg = sh_oph + (size_t)wib * m;
  const uint64_t kmask = K >= 32 ? ~0ull : ((1ull << (2 * K)) - 1ull);
  const uint32_t vmask = (1u << bits) - 1u;
  const int64_t warps = (int64_t)gridDim.x * kOphWarps;
  for (int64_t c = (int64_t)blockIdx.x * kOphWarps + wib; c < a.n; c += warps) {
    for (uint32_t r = lane; r < m; r += 32) reg[r] = kEmpty;
    __syncwarp();
    const int64_t s = a.offsets[c], e = a.offsets[c + 1];
    if (e - s >= K) {
      const int64_t w0 = s >> 4, w1 = (e + 15) >> 4;
      uint32_t c1 = 0, c2 = 0, b1 = 0xFFFFu, b2 = 0xFFFFu;   // the two words before w0
      for (int64_t base = w0; base < w1; base += 32) {
        const int64_t wi = base + lane;
        uint32_t cur = 0, bad = 0xFFFFu;
        if (wi < w1) {
          cur = __ldg(a.packed + wi);
          bad = invalid16(a.nmask, wi, s, e);
        }
        uint32_t p1 = __shfl_up_sync(0xffffffffu, cur, 1), q1 = __shfl_up_sync(0xffffffffu, bad, 1);
        uint32_t p2 = __shfl_up_sync(0xffffffffu, cur, 2), q2 = __shfl_up_sync(0xffffffffu, bad, 2);
        if (lane == 0) { p1 = c1; q1 = b1; p2 = c2; q2 = b2; }
        if (lane == 1) { p2 = c1; q2 = b1; }
        c2 = __shfl_sync(0xffffffffu, cur, 30);
        b2 = __shfl_sync(0xffffffffu, bad, 30);
        c1 = __shfl_sync(0xffffffffu, cur, 31);
        b1 = __shfl_sync(0xffffffffu, bad, 31);
        if (wi >= w1) continue;
        // bit 15 - p: base p of the word (p < 0: the words before); a window
        // ending at base t is valid when bits 15-t .. 15-t+K-1 are all clear
        const uint64_t wbad = ((uint64_t)q2 << 32) | ((uint64_t)q1 << 16) | bad;
        uint64_t any = wbad;
        for (int q = 1; q < K; ++q) any |= wbad >> q;
        uint32_t kv = ~(uint32_t)any & 0xFFFFu;
        const uint64_t lo = ((uint64_t)p1 << 32) | cur;
        while (kv) {
          const int bp = __ffs(kv) - 1;                // = 15 - t
          kv &= kv - 1;
          const int sh = 2 * bp;
          const uint64_t fwd = (sh ? (lo >> sh) | ((uint64_t)p2 << (64 - sh)) : lo) & kmask;
          const uint64_t rc = oph_revcomp(fwd, K);
          const uint64_t h = oph_fmix(fwd < rc ? fwd : rc, seed);
          atomicMin(&reg[oph_bucket(h, m)], (uint32_t)h);
        }
      }
    }
    __syncwarp();
    if (a.oph_keys) {
      // KmerSketch::getKeys (src/rabbit_sketch.h:166-175): one key per
      // non-empty bucket, murmur3_fmix((bucket << 32) | register, seed ^
      // 0x51A3C2B7); 0 marks an empty bucket here (no key)
      for (uint32_t r = lane; r < m; r += 32) {
        const uint32_t v = reg[r];
        a.oph_keys[c * m + r] =
            v == kEmpty ? 0ull : oph_fmix(((uint64_t)r << 32) | v, seed ^ 0x51A3C2B7ull);
      }
      __syncwarp();
      continue;
    }
    uint32_t ne = 0;
    for (uint32_t r = lane; r < m; r += 32) ne += reg[r] != kEmpty;
    ne = __reduce_add_sync(0xffffffffu, ne);
    uint8_t *ca = a.codesA + c * a.mpad, *cb = a.codesB + c * a.mpad;
    for (uint32_t r = lane; r < (uint32_t)a.mpad; r += 32) {
      if (r >= m) {                                    // padding never matches
        ca[r] = 0;
        cb[r] = 0xFF;
        continue;
      }
      uint32_t v = reg[r];
      if (ne == 0) {
        v = 0;
      } else if (v == kEmpty) {
        // densify: the shared probe sequence of bucket r
        const uint64_t pb = oph_fmix((uint64_t)r, seed ^ 0xA5A5A5A5DEADBEEFull);
        const uint64_t step = oph_fmix((uint64_t)r, seed ^ 0x123456789ABCDEF0ull) | 1ull;
        uint64_t cur = pb;
        v = 0;
        for (uint32_t t = 1; t <= m; ++t) {
          cur += step;
          const uint32_t x = reg[oph_bucket(cur, m)];
          if (x != kEmpty) {
            v = x ^ (uint32_t)oph_fmix((uint64_t)t, 0x9E3779B97F4A7C15ull);
            break;
          }
        }
      }
      const uint8_t code = (uint8_t)((v & vmask) + 1u);
      ca[r] = code;
      cb[r] = code;
    }
    __syncwarp();
  }
}

}  // namespace

namespace {
// Bucket values (code - 1) of n code rows, m per row, packed.
__global__ void k_oph_values(const uint8_t *__restrict__ codes, int64_t n, int m, int mpad,
                             uint8_t *__restrict__ out) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * m) return;
  const int64_t i = t / m, r = t - i * m;
  out[t] = (uint8_t)(codes[i * mpad + r] - 1u);
}
}  // namespace

void launch_oph_values(const uint8_t *codes, int64_t n, int m, int mpad, uint8_t *out,
                       cudaStream_t s) {
  if (n <= 0) return;
  const int64_t tot = n * m;
  k_oph_values<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(codes, n, m, mpad, out);
}

void launch_oph(const SketchArgs &a, int K, int bits, uint64_t seed, cudaStream_t s) {
  if (a.n == 0) return;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t smem = (size_t)kOphWarps * a.m * sizeof(uint32_t);
  smem_cap_max((const void *)k_oph);
  const int64_t blocks = (a.n + kOphWarps - 1) / kOphWarps;
  const int64_t grid = std::max<int64_t>(1, std::min<int64_t>(blocks, (int64_t)sms * 8));
  k_oph<<<(unsigned)grid, kOphWarps * 32, smem, s>>>(a, K, bits, seed);
}

}  // namespace rbg
