// DEFLATE decoder (RFC 1951) for one BGZF block, host and device.
//
// A BGZF member holds at most 64 KiB of output, and its deflate stream refers
// only to bytes of the same member, so every block decodes on its own: the
// device runs one warp per block.  All lanes of the warp decode the same
// symbols in lockstep (same bits, same tables: no divergence, broadcast loads);
// the lanes store literals and copy matches and stored blocks together (a match
// that overlaps itself repeats its first `distance` bytes, all of them written
// before it).  The code is written against a Lanes type: one lane on the host
// (SerialLanes), the warp on the device (WarpLanes), and in the tests 32 lanes that
// take turns on the host, which run the warp's branches (Lanes::kWarp) on plain
// memory.  Symbols are decoded with a 10-bit (literal /
// length) and 8-bit (distance) lookup table of 32-bit entries that carry each
// symbol's meaning (one or two literal bytes, length or distance base, extra
// bits), with a search over the code lengths for longer codes.  Every read stays inside [in, in + inlen),
// every write inside [out, out + outlen), and every match must point into
// bytes already written: a stream that breaks a rule ends with a status, never
// with an access out of bounds.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define RBG_IHD __host__ __device__ __forceinline__
#else
#define RBG_IHD inline
#endif

namespace rbg {
namespace inflate {

enum Status : int32_t {
  kOk = 0,
  kErrInput = 1,        // the stream ends early
  kErrBlockType = 2,    // reserved block type 3
  kErrStored = 3,       // stored block length and its complement disagree
  kErrCodes = 4,        // over-subscribed or empty code lengths, bad repeat
  kErrSymbol = 5,       // a code that is not in the table, or symbol 286/287, 30/31
  kErrDistance = 6,     // a match reaching before the start of the output
  kErrOutput = 7,       // more output than the block's ISIZE
  kErrShort = 8         // less output than the block's ISIZE
};

constexpr int kLitBits = 10, kDistBits = 8;

// The lanes that decode one block: one host thread, or one device warp.  A warp's
// match(v) is the set of lanes with the same v, from(v, i) lane i's v.
struct SerialLanes {
  static constexpr bool kWarp = false;
  RBG_IHD int lane() const { return 0; }
  RBG_IHD int width() const { return 1; }
  RBG_IHD bool leader() const { return true; }
  RBG_IHD void sync() const {}
  RBG_IHD uint32_t match(int) const { return 1; }
  RBG_IHD uint32_t from(uint32_t v, int) const { return v; }
};
#ifdef __CUDACC__
struct WarpLanes {
  static constexpr bool kWarp = true;
  int l;
  __device__ __forceinline__ int lane() const { return l; }
  __device__ __forceinline__ int width() const { return 32; }
  __device__ __forceinline__ bool leader() const { return l == 0; }
  __device__ __forceinline__ void sync() const { __syncwarp(); }
  __device__ __forceinline__ uint32_t match(int v) const { return __match_any_sync(0xffffffffu, v); }
  __device__ __forceinline__ uint32_t from(uint32_t v, int i) const {
    return __shfl_sync(0xffffffffu, v, i);
  }
};
#endif

RBG_IHD int bits_set(uint32_t v) {
#ifdef __CUDA_ARCH__
  return __popc(v);
#else
  return __builtin_popcount(v);
#endif
}
RBG_IHD uint64_t load8(const uint64_t *p) {
#ifdef __CUDA_ARCH__
  return __ldg(p);
#else
  return *p;
#endif
}

// One Huffman code: lookup table for codes up to kBits bits and the canonical
// tables for the rest.  A table entry carries what the symbol means, so the
// decode loop needs no per-symbol arithmetic:
//   bits 0-3   code length (0: longer code, or no code)
//   bits 4-5   kind: 0 literal / distance / code-length symbol, 1 length,
//              2 end of block, 3 invalid symbol
//   bits 6-9   extra bits that follow the code; 1 for a literal: two of them
//   bits 16-31 value: the literal byte (then the second one's), the length or
//              distance base, or the code-length symbol
template <int kBits, int kSyms>
struct Code {
  uint32_t lut[1 << kBits];
  uint16_t count[16];
  uint16_t sym[kSyms];
};
constexpr uint32_t kEndOfInput = 0xFFFFFFFFu, kNoCode = 0xFFFFFFFEu;

struct Tables {
  Code<kLitBits, 288> lit;
  Code<kDistBits, 32> dist;
  uint16_t next[16], offs[16];   // while a code is built
  uint8_t lens[320];          // code lengths being read (litlen then distance)
  uint8_t clens[20];          // code-length code lengths
};

template <bool kWarp>
struct Bits {
  const uint8_t *p;
  uint32_t n, pos;
  uint64_t buf;
  int cnt;
  RBG_IHD void refill() {
    if constexpr (kWarp) {
      // two aligned 8-byte loads and a funnel shift; the device buffers hold the
      // input from a 256-byte aligned start with 16 bytes of slack after its end,
      // and bytes past the stream's end are masked off
      if (pos >= n || cnt > 56) return;
      const uintptr_t a = (uintptr_t)(p + pos);
      const uint64_t *q = (const uint64_t *)(a & ~(uintptr_t)7);
      const uint32_t sh = (uint32_t)(a & 7) * 8;
      uint64_t w = load8(q) >> sh;
      if (sh) w |= load8(q + 1) << (64 - sh);
      uint32_t take = (uint32_t)(63 - cnt) >> 3;
      if (take > n - pos) take = n - pos;
      w &= take >= 8 ? ~0ull : ((1ull << (8 * take)) - 1);
      buf |= w << cnt;
      pos += take;
      cnt += 8 * (int)take;
    } else {
      while (cnt <= 56 && pos < n) {
        buf |= (uint64_t)p[pos++] << cnt;
        cnt += 8;
      }
    }
  }
  RBG_IHD bool need(int k) {
    if (cnt < k) refill();
    return cnt >= k;
  }
  RBG_IHD uint32_t peek(int k) const { return (uint32_t)(buf & ((1ull << k) - 1)); }
  RBG_IHD void drop(int k) {
    buf >>= k;
    cnt -= k;
  }
  RBG_IHD bool get(int k, uint32_t &v) {
    if (!need(k)) return false;
    v = peek(k);
    drop(k);
    return true;
  }
};

RBG_IHD uint32_t reverse_bits(uint32_t v, int n) {
#ifdef __CUDA_ARCH__
  return __brev(v) >> (32 - n);        // n >= 1
#else
  uint32_t r = 0;
  for (int i = 0; i < n; ++i) {
    r = (r << 1) | (v & 1);
    v >>= 1;
  }
  return r;
#endif
}

// Length symbols 257 + i: i < 8 give 3 + i with no extra bits; then groups of
// four with e = (i - 4) / 4 extra bits starting at ((4 + (i & 3)) << e) + 3;
// i = 28 (symbol 285) is 258.  Distance symbols d < 4 give d + 1; then pairs
// with e = (d - 2) / 2 extra bits starting at ((2 + (d & 1)) << e) + 1.
RBG_IHD int len_extra(int i) { return (i < 8 || i == 28) ? 0 : (i - 4) / 4; }
RBG_IHD uint32_t len_base(int i) {
  return i < 8 ? 3u + i : (i == 28 ? 258u : ((4u + (i & 3)) << len_extra(i)) + 3u);
}
RBG_IHD int dist_extra(int d) { return d < 4 ? 0 : (d - 2) / 2; }
RBG_IHD uint32_t dist_base(int d) { return d < 4 ? 1u + d : ((2u + (d & 1)) << dist_extra(d)) + 1u; }


// Table entries of the three codes.
struct LitEntry {
  static constexpr bool kPairs = true;
  RBG_IHD static uint32_t make(int s, int l) {
    if (s < 256) return (uint32_t)s << 16 | (uint32_t)l;
    if (s == 256) return 2u << 4 | (uint32_t)l;
    const int i = s - 257;
    if (i >= 29) return 3u << 4 | (uint32_t)l;
    return len_base(i) << 16 | (uint32_t)len_extra(i) << 6 | 1u << 4 | (uint32_t)l;
  }
};
struct DistEntry {
  static constexpr bool kPairs = false;
  RBG_IHD static uint32_t make(int s, int l) {
    if (s >= 30) return 3u << 4 | (uint32_t)l;
    return dist_base(s) << 16 | (uint32_t)dist_extra(s) << 6 | (uint32_t)l;
  }
};
struct PlainEntry {
  static constexpr bool kPairs = false;
  RBG_IHD static uint32_t make(int s, int l) { return (uint32_t)s << 16 | (uint32_t)l; }
};

// Table entry of two literals in a row, when e1 at index idx is a literal and the
// bits after it hold another whole one; 0 otherwise.
template <int kBits>
RBG_IHD uint32_t literal_pair(uint32_t e1, uint32_t e2) {
  const uint32_t l1 = e1 & 0x3F, l2 = e2 & 0x3F;       // length and kind: 1..15 for a literal
  if (l1 - 1u >= 15u || l2 - 1u >= 15u || l1 + l2 > (uint32_t)kBits) return 0;
  return (e2 >> 16) << 24 | (e1 >> 16) << 16 | 1u << 6 | (l1 + l2);
}

// Builds a code from `n` code lengths.  Incomplete codes are accepted (a code
// of one distance symbol is legal); over-subscribed ones are not.  The lanes take
// 32 symbols at a time: a symbol's canonical code follows from the symbols of its
// length before it (the lanes below with the same length).
template <class Entry, int kBits, int kSyms, class Lanes>
RBG_IHD int build(Code<kBits, kSyms> &c, Tables &T, const uint8_t *len, int n, const Lanes &L) {
  const int lane = L.lane(), W = L.width();
  L.sync();
  for (int i = lane; i < 16; i += W) c.count[i] = 0;
  for (int i = lane; i < (1 << kBits); i += W) c.lut[i] = 0;
  L.sync();
  for (int s0 = 0; s0 < n; s0 += W) {
    const int l = s0 + lane < n ? len[s0 + lane] : 0;
    const uint32_t same = L.match(l);
    if (l && (same & ((1u << lane) - 1u)) == 0)          // the lowest lane of the length
      c.count[l] = (uint16_t)(c.count[l] + bits_set(same));
    L.sync();
  }
  // a code of l bits takes 2^(15 - l) of the 2^15 values of 15 bits
  uint32_t taken = 0;
  for (int l = 1; l < 16; ++l) taken += (uint32_t)c.count[l] << (15 - l);
  if (taken > 1u << 15) return kErrCodes;
  // canonical codes in symbol order
  if (L.leader()) {
    uint32_t code = 0, at = 0;
    for (int l = 1; l < 16; ++l) {
      code = (code + c.count[l - 1]) << 1;             // count[0] is 0
      T.next[l] = (uint16_t)code;
      T.offs[l] = (uint16_t)at;
      at += c.count[l];
    }
  }
  L.sync();
  for (int s0 = 0; s0 < n; s0 += W) {
    const int s = s0 + lane;
    const int l = s < n ? len[s] : 0;
    uint32_t cd = 0, at = 0;
    const uint32_t same = L.match(l);
    const uint32_t rank = (uint32_t)bits_set(same & ((1u << lane) - 1u));
    if (l) {
      cd = T.next[l] + rank;
      at = T.offs[l] + rank;
    }
    L.sync();
    if (l && rank == 0) {
      T.next[l] = (uint16_t)(T.next[l] + bits_set(same));
      T.offs[l] = (uint16_t)(T.offs[l] + bits_set(same));
    }
    if (l) {
      c.sym[at] = (uint16_t)s;
      if (l <= kBits) {                                // entered bit-reversed into the table
        const uint32_t r = reverse_bits(cd, l), e = Entry::make(s, l);
        for (uint32_t f = r; f < (1u << kBits); f += (1u << l)) c.lut[f] = e;
      }
    }
    L.sync();
  }
  if (Entry::kPairs) {
    // from the last entry down: the bits after a literal index an entry at half
    // the index or below, which still holds its single symbol
    for (int i0 = (1 << kBits) - W; i0 >= 0; i0 -= W) {
      const uint32_t e1 = c.lut[i0 + lane];
      const uint32_t e = literal_pair<kBits>(e1, c.lut[(uint32_t)(i0 + lane) >> (e1 & 15)]);
      L.sync();
      if (e) c.lut[i0 + lane] = e;
      L.sync();
    }
  }
  return kOk;
}

// Decodes one symbol and returns its table entry; kEndOfInput when the stream
// ends, kNoCode for a code that is not in the table.
template <class Entry, int kBits, int kSyms, bool kWarp>
RBG_IHD uint32_t decode(const Code<kBits, kSyms> &c, Bits<kWarp> &b) {
  if (b.cnt < 15) b.refill();
  // bits above cnt are zero, so the table index is defined near the end too;
  // an entry counts only when its whole code is in the buffer
  const uint32_t e = c.lut[b.peek(kBits)];
  if (e && (int)(e & 15) <= b.cnt) {
    b.drop(e & 15);
    return e;
  }
  // Codes longer than the table.  Read as 15-bit numbers, first bit highest, the
  // canonical codes of each length fill the range that follows the shorter ones', a
  // code of l bits 2^(15 - l) numbers of it: the next 15 bits (zeros past the end of
  // the stream) lie in the range of their length.
  uint32_t at = reverse_bits(b.peek(15), 15), sym = 0;   // place past the shorter lengths' ranges
  for (int l = 1; l < 16; ++l) {
    const uint32_t cnt = c.count[l];
    if (at < cnt << (15 - l)) {
      if (l > b.cnt) return kEndOfInput;
      b.drop(l);
      return Entry::make(c.sym[sym + (at >> (15 - l))], l);
    }
    at -= cnt << (15 - l);
    sym += cnt;
  }
  return b.cnt < 15 ? kEndOfInput : kNoCode;
}

// Inflates one raw deflate stream into out[0, outlen).  Returns kOk when the
// final block ends with exactly outlen bytes written.
template <class Lanes>
RBG_IHD int inflate_block(const uint8_t *in, uint32_t inlen, uint8_t *out, uint32_t outlen,
                          Tables &T, const Lanes &L) {
  const int lane = L.lane(), W = L.width();
  constexpr bool kWarp = Lanes::kWarp;
  Bits<kWarp> b{in, inlen, 0, 0, 0};
  uint32_t o = 0;
  uint32_t held = 0, held_at = 0;      // (warp) a copy read but not stored: lane k's byte of `held`
  uint8_t held_v = 0;
  for (;;) {
    uint32_t hdr;
    if (!b.get(3, hdr)) return kErrInput;
    const uint32_t final = hdr & 1, type = hdr >> 1;
    if (type == 0) {
      // stored: skip to a byte boundary, LEN, NLEN, bytes
      b.drop(b.cnt & 7);
      uint32_t len, nlen;
      if (!b.get(16, len) || !b.get(16, nlen)) return kErrInput;
      if ((len ^ 0xffffu) != nlen) return kErrStored;
      // bytes still held in the bit buffer come first
      while (len && b.cnt >= 8) {
        if (o >= outlen) return kErrOutput;
        if (L.leader()) out[o] = (uint8_t)b.peek(8);
        ++o;
        b.drop(8);
        --len;
      }
      if (len > b.n - b.pos) return kErrInput;
      if (len > outlen - o) return kErrOutput;
      for (uint32_t i = lane; i < len; i += W) out[o + i] = b.p[b.pos + i];
      o += len;
      b.pos += len;
    } else if (type == 1 || type == 2) {
      // no lane may still read the previous block's tables
      L.sync();
      int nlen = 288, ndist = 30;
      if (type == 1) {
        for (int s = 0; s < 144; ++s) T.lens[s] = 8;
        for (int s = 144; s < 256; ++s) T.lens[s] = 9;
        for (int s = 256; s < 280; ++s) T.lens[s] = 7;
        for (int s = 280; s < 288; ++s) T.lens[s] = 8;
        for (int s = 0; s < 30; ++s) T.lens[288 + s] = 5;
      } else {
        uint32_t hlit, hdist, hclen;
        if (!b.get(5, hlit) || !b.get(5, hdist) || !b.get(4, hclen)) return kErrInput;
        nlen = (int)hlit + 257;
        ndist = (int)hdist + 1;
        if (nlen > 286 || ndist > 30) return kErrCodes;
        // code-length code: lengths in the fixed permuted order
        const uint8_t ord[19] = {16, 17, 18, 0, 8, 7, 9, 6, 10, 5, 11, 4, 12, 3, 13, 2, 14, 1, 15};
        uint8_t *cl = T.clens;                         // the lanes write the same values
        for (int i = 0; i < 19; ++i) cl[i] = 0;
        for (uint32_t i = 0; i < hclen + 4; ++i) {
          uint32_t v;
          if (!b.get(3, v)) return kErrInput;
          cl[ord[i]] = (uint8_t)v;
        }
        // the code-length code decodes through the distance table's storage
        // (it has 19 symbols and codes of at most 7 bits)
        Code<kDistBits, 32> &cc = T.dist;
        if (build<PlainEntry>(cc, T, T.clens, 19, L) != kOk) return kErrCodes;
        int i = 0;
        while (i < nlen + ndist) {
          const uint32_t ce = decode<PlainEntry>(cc, b);
          if (ce >= kNoCode) return ce == kEndOfInput ? kErrInput : kErrSymbol;
          const int sym = (int)(ce >> 16);
          if (sym < 16) {
            T.lens[i < nlen ? i : 288 + (i - nlen)] = (uint8_t)sym;
            ++i;
            continue;
          }
          uint32_t rep;
          uint8_t val = 0;
          if (sym == 16) {
            if (i == 0) return kErrCodes;
            const int prev = i - 1;
            val = T.lens[prev < nlen ? prev : 288 + (prev - nlen)];
            if (!b.get(2, rep)) return kErrInput;
            rep += 3;
          } else if (sym == 17) {
            if (!b.get(3, rep)) return kErrInput;
            rep += 3;
          } else {
            if (!b.get(7, rep)) return kErrInput;
            rep += 11;
          }
          if ((int)(i + rep) > nlen + ndist) return kErrCodes;
          for (uint32_t r = 0; r < rep; ++r, ++i) T.lens[i < nlen ? i : 288 + (i - nlen)] = val;
        }
        if (T.lens[256] == 0) return kErrCodes;       // no end-of-block code
      }
      L.sync();
      if (build<LitEntry>(T.lit, T, T.lens, nlen, L) != kOk) return kErrCodes;
      if (build<DistEntry>(T.dist, T, T.lens + 288, ndist, L) != kOk) return kErrCodes;
      L.sync();
      for (;;) {
        // one or two literals from the table, the common case
        if (b.cnt < 15) b.refill();
        const uint32_t q = T.lit.lut[b.peek(kLitBits)];
        if ((q & 0x3F) - 1u < 15u && (int)(q & 15) <= b.cnt) {
          const uint32_t two = (q >> 6) & 1;
          b.drop(q & 15);
          if (o + two >= outlen) return kErrOutput;
          if constexpr (kWarp) {
            if ((uint32_t)lane <= two) out[o + lane] = (uint8_t)(q >> (16 + 8 * lane));
          } else {
            out[o] = (uint8_t)(q >> 16);
            if (two) out[o + 1] = (uint8_t)(q >> 24);
          }
          o += 1 + two;
          continue;
        }
        const uint32_t e = decode<LitEntry>(T.lit, b);
        if (e >= kNoCode) return e == kEndOfInput ? kErrInput : kErrSymbol;
        const uint32_t kind = (e >> 4) & 3;
        if (kind == 0) {
          if (o >= outlen) return kErrOutput;
          if (L.leader()) out[o] = (uint8_t)(e >> 16);
          ++o;
          continue;
        }
        if (kind == 2) {
          if (kWarp && (uint32_t)lane < held) out[held_at + lane] = held_v;
          held = 0;
          break;
        }
        if (kind == 3) return kErrSymbol;
        uint32_t len = e >> 16, ex;
        const int le = (int)((e >> 6) & 15);
        if (le) {
          if (!b.get(le, ex)) return kErrInput;
          len += ex;
        }
        const uint32_t d = decode<DistEntry>(T.dist, b);
        if (d >= kNoCode) return d == kEndOfInput ? kErrInput : kErrSymbol;
        if (((d >> 4) & 3) == 3) return kErrSymbol;
        uint32_t dist = d >> 16;
        const int de = (int)((d >> 6) & 15);
        if (de) {
          if (!b.get(de, ex)) return kErrInput;
          dist += ex;
        }
        if (dist > o) return kErrDistance;
        if (len > outlen - o) return kErrOutput;
        // the bytes read are all written before the match: a match longer than its
        // distance repeats the first `dist` of them
        const uint8_t *src = out + (o - dist);
        uint8_t *dst = out + o;
        if constexpr (kWarp) {
          // The copy of up to 32 bytes is stored at the next one: the loads' latency
          // passes under the symbols decoded in between.
          if ((uint32_t)lane < held) out[held_at + lane] = held_v;
          held = 0;
          L.sync();
          if (len <= 32) {
            if ((uint32_t)lane < len) held_v = src[dist >= len ? lane : lane % dist];
            held = len;
            held_at = o;
          } else if (dist >= len) {
            for (uint32_t k = lane; k < len; k += W) dst[k] = src[k];
          } else {
            for (uint32_t k = lane; k < len; k += W) dst[k] = src[k % dist];
          }
        } else {
          for (uint32_t k = 0; k < len; ++k) dst[k] = src[dist >= len ? k : k % dist];
        }
        o += len;
      }
    } else {
      return kErrBlockType;
    }
    if (final) break;
  }
  return o == outlen ? kOk : kErrShort;
}

// CRC-32 (IEEE 802.3, reflected polynomial 0xEDB88320) with a 256-entry table.
// The lanes each take one segment of the block and run the table CRC from 0;
// the segments are joined with the CRC's linearity: crc(A || B) = crc(A) * x^(8|B|)
// + crc(B) over GF(2) modulo the polynomial, and the standard pre- and post-
// inversion is applied to the whole: crc = raw(data) + 0xffffffff * x^(8n) +
// 0xffffffff.  In the reflected representation bit 31 holds x^0.
constexpr uint32_t kCrcPoly = 0xEDB88320u;

RBG_IHD void crc32_table(uint32_t *t) {
  for (uint32_t i = 0; i < 256; ++i) {
    uint32_t c = i;
    for (int k = 0; k < 8; ++k) c = (c & 1) ? kCrcPoly ^ (c >> 1) : c >> 1;
    t[i] = c;
  }
}
RBG_IHD uint32_t crc_raw(const uint32_t *t, uint32_t c, const uint8_t *p, uint32_t n) {
  for (uint32_t i = 0; i < n; ++i) c = t[(c ^ p[i]) & 0xff] ^ (c >> 8);
  return c;
}
// a * b modulo the polynomial (shift-and-add; b is multiplied by x each step)
RBG_IHD uint32_t gf2_mul(uint32_t a, uint32_t b) {
  uint32_t r = 0;
  for (uint32_t m = 1u << 31; m; m >>= 1) {
    if (a & m) r ^= b;
    b = (b & 1) ? (b >> 1) ^ kCrcPoly : b >> 1;
  }
  return r;
}
// x^(8 n) modulo the polynomial, by squaring
RBG_IHD uint32_t x_pow8(uint32_t n) {
  uint32_t r = 1u << 31, sq = 1u << (31 - 8);      // x^0, x^8
  while (n) {
    if (n & 1) r = gf2_mul(r, sq);
    sq = gf2_mul(sq, sq);
    n >>= 1;
  }
  return r;
}
template <class Lanes>
RBG_IHD uint32_t crc32(const uint32_t *t, const uint8_t *p, uint32_t n, const Lanes &L) {
  const uint32_t W = (uint32_t)L.width();
  const uint32_t seg = (n + W - 1) / W;
  uint32_t acc = 0;
  if constexpr (Lanes::kWarp) {
    const uint32_t a = (uint32_t)L.lane() * seg;
    const uint32_t e = a + seg < n ? a + seg : n;
    const uint32_t c = a < n ? crc_raw(t, 0u, p + a, e - a) : 0u;
    const uint32_t xs = x_pow8(seg);
    // Horner over the lanes: acc = acc * x^(8 len_i) + c_i
    for (uint32_t i = 0; i < W; ++i) {
      const uint32_t ci = L.from(c, (int)i);
      const uint32_t ai = i * seg;
      const uint32_t li = ai >= n ? 0u : (ai + seg < n ? seg : n - ai);
      if (li == seg) acc = gf2_mul(acc, xs) ^ ci;
      else if (li) acc = gf2_mul(acc, x_pow8(li)) ^ ci;
    }
  } else {
    // one lane: the same joining, over W = 32 virtual segments
    const uint32_t vs = (n + 31) / 32;
    const uint32_t xs = x_pow8(vs);
    for (uint32_t a = 0; a < n; a += vs) {
      const uint32_t li = a + vs < n ? vs : n - a;
      const uint32_t ci = crc_raw(t, 0u, p + a, li);
      acc = gf2_mul(acc, li == vs ? xs : x_pow8(li)) ^ ci;
    }
  }
  return acc ^ gf2_mul(0xffffffffu, x_pow8(n)) ^ 0xffffffffu;
}

}  // namespace inflate
}  // namespace rbg
