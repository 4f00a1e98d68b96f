// Test harness: the warp's branches of the DEFLATE decoder and CRC
// (rabbitbin_b200/csrc/inflate.cuh) on 32 lanes that take turns on the host, over a
// file of streams (records of u32 input length, u32 output length, input bytes),
// against the one-lane decoder.  A lane runs until its next sync; a round lets every
// lane run once, upwards, downwards or from the middle, so that a value read or
// written without a sync between the lanes shows as a difference.  Built with
// AddressSanitizer by tests/test_inflate_lanes_cpu.py.  Not part of the library.
#include <ucontext.h>

#include <cstdint>
#include <cstdio>
#include <cstring>
#include <memory>
#include <vector>

#include "../../rabbitbin_b200/csrc/inflate.cuh"

#ifdef __SANITIZE_ADDRESS__
#include <sanitizer/common_interface_defs.h>
#endif

namespace {

using namespace rbg::inflate;
constexpr int kLanes = 32;
constexpr size_t kStack = 256 << 10;

struct Warp;
void run_lane(unsigned lo, unsigned hi);

struct Warp {
  ucontext_t main, lane[kLanes];
  std::vector<std::unique_ptr<char[]>> stack;
  bool done[kLanes];
  bool diverged = false;
  uint32_t slot[kLanes];
  int cur = 0;
  void *fake = nullptr;
  const void *main_stack = nullptr;
  size_t main_size = 0;
  void (*body)(Warp &, int) = nullptr;
  // the block at hand
  const uint8_t *in;
  uint32_t inlen, outlen;
  uint8_t *out;
  Tables *tabs;
  const uint32_t *crc_t;
  int st[kLanes];
  uint32_t crc[kLanes];

  Warp() {
    for (int l = 0; l < kLanes; ++l) stack.emplace_back(new char[kStack]);
  }
  // Back to the scheduler; returns when the lane's next turn comes.
  void yield(int l, bool last = false) {
    (void)last;
#ifdef __SANITIZE_ADDRESS__
    void *f = nullptr;
    __sanitizer_start_switch_fiber(last ? nullptr : &f, main_stack, main_size);
    swapcontext(&lane[l], &main);
    __sanitizer_finish_switch_fiber(f, &main_stack, &main_size);
#else
    swapcontext(&lane[l], &main);
#endif
  }
  void enter(int l) {
#ifdef __SANITIZE_ADDRESS__
    __sanitizer_start_switch_fiber(&fake, stack[l].get(), kStack);
    swapcontext(&main, &lane[l]);
    __sanitizer_finish_switch_fiber(fake, nullptr, nullptr);
#else
    swapcontext(&main, &lane[l]);
#endif
  }
  // Runs body on every lane; order 0 upwards, 1 downwards, 2 from lane 13 on.
  void run(void (*b)(Warp &, int), int order) {
    body = b;
    diverged = false;
    for (int l = 0; l < kLanes; ++l) {
      done[l] = false;
      getcontext(&lane[l]);
      lane[l].uc_stack.ss_sp = stack[l].get();
      lane[l].uc_stack.ss_size = kStack;
      lane[l].uc_link = nullptr;
      const uintptr_t p = (uintptr_t)this;
      cur = l;
      makecontext(&lane[l], (void (*)())run_lane, 2, (unsigned)p, (unsigned)(p >> 32));
    }
    for (;;) {
      int left = 0;
      for (int i = 0; i < kLanes; ++i) {
        const int l = order == 0 ? i : order == 1 ? kLanes - 1 - i : (i + 13) % kLanes;
        if (done[l]) continue;
        cur = l;
        enter(l);
        left += !done[l];
      }
      if (left == 0) return;
      if (left != kLanes) diverged = true;              // some lanes ended before a sync of others
    }
  }
};

void run_lane(unsigned lo, unsigned hi) {
  Warp &w = *(Warp *)((uintptr_t)lo | (uintptr_t)hi << 32);
#ifdef __SANITIZE_ADDRESS__
  __sanitizer_finish_switch_fiber(nullptr, &w.main_stack, &w.main_size);
#endif
  const int l = w.cur;
  w.body(w, l);
  w.done[l] = true;
  w.yield(l, true);
}

struct EmuLanes {
  static constexpr bool kWarp = true;
  Warp *w;
  int l;
  int lane() const { return l; }
  int width() const { return kLanes; }
  bool leader() const { return l == 0; }
  void sync() const { w->yield(l); }
  uint32_t match(int v) const {
    w->slot[l] = (uint32_t)v;
    sync();
    uint32_t m = 0;
    for (int i = 0; i < kLanes; ++i) m |= (uint32_t)(w->slot[i] == (uint32_t)v) << i;
    sync();
    return m;
  }
  uint32_t from(uint32_t v, int i) const {
    w->slot[l] = v;
    sync();
    const uint32_t r = w->slot[i];
    sync();
    return r;
  }
};

void decode_lane(Warp &w, int l) {
  w.st[l] = inflate_block(w.in, w.inlen, w.out, w.outlen, *w.tabs, EmuLanes{&w, l});
}
void crc_lane(Warp &w, int l) { w.crc[l] = crc32(w.crc_t, w.out, w.outlen, EmuLanes{&w, l}); }

}  // namespace

int main(int argc, char **argv) {
  if (argc < 2) return 2;
  FILE *f = std::fopen(argv[1], "rb");
  if (!f) return 2;
  std::unique_ptr<Tables> t1(new Tables()), t32(new Tables());
  uint32_t crc_t[256];
  crc32_table(crc_t);
  Warp w;
  w.tabs = t32.get();
  w.crc_t = crc_t;
  long runs = 0, ok = 0;
  for (;;) {
    uint32_t hdr[2];
    if (std::fread(hdr, 4, 2, f) != 2) break;
    std::vector<uint8_t> in(hdr[0]);
    if (hdr[0] && std::fread(in.data(), 1, hdr[0], f) != hdr[0]) return 3;
    const uint32_t n = hdr[1];
    std::unique_ptr<uint8_t[]> want(new uint8_t[n ? n : 1]);
    std::memset(want.get(), 0xA5, n);
    const int st = inflate_block(in.data(), hdr[0], want.get(), n, *t1, SerialLanes{});
    // the device's input: any alignment, 16 bytes of slack (exact-size buffers, so that
    // the sanitizer sees any overrun)
    const uint32_t shift = (uint32_t)(runs * 5 % 8);
    std::unique_ptr<uint64_t[]> ib(new uint64_t[(shift + hdr[0] + 16 + 7) / 8]);
    std::memset(ib.get(), 0xEE, (shift + hdr[0] + 16 + 7) / 8 * 8);
    uint8_t *p = (uint8_t *)ib.get() + shift;
    if (hdr[0]) std::memcpy(p, in.data(), hdr[0]);
    std::unique_ptr<uint8_t[]> ob(new uint8_t[n ? n : 1]);
    std::memset(ob.get(), 0x5A, n);
    w.in = p;
    w.inlen = hdr[0];
    w.out = ob.get();
    w.outlen = n;
    w.run(decode_lane, (int)(runs % 3));
    for (int l = 0; l < kLanes; ++l)
      if (w.st[l] != st) {
        std::fprintf(stderr, "stream %ld: lane %d ends with %d, one lane with %d\n", runs, l, w.st[l], st);
        return 4;
      }
    if (w.diverged) {
      std::fprintf(stderr, "stream %ld: lanes parted\n", runs);
      return 5;
    }
    if (st == kOk) {
      if (std::memcmp(ob.get(), want.get(), n) != 0) {
        std::fprintf(stderr, "stream %ld: bytes differ\n", runs);
        return 6;
      }
      w.run(crc_lane, (int)(runs % 3));
      const uint32_t c = crc32(crc_t, want.get(), n, SerialLanes{});
      for (int l = 0; l < kLanes; ++l)
        if (w.crc[l] != c || w.diverged) {
          std::fprintf(stderr, "stream %ld: CRC of lane %d\n", runs, l);
          return 7;
        }
      ++ok;
    }
    ++runs;
  }
  std::fclose(f);
  std::printf("%ld %ld\n", runs, ok);
  return 0;
}
