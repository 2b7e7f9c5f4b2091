// The emit pass's output sink (see WindowSink).  Like k2j_format.cuh this header also compiles as plain C++
// (K2J_HD drops the CUDA qualifiers), so the window logic can be exercised on a CPU: there the "shared memory"
// window and the "global memory" output are ordinary host arrays.
#pragma once
#include <stdint.h>

#include "k2j_format.cuh"

namespace k2j {

// (hi:lo << s) >> 32 for s in 0..31: the bytes that a left shift by s pushes out of lo, below hi's shifted bytes
K2J_HD uint32_t funnel_l(uint32_t lo, uint32_t hi, uint32_t s) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, s);
#else
  return s ? (hi << s) | (lo >> (32u - s)) : hi;
#endif
}
// the 32 bits of (hi:lo) from bit s on, s in 0..31
K2J_HD uint32_t funnel_r(uint32_t lo, uint32_t hi, uint32_t s) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_r(lo, hi, s);
#else
  return s ? (lo >> s) | (hi << (32u - s)) : lo;
#endif
}
// one 256-bit store to a 32-byte aligned address
K2J_HD void store32(uint8_t* p, uint64_t a, uint64_t b, uint64_t c, uint64_t d) {
#if defined(__CUDA_ARCH__)
  asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
#else
  uint64_t v[4] = {a, b, c, d};
  memcpy(p, v, 32);
#endif
}

// ---- output sink: a per-thread window in shared memory, flushed in 32-byte blocks ----------------------
// Every thread owns a window of kWinBytes in shared memory that mirrors the part of its event being written:
// window byte p stands for global address gbase + p, and gbase is 32-byte aligned, so window and output agree
// modulo 32.  Appending is cheap: text arrives in 32-bit pieces, a funnel shift puts each piece at the byte phase
// of the write position, and plain 32-bit stores put it into the window (the word being filled is kept in a
// register and stored again as it grows).  When the window runs out of room the thread writes its complete
// 32-byte blocks to global memory, each as one 256-bit store (a full DRAM sector, so the L2 never has to fetch
// the rest of one), moves the open block to the front of the window and goes on.
// The windows of a warp are interleaved word by word: word k of lane t sits at [k][t], i.e. in bank t wherever
// the lanes' write positions are, so no window access of a warp ever meets a bank conflict.
// The two 8-byte words an event may share with its neighbours are written without knowing the neighbour's
// bytes: every event begins with "\n  {\n   " and ends with "\n  },", so the neighbour's (at most three) bytes
// inside a shared 4-byte half are known constants, and a half that belongs wholly to the neighbour is not
// touched.  Both owners write a shared half with the same bytes.  The other words of an event's first and last
// (partial) block leave as 8-byte stores.
constexpr uint64_t kEventHead8 = 0x2020200A7B20200Aull;  // "\n  {\n   "  first 8 bytes of every event
constexpr uint64_t kEventTail8 = 0x2C7D20200A000000ull;  // "\n  },"      last 5 bytes of every event, in the top bytes
constexpr uint32_t kMinEventBytes = 16;
constexpr int kWinBytes = 160;
constexpr int kWinWords = kWinBytes / 4;
constexpr int kWinStride = 32;              // words between consecutive words of one window (the lanes of a warp)
constexpr int kWinPadWords = 8 * kWinStride;  // after the last warp's windows: the move of the open block reads a whole block,
                                              // which may reach past the end of a window (into the next warp's rows, or this pad)
constexpr uint32_t kWinSlack = 40;          // room that always stays free after ensure(): 32 bytes of small appends that
                                            // do not ask first, and the word past the end that an append may touch
K2J_HD uint64_t pack64(uint32_t lo, uint32_t hi) { return (uint64_t)lo | ((uint64_t)hi << 32); }

// A window: on the GPU the 32-bit shared-memory address of its word 0 (so that out-of-line functions that take one read and
// write shared memory, not generic addresses), on a CPU a pointer to it.
#if defined(__CUDACC__)
using Win = uint32_t;
__device__ __forceinline__ uint32_t win_ld(Win w, uint32_t k) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(w + k * (uint32_t)(4 * kWinStride)));
  return v;
}
__device__ __forceinline__ void win_st(Win w, uint32_t k, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(w + k * (uint32_t)(4 * kWinStride)), "r"(v));
}
__device__ __forceinline__ Win win_from(Win w, uint32_t k) { return w + k * (uint32_t)(4 * kWinStride); }
#else
using Win = uint32_t*;
inline uint32_t win_ld(Win w, uint32_t k) { return w[k * (uint32_t)kWinStride]; }
inline void win_st(Win w, uint32_t k, uint32_t v) { w[k * (uint32_t)kWinStride] = v; }
inline Win win_from(Win w, uint32_t k) { return w + k * (uint32_t)kWinStride; }
#endif
// the same as two 128-bit stores, for code out of line: in a function that was called, 256-bit stores left three quarters of
// a block unwritten (ptxas 12.9; the same source in line is right; why was not found)
K2J_HD void store16x2(uint8_t* p, uint64_t a, uint64_t b, uint64_t c, uint64_t d) {
#if defined(__CUDA_ARCH__)
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(a, b);
  *reinterpret_cast<ulonglong2*>(p + 16) = make_ulonglong2(c, d);
#else
  uint64_t v[4] = {a, b, c, d};
  memcpy(p, v, 32);
#endif
}
template <bool WIDE> K2J_HD void store_block(uint8_t* p, uint64_t a, uint64_t b, uint64_t c, uint64_t d) {
  if (WIDE) store32(p, a, b, c, d); else store16x2(p, a, b, c, d);
}
template <bool WIDE> K2J_HD void win_block_out(Win win, uint8_t* gbase, uint32_t b) {
  const uint32_t k = 8u * b;
  const uint32_t x0 = win_ld(win, k), x1 = win_ld(win, k + 1), x2 = win_ld(win, k + 2), x3 = win_ld(win, k + 3), x4 = win_ld(win, k + 4),
                 x5 = win_ld(win, k + 5), x6 = win_ld(win, k + 6), x7 = win_ld(win, k + 7);
  store_block<WIDE>(gbase + 32u * b, pack64(x0, x1), pack64(x2, x3), pack64(x4, x5), pack64(x6, x7));
}
// Writes the complete 32-byte blocks of a window to global memory and moves the open block to the front; returns their
// number.  `open`: 0, or the offset of the first word that the first block has still to write (its earlier words are out).
template <bool WIDE>
K2J_HD uint32_t window_flush(Win win, uint32_t pos, uint32_t carry, uint8_t* gbase, uint32_t open) {
  win_st(win, pos >> 2, carry);
  const uint32_t nb = pos >> 5;
  uint32_t b = 0;
  if (open != 0u && nb != 0u) {  // a block whose first words are out already: whole words only
    for (uint32_t o = open; o < 32u; o += 8u) *reinterpret_cast<uint64_t*>(gbase + o) = pack64(win_ld(win, o >> 2), win_ld(win, (o >> 2) + 1u));
    b = 1;
  }
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
  for (; b + 2u <= nb; b += 2u) {  // two blocks at a time: sixteen loads in flight before the two stores
    const uint32_t k = 8u * b;
    const uint32_t x0 = win_ld(win, k), x1 = win_ld(win, k + 1), x2 = win_ld(win, k + 2), x3 = win_ld(win, k + 3), x4 = win_ld(win, k + 4),
                   x5 = win_ld(win, k + 5), x6 = win_ld(win, k + 6), x7 = win_ld(win, k + 7);
    const uint32_t y0 = win_ld(win, k + 8), y1 = win_ld(win, k + 9), y2 = win_ld(win, k + 10), y3 = win_ld(win, k + 11), y4 = win_ld(win, k + 12),
                   y5 = win_ld(win, k + 13), y6 = win_ld(win, k + 14), y7 = win_ld(win, k + 15);
    store_block<WIDE>(gbase + 32u * b, pack64(x0, x1), pack64(x2, x3), pack64(x4, x5), pack64(x6, x7));
    store_block<WIDE>(gbase + 32u * b + 32u, pack64(y0, y1), pack64(y2, y3), pack64(y4, y5), pack64(y6, y7));
  }
  if (b < nb) win_block_out<WIDE>(win, gbase, b);
  if (nb != 0u) {
    const uint32_t k = 8u * nb;
    const uint32_t x0 = win_ld(win, k), x1 = win_ld(win, k + 1), x2 = win_ld(win, k + 2), x3 = win_ld(win, k + 3), x4 = win_ld(win, k + 4),
                   x5 = win_ld(win, k + 5), x6 = win_ld(win, k + 6), x7 = win_ld(win, k + 7);
    win_st(win, 0, x0); win_st(win, 1, x1); win_st(win, 2, x2); win_st(win, 3, x3);
    win_st(win, 4, x4); win_st(win, 5, x5); win_st(win, 6, x6); win_st(win, 7, x7);
  }
  return nb;
}

// WIDE: blocks leave as 256-bit stores.  Only a sink that lives in a kernel's own code, with everything it is handed to in
// line, may do that (see store16x2): such a kernel names InlineSink.  WindowSink is right everywhere.
template <bool WIDE> struct Sink {
  static constexpr bool kCounting = false, kWide = WIDE;
  Win win;                // this thread's window
  uint32_t pos;           // window offset of the next byte
  uint32_t carry;         // the 32-bit word being filled: bytes below pos & 3 are set, the rest is zero
  uint32_t open;          // 0, or: the window's first block has been written up to this offset (see window_flush)
  uint8_t* gbase;         // global address of window byte 0, 32-byte aligned
  K2J_HD uint64_t W64(uint32_t k) const { return pack64(win_ld(win, k), win_ld(win, k + 1u)); }  // the 8 bytes from word k on
  K2J_HD void init(uint8_t* dst, uint32_t, Win window) {
    const uint32_t phase32 = (uint32_t)(reinterpret_cast<uintptr_t>(dst) & 31u), phase = phase32 & 7u, sh = 8u * phase;
    win = window; gbase = dst - phase32; pos = phase32; carry = 0u;
    const uint32_t w0 = phase32 & ~7u;  // the event's first 8-byte word is written here and now
    open = phase32 ? w0 + 8u : 0u;
    const uint64_t w = ((kEventTail8 >> 1) >> (63u - sh)) | (kEventHead8 << sh);
    if (phase < 4u) *reinterpret_cast<uint64_t*>(gbase + w0) = w;
    else *reinterpret_cast<uint32_t*>(gbase + w0 + 4) = (uint32_t)(w >> 32);
  }
  // Writes the complete 32-byte blocks of the window to global memory and moves the open block to the front.
  template <bool W = WIDE> K2J_HD void flush() {
    const uint32_t nb = window_flush<W>(win, pos, carry, gbase, open);
    if (nb != 0u) open = 0u;
    gbase += 32u * nb; pos -= 32u * nb;
  }
  // After this call n more bytes fit, with kWinSlack to spare.  n <= kWinBytes - 32 - kWinSlack.
  // On the GPU the lanes of a warp that are executing together flush together, as soon as one of them needs
  // the room: a flush that only some lanes take costs the warp as much as one that all of them take, and windows
  // of a warp fill at about the same rate.  (A flush that comes early only writes the blocks that are complete.)
  K2J_HD void ensure(uint32_t n) {
#if defined(__CUDA_ARCH__)
    if (__any_sync(__activemask(), pos + n + kWinSlack > (uint32_t)kWinBytes)) flush();
#else
    if (pos + n + kWinSlack > (uint32_t)kWinBytes) flush();
#endif
  }
  // The same without the slack, for callers that count every byte they append: n <= kWinBytes - 40 bytes fit (an append may
  // touch the word behind its last byte).
  K2J_HD void room(uint32_t n) {
#if defined(__CUDA_ARCH__)
    if (__any_sync(__activemask(), pos + n + 8u > (uint32_t)kWinBytes)) flush();
#else
    if (pos + n + 8u > (uint32_t)kWinBytes) flush();
#endif
  }
  // A long string from an 8-byte aligned word array (words up to one behind its last byte are readable): past the window,
  // straight from registers to the output.  The bytes up to the output's next 8-byte boundary and those behind the last one
  // go through the window.
  template <bool W = WIDE> K2J_HD void long_words(const uint64_t* w, uint32_t len) {
    uint32_t h = (0u - pos) & 7u;
    h = h < len ? h : len;
    uint64_t cur = len != 0u ? w[0] : 0ull;
    put64(h != 0u ? cur & (~0ull >> (8u * (8u - h))) : 0ull, h);
    uint32_t n = (len - h) >> 3;  // whole words of output
    if (n != 0u) {
      flush<W>();
      for (uint32_t o = open; o < pos; o += 8u) *reinterpret_cast<uint64_t*>(gbase + o) = W64(o >> 2);
      uint8_t* dst = gbase + pos;
      const uint32_t odd = h & 4u, sh = 8u * (h & 3u);
      auto shifted = [&](uint64_t x, uint64_t y) {  // the 8 bytes from byte h of (x, y) on
        const uint32_t w0 = odd ? (uint32_t)(x >> 32) : (uint32_t)x, w1 = odd ? (uint32_t)y : (uint32_t)(x >> 32), w2 = odd ? (uint32_t)(y >> 32) : (uint32_t)y;
        return pack64(funnel_r(w0, w1, sh), funnel_r(w1, w2, sh));
      };
      for (; n != 0u && (reinterpret_cast<uintptr_t>(dst) & 31u) != 0u; n--, dst += 8) {
        const uint64_t y = *++w;
        *reinterpret_cast<uint64_t*>(dst) = shifted(cur, y);
        cur = y;
      }
      uint64_t y[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
      for (uint32_t k = 0; k < 8u; k++) if (k < (n & ~3u)) y[k] = w[k + 1u];
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
      while (n >= 4u) {  // two blocks a round; the next round's words are on their way while these are written
        uint64_t x[8];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
        for (uint32_t k = 0; k < 8u; k++) x[k] = y[k];
        const uint32_t m = n >= 8u ? 8u : 4u;
        w += m; n -= m;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
        for (uint32_t k = 0; k < 8u; k++) if (k < (n & ~3u)) y[k] = w[k + 1u];
        store_block<W>(dst, shifted(cur, x[0]), shifted(x[0], x[1]), shifted(x[1], x[2]), shifted(x[2], x[3]));
        cur = x[3];
        if (m == 8u) {
          store_block<W>(dst + 32, shifted(cur, x[4]), shifted(x[4], x[5]), shifted(x[5], x[6]), shifted(x[6], x[7]));
          cur = x[7];
        }
        dst += 8u * m;
      }
      for (; n != 0u; n--, dst += 8) {
        const uint64_t y = *++w;
        *reinterpret_cast<uint64_t*>(dst) = shifted(cur, y);
        cur = y;
      }
      pos = (uint32_t)(reinterpret_cast<uintptr_t>(dst) & 31u); open = pos; carry = 0u;
      gbase = dst - pos;
    }
    const uint32_t r = (len - h) & 7u;  // (h is below 8: cur holds the first of them)
    if (r != 0u) {
      const uint64_t y = h + r > 8u ? w[1] : 0ull;
      const uint64_t x = (cur >> (8u * h)) | ((y << 1) << (63u - 8u * h));
      put64(x & (~0ull >> (8u * (8u - r))), r);
    }
  }
  // append the low `len` (0..4) bytes of w; bytes above len must be zero
  K2J_HD void put(uint32_t w, int len) {
    const uint32_t ph = pos & 3u, s = ph << 3;
    const uint32_t t = carry | (w << s);
    win_st(win, pos >> 2, t);
    carry = ph + (uint32_t)len >= 4u ? funnel_l(w, 0u, s) : t;  // the funnel shift gives w >> (32 - s), and 0 for s = 0
    pos += (uint32_t)len;
  }
  K2J_HD void put4(uint32_t w) {
    const uint32_t s = (pos & 3u) << 3;
    win_st(win, pos >> 2, carry | (w << s));
    carry = funnel_l(w, 0u, s);
    pos += 4u;
  }
  // append the low `len` (0..8) bytes of w; bytes above len must be zero
  K2J_HD void put64(uint64_t w, uint32_t len) {
    const uint32_t lo = (uint32_t)w, hi = (uint32_t)(w >> 32);
    const uint32_t ph = pos & 3u, s = ph << 3, i = pos >> 2;
    const uint32_t t0 = carry | (lo << s), t1 = funnel_l(lo, hi, s), t2 = funnel_l(hi, 0u, s);
    win_st(win, i, t0); win_st(win, i + 1, t1);
    const uint32_t k = (ph + len) >> 2;  // words completed: 0..2
    carry = k == 0u ? t0 : (k == 1u ? t1 : t2);
    pos += len;
  }
  K2J_HD void put8w(uint64_t w) {  // append 8 bytes
    const uint32_t lo = (uint32_t)w, hi = (uint32_t)(w >> 32);
    const uint32_t s = (pos & 3u) << 3, i = pos >> 2;
    win_st(win, i, carry | (lo << s)); win_st(win, i + 1, funnel_l(lo, hi, s));
    carry = funnel_l(hi, 0u, s);
    pos += 8u;
  }
  K2J_HD void skip(uint32_t) {}
  template <int N> K2J_HD void lit(const Lit<N>& l) {
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < N / 4; i++) put4(l.w[i]);
    if (N % 4) put(l.w[N / 4], N % 4);
  }
  // the first n (at most 64) bytes of eight words; the caller has asked for the room
  K2J_HD void piece(const uint64_t (&x)[8], uint32_t n) {
    const uint32_t nw = n >> 3;
    const uint32_t s = (pos & 3u) << 3;
    uint32_t i = pos >> 2, c = carry;
    uint64_t last = x[0];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (uint32_t k = 0; k < 8u; k++) {
      if (k < nw) {
        const uint32_t lo = (uint32_t)x[k], hi = (uint32_t)(x[k] >> 32);
        win_st(win, i, c | (lo << s)); win_st(win, i + 1, funnel_l(lo, hi, s));
        c = funnel_l(hi, 0u, s);
        i += 2;
      }
      if (k == nw) last = x[k];
    }
    carry = c; pos += 8u * nw;
    const uint32_t rem = n & 7u;
    if (rem) put64(last & (~0ull >> (8u * (8u - rem))), rem);
  }
  // `len` bytes from an 8-byte aligned word array, any length: 64 bytes at a time, asking for room first.  The
  // words of a piece are all loaded before the first one is appended: a load that waits behind the append of
  // the word before it (the compiler cannot move it across the window's stores) pays the memory latency once
  // per word instead of once per piece.
  K2J_HD void words(const uint64_t* w, uint32_t len) {
    uint64_t x[8], y[8];
    {
      const uint32_t touched = ((len < 64u ? len : 64u) + 7u) >> 3;  // words read, the partial last one included
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
      for (uint32_t k = 0; k < 8u; k++) x[k] = k < touched ? w[k] : 0ull;
    }
    while (true) {
      const uint32_t n = len < 64u ? len : 64u;
      {  // the piece after this one is on its way while this one is appended
        const uint32_t left = len - n, touched = ((left < 64u ? left : 64u) + 7u) >> 3;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
        for (uint32_t k = 0; k < 8u; k++) y[k] = k < touched ? w[8 + k] : 0ull;
      }
      ensure(n);
      piece(x, n);
      len -= n;
      if (len == 0u) break;
      w += 8;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
      for (uint32_t k = 0; k < 8u; k++) x[k] = y[k];
    }
  }
  // `len` bytes from any address: the bytes up to the next 8-byte boundary, then whole words
  K2J_HD void bytes(const uint8_t* src, uint32_t len) {
    const uint32_t a = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 7u);
    const uint64_t* w = reinterpret_cast<const uint64_t*>(src - a);
    if (a != 0u && len != 0u) {
      const uint32_t n = len < 8u - a ? len : 8u - a;
      put64((w[0] >> (8u * a)) & (~0ull >> (8u * (8u - n))), n);
      len -= n; w += 1;
    }
    if (len) words(w, len);
  }
  // Writes what is left: the complete blocks, the complete words of the open block, then the word holding the
  // event's end.  Returns false if the byte count differs from the size the event was given.
  K2J_HD bool finish(const uint8_t* dst, uint32_t size) {
    flush();
    for (uint32_t o = open; o + 8u <= pos; o += 8u)  // the event's very first word was written by init
      *reinterpret_cast<uint64_t*>(gbase + o) = W64(o >> 2);
    const uint32_t e = pos & 7u;
    if (e) {
      const uint64_t lo = (pos & 4u) ? pack64(win_ld(win, (pos >> 2) - 1u), carry) : (uint64_t)carry;
      const uint64_t t = lo | (0x20200Aull << (8u * e));  // the next event begins "\n  "
      if (e > 4u) *reinterpret_cast<uint64_t*>(gbase + (pos & ~7u)) = t;
      else *reinterpret_cast<uint32_t*>(gbase + (pos & ~7u)) = (uint32_t)t;
    }
    return gbase + pos == dst + size;
  }
};
using WindowSink = Sink<false>;
using InlineSink = Sink<true>;

}  // namespace k2j
