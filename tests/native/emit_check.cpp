// CPU harness around the emit pass's way past the window for long strings (k2j_sink.cuh) and around doubles handed from one
// pass to the next as packed words (k2j_format.cuh).
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <random>
#include <string>
#include <vector>
#include "k2j_sink.cuh"

extern "C" {
// Events of short appends and long strings, in random order and at every alignment; 0, 1 + the first differing offset, or
// -1 when a sink reported a size mismatch.
int64_t ec_long_words(uint64_t seed, int n_events, int max_len) {
  std::mt19937_64 rng(seed);
  auto rnd = [&](uint64_t n) { return (uint64_t)(rng() % n); };
  auto text = [&](uint64_t n) { std::string s; for (uint64_t i = 0; i < n; i++) s += (char)(0x21 + rnd(0x5d)); return s; };
  std::vector<std::vector<std::string>> parts(n_events);  // even: short, odd: long
  std::vector<std::string> whole(n_events);
  std::vector<uint64_t> offs(n_events);
  std::string expected;
  for (int e = 0; e < n_events; e++) {
    const int n = (int)rnd(4);
    std::string t = "\n  {\n   \"ph\"";
    for (int k = 0; k < n; k++) { parts[e].push_back(text(rnd(20))); parts[e].push_back(text(rnd(max_len + 1))); t += parts[e][2 * k] + parts[e][2 * k + 1]; }
    whole[e] = t + "\n  },";
    offs[e] = expected.size();
    expected += whole[e];
  }
  std::vector<uint8_t> raw(expected.size() + 160, 0xEE);
  uint8_t* out = raw.data() + (32 - (reinterpret_cast<uintptr_t>(raw.data()) & 31)) % 32;
  static uint32_t window[k2j::kWinWords * k2j::kWinStride + k2j::kWinPadWords];
  std::vector<int> order(n_events);
  for (int i = 0; i < n_events; i++) order[i] = i;
  for (int i = n_events - 1; i > 0; i--) std::swap(order[i], order[rnd(i + 1)]);
  bool ok = true;
  auto put = [](k2j::WindowSink& s, const std::string& t) {
    for (size_t i = 0; i < t.size(); i += 8) {
      const uint32_t n = (uint32_t)std::min<size_t>(8, t.size() - i);
      uint64_t w = 0;
      memcpy(&w, t.data() + i, n);
      s.room(8);
      s.put64(w, n);
    }
  };
  for (int e : order) {
    for (auto& x : window) x = 0xA5A5A5A5u;
    k2j::WindowSink s;
    s.init(out + offs[e], (uint32_t)whole[e].size(), window);
    put(s, "\n  {\n   \"ph\"");
    for (size_t k = 0; k < parts[e].size(); k += 2) {
      put(s, parts[e][k]);
      const std::string& t = parts[e][k + 1];
      std::vector<uint64_t> w(t.size() / 8 + 2, 0x5555555555555555ull);  // one word behind the last byte's is readable
      memcpy(w.data(), t.data(), t.size());
      s.room(16);
      if (k & 2) s.long_words<true>(w.data(), (uint32_t)t.size()); else s.long_words<false>(w.data(), (uint32_t)t.size());
    }
    put(s, "\n  },");
    ok = s.finish(out + offs[e], (uint32_t)whole[e].size()) && ok;
  }
  if (!ok) return -1;
  for (size_t i = 0; i < expected.size(); i++) if (out[i] != (uint8_t)expected[i]) return 1 + (int64_t)i;
  return 0;
}
// Number of values whose packed word prints differently from the value itself; *n_left: values that pack_double leaves out.
int64_t ec_packed_doubles(const double* v, int64_t n, int64_t* n_left) {
  int64_t bad = 0;
  *n_left = 0;
  for (int64_t i = 0; i < n; i++) {
    const uint64_t w = k2j::pack_double(v[i]);
    if (w == 0) { ++*n_left; continue; }
    k2j::StringSink a, b; k2j::CountSink c;
    k2j::put_double_value(a, v[i]); k2j::put_packed_double(b, w); k2j::put_packed_double(c, w);
    bad += a.s != b.s || c.n != b.s.size();
  }
  return bad;
}
}
