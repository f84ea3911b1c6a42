// Ordered sums by scans (hmp_ordered_sum.h) against the sequential FP32 sum, on the CPU: the run of
// elements is grouped into random blocks, composed block by block as the kernel's threads, warps and
// chunks do, and the first partial sum outside the binade falls back to a plain addition.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "hmp_ordered_sum.h"

static float scanned(const std::vector<float>& x, std::mt19937& rng, long& steps) {
  float s = 0.f;
  size_t pos = 0;
  while (pos < x.size()) {
    float scale, unit;
    if (!hmp::ordered_scale(s, scale, unit)) {
      s += x[pos++];
      ++steps;
      continue;
    }
    // blocks of 1..64 elements: the composed run of each must give the partial sum at its end
    int S = int(s * scale);
    bool failed = false;
    while (pos < x.size() && !failed) {
      const size_t end = std::min(x.size(), pos + 1 + rng() % 64);
      hmp::OrderedRun run{0, 0};
      int P = S;
      size_t i = pos;
      for (; i < end; ++i) {
        hmp::OrderedRun e;
        const bool whole = hmp::ordered_element(x[i] * scale, e);
        int d = 0;
        if (hmp::ordered_plain(x[i] * scale, d) != (whole && e.d0 == e.d1) || (whole && e.d0 == e.d1 && d != e.d0)) {
          std::printf("plain element differs\n");
          std::exit(1);
        }
        if (!whole) break;
        const int n = hmp::ordered_apply(e, P);
        if (!hmp::ordered_inside(n)) break;
        P = n;
        run = hmp::ordered_then(run, e);
      }
      if (hmp::ordered_apply(run, S) != P) {
        std::printf("composition differs\n");
        std::exit(1);
      }
      S = P;
      if (i < end) {
        s = float(S) * unit + x[i];
        ++steps;
        failed = true;
        pos = i + 1;
      } else {
        pos = end;
      }
    }
    if (!failed) s = float(S) * unit;
  }
  return s;
}

int main() {
  std::mt19937 rng(11);
  long sums = 0, steps = 0, elements = 0;
  for (int trial = 0; trial < 3000; ++trial) {
    const int n = 1 + int(rng() % 3000), kind = int(rng() % 8);
    std::normal_distribution<float> N(0.f, 1.f);
    const float mean = N(rng) * 4.f;
    std::vector<float> x(n);
    for (auto& v : x) {
      switch (kind) {
        case 0: v = mean + 0.1f * N(rng); break;                        // a moving camera
        case 1: v = 0.05f * N(rng); break;                              // a still one: sums near zero
        case 2: v = float(int(rng() % 9)) * 0.5f - 2.f; break;          // halves: exact and tied sums
        case 3: v = std::ldexp(N(rng), int(rng() % 60) - 30); break;    // every magnitude
        case 4: v = rng() % 3 ? 0.f : -0.f; break;
        case 5: v = 16777216.f * (rng() % 2 ? 1.f : -1.f) + float(rng() % 5); break;
        case 6: v = 1.f + std::ldexp(1.f, -1 - int(rng() % 24)); break; // ties at each binade
        default: v = rng() % 500 ? N(rng) : (rng() % 2 ? INFINITY : NAN); break;
      }
    }
    float ref = 0.f;
    for (float v : x) ref += v;
    const float got = scanned(x, rng, steps);
    if (std::memcmp(&ref, &got, 4) && !(ref != ref && got != got)) {
      std::printf("trial %d kind %d n %d: %a vs %a\n", trial, kind, n, double(got), double(ref));
      return 1;
    }
    ++sums;
    elements += n;
  }
  std::printf("%ld sums, %ld elements, %ld added one by one\n", sums, elements, steps);
  return 0;
}
