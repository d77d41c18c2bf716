// finish_choose (cccl_gb300/csrc/sort_policy.h) on the CPU: the digits the plain sort partitions
// by, from the sample's pair counts of known distributions.
#include <cstdint>
#include <cstdio>
#include <initializer_list>

#include <algorithm>
#include <vector>

#include "sort_policy.h"

using namespace gb300;

static int failures = 0;

// Pairs a sample of S keys is expected to hold when the top l digits split n keys into buckets
// of `bucket[l - 1]` keys each (0: none to be seen).
static int choose(int kb, unsigned long long n, int cap, uint32_t trivial, std::initializer_list<double> bucket,
                  std::initializer_list<unsigned> heavy, int mode, uint32_t* piece)
{
  const uint32_t S = finish_sample_items(n);
  unsigned long long light[8] = {};
  uint32_t hv[8]              = {};
  int l                       = 0;
  for (double b : bucket)
  {
    light[l++] = (unsigned long long) (b * double(S) * double(S) / double(n) + 0.5);
  }
  l = 0;
  for (unsigned h : heavy)
  {
    hv[l++] = h;
  }
  *piece = 0;
  return finish_choose(kb, trivial, light, hv, n, S, uint32_t(cap), finish_cost(kb, 4), mode, piece);
}

static void expect(const char* what, int got, int want, const uint32_t& piece, int cap)
{
  if (got != want || (got != 0 && (piece < uint32_t(cap / FINISH_SMALLEST_PIECE) || piece > uint32_t(cap))))
  {
    std::printf("%s: digits %d, expected %d, piece %u of %d\n", what, got, want, piece, cap);
    ++failures;
  }
}

int main()
{
  uint32_t piece = 0;
  const int cap = finish_cap(8, 4, false);
  const int SEP = PLAN_MODE_SEPARATE, DBL = PLAN_MODE_DOUBLE;
  const unsigned long long n28 = 1ull << 28, n24 = 1ull << 24;
  const uint32_t S28 = finish_sample_items(n28), S24 = finish_sample_items(n24);
  expect("2^28 uniform", choose(8, n28, cap, 0, {0, 4096, 16}, {S28}, SEP, &piece), 2, piece, cap);
  expect("2^28 uniform, double buffer", choose(8, n28, cap, 0, {0, 4096, 16}, {S28}, DBL, &piece), 2, piece, cap);
  expect("2^24 uniform", choose(8, n24, cap, 0, {0, 256, 1}, {S24}, SEP, &piece), 2, piece, cap);
  expect("buckets above the capacity", choose(8, 1ull << 29, cap, 0, {0, 8192, 32}, {8192}, SEP, &piece), 3, piece, cap);
  // an odd number of passes takes one more in a double buffer
  expect("three digits, double buffer", choose(8, 1ull << 29, cap, 0, {0, 8192, 32}, {8192}, DBL, &piece), 3, piece, cap);
  expect("three constant digits on top", choose(8, n24, cap, 0xe0, {0, 0, 0, 0, 256, 1}, {S24, S24, S24, S24}, SEP, &piece),
         5, piece, cap);
  expect("only low digits vary", choose(8, n24, cap, 0xfc, {0, 0, 0, 0, 0, 0, 0, 256},
                                        {S24, S24, S24, S24, S24, S24, S24}, SEP, &piece), 0, piece, cap);
  expect("all equal", choose(8, n24, cap, 0xff, {}, {S24, S24, S24, S24, S24, S24, S24, 0}, SEP, &piece), 0, piece, cap);
  expect("a tenth in one bucket", choose(8, n24, cap, 0, {0, 256, 1}, {S24, S24 / 10, S24 / 10, S24 / 10, S24 / 10, S24 / 10, S24 / 10, 0}, SEP, &piece),
         2, piece, cap);
  expect("half in one bucket", choose(8, n24, cap, 0, {0, 256, 1}, {S24, S24 / 2, S24 / 2, S24 / 2, S24 / 2, S24 / 2, S24 / 2, 0}, SEP, &piece),
         0, piece, cap);
  expect("every key 64 times", choose(8, n24, cap, 0, {0, 256, 64, 64, 64, 64, 64, 64}, {S24}, SEP, &piece), 0, piece, cap);
  expect("a key 4000 times", choose(8, n24, cap, 0, {0, 256, 3, 3, 3, 3, 3, 0}, {S24, 0, 0, 0, 0, 0, 0, 3}, SEP, &piece), 2, piece,
         cap);
  expect("clusters at every scale", choose(8, n28, cap, 0, {0, 4000, 600, 90, 14, 2}, {S28}, SEP, &piece), 0, piece, cap);
  expect("4-byte uniform", choose(4, n28, finish_cap(4, 0, false), 0, {0, 4096, 16}, {S28}, SEP, &piece), 2, piece,
         finish_cap(4, 0, false));
  expect("4-byte, three digits needed", choose(4, 1ull << 29, finish_cap(4, 0, false), 0, {0, 8192, 32}, {8192}, SEP, &piece), 0,
         piece, finish_cap(4, 0, false));
  // shared memory of every shape: two CTAs and one per SM of 227 KB, 1 KB reserved each
  for (int kb : {4, 8})
  {
    for (int vb : {0, 4, 8})
    {
      if (2 * (finish_smem_bytes(kb, vb, false) + 1024) > 228 * 1024 || finish_smem_bytes(kb, vb, true) > 227 * 1024
          || finish_tpb(kb, vb, true) + 32 > 1024 || finish_cap(kb, vb, false) > 8191 || finish_cap(kb, vb, true) > 16383
          || finish_bins(kb, vb, true) > 8192)
      {
        std::printf("shape of %d + %d bytes\n", kb, vb);
        ++failures;
      }
    }
  }
  // The places sampled: distinct, inside the array, and spread at random: as many pairs of neighbours
  // (within a stretch of n / samples places) as independent places have, within five deviations.
  for (uint32_t n : {(1u << 22), (1u << 22) + 1u, 5000011u, 100000007u, 1u << 28, (1u << 30) + 12345u, (1u << 31) - 1u})
  {
    const uint32_t samples = finish_sample_items(n);
    const int half         = finish_sample_half(n);
    std::vector<uint32_t> at;
    for (uint32_t i = 0; i < samples; ++i)
    {
      at.push_back(finish_sample_place(i, n, half));
    }
    std::sort(at.begin(), at.end());
    const uint32_t width = n / samples;
    double pairs         = 0;
    for (size_t i = 0, j = 0; i < at.size(); i = j)
    {
      for (j = i; j < at.size() && at[j] / width == at[i] / width; ++j)
      {
      }
      pairs += 0.5 * double(j - i) * double(j - i - 1);
    }
    const double expected = 0.5 * samples;
    if (at.back() >= n || std::adjacent_find(at.begin(), at.end()) != at.end()
        || (pairs - expected) * (pairs - expected) > 25 * expected)
    {
      std::printf("places of %u: %g pairs, %g expected\n", n, pairs, expected);
      ++failures;
    }
  }
  std::printf("%d failures\n", failures);
  return failures != 0;
}
