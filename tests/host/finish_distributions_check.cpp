// finish_choose (cccl_gb300/csrc/sort_policy.h) on the CPU, on samples of keys of known distributions counted
// as finish_sample counts them: what the finish can order is partitioned, keys that cluster at every
// scale are not. Built and run by tests/test_finish_distributions.py.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <functional>
#include <initializer_list>
#include <random>
#include <unordered_map>
#include <vector>

#include "sort_policy.h"

using namespace gb300;

static std::mt19937_64 gen(20240613);

static double unit()
{
  return double(gen() >> 11) / 9007199254740992.0;
}

// Whether a sample of a sort of n keys (with 4-byte values) leads to the partition.
static bool partitions(const std::function<uint64_t()>& key, double n)
{
  const uint32_t samples = finish_sample_items((unsigned long long) n);
  const uint32_t cap     = uint32_t(finish_cap(8, 4, false));
  const double mean      = double(cap) * samples / n;
  auto heavy_size        = [](double m) {
    return uint32_t(2.0 + 1.3 * m + 4.0 * std::sqrt(m) + 0.5); // as radix_plan.cpp sets it
  };
  const uint32_t limit = heavy_size(mean), first_limit = heavy_size(mean * HISTOGRAM_LANES_TPB / samples);
  std::vector<uint64_t> keys(samples);
  for (auto& k : keys)
  {
    k = key();
  }
  unsigned long long light[MAX_PASSES] = {};
  uint32_t heavy[MAX_PASSES] = {}, partners[MAX_PASSES] = {}, paired[MAX_PASSES] = {}, trivial = 0, piece = 0;
  for (int l = 1; l <= 8; ++l)
  {
    auto group = [&](uint64_t k) {
      return k >> (64 - 8 * l);
    };
    std::unordered_map<uint64_t, uint32_t> first, all;
    uint32_t many = 0;
    for (int i = 0; i < HISTOGRAM_LANES_TPB; ++i)
    {
      ++first[group(keys[i])];
    }
    for (int i = 0; i < HISTOGRAM_LANES_TPB; ++i)
    {
      many += first[group(keys[i])] >= first_limit ? 1 : 0;
    }
    if (many > uint32_t(HISTOGRAM_LANES_TPB / 2))
    {
      heavy[l - 1] = uint32_t((unsigned long long) many * samples / HISTOGRAM_LANES_TPB);
      continue;
    }
    for (const uint64_t k : keys)
    {
      ++all[group(k)];
    }
    for (const uint64_t k : keys)
    {
      const uint32_t c = all[group(k)];
      const bool few   = c < (l == 8 ? std::min(limit, 4u) : limit);
      light[l - 1] += few ? c - 1 : 0;
      heavy[l - 1] += l == 8 ? (c < limit ? c - 1 : 0) : few ? 0 : 1;
      partners[l - 1] += c - 1;
      paired[l - 1] += c > 1 && c <= 4 ? 1 : 0;
    }
  }
  for (int q = 0; q < 8; ++q)
  {
    const bool same = std::all_of(keys.begin(), keys.end(), [&](uint64_t k) {
      return ((k ^ keys[0]) >> (8 * q) & 255u) == 0;
    });
    trivial |= same ? 1u << q : 0u;
  }
  return finish_choose(8, trivial, light, heavy, (unsigned long long) n, samples, cap, finish_cost(8, 4), PLAN_MODE_SEPARATE,
                       &piece, partners, paired)
      != 0;
}

static uint64_t bits_of(double d)
{
  uint64_t u;
  std::memcpy(&u, &d, 8);
  return u >> 63 ? ~u : u | 1ull << 63;
}

int main()
{
  std::normal_distribution<double> normal;
  struct Case
  {
    const char* name;
    std::function<uint64_t()> key;
    bool partition;
  };
  auto clump = [&](double share, uint64_t high, int low_bits) {
    return [=] {
      return unit() < share ? high << low_bits | gen() >> (64 - low_bits) : gen();
    };
  };
  const Case cases[] = {
    {"uniform", [] { return gen(); }, true},
    {"below 2^40", [] { return gen() >> 24; }, true},
    {"normal doubles", [&] { return bits_of(normal(gen)); }, true},
    {"lognormal doubles", [&] { return bits_of(std::exp(3.0 * normal(gen))); }, true},
    {"2 % in one bucket", clump(0.02, 0x1234, 48), true},
    {"5 % in a narrow range", clump(0.05, 0x123456789, 28), true},
    {"1 % in a narrow range", clump(0.01, 0x123456789, 28), true},
    {"AND of two words", [] { return gen() & gen(); }, false},
    {"AND of three words", [] { return gen() & gen() & gen(); }, false},
  };
  int failures = 0;
  for (const Case& c : cases)
  {
    for (const double n : {4.3e6, 7.4e6, 2.1e7, 6.7e7, 2.6e8})
    {
      int taken = 0;
      for (int t = 0; t < 20; ++t)
      {
        taken += partitions(c.key, n) ? 1 : 0;
      }
      if (c.partition ? taken < 18 : taken > 3)
      {
        std::printf("%s, %.2g keys: partitioned %d of 20 times\n", c.name, n, taken);
        ++failures;
      }
    }
  }
  return failures == 0 ? 0 : 1;
}
