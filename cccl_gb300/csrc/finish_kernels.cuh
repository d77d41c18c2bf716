// Partition and finish: the plain sort of whole 4- and 8-byte keys by its top digits only.
//
// An LSD radix sort reads and writes every item once per digit. When the top P digits
// already split the keys into buckets that fit in shared memory, the remaining digits need
// no passes over memory: the P stable digit passes (the onesweep passes of those digits)
// leave the keys ordered by their top 8 P bits, and one more read and write of the items,
// a shared-memory sort of every piece, finishes the job. 2^28 u64 keys with u32 values take
// 2 passes and the finish instead of 8 passes.
//
// Whether the top digits split the keys well enough is read off a sample of at most 2^13 keys,
// counted inside the histogram kernel (finish_sample); its last CTA picks the route
// (finish_choose in sort_policy.h) and writes the pass plan: the passes of the digits below
// the partition are skipped like passes of constant digits. No host synchronisation, so the
// sort stays capturable. Then
//   * gb300_finish cuts the partitioned array into pieces at bucket starts and sorts every
//     piece of up to about 5000 items in place, a CTA a piece;
//   * gb300_finish_tail does the same for the few pieces of up to twice that or with many repeated
//     keys, and sorts larger ones by an LSD sort over their items alone. Without such pieces,
//     the usual case, it returns at once.
// Every kernel returns at once when the route is the LSD one.
//
// Stability: the partition passes are stable and the finish orders equal keys by their place
// in the piece, the rest by a stable LSD sort, so the result is the one of all the passes.
#pragma once

#include "sort_policy.h"
#include "tile_rank.cuh"

namespace gb300
{

// Low bits dropped: the bucket a key belongs to (keys are ordered by it after the partition).
template <class U, int FP>
__device__ __forceinline__ U finish_prefix(U raw, const KeyCodec& c, int shift)
{
  return U(digit_source<U, FP>(encode_key<U>(raw, c)) >> shift);
}

// ---------------------------------------------------------------------------------------
// Sample: how large the buckets of the top `level` digits are. One CTA of the histogram
// kernel per level counts the groups of equal prefixes among p.sample_items keys
// (finish_sample_place), in an open-addressing table in shared memory (word = 18 bits of a 32-bit hash
// of the prefix << 14 | count; the other 14 choose the slot).
// Written: the sum of (group size - 1) over the sampled keys of small groups, from which the
// mean bucket size follows, and the number of sampled keys in groups of at least
// p.sample_heavy keys, whose buckets the finish cannot take.
// It takes 8 us for 4096 keys, 20 us for 8192 beside the count (histogram_lanes_count): a
// shared-memory access of all its threads takes 100 clocks (a compare-and-swap 250), so a key costs
// few of them. In rounds of stores without
// compare-and-swap it took 26 us with the keys' state in registers, 23 us with it in shared memory.
// ---------------------------------------------------------------------------------------
constexpr uint32_t FINISH_NO_SLOT = 0xffffffffu;

// The choice for one set of trivial digits, by one thread.
template <int KB>
__device__ __noinline__ uint32_t finish_digits(const HistogramParams& p, uint32_t trivial_mask, uint32_t* piece)
{
  const FinishControl* f = p.finish;
  unsigned long long light[8];
  uint32_t heavy[8], partners[8], paired[8];
  for (int l = 0; l < KB; ++l)
  {
    light[l]    = __ldcg(&f->light[l]);
    heavy[l]    = __ldcg(&f->heavy[l]);
    partners[l] = __ldcg(&f->partners[l]);
    paired[l]   = __ldcg(&f->paired[l]);
  }
  return uint32_t(finish_choose(KB, trivial_mask, light, heavy, p.num_items, p.sample_items, p.finish_cap, p.finish_cost,
                                p.plan_mode, piece, partners, paired));
}

// A level is sampled: the thread that counts the last one makes the choice for no trivial digit.
template <int KB>
__device__ __forceinline__ void finish_sampled(const HistogramParams& p)
{
  __threadfence();
  if (atomicAdd(&p.finish->levels_done, 1u) + 1u == uint32_t(p.sample_levels))
  {
    __threadfence();
    uint32_t piece           = 0;
    p.finish->sampled_digits = finish_digits<KB>(p, 0u, &piece);
    p.finish->sampled_piece  = piece;
  }
}

template <int KB, int FP, int TPB>
__device__ __noinline__ void finish_sample(const HistogramParams& p, unsigned char* smem, int level)
{
  using U                = typename uint_of<KB>::type;
  const int tid          = threadIdx.x;
  const uint32_t samples = p.sample_items; // a multiple of TPB
  const uint32_t slots   = finish_sample_slots(samples);
  const int shift        = 8 * KB - 8 * level;
  const U* keys          = static_cast<const U*>(p.keys);
  uint32_t* table        = reinterpret_cast<uint32_t*>(smem);          // [slots]
  U* sampled             = reinterpret_cast<U*>(smem + 4 * size_t(slots)); // [samples], later every key's slot
  __shared__ uint32_t light_sum, heavy_sum, partners_sum, paired_sum;
  const uint32_t n = uint32_t(p.num_items); // below 2^31
  const int half   = finish_sample_half(n);
#pragma unroll 1
  for (uint32_t i = tid; i < samples; i += TPB)
  {
    const U* src = keys + finish_sample_place(i, n, half);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(sampled + i)), "l"(src), "n"(KB) : "memory");
  }
#pragma unroll 1
  for (uint32_t i = tid; i < slots / 4; i += TPB)
  {
    reinterpret_cast<uint4*>(table)[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  if (tid == 0)
  {
    light_sum    = 0u;
    heavy_sum    = 0u;
    partners_sum = 0u;
    paired_sum   = 0u;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  uint32_t limit = p.sample_heavy_first;
#pragma unroll 1
  for (uint32_t i = tid; i < samples; i += TPB)
  {
    const unsigned long long x = finish_prefix<U, FP>(sampled[i], p.codec, shift);
    // the words mixed by odd multipliers, then a 32-bit finaliser of Chris Wellons' hash-prospector list
    // (public domain): 15 2c1b3c6d 12 297a2d39 15
    uint32_t h = uint32_t(x) * 0x9e3779b1u + uint32_t(x >> 32) * 0x85ebca77u + 0x27d4eb2fu;
    h          = (h ^ (h >> 15)) * 0x2c1b3c6du;
    h          = (h ^ (h >> 12)) * 0x297a2d39u;
    h ^= h >> 15;
    const uint32_t print = h & 0xffffc000u;
    uint32_t s           = (h ^ (h >> 17)) & (slots - 1u);
    // four places, in a table half full at most: the few keys that find none count as single ones
    uint32_t slot = FINISH_NO_SLOT;
    for (int probe = 0; probe < 4; ++probe)
    {
      uint32_t w = *reinterpret_cast<volatile uint32_t*>(table + s);
      if (w == 0u)
      {
        w = atomicCAS(table + s, 0u, print | 1u);
        if (w == 0u)
        {
          slot = s;
          break;
        }
      }
      if ((w & 0xffffc000u) == print)
      {
        atomicAdd(table + s, 1u); // at most 2^13 keys
        slot = s;
        break;
      }
      s = (s + 1u) & (slots - 1u);
    }
    reinterpret_cast<uint32_t*>(sampled)[i * (KB / 4)] = slot;
    if (i < uint32_t(TPB))
    {
      // The first TPB keys (the loop's first round, of all threads): a level with most keys in
      // large groups is settled by them, and counting the others would be a long queue at few
      // counters.
      __syncthreads();
      const uint32_t many = __popc(__ballot_sync(0xffffffffu, slot != FINISH_NO_SLOT && (table[slot] & 0x3fffu) >= limit));
      if ((tid & 31) == 0)
      {
        atomicAdd(&heavy_sum, many);
      }
      __syncthreads();
      const uint32_t heavy = heavy_sum;
      if (heavy > uint32_t(TPB / 2))
      {
        if (tid == 0)
        {
          p.finish->heavy[level - 1] = uint32_t((unsigned long long) heavy * samples / TPB);
          finish_sampled<KB>(p);
        }
        __syncthreads(); // the shared memory is the histogram's again
        return;          // uniform
      }
      limit = p.sample_heavy;
    }
  }
  __syncthreads();
  uint32_t light = 0u; // groups below the limit: their sum fits
  uint32_t heavy = 0u;
  uint32_t partners = 0u, paired = 0u; // sum of (size - 1) over all keys, and keys in groups of 2 to 4
#pragma unroll 1
  for (uint32_t i = tid; i < samples; i += TPB)
  {
    const uint32_t slot = reinterpret_cast<uint32_t*>(sampled)[i * (KB / 4)];
    const uint32_t c    = slot != FINISH_NO_SLOT ? table[slot] & 0x3fffu : 1u;
    // Whole keys: a few keys that fill large groups of their own (zeros) do not matter, many keys
    // with several copies do. light: groups of 2 and 3, heavy: the other keys of all small groups
    // (what equal keys add to light at the other levels).
    const bool few = c < (level == KB ? min(limit, 4u) : limit);
    light += few ? c - 1u : 0u;
    heavy += level == KB ? (c < limit ? c - 1u : 0u) : few ? 0u : 1u;
    partners += c - 1u; // below 2^26
    paired += c > 1u && c <= 4u ? 1u : 0u;
  }
  light    = __reduce_add_sync(0xffffffffu, light);
  heavy    = __reduce_add_sync(0xffffffffu, heavy);
  partners = __reduce_add_sync(0xffffffffu, partners);
  paired   = __reduce_add_sync(0xffffffffu, paired);
  if (tid == 0)
  {
    heavy_sum = 0u;
  }
  __syncthreads();
  if ((tid & 31) == 0)
  {
    atomicAdd(&light_sum, light);
    atomicAdd(&heavy_sum, heavy);
    atomicAdd(&partners_sum, partners);
    atomicAdd(&paired_sum, paired);
  }
  __syncthreads();
  if (tid == 0)
  {
    p.finish->light[level - 1] = light_sum;
    p.finish->heavy[level - 1] = heavy_sum;
    p.finish->partners[level - 1] = partners_sum;
    p.finish->paired[level - 1]   = paired_sum;
    finish_sampled<KB>(p);
  }
  __syncthreads(); // the shared memory is the histogram's again
}

// Route of the sort, by one thread of the histogram's last CTA. Returns the digits below
// the partition as extra skippable passes (0: the LSD route). With no trivial digit the choice is
// the one that the last sampling CTA made while the others counted (finish_sampled): it takes
// 3 us, and every other CTA would wait for it here.
template <int KB>
__device__ __noinline__ uint32_t finish_route(const HistogramParams& p, uint32_t trivial_mask)
{
  FinishControl* f      = p.finish;
  uint32_t piece        = __ldcg(&f->sampled_piece);
  const uint32_t digits = trivial_mask == 0u ? __ldcg(&f->sampled_digits) : finish_digits<KB>(p, trivial_mask, &piece);
  if (digits == 0)
  {
    return 0u;
  }
  f->piece_items  = piece;
  f->num_pieces   = uint32_t((p.num_items + piece - 1) / piece);
  f->prefix_shift = uint32_t(8 * (KB - digits));
  // gallop by about the size of a bucket: large buckets go with small pieces
  f->search_step = piece < p.finish_cap / 2 ? 512u : 64u;
  f->route       = 1u;
  return (1u << (KB - digits)) - 1u;
}

// First index >= x (1 <= x < n) whose key has another prefix than the key before x, or n: the
// first bucket start at or after x, of keys ordered by prefix. Four searches a warp, one per
// group of eight lanes (those with `active`): galloping by `step` items a lane (a power of 8),
// then narrowing by 8 a round, a handful of dependent reads. Called by whole warps.
template <class U, int FP>
__device__ __forceinline__ uint32_t
finish_bucket_start(const U* keys, uint32_t n, const KeyCodec& codec, int shift, uint32_t x, uint32_t step, bool active)
{
  const int lane        = threadIdx.x & 31;
  const int sub         = lane & 7;  // lane within the group of eight
  const int gfirst      = lane & 24; // the group's first lane
  const U p0            = active ? finish_prefix<U, FP>(__ldcg(keys + x - 1u), codec, shift) : U(0);
  unsigned long long lo = x;
  unsigned long long by = step;
  bool narrowed         = !active; // the start lies in [lo, lo + by)
  do
  {
    bool other = false;
    if (!narrowed)
    {
      const unsigned long long at = lo + sub * by + (by - 1);
      other = at >= n || finish_prefix<U, FP>(__ldcg(keys + at), codec, shift) != p0;
    }
    const uint32_t votes = (__ballot_sync(0xffffffffu, other) >> gfirst) & 0xffu;
    if (!narrowed)
    {
      narrowed = votes != 0u;
      lo += narrowed ? (__ffs(votes) - 1) * by : 8 * by;
      by = narrowed ? by : 8 * by;
    }
  } while (!__all_sync(0xffffffffu, narrowed));
  while (__any_sync(0xffffffffu, active && by > 1))
  {
    const unsigned long long part = by / 8;
    bool other                    = true; // the last part is known to hold it
    if (active && by > 1 && sub < 7)
    {
      const unsigned long long at = lo + sub * part + (part - 1);
      other = at >= n || finish_prefix<U, FP>(__ldcg(keys + at), codec, shift) != p0;
    }
    const uint32_t votes = (__ballot_sync(0xffffffffu, other) >> gfirst) & 0xffu;
    if (active && by > 1)
    {
      lo += (__ffs(votes) - 1) * part;
      by = part;
    }
  }
  return uint32_t(lo < n ? lo : n);
}

// ---------------------------------------------------------------------------------------
// finish: one piece of at most CAP items per CTA at a time, sorted in shared memory.
//
// A counting sort on the keys' place in the piece's key range: thousands of equal bins between
// the first bucket's lowest and the last bucket's highest possible key. One shared atomic per key
// gives its bin and its arrival place there, and the keys are put in bin order, each as one
// 32-bit word of its place in the range (the bin and some bits more) and its index in the piece.
// What is left is the order of the few keys of every bin (finish_order). The word order is
// the key order, and the input order for equal keys; words of equal place have their whole keys
// compared. The keys and values stay where the bulk copy put them; the sorted piece is written
// out through the indices, coalesced. It replaces up to six digit passes by about the time of
// one. It is bound by instruction issue and shared-memory accesses (random ones cost about 3.5
// wavefronts each), not by HBM, so the words carry all that the ordering reads. Four-byte
// integer keys without values need no indices: the words are the keys.
//
// One warp (the last) takes the tickets, reads the piece's bounds and key range, has the next
// piece fetched into L2 while the current one is sorted, and issues its bulk copies as soon as
// the other threads are done with the buffers. Two CTAs per SM hide each other's barriers.
// ---------------------------------------------------------------------------------------
struct FinishPiece
{
  unsigned long long lo; // lowest key of the piece's range (ordering key)
  uint32_t begin;
  uint32_t items;        // 0: no more pieces
  uint32_t scale;        // (t - lo) >> shift times scale: bin in the high word, place in it in the low one
  uint32_t shift;
  uint32_t bits;         // low key bits in which keys of the piece can differ
  uint32_t prefix_shift; // low key bits its keys are not ordered by
  uint32_t exact;        // different keys differ in the top 19 bits of bin and place
};

// Knots of a large piece's bins: the prefixes at FINISH_KNOTS evenly spaced places of the piece,
// which is ordered by prefix, cut its key range into stretches of about as many keys each, and every
// stretch gets its share of the bins.
struct FinishKnot
{
  unsigned long long lo; // lowest key of the stretch
  uint32_t scale;        // as FinishPiece::scale and shift, over the stretch
  uint32_t shift;
  uint32_t first_bin;
  uint32_t bins;
};

// Shape and shared memory of the finish (LARGE: of the second launch, finish_tail).
template <int KB, int VB, bool LARGE>
struct FinishSmem
{
  using U = typename uint_of<KB>::type;
  using V = typename value_word<VB>::type;
  static constexpr int TPB   = finish_tpb(KB, VB, LARGE); // sorting threads
  static constexpr int ITEMS = FINISH_ITEMS;              // per thread
  static constexpr int CAP   = TPB * ITEMS;
  static constexpr int BINS  = finish_bins(KB, VB, LARGE);
  // low bits of a word: the item's index in the piece; the others are its place in the key range
  static constexpr int INDEX_BITS = LARGE ? 14 : 13;
  static constexpr uint32_t INDEX = (1u << INDEX_BITS) - 1u;
  static constexpr int PLACE_BITS = 32 - INDEX_BITS - 13; // of the place in the bin: a word is bin, place, index
  // four-byte integer keys without values: equal keys cannot be told apart, the words are the
  // keys (not so floating-point keys, whose zeros are equal but differ)
  static constexpr bool DIRECT = KB == 4 && VB == 0 && !LARGE;
  static constexpr size_t keys_off   = 0;
  static constexpr size_t values_off = keys_off + round16(size_t(KB) * CAP) + 16;
  static constexpr size_t bins_off   = values_off + (VB > 0 ? round16(size_t(VB) * CAP) + 16 : 0);
  static constexpr size_t words_off  = bins_off + size_t(2) * BINS;
  static constexpr size_t knots_off  = words_off + round16(size_t(4) * CAP);
  static constexpr size_t misc_off   = knots_off + (LARGE ? sizeof(FinishKnot) * FINISH_KNOTS : 0);
  static constexpr size_t bytes      = misc_off + 512;
  static_assert(values_off % 16 == 0 && bins_off % 16 == 0 && words_off % 16 == 0 && misc_off % 16 == 0,
                "bulk copies, 16-byte groups and the mbarrier");
  static_assert(CAP <= int(INDEX) && BINS <= 8192, "indices and bins fit their fields");
};

// Whole piece by LSD passes of 7 bits over its indices: for pieces whose keys crowd into few bins.
// perm: [CAP] indices, the result; counts: [NW][128] words. Called by all sorting threads.
template <int KB, int VB, int FP>
__device__ __noinline__ void finish_piece_lsd(
  const typename uint_of<KB>::type* ks, uint32_t* perm, uint32_t* counts, uint32_t* scratch8, uint32_t n, int bits)
{
  using L             = FinishSmem<KB, VB, true>;
  using U             = typename L::U;
  constexpr int TPB   = L::TPB;
  constexpr int ITEMS = L::ITEMS;
  constexpr int NW    = TPB / 32;
  constexpr int BITS  = 7;
  constexpr int R     = 1 << BITS;
  static_assert(size_t(NW) * R * 4 <= size_t(2) * L::BINS, "the counters fit in the bins");
  auto sync = [] {
    asm volatile("bar.sync 3, %0;" ::"n"(TPB) : "memory");
  };
  const int tid  = threadIdx.x;
  const int wofs = (tid >> 5) * ITEMS * 32 + (tid & 31);
  uint32_t* mine = counts + (tid >> 5) * R;
  for (int i = 0; i < ITEMS; ++i)
  {
    const uint32_t s = uint32_t(wofs + i * 32);
    if (s < n)
    {
      perm[s] = s;
    }
  }
  for (int bit = 0; bit < bits; bit += BITS)
  {
    const uint32_t mask = (1u << min(BITS, bits - bit)) - 1u;
    for (int i = tid; i < NW * R; i += TPB)
    {
      counts[i] = 0u;
    }
    sync();
    uint32_t m[ITEMS];
    U keys[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
    {
      const uint32_t s = uint32_t(wofs + i * 32);
      m[i]             = s < n ? perm[s] : 0u;
      keys[i]          = s < n ? ks[m[i]] : U(~U(0)); // padding ranks last
    }
    warp_histogram<U, FP, ITEMS>(keys, mine, bit, mask);
    sync();
    if (tid < R)
    {
      uint32_t start;
      block_digit_offsets<NW, R>(counts, scratch8, &start, tid);
    }
    sync();
    uint32_t pos[ITEMS];
    warp_rank_stable<U, FP, ITEMS, BITS>(keys, pos, mine, bit, mask);
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
    {
      if (uint32_t(wofs + i * 32) < n)
      {
        perm[pos[i]] = m[i]; // every index was read before the last barrier
      }
    }
    sync();
  }
}

// Called by one warp. A stretch's knot is repeated at every place inside its first bucket.
template <class U, int FP>
__device__ __forceinline__ void
finish_knots(FinishKnot* knots, const U* ks, uint32_t n, const KeyCodec& codec, int prefix_shift, int bins)
{
  static_assert(FINISH_KNOTS == 32, "one lane a knot");
  const int lane   = threadIdx.x & 31;
  const U lo       = U(finish_prefix<U, FP>(ks[uint32_t(lane) * n / 32u], codec, prefix_shift) << prefix_shift);
  const U top      = U(U(finish_prefix<U, FP>(ks[n - 1u], codec, prefix_shift) << prefix_shift)
                  | U((U(1) << prefix_shift) - U(1)));
  const U before   = U(__shfl_up_sync(0xffffffffu, (unsigned long long) lo, 1));
  const uint32_t starts = __ballot_sync(0xffffffffu, lane == 0 || lo != before); // first knot of every stretch
  const uint32_t upto   = 0xffffffffu >> (31 - lane);
  const uint32_t later  = starts & ~upto;
  const int from   = 31 - __clz(starts & upto);
  const int to     = later != 0u ? __ffs(later) - 1 : 32;
  const U next     = U(__shfl_sync(0xffffffffu, (unsigned long long) lo, to & 31));
  const U width    = U((to == 32 ? top : U(next - U(1))) - lo);
  const int wbits  = sizeof(U) == 8 ? 64 - __clzll((long long) width) : 32 - __clz(int(uint32_t(width)));
  FinishKnot k;
  k.lo        = lo;
  k.shift     = wbits > 32 ? uint32_t(wbits - 32) : 0u;
  k.first_bin = uint32_t(from * bins / 32);
  k.bins      = uint32_t(to * bins / 32) - k.first_bin;
  const unsigned long long range = (unsigned long long) (width >> k.shift) + 1ull; // <= 2^32
  k.scale     = uint32_t(min(((unsigned long long) k.bins << 32) / range, 0xffffffffull));
  knots[lane] = k;
}

__device__ __forceinline__ void finish_exchange(uint32_t& a, uint32_t& b)
{
  const uint32_t x = min(a, b);
  b                = max(a, b);
  a                = x;
}

// Sorts c of at most 32 * PER words in shared memory by one warp (bitonic, PER consecutive words a lane).
template <int PER>
__device__ __forceinline__ void finish_sort_window(uint32_t* w, int c = 32 * PER)
{
  const int lane = threadIdx.x & 31;
  uint32_t x[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k)
  {
    x[k] = lane * PER + k < c ? w[lane * PER + k] : 0xffffffffu;
  }
#pragma unroll 1
  for (int size = 2; size <= 32 * PER; size <<= 1)
  {
#pragma unroll 1
    for (int o = size >> 1; o >= PER; o >>= 1)
    {
#pragma unroll
      for (int k = 0; k < PER; ++k)
      {
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x[k], o / PER);
        const int at     = lane * PER + k;
        x[k]             = ((at & o) == 0) == ((at & size) == 0) ? min(x[k], y) : max(x[k], y);
      }
    }
#pragma unroll
    for (int o = PER / 2; o >= 1; o >>= 1)
    {
      if (o < size)
      {
#pragma unroll
        for (int k = 0; k < PER; ++k)
        {
          if ((k & o) == 0)
          {
            const bool up     = ((lane * PER + k) & size) == 0;
            const uint32_t lo = min(x[k], x[k | o]);
            const uint32_t hi = max(x[k], x[k | o]);
            x[k]              = up ? lo : hi;
            x[k | o]          = up ? hi : lo;
          }
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < PER; ++k)
  {
    if (lane * PER + k < c)
    {
      w[lane * PER + k] = x[k];
    }
  }
}

// Sorts words[0, c) in shared memory by one warp: a bitonic network whose merges start with the mirrored
// comparison, so that all comparisons point the same way and those with places behind c are left out.
template <class Less>
__device__ __forceinline__ void finish_sort_words(uint32_t* words, uint32_t c, Less&& less)
{
  const uint32_t lane = threadIdx.x & 31;
  auto compare        = [&](uint32_t i, uint32_t j) {
    if (j < c)
    {
      const uint32_t a = words[i], b = words[j];
      if (less(b, a))
      {
        words[i] = b;
        words[j] = a;
      }
    }
  };
#pragma unroll 1
  for (uint32_t half = 1; half < c; half <<= 1) // merges sorted blocks of `half` words
  {
#pragma unroll 1
    for (uint32_t t = lane; t < (c + half) / 2u; t += 32) // the pairs behind have a place behind c
    {
      const uint32_t o = t & (half - 1u), first = (t - o) * 2u;
      compare(first + o, first + 2u * half - 1u - o);
    }
    __syncwarp();
#pragma unroll 1
    for (uint32_t d = half >> 1; d >= 1u; d >>= 1)
    {
#pragma unroll 1
      for (uint32_t t = lane; t < c / 2u; t += 32)
      {
        const uint32_t o = t & (d - 1u), first = (t - o) * 2u;
        compare(first + o, first + o + d);
      }
      __syncwarp();
    }
  }
}

// Bit k: a run of words of one place has its second word at place k of this thread's.
template <class L>
__device__ __forceinline__ uint32_t finish_tie_starts(uint32_t n, const uint32_t* words)
{
  const uint32_t first  = threadIdx.x * L::ITEMS;
  uint32_t ties         = 0; // bit k: the thread's k-th word is like the one before it
  const uint4* group    = reinterpret_cast<const uint4*>(words + first);
  const uint32_t before = first > 0u ? words[first - 1u] : ~words[0];
  uint32_t last         = before;
#pragma unroll
  for (int g = 0; g < L::ITEMS / 4; ++g)
  {
    const uint4 x = group[g];
    ties |= (last ^ x.x) <= L::INDEX ? 1u << (4 * g) : 0u;
    ties |= (x.x ^ x.y) <= L::INDEX ? 2u << (4 * g) : 0u;
    ties |= (x.y ^ x.z) <= L::INDEX ? 4u << (4 * g) : 0u;
    ties |= (x.z ^ x.w) <= L::INDEX ? 8u << (4 * g) : 0u;
    last = x.w;
  }
  if (first + L::ITEMS > n)
  {
    ties &= (1u << (n > first ? n - first : 0u)) - 1u;
  }
  const bool joined = (ties & 1u) != 0u && first > 1u && (words[first - 2u] ^ before) <= L::INDEX;
  return ties & ~(ties << 1) & (joined ? ~1u : ~0u);
}

// End of the run that starts at `from`, if it has FINISH_RUN_MAX words at most; else a place behind those.
template <class L>
__device__ __forceinline__ uint32_t finish_tie_end(uint32_t n, const uint32_t* words, uint32_t from)
{
  uint32_t end = from + 2u;
  while (end < n && end - from <= uint32_t(FINISH_RUN_MAX) && (words[end] ^ words[from]) <= L::INDEX)
  {
    ++end;
  }
  return end;
}

// Insertion sort of words[from, end), a run, by one thread: by index among equal keys, as which they come.
template <class L, int FP>
__device__ __forceinline__ void finish_insert(const typename L::U* ks, uint32_t* words, uint32_t from, uint32_t end)
{
  using U  = typename L::U;
  auto key = [&](uint32_t w) {
    return digit_source<U, FP>(ks[w & L::INDEX]);
  };
  U largest = key(words[from]);
  for (uint32_t r = from + 1u; r < end; ++r)
  {
    const uint32_t w = words[r];
    const U t        = key(w);
    if (!(t < largest))
    {
      largest = t; // of copies of one key, all the others
      continue;
    }
    uint32_t q = r;
    uint32_t o = words[r - 1u]; // the largest one's
    do
    {
      words[q] = o;
      --q;
      o = q > from ? words[q - 1u] : w;
    } while (t < key(o));
    words[q] = w;
  }
}

// Orders a run of words of one place, more than FINISH_RUN_MAX of at most `most`, by their keys, and by
// index among equal ones, as which they come. By one warp: mostly they are copies of a key, in order.
template <int KB, int VB, int FP, bool LARGE>
__device__ __forceinline__ void finish_run(const typename uint_of<KB>::type* ks, uint32_t* run, uint32_t most)
{
  using L             = FinishSmem<KB, VB, LARGE>;
  const uint32_t lane = threadIdx.x & 31;
  auto key            = [&](uint32_t w) {
    return digit_source<typename L::U, FP>(ks[w & L::INDEX]);
  };
  const uint32_t place = run[0];
  uint32_t c           = 0;
  uint32_t other       = 0;
  while (other == 0u)
  {
    const uint32_t i = c + lane;
    other            = __ballot_sync(0xffffffffu, i >= most || (run[i] ^ place) > L::INDEX);
    c += other != 0u ? uint32_t(__ffs(other)) - 1u : 32u;
  }
  bool wrong = false;
  for (uint32_t i = lane; i + 1u < c; i += 32)
  {
    wrong |= key(run[i + 1u]) < key(run[i]);
  }
  if (!__any_sync(0xffffffffu, wrong))
  {
    return;
  }
  finish_sort_words(run, c, [&](uint32_t x, uint32_t y) {
    const auto kx = key(x), ky = key(y);
    return kx < ky || (kx == ky && x < y);
  });
}

// The runs of words of one place: the whole keys decide, the index among equal ones. One thread a run; a
// warp the long ones, which only pieces with bins above FINISH_RUN_MAX (`deep`) hold. A function of its
// own for the registers of what is around it: inline, sorts of different keys took 1 % longer. 4.4 M u64
// keys, 5 % in clusters of 25 that differ in their low 21 bits: 222 us; 284 with every run by one
// thread, 257 by all digit passes. Called by all sorting threads, which have to wait for each other behind it.
template <int KB, int VB, int FP, bool LARGE>
__device__ __noinline__ void
finish_ties(const typename uint_of<KB>::type* ks, uint32_t n, uint32_t* words, bool deep)
{
  using L = FinishSmem<KB, VB, LARGE>;
  static_assert(L::ITEMS <= FINISH_RUN_MAX + 1, "at most one long run has its second word in a thread");
  const uint32_t first = threadIdx.x * L::ITEMS;
  uint32_t starts      = first < n ? finish_tie_starts<L>(n, words) : 0u;
  asm volatile("bar.sync 3, %0;" ::"n"(L::TPB) : "memory");
  uint32_t long_run = 0xffffffffu;
  while (starts != 0u)
  {
    const uint32_t from = first + uint32_t(__ffs(starts)) - 2u;
    starts &= starts - 1u;
    const uint32_t end = finish_tie_end<L>(n, words, from);
    if (end - from > uint32_t(FINISH_RUN_MAX))
    {
      long_run = from;
    }
    else
    {
      finish_insert<L, FP>(ks, words, from, end);
    }
  }
  if (deep)
  {
    for (uint32_t todo = __ballot_sync(0xffffffffu, long_run != 0xffffffffu); todo != 0u; todo &= todo - 1u)
    {
      const uint32_t from = __shfl_sync(0xffffffffu, long_run, __ffs(todo) - 1);
      finish_run<KB, VB, FP, LARGE>(ks, words + from, n - from);
    }
  }
}

// The bins of more than FINISH_BIN_MAX words, which the rounds of finish_order would take too long for:
// each is sorted by the warp whose threads hold its start. Most hold many copies of one key. False, with
// nothing sorted, where a warp would have more than FINISH_CROWD_MAX words to sort: the piece is left to
// the large form. Called by all sorting threads, the words in bin order.
// 2^26 i64 keys with i32 values, 5 % of the keys 67 times each: 1.87 ms; 5.43 with those pieces left to
// the large form, 3.48 by all digit passes, 1.46 with keys that differ. Bins of 17 to 64 words stay with
// the rounds: a network each took 2.73 ms where 30 % of the keys have 20 copies, the rounds 1.97.
template <int KB, int VB, bool LARGE>
__device__ __noinline__ bool finish_crowded(uint32_t n, const uint16_t* bin16, uint32_t* words, uint32_t* scan_w)
{
  using L           = FinishSmem<KB, VB, LARGE>;
  constexpr int TPB = L::TPB;
  constexpr int NW  = TPB / 32;
  constexpr int PER = L::BINS / TPB;
  const int tid     = threadIdx.x;
  const int lane    = tid & 31;
  auto sync         = [] {
    asm volatile("bar.sync 3, %0;" ::"n"(TPB) : "memory");
  };
  auto start_of = [&](int bin) {
    return bin < L::BINS ? uint32_t(bin16[bin]) : n;
  };
  uint32_t crowd = 0; // words that this warp would have to sort
#pragma unroll 1
  for (int j = 0; j < PER; ++j)
  {
    const uint32_t c = start_of(tid * PER + j + 1) - start_of(tid * PER + j);
    crowd += c > uint32_t(FINISH_BIN_MAX) ? c : 0u;
  }
  crowd = __reduce_add_sync(0xffffffffu, crowd);
  if (lane == 0)
  {
    scan_w[tid >> 5] = crowd;
  }
  sync();
  if (__reduce_max_sync(0xffffffffu, lane < NW ? scan_w[lane] : 0u) > uint32_t(FINISH_CROWD_MAX))
  {
    return false; // uniform
  }
#pragma unroll 1
  for (int j = 0; j < PER; ++j)
  {
    const uint32_t own   = start_of(tid * PER + j);
    const uint32_t count = start_of(tid * PER + j + 1) - own;
    for (uint32_t todo = __ballot_sync(0xffffffffu, count > uint32_t(FINISH_BIN_MAX)); todo != 0u; todo &= todo - 1u)
    {
      const int src    = __ffs(todo) - 1;
      uint32_t* bin    = words + __shfl_sync(0xffffffffu, own, src);
      const uint32_t c = __shfl_sync(0xffffffffu, count, src);
      if (c <= 128u)
      {
        finish_sort_window<4>(bin, int(c));
      }
      else
      {
        finish_sort_words(bin, c, [](uint32_t x, uint32_t y) {
          return x < y;
        });
      }
    }
  }
  sync(); // the bins are in order
  return true;
}

// Bin, then PLACE_BITS bits of the place in it, of a key `above` the piece's lowest (a key outside the range, of
// a partition that failed, still gets a bin of the table).
template <class L>
__device__ __forceinline__ uint32_t finish_place(typename L::U above, uint32_t shift, uint32_t scale)
{
  const unsigned long long z = (unsigned long long) uint32_t(above >> shift) * scale;
  return min(uint32_t(z >> (32 - L::PLACE_BITS)), (uint32_t(L::BINS) << L::PLACE_BITS) - 1u);
}

// Rounds that a warp's own words need: the keys of the fullest bin among theirs that the rounds sort. Few
// warps hold a piece's fullest bins. Called by whole warps that have words, these in bin order.
template <int KB, int VB, int FP, bool LARGE>
__device__ __noinline__ uint32_t
finish_rounds(const FinishPiece* piece, uint32_t n, const uint16_t* bin16, const uint32_t* words)
{
  using L               = FinishSmem<KB, VB, LARGE>;
  using U               = typename L::U;
  constexpr bool DIRECT = L::DIRECT && FP == FP_NONE;
  const uint32_t first  = (threadIdx.x >> 5) * (32 * L::ITEMS);
  auto bin_of           = [&](uint32_t q) {
    if constexpr (DIRECT)
    {
      return finish_place<L>(U(U(words[q]) - U(piece->lo)), piece->shift, piece->scale) >> L::PLACE_BITS;
    }
    else
    {
      return words[q] >> (L::INDEX_BITS + L::PLACE_BITS);
    }
  };
  const uint32_t last = bin_of(min(first + 32u * L::ITEMS, n) - 1u);
  uint32_t own        = 0;
#pragma unroll 1
  for (uint32_t b = bin_of(first) + (threadIdx.x & 31); b <= last; b += 32)
  {
    const uint32_t c = (b + 1u < uint32_t(L::BINS) ? uint32_t(bin16[b + 1u]) : n) - bin16[b];
    own              = max(own, c > uint32_t(FINISH_BIN_MAX) ? 0u : c);
  }
  return __reduce_max_sync(0xffffffffu, own);
}

// Orders one piece, the raw keys ks[0, n) (encoded here): words[q] is left with the q-th key's
// index in its low bits, or the key itself (DIRECT). False, with nothing ordered, when bins hold more
// keys than finish_crowded takes. The bins are zero on entry and used up on return. Called
// by all sorting threads. LARGE: the bins follow the knots (finish_knots), for pieces of uneven
// density, whose keys would crowd into few equal bins.
//
// In bin order the words are sorted but for the order inside every bin, so as many
// rounds of odd-even transposition as the fullest bin has keys sort them. Every thread does
// its rounds on ITEMS consecutive words in registers (two instructions a pair; one shuffle
// each way for the pair between two lanes), a warp its stretch of 32 * ITEMS; where a bin needs more
// than FINISH_ROUNDS_SURE, every warp looks up what its own bins need (above case of 20 copies: 2.09 ms
// without; a test for order in the loop made sorts of different keys 1 % slower). Bins that
// straddle two warps' stretches are finished by sorting the 16 or 64 words on either side.
// Against letting every key count the smaller words of its bin: 2^28 u64 + u32 2.18 -> 1.62 ms.
template <int KB, int VB, int FP, bool LARGE>
__device__ __forceinline__ bool finish_order(
  const KeyCodec& codec,
  const FinishPiece* piece,
  typename uint_of<KB>::type* ks,
  const uint32_t n,
  uint32_t* bins, // two 16-bit bins a word
  uint32_t* words,
  uint32_t* scan_w,
  const FinishKnot* knots)
{
  using L               = FinishSmem<KB, VB, LARGE>;
  using U               = typename L::U;
  constexpr int TPB     = L::TPB;
  constexpr int ITEMS   = L::ITEMS;
  constexpr int NW      = TPB / 32;
  constexpr bool DIRECT = L::DIRECT && FP == FP_NONE;
  constexpr int PLACE   = L::PLACE_BITS;
  static_assert(ITEMS % 4 == 0 && ITEMS * 32 >= 64, "16-byte groups; the windows between warps do not overlap");
  static_assert(FINISH_BIN_MAX <= 64 && ITEMS * 32 >= 128, "a bin across two stretches lies in its window");
  const uint16_t* bin16 = reinterpret_cast<const uint16_t*>(bins);
  const int tid         = threadIdx.x;
  const int lane        = tid & 31;
  const int warp        = tid >> 5;
  auto sync = [] {
    asm volatile("bar.sync 3, %0;" ::"n"(TPB) : "memory");
  };
  auto order_of = [](U t) {
    return digit_source<U, FP>(t);
  };

  // ---- word and arrival place in its bin of every key ----
  uint32_t mine[ITEMS], arrival[ITEMS]; // with keys as words, the bin in arrival's high half
  {
    [[maybe_unused]] const uint32_t scale = piece->scale;
    [[maybe_unused]] const uint32_t shift = piece->shift;
    [[maybe_unused]] const U lo           = U(piece->lo);
    const bool coded     = (codec.fwd_pos | codec.fwd_neg) != 0ull; // ascending unsigned keys are their own codes
#pragma unroll
    for (int j = 0; j < ITEMS; ++j)
    {
      const uint32_t i = uint32_t(tid + j * TPB);
      if (i < n)
      {
        U t = ks[i];
        if (coded)
        {
          t     = encode_key<U>(t, codec);
          ks[i] = t;
        }
        uint32_t place;
        if constexpr (LARGE)
        {
          const U o = order_of(t);
          int s     = 0; // the last knot at or below the key
#pragma unroll
          for (int b = FINISH_KNOTS / 2; b >= 1; b >>= 1)
          {
            s += U(knots[s + b].lo) <= o ? b : 0;
          }
          const FinishKnot& k        = knots[s];
          const unsigned long long z = (unsigned long long) uint32_t(U(o - U(k.lo)) >> k.shift) * k.scale;
          place = (k.first_bin << PLACE) + min(uint32_t(z >> (32 - PLACE)), (k.bins << PLACE) - 1u);
        }
        else
        {
          place = finish_place<L>(U(order_of(t) - lo), shift, scale);
        }
        const uint32_t bin  = place >> PLACE;
        const uint32_t half = (bin & 1u) * 16u;
        arrival[j]          = (atomicAdd(bins + (bin >> 1), 1u << half) >> half) & 0xffffu;
        if constexpr (DIRECT)
        {
          mine[j] = uint32_t(t);
          arrival[j] |= bin << 16;
        }
        else
        {
          mine[j] = place << L::INDEX_BITS | i;
        }
      }
    }
  }
  sync();
  // ---- the bins' starts, and the fullest bin ----
  uint32_t fullest = 0;
  {
    constexpr int PER = L::BINS / 8 / TPB; // 16-byte groups per thread
    static_assert(PER * TPB * 8 == L::BINS, "every bin has an owner");
    uint4* bins4   = reinterpret_cast<uint4*>(bins) + tid * PER;
    uint32_t two   = 0; // sums of the low and of the high halves: fewer than 2^13 keys
    uint32_t most  = 0;
#pragma unroll
    for (int g = 0; g < PER; ++g)
    {
      const uint4 v = bins4[g];
      two += v.x + v.y + v.z + v.w;
      most = __vmaxu2(__vmaxu2(most, __vmaxu2(v.x, v.y)), __vmaxu2(v.z, v.w));
    }
    const uint32_t sum = (two & 0xffffu) + (two >> 16);
    uint32_t x         = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o)
      {
        x += y;
      }
    }
    most = __reduce_max_sync(0xffffffffu, max(most & 0xffffu, most >> 16));
    if (lane == 31)
    {
      scan_w[warp] = x | most << 16;
    }
    sync();
    const uint32_t w = lane < NW ? scan_w[lane] : 0u;
    fullest          = __reduce_max_sync(0xffffffffu, w >> 16);
    uint32_t before  = __reduce_add_sync(0xffffffffu, lane < warp ? w & 0xffffu : 0u) + x - sum;
    auto place2      = [&](uint32_t v) {
      const uint32_t low = before;
      before += v & 0xffffu;
      const uint32_t e = low | before << 16;
      before += v >> 16;
      return e;
    };
#pragma unroll
    for (int g = 0; g < PER; ++g) // read again: fewer registers held across the barrier
    {
      uint4 v  = bins4[g];
      v.x      = place2(v.x);
      v.y      = place2(v.y);
      v.z      = place2(v.z);
      v.w      = place2(v.w);
      bins4[g] = v;
    }
  }
  sync();
  // ---- the words in bin order ----
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
  {
    const uint32_t i = uint32_t(tid + j * TPB);
    if (i < n)
    {
      words[DIRECT ? bin16[arrival[j] >> 16] + (arrival[j] & 0xffffu) : bin16[mine[j] >> (L::INDEX_BITS + PLACE)] + arrival[j]] = mine[j];
    }
  }
  sync();
  if (fullest > uint32_t(FINISH_BIN_MAX) && !finish_crowded<KB, VB, LARGE>(n, bin16, words, scan_w))
  {
    return false; // uniform
  }
  // ---- sorted inside every bin ----
  uint32_t rounds       = fullest;
  const uint32_t first  = uint32_t(tid) * ITEMS; // this thread's words
  const bool warp_works = uint32_t(warp) * (32 * ITEMS) < n;
  if (fullest > uint32_t(FINISH_ROUNDS_SURE) && warp_works)
  {
    rounds = finish_rounds<KB, VB, FP, LARGE>(piece, n, bin16, words);
  }
  if (warp_works)
  {
    uint32_t v[ITEMS];
    uint4* group = reinterpret_cast<uint4*>(words + first);
#pragma unroll
    for (int g = 0; g < ITEMS / 4; ++g)
    {
      const uint4 x = group[g];
      v[4 * g]      = x.x;
      v[4 * g + 1]  = x.y;
      v[4 * g + 2]  = x.z;
      v[4 * g + 3]  = x.w;
    }
    if (first + ITEMS > n)
    {
#pragma unroll
      for (int k = 0; k < ITEMS; ++k)
      {
        v[k] = first + k < n ? v[k] : 0xffffffffu; // behind the piece: stays behind
      }
    }
    for (uint32_t r = 0; r < rounds; r += 2)
    {
#pragma unroll
      for (int k = 0; k + 1 < ITEMS; k += 2)
      {
        finish_exchange(v[k], v[k + 1]);
      }
      const uint32_t above = __shfl_down_sync(0xffffffffu, v[0], 1);
      const uint32_t below = __shfl_up_sync(0xffffffffu, v[ITEMS - 1], 1);
#pragma unroll
      for (int k = 1; k + 1 < ITEMS; k += 2)
      {
        finish_exchange(v[k], v[k + 1]);
      }
      v[ITEMS - 1] = lane == 31 ? v[ITEMS - 1] : min(v[ITEMS - 1], above);
      v[0]         = lane == 0 ? v[0] : max(v[0], below);
    }
#pragma unroll
    for (int g = 0; g < ITEMS / 4; ++g)
    {
      group[g] = make_uint4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
    }
  }
  sync();
  // ---- bins across two warps' stretches: the words on either side of the border are sorted ----
  if (warp + 1 < NW && uint32_t(warp + 1) * (32 * ITEMS) < n) // the words behind n are all ones
  {
    uint32_t* border = words + (warp + 1) * (32 * ITEMS);
    if (fullest <= 16u)
    {
      finish_sort_window<1>(border - 16);
    }
    else
    {
      finish_sort_window<4>(border - 64);
    }
  }
  sync();
  if (!DIRECT && (LARGE || piece->exact == 0u))
  {
    finish_ties<KB, VB, FP, LARGE>(ks, n, words, fullest > uint32_t(FINISH_RUN_MAX));
    sync();
  }
  return true;
}

template <int KB, int VB, int FP, bool LARGE>
__device__ __forceinline__ void finish_body(const FinishParams& p)
{
  using L             = FinishSmem<KB, VB, LARGE>;
  using U             = typename L::U;
  using V             = typename L::V;
  constexpr int TPB   = L::TPB;
  constexpr int ITEMS = L::ITEMS;
  constexpr int CAP   = L::CAP;
  constexpr bool DIRECT = L::DIRECT && FP == FP_NONE;
  static_assert(L::bytes == finish_smem_bytes(KB, VB, LARGE), "finish shared-memory layout mismatch");
  extern __shared__ __align__(128) unsigned char smem[];
  U* kst          = reinterpret_cast<U*>(smem + L::keys_off);
  V* vst          = reinterpret_cast<V*>(smem + L::values_off);
  uint32_t* bins  = reinterpret_cast<uint32_t*>(smem + L::bins_off); // two bins a word
  uint32_t* words = reinterpret_cast<uint32_t*>(smem + L::words_off);
  [[maybe_unused]] auto* knots = reinterpret_cast<FinishKnot*>(smem + L::knots_off);
  uint64_t* full  = reinterpret_cast<uint64_t*>(smem + L::misc_off);
  auto* piece     = reinterpret_cast<FinishPiece*>(smem + L::misc_off + 16);
  uint32_t* word  = reinterpret_cast<uint32_t*>(smem + L::misc_off + 16 + sizeof(FinishPiece) + 8);
  uint32_t* scan_w = word + 8; // [NW]
  // word[2]: sticky failure, [3]: the sort's status at the start

  if (!gate_open(p.gate) || __ldcg(&p.ctrl->route) == 0u || (LARGE && __ldcg(&p.ctrl->large_pieces) == 0u))
  {
    return; // uniform
  }
  const int tid  = threadIdx.x;
  const int lane = tid & 31;
  U* keys        = static_cast<U*>(p.keys);
  V* values      = static_cast<V*>(p.values);
  if (tid == 0)
  {
    mbar_init(full, 1);
    mbar_init_fence();
    word[2] = 0u;
    word[3] = load_status(p.status);
  }
  if (tid < TPB)
  {
    for (int i = tid; i < L::BINS / 8; i += TPB)
    {
      reinterpret_cast<uint4*>(bins)[i] = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  __syncthreads();
  if (word[3] != 0u)
  {
    return; // a partition that failed is not touched
  }

  if (tid >= TPB)
  {
    // ================================ the fetching warp ================================
    const uint32_t pieces = __ldcg(LARGE ? &p.ctrl->large_pieces : &p.ctrl->num_pieces);
    const uint32_t size   = __ldcg(&p.ctrl->piece_items);
    const uint32_t step0  = __ldcg(&p.ctrl->search_step);
    const int shift       = int(__ldcg(&p.ctrl->prefix_shift));
    const unsigned long long kend = (unsigned long long) p.num_items * KB;
    const unsigned long long vend = (unsigned long long) p.num_items * VB;
    // Tickets are taken for three pieces at once (one, where that would leave CTAs idle): a warp
    // searches their four ends together, and the dependent reads cost a round trip per batch.
    const uint32_t batch = LARGE ? 1u : pieces >= gridDim.x * 8u ? 3u : 1u;
    bool busy            = false; // the buffers hold a piece the other threads may still be sorting
    while (true)
    {
      uint32_t c = 0;
      if (lane == 0)
      {
        c = atomicAdd(LARGE ? &p.ctrl->large_ticket : &p.ctrl->ticket, batch);
      }
      c                  = __shfl_sync(0xffffffffu, c, 0);
      const bool done    = c >= pieces;
      uint32_t begin     = 0;
      uint32_t next      = 0;
      if constexpr (!LARGE)
      {
        // piece c: from the first bucket start at or after c * size to the next piece's
        const uint32_t e  = c + uint32_t(lane >> 3); // the group's end
        const bool search = !done && uint32_t(lane >> 3) <= batch && e >= 1u && e < pieces;
        uint32_t start    = finish_bucket_start<U, FP>(keys, p.num_items, p.codec, shift, search ? e * size : 1u, step0, search);
        start             = e == 0u ? 0u : e >= pieces ? p.num_items : start;
        begin             = __shfl_sync(0xffffffffu, start, (lane * 8) & 31);
        next              = __shfl_sync(0xffffffffu, start, (lane * 8 + 8) & 31);
      }
      const bool take    = uint32_t(lane) < batch && c + lane < pieces;
      uint32_t own_items = 0;
      FinishPiece pc{};
      if (take)
      {
        c += lane;
        if constexpr (LARGE)
        {
          begin     = __ldcg(&p.large[c].begin);
          own_items = __ldcg(&p.large[c].items);
        }
        else
        {
          own_items          = next > begin ? next - begin : 0u;
          const bool to_rest = own_items > uint32_t(FinishSmem<KB, VB, true>::CAP);
          p.rest[c]          = FinishRange{begin, 0u};
          if (to_rest)
          {
            // its last bucket alone goes to the rest: often one repeated key, in order as it is
            const U last = finish_prefix<U, FP>(__ldcg(keys + next - 1u), p.codec, shift);
            uint32_t lo = begin, hi = next - 1u; // the first key of that bucket is in [lo, hi]
            while (lo < hi)
            {
              const uint32_t mid = lo + (hi - lo) / 2u;
              const bool below   = finish_prefix<U, FP>(__ldcg(keys + mid), p.codec, shift) != last;
              lo                 = below ? mid + 1u : lo;
              hi                 = below ? hi : mid;
            }
            p.rest[c] = FinishRange{lo, next - lo};
            atomicAdd(&p.ctrl->rest_items, (unsigned long long) (next - lo));
            if (lo - begin > 1u)
            {
              p.large[atomicAdd(&p.ctrl->large_pieces, 1u)] = FinishRange{begin, lo - begin};
            }
            own_items = 0u;
          }
          else if (own_items > uint32_t(CAP))
          {
            p.large[atomicAdd(&p.ctrl->large_pieces, 1u)] = FinishRange{begin, own_items};
          }
        }
        if (own_items <= 1u || own_items > uint32_t(CAP))
        {
          own_items = 0u;
        }
        else
        {
          // the piece is ordered by prefix: its first and last keys bound the others
          const U first   = finish_prefix<U, FP>(__ldcg(keys + begin), p.codec, shift);
          const U last    = finish_prefix<U, FP>(__ldcg(keys + begin + own_items - 1u), p.codec, shift);
          const U width   = U(U(U(last - first) << shift) | U((U(1) << shift) - U(1)));
          const U apart   = U(first ^ last); // prefix bits in which its keys can differ
          const int wbits = KB == 8 ? 64 - __clzll((long long) width) : 32 - __clz(int(uint32_t(width)));
          const int abits = KB == 8 ? 64 - __clzll((long long) apart) : 32 - __clz(int(uint32_t(apart)));
          pc.lo           = U(first << shift);
          pc.begin        = begin;
          pc.items        = own_items;
          pc.bits         = uint32_t(shift + abits);
          pc.prefix_shift = uint32_t(shift);
          pc.shift        = wbits > 32 ? uint32_t(wbits - 32) : 0u;
          const unsigned long long range = (unsigned long long) (width >> pc.shift) + 1ull; // <= 2^32
          // at most one bin per key; 2^32 - 1 for ranges below the bins still tells the keys apart
          pc.scale = uint32_t(min(((unsigned long long) L::BINS << 32) / range, 0xffffffffull));
          pc.exact = pc.shift == 0u && pc.scale >= 1u << (L::INDEX_BITS + 13) ? 1u : 0u;
        }
      }
      uint32_t todo = __ballot_sync(0xffffffffu, own_items != 0u);
      while (todo != 0u || done)
      {
        const int src        = done ? 0 : __ffs(todo) - 1; // the lane that holds the piece issues it
        const uint32_t at    = __shfl_sync(0xffffffffu, pc.begin, src);
        const uint32_t items = __shfl_sync(0xffffffffu, own_items, src); // 0: no more pieces
        // 16-byte ranges that cover the piece, inside the arrays; a last range that would pass
        // the array's end stops before it, and the few items behind it are read one by one
        const unsigned long long k0 = (unsigned long long) at * KB & ~15ull;
        const unsigned long long k1 = min(((unsigned long long) (at + items) * KB + 15ull) & ~15ull, kend & ~15ull);
        const unsigned long long v0 = (unsigned long long) at * VB & ~15ull;
        const unsigned long long v1 = min(((unsigned long long) (at + items) * VB + 15ull) & ~15ull, vend & ~15ull);
        const uint32_t kbytes       = items != 0u && k1 > k0 ? uint32_t(k1 - k0) : 0u;
        const uint32_t vbytes       = items != 0u && VB > 0 && v1 > v0 ? uint32_t(v1 - v0) : 0u;
        if (lane == src)
        {
          if (kbytes != 0u)
          {
            bulk_prefetch_l2(reinterpret_cast<const unsigned char*>(keys) + k0, kbytes);
          }
          if (vbytes != 0u)
          {
            bulk_prefetch_l2(reinterpret_cast<const unsigned char*>(values) + v0, vbytes);
          }
        }
        __syncwarp();
        bool failed = false;
        if (busy)
        {
          asm volatile("bar.sync 2, %0;" ::"n"(TPB + 32) : "memory"); // the previous piece is written out
          fence_proxy_async_smem();
          failed = *reinterpret_cast<volatile uint32_t*>(word + 2) != 0u;
          if (LARGE && lane == 0)
          {
            __threadfence();
            atomicAdd(&p.ctrl->large_done, 1u);
          }
        }
        if (items == 0u || failed)
        {
          // no more pieces, or a copy failed
          if (lane == src)
          {
            *piece = FinishPiece{};
            mbar_arrive_expect_tx(full, 0u);
          }
          return;
        }
        // items behind the bulk ranges (only at the arrays' end)
        for (unsigned long long i = (k1 > k0 ? k1 : k0) / KB + lane; i < (unsigned long long) at + items; i += 32)
        {
          kst[i - k0 / KB] = __ldcg(keys + i);
        }
        if constexpr (VB > 0)
        {
          for (unsigned long long i = (v1 > v0 ? v1 : v0) / VB + lane; i < (unsigned long long) at + items; i += 32)
          {
            vst[i - v0 / VB] = values[i];
          }
        }
        __syncwarp();
        if (lane == src)
        {
          *piece = pc;
          mbar_arrive_expect_tx(full, kbytes + vbytes);
          if (kbytes != 0u)
          {
            bulk_copy_g2s(kst, reinterpret_cast<const unsigned char*>(keys) + k0, kbytes, full);
          }
          if (vbytes != 0u)
          {
            bulk_copy_g2s(vst, reinterpret_cast<const unsigned char*>(values) + v0, vbytes, full);
          }
        }
        busy = true;
        todo &= todo - 1u;
      }
    }
  }

  // ================================ the sorting threads ================================
  auto sync = [] {
    asm volatile("bar.sync 3, %0;" ::"n"(TPB) : "memory");
  };
  const bool coded = (p.codec.fwd_pos | p.codec.fwd_neg) != 0ull; // ascending unsigned keys are their own codes
  uint32_t parity  = 0;
  while (true)
  {
    const bool data_ok = mbar_wait(full, parity);
    parity ^= 1u;
    if (!data_ok)
    {
      // the copy never completed: this CTA stores nothing from here on, and the fetching warp
      // ends the loop at its next barrier
      atomicOr(p.status, STATUS_LOOKBACK_TIMEOUT);
      *reinterpret_cast<volatile uint32_t*>(word + 2) = 1u;
    }
    const uint32_t n = min(*reinterpret_cast<volatile uint32_t*>(&piece->items), uint32_t(CAP));
    if (n == 0u)
    {
      return;
    }
    const uint32_t begin = piece->begin;
    U* ks                = kst + (begin * uint32_t(KB) & 15u) / KB;
    const V* vs          = vst + (VB > 0 ? (begin * uint32_t(VB > 0 ? VB : 1) & 15u) / (VB > 0 ? VB : 1) : 0u);

    // ---- sorted order of the items; the bins are left to be cleared ----
    bool ordered;
    if constexpr (LARGE)
    {
      if (tid < 32)
      {
        finish_knots<U, FP>(knots, ks, n, p.codec, int(piece->prefix_shift), L::BINS);
      }
      sync();
      ordered = finish_order<KB, VB, FP, true>(p.codec, piece, ks, n, bins, words, scan_w, knots);
      if (!ordered)
      {
        finish_piece_lsd<KB, VB, FP>(ks, words, bins, scan_w, n, int(piece->bits));
        ordered = true;
      }
    }
    else
    {
      ordered = finish_order<KB, VB, FP, false>(p.codec, piece, ks, n, bins, words, scan_w, nullptr);
      if (!ordered && tid == 0)
      {
        p.large[atomicAdd(&p.ctrl->large_pieces, 1u)] = FinishRange{begin, n}; // the piece stays as it was
      }
    }
    for (int i = tid; i < L::BINS / 8; i += TPB)
    {
      reinterpret_cast<uint4*>(bins)[i] = make_uint4(0u, 0u, 0u, 0u); // for the next piece
    }
    sync();
    if (*reinterpret_cast<volatile uint32_t*>(word + 2) == 0u && ordered)
    {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
      {
        const uint32_t q = uint32_t(tid + j * TPB);
        if (q < n)
        {
          const uint32_t m = words[q] & L::INDEX;
          const U t        = DIRECT ? U(words[q]) : ks[m];
          __stcs(keys + begin + q, coded ? decode_key<U>(t, p.codec) : t);
          if constexpr (VB > 0)
          {
            __stcs(values + begin + q, vs[m]);
          }
        }
      }
    }
    asm volatile("bar.arrive 2, %0;" ::"n"(TPB + 32) : "memory"); // the buffers are free
  }
}

// ---------------------------------------------------------------------------------------
// rest: the pieces the finish left, as one sequence. Their key ranges are disjoint and in
// order, so the sequence sorted as a whole is the pieces sorted one by one: its items are
// gathered into one half of the free buffer, sorted there by LSD digit passes between the two
// halves, and put back. When they are more than half of the array the whole array is sorted
// instead, between its own buffer and the free one. It shares a launch with the large pieces
// (finish_tail), in phases of work (finish_phase; every wait bounded): most sorts have neither,
// and should pay one empty launch for both, not a pass sequence.
// ---------------------------------------------------------------------------------------
// Waits (bounded) until *counter reaches `target`. Called by the whole CTA.
__device__ __forceinline__ bool finish_wait_for(const uint32_t* counter, uint32_t target, uint32_t* status)
{
  __shared__ uint32_t ok;
  __syncthreads();
  if (threadIdx.x == 0)
  {
    const uint64_t start = global_timer_ns();
    bool arrived         = true;
    while (load_status(counter) < target)
    {
      __nanosleep(64);
      if (global_timer_ns() - start > gb300_wait_limit_ns)
      {
        arrived = false;
        atomicOr(status, STATUS_LOOKBACK_TIMEOUT);
        break;
      }
    }
    __threadfence();
    ok = arrived ? 1u : 0u;
  }
  __syncthreads();
  return ok != 0u;
}

// One phase of work in `units` units: every CTA takes units (body(unit)) until none is left, then
// waits for those that others took. Only units that a running CTA took are waited for, so CTAs
// that have not started yet, or never do, hold nobody up.
template <class Body>
__device__ __forceinline__ bool
finish_phase(FinishControl* ctrl, int& phase, uint32_t units, uint32_t* status, Body&& body)
{
  __shared__ uint32_t unit;
  while (true)
  {
    __syncthreads();
    if (threadIdx.x == 0)
    {
      unit = atomicAdd(&ctrl->claimed[phase], 1u);
    }
    __syncthreads();
    const uint32_t b = unit;
    if (b >= units)
    {
      break;
    }
    body(b);
    __syncthreads();
    if (threadIdx.x == 0)
    {
      __threadfence();
      atomicAdd(&ctrl->done[phase], 1u);
    }
  }
  const bool ok = finish_wait_for(&ctrl->done[phase], units, status);
  ++phase;
  return ok;
}

// Sum of v over the CTA, returned to every thread; scratch: TPB / 32 words.
template <int TPB>
__device__ __forceinline__ uint32_t finish_block_sum(uint32_t v, uint32_t* scratch)
{
  v = __reduce_add_sync(0xffffffffu, v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0)
  {
    scratch[threadIdx.x >> 5] = v;
  }
  __syncthreads();
  uint32_t sum = 0;
#pragma unroll
  for (int w = 0; w < TPB / 32; ++w)
  {
    sum += scratch[w];
  }
  return sum;
}

template <int KB, int VB, int FP>
__device__ __forceinline__ void finish_rest_body(const FinishParams& p)
{
  using U             = typename uint_of<KB>::type;
  using V             = typename value_word<VB>::type;
  constexpr int TPB   = finish_tpb(KB, VB, true) + 32; // every thread of the launch
  constexpr int ITEMS = FINISH_REST_ITEMS;
  constexpr int TILE  = TPB * ITEMS;
  constexpr int NW    = TPB / 32;
  constexpr int R     = RADIX_DIGITS;
  extern __shared__ __align__(128) unsigned char smem[];
  uint32_t* whist    = reinterpret_cast<uint32_t*>(smem); // [NW][R]
  uint32_t* place    = whist + NW * R;                    // [R] output place of every digit's next key
  uint32_t* delta    = place + R;                         // [R]
  uint32_t* scratch  = delta + R;                         // [NW]
  uint32_t* dscratch = scratch + 32;                      // [8]
  static_assert(size_t(4) * (NW * R + 2 * R + 32 + 8) <= finish_smem_bytes(KB, VB, true), "rest shared memory");
  const unsigned long long found = __ldcg(&p.ctrl->rest_items);
  if (found == 0ull)
  {
    return; // uniform over the grid: only the first launch adds to it
  }
  __syncthreads(); // the large pieces' use of shared memory is over
  if (threadIdx.x == 0)
  {
    scratch[0] = load_status(p.status);
  }
  __syncthreads();
  if (scratch[0] != 0u)
  {
    return;
  }
  __syncthreads();
  const int tid         = threadIdx.x;
  const uint32_t n      = p.num_items;
  const uint32_t pieces = __ldcg(&p.ctrl->num_pieces);
  const bool whole      = 2 * found + 64 > n;
  const uint32_t m      = whole ? n : uint32_t(found);
  // The sequence in G shares. Few items make few: the walk over the shares' digit counts costs less.
  const uint32_t G = min(min(gridDim.x, uint32_t(FINISH_MAX_CTAS)), (m + TILE - 1) / TILE);
  if (whole && !finish_wait_for(&p.ctrl->large_done, __ldcg(&p.ctrl->large_pieces), p.status))
  {
    return; // the large pieces are part of the array: all of them have to be written
  }
  // the two buffers of the passes
  U* keys   = static_cast<U*>(p.keys);
  V* values = static_cast<V*>(p.values);
  U* kbuf[2];
  V* vbuf[2];
  kbuf[0] = whole ? keys : static_cast<U*>(p.free_keys);
  vbuf[0] = whole ? values : static_cast<V*>(p.free_values);
  kbuf[1] = static_cast<U*>(p.free_keys) + (whole ? 0u : (m + 15u) & ~15u);
  vbuf[1] = static_cast<V*>(p.free_values) + (whole ? 0u : (m + 15u) & ~15u);
  const uint32_t share = (m + G - 1) / G;
  auto share_begin     = [&](uint32_t b) {
    return min(b * share, m);
  };
  int phase_no = 0;
  auto phase   = [&](auto&& body) {
    return finish_phase(p.ctrl, phase_no, G, p.status, body);
  };

  // moves a share's items between their places in the array and the sequence
  auto transfer = [&](uint32_t b, bool gather, int buffer) {
    const uint32_t v0 = share_begin(b), v1 = share_begin(b + 1u);
    uint32_t c = 0, first = 0, items = 0; // current piece: [first, first + items) of the sequence
    for (uint32_t v = v0 + tid; v < v1; v += TPB)
    {
      if (v - first >= items)
      {
        // the last piece whose offset is <= v (empty pieces share the offset of the next one)
        uint32_t lo = 0, hi = pieces;
        while (hi - lo > 1)
        {
          const uint32_t mid = lo + (hi - lo) / 2;
          if (__ldcg(p.offsets + mid) <= v)
          {
            lo = mid;
          }
          else
          {
            hi = mid;
          }
        }
        c     = lo;
        first = __ldcg(p.offsets + c);
        items = __ldcg(&p.rest[c].items);
      }
      const size_t at = size_t(__ldcg(&p.rest[c].begin)) + (v - first);
      if (v - first < items && at < n)
      {
        if (gather)
        {
          kbuf[buffer][v] = __ldcg(keys + at);
          if constexpr (VB > 0)
          {
            vbuf[buffer][v] = __ldcg(values + at);
          }
        }
        else
        {
          keys[at] = __ldcg(kbuf[buffer] + v);
          if constexpr (VB > 0)
          {
            values[at] = __ldcg(vbuf[buffer] + v);
          }
        }
      }
    }
  };

  if (!whole)
  {
    // offsets of the pieces in the sequence: sums over stretches of pieces, then their prefixes
    const uint32_t per = (pieces + G - 1) / G;
    const bool ok      = phase([&](uint32_t b) {
      const uint32_t c0 = min(b * per, pieces), c1 = min(c0 + per, pieces);
      uint32_t sum      = 0;
      for (uint32_t c = c0 + tid; c < c1; c += TPB)
      {
        sum += __ldcg(&p.rest[c].items);
      }
      sum = finish_block_sum<TPB>(sum, scratch);
      if (tid == 0)
      {
        p.table[b] = sum;
      }
    })
    && phase([&](uint32_t b) {
      const uint32_t c0 = min(b * per, pieces), c1 = min(c0 + per, pieces);
      uint32_t before   = 0;
      for (uint32_t c = tid; c < b; c += TPB)
      {
        before += __ldcg(p.table + c);
      }
      before = finish_block_sum<TPB>(before, scratch);
      for (uint32_t c = c0; c < c1; c += TPB)
      {
        const uint32_t mine = c + tid < c1 ? __ldcg(&p.rest[c + tid].items) : 0u;
        uint32_t x          = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
          const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
          if ((tid & 31) >= o)
          {
            x += y;
          }
        }
        __syncthreads();
        if ((tid & 31) == 31)
        {
          scratch[tid >> 5] = x;
        }
        __syncthreads();
        uint32_t all = 0, warps_before = 0;
        for (int w = 0; w < NW; ++w)
        {
          warps_before += w < (tid >> 5) ? scratch[w] : 0u;
          all += scratch[w];
        }
        if (c + tid < c1)
        {
          p.offsets[c + tid] = before + warps_before + x - mine;
        }
        before += all;
      }
    })
    && phase([&](uint32_t b) {
      transfer(b, true, 0);
    });
    if (!ok)
    {
      return;
    }
  }

  // digits in which two keys differ: the others need no pass
  uint32_t* bits = p.table + size_t(FINISH_MAX_CTAS) * R; // [G][KB / 4][2] bits set, bits clear in a share's keys
  if (!phase([&](uint32_t b) {
        U ones = U(0), zeros = U(0);
        const uint32_t v1 = share_begin(b + 1u);
        for (uint32_t v = share_begin(b) + tid; v < v1; v += TPB)
        {
          const U t = digit_source<U, FP>(encode_key<U>(__ldcg(kbuf[0] + v), p.codec));
          ones |= t;
          zeros |= U(~t);
        }
        if (tid < 8)
        {
          dscratch[tid] = 0u;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < KB / 4; ++j)
        {
          const uint32_t o = __reduce_or_sync(0xffffffffu, uint32_t((unsigned long long) ones >> (32 * j)));
          const uint32_t z = __reduce_or_sync(0xffffffffu, uint32_t((unsigned long long) zeros >> (32 * j)));
          if ((tid & 31) == 0)
          {
            atomicOr(&dscratch[2 * j], o);
            atomicOr(&dscratch[2 * j + 1], z);
          }
        }
        __syncthreads();
        if (tid < KB / 2)
        {
          bits[b * (KB / 2) + tid] = dscratch[tid];
        }
      }))
  {
    return;
  }
  uint32_t vary = 0;
#pragma unroll
  for (int j = 0; j < KB / 4; ++j)
  {
    uint32_t ones = 0, zeros = 0;
    for (uint32_t o = tid & 31; o < G; o += 32)
    {
      ones |= __ldcg(bits + o * (KB / 2) + 2 * j);
      zeros |= __ldcg(bits + o * (KB / 2) + 2 * j + 1);
    }
    const uint32_t both = __reduce_or_sync(0xffffffffu, ones) & __reduce_or_sync(0xffffffffu, zeros);
#pragma unroll
    for (int q = 0; q < 4; ++q)
    {
      vary |= ((both >> (8 * q)) & 255u) != 0u ? 1u << (4 * j + q) : 0u;
    }
  }
  if (vary == 0u)
  {
    return; // one key: in order as it is
  }
  if (whole && (__popc(vary) & 1) != 0)
  {
    vary |= ~vary & (vary + 1u); // one more pass: the result must be back in buffer 0
  }
  int cur = 0;
#pragma unroll 1
  for (int q = 0; q < KB; ++q)
  {
    if (((vary >> q) & 1u) == 0u)
    {
      continue;
    }
    const U* src              = kbuf[cur];
    U* dst                    = kbuf[cur ^ 1];
    const V* vsrc             = vbuf[cur];
    V* vdst                   = vbuf[cur ^ 1];
    const int bit             = q * RADIX_BITS;
    cur ^= 1;
    const bool ok = phase([&](uint32_t b) {
      for (int i = tid; i < R; i += TPB)
      {
        place[i] = 0u;
      }
      __syncthreads();
      const uint32_t v1 = share_begin(b + 1u);
      for (uint32_t v = share_begin(b) + tid; v < v1; v += TPB)
      {
        atomicAdd(&place[extract_digit<U, FP>(encode_key<U>(__ldcg(src + v), p.codec), bit, R - 1u)], 1u);
      }
      __syncthreads();
      if (tid < R)
      {
        p.table[b * R + tid] = place[tid];
      }
    })
    && phase([&](uint32_t b) {
      const uint32_t v1 = share_begin(b + 1u);
      for (int i = tid; i < NW * R; i += TPB)
      {
        whist[i] = 0u;
      }
      if (tid < R)
      {
        uint32_t total = 0, below = 0;
#pragma unroll 8
        for (uint32_t o = 0; o < G; ++o)
        {
          const uint32_t c = __ldcg(p.table + o * R + tid);
          total += c;
          below += o < b ? c : 0u;
        }
        place[tid] = digit_exclusive_scan<R>(total, dscratch, tid) + below;
      }
      __syncthreads();
      for (uint32_t t = share_begin(b); t < v1; t += TILE)
      {
        const uint32_t valid = min(uint32_t(TILE), v1 - t);
        const int wofs       = (tid >> 5) * ITEMS * 32 + (tid & 31);
        U raw[ITEMS], coded[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
        {
          const uint32_t s = uint32_t(wofs + i * 32);
          raw[i]           = s < valid ? __ldcg(src + t + s) : U(0);
          coded[i]         = s < valid ? encode_key<U>(raw[i], p.codec) : U(~U(0)); // padding ranks last
        }
        uint32_t* counts = whist + (tid >> 5) * R;
        warp_histogram<U, FP, ITEMS>(coded, counts, bit, R - 1u);
        __syncthreads();
        if (tid < R)
        {
          uint32_t start;
          const uint32_t total = block_digit_offsets<NW>(whist, dscratch, &start, tid);
          delta[tid]           = place[tid] - start;
          place[tid] += total - (tid == R - 1 ? uint32_t(TILE) - valid : 0u);
        }
        __syncthreads();
        uint32_t pos[ITEMS];
        warp_rank_stable<U, FP, ITEMS>(coded, pos, counts, bit, R - 1u);
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
        {
          const uint32_t s = uint32_t(wofs + i * 32);
          const uint32_t g = delta[extract_digit<U, FP>(coded[i], bit, R - 1u)] + pos[i];
          if (s < valid && g < m)
          {
            dst[g] = raw[i];
            if constexpr (VB > 0)
            {
              vdst[g] = __ldcg(vsrc + t + s);
            }
          }
        }
        __syncthreads();
        for (int i = tid; i < NW * R; i += TPB)
        {
          whist[i] = 0u;
        }
        __syncthreads();
      }
    });
    if (!ok)
    {
      return;
    }
  }
  if (!whole)
  {
    phase([&](uint32_t b) {
      transfer(b, false, cur);
    });
  }
}

} // namespace gb300
