// Sort of a short segment by one warp, in registers: the shortest block class of the segmented sort
// for keys of up to 4 bytes.
//
// Lane l holds elements l * E to l * E + E - 1 of a bitonic network (Batcher) of 32 * E elements, E = 4, 8 or 16
// by the segment's length. Every merge starts with the mirrored comparison (element i of a block of k
// with element k - 1 - i), so all comparisons point the same way; comparisons inside a lane are a
// minimum and a maximum, those across lanes a shuffle, a comparison and a select.
//   * integer keys alone, ordered by all their bits: the keys themselves are sorted. Equal keys are
//     the same bytes, so no stability is needed.
//   * else the elements are the digit window above the source index, in 32 bits for windows of up to 16,
//     else in 64: distinct, and in the order that stable digit passes give. The raw keys wait in
//     shared memory, the values in the input. (A window of 8 bits of 4 M f32 keys with i32 values in
//     rows of 300: 71 us, 116 with 64 bits, 108 by the one digit pass of a CTA that it takes.)
//
// What bounds it: instruction issue, 2 to 3 instructions a slot and lane for the keys themselves, no
// barrier of the CTA and no pass over shared memory but the transposition in front of the
// coalesced stores. Sixteen million i32 keys in rows of about 200: 82 us, 442 with one CTA and four
// digit passes a segment; the class's share of 2^27 f32+i32 in uneven segments: 64 us, was 116.
#pragma once

#include "radix_kernels.cuh"

namespace gb300
{

__device__ __forceinline__ long long load_offset(const void* p, unsigned long long i, int wide)
{
  return wide ? static_cast<const long long*>(p)[i] : (long long) static_cast<const int*>(p)[i];
}

// Element r of every lane with element r of the lane `mask` away (MIRRORED: with its element E - 1 - r);
// the lane with `upper` set keeps the larger ones.
template <bool MIRRORED, class T, int E>
__device__ __forceinline__ void warp_bitonic_across(T (&x)[E], int mask, bool upper)
{
#pragma unroll
  for (int r = 0; r < (MIRRORED ? E / 2 : E); ++r)
  {
    const int q = MIRRORED ? E - 1 - r : r;
    const T a   = __shfl_xor_sync(0xffffffffu, x[q], mask);
    const T b   = MIRRORED ? __shfl_xor_sync(0xffffffffu, x[r], mask) : a;
    x[r]        = (x[r] < a) != upper ? x[r] : a;
    if (MIRRORED)
    {
      x[q] = (x[q] < b) != upper ? x[q] : b;
    }
  }
}

template <class T, int E>
__device__ __forceinline__ void warp_bitonic_exchange(T (&x)[E], int r, int o)
{
  const T a = x[r], b = x[o];
  const bool less = a < b;
  x[r]            = less ? a : b;
  x[o]            = less ? b : a;
}

// Compares every element with the one J behind it in its lane, then J / 2, ... 1.
template <int J, class T, int E>
__device__ __forceinline__ void warp_bitonic_inside(T (&x)[E])
{
#pragma unroll
  for (int j = J; j >= 1; j /= 2)
  {
#pragma unroll
    for (int r = 0; r < E; ++r)
    {
      if ((r & j) == 0)
      {
        warp_bitonic_exchange(x, r, r | j);
      }
    }
  }
}

// Merges the bitonic halves of blocks of 2 * m lanes, m >= 1: elements m lanes apart, then m / 2, ... 1,
// then inside the lanes.
template <class T, int E>
__device__ __forceinline__ void warp_bitonic_merge(T (&x)[E], int m)
{
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (; m >= 1; m >>= 1)
  {
    warp_bitonic_across<false>(x, m, (lane & m) != 0);
  }
  warp_bitonic_inside<E / 2>(x);
}

// The elements of every lane: blocks of K whose halves are sorted, then of 2 K, ... E.
template <int K, class T, int E>
__device__ __forceinline__ void warp_bitonic_lane(T (&x)[E])
{
  if constexpr (K <= E)
  {
#pragma unroll
    for (int r = 0; r < E; ++r)
    {
      const int o = (r & ~(K - 1)) | (K - 1 - (r & (K - 1))); // element i with element K - 1 - i of its block
      if (r < o)
      {
        warp_bitonic_exchange(x, r, o);
      }
    }
    warp_bitonic_inside<K / 4>(x);
    warp_bitonic_lane<2 * K>(x);
  }
}

// The steps across lanes are loops. Unrolled, the networks are some 70 KB of instructions: a warp with one
// segment spent its time fetching them (one of 304 i32 keys with i64 values beside 699 of 6000: the call
// 185 us, 162 so; 155 without that segment), and rows of about 200 i32 keys took 211 us, 191 so.
template <class T, int E>
__device__ __forceinline__ void warp_bitonic_sort(T (&x)[E])
{
  const int lane = threadIdx.x & 31;
  warp_bitonic_lane<2>(x);
#pragma unroll 1
  for (int m = 1; m < 32; m <<= 1)
  {
    warp_bitonic_across<true>(x, 2 * m - 1, (lane & m) != 0);
    warp_bitonic_merge(x, m >> 1);
  }
}

// Place of element i in the warp's transposition buffer: one word of padding per 32, so lanes E
// elements apart (a power of two) and lanes one element apart both reach 32 banks.
__device__ __forceinline__ int warp_sort_slot(int i)
{
  return i + (i >> 5);
}

constexpr int WARP_SORT_MAX   = 512; // elements
constexpr int GROUP_SORT_MAX  = 4 * WARP_SORT_MAX;
constexpr int WARP_SORT_SLOTS = WARP_SORT_MAX + WARP_SORT_MAX / 32;

template <int KB>
struct WarpSortSmem
{
  union
  {
    uint32_t keys[WARP_SORT_SLOTS]; // sorted keys on their way out
    struct
    {
      uint16_t order[WARP_SORT_SLOTS]; // sorted source indices
      typename uint_of<KB>::type raw[WARP_SORT_MAX];
    } pairs;
  };
};

// Segment ordered by elements of type T: the digit window above the source index.
template <class T, int KB, int VB, int FP, int E>
__device__ __forceinline__ void warp_sort_windows(
  const typename uint_of<KB>::type* kin,
  typename uint_of<KB>::type* kout,
  const typename value_word<VB>::type* vin,
  typename value_word<VB>::type* vout,
  int n,
  int begin_bit,
  int end_bit,
  const KeyCodec& codec,
  WarpSortSmem<KB>& sh)
{
  using U              = typename uint_of<KB>::type;
  using V              = typename value_word<VB>::type;
  constexpr int SHIFT  = 4 * sizeof(T);
  const int lane       = threadIdx.x & 31;
  const uint32_t dmask = end_bit - begin_bit >= 32 ? ~0u : (1u << (end_bit - begin_bit)) - 1u;
  T x[E];
#pragma unroll
  for (int r = 0; r < E; ++r)
  {
    const int i = r * 32 + lane;
    if (i < n)
    {
      const U k          = kin[i];
      sh.pairs.raw[i]    = k;
      const uint32_t key = (uint32_t(digit_source<U, FP>(encode_key<U>(k, codec))) >> begin_bit) & dmask;
      x[r]               = T(T(key) << SHIFT) | T(i);
    }
    else
    {
      x[r] = T(~T(0)); // above every element: an index has fewer bits than the space below the key
    }
  }
  warp_bitonic_sort(x);
#pragma unroll
  for (int r = 0; r < E; ++r)
  {
    sh.pairs.order[warp_sort_slot(lane * E + r)] = uint16_t(x[r]);
  }
  __syncwarp();
  uint32_t from[E];
#pragma unroll
  for (int r = 0; r < E; ++r)
  {
    const int i = r * 32 + lane;
    from[r]     = i < n ? min(uint32_t(sh.pairs.order[warp_sort_slot(i)]), uint32_t(n - 1)) : 0u;
  }
  if constexpr (VB > 0)
  {
    // all of them before the first store: input and output may be one buffer
    V v[E];
#pragma unroll
    for (int r = 0; r < E; ++r)
    {
      v[r] = vin[from[r]];
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < E; ++r)
    {
      if (r * 32 + lane < n)
      {
        vout[r * 32 + lane] = v[r];
      }
    }
  }
#pragma unroll
  for (int r = 0; r < E; ++r)
  {
    if (r * 32 + lane < n)
    {
      kout[r * 32 + lane] = sh.pairs.raw[from[r]];
    }
  }
}

template <int KB, int VB, int FP, int E>
__device__ __forceinline__ void warp_sort_segment(
  const typename uint_of<KB>::type* kin,
  typename uint_of<KB>::type* kout,
  const typename value_word<VB>::type* vin,
  typename value_word<VB>::type* vout,
  int n,
  int begin_bit,
  int end_bit,
  const KeyCodec& codec,
  WarpSortSmem<KB>& sh)
{
  using U        = typename uint_of<KB>::type;
  const int lane = threadIdx.x & 31;
  __syncwarp(); // the previous segment's reads of sh are done
  if (VB == 0 && FP == FP_NONE && begin_bit == 0 && end_bit == 8 * KB)
  {
    uint32_t x[E];
#pragma unroll
    for (int r = 0; r < E; ++r)
    {
      const int i = r * 32 + lane;
      x[r]        = i < n ? uint32_t(encode_key<U>(kin[i], codec)) : ~0u;
    }
    warp_bitonic_sort(x);
#pragma unroll
    for (int r = 0; r < E; ++r)
    {
      sh.keys[warp_sort_slot(lane * E + r)] = x[r];
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < E; ++r)
    {
      const int i = r * 32 + lane;
      if (i < n)
      {
        kout[i] = decode_key<U>(U(sh.keys[warp_sort_slot(i)]), codec);
      }
    }
  }
  else if (KB <= 2 || end_bit - begin_bit <= 16)
  {
    warp_sort_windows<uint32_t, KB, VB, FP, E>(kin, kout, vin, vout, n, begin_bit, end_bit, codec, sh);
  }
  else
  {
    warp_sort_windows<unsigned long long, KB, VB, FP, E>(kin, kout, vin, vout, n, begin_bit, end_bit, codec, sh);
  }
}

// Integer keys alone, ordered by all their bits: a segment by a group of four warps, 32 * E elements a
// warp, warp by warp. Each warp sorts its own, then the warps merge two by two: the steps across
// warps through shared memory (each warp's part of `sh`), the rest within them. `bar` (1 or 2) is the
// group's named barrier.
template <int KB, int E>
__device__ __forceinline__ void group_sort_segment(
  const typename uint_of<KB>::type* kin,
  typename uint_of<KB>::type* kout,
  int n,
  const KeyCodec& codec,
  uint32_t (*sh)[WARP_SORT_SLOTS],
  int bar)
{
  using U          = typename uint_of<KB>::type;
  constexpr int W  = 4;
  constexpr int WE = 32 * E; // elements of a warp
  const int lane   = threadIdx.x & 31;
  const int warp   = (threadIdx.x >> 5) % W;
  auto sync        = [&]() {
    // constant barrier numbers: a number in a register claims all of the CTA's barriers
    if (bar == 1)
    {
      asm volatile("bar.sync 1, %0;" ::"n"(32 * W) : "memory");
    }
    else
    {
      asm volatile("bar.sync 2, %0;" ::"n"(32 * W) : "memory");
    }
  };
  uint32_t x[E];
#pragma unroll
  for (int r = 0; r < E; ++r)
  {
    const int i = warp * WE + r * 32 + lane;
    x[r]        = i < n ? uint32_t(encode_key<U>(kin[i], codec)) : ~0u;
  }
  warp_bitonic_sort(x);
  // element i of this warp with element i of warp `other`, or (mirrored) with element WE - 1 - i
  auto exchange = [&](int other, bool mirrored) {
#pragma unroll
    for (int r = 0; r < E; ++r)
    {
      sh[warp][warp_sort_slot(lane * E + r)] = x[r];
    }
    sync();
#pragma unroll
    for (int r = 0; r < E; ++r)
    {
      const int i      = lane * E + r;
      const uint32_t a = sh[other][warp_sort_slot(mirrored ? WE - 1 - i : i)];
      x[r]             = warp < other ? min(x[r], a) : max(x[r], a);
    }
    sync(); // before the next writes
  };
  exchange(warp ^ 1, true);
  warp_bitonic_merge(x, 16);
  exchange(warp ^ 3, true);
  exchange(warp ^ 1, false);
  warp_bitonic_merge(x, 16);
#pragma unroll
  for (int r = 0; r < E; ++r)
  {
    sh[warp][warp_sort_slot(lane * E + r)] = x[r];
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < E; ++r)
  {
    const int i = warp * WE + r * 32 + lane;
    if (i < n)
    {
      kout[i] = decode_key<U>(U(sh[warp][warp_sort_slot(r * 32 + lane)]), codec);
    }
  }
  __syncwarp();
}

// block_s with keys alone: two groups of four warps a CTA, a segment of up to 2048 keys each. The
// groups take the list's segments in fixed turns.
template <int KB, int TPB>
__device__ __forceinline__ void seg_group_body(const SegSortParams& p, const uint32_t* list, uint32_t count_index)
{
  using U              = typename uint_of<KB>::type;
  constexpr int GROUPS = TPB / 128;
  static_assert(GROUPS == 2, "named barriers 1 and 2");
  extern __shared__ __align__(128) unsigned char smem[];
  const int group      = threadIdx.x / 128;
  auto* sh             = reinterpret_cast<uint32_t(*)[WARP_SORT_SLOTS]>(smem) + 4 * group;
  const uint32_t count = p.counters[count_index];
  for (uint32_t item = blockIdx.x * GROUPS + group; item < count; item += gridDim.x * GROUPS)
  {
    const uint32_t s  = list[item];
    const long long b = load_offset(p.begin_offsets, s, p.offsets_64);
    const int n       = int(min(load_offset(p.end_offsets, s, p.offsets_64) - b, (long long) GROUP_SORT_MAX));
    const U* kin      = static_cast<const U*>(p.keys_in) + b;
    U* kout           = static_cast<U*>(p.keys_out) + b;
    if (n <= GROUP_SORT_MAX / 2)
    {
      group_sort_segment<KB, 8>(kin, kout, n, p.codec, sh, 1 + group);
    }
    else
    {
      group_sort_segment<KB, 16>(kin, kout, n, p.codec, sh, 1 + group);
    }
  }
}

// Every warp takes the list's segments in fixed turns: their lengths differ by a factor of four at
// most, and a ticket per segment would be one atomic on one address for 500 bytes of keys.
template <int KB, int VB, int FP, int TPB>
__device__ __forceinline__ void seg_warp_body(const SegSortParams& p, const uint32_t* list, uint32_t count_index)
{
  using U = typename uint_of<KB>::type;
  using V = typename value_word<VB>::type;
  __shared__ WarpSortSmem<KB> smem[TPB / 32];
  WarpSortSmem<KB>& sh = smem[threadIdx.x / 32];
  const uint32_t count = p.counters[count_index];
  const uint32_t step  = gridDim.x * (TPB / 32);
  uint32_t item        = blockIdx.x * (TPB / 32) + threadIdx.x / 32;
  long long b = 0, e = 0;
  auto segment = [&](uint32_t i) {
    if (i < count)
    {
      const uint32_t s = list[i];
      b                = load_offset(p.begin_offsets, s, p.offsets_64);
      e                = load_offset(p.end_offsets, s, p.offsets_64);
    }
  };
  segment(item);
  for (; item < count; item += step)
  {
    const long long first = b;
    const int n           = int(min(e - b, (long long) WARP_SORT_MAX));
    segment(item + step); // its offsets arrive while this one is sorted
    const U* kin = static_cast<const U*>(p.keys_in) + first;
    U* kout      = static_cast<U*>(p.keys_out) + first;
    const V* vin = VB > 0 ? static_cast<const V*>(p.values_in) + first : nullptr;
    V* vout      = VB > 0 ? static_cast<V*>(p.values_out) + first : nullptr;
    if (n <= 128)
    {
      warp_sort_segment<KB, VB, FP, 4>(kin, kout, vin, vout, n, p.begin_bit, p.end_bit, p.codec, sh);
    }
    else if (n <= 256)
    {
      warp_sort_segment<KB, VB, FP, 8>(kin, kout, vin, vout, n, p.begin_bit, p.end_bit, p.codec, sh);
    }
    else
    {
      warp_sort_segment<KB, VB, FP, 16>(kin, kout, vin, vout, n, p.begin_bit, p.end_bit, p.codec, sh);
    }
  }
}

} // namespace gb300
