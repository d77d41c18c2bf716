// Sort of a short array by one thread-block cluster: the keys (and values) stay in the CTAs'
// registers and shared memory from the first load to the last store, and the digit passes
// exchange them through distributed shared memory.
//
// CTA b holds items [b * tile, (b + 1) * tile) of the current order; inside it, warp by warp, item
// i of a lane is 32 after item i - 1, so (CTA, warp, item, lane) order is source order. A pass
//   1. ranks each key among the keys of its warp with the same digit and counts the warp's
//      digits (ballots; the counts are the running offsets, so one walk gives both),
//   2. sums the counts over the warps and sends the CTA's 256 totals to every CTA,
//   3. orders the CTA's items by digit in its own shared memory while the totals travel,
//   4. after a cluster barrier adds the totals of lower digits and of the same digit in CTAs before,
//      and sends each digit's run to the CTAs that now own its places (the last pass: to the
//      output), whole warps to consecutive places; after a second barrier every CTA reloads its own.
// A pass in which all keys share the digit moves nothing.
//
// What bounds it: latency, about 3 us a pass for two cluster barriers, the exchange of totals and
// five barriers of the CTA, and from 2^15 items the ranking and the bytes sent. One launch takes
// the place of six to ten, whose starts and look-back chains are most of a short sort's time: a
// sort of 8000 u32 keys takes 16 us instead of 42, 50000 keys 25 instead of 42, 8000 u64+u32 pairs
// 35 instead of 75. Sending items straight from the registers, each to a place of its own, took
// 55 us instead of 45 at 10^5 f32+u32 pairs and 121 instead of 79 with u64 keys.
#pragma once

#include "sort_policy.h"
#include "tile_rank.cuh"

namespace gb300
{

__device__ __forceinline__ uint32_t cluster_cta_rank()
{
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ void cluster_arrive()
{
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}

__device__ __forceinline__ void cluster_wait()
{
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The same shared-memory location in CTA `rank` of the cluster.
template <class T>
__device__ __forceinline__ T* in_cta(T* local, uint32_t rank)
{
  uint64_t a;
  asm("mapa.u64 %0, %1, %2;" : "=l"(a) : "l"(local), "r"(rank));
  return reinterpret_cast<T*>(a);
}

template <int KB, int VB, int FP>
__device__ __forceinline__ void cluster_sort_body(const ClusterSortParams& p)
{
  using U             = typename uint_of<KB>::type;
  using V             = typename value_word<VB>::type;
  constexpr int TPB   = CLUSTER_TPB;
  constexpr int NW    = TPB / 32;
  constexpr int R     = RADIX_DIGITS;
  constexpr int G     = TPB / R; // groups of one thread per digit
  constexpr int C     = CLUSTER_CTAS;
  constexpr int ITEMS = cluster_items(KB, VB); // at most, per thread
  static_assert(TPB % R == 0 && NW % G == 0 && C % G == 0, "groups share the rows and the CTAs evenly");

  if (!gate_open(p.gate))
  {
    return; // uniform over the grid
  }
  extern __shared__ __align__(128) unsigned char smem[];
  uint32_t* whist     = reinterpret_cast<uint32_t*>(smem); // [NW][R]
  uint32_t* totals    = whist + NW * R;                    // [2][C][R], by pass parity
  uint32_t* part      = totals + 2 * C * R;                // [G][R]
  uint32_t* lstart    = part + G * R;                      // [R] first item of a digit in the CTA's order
  uint32_t* delta     = lstart + R;                        // [R] place of an item minus its place in the CTA's order
  uint32_t* scratch   = delta + R;                         // [16]
  const uint32_t ipt  = p.items_per_thread;
  const uint32_t tile = ipt * TPB;
  U* kbuf             = reinterpret_cast<U*>(scratch + 16); // the CTA's items between two passes
  U* kstage           = kbuf + tile;                        // ordered by digit
  V* vbuf             = reinterpret_cast<V*>(kstage + tile);
  V* vstage           = vbuf + tile;

  const int tid       = threadIdx.x;
  const int lane      = tid & 31;
  const int warp      = tid >> 5;
  const int digit     = tid & (R - 1); // of the thread in its group
  const int group     = tid / R;
  const uint32_t me   = cluster_cta_rank();
  const uint32_t n    = p.num_items;
  const uint32_t mine = min(n - min(n, me * tile), tile); // items of this CTA, the same in every pass
  const uint32_t le   = lanemask_le();
  const uint32_t slot = uint32_t(warp) * 32u * ipt + uint32_t(lane); // of item 0 in the CTA's tile
  cluster_arrive(); // waited for before the first store to another CTA: all of them have started

  U keys[ITEMS];
  V vals[VB > 0 ? ITEMS : 1];
  uint32_t pos[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
  {
    const uint32_t s = slot + 32u * i;
    keys[i]          = uint32_t(i) < ipt && s < mine ? static_cast<const U*>(p.keys_in)[me * tile + s] : U(0);
  }
  if constexpr (VB > 0)
  {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
    {
      const uint32_t s = slot + 32u * i;
      if (uint32_t(i) < ipt && s < mine)
      {
        vals[i] = static_cast<const V*>(p.values_in)[me * tile + s];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
  {
    keys[i] = encode_key<U>(keys[i], p.codec);
  }
  if (me == 0 && tid == 0)
  {
    *p.status = 0u;
  }

  uint32_t parity = 0;
  for (int bit = p.begin_bit; bit < p.end_bit; bit += RADIX_BITS)
  {
    const bool last      = bit + RADIX_BITS >= p.end_bit;
    const uint32_t dmask = (1u << min(RADIX_BITS, p.end_bit - bit)) - 1u;
    // ---- 1. ranks within the warp, the warp's counts ----
    uint32_t* row = whist + warp * R;
#pragma unroll
    for (int k = 0; k < R / 32; ++k)
    {
      row[lane + 32 * k] = 0u;
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
    {
      if (uint32_t(i) < ipt)
      {
        const bool valid      = slot + 32u * i < mine;
        const uint32_t d      = extract_digit<U, FP>(keys[i], bit, dmask);
        const uint32_t peers  = warp_match_digit(d) & __ballot_sync(0xffffffffu, valid);
        const int leader      = 31 - __clz(peers);
        const uint32_t cnt_le = __popc(peers & le);
        uint32_t b            = 0;
        if (valid && lane == leader)
        {
          b = atomicAdd(&row[d], cnt_le);
        }
        b      = __shfl_sync(0xffffffffu, b, leader & 31);
        pos[i] = b + cnt_le - 1u;
      }
    }
    __syncthreads();
    // ---- 2. the CTA's totals ----
    uint32_t rows[NW / G];
    uint32_t total = 0;
#pragma unroll
    for (int w = 0; w < NW / G; ++w)
    {
      rows[w] = whist[(group * (NW / G) + w) * R + digit];
      total += rows[w];
    }
    part[tid] = total;
    if (bit == p.begin_bit)
    {
      cluster_wait();
    }
    __syncthreads();
    uint32_t before = 0;
    total           = 0;
#pragma unroll
    for (int g = 0; g < G; ++g)
    {
      const uint32_t t = part[g * R + digit];
      before += g < group ? t : 0u;
      total += t;
    }
#pragma unroll
    for (int c = 0; c < C / G; ++c)
    {
      *in_cta(totals + (parity * C + me) * R + digit, uint32_t(group * (C / G) + c)) = total;
    }
    cluster_arrive();
    // ---- 3. the CTA's items by digit ----
#pragma unroll
    for (int w = 0; w < NW / G; ++w)
    {
      whist[(group * (NW / G) + w) * R + digit] = before;
      before += rows[w];
    }
    if (tid < R)
    {
      lstart[tid] = digit_exclusive_scan<R>(total, scratch, tid);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
    {
      if (uint32_t(i) < ipt && slot + 32u * i < mine)
      {
        const uint32_t d = extract_digit<U, FP>(keys[i], bit, dmask);
        const uint32_t s = min(lstart[d] + row[d] + pos[i], tile - 1u);
        kstage[s]        = keys[i];
        if constexpr (VB > 0)
        {
          vstage[s] = vals[i];
        }
      }
    }
    cluster_wait();
    // ---- 4. places ----
    bool all = false; // this digit is every key's
    if (tid < R)
    {
      uint32_t sum = 0, below = 0;
#pragma unroll
      for (int c = 0; c < C; ++c)
      {
        const uint32_t t = totals[(parity * C + c) * R + tid];
        sum += t;
        below += uint32_t(c) < me ? t : 0u;
      }
      delta[tid] = digit_exclusive_scan<R>(sum, scratch + 8, tid) + below - lstart[tid];
      all        = sum == n;
    }
    const bool same = __syncthreads_or(all) != 0; // equal in every CTA
    parity ^= 1u;
    if (same && !last)
    {
      continue; // the next pass's totals go to the other half of the table
    }
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
    {
      const uint32_t s = uint32_t(tid + i * TPB);
      if (uint32_t(i) < ipt && s < mine)
      {
        const U k        = kstage[s];
        const uint32_t q = delta[extract_digit<U, FP>(k, bit, dmask)] + s;
        if (last)
        {
          if (q < n)
          {
            static_cast<U*>(p.keys_out)[q] = decode_key<U>(k, p.codec);
            if constexpr (VB > 0)
            {
              static_cast<V*>(p.values_out)[q] = vstage[s];
            }
          }
        }
        else
        {
          const uint32_t owner = min(__umulhi(q, p.tile_magic), uint32_t(C - 1)); // q / tile
          const uint32_t at    = min(q - owner * tile, tile - 1u);
          *in_cta(kbuf + at, owner) = k;
          if constexpr (VB > 0)
          {
            *in_cta(vbuf + at, owner) = vstage[s];
          }
        }
      }
    }
    if (!last)
    {
      cluster_arrive();
      cluster_wait();
#pragma unroll
      for (int i = 0; i < ITEMS; ++i)
      {
        if (uint32_t(i) < ipt)
        {
          keys[i] = kbuf[slot + 32u * i];
          if constexpr (VB > 0)
          {
            vals[i] = vbuf[slot + 32u * i];
          }
        }
      }
    }
  }
}

} // namespace gb300
