// zsweep_pairs.cu -- the z sweep with each document's topic counts as a sorted
// list of (topic, count) pairs spread over a warp's registers (reference: the
// per-document HashMap of src/cu/hashmap.cuh:13-334 used by sample_topics,
// src/cu/topics.cu:36-105).
//
// One warp per document, 32 tokens at a time.  Before a chunk's first draw the
// list is made anew in shared memory: the topics with a count, and the topics
// that the chunk's dense draws would take, which the alias tables give before
// the draws' order matters.  A sparse draw takes a topic of the document, so no
// topic outside this list can come in during the chunk: the list stands still,
// its entries live in registers (lane l holds the l-th contiguous run, so lane
// order then slot is ascending topic order), and the gathers of q for the next
// token are issued before the current one is drawn.  Entries whose count is
// zero are not gathered, except the dense topic of the draw in flight.
//
// What bounds it: the gathers.  A document's topics lie in different sectors of
// a word's row (40 KB at K=10000), most of them in HBM: 61 sectors a token at
// 5.4 TB/s of DRAM traffic (K=10000, V=30000, 3e5 documents of 80 tokens), 225
// instructions a token, 13.7 ms.  But 7% of those entries are not zero.  FEW:
// where q does not fit L2, a bit for each of a word's topics does (38 MB for 1.2
// GB there); before a chunk's draws each lane collects its topics' bits for the
// chunk's words, many loads at a time, and only entries with mass are gathered:
// 9.5 ms, 321 instead of 1,083 bytes of DRAM traffic a token, bound by issue (60
// %) and a token's dependent steps.  (With the list in shared memory, searched
// and shifted at every draw, 430 instructions, it was 25.3 ms.)  Documents in
// device memory at K=4096 (2e4 documents of up to 5000 tokens, no lengths on the
// host), whose lists had to be sized for K entries each: an iteration of 32 ms
// now takes 12 to 15 while documents outgrow the registers (the first four of a
// chain) and 6.5 to 8 after.
//
// A list in registers holds at most kListMost entries.  A document that outgrows
// it is handed on with the token it stands at (its earlier tokens' new topics
// are in z) to a second kernel, whose lists stay in shared memory (long_chunk):
// the list standing still during a chunk, the positions of the tokens' topics
// and of their dense draws' topics are looked up before the chunk's first draw,
// a draw changes two counts in place, and each token walks the document's or its
// word's list, whichever is shorter.
#include <algorithm>
#include <cmath>

#include "../../include/gpulda.h"
#include "kernels.cuh"
#include "warp.cuh"

namespace gpulda {

namespace {

constexpr u32 kMaxDocLen = 65535u;
constexpr u32 kNone = 0xffffu;     // no topic (topics are below 32768)
constexpr u32 kSparseBit = 0x8000u;
constexpr u32 kLongAhead = 4;  // entries of a word's list that a lane reads ahead (2: up to a third slower)
// Lists in shared memory have their q values there if that leaves a block this
// many warps (three times the memory).  2,000 documents of 1,000 tokens of which
// the lengths are on the device only: 40 ms with one such warp (K=9000), 22 with
// two (K=6000), 20 and 14 with the q values loaded as they are summed and room for
// more warps; with lengths on the host and lists in shared memory for few of the
// documents the q values there save 10 % (K=6000, 18.2 for 21.3).
constexpr u32 kStagedWarps = 3;
constexpr u32 kBitsAhead = 4;  // tokens whose words' bits are loaded at a time (1: 11.3 ms, 2: 10.3, 8: 10.0)
constexpr u32 kBitsMost = 8;   // entries a lane with room for the bits in registers

// Shared memory per warp: the list (topic << 16 | count, `cap` entries), the
// positions of a merge's new entries, the chunk's staged tokens (32 bytes each,
// and one behind them), and for lists that stay there an index of the list by
// topic and, if they fit, the q values of the current token's and the next one's
// word at the list's topics.
struct WarpMem {
  u32* list;
  uint16_t* index;  // K: a topic's place in the list if it is there, else anything
  u32* q;           // 2 x cap, or null
  u32* at;
  uint4* stage;
  u32 cap;
};

// Of a list of `cap` entries; index: topics of its index (0: none).
__host__ __device__ constexpr size_t warp_mem_bytes(u32 cap, u32 index, bool with_q) {
  return (((size_t)cap * (with_q ? 12 : 4) + (size_t)index * 2 + 15) & ~(size_t)15) + 32 * 4 + 66 * 16;
}

__device__ __forceinline__ WarpMem warp_mem_at(unsigned char* base, u32 cap, bool with_q) {
  WarpMem wm;
  wm.stage = (uint4*)base;
  wm.at = (u32*)(wm.stage + 66);
  wm.list = wm.at + 32;
  wm.q = with_q ? wm.list + cap : nullptr;
  wm.index = (uint16_t*)(wm.list + (with_q ? 3 : 1) * cap);
  wm.cap = cap;
  return wm;
}

struct ListArgs {
  ModelDev m;
  ZLaunch z;
  u32 cap;       // entries of a list
  bool with_q;   // lists that stay in shared memory have their q values there
  double lg_Ka;  // lgamma(K * alpha)
  double lg_a;   // lgamma(alpha)
};

__device__ __forceinline__ u32 scan32(u32 x, u32 lane) {
#pragma unroll
  for (u32 o = 1; o < 32; o <<= 1) {
    const u32 y = __shfl_up_sync(kFullMask, x, o);
    x += lane >= o ? y : 0u;
  }
  return x;
}

// The warp's 32 keys in ascending order by lane (bitonic network).
__device__ __forceinline__ u32 sort32(u32 key, u32 lane) {
#pragma unroll
  for (u32 size = 2; size <= 32; size <<= 1) {
#pragma unroll
    for (u32 o = size >> 1; o > 0; o >>= 1) {
      const u32 other = __shfl_xor_sync(kFullMask, key, o);
      const bool low = ((lane & o) == 0) == ((lane & size) == 0 || size == 32);
      key = low ? min(key, other) : max(key, other);
    }
  }
  return key;
}

// Adds the lanes' topics (kNone: none) to the sorted list of n entries:
// `weight` per lane to the topic's count, with a new entry where there is none.
// Returns the new length; if that would pass the list's capacity, no entry is
// added and the length that was needed is returned.
static __device__ __noinline__ u32 list_merge(const WarpMem wm, u32 n, u32 topic, u32 weight, u32 lane) {
  u32* list = wm.list;
  const u32 c = sort32(topic, lane);
  const u32 prev = __shfl_up_sync(kFullMask, c, 1);
  const bool head = c != kNone && (lane == 0 || c != prev);
  const u32 heads = __ballot_sync(kFullMask, head);
  const u32 valid = __popc(__ballot_sync(kFullMask, c != kNone));
  u32 pos = 0;
  bool fresh = false;
  u32 count = 0;
  if (head) {
    const u32 later = lane == 31 ? 0u : heads >> (lane + 1);  // heads behind this one
    count = weight * ((later ? lane + (u32)__ffs((int)later) : valid) - lane);
    u32 hi = n;
    while (pos < hi) {  // first entry with a topic >= c
      const u32 mid = (pos + hi) >> 1;
      if (list[mid] >> 16 < c)
        pos = mid + 1;
      else
        hi = mid;
    }
    fresh = pos == n || list[pos] >> 16 != c;
  }
  __syncwarp();  // every lane has searched the list
  if (head && !fresh) list[pos] += count;
  __syncwarp();
  const u32 news = __ballot_sync(kFullMask, fresh);
  const u32 nn = __popc(news);
  if (n + nn > wm.cap || !nn) return n + nn;
  const u32 rank = __popc(news & ((1u << lane) - 1u));
  if (fresh) wm.at[rank] = pos;
  // An entry moves up by the number of new entries before it.  From the top
  // down, 32 entries at a time: what a round writes lies at or above what the
  // rounds after it read, and a round reads before it writes.
  for (u32 b = (n - 1) & ~31u; n && b < n; b -= 32) {
    __syncwarp();
    const u32 e = b + lane;
    const u32 v = e < n ? list[e] : 0u;
    u32 lo = 0, hi = nn;
    while (lo < hi) {  // new entries at positions <= e
      const u32 mid = (lo + hi) >> 1;
      if (wm.at[mid] <= e)
        lo = mid + 1;
      else
        hi = mid;
    }
    __syncwarp();
    if (e < n) list[e + lo] = v;
  }
  __syncwarp();
  if (fresh) list[pos + rank] = (c << 16) | count;
  __syncwarp();
  return n + nn;
}

// The draws of the chunk's nt tokens over the list of n entries, at most R per
// lane.  Drawn topics go to stage[2 j].x (kSparseBit beside them), the distinct
// topics without the token to stage[2 j].y.  The list in shared
// memory is left with the live entries; their number is returned.
template <u32 R, bool FEW>
__device__ __forceinline__ u32 list_chunk(const WarpMem& wm, const u32* __restrict__ bits, u32 stride, u32 n, u32 nt,
                                          u32 nz, u32 lane) {
  const u32 per = (n + 31) >> 5;
  constexpr bool BITS = FEW && R <= kBitsMost;
  u32 tp[R], ct[R], qn[R];
  u32 has[BITS ? R : 1];  // bit j: the topic has mass in token j's word
#pragma unroll
  for (u32 s = 0; s < R; ++s) {
    const u32 e = lane * per + s;
    const u32 v = s < per && e < n ? wm.list[e] : kNone << 16;
    tp[s] = v >> 16;
    ct[s] = v & 0xffffu;
    qn[s] = 0;
    if constexpr (BITS) has[s] = 0;
  }
  if constexpr (BITS) {
#pragma unroll(kBitsAhead)
    for (u32 j = 0; j < nt; ++j) {
      const u32* row = bits + (size_t)wm.stage[2 * j].w * stride;
#pragma unroll
      for (u32 s = 0; s < R; ++s)
        if (tp[s] != kNone) has[s] |= ((__ldg(row + (tp[s] >> 5)) >> (tp[s] & 31)) & 1u) << j;
    }
  }
  // moves a token: k in (kNone: none), z out
  auto move = [&](u32 k, u32 z) {
    int live = 0;
#pragma unroll
    for (u32 s = 0; s < R; ++s) {
      const u32 old = ct[s];
      if (tp[s] == k) ++ct[s];
      if (tp[s] == z) --ct[s];
      live += (int)min(ct[s], 1u) - (int)min(old, 1u);
    }
    nz += (u32)__reduce_add_sync(kFullMask, live);
  };
  // Staged token: topic | dense topic << 16, r0, r1, word; row of q, alpha A.
  uint4 a = wm.stage[0], b = wm.stage[1];
  auto fetch = [&](u32 pending) {
    const u32* row = (const u32*)(((u64)b.y << 32) | b.x);
#pragma unroll
    for (u32 s = 0; s < R; ++s) {
      if constexpr (BITS) {
        qn[s] = (has[s] & 1u) && (ct[s] || tp[s] == pending) ? __ldg(row + tp[s]) : 0u;
        has[s] >>= 1;
      } else if (ct[s] || (tp[s] == pending && pending != kNone)) {
        qn[s] = __ldg(row + tp[s]);
      }
    }
  };
  // (the entries of no topic have a zero count; nothing is added to or taken
  // from them: no token has that topic)
  fetch(kNone);
  move(kNone - 1u, a.x & 0xffffu);
#pragma unroll 1
  for (u32 j = 0; j < nt; ++j) {
    const u32 kd = a.x >> 16, r0 = a.y, r1 = a.z;
    const double aA = __hiloint2double((int)b.w, (int)b.z);
    u64 P[R];
    u64 x = 0;
#pragma unroll
    for (u32 s = 0; s < R; ++s) {
      x += (u64)ct[s] * qn[s];
      P[s] = x;
    }
    const bool more = j + 1 < nt;
    a = wm.stage[2 * (j + 1)];
    b = wm.stage[2 * (j + 1) + 1];
    if (more) fetch(kd);
    const u64 incl = group_scan<32>(x);
    const u64 B = __shfl_sync(kFullMask, incl, 31);
    const bool sp = sparse_test(r0, aA, B);
    u64 t = scale_u32(r1, B);
    const u32 f = __popc(__ballot_sync(kFullMask, incl <= t)) & 31u;
    t -= incl - x;
    u32 k = tp[R - 1];
#pragma unroll
    for (u32 s = R - 1; s-- > 0;)
      if (P[s] > t) k = tp[s];
    k = __shfl_sync(kFullMask, k, f);
    if (!sp) k = kd;
    if (lane == 0) {
      wm.stage[2 * j].x = k | (sp ? kSparseBit : 0u);
      wm.stage[2 * j].y = nz;
    }
    move(k, more ? a.x & 0xffffu : kNone - 1u);
  }
  // the live entries, in order
  u32 mine = 0;
#pragma unroll
  for (u32 s = 0; s < R; ++s) mine += min(ct[s], 1u);
  const u32 incl = scan32(mine, lane);
  __syncwarp();
  u32 o = incl - mine;
#pragma unroll
  for (u32 s = 0; s < R; ++s)
    if (ct[s]) wm.list[o++] = (tp[s] << 16) | ct[s];
  __syncwarp();
  return nz;
}

__device__ __forceinline__ void copy_word_async(u32* to, const u32* from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((u32)__cvta_generic_to_shared(to)), "l"(from)
               : "memory");
}

// list_chunk with the list left in shared memory, of any length.  A token's
// masses come from the shorter of two sides.  The document's: q is gathered at
// the list's topics, the next token's by asynchronous copies, so that a long
// list's gathers are all in flight at once; where there is no room for them they
// are loaded, eight at a time, as they are summed.  The word's: its list of
// nonzero q is read, the first entries of the next token's ahead, and its topics
// are looked up in the document's list through an index by topic.  Bound by the
// steps from one token to the next.  The side by length: twice or four times the
// word's entries for one of the document's 1.3 times slower (K=9000, 1,000
// documents of 2,000 tokens from a random start: 101, 133 and 138 ms).  The same
// documents with the document's side alone 165 ms; one of 13,000 tokens 203 -> 48
// (3.7 us a token), 41 of 5,000 143 -> 47.  A binary search in the list in place of
// the index: 300, 102 and 147 ms.
static __device__ __noinline__ u32 long_chunk(const WarpMem wm, const u32* q0, const u64* csr, u32 n, u32 nt, u32 nz,
                                              u32 lane) {
  u32* list = wm.list;
  uint16_t* index = wm.index;
  for (u32 e = lane; e < n; e += 32) index[list[e] >> 16] = (uint16_t)e;
  __syncwarp();
  if (lane < nt) {  // the staged topics become positions
    const u32 v = wm.stage[2 * lane].x;
    wm.stage[2 * lane].x = index[v & 0xffffu] | ((u32)index[v >> 16] << 16);
  }
  __syncwarp();
  // one token into entry `in` and one out of entry `out` (lanes 0 and 1)
  auto move = [&](bool add, u32 in, bool del, u32 out) {
    const bool act = !(add && del && in == out) && (lane == 0 ? add : lane == 1 && del);
    u32* e = list + (lane == 0 ? in : out);
    u32 c = 2;
    if (act) {
      c = *e & 0xffffu;
      *e += lane == 0 ? 1u : ~0u;
    }
    const u32 b = __ballot_sync(kFullMask, c == lane);  // lane 0: the count was 0; lane 1: it was 1
    nz += (b & 1u) - ((b >> 1) & 1u);
    __syncwarp();
  };
  auto row_of = [&](u32 j) {
    const uint4 b = wm.stage[2 * j + 1];
    return (const u32*)(((u64)b.y << 32) | b.x);
  };
  auto word_side = [&](u32 nw) { return nw < n; };
  constexpr u32 U = kLongAhead;
  u64 ent[U];  // the lane's first entries of a word's list
  auto read = [&](const u64* crow, u32 e, u32 end) {
#pragma unroll
    for (u32 u = 0; u < U; ++u) ent[u] = e + u < end ? __ldg(crow + e + u) : 0ull;
  };
  // What token j needs and does not depend on the counts.  Of the list's q values
  // those of entries without a count are left out, but for the one that the draw
  // in flight may fill.
  auto fetch = [&](u32 j, u32 pending) {
    const u32* row = row_of(j);
    const u32 nw = wm.stage[2 * j].w;
    if (word_side(nw)) {
      const u32 per = (nw + 31) >> 5, e0 = min(nw, lane * per);
      read(csr + (row - q0), e0, min(nw, e0 + per));
    } else if (wm.q) {
      u32* q = wm.q + (j & 1) * wm.cap;
      for (u32 e = lane; e < n; e += 32) {
        const u32 v = list[e];
        if ((v & 0xffffu) || e == pending) copy_word_async(q + e, row + (v >> 16));
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
  };
  // an entry of a word's list: its topic's place in the document's, and its mass
  // (a topic that is not there has any place)
  auto look_up = [&](u64 en, u32* at) {
    const u32 p = index[(u32)en & 0xffffu], v = p < n ? list[p] : 0u;
    *at = p;
    return v >> 16 == ((u32)en & 0xffffu) ? (u64)(v & 0xffffu) * (u32)(en >> 32) : 0ull;
  };
  fetch(0, n);
  __syncwarp();  // every lane has read the list before the move writes it
  move(false, 0, true, wm.stage[0].x & 0xffffu);
  for (u32 j = 0; j < nt; ++j) {
    const uint4 a = wm.stage[2 * j], b = wm.stage[2 * j + 1];
    const double aA = __hiloint2double((int)b.w, (int)b.z);
    const u32* row = row_of(j);
    const bool more = j + 1 < nt;
    u32 pos = a.x >> 16;
    bool sp;
    if (word_side(a.w)) {
      const u64* crow = csr + (row - q0);
      const u32 nw = a.w, per = (nw + 31) >> 5, e0 = min(nw, lane * per), e1 = min(nw, e0 + per);
      u64 P[U];  // sums over the lane's first entries
      u32 at[U];
      u64 x = 0;
#pragma unroll
      for (u32 u = 0; u < U; ++u) P[u] = x += look_up(ent[u], at + u);
      for (u32 e = e0 + U; e < e1; e += U) {
        read(crow, e, e1);
        u32 other;
#pragma unroll
        for (u32 u = 0; u < U; ++u) x += look_up(ent[u], &other);
      }
      __syncwarp();
      if (more) fetch(j + 1, pos);
      const u64 incl = group_scan<32>(x);
      const u64 B = __shfl_sync(kFullMask, incl, 31);
      sp = sparse_test(a.y, aA, B);
      if (sp) {
        u64 t = scale_u32(a.z, B);
        const u32 f = __popc(__ballot_sync(kFullMask, incl <= t)) & 31u;
        t -= __shfl_sync(kFullMask, incl - x, f);
        if (per <= U) {
          u32 p = at[U - 1];
#pragma unroll
          for (u32 u = U - 1; u-- > 0;)
            if (P[u] > t) p = at[u];
          pos = __shfl_sync(kFullMask, p, f);
        } else {  // the crossing lane's run, 32 entries at a time
          const u32 f1 = min(nw, f * per + per);
          for (u32 e = f * per; e < f1; e += 32) {
            u32 p;
            const u64 in2 = group_scan<32>(look_up(e + lane < f1 ? __ldg(crow + e + lane) : 0ull, &p));
            const u64 all = __shfl_sync(kFullMask, in2, 31);
            if (all > t) {
              pos = __shfl_sync(kFullMask, p, __popc(__ballot_sync(kFullMask, in2 <= t)));
              break;
            }
            t -= all;
          }
        }
      }
    } else {
      const u32* q = wm.q + (j & 1) * wm.cap;
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
      if (more) fetch(j + 1, pos);
      const u32 per = (n + 31) >> 5, e0 = min(n, lane * per), e1 = min(n, e0 + per);
      u64 x = 0;
      if (wm.q) {
#pragma unroll 4
        for (u32 e = e0; e < e1; ++e) {
          const u32 c = list[e] & 0xffffu;
          if (c) x += (u64)c * q[e];
        }
      } else {
        for (u32 e = e0; e < e1; e += 8) {
          u32 v[8], y[8];
#pragma unroll
          for (u32 u = 0; u < 8; ++u) v[u] = e + u < e1 ? list[e + u] : 0u;
#pragma unroll
          for (u32 u = 0; u < 8; ++u) y[u] = v[u] & 0xffffu ? __ldg(row + (v[u] >> 16)) : 0u;
#pragma unroll
          for (u32 u = 0; u < 8; ++u) x += (u64)(v[u] & 0xffffu) * y[u];
        }
      }
      __syncwarp();
      const u64 incl = group_scan<32>(x);
      const u64 B = __shfl_sync(kFullMask, incl, 31);
      sp = sparse_test(a.y, aA, B);
      if (sp) {
        u64 t = scale_u32(a.z, B);
        const u32 f = __popc(__ballot_sync(kFullMask, incl <= t)) & 31u;
        t -= __shfl_sync(kFullMask, incl - x, f);
        // the crossing lane's run, 32 entries at a time
        const u32 f1 = min(n, f * per + per);
        for (u32 e = f * per; e < f1; e += 32) {
          const u32 v = e + lane < f1 ? list[e + lane] : 0u;
          const u32 y = v & 0xffffu ? (wm.q ? q[e + lane] : __ldg(row + (v >> 16))) : 0u;
          const u64 in2 = group_scan<32>((u64)(v & 0xffffu) * y);
          const u64 all = __shfl_sync(kFullMask, in2, 31);
          if (all > t) {
            pos = e + __popc(__ballot_sync(kFullMask, in2 <= t));
            break;
          }
          t -= all;
        }
      }
    }
    if (lane == 0) wm.stage[2 * j].x = (list[pos] >> 16) | (sp ? kSparseBit : 0u);
    if (lane == 0) wm.stage[2 * j].y = nz;
    __syncwarp();  // every lane has read the list
    move(true, pos, more, more ? wm.stage[2 * (j + 1)].x & 0xffffu : 0u);
  }
  // the live entries, in order
  u32 out = 0;
  for (u32 b = 0; b < n; b += 32) {
    const u32 v = b + lane < n ? list[b + lane] : 0u;
    const u32 live = __ballot_sync(kFullMask, (v & 0xffffu) != 0);
    __syncwarp();
    if (v & 0xffffu) list[out + __popc(live & ((1u << lane) - 1u))] = v;
    out += __popc(live);
    __syncwarp();
  }
  return nz;
}

// LONG: the documents of z.rest, from the token each stands at, lists in shared
// memory.
template <bool LL, bool LONG, bool FEW>
__global__ void __launch_bounds__(256, 2) z_sweep_pairs_kernel(ListArgs a) {
  extern __shared__ __align__(16) unsigned char zsm[];
  __shared__ unsigned long long blk_stats[4];  // tokens, documents, sparse work, sparse draws
  if (threadIdx.x < 4) blk_stats[threadIdx.x] = 0;
  __syncthreads();
  const ModelDev& m = a.m;
  const ZLaunch& p = a.z;
  const u32 lane = threadIdx.x & 31;
  const u32 K = m.K, V = m.V, stride = bits_stride(m.K);
  const bool with_q = LONG && a.with_q;
  const WarpMem wm =
      warp_mem_at(zsm + (threadIdx.x >> 5) * warp_mem_bytes(a.cap, LONG ? K : 0u, with_q), a.cap, with_q);
  const u32 n_items = LONG ? *p.n_rest : p.n_docs;
  double ll_acc = 0.0, ll_skip = 0.0;
  u32 status = 0;

  while (true) {
    u32 doc = 0;
    if (lane == 0) doc = atomicAdd(p.work, 1u);
    doc = __shfl_sync(kFullMask, doc, 0);
    if (doc >= n_items) break;
    u32 start = 0;  // the tokens before it are drawn
    if (LONG) {
      const u64 item = p.rest[doc];
      doc = (u32)item;
      start = (u32)(item >> 32);
    } else if (p.order) {
      doc = p.order[doc];
    }
    const u32 L = p.d_len[doc];
    const u64 off = p.d_idx[doc];
    if (L > kMaxDocLen) {
      status |= kStatusDocTooLong;
      continue;
    }
    if (off + L > p.n_tokens) {
      status |= kStatusDocRange;
      continue;
    }
    const u32* w = p.w + off;
    u32* z = p.z + off;
    auto word = [&](u32 base) {
      u32 x = base + lane < L ? w[base + lane] : 0u;
      if (x >= V) {
        status |= kStatusBadWord;
        x %= V;
      }
      return x;
    };
    auto topic = [&](u32 base) {
      u32 k = base + lane < L ? z[base + lane] : kNone;
      if (base + lane < L && k >= K) {
        status |= kStatusBadTopic;
        k %= K;
      }
      return k;
    };
    // the words of the first chunks are on their way while the list is built
    // (word data two chunks ahead, alias entries and topics one ahead)
    u32 w1 = word(start), w2 = word(start + 32), w3 = word(start + 64);
    u32 nw1 = __ldg(m.nnz + w1), nw2 = __ldg(m.nnz + w2);
    u64 A1 = __ldg(m.A + w1), A2 = __ldg(m.A + w2);
    u32 n = 0;
    for (u32 base = 0; base < L && n <= a.cap; base += 32) n = list_merge(wm, n, topic(base), 1u, lane);
    u32 nz = n, work = 0, n_sparse = 0;
    // the first chunk's topics, Philox words and alias entries
    u32 z1 = topic(start);
    U4 r = draw4(p.tok_base + off + start + lane, p.t, kStreamZ, 0, m.key0, m.key1);
    auto alias = [&](u32 base, u32 wd, u32 nw, u32 r2) {
      return base + lane < L && nw ? __ldg(m.al + (u64)wd * K + (u32)(((u64)r2 * nw) >> 32)) : 0ull;
    };
    u64 al = alias(start, w1, nw1, r.z);
    bool over = n > a.cap;
    while (!over && start < L) {
      const u32 base = start, nt = min(32u, L - base);
      const bool valid = lane < nt;
      // a word whose every q is zero keeps the token's topic: nothing else has
      // mass, and its dense draw is that topic
      const u32 kd = !valid ? kNone : nw1 ? alias_pick(al, r.w) : z1;
      n = list_merge(wm, nz, kd, 0u, lane);
      if (n > a.cap) {
        over = true;
        break;
      }
      const u64 my_row = (u64)w1 * K;
      const u32 my_nw = nw1;
      {
        const u64 aA = (u64)__double_as_longlong(__dmul_rn((double)m.alpha, exact_double(A1)));
        const u64 row = (u64)(m.q + my_row);
        wm.stage[2 * lane] = make_uint4(z1 | (kd << 16), r.x, r.y, LONG ? my_nw : w1);
        wm.stage[2 * lane + 1] = make_uint4((u32)row, (u32)(row >> 32), (u32)aA, (u32)(aA >> 32));
      }
      __syncwarp();
      // the chunks ahead
      w1 = w2;
      nw1 = nw2;
      A1 = A2;
      z1 = topic(base + 32);
      r = draw4(p.tok_base + off + base + 32 + lane, p.t, kStreamZ, 0, m.key0, m.key1);
      al = alias(base + 32, w1, nw1, r.z);
      w2 = w3;
      nw2 = __ldg(m.nnz + w2);
      A2 = __ldg(m.A + w2);
      w3 = word(base + 96);
      const u32 per = (n + 31) >> 5;
      if (LONG)
        n = long_chunk(wm, m.q, m.csr, n, nt, nz, lane);
      else if (per <= 2)
        n = list_chunk<2, FEW>(wm, m.bits, stride, n, nt, nz, lane);
      else if (per == 3)
        n = list_chunk<3, FEW>(wm, m.bits, stride, n, nt, nz, lane);
      else if (per == 4)
        n = list_chunk<4, FEW>(wm, m.bits, stride, n, nt, nz, lane);
      else if (per <= 6)
        n = list_chunk<6, FEW>(wm, m.bits, stride, n, nt, nz, lane);
      else if (per <= 8)
        n = list_chunk<8, FEW>(wm, m.bits, stride, n, nt, nz, lane);
      else
        n = list_chunk<16, FEW>(wm, m.bits, stride, n, nt, nz, lane);
      nz = n;
      const u32 res = wm.stage[2 * lane].x, my_nz = wm.stage[2 * lane].y;
      const u32 new_z = res & 0x7fffu;
      const bool sp = valid && (res & kSparseBit);
      work += __reduce_add_sync(kFullMask, valid ? min(my_nz, my_nw) : 0u);
      n_sparse += __popc(__ballot_sync(kFullMask, sp));
      if (valid) {
        z[base + lane] = new_z;
        atomicAdd(m.n + my_row + new_z, 1u);
        if (LL) {  // log Phi[new topic][word], one token per lane
          const u32 qk = __ldg(m.q + my_row + new_z);
          if (qk)
            ll_acc += log((double)qk) - 22.18070977791825;  // 32 log 2
          else
            ll_skip += 1.0;
        }
      }
      start = base + nt;
      __syncwarp();
    }
    if (lane == 0) {
      atomicAdd(blk_stats + 2, (unsigned long long)work);
      atomicAdd(blk_stats + 3, (unsigned long long)n_sparse);
    }
    if (over) {  // the rest of the document is the other kernel's (whose lists are long enough)
      if (LONG)
        status |= kStatusListFull;
      else if (lane == 0)
        p.rest[atomicAdd(p.n_rest, 1u)] = (u64)start << 32 | doc;
      __syncwarp();
      continue;
    }
    if (lane == 0 && p.K_d) p.K_d[doc] = nz;
    if (LL) {
      double dl = 0.0;
      for (u32 e = lane; e < nz; e += 32) dl += lgamma((double)m.alpha + (double)(wm.list[e] & 0xffffu)) - a.lg_a;
      dl = warp_sum_f64(dl);
      if (lane == 0) ll_acc += dl + a.lg_Ka - lgamma((double)K * (double)m.alpha + (double)L);
    }
    if (lane == 0) {
      atomicAdd(blk_stats + 0, (unsigned long long)L);
      atomicAdd(blk_stats + 1, 1ull);
    }
    __syncwarp();
  }
  if (LL) {
    ll_acc = warp_sum_f64(ll_acc);
    ll_skip = warp_sum_f64(ll_skip);
    if (lane == 0) {
      atomicAdd(p.ll, ll_acc);
      atomicAdd(p.ll + 1, ll_skip);
    }
  }
  status = __reduce_or_sync(kFullMask, status);
  if (lane == 0 && status) atomicOr(p.status, status);
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(p.counters + kCtrTokens, blk_stats[0]);
    atomicAdd(p.counters + kCtrDocs, blk_stats[1]);
    atomicAdd(p.counters + kCtrSparseWork, blk_stats[2]);
    atomicAdd(p.counters + kCtrSparseDraws, blk_stats[3]);
  }
}

template <bool LONG, bool FEW>
void launch_lists(const ModelDev& m, const ZLaunch& z, cudaStream_t s, u32 cap) {
  if (!z.n_docs) return;
  ListArgs a;
  a.m = m;
  a.z = z;
  a.cap = cap;
  a.lg_a = std::lgamma((double)m.alpha);
  a.lg_Ka = std::lgamma((double)m.K * (double)m.alpha);
  auto kern = (z.flags & kZFlagLoglik) && z.ll ? z_sweep_pairs_kernel<true, LONG, FEW>
                                                   : z_sweep_pairs_kernel<false, LONG, FEW>;
  constexpr size_t kBudget = 200 * 1024;
  static_assert(warp_mem_bytes(GPULDA_MAX_K + 32, GPULDA_MAX_K, false) <= kBudget, "a list of every topic fits");
  const u32 index = LONG ? m.K : 0u;
  a.with_q = LONG && kStagedWarps * warp_mem_bytes(cap, index, true) <= kBudget;
  const size_t per_warp = warp_mem_bytes(cap, index, a.with_q);
  const u32 warps = (u32)std::min<size_t>(8, kBudget / per_warp);
  const size_t smem = warps * per_warp;
  if (smem > 47 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBudget);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * warps, smem);
  if (per_sm < 1) per_sm = 1;
  const u32 blocks = std::min<u32>((u32)(device_sm_count() * per_sm), (z.n_docs + warps - 1) / warps);
  kern<<<blocks, 32 * warps, smem, s>>>(a);
}

}  // namespace

void launch_z_sweep_pairs(const ModelDev& m, const ZLaunch& z, cudaStream_t s) {
  // The words' bits where q is in HBM (m.bits) and the sweep is bound by it: 8
  // documents for each of the GPU's warps.  With 7,900 documents of 110 tokens
  // (K=3683) their loads only made the documents' chains longer: 1.78 -> 1.9 ms.
  if (m.bits && z.n_docs >= 8u * 16u * (u32)device_sm_count())
    launch_lists<false, true>(m, z, s, kListMost);
  else
    launch_lists<false, false>(m, z, s, kListMost);
}

void launch_z_sweep_rest(const ModelDev& m, const ZLaunch& z, cudaStream_t s, u32 lmax) {
  launch_lists<true, false>(m, z, s, std::min(std::max(lmax, 1u), m.K) + 32);
}

}  // namespace gpulda
