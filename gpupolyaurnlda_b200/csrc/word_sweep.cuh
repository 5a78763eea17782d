// word_sweep.cuh -- the sequential topic draws of documents whose words have
// short lists of topics: documents' counts in shared memory, walks over the
// words' lists; shared by the Gibbs sweep (zsweep_words.cu) and the fold-in of
// new documents against a fixed model (serve.cu).
//
// Reference: sample_topics / count_topics / compute_product_cumsum /
// draw_wary_search / draw_alias, src/cu/topics.cu:36-105 and
// src/cu/topics.cuh:63-192.  A group of W lanes owns one document, so a warp
// advances 32/W documents in lock step; a document's counts m_d are a dense
// array of 16-bit counts.  The draw is that of doc_counts.cuh, with B and the
// prefix over the word's list of nonzero q, gathering m_dk: each lane of the
// group takes a contiguous run of the ascending list, so lane order then
// position is ascending topic order, and the masses are exact integers.
//
// Why over the words' lists only: once a chain's words have settled on some of
// the topics, their lists are as short as the documents' (mid corpus after 60
// iterations: 92 entries against 120 topics), need no upkeep when a document's
// topics change, are read in 128-byte pieces, and, not depending on the
// document, can be read a token ahead.  What is left of a token is a chain of
// dependent steps (gather, scan, test, selection, update) that costs 80
// instructions a token with four documents to a warp against 240 with one, and
// 313 with the walks of doc_counts.cuh: W = 8 for throughput, W = 32 for the
// fewest steps between a document's tokens.  Bound by the latency of those steps
// at 16 warps an SM and by the L1 data pipe (72 %, the random count gathers).
#pragma once

#include "common.cuh"
#include "kernels.cuh"
#include "warp.cuh"

namespace gpulda {

// Counts of topics 0..K-1, rounded up to 64 entries.  Entry word_doc_entries(K)
// is the count of no topic: what a document without a token adds and removes.
__host__ __device__ __forceinline__ u32 word_doc_entries(u32 K) { return (K + 63) & ~63u; }

// Shared memory per document of up to Kmax topics.
__host__ __device__ __forceinline__ size_t word_doc_bytes(u32 Kmax) { return (size_t)word_doc_entries(Kmax) * 2 + 16; }

// Staged tokens of a warp with 32/W documents: a chunk of W and the one after
// it per document, 32 bytes each.
__host__ __device__ constexpr size_t stage_bytes(u32 W) { return (32 / W) * (W + 1) * 32; }

// Shared memory per warp, with four documents or one.
__host__ __device__ __forceinline__ size_t word_warp_bytes(u32 Kmax) {
  return word_doc_bytes(Kmax) * 4 + stage_bytes(8);
}
__host__ __device__ __forceinline__ size_t word_warp_bytes_one(u32 Kmax) {
  return word_doc_bytes(Kmax) + stage_bytes(32);
}

// Flag beside a drawn topic: the sparse branch drew it.
constexpr u32 kWordSparse = 0x10000u;

// --- lane groups ----------------------------------------------------------------

template <u32 W>
__device__ __forceinline__ u32 group_lane(u32 lane) { return lane & (W - 1); }

// The group's bits of a warp ballot.
template <u32 W>
__device__ __forceinline__ u32 group_ballot(bool p, u32 lane) {
  const u32 b = __ballot_sync(kFullMask, p);
  return W == 32 ? b : (b >> (lane & (32 - W))) & ((1u << (W & 31)) - 1u);
}

template <u32 W, class T>
__device__ __forceinline__ T group_get(T x, u32 from) {
  return __shfl_sync(kFullMask, x, from, W);
}

// --- a document's counts ---------------------------------------------------------

struct WordDoc {
  uint16_t* cnt;  // dense counts
  u32 K;
  u32 none;  // the entry of no topic
  u32 nz;    // topics with a nonzero count
};

// The group's document in the warp's shared memory.
template <u32 W>
__device__ __forceinline__ WordDoc word_doc_at(unsigned char* wsm, u32 Kmax, u32 lane) {
  WordDoc dc;
  dc.cnt = (uint16_t*)(wsm + (size_t)(lane / W) * word_doc_bytes(Kmax));
  dc.none = word_doc_entries(Kmax);
  dc.K = Kmax;
  dc.nz = 0;
  return dc;
}

// Counts of the topics z[0..L) of the group's document with K topics.  A topic
// >= K is counted modulo K and reported in *status.
template <u32 W>
__device__ __forceinline__ void word_doc_build(WordDoc& dc, const u32* z, u32 L, u32 K, u32 lane, u32* status,
                                                 u32 bad_topic_bit) {
  const u32 l = group_lane<W>(lane);
  const u32 Ke = word_doc_entries(K);
  for (u32 i = l; i < Ke / 8; i += W) reinterpret_cast<uint4*>(dc.cnt)[i] = make_uint4(0, 0, 0, 0);
  __syncwarp();
  const u32 Lmax = W == 32 ? L : __reduce_max_sync(kFullMask, L);
  u32 nz = 0;
  for (u32 b = 0; b < Lmax; b += W) {
    const u32 i = b + l;
    bool born = false;
    if (i < L) {
      u32 k = z[i];
      if (k >= K) {
        *status |= bad_topic_bit;
        k %= K;
      }
      const u32 sh = (k & 1) * 16;
      born = ((atomicAdd(reinterpret_cast<u32*>(dc.cnt) + (k >> 1), 1u << sh) >> sh) & 0xffffu) == 0;
    }
    nz += __popc(group_ballot<W>(born, lane));
  }
  if (l == 0) dc.cnt[dc.none] = 0x4000;
  __syncwarp();
  dc.K = K;
  dc.nz = nz;
}

// cnt[k] += 1 and cnt[z] -= 1 by the group's lanes 0 and 1 in one step (nothing
// when they are the same).  Returns, in lane 0, whether k's count was 0, in
// lane 1, whether z's was 1.
template <u32 W>
__device__ __forceinline__ bool counts_move(const WordDoc& dc, u32 k, u32 z, u32 l) {
  uint16_t* p = dc.cnt + (l == 0 ? k : z);
  const u32 c = *p;
  const bool act = l < 2 && k != z;
  if (act) *p = (uint16_t)(c + 1u - 2u * l);
  __syncwarp();
  return act && c == l;
}

// --- draws -------------------------------------------------------------------------

__device__ __forceinline__ u64 mass_of(const uint16_t* cnt, u64 ent) {
  return (u64)cnt[(u32)ent] * (u32)(ent >> 32);
}

__device__ __forceinline__ u64 mass_of(const uint16_t* cnt, const ulonglong2& e) {
  return mass_of(cnt, e.x) + mass_of(cnt, e.y);
}

struct Staged {  // a token's data, read back by its group
  uint4 a, b;
  __device__ __forceinline__ u32 z() const { return a.x & 0xffffu; }
  __device__ __forceinline__ u32 kd() const { return a.x >> 16; }
  __device__ __forceinline__ u32 r0() const { return a.y; }
  __device__ __forceinline__ u32 r1() const { return a.z; }
  __device__ __forceinline__ u32 nw() const { return a.w; }
  __device__ __forceinline__ const ulonglong2* list() const {
    return (const ulonglong2*)(((u64)b.y << 32) | b.x);
  }
  __device__ __forceinline__ double aA() const { return __hiloint2double((int)b.w, (int)b.z); }
};

__device__ __forceinline__ Staged staged(const uint4* gs, u32 j) { return Staged{gs[2 * j], gs[2 * j + 1]}; }

// The draw of one token of each group over lists of any length.  Out of line:
// the common draws' loop stays small enough for the instruction cache.  Returns
// the topic, with kWordSparse.
template <u32 W>
static __device__ __noinline__ u32 long_draw(const uint16_t* cnt, Staged c, u32 lane) {
  const u32 l = group_lane<W>(lane);
  const u32 nw = c.nw();
  const Run r = lane_run<W>(nw, l);
  const u32 n = r.on ? r.n : 0u;
  const ulonglong2* list = c.list();
  // eight pairs at a time, the next eight on their way
  constexpr u32 NB = 8;
  ulonglong2 e[NB];
  auto fetch = [&](u32 p) {
#pragma unroll
    for (u32 u = 0; u < NB; ++u) {
      e[u] = make_ulonglong2(0, 0);
      if (p + u < n) e[u] = __ldg(list + r.at + (p + u) * 8);
    }
  };
  u64 x = 0, y = 0;
  fetch(0);
  for (u32 p = 0; p < n; p += NB) {
    ulonglong2 g[NB];
#pragma unroll
    for (u32 u = 0; u < NB; ++u) g[u] = e[u];
    fetch(p + NB);
#pragma unroll
    for (u32 u = 0; u < NB; u += 2) {
      x += mass_of(cnt, g[u]);
      y += mass_of(cnt, g[u + 1]);
    }
  }
  x += y;
  __syncwarp();
  const u64 incl = group_scan<W>(x);
  const u64 B = group_get<W>(incl, W - 1);
  const bool sp = sparse_test(c.r0(), c.aA(), B);
  u64 t = scale_u32(c.r1(), B);
  u32 f = __popc(group_ballot<W>(incl <= t, lane)) & (W - 1);
  t -= group_get<W>(incl - x, f);
  // the crossing lane's run is spread over the group until one pair is left
  u32 at = group_get<W>(r.at, f), len = group_get<W>(n, f);
  if (!sp) len = 0;
  while (__any_sync(kFullMask, len > W)) {
    const u32 per = (len + W - 1) / W;
    u64 v = 0;
    for (u32 i = 0; i < per; ++i)
      if (per * l + i < len) v += mass_of(cnt, __ldg(list + at + (per * l + i) * 8));
    __syncwarp();
    const u64 in2 = group_scan<W>(v);
    f = __popc(group_ballot<W>(in2 <= t, lane)) & (W - 1);
    t -= group_get<W>(in2 - v, f);
    at += f * per * 8;
    len = len ? min(per, len - f * per) : 0u;
  }
  u64 m0 = 0, m1 = 0;
  u32 k0 = 0, k1 = 0;
  if (l < len) {
    const ulonglong2 v = __ldg(list + at + l * 8);
    k0 = (u32)v.x;
    k1 = (u32)v.y;
    m0 = mass_of(cnt, v.x);
    m1 = mass_of(cnt, v.y);
  }
  __syncwarp();
  const u64 in2 = group_scan<W>(m0 + m1);
  f = __popc(group_ballot<W>(in2 <= t, lane)) & (W - 1);
  const u32 k = group_get<W>(in2 - m1 > t ? k0 : k1, f);
  return sp ? k | kWordSparse : c.kd();
}

// The draws of n tokens (tokens past a document's end are staged as tokens of
// no topic).  Lists of up to kShortList entries are walked with the next token's
// entries already on their way: a list's loads do not depend on the document,
// so they are issued a token ahead.  Longer lists go through long_draw.  Drawn
// topics go to gs[2 j].x (with kWordSparse); returns counts_move's answers, a bit
// per token.
//
// This one for four documents to a warp.
__device__ __forceinline__ u32 draw_chunk_quarter(const WordDoc& dc, uint4* gs, u32 n, u32 lane) {
  constexpr u32 W = 8, NP = 10;  // pairs per lane of a list of kShortList entries
  const u32 l = group_lane<W>(lane);
  const uint16_t* cnt = dc.cnt;
  u32 h = 0;
  ulonglong2 pre[NP];
#pragma unroll
  for (u32 p = 0; p < NP; ++p) pre[p] = make_ulonglong2(0, 0);
  Staged s = staged(gs, 0);
  u32 c8 = 0;  // pairs per lane
  bool on = false, wide;
  auto fetch = [&]() {
    wide = __any_sync(kFullMask, s.nw() > kShortList);
    if (wide) return;
    c8 = ((s.nw() + 31) >> 5) << 1;  // list_pairs, or 0 for an empty list
    on = 2 * c8 * l < s.nw();
    const ulonglong2* at = s.list() + l;
    if (on) {
#pragma unroll
      for (u32 p = 0; p < NP; p += 2)
        if (p == 0 || c8 > p) {
          pre[p] = __ldg(at + 8 * p);
          pre[p + 1] = __ldg(at + 8 * p + 8);
        }
    }
  };
  fetch();
#pragma unroll 2
  for (u32 j = 0; j < n; ++j) {
    const Staged c = s;
    u32 k;
    if (wide) {
      k = long_draw<W>(cnt, c, lane);
      s = staged(gs, j + 1);
      fetch();
    } else {
      const u32 cj = c8;
      u64 x = 0;
      if (on) {
        u64 y = 0;
#pragma unroll
        for (u32 p = 0; p < NP; p += 2)
          if (p == 0 || c8 > p) {
            x += mass_of(cnt, pre[p]);
            y += mass_of(cnt, pre[p + 1]);
          }
        x += y;
      }
      s = staged(gs, j + 1);
      fetch();

      const u64 incl = group_scan<W>(x);
      const u64 B = group_get<W>(incl, W - 1);
      const bool sp = sparse_test(c.r0(), c.aA(), B);
      u64 t = scale_u32(c.r1(), B);
      u32 f = __popc(group_ballot<W>(incl <= t, lane)) & (W - 1);
      // the crossing lane's run (an even number of pairs, at most 10) is spread
      // over the group, two pairs per lane
      t -= group_get<W>(incl - x, f);
      const ulonglong2* list = c.list() + f;
      u64 m0 = 0, m1 = 0, m2 = 0, m3 = 0;
      u32 k0 = 0, k1 = 0, k2 = 0, k3 = 0;
      if (sp && 2 * l < cj) {
        const ulonglong2 e = __ldg(list + 16 * l), g = __ldg(list + 16 * l + 8);
        k0 = (u32)e.x;
        k1 = (u32)e.y;
        k2 = (u32)g.x;
        k3 = (u32)g.y;
        m0 = mass_of(cnt, e.x);
        m1 = m0 + mass_of(cnt, e.y);
        m2 = m1 + mass_of(cnt, g.x);
        m3 = m2 + mass_of(cnt, g.y);
      }
      const u64 in2 = group_scan<W>(m3);
      f = __popc(group_ballot<W>(in2 <= t, lane)) & (W - 1);
      const u64 u = t - (in2 - m3);
      k = k3;
      if (m2 > u) k = k2;
      if (m1 > u) k = k1;
      if (m0 > u) k = k0;
      k = group_get<W>(k, f);
      k = sp ? k | kWordSparse : c.kd();
    }
    if (l == 0) gs[2 * j].x = k;
    if (counts_move<W>(dc, k & 0xffffu, s.z(), l)) h |= 1u << j;
  }
  return h;
}

// And for one document to a warp, where the time from one token to the next is
// what counts: every instruction between them adds to it.  Lists of up to 64
// entries, a pair per lane, have steps of their own.
__device__ __forceinline__ u32 draw_chunk_whole(const WordDoc& dc, uint4* gs, u32 n, u32 lane) {
  constexpr u32 W = 32, NP = 3;  // pairs per lane of a list of kShortList entries
  const uint16_t* cnt = dc.cnt;
  // the lane's pair of a list of up to 32 entries (lanes 0..15) and up to 64
  const u32 at2 = (lane & 1) * 8 + (lane >> 1), at4 = (lane & 3) * 8 + (lane >> 2);
  u32 h = 0;
  ulonglong2 pre[NP];
#pragma unroll
  for (u32 p = 0; p < NP; ++p) pre[p] = make_ulonglong2(0, 0);
  Staged s = staged(gs, 0);
  Run run{0, 0, false};
  u32 kind = 0;  // 0: up to 64 entries, 1: up to kShortList, 2: longer
  auto fetch = [&]() {
    const u32 nw = s.nw();
    if (!__any_sync(kFullMask, nw > 64)) {
      kind = 0;
      run.on = 2 * lane < nw;
      if (run.on) pre[0] = __ldg(s.list() + (nw <= 32 ? at2 : at4));
    } else if (!__any_sync(kFullMask, nw > kShortList)) {
      kind = 1;
      run = lane_run<W>(nw, lane);
      const ulonglong2* at = s.list() + run.at;
#pragma unroll
      for (u32 p = 0; p < NP; ++p)
        if (run.on && run.n > p) pre[p] = __ldg(at + 8 * p);
    } else {
      kind = 2;
    }
  };
  fetch();
#pragma unroll 2
  for (u32 j = 0; j < n; ++j) {
    const Staged c = s;
    u32 k;
    if (kind == 0) {
      // (a lane past the list's end has entries of an earlier token)
      const u32 T0 = (u32)pre[0].x, T1 = (u32)pre[0].y;
      const u64 m0 = mass_of(cnt, pre[0].x);
      const u64 m1 = m0 + mass_of(cnt, pre[0].y);
      const u64 x = run.on ? m1 : 0ull;
      s = staged(gs, j + 1);
      fetch();
      const u64 incl = group_scan<W>(x);
      const u64 B = group_get<W>(incl, W - 1);
      const bool sp = sparse_test(c.r0(), c.aA(), B);
      const u64 t = scale_u32(c.r1(), B);
      const u32 f = __popc(__ballot_sync(kFullMask, incl <= t)) & (W - 1);
      k = group_get<W>(m0 > t - (incl - x) ? T0 : T1, f);
      k = sp ? k | kWordSparse : c.kd();
    } else if (kind == 1) {
      u64 m[2 * NP];
      u32 T[2 * NP];
      u64 x = 0;
#pragma unroll
      for (u32 p = 0; p < NP; ++p) {
        T[2 * p] = (u32)pre[p].x;
        T[2 * p + 1] = (u32)pre[p].y;
        m[2 * p] = x + (run.n > p ? mass_of(cnt, pre[p].x) : 0ull);
        x = m[2 * p + 1] = m[2 * p] + (run.n > p ? mass_of(cnt, pre[p].y) : 0ull);
      }
      if (!run.on) x = 0;
      s = staged(gs, j + 1);
      fetch();
      const u64 incl = group_scan<W>(x);
      const u64 B = group_get<W>(incl, W - 1);
      const bool sp = sparse_test(c.r0(), c.aA(), B);
      const u64 t = scale_u32(c.r1(), B), u = t - (incl - x);
      const u32 f = __popc(__ballot_sync(kFullMask, incl <= t)) & (W - 1);
      k = T[2 * NP - 1];
#pragma unroll
      for (u32 i = 2 * NP - 1; i-- > 0;)
        if (m[i] > u) k = T[i];
      k = group_get<W>(k, f);
      k = sp ? k | kWordSparse : c.kd();
    } else {
      k = long_draw<W>(cnt, c, lane);
      s = staged(gs, j + 1);
      fetch();
    }
    if (lane == 0) gs[2 * j].x = k;
    if (counts_move<W>(dc, k & 0xffffu, s.z(), lane)) h |= 1u << j;
  }
  return h;
}

// --- a document's tokens ---------------------------------------------------------

// `Src` gives a group's tokens, W to a chunk:
//   word(c), topic(c)   the lane's word and topic in chunk c (loads)
//   valid(c)            whether the lane has a token there
//   words(c)            its Philox words
//   chunk_done(c, k, z) after chunk c: k its drawn topic, *z the next chunk's topic
// A chunk's words are loaded three chunks ahead, what they lead to two ahead,
// and its topics and the alias entries of its dense draws one ahead, so that
// nothing of it is waited for.
struct Rows {  // where a word's row of q and its list start
  const u64* row_off;   // null: w * K
  const u64* list_off;  // null: w * list_stride(K)
};

struct WordData {  // a lane's word in a chunk
  u32 w, nw;
  u64 A, row, list;
};

// Draws the topics of all the group's tokens, `n_chunks` (the warp's most)
// chunks.  sink(chunk, k, sparse, nzm, row, nw) receives each lane's results.
template <u32 W, class Src, class Sink>
__device__ __forceinline__ void sweep_doc(WordDoc& dc, uint4* stage, const ModelDev& m, const Rows& rows, u32 K,
                                          float alpha, u32 n_chunks, u32 lane, Src& src, Sink&& sink) {
  const u32 l = group_lane<W>(lane);
  uint4* gs = stage + 2 * (lane / W) * (W + 1);
  // chunk c's list length, mass and rows
  auto look_up = [&](u32 c, u32 w) {
    const bool v = src.valid(c);
    WordData d;
    d.w = w;
    d.nw = v ? __ldg(m.nnz + w) : 0u;
    d.A = v ? __ldg(m.A + w) : 0ull;
    d.row = rows.row_off ? (v ? __ldg(rows.row_off + w) : 0ull) : (u64)w * K;
    d.list = rows.list_off ? (v ? __ldg(rows.list_off + w) : 0ull) : (u64)w * list_stride(K);
    return d;
  };
  // its Philox words, and the alias entry of the dense draw's slot
  u32 r0 = 0, r1 = 0, r3 = 0;
  u64 al = 0;
  auto draw = [&](u32 c, const WordData& d) {
    const U4 r = src.words(c);
    r0 = r.x;
    r1 = r.y;
    r3 = r.w;
    al = d.nw ? __ldg(m.al + d.row + (u32)(((u64)r.z * d.nw) >> 32)) : 0ull;
  };
  WordData d1 = look_up(0, src.word(0));
  u32 w2 = src.word(1), w3 = src.word(2);
  u32 z1 = src.valid(0) ? src.topic(0) : dc.none;
  draw(0, d1);
  WordData d2 = look_up(1, w2);
  if (l == 0) gs[2 * W] = make_uint4(dc.none | (dc.none << 16), 0, 0, 0);  // behind a chunk: no token
  for (u32 c = 0; c < n_chunks; ++c) {
    // stage the chunk's tokens; a word whose every q is zero keeps the token's
    // topic: nothing else has mass, and its dense draw is that topic
    const u32 kd = d1.nw ? alias_pick(al, r3) : z1;
    const u32 z = z1, nw = d1.nw;
    const u64 row = d1.row;
    __syncwarp();
    {
      const u64 aA = (u64)__double_as_longlong(__dmul_rn((double)alpha, exact_double(d1.A)));
      const u64 cp = (u64)(m.lists + d1.list);
      gs[2 * l] = make_uint4(z | (kd << 16), r0, r1, nw);
      gs[2 * l + 1] = make_uint4((u32)cp, (u32)(cp >> 32), (u32)aA, (u32)(aA >> 32));
    }
    // the chunks ahead
    d1 = d2;
    z1 = src.valid(c + 1) ? src.topic(c + 1) : dc.none;
    draw(c + 1, d1);
    d2 = look_up(c + 2, w3);
    w3 = src.word(c + 3);
    __syncwarp();
    // the first token's topic leaves the counts (the others' leave with the
    // draw before them)
    const bool gone = counts_move<W>(dc, dc.none, gs[0].x & 0xffffu, l);
    dc.nz -= (group_ballot<W>(gone, lane) >> 1) & 1u;
    const u32 left = __ballot_sync(kFullMask, z != dc.none);
    const u32 n = W == 32 ? 32u - __clz((int)left) : W;
    const u32 hist = W == 8 ? draw_chunk_quarter(dc, gs, n, lane) : draw_chunk_whole(dc, gs, n, lane);
    __syncwarp();
    // results: the lane's topic, and the document's distinct topics without it
    const u32 kk = gs[2 * l].x;
    const u32 born = group_get<W>(hist, 0), died = group_get<W>(hist, 1);
    const u32 before = (1u << l) - 1u;
    sink(c, kk & 0xffffu, (kk & kWordSparse) != 0, dc.nz + __popc(born & before) - __popc(died & before), row, nw);
    dc.nz += __popc(born) - __popc(died);
    src.chunk_done(c, kk & 0xffffu, &z1);
  }
}

// sum over the group's document's topics of lgamma(alpha + m_dk) -
// lgamma(alpha) (every lane receives it).  The topics are gathered first, in
// the memory of the staged tokens, so that the lanes' lgamma calls are full.
template <u32 W>
__device__ __forceinline__ double word_lgamma_sum(const WordDoc& dc, uint4* stage, float alpha, double lg_a, u32 lane) {
  const u32 l = group_lane<W>(lane);
  uint16_t* list = (uint16_t*)(stage + 2 * (lane / W) * (W + 1));
  constexpr u32 kRoom = (W + 1) * 16;  // entries
  const u32 K = W == 32 ? dc.K : __reduce_max_sync(kFullMask, dc.K);
  const u32 below = (1u << l) - 1u;
  double dl = 0.0;
  u32 n = 0;
  __syncwarp();
  for (u32 b = 0; b < K; b += 2 * W) {
    const u32 pair = b < dc.K ? reinterpret_cast<const u32*>(dc.cnt)[(b >> 1) + l] : 0u;
    const u32 m0 = group_ballot<W>((pair & 0xffffu) != 0, lane), m1 = group_ballot<W>((pair >> 16) != 0, lane);
    u32 at = n + __popc(m0 & below) + __popc(m1 & below);
    if (pair & 0xffffu) list[at++] = (uint16_t)(b + 2 * l);
    if (pair >> 16) list[at] = (uint16_t)(b + 2 * l + 1);
    n += __popc(m0) + __popc(m1);
    if (__any_sync(kFullMask, n + 2 * W > kRoom) || b + 2 * W >= K) {
      __syncwarp();
      for (u32 e = l; e < n; e += W) dl += lgamma((double)alpha + (double)dc.cnt[list[e]]) - lg_a;
      __syncwarp();
      n = 0;
    }
  }
#pragma unroll
  for (u32 o = W / 2; o > 0; o >>= 1) dl += __shfl_xor_sync(kFullMask, dl, o, W);
  return dl;
}

}  // namespace gpulda
