// zsweep_words.cu -- the per-document topic sweep over the words' lists of topics
// (reference: sample_topics, src/cu/topics.cu:36-105), K <= kMapMinK.  The draws
// are in word_sweep.cuh; this kernel adds the count rebuild n[w][k] += 1 for
// every token's new topic, the statistics and the joint log-likelihood, and the
// choice of kernels for a whole sweep (launch_sweep).
#include <algorithm>
#include <cmath>

#include "kernels.cuh"
#include "word_sweep.cuh"

namespace gpulda {

namespace {

constexpr u32 kMaxDocLen = 65535u;
constexpr size_t kZMaxSmem = 200 * 1024;
constexpr u32 kSmSmem = 228 * 1024;      // an SM's shared memory
constexpr u32 kBlockSmem = 1024 + 64;    // a block's beside the warps': the system's and its statistics

struct ZWordArgs {
  ModelDev m;
  ZLaunch z;
  BatchDev b;    // problem tables (batched launches only)
  u32 Kmax;      // largest K of the launch (sets the shared-memory stride)
  u32 n_long;    // documents that take a warp each
  double lg_Ka;  // lgamma(K * alpha)
  double lg_a;   // lgamma(alpha)
};

// A group's document as sweep_doc's source of tokens.
template <u32 W>
struct ZSource {
  const u32* w_;
  const u32* z_;
  u32 L, K, V, l;
  u64 idx0;
  u32 t, key0, key1;
  u32 status;
  __device__ __forceinline__ bool valid(u32 c) const { return c * W + l < L; }
  __device__ __forceinline__ u32 word(u32 c) {
    u32 w = valid(c) ? w_[c * W + l] : 0u;
    if (w >= V) {
      status |= kStatusBadWord;
      w %= V;
    }
    return w;
  }
  __device__ __forceinline__ u32 topic(u32 c) const {
    const u32 k = z_[c * W + l];
    return k >= K ? k % K : k;
  }
  __device__ __forceinline__ U4 words(u32 c) const {
    return draw4(idx0 + c * W + l, t, kStreamZ, 0, key0, key1);
  }
  __device__ __forceinline__ void chunk_done(u32, u32, u32*) const {}
};

// What a lane gathers over the documents of its warp.
struct LaneSums {
  double ll, ll_skip;  // log-likelihood terms
  u32 status;
};

// 32/W documents from `first` of the order, W lanes to a document; they have
// about the same length.
//
// BATCH: the launch sweeps documents of many independent problems laid out in
// one set of arenas; each document's K, alpha, Philox key and token numbering
// come from its problem, and a token's (word, topic) row starts at
// b.row_off[w] instead of w * K.  Otherwise all parameters come from `m`.
//
// LL: the launch accumulates the joint log-likelihood.
template <u32 W, bool BATCH, bool LL>
__device__ __forceinline__ void sweep_documents(const ZWordArgs& a, unsigned char* wsm, u64 first,
                                                unsigned long long* blk_stats, LaneSums& sums, u32 lane) {
  const ModelDev& m = a.m;
  const ZLaunch& p = a.z;
  const u32 l = group_lane<W>(lane), V = m.V;
  WordDoc dc = word_doc_at<W>(wsm, a.Kmax, lane);
  uint4* stage = reinterpret_cast<uint4*>(wsm + word_doc_bytes(a.Kmax) * (32 / W));
  double ll_acc = 0.0, ll_skip = 0.0;
  u32 status = 0;
  // the group's document; a group without one goes along with length 0
  const u64 at = first + lane / W;
  bool have = at < p.n_docs;
  const u32 doc = have ? (p.order ? p.order[at] : (u32)at) : 0u;
  u32 L = have ? p.d_len[doc] : 0u;
  const u64 off = have ? p.d_idx[doc] : 0u;
  u32 K = m.K, key0 = m.key0, key1 = m.key1, pb = 0;
  float alpha = m.alpha;
  u64 tok_base = p.tok_base;
  double lg_a = a.lg_a, lg_Ka = a.lg_Ka;
  if (BATCH) {
    pb = a.b.pid[doc];
    K = a.b.K[pb];
    alpha = a.b.alpha[pb];
    key0 = a.b.key0[pb];
    key1 = a.b.key1[pb];
    tok_base = a.b.tok_base[pb];  // the problem's first token: local numbering
    lg_a = a.b.lg_a[pb];
    lg_Ka = a.b.lg_Ka[pb];
  }
  const u32 t = p.t_dev ? *p.t_dev : p.t;
  if (L > kMaxDocLen) {
    status |= kStatusDocTooLong;
    have = false;
    L = 0;
  } else if (off + L > p.n_tokens) {
    status |= kStatusDocRange;
    have = false;
    L = 0;
  }
  word_doc_build<W>(dc, p.z + off, L, K, lane, &status, kStatusBadTopic);
  u32 work = 0, n_sparse = 0;  // the lane's sparse work and draws

  const u32 Lmax = W == 32 ? L : __reduce_max_sync(kFullMask, L);
  ZSource<W> src{p.w + off, p.z + off, L, K, V, l,
                 // Philox index of the document's first token: its position in
                 // its corpus (batched problems count from their own first
                 // token) plus the buffer's offset
                 BATCH ? off - tok_base : tok_base + off, t, key0, key1, 0u};
  sweep_doc<W>(dc, stage, m, Rows{BATCH ? a.b.row_off : nullptr, BATCH ? a.b.list_off : nullptr}, K, alpha,
               (Lmax + W - 1) / W, lane, src,
               [&](u32 c, u32 new_z, bool sparse, u32 nzm, u64 row, u32 nw) {
                 const u32 i = c * W + l;
                 if (i >= L) return;
                 work += min(nzm, nw);
                 n_sparse += sparse;
                 p.z[off + i] = new_z;
                 atomicAdd(m.n + row + new_z, 1u);
                 if (LL) {  // log Phi[new topic][word], one token per lane
                   const u32 qk = __ldg(m.q + row + new_z);
                   if (qk)
                     ll_acc += log((double)qk) - 22.18070977791825;  // 32 log 2
                   else
                     ll_skip += 1.0;
                 }
               });
  status |= src.status;
  if (l == 0 && have && p.K_d) p.K_d[doc] = dc.nz;
  if (LL) {
    const double dl = word_lgamma_sum<W>(dc, stage, alpha, lg_a, lane);
    if (l == 0 && have) ll_acc += dl + lg_Ka - lgamma((double)K * (double)alpha + (double)L);
    if (BATCH) {  // per-problem sums
      double s0 = ll_acc, s1 = ll_skip;
#pragma unroll
      for (u32 o = W / 2; o > 0; o >>= 1) {
        s0 += __shfl_xor_sync(kFullMask, s0, o, W);
        s1 += __shfl_xor_sync(kFullMask, s1, o, W);
      }
      if (l == 0 && have) {
        atomicAdd(p.ll + 2 * pb, s0);
        atomicAdd(p.ll + 2 * pb + 1, s1);
      }
      ll_acc = ll_skip = 0.0;
    }
  }
  work = __reduce_add_sync(kFullMask, work);
  n_sparse = __reduce_add_sync(kFullMask, n_sparse);
  if (l == 0 && have) {
    atomicAdd(blk_stats + 0, (unsigned long long)L);
    atomicAdd(blk_stats + 1, 1ull);
  }
  if (lane == 0) {
    atomicAdd(blk_stats + 2, (unsigned long long)work);
    atomicAdd(blk_stats + 3, (unsigned long long)n_sparse);
  }
  __syncwarp();
  sums.ll += ll_acc;
  sums.ll_skip += ll_skip;
  sums.status |= status;
}

template <bool BATCH, bool LL>
__global__ void __launch_bounds__(256, 2) z_sweep_words_kernel(ZWordArgs a) {
  extern __shared__ __align__(16) unsigned char zsm[];
  __shared__ unsigned long long blk_stats[4];  // tokens, documents, sparse work, sparse draws
  if (a.z.shares && mostly_long_lists(a.z.shares)) return;  // the other sweep's
  if (threadIdx.x < 4) blk_stats[threadIdx.x] = 0;
  __syncthreads();
  const ZLaunch& p = a.z;
  const u32 lane = threadIdx.x & 31;
  unsigned char* wsm = zsm + (size_t)(threadIdx.x >> 5) * word_warp_bytes(a.Kmax);
  LaneSums sums{0.0, 0.0, 0u};
  auto claim = [&]() {
    u32 i = 0;
    if (lane == 0) i = atomicAdd(p.work, 1u);
    return __shfl_sync(kFullMask, i, 0);
  };
  u32 item = claim();
  const u32 n_long = p.n_long_dev ? *p.n_long_dev : a.n_long;
  for (; item < n_long; item = claim()) sweep_documents<32, BATCH, LL>(a, wsm, item, blk_stats, sums, lane);
  while (true) {
    const u64 first = n_long + 4 * (u64)(item - n_long);
    if (first >= p.n_docs) break;
    sweep_documents<8, BATCH, LL>(a, wsm, first, blk_stats, sums, lane);
    item = claim();
  }
  if (LL && !BATCH) {
    double ll_acc = warp_sum_f64(sums.ll);
    double ll_skip = warp_sum_f64(sums.ll_skip);
    if (lane == 0) {
      atomicAdd(p.ll, ll_acc);
      atomicAdd(p.ll + 1, ll_skip);
    }
  }
  const u32 status = __reduce_or_sync(kFullMask, sums.status);
  if (lane == 0 && status) atomicOr(p.status, status);
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(p.counters + kCtrTokens, blk_stats[0]);
    atomicAdd(p.counters + kCtrDocs, blk_stats[1]);
    atomicAdd(p.counters + kCtrSparseWork, blk_stats[2]);
    atomicAdd(p.counters + kCtrSparseDraws, blk_stats[3]);
  }
}

template <bool BATCH, bool LL>
void launch_impl(const ZWordArgs& a, cudaStream_t s, u32 wpb, u32 blocks_per_sm) {
  const size_t per_warp = word_warp_bytes(a.Kmax);
  // Warps per block: the request, or fewer where more of them are resident then.
  // (Above K = 1600 two blocks of 8 do not fit an SM's shared memory.  3e6 tokens
  // over lists of 100 topics, with 8 warps resident and with 15 at K=1700 or 12 at
  // K=2048: 0.84 -> 0.61 and 0.85 -> 0.71 ms.)
  u32 most = 0, warps = 1;
  for (u32 n = wpb; n; --n) {
    const u32 resident = std::min<u32>(16, kSmSmem / (u32)(per_warp * n + kBlockSmem) * n);
    if (per_warp * n <= kZMaxSmem && resident > most) {
      most = resident;
      warps = n;
    }
  }
  wpb = warps;
  const size_t smem = per_warp * wpb;
  // The ceiling, not this launch's size: captured graphs may hold launches of
  // several sizes.  (The kernel's static shared memory counts towards the 48 KB
  // that need no attribute.)
  if (smem > 47 * 1024)
    cudaFuncSetAttribute(z_sweep_words_kernel<BATCH, LL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kZMaxSmem);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, z_sweep_words_kernel<BATCH, LL>, 32 * wpb, smem);
  if (per_sm < 1) per_sm = 1;
  if (blocks_per_sm && (int)blocks_per_sm < per_sm) per_sm = (int)blocks_per_sm;
  const u64 items = a.z.n_long_dev ? a.z.n_docs : a.n_long + ((u64)a.z.n_docs - a.n_long + 3) / 4;
  const u32 blocks = (u32)std::min<u64>((u64)device_sm_count() * per_sm, (items + wpb - 1) / wpb);
  z_sweep_words_kernel<BATCH, LL><<<blocks, 32 * wpb, smem, s>>>(a);
}

}  // namespace

void launch_z_sweep_words(const ModelDev& m, const BatchDev* b, u32 Kmax, const ZLaunch& z, u32 n_long, cudaStream_t s,
                          u32 warps_per_block, u32 blocks_per_sm) {
  if (!z.n_docs) return;
  ZWordArgs a;
  a.m = m;
  a.z = z;
  a.b = b ? *b : BatchDev{};
  a.Kmax = Kmax;
  a.n_long = std::min(n_long, z.n_docs);
  a.lg_a = b ? 0.0 : std::lgamma((double)m.alpha);
  a.lg_Ka = b ? 0.0 : std::lgamma((double)m.K * (double)m.alpha);
  const bool ll = (z.flags & kZFlagLoglik) && z.ll;
  if (b && ll)
    launch_impl<true, true>(a, s, warps_per_block, blocks_per_sm);
  else if (b)
    launch_impl<true, false>(a, s, warps_per_block, blocks_per_sm);
  else if (ll)
    launch_impl<false, true>(a, s, warps_per_block, blocks_per_sm);
  else
    launch_impl<false, false>(a, s, warps_per_block, blocks_per_sm);
}

// A warp with four documents takes about 1.1 us a token of its longest, one with
// one document 0.45 us; a sweep over a full GPU takes 0.17 ns a token.  A
// document is long when its chain at a quarter of a warp would be half of that
// sweep.
u32 long_document(u64 n_tokens) {
  const double len = 0.5 * 0.17 / 1100.0 * (double)n_tokens;
  return len < 65535.0 ? (u32)len + 1 : 65536u;
}

u32 launch_sweep(const ModelDev& m, const BatchDev* b, u32 Kmax, ZLaunch zl, const SweepAux& x, cudaStream_t s,
                 u32 warps_per_block, u32 blocks_per_sm) {
  if (!zl.n_docs) return 0;
  zl.work = x.ctrs + kCtrWork;
  if (Kmax <= kMapMinK && !m.lists) {  // (no memory for them)
    zl.shares = nullptr;
    if (b)
      launch_z_sweep_batch(m, *b, Kmax, zl, s, warps_per_block, blocks_per_sm);
    else
      launch_z_sweep(m, zl, s);
    return 1;
  }
  if (Kmax <= kMapMinK) {
    // Both sweeps are launched where the words' lists may be long, and one of
    // them returns at once (3 us): which is known on the device only.
    const bool either = Kmax > kShortList;
    if (either) zl.shares = m.shares;
    launch_z_sweep_words(m, b, Kmax, zl, x.n_long, s, warps_per_block, blocks_per_sm);
    if (!either) return 1;
    if (b)
      launch_z_sweep_batch(m, *b, Kmax, zl, s, warps_per_block, blocks_per_sm);
    else
      launch_z_sweep(m, zl, s);
    return 2;
  }
  zl.rest = x.queue;
  zl.n_rest = x.ctrs + kCtrRest;
  launch_z_sweep_pairs(m, zl, s);
  // a list holds a document's topics and at most 32 more
  if (std::min(x.lmax, Kmax) + 32 <= kListMost) return 1;
  zl.work = x.ctrs + kCtrRestWork;
  launch_z_sweep_rest(m, zl, s, x.lmax);
  return 2;
}

}  // namespace gpulda
