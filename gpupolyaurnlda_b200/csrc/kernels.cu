// kernels.cu -- the sampler's device code for sm_100a.
//
// One iteration (reference: src/cu/train.cu:137-172) is
//   phi_draw      x[k][w] ~ Poisson(beta + n[k][w]); S[k] = sum_w x; n <- 0
//   alias_build   q[w][k] = floor(x * 2^32 / S[k]); A[w] = sum_k q; alias table of
//                 word w over topics with weights q[w][.]
//   doc_offsets   exclusive scan of document lengths
//   z_sweep       per document, sequentially per token: remove z_i, draw
//                 p(k) ~ q[w_i][k] * (alpha + m_dk), add back, n[w_i][z_i] += 1
// All arrays indexed by (word, topic) are word-major: index w*K + k.
#include "kernels.cuh"
#include "warp.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>

namespace gpulda {

namespace {

// ---------------------------------------------------------------------------
// Initial counts (reference: polya_urn_init, src/cu/polyaurn.cu:61-79):
// n[w][k] ~ Poisson(beta + floor(C[w] / K)).  One Philox block serves the
// four cells 4g .. 4g+3.
// ---------------------------------------------------------------------------
__global__ void init_counts_kernel(u32* __restrict__ n, u32 K, u32 V, const u32* __restrict__ C, PoisTables tb,
                                   double beta, u32 key0, u32 key1) {
  const u64 cells = (u64)K * V;
  const u64 groups = (cells + 3) / 4;
  for (u64 gi = (u64)blockIdx.x * blockDim.x + threadIdx.x; gi < groups; gi += (u64)gridDim.x * blockDim.x) {
    const U4 r = draw4(gi, 0, kStreamInitCounts, 0, key0, key1);
#pragma unroll
    for (u32 u = 0; u < 4; ++u) {
      const u64 c = gi * 4 + u;
      if (c < cells) {
        const u32 lam_n = C[c / K] / K;
        n[c] = poisson_draw(lam_n, beta, u4_word(r, u), c, 0, kStreamInitCounts, key0, key1, tb);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Phi draw (reference: polya_urn_sample + draw_poisson + polya_urn_reset,
// src/cu/polyaurn.cu:7-36,87-141).  Each block owns a contiguous range of
// rows; threads take groups of four cells (one Philox block, 16-byte loads and
// stores when the group lies inside the range).  Per-topic sums are gathered
// in shared memory (integer atomics: order-free) and flushed once per block.
// ---------------------------------------------------------------------------
// Cells [c0, c1) of one model (local cell indices; n and q point at its cell
// 0).  Nonzero draws are added to the per-topic sums: into shared memory when
// s_sum is given, else straight into S.
__device__ __forceinline__ void phi_rows(u32 K, u64 c0, u64 c1, u32* __restrict__ n, u32* __restrict__ q, u64* S,
                                         const PoisTables& tb, double beta, u32 key0, u32 key1, u32 t,
                                         unsigned long long* s_sum) {
  for (u64 gi = c0 / 4 + threadIdx.x; gi * 4 < c1; gi += blockDim.x) {
    const u64 cb = gi * 4;
    // topic of the group's first cell (c0 is a row's start; a range has fewer
    // than 2^32 - 4 cells, so 32 bits hold its cells' numbers)
    u32 k = (cb >= c0 ? (u32)(cb - c0) : K - (u32)(c0 - cb) % K) % K;
    const U4 r = draw4(gi, t, kStreamPhi, 0, key0, key1);
    const bool whole = cb >= c0 && cb + 4 <= c1;
    u32 nv[4];
    if (whole) {
      const uint4 v = *reinterpret_cast<const uint4*>(n + cb);
      nv[0] = v.x;
      nv[1] = v.y;
      nv[2] = v.z;
      nv[3] = v.w;
    } else {
#pragma unroll
      for (u32 u = 0; u < 4; ++u) nv[u] = (cb + u >= c0 && cb + u < c1) ? n[cb + u] : 0u;
    }
    u32 xv[4];
#pragma unroll
    for (u32 u = 0; u < 4; ++u) xv[u] = poisson_draw(nv[u], beta, u4_word(r, u), cb + u, t, kStreamPhi, key0, key1, tb);
    if (whole) {
      *reinterpret_cast<uint4*>(q + cb) = make_uint4(xv[0], xv[1], xv[2], xv[3]);
      *reinterpret_cast<uint4*>(n + cb) = make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (u32 u = 0; u < 4; ++u) {
      const u64 c = cb + u;
      if (c >= c0 && c < c1) {
        if (!whole) {
          q[c] = xv[u];
          n[c] = 0;
        }
        if (xv[u]) {
          if (s_sum)
            atomicAdd(&s_sum[k], (unsigned long long)xv[u]);
          else
            atomicAdd((unsigned long long*)&S[k], (unsigned long long)xv[u]);
        }
      }
      k = k + 1 == K ? 0u : k + 1;
    }
  }
}

// Four blocks per SM: the rejection sampler's registers otherwise held the
// kernel to two (1.4x faster at K=10000; its spills are on the rare path).
__global__ void __launch_bounds__(256, 4) phi_draw_kernel(ModelDev m, u32 t, u32 rows_per_block, int smem_sums) {
  extern __shared__ unsigned long long s_sum[];
  const u32 K = m.K;
  if (smem_sums) {
    for (u32 k = threadIdx.x; k < K; k += blockDim.x) s_sum[k] = 0;
    __syncthreads();
  }
  const u32 w0 = blockIdx.x * rows_per_block;
  const u32 w1 = min(m.V, w0 + rows_per_block);
  phi_rows(K, (u64)w0 * K, (u64)w1 * K, m.n, m.q, m.S, m.tables, (double)m.beta, m.key0, m.key1, t,
           smem_sums ? s_sum : nullptr);
  if (smem_sums) {
    __syncthreads();
    for (u32 k = threadIdx.x; k < K; k += blockDim.x)
      if (s_sum[k]) atomicAdd((unsigned long long*)&m.S[k], s_sum[k]);
  }
}

// Phi draw for K a multiple of 4 (the common case): block (bx, by) draws rows
// [bx * rows, (bx + 1) * rows) of topics [1024 by, 1024 (by + 1)).  A thread
// owns four consecutive topics, of every row of the block or, where a row's
// groups of four do not fill the block, of every 256 / (K / 4)-th: its 16-byte
// loads and stores are contiguous with its neighbours', and it keeps the four
// per-topic sums in registers across its rows (then one 64-bit atomic per block
// and topic, after a sum over the threads of a topic in shared memory where
// there are several).  With one row at a time whatever K, a block of K=20 had 5
// threads at work (K=20, V=5000: 1.7 ms, 36 us now).  Cell c = w K + k uses word
// c & 3 of Philox block c >> 2, exactly as phi_rows, so the draws are the same.
// Rows whose counts each thread loads before drawing any of them: the draw of
// a row waits on its 16-byte load, so loads of several rows in flight hide
// the memory latency one row at a time would expose.  With four rows the loop
// needs about 120 registers (two 256-thread blocks per SM); at 64 registers it
// spilled (mid corpus: 1.75 TB/s of its 12 B per cell against 1.51 TB/s with
// one row at a time and four blocks per SM).
constexpr u32 kPhiRowsInFlight = 4;

// MANY: several rows side by side (K <= 512: one tile).
template <bool MANY>
__global__ void __launch_bounds__(256, 2) phi_draw_cols_kernel(ModelDev m, u32 t, u32 rows_per_block) {
  __shared__ unsigned long long s_sum[MANY ? 512 : 1];
  const u32 K = m.K;
  const u32 groups = MANY ? K / 4 : 256u;         // of a row
  const u32 side = MANY ? 256u / groups : 1u;     // rows side by side
  const u32 r = MANY ? threadIdx.x / groups : 0u;  // this thread's among them
  const u32 k0 = blockIdx.y * 1024u + 4u * (threadIdx.x - r * groups);
  if (MANY) {
    for (u32 i = threadIdx.x; i < K; i += 256) s_sum[i] = 0;
    __syncthreads();
  } else if (k0 >= K) {
    return;
  }
  const u32 w0 = blockIdx.x * rows_per_block + r;
  const u32 w1 = !MANY || r < side ? min(m.V, blockIdx.x * rows_per_block + rows_per_block) : 0u;
  const double beta = (double)m.beta;
  // Most cells hold no tokens, and for n = 0 the inversion returns 0 exactly
  // when the cell's word is below the table's first CDF entry: that entry in
  // a register answers those cells without the guide and CDF loads (K=10000:
  // 4.06 against 3.86 TB/s; no difference at K=1000).
  const u32 cdf00 = __ldg(m.tables.cdf);
  u64 acc[4] = {0, 0, 0, 0};
  for (u32 wb = w0; wb < w1; wb += kPhiRowsInFlight * side) {
    uint4 v[kPhiRowsInFlight];
#pragma unroll
    for (u32 i = 0; i < kPhiRowsInFlight; ++i)
      v[i] = wb + i * side < w1 ? *reinterpret_cast<const uint4*>(m.n + (u64)(wb + i * side) * K + k0)
                                : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (u32 i = 0; i < kPhiRowsInFlight; ++i) {
      if (wb + i * side >= w1) break;
      const u64 cb = (u64)(wb + i * side) * K + k0;
      const U4 r = draw4(cb >> 2, t, kStreamPhi, 0, m.key0, m.key1);
      const u32 nv[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
      u32 xv[4];
#pragma unroll
      for (u32 u = 0; u < 4; ++u) {
        const u32 ru = u4_word(r, u);
        xv[u] = (nv[u] == 0 && ru < cdf00)
                    ? 0u
                    : poisson_draw(nv[u], beta, ru, cb + u, t, kStreamPhi, m.key0, m.key1, m.tables);
        acc[u] += xv[u];
      }
      *reinterpret_cast<uint4*>(m.q + cb) = make_uint4(xv[0], xv[1], xv[2], xv[3]);
      *reinterpret_cast<uint4*>(m.n + cb) = make_uint4(0, 0, 0, 0);
    }
  }
  if (MANY) {
    if (r < side) {
#pragma unroll
      for (u32 u = 0; u < 4; ++u)
        if (acc[u]) atomicAdd(&s_sum[k0 + u], (unsigned long long)acc[u]);
    }
    __syncthreads();
    for (u32 i = threadIdx.x; i < K; i += 256)
      if (s_sum[i]) atomicAdd((unsigned long long*)&m.S[i], s_sum[i]);
    return;
  }
#pragma unroll
  for (u32 u = 0; u < 4; ++u)
    if (acc[u]) atomicAdd((unsigned long long*)&m.S[k0 + u], (unsigned long long)acc[u]);
}

// Batched Phi draw: block b draws rows [w0, w1) (problem-local word ids) of
// problem p, with (p, w0, w1) from the block table.
__global__ void __launch_bounds__(256) phi_draw_batch_kernel(ModelDev ar, BatchPhiDev bp, const u32* t_dev) {
  extern __shared__ unsigned long long s_sum[];
  const uint4 e = bp.blocks[blockIdx.x];
  const u32 pb = e.x, K = bp.K[pb];
  for (u32 k = threadIdx.x; k < K; k += blockDim.x) s_sum[k] = 0;
  __syncthreads();
  const u64 cell0 = bp.cell_base[pb];
  PoisTables tb{bp.cdf + (size_t)pb * kPoisN * kPoisW, bp.guide + (size_t)pb * kPoisN * 256, bp.lfac + (size_t)pb * kLogFacN};
  u64* S = ar.S + bp.S_off[pb];
  phi_rows(K, (u64)e.y * K, (u64)e.z * K, ar.n + cell0, ar.q + cell0, S, tb, (double)bp.beta[pb], bp.key0[pb],
           bp.key1[pb], *t_dev, s_sum);
  __syncthreads();
  for (u32 k = threadIdx.x; k < K; k += blockDim.x)
    if (s_sum[k]) atomicAdd((unsigned long long*)&S[k], s_sum[k]);
}

// ---------------------------------------------------------------------------
// Deterministic parallel alias construction over n items with integer weights
// (reference: build_alias, src/cu/spalias.cu:88-174, which uses atomic work
// queues).  Slot capacity is A = sum_i q_i; item i carries w_i = n*q_i.
// Items with w_i < A are light, the rest heavy, each list in item order.
// The result equals the sequential sweep in which the front heavy fills the
// next light and, on falling below A, is itself filled by the following
// heavy before any further light.  With D_i the exclusive prefix of light
// deficits (A - w) and E_j the inclusive prefix of heavy excesses (w - A):
//   light i  -> alias = heavy j* = min{j : E_j >= D_i}, threshold w_i / A;
//   heavy j with E_j < D_total -> alias = heavy j+1, kept weight
//               A - (D_i + d_i - E_j) with i the light whose deficit interval
//               [D_i, D_i + d_i) contains E_j;
//   other heavies keep the whole slot.
// Every quantity is an exact integer (n <= K <= 32768 keeps n*A below 2^63).
// Entry of item i: threshold | key[i] << 32 | key[alias item] << 48.
// wq[n] holds the weights, key[n] the items' topics; vals[n], idx[n] scratch.
// Block-cooperative.
// ---------------------------------------------------------------------------
__device__ void alias_build_block(const u64* ent, u32 n, u64 A, u64* vals, uint16_t* idx, u64* out, u64* sh) {
  const u32 NT = blockDim.x, tid = threadIdx.x;
  const u32 chunk = (n + NT - 1) / NT;
  const u32 i0 = min(n, tid * chunk), i1 = min(n, i0 + chunk);
  u64 nl = 0, dl = 0, nh = 0, eh = 0;
  for (u32 i = i0; i < i1; ++i) {
    const u64 wi = (u64)n * (ent[i] >> 32);
    if (wi < A) {
      ++nl;
      dl += A - wi;
    } else {
      ++nh;
      eh += wi - A;
    }
  }
  u64 nL, Dtot, nH, Etot;
  u64 ol = block_excl_scan_u64(nl, sh, &nL);
  u64 od = block_excl_scan_u64(dl, sh, &Dtot);
  u64 oh = block_excl_scan_u64(nh, sh, &nH);
  u64 oe = block_excl_scan_u64(eh, sh, &Etot);
  for (u32 i = i0; i < i1; ++i) {
    const u64 wi = (u64)n * (ent[i] >> 32);
    if (wi < A) {
      vals[ol] = od;
      idx[ol] = (uint16_t)i;
      od += A - wi;
      ++ol;
    } else {
      oe += wi - A;
      vals[nL + oh] = oe;
      idx[nL + oh] = (uint16_t)i;
      ++oh;
    }
  }
  __syncthreads();
  const u64* Ev = vals + nL;
  const uint16_t* Hi = idx + nL;
  auto key = [&](u32 i) -> u64 { return ent[i] & 0xffffu; };
  for (u32 i = tid; i < (u32)nL; i += NT) {
    const u64 D = vals[i];
    u32 lo = 0, hi = (u32)nH - 1;  // first j with E_j >= D (exists: D < Dtot = E_last)
    while (lo < hi) {
      const u32 mid = (lo + hi) >> 1;
      if (Ev[mid] >= D) hi = mid; else lo = mid + 1;
    }
    const u32 l = idx[i];
    out[l] = (key(Hi[lo]) << 48) | (key(l) << 32) | alias_threshold((u64)n * (ent[l] >> 32), A);
  }
  for (u32 j = tid; j < (u32)nH; j += NT) {
    const u32 h = Hi[j];
    const u64 E = Ev[j];
    if (E < Dtot) {
      u32 lo = 0, hi = (u32)nL - 1;  // last i with D_i <= E (D_0 = 0)
      while (lo < hi) {
        const u32 mid = (lo + hi + 1) >> 1;
        if (vals[mid] <= E) lo = mid; else hi = mid - 1;
      }
      const u64 d = A - (u64)n * (ent[idx[lo]] >> 32);
      const u64 over = vals[lo] + d - E;
      out[h] = (key(Hi[j + 1]) << 48) | (key(h) << 32) | alias_threshold(A - over, A);
    } else {
      out[h] = (key(h) << 48) | (key(h) << 32) | 0xffffffffu;
    }
  }
}

// q = floor(x * 2^32 / S[k]), clamped to 32 bits.
__device__ __forceinline__ u64 fixed_phi(u32 x, u32 k, const u64* __restrict__ S, const u64* __restrict__ Sinv) {
  const u64 num = (u64)x << 32, sk = S[k];
  u64 qq;
  if (Sinv) {
    // floor(num / sk) from the reciprocal: the multiply-high is at most 2
    // below the quotient
    qq = __umul64hi(num, Sinv[k]);
    u64 r = num - qq * sk;
    if (r >= sk) {
      ++qq;
      r -= sk;
    }
    if (r >= sk) ++qq;
  } else {
    qq = num / sk;
  }
  return qq > 0xffffffffULL ? 0xffffffffULL : qq;
}

// Per word: q = floor(x * 2^32 / S[k]) (clamped) written back densely; the
// word's topics with q > 0 compacted in ascending order into its list
// (q << 32 | k, which is also the alias build's input), the dense mass A, nnz,
// and the sparse alias table over the list.  The dense pass gives each thread
// kPerThread consecutive topics per tile, so a tile needs one block scan.
// The alias build's scratch (10 bytes per nonzero) is shared memory when the
// word's nonzeros fit smem_items, else the block's slice of global scratch.
// listed: the draws (x << 32 | k) that stand in csrrow already, all of the row's,
// or 0.
constexpr u32 kPerThread = 8;
constexpr u32 kAliasWarps = 4;  // a block's, a word each
// Most topics of a word that a warp takes (18 bytes each set how many warps are
// resident); a longer word takes a block, above K = 2048 of a launch of its own.
// K=1000: 128, 256 and 512 take 218, 210 and 243 us at the mid corpus; K=10000,
// whose words' lists are longer, before that launch: 1350, 900 and 700 us.
inline u32 alias_items(u32 K) { return std::min(K, K <= kMapMinK ? 256u : 512u); }
__host__ __device__ constexpr size_t alias_warp_bytes(u32 most) { return ((size_t)most * 18 + 15) & ~(size_t)15; }

// Sets the bits of a list's topics; the first of the entries of a 32-bit word
// writes it.
__device__ __forceinline__ void list_bits(const u64* ent, u32 n, u32* bits, u32 first, u32 step) {
  for (u32 i = first; i < n; i += step) {
    const u32 at = ((u32)ent[i] & 0xffffu) >> 5;
    if (i && ((u32)ent[i - 1] & 0xffffu) >> 5 == at) continue;
    u32 b = 0;
    for (u32 j = i; j < n && ((u32)ent[j] & 0xffffu) >> 5 == at; ++j) b |= 1u << (ent[j] & 31);
    bits[at] = b;
  }
}

__device__ __forceinline__ void alias_word(u32 K, u32* __restrict__ qrow, const u64* __restrict__ S,
                                           const u64* __restrict__ Sinv, u64* alrow, u64* csrrow, u64* eighths,
                                           u32* bits, u64* A_out, u64* s_shares, u32* nnz_out, u32 listed,
                                           u64* s_vals, uint16_t* s_idx, u32 smem_items, u64* g_vals, uint16_t* g_idx,
                                           u64* sh) {
  u64 part = 0, nz = 0;
  u32 xsum = 0;
  if (bits)
    for (u32 i = threadIdx.x; i < bits_stride(K); i += blockDim.x) bits[i] = 0;
  if (listed) {
    bool zero = false;
    for (u32 i = threadIdx.x; i < listed; i += blockDim.x) {
      const u64 e = csrrow[i];
      const u64 qq = fixed_phi((u32)(e >> 32), (u32)e, S, Sinv);
      zero |= !qq;
      part += qq;
      xsum += (u32)(e >> 32);
      csrrow[i] = (qq << 32) | (u32)e;
    }
    if (__syncthreads_or(zero)) {  // a draw that rounds to q = 0 is not in the list: from the row, still as drawn
      listed = 0;
      part = 0;
      xsum = 0;
    } else {
      for (u32 i = threadIdx.x; i < listed; i += blockDim.x) qrow[(u32)csrrow[i]] = (u32)(csrrow[i] >> 32);
      nz = listed;
    }
  }
  const u32 tile = blockDim.x * kPerThread;
  for (u32 t0 = 0; !listed && t0 < K; t0 += tile) {
    const u32 k0 = t0 + threadIdx.x * kPerThread;
    u32 qv[kPerThread];
    u32 cnt = 0;
#pragma unroll
    for (u32 c = 0; c < kPerThread; ++c) {
      const u32 k = k0 + c;
      u64 qq = 0;
      if (k < K) {
        const u32 x = qrow[k];
        if (x) {  // a zero count is already a zero q
          xsum += x;
          qq = fixed_phi(x, k, S, Sinv);
          qrow[k] = (u32)qq;
        }
      }
      qv[c] = (u32)qq;
      cnt += qq != 0;
      part += qq;
    }
    u64 tot;
    u64 pos = nz + block_excl_scan_u64(cnt, sh, &tot);
#pragma unroll
    for (u32 c = 0; c < kPerThread; ++c)
      if (qv[c]) csrrow[pos++] = ((u64)qv[c] << 32) | (k0 + c);
    nz += tot;
  }
  const u64 A = block_sum_u64(part, sh);  // (also orders the list writes before the build)
  const u32 n = (u32)nz;
  if (bits) list_bits(csrrow, n, bits, threadIdx.x, blockDim.x);
  if (s_shares) {  // the word's tokens (its draws' sum), by its list's length
    xsum = __reduce_add_sync(kFullMask, xsum);
    if ((threadIdx.x & 31) == 0) {
      atomicAdd((unsigned long long*)s_shares, (unsigned long long)xsum);
      if (n > kShortList)
        atomicAdd((unsigned long long*)s_shares + 1, (unsigned long long)xsum * long_list_weight(n));
    }
  }
  if (eighths && n) {  // the list again, by eighths, with zeros to the end of the last
    const u32 c = list_pairs(n), recip = list_recip(c);
    const u32 end = (((n - 1) / 2 * recip >> 20) + 1) * 2 * c;
    for (u32 i = threadIdx.x; i < end; i += blockDim.x)
      eighths[list_pos(i, c, recip)] = i < n ? csrrow[i] : 0ull;
  }
  if (n) {
    const bool in_smem = n <= smem_items;
    alias_build_block(csrrow, n, A, in_smem ? s_vals : g_vals, in_smem ? s_idx : g_idx, alrow, sh);
  }
  if (threadIdx.x == 0) {
    *A_out = A;
    *nnz_out = n;
  }
  __syncthreads();
}

constexpr u32 kNnzWide = 0x80000000u;  // marks a word that its warp left to a block, beside its listed draws

// The aligned groups of four cells that a row lies in; it starts at cell `head` of
// the first.
__device__ __forceinline__ u32 row_head(const u32* qrow) { return (u32)((uintptr_t)qrow >> 2) & 3; }
__device__ __forceinline__ u32 row_groups(const u32* qrow, u32 K) { return (K + row_head(qrow) + 3) / 4; }

// Goes on through a row from its aligned group `g` of four cells: put(i, x << 32 | k)
// for its i-th nonzero draw, i from n on.  Returns their number; where that would
// pass `most`, the number before the groups from `g` on, else `g` is past the row.
template <class Put>
__device__ __forceinline__ u32 row_draws(const u32* qrow, u32 K, u32& g, u32 n, u32 most, Put put) {
  constexpr u32 kInFlight = 4;  // loads of 512 bytes; 8 take registers and a resident block (mid 212 -> 239 us)
  const u32 lane = threadIdx.x & 31, before = (1u << lane) - 1;
  const u32 head = row_head(qrow), groups = row_groups(qrow, K);
  for (; g < groups; g += 32 * kInFlight) {
    u32 v[kInFlight][4];
#pragma unroll
    for (u32 u = 0; u < kInFlight; ++u) {
      const i32 k = (i32)(4 * (g + 32 * u + lane)) - (i32)head;
      if (k >= 0 && k + 4 <= (i32)K) {
        const uint4 x = *reinterpret_cast<const uint4*>(qrow + k);
        v[u][0] = x.x, v[u][1] = x.y, v[u][2] = x.z, v[u][3] = x.w;
      } else {
#pragma unroll
        for (i32 c = 0; c < 4; ++c) v[u][c] = k + c >= 0 && k + c < (i32)K ? qrow[k + c] : 0u;
      }
    }
#pragma unroll
    for (u32 u = 0; u < kInFlight; ++u) {
      const u32 cnt = (v[u][0] != 0) + (v[u][1] != 0) + (v[u][2] != 0) + (v[u][3] != 0);
      if (!__any_sync(kFullMask, cnt)) continue;
      const u32 b0 = __ballot_sync(kFullMask, cnt & 1), b1 = __ballot_sync(kFullMask, cnt & 2),
                b2 = __ballot_sync(kFullMask, cnt & 4);
      u32 pos = n + __popc(b0 & before) + 2 * __popc(b1 & before) + 4 * __popc(b2 & before);
      const u32 after = n + __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2);
      if (after > most) {
        g += 32 * u;
        return n;
      }
      n = after;
      const u32 k = 4 * (g + 32 * u + lane) - head;
#pragma unroll
      for (u32 c = 0; c < 4; ++c)
        if (v[u][c]) put(pos++, ((u64)v[u][c] << 32) | (k + c));
    }
  }
  return n;
}

// The rest of a row of too many draws for the warp's memory: ent's n, then those
// from group `g` on, to the word's list.  Returns the word's marked number.
static __device__ __noinline__ u32 list_wide(const u32* qrow, u32 K, u32 g, const u64* ent, u32 n, u64* csrrow) {
  __syncwarp();
  for (u32 i = threadIdx.x & 31; i < n; i += 32) csrrow[i] = ent[i];
  return kNnzWide | row_draws(qrow, K, g, n, ~0u, [&](u32 i, u64 e) { csrrow[i] = e; });
}

// The same by one warp, for a word of at most `most` topics.  Returns 0, or
// kNnzWide for a word that is left to a block: with nothing written if a draw
// rounds to q = 0 (a topic's sum above 2^32) or there are too many in the first
// `from` halves of the row, else with their number beside it and the draws
// (x << 32 | k) listed in csrrow.  (Above K = 2048 all such rows are listed: K=4096,
// 2,000 words of 640 topics 66 us, 85 if the block looks through the row again;
// K=10000, 10,000 words of 750 349 and 646.  A block of the same launch looks
// through the rest of a row faster than a warp lists it, so there rows that are
// half done are: K=2000, 2,000 words of 320 topics 38 and 52 us, but 20,000 words
// from a random start 185 and 170.)  A trained word has some tens of topics, so a
// block on it waited at barriers: six scans of eight warps' sums for one or two
// entries a lane.  Here the row is only looked through for its nonzero draws,
// and everything after works on those: ent[most] holds them, vals and idx are
// the alias build's scratch, all the warp's own.  Bound by instructions (about
// 1,500 a word beside 4 KB of row at K=1000).  1e5 words of 65 topics (K=1000)
// 622 -> 212 us, 1.4e5 words 816 -> 259; 3e4 words, K=10000, 1185 -> 726 us
// where the rows' 1.2 GB take 183; from a random start (50,000 words of 100
// to 1000 topics) 337 -> 146.
__device__ __forceinline__ u32 alias_word_warp(u32 K, u32* qrow, const u64* __restrict__ S,
                                               const u64* __restrict__ Sinv, u64* alrow, u64* csrrow, u64* eighths,
                                               u32* bits, u64* A_out, u32* nnz_out, u64& x_all, u64& x_long, u64* ent,
                                               u64* vals, uint16_t* idx, u32 most, u32 from) {
  const u32 lane = threadIdx.x & 31;
  u32 g = 0;
  const u32 n = row_draws(qrow, K, g, 0, most, [&](u32 i, u64 e) { ent[i] = e; });
  const u32 groups = row_groups(qrow, K);
  if (g < groups) return g >= from * groups / 2 ? list_wide(qrow, K, g, ent, n, csrrow) : kNnzWide;
  __syncwarp();
  u64 part = 0, xsum = 0;
  bool zero = false;
  for (u32 i = lane; i < n; i += 32) {
    const u64 e = ent[i];
    const u64 qq = fixed_phi((u32)(e >> 32), (u32)e, S, Sinv);
    zero |= !qq;
    part += qq;
    xsum += e >> 32;
    ent[i] = (qq << 32) | (u32)e;
  }
  if (__any_sync(kFullMask, zero)) return kNnzWide;
  __syncwarp();
  const u64 A = warp_sum_u64(part);
  x_all += xsum;
  x_long += xsum * long_list_weight(n);
  for (u32 i = lane; i < n; i += 32) {
    const u64 e = ent[i];
    qrow[(u32)e] = (u32)(e >> 32);
    csrrow[i] = e;
  }
  if (bits) {
    for (u32 i = lane; i < bits_stride(K) / 4; i += 32) reinterpret_cast<uint4*>(bits)[i] = make_uint4(0, 0, 0, 0);
    __syncwarp();
    list_bits(ent, n, bits, lane, 32);
  }
  if (eighths && n) {  // as alias_word
    const u32 c = list_pairs(n), recip = list_recip(c);
    const u32 end = (((n - 1) / 2 * recip >> 20) + 1) * 2 * c;
    for (u32 i = lane; i < end; i += 32) eighths[list_pos(i, c, recip)] = i < n ? ent[i] : 0ull;
  }
  if (lane == 0) {
    *A_out = A;
    *nnz_out = n;
  }
  if (!n) return 0;
  // alias_build_block's steps
  const u32 chunk = (n + 31) / 32, i0 = min(n, lane * chunk), i1 = min(n, i0 + chunk);
  u32 nl = 0;
  u64 dl = 0, eh = 0;
  for (u32 i = i0; i < i1; ++i) {
    const u64 wi = (u64)n * (ent[i] >> 32);
    if (wi < A) {
      ++nl;
      dl += A - wi;
    } else {
      eh += wi - A;
    }
  }
  u32 ol = nl;
#pragma unroll
  for (u32 d = 1; d < 32; d *= 2) {
    const u32 o = __shfl_up_sync(kFullMask, ol, d);
    if (lane >= d) ol += o;
  }
  const u32 nL = __shfl_sync(kFullMask, ol, 31);
  ol -= nl;
  u64 od = warp_incl_scan_u64(dl, lane);
  const u64 Dtot = __shfl_sync(kFullMask, (unsigned long long)od, 31);
  od -= dl;
  u64 oe = warp_incl_scan_u64(eh, lane) - eh;
  u32 oh = nL + i0 - ol;
  for (u32 i = i0; i < i1; ++i) {
    const u64 wi = (u64)n * (ent[i] >> 32);
    if (wi < A) {
      vals[ol] = od;
      idx[ol++] = (uint16_t)i;
      od += A - wi;
    } else {
      oe += wi - A;
      vals[oh] = oe;
      idx[oh++] = (uint16_t)i;
    }
  }
  __syncwarp();
  for (u32 j = lane; j < n; j += 32) {
    const u32 i = idx[j];
    const u64 e = ent[i], v = vals[j], own = e & 0xffffu;
    if (j < nL) {
      u32 lo = nL, hi = n - 1;  // the first heavy with E >= D
      while (lo < hi) {
        const u32 mid = (lo + hi) >> 1;
        if (vals[mid] >= v) hi = mid; else lo = mid + 1;
      }
      alrow[i] = ((ent[idx[lo]] & 0xffffu) << 48) | (own << 32) | alias_threshold((u64)n * (e >> 32), A);
    } else if (v < Dtot) {
      u32 lo = 0, hi = nL - 1;  // the last light with D <= E (D_0 = 0)
      while (lo < hi) {
        const u32 mid = (lo + hi + 1) >> 1;
        if (vals[mid] <= v) lo = mid; else hi = mid - 1;
      }
      const u64 d = A - (u64)n * (ent[idx[lo]] >> 32);
      const u64 over = vals[lo] + d - v;
      alrow[i] = ((ent[idx[j + 1]] & 0xffffu) << 48) | (own << 32) | alias_threshold(A - over, A);
    } else {
      alrow[i] = (own << 48) | (own << 32) | 0xffffffffu;
    }
  }
  __syncwarp();
  return 0;
}

// The block's alias scratch for one word of up to `items` topics.
struct AliasScratch {
  u64* vals;
  uint16_t* idx;
};
__device__ __forceinline__ AliasScratch alias_scratch_at(unsigned char* raw, u32 items) {
  AliasScratch a;
  a.vals = (u64*)raw;
  a.idx = (uint16_t*)(a.vals + items);
  return a;
}

// A block's shared memory: its warps' scratch, or all of it for one word.
struct AliasSmem {
  u64 *ent, *vals;      // this warp's
  uint16_t* idx;
  AliasScratch all;     // the block's
};
__device__ __forceinline__ AliasSmem alias_smem(unsigned char* raw, u32 most, u32 items) {
  AliasSmem a;
  unsigned char* own = raw + (size_t)(threadIdx.x >> 5) * alias_warp_bytes(most);
  a.ent = (u64*)own;
  a.vals = a.ent + most;
  a.idx = (uint16_t*)(a.vals + most);
  a.all = alias_scratch_at(raw, items);
  return a;
}

// The i-th of a block's words: four neighbours at a time, or (spread) every
// gridDim-th.  Words are ranked by frequency, so those with many topics are
// neighbours, and a block builds those that its warps leave one after another.
__device__ __forceinline__ u64 alias_nth(u32 i, bool spread) {
  if (spread) return blockIdx.x + (u64)i * gridDim.x;
  return ((u64)(i / kAliasWarps) * gridDim.x + blockIdx.x) * kAliasWarps + i % kAliasWarps;
}

// Blocks of an alias build over V words with room for `resident` of them on the
// GPU, and whether they spread: with few words, so that each block has about one
// of many topics (K=2000, 2,000 words of 320 topics: 75 us with four neighbours to
// a block, 52 spread, when each still looked through its row again).  With many,
// the blocks are enough, and neighbours cost less (1e5 words 259 us, 269 spread).
struct AliasGrid {
  u32 blocks;
  bool spread;
};
inline AliasGrid alias_grid(u32 V, u32 K, u32 most, u32 resident) {
  AliasGrid g;
  g.spread = K > most && V < 16 * resident;
  g.blocks = std::max((V + kAliasWarps - 1) / kAliasWarps, g.spread ? std::min(V, resident) : 1u);
  g.blocks = std::min(g.blocks, 4 * resident);
  return g;
}

// f(w) for the block's words of [w0, w1) that are marked, every gridDim-th, all
// threads together.
template <class F>
__device__ __forceinline__ void for_wide_words(const u32* nnz, u64 w0, u64 w1, F&& f) {
  __shared__ u32 marked[8];  // by warp
  const u32 nw = blockDim.x >> 5;
  for (u64 first = w0 + blockIdx.x; first < w1; first += (u64)gridDim.x * blockDim.x) {
    const u64 w = first + (u64)threadIdx.x * gridDim.x;
    const u32 b = __ballot_sync(kFullMask, w < w1 && (nnz[w] & kNnzWide));
    if ((threadIdx.x & 31) == 0) marked[threadIdx.x >> 5] = b;
    __syncthreads();
    for (u32 i = 0; i < nw; ++i)
      for (u32 left = marked[i]; left; left &= left - 1)
        f(first + (u64)(32 * i + (u32)__ffs((int)left) - 1) * gridDim.x);
    __syncthreads();
  }
}

// Word w of the model by the block; g: its slice of global scratch.
__device__ __forceinline__ void alias_word_of(const ModelDev& m, u64 w, u64* s_shares, const AliasScratch& all,
                                              u32 smem_items, unsigned char* g, u64* sh) {
  const u32 K = m.K;
  const size_t row = (size_t)w * K;
  alias_word(K, m.q + row, m.S, m.Sinv, m.al + row, m.csr + row,
             m.lists ? m.lists + (size_t)w * list_stride(K) : nullptr,
             m.bits ? m.bits + (size_t)w * bits_stride(K) : nullptr, m.A + w, s_shares, m.nnz + w,
             m.nnz[w] & ~kNnzWide, all.vals, all.idx, smem_items, (u64*)g, g ? (uint16_t*)((u64*)g + K) : nullptr, sh);
}

// Word w of a batch.
__device__ __forceinline__ void alias_word_of(const ModelDev& ar, const BatchPhiDev& bp, u64 w, u64* s_shares,
                                              const AliasScratch& all, u32 smem_items, u64* sh) {
  const u32 pb = bp.wpid[w];
  const size_t row = bp.row_off[w];
  alias_word(bp.K[pb], ar.q + row, ar.S + bp.S_off[pb], nullptr, ar.al + row, ar.csr + row,
             ar.lists ? ar.lists + bp.list_off[w] : nullptr, nullptr, ar.A + w, s_shares, ar.nnz + w,
             ar.nnz[w] & ~kNnzWide, all.vals, all.idx, smem_items, nullptr, nullptr, sh);
}

// items: most topics of a word that the block takes (at least K, or 0: those that
// its warps leave are alias_wide_kernel's).
__global__ void __launch_bounds__(32 * kAliasWarps, 8) alias_build_kernel(ModelDev m, u32 most, u32 items,
                                                                       bool spread) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ u64 sh[33], sh_shares[2];
  __shared__ u32 wide;
  const u32 K = m.K, warp = threadIdx.x >> 5;
  if (threadIdx.x < 2) sh_shares[threadIdx.x] = 0;
  if (threadIdx.x == 0) wide = 0;
  __syncthreads();
  const AliasSmem sm = alias_smem(s_raw, most, items);
  u64 x_all = 0, x_long = 0;
  u64 w;
  for (u32 i = warp; (w = alias_nth(i, spread)) < m.V; i += kAliasWarps) {
    const size_t row = (size_t)w * K;
    const u32 left = alias_word_warp(K, m.q + row, m.S, m.Sinv, m.al + row, m.csr + row,
                                     m.lists ? m.lists + (size_t)w * list_stride(K) : nullptr,
                                     m.bits ? m.bits + (size_t)w * bits_stride(K) : nullptr, m.A + w, m.nnz + w, x_all,
                                     x_long, sm.ent, sm.vals, sm.idx, most, items ? 1u : 0u);
    if (!left) continue;
    if ((threadIdx.x & 31) == 0) {
      m.nnz[w] = left;
      wide = 1;
    }
    __syncwarp();
  }
  if (m.shares) {
    x_all = warp_sum_u64(x_all);
    x_long = warp_sum_u64(x_long);
    if ((threadIdx.x & 31) == 0) {
      atomicAdd((unsigned long long*)sh_shares, (unsigned long long)x_all);
      atomicAdd((unsigned long long*)sh_shares + 1, (unsigned long long)x_long);
    }
  }
  __syncthreads();
  if (wide && items) {
    for (u32 i = 0; (w = alias_nth(i, spread)) < m.V; ++i)
      if (m.nnz[w] & kNnzWide) alias_word_of(m, w, m.shares ? sh_shares : nullptr, sm.all, items, nullptr, sh);
    __syncthreads();
  }
  if (m.shares && threadIdx.x < 2)
    atomicAdd((unsigned long long*)m.shares + threadIdx.x, (unsigned long long)sh_shares[threadIdx.x]);
}

// The words that alias_build_kernel's warps left, a block to each, K > 2048 (where
// a word may need the block's slice of global scratch): K=4096, 2,000 words of 640
// topics, 66 us together (140 with four of them to a block of that kernel);
// K=12000, 1,000 words of 750, 69 (267); K=10000, 10,000 of 750, 348 (1337).  Bound
// by load latency and barriers.
__global__ void __launch_bounds__(256) alias_wide_kernel(ModelDev m, unsigned char* gscratch, size_t slice,
                                                         u32 smem_items) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ u64 sh[33];
  const AliasScratch all = alias_scratch_at(s_raw, smem_items);
  unsigned char* g = gscratch + (size_t)blockIdx.x * slice;
  for_wide_words(m.nnz, 0, m.V, [&](u64 w) { alias_word_of(m, w, nullptr, all, smem_items, g, sh); });
}

// Batched alias build over global words [w0, w1) of any problems; shared
// memory sized for the largest K among them.
__global__ void __launch_bounds__(32 * kAliasWarps, 8) alias_build_batch_kernel(ModelDev ar, BatchPhiDev bp, u32 most,
                                                                             u32 Kmax, u32 w0, u32 w1, bool spread) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ u64 sh[33], sh_shares[2];
  __shared__ u32 wide;
  const u32 warp = threadIdx.x >> 5;
  if (threadIdx.x < 2) sh_shares[threadIdx.x] = 0;
  if (threadIdx.x == 0) wide = 0;
  __syncthreads();
  const AliasSmem sm = alias_smem(s_raw, most, Kmax);
  u64 x_all = 0, x_long = 0;
  u64 w;
  for (u32 i = warp; (w = w0 + alias_nth(i, spread)) < w1; i += kAliasWarps) {
    const u32 pb = bp.wpid[w], K = bp.K[pb];
    const size_t row = bp.row_off[w];
    const u32 left = alias_word_warp(K, ar.q + row, ar.S + bp.S_off[pb], nullptr, ar.al + row, ar.csr + row,
                                     ar.lists ? ar.lists + bp.list_off[w] : nullptr, nullptr, ar.A + w, ar.nnz + w,
                                     x_all, x_long, sm.ent, sm.vals, sm.idx, most, 1u);
    if (!left) continue;
    if ((threadIdx.x & 31) == 0) {
      ar.nnz[w] = left;
      wide = 1;
    }
    __syncwarp();
  }
  x_all = warp_sum_u64(x_all);
  x_long = warp_sum_u64(x_long);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd((unsigned long long*)sh_shares, (unsigned long long)x_all);
    atomicAdd((unsigned long long*)sh_shares + 1, (unsigned long long)x_long);
  }
  __syncthreads();
  if (wide) {
    for (u32 i = 0; (w = w0 + alias_nth(i, spread)) < w1; ++i)
      if (ar.nnz[w] & kNnzWide) alias_word_of(ar, bp, w, sh_shares, sm.all, Kmax, sh);
    __syncthreads();
  }
  if (threadIdx.x < 2)
    atomicAdd((unsigned long long*)ar.shares + threadIdx.x, (unsigned long long)sh_shares[threadIdx.x]);
}

// Reciprocals of the per-topic normalisers, inv[k] = floor((2^64 - 1) / S[k])
// (0 for an empty topic): the alias build then divides by a multiply-high and
// at most two corrections instead of a 64-bit division per nonzero cell.
__global__ void topic_recip_kernel(const u64* __restrict__ S, u64* __restrict__ inv, u32 K) {
  const u32 k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < K) {
    const u64 sk = S[k];
    inv[k] = sk ? ~0ull / sk : 0ull;
  }
}

// Advances a device-side iteration counter (replayed graphs read it).
__global__ void bump_kernel(u32* t) { *t += 1; }

__global__ void debug_alias_kernel(const u32* q, u32 K, u64* out) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ u64 sh[33];
  u64* ent = (u64*)s_raw;  // (q << 32 | item)
  u64* vals = ent + K;
  uint16_t* idx = (uint16_t*)(vals + K);
  u64 part = 0;
  for (u32 k = threadIdx.x; k < K; k += blockDim.x) {
    ent[k] = ((u64)q[k] << 32) | k;
    part += q[k];
  }
  const u64 A = block_sum_u64(part, sh);
  alias_build_block(ent, K, A, vals, idx, out, sh);
}

// ---------------------------------------------------------------------------
// Document offsets (reference: compute_d_idx, src/cu/topics.cu:5-32).
// One block; each thread scans a contiguous chunk.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) doc_offsets_kernel(const u32* __restrict__ d_len, u32* __restrict__ d_idx,
                                                           u32 n_docs) {
  __shared__ u64 sh[33];
  const u32 chunk = (n_docs + blockDim.x - 1) / blockDim.x;
  const u32 i0 = min(n_docs, threadIdx.x * chunk), i1 = min(n_docs, i0 + chunk);
  u64 s = 0;
  for (u32 i = i0; i < i1; ++i) s += d_len[i];
  u64 total;
  u64 off = block_excl_scan_u64(s, sh, &total);
  for (u32 i = i0; i < i1; ++i) {
    // Saturate instead of wrapping: buffers hold fewer than 2^32 tokens, so an
    // offset of 2^32 - 1 fails the sweep's range check (offset + length must
    // not pass n_tokens) and is reported, where a wrapped offset could pass it.
    d_idx[i] = off < 0xffffffffull ? (u32)off : 0xffffffffu;
    off += d_len[i];
  }
}

// ---------------------------------------------------------------------------
// Document offsets, and the documents longest first, for lengths that are on
// the device only.  Three launches over blocks of kPlanDocs documents: token
// sums per block and a histogram of lengths; a scan of both; offsets and places
// in the order.  The order is by length bins (exact below 512 tokens, 128 tokens
// wide above), in no particular order inside a bin.  Bound by its launches (three
// of 3 us at 6e4 documents; one block scanning them all took 14 us).
// ---------------------------------------------------------------------------
constexpr u32 kPlanThreads = 256, kPlanDocs = 4096, kPlanBins = 1024;
static_assert(kPlanMostDocs <= kPlanDocs * kPlanBins, "the scan's block takes a block sum per thread");

// The bin of a length, longest first.
__host__ __device__ __forceinline__ u32 plan_bin(u32 len) {
  const u32 up = len < 512 ? len : 512 + (len - 512) / 128;
  return kPlanBins - 1 - (up < kPlanBins ? up : kPlanBins - 1);
}

__global__ void __launch_bounds__(kPlanThreads) doc_survey_kernel(const u32* __restrict__ d_len, u32 n_docs,
                                                                  DocPlan plan) {
  __shared__ u32 hist[kPlanBins];
  __shared__ u64 sh[33];
  for (u32 i = threadIdx.x; i < kPlanBins; i += kPlanThreads) hist[i] = 0;
  __syncthreads();
  u64 sum = 0;
  const u32 d1 = min(n_docs, (blockIdx.x + 1) * kPlanDocs);
  for (u32 d = blockIdx.x * kPlanDocs + threadIdx.x; d < d1; d += kPlanThreads) {
    const u32 len = d_len[d];
    sum += len;
    atomicAdd(hist + plan_bin(len), 1u);
  }
  sum = block_sum_u64(sum, sh);  // (orders the histogram before its flush)
  if (threadIdx.x == 0) plan.sums[blockIdx.x] = sum;
  for (u32 i = threadIdx.x; i < kPlanBins; i += kPlanThreads)
    if (hist[i]) atomicAdd(plan.bins + i, hist[i]);
}

// plan.sums and plan.bins become exclusive prefixes; *n_long receives the
// documents in the bins before long_bin's end.
__global__ void __launch_bounds__(kPlanBins) doc_scan_kernel(u32 n_blocks, u32 long_bin, DocPlan plan) {
  __shared__ u64 sh[33];
  const u32 i = threadIdx.x;
  u64 total;
  const u64 s0 = block_excl_scan_u64(i < n_blocks ? plan.sums[i] : 0, sh, &total);
  const u32 here = plan.bins[i];
  const u64 b0 = block_excl_scan_u64(here, sh, &total);
  if (i < n_blocks) plan.sums[i] = s0;
  plan.bins[i] = (u32)b0;
  if (i == long_bin) *plan.n_long = (u32)b0 + here;
}

__global__ void __launch_bounds__(kPlanThreads) doc_place_kernel(const u32* __restrict__ d_len, u32 n_docs,
                                                                 u32* __restrict__ d_idx, u32* __restrict__ order,
                                                                 DocPlan plan) {
  __shared__ u32 lens[kPlanDocs];
  __shared__ u32 bins[kPlanBins];  // the block's documents of a bin, then their next place
  __shared__ u64 sh[33];
  const u32 d0 = blockIdx.x * kPlanDocs, n = min(kPlanDocs, n_docs - d0);
  for (u32 i = threadIdx.x; i < kPlanBins; i += kPlanThreads) bins[i] = 0;
  __syncthreads();
  for (u32 i = threadIdx.x; i < n; i += kPlanThreads) {
    lens[i] = d_len[d0 + i];
    atomicAdd(bins + plan_bin(lens[i]), 1u);
  }
  __syncthreads();
  for (u32 i = threadIdx.x; i < kPlanBins; i += kPlanThreads)
    if (bins[i]) bins[i] = atomicAdd(plan.bins + i, bins[i]);
  constexpr u32 kEach = kPlanDocs / kPlanThreads;
  const u32 i0 = min(n, threadIdx.x * kEach), i1 = min(n, i0 + kEach);
  u64 s = 0;
  for (u32 i = i0; i < i1; ++i) s += lens[i];
  u64 total;
  u64 off = plan.sums[blockIdx.x] + block_excl_scan_u64(s, sh, &total);  // (orders the bins' places too)
  for (u32 i = i0; i < i1; ++i) {
    d_idx[d0 + i] = off < 0xffffffffull ? (u32)off : 0xffffffffu;  // as doc_offsets_kernel
    off += lens[i];
    order[atomicAdd(bins + plan_bin(lens[i]), 1u)] = d0 + i;
  }
}

// ---------------------------------------------------------------------------
// Count rebuild n[w][z] += 1 over a token range (reference: the atomicAdd per
// token at the end of sample_topics, src/cu/topics.cu:95).  Tokens are read
// four at a time (16-byte loads of w and z); per load slot the warp groups
// lanes whose tokens hit the same cell (__match_any_sync) and the group's
// lowest lane adds the group's size: one atomic per distinct cell per warp
// step instead of one per token.  Topics >= K and words >= V are reported
// and counted modulo K / V, like the sweeps.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) count_rebuild_kernel(u32* __restrict__ n, const u32* __restrict__ w,
                                                            const u32* __restrict__ z, u64 n_tokens, u32 K, u32 V,
                                                            u32* status) {
  const u32 lane = threadIdx.x & 31;
  const u64 groups = (n_tokens + 3) / 4;
  const u64 stride = (u64)gridDim.x * blockDim.x;
  u32 st = 0;
  // warp-uniform trip count: every lane of a warp takes the same number of steps
  const u64 g0 = (u64)blockIdx.x * blockDim.x + (threadIdx.x & ~31u);
  for (u64 gb = g0; gb < groups; gb += stride) {
    const u64 gi = gb + lane;
    u32 wv[4] = {0, 0, 0, 0}, zv[4] = {0, 0, 0, 0};
    u32 nv = 0;  // tokens of this group
    if (gi < groups) {
      const u64 t0 = gi * 4;
      nv = (u32)(n_tokens - t0 < 4 ? n_tokens - t0 : 4);
      if (nv == 4) {
        const uint4 a = *reinterpret_cast<const uint4*>(w + t0);
        const uint4 b = *reinterpret_cast<const uint4*>(z + t0);
        wv[0] = a.x, wv[1] = a.y, wv[2] = a.z, wv[3] = a.w;
        zv[0] = b.x, zv[1] = b.y, zv[2] = b.z, zv[3] = b.w;
      } else {
        for (u32 u = 0; u < nv; ++u) {
          wv[u] = w[t0 + u];
          zv[u] = z[t0 + u];
        }
      }
    }
#pragma unroll
    for (u32 u = 0; u < 4; ++u) {
      const bool on = u < nv;
      u32 wu = wv[u], zu = zv[u];
      if (on && wu >= V) {
        st |= kStatusBadWord;
        wu %= V;
      }
      if (on && zu >= K) {
        st |= kStatusBadTopic;
        zu %= K;
      }
      // lanes without a token get distinct keys that match no cell
      const u64 cell = on ? (u64)wu * K + zu : ~(u64)lane;
      const u32 peers = __match_any_sync(kFullMask, cell);
      if (on && lane == (u32)(__ffs(peers) - 1)) atomicAdd(n + cell, (u32)__popc(peers));
    }
  }
  st = __reduce_or_sync(kFullMask, st);
  if (lane == 0 && st) atomicOr(status, st);
}

__global__ void debug_philox_kernel(const u32* ctr, u32 n, u32 k0, u32 k1, u32* out) {
  const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const U4 r = philox4x32_10(U4{ctr[4 * i], ctr[4 * i + 1], ctr[4 * i + 2], ctr[4 * i + 3]}, k0, k1);
  out[4 * i] = r.x;
  out[4 * i + 1] = r.y;
  out[4 * i + 2] = r.z;
  out[4 * i + 3] = r.w;
}

__global__ void debug_poisson_kernel(ModelDev m, const u32* count, const u64* idx, u32 n, u32 t, u32 stream,
                                     u32 k0, u32 k1, u32* out) {
  const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const U4 r = draw4(idx[i] >> 2, t, stream, 0, k0, k1);
  out[i] = poisson_draw(count[i], (double)m.beta, u4_word(r, (u32)(idx[i] & 3)), idx[i], t, stream, k0, k1,
                        m.tables);
}

}  // namespace

static u32 alias_threads(u32 K);
static size_t alias_scratch_item_bytes(u32 n);

int device_sm_count() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 1;
  }
  return sms;
}

void launch_init_counts(const ModelDev& m, const u32* C, cudaStream_t s) {
  launch_init_counts_raw(m.n, m.K, m.V, C, m.tables, m.beta, m.key0, m.key1, s);
}

void launch_init_counts_raw(u32* n, u32 K, u32 V, const u32* C, const PoisTables& tb, float beta, u32 key0, u32 key1,
                            cudaStream_t s) {
  const u64 groups = ((u64)K * V + 3) / 4;
  const u32 blocks = (u32)std::max<u64>(1, std::min<u64>((groups + 255) / 256, (u64)device_sm_count() * 16));
  init_counts_kernel<<<blocks, 256, 0, s>>>(n, K, V, C, tb, (double)beta, key0, key1);
}

void launch_phi_draw_batch(const ModelDev& ar, const BatchPhiDev& bp, u32 n_blocks, u32 Kmax, const u32* t_dev,
                           cudaStream_t s) {
  if (!n_blocks) return;
  const size_t smem = (size_t)Kmax * 8;
  if (smem > 48 * 1024) cudaFuncSetAttribute(phi_draw_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  phi_draw_batch_kernel<<<n_blocks, 256, smem, s>>>(ar, bp, t_dev);
}

void launch_alias_build_batch(const ModelDev& ar, const BatchPhiDev& bp, u32 Kmax, u32 w0, u32 w1, cudaStream_t s) {
  if (w1 <= w0) return;
  const u32 most = alias_items(Kmax);
  const size_t need = std::max(kAliasWarps * alias_warp_bytes(most), alias_scratch_item_bytes(Kmax));
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, alias_build_batch_kernel, 32 * kAliasWarps, need);
  if (per_sm < 1) per_sm = 1;
  const AliasGrid g = alias_grid(w1 - w0, Kmax, most, (u32)(device_sm_count() * per_sm));
  alias_build_batch_kernel<<<g.blocks, 32 * kAliasWarps, need, s>>>(ar, bp, most, Kmax, w0, w1, g.spread);
}

void launch_bump(u32* t, cudaStream_t s) { bump_kernel<<<1, 1, 0, s>>>(t); }

void launch_phi_draw(const ModelDev& m, u32 t, cudaStream_t s) {
  if (m.K % 4 == 0) {
    // Rows per block: about 64 Ki cells per block, at least 8 rows; fewer where
    // that would leave SMs without a block (two are resident on each), down to
    // what the threads have in flight.
    const u32 tiles = (m.K + 1023) / 1024;
    const u32 side = m.K <= 512 ? 256u / (m.K / 4) : 1u;
    const u32 fill = (u32)((u64)m.V * tiles / (4u * device_sm_count()));
    const u32 rows = std::max<u32>(kPhiRowsInFlight * side,
                                   std::min<u32>(std::max<u32>(8u, 65536u / std::min<u32>(m.K, 1024u)), fill));
    const dim3 grid((m.V + rows - 1) / rows, tiles);
    if (side > 1)
      phi_draw_cols_kernel<true><<<grid, 256, 0, s>>>(m, t, rows);
    else
      phi_draw_cols_kernel<false><<<grid, 256, 0, s>>>(m, t, rows);
    return;
  }
  // (at most 64 Ki cells a block, and blocks for every SM: K=333, V=20011 went
  // from 102 blocks and 320 us to 58 us, with 32-bit topic arithmetic)
  const u32 rows = std::max<u32>(1u, std::min<u32>(65536u / m.K, m.V / (16u * device_sm_count())));
  const u32 blocks = (m.V + rows - 1) / rows;
  const int smem_sums = m.K <= 8192;
  const size_t smem = smem_sums ? (size_t)m.K * 8 : 0;
  if (smem > 48 * 1024) cudaFuncSetAttribute(phi_draw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  phi_draw_kernel<<<blocks, 256, smem, s>>>(m, t, rows, smem_sums);
}

static u32 alias_threads(u32 K) {
  u32 nw = (K + 255) / 256;
  if (nw < 1) nw = 1;
  if (nw > 8) nw = 8;
  return 32 * nw;
}

// Alias-build scratch for n items: vals (u64) then idx (u16), 16-byte rounded.
static size_t alias_scratch_item_bytes(u32 n) { return ((size_t)n * 10 + 15) & ~(size_t)15; }

// Items whose scratch the solo alias kernel keeps in shared memory; words with
// more nonzeros use the block's slice of global scratch.  Small shared memory
// keeps several blocks resident per SM at any K.
constexpr u32 kAliasSmemItems = 2048;
constexpr u32 kAliasBlocksPerSm = 4;

static size_t alias_slice_bytes(u32 K) { return (alias_scratch_item_bytes(K) + 255) & ~(size_t)255; }

size_t alias_build_scratch_bytes(u32 K) {
  if (K <= kAliasSmemItems) return 0;
  return alias_slice_bytes(K) * (size_t)device_sm_count() * kAliasBlocksPerSm;
}

u32 launch_alias_build(const ModelDev& m, cudaStream_t s, void* scratch, size_t scratch_bytes) {
  if (m.Sinv) topic_recip_kernel<<<(m.K + 255) / 256, 256, 0, s>>>(m.S, m.Sinv, m.K);
  const u32 most = alias_items(m.K), recip = m.Sinv ? 1u : 0u;
  const bool own = m.K <= kAliasSmemItems;
  const size_t need = std::max(kAliasWarps * alias_warp_bytes(most), own ? alias_scratch_item_bytes(m.K) : 0);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, alias_build_kernel, 32 * kAliasWarps, need);
  if (per_sm < 1) per_sm = 1;
  const u32 resident = (u32)(device_sm_count() * per_sm);
  if (own) {
    const AliasGrid g = alias_grid(m.V, m.K, most, resident);
    alias_build_kernel<<<g.blocks, 32 * kAliasWarps, need, s>>>(m, most, m.K, g.spread);
    return recip + 1;
  }
  const u32 blocks = std::min<u32>((m.V + kAliasWarps - 1) / kAliasWarps, resident);
  alias_build_kernel<<<blocks, 32 * kAliasWarps, need, s>>>(m, most, 0u, false);
  const u32 items = kAliasSmemItems, nt = alias_threads(m.K);
  const size_t smem = alias_scratch_item_bytes(items), slice = alias_slice_bytes(m.K);
  per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, alias_wide_kernel, nt, smem);
  if (per_sm < 1) per_sm = 1;
  const u32 wide = std::min({m.V, (u32)(device_sm_count() * per_sm), (u32)(scratch_bytes / slice)});
  if (!wide) return recip + 1;  // no scratch: the caller allocates alias_build_scratch_bytes(K)
  alias_wide_kernel<<<wide, nt, smem, s>>>(m, (unsigned char*)scratch, slice, items);
  return recip + 2;
}

void launch_count_rebuild(u32* n, const u32* w, const u32* z, u64 n_tokens, u32 K, u32 V, u32* status,
                          cudaStream_t s) {
  if (!n_tokens) return;
  const u64 groups = (n_tokens + 3) / 4;
  const u32 blocks = (u32)std::max<u64>(1, std::min<u64>((groups + 255) / 256, (u64)device_sm_count() * 8));
  count_rebuild_kernel<<<blocks, 256, 0, s>>>(n, w, z, n_tokens, K, V, status);
}

void launch_doc_offsets(const u32* d_len, u32* d_idx, u32 n_docs, cudaStream_t s) {
  if (!n_docs) return;
  doc_offsets_kernel<<<1, 1024, 0, s>>>(d_len, d_idx, n_docs);
}

cudaError_t launch_doc_plan(const u32* d_len, u32* d_idx, u32* order, u32 n_docs, u32 long_len, const DocPlan& plan,
                            cudaStream_t s) {
  const cudaError_t e = cudaMemsetAsync(plan.bins, 0, kPlanBins * 4, s);
  if (e != cudaSuccess) return e;
  const u32 blocks = (n_docs + kPlanDocs - 1) / kPlanDocs;
  doc_survey_kernel<<<blocks, kPlanThreads, 0, s>>>(d_len, n_docs, plan);
  doc_scan_kernel<<<1, kPlanBins, 0, s>>>(blocks, plan_bin(long_len), plan);
  doc_place_kernel<<<blocks, kPlanThreads, 0, s>>>(d_len, n_docs, d_idx, order, plan);
  return cudaGetLastError();
}

DocPlan doc_plan_at(u32* scratch) {
  static_assert(kPlanWords == 2 * kPlanBins + kPlanBins + 16, "DocPlan's arrays");
  return DocPlan{(u64*)scratch, scratch + 2 * kPlanBins, scratch + 3 * kPlanBins};
}

void launch_debug_philox(const u32* ctr, u32 n, u32 k0, u32 k1, u32* out, cudaStream_t s) {
  if (!n) return;
  debug_philox_kernel<<<(n + 127) / 128, 128, 0, s>>>(ctr, n, k0, k1, out);
}

void launch_debug_poisson(const ModelDev& m, const u32* count, const u64* idx, u32 n, u32 t, u32 stream,
                          u32 k0, u32 k1, u32* out, cudaStream_t s) {
  if (!n) return;
  debug_poisson_kernel<<<(n + 127) / 128, 128, 0, s>>>(m, count, idx, n, t, stream, k0, k1, out);
}

void launch_debug_alias(const u32* q, u32 K, u64* out, cudaStream_t s) {
  const size_t need = (size_t)K * 8 + alias_scratch_item_bytes(K);
  if (need > 48 * 1024) cudaFuncSetAttribute(debug_alias_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need);
  debug_alias_kernel<<<1, alias_threads(K), need, s>>>(q, K, out);
}

}  // namespace gpulda
