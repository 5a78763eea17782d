// kernels.cuh -- launch interface of the sampler's kernels (kernels.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace gpulda {

// Device status bits set by kernels when an input violates an invariant.
enum StatusBits : u32 {
  kStatusBadTopic = 1,    // a z value >= K (used modulo K)
  kStatusBadWord = 2,     // a w value >= V (used modulo V)
  kStatusDocRange = 4,    // a document runs past n_tokens (skipped)
  kStatusDocTooLong = 8,  // a document longer than the count width allows (skipped)
  kStatusListFull = 32,   // a list sized for its document was too small (cannot happen; the rest is skipped)
};

// Counter slots written by the z sweep.
enum CounterSlots { kCtrTokens = 0, kCtrDocs = 1, kCtrSparseWork = 2, kCtrSparseDraws = 3, kCtrN = 4 };

// Above this many topics a document's counts live in a list or a hash map (a
// dense per-document count array would cost 2 K bytes of shared memory).
constexpr u32 kMapMinK = 2048;

// A word's list (q << 32 | k for q > 0, ascending k) of n entries stored by
// eighths: it is cut into eighths of 2 c consecutive entries, c = list_pairs(n),
// and pair p of eighth e stands at pair p * 8 + e, so that eight lanes that walk
// an eighth each read 128 contiguous bytes at a time (each its own run of an
// ordinary list: 32 L1 wavefronts a load instead of 4).  Zero entries follow to
// the end of the eighth that the list ends in.  Beyond 160 entries c is 4 times
// an odd number: where a list holds most topics, the lanes' counts then lie in
// different banks.

__host__ __device__ inline u32 list_pairs(u32 n) {
  return n <= 160 ? (n ? ((n + 31) >> 5) << 1 : 2u) : (((n + 63) >> 6) | 1u) << 2;
}

// Entries from one word's list to the next.
__host__ __device__ inline u32 list_stride(u32 K) { return 16 * list_pairs(K); }

// Words from one word's bits to the next: whole sectors.
__host__ __device__ inline u32 bits_stride(u32 K) { return (K + 255) / 256 * 8; }

// Whether a large-K model keeps them (unless its sweeps are the hash map's, which
// do not read them): where q takes several times the 126 MB of
// L2, a gather of q mostly goes to HBM.  At 233 MB (K=7275, few documents) the
// bits made the sweep 2.23 -> 2.44 ms and the alias build 0.36 -> 0.46; at 1.2 GB
// 13.7 -> 9.6 and 0.73 -> 0.78.  Between them, 150,000 documents of 80 tokens:
// 5.80 -> 4.50 and 0.20 -> 0.22 at 320 MB, 6.37 -> 4.60 and 0.29 -> 0.30 at 580.
inline bool bits_pay(u32 K, u32 V) { return K > kMapMinK && (u64)K * V * 4 > (512ull << 20); }

// Where entry i of an eighths-stored list with c = list_pairs(n) stands; recip =
// ceil(2^20 / c) divides the at most 8 c <= 1056 pairs' numbers exactly.
__host__ __device__ inline u32 list_recip(u32 c) { return ((1u << 20) + c - 1) / c; }
__host__ __device__ inline u32 list_pos(u32 i, u32 c, u32 recip) {
  const u32 pi = i >> 1, e = (pi * recip) >> 20, p = pi - e * c;
  return 2 * (p * 8 + e) + (i & 1);
}

// A lane's run of a word's list: n pairs of entries from pair `at`, 8 pairs
// apart; `on` when any of them lies in the list.
struct Run {
  u32 at, n;
  bool on;
};

// Lane l of W lanes that walk a list of nw entries: W/8 lanes share an eighth.
template <u32 W>
__device__ __forceinline__ Run lane_run(u32 nw, u32 l) {
  constexpr u32 S = W / 8;
  const u32 c = list_pairs(nw);
  const u32 per = (c + S - 1) / S, e = l / S, p0 = (l % S) * per;
  Run r;
  r.n = S == 1 ? c : min(per, c > p0 ? c - p0 : 0u);
  r.at = p0 * 8 + e;
  r.on = 2 * (e * c + p0) < nw && (S == 1 || r.n);
  return r;
}

// A word's list is short up to this many entries.
constexpr u32 kShortList = 160;

// How many twelfths of a token whose word has a short list make up for one whose
// word has a list of nw entries (mostly_long_lists): 10 + nw^2 / 1e5 tokens.
__host__ __device__ inline u32 long_list_weight(u32 nw) { return nw > kShortList ? 120 + nw * nw / 8333 : 0; }

struct ModelDev {
  u32 K, V;
  float alpha, beta;
  u32 key0, key1;
  u32* n;      // V*K counts, word-major
  u32* q;      // V*K fixed-point Phi (raw x between the two Phi kernels)
  u64* al;     // V*K alias entries
  u64* csr;    // V*K per-word lists of (q << 32 | k) for q > 0, ascending k, nnz[w] used
  u64* lists;  // the same lists by eighths, list_stride(K) entries apart (K <= kMapMinK and memory allowing, else null)
  u32* bits;   // a bit for each of a word's topics with q > 0, bits_stride(K) words a row (training, if bits_pay and
               // memory allowing, else null)
  u64* A;      // V   dense mass per word
  u64* S;      // K   per-topic normalisers
  u64* Sinv;   // K   floor((2^64 - 1) / S[k]), written by the alias build's launch (null: divide)
  u32* nnz;    // V   nonzero x per word
  u64* shares; // 2   sum of x, and that of x * long_list_weight(nnz) (with `lists`, else null)
  PoisTables tables;
};

// Problem tables of a batched launch: many independent models laid out in one
// set of arenas.  Per problem p: K, alpha, Philox key, the index of its first
// token in the concatenated corpus, lgamma(alpha), lgamma(K alpha).  Per
// global document: its problem.  Per global word: where its (word, topic) row
// starts in the arenas.
struct BatchDev {
  const u32* pid;       // per document
  const u64* row_off;   // per word
  const u64* list_off;  // per word: where its list starts
  const u32* K;
  const float* alpha;
  const u32* key0;
  const u32* key1;
  const u64* tok_base;
  const double* lg_a;
  const double* lg_Ka;
};

// Tables of the batched Phi step: per problem K, cell_base (first cell of its
// rows in the arenas), S_off (its per-topic sums), beta, Philox key, and its
// Poisson tables at offset p in the table arenas; per global word its problem
// and row offset; per block of the draw kernel (problem, first row, end row).
struct BatchPhiDev {
  const uint4* blocks;
  const u32* K;
  const u64* cell_base;
  const u64* S_off;
  const float* beta;
  const u32* key0;
  const u32* key1;
  const u32* wpid;
  const u64* row_off;
  const u64* list_off;
  const u32* cdf;
  const uint8_t* guide;
  const double* lfac;
};

struct ZLaunch {
  const u32* w;
  u32* z;
  const u32* d_len;
  const u32* d_idx;
  const u32* order;  // processing order of the documents (longest first); may be null
  u32* K_d;       // may be null
  u32 n_docs;
  u64 n_tokens;
  u64 tok_base;   // global index of this buffer's first token in the iteration
  u32 t;
  const u32* t_dev = nullptr;  // when set, the iteration is read from device memory (graph replays)
  u32 flags;
  unsigned long long* counters;  // kCtrN slots, accumulated
  double* ll;                    // [0] sum, [1] skipped tokens (as double); may be null
  u32* work;                     // zeroed work-queue counter
  u32* status;
  // The shares of words with short and long lists that decide which of two
  // launches sweeps; null: this one does.
  const u64* shares = nullptr;
  const u32* n_long_dev = nullptr;  // documents that take a warp each, where the device counted them
  // Documents that the launch hands on: token reached << 32 | document, and
  // their number.  The list sweep writes them, the sweep of the rest reads
  // them in place of `order`.
  u64* rest = nullptr;
  u32* n_rest = nullptr;
};

// Memory for a table that sweeps are faster with and work without: `count`
// elements, or null where they would take more than half of what is free.  (The
// words' lists are another 9 bytes a cell at K=1000, beside 24.)
template <class T>
T* try_alloc(size_t count) {
  size_t free = 0, total = 0;
  void* p = nullptr;
  if (cudaMemGetInfo(&free, &total) == cudaSuccess && count * sizeof(T) > free / 2) return nullptr;
  if (cudaMalloc(&p, count * sizeof(T)) != cudaSuccess) p = nullptr;
  if (!p) cudaGetLastError();
  return (T*)p;
}

// Grid sizing helpers need the device's SM count.
int device_sm_count();

// Host-side error reporting shared by the entry points (gpulda.cu): records
// `code` as the last error and, in fatal mode, prints and exits.
int report_error(int code, const char* what);
int report_cuda_error(cudaError_t e, const char* where);
// The single model of gpulda.h, if initialized: its device arrays and the
// iteration of its last Phi step (-1 before the first).
bool current_model(ModelDev* out, int* t);

// n[w][k] ~ Poisson(beta + floor(C[w] / K)), iteration 0, stream kStreamInitCounts.
void launch_init_counts(const ModelDev& m, const u32* C, cudaStream_t s);
void launch_init_counts_raw(u32* n, u32 K, u32 V, const u32* C, const PoisTables& tb, float beta, u32 key0, u32 key1,
                            cudaStream_t s);
// Batched Phi step: the draw over n_blocks entries of bp.blocks (the
// iteration read from t_dev; S zeroed first), then the per-word alias build
// over global words [w0, w1).  Kmax bounds the K of the problems involved.
void launch_phi_draw_batch(const ModelDev& ar, const BatchPhiDev& bp, u32 n_blocks, u32 Kmax, const u32* t_dev,
                           cudaStream_t s);
void launch_alias_build_batch(const ModelDev& ar, const BatchPhiDev& bp, u32 Kmax, u32 w0, u32 w1, cudaStream_t s);
void launch_bump(u32* t, cudaStream_t s);
// x ~ Poisson(beta + n) into q (raw), n <- 0, S[k] += x.  S must be zeroed first.
void launch_phi_draw(const ModelDev& m, u32 t, cudaStream_t s);
// Per word: q from x and S, A, nnz and the alias table.
// Returns the number of launches.
u32 launch_alias_build(const ModelDev& m, cudaStream_t s, void* scratch, size_t scratch_bytes);
size_t alias_build_scratch_bytes(u32 K);
// n[w[i]][z[i]] += 1 for every token (warp-aggregated atomics); w and z
// 16-byte aligned.
void launch_count_rebuild(u32* n, const u32* w, const u32* z, u64 n_tokens, u32 K, u32 V, u32* status,
                          cudaStream_t s);
// d_idx = exclusive scan of d_len.
void launch_doc_offsets(const u32* d_len, u32* d_idx, u32 n_docs, cudaStream_t s);
// The same offsets and the documents' order, longest first, for at most
// kPlanMostDocs documents; *plan.n_long receives how many have at least about
// long_len tokens (the first of the order).
constexpr u32 kPlanMostDocs = 1u << 20;
constexpr u32 kPlanWords = 3 * 1024 + 16;
struct DocPlan {
  u64* sums;
  u32* bins;
  u32* n_long;
};
DocPlan doc_plan_at(u32* scratch);  // of kPlanWords words, 8-byte aligned
cudaError_t launch_doc_plan(const u32* d_len, u32* d_idx, u32* order, u32 n_docs, u32 long_len, const DocPlan& plan,
                            cudaStream_t s);
// ZLaunch.flags bits.
constexpr u32 kZFlagLoglik = 1u;  // accumulate the joint log-likelihood

// One sweep over a set of documents, one warp to a document, walking its topics
// or its words' lists, whichever is shorter.
void launch_z_sweep(const ModelDev& m, const ZLaunch& z, cudaStream_t s);
// One sweep over documents of many problems (arenas + tables), with the given
// warps per block and cap on blocks per SM (0: as many as fit).
void launch_z_sweep_batch(const ModelDev& arenas, const BatchDev& b, u32 Kmax, const ZLaunch& z, cudaStream_t s,
                          u32 warps_per_block, u32 blocks_per_sm);
// The same sweep over the words' lists only, K <= kMapMinK (b: documents of many
// problems, or null).  The first n_long documents take a warp each, the others a
// quarter.
void launch_z_sweep_words(const ModelDev& m, const BatchDev* b, u32 Kmax, const ZLaunch& z, u32 n_long, cudaStream_t s,
                          u32 warps_per_block, u32 blocks_per_sm);
// Whether so many tokens' words have long lists that the sweep over the
// documents' topics and the words' lists is the faster.  That one takes 0.27 to
// 0.34 ns a token (3e6 tokens in documents of 100, K=200 to 2000), the other 0.14 to
// 0.21 and, for a token whose word has a list of 200, 500, 1000 or 2000 entries,
// 1.0, 1.5, 2.5 or 6.3 ns more (its warp's other documents wait): they are even
// with one such token in 9, 10, 17 or 50; with documents of 400 in 20 or 70 of the
// last two.  (One in 12 whatever the lengths: 2.15 for 1.03 ms with 8 % of the
// tokens in lists of 2000 entries.)
__device__ __forceinline__ bool mostly_long_lists(const u64* shares) { return shares[1] > 12 * shares[0]; }
// The same sweep with each document's counts in a shared-memory hash map
// (large K).  Documents longer than lmax are reported, not swept.  Returns
// false without launching when lmax needs more shared memory than a block has.
bool launch_z_sweep_map(const ModelDev& m, const ZLaunch& z, cudaStream_t s, u32 lmax);
u32 z_map_slots(u32 K, u32 lmax);
// The same sweep with each document's topics as a list in a warp's registers
// (large K; the default there).  Documents whose list outgrows kListMost
// entries are handed on in z.rest.
constexpr u32 kListMost = 512;
void launch_z_sweep_pairs(const ModelDev& m, const ZLaunch& z, cudaStream_t s);
// The documents of z.rest, none longer than lmax, lists in shared memory.
void launch_z_sweep_rest(const ModelDev& m, const ZLaunch& z, cudaStream_t s, u32 lmax);

// A whole sweep over zl's documents by the kernels that suit them: up to kMapMinK
// topics the sweep over the words' lists or that over the shorter of the two
// sides, by the words' lists; above, the list sweep, then what outgrows its
// lists.  Returns the number of launches.
constexpr u32 kSweepCtrs = 4;  // counters of a sweep's launches, zeroed by the caller
enum SweepCtrSlots { kCtrWork = 0, kCtrRestWork = 1, kCtrRest = 2 };
struct SweepAux {
  u32* ctrs;   // kSweepCtrs
  u64* queue;  // a document each (K > kMapMinK)
  u32 lmax;    // longest document (K > kMapMinK)
  u32 n_long;  // documents to take a warp each (K <= kMapMinK; long_document)
};
u32 launch_sweep(const ModelDev& m, const BatchDev* b, u32 Kmax, ZLaunch zl, const SweepAux& x, cudaStream_t s,
                 u32 warps_per_block, u32 blocks_per_sm);
// Documents of at least this length take a warp each in a sweep of n_tokens.
u32 long_document(u64 n_tokens);

// Debug hooks.
void launch_debug_philox(const u32* ctr, u32 n, u32 k0, u32 k1, u32* out, cudaStream_t s);
void launch_debug_poisson(const ModelDev& m, const u32* count, const u64* idx, u32 n, u32 t,
                          u32 stream, u32 k0, u32 k1, u32* out, cudaStream_t s);
void launch_debug_alias(const u32* q, u32 K, u64* out, cudaStream_t s);

}  // namespace gpulda
