// Token sampling over rows of float32 logits, one block per row, nothing sorted.
//
// Filter chain in the reference's order (pygguf_engine/engine.py:91-134): repetition penalty on the
// unique ids of the recent tokens (92-97, a kernel of its own below), greedy when the temperature is
// at most 1e-5 (99-100, 146-147), else logits / temperature (102), top-k (104-108), softmax (110),
// min-p against the largest probability (112-114), top-p dropping entries whose preceding mass
// exceeds it (116-124).  Each filter keeps the entries above a threshold value, so the kept set is
// found by bitwise search on the order-preserving integer image of the values (counts for top-k,
// probability mass for top-p) instead of a sort.  The draw is the Gumbel-max rule,
// argmax(value_i + G_i) over kept entries, with G_i = -log(-log u_i) and u_i from a counter-based
// generator keyed by (seed, request, step, vocabulary index): the drawn token does not depend on
// the batch a request runs in.  (The reference draws with torch.multinomial, engine.py:149.)
//
// Two kernels when the caller lends scratch memory and the row is greedy or has a small top-k: the
// first cuts every row into chunks, one block each, and leaves each chunk's candidates (a set that
// holds its own top-k; or its largest entry); the second runs the filter chain on the candidates
// of a row, which hold every entry that the row's top-k can keep.
//   top-k up to kTopMax: the first leaves the largest value of every group of 8 to 512 neighbouring entries and nothing else
//     (sample_maxima_kernel); the second bounds the row's k-th value by the k-th of the maxima, which has k entries at or above
//     it, and reads again only the groups whose maximum reaches it.  A row whose groups tie (most entries one and the same
//     number) is searched whole.
//   larger top-k: chunks of kChunk entries in shared memory, threshold search (sample_chunks_kernel).
// A threshold search over a row takes 8 sweeps of 4 bits with per-thread counters (no atomics, fixed
// summation order) instead of 32 sweeps of one bit.
#include "api.h"
#include "common.cuh"

namespace pe {

constexpr int kSampleThreads = 1024;
constexpr int kMaxCompact = 1024;
constexpr int kChunk = 4096;        // entries of a row per block of the first kernel
constexpr int kChunkThreads = 256;
constexpr int kMaxChunks = 64;
constexpr int kMaxCandidates = 3072;  // candidates of a row that the second kernel takes
constexpr int kMaxGroups = 2560;        // groups of a row whose maxima the second kernel holds, in registers
constexpr int kGroupsPer = (kMaxGroups + kSampleThreads - 1) / kSampleThreads;
constexpr int kMaximaThreads = 256;
constexpr int kMaximaTask = 1024;       // entries a warp of the first kernel takes: eight 16-byte loads a lane
constexpr int kMaxGroupList = 1024;     // groups that the second kernel reads again
constexpr int kMaxRanked = 640;         // candidates up to which each is compared with every other
// Largest top-k for the groups.  They are at least 512 (see group_size), and the k-th largest of g maxima has about g ln(g / (g - k))
// entries at or above it: 56 for k = 50 and 295 for k = 224 where g = 512, 229 where g = 2,374 (a row of 151,936 entries).
constexpr int kTopMax = 224;

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ float uniform_of(unsigned long long key, int index) {
  const unsigned long long bits = mix64(key + (unsigned long long)index) >> 40;  // 24 bits
  return ((float)bits + 0.5f) * (1.0f / 16777216.0f);
}
__device__ __forceinline__ unsigned ordered_key(float v) {
  if (v != v) return 0u;  // NaN sorts lowest
  const unsigned u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// The smallest key above that of -infinity: entries below it weigh nothing and are never drawn.
constexpr unsigned kFirstKey = 0x00800000u;

struct ArgBest {
  float v;
  int i;
};
__device__ __forceinline__ ArgBest better(ArgBest a, ArgBest b) {
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}
__device__ ArgBest block_argbest(ArgBest x, ArgBest* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgBest y;
    y.v = __shfl_xor_sync(0xffffffffu, x.v, o);
    y.i = __shfl_xor_sync(0xffffffffu, x.i, o);
    x = better(x, y);
  }
  __syncthreads();
  if (lane == 0) scratch[warp] = x;
  __syncthreads();
  ArgBest r = (lane < nwarps) ? scratch[lane] : ArgBest{-INFINITY, 0x7fffffff};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgBest y;
    y.v = __shfl_xor_sync(0xffffffffu, r.v, o);
    y.i = __shfl_xor_sync(0xffffffffu, r.i, o);
    r = better(r, y);
  }
  return r;
}
__device__ int block_sum_int(int v, int* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  int r = (lane < nwarps) ? scratch[lane] : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;
}

// 16 sums at once over the block in a fixed order; every thread gets all of them.
template <typename T>
__device__ void block_sum16(T (&v)[16], T* scratch /* [33][16] */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
#pragma unroll
  for (int b = 0; b < 16; ++b)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[b] += __shfl_xor_sync(0xffffffffu, v[b], o);
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int b = 0; b < 16; ++b) scratch[warp * 16 + b] = v[b];
  __syncthreads();
  if (threadIdx.x < 16) {
    T r = T(0);
    for (int w = 0; w < nwarps; ++w) r += scratch[w * 16 + threadIdx.x];
    scratch[32 * 16 + threadIdx.x] = r;
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < 16; ++b) v[b] = scratch[32 * 16 + b];
}

// The largest key J such that the weight of the entries with key >= J reaches the target
// (STRICT: exceeds it), four bits of J per sweep.  `entry(i, key, weight)` yields entry i; entries
// of weight zero do not count.  The total weight must reach (exceed) the target.
template <bool STRICT, typename T, typename EntryFn>
__device__ unsigned search16(int n, T target, EntryFn entry, T* scratch) {
  unsigned prefix = 0u;
  T above = T(0);   // weight of the entries whose key is beyond every key with this prefix
  for (int shift = 28; shift >= 0; shift -= 4) {
    const unsigned hi_mask = shift == 28 ? 0u : (0xFFFFFFFFu << (shift + 4));
    T acc[16];
#pragma unroll
    for (int b = 0; b < 16; ++b) acc[b] = T(0);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      unsigned key;
      T w;
      entry(i, key, w);
      if ((key & hi_mask) != prefix) continue;
      const unsigned bin = (key >> shift) & 15u;
#pragma unroll
      for (int b = 0; b < 16; ++b) acc[b] += (bin == (unsigned)b) ? w : T(0);
    }
    block_sum16(acc, scratch);
    int b = 15;
    T run = above;
    for (; b > 0; --b) {
      const T t = run + acc[b];
      if (STRICT ? (t > target) : (t >= target)) break;
      run = t;
    }
    prefix |= (unsigned)b << shift;
    above = run;
  }
  return prefix;
}

struct SampleArgs {
  const float* logits;
  long long ld;
  int n_rows, vocab;
  float temperature;
  int top_k;
  float top_p, min_p;
  unsigned long long seed;
  const int* row_request;
  const int* row_step;
  int* out_tokens;
  int vec;                    // rows start on 16-byte boundaries
  // scratch of the two-kernel path (null: one kernel does everything)
  int n_chunks, cand_cap;     // chunks (groups) per row; room for candidates per chunk
  int group;                  // entries of a group whose maximum the first kernel left in cand_val [rows][groups], 0: chunks
  float* cand_val;            // [rows][chunks][cap] values / temperature, in index order
  int* cand_idx;              // [rows][chunks][cap]
  int* cand_cnt;              // [rows][chunks]; -1: more than cap entries tie for the chunk's top-k
};

__device__ __forceinline__ float scaled(float v, float mult) {
  v *= mult;
  return v == v ? v : -INFINITY;   // NaN sorts lowest
}

// Entries i .. i + 3 of a row's n; those beyond it come as -infinity.
__device__ __forceinline__ float4 load_quad(const float* src, int i, int n, int vec) {
  if (vec && i + 3 < n) return *reinterpret_cast<const float4*>(src + i);
  float4 q;
  q.x = i < n ? src[i] : -INFINITY;
  q.y = i + 1 < n ? src[i + 1] : -INFINITY;
  q.z = i + 2 < n ? src[i + 2] : -INFINITY;
  q.w = i + 3 < n ? src[i + 3] : -INFINITY;
  return q;
}

// Sum over the block's threads; every thread gets it.  scratch: one int a warp.
__device__ __forceinline__ int block_count(int v, int* scratch) {
  v = __reduce_add_sync(0xffffffffu, v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  int r = (threadIdx.x & 31) < (blockDim.x >> 5) ? scratch[threadIdx.x & 31] : 0;
  return __reduce_add_sync(0xffffffffu, r);
}

// A key with at least k of the block's entries at or above it, and exactly those of the k largest
// unless entries tie with the k-th (then its own key): one bit a step, ended early by a count of k.
// Each thread holds N keys; a key of 0 is no entry.
template <int N>
__device__ __forceinline__ unsigned block_kth_key(const unsigned (&key)[N], int k, int* scratch) {
  unsigned K = 0u;
  for (int bit = 31; bit >= 0; --bit) {
    const unsigned cand = K | (1u << bit);
    int mine = 0;
#pragma unroll
    for (int j = 0; j < N; ++j) mine += key[j] >= cand;
    const int count = block_count(mine, scratch);
    if (count >= k) K = cand;
    if (count == k) break;
  }
  return K;
}

// Where a thread's `mine` entries begin in a list over the block's threads; the list's length.
__device__ __forceinline__ int block_offset(int mine, int* scratch, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int add = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += add;
  }
  __syncthreads();
  if (lane == 31) scratch[warp] = incl;
  __syncthreads();
  const int w = lane < nwarps ? scratch[lane] : 0;
  *total = __reduce_add_sync(0xffffffffu, w);
  return __reduce_add_sync(0xffffffffu, lane < warp ? w : 0) + incl - mine;
}

// First kernel for top-k up to kTopMax.  grid: (tasks of eight warps, rows).  The largest value of every group, as it is in the row
// (NaN counts as -infinity); the reads are all it does.  A call for 64 rows of 151,936
// entries, top-k 50: 9.9 us, 12.3 the second kernel, 82 a call with its copies (26.1, 17.5 and 94 with chunks of which the first
// kernel also took the k-th value and the candidates).
__global__ void __launch_bounds__(kMaximaThreads) sample_maxima_kernel(SampleArgs a) {
  pdl_wait_block();
  pdl_launch_dependents();
  const int row = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lo = (blockIdx.x * (kMaximaThreads / 32) + warp) * kMaximaTask;
  if (lo >= a.vocab) return;
  const float* src = a.logits + (size_t)row * a.ld;
  constexpr int kLoads = kMaximaTask / 128;
  float m[kLoads];
#pragma unroll
  for (int j = 0; j < kLoads; ++j) {
    const float4 q = load_quad(src, lo + j * 128 + lane * 4, a.vocab, a.vec);
    m[j] = fmaxf(fmaxf(fmaxf(q.x, q.y), fmaxf(q.z, q.w)), -INFINITY);      // (the maximum of two NaN is NaN)
  }
  // a group is `lanes` lanes of a load, or all of `loads` loads
  const int lanes = min(32, a.group / 4), loads = max(1, a.group / 128);
#pragma unroll
  for (int j = 0; j < kLoads; ++j)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
      if (o < lanes) m[j] = fmaxf(m[j], __shfl_xor_sync(0xffffffffu, m[j], o));
  float* out = a.cand_val + (size_t)row * a.n_chunks;
  if (loads == 1) {
#pragma unroll
    for (int j = 0; j < kLoads; ++j) {
      const int g = (lo + j * 128 + lane * 4) / a.group;
      if (lane % lanes == 0 && g < a.n_chunks) out[g] = m[j];
    }
    return;
  }
#pragma unroll
  for (int o = 1; o < kLoads; o <<= 1)
    if (o < loads)
#pragma unroll
      for (int j = 0; j < kLoads; j += 2 * o) m[j] = fmaxf(m[j], m[j + o]);
#pragma unroll
  for (int j = 0; j < kLoads; ++j) {
    const int g = (lo + j * 128) / a.group;
    if (lane == 0 && j % loads == 0 && g < a.n_chunks) out[g] = m[j];
  }
}

// First kernel of the two-kernel path otherwise.  grid: (chunks, rows).
__global__ void __launch_bounds__(kChunkThreads) sample_chunks_kernel(SampleArgs a) {
  __shared__ float vals[kChunk];
  __shared__ int red_i[33 * 16];
  __shared__ ArgBest red_b[32];
  __shared__ int scan[kChunkThreads];
  pdl_wait_block();
  pdl_launch_dependents();
  const int row = blockIdx.y, chunk = blockIdx.x, tid = threadIdx.x;
  const int lo = chunk * kChunk, n = min(kChunk, a.vocab - lo);
  const float* src = a.logits + (size_t)row * a.ld + lo;
  const size_t slot = (size_t)row * a.n_chunks + chunk;
  float* out_val = a.cand_val + slot * a.cand_cap;
  int* out_idx = a.cand_idx + slot * a.cand_cap;
  const bool greedy = a.temperature <= 1e-5f;
  const float mult = greedy ? 1.0f : 1.0f / a.temperature;
  if (greedy || a.top_k <= 0) {
    // no filter: the row's draw is the best of its chunks' draws (value + Gumbel noise; greedy: value)
    const unsigned long long key =
        mix64(a.seed ^ mix64(((unsigned long long)(unsigned)a.row_request[row] << 32) | (unsigned)a.row_step[row]));
    ArgBest best{-INFINITY, 0x7fffffff};
    // all 16 loads of a thread in flight at once, 16 bytes each where rows allow it
    constexpr int kQuads = kChunk / (4 * kChunkThreads);
    float4 q[kQuads];
#pragma unroll
    for (int j = 0; j < kQuads; ++j) q[j] = load_quad(src, (j * kChunkThreads + tid) * 4, n, a.vec);
#pragma unroll
    for (int j = 0; j < kQuads; ++j) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = (j * kChunkThreads + tid) * 4 + c;
        if (i >= n) continue;
        float v = scaled((&q[j].x)[c], mult);
        if (!greedy && v != -INFINITY) v += -logf(-logf(uniform_of(key, lo + i)));
        best = better(best, ArgBest{v, lo + i});
      }
    }
    best = block_argbest(best, red_b);
    if (tid == 0) {
      out_val[0] = best.v;
      out_idx[0] = best.i;
      a.cand_cnt[slot] = 1;
    }
    return;
  }
  for (int i = tid; i < n; i += blockDim.x) vals[i] = scaled(src[i], mult);
  __syncthreads();
  const int k = min(a.top_k, n);
  const unsigned K = search16<false, int>(n, k, [&](int i, unsigned& key, int& w) { key = ordered_key(vals[i]); w = 1; }, red_i);
  // the entries with key >= K, in index order: each thread owns a contiguous run
  const int per = (n + blockDim.x - 1) / blockDim.x;
  const int i0 = min(n, tid * per), i1 = min(n, i0 + per);
  int mine = 0;
  for (int i = i0; i < i1; ++i) mine += ordered_key(vals[i]) >= K;
  scan[tid] = mine;
  __syncthreads();
  for (int o = 1; o < kChunkThreads; o <<= 1) {
    const int add = (tid >= o) ? scan[tid - o] : 0;
    __syncthreads();
    scan[tid] += add;
    __syncthreads();
  }
  const int total = scan[kChunkThreads - 1];
  if (total > a.cand_cap) {   // ties beyond the room: the second kernel reads the whole row instead
    if (tid == 0) a.cand_cnt[slot] = -1;
    return;
  }
  int pos = scan[tid] - mine;
  for (int i = i0; i < i1; ++i)
    if (ordered_key(vals[i]) >= K) {
      out_val[pos] = vals[i];
      out_idx[pos] = lo + i;
      ++pos;
    }
  if (tid == 0) a.cand_cnt[slot] = total;
}

// The second kernel, or the only one.  GROUPS: the first left groups' maxima.
template <bool GROUPS>
__global__ void __launch_bounds__(kSampleThreads) sample_kernel(SampleArgs a) {
  __shared__ float red_f[33 * 16];
  __shared__ int red_i[33 * 16];
  __shared__ ArgBest red_b[32];
  __shared__ float c_val[kMaxCompact];
  __shared__ int c_idx[kMaxCompact];
  __shared__ int scan[kSampleThreads];      // (GROUPS: the list of groups, later of kept entries)
  static_assert(kMaxGroupList <= kSampleThreads && kMaxRanked <= kSampleThreads, "lists in `scan`");
  __shared__ float l_val[kMaxCandidates];
  __shared__ int l_idx[kMaxCandidates];
  __shared__ int chunk_base[kMaxChunks], chunk_cnt[kMaxChunks];
  pdl_wait_block();
  pdl_launch_dependents();
  const int row = blockIdx.x;
  const int tid = threadIdx.x;
  const float* src = a.logits + (size_t)row * a.ld;
  const int V = a.vocab;
  const bool greedy = a.temperature <= 1e-5f;

  // candidates: the whole row (values scaled on the fly), the chunks' candidates, or, after top-k,
  // a compact list
  const float* vals = src;
  const int* idxs = nullptr;
  float mult = greedy ? 1.0f : 1.0f / a.temperature;
  int n = V;
  if (GROUPS) {
    // a bound of the row's k-th value: the largest key found bit by bit that k of the maxima reach, or a few more
    const float* maxima = a.cand_val + (size_t)row * a.n_chunks;
    unsigned gkey[kGroupsPer];
#pragma unroll
    for (int j = 0; j < kGroupsPer; ++j) {
      const int g = j * kSampleThreads + tid;
      gkey[j] = g < a.n_chunks ? ordered_key(scaled(maxima[g], mult)) : 0u;
    }
    const int k = min(a.top_k, V), slack = k / 8 + 8;
    unsigned bound = 0u;
    for (int bit = 31; bit >= 0; --bit) {
      const unsigned cand = bound | (1u << bit);
      int mine = 0;
#pragma unroll
      for (int j = 0; j < kGroupsPer; ++j) mine += gkey[j] >= cand;
      const int count = block_count(mine, red_i);
      if (count < k) continue;
      bound = cand;
      if (count <= k + slack) break;
    }
    bound = max(bound, kFirstKey);
    int mine = 0, n_list, total;
#pragma unroll
    for (int j = 0; j < kGroupsPer; ++j) mine += gkey[j] >= bound;
    int pos = block_offset(mine, red_i, &n_list);
    if (n_list <= kMaxGroupList) {      // (more only where groups tie)
      int* list = scan;
#pragma unroll
      for (int j = 0; j < kGroupsPer; ++j)
        if (gkey[j] >= bound) list[pos++] = j * kSampleThreads + tid;
      __syncthreads();
      // the groups' entries that reach the bound, a thread's quads one after the other: counted, then written (from the L1)
      const int quads = a.group / 4, n_quads = n_list * quads;
      auto quad_at = [&](int e, int& i) {
        i = list[e / quads] * a.group + e % quads * 4;
        return load_quad(src, i, V, a.vec);
      };
      auto reach = [&](unsigned least) {      // this thread's entries that reach `least`
        int n_reach = 0;
        for (int e = tid; e < n_quads; e += kSampleThreads) {
          int i;
          const float4 q = quad_at(e, i);
#pragma unroll
          for (int c = 0; c < 4; ++c) n_reach += i + c < V && ordered_key(scaled((&q.x)[c], mult)) >= least;
        }
        return n_reach;
      };
      mine = reach(bound);
      pos = block_offset(mine, red_i, &total);
      if (total > kMaxCandidates) {
        // Large entries next to each other (a row masked to one range, logits that fall with the id): the maxima bound the k-th value
        // from too far below, and the bound is raised bit by bit on the groups' entries until few enough reach it.  64 rows of
        // 151,936 falling logits, GPU time of a draw: 57 and 76 us at top-k 50 and 200 (a search over the whole row 818, other rows
        // 53 and 59).
        unsigned raised = 0u;
        for (int bit = 31; bit >= 0; --bit) {
          const unsigned cand = raised | (1u << bit);
          int count = kMaxCandidates;
          if (cand > bound && (count = block_count(reach(cand), red_i)) < k) continue;
          raised = cand;
          if (count <= kMaxRanked) break;
        }
        bound = max(bound, raised);
        mine = reach(bound);
        pos = block_offset(mine, red_i, &total);
      }
      if (total <= kMaxCandidates) {
        for (int e = tid; e < n_quads; e += kSampleThreads) {
          int i;
          const float4 q = quad_at(e, i);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float v = scaled((&q.x)[c], mult);
            if (i + c < V && ordered_key(v) >= bound) {
              l_val[pos] = v;
              l_idx[pos] = i + c;
              ++pos;
            }
          }
        }
        __syncthreads();
        vals = l_val;
        idxs = l_idx;
        mult = 1.0f;
        n = total;
      }
    }
  } else if (a.cand_cnt != nullptr) {
    // gather the chunks' candidates, a warp per chunk; a chunk that overflowed sends us to the row
    const int* cnt = a.cand_cnt + (size_t)row * a.n_chunks;
    static_assert(kMaxChunks <= kSampleThreads, "a thread per chunk");
    const int m = tid < a.n_chunks ? cnt[tid] : 0;
    const bool ok = __syncthreads_and(m >= 0);
    int total;
    const int base = block_offset(max(m, 0), red_i, &total);
    if (tid < kMaxChunks) {
      chunk_base[tid] = base;
      chunk_cnt[tid] = m;
    }
    __syncthreads();
    if (ok && total <= kMaxCandidates) {
      for (int c = tid >> 5; c < a.n_chunks; c += kSampleThreads / 32) {
        const int b = chunk_base[c];
        const size_t slot = ((size_t)row * a.n_chunks + c) * a.cand_cap;
        for (int i = tid & 31; i < chunk_cnt[c]; i += 32) {
          l_val[b + i] = a.cand_val[slot + i];
          l_idx[b + i] = a.cand_idx[slot + i];
        }
      }
      __syncthreads();
      vals = l_val;
      idxs = l_idx;
      mult = 1.0f;
      n = total;
    }
  }

  const bool drawn_in_chunks = idxs != nullptr && a.top_k <= 0;   // the candidates are the chunks' finished draws
  if (greedy || drawn_in_chunks) {
    ArgBest best{-INFINITY, 0x7fffffff};
    for (int i = tid; i < n; i += blockDim.x) best = better(best, ArgBest{scaled(vals[i], mult), idxs ? idxs[i] : i});
    best = block_argbest(best, red_b);
    if (tid == 0) a.out_tokens[row] = best.i == 0x7fffffff ? 0 : best.i;
    return;
  }

  unsigned keep_key = 0u;  // entries with ordered_key(value) >= keep_key are kept

  // largest value
  float mx = -INFINITY;
  for (int i = tid; i < n; i += blockDim.x) mx = fmaxf(mx, scaled(vals[i], mult));
  mx = block_max(mx, red_f);

  bool listed = false;   // the kept entries are the list in c_val
  if (GROUPS && idxs != nullptr && n <= kMaxRanked) {
    // few candidates: the k-th key is the smallest that fewer than k others exceed
    if (tid == 0) red_i[0] = -1;        // as unsigned the largest key there is
    for (int i = tid; i < n; i += kSampleThreads) c_idx[i] = (int)ordered_key(l_val[i]);
    __syncthreads();
    const int k = min(a.top_k, n);
    for (int i = tid; i < n; i += kSampleThreads) {
      const unsigned own = (unsigned)c_idx[i];
      int more = 0;
      for (int j = 0; j < n; ++j) more += (unsigned)c_idx[j] > own;
      if (more < k) atomicMin(reinterpret_cast<unsigned*>(red_i), own);
    }
    __syncthreads();
    keep_key = max((unsigned)red_i[0], kFirstKey);
    int mine = 0, total;
    for (int i = tid; i < n; i += kSampleThreads) mine += (unsigned)c_idx[i] >= keep_key;
    int pos = block_offset(mine, red_i, &total);
    for (int i = tid; i < n; i += kSampleThreads)
      if ((unsigned)c_idx[i] >= keep_key) {
        c_val[pos] = l_val[i];
        scan[pos++] = l_idx[i];
      }
    __syncthreads();
    vals = c_val;
    idxs = scan;
    n = total;
    listed = true;
  } else if (a.top_k > 0 && a.top_k < V && idxs != nullptr && a.top_k <= kTopMax) {
    // more of them: a few a thread, their keys in registers
    constexpr int kPer = kMaxCandidates / kSampleThreads;
    unsigned key[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int i = j * kSampleThreads + tid;
      key[j] = i < n ? ordered_key(l_val[i]) : 0u;
    }
    const unsigned K = max(block_kth_key(key, min(a.top_k, n), red_i), kFirstKey);
    int mine = 0, total;
#pragma unroll
    for (int j = 0; j < kPer; ++j) mine += key[j] >= K;
    int pos = block_offset(mine, red_i, &total);
    keep_key = K;
    if (total <= kMaxCompact) {   // always, but for hundreds of entries that tie with the k-th
#pragma unroll
      for (int j = 0; j < kPer; ++j)
        if (key[j] >= K) {
          c_val[pos] = l_val[j * kSampleThreads + tid];
          c_idx[pos] = l_idx[j * kSampleThreads + tid];
          ++pos;
        }
      __syncthreads();
      vals = c_val;
      idxs = c_idx;
      n = total;
      listed = true;
    }
  } else if (a.top_k > 0 && a.top_k < V) {
    // k-th largest value: the largest key K with count(key >= K) >= k
    // (masked entries stay out: with fewer than k others they would all tie with the k-th and fill the list)
    const unsigned K = max(kFirstKey, search16<false, int>(
        n, min(a.top_k, n), [&](int i, unsigned& key, int& w) { key = ordered_key(scaled(vals[i], mult)); w = 1; }, red_i));
    keep_key = K;
    if (a.top_k <= kMaxCompact) {
      // compact the candidates in index order (deterministic): count, scan, write
      int mine = 0;
      for (int i = tid; i < n; i += blockDim.x) mine += ordered_key(scaled(vals[i], mult)) >= K;
      scan[tid] = mine;
      __syncthreads();
      for (int o = 1; o < kSampleThreads; o <<= 1) {
        const int add = (tid >= o) ? scan[tid - o] : 0;
        __syncthreads();
        scan[tid] += add;
        __syncthreads();
      }
      int pos = scan[tid] - mine;
      const int total = scan[kSampleThreads - 1];
      // a thread's entries are strided, so positions within the list follow (thread, index) order;
      // the list is a set here: nothing below depends on its order
      for (int i = tid; i < n; i += blockDim.x) {
        const float v = scaled(vals[i], mult);
        if (ordered_key(v) >= K) {
          if (pos < kMaxCompact) {
            c_val[pos] = v;
            c_idx[pos] = idxs ? idxs[i] : i;
          }
          ++pos;
        }
      }
      __syncthreads();
      vals = c_val;
      idxs = c_idx;
      mult = 1.0f;
      n = min(total, kMaxCompact);
    }
  }

  // softmax denominator over the kept entries, relative to the largest value
  float z = 0.f;
  for (int i = tid; i < n; i += blockDim.x) {
    const float v = scaled(vals[i], mult);
    if (ordered_key(v) >= keep_key) z += expf(v - mx);
  }
  z = block_sum(z, red_f);

  if (a.min_p > 0.f) {
    // p_i < min_p * p_max  <=>  exp(v_i - max) < min_p   (p_max = 1 / z)
    // as a threshold on the value: v_i >= max + log(min_p)
    const float cut = mx + logf(a.min_p);
    const unsigned kc = ordered_key(cut);
    if (kc > keep_key) keep_key = kc;
  }

  if (a.top_p > 0.f && a.top_p < 1.f) {
    // keep entry i iff the mass of the kept entries with a larger value is <= top_p: the threshold
    // is the largest key J whose mass at or above it exceeds top_p (everything if none does, which
    // cannot be: the whole mass exceeds it)
    const float limit = a.top_p * z;
    const unsigned kk = keep_key;
    unsigned J = 0u;
    if (listed) {
      // few entries: each adds up the mass above itself; J is the smallest key that stays
      for (int i = tid; i < n; i += kSampleThreads) {
        const float v = vals[i];
        l_val[i] = ordered_key(v) >= kk ? expf(v - mx) : 0.f;
        l_idx[i] = (int)ordered_key(v);
      }
      if (tid == 0) red_i[0] = -1;   // as unsigned the largest key there is
      __syncthreads();
      for (int i = tid; i < n; i += kSampleThreads) {
        const unsigned own = (unsigned)l_idx[i];
        float mass = 0.f;
        for (int j = 0; j < n; ++j) mass += (unsigned)l_idx[j] > own ? l_val[j] : 0.f;
        if (!(mass > limit)) atomicMin(reinterpret_cast<unsigned*>(red_i), own);
      }
      __syncthreads();
      J = (unsigned)red_i[0];
    } else J = search16<true, float>(
        n, limit,
        [&](int i, unsigned& key, float& w) {
          const float v = scaled(vals[i], mult);
          key = ordered_key(v);
          w = key >= kk ? expf(v - mx) : 0.f;
        },
        red_f);
    if (J > keep_key) keep_key = J;
  }

  // draw
  const unsigned long long key =
      mix64(a.seed ^ mix64(((unsigned long long)(unsigned)a.row_request[row] << 32) | (unsigned)a.row_step[row]));
  ArgBest best{-INFINITY, 0x7fffffff};
  for (int i = tid; i < n; i += blockDim.x) {
    const float v = scaled(vals[i], mult);
    if (ordered_key(v) < keep_key || v == -INFINITY) continue;
    const int index = idxs ? idxs[i] : i;
    const float u = uniform_of(key, index);
    const float g = -logf(-logf(u));
    best = better(best, ArgBest{v + g, index});
  }
  best = block_argbest(best, red_b);
  if (tid == 0) {
    int tok = best.i;
    if (tok == 0x7fffffff) {  // nothing kept (all NaN): fall back to the first entry
      tok = 0;
    }
    a.out_tokens[row] = tok;
  }
}

// logits[row, id] for the unique ids among recent[row, 0..count): negative -> * penalty, else / penalty.
__global__ void repetition_penalty_kernel(float* logits, long long ld, int vocab, const int* recent, int recent_stride,
                                          const int* recent_count, float penalty) {
  pdl_wait_block();
  pdl_launch_dependents();
  const int row = blockIdx.x;
  const int n = min(recent_count[row], recent_stride);
  const int* r = recent + (size_t)row * recent_stride;
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const int id = r[t];
    if (id < 0 || id >= vocab) continue;
    bool first = true;
    for (int s = 0; s < t; ++s)
      if (r[s] == id) {
        first = false;
        break;
      }
    if (!first) continue;
    float* p = logits + (size_t)row * ld + id;
    const float v = *p;
    *p = v < 0.f ? v * penalty : v / penalty;
  }
}

}  // namespace pe

static bool unfiltered(float temperature, int top_k, float top_p, float min_p) {
  return temperature <= 1e-5f || ((top_k <= 0) && !(top_p > 0.f && top_p < 1.f) && !(min_p > 0.f));
}

// How a row is cut for the first kernel: chunks of how many entries, with room for how many candidates each.
struct SamplePlan {
  int chunk, n_chunks, cap;   // n_chunks 0: one kernel does everything; cap 0: groups of `chunk` entries, their maxima only
};
// Entries of a group: as few as keep a row's maxima in the second kernel's registers (so that a row has more than 512 groups).
static int group_size(int vocab) {
  int size = 8;
  while (size < 512 && (vocab + size - 1) / size > pe::kMaxGroups) size *= 2;
  return size;
}
static SamplePlan sample_plan(int vocab, float temperature, int top_k, float top_p, float min_p) {
  const SamplePlan none{0, 0, 0};
  const int small = (vocab + pe::kChunk - 1) / pe::kChunk;
  if (small < 2) return none;
  if (unfiltered(temperature, top_k, top_p, min_p))
    return small <= pe::kMaxChunks ? SamplePlan{pe::kChunk, small, 1} : none;
  if (top_k <= 0 || top_k >= vocab) return none;
  if (top_k <= pe::kTopMax) {
    const int size = group_size(vocab), groups = (vocab + size - 1) / size;
    if (groups <= pe::kMaxGroups) return SamplePlan{size, groups, 0};
  }
  if (small <= pe::kMaxChunks && (long long)small * top_k <= pe::kMaxCandidates)
    return SamplePlan{pe::kChunk, small, top_k + 8};   // 8: ties with a chunk's k-th value
  return none;
}

// Bytes of scratch with which pe_sample takes its two-kernel path for these settings (0: it has none).
extern "C" long long pe_sample_scratch_bytes(int n_rows, int vocab, float temperature, int top_k, float top_p, float min_p) {
  if (n_rows <= 0 || vocab <= 0) return 0;
  const SamplePlan plan = sample_plan(vocab, temperature, top_k, top_p, min_p);
  return (long long)n_rows * plan.n_chunks * (plan.cap * 8ll + 4ll);   // (a group's maximum: four bytes)
}

// scratch: null, or at least pe_sample_scratch_bytes(...) bytes, 4-byte aligned.
extern "C" int pe_sample(const float* logits, long long ld, int n_rows, int vocab, float temperature, int top_k,
                         float top_p, float min_p, unsigned long long seed, const int* row_request, const int* row_step,
                         int* out_tokens, void* scratch, long long scratch_bytes, cudaStream_t stream) {
  if (n_rows <= 0) return PE_OK;
  if (vocab <= 0 || ld < vocab) return PE_ERR_BAD_ARGUMENT;
  pe::SampleArgs a;
  a.logits = logits; a.ld = ld; a.n_rows = n_rows; a.vocab = vocab; a.temperature = temperature; a.top_k = top_k;
  a.top_p = top_p; a.min_p = min_p; a.seed = seed; a.row_request = row_request; a.row_step = row_step;
  a.out_tokens = out_tokens;
  a.vec = ((uintptr_t)logits % 16) == 0 && ld % 4 == 0;
  a.n_chunks = 0; a.cand_cap = 0; a.group = 0; a.cand_val = nullptr; a.cand_idx = nullptr; a.cand_cnt = nullptr;
  const long long need = pe_sample_scratch_bytes(n_rows, vocab, temperature, top_k, top_p, min_p);
  if (scratch != nullptr && need > 0 && scratch_bytes >= need && ((uintptr_t)scratch % 4) == 0) {
    const SamplePlan plan = sample_plan(vocab, temperature, top_k, top_p, min_p);
    a.n_chunks = plan.n_chunks;
    a.cand_cap = plan.cap;
    const size_t slots = (size_t)n_rows * a.n_chunks;
    a.cand_val = reinterpret_cast<float*>(scratch);
    a.cand_idx = reinterpret_cast<int*>(a.cand_val + slots * a.cand_cap);
    a.cand_cnt = a.cand_idx + slots * a.cand_cap;
    if (plan.cap == 0) {
      a.group = plan.chunk;
      const int tasks = (vocab + pe::kMaximaTask - 1) / pe::kMaximaTask, warps = pe::kMaximaThreads / 32;
      pe::launch(pe::sample_maxima_kernel, dim3((tasks + warps - 1) / warps, n_rows), pe::kMaximaThreads, 0, stream, a);
      PE_LAUNCH_CHECK();
      pe::launch(pe::sample_kernel<true>, n_rows, pe::kSampleThreads, 0, stream, a);
      PE_LAUNCH_CHECK();
      return PE_OK;
    }
    pe::launch(pe::sample_chunks_kernel, dim3(a.n_chunks, n_rows), pe::kChunkThreads, 0, stream, a);
    PE_LAUNCH_CHECK();
  }
  pe::launch(pe::sample_kernel<false>, n_rows, pe::kSampleThreads, 0, stream, a);
  PE_LAUNCH_CHECK();
  return PE_OK;
}

extern "C" int pe_repetition_penalty(float* logits, long long ld, int n_rows, int vocab, const int* recent,
                                     int recent_stride, const int* recent_count, float penalty, cudaStream_t stream) {
  if (n_rows <= 0 || penalty == 1.0f) return PE_OK;
  if (penalty <= 0.f) return PE_ERR_BAD_ARGUMENT;
  pe::launch(pe::repetition_penalty_kernel, n_rows, 256, 0, stream, logits, ld, vocab, recent, recent_stride, recent_count, penalty);
  PE_LAUNCH_CHECK();
  return PE_OK;
}
