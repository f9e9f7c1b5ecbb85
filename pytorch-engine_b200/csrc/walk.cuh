// The walk of a matrix-state recurrence over a step's tokens, with the state's columns spread over the chip.
//
// A head's state S [d, dv] changes column by column: what a token does to column j needs the token's vectors (k, q, the
// decays) and its own v_j, never another column.  So nothing has to be cut along the tokens: a warp takes four columns of a
// head through all tokens of the sequence, eight lanes a column with d / 8 rows each in registers, and a block's four warps
// share the tokens' vectors through shared memory (8 tokens a stage, three stages, cp.async).
//   kDelta:  S <- diag(g) S ;  u = beta (v - S^T k) ;  S <- S + k u^T ;  o = S^T q        (k, q of unit length)
//   kGated:  S <- keep S + take k v^T ;  o = S^T q                                        (keep, take: numbers of the token)
// The vectors are float32 and prepared by another kernel (unit lengths, decays, gates: once a token instead of once a block);
// o goes out as float32, before the head's norm, for a third.  With kGated one more column has v = 1: its state is the
// sum of the keys, its o the denominator's.
//
// What bounds it: for kDelta the chain from one token to the next (a product of 16 rows a lane, three shuffles, one
// update), for kGated the instructions issued and the shared-memory reads (8 16-byte reads a token and lane).  The sums o of
// eight tokens are added over a column's lanes together, seven shuffles for all eight.  Cutting the tokens into chunks instead
// needs, for kDelta, a d x d transition matrix per chunk, twice the work again, and a chain of their products.  Two sequences of
// 1,100 and 400 tokens, eight heads (chunked form before -> prepare, walk and finish now): 128 x 128 delta rule 854 -> 230 us
// (the walk 205), 128 x 256 gated memory 403 -> 269 us (the walk 212).
#pragma once
#include "common.cuh"

namespace pe {

enum WalkKind : int { kWalkDelta = 0, kWalkGated = 1 };

struct WalkArgs {
  const float* kq;        // [n_tokens, key_heads, 2, d]: k, then q
  const float* g;         // kDelta: [n_tokens, heads, d]
  const float* num;       // [n_tokens, heads, 2]: kDelta beta, -; kGated keep, take
  const void* v; long long v_ld;   // row of token t at v + t * v_ld, head h's values at h * dv; 16-byte aligned
  float* o;               // [n_tokens, heads, o_ld]
  int o_ld;               // dv, or (kGated) dv + 4: value dv is the denominator's
  float* S;               // [slots, heads, d, dv]
  float* n;               // kGated: [slots, heads, d]
  const int* seq_slot; const int* seq_qstart;
  int heads, key_heads, dv, n_slots;
  int* status;
};

constexpr int kWalkWarps = 4, kWalkCols = 16;     // columns a block
constexpr int kWalkTokens = 8, kWalkStages = 3;

template <typename T, int D>
struct WalkStage {
  float k[kWalkTokens][D];
  float q[kWalkTokens][D];
  float g[kWalkTokens][D];                        // kDelta
  T v[kWalkTokens][kWalkCols];
  float num[kWalkTokens][2];
};

__device__ __forceinline__ void walk_copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void walk_copy8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// grid: (heads, sequences, column blocks); d = D, dv a multiple of kWalkCols.  kGated: one column block more than dv has.
template <typename T, int D, int KIND>
__global__ void __launch_bounds__(kWalkWarps * 32, 3) walk_kernel(WalkArgs a) {
  constexpr int R = D / 32;                        // 16-byte pieces of a column a lane
  __shared__ __align__(16) WalkStage<T, D> st[kWalkStages];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int head = blockIdx.x, b = blockIdx.y;
  const int c0 = blockIdx.z * kWalkCols;
  const int p = lane & 7;                          // rows 32 r + 4 p + e
  const int j = c0 + warp * 4 + (lane >> 3);
  const bool norm_block = KIND == kWalkGated && c0 >= a.dv;   // its first column is the sum of the keys, the rest is idle
  pdl_wait_block();
  const int slot = a.seq_slot[b];
  if (slot < 0 || slot >= a.n_slots) {
    if (tid == 0 && head == 0 && blockIdx.z == 0) report(a.status, kStatusSlotOutOfRange, b, slot, a.n_slots);
    return;
  }
  const int t0 = a.seq_qstart[b], t1 = a.seq_qstart[b + 1];
  const int kh = head / (a.heads / a.key_heads);
  const bool live = j < a.dv || (norm_block && j == a.dv);
  float* state = norm_block ? a.n + ((size_t)slot * a.heads + head) * D : a.S + ((size_t)slot * a.heads + head) * D * a.dv + j;
  const int s_ld = norm_block ? 1 : a.dv;
  float S[R][4];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int e = 0; e < 4; ++e) S[r][e] = live ? state[(size_t)(32 * r + 4 * p + e) * s_ld] : 0.f;

  auto stage = [&](int batch) {
    const int tb = t0 + batch * kWalkTokens, nb = min(kWalkTokens, t1 - tb);
    if (nb > 0) {
      WalkStage<T, D>& w = st[batch % kWalkStages];
      constexpr int kPieces = D / 4;
      for (int i = tid; i < nb * kPieces; i += kWalkWarps * 32) {
        const int t = i / kPieces, c = i % kPieces * 4;
        const float* src = a.kq + ((size_t)(tb + t) * a.key_heads + kh) * 2 * D + c;
        walk_copy16(&w.k[t][c], src);
        walk_copy16(&w.q[t][c], src + D);
        if (KIND == kWalkDelta) walk_copy16(&w.g[t][c], a.g + ((size_t)(tb + t) * a.heads + head) * D + c);
      }
      constexpr int kV = kWalkCols * (int)sizeof(T) / 16;
      if (!norm_block && tid < nb * kV) {
        const int t = tid / kV, c = tid % kV * (16 / (int)sizeof(T));
        walk_copy16(&w.v[t][c], (const T*)a.v + (size_t)(tb + t) * a.v_ld + head * a.dv + c0 + c);
      }
      if (tid >= 96 && tid < 96 + nb) walk_copy8(w.num[tid - 96], a.num + ((size_t)(tb + tid - 96) * a.heads + head) * 2);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  const int batches = (t1 - t0 + kWalkTokens - 1) / kWalkTokens;
  stage(0);
  stage(1);
  for (int bt = 0; bt < batches; ++bt) {
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();             // this batch is there for everyone, and everyone is through with the one before
    stage(bt + 2);
    const WalkStage<T, D>& w = st[bt % kWalkStages];
    const int tb = t0 + bt * kWalkTokens, nb = min(kWalkTokens, t1 - tb);
    float o[kWalkTokens];
    struct Vectors {
      float4 k[R], q[R], g[R];
      float v, n0, n1;
    };
    auto fetch = [&](int t, Vectors& x) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        x.k[r] = *reinterpret_cast<const float4*>(&w.k[t][32 * r + 4 * p]);
        x.q[r] = *reinterpret_cast<const float4*>(&w.q[t][32 * r + 4 * p]);
        if (KIND == kWalkDelta) x.g[r] = *reinterpret_cast<const float4*>(&w.g[t][32 * r + 4 * p]);
      }
      x.v = norm_block ? 1.f : to_f32<T>(w.v[t][warp * 4 + (lane >> 3)]);
      x.n0 = w.num[t][0];
      x.n1 = KIND == kWalkGated ? w.num[t][1] : 0.f;
    };
    auto token = [&](const Vectors& x) {
      if (KIND == kWalkDelta) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};       // four sums side by side
#pragma unroll
        for (int r = 0; r < R; ++r) {
          S[r][0] *= x.g[r].x; S[r][1] *= x.g[r].y; S[r][2] *= x.g[r].z; S[r][3] *= x.g[r].w;
          acc[0] = fmaf(S[r][0], x.k[r].x, acc[0]);
          acc[1] = fmaf(S[r][1], x.k[r].y, acc[1]);
          acc[2] = fmaf(S[r][2], x.k[r].z, acc[2]);
          acc[3] = fmaf(S[r][3], x.k[r].w, acc[3]);
        }
        float dot = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
        for (int m = 1; m < 8; m <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, m);
        const float u = x.n0 * (x.v - dot);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          S[r][0] = fmaf(x.k[r].x, u, S[r][0]);
          S[r][1] = fmaf(x.k[r].y, u, S[r][1]);
          S[r][2] = fmaf(x.k[r].z, u, S[r][2]);
          S[r][3] = fmaf(x.k[r].w, u, S[r][3]);
        }
      } else {
        const float tv = x.n1 * x.v;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          S[r][0] = fmaf(x.n0, S[r][0], x.k[r].x * tv);
          S[r][1] = fmaf(x.n0, S[r][1], x.k[r].y * tv);
          S[r][2] = fmaf(x.n0, S[r][2], x.k[r].z * tv);
          S[r][3] = fmaf(x.n0, S[r][3], x.k[r].w * tv);
        }
      }
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int r = 0; r < R; ++r) {
        sum[0] = fmaf(S[r][0], x.q[r].x, sum[0]);
        sum[1] = fmaf(S[r][1], x.q[r].y, sum[1]);
        sum[2] = fmaf(S[r][2], x.q[r].z, sum[2]);
        sum[3] = fmaf(S[r][3], x.q[r].w, sum[3]);
      }
      return (sum[0] + sum[1]) + (sum[2] + sum[3]);
    };
    Vectors x[2];
    fetch(0, x[0]);
    if (nb == kWalkTokens) {     // no branches between the tokens, the next one's vectors on their way from shared memory
#pragma unroll
      for (int t = 0; t < kWalkTokens; ++t) {
        if (t + 1 < kWalkTokens) fetch(t + 1, x[(t + 1) & 1]);
        o[t] = token(x[t & 1]);
      }
    } else {
#pragma unroll
      for (int t = 0; t < kWalkTokens; ++t) {
        o[t] = 0.f;
        if (t < nb) {
          if (t > 0) fetch(t, x[0]);
          o[t] = token(x[0]);
        }
      }
    }
    // eight tokens' sums over eight lanes: lane p ends with token p's
    static_assert(kWalkTokens == 8, "eight lanes a column");
    float x4[4], x2[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float send = (p & 4) ? o[i] : o[i + 4], keep = (p & 4) ? o[i + 4] : o[i];
      x4[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float send = (p & 2) ? x4[i] : x4[i + 2], keep = (p & 2) ? x4[i + 2] : x4[i];
      x2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    }
    const float send = (p & 1) ? x2[0] : x2[1], mine = (p & 1) ? x2[1] : x2[0];
    const float total = mine + __shfl_xor_sync(0xffffffffu, send, 1);
    if (p < nb && live) a.o[((size_t)(tb + p) * a.heads + head) * a.o_ld + j] = total;
  }
  pdl_launch_dependents();      // not before: waiting blocks of the next kernel slow this one down
  if (live)
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) state[(size_t)(32 * r + 4 * p + e) * s_ld] = S[r][e];
}

template <typename T, int KIND>
inline void launch_walk(const WalkArgs& a, int d, int n_seqs, cudaStream_t stream) {
  const dim3 grid(a.heads, n_seqs, a.dv / kWalkCols + (KIND == kWalkGated ? 1 : 0));
  auto kern = d == 128 ? walk_kernel<T, 128, KIND> : (d == 64 ? walk_kernel<T, 64, KIND> : walk_kernel<T, 32, KIND>);
  // Not while the kernel before it drains: blocks that start early are packed onto the few SMs that are free by then, and stay
  // there (the delta rule's walk above took 812 us so, 242 started afterwards).
  launch_after(kern, grid, kWalkWarps * 32, 0, stream, a);
}
inline bool walk_takes(int d, int dv) { return (d == 32 || d == 64 || d == 128) && dv > 0 && dv % kWalkCols == 0; }

// ---- one token a sequence --------------------------------------------------------------------------------------------
// A step of single tokens is a pass over the states: a head's S is read once and written once, and the block that owned a whole
// head (a token's staging, three barriers, one column a thread) took 11 us for 64 KB.  Here a head's columns are shared out over
// a cluster of blocks of 16 or 32 columns each, whose 128 threads hold four neighbouring columns of every 32nd row: all of the
// state is on its way at once, and one pass of sums over the rows is enough, since what a token adds to S adds a known multiple of
// k.q to the read.  The head norm's sum goes through the cluster's shared memory.
constexpr int kStepThreads = 128;
inline bool step_takes(int d, int dv) {      // rows: up to four a thread; blocks of a head: one cluster of up to eight
  return d >= 8 && d <= 128 && dv % 16 == 0 && (dv <= 128 || (dv % 32 == 0 && dv <= 256));
}
inline int step_columns(int dv) { return dv <= 128 ? 16 : 32; }

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory"); }
__device__ __forceinline__ float cluster_read(const float* p, int rank) {
  uint32_t at;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(at) : "memory");
  return v;
}

// A thread's part of S: rows rg + 32 r, columns 4 cg .. + 3 of the block's (and 16 further on with CV == 2).
template <int CV> struct StepState {
  float4 s[4][CV];
  __device__ __forceinline__ void load(const float* S, int d, int dv, int col0, int rg, int cg) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int v = 0; v < CV; ++v)
        s[r][v] = rg + 32 * r < d ? *reinterpret_cast<const float4*>(S + (size_t)(rg + 32 * r) * dv + col0 + 16 * v + 4 * cg)
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __device__ __forceinline__ void store(float* S, int d, int dv, int col0, int rg, int cg) const {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int v = 0; v < CV; ++v)
        if (rg + 32 * r < d) *reinterpret_cast<float4*>(S + (size_t)(rg + 32 * r) * dv + col0 + 16 * v + 4 * cg) = s[r][v];
  }
};
// Sums over the rows a warp holds (lanes of one column group: every fourth).
__device__ __forceinline__ float4 step_rows_sum(float4 v) {
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o); v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    v.z += __shfl_xor_sync(0xffffffffu, v.z, o); v.w += __shfl_xor_sync(0xffffffffu, v.w, o);
  }
  return v;
}

// One block a cluster rank: grid (heads * ranks, n_seqs), cluster (ranks, 1, 1).
template <typename K, typename A>
inline cudaError_t launch_step(K kernel, int heads, int ranks, int n_seqs, cudaStream_t stream, const A& args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(heads * ranks, n_seqs); cfg.blockDim = dim3(kStepThreads); cfg.dynamicSmemBytes = 0; cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ranks; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, args);
}

}  // namespace pe
