// y[M, N] = x[M, K] . W[N, K]^T in float32 on the bfloat16 tensor cores (tcgen05.mma), without giving up float32's precision.
//
// Every operand is the sum of three bfloat16 numbers: x = hi + mid + lo, each the rounding of what is left, 8 bits apiece,
// so that the three hold float32's 24 bits (from 2^-110 on; what lies below is dealt with in second_look).  Of the nine products of two such sums the six largest are formed (hi hi, hi mid,
// mid hi, hi lo, lo hi, mid mid); what the other three would add is below 2^-25 of the product.  The products are exact in
// the tensor core; its sums are not rounded to nearest, so they are kept short: the accumulator in tensor memory covers 64 of
// K, small terms first, and is then added to float32 registers with ordinary rounding.  Against 64 bits the result is closer
// than the chain of K float32 multiply-adds that it replaces (1.1e-7 against 5.7e-7 at K = 1,024, 1.7e-7 against 1.2e-6 at 4,096).
//
// x is split once, by a kernel of its own, into three planes that TMA brings into shared memory; W, which would take 1.5 times its
// own memory, is split on its way in: float32 rows into registers, two chunks ahead, three parts into shared memory.  (With x
// split in here as well a thread had to hold twice as many values and could not ask for them early enough: a chunk of
// 128 x 128 x 64 took 1.95 us, of which the tensor core worked 0.8.)
//
// A block owns a tile of 128 rows of W (the MMA's M side, so that a thread's accumulators are one column of y for 80, 64 or 32
// rows, and a warp stores 32 neighbouring floats) and NT rows of x, and a range of K.  Its warps:
//   0-7    converters of W: 16-byte loads, split, stores as K-major tiles with the 128-byte swizzle;
//   8-15   accumulators: add each chunk's sums to their registers, store at the end;
//   16     issues the MMAs;
//   17     TMA producer: the three parts of the x tile.
// Operands that three parts cannot hold (infinities, NaN, numbers next to either end of float32's range) and results as small or
// as large are noticed, and what they touch is computed again as a plain chain of multiply-adds (second_look).
// What bounds it: no unit (600 x 30,720 outputs, K = 1,024, 240 us, 158 TFLOP/s; in tiles of 128 rows 261 us: tensor pipe 46 % busy,
// loads and stores of shared memory 43 %, issue slots 38 %).  A block takes 32 us for its 16 chunks; about 3 lie before the first chunk's sums and behind the
// last's, where nothing overlaps, and in between conversion, MMAs and addition of a chunk follow one another over two stages.
// 600 rows against the library's float32 product: 4,096 x 1,024 weights 37 against 123 us, 1,024 x 3,072 35 against 127, 151,936 x
// 1,024 1,106 against 3,204 (169 TFLOP/s); 24 rows, 4,096 x 1,024 13 against 27.
// All waits are bounded.
#include "api.h"
#include "common.cuh"
#include "tma.cuh"

namespace pe {
namespace umma32 {

constexpr int BM = 128, BK = 64;      // rows of W a tile; values of K a chunk
constexpr int kParts = 3;
constexpr int kConvWarps = 8, kAccWarps = 8;
constexpr int kThreads = (kConvWarps + kAccWarps + 2) * 32;
constexpr int kLoads = BM / 16;       // 16-byte loads of W a converter thread and chunk

template <int NT>
struct Tile {
  static constexpr int kA = BM * 128, kB = NT * 128;       // bytes of one part
  static constexpr int kStage = kParts * (kA + kB);
  static constexpr int kStages = NT >= 96 ? 2 : 3;
  static constexpr int kCols = NT <= 64 ? 128 : NT <= 128 ? 256 : 512;   // two accumulators of NT columns, in a power of two
  static constexpr int kAcc = NT / 2;                      // accumulators a thread
  static constexpr int kLd = NT > 128 ? 8 : 16;            // sums of a chunk that it reads at a time
};

struct Params {
  const float* x; long long ldx;
  const float* x_top; int segments;   // [M][segments]: a row's largest magnitude; infinity where its parts cut a value off
  const float* w;
  float* y; long long ldy;      // splits > 1: partial sums [splits][M][N]
  int M, N, K;
  int chunks_per_split;
  int* status;
};

__device__ __forceinline__ void tmem_alloc(uint32_t* holder, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tma::smem_addr(holder)), "r"(cols));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(cols));
}
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(tma::smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// 16 consecutive float32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// ... and 8
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
// K-major tile with the 128-byte swizzle (see gemm_umma.cu): rows of 64 bfloat16, groups of 8 rows 1,024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__host__ __device__ constexpr uint32_t instr_desc(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Two neighbouring values: the pair of their bfloat16 roundings, and what that leaves of them.
__device__ __forceinline__ uint32_t take_part(float& a, float& b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  const uint32_t u = *reinterpret_cast<const uint32_t*>(&h);
  a -= __uint_as_float(u << 16);
  b -= __uint_as_float(u & 0xFFFF0000u);
  return u;
}
// Values that three parts do not hold whole: what bfloat16's smallest subnormal, 2^-133, cuts off (see second_look).
constexpr float kCutOff = 7.7037198e-34f;       // 2^-110
__device__ __forceinline__ bool cut_off(float v) { return fabsf(v) < kCutOff && v != 0.f; }
__device__ __forceinline__ bool cut_off(float4 v) { return cut_off(v.x) || cut_off(v.y) || cut_off(v.z) || cut_off(v.w); }
__device__ __forceinline__ float largest(float m, float4 v) {
  return fmaxf(fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
}
// Four rows' four neighbouring values into the three parts' tiles, `bytes` apart, rows 16 apart: part by part over all four,
// so that eight conversions run side by side.
__device__ __forceinline__ void store_parts(float4* v, char* dst, int bytes) {
#pragma unroll
  for (int p = 0; p < kParts; ++p) {
    uint2 u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i].x = take_part(v[i].x, v[i].y), u[i].y = take_part(v[i].z, v[i].w);
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<uint2*>(dst + p * bytes + i * 16 * 128) = u[i];
  }
}

// x [M, K] into planes [3][M][Kp] of bfloat16, Kp = K up to a multiple of 64, the rest zeros; x_top as in Params.  A warp takes
// kSegment values of a row at a time.
constexpr int kSegment = 512;
__global__ void __launch_bounds__(256) gemm_split32_parts_kernel(const float* x, long long ldx, __nv_bfloat16* parts, float* x_top, int M, int K,
                                                                 int Kp) {
  pdl_wait_block();
  pdl_launch_dependents();
  const int segments = (Kp + kSegment - 1) / kSegment, lane = threadIdx.x & 31;
  const size_t total = (size_t)M * segments, plane = (size_t)M * Kp;
  for (size_t i = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5); i < total; i += (size_t)gridDim.x * 8) {
    const size_t m = i / segments;
    const int k0 = (int)(i - m * segments) * kSegment + lane * 4;
    float4 v[kSegment / 128];
#pragma unroll
    for (int j = 0; j < kSegment / 128; ++j) {
      const int k = k0 + j * 128;
      v[j] = k < K ? *reinterpret_cast<const float4*>(x + m * ldx + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    bool cut = false;
    float top = 0.f;
#pragma unroll
    for (int j = 0; j < kSegment / 128; ++j) {
      cut = cut || cut_off(v[j]);
      top = largest(top, v[j]);
      const int k = k0 + j * 128;
      if (k >= Kp) continue;
#pragma unroll
      for (int p = 0; p < kParts; ++p) {
        const uint32_t lo = take_part(v[j].x, v[j].y), hi = take_part(v[j].z, v[j].w);
        *reinterpret_cast<uint2*>(parts + p * plane + m * Kp + k) = make_uint2(lo, hi);
      }
    }
    // magnitudes are ordered as their bits
    const unsigned bits = __reduce_max_sync(0xffffffffu, cut ? 0x7f800000u : __float_as_uint(top));
    if (lane == 0) x_top[i] = __uint_as_float(bits);
  }
}

// ---- outputs whose products the parts do not carry -------------------------------------------------------------------
// Three parts hold a float32 value whole from 2^-110 to the largest that rounds to a finite bfloat16.  Below, the smallest
// subnormal of bfloat16 (2^-133) cuts the value off, by at most 2^-134; above, and for infinities and NaN, the parts give NaN.
// The tensor core's products and sums keep float32's subnormals but do not round to nearest, so results next to them suffer too.
// Such outputs are computed again as a plain chain of float32 multiply-adds.  Which they are:
//   * those that are infinite or NaN;
//   * those of magnitude below kSmall, and zeros whose operands' largest product is that small;
//   * those that a row's cut-off values could move by more than 2^-24 of the output: |y| < K 2^-110 (largest |w| if x was
//     cut off, plus largest |x| if w was).
// The product kernel only asks whether some output could be one: W's values may have been cut off (the converters have no time
// to look), x's not, or the row's largest magnitude says infinity.  Then the tile's operands are read again to decide.
constexpr float kSmall = 1.2037062e-35f;        // 2^-116
constexpr float kLargest = 3.4028235e38f;
constexpr int kExactK = 32;                     // values of K a step
constexpr int kExactWarps = kConvWarps + kAccWarps, kExactThreads = kExactWarps * 32;

__device__ __forceinline__ int exact_any(int v) {        // a barrier of these warps; whether any thread has v
  int any;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.s32 p, %1, 0;\n"
      "barrier.cta.red.or.pred q, 1, %2, p;\n"
      "selp.s32 %0, 1, 0, q;\n"
      "}\n" : "=r"(any) : "r"(v), "n"(kExactThreads) : "memory");
  return any;
}

// Every warp but the last two; a thread has one column and a quarter of the rows.  The tile's results are in y, shared memory is
// free.  A tile in which nothing is computed again reads its operands once more; otherwise the whole tile's chains run side by side.
// 600 x 4,096 outputs, K = 1,024, 37 us: 86 with one zero row of W (the tiles of its 128 rows look), 87 where every tile looks,
// 486 where everything is NaN (one NaN row of W took 4,519 when its outputs were one thread's).
template <int NT>
__device__ __noinline__ void second_look(const Params p) {      // (takes nothing that the product would have to keep for it)
  constexpr int kRows = NT / 4;
  extern __shared__ char smem_raw[];
  const int m0 = blockIdx.x * NT, n0 = blockIdx.y * BM;
  const int k_first = blockIdx.z * p.chunks_per_split * BK, k_last = min(p.K, k_first + p.chunks_per_split * BK);
  float* y = p.y + (gridDim.z > 1 ? (size_t)blockIdx.z * p.M * p.N : 0);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int col = t % BM, row0 = t / BM * kRows, n = n0 + col;
  float* top = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(smem_raw) + 15) & ~static_cast<uintptr_t>(15));
  int* cut = reinterpret_cast<int*>(top + NT + BM);          // [NT + BM] whether a row of x, of W has values that were cut off;
  float* xs = reinterpret_cast<float*>(cut + NT + BM);       // top: its largest magnitude.  [kExactK][NT + 4]
  float* ws = xs + kExactK * (NT + 4);                       // [kExactK][BM + 4]
  auto row_of = [&](int r) -> const float* {                 // the r-th row of x, then of W; null: not there
    if (r < NT) return m0 + r < p.M ? p.x + (size_t)(m0 + r) * p.ldx : nullptr;
    return n0 + r - NT < p.N ? p.w + (size_t)(n0 + r - NT) * p.K : nullptr;
  };
  for (int r = warp * 4; r < NT + BM; r += kExactWarps * 4) {
    const float* row[4];
    float mx[4] = {0.f, 0.f, 0.f, 0.f};
    bool low[4] = {false, false, false, false};
#pragma unroll
    for (int i = 0; i < 4; ++i) row[i] = row_of(r + i);
#pragma unroll 4
    for (int k = k_first + lane * 4; k < k_last; k += 128)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (row[i] != nullptr) {
          const float4 v = *reinterpret_cast<const float4*>(row[i] + k);
          mx[i] = largest(mx[i], v);
          low[i] = low[i] || cut_off(v);
        }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const unsigned bits = __reduce_max_sync(0xffffffffu, __float_as_uint(mx[i]));   // magnitudes are ordered as their bits
      const int any = __any_sync(0xffffffffu, low[i]);
      if (lane == 0) {
        top[r + i] = __uint_as_float(bits);
        cut[r + i] = any;
      }
    }
  }
  exact_any(0);
  uint64_t again = 0;
  const float len = (float)(k_last - k_first), w_top = top[NT + col], w_cut = cut[NT + col] ? 1.f : 0.f;
  if (n < p.N)
    for (int j = 0; j < kRows && m0 + row0 + j < p.M; ++j) {
      const float v = fabsf(y[(size_t)(m0 + row0 + j) * p.ldy + n]), x_top = top[row0 + j];
      const float lost = len * kCutOff * ((cut[row0 + j] ? w_top : 0.f) + w_cut * x_top);
      const bool tiny = v > 0.f ? v < kSmall : x_top > 0.f && w_top > 0.f && x_top * w_top * len < kSmall;
      if (!(v <= kLargest) || tiny || v < lost) again |= 1ull << j;
    }
  if (!exact_any(again != 0)) return;
  const bool mine = __any_sync(0xffffffffu, again != 0);
  float e[kRows];
#pragma unroll
  for (int j = 0; j < kRows; ++j) e[j] = 0.f;
  for (int k0 = k_first; k0 < k_last; k0 += kExactK) {
    exact_any(0);                // the step before has been read
    for (int i = t; i < (NT + BM) * (kExactK / 4); i += kExactThreads) {
      const int r = i / (kExactK / 4), q = i % (kExactK / 4) * 4;
      const float* row = row_of(r);
      const float4 v = row != nullptr && k0 + q < k_last ? *reinterpret_cast<const float4*>(row + k0 + q) : make_float4(0.f, 0.f, 0.f, 0.f);
      float* dst = r < NT ? xs + q * (NT + 4) + r : ws + q * (BM + 4) + r - NT;
      const int step = r < NT ? NT + 4 : BM + 4;
      dst[0] = v.x; dst[step] = v.y; dst[2 * step] = v.z; dst[3 * step] = v.w;
    }
    exact_any(0);
    if (!mine) continue;
#pragma unroll 1
    for (int k = 0; k < kExactK && k0 + k < k_last; ++k) {
      const float w = ws[k * (BM + 4) + col];
#pragma unroll
      for (int j = 0; j < kRows; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(xs + k * (NT + 4) + row0 + j);
        e[j] = fmaf(x.x, w, e[j]);
        e[j + 1] = fmaf(x.y, w, e[j + 1]);
        e[j + 2] = fmaf(x.z, w, e[j + 2]);
        e[j + 3] = fmaf(x.w, w, e[j + 3]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < kRows; ++j)
    if ((again >> j) & 1) y[(size_t)(m0 + row0 + j) * p.ldy + n] = e[j];
}

// grid: (tiles of x rows, tiles of W rows, splits of K).  xmap: the planes as [3 M, Kp], boxes of NT rows.
template <int NT>
__global__ void __launch_bounds__(kThreads, 1) gemm_split32_kernel(Params p, const __grid_constant__ CUtensorMap xmap) {
  using T = Tile<NT>;
  extern __shared__ char smem_raw[];
  __shared__ uint64_t full_bar[T::kStages], empty_bar[T::kStages], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_holder;
  __shared__ uint64_t drain_bar;
  __shared__ volatile int failed;
  char* smem = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * NT, n0 = blockIdx.y * BM;
  const int k_first = blockIdx.z * p.chunks_per_split * BK, k_last = min(p.K, k_first + p.chunks_per_split * BK);
  const int chunks = (k_last - k_first + BK - 1) / BK;      // at least one (the host's plan)
  constexpr int kMmaWarp = kConvWarps + kAccWarps;

  if (threadIdx.x == 0) {
    for (int s = 0; s < T::kStages; ++s) {
      tma::mbar_init(&full_bar[s], kConvWarps + 1);
      tma::mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tma::mbar_init(&acc_full[b], 1);
      tma::mbar_init(&acc_empty[b], kAccWarps);
    }
    tma::mbar_init(&drain_bar, 1);
    failed = 0;
    tma::fence_barrier_init();
  }
  if (warp == kMmaWarp) tmem_alloc(&tmem_holder, T::kCols);

  // A converter thread's place: row 2 warp + lane / 16 (+ 16 a load), values 4 (lane mod 16) .. + 3 of a chunk.  Nothing is
  // loaded with a check: rows beyond W repeat its last one (what they give is never stored), and K beyond the range repeats
  // its last values, against which the planes of x hold zeros.
  const int row_in = warp * 2 + (lane >> 4), quad = lane & 15;
  float4 buf[2][kLoads];
  auto load = [&](int c, float4 (&v)[kLoads]) {
    const float* at = p.w + min(k_first + c * BK + quad * 4, k_last - 4);
#pragma unroll
    for (int i = 0; i < kLoads; ++i) v[i] = *reinterpret_cast<const float4*>(at + (size_t)min(n0 + row_in + 16 * i, p.N - 1) * p.K);
  };
  if (warp < kConvWarps) {   // weights: nothing that an earlier kernel writes
    load(0, buf[0]);
    load(1, buf[1]);
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem_base = tmem_holder;
  pdl_wait_block();
  bool look = false;             // whether this thread's outputs call for a second look

  if (warp < kConvWarps) {
    int stage = 0;
    uint32_t phase = 0;
    // rows 16 apart have the same place in their group of 8, so the swizzle is the same for all of a thread's rows
    const uint32_t at = row_in * 128 + (((quad >> 1) ^ (row_in & 7)) << 4) + (quad & 1) * 8;
    auto convert = [&](int c, float4 (&v)[kLoads]) -> bool {
      if (!tma::mbar_wait(&empty_bar[stage], phase ^ 1)) {
        if (lane == 0) report(p.status, kStatusWaitTimedOut, 50, (int)blockIdx.y, c);
        failed = 1;
        return false;
      }
      char* sa = smem + stage * T::kStage;
#pragma unroll
      for (int i = 0; i < kLoads; i += 4) store_parts(v + i, sa + at + i * 16 * 128, T::kA);
      tma::fence_proxy_async();
      __syncwarp();
      if (lane == 0) tma::mbar_arrive(&full_bar[stage]);
      if (++stage == T::kStages) { stage = 0; phase ^= 1; }
      load(c + 2, v);        // two chunks ahead (past the last one: values that are not used)
      return true;
    };
    for (int c = 0; c < chunks && !failed; c += 2) {
      if (!convert(c, buf[0])) break;
      if (c + 1 < chunks && !convert(c + 1, buf[1])) break;
    }
  } else if (warp < kMmaWarp) {
    const int quarter = warp & 3, half = (warp - kConvWarps) >> 2;
    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + half * T::kAcc;
    float acc[T::kAcc];
#pragma unroll
    for (int j = 0; j < T::kAcc; ++j) acc[j] = 0.f;
    bool ok = true;
    // the largest magnitude of this warp's rows, some of their segments a chunk while the tensor core works
    const float* tops = p.x_top + (size_t)(m0 + half * T::kAcc) * p.segments;
    const int n_tops = min(T::kAcc, p.M - m0 - half * T::kAcc) * p.segments;
    float top = 0.f;
    for (int c = 0; c < chunks; ++c) {
      const int b = c & 1, at = c * 128 + lane;
      float seen[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) seen[i] = at + 32 * i < n_tops ? tops[at + 32 * i] : 0.f;
      if (failed || !tma::mbar_wait(&acc_full[b], (c >> 1) & 1)) {
        if (lane == 0 && !failed) report(p.status, kStatusWaitTimedOut, 51, (int)blockIdx.y, c);
        failed = 1;
        ok = false;
        break;
      }
      fence_after_sync();
#pragma unroll
      for (int h = 0; h < T::kAcc / T::kLd; ++h) {
        uint32_t v[T::kLd];
        if constexpr (T::kLd == 16) tmem_ld16(t_row + b * NT + h * 16, v);
        else tmem_ld8(t_row + b * NT + h * 8, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < T::kLd; ++j) acc[h * T::kLd + j] += __uint_as_float(v[j]);
      }
      fence_before_sync();
      __syncwarp();
      if (lane == 0) tma::mbar_arrive(&acc_empty[b]);
      top = fmaxf(fmaxf(top, fmaxf(seen[0], seen[1])), fmaxf(seen[2], seen[3]));
    }
    pdl_launch_dependents();
    for (int i = chunks * 128 + lane; i < n_tops; i += 32) top = fmaxf(top, tops[i]);     // (a short last range of K)
    // the least magnitude that an output has without a second look
    const float least = fmaxf(kSmall, __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(top))) * kCutOff * (float)p.K);
    const int n = n0 + quarter * 32 + lane;
    if (ok && n < p.N) {
      float* y = p.y + (gridDim.z > 1 ? (size_t)blockIdx.z * p.M * p.N : 0);
#pragma unroll
      for (int j = 0; j < T::kAcc; ++j) {
        const int m = m0 + half * T::kAcc + j;
        if (m >= p.M) break;
        y[(size_t)m * p.ldy + n] = acc[j];
        look = look || !(fabsf(acc[j]) >= least && fabsf(acc[j]) <= kLargest);
      }
    }
  } else if (warp == kMmaWarp) {
    if (lane == 0) {
      const uint32_t idesc = instr_desc(BM, NT);
      int stage = 0;
      uint32_t phase = 0;
      for (int c = 0; c < chunks && !failed; ++c) {
        const int b = c & 1;
        if (!tma::mbar_wait(&acc_empty[b], ((c >> 1) & 1) ^ 1) || !tma::mbar_wait(&full_bar[stage], phase)) {
          report(p.status, kStatusWaitTimedOut, 52, (int)blockIdx.y, c);
          failed = 1;
          break;
        }
        fence_after_sync();
        const uint32_t sa = tma::smem_addr(smem + stage * T::kStage);
        const uint32_t sb = sa + kParts * T::kA;
        const uint32_t d = tmem_base + b * NT;
        // small terms first: 0 hi, 1 mid, 2 lo
        constexpr int kPa[6] = {2, 0, 1, 1, 0, 0}, kPb[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
        for (int t = 0; t < 6; ++t)
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_bf16(d, smem_desc(sa + kPa[t] * T::kA + k * 32), smem_desc(sb + kPb[t] * T::kB + k * 32), idesc, (t > 0 || k > 0) ? 1u : 0u);
        umma_commit(&empty_bar[stage]);
        umma_commit(&acc_full[b]);
        if (++stage == T::kStages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (lane == 0) {
    int stage = 0;
    uint32_t phase = 0;
    for (int c = 0; c < chunks && !failed; ++c) {
      if (!tma::mbar_wait(&empty_bar[stage], phase ^ 1)) {
        report(p.status, kStatusWaitTimedOut, 53, (int)blockIdx.y, c);
        failed = 1;
        break;
      }
      char* sb = smem + stage * T::kStage + kParts * T::kA;
      tma::mbar_expect_tx(&full_bar[stage], kParts * T::kB);
#pragma unroll
      for (int q = 0; q < kParts; ++q) tma::load_2d(sb + q * T::kB, &xmap, k_first + c * BK, q * p.M + m0, &full_bar[stage]);
      if (++stage == T::kStages) { stage = 0; phase ^= 1; }
    }
  }
  fence_before_sync();
  const int again = __syncthreads_or(look);
  if (failed) {
    // Products in flight still use shared and tensor memory: wait for them; copies in flight get as long as a wait lasts at most
    // (nothing completes that phase) to land before the block gives its shared memory back.
    if (warp == kMmaWarp && lane == 0) {
      umma_commit(&drain_bar);
      tma::mbar_wait(&drain_bar, 0);
      tma::mbar_wait(&drain_bar, 1);
    }
    __syncthreads();
  }
  if (warp == kMmaWarp) {
    fence_after_sync();
    tmem_dealloc(tmem_base, T::kCols);
  }
  if (again && !failed && warp < kMmaWarp) second_look<NT>(p);
}

// y[m, n] = the ranges' partial sums, added in their order.
__global__ void __launch_bounds__(256) gemm_split32_add_kernel(const float* part, float* y, long long ldy, int M, int N, int splits) {
  pdl_wait_block();
  pdl_launch_dependents();
  const size_t total = (size_t)M * N, step = (size_t)gridDim.x * blockDim.x * 4;
  for (size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4; i < total; i += step) {   // N is a multiple of 4
    float4 s = *reinterpret_cast<const float4*>(part + i);
    for (int k = 1; k < splits; ++k) {
      const float4 v = *reinterpret_cast<const float4*>(part + (size_t)k * total + i);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    *reinterpret_cast<float4*>(y + i / N * ldy + i % N) = s;
  }
}

struct Plan { int nt, splits, chunks_per_split; };
// Tile and ranges of K by how many blocks come after one another on an SM.  Times in microseconds, measured on a B200: a chunk
// of a tile of 160, 128 or 64 rows, what a block costs beyond its chunks, the addition of partial sums.  Tiles of 160 rows are for
// one wave less: 527 x 4,096 outputs, K = 1,024, are 160 tiles of 128 rows (59 us) or 288 of 64 (63) but 128 of 160 (37); with 400 rows
// of 4,096 outputs, 128 tiles of 128 rows, 31 us against 37.
static Plan plan_for(int M, int N, int K, int n_sms) {
  const int chunks = (K + BK - 1) / BK, n_tiles = (N + BM - 1) / BM;
  Plan best{128, 1, chunks};
  double best_t = 1e30;
  for (int nt : {64, 128, 160}) {
    const long long tiles = (long long)((M + nt - 1) / nt) * n_tiles;
    for (int s = 1; s == 1 || (s <= 8 && s * 4 <= chunks); ++s) {
      if (s > 1 && (nt == 160 || N % 4 || (double)s * M * N * 4 > 64e6)) break;   // (the sums' memory is bounded, too)
      const int cps = (chunks + s - 1) / s, splits = (chunks + cps - 1) / cps;
      const long long waves = (tiles * splits + n_sms - 1) / n_sms;
      double t = waves * (cps * (nt == 160 ? 1.95 : nt == 128 ? 1.5 : 1.3) + 3.0);
      if (splits > 1) t += 3.0 + (double)(splits + 1) * M * N * 4 / 4e6;
      if (t < best_t) { best_t = t; best = Plan{nt, splits, cps}; }
    }
  }
  return best;
}
static long long padded_k(int K) { return (K + BK - 1) / BK * (long long)BK; }
static long long parts_floats(int M, int K) { return (kParts * (long long)M * padded_k(K) + 1) / 2; }   // a multiple of 32 (K's padding)
static int segments_of(int K) { return (int)((padded_k(K) + kSegment - 1) / kSegment); }
static long long top_floats(int M, int K) { return ((long long)M * segments_of(K) + 3) / 4 * 4; }

}  // namespace umma32
}  // namespace pe

extern "C" int pe_gemm_split32_supported(int M, int N, int K) {
  return M >= 1 && M <= (1 << 24) && N >= 1 && K >= 4 && K % 4 == 0 && (N + pe::umma32::BM - 1) / pe::umma32::BM <= 65535 ? 1 : 0;
}

// Floats of scratch that the product of these sizes takes.
extern "C" long long pe_gemm_split32_scratch_floats(int M, int N, int K, int n_sms) {
  if (!pe_gemm_split32_supported(M, N, K)) return 0;
  const pe::umma32::Plan plan = pe::umma32::plan_for(M, N, K, n_sms);
  return pe::umma32::parts_floats(M, K) + pe::umma32::top_floats(M, K) + (plan.splits > 1 ? (long long)plan.splits * M * N : 0);
}

// Kernels that one call launches.
extern "C" int pe_gemm_split32_launches(int M, int N, int K, int n_sms) {
  return pe::umma32::plan_for(M, N, K, n_sms).splits > 1 ? 3 : 2;
}

// x: float32 rows ldx apart, W: dense float32 rows, y: float32 rows ldy apart; all 16-byte aligned.  scratch: at least
// pe_gemm_split32_scratch_floats floats, 16-byte aligned.
extern "C" int pe_gemm_split32(const float* x, long long ldx, const float* w, float* y, long long ldy, int M, int N, int K,
                               float* scratch, int n_sms, int* status, cudaStream_t stream) {
  using namespace pe::umma32;
  if (M <= 0 || N <= 0) return PE_OK;
  if (!pe_gemm_split32_supported(M, N, K)) return PE_ERR_UNSUPPORTED_SIZE;
  if (((uintptr_t)x % 16) || ((uintptr_t)w % 16) || ((uintptr_t)y % 16) || ldx % 4 || ldx < K || ldy < N) return PE_ERR_BAD_ARGUMENT;
  const Plan plan = plan_for(M, N, K, n_sms);
  const bool sums = plan.splits > 1;
  if (scratch == nullptr || ((uintptr_t)scratch % 16) || (sums && ldy % 4)) return PE_ERR_BAD_ARGUMENT;
  const int Kp = (int)padded_k(K);
  __nv_bfloat16* parts = reinterpret_cast<__nv_bfloat16*>(scratch);
  float* x_top = scratch + parts_floats(M, K);
  float* partial = scratch + parts_floats(M, K) + top_floats(M, K);
  CUtensorMap xmap;
  const int e = pe::tma::make_map_2d_bf16(&xmap, parts, Kp, (uint64_t)kParts * M, Kp, BK, plan.nt);
  if (e != 0) return e < 0 ? e : PE_ERR_BAD_ARGUMENT;
  // eight segments a block; no more blocks than fit at a time, each with as many rounds as the others
  const long long units = ((long long)M * segments_of(K) + 7) / 8, rounds = (units + 8ll * n_sms - 1) / (8ll * n_sms);
  pe::launch(gemm_split32_parts_kernel, (int)((units + rounds - 1) / rounds), 256, 0, stream, x, ldx, parts, x_top, M, K, Kp);
  PE_LAUNCH_CHECK();
  Params p;
  p.x = x; p.ldx = ldx; p.x_top = x_top; p.segments = segments_of(K); p.w = w; p.y = sums ? partial : y; p.ldy = sums ? N : ldy; p.M = M; p.N = N; p.K = K;
  p.chunks_per_split = plan.chunks_per_split; p.status = status;
  auto kern = plan.nt == 160 ? gemm_split32_kernel<160> : plan.nt == 128 ? gemm_split32_kernel<128> : gemm_split32_kernel<64>;
  const size_t smem = 1024 + (plan.nt == 160 ? (size_t)Tile<160>::kStages * Tile<160>::kStage : plan.nt == 128 ? (size_t)Tile<128>::kStages * Tile<128>::kStage
                              : (size_t)Tile<64>::kStages * Tile<64>::kStage);
  cudaError_t ce = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (ce != cudaSuccess) return (int)ce;
  dim3 grid((M + plan.nt - 1) / plan.nt, (N + BM - 1) / BM, plan.splits);
  pe::launch(kern, grid, kThreads, smem, stream, p, xmap);
  PE_LAUNCH_CHECK();
  if (sums) {
    const long long q = (long long)M * N / 4;
    const int add_blocks = (int)((q + 255) / 256 < 4ll * n_sms ? (q + 255) / 256 : 4ll * n_sms);
    pe::launch(gemm_split32_add_kernel, add_blocks, 256, 0, stream, (const float*)partial, y, ldy, M, N, plan.splits);
    PE_LAUNCH_CHECK();
  }
  return PE_OK;
}
