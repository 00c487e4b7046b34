// Shared host/device helpers: error reporting, dropout RNG, TMA tensor-map encoding.
#pragma once
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <mutex>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "../../include/b200attn.h"
#include "ptx.cuh"

namespace b200attn {

// --------------------------------------------------------------- host errors
void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);

#define B200ATTN_CUDA_OK(expr)                                  \
  do {                                                          \
    cudaError_t _e = (expr);                                    \
    if (_e != cudaSuccess) return ::b200attn::cuda_fail(_e, #expr); \
  } while (0)

// How a kernel is launched beyond its grid: `chained`, it may overlap the previous kernel of the stream and calls
// pdl_wait() (ptx.cuh); `cluster` consecutive blocks form a cluster.
struct LaunchForm {
  bool chained = false;
  unsigned cluster = 1;
};
template <class... Params, class... Args>
inline int launch(const LaunchForm& form, void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem,
                  cudaStream_t stream, const Args&... args) {
  cudaLaunchAttribute attr[2] = {};
  unsigned n = 0;
  if (form.chained) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (form.cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = form.cluster;
    attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = 1;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = n;
  B200ATTN_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
  return B200ATTN_OK;
}
// The forward and decode kernels and the combine step of split keys are short enough for the gap between two launches
// to show, and are launched chained: B1 H4 128 x 128 D64 forward 6.5 -> 5.5 us a call replayed from a graph, paged
// decode of 32 sequences up to 4096 keys 96 -> 92 us. The backward's kernels are not: chained, its dK/dV pass runs
// beside the waiting blocks of the dQ conversion, and a step of B64 H32 512 x 512 D64 took 817 instead of 796 us.
// Not every launch gains (replayed from a graph, plain -> chained): decode of two rows per KV head, B2 Hq16 Hkv8 3001 keys,
// 13.4 -> 17.1 us, B16 H8 500 D64 7.6 -> 8.9; B2 H16 8192 36.9 -> 36.2, B4 Hq16 Hkv8 1000 D64 8.6 -> 8.1; paged H8 11401 D64,
// two sequences, 16.9 -> 15.8; back to back from Python the small ones are bound by the host either way.
constexpr LaunchForm CHAINED{true, 1};

// One-time set-up per device (kernel attributes, device properties) that any host thread may
// trigger: `run(f)` executes `f` once for the current device under std::call_once and hands back its
// return code to every caller; a failed attempt is remembered and reported again, not retried.
struct PerDeviceOnce {
  static constexpr int MAX_DEVICES = 64;
  std::once_flag flags[MAX_DEVICES];
  int rc[MAX_DEVICES] = {};
  template <class F>
  int run(F&& f) {
    int dev = 0;
    B200ATTN_CUDA_OK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= MAX_DEVICES) return f();  // beyond the table: set up on every call
    std::call_once(flags[dev], [&] { rc[dev] = f(); });
    return rc[dev];
  }
};

// Encodes a 4-D tiled tensor map over a [B, H, rows, D] tensor of 16-bit elements
// (dims listed innermost first: D, rows, H, B). `box_cols` x `box_rows` is the tile;
// `swizzle` is a CUtensorMapSwizzle value. Returns 0 or a negative B200ATTN_E* code.
int encode_tmap_4d(CUtensorMap* out, const b200attn_tensor& t, int elem_bytes, int64_t B, int64_t H,
                   int64_t rows, int64_t D, int box_cols, int box_rows, int swizzle,
                   const char* name, int box_heads = 1);

// Multiprocessor count of the current device, looked up once per device.
int sm_count();

// Checks the TMA requirements of one operand; returns 0 or B200ATTN_EINVAL.
int check_tma_operand(const b200attn_tensor& t, int elem_bytes, const char* name);

// delta[b,h,m] = sum_d o*do; optionally also clears a contiguous fp32 [B, H, M, D] array and, with `stats`, writes
// the padded per-query statistics that the backward kernels stream (aux_kernels.cu).
int bwd_delta(const b200attn_tensor* o, int32_t o_dtype, const b200attn_tensor* d_o, int32_t do_dtype,
              float* delta, int32_t B, int32_t H, int32_t M, int32_t D, void* stream, float* zero_rows,
              const float* lse, float2* stats, int Mpad);
// The statistics alone, with zero deltas (total attention).
int launch_stats(const float* lse, float2* stats, int B, int H, int M, int Mpad, cudaStream_t stream);

// Smallest integer threshold T such that a Philox word x (folded to [0, 2^31)) is KEPT iff x > T,
// equivalent to `float(x) * 4.6566127342e-10f > dropout_p` evaluated in fp32.
int32_t dropout_keep_threshold(float dropout_p);

// --------------------------------------------------------------- device RNG
// Philox-4x32 with 6 rounds, keyed by the 64-bit seed, counter = (ctr_lo, ctr_hi, 0, 0);
// returns output word 0. This is the generator behind the reference's `tl.rand(seed, offs,
// n_rounds=6)` (flash.py:474-477); only word 0 of each call is consumed there.
__host__ __device__ __forceinline__ uint32_t philox6_word0(uint32_t seed_lo, uint32_t seed_hi,
                                                           uint32_t ctr_lo, uint32_t ctr_hi) {
  constexpr uint32_t KEY_A = 0x9E3779B9u, KEY_B = 0xBB67AE85u;
  constexpr uint32_t ROUND_A = 0xD2511F53u, ROUND_B = 0xCD9E8D57u;
  uint32_t c0 = ctr_lo, c1 = ctr_hi, c2 = 0u, c3 = 0u;
  uint32_t k0 = seed_lo, k1 = seed_hi;
#pragma unroll
  for (int r = 0; r < 6; ++r) {
    const uint64_t pa = static_cast<uint64_t>(ROUND_A) * c0;
    const uint64_t pb = static_cast<uint64_t>(ROUND_B) * c2;
    const uint32_t n0 = static_cast<uint32_t>(pb >> 32) ^ c1 ^ k0;
    const uint32_t n2 = static_cast<uint32_t>(pa >> 32) ^ c3 ^ k1;
    c1 = static_cast<uint32_t>(pb);
    c3 = static_cast<uint32_t>(pa);
    c0 = n0;
    c2 = n2;
    k0 += KEY_A;
    k1 += KEY_B;
  }
  return c0;
}

// Per-launch dropout constants. Element (b,h,m,n) draws counter
// offset + ((b*H + h)*M + m)*N + n (flash.py:387-391). The reference's kernel does this
// arithmetic in 32 bits when `offset` fits in int32 (the counter's high word is then 0) and in
// 64 bits otherwise; `wide` selects between the two.
struct DropoutCtx {
  uint32_t seed_lo, seed_hi;
  uint64_t offset;
  int32_t keep_threshold;
  uint32_t wide;
  float inv_keep;  // 1 / (1 - p)
  // Optional cache of the keep decisions, written ahead of the forward and read by the forward and the backward
  // instead of evaluating Philox in both: bit keep_bit_of(i) of word keep_mask[((b * Hq + h) * mask_words + w) * M + m] says
  // whether (query m, key 32 * w + i) is kept. Word-major, so that both a thread per query row (forward,
  // dQ kernel) and 32 lanes holding 32 consecutive queries (dK/dV kernel) touch consecutive words.
  uint32_t* keep_mask;
  int mask_words;  // ceil(N / 32)
};

__host__ inline DropoutCtx make_dropout_ctx(float p, uint64_t seed, uint64_t offset) {
  DropoutCtx c;
  c.seed_lo = static_cast<uint32_t>(seed);
  c.seed_hi = static_cast<uint32_t>(seed >> 32);
  c.offset = offset;
  c.keep_threshold = dropout_keep_threshold(p);
  c.wide = offset >= (1ull << 31) ? 1u : 0u;
  c.inv_keep = 1.0f / (1.0f - p);
  c.keep_mask = nullptr;
  c.mask_words = 0;
  return c;
}

// Fills DropoutCtx::keep_mask for every (query, key) whose 128 x 128 tile the band leaves visible.
int launch_keep_mask(const DropoutCtx& ctx, int B, int H, int M, int N, int d_min, int d_max, cudaStream_t stream);

// keep-decision for the element whose exact 64-bit counter is `ctr`.
__device__ __forceinline__ bool dropout_keep(const DropoutCtx& c, uint64_t ctr) {
  const uint32_t lo = static_cast<uint32_t>(ctr);
  const uint32_t hi = c.wide ? static_cast<uint32_t>(ctr >> 32) : 0u;
  const int32_t x = static_cast<int32_t>(philox6_word0(c.seed_lo, c.seed_hi, lo, hi));
  const int32_t folded = x ^ (x >> 31);  // x < 0 ? -x - 1 : x
  return folded > c.keep_threshold;
}

// Order of 32 keep decisions in a word: decision i = 4 r + 2 q + h sits at bit 16 q + 8 h + r, so that after a left
// shift by 7 - r the decisions of the pairs (4 r, 4 r + 1) and (4 r + 2, 4 r + 3) are the sign bits of the four
// bytes, from where one byte permute with sign replication makes the mask of a packed 16-bit pair (keep_mask_pair)
// or of a 32-bit value (keep_mask_one): a test and a select per element cost about twice as much.
__host__ __device__ constexpr int keep_bit_of(int i) { return 16 * ((i >> 1) & 1) + 8 * (i & 1) + (i >> 2); }
__host__ __device__ constexpr int keep_index_of(int bit) { return 4 * (bit & 7) + 2 * (bit >> 4) + ((bit >> 3) & 1); }
__device__ __forceinline__ uint32_t replicate_signs(uint32_t x, uint32_t selector) {
  uint32_t r;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(x), "r"(selector));  // (__byte_perm() drops the sign bit of a selector)
  return r;
}
// 0xffff in each half whose element (i or i + 1, i even) is kept.
__device__ __forceinline__ uint32_t keep_mask_pair(uint32_t word, int i) {
  return replicate_signs(word << (7 - (i >> 2)), (i & 2) ? 0xbbaau : 0x9988u);
}
// All ones if element i is kept.
__device__ __forceinline__ uint32_t keep_mask_one(uint32_t word, int i) {
  return replicate_signs(word << (7 - (i >> 2)), 0x1111u * (8 + (i & 3)));
}

// Keep decisions of 32 consecutive counters base, base+1, ..., base+31 as a word in the order above. The
// counter's high word is the same for all 32 unless the low word wraps inside the run, so everything that depends
// on it is prepared once, the first round's product advances by a constant, and the remaining rounds are written out
// with the product halves that reach output word 0. The fold and the comparison are one range test (kept means
// x + T + 1 > 2 T + 1 as unsigned numbers) whose carry is shifted into the word. keep_mask_kernel takes 1.25 ms for 2^30
// decisions (858 G/s), and 1.38 with the loop over philox6_word0() with fold, compare and insert; forming the high halves on
// the double-precision pipe (2^84 + a * b rounded down to multiples of 2^32) measured 0.6 to 1.02 of the rate and is not used.
__device__ __forceinline__ uint32_t dropout_keep_word(const DropoutCtx& c, uint64_t base) {
  constexpr uint32_t KEY_A = 0x9E3779B9u, KEY_B = 0xBB67AE85u;
  constexpr uint32_t ROUND_A = 0xD2511F53u, ROUND_B = 0xCD9E8D57u;
  const uint32_t lo0 = static_cast<uint32_t>(base);
  uint32_t bits = 0u;
  if (lo0 <= 0xffffffffu - 31u) {
    const uint32_t hi = c.wide ? static_cast<uint32_t>(base >> 32) : 0u;
    const uint64_t first = static_cast<uint64_t>(ROUND_A) * lo0;
    const uint64_t second = static_cast<uint64_t>(ROUND_A) * (hi ^ c.seed_lo);
    const uint32_t ka2 = c.seed_lo + KEY_A, ka3 = c.seed_lo + 2 * KEY_A, ka4 = c.seed_lo + 3 * KEY_A, ka6 = c.seed_lo + 5 * KEY_A;
    const uint32_t kb2 = static_cast<uint32_t>(second >> 32) ^ (c.seed_hi + KEY_B);
    const uint32_t kb3 = static_cast<uint32_t>(second) ^ (c.seed_hi + 2 * KEY_B);
    const uint32_t kb4 = c.seed_hi + 3 * KEY_B, kb5 = c.seed_hi + 4 * KEY_B;
    const uint32_t shift = static_cast<uint32_t>(c.keep_threshold) + 1u;
    const uint32_t above = ~(2u * static_cast<uint32_t>(c.keep_threshold) + 1u);  // x + shift + above carries: kept
#pragma unroll
    for (int bit = 31; bit >= 0; --bit) {
      // words 0 and 2 after round r: xr, yr
      const uint64_t p1 = first + static_cast<uint64_t>(ROUND_A) * static_cast<uint32_t>(keep_index_of(bit));
      const uint32_t y1 = static_cast<uint32_t>(p1 >> 32) ^ c.seed_hi;
      const uint64_t p2 = static_cast<uint64_t>(ROUND_B) * y1;
      const uint32_t x2 = static_cast<uint32_t>(p2 >> 32) ^ ka2, y2 = static_cast<uint32_t>(p1) ^ kb2;
      const uint64_t p3 = static_cast<uint64_t>(ROUND_B) * y2, q3 = static_cast<uint64_t>(ROUND_A) * x2;
      const uint32_t x3 = static_cast<uint32_t>(p3 >> 32) ^ static_cast<uint32_t>(p2) ^ ka3;
      const uint32_t y3 = static_cast<uint32_t>(q3 >> 32) ^ kb3;
      const uint64_t q4 = static_cast<uint64_t>(ROUND_A) * x3;
      const uint32_t x4 = __umulhi(ROUND_B, y3) ^ static_cast<uint32_t>(p3) ^ ka4;
      const uint32_t y4 = static_cast<uint32_t>(q4 >> 32) ^ static_cast<uint32_t>(q3) ^ kb4;
      const uint32_t y5 = __umulhi(ROUND_A, x4) ^ static_cast<uint32_t>(q4) ^ kb5;
      const uint32_t x6 = __umulhi(ROUND_B, y5) ^ (ROUND_B * y4) ^ ka6;
      asm("{\n\t.reg .u32 sum;\n\tadd.cc.u32 sum, %1, %2;\n\taddc.u32 %0, %0, %0;\n\t}" : "+r"(bits) : "r"(x6 + shift), "r"(above));
    }
  } else {
#pragma unroll 1
    for (int i = 0; i < 32; ++i) bits |= (dropout_keep(c, base + i) ? 1u : 0u) << keep_bit_of(i);
  }
  return bits;
}

// Same for 32 counters base + i * stride (elements of one key column across consecutive queries).
__device__ __forceinline__ uint32_t dropout_keep_word_strided(const DropoutCtx& c, uint64_t base,
                                                              uint64_t stride) {
  uint32_t bits = 0u;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const uint64_t ctr = base + stride * static_cast<uint64_t>(i);
    const uint32_t hi = c.wide ? static_cast<uint32_t>(ctr >> 32) : 0u;
    const int32_t x = static_cast<int32_t>(philox6_word0(c.seed_lo, c.seed_hi, static_cast<uint32_t>(ctr), hi));
    bits |= ((x ^ (x >> 31)) > c.keep_threshold ? 1u : 0u) << keep_bit_of(i);
  }
  return bits;
}

// ------------------------------------------------------------ small helpers
__host__ __device__ constexpr int cdiv(int a, int b) { return (a + b - 1) / b; }
__host__ constexpr int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (BF16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}

template <bool BF16>
__device__ __forceinline__ float2 unpack2(uint32_t u) {
  if constexpr (BF16) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
  } else {
    return __half22float2(*reinterpret_cast<__half2*>(&u));
  }
}

// Band limits of the kernels (see FwdArgs::d_min): `causal` and the optional band of the C ABI
// folded together. Returns whether any side is finite.
__host__ inline bool fold_band(bool causal, int band, int dist_min, int dist_max, int* d_min, int* d_max) {
  constexpr int INF = 1 << 30;
  int lo = causal ? 0 : -INF, hi = INF;
  if (band) {
    const int bmin = dist_min < -INF ? -INF : (dist_min > INF ? INF : dist_min);
    const int bmax = dist_max < -INF ? -INF : (dist_max > INF ? INF : dist_max);
    if (bmin > lo) lo = bmin;
    if (bmax < hi) hi = bmax;
  }
  *d_min = lo;
  *d_max = hi;
  return lo > -INF || hi < INF;
}

// 1-D grid order. Blocks are numbered so that (batch, head) pairs are visited in chunks of `chunk`
// pairs; inside a chunk the row-block index z is the slow coordinate. With z sorted from the
// longest block to the shortest this dispatches long (causal) blocks first, while a chunk's K/V
// (or Q/dO) working set stays small enough to live in L2.
struct BlockCoord { int bh, z; };
__device__ __forceinline__ BlockCoord decode_block(int id, int BH, int n_z, int chunk) {
  const int per_chunk = chunk * n_z;
  const int full = BH / chunk;
  int c = id / per_chunk;
  int width = chunk;
  if (c >= full) { c = full; width = BH - full * chunk; }
  const int rem = id - c * per_chunk;
  BlockCoord out;
  out.z = rem / width;
  out.bh = c * chunk + rem - out.z * width;
  return out;
}
// Division of a non-negative 31-bit integer by a divisor fixed on the host: one high multiply and one
// shift (mul = ceil(2^(31 + ceil(log2 d)) / d)) instead of the ~40-instruction integer division.
struct FastDiv {
  uint32_t d, mul, shr;
  __host__ static FastDiv make(int64_t divisor) {
    FastDiv f;
    f.d = divisor < 1 ? 1u : static_cast<uint32_t>(divisor);
    f.mul = 0;
    f.shr = 0;
    if (f.d > 1) {
      uint32_t lg = 0;
      while ((1ull << lg) < f.d) ++lg;
      const uint32_t p = 31 + lg;
      f.mul = static_cast<uint32_t>(((1ull << p) + f.d - 1) / f.d);
      f.shr = p - 32;
    }
    return f;
  }
  __host__ __device__ __forceinline__ int div(int n) const {
#ifdef __CUDA_ARCH__
    return d == 1 ? n : static_cast<int>(__umulhi(static_cast<uint32_t>(n), mul) >> shr);
#else
    return d == 1 ? n : static_cast<int>(static_cast<uint32_t>((static_cast<uint64_t>(static_cast<uint32_t>(n)) * mul) >> 32) >> shr);
#endif
  }
};
// decode_block() with the divisions prepared on the host.
struct BlockOrder {
  FastDiv per_chunk, width, tail_width;
  int chunk, full;  // pairs per chunk, number of full chunks
  __host__ static BlockOrder make(int64_t BH, int n_z, int chunk) {
    BlockOrder o;
    o.chunk = chunk;
    o.full = static_cast<int>(BH / chunk);
    o.per_chunk = FastDiv::make(static_cast<int64_t>(chunk) * n_z);
    o.width = FastDiv::make(chunk);
    o.tail_width = FastDiv::make(BH - static_cast<int64_t>(o.full) * chunk);
    return o;
  }
  __host__ __device__ __forceinline__ BlockCoord decode(int id) const {
    int c = per_chunk.div(id);
    const bool tail = c >= full;
    if (tail) c = full;
    const int rem = id - c * static_cast<int>(per_chunk.d);
    BlockCoord out;
    out.z = tail ? tail_width.div(rem) : width.div(rem);
    out.bh = c * chunk + rem - out.z * static_cast<int>(tail ? tail_width.d : width.d);
    return out;
  }
};
// Number of (batch, head) pairs per chunk: all query heads of as many KV heads as fit `budget`
// bytes of streamed operand per KV head (`bytes_per_kv_head`), at least one KV head, and the chunks about equally large:
// a small last chunk starts its long blocks when nothing else is left to run beside them. (`kv_heads` in all, with
// batch. 32 of them, 22 to a budget: chunks of 22 and 10 -> 16 and 16, training step B4 Hq32 Hkv8 4096 causal D64
// 1740 -> 1530 us; B4 Hq32 Hkv8 2048 D128 665 -> 608.)
__host__ inline int grid_chunk(int groups, int64_t bytes_per_kv_head, bool causal, int64_t kv_heads) {
  if (!causal) return groups;
  const int64_t budget = 96ll << 20;
  int64_t n = budget / (bytes_per_kv_head > 0 ? bytes_per_kv_head : 1);
  if (n < 1) n = 1;
  if (n > 4096) n = 4096;
  n = cdiv(kv_heads, cdiv(kv_heads, n));
  return static_cast<int>(n) * groups;
}

// Status codes written to the optional device status word.
enum : int32_t {
  ST_OK = 0,
  ST_WAIT_TMA = 1,   // a TMA "full" barrier never completed
  ST_WAIT_MMA = 2,   // a tensor-core completion barrier never completed
  ST_WAIT_SOFTMAX = 3,
  ST_WAIT_EMPTY = 4,
};

__device__ __forceinline__ void report_status(int32_t* status, int32_t code) {
  if (status != nullptr) atomicCAS(status, 0, code);
}

// The bounded wait of every kernel role. Returns true once the barrier phase has completed; false
// when it gives up: after `limit_ns`, or as soon as this CTA (`abort_flag`, in shared memory) or any
// CTA of any launch sharing the status word has reported a failure. The caller then records its own
// code (report_status + *abort_flag = 1), leaves its loop and joins the kernel's final barrier, after
// which TMEM is released.
__device__ __forceinline__ bool bounded_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                             const int32_t* status, unsigned long long limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((++spins & 0xffu) == 0u) {
      if (*abort_flag) return false;
      if (status != nullptr && *reinterpret_cast<const volatile int32_t*>(status) != 0) return false;
      if (globaltimer_ns() - t0 > limit_ns) return false;
    }
  }
}

}  // namespace b200attn
