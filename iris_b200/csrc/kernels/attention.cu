// attention.cu — causal (or full) self-attention forward for head dimension 128 on the 5th-generation tensor cores.
//
//   O[b, s, h, :] = softmax(Q[b, s, h, :] . K[b, 0..s, h, :]^T / sqrt(128)) . V[b, 0..s, h, :]
//
// Q, K and V are the three column blocks of ONE matrix qkv[T = B * S, 3 * heads * 128] (the output of the fused
// all-gather -> GEMM of the tensor-parallel decoder block), O is [T, heads * 128]; 16-bit elements (bf16 or fp16),
// fp32 accumulation and softmax.  No counterpart in the reference (it has no model code); it replaces the library
// attention call inside iris_b200/models/tp_block.py.
//
// A CTA works on two 128-row sides, A and B, at once, so that the tensor cores compute the scores of one side while the
// other side is in its exponentials (the two take about the same time: 1024 cycles of MMAs and 1024 of ex2 per tile of
// 128 x 128).  Two ways to fill the sides:
//   pair    A and B are neighbouring tiles of 128 queries of one head and share every K / V tile: half the loads
//   split   A and B are the same queries, A takes the even key tiles and B the odd ones, and the two partial outputs are
//           merged at the end: half the serial chain, for problems whose query tiles do not fill the GPU
// Persistent: a CTA takes its items from a fixed list, longest first and dealt out back and forth so that the sums come
// out even, heads in groups whose K and V stay in L2.  Roles (320 threads):
//   warps 0-3, 4-7  softmax of side A, B, one thread per query row: tcgen05.ld of the row of scores, maximum, exp2, row
//                   sum, and P as 16-bit values back into tensor memory over the scores, where the MMA reads it as its A
//                   operand.  O stays in tensor memory for all key tiles and is rescaled there whenever the running maximum
//                   of one of the warp's rows has grown, which in most tiles it has.
//   warp 8          TMA producer: Q tiles, and K / V tiles through a ring of five slots (no multicast)
//   warp 9          one elected thread issues tcgen05.mma:  S = Q K^T, then O += P V (P from tensor memory, V as an
//                   MN-major operand: V[key][d] is read as stored), alternating between the sides; the first half of a
//                   product starts when the first half of P is there
// What bounds it: the chain of one side, scores -> softmax -> product: 4300 - 5000 cycles per step of a pair for 2048 of MMAs
// and 2048 of ex2; in a long run the GPU's power limit takes the clock besides.  8 x 2048 tokens x 32 heads bf16, causal /
// without a mask: from a rest, 1965 MHz, 317 / 524 us; a run of seconds, 1635 / 1612 MHz at 1010 W, 349 / 585 us.  A scale that is renewed only after a growth of 2^8 takes 287 / 467 us
// instead, but then a row's largest weight is rounded like the others and the error against 64 bits grows by 2 to 4 %
// (2.034e-3 -> 2.071e-3, 2.256e-3 -> 2.337e-3, both bf16).
// Before: one 128-row tile per CTA, two threads per row reading the scores twice, P through shared memory, O folded
// through registers after every tile: 659 us causal, 1091 without a mask.
//
// Every wait is bounded by timeout_ns: on expiry the CTA records a status, every role leaves its loop, tensor memory
// is released and the kernel returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <mutex>

#include "iris/iris.cuh"
#include "iris/ptx_sm100.cuh"

namespace iris {
namespace attn {

using namespace iris::ptx;

constexpr int D = 128;            // head dimension
constexpr int BQ = 128;           // queries per side
constexpr int BKV = 128;          // keys per tile
constexpr int kTileBytes = 128 * 128 * 2;   // one 128 x 128 tile of 16-bit elements (two 64-column swizzle blocks)
constexpr int kHalfBytes = kTileBytes / 2;  // one 64-column block: 128 rows x 128 bytes
constexpr int kThreads = 320;
constexpr int kSlots = 5;              // K / V ring
constexpr int kBarBytes = 1024;        // barriers and small shared words
// shared memory: barriers | Q of side A | Q of side B (split: row maxima and sums) | ring
constexpr int kSmemBytes = 1024 + kBarBytes + (2 + kSlots) * kTileBytes;
static_assert(kSmemBytes <= 227 * 1024, "shared-memory budget");

// The split form, in which the softmax of a tile is part of the chain that sets the time, makes one in so many pairs of
// exponentials on the FMA units instead of the special-function unit (1 x 4096 x 4 heads causal: 40.1 -> 38.1 us, 3 x 384 x 5
// 8.25 -> 8.12, 4 x 3072 x 7 without a mask 172 -> 166 from a rest; 2 x 1024 x 12 loses, 15.1 -> 15.4).  The pair form gains
// nothing from it.
constexpr int kPolyEvery = 4;

enum Site : uint32_t { kSiteLoad = 90, kSiteMma = 91, kSiteSoftmax = 92 };

// 2^x on the special-function unit (ex2.approx: 2 ulp, 2^-inf = 0), which is what bounds the softmax warps.
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Two fp32 operations in one instruction.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 x, x, y;\n\t"
      "mov.b64 {%0, %1}, x;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 x, x, y;\n\t"
      "mov.b64 {%0, %1}, x;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
// 2^t on the FMA units, for a share of the exponentials (see kPolyEvery).  t = k + f with k the nearest integer, 2^f from a
// polynomial of degree 5 with value 1 at 0, fitted here for the smallest largest relative error on [-1/2, 1/2]: 9.1e-08 in
// exact arithmetic, 1.7e-7 evaluated in fp32 (ex2.approx: 2.4e-7).  t below -126.5 gives 0, as ex2.approx.ftz does below -126,
// so that a masked key weighs nothing however large its value is: k is at least -127, whose scale has the bits of 0.  A NaN
// stays one.
__device__ __forceinline__ float2 poly_exp2(float2 t) {
  asm("max.NaN.f32 %0, %0, 0fC2FE0000;" : "+f"(t.x));   // -127
  asm("max.NaN.f32 %0, %0, 0fC2FE0000;" : "+f"(t.y));
  const float kMagic = 12582912.f;   // 1.5 * 2^23: the sum's last bits are the integer part
  const float2 r = add2(t, make_float2(kMagic, kMagic));
  const float2 k = add2(r, make_float2(-kMagic, -kMagic));
  const float2 f = fma2(k, make_float2(-1.f, -1.f), t);
  auto both = [](float c) { return make_float2(c, c); };
  float2 q = fma2(both(1.326472731e-03f), f, both(9.671512991e-03f));
  q = fma2(q, f, both(5.550733581e-02f));
  q = fma2(q, f, both(2.402224243e-01f));
  q = fma2(q, f, both(6.931470037e-01f));
  q = fma2(q, f, both(1.f));
  return mul2(q, make_float2(__uint_as_float((__float_as_uint(r.x) << 23) + 0x3f800000u),
                             __uint_as_float((__float_as_uint(r.y) << 23) + 0x3f800000u)));
}
template <bool F16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if (F16) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&b);
}

// Scores of the keys after `row` become minus infinity.
template <int N>
__device__ __forceinline__ void mask_after(uint32_t* v, int row) {
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (i > row) v[i] = 0xff800000u;
}

struct Params {
  CUtensorMap tm;        // qkv [T, 3 * heads * 128], box 64 columns x 128 rows, 128-byte swizzle
  void* out;             // [T, heads * 128]
  int64_t ldo;           // row pitch of out, elements
  StatusBlock* status;
  uint64_t timeout_ns;
  int batch, seq, heads;
  int causal;
  int blocks;            // items per head: query tiles (split) or pairs of them
  int group;             // heads whose items are dealt out together
  int items;
  float scale_log2;      // log2(e) / sqrt(128)
};

// One item of the list: head `bh`, query tiles qa and qa + 1 (pair) or qa (split), n key tiles loaded, of which side A
// uses na and side B nb (0: side B has nothing to do).
struct Item {
  int bh, qa, n, na, nb;
};

// Item of round r of CTA c, false past the end of the list.
template <bool SPLIT>
__device__ __forceinline__ bool item_of(const Params& p, int r, Item& it) {
  const int g = gridDim.x;
  const int idx = r * g + ((r & 1) ? g - 1 - (int)blockIdx.x : (int)blockIdx.x);
  if (idx >= p.items) return false;
  const int per = p.group * p.blocks;
  const int first = idx / per * p.group;
  const int left = p.batch * p.heads - first;
  const int hc = left < p.group ? left : p.group;
  const int rank = idx % per;
  it.bh = first + rank % hc;
  const int q = p.blocks - 1 - rank / hc;      // longest rows of work first
  const int nq = p.seq / BQ;
  if (SPLIT) {
    it.qa = q;
    it.n = p.causal ? q + 1 : nq;
    it.na = (it.n + 1) / 2;
    it.nb = it.n / 2;
  } else {
    it.qa = 2 * q;
    const bool b = it.qa + 1 < nq;
    it.na = p.causal ? it.qa + 1 : nq;
    it.nb = !b ? 0 : p.causal ? it.qa + 2 : nq;
    it.n = it.nb > it.na ? it.nb : it.na;
  }
  return true;
}

template <bool F16, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1) attention_fwd_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t bar0 = smem_u32(smem);
  const uint32_t q_s = bar0 + kBarBytes;           // side A, side B
  const uint32_t ring = q_s + 2 * kTileBytes;
  // barriers; [x] = side
  auto q_full = [&](int x) { return bar0 + 8u * (0 + x); };
  auto q_empty = [&](int x) { return bar0 + 8u * (2 + x); };
  auto s_full = [&](int x) { return bar0 + 8u * (4 + x); };    // scores complete (and everything issued before them)
  auto p_half = [&](int x) { return bar0 + 8u * (6 + x); };    // P of the first 64 keys in tensor memory, O rescaled
  auto o_full = [&](int x) { return bar0 + 8u * (8 + x); };    // last product of the item complete
  auto o_free = [&](int x) { return bar0 + 8u * (10 + x); };   // O has been read
  auto p_ready = [&](int x) { return bar0 + 8u * (14 + x); };  // all of P in tensor memory, scores read
  const uint32_t merge_bar = bar0 + 8u * 12;                   // split: both sides' maxima and sums are in shared memory
  const uint32_t drain_bar = bar0 + 8u * 13;
  auto kv_full = [&](int s) { return bar0 + 8u * (16 + s); };
  auto kv_empty = [&](int s) { return bar0 + 8u * (16 + kSlots + s); };
  volatile uint32_t* words = reinterpret_cast<volatile uint32_t*>(smem + 8 * (16 + 2 * kSlots));
  volatile uint32_t* tmem_slot = words;
  volatile uint32_t* abort_flag = words + 1;
  volatile uint32_t* never = words + 2;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // warp: uniform

  if (warp == 8 && elect_one()) {
    prefetch_tensormap(&p.tm);
    for (int x = 0; x < 2; ++x) {
      mbar_init(q_full(x), 1);
      mbar_init(q_empty(x), 1);
      mbar_init(s_full(x), 1);
      mbar_init(p_half(x), 4);                   // one arrival per softmax warp of the side
      mbar_init(p_ready(x), 4);
      mbar_init(o_full(x), 1);
      mbar_init(o_free(x), SPLIT ? 8 : 4);     // split: both sides read both outputs
    }
    mbar_init(merge_bar, 8);
    mbar_init(drain_bar, 1);
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(kv_full(s), 1);
      mbar_init(kv_empty(s), 1);
    }
    *abort_flag = 0;
    *never = 0;
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);   // S (and P) of A and B, O of A and B: 128 columns each
    tmem_relinquish();
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  grid_dependency_wait();
  grid_dependency_launch();

  // Ring order of an item's tiles: K_0 .. K_{lead-1}, then V_i, K_{i+lead}, V_{i+1}, ...: the order in which the MMA
  // thread needs them (pair: lead 1; split: lead 2, because each side starts with a key tile of its own).
  const int lead = SPLIT ? 2 : 1;

  if (warp == 8) {
    if (elect_one()) {
      bool ok = true;
      uint32_t pos = 0;                 // ring position
      uint32_t qn[2] = {0, 0};          // Q tiles loaded per side
      auto stop = [&](int what) {
        record_status(p.status, kTimeout, kSiteLoad, blockIdx.x, pos, what);
        *abort_flag = 1;
        ok = false;
      };
      auto load_tile = [&](uint32_t dst, int x, int y, uint32_t bar) {
        mbar_expect_tx(bar, kTileBytes);
        tma_load_2d(dst, &p.tm, x, y, bar);
        tma_load_2d(dst + kHalfBytes, &p.tm, x + 64, y, bar);
      };
      auto load_kv = [&](int x, int y) {
        if (!ok) return;
        const int s = pos % kSlots;
        const uint32_t use = pos / kSlots;
        if (use > 0 && !mbar_wait(kv_empty(s), (use - 1) & 1, p.timeout_ns, abort_flag)) return stop(0);
        load_tile(ring + s * kTileBytes, x, y, kv_full(s));
        ++pos;
      };
      auto load_q = [&](int side, int x, int y) {
        if (!ok) return;
        const uint32_t use = qn[side]++;
        if (use > 0 && !mbar_wait(q_empty(side), (use - 1) & 1, p.timeout_ns, abort_flag)) {
          qn[side]--;
          return stop(1);
        }
        load_tile(q_s + side * kTileBytes, x, y, q_full(side));
      };
      Item it;
      for (int r = 0; r * (int)gridDim.x < p.items && ok; ++r) {
        if (!item_of<SPLIT>(p, r, it)) continue;
        const int b = it.bh / p.heads, h = it.bh - b * p.heads;
        const int y0 = b * p.seq, xq = h * D, xk = (p.heads + h) * D, xv = (2 * p.heads + h) * D;
        load_q(0, xq, y0 + it.qa * BQ);
        load_kv(xk, y0);
        if (!SPLIT && it.nb > 0) load_q(1, xq, y0 + (it.qa + 1) * BQ);
        if (lead == 2 && it.n > 1) load_kv(xk, y0 + BKV);
        for (int i = 0; i < it.n && ok; ++i) {
          load_kv(xv, y0 + i * BKV);
          if (i + lead < it.n) load_kv(xk, y0 + (i + lead) * BKV);
        }
      }
      if (*abort_flag) {   // loads in flight still write into shared memory: wait for each, bounded
        for (int s = 0; s < kSlots; ++s) {
          const uint32_t n = (pos + kSlots - 1 - s) / kSlots;
          if (n > 0) mbar_wait(kv_full(s), (n - 1) & 1, 200000, never);
        }
        for (int x = 0; x < 2; ++x)
          if (qn[x] > 0) mbar_wait(q_full(x), (qn[x] - 1) & 1, 200000, never);
      }
    }
  } else if (warp == 9) {
    if (elect_one()) {   // elect.sync, not a lane number: see the same place in gemm_local.cu
      constexpr uint32_t idesc_qk = umma_idesc_f16_major(BQ, BKV, !F16, false, false);
      constexpr uint32_t idesc_pv = umma_idesc_f16_major(BQ, D, !F16, false, true);   // V is MN-major
      bool ok = true;
      uint32_t base = 0;                      // ring position of the current item's first tile
      uint32_t sn[2] = {0, 0};                // tiles whose P has been waited for, per side
      uint32_t qn[2] = {0, 0};                // Q tiles taken into use, per buffer
      uint32_t on[2] = {0, 0};                // items begun, per side
      bool ahead[2] = {false, false};         // the item's first scores are already under way
      auto stop = [&](int what) {
        record_status(p.status, kTimeout, kSiteMma, blockIdx.x, base, what);
        *abort_flag = 1;
        ok = false;
      };
      auto pos_k = [&](int i) { return (uint32_t)(i + (i >= lead ? i - lead + 1 : 0)); };
      auto pos_v = [&](const Item& it, int i) { return (uint32_t)(i + (i + lead < it.n ? i + lead : it.n)); };
      auto key_tile = [&](int x, int j) { return SPLIT ? 2 * j + x : j; };
      // a tile's slot is free after its last use: side B's where both sides use it
      auto last_use = [&](const Item& it, int x, int j) { return SPLIT || x == 1 || j >= it.nb; };
      // S = Q K_j^T of side x; `first` = ring position of the item's first tile
      auto scores = [&](const Item& it, uint32_t first, int x, int j) {
        const int kt = key_tile(x, j);
        const uint32_t pos = first + pos_k(kt);
        const int s = pos % kSlots;
        if (!mbar_wait(kv_full(s), (pos / kSlots) & 1, p.timeout_ns, abort_flag)) return stop(1);
        tc_fence_after();
        const uint64_t qd = umma_desc_k_sw128(q_s + (SPLIT ? 0 : x) * kTileBytes);
        const uint64_t kd = umma_desc_k_sw128(ring + s * kTileBytes);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = ((kk >> 2) * kHalfBytes + (kk & 3) * 32) >> 4;
          umma_f16_ss(tmem + x * 128, qd + off, kd + off, idesc_qk, kk ? 1u : 0u);
        }
        umma_commit(s_full(x));
        if (last_use(it, x, j)) umma_commit(kv_empty(s));
        // the queries have been read for the last time by the item's last scores (of both sides, when they share them)
        if (SPLIT ? kt == it.n - 1 : j == (x ? it.nb : it.na) - 1) umma_commit(q_empty(SPLIT ? 0 : x));
      };
      // waits for the item's queries on their first use
      auto begin = [&](const Item& it, uint32_t first, int x) {
        if (x == 0 || !SPLIT) {
          if (!mbar_wait(q_full(x), qn[x] & 1, p.timeout_ns, abort_flag)) return stop(0);
          ++qn[x];
        }
        scores(it, first, x, 0);
      };
      Item it, nx;
      int r = 0;
      auto fetch = [&](Item& to) {
        for (; r * (int)gridDim.x < p.items; ++r)
          if (item_of<SPLIT>(p, r, to)) {
            ++r;
            return true;
          }
        return false;
      };
      bool have = fetch(it);
      while (have && ok) {
        const bool more = fetch(nx);
        const uint32_t next = base + 2 * it.n;
        if (!ahead[0]) begin(it, base, 0);
        if (ok && it.nb > 0 && !ahead[1]) begin(it, base, 1);
        ahead[0] = ahead[1] = false;
        const int steps = it.na > it.nb ? it.na : it.nb;
        for (int j = 0; j < steps && ok; ++j) {
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int n = x ? it.nb : it.na;
            if (j >= n || !ok) continue;
            if (j == 0) {
              if (on[x] > 0 && !mbar_wait(o_free(x), (on[x] - 1) & 1, p.timeout_ns, abort_flag)) {
                stop(2);
                break;
              }
              ++on[x];
            }
            const uint32_t pos = base + pos_v(it, key_tile(x, j));
            const int s = pos % kSlots;
            if (!mbar_wait(kv_full(s), (pos / kSlots) & 1, p.timeout_ns, abort_flag) ||
                !mbar_wait(p_half(x), sn[x] & 1, p.timeout_ns, abort_flag)) {
              stop(3);
              break;
            }
            tc_fence_after();
            // 16 keys = two groups of 8 rows (1024 bytes apart); the second 64 columns of d are one half tile further on
            const uint64_t vd = umma_desc_mn_sw128(ring + s * kTileBytes, kHalfBytes, 1024);
            auto product = [&](int k0) {   // 64 keys
#pragma unroll
              for (int kk = k0; kk < k0 + BKV / 32; ++kk)
                umma_f16_ts(tmem + 256 + x * 128, tmem + x * 128 + kk * 8, vd + kk * (16 * 128 >> 4), idesc_pv,
                            (j > 0 || kk > 0) ? 1u : 0u);
            };
            product(0);   // runs while the other half's exponentials are made
            if (!mbar_wait(p_ready(x), sn[x] & 1, p.timeout_ns, abort_flag)) {
              stop(4);
              break;
            }
            ++sn[x];
            tc_fence_after();
            product(BKV / 32);
            if (last_use(it, x, j)) umma_commit(kv_empty(s));
            if (j + 1 < n) {
              scores(it, base, x, j + 1);
            } else {
              umma_commit(o_full(x));
              // go on with the next item on this side if its operands are there already
              if (more && (x == 0 || (nx.nb > 0 && ahead[0]))) {   // (B never before A: see last_use)
                const uint32_t np = next + pos_k(key_tile(x, 0));
                const bool q_here = (x == 1 && SPLIT) || mbar_test(q_full(x), qn[x] & 1);
                if (q_here && mbar_test(kv_full(np % kSlots), (np / kSlots) & 1)) {
                  begin(nx, next, x);
                  ahead[x] = true;
                }
              }
            }
          }
        }
        base = next;
        it = nx;
        have = more;
      }
      if (*abort_flag) {   // MMAs in flight still use shared and tensor memory
        umma_commit(drain_bar);
        mbar_wait(drain_bar, 0, 200000, never);
      }
    }
  } else {
    // ---- softmax: one thread per query row ----
    const int x = warp >> 2;                       // side
    const int row = (warp & 3) * 32 + lane;        // a warp reads the 32 tensor-memory lanes of its quadrant
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_t = tmem + lanes + x * 128, o_t = tmem + lanes + 256;
    volatile float* merge = reinterpret_cast<volatile float*>(smem + kBarBytes + kTileBytes);   // split: Q of B is unused
    bool ok = true;
    uint32_t sn = 0, dn = 0, bn = 0;               // score tiles, items (pair: of this side), items with a side B
    auto stop = [&](int j, int what) {
      if (lane == 0) record_status(p.status, kTimeout, kSiteSoftmax, blockIdx.x, j, what);
      *abort_flag = 1;
      ok = false;
    };
    const float2 scale2 = make_float2(p.scale_log2, p.scale_log2);
    Item it;
    for (int r = 0; r * (int)gridDim.x < p.items && ok; ++r) {
      if (!item_of<SPLIT>(p, r, it)) continue;
      const int n = x ? it.nb : it.na;
      if (n == 0 && !SPLIT) continue;
      const int qt = SPLIT ? it.qa : it.qa + x;
      float m_run = -INFINITY, l_run = 0.f;
#pragma unroll 1
      for (int j = 0; j < n; ++j) {
        if (!mbar_wait(s_full(x), sn & 1, p.timeout_ns, abort_flag)) {
          stop(j, 1);
          break;
        }
        ++sn;
        tc_fence_after();
        // 168 registers do not hold the row and everything else: its last part is read for the maximum and again when
        // its turn comes (P overwrites only the first half of the scores)
        constexpr int kKept = SPLIT ? 64 : 96;
        uint32_t v[kKept];
        const bool diag = p.causal && (SPLIT ? 2 * j + x : j) == qt;   // keys after the query: 0 after the exponential
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};    // four chains instead of one long one
        {
          uint32_t t[128 - kKept];
#pragma unroll
          for (int c = kKept; c < 128; c += 32) tmem_ld_32x32b_x32(s_t + c, t + c - kKept);
#pragma unroll
          for (int c = 0; c < kKept; c += 32) tmem_ld_32x32b_x32(s_t + c, v + c);
          tmem_wait_ld();
          if (diag) mask_after<128 - kKept>(t, row - kKept), mask_after<kKept>(v, row);
#pragma unroll
          for (int i = 0; i < 128 - kKept; i += 8)
#pragma unroll
            for (int c = 0; c < 4; ++c)
              m4[c] = max3(m4[c], __uint_as_float(t[i + 2 * c]), __uint_as_float(t[i + 2 * c + 1]));
        }
#pragma unroll
        for (int i = 0; i < kKept; i += 8)
#pragma unroll
          for (int c = 0; c < 4; ++c)
            m4[c] = max3(m4[c], __uint_as_float(v[i + 2 * c]), __uint_as_float(v[i + 2 * c + 1]));
        const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * p.scale_log2;
        if (j == 0) {
          m_run = mx;
        } else if (__any_sync(0xffffffffu, mx > m_run)) {
          // Each row takes its new maximum at once, so that its largest weight is exactly 1 in the 16 bits of P, and what has
          // been summed is rescaled.  These scores are complete, so the products issued before them are too, and the next
          // one waits for P.  (32 columns at a time and two to an instruction: 317 us for 8 x 2048 x 32 causal from a rest;
          // 16 at a time 328, one to an instruction 322, between the exponentials 336, two loads in flight 328.)
          const float m_new = fmaxf(m_run, mx);
          const float alpha = m_new == m_run ? 1.f : fast_exp2(m_run - m_new);
          const float2 alpha2 = make_float2(alpha, alpha);
          l_run *= alpha;
          m_run = m_new;
          const uint32_t o_x = o_t + x * 128;
#pragma unroll 1
          for (int c = 0; c < D; c += 32) {
            uint32_t o[32];
            tmem_ld_32x32b_x32(o_x + c, o);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const float2 r = mul2(make_float2(__uint_as_float(o[i]), __uint_as_float(o[i + 1])), alpha2);
              o[i] = __float_as_uint(r.x), o[i + 1] = __float_as_uint(r.y);
            }
            tmem_st_32x32b_x16(o_x + c, o);
            tmem_st_32x32b_x16(o_x + c + 16, o + 16);
          }
        }
        // (a row that has seen scores of minus infinity only: they weigh 0, and not the NaN of their difference)
        const float shift = m_run == -INFINITY ? 0.f : -m_run;
        const float2 neg = make_float2(shift, shift);
        float2 s2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c * 32 >= kKept) {   // into registers that are free again
            tmem_ld_32x32b_x32(s_t + c * 32, v + c * 32 % kKept);
            tmem_wait_ld();
            if (diag) mask_after<32>(v + c * 32 % kKept, row - c * 32);
          }
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int e = c * 32 % kKept + 2 * i;
            const float2 t = fma2(make_float2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), scale2, neg);
            const float2 q = SPLIT && i % kPolyEvery == kPolyEvery - 1 ? poly_exp2(t)
                                                              : make_float2(fast_exp2(t.x), fast_exp2(t.y));
            s2[i & 1] = add2(s2[i & 1], q);
            pk[i] = pack2<F16>(q.x, q.y);
          }
          tmem_st_32x32b_x16(s_t + c * 16, pk);   // P: two 16-bit values per column, over the scores this warp has read
          if (c == 1) {
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_half(x));
          }
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_ready(x));
        l_run += (s2[0].x + s2[0].y) + (s2[1].x + s2[1].y);
      }
      // ---- output ----
      const int b = it.bh / p.heads, h = it.bh - b * p.heads;
      uint8_t* orow = reinterpret_cast<uint8_t*>(p.out) +
                      ((int64_t)(b * p.seq + qt * BQ + row) * p.ldo + (int64_t)h * D) * 2;
      auto store = [&](int col, const float* f) {   // 8 columns
        uint4 o;
        o.x = pack2<F16>(f[0], f[1]);
        o.y = pack2<F16>(f[2], f[3]);
        o.z = pack2<F16>(f[4], f[5]);
        o.w = pack2<F16>(f[6], f[7]);
        *reinterpret_cast<uint4*>(orow + col * 2) = o;
      };
      auto release = [&](int side) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(o_free(side));
      };
      if (!SPLIT) {
        if (!ok) break;
        if (!mbar_wait(o_full(x), dn & 1, p.timeout_ns, abort_flag)) {
          stop(n, 2);
          break;
        }
        ++dn;
        tc_fence_after();
        const float inv = 1.f / l_run;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t o[32];
          tmem_ld_32x32b_x32(o_t + x * 128 + c * 32, o);
          tmem_wait_ld();
          if (c == 3) release(x);
          float f[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(o[i]) * inv;
#pragma unroll
          for (int q = 0; q < 4; ++q) store(c * 32 + q * 8, f + q * 8);
        }
      } else {
        // the two sides' maxima and sums, in buffers that alternate from item to item
        volatile float* mine = merge + (dn & 1) * 512;
        mine[x * 256 + row] = m_run;
        mine[x * 256 + 128 + row] = l_run;
        __syncwarp();
        if (lane == 0) mbar_arrive(merge_bar);
        if (!ok) break;
        bool w = mbar_wait(merge_bar, dn & 1, p.timeout_ns, abort_flag);
        w = w && mbar_wait(o_full(0), dn & 1, p.timeout_ns, abort_flag);
        if (it.nb > 0) w = w && mbar_wait(o_full(1), bn & 1, p.timeout_ns, abort_flag);
        if (!w) {
          stop(n, 3);
          break;
        }
        ++dn;
        if (it.nb > 0) ++bn;
        tc_fence_after();
        const float ma = mine[row], la = mine[128 + row], mb = mine[256 + row], lb = mine[384 + row];
        float fa = 1.f, fb = 0.f;
        if (it.nb > 0) {
          const float m = fmaxf(ma, mb);
          fa = ma == m ? 1.f : fast_exp2(ma - m);
          fb = mb == m ? 1.f : fast_exp2(mb - m);
        }
        const float inv = 1.f / (la * fa + (it.nb > 0 ? lb * fb : 0.f));
        fa *= inv;
        fb *= inv;
        // side A writes the first 64 columns, side B the others
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          const int col = x * 64 + c * 16;
          uint32_t o[16], o2[16];
          tmem_ld_32x32b_x16(o_t + col, o);
          if (it.nb > 0) tmem_ld_32x32b_x16(o_t + 128 + col, o2);
          tmem_wait_ld();
          if (c == 3) {
            release(0);
            if (it.nb > 0) release(1);
          }
          float f[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(o[i]) * fa;
          if (it.nb > 0) {
#pragma unroll
            for (int i = 0; i < 16; ++i) f[i] += __uint_as_float(o2[i]) * fb;
          }
          store(col, f);
          store(col + 8, f + 8);
        }
      }
    }
  }

  // ---- teardown ----
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    __syncwarp();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace attn
}  // namespace iris

// ================================================================================================
// Host side
// ================================================================================================
namespace {
thread_local char g_attn_err[256] = "";

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn attn_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, []() {
    void* q = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &r) == cudaSuccess &&
        r == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(q);
    else
      (void)cudaGetLastError();
  });
  return fn;
}
// Whether the two sides of a CTA share out the keys of one query tile instead of taking two query tiles: if the CTA with
// the most to do is done clearly earlier.  Time is counted in steps in which both sides do a tile of keys, plus one step
// per item for its start and its output.  Half the chain is what counts when there are few items (pairs -> keys shared out):
// 3 x 384 tokens x 5 heads 11.7 -> 8.1 us, 2 x 1024 x 12 causal 22.6 -> 15.4, 1 x 4096 x 4 causal 67.2 -> 38.1; with many items
// the pairs win, because they load every key tile once for 256 queries instead of 128.
bool split_keys(int batch, int seq, int heads, bool causal, int sms) {
  const long long nq = seq / iris::attn::BQ, bh = (long long)batch * heads;
  auto makespan = [&](bool split) {
    const long long blocks = split ? nq : (nq + 1) / 2;
    long long total = 0, longest = 0;
    for (long long b = 0; b < blocks; ++b) {
      const long long keys = !causal ? nq : split ? b + 1 : (2 * b + 2 < nq ? 2 * b + 2 : nq);
      const long long steps = (split ? (keys + 1) / 2 : keys) + 1;
      total += steps;
      if (steps > longest) longest = steps;
    }
    const long long even = (total * bh + sms - 1) / sms;
    // equal items: whole rounds
    const long long rounds = (blocks * bh + sms - 1) / sms;
    const long long t = causal ? even : rounds * longest;
    return t > longest ? t : longest;
  };
  return 1.15 * makespan(true) < makespan(false);
}
}  // namespace

extern "C" {

const char* iris_attention_last_error() { return g_attn_err; }

// qkv: [batch * seq, 3 * heads * 128] (row pitch ld_qkv elements): columns [0, heads*128) are Q, the next heads*128 K,
// the last heads*128 V, head h in columns h*128 .. of each block.  out: [batch * seq, heads * 128] (row pitch ldo).
// dtype: 0 = bf16, 1 = fp16.  seq must be a multiple of 128.  status: iris::StatusBlock on the device or null.
// Returns 0, or a negative code with a message in iris_attention_last_error().
int iris_k_attention_fwd(const void* qkv, int64_t ld_qkv, void* out, int64_t ldo, int batch, int seq, int heads,
                         int causal, int dtype, void* status, uint64_t timeout_ns, void* stream) {
  using namespace iris::attn;
  g_attn_err[0] = 0;
  if (!qkv || !out || batch < 1 || heads < 1 || seq < BQ || seq % BQ != 0) {
    snprintf(g_attn_err, sizeof(g_attn_err), "attention: need buffers, batch, heads >= 1 and seq a multiple of %d", BQ);
    return -1;
  }
  if (reinterpret_cast<uintptr_t>(qkv) % 16 || reinterpret_cast<uintptr_t>(out) % 16 || (ld_qkv * 2) % 16 ||
      (ldo * 2) % 16 || ld_qkv < 3ll * heads * D || ldo < (int64_t)heads * D) {
    snprintf(g_attn_err, sizeof(g_attn_err), "attention: 16-byte aligned buffers and pitches of at least the row");
    return -1;
  }
  if (dtype != 0 && dtype != 1) {
    snprintf(g_attn_err, sizeof(g_attn_err), "attention: dtype must be 0 (bf16) or 1 (fp16)");
    return -1;
  }
  EncodeTiledFn enc = attn_encode_fn();
  if (!enc) {
    snprintf(g_attn_err, sizeof(g_attn_err), "attention: cuTensorMapEncodeTiled is not available");
    return -2;
  }
  Params p;
  memset(&p, 0, sizeof(p));
  cuuint64_t dims[2] = {(cuuint64_t)3 * heads * D, (cuuint64_t)batch * seq};
  cuuint64_t strides[1] = {(cuuint64_t)ld_qkv * 2};
  cuuint32_t box[2] = {64, 128};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(&p.tm, dtype ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                   const_cast<void*>(qkv), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    snprintf(g_attn_err, sizeof(g_attn_err), "attention: cuTensorMapEncodeTiled failed with %d", (int)r);
    return -2;
  }
  p.out = out;
  p.ldo = ldo;
  p.status = static_cast<iris::StatusBlock*>(status);
  p.timeout_ns = timeout_ns ? timeout_ns : 2000000000ull;
  p.batch = batch;
  p.seq = seq;
  p.heads = heads;
  p.causal = causal ? 1 : 0;
  p.scale_log2 = 1.4426950408889634f / 11.313708498984761f;   // log2(e) / sqrt(128)
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) {
    snprintf(g_attn_err, sizeof(g_attn_err), "attention: no device");
    return -3;
  }
  const int split = split_keys(batch, seq, heads, causal != 0, sms) ? 1 : 0;
  auto kern = split ? (dtype ? attention_fwd_kernel<true, true> : attention_fwd_kernel<false, true>)
                    : (dtype ? attention_fwd_kernel<true, false> : attention_fwd_kernel<false, false>);
  static std::once_flag attr_once[4];
  cudaError_t e = cudaSuccess;
  std::call_once(attr_once[dtype * 2 + split], [&]() {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  });
  if (e != cudaSuccess) {
    snprintf(g_attn_err, sizeof(g_attn_err), "attention: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    return -3;
  }
  p.blocks = split ? seq / BQ : (seq / BQ + 1) / 2;
  // Heads dealt out together: two rounds of items, the lengths of which then add up to the same for every CTA, and whose
  // K and V (about 300 items x 256 rows x 512 bytes = 39 MB) stay in L2 until their last item.
  p.group = (2 * sms + p.blocks - 1) / p.blocks;
  if ((long long)batch * heads * p.blocks > 0x7fffffffLL / 2) {
    snprintf(g_attn_err, sizeof(g_attn_err), "attention: too many query tiles");
    return -1;
  }
  p.items = batch * heads * p.blocks;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.items < sms ? p.items : sms);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see grid_dependency_wait() in the kernel
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* args[] = {&p};
  e = cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(kern), args);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();   // reported here: it must not turn up at someone else's launch
    snprintf(g_attn_err, sizeof(g_attn_err), "attention: launch: %s", cudaGetErrorString(e));
    return -3;
  }
  return 0;
}

}  // extern "C"
