// gemm_local.cu — GEMM of a world of one on the 5th-generation tensor cores, from one row to a few waves of tiles.
//
//   C[M, N] = A[M, K] * B[N, K]^T        (both operands K-contiguous; C has the operands' element type)
//
// With one rank every collective of gemm_fused.cu is the identity, so what is left is the product.  The fused kernel
// has fixed 48 KB ring stages, tiles of 64 / 128 / 256 columns and one CTA (pair) per tile, which leaves most of the
// GPU idle on the shapes of a decode step or a short prefill: few tiles, each walking all of K alone.  Here
//   * the tile is 128 rows by any multiple of 16 columns up to 256, and the ring takes as many stages as fit, so that a
//     narrow tile still has about 190 KB of operands in flight per SM (bandwidth x latency of HBM asks for about 45 KB;
//     a narrow tile in the fused kernel had 32 KB);
//   * the operands may change places (`swap`: the 128 rows are rows of B, the columns are the few rows of A), so that a
//     matrix of one to 64 rows does not spend a 128-row operand tile on padding;
//   * the K range of a tile may be cut over the CTAs of a cluster (`split`): each keeps its partial sums in its own
//     tensor memory, sends them as fp32 through distributed shared memory to the CTA that owns the rows, and the owner
//     adds them in a fixed order.  No workspace, no flags, nothing to clear, and the result does not depend on timing;
//   * the SwiGLU of a gate and a linear projection, whose rows of B lie in two blocks, can be made on the way out of tensor
//     memory (`glu`): a tile takes half of its columns from either block, and neither projection is written to memory
//     (16384 tokens x 11008 x 4096: one pass of 1.08 GB less per layer, the four-layer decoder 22.6 -> 21.7 ms);
//   * with more tiles than SMs (split 1) a CTA walks over its tiles, two accumulators deep, as the fused kernel does.
//
// What bounds it: a few rows, the weights' bytes (1 x 4096 x 11008 bf16: 26.0 us in the fused kernel, 18.0 us here, 5.0 TB/s);
// hundreds of rows, loads out of L2 and the number of CTAs (256 x 4096 x 11008: 71 -> 24 us); thousands, the tensor cores
// and the GPU's power limit (8192 x 14336 x 4096 back to back: 769 -> 711 us, 1.35 PFLOP/s; int8 8192 x 3584 x 14336: 347 ->
// 302 us; fp32 2048 x 4096 x 4096: 130 -> 111 us).
//
// Roles (320 threads, one CTA per SM): warp 0 TMA producer, warp 1 MMA issuer, warps 2-9 epilogue.  The producer starts
// before the block's set-up barrier (it needs only the ring barriers, which it initialises itself).
//
// Every wait on an mbarrier is bounded by timeout_ns: on expiry the CTA records a status, its roles leave their loops,
// all CTAs still meet at the cluster barriers, tensor memory is released and the kernel returns.
//
// Replaces, for one rank, the reference's persistent kernels (examples/07_gemm_all_scatter/gemm_all_scatter.py:97-255
// and the copies in 08 and 09).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>

#include <mutex>
#include <new>

#include "gemm_fused.cuh"
#include "gemm_schedule.h"
#include "iris/iris.cuh"
#include "iris/ptx_sm100.cuh"

namespace iris {
namespace gemm_local {

using namespace iris::ptx;
using iris::gemm::elem_size;
using iris::gemm::kBf16;
using iris::gemm::kFp16;
using iris::gemm::kInt8;
using iris::gemm::kTf32;

constexpr int kRows = 128;             // rows of a tile (the M of the MMA)
constexpr int kMaxCols = 256;
constexpr int kRowsBytes = kRows * 128;  // one stage of the 128-row operand: 128 bytes of K per row
constexpr int kMaxStages = 12;
constexpr int kMaxCluster = 8;         // portable cluster size
constexpr int kEpiWarps = 8;
constexpr int kThreads = 64 + 32 * kEpiWarps;
constexpr int kBarBytes = 1024;        // barriers and the small shared words, in front of the ring
constexpr int kStagingBytes = kEpiWarps * 32 * 128;   // 32 rows x 128 bytes for every epilogue warp
constexpr int kSmemMax = 227 * 1024;
// Never less than this much shared memory: two CTAs on one SM would wait for one another's tensor memory.
constexpr int kSmemMin = 116 * 1024;

enum Site : uint32_t { kSiteLoad = 110, kSiteMmaAcc = 111, kSiteMmaFull = 112, kSiteEpilogue = 113 };

struct Params {
  CUtensorMap tm_rows;   // the operand whose rows are the tile's 128 rows; box 128 bytes x 128 rows, 128-byte swizzle
  CUtensorMap tm_cols;   // the other one; box 128 bytes x `tn` rows
  void* out;
  int64_t ldo;           // row pitch of out, elements
  StatusBlock* status;
  uint64_t timeout_ns;
  int M, N;              // C is M x N
  int swap;              // 0: tile rows are rows of A (C rows), 1: tile rows are rows of B (C columns)
  int kblocks;           // K in blocks of 128 bytes
  int tn;                // tile width
  int split;             // CTAs per tile along K = cluster size
  int stages;
  int glu;               // B holds N rows of a gate and N of a linear projection: C = silu(A gate^T) * (A linear^T); a tile has
                         // tn / 2 columns of each (split 1, not swapped, 16-bit types)
  int recv_apart;        // split > 1: the receive buffer lies behind the ring (1) or takes its place (0)
  int tiles_r, tiles_c, group;
};

__device__ __forceinline__ uint32_t pack2(float lo, float hi, bool f16) {
  if (f16) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
// 16 bytes into the shared memory of a CTA of the cluster (address in the cluster's shared window).
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// One accumulator value -> the element written to C.
template <int ET>
__device__ __forceinline__ void st_elem(void* out, int64_t index, uint32_t acc) {
  if constexpr (ET == kBf16) reinterpret_cast<__nv_bfloat16*>(out)[index] = __float2bfloat16_rn(__uint_as_float(acc));
  else if constexpr (ET == kFp16) reinterpret_cast<__half*>(out)[index] = __float2half_rn(__uint_as_float(acc));
  else if constexpr (ET == kTf32) reinterpret_cast<uint32_t*>(out)[index] = acc;
  else reinterpret_cast<uint8_t*>(out)[index] = (uint8_t)acc;
}
// 16 accumulator values -> 16 rows of one column of C, of which `rows` exist.  (All 16 without a test each where they do:
// one warp per scheduler runs this at the end of a short kernel, so its instructions count.)
template <int ET>
__device__ __forceinline__ void st_column(void* out, int64_t index, int64_t ldo, int rows, const uint32_t* v) {
  if (rows >= 16) {
#pragma unroll
    for (int i = 0; i < 16; ++i, index += ldo) st_elem<ET>(out, index, v[i]);
  } else {
#pragma unroll
    for (int i = 0; i < 15; ++i, index += ldo)
      if (i < rows) st_elem<ET>(out, index, v[i]);
  }
}
// 16 / sizeof(element) accumulator values -> 16 bytes of C.
template <int ET>
__device__ __forceinline__ uint4 pack16(const uint32_t* v) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (ET == kTf32) w[i] = v[i];
    else if constexpr (ET == kInt8)
      w[i] = (v[4 * i] & 0xffu) | ((v[4 * i + 1] & 0xffu) << 8) | ((v[4 * i + 2] & 0xffu) << 16) | (v[4 * i + 3] << 24);
    else w[i] = pack2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]), ET == kFp16);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
// a / (1 + e^-a), as the SwiGLU kernel of elementwise.cu has it
__device__ __forceinline__ float silu(float a) { return __fdividef(a, 1.f + __expf(-a)); }
template <int ET>
__device__ __forceinline__ uint32_t add_acc(uint32_t a, uint32_t b) {
  if constexpr (ET == kInt8) return a + b;
  else return __float_as_uint(__uint_as_float(a) + __uint_as_float(b));
}

// CG = 2: a pair of CTAs (the two SMs of a TPC) per tile of 256 rows; each loads its own 128 rows and half of the
// columns, the leader's thread issues cta_group::2 MMAs that read both CTAs' shared memory.
template <int ET, int CG>
__global__ void __launch_bounds__(kThreads, 1) local_gemm_kernel(const __grid_constant__ Params p) {
  constexpr int ES = elem_size(ET);
  constexpr int BKE = 128 / ES;   // K elements of a block
  constexpr int EC = 128 / ES;    // output columns of an epilogue piece (128 bytes per row)
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t bar0 = smem_u32(smem);
  const uint32_t ring = bar0 + kBarBytes;
  const uint32_t my_cols = (uint32_t)p.tn / CG;            // columns of the tile this CTA loads
  const uint32_t stage_bytes = kRowsBytes + my_cols * 128u;
  const uint32_t staging = ring + p.stages * stage_bytes;   // split 1: epilogue buffers
  const uint32_t recv = p.recv_apart ? staging : ring;      // split > 1: partial sums from the other pieces
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (kMaxStages + s); };
  auto acc_full_bar = [&](int b) { return bar0 + 8u * (2 * kMaxStages + b); };
  auto acc_empty_bar = [&](int b) { return bar0 + 8u * (2 * kMaxStages + 2 + b); };
  const uint32_t recv_bar = bar0 + 8u * (2 * kMaxStages + 4);
  volatile uint32_t* words = reinterpret_cast<volatile uint32_t*>(smem + 8 * (2 * kMaxStages + 5));
  volatile uint32_t* tmem_slot = words;
  volatile uint32_t* abort_flag = words + 1;
  volatile uint32_t* never = words + 2;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // uniform over the warp
  const int split = p.split;
  const int crank = split * CG > 1 ? (int)cluster_ctarank() : 0;
  const int pr = crank % CG, piece = crank / CG;           // position in the pair (0 = leader), piece of K
  const int lead = crank - pr;                             // cluster rank of the pair's leader
  const int tile0 = blockIdx.x / (split * CG);
  const int step = gridDim.x / (split * CG);
  const int total = p.tiles_r * p.tiles_c;
  const int kb0 = (int)((long long)p.kblocks * piece / split);
  const int kb1 = (int)((long long)p.kblocks * (piece + 1) / split);

  // ---- producer state: warp 0's elected thread; the first ring fill is issued before the set-up barrier ----
  int tile = tile0, kb = kb0, stage = 0;
  uint32_t phase = 0, fills = 0;
  int x_row = 0, x_col = 0;
  bool ok = true;
  auto place = [&](int t) {
    const iris::gemm::TileCoord tc = iris::gemm::raster(t, p.tiles_r, p.tiles_c, p.group);
    x_row = (tc.m_idx * CG + pr) * kRows;
    x_col = p.glu ? tc.n_idx * (p.tn / 2) + pr * p.N : tc.n_idx * p.tn + pr * (int)my_cols;
  };
  auto load_next = [&]() {   // one ring stage; the slot is known to be free
    const uint32_t dst = ring + stage * stage_bytes;
    if (CG == 1) {
      mbar_expect_tx(full_bar(stage), stage_bytes);
      tma_load_2d(dst, &p.tm_rows, kb * BKE, x_row, full_bar(stage));
      tma_load_2d(dst + kRowsBytes, &p.tm_cols, kb * BKE, x_col, full_bar(stage));
      if (p.glu)   // (a pair's CTAs load one half each)
        tma_load_2d(dst + kRowsBytes + p.tn / 2 * 128, &p.tm_cols, kb * BKE, x_col + p.N, full_bar(stage));
    } else {
      // both CTAs' bytes are counted on the leader's barrier, which the leader arms for the pair
      const uint32_t lead_full = mapa_shared(full_bar(stage), lead);
      if (pr == 0) mbar_expect_tx(full_bar(stage), 2 * stage_bytes);
      tma_load_2d_pair(dst, &p.tm_rows, kb * BKE, x_row, lead_full);
      tma_load_2d_pair(dst + kRowsBytes, &p.tm_cols, kb * BKE, x_col, lead_full);
    }
    ++fills;
    if (++stage == p.stages) {
      stage = 0;
      phase ^= 1;
    }
    if (++kb == kb1) {
      kb = kb0;
      tile += step;
      if (tile < total) place(tile);
    }
  };
  if (warp == 0 && elect_one()) {
    prefetch_tensormap(&p.tm_rows);
    prefetch_tensormap(&p.tm_cols);
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full_bar(b), 1);
      mbar_init(acc_empty_bar(b), kEpiWarps * CG);   // one arrival per epilogue warp of every CTA of the tile
    }
    mbar_init(recv_bar, split > 1 ? kEpiWarps * (split - 1) : 1);   // one arrival per sending warp
    *abort_flag = 0;
    *never = 0;
    mbar_fence_init();
    place(tile);
    if (CG == 1) {
      grid_dependency_wait();
      for (int s = 0; s < p.stages && tile < total; ++s) load_next();
    }
  }
  if (warp == 1) {
    if (CG == 1) {
      tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
      tmem_relinquish();
    } else {
      tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
      tmem_relinquish_pair();
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (split > 1 || CG == 2) cluster_arrive();
  if (CG == 2) cluster_wait();       // the leader's barriers exist before the partner's loads arrive on them
  tc_fence_after();
  // Everything up to here overlapped the end of the kernel in front; what follows touches memory.  (The next kernel's
  // blocks may be placed from now on: they find room only on SMs this kernel has left.)
  grid_dependency_wait();
  grid_dependency_launch();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      while (tile < total) {
        if (!mbar_wait(empty_bar(stage), phase ^ 1, p.timeout_ns, abort_flag)) {
          record_status(p.status, kTimeout, kSiteLoad, 0, tile, kb);
          *abort_flag = 1;
          break;
        }
        load_next();
      }
      if (*abort_flag && pr == 0) {
        // leaving early: wait, bounded, for the last fill of every ring slot, which still writes into shared memory
        // (the pair's barriers are the leader's, and the partner stays until the cluster barrier of the teardown)
        for (int s = 0; s < p.stages; ++s) {
          const uint32_t n = (fills + p.stages - 1 - s) / p.stages;
          if (n > 0) mbar_wait(full_bar(s), (n - 1) & 1, 200000, never);
        }
      }
    }
  } else if (warp == 1) {
    // One elected thread.  (Selected with elect.sync and not by its lane number: the compiler then knows that a single
    // thread is left and feeds the tensor-core instructions from uniform registers.  Time per K block of a 16-column
    // tile, which is all issue: 685 cycles with `lane == 0`, 450 with an election in every iteration, 327 like this.)
    if (pr == 0 && elect_one()) {
      constexpr int TM = kRows * CG;
      const uint32_t idesc = ET == kTf32   ? umma_idesc_tf32(TM, p.tn)
                             : ET == kInt8 ? umma_idesc_s8(TM, p.tn)
                                           : umma_idesc_f16(TM, p.tn, ET == kBf16);
      const uint32_t own0 = CG == 1 ? bar0 : mapa_shared(bar0, lead), other0 = CG == 1 ? 0u : mapa_shared(bar0, lead + 1);
      auto commit = [&](uint32_t bar) {   // arrive on this barrier, in both CTAs of a pair, once the MMAs have completed
        if (CG == 1) {
          umma_commit(bar);
        } else {
          umma_commit_pair(own0 + (bar - bar0));
          umma_commit_pair(other0 + (bar - bar0));
        }
      };
      const uint64_t desc0 = umma_desc_k_sw128(ring);
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int t = tile0; t < total && ok; t += step) {
        if (!mbar_wait(acc_empty_bar(acc), acc_phase ^ 1, p.timeout_ns, abort_flag)) {
          record_status(p.status, kTimeout, kSiteMmaAcc, 0, t, acc);
          *abort_flag = 1;
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem + acc * kMaxCols;
        for (int k = kb0; k < kb1; ++k) {
          if (!mbar_wait(full_bar(stage), phase, p.timeout_ns, abort_flag)) {
            record_status(p.status, kTimeout, kSiteMmaFull, 0, t, k);
            *abort_flag = 1;
            ok = false;
            break;
          }
          // (no tcgen05 fence: what the barrier announces was written by TMA, not by another thread's tcgen05 operations)
          // descriptor addresses count in 16-byte units; every kind covers 32 bytes of K per instruction
          const uint64_t a_desc = desc0 + (uint64_t)((stage * stage_bytes) >> 4);
          const uint64_t b_desc = a_desc + (kRowsBytes >> 4);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t accumulate = (k > kb0 || q > 0) ? 1u : 0u;
            if constexpr (ET == kTf32) {
              if (CG == 1) umma_tf32_ss(d, a_desc + 2 * q, b_desc + 2 * q, idesc, accumulate);
              else umma_tf32_ss_pair(d, a_desc + 2 * q, b_desc + 2 * q, idesc, accumulate);
            } else if constexpr (ET == kInt8) {
              if (CG == 1) umma_i8_ss(d, a_desc + 2 * q, b_desc + 2 * q, idesc, accumulate);
              else umma_i8_ss_pair(d, a_desc + 2 * q, b_desc + 2 * q, idesc, accumulate);
            } else {
              if (CG == 1) umma_f16_ss(d, a_desc + 2 * q, b_desc + 2 * q, idesc, accumulate);
              else umma_f16_ss_pair(d, a_desc + 2 * q, b_desc + 2 * q, idesc, accumulate);
            }
          }
          commit(empty_bar(stage));
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        commit(acc_full_bar(acc));
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
    }
  } else if (split == 1) {
    // ---- epilogue of whole tiles: two warps per 32 rows, which take turns with the 128-byte pieces of the tile's width.
    // Each works for itself (its 32 rows go through 4 KB of shared memory of its own), so nothing but its own latency
    // stands between the last MMA and the last store. ----
    const int quad = warp & 3, turn = (warp - 2) >> 2;
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const uint32_t sb = staging + (uint32_t)(warp - 2) * 4096u;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = tile0; t < total; t += step) {
      const iris::gemm::TileCoord tc = iris::gemm::raster(t, p.tiles_r, p.tiles_c, p.group);
      const int width = p.glu ? p.tn / 2 : p.tn;   // columns of C in this tile
      const int r0 = (tc.m_idx * CG + pr) * kRows, c0 = tc.n_idx * width;
      const uint32_t src = tmem + lane_addr + acc * kMaxCols;
      if (!mbar_wait(acc_full_bar(acc), acc_phase, p.timeout_ns, abort_flag)) {
        if (lane == 0) record_status(p.status, kTimeout, kSiteEpilogue, 0, t, acc);
        *abort_flag = 1;
        break;
      }
      tc_fence_after();
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (CG == 1) mbar_arrive(acc_empty_bar(acc));
          else mbar_arrive_cluster(mapa_shared(acc_empty_bar(acc), lead));
        }
      };
      if (p.swap) {
        // a thread holds one column of C: the 32 lanes of a store cover neighbouring columns of one row of C
        const int n = r0 + row;
        for (int c = turn * 16; c < p.tn; c += 32) {
          uint32_t v[16];
          tmem_ld_32x32b_x16(src + c, v);
          tmem_wait_ld();
          if (n < p.N) st_column<ET>(p.out, (int64_t)(c0 + c) * p.ldo + n, p.ldo, p.M - c0 - c, v);
        }
        release();
      } else {
        const int pieces = (width + EC - 1) / EC;
        if (turn >= pieces) release();
#pragma unroll 1
        for (int c = turn; c < pieces; c += 2) {
          uint32_t o[32];   // 128 bytes of this thread's row
          if constexpr (ES == 4) {
            tmem_ld_32x32b_x32(src + c * EC, o);
            tmem_wait_ld();
          } else if constexpr (ES == 2) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              uint32_t v[32];
              tmem_ld_32x32b_x32(src + c * EC + q * 32, v);
              if (p.glu) {
                uint32_t w[32];
                tmem_ld_32x32b_x32(src + width + c * EC + q * 32, w);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  v[j] = __float_as_uint(silu(__uint_as_float(v[j])) * __uint_as_float(w[j]));
              } else {
                tmem_wait_ld();
              }
#pragma unroll
              for (int j = 0; j < 16; ++j)
                o[q * 16 + j] = pack2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]), ET == kFp16);
            }
          } else {
#pragma unroll
            for (int s4 = 0; s4 < 4; ++s4) {
              uint32_t v[32];
              tmem_ld_32x32b_x32(src + c * EC + 32 * s4, v);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                const uint4 w = pack16<ET>(v + 16 * j);
                o[8 * s4 + 4 * j] = w.x;
                o[8 * s4 + 4 * j + 1] = w.y;
                o[8 * s4 + 4 * j + 2] = w.z;
                o[8 * s4 + 4 * j + 3] = w.w;
              }
            }
          }
          if (c + 2 >= pieces) release();
          __syncwarp();   // the piece before this one has been read
#pragma unroll
          for (int j = 0; j < 8; ++j)
            st_shared_v4(sb + lane * 128 + ((j ^ (lane & 7)) << 4), o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
          __syncwarp();
          // out of the buffer with 16-byte stores: 8 lanes cover 128 bytes of a row of C, a warp four rows
          const int left = p.N - (c0 + c * EC), mine = width - c * EC;
          const int bytes = (left < mine ? left : mine) * ES;   // of this piece's row that belong to C
          const int j = lane & 7;
          if (j * 16 < bytes) {
            const int64_t pitch = p.ldo * ES;
            int r = lane >> 3;
            uint8_t* to = reinterpret_cast<uint8_t*>(p.out) + ((int64_t)c0 + c * EC) * ES + j * 16 +
                          (r0 + quad * 32 + r) * pitch;
            const int rows = p.M - (r0 + quad * 32);
#pragma unroll
            for (int i = 0; i < 8; ++i, r += 4, to += 4 * pitch) {
              const uint4 w = ld_shared_v4(sb + r * 128 + ((j ^ (r & 7)) << 4));
              if (r < rows) *reinterpret_cast<uint4*>(to) = w;
            }
          }
        }
      }
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  }

  if (split > 1) {
    // ---- the pieces of a tile meet: the CTA with piece i owns `per` blocks of 16 columns and adds what the others hold
    // of them to its own accumulator.  A block travels as [4 groups of 4 columns][128 rows] x 16 bytes: the 32 lanes of
    // a store write 512 consecutive bytes of the owner's shared memory, and read them back without bank conflicts.
    // (Sending whole rows, 16 bytes per lane at the row pitch, took 3300 cycles for a 128 x 128 tile in two pieces.)
    constexpr uint32_t kBlock = 4 * kRows * 16;
    const int blocks = p.tn / 16;
    const int per = (blocks + split - 1) / split;
    const int quad = warp & 3, row = quad * 32 + lane;
    const int turn = (warp - 2) >> 2;   // two warps per 32 rows take turns with the blocks
    const uint32_t acc = tmem + ((uint32_t)(quad * 32) << 16);
    const iris::gemm::TileCoord tc = iris::gemm::raster(tile0, p.tiles_r, p.tiles_c, p.group);
    const int r = (tc.m_idx * CG + pr) * kRows + row, c0 = tc.n_idx * p.tn;
    bool good = true;
    if (warp >= 2) {
      good = mbar_wait(acc_full_bar(0), 0, p.timeout_ns, abort_flag);
      if (!good) {
        if (lane == 0) record_status(p.status, kTimeout, kSiteEpilogue, 0, tile0, piece);
        *abort_flag = 1;
      }
    }
    __syncwarp();
    if (CG == 1) cluster_wait();   // every CTA of the cluster has started
    if (!p.recv_apart) {
      // The ring is free once the accumulator is complete (every load has been read by an MMA); where the receive
      // buffer takes its place, all CTAs of the cluster have to be that far before anyone sends.
      cluster_sync_all();
    }
    if (warp >= 2) {
      tc_fence_after();
#pragma unroll 1
      for (int i = 1; i < split; ++i) {
        const int to = piece + i < split ? piece + i : piece + i - split;   // everyone starts with another owner
        const int slot = piece < to ? piece : piece - 1;       // the owner's own piece needs no slot
        const int b0 = to * per, b1 = b0 + per < blocks ? b0 + per : blocks;
        const uint32_t peer = mapa_shared(recv, to * CG + pr) + (uint32_t)(slot * per) * kBlock + row * 16;
#pragma unroll 1
        for (int b = b0 + turn; b < b1 && good; b += 2) {
          uint32_t v[16];
          tmem_ld_32x32b_x16(acc + b * 16, v);
          tmem_wait_ld();
          const uint32_t at = peer + (uint32_t)(b - b0) * kBlock;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            st_cluster_v4(at + j * (kRows * 16), v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
      }
      // One fence for all of it, then relaxed arrivals (a release per owner would wait for the stores each time).  The
      // fence comes after the warp's barrier: an arriving lane releases what it knows by its fence, and by the barrier it
      // knows the stores of all lanes.  After a failure the arrivals are made too, so that no one waits for this CTA.
      __syncwarp();
      fence_acq_rel_cluster();
      if (lane < split && lane != piece && lane * per < blocks)
        mbar_arrive_cluster_relaxed(mapa_shared(recv_bar, lane * CG + pr));
    }
    __syncwarp();
    cluster_arrive();   // nothing more is sent from here; waited for below, before this CTA may leave
    if (warp >= 2 && good && piece * per < blocks) {
      good = mbar_wait_cluster(recv_bar, 0, p.timeout_ns, abort_flag);
      if (!good && lane == 0) record_status(p.status, kTimeout, kSiteEpilogue, 1, tile0, piece);
    }
    if (warp >= 2 && good) {
      const int b0 = piece * per, b1 = b0 + per < blocks ? b0 + per : blocks;
#pragma unroll 1
      for (int b = b0 + turn; b < b1; b += 2) {
        uint32_t v[16];
        tmem_ld_32x32b_x16(acc + b * 16, v);
        tmem_wait_ld();
#pragma unroll 1
        for (int s = 0; s < split - 1; ++s) {
          const uint32_t at = recv + (uint32_t)(s * per + b - b0) * kBlock + row * 16;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint4 w = ld_shared_v4(at + j * (kRows * 16));
            v[4 * j] = add_acc<ET>(v[4 * j], w.x), v[4 * j + 1] = add_acc<ET>(v[4 * j + 1], w.y);
            v[4 * j + 2] = add_acc<ET>(v[4 * j + 2], w.z), v[4 * j + 3] = add_acc<ET>(v[4 * j + 3], w.w);
          }
        }
        const int c = c0 + b * 16;
        if (p.swap) {
          if (r < p.N) st_column<ET>(p.out, (int64_t)c * p.ldo + r, p.ldo, p.M - c, v);
        } else if (r < p.M) {
          constexpr int V = 16 / ES;   // columns in 16 bytes of C
#pragma unroll
          for (int q = 0; q < 16 / V; ++q)
            if (c + q * V < p.N)
              *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(p.out) + ((int64_t)r * p.ldo + c + q * V) * ES) =
                  pack16<ET>(v + q * V);
        }
      }
    }
    __syncwarp();
    cluster_wait();
  }

  // ---- teardown ----
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (CG == 2) cluster_sync_all();   // neither CTA of a pair leaves while the other may still touch its memory
  if (warp == 1) {
    __syncwarp();
    if (CG == 1) tmem_dealloc(tmem, 512);
    else tmem_dealloc_pair(tmem, 512);
  }
}

// ================================================================================================
// Host side
// ================================================================================================
namespace {

thread_local char g_err[256] = "";

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
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

int encode_operand(CUtensorMap* out, const void* ptr, int rows, int cols, int64_t ld, int box_rows, int et,
                   const char* what) {
  const int es = elem_size(et);
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    snprintf(g_err, sizeof(g_err), "cuTensorMapEncodeTiled is not available");
    return -1;
  }
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(ld * es)};
  cuuint32_t box[2] = {(cuuint32_t)(128 / es), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  const CUtensorMapDataType dt = et == kFp16   ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                 : et == kTf32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                 : et == kInt8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                               : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const CUresult r = fn(out, dt, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    snprintf(g_err, sizeof(g_err), "cuTensorMapEncodeTiled(%s) failed with %d", what, (int)r);
    return -1;
  }
  return 0;
}

struct Choice {
  int swap, cg, tn, split;
};

int ceil_div(int a, int b) { return (a + b - 1) / b; }
int k_blocks(int K, int es) { return (int)(((int64_t)K * es + 127) / 128); }   // blocks of 128 bytes

// Receive buffer of a split tile.  Up to 64 KB it gets room of its own, so that nobody has to wait for the other CTAs'
// last loads before sending; a larger one would cost too many ring stages and takes the ring's place.
int recv_bytes(int tn, int split) { return split > 1 ? (split - 1) * ceil_div(tn / 16, split) * 16 * kRows * 4 : 0; }
bool recv_apart(int tn, int split) { return split > 1 && recv_bytes(tn, split) <= 64 * 1024; }

// Ring stages and dynamic shared memory of a choice.
int stages_for(int cg, int tn, int split) {
  const int stage = kRowsBytes + tn / cg * 128;
  const int room = kSmemMax - 1024 - kBarBytes -
                   (split > 1 ? (recv_apart(tn, split) ? recv_bytes(tn, split) : 0) : kStagingBytes);
  const int s = room / stage;
  return s > kMaxStages ? kMaxStages : s;
}
int smem_for(int cg, int tn, int split) {
  const int ring = stages_for(cg, tn, split) * (kRowsBytes + tn / cg * 128);
  const int recv = recv_bytes(tn, split);
  const int body = split == 1 ? ring + kStagingBytes : recv_apart(tn, split) ? ring + recv : ring > recv ? ring : recv;
  const int bytes = 1024 + kBarBytes + body;
  return bytes < kSmemMin ? kSmemMin : bytes;
}

// Groups of `c` CTAs that a B200 holds at once with one CTA per SM (the answer of cudaOccupancyMaxActiveClusters: the
// SMs of a GPC do not divide by every cluster size).
int resident_groups(int c, int sms) {
  static const int kOf148[kMaxCluster + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
  const int g = kOf148[c] * sms / 148;
  return g < 1 ? 1 : g;
}

// Which operand supplies the 128-row tiles, CTA pairs or single CTAs, tile width and pieces of K: the combination with
// the smallest estimated time.  The estimate (in us; without what every combination has) has one term for each thing that
// was found to bind somewhere; its constants are a fit to 14600 timings of 330 products (1 .. 16384 rows, all four types) in
// CUDA graphs.  Over those the chosen combination takes 2.6 % more than the fastest one on average, 37 % at worst (a 5 us
// product); over 110 products drawn afterwards 3.6 % (median 0.4 %, one in ten more than 13 %), 34 % at worst (K of two blocks).
//   * a K block (128 bytes of K) takes the longest of: the MMAs, 2 cycles per column of the tile; 340 - 400 cycles of issue;
//     the 1.4 us from one use of a ring slot to the next, shared by the ring's stages; the loads of all SMs at 19 TB/s out
//     of L2.  Rows that do not start on 128 bytes touch one more L2 line each (12 % and 22 % on the last two), and rows past
//     the matrix' edge take time although nothing is loaded for them;
//   * reading every operand once, if that is longer than all K blocks: at 6.8 TB/s, or 8.7 below 50 MB, part of which a
//     program will find in L2;
//   * 1.1 us per wave of tiles and 19 ns per column for the epilogue;
//   * for a split, 1.4 us, and 0.11 us for each piece of 16 columns that a CTA adds up; clusters of three (1 us) and of
//     five or six (0.1 us) start later than the others.
double estimate(const Choice& c, int M, int N, int K, int es, int sms) {
  const int kblocks = k_blocks(K, es);
  const int rows = c.swap ? N : M, cols = c.swap ? M : N;
  const int tiles_r = ceil_div(rows, kRows * c.cg);
  const int cluster = c.cg * c.split;
  const double groups = (double)tiles_r * ceil_div(cols, c.tn);
  const int resident = resident_groups(cluster, sms);
  const double waves = groups <= resident ? 1.0 : (double)((long long)(groups + resident - 1) / resident);
  const double ctas = (groups < resident ? groups : resident) * cluster;
  const bool aligned = (long long)K * es % 128 == 0;
  double per = 2.0 * c.tn / 1900.0;
  const double issue = (c.cg == 1 ? 338.0 : 400.0) / 1900.0;
  if (issue > per) per = issue;
  const double ring = 1.404 * (aligned ? 1.0 : 1.123) / stages_for(c.cg, c.tn, c.split);
  if (ring > per) per = ring;
  const double l2 = ctas * (kRows + c.tn / c.cg) * 128.0 * (aligned ? 1.0 : 1.217) / 18.72e6;
  if (l2 > per) per = l2;
  if (!c.swap) per *= 1.0 + 0.49 * (1.0 - (double)rows / ((double)tiles_r * kRows * c.cg));
  double t = waves * ceil_div(kblocks, c.split) * per;
  const double bytes = ((double)M * K + (double)N * K + (double)M * N) * es;
  const double once = bytes / (bytes > 50e6 ? 6.8e6 : 8.73e6);
  if (once > t) t = once;
  t += 0.59 + 0.0188 * c.tn + (waves - 1.0) * 1.1;
  if (c.split > 1) {
    t += 1.387 + 0.113 * (c.split - 1) * ceil_div(c.tn / 16, c.split);
    t += cluster == 3 ? 1.0 : cluster == 5 || cluster == 6 ? 0.1 : 0.0;
  }
  return t;
}

// `whole`: only forms whose CTAs end with a whole tile (no swap, no split).
void choose(int M, int N, int K, int et, int sms, Choice* best, bool whole = false) {
  const int es = elem_size(et), kblocks = k_blocks(K, es);
  const int grain = et == kInt8 ? 32 : 16;   // N of an MMA
  static const int kSplits[] = {1, 2, 3, 4, 5, 6, 8};
  double best_t = 0;
  best->tn = 0;
  // Up to 64 rows the operands always change places: 128-row tiles that lie mostly past the edge load slowly besides
  // (1 x 22016 x 4096: 44 us against 35).
  for (int swap = M <= kRows / 2 && !whole ? 1 : 0; swap <= (M <= 2 * kRows && !whole ? 1 : 0); ++swap) {
    const int rows = swap ? N : M, cols = swap ? M : N;
    for (int cg = 1; cg <= (rows > kRows ? 2 : 1); ++cg) {
      for (int tn = grain; tn <= kMaxCols; tn += grain) {
        if (tn >= cols + grain) break;
        const double groups = (double)ceil_div(rows, kRows * cg) * ceil_div(cols, tn);
        for (int s : kSplits) {
          // a split is for tiles that do not fill the GPU by themselves
          if (s > 1 && (whole || cg * s > kMaxCluster || 2 * s > kblocks || groups > resident_groups(cg * s, sms))) break;
          const Choice c = {swap, cg, tn, s};
          const double t = estimate(c, M, N, K, es, sms);
          if (best->tn == 0 || t < best_t) {
            best_t = t;
            *best = c;
          }
        }
      }
    }
  }
}

using KernelFn = void (*)(const Params);
KernelFn kernel_for(int et, int cg) {
  if (cg == 2)
    return et == kFp16 ? local_gemm_kernel<kFp16, 2> : et == kTf32 ? local_gemm_kernel<kTf32, 2>
           : et == kInt8 ? local_gemm_kernel<kInt8, 2> : local_gemm_kernel<kBf16, 2>;
  return et == kFp16 ? local_gemm_kernel<kFp16, 1> : et == kTf32 ? local_gemm_kernel<kTf32, 1>
         : et == kInt8 ? local_gemm_kernel<kInt8, 1> : local_gemm_kernel<kBf16, 1>;
}

struct Plan {
  Params p;
  int grid, smem, et, cg, device;
};

constexpr int kMaxDevices = 64;

// Number of SMs of `device`; also allows the kernels their shared memory there, once.
int prepare_device(int device) {
  static std::once_flag once[kMaxDevices];
  static int sms[kMaxDevices];
  if (device < 0 || device >= kMaxDevices) return 0;
  std::call_once(once[device], [&]() {
    int prev = -1, n = 0;
    if (cudaGetDevice(&prev) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) {
      (void)cudaGetLastError();
      return;
    }
    bool fine = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) == cudaSuccess;
    for (int i = 0; i < 8; ++i)
      fine = fine && cudaFuncSetAttribute(kernel_for(i / 2, 1 + i % 2), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          kSmemMax) == cudaSuccess;
    cudaSetDevice(prev);
    if (fine) sms[device] = n;
    else (void)cudaGetLastError();
  });
  return sms[device];
}

int make_plan(Plan* plan, const void* a, int64_t lda, const void* bt, int64_t ldb, void* out, int64_t ldo, int M, int N,
              int K, int et, int device, void* status, uint64_t timeout_ns, int swap, int cg, int tn, int split,
              int glu = 0) {
  g_err[0] = 0;
  if (M < 1 || N < 1 || K < 1 || et < kBf16 || et > kInt8) {
    snprintf(g_err, sizeof(g_err), "M, N, K must be positive and the element type one of 0..3");
    return -1;
  }
  const int es = elem_size(et);
  if ((int64_t)N * es % 16 != 0 || (int64_t)K * es % 16 != 0) {
    snprintf(g_err, sizeof(g_err), "rows of N and of K elements must be multiples of 16 bytes");
    return -1;
  }
  if (reinterpret_cast<uintptr_t>(a) % 16 || reinterpret_cast<uintptr_t>(bt) % 16 || reinterpret_cast<uintptr_t>(out) % 16 ||
      (lda * es) % 16 || (ldb * es) % 16 || (ldo * es) % 16) {
    snprintf(g_err, sizeof(g_err), "base addresses and row pitches must be multiples of 16 bytes");
    return -1;
  }
  if (M > 1 && ldo < N) {   // (the operands' rows may overlap: they are only read)
    snprintf(g_err, sizeof(g_err), "the output's row pitch is smaller than its rows");
    return -1;
  }
  const int sms = prepare_device(device);
  if (sms < 1) {
    snprintf(g_err, sizeof(g_err), "device %d cannot be set up for the kernel", device);
    return -1;
  }
  Choice c;
  choose(M, glu ? 2 * N : N, K, et, sms, &c, glu != 0);
  if (swap >= 0) c.swap = swap ? 1 : 0;
  if (cg > 0) c.cg = cg;
  if (tn > 0) c.tn = tn;
  if (split > 0) c.split = split;
  const int kblocks = k_blocks(K, es);
  if (c.tn < 16 || c.tn > kMaxCols || c.tn % (et == kInt8 ? 32 : 16) != 0 || c.split < 1 ||
      c.split * c.cg > kMaxCluster || c.split > kblocks || c.cg > 2) {
    snprintf(g_err, sizeof(g_err), "tile width %d (a multiple of 16, of 32 for int8, up to 256) or split %d (clusters of "
             "up to %d, at most the number of K blocks) not possible", c.tn, c.split, kMaxCluster);
    return -1;
  }
  if (glu && (es != 2 || c.swap || c.split > 1)) {
    snprintf(g_err, sizeof(g_err), "the gated form is for 16-bit types, operands not swapped, K whole");
    return -1;
  }
  memset(plan, 0, sizeof(*plan));
  Params& p = plan->p;
  const int rows = c.swap ? N : M, cols = c.swap ? M : glu ? 2 * N : N;
  if (encode_operand(&p.tm_rows, c.swap ? bt : a, rows, K, c.swap ? ldb : lda, kRows, et, c.swap ? "B" : "A") ||
      encode_operand(&p.tm_cols, c.swap ? a : bt, cols, K, c.swap ? lda : ldb, c.tn / (glu ? 2 : c.cg), et, c.swap ? "A" : "B"))
    return -1;
  p.out = out;
  p.ldo = ldo;
  p.status = static_cast<StatusBlock*>(status);
  p.timeout_ns = timeout_ns ? timeout_ns : 2000000000ull;
  p.M = M;
  p.N = N;
  p.swap = c.swap;
  p.kblocks = kblocks;
  p.tn = c.tn;
  p.split = c.split;
  p.recv_apart = recv_apart(c.tn, c.split) ? 1 : 0;
  p.stages = stages_for(c.cg, c.tn, c.split);
  p.tiles_r = ceil_div(rows, kRows * c.cg);
  p.tiles_c = glu ? ceil_div(N, c.tn / 2) : ceil_div(cols, c.tn);
  p.glu = glu ? 1 : 0;
  p.group = 8;
  const int total = p.tiles_r * p.tiles_c;
  plan->grid = c.cg * (c.split > 1 ? total * c.split : (total < sms / c.cg ? total : sms / c.cg));
  plan->smem = smem_for(c.cg, c.tn, c.split);
  plan->et = et;
  plan->cg = c.cg;
  plan->device = device;
  return 0;
}

int launch(const Plan* plan, void* stream) {
  int prev = -1;
  if (cudaGetDevice(&prev) != cudaSuccess || (prev != plan->device && cudaSetDevice(plan->device) != cudaSuccess)) {
    (void)cudaGetLastError();
    snprintf(g_err, sizeof(g_err), "device %d cannot be made current", plan->device);
    return -1;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(plan->grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = plan->smem;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see grid_dependency_wait() in the kernel
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = plan->p.split * plan->cg;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = plan->p.split * plan->cg > 1 ? 2 : 1;
  void* args[] = {const_cast<Params*>(&plan->p)};
  const cudaError_t e = cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(kernel_for(plan->et, plan->cg)), args);
  if (prev != plan->device) cudaSetDevice(prev);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();   // reported here: it must not turn up at someone else's launch
    snprintf(g_err, sizeof(g_err), "launch failed: %s", cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

}  // namespace
}  // namespace gemm_local
}  // namespace iris

using namespace iris::gemm_local;

extern "C" {

const char* iris_gemm_local_last_error() { return g_err; }

// The combination choose() takes on a device of `sms` SMs, and its estimate; callable without a device.
double iris_gemm_local_choice(int M, int N, int K, int dtype, int sms, int* swap, int* cg, int* tn, int* split) {
  Choice c;
  choose(M, N, K, dtype, sms, &c);
  *swap = c.swap, *cg = c.cg, *tn = c.tn, *split = c.split;
  return estimate(c, M, N, K, elem_size(dtype), sms);
}
// What a plan settled on: swap, CTA group, tile width, pieces of K, CTAs, ring stages.
void iris_gemm_local_info(void* h, int* out) {
  const Plan* q = static_cast<Plan*>(h);
  const int v[6] = {q->p.swap, q->cg, q->p.tn, q->p.split, q->grid, q->p.stages};
  memcpy(out, v, sizeof(v));
}

// A prepared product on fixed buffers.  glu: bt has 2 N rows, the gate's and the linear projection's (see Params).  swap (-1), cg (0), tn (0), split (0): what the rule in choose() says.
void* iris_gemm_local_create(const void* a, int64_t lda, const void* bt, int64_t ldb, void* out, int64_t ldo, int M, int N,
                             int K, int dtype, int device, void* status, uint64_t timeout_ns, int swap, int cg, int tn,
                             int split, int glu) {
  Plan* plan = new (std::nothrow) Plan();
  if (!plan) return nullptr;
  if (make_plan(plan, a, lda, bt, ldb, out, ldo, M, N, K, dtype, device, status, timeout_ns, swap, cg, tn, split, glu)) {
    delete plan;
    return nullptr;
  }
  return plan;
}
int iris_gemm_local_launch(void* h, void* stream) { return launch(static_cast<Plan*>(h), stream); }
void iris_gemm_local_destroy(void* h) { delete static_cast<Plan*>(h); }

// The same in one call that keeps nothing.
int iris_gemm_local(const void* a, int64_t lda, const void* bt, int64_t ldb, void* out, int64_t ldo, int M, int N, int K,
                    int dtype, int device, void* status, uint64_t timeout_ns, int swap, int cg, int tn, int split,
                    void* stream) {
  Plan plan;
  if (make_plan(&plan, a, lda, bt, ldb, out, ldo, M, N, K, dtype, device, status, timeout_ns, swap, cg, tn, split)) return -1;
  return launch(&plan, stream);
}

}  // extern "C"
