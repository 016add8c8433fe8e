// The two products of the routed feed-forward (moe.cu) for prompts, bfloat16, on the 5th-generation tensor cores: tiles of
// up to 256 rows of one expert times 256 weight rows, a tile to a pair of multiprocessors.
//
// What bounds it: the tensor pipe.  A tile's operands come through the L2 cache, and a single multiprocessor's tile of
// 128 x 256 asks it for 94 bytes a clock at full rate, more than it gives; the pair (`tcgen05.mma.cta_group::2`, M = 256,
// N = 256) shares the weight rows - each block of a cluster of two holds 128 of the tile's rows and 128 of its
// weight rows - and needs 62.
//   warp 4   loads: per 64 columns of k one box of 128 weight rows and one of the block's 128 rows, both with the 128-byte
//            swizzle, into a ring of six stages.  down's rows lie in the experts' order; gate_up's are brought into it
//            by a copy in front (moe_gather_kernel).  (Gathered inside, by `tile::gather4` loads of four rows, a
//            stage waited for its 32 gathers: 43 ns each, 594 us for the product that takes 210 + 16 us so.)
//   warp 5   one thread of the even block issues the pair's MMAs; `tcgen05.commit` frees a stage in both blocks.
//   warps 0-3  write a finished tile out of tensor memory (its 512 columns hold two tiles: one is written while the other
//            is summed up).
// The grid is one pair per two multiprocessors; a pair takes every n-th of (row tile, weight tile), weight tiles
// fastest, so that all pairs together work on one or two experts, whose weights and rows the L2 cache holds.
//   gate_up  the even block's weight rows are 128 gate rows, the odd block's the up rows of the same columns, so
//            silu(gate) * up is formed by the thread that reads both halves of a row from tensor memory.
//   down     a row's result times its pair's routing weight, float32, to the pair's row.
// Every wait is bounded; a thread whose wait runs out raises an error flag (mll_take_device_error) and the block leaves its
// loops, meets the other block, frees its tensor memory and returns.  No load uses cluster multicast.
// Measured (16 experts of 2,048 x 2,048; us, copy and gate_up / down; in brackets the mma.sync kernel on tiles of 128 rows
// that took these steps before): 15,880 pairs 226 / 120 = 1.18 / 1.11 PFLOP/s (884 / 465); 8,192: 151 / 81 (510 / 269);
// 2,048: 85 / 43 (196 / 114), where each expert's weights from memory alone take 62 us; 528: 93 / 32 (135 / 72).
#include <cooperative_groups.h>
#include <cuda.h>

#include "common.cuh"
#include "device_error.h"
#include "moe.cuh"
#include "tensor_map.h"

namespace mll {

constexpr int MT5_THREADS = 192;
constexpr int MT5_ROWS = 128;                        // rows, and weight rows, of one block of a pair
constexpr int MT5_KB = 64;                           // columns of k a stage: one 128-byte swizzle span
constexpr int MT5_HALF = MT5_ROWS * MT5_KB * 2;      // bytes of one operand of a stage
constexpr int MT5_STAGE = 2 * MT5_HALF;
constexpr int MT5_STAGES = 6;
constexpr size_t MT5_SMEM = 1024 + (size_t)MT5_STAGES * MT5_STAGE + 256;
constexpr long long MT5_WAIT_CLOCKS = 2ll << 30;

struct MoeTc5Args {
  void* out;
  const float* pair_weight;  // [pairs] (down)
  MoePlan plan;
  int k, n;
  int* error;  // raised by a bounded wait that ran out: the flag of the tcgen05 products (device_error.h)
};

__device__ __forceinline__ unsigned g_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned g_of_rank(unsigned addr, unsigned rank) {  // the same place in block `rank` of the cluster
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void g_mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ bool g_mbar_try(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
__device__ __forceinline__ bool g_mbar_wait(unsigned bar, unsigned parity, volatile int* gave_up, int* error) {
  if (g_mbar_try(bar, parity)) return true;
  const long long began = clock64();
  while (clock64() - began < MT5_WAIT_CLOCKS) {
    if (g_mbar_try(bar, parity)) return true;
    if (*gave_up) return false;
  }
  *gave_up = 1;
  if (error) atomicExch(error, 1);
  return false;
}
__device__ __forceinline__ void g_tma_box(unsigned dst, const CUtensorMap* map, int c, int r, unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(c), "r"(r), "r"(bar) : "memory");
}
// K-major tile with rows of 128 bytes and the 128-byte swizzle (see linear_tc5.cu)
__device__ __forceinline__ unsigned long long g_desc(unsigned addr) {
  return (unsigned long long)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((unsigned long long)(1024 >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void g_mma_pair(unsigned tmem_d, unsigned long long a, unsigned long long b, unsigned accumulate) {
  // float32 accumulator, bfloat16 A and B, both K-major, N = 256, M = 256
  constexpr unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((256u >> 4) << 24);
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on the barrier at this place in both blocks once every MMA issued before is complete
__device__ __forceinline__ void g_commit_both(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((unsigned short)3) : "memory");
}
__device__ __forceinline__ void g_tmem_ld32(unsigned (&v)[32], unsigned addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(addr));
}
__device__ __forceinline__ unsigned g_pack(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const unsigned*>(&h);
}

__device__ __forceinline__ float g_swiglu(unsigned gate, unsigned up) {
  const float g = __uint_as_float(gate);
  return g / (1.f + __expf(-g)) * __uint_as_float(up);
}

// KIND 0: down; 1: gate_up (silu(gate) * up); 2: up alone with gelu (erf form)
template <int KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(MT5_THREADS, 1)
moe_tc5_kernel(const __grid_constant__ CUtensorMap rows_map, const __grid_constant__ CUtensorMap w_map, MoeTc5Args a) {
  constexpr int STEP = KIND == 1 ? MT5_ROWS : 2 * MT5_ROWS;  // output columns of a tile
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  // full[S], empty[S], tile_full[2], tile_empty[2]
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(base + (size_t)MT5_STAGES * MT5_STAGE);
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 2 * MT5_STAGES + 4);
  volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const unsigned full = g_smem(bars), empty = full + 8 * MT5_STAGES, tile_full = empty + 8 * MT5_STAGES,
                 tile_empty = tile_full + 16;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));

  if (tid == 0) {
    for (int s = 0; s < MT5_STAGES; ++s) {
      g_mbar_init(full + 8 * s, 1);   // the even block's: its loader's arrival and the bytes of both blocks
      g_mbar_init(empty + 8 * s, 1);  // one commit of the pair's MMAs
    }
    for (int b = 0; b < 2; ++b) {
      g_mbar_init(tile_full + 8 * b, 1);
      g_mbar_init(tile_empty + 8 * b, 8);  // the even block's: the writing warps of both blocks
    }
    *gave_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(g_smem(tmem_slot)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cooperative_groups::this_cluster().sync();  // both blocks' barriers stand
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = *tmem_slot;

  const int k_blocks = (a.k + MT5_KB - 1) / MT5_KB;
  const int across = (a.n + STEP - 1) / STEP;
  const int total = a.plan.n_tiles[0] * across;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  if (warp == 4) {
    // ---- loads ------------------------------------------------------------------------------------------------- //
    const unsigned full_even = g_of_rank(full, 0);
    int it = 0;
    bool ok = true;
    for (int work = pair; work < total && ok; work += pairs) {
      const int tile = work / across, n0 = (work % across) * STEP;
      const int e = a.plan.tile_expert[tile], row0 = a.plan.tile_row0[tile];
      const int w_row = KIND == 1 ? e * 2 * a.n + (int)rank * a.n + n0 : e * a.n + n0 + (int)rank * MT5_ROWS;
      for (int kb = 0; kb < k_blocks; ++kb, ++it) {
        const int s = it % MT5_STAGES;
        ok = g_mbar_wait(empty + 8 * s, ((it / MT5_STAGES) & 1) ^ 1, gave_up, a.error);
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        const unsigned dst = g_smem(base) + s * MT5_STAGE;
        if (lane == 0) {
          if (rank == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full + 8 * s),
                         "r"(2u * MT5_STAGE) : "memory");
          g_tma_box(dst + MT5_HALF, &w_map, kb * MT5_KB, w_row, full_even + 8 * s);
          g_tma_box(dst, &rows_map, kb * MT5_KB, row0 + (int)rank * MT5_ROWS, full_even + 8 * s);
        }
      }
    }
    // The commits that free the last stages arrive in both blocks and nothing above waits for them: a block that left before
    // could have one arrive in shared memory that is another's by then.  (A stage that was never filled passes at once.)
    for (int left = 0; left < MT5_STAGES && ok; ++left, ++it) {
      ok = g_mbar_wait(empty + 8 * (it % MT5_STAGES), ((it / MT5_STAGES) & 1) ^ 1, gave_up, a.error);
      ok = __all_sync(0xffffffffu, ok);
    }
  } else if (warp == 5) {
    // ---- products ---------------------------------------------------------------------------------------------- //
    if (rank == 0 && lane == 0) {
      int it = 0, t = 0;
      bool ok = true;
      for (int work = pair; work < total && ok; work += pairs, ++t) {
        const int b = t & 1;
        ok = g_mbar_wait(tile_empty + 8 * b, ((t >> 1) & 1) ^ 1, gave_up, a.error);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % MT5_STAGES;
          ok = g_mbar_wait(full + 8 * s, (it / MT5_STAGES) & 1, gave_up, a.error);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const unsigned at = g_smem(base) + s * MT5_STAGE;
#pragma unroll
          for (int ks = 0; ks < MT5_KB / 16; ++ks)
            g_mma_pair(tmem + b * 256, g_desc(at + ks * 32), g_desc(at + MT5_HALF + ks * 32), (kb | ks) ? 1u : 0u);
          g_commit_both(empty + 8 * s);
        }
        if (!ok) break;
        g_commit_both(tile_full + 8 * b);
      }
    }
  } else {
    // ---- results ------------------------------------------------------------------------------------------------ //
    const unsigned tile_empty_even = g_of_rank(tile_empty, 0);
    const unsigned lanes = tmem + ((unsigned)(warp * 32) << 16);
    int t = 0;
    for (int work = pair; work < total; work += pairs, ++t) {
      const int tile = work / across, n0 = (work % across) * STEP, b = t & 1;
      const int e = a.plan.tile_expert[tile];
      const int place = a.plan.tile_row0[tile] + (int)rank * MT5_ROWS + warp * 32 + lane;
      const bool mine = place < a.plan.offsets[e + 1];
      const int to = KIND == 0 ? (mine ? a.plan.order[place] : 0) : place;
      const float factor = KIND == 0 && mine ? a.pair_weight[to] : 0.f;
      const bool ok = g_mbar_wait(tile_full + 8 * b, (t >> 1) & 1, gave_up, a.error);
      if (!__all_sync(0xffffffffu, ok)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
      for (int c = 0; c < STEP; c += 32) {
        __syncwarp();  // the loads from tensor memory are the whole warp's
        unsigned v[32];
        g_tmem_ld32(v, lanes + b * 256 + c);
        if (KIND == 1) {
          unsigned u[32];
          g_tmem_ld32(u, lanes + b * 256 + MT5_ROWS + c);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int i = 0; i < 32; i += 2)
            v[i / 2] = g_pack(g_swiglu(v[i], u[i]), g_swiglu(v[i + 1], u[i + 1]));
        } else {
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (KIND == 2) {
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const float x = __uint_as_float(v[i]), y = __uint_as_float(v[i + 1]);
              v[i / 2] = g_pack(0.5f * x * (1.f + erff(x * 0.70710678118654752f)), 0.5f * y * (1.f + erff(y * 0.70710678118654752f)));
            }
          }
        }
        // a.n is a multiple of 8: eight columns are inside the matrix or outside as a whole
        if (!mine) {
        } else if (KIND == 0) {
          float* dst = (float*)a.out + (size_t)to * a.n + n0 + c;
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            if (n0 + c + i < a.n)
              *reinterpret_cast<float4*>(dst + i) = make_float4(factor * __uint_as_float(v[i]), factor * __uint_as_float(v[i + 1]),
                                                                factor * __uint_as_float(v[i + 2]), factor * __uint_as_float(v[i + 3]));
        } else {
          __nv_bfloat16* dst = (__nv_bfloat16*)a.out + (size_t)to * a.n + n0 + c;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (n0 + c + 8 * i < a.n)
              *reinterpret_cast<uint4*>(dst + 8 * i) = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(tile_empty_even + 8 * b) : "memory");
    }
  }
  if (*gave_up) {  // copies may still be on their way into this block's shared memory
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cooperative_groups::this_cluster().sync();  // the other block has read its tiles and needs these barriers no more
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 5)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// rows[place] = h[token of the place's pair], 16 bytes a thread: bound by memory (15,880 rows of 2,048: 16 us, 7.9 TB/s
// with the reads from the L2 cache)
__global__ void moe_gather_kernel(const uint4* __restrict__ h, uint4* __restrict__ rows, const int* __restrict__ order, int top,
                                  int words, long long total) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int place = (int)(i / words), c = (int)(i % words);
    rows[i] = h[(size_t)(order[place] / top) * words + c];
  }
}

template <int KIND>
int launch_moe_tc5(const void* rows, long long n_rows, const void* w, long long w_rows, MoeTc5Args a, int max_tiles,
                   cudaStream_t stream) {
  MllDeviceErrorWords errors;
  mll_device_error_words(&errors);  // all null if they cannot be had: a wait that ran out is then not reported
  a.error = errors.word[1];
  auto kernel = moe_tc5_kernel<KIND>;
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MT5_SMEM);
  if (err != cudaSuccess) {
    mll_set_error("moe (tc5): cannot reserve %zu bytes of shared memory: %s", MT5_SMEM, cudaGetErrorString(err));
    return (int)err;
  }
  CUtensorMap rows_map, w_map;
  if (tensor_map_bf16(rows, n_rows, a.k, MT5_ROWS, &rows_map) != 0) return -1;
  if (tensor_map_bf16(w, w_rows, a.k, MT5_ROWS, &w_map) != 0) return -1;
  const int step = KIND == 1 ? MT5_ROWS : 2 * MT5_ROWS;
  const long long most = (long long)max_tiles * ((a.n + step - 1) / step);
  const int pairs = (int)(most < mll_sm_count() / 2 ? most : mll_sm_count() / 2);
  MLL_LAUNCH((kernel), 2 * pairs, MT5_THREADS, MT5_SMEM, stream, rows_map, w_map, a);
  MLL_LAUNCH_CHECK();
  return 0;
}

}  // namespace mll

int mll_moe_tc5_rows() { return 2 * mll::MT5_ROWS; }

// The products of moe_mma.cu on tiles of mll_moe_tc5_rows() rows; n_pairs and n_experts (those with matrices) size the
// tensor maps; rows: room for [n_pairs, width] bfloat16.
int mll_moe_gate_up_tc5(const void* h, void* rows, const void* w, void* act, const mll::MoePlan& plan, int max_tiles,
                        int n_pairs, int n_experts, int width, int inter, int top, int form, cudaStream_t stream) {
  const long long total = (long long)n_pairs * (width / 8);
  long long blocks = (total + 255) / 256;
  if (blocks > mll_sm_count() * 16) blocks = mll_sm_count() * 16;
  MLL_LAUNCH((mll::moe_gather_kernel), (int)blocks, 256, 0, stream, (const uint4*)h, (uint4*)rows, (const int*)plan.order, top,
             width / 8, total);
  MLL_LAUNCH_CHECK();
  mll::MoeTc5Args a{act, nullptr, plan, width, inter, nullptr};
  if (form == 1) return mll::launch_moe_tc5<2>(rows, n_pairs, w, (long long)n_experts * inter, a, max_tiles, stream);
  return mll::launch_moe_tc5<1>(rows, n_pairs, w, (long long)n_experts * 2 * inter, a, max_tiles, stream);
}

int mll_moe_down_tc5(const void* act, const void* w, float* y, const float* pair_weight, const mll::MoePlan& plan,
                     int max_tiles, int n_pairs, int n_experts, int inter, int width, cudaStream_t stream) {
  mll::MoeTc5Args a{y, pair_weight, plan, inter, width, nullptr};
  return mll::launch_moe_tc5<0>(act, n_pairs, w, (long long)n_experts * width, a, max_tiles, stream);
}
