// Skinny bf16 GEMM on the 5th-generation tensor cores: C[M, N] = A[M, K] * W^T with the weight
// rows as the MMA M dimension (128 per CTA) and the tokens as the MMA N dimension, so a handful
// of tokens still fills a 128-row tcgen05.mma.  This is the tile engine the reference calls
// npu_gemm_mla_vec (src/fst_engine.cpp:465-575): weights stay in their native layout -- [N, K]
// (the b_col_maj kernels) or [K, N] (the b_row_maj kernel, 480) -- and are streamed from HBM
// exactly once.
//
// One CTA = one (128-row weight tile, token tile, K slice).  Warp 0 streams both operands with
// TMA through a ring of 128-byte-swizzled stages; one lane of warp 1 issues tcgen05.mma into a
// TMEM accumulator; warps 2-5 drain TMEM.  The K slices of one output tile form a thread-block
// cluster: every CTA parks its fp32 partial in its own shared memory and then reduces one
// column slice of the tile over all peers through distributed shared memory, in rank order
// (deterministic), without a round trip through global memory.
#include <algorithm>
#include <mutex>
#include <unordered_map>

#include "kernels.cuh"
#include "tc_common.cuh"

namespace fst {

namespace {

constexpr int BK = 64;       // K elements per stage: one 128-byte swizzle span
constexpr int W_TILE = 128;  // weight rows per CTA
constexpr int W_BYTES = W_TILE * BK * 2;
constexpr int GEMM_THREADS = 192;
constexpr int MAX_SPLITS = 8;  // portable cluster size

struct GemmTcParams {
  bf16* C;
  int* d_status;
  int M, N, K, ldc;
  long long c_bs;
  int splits, kc_total, stages;
  int nt, n_tiles, m_tiles, tiles;  // k_gemm_tc_tiles: token tile, weight / token tiles, tiles of all batch members
  int w_swap, a_swap;  // the batch index is the middle tensor-map coordinate (its stride is the smaller one)
  // side job (GemmArgs::rope_*): null source = none
  const bf16* rope_src;
  const float* rope_lut;
  bf16* rope_dst;
  int rope_T, rope_H, rope_q_head, rope_nope, rope_dims, rope_d_qk;
  const int* status_dev;  // GemmArgs::status_dev / status_host
  int* status_host;
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 16 bytes from the same shared-memory offset of the cluster's CTA `rank`.
__device__ __forceinline__ float4 ld_peer_f32x4(uint32_t local_addr, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(remote)
               : "memory");
  return v;
}

// NT: token tile (MMA N).  W_KN: the weight operand is stored [K, N] (N contiguous) and is read
// as an MN-major UMMA operand; otherwise [N, K], K-major.
template <int NT, bool W_KN>
__global__ void __launch_bounds__(GEMM_THREADS, 2)
k_gemm_tc(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmA, GemmTcParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  constexpr int A_BYTES = NT * BK * 2;
  constexpr int STAGE_BYTES = W_BYTES + A_BYTES;
  constexpr uint32_t TMEM_COLS = NT < 32 ? 32 : NT;
  constexpr int RED_BYTES = NT * W_TILE * 4;  // fp32 partial tile, parked over the ring
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int ring = p.stages * STAGE_BYTES;
  unsigned char* misc = smem + ((p.splits == 1 || ring > RED_BYTES) ? ring : RED_BYTES);
  uint64_t* full = reinterpret_cast<uint64_t*>(misc);
  uint64_t* empty = full + 8;
  uint64_t* acc_bar = empty + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * W_TILE;
  const int m_tile = blockIdx.y / p.splits, split = blockIdx.y % p.splits;
  const int m0 = m_tile * NT;
  // tokens that the MMAs and the reduction cover: with the largest tile, no padding beyond 16
  const int n_cols = NT == 256 ? min(NT, (p.M - m0 + 15) & ~15) : NT;
  const int z = blockIdx.z;
  const int kc0 = (int)((long long)p.kc_total * split / p.splits);
  const int kc1 = (int)((long long)p.kc_total * (split + 1) / p.splits);
  const int n_kc = kc1 - kc0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(acc_bar, 1);
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  if (warp == 1) tc::tmem_alloc(tmem_slot, TMEM_COLS);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // (warp-uniform code, one elected lane issues: see the MMA issuer)
    if (lane == 0) {
      tc::tma_prefetch_desc(&tmW);
      tc::tma_prefetch_desc(&tmA);
    }
    auto load_w = [&](int i, int s) {
      unsigned char* st = smem + (size_t)s * STAGE_BYTES;
      const int k0 = (kc0 + i) * BK;
      tc::mbar_expect_tx(&full[s], STAGE_BYTES);
      if (W_KN) {
        // two boxes of [64 k rows x 64 n]: n is the innermost coordinate
        tc::tma_load_3d(st, &tmW, &full[s], n0, k0, z);
        tc::tma_load_3d(st + W_BYTES / 2, &tmW, &full[s], n0 + 64, k0, z);
      } else {
        tc::tma_load_3d(st, &tmW, &full[s], k0, p.w_swap ? z : n0, p.w_swap ? n0 : z);
      }
    };
    auto load_a = [&](int i, int s) {
      tc::tma_load_3d(smem + (size_t)s * STAGE_BYTES + W_BYTES, &tmA, &full[s], (kc0 + i) * BK, p.a_swap ? z : m0,
                      p.a_swap ? m0 : z);
    };
    // Weights are written by no kernel: the first ring of weight tiles is requested while the
    // previous kernel still runs; the activations are its output and wait for it.
    const int first = min(n_kc, p.stages);
    for (int i = 0; i < first; ++i)
      if (tc::elect_one()) load_w(i, i);
    __syncwarp();
    pdl_launch();
    pdl_wait();
    for (int i = 0; i < first; ++i)
      if (tc::elect_one()) load_a(i, i);
    __syncwarp();
    int s = 0;
    uint32_t parity = 0;
    for (int i = first; i < n_kc; ++i) {
      if (!__all_sync(0xffffffffu, tc::mbar_wait(&empty[s], parity, abort_flag, p.d_status, ST_TMA_TIMEOUT))) break;
      if (tc::elect_one()) {
        load_w(i, s);
        load_a(i, s);
      }
      __syncwarp();
      if (++s == p.stages) {
        s = 0;
        parity ^= 1;
      }
    }
  } else if (warp == 1) {
    pdl_wait();
    // The whole warp walks the loop and one elected lane issues: with warp-uniform control flow the
    // descriptors stay in uniform registers (an MMA every 30 cycles; from a lane-0 branch every 65).
    // The next stage's barrier is asked before this stage's MMAs are issued, so that its answer
    // (about 200 cycles) is there when they are: 680 -> 300 cycles per stage, which with few tokens
    // was more than the stage's bytes need.
    uint32_t idesc = tc::umma_idesc_bf16(W_TILE, NT, W_KN ? 1 : 0, 0);
    if (NT == 256) idesc = tc::umma_idesc_bf16(W_TILE, 16, W_KN ? 1 : 0, 0) + ((uint32_t)((n_cols - 16) >> 3) << 17);
    // descriptors differ only in the start-address field: keep the rest in registers
    const uint64_t w_tmpl = W_KN ? tc::umma_desc_sw128(0, W_BYTES / 2, 1024) : tc::umma_desc_sw128(0, 16, 1024);
    const uint64_t a_tmpl = tc::umma_desc_sw128(0, 16, 1024);
    // 14-bit start-address field: inside a cluster the shared-window address of a CTA carries
    // its rank in high bits, which must not leak into the neighbouring descriptor fields
    const uint32_t base16 = (tc::smem_u32(smem) & 0x3FFFFu) >> 4;
    bool ok = true;
    int s = 0;
    uint32_t parity = 0;
    bool ready = n_kc > 0 && tc::mbar_try_wait(&full[0], 0);
    for (int i = 0; i < n_kc; ++i) {
      if (!__all_sync(0xffffffffu, ready))
        ok = __all_sync(0xffffffffu, tc::mbar_wait(&full[s], parity, abort_flag, p.d_status, ST_MMA_TIMEOUT));
      if (!ok) break;
      const uint32_t w16 = base16 + s * (STAGE_BYTES >> 4), a16 = w16 + (W_BYTES >> 4);
      uint64_t* done = &empty[s];
      if (++s == p.stages) {
        s = 0;
        parity ^= 1;
      }
      ready = i + 1 < n_kc && tc::mbar_test_wait(&full[s], parity);
      if (tc::elect_one()) {
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {
          // K-major: 16 k = 32 bytes along the row; MN-major: 16 k rows of 128 bytes
          const uint64_t da = w_tmpl | (uint64_t)(w16 + (W_KN ? k * 128 : k * 2));
          const uint64_t db = a_tmpl | (uint64_t)(a16 + k * 2);
          tc::umma_bf16(tmem, da, db, idesc, (i > 0 || k > 0) ? 1u : 0u);
        }
        tc::umma_commit(done);  // the stage is free once these MMAs have read it
        if (i + 1 == n_kc) tc::umma_commit(acc_bar);
      }
      __syncwarp();
    }
  } else {
    // epilogue warps: TMEM lane quadrant = warp % 4; thread = one weight row n
    pdl_wait();
    // side job while the accumulator is being built: RoPE of head z's rope pairs.  Few tokens: the
    // head's first block takes them all (spreading them bought nothing at 64 tokens); many tokens
    // (verify blocks, prefill): every block of the head takes a slice, or the one block's 16 rounds
    // of dependent loads outlast the whole GEMM.
    const int rope_blocks = p.rope_T > 128 ? (int)(gridDim.x * gridDim.y) : 1;
    const int rope_id = (int)(blockIdx.y * gridDim.x + blockIdx.x);
    if (p.rope_src && rope_id < rope_blocks) {
      const int half = p.rope_dims / 2, et = threadIdx.x - 64;  // 128 epilogue threads
      const int t_lo = (int)((long long)p.rope_T * rope_id / rope_blocks), t_hi = (int)((long long)p.rope_T * (rope_id + 1) / rope_blocks);
      const int n_items = t_hi * half;
      for (int i0 = t_lo * half + et; i0 < n_items; i0 += 8 * (GEMM_THREADS - 64)) {
        // eight items per thread and round, all loads before the first store
        __nv_bfloat162 x[8];
        float2 cs[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int i = i0 + u * (GEMM_THREADS - 64);
          if (i < n_items) {
            const int t = i / half, pr = i % half;
            x[u] = *reinterpret_cast<const __nv_bfloat162*>(p.rope_src + ((long long)t * p.rope_H + z) * p.rope_q_head + p.rope_nope + 2 * pr);
            cs[u] = *reinterpret_cast<const float2*>(p.rope_lut + (long long)t * p.rope_dims + 2 * pr);
          }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int i = i0 + u * (GEMM_THREADS - 64);
          if (i < n_items) {
            const int t = i / half, pr = i % half;
            const float x0 = __low2float(x[u]), x1 = __high2float(x[u]);
            *reinterpret_cast<__nv_bfloat162*>(p.rope_dst + ((long long)t * p.rope_H + z) * p.rope_d_qk + p.rope_d_qk - p.rope_dims + 2 * pr) =
                __floats2bfloat162_rn(x0 * cs[u].x - x1 * cs[u].y, x0 * cs[u].y + x1 * cs[u].x);
          }
        }
      }
    }
    const int quad = warp & 3;
    bool ok = n_kc == 0 || tc::mbar_wait(acc_bar, 0, abort_flag, p.d_status, ST_EPI_TIMEOUT);
    ok = __all_sync(0xffffffffu, ok);  // the TMEM loads below are warp-collective
    tc::tc_fence_after();
    const int row = quad * 32 + lane;
    const int n = n0 + row;
    // whether this block's output rows can go out as 8-byte stores (four weight rows per store)
    const bool wide_out = p.splits == 1 && (p.ldc % 4) == 0 && (p.c_bs % 4) == 0 && (n0 % 4) == 0 && n0 + W_TILE <= p.N &&
                          (reinterpret_cast<uintptr_t>(p.C) & 7) == 0;
    if (wide_out) {
      // the four epilogue warps take the staged path together or not at all (a wait that one of
      // them gave up must not leave the others at the barriers below)
      uint32_t all_ok;
      asm volatile(
          "{\n\t.reg .pred q, r;\n\t"
          "setp.ne.u32 q, %1, 0;\n\t"
          "bar.red.and.pred r, 1, 128, q;\n\t"
          "selp.u32 %0, 1, 0, r;\n\t}"
          : "=r"(all_ok)
          : "r"((uint32_t)ok)
          : "memory");
      ok = all_ok != 0;
    }
    if (ok && wide_out) {
      // No K split: the tile leaves through shared memory (the ring is idle once acc_bar fired), 32
      // tokens at a time, so that a warp writes 256 contiguous bytes of one token's row instead of
      // every thread two bytes per token.
      float* red = reinterpret_cast<float*>(smem);  // [32][128]
      const int e = threadIdx.x - 64;
      for (int c0 = 0; c0 < NT; c0 += 32) {
        if (m0 + c0 >= p.M) break;
        float v[32];
        if (n_kc > 0) {
          tc::tmem_ld32(tmem + ((uint32_t)(quad * 32) << 16) + c0, v);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0.0f;
        }
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (j < NT - c0) red[j * W_TILE + row] = v[j];
        asm volatile("bar.sync 1, 128;" ::: "memory");
        const int n_tok = min(min(32, NT - c0), p.M - m0 - c0);
        for (int idx = e; idx < n_tok * (W_TILE / 4); idx += GEMM_THREADS - 64) {
          const int tok = idx / (W_TILE / 4), r4 = (idx % (W_TILE / 4)) * 4;
          const float4 f = *reinterpret_cast<const float4*>(red + tok * W_TILE + r4);
          const __nv_bfloat162 lo = __floats2bfloat162_rn(f.x, f.y), hi = __floats2bfloat162_rn(f.z, f.w);
          *reinterpret_cast<uint2*>(p.C + z * p.c_bs + (long long)(m0 + c0 + tok) * p.ldc + n0 + r4) =
              make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
      }
    } else if (ok) {
      float* red = reinterpret_cast<float*>(smem);  // [NT][128]: the ring is idle once acc_bar fired
      for (int c0 = 0; c0 < NT; c0 += 32) {
        if (p.splits == 1 ? m0 + c0 >= p.M : c0 >= n_cols) break;
        float v[32];
        if (n_kc > 0) {
          tc::tmem_ld32(tmem + ((uint32_t)(quad * 32) << 16) + c0, v);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0.0f;
        }
        if (p.splits == 1) {
          if (n < p.N) {
            bf16* c = p.C + z * p.c_bs + n;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j < NT - c0 && m0 + c0 + j < p.M) c[(long long)(m0 + c0 + j) * p.ldc] = f2bf(v[j]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (j < NT - c0) red[(c0 + j) * W_TILE + row] = v[j];
        }
      }
    }
  }

  __syncwarp();  // the single-lane roles rejoin their warps before the aligned barriers below
  if (p.splits > 1) {
    // every K slice has parked its partial: reduce one column slice of the tile over the
    // cluster, peers in rank order
    cluster_sync_all();
    const uint32_t rank = cluster_ctarank();
    const int c_lo = (int)(n_cols * rank / p.splits), c_hi = (int)(n_cols * (rank + 1) / p.splits);
    const uint32_t red_addr = tc::smem_u32(smem);
    for (int e4 = c_lo * (W_TILE / 4) + threadIdx.x; e4 < c_hi * (W_TILE / 4); e4 += GEMM_THREADS) {
      const int col = e4 / (W_TILE / 4), row = (e4 % (W_TILE / 4)) * 4;
      float4 v[MAX_SPLITS];
#pragma unroll
      for (int s = 0; s < MAX_SPLITS; ++s)  // all loads in flight before the first add
        v[s] = s < p.splits ? ld_peer_f32x4(red_addr + (uint32_t)e4 * 16, (uint32_t)s) : make_float4(0.f, 0.f, 0.f, 0.f);
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < MAX_SPLITS; ++s) {
        acc[0] += v[s].x;
        acc[1] += v[s].y;
        acc[2] += v[s].z;
        acc[3] += v[s].w;
      }
      if (m0 + col < p.M) {
        bf16* c = p.C + z * p.c_bs + (long long)(m0 + col) * p.ldc + n0 + row;
        if (n0 + row + 3 < p.N && (reinterpret_cast<uintptr_t>(c) & 7) == 0) {
          // one 8-byte store (the output may be page-locked host memory: fewer, fuller writes)
          const __nv_bfloat162 lo = __floats2bfloat162_rn(acc[0], acc[1]), hi = __floats2bfloat162_rn(acc[2], acc[3]);
          *reinterpret_cast<uint2*>(c) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (n0 + row + j < p.N) c[j] = f2bf(acc[j]);
        }
      }
    }
    cluster_sync_all();  // nobody leaves while a peer still reads its shared memory
  }

  tc::tc_fence_before();
  __syncthreads();
  if (p.status_host && threadIdx.x == 0) {
    // (after this block's own waits: whatever it recorded itself is in the word it reads)
    const int st = *reinterpret_cast<const volatile int*>(p.status_dev);
    if (st != 0) *reinterpret_cast<volatile int*>(p.status_host) = st;
  }
  if (*abort_flag) {
    // a wait was given up: let copies and MMAs in flight settle before TMEM is released
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, TMEM_COLS);
  }
}

// Many tokens: a persistent kernel, one block (or pair of blocks) per SM (or pair).  A block walks output
// tiles (128 weight rows x up to 256 tokens, no K split); the accumulator is double-buffered in tensor
// memory and two groups of four epilogue warps take alternate tiles, so the operand ring and the tensor
// pipe run on while earlier tiles leave.  With a block per tile every tile paid its own start-up, first
// round trip and drain, 12-15 us a wave whatever its K.
//
// PAIR: two SMs share a tile of 256 weight rows (tcgen05 cta_group::2).  Each block fetches its own 128
// weight rows and HALF of the tokens, the MMAs read both halves, and each block's tensor memory gets its
// own rows of the product: 32 KB instead of 48 KB per block and K chunk.  What an SM can fetch, 55 bytes
// a clock, bounds the single-block form (891 cycles per chunk of 512 MMA cycles at K = 8192).  The leader
// (rank 0) issues; both blocks' copies report to the leader's barriers, its commits to the barriers of both.
constexpr int PG_THREADS = 320;          // warps: 0 copies, 1 issues MMAs, 2-5 and 6-9 the two epilogue groups
constexpr int PG_NT = 256;               // largest token tile
constexpr int PG_RING = 192 * 1024;      // operand ring
constexpr int PG_MAX_STAGES = 7;
constexpr int PG_OUT = 32 * W_TILE * 2;  // 32 tokens x 128 weight rows of bf16
constexpr int PG_SMEM = PG_RING + 4 * PG_OUT + 1024 /* alignment */ + 256 /* barriers */;

__device__ __forceinline__ uint32_t mapa_u32(const void* p, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(tc::smem_u32(p)), "r"(rank));
  return remote;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* dst, const CUtensorMap* m, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(tc::smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// One arrival at the barrier of this offset in both blocks of the pair.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(tc::smem_u32(bar)), "h"((uint16_t)3)
               : "memory");
}

template <bool W_KN, bool PAIR>
__global__ void __launch_bounds__(PG_THREADS, 1)
k_gemm_tc_tiles(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmA, GemmTcParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* s_out = smem + PG_RING;  // [group][2][32 tokens][128]
  uint64_t* full = reinterpret_cast<uint64_t*>(s_out + 4 * PG_OUT);
  uint64_t* empty = full + PG_MAX_STAGES;
  uint64_t* acc_full = empty + PG_MAX_STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int COLS = PAIR ? 2 * W_TILE : W_TILE;  // weight rows per tile
  const int rank = PAIR ? (int)cluster_ctarank() : 0;
  const int worker = PAIR ? blockIdx.x >> 1 : blockIdx.x, n_workers = PAIR ? gridDim.x >> 1 : gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      tc::mbar_init(&acc_full[a], 1);
      tc::mbar_init(&acc_empty[a], PAIR ? 8 : 4);  // one arrival per epilogue warp
    }
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  if (warp == 1) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(tmem_slot)), "r"(2 * PG_NT) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      tc::tmem_alloc(tmem_slot, 2 * PG_NT);
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();  // the peer's barriers exist
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int n_kc = p.kc_total, stage_bytes = W_BYTES + p.nt * BK * 2 / (PAIR ? 2 : 1);
  // tokens that the MMAs of a tile cover: a ragged last tile multiplies no padding
  auto tile_cols = [&](int m0) { return PAIR ? min(p.nt, (p.M - m0 + 31) & ~31) : min(p.nt, (p.M - m0 + 15) & ~15); };

  if (warp == 0) {
    if (lane == 0) {
      tc::tma_prefetch_desc(&tmW);
      tc::tma_prefetch_desc(&tmA);
    }
    const uint32_t full0 = PAIR ? mapa_u32(&full[0], 0) : 0;
    auto load = [&](void* dst, const CUtensorMap* map, int s, int x, int y, int z) {
      if (PAIR) tma_load_3d_pair(dst, map, full0 + s * 8, x, y, z);
      else tc::tma_load_3d(dst, map, &full[s], x, y, z);
    };
    auto load_w = [&](int tile, int kc, int s) {
      unsigned char* st = smem + s * stage_bytes;
      const int n0 = (tile % p.n_tiles) * COLS + rank * W_TILE, z = tile / p.n_tiles / p.m_tiles, k0 = kc * BK;
      if (rank == 0) tc::mbar_expect_tx(&full[s], PAIR ? 2 * stage_bytes : stage_bytes);
      if (W_KN) {
        load(st, &tmW, s, n0, k0, z);
        load(st + W_BYTES / 2, &tmW, s, n0 + 64, k0, z);
      } else {
        load(st, &tmW, s, k0, p.w_swap ? z : n0, p.w_swap ? n0 : z);
      }
    };
    auto load_a = [&](int tile, int kc, int s) {
      int m0 = tile / p.n_tiles % p.m_tiles * p.nt;
      const int z = tile / p.n_tiles / p.m_tiles;
      if (PAIR && rank) m0 += tile_cols(m0) / 2;
      load(smem + s * stage_bytes + W_BYTES, &tmA, s, kc * BK, p.a_swap ? z : m0, p.a_swap ? m0 : z);
    };
    // the first weight tiles before the wait for the kernel ahead (no kernel writes weights)
    const int first = min(n_kc, p.stages);
    for (int i = 0; i < first; ++i)
      if (tc::elect_one()) load_w(worker, i, i);
    __syncwarp();
    pdl_launch();
    pdl_wait();
    for (int i = 0; i < first; ++i)
      if (tc::elect_one()) load_a(worker, i, i);
    __syncwarp();
    int s = first % p.stages;
    uint32_t parity = first == p.stages ? 0 : 1;  // of the stage's last use; the first ring has none
    bool ok = true;
    for (int tile = worker, kc = first; tile < p.tiles && ok; tile += n_workers, kc = 0) {
      for (; kc < n_kc; ++kc) {
        // (parity 1 on a fresh barrier: passes at once)
        ok = __all_sync(0xffffffffu, tc::mbar_wait(&empty[s], parity, abort_flag, p.d_status, ST_TMA_TIMEOUT));
        if (!ok) break;
        if (tc::elect_one()) {
          load_w(tile, kc, s);
          load_a(tile, kc, s);
        }
        __syncwarp();
        if (++s == p.stages) {
          s = 0;
          parity ^= 1;
        }
      }
    }
  } else if (warp == 1 && rank == 0) {
    pdl_wait();  // (the limit of the waits below is for this kernel's own time, not for what is left of the one in front)
    // (warp-uniform walk, one elected lane issues, the next stage's barrier asked ahead: as in k_gemm_tc)
    const uint64_t w_tmpl = W_KN ? tc::umma_desc_sw128(0, W_BYTES / 2, 1024) : tc::umma_desc_sw128(0, 16, 1024);
    const uint64_t a_tmpl = tc::umma_desc_sw128(0, 16, 1024);
    const uint32_t base16 = (tc::smem_u32(smem) & 0x3FFFFu) >> 4;
    int s = 0, i = 0;
    uint32_t parity = 0;
    bool ok = true, ready = tc::mbar_try_wait(&full[0], 0);
    for (int tile = worker; tile < p.tiles && ok; tile += n_workers, ++i) {
      const int m0 = tile / p.n_tiles % p.m_tiles * p.nt;
      const uint32_t idesc = tc::umma_idesc_bf16(COLS, 16, W_KN ? 1 : 0, 0) + ((uint32_t)((tile_cols(m0) - 16) >> 3) << 17);
      const uint32_t d = tmem + (i & 1) * PG_NT;
      if (i >= 2) {
        ok = __all_sync(0xffffffffu, tc::mbar_wait(&acc_empty[i & 1], ((i >> 1) - 1) & 1, abort_flag, p.d_status, ST_MMA_TIMEOUT));
        if (!ok) break;
      }
      tc::tc_fence_after();
      for (int kc = 0; kc < n_kc; ++kc) {
        if (!__all_sync(0xffffffffu, ready))
          ok = __all_sync(0xffffffffu, tc::mbar_wait(&full[s], parity, abort_flag, p.d_status, ST_MMA_TIMEOUT));
        if (!ok) break;
        const uint32_t w16 = base16 + s * (stage_bytes >> 4), a16 = w16 + (W_BYTES >> 4);
        uint64_t* done = &empty[s];
        if (++s == p.stages) {
          s = 0;
          parity ^= 1;
        }
        ready = tc::mbar_test_wait(&full[s], parity);
        if (tc::elect_one()) {
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t dw = w_tmpl | (uint64_t)(w16 + (W_KN ? k * 128 : k * 2));
            const uint64_t da = a_tmpl | (uint64_t)(a16 + k * 2);
            if (PAIR) umma_bf16_pair(d, dw, da, idesc, (kc > 0 || k > 0) ? 1u : 0u);
            else tc::umma_bf16(d, dw, da, idesc, (kc > 0 || k > 0) ? 1u : 0u);
          }
          if (PAIR) umma_commit_pair(done);
          else tc::umma_commit(done);
          if (kc + 1 == n_kc) {
            if (PAIR) umma_commit_pair(&acc_full[i & 1]);
            else tc::umma_commit(&acc_full[i & 1]);
          }
        }
        __syncwarp();
      }
    }
  } else if (warp >= 2) {
    pdl_wait();
    const uint32_t acc_empty0 = PAIR ? mapa_u32(&acc_empty[0], 0) : 0;
    const int group = (warp - 2) >> 2, quad = warp & 3, et = (threadIdx.x - 64) & 127;
    if (p.rope_src) {
      // RoPE of the query's rope dims, four pairs (16 bytes) per item, spread over all blocks (32-bit index
      // arithmetic: the divisions are most of an item's instructions)
      const uint32_t per_row = p.rope_dims / 8;
      const uint32_t n_items = p.rope_T * p.rope_H * per_row, step = gridDim.x * 256;
      for (uint32_t i0 = blockIdx.x * 256 + (threadIdx.x - 64); i0 < n_items; i0 += 4 * step) {
        uint4 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t i = i0 + u * step, row = i / per_row;
          if (i < n_items)
            x[u] = *reinterpret_cast<const uint4*>(p.rope_src + (long long)row * p.rope_q_head + p.rope_nope + (i - row * per_row) * 8);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t i = i0 + u * step, row = i / per_row;
          if (i < n_items) {
            const uint32_t v = i - row * per_row;
            const float* lut = p.rope_lut + (long long)(row / (uint32_t)p.rope_H) * p.rope_dims + v * 8;
            uint32_t w[4] = {x[u].x, x[u].y, x[u].z, x[u].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&w[e]);
              const float x0 = __low2float(b), x1 = __high2float(b), c = lut[2 * e], sn = lut[2 * e + 1];
              const __nv_bfloat162 r = __floats2bfloat162_rn(x0 * c - x1 * sn, x0 * sn + x1 * c);
              w[e] = *reinterpret_cast<const uint32_t*>(&r);
            }
            *reinterpret_cast<uint4*>(p.rope_dst + (long long)row * p.rope_d_qk + p.rope_d_qk - p.rope_dims + v * 8) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
    }
    unsigned char* out = s_out + group * 2 * PG_OUT;
    const int row = quad * 32 + lane;
    int buf = 0;
    for (int tile = worker + group * n_workers, use = 0; tile < p.tiles; tile += 2 * n_workers, ++use) {
      const int n0 = (tile % p.n_tiles) * COLS + rank * W_TILE, m0 = tile / p.n_tiles % p.m_tiles * p.nt, z = tile / p.n_tiles / p.m_tiles;
      const bool ok = tc::mbar_wait(&acc_full[group], use & 1, abort_flag, p.d_status, ST_EPI_TIMEOUT);
      // the four warps of a group go on together or not at all
      uint32_t all_ok;
      asm volatile(
          "{\n\t.reg .pred q, r;\n\t"
          "setp.ne.u32 q, %1, 0;\n\t"
          "bar.red.and.pred r, %2, 128, q;\n\t"
          "selp.u32 %0, 1, 0, r;\n\t}"
          : "=r"(all_ok)
          : "r"((uint32_t)ok), "r"(1 + group)
          : "memory");
      if (!all_ok) break;
      tc::tc_fence_after();
      const int n_tok = min(p.nt, p.M - m0);
      bf16* c = p.C + z * p.c_bs + (long long)m0 * p.ldc + n0;
      for (int c0 = 0; c0 < n_tok; c0 += 32) {
        float v[32];
        tc::tmem_ld32(tmem + group * PG_NT + ((uint32_t)(quad * 32) << 16) + c0, v);
        if (c0 + 32 >= n_tok) {  // the accumulator has been read
          tc::tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if (PAIR) mbar_arrive_cluster(acc_empty0 + group * 8);
            else tc::mbar_arrive(&acc_empty[group]);
          }
        }
        bf16* so = reinterpret_cast<bf16*>(out + buf * PG_OUT) + row;
#pragma unroll
        for (int j = 0; j < 32; ++j) so[j * W_TILE] = f2bf(v[j]);
        asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
        // 16 threads per token row of 256 bytes; the next slice is staged in the other buffer, and this one
        // is written again only behind the next barrier
        const int r8 = (et & 15) * 8;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int tok = (et >> 4) + 8 * q;
          if (c0 + tok < n_tok && n0 + r8 < p.N)
            *reinterpret_cast<uint4*>(c + (long long)(c0 + tok) * p.ldc + r8) =
                *reinterpret_cast<const uint4*>(out + buf * PG_OUT + tok * (W_TILE * 2) + r8 * 2);
        }
        buf ^= 1;
      }
    }
  }

  __syncwarp();
  tc::tc_fence_before();
  __syncthreads();
  if (p.status_host && threadIdx.x == 0) {
    const int st = *reinterpret_cast<const volatile int*>(p.status_dev);
    if (st != 0) *reinterpret_cast<volatile int*>(p.status_host) = st;
  }
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);  // let copies and MMAs in flight settle
  }
  if (PAIR) {
    __syncwarp();
    cluster_sync_all();  // nobody leaves while the peer may still signal its barriers
  }
  if (warp == 1) {
    tc::tc_fence_after();
    if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * PG_NT) : "memory");
    else tc::tmem_dealloc(tmem, 2 * PG_NT);
  }
}

int pick_nt(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : M <= 128 ? 128 : 256; }

template <int NT, bool W_KN>
cudaError_t launch_one(const CUtensorMap& tmW, const CUtensorMap& tmA, const GemmTcParams& p, dim3 grid, size_t smem,
                       cudaStream_t st) {
  return launch_pdl(k_gemm_tc<NT, W_KN>, grid, dim3(GEMM_THREADS, 1, 1), smem, st, p.splits, tmW, tmA, p);
}

}  // namespace

bool gemm_tc_supported(const GemmArgs& g) {
  if (g.M <= 0 || g.N <= 0 || g.K <= 0) return false;
  if (g.K % 8 || g.lda % 8 || g.ldb % 8 || g.a_bs % 8 || g.b_bs % 8) return false;
  if ((reinterpret_cast<uintptr_t>(g.A) & 15) || (reinterpret_cast<uintptr_t>(g.B) & 15)) return false;
  if (g.b_kn && g.N % 8) return false;
  return true;
}

cudaError_t launch_gemm_tc(const GemmArgs& g, int* d_status, cudaStream_t st) {
  int dev = 0, n_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  static int sm_count[64] = {0};
  if (!sm_count[dev & 63]) cudaDeviceGetAttribute(&sm_count[dev & 63], cudaDevAttrMultiProcessorCount, dev);
  n_sm = sm_count[dev & 63];
  int NT = pick_nt(g.M);
  const int n_tiles = (g.N + W_TILE - 1) / W_TILE;
  const int m_tiles = (g.M + NT - 1) / NT;
  const int kc_total = (g.K + BK - 1) / BK;
  // K slices (a power of two, one cluster) while two CTAs per SM are not yet covered, keeping
  // at least two K chunks per CTA
  const long long tiles = (long long)n_tiles * m_tiles * g.batch;
  int splits = 1;
  // -- or, with more than 128 tokens, while there is one per SM: a block then streams its K slice of 128
  // weight rows and of all its tokens (up to 256).  Two tiles of 128 tokens fetched every weight row twice:
  // 192 tokens, 4096 x 4096 27.1 -> 24.6 us; 512 tokens, 4096 x 8192 45.8 -> 40.2.
  const long long room = NT == 256 ? n_sm : 2ll * n_sm;
  while (splits < MAX_SPLITS && tiles * splits * 2 <= room && kc_total / (splits * 2) >= 2) splits *= 2;
  // Output tiles that cover half of the SMs or more are not split at all: a block per SM with a ring
  // of eight stages and no cluster reduction beats two half-size blocks on a third of the SMs
  // (the q-expand GEMM, 96 tiles: 18.2 -> 16.5 us; cut in three or four it was slower still).
  // With a handful of tokens the split wins (one token: 14.5 against 16.3 us).
  if (NT >= 64 && NT < 256 && tiles * 2 >= n_sm && tiles <= n_sm) splits = 1;

  // Enough tokens and output tiles to give every SM one without a K split: the persistent kernel, with
  // the token tile (a multiple of 32) whose rounds of tiles fetch least: a tile's operands are its 128
  // weight rows and its tokens.  It stores 16 bytes at a time and rotates 16 bytes at a time.
  const bool persistent = g.M > 128 && splits == 1 && g.N % 8 == 0 && g.ldc % 8 == 0 && g.c_bs % 8 == 0 &&
                          (reinterpret_cast<uintptr_t>(g.C) & 15) == 0 &&
                          (!g.rope_src || (g.rope_q_head % 8 == 0 && g.rope_nope % 8 == 0 && g.rope_dims % 8 == 0 && g.rope_d_qk % 8 == 0 &&
                                           (long long)g.rope_T * g.rope_H * g.rope_dims < (1ll << 31) &&
                                           (reinterpret_cast<uintptr_t>(g.rope_src) & 15) == 0 && (reinterpret_cast<uintptr_t>(g.rope_dst) & 15) == 0));
  // Pairs of blocks fetch less per MMA; a product of one weight tile (the value projection of a head)
  // would leave the second block of every pair idle, and an odd tile number half of the last one.
  const bool pair = persistent && (n_tiles % 2 == 0 || n_tiles >= 8);
  const int cols = pair ? (n_tiles + 1) / 2 : n_tiles, workers = pair ? n_sm / 2 : n_sm;
  if (persistent) {
    long long best = 0;
    for (int nt = PG_NT; nt >= 128; nt -= 32) {
      const long long rounds = ((long long)cols * ((g.M + nt - 1) / nt) * g.batch + workers - 1) / workers;
      const int fetch = W_TILE + (pair ? nt / 2 : nt);
      if (best == 0 || rounds * fetch < best) {
        best = rounds * fetch;
        NT = nt;
      }
    }
  }

  CUtensorMap tmW, tmA;
  const char* err = nullptr;
  // dimension order {K, rows, batch}, or {K, batch, rows} when the batch stride is the smaller
  // one, so that the byte strides of the map ascend
  auto build = [&](CUtensorMap* out, const bf16* base, int rows, int ld, long long bs, int box_rows, int* swap) {
    const uint64_t row_b = (uint64_t)ld * 2;
    const uint64_t bat_b = g.batch > 1 ? (uint64_t)bs * 2 : row_b * (uint64_t)rows;
    *swap = g.batch > 1 && bat_b < row_b;
    if (*swap)
      return tc::cached_tmap(out, base, g.K, g.batch, rows, bat_b, row_b, BK, 1, box_rows, &err);
    return tc::cached_tmap(out, base, g.K, rows, g.batch, row_b, std::max<uint64_t>(bat_b, 16), BK, box_rows, 1, &err);
  };
  int w_swap = 0, a_swap = 0;
  bool ok;
  if (g.b_kn) {
    // W is [K, N]: dims {N, K, batch}, boxes of 64 n x 64 k
    const uint64_t row_b = (uint64_t)g.ldb * 2;
    const uint64_t bat_b = g.batch > 1 ? (uint64_t)g.b_bs * 2 : row_b * (uint64_t)g.K;
    ok = tc::cached_tmap(&tmW, g.B, g.N, g.K, g.batch, row_b, std::max<uint64_t>(bat_b, 16), 64, BK, 1, &err);
  } else {
    ok = build(&tmW, g.B, g.N, g.ldb, g.b_bs, W_TILE, &w_swap);
  }
  if (!ok || !build(&tmA, g.A, g.M, g.lda, g.a_bs, pair ? NT / 2 : NT, &a_swap)) return cudaErrorInvalidValue;

  GemmTcParams p;
  p.C = g.C; p.d_status = d_status;
  p.M = g.M; p.N = g.N; p.K = g.K; p.ldc = g.ldc; p.c_bs = g.c_bs;
  p.splits = splits; p.kc_total = kc_total; p.w_swap = w_swap; p.a_swap = a_swap;
  p.rope_src = g.rope_src; p.rope_lut = g.rope_lut; p.rope_dst = g.rope_dst;
  p.rope_T = g.rope_T; p.rope_H = g.rope_H; p.rope_q_head = g.rope_q_head; p.rope_nope = g.rope_nope;
  p.rope_dims = g.rope_dims; p.rope_d_qk = g.rope_d_qk;
  p.status_dev = g.status_host ? g.status_dev : nullptr; p.status_host = g.status_dev ? g.status_host : nullptr;
  if (persistent) {
    p.nt = NT; p.n_tiles = cols; p.m_tiles = (g.M + NT - 1) / NT;
    p.tiles = cols * p.m_tiles * g.batch;
    p.stages = std::min(PG_MAX_STAGES, PG_RING / (W_BYTES + NT * BK * 2 / (pair ? 2 : 1)));
    const dim3 grid(std::min(p.tiles, workers) * (pair ? 2 : 1)), block(PG_THREADS);
    if (pair)
      return g.b_kn ? launch_pdl(k_gemm_tc_tiles<true, true>, grid, block, PG_SMEM, st, 2, tmW, tmA, p)
                    : launch_pdl(k_gemm_tc_tiles<false, true>, grid, block, PG_SMEM, st, 2, tmW, tmA, p);
    return g.b_kn ? launch_pdl(k_gemm_tc_tiles<true, false>, grid, block, PG_SMEM, st, 1, tmW, tmA, p)
                  : launch_pdl(k_gemm_tc_tiles<false, false>, grid, block, PG_SMEM, st, 1, tmW, tmA, p);
  }
  const int stage_bytes = W_BYTES + NT * BK * 2;
  // Two blocks share an SM (96 KB of operand ring each) -- unless the grid has no more blocks than
  // there are SMs: then a block has the SM to itself anyway and takes a ring that holds its whole K
  // slice, so that every operand tile is requested at once instead of in two or three turns.
  const bool alone = tiles * splits <= n_sm;
  const int per_block = (kc_total + splits - 1) / splits;
  p.stages = std::max(2, std::min(std::min(8, alone ? per_block : 8), ((alone ? 192 : 96) * 1024) / stage_bytes));
  const size_t ring = (size_t)p.stages * stage_bytes, red = splits > 1 ? (size_t)NT * W_TILE * 4 : 0;
  const size_t smem = std::max(ring, red) + 1024 /* alignment */ + 256 /* barriers */;
  dim3 grid(n_tiles, m_tiles * splits, g.batch);

#define FST_GEMM_CASE(NTV)                                                                   \
  case NTV:                                                                                  \
    e = g.b_kn ? launch_one<NTV, true>(tmW, tmA, p, grid, smem, st)                          \
               : launch_one<NTV, false>(tmW, tmA, p, grid, smem, st);                        \
    break
  switch (NT) {
    FST_GEMM_CASE(16);
    FST_GEMM_CASE(32);
    FST_GEMM_CASE(64);
    FST_GEMM_CASE(128);
    default:
      e = g.b_kn ? launch_one<256, true>(tmW, tmA, p, grid, smem, st) : launch_one<256, false>(tmW, tmA, p, grid, smem, st);
      break;
  }
#undef FST_GEMM_CASE
  return e;
}

// ---- host: tensor map encoding through the driver entry point (no link-time libcuda) ----------
namespace tc {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

bool make_tmap_bf16(CUtensorMap* out, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                    const uint32_t* box, const char** err) {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || !p) {
      if (err) *err = "cuTensorMapEncodeTiled is not available";
      return false;
    }
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  cuuint64_t gd[5];
  cuuint64_t gs[5];
  cuuint32_t bx[5], es[5];
  for (int i = 0; i < rank; ++i) {
    gd[i] = dims[i];
    bx[i] = box[i];
    es[i] = 1;
    if (i > 0) gs[i - 1] = strides_bytes[i - 1];
  }
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), gd, gs, bx, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    if (err) *err = "cuTensorMapEncodeTiled failed";
    return false;
  }
  return true;
}

namespace {

struct TmapKey {
  const void* base;
  uint64_t d0, d1, d2, s1, s2;
  uint32_t b0, b1, b2;
  bool operator==(const TmapKey& o) const {
    return base == o.base && d0 == o.d0 && d1 == o.d1 && d2 == o.d2 && s1 == o.s1 && s2 == o.s2 && b0 == o.b0 &&
           b1 == o.b1 && b2 == o.b2;
  }
};
struct TmapHash {
  size_t operator()(const TmapKey& k) const {
    size_t h = reinterpret_cast<size_t>(k.base);
    for (uint64_t v : {k.d0, k.d1, k.d2, k.s1, k.s2, (uint64_t)k.b0, (uint64_t)k.b1, (uint64_t)k.b2}) h = h * 1000003u ^ (size_t)v;
    return h;
  }
};

std::mutex g_mu;
std::unordered_map<TmapKey, CUtensorMap, TmapHash> g_tmaps;

}  // namespace

bool cached_tmap(CUtensorMap* out, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t s1,
                 uint64_t s2, uint32_t b0, uint32_t b1, uint32_t b2, const char** err) {
  TmapKey key{base, d0, d1, d2, s1, s2, b0, b1, b2};
  std::lock_guard<std::mutex> lk(g_mu);
  auto it = g_tmaps.find(key);
  if (it != g_tmaps.end()) {
    *out = it->second;
    return true;
  }
  const uint64_t dims[3] = {d0, d1, d2};
  const uint64_t strides[2] = {s1, s2};
  const uint32_t box[3] = {b0, b1, b2};
  if (!make_tmap_bf16(out, base, 3, dims, strides, box, err)) return false;
  if (g_tmaps.size() > 4096) g_tmaps.clear();
  g_tmaps.emplace(key, *out);
  return true;
}

}  // namespace tc
}  // namespace fst
