// bf16 GEMM on CTA pairs (tcgen05 cta_group::2): one 256 x 256 output tile per pair of SMs.
//
// Each CTA of a pair loads 128 rows of A and half of B's 256 columns and holds 128 rows of the accumulator; the tensor
// cores of both SMs read B's halves from both shared memories, so that a 64-deep step costs an SM 32 KB of loads for
// the work that takes 48 KB in a CTA by itself.  Under a sustained load the part is limited by power, and moving less
// is what makes it faster: 8192 x 11264 x 2048 330 -> 301 us, 2999 x 4096 x 14336 337 -> 290 us, 4096 x 50304 x 2048
// 758 -> 663 us, a weight gradient of 5632 x 2048 over 8192 tokens 193 -> 167 us (each against one CTA a tile, in turn).
//
// Roles as in gemm.cu, per CTA: warp 0 TMA producer, warp 1 MMA issuer (of the leader, the even CTA), warps 2-5
// epilogue.  Barriers across the pair:
//   full   in the leader: one arrival (its producer's, which expects both CTAs' bytes) and the bytes of both CTAs' loads
//   empty  in each CTA  : the leader's commit arrives at both
//   tfull  in each CTA  : the leader's commit arrives at both
//   tempty in the leader: the epilogue warps of both CTAs
// No multicast loads.  Every wait is bounded; both CTAs meet at a cluster barrier before they exit.
#pragma once
#include "b200.cuh"
#include "host_util.cuh"

namespace b200pair {

using namespace b200;

constexpr int BM = 128;          // rows of A and of the output per CTA
constexpr int PAIR_M = 256, PAIR_N = 256;
constexpr int BK = 64;
constexpr int STAGES = 6;
constexpr int TILE_BYTES = BM * BK * 2;              // A and B tile of one CTA
constexpr int STAGE_BYTES = 2 * TILE_BYTES;
constexpr int EPI_WARPS = 4;
constexpr int STAGING_BYTES = 32 * 128;
constexpr int STAGING_OFF = STAGES * STAGE_BYTES;
constexpr int BAR_OFF = STAGING_OFF + EPI_WARPS * 2 * STAGING_BYTES;
constexpr int SMEM_BYTES = BAR_OFF + 256 + 1024;
constexpr int NUM_THREADS = 32 * (2 + EPI_WARPS);
constexpr int GROUP_M = 8;

struct PairParams {
  int M, N, K, batch;
  int accumulate;
  int* status;
  const int* k_range;   // as in gemm.cu
  int c_shared;         // as in gemm.cu
};

__device__ __forceinline__ uint32_t map_to_cta(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// this CTA's shared memory, completion on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_3d_pair(void* dst, const CUtensorMap* tm, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives at the barrier of this address in both CTAs once all MMAs issued so far have completed
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(smem_u32(bar)), "h"(static_cast<uint16_t>(3))
      : "memory");
}
__device__ __forceinline__ void arrive_remote(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// orders what this thread does next after arrivals from the other CTA that a wait has seen
__device__ __forceinline__ void fence_acquire_cluster() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }

template <bool A_MN, bool B_MN, bool OUT_F32>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmC, const PairParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + BAR_OFF);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const AbortCtx ab{abort_flag, p.status};

  const int warp = warp_uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int rank = blockIdx.x & 1;          // clusters are pairs of neighbouring blocks
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  const int tiles_m = (p.M + PAIR_M - 1) / PAIR_M;
  const int tiles_n = (p.N + PAIR_N - 1) / PAIR_N;
  const int per_batch = tiles_m * tiles_n;
  const int total_tiles = per_batch * p.batch;
  const int k_blocks = (p.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 2 * EPI_WARPS);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();       // both CTAs' barriers are initialised before anything arrives at them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  auto tile_coords = [&](int t, int& b, int& m0, int& n0) {
    b = t / per_batch;
    const int r = t - b * per_batch;
    const int group_size = GROUP_M * tiles_n;
    const int g = r / group_size;
    const int first_m = g * GROUP_M;
    const int gm = min(GROUP_M, tiles_m - first_m);
    const int in_group = r - g * group_size;
    m0 = (first_m + in_group % gm) * PAIR_M;
    n0 = (in_group / gm) * PAIR_N;
  };
  auto k_extent = [&](int b, int& kb0, int& kb1) -> bool {
    kb0 = 0;
    kb1 = k_blocks;
    if (p.k_range) {
      kb0 = p.k_range[2 * b] / BK;
      kb1 = (p.k_range[2 * b + 1] + BK - 1) / BK;
    }
    return kb1 > kb0;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      bool ok = true;
      int s = 0, ph = 1;
      for (int t = pair; t < total_tiles && ok; t += pairs) {
        int b, m0, n0, kb0, kb1;
        tile_coords(t, b, m0, n0);
        if (!k_extent(b, kb0, kb1)) continue;
        const int z = (p.k_range || p.c_shared) ? 0 : b;
        const int k_off = p.c_shared ? b * k_blocks : 0;
        const int am = m0 + rank * BM, bn = n0 + rank * BM;
        for (int kb = kb0 + k_off; kb < kb1 + k_off; ++kb) {
          if (!mbar_wait(&empty[s], ph, ab, ERR_WAIT_EMPTY)) { ok = false; break; }
          uint8_t* sA = smem + s * STAGE_BYTES;
          uint8_t* sB = sA + TILE_BYTES;
          const uint32_t bar = map_to_cta(&full[s], 0);
          if (rank == 0) mbar_expect_tx(&full[s], 2 * STAGE_BYTES);
          if (!A_MN) {
            tma_load_3d_pair(sA, &tmA, bar, kb * BK, am, z);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_3d_pair(sA + j * 8192, &tmA, bar, am + j * 64, kb * BK, z);
          }
          if (!B_MN) {
            tma_load_3d_pair(sB, &tmB, bar, kb * BK, bn, z);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_3d_pair(sB + j * 8192, &tmB, bar, bn + j * 64, kb * BK, z);
          }
          if (++s == STAGES) {
            s = 0;
            ph ^= 1;
          }
        }
      }
      if (!ok) {
        // give copies already in flight time to land before the CTA's shared memory goes away
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader only)
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(PAIR_M, PAIR_N, A_MN, B_MN);
      int s = 0, ph = 0;
      uint32_t tile_iter = 0;
      bool ok = true;
      for (int t = pair; t < total_tiles && ok; t += pairs) {
        int b, m0, n0, kb0, kb1;
        tile_coords(t, b, m0, n0);
        if (!k_extent(b, kb0, kb1)) continue;
        const uint32_t acc = tile_iter & 1;
        const uint32_t acc_ph = (tile_iter >> 1) & 1;
        ++tile_iter;
        if (!mbar_wait(&tempty[acc], acc_ph ^ 1, ab, ERR_WAIT_TMEM_EMPTY)) { ok = false; break; }
        fence_acquire_cluster();
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * PAIR_N;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&full[s], ph, ab, ERR_WAIT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_base = smem_u32(smem + s * STAGE_BYTES);
          const uint64_t adesc = make_smem_desc_sw128(a_base, A_MN ? 8192 : 16, 1024);
          const uint64_t bdesc = make_smem_desc_sw128(a_base + TILE_BYTES, B_MN ? 8192 : 16, 1024);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)   // the next 16 elements of K, in units of 16 bytes
            mma_pair(d_tmem, adesc + (A_MN ? k * 128 : k * 2), bdesc + (B_MN ? k * 128 : k * 2), idesc,
                     (kb != kb0 || k != 0) ? 1u : 0u);
          commit_pair(&empty[s]);
          if (++s == STAGES) {
            s = 0;
            ph ^= 1;
          }
        }
        if (ok) commit_pair(&tfull[acc]);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;  // TMEM lane quadrant this warp may access
    constexpr int COLS_PER_BOX = OUT_F32 ? 32 : 64;
    uint8_t* stage0 = smem + STAGING_OFF + (warp - 2) * 2 * STAGING_BYTES;
    const uint32_t tempty_leader[2] = {map_to_cta(&tempty[0], 0), map_to_cta(&tempty[1], 0)};
    uint32_t tile_iter = 0;
    uint32_t box_iter = 0;
    bool ok = true;
    for (int t = pair; t < total_tiles && ok; t += pairs) {
      int b, m0, n0, kb0, kb1;
      tile_coords(t, b, m0, n0);
      if (!k_extent(b, kb0, kb1)) continue;
      const uint32_t acc = tile_iter & 1;
      const uint32_t acc_ph = (tile_iter >> 1) & 1;
      ++tile_iter;
      if (!mbar_wait_warp(&tfull[acc], acc_ph, ab, ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const uint32_t t_row = tmem_base + acc * PAIR_N + (static_cast<uint32_t>(q * 32) << 16);
      const int row0 = m0 + rank * BM + q * 32;
#pragma unroll 1
      for (int j = 0; j < PAIR_N / COLS_PER_BOX; ++j) {
        const int col0 = n0 + j * COLS_PER_BOX;
        if (col0 >= p.N || row0 >= p.M) break;  // warp-uniform: nothing of this box is in range
        uint8_t* buf = stage0 + (box_iter & 1) * STAGING_BYTES;
        ++box_iter;
        if (lane == 0) tma_wait_group_read<1>();  // the store that last read this buffer is done
        __syncwarp();
        if (OUT_F32) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(t_row + j * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 8; ++c)
            *reinterpret_cast<uint4*>(buf + sw128_offset(lane, c)) = make_uint4(r[4 * c], r[4 * c + 1], r[4 * c + 2], r[4 * c + 3]);
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t r[32];
            tmem_ld_32x32b_x32(t_row + j * 64 + h * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              uint4 v;
              v.x = pack_bf16x2(__uint_as_float(r[8 * c + 0]), __uint_as_float(r[8 * c + 1]));
              v.y = pack_bf16x2(__uint_as_float(r[8 * c + 2]), __uint_as_float(r[8 * c + 3]));
              v.z = pack_bf16x2(__uint_as_float(r[8 * c + 4]), __uint_as_float(r[8 * c + 5]));
              v.w = pack_bf16x2(__uint_as_float(r[8 * c + 6]), __uint_as_float(r[8 * c + 7]));
              *reinterpret_cast<uint4*>(buf + sw128_offset(lane, h * 4 + c)) = v;
            }
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          const int zC = p.c_shared ? 0 : b;
          if (p.accumulate)
            tma_reduce_add_3d(&tmC, buf, col0, row0, zC);
          else
            tma_store_3d(&tmC, buf, col0, row0, zC);
          tma_commit_group();
        }
      }
      // every tcgen05.ld of this accumulator has completed: hand it back to the MMA issuer
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_remote(acc ? tempty_leader[1] : tempty_leader[0]);
    }
    if (lane == 0) tma_wait_group<0>();
  }

  // ------------------------------------------------------------------ teardown
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync();       // nothing of the other CTA arrives here, or reads this CTA's tiles, any more
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

template <bool A_MN, bool B_MN, bool OUT_F32>
int launch(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const PairParams& p, int pairs,
           cudaStream_t stream) {
  auto* kern = gemm_pair_kernel<A_MN, B_MN, OUT_F32>;
  static bool configured[b200host::kMaxDevices] = {};
  if (int rc = b200host::ensure_dynamic_smem(kern, SMEM_BYTES, configured)) return rc;
  kern<<<2 * pairs, NUM_THREADS, SMEM_BYTES, stream>>>(tmA, tmB, tmC, p);
  return static_cast<int>(cudaGetLastError());
}

inline int dispatch(bool a_mn, bool b_mn, bool out_f32, const CUtensorMap& tmA, const CUtensorMap& tmB,
                    const CUtensorMap& tmC, const PairParams& p, int pairs, cudaStream_t s) {
#define PAIR_CASE(A, B, F) \
  if (a_mn == A && b_mn == B && out_f32 == F) return launch<A, B, F>(tmA, tmB, tmC, p, pairs, s);
  PAIR_CASE(false, false, false)
  PAIR_CASE(false, false, true)
  PAIR_CASE(false, true, false)
  PAIR_CASE(false, true, true)
  PAIR_CASE(true, false, false)
  PAIR_CASE(true, false, true)
  PAIR_CASE(true, true, false)
  PAIR_CASE(true, true, true)
#undef PAIR_CASE
  return b200host::RC_BAD_SHAPE;
}

}  // namespace b200pair
