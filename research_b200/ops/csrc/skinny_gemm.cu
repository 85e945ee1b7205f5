// y = x W^T for a handful of rows (the linears of a decode step): x [rows <= 128, K], W [N, K], y [rows, N], bf16 with
// fp32 sums.  The time is that of streaming W once, so the weights are the 128-row operand of the tensor core and the
// tokens its columns (16, 32, 64 or 128, no padding to 128 rows), and K is cut over the CTAs of a cluster so that about
// two CTAs per SM stream at once:
//   warp 0     TMA producer: 128 x 64 tiles of W and the matching 64 columns of x through a ring
//              of 2 to 12 stages; launched as a programmatic dependent, it has its first W tiles brought into L2 before it
//              waits for the predecessor, and reads W and x after that
//   warp 1     MMA issuer: D[n][token] += W x^T in tensor memory
//   warps 2-5  move the partial D to shared memory, token by token
// The CTAs of a cluster then each sum 128 / cluster rows of D over all partials, read from one another's shared memory in
// rank order, and write bf16: no workspace, no finishing kernel, the same bits every time.  The four linears of a
// 2048-wide layer (wqkv, wo, w_gate_up, w_down) with 32 rows: 45 us as slices added into an fp32 workspace with
// reduce-adds and a kernel that converted it and cleared it, 32.4 us here; 28.3 us with one row.
#include "b200.cuh"
#include "host_util.cuh"

using namespace b200;

namespace {

constexpr int TILE_N = 128;   // weight rows per CTA
constexpr int BK = 64;
constexpr int W_BYTES = TILE_N * BK * 2;
constexpr int NUM_THREADS = 192;

constexpr int MAX_STAGES = 12;

template <int NT>
constexpr int stage_bytes() { return W_BYTES + NT * BK * 2; }

struct SkinnyParams {
  int rows, N, k_blocks, cluster, stages;
  long long ldo;
  __nv_bfloat16* out;
  int* status;
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t saddr, uint32_t rank) {
  uint32_t peer;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(saddr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(peer)
               : "memory");
  return v;
}

template <int NT>
__global__ void __launch_bounds__(NUM_THREADS)
skinny_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                   const SkinnyParams p) {
  constexpr int STAGE_BYTES = stage_bytes<NT>();
  constexpr int TMEM_COLS = NT < 32 ? 32 : NT;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full[MAX_STAGES], empty[MAX_STAGES], done[1];
  __shared__ uint32_t tmem_slot[1];
  __shared__ int abort_word;
  pdl_launch_dependents();   // the successor may take its place on the SMs; it waits for this grid itself
  volatile int* abort_flag = &abort_word;
  const AbortCtx ab{abort_flag, p.status};
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int rank = blockIdx.x % p.cluster, tile = blockIdx.x / p.cluster;
  const int per = (p.k_blocks + p.cluster - 1) / p.cluster;
  const int kb0 = rank * per;
  const int n_kb = max(min(per, p.k_blocks - kb0), 0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  float* red = reinterpret_cast<float*>(smem);   // [token][128], over the ring once every product has been made

  if (warp == 0) {
    if (elect_one()) {
      tma_prefetch_desc(&tmW);
      tma_prefetch_desc(&tmX);
      // The predecessor may be what writes W (the cast of an fp32 parameter, a copy into it): W is read after the wait
      // like x, and only brought into L2 ahead of it.
      for (int i = 0; i < min(n_kb, p.stages); ++i) tma_prefetch_l2_2d(&tmW, (kb0 + i) * BK, tile * TILE_N);
      pdl_wait();
      bool ok = true;
      for (int i = 0, s = 0, ph = 1; i < n_kb; ++i) {
        if (!mbar_wait(&empty[s], ph, ab, ERR_WAIT_EMPTY)) { ok = false; break; }
        mbar_expect_tx(&full[s], STAGE_BYTES);
        tma_load_2d(smem + s * STAGE_BYTES, &tmW, &full[s], (kb0 + i) * BK, tile * TILE_N);
        tma_load_2d(smem + s * STAGE_BYTES + W_BYTES, &tmX, &full[s], (kb0 + i) * BK, 0);
        if (++s == p.stages) {
          s = 0;
          ph ^= 1;
        }
      }
      if (!ok) {
        // give copies already in flight time to land before the CTA's shared memory goes away
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(TILE_N, NT, false, false);
      bool ok = true;
      for (int i = 0, s = 0, ph = 0; i < n_kb; ++i) {
        if (!mbar_wait(&full[s], ph, ab, ERR_WAIT_FULL)) { ok = false; break; }
        tc_fence_after();
        const uint32_t base = smem_u32(smem + s * STAGE_BYTES);
        const uint64_t adesc = make_smem_desc_sw128(base, 16, 1024), bdesc = make_smem_desc_sw128(base + W_BYTES, 16, 1024);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          tc_mma_ss(tmem, adesc + k * 2, bdesc + k * 2, idesc, (i != 0 || k != 0) ? 1u : 0u);
        tc_commit(&empty[s]);
        if (++s == p.stages) {
          s = 0;
          ph ^= 1;
        }
      }
      if (ok && n_kb > 0) tc_commit(done);
    }
  } else if (n_kb > 0) {
    const int q = warp & 3;   // TMEM lane quadrant of this warp: weight rows q * 32 ..
    if (mbar_wait_warp(done, 0, ab, ERR_WAIT_TMEM_FULL)) {
      tc_fence_after();
      const uint32_t t_row = tmem + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll
      for (int c = 0; c < NT; c += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(t_row + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) red[(c + i) * TILE_N + q * 32 + lane] = __uint_as_float(r[i]);
      }
    }
  } else {
    for (int i = threadIdx.x - 64; i < NT * TILE_N; i += NUM_THREADS - 64) red[i] = 0.f;   // a slice past the end of K
  }
  __syncwarp();
  tc_fence_before();
  if (p.cluster > 1)
    cluster_sync();
  else
    __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }

  // rows [rank, rank + 1) * 128 / cluster of D, summed over the cluster in rank order
  pdl_wait();   // what the output replaces may still be read by the predecessor
  const int width = TILE_N / p.cluster, vecs = width >> 2;
  const int items = p.rows * vecs;
  for (int it = threadIdx.x; it < items; it += NUM_THREADS) {
    const int token = it / vecs, nl = rank * width + (it - token * vecs) * 4;
    const int n = tile * TILE_N + nl;
    if (n >= p.N) continue;
    const uint32_t at = smem_u32(red + token * TILE_N + nl);
    float4 v;
    if (p.cluster == 1) {
      v = *reinterpret_cast<const float4*>(red + token * TILE_N + nl);
    } else {
      v = ld_cluster4(at, 0);
      for (int r = 1; r < p.cluster; ++r) {
        const float4 w = ld_cluster4(at, r);
        v.x += w.x;
        v.y += w.y;
        v.z += w.z;
        v.w += w.w;
      }
    }
    __nv_bfloat16* dst = p.out + token * p.ldo + n;
    if (((p.N | p.ldo) & 3) == 0) {
      uint2 o;
      o.x = pack_bf16x2(v.x, v.y);
      o.y = pack_bf16x2(v.z, v.w);
      *reinterpret_cast<uint2*>(dst) = o;
    } else {
      const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (n + i < p.N) dst[i] = __float2bfloat16(f[i]);
    }
  }
  if (p.cluster > 1) {
    __syncwarp();
    cluster_sync();   // peers may still read this CTA's partial sums
  }
}

template <int NT>
int launch_skinny(const CUtensorMap& tmW, const CUtensorMap& tmX, SkinnyParams p, int grid, cudaStream_t stream) {
  auto* kern = skinny_gemm_kernel<NT>;
  // The ring takes what the CTAs that share an SM leave each other: with 16 / 32 / 64 / 128 rows 12 / 11 / 9 / 7 stages
  // for one CTA, 6 / 5 / 4 / 3 for two and 4 / 3 / 3 / 2 for three.  32 rows, rings for one, two and three CTAs an SM:
  // 11264 x 2048, 88 CTAs 11.5 / 12.5 / 14.9 us; 50304 x 2048, 393 CTAs 39.2 / 37.8 / 33.8 us.
  const int sms = b200host::sm_count();
  int per_sm = grid <= sms ? 1 : (grid <= 2 * sms ? 2 : 3);
  // eight CTAs on eight SMs to themselves do not fit every part of the device at once (2048 x 5632: 12.6 us, 7.9 with room
  // for two on an SM)
  if (p.cluster == 8 && per_sm == 1) per_sm = 2;
  const int budget = (226 * 1024 / per_sm - 2048) / stage_bytes<NT>();
  const int slice = (p.k_blocks + p.cluster - 1) / p.cluster;
  p.stages = budget < MAX_STAGES ? budget : MAX_STAGES;
  if (p.stages > slice) p.stages = slice;
  if (p.stages < 2) p.stages = 2;
  const int ring = p.stages * stage_bytes<NT>(), sums = NT * TILE_N * 4;   // the partial sums reuse the ring
  const int smem_bytes = (ring > sums ? ring : sums) + 1024;
  static bool configured[b200host::kMaxDevices] = {};
  if (int rc = b200host::ensure_dynamic_smem(kern, 226 * 1024, configured)) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = b200host::pdl_enabled() ? 2 : 1;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kern, tmW, tmX, p));
}

}  // namespace

// out [rows, N] (row stride ldo) = x [rows, K] (lda) * W [N, K]^T (ldb); rows <= 128, K a multiple of 64, `cluster` (1, 2,
// 4 or 8) slices of K.  Strides in elements.
extern "C" int b200_gemm_skinny(const void* x, const void* w, void* out, int rows, int N, int K, int cluster,
                                long long lda, long long ldb, long long ldo, int* status, void* stream) {
  using namespace b200host;
  if (rows <= 0 || rows > 128 || N <= 0 || K <= 0 || K % BK) return RC_BAD_SHAPE;
  if (cluster != 1 && cluster != 2 && cluster != 4 && cluster != 8) return RC_BAD_SHAPE;
  if (reinterpret_cast<uintptr_t>(out) & 7) return RC_BAD_ALIGNMENT;
  const int NT = rows <= 16 ? 16 : (rows <= 32 ? 32 : (rows <= 64 ? 64 : 128));
  const CUtensorMapDataType bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  CUtensorMap tmW, tmX;
  int rc;
  if ((rc = make_map_2d(&tmW, bf, w, K, N, ldb * 2, BK, TILE_N))) return rc;
  if ((rc = make_map_2d(&tmX, bf, x, K, rows, lda * 2, BK, NT))) return rc;
  SkinnyParams p{rows, N, K / BK, cluster, 0, ldo, static_cast<__nv_bfloat16*>(out), status};
  const int grid = (N + TILE_N - 1) / TILE_N * cluster;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  switch (NT) {
    case 16: return launch_skinny<16>(tmW, tmX, p, grid, s);
    case 32: return launch_skinny<32>(tmW, tmX, p, grid, s);
    case 64: return launch_skinny<64>(tmW, tmX, p, grid, s);
    default: return launch_skinny<128>(tmW, tmX, p, grid, s);
  }
}
