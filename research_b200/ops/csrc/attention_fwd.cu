// Flash attention forward for sm_100a (tcgen05 + TMEM + TMA), bf16 in/out, fp32 softmax.
//
// One CTA owns 256 query rows of one (batch, head): two 128-row tiles that ping-pong through the
// tensor core so that the softmax of one tile overlaps the MMAs of the other.
//   warp 0      TMA producer: both Q tiles once, then K/V blocks of 128 rows through a 5-slot ring
//   warp 1      MMA issuer  : S_t = Q_t K^T (TMEM, 128 cols per tile), O_t += P_t V (TMEM, D cols)
//   warps 2-5   softmax of tile 0, warps 6-9 softmax of tile 1: one thread per query row reads its
//               row of S with tcgen05.ld, keeps the running max / sum, writes P (bf16) over the first
//               half of S in tensor memory, where the second MMA takes it as its A operand, and rescales
//               O in TMEM only when the running max moved by more than 2^8 (so most blocks skip the
//               rescale).
// What bounds it: a 128 x 128 block of a tile is 2 x 512 clocks of the tensor pipe and 16384 exponentials (1024 clocks of
// the special-function units), so the two tiles of a CTA have to overlap; the loop of one tile, softmax -> PV -> QK^T ->
// softmax, takes about 1600 + 1024 + 600 clocks and sets the pace.  The tensor pipe runs its MMAs in the order they are
// issued: PV(j) of a tile, which reads P, precedes QK^T(j+1), which overwrites it with the next S, and S(j+1) being
// complete says that PV(j) is, so neither needs a barrier of its own.  The scores are read from tensor memory once, the
// maximum takes three operands an instruction, the scaling and the sum two lanes, and the loop bounds that select
// descriptors are made warp-uniform (b200.cuh: warp_uniform).  With P in shared memory, a pass for the maximum and
// descriptors in ordinary registers the loop took 6100 clocks: 8 x 4096 tokens of 16 / 8 heads of 128, causal, 782 us,
// now 536 to 556 by box; 16384 tokens 1382 us, now 898 to 1050 by the clock under power.  A quarter of the exponentials as
// polynomials on the FMA pipes made it slower (920 us).
// Masks: every query row attends to kv positions in [lo[row], row] (causal) or [lo[row], S) (not
// causal); `lo` (int32 [B,S], non-decreasing along S, optional) encodes document starts and sliding
// windows, and whole kv blocks left of lo[first row] or right of the last row are skipped.
// GQA: query head h reads kv head h / (Hq / Hkv).  Writes O [B,S,Hq,D] and LSE [B,Hq,S] (natural log).
//
// Context parallelism (`ring.enabled`): K and V are the staging buffers of ring.cuh; the first `n_transfer` CTAs
// pull the rows from their owners while the others attend, and the TMA producer waits on a block's flag before it
// loads the block.
//
// Oracle: the reference's attention is softmax(QK^T / sqrt(D)) V with fp32 logits and probabilities
// cast to the compute dtype (models/components/attention.py:269-278); masks from
// models/components/masks.py:9-48.  Its vendored Blackwell comparator (other head dims, no backward, no
// document mask) is third_party/ThunderKittens/kernels/attention/bf16_b300_mha_causal/bf16_b300_mha_causal.cu.
#include <type_traits>

#include "b200.cuh"
#include "host_util.cuh"
#include "ring.cuh"

using namespace b200;

namespace {

constexpr int NT = 2;          // query tiles per CTA
constexpr int TILE_M = 128;    // query rows per tile
constexpr int BLOCK_N = 128;   // kv rows per block
constexpr int KV_SLOTS = 5;
constexpr int NUM_THREADS = 32 * (2 + 4 * NT);
constexpr float kRescaleThreshold = 8.0f;  // log2 units

template <int D>
struct FwdSmem {
  static constexpr int TILE_D_BYTES = 128 * D * 2;    // Q tile, K block, V block
  static constexpr int Q_OFF = 0;                     // a Q tile is also the staging of its output tile
  static constexpr int KV_OFF = Q_OFF + NT * TILE_D_BYTES;
  static constexpr int BAR_OFF = KV_OFF + KV_SLOTS * TILE_D_BYTES;
  static constexpr int TOTAL = BAR_OFF + 256;
};

struct FwdParams {
  int B, S, Skv, q_off, Hq, Hkv;  // S = query rows; Skv = kv rows; q_off = global position of query row 0
  int causal;
  float scale_log2;  // softmax scale * log2(e)
  const int* lo;     // [B, S] or nullptr
  float* lse;        // [B, Hq, S]
  int* status;
  b200ring::RingArgs ring;
};

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <int D>
__global__ void __launch_bounds__(NUM_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, const FwdParams p) {
  using L = FwdSmem<D>;
  constexpr int NBOX = D / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* kv_full = q_full + 1;
  uint64_t* kv_empty = kv_full + KV_SLOTS;
  uint64_t* s_full = kv_empty + KV_SLOTS;
  uint64_t* p_ready = s_full + NT;
  uint64_t* pv_done = p_ready + NT;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + NT);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const AbortCtx ab{abort_flag, p.status};

  const int warp = warp_uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;

  // context parallelism: the first CTAs of the grid stage K/V instead of attending
  const int n_xfer = p.ring.enabled ? p.ring.n_transfer : 0;
  const bool is_xfer = (int)blockIdx.x < n_xfer;
  const int cta = is_xfer ? 0 : (int)blockIdx.x - n_xfer;
  // heavy (late) query tiles first: causal work grows with the tile index
  const int q_tiles = (p.S + NT * TILE_M - 1) / (NT * TILE_M);
  // ... over the whole grid (all heads of the longest tile, then the next), which balances the tail
  const int nbh = p.B * p.Hq;
  const int qt = q_tiles - 1 - (cta / nbh);
  const int bh = cta % nbh;
  const int h = bh % p.Hq;
  const int b = bh / p.Hq;
  const int hkv = h / (p.Hq / p.Hkv);
  const int q0 = qt * NT * TILE_M;

  // kv block range of each tile and of the CTA (kv positions are global; query row r sits at global position
  // q_off + r).  The CTA streams the union; blocks are counted from its first.
  int t_begin[NT], t_end[NT];
  int kv_begin = 0x7fffffff, kv_end = 0;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const int first = q0 + t * TILE_M;
    t_begin[t] = t_end[t] = 0;
    if (first < p.S && !is_xfer) {
      if (p.lo) t_begin[t] = p.lo[(long long)b * p.S + first] / BLOCK_N;
      t_end[t] = (p.Skv + BLOCK_N - 1) / BLOCK_N;
      if (p.causal) t_end[t] = min(t_end[t], (p.q_off + min(first + TILE_M, p.S) - 1) / BLOCK_N + 1);
    }
    if (t_end[t] > t_begin[t]) {
      kv_begin = min(kv_begin, t_begin[t]);
      kv_end = max(kv_end, t_end[t]);
    }
  }
  const int n_blocks = warp_uniform(max(kv_end - kv_begin, 0));
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    if (t_end[t] <= t_begin[t]) t_begin[t] = t_end[t] = n_blocks ? kv_begin : 0;
    t_begin[t] = warp_uniform(t_begin[t] - (n_blocks ? kv_begin : 0));
    t_end[t] = warp_uniform(t_end[t] - (n_blocks ? kv_begin : 0));
  }

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < KV_SLOTS; ++s) {
      mbar_init(&kv_full[s], 1);
      mbar_init(&kv_empty[s], 1);
    }
    for (int t = 0; t < NT; ++t) {
      mbar_init(&s_full[t], 1);
      mbar_init(&p_ready[t], 4);
      mbar_init(&pv_done[t], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_S = tmem_base;              // NT * 128 columns
  const uint32_t tmem_O = tmem_base + NT * 128;   // NT * D columns

  if (is_xfer) {
    // ---------------------------------------------------------------- K/V transfer (context parallelism)
    // buffers and barriers of the copy pipelines sit in front of this kernel's own barriers (L::BAR_OFF)
    b200ring::transfer_cta<b200ring::pipes_for_window(L::BAR_OFF)>(p.ring, smem, ab);
  } else if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0 && n_blocks > 0) {
      tma_prefetch_desc(&tmQ);
      tma_prefetch_desc(&tmK);
      tma_prefetch_desc(&tmV);
      mbar_expect_tx(q_full, NT * L::TILE_D_BYTES);
      for (int t = 0; t < NT; ++t)
        for (int bx = 0; bx < NBOX; ++bx)
          tma_load_4d(smem + L::Q_OFF + t * L::TILE_D_BYTES + bx * 16384, &tmQ, q_full, bx * 64, h, q0 + t * TILE_M, b);
      // item order: K0, then for each block j: K(j+1) if it exists, V(j)
      uint32_t item = 0;
      bool ok = true;
      auto load_block = [&](const CUtensorMap* tm, int j) {
        const int slot = item % KV_SLOTS;
        const uint32_t ph = (item / KV_SLOTS) & 1;
        if (!mbar_wait(&kv_empty[slot], ph ^ 1, ab, ERR_WAIT_EMPTY)) { ok = false; return; }
        if (p.ring.enabled && !b200ring::wait_block(p.ring, b, kv_begin + j, p.status)) {
          *ab.flag = 1;   // the block never arrived: the other roles of this CTA stop waiting too
          ok = false;
          return;
        }
        mbar_expect_tx(&kv_full[slot], L::TILE_D_BYTES);
        for (int bx = 0; bx < NBOX; ++bx)
          tma_load_4d(smem + L::KV_OFF + slot * L::TILE_D_BYTES + bx * 16384, tm, &kv_full[slot], bx * 64, hkv,
                      (kv_begin + j) * BLOCK_N, b);
        ++item;
      };
      load_block(&tmK, 0);
      for (int j = 0; j < n_blocks && ok; ++j) {
        if (j + 1 < n_blocks) load_block(&tmK, j + 1);
        if (ok) load_block(&tmV, j);
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (n_blocks > 0 && elect_one()) {
      constexpr uint32_t idesc_qk = make_idesc_bf16(TILE_M, BLOCK_N, false, false);
      constexpr uint32_t idesc_pv = make_idesc_bf16(TILE_M, D, false, true);
      bool ok = mbar_wait(q_full, 0, ab, ERR_WAIT_FULL);
      uint32_t item = 0;
      // Shared-memory descriptors are built once per operand; the slice of one MMA instruction is that descriptor
      // plus a compile-time constant in its address field (units of 16 bytes).  A tile product is D / 16 (or
      // BLOCK_N / 16) instructions of 64 clocks each and one thread issues them all, so next to nothing may sit
      // between two of them.
      uint64_t dq[NT], dk[KV_SLOTS], dv[KV_SLOTS];
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        dq[t] = make_smem_desc_sw128(smem_u32(smem + L::Q_OFF + t * L::TILE_D_BYTES), 16, 1024);
      }
#pragma unroll
      for (int sl = 0; sl < KV_SLOTS; ++sl) {
        const uint32_t kv_base = smem_u32(smem + L::KV_OFF + sl * L::TILE_D_BYTES);
        dk[sl] = make_smem_desc_sw128(kv_base, 16, 1024);
        dv[sl] = make_smem_desc_sw128(kv_base, 16384, 1024);
      }
      auto slot_of = [](const uint64_t (&d)[KV_SLOTS], int slot) {
        uint64_t v = d[0];
#pragma unroll
        for (int sl = 1; sl < KV_SLOTS; ++sl) v = slot == sl ? d[sl] : v;
        return v;
      };
      auto issue_qk = [&](int t, int slot) {
        const uint64_t a0 = t == 0 ? dq[0] : dq[1], b0 = slot_of(dk, slot);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint64_t off = (uint64_t)(((kk >> 2) * 16384 + (kk & 3) * 32) >> 4);
          tc_mma_ss(tmem_S + t * 128, a0 + off, b0 + off, idesc_qk, kk != 0 ? 1u : 0u);
        }
        tc_commit(&s_full[t]);
      };
      // A = P in tensor memory, over the first 64 columns of S: 16 kv rows are 8 columns of packed bf16
      auto issue_pv = [&](int t, int slot, bool accumulate) {
        const uint64_t b0 = slot_of(dv, slot);
#pragma unroll
        for (int kk = 0; kk < BLOCK_N / 16; ++kk)
          tc_mma_ts(tmem_O + t * D, tmem_S + t * 128 + kk * 8, b0 + (uint64_t)((kk * 2048) >> 4), idesc_pv,
                    (accumulate || kk != 0) ? 1u : 0u);
      };
      auto kv_wait = [&](uint32_t it) {
        const bool got = mbar_wait(&kv_full[it % KV_SLOTS], (it / KV_SLOTS) & 1, ab, ERR_WAIT_FULL);
        tc_fence_after();
        return got;
      };
      if (ok && (ok = kv_wait(item))) {
#pragma unroll
        for (int t = 0; t < NT; ++t)
          if (t_begin[t] == 0 && t_end[t] > 0) issue_qk(t, 0);
        tc_commit(&kv_empty[0]);
        ++item;
      }
      for (int j = 0; j < n_blocks && ok; ++j) {
        const bool has_next = j + 1 < n_blocks;
        const uint32_t k_item = item, v_item = item + (has_next ? 1 : 0);
        const int k_slot = k_item % KV_SLOTS, v_slot = v_item % KV_SLOTS;
        bool k_there = false, v_there = false;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          if (ok && j >= t_begin[t] && j < t_end[t]) {
            // P(j) is in tensor memory and O is rescaled
            ok = mbar_wait(&p_ready[t], (j - t_begin[t]) & 1, ab, ERR_WAIT_P_READY) && (v_there || kv_wait(v_item));
            if (ok) {
              v_there = true;
              tc_fence_after();
              issue_pv(t, v_slot, j > t_begin[t]);
              if (j + 1 == t_end[t]) tc_commit(&pv_done[t]);
            }
          }
          if (ok && t == NT - 1) tc_commit(&kv_empty[v_slot]);
          if (ok && j + 1 >= t_begin[t] && j + 1 < t_end[t]) {
            ok = k_there || kv_wait(k_item);
            if (ok) {
              k_there = true;
              issue_qk(t, k_slot);
            }
          }
        }
        if (ok && has_next) tc_commit(&kv_empty[k_slot]);
        item = v_item + 1;
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax / correction / epilogue
    const int t = (warp - 2) >> 2;
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const int q_row = q0 + t * TILE_M + row;       // local row (indexes lo / lse / O)
    const int q_pos = p.q_off + q_row;             // global position (compared with kv positions)
    const uint32_t lane_sel = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t tS = tmem_S + t * 128 + lane_sel;
    const uint32_t tO = tmem_O + t * D + lane_sel;
    uint8_t* sO = smem + L::Q_OFF + t * L::TILE_D_BYTES;
    int lo_row = 0;
    if (p.lo) lo_row = p.lo[(long long)b * p.S + min(q_row, p.S - 1)];
    const int hi_row = p.causal ? min(q_pos, p.Skv - 1) : p.Skv - 1;
    const int j_begin = t == 0 ? t_begin[0] : t_begin[1], j_end = t == 0 ? t_end[0] : t_end[1];
    const uint64_t scale2 = f2_pack(p.scale_log2, p.scale_log2);
    float m_ref = -1.0e30f;
    float l_sum = 0.f;
    // rows that no kv row is visible to, a whole tile of them here: O = 0 and LSE = -inf, as for single such rows below
    const bool empty = j_end <= j_begin;
    bool ok = q0 + t * TILE_M < p.S;
    for (int j = j_begin; j < j_end && ok; ++j) {
      const int kv0 = (kv_begin + j) * BLOCK_N;
      if (!mbar_wait_warp(&s_full[t], (j - j_begin) & 1, ab, ERR_WAIT_S_READY)) { ok = false; break; }
      tc_fence_after();
      const bool masked = __any_sync(0xffffffffu, kv0 + BLOCK_N - 1 > hi_row || kv0 < lo_row);
      const int hi = hi_row - kv0, lo = lo_row - kv0;
      auto mask = [&](uint32_t (&r)[32], int c) {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (c * 32 + i > hi || c * 32 + i < lo) r[i] = 0xff800000u;   // -inf
      };
      uint64_t sum0 = 0, sum1 = 0;   // two partial sums of two lanes each
      float top;                     // largest exponent of the block relative to m_ref
      uint32_t ra[32], rb[32], packed[64];
      // exponentials of 32 scores relative to m_ref, their sum, and P as bf16 pairs
      auto emit = [&](uint32_t (&r)[32], int c, uint64_t minus_m, auto is_masked) {
        constexpr bool kMasked = decltype(is_masked)::value;
        if constexpr (kMasked) mask(r, c);
        float t0 = -INFINITY, t1 = -INFINITY;
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          float e0, e1, e2, e3;
          f2_unpack(f2_fma(f2_pack(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), scale2, minus_m), e0, e1);
          f2_unpack(f2_fma(f2_pack(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])), scale2, minus_m), e2, e3);
          t0 = max3(t0, e0, e1);
          t1 = max3(t1, e2, e3);
          e0 = ex2_approx(e0);
          e1 = ex2_approx(e1);
          e2 = ex2_approx(e2);
          e3 = ex2_approx(e3);
          sum0 = f2_add(sum0, f2_pack(e0, e1));
          sum1 = f2_add(sum1, f2_pack(e2, e3));
          packed[c * 16 + i / 2] = pack_bf16x2(e0, e1);
          packed[c * 16 + i / 2 + 1] = pack_bf16x2(e2, e3);
        }
        top = max3(top, t0, t1);
      };
      // Nearly every block but the first takes the reference maximum of the blocks before it: the lazy rule tolerates a
      // maximum up to 2^8 above it, and whether it held is known at the end of the pass, before P goes over the scores.
      // Otherwise the block's maximum is searched first, O and the sum are rescaled, and the pass is made again.
      bool search = j == j_begin;
#pragma unroll 1
      while (true) {
        if (search) {
          // block maximum of the scaled scores (scale > 0, so the maximum commutes with it)
          float bm = -INFINITY;
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            tmem_ld_32x32b_x32(tS + c * 32, ra);
            tmem_ld_wait();
            if (masked) mask(ra, c);
#pragma unroll
            for (int i = 0; i < 32; i += 2) bm = max3(bm, __uint_as_float(ra[i]), __uint_as_float(ra[i + 1]));
          }
          bm *= p.scale_log2;
          const float m_new = bm > m_ref + kRescaleThreshold ? bm : m_ref;
          const float alpha = ex2_approx(m_ref - m_new);
          if (j > j_begin) {
            // S(j) is complete, so PV(j-1), issued before it, is too: O holds the sum over the blocks before this one
#pragma unroll 1
            for (int c = 0; c < D / 32; ++c) {
              tmem_ld_32x32b_x32(tO + c * 32, ra);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) ra[i] = __float_as_uint(__uint_as_float(ra[i]) * alpha);
              tmem_st_32x32b_x32(tO + c * 32, ra);
            }
          }
          l_sum *= alpha;
          m_ref = m_new;
        }
        // one pass over the scores, the loads of 32 columns in flight while the 32 before are worked on
        const uint64_t minus_m = f2_pack(-m_ref, -m_ref);
        sum0 = sum1 = 0;
        top = -INFINITY;
        auto pass = [&](auto is_masked) {
          tmem_ld_32x32b_x32(tS, ra);
          tmem_ld_wait();
          tmem_ld_32x32b_x32(tS + 32, rb);
          emit(ra, 0, minus_m, is_masked);
          tmem_ld_wait();
          tmem_ld_32x32b_x32(tS + 64, ra);
          emit(rb, 1, minus_m, is_masked);
          tmem_ld_wait();
          tmem_ld_32x32b_x32(tS + 96, rb);
          emit(ra, 2, minus_m, is_masked);
          tmem_ld_wait();
          emit(rb, 3, minus_m, is_masked);
        };
        if (masked)
          pass(std::true_type{});
        else
          pass(std::false_type{});
        if (search || !__any_sync(0xffffffffu, top > kRescaleThreshold)) break;
        search = true;
      }
      tmem_st_32x32b_x64(tS, packed);
      float s0, s1, s2, s3;
      f2_unpack(sum0, s0, s1);
      f2_unpack(sum1, s2, s3);
      l_sum += (s0 + s1) + (s2 + s3);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[t]);
    }
    if (ok && !empty) ok = mbar_wait_warp(&pv_done[t], 0, ab, ERR_WAIT_O_READY);
    // an empty tile of a CTA that streams blocks for the other one: its Q tile, where O is staged, has to have landed
    if (ok && empty && n_blocks > 0) ok = mbar_wait_warp(q_full, 0, ab, ERR_WAIT_FULL);
    if (ok) {
      tc_fence_after();
      const float inv_l = l_sum > 0.f ? 1.f / l_sum : 0.f;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t r[32];
        if (!empty) {
          tmem_ld_32x32b_x32(tO + c * 32, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint4 v;
          v.x = pack_bf16x2(__uint_as_float(r[8 * i + 0]) * inv_l, __uint_as_float(r[8 * i + 1]) * inv_l);
          v.y = pack_bf16x2(__uint_as_float(r[8 * i + 2]) * inv_l, __uint_as_float(r[8 * i + 3]) * inv_l);
          v.z = pack_bf16x2(__uint_as_float(r[8 * i + 4]) * inv_l, __uint_as_float(r[8 * i + 5]) * inv_l);
          v.w = pack_bf16x2(__uint_as_float(r[8 * i + 6]) * inv_l, __uint_as_float(r[8 * i + 7]) * inv_l);
          *reinterpret_cast<uint4*>(sO + (c >> 1) * 16384 + sw128_offset(row, (c & 1) * 4 + i)) = v;
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      const int slab_row = q0 + t * TILE_M + quad * 32;
      if (lane == 0 && slab_row < p.S) {
        for (int bx = 0; bx < NBOX; ++bx)
          tma_store_4d(&tmO, sO + bx * 16384 + quad * 32 * 128, bx * 64, h, slab_row, b);
        tma_commit_group();
        tma_wait_group<0>();
      }
      if (q_row < p.S)
        p.lse[((long long)b * p.Hq + h) * p.S + q_row] =
            l_sum > 0.f ? m_ref * 0.6931471805599453f + logf(l_sum) : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int D>
int launch_fwd(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmO,
               const FwdParams& p, cudaStream_t stream) {
  using L = FwdSmem<D>;
  auto* kern = attn_fwd_kernel<D>;
  constexpr int smem_bytes = L::TOTAL + 1024;
  static bool configured[b200host::kMaxDevices] = {};   // per kernel instantiation and device
  if (int rc = b200host::ensure_dynamic_smem(kern, smem_bytes, configured)) return rc;
  const int q_tiles = (p.S + NT * TILE_M - 1) / (NT * TILE_M);
  const int grid = q_tiles * p.Hq * p.B + (p.ring.enabled ? p.ring.n_transfer : 0);
  kern<<<grid, NUM_THREADS, smem_bytes, stream>>>(tmQ, tmK, tmV, tmO, p);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace

// q: [B,S,Hq,D] view with element strides (q_row = between tokens, q_batch = between batches; heads are D
// apart); k, v: [B,Skv,Hkv,D] likewise; o: [B,S,Hq,D]; lse: [B,Hq,S] fp32; lo: [B,S] int32 or null.
// skv_and_qoff packs the kv length and the global position of query row 0 for context-parallel callers
// (0 = same length as the queries, offset 0): low 32 bits Skv, high 32 bits q_off (a multiple of 128).
static int attn_fwd_impl(const void* q, const void* k, const void* v, void* o, void* lse, const void* lo, int B, int S,
                         int Hq, int Hkv, int D, long long q_row, long long q_batch, long long k_row,
                         long long k_batch, long long v_row, long long v_batch, long long o_row, long long o_batch,
                         float scale, int causal, long long skv_and_qoff, const b200ring::RingHostArgs* ring,
                         int* status, void* stream) {
  using namespace b200host;
  const int Skv = (skv_and_qoff & 0xffffffffLL) ? (int)(skv_and_qoff & 0xffffffffLL) : S;
  const int q_off = (int)(skv_and_qoff >> 32);
  if (q_off % 128 != 0 || q_off < 0) return RC_BAD_SHAPE;
  if (B <= 0 || S <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv) return RC_BAD_SHAPE;
  if (D != 128 && D != 64) return RC_BAD_SHAPE;
  const CUtensorMapDataType bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  CUtensorMap tmQ, tmK, tmV, tmO;
  int rc;
  if ((rc = make_map_4d(&tmQ, bf, q, D, Hq, S, B, (uint64_t)D * 2, q_row * 2, q_batch * 2, 64, 1, 128))) return rc;
  if ((rc = make_map_4d(&tmK, bf, k, D, Hkv, Skv, B, (uint64_t)D * 2, k_row * 2, k_batch * 2, 64, 1, 128))) return rc;
  if ((rc = make_map_4d(&tmV, bf, v, D, Hkv, Skv, B, (uint64_t)D * 2, v_row * 2, v_batch * 2, 64, 1, 128))) return rc;
  if ((rc = make_map_4d(&tmO, bf, o, D, Hq, S, B, (uint64_t)D * 2, o_row * 2, o_batch * 2, 64, 1, 32))) return rc;
  FwdParams p{B, S, Skv, q_off, Hq, Hkv, causal, scale * 1.4426950408889634f, (const int*)lo, (float*)lse, status};
  if (ring) {
    // K and V are the staging buffers: dense [B, seq_len, Hkv, D], filled by this launch's transfer CTAs
    if (k_row != (long long)Hkv * D || v_row != k_row || k_batch != (long long)ring->seq_len * k_row ||
        v_batch != k_batch || Skv > ring->seq_len)
      return RC_BAD_SHAPE;
    if ((rc = b200ring::fill_ring_args(p.ring, *ring, const_cast<void*>(k), const_cast<void*>(v), B, Hkv, D))) return rc;
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (D == 128) return launch_fwd<128>(tmQ, tmK, tmV, tmO, p, s);
  return launch_fwd<64>(tmQ, tmK, tmV, tmO, p, s);
}

extern "C" int b200_attn_fwd(const void* q, const void* k, const void* v, void* o, void* lse, const void* lo, int B,
                             int S, int Hq, int Hkv, int D, long long q_row, long long q_batch, long long k_row,
                             long long k_batch, long long v_row, long long v_batch, long long o_row,
                             long long o_batch, float scale, int causal, long long skv_and_qoff, int* status,
                             void* stream) {
  return attn_fwd_impl(q, k, v, o, lse, lo, B, S, Hq, Hkv, D, q_row, q_batch, k_row, k_batch, v_row, v_batch, o_row,
                       o_batch, scale, causal, skv_and_qoff, nullptr, status, stream);
}

// The same with the K/V exchange of context parallelism inside the launch (ring.cuh): k, v are this rank's
// staging buffers [B, seq_len, Hkv, D]; `ring` says which blocks to pull from which rank's buffer.
extern "C" int b200_attn_fwd_ring(const void* q, const void* k, const void* v, void* o, void* lse, const void* lo,
                                  int B, int S, int Hq, int Hkv, int D, long long q_row, long long q_batch,
                                  long long k_row, long long k_batch, long long v_row, long long v_batch,
                                  long long o_row, long long o_batch, float scale, int causal,
                                  long long skv_and_qoff, const void* ring, int* status, void* stream) {
  if (!ring) return b200host::RC_BAD_SHAPE;
  return attn_fwd_impl(q, k, v, o, lse, lo, B, S, Hq, Hkv, D, q_row, q_batch, k_row, k_batch, v_row, v_batch, o_row,
                       o_batch, scale, causal, skv_and_qoff, static_cast<const b200ring::RingHostArgs*>(ring), status,
                       stream);
}
