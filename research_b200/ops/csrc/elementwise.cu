// Bandwidth-bound kernels of the training step for sm_100a: RMSNorm (+ residual add), QK-RMSNorm
// fused with interleaved-pair RoPE, SwiGLU, embedding gather / scatter-add, masked cross-entropy
// with z-loss that leaves dlogits in place, flat-arena AdamW with bf16 shadow write, sum of squares.
// All use 128-bit global accesses; reductions are warp shuffles, fp32 throughout.
//
// Math restated from the reference: RMSNorm and its scale (models/components/norm.py:12-38), RoPE over
// even/odd pairs (models/components/position.py:9-39), QK-norm before RoPE
// (models/components/attention.py:112-126, 228-234), SwiGLU (models/components/ffn.py:13-51), masked CE in
// fp32 log-softmax (steps/eval.py:27-37), z-loss (steps/train.py:597-602), AdamW (optim/build.py:29-31).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "b200.cuh"
#include "host_util.cuh"

namespace {

constexpr int kWarpsPerBlock = 8;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 v;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return v;
}
__device__ __forceinline__ void load8f(const float* p, float (&f)[8]) {
  float4 a = *reinterpret_cast<const float4*>(p);
  float4 b = *reinterpret_cast<const float4*>(p + 4);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
  f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

// Norm scales come as the caller holds them: an fp32 parameter, or the bf16 compute copy that the parameter store keeps
// of every parameter.  The kernels are templates on that type (a test at each load cost the forward kernel a fifth of
// its rate at 2999 rows of 4096).
__device__ __forceinline__ void load8w(const float* w, float (&f)[8]) { load8f(w, f); }
__device__ __forceinline__ void load8w(const __nv_bfloat16* w, float (&f)[8]) {
  unpack8(*reinterpret_cast<const uint4*>(w), f);
}
// four consecutive floats += v in one request (dst 16-byte aligned)
__device__ __forceinline__ void red_add4(float* dst, const float4& v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}

// ------------------------------------------------------------------------------------------------
// RMSNorm forward: optionally res_out = x + delta first.  One warp per row, H % 8 == 0.
// ------------------------------------------------------------------------------------------------
template <typename W>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ delta,
                   const W* __restrict__ w, __nv_bfloat16* __restrict__ res_out, __nv_bfloat16* __restrict__ y,
                   float* __restrict__ rstd_out, int rows, int H, float eps) {
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nvec = H >> 3;
  for (long long row = (long long)blockIdx.x * kWarpsPerBlock + warp; row < rows;
       row += (long long)gridDim.x * kWarpsPerBlock) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * H);
    const uint4* dr = delta ? reinterpret_cast<const uint4*>(delta + row * H) : nullptr;
    uint4* rr = res_out ? reinterpret_cast<uint4*>(res_out + row * H) : nullptr;
    float ss = 0.f;
    for (int v = lane; v < nvec; v += 32) {
      float f[8];
      unpack8(xr[v], f);
      if (dr) {
        float g[8];
        unpack8(dr[v], g);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] += g[i];
        uint4 s = pack8(f);
        rr[v] = s;
        unpack8(s, f);  // normalise exactly what was stored
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
    }
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / (float)H + eps);
    if (lane == 0 && rstd_out) rstd_out[row] = rstd;
    const uint4* src = dr ? reinterpret_cast<const uint4*>(res_out + row * H) : xr;
    uint4* yr = reinterpret_cast<uint4*>(y + row * H);
    for (int v = lane; v < nvec; v += 32) {
      float f[8], wv[8];
      unpack8(src[v], f);
      load8w(w + v * 8, wv);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = f[i] * rstd * wv[i];
      yr[v] = pack8(f);
    }
  }
}

// H == NV * 256: a warp keeps its whole row in registers, so every load of the row is in flight at once and the row
// is read from memory exactly once (the generic kernel above walks the row twice with one load in flight per lane).
template <int NV, typename W>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
rmsnorm_fwd_reg_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ delta,
                       const W* __restrict__ w, __nv_bfloat16* __restrict__ res_out, __nv_bfloat16* __restrict__ y,
                       float* __restrict__ rstd_out, int rows, float eps) {
  constexpr int H = NV * 256;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  for (long long row = (long long)blockIdx.x * kWarpsPerBlock + warp; row < rows;
       row += (long long)gridDim.x * kWarpsPerBlock) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * H);
    uint4 raw[NV], draw[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) raw[j] = xr[lane + 32 * j];
    if (delta) {
      const uint4* dr = reinterpret_cast<const uint4*>(delta + row * H);
#pragma unroll
      for (int j = 0; j < NV; ++j) draw[j] = dr[lane + 32 * j];
    }
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      float f[8];
      unpack8(raw[j], f);
      if (delta) {
        float g[8];
        unpack8(draw[j], g);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] += g[i];
        raw[j] = pack8(f);
        reinterpret_cast<uint4*>(res_out + row * H)[lane + 32 * j] = raw[j];
        unpack8(raw[j], f);  // normalise exactly what was stored
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
    }
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / (float)H + eps);
    if (lane == 0 && rstd_out) rstd_out[row] = rstd;
    uint4* yr = reinterpret_cast<uint4*>(y + row * H);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      float f[8], wv[8];
      unpack8(raw[j], f);
      load8w(w + (lane + 32 * j) * 8, wv);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = f[i] * rstd * wv[i];
      yr[lane + 32 * j] = pack8(f);
    }
  }
}

// The same for a handful of rows (a decode step): one block per row, so that a row's loads are issued by 256 threads at
// once instead of one warp walking it.
template <typename W>
__global__ void __launch_bounds__(256)
rmsnorm_fwd_row_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ delta,
                       const W* __restrict__ w, __nv_bfloat16* __restrict__ res_out, __nv_bfloat16* __restrict__ y,
                       float* __restrict__ rstd_out, int H, float eps) {
  __shared__ float part[8];
  b200::pdl_launch_dependents();   // no-ops unless launched as a dependent (decode steps)
  b200::pdl_wait();
  const long long row = blockIdx.x;
  const int nvec = H >> 3;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * H);
  const uint4* dr = delta ? reinterpret_cast<const uint4*>(delta + row * H) : nullptr;
  uint4* rr = res_out ? reinterpret_cast<uint4*>(res_out + row * H) : nullptr;
  float ss = 0.f;
  for (int v = threadIdx.x; v < nvec; v += 256) {
    float f[8];
    unpack8(xr[v], f);
    if (dr) {
      float g[8];
      unpack8(dr[v], g);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] += g[i];
      uint4 s = pack8(f);
      rr[v] = s;
      unpack8(s, f);  // normalise exactly what was stored
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
  __syncthreads();
  float total = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) total += part[i];
  const float rstd = rsqrtf(total / (float)H + eps);
  if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
  const uint4* src = dr ? reinterpret_cast<const uint4*>(res_out + row * H) : xr;
  uint4* yr = reinterpret_cast<uint4*>(y + row * H);
  for (int v = threadIdx.x; v < nvec; v += 256) {  // a thread re-reads only what it wrote itself
    float f[8], wv[8];
    unpack8(src[v], f);
    load8w(w + v * 8, wv);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = f[i] * rstd * wv[i];
    yr[v] = pack8(f);
  }
}

// RMSNorm backward.  dx = rstd * (dy*w - xhat * mean(dy*w*xhat)) (+ dres if given); dw += sum_rows dy*xhat
// Any H % 8 == 0: one warp per row, the dw partial sums of a block go through shared-memory atomics.
template <typename W>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const W* __restrict__ w, const float* __restrict__ rstd_in,
                   const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ dres,
                   __nv_bfloat16* __restrict__ dx, float* __restrict__ dw, int rows, int H) {
  extern __shared__ float dw_smem[];  // H floats
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nvec = H >> 3;
  for (int i = threadIdx.x; i < H; i += blockDim.x) dw_smem[i] = 0.f;
  __syncthreads();
  for (long long row = (long long)blockIdx.x * kWarpsPerBlock + warp; row < rows;
       row += (long long)gridDim.x * kWarpsPerBlock) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * H);
    const uint4* gr = reinterpret_cast<const uint4*>(dy + row * H);
    const float rstd = rstd_in[row];
    float dot = 0.f;
    for (int v = lane; v < nvec; v += 32) {
      float f[8], g[8], wv[8];
      unpack8(xr[v], f);
      unpack8(gr[v], g);
      load8w(w + v * 8, wv);
#pragma unroll
      for (int i = 0; i < 8; ++i) dot += g[i] * wv[i] * f[i] * rstd;
    }
    dot = warp_sum(dot) / (float)H;
    const uint4* rr = dres ? reinterpret_cast<const uint4*>(dres + row * H) : nullptr;
    uint4* dxr = reinterpret_cast<uint4*>(dx + row * H);
    for (int v = lane; v < nvec; v += 32) {
      float f[8], g[8], wv[8], o[8];
      unpack8(xr[v], f);
      unpack8(gr[v], g);
      load8w(w + v * 8, wv);
      float r[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (rr) unpack8(rr[v], r);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float xhat = f[i] * rstd;
        o[i] = rstd * (g[i] * wv[i] - xhat * dot) + r[i];
        atomicAdd(&dw_smem[v * 8 + i], g[i] * xhat);
      }
      dxr[v] = pack8(o);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    const float v = dw_smem[i];
    if (v != 0.f) atomicAdd(&dw[i], v);
  }
}

// RMSNorm backward for H = 8 * blockDim.x * VEC: a block walks groups of ROWS rows, a thread owns 8 * VEC columns of
// them, so x, dy and dres are read once, all 3 * ROWS * VEC 16-byte loads of a group are in flight at once, the dw
// partial sums are registers, and one block-wide reduction serves ROWS dot products.  What bounds it: memory traffic
// (three reads and one write of the rows); blocks of at most 256 threads leave room for several per SM, whose loads
// cover each other's reductions.  One warp per row, which re-reads x and dy for its second pass, took 150 us at 32768
// rows of 2048 and 294 us at 20000 rows of 3072 where this takes 107 us and 110 us (5.0 and 4.5 TB/s).
// AHEAD: the next group's loads are issued before the current one is reduced, for rows so wide that one block fills
// an SM (8000 rows of 8192: 109 us with, 122 us without).
template <int VEC, int ROWS, int MAXT, int MINB, bool AHEAD, typename W>
__global__ void __launch_bounds__(MAXT, MINB)
rmsnorm_bwd_cols_kernel(const __nv_bfloat16* __restrict__ x, const W* __restrict__ w, const float* __restrict__ rstd_in,
                        const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ dres,
                        __nv_bfloat16* __restrict__ dx, float* __restrict__ dw, int rows, int H) {
  extern __shared__ float dw_smem[];  // H floats
  __shared__ float red[2][ROWS][32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int warps = blockDim.x >> 5, threads = blockDim.x;
  const long long nvec = H >> 3;
  const float inv_h = 1.f / (float)H;
  float wv[VEC][8], acc[VEC][8];
#pragma unroll
  for (int v = 0; v < VEC; ++v) {
    load8w(w + (t + v * threads) * 8, wv[v]);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[v][i] = 0.f;
  }
  uint4 xc[ROWS][VEC], gc[ROWS][VEC], rc[ROWS][VEC];
  float rs[ROWS];
  auto load = [&](long long row0, uint4 (&xl)[ROWS][VEC], uint4 (&gl)[ROWS][VEC], uint4 (&rl)[ROWS][VEC],
                  float (&rsl)[ROWS]) {
    const uint4 zero = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const long long row = row0 + r;
      const bool in = row < rows;
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        const long long at = row * nvec + t + v * threads;
        xl[r][v] = in ? reinterpret_cast<const uint4*>(x)[at] : zero;
        gl[r][v] = in ? reinterpret_cast<const uint4*>(dy)[at] : zero;
        rl[r][v] = in && dres ? reinterpret_cast<const uint4*>(dres)[at] : zero;
      }
      rsl[r] = in ? rstd_in[row] : 0.f;
    }
  };
  const long long step = (long long)gridDim.x * ROWS;
  int parity = 0;
  if constexpr (AHEAD) load((long long)blockIdx.x * ROWS, xc, gc, rc, rs);
  for (long long row0 = (long long)blockIdx.x * ROWS; row0 < rows; row0 += step, parity ^= 1) {
    uint4 xn[ROWS][VEC], gn[ROWS][VEC], rn[ROWS][VEC];
    float rsn[ROWS];
    if constexpr (AHEAD)
      load(row0 + step, xn, gn, rn, rsn);
    else
      load(row0, xc, gc, rc, rs);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      float d = 0.f;
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        float f[8], g[8];
        unpack8(xc[r][v], f);
        unpack8(gc[r][v], g);
#pragma unroll
        for (int i = 0; i < 8; ++i) d += g[i] * wv[v][i] * f[i];
      }
      d = warp_sum(d * rs[r]);
      if (lane == 0) red[parity][r][warp] = d;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const float dot = warp_sum(lane < warps ? red[parity][r][lane] : 0.f) * inv_h;
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        float f[8], g[8], b[8], o[8];
        unpack8(xc[r][v], f);
        unpack8(gc[r][v], g);
        unpack8(rc[r][v], b);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float xhat = f[i] * rs[r];
          o[i] = rs[r] * (g[i] * wv[v][i] - xhat * dot) + b[i];
          acc[v][i] += g[i] * xhat;
        }
        if (row0 + r < rows) reinterpret_cast<uint4*>(dx)[(row0 + r) * nvec + t + v * threads] = pack8(o);
      }
    }
    if constexpr (AHEAD) {
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
          xc[r][v] = xn[r][v];
          gc[r][v] = gn[r][v];
          rc[r][v] = rn[r][v];
        }
        rs[r] = rsn[r];
      }
    }
  }
  // dw: columns in order through shared memory, so that a warp's request covers 512 contiguous bytes (a thread's own
  // eight columns at a time touched 32 sectors a request, and same-sector adds of hundreds of blocks queue up)
#pragma unroll
  for (int v = 0; v < VEC; ++v)
#pragma unroll
    for (int i = 0; i < 2; ++i)
      reinterpret_cast<float4*>(dw_smem)[(t + v * threads) * 2 + i] =
          make_float4(acc[v][4 * i], acc[v][4 * i + 1], acc[v][4 * i + 2], acc[v][4 * i + 3]);
  __syncthreads();
  // dw may start anywhere in an arena: the elements up to the next 16 bytes and the last of the row by themselves
  const int head = (4 - static_cast<int>((reinterpret_cast<uintptr_t>(dw) >> 2) & 3)) & 3;
  for (int j = head + 4 * t; j + 4 <= H; j += 4 * threads) {
    const float* v = dw_smem + j;
    red_add4(dw + j, head ? make_float4(v[0], v[1], v[2], v[3]) : *reinterpret_cast<const float4*>(v));
  }
  if (head && t < 4) {
    const int i = t < head ? t : H - 4 + t;
    atomicAdd(dw + i, dw_smem[i]);
  }
}

// ------------------------------------------------------------------------------------------------
// QK-RMSNorm + RoPE (interleaved pairs) over the head dimension.  One warp handles one (token, head)
// vector of D elements (D % 8 == 0, D <= 256): lane l owns elements [8l, 8l+8) = 4 rotation pairs.
// in : [tokens, in_stride] with heads at column h*D;   out: [tokens, out_stride]
// w  : [D] fp32 norm scale or nullptr (no norm).  positions: [tokens] int32.  rope: 0 = skip rotation.
// Angle of pair i at position p: p * theta^(-2i/D).
// ------------------------------------------------------------------------------------------------
// sin and cos of an angle of any size: Cody-Waite reduction by 2*pi to [-pi, pi], then the special-function unit
__device__ __forceinline__ void sincos_reduced(float x, float* s, float* c) {
  const float k = rintf(x * 0.15915494309189535f);
  x = fmaf(k, -6.28318548202514648f, x);
  x = fmaf(k, 1.74845553e-7f, x);
  __sincosf(x, s, c);
}

// A head of D <= 256 elements is handled by LPH lanes (a power of two, 8 elements per lane), so a warp works on
// HPW = 32 / LPH heads at once; reductions stay inside the lane group.
//
// A block works on query heads or on key heads only, so one norm scale and one scale gradient live in registers; the
// first `blocks_first` blocks take the query heads.  A warp takes one token (or, when there are too few tokens to fill
// the device, a chunk of a token's heads) and walks its heads HPW at a time.  The angles of a token are the same for
// all of its heads: sine and cosine are computed once per token and lane.  The loads of BATCH groups of heads are
// issued before the first is used.  What bounds it: memory latency and traffic (one read and one write of the q and k
// columns forward, two reads and one write backward).  One warp per (token, two heads), with the angles and a 64-bit
// division for every head, was bound by instruction issue: 32768 tokens of 16 + 8 heads of 128 took 144 us forward and
// 390 us backward where this takes 87 us and 129 us (4.6 TB/s).
// Blocks per SM: 2 forward loads a lane and 64 registers beat 4 loads (88 us) and 80 or 48 registers (111 us at 48, which
// spills); backward 4 pairs of loads and 128 registers beat 2 pairs (139 us) and 80 registers (211 us, spills).
constexpr int kQkFwdBlocks = 4, kQkBwdBlocks = 2;

template <int LPH>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int off = LPH >> 1; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

struct QkShape {
  long long tokens;
  int heads, heads_first, D;  // heads [0, heads_first) take the first norm scale, the rest the second
  int blocks_first;           // blocks that work on the first kind of heads
  int per_chunk;              // groups of HPW heads that a warp takes of a token
  float log2_theta;
  int rope;
};

// What one block walks: heads [h0, h1) of all tokens, dealt to the warps of blocks `block` of `blocks`.
template <int LPH>
struct QkWalk {
  int h0, h1, units, chunks;
  long long item, items, step;
  __device__ __forceinline__ QkWalk(const QkShape& q, bool first) {
    constexpr int HPW = 32 / LPH;
    h0 = first ? 0 : q.heads_first;
    h1 = first ? q.heads_first : q.heads;
    units = (h1 - h0 + HPW - 1) / HPW;
    chunks = (units + q.per_chunk - 1) / q.per_chunk;
    items = q.tokens * chunks;
    const int block = first ? blockIdx.x : blockIdx.x - q.blocks_first;
    const int blocks = first ? q.blocks_first : gridDim.x - q.blocks_first;
    item = (long long)block * kWarpsPerBlock + (threadIdx.x >> 5);
    step = (long long)blocks * kWarpsPerBlock;
  }
  __device__ __forceinline__ long long at(const QkShape& q, int& u0, int& u1) const {
    if (chunks == 1) {
      u0 = 0;
      u1 = units;
      return item;
    }
    const long long t = item / chunks;
    u0 = (int)(item - t * chunks) * q.per_chunk;
    u1 = min(u0 + q.per_chunk, units);
    return t;
  }
};

__device__ __forceinline__ void qk_angles(const QkShape& q, const int* positions, long long t,
                                          const float (&inv_freq)[4], float (&sn)[4], float (&cs)[4]) {
  const float pos = (float)positions[t];
#pragma unroll
  for (int i = 0; i < 4; ++i) sincos_reduced(pos * inv_freq[i], &sn[i], &cs[i]);
}

template <int LPH, typename W>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, kQkFwdBlocks)
qknorm_rope_fwd_kernel(const __nv_bfloat16* __restrict__ in, long long in_stride, __nv_bfloat16* __restrict__ out,
                       long long out_stride, const W* w_first, const W* w_rest, const int* __restrict__ positions,
                       float* __restrict__ rstd_out, const QkShape q, float eps) {
  constexpr int HPW = 32 / LPH, BATCH = 2;
  const int lane = threadIdx.x & 31;
  const int sub = lane / LPH, l = lane % LPH;
  const bool has_cols = l * 8 < q.D;
  const bool first = (int)blockIdx.x < q.blocks_first;
  const W* w = first ? w_first : w_rest;
  const bool norm = w != nullptr;
  float inv_freq[4], wv[8] = {1, 1, 1, 1, 1, 1, 1, 1};
#pragma unroll
  for (int i = 0; i < 4; ++i) inv_freq[i] = exp2f(-q.log2_theta * (2.f * (float)(l * 4 + i)) / (float)q.D);
  b200::pdl_launch_dependents();   // no-ops unless launched as a dependent (decode steps)
  b200::pdl_wait();
  if (norm && has_cols) load8w(w + l * 8, wv);   // no __restrict__: a load that may not move above the wait
  for (QkWalk<LPH> k(q, first); k.item < k.items; k.item += k.step) {
    int u0, u1;
    const long long t = k.at(q, u0, u1);
    float sn[4] = {0, 0, 0, 0}, cs[4] = {1, 1, 1, 1};
    if (q.rope) qk_angles(q, positions, t, inv_freq, sn, cs);
    const __nv_bfloat16* src = in + t * in_stride + l * 8;
    __nv_bfloat16* dst = out + t * out_stride + l * 8;
#pragma unroll 1
    for (int u = u0; u < u1; u += BATCH) {
      uint4 raw[BATCH];
#pragma unroll
      for (int j = 0; j < BATCH; ++j) {
        const int h = k.h0 + (u + j) * HPW + sub;
        raw[j] = make_uint4(0, 0, 0, 0);
        if (u + j < u1 && has_cols && h < k.h1) raw[j] = *reinterpret_cast<const uint4*>(src + h * q.D);
      }
#pragma unroll
      for (int j = 0; j < BATCH; ++j) {
        if (u + j >= u1) break;
        const int h = k.h0 + (u + j) * HPW + sub;
        float f[8];
        unpack8(raw[j], f);
        if (norm) {
          float ss = 0.f;
#pragma unroll
          for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
          ss = group_sum<LPH>(ss);
          const float rstd = rsqrtf(ss / (float)q.D + eps);
          if (l == 0 && rstd_out && h < k.h1) rstd_out[t * q.heads + h] = rstd;
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] = f[i] * rstd * wv[i];
        }
        if (q.rope) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float x = f[2 * i], y = f[2 * i + 1];
            f[2 * i] = x * cs[i] - y * sn[i];
            f[2 * i + 1] = x * sn[i] + y * cs[i];
          }
        }
        if (has_cols && h < k.h1) *reinterpret_cast<uint4*>(dst + h * q.D) = pack8(f);
      }
    }
  }
}

// backward of the above: gradient of the pre-norm input, and of the scales (atomic fp32 adds, D columns).  `dout` and
// `din` may be the same buffer: a lane reads its elements of a head before it writes them, and no other lane does.
template <int LPH, typename W>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, kQkBwdBlocks)
qknorm_rope_bwd_kernel(const __nv_bfloat16* __restrict__ in, long long in_stride, const __nv_bfloat16* dout,
                       long long dout_stride, __nv_bfloat16* din, long long din_stride,
                       const W* __restrict__ w_first, const W* __restrict__ w_rest, const int* __restrict__ positions,
                       const float* __restrict__ rstd_in, float* __restrict__ dw_first, float* __restrict__ dw_rest,
                       const QkShape q) {
  constexpr int HPW = 32 / LPH, BATCH = 4;
  __shared__ float dw_smem[256];
  const int lane = threadIdx.x & 31;
  const int sub = lane / LPH, l = lane % LPH;
  const bool has_cols = l * 8 < q.D;
  const bool first = (int)blockIdx.x < q.blocks_first;
  const W* w = first ? w_first : w_rest;
  float* dw = first ? dw_first : dw_rest;
  const bool norm = w != nullptr;
  dw_smem[threadIdx.x] = 0.f;
  __syncthreads();
  float inv_freq[4], wv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < 4; ++i) inv_freq[i] = exp2f(-q.log2_theta * (2.f * (float)(l * 4 + i)) / (float)q.D);
  if (norm && has_cols) load8w(w + l * 8, wv);
  const float inv_d = 1.f / (float)q.D;
  float dw_acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (QkWalk<LPH> k(q, first); k.item < k.items; k.item += k.step) {
    int u0, u1;
    const long long t = k.at(q, u0, u1);
    float sn[4] = {0, 0, 0, 0}, cs[4] = {1, 1, 1, 1};
    if (q.rope) qk_angles(q, positions, t, inv_freq, sn, cs);
    const __nv_bfloat16* xsrc = in + t * in_stride + l * 8;
    const __nv_bfloat16* gsrc = dout + t * dout_stride + l * 8;
    __nv_bfloat16* dst = din + t * din_stride + l * 8;
    const float* rstds = rstd_in + t * q.heads;
#pragma unroll 1
    for (int u = u0; u < u1; u += BATCH) {
      uint4 graw[BATCH], xraw[BATCH];
      float rstd[BATCH];
#pragma unroll
      for (int j = 0; j < BATCH; ++j) {
        const int h = k.h0 + (u + j) * HPW + sub;
        const bool valid = u + j < u1 && h < k.h1;
        graw[j] = xraw[j] = make_uint4(0, 0, 0, 0);
        rstd[j] = 0.f;
        if (valid && has_cols) graw[j] = *reinterpret_cast<const uint4*>(gsrc + h * q.D);
        if (norm && valid) {
          if (has_cols) xraw[j] = *reinterpret_cast<const uint4*>(xsrc + h * q.D);
          rstd[j] = rstds[h];
        }
      }
#pragma unroll
      for (int j = 0; j < BATCH; ++j) {
        if (u + j >= u1) break;
        const int h = k.h0 + (u + j) * HPW + sub;
        float g[8];
        unpack8(graw[j], g);
        if (q.rope) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float x = g[2 * i], y = g[2 * i + 1];  // transpose of the rotation
            g[2 * i] = x * cs[i] + y * sn[i];
            g[2 * i + 1] = -x * sn[i] + y * cs[i];
          }
        }
        if (norm) {
          float f[8];
          unpack8(xraw[j], f);
          float dot = 0.f;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            f[i] *= rstd[j];
            dot += g[i] * wv[i] * f[i];
          }
          dot = group_sum<LPH>(dot) * inv_d;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            dw_acc[i] += g[i] * f[i];
            g[i] = rstd[j] * (g[i] * wv[i] - f[i] * dot);
          }
        }
        if (has_cols && h < k.h1) *reinterpret_cast<uint4*>(dst + h * q.D) = pack8(g);
      }
    }
  }
  if (norm && dw) {
    if (has_cols) {
#pragma unroll
      for (int i = 0; i < 8; ++i) atomicAdd(&dw_smem[l * 8 + i], dw_acc[i]);
    }
    __syncthreads();
    if (threadIdx.x < q.D) atomicAdd(&dw[threadIdx.x], dw_smem[threadIdx.x]);
  }
}

// ------------------------------------------------------------------------------------------------
// SwiGLU on a fused [rows, 2*I] gate|up buffer: h = silu(g) * u.
// ------------------------------------------------------------------------------------------------
// sigmoid through the hardware tanh (one special-function op instead of an exponential and a reciprocal; 11 good
// bits, more than a bf16 result keeps): sigmoid(x) = 0.5 + 0.5 tanh(x / 2)
__device__ __forceinline__ float sigmoid_fast(float x) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * x));
  return fmaf(0.5f, t, 0.5f);
}

// Rows and vectors are walked with 32-bit arithmetic (the launchers check that rows * I / 8 fits); a 64-bit divide
// per thread and the two special-function ops per element used to make these kernels issue-bound.
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ h, long long rows,
                                  int I) {
  const unsigned nvec = (unsigned)I >> 3;
  const unsigned total = (unsigned)rows * nvec;
  b200::pdl_launch_dependents();
  b200::pdl_wait();
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const unsigned r = i / nvec;
    const unsigned v = i - r * nvec;
    const __nv_bfloat16* base = gu + (long long)r * 2 * I;
    float g[8], u[8], o[8];
    unpack8(*reinterpret_cast<const uint4*>(base + v * 8), g);
    unpack8(*reinterpret_cast<const uint4*>(base + I + v * 8), u);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = g[k] * sigmoid_fast(g[k]) * u[k];
    *reinterpret_cast<uint4*>(h + (long long)r * I + v * 8) = pack8(o);
  }
}
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ dh,
                                  __nv_bfloat16* __restrict__ dgu, long long rows, int I) {
  const unsigned nvec = (unsigned)I >> 3;
  const unsigned total = (unsigned)rows * nvec;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const unsigned r = i / nvec;
    const unsigned v = i - r * nvec;
    const __nv_bfloat16* base = gu + (long long)r * 2 * I;
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(*reinterpret_cast<const uint4*>(base + v * 8), g);
    unpack8(*reinterpret_cast<const uint4*>(base + I + v * 8), u);
    unpack8(*reinterpret_cast<const uint4*>(dh + (long long)r * I + v * 8), d);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float sig = sigmoid_fast(g[k]);
      const float silu = g[k] * sig;
      du[k] = d[k] * silu;
      dg[k] = d[k] * u[k] * (sig + silu * (1.f - sig));
    }
    *reinterpret_cast<uint4*>(dgu + (long long)r * 2 * I + v * 8) = pack8(dg);
    *reinterpret_cast<uint4*>(dgu + (long long)r * 2 * I + I + v * 8) = pack8(du);
  }
}

// out = a * sigmoid(gate) (attention output gate) and its backward
__global__ void sigmoid_gate_fwd_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ gate,
                                        __nv_bfloat16* __restrict__ out, long long nvec) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    float x[8], g[8];
    unpack8(reinterpret_cast<const uint4*>(a)[i], x);
    unpack8(reinterpret_cast<const uint4*>(gate)[i], g);
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = x[k] * sigmoid_fast(g[k]);
    reinterpret_cast<uint4*>(out)[i] = pack8(x);
  }
}
__global__ void sigmoid_gate_bwd_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ gate,
                                        const __nv_bfloat16* __restrict__ dout, __nv_bfloat16* __restrict__ da,
                                        __nv_bfloat16* __restrict__ dgate, long long nvec) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    float x[8], g[8], d[8], o1[8], o2[8];
    unpack8(reinterpret_cast<const uint4*>(a)[i], x);
    unpack8(reinterpret_cast<const uint4*>(gate)[i], g);
    unpack8(reinterpret_cast<const uint4*>(dout)[i], d);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float sig = sigmoid_fast(g[k]);
      o1[k] = d[k] * sig;
      o2[k] = d[k] * x[k] * sig * (1.f - sig);
    }
    reinterpret_cast<uint4*>(da)[i] = pack8(o1);
    reinterpret_cast<uint4*>(dgate)[i] = pack8(o2);
  }
}

// ------------------------------------------------------------------------------------------------
// kv-side view of a per-query lower bound: hi[b][k] = offset + (number of q with lo[b][q] <= k) - 1, lo non-decreasing
// along S.  A thread searches one k; neighbours walk the same path, so all but the last steps hit L1.  One launch where
// an index range, a search, two additions and a conversion in tensor operators took five and 17 us of device time.
// ------------------------------------------------------------------------------------------------
__global__ void kv_upper_bound_kernel(const int* __restrict__ lo, int* __restrict__ hi, int S, int n, int offset) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int* row = lo + (long long)blockIdx.y * S;
  int a = 0, b = S;   // lo[q] <= k for q < a, lo[q] > k for q >= b
  while (a < b) {
    const int mid = (a + b) >> 1;
    if (row[mid] <= k)
      a = mid + 1;
    else
      b = mid;
  }
  hi[(long long)blockIdx.y * n + k] = a - 1 + offset;
}

// ------------------------------------------------------------------------------------------------
// Embedding gather (bf16 table) with optional scale, and scatter-add of gradients into fp32.
// ------------------------------------------------------------------------------------------------
__global__ void embedding_fwd_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ table,
                                     __nv_bfloat16* __restrict__ out, long long tokens, int H, float scale) {
  const int nvec = H >> 3;
  const long long total = tokens * nvec;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / nvec;
    const int v = (int)(i - t * nvec);
    uint4 val = *reinterpret_cast<const uint4*>(table + (long long)ids[t] * H + v * 8);
    if (scale != 1.f) {
      float f[8];
      unpack8(val, f);
#pragma unroll
      for (int k = 0; k < 8; ++k) f[k] *= scale;
      val = pack8(f);
    }
    *reinterpret_cast<uint4*>(out + t * H + v * 8) = val;
  }
}
__global__ void embedding_bwd_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ dout,
                                     float* __restrict__ dtable, long long tokens, int H, float scale) {
  const int nvec = H >> 3;
  const long long total = tokens * nvec;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / nvec;
    const int v = (int)(i - t * nvec);
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(dout + t * H + v * 8), f);
    float* dst = dtable + (long long)ids[t] * H + v * 8;
#pragma unroll
    for (int k = 0; k < 8; ++k) atomicAdd(dst + k, f[k] * scale);
  }
}

// ------------------------------------------------------------------------------------------------
// Masked cross-entropy + z-loss over one chunk of logits [rows, V] (bf16, row stride ld), in place:
//   loss_i = lse_i - logit_i[target_i];  z_i = lse_i^2            (only rows with mask != 0 count)
//   logits <- dlogits = grad_scale * mask_i * ((1 + 2 z_w lse_i) softmax - onehot)
// One block per row; three passes over the row (max, sum, write); the row stays in L1/L2.
// Sums are written per row (loss_row, z_row) so that the host-visible reduction is deterministic.
// vocab_offset/vocab_total support vocab-parallel logits: then max and sum come in precomputed
// (global_max / global_sum per row) and phase selects which pass runs.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(512)
ce_fwd_bwd_kernel(__nv_bfloat16* __restrict__ logits, long long ld, const int* __restrict__ targets,
                  const uint8_t* __restrict__ mask, float* __restrict__ loss_row, float* __restrict__ z_row,
                  float* __restrict__ lse_row, int V, float grad_scale, float z_weight, int write_grad) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  __nv_bfloat16* lr = logits + row * ld;
  const int nvec = V >> 3;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const bool masked = mask[row] == 0;
  if (masked && !write_grad) {
    if (threadIdx.x == 0) { loss_row[row] = 0.f; z_row[row] = 0.f; if (lse_row) lse_row[row] = 0.f; }
    return;
  }
  if (masked) {  // zero gradient row, no loss
    const uint4 z = make_uint4(0, 0, 0, 0);
    for (int v = threadIdx.x; v < nvec; v += blockDim.x) reinterpret_cast<uint4*>(lr)[v] = z;
    for (int c = nvec * 8 + threadIdx.x; c < V; c += blockDim.x) lr[c] = __float2bfloat16(0.f);
    if (threadIdx.x == 0) { loss_row[row] = 0.f; z_row[row] = 0.f; if (lse_row) lse_row[row] = 0.f; }
    return;
  }
  // pass 1: max
  float m = -INFINITY;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    float f[8];
    unpack8(reinterpret_cast<const uint4*>(lr)[v], f);
#pragma unroll
    for (int k = 0; k < 8; ++k) m = fmaxf(m, f[k]);
  }
  for (int c = nvec * 8 + threadIdx.x; c < V; c += blockDim.x) m = fmaxf(m, __bfloat162float(lr[c]));
  m = warp_max(m);
  if (lane == 0) red[warp] = m;
  __syncthreads();
  m = (lane < nwarps) ? red[lane] : -INFINITY;
  m = warp_max(m);
  __syncthreads();
  // pass 2: sum exp
  float s = 0.f;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    float f[8];
    unpack8(reinterpret_cast<const uint4*>(lr)[v], f);
#pragma unroll
    for (int k = 0; k < 8; ++k) s += __expf(f[k] - m);
  }
  for (int c = nvec * 8 + threadIdx.x; c < V; c += blockDim.x) s += __expf(__bfloat162float(lr[c]) - m);
  s = warp_sum(s);
  if (lane == 0) red[warp] = s;
  __syncthreads();
  s = (lane < nwarps) ? red[lane] : 0.f;
  s = warp_sum(s);
  const float lse = m + logf(s);
  const int tgt = targets[row];
  const float tl = __bfloat162float(lr[tgt]);
  __syncthreads();  // everyone has read the target logit before it is overwritten
  if (threadIdx.x == 0) {
    loss_row[row] = lse - tl;
    z_row[row] = lse * lse;
    if (lse_row) lse_row[row] = lse;
  }
  if (!write_grad) return;
  // pass 3: gradient in place
  const float coef = grad_scale * (1.f + 2.f * z_weight * lse);
  const float inv_s = 1.f / s;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    float f[8];
    unpack8(reinterpret_cast<const uint4*>(lr)[v], f);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      f[k] = coef * __expf(f[k] - m) * inv_s;
      if (v * 8 + k == tgt) f[k] -= grad_scale;
    }
    reinterpret_cast<uint4*>(lr)[v] = pack8(f);
  }
  for (int c = nvec * 8 + threadIdx.x; c < V; c += blockDim.x) {
    float g = coef * __expf(__bfloat162float(lr[c]) - m) * inv_s;
    if (c == tgt) g -= grad_scale;
    lr[c] = __float2bfloat16(g);
  }
}

// The same op with the row staged in shared memory: one bulk copy in, three passes over shared memory, one bulk
// copy out, so the logits cross the memory system once in each direction and two or three rows per SM overlap
// their phases.  V % 8 == 0 and 2 V bytes of dynamic shared memory; 16-byte aligned rows.
constexpr int kCeThreads = 512;
constexpr uint32_t kCeChunkBytes = 32768;
__global__ void __launch_bounds__(kCeThreads)
ce_fwd_bwd_staged_kernel(__nv_bfloat16* __restrict__ logits, long long ld, const int* __restrict__ targets,
                         const uint8_t* __restrict__ mask, float* __restrict__ loss_row, float* __restrict__ z_row,
                         float* __restrict__ lse_row, int V, float grad_scale, float z_weight, int write_grad,
                         int* __restrict__ status) {
  extern __shared__ __align__(128) unsigned char ce_row_smem[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ float red[2][32];
  __shared__ int abort_flag;
  const long long row = blockIdx.x;
  __nv_bfloat16* grow = logits + row * ld;
  uint4* srow = reinterpret_cast<uint4*>(ce_row_smem);
  const int nvec = V >> 3;
  const uint32_t bytes = (uint32_t)V * 2u;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (mask[row] == 0) {
    if (write_grad) {
      const uint4 z = make_uint4(0, 0, 0, 0);
      for (int v = threadIdx.x; v < nvec; v += kCeThreads) reinterpret_cast<uint4*>(grow)[v] = z;
    }
    if (threadIdx.x == 0) { loss_row[row] = 0.f; z_row[row] = 0.f; if (lse_row) lse_row[row] = 0.f; }
    return;
  }
  if (threadIdx.x == 0) {
    abort_flag = 0;
    b200::mbar_init(&bar, 1);
    b200::mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    b200::mbar_expect_tx(&bar, bytes);
    for (uint32_t off = 0; off < bytes; off += kCeChunkBytes)
      b200::bulk_g2s(ce_row_smem + off, reinterpret_cast<const unsigned char*>(grow) + off,
                     min(kCeChunkBytes, bytes - off), &bar);
  }
  const b200::AbortCtx ab{&abort_flag, status};
  const bool ok = b200::mbar_wait(&bar, 0, ab, b200::ERR_WAIT_FULL);
  if (!__syncthreads_and(ok)) {
    // the limit ran out (recorded in the status word): give the copies still in flight one more bounded wait so
    // that they do not land in shared memory of a CTA that has left, then leave without writing anything
    if (threadIdx.x == 0) {
      const uint64_t t0 = b200::globaltimer_ns();
      while (!b200::mbar_try_wait(&bar, 0) && b200::globaltimer_ns() - t0 < b200::kWaitLimitNs) {}
    }
    __syncthreads();
    return;
  }
  const int tgt = targets[row];
  const float tl = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(ce_row_smem)[tgt]);
  // pass 1: the maximum, on packed pairs (no conversion to fp32: bf16 compares exactly)
  __nv_bfloat162 m2v = __float2bfloat162_rn(-INFINITY);
  for (int v = threadIdx.x; v < nvec; v += kCeThreads) {
    const uint4 q = srow[v];
    m2v = __hmax2(m2v, *reinterpret_cast<const __nv_bfloat162*>(&q.x));
    m2v = __hmax2(m2v, *reinterpret_cast<const __nv_bfloat162*>(&q.y));
    m2v = __hmax2(m2v, *reinterpret_cast<const __nv_bfloat162*>(&q.z));
    m2v = __hmax2(m2v, *reinterpret_cast<const __nv_bfloat162*>(&q.w));
  }
  float m = fmaxf(__low2float(m2v), __high2float(m2v));
  m = warp_max(m);
  if (lane == 0) red[0][warp] = m;
  __syncthreads();
  m = warp_max(red[0][lane & (kCeThreads / 32 - 1)]);
  constexpr float kLog2e = 1.4426950408889634f;
  const float m2 = m * kLog2e;
  float s = 0.f;
  for (int v = threadIdx.x; v < nvec; v += kCeThreads) {
    float f[8];
    unpack8(srow[v], f);
#pragma unroll
    for (int k = 0; k < 8; ++k) s += b200::ex2_approx(fmaf(f[k], kLog2e, -m2));
  }
  s = warp_sum(s);
  if (lane == 0) red[1][warp] = s;
  __syncthreads();
  s = warp_sum(lane < kCeThreads / 32 ? red[1][lane] : 0.f);
  const float lse = m + logf(s);
  if (threadIdx.x == 0) {
    loss_row[row] = lse - tl;
    z_row[row] = lse * lse;
    if (lse_row) lse_row[row] = lse;
  }
  if (!write_grad) return;
  const float coef = grad_scale * (1.f + 2.f * z_weight * lse) / s;
  for (int v = threadIdx.x; v < nvec; v += kCeThreads) {
    float f[8];
    unpack8(srow[v], f);
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] = coef * b200::ex2_approx(fmaf(f[k], kLog2e, -m2));
    const int off = tgt - v * 8;
    if (off >= 0 && off < 8) {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k == off) f[k] -= grad_scale;
    }
    srow[v] = pack8(f);
  }
  b200::fence_proxy_async_smem();      // the generic-proxy writes above are read by the bulk store below
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t off = 0; off < bytes; off += kCeChunkBytes)
      b200::bulk_s2g(reinterpret_cast<unsigned char*>(grow) + off, ce_row_smem + off, min(kCeChunkBytes, bytes - off));
    b200::tma_commit_group();
    b200::tma_wait_group_read<0>();    // shared memory stays valid until the store has read it
  }
}

// ------------------------------------------------------------------------------------------------
// Flat-arena AdamW: p, m, v fp32 [n]; g bf16 or fp32 [n]; writes the bf16 shadow of p.
//   g' = g * gscale[0] (clip factor, device scalar; nullptr = 1)
//   m = b1 m + (1-b1) g';  v = b2 v + (1-b2) g'^2;  p -= lr * (mhat / (sqrt(vhat) + eps) + wd p)
// lr, bias corrections come from the host each step (schedule evaluated at the old step count).
// ------------------------------------------------------------------------------------------------
template <typename GT>
__global__ void adamw_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                             const GT* __restrict__ g, __nv_bfloat16* __restrict__ shadow,
                             const float* __restrict__ gscale, long long n, float lr, float b1, float b2, float eps,
                             float wd, float bc1, float bc2) {
  const float gs = gscale ? gscale[0] : 1.f;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float gi;
    if constexpr (sizeof(GT) == 2)
      gi = __bfloat162float(g[i]) * gs;
    else
      gi = g[i] * gs;
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float mhat = mi / bc1;
    const float vhat = vi / bc2;
    float pi = p[i];
    pi -= lr * (mhat / (sqrtf(vhat) + eps) + wd * pi);
    p[i] = pi;
    if (shadow) shadow[i] = __float2bfloat16(pi);
  }
}

// Four elements per thread with 16-byte accesses (n % 4 == 0, 16-byte aligned arenas).
template <typename GT>
__global__ void __launch_bounds__(256)
adamw_vec4_kernel(float4* __restrict__ p, float4* __restrict__ m, float4* __restrict__ v, const GT* __restrict__ g,
                  __nv_bfloat16* __restrict__ shadow, const float* __restrict__ gscale, long long nvec, float lr,
                  float b1, float b2, float eps, float wd, float bc1, float bc2) {
  const float gs = gscale ? gscale[0] : 1.f;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec;
       i += (long long)gridDim.x * blockDim.x) {
    float gi[4];
    if constexpr (sizeof(GT) == 2) {
      const uint2 raw = reinterpret_cast<const uint2*>(g)[i];
      const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
      const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
      gi[0] = a.x; gi[1] = a.y; gi[2] = b.x; gi[3] = b.y;
    } else {
      const float4 raw = reinterpret_cast<const float4*>(g)[i];
      gi[0] = raw.x; gi[1] = raw.y; gi[2] = raw.z; gi[3] = raw.w;
    }
    const float4 m4 = m[i], v4 = v[i], p4 = p[i];
    float mi[4] = {m4.x, m4.y, m4.z, m4.w}, vi[4] = {v4.x, v4.y, v4.z, v4.w}, pi[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float gk = gi[k] * gs;
      mi[k] = b1 * mi[k] + (1.f - b1) * gk;
      vi[k] = b2 * vi[k] + (1.f - b2) * gk * gk;
      const float mhat = mi[k] / bc1;
      const float vhat = vi[k] / bc2;
      pi[k] -= lr * (mhat / (sqrtf(vhat) + eps) + wd * pi[k]);
    }
    m[i] = make_float4(mi[0], mi[1], mi[2], mi[3]);
    v[i] = make_float4(vi[0], vi[1], vi[2], vi[3]);
    p[i] = make_float4(pi[0], pi[1], pi[2], pi[3]);
    if (shadow) {
      __nv_bfloat162 lo = __floats2bfloat162_rn(pi[0], pi[1]);
      __nv_bfloat162 hi = __floats2bfloat162_rn(pi[2], pi[3]);
      uint2 pk;
      pk.x = *reinterpret_cast<uint32_t*>(&lo);
      pk.y = *reinterpret_cast<uint32_t*>(&hi);
      reinterpret_cast<uint2*>(shadow)[i] = pk;
    }
  }
}

// sum of squares, two deterministic stages: per-block partials, then one block folds them
template <typename T>
__global__ void sumsq_partial_kernel(const T* __restrict__ x, long long n, float* __restrict__ partial) {
  __shared__ float red[32];
  float s = 0.f;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float f;
    if constexpr (sizeof(T) == 2)
      f = __bfloat162float(x[i]);
    else
      f = x[i];
    s += f * f;
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    s = warp_sum(s);
    if (threadIdx.x == 0) partial[blockIdx.x] = s;
  }
}
__global__ void sumsq_final_kernel(const float* __restrict__ partial, int nparts, float* __restrict__ out,
                                   int accumulate) {
  __shared__ float red[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) s += partial[i];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    s = warp_sum(s);
    if (threadIdx.x == 0) out[0] = accumulate ? out[0] + s : s;
  }
}

// fp32 -> bf16 cast with scale (used for the bf16 shadow of Muon-updated weights and grad casts)
__global__ void cast_f32_bf16_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, long long n,
                                     float scale) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16(x[i] * scale);
}

inline int grid_for(long long work_items, int block, int per_sm = 8) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  long long blocks = (work_items + block - 1) / block;
  long long cap = (long long)sms * per_sm;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

}  // namespace

#define STREAM(s) reinterpret_cast<cudaStream_t>(s)
#define LAST_ERR() static_cast<int>(cudaGetLastError())

template <typename W>
static int rmsnorm_fwd_launch(const void* x, const void* delta, const W* w, void* res_out, void* y, void* rstd, int rows,
                              int H, float eps, void* stream) {
  if (rows > 0 && rows <= 512) {
    // few rows = a decode step: launched as a dependent so that it is resident when its predecessor ends
    return static_cast<int>(b200host::launch_kernel(
        rmsnorm_fwd_row_kernel<W>, dim3(rows), dim3(256), 0, STREAM(stream), b200host::pdl_enabled() != 0,
        (const __nv_bfloat16*)x, (const __nv_bfloat16*)delta, w, (__nv_bfloat16*)res_out, (__nv_bfloat16*)y,
        (float*)rstd, H, eps));
  }
  const int grid = grid_for((long long)rows, kWarpsPerBlock, 8);
#define RMS_FWD(NV)                                                                                         \
  rmsnorm_fwd_reg_kernel<NV, W><<<grid, kWarpsPerBlock * 32, 0, STREAM(stream)>>>(                          \
      (const __nv_bfloat16*)x, (const __nv_bfloat16*)delta, w, (__nv_bfloat16*)res_out, (__nv_bfloat16*)y,  \
      (float*)rstd, rows, eps);                                                                             \
  return LAST_ERR()
  switch (H) {
    case 1024: RMS_FWD(4);
    case 2048: RMS_FWD(8);
    case 4096: RMS_FWD(16);
    default: break;
  }
#undef RMS_FWD
  rmsnorm_fwd_kernel<W><<<grid, kWarpsPerBlock * 32, 0, STREAM(stream)>>>(
      (const __nv_bfloat16*)x, (const __nv_bfloat16*)delta, w, (__nv_bfloat16*)res_out, (__nv_bfloat16*)y,
      (float*)rstd, rows, H, eps);
  return LAST_ERR();
}
extern "C" int b200_rmsnorm_fwd(const void* x, const void* delta, const void* w, int w_bf16, void* res_out, void* y,
                                void* rstd, int rows, int H, float eps, void* stream) {
  if (H % 8) return -2;
  if (w_bf16)
    return rmsnorm_fwd_launch(x, delta, (const __nv_bfloat16*)w, res_out, y, rstd, rows, H, eps, stream);
  return rmsnorm_fwd_launch(x, delta, (const float*)w, res_out, y, rstd, rows, H, eps, stream);
}
template <typename W>
static int rmsnorm_bwd_launch(const void* x, const W* w, const void* rstd, const void* dy, const void* dres, void* dx,
                              void* dw, int rows, int H, void* stream) {
#define RMS_BWD_COLS(VEC, ROWS, THREADS, MAXT, MINB, AHEAD)                                                           \
  do {                                                                                                                \
    rmsnorm_bwd_cols_kernel<VEC, ROWS, MAXT, MINB, AHEAD, W>                                                          \
        <<<grid_for(((long long)rows + ROWS - 1) / ROWS, 1, MINB * (MAXT / (THREADS))), THREADS, H * sizeof(float),   \
           STREAM(stream)>>>(                                                                                         \
            (const __nv_bfloat16*)x, w, (const float*)rstd, (const __nv_bfloat16*)dy, (const __nv_bfloat16*)dres,     \
            (__nv_bfloat16*)dx, (float*)dw, rows, H);                                                                 \
    return LAST_ERR();                                                                                                \
  } while (0)
  // whole warps of columns: one 16-byte vector of a row per thread up to 2048 columns, two above
  if (H % 256 == 0 && H <= 512) RMS_BWD_COLS(1, 4, H / 8, 64, 8, false);
  if (H % 256 == 0 && H <= 2048) RMS_BWD_COLS(1, 2, H / 8, 256, 4, false);
  if (H % 512 == 0 && H <= 4096) RMS_BWD_COLS(2, 1, H / 16, 256, 3, false);
  if (H % 512 == 0 && H <= 8192) RMS_BWD_COLS(2, 1, H / 16, 512, 1, true);
#undef RMS_BWD_COLS
  const int grid = grid_for((long long)rows, kWarpsPerBlock, 2);
  rmsnorm_bwd_kernel<W><<<grid, kWarpsPerBlock * 32, H * sizeof(float), STREAM(stream)>>>(
      (const __nv_bfloat16*)x, w, (const float*)rstd, (const __nv_bfloat16*)dy, (const __nv_bfloat16*)dres,
      (__nv_bfloat16*)dx, (float*)dw, rows, H);
  return LAST_ERR();
}
extern "C" int b200_rmsnorm_bwd(const void* x, const void* w, int w_bf16, const void* rstd, const void* dy,
                                const void* dres, void* dx, void* dw, int rows, int H, void* stream) {
  if (H % 8 || H * 4 > 48 * 1024) return -2;
  if (w_bf16)
    return rmsnorm_bwd_launch(x, (const __nv_bfloat16*)w, rstd, dy, dres, dx, dw, rows, H, stream);
  return rmsnorm_bwd_launch(x, (const float*)w, rstd, dy, dres, dx, dw, rows, H, stream);
}
static int lanes_per_head(int D) {
  int lph = 1;
  while (lph * 8 < D) lph <<= 1;
  return lph;
}
// A warp per token and kind of heads where that gives every scheduler of the device eight warps; with fewer tokens (a
// decode step, short sequences) a token's heads are dealt to more warps, down to one group of heads each.  The blocks
// are shared out between query and key heads by their number of groups.
static int qk_shape(QkShape& q, long long tokens, int heads_first, int heads, int D, float theta, int rope,
                    int blocks_per_sm) {
  const int hpw = 32 / lanes_per_head(D);
  const int first = (heads_first + hpw - 1) / hpw, rest = (heads - heads_first + hpw - 1) / hpw;
  const int most = first > rest ? first : rest;
  const long long want = 148 * 32;
  long long per = tokens >= want ? most : (tokens * (first + rest) + want - 1) / want;
  per = per < 1 ? 1 : (per > most ? most : per);
  const long long items_first = tokens * ((first + per - 1) / per), items_rest = tokens * ((rest + per - 1) / per);
  int grid = grid_for(items_first + items_rest, kWarpsPerBlock, blocks_per_sm);
  int blocks_first = grid * first / (first + rest);
  if (first && blocks_first == 0) blocks_first = 1;
  if (rest && blocks_first >= grid) grid = blocks_first + 1;
  if (!rest) blocks_first = grid;
  q = QkShape{tokens, heads, heads_first, D, blocks_first, (int)per, log2f(theta), rope};
  return grid;
}
#define QK_DISPATCH(D, CALL)            \
  switch (lanes_per_head(D)) {          \
    case 1: CALL(1);                    \
    case 2: CALL(2);                    \
    case 4: CALL(4);                    \
    case 8: CALL(8);                    \
    case 16: CALL(16);                  \
    default: CALL(32);                  \
  }
// Query and key heads of a packed projection in one launch: the first heads_q heads use wq, the next heads_k use wk
// (both or neither given); rstd is [tokens, heads_q + heads_k].
extern "C" int b200_qknorm_rope_fwd_qk(const void* in, long long in_stride, void* out, long long out_stride,
                                       const void* wq, const void* wk, int w_bf16, const void* positions, void* rstd,
                                       long long tokens, int heads_q, int heads_k, int D, float eps, float theta,
                                       int rope, void* stream) {
  if (D % 8 || D > 256 || (heads_k && (wq == nullptr) != (wk == nullptr))) return -2;
  if (tokens <= 0 || heads_q + heads_k <= 0) return 0;
  QkShape q;
  const int grid = qk_shape(q, tokens, heads_q, heads_q + heads_k, D, theta, rope, kQkFwdBlocks);
#define QK_FWD_AS(LPH, W)                                                                                             \
  return static_cast<int>(b200host::launch_kernel(                                                                    \
      qknorm_rope_fwd_kernel<LPH, W>, dim3(grid), dim3(kWarpsPerBlock * 32), 0, STREAM(stream),                       \
      tokens <= 512 && b200host::pdl_enabled() != 0, (const __nv_bfloat16*)in, in_stride, (__nv_bfloat16*)out,        \
      out_stride, (const W*)wq, (const W*)wk, (const int*)positions, (float*)rstd, q, eps))
#define QK_FWD(LPH)                          \
  if (w_bf16) QK_FWD_AS(LPH, __nv_bfloat16); \
  QK_FWD_AS(LPH, float)
  QK_DISPATCH(D, QK_FWD)
#undef QK_FWD
#undef QK_FWD_AS
}
extern "C" int b200_qknorm_rope_fwd(const void* in, long long in_stride, void* out, long long out_stride,
                                    const void* w, int w_bf16, const void* positions, void* rstd, long long tokens,
                                    int heads, int D, float eps, float theta, int rope, void* stream) {
  return b200_qknorm_rope_fwd_qk(in, in_stride, out, out_stride, w, nullptr, w_bf16, positions, rstd, tokens, heads, 0,
                                 D, eps, theta, rope, stream);
}
extern "C" int b200_qknorm_rope_bwd_qk(const void* in, long long in_stride, const void* dout, long long dout_stride,
                                       void* din, long long din_stride, const void* wq, const void* wk, int w_bf16,
                                       const void* positions, const void* rstd, void* dwq, void* dwk,
                                       long long tokens, int heads_q, int heads_k, int D, float theta, int rope,
                                       void* stream) {
  if (D % 8 || D > 256 || (heads_k && (wq == nullptr) != (wk == nullptr))) return -2;
  if (tokens <= 0 || heads_q + heads_k <= 0) return 0;
  QkShape q;
  const int grid = qk_shape(q, tokens, heads_q, heads_q + heads_k, D, theta, rope, kQkBwdBlocks);
#define QK_BWD_AS(LPH, W)                                                                                           \
  {                                                                                                                 \
    qknorm_rope_bwd_kernel<LPH, W><<<grid, kWarpsPerBlock * 32, 0, STREAM(stream)>>>(                               \
        (const __nv_bfloat16*)in, in_stride, (const __nv_bfloat16*)dout, dout_stride, (__nv_bfloat16*)din,          \
        din_stride, (const W*)wq, (const W*)wk, (const int*)positions, (const float*)rstd, (float*)dwq,             \
        (float*)dwk, q);                                                                                            \
    return LAST_ERR();                                                                                              \
  }
#define QK_BWD(LPH)                         \
  if (w_bf16) QK_BWD_AS(LPH, __nv_bfloat16) \
  QK_BWD_AS(LPH, float)
  QK_DISPATCH(D, QK_BWD)
#undef QK_BWD
#undef QK_BWD_AS
}
extern "C" int b200_qknorm_rope_bwd(const void* in, long long in_stride, const void* dout, long long dout_stride,
                                    void* din, long long din_stride, const void* w, int w_bf16, const void* positions,
                                    const void* rstd, void* dw, long long tokens, int heads, int D, float theta,
                                    int rope, void* stream) {
  return b200_qknorm_rope_bwd_qk(in, in_stride, dout, dout_stride, din, din_stride, w, nullptr, w_bf16, positions, rstd,
                                 dw, nullptr, tokens, heads, 0, D, theta, rope, stream);
}
#undef QK_DISPATCH
extern "C" int b200_kv_upper_bound(const void* lo, void* hi, int B, int S, int n, int offset, void* stream) {
  if (B <= 0 || B > 65535 || S <= 0 || n <= 0) return -2;
  kv_upper_bound_kernel<<<dim3((n + 127) / 128, B), 128, 0, STREAM(stream)>>>((const int*)lo, (int*)hi, S, n, offset);
  return LAST_ERR();
}
extern "C" int b200_swiglu_fwd(const void* gu, void* h, long long rows, int I, void* stream) {
  if (I % 8 || rows * (I / 8) >= (1LL << 32)) return -2;
  return static_cast<int>(b200host::launch_kernel(swiglu_fwd_kernel, dim3(grid_for(rows * (I / 8), 256)), dim3(256), 0,
                                                  STREAM(stream), rows <= 512 && b200host::pdl_enabled() != 0,
                                                  (const __nv_bfloat16*)gu, (__nv_bfloat16*)h, rows, I));
}
extern "C" int b200_swiglu_bwd(const void* gu, const void* dh, void* dgu, long long rows, int I, void* stream) {
  if (I % 8 || rows * (I / 8) >= (1LL << 32)) return -2;
  swiglu_bwd_kernel<<<grid_for(rows * (I / 8), 256), 256, 0, STREAM(stream)>>>(
      (const __nv_bfloat16*)gu, (const __nv_bfloat16*)dh, (__nv_bfloat16*)dgu, rows, I);
  return LAST_ERR();
}
extern "C" int b200_sigmoid_gate_fwd(const void* a, const void* gate, void* out, long long n, void* stream) {
  if (n % 8) return -2;
  sigmoid_gate_fwd_kernel<<<grid_for(n / 8, 256), 256, 0, STREAM(stream)>>>(
      (const __nv_bfloat16*)a, (const __nv_bfloat16*)gate, (__nv_bfloat16*)out, n / 8);
  return LAST_ERR();
}
extern "C" int b200_sigmoid_gate_bwd(const void* a, const void* gate, const void* dout, void* da, void* dgate,
                                     long long n, void* stream) {
  if (n % 8) return -2;
  sigmoid_gate_bwd_kernel<<<grid_for(n / 8, 256), 256, 0, STREAM(stream)>>>(
      (const __nv_bfloat16*)a, (const __nv_bfloat16*)gate, (const __nv_bfloat16*)dout, (__nv_bfloat16*)da,
      (__nv_bfloat16*)dgate, n / 8);
  return LAST_ERR();
}
extern "C" int b200_embedding_fwd(const void* ids, const void* table, void* out, long long tokens, int H,
                                  float scale, void* stream) {
  if (H % 8) return -2;
  embedding_fwd_kernel<<<grid_for(tokens * (H / 8), 256), 256, 0, STREAM(stream)>>>(
      (const int*)ids, (const __nv_bfloat16*)table, (__nv_bfloat16*)out, tokens, H, scale);
  return LAST_ERR();
}
extern "C" int b200_embedding_bwd(const void* ids, const void* dout, void* dtable, long long tokens, int H,
                                  float scale, void* stream) {
  if (H % 8) return -2;
  embedding_bwd_kernel<<<grid_for(tokens * (H / 8), 256), 256, 0, STREAM(stream)>>>(
      (const int*)ids, (const __nv_bfloat16*)dout, (float*)dtable, tokens, H, scale);
  return LAST_ERR();
}
extern "C" int b200_ce_fwd_bwd(void* logits, long long ld, const void* targets, const void* mask, void* loss_row,
                               void* z_row, void* lse_row, int rows, int V, float grad_scale, float z_weight,
                               int write_grad, void* status, void* stream) {
  if (rows <= 0) return 0;
  if (ld % 8) return -1;  // rows must stay 16-byte aligned for the vector path
  const size_t row_bytes = (size_t)V * 2;
  if (V % 8 == 0 && row_bytes <= 200 * 1024 && (reinterpret_cast<uintptr_t>(logits) & 15u) == 0 && status) {
    static bool configured[b200host::kMaxDevices] = {};
    if (int rc = b200host::ensure_dynamic_smem(ce_fwd_bwd_staged_kernel, 200 * 1024, configured)) return rc;
    ce_fwd_bwd_staged_kernel<<<rows, kCeThreads, row_bytes, STREAM(stream)>>>(
        (__nv_bfloat16*)logits, ld, (const int*)targets, (const uint8_t*)mask, (float*)loss_row, (float*)z_row,
        (float*)lse_row, V, grad_scale, z_weight, write_grad, (int*)status);
    return LAST_ERR();
  }
  ce_fwd_bwd_kernel<<<rows, 512, 0, STREAM(stream)>>>((__nv_bfloat16*)logits, ld, (const int*)targets,
                                                      (const uint8_t*)mask, (float*)loss_row, (float*)z_row,
                                                      (float*)lse_row, V, grad_scale, z_weight, write_grad);
  return LAST_ERR();
}
extern "C" int b200_adamw(void* p, void* m, void* v, const void* g, int g_is_bf16, void* shadow, const void* gscale,
                          long long n, float lr, float b1, float b2, float eps, float wd, float bc1, float bc2,
                          void* stream) {
  if (n <= 0) return 0;
  auto misaligned = [](const void* q, uintptr_t a) { return (reinterpret_cast<uintptr_t>(q) & (a - 1)) != 0; };
  if (n % 4 == 0 && !misaligned(p, 16) && !misaligned(m, 16) && !misaligned(v, 16) &&
      !misaligned(g, g_is_bf16 ? 8 : 16) && !misaligned(shadow, 8)) {
    const int vgrid = grid_for(n / 4, 256, 8);
    if (g_is_bf16)
      adamw_vec4_kernel<__nv_bfloat16><<<vgrid, 256, 0, STREAM(stream)>>>(
          (float4*)p, (float4*)m, (float4*)v, (const __nv_bfloat16*)g, (__nv_bfloat16*)shadow, (const float*)gscale,
          n / 4, lr, b1, b2, eps, wd, bc1, bc2);
    else
      adamw_vec4_kernel<float><<<vgrid, 256, 0, STREAM(stream)>>>((float4*)p, (float4*)m, (float4*)v, (const float*)g,
                                                                 (__nv_bfloat16*)shadow, (const float*)gscale, n / 4,
                                                                 lr, b1, b2, eps, wd, bc1, bc2);
    return LAST_ERR();
  }
  const int grid = grid_for(n, 256, 8);
  if (g_is_bf16)
    adamw_kernel<__nv_bfloat16><<<grid, 256, 0, STREAM(stream)>>>((float*)p, (float*)m, (float*)v,
                                                                   (const __nv_bfloat16*)g, (__nv_bfloat16*)shadow,
                                                                   (const float*)gscale, n, lr, b1, b2, eps, wd, bc1, bc2);
  else
    adamw_kernel<float><<<grid, 256, 0, STREAM(stream)>>>((float*)p, (float*)m, (float*)v, (const float*)g,
                                                           (__nv_bfloat16*)shadow, (const float*)gscale, n, lr, b1, b2,
                                                           eps, wd, bc1, bc2);
  return LAST_ERR();
}
// scratch: at least 1024 floats.  out[0] (+)= sum(x^2)
extern "C" int b200_sumsq(const void* x, int is_bf16, long long n, void* scratch, void* out, int accumulate,
                          void* stream) {
  int grid = grid_for(n, 512, 4);
  if (grid > 1024) grid = 1024;
  if (is_bf16)
    sumsq_partial_kernel<__nv_bfloat16><<<grid, 512, 0, STREAM(stream)>>>((const __nv_bfloat16*)x, n, (float*)scratch);
  else
    sumsq_partial_kernel<float><<<grid, 512, 0, STREAM(stream)>>>((const float*)x, n, (float*)scratch);
  sumsq_final_kernel<<<1, 256, 0, STREAM(stream)>>>((const float*)scratch, grid, (float*)out, accumulate);
  return LAST_ERR();
}
extern "C" int b200_cast_f32_bf16(const void* x, void* y, long long n, float scale, void* stream) {
  if (n <= 0) return 0;
  cast_f32_bf16_kernel<<<grid_for(n, 256, 8), 256, 0, STREAM(stream)>>>((const float*)x, (__nv_bfloat16*)y, n, scale);
  return LAST_ERR();
}
