// Bandwidth-bound fused kernels: RMSNorm (+residual add) fwd/bwd, SwiGLU/GeGLU
// fwd/bwd, in-place QK rotary embedding, embedding gather / deterministic
// scatter-add, cross-entropy on materialised logits.  All bf16 in/out with fp32
// math, 16-byte vector accesses, grids sized from the SM count.
//
// They replace the reference's Triton kernels (chronicals/kernels/
// triton_kernels.py:303-478 RMSNorm, :830-986 SwiGLU, :1296-1367 GeGLU,
// :1448-1625 QK-RoPE, :127-210 cross-entropy) and the Liger kernels its trainer
// patches in.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <utility>
#include <cooperative_groups.h>
#include "common.cuh"

// ---- optional index checks (compile with -DCHRONICALS_DEBUG_BOUNDS, e.g. CHRONICALS_DEBUG_BOUNDS=1 in the
// environment of csrc/build.py).  Release kernels already clamp or mask every gathered index; the debug build
// additionally records the first offending value in a device word that cb_debug_word() reads back.  Nothing
// traps: the kernel carries on with the clamped index.
enum { CB_DBG_TOKEN_ID = 401, CB_DBG_ROPE_POSITION = 402, CB_DBG_LABEL = 403 };
__device__ long long g_cb_debug_word[2] = {0, 0};
#ifdef CHRONICALS_DEBUG_BOUNDS
#define CB_DEBUG_CHECK(cond, code, value)                                                            \
  do {                                                                                               \
    if (!(cond) && atomicCAS(reinterpret_cast<unsigned long long*>(&g_cb_debug_word[0]), 0ull,       \
                             static_cast<unsigned long long>(code)) == 0ull)                        \
      g_cb_debug_word[1] = static_cast<long long>(value);                                            \
  } while (0)
#else
#define CB_DEBUG_CHECK(cond, code, value) do { } while (0)
#endif

namespace cg = cooperative_groups;

namespace cb {

constexpr int EW_THREADS = 256;

struct alignas(16) Vec8 {
  uint4 u;
};
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16x2(f[0], f[1]); u.y = pack_bf16x2(f[2], f[3]);
  u.z = pack_bf16x2(f[4], f[5]); u.w = pack_bf16x2(f[6], f[7]);
  return u;
}

// 16 bytes from global to this thread's own place in shared memory, without passing through registers.  A thread reads
// only what it copied itself, so a ring of such places needs no barrier: its own wait is enough.
__device__ __forceinline__ void cp_async16(uint4* dst, const uint4* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// How rows are laid over threads.  Up to 1024 columns a warp takes a row (shuffles only, eight rows a block); wider rows
// take a block that is just wide enough for two vectors of 8 a thread, and four beyond 5120 columns.
template <int VPL, bool WARP_ROW>
struct RowLayout {
  int t, tpr, group, groups;
  __device__ __forceinline__ RowLayout() {
    t = WARP_ROW ? static_cast<int>(threadIdx.x & 31) : static_cast<int>(threadIdx.x);
    tpr = WARP_ROW ? 32 : static_cast<int>(blockDim.x);
    group = WARP_ROW ? static_cast<int>(threadIdx.x >> 5) : 0;
    groups = WARP_ROW ? static_cast<int>(blockDim.x >> 5) : 1;
  }
};

// Sum over the threads of one row.  `sred` has two halves of 32 floats used in turn (`flip`), so that one barrier a row
// is enough: nobody writes a half again before everybody has left the barrier after reading it.
template <bool WARP_ROW>
__device__ __forceinline__ float row_sum(float v, float* sred, int flip) {
  v = warp_sum(v);
  if (WARP_ROW) return v;
  float* half = sred + 32 * flip;
  if ((threadIdx.x & 31) == 0) half[threadIdx.x >> 5] = v;
  __syncthreads();
  const int nw = static_cast<int>(blockDim.x >> 5);
  float t = 0.f;
  for (int i = 0; i < nw; ++i) t += half[i];
  return t;
}

// ------------------------------------------------------------------ RMSNorm forward
// h = x (+ res);  y = h * rsqrt(mean(h^2) + eps) * (w + offset);  rstd saved.
// N % 8 == 0, N <= 8 * VPL * (threads of a row).
template <int VPL, bool WARP_ROW>
__global__ void __launch_bounds__(WARP_ROW ? EW_THREADS : 320)
rmsnorm_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ res, const bf16* __restrict__ w,
                   bf16* __restrict__ y, bf16* __restrict__ h_out, float* __restrict__ rstd_out, int M, int N,
                   float eps, float offset) {
  __shared__ float sred[64];
  const RowLayout<VPL, WARP_ROW> L;
  const int nvec = N / 8;
  const int step = gridDim.x * L.groups;
  int flip = 0;
  for (long long row = blockIdx.x * L.groups + L.group; row < M; row += step) {
    const uint4* xp = reinterpret_cast<const uint4*>(x + row * N);
    const uint4* rp = res ? reinterpret_cast<const uint4*>(res + row * N) : nullptr;
    uint4* hp = h_out ? reinterpret_cast<uint4*>(h_out + row * N) : nullptr;
    uint4 hr[VPL];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i)
      if (L.t + i * L.tpr < nvec) hr[i] = xp[L.t + i * L.tpr];
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = L.t + i * L.tpr;
      if (v < nvec) {
        float f[8];
        unpack8(hr[i], f);
        if (rp) {
          float r[8];
          unpack8(rp[v], r);
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] += r[j];
          hr[i] = pack8(f);                          // the sum is stored in bf16; normalise what is stored
          if (hp) hp[v] = hr[i];
          unpack8(hr[i], f);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
      }
    }
    ss = row_sum<WARP_ROW>(ss, sred, flip);
    const float rstd = rsqrtf(ss / static_cast<float>(N) + eps);
    if (L.t == 0 && rstd_out) rstd_out[row] = rstd;
    uint4* yp = reinterpret_cast<uint4*>(y + row * N);
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = L.t + i * L.tpr;
      if (v < nvec) {
        float f[8], wf[8], o[8];
        unpack8(hr[i], f);
        unpack8(reinterpret_cast<const uint4*>(w)[v], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = f[j] * rstd * (wf[j] + offset);
        yp[v] = pack8(o);
      }
    }
    flip ^= 1;
  }
}

// ------------------------------------------------------------------ RMSNorm backward
// xhat = h*rstd; g = dy*(w+offset); dx = rstd*(g - xhat*mean(g*xhat)) (+ dres_in);
// dw[n] = sum_rows dy*xhat, accumulated per block in registers and written as one
// [gridDim.x, N] fp32 partial (reduced by rmsnorm_dw_reduce_kernel).
// Bound by memory (four tensors).  The sums of dw keep two blocks an SM at most, and with the loads of a row waiting
// behind the reduction and the stores of the one before, they kept memory busy two thirds of the time; now each thread
// has its vectors of the next RING - 1 rows in flight through the ring.  Measured: 16,384 x 5120 144 -> 109 us
// (6.1 TB/s), 16,384 x 2048 68 -> 49, 32,768 x 896 50 -> 43, 8192 x 896 16.3 -> 16.0.  The forward kernel has enough
// blocks an SM without a ring (16,384 x 5120: 66 us with one, 58 without).
// Dynamic shared memory: RING * (dres_in ? 3 : 2) * VPL * blockDim.x vectors, and no less than [groups, N] floats.
template <int VPL, bool WARP_ROW, int RING>
__global__ void __launch_bounds__(WARP_ROW ? EW_THREADS : 320, 2)
rmsnorm_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ h, const bf16* __restrict__ w,
                   const float* __restrict__ rstd_in, const bf16* __restrict__ dres_in, bf16* __restrict__ dx,
                   float* __restrict__ dw_part, int M, int N, float offset) {
  extern __shared__ __align__(16) uint4 ring[];
  __shared__ float sred[64];
  const RowLayout<VPL, WARP_ROW> L;
  const int nvec = N / 8;
  const int step = gridDim.x * L.groups;
  const int row0 = blockIdx.x * L.groups + L.group;
  const int inputs = dres_in ? 3 : 2;
  const auto slot = [&](int stage, int in, int i) { return ring + ((stage * inputs + in) * VPL + i) * blockDim.x + threadIdx.x; };
  const auto fetch = [&](long long row, int stage) {
    if (row < M) {
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int v = L.t + i * L.tpr;
        if (v < nvec) {
          cp_async16(slot(stage, 0, i), reinterpret_cast<const uint4*>(dy + row * N) + v);
          cp_async16(slot(stage, 1, i), reinterpret_cast<const uint4*>(h + row * N) + v);
          if (dres_in) cp_async16(slot(stage, 2, i), reinterpret_cast<const uint4*>(dres_in + row * N) + v);
        }
      }
    }
    cp_async_commit();
  };
  uint4 wr[VPL];
  float dwacc[VPL][8];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    if (L.t + i * L.tpr < nvec) wr[i] = reinterpret_cast<const uint4*>(w)[L.t + i * L.tpr];
#pragma unroll
    for (int j = 0; j < 8; ++j) dwacc[i][j] = 0.f;
  }
  for (int k = 0; k < RING - 1; ++k) fetch(row0 + static_cast<long long>(k) * step, k);
  float rstd_next = row0 < M ? rstd_in[row0] : 0.f;
  int stage = 0, flip = 0;
  for (long long row = row0; row < M; row += step) {
    const float rstd = rstd_next;
    if (row + step < M) rstd_next = rstd_in[row + step];
    fetch(row + static_cast<long long>(RING - 1) * step, stage == 0 ? RING - 1 : stage - 1);
    cp_async_wait<RING - 1>();
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (L.t + i * L.tpr < nvec) {
        float d[8], x[8], wf[8];
        unpack8(*slot(stage, 0, i), d);
        unpack8(*slot(stage, 1, i), x);
        unpack8(wr[i], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = x[j] * rstd;
          dot += d[j] * (wf[j] + offset) * xh;
          dwacc[i][j] += d[j] * xh;
        }
      }
    }
    dot = row_sum<WARP_ROW>(dot, sred, flip);
    const float mean = dot / static_cast<float>(N);
    uint4* dxp = reinterpret_cast<uint4*>(dx + row * N);
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = L.t + i * L.tpr;
      if (v < nvec) {
        float d[8], x[8], wf[8], o[8];
        unpack8(*slot(stage, 0, i), d);
        unpack8(*slot(stage, 1, i), x);
        unpack8(wr[i], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rstd * (d[j] * (wf[j] + offset) - x[j] * rstd * mean);
        if (dres_in) {
          float r[8];
          unpack8(*slot(stage, 2, i), r);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += r[j];
        }
        dxp[v] = pack8(o);
      }
    }
    stage = stage + 1 == RING ? 0 : stage + 1;
    flip ^= 1;
  }
  // one partial row of dw per block: with several rows in a block every group parks its sums in its own [N] row of
  // shared memory (the ring is done with) and the block adds them column by column (fixed order, no atomics)
  float* out = dw_part + static_cast<long long>(blockIdx.x) * N;
  if (WARP_ROW) {
    float* sdw = reinterpret_cast<float*>(ring);
    cp_async_wait<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = L.t + i * L.tpr;
      if (v < nvec) {
        float4* m = reinterpret_cast<float4*>(sdw + static_cast<size_t>(L.group) * N) + 2 * v;
        m[0] = make_float4(dwacc[i][0], dwacc[i][1], dwacc[i][2], dwacc[i][3]);
        m[1] = make_float4(dwacc[i][4], dwacc[i][5], dwacc[i][6], dwacc[i][7]);
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
      float a = 0.f;
#pragma unroll
      for (int r = 0; r < EW_THREADS / 32; ++r) a += sdw[static_cast<size_t>(r) * N + i];
      out[i] = a;
    }
  } else {
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = L.t + i * L.tpr;
      if (v < nvec) {
        reinterpret_cast<float4*>(out)[2 * v] = make_float4(dwacc[i][0], dwacc[i][1], dwacc[i][2], dwacc[i][3]);
        reinterpret_cast<float4*>(out)[2 * v + 1] = make_float4(dwacc[i][4], dwacc[i][5], dwacc[i][6], dwacc[i][7]);
      }
    }
  }
}

// Column sums of a bf16 matrix (bias gradients): part[block, n] = sum over the block's rows of x[row, n].
// Thread t of a block owns the 8 columns of vector (blockIdx.y * blockDim.x + t); blocks along x split the rows.
__global__ void __launch_bounds__(EW_THREADS)
colsum_partial_kernel(const bf16* __restrict__ x, long long ld, long long M, int N, float* __restrict__ part) {
  const int v = blockIdx.y * blockDim.x + threadIdx.x;
  if (v >= N / 8) return;
  const long long rows_per = (M + gridDim.x - 1) / gridDim.x;
  const long long r0 = blockIdx.x * rows_per;
  const long long r1 = (r0 + rows_per < M) ? r0 + rows_per : M;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  long long r = r0;
  for (; r + 4 <= r1; r += 4) {                    // four independent 16-byte loads in flight
    uint4 u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] = *reinterpret_cast<const uint4*>(x + (r + i) * ld + (static_cast<long long>(v) << 3));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float f[8];
      unpack8(u[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += f[j];
    }
  }
  for (; r < r1; ++r) {
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(x + r * ld + (static_cast<long long>(v) << 3)), f);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] += f[j];
  }
  float* o = part + static_cast<long long>(blockIdx.x) * N + (v << 3);
  reinterpret_cast<float4*>(o)[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
  reinterpret_cast<float4*>(o)[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
}

// 1024 threads = 32 columns x 32 row slices; each slice sums every 32nd partial row, then the slices combine.  The
// partials lie in L2 and the sum is bound by latency: with 32 slices (8 before) a thread waits for a quarter of the loads.
__global__ void __launch_bounds__(1024)
rmsnorm_dw_reduce_kernel(const float* __restrict__ part, int nblocks, int N, bf16* __restrict__ dw, int accumulate) {
  __shared__ float red[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int n = blockIdx.x * 32 + tx;
  float s = 0.f;
  if (n < N) {
#pragma unroll 4
    for (int b = ty; b < nblocks; b += 32) s += part[static_cast<long long>(b) * N + n];
  }
  red[ty][tx] = s;
  __syncthreads();
  const float t = warp_sum(red[tx][ty]);               // warp ty adds the slices of column ty
  const int m = blockIdx.x * 32 + ty;
  if (tx == 0 && m < N) dw[m] = __float2bfloat16(accumulate ? t + __bfloat162float(dw[m]) : t);
}

// ------------------------------------------------------------------ gated activations
__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + __expf(-x)); }
__device__ __forceinline__ float gelu_tanh(float x) {
  const float k = 0.7978845608028654f;
  return 0.5f * x * (1.f + tanhf(k * (x + 0.044715f * x * x * x)));
}
__device__ __forceinline__ float gelu_tanh_grad(float x) {
  const float k = 0.7978845608028654f;
  const float u = k * (x + 0.044715f * x * x * x);
  const float th = tanhf(u);
  return 0.5f * (1.f + th) + 0.5f * x * (1.f - th * th) * k * (1.f + 3.f * 0.044715f * x * x);
}

// out[m, i] = act(gate[m, i]) * up[m, i];  rows have pitch ld_in / ld_out (elements), I % 8 == 0
template <int GELU>
__global__ void __launch_bounds__(EW_THREADS)
glu_fwd_kernel(const bf16* __restrict__ gate, const bf16* __restrict__ up, bf16* __restrict__ out, long long M, int I,
               long long ld_in, long long ld_out) {
  const int vpr = I / 8;
  const long long total = M * vpr;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long m = idx / vpr;
    const int v = static_cast<int>(idx % vpr);
    float g[8], u[8], o[8];
    unpack8(*reinterpret_cast<const uint4*>(gate + m * ld_in + v * 8), g);
    unpack8(*reinterpret_cast<const uint4*>(up + m * ld_in + v * 8), u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = (GELU ? gelu_tanh(g[j]) : g[j] * sigmoidf_(g[j])) * u[j];
    *reinterpret_cast<uint4*>(out + m * ld_out + v * 8) = pack8(o);
  }
}

template <int GELU>
__global__ void __launch_bounds__(EW_THREADS)
glu_bwd_kernel(const bf16* __restrict__ dout, const bf16* __restrict__ gate, const bf16* __restrict__ up,
               bf16* __restrict__ dgate, bf16* __restrict__ dup, long long M, int I, long long ld_dout,
               long long ld_in, long long ld_din) {
  const int vpr = I / 8;
  const long long total = M * vpr;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long m = idx / vpr;
    const int v = static_cast<int>(idx % vpr);
    float d[8], g[8], u[8], dg[8], du[8];
    unpack8(*reinterpret_cast<const uint4*>(dout + m * ld_dout + v * 8), d);
    unpack8(*reinterpret_cast<const uint4*>(gate + m * ld_in + v * 8), g);
    unpack8(*reinterpret_cast<const uint4*>(up + m * ld_in + v * 8), u);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (GELU) {
        du[j] = d[j] * gelu_tanh(g[j]);
        dg[j] = d[j] * u[j] * gelu_tanh_grad(g[j]);
      } else {
        const float s = sigmoidf_(g[j]);
        du[j] = d[j] * g[j] * s;
        dg[j] = d[j] * u[j] * s * (1.f + g[j] * (1.f - s));
      }
    }
    *reinterpret_cast<uint4*>(dgate + m * ld_din + v * 8) = pack8(dg);
    *reinterpret_cast<uint4*>(dup + m * ld_din + v * 8) = pack8(du);
  }
}

// ------------------------------------------------------------------ rotary embedding, in place
// q: [T, hq, D] and k: [T, hk, D] with token pitches ldq / ldk (so both may live inside one
// fused QKV buffer).  cos/sin: [P, D/2] fp32.  pos: [T] int64 or null (position = token index).
// One thread rotates 8 pairs.  sign = -1 gives the inverse rotation (the backward).
template <int INTERLEAVED>
__global__ void __launch_bounds__(EW_THREADS)
qk_rope_kernel(bf16* __restrict__ q, bf16* __restrict__ k, const float* __restrict__ cosT,
               const float* __restrict__ sinT, const long long* __restrict__ pos, long long T, int hq, int hk, int D,
               long long ldq, long long ldk, float sign, long long table_len) {
  const int half = D / 2;
  const int tph = half / 8;  // threads per head
  const int heads = hq + hk;
  const long long total = T * heads * tph;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(idx % tph);
    const int hh = static_cast<int>((idx / tph) % heads);
    const long long t = idx / (static_cast<long long>(tph) * heads);
    long long p = pos ? pos[t] : t;
    CB_DEBUG_CHECK(p >= 0 && p < table_len, CB_DBG_ROPE_POSITION, p);
    p = p < 0 ? 0 : (p >= table_len ? table_len - 1 : p);   // never read outside the cos/sin tables
    bf16* base = hh < hq ? q + t * ldq + static_cast<long long>(hh) * D : k + t * ldk + static_cast<long long>(hh - hq) * D;
    const float4* cp = reinterpret_cast<const float4*>(cosT + p * half + c * 8);
    const float4* sp = reinterpret_cast<const float4*>(sinT + p * half + c * 8);
    const float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
    const float cs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const float sn[8] = {s0.x * sign, s0.y * sign, s0.z * sign, s0.w * sign,
                         s1.x * sign, s1.y * sign, s1.z * sign, s1.w * sign};
    if (INTERLEAVED) {
      uint4* p0 = reinterpret_cast<uint4*>(base + c * 16);
      float a[8], b[8];
      unpack8(p0[0], a);
      unpack8(p0[1], b);
      float o0[8], o1[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float x1 = a[2 * j], x2 = a[2 * j + 1];
        o0[2 * j] = x1 * cs[j] - x2 * sn[j];
        o0[2 * j + 1] = x2 * cs[j] + x1 * sn[j];
        const float y1 = b[2 * j], y2 = b[2 * j + 1];
        o1[2 * j] = y1 * cs[4 + j] - y2 * sn[4 + j];
        o1[2 * j + 1] = y2 * cs[4 + j] + y1 * sn[4 + j];
      }
      p0[0] = pack8(o0);
      p0[1] = pack8(o1);
    } else {
      uint4* p1 = reinterpret_cast<uint4*>(base + c * 8);
      uint4* p2 = reinterpret_cast<uint4*>(base + half + c * 8);
      float x1[8], x2[8], o1[8], o2[8];
      unpack8(*p1, x1);
      unpack8(*p2, x2);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        o1[j] = x1[j] * cs[j] - x2[j] * sn[j];
        o2[j] = x2[j] * cs[j] + x1[j] * sn[j];
      }
      *p1 = pack8(o1);
      *p2 = pack8(o2);
    }
  }
}

// ------------------------------------------------------------------ embedding
__global__ void __launch_bounds__(128)
embedding_fwd_kernel(const long long* __restrict__ ids, const bf16* __restrict__ table, bf16* __restrict__ out,
                     long long T, int N, long long V) {
  const int nvec = N / 8;
  for (long long t = blockIdx.x; t < T; t += gridDim.x) {
    long long id = ids[t];
    CB_DEBUG_CHECK(id >= 0 && id < V, CB_DBG_TOKEN_ID, id);
    if (id < 0 || id >= V) id = 0;   // out-of-range ids read row 0 instead of faulting
    const uint4* src = reinterpret_cast<const uint4*>(table + id * N);
    uint4* dst = reinterpret_cast<uint4*>(out + t * N);
    for (int v = threadIdx.x; v < nvec; v += blockDim.x) dst[v] = src[v];
  }
}

// Backward: dtable[id] = sum of dout over the tokens that carry `id`, in fp32, in token order, zero elsewhere.
//
// Step 1 writes the zeros (bound by memory: V x N bf16) and, in its first blocks, sorts the tokens by id while the
// stores drain: the place of token i is the number of tokens with a smaller id or with the same id and a smaller
// index, counted outright against all T ids.  That is T^2 integer compares, 64 tokens per block, a quarter of the
// ids per thread; no passes over keys, no scan, and the result does not depend on the order of anything.
// Measured, T = 8192, V = 151,936, N = 896: 59 us together; a fill of the same bytes alone took 70 us and a radix sort
// of the 64-bit ids 65 us before.
constexpr int EMB_RANK_TOKENS = 64;
constexpr int EMB_RANK_TILE = 4096;                    // ids staged in shared memory at a time
constexpr int EMB_NO_ROW = 0x7ffffffe;                 // ids outside [0, V): sorted last, never written

__global__ void __launch_bounds__(EW_THREADS)
embedding_rank_fill_kernel(const long long* __restrict__ ids, int* __restrict__ sorted_ids, int* __restrict__ perm, int T,
                           int rank_blocks, uint4* __restrict__ dtable, long long table_vecs, long long V) {
  __shared__ __align__(16) int tile[EMB_RANK_TILE];
  if (static_cast<int>(blockIdx.x) >= rank_blocks) {
    const long long step = static_cast<long long>(gridDim.x - rank_blocks) * EW_THREADS;
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    for (long long i = (blockIdx.x - rank_blocks) * static_cast<long long>(EW_THREADS) + threadIdx.x; i < table_vecs; i += step)
      dtable[i] = z;
    return;
  }
  const auto row_of = [&](int j) {
    const long long id = ids[j];
    return id >= 0 && id < V ? static_cast<int>(id) : EMB_NO_ROW;
  };
  const int lane = threadIdx.x & 31;
  const int slice = lane >> 3;                         // which quarter of every group of 16 ids this thread compares with
  const int i0 = blockIdx.x * EMB_RANK_TOKENS;
  const int i = i0 + (threadIdx.x >> 5) * 8 + (lane & 7);
  const int mine = i < T ? row_of(i) : 0;
  int rank = 0;
  for (int t0 = 0; t0 < T; t0 += EMB_RANK_TILE) {
    const int n = T - t0 < EMB_RANK_TILE ? T - t0 : EMB_RANK_TILE;
    __syncthreads();
    for (int k = threadIdx.x; k < (n + 15) / 16 * 16; k += EW_THREADS)
      tile[k] = k < n ? row_of(t0 + k) : 0x7fffffff;   // past the end: larger than any id
    __syncthreads();
    const int4* tv = reinterpret_cast<const int4*>(tile);
    if (t0 + EMB_RANK_TILE <= i0 || t0 >= i0 + EMB_RANK_TOKENS) {
      const int bound = mine + (t0 < i0 ? 1 : 0);      // ids before mine win ties, ids after it lose them
#pragma unroll 4
      for (int k = slice; k < (n + 15) / 16 * 4; k += 4) {
        const int4 o = tv[k];
        rank += (o.x < bound) + (o.y < bound) + (o.z < bound) + (o.w < bound);
      }
    } else {
      for (int k = slice; k < (n + 15) / 16 * 4; k += 4) {
        const int4 o = tv[k];
        const int j = t0 + 4 * k;
        rank += (o.x < mine + (j < i)) + (o.y < mine + (j + 1 < i)) + (o.z < mine + (j + 2 < i)) + (o.w < mine + (j + 3 < i));
      }
    }
  }
  rank += __shfl_xor_sync(0xffffffffu, rank, 8);
  rank += __shfl_xor_sync(0xffffffffu, rank, 16);
  if (slice == 0 && i < T) {
    sorted_ids[rank] = mine;
    perm[rank] = i;
  }
}

// Step 2: a block sums EMB_CHUNK sorted tokens, whatever runs of equal ids they form: token frequencies follow a power
// law, and a block per run left one block with hundreds of dependent row reads while the chip idled.  Eight row loads
// are in flight at a time.  A run inside the chunk is written to its table row; the part of a run that reaches
// over the chunk's start / end goes to part[chunk][0] / part[chunk][1] in fp32, and step 3 adds those up in order.
// Measured, 8192 tokens by Zipf's law (the commonest id 480 times), N = 896: 10 us and 7 us for
// step 3, against 292 us with a block per run.
constexpr int EMB_CHUNK = 32;

// Index type I: int as step 1 leaves them, long long as the library's sort does.
template <typename I>
__device__ __forceinline__ int emb_row(I id, long long V) { return id >= 0 && id < V ? static_cast<int>(id) : EMB_NO_ROW; }

template <typename I>
__global__ void __launch_bounds__(128)
embedding_bwd_kernel(const I* __restrict__ sorted_ids, const I* __restrict__ perm, const bf16* __restrict__ dout,
                     bf16* __restrict__ dtable, float* __restrict__ part, int T, int N, long long V) {
  __shared__ int sid[EMB_CHUNK + 2], src[EMB_CHUNK];   // sid[k + 1] = id of the chunk's k-th token, with both neighbours
  const int r0 = blockIdx.x * EMB_CHUNK;
  const int n = T - r0 < EMB_CHUNK ? T - r0 : EMB_CHUNK;
  for (int k = threadIdx.x; k < EMB_CHUNK + 2; k += blockDim.x) {
    const int r = r0 + k - 1;
    sid[k] = r >= 0 && r < T ? emb_row(sorted_ids[r], V) : -1;
    if (k >= 1 && k <= n) src[k - 1] = static_cast<int>(perm[r]);
  }
  __syncthreads();
  const int v = blockIdx.y * blockDim.x + threadIdx.x;
  if (v >= N / 8) return;
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  bool whole = sid[1] != sid[0];                       // the run being summed began inside this chunk
  for (int k0 = 0; k0 < n; k0 += 8) {
    uint4 u[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (k0 + q < n) u[q] = reinterpret_cast<const uint4*>(dout + static_cast<long long>(src[k0 + q]) * N)[v];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int k = k0 + q;
      if (k >= n) break;
      float d[8];
      unpack8(u[q], d);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += d[j];
      const bool ends = sid[k + 2] != sid[k + 1];      // also at the last token, whose neighbour is -1
      if (ends || k + 1 == n) {
        if (ends && whole) {
          if (sid[k + 1] != EMB_NO_ROW) reinterpret_cast<uint4*>(dtable + static_cast<long long>(sid[k + 1]) * N)[v] = pack8(acc);
        } else {
          float4* o = reinterpret_cast<float4*>(part + (2LL * blockIdx.x + (whole ? 1 : 0)) * N) + 2 * v;
          o[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
          o[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
        whole = true;
      }
    }
  }
}

// Step 3: the block of the chunk in which a run begins that its last token does not end adds the parts of the chunks
// that follow, in their order, and writes the row.
template <typename I>
__global__ void __launch_bounds__(128)
embedding_bwd_span_kernel(const I* __restrict__ sorted_ids, bf16* __restrict__ dtable, const float* __restrict__ part, int T, int N,
                          long long V) {
  const int r0 = blockIdx.x * EMB_CHUNK, last = r0 + EMB_CHUNK - 1;
  if (last + 1 >= T) return;
  const I id = sorted_ids[last];
  if (emb_row(id, V) == EMB_NO_ROW || sorted_ids[last + 1] != id) return;
  if (r0 > 0 && sorted_ids[r0] == id && sorted_ids[r0 - 1] == id) return;     // began before this chunk
  const int v = blockIdx.y * blockDim.x + threadIdx.x;
  if (v >= N / 8) return;
  int chunks = 0;                                      // chunks after this one that begin with the run
  for (long long r = r0 + EMB_CHUNK; r < T && sorted_ids[r] == id; r += EMB_CHUNK) ++chunks;
  const float4* p = reinterpret_cast<const float4*>(part) + 2 * v;
  const long long ld = N / 4;                          // one part row in float4
  const float4 a0 = p[(2LL * blockIdx.x + 1) * ld], b0 = p[(2LL * blockIdx.x + 1) * ld + 1];
  float acc[8] = {a0.x, a0.y, a0.z, a0.w, b0.x, b0.y, b0.z, b0.w};
#pragma unroll 4
  for (int c = 1; c <= chunks; ++c) {
    const float4 a = p[2LL * (blockIdx.x + c) * ld], b = p[2LL * (blockIdx.x + c) * ld + 1];
    acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
    acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
  }
  reinterpret_cast<uint4*>(dtable + static_cast<long long>(id) * N)[v] = pack8(acc);
}

// ------------------------------------------------------------------ cross-entropy on materialised logits
// Bound by memory: the logits are read once forward (log-sum-exp) and once backward, the gradient written once.
// A thread keeps CE_BATCH 16-byte loads in flight and does one running-maximum update per batch instead of one per
// value (the update costs a second exponential, and as a chain through every value it, not memory, set the pace).
// A row starts where it starts: the values before the first 16-byte boundary and after the last are read one by
// one, so odd vocabularies and pitches take the same path.  gridDim.y blocks share a row when there are fewer rows
// than the chip has room for; forward they form a cluster and meet in the shared memory of its first block.
// Rows without a valid label take no part: their loss and gradient are zero and their logits are not read.
// Measured, 2047 x 151,936 fp32 with a fifth of the rows masked (one value per load, every row read, before):
// forward 588 -> 145 us (6.9 TB/s, part of it from L2), backward 748 -> 365 us (6.1 TB/s).
constexpr int CE_BATCH = 4;

template <typename T>
struct CeVec {
  static constexpr int N = 16 / sizeof(T);
};
__device__ __forceinline__ void ce_unpack(const uint4& u, float (&f)[4]) {
  f[0] = __uint_as_float(u.x); f[1] = __uint_as_float(u.y); f[2] = __uint_as_float(u.z); f[3] = __uint_as_float(u.w);
}
__device__ __forceinline__ void ce_unpack(const uint4& u, float (&f)[8]) { unpack8(u, f); }
__device__ __forceinline__ uint4 ce_pack(const float (&f)[4]) {
  return make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
}
__device__ __forceinline__ uint4 ce_pack(const float (&f)[8]) { return pack8(f); }
__device__ __forceinline__ float ldf(const float* p) { return *p; }
__device__ __forceinline__ float ldf(const bf16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void stf(float* p, float v) { *p = v; }
__device__ __forceinline__ void stf(bf16* p, float v) { *p = __float2bfloat16(v); }

// values in front of the first 16-byte boundary of a row (at most V)
template <typename T>
__device__ __forceinline__ int ce_head(const T* p, int V) {
  const int h = static_cast<int>(((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) / sizeof(T));
  return h < V ? h : V;
}

template <int N>
__device__ __forceinline__ float ce_max(const uint4& u) {
  if (N == 4) return fmaxf(fmaxf(__uint_as_float(u.x), __uint_as_float(u.y)), fmaxf(__uint_as_float(u.z), __uint_as_float(u.w)));
  const bf162* h = reinterpret_cast<const bf162*>(&u);
  const float2 f = __bfloat1622float2(__hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3])));
  return fmaxf(f.x, f.y);
}

// running (max, sum of exp(v - max)); an all -inf prefix keeps the sum at 0, NaN stays NaN
struct CeAcc {
  float m = -INFINITY, s = 0.f, sum = 0.f;
  __device__ __forceinline__ static float base(float m) { return m == -INFINITY ? 0.f : m; }
  __device__ __forceinline__ void merge(float om, float os, float osum) {
    const float nm = fmaxf(m, om), b = base(nm);
    s = s * __expf(m - b) + os * __expf(om - b);
    m = nm;
    sum += osum;
  }
  __device__ __forceinline__ void add(float v) {
    const float nm = fmaxf(m, v), b = base(nm);
    s = s * __expf(m - b) + __expf(v - b);
    m = nm;
    sum += v;
  }
  // packed vectors of N values, those that are `in` the row; the maximum of bf16 values is taken in pairs, before they are
  // unpacked: held unpacked, a batch of 32 takes 62 registers and leaves an SM half the blocks
  template <int N>
  __device__ __forceinline__ void add(const uint4 (&u)[CE_BATCH], const bool (&in)[CE_BATCH]) {
    float nm = m;
#pragma unroll
    for (int i = 0; i < CE_BATCH; ++i)
      if (in[i]) nm = fmaxf(nm, ce_max<N>(u[i]));
    const float b = base(nm);
    float e = 0.f;
#pragma unroll
    for (int i = 0; i < CE_BATCH; ++i)
      if (in[i]) {
        float w[N];
        ce_unpack(u[i], w);
#pragma unroll
        for (int j = 0; j < N; ++j) {
          e += __expf(w[j] - b);
          sum += w[j];
        }
      }
    s = s * __expf(m - b) + e;
    m = nm;
  }
};

template <typename T>
__global__ void __launch_bounds__(EW_THREADS)
ce_logits_kernel(const T* __restrict__ logits, const long long* __restrict__ labels, long long ld, int V,
                 long long ignore_index, float smoothing, float z_weight, float* __restrict__ loss_rows,
                 float* __restrict__ lse_out) {
  constexpr int N = CeVec<T>::N;
  __shared__ float sm[EW_THREADS / 32], ss[EW_THREADS / 32], sl[EW_THREADS / 32];
  __shared__ float part[3][8];                         // (max, sum, sum of logits) of up to eight blocks of the cluster
  const long long row = blockIdx.x;
  const long long lab = labels[row];
  if (lab == ignore_index || lab < 0 || lab >= V) {    // the same answer in every block of the row
    if (threadIdx.x == 0 && blockIdx.y == 0) {
      loss_rows[row] = 0.f;
      lse_out[row] = 0.f;
    }
    return;
  }
  // the first block's shared memory may be written only once that block is known to run: everybody arrives here, and whoever
  // writes waits before it does, a row's reading later
  cg::cluster_group cl = cg::this_cluster();
  cg::cluster_group::arrival_token started;
  if (gridDim.y > 1) started = cl.barrier_arrive();
  const T* lp = logits + row * ld;
  const int head = ce_head(lp, V), nvec = (V - head) / N, tail0 = head + nvec * N;
  const uint4* vp = reinterpret_cast<const uint4*>(lp + head);
  const int step = blockDim.x * gridDim.y;
  CeAcc a;
  int c = blockIdx.y * blockDim.x + threadIdx.x;
  uint4 u[CE_BATCH];
  if (nvec > CE_BATCH * step) {                        // (a row of one batch goes the second way with all its threads)
    const bool all[CE_BATCH] = {true, true, true, true};
    for (; c + (CE_BATCH - 1) * step < nvec; c += CE_BATCH * step) {
#pragma unroll
      for (int i = 0; i < CE_BATCH; ++i) u[i] = vp[c + i * step];
      a.add<N>(u, all);
    }
  }
  if (c < nvec) {                                      // a batch that need not be full
    bool in[CE_BATCH];
#pragma unroll
    for (int i = 0; i < CE_BATCH; ++i) {
      in[i] = c + i * step < nvec;
      if (in[i]) u[i] = vp[c + i * step];
    }
    a.add<N>(u, in);
  }
  if (blockIdx.y == 0) {                               // at most N - 1 values at either end
    const int t = static_cast<int>(threadIdx.x);
    if (t < head) a.add(ldf(lp + t));
    if (tail0 + t < V) a.add(ldf(lp + tail0 + t));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float om = __shfl_xor_sync(0xffffffffu, a.m, o), os = __shfl_xor_sync(0xffffffffu, a.s, o);
    a.merge(om, os, __shfl_xor_sync(0xffffffffu, a.sum, o));
  }
  if ((threadIdx.x & 31) == 0) {
    sm[threadIdx.x >> 5] = a.m;
    ss[threadIdx.x >> 5] = a.s;
    sl[threadIdx.x >> 5] = a.sum;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    a = CeAcc();
    for (int i = 0; i < static_cast<int>(blockDim.x >> 5); ++i) a.merge(sm[i], ss[i], sl[i]);
  }
  if (gridDim.y > 1) {
    cl.barrier_wait(std::move(started));
    if (threadIdx.x == 0) {
      float* dst = cl.map_shared_rank(&part[0][0], 0);
      dst[blockIdx.y] = a.m;
      dst[8 + blockIdx.y] = a.s;
      dst[16 + blockIdx.y] = a.sum;
    }
    cl.sync();
    if (blockIdx.y != 0) return;
    if (threadIdx.x == 0) {
      a = CeAcc();
      for (unsigned i = 0; i < gridDim.y; ++i) a.merge(part[0][i], part[1][i], part[2][i]);
    }
  }
  if (threadIdx.x == 0) {
    const float lse = a.m + __logf(a.s);
    lse_out[row] = lse;
    float loss = lse - ldf(lp + lab);
    if (smoothing != 0.f) loss = (1.f - smoothing) * loss + smoothing * (lse - a.sum / static_cast<float>(V));
    loss_rows[row] = loss + z_weight * lse * lse;
  }
}

// The gradient may be written over the logits (every thread reads its values before it stores them): no __restrict__.
template <typename T>
__global__ void __launch_bounds__(EW_THREADS)
ce_logits_grad_kernel(const T* logits, T* dlogits, const long long* __restrict__ labels, const float* __restrict__ lse_in,
                      const float* __restrict__ gscale, const float* __restrict__ gout, long long ld, long long ldd, int V,
                      long long ignore_index, float smoothing, float z_weight) {
  constexpr int N = CeVec<T>::N;
  const long long row = blockIdx.x;
  const long long lab = labels[row];
  const bool valid = lab != ignore_index && lab >= 0 && lab < V;
  const T* lp = logits + row * ld;
  T* dp = dlogits + row * ldd;
  const int at = valid ? static_cast<int>(lab) : -1;
  const float lse = lse_in[row];
  const float gs = valid ? gscale[row] * gout[0] : 0.f;
  const float coef = 1.f + 2.f * z_weight * lse;
  const float smv = smoothing / static_cast<float>(V);
  const float hit = 1.f - smoothing;
  // bf16 results: the constants of the row are folded into two multiply-adds a value (error 1e-6, far below the rounding)
  constexpr float LOG2E_F = 1.4426950408889634f;
  const float lse2 = lse * LOG2E_F, coef_gs = coef * gs, smv_gs = smv * gs, hit_gs = hit * gs;
  const auto grad = [&](float v, int c) {
    if (sizeof(T) == 2) {
      const float p = fmaf(ex2_approx(fmaf(v, LOG2E_F, -lse2)), coef_gs, -smv_gs);
      return c == at ? p - hit_gs : p;
    }
    float p = __expf(v - lse) * coef - smv;
    if (c == at) p -= hit;
    return p * gs;
  };
  // source and destination rows may start at different distances from a 16-byte boundary: value by value then
  const bool vec = ((reinterpret_cast<uintptr_t>(lp) ^ reinterpret_cast<uintptr_t>(dp)) & 15) == 0;
  const int head = vec ? ce_head(lp, V) : V, nvec = (V - head) / N, tail0 = head + nvec * N;
  const uint4* vp = reinterpret_cast<const uint4*>(lp + head);
  uint4* wp = reinterpret_cast<uint4*>(dp + head);
  const int step = blockDim.x * gridDim.y;
  const int first = blockIdx.y * blockDim.x + threadIdx.x;
  if (!valid) {
    for (int c = first; c < nvec; c += step) wp[c] = make_uint4(0u, 0u, 0u, 0u);
    for (int c = first; c < head; c += step) stf(dp + c, 0.f);
    for (int c = tail0 + first; c < V; c += step) stf(dp + c, 0.f);
    return;
  }
  const auto put = [&](const uint4& u, int v) {
    float w[N];
    ce_unpack(u, w);
#pragma unroll
    for (int j = 0; j < N; ++j) w[j] = grad(w[j], head + v * N + j);
    wp[v] = ce_pack(w);
  };
  for (int c = first; c < nvec; c += CE_BATCH * step) {
    uint4 u[CE_BATCH];
#pragma unroll
    for (int i = 0; i < CE_BATCH; ++i)
      if (c + i * step < nvec) u[i] = vp[c + i * step];
#pragma unroll
    for (int i = 0; i < CE_BATCH; ++i)
      if (c + i * step < nvec) put(u[i], c + i * step);
  }
  for (int i = first; i < head; i += step) stf(dp + i, grad(ldf(lp + i), i));
  for (int i = tail0 + first; i < V; i += step) stf(dp + i, grad(ldf(lp + i), i));
}

// ------------------------------------------------------------------ LoRA on fused projections: pack / unpack
// Up to four adapters (one per split of a fused projection) are multiplied as ONE pair of matrices:
// A_cat [R, in] (the A matrices stacked) and the block-diagonal B_big [out, R] with adapter s's scaled B in rows
// [row0_s, row0_s + nrows_s), columns [r0_s, r0_s + rank_s).  lora_pack_kernel builds both from the parameters in
// one launch; lora_unpack_kernel turns the fp32 gradients of A_cat / B_big back into one bf16 gradient per
// parameter (B's scaled like the forward), written into one flat buffer the caller slices.
struct LoraPack {
  const bf16* a[4];
  const bf16* b[4];
  int rank[4], r0[4], row0[4], nrows[4];
  float scale[4];
  long long ga_off[4], gb_off[4];      // unpack: element offsets of dA_s / dB_s in the flat gradient buffer
  int n, in, out, R;
};

__global__ void lora_pack_kernel(const LoraPack p, bf16* __restrict__ a_cat, bf16* __restrict__ b_big) {
  const long long na = static_cast<long long>(p.R) * p.in;
  const long long nb = static_cast<long long>(p.out) * p.R;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < na + nb; i += stride) {
    if (i < na) {
      const int r = static_cast<int>(i / p.in), c = static_cast<int>(i - static_cast<long long>(r) * p.in);
      bf16 v = __float2bfloat16(0.f);
#pragma unroll
      for (int s = 0; s < 4; ++s)
        if (s < p.n && r >= p.r0[s] && r < p.r0[s] + p.rank[s]) v = p.a[s][static_cast<long long>(r - p.r0[s]) * p.in + c];
      a_cat[i] = v;
    } else {
      const long long k = i - na;
      const int o = static_cast<int>(k / p.R), j = static_cast<int>(k - static_cast<long long>(o) * p.R);
      float v = 0.f;
#pragma unroll
      for (int s = 0; s < 4; ++s)
        if (s < p.n && j >= p.r0[s] && j < p.r0[s] + p.rank[s] && o >= p.row0[s] && o < p.row0[s] + p.nrows[s])
          v = __bfloat162float(p.b[s][static_cast<long long>(o - p.row0[s]) * p.rank[s] + (j - p.r0[s])]) * p.scale[s];
      b_big[k] = __float2bfloat16(v);
    }
  }
}

__global__ void lora_unpack_kernel(const LoraPack p, const float* __restrict__ da_cat, const float* __restrict__ db_big,
                                   bf16* __restrict__ flat) {
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long tid = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  for (int s = 0; s < p.n; ++s) {
    const long long na = static_cast<long long>(p.rank[s]) * p.in;
    for (long long i = tid; i < na; i += stride)                         // dA_s: a row block of dA_cat
      flat[p.ga_off[s] + i] = __float2bfloat16(da_cat[static_cast<long long>(p.r0[s]) * p.in + i]);
    const long long nb = static_cast<long long>(p.nrows[s]) * p.rank[s];
    for (long long i = tid; i < nb; i += stride) {                       // dB_s: a block of dB_big, scaled
      const int o = static_cast<int>(i / p.rank[s]), j = static_cast<int>(i - static_cast<long long>(o) * p.rank[s]);
      flat[p.gb_off[s] + i] =
          __float2bfloat16(db_big[static_cast<long long>(p.row0[s] + o) * p.R + p.r0[s] + j] * p.scale[s]);
    }
  }
}

}  // namespace cb

// =========================================================================================== host side
namespace {
int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  }
  return n;
}
int grid_for(long long work_items, int per_block, int max_waves = 8) {
  long long b = (work_items + per_block - 1) / per_block;
  const long long cap = static_cast<long long>(sm_count()) * max_waves;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}
// Blocks that share one row of logits.  In the gradient, one is enough once the rows alone fill the chip (four blocks an SM); with
// fewer, a row is cut in 2, 4 or 8 as long as every piece keeps 4096 values.
int ce_split(long long rows, int V) {
  int split = 1;
  while (split < 8 && rows * split < 4LL * sm_count() && V / (2 * split) >= 4096) split *= 2;
  return split;
}
// In the forward pass, where a row is `nvec` 16-byte vectors, they form a cluster (a portable one has 8 at most) and meeting costs
// about a microsecond: long rows as above in pieces of 2048 vectors; very long ones in pieces of 4096 also when there are many,
// since rows that are masked leave the rest unevenly spread over one round of blocks; or rows so few that they leave half the
// SMs without a block.  Measured, bf16, one / two / four blocks a row: 16 x 32,000 6.2 / 5.4 / 4.4 us, 200 x 50,257 (one: 11 and
// more) 9.7 / 10.4, 400 x 16,384 6.3 / 8.1, 100 x 8192 3.5 / 4.4; 2047 x 151,936 fp32, a fifth of the rows masked, 173 / 145;
// 1000 x 100,000 bf16, half of them, 47 / 31.
int ce_cluster(long long rows, int nvec) {
  int split = 1;
  while (split < 8 && ((rows * split < 4LL * sm_count() && nvec / (2 * split) >= 2048) ||
                       (rows * split < 24LL * sm_count() && nvec / (2 * split) >= 4096) ||
                       (2 * rows * split <= sm_count() && nvec >= 3072 && nvec / (2 * split) >= 512)))
    split *= 2;
  return split;
}
// Threads of a block of a row of logits: with rows enough to fill the chip (four blocks an SM) as many as have a whole batch of
// vectors each, since a block of 256 for a row of a few kilobytes spends most of its time on reductions between threads without
// data (20,000 x 1000 bf16: forward 58 us with 256 threads, 22 with 32); with fewer rows, a thread a vector.
int ce_threads(long long rows, int V, int is_bf16) {
  const int nvec = V / (is_bf16 ? 8 : 4) + 1, each = rows > 4LL * sm_count() ? cb::CE_BATCH : 1;
  const int t = ((nvec + each - 1) / each + 31) / 32 * 32;
  return t < cb::EW_THREADS ? t : cb::EW_THREADS;
}
// Layout of a row of N columns (see RowLayout): vectors a thread, threads a block, rows a block; vpl = 0: too wide
// Two vectors a thread end at 320 threads, where registers and the ring still let an SM hold two blocks of the backward; built
// for 512 threads (64 registers, one block an SM) they take longer than four vectors and a ring of two (backward, 16,384 rows:
// 5376 columns 179 against 134 us, 8192 217 against 169; forward 66 / 61 and 90 / 87).
struct RowPlan {
  int vpl, threads, rows;
};
RowPlan row_plan(int N) {
  const int nvec = N / 8;
  if (nvec <= 32 * 4) return {4, cb::EW_THREADS, cb::EW_THREADS / 32};
  if (nvec <= 640) return {2, (nvec + 63) / 64 * 32, 1};
  if (nvec <= 256 * 4) return {4, (nvec + 127) / 128 * 32, 1};
  return {0, 0, 0};
}
constexpr int RMS_BWD_RING2 = 3, RMS_BWD_RING4 = 2;   // ring depth by vectors a thread
constexpr int RMS_MAX_DEVICES = 64;

// Dynamic shared memory that a backward kernel may be launched with on the current device.  A kernel's limit is one for all host
// threads, so it is raised once, to what the widest row of either layout takes with all three inputs, and never lowered again:
// set to a call's own size, it could shrink between another thread's setting and its launch, which then failed.
constexpr int RMS_BWD_SMEM_MAX = 96 * 1024;
static_assert(RMS_BWD_RING2 * 3 * 2 * 320 * 16 <= RMS_BWD_SMEM_MAX && RMS_BWD_RING4 * 3 * 4 * cb::EW_THREADS * 16 <= RMS_BWD_SMEM_MAX,
              "ring of the widest row");
template <typename K>
int allow_rms_smem(K kern, std::atomic<bool>* raised_on_device) {
  int dev = 0;
  const cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return static_cast<int>(e);
  const bool known = dev < RMS_MAX_DEVICES;
  if (known && raised_on_device[dev].load(std::memory_order_acquire)) return 0;
  const int r = static_cast<int>(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, RMS_BWD_SMEM_MAX));
  if (r == 0 && known) raised_on_device[dev].store(true, std::memory_order_release);
  return r;
}

int launch_rmsnorm_bwd(const void* dy, const void* h, const void* w, const float* rstd, const void* dres_in, void* dx,
                       float* part, int M, int N, float offset, int grid, cudaStream_t s) {
  const RowPlan pl = row_plan(N);
  const int ring = pl.vpl == 2 ? RMS_BWD_RING2 : RMS_BWD_RING4;
  size_t smem = static_cast<size_t>(ring) * (dres_in ? 3 : 2) * pl.vpl * pl.threads * 16;
  if (pl.rows > 1) smem = std::max(smem, static_cast<size_t>(pl.rows) * N * sizeof(float));
  static std::atomic<bool> raised[3][RMS_MAX_DEVICES] = {};
  const auto go = [&](auto kern, std::atomic<bool>* raised_on_device) {
    const int e = allow_rms_smem(kern, raised_on_device);
    if (e) return e;
    kern<<<grid, pl.threads, smem, s>>>(static_cast<const cb::bf16*>(dy), static_cast<const cb::bf16*>(h),
                                        static_cast<const cb::bf16*>(w), rstd, static_cast<const cb::bf16*>(dres_in),
                                        static_cast<cb::bf16*>(dx), part, M, N, offset);
    return static_cast<int>(cudaGetLastError());
  };
  if (pl.rows > 1) return go(cb::rmsnorm_bwd_kernel<4, true, RMS_BWD_RING4>, raised[0]);
  if (pl.vpl == 2) return go(cb::rmsnorm_bwd_kernel<2, false, RMS_BWD_RING2>, raised[1]);
  return go(cb::rmsnorm_bwd_kernel<4, false, RMS_BWD_RING4>, raised[2]);
}
}  // namespace

extern "C" {

int cb_rmsnorm_max_n() { return 256 * 4 * 8; }
// number of [N] fp32 partial rows the backward writes (size the scratch as blocks * N floats)
// Debug-build index checks: out[0] = first recorded code (0 = none), out[1] = offending value; clears the word.
// Returns 1 when the library was compiled with the checks, 0 otherwise.
int cb_debug_word(long long* out2) {
  long long h[2] = {0, 0};
  if (cudaMemcpyFromSymbol(h, g_cb_debug_word, sizeof(h)) != cudaSuccess) return -1;
  out2[0] = h[0];
  out2[1] = h[1];
  const long long z[2] = {0, 0};
  cudaMemcpyToSymbol(g_cb_debug_word, z, sizeof(z));
#ifdef CHRONICALS_DEBUG_BOUNDS
  return 1;
#else
  return 0;
#endif
}

int cb_rmsnorm_bwd_blocks(int M, int N) {
  const RowPlan pl = row_plan(N);
  if (pl.vpl == 0) return 0;
  // as many blocks as an SM's shared memory holds (16,384 x 5120: 145 us with one, 109 with two, 120 in a wave and a
  // half): two of 256 threads with four vectors each, else as many as make 672 threads
  const int per_sm = pl.vpl == 4 ? 2 : std::min(6, 672 / pl.threads);
  return grid_for(M, pl.rows, per_sm);
}

int cb_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* h_out, float* rstd, int M, int N,
                   float eps, float offset, void* stream) {
  if (N % 8 != 0) return -1;
  const RowPlan pl = row_plan(N);
  if (pl.vpl == 0) return -2;
  // enough short blocks that the last ones even out (16,384 x 5120: 65 us with 8 an SM, 58 with 16, 60 with one a row)
  const int grid = grid_for(M, pl.rows, 16);
  const auto go = [&](auto kern) {
    kern<<<grid, pl.threads, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const cb::bf16*>(x), static_cast<const cb::bf16*>(res), static_cast<const cb::bf16*>(w),
        static_cast<cb::bf16*>(y), static_cast<cb::bf16*>(h_out), rstd, M, N, eps, offset);
    return static_cast<int>(cudaGetLastError());
  };
  if (pl.rows > 1) return go(cb::rmsnorm_fwd_kernel<4, true>);
  if (pl.vpl == 2) return go(cb::rmsnorm_fwd_kernel<2, false>);
  return go(cb::rmsnorm_fwd_kernel<4, false>);
}

// dw_part: scratch of cb_rmsnorm_bwd_blocks(M, N) * N floats.
int cb_rmsnorm_bwd(const void* dy, const void* h, const void* w, const float* rstd, const void* dres_in, void* dx,
                   void* dw, float* dw_part, int M, int N, float offset, int accumulate_dw, void* stream) {
  if (N % 8 != 0) return -1;
  if (row_plan(N).vpl == 0) return -2;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int grid = cb_rmsnorm_bwd_blocks(M, N);
  const int e = launch_rmsnorm_bwd(dy, h, w, rstd, dres_in, dx, dw_part, M, N, offset, grid, s);
  if (e) return e;
  if (dw != nullptr)
    cb::rmsnorm_dw_reduce_kernel<<<(N + 31) / 32, 1024, 0, s>>>(dw_part, grid, N, static_cast<cb::bf16*>(dw), accumulate_dw);
  return static_cast<int>(cudaGetLastError());
}

// out[n] (bf16) = sum over rows of x[row, n]; x bf16 [M, N] with pitch ld (N and ld multiples of 8);
// part: fp32 scratch of cb_colsum_blocks(M) * N elements.
int cb_colsum_blocks(long long M) {
  long long b = (M + 15) / 16;
  const long long cap = static_cast<long long>(sm_count()) * 4;
  if (b > cap) b = cap;
  return static_cast<int>(b < 1 ? 1 : b);
}

int cb_colsum_bf16(const void* x, void* out, float* part, long long M, int N, long long ld, void* stream) {
  if (M <= 0 || N <= 0 || N % 8 != 0 || ld % 8 != 0) return -1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int blocks = cb_colsum_blocks(M);
  const int nvec = N / 8;
  dim3 grid(blocks, (nvec + cb::EW_THREADS - 1) / cb::EW_THREADS);
  cb::colsum_partial_kernel<<<grid, cb::EW_THREADS, 0, s>>>(static_cast<const cb::bf16*>(x), ld, M, N, part);
  cb::rmsnorm_dw_reduce_kernel<<<(N + 31) / 32, 1024, 0, s>>>(part, blocks, N, static_cast<cb::bf16*>(out), 0);
  return static_cast<int>(cudaGetLastError());
}

int cb_glu_fwd(const void* gate, const void* up, void* out, long long M, int I, long long ld_in, long long ld_out,
               int gelu, void* stream) {
  if (I % 8 != 0 || ld_in % 8 != 0 || ld_out % 8 != 0) return -1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int grid = grid_for(M * (I / 8), cb::EW_THREADS, 16);
  const cb::bf16* g = static_cast<const cb::bf16*>(gate);
  const cb::bf16* u = static_cast<const cb::bf16*>(up);
  if (gelu) cb::glu_fwd_kernel<1><<<grid, cb::EW_THREADS, 0, s>>>(g, u, static_cast<cb::bf16*>(out), M, I, ld_in, ld_out);
  else cb::glu_fwd_kernel<0><<<grid, cb::EW_THREADS, 0, s>>>(g, u, static_cast<cb::bf16*>(out), M, I, ld_in, ld_out);
  return static_cast<int>(cudaGetLastError());
}

int cb_glu_bwd(const void* dout, const void* gate, const void* up, void* dgate, void* dup, long long M, int I,
               long long ld_dout, long long ld_in, long long ld_din, int gelu, void* stream) {
  if (I % 8 != 0 || ld_in % 8 != 0 || ld_dout % 8 != 0 || ld_din % 8 != 0) return -1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int grid = grid_for(M * (I / 8), cb::EW_THREADS, 16);
  const cb::bf16* d = static_cast<const cb::bf16*>(dout);
  const cb::bf16* g = static_cast<const cb::bf16*>(gate);
  const cb::bf16* u = static_cast<const cb::bf16*>(up);
  if (gelu) cb::glu_bwd_kernel<1><<<grid, cb::EW_THREADS, 0, s>>>(d, g, u, static_cast<cb::bf16*>(dgate), static_cast<cb::bf16*>(dup), M, I, ld_dout, ld_in, ld_din);
  else cb::glu_bwd_kernel<0><<<grid, cb::EW_THREADS, 0, s>>>(d, g, u, static_cast<cb::bf16*>(dgate), static_cast<cb::bf16*>(dup), M, I, ld_dout, ld_in, ld_din);
  return static_cast<int>(cudaGetLastError());
}

// table_len: number of positions in the cos/sin tables; positions outside [0, table_len) are clamped.
int cb_qk_rope(void* q, void* k, const float* cosT, const float* sinT, const long long* pos, long long T, int hq,
               int hk, int D, long long ldq, long long ldk, int interleaved, int inverse, long long table_len,
               void* stream) {
  if (D % 16 != 0 || ldq % 8 != 0 || ldk % 8 != 0 || table_len <= 0) return -1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const long long total = T * (hq + hk) * (D / 16);
  const int grid = grid_for(total, cb::EW_THREADS, 16);
  const float sign = inverse ? -1.f : 1.f;
  if (interleaved) cb::qk_rope_kernel<1><<<grid, cb::EW_THREADS, 0, s>>>(static_cast<cb::bf16*>(q), static_cast<cb::bf16*>(k), cosT, sinT, pos, T, hq, hk, D, ldq, ldk, sign, table_len);
  else cb::qk_rope_kernel<0><<<grid, cb::EW_THREADS, 0, s>>>(static_cast<cb::bf16*>(q), static_cast<cb::bf16*>(k), cosT, sinT, pos, T, hq, hk, D, ldq, ldk, sign, table_len);
  return static_cast<int>(cudaGetLastError());
}

int cb_embedding_fwd(const long long* ids, const void* table, void* out, long long T, int N, long long V, void* stream) {
  if (N % 8 != 0) return -1;
  const int grid = grid_for(T, 1, 32);
  cb::embedding_fwd_kernel<<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(ids, static_cast<const cb::bf16*>(table), static_cast<cb::bf16*>(out), T, N, V);
  return static_cast<int>(cudaGetLastError());
}

// Most tokens that cb_embedding_rank_fill sorts itself; more of them are sorted by the caller.  Counting grows with the square
// of the tokens (counting / the library's sort, whole backward: 8192 tokens, 32,000 x 896: 56 / 128 us, 20,480 124 / 138, 22,528
// 134 / 140, 24,576 175 / 142, 32,768 267 / 150; 500 x 256: 22,528 122 / 122, 24,576 130 / 122).
int cb_embedding_rank_max() { return 22528; }

// Zeroes dtable [V, N] and, with sorted_ids / perm given (T int32 each), sorts the T ids (stable).
int cb_embedding_rank_fill(const long long* ids, int* sorted_ids, int* perm, void* dtable, long long T, int N, long long V,
                           void* stream) {
  if (N % 8 != 0 || T <= 0 || V <= 0 || V >= cb::EMB_NO_ROW) return -1;
  if (sorted_ids != nullptr && T > cb_embedding_rank_max()) return -2;
  const int rank_blocks = sorted_ids != nullptr ? static_cast<int>((T + cb::EMB_RANK_TOKENS - 1) / cb::EMB_RANK_TOKENS) : 0;
  const long long vecs = V * (N / 8);
  const int fill_blocks = grid_for(vecs, cb::EW_THREADS, 8);
  cb::embedding_rank_fill_kernel<<<rank_blocks + fill_blocks, cb::EW_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
      ids, sorted_ids, perm, static_cast<int>(T), rank_blocks, static_cast<uint4*>(dtable), vecs, V);
  return static_cast<int>(cudaGetLastError());
}

// Rows of N floats that `part` of cb_embedding_bwd holds for T tokens.
int cb_embedding_part_rows(long long T) { return static_cast<int>(2 * ((T + cb::EMB_CHUNK - 1) / cb::EMB_CHUNK)); }

// dtable [V, N] (zeroed) receives the sums of the rows of dout [T, N] over equal ids; sorted_ids ascending (ids outside [0, V)
// are no row of the table), perm the source token of each; both int32, or int64 with `wide`.
int cb_embedding_bwd(const void* sorted_ids, const void* perm, const void* dout, void* dtable, float* part, long long T, int N,
                     long long V, int wide, void* stream) {
  if (N % 8 != 0 || T <= 0 || T > 0x7fffff00LL || V <= 0 || V >= cb::EMB_NO_ROW) return -1;
  const dim3 grid(static_cast<unsigned>((T + cb::EMB_CHUNK - 1) / cb::EMB_CHUNK), (N / 8 + 127) / 128);
  const auto go = [&](const auto* ids, const auto* from) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cb::bf16* out = static_cast<cb::bf16*>(dtable);
    cb::embedding_bwd_kernel<<<grid, 128, 0, s>>>(ids, from, static_cast<const cb::bf16*>(dout), out, part, static_cast<int>(T), N, V);
    cb::embedding_bwd_span_kernel<<<grid, 128, 0, s>>>(ids, out, part, static_cast<int>(T), N, V);
    return static_cast<int>(cudaGetLastError());
  };
  if (wide) return go(static_cast<const long long*>(sorted_ids), static_cast<const long long*>(perm));
  return go(static_cast<const int*>(sorted_ids), static_cast<const int*>(perm));
}

int cb_ce_logits(const void* logits, const long long* labels, long long rows, long long ld, int V, int is_bf16,
                 long long ignore_index, float smoothing, float z_weight, float* loss_rows, float* lse, void* stream) {
  if (rows <= 0) return -1;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  const int split = ce_cluster(rows, V / (is_bf16 ? 8 : 4));
  cfg.gridDim = dim3(static_cast<unsigned>(rows), split);
  cfg.blockDim = dim3(ce_threads(rows, V, is_bf16));
  cfg.stream = static_cast<cudaStream_t>(stream);
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = split;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = split > 1 ? 1 : 0;
  if (is_bf16)
    return static_cast<int>(cudaLaunchKernelEx(&cfg, cb::ce_logits_kernel<cb::bf16>, static_cast<const cb::bf16*>(logits), labels,
                                               ld, V, ignore_index, smoothing, z_weight, loss_rows, lse));
  return static_cast<int>(cudaLaunchKernelEx(&cfg, cb::ce_logits_kernel<float>, static_cast<const float*>(logits), labels, ld, V,
                                             ignore_index, smoothing, z_weight, loss_rows, lse));
}

// ld / ldd: row pitches of the logits and of the gradient
int cb_ce_logits_grad(const void* logits, void* dlogits, const long long* labels, const float* lse, const float* gscale,
                      const float* gout, long long rows, long long ld, long long ldd, int V, int is_bf16,
                      long long ignore_index, float smoothing, float z_weight, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (rows <= 0) return -1;
  const dim3 grid(static_cast<unsigned>(rows), ce_split(rows, V));
  if (is_bf16) cb::ce_logits_grad_kernel<cb::bf16><<<grid, ce_threads(rows, V, 1), 0, s>>>(static_cast<const cb::bf16*>(logits), static_cast<cb::bf16*>(dlogits), labels, lse, gscale, gout, ld, ldd, V, ignore_index, smoothing, z_weight);
  else cb::ce_logits_grad_kernel<float><<<grid, ce_threads(rows, V, 0), 0, s>>>(static_cast<const float*>(logits), static_cast<float*>(dlogits), labels, lse, gscale, gout, ld, ldd, V, ignore_index, smoothing, z_weight);
  return static_cast<int>(cudaGetLastError());
}

// desc: host array of 4 x {a_ptr, b_ptr} (u64), then int arrays rank[4], r0[4], row0[4], nrows[4], then float scale[4]
// are passed separately to keep the ctypes side simple.
static int fill_lora_pack(cb::LoraPack* p, const unsigned long long* a_ptrs, const unsigned long long* b_ptrs,
                          const int* rank, const int* row0, const int* nrows, const float* scale, int n, int in, int out) {
  if (n < 1 || n > 4 || in <= 0 || out <= 0) return -1;
  memset(p, 0, sizeof(*p));
  int r0 = 0;
  long long off = 0;
  for (int s = 0; s < n; ++s) {
    p->a[s] = reinterpret_cast<const cb::bf16*>(a_ptrs[s]);
    p->b[s] = reinterpret_cast<const cb::bf16*>(b_ptrs[s]);
    p->rank[s] = rank[s]; p->r0[s] = r0; p->row0[s] = row0[s]; p->nrows[s] = nrows[s]; p->scale[s] = scale[s];
    if (rank[s] <= 0 || row0[s] < 0 || nrows[s] <= 0 || row0[s] + nrows[s] > out) return -1;
    p->ga_off[s] = off; off += static_cast<long long>(rank[s]) * in;
    p->gb_off[s] = off; off += static_cast<long long>(nrows[s]) * rank[s];
    r0 += rank[s];
  }
  p->n = n; p->in = in; p->out = out; p->R = r0;
  return 0;
}

// a_cat [R, in] and b_big [out, R] (bf16, contiguous) from n adapters; R = sum of the ranks.
int cb_lora_pack(const unsigned long long* a_ptrs, const unsigned long long* b_ptrs, const int* rank, const int* row0,
                 const int* nrows, const float* scale, int n, int in, int out, void* a_cat, void* b_big, void* stream) {
  cb::LoraPack p;
  if (fill_lora_pack(&p, a_ptrs, b_ptrs, rank, row0, nrows, scale, n, in, out)) return -1;
  const long long work = static_cast<long long>(p.R) * in + static_cast<long long>(out) * p.R;
  cb::lora_pack_kernel<<<grid_for(work, cb::EW_THREADS, 4), cb::EW_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
      p, static_cast<cb::bf16*>(a_cat), static_cast<cb::bf16*>(b_big));
  return static_cast<int>(cudaGetLastError());
}

// flat (bf16) receives dA_0 | dB_0 | dA_1 | dB_1 | ... from the fp32 gradients of a_cat [R, in] and b_big [out, R].
int cb_lora_unpack(const int* rank, const int* row0, const int* nrows, const float* scale, int n, int in, int out,
                   const float* da_cat, const float* db_big, void* flat, void* stream) {
  cb::LoraPack p;
  unsigned long long dummy[4] = {0, 0, 0, 0};
  if (fill_lora_pack(&p, dummy, dummy, rank, row0, nrows, scale, n, in, out)) return -1;
  long long work = 0;
  for (int s = 0; s < n; ++s) work = std::max(work, std::max(static_cast<long long>(rank[s]) * in, static_cast<long long>(nrows[s]) * rank[s]));
  cb::lora_unpack_kernel<<<grid_for(work, cb::EW_THREADS, 4), cb::EW_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
      p, da_cat, db_big, static_cast<cb::bf16*>(flat));
  return static_cast<int>(cudaGetLastError());
}

}  // extern "C"

// =========================================================================================== allocation-free entry point
// RMSNorm backward for callers that must not allocate (see chronicals_b200_noalloc.h).  The per-block
// dW partials, which cb_rmsnorm_bwd takes from a caller-allocated buffer, live in a file-scope device
// array here.  The array's name is only a host-side handle: its device address is fetched once per
// device with cudaGetSymbolAddress and that pointer is what the kernels receive.
#include "chronicals_b200_noalloc.h"

#include <mutex>

namespace {

constexpr int NOALLOC_MAX_BLOCKS = CB_NOALLOC_RMSNORM_MAX_BLOCKS;
constexpr int NOALLOC_MAX_N = CB_NOALLOC_RMSNORM_MAX_N;
constexpr int NOALLOC_MAX_DEVICES = 64;

static __device__ __align__(256) float g_noalloc_dw_partials[NOALLOC_MAX_BLOCKS * NOALLOC_MAX_N];

std::mutex g_noalloc_mutex;
float* g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {};

// device address of the scratch array on the current device; resolved on first use per device
int noalloc_scratch(float** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return -3;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (g_noalloc_ptr[dev] == nullptr) {
    float* p = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_dw_partials);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (p == nullptr) return -4;
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return 0;
}

}  // namespace

extern "C" {

int cb_rmsnorm_bwd_noalloc_max_n() { return NOALLOC_MAX_N; }

int cb_rmsnorm_bwd_noalloc(const void* dy, const void* h, const void* w, const float* rstd, const void* dres_in,
                           void* dx, void* dw, int M, int N, float offset, int accumulate_dw, void* stream) {
  if (M <= 0 || N <= 0 || N % 8 != 0) return -1;
  if (N > NOALLOC_MAX_N) return -2;                     // beyond the built-in scratch: use cb_rmsnorm_bwd
  const RowPlan pl = row_plan(N);
  if (pl.vpl == 0) return -2;
  float* part = nullptr;
  const int rc = noalloc_scratch(&part);
  if (rc != 0) return rc;
  int grid = grid_for(M, pl.rows, 1);
  if (grid > NOALLOC_MAX_BLOCKS) grid = NOALLOC_MAX_BLOCKS;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // every block writes all N entries of its own partial row before the reduction reads them, so
  // nothing left in the array by an earlier call can leak into this one
  const int e = launch_rmsnorm_bwd(dy, h, w, rstd, dres_in, dx, part, M, N, offset, grid, s);
  if (e) return e;
  if (dw != nullptr)
    cb::rmsnorm_dw_reduce_kernel<<<(N + 31) / 32, 1024, 0, s>>>(part, grid, N, static_cast<cb::bf16*>(dw), accumulate_dw);
  return static_cast<int>(cudaGetLastError());
}

}  // extern "C"
