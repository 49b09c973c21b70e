// Bandwidth-bound kernels for sm_100a: RMSNorm fwd/bwd (+residual-grad add, +re-emit), RoPE
// (rotate-half, partial, MRoPE), SwiGLU / GeGLU fwd/bwd, fused softmax cross-entropy, embedding
// gather / sorted scatter-add, multi-tensor AdamW, gated RMSNorm, L2 norm, top-k router.
// They replace the reference project's Triton kernels (flextrain/ops/_kernels/*.py). All use
// 16-byte vector accesses and keep a row in registers between the reduction and the write.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace {

typedef __nv_bfloat16 bf16;
typedef __nv_bfloat162 bf162;

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
template <int NW>
__device__ __forceinline__ float block_sum(float v, float* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  float t = (l < NW) ? sh[l] : 0.f;
  return warp_sum(t);
}
template <int NW>
__device__ __forceinline__ float block_max(float v, float* sh) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  float t = (l < NW) ? sh[l] : -INFINITY;
  return warp_max(t);
}

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const bf162* h = reinterpret_cast<const bf162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  bf162* h = reinterpret_cast<bf162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}

// ----------------------------------------------------------------------------- RMSNorm
// One CTA (256 threads) walks rows; a row of up to 8*256*MAXV elements lives in registers.
constexpr int RN_THREADS = 256;
constexpr int RN_MAXV = 8;  // D <= 16384

template <int MAXV>
__global__ void __launch_bounds__(RN_THREADS) rmsnorm_fwd_kernel(const bf16* __restrict__ x,
                                                                  const float* __restrict__ w, bf16* __restrict__ y,
                                                                  float* __restrict__ rstd_out, int T, int D,
                                                                  float eps, long ldx) {
  __shared__ float sh[32];
  const int nv = D >> 3;
  for (int row = blockIdx.x; row < T; row += gridDim.x) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * ldx);
    uint4 v[MAXV];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int i = threadIdx.x + j * RN_THREADS;
      if (i < nv) {
        v[j] = xr[i];
        float f[8];
        unpack8(v[j], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
      }
    }
    ss = block_sum<RN_THREADS / 32>(ss, sh);
    const float r = rsqrtf(ss / (float)D + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = r;
    uint4* yr = reinterpret_cast<uint4*>(y + (size_t)row * D);
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int i = threadIdx.x + j * RN_THREADS;
      if (i < nv) {
        float f[8];
        unpack8(v[j], f);
        if (w) {
          const float4 w0 = reinterpret_cast<const float4*>(w)[2 * i];
          const float4 w1 = reinterpret_cast<const float4*>(w)[2 * i + 1];
          f[0] *= r * w0.x; f[1] *= r * w0.y; f[2] *= r * w0.z; f[3] *= r * w0.w;
          f[4] *= r * w1.x; f[5] *= r * w1.y; f[6] *= r * w1.z; f[7] *= r * w1.w;
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] *= r;
        }
        yr[i] = pack8(f);
      }
    }
  }
}

// dx = (g - xhat * mean(g . xhat)) * rstd, g = dy * w; optional dx += dx_add (residual gradient),
// optional y_out = xhat * w (forward output re-emitted for the deferred weight-gradient GEMMs);
// partial dw[blockIdx.x, :] = sum over this CTA's rows of dy * xhat (fp32), reduced by a second kernel.
template <int MAXV>
__global__ void __launch_bounds__(RN_THREADS) rmsnorm_bwd_kernel(const bf16* __restrict__ dy,
                                                                  const bf16* __restrict__ x,
                                                                  const float* __restrict__ w,
                                                                  const float* __restrict__ rstd,
                                                                  const bf16* __restrict__ dx_add,
                                                                  bf16* __restrict__ dx, bf16* __restrict__ y_out,
                                                                  float* __restrict__ dw_partial, int T, int D,
                                                                  long ldx, long lddx) {
  __shared__ float sh[32];
  const int nv = D >> 3;
  float dwacc[MAXV][8];
#pragma unroll
  for (int j = 0; j < MAXV; ++j)
#pragma unroll
    for (int e = 0; e < 8; ++e) dwacc[j][e] = 0.f;

  // The next row's operands are requested before the current row's block-wide reduction, so its DRAM latency hides
  // behind the two barriers and the arithmetic of this row (the kernel is latency-bound otherwise: one row in flight
  // per CTA).
  uint4 nx[MAXV], ng[MAXV], na[MAXV];
  float nr = 0.f;
  auto prefetch = [&](int rw) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)rw * ldx);
    const uint4* dyr = reinterpret_cast<const uint4*>(dy + (size_t)rw * D);
    nr = rstd[rw];
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int i = threadIdx.x + j * RN_THREADS;
      if (i < nv) {
        nx[j] = xr[i];
        ng[j] = dyr[i];
        if (dx_add) na[j] = reinterpret_cast<const uint4*>(dx_add + (size_t)rw * D)[i];
      }
    }
  };
  constexpr bool AHEAD = MAXV <= 2;          // wider rows would halve the CTAs per SM with two rows in registers
  if (AHEAD && blockIdx.x < T) prefetch(blockIdx.x);
  for (int row = blockIdx.x; row < T; row += gridDim.x) {
    if (!AHEAD) prefetch(row);
    const float r = nr;
    uint4 xv[MAXV], gv[MAXV], av[MAXV];
#pragma unroll
    for (int j = 0; j < MAXV; ++j) { xv[j] = nx[j]; gv[j] = ng[j]; av[j] = na[j]; }
    if (AHEAD && row + (int)gridDim.x < T) prefetch(row + gridDim.x);
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int i = threadIdx.x + j * RN_THREADS;
      if (i < nv) {
        float xf[8], gf[8], wf[8];
        unpack8(xv[j], xf);
        unpack8(gv[j], gf);
        if (w) {
          const float4 w0 = reinterpret_cast<const float4*>(w)[2 * i];
          const float4 w1 = reinterpret_cast<const float4*>(w)[2 * i + 1];
          wf[0] = w0.x; wf[1] = w0.y; wf[2] = w0.z; wf[3] = w0.w; wf[4] = w1.x; wf[5] = w1.y; wf[6] = w1.z; wf[7] = w1.w;
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) wf[e] = 1.f;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float xh = xf[e] * r;
          dwacc[j][e] += gf[e] * xh;
          dot += gf[e] * wf[e] * xh;
        }
      }
    }
    dot = block_sum<RN_THREADS / 32>(dot, sh) / (float)D;
    uint4* dxr = reinterpret_cast<uint4*>(dx + (size_t)row * lddx);
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int i = threadIdx.x + j * RN_THREADS;
      if (i < nv) {
        float xf[8], gf[8], wf[8], o[8];
        unpack8(xv[j], xf);
        unpack8(gv[j], gf);
        if (w) {
          const float4 w0 = reinterpret_cast<const float4*>(w)[2 * i];
          const float4 w1 = reinterpret_cast<const float4*>(w)[2 * i + 1];
          wf[0] = w0.x; wf[1] = w0.y; wf[2] = w0.z; wf[3] = w0.w; wf[4] = w1.x; wf[5] = w1.y; wf[6] = w1.z; wf[7] = w1.w;
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) wf[e] = 1.f;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = (gf[e] * wf[e] - xf[e] * r * dot) * r;
        if (dx_add) {
          float a[8];
          unpack8(av[j], a);
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] += a[e];
        }
        dxr[i] = pack8(o);
        if (y_out) {
          float yv[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) yv[e] = xf[e] * r * wf[e];
          reinterpret_cast<uint4*>(y_out + (size_t)row * D)[i] = pack8(yv);
        }
      }
    }
  }
  if (dw_partial) {
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int i = threadIdx.x + j * RN_THREADS;
      if (i < nv) {
        float* o = dw_partial + (size_t)blockIdx.x * D + i * 8;
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = dwacc[j][e];
      }
    }
  }
}

// Forward of rows of up to 2048 elements: a warp per row, NV 16-byte pieces a lane, no barriers.  A block per row, as above, leaves
// most of its 256 threads without a piece there (96 of 768 / 8) and has one row in flight between two barriers.
// us, block per row / so, forward: 16384 x 768 22.7 / 9.9, 9377 x 1024 14.6 / 8.2, 16384 x 2048 28.7 / 25.4; backward with its sum
// of dw: 58.6 / 28.6, 37.9 / 22.6, 79.3 / 66.5, 8192 x 1152 36.6 / 24.7, 16384 x 3072 98.2 / 89.3.
template <int NV>
__global__ void __launch_bounds__(RN_THREADS) rmsnorm_warp_fwd_kernel(const bf16* __restrict__ x, const float* __restrict__ w,
                                                                      bf16* __restrict__ y, float* __restrict__ rstd_out, int T,
                                                                      int D, float eps, long ldx) {
  const int lane = threadIdx.x & 31, nv = D >> 3, step = gridDim.x * (RN_THREADS / 32);
  for (int row = blockIdx.x * (RN_THREADS / 32) + (threadIdx.x >> 5); row < T; row += step) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * ldx);
    uint4 v[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + j * 32;
      v[j] = i < nv ? xr[i] : make_uint4(0, 0, 0, 0);
    }
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      float f[8];
      unpack8(v[j], f);
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
    }
    const float r = rsqrtf(warp_sum(ss) / (float)D + eps);
    if (lane == 0 && rstd_out) rstd_out[row] = r;
    uint4* yr = reinterpret_cast<uint4*>(y + (size_t)row * D);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + j * 32;
      if (i < nv) {
        float f[8];
        unpack8(v[j], f);
        if (w) {
          const float4 w0 = reinterpret_cast<const float4*>(w)[2 * i];
          const float4 w1 = reinterpret_cast<const float4*>(w)[2 * i + 1];
          f[0] *= r * w0.x; f[1] *= r * w0.y; f[2] *= r * w0.z; f[3] *= r * w0.w;
          f[4] *= r * w1.x; f[5] *= r * w1.y; f[6] *= r * w1.z; f[7] *= r * w1.w;
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] *= r;
        }
        yr[i] = pack8(f);
      }
    }
  }
}

// The backward of rows of up to 3072: WPR warps to a row (one up to 768 elements, two up to 1536, four), which meet once a row.  NV
// stays at three: the operands of a row, the gain and the sums of dw are in registers together, and two blocks an SM have to
// keep enough rows on their way (a warp for 2048 took 241 registers and 88 us).  The groups of a block add up their parts of dw
// one after the other (a fixed order).
template <int NV, int WPR>
__global__ void __launch_bounds__(RN_THREADS, 2) rmsnorm_warp_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x,
                                                                      const float* __restrict__ w, const float* __restrict__ rstd,
                                                                      const bf16* __restrict__ dx_add, bf16* __restrict__ dx,
                                                                      bf16* __restrict__ y_out, float* __restrict__ dw_partial, int T,
                                                                      int D, long ldx, long lddx) {
  constexpr int LANES = 32 * WPR, GROUPS = RN_THREADS / LANES;
  __shared__ __align__(16) float dw_s[NV * LANES * 8];
  __shared__ float dot_s[2][RN_THREADS / 32];
  const int lane = threadIdx.x % LANES, group = threadIdx.x / LANES, nv = D >> 3, step = gridDim.x * GROUPS;
  int turn = 0;
  float dwacc[NV][8];
#pragma unroll
  for (int j = 0; j < NV; ++j)
#pragma unroll
    for (int e = 0; e < 8; ++e) dwacc[j][e] = 0.f;
  auto gain = [&](int i, float (&wf)[8]) {
    if (w) {
      const float4 w0 = reinterpret_cast<const float4*>(w)[2 * i];
      const float4 w1 = reinterpret_cast<const float4*>(w)[2 * i + 1];
      wf[0] = w0.x; wf[1] = w0.y; wf[2] = w0.z; wf[3] = w0.w; wf[4] = w1.x; wf[5] = w1.y; wf[6] = w1.z; wf[7] = w1.w;
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) wf[e] = 1.f;
    }
  };
  for (int row = blockIdx.x * GROUPS + group; row < T; row += step) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * ldx);
    const uint4* gr = reinterpret_cast<const uint4*>(dy + (size_t)row * D);
    const uint4* ar = reinterpret_cast<const uint4*>(dx_add + (size_t)row * D);
    const uint4 zero = make_uint4(0, 0, 0, 0);
    uint4 xv[NV], gv[NV], av[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + j * LANES;
      xv[j] = i < nv ? xr[i] : zero;
      gv[j] = i < nv ? gr[i] : zero;
      if (dx_add) av[j] = i < nv ? ar[i] : zero;
    }
    const float r = rstd[row];
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + j * LANES;
      if (i < nv) {
        float xf[8], gf[8], wf[8];
        unpack8(xv[j], xf);
        unpack8(gv[j], gf);
        gain(i, wf);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float xh = xf[e] * r;
          dwacc[j][e] += gf[e] * xh;
          dot += gf[e] * wf[e] * xh;
        }
      }
    }
    dot = warp_sum(dot);
    if constexpr (WPR > 1) {                       // (two buffers: the next row's sums do not meet this row's readers)
      if ((threadIdx.x & 31) == 0) dot_s[turn][threadIdx.x >> 5] = dot;
      asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(LANES) : "memory");
      dot = 0.f;
#pragma unroll
      for (int u = 0; u < WPR; ++u) dot += dot_s[turn][group * WPR + u];
      turn ^= 1;
    }
    dot /= (float)D;
    uint4* dxr = reinterpret_cast<uint4*>(dx + (size_t)row * lddx);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + j * LANES;
      if (i < nv) {
        float xf[8], gf[8], wf[8], o[8];
        unpack8(xv[j], xf);
        unpack8(gv[j], gf);
        gain(i, wf);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = (gf[e] * wf[e] - xf[e] * r * dot) * r;
        if (dx_add) {
          float a[8];
          unpack8(av[j], a);
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] += a[e];
        }
        dxr[i] = pack8(o);
        if (y_out) {
          float yv[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) yv[e] = xf[e] * r * wf[e];
          reinterpret_cast<uint4*>(y_out + (size_t)row * D)[i] = pack8(yv);
        }
      }
    }
  }
  if (dw_partial) {
    for (int t = 0; t < GROUPS; ++t) {
      if (group == t) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          float4* s = reinterpret_cast<float4*>(dw_s + (lane + j * LANES) * 8);
          float4 a = t ? s[0] : make_float4(0.f, 0.f, 0.f, 0.f), b = t ? s[1] : make_float4(0.f, 0.f, 0.f, 0.f);
          a.x += dwacc[j][0]; a.y += dwacc[j][1]; a.z += dwacc[j][2]; a.w += dwacc[j][3];
          b.x += dwacc[j][4]; b.y += dwacc[j][5]; b.z += dwacc[j][6]; b.w += dwacc[j][7];
          s[0] = a;
          s[1] = b;
        }
      }
      __syncthreads();
    }
    for (int c = threadIdx.x; c < D; c += RN_THREADS) dw_partial[(size_t)blockIdx.x * D + c] = dw_s[c];
  }
}

// out[c] (+)= sum over P partial rows.  A block owns 32 columns and adds 32 rows at a time; one thread per column, walking the
// rows by itself, left all but D / 256 SMs idle: 592 x 1024 28 us, 5 us so.
__global__ void __launch_bounds__(1024) colsum_accum_kernel(const float* __restrict__ partial, float* __restrict__ out, int P,
                                                            int D, int accumulate) {
  __shared__ float sh[32][33];
  const int lane = threadIdx.x & 31, r = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < D) {
#pragma unroll 4
    for (int p = r; p < P; p += 32) s += partial[(size_t)p * D + c];
  }
  sh[r][lane] = s;
  __syncthreads();
  s = warp_sum(sh[lane][r]);                        // warp r adds column r of the block
  const int o = blockIdx.x * 32 + r;
  if (lane == 0 && o < D) out[o] = accumulate ? out[o] + s : s;
}

// Small-D (per-head) RMSNorm: one warp per row of D <= 512 elements (QK-norm, D = head_dim).
__global__ void rmsnorm_small_fwd_kernel(const bf16* __restrict__ x, const float* __restrict__ w, bf16* __restrict__ y,
                                         float* __restrict__ rstd_out, long rows, int D, int heads_w, float eps) {
  const long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const bf16* xr = x + row * D;
  float ss = 0.f;
  for (int i = lane * 2; i < D; i += 64) {
    const float2 t = __bfloat1622float2(*reinterpret_cast<const bf162*>(xr + i));
    ss += t.x * t.x + t.y * t.y;
  }
  ss = warp_sum(ss);
  const float r = rsqrtf(ss / (float)D + eps);
  if (lane == 0 && rstd_out) rstd_out[row] = r;
  // heads_w > 1: weight has one row per head (full-row QK-norm over H*hd is handled by the big kernel).
  const float* wr = w ? w + (heads_w > 1 ? (row % heads_w) * D : 0) : nullptr;
  bf16* yr = y + row * D;
  for (int i = lane * 2; i < D; i += 64) {
    float2 t = __bfloat1622float2(*reinterpret_cast<const bf162*>(xr + i));
    t.x *= r * (wr ? wr[i] : 1.f);
    t.y *= r * (wr ? wr[i + 1] : 1.f);
    *reinterpret_cast<bf162*>(yr + i) = __floats2bfloat162_rn(t.x, t.y);
  }
}

__global__ void rmsnorm_small_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x,
                                         const float* __restrict__ w, const float* __restrict__ rstd,
                                         bf16* __restrict__ dx, float* __restrict__ dw, long rows, int D) {
  // One warp per row, grid-stride over rows.  dw (D,) partial sums stay in registers while a warp walks its rows
  // (D <= 512: 8 pairs per lane), are combined across the CTA's warps in shared memory and leave with ONE atomic per
  // element per CTA; a per-row atomic on D hot addresses serialises the whole grid.
  constexpr int MAXP = 8;
  extern __shared__ float dw_sh[];                 // D floats
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  float2 acc[MAXP];
#pragma unroll
  for (int p = 0; p < MAXP; ++p) acc[p] = make_float2(0.f, 0.f);
  for (int i = threadIdx.x; i < D; i += blockDim.x) dw_sh[i] = 0.f;
  __syncthreads();
  for (long row = (long)blockIdx.x * wpb + (threadIdx.x >> 5); row < rows; row += (long)gridDim.x * wpb) {
    const bf16* xr = x + row * D;
    const bf16* gr = dy + row * D;
    const float r = rstd[row];
    float dot = 0.f;
    for (int i = lane * 2; i < D; i += 64) {
      const float2 xv = __bfloat1622float2(*reinterpret_cast<const bf162*>(xr + i));
      const float2 gv = __bfloat1622float2(*reinterpret_cast<const bf162*>(gr + i));
      const float w0 = w ? w[i] : 1.f, w1 = w ? w[i + 1] : 1.f;
      dot += gv.x * w0 * xv.x * r + gv.y * w1 * xv.y * r;
    }
    dot = warp_sum(dot) / (float)D;
    bf16* dxr = dx + row * D;
#pragma unroll
    for (int p = 0; p < MAXP; ++p) {
      const int i = lane * 2 + p * 64;
      if (i < D) {
        const float2 xv = __bfloat1622float2(*reinterpret_cast<const bf162*>(xr + i));
        const float2 gv = __bfloat1622float2(*reinterpret_cast<const bf162*>(gr + i));
        const float w0 = w ? w[i] : 1.f, w1 = w ? w[i + 1] : 1.f;
        const float o0 = (gv.x * w0 - xv.x * r * dot) * r;
        const float o1 = (gv.y * w1 - xv.y * r * dot) * r;
        *reinterpret_cast<bf162*>(dxr + i) = __floats2bfloat162_rn(o0, o1);
        acc[p].x += gv.x * xv.x * r;
        acc[p].y += gv.y * xv.y * r;
      }
    }
  }
  if (dw) {
#pragma unroll
    for (int p = 0; p < MAXP; ++p) {
      const int i = lane * 2 + p * 64;
      if (i < D) {
        atomicAdd(&dw_sh[i], acc[p].x);
        atomicAdd(&dw_sh[i + 1], acc[p].y);
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < D; i += blockDim.x) atomicAdd(dw + i, dw_sh[i]);
  }
}

// Per-head norm straight out of (and, backward, into) a fused projection's rows: HD / 8 lanes per head, 16 bytes each, in
// place of a copy of the strided view, a warp per head with 4-byte loads, and a copy back.  Bound by memory.
// 9377 tokens, 16 + 8 heads of 128, twelve layers' norms: forward 308 us and 130 of copies, 169 us so; backward 446 us and 390
// of copies in and out, 358 us so.
template <int HD>
__device__ __forceinline__ float head_sum(float v) {          // over the HD / 8 lanes of a head
#pragma unroll
  for (int o = HD / 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void load_gain8(const float* w, int i, float (&f)[8]) {
  if (w == nullptr) {
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = 1.f;
    return;
  }
  const float4 a = reinterpret_cast<const float4*>(w)[i / 4], b = reinterpret_cast<const float4*>(w)[i / 4 + 1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

template <int HD>
__global__ void __launch_bounds__(256) rmsnorm_heads_fwd_kernel(const bf16* __restrict__ x, long ldx, long hx, const float* __restrict__ w,
                                                                bf16* __restrict__ y, float* __restrict__ rstd, int rows,
                                                                int H, float eps) {
  constexpr int L = HD / 8;
  const long id = (long)blockIdx.x * 256 + threadIdx.x;
  const int row = (int)(id / L), i = (int)(id % L) * 8;
  const bool on = row < rows;
  float f[8] = {};
  if (on) {
    const int t = row / H, h = row - t * H;
    unpack8(*reinterpret_cast<const uint4*>(x + t * ldx + h * hx + i), f);
  }
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
  ss = head_sum<HD>(ss);
  if (!on) return;
  const float r = rsqrtf(ss / (float)HD + eps);
  if (i == 0) rstd[row] = r;
  float g[8];
  load_gain8(w, i, g);
#pragma unroll
  for (int e = 0; e < 8; ++e) f[e] *= r * g[e];
  *reinterpret_cast<uint4*>(y + (long)row * HD + i) = pack8(f);
}

template <int HD>
__global__ void __launch_bounds__(256) rmsnorm_heads_bwd_kernel(const bf16* __restrict__ dy, long lddy, long hdy, const bf16* __restrict__ x,
                                                                long ldx, long hx, const float* __restrict__ w,
                                                                const float* __restrict__ rstd, bf16* __restrict__ dx,
                                                                long lddx, long hdx, float* __restrict__ dw, int rows, int H) {
  constexpr int L = HD / 8, PER = 256 / L;
  __shared__ float dw_sh[HD];
  const int i = (threadIdx.x % L) * 8, sub = threadIdx.x / L;
  float g[8], acc[8] = {};
  load_gain8(w, i, g);
  for (int c = threadIdx.x; c < HD; c += 256) dw_sh[c] = 0.f;
  __syncthreads();
  for (int row0 = blockIdx.x * PER; row0 < rows; row0 += gridDim.x * PER) {      // the same number of turns for every lane
    const int row = row0 + sub;
    const bool on = row < rows;
    const int t = on ? row / H : 0, h = on ? row - t * H : 0;
    float xh[8] = {}, gv[8] = {};
    float r = 0.f;
    if (on) {
      r = rstd[row];
      unpack8(*reinterpret_cast<const uint4*>(x + t * ldx + h * hx + i), xh);
      unpack8(*reinterpret_cast<const uint4*>(dy + t * lddy + h * hdy + i), gv);
    }
    float dot = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      xh[e] *= r;
      acc[e] += gv[e] * xh[e];
      gv[e] *= g[e];
      dot += gv[e] * xh[e];
    }
    dot = head_sum<HD>(dot) / (float)HD;
    if (on) {
      float o[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = (gv[e] - xh[e] * dot) * r;
      *reinterpret_cast<uint4*>(dx + t * lddx + h * hdx + i) = pack8(o);
    }
  }
  if (dw == nullptr) return;
#pragma unroll
  for (int e = 0; e < 8; ++e) atomicAdd(&dw_sh[i + e], acc[e]);
  __syncthreads();
  for (int c = threadIdx.x; c < HD; c += 256) atomicAdd(dw + c, dw_sh[c]);
}

// -------------------------------------------------------------------------------- RoPE
// out[t,h,:] = R(pos_t) x[t,h,:] over rotate-half pairs (i, i + rot/2), i < rot/2; channels past
// 2*half_rot are copied. x / out are (T, H, hd) with independent token strides (in place when equal),
// so Q and K can be rotated straight out of a fused QKV projection buffer. positions: (T) or (T,3).
__global__ void rope_kernel(const bf16* __restrict__ x, long in_stride, bf16* __restrict__ out, long out_stride,
                            const int* __restrict__ pos, const float* __restrict__ inv_freq, int T, int H, int hd,
                            int half_rot, int inverse, int pos_stride, int sec_h, int sec_w) {
  const int t = blockIdx.x;
  const int* pr = pos + (size_t)t * pos_stride;
  const int half_hd = hd >> 1;
  for (int idx = threadIdx.x; idx < H * half_hd; idx += blockDim.x) {
    const int h = idx / half_hd, i = idx - h * half_hd;
    const bf16* p = x + (size_t)t * in_stride + (size_t)h * hd;
    bf16* o = out + (size_t)t * out_stride + (size_t)h * hd;
    if (i < half_rot) {
      int axis = 0;
      if (pos_stride == 3) {
        // interleaved MRoPE: slot i takes axis (i % 3) while it lies inside that axis' section span
        const int a = i % 3;
        if (a == 1 && i < 3 * sec_h) axis = 1;
        if (a == 2 && i < 3 * sec_w) axis = 2;
      }
      const float ang = (float)pr[axis] * inv_freq[i];
      float s, c;
      sincosf(ang, &s, &c);
      if (inverse) s = -s;
      const float a = __bfloat162float(p[i]), b = __bfloat162float(p[i + half_rot]);
      o[i] = __float2bfloat16(a * c - b * s);
      o[i + half_rot] = __float2bfloat16(b * c + a * s);
    } else if (o != p) {
      // pass-through tail (partial rotary): channels [2*half_rot, hd)
      const int c0 = 2 * half_rot + 2 * (i - half_rot);
      o[c0] = p[c0];
      o[c0 + 1] = p[c0 + 1];
    }
  }
}

// Full-rotary fast path (one position axis, rot == hd, hd % 16 == 0, 16-byte aligned rows): one block per token.
// The hd/2 (sin, cos) pairs of the token are computed once into shared memory and reused by every head; each thread
// then rotates 8 pairs of one head with two 16-byte loads and two 16-byte stores.
__global__ void rope_full_vec_kernel(const bf16* __restrict__ x, long in_stride, bf16* __restrict__ out, long out_stride,
                                     const int* __restrict__ pos, const float* __restrict__ inv_freq, int T, int H,
                                     int hd, int inverse) {
  extern __shared__ float sc[];              // [half] sin, [half] cos
  const int t = blockIdx.x;
  const int half = hd >> 1;
  const float pf = (float)pos[t];
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    float sn, cs;
    sincosf(pf * inv_freq[i], &sn, &cs);
    sc[i] = inverse ? -sn : sn;
    sc[half + i] = cs;
  }
  __syncthreads();
  const int per_head = half >> 3;            // 8-pair chunks per head
  const bf16* xr = x + (size_t)t * in_stride;
  bf16* orow = out + (size_t)t * out_stride;
  for (int idx = threadIdx.x; idx < H * per_head; idx += blockDim.x) {
    const int h = idx / per_head, c = (idx - h * per_head) << 3;
    const uint4 ua = *reinterpret_cast<const uint4*>(xr + (size_t)h * hd + c);
    const uint4 ub = *reinterpret_cast<const uint4*>(xr + (size_t)h * hd + half + c);
    float a[8], b[8], ra[8], rb[8];
    unpack8(ua, a);
    unpack8(ub, b);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float sn = sc[c + e], cs = sc[half + c + e];
      ra[e] = a[e] * cs - b[e] * sn;
      rb[e] = b[e] * cs + a[e] * sn;
    }
    *reinterpret_cast<uint4*>(orow + (size_t)h * hd + c) = pack8(ra);
    *reinterpret_cast<uint4*>(orow + (size_t)h * hd + half + c) = pack8(rb);
  }
}

// Q, K and V of a projection in one pass: Q and K rotated (full rotary, one position axis), V copied, each (T, H, hd) with a token
// stride of its own.  Forward from the projection into the saved activations, and inverse from the attention's gradients (dQ
// still in fp32 as the kernel accumulated it) into the projection's gradient.  A block takes 512 / hd tokens, so that every
// thread works out one (sin, cos); a block per token left most threads of a narrow model idle, and V went by a library copy of
// two bytes an access.
// us, rotation of each, copy of V and rounding of dQ / so: 16384 x (32 + 2 x 8) x 128 97.5 / 65.5 forward, 156 / 82.3 backward; (6 + 2 x
// 6) x 128 54.1 / 31.1 and 67.4 / 32.5; (32 + 2 x 8) x 64 55.4 / 42.0 and 86.1 / 44.1.
template <typename TQ>
__global__ void __launch_bounds__(256) rope_qkv_kernel(const TQ* __restrict__ q, long q_is, bf16* __restrict__ qo, long q_os, int HQ,
                                                       const bf16* __restrict__ k, long k_is, bf16* __restrict__ ko, long k_os,
                                                       const bf16* __restrict__ v, long v_is, bf16* __restrict__ vo, long v_os, int HK,
                                                       int HV, const int* __restrict__ pos, const float* __restrict__ inv_freq, int T,
                                                       int hd, int inverse) {
  __shared__ float sn[256], cs[256];             // [token][pair]
  const int half = hd >> 1, t0 = blockIdx.x * (256 / half);
  {
    const int t = t0 + threadIdx.x / half;
    if (t < T) {
      float s, c;
      sincosf((float)pos[t] * inv_freq[threadIdx.x % half], &s, &c);
      sn[threadIdx.x] = inverse ? -s : s;
      cs[threadIdx.x] = c;
    }
  }
  __syncthreads();
  const int per_head = half >> 3, heads = HQ + HK + HV, units = heads * per_head, n = min(256 / half, T - t0);
  auto load_bf = [](const bf16* p, float (&f)[8]) { unpack8(*reinterpret_cast<const uint4*>(p), f); };
  for (int idx = threadIdx.x; idx < n * units; idx += 256) {
    const int tt = idx / units, u = idx - tt * units, h = u / per_head, c = (u - h * per_head) << 3;
    const long t = t0 + tt;
    if (h >= HQ + HK) {
      const long at = (long)(h - HQ - HK) * hd + c;
      const uint4 a = *reinterpret_cast<const uint4*>(v + t * v_is + at), b = *reinterpret_cast<const uint4*>(v + t * v_is + at + half);
      *reinterpret_cast<uint4*>(vo + t * v_os + at) = a;
      *reinterpret_cast<uint4*>(vo + t * v_os + at + half) = b;
      continue;
    }
    float a[8], b[8], ra[8], rb[8];
    bf16* o;
    if (h >= HQ) {
      const bf16* p = k + t * k_is + (long)(h - HQ) * hd + c;
      o = ko + t * k_os + (long)(h - HQ) * hd + c;
      load_bf(p, a);
      load_bf(p + half, b);
    } else {
      const TQ* p = q + t * q_is + (long)h * hd + c;
      o = qo + t * q_os + (long)h * hd + c;
      if constexpr (sizeof(TQ) == 4) {
#pragma unroll
        for (int e = 0; e < 8; e += 4) {
          const float4 x = *reinterpret_cast<const float4*>(p + e), y = *reinterpret_cast<const float4*>(p + half + e);
          a[e] = x.x; a[e + 1] = x.y; a[e + 2] = x.z; a[e + 3] = x.w;
          b[e] = y.x; b[e + 1] = y.y; b[e + 2] = y.z; b[e + 3] = y.w;
        }
      } else {
        load_bf(p, a);
        load_bf(p + half, b);
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float s1 = sn[tt * half + c + e], c1 = cs[tt * half + c + e];
      ra[e] = a[e] * c1 - b[e] * s1;
      rb[e] = b[e] * c1 + a[e] * s1;
    }
    *reinterpret_cast<uint4*>(o) = pack8(ra);
    *reinterpret_cast<uint4*>(o + half) = pack8(rb);
  }
}

// ------------------------------------------------------------------------ SwiGLU / GeGLU
__device__ __forceinline__ void act_and_grad(float g, int kind, float& a, float& da) {
  if (kind == 0) {
    const float s = 1.f / (1.f + __expf(-g));
    a = g * s;
    da = s * (1.f + g * (1.f - s));
  } else {
    const float k0 = 0.7978845608028654f, k1 = 0.044715f;
    const float t = tanhf(k0 * (g + k1 * g * g * g));
    a = 0.5f * g * (1.f + t);
    da = 0.5f * (1.f + t) + 0.5f * g * (1.f - t * t) * k0 * (1.f + 3.f * k1 * g * g);
  }
}

// Output gate of gated attention.  Bound by memory: one pass each way, 16 bytes a thread.  The heads of a projection lie
// [query | gate], so the gate is read (copy) and its gradient written (bwd) a head at a time, `ld` and `hs` elements apart.
// 16384 tokens, 16 heads of 256, us: copy 162 -> 53, out = x * sigmoid(gate) 620 -> 83, all of the backward 1810 -> 140 (chains of fp32
// element-wise passes before).
// The sigmoid is rounded as a chain of fp32 operations rounds it: e^-x by Cody and Waite's reduction, -x = n ln 2 + r with ln 2 in two
// parts, and the series of e^r, |r| < 0.35 (the term of r^8 is below 6e-9), then a reciprocal rounded to nearest; the
// hardware's exponential alone is off by |x| 2^-24 and more (9e-5 of the bf16 results for gates up to 80 were not the nearest, 5e-6 so,
// 2e-5 from the tensor library) and took 59 us where this takes 83, backward 123 and 140.  Past 88 the sigmoid is 0 or 1 in any case.
__device__ __forceinline__ float sigmoid_of(float x) {
  float y = -x;
  asm("min.NaN.f32 %0, %0, %1;" : "+f"(y) : "f"(88.f));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(y) : "f"(-87.f));
  const float shifted = fmaf(y, 1.44269504f, 12582912.f), n = shifted - 12582912.f;      // 1.5 * 2^23: n in the lowest bits
  float r = fmaf(n, -0.693359375f, y);             // 355 / 512
  r = fmaf(n, 2.12194440e-4f, r);                  // and what it is more than ln 2
  float p = 1.98412698e-4f;                        // 1 / k!, k = 7 .. 0
  p = fmaf(p, r, 1.38888889e-3f);
  p = fmaf(p, r, 8.33333333e-3f);
  p = fmaf(p, r, 4.16666667e-2f);
  p = fmaf(p, r, 1.66666667e-1f);
  p = fmaf(p, r, 0.5f);
  p = fmaf(p, r, 1.f);
  p = fmaf(p, r, 1.f);
  return __frcp_rn(fmaf(p, __uint_as_float((__float_as_uint(shifted) << 23) + 0x3f800000u), 1.f));
}

__global__ void __launch_bounds__(256) copy_heads_kernel(const bf16* __restrict__ x, long ld, long hs, bf16* __restrict__ y, long nvec,
                                                         int H, int hv) {
  const long v = (long)blockIdx.x * 256 + threadIdx.x;
  if (v >= nvec) return;
  const long row = v / hv, t = row / H;
  const int i = (int)(v - row * hv), h = (int)(row - t * H);
  reinterpret_cast<uint4*>(y)[v] = *reinterpret_cast<const uint4*>(x + t * ld + h * hs + i * 8);
}
__global__ void __launch_bounds__(256) attn_gate_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ gate,
                                                            bf16* __restrict__ y, long nvec) {
  const long v = (long)blockIdx.x * 256 + threadIdx.x;
  if (v >= nvec) return;
  float f[8], g[8];
  unpack8(reinterpret_cast<const uint4*>(x)[v], f);
  unpack8(reinterpret_cast<const uint4*>(gate)[v], g);
#pragma unroll
  for (int e = 0; e < 8; ++e) f[e] *= sigmoid_of(g[e]);
  reinterpret_cast<uint4*>(y)[v] = pack8(f);
}
// d (the gradient of y) becomes the gradient of x in place; y is written again, for the output projection's weight gradient.
__global__ void __launch_bounds__(256) attn_gate_bwd_kernel(bf16* __restrict__ d, const bf16* __restrict__ x,
                                                            const bf16* __restrict__ gate, bf16* __restrict__ y,
                                                            bf16* __restrict__ dgate, long ld, long hs, long nvec, int H, int hv) {
  const long v = (long)blockIdx.x * 256 + threadIdx.x;
  if (v >= nvec) return;
  float dv[8], f[8], g[8], a[8];
  unpack8(reinterpret_cast<const uint4*>(d)[v], dv);
  unpack8(reinterpret_cast<const uint4*>(x)[v], f);
  unpack8(reinterpret_cast<const uint4*>(gate)[v], g);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float s = sigmoid_of(g[e]);
    a[e] = f[e] * s;
    g[e] = dv[e] * f[e] * s * (1.f - s);
    dv[e] *= s;
  }
  const long row = v / hv, t = row / H;
  const int i = (int)(v - row * hv), h = (int)(row - t * H);
  reinterpret_cast<uint4*>(d)[v] = pack8(dv);
  reinterpret_cast<uint4*>(y)[v] = pack8(a);
  *reinterpret_cast<uint4*>(dgate + t * ld + h * hs + i * 8) = pack8(g);
}

// gate / up may be column slices of one (T, ld) buffer (a fused [gate | up] projection output).
__global__ void glu_fwd_kernel(const bf16* __restrict__ gate, const bf16* __restrict__ up, bf16* __restrict__ out,
                               long T, int F, int ld_in, int ld_out, int kind) {
  const long nvec = T * (F >> 3);
  for (long v = (long)blockIdx.x * blockDim.x + threadIdx.x; v < nvec; v += (long)gridDim.x * blockDim.x) {
    const long t = v / (F >> 3);
    const int c = (int)(v - t * (F >> 3)) << 3;
    float g[8], u[8], o[8];
    unpack8(*reinterpret_cast<const uint4*>(gate + t * ld_in + c), g);
    unpack8(*reinterpret_cast<const uint4*>(up + t * ld_in + c), u);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float a, da;
      act_and_grad(g[e], kind, a, da);
      o[e] = a * u[e];
    }
    *reinterpret_cast<uint4*>(out + t * ld_out + c) = pack8(o);
  }
}

__global__ void glu_bwd_kernel(const bf16* __restrict__ dact, const bf16* __restrict__ gate,
                               const bf16* __restrict__ up, bf16* __restrict__ dgate, bf16* __restrict__ dup,
                               bf16* __restrict__ act_out, long T, int F, int ld_in, int ld_d, int ld_act, int kind) {
  const long nvec = T * (F >> 3);
  for (long v = (long)blockIdx.x * blockDim.x + threadIdx.x; v < nvec; v += (long)gridDim.x * blockDim.x) {
    const long t = v / (F >> 3);
    const int c = (int)(v - t * (F >> 3)) << 3;
    float g[8], u[8], d[8], og[8], ou[8], oa[8];
    unpack8(*reinterpret_cast<const uint4*>(gate + t * ld_in + c), g);
    unpack8(*reinterpret_cast<const uint4*>(up + t * ld_in + c), u);
    unpack8(*reinterpret_cast<const uint4*>(dact + t * ld_act + c), d);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float a, da;
      act_and_grad(g[e], kind, a, da);
      og[e] = d[e] * u[e] * da;
      ou[e] = d[e] * a;
      oa[e] = a * u[e];
    }
    *reinterpret_cast<uint4*>(dgate + t * ld_d + c) = pack8(og);
    *reinterpret_cast<uint4*>(dup + t * ld_d + c) = pack8(ou);
    if (act_out) *reinterpret_cast<uint4*>(act_out + t * ld_act + c) = pack8(oa);
  }
}

// MoE expert backward through the gated activation with the router weight folded in, one CTA per expert-major row
// (the reference's swiglu_bwd_weighted kernel, flextrain/ops/_kernels/moe.py:77-145):
//   act = glu(gate, up);  d = w_row * dact_u;  dgate, dup from d;  act_w = w_row * act (left operand of the down-proj
//   weight gradient, so dy needs no separate scaling pass);  dw_row = sum_c dact_u * act (router-weight gradient).
__global__ void glu_bwd_weighted_kernel(const bf16* __restrict__ dact, const bf16* __restrict__ gate,
                                        const bf16* __restrict__ up, const float* __restrict__ w_row,
                                        bf16* __restrict__ dgate, bf16* __restrict__ dup, bf16* __restrict__ act_w,
                                        float* __restrict__ dw_row, int F, int ld_in, int ld_d, int kind) {
  __shared__ float red[32];
  const long t = blockIdx.x;
  const float wr = w_row[t];
  float dot = 0.f;
  for (int c = threadIdx.x << 3; c < F; c += blockDim.x << 3) {
    float g[8], u[8], d[8], og[8], ou[8], oa[8];
    unpack8(*reinterpret_cast<const uint4*>(gate + t * ld_in + c), g);
    unpack8(*reinterpret_cast<const uint4*>(up + t * ld_in + c), u);
    unpack8(*reinterpret_cast<const uint4*>(dact + t * (long)F + c), d);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float a, da;
      act_and_grad(g[e], kind, a, da);
      const float act = a * u[e];
      dot += d[e] * act;
      const float dd = d[e] * wr;
      og[e] = dd * u[e] * da;
      ou[e] = dd * a;
      oa[e] = act * wr;
    }
    *reinterpret_cast<uint4*>(dgate + t * ld_d + c) = pack8(og);
    *reinterpret_cast<uint4*>(dup + t * ld_d + c) = pack8(ou);
    *reinterpret_cast<uint4*>(act_w + t * (long)F + c) = pack8(oa);
  }
  dot = warp_sum(dot);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = dot;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    v = warp_sum(v);
    if (threadIdx.x == 0) dw_row[t] = v;
  }
}

// ----------------------------------------------------------------- softmax cross-entropy
// One CTA per row. Pass 1: online max / sum over V (bf16 logits). Pass 2: logits <- grad_scale *
// (softmax - onehot) in place (the second read hits L2). Optional tanh soft-cap chained through.
// A row is read twice (its second reading is for the gradient, which takes its place), CE_BATCH 16-byte pieces a thread at a
// time: with one piece in flight the kernel waited for memory.  GRAD = false: held-out loss, the logits are only read, once.
// Nothing is used up (two exponentials an element take half of the time, memory two thirds), so what counts is how much is in
// flight and that the second reading still finds the row in L2.  Rows of 112 KB and more: two blocks of 512 threads an SM, eight
// pieces a thread; 2048 x 128256 225 -> 210 us (before: four pieces, a test for the target at each element), 4096 x 151936 551 -> 523,
// 4096 x 262144 977 -> 948, with a soft-cap 1207 -> 1106; 2048 x 65544 117 -> 107.  Shorter rows, two blocks an SM of them and more: four
// blocks of 256, whose sums over the block weigh less; 8192 x 32000 232 -> 178 (216 as the long rows), 2048 x 50304 98 -> 84 (86);
// 65536: 113 (107); 128256: 240.  Few short rows as the long ones (16 x 50304 19.1 us, 19.8 with 256 threads).
constexpr int CE_BATCH = 8, CE_LONG = 57344, CE_ROWS = 2 * 148;
template <bool CAP>
__device__ __forceinline__ float ce_cap(float f, float softcap, float inv_cap, float& d) {
  if (!CAP) return f;
  const float t = tanhf(f * inv_cap);
  d = 1.f - t * t;
  return softcap * t;
}
template <bool GRAD, bool CAP, int CE_THREADS>
__global__ void __launch_bounds__(CE_THREADS, 1024 / CE_THREADS)
    softmax_ce_kernel(bf16* __restrict__ logits, const long* __restrict__ targets, const float* __restrict__ loss_mask,
                      float* __restrict__ loss, int T, int V, long ld, float grad_scale, float softcap, long ignore_index) {
  __shared__ float sh[32];
  const int row = blockIdx.x;
  bf16* z = logits + (size_t)row * ld;
  const long tgt = targets[row];
  bool valid = tgt != ignore_index && tgt >= 0 && tgt < V;
  if (loss_mask && loss_mask[row] <= 0.f) valid = false;
  const int nv = V >> 3;
  const float inv_cap = CAP ? 1.f / softcap : 0.f;
  if (!valid) {
    if constexpr (GRAD) {
      const uint4 zero = make_uint4(0, 0, 0, 0);
      for (int i = threadIdx.x; i < nv; i += CE_THREADS) reinterpret_cast<uint4*>(z)[i] = zero;
      for (int i = (nv << 3) + threadIdx.x; i < V; i += CE_THREADS) z[i] = __float2bfloat16(0.f);
    }
    if (threadIdx.x == 0) loss[row] = 0.f;
    return;
  }
  float m = -INFINITY, s = 0.f, unused;
  for (int i0 = threadIdx.x; i0 < nv; i0 += CE_BATCH * CE_THREADS) {
    uint4 v[CE_BATCH];
#pragma unroll
    for (int k = 0; k < CE_BATCH; ++k)
      if (i0 + k * CE_THREADS < nv) v[k] = reinterpret_cast<const uint4*>(z)[i0 + k * CE_THREADS];
#pragma unroll
    for (int k = 0; k < CE_BATCH; ++k) {
      if (i0 + k * CE_THREADS >= nv) break;
      float f[8];
      unpack8(v[k], f);
      float lm = -INFINITY;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        f[e] = ce_cap<CAP>(f[e], softcap, inv_cap, unused);
        lm = fmaxf(lm, f[e]);
      }
      const float nm = fmaxf(m, lm);
      float acc = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) acc += __expf(f[e] - nm);
      s = s * __expf(m - nm) + acc;
      m = nm;
    }
  }
  for (int i = (nv << 3) + threadIdx.x; i < V; i += CE_THREADS) {
    const float f = ce_cap<CAP>(__bfloat162float(z[i]), softcap, inv_cap, unused);
    const float nm = fmaxf(m, f);
    s = s * __expf(m - nm) + __expf(f - nm);
    m = nm;
  }
  const float gm = block_max<CE_THREADS / 32>(m, sh);
  s = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
  const float gs = block_sum<CE_THREADS / 32>(s, sh);
  const float lse = gm + logf(gs);
  float target = 0.f;                            // the target's gradient, written once all others are (thread 0)
  if (threadIdx.x == 0) {
    float d = 1.f;
    const float zt = ce_cap<CAP>(__bfloat162float(z[tgt]), softcap, inv_cap, d);
    loss[row] = lse - zt;
    target = (__expf(zt - lse) - 1.f) * grad_scale * d;
  }
  if constexpr (!GRAD) return;
  __syncthreads();  // the target logit is read before anyone overwrites it
  for (int i0 = threadIdx.x; i0 < nv; i0 += CE_BATCH * CE_THREADS) {
    uint4 v[CE_BATCH];
#pragma unroll
    for (int k = 0; k < CE_BATCH; ++k)
      if (i0 + k * CE_THREADS < nv) v[k] = reinterpret_cast<const uint4*>(z)[i0 + k * CE_THREADS];
#pragma unroll
    for (int k = 0; k < CE_BATCH; ++k) {
      const int i = i0 + k * CE_THREADS;
      if (i >= nv) break;
      float f[8];
      unpack8(v[k], f);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        float d = 1.f;
        const float zc = ce_cap<CAP>(f[e], softcap, inv_cap, d);
        f[e] = __expf(zc - lse) * grad_scale * d;
      }
      reinterpret_cast<uint4*>(z)[i] = pack8(f);
    }
  }
  for (int i = (nv << 3) + threadIdx.x; i < V; i += CE_THREADS) {
    float d = 1.f;
    const float f = ce_cap<CAP>(__bfloat162float(z[i]), softcap, inv_cap, d);
    z[i] = __float2bfloat16(__expf(f - lse) * grad_scale * d);
  }
  __syncthreads();
  if (threadIdx.x == 0) z[tgt] = __float2bfloat16(target);
}

template <bool GRAD>
void run_softmax_ce(bf16* logits, const long* targets, const float* loss_mask, float* loss, int T, int V, long ld, float grad_scale,
                    float softcap, long ignore_index, cudaStream_t s) {
  const bool cap = softcap > 0.f;
  auto wide = cap ? softmax_ce_kernel<GRAD, true, 512> : softmax_ce_kernel<GRAD, false, 512>;
  auto narrow = cap ? softmax_ce_kernel<GRAD, true, 256> : softmax_ce_kernel<GRAD, false, 256>;
  const bool is_long = V > CE_LONG || T < CE_ROWS;
  (is_long ? wide : narrow)<<<T, is_long ? 512 : 256, 0, s>>>(logits, targets, loss_mask, loss, T, V, ld, grad_scale, softcap,
                                                              ignore_index);
}

// ----------------------------------------------------------------------------- embedding
__global__ void embedding_fwd_kernel(const long* __restrict__ tokens, const bf16* __restrict__ table,
                                     bf16* __restrict__ out, int T, int D, float scale) {
  const int t = blockIdx.x;
  const long tok = tokens[t];
  const uint4* src = reinterpret_cast<const uint4*>(table + (size_t)tok * D);
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)t * D);
  for (int i = threadIdx.x; i < (D >> 3); i += blockDim.x) {
    uint4 v = src[i];
    if (scale != 1.f) {
      float f[8];
      unpack8(v, f);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] *= scale;
      v = pack8(f);
    }
    dst[i] = v;
  }
}

// Sorted scatter-add: sorted_tok ascending, order[i] = original row of sorted position i.
// The CTA at the head of each run sums the run in fp32 and adds it to the gradient row once.
__global__ void embedding_bwd_kernel(const long* __restrict__ sorted_tok, const long* __restrict__ order,
                                     const bf16* __restrict__ dy, void* __restrict__ grad, int T, int D, float scale,
                                     int grad_fp32) {
  const int i0 = blockIdx.x;
  const long tok = sorted_tok[i0];
  if (i0 > 0 && sorted_tok[i0 - 1] == tok) return;
  int i1 = i0 + 1;
  while (i1 < T && sorted_tok[i1] == tok) ++i1;
  for (int c = threadIdx.x; c < (D >> 3); c += blockDim.x) {
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int i = i0; i < i1; ++i) {
      float f[8];
      unpack8(reinterpret_cast<const uint4*>(dy + (size_t)order[i] * D)[c], f);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += f[e];
    }
    if (grad_fp32) {
      float* g = reinterpret_cast<float*>(grad) + (size_t)tok * D + c * 8;
#pragma unroll
      for (int e = 0; e < 8; ++e) g[e] += acc[e] * scale;
    } else {
      uint4* g = reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(grad) + (size_t)tok * D) + c;
      float f[8];
      unpack8(*g, f);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] += acc[e] * scale;
      *g = pack8(f);
    }
  }
}

// --------------------------------------------------------------------------- AdamW
// Multi-tensor: one launch updates up to ADAM_MAX tensors (a whole layer). dtype codes: 0 bf16, 1 fp32.
// Bound by memory: 22 bytes an element with bf16 weights and gradients and fp32 state (14 with bf16 state), each read
// and written once.  A thread takes 8 neighbouring elements, all of whose 16-byte loads are issued before the first
// use; the types are template arguments, chosen once per block (a block lies in one tensor).
// 218 M bf16 weights and gradients: fp32 state 931 us (5.2 TB/s) with one element a load, 691 us (6.9 TB/s) so; bf16
// state 741 us (4.1 TB/s) before, 441 us (6.9 TB/s) now.
constexpr int ADAM_MAX = 24;
struct AdamTensor {
  void* p; const void* g; void* m; void* v;
  long n;
  long block_start;  // first block of this tensor in the flattened grid
  float lr, wd;
  int p_dt, g_dt, s_dt;
  int vec;           // all four pointers on 16 bytes: whole groups of 8 elements go as vectors
};
struct AdamArgs {
  AdamTensor t[ADAM_MAX];
  int count;
  float beta1, beta2, eps, bc1, bc2, grad_scale;
};
constexpr int ADAM_THREADS = 256;
constexpr int ADAM_PER_BLOCK = ADAM_THREADS * 8;

__device__ __forceinline__ float ld_any(const void* p, long i, int dt) {
  return dt ? reinterpret_cast<const float*>(p)[i] : __bfloat162float(reinterpret_cast<const bf16*>(p)[i]);
}
__device__ __forceinline__ void st_any(void* p, long i, int dt, float v) {
  if (dt) reinterpret_cast<float*>(p)[i] = v;
  else reinterpret_cast<bf16*>(p)[i] = __float2bfloat16(v);
}

// Eight elements as they lie in memory: one 16-byte word of bf16, two of fp32.
template <bool F32> struct Raw8 { uint4 w[F32 ? 2 : 1]; };
template <bool F32>
__device__ __forceinline__ Raw8<F32> ld_raw8(const void* p, long i) {
  Raw8<F32> r;
  const uint4* q = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(p) + i * (F32 ? 4 : 2));
#pragma unroll
  for (int k = 0; k < (F32 ? 2 : 1); ++k) r.w[k] = __ldcs(q + k);
  return r;
}
template <bool F32>
__device__ __forceinline__ void unpack_raw8(const Raw8<F32>& r, float (&f)[8]) {
  if constexpr (F32) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      f[4 * k] = __uint_as_float(r.w[k].x); f[4 * k + 1] = __uint_as_float(r.w[k].y);
      f[4 * k + 2] = __uint_as_float(r.w[k].z); f[4 * k + 3] = __uint_as_float(r.w[k].w);
    }
  } else {
    unpack8(r.w[0], f);
  }
}
template <bool F32>
__device__ __forceinline__ void st_raw8(void* p, long i, const float (&f)[8]) {
  uint4* q = reinterpret_cast<uint4*>(reinterpret_cast<char*>(p) + i * (F32 ? 4 : 2));
  if constexpr (F32) {
#pragma unroll
    for (int k = 0; k < 2; ++k)
      __stcs(q + k, make_uint4(__float_as_uint(f[4 * k]), __float_as_uint(f[4 * k + 1]),
                               __float_as_uint(f[4 * k + 2]), __float_as_uint(f[4 * k + 3])));
  } else {
    __stcs(q, pack8(f));
  }
}

__device__ __forceinline__ void adamw_one(const AdamArgs& a, float lr, float wd, float g, float& p, float& m, float& v) {
  g *= a.grad_scale;
  p -= lr * wd * p;
  m = a.beta1 * m + (1.f - a.beta1) * g;
  v = a.beta2 * v + (1.f - a.beta2) * g * g;
  p -= lr * (m / a.bc1) / (sqrtf(v / a.bc2) + a.eps);
}

template <bool PF, bool GF, bool SF>
__device__ __forceinline__ void adamw_vec8(const AdamArgs& a, const AdamTensor& t, long i) {
  const Raw8<PF> rp = ld_raw8<PF>(t.p, i);
  const Raw8<GF> rg = ld_raw8<GF>(t.g, i);
  const Raw8<SF> rm = ld_raw8<SF>(t.m, i), rv = ld_raw8<SF>(t.v, i);
  float p[8], g[8], m[8], v[8];
  unpack_raw8<PF>(rp, p); unpack_raw8<GF>(rg, g); unpack_raw8<SF>(rm, m); unpack_raw8<SF>(rv, v);
#pragma unroll
  for (int j = 0; j < 8; ++j) adamw_one(a, t.lr, t.wd, g[j], p[j], m[j], v[j]);
  st_raw8<PF>(t.p, i, p); st_raw8<SF>(t.m, i, m); st_raw8<SF>(t.v, i, v);
}

__global__ void __launch_bounds__(ADAM_THREADS) adamw_kernel(const __grid_constant__ AdamArgs a) {
  int ti = 0;
#pragma unroll 1
  for (int i = 1; i < a.count; ++i)
    if ((long)blockIdx.x >= a.t[i].block_start) ti = i;
  const AdamTensor& t = a.t[ti];
  const long base = ((long)blockIdx.x - t.block_start) * ADAM_PER_BLOCK;
  const long i0 = base + (long)threadIdx.x * 8;
  if (t.vec && i0 + 8 <= t.n) {
    switch (t.p_dt * 4 + t.g_dt * 2 + t.s_dt) {
      case 0: adamw_vec8<false, false, false>(a, t, i0); break;
      case 1: adamw_vec8<false, false, true>(a, t, i0); break;
      case 2: adamw_vec8<false, true, false>(a, t, i0); break;
      case 3: adamw_vec8<false, true, true>(a, t, i0); break;
      case 4: adamw_vec8<true, false, false>(a, t, i0); break;
      case 5: adamw_vec8<true, false, true>(a, t, i0); break;
      case 6: adamw_vec8<true, true, false>(a, t, i0); break;
      default: adamw_vec8<true, true, true>(a, t, i0); break;
    }
    return;
  }
#pragma unroll 1
  for (long i = i0; i < i0 + 8 && i < t.n; ++i) {       // the last, incomplete group; tensors off the 16-byte grid
    float p = ld_any(t.p, i, t.p_dt), m = ld_any(t.m, i, t.s_dt), v = ld_any(t.v, i, t.s_dt);
    adamw_one(a, t.lr, t.wd, ld_any(t.g, i, t.g_dt), p, m, v);
    st_any(t.p, i, t.p_dt, p);
    st_any(t.m, i, t.s_dt, m);
    st_any(t.v, i, t.s_dt, v);
  }
}

// ------------------------------------------------------------------------------- Muon
// The elementwise parts of the Muon update for a batch of matrices of one size.  With gf = g * grad_scale and
// mf = beta * mom + gf, the update is u = gf + beta * mf (Nesterov) or mf, normalised by its Frobenius norm:
//   muon_norm      partial sums of u^2 per matrix (a block adds 16384 elements)
//   muon_prepare   mom = mf;  x = u / (||u|| + 1e-7) in bf16, the start of the Newton-Schulz iteration
//   muon_apply     p = p * (1 - lr * wd) - lr * scale * x
// u is computed twice rather than kept: its fp32 copy would cost more to write and read than g and mom do.  Bound by
// memory.  One launch each for up to MUON_MAX matrices, in place of twelve library kernels per matrix.
constexpr int MUON_MAX = 64;
constexpr int MUON_THREADS = 256;
constexpr int MUON_PER_BLOCK = MUON_THREADS * 64;
struct MuonArgs {
  const void* g[MUON_MAX];
  void* m[MUON_MAX];
  void* p[MUON_MAX];
  long n;                // elements of a matrix, a multiple of 8
  long x_stride;         // elements from one matrix to the next in x
  int g_dt, m_dt, nesterov;
  float beta, grad_scale, keep, step;
};

template <bool GF, bool MF>
__device__ __forceinline__ void muon_update8(const MuonArgs& a, int mat, long i, float (&mf)[8], float (&u)[8]) {
  float g[8];
  unpack_raw8<GF>(ld_raw8<GF>(a.g[mat], i), g);
  unpack_raw8<MF>(ld_raw8<MF>(a.m[mat], i), mf);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float gf = g[j] * a.grad_scale;
    mf[j] = a.beta * mf[j] + gf;
    u[j] = a.nesterov ? gf + a.beta * mf[j] : mf[j];
  }
}

template <bool GF, bool MF>
__global__ void __launch_bounds__(MUON_THREADS) muon_norm_kernel(const __grid_constant__ MuonArgs a, float* __restrict__ partial) {
  __shared__ float sh[MUON_THREADS / 32];
  const int mat = blockIdx.y;
  float s = 0.f;
  for (int k = 0; k < 8; ++k) {
    const long i = (long)blockIdx.x * MUON_PER_BLOCK + ((long)k * MUON_THREADS + threadIdx.x) * 8;
    if (i >= a.n) break;
    float mf[8], u[8];
    muon_update8<GF, MF>(a, mat, i, mf, u);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += u[j] * u[j];
  }
  s = block_sum<MUON_THREADS / 32>(s, sh);
  if (threadIdx.x == 0) partial[(long)mat * gridDim.x + blockIdx.x] = s;
}

template <bool GF, bool MF>
__global__ void __launch_bounds__(MUON_THREADS) muon_prepare_kernel(const __grid_constant__ MuonArgs a,
                                                                    const float* __restrict__ partial, bf16* __restrict__ x) {
  __shared__ float sh[MUON_THREADS / 32];
  const int mat = blockIdx.y;
  float s = 0.f;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += MUON_THREADS) s += partial[(long)mat * gridDim.x + b];
  const float norm = sqrtf(block_sum<MUON_THREADS / 32>(s, sh)) + 1e-7f;
  for (int k = 0; k < 8; ++k) {
    const long i = (long)blockIdx.x * MUON_PER_BLOCK + ((long)k * MUON_THREADS + threadIdx.x) * 8;
    if (i >= a.n) break;
    float mf[8], u[8];
    muon_update8<GF, MF>(a, mat, i, mf, u);
    st_raw8<MF>(a.m[mat], i, mf);
#pragma unroll
    for (int j = 0; j < 8; ++j) u[j] = u[j] / norm;
    *reinterpret_cast<uint4*>(x + mat * a.x_stride + i) = pack8(u);
  }
}

__global__ void __launch_bounds__(MUON_THREADS) muon_apply_kernel(const __grid_constant__ MuonArgs a, const bf16* __restrict__ x) {
  const int mat = blockIdx.y;
  for (int k = 0; k < 8; ++k) {
    const long i = (long)blockIdx.x * MUON_PER_BLOCK + ((long)k * MUON_THREADS + threadIdx.x) * 8;
    if (i >= a.n) break;
    float p[8], v[8];
    uint4* pp = reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(a.p[mat]) + i);
    unpack8(*pp, p);
    unpack8(*reinterpret_cast<const uint4*>(x + mat * a.x_stride + i), v);
#pragma unroll
    for (int j = 0; j < 8; ++j) p[j] = p[j] * a.keep - a.step * v[j];
    *pp = pack8(p);
  }
}

// ------------------------------------------------------------------------ sum of squares
// Sum of the squares of up to SQ_MAX tensors (the gradient norm): one pass that reads every element once, in place of a
// conversion to fp32, a squaring and a reduction per tensor.  A block adds 16384 elements in fp32 (64 a thread, then a
// tree) and leaves one partial sum; the second kernel adds the partials of all launches in double, always in the same order.
// Bound by memory: 0.5 G bf16 elements in 50 tensors 2350 us with three passes a tensor, 205 us (5 TB/s) so.
constexpr int SQ_MAX = 64;
constexpr int SQ_THREADS = 256;
constexpr int SQ_PER_BLOCK = SQ_THREADS * 64;
struct SqTensor { const void* p; long n; long block_start; int dt, vec; };
struct SqArgs { SqTensor t[SQ_MAX]; int count; };

__global__ void __launch_bounds__(SQ_THREADS) sumsq_kernel(const __grid_constant__ SqArgs a, float* __restrict__ partial) {
  __shared__ float sh[SQ_THREADS / 32];
  int ti = 0;
#pragma unroll 1
  for (int i = 1; i < a.count; ++i)
    if ((long)blockIdx.x >= a.t[i].block_start) ti = i;
  const SqTensor& t = a.t[ti];
  const long base = ((long)blockIdx.x - t.block_start) * SQ_PER_BLOCK;
  float s = 0.f;
#pragma unroll 4
  for (int j = 0; j < 8; ++j) {
    const long i = base + ((long)j * SQ_THREADS + threadIdx.x) * 8;
    if (t.vec && i + 8 <= t.n) {
      float f[8];
      if (t.dt) unpack_raw8<true>(ld_raw8<true>(t.p, i), f);
      else unpack_raw8<false>(ld_raw8<false>(t.p, i), f);
#pragma unroll
      for (int e = 0; e < 8; ++e) s += f[e] * f[e];
    } else {
      for (long e = i; e < i + 8 && e < t.n; ++e) { const float f = ld_any(t.p, e, t.dt); s += f * f; }
    }
  }
  s = block_sum<SQ_THREADS / 32>(s, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

__global__ void __launch_bounds__(1024) sumsq_total_kernel(const float* __restrict__ partial, long n, float* __restrict__ out) {
  __shared__ double sh[32];
  double s = 0.0;
  for (long i = threadIdx.x; i < n; i += 1024) s += (double)partial[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = sh[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) out[0] = (float)s;
  }
}

// ------------------------------------------------------------------- gated RMSNorm / L2
__global__ void gated_rmsnorm_fwd_kernel(const bf16* __restrict__ o, const bf16* __restrict__ z,
                                         const float* __restrict__ w, bf16* __restrict__ y, long rows, int D,
                                         float eps) {
  const long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  float ss = 0.f;
  for (int i = lane; i < D; i += 32) {
    const float v = __bfloat162float(o[row * D + i]);
    ss += v * v;
  }
  ss = warp_sum(ss);
  const float r = rsqrtf(ss / (float)D + eps);
  for (int i = lane; i < D; i += 32) {
    const float v = __bfloat162float(o[row * D + i]) * r * w[i];
    const float g = __bfloat162float(z[row * D + i]);
    y[row * D + i] = __float2bfloat16(v * g / (1.f + __expf(-g)));
  }
}

__global__ void l2norm_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, float* __restrict__ rnorm,
                                  long rows, int D, float eps) {
  const long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  float ss = 0.f;
  for (int i = lane; i < D; i += 32) {
    const float v = __bfloat162float(x[row * D + i]);
    ss += v * v;
  }
  ss = warp_sum(ss);
  const float r = rsqrtf(ss + eps);
  if (lane == 0 && rnorm) rnorm[row] = r;
  for (int i = lane; i < D; i += 32) y[row * D + i] = __float2bfloat16(__bfloat162float(x[row * D + i]) * r);
}

// ------------------------------------------------------------------------- MoE routing
// Top-k by iterative arg-max (lowest index wins ties), softmax over the k picks (mode 0) or
// full softmax then top-k (mode 1). One warp per token; E <= 256.
__global__ void topk_route_kernel(const bf16* __restrict__ logits, float* __restrict__ weights,
                                  int* __restrict__ experts, int T, int E, int K, int mode) {
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= T) return;
  const int lane = threadIdx.x & 31;
  float v[8];
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int e = lane + j * 32;
    v[j] = e < E ? __bfloat162float(logits[(size_t)t * E + e]) : -INFINITY;
    mx = fmaxf(mx, v[j]);
  }
  if (mode == 1) {
    mx = warp_max(mx);
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = (lane + j * 32 < E) ? __expf(v[j] - mx) : -INFINITY;
      if (lane + j * 32 < E) s += v[j];
    }
    s = warp_sum(s);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (lane + j * 32 < E) v[j] /= s;
  }
  float pick_v[16];
  float top = 0.f;
  for (int k = 0; k < K; ++k) {
    float bv = -INFINITY;
    int bi = 1 << 30;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int e = lane + j * 32;
      if (v[j] > bv) { bv = v[j]; bi = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if (k == 0) top = bv;
    pick_v[k] = bv;
    if ((bi & 31) == lane) v[bi >> 5] = -INFINITY;
    if (lane == 0) experts[(size_t)t * K + k] = bi;
  }
  if (lane == 0) {
    if (mode == 0) {
      float s = 0.f;
      for (int k = 0; k < K; ++k) { pick_v[k] = __expf(pick_v[k] - top); s += pick_v[k]; }
      for (int k = 0; k < K; ++k) weights[(size_t)t * K + k] = pick_v[k] / s;
    } else {
      for (int k = 0; k < K; ++k) weights[(size_t)t * K + k] = pick_v[k];
    }
  }
}

// Row gather/scatter for MoE dispatch: out[i, :] = in[idx[i], :] * (w ? w[i] : 1).
__global__ void gather_rows_kernel(const bf16* __restrict__ in, const int* __restrict__ idx,
                                   const float* __restrict__ w, bf16* __restrict__ out, long rows, int D, int idx_div) {
  const long r = blockIdx.x;
  if (r >= rows) return;
  const int raw = idx[r];
  if (raw < 0) {  // padding row of an expert-major layout
    for (int c = threadIdx.x; c < (D >> 3); c += blockDim.x)
      reinterpret_cast<uint4*>(out + r * D)[c] = make_uint4(0, 0, 0, 0);
    return;
  }
  const long src = raw / idx_div;
  const float s = w ? w[r] : 1.f;
  for (int c = threadIdx.x; c < (D >> 3); c += blockDim.x) {
    uint4 v = reinterpret_cast<const uint4*>(in + src * D)[c];
    if (w) {
      float f[8];
      unpack8(v, f);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] *= s;
      v = pack8(f);
    }
    reinterpret_cast<uint4*>(out + r * D)[c] = v;
  }
}

// Combine: out[t, :] = resid[t, :] + sum_k w[t,k] * y[inv[t*K+k], :]  (fp32 accumulation).
__global__ void moe_combine_kernel(const bf16* __restrict__ y, const int* __restrict__ inv,
                                   const float* __restrict__ w, const bf16* __restrict__ resid,
                                   bf16* __restrict__ out, int T, int K, int D) {
  const int t = blockIdx.x;
  for (int c = threadIdx.x; c < (D >> 3); c += blockDim.x) {
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (resid) unpack8(reinterpret_cast<const uint4*>(resid + (size_t)t * D)[c], acc);
    for (int k = 0; k < K; ++k) {
      const long src = inv[(size_t)t * K + k];
      const float wk = w ? w[(size_t)t * K + k] : 1.f;
      float f[8];
      unpack8(reinterpret_cast<const uint4*>(y + src * D)[c], f);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += wk * f[e];
    }
    reinterpret_cast<uint4*>(out + (size_t)t * D)[c] = pack8(acc);
  }
}

}  // namespace

#define CHECK_LAUNCH()                                   \
  do {                                                   \
    cudaError_t e_ = cudaGetLastError();                 \
    return e_ == cudaSuccess ? 0 : -400 - (int)e_;       \
  } while (0)

static int grid_rows(long rows, int cap) { return (int)(rows < cap ? rows : cap); }

extern "C" {

// x: rows ldx elements apart (a multiple of 8); y contiguous.
int ftb_rmsnorm_fwd_ld(const void* x, long ldx, const float* w, void* y, float* rstd, int T, int D, float eps,
                       cudaStream_t s) {
  if (T == 0) return 0;
  if (D % 8 || ldx % 8 || D > 8 * RN_THREADS * RN_MAXV) return -2;
  const int nv = D / 8;
#define FTB_RN_FWD(MV) \
  rmsnorm_fwd_kernel<MV><<<grid_rows(T, 148 * 8), RN_THREADS, 0, s>>>((const bf16*)x, w, (bf16*)y, rstd, T, D, eps, ldx)
#define FTB_RN_WARP(NV)                                                                                                \
  case NV:                                                                                                             \
    rmsnorm_warp_fwd_kernel<NV><<<grid_rows((T + 7L) / 8, 148 * 8), RN_THREADS, 0, s>>>((const bf16*)x, w, (bf16*)y, rstd, T, \
                                                                                        D, eps, ldx);                  \
    break
  switch ((nv + 31) / 32) {
    FTB_RN_WARP(1);
    FTB_RN_WARP(2);
    FTB_RN_WARP(3);
    FTB_RN_WARP(4);
    FTB_RN_WARP(5);
    FTB_RN_WARP(6);
    FTB_RN_WARP(7);
    FTB_RN_WARP(8);
    default:
      if (nv <= 2 * RN_THREADS) FTB_RN_FWD(2);
      else if (nv <= 4 * RN_THREADS) FTB_RN_FWD(4);
      else FTB_RN_FWD(8);
  }
#undef FTB_RN_WARP
#undef FTB_RN_FWD
  CHECK_LAUNCH();
}
int ftb_rmsnorm_fwd(const void* x, const float* w, void* y, float* rstd, int T, int D, float eps,
                    cudaStream_t s) {
  return ftb_rmsnorm_fwd_ld(x, D, w, y, rstd, T, D, eps, s);
}

// dw_partial: fp32 workspace of (ftb_rmsnorm_bwd_blocks(T) * D); dw (fp32, D) accumulated if dw != null.
int ftb_rmsnorm_bwd_blocks(int T) { return grid_rows(T, 148 * 4); }
// x and dx: rows ldx / lddx elements apart (multiples of 8); dy, dx_add and y_out contiguous.
int ftb_rmsnorm_bwd_ld(const void* dy, const void* x, long ldx, const float* w, const float* rstd, const void* dx_add, void* dx,
                       long lddx, void* y_out, float* dw_partial, float* dw, int dw_accumulate, int T, int D,
                       cudaStream_t s) {
  if (T == 0) return 0;
  if (D % 8 || ldx % 8 || lddx % 8 || D > 8 * RN_THREADS * RN_MAXV) return -2;
  int blocks = ftb_rmsnorm_bwd_blocks(T);
  const int nv = D / 8;
#define FTB_RN_BWD(MV)                                                                                              \
  rmsnorm_bwd_kernel<MV><<<blocks, RN_THREADS, 0, s>>>((const bf16*)dy, (const bf16*)x, w, rstd, (const bf16*)dx_add, \
                                                       (bf16*)dx, (bf16*)y_out, dw ? dw_partial : nullptr, T, D, ldx, lddx)
#define FTB_RN_WARP(NV, WPR)                                                                                                          \
  do {                                                                                                                                \
    blocks = grid_rows((T + 8L / WPR - 1) / (8 / WPR), 148 * 2);                                                                      \
    rmsnorm_warp_bwd_kernel<NV, WPR><<<blocks, RN_THREADS, 0, s>>>((const bf16*)dy, (const bf16*)x, w, rstd, (const bf16*)dx_add,     \
                                                                   (bf16*)dx, (bf16*)y_out, dw ? dw_partial : nullptr, T, D, ldx, lddx); \
  } while (0)
  if (nv <= 32) FTB_RN_WARP(1, 1);
  else if (nv <= 64) FTB_RN_WARP(2, 1);
  else if (nv <= 96) FTB_RN_WARP(3, 1);
  else if (nv <= 128) FTB_RN_WARP(2, 2);
  else if (nv <= 192) FTB_RN_WARP(3, 2);
  else if (nv <= 256) FTB_RN_WARP(2, 4);
  else if (nv <= 384) FTB_RN_WARP(3, 4);
  else if (nv <= 2 * RN_THREADS) FTB_RN_BWD(2);
  else if (nv <= 4 * RN_THREADS) FTB_RN_BWD(4);
  else FTB_RN_BWD(8);
#undef FTB_RN_WARP
#undef FTB_RN_BWD
  if (dw) colsum_accum_kernel<<<(D + 31) / 32, 1024, 0, s>>>(dw_partial, dw, blocks, D, dw_accumulate);
  CHECK_LAUNCH();
}
int ftb_rmsnorm_bwd(const void* dy, const void* x, const float* w, const float* rstd, const void* dx_add, void* dx,
                    void* y_out, float* dw_partial, float* dw, int dw_accumulate, int T, int D, cudaStream_t s) {
  return ftb_rmsnorm_bwd_ld(dy, x, D, w, rstd, dx_add, dx, D, y_out, dw_partial, dw, dw_accumulate, T, D, s);
}

// Norm of every head of (T, H, hd) tensors, hd 64, 128 or 256: x (and dy, dx) with a token stride, heads side by side.
// Heads h* elements apart (512 for the queries of [query | gate] pairs of 256: 16384 tokens, 16 heads, forward 224 -> 60 us and backward
// 503 -> 94 without the copies to and from heads side by side).
int ftb_rmsnorm_heads_fwd(const void* x, long ldx, long hx, const float* w, void* y, float* rstd, int T, int H, int hd, float eps,
                          cudaStream_t s) {
  const long rows = (long)T * H;
  if (rows == 0) return 0;
  if (rows > 0x7fffffffL || ldx % 8 || hx % 8 || ((uintptr_t)x & 15) || (hd != 64 && hd != 128 && hd != 256)) return -2;
  const unsigned blocks = (unsigned)((rows * (hd / 8) + 255) / 256);
  if (hd == 64) rmsnorm_heads_fwd_kernel<64><<<blocks, 256, 0, s>>>((const bf16*)x, ldx, hx, w, (bf16*)y, rstd, (int)rows, H, eps);
  else if (hd == 128) rmsnorm_heads_fwd_kernel<128><<<blocks, 256, 0, s>>>((const bf16*)x, ldx, hx, w, (bf16*)y, rstd, (int)rows, H, eps);
  else rmsnorm_heads_fwd_kernel<256><<<blocks, 256, 0, s>>>((const bf16*)x, ldx, hx, w, (bf16*)y, rstd, (int)rows, H, eps);
  CHECK_LAUNCH();
}
int ftb_rmsnorm_heads_bwd(const void* dy, long lddy, long hdy, const void* x, long ldx, long hx, const float* w, const float* rstd,
                          void* dx, long lddx, long hdx, float* dw, int T, int H, int hd, cudaStream_t s) {
  const long rows = (long)T * H;
  if (rows == 0) return 0;
  if (rows > 0x7fffffffL || ldx % 8 || lddy % 8 || lddx % 8 || hx % 8 || hdy % 8 || hdx % 8 || (((uintptr_t)x | (uintptr_t)dy | (uintptr_t)dx) & 15) ||
      (hd != 64 && hd != 128 && hd != 256))
    return -2;
  long blocks = (rows * (hd / 8) + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
#define FTB_RNH(HD) \
  rmsnorm_heads_bwd_kernel<HD><<<(unsigned)blocks, 256, 0, s>>>((const bf16*)dy, lddy, hdy, (const bf16*)x, ldx, hx, w, rstd, \
                                                                (bf16*)dx, lddx, hdx, dw, (int)rows, H)
  if (hd == 64) FTB_RNH(64);
  else if (hd == 128) FTB_RNH(128);
  else FTB_RNH(256);
#undef FTB_RNH
  CHECK_LAUNCH();
}

// y (T, H, hd) contiguous <- x, tokens ld and heads hs elements apart.
int ftb_copy_heads(const void* x, long ld, long hs, void* y, long T, int H, int hd, cudaStream_t s) {
  const long nvec = T * H * (hd / 8);
  if (nvec == 0) return 0;
  if (hd % 8 || ld % 8 || hs % 8 || (((uintptr_t)x | (uintptr_t)y) & 15)) return -2;
  copy_heads_kernel<<<(unsigned)((nvec + 255) / 256), 256, 0, s>>>((const bf16*)x, ld, hs, (bf16*)y, nvec, H, hd / 8);
  CHECK_LAUNCH();
}
int ftb_attn_gate_fwd(const void* x, const void* gate, void* y, long n, cudaStream_t s) {
  if (n == 0) return 0;
  if (n % 8 || (((uintptr_t)x | (uintptr_t)gate | (uintptr_t)y) & 15)) return -2;
  attn_gate_fwd_kernel<<<(unsigned)((n / 8 + 255) / 256), 256, 0, s>>>((const bf16*)x, (const bf16*)gate, (bf16*)y, n / 8);
  CHECK_LAUNCH();
}
int ftb_attn_gate_bwd(void* d, const void* x, const void* gate, void* y, void* dgate, long ld, long hs, long T, int H, int hd,
                      cudaStream_t s) {
  const long nvec = T * H * (hd / 8);
  if (nvec == 0) return 0;
  if (hd % 8 || ld % 8 || hs % 8 ||
      (((uintptr_t)d | (uintptr_t)x | (uintptr_t)gate | (uintptr_t)y | (uintptr_t)dgate) & 15))
    return -2;
  attn_gate_bwd_kernel<<<(unsigned)((nvec + 255) / 256), 256, 0, s>>>((bf16*)d, (const bf16*)x, (const bf16*)gate, (bf16*)y,
                                                                      (bf16*)dgate, ld, hs, nvec, H, hd / 8);
  CHECK_LAUNCH();
}

int ftb_rmsnorm_small_fwd(const void* x, const float* w, void* y, float* rstd, long rows, int D, int heads_w,
                          float eps, cudaStream_t s) {
  if (rows == 0) return 0;
  if (D % 2) return -2;
  rmsnorm_small_fwd_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, s>>>((const bf16*)x, w, (bf16*)y, rstd, rows, D,
                                                                       heads_w, eps);
  CHECK_LAUNCH();
}
int ftb_rmsnorm_small_bwd(const void* dy, const void* x, const float* w, const float* rstd, void* dx, float* dw,
                          long rows, int D, cudaStream_t s) {
  if (rows == 0) return 0;
  if (D % 2 || D > 512) return -2;
  long blocks = (rows + 7) / 8;
  if (blocks > 148 * 8) blocks = 148 * 8;
  rmsnorm_small_bwd_kernel<<<(unsigned)blocks, 256, D * sizeof(float), s>>>((const bf16*)dy, (const bf16*)x, w, rstd,
                                                                            (bf16*)dx, dw, rows, D);
  CHECK_LAUNCH();
}

int ftb_rope(const void* x, long in_stride, void* out, long out_stride, const int* pos, const float* inv_freq,
             int T, int H, int hd, int half_rot, int inverse, int pos_stride, int sec_h, int sec_w, cudaStream_t s) {
  if (T == 0) return 0;
  if (hd % 2 || 2 * half_rot > hd) return -2;
  if (pos_stride == 1 && 2 * half_rot == hd && hd % 16 == 0 && in_stride % 8 == 0 && out_stride % 8 == 0 &&
      (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    int thr = H * (hd / 16);
    thr = thr > 256 ? 256 : ((thr + 31) / 32) * 32;
    rope_full_vec_kernel<<<T, thr, hd * sizeof(float), s>>>((const bf16*)x, in_stride, (bf16*)out, out_stride, pos,
                                                            inv_freq, T, H, hd, inverse);
    CHECK_LAUNCH();
  }
  int threads = H * (hd / 2);
  threads = threads > 512 ? 512 : ((threads + 31) / 32) * 32;
  rope_kernel<<<T, threads, 0, s>>>((const bf16*)x, in_stride, (bf16*)out, out_stride, pos, inv_freq, T, H, hd,
                                    half_rot, inverse, pos_stride, sec_h, sec_w);
  CHECK_LAUNCH();
}

// One launch for the heads of a projection (see the kernel).  HQ, HK, HV may be 0.  -2: not what the kernel takes.
int ftb_rope_qkv(const void* q, int q_fp32, long q_is, void* qo, long q_os, int HQ, const void* k, long k_is, void* ko, long k_os,
                 int HK, const void* v, long v_is, void* vo, long v_os, int HV, const int* pos, const float* inv_freq, int T, int hd,
                 int inverse, cudaStream_t s) {
  if (T <= 0 || HQ + HK + HV == 0) return 0;
  if (hd != 64 && hd != 128 && hd != 256) return -2;
  const void* base[6] = {HQ ? q : nullptr, HQ ? qo : nullptr, HK ? k : nullptr, HK ? ko : nullptr, HV ? v : nullptr, HV ? vo : nullptr};
  const long ld[6] = {q_is, q_os, k_is, k_os, v_is, v_os};
  for (int i = 0; i < 6; ++i)
    if (base[i] && (((uintptr_t)base[i] & 15) || ld[i] % 8)) return -2;
  const unsigned blocks = (T + 512 / hd - 1) / (512 / hd);
  if (q_fp32)
    rope_qkv_kernel<float><<<blocks, 256, 0, s>>>((const float*)q, q_is, (bf16*)qo, q_os, HQ, (const bf16*)k, k_is, (bf16*)ko, k_os,
                                                  (const bf16*)v, v_is, (bf16*)vo, v_os, HK, HV, pos, inv_freq, T, hd, inverse);
  else
    rope_qkv_kernel<bf16><<<blocks, 256, 0, s>>>((const bf16*)q, q_is, (bf16*)qo, q_os, HQ, (const bf16*)k, k_is, (bf16*)ko, k_os,
                                                 (const bf16*)v, v_is, (bf16*)vo, v_os, HK, HV, pos, inv_freq, T, hd, inverse);
  CHECK_LAUNCH();
}

int ftb_glu_fwd(const void* gate, const void* up, void* out, long T, int F, int ld_in, int ld_out, int kind,
                cudaStream_t s) {
  if (T == 0) return 0;
  if (F % 8 || ld_in % 8 || ld_out % 8) return -2;
  const long nvec = T * (F / 8);
  const int blocks = (int)((nvec + 255) / 256 < 148 * 16 ? (nvec + 255) / 256 : 148 * 16);
  glu_fwd_kernel<<<blocks, 256, 0, s>>>((const bf16*)gate, (const bf16*)up, (bf16*)out, T, F, ld_in, ld_out, kind);
  CHECK_LAUNCH();
}
int ftb_glu_bwd(const void* dact, const void* gate, const void* up, void* dgate, void* dup, void* act_out, long T,
                int F, int ld_in, int ld_d, int ld_act, int kind, cudaStream_t s) {
  if (T == 0) return 0;
  if (F % 8 || ld_in % 8 || ld_d % 8 || ld_act % 8) return -2;
  const long nvec = T * (F / 8);
  const int blocks = (int)((nvec + 255) / 256 < 148 * 16 ? (nvec + 255) / 256 : 148 * 16);
  glu_bwd_kernel<<<blocks, 256, 0, s>>>((const bf16*)dact, (const bf16*)gate, (const bf16*)up, (bf16*)dgate,
                                        (bf16*)dup, (bf16*)act_out, T, F, ld_in, ld_d, ld_act, kind);
  CHECK_LAUNCH();
}

int ftb_glu_bwd_weighted(const void* dact, const void* gate, const void* up, const float* w_row, void* dgate, void* dup,
                         void* act_w, float* dw_row, long T, int F, int ld_in, int ld_d, int kind, cudaStream_t s) {
  if (T == 0) return 0;
  if (F % 8 || ld_in % 8 || ld_d % 8) return -2;
  glu_bwd_weighted_kernel<<<(unsigned)T, 128, 0, s>>>((const bf16*)dact, (const bf16*)gate, (const bf16*)up, w_row,
                                                      (bf16*)dgate, (bf16*)dup, (bf16*)act_w, dw_row, F, ld_in, ld_d, kind);
  CHECK_LAUNCH();
}

int ftb_softmax_ce(void* logits, const long* targets, const float* loss_mask, float* loss, int T, int V, long ld,
                   float grad_scale, float softcap, long ignore_index, cudaStream_t s) {
  if (T == 0) return 0;
  if (ld % 8) return -2;
  run_softmax_ce<true>((bf16*)logits, targets, loss_mask, loss, T, V, ld, grad_scale, softcap, ignore_index, s);
  CHECK_LAUNCH();
}
// The losses alone; the logits stay as they are.
int ftb_softmax_ce_loss(const void* logits, const long* targets, const float* loss_mask, float* loss, int T, int V, long ld,
                        float softcap, long ignore_index, cudaStream_t s) {
  if (T == 0) return 0;
  if (ld % 8) return -2;
  run_softmax_ce<false>((bf16*)logits, targets, loss_mask, loss, T, V, ld, 0.f, softcap, ignore_index, s);
  CHECK_LAUNCH();
}
// bytes of zeros at p (a memory node under capture)
int ftb_zero(void* p, long bytes, cudaStream_t s) {
  return bytes > 0 ? (int)cudaMemsetAsync(p, 0, (size_t)bytes, s) : 0;
}

int ftb_embedding_fwd(const long* tokens, const void* table, void* out, int T, int D, float scale, cudaStream_t s) {
  if (T == 0) return 0;
  if (D % 8) return -2;
  embedding_fwd_kernel<<<T, 128, 0, s>>>(tokens, (const bf16*)table, (bf16*)out, T, D, scale);
  CHECK_LAUNCH();
}
int ftb_embedding_bwd(const long* sorted_tok, const long* order, const void* dy, void* grad, int T, int D,
                      float scale, int grad_fp32, cudaStream_t s) {
  if (T == 0) return 0;
  if (D % 8) return -2;
  embedding_bwd_kernel<<<T, 128, 0, s>>>(sorted_tok, order, (const bf16*)dy, grad, T, D, scale, grad_fp32);
  CHECK_LAUNCH();
}

// Tensors are passed as parallel arrays (host memory) of length `count` <= 24.
int ftb_adamw_multi(int count, void** p, const void** g, void** m, void** v, const long* n, const float* lr,
                    const float* wd, const int* p_dt, const int* g_dt, const int* s_dt, float beta1, float beta2,
                    float eps, float bc1, float bc2, float grad_scale, cudaStream_t s) {
  if (count <= 0) return 0;
  if (count > ADAM_MAX) return -2;
  AdamArgs a;
  long blocks = 0;
  for (int i = 0; i < count; ++i) {
    a.t[i].p = p[i]; a.t[i].g = g[i]; a.t[i].m = m[i]; a.t[i].v = v[i];
    a.t[i].n = n[i]; a.t[i].block_start = blocks;
    a.t[i].lr = lr[i]; a.t[i].wd = wd[i];
    a.t[i].p_dt = p_dt[i]; a.t[i].g_dt = g_dt[i]; a.t[i].s_dt = s_dt[i];
    a.t[i].vec = (((uintptr_t)p[i] | (uintptr_t)g[i] | (uintptr_t)m[i] | (uintptr_t)v[i]) & 15) == 0;
    blocks += (n[i] + ADAM_PER_BLOCK - 1) / ADAM_PER_BLOCK;
  }
  a.count = count; a.beta1 = beta1; a.beta2 = beta2; a.eps = eps; a.bc1 = bc1; a.bc2 = bc2; a.grad_scale = grad_scale;
  if (blocks == 0) return 0;
  adamw_kernel<<<(unsigned)blocks, ADAM_THREADS, 0, s>>>(a);
  CHECK_LAUNCH();
}

// `count` <= 64 bf16 matrices of n elements each (a multiple of 8, all pointers on 16 bytes); partial: count * blocks floats,
// blocks = ceil(n / 16384); x: matrix i at x + i * x_stride.  dtype codes as for AdamW.
int ftb_muon_prepare(int count, const void** g, void** m, long n, long x_stride, int g_dt, int m_dt, float beta, int nesterov,
                     float grad_scale, float* partial, void* x, cudaStream_t s) {
  if (count <= 0 || n <= 0) return 0;
  if (count > MUON_MAX || (n & 7)) return -2;
  MuonArgs a;
  for (int i = 0; i < count; ++i) {
    if (((uintptr_t)g[i] | (uintptr_t)m[i]) & 15) return -2;
    a.g[i] = g[i]; a.m[i] = m[i]; a.p[i] = nullptr;
  }
  a.n = n; a.x_stride = x_stride; a.g_dt = g_dt; a.m_dt = m_dt; a.nesterov = nesterov; a.beta = beta;
  a.grad_scale = grad_scale; a.keep = 0.f; a.step = 0.f;
  const dim3 grid((unsigned)((n + MUON_PER_BLOCK - 1) / MUON_PER_BLOCK), count);
#define FTB_MUON(GF, MF)                                             \
  muon_norm_kernel<GF, MF><<<grid, MUON_THREADS, 0, s>>>(a, partial); \
  muon_prepare_kernel<GF, MF><<<grid, MUON_THREADS, 0, s>>>(a, partial, (bf16*)x)
  if (g_dt && m_dt) { FTB_MUON(true, true); }
  else if (g_dt) { FTB_MUON(true, false); }
  else if (m_dt) { FTB_MUON(false, true); }
  else { FTB_MUON(false, false); }
#undef FTB_MUON
  CHECK_LAUNCH();
}
int ftb_muon_apply(int count, void** p, const void* x, long n, long x_stride, float keep, float step, cudaStream_t s) {
  if (count <= 0 || n <= 0) return 0;
  if (count > MUON_MAX || (n & 7)) return -2;
  MuonArgs a;
  for (int i = 0; i < count; ++i) {
    if ((uintptr_t)p[i] & 15) return -2;
    a.g[i] = nullptr; a.m[i] = nullptr; a.p[i] = p[i];
  }
  a.n = n; a.x_stride = x_stride; a.g_dt = a.m_dt = a.nesterov = 0; a.beta = a.grad_scale = 0.f; a.keep = keep; a.step = step;
  muon_apply_kernel<<<dim3((unsigned)((n + MUON_PER_BLOCK - 1) / MUON_PER_BLOCK), count), MUON_THREADS, 0, s>>>(a, (const bf16*)x);
  CHECK_LAUNCH();
}

// Blocks (partial sums) a tensor of n elements takes in ftb_sumsq.
long ftb_sumsq_blocks(long n) { return (n + SQ_PER_BLOCK - 1) / SQ_PER_BLOCK; }
// partial[0 .. blocks) of `count` <= 64 tensors, in order; then ftb_sumsq_total over the partials of all calls.
int ftb_sumsq(int count, const void** p, const long* n, const int* dt, float* partial, cudaStream_t s) {
  if (count <= 0) return 0;
  if (count > SQ_MAX) return -2;
  SqArgs a;
  long blocks = 0;
  for (int i = 0; i < count; ++i) {
    a.t[i].p = p[i]; a.t[i].n = n[i]; a.t[i].block_start = blocks; a.t[i].dt = dt[i];
    a.t[i].vec = ((uintptr_t)p[i] & 15) == 0;
    blocks += ftb_sumsq_blocks(n[i]);
  }
  a.count = count;
  if (blocks == 0) return 0;
  sumsq_kernel<<<(unsigned)blocks, SQ_THREADS, 0, s>>>(a, partial);
  CHECK_LAUNCH();
}
int ftb_sumsq_total(const float* partial, long n, float* out, cudaStream_t s) {
  sumsq_total_kernel<<<1, 1024, 0, s>>>(partial, n, out);
  CHECK_LAUNCH();
}

int ftb_gated_rmsnorm_fwd(const void* o, const void* z, const float* w, void* y, long rows, int D, float eps,
                          cudaStream_t s) {
  if (rows == 0) return 0;
  gated_rmsnorm_fwd_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, s>>>((const bf16*)o, (const bf16*)z, w, (bf16*)y,
                                                                       rows, D, eps);
  CHECK_LAUNCH();
}
int ftb_l2norm_fwd(const void* x, void* y, float* rnorm, long rows, int D, float eps, cudaStream_t s) {
  if (rows == 0) return 0;
  l2norm_fwd_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, s>>>((const bf16*)x, (bf16*)y, rnorm, rows, D, eps);
  CHECK_LAUNCH();
}

// Router backward (one warp per token, E <= 256): dlogits (T, E) fp32 from the gradient of the K routing weights.
//   mode 0 (softmax over the K picks):  dl[e_k] = w_k (dw_k - sum_j w_j dw_j), 0 elsewhere
//   mode 1 (softmax over E, then pick): dl = p * (dp - sum p dp) with dp = dw scattered to the picks
// (flextrain/ops/_kernels/moe.py:360-458).
__global__ void topk_route_bwd_kernel(const float* __restrict__ dw, const bf16* __restrict__ logits,
                                      const float* __restrict__ w, const int* __restrict__ experts,
                                      float* __restrict__ dl, int T, int E, int K, int mode) {
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= T) return;
  const int lane = threadIdx.x & 31;
  float* out = dl + (size_t)t * E;
  const float* dwt = dw + (size_t)t * K;
  const int* et = experts + (size_t)t * K;
  if (mode == 0) {
    const float* wt = w + (size_t)t * K;
    float dot = 0.f;
    for (int k = 0; k < K; ++k) dot += wt[k] * dwt[k];
    for (int e = lane; e < E; e += 32) out[e] = 0.f;
    __syncwarp();
    if (lane < K) out[et[lane]] = wt[lane] * (dwt[lane] - dot);
    return;
  }
  float v[8], dp[8];
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int e = lane + j * 32;
    v[j] = e < E ? __bfloat162float(logits[(size_t)t * E + e]) : -INFINITY;
    dp[j] = 0.f;
    mx = fmaxf(mx, v[j]);
  }
  mx = warp_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) { v[j] = (lane + j * 32 < E) ? __expf(v[j] - mx) : 0.f; sum += v[j]; }
  sum = warp_sum(sum);
  for (int k = 0; k < K; ++k) {
    const int e = et[k];
    if ((e & 31) == lane) dp[e >> 5] = dwt[k];
  }
  float dot = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) { v[j] /= sum; dot += v[j] * dp[j]; }
  dot = warp_sum(dot);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int e = lane + j * 32;
    if (e < E) out[e] = v[j] * (dp[j] - dot);
  }
}

// Load-balance auxiliary gradient added into dlogits (flextrain/ops/_kernels/moe.py:601-646):
//   dl[t, e] += alpha * p[t, e] * (gvec[e] - sum_j p[t, j] gvec[j]),  p = softmax(logits[t, :]),
//   gvec[e] = counts[e] / n_slots * E / total_tokens   (the routed fractions are constants of the step).
// One warp per token, E <= 256.
__global__ void load_balance_bwd_kernel(const bf16* __restrict__ logits, const int* __restrict__ counts,
                                        float* __restrict__ dl, int T, int E, float alpha, float gscale) {
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= T) return;
  const int lane = threadIdx.x & 31;
  float v[8], gv[8];
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int e = lane + j * 32;
    v[j] = e < E ? __bfloat162float(logits[(size_t)t * E + e]) : -INFINITY;
    gv[j] = e < E ? (float)counts[e] * gscale : 0.f;
    mx = fmaxf(mx, v[j]);
  }
  mx = warp_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) { v[j] = (lane + j * 32 < E) ? __expf(v[j] - mx) : 0.f; sum += v[j]; }
  sum = warp_sum(sum);
  float dot = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) { v[j] /= sum; dot += v[j] * gv[j]; }
  dot = warp_sum(dot);
  float* out = dl + (size_t)t * E;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int e = lane + j * 32;
    if (e < E) out[e] += alpha * v[j] * (gv[j] - dot);
  }
}

int ftb_load_balance_bwd(const void* logits, const int* counts, float* dl, int T, int E, float alpha, float gscale,
                         cudaStream_t s) {
  if (T == 0) return 0;
  if (E > 256) return -2;
  load_balance_bwd_kernel<<<(T + 7) / 8, 256, 0, s>>>((const bf16*)logits, counts, dl, T, E, alpha, gscale);
  CHECK_LAUNCH();
}

int ftb_topk_route_bwd(const float* dw, const void* logits, const float* w, const int* experts, float* dl, int T, int E,
                       int K, int mode, cudaStream_t s) {
  if (T == 0) return 0;
  if (E > 256 || K > 32) return -2;
  topk_route_bwd_kernel<<<(T + 7) / 8, 256, 0, s>>>(dw, (const bf16*)logits, w, experts, dl, T, E, K, mode);
  CHECK_LAUNCH();
}

int ftb_topk_route(const void* logits, float* weights, int* experts, int T, int E, int K, int mode, cudaStream_t s) {
  if (T == 0) return 0;
  if (E > 256 || K > 16) return -2;
  topk_route_kernel<<<(T + 7) / 8, 256, 0, s>>>((const bf16*)logits, weights, experts, T, E, K, mode);
  CHECK_LAUNCH();
}
int ftb_gather_rows(const void* in, const int* idx, const float* w, void* out, long rows, int D, int idx_div,
                    cudaStream_t s) {
  if (rows == 0) return 0;
  if (D % 8) return -2;
  gather_rows_kernel<<<(unsigned)rows, 128, 0, s>>>((const bf16*)in, idx, w, (bf16*)out, rows, D, idx_div);
  CHECK_LAUNCH();
}
int ftb_moe_combine(const void* y, const int* inv, const float* w, const void* resid, void* out, int T, int K, int D,
                    cudaStream_t s) {
  if (T == 0) return 0;
  if (D % 8) return -2;
  moe_combine_kernel<<<T, 128, 0, s>>>((const bf16*)y, inv, w, (const bf16*)resid, (bf16*)out, T, K, D);
  CHECK_LAUNCH();
}

}  // extern "C"
