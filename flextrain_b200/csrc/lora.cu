// Gradients of rank-r adapters (r = 8, 16 or 32) of all the projections that share an input, in three launches:
//   down    xa_i = x A_i^T and dyb_i = dy_i B_i, (tokens, r) bf16: x is read once for up to three adapters
//   up      parts of gA_i = dyb_i^T x and gB_i = dy_i^T xa_i over runs of tokens, fp32
//   finish  g <- g + s * (sum of the parts), rounded once
// Four GEMMs a projection did the same on 128-row tensor-core tiles of which r columns are in use: x is read twice by
// each projection, few tiles are in flight, and a launch of some 10 us stands behind each.
// One projection of 4096 columns from 4096, r = 16: 16384 tokens 134 -> 116 us, 2048 tokens 71 -> 34; q, k and v of it (4096, 1024,
// 1024) 320 -> 144 and 194 -> 42; gate and up (2 x 14336) 468 -> 380 and 163 -> 91.  Reading x and dy twice takes 83, 104 and 333 us
// at 16384 tokens.
// Both kernels are bound by reading x and dy.  mma.sync, not tcgen05: with N = r there is one m16n8k16 for each 512 bytes that
// are read, and operands go from global memory (down) or shared memory (up) straight into its fragments.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace {

typedef __nv_bfloat16 bf16;
constexpr int MAXW = 3;                          // adapters that share an input
constexpr int MAXP = MAXW + 1;                   // operands to multiply: the input, and each projection's output gradient

__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t transpose8(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ldsm_t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

__device__ __forceinline__ void ldsm(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
// Where 16-byte piece c of row r of a (rows, R) tile lies within its row: the pieces that ldmatrix reads together, one of each of
// eight rows, are in eight different groups of banks.
template <int R>
__device__ __forceinline__ int zpiece(int r, int c) { return R == 16 ? c ^ ((r >> 2) & 1) : R == 32 ? c ^ ((r >> 1) & 3) : c; }

// ------------------------------------------------------------------------------------------------ down
constexpr int DROWS = 128;
// Rows through shared memory from here: blocks of 128 rows leave SMs idle below (K = N = 4096, r = 16, all three launches: 4096 tokens
// 54 us against 52 of `down`, 14336 to 4096 columns 120 against 89; 8192 tokens 77 against 85 and 153 against 144; 16384: 116 against
// 136 and 227 against 257).
constexpr int MANY_TOKENS = 8192;
__host__ __device__ constexpr int down_stages(int R) { return R == 32 ? 3 : 4; }
__host__ __device__ constexpr int down_stage_bytes(int R) { return (DROWS + MAXW * R + 8) * 128; }
struct Down {
  const bf16* x;                                 // (T, K), rows ld elements apart
  long ld;
  int K, nw, kn;                                 // kn: the weight is (K, r), else (r, K)
  const bf16* w[MAXW];
  bf16* out[MAXW];                               // (T, r)
};
struct DownArgs {
  Down p[MAXP];
  int T;
};

// A block has 32 rows, its warps parts of K.  Within 32 of K, lane (row, q) reads the 8 consecutive elements from 8 q on, 16 bytes; the
// multiplication takes them as k = 2 q, 2 q + 1, 2 q + 8, 2 q + 9 of two steps of 16, and the weight's fragments are read in the
// same order (a sum does not mind).
template <int R, int NW, bool KN>
__device__ __forceinline__ void down(const Down& p, int T, float* red) {
  constexpr int NB = R / 8;                      // column tiles of a weight
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = lane & 3, g = lane >> 2;
  const int row0 = blockIdx.x * 32;
  const bf16* xp[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) xp[i] = p.x + (long)min(row0 + g + 8 * i, T - 1) * p.ld + 8 * q;
  float acc[2][NW * NB][4] = {};
  const int groups = p.K / 32, per = (groups + 7) / 8, lo = warp * per, hi = min(groups, lo + per);
#pragma unroll 2
  for (int k = lo; k < hi; ++k) {
    uint4 x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const uint4*>(xp[i] + k * 32);
#pragma unroll
    for (int w = 0; w < NW; ++w)
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        uint32_t b[4];
        if (KN) {
#pragma unroll
          for (int s = 0; s < 4; ++s)            // rows 8 (j / 2) + 2 s + j % 2 of the group, j = g; turned over: pairs of K for a column
            b[s] = transpose8(*reinterpret_cast<const uint32_t*>(p.w[w] + (long)(k * 32 + 8 * (g >> 1) + 2 * s + (g & 1)) * R + nb * 8 + 2 * q));
        } else {
          const uint4 u = *reinterpret_cast<const uint4*>(p.w[w] + (long)(nb * 8 + g) * p.K + k * 32 + 8 * q);
          b[0] = u.x; b[1] = u.y; b[2] = u.z; b[3] = u.w;
        }
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          mma(acc[m][w * NB + nb], x[2 * m].x, x[2 * m + 1].x, x[2 * m].y, x[2 * m + 1].y, b[0], b[1]);
          mma(acc[m][w * NB + nb], x[2 * m].z, x[2 * m + 1].z, x[2 * m].w, x[2 * m + 1].w, b[2], b[3]);
        }
      }
  }
  // the parts of K are added up in shared memory: [part][row][column of all weights]
  constexpr int COLS = NW * R;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NW * NB; ++n) {
      float* at = red + ((warp * 32 + m * 16 + g) * COLS + n * 8 + 2 * q);
      *reinterpret_cast<float2*>(at) = make_float2(acc[m][n][0], acc[m][n][1]);
      *reinterpret_cast<float2*>(at + 8 * COLS) = make_float2(acc[m][n][2], acc[m][n][3]);
    }
  __syncthreads();
  for (int i = threadIdx.x; i < 32 * COLS / 2; i += 256) {
    const int r = i / (COLS / 2), c = (i - r * (COLS / 2)) * 2;
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float2 v = *reinterpret_cast<const float2*>(red + (u * 32 + r) * COLS + c);
      s.x += v.x;
      s.y += v.y;
    }
    const int row = row0 + r;
    if (row < T) *reinterpret_cast<__nv_bfloat162*>(p.out[c / R] + (long)row * R + c % R) = __floats2bfloat162_rn(s.x, s.y);
  }
}
template <int R>
__global__ void __launch_bounds__(256) lora_down_kernel(const DownArgs a) {
  extern __shared__ __align__(16) float red[];
  const Down& p = a.p[blockIdx.y];
  if (p.kn) down<R, 1, true>(p, a.T, red);
  else if (p.nw == 1) down<R, 1, false>(p, a.T, red);
  else if (p.nw == 2) down<R, 2, false>(p, a.T, red);
  else down<R, 3, false>(p, a.T, red);
}

// The same with everything through shared memory: 128 rows, K in steps of 64, four warps along the rows and two halves of a step.
// Here a warp reads its share of the weights from shared memory, where `down` reads all of them from L2.
template <int R, int NW, bool KN>
__device__ __forceinline__ void down_rows(const Down& p, int T, char* sm) {
  constexpr int NB = R / 8, NT = NW * NB, ZP = R / 8, ST = down_stages(R), STAGE = down_stage_bytes(R), XB = DROWS * 128;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wr = warp & 3, wk = warp >> 2;
  const int row0 = blockIdx.x * DROWS, steps = (p.K + 63) / 64;
  const int xr = tid >> 3, xc = tid & 7, K = p.K;
  const long ld = p.ld;
  const bf16 *x0 = p.x, *w0 = p.w[0], *w1 = p.w[1], *w2 = p.w[2];      // (copies: asm would have the arguments read again)
  const bf16* xp = x0 + (long)(row0 + xr) * ld + xc * 8;
  const uint32_t xd = smem_addr(sm) + xr * 128 + ((xc ^ (xr & 7)) << 4);
  auto fetch = [&](int s) {
    if (s < steps) {
      const uint32_t so = (s % ST) * STAGE, st = smem_addr(sm) + so;
      const int k0 = s * 64;
#pragma unroll
      for (int u = 0; u < DROWS / 32; ++u) {
        const bool on = row0 + xr + u * 32 < T && k0 + xc * 8 < K;
        cp16(xd + so + u * 32 * 128, on ? xp + (long)u * 32 * ld + k0 : x0, on);
      }
      if (KN) {
        for (int i = tid; i < 64 * ZP; i += 256) {
          const int r = i / ZP, c = i - r * ZP;
          const bool on = k0 + r < K;
          cp16(st + XB + r * (R * 2) + (zpiece<R>(r, c) << 4), w0 + (on ? (long)(k0 + r) * R + c * 8 : 0), on);
        }
      } else {
#pragma unroll
        for (int w = 0; w < NW; ++w)
          for (int i = tid; i < R * 8; i += 256) {
            const int r = i >> 3, c = i & 7;
            const bool on = k0 + c * 8 < K;
            const bf16* ws = w == 0 ? w0 : w == 1 ? w1 : w2;
            cp16(st + XB + (w * R + r) * 128 + ((c ^ (r & 7)) << 4), ws + (on ? (long)r * K + k0 + c * 8 : 0), on);
          }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int s = 0; s < ST - 1; ++s) fetch(s);
  float acc[2][NT][4] = {};
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
    __syncthreads();
    fetch(s + ST - 1);
    const uint32_t st = smem_addr(sm) + (s % ST) * STAGE;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int kb = wk * 2 + h;
      uint32_t x[2][4];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int r = wr * 32 + m * 16 + (lane & 15), c = kb * 2 + (lane >> 4);
        ldsm(x[m], st + r * 128 + ((c ^ (r & 7)) << 4));
      }
#pragma unroll
      for (int n = 0; n < NT; n += 2) {          // (with an odd number of tiles the last one's neighbour is read and not used)
        uint32_t b[4];
        if (KN) {
          const int r = kb * 16 + (lane & 15);
          ldsm_t(b, st + XB + r * (R * 2) + (zpiece<R>(r, NB == 1 ? 0 : n + (lane >> 4)) << 4));
        } else {
          const int r = n * 8 + (lane & 7) + ((lane >> 4) << 3), c = kb * 2 + ((lane >> 3) & 1);
          ldsm(b, st + XB + r * 128 + ((c ^ (r & 7)) << 4));
        }
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          mma(acc[m][n], x[m][0], x[m][1], x[m][2], x[m][3], b[0], b[1]);
          if (n + 1 < NT) mma(acc[m][n + (n + 1 < NT)], x[m][0], x[m][1], x[m][2], x[m][3], b[2], b[3]);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* red = reinterpret_cast<float*>(sm);     // the second half's sums, in the order of the first half's registers
  const int at = wr * 32 + lane;
  if (wk)
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
        *reinterpret_cast<float4*>(red + ((m * NT + n) * 128 + at) * 4) = make_float4(acc[m][n][0], acc[m][n][1], acc[m][n][2], acc[m][n][3]);
  __syncthreads();
  if (!wk)
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const float4 o = *reinterpret_cast<const float4*>(red + ((m * NT + n) * 128 + at) * 4);
        const int row = row0 + wr * 32 + m * 16 + (lane >> 2), c = (n % NB) * 8 + (lane & 3) * 2;
        bf16* out = p.out[n / NB] + (long)row * R + c;
        if (row < T) *reinterpret_cast<__nv_bfloat162*>(out) = __floats2bfloat162_rn(acc[m][n][0] + o.x, acc[m][n][1] + o.y);
        if (row + 8 < T) *reinterpret_cast<__nv_bfloat162*>(out + 8 * R) = __floats2bfloat162_rn(acc[m][n][2] + o.z, acc[m][n][3] + o.w);
      }
}
template <int R>
__global__ void __launch_bounds__(256) lora_down_rows_kernel(const DownArgs a) {
  extern __shared__ __align__(128) char sm[];
  const Down& p = a.p[blockIdx.y];
  if (p.kn) down_rows<R, 1, true>(p, a.T, sm);
  else if (p.nw == 1) down_rows<R, 1, false>(p, a.T, sm);
  else if (p.nw == 2) down_rows<R, 2, false>(p, a.T, sm);
  else down_rows<R, 3, false>(p, a.T, sm);
}

// ------------------------------------------------------------------------------------------------ up
struct Up {
  const bf16* y;                                 // (T, I), rows ld elements apart
  long ld;
  int I, nz, blocks;                             // blocks: the problem's column blocks of 128, counted with those before it
  const bf16* z[MAXW];                           // (T, r)
  float* part[MAXW];                             // (runs, I, r)
};
struct UpArgs {
  Up p[MAXP];
  int T, run;                                    // run: tokens of a part, a multiple of 64
};
constexpr int STAGES = 4, STEP = 64;
__host__ __device__ constexpr int up_stage_bytes(int R) { return STEP * 256 + MAXW * STEP * R * 2; }

// 128 columns of y against the r columns of up to three z, over a run of tokens; a warp has 32 columns.
template <int R>
__global__ void __launch_bounds__(128) lora_up_kernel(const UpArgs a) {
  extern __shared__ __align__(128) char sm[];
  constexpr int NB = R / 8, ZP = R / 8, STAGE = up_stage_bytes(R);           // ZP: 16-byte pieces in a row of z
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int pi = 0;
  while (static_cast<int>(blockIdx.x) >= a.p[pi].blocks) ++pi;
  const Up p = a.p[pi];                          // (a copy: the index is not known to the compiler, and asm would have it read again)
  const int col0 = (blockIdx.x - (pi ? a.p[pi - 1].blocks : 0)) * 128;
  const int t0 = blockIdx.y * a.run, t1 = min(a.T, t0 + a.run), steps = (t1 - t0 + STEP - 1) / STEP;
  const int yr = tid >> 4, yc = tid & 15;        // this thread's piece of y: rows yr + 8 u
  const bool yin = col0 + yc * 8 < p.I;
  const bf16* yp = p.y + (long)(t0 + yr) * p.ld + (yin ? col0 + yc * 8 : 0);
  const uint32_t yd = smem_addr(sm) + yr * 256 + (((yc & 8) | ((yc ^ yr) & 7)) << 4);
  auto fetch = [&](int s) {
    if (s < steps) {
      const uint32_t so = (s % STAGES) * STAGE, st = smem_addr(sm) + so;
      const int t = t0 + s * STEP, left = t1 - t;
      const bf16* src = yp + (long)s * STEP * p.ld;
#pragma unroll
      for (int u = 0; u < STEP / 8; ++u) {
        const bool on = yr + u * 8 < left && yin;
        cp16(yd + so + u * 8 * 256, on ? src + (long)u * 8 * p.ld : p.y, on);
      }
#pragma unroll
      for (int w = 0; w < MAXW; ++w)
        if (w < p.nz)
#pragma unroll
          for (int u = 0; u < (STEP * ZP + 127) / 128; ++u) {
            const int i = tid + u * 128, r = i / ZP, c = i - r * ZP;
            const bool on = r < left;
            if (STEP * ZP % 128 == 0 || r < STEP)
              cp16(st + STEP * 256 + (w * STEP + r) * (R * 2) + (zpiece<R>(r, c) << 4), p.z[w] + (on ? (long)(t + r) * R + c * 8 : 0), on);
          }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int s = 0; s < STAGES - 1; ++s) fetch(s);
  float acc[MAXW][2][NB][4] = {};
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();
    fetch(s + STAGES - 1);
    const uint32_t st = smem_addr(sm) + (s % STAGES) * STAGE;
#pragma unroll
    for (int kb = 0; kb < STEP / 16; ++kb) {
      uint32_t y[2][4];                          // y^T: rows = columns of y, k = tokens
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int r = kb * 16 + (lane & 7) + ((lane >> 4) << 3), c = warp * 4 + m * 2 + ((lane >> 3) & 1);
        ldsm_t(y[m], st + r * 256 + (((c & 8) | ((c ^ r) & 7)) << 4));
      }
#pragma unroll
      for (int w = 0; w < MAXW; ++w) {
        if (w < p.nz) {
#pragma unroll
          for (int n = 0; n < NB; n += 2) {
            uint32_t b[4];                       // (with one column tile it is read twice)
            const int r = kb * 16 + (lane & 15);
            ldsm_t(b, st + STEP * 256 + (w * STEP + r) * (R * 2) + (zpiece<R>(r, NB == 1 ? 0 : n + (lane >> 4)) << 4));
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              mma(acc[w][m][n], y[m][0], y[m][1], y[m][2], y[m][3], b[0], b[1]);
              if (NB > 1) mma(acc[w][m][n + (NB > 1)], y[m][0], y[m][1], y[m][2], y[m][3], b[2], b[3]);
            }
          }
        }
      }
    }
  }
#pragma unroll
  for (int w = 0; w < MAXW; ++w)
    if (w < p.nz)
#pragma unroll
      for (int n = 0; n < NB; ++n)
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int i = col0 + warp * 32 + (lane >> 2) + h * 8;
          if (i < p.I)
            *reinterpret_cast<float2*>(p.part[w] + ((long)blockIdx.y * p.I + i) * R + n * 8 + (lane & 3) * 2) =
                make_float2(acc[w][h >> 1][n][2 * (h & 1)], acc[w][h >> 1][n][2 * (h & 1) + 1]);
        }
}

// ------------------------------------------------------------------------------------------------ finish
struct Fin {
  const float* part;                             // (runs, I, r)
  void* g;                                       // (I, r), or (r, I) with `turned`
  int I, turned, blocks;                         // blocks: of 1024 elements, counted with those before
};
struct FinArgs {
  Fin p[2 * MAXW];
  int R, runs, fp32;
  float scale;
};
__global__ void __launch_bounds__(256) lora_finish_kernel(const FinArgs a) {
  __shared__ float turn[1024];
  int pi = 0;
  while (static_cast<int>(blockIdx.x) >= a.p[pi].blocks) ++pi;
  const Fin& p = a.p[pi];
  const long n = (long)p.I * a.R, e0 = (long)(blockIdx.x - (pi ? a.p[pi - 1].blocks : 0)) * 1024, e = e0 + threadIdx.x * 4;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (e < n)
    for (int u = 0; u < a.runs; ++u) {
      const float4 v = *reinterpret_cast<const float4*>(p.part + u * n + e);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
  float f[4] = {s.x, s.y, s.z, s.w};
  long at[4];
  if (p.turned) {                                // 1024 / r columns of g: elements of a column lie r apart, rows of g are written
    *reinterpret_cast<float4*>(turn + threadIdx.x * 4) = s;
    __syncthreads();
    const int w = 1024 / a.R;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int x = threadIdx.x + u * 256, r = x / w, c = x - r * w;
      f[u] = turn[c * a.R + r];
      at[u] = e0 / a.R + c < p.I ? (long)r * p.I + e0 / a.R + c : -1;
    }
  } else {
#pragma unroll
    for (int u = 0; u < 4; ++u) at[u] = e + u < n ? e + u : -1;
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
    if (at[u] >= 0) {
      if (a.fp32) reinterpret_cast<float*>(p.g)[at[u]] += a.scale * f[u];
      else {
        bf16* g = reinterpret_cast<bf16*>(p.g) + at[u];
        *g = __float2bfloat16(__bfloat162float(*g) + a.scale * f[u]);
      }
    }
}

template <int R>
int run_all(const DownArgs& d, int nd, const UpArgs& u, int nu, int runs, const FinArgs& f, int nf, int nw, cudaStream_t s) {
  cudaError_t e;
  auto rows = lora_down_rows_kernel<R>;
  auto direct = lora_down_kernel<R>;
  auto up = lora_up_kernel<R>;
  const bool many = d.T >= MANY_TOKENS;
  const int down_smem = many ? down_stages(R) * down_stage_bytes(R) : 8 * 32 * nw * R * 4;
  // (the most that a kernel may ever ask for, whatever this call needs: another thread's call may be between this and its launch)
  e = many ? cudaFuncSetAttribute(rows, cudaFuncAttributeMaxDynamicSharedMemorySize, down_stages(R) * down_stage_bytes(R))
           : cudaFuncSetAttribute(direct, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * 32 * MAXW * R * 4);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(up, cudaFuncAttributeMaxDynamicSharedMemorySize, STAGES * up_stage_bytes(R));
  if (e != cudaSuccess) return -300 - (int)e;
  if (many) rows<<<dim3((d.T + DROWS - 1) / DROWS, nd), 256, down_smem, s>>>(d);
  else direct<<<dim3((d.T + 31) / 32, nd), 256, down_smem, s>>>(d);
  up<<<dim3(u.p[nu - 1].blocks, runs), 128, STAGES * up_stage_bytes(R), s>>>(u);
  lora_finish_kernel<<<f.p[nf - 1].blocks, 256, 0, s>>>(f);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -400 - (int)e;
}

// Runs of tokens: as many as make (waves of 2 blocks an SM) x (steps of a run, and 4 for its start and its end) least, and as keep
// the parts (one_run bytes each) within the workspace that a plan sets aside.
constexpr long PART_BYTES = 64L << 20;
int runs_of(int T, int blocks, long one_run, int* run) {
  long best = 0;
  int runs = 1;
  *run = STEP;
  for (int n = 1; n <= 32 && (n - 1) * 256 < T && (n == 1 || n * one_run <= PART_BYTES); ++n) {
    const int steps = ((T + n - 1) / n + STEP - 1) / STEP;
    const long cost = (long)((blocks * n + 2 * 148 - 1) / (2 * 148)) * (steps + 4);
    if (n == 1 || cost < best) { best = cost; runs = n; *run = steps * STEP; }
  }
  return (T + *run - 1) / *run;
}
int blocks_of(int I) { return (I + 127) / 128; }

}  // namespace

extern "C" {

// Bytes of workspace for n adapters of rank R on an input of K columns with outputs of N[i] columns, T tokens.
long ftb_lora_wgrad_bytes(int n, int T, int K, const int* N, int R) {
  int blocks = blocks_of(K), run;
  long columns = (long)n * K;
  for (int i = 0; i < n; ++i) { blocks += blocks_of(N[i]); columns += N[i]; }
  return 2L * n * ((long)T * R * 2 + 256) + columns * R * 4 * runs_of(T, blocks, columns * R * 4, &run) + 256;
}

// ga_i (R, K) += scale * (dy_i b_i)^T x,  gb_i (N_i, R) += scale * dy_i^T (x a_i^T)  for n <= 3 adapters of one input x (T, K).
// dy_i (T, N_i) with rows ldy apart; a_i (R, K), b_i (N_i, R), x, dy bf16; gradients bf16 or fp32.  K and N_i multiples of 32, all on
// 16 bytes.  -2: not what the kernels take.
int ftb_lora_wgrad(int n, const void* x, long ldx, int T, int K, const void* const* dy, long ldy, const int* N, const void* const* a,
                   const void* const* b, void* const* ga, void* const* gb, int R, float scale, int fp32, void* work, cudaStream_t s) {
  if (T <= 0 || n <= 0) return 0;
  if (n > MAXW || (R != 8 && R != 16 && R != 32) || K % 32 || ldx % 8 || ldy % 8) return -2;
  uintptr_t all = (uintptr_t)x | (uintptr_t)work;
  for (int i = 0; i < n; ++i) {
    if (N[i] % 32) return -2;
    all |= (uintptr_t)dy[i] | (uintptr_t)a[i] | (uintptr_t)b[i] | (uintptr_t)ga[i] | (uintptr_t)gb[i];
  }
  if (all & 15) return -2;
  char* w = (char*)work;
  auto take = [&](long bytes) {
    char* at = w;
    w += (bytes + 255) / 256 * 256;
    return at;
  };
  DownArgs d = {};
  UpArgs u = {};
  FinArgs f = {};
  d.T = u.T = T;
  int blocks = blocks_of(K);
  long columns = (long)n * K;
  for (int i = 0; i < n; ++i) { blocks += blocks_of(N[i]); columns += N[i]; }
  const int runs = runs_of(T, blocks, columns * R * 4, &u.run);
  bf16 *xa[MAXW], *dyb[MAXW];
  for (int i = 0; i < n; ++i) {
    xa[i] = (bf16*)take((long)T * R * 2);
    dyb[i] = (bf16*)take((long)T * R * 2);
  }
  Down& dx = d.p[0];
  dx.x = (const bf16*)x; dx.ld = ldx; dx.K = K; dx.nw = n; dx.kn = 0;
  Up& ux = u.p[0];
  ux.y = dx.x; ux.ld = ldx; ux.I = K; ux.nz = n; ux.blocks = blocks_of(K);
  int fb = 0;
  for (int i = 0; i < n; ++i) {
    dx.w[i] = (const bf16*)a[i];
    dx.out[i] = xa[i];
    Down& dd = d.p[1 + i];
    dd.x = (const bf16*)dy[i]; dd.ld = ldy; dd.K = N[i]; dd.nw = 1; dd.kn = 1; dd.w[0] = (const bf16*)b[i]; dd.out[0] = dyb[i];
    ux.z[i] = dyb[i];
    ux.part[i] = (float*)take((long)runs * K * R * 4);
    Up& uu = u.p[1 + i];
    uu.y = dd.x; uu.ld = ldy; uu.I = N[i]; uu.nz = 1; uu.blocks = u.p[i].blocks + blocks_of(N[i]); uu.z[0] = xa[i];
    uu.part[0] = (float*)take((long)runs * N[i] * R * 4);
    Fin& fa = f.p[2 * i];
    fa.part = ux.part[i]; fa.g = ga[i]; fa.I = K; fa.turned = 1; fa.blocks = fb += (K * R + 1023) / 1024;
    Fin& fg = f.p[2 * i + 1];
    fg.part = uu.part[0]; fg.g = gb[i]; fg.I = N[i]; fg.turned = 0; fg.blocks = fb += (N[i] * R + 1023) / 1024;
  }
  f.R = R; f.runs = runs; f.fp32 = fp32; f.scale = scale;
  switch (R) {
    case 8: return run_all<8>(d, 1 + n, u, 1 + n, runs, f, 2 * n, n, s);
    case 16: return run_all<16>(d, 1 + n, u, 1 + n, runs, f, 2 * n, n, s);
    default: return run_all<32>(d, 1 + n, u, 1 + n, runs, f, 2 * n, n, s);
  }
}

}  // extern "C"
