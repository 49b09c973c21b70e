// Gated DeltaNet (gated delta rule) recurrence for sm_100a: forward and a hand-derived backward, token-recurrent.
//
// Per value head, with state S (dk x dv), log-decay g_t <= 0, write strength beta_t and unit-norm keys:
//     S^ = exp(g_t) S_{t-1};   r = S^^T k_t;   e = beta_t (v_t - r);   S_t = S^ + k_t e^T;   o_t = scale * S_t^T q_t
// The reference project calls FLA's chunked Triton kernels for this (flextrain/nn/blocks/linear_attn.py:1090-1145,
// 1702-1722).  Here the recurrence is run as written: the dv columns of S evolve independently, so a CTA owns a block
// of NC columns of one (sequence, head) and keeps its dk x NC slice of the state in registers for the whole
// sequence; sequences x heads x column blocks give thousands of CTAs for packed batches and HV * dv / NC CTAs for
// one long sequence.  No chunk-level triangular solves are needed.
//
// Thread layout (128 threads): ti = tid & 15 owns the row pairs {2 ti + 32 j, + 1} (one row, ti, at dk = 16), tj = tid >> 4
// owns columns {tj*CPT + cc}.  The state is kept and updated as pairs of rows in packed fp32 arithmetic (fma.rn.f32x2, one
// instruction for two fused multiply-adds, each rounded as the scalar one), which halves the instructions to issue: 16384
// tokens in 512 to 4096 long sequences, 32 heads of 128 x 128: pass F 6.4 -> 5.7 ms, pass R 6.7 -> 6.6 ms, forward 3.6 ms
// either way.  What bounds them then is the chain of a token (its reductions) in the longest sequences; the tokens of the
// next block are loaded under the current one (16 bytes a thread), which gave 3.7 -> 3.4, 5.7 -> 5.35 and 6.8 -> 6.15 ms.
// Reductions over rows (r, o, de) are 4 xor-shuffles inside a half warp; reductions over columns (dq, dk) are
// accumulated per warp in shared memory over a block of TB tokens and flushed with fp32 atomics once per block.
//
// Backward (adjoint dS of the state, reverse in time), for dO_t given:
//     dS' = dS_t + scale q_t dO_t^T;  de = dS'^T k_t;  dv = beta de;  dbeta = de.(v - r);  dr = -beta de
//     dk_t = dS' e  +  S^ dr;         dq_t = scale S_t dO_t;          dS_{t-1} = exp(g_t) (dS' + k_t dr^T)
//     dg_t = sum_{u >= t} ( q_u.dq_u - k_u.(dS'_u e_u) + k_u.(S^_u dr_u) )  (+ <dS_final, S_final>)
// The terms that need the state itself (dq, S^ dr) are produced by re-running the forward recurrence ("pass F") with
// de from the reverse pass ("pass R").  Both passes add their part of the per-token scalar q.dq - k.(dS' e) + k.(S^ dr)
// into `sacc`; the caller turns it into dg with a suffix sum per sequence.  dq / dk are written per value head in fp32.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace {

typedef __nv_bfloat16 bf16;
constexpr int TB = 8;            // tokens staged per block
constexpr int NT = 128;          // threads per CTA

// error word, read by the host after a step (3: bounds check)
static __device__ int g_error_word = 0;
static __device__ int g_error_where = 0;
__device__ __forceinline__ void set_error(int code, int where) {
  if (atomicCAS(&g_error_word, 0, code) == 0) g_error_where = where;
}

struct GdnArgs {
  const bf16* q;       // (T, HK, DK)
  const bf16* k;       // (T, HK, DK)
  const bf16* v;       // (T, HV, DV)
  const float* g;      // (T, HV)
  const float* beta;   // (T, HV)
  const int* cu;       // (Nseq + 1)
  const float* state_in;   // (Nseq, HV, DK, DV) or null
  float* state_out;        // (Nseq, HV, DK, DV) or null   (forward: final state; pass R: gradient of the initial state)
  bf16* o;             // (T, HV, DV)        forward output
  float* r;            // (T, HV, DV)        forward: prediction S^^T k (kept for the backward) or null
  const bf16* d_o;     // (T, HV, DV)        backward
  float* de;           // (T, HV, DV)        pass R writes, pass F reads
  bf16* dv;            // (T, HV, DV)        pass R
  float* dbeta;        // (T, HV)            pass R (atomic over column blocks)
  float* dq;           // (T, HV, DK) fp32   pass F (atomic over column blocks)
  float* dk;           // (T, HV, DK) fp32   pass R adds dS' e, pass F adds S^ dr (atomic)
  float* sacc;         // (T, HV) fp32       per-token scalar of the gate gradient: q.dq - k.(dS' e) + k.(S^ dr)
  int HK, HV, DV;
  float scale;
  int vec;             // every tensor of rows starts on 16 bytes
  // what is done again for the chunk kernels (REDO)
  long v_gap, dv_gap;  // elements of v / dv between a token's last head and the next token
  const int* only;     // (nseq, HV): run the (sequence, head) pairs marked there, leave the others alone
};

__device__ __forceinline__ float half_warp_sum(float x) {   // over the 16 lanes that share tj
  x += __shfl_xor_sync(0xffffffffu, x, 8);
  x += __shfl_xor_sync(0xffffffffu, x, 4);
  x += __shfl_xor_sync(0xffffffffu, x, 2);
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  return x;
}

// Four per-column partial sums reduced over the 16 lanes of a half warp in 5 shuffles instead of 16: each exchange
// halves the number of columns a lane is responsible for (reduce-scatter), so after the xor-8 and xor-4 steps a lane
// carries one column, c = 2 * bit3(lane) + bit2(lane), and the xor-2 / xor-1 steps finish its sum.
__device__ __forceinline__ float reduce_scatter4(float p0, float p1, float p2, float p3, int lane) {
  const bool hi8 = lane & 8;
  float k0 = hi8 ? p2 : p0, k1 = hi8 ? p3 : p1;
  k0 += __shfl_xor_sync(0xffffffffu, hi8 ? p0 : p2, 8);
  k1 += __shfl_xor_sync(0xffffffffu, hi8 ? p1 : p3, 8);
  const bool hi4 = lane & 4;
  float k = hi4 ? k1 : k0;
  k += __shfl_xor_sync(0xffffffffu, hi4 ? k0 : k1, 4);
  k += __shfl_xor_sync(0xffffffffu, k, 2);
  k += __shfl_xor_sync(0xffffffffu, k, 1);
  return k;
}
// ... and handed back to every lane of the half warp (4 more shuffles).
__device__ __forceinline__ void all_gather4(float k, int lane, float (&out)[4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) out[c] = __shfl_sync(0xffffffffu, k, (lane & 0x13) | (c << 2));
}

// ---- pairs of fp32
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float sum2(f32x2 v) {
  float a, b;
  unpack2(v, a, b);
  return a + b;
}
// The thread's j-th pair of a DK vector; with one row per thread (RPT = 1) the second element does not exist and is 0.
template <int RPT>
__device__ __forceinline__ f32x2 load_pair(const float* x, int ti, int j) {
  if constexpr (RPT == 1) return pack2(x[ti], 0.f);
  else return *reinterpret_cast<const f32x2*>(x + 2 * ti + 32 * j);
}
template <int RPT>
__device__ __forceinline__ void store_pair(float* x, int ti, int j, f32x2 v) {
  if constexpr (RPT == 1) x[ti] = __uint_as_float(static_cast<uint32_t>(v));
  else *reinterpret_cast<f32x2*>(x + 2 * ti + 32 * j) = v;
}
// The j-th pair of a column of a (DK, DV) state matrix.
template <int RPT>
__device__ __forceinline__ f32x2 load_state(const float* m, int DV, int ti, int j) {
  if constexpr (RPT == 1) return pack2(m[(size_t)ti * DV], 0.f);
  const size_t i = 2 * ti + 32 * j;
  return pack2(m[i * DV], m[(i + 1) * DV]);
}
template <int RPT>
__device__ __forceinline__ void store_state(float* m, int DV, int ti, int j, f32x2 v) {
  float a, b;
  unpack2(v, a, b);
  if constexpr (RPT == 1) { m[(size_t)ti * DV] = a; return; }
  const size_t i = 2 * ti + 32 * j;
  m[i * DV] = a;
  m[(i + 1) * DV] = b;
}
__device__ __forceinline__ f32x2 shfl_xor16_add(f32x2 v) {      // sum with the other half warp's pair
  float a, b;
  unpack2(v, a, b);
  a += __shfl_xor_sync(0xffffffffu, a, 16);
  b += __shfl_xor_sync(0xffffffffu, b, 16);
  return pack2(a, b);
}

// Sum over the lanes that hold one token's DK consecutive elements (DK lanes for DK = 16, the whole warp otherwise).
template <int DK>
__device__ __forceinline__ float segment_sum(float x) {
  if (DK >= 32) x += __shfl_xor_sync(0xffffffffu, x, 16);
  return half_warp_sum(x);
}

// One block of TB tokens on its way from global to shared memory: asked for while the block before is computed, a 16-byte
// piece of k and of q per thread, and a piece of v (threads from 0), of dO (from 32) or of the fp32 rows de / r (from 64).
__device__ __forceinline__ uint4 load_piece(const bf16* p, int vec) {
  if (vec) return *reinterpret_cast<const uint4*>(p);
  uint4 u;
  bf16* e = reinterpret_cast<bf16*>(&u);
#pragma unroll
  for (int i = 0; i < 8; ++i) e[i] = p[i];
  return u;
}
__device__ __forceinline__ uint4 load_piece(const float* p, int vec) {
  if (vec) return *reinterpret_cast<const uint4*>(p);
  return make_uint4(__float_as_uint(p[0]), __float_as_uint(p[1]), __float_as_uint(p[2]), __float_as_uint(p[3]));
}
__device__ __forceinline__ void put_bf16(float* dst, const uint4& u, float scale) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
  float f[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = __bfloat1622float2(h[i]);
    f[2 * i] = v.x * scale;
    f[2 * i + 1] = v.y * scale;
  }
  reinterpret_cast<float4*>(dst)[0] = make_float4(f[0], f[1], f[2], f[3]);
  reinterpret_cast<float4*>(dst)[1] = make_float4(f[4], f[5], f[6], f[7]);
}
template <int DK, int NC, bool GRAD, bool REDO>
struct Incoming {
  uint4 k, q, x;
  float g, b;
  __device__ __forceinline__ void fetch(const GdnArgs& a, const float* rows, int tb, int nt, int hk, int hv, int col0) {
    const int tid = threadIdx.x;
    if (tid < DK && tid / (DK / 8) < nt) {
      const size_t off = ((size_t)(tb + tid / (DK / 8)) * a.HK + hk) * DK + tid % (DK / 8) * 8;
      k = load_piece(a.k + off, a.vec);
      q = load_piece(a.q + off, a.vec);
    }
    const int e = GRAD && tid >= 64 ? (tid - 64) * 4 : (tid & 31) * 8;      // element of the block's TB x NC columns
    const int t = e / NC, c = e % NC;
    if (t < nt) {
      const size_t off = ((size_t)(tb + t) * a.HV + hv) * a.DV + col0 + c;
      if (tid < 32) x = load_piece(a.v + off + (REDO ? (tb + t) * a.v_gap : 0), a.vec);
      else if (GRAD && tid < 64) x = load_piece(a.d_o + off, a.vec);
      else if (GRAD) x = load_piece(rows + off, a.vec);
    }
    if (tid < nt) {
      g = a.g[(size_t)(tb + tid) * a.HV + hv];
      b = a.beta[(size_t)(tb + tid) * a.HV + hv];
    }
  }
  __device__ __forceinline__ void put(float* k_s, float* q_s, float* v_s, float* x_s, float* y_s, float* a_s, float* b_s,
                                      float scale, int nt) {
    const int tid = threadIdx.x;
    if (tid < DK && tid / (DK / 8) < nt) {
      put_bf16(k_s + tid * 8, k, 1.f);
      put_bf16(q_s + tid * 8, q, scale);
    }
    const int e = GRAD && tid >= 64 ? (tid - 64) * 4 : (tid & 31) * 8;
    if (e / NC < nt) {
      if (tid < 32) put_bf16(v_s + e, x, 1.f);
      else if (GRAD && tid < 64) put_bf16(x_s + e, x, 1.f);
      else if (GRAD) *reinterpret_cast<uint4*>(y_s + e) = x;
    }
    if (tid < nt) {
      a_s[tid] = __expf(g);
      b_s[tid] = b;
    }
  }
};

// MODE 0: forward (o, r, final state).  MODE 1: pass F of the backward (dq, dk += S^ dr).
template <int RPT, int CPT, int MODE, bool REDO>
__global__ void __launch_bounds__(NT) gdn_forward_kernel(const GdnArgs a) {
  constexpr int DK = 16 * RPT, NC = 8 * CPT, NP = RPT == 1 ? 1 : RPT / 2;
  __shared__ __align__(16) float k_s[TB][DK], q_s[TB][DK];
  __shared__ __align__(16) float v_s[TB][NC], x_s[MODE == 1 ? TB : 1][NC], y_s[MODE == 1 ? TB : 1][NC];
  __shared__ float a_s[TB], b_s[TB];
  __shared__ __align__(16) float acc_q[MODE == 1 ? 4 : 1][TB][MODE == 1 ? DK : 1];
  __shared__ __align__(16) float acc_k[MODE == 1 ? 4 : 1][TB][MODE == 1 ? DK : 1];
  const int tid = threadIdx.x, ti = tid & 15, tj = tid >> 4, warp = tid >> 5;
  const int col0 = blockIdx.x * NC, hv = blockIdx.y, seq = blockIdx.z;
  if (REDO && a.only[seq * a.HV + hv] == 0) return;
  const int hk = hv / (a.HV / a.HK);
  const int t0 = a.cu[seq], t1 = a.cu[seq + 1];
  f32x2 S[NP][CPT];
#pragma unroll
  for (int j = 0; j < NP; ++j)
#pragma unroll
    for (int cc = 0; cc < CPT; ++cc)
      S[j][cc] = a.state_in ? load_state<RPT>(a.state_in + ((size_t)seq * a.HV + hv) * DK * a.DV + col0 + tj * CPT + cc,
                                              a.DV, ti, j) : 0ull;
  Incoming<DK, NC, MODE == 1, REDO> in;
  if (t0 < t1) in.fetch(a, a.de, t0, min(TB, t1 - t0), hk, hv, col0);
  for (int tb = t0; tb < t1; tb += TB) {
    const int nt = min(TB, t1 - tb);
    __syncthreads();
    in.put(&k_s[0][0], &q_s[0][0], &v_s[0][0], &x_s[0][0], &y_s[0][0], a_s, b_s, a.scale, nt);
    __syncthreads();
    if (tb + TB < t1) in.fetch(a, a.de, tb + TB, min(TB, t1 - tb - TB), hk, hv, col0);
    // Forward, four columns a thread: the output of a token is reduced over the rows together with the prediction of the next
    // one (two independent chains of shuffles in place of one after the other).
    [[maybe_unused]] float last[4] = {0.f, 0.f, 0.f, 0.f}, last_r = 0.f;
    [[maybe_unused]] auto store_out = [&](int t, float o, float r) {
      if ((ti & 3) == 0) {                         // lanes 0, 4, 8, 12 of the half warp hold columns 0..3
        const size_t off = ((size_t)(tb + t) * a.HV + hv) * a.DV + col0 + tj * CPT + (ti >> 2);
        a.o[off] = __float2bfloat16(o);
        if (a.r) a.r[off] = r;
      }
    };
    for (int t = 0; t < nt; ++t) {
      const float at = a_s[t], bt = b_s[t];
      const f32x2 at2 = pack2(at, at);
      f32x2 kr[NP], qr[NP];
      float rj[CPT];
#pragma unroll
      for (int j = 0; j < NP; ++j) { kr[j] = load_pair<RPT>(k_s[t], ti, j); qr[j] = load_pair<RPT>(q_s[t], ti, j); }
      {
        float pp[CPT];
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) {
          f32x2 p = 0ull;
#pragma unroll
          for (int j = 0; j < NP; ++j) { S[j][cc] = mul2(S[j][cc], at2); p = fma2(kr[j], S[j][cc], p); }
          pp[cc] = sum2(p);
        }
        if constexpr (CPT == 4) {
          const float mine = reduce_scatter4(pp[0], pp[1], pp[2], pp[3], tid & 31);
          if constexpr (MODE == 0) {
            const float o = reduce_scatter4(last[0], last[1], last[2], last[3], tid & 31);
            if (t > 0) store_out(t - 1, o, last_r);
            last_r = mine;
          }
          all_gather4(mine, tid & 31, rj);
        } else {
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc) rj[cc] = half_warp_sum(pp[cc]);
        }
      }
      if (MODE == 1) {   // dk += S^ dr  with dr = -beta de   (S holds S^ here)
        f32x2 dr[CPT];
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) { const float d = -bt * y_s[t][tj * CPT + cc]; dr[cc] = pack2(d, d); }
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          f32x2 p = 0ull;
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc) p = fma2(S[j][cc], dr[cc], p);
          p = shfl_xor16_add(p);
          if ((tid & 16) == 0) store_pair<RPT>(acc_k[warp][t], ti, j, p);
        }
      }
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) {
        const float e = bt * (v_s[t][tj * CPT + cc] - rj[cc]);
        const f32x2 e2 = pack2(e, e);
#pragma unroll
        for (int j = 0; j < NP; ++j) S[j][cc] = fma2(kr[j], e2, S[j][cc]);
      }
      if (MODE == 0) {
        float pp[CPT];
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) {
          f32x2 p = 0ull;
#pragma unroll
          for (int j = 0; j < NP; ++j) p = fma2(qr[j], S[j][cc], p);
          pp[cc] = sum2(p);
        }
        if constexpr (CPT == 4) {
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) last[cc] = pp[cc];
        } else {
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc) {
            const float p = half_warp_sum(pp[cc]);
            if (ti == 0) {
              const size_t off = ((size_t)(tb + t) * a.HV + hv) * a.DV + col0 + tj * CPT + cc;
              a.o[off] = __float2bfloat16(p);
              if (a.r) a.r[off] = rj[cc];
            }
          }
        }
      } else {            // dq = scale S_t dO
        f32x2 d_o[CPT];
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) { const float d = x_s[t][tj * CPT + cc]; d_o[cc] = pack2(d, d); }
        const f32x2 sc2 = pack2(a.scale, a.scale);
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          f32x2 p = 0ull;
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc) p = fma2(S[j][cc], d_o[cc], p);
          p = mul2(shfl_xor16_add(p), sc2);
          if ((tid & 16) == 0) store_pair<RPT>(acc_q[warp][t], ti, j, p);
        }
      }
    }
    if constexpr (MODE == 0 && CPT == 4)
      store_out(nt - 1, reduce_scatter4(last[0], last[1], last[2], last[3], tid & 31), last_r);
    if (MODE == 1) {
      __syncthreads();
      if (tid < TB) a_s[tid] = 0.f;           // reused as the per-token scalar accumulator of this block
      __syncthreads();
      for (int idx = tid; idx < TB * DK; idx += NT) {           // uniform trip count: the shuffles need full warps
        const int t = idx / DK, i = idx - t * DK;
        float sc = 0.f;
        if (t < nt) {
          const size_t off = ((size_t)(tb + t) * a.HV + hv) * DK + i;
          const float vq = acc_q[0][t][i] + acc_q[1][t][i] + acc_q[2][t][i] + acc_q[3][t][i];
          const float vk = acc_k[0][t][i] + acc_k[1][t][i] + acc_k[2][t][i] + acc_k[3][t][i];
          atomicAdd(a.dq + off, vq);
          atomicAdd(a.dk + off, vk);
          sc = q_s[t][i] * vq / a.scale + k_s[t][i] * vk;
        }
        sc = segment_sum<DK>(sc);
        if ((idx & (DK < 32 ? DK - 1 : 31)) == 0 && t < nt) atomicAdd(&a_s[t], sc);
      }
      __syncthreads();
      if (tid < nt) atomicAdd(a.sacc + (size_t)(tb + tid) * a.HV + hv, a_s[tid]);
    }
  }
  if (MODE == 0 && a.state_out) {
#pragma unroll
    for (int j = 0; j < NP; ++j)
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc)
        store_state<RPT>(a.state_out + ((size_t)seq * a.HV + hv) * DK * a.DV + col0 + tj * CPT + cc, a.DV, ti, j, S[j][cc]);
  }
}

// Pass R: reverse in time.  state_in = gradient of the final state (or null), state_out = gradient of the initial one.
template <int RPT, int CPT, bool REDO>
__global__ void __launch_bounds__(NT) gdn_reverse_kernel(const GdnArgs a) {
  constexpr int DK = 16 * RPT, NC = 8 * CPT, NP = RPT == 1 ? 1 : RPT / 2;
  __shared__ __align__(16) float k_s[TB][DK], q_s[TB][DK];
  __shared__ __align__(16) float v_s[TB][NC], x_s[TB][NC], r_s[TB][NC];
  __shared__ float a_s[TB], b_s[TB];
  __shared__ __align__(16) float acc_k[4][TB][DK];
  __shared__ float acc_b[4][TB];
  const int tid = threadIdx.x, ti = tid & 15, tj = tid >> 4, warp = tid >> 5;
  const int col0 = blockIdx.x * NC, hv = blockIdx.y, seq = blockIdx.z;
  if (REDO && a.only[seq * a.HV + hv] == 0) return;
  const int hk = hv / (a.HV / a.HK);
  const int t0 = a.cu[seq], t1 = a.cu[seq + 1];
  f32x2 dS[NP][CPT];
#pragma unroll
  for (int j = 0; j < NP; ++j)
#pragma unroll
    for (int cc = 0; cc < CPT; ++cc)
      dS[j][cc] = a.state_in ? load_state<RPT>(a.state_in + ((size_t)seq * a.HV + hv) * DK * a.DV + col0 + tj * CPT + cc,
                                               a.DV, ti, j) : 0ull;
  const int nblk = (t1 - t0 + TB - 1) / TB;
  Incoming<DK, NC, true, REDO> in;
  if (nblk > 0) in.fetch(a, a.r, t0 + (nblk - 1) * TB, t1 - t0 - (nblk - 1) * TB, hk, hv, col0);
  for (int blk = nblk - 1; blk >= 0; --blk) {
    const int tb = t0 + blk * TB;
    const int nt = min(TB, t1 - tb);
    __syncthreads();
    in.put(&k_s[0][0], &q_s[0][0], &v_s[0][0], &x_s[0][0], &r_s[0][0], a_s, b_s, a.scale, nt);
    __syncthreads();
    if (blk > 0) in.fetch(a, a.r, tb - TB, TB, hk, hv, col0);
    for (int t = nt - 1; t >= 0; --t) {
      const float at = a_s[t], bt = b_s[t];
      f32x2 kr[NP], qr[NP];
      float de[CPT], ej[CPT];
#pragma unroll
      for (int j = 0; j < NP; ++j) { kr[j] = load_pair<RPT>(k_s[t], ti, j); qr[j] = load_pair<RPT>(q_s[t], ti, j); }
      float db = 0.f;
      {
        float pp[CPT];
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) {
          const float dO = x_s[t][tj * CPT + cc];
          const f32x2 dO2 = pack2(dO, dO);
          f32x2 p = 0ull;
#pragma unroll
          for (int j = 0; j < NP; ++j) { dS[j][cc] = fma2(qr[j], dO2, dS[j][cc]); p = fma2(kr[j], dS[j][cc], p); }
          pp[cc] = sum2(p);
        }
        if constexpr (CPT == 4) {
          all_gather4(reduce_scatter4(pp[0], pp[1], pp[2], pp[3], tid & 31), tid & 31, de);
        } else {
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc) de[cc] = half_warp_sum(pp[cc]);
        }
      }
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) {
        const float diff = v_s[t][tj * CPT + cc] - r_s[t][tj * CPT + cc];
        ej[cc] = bt * diff;
        db += de[cc] * diff;
        if (ti == 0) {
          const size_t off = ((size_t)(tb + t) * a.HV + hv) * a.DV + col0 + tj * CPT + cc;
          a.de[off] = de[cc];
          a.dv[off + (REDO ? (tb + t) * a.dv_gap : 0)] = __float2bfloat16(bt * de[cc]);
        }
      }
      db += __shfl_xor_sync(0xffffffffu, db, 16);       // every lane of a half warp holds the same db
      if ((tid & 31) == 0) acc_b[warp][t] = db;
      f32x2 e2[CPT];
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) e2[cc] = pack2(ej[cc], ej[cc]);
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        f32x2 p = 0ull;
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) p = fma2(dS[j][cc], e2[cc], p);
        p = shfl_xor16_add(p);
        if ((tid & 16) == 0) store_pair<RPT>(acc_k[warp][t], ti, j, p);
      }
      const f32x2 at2 = pack2(at, at);
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) {
        const float dr = -bt * de[cc];
        const f32x2 dr2 = pack2(dr, dr);
#pragma unroll
        for (int j = 0; j < NP; ++j) dS[j][cc] = mul2(at2, fma2(kr[j], dr2, dS[j][cc]));
      }
    }
    __syncthreads();
    if (tid < TB) a_s[tid] = 0.f;             // reused as the per-token scalar accumulator of this block
    __syncthreads();
    for (int idx = tid; idx < TB * DK; idx += NT) {             // uniform trip count: the shuffles need full warps
      const int t = idx / DK, i = idx - t * DK;
      float sc = 0.f;
      if (t < nt) {
        const float vk = acc_k[0][t][i] + acc_k[1][t][i] + acc_k[2][t][i] + acc_k[3][t][i];
        atomicAdd(a.dk + ((size_t)(tb + t) * a.HV + hv) * DK + i, vk);
        sc = -k_s[t][i] * vk;
      }
      sc = segment_sum<DK>(sc);
      if ((idx & (DK < 32 ? DK - 1 : 31)) == 0 && t < nt) atomicAdd(&a_s[t], sc);
    }
    __syncthreads();
    if (tid < nt) {
      atomicAdd(a.dbeta + (size_t)(tb + tid) * a.HV + hv, acc_b[0][tid] + acc_b[1][tid] + acc_b[2][tid] + acc_b[3][tid]);
      atomicAdd(a.sacc + (size_t)(tb + tid) * a.HV + hv, a_s[tid]);
    }
  }
  if (a.state_out) {
#pragma unroll
    for (int j = 0; j < NP; ++j)
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc)
        store_state<RPT>(a.state_out + ((size_t)seq * a.HV + hv) * DK * a.DV + col0 + tj * CPT + cc, a.DV, ti, j, dS[j][cc]);
  }
}

// dg[t, h] = sum_{u >= t, same sequence} s[u, h] + extra[seq, h].  A block owns 32 heads of one sequence; its 32 warps take
// 32 runs of tokens: totals of the runs, their suffix sums in shared memory, then the running sums within each run.  (A
// cumulative sum over all tokens along the slow axis, as the tensor library does it, kept one thread per head busy: 3.5 ms for
// 16384 x 32, below 0.02 ms so.)  T >= 0: the sequences have to cover the T tokens; if they do not, the error word says so.
__global__ void __launch_bounds__(1024) suffix_sum_kernel(const float* __restrict__ s, const float* __restrict__ extra,
                                                          const int* __restrict__ cu, int T, float* __restrict__ dg, int H) {
  __shared__ float tot[32][33];
  if (T >= 0 && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && (cu[0] != 0 || cu[gridDim.y] != T)) set_error(3, 300);
  const int lane = threadIdx.x & 31, run = threadIdx.x >> 5;
  const int h = blockIdx.x * 32 + lane, seq = blockIdx.y;
  const int t0 = cu[seq], n = cu[seq + 1] - t0;
  const int per = (n + 31) / 32;
  const int lo = min(run * per, n), hi = min(lo + per, n);
  const bool on = h < H;
  const float* sp = s + (size_t)t0 * H + h;
  float sum = 0.f;
  if (on) {
#pragma unroll 8
    for (int t = lo; t < hi; ++t) sum += sp[(size_t)t * H];
  }
  tot[run][lane] = sum;
  __syncthreads();
  if (!on) return;
  float acc = extra ? extra[(size_t)seq * H + h] : 0.f;
  for (int r = 31; r > run; --r) acc += tot[r][lane];
  float* dp = dg + (size_t)t0 * H + h;
#pragma unroll 8
  for (int t = hi - 1; t >= lo; --t) {
    acc += sp[(size_t)t * H];
    dp[(size_t)t * H] = acc;
  }
}

// Zeros where the two backward passes add up, for the pairs marked in `only`.
__global__ void __launch_bounds__(NT) gdn_clear_kernel(const GdnArgs a, int DK) {
  const int hv = blockIdx.x, seq = blockIdx.y;
  if (a.only[seq * a.HV + hv] == 0) return;
  const int t0 = a.cu[seq], t1 = a.cu[seq + 1];
  for (int t = t0; t < t1; ++t) {
    const size_t th = (size_t)t * a.HV + hv;
    for (int i = threadIdx.x; i < DK; i += NT) a.dq[th * DK + i] = a.dk[th * DK + i] = 0.f;
    if (threadIdx.x == 0) a.dbeta[th] = a.sacc[th] = 0.f;
  }
}

template <int RPT, int CPT, bool REDO>
int launch_all(int pass, const GdnArgs& a, int nseq, cudaStream_t s) {
  dim3 grid(a.DV / (8 * CPT), a.HV, nseq);
  if (pass == 0) gdn_forward_kernel<RPT, CPT, 0, REDO><<<grid, NT, 0, s>>>(a);
  else if (pass == 1) gdn_reverse_kernel<RPT, CPT, REDO><<<grid, NT, 0, s>>>(a);
  else gdn_forward_kernel<RPT, CPT, 1, REDO><<<grid, NT, 0, s>>>(a);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -400 - (int)e;
}

// Column block per CTA: 32 columns when that already gives two CTAs per SM, otherwise 16 or 8 so that one long
// sequence still spreads over the whole GPU (the recurrence is latency-bound per CTA).
int cols_per_thread(int nseq, int HV, int DV) {
  const long heads = (long)nseq * HV;
  if (DV % 32 == 0 && heads * (DV / 32) >= 296) return 4;
  if (DV % 16 == 0 && heads * (DV / 16) >= 296) return 2;
  if (DV % 8 == 0) return 1;
  return 0;
}

template <int RPT, bool REDO = false>
int launch_cols(int pass, const GdnArgs& a, int nseq, cudaStream_t s) {
  switch (cols_per_thread(nseq, a.HV, a.DV)) {
    case 4: return launch_all<RPT, 4, REDO>(pass, a, nseq, s);
    case 2: return launch_all<RPT, 2, REDO>(pass, a, nseq, s);
    case 1: return launch_all<RPT, 1, REDO>(pass, a, nseq, s);
    default: return -2;
  }
}

}  // namespace

extern "C" {

// pass: 0 forward, 1 backward reverse pass, 2 backward forward-direction pass.  DK in {16, 32, 64, 128}, DV % 8 == 0.
// Number of column blocks (CTAs per head) the kernels will use: the leading dimension of the dq / dk partial buffers.
int ftb_gdn_col_blocks(int nseq, int HV, int DV) {
  const int cpt = cols_per_thread(nseq, HV, DV);
  return cpt ? DV / (8 * cpt) : 0;
}

// dg (T, H) from the per-token scalars s (T, H); extra (nseq, H) or NULL is added to every token of its sequence.  T: tokens
// that the sequences have to cover, or -1.
int ftb_gate_sum(const float* s, const float* extra, const int* cu, int nseq, int T, float* dg, int H, cudaStream_t st) {
  if (nseq <= 0 || H <= 0) return T > 0 ? -2 : 0;
  if (nseq > 65535) return -2;
  suffix_sum_kernel<<<dim3((H + 31) / 32, nseq), 1024, 0, st>>>(s, extra, cu, T, dg, H);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -400 - (int)e;
}
int ftb_suffix_sum(const float* s, const float* extra, const int* cu, int nseq, float* dg, int H, cudaStream_t st) {
  return ftb_gate_sum(s, extra, cu, nseq, -1, dg, H, st);
}

int ftb_gdn_error(void) {
  int h[2] = {0, 0};
  cudaMemcpyFromSymbol(&h[0], g_error_word, sizeof(int));
  cudaMemcpyFromSymbol(&h[1], g_error_where, sizeof(int));
  if (h[0] != 0) {
    int z = 0;
    cudaMemcpyToSymbol(g_error_word, &z, sizeof(int));
    cudaMemcpyToSymbol(g_error_where, &z, sizeof(int));
  }
  return h[0] * 1000 + h[1];
}

int ftb_gdn(int pass, const void* q, const void* k, const void* v, const float* g, const float* beta, const int* cu,
            int nseq, const float* state_in, float* state_out, void* o, float* r, const void* d_o, float* de, void* dv,
            float* dbeta, float* dq, float* dk, float* sacc, int HK, int HV, int DK, int DV, float scale,
            cudaStream_t s) {
  if (nseq <= 0) return 0;
  if (HV % HK) return -2;
  GdnArgs a = {};
  a.q = (const bf16*)q; a.k = (const bf16*)k; a.v = (const bf16*)v; a.g = g; a.beta = beta; a.cu = cu;
  a.state_in = state_in; a.state_out = state_out; a.o = (bf16*)o; a.r = r; a.d_o = (const bf16*)d_o; a.de = de;
  a.dv = (bf16*)dv; a.dbeta = dbeta; a.dq = dq; a.dk = dk; a.sacc = sacc; a.HK = HK; a.HV = HV; a.DV = DV; a.scale = scale;
  a.vec = (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)d_o | (uintptr_t)de | (uintptr_t)r) & 15) == 0;
  switch (DK) {
    case 16: return launch_cols<1>(pass, a, nseq, s);
    case 32: return launch_cols<2>(pass, a, nseq, s);
    case 64: return launch_cols<4>(pass, a, nseq, s);
    case 128: return launch_cols<8>(pass, a, nseq, s);
    default: return -2;
  }
}

// What the chunk kernels (gdn_chunk.cu, heads of 128 x 128) marked in `only` (nseq, HV), because infinities or NaN came up in it,
// done again token by token, in place of what they wrote; v and dv with the token strides they may have there.  Blocks of
// pairs that are not marked return at once: 2 to 3 us a launch.
int ftb_gdn_redo_fwd(const int* only, const void* q, const void* k, const void* v, long v_ts, const float* g, const float* beta,
                     const int* cu, int nseq, const float* state_in, float* state_out, void* o, float* r, int HK, int HV, float scale,
                     cudaStream_t s) {
  if (nseq <= 0) return 0;
  GdnArgs a = {};
  a.q = (const bf16*)q; a.k = (const bf16*)k; a.v = (const bf16*)v; a.g = g; a.beta = beta; a.cu = cu; a.state_in = state_in;
  a.state_out = state_out; a.o = (bf16*)o; a.r = r; a.HK = HK; a.HV = HV; a.DV = 128; a.scale = scale;
  a.vec = 1; a.v_gap = v_ts - (long)HV * 128; a.only = only;
  return launch_cols<8, true>(0, a, nseq, s);
}
int ftb_gdn_redo_bwd(const int* only, const void* q, const void* k, const void* v, long v_ts, const float* g, const float* beta,
                     const int* cu, int nseq, const float* state_in, const float* dstate_in, float* dstate_out, const float* r,
                     const void* d_o, float* de, void* dv, long dv_ts, float* dbeta, float* dq, float* dk, float* sacc, int HK, int HV,
                     float scale, cudaStream_t s) {
  if (nseq <= 0) return 0;
  GdnArgs a = {};
  a.q = (const bf16*)q; a.k = (const bf16*)k; a.v = (const bf16*)v; a.g = g; a.beta = beta; a.cu = cu; a.state_in = dstate_in;
  a.state_out = dstate_out; a.r = const_cast<float*>(r); a.d_o = (const bf16*)d_o; a.de = de; a.dv = (bf16*)dv; a.dbeta = dbeta;
  a.dq = dq; a.dk = dk; a.sacc = sacc; a.HK = HK; a.HV = HV; a.DV = 128; a.scale = scale;
  a.vec = 1; a.v_gap = v_ts - (long)HV * 128; a.dv_gap = dv_ts - (long)HV * 128; a.only = only;
  gdn_clear_kernel<<<dim3(HV, nseq), NT, 0, s>>>(a, 128);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return -400 - (int)e;
  const int rc = launch_cols<8, true>(1, a, nseq, s);
  if (rc) return rc;
  a.state_in = state_in;
  a.state_out = nullptr;
  return launch_cols<8, true>(2, a, nseq, s);
}

}  // extern "C"
