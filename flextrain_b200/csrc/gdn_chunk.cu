// Gated DeltaNet in chunks of 64 tokens on the tensor cores (head size 128 x 128), forward and backward.
//
// The recurrence of gdn.cu, S_i = exp(g_i) S_{i-1} + k_i e_i^T with e_i = beta_i y_i, y_i = v_i - S^_i^T k_i, is solved for a
// chunk at once.  With G the running sum of g inside the chunk, D_ij = exp(G_i - G_j), S the state before the chunk:
//     (I + L B) Y = V - diag(exp G) K S,       L = strictly lower part of D o (K K^T),  B = diag(beta)
//     O = scale diag(exp G) Q S + P B Y,        P = lower part of scale D o (Q K^T)
//     S <- exp(G_C) S + (diag(exp(G_C - G)) K)^T B Y
// and backward, X the gradient of the state after the chunk (notation of gdn.cu: dr = -beta de, dv = -dr):
//     rhs = diag(exp(G_C - G)) K X + P^T dO;   (I + B L^T) dR = -B rhs
//     X <- exp(G_C) X + Q^T diag(scale exp G) dO + K^T diag(exp G) dR
//     dQ = scale diag(exp G) dO S^T + W1 K,    W1 = scale D o (dO Y^T) B
//     dK = diag(exp G) dR S^T + W2 K + diag(exp(G_C - G)) (B Y) X^T + W1^T Q + W2^T K,     W2 = strictly lower D o (dR Y^T) B
//     dbeta_i = rhs_i . y_i + sum_{j > i} L_ji (dr_j . y_i)
// The reference calls FLA's chunked Triton kernels here (flextrain/nn/blocks/linear_attn.py:1090-1145, 1702-1722).
//
// Precision.  q, k, v, dO are bf16 and enter the products as they are.  Everything the recurrence keeps in fp32 (state,
// inverse, Y, dR, decayed products) enters as the sum of three bf16 terms, cut so that the sum is the fp32 number itself; of
// the nine products of two such operands the six largest are formed, which leaves out 2^-24 of the result.  Sums are fp32
// throughout, G is summed in fp64 (differences of it are taken), the inverse is a forward substitution in fp32.  The tensor
// cores cut off what they add to an accumulator below its last bit, so a product over 16 has an accumulator of its own, which
// starts at zero and takes the smaller terms first, and is added to the sum in fp32, rounded to nearest.
//
// Why mma.sync and not tcgen05: the chain of a sequence is state -> prediction -> solve -> state.  A warp owns 16 of the 128
// value columns, which never meet those of another warp, and holds its slice of the state transposed as the accumulators of
// m16n8k16; these are, register for register, the A operand of the next product, so the whole chain stays in one warp's
// registers: no round trip through shared or tensor memory and no barrier between its products.  Shared memory holds only
// what the warps share (K, Q, the inverse).  The backward products that sum over value columns (dQ, dK) are the exception: there
// the state goes through shared memory once a chunk, and a warp owns tokens.
//
// Measured, ms, token by token (gdn.cu) / so, 32 heads: 16 x 1024 tokens forward 2.19 / 1.05, backward 7.98 / 4.22; one sequence
// of 16384 7.5 / 3.3 and 25.4 / 15.0; two of 8192 4.6 / 1.8 and 15.1 / 7.8; 512 tokens 0.22 / 0.13 and 0.81 / 0.51; 300 sequences of
// 33, mostly half-empty chunks, 1.60 / 1.29 and 5.16 / 5.33.  What bounds it now: the chain of a sequence, product after
// product; mma.sync (537 TFLOP/s) is in use for about half of the time.
//
// Errors against fp64 in 1e-8 (2-norm, four sequences of 512, mean of three seeds, token by token / so):
//                                final state   dq          dk          dbeta       dg
//   decay 0.25 a token           4.4 / 6.6     11.2 / 10.7 15.1 / 10.8 12.5 / 13.6 1003 / 400
//   gates as a model starts      37.7 / 9.6    44 / 14.9   49 / 16.9   45 / 16.0   156 / 118
//   decay 0.99 a token           336 / 10.9    305 / 16.3  349 / 20.2  321 / 18.7  513 / 75
//   keys that resemble each      36.5 / 15.7   42.5 / 19.1 49 / 19.3   45.5 / 28.1 154 / 153
//     other (cosine 0.5)
// Larger in two places, by a unit in the last place of fp32, where a state forgets three quarters of itself at each token.  (K K^T and
// Q K^T in one accumulator over all of 128, and the exponentials in fp32: a quarter more in dbeta.  The largest terms of every product
// in an accumulator of their own: those two figures 6.6 and 13.0, the others a tenth less, for 1.29 and 4.80 ms in place of 1.10 and 4.23.)
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace {

typedef __nv_bfloat16 bf16;
constexpr int C = 64, DK = 128, DV = 128, NT = 256;
constexpr int kBlk = 10;                         // 16 x 16 blocks on and below the diagonal of a chunk's 64 x 64 matrices
constexpr int kTri = kBlk * 256;                 // their elements

struct Args {
  const bf16* q;           // (T, HK, 128)
  const bf16* k;
  const bf16* v;           // (T, HV, 128), tokens v_ts elements apart
  const float* g;          // (T, HV)
  const float* beta;       // (T, HV)
  const int* cu;           // (nseq + 1)
  const float* state_in;   // (nseq, HV, 128, 128) or null: initial state (forward, pass F), gradient of the final one (pass R)
  float* state_out;        // or null: final state (forward), gradient of the initial one (pass R)
  bf16* o;                 // (T, HV, 128)
  float* r;                // (T, HV, 128)  v - y: forward writes (or null), backward reads
  const bf16* d_o;         // (T, HV, 128)
  float* dr;               // (T, HV, 128)  pass R writes, pass F reads
  bf16* dv;                // (T, HV, 128)  pass R, tokens dv_ts elements apart
  float* dbeta;            // (T, HV)       pass R writes rhs . y, pass F adds the rest
  float* dq;               // (T, HV, 128)  pass F
  float* dk;               // (T, HV, 128)  pass R writes the part of X, pass F adds the rest
  float* sacc;             // (T, HV)       q.dq - k.(dS' e) + k.(S^ dr), as in gdn.cu: pass R writes, pass F adds
  float* tri_t;            // (slots, HV, 10, 16, 16)  (I + L B)^-1 - I  (the identity is added in fp32)
  float* tri_p;            // (slots, HV, 10, 16, 16)  P
  double* gsum;            // (slots, HV, 64)          G in powers of two
  int* order;              // (nseq)  sequences, longest first
  int* redo;               // (nseq, HV)  1: infinities or NaN came up, the results do not count
  int HK, HV, nseq;
  long T, v_ts, dv_ts;
  float scale;
};

// A sequence's first chunk has this slot; the chunks of s take at most cu[s+1] / 64 - cu[s] / 64 + 1 slots.
__device__ __forceinline__ int first_slot(const int* cu, int s) { return cu[s] / C + s; }

__device__ __forceinline__ int blk_of(int ib, int jb) { return ib * (ib + 1) / 2 + jb; }

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// The next chunk's rows (64 of 128 elements of `es` bytes) on their way to L2.
__device__ __forceinline__ void prefetch_rows(const char* src, long row_bytes, int es, int n, int tid) {
  const int lines = es;                          // 128-byte lines in a row of 128 elements
  for (int i = tid; i < C * lines; i += NT) {
    const int r = i / lines;
    if (r < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(src + r * row_bytes + (i - r * lines) * 128));
  }
}
__device__ __forceinline__ void red_add2(float* p, float x, float y) {
  asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void ldsm(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm_t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void stsm_t(uint32_t a, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(r0), "r"(r1), "r"(r2), "r"(r3)
               : "memory");
}
__device__ __forceinline__ uint32_t transpose8(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma_zero(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// Two fp32 numbers as three packed pairs of bf16 whose sum they are (each term is the upper half of what the ones before leave).
__device__ __forceinline__ void split3(float x, float y, uint32_t& t0, uint32_t& t1, uint32_t& t2) {
  const uint32_t xu = __float_as_uint(x), yu = __float_as_uint(y);
  t0 = __byte_perm(xu, yu, 0x7632);
  const float x1 = x - __uint_as_float(xu & 0xffff0000u), y1 = y - __uint_as_float(yu & 0xffff0000u);
  const uint32_t x1u = __float_as_uint(x1), y1u = __float_as_uint(y1);
  t1 = __byte_perm(x1u, y1u, 0x7632);
  const float x2 = x1 - __uint_as_float(x1u & 0xffff0000u), y2 = y1 - __uint_as_float(y1u & 0xffff0000u);
  t2 = __byte_perm(__float_as_uint(x2), __float_as_uint(y2), 0x7632);
}
// The A operand (16 x 16) made of two neighbouring accumulator tiles, as three terms.
__device__ __forceinline__ void split_a(const float (&lo)[4], const float (&hi)[4], uint32_t (&a)[3][4]) {
  split3(lo[0], lo[1], a[0][0], a[1][0], a[2][0]);
  split3(lo[2], lo[3], a[0][1], a[1][1], a[2][1]);
  split3(hi[0], hi[1], a[0][2], a[1][2], a[2][2]);
  split3(hi[2], hi[3], a[0][3], a[1][3], a[2][3]);
}
__device__ __forceinline__ void add4(float (&c)[4], const float (&d)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) c[e] += d[e];
}
// c += a b, the smaller products first: a in three terms, b as it is
__device__ __forceinline__ void prod3(float (&c)[4], const uint32_t (&a)[3][4], uint32_t b0, uint32_t b1) {
  float d[4];
  mma_zero(d, a[2], b0, b1);
  mma(d, a[1], b0, b1);
  mma(d, a[0], b0, b1);
  add4(c, d);
}
// both as they are
__device__ __forceinline__ void prod1(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float d[4];
  mma_zero(d, a, b0, b1);
  add4(c, d);
}
// a as it is, b in three terms
__device__ __forceinline__ void prod3(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[3][2]) {
  float d[4];
  mma_zero(d, a, b[2][0], b[2][1]);
  mma(d, a, b[1][0], b[1][1]);
  mma(d, a, b[0][0], b[0][1]);
  add4(c, d);
}
// both in three terms
__device__ __forceinline__ void prod6(float (&c)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2]) {
  float d[4];
  mma_zero(d, a[2], b[0][0], b[0][1]);
  mma(d, a[0], b[2][0], b[2][1]);
  mma(d, a[1], b[1][0], b[1][1]);
  mma(d, a[1], b[0][0], b[0][1]);
  mma(d, a[0], b[1][0], b[1][1]);
  mma(d, a[0], b[0][0], b[0][1]);
  add4(c, d);
}
// the fragments of two neighbouring tiles in three planes: those of tile e
__device__ __forceinline__ void pick(uint32_t (&b)[3][2], const uint32_t (&planes)[3][4], int e) {
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    b[p][0] = planes[p][2 * e];
    b[p][1] = planes[p][2 * e + 1];
  }
}
__device__ __forceinline__ float2 bf2(uint32_t u) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
__device__ __forceinline__ uint32_t pack_bf(float x, float y) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// 2^x for a difference of sums, rounded once: the whole part goes into the exponent, 2^f, |f| <= 1/2, is its series in fp64 (the term
// of f^9 is below 2e-10).  The hardware's approximation is off by 2^-22, and rounding x to fp32 first would cost another |x| 2^-25.
__device__ __forceinline__ float exp2_of(double x) {
  if (x < -126.0) return 0.f;
  if (x > 127.0) return x > 128.0 ? __int_as_float(0x7f800000) : exp2f((float)x);
  const double n = rint(x), f = (x - n) * 0.69314718055994531;
  double p = 1.0 / 40320;                          // 1 / k!, k = 8 .. 0
  p = p * f + 1.0 / 5040;
  p = p * f + 1.0 / 720;
  p = p * f + 1.0 / 120;
  p = p * f + 1.0 / 24;
  p = p * f + 1.0 / 6;
  p = p * f + 0.5;
  p = p * f + 1.0;
  p = p * f + 1.0;
  return (float)p * __int_as_float(((int)n + 127) << 23);
}

// ---- shared-memory tiles.  (64, 128) bf16 with 256-byte rows: the 16-byte piece c of row r lies at piece c ^ (r & 7).
__device__ __forceinline__ uint32_t tile_at(int r, int c) { return r * 256 + (((c & 8) | ((c ^ r) & 7)) << 4); }
// 16 x 16 bf16 blocks with 32-byte rows: piece c (0, 1) of row r at c ^ (r / 4 & 1).
__device__ __forceinline__ uint32_t blk_at(int r, int c) { return r * 32 + ((c ^ ((r >> 2) & 1)) << 4); }

// Lane addresses of the four 8 x 8 matrices of an ldmatrix.x4.  `rows` x `cols` blocks in the order (0,0) (0,1) (1,0) (1,1):
__device__ __forceinline__ uint32_t tile_rc(int r0, int c0, int lane) {
  return tile_at(r0 + (lane & 7) + ((lane >> 4) << 3), c0 + ((lane >> 3) & 1));
}
// ... and (0,0) (1,0) (0,1) (1,1).
__device__ __forceinline__ uint32_t tile_cr(int r0, int c0, int lane) { return tile_at(r0 + (lane & 15), c0 + (lane >> 4)); }
__device__ __forceinline__ uint32_t blk_rc(int lane) { return blk_at((lane & 7) + ((lane >> 4) << 3), (lane >> 3) & 1); }
__device__ __forceinline__ uint32_t blk_cr(int lane) { return blk_at(lane & 15, lane >> 4); }

// One (64, 128) bf16 tile on its way to shared memory; rows from n on are zeros.
__device__ __forceinline__ void load_tile(uint32_t dst, const bf16* src, long row_stride, int n, int tid, int nthreads) {
  for (int i = tid; i < C * 16; i += nthreads) {
    const int r = i >> 4, c = i & 15;
    cp16(dst + tile_at(r, c), src + (r < n ? r * row_stride : 0) + c * 8, r < n);
  }
}

// fp32 blocks of a chunk's triangular matrix as three planes of bf16 blocks.
__device__ __forceinline__ void split_tri(char* planes, const float* src, int tid) {
  for (int f = tid; f < kTri / 4; f += NT) {
    const float4 x = reinterpret_cast<const float4*>(src)[f];
    const int b = f >> 6, r = (f >> 2) & 15, c = (f & 3) * 4;
    uint32_t t[3][2];
    split3(x.x, x.y, t[0][0], t[1][0], t[2][0]);
    split3(x.z, x.w, t[0][1], t[1][1], t[2][1]);
#pragma unroll
    for (int p = 0; p < 3; ++p)
      *reinterpret_cast<uint2*>(planes + p * kTri * 2 + b * 512 + blk_at(r, c >> 3) + (c & 7) * 2) = make_uint2(t[p][0], t[p][1]);
  }
}

// ================================================================================================ preparation
// Per chunk and key head: K K^T and Q K^T (lower 16 x 16 blocks: warp w has row w), then for each value head of that key head
// G, P and the inverse of I + L B by forward substitution, a thread per column.  Two value heads at a time.  Blocks on the
// first slots also put the sequences in order, the first and last clear what belongs to no sequence.
constexpr int kLd = 68;                                           // floats in a row of L B
constexpr int kPrepSmem = 2 * C * 256 + 2 * C * kLd * 4 + 2 * C * 8 + 2 * C * 4;

__global__ void __launch_bounds__(128, 3) gdn_prep_kernel(const Args a) {
  extern __shared__ __align__(128) char sm[];
  char* k_s = sm;
  char* q_s = sm + C * 256;
  float* lb = reinterpret_cast<float*>(sm + 2 * C * 256);          // [2][64][kLd]
  double* gs = reinterpret_cast<double*>(lb + 2 * C * kLd);        // [2][64]
  float* bs = reinterpret_cast<float*>(gs + 2 * C);                // [2][64]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int slot = blockIdx.x, hk = blockIdx.y;
  if (hk == 0 && slot * 128 < a.nseq) {          // rank of each sequence by length, ties by position (long lists: as they are)
    const int s = slot * 128 + tid;
    if (s < a.nseq) {
      int rank = s;
      if (a.nseq <= 1024) {
        const int n = a.cu[s + 1] - a.cu[s];
        rank = 0;
        for (int u = 0; u < a.nseq; ++u) {
          const int m = a.cu[u + 1] - a.cu[u];
          rank += m > n || (m == n && u < s);
        }
      }
      a.order[rank] = s;
    }
  }
  for (int side = 0; side < 2; ++side) {         // tokens before the first sequence and after the last
    if (!a.dq || slot != (side ? (int)gridDim.x - 1 : 0)) continue;
    const long lo = side ? a.cu[a.nseq] : 0, hi = side ? a.T : a.cu[0];
    const int rep = a.HV / a.HK;
    for (long t = lo; t < hi; ++t)
      for (int i = tid; i < rep * DK; i += 128) {
        const long at = (t * a.HV + hk * rep) * DK + i;
        a.dq[at] = a.dk[at] = 0.f;
        if (i < rep) a.dbeta[t * a.HV + hk * rep + i] = a.sacc[t * a.HV + hk * rep + i] = 0.f;
      }
  }
  int lo = 0, hi = a.nseq - 1;                                     // last sequence whose first slot is not after this one
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (first_slot(a.cu, mid) <= slot) lo = mid; else hi = mid - 1;
  }
  const int t0 = a.cu[lo] + (slot - first_slot(a.cu, lo)) * C, n = min(C, a.cu[lo + 1] - t0);
  if (n <= 0 || slot < first_slot(a.cu, 0)) return;
  load_tile(smem_addr(k_s), a.k + ((long)t0 * a.HK + hk) * DK, (long)a.HK * DK, n, tid, 128);
  load_tile(smem_addr(q_s), a.q + ((long)t0 * a.HK + hk) * DK, (long)a.HK * DK, n, tid, 128);
  cp_commit();
  cp_wait_all();
  __syncthreads();
  float kk[8][4] = {}, qk[8][4] = {};
#pragma unroll
  for (int kb = 0; kb < 8; ++kb) {
    uint32_t ka[4], qa[4], b[4];
    ldsm(ka, smem_addr(k_s) + tile_cr(warp * 16, kb * 2, lane));
    ldsm(qa, smem_addr(q_s) + tile_cr(warp * 16, kb * 2, lane));
#pragma unroll
    for (int jb = 0; jb < 4; ++jb)
      if (jb <= warp) {
        ldsm(b, smem_addr(k_s) + tile_rc(jb * 16, kb * 2, lane));
        prod1(kk[2 * jb], ka, b[0], b[1]);
        prod1(kk[2 * jb + 1], ka, b[2], b[3]);
        prod1(qk[2 * jb], qa, b[0], b[1]);
        prod1(qk[2 * jb + 1], qa, b[2], b[3]);
      }
  }
  const int rep = a.HV / a.HK;
  for (int h0 = 0; h0 < rep; h0 += 2) {
    const int nh = min(2, rep - h0);
    __syncthreads();
    if (tid < nh * C) {
      const int h = tid >> 6, i = tid & 63, hv = hk * rep + h0 + h;
      float g = 0.f, b = 0.f;
      if (i < n) {
        g = a.g[(long)(t0 + i) * a.HV + hv];
        b = a.beta[(long)(t0 + i) * a.HV + hv];
        if (g < -2000.f) g = -2000.f;              // exp of it is 0 all the same, and sums of it stay finite and exact enough
      }
      gs[tid] = (double)g * 1.4426950408889634;
      bs[tid] = b;
    }
    __syncthreads();
    if (warp < nh) {                               // running sums: two neighbours a lane, then over the lanes
      double x = gs[warp * C + 2 * lane], y = gs[warp * C + 2 * lane + 1], s = x + y;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, s, d);
        if (lane >= d) s += u;
      }
      __syncwarp();
      gs[warp * C + 2 * lane] = s - y;
      gs[warp * C + 2 * lane + 1] = s;
      double* out = a.gsum + ((long)slot * a.HV + hk * rep + h0 + warp) * C;
      out[2 * lane] = s - y;
      out[2 * lane + 1] = s;
    }
    __syncthreads();
    for (int h = 0; h < nh; ++h) {
      const long at = ((long)slot * a.HV + hk * rep + h0 + h) * kTri;
#pragma unroll
      for (int nb = 0; nb < 8; ++nb)
        if (nb < 2 * warp + 2)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = warp * 16 + (lane >> 2) + (e >> 1) * 8, j = nb * 8 + (lane & 3) * 2 + (e & 1);
            const float d = i >= j ? exp2_of(gs[h * C + i] - gs[h * C + j]) : 0.f;
            lb[(h * C + i) * kLd + j] = i > j ? d * kk[nb][e] * bs[h * C + j] : 0.f;
            a.tri_p[at + blk_of(warp, nb >> 1) * 256 + (i & 15) * 16 + (j & 15)] = i >= j ? a.scale * d * qk[nb][e] : 0.f;
          }
    }
    __syncthreads();
    if (tid < nh * C) {
      const int h = tid >> 6, j = tid & 63;
      const float* m = lb + h * C * kLd;
      float y[C];
#pragma unroll
      for (int i = 0; i < C; ++i) {
        float s[4] = {i == j ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < i; c += 4) {
          const float4 x = *reinterpret_cast<const float4*>(m + i * kLd + c);
          s[0] -= x.x * y[c];
          if (c + 1 < i) s[1] -= x.y * y[c + 1];
          if (c + 2 < i) s[2] -= x.z * y[c + 2];
          if (c + 3 < i) s[3] -= x.w * y[c + 3];
        }
        y[i] = (s[0] + s[1]) + (s[2] + s[3]);
      }
      float* out = a.tri_t + ((long)slot * a.HV + hk * rep + h0 + h) * kTri;
#pragma unroll
      for (int i = 0; i < C; ++i)
        if ((j >> 4) <= (i >> 4)) out[blk_of(i >> 4, j >> 4) * 256 + (i & 15) * 16 + (j & 15)] = i == j ? 0.f : y[i];
    }
  }
}

// ================================================================================================ chain kernels: common parts
// A stage holds a chunk's tiles and triangular blocks; two of them, the next chunk's loads run under the current chunk.
constexpr int kTile = C * 256;
struct alignas(16) Gates {     // of the chunk at work
  float gam[C];                // exp(G_i)
  float dec[C];                // exp(G_C - G_i)
  float bet[C];
  float end;                   // exp(G_C)
  int bad;                     // 1: something was not finite so far
};

__device__ __forceinline__ void make_gates(Gates* s, const Args& a, long slot, int t0, int n, int hv, int tid) {
  if (tid < C) {
    const double* gs = a.gsum + (slot * a.HV + hv) * C;
    const double gi = gs[tid], gc = gs[C - 1];
    s->gam[tid] = exp2_of(gi);
    s->dec[tid] = exp2_of(gc - gi);
    s->bet[tid] = tid < n ? a.beta[(long)(t0 + tid) * a.HV + hv] : 0.f;
    if (tid == 0) s->end = exp2_of(gc);
  }
}

// The warp's 16 value columns of a (128, 128) state, transposed: st[nb] has rows = value columns, columns = key rows 8 nb ...
__device__ __forceinline__ void load_state(float (&st)[16][4], const float* m, int col, int lane) {
#pragma unroll
  for (int nb = 0; nb < 16; ++nb)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      st[nb][e] = m ? m[(size_t)(nb * 8 + (lane & 3) * 2 + (e & 1)) * DV + col + (lane >> 2) + (e >> 1) * 8] : 0.f;
}
__device__ __forceinline__ void store_state(float* m, const float (&st)[16][4], int col, int lane) {
#pragma unroll
  for (int nb = 0; nb < 16; ++nb)
#pragma unroll
    for (int e = 0; e < 4; ++e) m[(size_t)(nb * 8 + (lane & 3) * 2 + (e & 1)) * DV + col + (lane >> 2) + (e >> 1) * 8] = st[nb][e];
}

// acc (16 value columns x 64 tokens) += state^T X^T for a tile X (64, 128) in shared memory, key rows 16 kb ..., `s` their terms.
__device__ __forceinline__ void state_times_tile(float (&acc)[8][4], const uint32_t (&s)[3][4], uint32_t tile, int kb, int lane) {
#pragma unroll
  for (int np = 0; np < 4; ++np) {
    uint32_t b[4];
    ldsm(b, tile + tile_rc(np * 16, kb * 2, lane));
    prod3(acc[2 * np], s, b[0], b[1]);
    prod3(acc[2 * np + 1], s, b[2], b[3]);
  }
}
// state^T (16 x 128) += x^T (16 x 16 tokens of block tb, three terms) X (those tokens of the tile).
__device__ __forceinline__ void state_add(float (&st)[16][4], const uint32_t (&x)[3][4], uint32_t tile, int tb, int lane) {
#pragma unroll
  for (int np = 0; np < 8; ++np) {
    uint32_t b[4];
    ldsm_t(b, tile + tile_cr(tb * 16, np * 2, lane));
    prod3(st[2 * np], x, b[0], b[1]);
    prod3(st[2 * np + 1], x, b[2], b[3]);
  }
}
// acc^T (16 x 64 tokens i) += x^T (16 x 64 tokens j) M^T for the lower triangular M (three planes of blocks): columns j <= i.
// acc may be x: a block is read before anything is added to it.
__device__ __forceinline__ void tri_times(float (&acc)[8][4], const float (&x)[8][4], uint32_t planes, int lane) {
#pragma unroll
  for (int jb = 3; jb >= 0; --jb) {
    uint32_t s[3][4];
    split_a(x[2 * jb], x[2 * jb + 1], s);
#pragma unroll
    for (int ib = jb; ib < 4; ++ib) {
      uint32_t b[3][4], bb[3][2];
#pragma unroll
      for (int p = 0; p < 3; ++p) ldsm(b[p], planes + p * kTri * 2 + blk_of(ib, jb) * 512 + blk_rc(lane));
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        pick(bb, b, e);
        prod6(acc[2 * ib + e], s, bb);
      }
    }
  }
}
// Infinities and NaN.  A triangular product multiplies the zeros above the diagonal of its 16 x 16 blocks too, and an infinity has no
// three terms, so a value that is not finite would reach tokens that it does not concern.  Each of the chain kernels marks
// the pairs of sequence and head where one came up, and these are done again token by token (ftb_gdn_redo_fwd and _bwd of
// gdn.cu).  What a token writes into the state stays in it: 0 * x, added up, is 0 for finite x alone, also of the state at the end.
// (The mark is in shared memory: a register for it would be one more to spill.)  16 x 1024 tokens, 32 heads: forward 1.00 -> 1.02 ms,
// backward 4.12 -> 4.19, for the look and the launches that follow.
__device__ __forceinline__ void add_zero_times(float& nan, float x) {
  asm volatile("fma.rn.f32 %0, %1, 0f00000000, %0;" : "+f"(nan) : "f"(x));
}
__device__ __forceinline__ void mark(Gates* gt, float nan) {
  if (__float_as_uint(nan) & 0x7fffffffu) gt->bad = 1;
}
template <int N>
__device__ __forceinline__ void look_at(Gates* gt, const float (&x)[N][4]) {
  float n[4] = {};
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) add_zero_times(n[e], x[i][e]);
  mark(gt, (n[0] + n[1]) + (n[2] + n[3]));
}
__device__ __forceinline__ void look_at(Gates* gt, float x, float y) {
  float n = 0.f;
  add_zero_times(n, x);
  add_zero_times(n, y);
  mark(gt, n);
}

// The value columns of a chunk's rows in shared memory (the warp's own 16 columns) out to global memory, 16 bytes a lane.
__device__ __forceinline__ void store_rows(bf16* dst, long row_stride, uint32_t tile, int warp, int n, int lane) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = i * 16 + (lane >> 1), c = warp * 2 + (lane & 1);
    uint32_t x[4];
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]) : "r"(tile + tile_at(r, c))
                 : "memory");
    if (r < n) *reinterpret_cast<uint4*>(dst + r * row_stride + c * 8) = make_uint4(x[0], x[1], x[2], x[3]);
  }
}

// ================================================================================================ forward
constexpr int kFwdStage = 3 * kTile + 2 * kTri * 4;
constexpr int kFwdSmem = 2 * kFwdStage + 2 * 3 * kTri * 2 + sizeof(Gates);

__global__ void __launch_bounds__(NT, 1) gdn_chunk_forward_kernel(const Args a) {
  extern __shared__ __align__(128) char sm[];
  char* planes_t = sm + 2 * kFwdStage;
  char* planes_p = planes_t + 3 * kTri * 2;
  Gates* gt = reinterpret_cast<Gates*>(planes_p + 3 * kTri * 2);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int hv = blockIdx.x, seq = a.order[blockIdx.y];
  const int hk = hv / (a.HV / a.HK);
  const int t0 = a.cu[seq], t1 = a.cu[seq + 1];
  const long slot0 = first_slot(a.cu, seq);
  const long qs = (long)a.HK * DK, vs = (long)a.HV * DV;
  const int nc = (t1 - t0 + C - 1) / C;
  auto fetch = [&](int c) {
    const uint32_t st = smem_addr(sm) + (c & 1) * kFwdStage;
    const int t = t0 + c * C, n = min(C, t1 - t);
    load_tile(st, a.k + (long)t * qs + hk * DK, qs, n, tid, NT);
    load_tile(st + kTile, a.q + (long)t * qs + hk * DK, qs, n, tid, NT);
    load_tile(st + 2 * kTile, a.v + (long)t * a.v_ts + hv * DV, a.v_ts, n, tid, NT);
    const float* tt = a.tri_t + ((slot0 + c) * a.HV + hv) * kTri;
    const float* pp = a.tri_p + ((slot0 + c) * a.HV + hv) * kTri;
    for (int i = tid; i < kTri / 4; i += NT) {
      cp16(st + 3 * kTile + i * 16, tt + i * 4, true);
      cp16(st + 3 * kTile + kTri * 4 + i * 16, pp + i * 4, true);
    }
    cp_commit();
  };
  float S[16][4];
  load_state(S, a.state_in ? a.state_in + ((size_t)seq * a.HV + hv) * DK * DV : nullptr, warp * 16, lane);
  if (nc > 0) fetch(0);
  if (tid == 0) gt->bad = 0;
  for (int c = 0; c < nc; ++c) {
    cp_wait_all();
    __syncthreads();                               // this chunk is there, and the one before is done with everything
    if (c + 1 < nc) fetch(c + 1);
    char* stage = sm + (c & 1) * kFwdStage;
    const uint32_t k_s = smem_addr(stage), q_s = k_s + kTile, v_s = k_s + 2 * kTile;
    const int t = t0 + c * C, n = min(C, t1 - t);
    make_gates(gt, a, slot0 + c, t, n, hv, tid);
    split_tri(planes_t, reinterpret_cast<const float*>(stage + 3 * kTile), tid);
    split_tri(planes_p, reinterpret_cast<const float*>(stage + 3 * kTile) + kTri, tid);
    float R[8][4] = {}, O[8][4] = {};
#pragma unroll
    for (int kb = 0; kb < 8; ++kb) {
      uint32_t s[3][4];
      split_a(S[2 * kb], S[2 * kb + 1], s);
      state_times_tile(R, s, k_s, kb, lane);
      state_times_tile(O, s, q_s, kb, lane);
    }
    __syncthreads();                               // gates and planes
#pragma unroll
    for (int np = 0; np < 4; ++np) {               // right-hand side
      uint32_t u[4];
      ldsm_t(u, v_s + tile_rc(np * 16, warp * 2, lane));
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int nb = 2 * np + h, i = nb * 8 + (lane & 3) * 2;
        const float2 gm = *reinterpret_cast<const float2*>(gt->gam + i), v0 = bf2(u[2 * h]), v1 = bf2(u[2 * h + 1]);
        R[nb][0] = v0.x - gm.x * R[nb][0];
        R[nb][1] = v0.y - gm.y * R[nb][1];
        R[nb][2] = v1.x - gm.x * R[nb][2];
        R[nb][3] = v1.y - gm.y * R[nb][3];
        O[nb][0] *= a.scale * gm.x;
        O[nb][1] *= a.scale * gm.y;
        O[nb][2] *= a.scale * gm.x;
        O[nb][3] *= a.scale * gm.y;
      }
    }
    tri_times(R, R, smem_addr(planes_t), lane);
    float (&Y)[8][4] = R;
    if (a.r) {
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        uint32_t u[4];
        ldsm_t(u, v_s + tile_rc(np * 16, warp * 2, lane));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int nb = 2 * np + h, i = nb * 8 + (lane & 3) * 2;
          const float2 v0 = bf2(u[2 * h]), v1 = bf2(u[2 * h + 1]);
          float* rp = a.r + (long)(t + i) * vs + hv * DV + warp * 16 + (lane >> 2);
          if (i < n) { rp[0] = v0.x - Y[nb][0]; rp[8] = v1.x - Y[nb][2]; }
          if (i + 1 < n) { rp[vs] = v0.y - Y[nb][1]; rp[vs + 8] = v1.y - Y[nb][3]; }
        }
      }
    }
#pragma unroll
    for (int nb = 0; nb < 8; ++nb) {
      const float2 b = *reinterpret_cast<const float2*>(gt->bet + nb * 8 + (lane & 3) * 2);
      Y[nb][0] *= b.x;
      Y[nb][1] *= b.y;
      Y[nb][2] *= b.x;
      Y[nb][3] *= b.y;
    }
    tri_times(O, Y, smem_addr(planes_p), lane);
    look_at(gt, O);
    __syncwarp();                                  // the output takes the place of v in the warp's own columns
#pragma unroll
    for (int np = 0; np < 4; ++np)
      stsm_t(v_s + tile_rc(np * 16, warp * 2, lane), pack_bf(O[2 * np][0], O[2 * np][1]), pack_bf(O[2 * np][2], O[2 * np][3]),
             pack_bf(O[2 * np + 1][0], O[2 * np + 1][1]), pack_bf(O[2 * np + 1][2], O[2 * np + 1][3]));
    __syncwarp();
    store_rows(a.o + (long)t * vs + hv * DV, vs, v_s, warp, n, lane);
    const float end = gt->end;
#pragma unroll
    for (int nb = 0; nb < 16; ++nb)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[nb][e] *= end;
#pragma unroll
    for (int tb = 0; tb < 4; ++tb) {
      float x[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float2 d = *reinterpret_cast<const float2*>(gt->dec + (2 * tb + h) * 8 + (lane & 3) * 2);
        x[h][0] = Y[2 * tb + h][0] * d.x;
        x[h][1] = Y[2 * tb + h][1] * d.y;
        x[h][2] = Y[2 * tb + h][2] * d.x;
        x[h][3] = Y[2 * tb + h][3] * d.y;
      }
      uint32_t s[3][4];
      split_a(x[0], x[1], s);
      state_add(S, s, k_s, tb, lane);
    }
  }
  if (a.state_out) store_state(a.state_out + ((size_t)seq * a.HV + hv) * DK * DV, S, warp * 16, lane);
  __syncthreads();
  look_at(gt, S);
  __syncthreads();
  if (tid == 0) a.redo[seq * a.HV + hv] = gt->bad;
}

// ================================================================================================ backward, reverse in time
// Sums over value columns are added up over the warps in shared memory: each warp leaves its part of (64 tokens x 32 key
// columns), then a thread adds eight parts of eight elements.
constexpr int kRedLd = 36;                                                   // floats in a row of a part
constexpr int kRedR = 8 * C * kRedLd * 4;
constexpr int kRevStage = 3 * kTile + 2 * kTri * 4;
constexpr int kRevSmem = 2 * kRevStage + kRedR + sizeof(Gates) + 8 * C * 4;  // (the planes lie in the parts' place)
static_assert(2 * 3 * kTri * 2 <= kRedR, "planes");

// y = v - r of the warp's 16 value columns as accumulator tiles (rows = value columns, columns = the chunk's tokens): asked for in
// one go, all of it on its way at once, and put together where it is used.
struct ColumnsOfY {
  float r[8][4];
  uint32_t v[8][2];
  __device__ __forceinline__ void ask(const Args& a, int t, int n, long vs, int hv, int col, int lane) {
    const int c = hv * DV + col + (lane >> 2);
    const unsigned short* vp = reinterpret_cast<const unsigned short*>(a.v);
#pragma unroll
    for (int nb = 0; nb < 8; ++nb)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = nb * 8 + (lane & 3) * 2 + h;
        const long ra = (long)(t + i) * vs + c, va = (long)(t + i) * a.v_ts + c;
        const bool on = i < n;
        r[nb][h] = on ? a.r[ra] : 0.f;
        r[nb][2 + h] = on ? a.r[ra + 8] : 0.f;
        v[nb][h] = on ? (uint32_t)vp[va] | (uint32_t)vp[va + 8] << 16 : 0u;
      }
  }
  __device__ __forceinline__ void get(float (&y)[4], int nb) const {
    const float2 v0 = bf2(v[nb][0]), v1 = bf2(v[nb][1]);
    y[0] = v0.x - r[nb][0];
    y[1] = v1.x - r[nb][1];
    y[2] = v0.y - r[nb][2];
    y[3] = v1.y - r[nb][3];
  }
};
// The same columns with the tokens as rows, as A operands of 16 tokens x 16 columns, times beta.
struct RowsOfY {
  float2 r[4][4];
  uint32_t v[4][4];
  __device__ __forceinline__ void ask(const Args& a, int t, int n, long vs, int hv, int col, int lane) {
#pragma unroll
    for (int tt = 0; tt < 4; ++tt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = tt * 16 + (lane >> 2) + (e & 1) * 8;
        const int c = hv * DV + col + (lane & 3) * 2 + (e >> 1) * 8;
        r[tt][e] = i < n ? *reinterpret_cast<const float2*>(a.r + (long)(t + i) * vs + c) : make_float2(0.f, 0.f);
        v[tt][e] = i < n ? *reinterpret_cast<const uint32_t*>(a.v + (long)(t + i) * a.v_ts + c) : 0u;
      }
  }
  __device__ __forceinline__ void get(uint32_t (&s)[3][4], const float* bet, int tt, int lane) const {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 x = bf2(v[tt][e]);
      const float b = bet[tt * 16 + (lane >> 2) + (e & 1) * 8];
      split3((x.x - r[tt][e].x) * b, (x.y - r[tt][e].y) * b, s[0][e], s[1][e], s[2][e]);
    }
  }
};
// fp32 rows of 128 in shared memory: the 16-byte piece c of row r lies at piece c ^ (r & 7).
__device__ __forceinline__ uint32_t row32_at(int r, int c) { return r * 512 + ((c ^ (r & 7)) << 4); }
// 16 rows x 16 columns of them as an A operand, three terms.
__device__ __forceinline__ void rows_a(uint32_t (&s)[3][4], const char* rows, int i0, int col, int lane) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int c = col + (lane & 3) * 2 + (e >> 1) * 8;
    const float2 u = *reinterpret_cast<const float2*>(rows + row32_at(i0 + (lane >> 2) + (e & 1) * 8, c >> 2) + (c & 3) * 4);
    split3(u.x, u.y, s[0][e], s[1][e], s[2][e]);
  }
}
// The state (16 value columns x 8 key rows of tile nb) as a B operand that sums over value columns, three terms.
__device__ __forceinline__ void state_b(uint32_t (&b)[3][2], const float (&st)[4]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t t0, t1, t2;
    split3(st[2 * h], st[2 * h + 1], t0, t1, t2);
    b[0][h] = transpose8(t0);
    b[1][h] = transpose8(t1);
    b[2][h] = transpose8(t2);
  }
}

__global__ void __launch_bounds__(NT, 1) gdn_chunk_reverse_kernel(const Args a) {
  extern __shared__ __align__(128) char sm[];
  char* planes_t = sm + 2 * kRevStage;
  char* planes_p = planes_t + 3 * kTri * 2;
  float* red = reinterpret_cast<float*>(sm + 2 * kRevStage);
  Gates* gt = reinterpret_cast<Gates*>(sm + 2 * kRevStage + kRedR);
  float* dot = reinterpret_cast<float*>(gt + 1);                   // [8][64]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int hv = blockIdx.x, seq = a.order[blockIdx.y];
  const int hk = hv / (a.HV / a.HK);
  const int t0 = a.cu[seq], t1 = a.cu[seq + 1];
  const long slot0 = first_slot(a.cu, seq);
  const long qs = (long)a.HK * DK, vs = (long)a.HV * DV;
  const int nc = (t1 - t0 + C - 1) / C;
  auto fetch = [&](int c) {
    const uint32_t st = smem_addr(sm) + (c & 1) * kRevStage;
    const int t = t0 + c * C, n = min(C, t1 - t);
    load_tile(st, a.k + (long)t * qs + hk * DK, qs, n, tid, NT);
    load_tile(st + kTile, a.q + (long)t * qs + hk * DK, qs, n, tid, NT);
    load_tile(st + 2 * kTile, a.d_o + (long)t * vs + hv * DV, vs, n, tid, NT);
    const float* tt = a.tri_t + ((slot0 + c) * a.HV + hv) * kTri;
    const float* pp = a.tri_p + ((slot0 + c) * a.HV + hv) * kTri;
    for (int i = tid; i < kTri / 4; i += NT) {
      cp16(st + 3 * kTile + i * 16, tt + i * 4, true);
      cp16(st + 3 * kTile + kTri * 4 + i * 16, pp + i * 4, true);
    }
    cp_commit();
  };
  float X[16][4];
  load_state(X, a.state_in ? a.state_in + ((size_t)seq * a.HV + hv) * DK * DV : nullptr, warp * 16, lane);
  if (nc > 0) fetch(nc - 1);
  if (tid == 0) gt->bad = 0;
  for (int c = nc - 1; c >= 0; --c) {
    cp_wait_all();
    __syncthreads();
    if (c > 0) fetch(c - 1);
    char* stage = sm + (c & 1) * kRevStage;
    const uint32_t k_s = smem_addr(stage), q_s = k_s + kTile, d_s = k_s + 2 * kTile;
    const int t = t0 + c * C, n = min(C, t1 - t);
    make_gates(gt, a, slot0 + c, t, n, hv, tid);
    split_tri(planes_t, reinterpret_cast<const float*>(stage + 3 * kTile), tid);
    split_tri(planes_p, reinterpret_cast<const float*>(stage + 3 * kTile) + kTri, tid);
    ColumnsOfY columns;
    columns.ask(a, t, n, vs, hv, warp * 16, lane);
    if (c > 0) {
      prefetch_rows(reinterpret_cast<const char*>(a.r + (long)(t - C) * vs + hv * DV), vs * 4, 4, C, tid);
      prefetch_rows(reinterpret_cast<const char*>(a.v + (long)(t - C) * a.v_ts + hv * DV), a.v_ts * 2, 2, C, tid);
    }
    float R[8][4] = {};
#pragma unroll
    for (int kb = 0; kb < 8; ++kb) {
      uint32_t s[3][4];
      split_a(X[2 * kb], X[2 * kb + 1], s);
      state_times_tile(R, s, k_s, kb, lane);
    }
    __syncthreads();
#pragma unroll
    for (int nb = 0; nb < 8; ++nb) {
      const float2 d = *reinterpret_cast<const float2*>(gt->dec + nb * 8 + (lane & 3) * 2);
      R[nb][0] *= d.x;
      R[nb][1] *= d.y;
      R[nb][2] *= d.x;
      R[nb][3] *= d.y;
    }
#pragma unroll
    for (int jb = 0; jb < 4; ++jb) {               // += dO^T P
      uint32_t x[4];
      ldsm_t(x, d_s + tile_rc(jb * 16, warp * 2, lane));
#pragma unroll
      for (int ib = 0; ib <= jb; ++ib) {
        uint32_t b[3][4], bb[3][2];
#pragma unroll
        for (int p = 0; p < 3; ++p) ldsm_t(b[p], smem_addr(planes_p) + p * kTri * 2 + blk_of(jb, ib) * 512 + blk_cr(lane));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          pick(bb, b, e);
          prod3(R[2 * ib + e], x, bb);
        }
      }
    }
#pragma unroll
    for (int nb = 0; nb < 8; ++nb) {               // rhs . y over the warp's columns, then rhs <- -beta rhs
      float y[4];
      columns.get(y, nb);
      float2 p = make_float2(R[nb][0] * y[0] + R[nb][2] * y[2], R[nb][1] * y[1] + R[nb][3] * y[3]);
#pragma unroll
      for (int m = 4; m < 32; m <<= 1) {
        p.x += __shfl_xor_sync(0xffffffffu, p.x, m);
        p.y += __shfl_xor_sync(0xffffffffu, p.y, m);
      }
      if (lane < 4) *reinterpret_cast<float2*>(dot + warp * C + nb * 8 + lane * 2) = p;
      const float2 b = *reinterpret_cast<const float2*>(gt->bet + nb * 8 + (lane & 3) * 2);
      R[nb][0] *= -b.x;
      R[nb][1] *= -b.y;
      R[nb][2] *= -b.x;
      R[nb][3] *= -b.y;
    }
#pragma unroll
    for (int jb = 0; jb < 4; ++jb) {               // dR^T, block by block in place (block jb is read before anything is added to it)
      uint32_t s[3][4];
      split_a(R[2 * jb], R[2 * jb + 1], s);
#pragma unroll
      for (int ib = 0; ib <= jb; ++ib) {
        uint32_t b[3][4], bb[3][2];
#pragma unroll
        for (int p = 0; p < 3; ++p) ldsm_t(b[p], smem_addr(planes_t) + p * kTri * 2 + blk_of(jb, ib) * 512 + blk_cr(lane));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          pick(bb, b, e);
          prod6(R[2 * ib + e], s, bb);
        }
      }
    }
    float (&Z)[8][4] = R;
    RowsOfY rows;
    rows.ask(a, t, n, vs, hv, warp * 16, lane);
#pragma unroll
    for (int nb = 0; nb < 8; ++nb) {
      const int i = nb * 8 + (lane & 3) * 2;
      const long at = (long)(t + i) * vs + hv * DV + warp * 16 + (lane >> 2);
      if (i < n) { a.dr[at] = Z[nb][0]; a.dr[at + 8] = Z[nb][2]; }
      if (i + 1 < n) { a.dr[at + vs] = Z[nb][1]; a.dr[at + vs + 8] = Z[nb][3]; }
    }
    __syncthreads();                               // every warp is done with the planes: their place takes the parts now
    // B Y X^T, decayed: rows of (beta y) against the gradient state
    {
      uint32_t s[4][3][4];
#pragma unroll
      for (int tt = 0; tt < 4; ++tt) rows.get(s[tt], gt->bet, tt, lane);
      float kd = 0.f;                              // the thread's part of k . dk of its row
      const int row = tid >> 2, c8 = (tid & 3) * 8;
#pragma unroll
      for (int gi = 0; gi < 4; ++gi) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          uint32_t b[3][2];
          state_b(b, X[gi * 4 + u]);
#pragma unroll
          for (int tt = 0; tt < 4; ++tt) {
            float acc[4] = {};
            prod6(acc, s[tt], b);
            float* p = red + (warp * C + tt * 16 + (lane >> 2)) * kRedLd + u * 8 + (lane & 3) * 2;
            *reinterpret_cast<float2*>(p) = make_float2(acc[0], acc[1]);
            *reinterpret_cast<float2*>(p + 8 * kRedLd) = make_float2(acc[2], acc[3]);
          }
        }
        __syncthreads();
        float x[8] = {};
#pragma unroll
        for (int w = 0; w < 8; ++w) {
          const float4* p = reinterpret_cast<const float4*>(red + (w * C + row) * kRedLd + c8);
          const float4 u = p[0], v = p[1];
          x[0] += u.x; x[1] += u.y; x[2] += u.z; x[3] += u.w;
          x[4] += v.x; x[5] += v.y; x[6] += v.z; x[7] += v.w;
        }
        const float d = gt->dec[row];
        uint32_t kr[4];
        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(kr[0]), "=r"(kr[1]), "=r"(kr[2]), "=r"(kr[3])
                     : "r"(k_s + tile_at(row, gi * 4 + (tid & 3))) : "memory");
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 k2 = bf2(kr[e]);
          x[2 * e] *= d;
          x[2 * e + 1] *= d;
          kd += k2.x * x[2 * e] + k2.y * x[2 * e + 1];
        }
        if (row < n) {
          float4* p = reinterpret_cast<float4*>(a.dk + ((long)(t + row) * a.HV + hv) * DK + gi * 32 + c8);
          p[0] = make_float4(x[0], x[1], x[2], x[3]);
          p[1] = make_float4(x[4], x[5], x[6], x[7]);
        }
        __syncthreads();
      }
      kd += __shfl_xor_sync(0xffffffffu, kd, 1);
      kd += __shfl_xor_sync(0xffffffffu, kd, 2);
      look_at(gt, kd, 0.f);
      if ((tid & 3) == 0 && row < n) a.sacc[(long)(t + row) * a.HV + hv] = -kd;
      if (tid < n) {
        float s8 = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) s8 += dot[w * C + tid];
        look_at(gt, s8, 0.f);
        a.dbeta[(long)(t + tid) * a.HV + hv] = s8;
      }
    }
    // X <- exp(G_C) X + Q^T (scale exp(G) dO) + K^T (exp(G) dR)
    const float end = gt->end;
#pragma unroll
    for (int nb = 0; nb < 16; ++nb)
#pragma unroll
      for (int e = 0; e < 4; ++e) X[nb][e] *= end;
#pragma unroll
    for (int tb = 0; tb < 4; ++tb) {
      uint32_t u[4], s[3][4];
      ldsm_t(u, d_s + tile_rc(tb * 16, warp * 2, lane));
      float x[2][4], z[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float2 gm = *reinterpret_cast<const float2*>(gt->gam + (2 * tb + h) * 8 + (lane & 3) * 2);
        const float2 d0 = bf2(u[2 * h]), d1 = bf2(u[2 * h + 1]);
        x[h][0] = d0.x * (a.scale * gm.x);
        x[h][1] = d0.y * (a.scale * gm.y);
        x[h][2] = d1.x * (a.scale * gm.x);
        x[h][3] = d1.y * (a.scale * gm.y);
        z[h][0] = Z[2 * tb + h][0] * gm.x;
        z[h][1] = Z[2 * tb + h][1] * gm.y;
        z[h][2] = Z[2 * tb + h][2] * gm.x;
        z[h][3] = Z[2 * tb + h][3] * gm.y;
      }
      split_a(x[0], x[1], s);
      state_add(X, s, q_s, tb, lane);
      split_a(z[0], z[1], s);
      state_add(X, s, k_s, tb, lane);
    }
    __syncwarp();                                  // dv = -dR takes the place of dO in the warp's own columns
#pragma unroll
    for (int np = 0; np < 4; ++np)
      stsm_t(d_s + tile_rc(np * 16, warp * 2, lane), pack_bf(-Z[2 * np][0], -Z[2 * np][1]), pack_bf(-Z[2 * np][2], -Z[2 * np][3]),
             pack_bf(-Z[2 * np + 1][0], -Z[2 * np + 1][1]), pack_bf(-Z[2 * np + 1][2], -Z[2 * np + 1][3]));
    __syncwarp();
    store_rows(a.dv + (long)t * a.dv_ts + hv * DV, a.dv_ts, d_s, warp, n, lane);
  }
  if (a.state_out) store_state(a.state_out + ((size_t)seq * a.HV + hv) * DK * DV, X, warp * 16, lane);
  __syncthreads();
  look_at(gt, X);
  __syncthreads();
  if (tid == 0) a.redo[seq * a.HV + hv] = gt->bad;
}

// ================================================================================================ backward, forward in time
// W1 and W2 of the chunk from products over all value columns (warps share the ten lower blocks; the diagonal of W1 stays in
// fp32, aside), then dQ and dK: a warp has 16 tokens and 64 key columns of both, and sums over all value columns by itself.  The
// state goes through shared memory for that, as three planes of bf16; its place is that of Y, which is done with by then.  (With
// every warp multiplying its own value columns, and the parts of dQ and dK added up over the warps, 16 key columns at a time,
// the warps met sixteen times a chunk and moved 1 MB through shared memory: 3.0 ms for 16 x 1024 tokens, 32 heads.)
constexpr int kPlane = DV * 256;                                             // (128 value columns, 128 key columns) bf16
constexpr int kFinSmem = 3 * kTile + 3 * kPlane + C * 512 + 2 * 3 * kTri * 2 + sizeof(Gates) + C * 8 + 2 * 4 * C * 4 + 3 * C * 4;
static_assert(3 * kTile <= 3 * kPlane, "planes of Y in the state's place");

__global__ void __launch_bounds__(NT, 1) gdn_chunk_grad_kernel(const Args a) {
  extern __shared__ __align__(128) char sm[];
  char* st_s = sm + 3 * kTile;                                     // planes of the state, or of Y
  char* dr_s = st_s + 3 * kPlane;                                  // dR as it is, fp32
  char* w1_s = dr_s + C * 512;
  char* w2_s = w1_s + 3 * kTri * 2;
  double* gs = reinterpret_cast<double*>(w2_s + 3 * kTri * 2);     // [64]
  float* col1 = reinterpret_cast<float*>(gs + C);                  // [4][64] column sums of W1 o QK^T without its diagonal, by block row
  float* col2 = col1 + 4 * C;                                      // [4][64] of D o KK^T o (dR Y^T)
  Gates* gt = reinterpret_cast<Gates*>(col2 + 4 * C);
  float* diag = reinterpret_cast<float*>(gt + 1);                  // [64] the diagonal of W1
  float* sums = diag + C;                                          // [2][64] q.dq + k.dk by halves of the key columns
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int hv = blockIdx.x, seq = a.order[blockIdx.y];
  const int hk = hv / (a.HV / a.HK);
  const int t0 = a.cu[seq], t1 = a.cu[seq + 1];
  const long slot0 = first_slot(a.cu, seq);
  const long qs = (long)a.HK * DK, vs = (long)a.HV * DV;
  const int nc = (t1 - t0 + C - 1) / C;
  const uint32_t k_s = smem_addr(sm), q_s = k_s + kTile, d_s = k_s + 2 * kTile, w1 = smem_addr(w1_s), w2 = smem_addr(w2_s);
  auto fetch = [&](int c) {
    const int t = t0 + c * C, n = min(C, t1 - t);
    load_tile(k_s, a.k + (long)t * qs + hk * DK, qs, n, tid, NT);
    load_tile(q_s, a.q + (long)t * qs + hk * DK, qs, n, tid, NT);
    load_tile(d_s, a.d_o + (long)t * vs + hv * DV, vs, n, tid, NT);
    for (int i = tid; i < C * 32; i += NT) {
      const int r = i >> 5, p = i & 31;
      cp16(smem_addr(dr_s) + row32_at(r, p), a.dr + (long)(t + (r < n ? r : 0)) * vs + hv * DV + p * 4, r < n);
    }
    cp_commit();
  };
  float S[16][4];
  load_state(S, a.state_in ? a.state_in + ((size_t)seq * a.HV + hv) * DK * DV : nullptr, warp * 16, lane);
  if (nc > 0) fetch(0);
  if (tid == 0) gt->bad = 0;
  for (int c = 0; c < nc; ++c) {
    const int t = t0 + c * C, n = min(C, t1 - t);
    make_gates(gt, a, slot0 + c, t, n, hv, tid);
    if (tid < C) gs[tid] = a.gsum[((slot0 + c) * a.HV + hv) * C + tid];
    for (int i = tid; i < 2 * 4 * C; i += NT) col1[i] = 0.f;
    {                                              // y as three planes of (64, 128)
      uint4 vv[4];
      float4 ra[4], rb[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = tid + u * NT, r = i >> 4, c8 = i & 15;
        const long at = (long)(t + r) * vs + hv * DV + c8 * 8;
        vv[u] = r < n ? *reinterpret_cast<const uint4*>(a.v + (long)(t + r) * a.v_ts + hv * DV + c8 * 8) : make_uint4(0, 0, 0, 0);
        ra[u] = r < n ? *reinterpret_cast<const float4*>(a.r + at) : make_float4(0.f, 0.f, 0.f, 0.f);
        rb[u] = r < n ? *reinterpret_cast<const float4*>(a.r + at + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = tid + u * NT, r = i >> 4, c8 = i & 15;
        uint32_t p[3][4];
        const float2 v0 = bf2(vv[u].x), v1 = bf2(vv[u].y), v2 = bf2(vv[u].z), v3 = bf2(vv[u].w);
        split3(v0.x - ra[u].x, v0.y - ra[u].y, p[0][0], p[1][0], p[2][0]);
        split3(v1.x - ra[u].z, v1.y - ra[u].w, p[0][1], p[1][1], p[2][1]);
        split3(v2.x - rb[u].x, v2.y - rb[u].y, p[0][2], p[1][2], p[2][2]);
        split3(v3.x - rb[u].z, v3.y - rb[u].w, p[0][3], p[1][3], p[2][3]);
#pragma unroll
        for (int j = 0; j < 3; ++j)
          *reinterpret_cast<uint4*>(st_s + j * kTile + tile_at(r, c8)) = make_uint4(p[j][0], p[j][1], p[j][2], p[j][3]);
      }
    }
    cp_wait_all();
    __syncthreads();
    if (c + 1 < nc) {                              // the next chunk's rows come closer meanwhile
      const int m = min(C, t1 - t - C);
      const long at = (long)(t + C) * vs + hv * DV, kt = (long)(t + C) * qs + hk * DK;
      prefetch_rows(reinterpret_cast<const char*>(a.r + at), vs * 4, 4, m, tid);
      prefetch_rows(reinterpret_cast<const char*>(a.dr + at), vs * 4, 4, m, tid);
      prefetch_rows(reinterpret_cast<const char*>(a.v + (long)(t + C) * a.v_ts + hv * DV), a.v_ts * 2, 2, m, tid);
      prefetch_rows(reinterpret_cast<const char*>(a.d_o + at), vs * 2, 2, m, tid);
      prefetch_rows(reinterpret_cast<const char*>(a.k + kt), qs * 2, 2, m, tid);
      prefetch_rows(reinterpret_cast<const char*>(a.q + kt), qs * 2, 2, m, tid);
    }
    // blocks 0..9 of W2 on warps 0-4 (two each), blocks of W1 on warps 5-7
    const bool second = warp < 5;
    const int b_lo = second ? warp * 2 : (warp - 5) * 3, b_hi = second ? b_lo + 2 : (warp == 7 ? 10 : b_lo + 3);
    for (int bl = b_lo; bl < b_hi; ++bl) {
      int ib = 0;
      while (blk_of(ib + 1, 0) <= bl) ++ib;
      const int jb = bl - blk_of(ib, 0);
      float m[2][4] = {}, x[2][4] = {};            // (dO or dR) Y^T and (Q or K) K^T
#pragma unroll
      for (int kb = 0; kb < 8; ++kb) {
        uint32_t y[3][4], f[4], b[4], bb[3][2];
#pragma unroll
        for (int p = 0; p < 3; ++p) ldsm(y[p], smem_addr(st_s) + p * kTile + tile_rc(jb * 16, kb * 2, lane));
        if (second) {
          uint32_t s[3][4];
          rows_a(s, dr_s, ib * 16, kb * 16, lane);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            pick(bb, y, e);
            prod6(m[e], s, bb);
          }
        } else {
          ldsm(f, d_s + tile_cr(ib * 16, kb * 2, lane));
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            pick(bb, y, e);
            prod3(m[e], f, bb);
          }
        }
        ldsm(f, (second ? k_s : q_s) + tile_cr(ib * 16, kb * 2, lane));
        ldsm(b, k_s + tile_rc(jb * 16, kb * 2, lane));
        prod1(x[0], f, b[0], b[1]);
        prod1(x[1], f, b[2], b[3]);
      }
      char* w = (second ? w2_s : w1_s) + bl * 512;
      float* col = (second ? col2 : col1) + ib * C + jb * 16;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float2 cs = make_float2(0.f, 0.f);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = ib * 16 + (lane >> 2) + h * 8, j = jb * 16 + e * 8 + (lane & 3) * 2;
          float d0 = 0.f, d1 = 0.f;
          if (i > j) d0 = exp2_of(gs[i] - gs[j]);
          if (i > j + 1) d1 = exp2_of(gs[i] - gs[j + 1]);
          if (!second && i == j) diag[i] = m[e][2 * h] * (a.scale * gt->bet[i]);
          if (!second && i == j + 1) diag[i] = m[e][2 * h + 1] * (a.scale * gt->bet[i]);
          d0 *= m[e][2 * h];
          d1 *= m[e][2 * h + 1];
          if (!second) { d0 *= a.scale * gt->bet[j]; d1 *= a.scale * gt->bet[j + 1]; }
          cs.x += d0 * x[e][2 * h];
          cs.y += d1 * x[e][2 * h + 1];
          if (second) { d0 *= gt->bet[j]; d1 *= gt->bet[j + 1]; }
          uint32_t p0, p1, p2;
          split3(d0, d1, p0, p1, p2);
          char* at = w + blk_at(i & 15, e) + (lane & 3) * 4;
          *reinterpret_cast<uint32_t*>(at) = p0;
          *reinterpret_cast<uint32_t*>(at + kTri * 2) = p1;
          *reinterpret_cast<uint32_t*>(at + 2 * kTri * 2) = p2;
        }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
          cs.x += __shfl_xor_sync(0xffffffffu, cs.x, o);
          cs.y += __shfl_xor_sync(0xffffffffu, cs.y, o);
        }
        if (lane < 4) *reinterpret_cast<float2*>(col + e * 8 + lane * 2) = cs;
      }
    }
    __syncthreads();                               // W1, W2 are there; the state takes the place of y
#pragma unroll
    for (int nb = 0; nb < 16; ++nb)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t p0, p1, p2;
        split3(S[nb][2 * h], S[nb][2 * h + 1], p0, p1, p2);
        char* at = st_s + tile_at(warp * 16 + (lane >> 2) + h * 8, nb) + (lane & 3) * 4;
        *reinterpret_cast<uint32_t*>(at) = p0;
        *reinterpret_cast<uint32_t*>(at + kPlane) = p1;
        *reinterpret_cast<uint32_t*>(at + 2 * kPlane) = p2;
      }
    __syncthreads();
    {
      const int tt = warp & 3, half = warp >> 2;   // 16 tokens, 64 key columns
      float q2[8][4] = {}, k2[8][4] = {};
#pragma unroll 1
      for (int kb = 0; kb < 8; ++kb) {             // the state's part: 16 value columns a time
        uint32_t f[4], d[3][4];
        ldsm(f, d_s + tile_cr(tt * 16, kb * 2, lane));
        rows_a(d, dr_s, tt * 16, kb * 16, lane);
#pragma unroll
        for (int np = 0; np < 4; ++np) {
          uint32_t b[3][4], bb[3][2];
#pragma unroll
          for (int p = 0; p < 3; ++p) ldsm_t(b[p], smem_addr(st_s) + p * kPlane + tile_cr(kb * 16, half * 8 + np * 2, lane));
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            pick(bb, b, e);
            prod3(q2[2 * np + e], f, bb);
            prod6(k2[2 * np + e], d, bb);
          }
        }
      }
      const int r0 = tt * 16 + (lane >> 2);        // the thread's rows: r0 and r0 + 8
      const float g0 = gt->gam[r0], g1 = gt->gam[r0 + 8];
#pragma unroll
      for (int nb = 0; nb < 8; ++nb) {
        q2[nb][0] *= a.scale * g0;
        q2[nb][1] *= a.scale * g0;
        q2[nb][2] *= a.scale * g1;
        q2[nb][3] *= a.scale * g1;
        k2[nb][0] *= g0;
        k2[nb][1] *= g0;
        k2[nb][2] *= g1;
        k2[nb][3] *= g1;
      }
#pragma unroll 1
      for (int jb = 0; jb <= tt; ++jb) {           // W1 K into dQ, W2 K into dK
        uint32_t x[3][4], z[3][4];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          ldsm(x[p], w1 + p * kTri * 2 + blk_of(tt, jb) * 512 + blk_cr(lane));
          ldsm(z[p], w2 + p * kTri * 2 + blk_of(tt, jb) * 512 + blk_cr(lane));
        }
#pragma unroll
        for (int np = 0; np < 4; ++np) {
          uint32_t b[4];
          ldsm_t(b, k_s + tile_cr(jb * 16, half * 8 + np * 2, lane));
          prod3(q2[2 * np], x, b[0], b[1]);
          prod3(q2[2 * np + 1], x, b[2], b[3]);
          prod3(k2[2 * np], z, b[0], b[1]);
          prod3(k2[2 * np + 1], z, b[2], b[3]);
        }
      }
#pragma unroll 1
      for (int jb = tt; jb < 4; ++jb) {            // W1^T Q and W2^T K into dK
        uint32_t x[3][4], z[3][4];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          ldsm_t(x[p], w1 + p * kTri * 2 + blk_of(jb, tt) * 512 + blk_rc(lane));
          ldsm_t(z[p], w2 + p * kTri * 2 + blk_of(jb, tt) * 512 + blk_rc(lane));
        }
#pragma unroll
        for (int np = 0; np < 4; ++np) {
          uint32_t b[4];
          ldsm_t(b, q_s + tile_cr(jb * 16, half * 8 + np * 2, lane));
          prod3(k2[2 * np], x, b[0], b[1]);
          prod3(k2[2 * np + 1], x, b[2], b[3]);
          ldsm_t(b, k_s + tile_cr(jb * 16, half * 8 + np * 2, lane));
          prod3(k2[2 * np], z, b[0], b[1]);
          prod3(k2[2 * np + 1], z, b[2], b[3]);
        }
      }
      // out, with the diagonal of W1; q.dq + k.dk without it (it has no part in the gate's scalars and would only cancel)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = r0 + h * 8;
        const float w_ii = diag[r];
        float sc = 0.f;
#pragma unroll
        for (int nb = 0; nb < 8; ++nb) {
          const uint32_t at = tile_at(r, half * 8 + nb) + (lane & 3) * 4;
          uint32_t qu, ku;
          asm volatile("ld.shared.b32 %0, [%1];" : "=r"(qu) : "r"(q_s + at) : "memory");
          asm volatile("ld.shared.b32 %0, [%1];" : "=r"(ku) : "r"(k_s + at) : "memory");
          const float2 qf = bf2(qu), kf = bf2(ku);
          float2 dq = make_float2(q2[nb][2 * h], q2[nb][2 * h + 1]), dk = make_float2(k2[nb][2 * h], k2[nb][2 * h + 1]);
          sc += (qf.x * dq.x + qf.y * dq.y) + (kf.x * dk.x + kf.y * dk.y);
          dq.x += w_ii * kf.x;
          dq.y += w_ii * kf.y;
          dk.x += w_ii * qf.x;
          dk.y += w_ii * qf.y;
          if (r < n) {
            const long o = ((long)(t + r) * a.HV + hv) * DK + half * 64 + nb * 8 + (lane & 3) * 2;
            *reinterpret_cast<float2*>(a.dq + o) = dq;
            red_add2(a.dk + o, dk.x, dk.y);        // to what pass R wrote, one addition: no order to depend on
          }
        }
        sc += __shfl_xor_sync(0xffffffffu, sc, 1);
        sc += __shfl_xor_sync(0xffffffffu, sc, 2);
        look_at(gt, sc, w_ii);
        if ((lane & 3) == 0) sums[half * C + r] = sc;
      }
    }
    ColumnsOfY columns;
    columns.ask(a, t, n, vs, hv, warp * 16, lane);
    // S <- exp(G_C) S + (exp(G_C - G) K)^T B Y
    const float end = gt->end;
#pragma unroll
    for (int nb = 0; nb < 16; ++nb)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[nb][e] *= end;
#pragma unroll
    for (int tb = 0; tb < 4; ++tb) {
      float x[2][4];
      uint32_t s[3][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = (2 * tb + h) * 8;
        columns.get(x[h], 2 * tb + h);
        const float2 d = *reinterpret_cast<const float2*>(gt->dec + i + (lane & 3) * 2);
        const float2 b = *reinterpret_cast<const float2*>(gt->bet + i + (lane & 3) * 2);
        x[h][0] = x[h][0] * b.x * d.x;
        x[h][1] = x[h][1] * b.y * d.y;
        x[h][2] = x[h][2] * b.x * d.x;
        x[h][3] = x[h][3] * b.y * d.y;
      }
      split_a(x[0], x[1], s);
      state_add(S, s, k_s, tb, lane);
    }
    __syncthreads();                               // the tiles, the state's planes and the sums are done with, or there
    if (c + 1 < nc) fetch(c + 1);
    // per-token scalars: q.dq + k.(W2 K + S^ dr) - k.(W1^T Q + W2^T K), the last by the column sums (k.dk has it with the sign turned)
    if (tid < n) {
      const float c1 = col1[tid] + col1[C + tid] + col1[2 * C + tid] + col1[3 * C + tid];
      const float c2 = col2[tid] + col2[C + tid] + col2[2 * C + tid] + col2[3 * C + tid];
      const long at = (long)(t + tid) * a.HV + hv;
      const float sc = (sums[tid] + sums[C + tid]) - 2.f * (c1 + gt->bet[tid] * c2);
      a.dbeta[at] += c2;
      a.sacc[at] += sc;
      look_at(gt, c2, sc);
    }
    __syncthreads();
  }
  __syncthreads();
  look_at(gt, S);
  __syncthreads();
  if (gt->bad && tid == 0) a.redo[seq * a.HV + hv] = 1;   // (or the reverse pass has seen one)
}

template <typename F>
int launch(F* kernel, dim3 grid, int threads, int smem, const Args& a, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return -400 - (int)e;
  kernel<<<grid, threads, smem, s>>>(a);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -400 - (int)e;
}

}  // namespace

extern "C" {

// Bytes of workspace for T tokens in nseq sequences: the triangular matrices and gate sums of every chunk, the order.
long ftb_gdn_chunk_bytes(long T, int nseq, int HV) {
  const long slots = T / C + nseq;
  return slots * HV * (2L * kTri * 4 + C * 8) + (nseq + 15L) / 16 * 64;
}

// What gdn.cu's pass 0 does (o, r, final state), for DK = DV = 128 and tensors on 16 bytes.  Returns -2 for anything else.  redo
// (nseq, HV): where ftb_gdn_redo_fwd has to follow (ftb_gdn_redo_bwd for the one below).
int ftb_gdn_chunk_fwd(const void* q, const void* k, const void* v, long v_ts, const float* g, const float* beta, const int* cu,
                      int nseq, long T, const float* state_in, float* state_out, void* o, float* r, void* work, int* redo, int HK, int HV,
                      float scale, cudaStream_t s) {
  if (nseq <= 0) return 0;
  if (HK <= 0 || HV % HK || nseq > 65535 || HK > 65535 || v_ts % 8) return -2;
  if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)o | (uintptr_t)r | (uintptr_t)work) & 15) != 0) return -2;
  Args a = {};
  a.q = (const bf16*)q; a.k = (const bf16*)k; a.v = (const bf16*)v; a.g = g; a.beta = beta; a.cu = cu; a.nseq = nseq; a.T = T;
  a.v_ts = v_ts; a.state_in = state_in; a.state_out = state_out; a.o = (bf16*)o; a.r = r; a.HK = HK; a.HV = HV; a.scale = scale;
  const long slots = T / C + nseq;
  a.gsum = (double*)work;
  a.tri_t = (float*)(a.gsum + slots * HV * C);
  a.tri_p = a.tri_t + slots * HV * kTri;
  a.order = (int*)(a.tri_p + slots * HV * kTri);
  a.redo = redo;
  const int rc = launch(gdn_prep_kernel, dim3((unsigned)slots, HK), 128, kPrepSmem, a, s);
  if (rc) return rc;
  return launch(gdn_chunk_forward_kernel, dim3(HV, nseq), NT, kFwdSmem, a, s);
}

// Both backward passes of gdn.cu.  dstate_in: gradient of the final state or null; dstate_out: of the initial one.
int ftb_gdn_chunk_bwd(const void* q, const void* k, const void* v, long v_ts, const float* g, const float* beta, const int* cu,
                      int nseq, long T, const float* state_in, const float* dstate_in, float* dstate_out, const float* r,
                      const void* d_o, float* dr, void* dv, long dv_ts, float* dbeta, float* dq, float* dk, float* sacc, void* work,
                      int* redo, int HK, int HV, float scale, cudaStream_t s) {
  if (nseq <= 0) return 0;
  if (HK <= 0 || HV % HK || nseq > 65535 || HK > 65535 || v_ts % 8 || dv_ts % 8) return -2;
  if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)r | (uintptr_t)d_o | (uintptr_t)dr | (uintptr_t)dv | (uintptr_t)dq |
        (uintptr_t)dk | (uintptr_t)work) & 15) != 0) return -2;
  Args a = {};
  a.q = (const bf16*)q; a.k = (const bf16*)k; a.v = (const bf16*)v; a.g = g; a.beta = beta; a.cu = cu; a.nseq = nseq; a.T = T;
  a.v_ts = v_ts; a.r = const_cast<float*>(r); a.d_o = (const bf16*)d_o; a.dr = dr; a.dv = (bf16*)dv; a.dv_ts = dv_ts;
  a.dbeta = dbeta; a.dq = dq; a.dk = dk; a.sacc = sacc; a.HK = HK; a.HV = HV; a.scale = scale;
  const long slots = T / C + nseq;
  a.gsum = (double*)work;
  a.tri_t = (float*)(a.gsum + slots * HV * C);
  a.tri_p = a.tri_t + slots * HV * kTri;
  a.order = (int*)(a.tri_p + slots * HV * kTri);
  a.redo = redo;
  int rc = launch(gdn_prep_kernel, dim3((unsigned)slots, HK), 128, kPrepSmem, a, s);
  if (rc) return rc;
  a.state_in = dstate_in;
  a.state_out = dstate_out;
  rc = launch(gdn_chunk_reverse_kernel, dim3(HV, nseq), NT, kRevSmem, a, s);
  if (rc) return rc;
  a.state_in = state_in;
  a.state_out = nullptr;
  return launch(gdn_chunk_grad_kernel, dim3(HV, nseq), NT, kFinSmem, a, s);
}

}  // extern "C"
