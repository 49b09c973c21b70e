// Flash attention for sm_100a on tcgen05 / TMEM: varlen, GQA, causal with bottom-right alignment (the Lq queries
// of a sequence are the last Lq positions of its Lk keys, which is what a chunk of a long sequence sees), optional
// sliding window.  Replaces the external flash-attn 2/3/4 wheels the reference dispatches to
// (flextrain/ops/_kernels/attention.py:180-368, 629-759).
//
// Forward, one CTA per (128-query tile, head):
//   warp 0      TMA producer: Q once, then K / V tiles of 128 keys through two-stage rings (no multicast)
//   warp 1      MMA issuer:   S = Q·Kᵀ into a double-buffered TMEM accumulator, then PV = P·V
//   warps 2-5   softmax:      one query row per thread; S is read from TMEM, P is written as bf16 into a
//                             128B-swizzled shared tile that feeds the second MMA; the running output row
//                             lives in registers (O = O·alpha + PV), so nothing is ever rescaled in TMEM
// S_{j+1} is issued before the softmax of tile j completes, so the tensor core works under the exponentials.
//
// Backward, one CTA per (128-key tile, KV head): loops over the query heads of the group and over the query
// tiles that see these keys; five MMAs per pair (S, dP, dV += Pᵀ·dO, dK += dSᵀ·Q, dQ += dS·K); dK / dV accumulate
// in TMEM across the loop (deterministic).  dQ goes into an fp32 workspace as tiled reduce-adds.  In deterministic mode
// the CTAs that add to the same (query tile, head) take turns in a fixed order of key tiles through a counter, which fixes
// the summation order and makes dQ bit-reproducible; the wait is normally already satisfied (see BWD_* for the orders).
#include "ptx.cuh"

namespace ftb {

constexpr int FA_THREADS = 192;
constexpr int TQ = 128;   // query rows per tile
constexpr int TK = 128;   // keys per tile

struct FwdParams {
  const int* cu_q;
  const int* cu_k;
  int num_seqs;
  int H, KV;
  __nv_bfloat16* out;     // (Tq, H, HD) contiguous
  float* lse;             // (H, Tq)
  int total_q;
  float scale;
  float softcap;          // 0 = none; else scores become softcap * tanh(scale * s / softcap) (Gemma 2)
  int causal;
  int window;             // 0 = unlimited
};

__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Sequence and first row of the `tile`-th tile when every sequence is cut into tiles of `unit` rows.  A whole warp looks
// at 32 sequences at a time (one load and a prefix sum): walking hundreds of short sequences one by one, each step waiting
// for its load, took longer than the tile itself.  Called by full warps; every lane gets the same answer.
__device__ __forceinline__ bool find_tile(const int* cu, int num_seqs, int tile, int unit, int& seq, int& row0) {
  const int lane = threadIdx.x & 31;
  int acc = 0;
  for (int s0 = 0; s0 < num_seqs; s0 += 32) {
    const int s = s0 + lane;
    const int nt = s < num_seqs ? (cu[s + 1] - cu[s] + unit - 1) / unit : 0;
    int upto = nt;                                   // tiles of this group's sequences up to and including the lane's
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned past = __ballot_sync(0xffffffffu, tile < acc + upto);
    if (past != 0) {
      const int src = __ffs(past) - 1;
      seq = s0 + src;
      row0 = (tile - acc - __shfl_sync(0xffffffffu, upto - nt, src)) * unit;
      return true;
    }
    acc += __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}
// Tiles of the first `count` sequences (same warp-wide form).
__device__ __forceinline__ int tiles_before(const int* cu, int count, int unit) {
  int n = 0;
  for (int s = threadIdx.x & 31; s < count; s += 32) n += (cu[s + 1] - cu[s] + unit - 1) / unit;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  return n;
}

// Byte offset of element (row, col) inside a K-major 128B-swizzled tile made of 64-column blocks of `rows` rows.
__device__ __forceinline__ uint32_t sw128_offset(int row, int col, int rows) {
  const int kb = col >> 6, c = col & 63;
  const int chunk = (c >> 3) ^ (row & 7);
  return static_cast<uint32_t>(kb * rows * 128 + row * 128 + chunk * 16 + (c & 7) * 2);
}

template <int HD, bool CAP>
__global__ void __launch_bounds__(FA_THREADS, 1)
fa_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
              const __grid_constant__ CUtensorMap tmV, const FwdParams p) {
  constexpr int KB = HD / 64;                 // 64-column blocks of the head dimension
  constexpr int Q_BYTES = TQ * HD * 2;
  constexpr int KV_BYTES = TK * HD * 2;
  constexpr int P_BYTES = TQ * TK * 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + Q_BYTES;                 // 2 stages
  uint8_t* sV = sK + 2 * KV_BYTES;            // 2 stages
  uint8_t* sP = sV + 2 * KV_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sP + P_BYTES);
  uint64_t* q_full = bars;                    // 1
  uint64_t* k_full = bars + 1;                // 2
  uint64_t* k_empty = bars + 3;               // 2
  uint64_t* v_full = bars + 5;                // 2
  uint64_t* v_empty = bars + 7;               // 2
  uint64_t* s_full = bars + 9;                // 2
  uint64_t* s_empty = bars + 11;              // 2
  uint64_t* p_full = bars + 13;               // 1
  uint64_t* pv_full = bars + 14;              // 1
  uint64_t* pv_empty = bars + 15;             // 1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int head = blockIdx.y;
  const int kvh = head / (p.H / p.KV);
  int seq = 0, q0 = 0;
  const bool live = find_tile(p.cu_q, p.num_seqs, blockIdx.x, TQ, seq, q0);
  if (!live) return;   // uniform for the CTA: nothing allocated yet
  const int qs = p.cu_q[seq], len_q = p.cu_q[seq + 1] - qs;
  const int ks = p.cu_k[seq], len_k = p.cu_k[seq + 1] - ks;
  const int off = len_k - len_q;
  const int rows = min(TQ, len_q - q0);
  int kv_hi = p.causal ? min(len_k, q0 + rows + off) : len_k;
  int kv_lo = (p.causal && p.window > 0) ? max(0, q0 + off - p.window + 1) : 0;
  kv_lo = (kv_lo / TK) * TK;
  const int n_tiles = kv_hi > kv_lo ? (kv_hi - kv_lo + TK - 1) / TK : 0;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&s_empty[i], 4);
    }
    mbar_init(p_full, 4); mbar_init(pv_full, 1); mbar_init(pv_empty, 4);
    fence_barrier_init();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tm_S = tmem_base;            // 2 x 128 columns
  const uint32_t tm_PV = tmem_base + 256;     // HD columns

  if (warp == 0) {
    if (lane == 0 && n_tiles > 0) {
      mbar_expect_tx(q_full, Q_BYTES);
#pragma unroll
      for (int kb = 0; kb < KB; ++kb) tma_load_3d(sQ + kb * (TQ * 128), &tmQ, q_full, kb * 64, head, qs + q0);
      bool ok = true;
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        const int key0 = ks + kv_lo + j * TK;
        if (!(ok = mbar_wait(&k_empty[st], ph ^ 1, abort_flag, 110))) break;
        mbar_expect_tx(&k_full[st], KV_BYTES);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
          tma_load_3d(sK + st * KV_BYTES + kb * (TK * 128), &tmK, &k_full[st], kb * 64, kvh, key0);
        if (!(ok = mbar_wait(&v_empty[st], ph ^ 1, abort_flag, 111))) break;
        mbar_expect_tx(&v_full[st], KV_BYTES);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
          tma_load_3d(sV + st * KV_BYTES + kb * (TK * 128), &tmV, &v_full[st], kb * 64, kvh, key0);
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && n_tiles > 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(TQ, TK, 0, 0);
      constexpr uint32_t idesc_pv = make_idesc_bf16(TQ, HD, 0, 1);
      const uint32_t aQ = smem_u32(sQ), aP = smem_u32(sP);
      bool ok = mbar_wait(q_full, 0, abort_flag, 120);
      auto issue_s = [&](int j) -> bool {
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        if (!mbar_wait(&k_full[st], ph, abort_flag, 121)) return false;
        if (!mbar_wait(&s_empty[st], ph ^ 1, abort_flag, 122)) return false;
        tc_fence_after();
        const uint32_t aK = smem_u32(sK + st * KV_BYTES);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_f16(tm_S + st * TK, make_smem_desc(aQ + kb * (TQ * 128) + kk * 32, 16, 1024),
                     make_smem_desc(aK + kb * (TK * 128) + kk * 32, 16, 1024), idesc_s, (kb | kk) != 0);
        umma_commit(&s_full[st]);
        umma_commit(&k_empty[st]);
        return true;
      };
      if (ok) ok = issue_s(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 1 < n_tiles) {
          if (!(ok = issue_s(j + 1))) break;
        }
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        if (!(ok = mbar_wait(p_full, j & 1, abort_flag, 123))) break;
        if (!(ok = mbar_wait(&v_full[st], ph, abort_flag, 124))) break;
        if (!(ok = mbar_wait(pv_empty, (j & 1) ^ 1, abort_flag, 125))) break;
        tc_fence_after();
        const uint32_t aV = smem_u32(sV + st * KV_BYTES);
#pragma unroll
        for (int s = 0; s < TK / 16; ++s) {
          const uint64_t ad = make_smem_desc(aP + (s >> 2) * (TQ * 128) + (s & 3) * 32, 16, 1024);
          const uint64_t bd = make_smem_desc(aV + s * (16 * 128), TK * 128, 1024);
          umma_f16(tm_PV, ad, bd, idesc_pv, s != 0);
        }
        umma_commit(pv_full);
        umma_commit(&v_empty[st]);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + output
    const int quad = warp & 3;
    const int r = quad * 32 + lane;                 // query row inside the tile
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const float c = p.scale * 1.4426950408889634f;  // scores are kept in log2 units
    constexpr bool capped = CAP;   // soft-cap is a template parameter: the plain path carries no extra work
    const float cap2 = p.softcap * 1.4426950408889634f;            // soft-cap in log2 units
    const float soc = capped ? p.scale / p.softcap : 0.f;
    float m = -INFINITY, l = 0.f, alpha_prev = 0.f;
    float o[HD];
#pragma unroll
    for (int i = 0; i < HD; ++i) o[i] = 0.f;
    const int qi = q0 + r + off;                    // last key this row may see (causal)
    bool ok = true;
    for (int j = 0; j < n_tiles && ok; ++j) {
      const int st = j & 1;
      const uint32_t ph = (j >> 1) & 1;
      const int key0 = kv_lo + j * TK;
      if (!(ok = mbar_wait(&s_full[st], ph, abort_flag, 130))) break;
      tc_fence_after();
      const uint32_t ts = tm_S + st * TK + lane_base;
      // pass 1: row maximum of the masked scores
      float mx = -INFINITY;
#pragma unroll 1
      for (int cb = 0; cb < TK; cb += 32) {
        uint32_t v[32];
        tmem_ld_32x32(ts + cb, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int kj = key0 + cb + i;
          bool keep = kj < len_k;
          if (p.causal) keep = keep && (kj <= qi) && (p.window <= 0 || kj > qi - p.window);
          if (keep) mx = fmaxf(mx, __uint_as_float(v[i]));
        }
      }
      // tanh is monotonic: the capped maximum is the cap of the maximum
      float m_new;
      if constexpr (CAP) m_new = fmaxf(m, mx == -INFINITY ? mx : cap2 * tanh_fast(mx * soc));
      else m_new = fmaxf(m, mx * c);
      const float alpha = (m == -INFINITY) ? 0.f : exp2f(m - m_new);
      // fold the previous tile's P·V into the running output (this also means the P tile is free again)
      if (j > 0) {
        if (!(ok = mbar_wait(pv_full, (j - 1) & 1, abort_flag, 131))) break;
        tc_fence_after();
#pragma unroll
        for (int cb = 0; cb < HD; cb += 32) {
          uint32_t v[32];
          tmem_ld_32x32(tm_PV + lane_base + cb, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[cb + i] = o[cb + i] * alpha_prev + __uint_as_float(v[i]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(pv_empty);
      }
      // pass 2: probabilities -> bf16 -> swizzled shared tile; row sum
      float sum = 0.f;
      const float mref = (m_new == -INFINITY) ? 0.f : m_new;
#pragma unroll 1
      for (int cb = 0; cb < TK; cb += 32) {
        uint32_t v[32];
        tmem_ld_32x32(ts + cb, v);
        tmem_ld_wait();
        float pr[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int kj = key0 + cb + i;
          bool keep = kj < len_k;
          if (p.causal) keep = keep && (kj <= qi) && (p.window <= 0 || kj > qi - p.window);
          // two textually separate forms: the plain one must stay a single multiply-add feeding the exponential
          if constexpr (CAP) pr[i] = keep ? exp2f(cap2 * tanh_fast(__uint_as_float(v[i]) * soc) - mref) : 0.f;
          else pr[i] = keep ? exp2f(__uint_as_float(v[i]) * c - mref) : 0.f;
          sum += pr[i];
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint4 pk;
          __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
          for (int e = 0; e < 4; ++e) h2[e] = __floats2bfloat162_rn(pr[g * 8 + 2 * e], pr[g * 8 + 2 * e + 1]);
          *reinterpret_cast<uint4*>(sP + sw128_offset(r, cb + g * 8, TQ)) = pk;
        }
      }
      l = l * alpha + sum;
      m = m_new;
      alpha_prev = alpha;
      tc_fence_before();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&s_empty[st]);
        mbar_arrive(p_full);
      }
    }
    if (ok && n_tiles > 0) {
      if (mbar_wait(pv_full, (n_tiles - 1) & 1, abort_flag, 132)) {
        tc_fence_after();
#pragma unroll
        for (int cb = 0; cb < HD; cb += 32) {
          uint32_t v[32];
          tmem_ld_32x32(tm_PV + lane_base + cb, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[cb + i] = o[cb + i] * alpha_prev + __uint_as_float(v[i]);
        }
      }
    }
    if (r < rows) {
      const float inv = l > 0.f ? 1.f / l : 0.f;
      const size_t row = static_cast<size_t>(qs + q0 + r);
      __nv_bfloat16* dst = p.out + (row * p.H + head) * HD;
#pragma unroll
      for (int i = 0; i < HD; i += 8) {
        uint4 pk;
        __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
        for (int e = 0; e < 4; ++e) h2[e] = __floats2bfloat162_rn(o[i + 2 * e] * inv, o[i + 2 * e + 1] * inv);
        *reinterpret_cast<uint4*>(dst + i) = pk;
      }
      // natural-log LSE of the scaled scores
      p.lse[static_cast<size_t>(head) * p.total_q + row] = (l > 0.f) ? (m + log2f(l)) * 0.6931471805599453f : -INFINITY;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}


// =====================================================================================================
// Forward, two query tiles per CTA (the default).  A CTA owns 256 consecutive query rows of one head as two 128-row
// tiles that share every K / V tile (half the K / V traffic of one tile per CTA) and run in ping-pong: while the four
// softmax warps of one tile work on their scores, the tensor core computes the other tile's S = Q·Kᵀ or O += P·V.
//   warps 0-3   softmax of tile 0        warps 4-7   softmax of tile 1
//   warp 8      TMA producer (Q tiles once, K / V through two-stage rings, no multicast)
//   warp 9      MMA issuer
// Tensor memory: S0 | S1 | O0 | O1 (4 x 128 columns).  The probabilities never touch shared memory: a softmax thread
// writes its row of P as packed bf16 over the first 64 columns of its S (tcgen05.st; the write position trails the
// read position of the second pass) and the P·V MMA takes its A operand from tensor memory.  O accumulates in tensor
// memory across the K / V tiles; it is rescaled only when a row maximum has grown by more than 2^8 since the last
// rescale (the probabilities are computed against that stale maximum, so they stay below 2^8 and the final division
// by the row sum is exact), which for real score distributions happens on the first tiles of a row only.
// =====================================================================================================
constexpr int FA2_THREADS = 320;
constexpr float FA2_RESCALE_LOG2 = 8.0f;

template <int HD, bool CAP>
__global__ void __launch_bounds__(FA2_THREADS, 1)
fa_fwd2_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
               const __grid_constant__ CUtensorMap tmV, const FwdParams p) {
  constexpr int KB = HD / 64;
  constexpr int Q_BYTES = TQ * HD * 2;
  constexpr int KV_BYTES = TK * HD * 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                         // 2 tiles
  uint8_t* sK = sQ + 2 * Q_BYTES;             // 2 stages
  uint8_t* sV = sK + 2 * KV_BYTES;            // 2 stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + 2 * KV_BYTES);
  uint64_t* q_full = bars;                    // 1
  uint64_t* k_full = bars + 1;                // 2
  uint64_t* k_empty = bars + 3;               // 2
  uint64_t* v_full = bars + 5;                // 2
  uint64_t* v_empty = bars + 7;               // 2
  uint64_t* s_full = bars + 9;                // 2 (per query tile)
  uint64_t* p_full = bars + 11;               // 2
  uint64_t* o_full = bars + 13;               // 2
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int head = blockIdx.y;
  const int kvh = head / (p.H / p.KV);
  int seq = 0, q0 = 0;
  // Blocks are handed out in increasing blockIdx; walking the tiles backwards puts the late query blocks of a sequence
  // (the ones with the most K / V tiles under a causal mask) first and leaves the short ones for the tail of the grid.
  if (!find_tile(p.cu_q, p.num_seqs, static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x), 2 * TQ, seq, q0))
    return;                                                            // uniform for the CTA: nothing allocated yet
  const int qs = p.cu_q[seq], len_q = p.cu_q[seq + 1] - qs;
  const int ks = p.cu_k[seq], len_k = p.cu_k[seq + 1] - ks;
  const int off = len_k - len_q;
  int kv_lo = (p.causal && p.window > 0) ? max(0, q0 + off - p.window + 1) : 0;
  kv_lo = (kv_lo / TK) * TK;
  // per query tile: live rows and K / V tiles it has to visit (scalars: no indexed local arrays)
  const int rows0 = max(0, min(TQ, len_q - q0)), rows1 = max(0, min(TQ, len_q - q0 - TQ));
  const int hi0 = rows0 == 0 ? 0 : (p.causal ? min(len_k, q0 + rows0 + off) : len_k);
  const int hi1 = rows1 == 0 ? 0 : (p.causal ? min(len_k, q0 + TQ + rows1 + off) : len_k);
  const int nt0 = hi0 > kv_lo ? (hi0 - kv_lo + TK - 1) / TK : 0;
  const int nt1 = hi1 > kv_lo ? (hi1 - kv_lo + TK - 1) / TK : 0;
  const int n_max = max(nt0, nt1);

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); mbar_init(&o_full[i], 1);
    }
    fence_barrier_init();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 8) {
    // ------------------------------------------------------------------------- TMA producer
    if (lane == 0 && n_max > 0) {
      const int nq = rows1 > 0 ? 2 : 1;
      mbar_expect_tx(q_full, nq * Q_BYTES);
      for (int t = 0; t < nq; ++t)
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
          tma_load_3d(sQ + t * Q_BYTES + kb * (TQ * 128), &tmQ, q_full, kb * 64, head, qs + q0 + t * TQ);
      bool ok = true;
      for (int j = 0; j < n_max && ok; ++j) {
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        const int key0 = ks + kv_lo + j * TK;
        if (!(ok = mbar_wait(&k_empty[st], ph ^ 1, abort_flag, 140))) break;
        mbar_expect_tx(&k_full[st], KV_BYTES);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
          tma_load_3d(sK + st * KV_BYTES + kb * (TK * 128), &tmK, &k_full[st], kb * 64, kvh, key0);
        if (!(ok = mbar_wait(&v_empty[st], ph ^ 1, abort_flag, 141))) break;
        mbar_expect_tx(&v_full[st], KV_BYTES);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
          tma_load_3d(sV + st * KV_BYTES + kb * (TK * 128), &tmV, &v_full[st], kb * 64, kvh, key0);
      }
    }
  } else if (warp == 9) {
    // --------------------------------------------------------------------------- MMA issuer
    if (lane == 0 && n_max > 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(TQ, TK, 0, 0);
      constexpr uint32_t idesc_pv = make_idesc_bf16(TQ, HD, 0, 1);
      bool ok = mbar_wait(q_full, 0, abort_flag, 150);
      // S_t(j) = Q_t · K_jᵀ into the tile's score columns (they are free: the tile's P·V of j-1 was issued before)
      const uint64_t dQ = make_smem_desc(smem_u32(sQ), 16, 1024), dK = make_smem_desc(smem_u32(sK), 16, 1024);
      const uint64_t dV = make_smem_desc(smem_u32(sV), TK * 128, 1024);
      auto issue_s = [&](int t, int j) {
        const uint64_t dq = dQ + t * (Q_BYTES >> 4), dk = dK + (j & 1) * (KV_BYTES >> 4);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_f16(tmem_base + t * TK, dq + (kb * (TQ * 128) + kk * 32 >> 4), dk + (kb * (TK * 128) + kk * 32 >> 4), idesc_s,
                     (kb | kk) != 0);
        umma_commit(&s_full[t]);
      };
      if (ok) ok = mbar_wait(&k_full[0], 0, abort_flag, 151);
      if (ok) {
        tc_fence_after();
        if (nt0 > 0) issue_s(0, 0);
        if (nt1 > 0) issue_s(1, 0);
        umma_commit(&k_empty[0]);
      }
      for (int j = 0; j < n_max && ok; ++j) {
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        const bool more = j + 1 < n_max;
        if (!(ok = mbar_wait(&v_full[st], ph, abort_flag, 152))) break;
        if (more && !(ok = mbar_wait(&k_full[st ^ 1], ((j + 1) >> 1) & 1, abort_flag, 153))) break;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int nt = t ? nt1 : nt0;
          if (!ok || j >= nt) continue;
          if (!(ok = mbar_wait(&p_full[t], j & 1, abort_flag, 154 + t))) break;
          tc_fence_after();
          const uint64_t dv = dV + st * (KV_BYTES >> 4);
#pragma unroll
          for (int s2 = 0; s2 < TK / 16; ++s2)       // P (tensor memory, 8 columns per 16 keys) times V
            umma_f16_ts(tmem_base + 256 + t * HD, tmem_base + t * TK + s2 * 8, dv + s2 * (16 * 128 >> 4), idesc_pv,
                        s2 == 0 ? j != 0 : 1);
          umma_commit(&o_full[t]);
          if (j + 1 < nt) issue_s(t, j + 1);
        }
        if (!ok) break;
        umma_commit(&v_empty[st]);
        if (more) umma_commit(&k_empty[st ^ 1]);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + output of tile t
    const int t = warp >> 2;
    const int quad = warp & 3;
    const int r = quad * 32 + lane;                 // query row inside the tile
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t tm_S = tmem_base + t * TK + lane_base;
    const uint32_t tm_O = tmem_base + 256 + t * HD + lane_base;
    const float c = p.scale * 1.4426950408889634f;  // scores are kept in log2 units
    const float cap2 = p.softcap * 1.4426950408889634f;
    const float soc = CAP ? p.scale / p.softcap : 0.f;
    const int n_tiles = t ? nt1 : nt0;
    const int rows = t ? rows1 : rows0;
    const int tq0 = q0 + t * TQ;
    const int qi = tq0 + r + off;                   // last key this row may see (causal)
    float m = -INFINITY, l = 0.f;                   // m: the maximum the probabilities are currently scaled against
    bool ok = true;
    for (int j = 0; j < n_tiles && ok; ++j) {
      const int key0 = kv_lo + j * TK;
      if (!(ok = mbar_wait(&s_full[t], j & 1, abort_flag, 160 + t))) break;
      tc_fence_after();
      // The whole score row of this tile goes into registers with one wait (four loads in flight), so tensor memory
      // is read once.  Only tiles that cross the causal diagonal, the window edge or the end of the keys pay for
      // masking (a masked score becomes -inf, whose exponential is 0); interior tiles run the bare
      // max / multiply-add / exp2 / pack stream.
      uint32_t sv[4][32];
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) tmem_ld_32x32(tm_S + q4 * 32, sv[q4]);
      tmem_ld_wait();
      const bool edge = (key0 + TK > len_k) ||
                        (p.causal && (key0 + TK - 1 > tq0 + off || (p.window > 0 && key0 <= tq0 + TQ - 1 + off - p.window)));
      if (edge) {
        // visible columns of this row inside the tile: [lo, hi] (one subtract and one unsigned compare per element)
        const int hi = (p.causal ? min(len_k - 1, qi) : len_k - 1) - key0;
        const int lo = (p.causal && p.window > 0) ? max(0, qi - p.window + 1 - key0) : 0;
        const unsigned span = hi >= lo ? static_cast<unsigned>(hi - lo) : 0u;
        const bool none = hi < lo;
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (none || static_cast<unsigned>(q4 * 32 + i - lo) > span) sv[q4][i] = 0xff800000u;   // -inf
      }
      float mx4[4];
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) {
        float a = __uint_as_float(sv[q4][0]);
#pragma unroll
        for (int i = 1; i < 32; ++i) a = fmaxf(a, __uint_as_float(sv[q4][i]));
        mx4[q4] = a;
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      float m_new;
      if constexpr (CAP) m_new = fmaxf(m, mx == -INFINITY ? mx : cap2 * tanh_fast(mx * soc));
      else m_new = fmaxf(m, mx * c);
      if (j == 0) {
        m = m_new;
      } else {
        const bool grow = m_new > m + FA2_RESCALE_LOG2;
        if (__any_sync(0xffffffffu, grow)) {
          // the tile's previous P·V must have landed before its output rows are rescaled in tensor memory
          if (!(ok = mbar_wait(&o_full[t], (j - 1) & 1, abort_flag, 162 + t))) break;
          tc_fence_after();
          const float alpha = grow ? exp2f(m - m_new) : 1.f;
#pragma unroll 1
          for (int cb = 0; cb < HD; cb += 32) {
            uint32_t v[32];
            tmem_ld_32x32(tm_O + cb, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
            tmem_st_32x32(tm_O + cb, v);
          }
          tmem_st_wait();
          l *= alpha;
          if (grow) m = m_new;
        }
      }
      // probabilities against m -> packed bf16 over the first half of this tile's S columns; row sum
      const float mref = (m == -INFINITY) ? 0.f : m;
      float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float p0, p1;
          // two textually separate forms: the plain one must stay a single multiply-add feeding the exponential
          if constexpr (CAP) {
            const float s0 = __uint_as_float(sv[q4][i]), s1 = __uint_as_float(sv[q4][i + 1]);
            p0 = s0 == -INFINITY ? 0.f : exp2f(cap2 * tanh_fast(s0 * soc) - mref);
            p1 = s1 == -INFINITY ? 0.f : exp2f(cap2 * tanh_fast(s1 * soc) - mref);
          } else {
            p0 = exp2f(__uint_as_float(sv[q4][i]) * c - mref);
            p1 = exp2f(__uint_as_float(sv[q4][i + 1]) * c - mref);
          }
          sum4[q4] += p0 + p1;
          const __nv_bfloat162 h2 = __floats2bfloat162_rn(p0, p1);
          pk[i >> 1] = *reinterpret_cast<const uint32_t*>(&h2);
        }
        tmem_st_32x16(tm_S + q4 * 16, pk);
      }
      const float sum = (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
      l += sum;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[t]);
    }
    if (ok && n_tiles > 0 && mbar_wait(&o_full[t], (n_tiles - 1) & 1, abort_flag, 164 + t)) {
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      const size_t row = static_cast<size_t>(qs + tq0 + min(r, max(rows - 1, 0)));
      __nv_bfloat16* dst = p.out + (row * p.H + head) * HD;
#pragma unroll 1
      for (int cb = 0; cb < HD; cb += 32) {
        uint32_t v[32];
        tmem_ld_32x32(tm_O + cb, v);
        tmem_ld_wait();
        if (r < rows) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 o4;
            __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&o4);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              h2[e] = __floats2bfloat162_rn(__uint_as_float(v[i + 2 * e]) * inv, __uint_as_float(v[i + 2 * e + 1]) * inv);
            *reinterpret_cast<uint4*>(dst + cb + i) = o4;
          }
        }
      }
      // natural-log LSE of the scaled scores
      if (r < rows)
        p.lse[static_cast<size_t>(head) * p.total_q + row] = (l > 0.f) ? (m + log2f(l)) * 0.6931471805599453f : -INFINITY;
    } else if (n_tiles == 0 && r < rows) {
      // no visible key at all (cannot happen with causal bottom-right alignment, kept for completeness)
      const size_t row = static_cast<size_t>(qs + tq0 + r);
      __nv_bfloat16* dst = p.out + (row * p.H + head) * HD;
      for (int i = 0; i < HD; i += 8) *reinterpret_cast<uint4*>(dst + i) = make_uint4(0, 0, 0, 0);
      p.lse[static_cast<size_t>(head) * p.total_q + row] = -INFINITY;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// (rows, heads, hd) bf16 tensor with token stride `row_stride` elements; box = 64 x 1 x box_rows.
static int make_tmap_3d(CUtensorMap* out, const void* base, int hd, int heads, long rows, long row_stride,
                        int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return -100;
  cuuint64_t gdim[3] = {(cuuint64_t)hd, (cuuint64_t)heads, (cuuint64_t)rows};
  cuuint64_t gstr[2] = {(cuuint64_t)hd * 2, (cuuint64_t)row_stride * 2};
  cuuint32_t box[3] = {64, 1, (cuuint32_t)box_rows};
  cuuint32_t es[3] = {1, 1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), gdim, gstr, box, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -200 - static_cast<int>(r);
}

template <int HD, bool CAP>
static int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& p,
                      int tiles, cudaStream_t s) {
  constexpr int SMEM = TQ * HD * 2 + 4 * TK * HD * 2 + TQ * TK * 2 + 256 + 1024;
  auto kern = fa_fwd_kernel<HD, CAP>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return -300 - static_cast<int>(e);
    configured = true;
  }
  dim3 grid(tiles, p.H);
  kern<<<grid, FA_THREADS, SMEM, s>>>(tq, tk, tv, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -400 - static_cast<int>(e);
}

template <int HD, bool CAP>
static int launch_fwd2(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& p,
                       int tiles, cudaStream_t s) {
  constexpr int SMEM = 2 * TQ * HD * 2 + 4 * TK * HD * 2 + 256 + 1024;
  auto kern = fa_fwd2_kernel<HD, CAP>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return -300 - static_cast<int>(e);
    configured = true;
  }
  dim3 grid(tiles, p.H);
  kern<<<grid, FA2_THREADS, SMEM, s>>>(tq, tk, tv, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -400 - static_cast<int>(e);
}

}  // namespace ftb

using namespace ftb;

static int g_fwd_two_tiles = 1;     // ftb_attn_set_two_tiles(0) selects the one-tile-per-CTA forward kernel

extern "C" {

void ftb_attn_set_two_tiles(int on) { g_fwd_two_tiles = on; }

// q (Tq, H, hd), k / v (Tk, KV, hd) bf16 with token strides (elements) q_stride / k_stride / v_stride;
// out (Tq, H, hd) contiguous; lse (H, Tq) fp32. cu_q / cu_k: device int32 (num_seqs + 1).
// max_tiles >= sum over sequences of ceil(len_q / 128); Tq / 128 + num_seqs always suffices.
int ftb_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse, const int* cu_q, const int* cu_k,
                 int num_seqs, int total_q, int total_k, int H, int KV, int hd, long q_stride, long k_stride,
                 long v_stride, float scale, float softcap, int causal, int window, int max_tiles,
                 cudaStream_t stream) {
  if (total_q <= 0 || num_seqs <= 0) return 0;
  if ((hd != 64 && hd != 128) || H % KV) return -2;
  if ((q_stride & 7) || (k_stride & 7) || (v_stride & 7)) return -2;
  CUtensorMap tq, tk, tv;
  int rc = make_tmap_3d(&tq, q, hd, H, total_q, q_stride, TQ);
  if (rc) return rc;
  rc = make_tmap_3d(&tk, k, hd, KV, total_k, k_stride, TK);
  if (rc) return rc;
  rc = make_tmap_3d(&tv, v, hd, KV, total_k, v_stride, TK);
  if (rc) return rc;
  FwdParams p;
  p.cu_q = cu_q; p.cu_k = cu_k; p.num_seqs = num_seqs; p.H = H; p.KV = KV;
  p.out = reinterpret_cast<__nv_bfloat16*>(out); p.lse = lse; p.total_q = total_q;
  p.scale = scale; p.softcap = softcap; p.causal = causal; p.window = window;
  if (g_fwd_two_tiles) {
    const int tiles2 = (total_q + 2 * TQ - 1) / (2 * TQ) + num_seqs;   // >= sum over sequences of ceil(len_q / 256)
    if (softcap > 0.f)
      return hd == 128 ? launch_fwd2<128, true>(tq, tk, tv, p, tiles2, stream)
                       : launch_fwd2<64, true>(tq, tk, tv, p, tiles2, stream);
    return hd == 128 ? launch_fwd2<128, false>(tq, tk, tv, p, tiles2, stream)
                     : launch_fwd2<64, false>(tq, tk, tv, p, tiles2, stream);
  }
  if (softcap > 0.f)
    return hd == 128 ? launch_fwd<128, true>(tq, tk, tv, p, max_tiles, stream)
                     : launch_fwd<64, true>(tq, tk, tv, p, max_tiles, stream);
  return hd == 128 ? launch_fwd<128, false>(tq, tk, tv, p, max_tiles, stream)
                   : launch_fwd<64, false>(tq, tk, tv, p, max_tiles, stream);
}

int ftb_attn_error(void) {
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

}  // extern "C"

static int g_dq_bulk = 1;     // ftb_attn_set_dq_bulk(0): per-thread vector reductions (the earlier drain), for A/B runs

// =====================================================================================================
// Backward
// =====================================================================================================
namespace ftb {

// Orders of the backward's work.  A CTA that adds to a query tile in a fixed order may only wait for CTAs that were handed
// out before it (one that waited for a later CTA could fill the GPU with waiters and starve it), and should come to the
// tile after them by itself.
//   FIRST_FIRST  key tiles ascending (the causal ones with the most query tiles first, so the short ones fill the end of
//                the grid), head by head, query tiles ascending.  For dQ added in any order.
//   LAST_FIRST   key tiles descending, head by head, query tiles ascending: every key tile starts at its own diagonal and
//                so comes to a query tile one step after the key tile above it.  But the longest CTAs come last.
//   IN_STEP      key tiles ascending, query tiles descending with the heads of the group inside: all key tiles of a
//                sequence walk the same (query tile, head) list in step, the short ones leave it early.  The longest CTAs
//                come first; the price is a wait per key tile at the start and additions that meet at the same addresses.
// With a fixed order, LAST_FIRST against IN_STEP, causal, us of this kernel, all taken in turn on one GPU.  Head dim 128,
// 32 / 8 heads: 16 x 1024 tokens 609 / 636, 4 x 4096 2041 / 1940, 2 x 8192 4347 / 3607, 1 x 16384 9013 / 7018; 16 / 8 heads:
// 4 x 4096 1043 / 1054, 2 x 8192 1967 / 1925, 1 x 16384 4272 / 3635; 16 / 16 heads: 4 x 4096 1030 / 1154, 2 x 8192 1927 / 2037,
// 1 x 16384 4175 / 3765.  Head dim 64, 32 / 8 heads: 16 x 1024 468 / 462, 8 x 2048 810 / 756, 1 x 16384 5810 / 4866; 16 / 16
// heads: 16 x 1024 291 / 311, 8 x 2048 453 / 471, 2 x 8192 1399 / 1403.  The more heads share a key, the earlier IN_STEP wins; it
// is taken where the longest sequence has more than 4096 keys (1024 at head dim 64, whose tile pairs are shorter), where the two
// differ by 5 to 7 % either way.
constexpr int BWD_FIRST_FIRST = 0, BWD_LAST_FIRST = 1, BWD_IN_STEP = 2;

struct BwdParams {
  const int* cu_q;
  const int* cu_k;
  int num_seqs;
  int H, KV;
  float* dq_acc;            // (Tq, H, HD) fp32, zero-initialised by the caller
  int* dq_sem;              // deterministic mode: a flag and one counter per (query tile, head, 32 rows), zeroed; else NULL
  int order;                // BWD_*: the order of the key tiles over the grid and of the query tiles in a CTA
  int dq_bulk;              // 1: dQ tiles leave through shared memory as tiled reduce-adds; 0: per-thread vector reductions
  __nv_bfloat16* dk;        // (Tk, KV, HD) contiguous
  __nv_bfloat16* dv;
  const float* lse;         // (H, Tq)
  const float* delta;       // (H, Tq)  rowsum(dO * O)
  int total_q;
  float scale;
  float softcap;
  int causal;
  int window;
};

// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d]; hd / 8 lanes per (t, h), each with one 16-byte load of either tensor.
// Bound by memory; 16384 x 32 heads of 128: 110 us (2.4 TB/s) with a warp per row and 4-byte loads, 54 us (5.0 TB/s)
// so.
template <int HD>
__global__ void fa_delta_kernel(const __nv_bfloat16* __restrict__ dout, long do_stride, const __nv_bfloat16* __restrict__ out,
                                long o_stride, float* __restrict__ delta, int T, int H) {
  constexpr int LANES = HD / 8;
  const long w = ((long)blockIdx.x * blockDim.x + threadIdx.x) / LANES;
  const int part = threadIdx.x % LANES;
  if (w >= (long)T * H) return;                     // whole groups of LANES lanes leave together
  const int t = (int)(w / H), h = (int)(w % H);
  const uint4 a = __ldg(reinterpret_cast<const uint4*>(dout + (size_t)t * do_stride + (size_t)h * HD) + part);
  const uint4 b = __ldg(reinterpret_cast<const uint4*>(out + (size_t)t * o_stride + (size_t)h * HD) + part);
  const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&a);
  const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&b);
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 x = __bfloat1622float2(a2[i]), y = __bfloat1622float2(b2[i]);
    s += x.x * y.x + x.y * y.y;
  }
  const unsigned mask = ((1u << LANES) - 1u) << ((threadIdx.x & 31) / LANES * LANES);
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_xor_sync(mask, s, o);
  if (part == 0) delta[(size_t)h * T + t] = s;
}

// Backward thread layout: warps 0-7 softmax, warps 8-11 dQ drain, warp 12 loads, warp 13 MMA.
//
// Scores are formed transposed (Sᵀ = K·Qᵀ, dPᵀ = V·dOᵀ; one key row per thread), so that Pᵀ goes back into tensor memory
// as packed bf16 over the score columns it came from and is the A operand of dV += Pᵀ·dO without touching shared memory.
// dSᵀ is one shared tile that feeds dK += dSᵀ·Q (K-major) and dQ = dS·K (M-major).  The MMAs are issued one query tile
// ahead:
//     ... dQ(j) S(j+1) dK(j) | dP(j+1) dV(j+1) | dQ(j+1) S(j+2) dK(j+1) ...
// P(j+1) is computed under dK(j) and dP(j+1); dS(j+1) under dV(j+1); the dQ tile is emptied by warps of its own under
// S(j+1) and dK(j), and leaves under what follows; Q(j+2) takes the place of Q(j) and has dP, dV and dQ of j+1 to arrive.
// At head dim 128 the tensor memory is full (S, dP, dV, dK) and dQ(j) takes dP(j)'s columns, which the softmax warps have
// read by then; dP(j+1) waits until they are empty.
// Two softmax warps share a tensor-memory lane quadrant (rows) and split the 128 query columns.
//
// In the transposed scores a query's lse and delta belong to a column, the same for all 32 lanes: read from shared memory
// they cost a pass of its pipe per warp and column, 1500 cycles a tile pair, half of them in the chain.  Instead the tensor
// core subtracts them: one more step of 16 in the reduction, whose A rows are (1, 1, 1, 0 ...) and whose B rows hold
// -lse / scale (or -delta) as the sum of three bf16 (24 bits, as exact as the fp32 value).
// Causal, 32 / 8 heads of 128, dQ in any order: 16 x 1024 tokens 771 us with one chain S, dP -> softmax -> dV, dK, dQ ->
// drain per tile pair, 514 us so; 1 x 16384 9160 us (600 TFLOP/s) before, 5710 us (963) so.  With dQ in a fixed order 926 ->
// 609 us and 12300 -> 7018 us.
constexpr int FAB_THREADS = 448;
constexpr int FAB_SOFTMAX_WARPS = 8;

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// One answer for the whole warp: its lanes go on together or leave their loops together.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int where) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, where));
}

// A 128 x 16 bf16 operand (K-major, 32-byte swizzle): row r is 32 bytes, its two 16-byte halves swapped in every other
// group of four rows; eight rows (256 bytes) repeat.
constexpr int AUG_BYTES = 128 * 32;
__device__ __forceinline__ uint64_t make_aug_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(1) << 16;            // LBO: not used, one atom wide
  d |= static_cast<uint64_t>(256 >> 4) << 32;     // SBO: eight rows
  d |= static_cast<uint64_t>(1) << 46;            // descriptor version (Blackwell)
  d |= static_cast<uint64_t>(6) << 61;            // SWIZZLE_32B
  return d;
}
__device__ __forceinline__ void write_aug_row(uint8_t* tile, int row, float v) {
  const __nv_bfloat16 hi = __float2bfloat16(v);
  float rest = v - __bfloat162float(hi);
  if (!isfinite(v)) rest = 0.f;                   // an infinite or undefined value stands alone
  const __nv_bfloat16 mid = __float2bfloat16(rest);
  const __nv_bfloat16 lo = __float2bfloat16(rest - __bfloat162float(mid));
  const __nv_bfloat162 a = __halves2bfloat162(hi, mid), b = __halves2bfloat162(lo, __float2bfloat16(0.f));
  const int swap = (row >> 2) & 1;
  *reinterpret_cast<uint4*>(tile + row * 32 + swap * 16) =
      make_uint4(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b), 0u, 0u);
  *reinterpret_cast<uint4*>(tile + row * 32 + (swap ^ 1) * 16) = make_uint4(0u, 0u, 0u, 0u);
}

template <int HD>
struct BwdSmem {
  static constexpr int T_BYTES = 128 * HD * 2;       // one Q / dO / K / V tile
  static constexpr int DS_BYTES = 128 * 128 * 2;
  static constexpr int STAGE_BYTES = 32 * 32 * 4;    // 32 rows x 32 fp32 columns of dQ; STAGES of them per drain warp
  static constexpr int STAGES = HD == 128 ? 1 : 2;
  static constexpr int USED = 5 * T_BYTES + DS_BYTES + 4 * STAGES * STAGE_BYTES + 3 * AUG_BYTES + 256;
  static constexpr int SIZE = USED + 1024 < 232448 ? USED + 1024 : 232448;      // the 227 KB a CTA may have
};

template <int HD, bool CAP>
__global__ void __launch_bounds__(FAB_THREADS, 1)
fa_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
              const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
              const __grid_constant__ CUtensorMap tmDQ, const BwdParams p) {
  using L = BwdSmem<HD>;
  constexpr int KB = HD / 64;
  constexpr int T_BYTES = L::T_BYTES;
  constexpr bool DQ_OVER_DP = HD == 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + T_BYTES;
  uint8_t* sQ = sV + T_BYTES;                 // 2 stages
  uint8_t* sDO = sQ + 2 * T_BYTES;
  uint8_t* sDS = sDO + T_BYTES;
  uint8_t* sStg = sDS + L::DS_BYTES;          // dQ staging
  uint8_t* sOnes = sStg + 4 * L::STAGES * L::STAGE_BYTES;
  uint8_t* sLse = sOnes + AUG_BYTES;                        // -lse / scale of the query tile
  uint8_t* sDelta = sLse + AUG_BYTES;                       // -delta
  float* sStat = reinterpret_cast<float*>(sLse);            // with soft-cap instead: [stage][128] lse in log2 units
  uint64_t* bars = reinterpret_cast<uint64_t*>(sDelta + AUG_BYTES);
  uint64_t* kv_full = bars;
  uint64_t* q_full = bars + 1;                // 2
  uint64_t* q_empty = bars + 3;               // 2
  uint64_t* do_full = bars + 5;
  uint64_t* do_empty = bars + 6;
  uint64_t* lse_full = bars + 7;              // 2
  uint64_t* s_full = bars + 9;
  uint64_t* p_full = bars + 10;
  uint64_t* dp_full = bars + 11;
  uint64_t* ds_full = bars + 12;
  uint64_t* dq_full = bars + 13;
  uint64_t* dq_empty = bars + 14;
  uint64_t* acc_full = bars + 15;
  uint64_t* delta_full = bars + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  if (smem + L::USED > smem_raw + L::SIZE) {  // the base of the block's shared memory is aligned in practice
    set_error(5, 241);
    return;
  }

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = blockIdx.x % p.KV;
  const int rep = p.H / p.KV;
  int seq = 0, k0 = 0;
  // Blocks are handed out in increasing blockIdx: all heads of a key tile, then the next key tile; see BWD_*.  (One grid
  // dimension for both: the second one ends at 65535, fewer than the key tiles of a batch of very many sequences.)
  const int tile = static_cast<int>(p.order == BWD_LAST_FIRST ? gridDim.x - 1 - blockIdx.x : blockIdx.x) / p.KV;
  if (!find_tile(p.cu_k, p.num_seqs, tile, TK, seq, k0)) return;
  const int qs = p.cu_q[seq], len_q = p.cu_q[seq + 1] - qs;
  const int ks = p.cu_k[seq], len_k = p.cu_k[seq + 1] - ks;
  const int off = len_k - len_q;
  const int kr = min(128, len_k - k0);
  int i_lo = p.causal ? max(0, k0 - off) : 0;
  int i_hi = (p.causal && p.window > 0) ? min(len_q, k0 + kr + p.window - 1 - off) : len_q;
  i_lo = (i_lo / 128) * 128;
  const int n_qt = i_hi > i_lo ? (i_hi - i_lo + 127) / 128 : 0;
  const int n_iter = n_qt * rep;
  const bool in_step = p.order == BWD_IN_STEP;
  const int qt_first = in_step ? i_lo + (n_qt - 1) * 128 : i_lo;
  auto next_tile = [&](int& h, int& qt) {
    if (in_step) {
      if (++h == (kvh + 1) * rep) { h = kvh * rep; qt -= 128; }
    } else {
      qt += 128;
      if (qt == i_lo + n_qt * 128) { qt = i_lo; ++h; }
    }
  };

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(kv_full, 1); mbar_init(do_full, 1); mbar_init(do_empty, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); mbar_init(&lse_full[i], 1); }
    mbar_init(delta_full, 1);
    mbar_init(s_full, 1); mbar_init(p_full, FAB_SOFTMAX_WARPS); mbar_init(dp_full, 1);
    mbar_init(ds_full, FAB_SOFTMAX_WARPS); mbar_init(dq_full, 1); mbar_init(dq_empty, 4); mbar_init(acc_full, 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmDO); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
  }
  if (warp == 13) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (threadIdx.x < 128) {                    // the constant A rows (1, 1, 1, 0 ...)
    const int swap = (threadIdx.x >> 2) & 1;
    *reinterpret_cast<uint4*>(sOnes + threadIdx.x * 32 + swap * 16) = make_uint4(0x3f803f80u, 0x00003f80u, 0u, 0u);
    *reinterpret_cast<uint4*>(sOnes + threadIdx.x * 32 + (swap ^ 1) * 16) = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tm_S = tmem_base, tm_dP = tmem_base + 128, tm_dV = tmem_base + 256, tm_dK = tmem_base + 256 + HD;
  const uint32_t tm_dQ = DQ_OVER_DP ? tm_dP : tmem_base + 256 + 2 * HD;

  if (warp == 12) {
    // ------------------------------------------------------------------------- loads
    if (lane == 0 && n_iter > 0) {
      mbar_expect_tx(kv_full, 2 * T_BYTES);
#pragma unroll
      for (int kb = 0; kb < KB; ++kb) {
        tma_load_3d(sK + kb * (128 * 128), &tmK, kv_full, kb * 64, kvh, ks + k0);
        tma_load_3d(sV + kb * (128 * 128), &tmV, kv_full, kb * 64, kvh, ks + k0);
      }
    }
    const float inv_scale = 1.f / p.scale;
    int h = kvh * rep, qt = qt_first;
    for (int it = 0; it < n_iter; ++it) {
      const int st = it & 1;
      float l[4], dl[4];
      const size_t base = static_cast<size_t>(h) * p.total_q + qs + qt;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const bool vq = qt + e * 32 + lane < len_q;
        l[e] = vq ? p.lse[base + e * 32 + lane] : -INFINITY;
        dl[e] = vq ? p.delta[base + e * 32 + lane] : 0.f;
      }
      // the stage's last tenant has been through its dK product
      if (!mbar_wait_warp(&q_empty[st], ((it >> 1) & 1) ^ 1, abort_flag, 210)) break;
      if (lane == 0) {
        mbar_expect_tx(&q_full[st], T_BYTES);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
          tma_load_3d(sQ + st * T_BYTES + kb * (128 * 128), &tmQ, &q_full[st], kb * 64, h, qs + qt);
      }
      if constexpr (CAP) {
#pragma unroll
        for (int e = 0; e < 4; ++e)            // a query past the end, or one that sees no key: P = 0
          sStat[st * 128 + e * 32 + lane] = l[e] == -INFINITY ? INFINITY : l[e] * 1.4426950408889634f;
      } else {
        if (it > 0 && !mbar_wait_warp(s_full, (it - 1) & 1, abort_flag, 212)) break;     // S of the last tile has read it
#pragma unroll
        for (int e = 0; e < 4; ++e)
          write_aug_row(sLse, e * 32 + lane, l[e] == -INFINITY ? copysignf(1e30f, -p.scale) : -l[e] * inv_scale);
        fence_proxy_async();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&lse_full[st]);
      if (!mbar_wait_warp(do_empty, (it & 1) ^ 1, abort_flag, 211)) break;
      if (lane == 0) {
        mbar_expect_tx(do_full, T_BYTES);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
          tma_load_3d(sDO + kb * (128 * 128), &tmDO, do_full, kb * 64, h, qs + qt);
      }
      // (dV of the last tile is done, so its dP, which has read these rows, is too)
#pragma unroll
      for (int e = 0; e < 4; ++e) write_aug_row(sDelta, e * 32 + lane, -dl[e]);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(delta_full);
      next_tile(h, qt);
    }
  } else if (warp == 13) {
    // --------------------------------------------------------------------------- MMA issuer
    if (lane == 0 && n_iter > 0) {
      constexpr uint32_t id_s = make_idesc_bf16(128, 128, 0, 0);       // Sᵀ, dPᵀ: both operands K-major
      constexpr uint32_t id_v = make_idesc_bf16(128, HD, 0, 1);        // dV (A in tensor memory), dK: MN-major B
      constexpr uint32_t id_q = make_idesc_bf16(128, HD, 1, 1);        // dQ: transposed A, MN-major B
      // Operand descriptors of whole tiles, K-major (_k) and MN-major (_m); a step adds its byte offset / 16.  Built once: with
      // a descriptor put together for every MMA this thread needed some 100 cycles for each, and the tensor core 64.
      const uint64_t dK_k = make_smem_desc(smem_u32(sK), 16, 1024), dK_m = make_smem_desc(smem_u32(sK), 128 * 128, 1024);
      const uint64_t dV_k = make_smem_desc(smem_u32(sV), 16, 1024);
      const uint64_t dQ_k = make_smem_desc(smem_u32(sQ), 16, 1024), dQ_m = make_smem_desc(smem_u32(sQ), 128 * 128, 1024);
      const uint64_t dDO_k = make_smem_desc(smem_u32(sDO), 16, 1024), dDO_m = make_smem_desc(smem_u32(sDO), 128 * 128, 1024);
      const uint64_t dDS_k = make_smem_desc(smem_u32(sDS), 16, 1024), dDS_m = make_smem_desc(smem_u32(sDS), 128 * 128, 1024);
      const uint64_t dOnes = make_aug_desc(smem_u32(sOnes)), dLse = make_aug_desc(smem_u32(sLse));
      const uint64_t dDelta = make_aug_desc(smem_u32(sDelta));
      auto issue_s = [&](int j) {
        const uint64_t dq = dQ_k + (j & 1) * (T_BYTES >> 4);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const uint32_t o = (kb * (128 * 128) + kk * 32) >> 4;
            umma_f16(tm_S, dK_k + o, dq + o, id_s, (kb | kk) != 0);
          }
        if constexpr (!CAP) umma_f16(tm_S, dOnes, dLse, id_s, 1);
        umma_commit(s_full);
      };
      auto issue_dp = [&]() {
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const uint32_t o = (kb * (128 * 128) + kk * 32) >> 4;
            umma_f16(tm_dP, dV_k + o, dDO_k + o, id_s, (kb | kk) != 0);
          }
        umma_f16(tm_dP, dOnes, dDelta, id_s, 1);
        umma_commit(dp_full);
      };
      auto issue_dv = [&](int j) {          // Pᵀ: 16 queries in 8 columns; the second half starts at column 64
#pragma unroll
        for (int s = 0; s < 8; ++s)
          umma_f16_ts(tm_dV, tm_S + (s >> 2) * 64 + (s & 3) * 8, dDO_m + s * (16 * 128 >> 4), id_v, s == 0 ? j != 0 : 1);
        umma_commit(do_empty);
      };
      bool ok = mbar_wait(kv_full, 0, abort_flag, 220) && mbar_wait(&q_full[0], 0, abort_flag, 221) &&
                (CAP || mbar_wait(&lse_full[0], 0, abort_flag, 221));
      if (ok) { tc_fence_after(); issue_s(0); }
      for (int j = -1; j < n_iter && ok; ++j) {
        const bool more = j + 1 < n_iter;
        if (j >= 0) {
          if (!(ok = mbar_wait(ds_full, j & 1, abort_flag, 222))) break;
          if (!DQ_OVER_DP && j > 0 && !(ok = mbar_wait(dq_empty, (j - 1) & 1, abort_flag, 223))) break;
          tc_fence_after();
#pragma unroll
          for (int s = 0; s < 8; ++s)        // reduction over the 128 keys, 16 per step
            umma_f16(tm_dQ, dDS_m + s * (16 * 128 >> 4), dK_m + s * (16 * 128 >> 4), id_q, s != 0);
          umma_commit(dq_full);
          if (more) {
            if (!(ok = mbar_wait(&q_full[(j + 1) & 1], ((j + 1) >> 1) & 1, abort_flag, 227))) break;
            if (!CAP && !(ok = mbar_wait(&lse_full[(j + 1) & 1], ((j + 1) >> 1) & 1, abort_flag, 228))) break;
            tc_fence_after();
            issue_s(j + 1);
          }
          // what dP(j+1) needs has normally come by now; waited for here, the waits cost nothing behind S and before dK
          if (more && !(ok = mbar_wait(do_full, (j + 1) & 1, abort_flag, 224))) break;
          if (more && !(ok = mbar_wait(delta_full, (j + 1) & 1, abort_flag, 229))) break;
          if (more && DQ_OVER_DP && !(ok = mbar_wait(dq_empty, j & 1, abort_flag, 225))) break;
          const uint64_t dq = dQ_m + (j & 1) * (T_BYTES >> 4);
#pragma unroll
          for (int s = 0; s < 8; ++s)        // reduction over the 128 queries
            umma_f16(tm_dK, dDS_k + ((s >> 2) * (128 * 128 >> 4) + (s & 3) * 2), dq + s * (16 * 128 >> 4), id_v,
                     s == 0 ? j != 0 : 1);
          umma_commit(&q_empty[j & 1]);
        }
        if (more) {
          if (j < 0 && !(ok = mbar_wait(do_full, 0, abort_flag, 224) && mbar_wait(delta_full, 0, abort_flag, 229))) break;
          tc_fence_after();
          issue_dp();
          if (!(ok = mbar_wait(p_full, (j + 1) & 1, abort_flag, 226))) break;
          tc_fence_after();
          issue_dv(j + 1);
        }
      }
      if (ok) umma_commit(acc_full);
    }
  } else if (warp < FAB_SOFTMAX_WARPS) {
    // ------------------------------------------------------------------------- softmax: P and dS
    const int quad = warp & 3;
    const int half = warp >> 2;                     // which half of the query columns this warp owns
    const int r = quad * 32 + lane;                 // key row inside the tile
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const float c = p.scale * 1.4426950408889634f;
    const float cap2 = p.softcap * 1.4426950408889634f;
    const float soc = CAP ? p.scale / p.softcap : 0.f;
    const int win = min(p.window, 1 << 29);
    constexpr float HIDDEN = -3.402823466e38f;      // (with soft-cap) finite: its product with a scale of 0 is a number
    bool ok = true;
    int h = kvh * rep, qt = qt_first;
    for (int it = 0; it < n_iter && ok; ++it) {
      const uint32_t ph = it & 1;
      const float4* lse4 = reinterpret_cast<const float4*>(sStat + ph * 128 + half * 64);      // (soft-cap)
      // a tile needs masking only if it touches the end of the queries / keys, the causal diagonal or the window edge
      const bool edge = (qt + 128 > len_q) || (k0 + 128 > len_k) ||
                        (p.causal && (k0 + 127 > qt + off || (p.window > 0 && k0 <= qt + 127 + off - p.window)));
      if (CAP && !(ok = mbar_wait_warp(&lse_full[ph], (it >> 1) & 1, abort_flag, 230))) break;
      if (!(ok = mbar_wait_warp(s_full, ph, abort_flag, 231))) break;
      tc_fence_after();
      uint32_t sv[2][32];                           // scores, then P (with soft-cap: the raw scores)
      tmem_ld_32x32(tm_S + lane_base + half * 64, sv[0]);
      tmem_ld_32x32(tm_S + lane_base + half * 64 + 32, sv[1]);
      tmem_ld_wait();
      if (edge) {
        // query columns this key row is seen by: [lo, hi)
        const int kj = k0 + r;
        const int first = p.causal ? kj - off - qt : 0;
        const int lo = (kj < len_k ? first : 1 << 30) - half * 64;
        const int hi = min(len_q - qt, (p.causal && win > 0) ? first + win : 128) - half * 64;
        // infinitely far on the side where the exponential is 0 (soft-cap: a value that is looked for)
        const uint32_t hidden = __float_as_uint(CAP ? HIDDEN : copysignf(INFINITY, -c));
#pragma unroll
        for (int q2 = 0; q2 < 2; ++q2)
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (q2 * 32 + e < lo || q2 * 32 + e >= hi) sv[q2][e] = hidden;
      }
#pragma unroll
      for (int q2 = 0; q2 < 2; ++q2) {
        uint32_t pk[16];
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          float pe[4];
          if constexpr (CAP) {
            const float4 l4 = lse4[q2 * 8 + g];
            const float ls[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float s = __uint_as_float(sv[q2][g * 4 + e]);
              pe[e] = s == HIDDEN ? 0.f : ex2_approx(cap2 * tanh_fast(s * soc) - ls[e]);
            }
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              pe[e] = ex2_approx(__uint_as_float(sv[q2][g * 4 + e]) * c);      // (the score less lse / scale)
              sv[q2][g * 4 + e] = __float_as_uint(pe[e]);
            }
          }
          const __nv_bfloat162 a = __floats2bfloat162_rn(pe[0], pe[1]), b = __floats2bfloat162_rn(pe[2], pe[3]);
          pk[g * 2] = *reinterpret_cast<const uint32_t*>(&a);
          pk[g * 2 + 1] = *reinterpret_cast<const uint32_t*>(&b);
        }
        // over the columns that this warp itself has read
        tmem_st_32x16(tm_S + lane_base + half * 64 + q2 * 16, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      if (!(ok = mbar_wait_warp(dp_full, ph, abort_flag, 232))) break;
      tc_fence_after();
#pragma unroll
      for (int q2 = 0; q2 < 2; ++q2) {
        uint32_t vd[32];                            // dP - delta
        tmem_ld_32x32(tm_dP + lane_base + half * 64 + q2 * 32, vd);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          float ds[8];
          if constexpr (CAP) {
            const float4 la = lse4[q2 * 8 + g * 2], lb = lse4[q2 * 8 + g * 2 + 1];
            const float ls[8] = {la.x, la.y, la.z, la.w, lb.x, lb.y, lb.z, lb.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float s = __uint_as_float(sv[q2][g * 8 + e]);
              const float th = tanh_fast(s * soc);
              const float pe = s == HIDDEN ? 0.f : ex2_approx(cap2 * th - ls[e]);
              // d(cap * tanh(scale * s / cap)) / ds = scale * (1 - tanh^2)
              ds[e] = pe * __uint_as_float(vd[g * 8 + e]) * p.scale * (1.f - th * th);
            }
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              ds[e] = __uint_as_float(sv[q2][g * 8 + e]) * __uint_as_float(vd[g * 8 + e]) * p.scale;
          }
          uint4 b;
          __nv_bfloat162* b2 = reinterpret_cast<__nv_bfloat162*>(&b);
#pragma unroll
          for (int e = 0; e < 4; ++e) b2[e] = __floats2bfloat162_rn(ds[2 * e], ds[2 * e + 1]);
          *reinterpret_cast<uint4*>(sDS + sw128_offset(r, half * 64 + q2 * 32 + g * 8, 128)) = b;
        }
      }
      tc_fence_before();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
      next_tile(h, qt);
    }
    // dK / dV of this key tile (thread = key row)
    constexpr int HC2 = HD / 2;
    if (n_iter > 0 && ok) ok = mbar_wait_warp(acc_full, 0, abort_flag, 233);
    // Through shared memory (the Q stages, which nothing reads any more), so that the stores to global memory are whole
    // rows: a row per thread wrote 32 lines an instruction, 4.0 us a tile.
    const bool have = n_iter > 0 && ok;
    tc_fence_after();
#pragma unroll 1
    for (int cb = half * HC2; cb < half * HC2 + HC2; cb += 32) {
      uint32_t a[32], b[32];
      if (have) {
        tmem_ld_32x32(tm_dV + lane_base + cb, a);
        tmem_ld_32x32(tm_dK + lane_base + cb, b);
        tmem_ld_wait();
      }
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        uint4 x = make_uint4(0, 0, 0, 0), y = x;
        if (have) {
          __nv_bfloat162* x2 = reinterpret_cast<__nv_bfloat162*>(&x);
          __nv_bfloat162* y2 = reinterpret_cast<__nv_bfloat162*>(&y);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            x2[e] = __floats2bfloat162_rn(__uint_as_float(a[g * 8 + 2 * e]), __uint_as_float(a[g * 8 + 2 * e + 1]));
            y2[e] = __floats2bfloat162_rn(__uint_as_float(b[g * 8 + 2 * e]), __uint_as_float(b[g * 8 + 2 * e + 1]));
          }
        }
        const uint32_t o = sw128_offset(r, cb + g * 8, 128);
        *reinterpret_cast<uint4*>(sQ + o) = x;
        *reinterpret_cast<uint4*>(sQ + T_BYTES + o) = y;
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(FAB_SOFTMAX_WARPS * 32) : "memory");
    constexpr int CH = HD / 8;                      // 16-byte pieces of a row
#pragma unroll 4
    for (int i = threadIdx.x; i < 128 * CH; i += FAB_SOFTMAX_WARPS * 32) {
      const int rr = i / CH, cc = (i % CH) * 8;
      if (rr < kr) {
        const size_t at = (static_cast<size_t>(ks + k0 + rr) * p.KV + kvh) * HD + cc;
        const uint32_t o = sw128_offset(rr, cc, 128);
        *reinterpret_cast<uint4*>(p.dv + at) = *reinterpret_cast<const uint4*>(sQ + o);
        *reinterpret_cast<uint4*>(p.dk + at) = *reinterpret_cast<const uint4*>(sQ + T_BYTES + o);
      }
    }
  } else if (warp < 12) {
    // ------------------------------------------------------------------------- dQ drain, 32 query rows a warp
    // Tensor memory -> registers -> fp32 staging in shared memory (blocks of 32 rows x 32 columns, 128-byte swizzle) ->
    // tiled reduce-adds into the fp32 workspace: L2 sees whole 128-byte lines per reduction.  Each warp is on its own.  A
    // tile of hd 128 takes some 4300 cycles to leave, about the rate at which an SM's reductions are taken (16 bytes a
    // cycle); blocks of 16 rows took 7000, blocks of 64 rows shared by two warps (who then wait for each other) 6500.
    // Rows past the end of the sequence hold exact zeros (their P and dS were masked), so adding them is harmless.
    const int quad = warp & 3;
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    uint8_t* stg = sStg + quad * L::STAGES * L::STAGE_BYTES;
    // index of this sequence's first query tile (semaphores)
    const int qtile_base = p.dq_sem != nullptr ? tiles_before(p.cu_q, seq, 128) : 0;
    auto stage = [&](int slot, const uint32_t (&v)[32]) {
      uint8_t* rowp = stg + slot * L::STAGE_BYTES + lane * 128;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<uint4*>(rowp + ((j ^ (lane & 7)) << 4)) =
            make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    };
    auto add_row = [&](float* dst, const uint32_t (&v)[32]) {
#pragma unroll
      for (int e = 0; e < 32; e += 4)
        red_add_v4_f32(dst + e, __uint_as_float(v[e]), __uint_as_float(v[e + 1]), __uint_as_float(v[e + 2]),
                       __uint_as_float(v[e + 3]));
    };
    // In a fixed order, a tile's turn passes on when its additions have been performed.  LAST_FIRST, whose next key tile
    // comes a step later by itself, looks at that only before the staging block is needed again: waiting at once held this
    // warp for another 1400 cycles a tile (16 x 1024 tokens 4 % more).  IN_STEP, where the next key tile is
    // waiting, passes on at once (1 x 16384: later, 4 % more).
    int* passing = nullptr;
    auto pass_on = [&]() {
      if (passing != nullptr) {
        bulk_wait_all();
        red_release_gpu_add_s32(passing, 1);
        passing = nullptr;
      }
    };
    int h = kvh * rep, qt = qt_first;
    for (int it = 0; it < n_iter; ++it) {
      if (!mbar_wait_warp(dq_full, it & 1, abort_flag, 235)) break;
      tc_fence_after();
      const bool live = qt + quad * 32 < len_q;
      int* sem = nullptr;
      if (p.dq_sem != nullptr && live)
        // deterministic order, for each 32 rows of a query tile (word 0 of the array is the give-up flag)
        sem = p.dq_sem + 1 + ((static_cast<size_t>(qtile_base + qt / 128)) * p.H + h) * 4 + quad;
      auto wait_turn = [&]() {
        // wait until the key tiles before this one in the order have added their share of these rows.  Giving up loses the order, not
        // data; the flag makes every later wait of this launch return at once, so one lost turn costs one time limit
        // (about a second), not one per tile.
        int expected;
        if (in_step) {
          expected = k0 / 128 - (p.causal && p.window > 0 ? max(0, qt + off - p.window + 1) / 128 : 0);
        } else {
          const int n_kt = (len_k + 127) / 128;
          expected = (p.causal ? min(n_kt - 1, (qt + 127 + off) / 128) : n_kt - 1) - k0 / 128;
        }
        uint32_t spins = 0;
        volatile int* gave_up = p.dq_sem;
        while (expected > 0 && !*gave_up && ld_acquire_gpu_s32(sem) < expected) {
          if (++spins > (1u << 21) || *abort_flag) { *gave_up = 1; set_error(4, 240); break; }
          __nanosleep(32);
        }
      };
      // Blocks of 32 columns; the first is staged as soon as it is read, so that three blocks of registers are enough to
      // empty the columns before anything is waited for.
      constexpr int NB = HD / 32;
      uint32_t v[3][32];
      auto load = [&](int cb) { tmem_ld_32x32(tm_dQ + lane_base + cb * 32, v[cb % 3]); };
      load(0);
      load(1);
      if constexpr (NB > 2) load(2);
      tmem_ld_wait();
      if (live && p.dq_bulk) {
        if (lane == 0) { pass_on(); bulk_wait_read_all(); }      // the last tile has left the staging blocks
        __syncwarp();
        stage(0, v[0]);
        if constexpr (NB > 3) { load(3); tmem_ld_wait(); }
      }
      if (!live || p.dq_bulk) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(dq_empty);           // the columns may be written again
      }
      if (live && p.dq_bulk) {
#pragma unroll
        for (int cb = 0; cb < NB; cb += L::STAGES) {
          if (cb > 0) {
            if (lane == 0) bulk_wait_read_all();
            __syncwarp();
            stage(0, v[cb % 3]);
          }
          if constexpr (L::STAGES == 2) stage(1, v[(cb + 1) % 3]);
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            if (cb == 0 && sem != nullptr) wait_turn();
#pragma unroll
            for (int i = 0; i < L::STAGES; ++i)
              tma_reduce_add_2d(&tmDQ, stg + i * L::STAGE_BYTES, h * HD + (cb + i) * 32, qs + qt + quad * 32);
            bulk_commit();
          }
        }
        if (lane == 0) {
          passing = sem;
          if (in_step) pass_on();
        }
      } else if (live) {                                // 16-byte reductions, one row per thread
        const int i = qt + quad * 32 + lane;
        float* dst = p.dq_acc + (static_cast<size_t>(qs + min(i, len_q - 1)) * p.H + h) * HD;
        if (lane == 0 && sem != nullptr) wait_turn();
        __syncwarp();
        if (i < len_q) add_row(dst, v[0]);
        if constexpr (NB > 3) {
          __syncwarp();
          load(3);
          tmem_ld_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(dq_empty);
        if (i < len_q) {
#pragma unroll
          for (int cb = 1; cb < NB; ++cb) add_row(dst + cb * 32, v[cb % 3]);
        }
        if (sem != nullptr) {
          __threadfence();
          __syncwarp();
          if (lane == 0) red_release_gpu_add_s32(sem, 1);
        }
      }
      next_tile(h, qt);
    }
    if (p.dq_bulk && lane == 0) { pass_on(); bulk_wait_all(); }      // none of this thread's reduce-adds outlives the kernel
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 13) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int HD, bool CAP>
static int launch_bwd(const CUtensorMap& tq, const CUtensorMap& tdo, const CUtensorMap& tk, const CUtensorMap& tv,
                      const CUtensorMap& tdq, const BwdParams& p, int tiles, cudaStream_t s) {
  constexpr int SMEM = BwdSmem<HD>::SIZE;
  auto kern = fa_bwd_kernel<HD, CAP>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return -300 - static_cast<int>(e);
    configured = true;
  }
  if (static_cast<long>(p.KV) * tiles > 0x7fffffffL) return -2;
  kern<<<static_cast<unsigned>(p.KV * tiles), FAB_THREADS, SMEM, s>>>(tq, tdo, tk, tv, tdq, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -400 - static_cast<int>(e);
}

}  // namespace ftb

extern "C" {

// dout / q / out (Tq, H, hd), k / v (Tk, KV, hd) bf16 with token strides; lse (H, Tq) from the forward.
// Workspaces supplied by the caller: delta (H, Tq) fp32, dq_acc (Tq, H, hd) fp32 ZEROED.
// Outputs: dQ, in fp32 in dq_acc; dk, dv (Tk, KV, hd) bf16 contiguous, every row written.
// dq_sem: NULL, or 1 + (sum over sequences of ceil(len_q / 128)) x H x 4 int32 words, ZEROED (word 0 is the kernel's
//   give-up flag, the rest one counter per (query tile, head, 32 rows)): makes the dQ summation order
// fixed (bit-reproducible gradients) at the price of ordering the CTAs that share a query tile.
// max_k: the longest sequence's keys (it chooses the order of the work only).
int ftb_attn_bwd(const void* dout, const void* q, const void* k, const void* v, const void* out, const float* lse,
                 float* delta, float* dq_acc, int* dq_sem, void* dk, void* dv, const int* cu_q, const int* cu_k, int num_seqs,
                 int total_q, int total_k, int H, int KV, int hd, long q_stride, long k_stride,
                 long v_stride, long do_stride, long o_stride, float scale, float softcap, int causal, int window,
                 int max_tiles, int max_k, cudaStream_t stream) {
  if (total_q <= 0 || num_seqs <= 0) return 0;
  if ((hd != 64 && hd != 128) || H % KV) return -2;
  // (dout and out are read in 16-byte pieces before any tensor map is made; the maps check the others)
  if ((q_stride & 7) || (k_stride & 7) || (v_stride & 7) || (do_stride & 7) || (o_stride & 7) ||
      ((reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(out)) & 15))
    return -2;
  {
    const long threads = (long)total_q * H * (hd / 8);
    (hd == 128 ? fa_delta_kernel<128> : fa_delta_kernel<64>)<<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>(
        (const __nv_bfloat16*)dout, do_stride, (const __nv_bfloat16*)out, o_stride, delta, total_q, H);
  }
  CUtensorMap tq, tdo, tk, tv;
  int rc = make_tmap_3d(&tq, q, hd, H, total_q, q_stride, 128);
  if (rc) return rc;
  rc = make_tmap_3d(&tdo, dout, hd, H, total_q, do_stride, 128);
  if (rc) return rc;
  rc = make_tmap_3d(&tk, k, hd, KV, total_k, k_stride, 128);
  if (rc) return rc;
  rc = make_tmap_3d(&tv, v, hd, KV, total_k, v_stride, 128);
  if (rc) return rc;
  // fp32 workspace as a 2-D tensor (total_q rows of H * hd columns): boxes of 32 rows x 32 columns for the reduce-adds
  CUtensorMap tdq;
  {
    EncodeTiledFn enc = get_encode();
    if (enc == nullptr) return -100;
    cuuint64_t gdim[2] = {(cuuint64_t)H * hd, (cuuint64_t)total_q};
    cuuint64_t gstr[1] = {(cuuint64_t)H * hd * 4};
    cuuint32_t box[2] = {32, 32};
    cuuint32_t es[2] = {1, 1};
    CUresult r = enc(&tdq, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, dq_acc, gdim, gstr, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return -200 - static_cast<int>(r);
  }
  BwdParams p;
  p.cu_q = cu_q; p.cu_k = cu_k; p.num_seqs = num_seqs; p.H = H; p.KV = KV; p.dq_bulk = g_dq_bulk;
  p.dq_acc = dq_acc; p.dq_sem = dq_sem; p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv; p.lse = lse; p.delta = delta;
  p.order = dq_sem == nullptr ? BWD_FIRST_FIRST : max_k > (hd == 128 ? 4096 : 1024) ? BWD_IN_STEP : BWD_LAST_FIRST;
  p.total_q = total_q; p.scale = scale; p.softcap = softcap; p.causal = causal; p.window = window;
  // The plain form divides lse by the scale.  A scale of 0 (or so small that the quotient leaves fp32) takes the soft-cap form,
  // which subtracts lse after scaling: a cap of 1 leaves scores that are all next to 0 as they are.
  if (!(softcap > 0.f) && fabsf(scale) < 1e-20f) p.softcap = 1.f;
  if (p.softcap > 0.f)
    rc = (hd == 128) ? launch_bwd<128, true>(tq, tdo, tk, tv, tdq, p, max_tiles, stream)
                     : launch_bwd<64, true>(tq, tdo, tk, tv, tdq, p, max_tiles, stream);
  else
    rc = (hd == 128) ? launch_bwd<128, false>(tq, tdo, tk, tv, tdq, p, max_tiles, stream)
                     : launch_bwd<64, false>(tq, tdo, tk, tv, tdq, p, max_tiles, stream);
  return rc;
}

// 1 (default): dQ leaves the SM as tiled reduce-adds from shared memory; 0: per-thread vector reductions
void ftb_attn_set_dq_bulk(int on) { g_dq_bulk = on; }

}  // extern "C"
