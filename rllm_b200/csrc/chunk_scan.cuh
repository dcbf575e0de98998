// A recurrence over a per-request state in chunks of 64 tokens, float arithmetic throughout, for long portions:
//     S_t = diag(a_t) S_(t-1) + k_t u_t^T,   o_t = S_t^T q_t (+ skip v_t)
// with u_t = beta_t (v_t - (diag(a_t) S_(t-1))^T k_t) (DELTA) or f_t v_t, decays per key channel (PERCH) or per head. With a
// BONUS b a token reads the state before it and its own product times b: o_t = S_(t-1)^T q_t + v_t sum_c q_t b k_t.
//
// Token by token this is one chain: a token's sums over the channels wait for the one before. Inside a chunk, with P_t the
// product of the decays up to t and P_t / P_j that of the decays after j (always formed as a product of factors, never as a
// quotient, so that nothing overflows where the decays are strong), everything is a product of matrices:
//     (I + L) U = diag(beta) (V - (P k) S_0),   L[t][j] = beta_t sum_c k_t k_j P_t / P_j  for j < t
//     O = (P q) S_0 + M U,                      M[t][j] = sum_c q_t k_j P_t / P_j         for j <= t
//     S_end = diag(P_end) S_0 + (k P_end / P)^T U
//   chunk_prep_kernel   a CTA a (chunk, head), all chunks side by side: M, P q, k P_end / P, and for DELTA W = (I + L)^-1 beta P k
//                       and (I + L)^-1 beta V, the inverse by blocks of 16 (what is left of U is - W S_0).
//   chunk_carry_kernel  a CTA a (sequence, head, NC value columns) walks the chunks: keeps the state it meets for the last
//                       kernel, U -= W S, S = P_end S + (k P_end / P)^T U. The rows of the chunk after the next travel meanwhile.
//   chunk_out_kernel    a CTA a (chunk, head, 64 value columns), all side by side: O.
// What a kernel leaves for the next lies in the scratch as the next one's shared memory holds it (rows padded, value columns
// in tiles of 16), so that a few bulk copies by one thread bring it (16-byte copies by all threads cost as much as the sums).
// Decays per channel do not factor out of M and L. Blocks of 16 x 16 below the diagonal are a product of rows scaled by the
// decays since their own block's beginning with rows scaled by the decays up to it (both at most 1); the ones on the diagonal
// are summed with a running product per channel.
// What bounds it: FMAs and the shared memory that feeds them (a token costs a head about 73,000 FMAs at 128 x 128, no fewer
// than token by token), no longer a chain; a product's operands come in tiles of 32 x 16 a warp, 64 FMAs for 8 loads of 16
// bytes (8 x 8 outputs a thread, half the loads: level, and 85 us against 59 where a CTA's sum is short).
// 2,048 tokens, bfloat16 runs, us (token by token before): delta rule with decays per channel, 16 heads of 128 x 128
// 272 (1,061); with a decay per head, 32 heads 422 (1,050); state space, 32 heads of 128 x 64 214 (745); gated linear attention,
// 16 heads 212 (405 in three passes over chunks).
// 64 tokens: with 32 the walk over the chunks has twice the barriers for the same FMAs, with 128 the triangles cost more than
// the rest. Sums are grouped differently than token by token, by fours and sixteens, so that no chain is long: outputs' distance from
// 64 bits (2-norm, 1,024 tokens) 2.1e-7 where decays are slow (row by row 3.0e-7), 1.1e-7 (1.0e-7) where half the state is gone with
// every token; as chains of 64 and 128 they were at 3.3e-7 and 1.9 to 2.5e-7. The loads hide the additions.
#pragma once
#include "common.cuh"
#include "sm100.cuh"

namespace rllm {
namespace chunked {

constexpr int C = 64;      // tokens a chunk
constexpr int SB = 16;     // tokens a block of the triangles
constexpr int LC = C + 4;  // row stride of a [64][64] matrix in shared memory
constexpr int THREADS = 256;

struct Args {
  const void* q; const void* k; const void* v;        // rows of TI, column offset folded in
  long long q_ld, k_ld, v_ld;
  int q_heads, k_heads;
  float qscale;
  const float* decay;                                 // [T, H * D] (PERCH) or [T, H]
  const void* beta; long long beta_ld; int beta_bf16; // logits (DELTA)
  const float* vscale;                                // [T, H] or null
  const float* skip;                                  // [H] or null
  const float* bonus;                                 // [H, D] (BONUS)
  int H, vdim;
  const int* cu_q; int num_seqs; const int* state_slots;
  int long_from;                                      // sequences with fewer rows are left to another kernel
  float* state;                                       // [slots, H, D, vdim]
  float* out;                                         // [T, H, vdim]
  float* scratch;                                     // per (chunk, head): see Place
  int* err;                                           // device word that a wait which runs out leaves its mark in
};

// One (chunk, head)'s share of the scratch: M [C][LC], P q [C][D + 4], k P_end / P [C][D], W [C][D + 4] (DELTA), U and the state the
// chunk meets in tiles of 16 columns, [C][16] and [D][16] each, P_end [D]. Every piece a multiple of 16 bytes.
template <int D>
struct Place {
  float *m, *qd, *kt, *w, *u, *s, *pc;
  __host__ __device__ static long long floats(int vdim, bool delta) {
    return (long long)C * LC + C * (D + 4) + C * D + (delta ? C * (D + 4) : 0) + (long long)C * vdim + (long long)D * vdim + D;
  }
  __device__ Place(float* base, long long x, int vdim, bool delta) {
    m = base + x * floats(vdim, delta);
    qd = m + C * LC;
    kt = qd + C * (D + 4);
    w = kt + C * D;
    u = w + (delta ? C * (D + 4) : 0);
    s = u + (long long)C * vdim;
    pc = s + (long long)D * vdim;
  }
};

// Chunks of a sequence of n rows; which sequence and chunk a CTA has (false: none).
__device__ __forceinline__ int chunks_of(int n, int long_from) { return n < long_from ? 0 : (n + C - 1) / C; }
__device__ __forceinline__ bool find_chunk(const Args& a, int b, int& row0, int& n) {
  int at = 0;
  for (int s = 0; s < a.num_seqs; ++s) {
    const int r0 = a.cu_q[s], rows = a.cu_q[s + 1] - r0, cs = chunks_of(rows, a.long_from);
    if (b < at + cs) { row0 = r0 + (b - at) * C; n = min(C, rows - (b - at) * C); return true; }
    at += cs;
  }
  return false;
}

// n floats (a multiple of 4) into shared memory, counted by the barrier; one thread.
__device__ __forceinline__ void bulk(float* smem, const float* gmem, int n, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sm100::smem_u32(smem)),
               "l"(gmem), "r"(4 * n), "r"(sm100::smem_u32(bar)) : "memory");
}
// A wait has run out: it leaves its mark and waits once more for the copies that may still be on their way into this CTA's memory,
// this one and the one after (null: none). Out of line, so that the walk's code is not arranged around it.
__device__ __noinline__ void give_up(uint64_t* bar, uint32_t parity, uint64_t* next, uint32_t next_parity, volatile int* abort_flag,
                                     int* err, int role) {
  *abort_flag = 1;
  sm100::record_failure(err, role);
  volatile int none = 0;
  sm100::mbar_wait(bar, parity, &none);
  if (next) sm100::mbar_wait(next, next_parity, &none);
}
// All threads wait for a barrier's phase; false: some wait ran out, and the CTA's work ends.
__device__ __forceinline__ bool landed(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* err, int role,
                                       uint64_t* next = nullptr, uint32_t next_parity = 0) {
  const bool ok = sm100::mbar_wait(bar, parity, abort_flag);
  if (!ok) give_up(bar, parity, next, next_parity, abort_flag, err, role);
  return __syncthreads_and(ok);
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const bf16* p) {
  const uint2 x = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// acc[i][c] += sum_k A[row + 8 i][k] B[k][col + c]: a warp's tile of 32 x 16, `row` = first row + lane / 4, `col` = first column +
// 4 (lane % 4). K a multiple of 16; A's rows 16 bytes apart in bank phase (stride 4 mod 32). Four products are added up, then four such
// sums, then those (no chain longer than K / 16): 0.4 of the error that one chain leaves, and as fast, since the loads bound it.
__device__ __forceinline__ void add16(float (&acc)[4][4], const float (&s)[4][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[i][c] += s[i][c];
}
__device__ __forceinline__ void tile_product(float (&acc)[4][4], const float* A, int lda, const float* B, int ldb, int K) {
#pragma unroll 1
  for (int k0 = 0; k0 < K; k0 += 16) {
    float part[4][4] = {};
#pragma unroll
    for (int k = k0; k < k0 + 16; k += 4) {
      float4 x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(A + 8 * i * lda + k);
      float sum[4][4] = {};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float4 y = *reinterpret_cast<const float4*>(B + (k + e) * ldb);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float xv = e == 0 ? x[i].x : e == 1 ? x[i].y : e == 2 ? x[i].z : x[i].w;
          sum[i][0] = fmaf(xv, y.x, sum[i][0]);
          sum[i][1] = fmaf(xv, y.y, sum[i][1]);
          sum[i][2] = fmaf(xv, y.z, sum[i][2]);
          sum[i][3] = fmaf(xv, y.w, sum[i][3]);
        }
      }
      add16(part, sum);
    }
    add16(acc, part);
  }
}

// The same for the lower triangle of a [64][64] A, the warp's rows its upper (half 0) or lower 32: what lies right of the
// diagonal is left out, not multiplied as zero. A token's sum then holds nothing of the tokens after it, which zero times an
// infinity or NaN of theirs would bring in.
__device__ __forceinline__ void triangle_product(float (&acc)[4][4], const float* A, int lda, const float* B, int ldb, int half, int row) {
  if (half) tile_product(acc, A, lda, B, ldb, C / 2);
  A += half * (C / 2);
  B += half * (C / 2) * ldb;
#pragma unroll
  for (int k0 = 0; k0 < C / 2; k0 += 8) {
    float sum[4][4] = {};
#pragma unroll
    for (int k = k0; k < k0 + 8; k += 4) {
      float4 x[4];
#pragma unroll
      for (int i = k / 8; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(A + 8 * i * lda + k);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float4 y = *reinterpret_cast<const float4*>(B + (k + e) * ldb);
#pragma unroll
        for (int i = k / 8; i < 4; ++i) {
          const float xv = e == 0 ? x[i].x : e == 1 ? x[i].y : e == 2 ? x[i].z : x[i].w;
          if (i > k / 8 || k % 8 + e <= row) {
            sum[i][0] = fmaf(xv, y.x, sum[i][0]);
            sum[i][1] = fmaf(xv, y.y, sum[i][1]);
            sum[i][2] = fmaf(xv, y.z, sum[i][2]);
            sum[i][3] = fmaf(xv, y.w, sum[i][3]);
          }
        }
      }
    }
    add16(acc, sum);
  }
}

__device__ __forceinline__ float dot4(float4 a, float4 b, float c) {
  return c + fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w)));     // a chain of sums of four
}

// X (lower triangular, [64][LC]) = (I + L)^-1, L strictly lower [64][LC]; tmp: 3 x 16 x 17 floats. Blocks of 16 on the diagonal
// column by column, then the block diagonals below: X_IJ = -X_II sum_K L_IK X_KJ.
__device__ __forceinline__ void unit_lower_inverse(const float* L, float* X, float* tmp) {
  const int tid = threadIdx.x;
  for (int x = tid; x < C * C; x += THREADS) {
    const int t = x / C, j = x % C;
    if ((t / SB) != (j / SB)) X[t * LC + j] = 0.f;
  }
  if (tid < C) {
    const int b = tid / SB * SB, j = tid % SB;
    float x[SB];
#pragma unroll
    for (int t = 0; t < SB; ++t) {
      float r = t == j ? 1.f : 0.f;
#pragma unroll
      for (int m = 0; m < t; ++m) r = fmaf(-L[(b + t) * LC + b + m], x[m], r);
      x[t] = r;
    }
#pragma unroll
    for (int t = 0; t < SB; ++t) X[(b + t) * LC + b + j] = x[t];
  }
  __syncthreads();
  const int t = tid / SB, j = tid % SB;
#pragma unroll
  for (int d = 1; d < C / SB; ++d) {
#pragma unroll
    for (int J = 0; J < C / SB - d; ++J) {
      const int I = J + d;
      float y = 0.f;
#pragma unroll
      for (int m = 0; m < SB * d; m += 4) {
        const float4 l = *reinterpret_cast<const float4*>(L + (I * SB + t) * LC + J * SB + m);
        const float* xc = X + (J * SB + m) * LC + J * SB + j;
        y += fmaf(l.x, xc[0], fmaf(l.y, xc[LC], fmaf(l.z, xc[2 * LC], l.w * xc[3 * LC])));
      }
      tmp[(J * SB + t) * (SB + 1) + j] = y;
    }
    __syncthreads();
#pragma unroll
    for (int J = 0; J < C / SB - d; ++J) {
      const int I = J + d;
      float x = 0.f;
#pragma unroll
      for (int m = 0; m < SB; ++m)
        if (m <= t) x = fmaf(X[(I * SB + t) * LC + I * SB + m], tmp[(J * SB + m) * (SB + 1) + j], x);
      X[(I * SB + t) * LC + J * SB + j] = -x;
    }
    __syncthreads();
  }
}

template <typename TI, int D, bool PERCH, bool DELTA, bool BONUS>
__global__ void __launch_bounds__(THREADS, 2) chunk_prep_kernel(Args a) {
  pdl_launch();
  pdl_wait();
  constexpr int LDD = D + 4, NV = D / 4;
  extern __shared__ __align__(16) float sm[];
  float* few = sm;                                      // [C] decays, [C] beta or value scales
  float* Q = few + 2 * C;                               // [C][LDD] each
  float* K = Q + C * LDD;
  float* A = K + C * LDD;                               // PERCH: decays, later k scaled up to the next block, later L and the inverse
  float* blk = A + C * LDD;                             // PERCH: [4][D] products of blocks
  float* G2 = A;                                        // [C][LC] L (DELTA)
  float* G1 = A + (DELTA ? C * LC : 0);                 // [C][LC] ratios of decays (per head); the inverse (DELTA)
  float* tmp = G1 + C * LC;                             // 3 x 16 x 17 for the inverse, or 5 x 64 products (per head)
  // L of the decays per channel waits in W's place of the scratch until A's is free (a second CTA fits the SM that way)
  int row0, n;
  if (!find_chunk(a, blockIdx.x, row0, n)) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int H = a.H, h = blockIdx.y, V = a.vdim;
  const Place<D> to(a.scratch, (long long)blockIdx.x * H + h, V, DELTA);
  const TI* qg = reinterpret_cast<const TI*>(a.q) + (h / (H / a.q_heads)) * D;
  const TI* kg = reinterpret_cast<const TI*>(a.k) + (h / (H / a.k_heads)) * D;
  const TI* vg = reinterpret_cast<const TI*>(a.v) + (long long)h * V;
  for (int x = tid; x < C * NV; x += THREADS) {
    const int t = x / NV, c = x % NV * 4;
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f), k = q, d = make_float4(1.f, 1.f, 1.f, 1.f);
    if (t < n) {
      const long long r = row0 + t;
      q = load4(qg + r * a.q_ld + c);
      k = load4(kg + r * a.k_ld + c);
      if (PERCH) d = load4(a.decay + (r * H + h) * D + c);
      q.x *= a.qscale; q.y *= a.qscale; q.z *= a.qscale; q.w *= a.qscale;
    }
    *reinterpret_cast<float4*>(Q + t * LDD + c) = q;
    *reinterpret_cast<float4*>(K + t * LDD + c) = k;
    if (PERCH) *reinterpret_cast<float4*>(A + t * LDD + c) = d;
  }
  if (tid < C) {
    const long long r = row0 + tid;
    if (!PERCH) few[tid] = tid < n ? a.decay[r * H + h] : 1.f;
    float b = 0.f;
    if (tid < n) {
      if (DELTA) {
        const float z = a.beta_bf16 ? to_f32(reinterpret_cast<const bf16*>(a.beta)[r * a.beta_ld + h])
                                    : reinterpret_cast<const float*>(a.beta)[r * a.beta_ld + h];
        b = 1.f / (1.f + expf(-z));
      } else {
        b = a.vscale ? a.vscale[r * H + h] : 1.f;
      }
    }
    few[C + tid] = b;
  }
  __syncthreads();
  const float* beta = few + C;

  if constexpr (!PERCH) {
    // one decay a head: the ratios of products are a matrix of their own, G1[t][j] = a_(j+1) ... a_t: inside a block of 16 one by
    // one, below as (up to the end of j's block) (the blocks between) (from the beginning of t's block)
    float* upto = tmp;                                   // [C] from the block's beginning
    float* rest = tmp + C;                               // [C] to the block's end
    if (tid < C) {
      const int b = tid & ~(SB - 1), j = tid;
      float r = 1.f;
      for (int t = b; t <= j; ++t) r *= few[t];
      upto[j] = r;
      r = 1.f;
#pragma unroll
      for (int e = 0; e < SB; ++e) {
        const int t = b + e;
        if (t > j) r *= few[t];
        G1[t * LC + j] = r;                              // 1 where t <= j
      }
      rest[j] = r;
    }
    __syncthreads();
    for (int x = tid; x < C * C; x += THREADS) {
      const int t = x / C, j = x % C, I = t / SB, J = j / SB;
      if (J < I) {
        float r = rest[j];
        for (int b = J + 1; b < I; ++b) r *= upto[b * SB + SB - 1];
        G1[t * LC + j] = r * upto[t];
      }
    }
    __syncthreads();
    const float first = few[0];
    const int r0 = (warp >> 1) * 16 + (lane >> 3), c0 = (warp & 1) * 32 + (lane & 7);
    float m[4][4] = {}, l[4][4] = {};
    if ((warp & 1) * 32 < (warp >> 1) * 16 + 16) {      // else wholly above the diagonal
#pragma unroll 1
      for (int cc = 0; cc < D; cc += 16) {
        float mp[4][4] = {}, lp[4][4] = {};
#pragma unroll 1
        for (int c = cc; c < cc + 16; c += 4) {
          float4 q[4], k[4], kc[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            q[i] = *reinterpret_cast<const float4*>(Q + (r0 + 4 * i) * LDD + c);
            if (DELTA) k[i] = *reinterpret_cast<const float4*>(K + (r0 + 4 * i) * LDD + c);
            kc[i] = *reinterpret_cast<const float4*>(K + (c0 + 8 * i) * LDD + c);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              mp[i][j] = dot4(q[i], kc[j], mp[i][j]);
              if (DELTA) lp[i][j] = dot4(k[i], kc[j], lp[i][j]);
            }
        }
        add16(m, mp);
        if (DELTA) add16(l, lp);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = r0 + 4 * i, s = c0 + 8 * j;
        const float r = s <= t ? G1[t * LC + s] : 0.f;
        to.m[t * LC + s] = s <= t ? m[i][j] * r : 0.f;
        if (DELTA) G2[t * LC + s] = s < t ? beta[t] * l[i][j] * r : 0.f;
      }
    // P q and k P_end / P; what K holds afterwards is k P (times beta) for the last product
    for (int x = tid; x < C * NV; x += THREADS) {
      const int t = x / NV, c = x % NV * 4;
      const float p = first * G1[t * LC], e = G1[(C - 1) * LC + t];
      float4 q = *reinterpret_cast<float4*>(Q + t * LDD + c), k = *reinterpret_cast<float4*>(K + t * LDD + c);
      *reinterpret_cast<float4*>(to.qd + t * LDD + c) = make_float4(q.x * p, q.y * p, q.z * p, q.w * p);
      *reinterpret_cast<float4*>(to.kt + t * D + c) = make_float4(k.x * e, k.y * e, k.z * e, k.w * e);
    }
    if (tid < D) to.pc[tid] = first * G1[(C - 1) * LC];
    if (DELTA) {
      __syncthreads();
      for (int x = tid; x < C * NV; x += THREADS) {
        const int t = x / NV, c = x % NV * 4;
        const float p = first * G1[t * LC] * beta[t];
        float4* k = reinterpret_cast<float4*>(K + t * LDD + c);
        *k = make_float4(k->x * p, k->y * p, k->z * p, k->w * p);
      }
    }
  } else {
    // blocks on the diagonal: a thread has key token j of a block and every fourth group of four channels, and walks the
    // tokens after it with the running product of the decays
    {
      const int b = (tid >> 6) * SB, j = (tid >> 2) & 15, s = tid & 3;
      float m[SB], l[DELTA ? SB : 1];
#pragma unroll
      for (int e = 0; e < SB; ++e) { m[e] = 0.f; if (DELTA) l[e] = 0.f; }
      for (int c = 4 * s; c < D; c += 16) {
        float4 x = *reinterpret_cast<const float4*>(K + (b + j) * LDD + c);
        if (BONUS) {
          const float4 u = load4(a.bonus + (long long)h * D + c);
          const float4 q = *reinterpret_cast<const float4*>(Q + (b + j) * LDD + c);
          m[0] = fmaf(q.x * x.x, u.x, fmaf(q.y * x.y, u.y, fmaf(q.z * x.z, u.z, fmaf(q.w * x.w, u.w, m[0]))));
        } else {
          m[0] = dot4(*reinterpret_cast<const float4*>(Q + (b + j) * LDD + c), x, m[0]);
        }
#pragma unroll
        for (int e = 1; e < SB; ++e) {
          if (j + e < SB) {
            const int t = (b + j + e) * LDD + c;
            const float4 d = *reinterpret_cast<const float4*>(A + t);
            if (BONUS) m[e] = dot4(*reinterpret_cast<const float4*>(Q + t), x, m[e]);
            x.x *= d.x; x.y *= d.y; x.z *= d.z; x.w *= d.w;
            if (!BONUS) m[e] = dot4(*reinterpret_cast<const float4*>(Q + t), x, m[e]);
            if (DELTA) l[e] = dot4(*reinterpret_cast<const float4*>(K + t), x, l[e]);
          }
        }
      }
#pragma unroll
      for (int e = 0; e < SB; ++e) {
        m[e] += __shfl_xor_sync(0xffffffffu, m[e], 1);
        m[e] += __shfl_xor_sync(0xffffffffu, m[e], 2);
        if (DELTA) { l[e] += __shfl_xor_sync(0xffffffffu, l[e], 1); l[e] += __shfl_xor_sync(0xffffffffu, l[e], 2); }
      }
      if (s == 0) {
#pragma unroll
        for (int e = 0; e < SB; ++e) {
          if (j + e < SB) {
            to.m[(b + j + e) * LC + b + j] = m[e];
            if (DELTA) to.w[(b + j + e) * LC + b + j] = e ? beta[b + j + e] * l[e] : 0.f;
          }
        }
      }
    }
    for (int x = tid; x < C * C; x += THREADS) {           // nothing above the diagonal
      const int t = x / C, j = x % C;
      if (j > t) { to.m[t * LC + j] = 0.f; if (DELTA) to.w[t * LC + j] = 0.f; }
    }
    __syncthreads();
    // rows scaled by the decays since their block's beginning (q, k), and k by those up to the block's end (in A's place)
    for (int x = tid; x < (C / SB) * D; x += THREADS) {
      const int b = x / D, c = x % D;
      float d[SB];
#pragma unroll
      for (int t = 0; t < SB; ++t) d[t] = A[(b * SB + t) * LDD + c];
      float p = 1.f;
#pragma unroll
      for (int t = SB - 1; t >= 0; --t) {
        A[(b * SB + t) * LDD + c] = K[(b * SB + t) * LDD + c] * p;
        p *= d[t];
      }
      blk[x] = p;
      p = 1.f;
#pragma unroll
      for (int t = 0; t < SB; ++t) {
        const int at = (b * SB + t) * LDD + c;
        if (BONUS) Q[at] *= p;
        p *= d[t];
        if (!BONUS) Q[at] *= p;
        if (DELTA) K[at] *= p;
      }
    }
    __syncthreads();
    const int t = tid >> 4, j = tid & 15;
#pragma unroll
    for (int I = 1; I < C / SB; ++I) {
      float m[C / SB - 1] = {}, l[C / SB - 1] = {};
      for (int c0 = 0; c0 < D; c0 += 16) {
        float mp[C / SB - 1] = {}, lp[C / SB - 1] = {};
#pragma unroll
        for (int c = c0; c < c0 + 16; c += 4) {
          const float4 q = *reinterpret_cast<const float4*>(Q + (I * SB + t) * LDD + c);
          float4 k;
          if (DELTA) k = *reinterpret_cast<const float4*>(K + (I * SB + t) * LDD + c);
#pragma unroll
          for (int J = 0; J < I; ++J) {
            const float4 x = *reinterpret_cast<const float4*>(A + (J * SB + j) * LDD + c);
            mp[J] = dot4(q, x, mp[J]);
            if (DELTA) lp[J] = dot4(k, x, lp[J]);
          }
        }
#pragma unroll
        for (int J = 0; J < I; ++J) { m[J] += mp[J]; if (DELTA) l[J] += lp[J]; }
      }
#pragma unroll
      for (int J = 0; J < I; ++J) {
        to.m[(I * SB + t) * LC + J * SB + j] = m[J];
        if (DELTA) to.w[(I * SB + t) * LC + J * SB + j] = beta[I * SB + t] * l[J];
      }
      __syncthreads();
      for (int x = tid; x < I * SB * NV; x += THREADS) {   // up to the end of block I
        const int c = x % NV * 4;
        float4* y = reinterpret_cast<float4*>(A + x / NV * LDD + c);
        const float4 d = *reinterpret_cast<const float4*>(blk + I * D + c);
        *y = make_float4(y->x * d.x, y->y * d.y, y->z * d.z, y->w * d.w);
      }
      __syncthreads();
    }
    for (int x = tid; x < C * NV; x += THREADS) {
      const int t2 = x / NV, c = x % NV * 4;
      float4 p = make_float4(1.f, 1.f, 1.f, 1.f);
      for (int b = 0; b < t2 / SB; ++b) {
        const float4 d = *reinterpret_cast<const float4*>(blk + b * D + c);
        p = make_float4(p.x * d.x, p.y * d.y, p.z * d.z, p.w * d.w);
      }
      const float4 q = *reinterpret_cast<const float4*>(Q + t2 * LDD + c);
      *reinterpret_cast<float4*>(to.qd + t2 * LDD + c) = make_float4(q.x * p.x, q.y * p.y, q.z * p.z, q.w * p.w);
      *reinterpret_cast<float4*>(to.kt + t2 * D + c) = *reinterpret_cast<const float4*>(A + t2 * LDD + c);
      if (DELTA) {
        float4* k = reinterpret_cast<float4*>(K + t2 * LDD + c);
        const float b = beta[t2];
        *k = make_float4(k->x * p.x * b, k->y * p.y * b, k->z * p.z * b, k->w * p.w * b);
      }
    }
    if (tid < D) to.pc[tid] = blk[tid] * blk[D + tid] * blk[2 * D + tid] * blk[3 * D + tid];
  }

  if constexpr (!DELTA) {
    for (int x = tid; x < C * (V / 4); x += THREADS) {
      const int t = x / (V / 4), c = x % (V / 4) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < n) v = load4(vg + (long long)(row0 + t) * a.v_ld + c);
      const float f = beta[t];
      *reinterpret_cast<float4*>(to.u + (c / 16 * C + t) * 16 + c % 16) = make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
    }
  } else {
    __syncthreads();                                       // Q is done with, L and K are whole
    if (PERCH) {
      for (int x = tid; x < C * LC / 4; x += THREADS) *reinterpret_cast<float4*>(G2 + 4 * x) = *reinterpret_cast<const float4*>(to.w + 4 * x);
      __syncthreads();
    }
    unit_lower_inverse(G2, G1, tmp);
    // W = X (beta P k), then X (beta v), D value columns at a time in Q's place
    const int rl = (warp & 1) * 32 + (lane >> 2), cl = (warp >> 1) * 16 + 4 * (lane & 3);
    for (int c = 0; c < D; c += 64) {
      float acc[4][4] = {};
      triangle_product(acc, G1 + rl * LC, LC, K + c + cl, LDD, warp & 1, lane >> 2);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(to.w + (rl + 8 * i) * LDD + c + cl) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
    for (int v0 = 0; v0 < V; v0 += D) {
      const int nv = min(D, V - v0);
      __syncthreads();
      for (int x = tid; x < C * (nv / 4); x += THREADS) {
        const int t = x / (nv / 4), c = x % (nv / 4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < n) v = load4(vg + (long long)(row0 + t) * a.v_ld + v0 + c);
        const float f = beta[t];
        *reinterpret_cast<float4*>(Q + t * LDD + c) = make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
      }
      __syncthreads();
      for (int c = 0; c + (warp >> 1) * 16 < nv; c += 64) {
        float acc[4][4] = {};
        triangle_product(acc, G1 + rl * LC, LC, Q + c + cl, LDD, warp & 1, lane >> 2);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<float4*>(to.u + ((v0 + c + cl) / 16 * C + rl + 8 * i) * 16 + cl % 16) =
              make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      }
    }
  }
}

// NC value columns a CTA (16, or 32 where there are CTAs enough), eight warps: for U two halves of the rows x four quarters of
// the channels, for S groups of 32 channels x parts of the tokens, tiles of 4 x 4 (x 2) a thread, partial sums joined through
// shared memory. (A row of U and two channels of S a thread over whole sums, without joining: 141 us against 109 at 16 heads
// of 128 x 128 and 2,048 tokens. What counts is the bytes that a sum's operands move out of shared memory: 128 a cycle, so
// that a 16-byte load costs a warp four cycles whether its lanes share addresses or not.)
template <int D, int NC, bool DELTA>
__global__ void __launch_bounds__(THREADS) chunk_carry_kernel(Args a) {
  pdl_launch();
  pdl_wait();
  constexpr int LDW = D + 4, NT = NC / 16, RG = D / 32, JG = 8 / RG;     // S: RG groups of 32 channels x JG parts of the tokens
  constexpr int STAGE = (DELTA ? C * LDW : 0) + C * D + C * NC + D;
  extern __shared__ __align__(128) float sm[];
  __shared__ __align__(8) uint64_t full[2];
  __shared__ int abort_flag;
  float* S = sm + 2 * STAGE;                             // [NT][D][16]
  float* part = S + D * NC;                              // [4][NT][C][16] sums of U, or [JG - 1][NT][D][16] of S
  const int h = blockIdx.y, v0 = blockIdx.z * NC, H = a.H, V = a.vdim;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int seq = 0, base = 0, chunks = 0;                     // the long sequence of this number, its first chunk, how many it has
  for (int before = 0; seq < a.num_seqs; ++seq) {
    chunks = chunks_of(a.cu_q[seq + 1] - a.cu_q[seq], a.long_from);
    if (chunks > 0 && before++ == (int)blockIdx.x) break;
    base += chunks;
  }
  if (seq == a.num_seqs) return;
  const int slot = a.state_slots ? a.state_slots[seq] : -1;
  float* sp = a.state + ((long long)(slot < 0 ? 0 : slot) * H + h) * D * V + v0;
  if (tid == 0) {
    abort_flag = 0;
    sm100::mbar_init(&full[0], 1);
    sm100::mbar_init(&full[1], 1);
    sm100::fence_barrier_init();
  }
  auto issue = [&](int ci) {                             // one thread
    const Place<D> in(a.scratch, (long long)(base + ci) * H + h, V, DELTA);
    float* ws = sm + (ci & 1) * STAGE;
    float* ks = ws + (DELTA ? C * LDW : 0);
    uint64_t* bar = &full[ci & 1];
    sm100::mbar_expect_tx(bar, STAGE * 4);
    if (DELTA) bulk(ws, in.w, C * LDW, bar);
    bulk(ks, in.kt, C * D, bar);
    bulk(ks + C * D, in.u + (long long)(v0 / 16) * C * 16, C * NC, bar);
    bulk(ks + C * D + C * NC, in.pc, D, bar);
  };
  if (tid == 0) {
    issue(0);
    if (chunks > 1) issue(1);
  }
  const int c = 4 * (lane & 3);
  for (int x = tid; x < D * (NC / 4); x += THREADS) {
    const int k = x / (NC / 4), v = x % (NC / 4) * 4;
    *reinterpret_cast<float4*>(S + (v / 16 * D + k) * 16 + v % 16) =
        slot >= 0 ? *reinterpret_cast<const float4*>(sp + (long long)k * V + v) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  for (int ci = 0; ci < chunks; ++ci) {
    const Place<D> in(a.scratch, (long long)(base + ci) * H + h, V, DELTA);
    float* ws = sm + (ci & 1) * STAGE;
    const float* ks = ws + (DELTA ? C * LDW : 0);
    float* us = ws + (DELTA ? C * LDW : 0) + C * D;      // [NT][C][16]
    const float* ps = us + C * NC;
    for (int x = tid; x < D * (NC / 4); x += THREADS)    // the state that the chunk meets
      *reinterpret_cast<float4*>(in.s + (long long)(v0 / 16) * D * 16 + 4 * x) = *reinterpret_cast<const float4*>(S + 4 * x);
    if (!landed(&full[ci & 1], (uint32_t)(ci >> 1) & 1u, &abort_flag, a.err, 41, ci + 1 < chunks ? &full[(ci + 1) & 1] : nullptr,
                (uint32_t)((ci + 1) >> 1) & 1u)) return;
    if (DELTA) {
      const int r = (warp & 1) * 32 + (lane >> 2), k0 = (warp >> 1) * (D / 4);
      float acc[NT][4][4] = {};
#pragma unroll 2
      for (int k = k0; k < k0 + D / 4; k += 4) {
        float4 x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(ws + (r + 8 * i) * LDW + k);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            const float4 y = *reinterpret_cast<const float4*>(S + (t * D + k + e) * 16 + c);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float xv = e == 0 ? x[i].x : e == 1 ? x[i].y : e == 2 ? x[i].z : x[i].w;
              acc[t][i][0] = fmaf(xv, y.x, acc[t][i][0]); acc[t][i][1] = fmaf(xv, y.y, acc[t][i][1]);
              acc[t][i][2] = fmaf(xv, y.z, acc[t][i][2]); acc[t][i][3] = fmaf(xv, y.w, acc[t][i][3]);
            }
          }
      }
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<float4*>(part + (((warp >> 1) * NT + t) * C + r + 8 * i) * 16 + c) =
              make_float4(acc[t][i][0], acc[t][i][1], acc[t][i][2], acc[t][i][3]);
      __syncthreads();
      for (int x = tid; x < C * (NC / 4); x += THREADS) {
        const float4 p0 = *reinterpret_cast<const float4*>(part + 4 * x), p1 = *reinterpret_cast<const float4*>(part + C * NC + 4 * x);
        const float4 p2 = *reinterpret_cast<const float4*>(part + 2 * C * NC + 4 * x), p3 = *reinterpret_cast<const float4*>(part + 3 * C * NC + 4 * x);
        float4 u = *reinterpret_cast<const float4*>(us + 4 * x);
        u.x -= (p0.x + p1.x) + (p2.x + p3.x); u.y -= (p0.y + p1.y) + (p2.y + p3.y);
        u.z -= (p0.z + p1.z) + (p2.z + p3.z); u.w -= (p0.w + p1.w) + (p2.w + p3.w);
        *reinterpret_cast<float4*>(us + 4 * x) = u;
        *reinterpret_cast<float4*>(in.u + (long long)(v0 / 16) * C * 16 + 4 * x) = u;
      }
      __syncthreads();
    }
    const int k = (warp % RG) * 32 + 4 * (lane >> 2), jg = warp / RG;
    float acc[NT][4][4] = {};
#pragma unroll 8
    for (int j = jg * (C / JG); j < (jg + 1) * (C / JG); ++j) {
      const float4 x = *reinterpret_cast<const float4*>(ks + j * D + k);
      const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const float4 y = *reinterpret_cast<const float4*>(us + (t * C + j) * 16 + c);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[t][i][0] = fmaf(xs[i], y.x, acc[t][i][0]); acc[t][i][1] = fmaf(xs[i], y.y, acc[t][i][1]);
          acc[t][i][2] = fmaf(xs[i], y.z, acc[t][i][2]); acc[t][i][3] = fmaf(xs[i], y.w, acc[t][i][3]);
        }
      }
    }
    if (jg > 0) {
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<float4*>(part + (((jg - 1) * NT + t) * D + k + i) * 16 + c) =
              make_float4(acc[t][i][0], acc[t][i][1], acc[t][i][2], acc[t][i][3]);
    }
    __syncthreads();
    if (jg == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float p = ps[k + i];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          float4* sv = reinterpret_cast<float4*>(S + (t * D + k + i) * 16 + c);
          float4 x = make_float4(acc[t][i][0], acc[t][i][1], acc[t][i][2], acc[t][i][3]);
#pragma unroll
          for (int g = 0; g < JG - 1; ++g) {
            const float4 y = *reinterpret_cast<const float4*>(part + ((g * NT + t) * D + k + i) * 16 + c);
            x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
          }
          *sv = make_float4(fmaf(p, sv->x, x.x), fmaf(p, sv->y, x.y), fmaf(p, sv->z, x.z), fmaf(p, sv->w, x.w));
        }
      }
    }
    __syncthreads();                                     // this stage is done with, S is whole
    if (tid == 0 && ci + 2 < chunks) {
      sm100::fence_proxy_async();
      issue(ci + 2);
    }
  }
  if (slot >= 0)
    for (int x = tid; x < D * (NC / 4); x += THREADS) {
      const int k = x / (NC / 4), v = x % (NC / 4) * 4;
      *reinterpret_cast<float4*>(sp + (long long)k * V + v) = *reinterpret_cast<const float4*>(S + (v / 16 * D + k) * 16 + v % 16);
    }
}

// O of a chunk: M U, then (P q) S on top, 64 value columns a CTA; the first product's operands (the smaller ones) land first.
template <typename TI, int D, bool DELTA>
__global__ void __launch_bounds__(THREADS, D == 64 ? 3 : 2) chunk_out_kernel(Args a) {
  pdl_launch();
  pdl_wait();
  constexpr int LDD = D + 4;
  extern __shared__ __align__(128) float sm[];
  __shared__ __align__(8) uint64_t full[2];
  __shared__ int abort_flag;
  float* M = sm;                                         // [C][LC]
  float* Q = M + C * LC;                                 // [C][LDD]
  float* U = Q + C * LDD;                                // [4][C][16]
  float* S = U + 4 * C * 16;                             // [4][D][16]
  int row0, n;
  if (!find_chunk(a, blockIdx.x, row0, n)) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int H = a.H, h = blockIdx.y, V = a.vdim, v0 = blockIdx.z * 64, tiles = min(4, (V - v0) / 16);
  if (tid == 0) {
    abort_flag = 0;
    sm100::mbar_init(&full[0], 1);
    sm100::mbar_init(&full[1], 1);
    sm100::fence_barrier_init();
    const Place<D> in(a.scratch, (long long)blockIdx.x * H + h, V, DELTA);
    sm100::mbar_expect_tx(&full[0], 4 * (C * LC + tiles * C * 16));
    bulk(M, in.m, C * LC, &full[0]);
    bulk(U, in.u + (long long)(v0 / 16) * C * 16, tiles * C * 16, &full[0]);
    sm100::mbar_expect_tx(&full[1], 4 * (C * LDD + tiles * D * 16));
    bulk(Q, in.qd, C * LDD, &full[1]);
    bulk(S, in.s + (long long)(v0 / 16) * D * 16, tiles * D * 16, &full[1]);
  }
  __syncthreads();
  const int tile = warp >> 1, r = (warp & 1) * 32 + (lane >> 2), c = 4 * (lane & 3);
  float acc[4][4] = {};
  const bool ok0 = landed(&full[0], 0, &abort_flag, a.err, 42);
  if (ok0 && tile < tiles)
    triangle_product(acc, M + r * LC, LC, U + tile * C * 16 + c, 16, warp & 1, lane >> 2);
  if (!landed(&full[1], 0, &abort_flag, a.err, 43) || !ok0 || tile >= tiles) return;
  float from[4][4] = {};                                 // apart from M U: where the state is small its parts would each round the whole sum
  tile_product(from, Q + r * LDD, LDD, S + tile * D * 16 + c, 16, D);
  add16(acc, from);
  const float skip = a.skip ? a.skip[h] : 0.f;
  const TI* vg = reinterpret_cast<const TI*>(a.v) + (long long)h * V + v0 + tile * 16 + c;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = r + 8 * i;
    if (t >= n) continue;
    float4 o = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    if (a.skip) {
      const float4 v = load4(vg + (long long)(row0 + t) * a.v_ld);
      o.x = fmaf(skip, v.x, o.x); o.y = fmaf(skip, v.y, o.y); o.z = fmaf(skip, v.z, o.z); o.w = fmaf(skip, v.w, o.w);
    }
    *reinterpret_cast<float4*>(a.out + ((long long)(row0 + t) * H + h) * V + v0 + tile * 16 + c) = o;
  }
}

// Sizes and alignments that the kernels take: heads of 64 or 128 key channels, value heads a multiple of 16, rows of four
// neighbouring numbers on a boundary of their size.
template <typename TI>
inline bool takes(const Args& a, int dim) {
  auto fits = [](const void* p, long long ld) { return !((uintptr_t)p % (4 * sizeof(TI))) && ld % 4 == 0; };
  return a.err != nullptr && (dim == 64 || dim == 128) && a.vdim > 0 && a.vdim % 16 == 0 && fits(a.q, a.q_ld) && fits(a.k, a.k_ld) && fits(a.v, a.v_ld) &&
         !((uintptr_t)a.decay & 15) && !((uintptr_t)a.state & 15) && !((uintptr_t)a.out & 15) && !((uintptr_t)a.bonus & 15) &&
         !((uintptr_t)a.scratch & 15) && a.H <= 65535 && a.vdim / 16 <= 65535;
}

// Floats of scratch a (chunk, head).
inline long long scratch_floats(int dim, int vdim, bool delta) {
  return dim == 64 ? Place<64>::floats(vdim, delta) : Place<128>::floats(vdim, delta);
}

template <typename TI, int D, bool PERCH, bool DELTA, bool BONUS>
int launch(const Args& a, int longs, int chunks, cudaStream_t s) {   // long sequences and their chunks, at most
  if (longs <= 0 || chunks <= 0) return 0;
  constexpr int LDD = D + 4;
  constexpr int INV = 3 * SB * (SB + 1), MATS = DELTA ? 2 * C * LC + INV : PERCH ? 0 : C * LC + 2 * C;    // from A on
  constexpr int OWN = PERCH ? C * LDD + 4 * D : 0;                                                        // A and blk
  constexpr size_t prep = sizeof(float) * (2 * C + 2 * C * LDD + (MATS > OWN ? MATS : OWN));
  constexpr size_t outs = sizeof(float) * (C * LC + C * LDD + 4 * C * 16 + 4 * D * 16);
  static bool ok_prep[64], ok_out[64], ok_16[64], ok_32[64];
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return -5;
  }
  auto prep_k = chunk_prep_kernel<TI, D, PERCH, DELTA, BONUS>;
  int rc = allow_dynamic_smem(prep_k, (int)prep, ok_prep);
  if (rc) return rc;
  rc = launch_ex(prep_k, dim3(chunks, a.H), dim3(THREADS), prep, s, 1, a);
  if (rc) return rc;
  auto carry = [&](auto kernel, int nc, bool (&ok)[64]) {
    const size_t stage = (DELTA ? C * (D + 4) : 0) + C * D + C * nc + D;
    constexpr int RG = D / 32, JG = 8 / RG;
    const size_t part = (size_t)nc * (DELTA && 4 * C > (JG - 1) * D ? 4 * C : (JG - 1) * D);
    const size_t bytes = sizeof(float) * (2 * stage + D * nc + part);
    const int rc2 = allow_dynamic_smem(kernel, (int)bytes, ok);
    return rc2 ? rc2 : launch_ex(kernel, dim3(longs, a.H, a.vdim / nc), dim3(THREADS), bytes, s, 1, a);
  };
  // 16 columns a CTA put twice as many CTAs on the walk; 32 read the rows of W and k half as often. The line is the number
  // of SMs: with more CTAs than that a walk of 16 columns is two waves long.
  if (a.vdim % 32 == 0 && (long long)longs * a.H * (a.vdim / 16) > sms)
    rc = carry(chunk_carry_kernel<D, 32, DELTA>, 32, ok_32);
  else
    rc = carry(chunk_carry_kernel<D, 16, DELTA>, 16, ok_16);
  if (rc) return rc;
  auto out_k = chunk_out_kernel<TI, D, DELTA>;
  rc = allow_dynamic_smem(out_k, (int)outs, ok_out);
  if (rc) return rc;
  return launch_ex(out_k, dim3(chunks, a.H, (a.vdim + 63) / 64), dim3(THREADS), outs, s, 1, a);
}

}  // namespace chunked
}  // namespace rllm
