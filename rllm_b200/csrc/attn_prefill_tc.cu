// Prefill attention over the paged bfloat16 cache on the 5th-generation tensor cores (tcgen05),
// head sizes 64 and 128: both products of a tile run as UMMA with their accumulators in TMEM.
// The text below gives the sizes for head size 64 (key tiles of 128); with 128 a key tile has 64
// keys, a row's scores are 64, and Q, K and V are two 128-byte atoms wide (see `Shape`).
//
// A work item is a pair of row tiles, 2 x 128 rows: (query token, query head) pairs of ONE kv head
// (row r of a sequence is token r / G, head kvh*G + r % G, as in the mma.sync kernel). Both tiles
// walk the keys they can see in tiles of 128 and share every K and V tile that is fetched:
//   warps 0..2  fetch the Q rows once and the K and V tiles through the block table into 128-byte
//               swizzled shared memory, three stages. Pages of a power of two from 8 keys up come
//               by TMA, one copy per page (or per 128 keys of a larger page) and cache, issued by
//               warp 0 alone and counted by the stage's mbarrier; any other page size comes by
//               16-byte cp.async, the three warps taking turns tile by tile, one stage each;
//   warp 3      one thread issues the products of both row tiles in turn:  S = Q K^T  (M 128,
//               N 128 keys, K 64) into the row tile's S accumulator, and  PV = P V  (M 128, N 64,
//               K 128 keys) with P read from TMEM and V as it lies in the cache tile (an
//               MN-major operand: the contraction runs over key rows);
//   warps 4..7  the softmax of the first row tile, one thread per row; warps 8..11 of the second.
//               A thread reads its row of S (128 scores) from TMEM, takes the maximum, exp2 and
//               the sum in float (scale, subtraction and sum two scores an instruction) and writes P
//               as bf16 over the scores' own columns, two keys a column. P used to go through shared
//               memory, in the swizzled layout of an A operand and behind a proxy fence, and a step
//               waited for the PV product before it with its exponentials: 595 us at 8,192 tokens (32 / 8
//               heads of 64) against 431, 58 against 49 at 2,048; heads of 128 688 against 626, 60 against 55.
//               What bounds a step is what its two warps a scheduler issue and wait for, not the
//               exponentials' unit: a quarter of them on the FMA pipe (a polynomial) cost 441 and 689 us,
//               an S accumulator a row tile with P beside it was slower too, but is faster at heads of 128 since one elected thread issues (Shape).
//               The row's output stays in TMEM, where PV of tile after tile is added up. The
//               exponentials are taken against a maximum that is moved only when the true one
//               has grown by more than 2^8 since (P then stays below 2^8, which bf16 holds as
//               well as values below 1); when it moves, the thread scales its row of the output
//               in TMEM (tcgen05.ld / st) before the next PV is added.
// The (row tile, K tile) steps are numbered k = 0, 1, ... in the order A0 B0 A1 B1 ... With heads of 64, and wherever scores are bounded, S of step k
// lands in accumulator k % 3 once PV of step k - 3, whose P lay there, is complete; keys of 128 and more with unbounded scores have an accumulator a row
// tile and P beside it (Shape). Either way, while both row tiles are in their softmax the scores of the step
// after are computed already, and a row tile that has written its P goes on at once: the four warp
// schedulers always have a warp with work (two warps each, one of either tile).
// TMEM: the S accumulators (and P) and PV of both tiles, 512 columns.
// Where a work item's two row tiles lie: next to each other, or (`fold`) as far from one end of the sequence's rows as from the other. Items of
// neighbours are as long as the keys they see, which balances where every CTA gets several; where the items are no more than the
// SMs, the longest is the launch, and folded ones are all alike. 16 / 4 heads of 128 over
// 2,048 tokens 42.3 -> 38.8 us, 512 over 512 with 32 / 8 heads of 64 15.0 -> 13.6; 16 heads of 192 / 128 over 2,048 62 -> 39.5 with both changes.
// A key j is visible when j <= position of the row and j > position - window, or when j <= position and j <
// keep_first (kept first keys): the tiles of the kept keys that the window's walk does not reach are walked first, then
// the window's, as one list. With `sigmoid` a visible key's weight is sigmoid(score + bias[head]) in place of the
// softmax's: no maximum, no rescaling, no denominator.
//
// Formulas: src/gpu/cuda/shaders/attention.cu:573-618 and :328-388 of the reference (scale,
// softmax with the maximum subtracted, weighted V, head h -> kv head h / G, window); unlike the
// reference's prefill kernel a portion also sees what earlier steps left in the cache.
// Every mbarrier wait is bounded; a wait that runs out records an error word and the CTA leaves
// in an orderly way (TMEM freed).
#include "common.cuh"
#include "sm100.cuh"
#include <mutex>
#include <type_traits>
#include <unordered_map>

using namespace rllm;
using namespace sm100;

namespace {

constexpr int PM = 128;          // rows per row tile
constexpr int RT = 2;            // row tiles per work item
constexpr int LOADERS = 3;       // loader warps
constexpr int MMA_WARP = LOADERS;
constexpr int SOFTMAX_WARP0 = LOADERS + 1;      // a multiple of 4: warp w reads TMEM lanes 32 (w % 4) ...
static_assert(SOFTMAX_WARP0 % 4 == 0, "softmax warp w must own TMEM lane quadrant w % 4");
constexpr int THREADS = (LOADERS + 1 + 4 * RT) * 32;
// registers per thread: 168 each at launch (65,536 / 384, in eights); then 4 warps keep 56 and 8 warps have 224
constexpr int REGS_LOW = 56, REGS_HIGH = 224;
static_assert(SOFTMAX_WARP0 * 32 * REGS_LOW + 4 * RT * 32 * REGS_HIGH <= 168 * THREADS, "more registers than the launch has");
                                 // K/V stages with TMA (one loader, tile after tile): Shape::KVS. Without TMA only LOADERS of them
                                 // are used: loader warp w always fills stage w (tiles w, w + 3, ...), so its waits
                                 // on that stage's barriers follow one another phase by phase; a warp that moved
                                 // between stages could be two phases ahead, which a parity cannot tell
constexpr int TMEM_COLS = 512;

// Sizes that follow from the head sizes: keys of KD and values of VD numbers, 64 / 64, 128 / 128 or 192 / 128. Operands lie in
// shared memory as "atoms" of 128-byte rows (64 values), swizzled: a tile wider than 64 values is several atoms one after
// the other. With keys of 192 the queries leave room for three stages.
template <int KD, int VD, bool CAP = false> struct Shape {
  static_assert((KD == 64 && VD == 64) || (KD == 128 && VD == 128) || (KD == 192 && VD == 128), "head sizes");
  static constexpr int PN = KD == 64 ? 128 : 64;     // keys per tile (a V tile is 16 KB either way)
  static constexpr int KVS = KD == 192 ? 3 : 4;      // K/V stages
  static constexpr int HA = KD / 64;                 // atoms along the head dimension (Q, K)
  static constexpr int VA = VD / 64;                 // (V)
  static constexpr int ATOM_ROWS = PM * 128;         // bytes of one atom of Q (128 rows)
  static constexpr int ATOM_KEYS = PN * 128;         // bytes of one atom of K or V (PN rows)
  static constexpr int K_BYTES = HA * ATOM_KEYS, V_BYTES = VA * ATOM_KEYS;     // one tile
  static constexpr int Q_BYTES = HA * ATOM_ROWS;     // one row tile of Q
  static constexpr int SMEM_BYTES = 1024 + RT * Q_BYTES + KVS * (K_BYTES + V_BYTES);   // Q[2], K[KVS], V[KVS]
  // TMEM: the S accumulators and P, then the output of both row tiles. Heads of 64: three accumulators that the steps take in turn, P of a
  // step in S's place. Keys of 128 and more, unbounded (BESIDE): an accumulator a row tile and P beside it, so that a row tile's next S is computed as
  // soon as its scores are in registers, and not when the PV of the step three before is complete. 8,192 tokens: heads of 128
  // 555 -> 497 us (2,048: 45.7 -> 42.3), heads of 64 410 -> 484; bounded scores (CAP), heads of 128, 741 -> 853.
  static constexpr bool BESIDE = KD > 64 && !CAP;
  static constexpr int SB = BESIDE ? RT : 3;
  static constexpr int S_COL = 0, P_COL = BESIDE ? RT * PN : 0, O_COL = BESIDE ? RT * PN + RT * PN / 2 : SB * PN;
  static_assert(O_COL + RT * VD <= TMEM_COLS, "S and the outputs must fit in TMEM");
};

struct PfParams {
  const bf16* q; int q_stride;
  const bf16* kc; const bf16* vc;
  bf16* out; int out_stride;
  const int* cu_q; const int* kv_lens; const int* block_table; int bt_stride;
  int nh, nkv, page_size, page_shift, window;
  int chunk;             // > 0: a row sees only the keys of its own block of this many positions
  const float* sinks;    // per head, or null: exp(sink) joins a row's denominator (no key, no value); with
                         // `sigmoid` the heads' biases instead
  int keep_first;        // positions below this number are seen whatever the window says
  int sigmoid;           // != 0: weights sigmoid(score + bias), not normalised
  const float* gate;     // float logits [T, gate_ld] or null: head h's output times sigmoid(gate[t, h])
  int gate_ld;
  SoftCap cap;           // cap.c > 0: scores are bounded, cap tanh(score / cap), before mask and softmax (the sink is not)
  float cap_z;           // scale / cap
  int box_rows;          // TMA variant: keys per copy = min(page size, 128)
  int row_pairs, num_seqs, sm_count;
  int fold;              // an item's row tiles are the i-th from either end of the sequence's (no window, no blocks)
  int long_from;         // CROSS, DENSE: sequences with fewer rows are left out (another kernel's)
  float* cross;          // not null: every query head meets every kv head's values, and the output is the floats
                         // [token][query head][kv head of the values][VD] here
  // DENSE: keys and values of a sequence lie one after the other (a row per position, the sequences that are not left out
  // in order), the maps see them as [heads][rows][128]; with KD 192 the last 64 numbers of a key are shared by the heads
  // (map tmap_r) and those of a query lie in rows of their own
  int q_head;            // numbers between a row's query heads
  const bf16* q2; long long q2_stride; int q2_head;
  const bf16* gate_h; int gate_h_ld, gate_cols;   // logits [T, gate_h_ld] or null: a column per head, or (gate_cols) per output
  float scale_log2e;
  int* err;
};

__device__ __forceinline__ float fast_rcp(float x) {           // 1 / inf = 0; relative error about 2^-23
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_exp2(float x) {          // exp2(-inf) = 0
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void cp_async16z(uint32_t dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;                         // 0 bytes read: the 16 bytes are zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ uint32_t bits_below(int n) { return n <= 0 ? 0u : n >= 32 ? 0xffffffffu : (1u << n) - 1u; }
// instruction descriptor: bf16 x bf16 -> f32, A K-major, B K-major or MN-major
__host__ __device__ constexpr uint32_t idesc(int M, int N, bool b_mn_major) {
  return umma_idesc_bf16(M, N) | (b_mn_major ? (1u << 16) : 0u);
}

// Two scores at a time: x = (x0, x1), bounded, in the log2 domain. tanh(z) = z P(z^2) on |z| <= 1 with a polynomial of
// degree 6 (interpolated at the Chebyshev points of [0, 1] in z^2: 4e-8 from tanh before rounding), which runs on the FMA
// pipe and leaves the transcendental unit to the softmax.
__device__ __forceinline__ uint64_t f32x2(float a, float b) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void split2(uint64_t d, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(d));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ void softcap_poly2(uint32_t& x0, uint32_t& x1, float zscale, float c) {
  const uint64_t z = mul2(f32x2(__uint_as_float(x0), __uint_as_float(x1)), f32x2(zscale, zscale));
  const uint64_t t = mul2(z, z);
  uint64_t q = fma2(t, f32x2(0.0010380251f, 0.0010380251f), f32x2(-0.00619432483f, -0.00619432483f));
  q = fma2(q, t, f32x2(0.0202797083f, 0.0202797083f));
  q = fma2(q, t, f32x2(-0.0534516464f, -0.0534516464f));
  q = fma2(q, t, f32x2(0.133250761f, 0.133250761f));
  q = fma2(q, t, f32x2(-0.33332828f, -0.33332828f));
  q = fma2(q, t, f32x2(0.999999949f, 0.999999949f));
  const uint64_t r = mul2(mul2(z, f32x2(c, c)), q);
  asm("mov.b64 {%0, %1}, %2;" : "=r"(x0), "=r"(x1) : "l"(r));
}

// TMA: the K and V tiles come by tensor copies over the caches seen as [pages * kv heads][page size][HD].
// CAP: scores are bounded (p.cap).
// MODE PLAIN: pages. CROSS: pages, every head over every kv head's values, float outputs (PfParams). DENSE: keys and values in
// rows, by tensor copies of whole tiles.
enum : int { PLAIN = 0, CROSS = 1, DENSE_ROWS = 2 };
template <int KD, int VD, bool TMA, bool CAP, int MODE>
__global__ void __launch_bounds__(THREADS, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                       const __grid_constant__ CUtensorMap tmap_r, const PfParams p) {
  constexpr bool DENSE = MODE == DENSE_ROWS;
  static_assert(TMA || MODE == PLAIN, "the other forms come by tensor copies");
  typedef Shape<KD, VD, CAP> C;
  constexpr int KVS = C::KVS, SB = C::SB;
  constexpr bool BESIDE = C::BESIDE;
  extern __shared__ uint8_t pf_smem_raw[];
  __shared__ __align__(8) uint64_t kv_full[KVS], kv_empty[KVS], s_full[SB], s_free[SB], p_full[RT], pv_full[RT], q_full;
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* smem = (uint8_t*)(((uintptr_t)pf_smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int PN = C::PN;
  const uint32_t q_s = smem_u32(smem);
  const uint32_t k_s = q_s + RT * C::Q_BYTES, v_s = k_s + KVS * C::K_BYTES;

  const int G = p.nh / p.nkv;
  constexpr int NST = TMA ? KVS : LOADERS;              // K/V stages in use
  if (threadIdx.x == 0) abort_flag = 0;
  if (TMA) {
    // A copy brings whole pages: rows past a sequence's last key keep what the stage held before.
    // The scores of such keys are masked, and their weights are exact zeros, but zero times what
    // an earlier kernel left here need not be zero: start from zeros (later leftovers are keys).
    if (warp == 0 && lane == 0) { prefetch_tensormap(&tmap_k); prefetch_tensormap(&tmap_v); }
    uint4* kv = reinterpret_cast<uint4*>(smem + RT * C::Q_BYTES);
    for (int i = threadIdx.x; i < KVS * (C::K_BYTES + C::V_BYTES) / 16; i += THREADS) kv[i] = make_uint4(0, 0, 0, 0);
    fence_proxy_async();
  }
  if (warp == MMA_WARP) { tmem_alloc(&tmem_base_slot, TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch();
  pdl_wait();                                           // q and the newest keys come from the kernel before
  const uint32_t tmem_base = tmem_base_slot;

  // The CTAs (one per SM) share the (pair of row tiles, kv head, sequence) items out among
  // themselves: items are numbered from the row tiles that see the most keys down, and round r
  // gives CTA c item r * C + c, or r * C + (C - 1 - c) in odd rounds, so that every CTA gets a
  // like share of long and short ones.
  // The warps 0..3 (loaders, products) need few registers, the softmax warps many (a row of 128
  // scores each): the first warpgroup gives registers up, the other two take them, and each side
  // walks the items in its own copy of the loop (the block-wide barriers are the same ones).
  auto walk = [&](auto softmax_side) {
  constexpr bool SOFTMAX = decltype(softmax_side)::value;
  const int vheads = MODE == CROSS ? p.nkv : 1;
  const int items = p.row_pairs * p.nkv * vheads * p.num_seqs;
  for (int round = 0;; ++round) {
  const int item = round * (int)gridDim.x + ((round & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
  if (item >= items) break;
  const int place = item / (p.nkv * vheads * p.num_seqs);
  const int kvh = item % p.nkv, seq = (item / (p.nkv * vheads)) % p.num_seqs;
  const int vh = MODE == CROSS ? item / p.nkv % p.nkv : kvh;                         // the kv head of the values
  // the item's row tiles, the second at least as late as the first. An item beyond its sequence's rows (a short portion beside long
  // ones) is skipped by all threads alike
  const int n_rows = ((p.cu_q[seq + 1] - p.cu_q[seq]) * G + PM - 1) / PM;              // row tiles that the sequence has
  int tile[RT];
  if (p.fold) { tile[1] = n_rows - 1 - place; tile[0] = place < tile[1] ? place : n_rows; }
  else { tile[0] = (p.row_pairs - 1 - place) * RT; tile[1] = tile[0] + 1; }
  if (p.fold ? place > tile[1] : tile[0] >= n_rows) continue;
  if (MODE != PLAIN && p.cu_q[seq + 1] - p.cu_q[seq] < p.long_from) continue;
  __syncthreads();                                      // everybody has left the item before
  if (threadIdx.x == 0) {
    for (int i = 0; i < KVS; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
    for (int i = 0; i < SB; ++i) { mbar_init(&s_full[i], 1); mbar_init(&s_free[i], BESIDE ? 4 : 1); }
    for (int i = 0; i < RT; ++i) { mbar_init(&p_full[i], 4); mbar_init(&pv_full[i], 1); }
    mbar_init(&q_full, TMA ? 4 * RT : RT);             // TMA: one arrival per softmax warp, which brings its own rows of Q
    fence_barrier_init();
  }
  __syncthreads();
  if (abort_flag) break;                                // a wait ran out in an earlier item: the kernel's output is void anyway

  const int q0 = p.cu_q[seq];
  const int q_len = p.cu_q[seq + 1] - q0;
  const int kv_len = p.kv_lens[seq];
  const int rows_total = q_len * G;
  // keys the item's rows can see at all: from the first row's window (or 0) to the last row's position.
  // The later row tile sees at least as far as the earlier one; both start from the same tile.
  // With kept first keys the tiles [0, n_kept) of those keys come first in the list (only the ones that lie wholly
  // before the window's first tile; a kept key inside the window's tiles is seen there).
  int kv_begin = 0, n_kept = 0, n_t[RT];
  {
    const int p_min = kv_len - q_len + (min(tile[0], tile[1]) * PM) / G;
    int first = (p.window > 0 && p_min - p.window + 1 > 0) ? p_min - p.window + 1 : 0;
    if (p.chunk > 0) first = max(first, p_min / p.chunk * p.chunk);
    kv_begin = first / PN * PN;
    n_kept = min((min(p.keep_first, first) + PN - 1) / PN, kv_begin / PN);
#pragma unroll
    for (int g = 0; g < RT; ++g) {
      const bool active = tile[g] < n_rows;                      // uniform: a row tile beyond the sequence's rows is empty
      const int p_max = kv_len - q_len + min(q_len - 1, (tile[g] * PM + PM - 1) / G);
      n_t[g] = active ? n_kept + (p_max + 1 - kv_begin + PN - 1) / PN : 0;
    }
  }
  auto tile_first = [&](int t) { return t < n_kept ? t * PN : kv_begin + (t - n_kept) * PN; };   // first key of tile t of the list
  const int n_tiles = max(n_t[0], n_t[1]);
  // step k is (row tile, K tile) = (k & 1, k >> 1) while both row tiles have tiles left, then the later one alone
  const int n_both = min(n_t[0], n_t[1]), g_long = n_t[1] > n_t[0] ? 1 : 0, n_steps = n_t[0] + n_t[1];

  // Q rows r0 .. r0 + n - 1 of the item (one warp), rows beyond the sequence zero
  auto load_q = [&](int r0, int n) {
    const int ch = lane & 7, rbase = lane >> 3;
#pragma unroll 4
    for (int i = 0; i < n / 4; ++i) {
      const int r = r0 + rbase + 4 * i;                  // row of the item: row tile r / 128, row r % 128 of it
      const int row = tile[r / PM] * PM + r % PM;
      const bool valid = row < rows_total;
      const int tok = valid ? row / G : 0, head = kvh * G + (valid ? row % G : 0);
      const bf16* src = p.q + (size_t)(q0 + tok) * p.q_stride + (size_t)head * KD + ch * 8;
      const uint32_t dst = q_s + (uint32_t)((r / PM) * C::Q_BYTES + (r % PM) * 128 + ((ch ^ (r & 7)) << 4));
#pragma unroll
      for (int a = 0; a < C::HA; ++a) cp_async16z(dst + (uint32_t)(a * C::ATOM_ROWS), src + a * 64, valid);
    }
  };

  if constexpr (!SOFTMAX) {
  // ---- the products. Step k is (row tile g, K tile t); its S lands in accumulator acc_of(k, g), used for the turn_of(k, t)-th time.
  constexpr uint32_t id_s = idesc(PM, PN, false);
  constexpr uint32_t id_pv = idesc(PM, 64, true);       // 64 output values at a time
  auto step = [&](int k, int& g, int& t) {
    if (k < 2 * n_both) { g = k & 1; t = k >> 1; } else { g = g_long; t = n_both + (k - 2 * n_both); }
  };
  auto acc_of = [&](int k, int g) { return BESIDE ? g : k % SB; };
  auto turn_of = [&](int k, int t) { return BESIDE ? t : k / SB; };
  // descriptors move with the address: 16 bytes are one unit of the start-address field
  const uint64_t dq0 = umma_desc_sw128(q_s), dk0 = umma_desc_sw128(k_s), dv0 = umma_desc_sw128(v_s);
  auto issue_s = [&](int k, bool& ok) {                 // S = Q K^T of step k (one thread)
    int g, t;
    step(k, g, t);
    const int ks = t % NST;
    if (BESIDE ? t > 0 : k >= SB) {
      // BESIDE: the row tile's threads have its scores before in their registers; else the PV product of step k - 3 is complete, whose P
      // lay in the accumulator's place
      if (!mbar_wait(&s_free[acc_of(k, g)], (uint32_t)(turn_of(k, t) - 1) & 1u, &abort_flag)) {
        abort_flag = 1; record_failure(p.err, 28, k); ok = false; return;
      }
    }
    if (!mbar_wait(&kv_full[ks], (uint32_t)(t / NST) & 1u, &abort_flag)) {
      abort_flag = 1; record_failure(p.err, 22, t); ok = false; return;
    }
    tc_fence_after();
    const uint64_t dq = dq0 + (uint64_t)(g * (C::Q_BYTES >> 4)), dk = dk0 + (uint64_t)(ks * (C::K_BYTES >> 4));
    const uint32_t acc = tmem_base + C::S_COL + (uint32_t)acc_of(k, g) * PN;
#pragma unroll
    for (int kk = 0; kk < KD / 16; ++kk)                // 16 values a product: atom kk / 4, 32 bytes on within it
      umma_bf16(acc, dq + (uint64_t)((kk >> 2) * (C::ATOM_ROWS >> 4) + (kk & 3) * 2),
                dk + (uint64_t)((kk >> 2) * (C::ATOM_KEYS >> 4) + (kk & 3) * 2), id_s, kk > 0);
    umma_commit(&s_full[acc_of(k, g)]);
  };
  auto issue_pv = [&](int k, bool& ok) {                // PV of step k, added to the row tile's output (one thread)
    int g, t;
    step(k, g, t);
    // P of this step is written (and the row tile's PV before is complete: its threads waited for it)
    if (!mbar_wait(&p_full[g], (uint32_t)t & 1u, &abort_flag)) {
      abort_flag = 1; record_failure(p.err, 23, t); ok = false; return;
    }
    tc_fence_after();
    const uint64_t dv = dv0 + (uint64_t)((t % NST) * (C::V_BYTES >> 4));
    const uint32_t acc = tmem_base + C::O_COL + (uint32_t)g * VD, pa = tmem_base + (BESIDE ? C::P_COL + (uint32_t)g * (PN / 2) : C::S_COL + (uint32_t)(k % SB) * PN);
#pragma unroll
    for (int a = 0; a < C::VA; ++a)                     // 64 output values = one atom of V
#pragma unroll
      for (int ks = 0; ks < PN / 16; ++ks)
        // P: 16 keys are 8 columns; V: MN-major, 16 key rows = 2 KB per step
        umma_bf16_ts(acc + (uint32_t)(a * 64), pa + (uint32_t)(ks * 8), dv + (uint64_t)(a * (C::ATOM_KEYS >> 4) + ks * (2048 >> 4)),
                     id_pv, t > 0 || ks > 0);
    umma_commit(&pv_full[g]);
    if (!BESIDE) umma_commit(&s_free[k % SB]);
    if (g == 1 || t >= n_both) umma_commit(&kv_empty[t % NST]);     // the last reader of this K and V stage
  };
  if (warp < LOADERS && TMA) {
    // ------------------------------------------------------------ loader (TMA): warp 0 alone, tile after tile.
    // Lane c looks up the page of the tile's c-th copy; lane 0 tells the stage's barrier how many
    // bytes are coming; every lane with a page issues its two copies. Nothing waits for a tile to
    // land: up to NST tiles are on their way.
    if (warp == 0 && DENSE) {
      // a lane a copy: the atoms of K that are the head's own, those of V, the one of K that the heads share
      int base = 0;                                        // the sequence's first row: the keys of those before it
      for (int i = lane; i < seq; i += 32) base += p.cu_q[i + 1] - p.cu_q[i] < p.long_from ? 0 : p.kv_lens[i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) base += __shfl_xor_sync(0xffffffffu, base, o);
      constexpr int KO = KD == 192 ? 2 : C::HA;
      for (int t = 0; t < n_tiles; ++t) {
        const int s = t % NST;
        if (t >= NST) {
          int w_ok = 1;
          if (lane == 0 && !mbar_wait(&kv_empty[s], (uint32_t)(t / NST - 1) & 1u, &abort_flag)) {
            abort_flag = 1; record_failure(p.err, 21, t); w_ok = 0;
          }
          if (__shfl_sync(0xffffffffu, w_ok, 0) == 0) break;
        }
        if (lane == 0) mbar_expect_tx(&kv_full[s], C::K_BYTES + C::V_BYTES);
        __syncwarp();
        const int row = base + tile_first(t);
        const uint32_t kd = k_s + (uint32_t)(s * C::K_BYTES), vd = v_s + (uint32_t)(s * C::V_BYTES);
        if (lane < KO) tma_load_3d(kd + (uint32_t)(lane * C::ATOM_KEYS), &tmap_k, &kv_full[s], lane * 64, row, kvh);
        else if (lane < KO + C::VA) tma_load_3d(vd + (uint32_t)((lane - KO) * C::ATOM_KEYS), &tmap_v, &kv_full[s], (lane - KO) * 64, row, kvh);
        else if (KD == 192 && lane == KO + C::VA) tma_load_3d(kd + (uint32_t)(2 * C::ATOM_KEYS), &tmap_r, &kv_full[s], 0, row, 0);
      }
    } else if (warp == 0) {
      const int* bt = p.block_table + (size_t)seq * p.bt_stride;
      const int copies = PN / p.box_rows;                  // runs of keys per tile; each is one copy per atom and cache
      const uint32_t copy_bytes = (uint32_t)p.box_rows * 128;
      const int cp = lane / C::HA, at = lane % C::HA;      // this lane's run of keys and its atom of 64 values
      for (int t = 0; t < n_tiles; ++t) {
        const int s = t % NST;
        if (t >= NST) {
          int w_ok = 1;
          if (lane == 0 && !mbar_wait(&kv_empty[s], (uint32_t)(t / NST - 1) & 1u, &abort_flag)) {
            abort_flag = 1; record_failure(p.err, 21, t); w_ok = 0;
          }
          if (__shfl_sync(0xffffffffu, w_ok, 0) == 0) break;
        }
        const int j = tile_first(t) + cp * p.box_rows;                  // first key of this lane's copy
        const bool mine = cp < copies && j < kv_len;
        const int page = mine ? __ldg(bt + (j >> p.page_shift)) : 0;
        const uint32_t n = __popc(__ballot_sync(0xffffffffu, mine));
        if (lane == 0) mbar_expect_tx(&kv_full[s], 2 * n * copy_bytes);
        __syncwarp();
        if (mine) {
          const uint32_t dst = (uint32_t)(s * C::K_BYTES) + (uint32_t)at * C::ATOM_KEYS + (uint32_t)cp * copy_bytes;
          const int off = j & (p.page_size - 1);
          tma_load_3d(k_s + dst, &tmap_k, &kv_full[s], at * 64, off, page * p.nkv + kvh);
          tma_load_3d(v_s + dst, &tmap_v, &kv_full[s], at * 64, off, page * p.nkv + vh);
        }
      }
    } else if (warp == 2) {
      // (Q comes from the softmax warps, each thread its own row: one warp fetching a row tile spent 5 us
      // of every item on the addresses of its 1,024 copies)
      if (elect_one() && n_steps > 0) {
        // ... and warp 2 then issues the S products, as far ahead as accumulators are free
        bool ok = true;
        if (!mbar_wait(&q_full, 0u, &abort_flag)) { abort_flag = 1; record_failure(p.err, 27, 0); ok = false; }
        for (int k = 0; k < n_steps && ok; ++k) issue_s(k, ok);
      }
    }
  } else if (warp < LOADERS) {
    // ------------------------------------------------------------ loaders (any page size): warp w fetches the
    // tiles w, w + 3, ... whole, waits until they have landed and announces them at once, so a
    // tile is ready long before its turn (up to NST tiles are on the way, from different warps).
    const int* bt = p.block_table + (size_t)seq * p.bt_stride;
    const int ch = lane & 7;                              // this lane's 16-byte chunk of a 128-byte row
    const int rbase = lane >> 3;                          // its rows: rbase + 4 i, i < PN / 4
    for (int t = warp; t < n_tiles; t += LOADERS) {
      const int s = t % NST;
      if (t >= NST) {
        int w_ok = 1;
        if (lane == 0 && !mbar_wait(&kv_empty[s], (uint32_t)(t / NST - 1) & 1u, &abort_flag)) {
          abort_flag = 1; record_failure(p.err, 21, t); w_ok = 0;
        }
        if (__shfl_sync(0xffffffffu, w_ok, 0) == 0) break;
      }
      if (t == 0) load_q(0, RT * PM);                     // lands with the tile, announced by its barrier
      const int j0 = tile_first(t);
      const uint32_t kd = k_s + (uint32_t)(s * C::K_BYTES), vd = v_s + (uint32_t)(s * C::V_BYTES);
#pragma unroll 1
      for (int i0 = 0; i0 < PN / 4; i0 += 8) {
        int page[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {                     // eight page lookups in flight together
          const int j = j0 + rbase + 4 * (i0 + i);
          const int pg = p.page_shift >= 0 ? (j >> p.page_shift) : j / p.page_size;
          page[i] = j < kv_len ? __ldg(bt + pg) : -1;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = rbase + 4 * (i0 + i);
          const int j = j0 + r;
          const int off = p.page_shift >= 0 ? (j & (p.page_size - 1)) : j % p.page_size;
          const bool valid = page[i] >= 0;
          const size_t src = valid ? ((((size_t)page[i] * p.nkv + kvh) * p.page_size + off) * KD + ch * 8) : 0;
          const uint32_t dst = (uint32_t)(r * 128 + ((ch ^ (r & 7)) << 4));
#pragma unroll
          for (int a = 0; a < C::HA; ++a) {
            cp_async16z(kd + dst + (uint32_t)(a * C::ATOM_KEYS), p.kc + src + a * 64, valid);
            cp_async16z(vd + dst + (uint32_t)(a * C::ATOM_KEYS), p.vc + src + a * 64, valid);
          }
        }
      }
      cp_async_commit();
      cp_async_wait<0>();                                 // the tile has landed
      fence_proxy_async();                                // for the tensor core's reads
      __syncwarp();
      if (lane == 0) mbar_arrive(&kv_full[s]);
    }
  } else if (warp == MMA_WARP) {
    // ------------------------------------------------------------ the PV products (one thread); without
    // TMA the loaders are all busy and this thread issues S as well
    if (elect_one() && n_tiles > 0) {
      bool ok = true;
      const int ahead = BESIDE ? (n_both > 0 ? 2 : 1) : SB;       // without TMA: steps that S is ahead of PV
      if (!TMA)
        for (int k = 0; k < ahead && k < n_steps && ok; ++k) issue_s(k, ok);
      for (int k = 0; k < n_steps && ok; ++k) {
        if (!TMA && BESIDE && k + ahead < n_steps) issue_s(k + ahead, ok);
        if (ok) issue_pv(k, ok);
        if (!TMA && !BESIDE && ok && k + ahead < n_steps) issue_s(k + ahead, ok);
      }
      // nothing of this item may still be on its way to a barrier when the next item sets them up again (BESIDE: S and the last PV have been
      // waited for by the softmax warps)
      for (int k = max(0, n_steps - SB); !BESIDE && k < n_steps && ok; ++k)
        if (!mbar_wait(&s_free[k % SB], (uint32_t)(k / SB) & 1u, &abort_flag)) {
          abort_flag = 1; record_failure(p.err, 29, k); ok = false;
        }
      for (int t = max(0, n_tiles - NST); t < n_tiles && ok; ++t)
        if (!mbar_wait(&kv_empty[t % NST], (uint32_t)(t / NST) & 1u, &abort_flag)) {
          abort_flag = 1; record_failure(p.err, 26, t); ok = false;
        }
    }
  }
  } else {
  if (n_t[(warp - SOFTMAX_WARP0) >> 2] > 0) {
    // ------------------------------------------------------------ softmax warps: one thread per row
    const int g = (warp - SOFTMAX_WARP0) >> 2;           // the row tile
    const int n_mine = n_t[g];
    const int quad = warp & 3;                            // the TMEM lanes this warp may read: 32 quad ...
    const int r = quad * 32 + lane;
    const int row = tile[g] * PM + r;
    const bool valid = row < rows_total;
    const int tok = valid ? row / G : 0, head = kvh * G + (valid ? row % G : 0);
    const int pos = valid ? kv_len - q_len + tok : kv_len - 1;      // a row beyond the sequence: zeros that look on like the last one's
    int lo = p.window > 0 ? pos - p.window + 1 : 0;
    if (p.chunk > 0) lo = max(lo, pos / p.chunk * p.chunk);
    if (TMA) {
      // this thread's own row of Q into the A-operand layout (rows beyond the sequence zero), while the
      // first K and V tiles are on their way
      const bf16* src = p.q + (size_t)(q0 + tok) * p.q_stride + (size_t)head * (DENSE ? p.q_head : KD);
      const bf16* src2 = KD == 192 ? p.q2 + (size_t)(q0 + tok) * p.q2_stride + (size_t)head * p.q2_head : src;
      const uint32_t drow = q_s + (uint32_t)(g * C::Q_BYTES + r * 128);
#pragma unroll
      for (int a = 0; a < C::HA; ++a)
#pragma unroll
        for (int ch = 0; ch < 8; ++ch)
          cp_async16z(drow + (uint32_t)(a * C::ATOM_ROWS) + (uint32_t)((ch ^ (r & 7)) << 4), (KD == 192 && a == 2 ? src2 : src + a * 64) + ch * 8, valid);
      cp_async_commit();
      cp_async_wait<0>();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&q_full);
    }
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
    const uint32_t pv_addr = lane_addr + C::O_COL + (uint32_t)g * VD;
    constexpr int NC = PN / 32;                           // the row's scores come 32 at a time
    const float sl = CAP ? 1.f : p.scale_log2e;        // bounded scores leave the bound in the log2 domain
    // m: what the exponentials are taken against, up to 2^8 behind the true maximum. A sink opens the row's
    // running softmax as a key of score `sink` (not scaled) and value zero.
    const bool sig = p.sigmoid != 0;
    const bool sunk = !sig && p.sinks != nullptr && valid;
    float m = sunk ? p.sinks[head] * 1.4426950408889634f : -INFINITY, l = sunk ? 1.f : 0.f;
    const float sb = (sig && p.sinks != nullptr && valid) ? p.sinks[head] * 1.4426950408889634f : 0.f;   // the bias, log2 domain
    const int kf = p.keep_first;
    bool ok = true;

    auto wait_on = [&](uint64_t* bar, uint32_t parity, int role, int t) -> bool {
      bool got = mbar_wait(bar, parity, &abort_flag);
      if (!got) { abort_flag = 1; record_failure(p.err, role, t); }
      return __all_sync(0xffffffffu, got);
    };

    for (int t = 0; t < n_mine; ++t) {
      const int j0 = tile_first(t);
      const int k = t < n_both ? 2 * t + g : 2 * n_both + (t - n_both);
      const int sa = BESIDE ? g : k % SB;
      const uint32_t s_addr = lane_addr + C::S_COL + (uint32_t)sa * PN;          // this step's S accumulator
      const uint32_t p_addr = BESIDE ? lane_addr + C::P_COL + (uint32_t)g * (PN / 2) : s_addr;
      if (!wait_on(&s_full[sa], (uint32_t)(BESIDE ? t : k / SB) & 1u, 24, t)) { ok = false; break; }
      tc_fence_after();
      // ---- the row's PN scores, the hidden ones -inf, and their maximum
      uint32_t v[NC][32];
#pragma unroll
      for (int c = 0; c < NC; ++c) tmem_ld32(s_addr + 32 * c, v[c]);
      tmem_ld_wait();
      if (BESIDE) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_free[g]);           // the row tile's next S may be computed
      }
      if (CAP) {
        float far[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          far[c] = 0.f;
#pragma unroll
          for (int i = 0; i < 32; i += 2) far[c] = fmax3(far[c], fabsf(__uint_as_float(v[c][i])), fabsf(__uint_as_float(v[c][i + 1])));
        }
        float mz = far[0];
#pragma unroll
        for (int c = 1; c < NC; ++c) mz = fmaxf(mz, far[c]);
        if (__all_sync(0xffffffffu, mz * fabsf(p.cap_z) <= 1.f)) {        // every score of the warp's rows within the bound
#pragma unroll
          for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int i = 0; i < 32; i += 2) softcap_poly2(v[c][i], v[c][i + 1], p.cap_z, p.cap.c);
        } else {
#pragma unroll
          for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i) v[c][i] = __float_as_uint(softcap_log2(__uint_as_float(v[c][i]), p.cap));
        }
      }
      const bool hides = j0 + PN - 1 > pos || (j0 < lo && j0 + PN > kf);      // some key is hidden from this row
      if (hides) {
        // A bit a key of each 32: not after the row's position, and not before its window unless kept. With the conditions spelled
        // out key by key a tile that hides keys cost 3.5 us more than one that does not (now 0.2), and rows beyond the sequence's, which
        // used to hide every key, cost it in every tile: 1,905 tokens over 6,001 keys (32 / 8
        // heads of 64) 269 us, now 140; 76 over 1,100 54, now 23; 512 over 512 20.6, now 15.0; 2,048 over 2,048 50.7, now 40.4.
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const int j = j0 + 32 * c;
          const uint32_t seen = bits_below(pos + 1 - j) & (~bits_below(lo - j) | bits_below(kf - j));
#pragma unroll
          for (int i = 0; i < 32; ++i) v[c][i] = (seen >> i) & 1u ? v[c][i] : 0xff800000u;
        }
        // The copies of the last tile brought rows beyond the sequence: another request's, or what a page's last holder left.
        // Their weights are zero, but zero times an infinity is not: those rows of V become zeros before the product reads them
        // (both row tiles' threads may write the same zeros; V landed with K, whose product is done). Every row has hidden keys in
        // such a tile; in front of `p_full` instead, or by a loader's warp, 8,192 tokens cost 1 to 4 % more.
        if (TMA && j0 + PN > kv_len) {
          if (r < PN && j0 + r >= kv_len) {
            const uint32_t vrow = v_s + (uint32_t)(t % NST * C::V_BYTES + r * 128);
#pragma unroll 1
            for (int i = 0; i < C::VA * 8; ++i)
              asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(vrow + (uint32_t)((i >> 3) * C::ATOM_KEYS + (i & 7) * 16)), "r"(0) : "memory");
          }
          fence_proxy_async();
        }
      }
      float mq[NC];                                       // chains side by side, not one of 64 links
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        mq[c] = -INFINITY;
#pragma unroll
        for (int i = 0; i < 32; i += 2) mq[c] = fmax3(mq[c], __uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1]));
      }
      float mx = mq[0];
#pragma unroll
      for (int c = 1; c < NC; ++c) mx = fmaxf(mx, mq[c]);
      const float cand = fmaxf(m, mx * sl);               // the scale is positive: it commutes with max
      const bool move = !sig && cand > m + 8.f;           // also the first visible key (m = -inf)
      float corr = 1.f;
      if (move) { corr = fast_exp2(m - cand); m = cand; l *= corr; }      // exp2(-inf) = 0
      // PV of the tile before has to be complete where the output is touched, or (BESIDE) where its P lies in this one's place; else the
      // wait comes behind the exponentials (a phase is never skipped, so that a parity says which one it is)
      auto pv_before = [&]() { return t == 0 || wait_on(&pv_full[g], (uint32_t)(t - 1) & 1u, 25, t); };
      const bool moves = __any_sync(0xffffffffu, move);
      if (BESIDE || moves) {
        if (!pv_before()) { ok = false; break; }
      }
      if (moves) {
        if (t > 0) {
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < VD / 16; ++c) {
            uint32_t ov[16];
            tmem_ld16(pv_addr + 16 * c, ov);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * corr);
            tmem_st16(pv_addr + 16 * c, ov);
          }
        }
      }
      // ---- exponentials, their sum, P as bf16 into the scores' place, two keys a column
      const float use = (m == -INFINITY) ? 0.f : m;
      // two scores an instruction where the pipe takes two: what bounds a step is the instructions its warps issue
      const uint64_t sl2 = f32x2(sl, sl), use2 = f32x2(-use, -use);
      uint64_t lq[4];                                     // eight partial sums side by side, added up in a fixed order
#pragma unroll
      for (int i = 0; i < 4; ++i) lq[i] = f32x2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        uint32_t pk[16];
        if (sig) {
          // sigmoid(x) = 1 / (1 + 2^(-x log2 e)); hidden keys hold -inf: 1 / (1 + inf) = 0
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float e0 = fast_rcp(1.f + fast_exp2(-fmaf(__uint_as_float(v[c][2 * i]), sl, sb)));
            const float e1 = fast_rcp(1.f + fast_exp2(-fmaf(__uint_as_float(v[c][2 * i + 1]), sl, sb)));
            pk[i] = pack_bf16(e0, e1);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float e0, e1;
            split2(fma2(f32x2(__uint_as_float(v[c][2 * i]), __uint_as_float(v[c][2 * i + 1])), sl2, use2), e0, e1);
            e0 = fast_exp2(e0); e1 = fast_exp2(e1);         // hidden keys hold -inf: 0
            lq[i & 3] = add2(lq[i & 3], f32x2(e0, e1));
            pk[i] = pack_bf16(e0, e1);
          }
        }
        tmem_st16(p_addr + 16 * c, pk);
      }
      tmem_st_wait();
      if (!BESIDE && !moves && !pv_before()) { ok = false; break; }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[g]);
      float ls[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) split2(lq[i], ls[2 * i], ls[2 * i + 1]);
      l += ((ls[0] + ls[1]) + (ls[2] + ls[3])) + ((ls[4] + ls[5]) + (ls[6] + ls[7]));
    }
    if (ok && wait_on(&pv_full[g], (uint32_t)(n_mine - 1) & 1u, 25, n_mine)) {
      tc_fence_after();
      float inv = sig ? 1.f : (l > 0.f ? 1.f / l : 0.f);
      if (p.gate && valid) inv *= 1.f / (1.f + __expf(-p.gate[(size_t)(q0 + tok) * p.gate_ld + head]));
      const bf16* gh = nullptr;
      if (DENSE && p.gate_h && valid) {
        gh = p.gate_h + (size_t)(q0 + tok) * p.gate_h_ld + (p.gate_cols ? head * VD : head);
        if (!p.gate_cols) { inv *= 1.f / (1.f + __expf(-__bfloat162float(*gh))); gh = nullptr; }
      }
      bf16* dst = p.out + (size_t)(q0 + tok) * p.out_stride + (size_t)head * VD;
      float* fdst = MODE == CROSS ? p.cross + (((size_t)(q0 + tok) * p.nh + head) * p.nkv + vh) * VD : nullptr;
#pragma unroll
      for (int c = 0; c < VD / 32; ++c) {
        uint32_t ov[32];
        tmem_ld32(pv_addr + 32 * c, ov);
        tmem_ld_wait();
        if (MODE == CROSS) {
          if (!valid) continue;
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<float4*>(fdst + 32 * c + i) =
                make_float4(__uint_as_float(ov[i]) * inv, __uint_as_float(ov[i + 1]) * inv, __uint_as_float(ov[i + 2]) * inv,
                            __uint_as_float(ov[i + 3]) * inv);
        } else if (valid) {
          if (DENSE && gh) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              const uint4 g8 = *reinterpret_cast<const uint4*>(gh + 32 * c + i);
              const uint32_t gw[4] = {g8.x, g8.y, g8.z, g8.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 z = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gw[e]));
                ov[i + 2 * e] = __float_as_uint(__uint_as_float(ov[i + 2 * e]) / (1.f + __expf(-z.x)));
                ov[i + 2 * e + 1] = __float_as_uint(__uint_as_float(ov[i + 2 * e + 1]) / (1.f + __expf(-z.y)));
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 w;
            w.x = pack_bf16(__uint_as_float(ov[i]) * inv, __uint_as_float(ov[i + 1]) * inv);
            w.y = pack_bf16(__uint_as_float(ov[i + 2]) * inv, __uint_as_float(ov[i + 3]) * inv);
            w.z = pack_bf16(__uint_as_float(ov[i + 4]) * inv, __uint_as_float(ov[i + 5]) * inv);
            w.w = pack_bf16(__uint_as_float(ov[i + 6]) * inv, __uint_as_float(ov[i + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + 32 * c + i) = w;
          }
        }
      }
      tc_fence_before();
    }
  } else if (TMA) {
    if (lane == 0) mbar_arrive(&q_full);                  // a row tile beyond the sequence's rows: nothing to bring
  }
  }
  }   // items
  };
  if (warp < SOFTMAX_WARP0) {
    regs_give_up<REGS_LOW>();
    walk(std::false_type{});
  } else {
    regs_take<REGS_HIGH>();
    walk(std::true_type{});
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, TMEM_COLS); }
}

// ---- tensor maps over the caches (they live as long as the process, like the caches' addresses)
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;
std::mutex g_mu;
struct MapKey {
  const void* p; long long planes; int page_size, hd;
  bool operator==(const MapKey& o) const { return p == o.p && planes == o.planes && page_size == o.page_size && hd == o.hd; }
};
struct MapHash {
  size_t operator()(const MapKey& k) const {
    return std::hash<const void*>()(k.p) ^ (std::hash<long long>()(k.planes * 2654435761LL + k.page_size * 257 + k.hd) << 1);
  }
};
std::unordered_map<MapKey, CUtensorMap, MapHash> g_maps;

int find_encode() {                                      // under g_mu
  if (g_encode) return 0;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess ||
      qres != cudaDriverEntryPointSuccess || !fn) {
    cudaGetLastError();
    return -5;
  }
  g_encode = (EncodeTiledFn)fn;
  return 0;
}

// cache [planes = pages * kv heads][page_size][hd] bf16; a copy brings 64 values of box_rows keys of one plane
int cache_map(CUtensorMap* out, const void* ptr, long long planes, int page_size, int hd, int box_rows) {
  std::lock_guard<std::mutex> lk(g_mu);
  if (find_encode()) return -5;
  MapKey key{ptr, planes, page_size, hd};
  auto it = g_maps.find(key);
  if (it == g_maps.end()) {
    CUtensorMap m;
    cuuint64_t dims[3] = {(cuuint64_t)hd, (cuuint64_t)page_size, (cuuint64_t)planes};
    cuuint64_t strides[2] = {(cuuint64_t)hd * 2, (cuuint64_t)page_size * hd * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    if (g_encode(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                 CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) return -5;
    if (g_maps.size() > 4096) g_maps.clear();
    it = g_maps.emplace(key, m).first;
  }
  *out = it->second;
  return 0;
}

template <int KD, int VD, bool TMA, bool CAP, int MODE>
int launch_pf_c(const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mr, const PfParams& p, int ctas, cudaStream_t s) {
  static bool configured[64] = {};
  constexpr int smem = Shape<KD, VD, CAP>::SMEM_BYTES;
  if (allow_dynamic_smem(attn_prefill_tc_kernel<KD, VD, TMA, CAP, MODE>, smem, configured)) return -5;
  return launch_ex(attn_prefill_tc_kernel<KD, VD, TMA, CAP, MODE>, dim3(ctas), dim3(THREADS), smem, s, 1, mk, mv, mr, p);
}

template <int HD, bool TMA>
int launch_pf(const CUtensorMap& mk, const CUtensorMap& mv, const PfParams& p, int ctas, cudaStream_t s) {
  if constexpr (TMA) {
    if (p.cross) return launch_pf_c<HD, HD, true, false, CROSS>(mk, mv, mk, p, ctas, s);
  }
  return p.cap.c > 0.f ? launch_pf_c<HD, HD, TMA, true, PLAIN>(mk, mv, mk, p, ctas, s)
                       : launch_pf_c<HD, HD, TMA, false, PLAIN>(mk, mv, mk, p, ctas, s);
}

// Rows of 128 (or the heads' shared 64) numbers by tensor copies of 64 rows: [heads][rows][n], strides in numbers.
int dense_map(CUtensorMap* out, const void* ptr, int n, long long rows, long long row_stride, int heads, long long head_stride) {
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (find_encode()) return -5;
  }
  cuuint64_t dims[3] = {(cuuint64_t)n, (cuuint64_t)rows, (cuuint64_t)heads};
  cuuint64_t strides[2] = {(cuuint64_t)row_stride * 2, (cuuint64_t)head_stride * 2};
  cuuint32_t box[3] = {64, 64, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return g_encode(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -5;
}

int multiprocessors(int asked, int& sms) {
  sms = asked;
  if (sms > 0) return 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return -5;
  }
  return 0;
}

}  // namespace

// q: [T, ...] bf16 rows with stride q_stride, head h at h*hd; out likewise (16-byte aligned rows).
// kcache / vcache: [num_pages][nkv][page_size][hd] bf16. cu_q [S+1], kv_lens [S], block_table [S, bt_stride].
// max_q_len: the longest portion in the batch (sizes the list of work items). Head sizes 64 and 128.
// chunk > 0: a query sees only the keys of its own block of `chunk` positions (blocks counted from position 0);
// sinks: float [nh] or null; gate: float logits [T, gate_ld] or null (see PfParams); keep_first, sigmoid: see PfParams.
// softcap > 0: bounded scores. cross, long_from: see PfParams. sm_count: CTAs to launch at most (0: asked from the device).
RLLM_API int rllm_attention_prefill_tc(const void* q, int q_stride, const void* kcache, const void* vcache,
                                       void* out, int out_stride, const int* cu_q, const int* kv_lens,
                                       const int* block_table, int bt_stride, int num_seqs, int max_q_len,
                                       int num_pages, int nh, int nkv, int hd, int page_size, float scale, int window,
                                       int chunk, const float* sinks, const float* gate, int gate_ld,
                                       int keep_first, int sigmoid, float softcap, int long_from, float* cross, int* err,
                                       int sm_count, void* stream) {
  if (num_seqs <= 0 || max_q_len <= 0) return 0;
  if ((hd != 64 && hd != 128) || nkv <= 0 || nh % nkv || page_size <= 0 || num_pages <= 0 || keep_first < 0 || scale <= 0.f)
    return ERR_BAD_SIZE;
  if (q_stride % 8 || out_stride % 8 || ((uintptr_t)q & 15) || ((uintptr_t)out & 15) ||
      ((uintptr_t)kcache & 15) || ((uintptr_t)vcache & 15)) return ERR_BAD_ALIGN;
  if (long_from > 0 && !cross) return ERR_BAD_SIZE;
  if (cross && (softcap > 0.f || sigmoid || gate || ((uintptr_t)cross & 15))) return ERR_BAD_SIZE;
  PfParams p = {};
  p.long_from = long_from; p.cross = cross;
  p.q = (const bf16*)q; p.q_stride = q_stride; p.kc = (const bf16*)kcache; p.vc = (const bf16*)vcache;
  p.out = (bf16*)out; p.out_stride = out_stride; p.cu_q = cu_q; p.kv_lens = kv_lens;
  p.block_table = block_table; p.bt_stride = bt_stride; p.nh = nh; p.nkv = nkv; p.page_size = page_size;
  p.page_shift = -1;
  if ((page_size & (page_size - 1)) == 0) { p.page_shift = 0; while ((1 << p.page_shift) < page_size) ++p.page_shift; }
  p.chunk = chunk; p.sinks = sinks; p.gate = gate; p.gate_ld = gate_ld; p.keep_first = keep_first; p.sigmoid = sigmoid;
  p.cap = make_softcap(softcap, scale); p.cap_z = softcap > 0.f ? scale / softcap : 0.f;
  p.window = window; p.scale_log2e = scale * 1.4426950408889634f; p.err = err;
  const int G = nh / nkv;
  p.row_pairs = (max_q_len * G + RT * PM - 1) / (RT * PM); p.num_seqs = num_seqs;
  const long long items = (long long)p.row_pairs * nkv * (cross ? nkv : 1) * num_seqs;
  if (items > 2147483647LL) return ERR_TOO_LARGE;
  int sms;
  if (int rc = multiprocessors(sm_count, sms)) return rc;
  p.fold = p.window <= 0 && p.chunk <= 0 && p.row_pairs > 1 && items <= sms;
  const int ctas = items < sms ? (int)items : sms;
  // pages of a power of two from 8 keys up (whole 1 KB swizzle atoms) come by tensor copies
  const bool tma = p.page_shift >= 3 && (long long)num_pages * nkv <= 2147483647LL;
  CUtensorMap mk, mv;
  cudaStream_t s = (cudaStream_t)stream;
  if (tma) {
    const int pn = hd == 64 ? Shape<64, 64>::PN : Shape<128, 128>::PN;
    p.box_rows = page_size < pn ? page_size : pn;
    int rc;
    if ((rc = cache_map(&mk, kcache, (long long)num_pages * nkv, page_size, hd, p.box_rows))) return rc;
    if ((rc = cache_map(&mv, vcache, (long long)num_pages * nkv, page_size, hd, p.box_rows))) return rc;
    return hd == 64 ? launch_pf<64, true>(mk, mv, p, ctas, s) : launch_pf<128, true>(mk, mv, p, ctas, s);
  }
  if (cross) return ERR_BAD_SIZE;                        // only where tensor copies bring the pages
  p.box_rows = 0;
  memset(&mk, 0, sizeof(mk));
  mv = mk;
  return hd == 64 ? launch_pf<64, false>(mk, mv, p, ctas, s) : launch_pf<128, false>(mk, mv, p, ctas, s);
}

// The same attention over keys and values that lie in rows, a key and a value per query head (PfParams, DENSE): k at
// row * kv_stride + head * k_head, v likewise, `rows` of them; keys of 128 numbers, or (r not null) 192, of which the last 64 are
// r's row. q [T, ...]: head h at h * q_head, its last 64 of 192 at q2 + h * q2_head. Values of 128. gate: bf16 logits or null.
RLLM_API int rllm_attention_prefill_dense(const void* q, int q_stride, int q_head, const void* q2, long long q2_stride, int q2_head,
                                          const void* k, const void* v, long long kv_stride, int k_head, int v_head, const void* r,
                                          int r_stride, long long rows, void* out, int out_stride, const int* cu_q,
                                          const int* kv_lens, int num_seqs, int max_q_len, int nh, float scale, int window,
                                          const void* gate, int gate_ld, int gate_cols, int long_from, int* err, int sm_count,
                                          void* stream) {
  if (num_seqs <= 0 || max_q_len <= 0 || rows <= 0) return 0;
  if (nh <= 0 || scale <= 0.f || rows > 2147483647LL || (r && !q2)) return ERR_BAD_SIZE;
  if (q_stride % 8 || q_head % 8 || q2_stride % 8 || q2_head % 8 || kv_stride % 8 || k_head % 8 || v_head % 8 || r_stride % 8 ||
      out_stride % 8 || ((uintptr_t)q & 15) || ((uintptr_t)q2 & 15) || ((uintptr_t)k & 15) || ((uintptr_t)v & 15) ||
      ((uintptr_t)r & 15) || ((uintptr_t)out & 15) || (gate_cols && (gate_ld % 8 || ((uintptr_t)gate & 15)))) return ERR_BAD_ALIGN;
  PfParams p = {};
  p.q = (const bf16*)q; p.q_stride = q_stride; p.q_head = q_head;
  p.q2 = (const bf16*)q2; p.q2_stride = q2_stride; p.q2_head = q2_head;
  p.out = (bf16*)out; p.out_stride = out_stride; p.cu_q = cu_q; p.kv_lens = kv_lens;
  p.nh = p.nkv = nh; p.page_size = 1; p.page_shift = 0; p.window = window;
  p.gate_h = (const bf16*)gate; p.gate_h_ld = gate_ld; p.gate_cols = gate_cols; p.long_from = long_from;
  p.scale_log2e = scale * 1.4426950408889634f; p.err = err;
  p.row_pairs = (max_q_len + RT * PM - 1) / (RT * PM); p.num_seqs = num_seqs;
  const long long items = (long long)p.row_pairs * nh * num_seqs;
  if (items > 2147483647LL) return ERR_TOO_LARGE;
  int sms;
  if (int rc = multiprocessors(sm_count, sms)) return rc;
  p.fold = p.window <= 0 && p.chunk <= 0 && p.row_pairs > 1 && items <= sms;
  const int ctas = items < sms ? (int)items : sms;
  CUtensorMap mk, mv, mr;
  int rc;
  if ((rc = dense_map(&mk, k, 128, rows, kv_stride, nh, k_head))) return rc;
  if ((rc = dense_map(&mv, v, 128, rows, kv_stride, nh, v_head))) return rc;
  mr = mk;
  if (r && (rc = dense_map(&mr, r, 64, rows, r_stride, 1, rows * r_stride))) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  return r ? launch_pf_c<192, 128, true, false, DENSE_ROWS>(mk, mv, mr, p, ctas, s)
           : launch_pf_c<128, 128, true, false, DENSE_ROWS>(mk, mv, mr, p, ctas, s);
}
