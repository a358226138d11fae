// RWKV6 wkv on tcgen05: chunked forward and backward with split-precision operands.
//
// Maths (one (batch, head), chunk of L = 64 tokens, S is the [K][V] state; reference:
// rwkv_ops/rwkv6_kernel/ops_rwkv_kernel.py:63-80):
//   g = -exp(w), gi / ge inclusive / exclusive prefix sums of g inside the chunk, gref = gi at token 31,
//   glast = gi at token 63,  r~ = r e^{ge-gref},  k~ = k e^{gref-gi},  S~0 = diag(e^{gref}) S0
//   A = stril(r~ k~^T) + diag(sum_k r u k)
//   y   = r~ S~0 + A v
//   S_L = diag(e^{glast-gref}) (S~0 + k~^T v)
// Backward (dy, dS_L given; dS^ = diag(e^{glast-gref}) dS_L):
//   dv = A^T dy + k~ dS^        dA = dy v^T (strictly lower part -> r~, k~; diagonal -> the u term)
//   dr~ = dy S~0^T + stril(dA) k~      dk~ = stril(dA)^T r~ + v dS^^T      dS0 = diag(e^{gref}) (r~^T dy + dS^)
//   dge = dr~ r~,  dgi = -dk~ k~,  dglast = sum_v dS_L S_L,  dg_j = sum_{i>j} dge_i + sum_{i>=j} dgi_i + dglast
//   (computed without the cancellation between dglast and the state part of dgi: with X = v dS^^T,
//    dg_j = sum_{i>j} dge_i - sum_{i>=j} (stril(dA)^T r~)_i k~_i + sum_v dS^ S~0 + sum_{i<j} X_i k~_i)
//   dw = dg g;   with dd_i = dy_i . v_i:  dr += dd u k,  dk += dd r u,  du += sum_i dd r k
//
// Precision.  The parity bar for float32 inputs is 1e-4, which bf16 operands cannot meet, so every
// operand X is split as X = hi + lo (two bf16 tiles) and every product is the three tensor-core
// products hi*hi + hi*lo + lo*hi accumulated in fp32 TMEM (relative error ~2^-16 per term).
//
// A CTA of 256 threads per (batch, head) walks the chunks in order; in the forward, where that would leave SMs idle, a cluster
// of CTAs takes the chunks of a unit in turn (a single chunk: 512 threads).  The fp32 state (its gradient in the
// backward) lives in the registers of the threads that own its rows, the products in TMEM, and nothing but
// the inputs and outputs touches HBM in the forward pass (plus, for the backward, the fp32 state at every
// chunk boundary).  The raw rows of the next chunk arrive by TMA while the current chunk is worked on.
// Tile and TMEM conventions are those of tc.cuh.
#include <type_traits>

#include "common.cuh"
#include "tc.cuh"

namespace rwkvb200 {
namespace w6c {

using namespace tc;
typedef __nv_bfloat16 bf16;

constexpr int L = 64;
constexpr int NROW = 68;
// All decay sums are kept in units of log 2 (tc::ex2: a scale factor is one instruction); nothing is clamped.
constexpr float EXP2_FLOOR = -126.f;      // 2^x below this is flushed to zero anyway
// The scaled operands carry e^{+-(gi - gref)}, whose exponent reaches the sum of |g| over half a chunk.  Range
// alone would allow about 60 (every factor, and the low half of every split operand, stays a normal number),
// but the decay gradient is a difference of prefix sums that cancel the more the faster the state decays:
// measured against a float64 oracle with every channel decaying at the same rate, its relative error grows
// from 2e-5 at |g| = 0.3 per token to 1e-4 (the parity bar) at |g| = 1.55.  DECAY_LIMIT = 45 (|g| <= 1.4 per
// token, w <= 0.34) keeps it below the bar.  A (batch, head) unit that exceeds the limit in any channel of any
// chunk is marked by the forward kernel and recomputed by the float32 recurrence (wkv6.cu), forward and
// backward, so that no value computed from a clamped exponent is ever returned.
constexpr float DECAY_LIMIT = 45.f;
// Sequences shorter than this take the recurrence as well (marked in the same flags): with two or three tokens and
// fast decays the decay gradient is the small remainder of pair sums that cancel (every pair of tokens enters the
// row sums of dr~ r~ and the column sums of dk~ k~ with opposite signs, computed by different tensor-core
// products), and the 2^-17 roundings of the split operands reached 5e-4 of dw there; the recurrence costs nothing
// at that length.
constexpr int SHORT_SEQ = 8;
constexpr int MARKED = 1 << 30;      // in the forward's count of stretches done: one of them has to be recomputed

// two values as packed bf16 pairs hi and lo with x = hi + lo (+ an error of about 2^-17 |x|)
__device__ __forceinline__ void split_pair(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16(x0, x1);
  lo = pack_bf16(x0 - bf16_lo(hi), x1 - bf16_hi(hi));
}
// write 4 consecutive values (columns col .. col+3, col a multiple of 4) of `row` into a hi and a lo tile
template <bool LO = true>
__device__ __forceinline__ void store_split4(unsigned char* hi_t, unsigned char* lo_t, int row, int col, float4 x) {
  uint2 h, l;
  split_pair(x.x, x.y, h.x, l.x);
  split_pair(x.z, x.w, h.y, l.y);
  const uint32_t off = tile_off(row, col);
  *reinterpret_cast<uint2*>(hi_t + off) = h;
  if constexpr (LO) *reinterpret_cast<uint2*>(lo_t + off) = l;
}
// write CW consecutive fp32 values of `row` (columns col0 .., col0 a multiple of 8) into a hi and a lo tile
template <int CW>
__device__ __forceinline__ void store_split_row(unsigned char* hi_t, unsigned char* lo_t, int row, int col0, const float* x) {
#pragma unroll
  for (int c = 0; c < CW / 8; ++c) {
    uint4 h, l;
    split_pair(x[8 * c + 0], x[8 * c + 1], h.x, l.x);
    split_pair(x[8 * c + 2], x[8 * c + 3], h.y, l.y);
    split_pair(x[8 * c + 4], x[8 * c + 5], h.z, l.z);
    split_pair(x[8 * c + 6], x[8 * c + 7], h.w, l.w);
    const uint32_t off = tile_chunk_off(row, (col0 >> 3) + c);
    *reinterpret_cast<uint4*>(hi_t + off) = h;
    *reinterpret_cast<uint4*>(lo_t + off) = l;
  }
}

// How a CTA of NTHR threads (256 or 512) splits a chunk of 64 tokens x 64 channels: a token row is 16 threads wide (four
// channels each); a (channel, part) thread owns PL consecutive tokens; a thread that reads an accumulator takes CW
// columns of its lane.
template <int NTHR>
struct Split {
  static constexpr int NE = 1024 / NTHR;        // token rows per thread
  static constexpr int PARTS = NTHR / 64, PL = 64 / PARTS;
  static constexpr int CW = 8192 / NTHR;
};
// sums over the parts of the first / second half of the chunk, from the sums over the parts
template <int PARTS>
__device__ __forceinline__ float half_sum(const float (*tot)[64], int half, int ch) {
  float x = tot[half * (PARTS / 2)][ch];
#pragma unroll
  for (int q = 1; q < PARTS / 2; ++q) x += tot[half * (PARTS / 2) + q][ch];
  return x;
}
// What to add to the prefix sums of a part (its own sum is `run`) so that they count from the end of the first half.
template <int PARTS>
__device__ __forceinline__ float from_middle(const float (*tot)[64], int part, int ch, float run) {
  constexpr int HALF = PARTS / 2;
  float add = part < HALF ? -run : 0.f;
#pragma unroll
  for (int q = 0; q < HALF; ++q) {
    if (part < HALF && q > part) add -= tot[q][ch];
    if (part >= HALF && HALF + q < part) add += tot[HALF + q][ch];
  }
  return add;
}

// D (+)= X Y with X = xh + xl, Y = yh + yl (lo tile = hi tile + TILE_BYTES): hi*hi + hi*lo + lo*hi.  A_LO / B_LO = false: that
// operand's lo tile would be zero (v and dy of bfloat16 tokens) and is neither written nor multiplied.
template <int M, int N, int A_MN, int B_MN, bool A_LO = true, bool B_LO = true>
__device__ __forceinline__ void umma_split(uint32_t tmem_d, uint32_t a_hi, uint32_t b_hi, bool accumulate) {
  umma_tile<M, N, A_MN, B_MN>(tmem_d, a_hi, b_hi, accumulate);
  if constexpr (B_LO) umma_tile<M, N, A_MN, B_MN>(tmem_d, a_hi, b_hi + TILE_BYTES, true);
  if constexpr (A_LO) umma_tile<M, N, A_MN, B_MN>(tmem_d, a_hi + TILE_BYTES, b_hi, true);
}
// whether token values have a lo part
template <typename T> constexpr bool has_lo() { return !std::is_same<T, __nv_bfloat16>::value; }

// Row `lr` (0..15) of a warp's 16 x CW block of a 64 x 64 product that is kept strictly below the diagonal, the
// diagonal itself set to `diag`, split and stored.  Where the diagonal crosses the block depends on the warp alone:
// left of column JLO (of the block's CW) every element is kept, from JLO + 16 on every element is zero, and only
// the 16 columns between take a per-element choice.  JLO = CW: the whole block is kept; JLO = -16: all zero
// (`rr` is not read).
template <int CW, int JLO>
__device__ __forceinline__ void store_masked_row(const uint32_t (&rr)[CW], int lr, float diag, unsigned char* hi_t,
                                                 int row, int col0) {
  float x[CW];
#pragma unroll
  for (int j = 0; j < CW; ++j) {
    if (j < JLO) x[j] = __uint_as_float(rr[j]);
    else if (j >= JLO + 16) x[j] = 0.f;
    else x[j] = (j - JLO) < lr ? __uint_as_float(rr[j]) : ((j - JLO) == lr ? diag : 0.f);
  }
  store_split_row<CW>(hi_t, hi_t + TILE_BYTES, row, col0, x);
}
// Row `lr` of the same block as values, `other` in the lanes that do not hold a row of it.  All lanes of the warp call it.
template <int CW>
__device__ __forceinline__ void load_masked_row(uint32_t taddr, int wq, int hsel, int lr, float diag, bool active,
                                                const float (&other)[CW], float (&x)[CW]) {
  const int jlo = 16 * wq - CW * hsel;
  if (jlo < 0) {
#pragma unroll
    for (int j = 0; j < CW; ++j) x[j] = active ? 0.f : other[j];
    return;
  }
  uint32_t rr[CW];
  tmem_ld<CW>(taddr, rr);
  tmem_ld_wait();
  auto crossed_at = [&](int at) {      // left of column `at` everything is kept, from at + 16 on nothing
#pragma unroll
    for (int j = 0; j < CW; ++j) {
      const float f = __uint_as_float(rr[j]);
      const float m = j < at ? f : j >= at + 16 ? 0.f : (j - at) < lr ? f : (j - at) == lr ? diag : 0.f;
      x[j] = active ? m : other[j];
    }
  };
  if (jlo >= CW) crossed_at(CW);
  else if (CW == 32 && jlo == 16) crossed_at(16);
  else crossed_at(0);
}
// the same for a warp whose rows are 16*wq .. and whose columns are CW*hsel ..; all lanes of the warp call it
template <int CW>
__device__ __forceinline__ void load_store_masked_row(uint32_t taddr, int wq, int hsel, int lr, float diag,
                                                      unsigned char* hi_t, int row, bool active) {
  const int jlo = 16 * wq - CW * hsel;
  uint32_t rr[CW];
  if (jlo < 0) {
    if (active) store_masked_row<CW, -16>(rr, lr, diag, hi_t, row, CW * hsel);
    return;
  }
  tmem_ld<CW>(taddr, rr);
  tmem_ld_wait();
  if (!active) return;
  if (jlo >= CW) store_masked_row<CW, CW>(rr, lr, diag, hi_t, row, CW * hsel);
  else if (CW == 32 && jlo == 16) store_masked_row<CW, 16>(rr, lr, diag, hi_t, row, CW * hsel);
  else store_masked_row<CW, 0>(rr, lr, diag, hi_t, row, CW * hsel);
}

__device__ __forceinline__ long long state_row(const int32_t* smap, int n_state, int bi) {
  if (n_state == 1) return 0;
  if (!smap) return bi;
  int m = smap[bi];
  return m < 0 ? 0 : (m >= n_state ? n_state - 1 : m);
}

// Where the tokens of a unit's sequence lie.  Dense batches: row bi of [B][T][H][64], Tn tokens.  Packed batches
// (PACKED): the sequences lie end to end in one row [1][total][H][64]; sequence bi is tokens start[bi] ..
// start[bi] + len[bi] - 1, and the rows of a chunk past the end of the sequence belong to the next one: they are
// read as zeros and never stored.
struct Seqs {
  const int32_t* start;
  const int32_t* len;
  int nts;      // chunk-boundary state slots per unit in `states` (chunks of the longest sequence + 1)
};

// The counters of the stretches, as a kernel: a memset would hold the next kernel's launch up.
__global__ void w6c_clear_kernel(int* p, int n) {
  earlier_kernels_done();
  later_kernels_may_start();
  for (int i = threadIdx.x; i < n; i += blockDim.x) p[i] = 0;
}

// ---------------------------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------------------------
struct FwdSmem {
  unsigned char rt[2][TILE_BYTES];    // r~ hi, lo      [token][k]
  unsigned char kt[2][TILE_BYTES];    // k~ hi, lo      [token][k]
  unsigned char vt[2][TILE_BYTES];    // v hi, lo       [token][v]
  unsigned char at[2][TILE_BYTES];    // A hi, lo       [token i][token j]
  unsigned char st[2][TILE_BYTES];    // S~0 hi, lo     [k][v]
  float gs[L * NROW];                 // gi - gref (prefix of g relative to the reference point); later the staged y rows
  float qtot[8][64];
  float dgs[64];                      // sum_k r u k per token
  uint64_t bar_1, bar_2, bar_in;
  uint64_t bar_state, bar_free;       // RELAY: the state is here (16 KB); the next CTA can take another one
  uint32_t tmem_base;
  int next_item, state_seen;
  int marks[8];                       // RELAY: what each CTA of the cluster has marked (in the first one)
};

// The raw r, k, v, w rows of a chunk (64 rows of 64 elements each) arrive by TMA in the space of the tile
// pairs they are turned into (r -> rt, k -> kt, v -> vt, w -> at), requested for the next chunk as soon as
// the last MMA of the current one has read those tiles; a thread reads its elements, all threads meet at a
// barrier, and then the split tiles are written over the raw rows.
// S0 of every chunk (and the final state) goes to `states` [B*H][NT+1][64][64] when it is not NULL.
template <typename T, bool PACKED, int NTHR, bool RELAY>
__global__ void __launch_bounds__(NTHR, 512 / NTHR)
wkv6c_fwd_kernel(const T* __restrict__ r, const T* __restrict__ k, const T* __restrict__ v, const T* __restrict__ w,
                 const void* __restrict__ u, const void* __restrict__ s0, int n_state,
                 const int32_t* __restrict__ smap, T* __restrict__ y, void* __restrict__ sT, int typed,
                 float* __restrict__ states, int* __restrict__ flags, const __grid_constant__ CUtensorMap tmap_r,
                 const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                 const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_y, int Tn_dense, int H,
                 Seqs seqs, int n_units, int per_item, int parts,
                 float* __restrict__ handoff, int* __restrict__ handoff_flags, int* status, long long* dbg) {
#ifdef RWKVB200_DEVTOOLS
#define W6C_STAMP(n) do { if (dbg && tid == 0 && item == gridDim.x / 2 && c == 2) dbg[n] = clock64(); } while (0)
#else
#define W6C_STAMP(n) do {} while (0)
#endif
  extern __shared__ unsigned char smem_raw[];
  FwdSmem& sm = *reinterpret_cast<FwdSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wq = warp & 3, hsel = warp >> 2;
  constexpr int NE = Split<NTHR>::NE, PARTS = Split<NTHR>::PARTS, PL = Split<NTHR>::PL, CW = Split<NTHR>::CW;
  const long long tstride = (long long)H * HS;
  const int srow = 16 * wq + (lane & 15);     // state row k (upper lane halves) / token row (lower lane halves)
  const bool tok_lane = lane < 16;            // lower lane halves hold token rows, upper halves state rows

  if (tid == 0) {
    // MMA batch 1 has two accumulators and two issuing threads (of warps 0 and 1) and completes with both arrivals
    mbar_init(&sm.bar_1, 2); mbar_init(&sm.bar_2, 1); mbar_init(&sm.bar_in, 1);
    mbar_init(&sm.bar_state, 1); mbar_init(&sm.bar_free, 1);
    fence_mbar_init();
  }
  if (tid == 32) tma_prefetch_maps(tmap_r, tmap_k, tmap_v, tmap_w, tmap_y);
  if (warp == 0) tmem_alloc(&sm.tmem_base, 128);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  earlier_kernels_done();
  later_kernels_may_start();
  const uint32_t tm = sm.tmem_base;
  // TMEM: columns 0..63 lower halves = r~ k~^T; columns 64..127 lower halves = y, upper halves = k~^T v
  const uint32_t tm_a = tmem_addr(tm, 32 * wq, CW * hsel);
  const uint32_t tm_ys = tmem_addr(tm, 32 * wq, 64 + CW * hsel);

  const int c4 = tid & 15;
  const T* raw_r = reinterpret_cast<const T*>(sm.rt[0]);
  const T* raw_k = reinterpret_cast<const T*>(sm.kt[0]);
  const T* raw_v = reinterpret_cast<const T*>(sm.vt[0]);
  const T* raw_w = reinterpret_cast<const T*>(sm.at[0]);

  // Work items.  parts == 1: an item is a (batch, head) unit and the grid has one CTA per unit.  parts > 1: every unit is
  // `parts` items, stretches of `per_item` of its chunks, on a persistent grid whose CTAs take items from a counter
  // (handoff_flags[n_units]), one ahead of the one they work on; all first stretches come first in that order.  The state
  // travels from stretch to stretch through `states`, where a training forward leaves it anyway, or `handoff`;
  // handoff_flags[unit] counts the stretches of the unit that have left theirs (MARKED: one of them left the decay range).
  // The first item of those not done yet waits for none, and its CTA is at work on it: the wait needs no assumption
  // about which CTAs are resident.  A chunk needs the state only for its second batch of products and has its own
  // contribution to it by then, so one chunk waits for another only for a state to be fetched, scaled and left.
  // RELAY (parts == 1): the CTAs of a cluster, at most eight, work on the chunks of one unit in turn, and the state goes from
  // one's registers into the shared memory of the next.  A chunk then takes the unit a state's way from barrier to
  // barrier (1.6 us) instead of its whole chain of phases (4.3): 1 sequence of 4096 tokens, 32 heads, bfloat16, 273 -> 101 us;
  // 148 units of 777 tokens, where two CTAs to a unit fill the device, 66 -> 57.
  const int n_items = parts * n_units;
  bool ok = true;
  uint32_t n_done = 0;      // chunks this CTA has worked on: every barrier completes once per chunk
  uint32_t n_fetched = 0, n_sent = 0;      // RELAY: states received and sent
  const int rank = RELAY ? (int)blockIdx.y : 0, n_cta = RELAY ? (int)gridDim.y : 1;
  const uint32_t succ = RELAY ? (rank + 1 == n_cta ? 0 : rank + 1) : 0, pred = RELAY ? (rank ? rank - 1 : n_cta - 1) : 0;
  if constexpr (RELAY) cluster_sync();      // the barriers of all CTAs are set up
  int item = blockIdx.x;
  if (parts > 1) {
    if (tid == 0) sm.next_item = atomicAdd(handoff_flags + n_units, 1);
    __syncthreads();
    item = sm.next_item;
  }
  struct Stretch {
    int unit, part, bi, hi, Tn, tok0, brow, NT, c_lo, c_hi;
  };
  auto stretch = [&](int i) {
    Stretch x;
    x.unit = i % n_units; x.part = i / n_units;
    x.bi = x.unit / H; x.hi = x.unit % H;
    x.Tn = PACKED ? seqs.len[x.bi] : Tn_dense;
    x.tok0 = PACKED ? seqs.start[x.bi] : 0;       // first token row of the sequence in its batch row
    x.brow = PACKED ? 0 : x.bi;
    x.NT = (x.Tn + L - 1) / L;
    x.c_lo = x.part * per_item;      // the chunks c_lo .. c_hi - 1; none in a sequence that ends before them
    x.c_hi = min(x.c_lo + per_item, x.NT);
    return x;
  };
  auto load_in = [&](const Stretch& x, int c) {      // one thread; rows past the end of the sequence arrive as zeros
    mbar_expect_tx(&sm.bar_in, 4 * 64 * 64 * (uint32_t)sizeof(T));
    tma_load_4d(sm.at[0], &tmap_w, &sm.bar_in, 0, x.tok0 + c * L, x.hi, x.brow);
    tma_load_4d(sm.vt[0], &tmap_v, &sm.bar_in, 0, x.tok0 + c * L, x.hi, x.brow);
    tma_load_4d(sm.rt[0], &tmap_r, &sm.bar_in, 0, x.tok0 + c * L, x.hi, x.brow);
    tma_load_4d(sm.kt[0], &tmap_k, &sm.bar_in, 0, x.tok0 + c * L, x.hi, x.brow);
  };
  if (item < n_items && warp == 0 && elect_one()) {
    const Stretch x = stretch(item);
    if (x.c_lo + rank < x.c_hi) load_in(x, x.c_lo + rank);
  }
  // an item without a chunk (of a packed batch) takes the next one by itself
  auto take_next = [&]() {
    if (warp == 0 && elect_one()) {
      sm.next_item = atomicAdd(handoff_flags + n_units, 1);
      if (sm.next_item < n_items) {
        const Stretch x = stretch(sm.next_item);
        if (x.c_lo < x.c_hi) load_in(x, x.c_lo);
      }
    }
  };
  while (item < n_items && ok) {
  const Stretch cur = stretch(item);
  const int unit = cur.unit, part = cur.part, hi = cur.hi, Tn = cur.Tn, c_lo = cur.c_lo, c_hi = cur.c_hi;
  const long long base = (((long long)cur.brow * Tn_dense + cur.tok0) * H + hi) * HS;   // Tn_dense: rows per batch row
  const size_t nts = PACKED ? (size_t)seqs.nts : (size_t)(cur.NT + 1);
  const bool last_part = c_hi == cur.NT;
  if (c_lo < c_hi || (c_hi == 0 && (!PACKED || part == 0))) {      // (c_hi == 0: an empty sequence, which just hands its state on)
  // per-thread slice of u (4 channels) for the diagonal term
  const float4 u4 = load4_as<T>(u, hi * HS + 4 * c4, typed);
  int marked = Tn < SHORT_SEQ;      // thread-wise until the end of the item

  // ---- state at the item's first chunk: rows k on the upper lane halves, this warp's 32 columns
  float sreg[CW];
#pragma unroll
  for (int j = 0; j < CW; ++j) sreg[j] = 0.f;
  if (part == 0 && rank == 0 && !tok_lane && s0 && n_state > 0) {
    const long long S = ((state_row(smap, n_state, cur.bi) * H + hi) * HS + srow) * HS + CW * hsel;
#pragma unroll
    for (int j = 0; j < CW; j += 4) {
      const float4 fv = load4_as<T>(s0, S + j, typed);
      sreg[j] = fv.x; sreg[j + 1] = fv.y; sreg[j + 2] = fv.z; sreg[j + 3] = fv.w;
    }
  }
  // where the state before chunk c travels
  auto state_slot = [&](int c) {
    return (states ? states + ((size_t)unit * nts + c) * (HS * HS) : handoff + (size_t)unit * (HS * HS)) + srow * HS + CW * hsel;
  };
  // The state the item's first chunk starts from: what the stretch before it has left (bounded wait; all threads).
  auto fetch_state = [&]() {
    if (tid == 0) {
      int seen = 0;
      uint32_t polls = 0;
      while (true) {
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(handoff_flags + unit) : "memory");
        if ((seen & ~MARKED) >= part || ++polls > (WAIT_LIMIT << 2)) break;
        __nanosleep(100);
      }
      if ((seen & ~MARKED) < part) { atomicExch(status, 405); seen = -1; }
      sm.state_seen = seen;
    }
    __syncthreads();
    const int seen = sm.state_seen;
    if (seen < 0) return false;
    marked |= seen & MARKED;
    if (!tok_lane) {
      const float* S = state_slot(c_lo);
#pragma unroll
      for (int j = 0; j < CW; j += 4) {
        const float4 fv = __ldcg(reinterpret_cast<const float4*>(S + j));
        sreg[j] = fv.x; sreg[j + 1] = fv.y; sreg[j + 2] = fv.z; sreg[j + 3] = fv.w;
      }
    }
    return true;
  };
  // RELAY: a row piece of the state travels through the 2 x 64 bytes that its S~0 takes up as hi and lo parts
  auto piece = [&](int j) { return tile_chunk_off(srow, 4 * hsel + (j & 3)) + (j >> 2) * TILE_BYTES; };
  auto receive_state = [&]() {
    if (!mbar_wait<true>(&sm.bar_state, n_fetched & 1, status, 406)) return false;
    if (!tok_lane) {
#pragma unroll
      for (int j = 0; j < CW / 4; ++j) {
        const float4 fv = *reinterpret_cast<const float4*>(sm.st[0] + piece(j));
        sreg[4 * j] = fv.x; sreg[4 * j + 1] = fv.y; sreg[4 * j + 2] = fv.z; sreg[4 * j + 3] = fv.w;
      }
    }
    return true;
  };
  auto send_state = [&](const float (&x)[CW]) {      // the CTA of the next chunk has no more use for its S~0
    if (!tok_lane) {
      const uint32_t to = cluster_addr(smem_u32(sm.st[0]), succ), bar = cluster_addr(smem_u32(&sm.bar_state), succ);
#pragma unroll
      for (int j = 0; j < CW / 4; ++j)
        store_async_16(to + piece(j), make_float4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]), bar);
    }
  };
  auto keep_state = [&](int c) {      // the state before chunk c
    float* dst = state_slot(c);
#pragma unroll
    for (int j = 0; j < CW; j += 4)
      *reinterpret_cast<float4*>(dst + j) = make_float4(sreg[j], sreg[j + 1], sreg[j + 2], sreg[j + 3]);
  };
  if (states && !tok_lane && part == 0 && rank == 0) keep_state(0);
  if (RELAY && rank > 0 && rank < c_hi && warp == 1 && elect_one()) mbar_arrive_cluster(cluster_addr(smem_u32(&sm.bar_free), pred));

  for (int c = c_lo + rank; c < c_hi && ok; c += n_cta, ++n_done) {
    const int t0 = c * L;
    const uint32_t par = n_done & 1;
    W6C_STAMP(0);
    // the next item is taken here and handed to the others once it has arrived
    const bool take = !RELAY && parts > 1 && c + 1 == c_hi;
    int ticket = 0;
    if (take && tid == NTHR - 1) ticket = atomicAdd(handoff_flags + n_units, 1);
    if (RELAY && c > 0 && warp == 0 && elect_one()) mbar_expect_tx(&sm.bar_state, HS * HS * (uint32_t)sizeof(float));
    // ---- the raw rows of the chunk have landed: this thread's w and v elements
    ok = mbar_wait(&sm.bar_in, par, status, 403) && ok;
    float4 gw[NE], vv4[NE];
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      const int e = tid + NTHR * n, row = e >> 4;
      gw[n] = load4_shared(raw_w + row * 64 + 4 * c4);
      if constexpr (has_lo<T>()) {
        vv4[n] = load4_shared(raw_v + row * 64 + 4 * c4);
        if (PACKED && t0 + row >= Tn) vv4[n] = make_float4(0.f, 0.f, 0.f, 0.f);      // the next sequence's row
      } else {
        // bfloat16 rows have arrived as the tile that the products read
        if (PACKED && t0 + row >= Tn) *reinterpret_cast<uint2*>(sm.vt[0] + tile_off(row, 4 * c4)) = make_uint2(0u, 0u);
      }
    }
    if (warp == 1 && elect_one()) bulk_wait_read();      // the last y rows have left the space of gs
    __syncthreads();      // every raw v element is in registers: the split v tiles may overwrite the rows
    // ---- pass W: g and its prefix sums; pass V
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      const int e = tid + NTHR * n, row = e >> 4, tok = t0 + row;
      float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
      if (tok < Tn)
        f = make_float4(-LOG2E * ex2(LOG2E * gw[n].x), -LOG2E * ex2(LOG2E * gw[n].y), -LOG2E * ex2(LOG2E * gw[n].z),
                        -LOG2E * ex2(LOG2E * gw[n].w));
      gw[n] = f;
      *reinterpret_cast<float4*>(&sm.gs[row * NROW + 4 * c4]) = f;
      if constexpr (has_lo<T>()) store_split4(sm.vt[0], sm.vt[1], row, 4 * c4, vv4[n]);
    }
    __syncthreads();
    W6C_STAMP(1);
    {
      const int ch = tid & 63, part = tid >> 6;
      float gv[PL];
#pragma unroll
      for (int j = 0; j < PL; ++j) gv[j] = sm.gs[(PL * part + j) * NROW + ch];
      float run = 0.f;
#pragma unroll
      for (int j = 0; j < PL; ++j) { run += gv[j]; gv[j] = run; }
      sm.qtot[part][ch] = run;
      __syncthreads();
      const float add = from_middle<PARTS>(sm.qtot, part, ch, run);
#pragma unroll
      for (int j = 0; j < PL; ++j) sm.gs[(PL * part + j) * NROW + ch] = gv[j] + add;
    }
    __syncthreads();
    W6C_STAMP(2);
    // decay factors of the state rows: e^{gref} of this chunk scales the incoming state, e^{glast-gref} the outgoing
    float e0 = 1.f, dlast = 1.f;
    if (!tok_lane) {
      const float tot0 = half_sum<PARTS>(sm.qtot, 0, srow), tot1 = half_sum<PARTS>(sm.qtot, 1, srow);
      e0 = ex2(fmaxf(tot0, EXP2_FLOOR));
      dlast = ex2(fmaxf(tot1, EXP2_FLOOR));
      // a half-chunk decay sum beyond the limit: the unit is recomputed by the float32 recurrence
      marked |= fminf(tot0, tot1) < -DECAY_LIMIT * LOG2E;
    }
    W6C_STAMP(3);
    // ---- pass RK: scaled r, k (split hi/lo) and the diagonal term
    float4 rr4[NE], kk4[NE];
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      const int row = (tid + NTHR * n) >> 4;
      rr4[n] = load4_shared(raw_r + row * 64 + 4 * c4);
      kk4[n] = load4_shared(raw_k + row * 64 + 4 * c4);
      if (PACKED && t0 + row >= Tn) { rr4[n] = make_float4(0.f, 0.f, 0.f, 0.f); kk4[n] = rr4[n]; }
    }
    __syncthreads();      // every raw r, k element is in registers
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      const int e = tid + NTHR * n, row = e >> 4;
      const float4 r4 = rr4[n], k4 = kk4[n];
      const float4 gp = *reinterpret_cast<const float4*>(&sm.gs[row * NROW + 4 * c4]);
      const float d1x = gp.x, d1y = gp.y, d1z = gp.z, d1w = gp.w;   // gi - gref
      const float4 rs = make_float4(r4.x * ex2(d1x - gw[n].x), r4.y * ex2(d1y - gw[n].y),
                                    r4.z * ex2(d1z - gw[n].z), r4.w * ex2(d1w - gw[n].w));
      const float4 ks = make_float4(k4.x * ex2(-d1x), k4.y * ex2(-d1y), k4.z * ex2(-d1z), k4.w * ex2(-d1w));
      store_split4(sm.rt[0], sm.rt[1], row, 4 * c4, rs);
      store_split4(sm.kt[0], sm.kt[1], row, 4 * c4, ks);
      float dg = r4.x * u4.x * k4.x + r4.y * u4.y * k4.y + r4.z * u4.z * k4.z + r4.w * u4.w * k4.w;
#pragma unroll
      for (int m = 8; m >= 1; m >>= 1) dg += __shfl_xor_sync(0xffffffffu, dg, m);
      if (c4 == 0) sm.dgs[row] = dg;
    }
    if (take && tid == NTHR - 1) sm.next_item = ticket;
    fence_async_smem();
    tc_fence_before();
    __syncthreads();

    W6C_STAMP(4);
    // ---- batch 1: r~ k~^T (columns 0..63), k~^T v (columns 64.., upper halves)
    if (warp < 2 && elect_one()) {
      tc_fence_after();
      if (warp == 0) umma_split<64, 64, 0, 0>(tmem_addr(tm, 0, 0), smem_u32(sm.rt[0]), smem_u32(sm.kt[0]), false);
      else           umma_split<64, 64, 1, 1, true, has_lo<T>()>(tmem_addr(tm, 16, 64), smem_u32(sm.kt[0]), smem_u32(sm.vt[0]), false);
      umma_commit(&sm.bar_1);
    }
    // ask for the next chunk's rows to be brought into L2 while this chunk is in its MMA phases
    if (warp == 2 && elect_one()) {
      Stretch x = cur;
      int cn = c + n_cta;
      if (take && sm.next_item < n_items) { x = stretch(sm.next_item); cn = x.c_lo; }
      if (cn < x.c_hi) {
        tma_prefetch_4d(&tmap_w, 0, x.tok0 + cn * L, x.hi, x.brow);
        tma_prefetch_4d(&tmap_v, 0, x.tok0 + cn * L, x.hi, x.brow);
        tma_prefetch_4d(&tmap_r, 0, x.tok0 + cn * L, x.hi, x.brow);
        tma_prefetch_4d(&tmap_k, 0, x.tok0 + cn * L, x.hi, x.brow);
      }
    }
    const bool need_state = RELAY ? c > 0 : part > 0 && c == c_lo, hand_on = !RELAY && c + 1 == c_hi && !last_part;
    if (!RELAY && need_state) ok = fetch_state() && ok;
    ok = mbar_wait(&sm.bar_1, par, status, 401) && ok;
    tc_fence_after();
    W6C_STAMP(5);
    if (ok) {
      // state rows: S~0 = e^{gref} S0, and (k~^T v on the upper halves of columns 64..127) S_L = e^{glast-gref} (S~0 + k~^T v)
      float next_s[CW];
      {
        uint32_t rr[CW];
        tmem_ld<CW>(tm_ys, rr);
        tmem_ld_wait();
        const bool send = RELAY && c + 1 < c_hi;      // (what can be waited for before the state arrives is)
        if (send) ok = mbar_wait<true>(&sm.bar_free, n_sent & 1, status, 407);
        if (RELAY && need_state) ok = receive_state() && ok;
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          sreg[j] = __fmul_rn(sreg[j], e0);
          next_s[j] = (sreg[j] + __uint_as_float(rr[j])) * dlast;
        }
        if (send && ok) send_state(next_s);
      }
      // A rows (lower halves of columns 0..63), strictly lower part plus the diagonal term, and S~0 rows: split, stored
      float x[CW];
      load_masked_row<CW>(tm_a, wq, hsel, lane & 15, tok_lane ? sm.dgs[srow] : 0.f, tok_lane, sreg, x);
      unsigned char* hi_t = tok_lane ? sm.at[0] : sm.st[0];
      store_split_row<CW>(hi_t, hi_t + TILE_BYTES, srow, CW * hsel, x);
#pragma unroll
      for (int j = 0; j < CW; ++j) sreg[j] = next_s[j];
      if (hand_on && !tok_lane) { keep_state(c + 1); __threadfence(); }
    }
    fence_async_smem();
    tc_fence_before();
    if (need_state) ++n_fetched;
    if (c + 1 < c_hi) ++n_sent;
    if (hand_on) marked = __syncthreads_or(marked);
    ok = __syncthreads_and(ok);

    W6C_STAMP(6);
    // ---- batch 2: y = r~ S~0 + A v
    if (warp == 0 && elect_one() && ok) {
      tc_fence_after();
      umma_split<64, 64, 0, 1>(tmem_addr(tm, 0, 64), smem_u32(sm.rt[0]), smem_u32(sm.st[0]), false);
      umma_split<64, 64, 0, 1, true, has_lo<T>()>(tmem_addr(tm, 0, 64), smem_u32(sm.at[0]), smem_u32(sm.vt[0]), true);
      umma_commit(&sm.bar_2);
    }
    if (hand_on && warp == 1 && elect_one() && ok)
      asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(handoff_flags + unit), "r"((part + 1) | (marked ? MARKED : 0)) : "memory");
    // the state of the next chunk's start, stored here because the next proxy fence, which waits for global stores too, is
    // most of a chunk away
    if (states && !tok_lane && ok && !hand_on) keep_state(c + 1);
    ok = mbar_wait(&sm.bar_2, par, status, 402) && ok;
    tc_fence_after();
    W6C_STAMP(7);
    if (RELAY && c + n_cta < c_hi && warp == 1 && elect_one() && ok)      // and so has S~0
      mbar_arrive_cluster(cluster_addr(smem_u32(&sm.bar_free), pred));
    if (warp == 0 && elect_one() && ok) {      // the tiles of this chunk have been read for the last time
      if (c + n_cta < c_hi) {
        load_in(cur, c + n_cta);
      } else if (take && sm.next_item < n_items) {
        const Stretch x = stretch(sm.next_item);
        if (x.c_lo < x.c_hi) load_in(x, x.c_lo);
      }
    }
    // the y rows as swizzled tiles (of 32 channels each in float32) in the prefix-sum area
    unsigned char* yt = reinterpret_cast<unsigned char*>(sm.gs);
    if (ok && y) {
      uint32_t rr[CW];
      tmem_ld<CW>(tm_ys, rr);
      tmem_ld_wait();
      if (tok_lane) {
#pragma unroll
        for (int j = 0; j < CW; j += 16 / sizeof(T)) {
          uint4 u = make_uint4(rr[j], rr[j + 1], rr[j + 2], rr[j + 3]);
          if constexpr (sizeof(T) == 2) {
            auto pair = [&](int i) {
              const float a = __uint_as_float(rr[j + i]), b = __uint_as_float(rr[j + i + 1]);
              const T p[2] = {from_f32<T>(a), from_f32<T>(b)};
              return *reinterpret_cast<const uint32_t*>(p);
            };
            u = make_uint4(pair(0), pair(2), pair(4), pair(6));
          }
          const int q = (CW * hsel + j) * (int)sizeof(T) / 16;      // 16-byte piece of the row
          *reinterpret_cast<uint4*>(yt + (q >> 3) * TILE_BYTES + tile_chunk_off(srow, q & 7)) = u;
        }
      }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    W6C_STAMP(8);
    if (y && ok) {
      constexpr int ROW = HS * (int)sizeof(T) / 16;      // pieces per row
      if (PACKED && t0 + L > Tn) {      // the last rows of a box belong to the next sequence: row by row
        for (int e = tid; e < 64 * ROW; e += NTHR) {
          const int row = e / ROW, q = e % ROW;
          if (t0 + row < Tn)
            *reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(y + base + (long long)(t0 + row) * tstride) + 16 * q) =
                *reinterpret_cast<const uint4*>(yt + (q >> 3) * TILE_BYTES + tile_chunk_off(row, q & 7));
        }
        __syncthreads();      // the rows have been read
      } else if (warp == 1 && elect_one()) {      // rows past the end of the tensor are clipped
        for (int h = 0; h < ROW / 8; ++h)
          tma_store_4d(&tmap_y, yt + h * TILE_BYTES, h * (128 / (int)sizeof(T)), cur.tok0 + t0, hi, cur.brow);
        bulk_commit();
      }
    }
    W6C_STAMP(9);
  }
#undef W6C_STAMP
  // ---- the unit's final state
  if (last_part) {
    if (!tok_lane && ok && sT && (!RELAY || max(c_hi - 1, 0) % n_cta == rank)) {
      const long long dst = (((long long)unit * HS) + srow) * HS + CW * hsel;
#pragma unroll
      for (int j = 0; j < CW; j += 4)
        store4_as<T>(sT, dst + j, typed, make_float4(sreg[j], sreg[j + 1], sreg[j + 2], sreg[j + 3]));
    }
    marked = __syncthreads_or(marked);
    if constexpr (RELAY) {
      if (tid == 0) store_cluster(cluster_addr(smem_u32(&sm.marks[rank]), 0), marked);
      __syncwarp();
      cluster_sync();      // from here on no CTA of the cluster touches another one
      for (int i = 0; i < n_cta; ++i) marked |= sm.marks[i];
    }
    if (tid == 0 && rank == 0) flags[unit] = marked != 0;
    if (PACKED && !RELAY && parts > 1 && c_hi == 0) take_next();
  }
  } else if (!PACKED || parts > 1) {
    take_next();
  }
  if (parts == 1) break;
  __syncthreads();      // the tiles and next_item are the next item's
  item = sm.next_item;
  __syncthreads();
  }   // items
  if (warp == 1 && elect_one()) bulk_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 128);
}

// ---------------------------------------------------------------------------------------------
// backward: one CTA per (batch, head), chunks in reverse; `states` holds the forward state at every
// chunk boundary (written by the forward kernel)
// ---------------------------------------------------------------------------------------------
// index of (row, channel) in a 64 x 64 fp32 array whose 16-byte pieces are permuted by the row: threads that own a row and
// threads that own a channel both access it without bank conflicts
__device__ __forceinline__ int sw64(int row, int c) { return row * 64 + ((((c >> 2) ^ (row & 7)) << 2) | (c & 3)); }

struct BwdSmem {
  unsigned char rt[2][TILE_BYTES];    // r~            [token][k]
  unsigned char kt[2][TILE_BYTES];    // k~            [token][k]
  // most of the twelve tiles below are used again for the fp32 staging arrays: v, S~0 and stril(dA) once the first part of
  // MMA batch 2 has completed, dy and A once all of it has
  unsigned char vt[2][TILE_BYTES];    // v             [token][v]
  unsigned char dyt[2][TILE_BYTES];   // dy            [token][v]
  unsigned char at[2][TILE_BYTES];    // A             [i][j]
  unsigned char dat[2][TILE_BYTES];   // stril(dA)     [i][j]
  unsigned char st[2][TILE_BYTES];    // S~0           [k][v]
  unsigned char dst[2][TILE_BYTES];   // dS^           [k][v]
  float gs[L * NROW];                 // gi - gref (prefix of g relative to the reference point)
  float gg[L * NROW];                 // g log2(e)
  float red_e[L * 64];                // dr~ r~ (sw64)
  float qtot[8][64];
  float rqtot[8][64];
  float pqtot[8][64];
  float dgs[64];                      // sum_k r u k per token
  float dds[64];                      // dy_i . v_i per token
  float dgl[4][64];                   // sum_v dS^ S~0, one partial per group of columns
  float du_s[64];
  // raw rows of the next chunk, requested by TMA a chunk ahead: w and dy (needed first) here; r and k land
  // in the space of rt / kt once the last epilogue has read those, v in red_e once the decay gradient has
  alignas(128) unsigned char raw_w[L * 64 * 4];
  alignas(128) unsigned char raw_dy[L * 64 * 4];
  uint64_t bar_1, bar_2, bar_2a, bar_in_a, bar_in_b, bar_in_c, bar_s;
  uint32_t tmem_base;
  int handoff_ok, next_item;
};
static_assert(sizeof(BwdSmem) + 1024 <= 227 * 1024, "backward shared memory");

// 512 threads: half the work of a phase per thread.  That pays only without spills (with shared memory taken to its limit there
// is no L1 for them): so the read-out takes eight columns at a time and stages them at once, and r and k are fetched again
// for the output rows.  B 16, T 4096, 32 heads, float32: 2237 us with 256 threads, 2032 with 512 (2750 with 280 bytes of
// spills).
constexpr int BWD_THREADS = 512;

template <typename T, bool PACKED>
__global__ void __launch_bounds__(BWD_THREADS)
wkv6c_bwd_kernel(const T* __restrict__ r, const T* __restrict__ k, const T* __restrict__ v, const T* __restrict__ w,
                 const float* __restrict__ u, const T* __restrict__ d_y, const float* __restrict__ d_sT,
                 const float* __restrict__ states, T* __restrict__ dr, T* __restrict__ dk, T* __restrict__ dv,
                 T* __restrict__ dw, float* __restrict__ du_partial, float* __restrict__ d_s0,
                 const __grid_constant__ CUtensorMap tmap_r, const __grid_constant__ CUtensorMap tmap_k,
                 const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_w,
                 const __grid_constant__ CUtensorMap tmap_dy, const __grid_constant__ CUtensorMap tmap_s, int Tn_dense, int H, Seqs seqs, int n_units,
                 int split, float* __restrict__ handoff, int* __restrict__ handoff_flags, int* status,
                 long long* dbg) {
#ifdef RWKVB200_DEVTOOLS
#define W6C_STAMP(n) do { if (dbg && tid == 0 && item == gridDim.x / 2 && c == NT - 2) dbg[n] = clock64(); } while (0)
#else
#define W6C_STAMP(n) do {} while (0)
#endif
  extern __shared__ unsigned char smem_raw[];
  BwdSmem& sm = *reinterpret_cast<BwdSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wq = warp & 3, hsel = warp >> 2;
  constexpr int NTHR = BWD_THREADS;
  constexpr int NE = Split<NTHR>::NE, PARTS = Split<NTHR>::PARTS, PL = Split<NTHR>::PL, CW = Split<NTHR>::CW;
  const long long tstride = (long long)H * HS;
  const int srow = 16 * wq + (lane & 15);
  const bool lower = lane < 16;
  const int c4 = tid & 15;
  // fp32 arrays (sw64) over tiles that the products are done with
  float* stage_dr = reinterpret_cast<float*>(sm.vt[0]);       // these three once the first part of batch 2 has completed
  float* stage_dk = reinterpret_cast<float*>(sm.st[0]);
  float* red_i = reinterpret_cast<float*>(sm.dat[0]);
  float* stage_dv = reinterpret_cast<float*>(sm.dyt[0]);
  float* stage_dw = reinterpret_cast<float*>(sm.at[0]);
  float* red_x = stage_dw;                     // X k~ per (token, channel), read before dw is staged over it

  if (tid == 0) {
    // every MMA batch is issued by two threads (of warps 0 and 1, each with accumulators of its own) and completes
    // with the arrival of both
    mbar_init(&sm.bar_1, 2); mbar_init(&sm.bar_2, 2); mbar_init(&sm.bar_2a, 2);
    mbar_init(&sm.bar_in_a, 1); mbar_init(&sm.bar_in_b, 1); mbar_init(&sm.bar_in_c, 1); mbar_init(&sm.bar_s, 1);
    fence_mbar_init();
  }
  if (tid == 32) tma_prefetch_maps(tmap_r, tmap_k, tmap_v, tmap_w, tmap_dy, tmap_s);
  if (warp == 0) tmem_alloc(&sm.tmem_base, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  earlier_kernels_done();
  later_kernels_may_start();
  const uint32_t tm = sm.tmem_base;
  const uint32_t tm_c0 = tmem_addr(tm, 32 * wq, CW * hsel);          // A (lower), dA (upper)
  const uint32_t tm_c1 = tmem_addr(tm, 32 * wq, 64 + CW * hsel);     // dk~ (lower), dr~ (upper)
  const uint32_t tm_c2 = tmem_addr(tm, 32 * wq, 128 + CW * hsel);    // dv (lower), dS~0 (upper)
  const uint32_t tm_c3 = tmem_addr(tm, 32 * wq, 192 + CW * hsel);    // X = v dS^^T (lower): the state part of dk~

  constexpr uint32_t RAW_BYTES = 64 * 64 * (uint32_t)sizeof(T);
  const T* raw_w = reinterpret_cast<const T*>(sm.raw_w);
  const T* raw_dy = reinterpret_cast<const T*>(sm.raw_dy);
  const T* raw_v = reinterpret_cast<const T*>(sm.red_e);
  const T* raw_r = reinterpret_cast<const T*>(sm.rt[0]);
  const T* raw_k = reinterpret_cast<const T*>(sm.kt[0]);

  // Work items.  Without `split` an item is a (batch, head) unit and the grid has one CTA per unit.  With it
  // (more units than SMs) every unit is two items, the later half of its chunks and the earlier half, and the
  // grid is one persistent CTA per SM; a CTA that is free takes the next item from a counter (handoff_flags
  // [n_units]).  All later halves come first in that order, so when an earlier half is taken its later half has
  // been taken before, by a CTA that is running, and the state gradient travels between them through `handoff` (a
  // flag per unit says it is there).  Halves of units instead of whole units even out the last round of CTAs
  // (512 units on 148 SMs: 3.5 unit times instead of 4).
  const int n_items = split ? 2 * n_units : n_units;
  bool ok = true;
  uint32_t n_done = 0;      // chunks this CTA has worked on: every barrier completes once per chunk
  for (bool first = true; ok; first = false) {
  if (split) {
    if (tid == 0) sm.next_item = atomicAdd(handoff_flags + n_units, 1);
    __syncthreads();
  } else if (!first) {
    break;
  }
  const int item = split ? sm.next_item : (int)blockIdx.x;
  if (item >= n_items) break;
  const int unit = split ? item % n_units : item;
  const bool early_half = split && item >= n_units;
  const int bi = unit / H, hi = unit % H;
  const int Tn = PACKED ? seqs.len[bi] : Tn_dense;
  const int tok0 = PACKED ? seqs.start[bi] : 0;
  const int brow = PACKED ? 0 : bi;
  const long long base = (((long long)brow * Tn_dense + tok0) * H + hi) * HS;
  const int NT = (Tn + L - 1) / L;
  const size_t nts = PACKED ? (size_t)seqs.nts : (size_t)(NT + 1);
  const int mid = split ? NT / 2 : 0;                 // the later half is chunks mid .. NT-1, the earlier 0 .. mid-1
  const int c_hi = early_half ? mid - 1 : NT - 1;     // first chunk of this item (chunks go in reverse)
  const int c_lo = early_half ? 0 : mid;              // last chunk of this item
  if (c_hi < c_lo) {                                  // an earlier half with nothing in it (a one-chunk sequence)
    if (tid < 64) du_partial[(size_t)item * HS + tid] = 0.f;
    __syncthreads();      // next_item is rewritten at the top
    continue;
  }
  const float4 u4 = *reinterpret_cast<const float4*>(u + hi * HS + 4 * c4);
  if (tid < 64) sm.du_s[tid] = 0.f;

  // gradient of the state after the current chunk: row k = srow (upper lane halves), 32 columns
  float dsreg[CW];
#pragma unroll
  for (int j = 0; j < CW; ++j) dsreg[j] = 0.f;
  if (early_half) {
    // wait for the later half of this unit (taken before this item, by a CTA that is running): bounded
    if (tid == 0) {
      uint32_t polls = 0;
      int seen = 0;
      while (true) {
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(handoff_flags + unit) : "memory");
        if (seen || ++polls > (WAIT_LIMIT << 2)) break;
        __nanosleep(200);
      }
      if (!seen) { atomicExch(status, 417); sm.handoff_ok = 0; } else { sm.handoff_ok = 1; }
    }
    __syncthreads();
    ok = sm.handoff_ok != 0;
    if (!lower && ok) {
      const float* S = handoff + (((size_t)unit * HS) + srow) * HS + CW * hsel;
#pragma unroll
      for (int j = 0; j < CW; j += 4) {
        const float4 f = __ldcg(reinterpret_cast<const float4*>(S + j));
        dsreg[j] = f.x; dsreg[j + 1] = f.y; dsreg[j + 2] = f.z; dsreg[j + 3] = f.w;
      }
    }
  } else if (!lower && d_sT) {
    const float* S = d_sT + (((size_t)unit * HS) + srow) * HS + CW * hsel;
#pragma unroll
    for (int j = 0; j < CW; j += 4) {
      const float4 f = *reinterpret_cast<const float4*>(S + j);
      dsreg[j] = f.x; dsreg[j + 1] = f.y; dsreg[j + 2] = f.z; dsreg[j + 3] = f.w;
    }
  }
  float4 du_acc = make_float4(0.f, 0.f, 0.f, 0.f);

  auto load_in_a = [&](int c) {      // tid 0; rows past the end of the sequence arrive as zeros
    mbar_expect_tx(&sm.bar_in_a, 2 * RAW_BYTES);
    tma_load_4d(sm.raw_w, &tmap_w, &sm.bar_in_a, 0, tok0 + c * L, hi, brow);
    tma_load_4d(sm.raw_dy, &tmap_dy, &sm.bar_in_a, 0, tok0 + c * L, hi, brow);
  };
  auto load_in_b = [&](int c) {
    mbar_expect_tx(&sm.bar_in_b, 2 * RAW_BYTES);
    tma_load_4d(sm.rt[0], &tmap_r, &sm.bar_in_b, 0, tok0 + c * L, hi, brow);
    tma_load_4d(sm.kt[0], &tmap_k, &sm.bar_in_b, 0, tok0 + c * L, hi, brow);
  };
  auto load_in_c = [&](int c) {
    mbar_expect_tx(&sm.bar_in_c, RAW_BYTES);
    tma_load_4d(sm.red_e, &tmap_v, &sm.bar_in_c, 0, tok0 + c * L, hi, brow);
  };
  if (warp == 0 && elect_one() && ok) { load_in_a(c_hi); load_in_c(c_hi); load_in_b(c_hi); }

  for (int c = c_hi; c >= c_lo && ok; --c, ++n_done) {
    const int t0 = c * L;
    const uint32_t par = n_done & 1;
    W6C_STAMP(32);
    float4 gw[NE], rr4[NE], kk4[NE];
    {
      ok = mbar_wait(&sm.bar_in_a, par, status, 413) && ok;
      // ---- pass W: g; pass DY: split tiles
#pragma unroll
      for (int n = 0; n < NE; ++n) {
        const int e = tid + NTHR * n, row = e >> 4, tok = t0 + row;
        const float4 w4 = load4_shared(raw_w + row * 64 + 4 * c4);
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tok < Tn)
          f = make_float4(-LOG2E * ex2(LOG2E * w4.x), -LOG2E * ex2(LOG2E * w4.y), -LOG2E * ex2(LOG2E * w4.z),
                          -LOG2E * ex2(LOG2E * w4.w));
        gw[n] = f;
        *reinterpret_cast<float4*>(&sm.gg[row * NROW + 4 * c4]) = f;
        float4 y4 = load4_shared(raw_dy + row * 64 + 4 * c4);
        if (PACKED && tok >= Tn) y4 = make_float4(0.f, 0.f, 0.f, 0.f);      // the next sequence's row
        store_split4<has_lo<T>()>(sm.dyt[0], sm.dyt[1], row, 4 * c4, y4);
      }
    }
    __syncthreads();
    W6C_STAMP(33);
    // S0 of this chunk (fp32, two 64 x 32 halves swizzled like the tiles) into the space of A, which nothing else uses until
    // MMA batch 1 is read out.  By TMA, because loads to registers are uncoalesced here and the proxy fence before batch
    // 1 waits for them.
    if (warp == 1 && elect_one() && ok) {
      fence_async_smem();
      const int srow0 = (int)(((size_t)unit * nts + c) * HS);
      mbar_expect_tx(&sm.bar_s, 2 * TILE_BYTES);
      tma_load_4d(sm.at[0], &tmap_s, &sm.bar_s, 0, srow0, 0, 0);
      tma_load_4d(sm.at[1], &tmap_s, &sm.bar_s, 32, srow0, 0, 0);
    }

    {
      const int ch = tid & 63, part = tid >> 6;
      float gv[PL];
#pragma unroll
      for (int j = 0; j < PL; ++j) gv[j] = sm.gg[(PL * part + j) * NROW + ch];
      float run = 0.f;
#pragma unroll
      for (int j = 0; j < PL; ++j) { run += gv[j]; gv[j] = run; }
      sm.qtot[part][ch] = run;
      __syncthreads();
      const float add = from_middle<PARTS>(sm.qtot, part, ch, run);
#pragma unroll
      for (int j = 0; j < PL; ++j) sm.gs[(PL * part + j) * NROW + ch] = gv[j] + add;
    }
    __syncthreads();
    W6C_STAMP(35);
    // ---- pass RK: scaled r, k (split, written over the raw rows once every thread has its elements) and
    // the diagonal term
    ok = mbar_wait(&sm.bar_in_b, par, status, 415) && ok;
    ok = mbar_wait(&sm.bar_in_c, par, status, 414) && ok;
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      const int row = (tid + NTHR * n) >> 4;
      rr4[n] = load4_shared(raw_r + row * 64 + 4 * c4);
      kk4[n] = load4_shared(raw_k + row * 64 + 4 * c4);
      // pass V: split tiles and dd_i = dy_i . v_i
      float4 v4 = load4_shared(raw_v + row * 64 + 4 * c4), y4 = load4_shared(raw_dy + row * 64 + 4 * c4);
      if (PACKED && t0 + row >= Tn) {
        v4 = make_float4(0.f, 0.f, 0.f, 0.f); y4 = v4; rr4[n] = v4; kk4[n] = v4;
      }
      store_split4<has_lo<T>()>(sm.vt[0], sm.vt[1], row, 4 * c4, v4);
      float dd = v4.x * y4.x + v4.y * y4.y + v4.z * y4.z + v4.w * y4.w;
#pragma unroll
      for (int m = 8; m >= 1; m >>= 1) dd += __shfl_xor_sync(0xffffffffu, dd, m);
      if (c4 == 0) sm.dds[row] = dd;
    }
    __syncthreads();
    if (warp == 0 && elect_one() && ok && c > c_lo) load_in_a(c - 1);      // every thread has taken its w and dy elements
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      const int e = tid + NTHR * n, row = e >> 4;
      const float4 r4 = rr4[n], k4 = kk4[n];
      const float4 gp = *reinterpret_cast<const float4*>(&sm.gs[row * NROW + 4 * c4]);
      const float d1x = gp.x, d1y = gp.y, d1z = gp.z, d1w = gp.w;   // gi - gref
      const float4 rs = make_float4(r4.x * ex2(d1x - gw[n].x), r4.y * ex2(d1y - gw[n].y),
                                    r4.z * ex2(d1z - gw[n].z), r4.w * ex2(d1w - gw[n].w));
      const float4 ks = make_float4(k4.x * ex2(-d1x), k4.y * ex2(-d1y), k4.z * ex2(-d1z), k4.w * ex2(-d1w));
      store_split4(sm.rt[0], sm.rt[1], row, 4 * c4, rs);
      store_split4(sm.kt[0], sm.kt[1], row, 4 * c4, ks);
      float dg = r4.x * u4.x * k4.x + r4.y * u4.y * k4.y + r4.z * u4.z * k4.z + r4.w * u4.w * k4.w;
#pragma unroll
      for (int m = 8; m >= 1; m >>= 1) dg += __shfl_xor_sync(0xffffffffu, dg, m);
      if (c4 == 0) sm.dgs[row] = dg;
    }
    if (warp == 0 && elect_one() && c > c_lo) {   // bring the previous chunk's rows into L2 while this chunk is in its MMA phases
      tma_prefetch_4d(&tmap_w, 0, tok0 + t0 - L, hi, brow);
      tma_prefetch_4d(&tmap_dy, 0, tok0 + t0 - L, hi, brow);
      tma_prefetch_4d(&tmap_v, 0, tok0 + t0 - L, hi, brow);
      tma_prefetch_4d(&tmap_r, 0, tok0 + t0 - L, hi, brow);
      tma_prefetch_4d(&tmap_k, 0, tok0 + t0 - L, hi, brow);
      // and the chunk-boundary state the previous chunk starts from
      bulk_prefetch_l2(states + ((size_t)unit * nts + c - 1) * HS * HS, HS * HS * (uint32_t)sizeof(float));
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();

    W6C_STAMP(36);
    // ---- batch 1: r~ k~^T (lower halves) and dy v^T (upper halves), columns 0..63
    if (warp == 0 && elect_one()) {
      tc_fence_after();
      umma_split<64, 64, 0, 0>(tmem_addr(tm, 0, 0), smem_u32(sm.rt[0]), smem_u32(sm.kt[0]), false);
      umma_commit(&sm.bar_1);
    }
    if (warp == 1 && elect_one()) {
      tc_fence_after();
      umma_split<64, 64, 0, 0, has_lo<T>(), has_lo<T>()>(tmem_addr(tm, 16, 0), smem_u32(sm.dyt[0]), smem_u32(sm.vt[0]), false);
      umma_commit(&sm.bar_1);
    }
    // decay factors of state row k = srow (both lanes of a pair work on that row below)
    const float e0 = ex2(fmaxf(half_sum<PARTS>(sm.qtot, 0, srow), EXP2_FLOOR));
    const float dlast = ex2(fmaxf(half_sum<PARTS>(sm.qtot, 1, srow), EXP2_FLOOR));
    // ---- state rows, while MMA batch 1 runs (it reads neither of the two tiles written here): the upper lane of a
    // pair holds dS and takes sum_v dS^ S~0 (the part of dglast that nothing
    // cancels) and dS^ = e^{glast-gref} dS_L, the lower lane takes S~0 = e^{gref} S0; one split-and-store call
    // serves both
    ok = mbar_wait(&sm.bar_s, par, status, 418) && ok;
    float4 srow4[CW / 4];      // the row of S0 (both lanes of a pair: the lower one for S~0, the upper one for sum_v dS^ S~0)
#pragma unroll
    for (int j = 0; j < CW / 4; ++j) {
      const int q = CW / 4 * hsel + j;      // 16-byte piece of the row
      srow4[j] = *reinterpret_cast<const float4*>(sm.at[q >> 3] + tile_chunk_off(srow, q & 7));
    }
    {
      float x[CW];
      if (!lower) {
        float acc = 0.f;
#pragma unroll
        for (int j = 0; j < CW; j += 4) {
          const float4 f = srow4[j >> 2];
          acc += dsreg[j] * f.x + dsreg[j + 1] * f.y + dsreg[j + 2] * f.z + dsreg[j + 3] * f.w;
        }
        sm.dgl[hsel][srow] = acc * (e0 * dlast);      // sum_v dS^ S~0 = e^{gref} e^{glast-gref} sum_v dS_L S0
#pragma unroll
        for (int j = 0; j < CW; ++j) { dsreg[j] *= dlast; x[j] = dsreg[j]; }     // dsreg now holds dS^
      } else {
#pragma unroll
        for (int j = 0; j < CW; j += 4) {
          const float4 f = srow4[j >> 2];
          x[j] = f.x * e0; x[j + 1] = f.y * e0; x[j + 2] = f.z * e0; x[j + 3] = f.w * e0;
        }
      }
      unsigned char* hi_t = lower ? sm.st[0] : sm.dst[0];
      store_split_row<CW>(hi_t, hi_t + TILE_BYTES, srow, CW * hsel, x);
    }
    ok = mbar_wait(&sm.bar_1, par, status, 411) && ok;
    tc_fence_after();
    ok = __syncthreads_and(ok);      // S0 has been read by every thread: A goes over it
    W6C_STAMP(37);
    if (ok) {
      const float dgi = lower ? sm.dgs[srow] : 0.f;     // the diagonal of A carries the u term; dA's does not
      // one call: both lane halves run the same code
      load_store_masked_row<CW>(tm_c0, wq, hsel, lane & 15, dgi, lower ? sm.at[0] : sm.dat[0], srow, true);
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);

    W6C_STAMP(38);
    // ---- batch 2, committed in two parts: the products the heavier part of the read-out needs first, so that its
    // arithmetic runs while the tensor pipe works on the rest (its results stay in registers until then: the
    // staging arrays lie over operand tiles of the products still running)
    if (warp == 0 && elect_one() && ok) {
      tc_fence_after();
      // dr~ = dy S~0^T + stril(dA) k~               (upper halves, columns 64..127)
      umma_split<64, 64, 0, 0, has_lo<T>(), true>(tmem_addr(tm, 16, 64), smem_u32(sm.dyt[0]), smem_u32(sm.st[0]), false);
      umma_split<64, 64, 0, 1>(tmem_addr(tm, 16, 64), smem_u32(sm.dat[0]), smem_u32(sm.kt[0]), true);
      umma_commit(&sm.bar_2a);
      // dv = A^T dy + k~ dS^                        (lower halves, columns 128..191)
      umma_split<64, 64, 1, 1, true, has_lo<T>()>(tmem_addr(tm, 0, 128), smem_u32(sm.at[0]), smem_u32(sm.dyt[0]), false);
      umma_split<64, 64, 0, 1>(tmem_addr(tm, 0, 128), smem_u32(sm.kt[0]), smem_u32(sm.dst[0]), true);
      umma_commit(&sm.bar_2);
    }
    if (warp == 1 && elect_one() && ok) {
      tc_fence_after();
      // the part of dk~ from inside the chunk, stril(dA)^T r~   (lower halves, columns 64..127: beside dr~, so
      // that one piece of code scales both in the epilogue)
      umma_split<64, 64, 1, 1>(tmem_addr(tm, 0, 64), smem_u32(sm.dat[0]), smem_u32(sm.rt[0]), false);
      // its state part X = v dS^^T apart (lower halves, columns 192..255): the decay gradient takes the two
      // parts of dk~ k~ in different sums
      umma_split<64, 64, 0, 0, has_lo<T>(), true>(tmem_addr(tm, 0, 192), smem_u32(sm.vt[0]), smem_u32(sm.dst[0]), false);
      umma_commit(&sm.bar_2a);
      // dS~0 = r~^T dy                              (upper halves, columns 128..191)
      umma_split<64, 64, 1, 1, true, has_lo<T>()>(tmem_addr(tm, 16, 128), smem_u32(sm.rt[0]), smem_u32(sm.dyt[0]), false);
      umma_commit(&sm.bar_2);
    }
    ok = mbar_wait(&sm.bar_2a, par, status, 416) && ok;
    tc_fence_after();
    const int c0 = CW * hsel;
    float rs[CW];
    if (ok) {
      float* so = lower ? stage_dk : stage_dr;
      float* sd = lower ? red_i : sm.red_e;
      // RB columns at a time (registers); what the remaining products still read is not written over yet
      constexpr int RB = 8;
#pragma unroll
      for (int jb = 0; jb < CW; jb += RB) {
        // r1: the part of dk~ from inside the chunk (lower halves) / dr~ (upper halves), row of token srow; rx: the
        // state part of dk~ (lower halves only)
        uint32_t r1[RB], rx[RB];
        tmem_ld<RB>(tm_c1 + jb, r1);
        tmem_ld<RB>(tm_c3 + jb, rx);
        float th[RB], tl[RB];
        tile_load_row<RB>(lower ? sm.kt[0] : sm.rt[0], srow, c0 + jb, th);
        tile_load_row<RB>(lower ? sm.kt[1] : sm.rt[1], srow, c0 + jb, tl);
        tmem_ld_wait();
#pragma unroll
        for (int j4 = 0; j4 < RB; j4 += 4) {
          const int cc = c0 + jb + j4;
          const float4 gs4 = *reinterpret_cast<const float4*>(&sm.gs[srow * NROW + cc]);
          const float4 gg4 = *reinterpret_cast<const float4*>(&sm.gg[srow * NROW + cc]);
          const float gsv[4] = {gs4.x, gs4.y, gs4.z, gs4.w}, ggv[4] = {gg4.x, gg4.y, gg4.z, gg4.w};
          float o[4], rd[4];
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            const int j = j4 + m;
            const float d1 = gsv[m];                                   // gi - gref
            const float tt = th[j] + tl[j];                            // k~ (lower) / r~ (upper)
            const float x = __uint_as_float(r1[j]);
            const float xs = lower ? __uint_as_float(rx[j]) : 0.f;
            o[m] = (x + xs) * ex2(lower ? -d1 : d1 - ggv[m]);          // dk = dk~ e^{gref-gi},  dr = dr~ e^{ge-gref}
            rd[m] = lower ? -x * tt : x * tt;                          // -(stril(dA)^T r~) k~,  dge = dr~ r~
            rs[jb + j] = xs * tt;                                      // X k~
          }
          *reinterpret_cast<float4*>(&so[sw64(srow, cc)]) = make_float4(o[0], o[1], o[2], o[3]);
          *reinterpret_cast<float4*>(&sd[sw64(srow, cc)]) = make_float4(rd[0], rd[1], rd[2], rd[3]);
        }
      }
    }
    ok = mbar_wait(&sm.bar_2, par, status, 412) && ok;
    tc_fence_after();
    W6C_STAMP(39);
    if (ok) {
      if (lower) {
#pragma unroll
        for (int j4 = 0; j4 < CW; j4 += 4)
          *reinterpret_cast<float4*>(&red_x[sw64(srow, c0 + j4)]) = make_float4(rs[j4], rs[j4 + 1], rs[j4 + 2], rs[j4 + 3]);
      }
      // dv row of token srow (lower halves) / dS~0 row k = srow (upper halves)
      uint32_t r2[CW];
      tmem_ld<CW>(tm_c2, r2);
      tmem_ld_wait();
      if (!lower) {
#pragma unroll
        for (int j = 0; j < CW; ++j) dsreg[j] = e0 * (__uint_as_float(r2[j]) + dsreg[j]);   // dS0 = e^{gref}(r~^T dy + dS^)
      } else {
#pragma unroll
        for (int j4 = 0; j4 < CW; j4 += 4)
          *reinterpret_cast<float4*>(&stage_dv[sw64(srow, c0 + j4)]) =
              make_float4(__uint_as_float(r2[j4]), __uint_as_float(r2[j4 + 1]), __uint_as_float(r2[j4 + 2]),
                          __uint_as_float(r2[j4 + 3]));
      }
    }
    // r and k once more, for the u terms of the output rows (they would take registers from here on back to where they were
    // scaled; these rows are in L2)
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      const int row = (tid + NTHR * n) >> 4;
      rr4[n] = kk4[n] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t0 + row < Tn) {
        const long long off = base + (long long)(t0 + row) * tstride + 4 * c4;
        rr4[n] = load4(r + off);
        kk4[n] = load4(k + off);
      }
    }
    tc_fence_before();
    ok = __syncthreads_and(ok);
    if (warp == 0 && elect_one() && ok && c > c_lo) load_in_b(c - 1);      // the epilogue above was the last reader of rt / kt
    W6C_STAMP(40);
    // ---- decay gradient, with I_i = -(stril(dA)^T r~)_i k~_i and X_i k~_i the two parts of dgi_i = -dk~_i k~_i:
    // dg_j = sum_{i>j} (dge_i + I_i) + I_j + sum_v dS^ S~0 + sum_{i<j} X_i k~_i;   dw = dg g.
    // (dglast = sum_v dS_L S_L contains sum_i X_i k~_i; taking the sum over i < j instead of dglast minus the
    // sum over i >= j keeps the two large, nearly equal terms from cancelling.)
    {
      const int ch = tid & 63, part = tid >> 6;
      float rv[PL], px[PL];
#pragma unroll
      for (int j = 0; j < PL; ++j) {
        const int at = sw64(PL * part + j, ch);
        rv[j] = red_i[at] + sm.red_e[at];
        px[j] = red_x[at];
      }
      float run = 0.f, prun = 0.f;
#pragma unroll
      for (int j = PL - 1; j >= 0; --j) { const float t = rv[j]; rv[j] = run; run += t; }      // sums over i > j
#pragma unroll
      for (int j = 0; j < PL; ++j) { const float t = px[j]; px[j] = prun; prun += t; }          // sums over i < j
      sm.rqtot[part][ch] = run;
      sm.pqtot[part][ch] = prun;
      __syncthreads();
      float add = 0.f;
#pragma unroll
      for (int q2 = 0; q2 < 64 / CW; ++q2) add += sm.dgl[q2][ch];
#pragma unroll
      for (int q2 = 1; q2 < PARTS; ++q2) if (q2 > part) add += sm.rqtot[q2][ch];
#pragma unroll
      for (int q2 = 0; q2 < PARTS - 1; ++q2) if (q2 < part) add += sm.pqtot[q2][ch];
#pragma unroll
      for (int j = 0; j < PL; ++j) {
        const int ii = PL * part + j;
        const float dg = (rv[j] + px[j]) + add + red_i[sw64(ii, ch)];
        // stage_dw lies over red_x: this thread has read its entries above and writes the same ones
        stage_dw[sw64(ii, ch)] = dg * (LN2 * sm.gg[ii * NROW + ch]);      // dw = dg g, g = gg ln 2
      }
    }
    __syncthreads();
    if (warp == 0 && elect_one() && ok && c > c_lo) load_in_c(c - 1);      // red_e has been read for the last time
    W6C_STAMP(41);
    // ---- outputs, coalesced, plus the u-term parts of dr, dk and du
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      const int e = tid + NTHR * n, row = e >> 4, tok = t0 + row;
      if (tok < Tn) {
        const long long off = base + (long long)tok * tstride + 4 * c4;
        const float4 r4 = rr4[n], k4 = kk4[n];
        const float dd = sm.dds[row];
        float4 a = *reinterpret_cast<const float4*>(&stage_dr[sw64(row, 4 * c4)]);
        a.x += dd * u4.x * k4.x; a.y += dd * u4.y * k4.y; a.z += dd * u4.z * k4.z; a.w += dd * u4.w * k4.w;
        store4(dr + off, a);
        float4 b = *reinterpret_cast<const float4*>(&stage_dk[sw64(row, 4 * c4)]);
        b.x += dd * r4.x * u4.x; b.y += dd * r4.y * u4.y; b.z += dd * r4.z * u4.z; b.w += dd * r4.w * u4.w;
        store4(dk + off, b);
        store4(dv + off, *reinterpret_cast<const float4*>(&stage_dv[sw64(row, 4 * c4)]));
        store4(dw + off, *reinterpret_cast<const float4*>(&stage_dw[sw64(row, 4 * c4)]));
        du_acc.x += dd * r4.x * k4.x; du_acc.y += dd * r4.y * k4.y;
        du_acc.z += dd * r4.z * k4.z; du_acc.w += dd * r4.w * k4.w;
      }
    }
    __syncthreads();
    W6C_STAMP(42);
  }
#undef W6C_STAMP
  // ---- du of this item and the gradient of the state at its first token: the initial state's, or what the
  // earlier half of the unit starts from
  atomicAdd(&sm.du_s[4 * c4], du_acc.x); atomicAdd(&sm.du_s[4 * c4 + 1], du_acc.y);
  atomicAdd(&sm.du_s[4 * c4 + 2], du_acc.z); atomicAdd(&sm.du_s[4 * c4 + 3], du_acc.w);
  __syncthreads();
  if (tid < 64) du_partial[(size_t)item * HS + tid] = sm.du_s[tid];
  const bool hand_on = split && !early_half && mid > 0;
  float* dS_out = hand_on ? handoff : d_s0;
  if (!lower && dS_out && ok) {
    float* dst = dS_out + (((size_t)unit * HS) + srow) * HS + CW * hsel;
#pragma unroll
    for (int j = 0; j < CW; j += 4)
      *reinterpret_cast<float4*>(dst + j) = make_float4(dsreg[j], dsreg[j + 1], dsreg[j + 2], dsreg[j + 3]);
  }
  if (hand_on) {
    __threadfence();
    __syncthreads();
    if (warp == 0 && elect_one() && ok) asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(handoff_flags + unit), "r"(1) : "memory");
  }
  __syncthreads();      // du_s and the tiles are the next item's
  }   // items
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 256);
}

// How many CTAs relay the chunks of a unit: a power of two, as many as there are chunks for and as can all be resident with
// the other units' clusters.
template <auto Kernel>
int relay_ctas(const DeviceFacts& dev, int smem, int n_units, int chunks) {
  int best = 2;
  for (int n = 2; n <= 8 && (n == 2 || 2 * chunks > n); n *= 2)
    if (n_units <= resident_clusters<Kernel>(dev, 256, smem, n)) best = n;
  return best;
}

}  // namespace w6c

int launch_wkv6_chunked_fwd(const void* r, const void* k, const void* v, const void* w, const void* u,
                            const void* s0, int n_state, const int32_t* smap, void* y, void* sT,
                            float* states, int* flags, float* handoff, int* hflags, int B, int Tn, int H,
                            int dtype, cudaStream_t st, const int32_t* seq_start, const int32_t* seq_len,
                            int T_total, bool typed) {
  using namespace w6c;
  // a packed batch: B sequences (the longest of Tn tokens) end to end in one row of T_total tokens
  const bool packed = seq_start != nullptr;
  const int mapB = packed ? 1 : B, mapT = packed ? T_total : Tn;
  const Seqs seqs{seq_start, seq_len, (Tn + L - 1) / L + 1};
  DeviceFacts dev;
  int e = device_facts(&dev);
  if (e) return e;
  int* status = dev.status;
  const int smem = (int)sizeof(FwdSmem) + 1024;
  const int esz = dtype == RWKVB200_F32 ? 4 : 2;
  CUtensorMap tm_r, tm_k, tm_v, tm_w, tm_y;
  e = make_row_tensor_map(&tm_r, r, mapB, mapT, H, esz);
  if (!e) e = make_row_tensor_map(&tm_k, k, mapB, mapT, H, esz);
  if (!e) e = make_row_tensor_map(&tm_v, v, mapB, mapT, H, esz, dtype == RWKVB200_BF16);      // as a tile, where that is all v needs
  if (!e) e = make_row_tensor_map(&tm_w, w, mapB, mapT, H, esz);
  if (!e) e = make_row_tensor_map(&tm_y, y ? y : r, mapB, mapT, H, esz, true);      // (unused without y)
  if (e) return e;
#define W6C_DISPATCH_PACKED(...) do { if (packed) { constexpr bool P = true; __VA_ARGS__; } else { constexpr bool P = false; __VA_ARGS__; } } while (0)
  {
    const int sms = dev.sms;
    const int n_units = B * H, slots = 2 * sms, NTmax = (Tn + L - 1) / L;
    int per_item = NTmax;
    if (n_units > slots) {
      // more units than the two CTAs per SM hold at once: every unit as 2 or 4 stretches of its chunks, whichever evens out
      // the last round best
      double best = (double)((n_units + slots - 1) / slots);      // rounds, in unit times
      for (int p2 = 2; p2 <= 4 && NTmax >= 4 * p2; p2 *= 2) {
        const double rounds = (double)(((long long)n_units * p2 + slots - 1) / slots) / p2;
        if (rounds < best - 1e-9) { best = rounds; per_item = (NTmax + p2 - 1) / p2; }
      }
    }
    const int parts = (NTmax + per_item - 1) / per_item;
    const int grid = parts > 1 ? slots : n_units;
    if (parts > 1)
      if (int rc = launch(w6c_clear_kernel, 1, 256, 0, st, 1, hflags, n_units + 1)) return rc;
    ProfScope prof("wkv6c_fwd_kernel", st);
    // few units: clusters of up to eight CTAs relay the chunks of one (see the kernel); a single chunk per unit: 512 threads, since
    // nothing else on the SM fills the waits of 256
#define W6C_LAUNCH_FWD(NTHR, RELAY)                                                                                \
    RWKVB200_DISPATCH_DTYPE(dtype, W6C_DISPATCH_PACKED(                                                               \
      if (allow_smem<wkv6c_fwd_kernel<T, P, NTHR, RELAY>>(dev, smem)) return RWKVB200_E_CUDA;                         \
      const int cluster = RELAY ? relay_ctas<wkv6c_fwd_kernel<T, P, NTHR, RELAY>>(dev, smem, n_units, NTmax) : 1;     \
      if (int rc = launch(wkv6c_fwd_kernel<T, P, NTHR, RELAY>, dim3(grid, cluster), NTHR, smem, st, cluster,          \
          (const T*)r, (const T*)k, (const T*)v, (const T*)w, u, s0, n_state, smap, (T*)y, sT, (int)typed, states, flags, \
          tm_r, tm_k, tm_v, tm_w, tm_y, mapT, H, seqs, n_units, per_item, parts, handoff, hflags, status, debug_stamp_buffer())) return rc))
    if (NTmax == 1 && n_units <= sms) W6C_LAUNCH_FWD(512, false)
    else if (2 * n_units <= slots)    W6C_LAUNCH_FWD(256, true)
    else                              W6C_LAUNCH_FWD(256, false)
#undef W6C_LAUNCH_FWD
  }
  e = check_launch();
  if (e) return e;
  // the marked units again, exactly: outputs, final state and (for the backward) the chunk-boundary states
  const long long unit_floats = (long long)seqs.nts * HS * HS;
  const UnitSel sel{flags, seq_start, seq_len, states ? unit_floats : 0};
  return launch_wkv6_fwd(r, k, v, w, u, s0, n_state, smap, y, sT, states, B, Tn, H, dtype, st, &sel, L, HS, typed);
}

}  // namespace rwkvb200

namespace rwkvb200 {

// workspace of the backward: [chunk-boundary states | du rows, two per unit | du rows of the recurrent
// fallback, four per unit | unit flags | state gradients handed from the later to the earlier half of a unit |
// their flags]; the forward fills the states and the unit flags
namespace {
struct W6Workspace { float* states; float* du_partial; float* du_partial_rec; int* flags; float* handoff; int* hflags; };
inline size_t a256(size_t x) { return (x + 255) & ~size_t(255); }
inline size_t w6_states_bytes(int B, int Tn, int H) {
  const size_t nt = (size_t)(Tn + w6c::L - 1) / w6c::L;
  return a256((size_t)B * H * (nt + 1) * HS * HS * sizeof(float));
}
inline W6Workspace w6_carve(void* workspace, int B, int Tn, int H) {
  char* p = reinterpret_cast<char*>(workspace);
  W6Workspace w;
  w.states = reinterpret_cast<float*>(p);
  p += w6_states_bytes(B, Tn, H);
  w.du_partial = reinterpret_cast<float*>(p);
  p += a256((size_t)B * H * 2 * HS * sizeof(float));
  w.du_partial_rec = reinterpret_cast<float*>(p);
  p += a256((size_t)B * H * 4 * HS * sizeof(float));
  w.flags = reinterpret_cast<int*>(p);
  p += a256((size_t)B * H * sizeof(int));
  w.handoff = reinterpret_cast<float*>(p);
  p += a256((size_t)B * H * HS * HS * sizeof(float));
  w.hflags = reinterpret_cast<int*>(p);      // one flag per unit, then the item counter
  return w;
}
}  // namespace

size_t wkv6_chunked_flags_bytes(int B, int H) { return a256((size_t)B * H * sizeof(int)); }

// scratch of a forward that keeps nothing for a backward: [unit flags | state hand-off | its flags and counter]
size_t wkv6_chunked_fwd_scratch_bytes(int B, int H) {
  return wkv6_chunked_flags_bytes(B, H) + a256((size_t)B * H * HS * HS * sizeof(float)) +
         a256(((size_t)B * H + 1) * sizeof(int));
}
void wkv6_chunked_fwd_scratch(void* workspace, int B, int H, int** flags, float** handoff, int** hflags) {
  char* p = reinterpret_cast<char*>(workspace);
  *flags = reinterpret_cast<int*>(p);
  p += wkv6_chunked_flags_bytes(B, H);
  *handoff = reinterpret_cast<float*>(p);
  p += a256((size_t)B * H * HS * HS * sizeof(float));
  *hflags = reinterpret_cast<int*>(p);
}
// the same three parts inside the backward's workspace (a forward that keeps its chunk-boundary states)
void wkv6_chunked_workspace_parts(void* workspace, int B, int Tn, int H, int** flags, float** handoff, int** hflags) {
  const W6Workspace w = w6_carve(workspace, B, Tn, H);
  *flags = w.flags; *handoff = w.handoff; *hflags = w.hflags;
}

size_t wkv6_chunked_bwd_workspace_bytes(int B, int Tn, int H) {
  return w6_states_bytes(B, Tn, H) + a256((size_t)B * H * 2 * HS * sizeof(float)) +
         a256((size_t)B * H * 4 * HS * sizeof(float)) + wkv6_chunked_flags_bytes(B, H) +
         a256((size_t)B * H * HS * HS * sizeof(float)) + a256(((size_t)B * H + 1) * sizeof(int));
}


int launch_wkv6_chunked_bwd(const void* r, const void* k, const void* v, const void* w, const float* u,
                            const float* s0, int n_state, const int32_t* smap, const void* d_y, const float* d_sT,
                            void* dr, void* dk, void* dv, void* dw, float* du, float* d_s0, void* workspace,
                            int B, int Tn, int H, int dtype, bool kept, cudaStream_t st,
                            const int32_t* seq_start, const int32_t* seq_len, int T_total) {
  using namespace w6c;
  const bool packed = seq_start != nullptr;
  const int mapB = packed ? 1 : B, mapT = packed ? T_total : Tn;
  const Seqs seqs{seq_start, seq_len, (Tn + L - 1) / L + 1};
  const W6Workspace ws = w6_carve(workspace, B, Tn, H);
  float* states = ws.states;
  float* du_partial = ws.du_partial;
  int e = RWKVB200_OK;
  if (!kept) {   // the workspace does not hold the chunk-boundary states yet: run the forward for them
    e = launch_wkv6_chunked_fwd(r, k, v, w, u, s0, n_state, smap, nullptr, nullptr, states, ws.flags, ws.handoff,
                                ws.hflags, B, Tn, H, dtype, st, seq_start, seq_len, T_total);
    if (e) return e;
  }
  DeviceFacts dev;
  e = device_facts(&dev);
  if (e) return e;
  int* status = dev.status;
  const int smem = (int)sizeof(BwdSmem) + 1024;
  bool split = false;
  {
    const int esz = dtype == RWKVB200_F32 ? 4 : 2;
    CUtensorMap tm_r, tm_k, tm_v, tm_w, tm_dy, tm_s;
    e = make_row_tensor_map(&tm_r, r, mapB, mapT, H, esz);
    if (!e) e = make_row_tensor_map(&tm_k, k, mapB, mapT, H, esz);
    if (!e) e = make_row_tensor_map(&tm_v, v, mapB, mapT, H, esz);
    if (!e) e = make_row_tensor_map(&tm_w, w, mapB, mapT, H, esz);
    if (!e) e = make_row_tensor_map(&tm_dy, d_y, mapB, mapT, H, esz);
    if (!e) e = make_state_tensor_map(&tm_s, states, (long long)B * H * seqs.nts * HS);
    if (e) return e;
    // more units than SMs: every unit as two half-length items on one persistent CTA per SM, which evens out
    // the last round (see the kernel); else one CTA per unit
    const int sms = dev.sms;
    const int n_units = B * H;
    split = n_units > sms && (Tn + L - 1) / L >= 4;
    const int grid = split ? sms : n_units;
    if (split)
      if (int rc = launch(w6c_clear_kernel, 1, 256, 0, st, 1, ws.hflags, n_units + 1)) return rc;
    ProfScope prof("wkv6c_bwd_kernel", st);
    RWKVB200_DISPATCH_DTYPE(dtype, W6C_DISPATCH_PACKED(
      if (allow_smem<wkv6c_bwd_kernel<T, P>>(dev, smem)) return RWKVB200_E_CUDA;
      if (int rc = launch(wkv6c_bwd_kernel<T, P>, grid, BWD_THREADS, smem, st, 1, (const T*)r, (const T*)k, (const T*)v, (const T*)w, u,
                          (const T*)d_y, d_sT, states, (T*)dr, (T*)dk, (T*)dv, (T*)dw,
                          du_partial, d_s0, tm_r, tm_k, tm_v, tm_w, tm_dy, tm_s, mapT, H, seqs,
                          n_units, split ? 1 : 0, ws.handoff, ws.hflags, status,
                          debug_stamp_buffer())) return rc));
  }
  e = check_launch();
  if (e) return e;
  // the units the forward marked: gradients from the float32 recurrence, which restarts from the (exact)
  // chunk-boundary states the fallback forward left in the workspace
  {
    const UnitSel sel{ws.flags, seq_start, seq_len, (long long)seqs.nts * HS * HS};
    e = launch_wkv6_bwd_coarse(r, k, v, w, u, d_y, d_sT, states, dr, dk, dv, dw, ws.du_partial_rec, d_s0, B, Tn, H,
                               dtype, st, &sel);
    if (e) return e;
  }
  return launch_wkv6_du_reduce_mixed(du_partial, ws.du_partial_rec, ws.flags, du, B, H, st, split ? 2 : 1);
}

}  // namespace rwkvb200
