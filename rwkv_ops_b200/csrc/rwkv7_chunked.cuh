// Chunked RWKV7 delta rule on tcgen05: shared definitions of the forward and backward kernels.
//
// Notation (one (batch, head), one chunk of L = 64 tokens, h = S^T is the [K][V] state):
//   g = -exp(w) per token and channel, gi / ge its inclusive / exclusive prefix sums inside the chunk,
//   gref = gi at token 31 (the reference point that keeps every exponent within +-32 |g|max),
//   glast = gi at token 63.
//   q~ = q e^{gi-gref}   k~ = k e^{gref-gi}   a~ = a e^{ge-gref}   b~ = b e^{gref-gi}
//   A_qk = tril(q~ k~^T)  A_qb = tril(q~ b~^T)  A_ak = stril(a~ k~^T)  A_ab = stril(a~ b~^T)
//   Ainv = (I - A_ab)^-1,  W = Ainv a~,  U = Ainv A_ak v
//   with h~0 = diag(e^{gref}) h0:
//     sa  = W h~0 + U                       (rows a_i^T h_{i-1})
//     o   = q~ h~0 + A_qk v + A_qb sa
//     h_L = diag(e^{glast-gref}) (h~0 + k~^T v + b~^T sa)
// Backward (do = grad of o, dh_L = grad of the state after the chunk, gref held constant: the result
// does not depend on it):
//     dh^  = diag(e^{glast-gref}) dh_L
//     dz   = Ainv^T (A_qb^T do + b~ dh^)  = C^T do + B2 dh^      (z = a~ h~0 + A_ak v,  sa = Ainv z)
//     with C = A_qb Ainv and B2 = Ainv^T b~
//     dh~0 = q~^T do + a~^T dz + dh^,   dh0 = diag(e^{gref}) dh~0
//     dv   = A_qk^T do + A_ak^T dz + k~ dh^
//     dA_qk = tril(do v^T)  dA_qb = tril(do sa^T)  dA_ak = stril(dz v^T)  dA_ab = stril(dz sa^T)
//     dq~ = do h~0^T + dA_qk k~ + dA_qb b~        da~ = dz h~0^T + dA_ak k~ + dA_ab b~
//     dk~ = dA_qk^T q~ + dA_ak^T a~ + v dh^^T     db~ = dA_qb^T q~ + dA_ab^T a~ + sa dh^^T
//     dq = dq~ e^{gi-gref} ...;  dgi = dq~ q~ - dk~ k~ - db~ b~;  dge = da~ a~;  dglast = sum_v dh^ X
//     dg_j = sum_{i>=j} (dgi_i + dge_i) - dge_j + dglast;   dw = dg g
// (reference: chunk_o_bwd.py:111-113,246-277,364-381, chunk_h_bwd.py:141-157, wy_fast_bwd.py:99-193,
// chunk_A_bwd.py:146-250,318-320 under rwkv_ops/rwkv7_kernel/triton_kernel/).
// These are the chunk equations of the reference's kernels (rwkv_ops/rwkv7_kernel/triton_kernel/
// chunk_A_fwd.py:111-165, wy_fast_fwd.py:57-62,273-321, chunk_h_fwd.py:140-150, chunk_o_fwd.py:82-136)
// rewritten around one reference point per chunk so that all four A matrices come out of a single
// 128x128x64 tensor-core product of pre-scaled bf16 operands.
//
// Two kernels per direction: an "intra" kernel, parallel over (batch, head, chunk), that produces the
// state-independent tiles, and a "scan" kernel, one CTA per (batch, head), that walks the chunks in
// order with the fp32 state resident in TMEM.  Tiles travel between them through the caller's
// workspace as raw 8 KB images of the swizzled shared-memory layout (tc.cuh), moved by bulk copies.
#pragma once

#include "common.cuh"
#include "tc.cuh"

namespace rwkvb200 {
namespace r7c {

constexpr int L = 64;                 // chunk length
// tiles of one chunk in the workspace, in this order (the first FWD_TILES feed the forward scan)
enum Slot { S_KT = 0, S_AQK, S_W, S_U, S_QT, S_BT, S_AQB, FWD_TILES,
            // kept for the backward: a~, A_ak (intra kernel); sa, h~0 and X = h~0 + k~^T v + b~^T sa (forward scan);
            // C = A_qb Ainv and B2 = Ainv^T b~ (intra kernel)
            S_AT = FWD_TILES, S_AAK, S_SA, S_H0, S_X, S_C, S_B2,
            // written by the reverse scan: dz = Ainv^T dsa and dh^ = e^{glast-gref} dh_L
            S_DZ, S_DHH, ALL_TILES };
constexpr int AUX_FLOATS = 128;       // per chunk: e^{gref}[64], e^{glast-gref}[64]

inline int num_chunks(int T) { return (T + L - 1) / L; }

// Which tokens a sequence occupies.  A dense batch has B sequences of Tn tokens, sequence bi in batch row
// bi of the token tensors.  A packed variable-length batch (start != nullptr) has its sequences laid end
// to end in ONE batch row; sequence bi is tokens start[bi] .. start[bi] + len[bi] - 1 of that row and Tn is
// the longest length: every sequence owns ceil(Tn / 64) chunk slots of the workspace and uses the first
// ceil(len / 64) of them.
// The kernels are compiled for both cases (template parameter PACKED), so that the dense case pays nothing.
struct SeqView {
  const int* start;   // device pointers, one entry per sequence, or nullptr
  const int* len;
  int Tn;
  template <bool PACKED> __device__ __forceinline__ int first(int bi) const {
    if constexpr (PACKED) return __ldg(start + bi); else return 0;
  }
  template <bool PACKED> __device__ __forceinline__ int length(int bi) const {
    if constexpr (PACKED) return __ldg(len + bi); else return Tn;
  }
  template <bool PACKED> __device__ __forceinline__ int row(int bi) const {
    if constexpr (PACKED) return 0; else return bi;
  }
};

// The chunk-heads that the persistent CTAs of a kernel work on, and in which order; `ch` is the workspace slot, n_ch after the
// last one.
struct ChunkPos { int ch, bi, hi, c; };
// (a kernel parameter, made on the host: computed in the kernels it would take registers that they do not have)
struct WalkDims {
  int H, NT, B, n_ch;
  int dh, db, dc;      // dense: the grid size as heads + H * (sequences + B * chunks), or, by unit, as chunks + NT * (heads + H * sequences)
  WalkDims(int H_, int NT_, int B_, int grid, bool by_unit = false)
      : H(H_), NT(NT_), B(B_), n_ch(H_ * NT_ * B_), dh(by_unit ? grid / NT_ % H_ : grid % H_),
        db(by_unit ? grid / NT_ / H_ : grid / H_ % B_), dc(by_unit ? grid % NT_ : grid / H_ / B_) {}
};
// Dense, by rows: every gridDim.x-th of a list in which the heads of one chunk of tokens follow each other, so that the CTAs at work
// at one time read and write whole token rows (H * 128 bytes) between them.  It goes through all sequences at once, from the last chunk
// to the first: what the kernel touches last is what the scan starts with, while it is still in L2.
struct RowWalk {
  const WalkDims& d;
  __device__ __forceinline__ void place(ChunkPos& p, int level) const {
    p.c = d.NT - 1 - level;
    p.ch = level < d.NT ? (p.bi * d.H + p.hi) * d.NT + p.c : d.n_ch;
  }
  __device__ __forceinline__ ChunkPos first() const {
    ChunkPos p;
    const int i = blockIdx.x;
    p.hi = i % d.H; p.bi = i / d.H % d.B;
    place(p, i / d.H / d.B);
    return p;
  }
  __device__ __forceinline__ ChunkPos after(ChunkPos p, int) const {      // p is in the list
    int level = d.NT - 1 - p.c + d.dc;
    p.hi += d.dh;
    p.bi += d.db;
    if (p.hi >= d.H) { p.hi -= d.H; ++p.bi; }
    if (p.bi >= d.B) { p.bi -= d.B; ++level; }
    place(p, level);
    return p;
  }
};

// Dense, by unit: every gridDim.x-th in the order of the workspace (WalkDims by unit).
struct UnitWalk {
  const WalkDims& d;
  __device__ __forceinline__ ChunkPos first() const {
    const int i = blockIdx.x;
    return ChunkPos{i, i / d.NT / d.H, i / d.NT % d.H, i % d.NT};
  }
  __device__ __forceinline__ ChunkPos after(ChunkPos p, int) const {
    p.ch += gridDim.x;
    p.c += d.dc;
    p.hi += d.dh;
    p.bi += d.db;
    if (p.c >= d.NT) { p.c -= d.NT; ++p.hi; }
    if (p.hi >= d.H) { p.hi -= d.H; ++p.bi; }
    return p;
  }
};

// Packed: the heads of one chunk, then of the next one of its sequence, then the next sequence; no slot past a sequence's end.  Again
// every gridDim.x-th, which may be many short sequences on: so the intra kernel's CTAs write down which sequence and chunk each of
// theirs is, once, and both kernels read that.  (A search from one to the next, every thread for itself: 4000 sequences of 8 .. 64
// tokens, one head, intra / final kernel 412 / 443 us against 127 / 148.  A stretch of neighbours for each CTA instead needs no list, but
// the CTAs then share no token rows: 8 sequences of up to 4096 tokens, 32 heads, 838 -> 880 us forward and backward.  Slots past a sequence's end left in the
// list, so that no search is needed: 1000 sequences of 30 .. 500 tokens, 12 heads, 2465 / 2816 us against 1670 / 1825.)
struct ListWalk {
  const WalkDims& d;
  const int2* list;      // of every chunk-head: sequence, chunk; -1 after the last one of each CTA
  __device__ __forceinline__ ChunkPos at(int i, int hi) const {
    const int2 e = __ldcg(list + i);
    return ChunkPos{e.x < 0 ? d.n_ch : (e.x * d.H + hi) * d.NT + e.y, e.x, hi, e.y};
  }
  __device__ __forceinline__ ChunkPos first() const { return at(blockIdx.x, blockIdx.x % d.H); }
  __device__ __forceinline__ ChunkPos after(const ChunkPos& p, int it) const {      // p: the CTA's it-th
    const int hi = p.hi + d.dh;
    return at(blockIdx.x + (it + 1) * gridDim.x, hi >= d.H ? hi - d.H : hi);
  }
};
// A CTA's part of the list; all 256 threads.  `sums`: shared memory of 8 ints.
__device__ __forceinline__ void write_list(int2* list, const SeqView& sv, const WalkDims& d, int* sums, int tid) {
  auto chunks = [&](int bi) { return min(max((sv.length<true>(bi) + L - 1) / L, 0), d.NT); };
  const int per = (d.B + 255) / 256, s0 = min(tid * per, d.B), s1 = min(s0 + per, d.B);
  int mine = 0;      // chunks of the sequences s0 .. s1 - 1
  for (int s = s0; s < s1; ++s) mine += chunks(s);
  int upto = mine;
#pragma unroll
  for (int o = 1; o < 32; o *= 2) {
    const int x = __shfl_up_sync(0xffffffffu, upto, o);
    if ((tid & 31) >= o) upto += x;
  }
  if ((tid & 31) == 31) sums[tid >> 5] = upto;
  __syncthreads();
  int from = upto - mine;
  for (int w = 0; w < (tid >> 5); ++w) from += sums[w];
  const int step = gridDim.x;
  int i = blockIdx.x;      // the CTA's first chunk-head in these sequences
  if (from * d.H > i) i += (from * d.H - i + step - 1) / step * step;
  for (int s = s0; s < s1; ++s) {
    const int n = chunks(s);
    for (; i < (from + n) * d.H; i += step) list[i] = make_int2(s, i / d.H - from);
    from += n;
  }
  if (tid == 255) list[i] = make_int2(-1, 0);
  __syncthreads();
}

// The unit of a scan's block in a packed batch where the blocks come in more than one round and that pays (scans_sorted): the longest
// sequences come first, so that the blocks which start when others have ended are short ones.  The sequences (MAX_SORTED at most) are
// ranked by length, by the threads of the block.
constexpr int MAX_SORTED = 256;
struct SortedSeqs { int len[MAX_SORTED], at; };
__device__ __forceinline__ int sorted_scan_unit(const SeqView& sv, int H, SortedSeqs* sorted, int tid) {
  const int n_seq = gridDim.x / H, b = blockIdx.x;
  if (tid < n_seq) sorted->len[tid] = __ldg(sv.len + tid);
  __syncthreads();
  if (tid < n_seq) {
    const int mine = sorted->len[tid];
    int rank = 0;
    for (int i = 0; i < n_seq; ++i) rank += sorted->len[i] > mine || (sorted->len[i] == mine && i < tid);
    if (rank == b / H) sorted->at = tid;
  }
  __syncthreads();
  return sorted->at * H + b % H;
}
// Whether the scans run one block to an SM.  Dense: with at most a sequence and head per SM.  Packed: also where an estimate of the
// two kernels' times says so (us, from the longest sequence, the mean and the units; the constants of a direction from the times of
// both on 23 batches, 3 .. 200 sequences of 8 .. 8000 tokens, 2 .. 64 heads; there and on 19 others it cost 7 % at most, 11 % once).  A block
// alone takes `chunk` per chunk and `block` besides; with two to an SM a chunk takes `free` .. `shared`, by how often an SM has
// two, but the start and end of one block lie under the other; and both move `kb` KB per chunk, at 6 TB/s at best.
// Forward / reverse, alone and two: 8 sequences of 1093 .. 4096 tokens, 32 heads 203 and 218 / 113 and 124; 8 of 2048 158 and 138 / 91 and
// 84; one of 8000 and 60 of 100, 16 heads 196 and 345 / 153 and 166; one of 3000 and 100 of 8, 64 heads 318 and 239 / 267 and 166.
struct ScanTimes { float kb, alone_memory, chunk, block, free, shared, slope; };
constexpr ScanTimes SCAN_FWD{96.f, 1.2f, 1.5f, 5.8f, 2.3f, 3.4f, 1.5f}, SCAN_REVERSE{47.f, 1.15f, 1.2f, 5.f, 1.28f, 1.94f, 0.9f};
inline bool scans_alone(int n_seq, int Tn, int T_total, int H, int sms, bool packed, const ScanTimes& t) {
  const int units = n_seq * H;
  if (units <= sms) return true;
  if (!packed || n_seq > MAX_SORTED) return false;
  const float longest = (float)num_chunks(Tn), mean = (float)T_total / n_seq / L + 0.5f, blocks = (float)units / sms;
  const float memory = units * mean * t.kb / 6000.f;
  const float alone = fmaxf(fmaxf(longest * t.chunk + t.block, memory * t.alone_memory + 3.f * blocks),
                            (blocks + 0.4f) * mean * t.chunk + blocks * t.block);
  const float two = fmaxf(longest * fminf(t.shared, t.free + t.slope * (blocks - 1.f)) + 5.f, memory + 2.9f * blocks);
  return alone < two;
}

// Whether the blocks of a packed batch's scans come longest sequence first.  Ranking the sequences costs a block 1 us and more (and the
// kernel its uniform registers), so with two blocks to an SM and several rounds of them it takes one sequence well above the mean
// (forward scan in order and sorted: 24 sequences of 300 .. 6000 tokens, 16 heads 411 and 358 us, 48 heads 887 and 790; 100 of 50 .. 600,
// 12 heads 133 and 145; 256 of 64, 12 heads 79 and 136).
inline bool scans_sorted(int n_seq, int Tn, int T_total, int H, int sms, bool alone) {
  const int units = n_seq * H;
  if (n_seq > MAX_SORTED || units <= (alone ? sms : 2 * sms)) return false;
  const float longest = (float)num_chunks(Tn), mean = (float)T_total / n_seq / L + 0.5f;
  return alone || longest - mean > (float)units / sms;
}

// Fused producers (template parameter FUSED of the intra and final kernels).  The three inputs w, a, b of
// the delta rule are then computed on the fly from pre-activations p, u, q of the same shape,
//   w = -e^{-1/2} sigmoid(p),   kk = u / max(|u|_2, 1e-12) over the 64 channels of a head,
//   a = -kk,   b = kk sigmoid(q),
// the elementwise tail of an RWKV7 time-mix block; each is rounded to bfloat16 exactly as if it had been
// materialised as a bfloat16 tensor, so the fused and the unfused operator return the same bits.
constexpr float W_SCALE = -0.60653065971263342f;
__device__ __forceinline__ float sigmoidf_(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// Rows 0 .. n_rows-1 of a swizzled bf16 tile to token rows `dst`, `dst + st`, ... (st in elements), by all
// NTHREADS threads of the CTA: the store of a chunk whose last rows belong to the next packed sequence,
// which a TMA store of the whole box would overwrite.
// (Kept out of line: it runs for one chunk per sequence and would only lengthen the persistent loops.)
template <int NTHREADS>
__device__ __noinline__ void store_tile_rows(__nv_bfloat16* dst, long long st, const unsigned char* tile,
                                                int n_rows, int tid) {
  for (int e = tid; e < 512; e += NTHREADS) {
    const int row = e >> 3, cc = e & 7;
    if (row < n_rows)
      *reinterpret_cast<uint4*>(dst + row * st + 8 * cc) = *reinterpret_cast<const uint4*>(tile + tc::tile_chunk_off(row, cc));
  }
}

struct Workspace {
  unsigned char* tiles;   // [n_chunks_total][tiles_per_chunk][8192]
  float* aux;             // [n_chunks_total][128]
  int* flags;             // [B*H] nonzero: the unit's decay left the range of the scaled operands (DECAY_LIMIT); written by
                          // the forward scan, from the signs of the e^{glast-gref} in aux
  int2* list;             // [n_chunks_total + MAX_GRID] which sequence and chunk the chunk-heads of a packed batch are (ListWalk)
  int tiles_per_chunk;
};
// The intra and the final kernel are persistent, two CTAs per SM; both have the same grid (ListWalk).
constexpr int MAX_GRID = 1024;
inline int persistent_grid(int n_ch, int sms) {
  const int most = 2 * sms < MAX_GRID ? 2 * sms : MAX_GRID;
  return n_ch < most ? n_ch : most;
}

// The scaled operands carry e^{+-(gi - gref)}: with the reference point in the middle of the chunk the
// exponent of a channel reaches the sum of |g| over half a chunk.  Up to DECAY_LIMIT every factor and every
// scaled state entry stays a normal bfloat16 / float32 number and the chunk equations are exact; a
// chunk with a larger half-chunk sum in a channel has that channel's e^{glast-gref} negated by the intra kernel, and a
// (batch, head) unit with such a chunk is recomputed by the float32 recurrence (rwkv7_recurrent.cuh: its outputs by the
// forward scan, which gathers the marks into Workspace::flags, its gradients by those flags), so the operator never
// returns values computed from clamped exponents.  |g| <= 1.875 per token never reaches the limit; RWKV7's
// own parametrisation keeps |g| below 0.61.
constexpr float DECAY_LIMIT = 60.f;
// Sequences shorter than this are recomputed by the recurrence as well (marked the same way): with one or
// two tokens the decay gradient is what is left of sums over the whole chunk that cancel almost completely
// (exactly zero for one token and no initial state), so the bfloat16 roundings of the chunk products would be all
// there is in dw; the recurrence costs nothing at that length.
constexpr int SHORT_SEQ = 8;

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

inline size_t fwd_workspace_bytes(int B, int T, int H, int tiles_per_chunk) {
  const size_t n = (size_t)B * H * num_chunks(T);
  return align256(n * tiles_per_chunk * tc::TILE_BYTES) + align256(n * AUX_FLOATS * sizeof(float)) +
         align256((size_t)B * H * sizeof(int)) + align256((n + MAX_GRID) * sizeof(int2)) + 1024;
}

inline Workspace carve(void* ws, int B, int T, int H, int tiles_per_chunk) {
  const size_t n = (size_t)B * H * num_chunks(T);
  Workspace w;
  uintptr_t p = (reinterpret_cast<uintptr_t>(ws) + 1023) & ~uintptr_t(1023);
  w.tiles = reinterpret_cast<unsigned char*>(p);
  w.aux = reinterpret_cast<float*>(p + align256(n * tiles_per_chunk * tc::TILE_BYTES));
  w.flags = reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(w.aux) + align256(n * AUX_FLOATS * sizeof(float)));
  w.list = reinterpret_cast<int2*>(reinterpret_cast<unsigned char*>(w.flags) + align256((size_t)B * H * sizeof(int)));
  w.tiles_per_chunk = tiles_per_chunk;
  return w;
}

}  // namespace r7c

// Phases of a forward / backward call (bit mask).  A whole call runs all of them in order; a caller that splits
// a sequence over several GPUs runs the state-independent phase on every GPU at once and only the scans one GPU
// after the other (the workspace carries everything from one phase to the next).
//   forward:  PREPARE = intra-chunk kernel;            SCAN = state scan over the chunks (+ exact fallback)
//   backward: PREPARE = forward recomputation (nothing, when the forward left its tiles);
//             SCAN = reverse scan (gradient of the state);   FINISH = token gradients (+ exact fallback)
enum Phase { PHASE_PREPARE = 1, PHASE_SCAN = 2, PHASE_FINISH = 4, PHASE_ALL = 7 };

// Backward of the chunked path; `workspace` must hold fwd_workspace_bytes(B, T, H, ALL_TILES).
// Packed variable-length batches: seq_start / seq_len are device arrays of B entries, Tn the longest length
// and T_total the number of tokens in the one batch row; dense batches pass nullptr, nullptr, 0.
// `fused`: w, a, b are the pre-activations p, u, q (dense batches only).
int launch_rwkv7_chunked_bwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                             const float* h0, int n_state, const void* d_o, const float* d_ht,
                             void* dr, void* dw, void* dk, void* dv, void* da, void* db, float* d_h0,
                             void* workspace, int B, int Tn, int H, int head_first, bool kept, cudaStream_t st,
                             const int* seq_start = nullptr, const int* seq_len = nullptr, int T_total = 0,
                             bool fused = false, int phases = PHASE_ALL);

int launch_rwkv7_chunked_fwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                             const float* h0, int n_state, void* o, float* ht, void* workspace,
                             int B, int Tn, int H, int head_first, bool keep_for_bwd, cudaStream_t st,
                             const int* seq_start = nullptr, const int* seq_len = nullptr, int T_total = 0,
                             bool fused = false, int phases = PHASE_ALL);

// Fused producers, backward: dw, da, db (in place in the three buffers) -> dp, du, dq.
int launch_rwkv7_producer_bwd(const void* p, const void* u, const void* q, void* dw_dp, void* da_du, void* db_dq,
                              long long n_rows, cudaStream_t st);

}  // namespace rwkvb200
