// Chunked RWKV7 forward on tcgen05 (bf16 token tensors, fp32 state).  Equations and the
// two-kernel structure are described in rwkv7_chunked.cuh.
#include "rwkv7_chunked.cuh"

namespace rwkvb200 {
namespace r7c {

using namespace tc;
typedef __nv_bfloat16 bf16;

// All decay sums of this file are in units of log 2 (tc::ex2).  No exponent is clamped: inside DECAY_LIMIT every
// factor is a normal number, and a unit beyond it is recomputed by the float32 recurrence whatever the
// tensor-core kernels wrote for it.
constexpr float EXP2_FLOOR = -126.f;      // 2^x below this is flushed to zero anyway

// ---------------------------------------------------------------------------------------------
// intra-chunk kernel: persistent CTAs of 256 threads over the B*H*NT chunk-heads
// ---------------------------------------------------------------------------------------------
// Tiles whose space is used over again; each line says what a tile holds in turn.  The order puts what is copied out
// together side by side: [q~ a~ k~ b~], [Q P N O' G B2], [W U].
struct IntraSmem {
  unsigned char qt[TILE_BYTES], at[TILE_BYTES];     // [q~; a~]  (128-row A operand)
  unsigned char kt[TILE_BYTES], bt[TILE_BYTES];     // [k~; b~]  (128-row B operand); bt: then Q
  unsigned char aqb[TILE_BYTES];                    // A_qb; P
  float nmat[L * 64];                               // the diagonal 32 x 32 blocks of A_ab, fp32; N (sw64)
  unsigned char aqk[TILE_BYTES];                    // A_qk; M_w; W^; O'
  unsigned char ainv[TILE_BYTES];                   // X = diag(X_A, X_B), completed to Ainv; G
  unsigned char x1[TILE_BYTES];                     // N_BA; B2
  unsigned char y[TILE_BYTES], aak[TILE_BYTES];     // e^{gi-gref}, fp32 (sw64, both tiles); then
                                                    //   y: v (TMA); Y = A_ak v; M_u; W      aak: A_ak; S; U
  unsigned char wv[TILE_BYTES];                     // raw w (TMA)
  float qtot[4][64];                                // sums of g over the four quarters of the chunk
  float vec[3][64];                                 // e^{gref}, e^{glast-gref}, e^{-gref}
  uint64_t bar_v, bar_w, bar_in, bar_b, bar_m1, bar_m2, bar_m3, bar_m4, bar_m5;
  uint32_t tmem_base;
};
static_assert(sizeof(IntraSmem) + 1024 <= 116736, "two CTAs per SM");

// Persistent: CTAs (two per SM) walk over chunk-heads ch = blockIdx.x, blockIdx.x + gridDim.x, ...  The raw tiles of
// the next chunk-head are requested by TMA as soon as the tiles they land in are free.
//
// What bounds it is the chain of phases inside a chunk-head (products -> read-out -> products ...), with two CTAs per SM
// filling each other's waits.  The triangular inverse Ainv = (I - N)^-1, N = stril(A_ab), therefore takes two turns:
//   * the two diagonal 32 x 32 blocks X_A, X_B in fp32, one column per thread, by the two warps that read those blocks of
//     A_ab from TMEM, beside MMA 2 of the other six warps;
//   * the rest on the tensor cores without ever waiting for Ainv itself: with X = diag(X_A, X_B), M = X [a~ | Y] and
//     S = X N_BA (MMA 3), [W | U] = Ainv [a~ | Y] = M + S M and the last block of Ainv is S X (MMA 4).  (S is a
//     correction: rounding it and the M it multiplies to bf16 changes less than the rounding of W and U does.)
// An issuing thread gets an MMA out every 80 cycles, so the accumulators of a group have issuing threads of their own.
// TMEM: columns 0..127 MMA 1; then (M = 64 accumulators pair up on the two lane halves)
//   0..63 P | Q;   64..127 M, then W | U;   128..191 Y, then S | S X, then G | B2;   192..255 N | O' (from MMA 2 on).
// 256 threads: warp w reads TMEM lanes 32*(w&3).. and the two warps that share a lane window split
// the columns (hsel = w>>2).
template <bool PACKED, bool FUSED>
__global__ void __launch_bounds__(256, 2)
r7c_intra_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_w,
                     const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_a,
                     const __grid_constant__ CUtensorMap tmap_b,
                     const __grid_constant__ CUtensorMap tmap_v, unsigned char* __restrict__ ws_tiles,
                     float* __restrict__ ws_aux, int* __restrict__ ws_flags, int tiles_per_chunk,
                     int keep_for_bwd, SeqView sv, int H, int NT, int n_ch, int* status, long long* dbg) {
#ifdef RWKVB200_DEVTOOLS
#define R7C_STAMP(n) do { if (dbg && tid == 0 && blockIdx.x == gridDim.x / 2 && it == 15) dbg[n] = clock64(); } while (0)
#define R7C_STAMPD(n) do { if (dbg && tid == 192 && blockIdx.x == gridDim.x / 2 && it == 15) dbg[n] = clock64(); } while (0)
#else
#define R7C_STAMP(n) do {} while (0)
#define R7C_STAMPD(n) do {} while (0)
#endif
  extern __shared__ unsigned char smem_raw[];
  IntraSmem& sm = *reinterpret_cast<IntraSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wq = warp & 3, hsel = warp >> 2;
  const bool st_thread = tid == 64;      // requests raw tiles, copies results out
  // threads 0, 32, 96, 128 issue the MMAs
  const int issuer = lane == 0 ? (warp < 2 ? warp : warp == 3 || warp == 4 ? warp - 1 : -1) : -1;

  if (tid == 0) {
    mbar_init(&sm.bar_v, 1); mbar_init(&sm.bar_w, 1); mbar_init(&sm.bar_in, 1); mbar_init(&sm.bar_b, 1);
    mbar_init(&sm.bar_m1, 1); mbar_init(&sm.bar_m2, 3); mbar_init(&sm.bar_m3, 3); mbar_init(&sm.bar_m4, 3);
    mbar_init(&sm.bar_m5, 4);
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(&sm.tmem_base, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = sm.tmem_base;

  // The raw tiles of a chunk-head (rows past the end of the sequence arrive as zeros); all of st_thread
  auto load = [&](unsigned char* dst, const CUtensorMap* map, uint64_t* bar, const ChunkPos& p) {
    tma_load_4d(dst, map, bar, 0, sv.first<PACKED>(p.bi) + p.c * L, p.hi, sv.row<PACKED>(p.bi));
  };
  auto load_w = [&](const ChunkPos& p) { mbar_expect_tx(&sm.bar_w, TILE_BYTES); load(sm.wv, &tmap_w, &sm.bar_w, p); };
  auto load_v = [&](const ChunkPos& p) { mbar_expect_tx(&sm.bar_v, TILE_BYTES); load(sm.y, &tmap_v, &sm.bar_v, p); };
  // q, k, a share a barrier; k comes first
  auto load_k = [&](const ChunkPos& p) { mbar_expect_tx(&sm.bar_in, 3 * TILE_BYTES); load(sm.kt, &tmap_k, &sm.bar_in, p); };
  auto load_q = [&](const ChunkPos& p) { load(sm.qt, &tmap_q, &sm.bar_in, p); };
  auto load_a = [&](const ChunkPos& p) { load(sm.at, &tmap_a, &sm.bar_in, p); };
  auto load_b = [&](const ChunkPos& p) { mbar_expect_tx(&sm.bar_b, TILE_BYTES); load(sm.bt, &tmap_b, &sm.bar_b, p); };
  // chunk slots past the end of a (packed) sequence are skipped
  auto empty = [&](const ChunkPos& p) {
    if constexpr (!PACKED) return false;      // a dense batch has no empty slots
    return p.c * L >= sv.length<PACKED>(p.bi);
  };
  auto advance = [&](ChunkPos p) {
    do { chunk_step(p, gridDim.x, NT, H); } while (p.ch < n_ch && empty(p));
    return p;
  };
  // Ask for the token rows that are loaded late in a chunk-head to be brought into L2 before.
  auto prefetch_rows = [&](const ChunkPos& p) {      // one thread
    const int tt = sv.first<PACKED>(p.bi) + p.c * L, br = sv.row<PACKED>(p.bi);
    tma_prefetch_4d(&tmap_a, 0, tt, p.hi, br);
    tma_prefetch_4d(&tmap_q, 0, tt, p.hi, br);
    tma_prefetch_4d(&tmap_b, 0, tt, p.hi, br);
    tma_prefetch_4d(&tmap_v, 0, tt, p.hi, br);
  };
  ChunkPos cur = chunk_pos(blockIdx.x, NT, H);
  if (cur.ch < n_ch && empty(cur)) cur = advance(cur);
  if (cur.ch < n_ch && st_thread) { load_w(cur); load_k(cur); load_q(cur); load_a(cur); load_b(cur); }
  // The two CTAs that share an SM would otherwise run their phases in lockstep and compete for the same unit; start
  // every other CTA half a chunk-head late, where there is more than one chunk-head per CTA.
  if ((blockIdx.x & 1) && n_ch > 2 * gridDim.x) __nanosleep(6000);

  bool ok = true;
  int it = 0;
  for (ChunkPos nxt; cur.ch < n_ch && ok; cur = nxt, ++it) {
    const int ch = cur.ch, bi = cur.bi, hi = cur.hi, t0 = cur.c * L;
    const int Tn = sv.length<PACKED>(bi);
    unsigned char* out_tiles = ws_tiles + (size_t)ch * tiles_per_chunk * TILE_BYTES;
    const uint32_t par = it & 1;
    nxt = advance(cur);
    const bool more = nxt.ch < n_ch;

    R7C_STAMP(0);
    // ---- phase A: decay prefix sums (in units of log 2), thread = (channel, quarter of the chunk), straight from the
    // raw w tile; what everybody needs of them is e^{gi-gref}: its reciprocal is the factor of k~ and b~, and the row
    // before gives the factor of a~
    float* eqs = reinterpret_cast<float*>(sm.y);
    ok = mbar_wait(&sm.bar_w, par, status, 206) && ok;
    {
      const int c = tid & 63, quarter = tid >> 6;
      float gi[16];
      float run = 0.f;
      const int n_rows = Tn - t0 - 16 * quarter;      // rows of this quarter inside the sequence
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        float w = __uint_as_float((uint32_t)*reinterpret_cast<const unsigned short*>(sm.wv + tile_off(16 * quarter + j, c)) << 16);
        if constexpr (FUSED) w = round_bf16(W_SCALE * sigmoidf_(w));      // the tile holds p: w = -e^{-1/2} sigmoid(p), as bfloat16
        const float e = ex2(LOG2E * w);
        if (j < n_rows) run -= LOG2E * e;
        gi[j] = run;
      }
      sm.qtot[quarter][c] = run;
      __syncthreads();
      if (st_thread && more) load_w(nxt);      // every thread has taken its w
      R7C_STAMP(1);
      // gi - gref: the prefix inside the half; the reference point is the end of the first half
      const float add = quarter == 0 ? -(run + sm.qtot[1][c]) : quarter == 1 ? -run : quarter == 3 ? sm.qtot[2][c] : 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) eqs[sw64(16 * quarter + j, c)] = ex2(gi[j] + add);
      if (quarter == 0) {
        const float tot0 = -add, tot1 = sm.qtot[2][c] + sm.qtot[3][c];
        const float eg = ex2(fmaxf(tot0, EXP2_FLOOR)), dl = ex2(fmaxf(tot1, EXP2_FLOOR));
        sm.vec[0][c] = eg;                                   // e^{gref}
        sm.vec[1][c] = dl;                                   // e^{glast-gref}
        sm.vec[2][c] = ex2(add);                             // for the exclusive prefix of the first token
        ws_aux[(size_t)ch * AUX_FLOATS + c] = eg;
        ws_aux[(size_t)ch * AUX_FLOATS + 64 + c] = dl;
        // a half-chunk decay sum beyond the limit: the unit is recomputed by the float32 recurrence
        if (fminf(tot0, tot1) < -DECAY_LIMIT * LOG2E || Tn < SHORT_SEQ) ws_flags[bi * H + hi] = 1;
      }
    }
    R7C_STAMP(71);
    ok = mbar_wait(&sm.bar_in, par, status, 207) && ok;
    R7C_STAMP(72);
    __syncthreads();
    R7C_STAMP(73);
    // ---- the raw q, k, a, b: each thread scales its own 2 x 16 bytes (8 channels of a token) in place; b, which comes
    // last, after the others
    float ek[2][8];
    uint4 fb[2];      // FUSED: b
    if constexpr (FUSED) ok = mbar_wait(&sm.bar_b, par, status, 208) && ok;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int e = tid + 256 * n, row = e >> 3, cc = e & 7;
      const uint32_t off = tile_chunk_off(row, cc);
      uint4 rq = *reinterpret_cast<const uint4*>(sm.qt + off), rk = *reinterpret_cast<const uint4*>(sm.kt + off);
      uint4 ra = *reinterpret_cast<const uint4*>(sm.at + off);
      if (PACKED && t0 + row >= Tn) {      // in a packed batch these rows belong to the next sequence
        rq = make_uint4(0u, 0u, 0u, 0u); rk = rq; ra = rq;
      }
      if constexpr (FUSED) {      // the a / b tiles hold u and q: a = -kk, b = kk sigmoid(q), kk = u / |u|
        const uint4 rb = *reinterpret_cast<const uint4*>(sm.bt + off);
        const uint32_t uu[4] = {ra.x, ra.y, ra.z, ra.w}, qq[4] = {rb.x, rb.y, rb.z, rb.w};
        float uv[8], ss = 0.f;
#pragma unroll
        for (int m = 0; m < 4; ++m) { uv[2 * m] = bf16_lo(uu[m]); uv[2 * m + 1] = bf16_hi(uu[m]); }
#pragma unroll
        for (int x = 0; x < 8; ++x) ss += uv[x] * uv[x];
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);      // the 8 threads of a token row are neighbouring lanes
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        ss += __shfl_xor_sync(0xffffffffu, ss, 4);
        const float inv = rsqrtf(fmaxf(ss, 1e-24f));      // 1 / max(|u|, 1e-12)
        uint32_t na[4], nb[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const float k0 = uv[2 * m] * inv, k1 = uv[2 * m + 1] * inv;
          na[m] = pack_bf16(-k0, -k1);
          nb[m] = pack_bf16(k0 * sigmoidf_(bf16_lo(qq[m])), k1 * sigmoidf_(bf16_hi(qq[m])));
        }
        ra = make_uint4(na[0], na[1], na[2], na[3]);
        fb[n] = make_uint4(nb[0], nb[1], nb[2], nb[3]);
      }
      float eq[8], ea[8];      // e^{gi-gref} of the row; e^{ge-gref}: of the row before it
      *reinterpret_cast<float4*>(eq) = *reinterpret_cast<const float4*>(&eqs[sw64(row, 8 * cc)]);
      *reinterpret_cast<float4*>(eq + 4) = *reinterpret_cast<const float4*>(&eqs[sw64(row, 8 * cc + 4)]);
      const float* g0 = row ? &eqs[sw64(row - 1, 8 * cc)] : &sm.vec[2][8 * cc];
      const float* g1 = row ? &eqs[sw64(row - 1, 8 * cc + 4)] : &sm.vec[2][8 * cc + 4];
      *reinterpret_cast<float4*>(ea) = *reinterpret_cast<const float4*>(g0);
      *reinterpret_cast<float4*>(ea + 4) = *reinterpret_cast<const float4*>(g1);
      const uint32_t uq[4] = {rq.x, rq.y, rq.z, rq.w}, uk[4] = {rk.x, rk.y, rk.z, rk.w}, ua[4] = {ra.x, ra.y, ra.z, ra.w};
      uint32_t oq[4], ok_[4], oa[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        ek[n][2 * m] = rcp(eq[2 * m]); ek[n][2 * m + 1] = rcp(eq[2 * m + 1]);
        float x0, x1;
        mul2(x0, x1, bf16_lo(uq[m]), bf16_hi(uq[m]), eq[2 * m], eq[2 * m + 1]); oq[m] = pack_bf16(x0, x1);
        mul2(x0, x1, bf16_lo(uk[m]), bf16_hi(uk[m]), ek[n][2 * m], ek[n][2 * m + 1]); ok_[m] = pack_bf16(x0, x1);
        mul2(x0, x1, bf16_lo(ua[m]), bf16_hi(ua[m]), ea[2 * m], ea[2 * m + 1]); oa[m] = pack_bf16(x0, x1);
      }
      *reinterpret_cast<uint4*>(sm.qt + off) = make_uint4(oq[0], oq[1], oq[2], oq[3]);
      *reinterpret_cast<uint4*>(sm.kt + off) = make_uint4(ok_[0], ok_[1], ok_[2], ok_[3]);
      *reinterpret_cast<uint4*>(sm.at + off) = make_uint4(oa[0], oa[1], oa[2], oa[3]);
    }
    if constexpr (!FUSED) ok = mbar_wait(&sm.bar_b, par, status, 208) && ok;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int e = tid + 256 * n, row = e >> 3;
      const uint32_t off = tile_chunk_off(row, e & 7);
      uint4 rb;
      if constexpr (FUSED) rb = fb[n]; else rb = *reinterpret_cast<const uint4*>(sm.bt + off);
      if (PACKED && t0 + row >= Tn) rb = make_uint4(0u, 0u, 0u, 0u);
      const uint32_t ub[4] = {rb.x, rb.y, rb.z, rb.w};
      uint32_t ob[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        float x0, x1;
        mul2(x0, x1, bf16_lo(ub[m]), bf16_hi(ub[m]), ek[n][2 * m], ek[n][2 * m + 1]); ob[m] = pack_bf16(x0, x1);
      }
      *reinterpret_cast<uint4*>(sm.bt + off) = make_uint4(ob[0], ob[1], ob[2], ob[3]);
    }
    if (st_thread) bulk_wait_read();      // the previous results have left their tiles, which are rewritten from here on
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);

    R7C_STAMP(2);
    // ---- MMA 1: [q~; a~] [k~; b~]^T  ->  TMEM columns 0..127, row r on lane r
    if (tid == 0 && ok) {
      tc_fence_after();
      umma_tile<128, 128, 0, 0>(tm, smem_u32(sm.qt), smem_u32(sm.kt), false);
      umma_commit(&sm.bar_m1);
    }
    if (st_thread && ok) {
      load_v(cur);      // the prefix sums have been read
      if (keep_for_bwd) {
        bulk_store(out_tiles + S_QT * TILE_BYTES, sm.qt, 4 * TILE_BYTES);      // q~, a~, k~, b~
        bulk_commit();
      }
    }
    if (more && tid == 128) prefetch_rows(nxt);
    ok = ok && mbar_wait(&sm.bar_m1, par, status, 201);
    tc_fence_after();
    R7C_STAMP(3);
    // Rows r < 64 are q~'s, the others a~'s; the warp's 32 rows are i = 32*ihalf + lane, so which side of the diagonal
    // a block of 32 columns lies on is the same for the whole warp: left of the diagonal block every element is kept,
    // right of it every element is zero (TMEM is not read), and only the diagonal block takes a per-element choice.
    const int ihalf = wq & 1;
    if (warp < 6) {      // A_qk (warps 0, 1), A_ak (2, 3), A_qb (4, 5)
      if (ok) {
        const int i = 32 * ihalf + lane;
        const bool strict = wq >= 2;
        unsigned char* dst = hsel ? sm.aqb : strict ? sm.aak : sm.aqk;
#pragma unroll
        for (int pp = 0; pp < 2; ++pp) {
          float x[32];
          uint32_t rr[32];
          if (pp > ihalf) {
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] = 0.f;
          } else {
            tmem_ld32(tmem_addr(tm, 32 * wq, 64 * hsel + 32 * pp), rr);   // hsel 0: products with k~, 1: with b~
            tmem_ld_wait();
            if (pp < ihalf) {
#pragma unroll
              for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) x[j] = (strict ? j < lane : j <= lane) ? __uint_as_float(rr[j]) : 0.f;
            }
          }
          tile_store_row32(dst, i, 32 * pp, x);
        }
      }
      fence_async_smem();
      tc_fence_before();
      ok = bar_sync_and(1, 192, ok);

      R7C_STAMP(4);
      // ---- MMA 2: Y = A_ak v (columns 128..191), and the first terms of N = k~^T v | O' = A_qk v (columns 192..255)
      if (issuer >= 0 && issuer < 3 && ok) {
        ok = mbar_wait(&sm.bar_v, par, status, 202);
        tc_fence_after();
        R7C_STAMP(68);
        if (issuer == 0)      umma_tile<64, 64, 0, 1>(tmem_addr(tm, 0, 128), smem_u32(sm.aak), smem_u32(sm.y), false);
        else if (issuer == 1) umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, 192), smem_u32(sm.kt), smem_u32(sm.y), false);
        else                  umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 192), smem_u32(sm.aqk), smem_u32(sm.y), false);
        umma_commit(&sm.bar_m2);
      }
      if (st_thread && ok && keep_for_bwd) {
        bulk_store(out_tiles + S_AQK * TILE_BYTES, sm.aqk, TILE_BYTES);
        bulk_store(out_tiles + S_AAK * TILE_BYTES, sm.aak, TILE_BYTES);
        bulk_commit();
      }
      ok = ok && mbar_wait(&sm.bar_m2, par, status, 203);
      tc_fence_after();
      R7C_STAMP(69);
      if (ok) {      // Y rows (lower lane halves); warps 2, 3 take both column halves of theirs
#pragma unroll
        for (int pp = 0; pp < 2; ++pp) {
          if (pp != hsel && wq < 2) continue;
          uint32_t rr[32];
          tmem_ld32(tmem_addr(tm, 32 * wq, 128 + 32 * pp), rr);
          tmem_ld_wait();
          if (lane < 16) {
            float x[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
            tile_store_row32(sm.y, 16 * wq + lane, 32 * pp, x);
          }
        }
      }
      if (st_thread && ok) {
        bulk_wait_read();                // q~, a~, k~, b~, A_qk, A_ak have left shared memory
        if (more) load_k(nxt);           // MMA 2 was the last to read k~
      }
    } else {             // warps 6, 7: the diagonal blocks of A_ab, inverted at once; warp 7 also N_BA
      if (ok) {
        R7C_STAMPD(64);
        float* nd = sm.nmat + 1024 * ihalf;       // this warp's 32 x 32 block, one row per lane
        uint32_t rr[32];
        float x[32];
        tmem_ld32(tmem_addr(tm, 32 * wq, 64 + 32 * ihalf), rr);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; j += 4)      // (entries at or right of the diagonal are never used)
          *reinterpret_cast<uint4*>(&nd[32 * lane + (((j >> 2) ^ (lane & 7)) << 2)]) = make_uint4(rr[j], rr[j + 1], rr[j + 2], rr[j + 3]);
        if (ihalf) {
          tmem_ld32(tmem_addr(tm, 32 * wq, 64), rr);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
          tile_store_row32(sm.x1, 32 + lane, 0, x);         // N_BA, and zeros to its right (MMA 3 reads rows 32..63)
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = 0.f;
        if (ihalf) tile_store_row32(sm.x1, 32 + lane, 32, x);
        tile_store_row32(sm.ainv, ihalf ? lane : 32 + lane, ihalf ? 32 : 0, x);      // the off-diagonal blocks of X
        __syncwarp();
        R7C_STAMPD(65);
        // Column `lane` of (I - N)^-1, row after row: x[r] = [r == lane] + sum_{j<r} N[r][j] x[j], two terms per
        // instruction, and the newest x last, so that the chain from row to row is one multiply-add.  The row after
        // the current one is on its way from shared memory.
        float4 nr[2][8];
        nr[1][0] = *reinterpret_cast<const float4*>(&nd[32 * 1 + ((0 ^ 1) << 2)]);
        x[0] = lane == 0 ? 1.f : 0.f;
#pragma unroll
        for (int r = 1; r < 32; ++r) {
          if (r + 1 < 32) {
#pragma unroll
            for (int m = 0; m < (r + 4) / 4; ++m)
              nr[(r + 1) & 1][m] = *reinterpret_cast<const float4*>(&nd[32 * (r + 1) + ((m ^ ((r + 1) & 7)) << 2)]);
          }
          const float* n = reinterpret_cast<const float*>(nr[r & 1]);
          float p0 = r == lane ? 1.f : 0.f, p1 = 0.f;
#pragma unroll
          for (int j = 0; j + 1 < r - 1; j += 2) fma2(p0, p1, n[j], n[j + 1], x[j], x[j + 1], p0, p1);
          if (r >= 2 && (r & 1) == 0) p1 += n[r - 2] * x[r - 2];
          x[r] = n[r - 1] * x[r - 1] + (p0 + p1);
        }
        R7C_STAMPD(66);
#pragma unroll
        for (int r = 0; r < 32; r += 2) {
          const uint32_t u = pack_bf16(x[r], x[r + 1]);
          *reinterpret_cast<unsigned short*>(sm.ainv + tile_off(32 * ihalf + r, 32 * ihalf + lane)) = (unsigned short)u;
          *reinterpret_cast<unsigned short*>(sm.ainv + tile_off(32 * ihalf + r + 1, 32 * ihalf + lane)) = (unsigned short)(u >> 16);
        }
        R7C_STAMPD(67);
      }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);

    R7C_STAMP(5);
    const int i = 16 * wq + (lane & 15), c0 = 32 * hsel;
    const bool lo = lane < 16;
    // ---- MMA 3: M = X a~ | X Y (columns 64..127), S = X N_BA (columns 128..191)
    if (issuer >= 0 && issuer < 3 && ok) {
      tc_fence_after();
      if (issuer == 0)      umma_tile<64, 64, 0, 1>(tmem_addr(tm, 0, 64), smem_u32(sm.ainv), smem_u32(sm.at), false);
      else if (issuer == 1) umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 64), smem_u32(sm.ainv), smem_u32(sm.y), false);
      else                  umma_tile<64, 64, 0, 1, 2, 2>(tmem_addr(tm, 0, 128), smem_u32(sm.ainv), smem_u32(sm.x1), false);
      umma_commit(&sm.bar_m3);
    }
    ok = ok && mbar_wait(&sm.bar_m3, par, status, 204);
    tc_fence_after();
    R7C_STAMP(6);
    if (st_thread && ok && more) load_a(nxt);      // MMA 3 was the last to read a~
    if (ok) {      // rows 0..31 of M (what S multiplies); S (its first 32 columns, zero in rows 0..31)
      uint32_t rr[32];
      float x[32];
      if (wq < 2) {
        tmem_ld32(tmem_addr(tm, 32 * wq, 64 + c0), rr);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
        tile_store_row32(lo ? sm.aqk : sm.y, i, c0, x);
      } else if (!hsel) {
        tmem_ld32(tmem_addr(tm, 32 * wq, 128), rr);
        tmem_ld_wait();
        if (lo) {
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
          tile_store_row32(sm.aak, i, 0, x);
        }
      } else if (lo) {
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = 0.f;
        tile_store_row32(sm.aak, i - 32, 0, x);
      }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);

    R7C_STAMP(7);
    // ---- MMA 4: W | U = M + S M (columns 64..127), the last block of Ainv S X (columns 128..191, upper halves)
    if (issuer >= 0 && issuer < 3 && ok) {
      tc_fence_after();
      if (issuer == 0)      umma_tile<64, 64, 0, 1, 2>(tmem_addr(tm, 0, 64), smem_u32(sm.aak), smem_u32(sm.aqk), true);
      else if (issuer == 1) umma_tile<64, 64, 0, 1, 2>(tmem_addr(tm, 16, 64), smem_u32(sm.aak), smem_u32(sm.y), true);
      else                  umma_tile<64, 64, 0, 1, 2>(tmem_addr(tm, 16, 128), smem_u32(sm.aak), smem_u32(sm.ainv), false);
      umma_commit(&sm.bar_m4);
    }
    ok = ok && mbar_wait(&sm.bar_m4, par, status, 209);
    tc_fence_after();
    R7C_STAMP(8);
    if (ok) {
      uint32_t rr[32];
      float x[32];
      tmem_ld32(tmem_addr(tm, 32 * wq, 64 + c0), rr);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
      if (!lo) {
        tile_store_row32(sm.aak, i, c0, x);                         // U
      } else {
        if (keep_for_bwd) tile_store_row32(sm.y, i, c0, x);         // W
#pragma unroll
        for (int j = 0; j < 32; j += 4) {                           // W^
          const float4 e = *reinterpret_cast<const float4*>(&sm.vec[0][c0 + j]);
          mul2(x[j], x[j + 1], x[j], x[j + 1], e.x, e.y);
          mul2(x[j + 2], x[j + 3], x[j + 2], x[j + 3], e.z, e.w);
        }
        tile_store_row32(sm.aqk, i, c0, x);
      }
      if (keep_for_bwd && wq >= 2 && !hsel) {      // rows 32..63, columns 0..31 of Ainv
        tmem_ld32(tmem_addr(tm, 32 * wq, 128), rr);
        tmem_ld_wait();
        if (!lo) {
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
          tile_store_row32(sm.ainv, i, 0, x);
        }
      }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);

    R7C_STAMP(9);
    // ---- MMA 5: P = b~^T W^ | Q = A_qb W^ (columns 0..63); N += b~^T U | O' += A_qb U (columns 192..255); for the
    // backward G = A_qb Ainv | B2 = Ainv^T b~ (columns 128..191)
    if (issuer >= 0 && ok) {
      tc_fence_after();
      if (issuer == 0) {
        umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, 0), smem_u32(sm.bt), smem_u32(sm.aqk), false);
      } else if (issuer == 1) {
        umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, 192), smem_u32(sm.bt), smem_u32(sm.aak), true);
      } else if (issuer == 2) {
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 0), smem_u32(sm.aqb), smem_u32(sm.aqk), false);
        if (keep_for_bwd) umma_tile<64, 64, 0, 1>(tmem_addr(tm, 0, 128), smem_u32(sm.aqb), smem_u32(sm.ainv), false);
      } else {
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 192), smem_u32(sm.aqb), smem_u32(sm.aak), true);
        if (keep_for_bwd) umma_tile<64, 64, 1, 1>(tmem_addr(tm, 16, 128), smem_u32(sm.ainv), smem_u32(sm.bt), false);
      }
      umma_commit(&sm.bar_m5);
    }
    if (st_thread && ok && keep_for_bwd) {
      bulk_store(out_tiles + S_W * TILE_BYTES, sm.y, 2 * TILE_BYTES);      // W, U
      bulk_commit();
    }
    ok = ok && mbar_wait(&sm.bar_m5, par, status, 205);
    tc_fence_after();
    R7C_STAMP(10);
    if (ok) {
      uint32_t rr[32];
      float x[32];
      tmem_ld32(tmem_addr(tm, 32 * wq, c0), rr);
      tmem_ld_wait();
      const float dl = sm.vec[1][i];
      if (lo) {      // P, row i = key channel
#pragma unroll
        for (int j = 0; j < 32; j += 2) mul2(x[j], x[j + 1], __uint_as_float(rr[j]), __uint_as_float(rr[j + 1]), dl, dl);
      } else {       // Q = q~ e^{gref} + A_qb W^, row i = token
        tile_load_row32(sm.qt, i, c0, x);
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 e = *reinterpret_cast<const float4*>(&sm.vec[0][c0 + j]);
          fma2(x[j], x[j + 1], x[j], x[j + 1], e.x, e.y, __uint_as_float(rr[j]), __uint_as_float(rr[j + 1]));
          fma2(x[j + 2], x[j + 3], x[j + 2], x[j + 3], e.z, e.w, __uint_as_float(rr[j + 2]), __uint_as_float(rr[j + 3]));
        }
      }
      tile_store_row32(lo ? sm.aqb : sm.bt, i, c0, x);
      tmem_ld32(tmem_addr(tm, 32 * wq, 192 + c0), rr);
      tmem_ld_wait();
      if (lo) {      // N, float32
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          *reinterpret_cast<float4*>(&sm.nmat[sw64(i, c0 + j)]) =
              make_float4(__uint_as_float(rr[j]) * dl, __uint_as_float(rr[j + 1]) * dl, __uint_as_float(rr[j + 2]) * dl,
                          __uint_as_float(rr[j + 3]) * dl);
      } else {       // O'
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
        tile_store_row32(sm.aqk, i, c0, x);
      }
      if (keep_for_bwd) {      // G | B2
        tmem_ld32(tmem_addr(tm, 32 * wq, 128 + c0), rr);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
        tile_store_row32(lo ? sm.ainv : sm.x1, i, c0, x);
      }
    }
    if (st_thread) bulk_wait_read();      // W, U have left their tiles, which take the next prefix sums
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    R7C_STAMP(11);
    if (st_thread && ok) {
      bulk_store(out_tiles + S_Q * TILE_BYTES, sm.bt, TILE_BYTES);                                   // Q
      bulk_commit();
      bulk_store(out_tiles + S_P * TILE_BYTES, sm.aqb, (keep_for_bwd ? 6 : 4) * TILE_BYTES);         // P, N, O' (G, B2)
      bulk_commit();
      if (more) {
        load_q(nxt);              // q~ was last read by the epilogue
        bulk_wait_read_1();       // Q has left its tile
        load_b(nxt);
      }
    }
  }
  if (st_thread) bulk_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 256);
#undef R7C_STAMP
}

// ---------------------------------------------------------------------------------------------
// scan kernel: grid = B*H, 256 threads, chunks in order: h <- e^{glast} h + P h + N,  o = Q h + O'
// ---------------------------------------------------------------------------------------------
// One 128x64x64 product per chunk, [Q; P] h, row r on TMEM lane r: warps 2, 3 (and 6, 7 for the upper 32 columns) own
// the state rows, warps 0, 1 (4, 5) the token rows.  The two groups meet through mbarriers only.  The chain from
// chunk to chunk runs through the state warps: h (fp32, registers) -> bf16 tile -> product -> read-out -> h; the token
// warps write the output a chunk behind, from the other one of two accumulators.
// STAGES = 2: two CTAs (two sequences) share an SM, the choice when there are more sequences than SMs; bound by the
// 40 KB of tiles per chunk there.  STAGES = 4: one CTA per SM with loads three chunks ahead, for few sequences; the
// latency of the chain bounds it.
struct ScanStage {
  unsigned char q[TILE_BYTES], p[TILE_BYTES];      // [Q; P]  (128-row A operand)
  float n[L * 64];                                 // N
  unsigned char o[TILE_BYTES];                     // O'
};
template <int STAGES>
struct ScanSmem {
  ScanStage st[STAGES];
  unsigned char ht[TILE_BYTES];             // h as bf16, [k][v]
  unsigned char hs[2][TILE_BYTES];          // h~0 = e^{gref} h as bf16 (kept for the backward)
  unsigned char ot[TILE_BYTES];             // output rows of a chunk, staged for a TMA store
  uint64_t bar_ld[STAGES], bar_free[STAGES], bar_m[2], bar_o[2];
  uint32_t tmem_base;
};
static_assert(sizeof(ScanSmem<2>) <= 115712, "two CTAs per SM");

template <int STAGES, bool PACKED>
__global__ void __launch_bounds__(256, STAGES == 2 ? 2 : 1)
r7c_scan_fwd_kernel(const unsigned char* __restrict__ ws_tiles, const float* __restrict__ ws_aux, int tiles_per_chunk,
                    unsigned char* __restrict__ bwd_tiles, unsigned char* __restrict__ fin_tiles,
                    const float* __restrict__ h0, int n_state, const __grid_constant__ CUtensorMap tmap_o,
                    int write_o, float* __restrict__ ht, bf16* __restrict__ o_rows, SeqView sv, int H, int NT_slots,
                    TokLayout lay, int* status) {
  extern __shared__ __align__(1024) unsigned char smem_al[];
  ScanSmem<STAGES>& sm = *reinterpret_cast<ScanSmem<STAGES>*>(smem_al);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wq = warp & 3, hsel = warp >> 2, c0 = 32 * hsel;
  if (smem_u32(smem_al) & 1023u) {      // the swizzled tiles need this alignment; there is no room to align by hand
    if (tid == 0) atomicCAS(status, 0, 216);
    return;
  }
  const int unit = blockIdx.x, bi = unit / H, hi = unit % H;
  const size_t ch0 = (size_t)unit * NT_slots;
  const int Tn = sv.length<PACKED>(bi), tb = sv.first<PACKED>(bi), brow = sv.row<PACKED>(bi);
  const int NT = (Tn + L - 1) / L;           // chunks of this sequence (at least one)
  const bool state_warp = wq >= 2;
  const int row = 32 * (wq & 1) + lane;      // state row k or token row i

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&sm.bar_ld[s], 1); mbar_init(&sm.bar_free[s], 8); }
    for (int t = 0; t < 2; ++t) { mbar_init(&sm.bar_m[t], 1); mbar_init(&sm.bar_o[t], 4); }
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(&sm.tmem_base, 128);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = sm.tmem_base;

  auto issue_load = [&](int c) {
    ScanStage& g = sm.st[c % STAGES];
    mbar_expect_tx(&sm.bar_ld[c % STAGES], sizeof(ScanStage));
    bulk_load(g.q, ws_tiles + (ch0 + c) * (size_t)tiles_per_chunk * TILE_BYTES, sizeof(ScanStage), &sm.bar_ld[c % STAGES]);
  };
  bool ok = true;
  if (state_warp) {
    float x[32];      // h[k = row][c0 .. c0 + 31]
    if (n_state > 0) {
      const float* S = h0 + (size_t)(n_state == 1 ? hi : unit) * 4096;   // S[v][k], h[k][v] = S[v][k]
#pragma unroll
      for (int j = 0; j < 32; ++j) x[j] = S[(c0 + j) * 64 + row];
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) x[j] = 0.f;
    }
    float eg_next = ws_aux[ch0 * AUX_FLOATS + row], dl_next = ws_aux[ch0 * AUX_FLOATS + 64 + row];
    for (int c = 0; c < NT; ++c) {
      const int s = c % STAGES, t = c & 1;
      const uint32_t sp = (c / STAGES) & 1, tp = (c >> 1) & 1;
      const float eg = eg_next, dl = dl_next;
      if (c + 1 < NT) {      // fetched a chunk ahead
        eg_next = ws_aux[(ch0 + c + 1) * AUX_FLOATS + row];
        dl_next = ws_aux[(ch0 + c + 1) * AUX_FLOATS + 64 + row];
      }
      tile_store_row32(sm.ht, row, c0, x);
      if (tid == 96 && bwd_tiles) bulk_wait_read();      // the h~0 tile about to be rewritten has left shared memory
      fence_async_smem();
      tc_fence_before();
      ok = bar_sync_and(1, 128, ok);      // the one place where the group may leave the loop: all of it or none
      if (!ok) break;
      if (tid == 64) {
        ok = mbar_wait(&sm.bar_ld[s], sp, status, 211);
        if (c >= 2) ok = mbar_wait(&sm.bar_o[t], ((c >> 1) - 1) & 1, status, 212) && ok;      // this accumulator has been read
        if (ok) {
          tc_fence_after();
          umma_tile<128, 64, 0, 1>(tmem_addr(tm, 0, 64 * t), smem_u32(sm.st[s].q), smem_u32(sm.ht), false);
          umma_commit(&sm.bar_m[t]);
        }
      }
      if (bwd_tiles) {      // h~0 for the backward, under the product; its tile of the chunk before goes out now
        if (tid == 96 && c > 0) {
          bulk_store(bwd_tiles + ((ch0 + c - 1) * (size_t)tiles_per_chunk + S_H0) * TILE_BYTES, sm.hs[t ^ 1], TILE_BYTES);
          bulk_commit();
        }
        float y[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) y[j] = x[j] * eg;
        tile_store_row32(sm.hs[t], row, c0, y);
      }
      ok = ok && mbar_wait(&sm.bar_ld[s], sp, status, 213);
      ok = ok && mbar_wait(&sm.bar_m[t], tp, status, 214);
      tc_fence_after();
      if (ok) {
        uint32_t r[32];
        tmem_ld32(tmem_addr(tm, 32 * wq, 64 * t + c0), r);
        tmem_ld_wait();
        const float et = eg * dl;
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 n4 = *reinterpret_cast<const float4*>(&sm.st[s].n[sw64(row, c0 + j)]);
          x[j] = et * x[j] + (__uint_as_float(r[j]) + n4.x);
          x[j + 1] = et * x[j + 1] + (__uint_as_float(r[j + 1]) + n4.y);
          x[j + 2] = et * x[j + 2] + (__uint_as_float(r[j + 2]) + n4.z);
          x[j + 3] = et * x[j + 3] + (__uint_as_float(r[j + 3]) + n4.w);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.bar_free[s]);
      }
    }
    // ---- the final state: fp32 for the caller, a bf16 tile for the backward
    if (ok && ht) {
      float* S = ht + (size_t)unit * 4096;
#pragma unroll
      for (int j = 0; j < 32; ++j) S[(c0 + j) * 64 + row] = x[j];
    }
    if (bwd_tiles) {
      if (ok) tile_store_row32(sm.ht, row, c0, x);
      fence_async_smem();
      ok = bar_sync_and(1, 128, ok);
      if (tid == 96) {
        if (ok) {
          bulk_store(bwd_tiles + ((ch0 + NT - 1) * (size_t)tiles_per_chunk + S_H0) * TILE_BYTES, sm.hs[(NT - 1) & 1], TILE_BYTES);
          bulk_store(fin_tiles + (size_t)unit * TILE_BYTES, sm.ht, TILE_BYTES);
          bulk_commit();
        }
        bulk_wait_all();
      }
    }
  } else {
    const bool ld_thread = tid == 0;
    bool ld_ok = true;
    if (ld_thread)
      for (int c = 0; c < STAGES && c < NT; ++c) issue_load(c);
    for (int c = 0; c < NT; ++c) {
      const int s = c % STAGES, t = c & 1, t0 = c * L;
      const uint32_t sp = (c / STAGES) & 1, tp = (c >> 1) & 1;
      ok = mbar_wait(&sm.bar_ld[s], sp, status, 215);
      ok = ok && mbar_wait(&sm.bar_m[t], tp, status, 217);
      tc_fence_after();
      if (ok) {
        uint32_t r[32];
        float x[32];
        tmem_ld32(tmem_addr(tm, 32 * wq, 64 * t + c0), r);
        tmem_ld_wait();
        tc_fence_before();
        tile_load_row32(sm.st[s].o, row, c0, x);
        __syncwarp();
        if (lane == 0) { mbar_arrive(&sm.bar_o[t]); mbar_arrive(&sm.bar_free[s]); }
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] += __uint_as_float(r[j]);
        if (ld_thread) bulk_wait_read();      // the output tile of the chunk before has left shared memory
        bar_sync(2, 128);
        tile_store_row32(sm.ot, row, c0, x);
        fence_async_smem();
      } else {
        bar_sync(2, 128);
      }
      ok = bar_sync_and(2, 128, ok && ld_ok);      // the one place where the group may leave the loop
      if (!ok) break;
      if (write_o) {
        if (PACKED && t0 + L > Tn) {  // the last rows of the box belong to the next sequence: row by row
          store_tile_rows<128>(o_rows + brow * lay.sb + hi * lay.sh + (long long)(tb + t0) * lay.st, lay.st,
                               sm.ot, Tn - t0, 32 * ((warp & 1) + 2 * hsel) + lane);
        } else if (ld_thread) {           // rows past the end of the tensor are clipped by the TMA store
          tma_store_4d(&tmap_o, sm.ot, 0, tb + t0, hi, brow);
          bulk_commit();
        }
      }
      if (ld_thread && c + STAGES < NT) {
        ld_ok = mbar_wait(&sm.bar_free[s], sp, status, 218);
        if (ld_ok) issue_load(c + STAGES);
      }
    }
    if (ld_thread) bulk_wait_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 128);
}

}  // namespace r7c

int launch_rwkv7_chunked_fwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                             const float* h0, int n_state, void* o, float* ht, void* workspace,
                             int B, int Tn, int H, int head_first, bool keep_for_bwd, cudaStream_t st,
                             const int* seq_start, const int* seq_len, int T_total, bool fused, int phases) {
  using namespace r7c;
  typedef __nv_bfloat16 bf16;
  if (fused && seq_start) return RWKVB200_E_UNSUPPORTED;
  const SeqView sv{seq_start, seq_len, Tn};
  const int mapB = seq_start ? 1 : B, mapT = seq_start ? T_total : Tn;   // shape of the token tensors
  int* status = device_status_ptr();
  if (!status) { last_cuda_error_slot() = 99999; return RWKVB200_E_CUDA; }
  CUtensorMap tmap_v, tmap_o;
  int e = make_token_tensor_map(&tmap_v, v, mapB, mapT, H, head_first);
  if (e) return e;
  e = make_token_tensor_map(&tmap_o, o ? o : v, mapB, mapT, H, head_first);   // unused when o is NULL
  if (e) return e;
  CUtensorMap tmap_in[5];
  const void* ins[5] = {r, w, k, a, b};
  for (int i = 0; i < 5; ++i) {
    e = make_token_tensor_map(&tmap_in[i], ins[i], mapB, mapT, H, head_first);
    if (e) return e;
  }
  const int NT = num_chunks(Tn);
  const int tpc = keep_for_bwd ? (int)ALL_TILES : (int)FWD_TILES;
  Workspace ws = carve(workspace, B, Tn, H, tpc);
  TokLayout lay(mapT, H, head_first);
  if (phases & PHASE_PREPARE) {
    if (cuda_ok(cudaMemsetAsync(ws.flags, 0, (size_t)B * H * sizeof(int), st))) return RWKVB200_E_CUDA;
    const int smem = (int)sizeof(IntraSmem) + 1024;
    ProfScope prof("r7c_intra_fwd_kernel", st);
    const int n_ch = B * H * NT;
    int dev = 0, sms = 0;
    if (cuda_ok(cudaGetDevice(&dev)) || cuda_ok(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)))
      return RWKVB200_E_CUDA;
    const int grid = n_ch < 2 * sms ? n_ch : 2 * sms;     // persistent: two CTAs per SM
#define R7C_LAUNCH_INTRA(P, F)                                                                                     \
    do {                                                                                                           \
      if (cuda_ok(cudaFuncSetAttribute(r7c_intra_fwd_kernel<P, F>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem))) \
        return RWKVB200_E_CUDA;                                                                                    \
      r7c_intra_fwd_kernel<P, F><<<grid, 256, smem, st>>>(tmap_in[0], tmap_in[1], tmap_in[2], tmap_in[3], tmap_in[4], \
          tmap_v, ws.tiles, ws.aux, ws.flags, tpc, keep_for_bwd ? 1 : 0, sv, H, NT, n_ch, status,                 \
          debug_stamp_buffer());                                                                                   \
    } while (0)
    if (seq_start) R7C_LAUNCH_INTRA(true, false);
    else if (fused) R7C_LAUNCH_INTRA(false, true);
    else R7C_LAUNCH_INTRA(false, false);
#undef R7C_LAUNCH_INTRA
  }
  e = check_launch();
  if (e || !(phases & PHASE_SCAN)) return e;
  {
    int dev = 0, sms = 0;
    if (cuda_ok(cudaGetDevice(&dev)) || cuda_ok(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)))
      return RWKVB200_E_CUDA;
    ProfScope prof("r7c_scan_fwd_kernel", st);
    // more sequences than SMs: two CTAs per SM with two stages each; else one CTA per SM with loads further ahead
#define R7C_LAUNCH_SCAN(S, P)                                                                                      \
    do {                                                                                                           \
      const int smem = (int)sizeof(ScanSmem<S>);                                                                   \
      if (cuda_ok(cudaFuncSetAttribute(r7c_scan_fwd_kernel<S, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem))) \
        return RWKVB200_E_CUDA;                                                                                    \
      r7c_scan_fwd_kernel<S, P><<<B * H, 256, smem, st>>>(ws.tiles, ws.aux, tpc, keep_for_bwd ? ws.tiles : nullptr, \
          ws.fin, h0, n_state, tmap_o, o ? 1 : 0, ht, (bf16*)o, sv, H, NT, lay, status);                           \
    } while (0)
    if (B * H > sms) { if (seq_start) R7C_LAUNCH_SCAN(2, true); else R7C_LAUNCH_SCAN(2, false); }
    else             { if (seq_start) R7C_LAUNCH_SCAN(4, true); else R7C_LAUNCH_SCAN(4, false); }
#undef R7C_LAUNCH_SCAN
  }
  e = check_launch();
  if (e || fused) return e;      // fused producers bound |g| by e^{-1/2}: no unit can be marked
  // units whose decay left the range of the scaled operands: exact float32 recurrence over them (the
  // kernel's other CTAs leave at once)
  if (o || ht) {
    const UnitSel sel{ws.flags, seq_start, seq_len, 0};
    e = launch_rwkv7_rec_fwd(r, w, k, v, a, b, h0, n_state, o, ht, nullptr, R7_CKPT, B, Tn, H, RWKVB200_BF16,
                             head_first, st, &sel, seq_start ? T_total : 0);
  }
  return e;
}

}  // namespace rwkvb200
