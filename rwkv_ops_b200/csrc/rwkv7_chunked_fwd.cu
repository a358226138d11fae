// Chunked RWKV7 forward on tcgen05 (bf16 token tensors, fp32 state).  Equations and the
// two-kernel structure are described in rwkv7_chunked.cuh.
#include "rwkv7_chunked.cuh"
#include "rwkv7_recurrent.cuh"

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
constexpr int NROW = 68;   // padded row of a 64 x 64 fp32 array (keeps float4 alignment)

struct IntraSmem {
  unsigned char qt[TILE_BYTES], at[TILE_BYTES];     // [q~; a~]  (128-row A operand)
  unsigned char kt[TILE_BYTES], bt[TILE_BYTES];     // [k~; b~]  (128-row B operand)
  unsigned char aqk[TILE_BYTES], aak[TILE_BYTES];   // [A_qk; A_ak] (128-row A operand); aak later holds W
  unsigned char cm[TILE_BYTES];                     // C = A_qb Ainv
  unsigned char aqb[TILE_BYTES];
  unsigned char v[TILE_BYTES];                      // raw a, then v
  unsigned char ainv[TILE_BYTES];                   // later holds B2
  unsigned char y[TILE_BYTES];                      // A_ak v
  float gs[L * NROW];                               // gi - gref; before that the raw b tile, later the inverse's blocks
  float qtot[4][64];                                // sums of g over the four quarters of the chunk
  uint64_t bar_v, bar_w, bar_in, bar_b, bar_m1, bar_m2, bar_m3, bar_m4, bar_m5;
  uint32_t tmem_base;
};

// Persistent: CTAs (two per SM) walk over the chunk-heads (RowWalk, ListWalk).
// 256 threads: warp w reads TMEM lanes 32*(w&3).. and the two warps that share a lane window split
// the columns (hsel = w>>2); warps 6 and 7 invert the diagonal blocks of A_ab while the other warps mask the rest of
// MMA 1, issue MMA 2 and drain it.
// What bounds it: 17 tiles per chunk-head through memory (348 us at B 8, T 4096, 32 heads) if two CTAs per SM can
// overlap their chains of phases well enough: 503 us before the inverse went to two warps and the raw tiles were requested
// early, 467 us now.  The backward takes the difference of large sums over the tiles made here: a change of their arithmetic in
// the last bit shows in dw (a 32 x 32 substitution and reciprocals for e^{gref-gi} gave 412 us and were taken back).
template <bool PACKED, bool FUSED>
__global__ void __launch_bounds__(256, 2)
r7c_intra_fwd_kernel(const bf16* __restrict__ q, const bf16* __restrict__ w, const bf16* __restrict__ k,
                     const bf16* __restrict__ a, const bf16* __restrict__ b,
                     const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_w,
                     const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_a,
                     const __grid_constant__ CUtensorMap tmap_b,
                     const __grid_constant__ CUtensorMap tmap_v, unsigned char* __restrict__ ws_tiles,
                     float* __restrict__ ws_aux, int tiles_per_chunk,
                     int keep_for_bwd, SeqView sv, const __grid_constant__ WalkDims dims, int2* list, TokLayout lay, int* status, long long* dbg) {
#ifdef RWKVB200_DEVTOOLS
#define R7C_STAMP(n) do { if (dbg && tid == 0 && blockIdx.x == gridDim.x / 2 && it == 30) dbg[n] = clock64(); } while (0)
#else
#define R7C_STAMP(n) do {} while (0)
#endif
  extern __shared__ unsigned char smem_raw[];
  IntraSmem& sm = *reinterpret_cast<IntraSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wq = warp & 3, hsel = warp >> 2;

  if (tid == 0) {
    mbar_init(&sm.bar_v, 1); mbar_init(&sm.bar_w, 1); mbar_init(&sm.bar_in, 1); mbar_init(&sm.bar_b, 1); mbar_init(&sm.bar_m1, 1); mbar_init(&sm.bar_m2, 1); mbar_init(&sm.bar_m3, 1);
    mbar_init(&sm.bar_m4, 1); mbar_init(&sm.bar_m5, 1);
    fence_mbar_init();
  }
  if (tid == 32) {
    tma_prefetch_maps(tmap_q, tmap_w, tmap_k, tmap_a, tmap_b, tmap_v);
    if constexpr (!PACKED) {      // the first rows into L2, while the kernel before runs out
      const ChunkPos p = RowWalk{dims}.first();
      tma_prefetch_4d(&tmap_w, 0, p.c * L, p.hi, p.bi);
      tma_prefetch_4d(&tmap_q, 0, p.c * L, p.hi, p.bi);
      tma_prefetch_4d(&tmap_k, 0, p.c * L, p.hi, p.bi);
      tma_prefetch_4d(&tmap_a, 0, p.c * L, p.hi, p.bi);
      tma_prefetch_4d(&tmap_b, 0, p.c * L, p.hi, p.bi);
    }
  }
  if (warp == 0) tmem_alloc(&sm.tmem_base, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  earlier_kernels_done();
  later_kernels_may_start();
  const uint32_t tm = sm.tmem_base;

  auto coords = [&](const ChunkPos& p, int& bi, int& hi, int& t0) { bi = p.bi; hi = p.hi; t0 = p.c * L; };
  // The raw tiles of a chunk-head (rows past the end of the sequence arrive as zeros), requested most of a chunk-head
  // before they are needed: w, q, k land in the A_qk, q~, k~ tiles and a in the v tile as soon as MMA 2 has completed (the
  // copies to the workspace have left shared memory by then), b in the space of the decay factors once the diagonal
  // blocks have been inverted there.  Only v, needed last, is requested in its own chunk-head, when a has been scaled.
  auto load = [&](unsigned char* dst, const CUtensorMap* map, uint64_t* bar, const ChunkPos& p) {      // one thread
    tma_load_4d(dst, map, bar, 0, sv.first<PACKED>(p.bi) + p.c * L, p.hi, sv.row<PACKED>(p.bi));
  };
  auto load_w = [&](const ChunkPos& p) { mbar_expect_tx(&sm.bar_w, TILE_BYTES); load(sm.aqk, &tmap_w, &sm.bar_w, p); };
  auto load_qka = [&](const ChunkPos& p) {
    mbar_expect_tx(&sm.bar_in, 3 * TILE_BYTES);
    load(sm.qt, &tmap_q, &sm.bar_in, p);
    load(sm.kt, &tmap_k, &sm.bar_in, p);
    load(sm.v, &tmap_a, &sm.bar_in, p);
  };
  auto load_b = [&](const ChunkPos& p) { mbar_expect_tx(&sm.bar_b, TILE_BYTES); load(reinterpret_cast<unsigned char*>(sm.gs), &tmap_b, &sm.bar_b, p); };
  auto load_v = [&](const ChunkPos& p) { mbar_expect_tx(&sm.bar_v, TILE_BYTES); load(sm.v, &tmap_v, &sm.bar_v, p); };
  // Ask for a chunk-head's token rows to be brought into L2, ahead of the TMA loads above.
  auto prefetch_rows = [&](const ChunkPos& p) {      // one thread
    const int tt = sv.first<PACKED>(p.bi) + p.c * L, br = sv.row<PACKED>(p.bi);
    tma_prefetch_4d(&tmap_w, 0, tt, p.hi, br);
    tma_prefetch_4d(&tmap_q, 0, tt, p.hi, br);
    tma_prefetch_4d(&tmap_k, 0, tt, p.hi, br);
    tma_prefetch_4d(&tmap_a, 0, tt, p.hi, br);
    tma_prefetch_4d(&tmap_b, 0, tt, p.hi, br);
    tma_prefetch_4d(&tmap_v, 0, tt, p.hi, br);
  };
  if constexpr (PACKED) write_list(list, sv, dims, reinterpret_cast<int*>(sm.qtot), tid);
  const auto walk = [&] {
    if constexpr (PACKED) return ListWalk{dims, list}; else return RowWalk{dims};
  }();
  ChunkPos cur = walk.first();
  if (cur.ch < dims.n_ch && warp == 0 && elect_one()) { load_w(cur); load_qka(cur); load_b(cur); }
  // The two CTAs that share an SM would otherwise run their phases in lockstep and compete for the
  // same unit (shared-memory pipe during the triangular solve); start every other CTA half a
  // chunk-head late (unless it has a single one to do, or none: then the delay would be all it adds).
  if ((blockIdx.x & 1) && dims.n_ch > 2 * (int)gridDim.x) __nanosleep(6000);

  bool ok = true;
  int it = 0;
  for (ChunkPos nxt; cur.ch < dims.n_ch && ok; cur = nxt, ++it) {
    const int ch = cur.ch;
    int bi, hi, t0; coords(cur, bi, hi, t0);
    const int Tn = sv.length<PACKED>(bi);
    unsigned char* out_tiles = ws_tiles + (size_t)ch * tiles_per_chunk * TILE_BYTES;
    const uint32_t par = it & 1;
    nxt = walk.after(cur, it);
    const int next = nxt.ch;

    R7C_STAMP(0);
    if (next < dims.n_ch && warp == 1 && elect_one()) prefetch_rows(nxt);
    // ---- phase A: decay prefix sums (in units of log 2), thread = (channel, quarter of the chunk), straight from the
    // raw w tile.
    ok = mbar_wait(&sm.bar_b, par, status, 208) && ok;
    uint4 rb[2];      // this thread's 2 x 16 bytes (8 channels of one token) of the raw b tile, which lies where the factors will
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int e = tid + 256 * n;
      rb[n] = *reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned char*>(sm.gs) + tile_chunk_off(e >> 3, e & 7));
    }
    ok = mbar_wait(&sm.bar_w, par, status, 206) && ok;
    {
      const int c = tid & 63, quarter = tid >> 6;
      float gi[16];
      float run = 0.f;
      const int n_rows = Tn - t0 - 16 * quarter;      // rows of this quarter inside the sequence
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        unsigned short* raw = reinterpret_cast<unsigned short*>(sm.aqk + tile_off(16 * quarter + j, c));
        float w = __uint_as_float((uint32_t)*raw << 16);
        if constexpr (FUSED) {      // the tile holds p: w = -e^{-1/2} sigmoid(p), as bfloat16, goes back for the scaling
          w = round_bf16(W_SCALE * sigmoidf_(w));
          *raw = (unsigned short)(__float_as_uint(w) >> 16);
        }
        run += j < n_rows ? __fmul_rn(-LOG2E, ex2(LOG2E * w)) : 0.f;      // (rounded as in the scaling below)
        gi[j] = run;
      }
      sm.qtot[quarter][c] = run;
      __syncthreads();
      R7C_STAMP(1);
      // gi - gref: the prefix inside the half; the reference point is the end of the first half
      const float add = quarter == 0 ? -(run + sm.qtot[1][c]) : quarter == 1 ? -run : quarter == 3 ? sm.qtot[2][c] : 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) sm.gs[(16 * quarter + j) * NROW + c] = gi[j] + add;
      if (quarter == 0) {
        const float tot0 = -add, tot1 = sm.qtot[2][c] + sm.qtot[3][c];
        ws_aux[(size_t)ch * AUX_FLOATS + c] = ex2(fmaxf(tot0, EXP2_FLOOR));          // e^{gref}
        // a half-chunk decay sum beyond the limit: the unit is recomputed by the float32 recurrence.  The mark is the
        // factor's sign; the scan, which reads every factor of its unit anyway, gathers it into Workspace::flags.
        const bool mark = fminf(tot0, tot1) < -DECAY_LIMIT * LOG2E || Tn < SHORT_SEQ;
        ws_aux[(size_t)ch * AUX_FLOATS + 64 + c] = copysignf(ex2(fmaxf(tot1, EXP2_FLOOR)), mark ? -1.f : 1.f);   // e^{glast-gref}
      }
    }
    __syncthreads();
    {
      // the raw q, k, a, b: each thread scales its own 2 x 16 bytes (the previous chunk-head's W, U,
      // A_qb copies may still be reading their tiles: those are rewritten only after MMA 1)
      uint4 rq[2], rk[2], ra[2];
      ok = mbar_wait(&sm.bar_in, par, status, 207) && ok;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int e = tid + 256 * n;
        const uint32_t off = tile_chunk_off(e >> 3, e & 7);
        rq[n] = *reinterpret_cast<const uint4*>(sm.qt + off);
        rk[n] = *reinterpret_cast<const uint4*>(sm.kt + off);
        ra[n] = *reinterpret_cast<const uint4*>(sm.v + off);
        if (PACKED && t0 + (e >> 3) >= Tn) {      // in a packed batch these rows belong to the next sequence
          rq[n] = make_uint4(0u, 0u, 0u, 0u); rk[n] = rq[n]; ra[n] = rq[n]; rb[n] = rq[n];
        }
        if constexpr (FUSED) {      // the a / b tiles hold u and q: a = -kk, b = kk sigmoid(q), kk = u / |u|
          const uint32_t uu[4] = {ra[n].x, ra[n].y, ra[n].z, ra[n].w}, qq[4] = {rb[n].x, rb[n].y, rb[n].z, rb[n].w};
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
          ra[n] = make_uint4(na[0], na[1], na[2], na[3]);
          rb[n] = make_uint4(nb[0], nb[1], nb[2], nb[3]);
        }
      }
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int e = tid + 256 * n, row = e >> 3, cc = e & 7;
        float gl[8];      // gi - gref
        *reinterpret_cast<float4*>(gl) = *reinterpret_cast<const float4*>(&sm.gs[row * NROW + 8 * cc]);
        *reinterpret_cast<float4*>(gl + 4) = *reinterpret_cast<const float4*>(&sm.gs[row * NROW + 8 * cc + 4]);
        const uint4 rw = *reinterpret_cast<const uint4*>(sm.aqk + tile_chunk_off(row, cc));
        const uint32_t uw[4] = {rw.x, rw.y, rw.z, rw.w};
        const uint32_t uq[4] = {rq[n].x, rq[n].y, rq[n].z, rq[n].w};
        const uint32_t uk[4] = {rk[n].x, rk[n].y, rk[n].z, rk[n].w};
        const uint32_t ua[4] = {ra[n].x, ra[n].y, ra[n].z, ra[n].w};
        const uint32_t ub[4] = {rb[n].x, rb[n].y, rb[n].z, rb[n].w};
        uint32_t oq[4], ok_[4], oa[4], ob[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          float eq[2], ek[2], ea[2];
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            const float d1 = gl[2 * m + hh];
            const float w = hh ? bf16_hi(uw[m]) : bf16_lo(uw[m]);
            const float g = t0 + row < Tn ? __fmul_rn(-LOG2E, ex2(LOG2E * w)) : 0.f;
            eq[hh] = ex2(d1); ek[hh] = ex2(-d1); ea[hh] = ex2(d1 - g);
          }
          oq[m] = pack_bf16(bf16_lo(uq[m]) * eq[0], bf16_hi(uq[m]) * eq[1]);
          ok_[m] = pack_bf16(bf16_lo(uk[m]) * ek[0], bf16_hi(uk[m]) * ek[1]);
          oa[m] = pack_bf16(bf16_lo(ua[m]) * ea[0], bf16_hi(ua[m]) * ea[1]);
          ob[m] = pack_bf16(bf16_lo(ub[m]) * ek[0], bf16_hi(ub[m]) * ek[1]);
        }
        const uint32_t off = tile_chunk_off(row, cc);
        *reinterpret_cast<uint4*>(sm.qt + off) = make_uint4(oq[0], oq[1], oq[2], oq[3]);
        *reinterpret_cast<uint4*>(sm.kt + off) = make_uint4(ok_[0], ok_[1], ok_[2], ok_[3]);
        *reinterpret_cast<uint4*>(sm.at + off) = make_uint4(oa[0], oa[1], oa[2], oa[3]);
        *reinterpret_cast<uint4*>(sm.bt + off) = make_uint4(ob[0], ob[1], ob[2], ob[3]);
      }
    }
    fence_async_smem();
    __syncthreads();

    R7C_STAMP(2);
    // ---- MMA 1: [q~; a~] [k~; b~]^T  ->  TMEM columns 0..127, row r on lane r
    if (warp == 0 && elect_one()) {
      bulk_wait_read();      // the previous W, U copies are done: the epilogue below rewrites their tiles
      tc_fence_after();
      umma_tile<128, 128, 0, 0>(tm, smem_u32(sm.qt), smem_u32(sm.kt), false);
      umma_commit(&sm.bar_m1);
      load_v(cur);           // the raw a has been scaled
    }
    ok = mbar_wait(&sm.bar_m1, par, status, 201) && ok;
    tc_fence_after();
    R7C_STAMP(3);
    if (warp == 0 && elect_one() && ok) {      // MMA 1 was the last reader of q~, k~, b~ in shared memory: copy them out now
      bulk_store(out_tiles + S_QT * TILE_BYTES, sm.qt, TILE_BYTES);
      bulk_store(out_tiles + S_KT * TILE_BYTES, sm.kt, TILE_BYTES);
      bulk_store(out_tiles + S_BT * TILE_BYTES, sm.bt, TILE_BYTES);
      bulk_commit();
    }
    // Rows r < 64 are q~'s, the others a~'s; the warp's 32 rows are i = 32*ihalf + lane, so which side of the diagonal
    // a block of 32 columns lies on is the same for the whole warp: left of the diagonal block every element is kept,
    // right of it every element is zero (TMEM is not read), and only the diagonal block takes a per-element choice.
    const int ihalf = wq & 1;
    if (warp < 6) {      // A_qk (warps 0, 1), A_ak (2, 3), A_qb (4, 5)
      if (ok) {
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
          tile_store_row32(dst, 32 * ihalf + lane, 32 * pp, x);
        }
      }
      fence_async_smem();
      tc_fence_before();
      asm volatile("bar.sync 1, 192;" ::: "memory");

      R7C_STAMP(4);
      // ---- MMA 2: Y = A_ak v  ->  TMEM columns 128..191 (lower lane halves)
      if (warp == 0 && elect_one()) {
        ok = mbar_wait(&sm.bar_v, par, status, 202) && ok;
        tc_fence_after();
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 0, 128), smem_u32(sm.aak), smem_u32(sm.v), false);
        umma_commit(&sm.bar_m2);
        bulk_store(out_tiles + S_AQK * TILE_BYTES, sm.aqk, TILE_BYTES);
        if (keep_for_bwd) {   // A_ak, a~ are operands of the backward
          bulk_store(out_tiles + S_AAK * TILE_BYTES, sm.aak, TILE_BYTES);
          bulk_store(out_tiles + S_AT * TILE_BYTES, sm.at, TILE_BYTES);
        }
        bulk_commit();
      }
      if (warp == 3 && ok) {      // Q: N_BA in rows 32..63 (its other rows and columns are not used)
        uint32_t rr[32];
        tmem_ld32(tmem_addr(tm, 32 * wq, 64), rr);
        tmem_ld_wait();
        float x[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
        tile_store_row32(sm.cm, 32 + lane, 0, x);
      }
      if (warp == 1) {            // the upper right block of X
        const float x[32] = {};
        tile_store_row32(sm.ainv, lane, 32, x);
      }
      ok = mbar_wait(&sm.bar_m2, par, status, 203) && ok;
      tc_fence_after();
      if (ok) {      // Y rows; warps 2, 3 take both column halves of theirs
#pragma unroll
        for (int pp = 0; pp < 2; ++pp) {
          if (pp != hsel && wq < 2) continue;
          uint32_t rr[32];
          tmem_ld32(tmem_addr(tm, 32 * wq, 128 + 32 * pp), rr);
          tmem_ld_wait();
          if (lane < 16) {        // an M = 64 accumulator lives on the lower 16 lanes of every warp's window
            float x[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
            tile_store_row32(sm.y, 16 * wq + lane, 32 * pp, x);
          }
        }
      }
      if (warp == 0 && elect_one()) {
        bulk_wait_read();                  // q~, k~, b~, A_qk (and the tiles kept for the backward) have left shared memory
        if (next < dims.n_ch) { load_w(nxt); load_qka(nxt); }      // nothing reads A_qk, q~, k~, v any more
      }
    } else if (ok) {     // warps 6, 7: the diagonal 32 x 32 blocks of A_ab, inverted (fp32); warp 7 also N_BA
      // Ainv = X = (I - N)^-1, N = stril(A_ab); with A = rows 0..31, B = rows 32..63 its blocks are X_A = (I - N_AA)^-1,
      // X_B = (I - N_BB)^-1 and X_BA = X_B N_BA X_A.  A 32 x 32 block is inverted by its 16 x 16 blocks: D_0, D_1 by
      // substitution, one column per lane, side by side, then X_10 = D_1 (N_10 D_0), half a column per lane.
      float* nd = sm.gs + 1024 * ihalf;                 // this warp's block transposed: nd[32 j + i] = N[i][j]; later D_1
      uint32_t rr[32];
      tmem_ld32(tmem_addr(tm, 32 * wq, 64 + 32 * ihalf), rr);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j) nd[32 * j + lane] = __uint_as_float(rr[j]);      // (at or above the diagonal: never used)
      __syncwarp();
      const int bl = lane >> 4, cl = lane & 15;
      // Once x[j] is known its products with column j of N go into all later rows (of the first, then of the second eight:
      // registers), two rows per instruction and independent of one another; a row collects them in four partial sums, by
      // j mod 4.  The next column is on its way.
      float xb[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) xb[i] = i == cl ? 1.f : 0.f;
#pragma unroll
      for (int h8 = 0; h8 < 16; h8 += 8) {
        const float* nb = nd + (32 + 1) * 16 * bl + h8;      // rows h8 .. h8 + 7 of column j of the block: nb + 32 j
        float p[4][8];
        float4 nc[2][2];
        nc[0][0] = *reinterpret_cast<const float4*>(nb);
        nc[0][1] = *reinterpret_cast<const float4*>(nb + 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) p[0][i] = p[1][i] = p[2][i] = p[3][i] = 0.f;
#pragma unroll
        for (int j = 0; j < h8 + 7; ++j) {
          if (j + 1 < h8 + 7) {
            nc[(j + 1) & 1][0] = *reinterpret_cast<const float4*>(nb + 32 * (j + 1));
            nc[(j + 1) & 1][1] = *reinterpret_cast<const float4*>(nb + 32 * (j + 1) + 4);
          }
          const float* n = reinterpret_cast<const float*>(nc[j & 1]);
          float* q = p[j & 3];
          const int first = j + 1 > h8 ? j + 1 - h8 : 0;      // rows after j
          if (first & 1) q[first] = __fmaf_rn(n[first], xb[j], q[first]);
#pragma unroll
          for (int i = (first + 1) & ~1; i < 8; i += 2) fma2(q[i], q[i + 1], n[i], n[i + 1], xb[j], xb[j], q[i], q[i + 1]);
          if (j + 1 >= h8) xb[j + 1] += (p[0][j + 1 - h8] + p[1][j + 1 - h8]) + (p[2][j + 1 - h8] + p[3][j + 1 - h8]);
        }
      }
      // P = N_10 D_0 and X_10 = D_1 P, rows 8 bl .. 8 bl + 7 of column cl; in groups of four terms
      float col[16], acc[8];
      auto product = [&](const float* m, int ld) {      // acc[q] = sum_k m[ld k + q] col[k]
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          float t[8];
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            float n[8];
            *reinterpret_cast<float4*>(n) = *reinterpret_cast<const float4*>(m + ld * (4 * jj + kk));
            *reinterpret_cast<float4*>(n + 4) = *reinterpret_cast<const float4*>(m + ld * (4 * jj + kk) + 4);
#pragma unroll
            for (int q = 0; q < 8; ++q) t[q] = kk ? __fmaf_rn(n[q], col[4 * jj + kk], t[q]) : __fmul_rn(n[q], col[4 * jj]);
          }
#pragma unroll
          for (int q = 0; q < 8; ++q) acc[q] = jj ? __fadd_rn(acc[q], t[q]) : t[q];
        }
      };
#pragma unroll
      for (int kk = 0; kk < 16; ++kk) col[kk] = __shfl_sync(0xffffffffu, xb[kk], cl);      // D_0[:, cl]
      product(nd + 16 + 8 * bl, 32);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float other = __shfl_xor_sync(0xffffffffu, acc[q], 16);
        col[q] = bl ? other : acc[q];
        col[8 + q] = bl ? acc[q] : other;
      }
      __syncwarp();
      if (bl) {
#pragma unroll
        for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(&nd[16 * cl + i]) = make_float4(xb[i], xb[i + 1], xb[i + 2], xb[i + 3]);
      }
      __syncwarp();
      product(nd + 8 * bl, 16);
      auto put = [&](int row, int c, float f) {
        *reinterpret_cast<bf16*>(sm.ainv + tile_off(32 * ihalf + row, 32 * ihalf + c)) = __float2bfloat16_rn(f);
      };
#pragma unroll
      for (int i = 0; i < 16; ++i) put(16 * bl + i, 16 * bl + cl, xb[i]);
#pragma unroll
      for (int q = 0; q < 8; ++q) put(16 + 8 * bl + q, cl, acc[q]);
      if (lane < 16) {      // the upper right 16 x 16 block
        *reinterpret_cast<uint4*>(sm.ainv + tile_chunk_off(32 * ihalf + lane, 4 * ihalf + 2)) = make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(sm.ainv + tile_chunk_off(32 * ihalf + lane, 4 * ihalf + 3)) = make_uint4(0u, 0u, 0u, 0u);
      }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);

    R7C_STAMP(10);
    // ---- X_BA on the tensor cores: T = N_BA X_A, then X_B T, with bf16 operands (N_BA is a small correction: rounding
    // it, X_A, X_B and T to bf16 changes the rounded inverse by less than the rounding of the inverse itself).  Only rows
    // 32..63 of both products are used, and only half of the 64 contraction elements are not zero.
    if (warp == 0 && elect_one() && ok) {
      tc_fence_after();
      umma_tile<64, 64, 0, 1, 2>(tmem_addr(tm, 0, 128), smem_u32(sm.cm), smem_u32(sm.ainv), false);
      umma_commit(&sm.bar_m4);
      if (next < dims.n_ch) load_b(nxt);      // the diagonal blocks have been read
    }
    ok = ok && mbar_wait(&sm.bar_m4, par, status, 209);
    tc_fence_after();
    R7C_STAMP(11);
    if (ok && wq >= 2) {      // T's rows 32..63 (the A_ak tile is free: its copy has left it, MMA 2 has read it)
      uint32_t rr[32];
      tmem_ld32(tmem_addr(tm, 32 * wq, 128 + 32 * hsel), rr);
      tmem_ld_wait();
      if (lane < 16) {
        float x[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
        tile_store_row32(sm.aak, 16 * wq + lane, 32 * hsel, x);
      }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    R7C_STAMP(12);
    if (warp == 0 && elect_one() && ok) {
      tc_fence_after();
      // contraction elements 32..63: 64 bytes into the rows of A, 32 rows into B
      umma_tile<64, 64, 0, 1, 2>(tmem_addr(tm, 0, 128), smem_u32(sm.ainv) + 64, smem_u32(sm.aak) + 32 * 128, false);
      umma_commit(&sm.bar_m5);
    }
    ok = ok && mbar_wait(&sm.bar_m5, par, status, 210);
    tc_fence_after();
    if (ok && hsel == 0 && wq >= 2) {      // rows 32..63, columns 0..31: the BA quadrant of Ainv
      uint32_t rr[32];
      tmem_ld32(tmem_addr(tm, 32 * wq, 128), rr);
      tmem_ld_wait();
      if (lane < 16) {
        float x[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
        tile_store_row32(sm.ainv, 16 * wq + lane, 0, x);
      }
    }
    R7C_STAMP(13);
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);

    R7C_STAMP(6);
    // ---- MMA 3: W = Ainv a~ (lower lane halves), U = Ainv Y (upper lane halves) -> TMEM columns 0..63; for the
    // backward B2 = Ainv^T b~ and C = A_qb Ainv -> columns 64..127
    if (warp == 0 && elect_one()) {
      tc_fence_after();
      umma_tile<64, 64, 0, 1>(tmem_addr(tm, 0, 0), smem_u32(sm.ainv), smem_u32(sm.at), false);
      umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 0), smem_u32(sm.ainv), smem_u32(sm.y), false);
      if (keep_for_bwd) {
        umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, 64), smem_u32(sm.ainv), smem_u32(sm.bt), false);
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 64), smem_u32(sm.aqb), smem_u32(sm.ainv), false);
      }
      umma_commit(&sm.bar_m3);
      bulk_store(out_tiles + S_AQB * TILE_BYTES, sm.aqb, TILE_BYTES);
      bulk_commit();
    }
    ok = mbar_wait(&sm.bar_m3, par, status, 204) && ok;
    tc_fence_after();
    R7C_STAMP(7);

    {
      // W -> the A_ak tile (free since MMA 2), U -> the Y tile, B2 -> the Ainv tile (free: MMA 3 has completed)
      const int i = 16 * wq + (lane & 15);
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        if (part && !keep_for_bwd) break;
        unsigned char* dst = part ? (lane < 16 ? sm.ainv : sm.cm) : (lane < 16 ? sm.aak : sm.y);
        uint32_t rr[32];
        tmem_ld32(tmem_addr(tm, 32 * wq, 64 * part + 32 * hsel), rr);
        tmem_ld_wait();
        float x[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
        tile_store_row32(dst, i, 32 * hsel, x);
      }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    R7C_STAMP(8);
    if (warp == 0 && elect_one() && ok) {
      bulk_store(out_tiles + S_W * TILE_BYTES, sm.aak, TILE_BYTES);
      bulk_store(out_tiles + S_U * TILE_BYTES, sm.y, TILE_BYTES);
      if (keep_for_bwd) {
        bulk_store(out_tiles + S_C * TILE_BYTES, sm.cm, TILE_BYTES);
        bulk_store(out_tiles + S_B2 * TILE_BYTES, sm.ainv, TILE_BYTES);
      }
      bulk_commit();
    }
    R7C_STAMP(9);
  }
  if (warp == 0 && elect_one()) bulk_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 256);
#undef R7C_STAMP
}

// ---------------------------------------------------------------------------------------------
// scan kernel: grid = B*H, 256 threads, chunks in order.  Warp w reads TMEM lanes 32*(w&3)..; the two warps that share a
// lane window take 32 of the 64 columns each (hsel = w>>2).  Lanes 0-15 of a warp own state rows, lanes 16-31 token rows.
// ---------------------------------------------------------------------------------------------
// For more sequences than SMs: two CTAs (two sequences) share an SM, and memory bounds it (eight tiles in, four out per
// chunk).  The products of a chunk accumulate onto its state (fp32, in TMEM); the output rows of a chunk are read out with
// sa of the next one; copies are waited for a phase after they were issued.
// Operand tiles come in two groups, each requested again once the MMAs that read it have completed.  U, which is only
// added row by row, does not enter shared memory: every thread fetches its row into registers at the top of a chunk.
struct ScanGroup1 {         // free once W h~0 and q~ h~0 have been computed
  unsigned char kt[TILE_BYTES], aqk[TILE_BYTES], w[TILE_BYTES];   // adjacent slots
  unsigned char v[TILE_BYTES], qt[TILE_BYTES];
};
struct ScanGroup2 {         // free at the end of the chunk
  unsigned char bt[TILE_BYTES], aqb[TILE_BYTES];  // adjacent slots
};
struct ScanSmem {
  ScanGroup1 g1;
  ScanGroup2 g2;
  unsigned char ht[2][TILE_BYTES];          // h~0 as bf16, [k][v]
  unsigned char sa[TILE_BYTES];             // sa as bf16, [token][v]
  unsigned char xt[TILE_BYTES];             // X = h~0 + k~^T v + b~^T sa as bf16 (kept for the backward)
  unsigned char ot[TILE_BYTES];             // output rows of a chunk, staged for a TMA store
  uint64_t bar_g1, bar_g2, bar_a, bar_c, bar_o;
  uint32_t tmem_base;
};

// A marked unit again, by the exact recurrence: 256 threads, half of them holding two rows each, in place of what the chunks
// gave (inside the scan kernels, because a launch of its own over all units costs every call 2 us of device time and as much
// on the host).  Out of line: it would only take registers from the loop over the chunks.
__device__ __noinline__ void exact_unit(r7rec::FwdArgs<bf16> args, unsigned char* smem, int tid, int unit, int hi, int brow,
                                           int tb, int Tn, const float* h0, int n_state, float* ht, const TokLayout& lay) {
  args.base = brow * lay.sb + hi * lay.sh + tb * lay.st;
  args.Tn = Tn;
  args.S0 = n_state > 0 ? h0 + (size_t)(n_state == 1 ? hi : unit) * 4096 : nullptr;
  args.ht = ht ? ht + (size_t)unit * 4096 : nullptr;
  typedef r7rec::FwdSmem<64, 64, 16> Smem;
  static_assert(sizeof(Smem) <= sizeof(ScanSmem), "the recurrence runs in the scan's shared memory");
  r7rec::fwd_rows<bf16, 64, 64, 2, 16, 256>(args, *reinterpret_cast<Smem*>(smem), 0, tid);
}

template <bool PACKED, bool SORTED>
__global__ void __launch_bounds__(256, 2)
r7c_scan_fwd_kernel(const __grid_constant__ CUtensorMap tmap_v, const unsigned char* __restrict__ ws_tiles,
                    const float* __restrict__ ws_aux, int* __restrict__ ws_flags, int tiles_per_chunk,
                    unsigned char* __restrict__ bwd_tiles,
                    const float* __restrict__ h0, int n_state, const __grid_constant__ CUtensorMap tmap_o,
                    int write_o, float* __restrict__ ht, bf16* __restrict__ o_rows, SeqView sv, int H, int NT_slots,
                    TokLayout lay, r7rec::FwdArgs<bf16> exact, int* status, long long* dbg) {
#ifdef RWKVB200_DEVTOOLS
#define R7C_STAMP(n) do { if (dbg && tid == 0 && blockIdx.x == gridDim.x / 2 && c == 2) dbg[n] = clock64(); } while (0)
#else
#define R7C_STAMP(n) do {} while (0)
#endif
  extern __shared__ unsigned char smem_raw[];
  ScanSmem& sm = *reinterpret_cast<ScanSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wq = warp & 3, hsel = warp >> 2, c0 = 32 * hsel;
  const int row = 16 * wq + (lane & 15);     // state row k (lanes 0-15) or token row i (lanes 16-31)
  const bool state_lane = lane < 16;
  // Single-thread jobs: warp 0 issues the MMAs, ld_warp requests operand tiles, st_warp copies sa, h~0 and X out for the
  // backward, out_warp the output rows.  Bulk-copy groups belong to the thread that committed them, so each storing
  // thread waits for its own copies.
  constexpr int ld_warp = 1, st_warp = 2, out_warp = 3;

  // A packed batch may have many short sequences, whose blocks come in many rounds: where theirs lies is asked for before the TMEM is
  // (4000 of up to 64 tokens, 16 heads: 1404 -> 1357 us).
  if constexpr (PACKED) earlier_kernels_done();
  int unit = blockIdx.x;
  if constexpr (SORTED) unit = sorted_scan_unit(sv, H, reinterpret_cast<SortedSeqs*>(sm.ot), tid);
  const int bi = unit / H, hi = unit % H;
  const int Tn = sv.length<PACKED>(bi), tb = sv.first<PACKED>(bi), brow = sv.row<PACKED>(bi);
  const int NT = (Tn + L - 1) / L;           // chunks of this sequence (at least one)
  if (tid == 0) {
    mbar_init(&sm.bar_g1, 1); mbar_init(&sm.bar_g2, 1);
    mbar_init(&sm.bar_a, 1); mbar_init(&sm.bar_c, 1); mbar_init(&sm.bar_o, 1);
    fence_mbar_init();
  }
  if (tid == 32) tma_prefetch_maps(tmap_v, tmap_o);
  if (warp == 0) tmem_alloc(&sm.tmem_base, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if constexpr (!PACKED) earlier_kernels_done();
  later_kernels_may_start();
  const size_t ch0 = (size_t)unit * NT_slots;
  const uint32_t tm = sm.tmem_base;
  // TMEM: columns 0..63 lower lane halves = W h~0; columns 64 + 64 p .., p = parity of the chunk: lower halves
  // k~^T v + b~^T sa, upper halves the output rows
  const uint32_t tm_sa = tmem_addr(tm, 32 * wq, c0);

  auto issue_g1 = [&](int c) {      // one thread
    const unsigned char* tiles = ws_tiles + (ch0 + c) * (size_t)tiles_per_chunk * TILE_BYTES;
    mbar_expect_tx(&sm.bar_g1, 5 * TILE_BYTES);
    bulk_load(sm.g1.kt, tiles + S_KT * TILE_BYTES, 3 * TILE_BYTES, &sm.bar_g1);
    bulk_load(sm.g1.qt, tiles + S_QT * TILE_BYTES, TILE_BYTES, &sm.bar_g1);
    tma_load_4d(sm.g1.v, &tmap_v, &sm.bar_g1, 0, tb + c * L, hi, brow);
  };
  auto issue_g2 = [&](int c) {      // one thread
    const unsigned char* tiles = ws_tiles + (ch0 + c) * (size_t)tiles_per_chunk * TILE_BYTES;
    mbar_expect_tx(&sm.bar_g2, 2 * TILE_BYTES);
    bulk_load(sm.g2.bt, tiles + S_BT * TILE_BYTES, 2 * TILE_BYTES, &sm.bar_g2);
  };
  if (warp == ld_warp && elect_one()) { issue_g1(0); issue_g2(0); }

  // ---- initial state: h~0 = e^{gref(chunk 0)} h0, fp32 in the registers of the state lanes, bf16 in the tile
  float h[32];
#pragma unroll
  for (int vv = 0; vv < 32; ++vv) h[vv] = 0.f;
  if (state_lane) {
    const float e0 = ws_aux[ch0 * AUX_FLOATS + row];
    if (n_state > 0) {
      const float* S = h0 + (size_t)(n_state == 1 ? hi : unit) * 4096;   // S[v][k], h[k][v] = S[v][k]
#pragma unroll
      for (int vv = 0; vv < 32; ++vv) h[vv] = e0 * S[(c0 + vv) * 64 + row];
    }
    tile_store_row32(sm.ht[0], row, c0, h);
  }
  bool ok = true;
  {
    uint32_t rh[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) rh[j] = __float_as_uint(h[j]);
    tmem_st32(tmem_addr(tm, 32 * wq, 64 + c0), rh);
    tmem_st_wait();
  }
  fence_async_smem();
  tc_fence_before();
  ok = __syncthreads_and(ok);

  int marked = 0;       // a chunk's decay left the range of the scaled operands (the sign of its factors)
  uint4 xp[4];          // X of the previous chunk, packed (state lanes)
  auto store_x = [&]() {
#pragma unroll
    for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(sm.xt + tile_chunk_off(row, 4 * hsel + q)) = xp[q];
  };
  for (int c = 0; c < NT && ok; ++c) {
    const int p = c & 1;
    R7C_STAMP(48);
    // (a) SA = W h~0, and the products that do not need sa: k~^T v (lower lane halves), A_qk v + q~ h~0 (upper)
    const uint32_t acc = 64 + 64 * p;
    if (warp == 0 && elect_one()) {
      ok = mbar_wait(&sm.bar_g1, c & 1, status, 211);
      if (ok) {
        tc_fence_after();
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 0, 0), smem_u32(sm.g1.w), smem_u32(sm.ht[p]), false);
        umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, acc), smem_u32(sm.g1.kt), smem_u32(sm.g1.v), true);      // onto h~0
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, acc), smem_u32(sm.g1.aqk), smem_u32(sm.g1.v), false);
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, acc), smem_u32(sm.g1.qt), smem_u32(sm.ht[p]), true);
        umma_commit(&sm.bar_a);
      }
    }
    if (bwd_tiles && warp == st_warp && elect_one()) {
      bulk_store(bwd_tiles + ((ch0 + c) * (size_t)tiles_per_chunk + S_H0) * TILE_BYTES, sm.ht[p], TILE_BYTES);
      bulk_commit();
    }
    // this thread's row of U (state lanes), and the decay factors needed at the end of this chunk
    // (applied one after the other: their product can underflow float32 where neither factor does)
    uint4 addrow[4];
    float scale = 1.f, scale_next = 1.f;
    if (state_lane) {
      const unsigned char* tile = ws_tiles + ((ch0 + c) * (size_t)tiles_per_chunk + S_U) * TILE_BYTES;
#pragma unroll
      for (int q = 0; q < 4; ++q) addrow[q] = __ldg(reinterpret_cast<const uint4*>(tile + tile_chunk_off(row, 4 * hsel + q)));
      if (c + 1 < NT && hsel == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(tile + (size_t)tiles_per_chunk * TILE_BYTES + row * 128));
      scale = ws_aux[(ch0 + c) * AUX_FLOATS + 64 + row];                       // e^{glast-gref} of this chunk
      if (c + 1 < NT) scale_next = ws_aux[(ch0 + c + 1) * AUX_FLOATS + row];    // e^{gref} of the next chunk
      if (bwd_tiles && c > 0) store_x();
    }
    ok = ok && mbar_wait(&sm.bar_a, c & 1, status, 212);
    tc_fence_after();
    R7C_STAMP(50);
    // (b) sa = W h~0 + U (state lanes); the output rows of the previous chunk (token lanes)
    if (ok) {
      unsigned char* dst = state_lane ? sm.sa : sm.ot;
      const bool act = state_lane || (c > 0 && write_o);
      const uint32_t tm_o = tmem_addr(tm, 32 * wq, 64 + 64 * (p ^ 1) + c0);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t r[16], ro[16];
        tmem_ld16(tm_sa + 16 * half, r);
        tmem_ld16(tm_o + 16 * half, ro);
        tmem_ld_wait();
        float x[16];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint4 u = addrow[2 * half + q];
          const uint32_t uu[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            const int j = 8 * q + 2 * m;
            x[j] = state_lane ? __uint_as_float(r[j]) + bf16_lo(uu[m]) : __uint_as_float(ro[j]);
            x[j + 1] = state_lane ? __uint_as_float(r[j + 1]) + bf16_hi(uu[m]) : __uint_as_float(ro[j + 1]);
          }
        }
        if (act) {
#pragma unroll
          for (int q = 0; q < 2; ++q)
            *reinterpret_cast<uint4*>(dst + tile_chunk_off(row, 4 * hsel + 2 * half + q)) =
                make_uint4(pack_bf16(x[8 * q], x[8 * q + 1]), pack_bf16(x[8 * q + 2], x[8 * q + 3]),
                           pack_bf16(x[8 * q + 4], x[8 * q + 5]), pack_bf16(x[8 * q + 6], x[8 * q + 7]));
        }
      }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    R7C_STAMP(51);
    // (c) H += b~^T sa, then the rest of the output rows, A_qb sa
    if (warp == 0 && elect_one() && ok) {
      ok = mbar_wait(&sm.bar_g2, c & 1, status, 214);
      if (ok) {
        tc_fence_after();
        umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, acc), smem_u32(sm.g2.bt), smem_u32(sm.sa), true);
        umma_commit(&sm.bar_c);
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, acc), smem_u32(sm.g2.aqb), smem_u32(sm.sa), true);
        umma_commit(&sm.bar_o);
      }
    }
    if (warp == ld_warp && elect_one() && ok && c + 1 < NT) issue_g1(c + 1);
    if (bwd_tiles && warp == st_warp && elect_one() && ok) {   // the backward needs sa, h~0 and X of every chunk
      unsigned char* tiles = bwd_tiles + (ch0 + c) * (size_t)tiles_per_chunk * TILE_BYTES;
      bulk_store(tiles + S_SA * TILE_BYTES, sm.sa, TILE_BYTES);
      if (c > 0) bulk_store(tiles - ((size_t)tiles_per_chunk - S_X) * TILE_BYTES, sm.xt, TILE_BYTES);
      bulk_commit();
    }
    if (write_o && c > 0 && warp == out_warp && elect_one() && ok) {      // a chunk that is not the last one is whole
      tma_store_4d(&tmap_o, sm.ot, 0, tb + (c - 1) * L, hi, brow);
      bulk_commit();
    }
    R7C_STAMP(52);
    ok = ok && mbar_wait(&sm.bar_c, c & 1, status, 213);
    tc_fence_after();
    R7C_STAMP(53);
    // (d) X and the next h~0
    if (ok) {
      const bool last = c + 1 == NT;
      uint32_t r[32];
      tmem_ld32(tmem_addr(tm, 32 * wq, 64 + 64 * p + c0), r);
      tmem_ld_wait();
      if (state_lane) {
#pragma unroll
        for (int j = 0; j < 32; ++j) h[j] = __uint_as_float(r[j]);
        if (bwd_tiles) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            xp[q] = make_uint4(pack_bf16(h[8 * q], h[8 * q + 1]), pack_bf16(h[8 * q + 2], h[8 * q + 3]),
                               pack_bf16(h[8 * q + 4], h[8 * q + 5]), pack_bf16(h[8 * q + 6], h[8 * q + 7]));
        }
        marked |= scale < 0.f;
        const float sc = fabsf(scale);
#pragma unroll
        for (int j = 0; j < 32; ++j) { h[j] = (h[j] * sc) * scale_next; r[j] = __float_as_uint(h[j]); }
        if (!last) tile_store_row32(sm.ht[p ^ 1], row, c0, h);
      }
      tmem_st32(tmem_addr(tm, 32 * wq, 64 + 64 * (p ^ 1) + c0), r);      // (the upper lane halves there have been read)
      tmem_st_wait();
    }
    // the copies out of sa, h~0, X and of the output rows have left their tiles: the next chunk rewrites them
    if ((warp == st_warp || warp == out_warp) && elect_one()) bulk_wait_read();
    if (warp == ld_warp && elect_one() && ok && c + 1 < NT) {      // group 2 has been read
      ok = mbar_wait(&sm.bar_o, c & 1, status, 216);
      if (ok) issue_g2(c + 1);
    }
    R7C_STAMP(54);
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    R7C_STAMP(55);
  }
#undef R7C_STAMP
  // ---- what the last chunk still holds: its output rows and X, and the final state
  ok = ok && mbar_wait(&sm.bar_o, (NT - 1) & 1, status, 217);
  tc_fence_after();
  if (ok) {
    uint32_t r[32];
    tmem_ld32(tmem_addr(tm, 32 * wq, 64 + 64 * ((NT - 1) & 1) + c0), r);
    tmem_ld_wait();
    if (state_lane) {
      if (bwd_tiles) store_x();
      if (ht) {
        float* S = ht + (size_t)unit * 4096;
#pragma unroll
        for (int j = 0; j < 32; ++j) S[(c0 + j) * 64 + row] = h[j];
      }
    } else if (write_o) {
      float x[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(r[j]);
      tile_store_row32(sm.ot, row, c0, x);
    }
  }
  fence_async_smem();
  tc_fence_before();
  ok = __syncthreads_and(ok);
  if (ok) {
    const int t0 = (NT - 1) * L;
    if (bwd_tiles && warp == st_warp && elect_one()) {
      bulk_store(bwd_tiles + ((ch0 + NT - 1) * (size_t)tiles_per_chunk + S_X) * TILE_BYTES, sm.xt, TILE_BYTES);
      bulk_commit();
    }
    if (write_o) {
      if (PACKED && t0 + L > Tn) {  // the last rows of the box belong to the next sequence: row by row
        store_tile_rows<256>(o_rows + brow * lay.sb + hi * lay.sh + (long long)(tb + t0) * lay.st, lay.st, sm.ot, Tn - t0, tid);
      } else if (warp == out_warp && elect_one()) {           // rows past the end of the tensor are clipped by the TMA store
        tma_store_4d(&tmap_o, sm.ot, 0, tb + t0, hi, brow);
        bulk_commit();
      }
    }
  }
  if ((warp == st_warp || warp == out_warp) && elect_one()) bulk_wait_all();
  marked = __syncthreads_or(marked);
  if (tid == 0) ws_flags[unit] = marked;
  if (warp == 0) tmem_dealloc(tm, 256);
  if (marked && exact.r && ok) exact_unit(exact, smem_raw, tid, unit, hi, brow, tb, Tn, h0, n_state, ht, lay);
}

// The same scan for fewer sequences than SMs: one CTA per SM, nothing else there to cover a wait, and the chain from
// chunk to chunk bounds it.  So every kind of work has warps of its own and they meet at mbarriers only: warps 0-7 read
// accumulators out (as above), one thread each of warps 8, 9, 10 issues the MMAs, fetches operand tiles and copies results
// out.  (With everything between two block barriers the issue of 24 MMAs per chunk, which waits for the tensor pipe, the
// requests for tiles and the waits for copies all held the read-outs up.)  The chain that is left: W h~0, its read-out
// plus U -> sa, b~^T sa, its read-out -> h; the other products run beside the read-outs, and the output rows of a
// chunk are read out while b~^T sa of the next one is computed.  The readers load nothing from global memory: a proxy fence
// waits for such loads too (1200 cycles from W h~0 to sa instead of 320), so U and the decay factors come with the tiles.
// B 2, T 4096, 32 heads, training: 123 -> 100 us (5.0 TB/s with twice the sequences).
struct AloneSmem {
  struct { unsigned char kt[TILE_BYTES], aqk[TILE_BYTES], w[TILE_BYTES], u[TILE_BYTES], v[TILE_BYTES]; } g1[2];
  struct { unsigned char qt[TILE_BYTES], bt[TILE_BYTES], aqb[TILE_BYTES]; } g2[2];
  unsigned char ht[2][TILE_BYTES], sa[2][TILE_BYTES], xt[2][TILE_BYTES], ot[2][TILE_BYTES];
  float aux[2][AUX_FLOATS];         // the chunks' decay factors, with the first group
  uint64_t bar_g1[2], bar_g2[2];
  uint64_t bar_h, bar_s;            // h~0, sa of a chunk are in shared memory (one arrival per reading warp)
  uint64_t bar_a, bar_c;            // W h~0; b~^T sa
  // All products of a chunk have completed, one barrier per stage: the loading warp, whom nothing else holds back, waits
  // here before it fills the stage again, so this barrier cannot get a phase ahead of that wait.
  uint64_t bar_o[2];
  uint64_t bar_free;                // the copies issued in the previous chunk have left shared memory
  uint32_t tmem_base;
};
constexpr int ALONE_THREADS = 352;

template <bool PACKED, bool SORTED>
__global__ void __launch_bounds__(ALONE_THREADS, 1)
r7c_scan_fwd_alone_kernel(const __grid_constant__ CUtensorMap tmap_v, const unsigned char* __restrict__ ws_tiles,
                          const float* __restrict__ ws_aux, int* __restrict__ ws_flags, int tiles_per_chunk,
                          unsigned char* __restrict__ bwd_tiles, const float* __restrict__ h0, int n_state,
                          const __grid_constant__ CUtensorMap tmap_o, int write_o, float* __restrict__ ht,
                          bf16* __restrict__ o_rows, SeqView sv, int H, int NT_slots, TokLayout lay,
                          r7rec::FwdArgs<bf16> exact, int* status, long long* dbg) {
#ifdef RWKVB200_DEVTOOLS
#define R7C_STAMP(n) do { if (dbg && tid == 0 && blockIdx.x == gridDim.x / 2 && c == 2) dbg[n] = clock64(); } while (0)
#else
#define R7C_STAMP(n) do {} while (0)
#endif
  extern __shared__ unsigned char smem_raw[];
  AloneSmem& sm = *reinterpret_cast<AloneSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int unit = blockIdx.x, bi = unit / H, hi = unit % H;
  const int wq = warp & 3, c0 = 32 * (warp >> 2);
  const int row = 16 * wq + (lane & 15);     // state row k (lanes 0-15) or token row i (lanes 16-31)
  const bool state_lane = lane < 16;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&sm.bar_g1[i], 1); mbar_init(&sm.bar_g2[i], 1); mbar_init(&sm.bar_o[i], 1); }
    mbar_init(&sm.bar_h, 8); mbar_init(&sm.bar_s, 8);
    mbar_init(&sm.bar_a, 1); mbar_init(&sm.bar_c, 1); mbar_init(&sm.bar_free, 1);
    fence_mbar_init();
  }
  if (tid == 32) tma_prefetch_maps(tmap_v, tmap_o);
  if (warp == 0) tmem_alloc(&sm.tmem_base, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  earlier_kernels_done();
  later_kernels_may_start();
  if constexpr (SORTED) {
    unit = sorted_scan_unit(sv, H, reinterpret_cast<SortedSeqs*>(sm.ot[0]), tid);
    bi = unit / H; hi = unit % H;
  }
  const size_t ch0 = (size_t)unit * NT_slots;
  auto chunk_tiles = [&](int c) { return ws_tiles + (ch0 + c) * (size_t)tiles_per_chunk * TILE_BYTES; };
  const int Tn = sv.length<PACKED>(bi), tb = sv.first<PACKED>(bi), brow = sv.row<PACKED>(bi);
  const int NT = (Tn + L - 1) / L;           // chunks of this sequence (at least one)
  // TMEM: columns 0..63 lower lane halves = W h~0; three accumulators in turn: lower halves k~^T v + b~^T sa, upper halves
  // the output rows, which are read out while the next chunk is worked on and the state of the one after it is stored
  const uint32_t tm = sm.tmem_base;
  auto acc_col = [](int c) { return 64u + 64u * (uint32_t)(c % 3); };
  bool ok = true;
  int marked = 0;       // a chunk's decay left the range of the scaled operands (the sign of its factors)
  float h[32];          // state lanes: row of the state, columns c0 .. c0 + 31

  if (warp < 8) {       // ---- readers
    const uint32_t tm_w = tmem_addr(tm, 32 * wq, c0);
    auto store_row = [&](unsigned char* tile, const float* x) { tile_store_row32(tile, row, c0, x); };
    // this warp's writes and TMEM reads so far are done, for the async proxy and the tensor pipe too
    auto arrive = [&](uint64_t* bar) {
      fence_async_smem();
      tc_fence_before();
      __syncwarp();
      if (elect_one()) mbar_arrive(bar);
    };
    auto wait = [&](uint64_t* bar, int phase, int code) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar, phase & 1, status, code));
      tc_fence_after();
      return ok;
    };
    auto read_o = [&](int c) {      // the output rows of chunk c into their tile
      uint32_t r[32];
      tmem_ld32(tm_w + acc_col(c), r);
      tmem_ld_wait();
      float x[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(r[j]);
      if (!state_lane) store_row(sm.ot[c & 1], x);
    };
#pragma unroll
    for (int vv = 0; vv < 32; ++vv) h[vv] = 0.f;
    if (state_lane) {      // initial state: h~0 = e^{gref(chunk 0)} h0
      const float e0 = ws_aux[ch0 * AUX_FLOATS + row];
      if (n_state > 0) {
        const float* S = h0 + (size_t)(n_state == 1 ? hi : unit) * 4096;   // S[v][k], h[k][v] = S[v][k]
#pragma unroll
        for (int vv = 0; vv < 32; ++vv) h[vv] = e0 * S[(c0 + vv) * 64 + row];
      }
      store_row(sm.ht[0], h);
    }
    auto put_h = [&](int c) {      // the state at the start of chunk c into its accumulator, whose upper lane halves are free
      uint32_t rh[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) rh[j] = __float_as_uint(h[j]);
      tmem_st32(tm_w + acc_col(c), rh);
      tmem_st_wait();
    };
    put_h(0);
    arrive(&sm.bar_h);
    for (int c = 0; c < NT; ++c) {
      const int p = c & 1;
      R7C_STAMP(48);
      // sa = W h~0 + U
      if (!wait(&sm.bar_g1[p], c >> 1, 211)) break;
      uint4 u[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) u[q] = *reinterpret_cast<const uint4*>(sm.g1[p].u + tile_chunk_off(row, c0 / 8 + q));
      const float scale = sm.aux[p][64 + row];      // e^{glast-gref} of this chunk
      if (!wait(&sm.bar_a, c, 212)) break;
      R7C_STAMP(49);
      {
        uint32_t r[32];
        tmem_ld32(tm_w, r);
        tmem_ld_wait();
        float x[32];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t uu[4] = {u[q].x, u[q].y, u[q].z, u[q].w};
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            x[8 * q + 2 * m] = __uint_as_float(r[8 * q + 2 * m]) + bf16_lo(uu[m]);
            x[8 * q + 2 * m + 1] = __uint_as_float(r[8 * q + 2 * m + 1]) + bf16_hi(uu[m]);
          }
        }
        if (state_lane) store_row(sm.sa[p], x);
      }
      arrive(&sm.bar_s);
      R7C_STAMP(50);
      if (!wait(&sm.bar_free, c, 218)) break;
      if (write_o && c > 0) read_o(c - 1);
      R7C_STAMP(51);
      // X and the next h~0, scaled by e^{glast-gref} of this chunk and e^{gref} of the next
      // (one after the other: their product can underflow float32 where neither factor does)
      if (c + 1 < NT && !wait(&sm.bar_g1[p ^ 1], (c + 1) >> 1, 211)) break;
      const float scale_next = c + 1 < NT ? sm.aux[p ^ 1][row] : 1.f;
      if (!wait(&sm.bar_c, c, 213)) break;
      R7C_STAMP(52);
      {
        uint32_t r[32];
        tmem_ld32(tm_w + acc_col(c), r);
        tmem_ld_wait();
        uint4 xp[4];
#pragma unroll
        for (int j = 0; j < 32; ++j) h[j] = __uint_as_float(r[j]);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          xp[q] = make_uint4(pack_bf16(h[8 * q], h[8 * q + 1]), pack_bf16(h[8 * q + 2], h[8 * q + 3]),
                             pack_bf16(h[8 * q + 4], h[8 * q + 5]), pack_bf16(h[8 * q + 6], h[8 * q + 7]));
        if (state_lane) marked |= scale < 0.f;
        const float sc = fabsf(scale);
#pragma unroll
        for (int j = 0; j < 32; ++j) h[j] = (h[j] * sc) * scale_next;
        if (state_lane) store_row(sm.ht[p ^ 1], h);
        put_h(c + 1);
        arrive(&sm.bar_h);
        if (state_lane && bwd_tiles) {
#pragma unroll
          for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(sm.xt[p] + tile_chunk_off(row, c0 / 8 + q)) = xp[q];
        }
      }
      R7C_STAMP(53);
    }
    ok = ok && wait(&sm.bar_o[(NT - 1) & 1], (NT - 1) >> 1, 217);
  } else if (warp == 8) {      // ---- MMAs
    if (elect_one()) {
      for (int c = 0; c < NT && ok; ++c) {
        const uint32_t acc = acc_col(c);
        auto& g1 = sm.g1[c & 1];
        auto& g2 = sm.g2[c & 1];
        ok = mbar_wait(&sm.bar_g1[c & 1], (c >> 1) & 1, status, 211) && mbar_wait(&sm.bar_h, c & 1, status, 219);
        if (!ok) break;
        tc_fence_after();
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 0, 0), smem_u32(g1.w), smem_u32(sm.ht[c & 1]), false);        // W h~0
        umma_commit(&sm.bar_a);
        umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, acc), smem_u32(g1.kt), smem_u32(g1.v), true);              // h~0 + k~^T v
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, acc), smem_u32(g1.aqk), smem_u32(g1.v), false);           // A_qk v
        ok = mbar_wait(&sm.bar_g2[c & 1], (c >> 1) & 1, status, 214) && mbar_wait(&sm.bar_s, c & 1, status, 220);
        if (!ok) break;
        tc_fence_after();
        umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, acc), smem_u32(g2.bt), smem_u32(sm.sa[c & 1]), true);      // += b~^T sa
        umma_commit(&sm.bar_c);
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, acc), smem_u32(g2.qt), smem_u32(sm.ht[c & 1]), true);     // += q~ h~0
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, acc), smem_u32(g2.aqb), smem_u32(sm.sa[c & 1]), true);    // += A_qb sa
        umma_commit(&sm.bar_o[c & 1]);
      }
    }
    __syncwarp();
  } else if (warp == 9) {      // ---- operand tiles
    if (elect_one()) {
      auto load_1 = [&](int c) {
        auto& g = sm.g1[c & 1];
        uint64_t* bar = &sm.bar_g1[c & 1];
        mbar_expect_tx(bar, 5 * TILE_BYTES + AUX_FLOATS * (uint32_t)sizeof(float));
        bulk_load(g.kt, chunk_tiles(c) + S_KT * TILE_BYTES, 4 * TILE_BYTES, bar);      // k~, A_qk, W, U: adjacent slots
        tma_load_4d(g.v, &tmap_v, bar, 0, tb + c * L, hi, brow);
        bulk_load(sm.aux[c & 1], ws_aux + (ch0 + c) * AUX_FLOATS, AUX_FLOATS * (uint32_t)sizeof(float), bar);
      };
      auto load_2 = [&](int c) {
        mbar_expect_tx(&sm.bar_g2[c & 1], 3 * TILE_BYTES);
        bulk_load(sm.g2[c & 1].qt, chunk_tiles(c) + S_QT * TILE_BYTES, 3 * TILE_BYTES, &sm.bar_g2[c & 1]);     // q~, b~, A_qb
      };
      for (int c = 0; c < 2 && c < NT; ++c) { load_1(c); load_2(c); }
      for (int c = 0; c + 2 < NT && ok; ++c) {
        if (c + 4 < NT) {      // further ahead into L2
          bulk_prefetch_l2(chunk_tiles(c + 4), FWD_TILES * TILE_BYTES);
          tma_prefetch_4d(&tmap_v, 0, tb + (c + 4) * L, hi, brow);
        }
        ok = mbar_wait(&sm.bar_o[c & 1], (c >> 1) & 1, status, 216);      // the tiles of chunk c have been read
        if (ok) { load_1(c + 2); load_2(c + 2); }
      }
    }
    __syncwarp();
  } else {                     // ---- results
    if (elect_one()) {
      for (int c = 0; c < NT && ok; ++c) {
        ok = mbar_wait(&sm.bar_s, c & 1, status, 221);
        bulk_wait_read();      // what was issued a chunk ago
        if (!ok) break;
        mbar_arrive(&sm.bar_free);
        if (bwd_tiles) {       // the backward needs sa, h~0 and X of every chunk
          unsigned char* tiles = bwd_tiles + (ch0 + c) * (size_t)tiles_per_chunk * TILE_BYTES;
          bulk_store(tiles + S_H0 * TILE_BYTES, sm.ht[c & 1], TILE_BYTES);
          bulk_store(tiles + S_SA * TILE_BYTES, sm.sa[c & 1], TILE_BYTES);
          if (c > 0) bulk_store(tiles - ((size_t)tiles_per_chunk - S_X) * TILE_BYTES, sm.xt[(c + 1) & 1], TILE_BYTES);
        }
        if (write_o && c > 1) tma_store_4d(&tmap_o, sm.ot[c & 1], 0, tb + (c - 2) * L, hi, brow);     // staged in chunk c - 1
        bulk_commit();
      }
      bulk_wait_read();
    }
    __syncwarp();
  }
#undef R7C_STAMP
  // ---- what the last chunk still holds: its output rows, X, the final state, and the output rows of the chunk before
  ok = __syncthreads_and(ok);
  tc_fence_after();
  if (ok && warp < 8) {
    uint32_t r[32];
    tmem_ld32(tmem_addr(tm, 32 * wq, acc_col(NT - 1) + c0), r);
    tmem_ld_wait();
    float x[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(r[j]);
    if (!state_lane) {
      if (write_o) tile_store_row32(sm.ot[(NT - 1) & 1], row, c0, x);
    } else if (ht) {
      float* S = ht + (size_t)unit * 4096;
#pragma unroll
      for (int j = 0; j < 32; ++j) S[(c0 + j) * 64 + row] = h[j];
    }
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  if (ok) {
    const int t0 = (NT - 1) * L;
    const bool part = PACKED && t0 + L > Tn;      // the last rows of the box belong to the next sequence: row by row
    if (warp == 10 && elect_one()) {
      if (bwd_tiles)
        bulk_store(bwd_tiles + ((ch0 + NT - 1) * (size_t)tiles_per_chunk + S_X) * TILE_BYTES, sm.xt[(NT - 1) & 1], TILE_BYTES);
      if (write_o && NT > 1) tma_store_4d(&tmap_o, sm.ot[NT & 1], 0, tb + t0 - L, hi, brow);
      if (write_o && !part) tma_store_4d(&tmap_o, sm.ot[(NT - 1) & 1], 0, tb + t0, hi, brow);     // rows past the tensor's end are clipped
      bulk_commit();
    }
    if (write_o && part && warp < 8)
      store_tile_rows<256>(o_rows + brow * lay.sb + hi * lay.sh + (long long)(tb + t0) * lay.st, lay.st, sm.ot[(NT - 1) & 1],
                           Tn - t0, tid);
  }
  if (warp == 10 && elect_one()) bulk_wait_all();
  marked = __syncthreads_or(marked);
  if (tid == 0) ws_flags[unit] = marked;
  if (warp == 0) tmem_dealloc(tm, 256);
  if (warp < 8 && marked && exact.r && ok) exact_unit(exact, smem_raw, tid, unit, hi, brow, tb, Tn, h0, n_state, ht, lay);
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
  DeviceFacts dev;
  int e = device_facts(&dev);
  if (e) return e;
  int* status = dev.status;
  CUtensorMap tmap_v, tmap_o;
  e = make_token_tensor_map(&tmap_v, v, mapB, mapT, H, head_first);
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
    const int smem = (int)sizeof(IntraSmem) + 1024;
    ProfScope prof("r7c_intra_fwd_kernel", st);
    const int n_ch = B * H * NT;
    const int sms = dev.sms;
    const int grid = persistent_grid(n_ch, sms);
#define R7C_LAUNCH_INTRA(P, F)                                                                                     \
    do {                                                                                                           \
      if (allow_smem<r7c_intra_fwd_kernel<P, F>>(dev, smem)) \
        return RWKVB200_E_CUDA;                                                                                    \
      if (int rc = launch(r7c_intra_fwd_kernel<P, F>, grid, 256, smem, st, 1, (const bf16*)r, (const bf16*)w, (const bf16*)k,         \
          (const bf16*)a, (const bf16*)b, tmap_in[0], tmap_in[1], tmap_in[2], tmap_in[3], tmap_in[4], tmap_v,      \
          ws.tiles, ws.aux, tpc, keep_for_bwd ? 1 : 0, sv, WalkDims(H, NT, B, grid), ws.list, lay, status,                     \
          debug_stamp_buffer())) return rc;                                                                        \
    } while (0)
    if (seq_start) R7C_LAUNCH_INTRA(true, false);
    else if (fused) R7C_LAUNCH_INTRA(false, true);
    else R7C_LAUNCH_INTRA(false, false);
#undef R7C_LAUNCH_INTRA
  }
  e = check_launch();
  if (e || !(phases & PHASE_SCAN)) return e;
  {
    ProfScope prof("r7c_scan_fwd_kernel", st);
    // what a unit needs whose decay left the range of the scaled operands (fused producers bound |g| by e^{-1/2}: none)
    r7rec::FwdArgs<bf16> exact{};
    if (!fused && (o || ht))
      exact = r7rec::FwdArgs<bf16>{(const bf16*)r, (const bf16*)w, (const bf16*)k, (const bf16*)v, (const bf16*)a, (const bf16*)b,
                                   0, lay.st, 0, nullptr, (bf16*)o, nullptr, nullptr};
#define R7C_LAUNCH_SCAN(THREADS, SMEM, ...)                                                                         \
    do {                                                                                                           \
      const int smem = (int)sizeof(SMEM) + 1024;                                                                   \
      if (allow_smem<__VA_ARGS__>(dev, smem))                                                                      \
        return RWKVB200_E_CUDA;                                                                                    \
      if (int rc = launch(__VA_ARGS__, B * H, THREADS, smem, st, 1, tmap_v, ws.tiles, ws.aux, ws.flags, tpc,         \
          keep_for_bwd ? ws.tiles : nullptr, h0, n_state, tmap_o, o ? 1 : 0, ht, (bf16*)o, sv, H, NT, lay, exact,  \
          status, debug_stamp_buffer())) return rc;                                                                \
    } while (0)
    const bool packed = seq_start != nullptr, alone = scans_alone(B, Tn, T_total, H, dev.sms, packed, SCAN_FWD);
    const bool sorted = packed && scans_sorted(B, Tn, T_total, H, dev.sms, alone);
    if (!alone) {      // two CTAs per SM
      if (sorted)      R7C_LAUNCH_SCAN(256, ScanSmem, r7c_scan_fwd_kernel<true, true>);
      else if (packed) R7C_LAUNCH_SCAN(256, ScanSmem, r7c_scan_fwd_kernel<true, false>);
      else             R7C_LAUNCH_SCAN(256, ScanSmem, r7c_scan_fwd_kernel<false, false>);
    } else if (sorted) R7C_LAUNCH_SCAN(ALONE_THREADS, AloneSmem, r7c_scan_fwd_alone_kernel<true, true>);
    else if (packed)   R7C_LAUNCH_SCAN(ALONE_THREADS, AloneSmem, r7c_scan_fwd_alone_kernel<true, false>);
    else               R7C_LAUNCH_SCAN(ALONE_THREADS, AloneSmem, r7c_scan_fwd_alone_kernel<false, false>);
#undef R7C_LAUNCH_SCAN
  }
  return check_launch();
}

}  // namespace rwkvb200
