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
constexpr int NROW = 68;   // padded row of the fp32 copy of A_ab (keeps float4 alignment)

// Eleven tiles whose space is used over again; each line says what a tile holds in turn.
struct IntraSmem {
  unsigned char qt[TILE_BYTES], at[TILE_BYTES];     // [q~; a~]  (128-row A operand)
  unsigned char kt[TILE_BYTES], bt[TILE_BYTES];     // [k~; b~]  (128-row B operand)
  unsigned char aqk[TILE_BYTES], aak[TILE_BYTES];   // A_qk, A_ak; the inverse's Q, T; W^, U; N (fp32, both)
  unsigned char aqb[TILE_BYTES];                    // A_qb; P
  unsigned char v[TILE_BYTES];                      // v (TMA)
  unsigned char ainv[TILE_BYTES];                   // Ainv; G; Q
  unsigned char y[TILE_BYTES];                      // raw w (TMA); Y = A_ak v; W
  unsigned char x1[TILE_BYTES];                     // B2; O'
  float nmat[L * NROW];                             // g, then its prefix sums; stril(A_ab) in fp32
  float qtot[4][64];                                // sums of g over the four quarters of the chunk
  float vec[2][64];                                 // e^{gref}, e^{glast-gref}
  uint64_t bar_v, bar_w, bar_in, bar_dr, bar_m1, bar_m2, bar_m3, bar_m4, bar_m5, bar_m6;
  uint32_t tmem_base;
};

// Persistent: CTAs (two per SM) walk over chunk-heads ch = blockIdx.x, blockIdx.x + gridDim.x, ...  The raw tiles of
// the next chunk-head are requested by TMA as soon as the tiles they land in are free: k and v after MMA 2, a after
// MMA 3, w and b after MMA 4, q at the end; and its rows are asked into L2 before that.
// TMEM: columns 0..127 MMA 1; then (M = 64 accumulators pair up on the two lane halves)
//   0..63 G | B2, then P | Q;   64..127 N | O' (from MMA 2 on);   128..191 Y | the inverse's T, P T;   192..255 W | U.
// 256 threads: warp w reads TMEM lanes 32*(w&3).. and the two warps that share a lane window split
// the columns (hsel = w>>2).
template <bool PACKED, bool FUSED>
__global__ void __launch_bounds__(256, 2)
r7c_intra_fwd_kernel(const bf16* __restrict__ q, const bf16* __restrict__ w, const bf16* __restrict__ k,
                     const bf16* __restrict__ a, const bf16* __restrict__ b,
                     const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_w,
                     const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_a,
                     const __grid_constant__ CUtensorMap tmap_b,
                     const __grid_constant__ CUtensorMap tmap_v, unsigned char* __restrict__ ws_tiles,
                     float* __restrict__ ws_aux, int* __restrict__ ws_flags, int tiles_per_chunk,
                     int keep_for_bwd, SeqView sv, int H, int NT, int n_ch, TokLayout lay, int* status, long long* dbg) {
#ifdef RWKVB200_DEVTOOLS
#define R7C_STAMP(n) do { if (dbg && tid == 0 && blockIdx.x == gridDim.x / 2 && it == 15) dbg[n] = clock64(); } while (0)
#else
#define R7C_STAMP(n) do {} while (0)
#endif
  extern __shared__ unsigned char smem_raw[];
  IntraSmem& sm = *reinterpret_cast<IntraSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wq = warp & 3, hsel = warp >> 2;
  const bool st_thread = tid == 64;      // requests raw tiles, copies results out

  if (tid == 0) {
    mbar_init(&sm.bar_v, 1); mbar_init(&sm.bar_w, 1); mbar_init(&sm.bar_in, 1); mbar_init(&sm.bar_dr, 1);
    mbar_init(&sm.bar_m1, 1); mbar_init(&sm.bar_m2, 1); mbar_init(&sm.bar_m3, 2); mbar_init(&sm.bar_m4, 1);
    mbar_init(&sm.bar_m5, 1); mbar_init(&sm.bar_m6, 2);
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
  auto load_w = [&](const ChunkPos& p) { mbar_expect_tx(&sm.bar_w, TILE_BYTES); load(sm.y, &tmap_w, &sm.bar_w, p); };
  auto load_v = [&](const ChunkPos& p) { mbar_expect_tx(&sm.bar_v, TILE_BYTES); load(sm.v, &tmap_v, &sm.bar_v, p); };
  // q, k, a, b share a barrier; k comes first
  auto load_k = [&](const ChunkPos& p) { mbar_expect_tx(&sm.bar_in, 4 * TILE_BYTES); load(sm.kt, &tmap_k, &sm.bar_in, p); };
  auto load_q = [&](const ChunkPos& p) { load(sm.qt, &tmap_q, &sm.bar_in, p); };
  auto load_a = [&](const ChunkPos& p) { load(sm.at, &tmap_a, &sm.bar_in, p); };
  auto load_b = [&](const ChunkPos& p) { load(sm.bt, &tmap_b, &sm.bar_in, p); };
  // chunk slots past the end of a (packed) sequence are skipped
  auto empty = [&](const ChunkPos& p) {
    if constexpr (!PACKED) return false;      // a dense batch has no empty slots
    return p.c * L >= sv.length<PACKED>(p.bi);
  };
  auto advance = [&](ChunkPos p) {
    do { chunk_step(p, gridDim.x, NT, H); } while (p.ch < n_ch && empty(p));
    return p;
  };
  // Ask for a chunk-head's token rows to be brought into L2, ahead of the TMA loads above.
  auto prefetch_rows = [&](const ChunkPos& p) {      // one thread
    const int tt = sv.first<PACKED>(p.bi) + p.c * L, br = sv.row<PACKED>(p.bi);
    tma_prefetch_4d(&tmap_k, 0, tt, p.hi, br);
    tma_prefetch_4d(&tmap_v, 0, tt, p.hi, br);
    tma_prefetch_4d(&tmap_a, 0, tt, p.hi, br);
    tma_prefetch_4d(&tmap_w, 0, tt, p.hi, br);
    tma_prefetch_4d(&tmap_b, 0, tt, p.hi, br);
    tma_prefetch_4d(&tmap_q, 0, tt, p.hi, br);
  };
  ChunkPos cur = chunk_pos(blockIdx.x, NT, H);
  if (cur.ch < n_ch && empty(cur)) cur = advance(cur);
  if (cur.ch < n_ch && st_thread) { load_w(cur); load_k(cur); load_q(cur); load_a(cur); load_b(cur); load_v(cur); }
  // The two CTAs that share an SM would otherwise run their phases in lockstep and compete for the
  // same unit (shared-memory pipe during the triangular solve); start every other CTA half a
  // chunk-head late, where there is more than one chunk-head per CTA.
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
    if (more && tid == 96) prefetch_rows(nxt);
    // this thread's 2 x 16 bytes (8 channels of one token) of the raw w tile
    uint4 rw[2];
    ok = mbar_wait(&sm.bar_w, par, status, 206) && ok;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int e = tid + 256 * n;
      rw[n] = *reinterpret_cast<const uint4*>(sm.y + tile_chunk_off(e >> 3, e & 7));
    }
    // ---- phase A: decay prefix sums (in units of log 2) and the four scaled operands; the prefix sum over tokens goes
    // through shared memory (the fp32 area that later holds A_ab).
    {
      float* gs = sm.nmat;
      float gown[2][8];     // g of this thread's 2 x 8 (token, channel) entries
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int e = tid + 256 * n, row = e >> 3, cc = e & 7;
        const bool valid = t0 + row < Tn;
        const uint32_t u[4] = {rw[n].x, rw[n].y, rw[n].z, rw[n].w};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          float w0 = bf16_lo(u[m]), w1 = bf16_hi(u[m]);
          if constexpr (FUSED) {      // the tile holds p: w = -e^{-1/2} sigmoid(p), as a bfloat16 value
            w0 = round_bf16(W_SCALE * sigmoidf_(w0));
            w1 = round_bf16(W_SCALE * sigmoidf_(w1));
          }
          gown[n][2 * m] = valid ? -LOG2E * ex2(LOG2E * w0) : 0.f;
          gown[n][2 * m + 1] = valid ? -LOG2E * ex2(LOG2E * w1) : 0.f;
        }
        *reinterpret_cast<float4*>(&gs[row * NROW + 8 * cc]) = make_float4(gown[n][0], gown[n][1], gown[n][2], gown[n][3]);
        *reinterpret_cast<float4*>(&gs[row * NROW + 8 * cc + 4]) = make_float4(gown[n][4], gown[n][5], gown[n][6], gown[n][7]);
      }
      __syncthreads();
      R7C_STAMP(1);
      {
        const int c = tid & 63, quarter = tid >> 6;
        float gv[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) gv[j] = gs[(16 * quarter + j) * NROW + c];
        float run = 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j) { run += gv[j]; gv[j] = run; }
        sm.qtot[quarter][c] = run;
        __syncthreads();
        // gi - gref: the prefix inside the half; the reference point is the end of the first half
        const float add = quarter == 0 ? -(run + sm.qtot[1][c]) : quarter == 1 ? -run : quarter == 3 ? sm.qtot[2][c] : 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j) gs[(16 * quarter + j) * NROW + c] = gv[j] + add;
      }
      __syncthreads();
      if (tid < 64) {
        const float tot0 = sm.qtot[0][tid] + sm.qtot[1][tid], tot1 = sm.qtot[2][tid] + sm.qtot[3][tid];
        const float eg = ex2(fmaxf(tot0, EXP2_FLOOR)), dl = ex2(fmaxf(tot1, EXP2_FLOOR));
        sm.vec[0][tid] = eg;                                   // e^{gref}
        sm.vec[1][tid] = dl;                                   // e^{glast-gref}
        ws_aux[(size_t)ch * AUX_FLOATS + tid] = eg;
        ws_aux[(size_t)ch * AUX_FLOATS + 64 + tid] = dl;
        // a half-chunk decay sum beyond the limit: the unit is recomputed by the float32 recurrence
        if (fminf(tot0, tot1) < -DECAY_LIMIT * LOG2E || Tn < SHORT_SEQ) ws_flags[bi * H + hi] = 1;
      }
      // the raw q, k, a, b: each thread scales its own 2 x 16 bytes in place
      uint4 rq[2], rk[2], ra[2], rb[2];
      ok = mbar_wait(&sm.bar_in, par, status, 207) && ok;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int e = tid + 256 * n;
        const uint32_t off = tile_chunk_off(e >> 3, e & 7);
        rq[n] = *reinterpret_cast<const uint4*>(sm.qt + off);
        rk[n] = *reinterpret_cast<const uint4*>(sm.kt + off);
        ra[n] = *reinterpret_cast<const uint4*>(sm.at + off);
        rb[n] = *reinterpret_cast<const uint4*>(sm.bt + off);
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
        float gl[8];
        *reinterpret_cast<float4*>(gl) = *reinterpret_cast<const float4*>(&gs[row * NROW + 8 * cc]);
        *reinterpret_cast<float4*>(gl + 4) = *reinterpret_cast<const float4*>(&gs[row * NROW + 8 * cc + 4]);
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
            const int x = 2 * m + hh;
            const float d1 = gl[x];                                         // gi - gref
            eq[hh] = ex2(d1); ek[hh] = ex2(-d1); ea[hh] = ex2(d1 - gown[n][x]);
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
    if (st_thread) bulk_wait_read();      // the previous results have left their tiles, which the epilogue below rewrites
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
    if (st_thread && ok && keep_for_bwd) {
      bulk_store(out_tiles + S_QT * TILE_BYTES, sm.qt, TILE_BYTES);
      bulk_store(out_tiles + S_KT * TILE_BYTES, sm.kt, 2 * TILE_BYTES);      // k~, b~
      bulk_store(out_tiles + S_AT * TILE_BYTES, sm.at, TILE_BYTES);
      bulk_commit();
    }
    ok = ok && mbar_wait(&sm.bar_m1, par, status, 201);
    tc_fence_after();
    R7C_STAMP(3);
    if (ok) {
      const int r = 32 * wq + lane, i = r & 63;
      const bool lower = r >= 64;       // rows of a~: strictly lower triangle; rows of q~: lower incl. diagonal
      // The warp's 32 rows are i = 32*ihalf + lane, so which side of the diagonal a block of 32 columns lies on is
      // the same for the whole warp: left of the diagonal block every element is kept, right of it every element
      // is zero (TMEM is not read), and only the diagonal block takes a per-element choice.
      const int ihalf = wq & 1;
      auto emit = [&](const float (&x)[32], int j0) {
        if (!lower) {
          tile_store_row32(hsel ? sm.aqb : sm.aqk, i, j0, x);
        } else if (!hsel) {
          tile_store_row32(sm.aak, i, j0, x);
        } else {
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            *reinterpret_cast<float4*>(&sm.nmat[i * NROW + j0 + j]) = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
        }
      };
#pragma unroll
      for (int pp = 0; pp < 2; ++pp) {
        const int j0 = 32 * pp;
        float x[32];
        if (pp > ihalf) {
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] = 0.f;
          emit(x, j0);
          continue;
        }
        uint32_t rr[32];
        tmem_ld32(tmem_addr(tm, 32 * wq, 64 * hsel + 32 * pp), rr);   // hsel 0: products with k~, 1: with b~
        tmem_ld_wait();
        if (pp < ihalf) {
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
          emit(x, j0);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const bool keep = lower ? (j < lane) : (j <= lane);
            x[j] = keep ? __uint_as_float(rr[j]) : 0.f;
          }
          emit(x, j0);
        }
      }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);

    R7C_STAMP(4);
    // ---- MMA 2: Y = A_ak v (columns 128..191), and the first terms of N = k~^T v | O' = A_qk v (columns 64..127)
    if (tid == 0 && ok) {
      ok = mbar_wait(&sm.bar_v, par, status, 202);
      tc_fence_after();
      umma_tile<64, 64, 0, 1>(tmem_addr(tm, 0, 128), smem_u32(sm.aak), smem_u32(sm.v), false);
      umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, 64), smem_u32(sm.kt), smem_u32(sm.v), false);
      umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 64), smem_u32(sm.aqk), smem_u32(sm.v), false);
      umma_commit(&sm.bar_m2);
    }
    if (st_thread && ok && keep_for_bwd) {
      bulk_store(out_tiles + S_AQK * TILE_BYTES, sm.aqk, 2 * TILE_BYTES);      // A_qk, A_ak
      bulk_commit();
    }
    // ---- Ainv = X = (I - N)^-1, N = stril(A_ab), by two levels of block inversion:
    //   D. the four 16 x 16 diagonal blocks D_I = (I - N_II)^-1 in fp32, one column per thread, row by row --
    //      the only substitutions, all four side by side (in place in nmat);
    //   1. the two 32 x 32 diagonal blocks in fp32: X_10 = D_1 (N_10 D_0) and X_32 = D_3 (N_32 D_2), 64 threads
    //      each (in place; P = N_IJ D_J passes through the A_qk tile, free once MMA 2 has read it);
    //   2., 3. the last block X_BA = X_B N_BA X_A (A = rows 0..31, B = rows 32..63) as two tensor-core products.
    {
      const int c = tid & 63, I = tid >> 6;
      float* scratch = reinterpret_cast<float*>(sm.aqk);
      if ((c >> 4) == I) {       // step D (while MMA 2 runs)
        float xb[16];
#pragma unroll
        for (int rr = 0; rr < 16; ++rr) xb[rr] = (rr == (c & 15)) ? 1.f : 0.f;
#pragma unroll
        for (int rr = 1; rr < 16; ++rr) {
          const float* nrow = &sm.nmat[(16 * I + rr) * NROW + 16 * I];
          float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;   // entries at or right of the diagonal are 0
#pragma unroll
          for (int jj = 0; jj < (rr + 3) / 4; ++jj) {
            const float4 n = *reinterpret_cast<const float4*>(nrow + 4 * jj);
            p0 += n.x * xb[4 * jj];
            if (4 * jj + 1 < rr) p1 += n.y * xb[4 * jj + 1];
            if (4 * jj + 2 < rr) p2 += n.z * xb[4 * jj + 2];
            if (4 * jj + 3 < rr) p3 += n.w * xb[4 * jj + 3];
          }
          xb[rr] += (p0 + p1) + (p2 + p3);
        }
        __syncwarp((c & 16) ? 0xffff0000u : 0x0000ffffu);   // the 16 columns of a block share a half-warp
#pragma unroll
        for (int rr = 0; rr < 16; ++rr) sm.nmat[(16 * I + rr) * NROW + c] = xb[rr];
      }
      ok = ok && mbar_wait(&sm.bar_m2, par, status, 203);
      tc_fence_after();
      if (ok) {      // Y rows (lower lane halves)
        uint32_t rr[32];
        tmem_ld32(tmem_addr(tm, 32 * wq, 128 + 32 * hsel), rr);
        tmem_ld_wait();
        if (lane < 16) {
          float x[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
          tile_store_row32(sm.y, 16 * wq + lane, 32 * hsel, x);
        }
      }
      // the scratch area: MMA 2 is done with it, the copies kept for the backward have to be
      if (st_thread && ok) {
        bulk_wait_read();                          // (q~, k~, b~, a~ have left shared memory as well)
        if (more) { load_v(nxt); load_k(nxt); }    // MMA 2 was the last to read v and k~
      }
      ok = __syncthreads_and(ok);
      R7C_STAMP(10);
      if (I & 1) {               // step 1: row block I, column block I - 1
        const int cl = tid & 15, r0 = ((tid & 63) >> 4) * 4;
        const int rb = 16 * I, cbk = 16 * (I - 1);
        float* P = scratch + (I >> 1) * 256;
        float col[16], acc[4];
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) col[kk] = sm.nmat[(cbk + kk) * NROW + cbk + cl];     // D_J[:, cl]
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float* nrow = &sm.nmat[(rb + r0 + q) * NROW + cbk];
          float s_ = 0.f;
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            const float4 n = *reinterpret_cast<const float4*>(nrow + 4 * jj);
            s_ += n.x * col[4 * jj] + n.y * col[4 * jj + 1] + n.z * col[4 * jj + 2] + n.w * col[4 * jj + 3];
          }
          acc[q] = s_;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) P[(r0 + q) * 16 + cl] = acc[q];
        if (I == 1) bar_sync(1, 64); else bar_sync(2, 64);
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) col[kk] = P[kk * 16 + cl];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float* drow = &sm.nmat[(rb + r0 + q) * NROW + rb];       // D_I is stored in full (zeros above)
          float s_ = 0.f;
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            const float4 n = *reinterpret_cast<const float4*>(drow + 4 * jj);
            s_ += n.x * col[4 * jj] + n.y * col[4 * jj + 1] + n.z * col[4 * jj + 2] + n.w * col[4 * jj + 3];
          }
          acc[q] = s_;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) sm.nmat[(rb + r0 + q) * NROW + cbk + cl] = acc[q];
      }
      __syncthreads();
      R7C_STAMP(11);
      // steps 2 and 3 on the tensor cores.  With P = diag(X_A, X_B) (the two finished 32 x 32 blocks) and
      // Q = [0 0; N_BA 0], the missing block is X_BA = (P Q P)_BA: T = Q P, then P T, two 64x64x64 products
      // of bf16 operands (N_BA is a small correction: rounding it, X_A, X_B and T to bf16 changes the rounded
      // inverse by less than the rounding of the inverse itself).  P is the Ainv tile with a zero BA
      // quadrant; Q and T pass through the A_qk / A_ak tiles, free since MMA 2.
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int e = tid + 256 * n, row = e >> 3, cc = e & 7;
        const float4 f0 = *reinterpret_cast<const float4*>(&sm.nmat[row * NROW + 8 * cc]);
        const float4 f1 = *reinterpret_cast<const float4*>(&sm.nmat[row * NROW + 8 * cc + 4]);
        const uint4 val = make_uint4(pack_bf16(f0.x, f0.y), pack_bf16(f0.z, f0.w), pack_bf16(f1.x, f1.y), pack_bf16(f1.z, f1.w));
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        const bool ba = row >= 32 && cc < 4;
        *reinterpret_cast<uint4*>(sm.ainv + tile_chunk_off(row, cc)) = ba ? zero : val;
        *reinterpret_cast<uint4*>(sm.aqk + tile_chunk_off(row, cc)) = ba ? val : zero;
      }
      fence_async_smem();
      tc_fence_before();
      __syncthreads();
      R7C_STAMP(12);
      if (tid == 0) {
        tc_fence_after();
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 128), smem_u32(sm.aqk), smem_u32(sm.ainv), false);     // T = Q P
        umma_commit(&sm.bar_m4);
      }
      ok = mbar_wait(&sm.bar_m4, par, status, 209) && ok;
      tc_fence_after();
      if (ok) {
        uint32_t rr[32];
        tmem_ld32(tmem_addr(tm, 32 * wq, 128 + 32 * hsel), rr);
        tmem_ld_wait();
        if (lane >= 16) {
          float x[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
          tile_store_row32(sm.aak, 16 * wq + (lane & 15), 32 * hsel, x);
        }
      }
      fence_async_smem();
      tc_fence_before();
      ok = __syncthreads_and(ok);
      if (tid == 0 && ok) {
        tc_fence_after();
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 128), smem_u32(sm.ainv), smem_u32(sm.aak), false);     // P T
        umma_commit(&sm.bar_m5);
      }
      ok = ok && mbar_wait(&sm.bar_m5, par, status, 210);
      tc_fence_after();
      if (ok && hsel == 0) {      // rows 32..63, columns 0..31: the BA quadrant of Ainv
        uint32_t rr[32];
        tmem_ld32(tmem_addr(tm, 32 * wq, 128), rr);
        tmem_ld_wait();
        if (lane >= 16 && wq >= 2) {
          float x[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
          tile_store_row32(sm.ainv, 16 * wq + (lane & 15), 0, x);
        }
      }
      R7C_STAMP(13);
    }
    R7C_STAMP(5);
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);

    R7C_STAMP(6);
    // ---- MMA 3: W = Ainv a~ | U = Ainv Y (columns 192..255); for the backward G = A_qb Ainv | B2 = Ainv^T b~ (0..63)
    if (tid == 0 && ok) {
      tc_fence_after();
      umma_tile<64, 64, 0, 1>(tmem_addr(tm, 0, 192), smem_u32(sm.ainv), smem_u32(sm.at), false);
      umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 192), smem_u32(sm.ainv), smem_u32(sm.y), false);
      umma_commit(&sm.bar_m3);
    }
    if (tid == 32 && ok) {
      tc_fence_after();
      if (keep_for_bwd) {
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 0, 0), smem_u32(sm.aqb), smem_u32(sm.ainv), false);
        umma_tile<64, 64, 1, 1>(tmem_addr(tm, 16, 0), smem_u32(sm.ainv), smem_u32(sm.bt), false);
      }
      umma_commit(&sm.bar_m3);
    }
    ok = ok && mbar_wait(&sm.bar_m3, par, status, 204);
    tc_fence_after();
    R7C_STAMP(7);
    if (st_thread && ok && more) load_a(nxt);      // MMA 3 was the last to read a~
    const int i = 16 * wq + (lane & 15), c0 = 32 * hsel;
    const bool lo = lane < 16;
    if (ok) {
      uint32_t rr[32];
      float x[32];
      tmem_ld32(tmem_addr(tm, 32 * wq, 192 + c0), rr);
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
          x[j] *= e.x; x[j + 1] *= e.y; x[j + 2] *= e.z; x[j + 3] *= e.w;
        }
        tile_store_row32(sm.aqk, i, c0, x);
      }
      if (keep_for_bwd) {
        tmem_ld32(tmem_addr(tm, 32 * wq, c0), rr);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
        tile_store_row32(lo ? sm.ainv : sm.x1, i, c0, x);           // G | B2
      }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);

    R7C_STAMP(8);
    // ---- MMA 4: P = b~^T W^ | Q = A_qb W^ (columns 0..63); N += b~^T U | O' += A_qb U (columns 64..127)
    if (tid == 0 && ok) {
      tc_fence_after();
      umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, 0), smem_u32(sm.bt), smem_u32(sm.aqk), false);
      umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, 64), smem_u32(sm.bt), smem_u32(sm.aak), true);
      umma_commit(&sm.bar_m6);
    }
    if (tid == 32 && ok) {
      tc_fence_after();
      umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 0), smem_u32(sm.aqb), smem_u32(sm.aqk), false);
      umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 64), smem_u32(sm.aqb), smem_u32(sm.aak), true);
      umma_commit(&sm.bar_m6);
    }
    if (st_thread && ok) {
      if (keep_for_bwd) {
        bulk_store(out_tiles + S_G * TILE_BYTES, sm.ainv, TILE_BYTES);
        bulk_store(out_tiles + S_B2 * TILE_BYTES, sm.x1, TILE_BYTES);
        bulk_store(out_tiles + S_W * TILE_BYTES, sm.y, TILE_BYTES);
        bulk_store(out_tiles + S_U * TILE_BYTES, sm.aak, TILE_BYTES);
        bulk_commit();
        bulk_wait_read();
      }
      mbar_arrive(&sm.bar_dr);      // the copies have left the tiles that the epilogue rewrites
    }
    ok = ok && mbar_wait(&sm.bar_m6, par, status, 205);
    ok = ok && mbar_wait(&sm.bar_dr, par, status, 208);
    tc_fence_after();
    if (st_thread && ok && more) { load_w(nxt); load_b(nxt); }
    if (ok) {
      uint32_t rr[32];
      float x[32];
      tmem_ld32(tmem_addr(tm, 32 * wq, c0), rr);
      tmem_ld_wait();
      const float dl = sm.vec[1][i];
      if (lo) {      // P, row i = key channel
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]) * dl;
      } else {       // Q = q~ e^{gref} + A_qb W^, row i = token
        tile_load_row32(sm.qt, i, c0, x);
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 e = *reinterpret_cast<const float4*>(&sm.vec[0][c0 + j]);
          x[j] = x[j] * e.x + __uint_as_float(rr[j]);
          x[j + 1] = x[j + 1] * e.y + __uint_as_float(rr[j + 1]);
          x[j + 2] = x[j + 2] * e.z + __uint_as_float(rr[j + 2]);
          x[j + 3] = x[j + 3] * e.w + __uint_as_float(rr[j + 3]);
        }
      }
      tile_store_row32(lo ? sm.aqb : sm.ainv, i, c0, x);
      tmem_ld32(tmem_addr(tm, 32 * wq, 64 + c0), rr);
      tmem_ld_wait();
      if (lo) {      // N, float32
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          *reinterpret_cast<float4*>(sm.aqk + n_piece_off(i, (c0 + j) >> 2)) =
              make_float4(__uint_as_float(rr[j]) * dl, __uint_as_float(rr[j + 1]) * dl, __uint_as_float(rr[j + 2]) * dl,
                          __uint_as_float(rr[j + 3]) * dl);
      } else {       // O'
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
        tile_store_row32(sm.x1, i, c0, x);
      }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    R7C_STAMP(9);
    if (st_thread && ok) {
      bulk_store(out_tiles + S_P * TILE_BYTES, sm.aqb, TILE_BYTES);
      bulk_store(out_tiles + S_Q * TILE_BYTES, sm.ainv, TILE_BYTES);
      bulk_store(out_tiles + S_N * TILE_BYTES, sm.aqk, 2 * TILE_BYTES);
      bulk_store(out_tiles + S_O * TILE_BYTES, sm.x1, TILE_BYTES);
      bulk_commit();
      if (more) load_q(nxt);      // q~ was last read by the epilogue
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
// One 128x64x64 product per chunk, [P; Q] h, row r on TMEM lane r: warps 0, 1 (and 4, 5 for the upper 32 columns) own
// the state rows, warps 2, 3 (6, 7) the token rows.  The two groups meet through mbarriers only.  The chain from
// chunk to chunk runs through the state warps: h (fp32, registers) -> bf16 tile -> product -> read-out -> h; the token
// warps write the output a chunk behind, from the other one of two accumulators.
// STAGES = 2: two CTAs (two sequences) share an SM, the choice when there are more sequences than SMs; bound by the
// 40 KB of tiles per chunk there.  STAGES = 4: one CTA per SM with loads three chunks ahead, for few sequences; the
// latency of the chain bounds it.
struct ScanStage {
  unsigned char p[TILE_BYTES], q[TILE_BYTES];      // [P; Q]  (128-row A operand)
  unsigned char n[2 * TILE_BYTES];                 // N, fp32
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
  const bool state_warp = wq < 2;
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
    bulk_load(g.p, ws_tiles + (ch0 + c) * (size_t)tiles_per_chunk * TILE_BYTES, sizeof(ScanStage), &sm.bar_ld[c % STAGES]);
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
      if (tid == 32 && bwd_tiles) bulk_wait_read();      // the h~0 tile about to be rewritten has left shared memory
      fence_async_smem();
      tc_fence_before();
      ok = bar_sync_and(1, 128, ok);      // the one place where the group may leave the loop: all of it or none
      if (!ok) break;
      if (tid == 0) {
        ok = mbar_wait(&sm.bar_ld[s], sp, status, 211);
        if (c >= 2) ok = mbar_wait(&sm.bar_o[t], ((c >> 1) - 1) & 1, status, 212) && ok;      // this accumulator has been read
        if (ok) {
          tc_fence_after();
          umma_tile<128, 64, 0, 1>(tmem_addr(tm, 0, 64 * t), smem_u32(sm.st[s].p), smem_u32(sm.ht), false);
          umma_commit(&sm.bar_m[t]);
        }
      }
      if (bwd_tiles) {      // h~0 for the backward, under the product; its tile of the chunk before goes out now
        if (tid == 32 && c > 0) {
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
          const float4 n4 = *reinterpret_cast<const float4*>(sm.st[s].n + n_piece_off(row, (c0 + j) >> 2));
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
      if (tid == 32) {
        if (ok) {
          bulk_store(bwd_tiles + ((ch0 + NT - 1) * (size_t)tiles_per_chunk + S_H0) * TILE_BYTES, sm.hs[(NT - 1) & 1], TILE_BYTES);
          bulk_store(fin_tiles + (size_t)unit * TILE_BYTES, sm.ht, TILE_BYTES);
          bulk_commit();
        }
        bulk_wait_all();
      }
    }
  } else {
    const bool ld_thread = tid == 64;
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
      r7c_intra_fwd_kernel<P, F><<<grid, 256, smem, st>>>((const bf16*)r, (const bf16*)w, (const bf16*)k,         \
          (const bf16*)a, (const bf16*)b, tmap_in[0], tmap_in[1], tmap_in[2], tmap_in[3], tmap_in[4], tmap_v,      \
          ws.tiles, ws.aux, ws.flags, tpc, keep_for_bwd ? 1 : 0, sv, H, NT, n_ch, lay, status,                    \
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
