// Chunked RWKV7 backward on tcgen05 (bf16 token tensors).  Equations in rwkv7_chunked.cuh.
//
// Launch sequence (all on the caller's stream, tiles exchanged through the workspace):
//   1. forward intra kernel with keep_for_bwd (q~, k~, b~, a~, A_qk, A_ak, A_qb, W, U, C, B2, decay factors)
//   2. forward scan without output, keeping sa, h~0 and X of every chunk
//      (1 and 2 only if the forward pass did not keep its workspace)
//   3. r7c_bwd_scan_kernel   (one CTA per (b,h), chunks in reverse)  dz, dh^ per chunk, d initial state
//   4. r7c_bwd_final_kernel  (parallel over chunks)   dq, dk, dv, da, db, dw
#include "rwkv7_chunked.cuh"

namespace rwkvb200 {
namespace r7c {

using namespace tc;
typedef __nv_bfloat16 bf16;

// decay sums are kept in units of log 2 (tc::ex2), as in the forward kernels; nothing is clamped

// ---------------------------------------------------------------------------------------------
// 3. reverse scan: grid = B*H, 256 threads (the two warps of a TMEM lane window take 32 columns each)
// ---------------------------------------------------------------------------------------------
// For more sequences than SMs: two CTAs share an SM and memory bounds it (five tiles in, two out per chunk).
// The two products of a chunk that do not need dh, C^T do and
// q~^T do, are issued while the chunk before is read out, into accumulators of their own (by parity of the chunk).
struct BScanStage {
  unsigned char cm[TILE_BYTES], b2[TILE_BYTES];   // adjacent workspace slots: one bulk copy
  unsigned char at[TILE_BYTES], qt[TILE_BYTES], dout[TILE_BYTES];
};
struct BScanSmem {
  BScanStage st[2];
  unsigned char dhh[TILE_BYTES];    // dh^ as bf16, [k][v]
  unsigned char dz[TILE_BYTES];     // dz as bf16, [token][v]
  uint64_t bar_full[2], bar_m1, bar_m2;
  uint32_t tmem_base;
};

template <bool PACKED, bool SORTED>
__global__ void __launch_bounds__(256, 2)
r7c_bwd_scan_kernel(const __grid_constant__ CUtensorMap tmap_do, unsigned char* __restrict__ ws_tiles,
                    const float* __restrict__ ws_aux, int tiles_per_chunk, const float* __restrict__ d_ht,
                    float* __restrict__ d_h0, SeqView sv, int H, int NT_slots, int* status) {
  extern __shared__ unsigned char smem_raw[];
  BScanSmem& sm = *reinterpret_cast<BScanSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wq = warp & 3, hsel = warp >> 2, c0 = 32 * hsel;
  const int row = 16 * wq + (lane & 15);
  const bool state_lane = lane < 16;
  // single-thread jobs side by side: warp 0 issues the MMAs, st_warp copies dh^ and dz out (and waits for its own
  // bulk-copy groups), ld_warp requests the operand tiles of the chunk after the next
  constexpr int st_warp = 1, ld_warp = 2;

  // A packed batch may have many short sequences, whose blocks come in many rounds: where theirs lies is asked for before the TMEM is
  // (4000 of up to 64 tokens, 16 heads: 1125 -> 1087 us).
  if constexpr (PACKED) earlier_kernels_done();
  int unit = blockIdx.x;
  if constexpr (SORTED) unit = sorted_scan_unit(sv, H, reinterpret_cast<SortedSeqs*>(sm.dz), tid);
  const int bi = unit / H, hi = unit % H;
  const int Tn = sv.length<PACKED>(bi), tb = sv.first<PACKED>(bi), brow = sv.row<PACKED>(bi);
  const int NT = (Tn + L - 1) / L;           // chunks of this sequence (at least one)
  if (tid == 0) {
    mbar_init(&sm.bar_full[0], 1); mbar_init(&sm.bar_full[1], 1);
    mbar_init(&sm.bar_m1, 1); mbar_init(&sm.bar_m2, 1);
    fence_mbar_init();
  }
  if (tid == 32) tma_prefetch_maps(tmap_do);
  if (warp == 0) tmem_alloc(&sm.tmem_base, 128);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if constexpr (!PACKED) earlier_kernels_done();
  later_kernels_may_start();
  const size_t ch0 = (size_t)unit * NT_slots;
  const uint32_t tm = sm.tmem_base;
  // TMEM: columns 64 p .., p = parity of the chunk's place: lower lane halves q~^T do + a~^T dz, upper halves dz

  auto issue_loads = [&](int n) {     // n-th chunk in reverse order
    const int c = NT - 1 - n;
    BScanStage& s = sm.st[n & 1];
    unsigned char* tiles = ws_tiles + (ch0 + c) * (size_t)tiles_per_chunk * TILE_BYTES;
    mbar_expect_tx(&sm.bar_full[n & 1], 5 * TILE_BYTES);
    bulk_load(s.cm, tiles + S_C * TILE_BYTES, 2 * TILE_BYTES, &sm.bar_full[n & 1]);
    bulk_load(s.at, tiles + S_AT * TILE_BYTES, TILE_BYTES, &sm.bar_full[n & 1]);
    bulk_load(s.qt, tiles + S_QT * TILE_BYTES, TILE_BYTES, &sm.bar_full[n & 1]);
    tma_load_4d(s.dout, &tmap_do, &sm.bar_full[n & 1], 0, tb + c * L, hi, brow);
  };
  auto mma_ahead = [&](int n) {       // warp 0's thread: what the n-th chunk does not need dh for
    BScanStage& s = sm.st[n & 1];
    if (!mbar_wait(&sm.bar_full[n & 1], (n >> 1) & 1, status, 311)) return false;
    umma_tile<64, 64, 1, 1>(tmem_addr(tm, 16, 64 * (n & 1)), smem_u32(s.cm), smem_u32(s.dout), false);    // C^T do
    umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, 64 * (n & 1)), smem_u32(s.qt), smem_u32(s.dout), false);     // q~^T do
    return true;
  };
  bool ok = true;          // the same in every thread at the loop's head: the result of the last barrier
  if (warp == 0 && elect_one()) {
    issue_loads(0);
    if (NT > 1) issue_loads(1);
    ok = mma_ahead(0);
  }

  // gradient of the state after the current chunk, row k of dh[k][v] = d_ht[v][k]
  float dh[32];        // columns c0 .. c0 + 31
  if (state_lane && d_ht) {
    const float* S = d_ht + (size_t)unit * 4096;
#pragma unroll
    for (int vv = 0; vv < 32; ++vv) dh[vv] = S[(c0 + vv) * 64 + row];
  } else {
#pragma unroll
    for (int vv = 0; vv < 32; ++vv) dh[vv] = 0.f;
  }

  // the two decay factors of a chunk are fetched one chunk ahead: they head the chain of a chunk
  float dc_next = 1.f, e0_next = 1.f;
  if (state_lane) {
    dc_next = ws_aux[(ch0 + NT - 1) * AUX_FLOATS + 64 + row];
    e0_next = ws_aux[(ch0 + NT - 1) * AUX_FLOATS + row];
  }
  bool tail_ok = ok;       // this thread's wait at the end of the previous chunk
  ok = true;
  for (int n = 0; n < NT && ok; ++n) {
    const int c = NT - 1 - n;
    BScanStage& s = sm.st[n & 1];
    const uint32_t tm_w = tmem_addr(tm, 32 * wq, 64 * (n & 1) + c0);
    unsigned char* tiles = ws_tiles + (ch0 + c) * (size_t)tiles_per_chunk * TILE_BYTES;
    const float dc = fabsf(dc_next), e0 = e0_next;
    if (state_lane) {
#pragma unroll
      for (int vv = 0; vv < 32; ++vv) dh[vv] *= dc;      // dh^ = e^{glast-gref} dh_L
      tile_store_row32(sm.dhh, row, c0, dh);
      if (c > 0) {
        dc_next = ws_aux[(ch0 + c - 1) * AUX_FLOATS + 64 + row];
        e0_next = ws_aux[(ch0 + c - 1) * AUX_FLOATS + row];
      }
    }
    if (warp == st_warp && elect_one()) bulk_wait_read();    // the copy of the previous chunk's dz has left its tile, rewritten below
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(tail_ok);
    if (warp == 0 && elect_one() && ok) {
      tc_fence_after();
      umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 64 * (n & 1)), smem_u32(s.b2), smem_u32(sm.dhh), true);   // += B2 dh^
      umma_commit(&sm.bar_m1);
    }
    if (warp == st_warp && elect_one() && ok) {
      bulk_store(tiles + S_DHH * TILE_BYTES, sm.dhh, TILE_BYTES);
      bulk_commit();
    }
    ok = ok && mbar_wait(&sm.bar_m1, n & 1, status, 312);
    tc_fence_after();
    if (ok) {
      uint32_t r[32];
      tmem_ld32(tm_w, r);
      tmem_ld_wait();
      if (!state_lane) {      // dz = C^T do + B2 dh^
        float x[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(r[j]);
        tile_store_row32(sm.dz, row, c0, x);
      }
    }
    if (warp == st_warp && elect_one()) bulk_wait_read();    // the copy of dh^ has left its tile, rewritten at the top of the next chunk
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    if (warp == 0 && elect_one() && ok) {
      tc_fence_after();
      umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, 64 * (n & 1)), smem_u32(s.at), smem_u32(sm.dz), true);      // += a~^T dz
      umma_commit(&sm.bar_m2);
      // the next chunk's accumulators were read out before the barrier at the head of this one
      if (n + 1 < NT) ok = mma_ahead(n + 1);
    }
    if (warp == st_warp && elect_one() && ok) {
      bulk_store(tiles + S_DZ * TILE_BYTES, sm.dz, TILE_BYTES);
      bulk_commit();
    }
    tail_ok = ok && mbar_wait(&sm.bar_m2, n & 1, status, 313);
    tc_fence_after();
    // this stage has been read by the two MMA groups
    if (warp == ld_warp && elect_one() && tail_ok && n + 2 < NT) issue_loads(n + 2);
    if (tail_ok) {
      uint32_t r[32];
      tmem_ld32(tm_w, r);
      tmem_ld_wait();
      if (state_lane) {       // dh0 = e^{gref} (q~^T do + a~^T dz + dh^)
#pragma unroll
        for (int j = 0; j < 32; ++j) dh[j] = e0 * (__uint_as_float(r[j]) + dh[j]);
      }
    }
    // no barrier here: the next one (after dh^ of the next chunk is in its tile) orders these TMEM reads
    // before the MMAs that overwrite the accumulators
  }
  if (state_lane && d_h0 && ok && tail_ok) {
    float* S = d_h0 + (size_t)unit * 4096;
#pragma unroll
    for (int vv = 0; vv < 32; ++vv) S[(c0 + vv) * 64 + row] = dh[vv];
  }
  if (warp == st_warp && elect_one()) bulk_wait_all();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 128);
}

// The same for fewer sequences than SMs: one CTA per SM, and the chain dh^ -> B2 dh^ -> dz -> a~^T dz -> dh bounds it.
// Every kind of work has warps of its own that meet at mbarriers only, as in the forward scan: warps 0-7 read
// accumulators out, one thread each of warps 8, 9, 10 issues the MMAs, fetches tiles (four chunks of them) and copies dh^
// and dz out.  B 2, T 4096, 32 heads: 82 -> 75 us.
struct BAloneSmem {
  BScanStage st[4];
  unsigned char dhh[2][TILE_BYTES], dz[2][TILE_BYTES];
  float aux[4][AUX_FLOATS];     // the chunks' decay factors, with their tiles
  uint64_t bar_full[4];
  uint64_t bar_h, bar_z;        // dh^, dz of a chunk are in shared memory (one arrival per reading warp)
  uint64_t bar_m1;              // dz is in its accumulator
  // dh is in its accumulator and the chunk's tiles have been read: one barrier per stage, so that it cannot get a phase
  // ahead of the loading warp, which waits here before it fills the stage again
  uint64_t bar_m2[4];
  uint64_t bar_free;            // the copies issued in the previous chunk have left shared memory
  uint32_t tmem_base;
};
constexpr int BALONE_THREADS = 352;

template <bool PACKED, bool SORTED>
__global__ void __launch_bounds__(BALONE_THREADS, 1)
r7c_bwd_scan_alone_kernel(const __grid_constant__ CUtensorMap tmap_do, unsigned char* __restrict__ ws_tiles,
                          const float* __restrict__ ws_aux, int tiles_per_chunk, const float* __restrict__ d_ht,
                          float* __restrict__ d_h0, SeqView sv, int H, int NT_slots, int* status) {
  extern __shared__ unsigned char smem_raw[];
  BAloneSmem& sm = *reinterpret_cast<BAloneSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int unit = blockIdx.x, bi = unit / H, hi = unit % H;
  const int wq = warp & 3, c0 = 32 * (warp >> 2);
  const int row = 16 * wq + (lane & 15);
  const bool state_lane = lane < 16;

  if (tid == 0) {
    for (int i = 0; i < 4; ++i) { mbar_init(&sm.bar_full[i], 1); mbar_init(&sm.bar_m2[i], 1); }
    mbar_init(&sm.bar_h, 8); mbar_init(&sm.bar_z, 8);
    mbar_init(&sm.bar_m1, 1); mbar_init(&sm.bar_free, 1);
    fence_mbar_init();
  }
  if (tid == 32) tma_prefetch_maps(tmap_do);
  if (warp == 0) tmem_alloc(&sm.tmem_base, 128);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  earlier_kernels_done();
  later_kernels_may_start();
  if constexpr (SORTED) {
    unit = sorted_scan_unit(sv, H, reinterpret_cast<SortedSeqs*>(sm.dz[0]), tid);
    bi = unit / H; hi = unit % H;
  }
  const size_t ch0 = (size_t)unit * NT_slots;
  const int NT = (sv.length<PACKED>(bi) + L - 1) / L;      // chunks of this sequence
  const int tb = sv.first<PACKED>(bi), brow = sv.row<PACKED>(bi);
  auto chunk_tiles = [&](int n) { return ws_tiles + (ch0 + NT - 1 - n) * (size_t)tiles_per_chunk * TILE_BYTES; };
  // TMEM: columns 64 p .., p = parity of the chunk's place: lower lane halves q~^T do + a~^T dz, upper halves dz
  const uint32_t tm = sm.tmem_base;
  bool ok = true;
  if (warp < 8) {             // ---- readers
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
    // gradient of the state after the current chunk, row k of dh[k][v] = d_ht[v][k], columns c0 .. c0 + 31
    float dh[32];
#pragma unroll
    for (int vv = 0; vv < 32; ++vv) dh[vv] = 0.f;
    if (state_lane && d_ht) {
      const float* S = d_ht + (size_t)unit * 4096;
#pragma unroll
      for (int vv = 0; vv < 32; ++vv) dh[vv] = S[(c0 + vv) * 64 + row];
    }
    for (int n = 0; n < NT; ++n) {
      const uint32_t tm_w = tmem_addr(tm, 32 * wq, 64 * (n & 1) + c0);
      if (!wait(&sm.bar_full[n & 3], n >> 2, 311)) break;
      const float dc = fabsf(sm.aux[n & 3][64 + row]), e0 = sm.aux[n & 3][row];      // (the sign of dc is the intra kernel's mark)
#pragma unroll
      for (int vv = 0; vv < 32; ++vv) dh[vv] *= dc;      // dh^ = e^{glast-gref} dh_L
      if (state_lane) tile_store_row32(sm.dhh[n & 1], row, c0, dh);
      arrive(&sm.bar_h);
      if (!wait(&sm.bar_free, n, 318)) break;      // dz and dh^ of the chunk before have left their tiles but for the last copies
      if (!wait(&sm.bar_m1, n, 312)) break;
      {
        uint32_t r[32];
        tmem_ld32(tm_w, r);
        tmem_ld_wait();
        float x[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(r[j]);
        if (!state_lane) tile_store_row32(sm.dz[n & 1], row, c0, x);      // dz = C^T do + B2 dh^
      }
      arrive(&sm.bar_z);
      if (!wait(&sm.bar_m2[n & 3], n >> 2, 313)) break;
      {
        uint32_t r[32];
        tmem_ld32(tm_w, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) dh[j] = e0 * (__uint_as_float(r[j]) + dh[j]);      // dh0 = e^{gref} (q~^T do + a~^T dz + dh^)
      }
    }
    if (state_lane && d_h0 && ok) {
      float* S = d_h0 + (size_t)unit * 4096;
#pragma unroll
      for (int vv = 0; vv < 32; ++vv) S[(c0 + vv) * 64 + row] = dh[vv];
    }
  } else if (warp == 8) {     // ---- MMAs
    if (elect_one()) {
      auto ahead = [&](int n) {       // what the n-th chunk does not need dh for
        BScanStage& s = sm.st[n & 3];
        if (!mbar_wait(&sm.bar_full[n & 3], (n >> 2) & 1, status, 311)) return false;
        umma_tile<64, 64, 1, 1>(tmem_addr(tm, 16, 64 * (n & 1)), smem_u32(s.cm), smem_u32(s.dout), false);    // C^T do
        umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, 64 * (n & 1)), smem_u32(s.qt), smem_u32(s.dout), false);     // q~^T do
        return true;
      };
      ok = ahead(0);
      for (int n = 0; n < NT && ok; ++n) {
        BScanStage& s = sm.st[n & 3];
        ok = mbar_wait(&sm.bar_h, n & 1, status, 319);
        if (!ok) break;
        tc_fence_after();
        umma_tile<64, 64, 0, 1>(tmem_addr(tm, 16, 64 * (n & 1)), smem_u32(s.b2), smem_u32(sm.dhh[n & 1]), true);   // += B2 dh^
        umma_commit(&sm.bar_m1);
        ok = mbar_wait(&sm.bar_z, n & 1, status, 321);
        if (!ok) break;
        tc_fence_after();
        umma_tile<64, 64, 1, 1>(tmem_addr(tm, 0, 64 * (n & 1)), smem_u32(s.at), smem_u32(sm.dz[n & 1]), true);     // += a~^T dz
        umma_commit(&sm.bar_m2[n & 3]);
        // the next chunk's accumulators were read out before this chunk's dh^ arrived
        if (n + 1 < NT) ok = ahead(n + 1);
      }
    }
    __syncwarp();
  } else if (warp == 9) {     // ---- operand tiles
    if (elect_one()) {
      auto load = [&](int n) {
        BScanStage& s = sm.st[n & 3];
        uint64_t* bar = &sm.bar_full[n & 3];
        mbar_expect_tx(bar, 5 * TILE_BYTES + AUX_FLOATS * (uint32_t)sizeof(float));
        bulk_load(sm.aux[n & 3], ws_aux + (ch0 + NT - 1 - n) * AUX_FLOATS, AUX_FLOATS * (uint32_t)sizeof(float), bar);
        tma_load_4d(s.dout, &tmap_do, bar, 0, tb + (NT - 1 - n) * L, hi, brow);
        bulk_load(s.cm, chunk_tiles(n) + S_C * TILE_BYTES, 2 * TILE_BYTES, bar);      // C, B2: adjacent slots
        bulk_load(s.qt, chunk_tiles(n) + S_QT * TILE_BYTES, TILE_BYTES, bar);
        bulk_load(s.at, chunk_tiles(n) + S_AT * TILE_BYTES, TILE_BYTES, bar);
      };
      for (int n = 0; n < 4 && n < NT; ++n) load(n);
      for (int n = 0; n + 4 < NT && ok; ++n) {
        ok = mbar_wait(&sm.bar_m2[n & 3], (n >> 2) & 1, status, 316);      // the tiles of the n-th chunk have been read
        if (ok) load(n + 4);
      }
    }
    __syncwarp();
  } else {                    // ---- results
    if (elect_one()) {
      for (int n = 0; n < NT && ok; ++n) {
        unsigned char* tiles = chunk_tiles(n);
        ok = mbar_wait(&sm.bar_h, n & 1, status, 322);
        bulk_wait_read();      // what was issued a chunk ago
        if (!ok) break;
        mbar_arrive(&sm.bar_free);
        bulk_store(tiles + S_DHH * TILE_BYTES, sm.dhh[n & 1], TILE_BYTES);
        bulk_commit();
        ok = mbar_wait(&sm.bar_z, n & 1, status, 323);
        if (!ok) break;
        bulk_store(tiles + S_DZ * TILE_BYTES, sm.dz[n & 1], TILE_BYTES);
        bulk_commit();
      }
      bulk_wait_all();
    }
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 128);
}

// ---------------------------------------------------------------------------------------------
// 4. all token gradients of one chunk: persistent CTAs of 256 threads over the B*H*NT chunk-heads
// ---------------------------------------------------------------------------------------------
// What bounds it: per chunk-head about 14 k warp instructions in phases that wait for one another (tiles ->
// products -> read-out -> products -> read-out -> prefix sums).  With one CTA per SM (213 KB of shared memory) the
// SM issued 1.0 instruction per cycle; two CTAs per SM fill each other's waits.  To fit two, a chunk-head lives in
// twelve tiles whose space is used over again (names below: what is loaded, then what replaces it) and one fp32
// array, and an accumulator that does not need the dA tiles is issued with the first MMA group, which frees its
// operands.  TMEM: dA columns 0..127, [dq~; da~] 128..191, dv 192..255 (lower lane halves); [dk~; db~] 0..63 once
// dA has been read.
struct FinalSmem {
  unsigned char dout[TILE_BYTES], dz[TILE_BYTES];       // [do; dz]   then dA_qk, dA_ak   then red1 (fp32)
  unsigned char aqk[TILE_BYTES], aak[TILE_BYTES];       // A_qk, A_ak then dA_qb, dA_ab   then red2 (fp32)
  unsigned char h0[TILE_BYTES];                         // h~0        then dv rows        then w, dw rows
  unsigned char dhh[TILE_BYTES];                        // dh^
  unsigned char v[TILE_BYTES], sa[TILE_BYTES];          // [v; sa]    (sa) then da~ a~ as bf16
  unsigned char qt[TILE_BYTES], at[TILE_BYTES];         // q~, a~     then dq, da rows
  unsigned char kt[TILE_BYTES], bt[TILE_BYTES];         // k~, b~     then dk, db rows
  float gs[L * 64];         // g log2(e), then (gi - gref) log2(e): inclusive prefix inside the chunk (sw64)
  float quart[3][64];       // sums over quarters of the chunk; [2] between the prefix sum and the epilogue: -gref
  uint64_t bar_l0, bar_l1, bar_l2, bar_w, bar_m1, bar_m2;
  uint32_t tmem_base;
};
// two CTAs per SM: 228 KB shared by both, 1 KB of each reserved by the system
static_assert(sizeof(FinalSmem) <= 115712, "two CTAs per SM");

// index of (row, channel) in a 64 x 64 fp32 array whose 16-byte pieces are permuted by the row, so that threads that
// own a row and threads that own a channel both access it without bank conflicts
__device__ __forceinline__ int sw64(int row, int c) { return row * 64 + ((((c >> 2) ^ (row & 7)) << 2) | (c & 3)); }

// 256 threads: warp w reads TMEM lanes 32*(w&3).. (its row), and the two warps that share a lane
// window split the columns (hsel = w>>2), so every elementwise phase is spread over 8 warps.
template <bool PACKED, bool FUSED>
__global__ void __launch_bounds__(256, 2)
r7c_bwd_final_kernel(const bf16* __restrict__ w, const __grid_constant__ CUtensorMap tmap_w,
                     const __grid_constant__ CUtensorMap tmap_do,
                     const __grid_constant__ CUtensorMap tmap_v, const unsigned char* __restrict__ ws_tiles,
                     int tiles_per_chunk, const __grid_constant__ CUtensorMap tmap_dq,
                     const __grid_constant__ CUtensorMap tmap_dw, const __grid_constant__ CUtensorMap tmap_dk,
                     const __grid_constant__ CUtensorMap tmap_dv, const __grid_constant__ CUtensorMap tmap_da,
                     const __grid_constant__ CUtensorMap tmap_db,
                     bf16* __restrict__ dq_rows, bf16* __restrict__ dw_rows, bf16* __restrict__ dk_rows,
                     bf16* __restrict__ dv_rows, bf16* __restrict__ da_rows, bf16* __restrict__ db_rows,
                     SeqView sv, const __grid_constant__ WalkDims dims, const int2* list, TokLayout lay, int* status, long long* dbg) {
#ifdef RWKVB200_DEVTOOLS
#define R7C_STAMP(n) do { if (dbg && tid == 0 && blockIdx.x == gridDim.x / 2 && it == 15) dbg[n] = clock64(); } while (0)
#else
#define R7C_STAMP(n) do {} while (0)
#endif
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  FinalSmem& sm = *reinterpret_cast<FinalSmem*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wq = warp & 3, hsel = warp >> 2;
  // The swizzled tiles need this alignment, and two CTAs per SM leave no room to align by hand (nor registers for a base that
  // is not a constant: 1.49 -> 1.71 ms per step at B 8, T 4096, 32 heads); the launch has made sure of it.
  if (smem_u32(smem_raw) & 1023u) {
    if (tid == 0) atomicCAS(status, 0, 320);
    return;
  }

  if (tid == 0) {
    // an MMA group is issued by several threads, one accumulator each, and completes with the arrival of all
    mbar_init(&sm.bar_l0, 1); mbar_init(&sm.bar_l1, 1); mbar_init(&sm.bar_l2, 1);
    mbar_init(&sm.bar_w, 1); mbar_init(&sm.bar_m1, 3); mbar_init(&sm.bar_m2, 2);
    fence_mbar_init();
  }
  if (tid == 32) tma_prefetch_maps(tmap_w, tmap_do, tmap_v, tmap_dq, tmap_dw, tmap_dk, tmap_dv, tmap_da, tmap_db);
  if (warp == 0) tmem_alloc(&sm.tmem_base, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  earlier_kernels_done();
  later_kernels_may_start();
  const uint32_t tm = sm.tmem_base;
  constexpr int st_warp = 3;      // requests the tiles, stores the results

  // the tiles of a chunk-head in the order in which their space becomes free
  auto load_0 = [&](const ChunkPos& p) {      // dh^, v
    const unsigned char* tiles = ws_tiles + (size_t)p.ch * tiles_per_chunk * TILE_BYTES;
    mbar_expect_tx(&sm.bar_l0, 2 * TILE_BYTES);
    bulk_load(sm.dhh, tiles + S_DHH * TILE_BYTES, TILE_BYTES, &sm.bar_l0);
    tma_load_4d(sm.v, &tmap_v, &sm.bar_l0, 0, sv.first<PACKED>(p.bi) + p.c * L, p.hi, sv.row<PACKED>(p.bi));
  };
  auto load_1a = [&](const ChunkPos& p) {     // the other operands of MMA group 1, but for sa, k~ and h~0
    const unsigned char* tiles = ws_tiles + (size_t)p.ch * tiles_per_chunk * TILE_BYTES;
    mbar_expect_tx(&sm.bar_l1, 7 * TILE_BYTES);
    tma_load_4d(sm.dout, &tmap_do, &sm.bar_l1, 0, sv.first<PACKED>(p.bi) + p.c * L, p.hi, sv.row<PACKED>(p.bi));
    bulk_load(sm.dz, tiles + S_DZ * TILE_BYTES, TILE_BYTES, &sm.bar_l1);
    bulk_load(sm.aqk, tiles + S_AQK * TILE_BYTES, TILE_BYTES, &sm.bar_l1);
    bulk_load(sm.aak, tiles + S_AAK * TILE_BYTES, TILE_BYTES, &sm.bar_l1);
  };
  auto load_sa = [&](const ChunkPos& p) {
    bulk_load(sm.sa, ws_tiles + ((size_t)p.ch * tiles_per_chunk + S_SA) * TILE_BYTES, TILE_BYTES, &sm.bar_l1);
  };
  auto load_2 = [&](const ChunkPos& p) {      // k~; q~, a~, b~ (MMA group 2 and the epilogue)
    const unsigned char* tiles = ws_tiles + (size_t)p.ch * tiles_per_chunk * TILE_BYTES;
    bulk_load(sm.kt, tiles + S_KT * TILE_BYTES, TILE_BYTES, &sm.bar_l1);
    mbar_expect_tx(&sm.bar_l2, 3 * TILE_BYTES);
    bulk_load(sm.qt, tiles + S_QT * TILE_BYTES, TILE_BYTES, &sm.bar_l2);
    bulk_load(sm.at, tiles + S_AT * TILE_BYTES, TILE_BYTES, &sm.bar_l2);
    bulk_load(sm.bt, tiles + S_BT * TILE_BYTES, TILE_BYTES, &sm.bar_l2);
  };
  auto load_1b = [&](const ChunkPos& p) {     // h~0
    const unsigned char* tiles = ws_tiles + (size_t)p.ch * tiles_per_chunk * TILE_BYTES;
    bulk_load(sm.h0, tiles + S_H0 * TILE_BYTES, TILE_BYTES, &sm.bar_l1);
  };
  auto load_w_tile = [&](const ChunkPos& p) { // the w rows once more (from L2), for the decay gradient
    mbar_expect_tx(&sm.bar_w, TILE_BYTES);
    tma_load_4d(sm.h0, &tmap_w, &sm.bar_w, 0, sv.first<PACKED>(p.bi) + p.c * L, p.hi, sv.row<PACKED>(p.bi));
  };
  // Ask for everything a chunk-head will load to be brought into L2 (issued most of a chunk-head ahead of the
  // loads themselves, which then take an L2 round trip instead of a DRAM one).
  auto prefetch_l2 = [&](const ChunkPos& p) {      // one warp
    const int t0 = p.c * L;
    const unsigned char* tiles = ws_tiles + (size_t)p.ch * tiles_per_chunk * TILE_BYTES;
    if (elect_one()) {
      tma_prefetch_4d(&tmap_do, 0, sv.first<PACKED>(p.bi) + t0, p.hi, sv.row<PACKED>(p.bi));
      tma_prefetch_4d(&tmap_v, 0, sv.first<PACKED>(p.bi) + t0, p.hi, sv.row<PACKED>(p.bi));
      bulk_prefetch_l2(tiles + S_KT * TILE_BYTES, 2 * TILE_BYTES);     // k~, A_qk
      bulk_prefetch_l2(tiles + S_QT * TILE_BYTES, 2 * TILE_BYTES);     // q~, b~
      bulk_prefetch_l2(tiles + S_AT * TILE_BYTES, 5 * TILE_BYTES);     // a~, A_ak, sa, h~0, X
      bulk_prefetch_l2(tiles + S_DZ * TILE_BYTES, 2 * TILE_BYTES);     // dz, dh^
    }
  };
  auto load_w = [&](const ChunkPos& p, uint4 (&rw)[2]) {   // all threads: 2 x 8 channels of the chunk's w rows
    const int t0 = p.c * L, Tn = sv.length<PACKED>(p.bi);
    const long long base = sv.row<PACKED>(p.bi) * lay.sb + p.hi * lay.sh + sv.first<PACKED>(p.bi) * lay.st;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int e = tid + 256 * n, row = e >> 3, cc = e & 7, tok = t0 + row;
      rw[n] = make_uint4(0u, 0u, 0u, 0u);
      if (tok < Tn) rw[n] = __ldg(reinterpret_cast<const uint4*>(w + base + (long long)tok * lay.st + 8 * cc));
    }
  };

  // Dense: unit by unit, for the 20 tiles that lie side by side in the workspace; by rows of tokens, as the intra kernel goes, this
  // one took 500 us against 489 (B 8, T 4096, 32 heads).
  const auto walk = [&] {
    if constexpr (PACKED) return ListWalk{dims, list}; else return UnitWalk{dims};
  }();
  ChunkPos cur = walk.first();

  uint4 rw[2];
  if (cur.ch < dims.n_ch) {
    if (warp == st_warp && elect_one()) { load_0(cur); load_1a(cur); load_sa(cur); load_2(cur); load_1b(cur); }
    load_w(cur, rw);
  }

  bool ok = true;
  int it = 0;
  for (ChunkPos nxt; cur.ch < dims.n_ch && ok; cur = nxt, ++it) {
    const int bi = cur.bi, hi = cur.hi, t0 = cur.c * L;
    const int Tn = sv.length<PACKED>(bi);
    // in a packed batch the last rows of a sequence's last chunk belong to the next sequence: such a chunk
    // is stored row by row instead of by TMA boxes
    const bool row_stores = PACKED && t0 + L > Tn;
    const long long out_base = sv.row<PACKED>(bi) * lay.sb + hi * lay.sh + (long long)(sv.first<PACKED>(bi) + t0) * lay.st;
    const int tt = sv.first<PACKED>(bi) + t0, br = sv.row<PACKED>(bi);
    const unsigned char* tiles = ws_tiles + (size_t)cur.ch * tiles_per_chunk * TILE_BYTES;
    const uint32_t par = it & 1;
    nxt = walk.after(cur, it);
    const bool more = nxt.ch < dims.n_ch;
    R7C_STAMP(16);

    // X, straight from the workspace: the threads of the last quarter hold a row each until they have dh^
    uint4 xa[8];
    if (tid >= 192) {
      const uint4* xr = reinterpret_cast<const uint4*>(tiles + S_X * TILE_BYTES);
#pragma unroll
      for (int q = 0; q < 8; ++q) xa[q] = __ldg(xr + (tile_chunk_off(tid & 63, q) >> 4));
    }
    // ---- g of every (token, channel), from the w rows already in registers
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int e = tid + 256 * n, row = e >> 3, cc = e & 7;
      const bool valid = t0 + row < Tn;
      const uint32_t u[4] = {rw[n].x, rw[n].y, rw[n].z, rw[n].w};
      float g[8];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        float w0 = bf16_lo(u[m]), w1 = bf16_hi(u[m]);
        if constexpr (FUSED) {      // the rows hold p: w = -e^{-1/2} sigmoid(p), as a bfloat16 value
          w0 = round_bf16(W_SCALE * sigmoidf_(w0));
          w1 = round_bf16(W_SCALE * sigmoidf_(w1));
        }
        g[2 * m] = valid ? -LOG2E * ex2(LOG2E * w0) : 0.f;
        g[2 * m + 1] = valid ? -LOG2E * ex2(LOG2E * w1) : 0.f;
      }
      *reinterpret_cast<float4*>(&sm.gs[sw64(row, 8 * cc)]) = make_float4(g[0], g[1], g[2], g[3]);
      *reinterpret_cast<float4*>(&sm.gs[sw64(row, 8 * cc + 4)]) = make_float4(g[4], g[5], g[6], g[7]);
    }
    R7C_STAMP(17);
    // ---- MMA group 1: all four dA products; dv; the state part of [dq~; da~]
    if (warp < 3 && elect_one()) {
      ok = mbar_wait(&sm.bar_l0, par, status, 321) && ok;
      ok = mbar_wait(&sm.bar_l1, par, status, 324) && ok;
      if (ok) {
        tc_fence_after();
        if (warp == 0) {
          umma_tile<128, 128, 0, 0>(tmem_addr(tm, 0, 0), smem_u32(sm.dout), smem_u32(sm.v), false);        // [do;dz] [v;sa]^T
        } else if (warp == 1) {
          umma_tile<64, 64, 1, 1, 8>(tmem_addr(tm, 0, 192), smem_u32(sm.aqk), smem_u32(sm.dout), false);   // A_qk^T do + A_ak^T dz
          umma_tile<64, 64, 0, 1>(tmem_addr(tm, 0, 192), smem_u32(sm.kt), smem_u32(sm.dhh), true);         // + k~ dh^
        } else {
          umma_tile<128, 64, 0, 0>(tmem_addr(tm, 0, 128), smem_u32(sm.dout), smem_u32(sm.h0), false);      // [do;dz] h~0^T
        }
        umma_commit(&sm.bar_m1);
      }
    }
    ok = __syncthreads_and(ok);
    R7C_STAMP(18);
    if (warp == 3 && more) prefetch_l2(nxt);
    // ---- meanwhile: prefix sums of g over tokens, thread = (channel, quarter of the chunk)
    float dglast = 0.f;       // threads of the last quarter: sum_v dh^[c][v] X[c][v]
    {
      const int c = tid & 63, quarter = tid >> 6;
      float gv[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) gv[j] = sm.gs[sw64(16 * quarter + j, c)];
      float run = 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) { run += gv[j]; gv[j] = run; }
      if (quarter == 1 || quarter == 2) sm.quart[quarter - 1][c] = run;
      __syncthreads();
      // gi - gref: the prefix inside the half; the first half lies before the reference point, the end of that half
      const float add = quarter == 0 ? -(run + sm.quart[0][c]) : quarter == 1 ? -run : quarter == 3 ? sm.quart[1][c] : 0.f;
      if (quarter == 0) sm.quart[2][c] = add;      // -gref: the exclusive prefix of the first token
#pragma unroll
      for (int j = 0; j < 16; ++j) sm.gs[sw64(16 * quarter + j, c)] = gv[j] + add;
      if (quarter == 3 && ok) {
        ok = mbar_wait(&sm.bar_l0, par, status, 325) && ok;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const uint4 da_ = *reinterpret_cast<const uint4*>(sm.dhh + tile_chunk_off(c, q));
          dglast += bf16_lo(xa[q].x) * bf16_lo(da_.x) + bf16_hi(xa[q].x) * bf16_hi(da_.x);
          dglast += bf16_lo(xa[q].y) * bf16_lo(da_.y) + bf16_hi(xa[q].y) * bf16_hi(da_.y);
          dglast += bf16_lo(xa[q].z) * bf16_lo(da_.z) + bf16_hi(xa[q].z) * bf16_hi(da_.z);
          dglast += bf16_lo(xa[q].w) * bf16_lo(da_.w) + bf16_hi(xa[q].w) * bf16_hi(da_.w);
        }
      }
    }
    ok = mbar_wait(&sm.bar_m1, par, status, 322) && ok;
    tc_fence_after();
    R7C_STAMP(19);
    if (ok) {
      const int r = 32 * wq + lane, i = r & 63;
      const bool lower = r >= 64;       // rows of dz: strictly lower; rows of do: lower incl. diagonal
      // The warp's 32 rows are i = 32*ihalf + lane, so which side of the diagonal a block of 32 columns lies on is
      // the same for the whole warp: left of the diagonal block every element is kept, right of it every element
      // is zero (TMEM is not read), and only the diagonal block takes a per-element choice.
      const int ihalf = wq & 1;
      // dA tiles, in the order dA_qk, dA_ak, dA_qb, dA_ab, over the operands of group 1
      unsigned char* dst = sm.dout + ((lower ? 1 : 0) + 2 * hsel) * TILE_BYTES;
#pragma unroll
      for (int pp = 0; pp < 2; ++pp) {
        const int part = 2 * hsel + pp;   // hsel 0: products with v (dA_qk / dA_ak); hsel 1: with sa (dA_qb / dA_ab)
        const int j0 = 32 * pp;
        float x[32];
        if (pp > ihalf) {
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] = 0.f;
          tile_store_row32(dst, i, j0, x);
          continue;
        }
        uint32_t rr[32];
        tmem_ld32(tmem_addr(tm, 32 * wq, 32 * part), rr);
        tmem_ld_wait();
        if (pp < ihalf) {
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
          tile_store_row32(dst, i, j0, x);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const bool keep = lower ? (j < lane) : (j <= lane);
            x[j] = keep ? __uint_as_float(rr[j]) : 0.f;
          }
          tile_store_row32(dst, i, j0, x);
        }
      }
      // dv rows sit on the lower lane halves of columns 192..255; each warp of a pair takes 32 columns
      const int row = 16 * wq + (lane & 15);
      uint32_t rr[32];
      tmem_ld32(tmem_addr(tm, 32 * wq, 192 + 32 * hsel), rr);
      tmem_ld_wait();
      if (lane < 16) {
        float x[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(rr[j]);
        tile_store_row32(sm.h0, row, 32 * hsel, x);
      }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    R7C_STAMP(20);

    // ---- MMA group 2: [dq~; da~] completed (columns 128..191), and [dk~; db~] (columns 0..63)
    if (warp < 2 && elect_one() && ok) {
      ok = mbar_wait(&sm.bar_l2, par, status, 326);
      if (ok) {
        tc_fence_after();
        if (warp == 0) {
          umma_tile<128, 64, 0, 1>(tmem_addr(tm, 0, 128), smem_u32(sm.dout), smem_u32(sm.kt), true);         // + [dA_qk;dA_ak] k~
          umma_tile<128, 64, 0, 1>(tmem_addr(tm, 0, 128), smem_u32(sm.aqk), smem_u32(sm.bt), true);          // + [dA_qb;dA_ab] b~
        } else {
          umma_tile<128, 64, 0, 0>(tmem_addr(tm, 0, 0), smem_u32(sm.v), smem_u32(sm.dhh), false);            // [v;sa] dh^^T
          umma_tile<128, 64, 1, 1>(tmem_addr(tm, 0, 0), smem_u32(sm.dout), smem_u32(sm.qt), true, 2 * TILE_BYTES);  // + [dA_qk|dA_qb]^T q~
          umma_tile<128, 64, 1, 1>(tmem_addr(tm, 0, 0), smem_u32(sm.dz), smem_u32(sm.at), true, 2 * TILE_BYTES);    // + [dA_ak|dA_ab]^T a~
        }
        umma_commit(&sm.bar_m2);
      }
    }
    if (warp == st_warp && elect_one() && ok && !row_stores) {
      tma_store_4d(&tmap_dv, sm.h0, 0, tt, hi, br);
      bulk_commit();
    }
    if (row_stores && ok) store_tile_rows<256>(dv_rows + out_base, lay.st, sm.h0, Tn - t0, tid);
    if (more) load_w(nxt, rw);
    ok = mbar_wait(&sm.bar_m2, par, status, 323) && ok;
    ok = mbar_wait(&sm.bar_l2, par, status, 327) && ok;      // the epilogue reads q~, a~, b~ (and k~, which came with group 1)
    ok = mbar_wait(&sm.bar_l1, par, status, 328) && ok;
    tc_fence_after();
    R7C_STAMP(21);
    if (warp == st_warp && elect_one() && ok) {
      if (more) load_0(nxt);      // dh^ and v have been read for the last time
      bulk_wait_read();           // the copy of dv has left its tile, which will hold w and then dw
      if (!FUSED && !row_stores) load_w_tile(cur);
    }

    // ---- epilogue.  Row r < 64 holds dq~_i and dk~_i (token i = r), row r >= 64 holds da~_i, db~_i; the
    // two warps of a lane window take 32 channels each.  red1 = dq~ q~ - dk~ k~ and red2 = da~ a~ - db~ b~ overlay
    // the dA tiles (dead once MMA group 2 has completed); the results replace q~, k~ / a~, b~ row by row.
    float* red1 = reinterpret_cast<float*>(sm.dout);
    float* red2 = reinterpret_cast<float*>(sm.aqk);
    if (ok) {
      const int r = 32 * wq + lane, i = r & 63;
      const bool second = r >= 64;
      float* red = second ? red2 : red1;
      unsigned char* tile1 = second ? sm.at : sm.qt;
      unsigned char* tile2 = second ? sm.bt : sm.kt;
      // exponents of the first factor: inclusive prefix for q~, exclusive (the previous token's) for a~
      const float* grow = second ? (i ? sm.gs + 64 * (i - 1) : sm.quart[2]) : sm.gs + 64 * i;
      const int gkey = second ? (i ? (i - 1) & 7 : 0) : i & 7;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int c0 = 32 * hsel + 16 * half;
        uint32_t r1[16], r2[16];
        tmem_ld16(tmem_addr(tm, 32 * wq, 128 + c0), r1);    // dq~ / da~
        tmem_ld16(tmem_addr(tm, 32 * wq, c0), r2);          // dk~ / db~
        tmem_ld_wait();
        float t1[16], t2[16];
        tile_load_row<16>(tile1, i, c0, t1);
        tile_load_row<16>(tile2, i, c0, t2);
#pragma unroll
        for (int j4 = 0; j4 < 16; j4 += 4) {
          const int c = c0 + j4;
          const float4 gs4 = *reinterpret_cast<const float4*>(&sm.gs[sw64(i, c)]);
          const float4 ge4 = *reinterpret_cast<const float4*>(grow + (((c >> 2) ^ gkey) << 2));
          const float gsv[4] = {gs4.x, gs4.y, gs4.z, gs4.w}, gev[4] = {ge4.x, ge4.y, ge4.z, ge4.w};
          float rd[4];
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            const int j = j4 + m;
            const float x1 = __uint_as_float(r1[j]), x2 = __uint_as_float(r2[j]);
            const float e1 = x1 * t1[j];
            rd[m] = e1 - x2 * t2[j];
            t1[j] = x1 * ex2(gev[m]);                                      // dq / da
            t2[j] = x2 * ex2(-gsv[m]);                                     // dk / db
            r1[j] = __float_as_uint(e1);
          }
          *reinterpret_cast<float4*>(&red[sw64(i, c)]) = make_float4(rd[0], rd[1], rd[2], rd[3]);
        }
        tile_store_row<16>(tile1, i, c0, t1);
        tile_store_row<16>(tile2, i, c0, t2);
        if (second) {      // da~ a~
#pragma unroll
          for (int j = 0; j < 16; ++j) t1[j] = __uint_as_float(r1[j]);
          tile_store_row<16>(sm.sa, i, c0, t1);
        }
      }
    }
    fence_async_smem();
    ok = __syncthreads_and(ok);
    R7C_STAMP(22);
    if (row_stores && ok) {
      if (!FUSED && warp == st_warp && elect_one()) load_w_tile(cur);      // (every thread has copied its dv rows out)
      store_tile_rows<256>(dq_rows + out_base, lay.st, sm.qt, Tn - t0, tid);
      store_tile_rows<256>(dk_rows + out_base, lay.st, sm.kt, Tn - t0, tid);
      store_tile_rows<256>(da_rows + out_base, lay.st, sm.at, Tn - t0, tid);
      store_tile_rows<256>(db_rows + out_base, lay.st, sm.bt, Tn - t0, tid);
    }
    if (warp == st_warp && elect_one() && ok && !row_stores) {
      tma_store_4d(&tmap_dq, sm.qt, 0, tt, hi, br);
      tma_store_4d(&tmap_dk, sm.kt, 0, tt, hi, br);
      tma_store_4d(&tmap_da, sm.at, 0, tt, hi, br);
      tma_store_4d(&tmap_db, sm.bt, 0, tt, hi, br);
      bulk_commit();
    }
    // reverse inclusive prefix over tokens, per channel; thread = (channel, quarter)
    {
      const int c = tid & 63, quarter = tid >> 6;
      float rv[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) rv[j] = red1[sw64(16 * quarter + j, c)] + red2[sw64(16 * quarter + j, c)];
      float run = dglast;
#pragma unroll
      for (int j = 15; j >= 0; --j) { run += rv[j]; rv[j] = run; }
      float gprev = 0.f;
      if constexpr (FUSED) {
        gprev = quarter ? sm.gs[sw64(16 * quarter - 1, c)] : sm.quart[2][c];
        __syncthreads();    // -gref has been read
      }
      if (quarter) sm.quart[quarter - 1][c] = run;      // the last quarter's sum carries dglast
      fence_async_smem();
      __syncthreads();      // red1 and red2 have been read
      if (warp == st_warp && elect_one() && ok && more) load_1a(nxt);
      float add = 0.f;
      for (int q2 = quarter; q2 < 3; ++q2) add += sm.quart[q2][c];
      if constexpr (!FUSED) ok = ok && mbar_wait(&sm.bar_w, par, status, 329);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int ii = 16 * quarter + j;
        const float e_ = __bfloat162float(*reinterpret_cast<const bf16*>(sm.sa + tile_off(ii, c)));
        const float dg = rv[j] + add - e_;
        // dw = dg g (g in units of log 2), with g from w itself: as the difference of two prefix sums (up to 87) the g of a
        // token that decays slowly among faster ones would lose its digits (15 % at g = e^-11), and that of a masked token
        // would not be 0.  Fused producers keep |g| within 0.54 .. 1: there the difference is good to 5e-6 and saves the
        // tile and the sigmoids (484 -> 472 us, B 4, T 2000, 32 heads, forward and backward).
        bf16* out = reinterpret_cast<bf16*>(sm.h0 + tile_off(ii, c));
        float g;
        if constexpr (FUSED) {
          const float gi = sm.gs[sw64(ii, c)];
          g = gi - gprev;
          gprev = gi;
        } else {
          g = -LOG2E * ex2(LOG2E * __bfloat162float(*out));
        }
        *out = __float2bfloat16_rn(dg * (LN2 * g));
      }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    if (row_stores) {
      if (ok) store_tile_rows<256>(dw_rows + out_base, lay.st, sm.h0, Tn - t0, tid);
      fence_async_smem();
      __syncthreads();      // the rows are read before their space is loaded again
    }
    if (warp == st_warp && elect_one() && ok) {
      if (!row_stores) {
        tma_store_4d(&tmap_dw, sm.h0, 0, tt, hi, br);
        bulk_commit();
      }
      if (more) {
        load_sa(nxt);
        bulk_wait_read_1();       // dq, dk, da, db have left their tiles
        load_2(nxt);
        bulk_wait_read();         // and dw
        load_1b(nxt);
      }
    }
    R7C_STAMP(23);
  }
  if (warp == st_warp && elect_one()) bulk_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 256);
#undef R7C_STAMP
}

// ---------------------------------------------------------------------------------------------
// 6. fused producers, backward: one 64-channel row per 8 threads (16 bytes each), in place
//      dp = dw W_SCALE s_p (1 - s_p),  s_p = sigmoid(p)
//      dkk = -da + db s_q,  s_q = sigmoid(q);   dq = db kk s_q (1 - s_q)
//      du = (dkk - kk (kk . dkk)) / |u|,  kk = u / |u|
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
r7c_producer_bwd_kernel(const bf16* __restrict__ p, const bf16* __restrict__ u, const bf16* __restrict__ q,
                        bf16* dw_dp, bf16* da_du, bf16* db_dq, long long n_rows) {
  earlier_kernels_done();
  later_kernels_may_start();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long row = t >> 3;
  const bool live = row < n_rows;
  const long long off = (live ? row : 0) * 64 + 8 * (t & 7);
  float pv[8], uv[8], qv[8], dw[8], da[8], db[8];
  auto load8 = [&](const bf16* src, float* x) {
    const uint4 w4 = *reinterpret_cast<const uint4*>(src + off);
    const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
    for (int m = 0; m < 4; ++m) { x[2 * m] = bf16_lo(w[m]); x[2 * m + 1] = bf16_hi(w[m]); }
  };
  auto store8 = [&](bf16* dst, const float* x) {
    *reinterpret_cast<uint4*>(dst + off) = make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]),
                                                      pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
  };
  load8(p, pv); load8(u, uv); load8(q, qv); load8(dw_dp, dw); load8(da_du, da); load8(db_dq, db);
  float ss = 0.f;
#pragma unroll
  for (int x = 0; x < 8; ++x) ss += uv[x] * uv[x];
  ss += __shfl_xor_sync(0xffffffffu, ss, 1);
  ss += __shfl_xor_sync(0xffffffffu, ss, 2);
  ss += __shfl_xor_sync(0xffffffffu, ss, 4);
  const float inv = rsqrtf(fmaxf(ss, 1e-24f));      // 1 / max(|u|, 1e-12)
  float kk[8], dkk[8], dot = 0.f, dp[8], dq[8], du[8];
#pragma unroll
  for (int x = 0; x < 8; ++x) {
    const float sp = sigmoidf_(pv[x]), sq = sigmoidf_(qv[x]);
    kk[x] = uv[x] * inv;
    dp[x] = dw[x] * W_SCALE * sp * (1.f - sp);
    dkk[x] = -da[x] + db[x] * sq;
    dq[x] = db[x] * kk[x] * sq * (1.f - sq);
    dot += kk[x] * dkk[x];
  }
  dot += __shfl_xor_sync(0xffffffffu, dot, 1);
  dot += __shfl_xor_sync(0xffffffffu, dot, 2);
  dot += __shfl_xor_sync(0xffffffffu, dot, 4);
#pragma unroll
  for (int x = 0; x < 8; ++x) du[x] = (dkk[x] - kk[x] * dot) * inv;
  if (live) { store8(dw_dp, dp); store8(da_du, du); store8(db_dq, dq); }
}

}  // namespace r7c

int launch_rwkv7_producer_bwd(const void* p, const void* u, const void* q, void* dw_dp, void* da_du, void* db_dq,
                              long long n_rows, cudaStream_t st) {
  typedef __nv_bfloat16 bf16;
  ProfScope prof("r7c_producer_bwd_kernel", st);
  const long long threads = n_rows * 8;
  return launch(r7c::r7c_producer_bwd_kernel, (unsigned)((threads + 255) / 256), 256, 0, st, 1, (const bf16*)p, (const bf16*)u,
                (const bf16*)q, (bf16*)dw_dp, (bf16*)da_du, (bf16*)db_dq, n_rows);
}

int launch_rwkv7_chunked_bwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                             const float* h0, int n_state, const void* d_o, const float* d_ht,
                             void* dr, void* dw, void* dk, void* dv, void* da, void* db, float* d_h0,
                             void* workspace, int B, int Tn, int H, int head_first, bool kept, cudaStream_t st,
                             const int* seq_start, const int* seq_len, int T_total, bool fused, int phases) {
  using namespace r7c;
  if (fused && (seq_start || head_first)) return RWKVB200_E_UNSUPPORTED;
  typedef __nv_bfloat16 bf16;
  int e = RWKVB200_OK;
  if (!kept && (phases & PHASE_PREPARE)) {   // the workspace does not hold a forward pass yet: recompute it from the inputs
    e = launch_rwkv7_chunked_fwd(r, w, k, v, a, b, h0, n_state, nullptr, nullptr, workspace, B, Tn, H, head_first,
                                 true, st, seq_start, seq_len, T_total, fused);
    if (e) return e;
  }
  DeviceFacts dev;
  e = device_facts(&dev);
  if (e) return e;
  int* status = dev.status;
  CUtensorMap tmap_do, tmap_v, tmap_w, tmap_out[6];
  const SeqView sv{seq_start, seq_len, Tn};
  const int mapB = seq_start ? 1 : B, mapT = seq_start ? T_total : Tn;   // shape of the token tensors
  e = make_token_tensor_map(&tmap_do, d_o, mapB, mapT, H, head_first);
  if (e) return e;
  e = make_token_tensor_map(&tmap_v, v, mapB, mapT, H, head_first);
  if (e) return e;
  e = make_token_tensor_map(&tmap_w, w, mapB, mapT, H, head_first);
  if (e) return e;
  void* outs[6] = {dr, dw, dk, dv, da, db};
  for (int i = 0; i < 6; ++i) {
    e = make_token_tensor_map(&tmap_out[i], outs[i], mapB, mapT, H, head_first);
    if (e) return e;
  }
  const int NT = num_chunks(Tn);
  Workspace ws = carve(workspace, B, Tn, H, ALL_TILES);
  TokLayout lay(mapT, H, head_first);
  if (phases & PHASE_SCAN) {
    ProfScope prof("r7c_bwd_scan_kernel", st);
#define R7C_LAUNCH_BSCAN(THREADS, SMEM, ...)                                                                       \
    do {                                                                                                          \
      const int smem = (int)sizeof(SMEM) + 1024;                                                                  \
      if (allow_smem<__VA_ARGS__>(dev, smem)) return RWKVB200_E_CUDA;                                             \
      if (int rc = launch(__VA_ARGS__, B * H, THREADS, smem, st, 1, tmap_do, ws.tiles, ws.aux, (int)ALL_TILES,    \
                          d_ht, d_h0, sv, H, NT, status)) return rc;                                              \
    } while (0)
    const bool packed = seq_start != nullptr, alone = scans_alone(B, Tn, T_total, H, dev.sms, packed, SCAN_REVERSE);
    const bool sorted = packed && scans_sorted(B, Tn, T_total, H, dev.sms, alone);
    if (!alone) {      // two CTAs per SM
      if (sorted)      R7C_LAUNCH_BSCAN(256, BScanSmem, r7c_bwd_scan_kernel<true, true>);
      else if (packed) R7C_LAUNCH_BSCAN(256, BScanSmem, r7c_bwd_scan_kernel<true, false>);
      else             R7C_LAUNCH_BSCAN(256, BScanSmem, r7c_bwd_scan_kernel<false, false>);
    } else if (sorted) R7C_LAUNCH_BSCAN(BALONE_THREADS, BAloneSmem, r7c_bwd_scan_alone_kernel<true, true>);
    else if (packed)   R7C_LAUNCH_BSCAN(BALONE_THREADS, BAloneSmem, r7c_bwd_scan_alone_kernel<true, false>);
    else               R7C_LAUNCH_BSCAN(BALONE_THREADS, BAloneSmem, r7c_bwd_scan_alone_kernel<false, false>);
#undef R7C_LAUNCH_BSCAN
  }
  e = check_launch();
  if (e) return e;
  // Units the forward marked (decay beyond the range of the scaled operands, or a very short sequence): their
  // gradients come from the float32 recurrence instead.  Its state checkpoints (16 KB per 8 tokens = 128 KB per
  // chunk) go into the unit's own tile region of the workspace (as much per chunk), whose contents are void for
  // such a unit.
  static_assert(ALL_TILES * TILE_BYTES >= L / R7_CKPT * HS * HS * (int)sizeof(float), "checkpoints fit a unit's tiles");
  auto exact_units = [&]() -> int {
    const long long unit_floats = (long long)NT * ALL_TILES * TILE_BYTES / (long long)sizeof(float);
    float* ckpt = reinterpret_cast<float*>(ws.tiles);
    const UnitSel sel{ws.flags, seq_start, seq_len, unit_floats};
    return launch_rwkv7_rec_bwd(r, w, k, v, a, b, h0, n_state, d_o, d_ht, ckpt, dr, dw, dk, dv, da, db, d_h0, B, Tn, H,
                                head_first, st, sel, seq_start ? T_total : 0);
  };
  if (!(phases & PHASE_FINISH)) {
    // a scan-only call hands the gradient of the initial state to its caller (who passes it to the rank on the
    // left) before the token gradients exist: the marked units' share of it has to be exact already
    if ((phases & PHASE_SCAN) && !fused) return exact_units();
    return e;
  }
  {
    const int smem = (int)sizeof(FinalSmem);
    ProfScope prof("r7c_bwd_final_kernel", st);
    const int n_ch = B * H * NT;
    const int sms = dev.sms;
    const int grid = persistent_grid(n_ch, sms);
    // Blocks that come while the reverse scan runs out save the 2 us between two kernels, but where the CTAs walk over
    // many chunk-heads the kernel is slower for it (which the launch alone does; why was not isolated).  Forward and backward, us,
    // with and without, 32 heads: B 1, T 4096 318 and 316; B 2 444 and 441; B 4, T 1024, 48 heads 310 and 303; B 16, T 8192, 64 heads
    // 11760 and 11665; 8 packed sequences of up to 4096 tokens 952 and 941.
    const int early = n_ch <= grid ? 1 : 0;
#define R7C_LAUNCH_FINAL(P, F)                                                                                    \
    do {                                                                                                          \
      if (int rc = need_aligned_smem<r7c_bwd_final_kernel<P, F>>(dev)) return rc;                                 \
      if (allow_smem<r7c_bwd_final_kernel<P, F>>(dev, smem)) \
        return RWKVB200_E_CUDA;                                                                                   \
      if (int rc = launch(r7c_bwd_final_kernel<P, F>, grid, 256, smem, st, early, (const bf16*)w, tmap_w, tmap_do, tmap_v, ws.tiles, (int)ALL_TILES, \
          tmap_out[0], tmap_out[1], tmap_out[2], tmap_out[3], tmap_out[4], tmap_out[5], (bf16*)dr, (bf16*)dw,     \
          (bf16*)dk, (bf16*)dv, (bf16*)da, (bf16*)db, sv, WalkDims(H, NT, B, grid, !P), ws.list, lay, status, debug_stamp_buffer())) return rc; \
    } while (0)
    if (seq_start) R7C_LAUNCH_FINAL(true, false);
    else if (fused) R7C_LAUNCH_FINAL(false, true);
    else R7C_LAUNCH_FINAL(false, false);
#undef R7C_LAUNCH_FINAL
  }
  if (fused) {      // dw, da, db -> gradients of the pre-activations, in place
    e = check_launch();
    if (e) return e;
    return launch_rwkv7_producer_bwd(w, a, b, dw, da, db, (long long)B * Tn * H, st);
  }
  e = check_launch();
  if (e) return e;
  return exact_units();
}


}  // namespace rwkvb200
