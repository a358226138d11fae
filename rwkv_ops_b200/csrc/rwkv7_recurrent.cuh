// The forward token-by-token recurrence of RWKV7 in float32 over value rows of one (batch, head) unit, as a device
// function: the whole of rwkv7_rec_fwd_kernel, the forward part of the exact fallback's backward, and what the chunked
// forward scan runs for a unit whose decay left the range of its scaled operands.
//
//   d_t = exp(-exp(w_t));  sa_t = S_{t-1} a_t;  S_t = S_{t-1} diag(d_t) + sa_t b_t^T + v_t k_t^T;  o_t = S_t r_t
#pragma once

#include "common.cuh"

namespace rwkvb200 {
namespace r7rec {

constexpr int VS = 16;        // value rows per CTA of the recurrent kernels
// A staged vector of N key channels is kept as segments of 16 with 4 floats of padding between them: the lanes
// of a quarter warp read the same 16 bytes of N/16 different segments, which 64 bytes apart would share banks.
__host__ __device__ constexpr int padk(int k) { return k + ((k >> 4) << 2); }
template <int N> __host__ __device__ constexpr int NP() { return N + N / 4; }

// `R` value rows of a unit worked on at once, `TL` tokens staged per tile
template <int N, int R, int TL>
struct FwdSmem {
  float tile[TL][5][NP<N>()];                  // r, d, k, a, b
  float vt[TL][R];
  float ot[TL][R];
};

template <typename T>
struct FwdArgs {
  const T *r, *w, *k, *v, *a, *b;
  long long base, st;           // this unit's first token, elements between tokens
  int Tn;
  const float* S0;              // the unit's initial state, or NULL
  T* o;                         // may be NULL
  float* ht;                    // the unit's final state, or NULL
  float* ckpt;                  // the unit's checkpoints (the state before every R7_CKPT-th token), or NULL
};

// Rows row0 .. row0 + R - 1, by NTHREADS threads (tid) that meet at barrier 1.  All of them stage; R / RPT * N / 16 of them hold
// RPT rows each.  The vectors of a token are read from shared memory once per thread, so two rows per thread halve what
// bounds a whole unit on one SM, and its tile is staged once for all 64 rows (16 units of 512 tokens out of range, forward call:
// 478 us with 64 threads and a tile of its own per 16 rows, 229 so; 512 units: 2055 and 878).
template <typename T, int N, int R, int RPT, int TL, int NTHREADS>
__device__ __forceinline__ void fwd_rows(const FwdArgs<T>& A, FwdSmem<N, R, TL>& sm, int row0, int tid) {
  constexpr int KSEG = N / 16;                 // lanes per state row
  constexpr int NC = R / RPT * KSEG;           // threads that hold rows
  static_assert(NC <= NTHREADS && NC % 32 == 0, "whole warps hold rows");
  const int vl = tid / KSEG, kq = tid % KSEG;  // rows vl + i R / RPT
  const int Tn = A.Tn;
  const bool rows = NC == NTHREADS || tid < NC;
  float S[RPT][16];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const float* p = A.S0 + (long long)(row0 + vl + i * (R / RPT)) * N + 16 * kq;
#pragma unroll
    for (int j = 0; j < 16; j += 4) {
      const float4 f = rows && A.S0 ? *reinterpret_cast<const float4*>(p + j) : make_float4(0.f, 0.f, 0.f, 0.f);
      S[i][j] = f.x; S[i][j + 1] = f.y; S[i][j + 2] = f.z; S[i][j + 3] = f.w;
    }
  }
  auto put_state = [&](float* to) {
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      float* p = to + (long long)(row0 + vl + i * (R / RPT)) * N + 16 * kq;
#pragma unroll
      for (int j = 0; j < 16; j += 4)
        *reinterpret_cast<float4*>(p + j) = make_float4(S[i][j], S[i][j + 1], S[i][j + 2], S[i][j + 3]);
    }
  };

  // The inputs of a tile travel global memory -> registers -> shared memory, and the loads of tile i + 1 are
  // issued before the tokens of tile i are worked on: few warps share an SM here, so a load that is waited for where
  // it is issued costs its full latency every time.
  constexpr int QUADS = TL * 5 * (N / 4), PER = (QUADS + NTHREADS - 1) / NTHREADS;      // float4 per thread and tile
  constexpr int VQUADS = TL * R / 4;
  static_assert(VQUADS <= NTHREADS, "one quad of v (and of o) per thread");
  float4 buf[PER], vbuf = make_float4(0.f, 0.f, 0.f, 0.f);
  auto fetch = [&](int t0) {
    const int nt = min(TL, Tn - t0);
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int e = tid + NTHREADS * m, row = e / (N / 4), tl = row / 5, which = row % 5;
      const T* src = which == 0 ? A.r : which == 1 ? A.w : which == 2 ? A.k : which == 3 ? A.a : A.b;
      buf[m] = tl < nt ? load4(src + A.base + (long long)(t0 + tl) * A.st + 4 * (e % (N / 4))) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (tid < nt * (R / 4))
      vbuf = load4(A.v + A.base + (long long)(t0 + tid / (R / 4)) * A.st + row0 + 4 * (tid % (R / 4)));
  };
  auto stash = [&]() {
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int e = tid + NTHREADS * m, row = e / (N / 4), tl = row / 5, which = row % 5;
      if (QUADS % NTHREADS && e >= QUADS) break;
      float4 f = buf[m];
      if (which == 1) f = make_float4(decay_of(f.x), decay_of(f.y), decay_of(f.z), decay_of(f.w));
      *reinterpret_cast<float4*>(&sm.tile[tl][which][padk(4 * (e % (N / 4)))]) = f;
    }
    if (tid < VQUADS) *reinterpret_cast<float4*>(&sm.vt[tid / (R / 4)][4 * (tid % (R / 4))]) = vbuf;
  };
  if (Tn > 0) fetch(0);
  for (int t0 = 0; t0 < Tn; t0 += TL) {
    const int nt = min(TL, Tn - t0);
    stash();
    asm volatile("bar.sync 1, %0;" ::"n"(NTHREADS) : "memory");
    if (t0 + TL < Tn) fetch(t0 + TL);

    for (int tl = 0; rows && tl < nt; ++tl) {
      if (A.ckpt && (t0 + tl) % R7_CKPT == 0) put_state(A.ckpt + (long long)((t0 + tl) / R7_CKPT) * N * N);
      const float* tr = &sm.tile[tl][0][20 * kq];
      const float* td = &sm.tile[tl][1][20 * kq];
      const float* tk = &sm.tile[tl][2][20 * kq];
      const float* ta = &sm.tile[tl][3][20 * kq];
      const float* tb = &sm.tile[tl][4][20 * kq];
      float sa[RPT], oo[RPT], vv[RPT];
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          s0 += S[i][j] * ta[j]; s1 += S[i][j + 1] * ta[j + 1]; s2 += S[i][j + 2] * ta[j + 2]; s3 += S[i][j + 3] * ta[j + 3];
        }
        sa[i] = (s0 + s1) + (s2 + s3);
        vv[i] = sm.vt[tl][vl + i * (R / RPT)];
      }
#pragma unroll
      for (int m = 1; m < KSEG; m <<= 1) {
#pragma unroll
        for (int i = 0; i < RPT; ++i) sa[i] += __shfl_xor_sync(0xffffffffu, sa[i], m);
      }
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          S[i][j]     = S[i][j]     * td[j]     + sa[i] * tb[j]     + vv[i] * tk[j];
          S[i][j + 1] = S[i][j + 1] * td[j + 1] + sa[i] * tb[j + 1] + vv[i] * tk[j + 1];
          S[i][j + 2] = S[i][j + 2] * td[j + 2] + sa[i] * tb[j + 2] + vv[i] * tk[j + 2];
          S[i][j + 3] = S[i][j + 3] * td[j + 3] + sa[i] * tb[j + 3] + vv[i] * tk[j + 3];
          o0 += S[i][j] * tr[j]; o1 += S[i][j + 1] * tr[j + 1]; o2 += S[i][j + 2] * tr[j + 2]; o3 += S[i][j + 3] * tr[j + 3];
        }
        oo[i] = (o0 + o1) + (o2 + o3);
      }
#pragma unroll
      for (int m = 1; m < KSEG; m <<= 1) {
#pragma unroll
        for (int i = 0; i < RPT; ++i) oo[i] += __shfl_xor_sync(0xffffffffu, oo[i], m);
      }
#pragma unroll
      for (int i = 0; i < RPT; ++i)
        if (kq == 0) sm.ot[tl][vl + i * (R / RPT)] = oo[i];
    }
    asm volatile("bar.sync 1, %0;" ::"n"(NTHREADS) : "memory");
    if (A.o && tid < nt * (R / 4))
      store4(A.o + A.base + (long long)(t0 + tid / (R / 4)) * A.st + row0 + 4 * (tid % (R / 4)),
             *reinterpret_cast<const float4*>(&sm.ot[tid / (R / 4)][4 * (tid % (R / 4))]));
    // the next tile's staging writes tile/vt only after every thread has passed the barrier
    // above; ot is rewritten only after the next barrier pair
  }
  if (A.ht && rows) put_state(A.ht);
}

}  // namespace r7rec
}  // namespace rwkvb200
