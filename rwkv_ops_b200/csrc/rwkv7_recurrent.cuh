// The forward token-by-token recurrence of RWKV7 in float32 over 16 value rows of one (batch, head) unit, as a device
// function: the whole of rwkv7_rec_fwd_kernel, the forward part of the exact fallback's backward, and what the chunked
// forward scan runs for a unit whose decay left the range of its scaled operands.
//
//   d_t = exp(-exp(w_t));  sa_t = S_{t-1} a_t;  S_t = S_{t-1} diag(d_t) + sa_t b_t^T + v_t k_t^T;  o_t = S_t r_t
#pragma once

#include "common.cuh"

namespace rwkvb200 {
namespace r7rec {

constexpr int VS = 16;        // value rows per group of N threads
// A staged vector of N key channels is kept as segments of 16 with 4 floats of padding between them: the lanes
// of a quarter warp read the same 16 bytes of N/16 different segments, which 64 bytes apart would share banks.
__host__ __device__ constexpr int padk(int k) { return k + ((k >> 4) << 2); }
template <int N> __host__ __device__ constexpr int NP() { return N + N / 4; }

template <int N>
struct FwdSmem {
  static constexpr int TL = 8;                 // tokens staged per tile
  float tile[TL][5][NP<N>()];                  // r, d, k, a, b
  float vt[TL][VS];
  float ot[TL][VS];
};

template <typename T>
struct FwdArgs {
  const T *r, *w, *k, *v, *a, *b;
  long long base, st;           // this unit's first token, elements between tokens
  int Tn;
  const float* S0;              // the unit's initial state, or NULL
  T* o;                         // may be NULL
  float* ht;                    // the unit's final state, or NULL
  float* ckpt;                  // the unit's checkpoints (the state before every ckpt_every-th token), or NULL
  int ckpt_every;
};

// Called by N threads per slice `y` of 16 rows (tid < N), by NTHREADS threads of the block at once (which meet at barrier 1).
template <typename T, int N, int NTHREADS>
__device__ __noinline__ void fwd_rows(const FwdArgs<T>& A, FwdSmem<N>& sm, int y, int tid) {
  constexpr int TL = FwdSmem<N>::TL;
  constexpr int KSEG = N / 16;      // lanes per state row
  const int vl = tid / KSEG, kq = tid % KSEG;
  const int Tn = A.Tn;
  float S[16];
  if (A.S0) {
    const float* p = A.S0 + (long long)(y * VS + vl) * N + 16 * kq;
#pragma unroll
    for (int j = 0; j < 16; j += 4) {
      float4 f = *reinterpret_cast<const float4*>(p + j);
      S[j] = f.x; S[j + 1] = f.y; S[j + 2] = f.z; S[j + 3] = f.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) S[j] = 0.f;
  }

  // The inputs of a tile travel global memory -> registers -> shared memory, and the loads of tile i + 1 are
  // issued before the tokens of tile i are worked on: few warps share an SM here, so a load that is waited for where
  // it is issued costs its full latency every time.
  constexpr int PER = TL * 5 / 4;      // float4 per thread per tile: TL tokens x 5 vectors x N/4 quads over N threads
  float4 buf[PER], vbuf = make_float4(0.f, 0.f, 0.f, 0.f);
  const int quad = tid % (N / 4), rq = tid / (N / 4);      // this thread's quad of channels; its rows are rq + 4 m
  auto fetch = [&](int t0) {
    const int nt = min(TL, Tn - t0);
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int row = rq + 4 * m, tl = row / 5, which = row % 5;
      const T* src = which == 0 ? A.r : which == 1 ? A.w : which == 2 ? A.k : which == 3 ? A.a : A.b;
      buf[m] = tl < nt ? load4(src + A.base + (long long)(t0 + tl) * A.st + 4 * quad) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (tid < nt * 4)
      vbuf = load4(A.v + A.base + (long long)(t0 + (tid >> 2)) * A.st + y * VS + 4 * (tid & 3));
  };
  auto stash = [&]() {
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int row = rq + 4 * m, tl = row / 5, which = row % 5;
      float4 f = buf[m];
      if (which == 1) f = make_float4(decay_of(f.x), decay_of(f.y), decay_of(f.z), decay_of(f.w));
      *reinterpret_cast<float4*>(&sm.tile[tl][which][padk(4 * quad)]) = f;
    }
    if (tid < TL * 4) *reinterpret_cast<float4*>(&sm.vt[tid >> 2][4 * (tid & 3)]) = vbuf;
  };
  if (Tn > 0) fetch(0);
  for (int t0 = 0; t0 < Tn; t0 += TL) {
    const int nt = min(TL, Tn - t0);
    stash();
    asm volatile("bar.sync 1, %0;" ::"n"(NTHREADS) : "memory");
    if (t0 + TL < Tn) fetch(t0 + TL);

    for (int tl = 0; tl < nt; ++tl) {
      const int t = t0 + tl;
      if (A.ckpt && (t % A.ckpt_every) == 0) {
        float* p = A.ckpt + (((long long)(t / A.ckpt_every) * N) + (y * VS + vl)) * N + 16 * kq;
#pragma unroll
        for (int j = 0; j < 16; j += 4)
          *reinterpret_cast<float4*>(p + j) = make_float4(S[j], S[j + 1], S[j + 2], S[j + 3]);
      }
      const float* tr = &sm.tile[tl][0][20 * kq];
      const float* td = &sm.tile[tl][1][20 * kq];
      const float* tk = &sm.tile[tl][2][20 * kq];
      const float* ta = &sm.tile[tl][3][20 * kq];
      const float* tb = &sm.tile[tl][4][20 * kq];
      float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        s0 += S[j] * ta[j]; s1 += S[j + 1] * ta[j + 1]; s2 += S[j + 2] * ta[j + 2]; s3 += S[j + 3] * ta[j + 3];
      }
      float sa = (s0 + s1) + (s2 + s3);
#pragma unroll
      for (int m = 1; m < KSEG; m <<= 1) sa += __shfl_xor_sync(0xffffffffu, sa, m);
      const float vv = sm.vt[tl][vl];
      float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        S[j]     = S[j]     * td[j]     + sa * tb[j]     + vv * tk[j];
        S[j + 1] = S[j + 1] * td[j + 1] + sa * tb[j + 1] + vv * tk[j + 1];
        S[j + 2] = S[j + 2] * td[j + 2] + sa * tb[j + 2] + vv * tk[j + 2];
        S[j + 3] = S[j + 3] * td[j + 3] + sa * tb[j + 3] + vv * tk[j + 3];
        o0 += S[j] * tr[j]; o1 += S[j + 1] * tr[j + 1]; o2 += S[j + 2] * tr[j + 2]; o3 += S[j + 3] * tr[j + 3];
      }
      float oo = (o0 + o1) + (o2 + o3);
#pragma unroll
      for (int m = 1; m < KSEG; m <<= 1) oo += __shfl_xor_sync(0xffffffffu, oo, m);
      if (kq == 0) sm.ot[tl][vl] = oo;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(NTHREADS) : "memory");
    if (A.o && tid < nt * 4) {
      const int tl = tid >> 2, quad = tid & 3;
      store4(A.o + A.base + (long long)(t0 + tl) * A.st + y * VS + 4 * quad,
             *reinterpret_cast<const float4*>(&sm.ot[tl][4 * quad]));
    }
    // the next tile's staging writes tile/vt only after every thread has passed the barrier
    // above; ot is rewritten only after the next barrier pair
  }
  if (A.ht) {
    float* p = A.ht + (long long)(y * VS + vl) * N + 16 * kq;
#pragma unroll
    for (int j = 0; j < 16; j += 4)
      *reinterpret_cast<float4*>(p + j) = make_float4(S[j], S[j + 1], S[j + 2], S[j + 3]);
  }
}

}  // namespace r7rec
}  // namespace rwkvb200
