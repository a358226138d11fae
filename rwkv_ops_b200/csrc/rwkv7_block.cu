// RWKV7 generalized delta rule in float32 on the CUDA cores, eight tokens at a time (forward and backward).
//
// The exact path of the reference's native operator (rwkv_ops/rwkv7_kernel/native_keras_op.py:80-91),
//
//   d_t = exp(-exp(w_t));  sa_t = S_{t-1} a_t;  S_t = S_{t-1} diag(d_t) + sa_t b_t^T + v_t k_t^T;  o_t = S_t r_t,
//
// for float32 and float16 tokens and for head size 128.  Token by token its time is a serial chain: two
// reductions over the key channels per token, 930 cycles forward and 2300 backward, whatever the size.  Written out
// over a block of W tokens that chain shrinks to one reduction per block.  With S the state before the block, D_j the
// product of the decays of tokens 0..j of the block and x_j^(i) = x_j times the decays in between,
//
//   sa_j = S (D_{j-1} a_j) + sum_{i<j} sa_i A_ab(j,i) + v_i A_ak(j,i)      A_ab(j,i) = b_i^(j-1) . a_j, ...
//   o_j  = S (D_j r_j)     + sum_{i<=j} sa_i A_qb(j,i) + v_i A_qk(j,i)     A_qb(j,i) = b_i^(j) . r_j, ...
//   S'   = S D_{W-1}       + sum_i sa_i b_i^(W-1) + v_i k_i^(W-1)
//
// and the scalars A do not depend on the state.  Substituting the first line into itself and into the second gives
// sa_j = S x_j + sum_l xv(j,l) v_l and o_j = S y_j + sum_l yv(j,l) v_l, with vectors x, y and scalars xv, yv that are
// prepared ahead of the state.  Every decay factor is a product of factors <= 1, so nothing over- or underflows that
// the token-by-token form would keep, and all arithmetic is float32.
//
// The gradient G of the state runs backward in time through the same equations with the roles exchanged
// (sa -> dsa, o -> dv, v -> do; a <-> b, r <-> k, every A transposed): the same code serves both directions.  The other
// five gradients do not feed the chain.  A kernel of their own computes them for every 16 tokens at once, from the states
// and state gradients that the two sweeps leave at those boundaries (as much memory as a state every 8 tokens).  The forward
// of a training call leaves its states for the backward; a backward without them sweeps forward first.
//
// B 2, T 1024, 16 heads, float32, in kernels: token by token forward 500 us, backward 1740; 106 (20 of preparation) and 235 (24 of
// preparation, 84 sweep, 127 gradients) here.
#include <type_traits>

#include "common.cuh"
#include "tc.cuh"

namespace rwkvb200 {

namespace {

constexpr int W = 8;          // tokens per block
constexpr int RV = 16;        // value rows per CTA
constexpr int GT = 2 * W;     // tokens per work item of the gradient kernel, and between two checkpoints

// packed pairs of float32
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
struct Quad { f32x2 lo, hi; };      // four consecutive floats
__device__ __forceinline__ Quad quad_of(float4 f) { return Quad{pack2(f.x, f.y), pack2(f.z, f.w)}; }
__device__ __forceinline__ Quad lds4(const float* p) { return quad_of(*reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float sum2(f32x2 v) { const float2 f = unpack2(v); return f.x + f.y; }

// A warp's 16-byte reads of shared memory take four cycles, but two where lanes that differ in bit 0 or bit 1 read the same
// address (measured: sharing along the higher bits saves nothing).  So in the kernels below the lanes that share an operand
// differ in one of these two bits, and where two operands are shared, each has one of them.

// Sum CNT values over the lanes that differ in the bits of MASK, MASK/2, .., LAST; the values are shared out on the
// way: a lane whose bit is set goes on with the upper half.
template <int CNT, int MASK, int LAST, int M>
__device__ __forceinline__ void reduce_scatter(float (&v)[M], int lane) {
  const bool up = lane & MASK;
#pragma unroll
  for (int k = 0; k < CNT / 2; ++k) {
    const float send = up ? v[k] : v[k + CNT / 2], keep = up ? v[k + CNT / 2] : v[k];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, MASK);
  }
  if constexpr (MASK > LAST) reduce_scatter<CNT / 2, MASK / 2, LAST>(v, lane);
}

__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }
// 16 bytes into shared memory, zeros when !live (the address must be valid all the same)
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <typename T> struct Vecs { const T* p[5]; };      // r, w, k, a, b
enum { VR = 0, VW = 1, VK = 2, VA = 3, VB = 4 };

// ---------------------------------------------------------------------------------------------
// the sweep over the blocks: forward (S, sa, o) or backward (G, dsa, dv)
// ---------------------------------------------------------------------------------------------
// A CTA owns 16 value rows of one (batch, head) unit.  Its state warps hold them in registers (ROWS rows and 8 columns to a
// lane, N/8 lanes to a row) and take them through the blocks; what a block needs besides the state, its stage, is prepared ahead
// of them.  In processing order p (time forward, or reversed):
template <int N, int VR_>
struct Stage {
  float x[W][N], y[W][N];       // sa_p = S x_p + xv[p][.] v ;  o_p = S y_p + yv[p][.] v
  float u1[W][N], u2[W][N];     // S' = S diag(d) + sum_p sa_p u1_p + v_p u2_p
  float d[N];
  float xv[W][W], yv[W][W];
  float vt[VR_][W];             // the tokens' v, for all N or for a CTA's RV rows
};
template <int N> constexpr uint32_t COMMON_BYTES = sizeof(Stage<N, RV>) - RV * W * sizeof(float);      // a stage without vt
constexpr uint32_t SLICE_BYTES = RV * W * sizeof(float);                                               // a CTA's rows of vt

template <int N>
struct Scalars {
  float d[W][N];                                      // decays
  float sx[W][W], sxv[W][W], sy[W][W], syv[W][W];     // the scalars A, processing order; never-written entries stay 0
};
// The preparation of one block by a group of N threads (thread q of them), in steps with a barrier of the group before each.
template <typename T, int N, bool BWD>
struct Preparer {
  static constexpr int NL = N / 4, HELD = 32 / NL;      // lanes per pair of source tokens
  Scalars<N>& sc;
  const int q, pi, gq, lane;
  float* dst[HELD];

  // The scalars: a thread takes four channels of the source tokens pi and 7 - pi (nine (source, later token) pairs
  // whatever pi, so all warps have the same work), 32 sums that N/4 lanes then reduce and share out.
  __device__ __forceinline__ Preparer(Scalars<N>& sc_, int q_) : sc(sc_), q(q_), pi(q_ / NL), gq(q_ % NL), lane(q_ & 31) {
    for (int e = q; e < 4 * W * W; e += N) (&sc.sx[0][0])[e] = 0.f;
#pragma unroll
    for (int h = 0; h < HELD; ++h) {
      const int e = gq * HELD + h;
      const int kind = e < 9 ? 0 : e < 18 ? 1 : e < 25 ? 2 : 3;           // A_qb, A_qk, A_ab, A_ak
      const int x = e - (kind == 0 ? 0 : kind == 1 ? 9 : kind == 2 ? 17 : 24);
      const int i = x <= 7 - pi ? pi : 7 - pi, j = x <= 7 - pi ? pi + x : 7 - pi + (8 - x);
      float (*m)[W] = BWD ? (kind == 0 ? sc.sxv : kind == 1 ? sc.syv : kind == 2 ? sc.sx : sc.sy)
                          : (kind == 0 ? sc.sy : kind == 1 ? sc.syv : kind == 2 ? sc.sx : sc.sxv);
      dst[h] = BWD ? &m[W - 1 - i][W - 1 - j] : &m[j][i];
    }
  }
  // the decays, 1 for tokens past the end
  __device__ __forceinline__ void decays(const T (*raw)[W][N], int n_live) {
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int t = 4 * m + q / NL, c = 4 * (q % NL);
      const float4 f = load4_shared(&raw[VW][t][c]);
      *reinterpret_cast<float4*>(&sc.d[t][c]) = t < n_live ? make_float4(decay_of(f.x), decay_of(f.y), decay_of(f.z), decay_of(f.w))
                                                           : make_float4(1.f, 1.f, 1.f, 1.f);
    }
  }
  __device__ __forceinline__ void scalars(const T (*raw)[W][N]) {
    float s[32];
#pragma unroll
    for (int e = 0; e < 32; ++e) s[e] = 0.f;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int i = half ? 7 - pi : pi, last = half ? pi : 7 - pi;      // later tokens i .. i + last
      Quad pb = quad_of(load4_shared(&raw[VB][i][4 * gq])), pk = quad_of(load4_shared(&raw[VK][i][4 * gq]));
#pragma unroll
      for (int x = 0; x < (half ? 4 : 8); ++x) {
        if (x > last) break;
        const int j = i + x, at = half ? 8 - x : x;
        if (x > 0) {
          const Quad aj = quad_of(load4_shared(&raw[VA][j][4 * gq])), dj = lds4(&sc.d[j][4 * gq]);
          s[17 + at] = sum2(fma2(pb.hi, aj.hi, mul2(pb.lo, aj.lo)));
          s[24 + at] = sum2(fma2(pk.hi, aj.hi, mul2(pk.lo, aj.lo)));
          pb.lo = mul2(pb.lo, dj.lo); pb.hi = mul2(pb.hi, dj.hi);
          pk.lo = mul2(pk.lo, dj.lo); pk.hi = mul2(pk.hi, dj.hi);
        }
        const Quad rj = quad_of(load4_shared(&raw[VR][j][4 * gq]));
        s[at] = sum2(fma2(pb.hi, rj.hi, mul2(pb.lo, rj.lo)));
        s[9 + at] = sum2(fma2(pk.hi, rj.hi, mul2(pk.lo, rj.lo)));
      }
    }
    __syncwarp();
    reduce_scatter<32, NL / 2, 1>(s, lane);
#pragma unroll
    for (int h = 0; h < HELD; ++h) *dst[h] = s[h];
  }
  // x and y by substitution, in processing order: of one channel, or of one column of A_ak and A_qk
  __device__ __forceinline__ void solve(float (&xs)[W], float (&ys_)[W]) {
#pragma unroll
    for (int p = 0; p < W; ++p) {
      float m[W];
#pragma unroll
      for (int i = 0; i < p; i += 4) *reinterpret_cast<float4*>(&m[i]) = *reinterpret_cast<const float4*>(&sc.sx[p][i]);
#pragma unroll
      for (int i = 0; i < p; ++i) xs[p] += m[i] * xs[i];
    }
#pragma unroll
    for (int p = 0; p < W; ++p) {
      float m[W];
#pragma unroll
      for (int i = 0; i <= p; i += 4) *reinterpret_cast<float4*>(&m[i]) = *reinterpret_cast<const float4*>(&sc.sy[p][i]);
#pragma unroll
      for (int i = 0; i <= p; ++i) ys_[p] += m[i] * xs[i];
    }
  }
  template <int VROWS>
  __device__ __forceinline__ void write(const T (*raw)[W][N], Stage<N, VROWS>& st) {      // all but vt; thread q: channel q
    {
      float xs[W], ys_[W], dd[W];
      float run = 1.f;
#pragma unroll
      for (int p = 0; p < W; ++p) {
        const int t = BWD ? W - 1 - p : p;
        dd[p] = sc.d[t][q];
        xs[p] = run * to_f32(raw[BWD ? VB : VA][t][q]);
        if (!BWD) run *= dd[p];
        ys_[p] = run * to_f32(raw[BWD ? VK : VR][t][q]);
        if (BWD) run *= dd[p];
      }
      st.d[q] = run;
      run = 1.f;
#pragma unroll
      for (int p = W - 1; p >= 0; --p) {
        const int t = BWD ? W - 1 - p : p;
        st.u1[p][q] = run * to_f32(raw[BWD ? VA : VB][t][q]);
        if (BWD) run *= dd[p];
        st.u2[p][q] = run * to_f32(raw[BWD ? VR : VK][t][q]);
        if (!BWD) run *= dd[p];
      }
      solve(xs, ys_);
#pragma unroll
      for (int p = 0; p < W; ++p) { st.x[p][q] = xs[p]; st.y[p][q] = ys_[p]; }
    }
    if (q < W) {
      float xs[W], ys_[W];
#pragma unroll
      for (int p = 0; p < W; ++p) { xs[p] = sc.sxv[p][q]; ys_[p] = sc.syv[p][q]; }
      solve(xs, ys_);
#pragma unroll
      for (int p = 0; p < W; ++p) { st.xv[p][q] = xs[p]; st.yv[p][q] = ys_[p]; }
    }
  }
};

// The state warps' part of one block: the rows' S in registers through one stage.
template <int N, int ROWS>
struct StateRows {
  // N/8 lanes per row; the lanes that read the same part of a vector are neighbours (see the note on 16-byte reads above)
  static constexpr int RG = 256 / N;           // groups of rows in a warp
  const int lane, r0, kq, jl, c0, c1;          // first row; this thread's columns: two quads of ROWS rows; its token
  Quad S[ROWS][2];

  __device__ __forceinline__ StateRows(int tid)
      : lane(tid & 31), r0(ROWS * (tid / 32 * RG + tid % RG)), kq((tid & 31) / RG), jl(kq & 7), c0(4 * kq), c1(N / 2 + 4 * kq) {}
  __device__ __forceinline__ void get(const float* p) {      // p: the CTA's first row, or nullptr
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      S[i][0] = S[i][1] = Quad{0ull, 0ull};
      if (p) {
        S[i][0] = quad_of(*reinterpret_cast<const float4*>(p + (long long)(r0 + i) * N + c0));
        S[i][1] = quad_of(*reinterpret_cast<const float4*>(p + (long long)(r0 + i) * N + c1));
      }
    }
  }
  __device__ __forceinline__ void put(float* p) const {
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float2 a = unpack2(S[i][h].lo), b = unpack2(S[i][h].hi);
        *reinterpret_cast<float4*>(p + (long long)(r0 + i) * N + (h ? c1 : c0)) = make_float4(a.x, a.y, b.x, b.y);
      }
    }
  }
  // S row . vector, for all rows and tokens: dots[ROWS p + i]
  __device__ __forceinline__ void dots(const float (*vec)[N], float* out) const {
    Quad xa[W], xb[W];
#pragma unroll
    for (int p = 0; p < W; ++p) { xa[p] = lds4(&vec[p][c0]); xb[p] = lds4(&vec[p][c1]); }
#pragma unroll
    for (int p = 0; p < W; ++p)
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
        out[ROWS * p + i] = sum2(fma2(S[i][1].hi, xb[p].hi, fma2(S[i][1].lo, xb[p].lo, fma2(S[i][0].hi, xa[p].hi, mul2(S[i][0].lo, xa[p].lo)))));
  }
  __device__ __forceinline__ void add_outer(const Quad& ua, const Quad& ub, int i, float f) {
    const f32x2 s = pack2(f, f);
    S[i][0].lo = fma2(s, ua.lo, S[i][0].lo); S[i][0].hi = fma2(s, ua.hi, S[i][0].hi);
    S[i][1].lo = fma2(s, ub.lo, S[i][1].lo); S[i][1].hi = fma2(s, ub.hi, S[i][1].hi);
  }
  // Leaves token jl's output of the thread's rows in oo: in every lane (N = 64: 8 lanes to a row), or in lanes 8-15 of a row.
  __device__ __forceinline__ void step(const Stage<N, RV>& st, float (&oo)[ROWS]) {
    float ax[(N == 64 ? 1 : 2) * W * ROWS], ay[W * ROWS];
    dots(st.x, ax);
    float sa[ROWS];
    if constexpr (N == 64) {
      reduce_scatter<W * ROWS, 4 * RG, RG>(ax, lane);
      dots(st.y, ay);
      reduce_scatter<W * ROWS, 4 * RG, RG>(ay, lane);
#pragma unroll
      for (int i = 0; i < ROWS; ++i) { sa[i] = ax[i]; oo[i] = ay[i]; }
    } else {
      dots(st.y, ax + W * ROWS);
      reduce_scatter<2 * W * ROWS, 8 * RG, RG>(ax, lane);
#pragma unroll
      for (int i = 0; i < ROWS; ++i) sa[i] = oo[i] = ax[i];
    }
    {
      const Quad da = lds4(&st.d[c0]), db = lds4(&st.d[c1]);
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        S[i][0].lo = mul2(S[i][0].lo, da.lo); S[i][0].hi = mul2(S[i][0].hi, da.hi);
        S[i][1].lo = mul2(S[i][1].lo, db.lo); S[i][1].hi = mul2(S[i][1].hi, db.hi);
      }
    }
#pragma unroll
    for (int l = 0; l < W; l += 4) {
      const float4 x = *reinterpret_cast<const float4*>(&st.xv[jl][l]), y = *reinterpret_cast<const float4*>(&st.yv[jl][l]);
      // the factors of tokens after jl are 0, but 0 times an infinity or NaN is not: their v counts as 0 as well
      const bool u0 = l <= jl, u1 = l + 1 <= jl, u2 = l + 2 <= jl, u3 = l + 3 <= jl;
      float vv[ROWS][4];
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        const float4 f = *reinterpret_cast<const float4*>(&st.vt[r0 + i][l]);
        vv[i][0] = f.x; vv[i][1] = f.y; vv[i][2] = f.z; vv[i][3] = f.w;
        const float4 m = make_float4(u0 ? f.x : 0.f, u1 ? f.y : 0.f, u2 ? f.z : 0.f, u3 ? f.w : 0.f);
        sa[i] += x.x * m.x + x.y * m.y + (x.z * m.z + x.w * m.w);
        oo[i] += y.x * m.x + y.y * m.y + (y.z * m.z + y.w * m.w);
      }
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const Quad ua = lds4(&st.u2[l + p][c0]), ub = lds4(&st.u2[l + p][c1]);
#pragma unroll
        for (int i = 0; i < ROWS; ++i) add_outer(ua, ub, i, vv[i][p]);
      }
    }
#pragma unroll
    for (int p = 0; p < W; ++p) {
      const Quad ua = lds4(&st.u1[p][c0]), ub = lds4(&st.u1[p][c1]);
#pragma unroll
      for (int i = 0; i < ROWS; ++i) add_outer(ua, ub, i, __shfl_sync(0xffffffffu, sa[i], lane % RG + RG * p));
    }
  }
  template <typename T>
  __device__ __forceinline__ void put_out(T* p, const float (&oo)[ROWS]) const {      // p: token jl's value channels of the CTA's rows
    if (N == 64 || kq >= 8) {
#pragma unroll
      for (int i = 0; i < ROWS; ++i) p[r0 + i] = from_f32<T>(oo[i]);
    }
  }
};
// where block n's state is kept: forward, the state before every GT tokens but the first; backward, the gradient after them, but
// the last; nullptr: nowhere
template <int N, bool BWD>
__device__ __forceinline__ float* state_slot(float* ckpt, int unit, int NG, int n) {
  const int m = n >> 1;
  if (!BWD && (n & 1) == 0 && m > 0) return ckpt + ((long long)unit * (NG - 1) + m - 1) * N * N;
  if (BWD && (n & 1) == 1 && m < NG - 1) return ckpt + ((long long)unit * (NG - 1) + m) * N * N;
  return nullptr;
}

// ---- blocks prepared by the CTA itself, for calls of a few blocks, or without workspace
// ROWS = 1 (2 at N = 128), four state warps, where a CTA has its SM to itself: the instructions of a warp are then what a
// block takes, and a warp of twice the rows needs 131 us per sweep where this takes 108 (B 2, T 1024, 16 heads).  ROWS = 2
// where CTAs share an SM, whose shared memory they fill: B 16, T 512, 16 heads, forward 332 us against 360.
template <typename T, int N>
struct Group {
  Stage<N, RV> stage;
  Scalars<N> scalars;
  T raw[2][5][W][N];            // the block at work and the next one (requested while the first is worked on)
  T rawv[2][W][RV];
};
// Groups that prepare blocks: as many as keep up with the state warps where a CTA has its SM to itself.  A group takes 34 KB of
// shared memory (60 at N = 128), so where there are more CTAs than SMs fewer of them let two or three CTAs share an SM and fill
// each other's waits: B 64, T 32, 32 heads, forward 329 us with four groups, 196 with two (B 16, T 1024, 64 heads: 3385 and 2765);
// N = 128, B 16, T 512, 16 heads: 1519 us with three, 1176 with one.  At 148 CTAs two groups lose, 48 us against 42 (T 300),
// and so they do in float16, where two CTAs of four groups fit an SM as it is (B 16, T 512, 16 heads: 339 us and 364).
template <int N> constexpr int FEW_CTAS = N == 64 ? 4 : 3;
template <typename T, int N> constexpr int MANY_CTAS = N == 128 ? 1 : sizeof(T) == 4 ? 2 : FEW_CTAS<N>;
template <int N> constexpr int FEW_CTAS_ROWS = N / 64;
constexpr int MANY_CTAS_ROWS = 2;
template <int N, int ROWS> constexpr int state_threads() { return RV / ROWS * N / 8; }

template <typename T, int N, bool BWD, int GROUPS, int ROWS>
__global__ void __launch_bounds__(state_threads<N, ROWS>() + N * GROUPS)
r7_sweep_inline_kernel(Vecs<T> in, const T* __restrict__ v, const float* __restrict__ s_in, int n_state,
                       T* __restrict__ out, float* __restrict__ s_out, float* __restrict__ ckpt, int Tn, int H, TokLayout lay) {
  constexpr int NCONS = state_threads<N, ROWS>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Group<T, N>* const group = reinterpret_cast<Group<T, N>*>(smem_raw);
  earlier_kernels_done();
  later_kernels_may_start();
  const int unit = blockIdx.x, ys = blockIdx.y, tid = threadIdx.x;
  const int bi = unit / H, hi = unit % H;
  const long long base = bi * lay.sb + hi * lay.sh;
  const int NB = (Tn + W - 1) / W;
  constexpr int FULL = 1 + GROUPS, EMPTY = 1 + 2 * GROUPS;      // named barriers: 1.. within a group, then these
  const long long rows = (long long)ys * RV * N;                // of the CTA's first row in a state

  if (tid < NCONS) {
    // ---- state warps
    const int NG = (Tn + GT - 1) / GT;
    StateRows<N, ROWS> S(tid);
    S.get(s_in && n_state > 0 ? s_in + (long long)(n_state == 1 ? hi : unit) * N * N + rows : nullptr);
    for (int idx = 0, g = 0; idx < NB; ++idx, g = g + 1 == GROUPS ? 0 : g + 1) {
      const int n = BWD ? NB - 1 - idx : idx;
      if (ckpt)
        if (float* p = state_slot<N, BWD>(ckpt, unit, NG, n)) S.put(p + rows);
      bar_sync(FULL + g, NCONS + N);
      float oo[ROWS];
      S.step(group[g].stage, oo);
      if (idx + GROUPS < NB) bar_arrive(EMPTY + g, NCONS + N);
      const int t = n * W + (BWD ? W - 1 - S.jl : S.jl);
      if (out && t < Tn) S.put_out(out + base + (long long)t * lay.st + ys * RV, oo);
    }
    if (s_out) S.put(s_out + (long long)unit * N * N + rows);
    return;
  }

  // ---- preparing groups
  const int g = (tid - NCONS) / N, q = (tid - NCONS) % N;
  Group<T, N>& pr = group[g];
  constexpr int EPC = 16 / sizeof(T), CPR = N / EPC, VPR = RV / EPC;     // elements per 16 bytes; copies per token row

  auto request = [&](int idx) {
    if (idx < NB) {
      const int t0 = (BWD ? NB - 1 - idx : idx) * W, buf = (idx / GROUPS) & 1;
#pragma unroll
      for (int m = 0; m < W * CPR / N; ++m) {
        const int e = q + N * m, row = e / CPR, ch = e % CPR;
        const bool live = t0 + row < Tn;
        const long long off = base + (live ? (long long)(t0 + row) * lay.st : 0) + ch * EPC;
#pragma unroll
        for (int i = 0; i < 5; ++i) cp_async16(&pr.raw[buf][i][row][ch * EPC], in.p[i] + off, live);
      }
      if (q < W * VPR) {
        const int row = q / VPR, ch = q % VPR;
        const bool live = t0 + row < Tn;
        cp_async16(&pr.rawv[buf][row][ch * EPC], v + base + (live ? (long long)(t0 + row) * lay.st : 0) + ys * RV + ch * EPC, live);
      }
    }
    cp_async_commit();
  };
  request(g);
  Preparer<T, N, BWD> prep(pr.scalars, q);
  for (int idx = g; idx < NB; idx += GROUPS) {
    const int t0 = (BWD ? NB - 1 - idx : idx) * W, buf = (idx / GROUPS) & 1;
    cp_async_wait();
    bar_sync(1 + g, N);             // the block's tokens are here, and the last block's scalars and decays have been read
    request(idx + GROUPS);
    prep.decays(pr.raw[buf], Tn - t0);
    bar_sync(1 + g, N);
    prep.scalars(pr.raw[buf]);
    if (idx >= GROUPS) bar_sync(EMPTY + g, NCONS + N);      // the stage has been read (and the group's scalars are written)
    else               bar_sync(1 + g, N);
    prep.write(pr.raw[buf], pr.stage);
    for (int e = q; e < RV * W; e += N) {
      const int p = e % W, row = e / W;
      pr.stage.vt[row][p] = to_f32(pr.rawv[buf][BWD ? W - 1 - p : p][row]);
    }
    bar_arrive(FULL + g, NCONS + N);
  }
  cp_async_wait();
}

// ---- blocks prepared by a kernel of their own, once for all the CTAs of a unit
// Prepared inside the sweep, a block is prepared N/16 times, and that is 60 % of the sweep's instructions and most of its
// shared-memory traffic.  Here the stages go through memory, 11 KB per block and unit (L2, where they fit), and a sweep's CTAs
// are state warps and one that fetches stages.  B 2, T 1024, 16 heads: 20 us and 80 per sweep against 105; B 16, T 512, 16 heads,
// forward 332 -> 223 us; head size 128 1170 -> 660.  What bounds the sweep now with one CTA per SM: 414 instructions per block and
// warp, one warp to a scheduler, and shared memory (682 of 1190 cycles).
template <typename T, int N>
struct PrepareSmem {
  Scalars<N> scalars;
  T raw[5][W][N];
};
constexpr int PREPARE_THREADS = 256;

template <typename T, int N, bool BWD>
__global__ void __launch_bounds__(PREPARE_THREADS)
r7_prepare_kernel(Vecs<T> in, const T* __restrict__ v, Stage<N, N>* __restrict__ stages, int Tn, int H, int unit0, int idx0, int nb,
                  int n_items, TokLayout lay) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int g = threadIdx.x / N, q = threadIdx.x % N, item = blockIdx.x * (PREPARE_THREADS / N) + g;
  PrepareSmem<T, N>& sm = reinterpret_cast<PrepareSmem<T, N>*>(smem_raw)[g];
  earlier_kernels_done();
  later_kernels_may_start();
  if (item >= n_items) return;      // the whole group
  const int unit = unit0 + item / nb, idx = idx0 + item % nb, NB = (Tn + W - 1) / W;
  const int t0 = (BWD ? NB - 1 - idx : idx) * W;
  const long long base = unit / H * lay.sb + unit % H * lay.sh;
  constexpr int EPC = 16 / sizeof(T), CPR = N / EPC;
#pragma unroll
  for (int m = 0; m < W * CPR / N; ++m) {
    const int e = q + N * m, row = e / CPR, ch = e % CPR;
    const bool live = t0 + row < Tn;
    const long long off = base + (live ? (long long)(t0 + row) * lay.st : 0) + ch * EPC;
#pragma unroll
    for (int i = 0; i < 5; ++i) cp_async16(&sm.raw[i][row][ch * EPC], in.p[i] + off, live);
  }
  cp_async_commit();
  Stage<N, N>& st = stages[item];
  {
    float f[W];
#pragma unroll
    for (int p = 0; p < W; ++p) {
      const int t = t0 + (BWD ? W - 1 - p : p);
      f[p] = t < Tn ? to_f32(v[base + (long long)t * lay.st + q]) : 0.f;
    }
#pragma unroll
    for (int p = 0; p < W; p += 4) *reinterpret_cast<float4*>(&st.vt[q][p]) = make_float4(f[p], f[p + 1], f[p + 2], f[p + 3]);
  }
  Preparer<T, N, BWD> prep(sm.scalars, q);
  cp_async_wait();
  bar_sync(1 + g, N);
  prep.decays(sm.raw, Tn - t0);
  bar_sync(1 + g, N);
  prep.scalars(sm.raw);
  bar_sync(1 + g, N);
  prep.write(sm.raw, st);
}

template <int N, int SLOTS>
struct SweepSmem {
  Stage<N, RV> stage[SLOTS];
  uint64_t full[SLOTS], empty[SLOTS];
};
// With at most one CTA to an SM, slots enough that no two CTAs fit one: they may come while the preparing kernel runs out, and
// would otherwise share the first SMs that are free (B 2, T 1024, 16 heads: 177 -> 230 us).
template <int N> constexpr int FEW_CTAS_SLOTS = 116 * 1024 / sizeof(Stage<N, RV>) + 1;
// What one launch takes through: units from unit0 on and their blocks idx0 .. idx0 + nb - 1 in processing order; the states before
// and after these (one per unit of the launch), nullptr where they are the sequence's own.
struct SweepPart { int unit0, idx0, nb; const float* from; float* to; };
// A warp beside the state warps fetches the stages.
template <typename T, int N, bool BWD, int SLOTS, int ROWS, int PER_SM>
__global__ void __launch_bounds__(state_threads<N, ROWS>() + 32, PER_SM)
r7_sweep_kernel(const Stage<N, N>* __restrict__ stages, const float* s_in, int n_state, T* __restrict__ out, float* s_out,
                float* __restrict__ ckpt, int Tn, int H, SweepPart part, TokLayout lay, int* status) {
  constexpr int NCONS = state_threads<N, ROWS>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& sm = *reinterpret_cast<SweepSmem<N, SLOTS>*>(smem_raw);
  const int unit = part.unit0 + blockIdx.x, ys = blockIdx.y, tid = threadIdx.x, nb = part.nb;
  const int bi = unit / H, hi = unit % H;
  if (tid == 0) {
    for (int i = 0; i < SLOTS; ++i) { tc::mbar_init(&sm.full[i], 1); tc::mbar_init(&sm.empty[i], NCONS / 32); }
    tc::fence_mbar_init();
  }
  __syncthreads();
  earlier_kernels_done();
  later_kernels_may_start();
  if (tid < NCONS) {
    const int NB = (Tn + W - 1) / W, NG = (Tn + GT - 1) / GT;
    const long long base = bi * lay.sb + hi * lay.sh, rows = (long long)ys * RV * N;
    StateRows<N, ROWS> S(tid);
    S.get(part.from ? part.from + (long long)blockIdx.x * N * N + rows
                    : s_in && n_state > 0 ? s_in + (long long)(n_state == 1 ? hi : unit) * N * N + rows : nullptr);
    for (int i = 0, slot = 0, phase = 0; i < nb; ++i) {
      const int n = BWD ? NB - 1 - part.idx0 - i : part.idx0 + i;
      if (ckpt)
        if (float* p = state_slot<N, BWD>(ckpt, unit, NG, n)) S.put(p + rows);
      if (!tc::mbar_wait(&sm.full[slot], phase, status, 501)) break;
      float oo[ROWS];
      S.step(sm.stage[slot], oo);
      __syncwarp();
      if (S.lane == 0) tc::mbar_arrive(&sm.empty[slot]);
      const int t = n * W + (BWD ? W - 1 - S.jl : S.jl);
      if (out && t < Tn) S.put_out(out + base + (long long)t * lay.st + ys * RV, oo);
      if (++slot == SLOTS) { slot = 0; phase ^= 1; }
    }
    if (part.to) S.put(part.to + (long long)blockIdx.x * N * N + rows);
    else if (s_out) S.put(s_out + (long long)unit * N * N + rows);
  } else if (tc::elect_one()) {
    const Stage<N, N>* src = stages + (long long)blockIdx.x * nb;
    for (int i = 0, slot = 0, phase = 1; i < nb; ++i, ++src) {
      if (i >= SLOTS && !tc::mbar_wait(&sm.empty[slot], phase, status, 502)) break;
      tc::mbar_expect_tx(&sm.full[slot], COMMON_BYTES<N> + SLICE_BYTES);
      tc::bulk_load(&sm.stage[slot], src, COMMON_BYTES<N>, &sm.full[slot]);
      tc::bulk_load(&sm.stage[slot].vt[0][0], &src->vt[ys * RV][0], SLICE_BYTES, &sm.full[slot]);
      if (++slot == SLOTS) { slot = 0; phase ^= 1; }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// the other gradients, 16 tokens of one unit per CTA
// ---------------------------------------------------------------------------------------------
// S = state before the tokens, G = gradient of the state after them.  With S_j, G_j the state after token j and its
// whole gradient, dr_j = S_j^T do_j, da_j = S_{j-1}^T dsa_j, dk_j = G_j^T v_j, db_j = G_j^T sa_j and
// dd_j = sum_v G_j S_{j-1}.  Three 64 x 64 states are multiplied with the block's vectors (rows: S a~ -> sa, G b^ ->
// dsa; columns: S^T [do dsa], G^T [sa v]), after which every channel is on its own: it steps S_j^T do_i, S_j^T dsa_i,
// G_j^T v_i and G_j^T sa_i through the 16 tokens with the scalars sa.do, v.do, sa.dsa, v.dsa (four threads to a
// channel).  dd_j is summed from the same quantities, positive decay factors throughout, so no term cancels that does not in
// the token-by-token form.  At N = 64 a CTA is 31 k warp instructions (1.9 per cycle and SM, of four) and 9.8 k shared-memory
// wavefronts of 16.8 k cycles, two CTAs to an SM, whose barriers cost as much as either.  B 2, T 1024, 16 heads, float32: 163 us when
// the lanes that share an operand lay apart, 134 before everything was requested at once and both states kept, 127 now.
template <int N> constexpr bool BOTH_STATES = N == 64;      // both fit; at N = 128 G replaces S and S is fetched again
template <int N>
struct GradSmem {
  float st[BOTH_STATES<N> ? 2 : 1][N][N + 4];      // S, G
  float raw[5][GT][N];                // r, d, k, a, b
  float xs[GT][N + 4];                // a~, then b^
  float cat1[N][36], cat2[N][36];     // [sa v], [do dsa], one row per value channel
  float outG[N][36], outS[N][36];     // G^T cat1, S^T cat2, one row per key channel
  float sc[4][GT][GT];                // A_qb, A_qk, A_ab, A_ak (row = later token)
  float sv[2 * GT][36], svT[2 * GT][36];      // cat1^T cat2 and its transpose
};

template <typename T, int N>
__global__ void __launch_bounds__(4 * N, N == 64 ? 2 : 1)
r7_grad_kernel(Vecs<T> in, const T* __restrict__ v, const T* __restrict__ d_o, const float* __restrict__ h0, int n_state,
               const float* __restrict__ d_ht, const float* __restrict__ states, const float* __restrict__ d_states,
               T* __restrict__ dr, T* __restrict__ dw, T* __restrict__ dk, T* __restrict__ da, T* __restrict__ db, int Tn, int H, TokLayout lay) {
  constexpr int NTHR = 4 * N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GradSmem<N>& sm = *reinterpret_cast<GradSmem<N>*>(smem_raw);
  earlier_kernels_done();
  later_kernels_may_start();
  const int tid = threadIdx.x, lane = tid & 31;
  const int NG = (Tn + GT - 1) / GT;
  const int unit = blockIdx.x / NG, m = blockIdx.x % NG, bi = unit / H, hi = unit % H;
  const int t0 = m * GT;
  const long long base = bi * lay.sb + hi * lay.sh + (long long)t0 * lay.st;
  const int nt = min(GT, Tn - t0);
  const long long cu = (long long)unit * (NG - 1) + m;      // this unit's boundaries lie between its groups of tokens
  const float* ckpt_any = reinterpret_cast<const float*>(v);      // (an address for copies of nothing)
  const float* Sg = m > 0 ? states + (cu - 1) * N * N : n_state > 0 ? h0 + (long long)(n_state == 1 ? hi : unit) * N * N : nullptr;
  const float* Gg = m < NG - 1 ? d_states + cu * N * N : d_ht ? d_ht + (long long)unit * N * N : nullptr;

  // ---- tokens and states; everything is requested before anything is waited for
  const int kq = tid % (N / 4), row0 = tid / (N / 4);      // quad of channels, token / state row (16 at a time)
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float (*const S)[N + 4] = sm.st[0];
  float (*const G)[N + 4] = sm.st[BOTH_STATES<N> ? 1 : 0];
  auto request_state = [&](float (*to)[N + 4], const float* g) {
#pragma unroll
    for (int x = 0; x < N / 16; ++x) {
      const int rr = row0 + 16 * x;
      cp_async16(&to[rr][4 * kq], g ? g + (long long)rr * N + 4 * kq : ckpt_any, g != nullptr);
    }
  };
  request_state(S, Sg);
  if constexpr (BOTH_STATES<N>) request_state(G, Gg);
  cp_async_commit();
  // four values down a column of an array whose rows are 36 floats long: every second lane starts with another one of
  // them, which leaves two of the eight lanes that would meet on a bank
  auto put_column = [&](const float (&f)[4], auto at) {
    const int by = kq >> 1;
    const float a0 = by & 1 ? f[1] : f[0], a1 = by & 1 ? f[2] : f[1], a2 = by & 1 ? f[3] : f[2], a3 = by & 1 ? f[0] : f[3];
    const float b[4] = {by & 2 ? a2 : a0, by & 2 ? a3 : a1, by & 2 ? a0 : a2, by & 2 ? a1 : a3};
#pragma unroll
    for (int x = 0; x < 4; ++x) *at((x + by) & 3) = b[x];
  };
  {
    const bool live = row0 < nt;
    const long long off = base + (live ? (long long)row0 * lay.st : 0) + 4 * kq;
    float4 f[5], fv = zero, fo = zero;
#pragma unroll
    for (int i = 0; i < 5; ++i) f[i] = live ? load4(in.p[i] + off) : zero;
    if (live) { fv = load4(v + off); fo = load4(d_o + off); }
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      if (i == VW) f[i] = live ? make_float4(decay_of(f[i].x), decay_of(f[i].y), decay_of(f[i].z), decay_of(f[i].w)) : make_float4(1.f, 1.f, 1.f, 1.f);
      *reinterpret_cast<float4*>(&sm.raw[i][row0][4 * kq]) = f[i];
    }
    const float ev[4] = {fv.x, fv.y, fv.z, fv.w}, eo[4] = {fo.x, fo.y, fo.z, fo.w};
    put_column(ev, [&](int x) { return &sm.cat1[4 * kq + x][GT + row0]; });
    put_column(eo, [&](int x) { return &sm.cat2[4 * kq + x][row0]; });
  }
  for (int e = tid; e < 4 * GT * GT; e += NTHR) (&sm.sc[0][0][0])[e] = 0.f;
  __syncthreads();

  // ---- scalars A: sources i and 15 - i per group of N/2 threads (17 pairs whatever i), two channels per thread
  {
    constexpr int NL = N / 2;
    const int pi = tid / NL, gq = tid % NL;
    float s[64];
#pragma unroll
    for (int e = 0; e < 64; ++e) s[e] = 0.f;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int i = half ? 15 - pi : pi, last = half ? pi : 15 - pi;
      f32x2 pb = *reinterpret_cast<const f32x2*>(&sm.raw[VB][i][2 * gq]), pk = *reinterpret_cast<const f32x2*>(&sm.raw[VK][i][2 * gq]);
#pragma unroll
      for (int x = 0; x < (half ? 8 : 16); ++x) {
        if (x > last) break;
        const int j = i + x, at = half ? 16 - x : x;
        if (x > 0) {
          const f32x2 aj = *reinterpret_cast<const f32x2*>(&sm.raw[VA][j][2 * gq]), dj = *reinterpret_cast<const f32x2*>(&sm.raw[VW][j][2 * gq]);
          s[33 + at] = sum2(mul2(pb, aj));
          s[48 + at] = sum2(mul2(pk, aj));
          pb = mul2(pb, dj); pk = mul2(pk, dj);
        }
        const f32x2 rj = *reinterpret_cast<const f32x2*>(&sm.raw[VR][j][2 * gq]);
        s[at] = sum2(mul2(pb, rj));
        s[17 + at] = sum2(mul2(pk, rj));
      }
    }
    __syncwarp();
    reduce_scatter<64, 16, 1>(s, lane);      // two sums per lane
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = 2 * lane + h;
      const int kind = e < 17 ? 0 : e < 34 ? 1 : e < 49 ? 2 : 3;
      const int x = e - (kind == 0 ? 0 : kind == 1 ? 17 : kind == 2 ? 33 : 48);
      const int i = x <= 15 - pi ? pi : 15 - pi, j = x <= 15 - pi ? pi + x : 15 - pi + (16 - x);
      if constexpr (N == 64) sm.sc[kind][j][i] = s[h];
      else                   atomicAdd(&sm.sc[kind][j][i], s[h]);      // two warps' halves: one addition to 0, one to the other
    }
  }
  // ---- a~_j = a_j times the decays before it in the block
  auto scaled = [&](bool back) {
    if (tid < N) {
      float run = 1.f;
#pragma unroll
      for (int p = 0; p < GT; ++p) {
        const int j = back ? GT - 1 - p : p;
        sm.xs[j][tid] = run * sm.raw[back ? VB : VA][j][tid];
        run *= sm.raw[VW][j][tid];
      }
    }
  };
  scaled(false);
  cp_async_wait();
  __syncthreads();

  // rows: dst[v][j] = sum_k st[v][k] xs[j][k]; a 4 x 4 tile per thread and a quarter of the channels
  auto row_product = [&](const float (*st)[N + 4], float (*dst)[36], int j0) {
    const int s = (tid >> 2) & 3, tj = (tid & 1) | ((tid >> 3) & 2), tv = ((tid >> 1) & 1) | (tid >> 5 << 1);
    f32x2 acc[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) acc[e] = 0ull;
#pragma unroll
    for (int x = 0; x < N / 16; ++x) {
      const int c = 4 * (s + 4 * x);
      Quad A[4], B[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) { A[e] = lds4(&st[4 * tv + e][c]); B[e] = lds4(&sm.xs[4 * tj + e][c]); }
#pragma unroll
      for (int e = 0; e < 16; ++e) acc[e] = fma2(A[e >> 2].hi, B[e & 3].hi, fma2(A[e >> 2].lo, B[e & 3].lo, acc[e]));
    }
    float r[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) r[e] = sum2(acc[e]);
    reduce_scatter<16, 8, 4>(r, lane);      // lane s keeps row s of the tile
    *reinterpret_cast<float4*>(&dst[4 * tv + s][j0 + 4 * tj]) = make_float4(r[0], r[1], r[2], r[3]);
  };
  // columns: acc(k, j) = sum_v A[v][k] B[v][j] over 4 x 4 tiles; NS lanes share the rows of a tile, RUN rows at a time each
  // (as many as put these lanes' rows, 36 or 68 floats apart, on different banks)
  auto col_product = [&](const float* A, int lda, const float (*B)[36], int tk, int tj, int s, int NS, int RUN, float (&r)[16]) {
    f32x2 acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0ull;
#pragma unroll 4
    for (int it = 0; it < N / NS; ++it) {
      const int x = it % RUN + RUN * (s + NS * (it / RUN));
      const Quad a = lds4(A + x * lda + 4 * tk);
      const float4 b = *reinterpret_cast<const float4*>(&B[x][4 * tj]);
      const f32x2 bb[4] = {pack2(b.x, b.x), pack2(b.y, b.y), pack2(b.z, b.z), pack2(b.w, b.w)};
#pragma unroll
      for (int j = 0; j < 4; ++j) { acc[j] = fma2(a.lo, bb[j], acc[j]); acc[4 + j] = fma2(a.hi, bb[j], acc[4 + j]); }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 lo = unpack2(acc[j]), hi = unpack2(acc[4 + j]);
      r[j] = lo.x; r[4 + j] = lo.y; r[8 + j] = hi.x; r[12 + j] = hi.y;      // r[4 k + j]
    }
  };
  auto state_cols = [&](const float (*st)[N + 4], float (*dst)[36], const float (*B)[36]) {
    const int s = (tid >> 2) & 1, tj = (tid & 1) | ((tid >> 2) & 6), tk = ((tid >> 1) & 1) | (tid >> 5 << 1);
    float r[16];
    col_product(&st[0][0], N + 4, B, tk, tj, s, 2, 4, r);
    reduce_scatter<16, 4, 4>(r, lane);      // lane s keeps channels 2 s, 2 s + 1
    *reinterpret_cast<float4*>(&dst[4 * tk + 2 * s][4 * tj]) = make_float4(r[0], r[1], r[2], r[3]);
    *reinterpret_cast<float4*>(&dst[4 * tk + 2 * s + 1][4 * tj]) = make_float4(r[4], r[5], r[6], r[7]);
  };

  row_product(S, sm.cat1, 0);
  __syncthreads();
  if (tid < N) {      // sa_j, one value row per thread
    float sa[GT], vv[GT];
#pragma unroll
    for (int j = 0; j < GT; j += 4) {
      const float4 y = *reinterpret_cast<const float4*>(&sm.cat1[tid][j]), f = *reinterpret_cast<const float4*>(&sm.cat1[tid][GT + j]);
      sa[j] = y.x; sa[j + 1] = y.y; sa[j + 2] = y.z; sa[j + 3] = y.w;
      vv[j] = f.x; vv[j + 1] = f.y; vv[j + 2] = f.z; vv[j + 3] = f.w;
    }
#pragma unroll
    for (int j = 1; j < GT; ++j) {
      float s1 = 0.f, s2 = 0.f;
#pragma unroll
      for (int i = 0; i < j; i += 4) {
        const float4 ab = *reinterpret_cast<const float4*>(&sm.sc[2][j][i]), ak = *reinterpret_cast<const float4*>(&sm.sc[3][j][i]);
        s1 += ak.x * vv[i];
        if (i + 1 < j) s1 += ak.y * vv[i + 1];
        if (i + 2 < j) s1 += ak.z * vv[i + 2];
        if (i + 3 < j) s1 += ak.w * vv[i + 3];
        s2 += ab.x * sa[i];
        if (i + 1 < j) s2 += ab.y * sa[i + 1];
        if (i + 2 < j) s2 += ab.z * sa[i + 2];
        if (i + 3 < j) s2 += ab.w * sa[i + 3];
      }
      sa[j] += s1 + s2;
    }
#pragma unroll
    for (int j = 0; j < GT; j += 4) *reinterpret_cast<float4*>(&sm.cat1[tid][j]) = make_float4(sa[j], sa[j + 1], sa[j + 2], sa[j + 3]);
  }
  // ---- sum_v G S (16 partial rows in outS); at N = 128 G replaces S on the way
  {
    float4 z = zero;
#pragma unroll
    for (int x = 0; x < N / 16; ++x) {
      const int rr = row0 + 16 * x;
      const float4 s4 = *reinterpret_cast<const float4*>(&S[rr][4 * kq]);
      float4 g4;
      if constexpr (BOTH_STATES<N>) {
        g4 = *reinterpret_cast<const float4*>(&G[rr][4 * kq]);
      } else {
        g4 = Gg ? __ldg(reinterpret_cast<const float4*>(Gg + (long long)rr * N + 4 * kq)) : zero;
        *reinterpret_cast<float4*>(&G[rr][4 * kq]) = g4;
      }
      z.x += g4.x * s4.x; z.y += g4.y * s4.y; z.z += g4.z * s4.z; z.w += g4.w * s4.w;
    }
    const float ez[4] = {z.x, z.y, z.z, z.w};
    put_column(ez, [&](int x) { return &sm.outS[4 * kq + x][row0]; });
  }
  scaled(true);
  __syncthreads();
  float zsum = 0.f;      // role 2 below: this channel's sum_v G S
  if (tid / N == 2) {
#pragma unroll
    for (int x = 0; x < 16; x += 4) {
      const float4 f = *reinterpret_cast<const float4*>(&sm.outS[tid % N][x]);
      zsum += (f.x + f.y) + (f.z + f.w);
    }
  }
  row_product(G, sm.cat2, GT);
  state_cols(G, sm.outG, sm.cat1);
  __syncthreads();
  if constexpr (!BOTH_STATES<N>) {
    request_state(S, Sg);
    cp_async_commit();
  }
  if (tid < N) {      // dsa_j, from the last token to the first
    float ds[GT], dov[GT];
#pragma unroll
    for (int j = 0; j < GT; j += 4) {
      const float4 e = *reinterpret_cast<const float4*>(&sm.cat2[tid][GT + j]), f = *reinterpret_cast<const float4*>(&sm.cat2[tid][j]);
      ds[j] = e.x; ds[j + 1] = e.y; ds[j + 2] = e.z; ds[j + 3] = e.w;
      dov[j] = f.x; dov[j + 1] = f.y; dov[j + 2] = f.z; dov[j + 3] = f.w;
    }
#pragma unroll
    for (int i = GT - 1; i >= 0; --i) {
      ds[i] += sm.sc[0][i][i] * dov[i];      // now final
#pragma unroll
      for (int j = 0; j < i; j += 4) {
        const float4 qb = *reinterpret_cast<const float4*>(&sm.sc[0][i][j]), ab = *reinterpret_cast<const float4*>(&sm.sc[2][i][j]);
        const float q_[4] = {qb.x, qb.y, qb.z, qb.w}, a_[4] = {ab.x, ab.y, ab.z, ab.w};
#pragma unroll
        for (int x = 0; x < 4; ++x) if (j + x < i) ds[j + x] += q_[x] * dov[i];
#pragma unroll
        for (int x = 0; x < 4; ++x) if (j + x < i) ds[j + x] += a_[x] * ds[i];
      }
    }
#pragma unroll
    for (int j = 0; j < GT; j += 4) *reinterpret_cast<float4*>(&sm.cat2[tid][GT + j]) = make_float4(ds[j], ds[j + 1], ds[j + 2], ds[j + 3]);
  }
  if constexpr (!BOTH_STATES<N>) cp_async_wait();
  __syncthreads();
  state_cols(S, sm.outS, sm.cat2);
  {
    constexpr int NS = NTHR / 64;      // 4 or 8 lanes per tile
    const int s = (tid >> 2) % NS, high = tid / (4 * NS);      // tj bit 0, ti bit 0, s, then the other two bits of ti and of tj
    const int ti = ((tid >> 1) & 1) | ((high & 3) << 1), tj = (tid & 1) | (high >> 2 << 1);
    float r[16];
    col_product(&sm.cat1[0][0], 36, sm.cat2, ti, tj, s, NS, 2, r);
    reduce_scatter<16, 2 * NS, 4>(r, lane);
    constexpr int KEEP = 16 / NS;
#pragma unroll
    for (int x = 0; x < KEEP; ++x) {
      const int e = s * KEEP + x, i = 4 * ti + (e >> 2), j = 4 * tj + (e & 3);
      sm.sv[i][j] = r[x];
      sm.svT[j][i] = r[x];
    }
  }
  __syncthreads();

  // ---- one channel per thread and role
  const int role = tid / N, c = tid % N;
  float d[GT];
#pragma unroll
  for (int j = 0; j < GT; ++j) d[j] = sm.raw[VW][j][c];
  float dd[GT];      // role 0: the parts of dd that come from the outputs; role 1: from dsa; role 2: from G
  if (role < 2) {
    float x[GT], p[GT];      // S_{j-1}^T do_i or dsa_i, and the vector of token i that meets it in G_j
#pragma unroll
    for (int j = 0; j < GT; j += 4) {
      const float4 f = *reinterpret_cast<const float4*>(&sm.outS[c][GT * role + j]);
      x[j] = f.x; x[j + 1] = f.y; x[j + 2] = f.z; x[j + 3] = f.w;
    }
#pragma unroll
    for (int j = 0; j < GT; ++j) p[j] = sm.raw[role == 0 ? VR : VA][j][c];
    T* const dst = role == 0 ? dr : da;
#pragma unroll
    for (int j = 0; j < GT; ++j) {
      const float bj = sm.raw[VB][j][c], kj = sm.raw[VK][j][c];
      float run = 1.f, s = 0.f;
      if (role == 0) {
        s = x[j] * p[j];
#pragma unroll
        for (int i = j + 1; i < GT; ++i) { run *= d[i]; s += x[i] * (run * p[i]); }
      } else {
        if (j < nt) dst[base + (long long)j * lay.st + c] = from_f32<T>(x[j]);
#pragma unroll
        for (int i = j + 1; i < GT; ++i) { s += x[i] * (run * p[i]); run *= d[i]; }
      }
      dd[j] = s;
#pragma unroll
      for (int i4 = j & ~3; i4 < GT; i4 += 4) {
        const float4 fs = *reinterpret_cast<const float4*>(&sm.sv[j][GT * role + i4]);
        const float4 fv = *reinterpret_cast<const float4*>(&sm.sv[GT + j][GT * role + i4]);
        const float es[4] = {fs.x, fs.y, fs.z, fs.w}, ev[4] = {fv.x, fv.y, fv.z, fv.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) if (i4 + e >= j) x[i4 + e] = x[i4 + e] * d[j] + (es[e] * bj + ev[e] * kj);
      }
      if (role == 0 && j < nt) dst[base + (long long)j * lay.st + c] = from_f32<T>(x[j]);
    }
    if (role == 1) {
#pragma unroll
      for (int j = 0; j < GT; j += 4) *reinterpret_cast<float4*>(&sm.outS[c][GT + j]) = make_float4(dd[j], dd[j + 1], dd[j + 2], dd[j + 3]);
    }
  } else {
    float x[GT];      // G_j^T v_i (role 2) or G_j^T sa_i (role 3)
    const int o = role == 2 ? GT : 0;
#pragma unroll
    for (int j = 0; j < GT; j += 4) {
      const float4 f = *reinterpret_cast<const float4*>(&sm.outG[c][o + j]);
      x[j] = f.x; x[j + 1] = f.y; x[j + 2] = f.z; x[j + 3] = f.w;
    }
    if (role == 2) {      // sum_v G S_{j-1}, times the decays after token j
      float q[GT], z = zsum, after = 1.f;
#pragma unroll
      for (int j = 0; j < GT; j += 4) {
        const float4 f = *reinterpret_cast<const float4*>(&sm.outG[c][j]);
        q[j] = f.x; q[j + 1] = f.y; q[j + 2] = f.z; q[j + 3] = f.w;
      }
#pragma unroll
      for (int j = 0; j < GT; ++j) { dd[j] = z; z = z * d[j] + (q[j] * sm.raw[VB][j][c] + x[j] * sm.raw[VK][j][c]); }
#pragma unroll
      for (int j = GT - 1; j >= 0; --j) { dd[j] *= after; after *= d[j]; }
#pragma unroll
      for (int j = 0; j < GT; j += 4) *reinterpret_cast<float4*>(&sm.outG[c][GT + j]) = make_float4(dd[j], dd[j + 1], dd[j + 2], dd[j + 3]);
    }
    T* const dst = role == 2 ? dk : db;
#pragma unroll
    for (int j = GT - 1; j >= 0; --j) {
      const float rj = sm.raw[VR][j][c], aj = sm.raw[VA][j][c];
#pragma unroll
      for (int i4 = 0; i4 <= j; i4 += 4) {
        const float4 fo = *reinterpret_cast<const float4*>(&sm.svT[j][o + i4]);
        const float4 fs = *reinterpret_cast<const float4*>(&sm.svT[GT + j][o + i4]);
        const float eo[4] = {fo.x, fo.y, fo.z, fo.w}, es[4] = {fs.x, fs.y, fs.z, fs.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (i4 + e == j) x[j] += eo[e] * rj;
          if (i4 + e < j) x[i4 + e] = (x[i4 + e] + eo[e] * rj) * d[j] + es[e] * aj;
        }
      }
      if (j < nt) dst[base + (long long)j * lay.st + c] = from_f32<T>(x[j]);
    }
  }
  // role 0 has the w rows fetched before it waits (one after the other they took a fifth of the kernel)
  float ew[GT];
  if (role == 0) {
#pragma unroll
    for (int j = 0; j < GT; ++j) ew[j] = j < nt ? to_f32(__ldg(in.p[VW] + base + (long long)j * lay.st + c)) : 0.f;
  }
  __syncthreads();
  if (role == 0) {
#pragma unroll
    for (int j = 0; j < GT; ++j) {
      const float s = dd[j] + sm.outS[c][GT + j] + sm.outG[c][GT + j];
      if (j < nt) dw[base + (long long)j * lay.st + c] = from_f32<T>(s * d[j] * -expf(ew[j]));
    }
  }
}

template <typename T, int N, bool BWD, int GROUPS, int ROWS>
int launch_inline(const DeviceFacts& dev, const Vecs<T>& in, const void* v, const float* s_in, int n_state, void* out, float* s_out,
                  float* ckpt, int B, int Tn, int H, const TokLayout& lay, cudaStream_t st) {
  constexpr int bytes = (int)sizeof(Group<T, N>);
  if (allow_smem<r7_sweep_inline_kernel<T, N, BWD, GROUPS, ROWS>>(dev, GROUPS * bytes)) return RWKVB200_E_CUDA;
  const int blocks = (Tn + W - 1) / W, groups = blocks < GROUPS ? blocks : GROUPS;      // a group without a block is left out
  ProfScope prof(BWD ? "r7_sweep_bwd_kernel" : "r7_sweep_fwd_kernel", st);
  return launch(r7_sweep_inline_kernel<T, N, BWD, GROUPS, ROWS>, dim3(B * H, N / RV), state_threads<N, ROWS>() + N * groups,
                groups * bytes, st, 1, in, (const T*)v, s_in, n_state, (T*)out, s_out, ckpt, Tn, H, lay);
}

template <typename T, int N, bool BWD, int SLOTS, int ROWS, int PER_SM>
int launch_sweep(const DeviceFacts& dev, const Stage<N, N>* stages, const float* s_in, int n_state, void* out, float* s_out, float* ckpt,
                 int n_units, int Tn, int H, const SweepPart& part, const TokLayout& lay, cudaStream_t st) {
  constexpr int bytes = (int)sizeof(SweepSmem<N, SLOTS>);
  if (allow_smem<r7_sweep_kernel<T, N, BWD, SLOTS, ROWS, PER_SM>>(dev, bytes)) return RWKVB200_E_CUDA;
  ProfScope prof(BWD ? "r7_sweep_bwd_kernel" : "r7_sweep_fwd_kernel", st);
  return launch(r7_sweep_kernel<T, N, BWD, SLOTS, ROWS, PER_SM>, dim3(n_units, N / RV), state_threads<N, ROWS>() + 32, bytes, st,
                PER_SM == 1 ? 1 : 0, stages, s_in, n_state, (T*)out, s_out, ckpt, Tn, H, part, lay, dev.status);
}

// From how many blocks per unit on they are prepared by a kernel of their own (forward, us; inside the sweep against apart):
// with at most one CTA per SM the sweep has to be long enough for the other kernel (12 units, T 128 15.8 and 15.0, T 300 32.7 and
// 29.3, T 1024 101 and 83; 37 units 16.0 and 18.5, 33.0 and 31.6, 101 and 96); at head size 64 two CTAs per SM inside keep up
// (60 units, T 300 57 and 60); beyond that it pays from the start (128 units, T 32 15.6 and 14.7, T 1024 364 and 227; head size
// 128, 64 units, T 1024 711 and 375).
constexpr int STAGED_BLOCKS = 4;
template <int N> bool prepared_apart(long long ctas, int NB, int sms) {
  if (ctas <= sms) return NB >= (N == 64 ? 48 : 12);
  return (N == 128 || ctas > 2 * sms) && NB >= STAGED_BLOCKS;
}
// Scratch of a sweep whose blocks are prepared apart, STAGES_BYTES at most: stages of `blocks` blocks (a stretch) of `units` units
// (a pass), and the units' states between one stretch and the next.  As many blocks as fit for all units; with very many units 8,
// whose 88 KB of stages are worth the 32 KB of a state left and fetched, for as many units as fit, at least 1100, which fill the
// device.  (More than L2 holds costs little: 1.4 KB per token and head, where the inputs take 1.5.)
constexpr size_t STAGES_BYTES = (size_t)256 << 20;
constexpr int STRETCH_BLOCKS = 8;
struct Staging { int blocks, units; };      // 0: the blocks are prepared inside the sweep, without scratch
template <int N> size_t unit_bytes(int blocks, int NB) {
  return blocks * sizeof(Stage<N, N>) + (blocks < NB ? N * N * sizeof(float) : 0);
}
template <int N> Staging staging(long long units, int Tn, int sms) {
  const int NB = (Tn + W - 1) / W;
  if (!prepared_apart<N>(units * (N / RV), NB, sms)) return Staging{0, 0};
  int blocks = NB;
  if (units * unit_bytes<N>(NB, NB) > STAGES_BYTES) {
    const long long share = STAGES_BYTES / units, fit = (share - (long long)(N * N * sizeof(float))) / (long long)sizeof(Stage<N, N>);
    blocks = (int)(fit > STRETCH_BLOCKS ? fit : NB < STRETCH_BLOCKS ? NB : STRETCH_BLOCKS);
  }
  const long long pass = STAGES_BYTES / unit_bytes<N>(blocks, NB);
  return Staging{blocks, (int)(pass < units ? pass : units)};
}
template <int N> size_t scratch_bytes(long long units, int Tn) {
  DeviceFacts dev;
  const Staging s = staging<N>(units, Tn, device_facts(&dev) ? 148 : dev.sms);      // (asked where there is no device)
  return s.units * unit_bytes<N>(s.blocks, (Tn + W - 1) / W);
}

template <typename T, int N, bool BWD>
int sweep(const Vecs<T>& in, const void* v, const float* s_in, int n_state, void* out, float* s_out, float* ckpt, int B,
          int Tn, int H, const TokLayout& lay, void* scratch, cudaStream_t st) {
  DeviceFacts dev;
  if (int e = device_facts(&dev)) return e;
  const int units = B * H, NB = (Tn + W - 1) / W;
  const bool many = units * (N / RV) > dev.sms;
  const Staging s = staging<N>(units, Tn, dev.sms);
  if (!scratch || !s.blocks)
    return many ? launch_inline<T, N, BWD, MANY_CTAS<T, N>, MANY_CTAS_ROWS>(dev, in, v, s_in, n_state, out, s_out, ckpt, B, Tn, H, lay, st)
                : launch_inline<T, N, BWD, FEW_CTAS<N>, FEW_CTAS_ROWS<N>>(dev, in, v, s_in, n_state, out, s_out, ckpt, B, Tn, H, lay, st);
  auto* stages = static_cast<Stage<N, N>*>(scratch);
  float* between = reinterpret_cast<float*>(stages + (size_t)s.units * s.blocks);
  constexpr int per_cta = PREPARE_THREADS / N, bytes = per_cta * (int)sizeof(PrepareSmem<T, N>);
  if (allow_smem<r7_prepare_kernel<T, N, BWD>>(dev, bytes)) return RWKVB200_E_CUDA;
  for (int unit0 = 0; unit0 < units; unit0 += s.units)
    for (int idx0 = 0; idx0 < NB; idx0 += s.blocks) {
      const int n_units = units - unit0 < s.units ? units - unit0 : s.units;
      const int nb = NB - idx0 < s.blocks ? NB - idx0 : s.blocks, n_items = n_units * nb;
      {
        ProfScope prof("r7_prepare_kernel", st);
        if (int e = launch(r7_prepare_kernel<T, N, BWD>, (n_items + per_cta - 1) / per_cta, PREPARE_THREADS, bytes, st, 1, in,
                           (const T*)v, stages, Tn, H, unit0, idx0, nb, n_items, lay)) return e;
      }
      const float* from = idx0 == 0 ? nullptr : between;
      float* to = idx0 + nb == NB ? nullptr : between;
      const SweepPart part{unit0, idx0, nb, from, to};
      const int e = many ? launch_sweep<T, N, BWD, 4, MANY_CTAS_ROWS, 3>(dev, stages, s_in, n_state, out, s_out, ckpt, n_units, Tn, H, part, lay, st)
                         : launch_sweep<T, N, BWD, FEW_CTAS_SLOTS<N>, FEW_CTAS_ROWS<N>, 1>(dev, stages, s_in, n_state, out, s_out, ckpt, n_units, Tn, H, part, lay, st);
      if (e) return e;
    }
  return RWKVB200_OK;
}

template <typename T, int N>
int fwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b, const float* h0, int n_state,
        void* o, float* ht, float* states, void* scratch, int B, int Tn, int H, int head_first, cudaStream_t st) {
  const Vecs<T> in{{(const T*)r, (const T*)w, (const T*)k, (const T*)a, (const T*)b}};
  return sweep<T, N, false>(in, v, h0, n_state, o, ht, Tn > GT ? states : nullptr, B, Tn, H, TokLayout(Tn, H, head_first, N), scratch, st);
}

template <typename T, int N>
int bwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b, const float* h0, int n_state,
        const void* d_o, const float* d_ht, const float* kept, float* ckpt, void* scratch, void* dr, void* dw, void* dk, void* dv, void* da,
        void* db, float* d_h0, int B, int Tn, int H, int head_first, cudaStream_t st) {
  const Vecs<T> in{{(const T*)r, (const T*)w, (const T*)k, (const T*)a, (const T*)b}};
  const TokLayout lay(Tn, H, head_first, N);
  int e = RWKVB200_OK;
  // the states between the groups of tokens: as the forward left them, or from another sweep; then their gradients
  const float* states = kept;
  float* d_states = ckpt;
  if (Tn > GT && !kept) {
    states = ckpt;
    d_states = ckpt + (long long)B * H * ((Tn + GT - 1) / GT - 1) * N * N;
    e = sweep<T, N, false>(in, v, h0, n_state, nullptr, nullptr, ckpt, B, Tn, H, lay, scratch, st);
  }
  if (!e) e = sweep<T, N, true>(in, d_o, d_ht, d_ht ? B * H : 0, dv, d_h0, Tn > GT ? d_states : nullptr, B, Tn, H, lay, scratch, st);
  if (e) return e;
  DeviceFacts dev;
  if ((e = device_facts(&dev))) return e;
  const int smem = (int)sizeof(GradSmem<N>);
  if (allow_smem<r7_grad_kernel<T, N>>(dev, smem)) return RWKVB200_E_CUDA;
  ProfScope prof("r7_grad_kernel", st);
  return launch(r7_grad_kernel<T, N>, B * H * ((Tn + GT - 1) / GT), 4 * N, smem, st, 1, in, (const T*)v, (const T*)d_o, h0,
                h0 ? n_state : 0, d_ht, states, (const float*)d_states, (T*)dr, (T*)dw, (T*)dk, (T*)da, (T*)db, Tn, H, lay);
}

}  // namespace

// bfloat16 at head size 64 stays token by token: what is asked for there is the chunked path's fallback, bit for bit
#define R7_BLOCK_DISPATCH(CALL)                                                                                        \
  if (head_size == 64 && dtype == RWKVB200_F32) { constexpr int N = 64; using T = float; return CALL; }                \
  if (head_size == 64 && dtype == RWKVB200_F16) { constexpr int N = 64; using T = __half; return CALL; }               \
  if (head_size == 128) { constexpr int N = 128; RWKVB200_DISPATCH_DTYPE(dtype, return CALL); }   \
  return RWKVB200_E_UNSUPPORTED;

size_t rwkv7_block_states_bytes(int B, int Tn, int H, int dtype, int head_size) {
  if (head_size == 64 && dtype == RWKVB200_BF16) return 0;      // token by token
  return Tn > GT ? (size_t)B * H * ((Tn + GT - 1) / GT - 1) * head_size * head_size * sizeof(float) : 0;
}

size_t rwkv7_block_scratch_bytes(int B, int Tn, int H, int dtype, int head_size) {
  if (head_size == 64) return dtype == RWKVB200_BF16 ? 0 : scratch_bytes<64>((long long)B * H, Tn);
  return scratch_bytes<128>((long long)B * H, Tn);
}

int launch_rwkv7_block_fwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                           const float* h0, int n_state, void* o, float* ht, int B, int Tn, int H, int dtype,
                           int head_first, cudaStream_t st, int head_size, float* states, void* scratch) {
  if (head_size == 64 && dtype == RWKVB200_BF16)
    return launch_rwkv7_rec_fwd(r, w, k, v, a, b, h0, n_state, o, ht, B, Tn, H, head_first, st);
  R7_BLOCK_DISPATCH((fwd<T, N>(r, w, k, v, a, b, h0, n_state, o, ht, states, scratch, B, Tn, H, head_first, st)))
}

int launch_rwkv7_block_bwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                           const float* h0, int n_state, const void* d_o, const float* d_ht, float* ckpt,
                           void* dr, void* dw, void* dk, void* dv, void* da, void* db, float* d_h0, int B, int Tn, int H,
                           int dtype, int head_first, cudaStream_t st, int head_size, const float* states, void* scratch) {
  if (head_size == 64 && dtype == RWKVB200_BF16)
    return launch_rwkv7_rec_bwd(r, w, k, v, a, b, h0, n_state, d_o, d_ht, ckpt, dr, dw, dk, dv, da, db, d_h0, B, Tn, H,
                                head_first, st, UnitSel{}, 0);
  R7_BLOCK_DISPATCH((bwd<T, N>(r, w, k, v, a, b, h0, n_state, d_o, d_ht, states, ckpt, scratch, dr, dw, dk, dv, da, db, d_h0, B, Tn, H,
                               head_first, st)))
}

}  // namespace rwkvb200
