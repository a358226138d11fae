// RWKV7 generalized delta rule, token by token in float32: the exact fallback of the chunked tensor-core path for the
// units its scaled operands cannot represent (backward here, forward inside its scan), the same for whole batches on
// request, and the single step at head size 128.  The same arithmetic as the reference's native operator (rwkv_ops/rwkv7_kernel/native_keras_op.py:80-91); whole
// float32 sequences run eight tokens at a time (rwkv7_block.cu).
//
// Row v of S[v][k] never mixes with another row, so the value rows are split 16 to a CTA: grid (B*H, N/16), N threads.
// In the "row role" thread (vl = tid / (N/16), kq = tid % (N/16)) holds S[vl][16*kq .. 16*kq+15] in registers and
// reductions over k take two or three shuffles.
//
// Backward.  With dS the gradient of the state flowing from the future,
//   dS += do_t r_t^T;  dr_t = S_t^T do_t;  dv_t = dS k_t;  dk_t = dS^T v_t;  dsa = dS b_t;  db_t = dS^T sa_t;
//   dd_t[k] = sum_v dS[v,k] S_{t-1}[v,k];  da_t = S_{t-1}^T dsa;  dS <- dS diag(d_t) + dsa a_t^T;
//   dw_t = dd_t * d_t * (-exp(w_t)).
// It needs S_{t-1} and S_t for every token: a forward sweep over the CTA's rows first stores the state every R7_CKPT
// tokens, and the kernel then walks the chunks in reverse, re-running each chunk forward into shared memory before
// sweeping it backward.  Reductions over v (dr, dk, db, da, dd) need
// all 64 rows: each thread also keeps a "column role" copy dS[0..15][k = tid] of the CTA's slab, the
// four CTAs of a (batch, head) form a thread-block cluster, and after each chunk every CTA sums the
// four partial results of a quarter of the chunk's tokens through distributed shared memory, in a
// fixed order (deterministic, no atomics, no scratch beyond the checkpoints).
#include <cooperative_groups.h>

#include "rwkv7_recurrent.cuh"

namespace cg = cooperative_groups;

namespace rwkvb200 {

namespace {

using namespace r7rec;

constexpr int CK = R7_CKPT;   // chunk of the backward = checkpoint interval

// ---------------------------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------------------------
template <typename T, int N, int TL>
__global__ void __launch_bounds__(N)
rwkv7_rec_fwd_kernel(FwdArgs<T> args, const float* __restrict__ h0, int n_state, float* __restrict__ ht, int H, TokLayout lay) {
  __shared__ __align__(16) FwdSmem<N, VS, TL> sm;
  earlier_kernels_done();
  later_kernels_may_start();
  const int unit = blockIdx.x, bi = unit / H, hi = unit % H;
  args.base = bi * lay.sb + hi * lay.sh;
  args.S0 = h0 && n_state > 0 ? h0 + (long long)(n_state == 1 ? hi : unit) * N * N : nullptr;
  args.ht = ht ? ht + (long long)unit * N * N : nullptr;
  fwd_rows<T, N, VS, 1, TL, N>(args, sm, VS * blockIdx.y, threadIdx.x);
}

// ---------------------------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------------------------
template <int N>
struct BwdSmem {
  float tile[CK][6][NP<N>()];         // r, d, exp(w), k, a, b
  float vt[CK][VS];
  float dot[CK][VS];
  float sa[CK][VS];
  float dvt[CK][VS];
  float dsa[2][VS];
  float Sbuf[CK + 1][VS][N + 1]; // state before token i of the chunk (i = nt: after the last), padded rows
  float part[2][CK][5][N];      // per-chunk partial dr, dk, db, da, dd of this CTA's 16 rows
};

// launched as clusters of N / 16 CTAs along y (one per 16 value rows of a unit)
template <typename T, int N>
__global__ void __launch_bounds__(N)
rwkv7_rec_bwd_kernel(const T* __restrict__ r, const T* __restrict__ w, const T* __restrict__ k,
                     const T* __restrict__ v, const T* __restrict__ a, const T* __restrict__ b,
                     const T* __restrict__ d_o, const float* __restrict__ d_ht, const float* __restrict__ h0, int n_state, float* ckpt,
                     T* __restrict__ dr, T* __restrict__ dw, T* __restrict__ dk, T* __restrict__ dv,
                     T* __restrict__ da, T* __restrict__ db, float* __restrict__ d_h0,
                     int Tn_dense, int H, TokLayout lay, UnitSel sel) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BwdSmem<N>& sm = *reinterpret_cast<BwdSmem<N>*>(smem_raw);
  constexpr int KSEG = N / 16, NQ = N / VS;
  cg::cluster_group cluster = cg::this_cluster();

  earlier_kernels_done();
  later_kernels_may_start();
  const int unit = blockIdx.x, y = blockIdx.y, tid = threadIdx.x;
  if (sel.flags && sel.flags[unit] == 0) return;      // the four CTAs of a cluster share the unit: all leave
  const int bi = unit / H, hi = unit % H;
  const int vl = tid / KSEG, kq = tid % KSEG;   // row role
  const int kc = tid;                      // column role
  const int Tn = sel.seq_len ? sel.seq_len[bi] : Tn_dense;
  const long long base = sel.seq_start ? hi * lay.sh + sel.seq_start[bi] * lay.st : bi * lay.sb + hi * lay.sh;
  const int NC = (Tn + CK - 1) / CK;
  ckpt += unit * (sel.ckpt_unit_stride ? sel.ckpt_unit_stride : (long long)((Tn_dense + CK - 1) / CK) * N * N);
  // The forward over this CTA's rows, for its checkpoints: every thread stores the very values that it loads below.
  {
    static_assert(sizeof(FwdSmem<N, VS, 16>) <= sizeof(BwdSmem<N>), "the forward's tiles live in the backward's shared memory");
    const FwdArgs<T> args{r, w, k, v, a, b, base, lay.st, Tn,
                          n_state > 0 ? h0 + (long long)(n_state == 1 ? hi : unit) * N * N : nullptr, nullptr, nullptr, ckpt};
    fwd_rows<T, N, VS, 1, 16, N>(args, *reinterpret_cast<FwdSmem<N, VS, 16>*>(smem_raw), VS * y, tid);
    __syncthreads();
  }

  float dSr[16], dSc[VS];
  if (d_ht) {
    const float* p = d_ht + ((long long)unit * N + (y * VS + vl)) * N + 16 * kq;
#pragma unroll
    for (int j = 0; j < 16; ++j) dSr[j] = p[j];
#pragma unroll
    for (int i = 0; i < VS; ++i) dSc[i] = d_ht[((long long)unit * N + (y * VS + i)) * N + kc];
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) dSr[j] = 0.f;
#pragma unroll
    for (int i = 0; i < VS; ++i) dSc[i] = 0.f;
  }

  // The inputs and the checkpoint of chunk c - 1 are requested (into registers) before chunk c is worked on,
  // and written to shared memory when chunk c is done: see the forward kernel.
  constexpr int PER = CK * 5 / 4;      // float4 per thread per chunk: CK tokens x (r, w, k, a, b) x N/4 quads
  float4 buf[PER], vbuf = make_float4(0.f, 0.f, 0.f, 0.f), dobuf = vbuf, Snext[4];
  const int quad = tid % (N / 4), rq = tid / (N / 4);
  auto fetch = [&](int c) {
    const int t0 = c * CK, nt = min(CK, Tn - t0);
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int row = rq + 4 * m, tl = row / 5, which = row % 5;
      const T* src = which == 0 ? r : which == 1 ? w : which == 2 ? k : which == 3 ? a : b;
      buf[m] = tl < nt ? load4(src + base + (long long)(t0 + tl) * lay.st + 4 * quad) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (tid < nt * 4) {
      const long long off = base + (long long)(t0 + (tid >> 2)) * lay.st + y * VS + 4 * (tid & 3);
      vbuf = load4(v + off);
      dobuf = load4(d_o + off);
    }
    const float* p = ckpt + (((long long)c * N) + (y * VS + vl)) * N + 16 * kq;
#pragma unroll
    for (int j = 0; j < 4; ++j) Snext[j] = *reinterpret_cast<const float4*>(p + 4 * j);
  };
  // tile rows: 0 r, 1 d, 2 exp(w), 3 k, 4 a, 5 b
  auto stash = [&]() {
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int row = rq + 4 * m, tl = row / 5, which = row % 5;
      const float4 f = buf[m];
      if (which == 1) {
        *reinterpret_cast<float4*>(&sm.tile[tl][1][padk(4 * quad)]) =
            make_float4(decay_of(f.x), decay_of(f.y), decay_of(f.z), decay_of(f.w));
        *reinterpret_cast<float4*>(&sm.tile[tl][2][padk(4 * quad)]) = make_float4(expf(f.x), expf(f.y), expf(f.z), expf(f.w));
      } else {
        *reinterpret_cast<float4*>(&sm.tile[tl][which == 0 ? 0 : which + 1][padk(4 * quad)]) = f;
      }
    }
    if (tid < CK * 4) {
      *reinterpret_cast<float4*>(&sm.vt[tid >> 2][4 * (tid & 3)]) = vbuf;
      *reinterpret_cast<float4*>(&sm.dot[tid >> 2][4 * (tid & 3)]) = dobuf;
    }
  };
  if (NC > 0) fetch(NC - 1);
  for (int c = NC - 1; c >= 0; --c) {
    const int t0 = c * CK, nt = min(CK, Tn - t0), pb = c & 1;
    // ---- the chunk's inputs, and its checkpoint (row role) for the forward re-run
    stash();
    float S[16];
#pragma unroll
    for (int j = 0; j < 4; ++j) { S[4 * j] = Snext[j].x; S[4 * j + 1] = Snext[j].y; S[4 * j + 2] = Snext[j].z; S[4 * j + 3] = Snext[j].w; }
    __syncthreads();
    if (c > 0) fetch(c - 1);
    for (int tl = 0; tl < nt; ++tl) {
      const float* td = &sm.tile[tl][1][20 * kq];
      const float* tk = &sm.tile[tl][3][20 * kq];
      const float* ta = &sm.tile[tl][4][20 * kq];
      const float* tb = &sm.tile[tl][5][20 * kq];
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int j = 0; j < 16; j += 2) {
        sm.Sbuf[tl][vl][16 * kq + j] = S[j];
        sm.Sbuf[tl][vl][16 * kq + j + 1] = S[j + 1];
        s0 += S[j] * ta[j]; s1 += S[j + 1] * ta[j + 1];
      }
      float sa = s0 + s1;
#pragma unroll
      for (int m = 1; m < KSEG; m <<= 1) sa += __shfl_xor_sync(0xffffffffu, sa, m);
      if (kq == 0) sm.sa[tl][vl] = sa;
      const float vv = sm.vt[tl][vl];
#pragma unroll
      for (int j = 0; j < 16; ++j) S[j] = S[j] * td[j] + sa * tb[j] + vv * tk[j];
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) sm.Sbuf[nt][vl][16 * kq + j] = S[j];
    __syncthreads();

    // ---- sweep the chunk backward
    float St[VS], Sp[VS];
#pragma unroll
    for (int i = 0; i < VS; ++i) St[i] = sm.Sbuf[nt][i][kc];
    for (int tl = nt - 1; tl >= 0; --tl) {
      const int buf = tl & 1;
      const float rk = sm.tile[tl][0][padk(kc)], dk_ = sm.tile[tl][1][padk(kc)], ak = sm.tile[tl][4][padk(kc)];
      const float* tr = &sm.tile[tl][0][20 * kq];
      const float* td = &sm.tile[tl][1][20 * kq];
      const float* tk = &sm.tile[tl][3][20 * kq];
      const float* ta = &sm.tile[tl][4][20 * kq];
      const float* tb = &sm.tile[tl][5][20 * kq];
      // row role: dS += do r^T ; dv = dS k ; dsa = dS b
      const float dor = sm.dot[tl][vl];
      float a0 = 0.f, a1 = 0.f, b0 = 0.f, b1 = 0.f;
#pragma unroll
      for (int j = 0; j < 16; j += 2) {
        dSr[j] += dor * tr[j]; dSr[j + 1] += dor * tr[j + 1];
        a0 += dSr[j] * tk[j]; a1 += dSr[j + 1] * tk[j + 1];
        b0 += dSr[j] * tb[j]; b1 += dSr[j + 1] * tb[j + 1];
      }
      float dvv = a0 + a1, dsa = b0 + b1;
#pragma unroll
      for (int m = 1; m < KSEG; m <<= 1) {
        dvv += __shfl_xor_sync(0xffffffffu, dvv, m);
        dsa += __shfl_xor_sync(0xffffffffu, dsa, m);
      }
      if (kq == 0) { sm.dvt[tl][vl] = dvv; sm.dsa[buf][vl] = dsa; }
      // column role, part 1 (does not need dsa)
      float p_dr = 0.f, p_dk = 0.f, p_db = 0.f, p_dd = 0.f;
#pragma unroll
      for (int i = 0; i < VS; ++i) {
        Sp[i] = sm.Sbuf[tl][i][kc];
        const float doi = sm.dot[tl][i];
        dSc[i] += doi * rk;
        p_dr += St[i] * doi;
        p_dk += dSc[i] * sm.vt[tl][i];
        p_db += dSc[i] * sm.sa[tl][i];
        p_dd += dSc[i] * Sp[i];
      }
      __syncthreads();   // dsa of this token visible to every thread
      float p_da = 0.f;
#pragma unroll
      for (int i = 0; i < VS; ++i) {
        const float ds = sm.dsa[buf][i];
        p_da += Sp[i] * ds;
        dSc[i] = dSc[i] * dk_ + ds * ak;
        St[i] = Sp[i];
      }
      const float dsr = sm.dsa[buf][vl];
#pragma unroll
      for (int j = 0; j < 16; ++j) dSr[j] = dSr[j] * td[j] + dsr * ta[j];
      sm.part[pb][tl][0][kc] = p_dr;
      sm.part[pb][tl][1][kc] = p_dk;
      sm.part[pb][tl][2][kc] = p_db;
      sm.part[pb][tl][3][kc] = p_da;
      sm.part[pb][tl][4][kc] = p_dd;
    }
    // ---- dv rows of this CTA
    __syncthreads();
    for (int i = tid; i < nt * VS; i += N) {
      const int tl = i >> 4, vi = i & 15;
      dv[base + (long long)(t0 + tl) * lay.st + y * VS + vi] = from_f32<T>(sm.dvt[tl][vi]);
    }
    // ---- sum the four CTAs' partial column results; this CTA finishes tokens tl = y, y+NQ, ...
    cluster.sync();
    for (int tl = y; tl < nt; tl += NQ) {
      float acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int rk_ = 0; rk_ < NQ; ++rk_) {
        const float* rp = cluster.map_shared_rank(&sm.part[pb][tl][0][0], rk_);
#pragma unroll
        for (int qn = 0; qn < 5; ++qn) acc[qn] += rp[qn * N + kc];
      }
      const long long off = base + (long long)(t0 + tl) * lay.st + kc;
      dr[off] = from_f32<T>(acc[0]);
      dk[off] = from_f32<T>(acc[1]);
      db[off] = from_f32<T>(acc[2]);
      da[off] = from_f32<T>(acc[3]);
      dw[off] = from_f32<T>(acc[4] * sm.tile[tl][1][padk(kc)] * (-sm.tile[tl][2][padk(kc)]));
    }
    // part[pb] is rewritten two chunks later, after the next chunk's cluster.sync(); the tile is
    // rewritten by the next chunk's staging, which only this CTA reads
    __syncthreads();
  }
  if (d_h0) {
    float* p = d_h0 + ((long long)unit * N + (y * VS + vl)) * N + 16 * kq;
#pragma unroll
    for (int j = 0; j < 16; ++j) p[j] = dSr[j];
  }
  cluster.sync();   // no CTA leaves while a peer may still read its shared memory
}

}  // namespace

int launch_rwkv7_rec_step(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                          const float* h0, int n_state, void* o, float* ht, int B, int H, int dtype, cudaStream_t st) {
  constexpr int N = 128;
  const TokLayout lay(1, H, 0, N);
  ProfScope prof("rwkv7_rec_fwd_kernel", st);
  RWKVB200_DISPATCH_DTYPE(dtype,
    const FwdArgs<T> args{(const T*)r, (const T*)w, (const T*)k, (const T*)v, (const T*)a, (const T*)b, 0, lay.st, 1,
                          nullptr, (T*)o, nullptr, nullptr};
    // (a tile of one token: 256 sequences of 16 heads 317 -> 134 us against a tile of 8)
    return launch(rwkv7_rec_fwd_kernel<T, N, 1>, dim3(B * H, N / VS), N, 0, st, 1, args, h0, n_state, ht, H, lay));
  return RWKVB200_OK;
}

int launch_rwkv7_rec_fwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                         const float* h0, int n_state, void* o, float* ht, int B, int Tn, int H, int head_first,
                         cudaStream_t st) {
  typedef __nv_bfloat16 T;
  const TokLayout lay(Tn, H, head_first);
  ProfScope prof("rwkv7_rec_fwd_kernel", st);
  const FwdArgs<T> args{(const T*)r, (const T*)w, (const T*)k, (const T*)v, (const T*)a, (const T*)b, 0, lay.st, Tn,
                        nullptr, (T*)o, nullptr, nullptr};
  // tiles of 8 tokens: with 16, half as many CTAs fit an SM (B 16, T 512, 32 heads: 2269 us against 1281; 16 units 320 and 324)
  return launch(rwkv7_rec_fwd_kernel<T, HS, 8>, dim3(B * H, HS / VS), HS, 0, st, 1, args, h0, n_state, ht, H, lay);
}

int launch_rwkv7_rec_bwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                         const float* h0, int n_state, const void* d_o, const float* d_ht, float* ckpt,
                         void* dr, void* dw, void* dk, void* dv, void* da, void* db, float* d_h0,
                         int B, int Tn, int H, int head_first, cudaStream_t st, const UnitSel& sel, int T_total) {
  typedef __nv_bfloat16 T;
  constexpr int N = HS;
  const TokLayout lay(T_total ? T_total : Tn, H, head_first);
  ProfScope prof("rwkv7_rec_bwd_kernel", st);
  const int smem = (int)sizeof(BwdSmem<N>);
  DeviceFacts dev;
  if (int e = device_facts(&dev)) return e;
  if (allow_smem<rwkv7_rec_bwd_kernel<T, N>>(dev, smem)) return RWKVB200_E_CUDA;
  // a cluster: the CTAs of a unit exchange partial sums
  return launch(rwkv7_rec_bwd_kernel<T, N>, dim3(B * H, N / VS), N, smem, st, N / VS, (const T*)r, (const T*)w, (const T*)k,
                (const T*)v, (const T*)a, (const T*)b, (const T*)d_o, d_ht, h0, n_state, ckpt, (T*)dr, (T*)dw, (T*)dk, (T*)dv,
                (T*)da, (T*)db, d_h0, Tn, H, lay, sel);
}

}  // namespace rwkvb200
