// Shared helpers for the rwkv_ops_b200 kernels: element-type conversion, vector loads,
// argument checks.  Everything computes in float32; token tensors may be f32, bf16 or f16.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <utility>

#include "../../include/rwkv_ops_b200.h"

namespace rwkvb200 {

constexpr int HS = 64;  // head size (key and value)

template <typename T> __device__ __forceinline__ float to_f32(T x);
template <> __device__ __forceinline__ float to_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <> __device__ __forceinline__ float to_f32<__half>(__half x) { return __half2float(x); }

template <typename T> __device__ __forceinline__ T from_f32(float x);
template <> __device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ __half from_f32<__half>(float x) { return __float2half_rn(x); }

// Load four consecutive elements (16-byte aligned for f32, 8-byte for 16-bit types) as float4.
template <typename T> __device__ __forceinline__ float4 load4(const T* p);
template <> __device__ __forceinline__ float4 load4<float>(const float* p) {
  return __ldg(reinterpret_cast<const float4*>(p));
}
template <> __device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
  uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
  float4 f;
  f.x = __uint_as_float(u.x << 16);
  f.y = __uint_as_float(u.x & 0xffff0000u);
  f.z = __uint_as_float(u.y << 16);
  f.w = __uint_as_float(u.y & 0xffff0000u);
  return f;
}
template <> __device__ __forceinline__ float4 load4<__half>(const __half* p) {
  uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
  __half2 h0 = *reinterpret_cast<__half2*>(&u.x), h1 = *reinterpret_cast<__half2*>(&u.y);
  float2 a = __half22float2(h0), b = __half22float2(h1);
  return make_float4(a.x, a.y, b.x, b.y);
}

// The same from shared memory (load4 reads through the read-only global path and must not be given a
// shared-memory address).
template <typename T> __device__ __forceinline__ float4 load4_shared(const T* p);
template <> __device__ __forceinline__ float4 load4_shared<float>(const float* p) {
  return *reinterpret_cast<const float4*>(p);
}
template <> __device__ __forceinline__ float4 load4_shared<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u),
                     __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
template <> __device__ __forceinline__ float4 load4_shared<__half>(const __half* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
  const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// Store four consecutive elements from a float4 (same alignment rule as load4).
template <typename T> __device__ __forceinline__ void store4(T* p, float4 f);
template <> __device__ __forceinline__ void store4<float>(float* p, float4 f) {
  *reinterpret_cast<float4*>(p) = f;
}
template <> __device__ __forceinline__ void store4<__nv_bfloat16>(__nv_bfloat16* p, float4 f) {
  __nv_bfloat162 lo = __floats2bfloat162_rn(f.x, f.y), hi = __floats2bfloat162_rn(f.z, f.w);
  uint2 u;
  u.x = *reinterpret_cast<uint32_t*>(&lo);
  u.y = *reinterpret_cast<uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(p) = u;
}
template <> __device__ __forceinline__ void store4<__half>(__half* p, float4 f) {
  __half2 lo = __floats2half2_rn(f.x, f.y), hi = __floats2half2_rn(f.z, f.w);
  uint2 u;
  u.x = *reinterpret_cast<uint32_t*>(&lo);
  u.y = *reinterpret_cast<uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(p) = u;
}

// Four consecutive elements of an array that holds T (`typed`) or float32.
template <typename T> __device__ __forceinline__ float4 load4_as(const void* p, long long i, bool typed) {
  return typed ? load4(static_cast<const T*>(p) + i) : load4(static_cast<const float*>(p) + i);
}
template <typename T> __device__ __forceinline__ void store4_as(void* p, long long i, bool typed, float4 f) {
  if (typed) store4(static_cast<T*>(p) + i, f); else store4(static_cast<float*>(p) + i, f);
}

// The decay every operator applies to its w input.
__device__ __forceinline__ float decay_of(float w) { return expf(-expf(w)); }

// Strides (in elements) of a [B,T,H,64] or [B,H,T,64] token tensor.
struct TokLayout {
  long long sb, st, sh;
  __host__ __device__ TokLayout(int T, int H, int head_first, int hs = HS) {
    sb = (long long)T * H * hs;
    if (head_first) { sh = (long long)T * hs; st = hs; }
    else            { sh = hs;                st = (long long)H * hs; }
  }
};

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Last CUDA runtime error seen by this library (cudaSuccess if none); see rwkvb200_last_cuda_error().
int& last_cuda_error_slot();

inline int cuda_ok(cudaError_t e) {
  if (e == cudaSuccess) return RWKVB200_OK;
  last_cuda_error_slot() = (int)e;
  return RWKVB200_E_CUDA;
}

inline int check_launch() { return cuda_ok(cudaGetLastError()); }

// What a launch needs to know about the current device, asked once per device (tc_host.cu): a call launches up to nine
// kernels, and the attribute queries and settings between them were a third of its host time.
struct DeviceFacts { int dev, sms; int* status; };      // status: the device status word of the kernels' bounded waits
int device_facts(DeviceFacts* out);

// Allow `Kernel` its dynamic shared memory, once per device.
template <auto Kernel>
int allow_smem(const DeviceFacts& f, int bytes) {
  static std::atomic<uint64_t> done{0};
  const uint64_t bit = uint64_t(1) << f.dev;
  if (done.load(std::memory_order_acquire) & bit) return RWKVB200_OK;
  if (cuda_ok(cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes))) return RWKVB200_E_CUDA;
  done.fetch_or(bit, std::memory_order_release);
  return RWKVB200_OK;
}

// How many clusters of `ctas` CTAs of `Kernel` (2, 4 or 8, along y) the device holds at once, asked once per device and size; a
// cluster's CTAs share a group of SMs, so this can be less than the SMs alone would allow.
template <auto Kernel>
int resident_clusters(const DeviceFacts& f, int threads, int smem, int ctas) {
  static std::atomic<int> known[64][3];      // plus one
  std::atomic<int>& slot = known[f.dev][ctas == 2 ? 0 : ctas == 4 ? 1 : 2];
  int n = slot.load(std::memory_order_acquire);
  if (!n) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, ctas);
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 1; attr.val.clusterDim.y = ctas; attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, Kernel, &cfg) != cudaSuccess) { (void)cudaGetLastError(); fit = 0; }
    n = fit + 1;
    slot.store(n, std::memory_order_release);
  }
  return n - 1;
}

// Whether a block's dynamic shared memory starts 1024-byte aligned, as swizzled tiles need it: it follows what the system
// reserves and the kernel's static arrays.
inline bool smem_starts_aligned(int reserved, int static_bytes) { return (reserved + static_bytes) % 1024 == 0; }
// The same for `Kernel` on the current device, asked once per device: RWKVB200_E_UNSUPPORTED where it does not.  For a kernel
// that has no room to align by hand; without this its own check would leave the outputs unwritten.
template <auto Kernel>
int need_aligned_smem(const DeviceFacts& f) {
  static std::atomic<int> known[64];      // 1: yes, 2: no
  int n = known[f.dev].load(std::memory_order_acquire);
  if (!n) {
    int reserved = 0;
    cudaFuncAttributes a;
    if (cuda_ok(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, f.dev)) ||
        cuda_ok(cudaFuncGetAttributes(&a, Kernel)))
      return RWKVB200_E_CUDA;
    n = smem_starts_aligned(reserved, (int)a.sharedSizeBytes) ? 1 : 2;
    known[f.dev].store(n, std::memory_order_release);
  }
  return n == 1 ? RWKVB200_OK : RWKVB200_E_UNSUPPORTED;
}

// The kernels of the library (but where a launch says why not) are launched so that their blocks may come onto the SMs while the kernel before runs
// out: what they do before earlier_kernels_done() (barriers, TMEM) overlaps with its last blocks, and so does the launch
// itself.  No kernel touches global memory before that call but to prefetch into L2, every thread makes it, and it returns when all earlier
// kernels have completed.  later_kernels_may_start() lets the next kernel's blocks come once all blocks of this one have
// called it; a kernel that allocates TMEM calls it after the allocation, so that blocks of the next one, which wait for
// this one, never hold TMEM that a block of this one still needs.
// (1 prompt of 1000 tokens, 32 heads, two kernels: 2.2 us between two kernels before.)
__device__ __forceinline__ void earlier_kernels_done() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void later_kernels_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// cluster_y: CTAs of a cluster along y; 0: none, and the kernel starts when all earlier ones have completed.  (Blocks that come
// early take the SMs that are free first, as many of them as fit, and leave others without any.)
template <typename... P, typename... A>
int launch(void (*kernel)(P...), dim3 grid, dim3 block, int smem, cudaStream_t st, int cluster_y, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = cluster_y; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster_y > 1 ? 2 : cluster_y;
  const int e = cuda_ok(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
  return e ? e : check_launch();
}

// Brackets one kernel launch with timing events when profiling is on (see profile.cu).
struct ProfScope {
  ProfScope(const char* name, cudaStream_t st);
  ~ProfScope();
  cudaStream_t st_;
  int idx_;
};

// Host-side dispatch on the dtype code.
#define RWKVB200_DISPATCH_DTYPE(dtype, ...)                                  \
  switch (dtype) {                                                           \
    case RWKVB200_F32:  { using T = float;          __VA_ARGS__; break; }    \
    case RWKVB200_BF16: { using T = __nv_bfloat16;  __VA_ARGS__; break; }    \
    case RWKVB200_F16:  { using T = __half;         __VA_ARGS__; break; }    \
    default: return RWKVB200_E_DTYPE;                                        \
  }

// Which (batch, head) units a recurrent kernel works on, and where their tokens and checkpoints lie.  The
// recurrent kernels double as the exact fallback of the chunked tensor-core paths: a chunked kernel marks
// the units whose decay leaves the range its scaled operands can represent, and the recurrent kernel is
// then launched over all units with `flags` set, so that only the marked ones run.
struct UnitSel {
  const int* flags;             // one entry per unit, nonzero = run it; nullptr = run every unit
  const int* seq_start;         // packed variable-length batch: first token and length of every sequence
  const int* seq_len;           //   (all in batch row 0); nullptr = dense batch
  long long ckpt_unit_stride;   // floats between the checkpoint regions of consecutive units; 0 = dense
};

// Kernel launchers implemented in the .cu files (internal linkage across the library only).
int launch_rwkv7_decode_step(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                             void* state, int state_dtype, void* o, int B, int H, int dtype, cudaStream_t st);
int launch_rwkv7_step(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                      const float* s_in, int n_state, float* s_out, void* o, int B, int H, int dtype,
                      cudaStream_t st);

// One token of the float32 recurrence at head size 128.
int launch_rwkv7_rec_step(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                          const float* h0, int n_state, void* o, float* ht, int B, int H, int dtype, cudaStream_t st);
// The token-by-token recurrence, bfloat16 at head size 64.  Backward: over the units marked in sel.flags, or all of a dense
// batch; ckpt: sel.ckpt_unit_stride floats of scratch per unit (0: dense), 4096 for every R7_CKPT tokens.
int launch_rwkv7_rec_fwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                         const float* h0, int n_state, void* o, float* ht, int B, int Tn, int H, int head_first,
                         cudaStream_t st);
int launch_rwkv7_rec_bwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                         const float* h0, int n_state, const void* d_o, const float* d_ht, float* ckpt,
                         void* dr, void* dw, void* dk, void* dv, void* da, void* db, float* d_h0,
                         int B, int Tn, int H, int head_first, cudaStream_t st, const UnitSel& sel, int T_total);
// Float32 recurrence over blocks of tokens (rwkv7_block.cu), head size 64 or 128; o and ht may be NULL.  ckpt: room for
// a state every R7_CKPT tokens of each unit.  states (may be NULL): rwkv7_block_states_bytes of memory in which the forward
// leaves the states its backward starts from; a backward that is given them needs only as much for ckpt.
size_t rwkv7_block_states_bytes(int B, int Tn, int H, int dtype, int head_size);
// scratch (may be NULL: slower): this much memory for what a sweep over the blocks needs besides the state.
size_t rwkv7_block_scratch_bytes(int B, int Tn, int H, int dtype, int head_size);
int launch_rwkv7_block_fwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                           const float* h0, int n_state, void* o, float* ht, int B, int Tn, int H, int dtype,
                           int head_first, cudaStream_t st, int head_size = HS, float* states = nullptr, void* scratch = nullptr);
int launch_rwkv7_block_bwd(const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                           const float* h0, int n_state, const void* d_o, const float* d_ht, float* ckpt,
                           void* dr, void* dw, void* dk, void* dv, void* da, void* db, float* d_h0, int B, int Tn, int H,
                           int dtype, int head_first, cudaStream_t st, int head_size = HS, const float* states = nullptr,
                           void* scratch = nullptr);
constexpr int R7_CKPT = 8;   // tokens between state checkpoints of the recurrent backward

int launch_wkv6_fwd(const void* r, const void* k, const void* v, const void* w, const void* u,
                    const void* s0, int n_state, const int32_t* smap, void* y, void* sT,
                    float* ckpt, int B, int Tn, int H, int dtype, cudaStream_t st, const UnitSel* sel = nullptr,
                    int ckpt_every = 0, int head_size = HS, bool typed = false);
int launch_wkv6_bwd_coarse(const void* r, const void* k, const void* v, const void* w, const float* u,
                           const void* d_y, const float* d_sT, const float* ckpt,
                           void* dr, void* dk, void* dv, void* dw, float* du_partial, float* d_s0,
                           int B, int Tn, int H, int dtype, cudaStream_t st, const UnitSel* sel);
int launch_wkv6_du_reduce_mixed(const float* part_chunked, const float* part_rec, const int* flags, float* du,
                                int B, int H, cudaStream_t st, int rows = 1);
int launch_wkv6_bwd(const void* r, const void* k, const void* v, const void* w, const float* u,
                    const void* d_y, const float* d_sT, const float* ckpt,
                    void* dr, void* dk, void* dv, void* dw, float* du_partial, float* du, float* d_s0,
                    int B, int Tn, int H, int dtype, cudaStream_t st, int head_size = HS);
constexpr int W6_CKPT = 8;

// `typed`: u, s0 and sT hold the token dtype instead of float32.
// Chunked tcgen05 wkv6 (wkv6_chunked.cu).  `states` (may be NULL) receives the fp32 state at every chunk
// boundary, [B*H][ceil(T/64)+1][64][64].
int launch_wkv6_chunked_fwd(const void* r, const void* k, const void* v, const void* w, const void* u,
                            const void* s0, int n_state, const int32_t* smap, void* y, void* sT,
                            float* states, int* flags, float* handoff, int* hflags, int B, int Tn, int H, int dtype,
                            cudaStream_t st, const int32_t* seq_start = nullptr, const int32_t* seq_len = nullptr,
                            int T_total = 0, bool typed = false);
size_t wkv6_chunked_fwd_scratch_bytes(int B, int H);
void wkv6_chunked_fwd_scratch(void* workspace, int B, int H, int** flags, float** handoff, int** hflags);
void wkv6_chunked_workspace_parts(void* workspace, int B, int Tn, int H, int** flags, float** handoff, int** hflags);
size_t wkv6_chunked_bwd_workspace_bytes(int B, int Tn, int H);
size_t wkv6_chunked_flags_bytes(int B, int H);
int launch_wkv6_chunked_bwd(const void* r, const void* k, const void* v, const void* w, const float* u,
                            const float* s0, int n_state, const int32_t* smap, const void* d_y, const float* d_sT,
                            void* dr, void* dk, void* dv, void* dw, float* du, float* d_s0, void* workspace,
                            int B, int Tn, int H, int dtype, bool kept, cudaStream_t st,
                            const int32_t* seq_start = nullptr, const int32_t* seq_len = nullptr, int T_total = 0);

}  // namespace rwkvb200
