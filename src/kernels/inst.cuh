// Kernel entry points for one element type; included by one .cu file per type so the types
// compile in parallel.
#pragma once
#include "kernels/coll_body.cuh"
#include "kernels/roles_body.cuh"
#include "kernels/ring_body.cuh"
#include "kernels/ll_body.cuh"
#include "kernels/launch.h"

namespace hx {

// World form: the argument blocks of all ranks travel as one kernel parameter (at most 16 x 0.9 KB,
// of the 32 KB a launch may carry). Staged through device memory they cost a stream
// synchronisation (an earlier launch might still read the buffer) and a pageable copy per call:
// 8 ranks, 41 KB bf16: 34.3 us a call staged, 22.6 us as parameters; 8 ranks, 8 B: 19.0 and 15.2 us.
// Kernels compiled for up to kN ranks carry kN blocks; the others (kN = 0: the copies, the ring, and the
// folds' and lines' general forms) carry sixteen.
template <typename Args, int kN = 0>
struct WorldArgs {
  Args rank[kN ? kN : kMaxRanks];
};

// kN: the rank count the fold is unrolled for (see cta_fold, fold.cuh); HX_BY_RANKS picks it.
template <typename T, int kN>
__global__ void __launch_bounds__(512) k_xchg_fold(const __grid_constant__ XchgArgs a) {
  __shared__ FoldShared sh;
  xchg_body<T, true, kN>(a, blockIdx.x, gridDim.x, sh);
}
template <typename T, int kN>
__global__ void __launch_bounds__(512) k_xchg_fold_world(const __grid_constant__ WorldArgs<XchgArgs, kN> a) {
  __shared__ FoldShared sh;
  xchg_body<T, true, kN>(a.rank[blockIdx.y], blockIdx.x, gridDim.x, sh);
}
template <typename T, int kN>
__global__ void __launch_bounds__(512) k_twoshot(const __grid_constant__ TwoShotArgs a) {
  __shared__ FoldShared sh;
  twoshot_body<T, kN>(a, blockIdx.x, gridDim.x, sh);
}
template <typename T, int kN>
__global__ void __launch_bounds__(512) k_twoshot_world(const __grid_constant__ WorldArgs<TwoShotArgs, kN> a) {
  __shared__ FoldShared sh;
  twoshot_body<T, kN>(a.rank[blockIdx.y], blockIdx.x, gridDim.x, sh);
}

// fp32 buffers, T on the wire (instantiated for fp16 and bf16 only)
template <typename T, int kN>
__global__ void __launch_bounds__(512) k_twoshot_cast(const __grid_constant__ TwoShotArgs a) {
  __shared__ FoldShared sh;
  twoshot_body<T, kN, true>(a, blockIdx.x, gridDim.x, sh);
}
template <typename T, int kN>
__global__ void __launch_bounds__(512) k_twoshot_cast_world(const __grid_constant__ WorldArgs<TwoShotArgs, kN> a) {
  __shared__ FoldShared sh;
  twoshot_body<T, kN, true>(a.rank[blockIdx.y], blockIdx.x, gridDim.x, sh);
}

template <typename T, int kN>
__global__ void __launch_bounds__(512) k_twoshot_roles(const __grid_constant__ TwoShotArgs a) {
  __shared__ FoldShared sh;
  twoshot_roles_body<T, kN>(a, blockIdx.x, gridDim.x, sh);
}
template <typename T, int kN>
__global__ void __launch_bounds__(512) k_twoshot_roles_world(const __grid_constant__ WorldArgs<TwoShotArgs, kN> a) {
  __shared__ FoldShared sh;
  twoshot_roles_body<T, kN>(a.rank[blockIdx.y], blockIdx.x, gridDim.x, sh);
}

template <typename T>
__global__ void __launch_bounds__(512) k_ring(const __grid_constant__ TwoShotArgs a) {
  __shared__ FoldShared sh;
  ring_body<T>(a, blockIdx.x, gridDim.x, sh);
}
template <typename T>
__global__ void __launch_bounds__(512, 2) k_ring_world(const __grid_constant__ WorldArgs<TwoShotArgs> a) {
  __shared__ FoldShared sh;
  ring_body<T>(a.rank[blockIdx.y], blockIdx.x, gridDim.x, sh);
}

template <typename T, int kN>
__global__ void __launch_bounds__(256, 1) k_ll(const __grid_constant__ LLArgs a) {
  __shared__ FoldShared sh;
  ll_body<T, kN>(a, blockIdx.x, gridDim.x, sh);
}
template <typename T, int kN>
__global__ void __launch_bounds__(256, 1) k_ll_world(const __grid_constant__ WorldArgs<LLArgs, kN> a) {
  __shared__ FoldShared sh;
  ll_body<T, kN>(a.rank[blockIdx.y], blockIdx.x, gridDim.x, sh);
}

template <int kN = 0, typename Args>
cudaError_t launch_world(const void* kernel, const Args* args, LaunchShape s, cudaStream_t st) {
  static_assert(sizeof(WorldArgs<Args, kN>) <= 32764, "kernel parameters");
  if (s.world > (kN ? kN : kMaxRanks)) return cudaErrorInvalidValue;
  WorldArgs<Args, kN> all;  // blocks of ranks that do not exist stay unset: no CTA reads them
  memcpy(all.rank, args, sizeof(Args) * size_t(s.world));
  void* params[] = {&all};
  return cudaLaunchCooperativeKernel(kernel, dim3(s.ctas, s.world), dim3(s.threads), params, 0, st);
}

// Launches KERNEL<T, kN>, or KERNEL_world<T, kN> for a world, for the rank count of args[0].
#define HX_LAUNCH_RANKS(KERNEL, KN)                                                                       \
  if (s.world) return launch_world<KN>(reinterpret_cast<const void*>(&KERNEL##_world<T, KN>), args, s, st); \
  KERNEL<T, KN><<<s.ctas, s.threads, 0, st>>>(*args);                                                     \
  return cudaGetLastError()
#define HX_BY_RANKS(KERNEL)                                                          \
  const int n = args[0].w.n;                                                         \
  if (n == 2) { HX_LAUNCH_RANKS(KERNEL, 2); }                                        \
  if (n == 3 || n == 4) { HX_LAUNCH_RANKS(KERNEL, 4); }                              \
  if (n > 4 && n <= kFastRanks) { HX_LAUNCH_RANKS(KERNEL, 8); }                      \
  HX_LAUNCH_RANKS(KERNEL, 0)

template <typename T>
cudaError_t launch_xchg_fold_t(const XchgArgs* args, LaunchShape s, cudaStream_t st) {
  HX_BY_RANKS(k_xchg_fold);
}
template <typename T>
cudaError_t launch_twoshot_t(const TwoShotArgs* args, LaunchShape s, cudaStream_t st) {
  HX_BY_RANKS(k_twoshot);
}
template <typename T>
cudaError_t launch_twoshot_cast_t(const TwoShotArgs* args, LaunchShape s, cudaStream_t st) {
  HX_BY_RANKS(k_twoshot_cast);
}
template <typename T>
cudaError_t launch_twoshot_roles_t(const TwoShotArgs* args, LaunchShape s, cudaStream_t st) {
  HX_BY_RANKS(k_twoshot_roles);
}

template <typename T>
cudaError_t launch_ring_t(const TwoShotArgs* args, LaunchShape s, cudaStream_t st) {
  if (s.world) return launch_world(reinterpret_cast<const void*>(&k_ring_world<T>), args, s, st);
  k_ring<T><<<s.ctas, s.threads, 0, st>>>(*args);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_ll_t(const LLArgs* args, LaunchShape s, cudaStream_t st) {
  const int n = args[0].w.n;  // loops of a fixed length for 2, 4 and 8 ranks only
  if (n == 2) { HX_LAUNCH_RANKS(k_ll, 2); }
  if (n == 4) { HX_LAUNCH_RANKS(k_ll, 4); }
  if (n == 8) { HX_LAUNCH_RANKS(k_ll, 8); }
  HX_LAUNCH_RANKS(k_ll, 0);
}

// ---- standalone elementwise kernels --------------------------------------------------------
template <typename T>
__global__ void k_reduce(T* dst, const T* src, size_t n, int op) {
  constexpr int V = 16 / sizeof(T);
  const size_t tid = blockIdx.x * size_t(blockDim.x) + threadIdx.x, nth = size_t(gridDim.x) * blockDim.x;
  const bool aligned = ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15u) == 0;
  const size_t nvec = aligned ? n / V : 0;
  for (size_t v = tid; v < nvec; v += nth) {
    Vec16<T> a, b;
    a.raw = ld16(reinterpret_cast<const char*>(dst) + (v << 4));
    b.raw = ld16(reinterpret_cast<const char*>(src) + (v << 4));
    st16(reinterpret_cast<char*>(dst) + (v << 4), combine_lanes(a, b, op).raw);
  }
  for (size_t e = nvec * V + tid; e < n; e += nth) dst[e] = apply(dst[e], src[e], op);
}
// dst = src * scalar; also the whole of an AllReduce over one rank that scales (Avg of floats,
// PreMulSum). Bound by memory: warps take runs of four times 512 bytes, so that a thread has four loads
// in flight. 28 MB fp32 in place (it stays in L2): 8.9 us; as a one-rank two-shot launch, whose
// fold goes element by element for one rank and which ends in a hand-shake, 61.6 us.
template <typename T>
__global__ void __launch_bounds__(256) k_scale(T* dst, const T* src, size_t n, unsigned long long scalar_bits,
                                               const void* scalar_ptr) {
  T k;
  if (scalar_ptr) k = *static_cast<const T*>(scalar_ptr);
  else memcpy(&k, &scalar_bits, sizeof(T));
  constexpr int V = 16 / sizeof(T), U = 4;
  const size_t tid = blockIdx.x * size_t(blockDim.x) + threadIdx.x, nth = size_t(gridDim.x) * blockDim.x;
  const bool aligned = ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15u) == 0;
  const size_t nvec = aligned ? n / V : 0;
  for (size_t v = (tid >> 5) * (32 * U) + (tid & 31u); v < nvec; v += nth * U) {
    const char* from = reinterpret_cast<const char*>(src) + (v << 4);
    char* to = reinterpret_cast<char*>(dst) + (v << 4);
    Vec16<T> a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) a[u].raw = ld16_if(v + u * 32 < nvec, from + u * 512);
#pragma unroll
    for (int u = 0; u < U; ++u) st16_if(v + u * 32 < nvec, to + u * 512, scale_lanes(a[u], k).raw);
  }
  for (size_t e = nvec * V + tid; e < n; e += nth) dst[e] = scale(src[e], k);
}
template <typename T>
__global__ void k_divide(T* buf, size_t n, int divisor) {
  const size_t tid = blockIdx.x * size_t(blockDim.x) + threadIdx.x, nth = size_t(gridDim.x) * blockDim.x;
  for (size_t e = tid; e < n; e += nth) buf[e] = div_trunc(buf[e], divisor);
}

inline int elementwise_grid(size_t count, int per_thread) {
  size_t blocks = (count / per_thread + 255) / 256;
  if (blocks < 1) blocks = 1;
  if (blocks > 148 * 16) blocks = 148 * 16;  // persistent-style: 16 CTAs per SM, grid-stride
  return static_cast<int>(blocks);
}
template <typename T>
cudaError_t launch_reduce_t(void* dst, const void* src, size_t count, int op, cudaStream_t st) {
  k_reduce<T><<<elementwise_grid(count, 16 / sizeof(T)), 256, 0, st>>>(
      static_cast<T*>(dst), static_cast<const T*>(src), count, op);
  return cudaGetLastError();
}
template <typename T>
cudaError_t launch_scale_t(void* dst, const void* src, size_t count, unsigned long long bits,
                           const void* scalar_ptr, cudaStream_t st) {
  // off the 16-byte grid the kernel goes element by element: a thread for each, not for each run of vectors
  // (16 KiB e4m3 at an odd address, in place: 8.3 us a call on one B200, 23.0 with the vectors' grid)
  const bool vectors = ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15u) == 0;
  k_scale<T><<<elementwise_grid(count, vectors ? 4 * 16 / sizeof(T) : 1), 256, 0, st>>>(
      static_cast<T*>(dst), static_cast<const T*>(src), count, bits, scalar_ptr);
  return cudaGetLastError();
}
template <typename T>
cudaError_t launch_divide_t(void* buf, size_t count, int divisor, cudaStream_t st) {
  k_divide<T><<<elementwise_grid(count, 1), 256, 0, st>>>(static_cast<T*>(buf), count, divisor);
  return cudaGetLastError();
}

#define HX_INSTANTIATE_TYPE(T)                                                               \
  template cudaError_t launch_xchg_fold_t<T>(const XchgArgs*, LaunchShape, cudaStream_t);    \
  template cudaError_t launch_twoshot_t<T>(const TwoShotArgs*, LaunchShape, cudaStream_t);   \
  template cudaError_t launch_twoshot_roles_t<T>(const TwoShotArgs*, LaunchShape, cudaStream_t); \
  template cudaError_t launch_ring_t<T>(const TwoShotArgs*, LaunchShape, cudaStream_t);      \
  template cudaError_t launch_ll_t<T>(const LLArgs*, LaunchShape, cudaStream_t);             \
  template cudaError_t launch_reduce_t<T>(void*, const void*, size_t, int, cudaStream_t);    \
  template cudaError_t launch_scale_t<T>(void*, const void*, size_t, unsigned long long,     \
                                         const void*, cudaStream_t);                         \
  template cudaError_t launch_divide_t<T>(void*, size_t, int, cudaStream_t);

}  // namespace hx
