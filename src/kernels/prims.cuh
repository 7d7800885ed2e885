// Device-side building blocks: system-scope flag accesses, bounded waits, vector copies.
#pragma once
#include <cstdint>
#include <type_traits>

#include "device/proto.h"
#include "math/elem.h"

namespace hx {

__device__ __forceinline__ unsigned long long ld_acquire_sys(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed_sys(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed_sys(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned long long* flag_at(char* win, size_t base, int cta, int src) {
  return reinterpret_cast<unsigned long long*>(win + base) + size_t(cta) * kMaxRanks + src;
}

// Records a sticky failure and tells every peer to stop waiting.
__device__ inline void raise_failure(const WinView& w, unsigned code, unsigned long long detail) {
  const unsigned long long word = (static_cast<unsigned long long>(code) << 56) | (detail & 0xffffffffffffffull);
  atomicCAS(w.status, 0ull, word);
  for (int p = 0; p < w.n; ++p)
    if (p != w.rank)
      st_relaxed_sys(reinterpret_cast<unsigned long long*>(w.win[p] + kOffAbort), 1ull);
  __threadfence_system();
}

// Spins until *flag >= want. Gives up when the limit passes (timeout) or a peer raised this
// window's abort word (remote failure). Returns true on success.
__device__ inline bool wait_flag(const WinView& w, const unsigned long long* flag,
                                 unsigned long long want, int peer) {
  if (ld_acquire_sys(flag) >= want) return true;
  const unsigned long long t0 = now_ns();
  const unsigned long long* abort_word =
      reinterpret_cast<const unsigned long long*>(w.win[w.rank] + kOffAbort);
  for (unsigned spins = 1;; ++spins) {
    if (ld_acquire_sys(flag) >= want) return true;
    if ((spins & 63u) == 0) {
      if (ld_relaxed_sys(abort_word) != 0) {
        atomicCAS(w.status, 0ull, (static_cast<unsigned long long>(kStatRemote) << 56) | unsigned(peer));
        return false;
      }
      if (now_ns() - t0 > w.wait_ns) {
        raise_failure(w, kStatTimeout, unsigned(peer));
        return false;
      }
    }
  }
}

// Hand-over between ranks, called by every thread of the CTA. signal_all: threads 0..n-1 each
// tell one peer "my stores up to here are in your window" (the CTA's stores are fenced first).
// wait_all: the same threads wait for their peer's signal of `epoch`; false (to all threads)
// when any wait gave up.
__device__ inline void signal_all(const WinView& w, size_t flag_base, int cta, unsigned long long epoch) {
  __syncthreads();
  const int t = threadIdx.x;
  // st.release.sys orders the flag after every store the CTA made before the barrier above
  // (release is cumulative over what the barrier made visible to this thread); no separate
  // fence.sc is needed, and it is expensive at system scope
  if (t < w.n && t != w.rank) st_release_sys(flag_at(w.win[t], flag_base, cta, w.rank), epoch);
}
__device__ inline bool wait_all(const WinView& w, size_t flag_base, int cta, unsigned long long epoch,
                                int* sh_fail) {
  const int t = threadIdx.x;
  if (t < w.n && t != w.rank)
    if (!wait_flag(w, flag_at(w.win[w.rank], flag_base, cta, t), epoch, t)) *sh_fail = 1;
  __syncthreads();
  return *sh_fail == 0;
}
__device__ inline bool signal_and_wait(const WinView& w, size_t flag_base, int cta,
                                       unsigned long long epoch, int* sh_fail) {
  signal_all(w, flag_base, cta, epoch);
  return wait_all(w, flag_base, cta, epoch, sh_fail);
}

// Where step k of a launch stages its data. A single-step launch uses the half picked by its
// epoch's parity (see proto.h). A multi-step launch owns the whole staging area between its
// entry hand-shake and its closing one and cycles through kRing buffers, so that step k+1 can
// be pushed while step k is still being consumed.
constexpr int kRing = 4;
struct Staging {
  size_t base0, buf_bytes;
  int ring;
  __device__ Staging(const WinView& w, unsigned long long epoch0, int steps) {
    if (steps == 1) {
      base0 = w.half_off[epoch0 & 1];
      buf_bytes = w.half_bytes;
      ring = 1;
    } else {
      base0 = w.half_off[0];
      buf_bytes = (2 * w.half_bytes / kRing) & ~size_t(255);
      ring = kRing;
    }
  }
  __device__ size_t at(int step) const { return base0 + size_t(step % ring) * buf_bytes; }
};

// Phase timer of one CTA (see WinView::trace). lap(slot) adds the time since the previous lap.
struct PhaseTimer {
  unsigned long long* acc;
  unsigned long long last, first;
  __device__ PhaseTimer(const WinView& w, int cta) : acc(nullptr), last(0), first(0) {
    if (w.trace && threadIdx.x == 0) {
      acc = w.trace + size_t(cta) * kTraceSlots;
      last = first = now_ns();
    }
  }
  __device__ __forceinline__ void lap(int slot) {
    if (acc) {
      const unsigned long long t = now_ns();
      acc[slot] += t - last;
      last = t;
    }
  }
  __device__ __forceinline__ void done() {
    if (acc) acc[kTrAll] += now_ns() - first;
  }
};

// ---- bulk copies (all threads of the CTA take part) --------------------------------------------

__device__ __forceinline__ uint4 ld16(const void* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ void st16(void* p, uint4 v) { *reinterpret_cast<uint4*>(p) = v; }
// The same under a predicate, as one instruction each: written as `if (ok) r = ld16(p)`, unrolled
// loads of a partial round become a ladder of branches that waits for one load before the next.
// A load that does not take place gives zeros: left undefined, its registers would count as live
// from the kernel's start, and every such loop would spill those of the others.
__device__ __forceinline__ uint4 ld16_if(bool ok, const void* p) {
  uint4 v;
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.u32 q, %5, 0;\n mov.u32 %0, 0;\n mov.u32 %1, 0;\n mov.u32 %2, 0;\n mov.u32 %3, 0;\n"
      " @q ld.global.v4.u32 {%0,%1,%2,%3}, [%4];\n}"
      : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w)
      : "l"(p), "r"(unsigned(ok))
      : "memory");
  return v;
}
__device__ __forceinline__ void st16_if(bool ok, void* p, uint4 v) {
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %5, 0;\n @q st.global.v4.u32 [%4], {%0,%1,%2,%3};\n}" ::"r"(v.x), "r"(v.y),
               "r"(v.z), "r"(v.w), "l"(p), "r"(unsigned(ok))
               : "memory");
}
// Evict-first in the second-level cache, for data that is not read again soon: a caller's inputs and
// outputs and, once read, the staged bytes. What is left to L2 are the bytes that a peer is still to
// read. Staged traffic is two thirds of an AllReduce's, and much of it goes to DRAM and back. One B200, the
// same build without the hints and with them, DRAM bytes of a launch (ncu) and us a call:
//   4 ranks, 16 MiB fp32            216 and 177 MB, 62.8 and 59.0
//   8 ranks, 16 MiB e4m3            659 and 504 MB, 136.2 and 131.6
//   7 ranks, 28 MB fp32 average    1023 and 873 MB, 186.5 and 186.1
//   8 ranks, AllGather of 1 MiB blocks              40.9 and 35.8
// Messages of 1 to 4 MiB, which fit L2 as they are, lose 4 to 9 % (4 ranks, 4 MiB e4m3: 24.4 and 26.8).
__device__ __forceinline__ unsigned long long once_policy() {
  unsigned long long p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint4 ld16_once_if(bool ok, const void* p, unsigned long long policy) {
  uint4 v;
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.u32 q, %5, 0;\n mov.u32 %0, 0;\n mov.u32 %1, 0;\n mov.u32 %2, 0;\n mov.u32 %3, 0;\n"
      " @q ld.global.L1::no_allocate.L2::cache_hint.v4.u32 {%0,%1,%2,%3}, [%4], %6;\n}"
      : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w)
      : "l"(p), "r"(unsigned(ok)), "l"(policy)
      : "memory");
  return v;
}
__device__ __forceinline__ void st16_once_if(bool ok, void* p, uint4 v, unsigned long long policy) {
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %5, 0;\n @q st.global.L2::cache_hint.v4.u32 [%4], {%0,%1,%2,%3}, %6;\n}" ::"r"(v.x),
               "r"(v.y), "r"(v.z), "r"(v.w), "l"(p), "r"(unsigned(ok)), "l"(policy)
               : "memory");
}
// streaming variants for data that is touched once
__device__ __forceinline__ uint4 ld16_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// Bytes s .. s+15 of the 32 bytes a, b (0 <= s < 16).
__device__ __forceinline__ uint4 bytes_of_pair(uint4 a, uint4 b, unsigned s) {
  unsigned w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int k = 0; k < 6; ++k) w[k] = (s & 8u) ? w[k + 2] : w[k];
#pragma unroll
  for (int k = 0; k < 5; ++k) w[k] = (s & 4u) ? w[k + 1] : w[k];
  const unsigned bits = (s & 3u) * 8u;
  return make_uint4(__funnelshift_r(w[0], w[1], bits), __funnelshift_r(w[1], w[2], bits),
                    __funnelshift_r(w[2], w[3], bits), __funnelshift_r(w[3], w[4], bits));
}

// The thread's index, read anew: what is computed from it is not hoisted out of the loop over a
// kernel's steps, where the address arithmetic of every phase together would not fit the registers.
__device__ __forceinline__ unsigned fresh_tid() {
  unsigned t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

// dst[0,n) = src[0,n); any alignment. Whole 16-byte vectors of dst are stored; where src lies at
// another offset within its vectors, each one is cut out of the two aligned vectors it spans (the
// second is the neighbour lane's first, so it comes from L1). Byte by byte this was bound by the
// number of loads: 8 ranks exchanging blocks of about 1 MiB at odd offsets, 1767 us against
// 80 us a call on one B200 (59 with two CTAs per SM).
// A warp moves runs of eight (four) times 512 bytes, so that the loads of a run differ by a constant
// and eight are in flight per thread. A share of 64 GiB or more does not occur.
__device__ inline void cta_copy(char* dst, const char* src, size_t n) {
  const unsigned t = fresh_tid(), lane = t & 31u, warp = t >> 5, warps = blockDim.x >> 5;
  unsigned head = unsigned(-reinterpret_cast<intptr_t>(dst)) & 15u;
  if (head > n) head = unsigned(n);
  if (t < head) dst[t] = src[t];
  dst += head;
  src += head;
  n -= head;
  const unsigned nv = unsigned(n >> 4), tail = unsigned(n) & 15u;
  const unsigned s = unsigned(reinterpret_cast<uintptr_t>(src) & 15u);
  if (s == 0) {
    constexpr int U = 8;
    for (unsigned i = warp * (32 * U) + lane; i < nv; i += warps * (32 * U)) {
      const char* from = src + (size_t(i) << 4);
      char* to = dst + (size_t(i) << 4);
      const unsigned left = nv - i;
      uint4 r[U];
#pragma unroll
      for (int u = 0; u < U; ++u) r[u] = ld16_if(u * 32 < left, from + u * 512);
#pragma unroll
      for (int u = 0; u < U; ++u) st16_if(u * 32 < left, to + u * 512, r[u]);
    }
  } else {
    constexpr int U = 4;
    for (unsigned i = warp * (32 * U) + lane; i < nv; i += warps * (32 * U)) {
      const char* from = src - s + (size_t(i) << 4);
      char* to = dst + (size_t(i) << 4);
      const unsigned left = nv - i;
      uint4 r[U], q[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        r[u] = ld16_if(u * 32 < left, from + u * 512);
        q[u] = ld16_if(u * 32 < left, from + u * 512 + 16);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) st16_if(u * 32 < left, to + u * 512, bytes_of_pair(r[u], q[u], s));
    }
  }
  if (t < tail) dst[(size_t(nv) << 4) + t] = src[(size_t(nv) << 4) + t];
}

__device__ __forceinline__ void mc_st16(char* mc_addr, uint4 v) {
  asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(mc_addr), "r"(v.x), "r"(v.y),
               "r"(v.z), "r"(v.w)
               : "memory");
}
// The same bytes to every rank at once: mc_dst is an address in the multicast alias of the
// windows. Whole 16-byte vectors only (both addresses 16-byte aligned); returns the bytes it
// covered, the caller sends the rest peer by peer.
__device__ inline size_t cta_copy_multicast(char* mc_dst, const char* src, size_t n) {
  const int t = threadIdx.x, nt = blockDim.x;
  const size_t nv = n >> 4;
  size_t i = t;
  for (; i + 3 * size_t(nt) < nv; i += 4 * size_t(nt)) {
    uint4 r[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) r[u] = ld16(src + ((i + u * size_t(nt)) << 4));
#pragma unroll
    for (int u = 0; u < 4; ++u) mc_st16(mc_dst + ((i + u * size_t(nt)) << 4), r[u]);
  }
  for (; i < nv; i += nt) mc_st16(mc_dst + (i << 4), ld16(src + (i << 4)));
  return nv << 4;
}

// ---- bulk asynchronous copies (the TMA unit, untiled form) ------------------------------------------
// A copy whose source is this GPU's memory and whose destination is a peer's window can be
// driven by one thread: cp.async.bulk brings a chunk into shared memory (completion on an
// mbarrier), a second cp.async.bulk writes it to the destination, and several chunks are in
// flight at once. The copy unit issues large transactions on its own, so no warp spends
// instructions on moving bytes. Loads never use cluster multicast. Both addresses and the size
// must be multiples of 16 bytes (the caller checks). Every wait is bounded: when one runs out,
// the function stops issuing, waits for its stores in flight and returns false.
constexpr int kBulkStages = 4;
constexpr unsigned kBulkChunk = 32 * 1024;
constexpr size_t kBulkSmemBytes = size_t(kBulkStages) * kBulkChunk;
struct BulkPipe {
  unsigned char* buf;        // kBulkSmemBytes of shared memory, 128-byte aligned
  unsigned long long* bars;  // kBulkStages mbarriers, initialised once per kernel by bulk_pipe_init
  unsigned phase;            // bit s = parity the next wait on stage s expects (kept by the issuing thread)
};
__device__ __forceinline__ unsigned smem_addr(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
// all threads call; leaves with a barrier
__device__ inline void bulk_pipe_init(BulkPipe& pipe, unsigned char* buf, unsigned long long* bars) {
  pipe.buf = buf;
  pipe.bars = bars;
  pipe.phase = 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kBulkStages; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bars[s])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
}
// Called by ONE thread. dst[0, n) = src[0, n).
__device__ inline bool bulk_copy_by_one_thread(BulkPipe& pipe, char* dst, const char* src, size_t n) {
  const size_t chunks = (n + kBulkChunk - 1) / kBulkChunk;
  auto chunk_len = [&](size_t c) { return unsigned(n - c * kBulkChunk < kBulkChunk ? n - c * kBulkChunk : kBulkChunk); };
  auto load = [&](size_t c) {
    const int s = int(c % kBulkStages);
    const unsigned len = chunk_len(c), bar = smem_addr(&pipe.bars[s]);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(len) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(pipe.buf + size_t(s) * kBulkChunk)),
                 "l"(src + c * kBulkChunk), "r"(len), "r"(bar)
                 : "memory");
  };
  // loads run kBulkStages - 1 chunks ahead of the stores; a stage is loaded again only after the
  // store that read it has finished reading (wait_group.read keeps one store group outstanding)
  size_t issued = 0;
  for (; issued < chunks && issued < size_t(kBulkStages - 1); ++issued) load(issued);
  bool ok = true;
  for (size_t c = 0; c < chunks && ok; ++c) {
    const int s = int(c % kBulkStages);
    const unsigned bar = smem_addr(&pipe.bars[s]), parity = (pipe.phase >> s) & 1u;
    unsigned done = 0;
    for (unsigned spins = 0; !done; ++spins) {
      asm volatile(
          "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
          : "=r"(done)
          : "r"(bar), "r"(parity)
          : "memory");
      if (!done && spins > (1u << 22)) {  // far beyond any copy: give up
        ok = false;
        break;
      }
    }
    if (!ok) break;
    pipe.phase ^= 1u << s;
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst + c * kBulkChunk),
                 "r"(smem_addr(pipe.buf + size_t(s) * kBulkChunk)), "r"(chunk_len(c))
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    if (issued < chunks) {
      // chunk `issued` reuses the stage of chunk issued - kBulkStages = c - 1, whose store is one group back
      asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
      load(issued);
      ++issued;
    }
  }
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // every store has been performed
  return ok;
}

// 16 bytes of elements of type T
template <typename T>
union Vec16 {
  uint4 raw;
  T e[16 / sizeof(T)];
};

// ---- a whole vector of elements through the element rule ------------------------------------------
// out.e[l] = apply(a.e[l], b.e[l], op) for every lane. The generic form is the lane loop; the
// fp8 types go two lanes at a time, because their hardware converters work on pairs
// (cvt...x2) and converting one value per instruction, as the scalar rule in math/fpconv.h does,
// leaves half of the converter's rate unused, which is what bounds an fp8 fold.
template <typename T>
__device__ __forceinline__ Vec16<T> apply_lanes(const Vec16<T>& a, const Vec16<T>& b, int op) {
  Vec16<T> out;
#pragma unroll
  for (int l = 0; l < int(16 / sizeof(T)); ++l) out.e[l] = apply(a.e[l], b.e[l], op);
  return out;
}

template <typename T>
__device__ __forceinline__ Vec16<T> splat(T k) {
  Vec16<T> v;
#pragma unroll
  for (int l = 0; l < int(16 / sizeof(T)); ++l) v.e[l] = k;
  return v;
}

__device__ __forceinline__ float2 f16x2_to_f32(unsigned pair) {
  float lo, hi;
  asm("cvt.f32.f16 %0, %1;" : "=f"(lo) : "h"(static_cast<unsigned short>(pair & 0xffffu)));
  asm("cvt.f32.f16 %0, %1;" : "=f"(hi) : "h"(static_cast<unsigned short>(pair >> 16)));
  return make_float2(lo, hi);
}
// two e4m3 codes (low byte = first element) -> two floats, exact
__device__ __forceinline__ float2 decode_pair(unsigned short codes, e4m3) {
  unsigned pair;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(pair) : "h"(codes));
  return f16x2_to_f32(pair);
}
// an e5m2 code is the upper byte of an fp16
__device__ __forceinline__ float2 decode_pair(unsigned short codes, e5m2) {
  return f16x2_to_f32(((unsigned(codes) & 0xff00u) << 16) | ((unsigned(codes) & 0xffu) << 8));
}
// two floats -> two codes under the library's rules (math/fpconv.h: hardware rounding, then the
// overflow and NaN codes patched in, per element exactly as from_f32 does)
__device__ __forceinline__ unsigned short encode_pair(float lo, float hi, e4m3) {
  unsigned short pair;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(pair) : "f"(hi), "f"(lo));
  const uint32_t ul = f32_bits(lo), al = ul & 0x7fffffffu, uh = f32_bits(hi), ah = uh & 0x7fffffffu;
  unsigned r0 = pair & 0xffu, r1 = pair >> 8;
  if (al > 0x43e80000u) r0 = al > 0x7f800000u ? 0x7fu : (((ul >> 24) & 0x80u) | 0x7fu);
  if (ah > 0x43e80000u) r1 = ah > 0x7f800000u ? 0x7fu : (((uh >> 24) & 0x80u) | 0x7fu);
  return static_cast<unsigned short>(r0 | (r1 << 8));
}
__device__ __forceinline__ unsigned short encode_pair(float lo, float hi, e5m2) {
  unsigned short pair;
  asm("cvt.rn.satfinite.e5m2x2.f32 %0, %1, %2;" : "=h"(pair) : "f"(hi), "f"(lo));
  const uint32_t ul = f32_bits(lo), al = ul & 0x7fffffffu, uh = f32_bits(hi), ah = uh & 0x7fffffffu;
  unsigned r0 = pair & 0xffu, r1 = pair >> 8;
  if (al >= 0x47700000u) r0 = al > 0x7f800000u ? 0x7eu : (((ul >> 24) & 0x80u) | 0x7cu);
  if (ah >= 0x47700000u) r1 = ah > 0x7f800000u ? 0x7eu : (((uh >> 24) & 0x80u) | 0x7cu);
  return static_cast<unsigned short>(r0 | (r1 << 8));
}
template <typename F8>
__device__ __forceinline__ Vec16<F8> apply_lanes_fp8(const Vec16<F8>& a, const Vec16<F8>& b, int op) {
  Vec16<F8> out;
  const unsigned wa[4] = {a.raw.x, a.raw.y, a.raw.z, a.raw.w}, wb[4] = {b.raw.x, b.raw.y, b.raw.z, b.raw.w};
  unsigned wo[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    unsigned short half[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float2 x = decode_pair(static_cast<unsigned short>(wa[k] >> (16 * h)), F8{});
      const float2 y = decode_pair(static_cast<unsigned short>(wb[k] >> (16 * h)), F8{});
      half[h] = encode_pair(narrow_combine(x.x, y.x, op), narrow_combine(x.y, y.y, op), F8{});
    }
    wo[k] = unsigned(half[0]) | (unsigned(half[1]) << 16);
  }
  out.raw = make_uint4(wo[0], wo[1], wo[2], wo[3]);
  return out;
}
template <>
__device__ __forceinline__ Vec16<e4m3> apply_lanes<e4m3>(const Vec16<e4m3>& a, const Vec16<e4m3>& b, int op) {
  return apply_lanes_fp8<e4m3>(a, b, op);
}
template <>
__device__ __forceinline__ Vec16<e5m2> apply_lanes<e5m2>(const Vec16<e5m2>& a, const Vec16<e5m2>& b, int op) {
  return apply_lanes_fp8<e5m2>(a, b, op);
}

// ---- Sum and Prod without the rare cases -----------------------------------------------------------
// What the element rules add to a plain sum or product concerns NaN (whose payload survives, which
// code it gets) and, for the 8-bit floats, overflow. Lanes<T> computes the plain form in the widest
// instructions there are and sets `odd` when some lane may need more; the caller then takes the
// whole vector through the rule (apply, apply_lanes). Acc holds the lanes as the chain of
// combinations needs them: the vector itself, or, for the 8-bit floats, the f16 values of the codes,
// so that a fold decodes every input once and its running value never.
//
// The packed 16-bit forms round once where the rule rounds to fp32 and then to the type. Both give
// the same bits: an intermediate of q bits is innocuous for + and x from p-bit operands when
// q >= 2p + 1 and q >= 2p (Figueroa, "When is double rounding innocuous?", 1995), here 24 against
// p = 11 (fp16) and 8 (bf16), and the exact result of the operands' grids is representable in the
// intermediate wherever the result is subnormal. The same holds for the 8-bit floats in f16:
// 11 against p = 4 (e4m3) and 3 (e5m2); their products have at most 8 bits and are exact in f16
// or lie below a quarter of the smallest code, and what overflows f16 overflows them.
template <typename T>
struct Lanes {
  using Acc = Vec16<T>;
  static __device__ __forceinline__ Acc open(const Vec16<T>& v) { return v; }
  static __device__ __forceinline__ Vec16<T> close(const Acc& a) { return a; }
  template <int kOp>
  static __device__ __forceinline__ Acc combine(const Acc& a, const Acc& b, bool& odd) {
    Acc r;
#pragma unroll
    for (int l = 0; l < int(16 / sizeof(T)); ++l) {
      if constexpr (std::is_floating_point<T>::value) {
        r.e[l] = kOp == kSum ? add_rn(a.e[l], b.e[l]) : mul_rn(a.e[l], b.e[l]);
        odd |= r.e[l] != r.e[l];
      } else {
        r.e[l] = apply(a.e[l], b.e[l], kOp);
      }
    }
    return r;
  }
};
// f16 / bf16: two lanes per instruction; kInf is the type's infinity in both halves, so a magnitude
// above it (NaN) carries into the sign bits of the sum below.
template <typename T, unsigned kInf>
struct PackedLanes {
  using Acc = Vec16<T>;
  static __device__ __forceinline__ Acc open(const Vec16<T>& v) { return v; }
  static __device__ __forceinline__ Vec16<T> close(const Acc& a) { return a; }
  template <int kOp>
  static __device__ __forceinline__ Acc combine(const Acc& a, const Acc& b, bool& odd) {
    const unsigned wa[4] = {a.raw.x, a.raw.y, a.raw.z, a.raw.w}, wb[4] = {b.raw.x, b.raw.y, b.raw.z, b.raw.w};
    unsigned r[4], nan = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if constexpr (std::is_same<T, f16>::value) {
        if constexpr (kOp == kSum) asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r[k]) : "r"(wa[k]), "r"(wb[k]));
        else asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r[k]) : "r"(wa[k]), "r"(wb[k]));
      } else {
        if constexpr (kOp == kSum) asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(r[k]) : "r"(wa[k]), "r"(wb[k]));
        else asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r[k]) : "r"(wa[k]), "r"(wb[k]));
      }
      nan |= (r[k] & 0x7fff7fffu) + (0x7fff7fffu - kInf);
    }
    odd |= (nan & 0x80008000u) != 0;
    Acc out;
    out.raw = make_uint4(r[0], r[1], r[2], r[3]);
    return out;
  }
};
template <>
struct Lanes<f16> : PackedLanes<f16, 0x7c007c00u> {};
template <>
struct Lanes<bf16> : PackedLanes<bf16, 0x7f807f80u> {};

// e4m3 / e5m2: 16 lanes as eight f16 pairs plus the codes they stand for. The saturating encoder
// gives the rule's code except above the largest finite value and for NaN; such lanes carry a code of
// at least kTop (the largest finite code) or the hardware's NaN, and set `odd`.
template <typename F8, unsigned kTop>
struct Fp8Lanes {
  struct Acc {
    unsigned h[8];
    uint4 codes;
  };
  static __device__ __forceinline__ unsigned decode(unsigned short two) {
    unsigned pair;
    if constexpr (std::is_same<F8, e4m3>::value) asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(pair) : "h"(two));
    else asm("cvt.rn.f16x2.e5m2x2 %0, %1;" : "=r"(pair) : "h"(two));
    return pair;
  }
  static __device__ __forceinline__ unsigned encode(unsigned pair) {
    unsigned short two;
    if constexpr (std::is_same<F8, e4m3>::value) asm("cvt.rn.satfinite.e4m3x2.f16x2 %0, %1;" : "=h"(two) : "r"(pair));
    else asm("cvt.rn.satfinite.e5m2x2.f16x2 %0, %1;" : "=h"(two) : "r"(pair));
    return two;
  }
  static __device__ __forceinline__ Acc open(const Vec16<F8>& v) {
    Acc a;
    a.codes = v.raw;
    const unsigned w[4] = {v.raw.x, v.raw.y, v.raw.z, v.raw.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      a.h[2 * k] = decode(static_cast<unsigned short>(w[k] & 0xffffu));
      a.h[2 * k + 1] = decode(static_cast<unsigned short>(w[k] >> 16));
    }
    return a;
  }
  static __device__ __forceinline__ Vec16<F8> close(const Acc& a) {
    Vec16<F8> v;
    v.raw = a.codes;
    return v;
  }
  template <int kOp>
  static __device__ __forceinline__ Acc combine(const Acc& a, const Acc& b, bool& odd) {
    unsigned w[4], top = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      unsigned s[2];
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if constexpr (kOp == kSum) asm("add.rn.f16x2 %0, %1, %2;" : "=r"(s[h]) : "r"(a.h[2 * k + h]), "r"(b.h[2 * k + h]));
        else asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(s[h]) : "r"(a.h[2 * k + h]), "r"(b.h[2 * k + h]));
      w[k] = encode(s[0]) | (encode(s[1]) << 16);
      top |= (w[k] & 0x7f7f7f7fu) + (0x80u - kTop) * 0x01010101u;
    }
    odd |= (top & 0x80808080u) != 0;
    Vec16<F8> v;
    v.raw = make_uint4(w[0], w[1], w[2], w[3]);
    return open(v);
  }
};
template <>
struct Lanes<e4m3> : Fp8Lanes<e4m3, 0x7eu> {};
template <>
struct Lanes<e5m2> : Fp8Lanes<e5m2, 0x7bu> {};

// apply for every lane, any operator
template <typename T>
__device__ __forceinline__ Vec16<T> combine_lanes(const Vec16<T>& a, const Vec16<T>& b, int op) {
  using L = Lanes<T>;
  bool odd = false;
  Vec16<T> out;
  if (op == kSum)
    out = L::close(L::template combine<kSum>(L::open(a), L::open(b), odd));
  else if (op == kProd)
    out = L::close(L::template combine<kProd>(L::open(a), L::open(b), odd));
  else
    return apply_lanes(a, b, op);
  return odd ? apply_lanes(a, b, op) : out;
}
// value * scalar for every lane under the Prod rule
template <typename T>
__device__ __forceinline__ Vec16<T> scale_lanes(const Vec16<T>& v, T k) {
  return combine_lanes(v, splat(k), kProd);
}

}  // namespace hx
