// Combining the ranks' values in a prescribed order (device/proto.h: FoldSpec), fused with the
// pre-scale of the local input and the integer post-divide, so a reduction needs no separate
// scale, reduce or divide pass (the reference runs k_scale, k_reduce and k_div as separate
// kernels around its copies: src/gpu_reduce.cu:20-39, src/memops_device.cc:33-57).
#pragma once
#include "kernels/prims.cuh"

namespace hx {

template <typename T>
__device__ __forceinline__ T load_scalar(const FoldSpec& f) {
  T k;
  if (f.scalar_ptr) {
    k = *reinterpret_cast<const T*>(f.scalar_ptr);
  } else {
    const unsigned long long bits = f.scalar_bits;  // little endian: low bytes hold the value
    memcpy(&k, &bits, sizeof(T));
  }
  return k;
}

struct FoldShared {
  const char* src[kMaxRanks];       // per rank: where this CTA's part of its data starts
  char* remote[kMaxRanks];          // extra destinations of the result (peers' windows)
  char* mc_dst;                     // multicast alias of those destinations, or null
  unsigned long long bound[kMaxRanks + 1];  // ring-block boundaries, in elements
  const char* piece_src[kMaxRanks];  // pieces of the copy at hand (cta_pieces)
  char* piece_dst[kMaxRanks];
  size_t piece_len[kMaxRanks];
  FoldSpec spec;  // of the launch (open_fold)
  int rank, n;
  int fail;
};

// Once per kernel, by all threads; the caller's next barrier makes it visible. The phases below are
// functions of their own (not inlined), so that each has the whole register budget to itself, and take
// what the launch fixes from here rather than from the kernel's parameters.
__device__ inline void fill_ring_bounds(FoldShared& sh, size_t count, int n);
__device__ inline void open_fold(FoldShared& sh, const FoldSpec& f, int rank, int n) {
  if (threadIdx.x == 0) {
    sh.spec = f;
    sh.rank = rank;
    sh.n = n;
    sh.fail = 0;
  }
  if (f.kind == kFoldLinear && f.ring) fill_ring_bounds(sh, f.ring_count, n);
}

// ring-block boundaries of `count` elements over n ranks, once per kernel
__device__ inline void fill_ring_bounds(FoldShared& sh, size_t count, int n) {
  if (threadIdx.x <= unsigned(n)) {
    const int k = threadIdx.x;
    const size_t base = count / n, extra = count % n;
    sh.bound[k] = k == n ? count : size_t(k) * base + (size_t(k) < extra ? size_t(k) : extra);
  }
}
__device__ __forceinline__ int ring_block_of(const FoldShared& sh, unsigned long long e, int n) {
  int c = 0;
  for (int k = 1; k < n; ++k) c += (e >= sh.bound[k]) ? 1 : 0;
  return c;
}

// The order-defining part for one element. x[i] is rank i's (already scaled) value.
template <typename T>
__device__ inline T fold_one(const T* x, int n, int rank, const FoldSpec& f, int block) {
  const int op = f.op;
  if (f.kind == kFoldLinear) {
    int idx = (f.start + (f.ring ? block : 0)) % n;
    T acc = x[idx];
    for (int k = 1; k < n; ++k) {
      idx += f.dir;
      idx = idx >= n ? idx - n : (idx < 0 ? idx + n : idx);
      acc = apply(x[idx], acc, op);
    }
    return acc;
  }
  if (f.kind == kFoldDoubling) {
    int p = 1;
    while (2 * p <= n) p *= 2;
    const int spare = n - p;
    T lv[kMaxRanks];
    for (int q = 0; q < p; ++q)  // pairs first: the odd rank combines its own value with the even one's
      lv[q] = q < spare ? apply(x[2 * q + 1], x[2 * q], op) : x[q + spare];
    for (int bit = 1; bit < p; bit <<= 1) {
      T nx[kMaxRanks];
      for (int q = 0; q < p; ++q) nx[q] = apply(lv[q], lv[q ^ bit], op);
      for (int q = 0; q < p; ++q) lv[q] = nx[q];
    }
    const int mine = rank < 2 * spare ? rank / 2 : rank - spare;
    return lv[mine];
  }
  // binomial tree toward the root, in positions relative to it
  T acc[kMaxRanks];
  for (int v = n - 1; v >= 0; --v) {
    int real = v + f.root;
    real = real >= n ? real - n : real;
    T a = x[real];
    const int low = v == 0 ? n : (v & -v);  // children sit at v+1, v+2, v+4, ... below v's low bit
    for (int m = 1; m < low && v + m < n; m <<= 1) a = apply(a, acc[v + m], op);
    acc[v] = a;
  }
  return acc[0];
}

// One element of recursive doubling over N = 2, 4 or 8 ranks: x[q] is the value of rank (r ^ q) and
// the result rank r's (the tree is explained at fold_vectors).
template <typename T, int N>
__device__ __forceinline__ T fold_doubling_pow2(T (&x)[N], int op) {
#pragma unroll
  for (int bit = 1; bit < N; bit <<= 1)
#pragma unroll
    for (int q = 0; q < N; q += 2 * bit) x[q] = apply(x[q], x[q + bit], op);
  return x[0];
}

// One element through the general path: any fold kind, any rank count, any alignment.
template <typename T>
__device__ inline T fold_element(const FoldShared& sh, size_t e, size_t elem0, bool premul, T scalar) {
  const FoldSpec& f = sh.spec;
  const int rank = sh.rank, n = sh.n;
  T x[kMaxRanks];
  for (int i = 0; i < n; ++i) x[i] = reinterpret_cast<const T*>(sh.src[i])[e];
  if (premul) x[rank] = scale(x[rank], scalar);
  const int b = (f.kind == kFoldLinear && f.ring) ? ring_block_of(sh, elem0 + e, n) : 0;
  const T r = fold_one(x, n, rank, f, b);
  return f.postdiv ? div_trunc(r, f.postdiv) : r;
}
// dst may have any alignment that its element type has; the remote destinations are window slots
// (16-byte aligned). kDstOnce: dst is not read again soon (a caller's buffer).
template <typename T, bool kDstOnce>
__device__ __forceinline__ void fold_store(char* dst, bool dst_aligned, const FoldShared& sh, int nremote, unsigned v,
                                           const Vec16<T>& out, unsigned long long policy) {
  const size_t off = size_t(v) << 4;
  if (dst_aligned) {
    if (kDstOnce) st16_once_if(true, dst + off, out.raw, policy);
    else st16(dst + off, out.raw);
  } else {
#pragma unroll
    for (int l = 0; l < int(16 / sizeof(T)); ++l) reinterpret_cast<T*>(dst + off)[l] = out.e[l];
  }
  if (sh.mc_dst) {
    mc_st16(sh.mc_dst + off, out.raw);
  } else {
    for (int r = 0; r < nremote; ++r) st16(sh.remote[r] + off, out.raw);
  }
}

// The loop of both orders over whole vectors [v_lo, v_hi) that all take the sources in the same
// sequence (rank `first`, first + dir, ... for the linear orders; rank ^ 0, rank ^ 1, ... for recursive
// doubling), for N/2 < n <= N ranks: U vectors per thread and iteration, all n * U loads issued before
// the first combine. kOp: kSum, or -1 for any operator at run time.
//
// Recursive doubling over n = N ranks as rank r sees it: its value after a level is its own value of
// the level before on the left and its partner's on the right, and the partner's is formed the same way
// from the partner's side. Only N - 1 of the N log N combinations of the butterfly feed rank r's
// result, and with the sources in the order r ^ q they are a plain binary tree.
template <typename T, int N, int U, int kOp, bool kTree, bool kDstOnce>
__device__ __forceinline__ void fold_vectors(char* dst, bool dst_aligned, const FoldShared& sh, int nremote, unsigned v_lo,
                                             unsigned v_hi, int first, bool premul, T scalar) {
  using L = Lanes<T>;
  const FoldSpec& f = sh.spec;
  const int rank = sh.rank, n = kTree ? N : sh.n;
  const unsigned long long policy = once_policy();  // every source is read for the last time
  constexpr int V = 16 / sizeof(T);
  const unsigned t = fresh_tid(), lane = t & 31u, warp = t >> 5, warps = blockDim.x >> 5;
  // the rank whose value comes k-th; its address is read from shared memory where it is needed (eight
  // pointers held over the loop cost sixteen registers)
  auto rank_at = [&](int k) {
    if constexpr (kTree) return rank ^ k;
    const int idx = first + (f.dir < 0 ? n - k : k);
    return idx >= n ? idx - n : idx;
  };
  // window slots are aligned; this rank's own input need not be
  const unsigned shift = unsigned(reinterpret_cast<uintptr_t>(sh.src[rank]) & 15u);
  for (unsigned v0 = v_lo + warp * (32 * U) + lane; v0 < v_hi; v0 += warps * (32 * U)) {  // a warp takes runs of U x 512 bytes
    const unsigned left = v_hi - v0;
    Vec16<T> in[U][N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int idx = k < n ? rank_at(k) : rank;
      const char* p = sh.src[idx] + (size_t(v0) << 4) - (idx == rank ? shift : 0u);
#pragma unroll
      for (int u = 0; u < U; ++u) in[u][k].raw = ld16_once_if(u * 32 < left && k < n, p + u * 512, policy);
    }
    if (shift) {  // cut the own vectors out of the two aligned ones they span
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint4 next = ld16_if(u * 32 < left, sh.src[rank] + (size_t(v0) << 4) - shift + u * 512 + 16);
#pragma unroll
        for (int k = 0; k < N; ++k)
          if (k < n && rank_at(k) == rank) in[u][k].raw = bytes_of_pair(in[u][k].raw, next, shift);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned v = v0 + u * 32;
      if (u * 32 >= left) continue;
      Vec16<T> out;
      bool odd = false;
      if constexpr (kOp >= 0 && kTree) {
        typename L::Acc x[N];
#pragma unroll
        for (int k = 0; k < N; ++k) x[k] = L::open(in[u][k]);
        if (premul) x[0] = L::template combine<kProd>(x[0], L::open(splat(scalar)), odd);  // rank ^ 0 is this rank
#pragma unroll
        for (int bit = 1; bit < N; bit <<= 1)
#pragma unroll
          for (int q = 0; q < N; q += 2 * bit) x[q] = L::template combine<kOp>(x[q], x[q + bit], odd);
        out = L::close(x[0]);
      } else if constexpr (kOp >= 0) {
        typename L::Acc acc;
#pragma unroll
        for (int k = 0; k < N; ++k) {
          if (k >= n) continue;
          typename L::Acc x = L::open(in[u][k]);
          if (premul && rank_at(k) == rank) x = L::template combine<kProd>(x, L::open(splat(scalar)), odd);
          acc = k == 0 ? x : L::template combine<kOp>(x, acc, odd);
        }
        out = L::close(acc);
      } else {
#pragma unroll
        for (int k = 0; k < N; ++k)
          if (premul && k < n && rank_at(k) == rank) in[u][k] = apply_lanes(in[u][k], splat(scalar), kProd);
        if constexpr (kTree) {
#pragma unroll
          for (int bit = 1; bit < N; bit <<= 1)
#pragma unroll
            for (int q = 0; q < N; q += 2 * bit) in[u][q] = apply_lanes(in[u][q], in[u][q + bit], f.op);
          out = in[u][0];
        } else {
          out = in[u][0];
#pragma unroll
          for (int k = 1; k < N; ++k)
            if (k < n) out = apply_lanes(in[u][k], out, f.op);
        }
      }
      if (odd) {  // rare: lane by lane under the rule, from the sources, which are still as they were
#pragma unroll 1
        for (int l = 0; l < V; ++l) {
          const size_t e = size_t(v) * V + l;
          T y[N];
#pragma unroll
          for (int k = 0; k < N; ++k) {
            if (k >= n) continue;
            y[k] = reinterpret_cast<const T*>(sh.src[rank_at(k)])[e];
            if (premul && rank_at(k) == rank) y[k] = scale(y[k], scalar);
          }
          T r = y[0];
          if constexpr (kTree) {
            r = fold_doubling_pow2<T, N>(y, f.op);
          } else {
#pragma unroll
            for (int k = 1; k < N; ++k)
              if (k < n) r = apply(y[k], r, f.op);
          }
          reinterpret_cast<T*>(dst)[e] = r;
          for (int q = 0; q < nremote; ++q) reinterpret_cast<T*>(sh.remote[q])[e] = r;
        }
        continue;
      }
      if (f.postdiv) {
#pragma unroll
        for (int l = 0; l < V; ++l) out.e[l] = div_trunc(out.e[l], f.postdiv);
      }
      fold_store<T, kDstOnce>(dst, dst_aligned, sh, nremote, v, out, policy);
    }
  }
}

// Folds `nbytes` bytes (whole elements). sh.src[i] points at rank i's data for this range
// (sh.src[rank] is the local input, unscaled when `premul`), elem0 is the index of the first element
// in the full vector. The result goes to dst and to each of sh.remote[0..nremote); when sh.mc_dst is
// set, whole vectors reach the remote destinations through one multimem.st instead (tails still go
// peer by peer).
//
// The ring order changes its starting rank from ring block to ring block. A share is usually inside
// one block, so the block is looked up once per stretch of vectors between two block ends, not per
// vector; a vector that straddles two blocks goes element by element, like the tail.
// The linear orders keep every source of a vector in registers: kN is 2, 4 or 8 with kN/2 < n <= kN,
// one kernel each (a kernel that carries all of them spills), and 0 for one rank and for nine to sixteen,
// whose loop is sixteen wide. What is left goes element by element with the values in local memory:
// tails, trees, recursive doubling over other counts. One B200, us a call: 7 ranks, 28 MB fp32 average, 677 by
// that general path and 243 by vectors (111 CTAs); 9 ranks, 16 MiB e4m3, 748 and 165; 12 ranks, 16 MiB
// fp32, 355 and 201.
template <typename T, int kN, bool kDstOnce = true>
static __device__ __noinline__ void cta_fold(char* dst, const FoldShared& sh, int nremote, size_t nbytes, size_t elem0,
                                             bool premul, T scalar) {
  const FoldSpec& f = sh.spec;
  const int n = sh.n;
  constexpr int V = 16 / sizeof(T);
  const unsigned t = threadIdx.x, nt = blockDim.x;
  const unsigned total = unsigned(nbytes / sizeof(T));
  auto element = [&](unsigned e) {
    const T r = fold_element<T>(sh, e, elem0, premul, scalar);
    reinterpret_cast<T*>(dst)[e] = r;
    for (int q = 0; q < nremote; ++q) reinterpret_cast<T*>(sh.remote[q])[e] = r;
  };
  constexpr int N = kN ? kN : kMaxRanks;
  // sixteen 16-byte loads in flight per thread; with eight, the ReduceScatter + AllGather of 14 MB on
  // 8 ranks took 132 us instead of 125, 7 ranks' 28 MB fp32 average 195 instead of 188
  constexpr int U = 16 / N;
  const bool dst_aligned = (reinterpret_cast<uintptr_t>(dst) & 15u) == 0;
  const bool ring = f.kind == kFoldLinear && f.ring, tree = f.kind == kFoldDoubling && n == kN;
  // below four elements per thread the sixteen-wide loop leaves most threads idle (9 ranks, 1 MiB fp32 max:
  // 26.9 us a call, by elements 24.5)
  const bool vectors = (f.kind == kFoldLinear && (kN || total > 4 * nt)) || tree;
  const unsigned nvec = vectors ? unsigned(nbytes >> 4) : 0;
  for (unsigned v = 0; v < nvec;) {
    unsigned v_hi = nvec;  // whole vectors up to here take the sources in the same sequence
    int first = f.start;
    if (ring) {
      const int block = ring_block_of(sh, elem0 + size_t(v) * V, n);
      const size_t left = (block + 1 < n ? sh.bound[block + 1] : ~0ull) - elem0;  // elements up to the block's end
      if (left / V < nvec) v_hi = unsigned(left / V);
      first = (f.start + block) % n;
    }
    if (v_hi == v) {  // the vector straddles the end of the block
      if (t < unsigned(V)) element(v * V + t);
      ++v;
      continue;
    }
    if constexpr (kN >= 2) {
      if (tree) {
        if (f.op == kSum)
          fold_vectors<T, N, 1, kSum, true, kDstOnce>(dst, dst_aligned, sh, nremote, v, v_hi, 0, premul, scalar);
        else
          fold_vectors<T, N, 1, -1, true, kDstOnce>(dst, dst_aligned, sh, nremote, v, v_hi, 0, premul, scalar);
        v = v_hi;
        continue;
      }
    }
    if (f.op == kSum)
      fold_vectors<T, N, U, kSum, false, kDstOnce>(dst, dst_aligned, sh, nremote, v, v_hi, first, premul, scalar);
    else
      fold_vectors<T, N, 1, -1, false, kDstOnce>(dst, dst_aligned, sh, nremote, v, v_hi, first, premul, scalar);
    v = v_hi;
  }
  for (unsigned e = nvec * V + t; e < total; e += nt) element(e);
}

// ---- moving the pieces of a step ---------------------------------------------------------------------
// A step moves one piece per peer. Walked piece by piece, a CTA has only as many loads in flight as a
// piece has vectors, and pays a memory latency per piece; cta_pieces walks all of them as one range, so
// small pieces fill the machine as large ones do. A mover says what happens to a 16-byte vector of the
// window side on its way:
//   load(ok, src, i)       vector i of a piece, into registers, where ok
//   store(ok, dst, i, v)
//   element(dst, src, e)   one element, any alignment (tails, and pieces of odd alignment)
//   fits(dst, src)         whether load / store may be used for a piece with these addresses
template <typename M>
__device__ __forceinline__ void cta_pieces_one_by_one(const FoldShared& sh, int np, const M& m) {
  for (int j = 0; j < np; ++j) {
    const unsigned total = unsigned(sh.piece_len[j] / sizeof(typename M::Elem));
    for (unsigned e = threadIdx.x; e < total; e += blockDim.x) m.element(sh.piece_dst[j], sh.piece_src[j], e);
  }
}
// The caller has filled sh.piece_*[0..np) (threads below np, one each); no piece is longer than
// `longest`. Called by all threads; begins with the barrier that makes the table visible.
template <typename M>
__device__ __forceinline__ void cta_pieces(const FoldShared& sh, int np, size_t longest, M m) {
  constexpr int U = M::kUnroll, V = 16 / sizeof(typename M::Elem);
  const unsigned t = fresh_tid(), lane = t & 31u, nt = blockDim.x;
  __syncthreads();
  const bool fits = t >= unsigned(np) || sh.piece_len[t] == 0 || m.fits(sh.piece_dst[t], sh.piece_src[t]);
  if (!__syncthreads_and(fits)) {
    m.odd_pieces(sh, np);
    return;
  }
  // the range is cut into chunks of 32 vectors; a warp takes U consecutive ones at a time
  const unsigned row = unsigned((longest + 511) >> 9);  // chunks a piece takes in the walk
  const unsigned all = unsigned(np) * row;
  for (unsigned c0 = (t >> 5) * U; c0 < all; c0 += (nt >> 5) * U) {
    typename M::Reg r[U];
    const unsigned j0 = c0 / row, i0 = c0 - j0 * row;
    unsigned j = j0, i = i0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned v = i * 32 + lane;
      const bool ok = j < unsigned(np) && v < unsigned(sh.piece_len[j < unsigned(np) ? j : 0] >> 4);
      r[u] = m.load(ok, sh.piece_src[j < unsigned(np) ? j : 0], v);
      if (++i == row) i = 0, ++j;
    }
    j = j0;
    i = i0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned v = i * 32 + lane;
      const bool ok = j < unsigned(np) && v < unsigned(sh.piece_len[j < unsigned(np) ? j : 0] >> 4);
      m.store(ok, sh.piece_dst[j < unsigned(np) ? j : 0], v, r[u]);
      if (++i == row) i = 0, ++j;
    }
  }
  for (unsigned k = t; k < unsigned(np) * V; k += nt) {  // the elements behind each piece's last vector
    const unsigned p = k / V, e = k % V;
    const size_t len = sh.piece_len[p];
    if (e < unsigned(len & 15u) / unsigned(sizeof(typename M::Elem)))
      m.element(sh.piece_dst[p], sh.piece_src[p], unsigned(len >> 4) * V + e);
  }
}

// kOnceIn / kOnceOut: the source / the destination is not touched again soon
template <bool kOnceIn, bool kOnceOut>
struct CopyMover {
  using Elem = char;
  using Reg = uint4;
  static constexpr int kUnroll = 8;
  unsigned long long policy;
  __device__ __forceinline__ CopyMover() : policy(once_policy()) {}
  __device__ __forceinline__ bool fits(const char* dst, const char* src) const {
    return ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15u) == 0;
  }
  __device__ __forceinline__ uint4 load(bool ok, const char* src, unsigned i) const {
    const char* p = src + (size_t(i) << 4);
    return kOnceIn ? ld16_once_if(ok, p, policy) : ld16_if(ok, p);
  }
  __device__ __forceinline__ void store(bool ok, char* dst, unsigned i, uint4 v) const {
    char* p = dst + (size_t(i) << 4);
    if (kOnceOut) st16_once_if(ok, p, v, policy);
    else st16_if(ok, p, v);
  }
  __device__ __forceinline__ void element(char* dst, const char* src, unsigned e) const { dst[e] = src[e]; }
  __device__ __forceinline__ void odd_pieces(const FoldShared& sh, int np) const {
    for (int j = 0; j < np; ++j) cta_copy(sh.piece_dst[j], sh.piece_src[j], sh.piece_len[j]);
  }
};
// dst = src * scalar (pre-scaled pushes)
template <typename T>
struct ScaleMover {
  using Elem = T;
  using Reg = uint4;
  static constexpr int kUnroll = 8;
  T scalar;
  unsigned long long policy;
  __device__ __forceinline__ explicit ScaleMover(T k) : scalar(k), policy(once_policy()) {}
  __device__ __forceinline__ bool fits(const char* dst, const char* src) const {
    return ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15u) == 0;
  }
  __device__ __forceinline__ uint4 load(bool ok, const char* src, unsigned i) const { return ld16_once_if(ok, src + (size_t(i) << 4), policy); }
  __device__ __forceinline__ void store(bool ok, char* dst, unsigned i, uint4 v) const {
    Vec16<T> x;
    x.raw = v;
    st16_if(ok, dst + (size_t(i) << 4), scale_lanes(x, scalar).raw);
  }
  __device__ __forceinline__ void element(char* dst, const char* src, unsigned e) const {
    reinterpret_cast<T*>(dst)[e] = scale(reinterpret_cast<const T*>(src)[e], scalar);
  }
  // an aligned destination (a window slot) still takes whole vectors, cut out of the source's
  __device__ __forceinline__ void odd_pieces(const FoldShared& sh, int np) const {
    for (int j = 0; j < np; ++j) {
      char* dst = sh.piece_dst[j];
      const char* src = sh.piece_src[j];
      const unsigned s = unsigned(reinterpret_cast<uintptr_t>(src) & 15u), t = fresh_tid(), nt = blockDim.x;
      const unsigned nvec = (reinterpret_cast<uintptr_t>(dst) & 15u) == 0 ? unsigned(sh.piece_len[j] >> 4) : 0;
      for (unsigned i = (t >> 5) * 64 + (t & 31u); i < nvec; i += nt * 2) {  // runs of 2 x 512 bytes per warp
        const char* p = src - s + (size_t(i) << 4);
        uint4 r[2], q[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          r[u] = ld16_if(u * 32 < nvec - i, p + u * 512);
          q[u] = ld16_if(u * 32 < nvec - i && s, p + u * 512 + 16);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) store(u * 32 < nvec - i, dst, i + u * 32, bytes_of_pair(r[u], q[u], s));
      }
      const unsigned total = unsigned(sh.piece_len[j] / sizeof(T));
      for (unsigned e = nvec * unsigned(16 / sizeof(T)) + t; e < total; e += nt) element(dst, src, e);
    }
  }
};
// dst = src * scalar for one piece (the NVLS kernels)
template <typename T>
__device__ inline void cta_scale_copy(char* dst, const char* src, size_t nbytes, T scalar) {
  constexpr int V = 16 / sizeof(T);
  const unsigned t = threadIdx.x, nt = blockDim.x;
  const ScaleMover<T> m(scalar);
  const unsigned nvec = m.fits(dst, src) ? unsigned(nbytes >> 4) : 0;
  for (unsigned i = t; i < nvec; i += nt) m.store(true, dst, i, m.load(true, src, i));
  const unsigned total = unsigned(nbytes / sizeof(T));
  for (unsigned e = nvec * V + t; e < total; e += nt) m.element(dst, src, e);
}

// ---- fp32 buffers with a narrow type on the wire (gradient buckets) --------------------------------
// Eight fp32 values rounded to T under the library's rule: the packed converter rounds to nearest even
// and overflows to infinity as the rule does; only its NaN code differs.
__device__ __forceinline__ unsigned narrow_pair(float lo, float hi, f16) {
  unsigned r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ unsigned narrow_pair(float lo, float hi, bf16) {
  unsigned r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
template <typename T>
__device__ __forceinline__ Vec16<T> narrow_lanes(const uint4& a, const uint4& b) {
  const float in[8] = {bits_f32(a.x), bits_f32(a.y), bits_f32(a.z), bits_f32(a.w),
                       bits_f32(b.x), bits_f32(b.y), bits_f32(b.z), bits_f32(b.w)};
  Vec16<T> x;
  x.raw = make_uint4(narrow_pair(in[0], in[1], T{}), narrow_pair(in[2], in[3], T{}), narrow_pair(in[4], in[5], T{}),
                     narrow_pair(in[6], in[7], T{}));
#pragma unroll
  for (int l = 0; l < 8; ++l)
    if (in[l] != in[l]) from_f32(in[l], &x.e[l]);
  return x;
}

// dst[i] = scale(narrow(src[i]), scalar): rounds fp32 values to T (nearest even, the library's
// overflow and NaN rules) and applies the pre-scale in T's rule, as a cast followed by the
// ordinary pre-scaled push would. Piece lengths count bytes of T.
template <typename T>
struct NarrowMover {
  using Elem = T;
  struct Reg {
    uint4 a, b;
  };
  static constexpr int kUnroll = 4;
  T scalar;
  bool premul;
  __device__ __forceinline__ NarrowMover(T k, bool p) : scalar(k), premul(p) {}
  __device__ __forceinline__ bool fits(const char* dst, const char* src) const {
    return ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15u) == 0;
  }
  __device__ __forceinline__ Reg load(bool ok, const char* src, unsigned i) const {
    const char* p = src + (size_t(i) << 5);
    return Reg{ld16_if(ok, p), ld16_if(ok, p + 16)};  // through L1: the two share sectors
  }
  __device__ __forceinline__ void store(bool ok, char* dst, unsigned i, const Reg& r) const {
    Vec16<T> x = narrow_lanes<T>(r.a, r.b);
    if (premul) x = scale_lanes(x, scalar);
    st16_if(ok, dst + (size_t(i) << 4), x.raw);
  }
  __device__ __forceinline__ void element(char* dst, const char* src, unsigned e) const {
    T x;
    from_f32(reinterpret_cast<const float*>(src)[e], &x);
    reinterpret_cast<T*>(dst)[e] = premul ? scale(x, scalar) : x;
  }
  __device__ __forceinline__ void odd_pieces(const FoldShared& sh, int np) const { cta_pieces_one_by_one(sh, np, *this); }
};
// dst[i] = float(src[i]) (exact). Piece lengths count bytes of T.
template <typename T>
struct WidenMover {
  using Elem = T;
  using Reg = uint4;
  static constexpr int kUnroll = 4;
  unsigned long long policy;
  __device__ __forceinline__ WidenMover() : policy(once_policy()) {}
  __device__ __forceinline__ bool fits(const char* dst, const char* src) const {
    return ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15u) == 0;
  }
  __device__ __forceinline__ uint4 load(bool ok, const char* src, unsigned i) const { return ld16_once_if(ok, src + (size_t(i) << 4), policy); }
  __device__ __forceinline__ void store(bool ok, char* dst, unsigned i, uint4 v) const {
    Vec16<T> x;
    x.raw = v;
    unsigned f[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) f[l] = f32_bits(to_f32(x.e[l]));
    char* out = dst + (size_t(i) << 5);
    st16_if(ok, out, make_uint4(f[0], f[1], f[2], f[3]));
    st16_if(ok, out + 16, make_uint4(f[4], f[5], f[6], f[7]));
  }
  __device__ __forceinline__ void element(char* dst, const char* src, unsigned e) const {
    reinterpret_cast<float*>(dst)[e] = to_f32(reinterpret_cast<const T*>(src)[e]);
  }
  __device__ __forceinline__ void odd_pieces(const FoldShared& sh, int np) const { cta_pieces_one_by_one(sh, np, *this); }
};

}  // namespace hx
